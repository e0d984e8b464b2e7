"""Child process of test_gpu_alloc_failure.py, started with a stand-in for
cudaMalloc preloaded that refuses requests from a given size on (the real call
with a size no device has, so that the runtime's own error state is that of a
real refusal). It runs without torch. Prints "ok"."""
import ctypes
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import risa_gb300 as rg  # noqa: E402
from tests import noalloc_reset_child as rt  # noqa: E402

FAKE = ctypes.CDLL(sys.argv[2])
FAKE.fake_refuse_from.argtypes = [ctypes.c_size_t]
ENOMEM = -5
Pp, Dp, N = 64, 256, 256


class Refused:
    """Requests of `size` bytes and more are refused; at least one has to be."""
    def __init__(self, size):
        self.size = size

    def __enter__(self):
        self.before = FAKE.fake_refusals()
        FAKE.fake_refuse_from(self.size)

    def __exit__(self, *exc):
        FAKE.fake_refuse_from(ctypes.c_size_t(-1).value)
        assert exc[0] is not None or FAKE.fake_refusals() > self.before, "nothing was refused"


def handle(pp=Pp, dp=Dp, n=N):
    return rg.Backprojection(rg.make_geometry(n_par_proj=pp, n_par_det=dp, n_pixels=n), rg.make_params(masking=True))


def sinograms(n, pp=Pp, dp=Dp):
    return np.random.default_rng(n).standard_normal((n, pp, dp)).astype(np.float32)


def backproject(bp, sino, N=N):
    n = sino.shape[0]
    d, img = rt.upload(sino), rt.upload(np.full((n, N, N), np.nan, np.float32))
    bp.enqueue(d, img, n)
    bp.check()
    out = rt.download(img, (n, N, N), np.float32)
    for p in (d, img):
        rt.ck(rt.RT.cudaFree(ctypes.c_void_p(p)), "cudaFree")
    return out


def reserve():
    """A refused reservation is an error and leaves the handle as it was."""
    for first, n in ((0, 2), (2, 2), (8, 2), (8, 8)):
        bp, sino = handle(), sinograms(n)
        if first:
            bp.reserve(first)
        before = backproject(bp, sino)
        with Refused(16 << 20):
            try:
                bp.reserve(1000)
            except rg.RisaError as e:
                assert e.status == ENOMEM, e.status
            else:
                raise AssertionError("the reservation was not refused")
        np.testing.assert_array_equal(backproject(bp, sino), before, err_msg=f"{first} {n}")


def create():
    """A new handle does without its optional buffers (here 4 MB of partial images and
    2 MB of staged rows; its tables are below 1.5 MB each)."""
    pp, dp, n_pix = 512, 256, 360
    with Refused(2 << 20):
        bp = handle(pp, dp, n_pix)
    plenty = handle(pp, dp, n_pix)
    for n in (1, 2, 3, 5):
        sino = sinograms(n, pp, dp)
        got, exp = backproject(bp, sino, n_pix), backproject(plenty, sino, n_pix)
        assert np.abs(got - exp).max() < 1e-5 * np.abs(exp).max(), n
    bp.reserve(8)
    plenty.reserve(8)
    sino = sinograms(8, pp, dp)
    np.testing.assert_array_equal(backproject(bp, sino, n_pix), backproject(plenty, sino, n_pix))


def sweep():
    """A large sweep does without the partial images of its symmetric sets (80 MB here)."""
    inst = [dict(n_pixels=1024, n_par_proj=pp, n_par_det=160, filter_type="ramp", ref_level=40200.0, dark_level=200.0,
                 masking=True) for pp in (8, 10, 12, 8, 9)]
    out = []
    for refuse in (True, False):
        if refuse:
            with Refused(64 << 20):
                sw = rg.Sweep(inst)
        else:
            sw = rg.Sweep(inst)
        raw_total, img_total = sw.layout()[2:]
        raw = np.random.default_rng(3).integers(300, 40000, raw_total).astype(np.uint16)
        d, img = rt.upload(raw), rt.upload(np.full(img_total, np.nan, np.float32))
        sw.enqueue(d, img)
        sw.check()
        out.append(rt.download(img, (img_total,), np.float32))
    assert np.abs(out[0] - out[1]).max() < 1e-5 * np.abs(out[1]).max()


def main():
    rt.RT = rt.cudart()
    rt.ck(rt.RT.cudaSetDevice(0), "cudaSetDevice")
    globals()[sys.argv[1]]()
    print("ok")


if __name__ == "__main__":
    main()
