"""Defect runs where their order and their wraps matter (first column, last
column, both, every column), in detector-major and module-major frames, with few
frames and with a batch, columns in aligned octets and not: flags and repaired
frames bit for bit against the oracle, and the engine's repair on the fly gives
the image of the frames repaired beforehand, bit for bit. And the filter at
transform length 256, which shares the engine's rows of two at a time."""
import numpy as np
import pytest

import oracle
import risa_gb300 as rg
from tests.helpers import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
QUIRKS = [rg.QUIRKS_RISA, rg.QUIRKS_NONE]


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _frames(n, P, D, cols):
    rng = np.random.default_rng(D + P)
    f = rng.integers(20000, 22000, (n, P, D)).astype(np.uint16)
    for b in range(n):
        f[b][:, [c % D for c in cols]] = 300 + b  # dead
        f[b][:, (7 * b + 40) % D] = rng.integers(0, 65535, P)  # flickering
    return f


EDGES = [[0], [-1], [0, -1], [0, 1, 2, -2, -1], [1, -1, 30, 31], list(range(0, 24, 2)), [0, 1, 5, 6, -1]]


@pytest.mark.parametrize("quirk", QUIRKS)
@pytest.mark.parametrize("P,D,modules,n", [
    (60, 432, 0, 1), (60, 432, 27, 3), (9, 2080, 0, 2), (33, 248, 31, 1), (60, 434, 0, 2),  # few frames
    (60, 432, 18, 1), (60, 432, 36, 2),  # module widths of 24 and of 12
    (17, 256, 0, 160), (17, 2304, 0, 153), (17, 256, 8, 160),  # a batch
    (2, 64, 0, 1)])
def test_flags_and_repair(P, D, modules, n, quirk):
    g = rg.make_geometry(n_fan_det=D, n_fan_proj=P, n_modules=modules or 1)
    h = rg.Defects(g, rg.make_params(quirks=quirk, module_major=modules > 0), max_batch=n)
    ws = torch.empty(h.workspace_bytes(n), dtype=torch.uint8, device="cuda")
    for cols in EDGES if n < 100 else EDGES[3:4]:
        f = _frames(n, P, D, cols)
        t = torch.from_numpy((rg.to_module_major(f, modules) if modules else f).view(np.int16).copy()).cuda()
        flags = torch.zeros((n, D), dtype=torch.int32, device="cuda")
        h.enqueue(t, n, ws, flags_out=flags)
        got, gf = t.cpu().numpy().view(np.uint16), flags.cpu().numpy()
        for b in range(n):
            of = oracle.find_defects(f[b], 0.67, 1.5, quirk)
            np.testing.assert_array_equal(gf[b], of[:D])
            exp = oracle.interpolate_defects(f[b], of, quirk)
            np.testing.assert_array_equal(got[b], rg.to_module_major(exp[None], modules)[0] if modules else exp)


@pytest.mark.parametrize("quirk", QUIRKS)
@pytest.mark.parametrize("D,modules", [(432, 0), (432, 27), (434, 0), (433, 0)])
def test_engine_repairs_on_the_fly(D, modules, quirk):
    P, n = 62, 5
    kw = dict(quirks=quirk, module_major=modules > 0)
    dp = 256 if quirk == rg.QUIRKS_RISA else 96  # filter length 256 in both
    g = rg.make_geometry(n_fan_det=D, n_fan_proj=P, n_par_proj=64, n_par_det=dp, n_pixels=64, n_modules=modules or 1)
    ref = np.full((1, 1, P, D), 40000, np.uint16)
    dark = np.full((1, 1, P, D), 150, np.uint16)
    with_repair = rg.FBP(g, rg.make_params(defects=True, **kw), ref, 1, dark, 1, max_batch=n)
    without = rg.FBP(g, rg.make_params(defects=False, **kw), ref, 1, dark, 1, max_batch=n)
    h = rg.Defects(g, rg.make_params(**kw), max_batch=n)
    ws = torch.empty(h.workspace_bytes(n), dtype=torch.uint8, device="cuda")
    for cols in EDGES:
        f = _frames(n, P, D, cols)
        raw = torch.from_numpy((rg.to_module_major(f, modules) if modules else f).view(np.int16).copy()).cuda()
        img = [torch.full((n, 64, 64), float("nan"), dtype=torch.float32, device="cuda") for _ in range(2)]
        with_repair.enqueue(raw, img[0], 0, n)
        torch.cuda.synchronize()
        h.enqueue(raw, n, ws)
        without.enqueue(raw, img[1], 0, n)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(img[0].cpu().numpy(), img[1].cpu().numpy())
        assert np.isfinite(img[0].cpu().numpy()).all()


@pytest.mark.parametrize("dp,quirk,rows", [(100, rg.QUIRKS_NONE, 1), (128, rg.QUIRKS_NONE, 17),
                                           (65, rg.QUIRKS_NONE, 15), (256, rg.QUIRKS_RISA, 37)])
def test_filter_length_256(dp, quirk, rows):
    g = rg.make_geometry(n_par_proj=rows, n_par_det=dp, n_pixels=64)
    filt = rg.Filter(g, rg.make_params(quirks=quirk, filter_type="hamming", cutoff=0.9))
    n, _ = filt.response()
    assert n == 256
    x = np.abs(np.random.default_rng(dp).standard_normal((3, rows, dp))).astype(np.float32)
    t = torch.from_numpy(x).cuda()
    filt.enqueue(t, 3)
    got = t.cpu().numpy()
    ho = oracle.design_filter(n, rg.FILTERS["hamming"], 0.9, quirk)
    for b in range(3):
        assert rel_err(got[b], oracle.filter_rows(x[b], n, ho))[0] < 1e-5
