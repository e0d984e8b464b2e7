"""The 2 x 2 patch backprojection (variant patch_2x2, the default): every shape
its launch rule picks (one quad of slices to several CTAs of 16 quads), every
class of angles (bins per pixel from below 1/2 to 2, where the patch's offsets
cross 1 and 2 bins), mirrored axes (rotation offsets that turn the signs of the
angle coefficients), odd sizes, partial tiles and quads, and rows that hold
infinities or NaN. FP32 bar: 1e-5 of the largest magnitude against the FP64
oracle."""
import numpy as np
import pytest

import oracle
import risa_gb300 as rg
from risa_gb300 import phantom
from tests.helpers import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MAX_REL = 1e-5


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.init()


def _variant(name):
    return [rg.Backprojection.variant_name(v) for v in range(rg.Backprojection.variant_count())].index(name)


def _run(bp, sino, N, n):
    img = torch.full((n, N, N), float("nan"), dtype=torch.float32, device="cuda")
    bp.enqueue(sino, img, n)
    torch.cuda.synchronize()
    bp.check()
    return img.cpu().numpy()


@pytest.mark.parametrize("Dp,N", [(33, 97), (96, 97), (64, 64), (81, 65), (96, 64), (127, 64), (128, 64), (65, 33)])
@pytest.mark.parametrize("quirk", [rg.QUIRKS_NONE, rg.QUIRKS_RISA])
def test_patch_classes(Dp, N, quirk):
    """Bins per pixel 0.34 .. 2 (2 exactly: |a| = 2 at angle 0), three rotation offsets."""
    Pp, n = 50, 3
    sino, _ = phantom.parallel_sinograms(n, Pp, Dp, 200.0, seed=Dp + N)
    for rot in (0.0, -37.5, 200.0):
        g = rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N, rotation_offset=rot)
        for masking in (False, True):
            bp = rg.Backprojection(g, rg.make_params(quirks=quirk, masking=masking, masking_value=-3.0))
            bp.set_variant(_variant("patch_2x2"))
            got = _run(bp, torch.from_numpy(sino).cuda(), N, n)
            for b in range(n):
                exp = oracle.backproject(sino[b], N, rot, 0, quirk)
                if masking:
                    exp = oracle.mask(exp, -3.0)
                mr, _ = rel_err(got[b], exp)
                assert mr < MAX_REL, (rot, masking, b, mr)


@pytest.mark.parametrize("Dp", [40, 80])  # 1 and 2 bins per pixel: the two halves of the launch rule
@pytest.mark.parametrize("n", [1, 4, 5, 8, 9, 16, 17, 31, 33, 63, 65, 97])
def test_patch_slice_counts(n, Dp):
    """Every split of the slices over quads, threads and CTAs gives the bits of
    the same slices one quad at a time, and the oracle's values."""
    Pp, N = 23, 40
    g = rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N, rotation_offset=5.0)
    bp = rg.Backprojection(g, rg.make_params(masking=True))
    bp.reserve(n)
    base, _ = phantom.parallel_sinograms(7, Pp, Dp, 200.0, seed=n)
    sino = torch.from_numpy(np.ascontiguousarray(base[np.arange(n) % 7])).cuda()
    got = _run(bp, sino, N, n)
    for b in range(0, n, 4):
        m = min(4, n - b)
        one = _run(bp, sino[b:b + m].contiguous(), N, m)
        np.testing.assert_array_equal(got[b:b + m].view(np.uint32), one.view(np.uint32))
    for b in range(min(n, 7)):
        mr, _ = rel_err(got[b], oracle.mask(oracle.backproject(base[b], N, 5.0), 0.0))
        assert mr < MAX_REL, (b, mr)


def test_patch_angle_limits():
    """2048 angles run; one more, and more than 2 bins per pixel, take the general variant."""
    for Pp, Dp, N in ((2048, 40, 32), (2049, 40, 32), (1, 40, 32), (30, 130, 64)):
        g = rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N)
        bp = rg.Backprojection(g, rg.make_params())
        sino, _ = phantom.parallel_sinograms(1, Pp, Dp, 200.0, seed=3)
        got = _run(bp, torch.from_numpy(sino).cuda(), N, 1)
        mr, _ = rel_err(got[0], oracle.backproject(sino[0], N))
        assert mr < MAX_REL, (Pp, Dp, N, mr)


@pytest.mark.parametrize("N,Dp,Pp", [(97, 96, 150), (97, 132, 97), (64, 128, 130), (33, 12, 65), (400, 400, 70),
                                     (41, 41, 20)])
def test_patch_single_frames(N, Dp, Pp):
    """Handles that were never reserved for more than two slices read the
    sinogram itself (four and two groups of angles; chunks of 64 angles with
    partial ones; Dp % 4 != 0 takes the staged quads): the oracle's values, and
    the same bits for two slices at once and one by one."""
    for rot in (0.0, 143.0):
        g = rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N, rotation_offset=rot)
        bp = rg.Backprojection(g, rg.make_params(masking=True, masking_value=2.0))
        sino, _ = phantom.parallel_sinograms(2, Pp, Dp, 200.0, seed=Pp)
        t = torch.from_numpy(sino).cuda()
        got = _run(bp, t, N, 2)
        for b in range(2):
            mr, _ = rel_err(got[b], oracle.mask(oracle.backproject(sino[b], N, rot), 2.0))
            assert mr < MAX_REL, (rot, b, mr)
            one = _run(bp, t[b:b + 1].contiguous(), N, 1)
            np.testing.assert_array_equal(one[0].view(np.uint32), got[b].view(np.uint32))
        # an unaligned sinogram takes the staged quads
        shifted = torch.empty(sino.size + 1, dtype=torch.float32, device="cuda")[1:].view(sino.shape)
        shifted.copy_(t)
        mr, _ = rel_err(_run(bp, shifted, N, 2)[1], got[1])
        assert mr < MAX_REL, mr


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("n", [1, 6, 40])
def test_patch_nonfinite_rows(value, n):
    """A non-finite sample reaches the pixels whose two bins it is one of and no
    others, as in the general kernel; slices of other quads keep their bits."""
    Pp, Dp, N = 20, 72, 48
    g = rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N, rotation_offset=3.3)
    bp = rg.Backprojection(g, rg.make_params())
    bp.reserve(n)
    base, _ = phantom.parallel_sinograms(n, Pp, Dp, 200.0, seed=8)
    bad = base.copy()
    bad[n // 2, 7, 30] = value
    clean = _run(bp, torch.from_numpy(base).cuda(), N, n)
    got = _run(bp, torch.from_numpy(bad).cuda(), N, n)
    bp.set_variant(_variant("tile32_p4_a32"))
    exp = _run(bp, torch.from_numpy(bad).cuda(), N, n)
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(exp))
    assert not np.isfinite(got[n // 2]).all()
    fine = np.isfinite(exp)
    assert np.abs(got[fine] - exp[fine]).max() < MAX_REL * np.abs(exp[fine]).max()
    far = [b for b in range(n) if b // 64 != (n // 2) // 64]
    np.testing.assert_array_equal(got[far], clean[far])
    # the flags are per call: a clean call after it is the clean result again
    bp.set_variant(_variant("patch_2x2"))
    np.testing.assert_array_equal(_run(bp, torch.from_numpy(base).cuda(), N, n), clean)


@pytest.mark.parametrize("N,Dp,n", [
    (400, 400, 29), (400, 400, 64), (400, 380, 61), (64, 64, 30), (400, 400, 33),  # four quads per thread, and not
    (350, 525, 64), (350, 700, 61), (350, 700, 36), (350, 480, 20), (64, 128, 30), (64, 100, 61)])
def test_shapes_add_the_same_terms(N, Dp, n):
    """Large batches and images take other shapes than 8 slices do, with the same bits."""
    g = rg.make_geometry(n_par_proj=37, n_par_det=Dp, n_pixels=N, rotation_offset=11.0)
    bp = rg.Backprojection(g, rg.make_params(masking=True))
    bp.reserve(n)
    sino = torch.from_numpy(np.random.default_rng(Dp).standard_normal((n, 37, Dp)).astype(np.float32)).cuda()
    got = _run(bp, sino, N, n)
    for i in range(0, n, 8):
        m = min(8, n - i)
        if m <= 2 and n > 2:  # the tail as part of a full group
            i, m = n - 8, 8
        np.testing.assert_array_equal(got[i:i + m], _run(bp, sino[i:i + m].contiguous(), N, m))
