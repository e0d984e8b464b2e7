"""Infinities and NaN in the rows of the patch backprojection: a non-finite sample
reaches the pixels whose two bins it is one of and no others, and the slices
without one keep the bits of a clean batch."""
import numpy as np
import pytest

import risa_gb300 as rg

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


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("Dp", [48, 72, 96])  # 1, 1.5 and 2 bins per pixel: the shapes of the launch rule
@pytest.mark.parametrize("n,bad", [(100, [(50, 7, 30), (53, 19, 2)]), (7, [(1, 0, 0)]), (64, [(63, 11, 40)])])
def test_nonfinite_slices_alone_leave_the_patches(value, Dp, n, bad):
    """Every slice without a non-finite sample has the bits of a clean batch, also the
    others of its quad and of its CTA; the bad slices are the general kernel's."""
    Pp, N = 20, 48
    g = rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N, rotation_offset=3.3)
    bp = rg.Backprojection(g, rg.make_params(masking=True))
    bp.reserve(n)
    base = np.random.default_rng(n).standard_normal((n, Pp, Dp)).astype(np.float32)
    hurt = base.copy()
    for at in bad:
        hurt[at] = value
    clean = _run(bp, torch.from_numpy(base).cuda(), N, n)
    got = _run(bp, torch.from_numpy(hurt).cuda(), N, n)
    fine = [b for b in range(n) if b not in [at[0] for at in bad]]
    np.testing.assert_array_equal(got[fine], clean[fine])
    bp.set_variant(_variant("tile32_p4_a32"))
    exp = _run(bp, torch.from_numpy(hurt).cuda(), N, n)
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(exp))
    ok = np.isfinite(exp)
    assert np.abs(got[ok] - exp[ok]).max() < MAX_REL * np.abs(exp[ok]).max()


@pytest.mark.parametrize("n", [3, 7, 40])
def test_nonfinite_sample_between_exact_bins(n):
    """One bin per pixel at angle 0: every coordinate is a whole number k, whose bins are k and k + 1."""
    Pp, N = 12, 40
    bp = rg.Backprojection(rg.make_geometry(n_par_proj=Pp, n_par_det=N, n_pixels=N), rg.make_params())
    bp.reserve(n)
    sino = np.ones((n, Pp, N), np.float32)
    sino[1, 0, 17] = sino[2, 0, 22] = np.inf
    got = ~np.isfinite(_run(bp, torch.from_numpy(sino).cuda(), N, n))
    exp = np.zeros((n, N, N), bool)
    exp[1, :, 16:18] = exp[2, :, 21:23] = True
    np.testing.assert_array_equal(got, exp)


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("row", [0, 3, 5, 10, 15, 17])  # alone, alone (Pp / 4 ..), and each of a symmetric set
@pytest.mark.parametrize("n", [1, 2])
def test_nonfinite_samples_of_unrotated_frames(n, row, value):
    """The symmetric sets and the angles outside them (rows 0, 5, 10 and 15 of 20)."""
    Pp, Dp, N = 20, 72, 47
    g = rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N)
    bp = rg.Backprojection(g, rg.make_params())
    sino = np.random.default_rng(row).standard_normal((n, Pp, Dp)).astype(np.float32)
    sino[n - 1, row, 31] = value
    got = _run(bp, torch.from_numpy(sino).cuda(), N, n)
    bp.set_variant(_variant("tile32_p4_a32"))
    exp = _run(bp, torch.from_numpy(sino).cuda(), N, n)
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(exp))
    assert not np.isfinite(exp[n - 1]).all()
    ok = np.isfinite(exp)
    assert np.abs(got[ok] - exp[ok]).max() < MAX_REL * np.abs(exp[ok]).max()
