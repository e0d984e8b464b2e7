"""A few slices: the nearest-neighbour backprojection with its angles split over
thread groups picks the same bins as the tile kernel that a larger batch takes
(whole-number sinograms, whose sums are exact in any order), and the
normalisation's minimum and maximum by a cluster are those of the image."""
import numpy as np
import pytest

import risa_gb300 as rg

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("quirk", [rg.QUIRKS_RISA, rg.QUIRKS_NONE])
@pytest.mark.parametrize("interp", [rg.INTERP_NEAREST, rg.INTERP_NEAREST_TRUNC])
@pytest.mark.parametrize("Pp,Dp,N,rot,masking", [
    (1, 32, 16, 0.0, False), (3, 33, 40, 12.0, True), (90, 128, 97, -7.5, True), (513, 100, 64, 0.0, False),
    (700, 700, 129, 90.0, True), (361, 301, 231, 0.0, False)])
def test_nearest_split_picks_the_same_bins(Pp, Dp, N, rot, masking, interp, quirk):
    g = rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N, rotation_offset=rot)
    bp = rg.Backprojection(g, rg.make_params(quirks=quirk, interp=interp, masking=masking, masking_value=-2.0))
    tiles = ((N + 31) // 32) ** 2
    big = 512 // tiles + 1  # one slice more than the split form takes
    sino = torch.from_numpy(np.random.default_rng(N).integers(-999, 1000, (big, Pp, Dp)).astype(np.float32)).cuda()
    exp = torch.full((big, N, N), float("nan"), dtype=torch.float32, device="cuda")
    bp.enqueue(sino, exp, big)
    for n in {1, 2, big - 1} - {0}:
        got = torch.full((n, N, N), float("nan"), dtype=torch.float32, device="cuda")
        bp.enqueue(sino[:n].contiguous(), got, n)
        np.testing.assert_array_equal(got.cpu().numpy(), exp[:n].cpu().numpy())


@pytest.mark.parametrize("quirk", [rg.QUIRKS_RISA, rg.QUIRKS_NONE])
@pytest.mark.parametrize("interp", [rg.INTERP_NEAREST, rg.INTERP_NEAREST_TRUNC])
@pytest.mark.parametrize("Dp,N,n,masking", [(600, 750, 2, True), (601, 737, 3, False), (1100, 750, 7, True),
                                            (2990, 750, 5, False), (33, 740, 4, False)])
def test_nearest_batches_match_single_slices(Dp, N, n, masking, interp, quirk):
    """Two or four slices per thread against the one-slice tiles that one slice of more than 512
    tiles takes, bit for bit; angles that are no multiple of a chunk, partial groups of slices."""
    Pp = 45
    g = rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N, rotation_offset=-33.0)
    bp = rg.Backprojection(g, rg.make_params(quirks=quirk, interp=interp, masking=masking, masking_value=7.0))
    sino = torch.from_numpy(np.random.default_rng(N).standard_normal((n, Pp, Dp)).astype(np.float32)).cuda()
    got = torch.full((n, N, N), float("nan"), dtype=torch.float32, device="cuda")
    bp.enqueue(sino, got, n)
    for i in range(n):
        exp = torch.full((1, N, N), float("nan"), dtype=torch.float32, device="cuda")
        bp.enqueue(sino[i:i + 1].contiguous(), exp, 1)
        np.testing.assert_array_equal(got[i].cpu().numpy(), exp[0].cpu().numpy())


@pytest.mark.parametrize("N,n", [(16, 1), (17, 3), (90, 1), (91, 2), (181, 5), (512, 1)])
def test_normalisation_range(N, n):
    g = rg.make_geometry(n_pixels=N)
    m = rg.Masking(g, rg.make_params(masking=True, masking_value=3.0, normalize=True))
    rng = np.random.default_rng(N)
    img = rng.standard_normal((n, N, N)).astype(np.float32)
    img[0].flat[-1] = 9.0  # the last pixel and the first are the first image's extremes, outside the circle
    img[0].flat[0] = -9.0
    img[n - 1].flat[N * N // 2] = np.nan  # not a number is passed over
    t = torch.from_numpy(img).cuda()
    ws = torch.full((m.workspace_bytes(n),), 255, dtype=torch.uint8, device="cuda")
    m.enqueue(t, n, ws)
    lo = np.nanmin(img, axis=(1, 2), keepdims=True)
    hi = np.nanmax(img, axis=(1, 2), keepdims=True)
    d = np.arange(N) - 0.5 * (N - 1)
    outside = d[:, None] ** 2 + d[None, :] ** 2 > 0.25 * N * N
    np.testing.assert_array_equal(t.cpu().numpy(), np.where(outside, np.float32(3.0), (img - lo) / (hi - lo)))
