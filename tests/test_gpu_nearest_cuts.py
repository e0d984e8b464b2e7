"""A nearest-neighbour job gives the same bits however it is cut: one slice, a few
(angles split over groups of threads), batches (two and four slices per thread) and
large images (one slice per thread) add a pixel's angles in the same order."""
import numpy as np
import pytest

import risa_gb300 as rg

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reserved", [False, True])
@pytest.mark.parametrize("interp", [rg.INTERP_NEAREST, rg.INTERP_NEAREST_TRUNC])
@pytest.mark.parametrize("Pp,Dp,N,n,cuts", [
    (1, 32, 40, 130, [1, 2]), (4, 33, 40, 129, [1, 127]), (17, 33, 97, 140, [1, 3, 40]),
    (361, 301, 231, 17, [1, 3, 8]), (700, 260, 129, 24, [1, 2, 5, 20]), (45, 700, 160, 44, [1, 7]),  # 4.4 bins per pixel
    (130, 600, 750, 5, [1, 2, 3])])
def test_nearest_cuts(Pp, Dp, N, n, cuts, interp, reserved):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    bp = rg.Backprojection(rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N, rotation_offset=11.0),
                           rg.make_params(interp=interp, masking=True, masking_value=-1.0))
    if reserved:
        bp.reserve(n)
    sino = torch.from_numpy(np.random.default_rng(N).standard_normal((n, Pp, Dp)).astype(np.float32)).cuda()
    whole = torch.full((n, N, N), float("nan"), dtype=torch.float32, device="cuda")
    bp.enqueue(sino, whole, n)
    exp = whole.cpu().numpy()
    for m in cuts:
        for first in sorted({0, (n - m) // 2, n - m}):
            got = torch.full((m, N, N), float("nan"), dtype=torch.float32, device="cuda")
            bp.enqueue(sino[first:first + m].contiguous(), got, m)
            np.testing.assert_array_equal(got.cpu().numpy().view(np.uint32), exp[first:first + m].view(np.uint32))
