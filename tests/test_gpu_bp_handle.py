"""A backprojection handle's own buffers, and the kernels that do without them."""
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


def _handle(Pp, Dp, N, rot=0.0):
    return rg.Backprojection(rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N, rotation_offset=rot),
                             rg.make_params(masking=True))


def _sino(n, Pp, Dp, seed):
    return torch.from_numpy(np.random.default_rng(seed).standard_normal((n, Pp, Dp)).astype(np.float32)).cuda()


def _run(bp, sino, N, stream=None):
    img = torch.full((sino.shape[0], N, N), float("nan"), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    bp.enqueue(sino, img, sino.shape[0], stream)
    bp.check()
    return img.cpu().numpy()


@pytest.mark.parametrize("n", [1, 2])
def test_single_frames_need_no_staged_rows(n):
    """2048 angles x 2048 bins: four slices of staged rows are more than a new handle
    holds, which frames that are read in place do not miss."""
    Pp, Dp, N = 2048, 2048, 1024
    sino = _sino(n, Pp, Dp, n)
    reserved = _handle(Pp, Dp, N)
    reserved.reserve(2)
    np.testing.assert_array_equal(_run(_handle(Pp, Dp, N), sino, N), _run(reserved, sino, N))
