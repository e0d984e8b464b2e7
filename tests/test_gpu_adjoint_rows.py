"""The adjoint over slice-interleaved image copies, at the edges of its launch
rule: up to 4 and more than 4 slices of a group, groups of 8 slices on one warp
and on two, 1 to 8 angles per CTA, 1 to 4 candidate pixels per row (bins per pixel
from 0.3 to 2), rays that miss the image, and image sides too large for eight
angles' line starts -- against the direct gather (no scratch), whose terms and
their order are the same."""
import numpy as np
import pytest

import risa_gb300 as rg

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Pp,Dp,N,n,rot", [
    (33, 50, 40, 1, 0.0), (33, 50, 40, 4, -77.0), (33, 50, 40, 5, 12.5), (9, 31, 97, 8, 0.0),  # 0.32 bins per pixel
    (40, 130, 65, 9, 30.0), (17, 64, 200, 3, 45.0),  # 2 bins; 0.32 bins
    (300, 300, 64, 2, 0.0),   # 3000 warps, most rays outside the image's middle rows
    (400, 500, 48, 13, 10.0),  # over 4864 warps: 8 slices per warp, bins far outside the image
    (5, 40, 800, 2, 7.0), (4, 24, 3200, 1, 90.0),  # fewer angles per CTA; 0.0075 bins per pixel
])
def test_adjoint_rows(Pp, Dp, N, n, rot):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    # rays reach past the image when the detector is wider than it: scale Dp / N as given
    g = rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N, rotation_offset=rot)
    direct, fast = rg.Backprojection(g, rg.make_params()), rg.Backprojection(g, rg.make_params())
    fast.reserve_adjoint(n)
    img = torch.from_numpy(np.random.default_rng(N).standard_normal((n, N, N)).astype(np.float32)).cuda()
    img[n - 1, N // 2, N // 3] = float("inf")  # reaches the bins of its rays and no others
    a, b = (torch.full((n, Pp, Dp), float("nan"), dtype=torch.float32, device="cuda") for _ in range(2))
    direct.enqueue_adjoint(img, a, n)
    fast.enqueue_adjoint(img, b, n)
    a, b = a.cpu().numpy().astype(np.float64), b.cpu().numpy().astype(np.float64)
    np.testing.assert_array_equal(np.isfinite(a), np.isfinite(b))
    fine = np.isfinite(a)
    assert not fine.all()
    np.testing.assert_array_equal(a[fine], b[fine])
