"""The taps gradient at every radix-16 length, with rows of at most half the
transform (their zero half not transformed) and longer ones, one row up to more
rows than one pass of the grid, odd row counts, against the direct FP64 sum
grad[j] = sum over rows and n of g[n] x[n - (j - n_taps/2)]."""
import numpy as np
import pytest

import risa_gb300 as rg

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Pp,Dp,n_taps,pad,n", [
    (1, 33, 7, 0, 1),       # length 64: the general transform
    (1, 200, 300, 0, 1),    # 512, half; a single row
    (3, 257, 129, 0, 3),    # 512, over half; an odd number of rows
    (2100, 40, 9, 512, 1),  # 512: more pairs than one pass of the grid
    (5, 512, 400, 0, 2),    # 1024, exactly half
    (7, 600, 400, 0, 1),    # 1024, over half
    (1, 1000, 1025, 0, 2), (3, 1500, 500, 0, 1),  # 2048
    (3, 2000, 2049, 0, 1), (2, 3000, 100, 0, 2),  # 4096
])
def test_taps_gradient_lengths(Pp, Dp, n_taps, pad, n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=32)
    rng = np.random.default_rng(Dp)
    filt = rg.Filter(g, rg.make_params(pad=pad), taps=rng.standard_normal(n_taps).astype(np.float32))
    x = rng.standard_normal((n, Pp, Dp)).astype(np.float32)
    d = rng.standard_normal((n, Pp, Dp)).astype(np.float32)
    got = torch.full((n_taps,), float("nan"), dtype=torch.float32, device="cuda")
    ws = torch.empty(filt.taps_grad_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    filt.taps_grad(torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda(), got, n, ws)
    got = got.cpu().numpy().astype(np.float64)
    ln = 2 * Dp + n_taps
    corr = np.fft.irfft((np.fft.rfft(d.astype(np.float64), ln) * np.fft.rfft(x.astype(np.float64), ln).conj())
                        .sum((0, 1)), ln)
    lag = np.arange(n_taps) - n_taps // 2
    exp = np.where(np.abs(lag) < Dp, corr[lag % ln], 0.0)
    assert np.abs(got - exp).max() <= 1e-5 * np.abs(exp).max()
