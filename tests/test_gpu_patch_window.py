"""Ray coordinates from two FP32 numbers per coefficient, where their rounded sum
reaches an integer that the coordinate lies just below (geometries searched for
that with the same FP32 steps): the tile windows of the patch kernels and the
single angles of symmetric sets keep FP64's bins.

Rows of alternating +1 and -1 show a coordinate's error doubled. In a tile the
coordinate is at most 44 bins from its window: two roundings of half a unit there
(2^-19 each), 15 pixels by the FP32 rounding of |a| and |b| (2^-24 each), 6e-6 of a
bin together, so 1.2e-5; the bar is 2e-5. An integer reached half a unit of 2^10
bins early is 6e-5 of a bin off, 1.2e-4."""
import numpy as np
import pytest

import risa_gb300 as rg

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BAR = 2e-5
f32 = np.float32


def _coefficients(Pp, Dp, N, rot, i):
    th = i * np.pi / Pp + rot * np.pi / 180.0
    a, b = Dp / N * np.cos(th), Dp / N * np.sin(th)
    return a, b, Dp * 0.5 - 0.5 - (N - 1.0) * 0.5 * (a + b)


def _rounds_up(t0, a, b, x, y, align):
    """How far (bins) the rounded sum lies above the coordinate where the floors differ."""
    def split(v):
        hi = f32(v)
        return hi, f32(v - np.float64(hi))

    def fma(p, q, r):
        return f32(np.longdouble(p) * np.longdouble(q) + np.longdouble(r))
    (th, tl), (ah, al), (bh, bl) = split(t0), split(a), split(b)
    x, y = f32(x), f32(y)
    p, q = x * ah, y * bh
    pe, qe = fma(x, al, fma(x, ah, -p)), fma(y, bl, fma(y, bh, -q))
    s = th + p
    se = (th - (s - (s - th))) + (p - (s - th))
    u = s + q
    ue = (s - (u - (u - s))) + (q - (u - s))
    top = u + ((se + ue) + ((pe + qe) + tl))
    exact = t0 + np.float64(x) * a + np.float64(y) * b
    early = (np.floor(top) > exact) & (np.floor(top).astype(np.int64) % align == 0)
    return np.where(early, np.floor(top) - exact, 0.0).max()


def _expected(row, a, b, t0, N):
    pix = np.arange(N)
    s = t0 + pix[None, :] * a + pix[:, None] * b
    k = np.floor(s).astype(np.int64)
    pad = np.concatenate([[0.0, 0.0], row, [0.0, 0.0]])
    at = np.clip(k + 2, 0, len(row) + 2)
    return pad[at] + (s - k) * (pad[at + 1] - pad[at])


def _check(bp, row_index, Pp, Dp, N, n, coef):
    sino = np.zeros((n, Pp, Dp), f32)
    sino[:, row_index] = 1.0 - 2.0 * (np.arange(Dp) % 2)
    img = torch.full((n, N, N), float("nan"), dtype=torch.float32, device="cuda")
    bp.enqueue(torch.from_numpy(sino).cuda(), img, n)
    bp.check()
    norm = np.pi / Pp / (Dp / N)
    exp = _expected(sino[0, row_index].astype(np.float64), *coef, N)
    got = img.cpu().numpy().astype(np.float64) / norm
    assert np.abs(got - exp).max() < BAR


@pytest.mark.parametrize("n", [1, 3])  # over the sinogram itself (windows at multiples of 4 bins), and staged
def test_tile_windows(n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    Pp, Dp, N = 1, 2048, 1024
    rng = np.random.default_rng(7)
    tx, ty = np.meshgrid(np.arange(0, N, 16), np.arange(0, N, 16))
    for _ in range(2000):
        rot = float(rng.uniform(-180.0, 180.0))
        a, b, t0 = _coefficients(Pp, Dp, N, rot, 0)
        if _rounds_up(t0, a, b, tx + (15 if a < 0 else 0), ty + (15 if b < 0 else 0), 4 if n == 1 else 1) > 3e-5:
            break
    else:
        raise AssertionError("no such geometry")
    bp = rg.Backprojection(rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N, rotation_offset=rot),
                           rg.make_params())
    _check(bp, 0, Pp, Dp, N, n, (a, b, t0))


def test_single_angles_of_symmetric_sets():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    Pp, N = 8, 1024
    pix = np.arange(N)
    for Dp in range(2048, 1024, -4):
        found = [i for i in (2, 6) if _rounds_up(*[_coefficients(Pp, Dp, N, 0.0, i)[j] for j in (2, 0, 1)],
                                                 pix[None, :], pix[:, None], 1) > 1.5e-5]
        if found:
            break
    else:
        raise AssertionError("no such geometry")
    bp = rg.Backprojection(rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N), rg.make_params())
    _check(bp, found[0], Pp, Dp, N, 1, _coefficients(Pp, Dp, N, 0.0, found[0]))
