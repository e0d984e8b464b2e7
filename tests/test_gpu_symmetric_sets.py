"""Angles taken in sets of four (theta, pi - theta, pi/2 +- theta) by the uneven
sweep and by single-frame backprojections: angle counts around the smallest that
has a set, counts that are and are not multiples of 4, odd and rotated ones
(taken singly), with and without the circular mask, image sides off the tile
grid -- against the FP64 oracle, and the same bits on a second launch."""
import numpy as np
import pytest

import oracle
import risa_gb300 as rg
from risa_gb300 import phantom
from tests.helpers import rel_err
from tests.test_gpu_sweep import _oracle, _run

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MAX_REL = 1e-5
SHAPES = [(33, 6, 160, True, 0.0), (33, 8, 160, False, 0.0), (64, 10, 160, True, 0.0), (65, 12, 200, False, 0.0),
          (130, 182, 170, False, 0.0), (47, 184, 140, True, 0.0), (47, 183, 140, True, 0.0), (47, 184, 140, True, 90.0)]


def test_sweep_symmetric_sets():
    # large enough for sets: the last instances fill the sweep to over 5000 tiles
    fill = [(1024, 8, 160, True, 0.0)] * 5
    inst = [dict(n_pixels=n, n_par_proj=pp, n_par_det=dp, filter_type="ramp", cutoff=1.0, rotation_offset=rot,
                 ref_level=40200.0, dark_level=200.0, masking=m, masking_value=-2.0 if m else 0.0, defect_map=None)
            for n, pp, dp, m, rot in SHAPES + fill]
    sw, raws, img, io = _run(inst, 900)
    for i, d in enumerate(inst[:len(SHAPES) + 1]):
        n = d["n_pixels"]
        got = img[io[i]:io[i] + n * n].reshape(n, n)
        mr, l2 = rel_err(got, _oracle(d, raws[i]))
        assert mr < MAX_REL and l2 < MAX_REL, (i, mr, l2)
    packed = torch.from_numpy(np.concatenate([r.ravel() for r in raws]).view(np.int16)).cuda()
    again = torch.full((img.size,), float("nan"), dtype=torch.float32, device="cuda")
    sw.enqueue(packed, again)
    sw.check()
    np.testing.assert_array_equal(again.cpu().numpy().view(np.uint32), img.view(np.uint32))
    first, done, launch = sw.times()  # every instance has started and ended
    assert (done > first).all() and (first >= launch).all()


@pytest.mark.parametrize("Pp", [1, 2, 4, 6, 8, 10, 12, 180])
@pytest.mark.parametrize("N,Dp,masking", [(40, 40, False), (41, 80, True), (400, 64, True)])
def test_single_frame_symmetric_sets(Pp, N, Dp, masking):
    g = rg.make_geometry(n_par_proj=Pp, n_par_det=Dp, n_pixels=N)
    bp = rg.Backprojection(g, rg.make_params(masking=masking, masking_value=4.0))
    sino, _ = phantom.parallel_sinograms(2, Pp, Dp, 200.0, seed=Pp)
    t = torch.from_numpy(sino).cuda()
    img = torch.full((2, N, N), float("nan"), dtype=torch.float32, device="cuda")
    bp.enqueue(t, img, 2)
    bp.check()
    got = img.cpu().numpy()
    for b in range(2):
        exp = oracle.backproject(sino[b], N)
        mr, _ = rel_err(got[b], oracle.mask(exp, 4.0) if masking else exp)
        assert mr < MAX_REL, (b, mr)
