"""A backprojection handle's own buffers, and the kernels that do without them."""
import threading

import numpy as np
import pytest

import oracle
import risa_gb300 as rg
from risa_gb300 import phantom
from tests.helpers import SMALL, geom, rel_err

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


def _capture(bp, sino, img, stream):
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        bp.enqueue(sino, img, sino.shape[0], stream)
    return graph


def _images(n, N):
    return torch.full((n, N, N), float("nan"), dtype=torch.float32, device="cuda")


@pytest.mark.parametrize("reserved", [0, 2, 8])
@pytest.mark.parametrize("n", [1, 2, 4, 8])
def test_captured_enqueue_outlives_a_reservation(n, reserved):
    Pp, Dp, N = 64, 128, 128
    bp = _handle(Pp, Dp, N)
    if reserved:
        bp.reserve(reserved)
    sino, img = _sino(n, Pp, Dp, n), _images(n, N)
    exp = [oracle.mask(oracle.backproject(s, N), 0.0) for s in sino.cpu().numpy()]
    graph = _capture(bp, sino, img, torch.cuda.Stream())
    bp.reserve(64)  # the staged rows move
    many = _sino(64, Pp, Dp, 5)
    other = _run(bp, many, N)
    for _ in range(2):
        img.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        for b in range(n):
            mr, _ = rel_err(img[b].cpu().numpy(), exp[b])
            assert mr < MAX_REL, (b, mr)
        np.testing.assert_array_equal(_run(bp, many, N), other)


@pytest.mark.parametrize("n", [1, 4])
def test_captured_enqueue_beside_other_calls(n):
    """Replays on one stream, calls of the same handle on another: the bits of each alone."""
    Pp, Dp, N = 180, 256, 256
    bp = _handle(Pp, Dp, N)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    sino, img = _sino(n, Pp, Dp, 1), _images(n, N)
    graph = _capture(bp, sino, img, a)
    with torch.cuda.stream(a):
        graph.replay()
    torch.cuda.synchronize()
    alone = img.cpu().numpy()
    sino2, img2 = _sino(n, Pp, Dp, 2), _images(n, N)
    alone2 = _run(bp, sino2, N)
    for _ in range(20):
        img.fill_(float("nan"))
        img2.fill_(float("nan"))
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            graph.replay()
        bp.enqueue(sino2, img2, n, b)
        with torch.cuda.stream(a):
            graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(img.cpu().numpy(), alone)
        np.testing.assert_array_equal(img2.cpu().numpy(), alone2)
    bp.check()


@pytest.mark.parametrize("threads", [False, True])
@pytest.mark.parametrize("n,reserved,aligned", [(1, 0, True), (2, 0, True), (2, 0, False), (4, 0, True), (6, 0, True),
                                                (1, 2, True), (16, 16, True)])
def test_two_streams(n, reserved, aligned, threads):
    """Two streams, from one host thread and from two: the bits of each call alone."""
    Pp, Dp, N = 180, 256, 256
    bp = _handle(Pp, Dp, N)
    if reserved:
        bp.reserve(reserved)
    sinos = []
    for seed in (1, 2):
        t = torch.empty(n * Pp * Dp + 1, dtype=torch.float32, device="cuda")[0 if aligned else 1:][:n * Pp * Dp]
        t = t.view(n, Pp, Dp)
        t.copy_(_sino(n, Pp, Dp, seed))
        sinos.append(t)
    alone = [_run(bp, s, N) for s in sinos]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    imgs = [[_images(n, N) for _ in range(12)] for _ in sinos]
    torch.cuda.synchronize()

    def calls(i):
        for img in imgs[i]:
            bp.enqueue(sinos[i], img, n, streams[i])

    if threads:
        work = [threading.Thread(target=calls, args=(i,)) for i in range(2)]
        for w in work:
            w.start()
        for w in work:
            w.join()
    else:
        for a, b in zip(*imgs):
            bp.enqueue(sinos[0], a, n, streams[0])
            bp.enqueue(sinos[1], b, n, streams[1])
    bp.check()
    for i in range(2):
        for img in imgs[i]:
            np.testing.assert_array_equal(img.cpu().numpy(), alone[i])


@pytest.mark.parametrize("batch", [1, 4])
def test_engine_beside_its_own_handle(batch):
    """An engine's runs and replays on one stream, direct calls of its backprojection on another."""
    d = dict(SMALL, n_par_proj=128, n_par_det=256, n_pixels=256)
    sc = phantom.make_scan(batch, 1, 500, 432, 215.0, 240.0, seed=3, distinct=batch)
    p = rg.make_params(masking=True)
    fbp = rg.FBP(geom(d), p, sc.ref, 1, sc.dark, 1, max_batch=batch)
    bp = fbp.backprojection()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    raw = torch.from_numpy(sc.raw.view(np.int16)).cuda()
    img, img2 = _images(batch, 256), _images(batch, 256)
    sino = _sino(batch, 128, 256, 9)
    torch.cuda.synchronize()
    graph = fbp.graph_capture(raw, img, 0, batch, a)
    graph.replay(a)
    torch.cuda.synchronize()
    alone = img.cpu().numpy()
    alone2 = _run(bp, sino, 256)
    for _ in range(20):
        img.fill_(float("nan"))
        img2.fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay(a)
        bp.enqueue(sino, img2, batch, b)
        fbp.enqueue(raw, img, 0, batch, a)
        bp.enqueue(sino, img2, batch, b)
        bp.check()
        np.testing.assert_array_equal(img.cpu().numpy(), alone)
        np.testing.assert_array_equal(img2.cpu().numpy(), alone2)


@pytest.mark.parametrize("rot", [0.0, 21.0])
@pytest.mark.parametrize("reserved,n,cuts", [(2, 2, [1]), (5, 5, [1, 2, 4]), (40, 40, [1, 2, 4, 5, 17])])
def test_cuts_of_a_reserved_handle(reserved, n, cuts, rot):
    """A linear handle reserved for a job's largest batch gives the same bits however the job is cut."""
    Pp, Dp, N = 60, 96, 90
    bp = _handle(Pp, Dp, N, rot)
    bp.reserve(reserved)
    sino = _sino(n, Pp, Dp, n)
    whole = _run(bp, sino, N)
    for m in cuts:
        for first in sorted({0, (n - m) // 2, n - m}):
            np.testing.assert_array_equal(_run(bp, sino[first:first + m].contiguous(), N), whole[first:first + m])


@pytest.mark.parametrize("rot", [0.0, 21.0])
def test_batches_of_an_unreserved_handle(rot):
    """Two, four, five and more slices take different kernels without a reservation."""
    Pp, Dp, N = 60, 96, 90
    bp = _handle(Pp, Dp, N, rot)
    sino = _sino(9, Pp, Dp, 3)
    exp = [oracle.mask(oracle.backproject(s, N, rot), 0.0) for s in sino.cpu().numpy()]
    for n in (1, 2, 3, 4, 5, 9):
        got = _run(bp, sino[:n].contiguous(), N)
        np.testing.assert_array_equal(_run(bp, sino[:n].contiguous(), N), got)
        for b in range(n):
            mr, _ = rel_err(got[b], exp[b])
            assert mr < MAX_REL, (n, b, mr)


@pytest.mark.parametrize("n", [1, 4])
def test_default_and_other_streams_in_turn(n):
    """The legacy stream, whose use is recorded only when another stream follows, and two others."""
    Pp, Dp, N = 180, 256, 256
    bp = _handle(Pp, Dp, N)
    streams = [None, torch.cuda.Stream(), torch.cuda.Stream()]
    sinos = [_sino(n, Pp, Dp, seed) for seed in range(3)]
    alone = [_run(bp, s, N) for s in sinos]
    order = [0, 1, 0, 0, 2, 1, 1, 0, 2, 2, 0, 1] * 3
    imgs = [_images(n, N) for _ in order]
    torch.cuda.synchronize()
    for i, img in zip(order, imgs):
        bp.enqueue(sinos[i], img, n, streams[i])
    bp.check()
    for i, img in zip(order, imgs):
        np.testing.assert_array_equal(img.cpu().numpy(), alone[i])
