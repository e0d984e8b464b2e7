"""Performance cases of the reconstruction chain, from one frame to a streaming job.

Every case goes through the package's public classes as a program would: handles,
tables, buffers and captured graphs are made once by prepare(), run() makes the
calls of one pass. Inputs are synthetic and seeded: ellipse phantoms, Poisson
uint16 counts (I0 = 40000, dark level 200), about 1% defective detector columns.
exact() restates each path in 64-bit torch arithmetic.

Kinds of case
  engine     raw frames -> images by the batched engine (enqueue, or the replay of a
             captured graph), backprojection kernel as created or autotuned in set-up
  host       raw frames in pinned host memory -> images in pinned host memory
  stages     one call per stage, as a pipeline of stage objects makes them
  parallel   filtering and backprojection of parallel-beam sinograms
  toeplitz   the tensor-core form of the filter
  gradient   parallel sinograms: forward map and gradients of sinograms and taps
  fan_gradient  the same from fan sinograms, with the rebinning and its transpose
  sweep      many reconstructions of different shapes in one launch
"""
from __future__ import annotations

import math

import numpy as np
import torch

import risa_gb300 as rg

I0, DARK = 40000.0, 200.0
PLANES = rg.PLANES_INTERLEAVED
RING = dict(source_offset=0.0, detector_diameter=480.0, image_width=200.0, source_diameter=[430.0] * 4,
            delta_x=[0.0] * 4, delta_z=[1417.0, 1430.0, 1417.0, 1430.0], source_angle=[360.0] * 4)
# two tilted planes with a limited source arc: the scanner of the example configuration file
ROFEX = dict(source_offset=23.2, detector_diameter=216.0, image_width=190.0, source_diameter=[365.0, 370.0] * 2,
             delta_x=[815.0] * 4, delta_z=[1417.0, 1430.0] * 2, source_angle=[240.0] * 4)
ROFEX_FIX = dict(lower_lim_offset=47.0, upper_lim_offset=313.0, fix_points=(43, 285, 175, 362, 0, 431))


def listed():
    return [
        # full-rate streaming: one chunk of a two-plane scan replayed as a graph, the kernel tuned at set-up
        _scan("stream_chunk_512", planes=2, det=1152, proj=1000, angles=1024, rays=1024, pixels=512, frames=512,
              filter="sheppLogan", defects=True, masking=True, tune=True, graph=True),
        # the same scan while it is watched live: one frame of each plane per call
        _scan("stream_pair", planes=2, det=1152, proj=1000, angles=1024, rays=1024, pixels=512, frames=2,
              filter="sheppLogan", defects=True, masking=True),
        # the batched pipeline program: host frames in, host images out
        _scan("host_job_128", kind="host", planes=2, det=1152, proj=1000, angles=1024, rays=1024, pixels=512,
              frames=128, chunk=64, filter="sheppLogan", defects=True, masking=True),
        # small single-plane scan, all its frames in one call
        _scan("plain_small_64", planes=1, det=432, proj=500, angles=256, rays=256, pixels=256, frames=64),
        # the example configuration file through the pipeline's stages, one frame per call
        _scan("rofex_stage_frame", kind="stages", quirks=1, planes=2, det=432, proj=500, angles=512, rays=256,
              pixels=256, frames=1, filter="sheppLogan", defects=True, masking=True, normalize=True, relevant=True),
        # the same configuration through the engine, frames module by module as the loader reads them
        _scan("rofex_engine_30", quirks=1, planes=2, det=432, proj=500, angles=512, rays=256, pixels=256, frames=30,
              filter="sheppLogan", defects=True, masking=True, relevant=True, modules=27),
        # parallel-beam data at high resolution: filter and backprojection of a stack of slices
        _parallel("parallel_1024_16", slices=16, angles=1024, rays=1024, pixels=1024, filter="ramp"),
        # one odd-sized parallel slice, nearest-neighbour backprojection, normalised and masked
        _parallel("parallel_nearest_1", slices=1, angles=361, rays=301, pixels=231, filter="hamming", interp=1,
                  masking=True, normalize=True),
        # the filter as a tensor-core contraction, 22-bit operands
        dict(name="toeplitz_f16_64", kind="toeplitz", slices=64, angles=1024, rays=1024, filter="ramp", split=1),
        # learning a filter: forward map, gradients of the sinograms and of 1024 taps
        dict(name="gradient_512_16", kind="gradient", slices=16, angles=720, rays=768, pixels=512, taps=1024),
        # the same from fan sinograms of the small scan, a few slices at a time
        dict(name="fan_gradient_4", kind="fan_gradient", slices=4, det=432, proj=500, angles=256, rays=256,
             pixels=256, taps=129),
        # uneven sweep: image sides, angles and filters drawn per instance
        dict(name="sweep_64", kind="sweep", instances=64, side_min=128, side_max=1024, angles_min=180,
             angles_max=1440, shapes=5),
    ]


def _scan(name=None, **kw):
    c = dict(kind="engine", quirks=0, planes=1, det=432, proj=500, angles=256, rays=256, pixels=256, frames=1, chunk=0,
             filter="ramp", interp=0, defects=False, masking=False, normalize=False, relevant=False, modules=0,
             tune=False, graph=False)
    c.update(kw)
    return dict(name=name, **c) if name else c


def _parallel(name=None, **kw):
    c = dict(kind="parallel", slices=1, angles=256, rays=256, pixels=256, filter="ramp", interp=0, masking=False,
             normalize=False)
    c.update(kw)
    return dict(name=name, **c) if name else c


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["engine", "engine", "engine", "host", "stages", "parallel", "parallel", "toeplitz", "gradient",
                       "fan_gradient", "sweep"])
    filt = rng.choice(["ramp", "sheppLogan", "cosine", "hamming", "hanning"])
    if kind in ("engine", "host", "stages"):
        pixels = _log_int(rng, 96, 512)
        rays = 2 * max(32, int(round(pixels * rng.uniform(0.5, 1.0))))
        rofex = rng.random() < 0.3
        if rofex:
            rays = 1 << max(6, min(9, rays.bit_length() - 1))
        wide = not rofex and rng.random() < 0.5
        planes = 2 if rofex else rng.choice([1, 1, 2])
        frames = 1 if kind == "stages" else planes * _log_int(rng, 1, 96)
        angles = int(rays * rng.uniform(0.7, 1.3))
        return _scan(kind=kind, quirks=1 if rofex else 0, planes=planes, det=1152 if wide else 432,
                     proj=rng.choice([1000, 720]) if wide else 500, angles=angles, rays=rays, pixels=pixels,
                     frames=frames, chunk=planes * max(1, frames // planes // rng.choice([1, 2, 4])) if kind == "host"
                     else 0, filter=filt, interp=rng.choice([0, 0, 0, 0, 1, 2]), defects=rng.random() < 0.7,
                     masking=rng.random() < 0.7, normalize=rng.random() < 0.2, relevant=rofex,
                     modules=rng.choice([0, 0, 27]) if not wide and kind == "engine" else 0,
                     tune=kind == "engine" and rng.random() < 0.4, graph=kind == "engine" and rng.random() < 0.4)
    if kind == "parallel":
        pixels = _log_int(rng, 100, 1024)
        rays = max(64, int(pixels * rng.uniform(0.8, 1.5)))
        return _parallel(slices=_log_int(rng, 1, 16), angles=_log_int(rng, 90, 1440), rays=rays, pixels=pixels,
                         filter=filt, interp=rng.choice([0, 0, 0, 1, 2]), masking=rng.random() < 0.5,
                         normalize=rng.random() < 0.2)
    if kind == "toeplitz":
        return dict(kind="toeplitz", slices=_log_int(rng, 1, 64), angles=_log_int(rng, 90, 1024),
                    rays=128 * rng.randint(1, 8), filter=filt, split=rng.choice([0, 1]))
    if kind == "gradient":
        pixels = _log_int(rng, 96, 512)
        return dict(kind="gradient", slices=_log_int(rng, 1, 16), angles=_log_int(rng, 90, 720),
                    rays=int(pixels * rng.uniform(1.0, 1.5)), pixels=pixels, taps=_log_int(rng, 31, 1024))
    if kind == "fan_gradient":
        pixels = _log_int(rng, 64, 256)
        return dict(kind="fan_gradient", slices=_log_int(rng, 1, 8), det=432, proj=500,
                    angles=_log_int(rng, 64, 256), rays=2 * _log_int(rng, 32, 128), pixels=pixels,
                    taps=_log_int(rng, 31, 257))
    return dict(kind="sweep", instances=_log_int(rng, 4, 64), side_min=rng.randint(120, 192),
                side_max=rng.randint(256, 1024), angles_min=rng.randint(90, 180), angles_max=rng.randint(360, 1440),
                shapes=rng.randint(0, 10 ** 6))


# --------------------------------------------------------------------------- geometry, parameters
def _scan_geom(c):
    return rg.make_geometry(n_planes=c["planes"], n_fan_det=c["det"], n_fan_proj=c["proj"], n_par_proj=c["angles"],
                            n_par_det=c["rays"], n_pixels=c["pixels"], n_modules=27 if c["det"] % 27 == 0 else 1,
                            **(ROFEX if c["quirks"] else RING))


def _scan_params(c):
    return rg.make_params(quirks=c["quirks"], filter_type=c["filter"], interp=c["interp"], defects=c["defects"],
                          masking=c["masking"], masking_value=0.0, normalize=c["normalize"],
                          relevant_mask=c["relevant"], module_major=bool(c["modules"]),
                          **(ROFEX_FIX if c["relevant"] else {}))


def _par_geom(c):
    return rg.make_geometry(n_par_proj=c["angles"], n_par_det=c["rays"], n_pixels=c["pixels"] if "pixels" in c else 64)


# --------------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _ellipses(seed, n, fov, how_many=8):
    """[n][how_many] ellipses (cx, cy, a, b, phi, mu) inside the field of view, as tensors [n, how_many, 1, 1]."""
    rng = np.random.default_rng(int(seed) * 104729 + 7)
    s = fov / 200.0
    ax = rng.uniform(5.0 * s, 60.0 * s, (n, how_many, 2))
    r = np.maximum(fov / 2.0 - ax.max(-1), 0.0) * np.sqrt(rng.uniform(size=(n, how_many)))
    ang = rng.uniform(0, 2 * np.pi, (n, how_many))
    phi, mu = rng.uniform(0, np.pi, (n, how_many)), rng.uniform(0.005, 0.05, (n, how_many))
    cols = (r * np.cos(ang), r * np.sin(ang), ax[..., 0], ax[..., 1], phi, mu)
    return [torch.from_numpy(np.ascontiguousarray(v, dtype=np.float32)).cuda()[..., None, None] for v in cols]


def _fan_integrals(el, c, geo):
    """Line integrals [n, proj, det] from every source position to every detector."""
    cx, cy, a, b, phi, mu = el
    proj, det = c["proj"], c["det"]
    th = torch.deg2rad(torch.arange(proj, device="cuda") * (360.0 / proj) - geo["source_offset"])[:, None]
    ga = torch.deg2rad(torch.arange(det, device="cuda") * (360.0 / det))[None, :] + math.pi / 2
    rs, rd = geo["source_diameter"][0] / 2, geo["detector_diameter"] / 2
    sx, sy, ex, ey = rs * torch.cos(th), rs * torch.sin(th), rd * torch.cos(ga), rd * torch.sin(ga)
    dx, dy = ex - sx, ey - sy
    length = torch.sqrt(dx * dx + dy * dy)
    out = torch.zeros(cx.shape[0], proj, det, device="cuda")
    for e in range(cx.shape[1]):
        co, si = torch.cos(phi[:, e]), torch.sin(phi[:, e])
        qx = ((sx - cx[:, e]) * co + (sy - cy[:, e]) * si) / a[:, e]
        qy = ((sy - cy[:, e]) * co - (sx - cx[:, e]) * si) / b[:, e]
        ux, uy = (dx * co + dy * si) / a[:, e], (dy * co - dx * si) / b[:, e]
        aa, bb, cc = ux * ux + uy * uy, qx * ux + qy * uy, qx * qx + qy * qy - 1
        disc = torch.clamp(bb * bb - aa * cc, min=0).sqrt()
        t0, t1 = ((-bb - disc) / aa).clamp(0, 1), ((-bb + disc) / aa).clamp(0, 1)
        out += (t1 - t0) * length * mu[:, e]
    return out


def _par_integrals(el, angles, rays, width, rows=None):
    """Parallel-beam line integrals [n, angles, rays], bins centred."""
    cx, cy, a, b, phi, mu = el
    th = (torch.arange(angles, device="cuda", dtype=torch.float32) * (math.pi / angles))[:, None]
    s = (torch.arange(rays, device="cuda", dtype=torch.float32)[None, :] + 0.5 - rays / 2.0) * (width / rays)
    out = torch.zeros(cx.shape[0], angles, rays, device="cuda")
    for e in range(cx.shape[1]):
        sp = s - (cx[:, e] * torch.cos(th) + cy[:, e] * torch.sin(th))
        a2 = (a[:, e] * torch.cos(th - phi[:, e])) ** 2 + (b[:, e] * torch.sin(th - phi[:, e])) ** 2
        out += 2 * mu[:, e] * a[:, e] * b[:, e] * torch.clamp(a2 - sp * sp, min=0).sqrt() / a2
    return out


def _counts(li, gen):
    lam = I0 * torch.exp(-li) + DARK
    return torch.poisson(lam, generator=gen).clamp_(max=65535)


def _plant(counts, cols, gen):
    """Every other chosen column dead (reads the dark level), the others flickering by up to half."""
    for i, col in enumerate(cols):
        if i % 2 == 0:
            counts[..., col] = DARK
        else:
            f = 0.5 + torch.rand(counts.shape[:-1], device="cuda", generator=gen)
            counts[..., col] = (counts[..., col] * f).round().clamp(max=65535)
    return counts


def _u16(x):
    """Counts as the 16-bit patterns the library reads (torch int16 storage)."""
    v = x.to(torch.int32)
    return torch.where(v > 32767, v - 65536, v).to(torch.int16)


def _scan_data(c, seed):
    """(frames int16 [n, proj, det] on the GPU, index of each frame's distinct source, reference and dark host frames)."""
    geo = ROFEX if c["quirks"] else RING
    gen = _gen(seed)
    distinct = min(c["frames"], 8 if c["pixels"] >= 256 else 16)
    distinct -= distinct % c["planes"] if distinct > c["planes"] else 0
    distinct = max(1, distinct)
    el = _ellipses(seed, distinct, 0.9 * min(geo["image_width"], geo["detector_diameter"]))
    pool = _counts(_fan_integrals(el, c, geo), gen)
    rng = np.random.default_rng(int(seed) + 31)
    cols = sorted(int(v) for v in rng.choice(c["det"], max(1, c["det"] // 100), replace=False)) if c["defects"] else []
    shape = (c["planes"], c["proj"], c["det"])
    ref = _plant(_counts(torch.zeros(shape, device="cuda"), gen), cols, gen)
    dark = torch.poisson(torch.full(shape, DARK, device="cuda"), generator=gen)
    pool = _u16(_plant(pool, cols, gen))
    host = [np.ascontiguousarray(_u16(v).cpu().numpy().view(np.uint16)) for v in (ref, dark)]
    index = torch.arange(c["frames"], device="cuda") % distinct
    return pool, index, host[0], host[1]


def _module_major(frames, modules):
    n, proj, det = frames.shape
    return frames.view(n, proj, modules, det // modules).transpose(1, 2).contiguous().view(n, proj, det)


def _sinograms(c, seed, distinct=8):
    n = min(c["slices"], distinct)
    pool = _par_integrals(_ellipses(seed, n, 200.0), c["angles"], c["rays"], 200.0)
    return pool[torch.arange(c["slices"], device="cuda") % n].contiguous()


def _taps(c, seed):
    """A spatial ramp with a small random perturbation, as a filter under training has it."""
    n = c["taps"]
    k = np.arange(n) - n // 2
    h = np.where(k % 2 != 0, -1.0 / (np.pi * np.where(k == 0, 1, k)) ** 2, 0.0)
    h[k == 0] = 0.25
    rng = np.random.default_rng(int(seed) + 5)
    return (h + 0.05 * rng.standard_normal(n) / n).astype(np.float32)


def _sweep_instances(c, seed):
    """Shapes from the case (a user's list of jobs), defect columns from the seed."""
    rng = np.random.default_rng(c["shapes"])
    pick = np.random.default_rng(int(seed) + 77)
    out = []
    for _ in range(c["instances"]):
        side = int(round(math.exp(rng.uniform(math.log(c["side_min"]), math.log(c["side_max"])))))
        angles = int(rng.integers(c["angles_min"], c["angles_max"] + 1))
        rays = max(32, 32 * int(round(1.25 * side / 32.0)))
        dmap = np.zeros(rays, np.uint8)
        dmap[pick.choice(rays, int(round(pick.uniform(0.0, 0.02) * rays)), replace=False)] = 1
        out.append(dict(n_pixels=side, n_par_proj=angles, n_par_det=rays, cutoff=1.0, rotation_offset=0.0,
                        filter_type="ramp" if rng.uniform() < 0.5 else "hanning", ref_level=I0 + DARK,
                        dark_level=DARK, masking=True, masking_value=0.0, defect_map=dmap))
    return out


def _sweep_raw(inst, seed):
    gen, raws = _gen(seed), []
    els = _ellipses(seed, len(inst), 200.0)
    for i, d in enumerate(inst):
        li = _par_integrals([v[i:i + 1] for v in els], d["n_par_proj"], d["n_par_det"], 200.0)[0]
        raws.append(_u16(_plant(_counts(li, gen), np.flatnonzero(d["defect_map"]).tolist(), gen)).reshape(-1))
    return raws


# --------------------------------------------------------------------------- prepare
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


_streams = []


def _work_stream():
    """The one stream on which the program replays its graphs."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def _engine(c, ref, dark, batch):
    return rg.FBP(_scan_geom(c), _scan_params(c), ref, 1, dark, 1, max_batch=batch)


def _prepare_engine(c, seed):
    pool, index, ref, dark = _scan_data(c, seed)
    if c["modules"]:
        pool = _module_major(pool, c["modules"])
    raw = pool[index].contiguous()
    n, N = c["frames"], c["pixels"]
    fbp = _engine(c, ref, dark, n)
    img = torch.empty((n, N, N), device="cuda")
    st = dict(case=c, fbp=fbp, raw=raw, img=img)
    torch.cuda.synchronize()
    if c["tune"] and c["interp"] == 0:
        some = min(n, 64) // c["planes"] * c["planes"]
        fbp.enqueue(raw, img, PLANES, some)
        fbp.backprojection().autotune(fbp.intermediates()[1], img, some)
    if c["graph"]:
        st["stream"] = _work_stream()
        st["graph"] = fbp.graph_capture(raw, img, PLANES, n, st["stream"])
    return st


def _prepare_host(c, seed):
    pool, index, ref, dark = _scan_data(c, seed)
    n, N = c["frames"], c["pixels"]
    raw = torch.empty((n, c["proj"], c["det"]), dtype=torch.int16, pin_memory=True)
    raw.copy_(pool[index])
    img = torch.empty((n, N, N), pin_memory=True)
    return dict(case=c, fbp=_engine(c, ref, dark, c["chunk"]), raw=raw, img=img)


def _prepare_stages(c, seed):
    pool, _, ref, dark = _scan_data(c, seed)
    g, p = _scan_geom(c), _scan_params(c)
    N = c["pixels"]
    st = dict(case=c, raw=pool[:1].clone(), frame=torch.empty_like(pool[:1]),
              att=rg.Attenuation(g, p, ref, 1, dark, 1), f2p=rg.Fan2Para(g, p), filt=rg.Filter(g, p),
              bp=rg.Backprojection(g, p), mask=rg.Masking(g, p), img=torch.empty((1, N, N), device="cuda"),
              fan=torch.empty((1, c["proj"], c["det"]), device="cuda"),
              par=torch.empty((1, c["angles"], c["rays"]), device="cuda"))
    st["mask_ws"] = torch.empty(st["mask"].workspace_bytes(1), dtype=torch.uint8, device="cuda")
    if c["defects"]:
        st["defects"] = rg.Defects(g, p, max_batch=1)
        st["ws"] = torch.empty(st["defects"].workspace_bytes(1), dtype=torch.uint8, device="cuda")
        st["flags"] = torch.empty((1, c["det"]), dtype=torch.int32, device="cuda")
    return st


def _prepare_parallel(c, seed):
    g = _par_geom(c)
    p = rg.make_params(filter_type=c["filter"], interp=c["interp"], masking=c["masking"], normalize=c["normalize"])
    n, N = c["slices"], c["pixels"]
    st = dict(case=c, sino=_sinograms(c, seed), filt=rg.Filter(g, p), bp=rg.Backprojection(g, p),
              mask=rg.Masking(g, p), img=torch.empty((n, N, N), device="cuda"))
    st["work"] = torch.empty_like(st["sino"])
    st["mask_ws"] = torch.empty(st["mask"].workspace_bytes(n), dtype=torch.uint8, device="cuda")
    if c["interp"] == 0:
        st["bp"].reserve(n)
    return st


def _prepare_toeplitz(c, seed):
    g, p = _par_geom(c), rg.make_params(filter_type=c["filter"])
    st = dict(case=c, sino=_sinograms(c, seed), tz=rg.Toeplitz(g, p))
    st["tz"].set_precision(c["split"])
    st["work"] = torch.empty_like(st["sino"])
    st["ws"] = torch.empty(st["tz"].workspace_bytes(c["slices"]), dtype=torch.uint8, device="cuda")
    return st


def _prepare_gradient(c, seed):
    g, p = _par_geom(c), rg.make_params()
    n, N = c["slices"], c["pixels"]
    st = dict(case=c, sino=_sinograms(c, seed), filt=rg.Filter(g, p, taps=_taps(c, seed)), bp=rg.Backprojection(g, p),
              target=0.02 * torch.rand((n, N, N), device="cuda", generator=_gen(seed)),
              img=torch.empty((n, N, N), device="cuda"), dtaps=torch.empty(c["taps"], device="cuda"))
    st["q"], st["dq"], st["dsino"] = (torch.empty_like(st["sino"]) for _ in range(3))
    st["ws"] = torch.empty(st["filt"].taps_grad_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    st["bp"].reserve(n)
    st["bp"].reserve_adjoint(n)
    return st


def _prepare_fan_gradient(c, seed):
    g = rg.make_geometry(n_fan_det=c["det"], n_fan_proj=c["proj"], n_par_proj=c["angles"], n_par_det=c["rays"],
                         n_pixels=c["pixels"], **RING)
    p = rg.make_params()
    n, N = c["slices"], c["pixels"]
    el = _ellipses(seed, n, 180.0)
    st = dict(case=c, fan=_fan_integrals(el, c, RING), f2p=rg.Fan2Para(g, p), bp=rg.Backprojection(g, p),
              filt=rg.Filter(g, p, taps=_taps(c, seed)), img=torch.empty((n, N, N), device="cuda"),
              target=0.02 * torch.rand((n, N, N), device="cuda", generator=_gen(seed)),
              dtaps=torch.empty(c["taps"], device="cuda"))
    st["dfan"] = torch.empty_like(st["fan"])
    st["par"], st["q"], st["dq"] = (torch.empty((n, c["angles"], c["rays"]), device="cuda") for _ in range(3))
    st["ws"] = torch.empty(st["filt"].taps_grad_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    st["bp"].reserve_adjoint(n)
    return st


def _prepare_sweep(c, seed):
    inst = _sweep_instances(c, seed)
    sweep = rg.Sweep(inst)
    _, _, _, total = sweep.layout()
    return dict(case=c, sweep=sweep, raw=torch.cat(_sweep_raw(inst, seed)), img=torch.empty(total, device="cuda"))


# --------------------------------------------------------------------------- run
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def _run_engine(st):
    if "graph" in st:
        st["graph"].replay(st["stream"])
    else:
        st["fbp"].enqueue(st["raw"], st["img"], PLANES, st["case"]["frames"])
    return st["img"]


def _run_host(st):
    st["fbp"].run_host(st["raw"], st["img"], st["case"]["frames"], PLANES)
    return st["img"]


def _run_stages(st):
    st["frame"].copy_(st["raw"])
    out = {}
    if "defects" in st:
        st["defects"].enqueue(st["frame"], 1, st["ws"], st["flags"])
        out = dict(frame=st["frame"], flags=st["flags"])
    st["att"].enqueue(st["frame"], st["fan"], 0, 1)
    st["f2p"].enqueue(st["fan"], st["par"], 0, 1)
    st["filt"].enqueue(st["par"], 1)
    st["bp"].enqueue(st["par"], st["img"], 1)
    if st["case"]["normalize"]:
        st["mask"].enqueue(st["img"], 1, st["mask_ws"])
    return dict(out, image=st["img"])


def _run_parallel(st):
    n = st["case"]["slices"]
    st["work"].copy_(st["sino"])
    st["filt"].enqueue(st["work"], n)
    st["bp"].enqueue(st["work"], st["img"], n)
    if st["case"]["normalize"]:
        st["mask"].enqueue(st["img"], n, st["mask_ws"])
    return dict(filtered=st["work"], image=st["img"])


def _run_toeplitz(st):
    st["work"].copy_(st["sino"])
    st["tz"].enqueue(st["work"], st["case"]["slices"], st["ws"])
    return st["work"]


def _run_gradient(st):
    """Image and the gradients of |image - target|^2 / 2 with respect to sinograms and taps."""
    n = st["case"]["slices"]
    st["q"].copy_(st["sino"])
    st["filt"].enqueue(st["q"], n)
    st["bp"].enqueue(st["q"], st["img"], n)
    res = st["img"] - st["target"]
    st["bp"].enqueue_adjoint(res, st["dq"], n)
    st["filt"].taps_grad(st["sino"], st["dq"], st["dtaps"], n, st["ws"])
    st["dsino"].copy_(st["dq"])
    st["filt"].enqueue_adjoint(st["dsino"], n)
    return dict(image=st["img"], sinogram=st["dsino"], taps=st["dtaps"])


def _run_fan_gradient(st):
    n = st["case"]["slices"]
    st["f2p"].enqueue(st["fan"], st["par"], 0, n)
    st["q"].copy_(st["par"])
    st["filt"].enqueue(st["q"], n)
    st["bp"].enqueue(st["q"], st["img"], n)
    res = st["img"] - st["target"]
    st["bp"].enqueue_adjoint(res, st["dq"], n)
    st["filt"].taps_grad(st["par"], st["dq"], st["dtaps"], n, st["ws"])
    st["filt"].enqueue_adjoint(st["dq"], n)
    st["f2p"].enqueue_adjoint(st["dq"], st["dfan"], 0, n)
    return dict(image=st["img"], fan=st["dfan"], taps=st["dtaps"])


def _run_sweep(st):
    st["sweep"].enqueue(st["raw"], st["img"])
    return st["img"]


# --------------------------------------------------------------------------- work
def work(case):
    """Inputs read once, outputs written once; 6 operations per pixel x angle update
    (ray coordinate, weight, interpolation, accumulation), 5 n log2 n per transform."""
    c, k = case, case["kind"]

    def image_flops(n, pixels, angles, masked):
        return 6.0 * n * pixels * pixels * (math.pi / 4 if masked else 1.0) * angles

    def filter_flops(rows, rays, pad=None):
        ln = pad or 2 * rays
        return rows * 2 * 2.5 * ln * math.log2(ln)

    if k in ("engine", "host", "stages"):
        n, px = c["frames"], c["proj"] * c["det"]
        rows = n * c["angles"]
        return {"bytes": n * (2.0 * px + 4.0 * c["pixels"] ** 2),
                "flops": 4.0 * n * px + 12.0 * rows * c["rays"] + filter_flops(rows, c["rays"])
                + image_flops(n, c["pixels"], c["angles"], c["masking"])}
    if k == "parallel":
        n, rows = c["slices"], c["slices"] * c["angles"]
        return {"bytes": 8.0 * rows * c["rays"] + 4.0 * n * c["pixels"] ** 2,
                "flops": filter_flops(rows, c["rays"]) + image_flops(n, c["pixels"], c["angles"], c["masking"])}
    if k == "toeplitz":
        rows = c["slices"] * c["angles"]
        return {"bytes": 8.0 * rows * c["rays"], "flops": 2.0 * rows * c["rays"] ** 2}
    if k == "gradient":
        n, rows, img = c["slices"], c["slices"] * c["angles"], c["slices"] * c["pixels"] ** 2
        return {"bytes": 8.0 * rows * c["rays"] + 8.0 * img + 8.0 * c["taps"],
                "flops": 4 * filter_flops(rows, c["rays"]) + 2 * image_flops(n, c["pixels"], c["angles"], False)}
    if k == "fan_gradient":
        n, rows, img = c["slices"], c["slices"] * c["angles"], c["slices"] * c["pixels"] ** 2
        return {"bytes": 8.0 * n * c["proj"] * c["det"] + 8.0 * img,
                "flops": 4 * filter_flops(rows, c["rays"]) + 24.0 * rows * c["rays"]
                + 2 * image_flops(n, c["pixels"], c["angles"], False)}
    b = f = 0.0
    for d in _sweep_instances(c, 0):
        b += 2.0 * d["n_par_proj"] * d["n_par_det"] + 4.0 * d["n_pixels"] ** 2
        f += filter_flops(d["n_par_proj"], d["n_par_det"]) + image_flops(1, d["n_pixels"], d["n_par_proj"], True)
    return {"bytes": b, "flops": f}


# --------------------------------------------------------------------------- exact, in 64 bits
F64 = dict(dtype=torch.float64, device="cuda")


def _response(length, name):
    """Window-designed response at 0 .. length/2, over the transform's length."""
    i = torch.arange(length // 2 + 1, **F64)
    w, f = 2 * math.pi * i / length, 2 * i / length
    if name == "hamming":
        f = f * (0.54 + 0.46 * torch.cos(w))
    elif name == "hanning":
        f = f * (1 + torch.cos(w)) / 2
    elif name == "cosine":
        f = f * torch.cos(w / 2)
    elif name == "sheppLogan":
        f = f * torch.where(i > 0, torch.sin(w / 2) / torch.where(i > 0, w / 2, torch.ones_like(w)),
                            torch.ones_like(w))
    return f


def _filtered(x, name):
    rays = x.shape[-1]
    length = 1
    while length < 2 * rays:
        length *= 2
    length = max(32, length)
    h = _response(length, name)
    return torch.stack([torch.fft.irfft(torch.fft.rfft(s.double(), length) * h, length)[..., :rays] for s in x])


def _convolved(x, taps, adjoint=False):
    """Linear convolution (or correlation) with centred taps, rows on the last axis."""
    t = torch.from_numpy(taps.astype(np.float64)).cuda()
    if adjoint:
        t = t.flip(0)
    n, rays = t.numel(), x.shape[-1]
    at = (n - 1 - n // 2) if adjoint else n // 2
    ln = rays + n
    ht = torch.fft.rfft(t, ln)
    return torch.stack([torch.fft.irfft(torch.fft.rfft(s.double(), ln) * ht, ln)[..., at:at + rays] for s in x])


def _coords(angles, rays, N, i):
    """Bin coordinate of every pixel for angle i (bin k centred at k)."""
    th, scale = i * math.pi / angles, rays / N
    u = torch.arange(N, **F64) - (N - 1) / 2
    return scale * (u[None, :] * math.cos(th) + u[:, None] * math.sin(th)) + rays / 2 - 0.5


def _backprojected(q, N, interp=0):
    n, angles, rays = q.shape
    out = torch.zeros(n, N * N, **F64)
    pad = torch.nn.functional.pad(q.double(), (2, 2))
    for i in range(angles):
        t = _coords(angles, rays, N, i).reshape(-1)
        row = pad[:, i]
        if interp == 0:
            k = torch.floor(t)
            f = t - k
            k = (k.long() + 2).clamp(0, rays + 2)
            out += row[:, k] * (1 - f) + row[:, (k + 1)] * f
        else:  # 1: the nearest bin; 2: truncated toward zero, as the reference's texture variant
            k = (torch.floor(t + 0.5) if interp == 1 else torch.trunc(t + 0.5)).long() + 2
            out += row[:, k.clamp(0, rays + 3)]
    return (out * (math.pi / angles / (rays / N))).reshape(n, N, N)


def _projected(img, angles, rays):
    """The transpose of the linear backprojection: segment sums over pixels sorted by bin."""
    n, N = img.shape[0], img.shape[-1]
    flat = img.double().reshape(n, -1)
    out = torch.zeros(n, angles, rays + 4, **F64)
    bins = torch.arange(rays + 4, device="cuda")
    for i in range(angles):
        t = _coords(angles, rays, N, i).reshape(-1)
        k, order = torch.sort((torch.floor(t).long() + 2).clamp(0, rays + 2))
        f = (t - torch.floor(t))[order]
        v = flat[:, order]
        end = torch.searchsorted(k, bins, right=True)
        for w, shift in ((v * (1 - f), 0), (v * f, 1)):
            cs = torch.nn.functional.pad(torch.cumsum(w, 1), (1, 0))[:, end]
            seg = torch.diff(cs, dim=1, prepend=torch.zeros(n, 1, **F64))
            out[:, i, shift:] += seg[:, :rays + 4 - shift]
    return out[..., 2:rays + 2] * (math.pi / angles / (rays / N))


def _masked(img, normalize, masking, value=0.0):
    N = img.shape[-1]
    if normalize:
        lo, hi = img.amin((1, 2), keepdim=True), img.amax((1, 2), keepdim=True)
        img = (img - lo) / (hi - lo)
    if masking:
        u = torch.arange(N, **F64) - (N - 1) / 2
        img = torch.where(u[:, None] ** 2 + u[None, :] ** 2 > N * N / 4, torch.full_like(img, value), img)
    return img


def _locate(a, origin, n):
    p = (a + origin) / (2 * math.pi / n)
    p = p - n * torch.floor(p / n)
    b = torch.floor(p)
    return b.long() % n, (b.long() + 1) % n, p - b


def _rebin_plan(c):
    """Per sample of the folded sinogram: the two rays of the sample and of its mirrored partner."""
    angles, rays, proj, det = c["angles"], c["rays"], c["proj"], c["det"]
    rs, rd, wid = RING["source_diameter"][0] / 2, RING["detector_diameter"] / 2, RING["image_width"]
    plan = []
    for half in range(2):
        j = torch.arange(angles, **F64)[:, None] + half * angles
        i = torch.arange(rays, **F64)[None, :]
        i = i if half == 0 else rays - 1 - i
        al = (j * (math.pi / angles) + math.pi / 2) % (2 * math.pi)
        s = -0.5 * wid + (i + 0.5) * wid / rays
        at, ed = torch.asin(s / rs), torch.asin(s / rd)
        for th, ga in ((al - at, ed + al - 1.5 * math.pi), (al + at - math.pi, -ed + al - 0.5 * math.pi)):
            plan.append(_locate(th, 0.0, proj) + _locate(ga, 0.0, det))
    return plan


def _rebinned(fan, plan):
    out = 0
    for tb, ta, u, gb, ga, v in plan:
        out = out + 0.25 * ((1 - u) * ((1 - v) * fan[:, tb, gb] + v * fan[:, tb, ga])
                            + u * ((1 - v) * fan[:, ta, gb] + v * fan[:, ta, ga]))
    return out


def _rebinned_back(par, plan, shape):
    out = torch.zeros(shape[0], shape[1] * shape[2], **F64)
    flat = par.reshape(shape[0], -1)
    for tb, ta, u, gb, ga, v in plan:
        for r, d, w in ((tb, gb, (1 - u) * (1 - v)), (tb, ga, (1 - u) * v), (ta, gb, u * (1 - v)), (ta, ga, u * v)):
            out.index_add_(1, (r * shape[2] + d).reshape(-1), 0.25 * w.reshape(1, -1) * flat)
    return out.reshape(shape)


_SMOOTH = np.array([0.5, 1.0, 1.0, 1.0, 1.5, 2.0, 3.0, 3.5, 2.0]) / 29.0


def _repaired(frames):
    """Frames (uint16 values, int64 [n, P, D]) with their defective columns interpolated."""
    n, P, D = frames.shape
    tv = (frames[:, 1:] - frames[:, :-1]).abs().sum(1)
    rg_ = frames[:, :-1].amax(1) - frames[:, :-1].amin(1)
    var = tv.double() * (rg_ * rg_).double()
    H = D // 2
    halves = var[:, :2 * H].reshape(n, 2, H)
    th = torch.zeros_like(halves)
    for j in range(9):
        th = th + _SMOOTH[j] * torch.roll(halves, j, -1)
        th = th + _SMOOTH[j] * torch.roll(halves, -j, -1)
    flags = torch.zeros(n, D, dtype=torch.bool, device="cuda")
    flags[:, :2 * H] = (halves < 0.67 * th).reshape(n, -1)
    high = torch.zeros_like(flags)
    high[:, :2 * H] = (halves > 1.5 * th).reshape(n, -1)
    for off in range(-2, 3):
        flags |= torch.roll(high, off, -1)
    out = frames.clone()
    for b, fl in enumerate(flags.cpu().numpy()):
        if fl.all():
            continue
        _repair_runs(out[b], frames[b], fl)
    return out


def _repair_runs(out, src, fl):
    D = fl.size
    for d in np.flatnonzero(fl & ~np.roll(fl, 1)):
        ln = 1
        while fl[(d + ln) % D]:
            ln += 1
        left, right = src[:, (d - 1) % D], src[:, (d + ln) % D]
        for m in range(ln):
            w1 = np.float32(m + 1) / np.float32(ln + 1)
            w0 = np.float32(1) - w1
            v = (left.float() * float(w0)) + (right.float() * float(w1))
            out[:, (d + m) % D] = torch.floor(v + 0.5).long()


def _values(x):
    return x.to(torch.int64) & 0xFFFF


def _scan_exact(c, seed):
    """Images of the distinct frames, then one per frame of the case."""
    if c["quirks"]:
        return None  # decided by the reference's own 32-bit index steps
    pool, index, ref, dark = _scan_data(c, seed)
    ref = _repaired(_values(torch.from_numpy(ref.view(np.int16)).cuda())).double()
    dk = _values(torch.from_numpy(dark.view(np.int16)).cuda()).double().mean(1)
    frames = _values(pool)
    if c["defects"]:
        frames = _repaired(frames)
    # frame b of a scan is of plane b % planes, and the distinct frames hold whole plane groups
    plane = torch.arange(frames.shape[0], device="cuda") % c["planes"]
    num = (frames.double() - dk[plane][:, None, :]).clamp(min=1e-5)
    fan = torch.log((ref - dk[:, None, :]).clamp(min=1e-5))[plane] - torch.log(num)
    par = _rebinned(fan, _rebin_plan(c))
    img = _backprojected(_filtered(par, c["filter"]), c["pixels"], c["interp"])
    # the masking stage always masks; the engine's normalisation does so when asked to
    img = _masked(img, c["normalize"], c["masking"] or (c["normalize"] and c["kind"] == "stages"))
    return frames, img, index


def exact(case, seed):
    c, k = case, case["kind"]
    if k in ("engine", "host"):
        got = _scan_exact(c, seed)
        return None if got is None else got[1][got[2]]
    if k == "stages":
        got = _scan_exact(c, seed)
        if got is None:
            return None
        image = got[1][:1]
        return dict(frame=None, flags=None, image=image) if c["defects"] else dict(image=image)
    if k == "parallel":
        q = _filtered(_sinograms(c, seed), c["filter"])
        img = _backprojected(q, c["pixels"], c["interp"])
        return dict(filtered=q, image=_masked(img, c["normalize"], c["masking"] or c["normalize"]))
    if k == "toeplitz":
        return _filtered(_sinograms(c, seed), c["filter"])
    if k in ("gradient", "fan_gradient"):
        return _gradient_exact(c, seed)
    inst = _sweep_instances(c, seed)
    out = []
    for d, raw in zip(inst, _sweep_raw(inst, seed)):
        v = _values(raw).reshape(d["n_par_proj"], d["n_par_det"])
        fixed = v.clone()
        _repair_runs(fixed, v, d["defect_map"].astype(bool))
        att = math.log(I0) - torch.log((fixed.double() - DARK).clamp(min=1e-5))
        img = _backprojected(_filtered(att[None], d["filter_type"]), d["n_pixels"])
        out.append(_masked(img, False, True).reshape(-1))
    return torch.cat(out)


def _gradient_exact(c, seed):
    n, N, taps = c["slices"], c["pixels"], _taps(c, seed)
    target = 0.02 * torch.rand((n, N, N), device="cuda", generator=_gen(seed))
    if c["kind"] == "gradient":
        sino = _sinograms(c, seed).double()
    else:
        plan = _rebin_plan(c)
        fan = _fan_integrals(_ellipses(seed, n, 180.0), c, RING).double()
        sino = _rebinned(fan, plan)
    img = _backprojected(_convolved(sino, taps), N)
    dq = _projected(img - target.double(), c["angles"], c["rays"])
    # taps[j] meets x[m - (j - n_taps // 2)]
    ln = 2 * c["rays"] + c["taps"]
    corr = sum(torch.fft.irfft((torch.fft.rfft(g, ln) * torch.fft.rfft(x, ln).conj()).sum(0), ln)
               for g, x in zip(dq, sino))
    lag = torch.arange(c["taps"], device="cuda") - c["taps"] // 2
    dtaps = torch.where(lag.abs() < c["rays"], corr[lag % ln], torch.zeros_like(corr[lag % ln]))
    dsino = _convolved(dq, taps, adjoint=True)
    if c["kind"] == "gradient":
        return dict(image=img, sinogram=dsino, taps=dtaps)
    return dict(image=img, fan=_rebinned_back(dsino, plan, fan.shape), taps=dtaps)
