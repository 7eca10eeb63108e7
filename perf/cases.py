"""The work this framework is used for, as cases that can be timed.

A case is a dict of plain values. `prepare` makes what a program holds before
the call (a context with the scene uploaded, a film, a network, rays),
`run` makes one pass through the public entry points, `work` says what the
pass cannot do without, `exact` gives the result in 64 bits where it has one.

Kinds:
  render   one frame through tr_render_dev ("dev"), tr_render ("host": the film
           comes back to host memory), tr_render_dev_noalloc ("noalloc") or
           tr_render_guided_dev ("guided"); "post" adds the output path
  batch    many scenes of uneven sizes in one tr_render_batch_dev call
  trace    closest-hit and shadow rays against a triangle soup
  network  the guiding network's forward and backward pass
  train    one optimiser step of the guiding network
"""
import ctypes as C
import math

import numpy as np
import torch

from tracer_gb300 import scenes
from tracer_gb300.abi import TrCamera, TrFilter, TrRenderParams, TrStats, make_guide, make_params
from tracer_gb300.native import GpuContext

DEV = "cuda:0"

# Per scene family: triangles or spheres, path vertices per camera sample,
# lights, and the most camera samples a drawn frame takes (what keeps a drawn
# case below the largest listed one).
FAMILY = {
    "cornell": dict(prims=36, vertices=4.0, lights=2, samples=2.5e6),
    "cornell_mixed": dict(prims=36, vertices=4.0, lights=2, samples=2.5e6),
    "outdoor": dict(prims=8, vertices=3.0, lights=3, samples=4e6),
    "mapped": dict(prims=9, vertices=3.0, lights=3, samples=4e6),
    "disney15": dict(prims=9, vertices=3.0, lights=3, samples=4e6),
    "disney_grid": dict(prims=262, vertices=2.0, lights=4, samples=16e6),
    "room": dict(prims=500_030, vertices=6.0, lights=12, samples=6e6),
}
ROOM_BOX = ((-4.0, 0.0, -3.0), (4.0, 4.0, 3.0))
LAYERS = ((7, 64), (64, 64), (64, 64), (64, 64), (64, 40))


def listed():
    return [
        # the smallest frame an interactive viewer asks for while the camera moves, with the whole output path to 8 bits
        dict(name="preview", kind="render", scene="cornell_mixed", width=61, height=47, spp=1, entry="dev", fp64=False, post=True),
        # a frame loop that shares the GPU with an allocator: no device memory is taken by the call
        dict(name="preview_noalloc", kind="render", scene="cornell", width=125, height=93, spp=2, entry="noalloc", fp64=False, post=False),
        # the configured Cornell box, film back on the host as an offline user has it
        dict(name="cornell", kind="render", scene="cornell", width=256, height=256, spp=16, entry="host", fp64=False, post=False),
        # every material kind and an environment light, a medium frame
        dict(name="outdoor", kind="render", scene="outdoor", width=320, height=180, spp=8, entry="dev", fp64=False, post=False),
        # image maps on every material kind at a large odd film, with the output path
        dict(name="mapped_large", kind="render", scene="mapped", width=1001, height=563, spp=4, entry="dev", fp64=False, post=True),
        # the configured Disney grid (fewer samples)
        dict(name="disney_grid", kind="render", scene="disney_grid", width=1024, height=1024, spp=16, entry="dev", fp64=False, post=False),
        # the configured occluded-light room: the framework's headline
        dict(name="room", kind="render", scene="room", width=1024, height=768, spp=16, entry="dev", fp64=False, post=False),
        # a guided pass of the room as it is accumulated toward convergence: 64-bit film, light table, records kept
        dict(name="room_guided", kind="render", scene="room", width=1024, height=768, spp=8, entry="guided", fp64=True, post=False),
        # batched rendering: scenes of uneven triangle counts, resolutions and samples in one call
        dict(name="batch", kind="batch", scenes=12, min_tris=10_000, max_tris=300_000),
        # the traversal test: a million triangles, closest-hit rays and shadow rays
        dict(name="traversal", kind="trace", tris=1 << 20, rays=1 << 21, host=False),
        # the guiding network on an odd number of path vertices, both directions
        dict(name="network", kind="network", rows=100_003),
        # one Adam step on the configured batch
        dict(name="train", kind="train", rows=65_536),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["small", "medium", "large", "noalloc", "guided", "batch", "trace", "network", "train"])
    if kind == "batch":
        lo = _log(rng, 10_000, 100_000)
        return dict(kind="batch", scenes=rng.randint(2, 12), min_tris=lo, max_tris=_log(rng, lo, 300_000))
    if kind == "trace":
        return dict(kind="trace", tris=_log(rng, 1_000, 1 << 20), rays=_log(rng, 1_000, 1 << 21), host=rng.random() < 0.25)
    if kind in ("network", "train"):
        return dict(kind=kind, rows=_log(rng, 100, 1 << 18))
    aspect = rng.choice([1.0, 4.0 / 3.0, 16.0 / 9.0, 0.75])
    scene = rng.choice([s for s in FAMILY if s != "room"])
    entry = rng.choice(["dev", "dev", "host"])
    post = rng.random() < 0.3 and entry == "dev"
    if kind == "noalloc":
        # films whose scratch fits the static array (324 + 76 bytes a light and pixel), scenes without image maps
        scene = rng.choice(["cornell", "outdoor", "disney15", "disney_grid"])
        pixels, spp, entry, post = _log(rng, 500, 20_000), rng.randint(1, 4), "noalloc", False
    elif kind == "small":
        pixels, spp = _log(rng, 300, 40_000), rng.randint(1, 4)
    elif kind == "medium":
        pixels, spp = _log(rng, 16_384, 131_000), _log(rng, 2, 16)
    else:
        scene = "room" if kind == "guided" else rng.choice(list(FAMILY))
        pixels, spp = _log(rng, 140_000, 1 << 20), _log(rng, 1, 16)
        if kind == "guided":
            entry, post, pixels, spp = "guided", False, min(pixels, 600_000), min(spp, 8)
    spp = max(1, min(spp, int(FAMILY[scene]["samples"] / pixels)))
    width = max(8, int(math.sqrt(pixels * aspect)))
    return dict(kind="render", scene=scene, width=width, height=max(8, pixels // width), spp=spp, entry=entry,
                fp64=entry != "noalloc" and rng.random() < 0.25, post=post)


# ---------------------------------------------------------------- inputs


def _scene(case, seed):
    w, h, s, name = case["width"], case["height"], case["spp"], case["scene"]
    if name == "cornell":
        sc, cam, filt, par = scenes.cornell(w, h, s)
    elif name == "cornell_mixed":
        sc, cam, filt, par = scenes.cornell(w, h, s, glass=True, metal=True, textured=True)
    elif name == "outdoor":
        sc, cam, filt, par = scenes.outdoor(w, h, s)
    elif name == "mapped":
        sc, cam, filt, par = scenes.mapped_materials(w, h, s)
    elif name == "disney15":
        sc, cam, filt, par = scenes.disney15_row(w, h, s)
    elif name == "disney_grid":
        sc, cam, filt, par = scenes.disney_grid(w, h, s, max_depth=8, min_depth=5, seed=seed)
    else:
        sc, cam, filt, par = scenes.occluded_room(w, h, s, max_depth=10, min_depth=3, seed=seed)
    par = make_params(w, h, s, par.min_depth, par.max_depth, seed_base=(seed * 7919) & 0x3FFFFFFF)
    return sc, cam, filt, par


def _rand(seed, *shape, normal=False):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    f = torch.randn if normal else torch.rand
    return f(*shape, generator=g, device=DEV, dtype=torch.float32)


def _vertices(seed, n):
    """Path vertices of the room as the network sees them (position in the
    box, outgoing direction, roughness), the directions their light came
    from (mostly from the slit) and the weights of those samples."""
    x = torch.empty(n, 7, device=DEV)
    x[:, :3] = 2 * _rand(seed, n, 3) - 1
    x[:, 3:6] = torch.nn.functional.normalize(_rand(seed + 1, n, 3, normal=True), dim=1)
    x[:, 6] = 1.0
    half = torch.tensor([4.0, 2.0, 3.0], device=DEV)
    slit = torch.tensor([4.0, 2.0, 0.0], device=DEV) + (_rand(seed + 2, n, 3) - 0.5) * torch.tensor([0.0, 3.0, 0.1], device=DEV)
    pos = x[:, :3] * half + torch.tensor([0.0, 2.0, 0.0], device=DEV)
    d = torch.nn.functional.normalize(slit - pos, dim=1)
    d = torch.nn.functional.normalize(d + 0.3 * _rand(seed + 3, n, 3, normal=True), dim=1)
    w = torch.exp(_rand(seed + 4, n, normal=True))
    return x, d.contiguous(), w


def prepare(case, seed):
    kind = case["kind"]
    ctx = GpuContext(0)
    st = {"kind": kind, "ctx": ctx, "case": case}
    if kind == "render":
        sc, cam, filt, par = _scene(case, seed)
        ctx.upload(sc)
        n = case["width"] * case["height"]
        st.update(cam=cam, filt=filt, par=par, n=n)
        st["film"] = torch.zeros(case["height"], case["width"], 4, dtype=torch.float64 if case["fp64"] else torch.float32, device=DEV)
        if case["post"]:
            st["rgb"] = torch.zeros(n, 3, device=DEV)
            st["rgb8"] = torch.zeros(n, 3, dtype=torch.uint8, device=DEV)
            st["rgbe"] = torch.zeros(n, 4, dtype=torch.uint8, device=DEV)
        if case["entry"] == "noalloc":
            f = ctx.L.tr_render_dev_noalloc
            f.restype = C.c_int
            f.argtypes = [C.c_void_p, C.POINTER(TrCamera), C.POINTER(TrFilter), C.POINTER(TrRenderParams), C.c_void_p, C.POINTER(TrStats)]
            st["call"] = f
        if case["entry"] == "guided":
            ctx.guide_init(seed=seed)
            ctx.guide_set_params(_initial(seed))
            x, d, w = _vertices(seed, 16384)
            torch.cuda.synchronize()
            for _ in range(40):  # the mixture of a run under way, not an untrained one
                ctx.guide_train_step_dev(x.data_ptr(), d.data_ptr(), w.data_ptr(), len(w), 3e-3)
            ctx.guide_light_init((32, 16, 24), 8)
            st["guide"] = make_guide(0.25, *ROOM_BOX, record=8, light_guide=True, light_record=True)
    elif kind == "batch":
        n = case["scenes"]
        parts, jobs, films = [], [], []
        for k in range(n):
            f = k / max(n - 1, 1)
            t = int(case["min_tris"] * (case["max_tris"] / case["min_tris"]) ** f)
            sc, cam, filt, par = scenes.batch_scene(seed * 64 + k, (t, t + 1))
            res, spp = (128, 512, 256, 1024)[k % 4], (16, 4, 16, 4, 4)[k % 5]
            par = make_params(res, res, spp, 3, 6, seed_base=((seed * 64 + k) * 7919) & 0x3FFFFFFF)
            parts.append(sc)
            films.append(torch.zeros(res, res, 4, device=DEV))
            jobs.append((k, cam, filt, par, films[-1].data_ptr()))
        ctx.upload_set(parts)
        st.update(jobs=jobs, films=films)
    elif kind == "trace":
        ctx.upload(scenes.traversal(case["tris"], seed))
        n = case["rays"]
        close, shadow = _rays(case, seed)
        if case["host"]:
            st["close"], st["shadow"] = (r.cpu().numpy().view(scenes.RAY_DTYPE).reshape(-1) for r in (close, shadow))
        else:
            st.update(close=close, shadow=shadow, n=n, prim=torch.empty(n, dtype=torch.int32, device=DEV),
                      t=torch.empty(n, device=DEV), hit=torch.empty(n, dtype=torch.uint8, device=DEV))
    else:
        n = case["rows"]
        ctx.guide_init(seed=seed)
        ctx.guide_set_params(_initial(seed))
        x, d, w = _vertices(seed, n)
        st.update(n=n, x=x, d=d, w=w, out=torch.empty(n, 40, device=DEV), grads=torch.empty(GpuContext.GUIDE_PARAMS, device=DEV))
        if kind == "network":
            st["dout"] = _rand(seed + 5, n, 40, normal=True) / n
    torch.cuda.synchronize()
    return st


def _rays(case, seed):
    """Closest-hit rays from the unit cube's surface and shadow rays of length
    uniform in (0, 1): o, t_min, d, t_max as the ray record lays them out."""
    n, out = case["rays"], []
    for k in (0, 1):
        o = _rand(seed + 10 * k + 1, n, 3)
        g = torch.Generator(device=DEV)
        g.manual_seed(seed + 10 * k + 2)
        face = torch.randint(0, 6, (n,), generator=g, device=DEV)
        o[torch.arange(n, device=DEV), face // 2] = (face % 2).float()
        d = _rand(seed + 10 * k + 3, n, 3, normal=True).double()
        d = (d / d.norm(dim=1, keepdim=True)).float()
        r = torch.zeros(n, 8, device=DEV)
        at = {name: scenes.RAY_DTYPE.fields[name][1] // 4 for name in ("o", "d", "t_min", "t_max")}
        r[:, at["o"]:at["o"] + 3] = o
        r[:, at["d"]:at["d"] + 3] = d
        r[:, at["t_max"]] = _rand(seed + 10 * k + 4, n) if k else 3.4028234663852886e38
        out.append(r)
    return out


# ---------------------------------------------------------------- one pass


def run(st):
    case, ctx, kind = st["case"], st["ctx"], st["kind"]
    if kind == "render":
        film, entry = st["film"], case["entry"]
        if entry == "host":
            return ctx.render(st["cam"], st["filt"], st["par"], fp64=case["fp64"])[0]
        if entry == "guided":
            ctx.render_guided_dev(st["cam"], st["filt"], st["par"], st["guide"], film.data_ptr(), fp64=case["fp64"])
            return film
        if entry == "noalloc":
            ctx._check(st["call"](ctx.h, C.byref(st["cam"]), C.byref(st["filt"]), C.byref(st["par"]), film.data_ptr(), None))
            return film
        ctx.render_dev(st["cam"], st["filt"], st["par"], film.data_ptr(), fp64=case["fp64"])
        if not case["post"]:
            return film
        n, rgb = st["n"], st["rgb"].data_ptr()
        ctx.film_resolve_dev(film.data_ptr(), n, rgb, fp64=case["fp64"])
        ctx.to_rgbe_dev(rgb, n, st["rgbe"].data_ptr())
        ctx.aces_tone_map_dev(rgb, n, 1.5)
        ctx.to_rgb8_dev(rgb, n, st["rgb8"].data_ptr())
        return film, st["rgb"], st["rgbe"], st["rgb8"]
    if kind == "batch":
        ctx.render_batch_dev(st["jobs"])
        return st["films"]
    if kind == "trace":
        if case["host"]:
            prim, t = ctx.trace_closest(st["close"])
            return prim, t, ctx.trace_any(st["shadow"])
        ctx.trace_closest_dev(st["close"].data_ptr(), st["n"], st["prim"].data_ptr(), st["t"].data_ptr())
        ctx.trace_any_dev(st["shadow"].data_ptr(), st["n"], st["hit"].data_ptr())
        return st["prim"], st["t"], st["hit"]
    if kind == "network":
        ctx.guide_forward_dev(st["x"].data_ptr(), st["n"], st["out"].data_ptr())
        ctx.guide_backward_dev(st["x"].data_ptr(), st["dout"].data_ptr(), st["n"], st["grads"].data_ptr())
        return st["out"], st["grads"]
    loss = ctx.guide_train_step_dev(st["x"].data_ptr(), st["d"].data_ptr(), st["w"].data_ptr(), st["n"], 1e-3)
    return loss, ctx.guide_params()


# ---------------------------------------------------------------- what a pass cannot do without


def _frame_work(samples, pixels, prims, vertices, lights, film_bytes):
    # a vertex: the BSDF (about 200 operations), a light sample and shadow ray per light, a continuation ray; a ray:
    # two box tests of 12 operations per level of the tree and three triangle tests of 50
    ray = 24 * math.log2(max(prims, 2)) + 150
    ops = samples * vertices * (200 + lights * (100 + ray) + ray)
    scene = prims * (64 + 48 + 128 + 32)
    return scene + pixels * film_bytes, ops


def work(case):
    kind = case["kind"]
    if kind == "render":
        f = FAMILY[case["scene"]]
        px = case["width"] * case["height"]
        b, o = _frame_work(px * case["spp"], px, f["prims"], f["vertices"], f["lights"], 32 if case["fp64"] else 16)
        if case["post"]:
            b += px * (16 + 12 + 4 + 3)
        if case["entry"] == "guided":  # the network at the walls' vertices
            o += px * case["spp"] * f["vertices"] * 0.5 * 2 * sum(i * j for i, j in LAYERS)
        return {"bytes": b, "flops": o}
    if kind == "batch":
        b = o = 0.0
        for k in range(case["scenes"]):
            t = case["min_tris"] * (case["max_tris"] / case["min_tris"]) ** (k / max(case["scenes"] - 1, 1))
            px = (128, 512, 256, 1024)[k % 4] ** 2
            x, y = _frame_work(px * (16, 4, 16, 4, 4)[k % 5], px, t, 2.0, 5, 16)
            b, o = b + x, o + y
        return {"bytes": b, "flops": o}
    if kind == "trace":
        n, t = case["rays"], case["tris"]
        return {"bytes": t * (64 + 48) + n * (2 * 32 + 8 + 1), "flops": 2 * n * (24 * math.log2(t) + 150)}
    n, mac = case["rows"], sum(i * j for i, j in LAYERS)
    params = 4 * GpuContext.GUIDE_PARAMS
    if kind == "network":  # forward; forward again and two products per layer in the backward pass
        return {"bytes": n * 4 * (7 + 40 + 7 + 40) + 2 * params, "flops": n * 2 * mac * 3}
    return {"bytes": n * 4 * (7 + 3 + 1) + 7 * params, "flops": n * 2 * mac * 3}


# ---------------------------------------------------------------- the result in 64 bits


def _parameters(flat):
    p, o, out = torch.from_numpy(flat).to(DEV).double(), 0, []
    for i, j in LAYERS:
        out.append((p[o:o + i * j].reshape(j, i).clone().requires_grad_(), p[o + i * j:o + i * j + j].clone().requires_grad_()))
        o += i * j + j
    return out


def _forward(layers, x):
    h = x.double()
    for k, (w, b) in enumerate(layers):
        h = h @ w.T + b
        if k < len(layers) - 1:
            h = torch.relu(h)
    return h


def _initial(seed):
    """A network's first parameters: uniform in +-1 / sqrt(inputs), layer by layer, weights then biases."""
    rng = np.random.default_rng(seed)
    return np.concatenate([rng.uniform(-1, 1, i * j + j).astype(np.float32) / np.float32(math.sqrt(i)) for i, j in LAYERS])


def _log_density(z, d):
    """log of the 8-lobe von Mises-Fisher mixture of network outputs z at d."""
    z = z.reshape(-1, 8, 5)
    log_pi = torch.log_softmax(z[:, :, 0], dim=1)
    kappa = torch.exp(torch.clamp(z[:, :, 1], -4.0, 7.0))
    m = z[:, :, 2:5]
    mu = m / (m.norm(dim=2, keepdim=True) + 1e-6)
    cos = (mu * d.double()[:, None, :]).sum(2)
    norm = torch.log(kappa) - math.log(2 * math.pi) - torch.log1p(-torch.exp(-2 * kappa))
    return torch.logsumexp(log_pi + norm + kappa * (cos - 1), dim=1)


def _closest(tris, rays):
    """Hit distance of every ray against all triangles, both sides, FLT_MAX where it hits none."""
    v = torch.from_numpy(tris.positions[tris.indices.reshape(-1)].reshape(-1, 3, 3)).to(DEV).double()
    a, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    at = {name: scenes.RAY_DTYPE.fields[name][1] // 4 for name in ("o", "d")}
    o, d = (rays[:, at[k]:at[k] + 3].double() for k in ("o", "d"))
    best = torch.full((len(rays),), 3.4028234663852886e38, dtype=torch.float64, device=DEV)
    step = max(1, (1 << 24) // len(rays))
    n = torch.cross(e1, e2, dim=1)
    for k in range(0, len(v), step):
        # the determinants of Moeller and Trumbore's test as matrix products over the chunk
        aa, b1, b2, nn = a[k:k + step], e1[k:k + step], e2[k:k + step], n[k:k + step]
        det = -(d @ nn.T)
        od = torch.cross(o, d, dim=1)
        num_u = od @ b2.T - d @ torch.cross(b2, aa, dim=1).T
        num_v = -(od @ b1.T) + d @ torch.cross(b1, aa, dim=1).T
        num_t = o @ nn.T - (aa * nn).sum(1)
        u, w, t = num_u / det, num_v / det, num_t / det
        t = torch.where((u >= 0) & (w >= 0) & (u + w <= 1) & (t >= 0), t, torch.inf)
        best = torch.minimum(best, t.min(dim=1).values)
    return best


def exact(case, seed):
    kind = case["kind"]
    if kind in ("render", "batch"):
        return None  # millions of random walks: another rounding of one direction is another walk
    if kind == "trace":
        if case["tris"] * case["rays"] > 1 << 33:
            return None  # every ray against every triangle would take minutes
        return None, _closest(scenes.traversal(case["tris"], seed), _rays(case, seed)[0]), None
    n = case["rows"]
    layers = _parameters(_initial(seed))
    flat = [p for wb in layers for p in wb]
    x, d, w = _vertices(seed, n)
    z = _forward(layers, x)
    if kind == "network":
        grads = torch.autograd.grad((z * (_rand(seed + 5, n, 40, normal=True) / n).double()).sum(), flat)
        return z.detach(), torch.cat([g.reshape(-1) for g in grads])
    loss = -(w.double() * _log_density(z, d)).sum() / w.double().sum()
    grads = torch.autograd.grad(loss, flat)
    # Adam's first step from zero moments
    new = torch.cat([(p - 1e-3 * g / (g.abs() + 1e-8)).reshape(-1) for p, g in zip(flat, grads)])
    return float(loss.detach()), new.detach()
