"""Performance cases of the volume -> mesh path.

Each case is one call (or the two or three calls that belong together) a
program makes through the public front end: meshing volumes in device or host
memory, the batched atlas, a fitting step through the adjoint, HC smoothing
and mesh encoding.  Volumes are seeded stand-ins made on the GPU: solid noisy
spheres, CT-like scans (noise, salt, lobulated hollow structures), brain-like
shells and power-law Voronoi label volumes, the distributions of
nii2mesh_gb300/synth.py at any size.
"""
import math

import numpy as np
import torch

import nii2mesh_gb300 as n2m
from nii2mesh_gb300.autograd import MeshifyFunction, sphere_loss

DEV = "cuda:0"

# volume cases: entry = how the volume is handed over
#   "device"  float32 in GPU memory, mesh stays there (Context.meshify_device)
#   "into"    float32 in pinned host memory, mesh into the caller's pinned arrays (Context.meshify_into)
#   "typed"   raw uint8 / int16 voxels in host memory, mesh in fresh host memory (Context.meshify_typed)
#   "raw"     raw uint8 / int16 voxels in pinned host memory, copied to the GPU and cast there
#             (Context.cast_voxels_device), mesh stays there
# Meshes in a context's memory last until its next call, so the program copies them into tensors of
# its own (on the context's stream); those have room for the largest mesh it expects.
_VOLUME = dict(kind="volume", entry="device", cubes=n2m.MC33, pre=True, largest=False, bubbles=False, post=0,
               otsu=0, dtype="float32")


def listed():
    return [
        # a small region of interest with the program's default options: launches and host round trips count
        dict(_VOLUME, name="sphere64", content="spheres", nx=64, ny=64, nz=64, iso=50.0, largest=True),
        # a head scan as read from disk (uint8), every option on, 20 HC iterations
        dict(_VOLUME, name="brain_u8", content="brain", nx=182, ny=218, nz=182, iso=54.0, entry="raw", dtype="uint8",
             largest=True, bubbles=True, post=20),
        # the default flow of the program on a 1 mm template grid (odd rows): Otsu isolevel, then meshing with
        # the classic case table (-o 1)
        dict(_VOLUME, name="brain_otsu", content="brain", nx=181, ny=217, nz=181, iso=54.0, otsu=2, largest=True,
             bubbles=True, cubes=n2m.CLASSIC_TABLE),
        # a large CT scan resident in GPU memory: the whole surface (the benchmark's own workload)
        dict(_VOLUME, name="ct512", content="ct", nx=512, ny=512, nz=512, iso=300.0),
        # the same with the program's default clustering plus bubble filling
        dict(_VOLUME, name="ct512_cluster", content="ct", nx=512, ny=512, nz=512, iso=300.0, largest=True, bubbles=True),
        # a clinical stack (512 x 512 slices, odd count) through the default make's classic cubes
        dict(_VOLUME, name="ct_oldcubes", content="ct", nx=512, ny=512, nz=287, iso=300.0, cubes=n2m.OLDCUBES),
        # a large scan from host memory to a mesh in host memory, buffers reused from call to call
        dict(_VOLUME, name="ct512_host", content="ct", nx=512, ny=512, nz=512, iso=300.0, entry="into"),
        # int16 CT voxels as read from disk to a mesh in fresh host memory, no pre-smooth, odd sizes
        dict(_VOLUME, name="ct_i16_raw", content="ct", nx=401, ny=388, nz=211, iso=300.0, entry="typed", dtype="int16",
             pre=False, largest=True),
        # every region of a label volume in one call, as the atlas mode meshes them
        dict(name="atlas256", kind="atlas", nx=256, ny=256, nz=256, labels=250, post=5),
        # one step of fitting a volume to a shape: vertices, triangles and the gradient of every voxel
        dict(name="fit128", kind="fit", nx=128, ny=128, nz=128, post=10),
        # writing a large mesh that is still in GPU memory: gzip'ed mz3, the program's default format
        dict(name="mz3_gz", kind="encode", n=384, fmt="mesh.mz3", gz=True),
        # post-smoothing of a mesh in host memory through the reference's own entry point
        dict(name="hc_dropin", kind="hc", nvert=250000, iters=20),
    ]


def _size(rng, lo, hi):
    """log-uniform size; half of them as drawn, the others a multiple of 4 (aligned rows)"""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n if rng.random() < 0.5 else max(lo, n // 4 * 4)


def draw(rng):
    kind = rng.choice(["volume"] * 7 + ["atlas", "fit", "encode", "hc"])
    if kind == "volume":
        content = rng.choice(["spheres", "brain", "ct", "ct"])
        entry = rng.choice(["device", "device", "into", "typed", "raw"])
        c = dict(_VOLUME, content=content, entry=entry, nx=_size(rng, 48, 512), ny=_size(rng, 48, 512),
                 nz=_size(rng, 48, 512), iso={"spheres": 50.0, "brain": 54.0, "ct": 300.0}[content],
                 cubes=rng.choice([n2m.MC33, n2m.MC33, n2m.CLASSIC_TABLE, n2m.OLDCUBES]), pre=rng.random() < 0.8,
                 largest=rng.random() < 0.5, bubbles=rng.random() < 0.4, post=rng.choice([0, 0, 5, 20]))
        if entry in ("typed", "raw"):
            c["dtype"] = "uint8" if content == "brain" else "int16"
        elif content == "brain" and entry == "device":
            c["otsu"] = rng.choice([0, 2])
        return c
    if kind == "atlas":
        return dict(kind="atlas", nx=_size(rng, 64, 256), ny=_size(rng, 64, 256), nz=_size(rng, 64, 256),
                    labels=rng.randrange(8, 251), post=rng.choice([0, 5]))
    if kind == "fit":
        return dict(kind="fit", nx=_size(rng, 48, 160), ny=_size(rng, 48, 160), nz=_size(rng, 48, 160),
                    post=rng.choice([0, 5, 10]))
    if kind == "encode":
        fmt, gz = rng.choice([("mesh.mz3", True), ("mesh.mz3", False), ("mesh.gii", True), ("mesh.obj", False),
                              ("mesh.stl", False), ("mesh.ply", False)])
        return dict(kind="encode", n=_size(rng, 96, 384), fmt=fmt, gz=gz)
    return dict(kind="hc", nvert=int(math.exp(rng.uniform(math.log(4000), math.log(250000)))), iters=rng.choice([1, 10, 20]))


# ---- inputs -------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _axes(nx, ny, nz):
    f = lambda n: torch.arange(n, device=DEV, dtype=torch.float32)
    return f(nx).view(1, 1, nx), f(ny).view(1, ny, 1), f(nz).view(nz, 1, 1)


def _spheres(nx, ny, nz, seed):
    """eight solid spheres of 100 on 0 with N(0, 5) noise"""
    rng = np.random.default_rng(seed)
    vol = torch.randn((nz, ny, nx), generator=_gen(seed), device=DEV) * 5.0
    x, y, z = _axes(nx, ny, nz)
    m = min(nx, ny, nz)
    inside = torch.zeros((nz, ny, nx), dtype=torch.bool, device=DEV)
    for _ in range(8):
        c = rng.uniform(0.19, 0.81, 3) * (nx, ny, nz)
        r = rng.uniform(0.094, 0.22) * m
        inside |= (x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2 <= r * r
    return vol + inside * 100.0


def _brain(nx, ny, nz, seed):
    """perturbed ellipsoid shell with a hollow and a solid ball, whole numbers 0..255"""
    rng = np.random.default_rng(seed)
    g = _gen(seed)
    x, y, z = _axes(nx, ny, nz)
    cx, cy, cz = (nx - 1) / 2, (ny - 1) / 2, (nz - 1) / 2
    ax, ay, az = 0.385 * nx, 0.39 * ny, 0.357 * nz
    mean = (ax + ay + az) / 3
    d = (torch.sqrt(((x - cx) / ax) ** 2 + ((y - cy) / ay) ** 2 + ((z - cz) / az) ** 2) - 1.0) * mean
    s = mean / 73.3
    amp = rng.uniform(0.5, 1.0, 32)
    amp *= 16.0 * s / amp.sum()
    for a in amp:   # low-frequency Fourier modes
        k = rng.integers(-4, 5, 3)
        d += a * torch.cos(2 * math.pi * (k[0] * x / nx + k[1] * y / ny + k[2] * z / nz) + rng.uniform(0, 2 * math.pi))
    tissue = (d < 0) & (d > -25.0 * s)
    r1 = torch.sqrt((x - (cx - 15 * s)) ** 2 + (y - (cy + 10 * s)) ** 2 + (z - cz) ** 2)
    r2 = torch.sqrt((x - (cx + 14 * s)) ** 2 + (y - (cy - 12 * s)) ** 2 + (z - (cz + 5 * s)) ** 2)
    tissue |= (r1 <= 10.0 * s) & (r1 >= 6.5 * s)
    tissue |= r2 <= 8.0 * s
    bg = torch.randn((nz, ny, nx), generator=g, device=DEV) * 3.0 + 5.0
    fg = torch.randn((nz, ny, nx), generator=g, device=DEV) * 15.0 + 110.0
    return torch.where(tissue, fg, bg).round_().clamp_(0, 255)


def _ct(nx, ny, nz, seed):
    """N(-1000, 20) background, rotated lobulated and partly hollow ellipsoids of 400..1200
    (300 in 512^3, the same density at other sizes), 1 % salt at 2000"""
    rng = np.random.default_rng(seed)
    g = _gen(seed)
    dims = np.array([nx, ny, nz])
    vol = torch.randn((nz, ny, nx), generator=g, device=DEV) * 20.0 - 1000.0
    amax = min(40.0, 0.3 * dims.min())
    for _ in range(max(4, int(round(300 * float(np.prod(dims / 512.0)))))):
        ab = rng.uniform(4.0, amax, 3)
        c = rng.uniform(0.0, 1.0, 3) * dims
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        val = float(rng.uniform(400.0, 1200.0))
        hollow, wall = rng.random() < 0.6, rng.uniform(2.5, 6.0)
        lobes, lamp, lph = rng.integers(-3, 4, (4, 3)), rng.uniform(0.0, 0.12, 4), rng.uniform(0, 2 * np.pi, 4)
        r = int(np.ceil(ab.max() * 1.15)) + 1
        lo = np.maximum(np.floor(c - r).astype(int), 0)
        hi = np.minimum(np.ceil(c + r).astype(int) + 1, dims)
        if np.any(hi <= lo):
            continue
        p = [torch.arange(int(lo[i]), int(hi[i]), device=DEV, dtype=torch.float32) - float(c[i]) for i in range(3)]
        p = [p[0].view(1, 1, -1), p[1].view(1, -1, 1), p[2].view(-1, 1, 1)]
        u = [(p[0] * float(q[0, j]) + p[1] * float(q[1, j]) + p[2] * float(q[2, j])) / float(ab[j]) for j in range(3)]
        rho = torch.sqrt(u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
        ang = 1.0
        for k, a, ph in zip(lobes, lamp, lph):
            ang = ang + float(a) * torch.cos((u[0] * int(k[0]) + u[1] * int(k[1]) + u[2] * int(k[2])) * math.pi + float(ph))
        rho = rho * ang
        inside = rho <= 1.0
        if hollow:
            inside &= rho > 1.0 - wall / ab.min()
        vol[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]].masked_fill_(inside, val)
    vol.masked_fill_(torch.rand((nz, ny, nx), generator=g, device=DEV) < 0.01, 2000.0)
    return vol


def _labels(nx, ny, nz, labels, seed):
    """multiplicatively weighted Voronoi partition of a head-sized ellipsoid, power-law weights"""
    rng = np.random.default_rng(seed)
    x, y, z = _axes(nx, ny, nz)
    c = (np.array([nx, ny, nz]) - 1) / 2
    axes = np.array([0.42, 0.46, 0.40]) * [nx, ny, nz]
    p = rng.uniform(-1, 1, (8 * labels + 64, 3))
    seeds = c + p[(p ** 2).sum(1) <= 1.0][:labels] * axes
    w = np.minimum(rng.pareto(1.6, len(seeds)) + 1.0, 12.0)
    best = torch.full((nz, ny, nx), math.inf, device=DEV)
    lab = torch.zeros((nz, ny, nx), dtype=torch.int16, device=DEV)
    for i, (s, wi) in enumerate(zip(seeds, w)):
        d2 = ((x - float(s[0])) ** 2 + (y - float(s[1])) ** 2 + (z - float(s[2])) ** 2) * float(1.0 / (wi * wi))
        lab.masked_fill_(d2 < best, i + 1)
        torch.minimum(best, d2, out=best)
    out = ((x - float(c[0])) / float(axes[0])) ** 2 + ((y - float(c[1])) / float(axes[1])) ** 2 \
        + ((z - float(c[2])) / float(axes[2])) ** 2 > 1.0
    return lab.masked_fill_(out, 0)


def _tubes(nvert, seed):
    """closed rings and open tubes (a mesh cut by the field of view) with voxel noise, vertices in
    raster order as marching cubes numbers them: (vertices float64, triangles int32)"""
    rng = np.random.default_rng(seed)
    parts, tris, base = [], [], 0
    pieces = 8
    a = max(8, int(round(math.sqrt(nvert / pieces / 4.0))))
    b = max(8, nvert // pieces // a)
    for k in range(pieces):
        closed = k % 2 == 0
        u = np.arange(a) * (2 * np.pi / a)
        v = np.arange(b) * (2 * np.pi / b) * (1.0 if closed else 0.7)
        U, V = np.meshgrid(u, v, indexing="ij")
        r = a / (2 * np.pi) * 0.9
        R = b / (2 * np.pi) * 0.9 + r
        c = rng.uniform(0, 2 * R, 3)
        P = np.stack([(R + r * np.cos(U)) * np.cos(V), (R + r * np.cos(U)) * np.sin(V), r * np.sin(U)], -1).reshape(-1, 3)
        parts.append(P @ np.linalg.qr(rng.normal(size=(3, 3)))[0] + c + rng.normal(0, 0.15, P.shape))
        i, j = np.meshgrid(np.arange(a), np.arange(b if closed else b - 1), indexing="ij")
        q = lambda i, j: base + (i % a) * b + j % b
        tris.append(np.stack([q(i, j), q(i + 1, j), q(i + 1, j + 1)], -1).reshape(-1, 3))
        tris.append(np.stack([q(i, j), q(i + 1, j + 1), q(i, j + 1)], -1).reshape(-1, 3))
        base += a * b
    pts = np.concatenate(parts).astype(np.float32).astype(np.float64)
    t = np.concatenate(tris)
    f = np.floor(pts)
    order = np.lexsort((f[:, 0], f[:, 1], f[:, 2]))
    rank = np.empty(len(order), np.int64)
    rank[order] = np.arange(len(order))
    t = rank[t]
    return pts[order], np.ascontiguousarray(t[np.argsort(t.min(1), kind="stable")], dtype=np.int32)


def _volume(case, seed):
    make = {"spheres": _spheres, "brain": _brain, "ct": _ct}[case["content"]]
    return make(case["nx"], case["ny"], case["nz"], seed)


class _Device:
    """view of device memory that a context owns; keeps the context as long as a tensor refers to it"""

    def __init__(self, ctx, ptr, shape, typestr):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 2,
                                         "strides": None}


def _view(ctx, ptr, shape, typestr):
    return torch.as_tensor(_Device(ctx, ptr, shape, typestr), device=DEV)


def _room(case):
    """vertices the program keeps room for (twice as many triangles)"""
    nv, _ = _mesh_size(dict(case, largest=False))
    return 3 * nv + 60000 if nv < 1000000 else 2 * nv


def _buffers(nv, **kw):
    return {"pts": torch.zeros((nv, 3), dtype=torch.float64, **kw), "tris": torch.zeros((2 * nv, 3), dtype=torch.int32, **kw)}


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "hc":
        st["pts"], st["tris"] = _tubes(case["nvert"], seed)
        return st
    ctx = st["ctx"] = n2m.Context()
    st["stream"] = torch.cuda.ExternalStream(ctx.stream)
    if kind == "volume":
        v = _volume(case, seed)
        st["opts"] = dict(cubes=case["cubes"], pre_smooth=case["pre"], only_largest=case["largest"],
                          fill_bubbles=case["bubbles"], post_smooth=case["post"])
        if case["entry"] in ("typed", "raw"):
            v = v.round().to(getattr(torch, case["dtype"]))
        if case["entry"] == "into":
            st["keep"] = dict(_buffers(_room(case), pin_memory=True), vol=torch.empty(v.shape, pin_memory=True).copy_(v))
            st.update({k: t.numpy() for k, t in st["keep"].items()})
        elif case["entry"] == "typed":
            st["vol"] = v.cpu().numpy()
            st.update({k: t.numpy() for k, t in _buffers(_room(case)).items()})
        else:
            st.update(_buffers(_room(case), device=DEV))
            if case["entry"] == "raw":
                st["raw"] = torch.empty(v.shape, dtype=v.dtype, pin_memory=True).copy_(v)
                st["draw"], st["vol"] = torch.empty_like(v), torch.empty(v.shape, device=DEV)
            else:
                st["vol"] = v.contiguous()
    elif kind == "atlas":
        st["labels"] = _labels(case["nx"], case["ny"], case["nz"], case["labels"], seed)
        st.update(_buffers(int(40 * (case["nx"] * case["ny"] * case["nz"]) ** (2 / 3) * case["labels"] ** (1 / 3)) + 60000, device=DEV))
    elif kind == "fit":
        st["vol"] = _spheres(case["nx"], case["ny"], case["nz"], seed).requires_grad_()
        m = min(case["nx"], case["ny"], case["nz"])
        st["target"] = ([(case[k] - 1) / 2 for k in ("nx", "ny", "nz")], 40.0 * m / 128)
        st.update(_buffers(_room(dict(case, content="spheres")), device=DEV))
    else:
        n = case["n"]
        v = _ct(n, n, n, seed)
        torch.cuda.synchronize()
        tp, pp, nt, npt, _ = ctx.meshify_device(v.data_ptr(), (n, n, n), 300.0, only_largest=False)
        st["tris"], st["pts"] = _view(ctx, tp, (nt, 3), "<i4").clone(), _view(ctx, pp, (npt, 3), "<f8").clone()
        st["file"] = torch.zeros(200 * _room(dict(_VOLUME, content="ct", nx=n, ny=n, nz=n)) // 2, dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()   # a context works on its own stream
    return st


def _keep(state, **views):
    """the results into the program's own tensors, behind the context's work"""
    with torch.cuda.stream(state["stream"]):
        for name, v in views.items():
            state[name][:len(v)].copy_(v)


def _meshed(state, tp, pp, nt, npt):
    ctx = state["ctx"]
    _keep(state, tris=_view(ctx, tp, (nt, 3), "<i4"), pts=_view(ctx, pp, (npt, 3), "<f8"))
    return state["tris"], state["pts"], nt, npt


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "hc":
        return n2m.laplacian_smoothHC(state["pts"], state["tris"], iters=case["iters"])
    ctx = state["ctx"]
    if kind == "volume":
        v, o, iso = state["vol"], state["opts"], case["iso"]
        if case["entry"] == "into":
            nt, npt, _ = ctx.meshify_into(v, state["tris"], state["pts"], iso, **o)
            return state["tris"], state["pts"], nt, npt
        if case["entry"] == "typed":
            t, p, _ = ctx.meshify_typed(v, 1.0, 0.0, iso, **o)
            state["tris"][:len(t)], state["pts"][:len(p)] = t, p
            return state["tris"], state["pts"], len(t), len(p)
        if case["entry"] == "raw":
            state["draw"].copy_(state["raw"], non_blocking=True)
            state["stream"].wait_stream(torch.cuda.current_stream())
            ctx.cast_voxels_device(state["draw"].data_ptr(), case["dtype"], 1.0, 0.0, v.numel(), v.data_ptr())
        if case["otsu"]:
            iso = ctx.set_threshold_device(v.data_ptr(), v.numel(), case["otsu"])
        tp, pp, nt, npt, _ = ctx.meshify_device(v.data_ptr(), (v.shape[2], v.shape[1], v.shape[0]), iso, **o)
        return *_meshed(state, tp, pp, nt, npt), iso
    if kind == "atlas":
        # through the C ABI: the front end's atlas_device returns counts only
        return _atlas(state, ctx, state["labels"], case["post"])
    if kind == "fit":
        vol = state["vol"]
        vol.grad = None
        pts, tris = MeshifyFunction.apply(vol, ctx, 50.0, case["post"])
        sphere_loss(pts, *state["target"]).backward()
        state["pts"][:len(pts)].copy_(pts.detach())
        state["tris"][:len(tris)].copy_(tris)
        return state["pts"], state["tris"], len(pts), len(tris), vol.grad
    t, p = state["tris"], state["pts"]
    ptr, n = ctx.encode_mesh_to_device(case["fmt"], t.data_ptr(), p.data_ptr(), len(t), len(p), case["gz"])
    _keep(state, file=_view(ctx, ptr, (n,), "|u1"))
    return state["file"], n


def _atlas(state, ctx, labels, post):
    C, L = n2m.C, n2m.lib()
    nz, ny, nx = labels.shape
    o = n2m.Options(n2m.MC33, 0.5, True, True, True, post, False)
    nm, mp = C.c_int(), C.POINTER(n2m.AtlasMesh)()
    pp, tp, npt, nt = C.c_void_p(), C.c_void_p(), C.c_int64(), C.c_int64()
    n2m._lib.check(L.n2m_atlas_device(ctx.h, C.c_void_p(labels.data_ptr()), (C.c_int * 3)(nx, ny, nz), C.byref(o),
                                      n2m.ATLAS_BATCHED, C.byref(nm), C.byref(mp), C.byref(pp), C.byref(tp),
                                      C.byref(npt), C.byref(nt), None))
    table = np.zeros((state["case"]["labels"], 6), np.int64)   # one row per label
    for i, m in enumerate(mp[:nm.value]):
        table[i] = m.label, m.status, m.nvert, m.ntri, m.vert_offset, m.tri_offset
    return table, *_meshed(state, tp.value, pp.value, nt.value, npt.value)


# ---- what a pass cannot do without ------------------------------------------------------
def _mesh_size(case):
    """expected vertices and triangles, from the surface area of the generators' structures"""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n, m = nx * ny * nz, min(nx, ny, nz)
    if case.get("content") == "ct":
        pieces = max(4, round(300 * n / 512 ** 3))
        r = (4.0 + min(40.0, 0.3 * m)) / 2
        nv = pieces * 24.5 * r * r
        if not case["pre"]:
            nv += 0.06 * n   # every salt voxel has its own surface
        if case["largest"]:
            nv *= min(1.0, 15.0 / pieces)
    elif case.get("content") == "brain":
        nv = 1.5 * 2 * 4 * math.pi * (0.377 * (n ** (1 / 3))) ** 2
    else:
        nv = 1.5 * 8 * 4 * math.pi * (0.157 * m) ** 2 * (0.3 if case.get("largest") else 0.8)
    return int(nv) + 4096, 2 * int(nv) + 8192


def work(case):
    """bytes: inputs once, outputs once (24 per vertex, 12 per triangle); flops: the 15 taps of the
    pre-smooth, HC's neighbour sums"""
    kind = case["kind"]
    if kind == "hc":
        nv, nt = case["nvert"], 2 * case["nvert"]
        return {"bytes": 48 * nv + 12 * nt, "flops": case["iters"] * nv * 96}
    if kind == "encode":
        nv = (case["n"] / 512) ** 3 * 3.5e6
        return {"bytes": int(24 * nv + 24 * nv + (14 if case["gz"] else 36) * nv), "flops": 0}
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "atlas":
        nv = 9.0 * n ** (2 / 3) * case["labels"] ** (1 / 3)
        return {"bytes": int(2 * n + 24 * nv + 24 * nv), "flops": int(30 * n + 96 * nv * case["post"])}
    if kind == "fit":
        nv, nt = _mesh_size(dict(case, content="spheres"))
        return {"bytes": 8 * n + 36 * nv + 12 * nt, "flops": 60 * n + 192 * nv * case["post"]}
    nv, nt = _mesh_size(case)
    voxel = {"uint8": 1, "int16": 2, "float32": 4}[case["dtype"]]
    return {"bytes": voxel * n + 24 * nv + 12 * nt, "flops": (30 * n if case["pre"] else 0) + 96 * nv * case["post"]}


# ---- 64-bit values ------------------------------------------------------------------------
def exact(case, seed):
    """HC smoothing in float64.  The other cases have no such value: a mesh is defined by the
    reference's own float32 rounding, operation for operation (signs, tilings, welds and the
    degenerate filter follow from it), and files are bytes."""
    if case["kind"] != "hc":
        return None
    pts, tris = _tubes(case["nvert"], seed)
    n = len(pts)
    t = torch.from_numpy(tris.astype(np.int64))
    rows, cols = t.reshape(-1).repeat_interleave(2), t[:, [1, 2, 0, 2, 0, 1]].reshape(-1)
    num = torch.bincount(rows, minlength=n).to(torch.float64)

    def mean(x):
        s = torch.zeros_like(x).index_add_(0, rows, x[cols])
        return torch.where(num[:, None] > 0, s / num.clamp(min=1)[:, None], x)

    o = torch.from_numpy(pts)
    p, alpha, beta = o.clone(), 0.1, 0.5
    for _ in range(case["iters"]):
        q = p
        p = mean(q)
        b = p - (alpha * o + (1 - alpha) * q)
        p = p - (beta * b + (1 - beta) * mean(b))
    e = torch.sort(torch.stack([rows, cols], 1), 1).values[:, 0] * n + torch.sort(torch.stack([rows, cols], 1), 1).values[:, 1]
    u, cnt = torch.unique(e, return_counts=True)
    rim = u[cnt == 2]   # an edge of one triangle (listed from both ends)
    border = torch.zeros(n, dtype=torch.bool)
    border[rim // n] = True
    border[rim % n] = True
    p[border] = o[border]
    return p.numpy()
