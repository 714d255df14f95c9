"""The work that a program has this library do, as cases that can be timed.

Each case is one call, or one short sequence of calls, of the public front end
(meshtrex_b200.api) on a synthetic volume of the kinds the library's own
benchmark and tests use: a radial ramp with fractal noise ("ball"), noisy
Gaussian blobs ("blobs"), a noisy gyroid ("gyroid"), a torus distance field
("torus") and meshtrex's sphere fixture ("sphere").  Volumes are [z, y, x].
The seed bends a volume's values on either side of the isovalues, so inputs of
two seeds differ at nearly every voxel and their meshes have the same size.

  listed()             the named cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  volume, context and plan, on the GPU, from the seed alone
  run(state)           one pass through the public entry points, and its outputs
  work(case)           bytes and operations that one pass cannot do without
  exact(case, seed)    the computed outputs in 64 bits, by plain torch

Kinds of pass:
  dropin    the staged calls of meshtrex's main, outputs copied out (api.extract)
  async     the whole path in one call with preallocated outputs, no host wait
  shaded    staged calls for a renderer: VertexData in NDC with normals, then
            meshlets of at most 64 vertices and 126 triangles
  backward  the adjoint of an extraction, for a given dL/dvertex
  fit       one step of fitting a field: staged forward, loss gradient, adjoint
  batch     many (volume, isovalue) jobs in one run
  upload    a pinned host volume uploaded under its min/max, then several
            isovalues from the same min/max
"""
import math

import numpy as np
import torch

from meshtrex_b200 import _lib as L
from meshtrex_b200 import api

_DTYPES = {"u8": torch.uint8, "u16": torch.uint16, "f32": torch.float32}
_BYTES = {"u8": 1, "u16": 2, "f32": 4}
_SCALE = {"u8": 255.0, "u16": 65535.0, "f32": 1.0}
_SHADED = dict(vertex_format=L.VERTEX_DATA, frame=L.FRAME_NDC, normals=True)


# ------------------------------------------------------------------- cases

def _case(name, kind, field, dtype, x, y, z, block, iso, **more):
    c = {"kind": kind, "field": field, "dtype": dtype, "x": x, "y": y, "z": z, "block": block, "iso": iso}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # meshtrex's own start-up fixture at main's block edge: a viewer opening a small model; latency counts
        _case("sphere_64_u8_b3", "dropin", "sphere", "u8", 64, 64, 64, 3, 128.0),
        # a small scan re-extracted while a user moves a slider: fits L2, launches and latency count
        _case("blobs_256_u8_b8", "async", "blobs", "u8", 256, 256, 256, 8, 128.0),
        # main's scan shape at main's block edge 3, the staged path as the reference program runs it
        _case("scan_1024x1024x314_u8_b3", "dropin", "ball", "u8", 1024, 1024, 314, 3, 80.0),
        # the headline volume: 2 GiB of 16-bit voxels, larger than L2, the lowest (largest) of its isovalues
        _case("ball_1024_u16_b8", "async", "ball", "u16", 1024, 1024, 1024, 8, 16384.0),
        # a simulation field with surface nearly everywhere: many triangles for each voxel
        _case("gyroid_512_f32_b8", "async", "gyroid", "f32", 512, 512, 512, 8, 0.0),
        # a renderer's input from a scan of odd size: rows that are not 16-byte aligned
        _case("shaded_509x387x301_u16_b8", "shaded", "ball", "u16", 509, 387, 301, 8, 32768.0),
        # the other block edges that the autotuner offers, on float and on 16-bit volumes
        _case("gyroid_384x320x256_f32_b4", "async", "gyroid", "f32", 384, 320, 256, 4, 0.0),
        _case("ball_640x512x448_u16_b16", "async", "ball", "u16", 640, 512, 448, 16, 32768.0),
        # inverse problems: gradients of a loss on the mesh with respect to the field
        _case("backward_512_f32", "backward", "torus", "f32", 512, 512, 512, 8, 0.0, mode="atomic"),
        _case("fit_250x198x171_f32", "fit", "torus", "f32", 250, 198, 171, 8, 0.0, mode="deterministic"),
        # a study: many volumes of mixed shapes and types, several isovalues each
        _case("batch_16_mixed", "batch", "blobs", "mixed", 256, 256, 256, 8, 0.0, volumes=16, smallest=64),
        # a volume that arrives on the host, looked at at three isovalues
        _case("upload_384_u16_b8", "upload", "ball", "u16", 384, 384, 384, 8, 32768.0),
    ]


def draw(rng):
    kind = rng.choice(["dropin", "async", "async", "async", "shaded", "backward", "fit", "batch", "upload"])
    if kind == "batch":
        largest = rng.choice([96, 128, 160, 192, 224, 256])
        return _case("", "batch", "blobs", "mixed", largest, largest, largest, 8, 0.0,
                     volumes=rng.randint(3, 14), smallest=rng.choice([24, 32, 48, 64]))
    dtype = rng.choice(["u8", "u16", "f32"])
    if kind in ("backward", "fit"):
        dtype = "f32"
    field = {"u8": ["ball", "blobs", "sphere"], "u16": ["ball", "ball", "blobs"],
             "f32": ["gyroid", "torus"]}[dtype]
    field = rng.choice(["torus"] if kind in ("backward", "fit") else field)
    # voxels: log-uniform up to the largest listed case of the kind
    top = {"dropin": 28.0, "async": 30.0 if field == "ball" else 27.0, "shaded": 25.5, "backward": 27.0,
           "fit": 24.0, "upload": 25.5}[kind]
    edge = 2.0 ** (rng.uniform(18.0, top) / 3.0)
    stretch = [2.0 ** rng.uniform(-0.6, 0.6) for _ in range(2)]
    dims = [edge * stretch[0], edge * stretch[1], edge / (stretch[0] * stretch[1])]
    x, y, z = (max(24, int(d)) for d in dims)
    if rng.random() < 0.5:  # half of the scans have rows of a round size
        x = max(32, x // 16 * 16)
    blocks = [8, 8, 8, 4, 3, 16] if kind in ("dropin", "async") else [8, 8, 4]
    iso = {"ball": 0.25 * rng.randint(1, 3), "blobs": 0.1 * rng.randint(2, 6), "sphere": 0.5}.get(field, 0.0)
    more = {"mode": rng.choice(["atomic", "deterministic"])} if kind in ("backward", "fit") else {}
    return _case("", kind, field, dtype, x, y, z, rng.choice(blocks), float(int(iso * _SCALE[dtype])), **more)


# ------------------------------------------------------------------ fields

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _axis(n):
    return torch.arange(n, device="cuda", dtype=torch.float32) / max(n - 1, 1)


def _hat(n, cells):
    """[n, cells + 1] weights of smooth interpolation from a lattice to n samples."""
    p = _axis(n) * cells
    i = p.floor().clamp(max=cells - 1)
    f = p - i
    w = f * f * (3.0 - 2.0 * f)
    m = torch.zeros((n, cells + 1), device="cuda")
    at = i.long().unsqueeze(1)
    m.scatter_(1, at, (1.0 - w).unsqueeze(1))
    m.scatter_(1, at + 1, w.unsqueeze(1))
    return m


class _Noise:
    """Fractal value noise: octaves of random lattices, each twice as fine and half as strong."""

    def __init__(self, shape, octaves, g):
        self.parts = []
        for o in range(octaves):
            c = 4 << o
            lattice = torch.rand((c + 1, c + 1, c + 1), generator=g, device="cuda") * 2.0 - 1.0
            wz, wy, wx = (_hat(n, c) for n in shape)
            self.parts.append((0.5 ** o, lattice, wz, wy, wx.t().contiguous()))

    def slab(self, z0, z1):
        out = None
        for amp, lattice, wz, wy, wxt in self.parts:
            t = torch.tensordot(wz[z0:z1], lattice, dims=([1], [0]))  # [z, c, c]
            t = torch.matmul(torch.matmul(wy, t), wxt) * amp          # [z, Y, X]
            out = t if out is None else out.add_(t)
        return out


def _store(f, dtype, isos, m):
    """The field f in the volume's type, its values bent by the factors m (around 1) between the isovalues: each voxel
    stays on its side of every isovalue, or on it, so that every seed's surface has the same topology and size."""
    whole = dtype != "f32"
    if whole:
        f = f.mul_(_SCALE[dtype]).round_().clamp_(0.0, _SCALE[dtype])
    cuts = sorted({float(np.float32(i)) for i in isos})
    inf = float("inf")

    def above(v):
        return v + 1.0 if whole else float(np.nextafter(np.float32(v), np.float32(inf)))

    def below(v):
        return v - 1.0 if whole else float(np.nextafter(np.float32(v), np.float32(-inf)))

    out = torch.where(f < cuts[0], (cuts[0] - (cuts[0] - f) * m).clamp(max=below(cuts[0])), f)
    for lo, hi in zip(cuts, cuts[1:]):
        bent = lo + (hi - lo) * ((f - lo) / (hi - lo)).clamp(0.0, 1.0) ** m
        bent = (bent.round() if whole else bent).clamp(above(lo), below(hi))
        out = torch.where((f > lo) & (f < hi), bent, out)
    out = torch.where(f > cuts[-1], (cuts[-1] + (f - cuts[-1]) * m).clamp(min=above(cuts[-1])), out)
    if not whole:
        return out
    out = out.round_().clamp_(0.0, _SCALE[dtype])
    return out.to(torch.uint8) if dtype == "u8" else out.to(torch.int32).to(torch.uint16)


def _field(field, dtype, shape, isos, seed, shape_seed=1):
    """The volume, made in z-slabs on the GPU: the field of shape_seed, its values bent by the seed."""
    Z, Y, X = shape
    g = _generator(shape_seed)
    bend = _Noise(shape, 2, _generator(seed))
    vol = torch.empty(shape, dtype=_DTYPES[dtype], device="cuda")
    x, y = _axis(X).view(1, 1, -1), _axis(Y).view(1, -1, 1)
    zs = _axis(Z).view(-1, 1, 1)
    shift = ((torch.rand(3, generator=g, device="cuda") - 0.5) * 0.02).tolist()
    if field in ("ball", "torus"):
        noise = _Noise(shape, 5 if field == "ball" else 4, g)
    elif field == "blobs":
        centres = (0.2 + 0.6 * torch.rand((8, 3), generator=g, device="cuda")).tolist()
        sigmas = (0.05 + 0.10 * torch.rand(8, generator=g, device="cuda")).tolist()
        amps = (0.3 + 0.4 * torch.rand(8, generator=g, device="cuda")).tolist()
    step = max(1, (1 << 25) // (X * Y))
    for z0 in range(0, Z, step):
        z1 = min(Z, z0 + step)
        z = zs[z0:z1]
        if field == "ball":
            r = torch.sqrt((x - 0.5 - shift[0]) ** 2 + (y - 0.5 - shift[1]) ** 2 + (z - 0.5 - shift[2]) ** 2)
            f = 0.5 * (0.35 - r) / 0.35 + 0.08 * noise.slab(z0, z1)
            f = 0.5 + (4.0 if dtype == "u8" else 1.0) * f  # 8-bit scans are windowed
        elif field == "torus":
            q = torch.sqrt((x - 0.5 - shift[0]) ** 2 + (y - 0.5 - shift[1]) ** 2) - 0.3
            f = torch.sqrt(q ** 2 + (z - 0.5 - shift[2]) ** 2) - 0.1 + 0.05 * noise.slab(z0, z1)
        elif field == "blobs":
            f = torch.zeros((z1 - z0, Y, X), device="cuda")
            for c, s, a in zip(centres, sigmas, amps):
                k = -0.5 / (s * s)
                f += a * torch.exp(k * (z - c[2]) ** 2) * (torch.exp(k * (y - c[1]) ** 2) * torch.exp(k * (x - c[0]) ** 2))
            f += (4.0 / 255.0) * torch.randn(f.shape, generator=g, device="cuda")
        elif field == "gyroid":  # 12 periods over 2048 voxels, at any size
            kx, ky, kz = (2.0 * math.pi * 12.0 * (n - 1) / 2047.0 for n in (X, Y, Z))
            ax, ay, az = kx * x + 9.0 * shift[0], ky * y + 9.0 * shift[1], kz * z + 9.0 * shift[2]
            f = torch.sin(ax) * torch.cos(ay) + torch.sin(ay) * torch.cos(az) + torch.sin(az) * torch.cos(ax)
            f = f + 0.02 * torch.randn(f.shape, generator=g, device="cuda")
        else:  # meshtrex's sphere fixture (a clamped distance), as steep at every size as at 64 voxels
            w = max(X - 1, 1)
            dx, dy, dz = (w * (a - 0.5 - s) * e for a, s, e in
                          ((x, shift[0], 1.0), (y, shift[1], (Y - 1) / w), (z, shift[2], (Z - 1) / w)))
            radius = 0.4 * X
            f = ((torch.sqrt(dx * dx + dy * dy + dz * dz) - radius) * (127.0 / 25.6) + 128.0) / 255.0
        vol[z0:z1] = _store(f, dtype, isos, torch.exp(0.2 * bend.slab(z0, z1)))
    return vol


def _volume(case, seed):
    isos = _isos(case) if case["kind"] == "upload" else [case["iso"]]
    return _field(case["field"], case["dtype"], (case["z"], case["y"], case["x"]), isos, seed)


def _mix(case, seed):
    """The volumes and (volume, isovalue) jobs of a batch: shapes, types and counts by the case alone."""
    edges = [e for e in (24, 32, 48, 64, 96, 128, 160, 192, 224, 256) if case["smallest"] <= e <= case["x"]]
    vols, jobs = [], []
    for i in range(case["volumes"]):
        dtype = ("u8", "u16", "f32")[i % 3]
        shape = tuple(edges[(i * m + case["volumes"]) % len(edges)] for m in (1, 3, 5))
        isos = [0.15 + 0.11 * k for k in range(1 + (3 * i) % 5)]
        isos = [float(int(v * _SCALE[dtype])) if dtype != "f32" else float(np.float32(v)) for v in isos]
        vols.append(_field("blobs", dtype, shape, isos, 1000 * seed + i, shape_seed=i))
        jobs += [(i, iso) for iso in isos]
    return vols, jobs


def _isos(case):
    """The three isovalues of an upload pass."""
    i = int(case["iso"])
    return [case["iso"], float(i + i // 4), float(i - i // 4)] if case["dtype"] != "f32" else [case["iso"], 0.25, -0.25]


# ----------------------------------------------------------------- prepare

def _plan(ctx, vol, case, options=None):
    """Staged extraction: (push constants, MinMax, Filtering, Extraction)."""
    v = api.wrap_volume(vol)
    pc = api.push_constants((vol.shape[2], vol.shape[1], vol.shape[0]), case["block"], case["iso"])
    mm = api.compute_min_max_mip(ctx, v, pc)
    f = api.filter_active_blocks(ctx, mm, pc)
    api.read_active_block_count(ctx, f)
    return v, pc, mm, f, api.extract_meshlet_descriptors(ctx, mm, f, pc, options)


def prepare(case, seed):
    kind = case["kind"]
    ctx = api.Context()
    s = {"case": case, "ctx": ctx}
    if kind == "batch":
        vols, jobs = _mix(case, seed)
        edges = [case["block"]] * len(vols)
        probe = api.Batch(ctx, vols, edges, jobs, vertex_capacity=1 << 20, triangle_capacity=1 << 20, use_graph=False)
        probe.run()
        need = probe.results(check=False)[1]
        probe.close()
        s["batch"] = api.Batch(ctx, vols, edges, jobs, max_active_blocks=need["activeBlocks"],
                               vertex_capacity=need["vertexCount"], triangle_capacity=need["triangleCount"])
        return s
    vol = _volume(case, seed)
    s["vol"] = vol
    if kind == "upload":
        s["host"] = vol.cpu().pin_memory().numpy()
        del s["vol"]
    elif kind == "async":  # outputs sized from one staged extraction
        v, pc, mm, f, x = _plan(ctx, vol, case)
        s["x"] = api.AsyncExtractor(ctx, vol, case["block"], case["iso"], x.vertex_count + 1024,
                                    x.index_count // 3 + 1024, max_active_blocks=f.active_block_count + 1024)
        s["x"].vertices.zero_()
        s["x"].indices.zero_()
        for o in (x, f, mm):
            o.free()
    elif kind == "backward":
        s["plan"] = _plan(ctx, vol, case)
        s["grad"] = _gradient(s["plan"][4].vertex_count, seed)
    elif kind == "shaded":
        s["options"] = api.extract_options(**_SHADED)
    return s


def _gradient(n, seed):
    return torch.randn((n, 3), generator=_generator(seed + 77), device="cuda")


def _loss_gradient(v, case):
    """Gradient of the mean over vertices of (|v - c| - r)^2, in voxel units."""
    c = torch.tensor([case["x"] / 2.0, case["y"] / 2.0, case["z"] / 2.0], dtype=v.dtype, device=v.device)
    d = v - c
    n = d.norm(dim=1, keepdim=True)
    return (2.0 / max(1, v.shape[0])) * (n - 0.35 * case["x"]) * d / n


# --------------------------------------------------------------------- run

def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    mode = L.ADJOINT_DETERMINISTIC if case.get("mode") == "deterministic" else L.ADJOINT_ATOMIC
    if kind == "dropin":
        m = api.extract(s["vol"], case["block"], case["iso"], ctx=ctx)
        return {"vertices": m.vertices, "indices": m.indices, "meshlets": m.meshlets, "ids": m.active_ids,
                "leaf": m.leaf}
    if kind == "async":
        s["x"].run()
        return {"vertices": s["x"].vertices, "indices": s["x"].indices, "counters": s["x"].counters}
    if kind == "shaded":
        v, pc, mm, f, x = _plan(ctx, s["vol"], case, s["options"])
        m = api.build_meshlets(ctx, x)
        out = {"vertices": x.vertices(), "indices": x.indices(), "meshlets": m.descriptors,
               "meshlet_ids": m.vertex_ids, "meshlet_vertices": m.vertices, "meshlet_indices": m.indices}
        for o in (x, f, mm):
            o.free()
        return out
    if kind == "backward":
        v, pc, mm, f, x = s["plan"]
        dfield, diso = api.extract_backward(ctx, v, pc, f, x.out.meshletDescriptorBuffer.ptr, x.vertex_count,
                                            s["grad"], mode=mode)
        return {"dfield": dfield, "diso": diso}
    if kind == "fit":
        v, pc, mm, f, x = _plan(ctx, s["vol"], case)
        verts = x.vertices()
        dfield, diso = api.extract_backward(ctx, v, pc, f, x.out.meshletDescriptorBuffer.ptr, x.vertex_count,
                                            _loss_gradient(verts, case), mode=mode)
        for o in (x, f, mm):
            o.free()
        return {"vertices": verts, "dfield": dfield, "diso": diso}
    if kind == "batch":
        b = s["batch"]
        b.run()
        jobs, t = b.results()
        o = b.out
        out = {"vertices": api.device_view(o.vertexBuffer.ptr, (t["vertexCount"], 3), torch.float32),
               "indices": api.device_view(o.indexBuffer.ptr, (t["triangleCount"], 3), torch.int32),
               "meshlets": api.device_view(o.meshletDescriptorBuffer.ptr, (t["activeBlocks"], 4), torch.int32)}
        for view in out.values():
            view.owner = b  # the views are of the batch's own buffers: it lives as long as they do
        out["jobs"] = np.array([[j["vertexCount"], j["indexCount"], j["meshletCount"]] for j in jobs])
        return out
    # upload
    pcs = [api.push_constants((case["x"], case["y"], case["z"]), case["block"], i) for i in _isos(case)]
    v, mm = api.upload_compute_min_max_mip(ctx, s["host"], pcs[0])
    out = {}
    for k, pc in enumerate(pcs):
        f = api.filter_active_blocks(ctx, mm, pc)
        api.read_active_block_count(ctx, f)
        x = api.extract_meshlet_descriptors(ctx, mm, f, pc)
        out["vertices%d" % k], out["indices%d" % k] = x.vertices(), x.indices()
        x.free()
        f.free()
    mm.free()
    api.free_volume(ctx, v)
    return out


# ------------------------------------------------------------------- exact

def _values(vol, z0, z1):
    """Slices z0..z1 as float32 (exact for the integer types)."""
    return vol[z0:z1].to(torch.float32)


def _cut_edges(vol, block, iso):
    """(flat index of the owner voxel, axis) of every cut edge, in the library's order: owner block (x fastest),
    owner voxel in the block (x fastest), axis."""
    Z, Y, X = vol.shape
    B = block
    gx, gy = -(-X // B), -(-Y // B)
    keys, iso32 = [], torch.tensor(iso, dtype=torch.float32, device=vol.device)
    step = max(1, (1 << 26) // (X * Y))
    for z0 in range(0, Z, step):
        z1 = min(Z, z0 + step)
        inside = _values(vol, z0, min(Z, z1 + 1)) <= iso32
        own = inside[:z1 - z0]
        cut = (own[:, :, :-1] ^ own[:, :, 1:], own[:, :-1] ^ own[:, 1:],
               inside[:-1] ^ inside[1:])  # along z: one slice less at the end of the volume
        for a in range(3):
            z, y, x = (i for i in cut[a].nonzero(as_tuple=True))
            z = z + z0
            block_id = ((z // B) * gy + y // B) * gx + x // B
            local = ((z % B) * B + y % B) * B + x % B
            keys.append(((block_id * (B * B * B) + local) * 3 + a, (z * Y + y) * X + x))
    order = torch.cat([k[0] for k in keys])
    flat = torch.cat([k[1] for k in keys])
    order, at = torch.sort(order)
    return flat[at], order % 3


def _at(vol, flat):
    """Voxel values at flat indices, float64."""
    if vol.dtype == torch.uint16:
        return (vol.view(torch.int16).reshape(-1)[flat].to(torch.int32) & 0xffff).to(torch.float64)
    return vol.reshape(-1)[flat].to(torch.float64)


def _edges(vol, block, iso):
    Z, Y, X = vol.shape
    flat, axis = _cut_edges(vol, block, iso)
    step = torch.tensor([1, X, X * Y], device=vol.device)[axis]
    fa, fb = _at(vol, flat), _at(vol, flat + step)
    iso = float(np.float32(iso))
    d = fb - fa
    fine = d.abs() > 1e-5
    t = torch.where(fine, (iso - fa) / torch.where(fine, d, torch.ones_like(d)), torch.full_like(d, 0.5)).clamp(0.0, 1.0)
    x, y, z = flat % X, (flat // X) % Y, flat // (X * Y)
    pos = torch.stack([x, y, z], 1).to(torch.float64)
    pos[torch.arange(len(flat), device=vol.device), axis] += t
    return flat, axis, step, fa, fb, t, fine, pos


def _voxel_normal(vol, flat):
    Z, Y, X = vol.shape
    c = (flat % X, (flat // X) % Y, flat // (X * Y))
    n = []
    for a, (size, stride) in enumerate(((X, 1), (Y, X), (Z, X * Y))):
        lo, hi = (c[a] - 1).clamp(min=0), (c[a] + 1).clamp(max=size - 1)
        n.append(_at(vol, flat + (lo - c[a]) * stride) - _at(vol, flat + (hi - c[a]) * stride))
    n = torch.stack(n, 1)
    length = n.norm(dim=1, keepdim=True)
    return torch.where(length > 0, n / length.clamp(min=1e-300), torch.zeros_like(n))


def _adjoint(vol, case, grad, iso):
    flat, axis, step, fa, fb, t, fine, pos = _edges(vol, case["block"], iso)
    g = grad[torch.arange(len(flat), device=vol.device), axis]
    d = torch.where(fine, fb - fa, torch.ones_like(fa))
    g = torch.where(fine, g, torch.zeros_like(g))
    iso = float(np.float32(iso))
    out = torch.zeros(vol.numel(), dtype=torch.float64, device=vol.device)
    out.index_add_(0, flat, g * (iso - fb) / (d * d))
    out.index_add_(0, flat + step, g * (fa - iso) / (d * d))
    return out.view(vol.shape), (g / d).sum().reshape(1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        vols, jobs = _mix(case, seed)
        v = torch.cat([_edges(vols[i], case["block"], iso)[7] for i, iso in jobs])
        return {"vertices": v, "indices": None, "meshlets": None, "jobs": None}
    vol = _volume(case, seed)
    if kind == "upload":
        out = {}
        for k, iso in enumerate(_isos(case)):
            out["vertices%d" % k], out["indices%d" % k] = _edges(vol, case["block"], iso)[7], None
        return out
    if kind == "backward":
        n = len(_cut_edges(vol, case["block"], case["iso"])[0])
        dfield, diso = _adjoint(vol, case, _gradient(n, seed).double(), case["iso"])
        return {"dfield": dfield, "diso": diso}
    flat, axis, step, fa, fb, t, fine, pos = _edges(vol, case["block"], case["iso"])
    if kind == "dropin":
        return {"vertices": pos, "indices": None, "meshlets": None, "ids": None, "leaf": None}
    if kind == "async":
        spare = torch.zeros((1024, 3), dtype=torch.float64, device=vol.device)
        return {"vertices": torch.cat([pos, spare]), "indices": None, "counters": None}
    if kind == "fit":
        dfield, diso = _adjoint(vol, case, _loss_gradient(pos, case), case["iso"])
        return {"vertices": pos, "dfield": dfield, "diso": diso}
    # shaded
    dims = torch.tensor([case["x"], case["y"], case["z"]], dtype=torch.float64, device=vol.device)
    w = t.unsqueeze(1)
    n = _voxel_normal(vol, flat) * (1.0 - w) + _voxel_normal(vol, flat + step) * w
    length = n.norm(dim=1, keepdim=True)
    n = torch.where(length > 0, n / length.clamp(min=1e-300), torch.zeros_like(n))
    one = torch.ones((len(flat), 1), dtype=torch.float64, device=vol.device)
    return {"vertices": torch.cat([pos / dims * 2.0 - 1.0, one, n, 0.0 * one], 1), "indices": None,
            "meshlets": None, "meshlet_ids": None, "meshlet_vertices": None, "meshlet_indices": None}


# -------------------------------------------------------------------- work

def work(case):
    """Volume read once, mesh (or gradient) written once; a mesh has two triangles for each vertex.  The number of
    vertices is counted on the volume of seed 0.  Operations: one compare for each voxel and extraction, about ten
    for each vertex."""
    kind = case["kind"]
    if kind == "batch":
        vols, jobs = _mix(case, 0)
        n = sum(len(_cut_edges(vols[i], case["block"], iso)[0]) for i, iso in jobs)
        volume = sum(v.numel() * v.element_size() for v in vols)
        return {"bytes": volume + 36 * n, "flops": sum(vols[i].numel() for i, _ in jobs) + 10 * n}
    vol = _volume(case, 0)
    voxels, volume = vol.numel(), vol.numel() * _BYTES[case["dtype"]]
    isos = _isos(case) if kind == "upload" else [case["iso"]]
    n = sum(len(_cut_edges(vol, case["block"], i)[0]) for i in isos)
    mesh = 36 * n  # 12 bytes a vertex, 24 of indices
    if kind == "shaded":  # 32-byte vertices and indices, then both again as meshlets
        mesh = 2 * (32 + 24) * n
    if kind == "backward":  # both ends of every edge, its gradient, the dense field gradient
        return {"bytes": 20 * n + 4 * voxels, "flops": 12 * n}
    if kind == "fit":
        return {"bytes": volume + 24 * n + 4 * voxels, "flops": voxels + 30 * n}
    return {"bytes": volume + mesh, "flops": len(isos) * voxels + 10 * n}
