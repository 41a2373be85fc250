"""The extractions that this framework is used for, as cases with inputs, one pass each, and the work they stand for.

A case is one call of the public Python binding (tmc_gb300.native): DMC or TMC of one volume or of
a batch of volumes, with the outputs and simplification a caller asks for.
listed() holds the cases by name, draw() gives others of the same ranges, prepare() makes a case's
inputs from a seed, run() makes one call, work() counts the bytes and operations a call cannot do
without, and exact() restates in 64 bits the outputs that have such a value.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from tmc_gb300 import native

# ---------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------
# algo        "dmc" or "tmc"
# field       "blobs" (sums of Gaussians), "periodic" (sin kx cos ky + sin ky cos kz + sin kz cos kx),
#             "noise" (a coarse random grid upsampled, plus noise: ambiguous cells everywhere) or
#             "saddle" (the periodic field with near-singular bilinear saddles on a fifth of a face family)
# nx, ny, nz  grid points; a batch has `count` volumes whose sizes, fields and isovalues follow `sizes`
# iso         isovalue; k: frequency of the periodic field
# simplify, triangles, halfedges, f64   the call's options; host: field and mesh in host memory


def _case(algo, field, nx, ny, nz, iso=0.0, k=0.0, simplify=False, triangles=False, halfedges=False, f64=False,
          host=False, count=0, sizes=0, **name):
    return dict(name, algo=algo, field=field, nx=nx, ny=ny, nz=nz, iso=iso, k=k, simplify=simplify,
                triangles=triangles, halfedges=halfedges, f64=f64, host=host, count=count, sizes=sizes)


def listed():
    pi = math.pi
    return [
        # the smallest calls: an interactive isosurface of a small field, one call per frame
        _case("dmc", "blobs", 64, 64, 64, iso=0.5, name="dmc_blobs_64"),
        _case("tmc", "periodic", 57, 48, 71, iso=0.1, k=3 * pi, halfedges=True, name="tmc_halfedge_57x48x71"),
        # ordinary requests of a service: the whole DMC pipeline, and TMC with float64 positions
        _case("dmc", "periodic", 131, 117, 140, iso=-0.2, k=5 * pi, simplify=True, triangles=True, halfedges=True,
              f64=True, name="dmc_full_131x117x140"),
        _case("tmc", "blobs", 190, 151, 171, iso=0.4, f64=True, name="tmc_f64_190x151x171"),
        # many uneven volumes in one call
        _case("dmc", "mixed", 0, 0, 0, count=20, sizes=7, name="dmc_batch_20"),
        _case("tmc", "mixed", 0, 0, 0, count=20, sizes=7, name="tmc_batch_20"),
        # a C++ program's call: field and mesh in (pinned) host memory
        _case("dmc", "noise", 256, 256, 256, simplify=True, triangles=True, halfedges=True, host=True,
              name="dmc_host_256"),
        # a smooth large field, as a scan or a simulation gives it
        _case("dmc", "periodic", 512, 512, 512, iso=0.1, k=6 * pi, name="dmc_periodic_512"),
        # the framework's default benchmark: a large field of dense ambiguity, both algorithms
        _case("tmc", "noise", 512, 512, 512, name="tmc_noise_512"),
        _case("dmc", "noise", 512, 512, 512, simplify=True, triangles=True, halfedges=True, name="dmc_noise_512"),
        # planes of the 1024^3 precision workload: near-singular saddles, the float64 fallbacks
        _case("tmc", "saddle", 1024, 1024, 64, k=6 * pi, name="tmc_saddle_1024x1024x64"),
        _case("dmc", "saddle", 1024, 1024, 64, k=6 * pi, triangles=True, f64=True, name="dmc_saddle_1024x1024x64"),
    ]


def draw(rng):
    pi = math.pi
    algo = rng.choice(["dmc", "tmc"])
    # sizes of the call: 40 thousand to 60 million points, uneven axes
    points = math.exp(rng.uniform(math.log(4e4), math.log(6e7)))
    stretch = [math.exp(rng.uniform(-0.5, 0.5)) for _ in range(3)]
    edge = (points / (stretch[0] * stretch[1] * stretch[2])) ** (1 / 3)
    nx, ny, nz = (max(17, min(900, round(edge * s))) for s in stretch)
    kind = rng.random()
    if kind < 0.2:  # a batch
        return _case(algo, "mixed", 0, 0, 0, count=rng.randint(2, 16), sizes=rng.randrange(1 << 20),
                     f64=rng.random() < 0.25)
    field = rng.choice(["blobs", "periodic", "noise", "saddle"])
    iso = {"blobs": rng.uniform(0.2, 0.8), "periodic": rng.uniform(-0.3, 0.3)}.get(field, 0.0)
    k = rng.uniform(2 * pi, 8 * pi) if field in ("periodic", "saddle") else 0.0
    dmc = algo == "dmc"
    return _case(algo, field, nx, ny, nz, iso=iso, k=k, simplify=dmc and rng.random() < 0.5,
                 triangles=dmc and rng.random() < 0.5, halfedges=rng.random() < 0.5, f64=rng.random() < 0.3,
                 host=rng.random() < 0.15)


def _flags(case):
    f = native.OUT_POS_F64 if case["f64"] else 0
    if case["algo"] == "dmc":
        f |= native.DMC_SIMPLIFY if case["simplify"] else 0
        f |= native.OUT_TRIANGLES if case["triangles"] else 0
    f |= native.OUT_HALFEDGES if case["halfedges"] else 0
    return f | (native.OUT_HOST if case["host"] else 0)


# ---------------------------------------------------------------------------------------------
# fields (float32 on the GPU, shape (nz, ny, nx)), on [-1, 1]^3
# ---------------------------------------------------------------------------------------------
def _axes(nx, ny, nz):
    return [torch.linspace(-1, 1, n, dtype=torch.float64, device="cuda") for n in (nx, ny, nz)]


def _blobs(nx, ny, nz, rng):
    c, s = rng.uniform(-0.6, 0.6, size=(8, 3)), rng.uniform(0.15, 0.35, size=8)
    x, y, z = _axes(nx, ny, nz)
    f = torch.zeros((nz, ny, nx), dtype=torch.float64, device="cuda")
    for i in range(8):
        ex, ey, ez = (torch.exp(-((a - float(c[i, d])) ** 2) / float(2 * s[i] ** 2)) for d, a in enumerate((x, y, z)))
        f += ez[:, None, None] * (ey[:, None] * ex[None, :])[None]
    return f.float()


def _periodic(nx, ny, nz, k, rng):
    x, y, z = (a * k + float(p) for a, p in zip(_axes(nx, ny, nz), rng.uniform(0, 2 * math.pi, size=3)))
    f = (torch.sin(x)[None, :] * torch.cos(y)[:, None])[None].float()
    f = f + (torch.sin(y)[None, :] * torch.cos(z)[:, None])[:, :, None].float()
    return f + (torch.sin(z)[:, None] * torch.cos(x)[None, :])[:, None, :].float()


def _noise(nx, ny, nz, rng):
    # 1/16 of the points per axis, at least 5, as coarse random values; trilinear between them
    f = torch.from_numpy(rng.uniform(-1, 1, size=[max(5, round(n / 16) + 1) for n in (nz, ny, nx)])).float().cuda()
    f = torch.nn.functional.interpolate(f[None, None], size=(nz, ny, nx), mode="trilinear", align_corners=True)[0, 0]
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 62)))
    return f + 0.02 * torch.randn((nz, ny, nx), generator=g, device="cuda")


def _saddle(nx, ny, nz, k, rng):
    f = _periodic(nx, ny, nz, k, rng)
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 62)))
    shape = (nz, ny // 2, nx // 2)
    pick = torch.rand(shape, generator=g, device="cuda") < 0.2
    a, b, c = (0.2 + 0.8 * torch.rand(shape, generator=g, device="cuda") for _ in range(3))
    d = (a.double() * b / c).float()  # the decider (ab - cd) / (a + b + c + d) is zero up to a rounding
    s = torch.where(torch.rand(shape, generator=g, device="cuda") < 0.5, -1.0, 1.0)
    for dj, di, val in ((0, 0, s * a), (1, 1, s * b), (0, 1, -s * c), (1, 0, -s * d)):
        at = f[:, dj:2 * (ny // 2):2, di:2 * (nx // 2):2]
        at.copy_(torch.where(pick, val, at))
    return f


def _volumes(case):
    """(field, nx, ny, nz, iso, k) of each of the case's volumes."""
    if not case["count"]:
        return [(case["field"], case["nx"], case["ny"], case["nz"], case["iso"], case["k"])]
    # a batch: axes log-uniform in 32..192, blob and periodic fields in turn
    rng = np.random.Generator(np.random.PCG64(case["sizes"]))
    out = []
    for q in range(case["count"]):
        nx, ny, nz = (int(n) for n in np.exp(rng.uniform(math.log(32), math.log(193), size=3)))
        u, k = rng.uniform(0, 1), rng.uniform(2 * math.pi, 8 * math.pi)
        out.append(("periodic", nx, ny, nz, 0.6 * u - 0.3, k) if q % 2 else ("blobs", nx, ny, nz, 0.2 + 0.6 * u, 0.0))
    return out


def _varied(f, iso, kind, rng):
    """The field f with its differences to the isovalue scaled by positive factors.  One factor per
    plane, row and column keeps every point's side and every saddle's (both of its products get the
    same factors), so the meshes of all seeds have one size.  Smooth factors for smooth fields; powers
    of two, which round nothing, where a rounding could decide a saddle: with one step per axis for
    noise, the same everywhere for near-singular saddles."""
    if kind == "saddle":
        return f * 2.0 ** int(rng.integers(-8, 9))
    scale = []
    for n in reversed(f.shape):
        at, phase = torch.arange(n, device="cuda") / n, float(rng.uniform(0.1, 0.9))
        scale.append(1.0 + (at > phase) if kind == "noise" else torch.exp(0.3 * torch.sin(5 * (at + phase))).double())
    if kind == "noise":
        return f * scale[0] * scale[1][:, None] * scale[2][:, None, None]
    g = ((f.double() - iso) * scale[0] * scale[1][:, None] * scale[2][:, None, None] + iso).float()
    high = f.double() >= iso  # the side that a rounding at the isovalue could have changed
    g = torch.where(high & (g.double() < iso), torch.full_like(g, iso).nextafter(torch.full_like(g, 9.0)), g)
    return torch.where(~high & (g.double() >= iso), torch.full_like(g, iso).nextafter(torch.full_like(g, -9.0)), g)


def _fields(case, seed):
    """Each volume's field, origin and spacing."""
    made = []
    for q, (kind, nx, ny, nz, iso, k) in enumerate(_volumes(case)):
        rng = np.random.Generator(np.random.PCG64([q, nx, ny, nz, 77]))
        if kind == "blobs":
            f = _blobs(nx, ny, nz, rng)
        elif kind == "periodic":
            f = _periodic(nx, ny, nz, k, rng)
        elif kind == "noise":
            f = _noise(nx, ny, nz, rng)
        else:
            f = _saddle(nx, ny, nz, k, rng)
        rng = np.random.Generator(np.random.PCG64([int(seed), q]))
        f = _varied(f, iso, kind, rng)
        origin = [float(x) for x in rng.uniform(-1.2, -0.8, size=3)]
        spacing = [2.0 / (n - 1) * math.exp(x) for n, x in zip((nx, ny, nz), rng.uniform(-0.2, 0.2, size=3))]
        made.append((f.contiguous(), origin, spacing))
    return made


# ---------------------------------------------------------------------------------------------
# one call
# ---------------------------------------------------------------------------------------------
_ctx = None


def _context():
    """The context a program keeps for its calls."""
    global _ctx
    if _ctx is None:
        _ctx = native.Context(0)
    return _ctx


def prepare(case, seed):
    s = {"ctx": _context(), "flags": _flags(case), "case": case, "fields": [], "volumes": [], "isos": []}
    for (f, origin, spacing), (_, nx, ny, nz, iso, _) in zip(_fields(case, seed), _volumes(case)):
        if case["host"]:
            f = f.cpu().pin_memory()
        v = native.Volume()
        v.nx, v.ny, v.nz = nx, ny, nz
        v.origin, v.spacing = (ctypes.c_double * 3)(*origin), (ctypes.c_double * 3)(*spacing)
        v.data, v.on_device = f.data_ptr(), 0 if case["host"] else 1
        s["fields"].append(f)
        s["volumes"].append(v)
        s["isos"].append(iso)
    torch.cuda.synchronize()  # the context's stream does not wait for torch's
    return s


class _Mesh:
    """A mesh that is freed when the last of its arrays goes."""

    def __init__(self, ctx, mesh):
        self.ctx, self.mesh = ctx, mesh

    def __del__(self):
        self.ctx.free(self.mesh)


class _OnDevice:
    """A device array of a mesh, as torch takes it without a copy."""

    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": kind, "version": 2}


def _array(owner, ptr, shape, kind):
    if not ptr or not shape[0]:
        return torch.empty(shape, dtype={"<f4": torch.float32, "<f8": torch.float64}.get(kind, torch.int32))
    if owner.mesh.on_device:
        return torch.as_tensor(_OnDevice(owner, ptr, shape, kind), device="cuda")
    buf = (ctypes.c_char * (math.prod(shape) * int(kind[2]))).from_address(ptr)
    buf.owner = owner
    return np.frombuffer(buf, dtype=kind).reshape(shape)


def _outputs(ctx, m, case):
    o = _Mesh(ctx, m)
    dmc = case["algo"] == "dmc"
    out = {"v": _array(o, m.v, (m.nr_v, 3), "<f4"), "n": _array(o, m.n, (m.nr_v, 3), "<f4")}
    if case["f64"]:
        out["v64"] = _array(o, m.v64, (m.nr_v, 3), "<f8")
    if dmc:
        out["quads"] = _array(o, m.quads, (m.nr_q, 4), "<i4")
    if not dmc or case["triangles"]:
        out["tris"] = _array(o, m.tris, (m.nr_t, 3), "<i4")
    if case["halfedges"]:
        out["he"] = _array(o, m.he, (m.nr_he, 4), "<i4")
        out["he_v"] = _array(o, m.he_v, (m.nr_v,), "<i4")
        out["he_f"] = _array(o, m.he_f, (m.nr_q if dmc else m.nr_t,), "<i4")
    return out


def run(state):
    ctx, flags, case = state["ctx"], state["flags"], state["case"]
    dmc = case["algo"] == "dmc"
    if case["count"]:
        n = case["count"]
        algo = native.ALGO_DMC if dmc else native.ALGO_TMC
        return [_outputs(ctx, m, case)
                for m in ctx.batch_raw(state["volumes"], state["isos"], [algo] * n, [flags] * n)]
    vol, iso = state["volumes"][0], state["isos"][0]
    m = ctx.dmc_raw(vol, iso, flags) if dmc else ctx.tmc_raw(vol, iso, flags, case["halfedges"])
    return _outputs(ctx, m, case)


# ---------------------------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------------------------
def _crossed(high):
    """Crossed grid edges per axis (x, y, z), as masks."""
    return high[:, :, 1:] != high[:, :, :-1], high[:, 1:] != high[:, :-1], high[1:] != high[:-1]


def work(case):
    """The field read once and the mesh written once, its size counted on the field: a TMC vertex per
    crossed grid edge and two triangles per vertex, a DMC quad per crossed interior edge and about as
    many vertices, five sixths of them after the simplification.  Operations: a comparison per point,
    the interpolation of a position and a normal per vertex (about 100), and for a DMC vertex 49
    projection samples of about 30 each."""
    nbytes = flops = 0
    for (f, _, _), (_, nx, ny, nz, iso, _) in zip(_fields(case, 0), _volumes(case)):
        x, y, z = _crossed(f.double() >= iso if f.numel() < 1 << 24 else f >= iso)
        points = nx * ny * nz
        nbytes += 4 * points
        if case["algo"] == "dmc":
            nq = int(x[1:-1, 1:-1].sum() + y[1:-1, :, 1:-1].sum() + z[:, 1:-1, 1:-1].sum())
            flops += points + nq * (100 + 49 * 30)
            nv = nq = nq * 5 // 6 if case["simplify"] else nq
            nbytes += 16 * nq + (24 * nq if case["triangles"] else 0)
            nbytes += (64 * nq + 4 * nq + 4 * nv) if case["halfedges"] else 0
        else:
            nv = int(x.sum() + y.sum() + z.sum())
            flops += points + 100 * nv
            nbytes += 12 * 2 * nv + ((48 + 4) * 2 * nv + 4 * nv if case["halfedges"] else 0)
        nbytes += (24 + (24 if case["f64"] else 0)) * nv
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------------------------
# the outputs in 64 bits
# ---------------------------------------------------------------------------------------------
# A cell's corner v sits at (v & 1, v >> 1 & 1, v >> 2); its edges and faces (corner pairs, and per
# face the corners in rows of two) in the order in which the outputs are numbered.
_EDGES = ((0, 1), (1, 3), (2, 3), (0, 2), (4, 5), (5, 7), (6, 7), (4, 6), (0, 4), (1, 5), (3, 7), (2, 6))
_FACES = ((0, 1, 2, 3), (4, 5, 6, 7), (0, 1, 4, 5), (2, 3, 6, 7), (0, 2, 4, 6), (1, 3, 5, 7))
_EDGE_OF = {frozenset(e): q for q, e in enumerate(_EDGES)}


def _saddle_faces(cs):
    """The faces of MC case cs whose diagonal corners are on one side."""
    out = []
    for q, (a, b, c, d) in enumerate(_FACES):
        s = [cs >> v & 1 for v in (a, b, c, d)]
        if s[0] == s[3] and s[1] == s[2] and s[0] != s[1]:
            out.append(q)
    return out


def _contours(cs, joined):
    """The polygons of MC case cs as edge lists, by lowest edge; joined: bit per face, whether the
    high corners of a saddle face are connected across it."""
    link = {e: [] for e in range(12)}
    for q, (a, b, c, d) in enumerate(_FACES):
        ring = (a, b, d, c)
        side = [cs >> v & 1 for v in ring]
        cut = [_EDGE_OF[frozenset((ring[r], ring[(r + 1) % 4]))] for r in range(4)]
        if side[0] == side[2] and side[1] == side[3] and side[0] != side[1]:
            # the edges at each corner that is cut off: the low ones when the high are connected
            pairs = [(cut[r], cut[(r + 3) % 4]) for r in range(4) if side[r] == (0 if joined >> q & 1 else 1)]
        else:
            on = [cut[r] for r in range(4) if side[r] != side[(r + 1) % 4]]
            pairs = [tuple(on)] if on else []
        for x, y in pairs:
            link[x].append(y)
            link[y].append(x)
    seen, out = set(), []
    for e in range(12):
        if link[e] and e not in seen:
            ring, prev, at = [], None, e
            while at not in ring:
                ring.append(at)
                nxt = [x for x in link[at] if x != prev] or link[at]
                prev, at = at, nxt[0]
            seen.update(ring)
            out.append(ring)
    return out


def _corner(f, i, j, k, v):
    return f[k + (v >> 2), j + (v >> 1 & 1), i + (v & 1)]


def _cells(f, iso):
    """The crossed cells in order: i, j, k, and their MC cases."""
    high = (f >= iso)
    cs = sum(high[v >> 2:high.shape[0] - 1 + (v >> 2), (v >> 1 & 1):high.shape[1] - 1 + (v >> 1 & 1),
                  (v & 1):high.shape[2] - 1 + (v & 1)].to(torch.uint8) << v for v in range(8))
    k, j, i = torch.nonzero((cs != 0) & (cs != 255), as_tuple=True)
    return i, j, k, cs[k, j, i].long()


def _difference(f, i, j, k, axis, h, one_sided):
    """The field's difference quotient along an axis at grid points.  one_sided: TMC's border rule;
    else DMC's: a point beyond the upper border is replaced by point 0 (index max - i), below the
    lower by point 0, both over twice the spacing."""
    at = [k, j, i]
    n = f.shape[2 - axis]
    p = at[2 - axis]
    if one_sided:
        lo, hi = (p - 1).clamp(min=0), (p + 1).clamp(max=n - 1)
        step = h * (hi - lo).double()
    else:
        lo, hi = (p - 1).clamp(min=0), torch.where(p + 1 >= n, n - (p + 1), p + 1)
        step = 2 * h
    a, b = list(at), list(at)
    a[2 - axis], b[2 - axis] = lo, hi
    return (f[tuple(b)] - f[tuple(a)]) / step


def _exact_tmc(f, iso, origin, h):
    """Positions and normals of TMC's edge vertices, in order; None where cells have saddle faces or
    opposite corners alone on a side (their inner vertices interleave)."""
    i, j, k, cs = _cells(f, iso)
    free = torch.tensor([not _saddle_faces(c) and c not in (0x81, 0x42, 0x24, 0x18, 0x7e, 0xbd, 0xdb, 0xe7)
                         for c in range(256)], device=f.device)
    if not bool(free[cs].all()):
        return None
    keys, pos, nor = [], [], []
    for e, (a, b) in enumerate(_EDGES):
        axis = {1: 0, 2: 1, 4: 2}[b - a]
        own = ((cs >> a ^ cs >> b) & 1).bool()
        for d, p in enumerate((i, j, k)):
            if d != axis and not a >> d & 1:
                own &= p == 0  # a lower neighbour creates the vertex
        ii, jj, kk = i[own], j[own], k[own]
        p0 = [ii + (a & 1), jj + (a >> 1 & 1), kk + (a >> 2)]
        p1 = [ii + (b & 1), jj + (b >> 1 & 1), kk + (b >> 2)]
        f0, f1 = f[p0[2], p0[1], p0[0]], f[p1[2], p1[1], p1[0]]
        t = (iso - f0) / (f1 - f0)
        pos.append(torch.stack([origin[d] + ((1 - t) * x + t * y) * h[d] for d, (x, y) in enumerate(zip(p0, p1))], 1))
        n0, n1 = (torch.stack([_difference(f, *p, d, h[d], True) for d in range(3)], 1) for p in (p0, p1))
        nor.append((1 - t)[:, None] * n0 + t[:, None] * n1)
        keys.append(torch.nonzero(own)[:, 0] * 12 + e)
    order = torch.argsort(torch.cat(keys))
    n = torch.cat(nor)[order]
    return torch.cat(pos)[order], n / n.norm(dim=1, keepdim=True)


def _interior(i, j, k, e, n):
    """Whether edge e of each cell has four cells around it."""
    a, b = _EDGES[e]
    axis = {1: 0, 2: 1, 4: 2}[b - a]
    ok = torch.ones_like(i, dtype=torch.bool)
    for d, p in enumerate((i, j, k)):
        if d != axis:
            q = p + (a >> d & 1)
            ok &= (q >= 1) & (q <= n[d] - 2)
    return ok


def _nearest_sample(F, iso, mean, lo, hi, plane, others, count):
    """The projection sample nearest to the contour's mean point, where there is a valid one: F the
    corners with the projection's axes first, lo and hi the contour's box in that order."""
    A, B, W = plane
    s = torch.arange(1, count - 1, dtype=torch.float64, device=F.device) / (count - 1)
    u = (lo[:, A, None] + s * (hi - lo)[:, A, None])[:, :, None]
    v = (lo[:, B, None] + s * (hi - lo)[:, B, None])[:, None, :]
    c = F[:, :, None, None]
    g1 = (1 - v) * ((1 - u) * c[:, 0] + u * c[:, 1]) + v * ((1 - u) * c[:, 2] + u * c[:, 3])
    g2 = (1 - v) * ((1 - u) * c[:, 4] + u * c[:, 5]) + v * ((1 - u) * c[:, 6] + u * c[:, 7])
    w = (iso - g1) / (g2 - g1)
    flat = ((hi - lo)[:, W] < 1e-5).double() * 1e-5
    ok = (w >= (lo[:, W] - flat)[:, None, None] - 1e-12) & (w <= (hi[:, W] + flat)[:, None, None] + 1e-12)
    for olo, ohi in others:
        x = [olo[:, d, None, None] for d in (A, B, W)], [ohi[:, d, None, None] for d in (A, B, W)]
        ok &= ~((u >= x[0][0]) & (u <= x[1][0]) & (v >= x[0][1]) & (v <= x[1][1]) & (w >= x[0][2]) & (w <= x[1][2]))
    d = (mean[:, A, None, None] - u) ** 2 + (mean[:, B, None, None] - v) ** 2 + (mean[:, W, None, None] - w) ** 2
    d = torch.where(ok, d, torch.inf).flatten(1)
    q = d.argmin(1)
    m = count - 2
    at = torch.arange(len(q), device=F.device)
    p = torch.empty_like(mean)
    p[:, A], p[:, B], p[:, W] = u[at, q // m, 0], v[at, 0, q % m], w[at, q // m, q % m]
    return p, torch.isfinite(d[at, q])


def _exact_dmc(f, iso, origin, h):
    """Positions and normals of DMC's vertices before any simplification, in order."""
    i, j, k, cs = _cells(f, iso)
    n = f.shape[::-1]
    F = torch.stack([_corner(f, i, j, k, v) for v in range(8)], 1)
    key = cs.clone()
    for q, (a, b, c, d) in enumerate(_FACES):
        on = torch.tensor([q in _saddle_faces(x) for x in range(256)], device=f.device)[cs]
        num = F[:, a] * F[:, d] - F[:, b] * F[:, c]
        join = num / (F[:, a] + F[:, d] - F[:, b] - F[:, c]) >= iso
        key |= (on & join).long() << (8 + q)
    order, pos, loc, cell = [], [], [], []
    for x in torch.unique(key).tolist():
        sel = torch.nonzero(key == x)[:, 0]
        contours = _contours(x & 255, x >> 8)
        ci, cj, ck, c = i[sel], j[sel], k[sel], F[sel]
        pts = {}
        for ring in contours:
            for e in ring:
                a, b = _EDGES[e]
                t = (iso - c[:, a]) / (c[:, b] - c[:, a])
                t = t.float().double()  # an edge coordinate is a float32 in the algorithm itself
                pts[e] = torch.stack([t if (a ^ b) >> d & 1 else torch.full_like(t, a >> d & 1) for d in range(3)], 1)
        boxes = [(torch.stack([pts[e] for e in r]).amin(0), torch.stack([pts[e] for e in r]).amax(0)) for r in contours]
        for t, ring in enumerate(contours):
            used = torch.zeros_like(ci, dtype=torch.bool)
            for e in ring:
                used |= _interior(ci, cj, ck, e, n)
            mean, (lo, hi) = torch.stack([pts[e] for e in ring]).mean(0), boxes[t]
            if len(ring) >= 6:  # the projection along the largest component of the gradient at the mean point
                u, v, w = mean.unbind(1)
                size = torch.stack([
                    (1 - w) * ((1 - v) * (c[:, 1] - c[:, 0]) + v * (c[:, 3] - c[:, 2]))
                    + w * ((1 - v) * (c[:, 5] - c[:, 4]) + v * (c[:, 7] - c[:, 6])),
                    (1 - w) * ((1 - u) * (c[:, 2] - c[:, 0]) + u * (c[:, 3] - c[:, 1]))
                    + w * ((1 - u) * (c[:, 6] - c[:, 4]) + u * (c[:, 7] - c[:, 5])),
                    (1 - v) * ((1 - u) * (c[:, 4] - c[:, 0]) + u * (c[:, 5] - c[:, 1]))
                    + v * ((1 - u) * (c[:, 6] - c[:, 2]) + u * (c[:, 7] - c[:, 3]))], 1).abs()
            else:  # or along the box's shortest side
                size = -(hi - lo)
            along = 2 - size.flip(1).argmax(1)  # z before y before x on ties
            others = [boxes[q] for q, r in enumerate(contours) if q != t and len(r) == 3] if len(ring) != 3 else []
            p = mean.clone()
            for W in range(3):
                A, B = [d for d in range(3) if d != W]
                m = torch.nonzero(along == W)[:, 0]
                perm = [(q & 1) << A | (q >> 1 & 1) << B | (q >> 2) << W for q in range(8)]
                for count in (9, 28):
                    if len(m):
                        got, ok = _nearest_sample(c[m][:, perm], iso, mean[m], lo[m], hi[m], (A, B, W),
                                                  [(a[m], b[m]) for a, b in others], count)
                        p[m[ok]] = got[ok]
                        m = m[~ok]
            order.append(sel[used] * 4 + t)
            loc.append(p[used])
            cell.append(torch.stack([ci, cj, ck], 1)[used])
    order = torch.argsort(torch.cat(order))
    loc, cell = torch.cat(loc)[order], torch.cat(cell)[order]
    origin, step = (torch.tensor(x, dtype=torch.float64, device=f.device) for x in (origin, h))
    pos = origin + (cell + loc) * step
    nor = torch.zeros_like(loc)
    for v in range(8):
        weight = torch.ones_like(loc[:, 0])
        for d in range(3):
            weight = weight * (loc[:, d] if v >> d & 1 else 1 - loc[:, d])
        p = [cell[:, d] + (v >> d & 1) for d in range(3)]
        nor += weight[:, None] * torch.stack([_difference(f, *p, d, h[d], False) for d in range(3)], 1)
    return pos, nor / nor.norm(dim=1, keepdim=True)


def exact(case, seed):
    """Positions and normals in 64 bits.  None for simplified meshes (their merges are a choice of
    the mesh as a whole), for TMC meshes with inner vertices, and for the largest fields of many
    vertices, where this would take too long."""
    many = case["field"] in ("noise", "saddle") and case["nx"] * case["ny"] * case["nz"] > 1 << 23
    if case["simplify"] or many:
        return None
    outs = []
    for (f, origin, spacing), (_, _, _, _, iso, _) in zip(_fields(case, seed), _volumes(case)):
        got = (_exact_dmc if case["algo"] == "dmc" else _exact_tmc)(f.double(), iso, origin, spacing)
        v, n = got if got is not None else (None, None)
        outs.append({"v": v, "n": n, "v64": v} if case["f64"] else {"v": v, "n": n})
        for key, on in (("quads", case["algo"] == "dmc"), ("tris", case["algo"] == "tmc" or case["triangles"]),
                        ("he", case["halfedges"]), ("he_v", case["halfedges"]), ("he_f", case["halfedges"])):
            if on:
                outs[-1][key] = None
    if all(x is None for o in outs for x in o.values()):
        return None
    return outs if case["count"] else outs[0]
