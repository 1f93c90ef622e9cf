"""Workloads of the voxelizer: what a program that uses gpview_gb300 has it do.

listed() names the cases, draw(rng) makes one more of the same ranges, prepare(case, seed) builds
the inputs and the context that a caller keeps, run(state) makes one call and returns its outputs,
work(case) states the bytes and float operations such a call cannot do without, and
exact(case, seed) gives the normals (the only outputs that are computed numbers rather than
decisions, counts or indices) in 64 bits.

A case is a plain dict:
  kind    device    gpv_voxelize on device triangles, outputs left on the device
          level1    the same without a Level2 grid (an occupancy grid)
          stencil   the same with the rasterised inside fill
          normals   the same with float normals of both levels
          batch     gpv_voxelize_batch over many meshes in one call
          host      gpv_voxelize_to_host, page-locked triangles in, page-locked outputs out
          object    the Object mirror: host triangles in, numpy arrays and float normals out
          noalloc   gpv_voxelize_level1_noalloc into the caller's arrays
          shims     the reference-named Level2 calls on lists that the caller keeps
  mesh    sphere, torus, star, superellipsoid (generators) or cessna (the reference's own model,
          turned by a shape other than 0); size is the generator's resolution, shape its seed
  nx..nz  Level1 divisions; n2x..n2z Level2 divisions (0: none)
"""
import ctypes as C
import functools
import json
import math
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import gpview_gb300 as gpv

_CESSNA = os.path.join("tests", "golden", "cessna.obj")


def _case(name, kind, mesh, size, n1, n2, shape=1):
    n1 = (n1,) * 3 if isinstance(n1, int) else n1
    n2 = (n2,) * 3 if isinstance(n2, int) else n2
    return {"name": name, "kind": kind, "mesh": mesh, "size": size, "shape": shape, "nx": n1[0], "ny": n1[1],
            "nz": n1[2], "n2x": n2[0], "n2y": n2[1], "n2z": n2[2]}


def listed():
    return [
        # the reference's own model at its own default sizing (voxelCount 8, voxelCount2 4) through
        # the Object interface: the smallest call, host arrays and normals out
        {"name": "object-default", "kind": "object", "mesh": "cessna", "size": 0, "shape": 0,
         "count1": 8, "count2": 4},
        # a small scanned part, the quick interactive call
        _case("sphere-16k", "device", "sphere", 64, 64, 4),
        # a low-polygon model (triangles large against the cells) on a fine uneven grid
        _case("cessna-fine", "device", "cessna", 0, (150, 170, 130), 6),
        # the ordinary call: a quarter of a million triangles, 128^3 with 8^3 inside
        _case("torus-262k", "device", "torus", 256, 128, 8),
        # the largest plain call
        _case("star-1310k", "device", "star", 8, 256, 16),
        # an occupancy grid for simulation or printing: Level1 only, at high resolution
        _case("occupancy-512", "level1", "torus", 512, 512, 0),
        # a model library voxelized in one call: mixed shapes, sizes and grids
        {"name": "batch-256", "kind": "batch", "mesh": "mixed", "shape": 1, "count": 256, "tmin": 500, "tmax": 200000},
        # the ordinary call with the rasterised fill, the reference's own build switch
        _case("stencil-262k", "stencil", "torus", 256, 128, 8),
        # both levels' normals as floats (rendering and collision queries read them)
        _case("normals-131k", "normals", "torus", 181, (97, 101, 90), 8),
        # host to host: the mesh from a loader's buffer, every output back in host memory
        _case("host-328k", "host", "star", 7, 192, 8),
        # Level1 inside a host program that forbids allocations
        _case("noalloc-66k", "noalloc", "torus", 128, (128, 120, 100), 0),
        # a reference program relinked against the library: its two Level2 calls
        _case("shims-33k", "shims", "torus", 91, 64, 4),
    ]


# ---- drawn cases ------------------------------------------------------------------------------
def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


# largest number of Level2 cells of boundary voxels (by 6 n^2 of them) that a drawn case has
_CELLS = {"device": 6e8, "stencil": 1.5e8, "normals": 6e7, "host": 2e8, "shims": 2e7}


def draw(rng):
    kind = rng.choice(["device"] * 4 + ["level1", "batch", "stencil", "normals", "host", "object",
                                        "noalloc", "shims"])
    shape = rng.randint(1, 1 << 20)
    if kind == "batch":
        tmin = int(_log(rng, 300, 2000))
        return {"kind": kind, "mesh": "mixed", "shape": shape, "count": int(_log(rng, 8, 256)), "tmin": tmin,
                "tmax": int(_log(rng, 20000, 200000))}
    mesh = rng.choice(["sphere", "torus", "star", "superellipsoid", "cessna"])
    if kind == "object":
        return {"kind": kind, "mesh": mesh, "size": _size(rng, mesh, 300, 60000), "shape": shape,
                "count1": rng.randint(5, 40), "count2": rng.choice([2, 3, 4, 5, 6])}
    tmax = {"noalloc": 150000, "shims": 60000, "normals": 300000}.get(kind, 1300000)
    size = _size(rng, mesh, 500, tmax)
    top = {"level1": 512, "noalloc": 160, "shims": 80, "normals": 160}.get(kind, 256)
    base = _log(rng, 16, top)
    n1 = [max(8, int(round(base * rng.uniform(0.6, 1.0)))) for _ in range(3)]
    if kind in ("level1", "noalloc"):
        return _unnamed(_case("", kind, mesh, size, tuple(n1), 0, shape))
    while True:
        n2 = [rng.choice([1, 2, 3, 4, 5, 6, 8, 8, 10, 12, 16])] * 3
        if rng.random() < 0.3:
            n2 = [max(1, v + rng.choice([-1, 0, 1])) for v in n2]
        if 6 * base * base * n2[0] * n2[1] * n2[2] <= _CELLS[kind]:
            return _unnamed(_case("", kind, mesh, size, tuple(n1), tuple(n2), shape))


def _unnamed(c):
    c.pop("name")
    return c


def _size(rng, mesh, tmin, tmax):
    """A generator resolution with between tmin and tmax triangles, spread over the logarithm."""
    t = _log(rng, tmin, tmax)
    if mesh == "star":
        return max(2, min(8, int(round(math.log(t / 20.0, 4)))))
    return max(6, int(round(math.sqrt(t / 4.0))))


# ---- inputs -----------------------------------------------------------------------------------
# The case fixes the shape; the seed places it, by whole cells, in the grid (and turns the order of
# the triangles).  Coordinates lie in [1, 2), vertices on odd multiples of 2^-20 and cell edges on
# multiples of 2^-19, as a quantised model's do, so a move by whole cells is exact and a case has
# the same number of boundary voxels, and outputs of the same sizes, whatever its seed.
_Q = 1 << 19


def _rotation(rng):
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    return q * np.sign(np.diag(r))


def _shape(mesh, size, shape):
    """Triangles [T, 3, 3] of a shape."""
    rng = np.random.default_rng([shape, 77])
    g = int(rng.integers(1, 1 << 31))
    centre = (0.5, 0.5, 0.5)
    if mesh == "sphere":
        t = gpv.gen_uvsphere(g, 2 * size, size, centre, 0.4, 0.002)
    elif mesh == "torus":
        t = gpv.gen_torus(g, 2 * size, size, centre, 0.35, float(rng.uniform(0.1, 0.13)), 0.01)
    elif mesh == "star":
        t = gpv.gen_star(g, size, centre, 0.3, 0.2, (1.0, 1.0, 6.0))
    elif mesh == "superellipsoid":
        e = rng.uniform(0.3, 2.0, 2)
        t = gpv.gen_superellipsoid(g, 2 * size, size, centre, rng.uniform(0.2, 0.45, 3), e[0], e[1],
                                   _rotation(rng).astype(np.float32))
    else:
        o = gpv.Object()
        o.ReadObject(_CESSNA)
        o.CreateFlatTriangleData()
        t = o.flatCPUTriangleData
        if shape:
            t = (t.reshape(-1, 3).astype(np.float64) @ _rotation(rng).T).astype(np.float32)
    return t.reshape(-1, 3, 3)


def _place(t, n, cell, margin, slack, seed):
    """The shape fitted into the grid of n cells of size `cell` from 1.0, `margin` cells from its low
    side, and moved by up to `slack` whole cells per axis."""
    lo, hi = t.min((0, 1)).astype(np.float64), t.max((0, 1)).astype(np.float64)
    out = np.empty_like(t)
    for a in range(3):
        room = (n[a] - 2 * margin - slack[a]) * cell[a]
        x = 1.0 + margin * cell[a] + (t[..., a] - lo[a]) * (room / max(hi[a] - lo[a], 1e-30))
        k = np.floor(x * _Q)
        out[..., a] = (2 * k + 1) / (2 * _Q) + (seed % (slack[a] + 1)) * cell[a]
        seed //= slack[a] + 1
    return np.ascontiguousarray(np.roll(out, seed % 97, axis=0), np.float32).reshape(-1)


def _spec(n, cell, n2):
    s = gpv.GridSpec()
    for a in range(3):
        s.bbox_min[a], s.bbox_max[a] = 1.0, 1.0 + n[a] * cell[a]
        s.ndiv[a], s.ndiv2[a] = n[a], n2[a]
    return s


def _gridded(t, n, n2, seed):
    """A shape in an explicit grid, at least one empty cell on each side."""
    cell = [math.floor(_Q / k) / _Q for k in n]
    slack = [max(1, k // 16) for k in n]
    return _place(t, n, cell, 1, slack, seed), _spec(n, cell, n2)


def _sized(t, count1, count2, seed):
    """A shape in the grid of the reference's own sizing (its divisions follow from the bounds)."""
    ext = (t.max((0, 1)) - t.min((0, 1))).astype(np.float64)
    ext *= 0.99 / ext.max()
    while True:
        mx = [1.0 + e for e in ext]
        n = list(gpv.grid_reference((1.0,) * 3, mx, float(ext.max()), count1, count2).ndiv)
        cell = [math.floor(ext[a] / n[a] * _Q) / _Q for a in range(3)]
        mx = [1.0 + n[a] * cell[a] for a in range(3)]
        size = max(n[a] * cell[a] for a in range(3))
        spec = gpv.grid_reference((1.0,) * 3, mx, size, count1, count2)
        if list(spec.ndiv) == n:
            return _place(t, n, cell, 0.02, [1 if k < 8 else 2 for k in n], seed), spec, size
        ext *= 0.98


def _inputs(case, seed):
    """(triangles float32[9 T], grid, model size for the reference's sizing)"""
    t = _shape(case["mesh"], case["size"], case["shape"])
    if case["kind"] == "object":
        return _sized(t, case["count1"], case["count2"], seed)
    return _gridded(t, (case["nx"], case["ny"], case["nz"]), (case["n2x"], case["n2y"], case["n2z"]), seed) + (1.0,)


def _batch(case, seed):
    """Meshes of three families, triangle counts spread over the logarithm, mixed grids."""
    rng = np.random.default_rng([case["shape"], 78])
    params = []
    for i in range(case["count"]):
        t = math.exp(rng.uniform(math.log(case["tmin"]), math.log(case["tmax"])))
        params.append((("sphere", "torus", "superellipsoid")[int(rng.integers(0, 3))],
                       max(6, int(round(math.sqrt(t / 4.0)))), int(rng.integers(1, 1 << 30)),
                       int(rng.choice([32, 48, 64, 96, 128])), int(rng.choice([2, 4, 8]))))
    with ThreadPoolExecutor(max_workers=min(16, os.cpu_count() or 4)) as ex:
        return list(ex.map(lambda p: _gridded(_shape(*p[:3]), (p[3],) * 3, (p[4],) * 3, seed), params))


# ---- states -----------------------------------------------------------------------------------
class _Array:
    """A device array of the library's, for torch.as_tensor (no copy).  A tensor made from it keeps the
    state that owns the memory alive."""

    def __init__(self, owner, ptr, count, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": kind, "data": (ptr, False),
                                         "version": 3, "strides": None}


_EMPTY = {"|u1": torch.uint8, "<i4": torch.int32, "<f4": torch.float32}


def _tensor(owner, ptr, count, kind):
    if count == 0 or not ptr:
        return torch.empty(0, dtype=_EMPTY[kind], device="cuda")
    return torch.as_tensor(_Array(owner, ptr, count, kind), device="cuda")


def _cells(r):
    return r.spec.ndiv2[0] * r.spec.ndiv2[1] * r.spec.ndiv2[2]


def _counts(r):
    return [r.num_boundary, r.num_level1_inside, r.num_level2_inside, r.num_level2_boundary,
            r.num_pairs, r.work.sat1, r.work.sat2, r.work.ray1, r.work.ray2]


class _Device:
    """Plain calls on device triangles.  The outputs are the context's arrays, valid until the next
    call on the state (which gives them back first, as a caller's loop does)."""

    def __init__(self, case, seed):
        tris, self.spec, _ = _inputs(case, seed)
        self.tris = torch.from_numpy(tris).cuda()
        self.count = tris.size // 9
        self.ctx = gpv.Context(0)
        if case["kind"] == "stencil":
            self.ctx.set_fill(gpv.FILL_STENCIL)
        self.normals = case["kind"] == "normals"
        if self.normals:
            self.ctx.set_normals(gpv.NORMALS_FLOAT)
        self.res = None

    def run(self):
        if self.res is not None:
            self.ctx.release(self.res)
            self.res = None
        r = self.res = self.ctx.voxelize_device(self.tris.data_ptr(), self.count, self.spec,
                                                torch.cuda.current_stream().cuda_stream)
        n1, b, n2 = r.num_level1, r.num_boundary, r.num_boundary * _cells(r)
        out = [_tensor(self, r.level1_inout, n1, "|u1"), _tensor(self, r.level1_prefix, n1, "<i4"),
               _tensor(self, r.boundary_index, b, "<i4"), _tensor(self, r.level2_inout, n2, "|u1")]
        if self.normals:
            out += [_tensor(self, r.level1_normal, 3 * n1, "<f4"), _tensor(self, r.level2_normal, 3 * n2, "<f4")]
        return out + _counts(r)


class _Batch:
    def __init__(self, case, seed):
        meshes = _batch(case, seed)
        self.tris = [torch.from_numpy(t).cuda() for t, _ in meshes]
        self.ptrs = [t.data_ptr() for t in self.tris]
        self.counts = [t.numel() // 9 for t in self.tris]
        self.specs = [s for _, s in meshes]
        self.ctx = gpv.Context(0)
        self.res = None

    def run(self):
        if self.res is not None:
            for r in self.res:
                self.ctx.release(r)
            self.res = None
        res = self.res = self.ctx.voxelize_batch(self.ptrs, self.counts, self.specs,
                                                 torch.cuda.current_stream().cuda_stream)
        # every array of a batch is one block of memory when the meshes' grids leave no gaps
        sizes = [(r.num_level1, r.num_boundary, r.num_boundary * _cells(r)) for r in res]
        out = []
        for field, k, width, kind in (("level1_inout", 0, 1, "|u1"), ("level1_prefix", 0, 4, "<i4"),
                                      ("boundary_index", 1, 4, "<i4"), ("level2_inout", 2, 1, "|u1")):
            at = [getattr(r, field) for r in res]
            if all(at[i] + width * sizes[i][k] == at[i + 1] for i in range(len(at) - 1)):
                out.append(_tensor(self, at[0], sum(s[k] for s in sizes), kind))
            else:
                out.append(torch.cat([_tensor(self, p, s[k], kind) for p, s in zip(at, sizes)]))
        out.append(np.array([(r.num_boundary, r.num_level1_inside, r.num_level2_inside,
                              r.num_level2_boundary) for r in res], np.int64))
        return out


class _Host:
    def __init__(self, case, seed):
        tris, self.spec, _ = _inputs(case, seed)
        self.tris = torch.from_numpy(tris).pin_memory()
        self.count = tris.size // 9
        self.ctx = gpv.Context(0)
        # the buffers' sizes, from a Level1 call
        flat = gpv.GridSpec.from_buffer_copy(self.spec)
        for a in range(3):
            flat.ndiv2[a] = 0
        r = self.ctx.voxelize_host(tris, flat)
        b = r.num_boundary
        n1, n2 = r.num_level1, b * self.spec.ndiv2[0] * self.spec.ndiv2[1] * self.spec.ndiv2[2]
        self.ctx.release(r)
        self.l1 = torch.empty(n1, dtype=torch.uint8, pin_memory=True)
        self.prefix = torch.empty(n1, dtype=torch.int32, pin_memory=True)
        self.index = torch.empty(max(b, 1), dtype=torch.int32, pin_memory=True)
        self.l2 = torch.empty(max(n2, 1), dtype=torch.uint8, pin_memory=True)
        self.n2 = n2

    def run(self):
        _, r = self.ctx.voxelize_to_host(
            self.tris.data_ptr(), self.count, self.spec, self.l1.data_ptr(), self.prefix.data_ptr(),
            self.index.data_ptr(), self.l2.data_ptr(), self.n2, 0, torch.cuda.current_stream().cuda_stream)
        counts = _counts(r)
        self.ctx.release(r)
        return [self.l1, self.prefix, self.index, self.l2] + counts


class _Object:
    def __init__(self, case, seed):
        self.obj = gpv.Object(gpv.Context(0))
        tris, spec, size = _inputs(case, seed)
        self.obj.flatCPUTriangleData = tris
        self.obj.totalNumTriangles = tris.size // 9
        self.obj.bBoxMin = np.array(spec.bbox_min, np.float32)
        self.obj.bBoxMax = np.array(spec.bbox_max, np.float32)
        self.obj.maxModelSize = size
        self.params = gpv.GLParameters(case["count1"], case["count2"], True, False)

    def run(self):
        v = self.obj.PerformVoxelization(self.params)
        return [v.level1InOut, v.boundaryPrefixSum, v.boundaryIndex, v.level2InOut, v.level1Normal,
                v.level2Normal]


class _Noalloc:
    def __init__(self, case, seed):
        tris, self.spec, _ = _inputs(case, seed)
        self.tris = torch.from_numpy(tris).cuda()
        n1 = case["nx"] * case["ny"] * case["nz"]
        self.l1 = torch.zeros(n1, dtype=torch.uint8, device="cuda")
        self.prefix = torch.zeros(n1, dtype=torch.int32, device="cuda")
        self.index = torch.zeros(n1, dtype=torch.int32, device="cuda")

    def run(self):
        b = C.c_int64()
        rc = gpv.lib().gpv_voxelize_level1_noalloc(
            self.tris.data_ptr(), self.tris.numel() // 9, C.byref(self.spec), self.l1.data_ptr(),
            self.prefix.data_ptr(), self.index.data_ptr(), C.byref(b), torch.cuda.current_stream().cuda_stream)
        if rc:
            raise gpv.GpvError(rc, gpv.lib().gpv_noalloc_last_error().decode())
        return [self.l1, self.prefix, self.index[:b.value], b.value]


def _first(seed, n):
    return seed * 7919 % max(n, 1)


class _F3(C.Structure):
    _fields_ = [("x", C.c_float), ("y", C.c_float), ("z", C.c_float)]


class _I3(C.Structure):
    _fields_ = [("x", C.c_int), ("y", C.c_int), ("z", C.c_int)]


class _Shims:
    """The lists that the reference's host code builds between its two levels, then its calls
    CUDAClassifyInOutLevel2 and CUDAClassifyTessellationLevel2 into cleared arrays.  The order of the
    boundary voxels is the caller's: here it starts at a voxel that the seed picks."""

    def __init__(self, case, seed):
        tris, spec, _ = _inputs(case, seed)
        g = _Tables(spec)
        self.tris = torch.from_numpy(tris).cuda()
        voxel, tri = _pairs(self.tris.view(-1, 9), g)  # sorted by (voxel, triangle)
        n1 = g.n[0] * g.n[1] * g.n[2]
        self.index = torch.unique(voxel).to(torch.int32)
        self.index = torch.roll(self.index, -_first(seed, self.index.numel()))
        self.cnt = torch.bincount(voxel, minlength=n1).to(torch.int32)
        self.first = (torch.cumsum(self.cnt, 0) - self.cnt).to(torch.int32)
        self.flat = tri.to(torch.int32)
        ncol, t = g.n[0] * g.n[1], tris.size // 9
        both = torch.unique((voxel % ncol) * t + tri)
        self.xcnt = torch.bincount(both // t, minlength=ncol).to(torch.int32)
        self.xfirst = (torch.cumsum(self.xcnt, 0) - self.xcnt).to(torch.int32)
        self.xflat = (both % t).to(torch.int32)
        v = self.index.long()
        self.mid = torch.stack([g.c1[0][v % g.n[0]], g.c1[1][(v // g.n[0]) % g.n[1]], g.c1[2][v // ncol]], 1).reshape(-1)
        self.b = self.index.numel()
        cells = g.n2[0] * g.n2[1] * g.n2[2]
        self.state = torch.empty(self.b * cells, dtype=torch.float32, device="cuda")
        self.normal = torch.empty(self.b * cells * 4, dtype=torch.float32, device="cuda")
        self.n, self.n2 = _I3(*g.n), _I3(*g.n2)
        self.e1, self.e2 = _F3(*g.e1), _F3(*g.e2)
        L = gpv.lib()
        vp = C.c_void_p
        L.CUDAClassifyTessellationLevel2.argtypes = [vp] * 8 + [C.c_int, _I3, _F3, _F3]
        L.CUDAClassifyInOutLevel2.argtypes = [vp] * 7 + [C.c_int, _I3, _I3, _F3, _F3]
        self.lib = L

    def run(self):
        self.state.zero_()
        self.normal.zero_()
        p = torch.Tensor.data_ptr
        self.lib.CUDAClassifyInOutLevel2(p(self.tris), p(self.state), p(self.mid), p(self.index), p(self.xcnt),
                                         p(self.xfirst), p(self.xflat), self.b, self.n, self.n2, self.e1, self.e2)
        self.lib.CUDAClassifyTessellationLevel2(p(self.tris), p(self.state), p(self.normal), p(self.mid),
                                                p(self.index), p(self.cnt), p(self.first), p(self.flat), self.b,
                                                self.n2, self.e1, self.e2)
        return [self.state, self.normal]


_STATES = {"device": _Device, "level1": _Device, "stencil": _Device, "normals": _Device, "batch": _Batch,
           "host": _Host, "object": _Object, "noalloc": _Noalloc, "shims": _Shims}


def prepare(case, seed):
    return _STATES[case["kind"]](case, seed)


def run(state):
    return state.run()


# ---- work -------------------------------------------------------------------------------------
def work(case):
    return dict(_work(json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)))


@functools.lru_cache(maxsize=None)
def _work(text):
    """Bytes: the triangles read once, every output written once.  Operations: one passing SAT (about
    140 float operations) for each boundary voxel and cell, one ray test (about 50) for each crossing
    of a column or sub-column.  A surface patch meets |n|_1 / h^2 cells of size h per unit of area."""
    case = json.loads(text)
    kind = case["kind"]
    if kind == "batch":
        meshes = _batch(case, 0)
    else:
        meshes = [_inputs(case, 0)[:2]]
    nbytes = flops = 0.0
    for t, spec in meshes:
        v = t.reshape(-1, 3, 3).astype(np.float64)
        area = np.abs(np.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])).sum(0) / 2
        h = [(spec.bbox_max[a] - spec.bbox_min[a]) / spec.ndiv[a] for a in range(3)]
        n1 = spec.ndiv[0] * spec.ndiv[1] * spec.ndiv[2]
        cells = spec.ndiv2[0] * spec.ndiv2[1] * spec.ndiv2[2]

        def met(h):
            return area[0] / (h[1] * h[2]) + area[1] / (h[0] * h[2]) + area[2] / (h[0] * h[1])

        b = min(met(h), n1)
        if kind == "shims":
            nbytes += t.nbytes + 20.0 * b * cells
        else:
            nbytes += t.nbytes + 5.0 * n1 + 4.0 * b + b * cells
            flops += 140 * b + 50 * area[2] / (h[0] * h[1])
        if kind in ("normals", "object"):
            nbytes += 12.0 * (n1 + b * cells)
        if cells:
            h2 = [h[a] / spec.ndiv2[a] for a in range(3)]
            flops += 140 * min(met(h2), b * cells) + 50 * area[2] / (h2[0] * h2[1])
    return {"bytes": nbytes, "flops": flops}


# ---- 64-bit normals ---------------------------------------------------------------------------
# A normal is the mean of the unit face normals of the triangles that meet a voxel or cell, scaled to
# unit length.  Which triangles meet it is decided by the 32-bit Akenine-Moller test in the reference's
# own order of operations (a decision, so it is taken as that test takes it); the sums are in 64 bits.
class _Tables:
    """Divisions, half sizes and centres of a grid (double expressions rounded to float)."""

    def __init__(self, spec):
        f = np.float32
        self.mn, self.mx = [f(v) for v in spec.bbox_min], [f(v) for v in spec.bbox_max]
        self.n, self.n2 = [int(v) for v in spec.ndiv], [int(v) for v in spec.ndiv2]
        self.e1, self.e2, self.c1, self.c2 = [], [], [], []
        for a in range(3):
            g = f(float(self.mx[a] - self.mn[a]) / self.n[a])
            g2 = f(float(g) / max(self.n2[a], 1))
            self.e1.append(float(f(float(g) / 2)))
            self.e2.append(float(f(float(g2) / 2)))
            mid = ((np.arange(self.n[a]) + 0.5) * self.e1[a] * 2 + float(self.mn[a])).astype(f)
            sub = (np.arange(max(self.n2[a], 1)) + 0.5) * float(g2)
            c2 = (sub[None, :] + mid[:, None].astype(np.float64) - self.e1[a]).astype(f)
            self.c1.append(torch.from_numpy(mid).cuda())
            self.c2.append(torch.from_numpy(c2).cuda())


def _apart(a, b, rad):
    return (torch.minimum(a, b) > rad) | (torch.maximum(a, b) < -rad)


def _meets(t, c, h):
    """The SAT of triangles t [N, 9] against boxes of centres c (three [N]) and half sizes h."""
    v = [[t[:, 3 * i + a] - c[a] for a in range(3)] for i in range(3)]
    e = [[v[(i + 1) % 3][a] - v[i][a] for a in range(3)] for i in range(3)]
    ok = torch.ones(t.shape[0], dtype=torch.bool, device=t.device)
    for a in range(3):
        lo = torch.minimum(torch.minimum(v[0][a], v[1][a]), v[2][a])
        hi = torch.maximum(torch.maximum(v[0][a], v[1][a]), v[2][a])
        ok &= ~((lo > h[a]) | (hi < -h[a]))
    for i, xs, ys, zs in ((0, (0, 2), (0, 2), (1, 2)), (1, (0, 2), (0, 2), (0, 1)), (2, (0, 1), (0, 1), (1, 2))):
        ex, ey, ez = e[i]
        fx, fy, fz = ex.abs(), ey.abs(), ez.abs()
        p = [ez * v[k][1] - ey * v[k][2] for k in xs]
        ok &= ~_apart(p[0], p[1], fz * h[1] + fy * h[2])
        p = [-ez * v[k][0] + ex * v[k][2] for k in ys]
        ok &= ~_apart(p[0], p[1], fz * h[0] + fx * h[2])
        p = [ey * v[k][0] - ex * v[k][1] for k in zs]
        ok &= ~_apart(p[0], p[1], fy * h[0] + fx * h[1])
    n = [e[0][1] * e[1][2] - e[0][2] * e[1][1], e[0][2] * e[1][0] - e[0][0] * e[1][2],
         e[0][0] * e[1][1] - e[0][1] * e[1][0]]
    lo, hi = [], []
    for a in range(3):
        up = n[a] > 0
        lo.append(n[a] * torch.where(up, -h[a] - v[0][a], h[a] - v[0][a]))
        hi.append(n[a] * torch.where(up, h[a] - v[0][a], -h[a] - v[0][a]))
    return ok & ~(lo[0] + lo[1] + lo[2] > 0) & (hi[0] + hi[1] + hi[2] >= 0)


def _spread(counts, limit=1 << 23):
    """(row, position within the row) of counts[row] items each, in pieces of about `limit` items."""
    end = torch.cumsum(counts, 0)
    a, n = 0, counts.numel()
    while a < n:
        base = int(end[a - 1]) if a else 0
        b = max(a + 1, int(torch.searchsorted(end, base + limit, right=True)))
        c = counts[a:b]
        row = torch.repeat_interleave(torch.arange(a, b, device=c.device), c)
        start = torch.repeat_interleave(end[a:b] - c - base, c)
        yield row, torch.arange(row.numel(), device=c.device) - start
        a = b


def _pairs(t, g):
    """(voxel, triangle) of every triangle recorded in a Level1 voxel, sorted."""
    lo, hi = [], []
    for a in range(3):
        cells = []
        for k in range(3):
            q = (t[:, 3 * k + a] - float(g.mn[a])) / float(g.mx[a] - g.mn[a]) * float(g.n[a])
            c = q.clamp(-1, g.n[a] + 1).to(torch.int64)
            cells.append(torch.where((c == g.n[a]) & (t[:, 3 * k + a] == float(g.mx[a])), c - 1, c))
        c = torch.stack(cells)
        lo.append(c.min(0).values.clamp(min=0))
        hi.append(c.max(0).values.clamp(max=g.n[a] - 1))
    n = [(hi[a] - lo[a] + 1).clamp(min=0) for a in range(3)]
    voxels, ids = [], []
    for row, at in _spread(n[0] * n[1] * n[2]):
        i = lo[0][row] + at % n[0][row]
        j = lo[1][row] + at // n[0][row] % n[1][row]
        k = lo[2][row] + at // (n[0][row] * n[1][row])
        ok = _meets(t[row], (g.c1[0][i], g.c1[1][j], g.c1[2][k]), g.e1)
        voxels.append(((k * g.n[1] + j) * g.n[0] + i)[ok])
        ids.append(row[ok])
    key = torch.sort(torch.cat(voxels) * t.shape[0] + torch.cat(ids)).values
    return key // t.shape[0], key % t.shape[0]


def _unit(v):
    m = v.square().sum(1, keepdim=True).sqrt()
    return torch.where(m > 0, v / m, v)


def _face_normals(t):
    d = t.double()
    return _unit(torch.linalg.cross(d[:, 3:6] - d[:, 0:3], d[:, 6:9] - d[:, 0:3]))


def _cell_sums(t, g, voxel, tri, face):
    """Sums of the face normals and counts per Level2 cell of the boundary voxels (index order)."""
    index = torch.unique(voxel)
    rank = torch.searchsorted(index, voxel)
    cells = g.n2[0] * g.n2[1] * g.n2[2]
    sums = torch.zeros(index.numel() * cells, 4, dtype=torch.float64, device=t.device)
    for row, at in _spread(torch.full_like(voxel, cells)):
        p, q, r = at % g.n2[0], at // g.n2[0] % g.n2[1], at // (g.n2[0] * g.n2[1])
        v = voxel[row]
        i, j, k = v % g.n[0], v // g.n[0] % g.n[1], v // (g.n[0] * g.n[1])
        ok = _meets(t[tri[row]], (g.c2[0][i, p], g.c2[1][j, q], g.c2[2][k, r]), g.e2)
        f = face[tri[row[ok]]]
        sums.index_add_(0, (rank[row] * cells + at)[ok], torch.cat([f, torch.ones_like(f[:, :1])], 1))
    return sums


def exact(case, seed):
    if case["kind"] not in ("normals", "object", "shims"):
        return None  # states, indices and counts: decisions, compared as they are
    tris, spec, _ = _inputs(case, seed)
    g = _Tables(spec)
    t = torch.from_numpy(tris).cuda().view(-1, 9)
    face = _face_normals(t)
    voxel, tri = _pairs(t, g)
    cell = _cell_sums(t, g, voxel, tri, face)
    if case["kind"] == "shims":
        b = torch.unique(voxel).numel()
        return [None, torch.roll(cell.view(b, -1), -_first(seed, b), 0).reshape(-1)]
    level1 = torch.zeros(g.n[0] * g.n[1] * g.n[2], 4, dtype=torch.float64, device=t.device)
    f = face[tri]
    level1.index_add_(0, voxel, torch.cat([f, torch.ones_like(f[:, :1])], 1))
    mean = [_unit(s[:, :3] / s[:, 3:].clamp(min=1)) for s in (level1, cell)]
    if case["kind"] == "object":
        return [None] * 4 + mean
    return [None] * 4 + [m.reshape(-1) for m in mean] + [None] * 9
