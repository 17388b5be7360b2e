"""What this framework is timed on: the calls a user's program makes, from the smallest grid to the largest.

A case is a dict of plain values; ``prepare`` makes what a program has in hand (fields, grids, plans, caller-held
outputs), ``run`` is one pass through the public entry points, ``exact`` the same outputs in 64 bits by torch alone.
Fields are the Gaussian blobs of ``daxtoolkit_gb300.synthetic`` and, for the reference's own benchmarks, the
magnitude of the coordinates and the Mandelbulb.  A case fixes the shape of its field and so the sizes of its results;
the seed draws a noise on every value that takes no point across the isovalue or out of its interval, so that every
position, weight and gradient is another one.
"""
import ctypes
import math

import numpy as np
import torch

from daxtoolkit_gb300 import capi, cont, synthetic

DEV = "cuda"


def listed():
    return [
        # a probe or an interactive slider on a tiny block: launches and the size read are all there is
        dict(name="mc_tiny", kind="mc", nx=33, ny=29, nz=26, api="call", merge=True, iso=0.5),
        # the reference's MarchingCubes benchmark at its default size, points not merged
        dict(name="mc_bench_128", kind="mc_bench", n=128, merge=False),
        # one frame of an in-situ visualisation at the headline size, outputs held by the caller
        dict(name="mc_frame_512", kind="mc", nx=512, ny=512, nz=512, api="frame", merge=True, iso=0.5),
        # count, generate and CompactPointField of a vector field through the dispatchers, ragged extents
        dict(name="mc_dispatch_ragged", kind="mc", nx=301, ny=257, nz=199, api="dispatch", merge=True, iso=0.4),
        # a material interval cut out of a simulation volume, with the field carried along
        dict(name="threshold_512", kind="threshold", nx=512, ny=512, nz=512, lo=0.3, hi=0.7),
        # an oblique cutting plane through a volume of odd extents
        dict(name="slice_ragged", kind="slice", nx=383, ny=405, nz=331, merge=True),
        # one optimisation step: surface and cell gradients forward, the field's gradient backward
        dict(name="adjoint_step", kind="adjoint", nx=385, ny=321, nz=289, iso=0.5),
        # the same step over a set of uneven blocks (an AMR level), one launch per pass for all of them
        dict(name="batch_step_32", kind="batch", count=32, lo=64, hi=160, noise=0.0),
        # sorting a large point or edge list with its payload
        dict(name="sort_pairs_100m", kind="sort", n=100_000_000, key="int32", words=1, descending=False),
        # offsets from counts and the compaction they drive, over a long array
        dict(name="scan_compact_100m", kind="scan_compact", n=100_000_000, key="int32", words=1, density=0.3),
        # marching tetrahedra on an unstructured mesh of 83 million cells, points merged
        dict(name="mt_merged_256", kind="mt", nx=256, ny=256, nz=256, merge=True, iso=0.5),
        # the Mandelbulb demo at its default size: the next volume, surface and cut of this one, normals and colours
        dict(name="mandelbulb_200", kind="mandelbulb", n=200, cut=0.8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi):
    """Three extents of one drawn scale, each up to a third away from it."""
    n = _log_int(rng, lo, hi)
    return {a: max(lo, min(hi, int(round(n * rng.uniform(0.75, 1.33))))) for a in ("nx", "ny", "nz")}


def draw(rng):
    kind = rng.choice(["mc", "mc", "mc_bench", "threshold", "slice", "adjoint", "batch", "sort", "sort", "scan_compact",
                       "mt", "mandelbulb"])
    if kind == "mc":
        return dict(kind=kind, **_dims(rng, 24, 512), api=rng.choice(["call", "frame", "dispatch"]),
                    merge=rng.random() < 0.7, iso=round(rng.uniform(0.3, 0.7), 3))
    if kind == "mc_bench":
        return dict(kind=kind, n=_log_int(rng, 110, 400), merge=rng.random() < 0.5)
    if kind == "threshold":
        lo = round(rng.uniform(0.1, 0.5), 3)
        return dict(kind=kind, **_dims(rng, 24, 512), lo=lo, hi=round(lo + rng.uniform(0.1, 0.4), 3))
    if kind == "slice":
        return dict(kind=kind, **_dims(rng, 24, 512), merge=rng.random() < 0.7)
    if kind == "adjoint":
        return dict(kind=kind, **_dims(rng, 24, 384), iso=round(rng.uniform(0.3, 0.7), 3))
    if kind == "batch":
        return dict(kind=kind, count=_log_int(rng, 4, 48), lo=32, hi=_log_int(rng, 64, 160), noise=rng.choice([0.0, 0.01]))
    if kind == "sort":
        return dict(kind=kind, n=_log_int(rng, 1000, 60_000_000), key=rng.choice(["int32", "float32", "int64"]),
                    words=rng.choice([0, 1, 3]), descending=rng.random() < 0.3)
    if kind == "scan_compact":
        return dict(kind=kind, n=_log_int(rng, 1000, 100_000_000), key=rng.choice(["int32", "float32", "int64"]),
                    words=rng.choice([0, 1, 3]), density=round(rng.uniform(0.05, 0.9), 2))
    if kind == "mt":
        return dict(kind=kind, **_dims(rng, 24, 240), merge=rng.random() < 0.7, iso=round(rng.uniform(0.3, 0.7), 3))
    return dict(kind=kind, n=_log_int(rng, 48, 220), cut=round(rng.uniform(0.55, 0.95), 2))


# ---- inputs -----------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _noisy(field, seed, amp, lo, hi=math.inf):
    """The field with noise of up to amp on its values; a value that would change sides of (lo, hi] or [lo, hi] stays."""
    f = field + amp * (2 * torch.rand(field.shape, generator=_generator(seed), device=DEV) - 1)
    lo, hi = (torch.tensor(v, dtype=torch.float32, device=DEV) for v in (lo, hi))
    same = ((f > lo) == (field > lo)) & ((f >= lo) == (field >= lo)) & ((f > hi) == (field > hi)) & ((f >= hi) == (field >= hi))
    return torch.where(same, f, field)


def _field(dims, seed, lo, hi=math.inf, blobs=20260101, rough=0.0):
    """Blobs (rough: with noise that is part of the shape, the same for every seed), then the seed's noise."""
    f = synthetic.blob_field(dims, seed=blobs, device=DEV)
    if rough:
        f += rough * (2 * torch.rand(f.shape, generator=_generator(blobs), device=DEV) - 1)
    return _noisy(f, seed, 0.002, lo, hi)


def _unit_grid(dims):
    return cont.UniformGrid(dims, spacing=tuple(1.0 / (n - 1) for n in dims))


def _case_dims(case):
    return (case["nx"], case["ny"], case["nz"])


def _slice(case, seed):
    """Grid and plane of a slice.  The seed draws the unit of length, a power of two, which leaves every sign as it is."""
    rng = np.random.default_rng(sum(_case_dims(case)))
    normal = rng.uniform(0.2, 1.0, size=3) * rng.choice([-1.0, 1.0], size=3)
    unit = 2.0 ** (int(seed) % 41 - 20)
    grid = cont.UniformGrid(_case_dims(case), spacing=tuple(unit / (n - 1) for n in _case_dims(case)))
    # the reference's plane is dot(N, x - O) = dot(N, O): it passes through 2 O
    return (grid, tuple(float(v * unit) for v in rng.uniform(0.2, 0.3, size=3)),
            tuple(float(v) for v in normal / np.linalg.norm(normal)))


def _batch(case, seed):
    dims = synthetic.batch_grid_dims(case["count"], case["lo"], case["hi"], 20 + case["count"])
    isos = synthetic.batch_isovalues(case["count"], 0.3, 0.6, 20 + case["count"])
    fields = [_field(d, seed + i, isos[i], blobs=100 + i, rough=case["noise"]) for i, d in enumerate(dims)]
    return dims, fields, isos


def _sort_inputs(case, seed):
    g = _generator(seed)
    n = case["n"]
    if case["key"] == "float32":
        keys = torch.randn(n, generator=g, device=DEV)
    elif case["key"] == "int32":
        keys = torch.randint(-2 ** 31, 2 ** 31 - 1, (n,), generator=g, device=DEV, dtype=torch.int32)
    else:
        keys = torch.randint(-2 ** 62, 2 ** 62, (n,), generator=g, device=DEV, dtype=torch.int64)
    vals = torch.arange(n * case["words"], dtype=torch.int32, device=DEV) if case["words"] else None
    if vals is not None and case["words"] > 1:
        vals = vals.reshape(n, case["words"])
    return keys, vals


def _scan_inputs(case, seed):
    g = _generator(seed)
    n = case["n"]
    stencil = (torch.rand(n, generator=_generator(n), device=DEV) < case["density"]).to(torch.int32)
    counts = stencil * torch.randint(1, 6, (n,), generator=g, device=DEV, dtype=torch.int32)
    if case["key"] == "float32":
        counts = counts * torch.rand(n, generator=g, device=DEV)
    elif case["key"] == "int64":
        counts = counts.to(torch.int64) * 3_000_000_019
    values = torch.rand(n * case["words"], generator=g, device=DEV) if case["words"] else None
    if values is not None and case["words"] > 1:
        values = values.reshape(n, case["words"])
    return counts, stencil, values


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind == "mc":
        dims = _case_dims(case)
        s.update(grid=_unit_grid(dims), field=_field(dims, seed, case["iso"]))
        if case["api"] == "frame":  # a frame loop holds its outputs and its scratch
            out = cont.marching_cubes(s["grid"], s["field"], case["iso"], merge=case["merge"])
            s.update(verts=torch.zeros_like(out["verts"]), conn=torch.zeros_like(out["conn"]), scratch=cont.Scratch())
        elif case["api"] == "dispatch":
            s["velocity"] = torch.rand((len(s["field"]), 3), generator=_generator(seed + 1), device=DEV)
    elif kind == "mc_bench":
        s["grid"] = cont.UniformGrid((case["n"],) * 3)
        s["field"] = _noisy(cont.point_magnitude(s["grid"]), seed, 0.2, 100.0)
    elif kind == "threshold":
        dims = _case_dims(case)
        s.update(grid=_unit_grid(dims), field=_field(dims, seed, case["lo"], case["hi"]))
    elif kind == "slice":
        s["grid"], s["origin"], s["normal"] = _slice(case, seed)
    elif kind == "adjoint":
        dims = _case_dims(case)
        s.update(grid=_unit_grid(dims), field=_field(dims, seed, case["iso"]), scratch=cont.Scratch())
    elif kind == "batch":
        dims, fields, isos = _batch(case, seed)
        s["plan"] = cont.MarchingCubesBatch([_unit_grid(d) for d in dims], fields, isos)
    elif kind == "sort":
        s["keys"], s["vals"] = _sort_inputs(case, seed)
        s["k"] = torch.empty_like(s["keys"])
        s["v"] = None if s["vals"] is None else torch.empty_like(s["vals"])
    elif kind == "scan_compact":
        s["counts"], s["stencil"], s["values"] = _scan_inputs(case, seed)
        s["scan"] = torch.empty_like(s["counts"])
    elif kind == "mt":
        dims = _case_dims(case)
        s.update(mesh=cont.tetrahedralize(_unit_grid(dims)), field=_field(dims, seed, case["iso"]))
    elif kind == "mandelbulb":  # the volume on display, and where the next one of a slow pan lies
        n = case["n"]
        vol = cont.compute_mandlebulb((-1.0,) * 3, (2.0 / n,) * 3, (n, n, n))
        s["volume"] = cont.MandlebulbVolume(vol.Grid, _noisy(vol.EscapeIteration, seed, 0.3, 3.5))
        s["next"] = tuple(float(v) for v in -1.0 + np.random.default_rng(seed).uniform(0.0, 0.5 / n, size=3))
    return s


# ---- one pass ---------------------------------------------------------------

def _run_mc(s):
    if s["api"] == "frame":
        cont.marching_cubes_pipelined(s["grid"], s["field"], s["iso"], s["verts"], s["conn"], merge=s["merge"],
                                      scratch=s["scratch"], read_sizes=False)
        return dict(verts=s["verts"], conn=s["conn"])
    if s["api"] == "call":
        return cont.marching_cubes(s["grid"], s["field"], s["iso"], merge=s["merge"])
    count = cont.DispatcherMapCell(cont.MarchingCubesCount(s["iso"])).Invoke(s["grid"], s["field"])
    d = cont.DispatcherGenerateInterpolatedCells(count, cont.MarchingCubesGenerate(s["iso"]))
    d.SetRemoveDuplicatePoints(s["merge"])
    mesh = d.Invoke(s["grid"], s["field"])
    return dict(verts=mesh.GetPointCoordinates(), conn=mesh.GetCellConnections(), count=count,
                velocity=d.CompactPointField(s["velocity"]))


def _run_adjoint(s):
    """Loss = (|vertices|^2 + |cell gradients|^2) / 2, so its derivatives are the outputs themselves."""
    grid, field, iso = s["grid"], s["field"], s["iso"]
    out = cont.marching_cubes(grid, field, iso, merge=True, scratch=s["scratch"])
    grad = cont.cell_gradient(grid, field)
    dfield = torch.empty_like(field)
    g = grid.desc()
    nbytes = capi.lib().dax_gb300_mc_scratch_bytes(ctypes.byref(g))
    buf = s["scratch"].get(nbytes)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    capi.call("dax_gb300_field_adjoint", ctypes.byref(g), p(field), iso, p(buf), buf.numel(), p(out["verts"]), p(grad),
              p(dfield), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return dict(verts=out["verts"], conn=out["conn"], grad=grad, dfield=dfield)


def _run_batch(s):
    plan = s["plan"]
    verts, conn, tri, vert = plan.run(merge=True)
    grad = plan.cell_gradient()
    dfield = plan.field_adjoint(verts, grad)
    return dict(verts=verts, conn=conn, tri=np.asarray(tri), vert=np.asarray(vert), grad=grad, dfield=dfield)


def _run_mandelbulb(s):
    n, vol = s["n"], s["volume"]
    out = dict(field=cont.compute_mandlebulb(s["next"], (2.0 / n,) * 3, (n, n, n)).EscapeIteration)
    for name, surf in (("surface", cont.extract_surface(vol, 3.5)), ("cut", cont.extract_cut(vol, s["cut"], 3.5))):
        out[name] = dict(verts=surf.Data.GetPointCoordinates(), conn=surf.Data.GetCellConnections(), norms=surf.Norms,
                         colors=surf.Colors)
    return out


def run(state):
    s = state
    kind = s["kind"]
    if kind == "mc":
        return _run_mc(s)
    if kind == "mc_bench":
        return cont.marching_cubes(s["grid"], s["field"], 100.0, merge=s["merge"])
    if kind == "threshold":
        return cont.threshold(s["grid"], s["field"], s["lo"], s["hi"])
    if kind == "slice":
        return cont.slice(s["grid"], s["origin"], s["normal"], merge=s["merge"])
    if kind == "adjoint":
        return _run_adjoint(s)
    if kind == "batch":
        return _run_batch(s)
    if kind == "sort":  # the sort is in place: a program that keeps its list sorts a copy
        keys = cont.Algorithm.Copy(s["keys"], s["k"])
        vals = None if s["vals"] is None else cont.Algorithm.Copy(s["vals"], s["v"])
        cont.Algorithm.SortByKey(keys, vals, cont.SortGreater() if s["descending"] else None)
        return dict(keys=keys, vals=vals)
    if kind == "scan_compact":
        total, scan = cont.Algorithm.ScanExclusive(s["counts"], s["scan"])
        kept = cont.Algorithm.StreamCompact(s["stencil"]) if s["values"] is None else \
            cont.Algorithm.StreamCompact(s["values"], s["stencil"])
        return dict(total=total, scan=scan, kept=kept)
    if kind == "mt":
        return cont.marching_tetrahedra(s["mesh"], s["field"], s["iso"], merge=s["merge"])
    return _run_mandelbulb(s)


# ---- what a pass cannot do without -------------------------------------------

def work(case):
    """Inputs read once and outputs written once.  Surface sizes are those of the blob fields: about 4.2 n^2 triangles
    on n^3 points, half as many merged vertices."""
    kind = case["kind"]
    if kind in ("mc", "threshold", "slice", "adjoint", "mt"):
        nx, ny, nz = _case_dims(case)
        P, C = nx * ny * nz, (nx - 1) * (ny - 1) * (nz - 1)
        T = 4.2 * P ** (2 / 3)
    if kind == "mc":
        V = T / 2 if case["merge"] else 3 * T
        extra = 4 * C + 24 * V + 12 * V if case["api"] == "dispatch" else 0
        return dict(bytes=4 * P + 12 * V + 12 * T + extra, flops=3 * C + 20 * V)
    if kind == "mc_bench":
        P, T = case["n"] ** 3, 47_000
        V = T / 2 if case["merge"] else 3 * T
        return dict(bytes=4 * P + 12 * V + 12 * T, flops=3 * P + 20 * V)
    if kind == "threshold":
        K = 0.25 * (case["hi"] - case["lo"]) * C
        return dict(bytes=4 * P + 32 * K + 16 * 1.04 * K, flops=2 * P)
    if kind == "slice":
        T = 4.0 * P ** (2 / 3)
        V = T / 2 if case["merge"] else 3 * T
        return dict(bytes=12 * V + 12 * T, flops=20 * V)
    if kind == "adjoint":  # field in, surface and gradients out and in again, dfield out
        return dict(bytes=8 * P + 24 * C + 12 * T + 12 * T, flops=60 * C + 40 * T)
    if kind == "batch":
        P = C = T = 0
        for nx, ny, nz in synthetic.batch_grid_dims(case["count"], case["lo"], case["hi"], 20 + case["count"]):
            P, C = P + nx * ny * nz, C + (nx - 1) * (ny - 1) * (nz - 1)
            T += 4.2 * (nx * ny * nz) ** (2 / 3)
        return dict(bytes=8 * P + 24 * C + 24 * T, flops=60 * C + 40 * T)
    if kind == "sort":
        row = (8 if case["key"] == "int64" else 4) + 4 * case["words"]
        return dict(bytes=2 * row * case["n"], flops=case["n"])
    if kind == "scan_compact":
        row = 8 if case["key"] == "int64" else 4
        kept = case["density"] * case["n"] * max(4, 4 * case["words"])
        return dict(bytes=(2 * row + 4) * case["n"] + kept * (2 if case["words"] else 1), flops=case["n"])
    if kind == "mt":
        V = T if case["merge"] else 3 * T
        return dict(bytes=80 * C + 4 * P + 12 * V + 12 * 3.3 * T, flops=15 * C + 20 * V)
    P, T = (case["n"] + 1) ** 3, 37.0 * (case["n"] + 1) ** 2
    # per point about ten escape iterations of two arctangents, a power, three sines, a tangent
    return dict(bytes=4 * P + 2 * T * (36 + 12 + 36 + 12), flops=10 * 150 * P)


# ---- the same in 64 bits -------------------------------------------------------

def _axes(origin, spacing, dims):
    """The grid's float32 point coordinates per axis, widened."""
    f = lambda v: torch.tensor(v, dtype=torch.float32, device=DEV)  # noqa: E731
    return [(f(origin[a]) + f(spacing[a]) * torch.arange(dims[a], device=DEV, dtype=torch.float32)).double() for a in range(3)]


def _surface64(inside, values, iso, axes):
    """Merged vertices in (owner point, axis) order, and their end points A and B and weights; values: float64 [P]."""
    nz, ny, nx = inside.shape
    cross = torch.zeros((nz, ny, nx, 3), dtype=torch.bool, device=DEV)
    cross[:, :, :-1, 0] = inside[:, :, 1:] != inside[:, :, :-1]
    cross[:, :-1, :, 1] = inside[:, 1:] != inside[:, :-1]
    cross[:-1, :, :, 2] = inside[1:] != inside[:-1]
    e = cross.reshape(-1).nonzero().squeeze(1)
    a, axis = e // 3, e % 3
    b = a + torch.tensor([1, nx, nx * ny], device=DEV)[axis]
    w = (iso - values[a]) / (values[b] - values[a])
    xyz = lambda p: torch.stack([axes[0][p % nx], axes[1][p // nx % ny], axes[2][p // (nx * ny)]], dim=1)  # noqa: E731
    ca = xyz(a)
    return ca + w[:, None] * (xyz(b) - ca), a, b, w


def _gradient64(f3, axes):
    """Cell gradients [C, 3] of the float64 field [nz, ny, nx]."""
    out = []
    for a, dim in ((0, 2), (1, 1), (2, 0)):
        d = f3.diff(dim=dim)
        for other in range(3):
            if other != dim:
                n = d.shape[other]
                d = d.narrow(other, 0, n - 1) + d.narrow(other, 1, n - 1)
        shape = [1, 1, 1]
        shape[dim] = -1
        out.append(0.25 * d / axes[a].diff().reshape(shape))
    return torch.stack(out, dim=3).reshape(-1, 3)


def _adjoint64(field, dims, iso, axes):
    """Vertices, cell gradients and dL/dfield of the loss of _run_adjoint."""
    nx, ny, nz = dims
    f = field.double()
    f3 = f.reshape(nz, ny, nx)
    iso32 = torch.tensor(iso, dtype=torch.float32, device=DEV)
    verts, a, b, w = _surface64(field.reshape(nz, ny, nx) > iso32, f, float(iso32), axes)
    grad = _gradient64(f3, axes)
    xyz = lambda p: torch.stack([axes[0][p % nx], axes[1][p // nx % ny], axes[2][p // (nx * ny)]], dim=1)  # noqa: E731
    dw = (verts * (xyz(b) - xyz(a))).sum(1)  # dL/dvertex is the vertex itself
    d = f[b] - f[a]
    df = torch.zeros_like(f)
    df.index_add_(0, a, dw * (w - 1) / d)
    df.index_add_(0, b, -dw * w / d)
    df3 = df.reshape(nz, ny, nx)
    g4 = grad.reshape(nz - 1, ny - 1, nx - 1, 3)
    for c, dim in ((0, 2), (1, 1), (2, 0)):  # dL/dgradient is the gradient itself
        shape = [1, 1, 1]
        shape[dim] = -1
        t = 0.25 * g4[..., c] / axes[c].diff().reshape(shape)
        for k in (0, 1):
            for j in (0, 1):
                for i in (0, 1):
                    sign = (1.0, -1.0)[(i, j, k)[c] == 0]
                    df3[k:nz - 1 + k, j:ny - 1 + j, i:nx - 1 + i] += sign * t
    return verts, grad, df


def _exact_threshold(field, dims, lo, hi, axes):
    nx, ny, nz = dims
    f3 = field.reshape(nz, ny, nx)
    t = lambda v: torch.tensor(v, dtype=torch.float32, device=DEV)  # noqa: E731
    ok = (f3 >= t(lo)) & (f3 <= t(hi))
    kept = ok[1:] & ok[:-1]
    kept = kept[:, 1:] & kept[:, :-1]
    kept = kept[:, :, 1:] & kept[:, :, :-1]
    used = torch.zeros_like(ok)
    for k in (0, 1):
        for j in (0, 1):
            for i in (0, 1):
                used[k:nz - 1 + k, j:ny - 1 + j, i:nx - 1 + i] |= kept
    p = used.reshape(-1).nonzero().squeeze(1)
    coords = torch.stack([axes[0][p % nx], axes[1][p // nx % ny], axes[2][p // (nx * ny)]], dim=1)
    return dict(conn=None, coords=coords, field=field.double()[p])


#: The reference's split of a voxel into five tetrahedra (corners in voxel order), for even cell ids and for odd ones.
SPLIT = (((2, 1, 5, 0), (0, 2, 3, 7), (2, 5, 6, 7), (0, 7, 4, 5), (0, 2, 7, 5)),
         ((1, 3, 6, 2), (0, 1, 3, 4), (1, 4, 5, 6), (3, 6, 7, 4), (1, 4, 6, 3)))


def _tets(dims):
    """The mesh of tetrahedralize, [5 C, 4], by torch."""
    nx, ny, nz = dims
    c = torch.arange((nx - 1) * (ny - 1) * (nz - 1), device=DEV)
    first = c % (nx - 1) + nx * (c // (nx - 1) % (ny - 1) + ny * (c // ((nx - 1) * (ny - 1))))
    corner = torch.tensor([0, 1, nx + 1, nx, nx * ny, nx * ny + 1, nx * ny + nx + 1, nx * ny + nx], device=DEV)
    return (first[:, None, None] + corner[torch.tensor(SPLIT, device=DEV)][c % 2]).reshape(-1, 4)


def _exact_mt(case, seed):
    dims = _case_dims(case)
    field = _field(dims, seed, case["iso"])
    conn = _tets(dims)
    axes = _axes((0.0, 0.0, 0.0), tuple(1.0 / (n - 1) for n in dims), dims)
    z, y, x = torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    pts = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], dim=1)
    iso32 = torch.tensor(case["iso"], dtype=torch.float32, device=DEV)
    inside = field > iso32
    keys = []
    for i, j in ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)):
        at = (inside[conn[:, i]] != inside[conn[:, j]]).nonzero().squeeze(1)
        u, v = conn[at, i].long(), conn[at, j].long()
        keys.append(torch.unique(torch.minimum(u, v) * len(field) + torch.maximum(u, v)))
    keys = torch.unique(torch.cat(keys))
    a, b = keys // len(field), keys % len(field)
    f = field.double()
    w = (float(iso32) - f[a]) / (f[b] - f[a])
    return dict(verts=pts[a] + w[:, None] * (pts[b] - pts[a]), conn=None)


def exact(case, seed):
    kind = case["kind"]
    if kind == "mc" and case["merge"]:
        dims = _case_dims(case)
        field = _field(dims, seed, case["iso"])
        grid = _unit_grid(dims)
        iso32 = torch.tensor(case["iso"], dtype=torch.float32, device=DEV)
        verts, a, b, w = _surface64(field.reshape(dims[::-1]) > iso32, field.double(), float(iso32),
                                    _axes(grid.Origin, grid.Spacing, dims))
        if case["api"] != "dispatch":
            return dict(verts=verts, conn=None)
        vel = torch.rand((len(field), 3), generator=_generator(seed + 1), device=DEV).double()
        return dict(verts=verts, conn=None, count=None, velocity=vel[a] + w[:, None] * (vel[b] - vel[a]))
    if kind == "threshold":
        dims = _case_dims(case)
        grid = _unit_grid(dims)
        return _exact_threshold(_field(dims, seed, case["lo"], case["hi"]), dims, case["lo"], case["hi"],
                                _axes(grid.Origin, grid.Spacing, dims))
    if kind == "adjoint":
        dims = _case_dims(case)
        grid = _unit_grid(dims)
        verts, grad, df = _adjoint64(_field(dims, seed, case["iso"]), dims, case["iso"],
                                     _axes(grid.Origin, grid.Spacing, dims))
        return dict(verts=verts, conn=None, grad=grad, dfield=df)
    if kind == "batch":
        parts = []
        for d, field, iso in zip(*_batch(case, seed)):
            grid = _unit_grid(d)
            parts.append(_adjoint64(field, d, iso, _axes(grid.Origin, grid.Spacing, d)))
        verts, grad, df = (torch.cat(x) for x in zip(*parts))
        return dict(verts=verts, conn=None, tri=None, vert=None, grad=grad, dfield=df)
    if kind == "sort" and case["key"] == "float32":
        return dict(keys=_sort_inputs(case, seed)[0].double().sort(descending=case["descending"])[0], vals=None)
    if kind == "scan_compact":
        counts, stencil, values = _scan_inputs(case, seed)
        kept = None if values is None else values[stencil != 0].double()
        if case["key"] != "float32":
            return dict(total=None, scan=None, kept=kept)
        c = counts.double().cumsum(0)
        return dict(total=float(c[-1]), scan=c - counts.double(), kept=kept)
    if kind == "mt" and case["merge"]:
        return _exact_mt(case, seed)
    if kind == "slice" and case["merge"]:
        grid, origin, normal = _slice(case, seed)
        axes = _axes(grid.Origin, grid.Spacing, grid.dims)
        o, n = (torch.tensor(v, dtype=torch.float32, device=DEV) for v in (origin, normal))
        t = [n[a] * (axes[a].float() - o[a]) for a in range(3)]  # which side, as float32 sums say
        iso = n[0] * o[0] + n[1] * o[1] + n[2] * o[2]
        inside = (t[0][None, None, :] + t[1][None, :, None]) + t[2][:, None, None] > iso
        t = [n[a].double() * (axes[a] - o[a].double()) for a in range(3)]
        values = (t[0][None, None, :] + t[1][None, :, None]) + t[2][:, None, None]
        return dict(verts=_surface64(inside, values.reshape(-1), float((n.double() * o.double()).sum()), axes)[0], conn=None)
    # triangle soups need the case table, and the escape iteration is chaotic on the fractal's boundary: they are held
    # to the bounds of their types
    return None
