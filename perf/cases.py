"""The work a user of this framework has it do, through its public entry points.

Ten kinds of call, each over a range of sizes, value types and modes:

  extract   kvsmc_extract_device on a resident volume: one isosurface
  mapper    the MarchingCubes class on a host array: the drop-in's whole call
  sweep     kvsmc_extract_batch: many isovalues of one resident volume
  plan      a replayed kvsmc_plan over many volumes of uneven size and type
  frame     a field that arrives as a device array, extracted once and dropped
  slice     kvsmc_slice_extract_device: one oblique plane through a volume
  cells     kvsmc_marching_cells_device / _sweep_device: unstructured meshes
  stl       kvsmc_stl_records: a device mesh serialised for a binary STL file

Volumes are (nx, ny, nz) nodes, x fastest.  "fields": fbm is 5-octave
gradient noise in [0, 1]; blobs are Gaussians plus noise; phantom is nested
ellipsoidal shells plus noise over the value type's range; lattice is
interpolated white noise over the value type's range.
"""
import ctypes as C

import numpy as np
import torch

from kvs_gb300 import _abi
from kvs_gb300 import synthetic as S
from kvs_gb300.default_colormap import BREWER_RDBU_256
from kvs_gb300.marching_cubes import MarchingCubes, PolygonObject, StructuredVolumeObject, default_context

DUP, SHARED, VERTEX = 0, 1, 2   # kvsmc_mode: duplicated, shared vertices, shared vertices with vertex normals
MODE_NAMES = {"dup": DUP, "shared": SHARED, "vertex": VERTEX}
BYTES = {"int8": 1, "uint8": 1, "int16": 2, "uint16": 2, "int32": 4, "float32": 4, "int64": 8, "float64": 8}


def listed():
    return [
        # one isosurface of a small scanned volume, as an interactive viewer asks for: latency
        {"name": "extract_u8_small", "kind": "extract", "dtype": "uint8", "nx": 64, "ny": 64, "nz": 64,
         "field": "phantom", "iso": 0.45, "mode": "dup"},
        # a simulation's double-precision field, one isosurface, odd sizes
        {"name": "extract_f64", "kind": "extract", "dtype": "float64", "nx": 201, "ny": 173, "nz": 187,
         "field": "fbm", "iso": 0.5, "mode": "dup"},
        # the drop-in mapper on a host array: the reference's own CPU-sized workload
        {"name": "mapper_f32", "kind": "mapper", "dtype": "float32", "nx": 128, "ny": 128, "nz": 128,
         "field": "blobs", "iso": 0.5, "mode": "dup"},
        # the same in the reference example's mode (vertex normals), 16-bit data, uneven sizes
        {"name": "mapper_u16_vertex", "kind": "mapper", "dtype": "uint16", "nx": 99, "ny": 130, "nz": 83,
         "field": "phantom", "iso": 0.45, "mode": "vertex"},
        # an isovalue sweep of a large float field in one batched call, the headline form
        {"name": "sweep_f32", "kind": "sweep", "dtype": "float32", "nx": 640, "ny": 704, "nz": 600,
         "field": "fbm", "lo": 0.2, "hi": 0.8, "niso": 16, "mode": "dup"},
        # the sweep in the reference example's mode: shared vertices with vertex normals
        {"name": "sweep_f32_vertex", "kind": "sweep", "dtype": "float32", "nx": 385, "ny": 320, "nz": 352,
         "field": "fbm", "lo": 0.35, "hi": 0.65, "niso": 8, "mode": "vertex"},
        # output-heavy 16-bit data, a few isovalues at its middle percentiles
        {"name": "sweep_u16_heavy", "kind": "sweep", "dtype": "uint16", "nx": 1024, "ny": 768, "nz": 640,
         "field": "lattice", "lo": 0.45, "hi": 0.6, "niso": 4, "mode": "dup"},
        # many volumes of uneven size and type, extracted again and again: a replayed plan
        {"name": "plan_uneven", "kind": "plan", "volumes": 48, "smallest": 32, "largest": 320},
        # in-situ: the field is on the device, new every frame, extracted once
        {"name": "frame_f32", "kind": "frame", "dtype": "float32", "nx": 301, "ny": 256, "nz": 270,
         "field": "fbm", "iso": 0.5, "mode": "dup"},
        # one oblique slice with colours through a large volume
        {"name": "slice_f32", "kind": "slice", "dtype": "float32", "nx": 512, "ny": 480, "nz": 500, "field": "fbm"},
        # a tetrahedral mesh, one isovalue
        {"name": "cells_tet_f32", "kind": "cells", "cell": "tetra", "dtype": "float32", "nx": 121, "ny": 110, "nz": 117,
         "niso": 1},
        # an extracted mesh on its way to a file
        {"name": "stl_dup", "kind": "stl", "triangles": 4000037, "mode": "dup"},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _dims(rng, lo, hi):
    """Three sizes around a common scale, uneven and mostly odd."""
    n = _log(rng, lo, hi)
    return {k: max(lo, min(hi, int(n * rng.uniform(0.75, 1.25)))) for k in ("nx", "ny", "nz")}


def draw(rng):
    kind = rng.choice(["extract", "extract", "mapper", "sweep", "sweep", "plan", "frame", "slice", "cells", "stl"])
    narrow = ["uint8", "int8", "uint16", "int16", "float32"]
    if kind == "extract":
        dt = rng.choice(narrow + ["int32", "float64"])
        return {"kind": kind, "dtype": dt, **_dims(rng, 24, 220 if dt in ("int32", "float64") else 400),
                "field": rng.choice(["phantom", "fbm"]), "iso": round(rng.uniform(0.3, 0.7), 3),
                "mode": rng.choice(["dup", "dup", "shared", "vertex"])}
    if kind == "mapper":
        return {"kind": kind, "dtype": rng.choice(narrow + ["int32", "float64"]), **_dims(rng, 20, 180),
                "field": rng.choice(["phantom", "blobs"]), "iso": round(rng.uniform(0.35, 0.6), 3),
                "mode": rng.choice(["dup", "shared", "vertex"])}
    if kind == "sweep":
        mode = rng.choice(["dup", "dup", "shared", "vertex"])
        dims = _dims(rng, 48, 600 if mode == "dup" else 320)
        smooth = min(dims.values()) >= 150   # the lattice's cells are 48 nodes wide
        return {"kind": kind, "dtype": rng.choice(["uint8", "uint16", "float32", "float32"]), **dims,
                "field": rng.choice(["fbm", "lattice"]) if smooth else "fbm",
                "lo": round(rng.uniform(0.2, 0.45), 3), "hi": round(rng.uniform(0.55, 0.8), 3),
                "niso": rng.randint(2, 16 if mode == "dup" else 8), "mode": mode}
    if kind == "plan":
        lo = _log(rng, 16, 64)
        return {"kind": kind, "volumes": rng.randint(4, 48), "smallest": lo, "largest": rng.randint(2 * lo, 300)}
    if kind == "frame":
        return {"kind": kind, "dtype": rng.choice(narrow), **_dims(rng, 32, 400), "field": rng.choice(["fbm", "phantom"]),
                "iso": round(rng.uniform(0.3, 0.7), 3), "mode": rng.choice(["dup", "dup", "vertex"])}
    if kind == "slice":
        return {"kind": kind, "dtype": rng.choice(narrow + ["float64"]), **_dims(rng, 32, 500), "field": "fbm"}
    if kind == "cells":
        return {"kind": kind, "cell": rng.choice(["tetra", "tetra", "hexa"]), "dtype": rng.choice(["float32", "float32", "float64"]),
                **_dims(rng, 12, 120), "niso": rng.choice([1, 1, 6])}
    return {"kind": "stl", "triangles": _log(rng, 500, 4000000), "mode": rng.choice(["dup", "shared", "vertex"])}


# ------------------------------------------------------------------ inputs


def _span(dtype):
    dt = np.dtype(dtype)
    return (0.0, 1.0) if dt.kind == "f" else (float(np.iinfo(dt).min), float(np.iinfo(dt).max))


def _pattern(case, device="cuda"):
    """The case's structure, the same for every seed: values on the device, shaped (nz, ny, nx)."""
    shape = (case["nz"], case["ny"], case["nx"])
    dtype, wide = np.dtype(case["dtype"]), case["dtype"] in ("int32", "int64", "float64")
    at = (case["nx"] * 31 + case["ny"] * 17 + case["nz"]) % 1000
    if case["field"] == "phantom" and not wide:
        return S.ellipsoid_phantom(shape, dtype, seed=at, device=device)
    if case["field"] == "lattice":
        return S.lattice_noise(shape, dtype, seed=at, device=device, spacing=48)
    if case["field"] == "blobs":
        # the reference workload's blobs (sigma 8 to 24 nodes of 128), scaled to the volume
        s = max(shape) / 128.0
        f = S.gaussian_blobs(shape, sigma=(8.0 * s, 24.0 * s), seed=at, device=device).clamp_(0.0, 1.0)
    elif case["field"] == "phantom":
        f = S.ellipsoid_phantom(shape, np.float32, seed=at, device=device)
    else:
        f = S.fbm(shape, seed=at, device=device)
    if case["dtype"] == "float32":
        return f
    if case["dtype"] == "float64":   # digits beyond float, as a double-precision solver leaves them
        return f.double() * (1.0 + 1e-12 * np.pi) + 1e-11
    lo, hi = (-2.0e9, 2.0e9) if case["dtype"] == "int32" else _span(dtype)
    return S._cast(f.double() * (hi - lo) + lo, dtype)


def _field(case, seed, levels, device="cuda"):
    """The case's volume for one seed: its pattern, with every value moved between the levels around it by an amount of
    the seed's own.  Which nodes lie above a level stays, so outputs of all seeds have one size; where the surface cuts
    each edge does not."""
    f = _pattern(case, device)
    amount = 0.75 * (2.0 * np.random.default_rng(seed).random() - 1.0)
    if abs(amount) < 0.05:
        amount = 0.05
    lo, hi = (-2.0e9, 2.0e9) if case["dtype"] == "int32" else _span(case["dtype"])
    cuts = torch.tensor([lo, *sorted(levels), hi], dtype=torch.float64, device=device)
    for part in f.split(64):
        v = part.double()
        k = torch.bucketize(v, cuts).clamp_(1, len(cuts) - 1)   # cuts[k - 1] < v <= cuts[k]
        a, w = cuts[k - 1], cuts[k] - cuts[k - 1]
        u = (v - a) / w
        new = a + w * (u + amount * u * (1.0 - u))
        new = (new if f.dtype.is_floating_point else new.round()).to(f.dtype)
        keep = torch.bucketize(new.double(), cuts).clamp_(1, len(cuts) - 1) != k
        part.copy_(torch.where(keep, v, new.double()).to(f.dtype))
    return f


def _place(seed):
    """The volume's place and node spacing in the user's coordinates: kvsmc_params' min_coord and scale."""
    rng = np.random.default_rng((seed, 1))
    return [float(np.float32(x)) for x in rng.uniform(-20.0, 20.0, 3)], [float(np.float32(x)) for x in rng.uniform(0.5, 2.0, 3)]


def _moved(points, place):
    """(p + min_coord) * scale of points (..., 3)."""
    lo, scale = (torch.tensor(x, dtype=torch.float64, device=points.device) for x in place)
    return (points + lo) * scale


def _level(case, fraction):
    lo, hi = (-2.0e9, 2.0e9) if case["dtype"] == "int32" else _span(case["dtype"])
    return lo + fraction * (hi - lo)


def _levels(case):
    return [_level(case, f) for f in np.linspace(case["lo"], case["hi"], case["niso"])]


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _requests(ctx, vols, params, in_one=False):
    """Requests with device outputs sized by a count, as a program allocates them.  in_one: every
    request's outputs in two shared arrays."""
    n = len(params)
    reqs = (_abi.Request * n)()
    for r, v, p in zip(reqs, vols, params):
        r.volume, r.params = v.handle, p
    ctx.check(ctx.lib.kvsmc_count_batch(ctx.handle, reqs, n), "kvsmc_count_batch")
    outs = []
    need = [(r.sizes.ncoords, r.sizes.nnormals, r.sizes.nconnections) for r in reqs]
    if in_one:
        at = np.cumsum([0] + [-(-a // 64) * 64 for a, _, _ in need]), np.cumsum([0] + [-(-b // 64) * 64 for _, b, _ in need])
        outs = [torch.zeros(max(1, int(a[-1])), device="cuda") for a in at]
        for i, r in enumerate(reqs):
            r.d_coords, r.coords_capacity = outs[0].data_ptr() + 4 * int(at[0][i]), need[i][0]
            r.d_normals, r.normals_capacity = outs[1].data_ptr() + 4 * int(at[1][i]), need[i][1]
        return reqs, outs
    for r, (a, b, k) in zip(reqs, need):
        c, m = torch.zeros(max(1, a), device="cuda"), torch.zeros(max(1, b), device="cuda")
        r.d_coords, r.coords_capacity, r.d_normals, r.normals_capacity = c.data_ptr(), a, m.data_ptr(), b
        out = [c[:a], m[:b]]
        if r.params.mode != DUP:
            conn = torch.zeros(max(1, k), dtype=torch.int32, device="cuda")
            r.d_connections, r.connections_capacity = conn.data_ptr(), k
            out.append(conn[:k])
        outs.append(out)
    return reqs, outs


def _uneven(case):
    """The plan's volumes: sizes, types, isovalues as fractions of the range; drawn from the case."""
    rng = np.random.default_rng(case["volumes"] * 1000 + case["largest"])
    for _ in range(case["volumes"]):
        d = rng.integers(case["smallest"], case["largest"] + 1, 3)
        yield {"nx": int(d[0]), "ny": int(d[1]), "nz": int(d[2]), "dtype": ("uint8", "uint16", "float32")[int(rng.integers(3))],
               "field": "phantom", "iso": float(rng.uniform(0.2, 0.8))}


def _plane(case):
    """An oblique plane through the middle of the volume; drawn from the case."""
    rng = np.random.default_rng(case["nx"] * 1000 + case["nz"])
    n = rng.uniform(0.3, 1.0, 3) * rng.choice([-1.0, 1.0], 3)
    mid = (np.array([case["nx"], case["ny"], case["nz"]]) - 1) * rng.uniform(0.45, 0.55, 3)
    return np.array([*n, -float(n @ mid)], np.float32)


_TETS = [0, 1, 2, 6, 0, 2, 3, 6, 0, 3, 7, 6, 0, 7, 4, 6, 0, 4, 5, 6, 0, 5, 1, 6]   # a hexahedron as six tetrahedra


def _mesh(case, seed):
    """A jittered grid split into cells: values, coords (N, 3), connections, isovalues."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    z, y, x = torch.meshgrid(*(torch.arange(n, device="cuda") for n in (nz, ny, nx)), indexing="ij")
    xyz = torch.stack([x, y, z], -1).reshape(-1, 3).float()
    xyz += (torch.rand(xyz.shape, generator=gen, device="cuda") - 0.5) * 0.4
    levels = [0.5] if case["niso"] == 1 else np.linspace(0.3, 0.7, case["niso"]).tolist()
    values = _field({**case, "field": "fbm"}, seed, levels).reshape(-1)
    node = torch.arange(nx * ny * nz, device="cuda").reshape(nz, ny, nx)[:-1, :-1, :-1].reshape(-1, 1)
    s = nx * ny
    hexa = node + torch.tensor([0, 1, 1 + nx, nx, s, s + 1, s + 1 + nx, s + nx], device="cuda")
    conn = hexa if case["cell"] == "hexa" else hexa[:, _TETS].reshape(-1, 4)
    return values, xyz.contiguous(), conn.to(torch.int32).contiguous(), levels


def _soup(case, seed):
    """A triangle mesh of the mode's layout: coords, normals, connections (None when duplicated)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    t = case["triangles"]
    if case["mode"] == "dup":
        return (torch.rand(9 * t, generator=gen, device="cuda") * 512, torch.rand(3 * t, generator=gen, device="cuda") - 0.5,
                None)
    v = t // 2 + 2   # a closed surface's vertices
    # each triangle's corners near its place along the surface, as an extraction numbers them
    base = (torch.arange(t, device="cuda") // 2)[:, None] + torch.randint(0, 64, (t, 3), generator=gen, device="cuda")
    conn = base.clamp_(max=v - 1).to(torch.int32).reshape(-1)
    normals = torch.rand(3 * (v if case["mode"] == "vertex" else t), generator=gen, device="cuda") - 0.5
    return torch.rand(3 * v, generator=gen, device="cuda") * 512, normals, conn


def prepare(case, seed):
    kind = case["kind"]
    ctx = default_context()
    st = {"kind": kind, "ctx": ctx}
    if kind == "mapper":
        iso = _level(case, case["iso"])
        st.update(values=S.to_numpy(_field(case, seed, [iso])), iso=iso, mode=case["mode"])
    elif kind in ("extract", "frame", "sweep"):
        isos = _levels(case) if kind == "sweep" else [_level(case, case["iso"])]
        f = _field(case, seed, isos)
        torch.cuda.synchronize()
        dt, shape = np.dtype(case["dtype"]), tuple(f.shape)
        vol = _abi.DeviceVolume.from_device(ctx, f.data_ptr(), dt, shape)
        ctx.synchronize()
        place = _place(seed)
        params = [_abi.make_params(i, MODE_NAMES[case["mode"]], None, *place) for i in isos]
        reqs, outs = _requests(ctx, [vol] * len(isos), params)
        st.update(reqs=reqs, outs=outs)
        if kind == "frame":
            vol.free()
            st.update(field=f, dtype=dt, shape=shape)
        else:
            st.update(vol=vol)
    elif kind == "plan":
        vols, params = [], []
        place = _place(seed)
        for i, c in enumerate(_uneven(case)):
            iso = _level(c, c["iso"])
            f = _field(c, (seed, i), [iso])
            torch.cuda.synchronize()
            vols.append(_abi.DeviceVolume.from_device(ctx, f.data_ptr(), np.dtype(c["dtype"]), tuple(f.shape)))
            ctx.synchronize()
            params.append(_abi.make_params(iso, DUP, None, *place))
        reqs, outs = _requests(ctx, vols, params, in_one=True)
        torch.cuda.synchronize()
        st.update(vols=vols, reqs=reqs, outs=outs, plan=_abi.Plan(ctx, reqs))
    elif kind == "slice":
        f = _field(case, seed, [_level(case, 0.5)])
        torch.cuda.synchronize()
        vol = _abi.DeviceVolume.from_device(ctx, f.data_ptr(), np.dtype(case["dtype"]), tuple(f.shape))
        ctx.synchronize()
        table = np.frombuffer(BREWER_RDBU_256, np.uint8).copy()
        p = _abi.SliceParams()
        p.coefficients[:] = [float(c) for c in _plane(case)]
        p.min_coord[:], p.scale[:] = _place(seed)
        lo, hi = _span(case["dtype"])
        p.tf_min, p.tf_max, p.tf_resolution, p.tf_table = lo, hi, 256, table.ctypes.data
        n = C.c_uint64()
        ctx.check(ctx.lib.kvsmc_slice_count(ctx.handle, vol.handle, C.byref(p), C.byref(n)), "kvsmc_slice_count")
        t = n.value
        st.update(vol=vol, table=table, params=p, t=t, coords=torch.zeros(9 * t, device="cuda"),
                  normals=torch.zeros(3 * t, device="cuda"), colors=torch.zeros(9 * t, dtype=torch.uint8, device="cuda"))
    elif kind == "cells":
        values, xyz, conn, levels = _mesh(case, seed)
        lo, hi = float(values.min()), float(values.max())
        st.update(values=values, xyz=xyz, conn=conn, levels=(C.c_double * len(levels))(*levels), lo=lo, hi=hi,
                  type={"tetra": 0, "hexa": 1}[case["cell"]], sizes=(_abi.Sizes * len(levels))())
        torch.cuda.synchronize()
        # sized by one empty-handed call, which reports what it needs
        n = len(levels)
        _cells(st, None, [0] * n, None, [0] * n)
        t = [s.ntriangles for s in st["sizes"]]
        coords = [torch.zeros(9 * k, device="cuda") for k in t]
        normals = [torch.zeros(3 * k, device="cuda") for k in t]
        st.update(coords=coords, normals=normals, pc=(C.c_void_p * n)(*[c.data_ptr() for c in coords]),
                  pn=(C.c_void_p * n)(*[c.data_ptr() for c in normals]), cc=[9 * k for k in t], cn=[3 * k for k in t])
    else:
        coords, normals, conn = _soup(case, seed)
        st.update(coords=coords, normals=normals, conn=conn, mode=MODE_NAMES[case["mode"]], t=case["triangles"],
                  records=torch.zeros(50 * case["triangles"], dtype=torch.uint8, device="cuda"))
    torch.cuda.synchronize()
    return st


def _cells(st, pc, cc, pn, cn):
    ctx, n = st["ctx"], len(st["levels"])
    nnodes, ncells = st["values"].numel(), st["conn"].shape[0]
    dt = 8 if st["values"].dtype == torch.float32 else 9
    if n == 1:
        return ctx.lib.kvsmc_marching_cells_device(
            ctx.handle, st["type"], _ptr(st["values"]), dt, nnodes, _ptr(st["xyz"]), _ptr(st["conn"]), ncells,
            st["levels"][0], 1, st["lo"], st["hi"], pc and pc[0], cc[0], pn and pn[0], cn[0], C.byref(st["sizes"][0]))
    return ctx.lib.kvsmc_marching_cells_sweep_device(
        ctx.handle, st["type"], _ptr(st["values"]), dt, nnodes, _ptr(st["xyz"]), _ptr(st["conn"]), ncells, st["levels"], n,
        1, st["lo"], st["hi"], pc, (C.c_uint64 * n)(*cc), pn, (C.c_uint64 * n)(*cn), st["sizes"])


# -------------------------------------------------------------------- runs


def run(st):
    kind, ctx = st["kind"], st["ctx"]
    lib = ctx.lib
    if kind == "mapper":
        ntype = PolygonObject.VertexNormal if st["mode"] == "vertex" else PolygonObject.PolygonNormal
        mc = MarchingCubes(StructuredVolumeObject(st["values"]), st["iso"], ntype, st["mode"] == "dup", context=ctx)
        out = [mc.coords(), mc.normals()]
        return out if st["mode"] == "dup" else out + [mc.connections().view(np.int32)]
    if kind == "frame":
        vol = _abi.DeviceVolume.from_device(ctx, st["field"].data_ptr(), st["dtype"], st["shape"])
        r = st["reqs"][0]
        ctx.check(lib.kvsmc_extract_device(ctx.handle, vol.handle, C.byref(r.params), r.d_coords, r.coords_capacity,
                                           r.d_normals, r.normals_capacity, r.d_connections, r.connections_capacity,
                                           C.byref(r.sizes)), "kvsmc_extract_device")
        vol.free()
        return st["outs"][0]
    if kind == "extract":
        r = st["reqs"][0]
        ctx.check(lib.kvsmc_extract_device(ctx.handle, r.volume, C.byref(r.params), r.d_coords, r.coords_capacity,
                                           r.d_normals, r.normals_capacity, r.d_connections, r.connections_capacity,
                                           C.byref(r.sizes)), "kvsmc_extract_device")
        return st["outs"][0]
    if kind == "sweep":
        ctx.check(lib.kvsmc_extract_batch(ctx.handle, st["reqs"], len(st["reqs"])), "kvsmc_extract_batch")
        return st["outs"]
    if kind == "plan":
        st["plan"].launch()
        st["plan"].wait()
        return st["outs"]
    if kind == "slice":
        n, t = C.c_uint64(), st["t"]
        ctx.check(lib.kvsmc_slice_extract_device(ctx.handle, st["vol"].handle, C.byref(st["params"]), _ptr(st["coords"]),
                                                 9 * t, _ptr(st["colors"]), 9 * t, _ptr(st["normals"]), 3 * t, C.byref(n)),
                  "kvsmc_slice_extract_device")
        return [st["coords"], st["normals"], st["colors"]]
    if kind == "cells":
        ctx.check(_cells(st, st["pc"], st["cc"], st["pn"], st["cn"]), "kvsmc_marching_cells")
        return [st["coords"], st["normals"]]
    conn = st["conn"]
    ctx.check(lib.kvsmc_stl_records(ctx.handle, st["mode"], _ptr(st["coords"]), _ptr(st["normals"]),
                                    _ptr(conn) if conn is not None else None, st["coords"].numel() // 3, st["t"],
                                    _ptr(st["records"])), "kvsmc_stl_records")
    return st["records"]


# -------------------------------------------------------------------- work

# triangles a cell and isovalue has on these fields, measured over their seeds and the isovalues used here (rounded)
DENSITY = {"fbm": 0.05, "blobs": 0.02, "phantom": 0.05, "lattice": 0.06}


def work(case):
    kind = case["kind"]
    if kind == "stl":
        t = case["triangles"]
        v = t // 2 + 2
        mesh = {"dup": 48 * t, "shared": 12 * v + 24 * t, "vertex": 24 * v + 12 * t}[case["mode"]]
        return {"bytes": mesh + 50 * t, "flops": 0 if case["mode"] != "vertex" else 9 * t}
    if kind == "plan":
        mean = (case["smallest"] + case["largest"]) / 2.0
        cells = case["volumes"] * mean ** 3
        return {"bytes": cells * (7 / 3 + 48 * DENSITY["phantom"]), "flops": cells * DENSITY["phantom"] * 100}
    cells = float(case["nx"]) * case["ny"] * case["nz"]
    if kind == "cells":
        per = 6 if case["cell"] == "tetra" else 1
        tri = cells * per * 0.06 * case["niso"]
        return {"bytes": cells * (per * 4 * (4 if per == 6 else 8) + BYTES[case["dtype"]] + 12) + 48 * tri, "flops": 150 * tri}
    if kind == "slice":
        # two triangles for each cut cell; the values are read at the cut edges' ends only
        tri = 2.5 * cells ** (2.0 / 3.0)
        return {"bytes": tri * (57 + 2 * BYTES[case["dtype"]]), "flops": 200 * tri}
    n = case.get("niso", 1)
    tri = cells * n * DENSITY[case["field"]]
    # duplicated: 48 bytes a triangle; shared: half as many vertices as triangles
    out = {"dup": 48, "shared": 6 + 24, "vertex": 12 + 12}[case["mode"]]
    return {"bytes": cells * BYTES[case["dtype"]] + out * tri, "flops": cells * n + 100 * tri}


# ------------------------------------------------------- the same in 64 bits

# case -> its triangles' edges, four bits each from the low end, three a triangle
# (the reference's TriangleID in the order its mappers emit the corners)
CUBE = """
    0 830 190 819831 2a1 2a1830 2902a9 98aa82832 b23 b08b20 3b2901 8b99b1b21 a3ba13 ba88a0a10 a9bb93903 8ba8a9 784
    347304 478190 317714194 4782a1 2a1043473 4780292a9 947732972a92 b23478 4224b47b 3b2478019 219b294b97b4 847ba3a13
    b470414b1ba1 3bba90b9784 ba9b947b4 549 830549 501540 153358548 5492a1 9542a1083 244252a5 483543253a52 3b2549
    9548b0b20 3b2150540 8548b2582152 54913a3ba ba8a18810954 3bba50b5405 8ba8a5485 795789 735539309 571170780 573531
    12a579789 73530550912a 52a578258028 573532a52 b23897957 7b2209729579 5717811803b2 15717b21b 3ba13a578589
    a0b0a1b07095705 70507850a03ba0b b57a5b 65a a65830 a65019 a65981831 612651 83261651 260069659 283265825985 65a3b2
    65a20b08b a653b2190 8b9b29921a65 1355363b6 b65510b508b0 590650360b63 98b9b6596 784a65 5a6734304 478a65901
    94773197165a 784516126 473043265251 260650059478 692965293947397 65a847b23 7b2204724a65 a653b2784190
    a65b474b9b29219 b65513b53478 4b0b470b1b651b5 47863b360650590 b977949b6596 4a649a 8309a4a64 40660a01a
    1a6648168318 642241491 642492291083 264240 264248328 23b64a49a a649a48b2820 1a6640160b23 b181b28141a6416
    63b139369649 41614961b108b18 640603b63 68b486 9a88a7a67 7a69a0a70730 801781a7167a 73171a67a 678891681261
    397930796912692 26067807 726327 67889a68a3b2 a797a69707b2072 3b27a6a71781801 71661a17b21b 36163b169678968 67b910
    60bb03067807 b67 6b7 76b083 76b190 76b318198 b7612a b760832a1 b76a92902 98a83aa32b76 276237 206607087 190372762
    768981861621 37117a76a 818717a176a a76a907a0370 a98a876a7 86b846 4600636b3 194686b8 36b319639469 a12b86846
    4606b00b32a1 a922906b4b84 63436b43932a93a 624428238 624420 384462342901 462421941 a16468618138 4606a10a
    93a390a36384634 a4694a 6b7954 76b954830 6b7405015 15354334876b 6b712a549 9548302a1b76 242a44a56b7
    76b52a253543483 495627237 876620860549 405501763623 581854182876286 37176116a549 5497080717616a1 7a3a763a0a540a4
    8a44a5a876a7 89bb96956 9505606306b3 6b51505b0b80 315356b36 56bb895b92a1 2a16959606b0b30 25052a05856b85b
    53aa32356b36 823625285895 620609569 286823685801581 162561 9686958636a1361 60550906a10a 6a5380 56a 5b75ab
    30875b5ab 901ab5b75 318819b7a75a 51771b12b 2b7751271830 b72029279759 8292839252b7527 7533525a2 25a758528208
    a23375a35019 52725a728219829 753351 751710870 375359039 975879 b8aa85845 30bab5b05045 45aab84a8190
    14341934b45ab4a 584b82852512 1b5b125b4b304b0 85b584b52590250 b32459 8434535235a2 204245a25 1905848535a3a23
    429921245a25 513538458 51450 350059538458 459 ab99b4b74 ab9b79974830 4b7401b41ab1 b4a4b7a41483143 1292b9b49b74
    830b121b9b79749 40242b74b 24334842b74b 4973727929a2 7270827a749a79 a4a014a7a237a3 748a21 137174914 718810174914
    437034 874 b8aa89 9ab9b3093 ab8a801a0 3ab1a3 b89b912b1 b922919b3093 b82b0 2b3 89a8a2382 920a29 a811808a2382 a21
    189381 910 380 0
""".split()
TETRA = "0 12 530 253312 134 34420 105541 254 452 145501 24430 431 213352 35 210 0".split()
CORNERS = [0, 1, 3, 2, 4, 5, 7, 6]   # case bit -> corner (dx + 2 dy + 4 dz)
CUBE_EDGES = [(0, 1), (1, 3), (3, 2), (2, 0), (4, 5), (5, 7), (7, 6), (6, 4), (0, 4), (1, 5), (3, 7), (2, 6)]   # corners
HEXA_EDGES = [(0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (4, 0), (5, 1), (6, 2), (7, 3)]   # local nodes
TETRA_EDGES = [(0, 1), (0, 2), (0, 3), (1, 2), (2, 3), (3, 1)]                                                 # local nodes


def _table(packed, longest, device):
    """(triangles per case, edges (case, triangle, corner))."""
    count = torch.zeros(len(packed), dtype=torch.int64)
    edges = torch.zeros((len(packed), longest, 3), dtype=torch.int64)
    for c, text in enumerate(packed):
        # edge 0 may be the highest digit, so a case's digits are padded to whole triangles
        digits = [int(ch, 16) for ch in reversed(text)] if text != "0" else []
        digits += [0] * (-len(digits) % 3)
        count[c] = len(digits) // 3
        for i, e in enumerate(digits):
            edges[c, i // 3, i % 3] = e
    return count.to(device), edges.to(device)


def _triangles(code, count, edges):
    """Per triangle of the cells, in cell and table order: its cell's place in `code` and its three edges."""
    n = count[code]
    cell = torch.repeat_interleave(torch.arange(code.numel(), device=code.device), n)
    first = torch.cumsum(n, 0) - n
    k = torch.arange(cell.numel(), device=code.device) - first[cell]
    return cell, edges[code[cell], k]


def _cube_cases(above):
    code = torch.zeros([n - 1 for n in above.shape], dtype=torch.uint8, device=above.device)
    for bit, c in enumerate(CORNERS):
        dx, dy, dz = c & 1, (c >> 1) & 1, c >> 2
        nz, ny, nx = above.shape
        code |= above[dz:nz - 1 + dz, dy:ny - 1 + dy, dx:nx - 1 + dx].to(torch.uint8) << bit
    return code


def _cross(p):
    """(b - a) x (c - a) of triangles (T, 3, 3)."""
    u, v = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    return torch.linalg.cross(u, v)


CHUNK = 1 << 21   # active cells at a time


def _dup64(f, level, place):
    """Duplicated triangles of one isovalue: coords, normals, 64 bits."""
    above = f.double() > level if f.dtype != torch.float32 or f.numel() < 1 << 27 else _above_by_slab(f, level)
    code = _cube_cases(above).reshape(-1)
    del above
    active = torch.nonzero((code != 0) & (code != 255)).reshape(-1)
    count, edges = _table(CUBE, 5, f.device)
    ends = torch.tensor(CUBE_EDGES, device=f.device)
    nz, ny, nx = f.shape
    flat = f.reshape(-1)
    coords, normals = [], []
    for a in active.split(CHUNK):
        cell, e = _triangles(code[a].long(), count, edges)
        lin = a[cell]
        xyz = torch.stack([lin % (nx - 1), lin // (nx - 1) % (ny - 1), lin // ((nx - 1) * (ny - 1))], -1)
        c = ends[e]                                                       # (T, 3, 2): corners
        at = xyz[:, None, None, :] + torch.stack([c & 1, (c >> 1) & 1, c >> 2], -1)   # (T, 3, 2, 3): nodes
        p = _moved(_between(flat, (at[..., 2] * ny + at[..., 1]) * nx + at[..., 0], at.double(), level), place)
        coords.append(p.reshape(-1))
        normals.append(_cross(p).reshape(-1))
    if not coords:
        return [torch.zeros(0, dtype=torch.float64, device=f.device)] * 2
    return [torch.cat(coords), torch.cat(normals)]


def _above_by_slab(f, level):
    return torch.cat([s.double() > level for s in f.split(32)])


def _between(flat, node, at, level):
    """The point where the value crosses the level, between an edge's two ends (..., 2)."""
    v = flat[node].double()
    r = ((level - v[..., 0]) / (v[..., 1] - v[..., 0])).abs().unsqueeze(-1)
    return (1 - r) * at[..., 0, :] + r * at[..., 1, :]


def _shared64(f, level, place, mode):
    """Shared vertices of one isovalue: coords, normals in 64 bits; no value for the connections."""
    above = f.double() > level
    nz, ny, nx = f.shape
    cut = torch.zeros((nz, ny, nx, 3), dtype=torch.bool, device=f.device)
    cut[:, :, :-1, 0] = above[:, :, 1:] != above[:, :, :-1]
    cut[:, :-1, :, 1] = above[:, 1:] != above[:, :-1]
    cut[:-1, :, :, 2] = above[1:] != above[:-1]
    at = torch.nonzero(cut.reshape(-1)).reshape(-1)
    node, axis = at // 3, at % 3
    step = torch.tensor([1, nx, nx * ny], device=f.device)[axis]
    lo = torch.stack([node % nx, node // nx % ny, node // (nx * ny)], -1).double()
    hi = lo + torch.nn.functional.one_hot(axis, 3).double()
    coords = _between(f.reshape(-1), torch.stack([node, node + step], -1), torch.stack([lo, hi], -2), level)
    coords = _moved(coords, place)
    ids = torch.cumsum(cut.reshape(-1).int(), 0, dtype=torch.int32) - 1
    code = _cube_cases(above).reshape(-1)
    active = torch.nonzero((code != 0) & (code != 255)).reshape(-1)
    count, edges = _table(CUBE, 5, f.device)
    ends = torch.tensor(CUBE_EDGES, device=f.device)
    normals = torch.zeros((coords.shape[0], 3), dtype=torch.float64, device=f.device)
    faces = []
    for a in active.split(CHUNK):
        cell, e = _triangles(code[a].long(), count, edges)
        lin = a[cell]
        base = (lin // ((nx - 1) * (ny - 1)) * ny + lin // (nx - 1) % (ny - 1)) * nx + lin % (nx - 1)
        c = ends[e]
        low, d = c.amin(-1), (c[..., 0] ^ c[..., 1])
        n = base[:, None] + (low & 1) + ((low >> 1) & 1) * nx + (low >> 2) * (nx * ny)
        v = ids[n * 3 + torch.where(d == 4, 2, torch.where(d == 2, 1, 0))].long()
        face = _cross(coords[v])
        if mode == "vertex":
            for k in range(3):
                normals.index_add_(0, v[:, k], face)
        else:
            faces.append(face)
    if mode != "vertex":
        normals = torch.cat(faces) if faces else normals[:0]
    return [coords.reshape(-1), normals.reshape(-1), None]


def _slice64(case, seed):
    """The slice's triangles in 64 bits; which cells the plane cuts is decided in float, as the mapper's definition has it."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    co = [float(c) for c in _plane(case)]
    x, y, z = (torch.arange(n, device="cuda", dtype=torch.float32) for n in (nx, ny, nz))
    plane = ((co[0] * x)[None, None, :] + (co[1] * y)[None, :, None]) + (co[2] * z)[:, None, None] + co[3]
    code = _cube_cases(plane > 0).reshape(-1)
    active = torch.nonzero((code != 0) & (code != 255)).reshape(-1)
    count, edges = _table(CUBE, 5, "cuda")
    ends = torch.tensor(CUBE_EDGES, device="cuda")
    cell, e = _triangles(code[active].long(), count, edges)
    lin = active[cell]
    xyz = torch.stack([lin % (nx - 1), lin // (nx - 1) % (ny - 1), lin // ((nx - 1) * (ny - 1))], -1)
    c = ends[e]
    at = (xyz[:, None, None, :] + torch.stack([c & 1, (c >> 1) & 1, c >> 2], -1)).double()
    p = at @ torch.tensor(co[:3], dtype=torch.float64, device="cuda") + co[3]
    r = (p[..., 0] / (p[..., 1] - p[..., 0])).abs().unsqueeze(-1)
    q = _moved((1 - r) * at[..., 0, :] + r * at[..., 1, :], _place(seed))
    return [q.reshape(-1), _cross(q).reshape(-1), None]   # -((c - a) x (b - a)); the colours are bytes


def _cells64(case, seed):
    values, xyz, conn, levels = _mesh(case, seed)
    tetra = case["cell"] == "tetra"
    count, edges = _table(TETRA if tetra else CUBE, 2 if tetra else 5, "cuda")
    ends = torch.tensor(TETRA_EDGES if tetra else HEXA_EDGES, device="cuda")
    local = conn.long() if tetra else conn.long()[:, [4, 5, 6, 7, 0, 1, 2, 3]]
    coords, normals = [], []
    for level in levels:
        above = (values.double() > level)[local].long()
        code = (above << torch.arange(above.shape[1], device="cuda")).sum(1)
        cell, e = _triangles(code, count, edges)
        node = local[cell[:, None, None], ends[e]]
        p = _between(values, node, xyz.double()[node], level)
        coords.append(p.reshape(-1))
        normals.append(_cross(p).reshape(-1))
    return [coords, normals]


def exact(case, seed):
    kind = case["kind"]
    if kind == "stl":
        return None   # bytes
    if kind == "cells":
        return _cells64(case, seed)
    if kind == "plan":
        coords, normals = [], []
        for i, c in enumerate(_uneven(case)):
            iso = _level(c, c["iso"])
            f = _field(c, (seed, i), [iso])
            a, b = _dup64(f.int() if f.dtype == torch.uint16 else f, iso, _place(seed))
            for to, part in ((coords, a), (normals, b)):
                to.append(torch.nn.functional.pad(part, (0, -part.numel() % 64)))
        return [torch.cat(coords), torch.cat(normals)]
    if kind == "slice":
        return _slice64(case, seed)
    levels = _levels(case) if kind == "sweep" else [_level(case, case["iso"])]
    f = _field(case, seed, levels)
    f = f.int() if f.dtype == torch.uint16 else f   # torch indexes no 16-bit unsigned tensors
    place = ([0.0] * 3, [1.0] * 3) if kind == "mapper" else _place(seed)
    out = [_dup64(f, i, place) if case["mode"] == "dup" else _shared64(f, i, place, case["mode"]) for i in levels]
    return out if kind == "sweep" else out[0]
