"""The emit over listed cells and the one-isolevel count (duplicated mode):
edges of the segments, of the blocks of units and of the list, against the
oracle; a list that overflows, against the requests run alone.
"""
import numpy as np
import pytest

from kvs_gb300 import _abi
from kvs_gb300 import synthetic as S

from .helpers import first_diff, same_bits
from .test_stream_gpu import extract_batch

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [np.int8, np.uint8, np.int16, np.uint16, np.float32])
@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 34, 9), (9, 3, 129), (5, 6, 130), (4, 70, 257), (6, 5, 258), (3, 4, 700)])
def test_sizes_and_isolevel_counts(kvsmc_ctx, oracle_lib, dtype, shape):
    """One, two and sixteen isolevels; smooth and noisy values (every cell
    crossed: more pairs a step than the count's and the emit's buffers)."""
    rng = np.random.default_rng(sum(shape))
    lo_t, hi_t = (0.0, 1.0) if dtype == np.float32 else (np.iinfo(dtype).min, np.iinfo(dtype).max)
    f = S.to_numpy(S.fbm(shape, base_freq=1.0 / 8.0, seed=shape[2], device="cuda")).astype(np.float64)
    for field in (f, rng.random(shape)):
        v = (lo_t + field * (hi_t - lo_t)).astype(dtype)
        lo, hi = float(v.min()), float(v.max())
        if lo == hi:
            continue
        vol = _abi.DeviceVolume.upload(kvsmc_ctx, v)
        for n in (1, 2, 16):
            isos = [lo + (hi - lo) * (k + 0.5) / n for k in range(n)]
            out = extract_batch(kvsmc_ctx, [vol] * n, [_abi.make_params(x, 0) for x in isos], _abi.PATH_AUTO)
            for x, o in zip(isos, out):
                ref = oracle_lib.extract(v, x, 0, lo, hi)
                assert o["ntri"] == ref["coords"].size // 9, (shape, n, x)
                assert same_bits(o["coords"], ref["coords"]), (shape, n, x, first_diff(o["coords"], ref["coords"]))
                assert same_bits(o["normals"], ref["normals"]), (shape, n, x)
        vol.free()


def test_single_isolevel_on_and_between_integer_values(kvsmc_ctx, oracle_lib):
    rng = np.random.default_rng(4)
    for dtype in (np.int8, np.uint16):
        v = rng.integers(0, 4, (6, 7, 140)).astype(dtype)
        vol = _abi.DeviceVolume.upload(kvsmc_ctx, v)
        for iso in (-1.0, 0.0, 0.5, 1.0, 2.999999, 3.0, 1e30):
            o = extract_batch(kvsmc_ctx, [vol], [_abi.make_params(iso, 0)], _abi.PATH_AUTO)[0]
            ref = oracle_lib.extract(v, iso, 0, 0.0, 3.0)
            assert same_bits(o["coords"], ref["coords"]) and same_bits(o["normals"], ref["normals"]), (dtype, iso)
        vol.free()


def test_several_isolevels_on_and_past_integer_values(kvsmc_ctx, oracle_lib):
    rng = np.random.default_rng(9)
    for dtype in (np.int8, np.uint8, np.int16, np.uint16):
        i = np.iinfo(dtype)
        v = rng.integers(i.min, i.max, (5, 6, 140), endpoint=True).astype(dtype)
        v[0, 0, :4] = (i.min, i.max, 0, 1)
        vol = _abi.DeviceVolume.upload(kvsmc_ctx, v)
        isos = [-1e30, i.min - 1.0, i.min, i.min + 0.5, -1.0, -0.0, 0.5, 1.0, 2.999999, 3.0, i.max - 0.5, float(i.max),
                i.max + 1.0, 1e30]
        out = extract_batch(kvsmc_ctx, [vol] * len(isos), [_abi.make_params(x, 0) for x in isos], _abi.PATH_AUTO)
        for x, o in zip(isos, out):
            ref = oracle_lib.extract(v, x, 0, float(i.min), float(i.max))
            assert same_bits(o["coords"], ref["coords"]) and same_bits(o["normals"], ref["normals"]), (dtype, x)
        vol.free()


@pytest.mark.parametrize("mode", [0, 2])
def test_crowded_isolevels_and_extreme_values(kvsmc_ctx, mode):
    """Equal isolevels and several in one bucket of the threshold table beside
    far ones, values at both ends of the float range, infinities and NaN:
    together and alone (one isolevel's plain compares)."""
    rng = np.random.default_rng(7 + mode)
    v = rng.random((7, 9, 300)).astype(np.float32)
    flat = v.reshape(-1)
    for i, x in enumerate((3.4e38, -3.4e38, np.inf, -np.inf, np.nan, -0.0, 1e-45)):
        flat[rng.integers(0, flat.size, 40)] = np.float32(x)
    vol = _abi.DeviceVolume.upload(kvsmc_ctx, v)
    for isos in ([0.5] * 9 + [0.5 + 1e-9, 0.5 + 6e-8, 0.50001, 0.7, 0.7, -1e30, 1e30],
                 [np.nextafter(np.float32(0.25), np.float32(1)), 0.25, 0.25, 1.0]):
        params = [_abi.make_params(float(x), mode) for x in isos]
        together = extract_batch(kvsmc_ctx, [vol] * len(isos), params, _abi.PATH_AUTO)
        for x, p, o in zip(isos, params, together):
            alone = extract_batch(kvsmc_ctx, [vol], [p], _abi.PATH_AUTO)[0]
            assert o["status"] == alone["status"] == _abi.OK
            assert all(same_bits(o[k], alone[k]) for k in ("coords", "normals")), (mode, x)
            assert np.array_equal(o["connections"], alone["connections"]), (mode, x)
    vol.free()


def test_a_list_that_overflows(kvsmc_ctx):
    """16 isolevels of noise cross nearly every cell: 6e8 pairs, more than the
    list holds, so the triangles come from the classifying emit, in a batch and
    in a replayed plan.  Only two requests have outputs."""
    n = 341
    gen = torch.Generator(device="cuda").manual_seed(3)
    v = torch.randint(0, 256, (n, n, n), generator=gen, device="cuda", dtype=torch.uint8)
    torch.cuda.synchronize()
    vol = _abi.DeviceVolume.from_device(kvsmc_ctx, v.data_ptr(), np.uint8, (n, n, n))
    isos = [110.5 + 2.0 * k for k in range(16)]
    params = [_abi.make_params(x, 0) for x in isos]
    want = {}
    for i in (3, 12):
        o = _abi.Sizes()
        kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_count(kvsmc_ctx.handle, vol.handle, params[i], o), "count")
        c, m = torch.zeros(o.ncoords, device="cuda"), torch.zeros(o.nnormals, device="cuda")
        torch.cuda.synchronize()
        kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_extract_device(kvsmc_ctx.handle, vol.handle, params[i], c.data_ptr(), o.ncoords,
                                                           m.data_ptr(), o.nnormals, None, 0, o), "extract")
        want[i] = (c, m)
    reqs = (_abi.Request * 16)()
    got = {i: tuple(torch.zeros_like(t) for t in want[i]) for i in want}
    torch.cuda.synchronize()
    for i in range(16):
        reqs[i].volume, reqs[i].params = vol.handle, params[i]
        if i in got:
            c, m = got[i]
            reqs[i].d_coords, reqs[i].coords_capacity = c.data_ptr(), c.numel()
            reqs[i].d_normals, reqs[i].normals_capacity = m.data_ptr(), m.numel()
    st = kvsmc_ctx.lib.kvsmc_extract_batch(kvsmc_ctx.handle, reqs, 16)
    assert st == _abi.ERR_CAPACITY
    for i in want:
        assert reqs[i].status == _abi.OK
        assert all(torch.equal(a, b) for a, b in zip(got[i], want[i])), i
        for t in got[i]:
            t.zero_()
    torch.cuda.synchronize()
    plan = _abi.Plan(kvsmc_ctx, reqs)
    plan.launch()
    plan.wait(check=False)
    for i in want:
        assert reqs[i].status == _abi.OK
        assert all(torch.equal(a, b) for a, b in zip(got[i], want[i])), i
    plan.close()
    vol.free()


def test_a_list_that_overflows_in_the_shared_modes(kvsmc_ctx):
    """The same noise with shared vertices: together the pairs overflow their
    list (the connections classify again, the vertex normals sort), alone they
    do not (connections over pairs, normals by cell).  Only two requests have
    outputs."""
    n = 341
    gen = torch.Generator(device="cuda").manual_seed(3)
    v = torch.randint(0, 256, (n, n, n), generator=gen, device="cuda", dtype=torch.uint8)
    torch.cuda.synchronize()
    vol = _abi.DeviceVolume.from_device(kvsmc_ctx, v.data_ptr(), np.uint8, (n, n, n))
    params = [_abi.make_params(110.5 + 2.0 * k, 1 if k == 3 else 2) for k in range(16)]

    def outputs(s):
        t = (torch.zeros(s.ncoords, device="cuda"), torch.zeros(s.nnormals, device="cuda"),
             torch.zeros(s.nconnections, dtype=torch.int32, device="cuda"))
        torch.cuda.synchronize()
        return t

    want = {}
    for i in (3, 12):
        o = _abi.Sizes()
        kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_count(kvsmc_ctx.handle, vol.handle, params[i], o), "count")
        c, m, k = outputs(o)
        kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_extract_device(kvsmc_ctx.handle, vol.handle, params[i], c.data_ptr(), o.ncoords,
                                                           m.data_ptr(), o.nnormals, k.data_ptr(), o.nconnections, o),
                        "extract")
        want[i] = (c, m, k, o)
    reqs = (_abi.Request * 16)()
    got = {i: outputs(want[i][3]) for i in want}
    for i in range(16):
        reqs[i].volume, reqs[i].params = vol.handle, params[i]
        if i in got:
            c, m, k = got[i]
            reqs[i].d_coords, reqs[i].coords_capacity = c.data_ptr(), c.numel()
            reqs[i].d_normals, reqs[i].normals_capacity = m.data_ptr(), m.numel()
            reqs[i].d_connections, reqs[i].connections_capacity = k.data_ptr(), k.numel()
    assert kvsmc_ctx.lib.kvsmc_extract_batch(kvsmc_ctx.handle, reqs, 16) == _abi.ERR_CAPACITY
    for i in want:
        assert reqs[i].status == _abi.OK
        assert all(torch.equal(a, b) for a, b in zip(got[i], want[i])), i
    vol.free()


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.float32, np.float64])
@pytest.mark.parametrize("shape", [(2, 2, 2), (2, 3, 33), (3, 2, 257), (5, 4, 256), (4, 34, 70), (40, 3, 9)])
def test_shared_modes_over_listed_pairs(kvsmc_ctx, oracle_lib, dtype, shape):
    """Volumes that are mostly faces (vertices that lack cells around their
    edge, node rows and planes past the last cells), every cell crossed: one
    request, three and sixteen in a batch."""
    rng = np.random.default_rng(sum(shape))
    v = rng.random(shape).astype(dtype) if np.dtype(dtype).kind == "f" else rng.integers(0, 100, shape).astype(dtype)
    lo, hi = float(v.min()), float(v.max())
    vol = _abi.DeviceVolume.upload(kvsmc_ctx, v)
    for n in (1, 3, 16):
        isos = [lo + (hi - lo) * (k + 0.37) / n for k in range(n)]
        modes = [1 + (k & 1) if n > 1 else 2 for k in range(n)]
        out = extract_batch(kvsmc_ctx, [vol] * n, [_abi.make_params(x, m) for x, m in zip(isos, modes)], _abi.PATH_AUTO)
        for x, m, o in zip(isos, modes, out):
            ref = oracle_lib.extract(v, x, m, lo, hi)
            assert same_bits(o["coords"], ref["coords"]), (shape, n, x, first_diff(o["coords"], ref["coords"]))
            assert same_bits(o["normals"], ref["normals"]), (shape, n, x, m)
            assert np.array_equal(o["connections"], ref["connections"].view(np.uint32)), (shape, n, x)
    vol.free()
