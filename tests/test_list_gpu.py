"""The list of crossed cells: its room, and what runs when it has none."""
import numpy as np
import pytest

from kvs_gb300 import _abi

from .helpers import same_bits
from .test_stream_gpu import extract_batch

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("shape", [(600, 600, 2), (340, 900, 3), (90, 2100, 2), (2, 2, 2)])
@pytest.mark.parametrize("dtype", [np.uint8, np.float32])
def test_narrow_volumes_in_a_plan(kvsmc_ctx, dtype, shape):
    """Few cells a task and many tasks: every counting warp holds a run of list
    entries that it leaves nearly unused, beyond the cells there are.  A plan
    whose list has room for all of them records no other emit."""
    rng = np.random.default_rng(5)
    v = (rng.random(shape) * 200).astype(dtype)
    vol = _abi.DeviceVolume.upload(kvsmc_ctx, v)
    params = [_abi.make_params(x, 0) for x in (60.5, 100.5, 140.5)]
    want = extract_batch(kvsmc_ctx, [vol] * 3, params, _abi.PATH_GATHER)
    for group in ([0], [1], [0, 1, 2]):
        reqs = (_abi.Request * len(group))()
        outs = []
        for r, i in zip(reqs, group):
            c, n = torch.zeros(want[i]["coords"].size + 1, device="cuda"), torch.zeros(want[i]["normals"].size + 1, device="cuda")
            outs.append((c, n))
            r.volume, r.params = vol.handle, params[i]
            r.d_coords, r.coords_capacity, r.d_normals, r.normals_capacity = c.data_ptr(), c.numel(), n.data_ptr(), n.numel()
        torch.cuda.synchronize()
        plan = _abi.Plan(kvsmc_ctx, reqs)
        for _ in range(2):
            plan.launch()
            plan.wait()
        for (c, n), i in zip(outs, group):
            assert same_bits(c[:-1].cpu().numpy(), want[i]["coords"]) and same_bits(n[:-1].cpu().numpy(), want[i]["normals"])
        plan.close()
    vol.free()


@pytest.mark.parametrize("dtype", [np.uint16, np.float32])
@pytest.mark.parametrize("noisy", [9, 70, 130, 257, 600])
def test_crowded_steps(kvsmc_ctx, dtype, noisy):
    """16 isolevels, noise in the first columns of rows that are smooth behind
    them: steps whose pairs are few, many in a few lanes, and many in all (more
    than the count's buffer holds); triangles and shared vertices."""
    rng = np.random.default_rng(noisy)
    v = np.broadcast_to(np.linspace(0.1, 0.9, 600), (5, 6, 600)).copy()
    v[:, :, :noisy] = rng.random((5, 6, noisy))
    v = (v * 60000).astype(dtype)
    vol = _abi.DeviceVolume.upload(kvsmc_ctx, v)
    isos = [20000.5 + 1300 * k for k in range(16)]
    for mode in (0, 2):
        params = [_abi.make_params(x, mode) for x in isos]
        want = extract_batch(kvsmc_ctx, [vol] * 16, params, _abi.PATH_GATHER)
        got = extract_batch(kvsmc_ctx, [vol] * 16, params, _abi.PATH_AUTO)
        for w, g in zip(want, got):
            assert g["status"] == _abi.OK and g["ntri"] == w["ntri"]
            assert same_bits(g["coords"], w["coords"]) and same_bits(g["normals"], w["normals"])
            assert np.array_equal(g["connections"], w["connections"])
    vol.free()


@pytest.mark.parametrize("entries", [0, 40])
@pytest.mark.parametrize("dtype", _abi.DTYPES)
def test_no_room_for_the_list(kvsmc_ctx, dtype, entries):
    """Without a list, or with one that overflows, the emit classifies the volume
    again: every mode, one request and several, device and host calls, a plan."""
    rng = np.random.default_rng(3)
    v = (rng.random((7, 20, 270)) * 100).astype(dtype)
    vol = _abi.DeviceVolume.upload(kvsmc_ctx, v)
    isos = (30.5, 50.25, 70.75)

    def calls():
        out = []
        for n in (1, 3):
            for mode in (0, 1, 2):
                res = extract_batch(kvsmc_ctx, [vol] * n, [_abi.make_params(x, mode) for x in isos[:n]], _abi.PATH_AUTO)
                assert all(r["status"] == _abi.OK and r["ntri"] > 0 for r in res)
                out += [a for r in res for a in (r["coords"], r["normals"], r["connections"])]
        for mode in (0, 1, 2):
            out += list(_abi.marching_cubes_host(kvsmc_ctx, v, _abi.make_params(isos[0], mode))[:3])
        for n in (1, 3):
            res = _abi.extract_batch_host(kvsmc_ctx, v, [_abi.make_params(x, k % 3) for k, x in enumerate(isos[:n])])
            out += [r[a] for r in res for a in ("coords", "normals", "connections")]
        if v.itemsize <= 2 or dtype == np.float32:
            reqs, outs = (_abi.Request * 3)(), []
            for r, x in zip(reqs, isos):
                c, m = torch.zeros(v.size * 45, device="cuda"), torch.zeros(v.size * 15, device="cuda")
                outs += [c, m]
                r.volume, r.params = vol.handle, _abi.make_params(x, 0)
                r.d_coords, r.coords_capacity, r.d_normals, r.normals_capacity = c.data_ptr(), c.numel(), m.data_ptr(), m.numel()
            torch.cuda.synchronize()
            plan = _abi.Plan(kvsmc_ctx, reqs)
            for _ in range(2):
                plan.launch()
                plan.wait()
            out += [t.cpu().numpy() for t in outs]
            plan.close()
        return out

    want = calls()
    kvsmc_ctx.set_list_limit(entries)
    try:
        got = calls()
    finally:
        kvsmc_ctx.set_list_limit()
    assert len(want) == len(got)
    for a, b in zip(want, got):
        assert np.array_equal(np.asarray(a).view(np.uint8), np.asarray(b).view(np.uint8))
    vol.free()
