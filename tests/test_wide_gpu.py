"""32/64-bit integer and double volumes on the streaming layout, against the
oracle: edges of the 256-cell segments and of the plane chunks, values that
only an exact compare tells apart, special doubles, clamp ranges that push
the ratio out of [0, 1].
"""
import numpy as np
import pytest

from kvs_gb300 import _abi

from .helpers import first_diff, same_bits
from .test_stream_gpu import extract_batch

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

WIDE = [np.int32, np.int64, np.uint32, np.uint64, np.float64]


def _check(ctx, oracle_lib, v, isos, minmax=None):
    lo, hi = minmax if minmax else (float(np.nanmin(v)), float(np.nanmax(v)))
    vol = _abi.DeviceVolume.upload(ctx, v)
    reqs = [(x, m) for x in isos for m in (0, 1, 2)]
    params = [_abi.make_params(x, m, (lo, hi)) for x, m in reqs]
    out = extract_batch(ctx, [vol] * len(reqs), params, _abi.PATH_AUTO)
    n = 0
    for (x, m), o in zip(reqs, out):
        ref = oracle_lib.extract(v, x, m, lo, hi)
        tag = (v.dtype, v.shape, x, m)
        assert o["status"] == _abi.OK, tag
        assert same_bits(o["coords"], ref["coords"]), (tag, first_diff(o["coords"], ref["coords"]))
        assert same_bits(o["normals"], ref["normals"]), (tag, first_diff(o["normals"], ref["normals"]))
        if m:
            assert np.array_equal(o["connections"], ref["connections"].view(np.uint32)), tag
        n += o["ntri"]
    vol.free()
    return n


@pytest.mark.parametrize("dtype", WIDE)
@pytest.mark.parametrize("shape", [(2, 2, 2), (70, 3, 33), (5, 7, 255), (4, 3, 256), (9, 4, 257), (3, 5, 258), (6, 9, 513)])
def test_sizes(kvsmc_ctx, oracle_lib, dtype, shape):
    rng = np.random.default_rng(sum(shape))
    x = np.linspace(0.0, 7.0, shape[2])[None, None, :] + np.linspace(0.0, 2.0, shape[0])[:, None, None]
    f = np.sin(x) + 0.3 * rng.random(shape)
    if dtype == np.float64:
        v, isos = f, [0.5, 0.1234567890123]
    else:
        base = 0 if np.dtype(dtype).kind == "i" else 2_000_000_000
        v, isos = (base + f * 9.0e8).astype(dtype), [base + 1.0e8, base + 3.5]
    assert _check(kvsmc_ctx, oracle_lib, v, isos) > 0


@pytest.mark.parametrize("dtype,around", [(np.int64, 2 ** 53), (np.int64, -(2 ** 62)), (np.uint64, 2 ** 63), (np.uint64, 5),
                                          (np.int64, 2 ** 63 - 64), (np.int64, -(2 ** 63) + 32), (np.uint64, 2 ** 64 - 64)])
def test_neighbouring_64_bit_integers(kvsmc_ctx, oracle_lib, dtype, around):
    """Values that round to the same double, isolevels on and beside them."""
    rng = np.random.default_rng(7)
    info = np.iinfo(dtype)
    lo, hi = max(info.min, around - 2048), min(info.max, around + 2048)
    v = rng.integers(lo, hi, (6, 5, 70), dtype=dtype, endpoint=True)
    at = float(v.reshape(-1)[3])
    _check(kvsmc_ctx, oracle_lib, v, [at, np.nextafter(at, -np.inf), np.nextafter(at, np.inf), float(info.min) * 1.5 - 1, 1e300])


def test_special_doubles(kvsmc_ctx, oracle_lib):
    rng = np.random.default_rng(9)
    v = rng.normal(size=(7, 6, 60))
    flat = v.reshape(-1)
    flat[rng.integers(0, flat.size, 60)] = 0.0
    flat[rng.integers(0, flat.size, 60)] = -0.0
    flat[rng.integers(0, flat.size, 40)] = 5e-324
    flat[rng.integers(0, flat.size, 40)] = -5e-324
    _check(kvsmc_ctx, oracle_lib, v, [0.0, -0.0, 5e-324, -5e-324])
    flat[rng.integers(0, flat.size, 20)] = np.nan
    flat[rng.integers(0, flat.size, 10)] = np.inf
    flat[rng.integers(0, flat.size, 10)] = -np.inf
    flat[rng.integers(0, flat.size, 10)] = 1.7e308
    flat[rng.integers(0, flat.size, 10)] = -1.7e308
    _check(kvsmc_ctx, oracle_lib, v, [0.25, 0.0, 1e308], (-1.7e308, 1.7e308))
    _check(kvsmc_ctx, oracle_lib, v, [0.25], (-np.inf, np.inf))
    # a preset range that leaves the isolevel outside
    _check(kvsmc_ctx, oracle_lib, v, [0.25], (0.3, 0.9))


def test_timeout_leaves_nothing_behind(kvsmc_ctx):
    """The bounded waits give up in the count, then in the emit; the next call is exact."""
    rng = np.random.default_rng(2)
    v = rng.random((12, 9, 300))
    vol = _abi.DeviceVolume.upload(kvsmc_ctx, v)
    p = [_abi.make_params(0.5, 0), _abi.make_params(0.4, 2)]
    good = extract_batch(kvsmc_ctx, [vol] * 2, p, _abi.PATH_AUTO)
    for limits in ((0, -1), (-1, 0)):
        reqs = (_abi.Request * 2)()
        bufs = []
        for i in range(2):
            c = torch.zeros(good[i]["coords"].size, device="cuda")
            n = torch.zeros(good[i]["normals"].size, device="cuda")
            k = torch.zeros(max(1, good[i]["connections"].size), dtype=torch.int32, device="cuda")
            bufs.append((c, n, k))
            reqs[i].volume, reqs[i].params = vol.handle, p[i]
            reqs[i].d_coords, reqs[i].coords_capacity = c.data_ptr(), c.numel()
            reqs[i].d_normals, reqs[i].normals_capacity = n.data_ptr(), n.numel()
            reqs[i].d_connections, reqs[i].connections_capacity = k.data_ptr(), k.numel()
        torch.cuda.synchronize()
        kvsmc_ctx.set_wait_limit(*limits)
        try:
            st = kvsmc_ctx.lib.kvsmc_extract_batch(kvsmc_ctx.handle, reqs, 2)
        finally:
            kvsmc_ctx.set_wait_limit()
        assert st == _abi.ERR_TIMEOUT
    again = extract_batch(kvsmc_ctx, [vol] * 2, p, _abi.PATH_AUTO)
    for a, b in zip(good, again):
        assert same_bits(a["coords"], b["coords"]) and same_bits(a["normals"], b["normals"])
    vol.free()
