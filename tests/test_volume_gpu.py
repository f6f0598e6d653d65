"""Resident volumes: the pass that lays the values out, takes their range and
their brick table (kvsmc_volume_upload / _from_device / _update,
kvsmc_volume_minmax), at the edges of its bricks (8 cell planes x 2 cell rows
x 128 cells), for every value type.
"""
import numpy as np
import pytest

from kvs_gb300 import _abi

from .helpers import same_bits
from .test_stream_gpu import extract_batch

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = [(1, 1, 1), (1, 1, 130), (3, 1, 5), (1, 4, 129), (2, 2, 2), (8, 2, 128), (9, 3, 129), (10, 4, 130), (17, 5, 257),
          (18, 6, 131), (33, 7, 40)]


def _range(v):
    """GetMinMaxValues: the scan from values[0], the first of equal values, a NaN at [0] stays."""
    lo = hi = v.reshape(-1)[0]
    for x in v.reshape(-1)[1:]:
        lo = x if x < lo else lo
        hi = x if x > hi else hi
    return np.array([lo, hi]).astype(np.float64)


def _values(shape, dtype, seed):
    rng = np.random.default_rng(seed)
    if np.dtype(dtype).kind == "f":
        return rng.normal(size=shape).astype(dtype)
    info = np.iinfo(dtype)
    return rng.integers(info.min, info.max, shape, dtype=dtype, endpoint=True)


def _check(dv, v):
    assert np.array_equal(dv.download().view(np.uint8), v.view(np.uint8))
    with np.errstate(invalid="ignore"):
        assert same_bits(np.array(dv.minmax()), _range(v))


@pytest.mark.parametrize("dtype", _abi.DTYPES)
def test_layout_and_range(kvsmc_ctx, dtype):
    for i, shape in enumerate(SHAPES):
        v = _values(shape, dtype, 7 * i)
        dv = _abi.DeviceVolume.upload(kvsmc_ctx, v)
        _check(dv, v)
        w = _values(shape, dtype, 7 * i + 1)
        kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_volume_update(kvsmc_ctx.handle, dv.handle, w.ctypes.data), "update")
        _check(dv, w)
        dv.free()
        # device values where the kernel may read them, and one byte off that
        raw = torch.zeros(v.nbytes + 64, dtype=torch.uint8, device="cuda")
        for off in (0, v.itemsize, 1):
            raw[off:off + v.nbytes] = torch.from_numpy(v.reshape(-1).view(np.uint8).copy()).cuda()
            torch.cuda.synchronize()
            dv = _abi.DeviceVolume.from_device(kvsmc_ctx, raw.data_ptr() + off, dtype, shape)
            _check(dv, v)
            dv.free()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_range_of_special_values(kvsmc_ctx, dtype):
    """Zeros of both signs, infinities, NaN at the start, inside and everywhere."""
    base = np.abs(_values((10, 4, 130), dtype, 3)) + 1
    for edit in (
        lambda a: a.put([5, 700], [-0.0, 0.0]), lambda a: a.put([5, 700], [0.0, -0.0]),
        lambda a: a.put([4000, 4001], [-np.inf, np.inf]), lambda a: a.put([3, 999], [np.nan, -1.0]),
        lambda a: a.put([0], [np.nan]), lambda a: a.fill(np.nan), lambda a: a.fill(np.inf), lambda a: a.fill(-0.0),
        lambda a: (a.__imul__(-1), a.put([129, 128 * 30], [0.0, -0.0])),
    ):
        v = base.copy()
        edit(v)
        dv = _abi.DeviceVolume.upload(kvsmc_ctx, v)
        with np.errstate(invalid="ignore"):
            assert same_bits(np.array(dv.minmax()), _range(v))
        dv.free()


@pytest.mark.parametrize("shape", [(9, 3, 129), (18, 6, 300), (41, 35, 131)])
def test_sparse_volumes_after_freed_ones(kvsmc_ctx, oracle_lib, shape):
    """Features in single bricks, in blocks that earlier volumes gave back: a
    stale or misplaced brick table would skip them."""
    rng = np.random.default_rng(1)
    for _ in range(6):
        v = np.zeros(shape, np.uint8)
        at = tuple(int(rng.integers(0, n)) for n in shape)
        v[at] = 200
        dv = _abi.DeviceVolume.upload(kvsmc_ctx, v)
        got = extract_batch(kvsmc_ctx, [dv], [_abi.make_params(100.0, 0)], _abi.PATH_AUTO)[0]
        ref = oracle_lib.extract(v, 100.0, 0, 0.0, 200.0)
        assert got["ntri"] > 0 and same_bits(got["coords"], ref["coords"]) and same_bits(got["normals"], ref["normals"])
        dv.free()
