"""Counts alone of 32/64-bit integer and double volumes: by cells or by the
streaming kernels, by the volume's size, its rows and the requests of the call;
the same sizes either way, and the extraction's.
"""
import numpy as np
import pytest

from kvs_gb300 import _abi

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

WIDE = [np.int32, np.uint32, np.int64, np.uint64, np.float64]


def _counts(ctx, vol, params, path):
    reqs = (_abi.Request * len(params))()
    for r, p in zip(reqs, params):
        r.volume, r.params = vol.handle, p
    ctx.set_kernel_path(path)
    ctx.check(ctx.lib.kvsmc_count_batch(ctx.handle, reqs, len(params)), "count_batch")
    ctx.set_kernel_path(_abi.PATH_AUTO)
    return [_abi.sizes_dict(r.sizes) for r in reqs]


@pytest.mark.parametrize("dtype", WIDE)
@pytest.mark.parametrize("shape", [(6, 7, 2), (6, 7, 3), (6, 7, 4), (5, 9, 33), (5, 9, 34), (3, 40, 300), (2, 2, 2)])
def test_small_volumes(kvsmc_ctx, oracle_lib, dtype, shape):
    rng = np.random.default_rng(sum(shape))
    v = (rng.random(shape) * 1000).astype(dtype)
    lo, hi = float(v.min()), float(v.max())
    vol = _abi.DeviceVolume.upload(kvsmc_ctx, v)
    for mode in (0, 1, 2):
        params = [_abi.make_params(lo + (hi - lo) * (k + 0.5) / 3, mode) for k in range(3)]
        for group in (params[:1], params[1:], params):
            got = _counts(kvsmc_ctx, vol, group, _abi.PATH_AUTO)
            assert got == _counts(kvsmc_ctx, vol, group, _abi.PATH_GATHER)
            for p, s in zip(group, got):
                ref = oracle_lib.extract(v, p.isolevel, mode, lo, hi)
                assert s["ncoords"] == ref["coords"].size and s["nnormals"] == ref["normals"].size
                assert s["nconnections"] == (ref["connections"].size if mode else 0)
    vol.free()


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64, torch.float64])
@pytest.mark.parametrize("shape", [(170, 170, 173), (180, 171, 172), (300, 316, 320), (320, 300, 321)])
def test_sizes_around_the_rule(kvsmc_ctx, dtype, shape):
    """Either side of 5 and 30 million cells."""
    gen = torch.Generator(device="cuda").manual_seed(shape[0])
    t = torch.randint(0, 1000, shape, generator=gen, device="cuda").to(dtype)
    torch.cuda.synchronize()
    code = {torch.int32: np.int32, torch.int64: np.int64, torch.float64: np.float64}[dtype]
    vol = _abi.DeviceVolume.from_device(kvsmc_ctx, t.data_ptr(), code, shape)
    for mode in (0, 2):
        for isos in ([500.5], [300.0, 700.25]):
            params = [_abi.make_params(x, mode) for x in isos]
            assert _counts(kvsmc_ctx, vol, params, _abi.PATH_AUTO) == _counts(kvsmc_ctx, vol, params, _abi.PATH_GATHER)
    vol.free()


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64, torch.float64])
@pytest.mark.parametrize("shape", [(260, 316, 33), (290, 300, 33), (500, 555, 2), (520, 560, 2), (700, 870, 3), (740, 850, 3)])
def test_short_rows_together(kvsmc_ctx, dtype, shape):
    """Several requests on rows of few cells, either side of the rule."""
    gen = torch.Generator(device="cuda").manual_seed(shape[0])
    t = torch.randint(0, 1000, shape, generator=gen, device="cuda").to(dtype)
    torch.cuda.synchronize()
    code = {torch.int32: np.int32, torch.int64: np.int64, torch.float64: np.float64}[dtype]
    vol = _abi.DeviceVolume.from_device(kvsmc_ctx, t.data_ptr(), code, shape)
    params = [_abi.make_params(x, 0) for x in (100.5, 500.5, 900.25)]
    assert _counts(kvsmc_ctx, vol, params, _abi.PATH_AUTO) == _counts(kvsmc_ctx, vol, params, _abi.PATH_GATHER)
    vol.free()


@pytest.mark.parametrize("dtype", [torch.uint8, torch.int16, torch.float32])
@pytest.mark.parametrize("shape", [(500, 520, 9), (480, 520, 9), (520, 540, 8), (126, 126, 129), (215, 217, 217), (217, 217, 216)])
def test_shared_counts_of_narrow_types(kvsmc_ctx, dtype, shape):
    """One shared-vertex request, and two of one call, either side of 2 and 10
    million cells and of 8 cells a row."""
    gen = torch.Generator(device="cuda").manual_seed(shape[0])
    t = torch.randint(0, 100, shape, generator=gen, device="cuda").to(dtype)
    torch.cuda.synchronize()
    code = {torch.uint8: np.uint8, torch.int16: np.int16, torch.float32: np.float32}[dtype]
    vol = _abi.DeviceVolume.from_device(kvsmc_ctx, t.data_ptr(), code, shape)
    for mode in (1, 2):
        for isos in ([50.5], [30.0, 70.25]):
            params = [_abi.make_params(x, mode) for x in isos]
            assert _counts(kvsmc_ctx, vol, params, _abi.PATH_AUTO) == _counts(kvsmc_ctx, vol, params, _abi.PATH_GATHER)
    vol.free()
