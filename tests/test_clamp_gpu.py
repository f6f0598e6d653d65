"""Vertices of 8/16-bit volumes under a preset min/max whose ends cut into the
data: the interpolation clamps the corner values to them, and an end that is a
float but no whole number makes the difference of two clamped values one that
a single float does not hold.  All three modes, alone and in a batch, against
the oracle.
"""
import numpy as np
import pytest

from kvs_gb300 import _abi

from .helpers import first_diff, same_bits
from .test_stream_gpu import extract_batch

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")


def _f(x):
    return float(np.float32(x))


# per type: the range's ends, then isolevels
RANGES = {
    np.uint8: [(_f(10.1), _f(200.7), (100.3, 11.0, 200.0)), (_f(0.1), 255.0, (100.0, 3.5, 0.7)),
               (0.0, _f(100.0625), (100.0, 50.25)), (20.0, 200.0, (100.3, 20.5, 199.9)),
               (-0.5, 255.5, (100.3, 0.5)), (_f(10.3), 1e6, (50.5, 10.6))],
    np.int8: [(_f(-100.3), _f(90.7), (0.5, -100.0, 90.5)), (-128.0, _f(10.1), (3.3, 10.05)), (-50.0, 50.0, (0.25, -49.5)),
              (_f(-1e-3), _f(1e-3), (0.0, 0.0005))],
    np.uint16: [(_f(1234.567), _f(60000.37), (30000.5, 1300.0, 60000.2)), (_f(0.1), 65535.0, (777.0, 60000.75)),
                (1000.0, 60000.0, (30000.5, 1000.5)), (-1.5, 65535.5, (30000.5,))],
    np.int16: [(_f(-30000.7), _f(29999.3), (0.5, -123.25, 29999.1)), (_f(-0.3), _f(0.7), (0.0, 0.5)),
               (-20000.0, 20000.0, (0.5, 19999.5))],
}


@pytest.mark.parametrize("dtype", list(RANGES))
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_a_range_that_cuts_the_data(kvsmc_ctx, oracle_lib, dtype, mode):
    rng = np.random.default_rng(3 + mode)
    info = np.iinfo(dtype)
    # noise over the type's range, and a volume of small steps around the isolevels
    noise = rng.integers(info.min, info.max, (7, 24, 130), dtype=dtype, endpoint=True)
    for lo, hi, isos in RANGES[dtype]:
        mid = np.clip(np.round(isos[0] + rng.normal(0, (hi - lo) / 4, (6, 11, 60))), info.min, info.max).astype(dtype)
        for v in (noise, mid):
            vol = _abi.DeviceVolume.upload(kvsmc_ctx, v)
            params = [_abi.make_params(x, mode, (lo, hi)) for x in isos]
            together = extract_batch(kvsmc_ctx, [vol] * len(isos), params, _abi.PATH_AUTO)
            for x, p, o in zip(isos, params, together):
                ref = oracle_lib.extract(v, x, mode, lo, hi)
                alone = extract_batch(kvsmc_ctx, [vol], [p], _abi.PATH_AUTO)[0]
                for how, got in (("together", o), ("alone", alone)):
                    tag = (how, np.dtype(dtype).name, mode, lo, hi, x)
                    assert same_bits(got["coords"], ref["coords"]), (tag, first_diff(got["coords"], ref["coords"]))
                    assert same_bits(got["normals"], ref["normals"]), (tag, first_diff(got["normals"], ref["normals"]))
                    if mode:
                        assert np.array_equal(got["connections"], ref["connections"].view(np.uint32)), tag
            vol.free()


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("dtype,lo,hi,isos", [
    (np.uint8, 0.0, 100.0625, (100.07, 100.5, 100.99)), (np.int8, -100.0, -3.75, (-3.7, -3.5, -3.01)),
    (np.uint16, 0.0, 1000.5, (1000.51, 1000.75)), (np.int16, -30000.0, 0.25, (0.25, 0.3, 0.9)),
])
def test_an_isolevel_past_the_upper_end(kvsmc_ctx, oracle_lib, dtype, lo, hi, isos, mode):
    """The upper end lies below the isolevel, with no value of the type between
    them: an edge's clamped values are both below it, and the interpolation
    ratio, an absolute value, starts from a negative quotient."""
    info = np.iinfo(dtype)
    v = np.random.default_rng(8).integers(info.min, info.max, (6, 13, 70), dtype=dtype, endpoint=True)
    vol = _abi.DeviceVolume.upload(kvsmc_ctx, v)
    params = [_abi.make_params(x, mode, (lo, hi)) for x in isos]
    together = extract_batch(kvsmc_ctx, [vol] * len(isos), params, _abi.PATH_AUTO)
    for x, p, o in zip(isos, params, together):
        ref = oracle_lib.extract(v, x, mode, lo, hi)
        assert ref["coords"].size
        for got in (o, extract_batch(kvsmc_ctx, [vol], [p], _abi.PATH_AUTO)[0]):
            assert same_bits(got["coords"], ref["coords"]), (x, first_diff(got["coords"], ref["coords"]))
            assert same_bits(got["normals"], ref["normals"]), (x, first_diff(got["normals"], ref["normals"]))
    vol.free()
