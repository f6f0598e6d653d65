"""Resident volumes at the edges of the pass that lays them out: uploads on two
streams, warps that go on to a second brick.
"""
import numpy as np
import pytest

from kvs_gb300 import _abi

from .helpers import same_bits

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("update", [False, True])
def test_uploads_on_two_streams(kvsmc_ctx, update):
    """Host volumes with padded rows go through one staging buffer of the
    context: an upload on one stream must not overwrite what the pass of an
    upload on another one still reads."""
    shape = (60, 300, 301)
    sizes = [shape, (60, 301, 299), (7, 9, 5), shape]   # (padded rows, the last ones smaller than the buffer)
    hosts = []
    for i, s in enumerate(sizes):
        pinned = torch.empty(int(np.prod(s)) * 4, dtype=torch.uint8).pin_memory()
        h = pinned.numpy().view(np.float32).reshape(s)
        h[...] = np.arange(h.size, dtype=np.float32).reshape(s) % 997 + 1000 * i
        hosts.append((pinned, h))
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    vols = [_abi.DeviceVolume.upload(kvsmc_ctx, h) for _, h in hosts] if update else [None] * len(hosts)
    kvsmc_ctx.synchronize()
    torch.cuda.synchronize()
    try:
        for turn in range(6):
            order = range(len(hosts)) if turn % 2 == 0 else reversed(range(len(hosts)))
            for j, i in enumerate(order):
                kvsmc_ctx.set_stream(streams[j % 2].cuda_stream)
                if j == 0:
                    with torch.cuda.stream(streams[0]):
                        torch.cuda._sleep(2_000_000)   # the first one starts behind other work
                if update:
                    kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_volume_update(kvsmc_ctx.handle, vols[i].handle,
                                                                      hosts[i][1].ctypes.data), "update")
                else:
                    vols[i] = _abi.DeviceVolume.upload(kvsmc_ctx, hosts[i][1])
            torch.cuda.synchronize()
            for i, (_, h) in enumerate(hosts):
                assert np.array_equal(vols[i].download(), h), (turn, i)
                if not update:
                    vols[i].free()
    finally:
        torch.cuda.synchronize()
        kvsmc_ctx.set_stream(None)
    if update:
        for v in vols:
            v.free()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("sign", [1, -1])
def test_sign_of_a_zero_end_across_bricks(kvsmc_ctx, dtype, sign):
    """The range keeps the first of equal values in index order.  With more
    bricks in a plane than warps on the GPU, a warp meets a brick's high planes
    before the low planes of a later brick."""
    bricks = torch.cuda.get_device_properties(0).multi_processor_count * 64
    base = np.full((9, 2 * bricks + 9, 2), 3.0 * sign, dtype)
    for first, second in ((-0.0, 0.0), (0.0, -0.0)):
        v = base.copy()
        v[0, 2 * bricks + 1, 0] = first    # the lowest index, in no brick but the first warp's second one
        v[7, 0, 0] = second                # in its first one
        dv = _abi.DeviceVolume.upload(kvsmc_ctx, v)
        lo, hi = dv.minmax()
        want = (first, 3.0) if sign > 0 else (-3.0, first)
        assert same_bits(np.array([lo, hi]), np.array(want)), (lo, hi, want)
        dv.free()
