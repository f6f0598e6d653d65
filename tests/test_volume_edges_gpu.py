"""Resident volumes at the edges of the pass that lays them out: uploads on two
streams, warps that go on to a second brick; volumes freed while other work is
under way.
"""
import ctypes as C
import threading
import time

import numpy as np
import pytest

from kvs_gb300 import _abi, ingest

from .helpers import same_bits
from .test_volume_gpu import _check, _values

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


def test_a_volume_freed_while_another_thread_captures(kvsmc_ctx):
    """A wait for the whole device is refused during a capture and ends it:
    giving a volume's block back must not need one."""
    x = torch.zeros(1000, device="cuda")
    vols = [_abi.DeviceVolume.upload(kvsmc_ctx, np.full((20, 30, 40), 5, np.uint8)) for _ in range(3)]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        x += 1
        t = threading.Thread(target=lambda: [v.free() for v in vols])
        t.start()
        t.join()
        x += 1
    g.replay()
    torch.cuda.synchronize()
    assert x.eq(2).all()


def test_a_volume_freed_behind_a_queued_upload(kvsmc_ctx):
    """The upload waits on one stream while the volume is freed from another:
    the next volume in its block must not get the late values."""
    def host(value):
        pinned = torch.empty(40 * 64 * 64 * 4, dtype=torch.uint8).pin_memory()
        h = pinned.numpy().view(np.float32).reshape(40, 64, 64)
        h[...] = value
        return pinned, h

    (p1, first), (p2, second) = host(1.0), host(2.0)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    try:
        for _ in range(4):
            with torch.cuda.stream(a):
                torch.cuda._sleep(5_000_000)
            kvsmc_ctx.set_stream(a.cuda_stream)
            v1 = _abi.DeviceVolume.upload(kvsmc_ctx, first)
            kvsmc_ctx.set_stream(b.cuda_stream)
            v1.free()
            v2 = _abi.DeviceVolume.upload(kvsmc_ctx, second)
            torch.cuda.synchronize()
            assert np.array_equal(v2.download(), second) and v2.minmax() == (2.0, 2.0)
            v2.free()
    finally:
        torch.cuda.synchronize()
        kvsmc_ctx.set_stream(None)


def test_a_volume_freed_behind_a_replay(kvsmc_ctx):
    """A plan's replay is queued on a stream of the caller's when its volume is
    freed and others are uploaded: it still reads the volume's own values."""
    rng = np.random.default_rng(2)
    v = rng.random((30, 32, 36)).astype(np.float32)
    w = np.zeros_like(v)
    vol = _abi.DeviceVolume.upload(kvsmc_ctx, v)
    params = _abi.make_params(0.5, 0)
    s = _abi.Sizes()
    kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_count(kvsmc_ctx.handle, vol.handle, params, s), "count")
    want, got = [torch.zeros(s.ncoords, device="cuda") for _ in range(2)]
    normals = torch.zeros(s.nnormals, device="cuda")
    torch.cuda.synchronize()
    reqs = (_abi.Request * 1)()
    reqs[0].volume, reqs[0].params = vol.handle, params
    reqs[0].d_normals, reqs[0].normals_capacity = normals.data_ptr(), normals.numel()
    reqs[0].d_coords, reqs[0].coords_capacity = want.data_ptr(), want.numel()
    kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_extract_batch(kvsmc_ctx.handle, reqs, 1), "extract")
    reqs[0].d_coords = got.data_ptr()
    plan = _abi.Plan(kvsmc_ctx, reqs)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(5_000_000)
    plan.launch(stream.cuda_stream)
    vol.free()
    later = [_abi.DeviceVolume.upload(kvsmc_ctx, w) for _ in range(4)]
    plan.wait()
    torch.cuda.synchronize()
    assert torch.equal(want, got)
    plan.close()
    for x in later:
        x.free()


def test_a_request_behind_a_queued_update(kvsmc_ctx):
    """A served volume is updated on a busy stream and asked for again: the
    workers wait for the new values, whether they have seen the volume before
    or not."""
    def host(value):
        pinned = torch.empty(32 * 32 * 32 * 4, dtype=torch.uint8).pin_memory()
        h = pinned.numpy().view(np.float32).reshape(32, 32, 32)
        h[...] = 0.0
        h[8:8 + value, 8:20, 8:20] = 1.0
        return pinned, h

    hosts = [host(k) for k in (3, 7, 11, 2)]
    params = _abi.make_params(0.5, 0, (0.0, 1.0))
    want = []
    for _, h in hosts:
        v = _abi.DeviceVolume.upload(kvsmc_ctx, h)
        s = _abi.Sizes()
        kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_count(kvsmc_ctx.handle, v.handle, params, s), "count")
        want.append(s.ntriangles)
        v.free()
    assert len(set(want)) == len(want)
    vol = _abi.DeviceVolume.upload(kvsmc_ctx, hosts[-1][1])
    stream = torch.cuda.Stream()
    srv = _abi.Server(kvsmc_ctx, budget_bytes=1 << 26, max_batch=4, workers=2)
    try:
        for turn in range(3):
            for (_, h), n in zip(hosts, want):
                with torch.cuda.stream(stream):
                    torch.cuda._sleep(3_000_000)
                kvsmc_ctx.set_stream(stream.cuda_stream)
                kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_volume_update(kvsmc_ctx.handle, vol.handle, h.ctypes.data), "update")
                kvsmc_ctx.set_stream(None)
                ticket, done = srv.submit(vol, params), []
                while not done:
                    done = srv.poll(timeout_ms=2000)
                assert [c.ticket for c in done] == [ticket] and done[0].status == _abi.OK
                assert done[0].sizes.ntriangles == n, (turn, n)
                srv.release(ticket)
    finally:
        kvsmc_ctx.set_stream(None)
        srv.close()
        torch.cuda.synchronize()
        vol.free()


def test_the_longest_row(kvsmc_ctx):
    """2^32 - 1 nodes: the last brick's end is not a 32-bit number."""
    n = (1 << 32) - 1
    src = torch.full((n,), 100, dtype=torch.uint8, device="cuda")
    src[-1], src[n - 200] = 7, 201
    torch.cuda.synchronize()
    vol = _abi.DeviceVolume.from_device(kvsmc_ctx, src.data_ptr(), np.uint8, (1, 1, n))
    assert vol.minmax() == (7.0, 201.0)
    vol.free()


@pytest.mark.parametrize("dtype", _abi.DTYPES)
def test_volumes_without_a_brick_table(kvsmc_ctx, dtype):
    """One node thick, rows wider than the streaming kernels', and the wide
    types: values in index order, 256 at a time, rows longer and much shorter
    than that; the range is taken when it is asked for."""
    for i, shape in enumerate([(1, 700, 3), (5, 3, 257), (2, 2, 4100), (300, 1, 2), (257, 1, 1), (1, 1, 256), (3, 5, 64)]):
        v = _values(shape, dtype, i)
        if np.dtype(dtype).kind == "f":
            v.reshape(-1)[[1, 300 % v.size, v.size - 1]] = (-np.inf, np.nan, np.inf)
        dv = _abi.DeviceVolume.upload(kvsmc_ctx, v)
        _check(dv, v)
        w = _values(shape, dtype, 50 + i)
        kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_volume_update(kvsmc_ctx.handle, dv.handle, w.ctypes.data), "update")
        _check(dv, w)
        dv.free()
        raw = torch.from_numpy(v.reshape(-1).view(np.uint8).copy()).cuda()
        torch.cuda.synchronize()
        dv = _abi.DeviceVolume.from_device(kvsmc_ctx, raw.data_ptr(), dtype, shape)
        _check(dv, v)
        dv.free()


def test_zero_signs_of_doubles(kvsmc_ctx):
    base = np.full((4, 9, 301), 2.0)
    for at, want in (([3, 700], -0.0), ([700, 3], 0.0), ([5000, 9], 0.0), ([0, 4], -0.0)):
        for sign in (1.0, -1.0):
            v = base * sign
            v.put(at, [-0.0, 0.0])
            dv = _abi.DeviceVolume.upload(kvsmc_ctx, v)
            lo, hi = dv.minmax()
            assert same_bits(np.array([lo, hi]), np.array([want, 2.0] if sign > 0 else [-2.0, want])), (at, sign, lo, hi)
            dv.free()


@pytest.mark.parametrize("dtype", [np.float64, np.uint64, np.int32])
def test_the_range_asked_for_by_two_contexts(kvsmc_ctx, dtype):
    """One context's pass for a volume's range waits on a busy stream: another
    context that asks for it meanwhile takes its own."""
    v = _values((40, 50, 64), dtype, 5)   # (no padding: the upload leaves the range to whoever asks)
    dv = _abi.DeviceVolume.upload(kvsmc_ctx, v)
    kvsmc_ctx.synchronize()
    other = _abi.Context(0)
    stream = torch.cuda.Stream()
    got = {}

    def ask(ctx, name):
        lo, hi = C.c_double(), C.c_double()
        ctx.check(ctx.lib.kvsmc_volume_minmax(ctx.handle, dv.handle, C.byref(lo), C.byref(hi)), "minmax")
        got[name] = (lo.value, hi.value)

    with torch.cuda.stream(stream):
        torch.cuda._sleep(200_000_000)
    other.set_stream(stream.cuda_stream)
    t = threading.Thread(target=ask, args=(other, "other"))
    t.start()
    time.sleep(0.02)
    ask(kvsmc_ctx, "first")
    t.join()
    torch.cuda.synchronize()
    other.set_stream(None)
    other.close()
    want = (float(v.min()), float(v.max()))
    assert got == {"first": want, "other": want}
    dv.free()


@pytest.mark.parametrize("dtype", [np.uint8, np.float32, np.float64])
@pytest.mark.parametrize("nx", [64, 61])
def test_a_captured_update(kvsmc_ctx, dtype, nx):
    """An update from pinned memory captured into a graph: each replay brings the
    buffer's present values, whatever the context uploaded in between."""
    shape = (20, 30, nx)
    n = int(np.prod(shape)) * np.dtype(dtype).itemsize
    pinned = torch.empty(n, dtype=torch.uint8).pin_memory()
    h = pinned.numpy().view(dtype).reshape(shape)
    h[...] = _values(shape, dtype, 1)
    dv = _abi.DeviceVolume.upload(kvsmc_ctx, h)
    kvsmc_ctx.synchronize()
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    try:
        with torch.cuda.graph(graph, stream=stream):
            kvsmc_ctx.set_stream(stream.cuda_stream)
            st = kvsmc_ctx.lib.kvsmc_volume_update(kvsmc_ctx.handle, dv.handle, h.ctypes.data)
    finally:
        kvsmc_ctx.set_stream(None)
    assert st == _abi.OK
    for turn in (2, 3):
        h[...] = v = _values(shape, dtype, turn)
        later = _abi.DeviceVolume.upload(kvsmc_ctx, _values((30, 40, nx), dtype, 7))
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(dv.download(), v)
        params = _abi.make_params(float(np.median(v)), 0, (float(v.min()), float(v.max())))
        s, w = _abi.Sizes(), _abi.Sizes()
        kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_count(kvsmc_ctx.handle, dv.handle, params, s), "count")
        fresh = _abi.DeviceVolume.upload(kvsmc_ctx, v)
        kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_count(kvsmc_ctx.handle, fresh.handle, params, w), "count")
        assert s.ntriangles == w.ntriangles > 0
        later.free()
        fresh.free()
    # an update outside the graph still works, and so does freeing
    v = _values(shape, dtype, 9)
    kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_volume_update(kvsmc_ctx.handle, dv.handle, v.ctypes.data), "update")
    _check(dv, v)
    dv.free()


@pytest.mark.parametrize("dtype,nx", [(np.float64, 1023), (np.float64, 1025), (np.uint64, 4097), (np.int32, 2047),
                                      (np.int32, 2049), (np.uint8, 8191), (np.uint8, 8193), (np.float32, 4099)])
def test_long_padded_rows(kvsmc_ctx, dtype, nx):
    """Volumes without a table, either side of the row length that is staged: the
    values, the range, and a count."""
    v, w = _values((3, 5, nx), dtype, nx), _values((3, 5, nx), dtype, nx + 1)
    dv = _abi.DeviceVolume.upload(kvsmc_ctx, v)
    _check(dv, v)
    kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_volume_update(kvsmc_ctx.handle, dv.handle, w.ctypes.data), "update")
    _check(dv, w)
    sizes = [_abi.Sizes(), _abi.Sizes()]
    for path, s in zip((_abi.PATH_AUTO, _abi.PATH_GATHER), sizes):
        kvsmc_ctx.set_kernel_path(path)
        kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_count(kvsmc_ctx.handle, dv.handle, _abi.make_params(float(np.median(w)), 0), s), "count")
    kvsmc_ctx.set_kernel_path(_abi.PATH_AUTO)
    assert sizes[0].ntriangles == sizes[1].ntriangles > 0
    dv.free()


def test_an_update_behind_a_loaded_file(kvsmc_ctx, tmp_path):
    """Doubles of the other byte order, whose range the header gives, are turned by
    a pass that the load leaves running: an update on another stream waits for it."""
    shape = (32, 64, 64)
    v, w = _values(shape, np.float64, 1), _values(shape, np.float64, 2)
    (tmp_path / "v.dat").write_bytes(v.astype(">f8").tobytes())
    (tmp_path / "v.kvsml").write_text(
        '<?xml version="1.0" ?><KVSML><Object type="StructuredVolumeObject"><StructuredVolumeObject grid_type="uniform" '
        'resolution="64 64 32"><Node><Value veclen="1" min_value="-9" max_value="9"><DataArray type="double" '
        'format="binary" file="v.dat" endian="big" /></Value></Node></StructuredVolumeObject></Object></KVSML>')
    pinned = torch.from_numpy(w.copy()).pin_memory()
    busy = torch.ones(1 << 28, device="cuda")
    a, b, c = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    try:
        for turn in range(2):
            with torch.cuda.stream(c):
                for _ in range(300):
                    busy.sin_()   # (the GPU's SMs are taken)
            kvsmc_ctx.set_stream(a.cuda_stream)
            dv, info = ingest.load_kvsml(kvsmc_ctx, tmp_path / "v.kvsml")
            assert info["byte_swap"] and info["volume_max"] == 9.0
            if turn == 1:
                kvsmc_ctx.set_stream(b.cuda_stream)
                kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_volume_update(kvsmc_ctx.handle, dv.handle, pinned.data_ptr()), "update")
            torch.cuda.synchronize()
            assert np.array_equal(dv.download(), w if turn == 1 else v)
            dv.free()
    finally:
        torch.cuda.synchronize()
        kvsmc_ctx.set_stream(None)
