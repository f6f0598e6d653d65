"""Many isolevels of a mesh: the emit's blocks of cells are larger than the
count's, by the isolevels times the mesh's size.
"""
import ctypes as C

import numpy as np
import pytest

from kvs_gb300 import _abi
from oracle import cells as ocells

from . import cell_meshes as cm
from .helpers import same_bits

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ncells,niso", [(1, 64), (31, 64), (1025, 64), (9728 * 32 // 32 + 5, 64), (100003, 40), (200001, 64),
                                         (640033, 3)])
@pytest.mark.parametrize("ct", [0, 2])
def test_blocks_of_a_sweep(kvsmc_ctx, ct, ncells, niso):
    rng = np.random.default_rng(ncells + ct)
    nodes = max(64, ncells // 4)
    xyz = rng.uniform(-4, 4, (nodes, 3)).astype(np.float32)
    conn = (rng.integers(0, nodes - 32, (ncells, 1)) + rng.integers(0, 32, (ncells, cm.NODES[ct]))).astype(np.uint32)
    v = (np.arange(nodes) / nodes).astype(np.float32)
    isos = [(k + 0.5) / niso for k in range(niso)]
    dv, dx, dk = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (v, xyz, conn.view(np.int32)))
    torch.cuda.synchronize()
    mesh = (kvsmc_ctx.handle, ct, dv.data_ptr(), 8, nodes, dx.data_ptr(), dk.data_ptr(), ncells)
    sizes = (_abi.Sizes * niso)()
    zero = (C.c_uint64 * niso)()
    il = (C.c_double * niso)(*isos)
    sweep = kvsmc_ctx.lib.kvsmc_marching_cells_sweep_device
    sweep(*mesh, il, niso, 1, 0.0, 1.0, None, zero, None, zero, sizes)
    t = [s.ntriangles for s in sizes]
    oc, on = ([torch.zeros(max(1, w * k), device="cuda") for k in t] for w in (9, 3))
    torch.cuda.synchronize()
    kvsmc_ctx.check(sweep(*mesh, il, niso, 1, 0.0, 1.0, (C.c_void_p * niso)(*[x.data_ptr() for x in oc]),
                          (C.c_uint64 * niso)(*[x.numel() for x in oc]), (C.c_void_p * niso)(*[x.data_ptr() for x in on]),
                          (C.c_uint64 * niso)(*[x.numel() for x in on]), sizes), "sweep")
    assert sum(t) > 0 or ncells < 100
    for i, iso in enumerate(isos):
        c, n, s = torch.zeros_like(oc[i]), torch.zeros_like(on[i]), _abi.Sizes()
        torch.cuda.synchronize()
        kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_marching_cells_device(*mesh, iso, 1, 0.0, 1.0, c.data_ptr(), c.numel(),
                                                                  n.data_ptr(), n.numel(), C.byref(s)), "cells")
        assert s.ntriangles == t[i] and torch.equal(c, oc[i]) and torch.equal(n, on[i]), i
    for i in (0, niso // 2, niso - 1):
        w = ocells.marching_cells(ct, v, xyz, conn, isos[i], (0.0, 1.0))
        assert same_bits(oc[i][:9 * t[i]].cpu().numpy(), w["coords"]) and same_bits(on[i][:3 * t[i]].cpu().numpy(), w["normals"])


@pytest.mark.parametrize("ncells", [640033, 1300001])
@pytest.mark.parametrize("niso", [1, 2])
def test_few_isolevels_of_noise(kvsmc_ctx, ncells, niso):
    """Nearly every cell cut: where the count's blocks are of several groups, the
    emit's are no smaller."""
    rng = np.random.default_rng(ncells)
    nodes = ncells // 4
    xyz = rng.uniform(-4, 4, (nodes, 3)).astype(np.float32)
    conn = rng.integers(0, nodes, (ncells, 4)).astype(np.uint32)
    dv, dx, dk = (torch.from_numpy(a).cuda() for a in (rng.random(nodes).astype(np.float32), xyz, conn.view(np.int32)))
    mesh = (kvsmc_ctx.handle, 0, dv.data_ptr(), 8, nodes, dx.data_ptr(), dk.data_ptr(), ncells)
    want, isos = [], [0.4, 0.7][:niso]
    for iso in isos:
        c, n, s = torch.zeros(18 * ncells, device="cuda"), torch.zeros(6 * ncells, device="cuda"), _abi.Sizes()
        torch.cuda.synchronize()
        kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_marching_cells_device(*mesh, iso, 1, 0.0, 1.0, c.data_ptr(), c.numel(),
                                                                  n.data_ptr(), n.numel(), C.byref(s)), "cells")
        want.append((c, n, s.ntriangles))
    got = [(torch.zeros_like(c), torch.zeros_like(n)) for c, n, _ in want]
    torch.cuda.synchronize()
    sizes = (_abi.Sizes * niso)()
    kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_marching_cells_sweep_device(
        *mesh, (C.c_double * niso)(*isos), niso, 1, 0.0, 1.0, (C.c_void_p * niso)(*[c.data_ptr() for c, _ in got]),
        (C.c_uint64 * niso)(*[c.numel() for c, _ in got]), (C.c_void_p * niso)(*[n.data_ptr() for _, n in got]),
        (C.c_uint64 * niso)(*[n.numel() for _, n in got]), sizes), "sweep")
    for (c, n, t), (gc, gn), s in zip(want, got, sizes):
        assert s.ntriangles == t > ncells // 2 and torch.equal(c, gc) and torch.equal(n, gn)
