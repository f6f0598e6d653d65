"""Unstructured cells, structured slices and STL records, at the edges of their
warps' blocks of cells, groups of rows and tiles, against the oracles."""
import numpy as np
import pytest

from kvs_gb300 import _abi
from kvs_gb300.marching_cubes import StructuredVolumeObject, TransferFunction
from kvs_gb300.slice_plane import SlicePlane
from oracle import cells as ocells
from oracle import export as oexport
from oracle import slice as oslice

from . import cell_meshes as cm
from .helpers import first_diff, golden, same_bits

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ct", [0, 1, 2, 3])
@pytest.mark.parametrize("ncells", [1, 31, 33, 127, 1025, 700001])
def test_cells_in_blocks(kvsmc_ctx, ct, ncells):
    """Random connectivity (most cells cut: rounds end at the vertex pool);
    blocks of one group, of several (700001 cells), a partial last one, and a
    mesh whose triangles are few and far between."""
    xyz, conn = cm.random_mesh(ct, 4000, ncells, seed=ncells + ct)
    v = np.random.default_rng(ncells).standard_normal(4000).astype(np.float32)
    isos = (0.1,) if ncells > 100000 else (0.1, float(np.sort(v)[-2]))
    for iso in isos:
        c, n, _ = _abi.marching_cells_host(kvsmc_ctx, ct, v, xyz, conn, iso, (-3.0, 3.0))
        o = ocells.marching_cells(ct, v, xyz, conn, iso, (-3.0, 3.0))
        assert same_bits(c, o["coords"]), (ct, ncells, iso, first_diff(c, o["coords"]))
        assert same_bits(n, o["normals"]), (ct, ncells, iso)


@pytest.mark.parametrize("shape", [(2, 2, 2), (5, 34, 3), (9, 7, 40), (3, 5, 700), (4, 3, 4100)])
def test_slice_planes(kvsmc_ctx, shape):
    """Planes across, along and nearly along the rows (32 rows to one row a
    warp), through nodes, on the volume's faces, past it, with coefficients far
    apart in size: the intervals of cells a row is searched in hold every cut
    cell."""
    nz, ny, nx = shape
    rng = np.random.default_rng(nx)
    v = rng.random(shape).astype(np.float32)
    table = golden()[1]["colormap256"]
    mid = [(nx - 1) / 2, (ny - 1) / 2, (nz - 1) / 2]
    normals = [(1, 0, 0), (0, -1, 0), (0, 0, 1), (1, 1, 1), (-0.37, 0.81, 0.45), (0.02, 1, -0.6), (1e-3, 0.5, 0.25),
               (1e-9, 0, 1), (1e-42, 0.5, 0.25), (3e-20, 5e-20, -2e-20), (1e30, -3e30, 2e30), (1, 1e-7, 1e6)]
    planes = [(*n, -float(np.dot(n, mid)) + off * float(np.abs(n).max())) for n in normals for off in (0.0, 0.31)]
    planes += [(1, 0, 0, 0), (1, 0, 0, -(nx - 1)), (0, 0, -1, nz - 1), (1, 2, 3, 1e9), (0, 0, 0, 1), (0, 0, 0, -1)]
    for coef in planes:
        s = SlicePlane(StructuredVolumeObject(v), coefficients=coef, transfer_function=TransferFunction(256),
                       context=kvsmc_ctx)
        c, rgb, n = oslice.slice_plane(v, s.coefficients(), table, np.float32(v.min()), np.float32(v.max()))
        assert same_bits(s.coords(), c), (coef, first_diff(s.coords(), c))
        assert np.array_equal(s.colors(), rgb), coef
        assert same_bits(s.normals(), n), coef


@pytest.mark.parametrize("ntri", [1, 2, 63, 64, 65, 128, 5000, 700003])
@pytest.mark.parametrize("shift", [0, 1])
def test_stl_records_in_tiles(kvsmc_ctx, ntri, shift):
    """Partial and whole tiles, two and more a warp, from arrays on and off a
    16-byte boundary; nothing is written past the last record."""
    rng = np.random.default_rng(ntri)
    coords = rng.standard_normal(9 * ntri).astype(np.float32)
    normals = rng.standard_normal(3 * ntri).astype(np.float32)
    want = oexport.stl_binary(coords, normals, np.zeros(0, np.uint32), oexport.POLYGON_NORMAL)[84:]
    c = torch.zeros(9 * ntri + 4, device="cuda")
    n = torch.zeros(3 * ntri + 4, device="cuda")
    c[shift:shift + 9 * ntri] = torch.from_numpy(coords).cuda()
    n[shift:shift + 3 * ntri] = torch.from_numpy(normals).cuda()
    out = torch.full((50 * ntri + 64,), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    kvsmc_ctx.check(kvsmc_ctx.lib.kvsmc_stl_records(kvsmc_ctx.handle, _abi.MODE_DUP_POLYGON_NORMAL, c[shift:].data_ptr(),
                                                    n[shift:].data_ptr(), None, 3 * ntri, ntri, out.data_ptr()), "records")
    got = out.cpu().numpy()
    assert got[:50 * ntri].tobytes() == want and (got[50 * ntri:] == 7).all()
