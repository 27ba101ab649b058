"""Coarse levels kept from one response to the next, and the smallest meshes
that have them: fixed rows changed on one mesh, the levels switched off and on,
1024 to 8191 nodes with every smoother; and the model update on values that are
not finite.

Tolerance: as in the comparison of every smoother with the plain FP64 PCG, 1e-8
of the potentials' column maximum; kept levels give the fresh operator's result
bit for bit."""
import os

import numpy as np
import pytest

from pygimli_gb300 import DataContainerERT, Mesh, create_box_mesh_3d
from pygimli_gb300.data import geometricFactors, grid_line_scheme

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    from pygimli_gb300 import build
    build.build()
    return t


def box(nx, ny, h, **kw):
    e = np.array([(x, y) for x in np.arange(nx) * 4.0 for y in np.arange(ny) * 4.0])
    mesh = create_box_mesh_3d(e, h=h, **kw)
    data = DataContainerERT(np.column_stack([e, np.zeros(len(e))]), grid_line_scheme((nx, ny), "pd"))
    data.set("k", geometricFactors(data, 3))
    return mesh, data


def operator(mesh, data, form, **kw):
    import pygimli_gb300
    from pygimli_gb300 import ERTModelling
    if form == "learned":
        kw["weights"] = os.path.join(os.path.dirname(pygimli_gb300.__file__), "weights", "box_3d.npz")
    if form != "fp64":
        kw.update(precision="mixed", precond=form)
    f = ERTModelling(maxIter=200000, **kw)
    f.setData(data)
    f.setMesh(mesh, ignoreRegionManager=True)
    return f


def ground(mesh, seed):
    return np.exp(np.random.default_rng(seed).normal(np.log(100.0), 1.0, mesh.cellCount()))


@pytest.mark.parametrize("form", ["fp64", "fsai"])
def test_changed_fixed_rows(torch, form):
    """Other calibration nodes through the library's own call, the mesh kept."""
    mesh, data = box(5, 3, 2.0, para_depth=10.0, outer=120.0, growth=1.5)
    data.set("k", np.ones(data.size()))
    bm = np.array(mesh.boundary_markers)
    bm[bm == -2] = -1  # closed domain

    def closed(calib):
        nm = np.array(mesh.node_markers)
        nm[calib] = -1000
        return Mesh(3, mesh.nodes, mesh.cells, mesh.cell_markers, nm, mesh.boundaries, bm, mesh.boundary_cells)

    rho = ground(mesh, 1)
    f = operator(closed(7), data, form, sr=False)
    f.response(rho)
    for calib in ([4321], [7], [100, 2000, 9000]):
        nodes = np.asarray(calib, np.int32)
        f._check(f._lib.ertgb_set_reference(f._ctx, int(f._bc.ref_elec), -1, len(nodes), nodes.ctypes.data))
        fresh = operator(closed(calib), data, form, sr=False)
        assert np.array_equal(f.response(rho), fresh.response(rho))
        assert f.stats()["iterations"] == fresh.stats()["iterations"] <= 90


@pytest.mark.parametrize("form", ["fp64", "jacobi", "fsai"])
def test_switched(torch, form):
    mesh, data = box(4, 3, 4.0, para_depth=10.0, outer=80.0)
    a, b = ground(mesh, 1), ground(mesh, 2)
    f = operator(mesh, data, form)
    on = [f.response(a), f.response(b)]
    few = f.stats()["iterations"]
    f.setCoarseLevels(False)
    off = [f.response(a), f.response(b)]
    assert f.stats()["iterations"] > 2 * few
    f.setCoarseLevels(True)
    assert all(np.array_equal(x, f.response(r)) for x, r in zip(on, (a, b)))
    g = operator(mesh, data, form)
    g.setCoarseLevels(False)
    assert all(np.array_equal(x, g.response(r)) for x, r in zip(off, (a, b)))


@pytest.mark.parametrize("form", ["fp64", "jacobi", "fsai", "learned"])
@pytest.mark.parametrize("outer,growth,lo,hi", [(60.0, 2.6, 1024, 1900), (60.0, 1.8, 1900, 4096), (120.0, 1.45, 4096, 8192)])
def test_small_meshes(torch, form, outer, growth, lo, hi):
    mesh, data = box(4, 2, 4.0, para_depth=8.0, outer=outer, growth=growth)
    assert lo <= mesh.nodeCount() < hi
    fast, exact = operator(mesh, data, form), operator(mesh, data, "fp64", rtol=1e-12)
    exact.setCoarseLevels(False)
    for seed in (1, 2):
        rho = ground(mesh, seed)
        r, r0 = fast.response(rho), exact.response(rho)
        u, u0 = fast.subPotentials(), exact.subPotentials()
        assert float(np.max(np.abs(u - u0).max(axis=2) / np.abs(u0).max(axis=2))) <= 1e-8
        assert float(np.max(np.abs(r - r0) / np.maximum(np.abs(r0), 1e-3))) <= 1e-5
        st = fast.stats()
        assert 0 < st["iterations"] <= 90 and st["stalled_columns"] == 0


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_update_on_values_not_finite(torch, value):
    """Unaligned FP32 rows are widened by integer operations: infinities and NaN
    stay what they are and stop the update as in FP64."""
    from pygimli_gb300.inversion import cgls
    rng = np.random.default_rng(1)
    J = rng.standard_normal((9, 37)).astype(np.float32)
    J[4, 11] = value
    n = 36
    C = (np.arange(0, 2 * n + 1, 2, dtype=np.int64), np.stack([np.arange(n), np.arange(1, n + 1)], 1).ravel().astype(np.int32),
         np.tile([1.0, -1.0], n), 37)
    for dt in (np.float32, np.float64):
        with pytest.raises(Exception, match="non-finite"):
            cgls(torch.as_tensor(J.astype(dt), device="cuda"), C, np.ones(9), np.ones(9), np.ones(37), np.ones(n),
                 np.ones(37), np.ones(37), np.ones(9), 20.0, np.zeros(n), max_iter=4, tol=0.0)
