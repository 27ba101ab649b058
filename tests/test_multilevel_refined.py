"""Coarse levels on the H2 and P2 refinements of electrode boxes, the forward
meshes of an inversion: their matrices coarsen to stars, whose rows all couple
to one hub.

Tolerance as for the other meshes: 1e-8 of the potentials' column maximum
against the plain FP64 PCG at rtol 1e-12.  The single level takes 256 (31,605
nodes) and 704 to 832 iterations (124,605 nodes, FSAI); the bars are about half
of that and a fifth."""
import numpy as np
import pytest

from pygimli_gb300 import DataContainerERT, create_box_mesh_3d
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


def operator(mesh, data, **kw):
    from pygimli_gb300 import ERTModelling
    f = ERTModelling(maxIter=200000, **kw)
    f.setData(data)
    f.setMesh(mesh, ignoreRegionManager=True)
    return f


@pytest.mark.parametrize("refine", ["createH2", "createP2"])
@pytest.mark.parametrize("form,small,bar", [
    (dict(), True, 120), (dict(precision="mixed"), True, 120), (dict(precision="mixed", precond="fsai"), True, 120),
    (dict(precision="mixed", precond="fsai"), False, 150)])
def test_refined(torch, refine, form, small, bar):
    e = np.array([(x, y) for x in np.arange(4) * 4.0 for y in np.arange(3) * 4.0])
    coarse = create_box_mesh_3d(e, h=4.0, **(dict(para_depth=10.0, outer=80.0) if small else {}))
    mesh = getattr(coarse, refine)()
    data = DataContainerERT(np.column_stack([e, np.zeros(len(e))]), grid_line_scheme((4, 3), "pd"))
    data.set("k", geometricFactors(data, 3))
    rho = np.exp(np.random.default_rng(1).normal(np.log(100.0), 1.0, coarse.cellCount()))
    fast, exact = operator(mesh, data, **form), operator(mesh, data, rtol=1e-12)
    exact.setCoarseLevels(False)
    r, r0 = fast.response(rho), exact.response(rho)
    u, u0 = fast.subPotentials(), exact.subPotentials()
    assert float(np.max(np.abs(u - u0).max(axis=2) / np.abs(u0).max(axis=2))) <= 1e-8
    assert float(np.max(np.abs(r - r0) / np.maximum(np.abs(r0), 1e-3))) <= 1e-5
    st = fast.stats()
    assert 0 < st["iterations"] <= bar and st["stalled_columns"] == 0, st
