"""The wavenumber-outermost Jacobian kernel against the general one on the same
potentials: the general one runs when a parameter has more than eight cells,
which leaves every other parameter's column as it was.  One and several cells
per parameter, an empty parameter, poles, one to several data chunks, tile
widths, linear and quadratic cells, 2.5-D and 3-D, FP64 and FP32.

Tolerance: FP64 sums of the same FP64 terms in another order, at most 1e5
cancellation in a term: 1e-10 of the column block's norm; FP32 products of
differences rounded from FP64: 2e-6."""
import numpy as np
import pytest

from pygimli_gb300 import DataContainerERT, Mesh, create_box_mesh_3d, create_para_mesh_2d, createData
from pygimli_gb300.data import geometricFactors

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    from pygimli_gb300 import build
    build.build()
    return t


def columns(torch, mesh, data, markers, rho, dtype, **kw):
    from pygimli_gb300 import ERTModelling
    m = Mesh(mesh.dim(), mesh.nodes, mesh.cells, markers, mesh.node_markers, mesh.boundaries, mesh.boundary_markers,
             mesh.boundary_cells)
    f = ERTModelling(**kw)
    f.setData(data)
    f.setMesh(m, ignoreRegionManager=True)
    f.response(rho[markers])
    return f.createJacobian(rho, dtype=dtype).double()


def check(torch, mesh, data, per, **kw):
    C = mesh.cellCount()
    P = C // per
    small = np.minimum(np.arange(C) // per, P - 1).astype(np.int32)  # per cells each (the last a few more)
    small[small == 3] = 2                                             # one double, one empty parameter
    small[small == P - 1] = P - 2 if per == 1 else P - 1
    cnt = np.bincount(small)
    assert cnt.max() <= 8
    big = small.copy()
    big[np.isin(small, np.arange(10, 20))] = 10                       # one with at least ten cells
    rng = np.random.default_rng(per)
    rho = np.exp(rng.normal(np.log(100.0), 1.0, small.max() + 1))
    rho[10:20] = rho[10]
    for dtype, tol in (("float64", 1e-10), ("float32", 2e-6)):
        J, G = (columns(torch, mesh, data, mk, rho, dtype, **kw) for mk in (small, big))
        keep = torch.ones(J.shape[1], dtype=torch.bool, device=J.device)
        keep[10:20] = False
        assert bool(torch.isfinite(J).all())
        e = float(torch.linalg.vector_norm((J - G)[:, keep]) / torch.linalg.vector_norm(G[:, keep]))
        assert e <= tol, (dtype, e)
        one = torch.linalg.vector_norm(J[:, 10:20].sum(dim=1) - G[:, 10]) / torch.linalg.vector_norm(G[:, 10])
        assert float(one) <= tol, (dtype, float(one))
        assert float(J[:, 3].abs().max()) == 0.0


@pytest.mark.parametrize("ne,dx,scheme,per", [
    (8, 0.5, "wa", 1),        # few data, all wavenumbers at once
    (21, 0.5, "dd", 3),       # several cells per parameter
    (41, 0.5, "pd", 4),       # poles, one chunk
    (60, 0.5, "pd+wa", 1),    # several data chunks
    (72, 0.5, "dd+wa", 2),    # narrow tiles, one or two wavenumbers at a time
])
def test_lines(torch, ne, dx, scheme, per):
    xs = np.arange(float(ne))
    mesh = create_para_mesh_2d(xs, para_dx=dx, para_depth=max(2.0, ne / 6.0))
    parts = [createData(xs, s) for s in scheme.split("+")]
    data = DataContainerERT(parts[0].sensorPositions(), np.vstack([p.abmn() for p in parts]))
    data.set("k", geometricFactors(data, 2))
    check(torch, mesh, data, per, precond="band")


def test_quadratic_line(torch):
    xs = np.arange(12.0)
    mesh = create_para_mesh_2d(xs, para_dx=0.5, para_depth=3.0).createP2()
    data = createData(xs, "dd")
    data.set("k", geometricFactors(data, 2))
    check(torch, mesh, data, 2, precond="band")


@pytest.mark.parametrize("p2", [False, True])
def test_box(torch, p2):
    e = np.array([(x, y) for x in np.arange(6) * 4.0 for y in np.arange(4) * 4.0])
    mesh = create_box_mesh_3d(e, h=4.0, para_margin=(1, 1), para_depth=4.0, outer=60.0, growth=2.0, depth_growth=1.6)
    if p2:
        mesh = mesh.createP2()
    rng = np.random.default_rng(2)
    ab = np.array([rng.permutation(24)[:4] for _ in range(300)], np.int32)
    data = DataContainerERT(np.column_stack([e, np.zeros(24)]), ab)
    data.set("k", rng.uniform(1.0, 9.0, 300))
    check(torch, mesh, data, 4, precision="mixed", precond="fsai")
