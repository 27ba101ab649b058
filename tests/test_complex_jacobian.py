"""The staged complex Jacobian (one cell per parameter) against the general
kernel on the same potentials: the general one runs when two cells share a
parameter, which leaves every other column's sum unchanged.  Electrode counts
for each tile width, a ragged last tile, poles, an empty parameter, quadratic
cells.

Tolerance: both sum the same FP64 products of potentials in another order; each
term cancels by at most the ratio of a cell's potential differences to its
potentials (about 1e5 far from a dipole), so 1e-9 of the Jacobian's norm leaves
two digits."""
import numpy as np
import pytest

from pygimli_gb300 import DataContainerERT, Mesh, create_box_mesh_3d

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    from pygimli_gb300 import build
    build.build()
    return t


@pytest.mark.parametrize("nx,ny,p2", [(4, 3, False), (10, 6, False), (13, 10, False), (4, 3, True)])
def test_against_general_kernel(torch, nx, ny, p2):
    from pygimli_gb300 import ERTModelling
    e = np.array([(x, y) for x in np.arange(nx) * 4.0 for y in np.arange(ny) * 4.0])
    mesh = create_box_mesh_3d(e, h=4.0, para_margin=(1, 1), para_depth=4.0, outer=60.0, growth=2.0, depth_growth=1.6)
    if p2:
        mesh = mesh.createP2()
    rng = np.random.default_rng(nx)
    ab = np.array([rng.permutation(len(e))[:4] for _ in range(37)], np.int32)
    ab[::5, 1] = -1
    ab[1::7, 3] = -1
    data = DataContainerERT(np.column_stack([e, np.zeros(len(e))]), ab)
    data.set("k", rng.uniform(1.0, 9.0, data.size()))
    C = mesh.cellCount()
    z = np.exp(rng.normal(np.log(100.0), 1.0, C)) * np.exp(-1j * rng.uniform(0.0, 0.1, C))
    z[1] = z[0]

    def jac(markers):
        m = Mesh(3, mesh.nodes, mesh.cells, markers, mesh.node_markers, mesh.boundaries, mesh.boundary_markers,
                 mesh.boundary_cells)
        f = ERTModelling(precision="mixed")
        f.setData(data)
        f.setMesh(m, ignoreRegionManager=True)
        f.setComplex(True)
        f.response(z)
        return f.createJacobian(z)

    own = np.arange(C, dtype=np.int32)
    shared = own.copy()
    shared[1] = 0  # parameter 1 is empty
    J, J2 = jac(own), jac(shared)
    assert float(torch.abs(J2[:, 1]).max()) == 0.0
    assert float(torch.linalg.vector_norm(J[:, 2:] - J2[:, 2:]) / torch.linalg.vector_norm(J2[:, 2:])) <= 1e-9
    both = J[:, 0] + J[:, 1]
    assert float(torch.linalg.vector_norm(both - J2[:, 0]) / torch.linalg.vector_norm(J2[:, 0])) <= 1e-9
    hole = own.copy()
    hole[5] = -1  # one parameter without a cell, one cell per other parameter
    J3 = jac(hole)
    assert float(torch.abs(J3[:, 5]).max()) == 0.0
