"""Rounding of the wavenumber-outermost Jacobian kernel in FP32 and the rule
that leaves one-wavenumber schemes to the tile kernel.

Both kernels form the same FP32 table entries and round one sum per staged
wavenumbers (here) or per wavenumber (there), so their errors against the FP64
Jacobian are equal on average; one realisation differs by up to 1.4 times either
way, the geometric mean over twelve by a tenth of that's logarithm.  The bar is
1.1.  Adding every product to the running sum would give 1.15 to 1.3."""
import math

import numpy as np
import pytest

from pygimli_gb300 import DataContainerERT, Mesh, createData, create_box_mesh_3d, create_para_mesh_2d
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


def jacobians(mesh, data, markers, rho, **kw):
    from pygimli_gb300 import ERTModelling
    f = ERTModelling(**kw)
    f.setData(data)
    f.setMesh(Mesh(mesh.dim(), mesh.nodes, mesh.cells, markers, mesh.node_markers, mesh.boundaries,
                   mesh.boundary_markers, mesh.boundary_cells), ignoreRegionManager=True)
    f.response(rho[markers])
    return f.createJacobian(rho, dtype="float64"), f.createJacobian(rho, dtype="float32").double()


def test_error_not_larger(torch):
    logs = []
    for ne, dx in ((8, 0.25), (16, 0.5)):
        for scheme in ("wa", "dd", "pd"):
            xs = np.arange(float(ne))
            mesh = create_para_mesh_2d(xs, para_dx=dx, para_depth=max(2.0, ne / 4.0)).createH2()
            data = createData(xs, scheme, maxSeparation=12)
            data.set("k", geometricFactors(data, 2))
            small = np.asarray(mesh.cell_markers)
            big = small.copy()
            big[np.isin(small, np.arange(10, 20))] = 10  # forty cells: the tile kernel for all
            for seed in (1, 2):
                rho = np.exp(np.random.default_rng(seed).normal(np.log(100.0), 1.0, small.max() + 1))
                rho[10:20] = rho[10]
                keep = torch.ones(len(rho), dtype=torch.bool, device="cuda")
                keep[10:20] = False
                e = []
                for mk in (small, big):
                    J, F = jacobians(mesh, data, mk, rho, precond="band")
                    e.append(float(torch.linalg.vector_norm((F - J)[:, keep]) / torch.linalg.vector_norm(J[:, keep])))
                assert max(e) <= 2e-6
                logs.append(math.log(e[0] / e[1]))
    assert math.exp(sum(logs) / len(logs)) <= 1.1, [round(math.exp(v), 2) for v in logs]


@pytest.mark.parametrize("per", [2, 3, 4])
@pytest.mark.parametrize("n", [24, 25, 33, 34, 49, 50, 66, 67, 99, 100])  # n * per about 100 and 200
def test_one_wavenumber(torch, per, n):
    e = np.array([(x, y) for x in np.arange(6) * 4.0 for y in np.arange(4) * 4.0])
    mesh = create_box_mesh_3d(e, h=4.0, para_margin=(1, 1), para_depth=4.0, outer=60.0, growth=2.0, depth_growth=1.6)
    rng = np.random.default_rng(n)
    ab = np.array([rng.permutation(24)[:4] for _ in range(n)], np.int32)
    data = DataContainerERT(np.column_stack([e, np.zeros(24)]), ab)
    data.set("k", rng.uniform(1.0, 9.0, n))
    C = mesh.cellCount()
    small = (np.arange(C) // per).astype(np.int32)
    big = small.copy()
    big[small < 10] = 0  # more than eight cells: the tile kernel
    rho = np.exp(rng.normal(np.log(100.0), 1.0, small.max() + 1))
    rho[:10] = rho[0]
    (J, F), (G, H) = (jacobians(mesh, data, mk, rho, precision="mixed", precond="fsai") for mk in (small, big))
    for a, b, tol in ((J, G, 1e-10), (F, H, 2e-6)):  # as in the comparison of the kernels over all forms
        assert float(torch.linalg.vector_norm((a - b)[:, 10:]) / torch.linalg.vector_norm(b[:, 10:])) <= tol
