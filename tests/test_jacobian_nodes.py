"""The FP32 Jacobian of 3-D P1 cells with its dipole tables built node by node
(tiles of consecutive cells, few distinct nodes) against the general table
build, which runs on the same cells when their parameter numbers are scattered
(more than 32 distinct nodes per tile).  The potentials are the same, and the
two builds do the same operations in the same order: equal to the last bit,
also for parameters without a cell whose model value has no finite inverse
square in FP32."""
import ctypes

import numpy as np
import pytest

from pygimli_gb300 import DataContainerERT, Mesh, create_box_mesh_3d
from pygimli_gb300.data import geometricFactors, grid_line_scheme

pytestmark = pytest.mark.gpu
JACOBIAN32 = 4  # ERTGB_KERNEL_JACOBIAN32


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    from pygimli_gb300 import build
    build.build()
    return t


def box(nx, ny, h=4.0):
    e = np.array([(x, y) for x in np.arange(nx) * 4.0 for y in np.arange(ny) * 4.0])
    mesh = create_box_mesh_3d(e, h=h, para_depth=10.0, outer=120.0, growth=1.5)
    data = DataContainerERT(np.column_stack([e, np.zeros(len(e))]), grid_line_scheme((nx, ny), "pd"))
    data.set("k", geometricFactors(data, 3))
    return mesh, data


def operator(mesh, data, markers):
    from pygimli_gb300 import ERTModelling
    m = Mesh(3, mesh.nodes, mesh.cells, markers.astype(np.int32), mesh.node_markers, mesh.boundaries,
             mesh.boundary_markers, mesh.boundary_cells)
    f = ERTModelling(precision="mixed")
    f.setData(data)
    f.setMesh(m, ignoreRegionManager=True)
    return f


def most_nodes(mesh, markers):
    order = np.full(markers.max() + 1, -1)
    order[markers] = np.arange(mesh.cellCount())
    tiles = [order[t:t + 32] for t in range(0, len(order), 32)]
    return max(len(np.unique(mesh.cells[t[t >= 0]])) for t in tiles)


@pytest.mark.parametrize("absent", [0.0, np.nan, 1e-25, 100.0])
@pytest.mark.parametrize("empty", [1, 2, 3])  # row lengths of every store width
def test_builds_agree(torch, empty, absent):
    mesh, data = box(5, 3)
    C = mesh.cellCount()
    P = C + empty
    near = np.arange(C)
    for p in range(empty):
        near[near >= 40 + 7 * p] += 1  # parameters 40, 47, 54 hold no cell
    far = (near * 7919) % P
    assert np.gcd(7919, P) == 1 and most_nodes(mesh, near) <= 32 < most_nodes(mesh, far)
    rng = np.random.default_rng(empty)
    rho = np.exp(rng.normal(np.log(100.0), 1.0, C))
    rho_d = torch.from_numpy(rho).cuda()
    out = []
    for mk in (near, far):
        f = operator(mesh, data, mk)
        model = np.full(P, absent)
        model[mk] = rho
        f.response(rho_d)
        J = f.createJacobian(model, dtype="float32")
        without = torch.ones(P, dtype=torch.bool, device="cuda")
        without[torch.from_numpy(mk).cuda()] = False
        assert int(without.sum()) == empty and bool((J[:, without] == 0).all())
        out.append(J[:, torch.from_numpy(mk).cuda()])
    assert bool(torch.isfinite(out[0]).all()) and torch.equal(out[0], out[1])


@pytest.mark.parametrize("grid", [(20, 21), (29, 30), (30, 30)])
def test_many_electrodes(torch, grid):
    """The stiffness kernel's plan where the node-wise build leaves most of the
    table space, about half of what the general one leaves (that one is taken)
    and none.  The plan shows in the operation count of the kernel's profile."""
    e = np.array([(x, y) for x in np.arange(grid[0]) * 4.0 for y in np.arange(grid[1]) * 4.0])
    mesh = create_box_mesh_3d(e, h=4.0, para_depth=8.0, outer=120.0, growth=2.0)
    nE, D, C = len(e), 300, mesh.cellCount()
    assert most_nodes(mesh, np.arange(C)) <= 32
    rng = np.random.default_rng(nE)
    ab = np.array([rng.permutation(nE)[:4] for _ in range(D)], np.int32)
    data = DataContainerERT(np.column_stack([e, np.zeros(nE)]), ab)
    data.set("k", rng.uniform(1.0, 9.0, D))
    f = operator(mesh, data, np.arange(C))
    rho = np.exp(rng.normal(np.log(100.0), 0.5, C))
    f.response(rho)
    J, F = f.createJacobian(rho, dtype="float64"), f.createJacobian(rho, dtype="float32")
    assert float(torch.linalg.vector_norm(F.double() - J) / torch.linalg.vector_norm(J)) <= 2e-6
    ms, nbytes, flops = ctypes.c_double(), ctypes.c_double(), ctypes.c_double()
    f._check(f._lib.ertgb_profile_kernel(f._ctx, JACOBIAN32, 1, ctypes.c_void_p(F.data_ptr()), ctypes.byref(ms),
                                         ctypes.byref(nbytes), ctypes.byref(flops)))
    nA, nM = len(np.unique(ab[:, :2], axis=0)), len(np.unique(ab[:, 2:], axis=0))
    assert flops.value == C * ((nE + 1) * 3 + (nA + nM) * 9.0 + nA * 18.0) + D * C * 8.0
