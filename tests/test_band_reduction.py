"""The block cyclic reduction of the banded direct solve against the oracle's
SuperLU factors: block counts of one, two and odd numbers, a ragged last
block, bandwidths below the smallest block and beyond the widest one (the
serial band Cholesky), more sources than one column tile holds.

Tolerance: both solve the same FP64 systems directly; the smallest-wavenumber
matrices of these meshes have condition numbers up to ~1e6, so potentials agree
to 1e-9 of the column maximum with three digits to spare, and the responses,
rounded to 1e-10 V, likewise."""
import numpy as np
import pytest

from oracle import ert_oracle as O
from pygimli_gb300 import Mesh, createData, create_para_mesh_2d
from pygimli_gb300.data import geometricFactors
from pygimli_gb300.kwave import init_kwave_list

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    from pygimli_gb300 import build
    build.build()
    return t


def strip(nx, ny):
    """nx x ny structured strip of triangles, the shorter side numbered first
    (bandwidth ~ ny + 1), Neumann surface, mixed sides and bottom."""
    xs, ys = np.arange(float(nx)), -np.arange(float(ny))
    nodes = np.array([(x, y, 0.0) for x in xs for y in ys])
    idx = np.arange(nx * ny).reshape(nx, ny)
    a, b, c, d = idx[:-1, :-1].ravel(), idx[1:, :-1].ravel(), idx[1:, 1:].ravel(), idx[:-1, 1:].ravel()
    cells = np.vstack([np.column_stack([a, d, b]), np.column_stack([b, d, c])]).astype(np.int32)
    top = np.column_stack([idx[:-1, 0], idx[1:, 0]])
    rest = np.vstack([np.column_stack([idx[:-1, -1], idx[1:, -1]]), np.column_stack([idx[0, :-1], idx[0, 1:]]),
                      np.column_stack([idx[-1, :-1], idx[-1, 1:]])])
    bnd = np.vstack([top, rest]).astype(np.int32)
    marks = np.r_[np.full(len(top), -1), np.full(len(rest), -2)].astype(np.int32)
    nm = np.zeros(len(nodes), np.int32)
    return Mesh(2, nodes, cells, np.arange(len(cells), dtype=np.int32), nm, bnd, marks), idx[:, 0]


def check(mesh, data, seed):
    from pygimli_gb300 import ERTModelling
    rho = np.exp(np.random.default_rng(seed).normal(np.log(100.0), 1.0, mesh.cellCount()))
    k, w = init_kwave_list(2, data.sensorPositions())
    P = O.Problem(mesh, data.sensorPositions(), data.abmn(), data["k"], k, w)
    ro, uo = P.response(rho)
    fop = ERTModelling(precond="band")
    fop.setData(data)
    fop.setMesh(mesh, ignoreRegionManager=True)
    for _ in range(2):  # the second pass finds the factor's buffers in use
        r = fop.response(rho)
        u = fop.subPotentials()
        e_u = float(np.max(np.abs(u - uo).max(axis=2) / np.abs(uo).max(axis=2)))
        e_r = float(np.max(np.abs(r - ro) / ro))
        assert e_u <= 1e-9 and e_r <= 1e-8, (e_u, e_r)


@pytest.mark.parametrize("nx,ny,ne", [
    (9, 3, 5),      # bandwidth below the smallest block
    (16, 4, 8),     # an even number of full blocks
    (21, 7, 6),     # odd block count, ragged last block
    (40, 6, 37),    # more sources than one narrow tile
    (70, 17, 60),   # two column tiles
    (12, 11, 6),    # few blocks
    (120, 63, 12),  # wide blocks
    (130, 111, 9),  # the widest block
    (125, 118, 9),  # beyond it: the serial form
])
def test_strips(torch, nx, ny, ne):
    mesh, top = strip(nx, ny)
    at = top[(nx - ne) // 2:(nx - ne) // 2 + ne]
    mesh.node_markers[at] = -99
    data = createData(mesh.nodes[at, 0], "wa" if ne < 8 else "dd", maxSeparation=3)
    data.set("k", geometricFactors(data, 2))
    check(mesh, data, nx + ny)


def test_refined_and_quadratic(torch):
    """Bandwidths of the refined and the P2 forward mesh of a line."""
    xs = np.arange(10.0)
    mesh = create_para_mesh_2d(xs, para_dx=0.5, para_depth=3.0)
    data = createData(xs, "dd")
    data.set("k", geometricFactors(data, 2))
    check(mesh.createH2(), data, 1)
    check(mesh.createP2(), data, 2)
