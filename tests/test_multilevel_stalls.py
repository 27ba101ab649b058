"""Ground on which the FP32 phase of the mixed solver rests or stalls with
coarse levels: a stalled model leaves no trace on the next one, very rough
ground converges in FP32, and the FP64 finish of columns that FP32 cannot solve
has the coarse levels too.

Iteration bars: the single level needs 384 to 1730 FP32 iterations on the rough
ground and 660 to 880 FP64 iterations in the finish; the coarse levels were
measured at 160 to 560 and 50 to 150."""
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


@pytest.fixture(scope="module")
def grid():
    e = np.array([(x, y) for x in np.arange(12) * 4.0 for y in np.arange(8) * 4.0])
    mesh = create_box_mesh_3d(e, h=4.0)
    data = DataContainerERT(np.column_stack([e, np.zeros(len(e))]), grid_line_scheme((12, 8), "pd"))
    data.set("k", geometricFactors(data, 3))
    return mesh, data


def operator(grid, **kw):
    from pygimli_gb300 import ERTModelling
    f = ERTModelling(maxIter=200000, precision="mixed", **kw)
    f.setData(grid[1])
    f.setMesh(grid[0], ignoreRegionManager=True)
    return f


def lognormal(mesh, sigma, seed):
    return np.exp(np.random.default_rng(seed).normal(np.log(100.0), sigma, mesh.cellCount()))


def bodies(mesh, factor):
    c, rho = mesh.cellCenters(), lognormal(mesh, 1.0, 1)
    rho[np.linalg.norm(c - [12.0, 8.0, -4.0], axis=1) < 4.0] = 100.0 / factor
    rho[np.linalg.norm(c - [28.0, 16.0, -5.0], axis=1) < 4.0] = 100.0 * factor
    return rho


@pytest.mark.parametrize("precond", ["jacobi", "fsai"])
def test_stall_is_not_carried_over(torch, grid, precond):
    ordinary = lognormal(grid[0], 1.0, 9)
    f = operator(grid, precond=precond)
    first, its = f.response(ordinary), f.stats()["iterations"]
    for _ in range(2):
        f.response(bodies(grid[0], 1e9))
        assert f.stats()["stalled_columns"] >= 48  # half of the sources and more
        again, st = f.response(ordinary), f.stats()
        assert st["stalled_columns"] == 0 and st["iterations"] == its
        assert np.array_equal(first, again)


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_rough_ground_converges_in_fp32(torch, grid, seed):
    f = operator(grid, precond="fsai")
    f.response(lognormal(grid[0], 5.0, seed))
    st = f.stats()
    assert st["stalled_columns"] == 0 and st["iterations"] <= 900 and st["max_rel_residual"] <= 1e-10, st


@pytest.mark.parametrize("precond", ["jacobi", "fsai"])
def test_finish_has_coarse_levels(torch, grid, precond):
    f = operator(grid, precond=precond)
    f.response(bodies(grid[0], 1e9))
    st = f.stats()
    assert st["stalled_columns"] >= 48 and st["iterations"] <= 400 and st["max_rel_residual"] <= 1e-10, st


@pytest.mark.parametrize("ground", ["rough", "bodies"])
def test_complex_finish_has_coarse_levels(torch, ground):
    """Complex columns that stall in FP32; the single level needs 11000 and 950
    iterations on these models."""
    e = np.array([(x, y) for x in np.arange(9) * 4.0 for y in np.arange(7) * 4.0])
    mesh = create_box_mesh_3d(e, h=4.0)
    data = DataContainerERT(np.column_stack([e, np.zeros(len(e))]), grid_line_scheme((9, 7), "pd"))
    data.set("k", geometricFactors(data, 3))
    f = operator((mesh, data))
    f.setComplex(True)
    rho = lognormal(mesh, 5.0, 505) if ground == "rough" else bodies(mesh, 1e8)
    ph = -0.03 * np.random.default_rng(1).uniform(0.2, 1.0, len(rho))
    f.response(np.concatenate([rho * np.cos(ph), rho * np.sin(ph)]))
    st = f.stats()
    assert st["stalled_columns"] > 0 and st["max_rel_residual"] <= 1e-10
    assert st["iterations"] <= (3000 if ground == "rough" else 500), st
