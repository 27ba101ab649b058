"""Device memory running out in a solver with extra workspaces: the call goes on
without them and the next one with free memory has them again.  The shortage is
an accounting limit of the calling thread (no allocation is made to fail on the
device).

Tolerance: two solver forms at the default rtol 1e-10, whose potentials are
within 1e-8 of the column maximum of each other (100 times the accuracy of
either); the direct solves within 1e-9."""
import ctypes
import gc

import numpy as np
import pytest

from pygimli_gb300 import DataContainerERT, createData, create_box_mesh_3d, create_para_mesh_2d
from pygimli_gb300.batch import BatchedERTModelling
from pygimli_gb300.data import geometricFactors, grid_line_scheme

pytestmark = pytest.mark.gpu
FORMS = [dict(), dict(precision="mixed"), dict(precision="mixed", precond="fsai"), dict(precond="band"),
         dict(precision="mixed", cplx=True)]


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    from pygimli_gb300 import build
    build.build()
    return t


@pytest.fixture()
def limit(torch):
    from pygimli_gb300 import _native
    lib = _native.load()

    def set_limit(nbytes):
        used = ctypes.c_int64()
        lib.ertgb_alloc_limit(nbytes, ctypes.byref(used))
        return used.value

    yield set_limit
    set_limit(-1)


def operator(form):
    from pygimli_gb300 import ERTModelling
    kw = dict(form)
    cplx = kw.pop("cplx", False)
    if kw.get("precond") == "band":
        xs = np.arange(24.0)
        mesh = create_para_mesh_2d(xs, para_dx=0.5, para_depth=6.0)
        data = createData(xs, "dd", maxSeparation=6)
    else:
        e = np.array([(x, y) for x in np.arange(5) * 4.0 for y in np.arange(3) * 4.0])
        mesh = create_box_mesh_3d(e, h=2.0, para_depth=10.0, outer=120.0, growth=1.5)
        data = DataContainerERT(np.column_stack([e, np.zeros(len(e))]), grid_line_scheme((5, 3), "pd"))
    data.set("k", geometricFactors(data, mesh.dim()))
    f = ERTModelling(maxIter=200000, **kw)
    f.setData(data)
    f.setMesh(mesh, ignoreRegionManager=True)
    rho = np.exp(np.random.default_rng(1).normal(np.log(100.0), 1.0, mesh.cellCount()))
    if cplx:
        f.setComplex(True)
        rho = np.concatenate([rho, -0.02 * rho])
    return f, rho


def potentials(f, r, cplx):
    return r if cplx else f.subPotentials()


@pytest.mark.parametrize("form", FORMS)
def test_response(torch, limit, form):
    cplx = "cplx" in form
    gc.collect()
    f, rho = operator(form)
    before = limit(-1)
    full = f.response(rho)
    u, st = potentials(f, full, cplx), f.stats()
    need = limit(-1) - before
    del f
    gc.collect()
    f, rho = operator(form)
    before = limit(need - 1)  # the last allocation of the full form does not fit
    for _ in range(2):
        r = f.response(rho)
        v = potentials(f, r, cplx)
        assert limit(0) - before <= need - 1
        limit(before + need - 1 - limit(0))
        assert float(np.max(np.abs(u - v).max(axis=-1) / np.abs(u).max(axis=-1))) <= 1e-8
        if "precond" not in form or form["precond"] != "band":
            assert f.stats()["iterations"] > 2 * st["iterations"]
    limit(-1)
    assert np.array_equal(f.response(rho), full) and f.stats()["iterations"] == st["iterations"]
    limit(need // 4)  # what nothing can be done with stays an error
    with pytest.raises(Exception, match="limit on device memory"):
        f2, _ = operator(form)
        f2.response(rho)


@pytest.mark.parametrize("form", FORMS[:4])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_jacobian(torch, limit, monkeypatch, form, dtype):
    f, rho = operator(form)
    f.response(rho)
    J = f.createJacobian(rho, dtype=dtype)
    f, rho = operator(form)
    f.response(rho)
    held = limit(0)  # the library's scales (and split potentials) do not fit beside the solver's workspaces
    assert torch.equal(f.createJacobian(rho, dtype=dtype), J)
    assert limit(-1) < held
    f.response(rho)
    held, empty, calls = limit(-1), torch.empty, []

    def full(*a, **kw):  # the Jacobian itself does not fit at first
        if isinstance(a[0], tuple) and len(a[0]) == 2 and not calls:
            calls.append(a)
            raise torch.cuda.OutOfMemoryError("out of memory")
        return empty(*a, **kw)

    monkeypatch.setattr(torch, "empty", full)
    assert torch.equal(f.createJacobian(rho, dtype=dtype), J) and calls
    assert limit(-1) < held


def test_batch(torch, limit):
    """The batch's wider right-hand sides do not fit beside what the operators
    kept from single responses."""
    fs, rhos = zip(*(operator(dict(precond="band")) for _ in range(2)))
    ref = [f.response(r) for f, r in zip(fs, rhos)]
    b = BatchedERTModelling(list(fs))
    limit(0)
    try:
        out = b.response(list(rhos))
    except Exception as e:  # even so it may not fit: the same error as ever, and the operators stay usable
        assert "limit on device memory" in str(e)
        limit(-1)
        out = b.response(list(rhos))
    limit(-1)
    for a, r in zip(out, ref):
        assert float(np.max(np.abs(a - r) / r)) <= 1e-8
