"""Model update on an FP32 Jacobian whose rows are not 16-byte aligned: every
value widens to FP64 exactly and the sums keep the order of the FP64 form, so
the update equals the one on the same values stored in FP64, bit for bit."""
import numpy as np
import pytest


def _chain(P):
    """First differences of neighbouring parameters as CSR."""
    rows = max(P - 1, 0)
    rp = np.arange(0, 2 * rows + 1, 2, dtype=np.int64)
    ci = np.stack([np.arange(rows), np.arange(1, rows + 1)], 1).ravel().astype(np.int32)
    return rp, ci, np.tile([1.0, -1.0], rows), P


@pytest.mark.gpu
@pytest.mark.parametrize("D,P", [(1, 5), (2, 1), (3, 255), (17, 1025), (129, 1023), (40, 4099), (33, 2050)])
def test_update_of_an_fp32_jacobian_equals_the_fp64_form(D, P):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from pygimli_gb300.inversion import cgls

    rng = np.random.default_rng(100 * D + P)
    J = (rng.standard_normal((D, P)) * 10.0 ** rng.integers(-6, 3, (D, P))).astype(np.float32)
    flat = J.ravel()
    for k, v in enumerate([0.0, -0.0, 1e-42, -3e-45, 1.1754944e-38, -1.1754942e-38, 3.0e38]):
        if len(flat) > 20 * (k + 1):
            flat[7 * k + 3] = v
    C = _chain(P)
    nc = len(C[0]) - 1
    args = (C, rng.uniform(1, 2, D), rng.standard_normal(D), np.zeros(P), np.ones(nc), np.ones(P),
            rng.uniform(1, 2, P), rng.uniform(1, 2, D), 20.0, np.zeros(nc))
    x32, it32 = cgls(torch.as_tensor(J, device="cuda"), *args, max_iter=4, tol=0.0)
    x64, it64 = cgls(torch.as_tensor(J.astype(np.float64), device="cuda"), *args, max_iter=4, tol=0.0)
    assert P % 4 and it32 == it64
    assert np.isfinite(x64).all()
    np.testing.assert_array_equal(x32.view(np.int64), x64.view(np.int64))
