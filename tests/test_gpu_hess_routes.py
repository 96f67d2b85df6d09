"""rijk_soscf_hess_ints on both sides of its rule for aa_J (the pairs' J^{tu} first, or the diagonals (pp|Q) first),
with the half-transforms in one piece and in batches of 96 rows, and rijk_mo_ints at ragged active counts.  The
metric is the identity, so the fitted tensor is the random input itself.  Sums of n^2 and then n_aux products of
elements of size one, in another order than numpy's: (n + n_aux) eps = 3e-13 relative to sums of magnitudes that
exceed the results by at most a factor of n = 300 before cancellation, 1e-10 of the largest element."""
import numpy as np
import pytest

from nopt_b200 import rijk

pytestmark = pytest.mark.gpu

CASES = {
    "pairs": (70, 60, 5, 70), "pairs_one_active": (65, 40, 1, 61), "diagonals": (70, 40, 20, 67),
    "diagonals_batched": (300, 400, 26, 299), "pairs_batched": (300, 900, 26, 300),
}


def _pairs_first(n, naux, na, n_mo):
    npad = -(-n // 64) * 64
    te, t = npad * (npad + 64) // 2, na * (na + 1) // 2
    return t * (naux + 2 * n_mo) < 2 * n_mo * naux and t * te <= 96 * npad * naux


@pytest.mark.parametrize("name", list(CASES))
def test_hess_ints_by_either_order(name):
    n, naux, na, n_mo = CASES[name]
    assert _pairs_first(n, naux, na, n_mo) == name.startswith("pairs")
    rng = np.random.default_rng(n + naux)
    rows, cols = np.tril_indices(n)
    I3 = rng.normal(size=(len(rows), naux))
    MO = np.linalg.qr(rng.normal(size=(n, n)))[0][:n_mo].copy()
    n_c = 3
    with rijk.FockBuilder(0) as fb:
        fb.set_metric(np.eye(naux), rijk.METRIC_CHOLESKY)
        fb.set_3c(I3, n)
        gJ, gK = fb.soscf_hess_ints(MO, n_c, na)
        A = MO[n_c:n_c + na]
        gA, _, _ = fb.calc_2el_mo_ints_ri(None, MO, A, A, n_c, na, want_jk=False)
    X = np.empty((naux, n_mo, na))
    D = np.empty((naux, n_mo))
    for q in range(naux):
        B = np.zeros((n, n))
        B[rows, cols] = I3[:, q]
        B[cols, rows] = I3[:, q]
        half = MO @ B
        X[q] = half @ A.T
        D[q] = np.einsum("pm,pm->p", half, MO)
    Y = X[:, n_c:n_c + na].reshape(naux, na * na)
    J, K = D.T @ Y, np.einsum("qpt,qpu->ptu", X, X, optimize=True)
    for got, want in ((gJ, J), (gK, K), (gA, Y.T @ Y)):
        assert np.max(np.abs(got.reshape(want.shape) - want)) <= 1e-10 * np.max(np.abs(want))
