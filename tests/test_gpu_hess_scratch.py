"""rijk_soscf_hess_ints when the scratch of its order for aa_J is refused: the pairs' J^{tu} and the half-transform of all
rows at once give way to the diagonals (pp|Q) in batches of 96 rows, which take the least.  Against a call that met no
shortage to the rounding of sums in another order, 1e-10 of the largest element as in test_gpu_hess_routes.py."""
import numpy as np
import pytest

from nopt_b200 import rijk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,naux,na,n_mo,pairs", [(300, 400, 18, 299, True), (140, 130, 26, 130, False)])
def test_refused_scratch_takes_the_other_order(n, naux, na, n_mo, pairs):
    npad, t = -(-n // 64) * 64, na * (na + 1) // 2
    te, nd = npad * (npad + 64) // 2, t if pairs else naux
    assert pairs == (t * (naux + 2 * n_mo) < 2 * n_mo * naux and t * te <= 96 * npad * naux)
    assert npad * nd * n_mo <= 2 ** 25  # all rows at once
    rng = np.random.default_rng(n)
    I3 = rng.normal(size=(n * (n + 1) // 2, naux))
    MO = np.linalg.qr(rng.normal(size=(n, n)))[0][:n_mo].copy()
    met = []
    with rijk.FockBuilder(0) as fb:
        fb.set_metric(np.eye(naux), rijk.METRIC_CHOLESKY)
        fb.set_3c(I3, n)
        want = fb.soscf_hess_ints(MO, 3, na)
        for k in range(30):
            fb.selftest_alloc_refuse(k, 2)
            try:
                got = fb.soscf_hess_ints(MO, 3, na)
                for a, b in zip(got, want):
                    assert np.max(np.abs(a - b)) <= 1e-10 * np.max(np.abs(b))
                met.append("same" if np.array_equal(got[0], want[0]) else "other order")
            except rijk.RijkError as e:
                assert e.code == rijk.ERR_ALLOC
                met.append("refused")
            finally:
                fb.selftest_alloc_refuse(0, 0)
    first = len(met) - met[::-1].index("refused")  # after the buffers that both orders need
    # the packed pairs, J^{tu}, the diagonals and the half-transform; or the last two
    assert met[first:first + (4 if pairs else 2)] == (["other order"] * 4 if pairs else ["same"] * 2)
    assert set(met[first + 4:]) == {"same"}
