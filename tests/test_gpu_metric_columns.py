"""The metric contraction's columns at the edges of the 64 x 64 tiles: one orbital, a full tile, one past it, a
ragged last tile row, in both layouts and for both metric forms.  The two layouts reach the same stored elements
by different column counts (packed pairs, mirrored into the diagonal tiles; all rows of the square), from sums over
P in the same order, so J and K agree bit for bit; against numpy, which inverts V (condition below 10)
where the build factorises it, sums of at most n n_aux = 14,000 terms in double precision agree to
n n_aux eps = 3e-12 of the sum of magnitudes: 1e-11 of the largest element."""
import numpy as np
import pytest

from nopt_b200 import rijk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [rijk.METRIC_INVSQRT, rijk.METRIC_CHOLESKY])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 129, 200])
def test_columns_cover_the_stored_tiles(n, form):
    naux, nocc = 70, max(1, n // 5)
    rng = np.random.default_rng(n)
    A = rng.normal(size=(naux, naux))
    V = A @ A.T / naux + np.eye(naux)
    full = rng.normal(size=(n, n, naux))
    full = full + full.transpose(1, 0, 2)
    packed = np.ascontiguousarray(full[np.tril_indices(n)])
    MO = np.linalg.qr(rng.normal(size=(n, n)))[0].T.copy()
    D = MO[:nocc].T @ MO[:nocc]
    got = []
    for I3, layout in ((packed, rijk.LAYOUT_PACKED), (full.reshape(n * n, naux), rijk.LAYOUT_NOPT_FULL)):
        with rijk.FockBuilder(0) as fb:
            fb.set_metric(V, form)
            fb.set_3c(np.ascontiguousarray(I3), n, layout)
            got.append(fb.dm_to_f_transform_ri(D, MO, nocc))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    W = np.linalg.inv(V)
    J = np.einsum("mnp,p->mn", full, W @ np.einsum("mnp,mn->p", full, D))
    X = np.einsum("mnp,in->imp", full, MO[:nocc])
    K = np.einsum("imp,pq,inq->mn", X, W, X, optimize=True)
    J2, K2 = got[0]
    for have, want in ((J2, J), (K2, K)):
        scale = np.vdot(want, have) / np.vdot(want, want)  # the ABI's prefactor of the density
        assert abs(scale - round(scale)) <= 1e-10
        assert np.max(np.abs(have - round(scale) * want)) <= 1e-11 * np.max(np.abs(have))
