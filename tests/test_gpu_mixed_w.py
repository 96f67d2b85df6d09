"""The mixed Coulomb pair where its w kernel changes form: one aux function a warp, and from four CTAs an SM on two,
with an odd number of aux functions and a last chunk of one tile.  The metric is the identity, so the fitted tensor
is the random input; numpy forms J in double precision from the same split-BF16 values and the density rounded to
FP32.  What remains is the kernel's FP32 sum of eight products, at most 8 x 2^-24 of the sum of their magnitudes
per aux function; the bound carries that through J, doubled, plus 1e-12."""
import numpy as np
import pytest

from nopt_b200 import rijk

pytestmark = pytest.mark.gpu


def _bf16(x):
    u = x.astype(np.float32).view(np.uint32)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32)


@pytest.mark.parametrize("n,naux", [(1, 1), (72, 71), (300, 1181)])
def test_mixed_j_from_split_values(n, naux):
    rng = np.random.default_rng(naux)
    rows, cols = np.tril_indices(n)
    I3 = rng.normal(size=(len(rows), naux))
    nocc = min(2, n)
    MO = np.linalg.qr(rng.normal(size=(n, n)))[0][:nocc].copy()
    D = MO.T @ MO
    with rijk.FockBuilder(0) as fb:
        fb.set_metric(np.eye(naux), rijk.METRIC_CHOLESKY)
        fb.set_3c(I3, n)
        J, _ = fb.dm_to_f_transform_ri(D, MO, nocc, rijk.PREC_MIXED)
    hi = _bf16(I3).astype(np.float64)
    B = hi + _bf16(I3 - hi)
    d = np.where(rows == cols, D[rows, cols], D[rows, cols] + D[cols, rows]).astype(np.float32).astype(np.float64)
    w = d @ B
    Jp = B @ w
    scale = J[rows, cols] @ Jp / (Jp @ Jp)  # the ABI's prefactor of the density
    assert abs(scale - round(scale)) <= 1e-5
    bound = 2 * 8 * 2.0 ** -24 * (np.abs(B) @ (np.abs(d) @ np.abs(B))) + 1e-12
    assert np.all(np.abs(J[rows, cols] - round(scale) * Jp) <= abs(round(scale)) * bound)
    assert np.array_equal(J, J.T)
