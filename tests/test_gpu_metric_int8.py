"""The metric contraction on the int8 tensor cores (taken from 2e9 FLOPs on): the fitted tensor itself, read back
as the MO tensor of unit orbitals, against M (P|mu nu) in numpy at the edges of the contraction's blocks: aux counts
off multiples of 32 and 64, aux ranges that start inside a 64-row block of M, both layouts, both metric forms.
The metrics are well conditioned, so V^-1/2 and L^-1 of two routines agree to a few 1e-15, and both sides sum n_aux
products in double precision or better: 1e-12 of the largest element leaves two decades."""
import numpy as np
import pytest

import rijk_oracle as O
from nopt_b200 import rijk

pytestmark = pytest.mark.gpu


def _system(n, naux):
    rng = np.random.default_rng(n + naux)
    A = rng.normal(size=(naux, naux))
    V = A @ A.T / naux + np.eye(naux)
    I3 = rng.normal(size=(n * (n + 1) // 2, naux)) * np.exp(rng.uniform(-8, 0, size=(n * (n + 1) // 2, 1)))
    return V, I3


def _fitted(fb, n):
    C = np.eye(n)
    return fb.mo_tensor(C, C)  # [(mu nu)][Q]


@pytest.mark.parametrize("form", [rijk.METRIC_INVSQRT, rijk.METRIC_CHOLESKY])
@pytest.mark.parametrize("n,naux,layout", [(150, 203, rijk.LAYOUT_PACKED), (129, 321, rijk.LAYOUT_NOPT_FULL),
                                           (193, 160, rijk.LAYOUT_PACKED), (64, 705, rijk.LAYOUT_NOPT_FULL)])
def test_metric_int8_tensor_matches_numpy(n, naux, layout, form):
    npad = -(-n // 64) * 64
    assert 1.0 * npad * (npad + 64) * naux * naux >= 2e9  # 2 x packed elements x naux^2: the int8 side of the rule
    V, I3 = _system(n, naux)
    if form == rijk.METRIC_INVSQRT:
        w, U = np.linalg.eigh(V)
        M = (U / np.sqrt(w)) @ U.T
    else:
        M = np.linalg.inv(np.linalg.cholesky(V))
    full = O.unpack_3c(I3, n).reshape(n * n, naux)
    ref = full @ M.T
    with rijk.FockBuilder(0) as fb:
        fb.set_metric(V, form)
        fb.set_3c(full if layout == rijk.LAYOUT_NOPT_FULL else I3, n, layout)
        got = _fitted(fb, n)
        assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
        for q0, q1 in ((0, naux - 61), (37, naux), (naux - 90, naux - 3)):  # small ranges stay on the FP64 units
            fb.set_aux_range(q0, q1)
            fb.set_3c(full if layout == rijk.LAYOUT_NOPT_FULL else I3, n, layout)
            part = _fitted(fb, n)
            assert np.max(np.abs(part - ref[:, q0:q1])) <= 1e-12 * np.max(np.abs(ref))
