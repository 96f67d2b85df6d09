"""FP64 builds over functions of very unequal size.  Multiplying function mu by a power of two s_mu and dividing its
orbital coefficients by it changes nothing but K_mn by s_m s_n, exactly; so each element of K must keep its accuracy
against sqrt(K_mm K_nn), the size that goes along with the scaling, and J its against sqrt(J_mm J_nn).  The int8
exchange rounds its operands at 2^-55 of the largest of a row; the oracle and the FP64 kernels sum up to
n + n_aux n_c = 28,300 terms, each sum within its terms' number times 2^-53 of the sum of the terms' magnitudes, which
the Cauchy-Schwarz inequality bounds by sqrt(K_mm K_nn): 3.2e-12 in the worst case, 1e-11 allowed."""
import numpy as np
import pytest

import rijk_oracle as O
from nopt_b200 import rijk

pytestmark = pytest.mark.gpu
N, NAUX, NOCC = 260, 700, 40


@pytest.fixture(scope="module")
def system():
    rng = np.random.default_rng(7)
    A = rng.normal(size=(NAUX, NAUX))
    V = A @ A.T / NAUX + np.eye(NAUX)
    rows, cols = np.tril_indices(N)
    # pairs of functions fall off with their distance on a line, as those of a chain do
    I3 = rng.normal(size=(len(rows), NAUX)) * np.exp(-np.abs(rows - cols) / 40.0)[:, None]
    MO = np.linalg.qr(rng.normal(size=(N, N)))[0].T.copy()
    ref = O.dm_to_f_transform_ri(O.unpack_3c(I3, N), O.s05_calc(V)[0], O.gen_hf_dm(MO, N, NOCC), MO, NOCC, N)
    return V, I3, MO, ref


@pytest.mark.parametrize("precision", [rijk.PREC_FP64, rijk.PREC_FP64_TC])
@pytest.mark.parametrize("spread", [0, 6, 20, 60])
def test_k_keeps_its_accuracy_under_row_scales(system, spread, precision):
    V, I3, MO, (Jr, Kr) = system
    s = np.ldexp(1.0, -np.random.default_rng(spread).integers(0, spread + 1, N))
    rows, cols = np.tril_indices(N)
    scaled = MO / s
    with rijk.FockBuilder(0) as fb:
        fb.set_metric(V)
        fb.set_3c(I3 * (s[rows] * s[cols])[:, None], N)
        fb.set_profiling(True)
        J, K = fb.dm_to_f_transform_ri(O.gen_hf_dm(scaled, N, NOCC), scaled, NOCC, precision)
        assert {"xform_i8", "syrk_i8"} <= set(fb.stats()["stages"])
    J, K = J / np.outer(s, s), K / np.outer(s, s)
    d = np.sqrt(np.abs(np.diag(Kr)))
    assert np.max(np.abs(K - Kr) / np.outer(d, d)) <= 1e-11
    assert np.max(np.abs(J - Jr)) <= 1e-11 * np.max(np.abs(Jr))


@pytest.mark.parametrize("exponent", [0, -40, 40])
def test_rows_that_couple_to_nothing(system, exponent):
    """Functions without any integral, and one that couples only off the diagonal, between ordinary ones, whose sizes
    are all of one order or spread: the coefficients of the former are then of another order than all others."""
    V, I3, MO, _ = system
    rows, cols = np.tril_indices(N)
    s = np.ldexp(1.0, np.where(np.arange(N) % 3, exponent, exponent // 2))
    I3 = I3.copy()
    for dead in (0, 77, N - 1):
        I3[(rows == dead) | (cols == dead)] = 0.0
    I3[(rows == 130) & (cols == 130)] = 0.0
    I3[(rows == 130) ^ (cols == 130)] *= 2.0 ** -30
    Kr = O.dm_to_f_transform_ri(O.unpack_3c(I3, N), O.s05_calc(V)[0], O.gen_hf_dm(MO, N, NOCC), MO, NOCC, N)[1]
    C = MO / s
    for dead in (0, 77, N - 1):
        C[:, dead] = MO[:, dead]
    with rijk.FockBuilder(0) as fb:
        fb.set_metric(V)
        fb.set_3c(I3 * (s[rows] * s[cols])[:, None], N)
        K = fb.dm_to_f_transform_ri(O.gen_hf_dm(C, N, NOCC), C, NOCC)[1] / np.outer(s, s)
    d = np.sqrt(np.abs(np.diag(Kr)))
    assert np.all(np.abs(K - Kr) <= 1e-11 * np.outer(d, d))
