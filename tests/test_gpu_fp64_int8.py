"""FP64 builds whose exchange runs on the int8 tensor cores (the half-transform and K from exact products of byte
digits; taken from about 1e10 FLOPs and n > 192 on): J and K against the oracle at the edges of its work
decomposition.  128-row blocks that end in one 64-row tile or in a few rows, contraction lengths off a multiple
of 32, orbital batches of 16, 32, 48 and 64 and mixtures of them, part lengths of odd and even numbers of aux
functions, and both sides of the rule.  The digits keep 2^-55 of the largest element of an operand and the
oracle sums in double precision, so the two agree to the rounding of the oracle's own sums over n n_c n_aux
terms, far inside 1e-11 of the largest element of K (the metrics here are well conditioned)."""
import os

import numpy as np
import pytest

import rijk_oracle as O
from nopt_b200 import rijk

pytestmark = pytest.mark.gpu
TOL = 1e-11


def _system(n, naux, nocc, seed=0):
    rng = np.random.default_rng(seed + n + naux)
    A = rng.normal(size=(naux, naux))
    V = A @ A.T / naux + np.eye(naux)
    I3 = rng.normal(size=(n * (n + 1) // 2, naux)) * np.exp(rng.uniform(-8, 0, size=(n * (n + 1) // 2, 1)))
    C, _ = np.linalg.qr(rng.normal(size=(n, n)))
    MO = C.T.copy()
    return V, I3, O.gen_hf_dm(MO, n, nocc), MO


def _reference(V, I3, D, MO, n, nocc):
    Vm05, _ = O.s05_calc(V)
    return O.dm_to_f_transform_ri(O.unpack_3c(I3, n), Vm05, D, MO, nocc, n)


def _check(got, ref):
    for a, b in zip(got, ref):
        assert np.max(np.abs(a - b)) <= TOL * np.max(np.abs(b))


@pytest.mark.parametrize("n,naux,nocc", [
    (193, 3203, 1),    # one orbital in a batch of 16; one row past 192
    (257, 691, 33),    # 48 orbitals in one batch, one row in the last tile
    (320, 511, 64),    # a full batch; the last 128-row block half empty
    (321, 291, 65),    # 48 + 32
    (384, 207, 100),    # 64 + 48, every block full
    (448, 117, 129),    # 48 + 48 + 48; 448 ends in half a block
    (450, 67, 200),    # 64 + 48 + 48 + 48
])
def test_fp64_int8_matches_oracle(n, naux, nocc):
    npad, noccp = -(-n // 64) * 64, -(-nocc // 16) * 16
    assert npad > 192 and 3.0 * npad * npad * noccp * naux >= 1e10  # on the int8 side of the rule
    V, I3, D, MO = _system(n, naux, nocc)
    ref = _reference(V, I3, D, MO, n, nocc)
    with rijk.FockBuilder(0) as fb:
        fb.set_metric(V)
        fb.set_3c(I3, n)
        fb.set_profiling(True)
        got = fb.dm_to_f_transform_ri(D, MO, nocc)
        assert {"xform_i8", "syrk_i8"} <= set(fb.stats()["stages"])
        fb.set_profiling(False)
        _check(got, ref)
        again = fb.dm_to_f_transform_ri(D, MO, nocc)  # the side stream's schedule
        assert all(np.array_equal(a, b) for a, b in zip(got, again))


def test_fp64_below_the_rule_stays_on_dmma():
    V, I3, D, MO = _system(200, 40, 20)
    with rijk.FockBuilder(0) as fb:
        fb.set_metric(V)
        fb.set_3c(I3, 200)
        fb.set_profiling(True)
        got = fb.dm_to_f_transform_ri(D, MO, 20)
        assert {"xform_f64", "syrk_f64"} <= set(fb.stats()["stages"])
    _check(got, _reference(V, I3, D, MO, 200, 20))


def test_fp64_int8_follows_a_new_tensor_a_slice_and_a_file(tmp_path):
    """The digits belong to the present tensor: another one in the same context, an aux slice and its rest, and
    a tensor read from a file (whose magnitudes are not those of a metric contraction)."""
    n, naux, nocc = 260, 1400, 40
    first, second = _system(n, naux, nocc), _system(n, naux, nocc, seed=9)
    path = os.path.join(str(tmp_path), "b.rijk")
    with rijk.FockBuilder(0) as fb:
        for V, I3, D, MO in (first, second):
            fb.set_metric(V)
            fb.set_3c(I3 * 3.0, n)
            J, K = fb.dm_to_f_transform_ri(D, MO, nocc)
            _check((J, K), [9.0 * x for x in _reference(V, I3, D, MO, n, nocc)])
        fb.save(path)
        parts = []
        for q0, q1 in ((0, 699), (699, naux)):
            fb.set_aux_range(q0, q1)
            fb.set_3c(I3 * 3.0, n)
            parts.append(fb.dm_to_f_transform_ri(D, MO, nocc))
        _check([a + b for a, b in zip(*parts)], (J, K))
        fb.load(path)
        _check(fb.dm_to_f_transform_ri(D, MO, nocc), (J, K))


def test_fp64_without_room_for_the_digits():
    """An allocation failure at the digits of B is none of the caller's: the half-transform then stays on DMMA."""
    n, naux, nocc = 260, 700, 40
    V, I3, D, MO = _system(n, naux, nocc)
    with rijk.FockBuilder(0) as fb:
        fb.set_metric(V)
        fb.set_3c(I3, n)
        fb.dm_to_f_transform_ri(D, MO, 1)  # below the rule: the Coulomb buffers
        fb.selftest_alloc_failure(1)       # the staged orbitals, then the digits and all after them
        with pytest.raises(rijk.RijkError) as e:
            fb.dm_to_f_transform_ri(D, MO, nocc)
        assert e.value.code == rijk.ERR_ALLOC
        fb.selftest_alloc_failure(-1)
        _check(fb.dm_to_f_transform_ri(D, MO, nocc), _reference(V, I3, D, MO, n, nocc))


def test_fp64_int8_passes_on_what_is_not_finite():
    n, naux, nocc = 260, 700, 40
    V, I3, D, MO = _system(n, naux, nocc)
    MO = MO.copy()
    MO[3, 7] = np.nan
    with rijk.FockBuilder(0) as fb:
        fb.set_metric(V)
        fb.set_3c(I3, n)
        J, K = fb.dm_to_f_transform_ri(D, MO, nocc)
        assert np.isfinite(J).all() and np.isnan(K).all()
