"""FP64 builds on the int8 tensor cores when device memory runs short: the digits of B are a copy the library can
do without, so no allocation that fails while they are held, or that fails for them, is the caller's error.
rijk_selftest_alloc_refuse answers single requests for memory as an exhausted device would.  J and K against the
oracle as in test_gpu_fp64_int8.py (the same tolerance, derived there)."""
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
    I3 = rng.normal(size=(n * (n + 1) // 2, naux))
    C, _ = np.linalg.qr(rng.normal(size=(n, n)))
    MO = C.T.copy()
    D = O.gen_hf_dm(MO, n, nocc)
    ref = O.dm_to_f_transform_ri(O.unpack_3c(I3, n), O.s05_calc(V)[0], D, MO, nocc, n)
    return V, I3, D, MO, ref


def _set(fb, system, n):
    fb.set_metric(system[0])
    fb.set_3c(system[1], n)


def _build(fb, system, nocc, precision=rijk.PREC_FP64):
    """The build's kernels; J and K are checked."""
    fb.set_profiling(True)
    got = fb.dm_to_f_transform_ri(system[2], system[3], nocc, precision)
    fb.set_profiling(False)
    for a, b in zip(got, system[4]):
        assert np.max(np.abs(a - b)) <= TOL * np.max(np.abs(b))
    return set(fb.stats()["stages"])


def test_more_aux_functions_in_the_memory_of_earlier_digits():
    """The second tensor's digits fit the memory of the first's exactly, its exponents do not: the request for these is
    refused until the digits' memory has been given back."""
    first, second = _system(450, 660, 20), _system(300, 1100, 32)  # 660 x 10 and 1100 x 6 blocks
    with rijk.FockBuilder(0) as fb:
        _set(fb, first, 450)
        assert "xform_i8" in _build(fb, first, 20)
        _set(fb, second, 300)
        fb.dm_to_f_transform_ri(second[2], second[3], 1)  # below the rule: the Coulomb buffers
        fb.selftest_alloc_refuse(1, 2)  # after the staged orbitals
        assert "xform_i8" in _build(fb, second, 32)


def test_no_room_for_the_digits():
    system = _system(300, 1100, 32)
    with rijk.FockBuilder(0) as fb:
        _set(fb, system, 300)
        fb.dm_to_f_transform_ri(system[2], system[3], 1)
        fb.selftest_alloc_refuse(2, 2)  # after the staged orbitals and the exponents: the digits, asked for twice
        assert "xform_f64" in _build(fb, system, 32)
        assert "xform_f64" in _build(fb, system, 32)  # not asked for again with this tensor
        _set(fb, system, 300)
        assert "xform_i8" in _build(fb, system, 32)


def test_digits_make_room_for_a_larger_build():
    """Each request of a build with more orbitals is refused twice: the digits are given back, if it is not for one of
    their own buffers, and the build goes on without them."""
    n, nocc = 300, 90
    system = _system(n, 1100, nocc)
    seen = set()
    for k in range(20):
        with rijk.FockBuilder(0) as fb:
            _set(fb, system, n)
            fb.dm_to_f_transform_ri(system[2], system[3], 32)
            fb.selftest_alloc_refuse(k, 2)
            stages = _build(fb, system, nocc)
            fb.selftest_alloc_refuse(0, 0)
        seen |= stages
        if k > 0 and "xform_i8" in stages:  # no such request any more
            break
    assert k < 19 and {"xform_i8", "xform_f64"} <= seen


CALLS = {
    "mo_tensor": lambda fb, s: fb.mo_tensor(s[3][:5], s[3][:3]),
    "mo_calc": lambda fb, s: tuple(fb.mo_calc(s[3][:60], 3, 4, 53).values()),
    "mo_ints": lambda fb, s: fb.calc_2el_mo_ints_ri(None, s[3], s[3][:4], s[3][:4], 3, 4, want_jk=False)[0],
    "hess_ints": lambda fb, s: fb.soscf_hess_ints(s[3][:40], 3, 4),
    "grad": lambda fb, s: fb.grad(s[3], 4, np.eye(300), 0.0, want_3c=True, want_metric=True),
    "metric": lambda fb, s: fb.set_metric(s[0]),
    "three_centre": lambda fb, s: fb.set_3c(s[1], 300),
}


@pytest.mark.parametrize("name", list(CALLS))
def test_scratch_takes_the_memory_of_the_digits(name):
    """Scratch that is refused twice, the second time with the pool's spare blocks gone, has the digits' memory; refused
    once, the pool's alone.  The results are those of a call that met no shortage, and the next build forms the
    digits again."""
    n, nocc = 300, 32
    system = _system(n, 1100, nocc)
    call = CALLS[name]
    with rijk.FockBuilder(0) as fb:
        _set(fb, system, n)
        want = call(fb, system)
        for times in (1, 2):
            for after in (0, 3):
                if name == "metric":
                    _set(fb, system, n)
                assert "xform_i8" in _build(fb, system, nocc)
                fb.selftest_alloc_refuse(after, times)
                got = call(fb, system)
                fb.selftest_alloc_refuse(0, 0)
                if want is not None:
                    for a, b in zip(np.atleast_1d(want) if not isinstance(want, tuple) else want,
                                    np.atleast_1d(got) if not isinstance(got, tuple) else got):
                        assert np.array_equal(a, b)
        if name == "metric":
            _set(fb, system, n)
        assert "xform_i8" in _build(fb, system, nocc)


def test_digits_of_an_old_tensor_are_released():
    import torch
    system, small = _system(450, 700, 20), _system(70, 60, 5)
    with rijk.FockBuilder(0) as fb:
        _set(fb, system, 450)
        assert "xform_i8" in _build(fb, system, 20)
        before = torch.cuda.mem_get_info()[0]
        _set(fb, small, 70)
        # 700 aux functions x 10 blocks of 128 x 128 elements in 7 bytes each: 0.8 GB
        assert torch.cuda.mem_get_info()[0] - before > 700 * 10 * 128 * 128 * 7 // 2


def test_no_room_for_the_int8_exchange():
    """Each request of a first large build is refused three times: neither the pool's blocks nor the digits of B then
    make room, and the exchange runs on the FP64 units, which need less.  A new tensor tries the digits again."""
    n, nocc = 300, 40
    system = _system(n, 1100, nocc)
    seen = []
    for k in range(1, 20):
        with rijk.FockBuilder(0) as fb:
            _set(fb, system, n)
            fb.dm_to_f_transform_ri(system[2], system[3], 1)
            fb.selftest_alloc_refuse(k, 3)  # the staged orbitals, the one request without another way, go through
            seen.append(_build(fb, system, nocc))
            fb.selftest_alloc_refuse(0, 0)
            if "syrk_f64" in seen[-1]:
                assert "xform_f64" in seen[-1]
                assert "syrk_f64" in _build(fb, system, nocc)  # not asked for again with this tensor
                _set(fb, system, n)
                assert {"xform_i8", "syrk_i8"} <= _build(fb, system, nocc)
            elif "xform_i8" in seen[-1]:  # no such request any more
                break
    # the orbitals, X, its digits and their exponents (the partial sums of the small build are large enough)
    assert sum("syrk_f64" in s for s in seen) >= 4 and "xform_i8" in seen[-1]
