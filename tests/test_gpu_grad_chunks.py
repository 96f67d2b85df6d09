"""rijk_grad in chunks of aux functions: the chunk set by rijk_set_grad_chunk, or the one left when the scratch of all
aux functions is refused, bounds Y^Q and Gamma^Q.  Every element of every product keeps its terms and their order
whatever the chunk, so the derivatives are the same bits."""
import numpy as np
import pytest

from nopt_b200 import rijk

pytestmark = pytest.mark.gpu
N, NAUX, NOCC = 200, 700, 90


@pytest.fixture(scope="module")
def system():
    rng = np.random.default_rng(3)
    A = rng.normal(size=(NAUX, NAUX))
    V = A @ A.T / NAUX + np.eye(NAUX)
    I3 = rng.normal(size=(N * (N + 1) // 2, NAUX)) * 0.1
    MO = np.linalg.qr(rng.normal(size=(N, N)))[0].T.copy()
    return V, I3, MO, np.eye(N)


def _grad(fb, system, want_3c):
    out = fb.grad(system[2], NOCC, system[3], 0.0, want_3c=want_3c, want_metric=True)
    return [x for x in out if x is not None], fb.stats()["grad_qchunk"]


def _set(fb, system):
    fb.set_metric(system[0])
    fb.set_3c(system[1], N)


@pytest.mark.parametrize("want_3c", [True, False])
@pytest.mark.parametrize("chunk", [1, 29, 64, 699])
def test_chunks_give_the_same_bits(system, chunk, want_3c):
    with rijk.FockBuilder(0) as fb:
        _set(fb, system)
        want, whole = _grad(fb, system, want_3c)
        assert whole == NAUX
        fb.set_grad_chunk(chunk)
        got, used = _grad(fb, system, want_3c)
        assert used == chunk
    assert all(np.array_equal(a, b) for a, b in zip(want, got))


def test_a_chunk_bounds_the_scratch(system):
    """Scratch that the pool keeps after a first call, dE/d(P|Q) alone.  Y of all aux functions takes naux n_c' n_c, T and
    Gamma naux (npad n_c' + 10 x 64^2) doubles (n_c' = 96, npad = 256); a chunk of 14 a fiftieth of that.  The pool
    holds the block of raw integrals of the set-up already."""
    import torch
    whole, raw = 8 * NAUX * (96 * NOCC + 256 * 96 + 10 * 4096), 8 * NAUX * N * (N + 1) // 2
    used = {}
    for chunk in (0, 14):
        with rijk.FockBuilder(0) as fb:
            _set(fb, system)
            fb.grad(system[2], NOCC, system[3], 0.0)  # the build's own buffers
            fb.set_grad_chunk(chunk)
            before = torch.cuda.mem_get_info()[0]
            _grad(fb, system, False)
            used[chunk] = before - torch.cuda.mem_get_info()[0]
    assert used[0] >= 0.9 * whole - raw and used[14] <= 0.3 * whole


@pytest.mark.parametrize("want_3c", [True, False])
def test_refused_scratch_makes_smaller_chunks(system, want_3c):
    """Each request refused twice: those for Y and for Gamma come again for half as much, others are reported."""
    chunks = set()
    with rijk.FockBuilder(0) as fb:
        _set(fb, system)
        want, _ = _grad(fb, system, want_3c)
        done = 0
        for k in range(40):
            fb.selftest_alloc_refuse(k, 2)
            try:
                got, used = _grad(fb, system, want_3c)
            except rijk.RijkError as e:
                assert e.code == rijk.ERR_ALLOC
                continue
            finally:
                fb.selftest_alloc_refuse(0, 0)
            chunks.add(used)
            assert all(np.array_equal(a, b) for a, b in zip(want, got))
            done += 1
    assert chunks == {NAUX, NAUX // 2} and done >= 2
