"""The first build of a new context takes its small buffers from the scratch that the set-up has left in the context's
pool: device memory outside it stays as it was.  (The kernels' modules, which a first use loads, are there from an
earlier context.)  Results of two contexts on streams of their own, buffers grown between builds, agree to the bit."""
import numpy as np
import pytest

from nopt_b200 import ints, rijk
from nopt_b200.molecules import water_cluster

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hexamer():
    si = ints.SystemIntegrals(water_cluster((2, 3), seed=0), "cc-pvdz", "cc-pvdz-jkfit", ri_integrals=False)
    return si, np.linalg.qr(np.random.default_rng(2).normal(size=(si.n, si.n)))[0].T.copy()


def _build(fb, MO, nocc, precision=rijk.PREC_FP64):
    return fb.dm_to_f_transform_ri(MO[:nocc].T @ MO[:nocc], MO, nocc, precision)


def test_first_build_takes_no_new_memory(hexamer):
    import torch
    si, MO = hexamer
    for warm in (True, False):
        with rijk.FockBuilder(0) as fb:
            fb.set_basis(si.orb, si.aux)
            before = torch.cuda.mem_get_info()[0]
            _build(fb, MO, si.nocc)
            if not warm:
                assert torch.cuda.mem_get_info()[0] == before


def test_buffers_grow_beside_another_context(hexamer):
    import torch
    si, MO = hexamer
    sizes = [(1, rijk.PREC_FP64), (si.nocc, rijk.PREC_MIXED), (si.nocc, rijk.PREC_FP64), (90, rijk.PREC_FP64_TC),
             (90, rijk.PREC_MIXED), (144, rijk.PREC_FP64), (5, rijk.PREC_FP64)]
    want = []
    for nocc, precision in sizes:
        with rijk.FockBuilder(0) as fb:
            fb.set_basis(si.orb, si.aux)
            want.append(_build(fb, MO, nocc, precision))
    stream = torch.cuda.Stream()
    with rijk.FockBuilder(0) as one, rijk.FockBuilder(0) as two:
        two.set_stream(stream.cuda_stream)
        for fb in (one, two):
            fb.set_basis(si.orb, si.aux)
        for (nocc, precision), ref in zip(sizes, want):
            for fb in (one, two):
                T = fb.mo_tensor(MO[:9], MO[:4])  # pool scratch between the builds
                got = _build(fb, MO, nocc, precision)
                assert all(np.array_equal(a, b) for a, b in zip(got, ref))
                assert np.array_equal(T, fb.mo_tensor(MO[:9], MO[:4]))
