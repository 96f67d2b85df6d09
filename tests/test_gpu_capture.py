"""rijk_fock_device recorded into a CUDA graph.  A recorded build must not leave anything behind that only a replay
would have formed, and a replay must read the tensor that the context holds then: the next geometry of a molecule
has the same sizes and takes the same memory."""
import numpy as np
import pytest

import rijk_oracle as O
from nopt_b200 import rijk

pytestmark = pytest.mark.gpu
N, NAUX, NOCC = 300, 1100, 32


def _system(seed):
    rng = np.random.default_rng(seed)
    A = rng.normal(size=(NAUX, NAUX))
    V = A @ A.T / NAUX + np.eye(NAUX)
    I3 = rng.normal(size=(N * (N + 1) // 2, NAUX))
    MO = np.linalg.qr(rng.normal(size=(N, N)))[0].T.copy()
    D = O.gen_hf_dm(MO, N, NOCC)
    return V, I3, D, MO, O.dm_to_f_transform_ri(O.unpack_3c(I3, N), O.s05_calc(V)[0], D, MO, NOCC, N)


@pytest.mark.parametrize("precision", [rijk.PREC_FP64, rijk.PREC_FP64_TC])
def test_recorded_builds_and_the_digits_of_b(precision):
    import torch
    first, second = _system(1), _system(2)
    dev = torch.device("cuda", 0)
    stream = torch.cuda.Stream(dev)
    with rijk.FockBuilder(0) as fb:
        fb.set_stream(stream.cuda_stream)
        dD, dC = torch.empty(N, N, dtype=torch.float64, device=dev), torch.empty(NOCC, N, dtype=torch.float64, device=dev)
        dJ, dK = torch.empty_like(dD), torch.empty_like(dD)

        def load(s):
            dD.copy_(torch.from_numpy(np.ascontiguousarray(s[2])))
            dC.copy_(torch.from_numpy(np.ascontiguousarray(s[3][:NOCC])))
            torch.cuda.synchronize()

        def build():
            fb.fock_device(dD.data_ptr(), dC.data_ptr(), NOCC, dJ.data_ptr(), dK.data_ptr(), precision)

        def check(s):
            torch.cuda.synchronize()
            for got, want in zip((dJ, dK), s[4]):
                assert np.max(np.abs(got.cpu().numpy() - want)) <= 1e-11 * np.max(np.abs(want))

        fb.set_metric(first[0])
        fb.set_3c(first[1], N)
        load(first)
        build()  # every buffer and module is there
        check(first)
        # a new tensor, and the first build with it is only recorded
        fb.set_metric(second[0])
        fb.set_3c(second[1], N)
        load(second)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            build()
        dK.zero_()
        build()
        check(second)
        dK.zero_()
        torch.cuda.synchronize()
        graph.replay()
        check(second)
        # the graph after one more tensor of these sizes
        fb.set_metric(first[0])
        fb.set_3c(first[1], N)
        load(first)
        dK.zero_()
        torch.cuda.synchronize()
        graph.replay()
        check(first)
        del graph


@pytest.mark.parametrize("nocc", [NOCC, 2])
def test_a_recorded_first_build_is_refused(nocc):
    """A recording cannot allocate.  A build that would have to is refused, and leaves nothing behind: the next ordinary
    build takes its buffers and is right."""
    import torch
    s = _system(1)
    D = s[3][:nocc].T @ s[3][:nocc]
    stream = torch.cuda.Stream()
    with rijk.FockBuilder(0) as fb:
        fb.set_stream(stream.cuda_stream)
        fb.set_metric(s[0])
        fb.set_3c(s[1], N)
        want = fb.dm_to_f_transform_ri(D, s[3], nocc)
    with rijk.FockBuilder(0) as fb:
        fb.set_stream(stream.cuda_stream)
        fb.set_metric(s[0])
        fb.set_3c(s[1], N)
        dD = torch.from_numpy(np.ascontiguousarray(D)).cuda()
        dC = torch.from_numpy(np.ascontiguousarray(s[3][:nocc])).cuda()
        dJ, dK = torch.empty_like(dD), torch.empty_like(dD)
        torch.cuda.synchronize()
        refused = False
        try:
            with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=stream):
                try:
                    fb.fock_device(dD.data_ptr(), dC.data_ptr(), nocc, dJ.data_ptr(), dK.data_ptr())
                except rijk.RijkError as e:
                    refused = e.code == rijk.ERR_CUDA
        except RuntimeError:  # torch on the recording's end
            pass
        assert refused
        torch.cuda.synchronize()
        fb.fock_device(dD.data_ptr(), dC.data_ptr(), nocc, dJ.data_ptr(), dK.data_ptr())
        fb.sync()
        assert all(np.array_equal(a.cpu().numpy(), b) for a, b in zip((dJ, dK), want))
