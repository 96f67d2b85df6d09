"""A device without memory pools (some virtualised modes report none): the context works all the same, with scratch
from plain allocations.  A child process runs with cudaMemPoolCreate replaced by one that answers "not supported"."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = "int cudaMemPoolCreate(void** pool, const void* props) { *pool = 0; return 801; }\n"
PROGRAM = """
import sys
sys.path.insert(0, %r)
import numpy as np
from nopt_b200 import ints, rijk
from nopt_b200.molecules import water_cluster
si = ints.SystemIntegrals(water_cluster((1, 1, 2), seed=0), "cc-pvdz", "cc-pvdz-jkfit", ri_integrals=False)
MO = np.linalg.qr(np.random.default_rng(0).normal(size=(si.n, si.n)))[0].T.copy()
with rijk.FockBuilder(0) as fb:
    fb.set_basis(si.orb, si.aux)
    J, K = fb.dm_to_f_transform_ri(MO[:si.nocc].T @ MO[:si.nocc], MO, si.nocc)
    E, dC, d3, dV = fb.grad(MO, si.nocc, si.H, si.Enuc, want_3c=True, want_metric=True)
    np.savez(sys.argv[1], J=J, K=K, E=E, dC=dC, d3=d3, dV=dV, T=fb.mo_tensor(MO[:4], MO[:7]))
"""


def test_a_context_without_a_pool(tmp_path):
    shim = str(tmp_path / "nopool.so")
    open(str(tmp_path / "nopool.c"), "w").write(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", str(tmp_path / "nopool.c"), "-o", shim], check=True)
    got = []
    for preload in (None, shim):
        out = str(tmp_path / "r.npz")
        env = dict(os.environ, **({"LD_PRELOAD": preload} if preload else {}))
        subprocess.run([sys.executable, "-c", PROGRAM % ROOT, out], check=True, env=env, timeout=300)
        with np.load(out) as z:
            got.append({k: z[k] for k in z.files})
    for k in got[0]:
        assert np.array_equal(got[0][k], got[1][k]), k
