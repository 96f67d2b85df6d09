"""The integral kernels against the host engine where their work decomposition has edges: more aux shells
of one l than a tile of 64 (and just as many), contracted aux shells beside single primitives, contracted
d and f bra shells (accumulated over primitive pairs), Cartesian aux shells, which another kernel takes, and
g orbitals (la + lb above the thread kernel's range).  Both sum the same terms in double precision in another
order, so they agree to 1e-12 of the largest element, as in test_gpu_eri.py."""
import numpy as np
import pytest

from nopt_b200 import ints, rijk
from nopt_b200.basis import Shell

pytestmark = pytest.mark.gpu


def _shells(rng, spec):
    """spec: [(l, primitives, count), ...] at random centres within 3 bohr."""
    out = []
    for l, nprim, count in spec:
        for _ in range(count):
            exps = np.exp(rng.uniform(np.log(0.15), np.log(12.0), nprim))
            out.append(Shell(l, exps, rng.uniform(0.2, 1.0, nprim), rng.uniform(-1.5, 1.5, 3), 0))
    return out


ORB = [(0, 4, 2), (1, 2, 1), (2, 1, 1), (2, 3, 1), (3, 1, 1), (3, 2, 1)]
CASES = {
    "one_tile_full": (ORB, [(0, 1, 64), (2, 1, 3)], True, True),
    "tile_and_one": (ORB, [(1, 1, 65), (3, 1, 2)], True, True),
    "contracted_aux": (ORB, [(0, 1, 2), (0, 3, 1), (1, 2, 2), (4, 1, 1), (4, 2, 1)], True, True),
    "cartesian_orbitals": ([(1, 2, 1), (2, 1, 2), (3, 1, 2)], [(0, 1, 3), (2, 1, 2), (4, 1, 2)], False, True),
    "cartesian_contracted_f": ([(3, 2, 2)], [(4, 1, 2)], False, True),  # accumulators beyond shared memory
    "cartesian_aux": (ORB, [(0, 1, 3), (2, 1, 2), (3, 2, 1)], True, False),
    "g_orbitals": ([(0, 2, 1), (3, 1, 1), (4, 1, 2)], [(0, 1, 2), (1, 1, 1), (4, 1, 1)], True, True),
}


@pytest.mark.parametrize("layout", [rijk.LAYOUT_PACKED, rijk.LAYOUT_NOPT_FULL])
@pytest.mark.parametrize("name", list(CASES))
def test_integrals_match_host_at_tile_edges(name, layout):
    orb_spec, aux_spec, orb_pure, aux_pure = CASES[name]
    rng = np.random.default_rng(len(name))
    orb, aux = ints.Basis(_shells(rng, orb_spec), orb_pure), ints.Basis(_shells(rng, aux_spec), aux_pure)
    with rijk.FockBuilder(0) as fb:
        V, I3 = fb.eri2c(aux), fb.eri3c(orb, aux, layout)
    Vh, Ih = ints.coulomb_2c(aux), ints.coulomb_3c(orb, aux, layout)
    assert np.max(np.abs(V - Vh)) <= 1e-12 * np.max(np.abs(Vh))
    assert np.max(np.abs(I3.reshape(Ih.shape) - Ih)) <= 1e-12 * np.max(np.abs(Ih))
