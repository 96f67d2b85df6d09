"""Timed workloads of the RI-JK library: what quantum-chemistry programs call it for, as single calls.

A case names a call, a molecule (a water cluster or an n-alkane, every seed another geometry), its basis
pair and, for Fock builds, the precision.  The calls:

  fock_host    J, K of a density in host arrays (dm_to_f_transform_ri), the drop-in call of a CPU program
  fock_device  the same with the density, orbitals, J and K resident on the GPU (fock_device)
  scf          a whole restricted Hartree-Fock run from the superposition of atomic densities
  setup        a new geometry: integrals, metric and fitted tensor on the GPU, then the guess's build
  eri3c        (P|Q) and (mu nu|P) handed to a program that keeps its own three-index tensor
  grad         the energy derivatives with respect to orbitals, (P|mu nu) and (P|Q)
  casscf       the integrals of one CASSCF macro-iteration: core J, K and the active-space blocks
  mo_tensor    the MO-basis three-index tensors of a perturbation-theory step (mo_calc)

Molecules run from one water to C40H82 in double-zeta and to twelve waters in triple-zeta bases.
"""
import math

import numpy as np
import torch

from nopt_b200 import basis as basis_data
from nopt_b200 import ints, molecules, rijk

DZ, TZ = ("cc-pvdz", "cc-pvdz-jkfit"), ("cc-pvtz", "cc-pvtz-jkfit")
DZ_RI = ("cc-pvdz", "cc-pvdz-ri")
PRECISION = {"fp64": rijk.PREC_FP64, "mixed": rijk.PREC_MIXED, "fp64_tc": rijk.PREC_FP64_TC}
SCF_BUILDS = 12  # Fock builds a converged run cannot do without, about


def _case(call, molecule, size, pair, **more):
    return dict(call=call, molecule=molecule, size=size, orbital=pair[0], aux=pair[1], **more)


def listed():
    return [
        # a dimer's SCF iteration in a CPU program: latency of the call and its launches
        dict(_case("fock_host", "water", 2, DZ, precision="fp64"), name="fock_host_h2o2_dz"),
        # the reference's own size of run, through the drop-in call
        dict(_case("fock_host", "water", 6, DZ, precision="fp64"), name="fock_host_h2o6_dz"),
        # an ordinary medium molecule's build, everything resident on the GPU
        dict(_case("fock_device", "water", 16, DZ, precision="fp64"), name="fock_fp64_h2o16_dz"),
        # the largest FP64 build here: n_ao 970, a partial last tile, 161 orbitals
        dict(_case("fock_device", "alkane", 40, DZ, precision="fp64"), name="fock_fp64_c40h82_dz"),
        # the early iterations of a mixed-precision SCF, medium and large (odd carbon count)
        dict(_case("fock_device", "water", 16, DZ, precision="mixed"), name="fock_mixed_h2o16_dz"),
        dict(_case("fock_device", "alkane", 31, DZ, precision="mixed"), name="fock_mixed_c31h64_dz"),
        # FP64-accurate builds on the integer tensor cores, as an SCF's final iterations may ask
        dict(_case("fock_device", "alkane", 25, DZ, precision="fp64_tc"), name="fock_fp64tc_c25h52_dz"),
        # a whole RHF run of a medium molecule
        dict(_case("scf", "water", 16, DZ), name="scf_h2o16_dz"),
        # one geometry step's set-up in a triple-zeta basis
        dict(_case("setup", "water", 8, TZ), name="setup_h2o8_tz"),
        # the energy derivatives of a geometry step
        dict(_case("grad", "water", 8, DZ), name="grad_h2o8_dz"),
        # one CASSCF macro-iteration with ten active orbitals
        dict(_case("casscf", "alkane", 10, DZ, active=10), name="casscf_c10h22_dz"),
        # the MO tensors before a perturbation-theory step
        dict(_case("mo_tensor", "water", 6, DZ, active=6), name="mo_tensor_h2o6_dz"),
    ]


def _size(rng, molecule, high):
    low = 2 if molecule == "alkane" else 1
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    call = rng.choice(["fock_host", "fock_device", "fock_device", "scf", "setup", "eri3c", "grad", "casscf", "mo_tensor"])
    molecule = rng.choice(["water", "alkane"])
    if call in ("fock_host", "fock_device"):
        pair = rng.choice([DZ, DZ, TZ, DZ_RI])
        top = {("water", DZ): 24, ("water", DZ_RI): 24, ("water", TZ): 10, ("alkane", DZ): 36, ("alkane", DZ_RI): 36,
               ("alkane", TZ): 10}[molecule, pair]
        return _case(call, molecule, _size(rng, molecule, top), pair, precision=rng.choice(["fp64", "fp64", "mixed", "fp64_tc"]))
    if call == "scf":
        return _case(call, molecule, _size(rng, molecule, 14), DZ)
    if call == "setup":
        pair = rng.choice([DZ, TZ])
        return _case(call, molecule, _size(rng, molecule, 20 if pair is DZ else 10), pair)
    if call == "eri3c":
        pair = rng.choice([DZ, TZ])
        return _case(call, molecule, _size(rng, molecule, 8 if pair is DZ else 4), pair)
    if call == "grad":
        return _case(call, molecule, _size(rng, molecule, 12), DZ)
    return _case(call, molecule, _size(rng, molecule, 12), DZ, active=rng.randint(2, 12) if call == "casscf" else rng.randint(0, 10))


# ------------------------------------------------------------------------------ molecules ----

def _molecule(case, seed):
    k = case["size"]
    if case["molecule"] == "alkane":
        return molecules.alkane(k, seed=seed)
    side = max(1, math.ceil(k ** (1 / 3)))
    full = molecules.water_cluster((side, side, math.ceil(k / side ** 2)), seed=seed)
    return molecules.Molecule(full.symbols[:3 * k], full.coords_ang[:3 * k])


def _sizes(case):
    """(n_ao, n_aux, occupied orbitals)"""
    k = case["size"]
    atoms = {"O": k, "H": 2 * k} if case["molecule"] == "water" else {"C": k, "H": 2 * k + 2}
    count = []
    for name in (case["orbital"], case["aux"]):
        data = basis_data.read_gbs(name)
        count.append(sum(a * sum(2 * l + 1 for l, _, _ in data[el]) for el, a in atoms.items()))
    return count[0], count[1], sum(a * {"H": 1, "C": 6, "O": 8}[el] for el, a in atoms.items()) // 2


def _input(case, seed):
    """What the calls take: the bases and, from the molecule alone, S, H, the starting density and orbitals."""
    mol = _molecule(case, seed)
    si = ints.SystemIntegrals(mol, case["orbital"], case["aux"], ri_integrals=False)
    got = {"case": dict(case), "si": si, "n": si.n, "naux": si.naux, "nocc": si.nocc}
    if case["call"] in ("scf", "setup"):
        got["D0"], got["R"] = si.sad()
    if case["call"] not in ("setup", "eri3c"):  # orthonormal orbitals: eigenvectors of H, lowest first
        S, H = (torch.from_numpy(m).cuda() for m in (si.S, si.H))
        w, U = torch.linalg.eigh(S)
        X = U * w.rsqrt()
        C = X @ torch.linalg.eigh(X.T @ H @ X)[1]
        got["MO"] = C.T.contiguous().cpu().numpy()
        occupied = got["MO"][:si.nocc]
        got["D"] = np.ascontiguousarray(occupied.T @ occupied)
    return got


def prepare(case, seed):
    s = _input(case, seed)
    fb = s["fb"] = rijk.FockBuilder(torch.cuda.current_device())
    n = s["n"]
    if case["call"] in ("fock_host", "setup", "casscf"):
        s["J"], s["K"] = np.empty((n, n)), np.empty((n, n))
    if case["call"] in ("setup", "eri3c"):
        return s
    fb.set_basis(s["si"].orb, s["si"].aux)
    if case["call"] == "fock_device":
        fb.set_stream(torch.cuda.current_stream().cuda_stream)
        s["dD"], s["dC"] = (torch.from_numpy(np.ascontiguousarray(m)).cuda() for m in (s["D"], s["MO"][:s["nocc"]]))
        s["dJ"], s["dK"] = torch.empty_like(s["dD"]), torch.empty_like(s["dD"])
    if case["call"] == "grad":
        s["d3"], s["dV"] = np.empty((n * (n + 1) // 2, s["naux"])), np.empty((s["naux"], s["naux"]))
    return s


def run(s):
    case, fb, si = s["case"], s["fb"], s["si"]
    call, nocc = case["call"], s["nocc"]
    if call == "fock_device":
        fb.fock_device(s["dD"].data_ptr(), s["dC"].data_ptr(), nocc, s["dJ"].data_ptr(), s["dK"].data_ptr(),
                       PRECISION[case["precision"]])
        return s["dJ"], s["dK"]
    if call == "fock_host":
        return fb.dm_to_f_transform_ri(s["D"], s["MO"], nocc, PRECISION[case["precision"]], s["J"], s["K"])
    if call == "scf":
        energy, MO, _ = fb.scf(si.H, si.S, nocc, si.Enuc, guess=(s["D0"], s["R"]))
        return np.float64(energy), MO[:nocc].T @ MO[:nocc]
    if call == "setup":
        fb.set_basis(si.orb, si.aux)
        return fb.dm_to_f_transform_ri(s["D0"], s["R"], s["R"].shape[0], rijk.PREC_FP64, s["J"], s["K"])
    if call == "eri3c":
        return fb.eri2c(si.aux), fb.eri3c(si.orb, si.aux)
    if call == "grad":
        energy, dC, d3, dV = fb.grad(s["MO"], nocc, si.H, si.Enuc, want_3c=True, want_metric=True, out3=s["d3"],
                                     outV=s["dV"])
        return np.float64(energy), dC, d3, dV
    core, act = _spaces(case, s["n"], nocc)
    MO = s["MO"]
    if call == "casscf":
        active = np.ascontiguousarray(MO[core:core + act])
        Dc = MO[:core].T @ MO[:core]
        aa, J, K = fb.calc_2el_mo_ints_ri(Dc, MO, active, active, core, act)
        return (aa, J, K, fb.mo_ints_aaag(MO, core, act)) + fb.soscf_hess_ints(MO, core, act)
    return fb.mo_calc(MO, core, act, s["n"] - core - act)


def _spaces(case, n, nocc):
    """(core, active) orbitals: the active ones half occupied, around the Fermi level."""
    act = min(case["active"], n - nocc, 2 * nocc)
    return nocc - act // 2, act


def work(case):
    n, na, o = _sizes(case)
    pairs, square = n * (n + 1) // 2, n * n
    call = case["call"]
    build = 4 * pairs * na + 2 * square * o * na + n * (n + 1) * o * na
    tensor = 8 * pairs * na
    matrices = 8 * (3 * square + o * n)
    if call in ("fock_host", "fock_device"):
        return {"bytes": tensor // (2 if case["precision"] == "mixed" else 1) + matrices, "flops": build}
    if call == "scf":
        return {"bytes": SCF_BUILDS * (tensor + matrices), "flops": SCF_BUILDS * (build + 10 * n ** 3)}
    if call == "setup":
        return {"bytes": 2 * tensor + 16 * na * na + matrices, "flops": 2 * na * na * pairs + 11 * na ** 3 + build}
    if call == "eri3c":
        return {"bytes": tensor + 8 * na * na, "flops": 100 * pairs * na}
    if call == "grad":
        return {"bytes": 2 * tensor + 16 * na * na, "flops": build + (4 * o * o * n + 2 * pairs * o) * na + 4 * pairs * na * na + 4 * na ** 3}
    core, act = _spaces(case, n, o)
    if call == "casscf":
        half = 2 * square * act * na
        out = 8 * (act ** 4 + n * act ** 3 + 2 * n * act * act + 2 * square)
        all_pairs = 4 * square * n * na  # (pp|Q) of every orbital
        return {"bytes": tensor + out, "flops": build * core // max(o, 1) + half + 2 * square * act * na + all_pairs}
    vac = n - core - act
    out = (core * core + vac * core + act * act + core * act + vac * act) * na
    return {"bytes": tensor + 8 * out, "flops": 2 * square * (core + act) * na + 2 * n * out}


# ------------------------------------------------------- the same in 64 bits, in plain torch ----
# Integrals over Gaussians by Hermite expansion (McMurchie and Davidson, J. Comput. Phys. 26, 218 (1978)), the Boys
# function by Gauss-Legendre quadrature; every contraction as a plain matrix product.

def _carts(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _odd(k):
    return math.prod(range(k, 0, -2)) if k > 0 else 1


def _hermites(l):
    return [(t, u, k - t - u) for k in range(l + 1) for t in range(k + 1) for u in range(k - t + 1)]


def _harmonics(l):
    """Real solid harmonics m = -l .. l over the Cartesian functions, unit norm: (2l + 1) x carts."""
    index = {c: i for i, c in enumerate(_carts(l))}
    rows = []
    for m in range(-l, l + 1):
        a, row = abs(m), [0.0] * len(index)
        for k in range((l - a) // 2 + 1):  # r^2k z^(l-2k-a) of the associated Legendre part
            f = (-1) ** k * math.comb(l, k) * math.comb(2 * l - 2 * k, l) * math.perm(l - 2 * k, a)
            for i in range(a + 1):  # (x + iy)^a: even powers of iy for m >= 0, odd ones for m < 0
                if (i % 2 == 1) != (m < 0):
                    continue
                g = f * math.comb(a, i) * (-1) ** (i // 2)
                for p in range(k + 1):
                    for q in range(k - p + 1):
                        h = g * math.factorial(k) // (math.factorial(p) * math.factorial(q) * math.factorial(k - p - q))
                        row[index[(a - i + 2 * p, i + 2 * q, l - a - 2 * k + 2 * (k - p - q))]] += h
        norm = 0.0
        for c, v in zip(_carts(l), row):
            for d, w in zip(_carts(l), row):
                if not any((x + y) % 2 for x, y in zip(c, d)):
                    norm += v * w * math.prod(_odd(x + y - 1) for x, y in zip(c, d))
        rows.append([v / math.sqrt(norm / _odd(2 * l - 1)) for v in row])
    return torch.tensor(rows, dtype=torch.float64, device="cuda")


def _primitives(shells):
    """{l: (shell numbers, centres, exponents, coefficients)} of all primitives, and the shells' first functions."""
    by, first, at = {}, [], 0
    for i, sh in enumerate(shells):
        raw = [c * math.sqrt((4 * a) ** sh.l * (2 * a / math.pi) ** 1.5 / _odd(2 * sh.l - 1)) for a, c in zip(sh.exps, sh.coefs)]
        s = sum(x * y * _odd(2 * sh.l - 1) / (2 * (a + b)) ** sh.l * (math.pi / (a + b)) ** 1.5
                for a, x in zip(sh.exps, raw) for b, y in zip(sh.exps, raw))
        by.setdefault(sh.l, []).extend((i, *sh.center, a, c / math.sqrt(s)) for a, c in zip(sh.exps, raw))
        first.append(at)
        at += 2 * sh.l + 1
    table = {}
    for l, rows in by.items():
        t = torch.tensor(rows, dtype=torch.float64, device="cuda")
        table[l] = (t[:, 0].long(), t[:, 1:4], t[:, 4], t[:, 5])
    return table, torch.tensor(first, device="cuda"), at


def _expansion(la, lb, p, pa, pb, scale):
    """Hermite coefficients [functions a, functions b, hermite, primitive pair] of products of two primitives."""
    one = []
    for d in range(3):
        E = {(0, 0, 0): scale if d == 0 else torch.ones_like(p)}
        zero = torch.zeros_like(p)
        get = lambda i, j, t: E.get((i, j, t), zero)  # noqa: E731
        for i in range(la + 1):
            for j in range(lb + 1):
                for t in range(i + j + 1):
                    if i + j:
                        k, x = ((i - 1, j), pa) if i else ((i, j - 1), pb)
                        E[i, j, t] = get(*k, t - 1) / (2 * p) + x[:, d] * get(*k, t) + (t + 1) * get(*k, t + 1)
        one.append(E)
    h = {k: i for i, k in enumerate(_hermites(la + lb))}
    H = torch.zeros(len(_carts(la)), len(_carts(lb)), len(h), len(p), dtype=torch.float64, device="cuda")
    for i, a in enumerate(_carts(la)):
        for j, b in enumerate(_carts(lb)):
            for t in range(a[0] + b[0] + 1):
                for u in range(a[1] + b[1] + 1):
                    for v in range(a[2] + b[2] + 1):
                        H[i, j, h[t, u, v]] = one[0][a[0], b[0], t] * one[1][a[1], b[1], u] * one[2][a[2], b[2], v]
    return torch.einsum("xi,yj,ijhn->xyhn", _harmonics(la), _harmonics(lb), H)


def _boys(top, T):
    x, w = np.polynomial.legendre.leggauss(48)
    small, far = T.clamp(max=60.0), T.clamp(min=60.0)
    F = [None] * (top + 1)
    F[top] = sum(0.5 * wi * (0.5 * (1 + xi)) ** (2 * top) * torch.exp(-small * (0.5 * (1 + xi)) ** 2) for xi, wi in zip(x, w))
    e, ef = torch.exp(-small), torch.exp(-far)
    for m in range(top, 0, -1):
        F[m - 1] = (2 * small * F[m] + e) / (2 * m - 1)
    G = 0.5 * torch.sqrt(math.pi / far)
    for m in range(top + 1):
        F[m] = torch.where(T > 60.0, G, F[m])
        G = ((2 * m + 1) * G - ef) / (2 * far)
    return F


def _coulomb(bra, ket_shells, out, first_a, first_b, mirror):
    """out[mu, nu, P] += (ab|P) for the primitive pairs in bra: {(la, lb): (a, b, p, centre, pa, pb, scale)}."""
    kets, first_k, _ = _primitives(ket_shells)
    for (la, lb), (a, b, p, P, pa, pb, scale) in bra.items():
        H, hb = _expansion(la, lb, p, pa, pb, scale), _hermites(la + lb)
        na, nb = H.shape[:2]
        for lc, (k, C, g, c) in kets.items():
            zero = torch.zeros(len(g), 3, dtype=torch.float64, device="cuda")
            G, hk = _expansion(lc, 0, g, zero, zero, c)[:, 0], _hermites(lc)
            L = la + lb + lc
            index = {x: i for i, x in enumerate(_hermites(L))}
            step = max(1, int(6e7 // (len(index) * 2 + (2 * lc + 1) * len(hb)) // len(g)))
            cols = (first_k[k][:, None] + torch.arange(2 * lc + 1, device="cuda")).reshape(-1)
            for s in range(0, len(p), step):
                q = slice(s, s + step)
                pq, gq = p[q, None], g[None]
                al = pq * gq / (pq + gq)
                X = [P[q, d][:, None] - C[None, :, d] for d in range(3)]
                F = _boys(L, al * (X[0] ** 2 + X[1] ** 2 + X[2] ** 2))
                R = {}
                for m in range(L, -1, -1):
                    new = {(0, 0, 0): (-2 * al) ** m * F[m]}
                    for t in _hermites(L - m)[1:]:
                        d = next(i for i in range(3) if t[i])
                        low = tuple(v - (i == d) for i, v in enumerate(t))
                        new[t] = X[d] * R[low]
                        if t[d] > 1:
                            new[t] = new[t] + (t[d] - 1) * R[tuple(v - 2 * (i == d) for i, v in enumerate(t))]
                    R = new
                pref = 2 * math.pi ** 2.5 / (pq * gq * torch.sqrt(pq + gq))
                W = torch.zeros(2 * lc + 1, len(hb), *pref.shape, dtype=torch.float64, device="cuda")
                for i, y in enumerate(hk):
                    shifted = torch.stack([R[tuple(u + v for u, v in zip(x, y))] for x in hb])
                    W += (-1) ** sum(y) * G[:, i][:, None, None, :] * shifted
                val = torch.einsum("xyhn,chnk->nxykc", H[..., q], W * pref)
                mu = first_a[a[q]][:, None, None] + torch.arange(na, device="cuda")[None, :, None]
                nu = first_b[b[q]][:, None, None] + torch.arange(nb, device="cuda")[None, None, :]
                row = (mu * out.shape[1] + nu).reshape(-1)
                rows, inverse = torch.unique(row, return_inverse=True)
                part = torch.zeros(len(rows), out.shape[2], dtype=torch.float64, device="cuda")
                wide = torch.zeros(len(row), out.shape[2], dtype=torch.float64, device="cuda")
                wide.index_add_(1, cols, val.reshape(len(row), -1))
                part.index_add_(0, inverse, wide)
                out.view(-1, out.shape[2])[rows] += part
    if mirror:  # pairs of shells a > b were formed once
        for P in range(0, out.shape[2], 256):
            block = out[:, :, P:P + 256]
            low = torch.tril(torch.ones(out.shape[:2], dtype=torch.bool, device="cuda"))[:, :, None]
            out[:, :, P:P + 256] = torch.where(low, block, block.transpose(0, 1))


def _integrals(si):
    """(P|Q) and the full square (mu nu|P)."""
    orb, first, n = _primitives(si.orb.shells)
    pairs = {}
    for la, (i, A, ea, ca) in orb.items():
        for lb, (j, B, eb, cb) in orb.items():
            x, y = torch.where(i[:, None] >= j[None])
            a, b = ea[x], eb[y]
            p = a + b
            r = A[x] - B[y]
            scale = ca[x] * cb[y] * torch.exp(-a * b / p * (r * r).sum(1))
            keep = scale.abs() > 1e-22
            x, y, a, b, p, scale = (v[keep] for v in (x, y, a, b, p, scale))
            if len(p):
                P = (a[:, None] * A[x] + b[:, None] * B[y]) / p[:, None]
                pairs[la, lb] = (i[x], j[y], p, P, P - A[x], P - B[y], scale)
    aux, first_x, na = _primitives(si.aux.shells)
    I3 = torch.zeros(n, n, na, dtype=torch.float64, device="cuda")
    _coulomb(pairs, si.aux.shells, I3, first, first, True)
    V = torch.zeros(na, 1, na, dtype=torch.float64, device="cuda")
    single = {(l, 0): (i, torch.zeros_like(i), e, C, torch.zeros_like(C), torch.zeros_like(C), c) for l, (i, C, e, c) in aux.items()}
    _coulomb(single, si.aux.shells, V, first_x, torch.zeros(1, dtype=torch.long, device="cuda"), False)
    V = V[:, 0]
    return 0.5 * (V + V.T), I3


def _jk(B, D, C):
    """J and K from B[Q][mu][nu] and the orbital rows C."""
    J = torch.einsum("qmn,q->mn", B, torch.einsum("qmn,mn->q", B, D))
    X = torch.matmul(C, B).transpose(0, 1).reshape(len(C), -1, B.shape[2]).reshape(-1, B.shape[2])
    return J, X.T @ X


def _rhf(B, H, S, D, R, nocc):
    """Converged energy (without the nuclei) and density, by DIIS."""
    w, U = torch.linalg.eigh(S)
    X = U * w.rsqrt()
    J, K = _jk(B, D, R)
    F = H + 2 * J - K
    Fs, es, best = [], [], (math.inf, None, None)
    for _ in range(60):
        C = X @ torch.linalg.eigh(X.T @ F @ X)[1][:, :nocc]
        D = C @ C.T
        J, K = _jk(B, D, C.T.contiguous())
        F = H + 2 * J - K
        e = X.T @ (F @ D @ S - S @ D @ F) @ X
        off = float(e.abs().max())
        if off < best[0]:
            best = (off, float((D * (F + H)).sum()), D)
        if off < 1e-11 or (off > 2 * best[0] and best[0] < 1e-9):
            break
        Fs, es = (Fs + [F])[-8:], (es + [e])[-8:]
        m = len(es)
        A = -torch.ones(m + 1, m + 1, dtype=torch.float64, device="cuda")
        A[m, m] = 0
        for i in range(m):
            for j in range(m):
                A[i, j] = (es[i] * es[j]).sum()
        scale = float(A[:m, :m].diagonal().max())
        A[:m, :m] /= scale
        b = torch.zeros(m + 1, dtype=torch.float64, device="cuda")
        b[m] = -1
        c = torch.linalg.lstsq(A.cpu(), b.cpu()[:, None], driver="gelsd").solution[:m, 0]
        F = sum(float(x) * f for x, f in zip(c, Fs))
    return best[1], best[2]


def exact(case, seed):
    n, na, nocc = _sizes(case)
    if n * n * na > 5e8:  # the integrals alone would take too long
        return None
    s = _input(case, seed)
    si, call = s["si"], case["call"]
    V, I3 = _integrals(si)
    pairs = torch.tril_indices(n, n, device="cuda")
    if call == "eri3c":
        return V, I3[pairs[0], pairs[1]]
    w, U = torch.linalg.eigh(V)
    M = (U * w.rsqrt()) @ U.T
    B = (I3.reshape(n * n, na) @ M).T.contiguous().reshape(na, n, n)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    if call in ("fock_host", "fock_device"):
        return _jk(B, dev(s["D"]), dev(s["MO"][:nocc]))
    if call == "setup":
        return _jk(B, dev(s["D0"]), dev(s["R"]))
    if call == "scf":
        energy, D = _rhf(B, dev(si.H), dev(si.S), dev(s["D0"]), dev(s["R"]), nocc)
        return np.float64(energy + si.Enuc), D
    if call == "grad":
        C, D, H = dev(s["MO"][:nocc]), dev(s["D"]), dev(si.H)
        J, K = _jk(B, D, C)
        F = H + 2 * J - K
        Z = (M @ B.reshape(na, -1)).reshape(na, n, n)  # V^-1 (P|mu nu)
        Gamma = 4 * torch.einsum("qmn,mn->q", Z, D)[:, None, None] * D - 2 * C.T @ (C @ Z @ C.T) @ C
        d3 = Gamma[:, pairs[0], pairs[1]].T * torch.where(pairs[0] == pairs[1], 1.0, 2.0)[:, None]
        dV = -0.5 * Gamma.reshape(na, -1) @ Z.reshape(na, -1).T
        return np.float64(float((D * (F + H)).sum()) + si.Enuc), 4 * C @ F, d3, dV
    core, act = _spaces(case, n, nocc)
    MO = dev(s["MO"])
    A = MO[core:core + act]
    if call == "casscf":
        J, K = _jk(B, MO[:core].T @ MO[:core], MO[:core]) if core else (torch.zeros_like(B[0]), torch.zeros_like(B[0]))
        T = MO @ B @ A.T                      # (x v|Q) as [Q][x][v]
        Y = T[:, core:core + act]             # (t u|Q)
        aa = torch.einsum("qab,qcd->badc", Y.transpose(1, 2), Y.transpose(1, 2)).reshape(act * act, act * act)
        aaag = torch.einsum("qtu,qxv->tuvx", Y, T).reshape(act ** 3, n)
        diagonal = torch.einsum("pm,qpm->qp", MO, MO @ B)
        hess_J = torch.einsum("qp,qtu->ptu", diagonal, Y).reshape(n, act * act)
        hess_K = torch.einsum("qpt,qpu->ptu", T, T).reshape(n, act * act)
        return aa, J, K, aaag, hess_J, hess_K
    spaces = {"C": MO[:core], "A": A, "V": MO[core + act:]}
    block = lambda x, y: (spaces[x] @ B @ spaces[y].T).permute(1, 2, 0).reshape(-1, na)  # noqa: E731
    return {name: block(*name) for name in ("CC", "VC", "AA", "CA", "VA")}
