"""Performance cases of the integral-direct Cholesky ERI library.

Each case is one call sequence that a program of this package makes, on the
seeded molecules of ``molecules.py`` (the same shell recipes, atom densities
and thresholds as the benchmark configurations):

* ``job``: decomposition (chol_gammcor_Rkpq) and AO->MO transformation, from
  the smallest molecule of the many-molecule configuration to the f-shell
  recipe of the flagship configuration at the largest size whose pass stays
  near a second; stored Rkpq or direct transformation, host or device output,
  full-range or range-separated operator, all accuracy levels of production.
* ``transform``: the AO->MO transformation of another orbital block on a
  decomposition that the program keeps.
* ``batch``: many small molecules in one call, then their transformations.
* ``coulomb``: Coulomb energy with its nuclear gradient and Coulomb matrix
  through the autograd function.
* ``eri``: all (pq|rs) of a small molecule, into a caller's device buffer
  (the entry point that allocates nothing) or into host memory.
* ``inverse``: Cholesky factor and its inverse at the size of a pivot block.

The Cholesky vectors of two correct implementations differ: pivots whose
residual diagonals are equal by symmetry (the components of a shell at its own
atom) are taken in an order that rounding decides.  So the jobs return what
the vectors stand for, the whole block of MO integrals (ia|jb) = R^T R.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import gammcor_pkg

gammcor_pkg.load()
from gammcor_integrals_b200 import _capi, basis, molecules  # noqa: E402
from gammcor_integrals_b200 import cholesky_gammcor as cg  # noqa: E402
from gammcor_integrals_b200 import coulomb_grad as cgrad  # noqa: E402

# recipe -> shells, primitives per shell, exponent range (the configurations' own)
RECIPES = {"spd": (molecules.RECIPE_C1, (3, 3), (0.1, 1.0e3)),
           "spdf": (molecules.RECIPE_C2, (3, 6), (0.05, 5.0e3))}
TAU = {1: 1e-5, 2: 1e-6, 3: 1e-7}


def _cube(recipe, atoms, spread):
    """Edge of the cube: the many-molecule and small configurations use 8 bohr
    whatever the atom count ("packed"), the others a fixed atom density."""
    if spread == "packed":
        return 8.0
    return 12.0 * (atoms / 20.0) ** (1 / 3) if recipe == "spd" else 16.0 * (atoms / 40.0) ** (1 / 3)


def _molecule(case, seed, atoms=None):
    atoms = atoms or case["atoms"]
    shells, nprim, exps = RECIPES[case["recipe"]]
    cube = max(_cube(case["recipe"], atoms, case.get("spread", "density")), 2.5 * atoms ** (1 / 3))
    return molecules.random_molecule(seed, atoms, cube, shells, nprim, exps, TAU.get(case.get("accuracy", 2), 1e-6))


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # smallest molecule of the many-molecule configuration, the reference's own call sequence
        # (Rkpq stored and copied to the host, then Rkab): launches and host work count
        dict(name="job_42ao_stored", kind="job", recipe="spd", spread="packed", atoms=3, accuracy=1, omega=0.0,
             stored=True, output="host", occ=6, virt=18, buffer_mb=0),
        # the small configuration whole: 140 AOs, tau = 1e-6, 20 x 60 orbitals
        dict(name="job_140ao", kind="job", recipe="spd", spread="packed", atoms=10, accuracy=2, omega=0.0,
             stored=False, output="host", occ=20, virt=60, buffer_mb=0),
        # f shells, range-separated operator, the tightest production accuracy, stored vectors
        dict(name="job_90ao_f_omega", kind="job", recipe="spdf", spread="density", atoms=3, accuracy=3, omega=0.4,
             stored=True, output="host", occ=9, virt=41, buffer_mb=64),
        # the flagship recipe (f shells, 3-6 primitives, tau = 1e-6) at its atom density, the largest
        # molecule whose pass stays below two seconds
        dict(name="job_240ao_f", kind="job", recipe="spdf", spread="density", atoms=8, accuracy=2, omega=0.0,
             stored=False, output="device", occ=12, virt=180, buffer_mb=0),
        # another orbital block on a kept decomposition: the full-dimension integrals again
        dict(name="transform_210ao_f", kind="transform", recipe="spdf", spread="density", atoms=7, accuracy=1,
             omega=0.0, stored=False, output="device", occ=11, virt=60, buffer_mb=256),
        # many small molecules in one call
        dict(name="batch_8_molecules", kind="batch", recipe="spd", spread="packed", molecules=8, atoms_lo=3,
             atoms_hi=10, accuracy=1, omega=0.0, streams=16, occ=4, virt=20),
        # energy + nuclear gradient + Coulomb matrix, small and at the gradient configuration's size
        dict(name="coulomb_42ao", kind="coulomb", recipe="spd", spread="density", atoms=3, omega=0.0),
        dict(name="coulomb_280ao", kind="coulomb", recipe="spd", spread="density", atoms=20, omega=0.0),
        # all ERIs of a small molecule
        dict(name="eri_42ao_noalloc", kind="eri", recipe="spd", spread="packed", atoms=3, omega=0.0,
             output="device"),
        dict(name="eri_60ao_f", kind="eri", recipe="spdf", spread="density", atoms=2, omega=0.0, output="host"),
        # V_JJ of a few hundred AOs: Cholesky factor and its inverse
        dict(name="inverse_4001", kind="inverse", n=4001),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["job", "job", "job", "transform", "batch", "coulomb", "eri", "inverse"])
    omega = rng.choice([0.0, 0.0, round(rng.uniform(0.2, 1.0), 3)])
    if kind == "inverse":
        return dict(kind=kind, n=_log(rng, 130, 4001))
    if kind == "coulomb":
        return dict(kind=kind, recipe="spd", spread="density", atoms=_log(rng, 2, 19), omega=omega)
    recipe = rng.choice(["spd", "spdf"])
    if kind == "eri":
        device = recipe == "spd" and rng.random() < 0.5
        return dict(kind=kind, recipe=recipe, spread="density", atoms=rng.randint(1, 4 if recipe == "spd" else 2),
                    omega=omega, output="device" if device else "host")
    if kind == "batch":
        lo = rng.randint(2, 4)
        return dict(kind=kind, recipe="spd", spread="packed", molecules=rng.randint(2, 8), atoms_lo=lo,
                    atoms_hi=rng.randint(lo, 9), accuracy=rng.choice([1, 2]), omega=omega,
                    streams=rng.choice([0, 4, 16]), occ=rng.randint(2, 5), virt=rng.randint(7, 20))
    if recipe == "spd":
        atoms, spread = _log(rng, 2, 12), rng.choice(["packed", "density"])
        nao = 14 * atoms
    else:
        atoms, spread = _log(rng, 1, 7), "density"
        nao = 30 * atoms
    occ = rng.randint(1, max(1, nao // 10))
    virt = rng.randint(2, max(2, min(nao - occ, nao // 2, 1200 // occ)))
    stored = kind == "job" and nao <= 150 and rng.random() < 0.5
    return dict(kind=kind, recipe=recipe, spread=spread, atoms=atoms, accuracy=rng.choice([1, 2, 2, 3]), omega=omega,
                stored=stored, output=rng.choice(["host", "device"]), occ=occ, virt=virt,
                buffer_mb=rng.choice([0, 0, 64, 256]))


# ---------------------------------------------------------------- inputs
def _orbitals(nao, seed):
    """Orthonormal NAO x NAO coefficients, column-major host array and its device copy."""
    c = molecules.mo_coefficients(nao, seed)
    return c, torch.from_numpy(np.ascontiguousarray(c.T)).cuda()


def _lib_stream():
    s = C.c_void_p()
    _capi.check(_capi.lib().gci_get_stream(C.byref(s)))
    return torch.cuda.ExternalStream(s.value)


def _density(nao, seed):
    """X X^T with X ~ N(0, 0.1^2), NAO x 30: the density of the gradient configuration."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = 0.1 * torch.randn(nao, 30, dtype=torch.float64, device="cuda", generator=g)
    return x @ x.T


def _spd(n, seed):
    """SPD matrix with the spectrum of a pivot block: positive entries of decaying weight and a
    condition number of about 1e6."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    w = torch.logspace(0, -3, n, dtype=torch.float64, device="cuda")
    q = q * w
    a = q @ q.T / n
    return a + 1e-6 * torch.diag(torch.diagonal(a))


def prepare(case, seed):
    kind = case["kind"]
    _capi.check(_capi.lib().gci_init())
    st = dict(case=case, stream=_lib_stream())
    if kind == "inverse":
        st["a"] = _spd(case["n"], seed)
        st["x"] = torch.empty_like(st["a"])
        return st
    if kind == "batch":
        lo, hi, n = case["atoms_lo"], case["atoms_hi"], case["molecules"]
        atoms = [lo + (i * (hi - lo)) // max(n - 1, 1) for i in range(n)]
        st["bases"] = [basis.from_molecule(_molecule(case, 1000 * seed + i, a)) for i, a in enumerate(atoms)]
        st["mo"] = [_orbitals(b.NAO, seed + i)[0] for i, b in enumerate(st["bases"])]
        return st
    tb = st["basis"] = basis.from_molecule(_molecule(case, seed))
    nao = tb.NAO
    if kind == "coulomb":
        st["density"] = _density(nao, seed).requires_grad_()
        st["coords"] = torch.from_numpy(np.ascontiguousarray(tb.AtomCoords.T)).cuda().requires_grad_()
    elif kind == "eri":
        npq = nao * (nao + 1) // 2
        st["struct"] = tb.c_struct()
        if case["output"] == "device":
            st["out"] = torch.empty(npq, npq, dtype=torch.float64, device="cuda")
        else:
            st["out"] = np.zeros((npq, npq), order="F")
    else:
        st["mo"], st["mo_dev"] = _orbitals(nao, seed + 1)
        if kind == "transform":
            st["vecs"] = _decompose(st)
    return st


# ---------------------------------------------------------------- one pass
def _decompose(st):
    c = st["case"]
    return cg.chol_gammcor_Rkpq(st["basis"], c["accuracy"], c["omega"] or None, materialize=c["stored"],
                                copy_to_host=c["stored"])


def _transform(st, vecs):
    """Rkab of the occupied x virtual block, as a (NA NB, NVecs) tensor on the GPU."""
    c = st["case"]
    occ, virt = c["occ"], c["virt"]
    if c["output"] == "host":
        r = cg.chol_gammcor_Rkab(st["mo"], 1, occ, st["mo"], occ + 1, occ + virt, c["buffer_mb"], vecs, st["basis"])
        return torch.from_numpy(r.T).cuda()
    nao, nvecs = st["basis"].NAO, vecs.Chol2Data.NVecs
    r = torch.empty(occ * virt, nvecs, dtype=torch.float64, device="cuda")
    # the library's stream waits for what this program's stream still does with the buffer
    st["stream"].wait_stream(torch.cuda.current_stream())
    mo = C.c_void_p(st["mo_dev"].data_ptr())
    _capi.check(_capi.lib().gci_rkab_device(vecs.handle.ptr, mo, nao, 1, occ, mo, nao, occ + 1, occ + virt,
                                            c["buffer_mb"], _capi.GCI_PREC_FP64, C.c_void_p(r.data_ptr())))
    return r


def run(st):
    case = st["case"]
    kind = case["kind"]
    lib = _capi.lib()
    if kind in ("job", "transform"):
        vecs = st["vecs"] if kind == "transform" else _decompose(st)
        r = _transform(st, vecs)
        return {"iajb": r @ r.T}
    if kind == "batch":
        occ, virt = case["occ"], case["virt"]
        all_vecs = cg.chol_gammcor_Rkpq_batch(st["bases"], case["accuracy"], case["omega"] or None,
                                              materialize=False, copy_to_host=False, nstreams=case["streams"])
        out = []
        for tb, mo, vecs in zip(st["bases"], st["mo"], all_vecs):
            r = cg.chol_gammcor_Rkab(mo, 1, occ, mo, occ + 1, occ + virt, 0, vecs, tb)
            r = torch.from_numpy(r.T).cuda()
            out.append(r @ r.T)
        return out
    if kind == "coulomb":
        e = cgrad.coulomb_energy(st["coords"], st["density"], st["basis"], case["omega"])
        grad, jmat = torch.autograd.grad(e, (st["coords"], st["density"]))
        return {"energy": e.detach(), "gradient": grad, "coulomb": jmat}
    if kind == "eri":
        out, s = st["out"], st["struct"]
        if case["output"] == "device":
            stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
            _capi.check(lib.gci_eri_pairs_noalloc(C.byref(s), case["omega"], C.c_void_p(out.data_ptr()),
                                                  out.shape[0], stream))
        else:
            _capi.check(lib.gci_eri_pairs(C.byref(s), case["omega"], _capi.ptr(out), out.shape[0]))
        return out
    n = case["n"]
    a = st["a"].clone()          # the factor overwrites the matrix
    st["stream"].wait_stream(torch.cuda.current_stream())
    _capi.check(lib.gci_cholesky_inverse(n, C.c_void_p(a.data_ptr()), n, C.c_void_p(st["x"].data_ptr())))
    # column-major lower triangles: the row-major views are upper triangular
    return {"factor": a.triu(), "inverse": st["x"]}


# ---------------------------------------------------------------- work of one pass
def _herm(n):
    return (n + 1) * (n + 2) * (n + 3) // 6


def _pair_work(recipe, atoms, vectors):
    """Multiply-adds of the Hermite-matrix products and of the R recursion for every shell pair
    against `vectors` columns spread evenly over the pairs: sums over the pair classes with the
    mean primitive count of the recipe."""
    shells, (lo, hi), _ = RECIPES[recipe]
    prims = (0.5 * (lo + hi)) ** 2
    count = {}
    ls = [l for _ in range(atoms) for l in shells]
    by_l = {l: ls.count(l) for l in set(ls)}
    for a in by_l:
        for b in by_l:
            if b <= a:
                count[a + b] = count.get(a + b, 0) + (by_l[a] * by_l[b] if a != b else by_l[a] * (by_l[a] + 1) // 2)
    funcs = sum(2 * l + 1 for l in ls)
    npairs, npq = sum(count.values()), funcs * (funcs + 1) // 2
    bra = sum(n * prims * _herm(L) for L, n in count.items())
    ket = sum(n * prims * _herm(L) for L, n in count.items()) / npairs
    return 2.0 * bra * ket * vectors, npq


def work(case):
    kind = case["kind"]
    if kind == "inverse":
        n = case["n"]
        return {"bytes": 8.0 * 2.0 * n * n, "flops": 2.0 * n ** 3 / 3.0}
    if kind == "batch":
        tot = dict(bytes=0.0, flops=0.0)
        lo, hi, n = case["atoms_lo"], case["atoms_hi"], case["molecules"]
        for i in range(n):
            atoms = lo + (i * (hi - lo)) // max(n - 1, 1)
            one = work(dict(case, kind="job", atoms=atoms, stored=False))
            tot = {k: tot[k] + one[k] for k in tot}
        return tot
    atoms = case["atoms"]
    shells, (lo, hi), _ = RECIPES[case["recipe"]]
    nao = atoms * sum(2 * l + 1 for l in shells)
    npq = nao * (nao + 1) // 2
    if kind == "coulomb":
        one, _ = _pair_work(case["recipe"], atoms, 1.0)
        npairs = (atoms * len(shells)) * (atoms * len(shells) + 1) / 2
        # every primitive quartet, each bra level raised by one for the derivatives
        return {"bytes": 8.0 * 3 * nao * nao, "flops": 2.0 * one * npairs}
    if kind == "eri":
        flops, _ = _pair_work(case["recipe"], atoms, npq / 2.0)
        return {"bytes": 8.0 * npq * npq, "flops": flops}
    # about 11 vectors per AO at 1e-6, one AO-sized step per decade
    vectors = min(npq, nao * {1: 9.0, 2: 11.0, 3: 13.0}[case["accuracy"]])
    nab = case["occ"] * case["virt"]
    eri, _ = _pair_work(case["recipe"], atoms, vectors)
    passes = 1 if kind == "transform" else 2         # pivot columns, full dimension
    dense = 0.0 if kind == "transform" else vectors ** 2 * npq / 2.0 + 2.0 * vectors ** 3 / 3.0
    tomo = vectors ** 2 * nab + 2.0 * vectors * nao * case["occ"] * (nao + case["virt"])
    if case.get("stored"):
        dense += vectors ** 2 * npq
        tomo -= vectors ** 2 * nab
    return {"bytes": 8.0 * (2 * nao * nao + vectors * nab + nab * nab), "flops": passes * eri + dense + tomo}


def tolerance(case):
    """About four times what other orders of the same FP64 sums show.

    ERIs, energies and gradients are sums of a few thousand FP64 terms (measured
    against the 64-bit values below: 1e-13, 5e-14 and 5e-11).  The jobs' MO
    integrals agree to 1e-14 .. 1e-12 between two kernel families that take the
    same pivots, but they carry the decomposition's truncation (residual
    diagonals up to tau remain), and where pivots of equal diagonal change places
    that moves: up to 8e-7 of the integrals seen at tau = 1e-6.  It is absolute,
    and range-separated integrals are ten times smaller and more."""
    kind = case["kind"]
    if kind == "eri":
        return {"rel": 1e-12, "max": 1e-10}
    if kind == "coulomb":
        return {"rel": 2e-10, "max": 1e-8}
    if kind == "inverse":
        return {"rel": 3e-9, "max": 1e-6}
    rel = {1: 4e-5, 2: 4e-6, 3: 4e-7}[case["accuracy"]] * (10.0 if case["omega"] else 1.0)
    return {"rel": rel, "max": 10.0 * rel}


# ---------------------------------------------------------------- 64-bit values
# A plain McMurchie-Davidson evaluation in torch: Hermite expansion of every function pair,
# Hermite Coulomb integrals by the full recursion, blocks of primitive quartets at a time.
def _solid_harmonics(l):
    """Unnormalised real solid harmonics, rows m = -l..l, columns (x, y, z) powers with x then y
    descending (Helgaker, Jorgensen, Olsen 6.4.47); the Cartesian components themselves below d."""
    powers = [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]
    if l < 2:
        return powers, np.eye(len(powers))
    u = np.zeros((2 * l + 1, len(powers)))
    for m in range(-l, l + 1):
        am, odd = abs(m), 1 if m < 0 else 0
        for t in range((l - am) // 2 + 1):
            for k in range(t + 1):
                for v in range((am - odd) // 2 + 1):
                    tv = 2 * v + odd
                    c = (-1.0) ** (t + v) * 0.25 ** t * math.comb(l, t) * math.comb(l - t, am + t) * math.comb(t, k)
                    c *= math.comb(am, tv)
                    u[m + l, powers.index((2 * t + am - 2 * k - tv, 2 * k + tv, l - 2 * t - am))] += c
    return powers, u


def _shell_table(mol):
    """Per shell: atom, l, exponents, and coefficients (nfunc, nprim, ncart) of unit-normalised functions."""
    odd = lambda n: math.prod(range(n, 0, -2)) if n > 0 else 1  # noqa: E731
    out, loc = [], 0
    for atom, l, e, c in mol.shells:
        e, c = np.asarray(e, float), np.asarray(c, float) * np.asarray(e, float) ** ((2 * l + 3) / 4.0)
        powers, u = _solid_harmonics(l)
        p = e[:, None] + e[None, :]
        radial = float((c[:, None] * c[None, :] * (math.pi / p) ** 1.5 / (2.0 * p) ** l).sum())
        s = np.array([[0.0 if any((a[i] + b[i]) % 2 for i in range(3)) else
                       math.prod(odd(a[i] + b[i] - 1) for i in range(3)) for b in powers] for a in powers])
        norm = 1.0 / np.sqrt(np.einsum("mi,ij,mj->m", u, s, u) * radial)
        out.append(dict(atom=atom, l=l, e=e, t=norm[:, None] * u, c=c, loc=loc, n=len(u)))
        loc += len(u)
    return out, loc


def _tuv(n):
    return [(t, u, k - t - u) for k in range(n + 1) for t in range(k, -1, -1) for u in range(k - t, -1, -1)]


def _expansion(la, lb, a, b, ab):
    """E[i][j][t] along one axis: (x - A)^i (x - B)^j e^{..} = sum_t E Lambda_t, without the overlap factor."""
    p = a + b
    pa, pb = -b / p * ab, a / p * ab
    e = [[[None] * (i + j + 1) for j in range(lb + 1)] for i in range(la + 1)]
    zero = torch.zeros_like(p)
    get = lambda i, j, t: e[i][j][t] if 0 <= t <= i + j else zero  # noqa: E731
    e[0][0][0] = torch.ones_like(p)
    for i in range(la + 1):
        for j in range(lb + 1):
            if i == j == 0:
                continue
            x, (i0, j0) = (pa, (i - 1, j)) if i > 0 else (pb, (i, j - 1))
            for t in range(i + j + 1):
                e[i][j][t] = get(i0, j0, t - 1) / (2 * p) + x * get(i0, j0, t) + (t + 1) * get(i0, j0, t + 1)
    return e


def _pair_groups(mol, coords):
    """Shell pairs (A >= B, the second shell outermost) grouped by (lA, lB): for the primitive
    pairs of a group, exponent sum p, centre, Hermite expansion (n, nA, nB, H), the pair's
    first AOs and its position in the list of pairs."""
    shells, nao = _shell_table(mol)
    dev = coords.device
    groups, loc = {}, 0
    for ib, sb in enumerate(shells):
        for ia in range(ib, len(shells)):
            sa = shells[ia]
            g = groups.setdefault((sa["l"], sb["l"]), [])
            for ea, ca in zip(sa["e"], sa["c"]):
                for eb, cb in zip(sb["e"], sb["c"]):
                    g.append((ea, eb, ca * cb, ia, ib, loc))
            loc += sa["n"] * sb["n"] if ia != ib else sa["n"] * (sa["n"] + 1) // 2
    f64 = dict(dtype=torch.float64, device=dev)
    out = []
    for (la, lb), g in sorted(groups.items()):
        num = torch.tensor([r[:3] for r in g], **f64)
        idx = torch.tensor([r[3:] for r in g], device=dev)
        at = torch.tensor([s["atom"] for s in shells], device=dev)
        a, b, c = num[:, 0], num[:, 1], num[:, 2]
        ra, rb = coords[at[idx[:, 0]]], coords[at[idx[:, 1]]]
        # products far below the rounding of any integral are left out
        keep = (c.abs() * torch.exp(-a * b / (a + b) * ((ra - rb) ** 2).sum(1)) > 1e-24).nonzero()[:, 0]
        a, b, c, idx, ra, rb = a[keep], b[keep], c[keep], idx[keep], ra[keep], rb[keep]
        p = a + b
        ax = [_expansion(la, lb, a, b, (ra - rb)[:, k]) for k in range(3)]
        k0 = c * torch.exp(-a * b / p * ((ra - rb) ** 2).sum(1))
        pw_a, pw_b = _solid_harmonics(la)[0], _solid_harmonics(lb)[0]
        ta = torch.tensor(np.array([s["t"] if s["l"] == la else np.zeros((1, 1)) for s in shells if s["l"] == la]), **f64)
        tb = torch.tensor(np.array([s["t"] for s in shells if s["l"] == lb]), **f64)
        pos_a = {i: k for k, i in enumerate(i for i, s in enumerate(shells) if s["l"] == la)}
        pos_b = {i: k for k, i in enumerate(i for i, s in enumerate(shells) if s["l"] == lb)}
        sel_a = torch.tensor([pos_a.get(i, 0) for i in range(len(shells))], device=dev)[idx[:, 0]]
        sel_b = torch.tensor([pos_b.get(i, 0) for i in range(len(shells))], device=dev)[idx[:, 1]]
        cols = []
        for t, u, v in _tuv(la + lb):
            rows = []
            for xa in pw_a:
                for xb in pw_b:
                    if t > xa[0] + xb[0] or u > xa[1] + xb[1] or v > xa[2] + xb[2]:
                        rows.append(torch.zeros_like(p))
                    else:
                        rows.append(ax[0][xa[0]][xb[0]][t] * ax[1][xa[1]][xb[1]][u] * ax[2][xa[2]][xb[2]][v])
            m = torch.stack(rows, 1).reshape(-1, len(pw_a), len(pw_b)) * k0[:, None, None]
            cols.append(torch.einsum("nic,njd,ncd->nij", ta[sel_a], tb[sel_b], m))
        h = torch.stack(cols, -1) if len(p) else torch.zeros(0, ta.shape[1], tb.shape[1], _herm(la + lb), **f64)
        first = torch.tensor([s["loc"] for s in shells], device=dev)
        centre = (a[:, None] * ra + b[:, None] * rb) / p[:, None]
        out.append(dict(L=la + lb, p=p, r=centre, h=h, fa=first[idx[:, 0]], fb=first[idx[:, 1]], same=idx[:, 0] == idx[:, 1],
                        loc=idx[:, 2]))
    return out, nao


_BOYS = {}


def _boys_table(dev):
    """F_m at x = 0, 0.05 .. 36, m = 0..34: the all-positive series for the highest order, then downwards."""
    if dev not in _BOYS:
        x = torch.arange(0, 721, dtype=torch.float64, device=dev) * 0.05
        top = 34
        term = torch.full_like(x, 1.0 / (2 * top + 1))
        total = term.clone()
        for i in range(1, 260):
            term = term * 2 * x / (2 * top + 2 * i + 1)
            total = total + term
        f = [total * torch.exp(-x)]
        for m in range(top, 0, -1):
            f.insert(0, (2 * x * f[0] + torch.exp(-x)) / (2 * m - 1))
        _BOYS[dev] = torch.stack(f)
    return _BOYS[dev]


def _boys(n, x):
    tab = _boys_table(x.device)
    xs = x.clamp(max=35.9)
    j = (xs * 20 + 0.5).long()
    d = j.to(x.dtype) * 0.05 - xs
    f = tab[n + 7][j] / 7
    for k in range(6, -1, -1):
        f = tab[n + k][j] + d * (f if k == 6 else f / (k + 1))
    out, ex = [f], torch.exp(-xs)
    for m in range(n, 0, -1):
        out.insert(0, (2 * xs * out[0] + ex) / (2 * m - 1))
    far = x > 35.9
    if bool(far.any()):
        xf = x.clamp(min=1.0)
        g, ef = 0.5 * torch.sqrt(math.pi / xf), torch.exp(-xf)
        for m in range(n + 1):
            out[m] = torch.where(far, g, out[m])
            g = ((2 * m + 1) * g - ef) / (2 * xf)
    return out


def _hermite_coulomb(n, p, rp, q, rq, kappa):
    """{(t, u, v): R_tuv times the prefactor} for t + u + v <= n, tensors (len p, len q)."""
    p, q = p[:, None], q[None, :]
    d = [rp[:, None, k] - rq[None, :, k] for k in range(3)]
    den = p + q + kappa * p * q
    alpha = p * q / den
    f = _boys(n, alpha * (d[0] ** 2 + d[1] ** 2 + d[2] ** 2))
    pre = 2.0 * math.pi ** 2.5 / (p * q * torch.sqrt(den))
    cur = {}
    for j in range(n, -1, -1):
        new = {(0, 0, 0): f[j] * pre * (-2.0 * alpha) ** j}
        for t, u, v in _tuv(n - j)[1:]:
            k = 0 if t else 1 if u else 2
            c = [t, u, v]
            c[k] -= 1
            r = d[k] * cur[tuple(c)]
            if c[k] > 0:
                m = c[k]
                c[k] -= 1
                r = torch.add(r, cur[tuple(c)], alpha=m)
            new[(t, u, v)] = r
        cur = new
    return cur


def _levels(groups, vectors):
    """Concatenate the groups of each Hermite level; vectors[g] is (n, H, columns)."""
    out = {}
    for g, x in zip(groups, vectors):
        out.setdefault(g["L"], []).append((g["p"], g["r"], x))
    return {L: tuple(torch.cat([y[k] for y in v]) for k in range(3)) for L, v in out.items() if sum(len(y[0]) for y in v)}


def _potential(levels, kappa, raise_bra=0):
    """V[L] (n, H(L + raise), columns): the potential of the Hermite vectors at every primitive pair."""
    out = {}
    for L1, (p, rp, _) in levels.items():
        bra = _tuv(L1 + raise_bra)
        v = torch.zeros(len(p), len(bra), next(iter(levels.values()))[2].shape[2], dtype=p.dtype, device=p.device)
        for L2, (q, rq, x) in levels.items():
            ket = _tuv(L2)
            sign = torch.tensor([(-1.0) ** sum(g) for g in ket], dtype=p.dtype, device=p.device)
            xk = (x * sign[None, :, None]).transpose(0, 1).reshape(-1, x.shape[2])      # (H2 n2, columns)
            step = max(1, int(6e5 / len(q)))
            for c0 in range(0, len(p), step):
                r = _hermite_coulomb(L1 + raise_bra + L2, p[c0:c0 + step], rp[c0:c0 + step], q, rq, kappa)
                for k, (t, u, w) in enumerate(bra):
                    m = torch.cat([r[(t + a, u + b, w + c)] for a, b, c in ket], 1)
                    v[c0:c0 + step, k] += m @ xk
        out[L1] = v
    return out


def _function_pairs(g, build):
    """Sum over the function pairs of a group: build(i, j) gives (weights (n, columns)); diagonal
    pairs are counted once."""
    n, na, nb, H = g["h"].shape
    cols = None
    for i in range(na):
        for j in range(nb):
            w = build(i, j)
            cols = torch.zeros(n, H, w.shape[1], dtype=w.dtype, device=w.device) if cols is None else cols
            cols += g["h"][:, i, j, :, None] * w[:, None, :]
    return cols


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "inverse":
        a = _spd(case["n"], seed)
        l = torch.linalg.cholesky(a)
        x = torch.linalg.solve_triangular(l, torch.eye(case["n"], dtype=a.dtype, device=a.device), upper=False)
        return {"factor": l.T.contiguous(), "inverse": x.T.contiguous()}
    if kind == "batch":
        lo, hi, n = case["atoms_lo"], case["atoms_hi"], case["molecules"]
        out = []
        for i in range(n):
            atoms = lo + (i * (hi - lo)) // max(n - 1, 1)
            one = dict(case, kind="job", atoms=atoms, stored=False)
            out.append(_mo_integrals(one, _molecule(case, 1000 * seed + i, atoms), seed + i, dev)
                       if atoms <= 10 else None)
        return out
    omega = case["omega"]
    kappa = 1.0 / omega ** 2 if omega else 0.0
    mol = _molecule(case, seed)
    coords = torch.tensor(mol.atoms, dtype=torch.float64, device=dev)
    if kind in ("job", "transform"):
        # primitive pairs x Hermite indices, squared, times the orbital pairs
        if work(dict(case, kind="eri"))["flops"] / (0.5 * mol.nao * (mol.nao + 1) / 2) * \
                _npairs(mol) * case["occ"] * case["virt"] > 4e14:
            return None
        return {"iajb": _mo_integrals(case, mol, seed + 1, dev)}
    if kind == "eri":
        groups, nao = _pair_groups(mol, coords)
        npq = nao * (nao + 1) // 2
        vecs = []
        for g in groups:
            na, nb = g["h"].shape[1:3]

            def build(i, j):
                w = torch.zeros(len(g["p"]), npq, dtype=torch.float64, device=dev)
                at = g["loc"] + torch.where(g["same"], j * na - j * (j - 1) // 2 + (i - j), i + na * j)
                use = ~g["same"] | torch.tensor(i >= j, device=dev)
                w[torch.arange(len(w), device=dev)[use], at[use]] = 1.0
                return w

            vecs.append(_function_pairs(g, build))
        levels = _levels(groups, vecs)
        pot = _potential(levels, kappa)
        out = sum(levels[L][2].reshape(-1, npq).T @ pot[L].reshape(-1, npq) for L in levels)
        return out if case["output"] == "device" else out.cpu().numpy().T
    # Coulomb energy, gradient and matrix: potentials once, derivatives of the expansions by autograd
    dens = _density(mol.nao, seed).requires_grad_()
    coords.requires_grad_()
    groups, nao = _pair_groups(mol, coords)
    sym = 0.5 * (dens + dens.T)
    vecs = []
    for g in groups:
        twice = torch.where(g["same"], 1.0, 2.0).to(torch.float64)
        ia = g["fa"][:, None, None] + torch.arange(g["h"].shape[1], device=dev)[None, :, None]
        ib = g["fb"][:, None, None] + torch.arange(g["h"].shape[2], device=dev)[None, None, :]
        vecs.append((torch.einsum("nijh,nij->nh", g["h"], sym[ia, ib]) * twice[:, None])[:, :, None])
    with torch.no_grad():
        levels = _levels([{**g, "p": g["p"].detach(), "r": g["r"].detach()} for g in groups], [v.detach() for v in vecs])
        pot = _potential(levels, kappa, 1)
    live = _levels(groups, vecs)
    energy, total = 0.0, 0.0
    for L, (p, r, h) in live.items():
        bra = _tuv(L + 1)
        at = {c: k for k, c in enumerate(bra)}
        low = [at[c] for c in _tuv(L)]
        v = pot[L][:, :, 0]
        energy = energy + 0.5 * (h[:, :, 0] * v[:, low]).sum().detach()
        total = total + (h[:, :, 0] * v[:, low]).sum()
        for k in range(3):
            up = [at[tuple(c[i] + (i == k) for i in range(3))] for c in _tuv(L)]
            total = total + ((h[:, :, 0].detach() * v[:, up]).sum(1) * r[:, k]).sum()
    grad, jmat = torch.autograd.grad(total, (coords, dens))
    return {"energy": energy, "gradient": grad, "coulomb": jmat}


def _npairs(mol):
    return mol.nshells * (mol.nshells + 1) // 2


def _mo_integrals(case, mol, mo_seed, dev):
    omega, occ, virt = case["omega"], case["occ"], case["virt"]
    coords = torch.tensor(mol.atoms, dtype=torch.float64, device=dev)
    groups, nao = _pair_groups(mol, coords)
    c = torch.tensor(np.ascontiguousarray(molecules.mo_coefficients(nao, mo_seed)), dtype=torch.float64, device=dev)
    co, cv = c[:, :occ], c[:, occ:occ + virt]
    vecs = []
    for g in groups:
        def build(i, j):
            p, q = g["fa"] + i, g["fb"] + j
            w = cv[q][:, :, None] * co[p][:, None, :]            # column = a + occ * b: a fastest
            w = w + torch.where(g["same"], 0.0, 1.0)[:, None, None] * cv[p][:, :, None] * co[q][:, None, :]
            return w.reshape(len(w), -1)

        vecs.append(_function_pairs(g, build))
    levels = _levels(groups, vecs)
    pot = _potential(levels, 1.0 / omega ** 2 if omega else 0.0)
    n = occ * virt
    return sum(levels[L][2].reshape(-1, n).T @ pot[L].reshape(-1, n) for L in levels)
