"""GPU tests of the Hermite-matrix ERI kernels at the edges of their blocking:
primitive-pair counts below, at and above the row blocks (16, 8, 4, 2 and 1
primitive pairs) and column groups (4, 2, 1) of every Hermite level.

Reference: the class kernels (gci_eri_hm(0)), an independent evaluation.
Tolerance: both sum the same FP64 products of each integral, at most a few
thousand terms no larger than the largest integral's, in different orders:
1e-12 of the largest integral (the bound of the ERI parity tests).
"""
import ctypes as C
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from gammcor_integrals_b200 import _capi, basis as gbasis, molecules

pytestmark = pytest.mark.gpu


def _eri_pairs(lib, tb, omega, hm):
    npq = tb.NAO * (tb.NAO + 1) // 2
    out = np.full((npq, npq), np.nan, order="F")
    s = tb.c_struct()
    before = lib.gci_eri_hm(1 if hm else 0)
    try:
        _capi.check(lib.gci_eri_pairs(C.byref(s), omega, _capi.ptr(out), npq))
    finally:
        lib.gci_eri_hm(before)
    return out


@pytest.mark.parametrize("nprim,omega", [((1, 1), 0.0), ((2, 2), 0.0), ((1, 3), 0.5), ((3, 5), 0.0), ((6, 7), 0.0)])
def test_blocks_and_groups_match_class_kernels(gpu_lib, nprim, omega):
    # 1, 4, 1..9, 9..25 and 36..49 primitive pairs a shell pair before the screen
    mol = molecules.random_molecule(31, 2, 4.0, (0, 1, 2, 3), nprim, (0.1, 50.0))
    tb = gbasis.from_molecule(mol)
    got, ref = _eri_pairs(gpu_lib, tb, omega, True), _eri_pairs(gpu_lib, tb, omega, False)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))


def test_parts_and_pairs_without_primitives(gpu_lib):
    """Few long tasks (36 primitive pairs a side), which run in parts that are added up, among
    them pairs of steep shells on distant atoms that keep no primitive pair and leave no part."""
    mol = molecules.random_molecule(32, 2, 6.0, (0, 1, 3), (6, 6), (0.1, 5.0))
    steep = molecules.random_molecule(33, 2, 6.0, (0, 2), (2, 2), (200.0, 2000.0))
    atoms = np.array([[0.0, 0.0, 0.0], [5.0, 1.0, 0.5]])
    shells = sorted(mol.shells + steep.shells, key=lambda s: s[0])
    tb = gbasis.from_molecule(molecules.Molecule(atoms=atoms, shells=shells))
    got, ref = _eri_pairs(gpu_lib, tb, 0.0, True), _eri_pairs(gpu_lib, tb, 0.0, False)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
    # one block of each two pairs is evaluated and mirrored: exactly symmetric (the block of a pair
    # with itself is evaluated whole)
    n = [2 * s[1] + 1 for s in shells]
    sizes = [n[A] * n[B] if A != B else n[A] * (n[A] + 1) // 2 for B in range(len(n)) for A in range(B, len(n))]
    pair = np.repeat(np.arange(len(sizes)), sizes)
    other = pair[:, None] != pair[None, :]
    assert np.array_equal(got[other], got.T[other])
    # the parts are added in a fixed order: the same bits again
    assert np.array_equal(got, _eri_pairs(gpu_lib, tb, 0.0, True))


@pytest.mark.parametrize("nprim", [(2, 3), (5, 6)])
def test_noalloc_on_both_sides_of_its_scratch(gpu_lib, nprim):
    """The allocation-free ERI matrix: vectors that fit its scratch (Hermite-matrix kernels) and
    vectors that do not (class kernels), against gci_eri_pairs."""
    import torch
    tb = gbasis.from_molecule(molecules.random_molecule(34, 1, 4.0, molecules.RECIPE_C2, nprim, (0.1, 50.0)))
    npq = tb.NAO * (tb.NAO + 1) // 2
    out = torch.full((npq, npq + 5), float("nan"), dtype=torch.float64, device="cuda")
    s = tb.c_struct()
    stream = torch.cuda.current_stream()
    _capi.check(gpu_lib.gci_eri_pairs_noalloc(C.byref(s), 0.3, C.c_void_p(out.data_ptr()), npq + 5,
                                              C.c_void_p(stream.cuda_stream)))
    got, ref = out.cpu().numpy().T, _eri_pairs(gpu_lib, tb, 0.3, True)
    assert np.max(np.abs(got[:npq] - ref)) <= 1e-12 * np.max(np.abs(ref))
    assert np.all(got[npq:] == 0.0)


KEPT = """
import gammcor_pkg; gammcor_pkg.load()
import torch
from gammcor_integrals_b200 import basis, molecules, cholesky_gammcor as cg
tb = basis.from_molecule(molecules.random_molecule(61, 2, 5.9, molecules.RECIPE_C2, (3, 6), (0.05, 5e3)))
kept, free = [], []
for i in range(12):
    kept.append(cg.chol_gammcor_Rkpq(tb, 2, None, materialize=False, copy_to_host=False))
    free.append(torch.cuda.mem_get_info()[0])
print((free[1] - free[11]) / 10 / 2**20)
"""


def test_decompositions_do_not_keep_the_parts(gpu_lib):
    """Device memory a kept decomposition of 60 AOs with f shells adds, in MB, in a process of its own
    (the library's pool grows in steps of 32 MB): 45 to 48 with its inverse, Hermite vectors and column
    data; the parts of four streams would double it (96)."""
    root = Path(__file__).resolve().parent.parent
    out = subprocess.run([sys.executable, "-c", KEPT], cwd=root, check=True, capture_output=True, text=True, timeout=300)
    assert float(out.stdout.split()[-1]) < 72.0
