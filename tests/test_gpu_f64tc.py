"""The FP64 form's tensor-core contractions (vxc_f64tc.cu) at the sizes where their tiles end: AO counts
around the 32-AO K blocks, the 64-AO accumulation groups, the 48-column and 128-row tiles and the
1024-AO change of the integer sums' unit, one count beyond the kernel's 2048 (the SIMT form), partial
batches, and rows of zeros.

Bound: every contraction of k terms carries at most ~2^-53 per term of the operands' largest product (slice
rounding and the products left out; the SIMT form's FMA chain alike), T over m AOs and V over 128 points:
(m + 128) 2^-53 of the largest magnitude, times 50 for the functional's conditioning.
"""

import numpy as np
import pytest

from calchem_gb300 import BasisSet, GridLevel, MolecularGrid, RksVxcEngine, UksVxcEngine
from calchem_gb300.molecule import Atom, Molecule
from tests.helpers import oracle_basis

pytestmark = pytest.mark.gpu


def hydrogens(n):
    """n hydrogens (n AOs in STO-3G) on a slightly irregular cubic lattice, 1.3 Bohr apart."""
    k = int(np.ceil(n ** (1.0 / 3.0)))
    ijk = np.array([(a, b, c) for a in range(k) for b in range(k) for c in range(k)][:n], dtype=float)
    return Molecule([Atom.from_bohr("H", 1.3 * p + 0.1 * np.sin(3.0 * p + i)) for i, p in enumerate(ijk)],
                    charge=n % 2, multiplicity=1)


def points(mol, n, seed):
    rng = np.random.default_rng(seed)
    x = mol.coords_bohr[rng.integers(0, len(mol), n)] + rng.normal(size=(n, 3))
    xyzw = np.concatenate([x, rng.uniform(1e-3, 0.2, (n, 1))], axis=1)
    return MolecularGrid(xyzw, xyzw[:, 3], np.zeros(n, np.int32), GridLevel.COARSE)


def density(n, seed):
    rng = np.random.default_rng(seed)
    a = rng.normal(size=(n, max(2, n // 3))) / np.sqrt(n)
    p = a @ a.T + 0.01 * np.eye(n)
    p[n // 2] = p[:, n // 2] = 0.0  # a row of zeros
    return p


@pytest.mark.parametrize("n", [1, 31, 33, 48, 49, 64, 65, 96, 97, 128, 129, 145, 257, 1023, 1026, 2050])
def test_rks_and_uks_at_tile_edges(native_lib, oracle, n):
    mol = hydrogens(n)
    basis = BasisSet.from_name("sto-3g", mol)
    assert basis.n_ao == n
    grid = points(mol, 300 if n > 300 else 700, n)
    ob, og = oracle_basis(oracle, "sto-3g", mol), oracle.Grid.from_points(grid.xyzw)
    P, Pb = density(n, n + 1), 0.4 * density(n, n + 2)
    tol = 50.0 * (n + 128) * 2.0 ** -53
    eng = RksVxcEngine(basis, grid, batching="reference")
    for _ in range(2):  # the pass that fills the AO cache and one that reads it
        exc, V = eng.evaluate(basis, grid, "b3lyp", P)
        e, ne, Vr = oracle.vxc_rks_points(ob, og, P, "b3lyp")
        assert np.max(np.abs(V - Vr)) <= tol * np.max(np.abs(Vr))
        assert abs(exc - e) <= tol * abs(e) and abs(eng.last_nelec - ne) <= tol * abs(ne)
        assert np.array_equal(V, V.T)
    eng.close()
    eng = UksVxcEngine(basis, grid, batching="reference")
    exc, Va, Vb = eng.evaluate(basis, grid, "pbe", P, Pb)
    e, _, _, Var, Vbr = oracle.vxc_uks_points(ob, og, P, Pb, "pbe")
    eng.close()
    assert abs(exc - e) <= tol * abs(e)
    for v, r in ((Va, Var), (Vb, Vbr)):
        assert np.max(np.abs(v - r)) <= tol * np.max(np.abs(r))
