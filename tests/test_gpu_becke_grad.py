"""The Becke weight derivative of the FP64 gradient at the atom counts where its path changes: two atoms, rows
longer than a warp, the largest count with its pair tables in shared memory (becke.cu, 95 atoms) and the first
with them in device memory.  The points are near the atoms, between them and far outside (where
every cell function is small or many are alike); hydrogens, so that the size adjustments vanish, and a
mixed molecule, where they do not.

Bound of the FP64 form against the oracle: its own, 1e-10 Eh/Bohr for a molecule of a few atoms, per unit of
the largest component where that is above one.  The tensor-core form agrees with FP64 on integrated grids
(its AO part's error at single points near a nucleus is larger than any bound of interest here), so it is
held to the FP64 form on water clusters around the same atom counts, within the 5e-9 of large clusters.
"""

import numpy as np
import pytest

from calchem_gb300 import BasisSet, GridLevel, MolecularGrid, RksVxcEngine, workloads
from tests.helpers import oracle_basis
from tests.test_gpu_f64tc import density, hydrogens

pytestmark = pytest.mark.gpu


def scattered(mol, n, seed):
    """Points around the atoms at every distance from 0.01 to 30 Bohr, hosted by the atom they are drawn
    around, with raw weights that fall off as the density does."""
    rng = np.random.default_rng(seed)
    host = rng.integers(0, len(mol), n)
    u = rng.normal(size=(n, 3))
    r = np.exp(rng.uniform(np.log(1e-2), np.log(30.0), n))
    x = mol.coords_bohr[host] + r[:, None] * u / np.linalg.norm(u, axis=1)[:, None]
    raw = rng.uniform(0.1, 1.0, n)
    xyzw = np.concatenate([x, 0.5 * raw[:, None]], axis=1)
    return MolecularGrid(xyzw, raw, host.astype(np.int32), GridLevel.COARSE)


@pytest.mark.parametrize("n", [2, 3, 32, 33, 45, 46, 107])
def test_weight_derivative_at_team_sizes(native_lib, oracle, n):
    mol = hydrogens(n)
    check(oracle, mol, "sto-3g", density(n, n + 5), scattered(mol, 400, n))


@pytest.mark.parametrize("n", [95, 96])
def test_weight_derivative_where_tables_leave_shared_memory(native_lib, oracle, n):
    mol = hydrogens(n)
    check(oracle, mol, "sto-3g", density(n, n + 5), scattered(mol, 200, n))


def test_weight_derivative_with_size_adjustments(native_lib, oracle):
    mol = workloads.water_cluster(5, 5)
    P = workloads.seeded_density_rks(BasisSet.from_name("sto-3g", mol).overlap(), 25, 3)
    check(oracle, mol, "sto-3g", 0.5 * P, scattered(mol, 3000, 7))


@pytest.mark.parametrize("waters", [11, 14])
def test_tensor_core_form_on_both_team_shapes(native_lib, waters):
    mol = workloads.water_cluster(waters, waters)
    basis = BasisSet.from_name("sto-3g", mol)
    grid = MolecularGrid.build_for_basis(mol, basis, GridLevel.COARSE)
    half = 0.5 * workloads.seeded_density_rks(basis.overlap(), 5 * waters, 3)
    g = {}
    for precision in ("fp64", "mixed"):
        eng = RksVxcEngine(basis, grid, precision=precision)
        g[precision] = eng.nuclear_gradient(mol, grid, "pbe", half)
        assert np.array_equal(g[precision], eng.nuclear_gradient(mol, grid, "pbe", half))
        eng.close()
    assert np.max(np.abs(g["mixed"] - g["fp64"])) < 5e-9


@pytest.mark.parametrize("waters", [1, 3, 5, 6, 13, 24, 25])
def test_tensor_core_form_at_its_edges(native_lib, waters):
    """Teams of one, two and eight warps, one to three ranges of a row per atom, the last count with its pair
    tables in shared memory (72 atoms) and the first without."""
    test_tensor_core_form_on_both_team_shapes(native_lib, waters)


def check(oracle, mol, name, half, grid):
    basis = BasisSet.from_name(name, mol)
    eng = RksVxcEngine(basis, grid)
    g = [eng.nuclear_gradient(mol, grid, "b3lyp", half) for _ in range(2)]
    eng.close()
    og = oracle.Grid.from_points(grid.xyzw, grid.host_atom, grid.raw_weight)
    ref = oracle.xc_gradient(oracle_basis(oracle, name, mol), og, mol.z, mol.coords_bohr, half, half, "b3lyp")
    assert np.array_equal(g[0], g[1])  # fixed-order sums
    assert np.max(np.abs(g[0] - ref)) <= 1e-10 * max(1.0, np.max(np.abs(ref)))
