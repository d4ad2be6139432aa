"""Checks of the library's host code that run under the stand-in CUDA runtime (fake_cudart.cpp), one per process:
python host_calls.py <path of the stand-in> <name of a check>."""

import ctypes
import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

from calchem_gb300 import (BasisSet, FxcKernel, GpuVxcGrid, GridLevel, MolecularGrid, RksVxcEngine, UksVxcEngine,  # noqa: E402
                           VxcGroup, _native, workloads)
from tests.helpers import reference_layout  # noqa: E402


def molecule():
    """(molecule, basis, grid of scattered points, density)."""
    mol = workloads.water()
    basis = BasisSet.from_name("6-31g(d)", mol)
    rng = np.random.default_rng(1)
    host = rng.integers(0, 3, 3000).astype(np.int32)
    x = mol.coords_bohr[host] + rng.normal(size=(3000, 3))
    xyzw = np.concatenate([x, rng.uniform(0.1, 1.0, (3000, 1))], axis=1)
    return mol, basis, MolecularGrid(xyzw, xyzw[:, 3], host, GridLevel.COARSE), np.eye(basis.n_ao)


def dropin(basis, grid):
    pts, w, off, cs = reference_layout(basis, grid)
    return GpuVxcGrid.upload(*basis.gpu_arrays(), pts, off, cs, basis.n_ao), w


def check_uploads_come_before_kernels(fake):
    """No kernel is launched while something the legacy stream writes is not known to be done."""
    mol, basis, grid, P = molecule()
    for precision in ("fp64", "mixed"):
        rks = RksVxcEngine(basis, grid, precision=precision, tile=64)
        rks.evaluate(basis, grid, "pbe", P)
        assert fake.fake_unsettled() == 0, precision
        rks.set_point_atoms(grid.host_atom, 3)
        rks.evaluate_with_shares(basis, grid, "pbe", P)
        assert fake.fake_unsettled() == 0, precision
        rks.nuclear_gradient(mol, grid, "pbe", P)
        assert fake.fake_unsettled() == 0, precision
        rks.close()
        uks = UksVxcEngine(basis, grid, precision=precision, tile=64)
        uks.evaluate(basis, grid, "pbe", P, P)
        uks.close()
        fxc = FxcKernel(basis, grid, "pbe", P, precision)
        fxc.contract_batch([P, P])
        fxc.close()
        group = VxcGroup([(basis, grid), (basis, grid)], precision, tile=64)
        group.evaluate_rks("pbe", [P, P])
        group.close()
        assert fake.fake_unsettled() == 0, precision
    g, w = dropin(basis, grid)
    g.eval_rho_grad(P)
    _native.check("set_weights", _native.load().calchem_xc_set_weights(g.grid_id, _native.ptr(w), len(w)))
    g.accumulate_vxc(np.zeros((g.n_pts, 4)))
    assert fake.fake_unsettled() == 0


CHECKS = {k[len("check_"):]: v for k, v in list(globals().items()) if k.startswith("check_")}

if __name__ == "__main__":
    CHECKS[sys.argv[2]](ctypes.CDLL(sys.argv[1]))
