"""The FP64 forms on either side of the rules that choose between the tensor cores (vxc_f64tc.cu, xc_grad_f64tc.cu) and
the SIMT kernels (vxc_fp64.cu, xc_grad.cu): atom and AO counts where the gradient changes over, memory budgets that
leave no room for the tensor-core form's scratch, numbers that are not finite, and rows of widely differing entries.

Error of an integer-slice product (f64_slices.cuh), per term and relative to the product of the two operand rows'
largest entries: 2 x 2^-53 from rounding the operands to 53 bits at their row's largest entry; 20 x 2^-54 at most from
the slice products left out (five of i + j = 6, each up to 2^16 where the rows' largest digits multiply to 2^14 at
least); 12 x 2^-54 from the last accumulator's FP32 additions (24 per 64 terms, each within two units of 2^-36).  So
9 x 2^-52 covers it.  AO values from different exp functions agree to 100 x 2^-52 here (exponents up to ~40).
"""

import numpy as np
import pytest

from calchem_gb300 import BasisSet, GpuVxcGrid, RksVxcEngine, _native, workloads
from tests.helpers import distorted_water, make_positive_density, oracle_basis, reference_layout
from tests.test_gpu_becke_grad import check, scattered
from tests.test_gpu_f64tc import density, hydrogens, points

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52
SLICE = 9 * EPS
AO = 100 * EPS


@pytest.mark.parametrize("n", [256, 257])
def test_gradient_on_both_sides_of_256_atoms(native_lib, oracle, n):
    mol = hydrogens(n)
    check(oracle, mol, "sto-3g", density(n, n + 5), scattered(mol, 300, n))


@pytest.mark.parametrize("waters,basis_name,low,high", [(60, "6-31g(d)", 1025, 2048), (85, "6-31g(d,p)", 2049, 1 << 30)])
@pytest.mark.parametrize("closed", [True, False])
def test_gradient_with_long_contractions(native_lib, oracle, waters, basis_name, low, high, closed):
    """Above 1024 AOs (the integer sums' unit changes) and above 2048 (the SIMT form)."""
    mol = workloads.water_cluster(waters, waters)
    basis = BasisSet.from_name(basis_name, mol)
    grid = scattered(mol, 260, waters)
    pa, pb = density(basis.n_ao, 5), 0.5 * density(basis.n_ao, 6)
    eng = RksVxcEngine(basis, grid, batching="reference")
    assert low <= eng.plan_stats()[3] <= high
    g = eng.nuclear_gradient(mol, grid, "pbe", pa, None if closed else pb)
    eng.close()
    og = oracle.Grid.from_points(grid.xyzw, grid.host_atom, grid.raw_weight)
    ref = oracle.xc_gradient(oracle_basis(oracle, basis_name, mol), og, mol.z, mol.coords_bohr, pa, pa if closed else pb,
                             "pbe")
    assert np.max(np.abs(g - ref)) <= 1e-10 * max(1.0, np.max(np.abs(ref)))


class Grid:
    """A reference-layout upload with a memory budget and quadrature weights; limit=None: the least accepted, which
    leaves the FP64 tensor-core form no room."""

    def __init__(self, basis, layout, limit):
        self.lib, self.n = _native.load(), basis.n_ao
        pts, w, off, cs = layout

        def up(lim):
            return GpuVxcGrid.upload(*basis.gpu_arrays(), pts, off, cs, basis.n_ao, memory_limit=lim)
        if limit is None:
            lo, limit = 0, 1 << 36  # (the least is kept as self.limit)
            while limit - lo > 1:
                mid = (lo + limit) // 2
                try:
                    up(mid).release()
                    limit = mid
                except _native.CalchemXcError as e:
                    assert e.code == -3
                    lo = mid
        self.grid, self.limit = up(limit), limit
        _native.check("weights", self.lib.calchem_xc_set_weights(self.grid.grid_id, _native.ptr(w), len(w)))

    def launches(self):
        return self.lib.calchem_xc_last_launch_count(self.grid.grid_id)

    def evaluate(self, P, Pb=None, func=3):
        p, gid = _native.ptr, self.grid.grid_id
        exc, ne, va, vb = np.zeros(1), np.zeros(2), np.zeros((self.n, self.n)), np.zeros((self.n, self.n))
        if Pb is None:
            _native.check("rks", self.lib.calchem_xc_evaluate_rks(gid, func, 0, p(P), p(exc), p(ne), p(va)))
        else:
            _native.check("uks", self.lib.calchem_xc_evaluate_uks(gid, func, 0, p(P), p(Pb), p(exc), p(ne), p(va), p(vb)))
        return exc, ne, va, vb

    def fxc(self, P, trials, triplet):
        p, gid = _native.ptr, self.grid.grid_id
        _native.check("prepare", self.lib.calchem_xc_fxc_prepare(gid, 3, p(P)))
        out = np.zeros_like(trials)
        _native.check("fxc", self.lib.calchem_xc_fxc_contract(gid, triplet, p(trials), len(trials), p(out)))
        return out

    def release(self):
        self.grid.release()


@pytest.fixture(scope="module")
def water(native_lib):
    mol = distorted_water()
    basis = BasisSet.from_name("6-31g(d)", mol)
    layout = reference_layout(basis, points(mol, 900, 3))
    simt, tc = Grid(basis, layout, None), Grid(basis, layout, 1 << 36)
    yield basis, layout, simt, tc
    simt.release()
    tc.release()


def test_budget_without_room_for_the_scratch(water):
    """Every FP64 evaluation in both forms; the bound of tests/test_gpu_f64tc.py."""
    basis, _, simt, tc = water
    n = basis.n_ao
    P = make_positive_density(n, 7)
    rng = np.random.default_rng(4)
    trials = 0.02 * rng.normal(size=(3, n, n))
    trials += trials.transpose(0, 2, 1)
    wv = rng.normal(size=(tc.grid.n_pts, 4))
    tol = 50.0 * (n + 128) * 2.0 ** -53
    close = lambda a, b: np.max(np.abs(a - b)) <= tol * np.max(np.abs(b))  # noqa: E731
    for Pb in (None, 0.4 * make_positive_density(n, 8)):
        a, b = simt.evaluate(P, Pb), tc.evaluate(P, Pb)
        assert (simt.launches(), tc.launches()) == (2, 3)
        assert all(close(x, y) for x, y in zip(a, b))
    assert close(simt.grid.eval_rho_grad(P), tc.grid.eval_rho_grad(P))
    assert (simt.launches(), tc.launches()) == (1, 2)
    a, b = simt.grid.accumulate_vxc(wv), tc.grid.accumulate_vxc(wv)
    assert (simt.launches(), tc.launches()) == (1, 2)
    assert close(a, b) and not np.any(np.triu(a, 1)) and not np.any(np.triu(b, 1))
    for triplet in (0, 1):
        a, b = simt.fxc(P, trials, triplet), tc.fxc(P, trials, triplet)
        assert (simt.launches(), tc.launches()) == (1 + len(trials), 3 * len(trials))
        assert close(a, b) and np.array_equal(b, b.transpose(0, 2, 1))


def test_budgets_with_room_for_part_of_the_scratch(water):
    """From one CTA's scratch to all of them: the SIMT form up to a quarter of its own CTAs, then fewer CTAs."""
    basis, layout, simt, tc = water
    P = make_positive_density(basis.n_ao, 7)
    ref = tc.evaluate(P)
    tol = 50.0 * (basis.n_ao + 128) * 2.0 ** -53
    seen = []
    for extra in [0] + [2 ** k for k in range(16, 25)]:
        g = Grid(basis, layout, simt.limit + extra)
        for _ in range(2):
            assert all(np.max(np.abs(a - b)) <= tol * np.max(np.abs(b)) for a, b in zip(g.evaluate(P), ref))
        seen.append(g.launches())
        g.release()
    assert seen[0] == 2 and seen[-1] == 3 and seen == sorted(seen)


def test_force_call_at_its_least_limit(native_lib):
    """Half as many CTAs, or fewer, as without a limit: the same bits, as each batch has its own row of sums."""
    mol = distorted_water()
    basis = BasisSet.from_name("6-31g(d)", mol)
    g = Grid(basis, reference_layout(basis, points(mol, 40000, 3)), 1 << 36)
    P = make_positive_density(basis.n_ao, 7)
    w = np.random.default_rng(4).normal(size=(g.grid.n_pts, 8))
    free = g.grid.eval_grad_force(P, 0.5 * P, False, w, 3, memory_limit=1 << 36)
    lo, hi = 1, 1 << 36
    while hi - lo > 1:
        mid = (lo + hi) // 2
        try:
            g.grid.eval_grad_force(P, 0.5 * P, False, w, 3, memory_limit=mid)
            hi = mid
        except _native.CalchemXcError as e:
            assert e.code == -3
            lo = mid
    assert np.array_equal(g.grid.eval_grad_force(P, 0.5 * P, False, w, 3, memory_limit=hi), free)
    g.release()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_numbers_that_are_not_finite(water, bad):
    """They show in the results wherever the SIMT form's show them, and the next call's results are clean."""
    basis, _, simt, tc = water
    n = basis.n_ao
    P = make_positive_density(n, 7)
    B = P.copy()
    B[3, 5] = B[5, 3] = bad
    wv = np.random.default_rng(4).normal(size=(tc.grid.n_pts, 4))
    wb = wv.copy()
    wb[200] = bad
    calls = {"rks": lambda g, p, w: g.evaluate(p), "uks": lambda g, p, w: g.evaluate(P, p),
             "uks alpha": lambda g, p, w: g.evaluate(p, P), "rho": lambda g, p, w: (g.grid.eval_rho_grad(p),),
             "accum": lambda g, p, w: (g.grid.accumulate_vxc(w),)}
    for name, call in calls.items():
        bad_simt, bad_tc = call(simt, B, wb), call(tc, B, wb)
        assert not all(np.all(np.isfinite(x)) for x in bad_tc), name
        for a, b in zip(bad_simt, bad_tc):
            assert np.all(np.isfinite(a) | ~np.isfinite(b)), name
        assert all(np.all(np.isfinite(x)) for x in call(tc, P, wv)), name


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("closed", [True, False])
def test_gradient_of_a_density_that_is_not_finite(native_lib, bad, closed):
    """Every component: each atom's weight derivative takes in every point."""
    mol = distorted_water()
    basis = BasisSet.from_name("6-31g(d)", mol)
    grid = scattered(mol, 500, 3)
    P = make_positive_density(basis.n_ao, 7)
    B = P.copy()
    B[3, 5] = B[5, 3] = bad
    eng = RksVxcEngine(basis, grid)
    assert not np.any(np.isfinite(eng.nuclear_gradient(mol, grid, "b3lyp", B, None if closed else P)))
    assert np.all(np.isfinite(eng.nuclear_gradient(mol, grid, "b3lyp", P, None if closed else P)))
    eng.close()


def aos(ob, layout):
    """phi and its gradient at the layout's points, [4][points][AOs]."""
    pts = layout[0]
    v = np.asarray(ob.ao_grad(np.stack([pts["x"], pts["y"], pts["z"]], axis=1)))
    return np.moveaxis(v, [i for i, s in enumerate(v.shape) if s == 4][-1], 0).astype(np.longdouble)


@pytest.mark.parametrize("decades", [0, 12, 40])
def test_rows_of_widely_differing_entries(water, oracle, decades):
    """Densities, trial potentials and points graded over many orders of magnitude: in the tensor-core form an entry's
    error is relative to the largest products of its rows, in the SIMT form to its own terms; both within the bounds
    at the head of this file."""
    basis, layout, simt, tc = water
    n = basis.n_ao
    s = 10.0 ** (-decades * np.arange(n) / (n - 1.0))
    P = s[:, None] * make_positive_density(n, 7) * s[None]
    phi = aos(oracle_basis(oracle, "6-31g(d)", distorted_water()), layout)
    assert phi.shape == (4, tc.grid.n_pts, n)
    T = phi[0] @ P.T.astype(np.longdouble)
    ref = np.stack([(1 if k == 0 else 2) * (phi[k] * T).sum(1) for k in range(4)], axis=1)
    mag = np.abs(phi)
    own = mag[0] @ np.abs(P).T
    row = n * SLICE * np.abs(P).max(1)[None] * mag[0].max(1)[:, None]
    for g in (simt, tc):
        rg = g.grid.eval_rho_grad(P)
        for k in range(4):
            bound = 2 * (mag[k] * ((row if g is tc else 0.0) + (2 * AO + n * EPS) * own)).sum(1)
            assert np.all(np.abs(rg[:, k] - ref[:, k]) <= bound)
    wv = np.random.default_rng(4).normal(size=(tc.grid.n_pts, 4))
    wv *= 10.0 ** (-decades * (np.arange(len(wv)) % 128) / 127.0)[:, None]
    Z = sum(wv[:, k, None] * phi[k] for k in range(4))
    W = Z.T @ phi[0]
    Zm = sum(np.abs(wv[:, k, None]) * mag[k] for k in range(4))
    own = Zm.T @ mag[0]
    row = len(wv) * SLICE * np.outer(Zm.max(0), mag[0].max(0))
    for g in (simt, tc):
        bound = (row if g is tc else 0.0) + (2 * AO + len(wv) * EPS) * own
        v = g.grid.accumulate_vxc(wv)
        assert np.all(np.abs(v - np.tril(W + W.T)) <= np.tril(bound + bound.T))


def test_drop_in_calls_above_2048_aos(native_lib, oracle):
    n = 2050
    mol = hydrogens(n)
    basis = BasisSet.from_name("sto-3g", mol)
    layout = reference_layout(basis, points(mol, 200, n))
    g = Grid(basis, layout, 1 << 36)
    assert np.max(np.diff(layout[2])) == n  # (one AO per shell)
    P = density(n, 3)
    phi = aos(oracle_basis(oracle, "sto-3g", mol), layout).astype(float)
    T = phi[0] @ P.T
    ref = np.stack([(1 if k == 0 else 2) * (phi[k] * T).sum(1) for k in range(4)], axis=1)
    wv = np.random.default_rng(4).normal(size=(g.grid.n_pts, 4))
    W = sum(wv[:, k, None] * phi[k] for k in range(4)).T @ phi[0]
    tol = 50.0 * (n + 128) * 2.0 ** -53
    rg, v = g.grid.eval_rho_grad(P), g.grid.accumulate_vxc(wv)
    assert g.launches() == 1
    assert np.max(np.abs(rg - ref)) <= tol * np.max(np.abs(ref))
    assert np.max(np.abs(v - np.tril(W + W.T))) <= tol * np.max(np.abs(W))
    g.release()
