"""Inputs at the edge of what the FP64 forms on the tensor cores (vxc_f64tc.cu, xc_grad_f64tc.cu) accept, where the
SIMT forms they took over from gave plain answers."""

import numpy as np
import pytest

from calchem_gb300 import BasisSet, GpuVxcGrid, RksVxcEngine, _native
from tests.helpers import distorted_water, make_positive_density, reference_layout
from tests.test_gpu_f64tc import points

pytestmark = pytest.mark.gpu


def with_empty_batches(pts, w, off, cs, at):
    """The layout with a batch of five points and no candidate shells before each batch index in `at`."""
    out_p, out_w, out_off, out_cs, real = [], [], [0], [], []
    for b in range(len(off)):
        if b in at:
            e = np.zeros(5, dtype=pts.dtype)
            e["x"], e["batch_id"], e["host_atom"] = 200.0 + np.arange(5), len(out_off) - 1, 1
            out_p.append(e)
            out_w.append(np.full(5, 0.1))
            out_off.append(out_off[-1])
            real += [False] * 5
        if b == len(off) - 1:
            break
        rows = np.where(pts["batch_id"] == b)[0]
        q = pts[rows].copy()
        q["batch_id"] = len(out_off) - 1
        out_p.append(q)
        out_w.append(w[rows])
        out_cs.append(cs[off[b]:off[b + 1]])
        out_off.append(out_off[-1] + len(out_cs[-1]))
        real += [True] * len(rows)
    return (np.concatenate(out_p), np.concatenate(out_w), np.array(out_off, np.int32), np.concatenate(out_cs),
            np.array(real))


def weighted(basis, layout, n_ao):
    """An uploaded reference-layout grid with quadrature weights."""
    pts, w, off, cs = layout[:4]
    g = GpuVxcGrid.upload(*basis.gpu_arrays(), pts, off, cs, n_ao)
    _native.check("calchem_xc_set_weights", _native.load().calchem_xc_set_weights(g.grid_id, _native.ptr(w), len(w)))
    return g


def evaluate(g, P, Pb=None):
    lib, n = _native.load(), g.n_ao
    exc, ne = np.zeros(1), np.zeros(2)
    va, vb = np.zeros((n, n)), np.zeros((n, n))
    if Pb is None:
        _native.check("rks", lib.calchem_xc_evaluate_rks(g.grid_id, 3, 0, _native.ptr(P), _native.ptr(exc),
                                                          _native.ptr(ne), _native.ptr(va)))
    else:
        _native.check("uks", lib.calchem_xc_evaluate_uks(g.grid_id, 3, 0, _native.ptr(P), _native.ptr(Pb),
                                                          _native.ptr(exc), _native.ptr(ne), _native.ptr(va),
                                                          _native.ptr(vb)))
    return exc[0], ne, va, vb


@pytest.mark.parametrize("where", ["first", "middle", "last", "several"])
def test_batches_without_candidate_shells(native_lib, where):
    """An empty candidate list is a valid batch: its points get a density of zero and add nothing.  Per-point
    results of the other batches are the same bits; sums over batches agree to the order of their additions
    (64 roundings of 2^-53 of the largest entry cover the few batches here)."""
    mol = distorted_water()
    basis = BasisSet.from_name("6-31g(d)", mol)
    n = basis.n_ao
    plain = reference_layout(basis, points(mol, 900, 3))
    nb = len(plain[2]) - 1
    at = {"first": [0], "middle": [nb // 2], "last": [nb], "several": [0, 1, nb // 2, nb]}[where]
    holed = with_empty_batches(*plain, at)
    real = holed[4]
    P = make_positive_density(n, 7)
    rng = np.random.default_rng(5)
    wv, wxc = rng.normal(size=(len(real), 4)), rng.normal(size=(len(real), 8))
    a, b = weighted(basis, plain, n), weighted(basis, holed, n)
    close = lambda x, y: np.max(np.abs(x - y)) <= 64 * 2.0 ** -53 * np.max(np.abs(y))  # noqa: E731
    for _ in range(2):  # the pass that fills the AO cache and one that reads it
        ra, rb = a.eval_rho_grad(P), b.eval_rho_grad(P)
        assert np.array_equal(rb[real], ra) and not np.any(rb[~real])
        assert close(b.accumulate_vxc(wv), a.accumulate_vxc(wv[real]))
        assert close(b.eval_grad_force(P, P, True, wxc, 3), a.eval_grad_force(P, P, True, wxc[real], 3))
        for Pb in (None, 0.5 * P):
            for x, y in zip(evaluate(b, P, Pb), evaluate(a, P, Pb)):
                assert close(x, y)
    a.release()
    b.release()


def test_more_empty_batches_than_ctas(native_lib):
    """More empty batches than CTAs, so that CTAs meet several of them and nothing else."""
    mol = distorted_water()
    basis = BasisSet.from_name("6-31g(d)", mol)
    n = basis.n_ao
    pts, w, off, cs = reference_layout(basis, points(mol, 100, 3))
    k = 700
    empty = np.zeros(k, dtype=pts.dtype)
    empty["x"], empty["batch_id"] = 300.0, np.arange(k)
    shifted = pts.copy()
    shifted["batch_id"] += k
    layout = (np.concatenate([empty, shifted]), np.concatenate([np.ones(k), w]),
              np.concatenate([np.zeros(k, np.int32), off]).astype(np.int32), cs)
    P = make_positive_density(n, 7)
    a, b = weighted(basis, (pts, w, off, cs), n), weighted(basis, layout, n)
    for _ in range(2):
        rb = b.eval_rho_grad(P)
        assert np.array_equal(rb[k:], a.eval_rho_grad(P)) and not np.any(rb[:k])
    a.release()
    b.release()


def test_shares_alone_over_cached_batches(native_lib):
    """Per-atom shares without Vxc: batches follow each other without the V phase's barriers and
    copies, and from the second call on without the AO evaluation either.  The same bits as the full build's
    shares, every time."""
    mol = distorted_water()
    basis = BasisSet.from_name("6-31g(d)", mol)
    P = make_positive_density(basis.n_ao, 7)
    grid = points(mol, 60000, 11)
    rng = np.random.default_rng(2)
    for precision, code in (("fp64", 0), ("mixed", 1)):
        eng = RksVxcEngine(basis, grid, precision=precision, tile=64)
        eng.set_point_atoms(rng.integers(0, 3, len(grid)), 3)
        exc, _, ea, ta = eng.evaluate_with_shares(basis, grid, "b3lyp", P)
        e, ne, out = np.zeros(1), np.zeros(1), np.zeros(6)
        for _ in range(5):
            _native.check("atoms", native_lib.calchem_xc_evaluate_rks_atoms(
                eng.grid_id, 3, code, _native.ptr(P), _native.ptr(e), _native.ptr(ne), _native.ptr(out), None))
            assert e[0] == exc and np.array_equal(out[0::2], ea) and np.array_equal(out[1::2], ta)
        eng.close()


def test_grid_that_no_shell_reaches(native_lib):
    """Every batch's candidate list empty: zeros throughout."""
    from tests.host_calls import nothing_reached
    mol = distorted_water()
    basis = BasisSet.from_name("6-31g(d)", mol)
    P = make_positive_density(basis.n_ao, 7)
    g = nothing_reached(basis)
    assert not np.any(g.eval_rho_grad(P)) and not np.any(g.accumulate_vxc(np.ones((300, 4))))
    assert not np.any(g.eval_grad_force(P, P, True, np.ones((300, 8)), 3))
    w, host, f = np.ones(300), np.zeros(300, np.int32), np.ones((3, 3))
    p = _native.ptr
    _native.check("weights", native_lib.calchem_xc_set_weights(g.grid_id, p(w), 300))
    for Pb in (None, P):
        assert not any(np.any(x) for x in evaluate(g, P, Pb))
    z, xyz = np.array(mol.z, dtype=np.int32), np.ascontiguousarray(mol.coords_bohr)
    for precision in (0, 1):
        _native.check("gradient", native_lib.calchem_xc_nuclear_gradient(
            g.grid_id, 2, precision, 3, p(z), p(xyz), p(w), p(host), 300, p(P), None, p(f)))
        assert not np.any(f)
    g.release()
