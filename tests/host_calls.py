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
    return mol, basis, MolecularGrid(xyzw, xyzw[:, 3].copy(), host, GridLevel.COARSE), np.eye(basis.n_ao)


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


def host_calls():
    """(name, call -> status, the call's outputs) of every evaluation on host buffers, both precisions."""
    lib = _native.load()
    mol, basis, grid, P = molecule()
    n = basis.n_ao
    z, xyz = np.array(mol.z, dtype=np.int32), np.ascontiguousarray(mol.coords_bohr)
    p = _native.ptr
    out = lambda *shape: np.full(shape, 7.0)  # noqa: E731
    for prec, name in ((0, "fp64"), (1, "mixed")):
        eng = RksVxcEngine(basis, grid, precision=name, tile=64)
        eng.set_point_atoms(grid.host_atom, 3)
        e, ne, v, vb, sh, pt, g = out(1), out(2), out(n, n), out(n, n), out(6), out(len(grid), 2), np.zeros((3, 3))
        gid = eng.grid_id
        yield name + " rks", lambda: lib.calchem_xc_evaluate_rks(gid, 2, prec, p(P), p(e), p(ne), p(v)), (e, ne, v)
        yield name + " uks", lambda: lib.calchem_xc_evaluate_uks(
            gid, 2, prec, p(P), p(P), p(e), p(ne), p(v), p(vb)), (e, ne, v, vb)
        yield name + " points", lambda: lib.calchem_xc_evaluate_rks_points(
            gid, 2, prec, p(P), p(e), p(ne), p(pt)), (e, ne, pt)
        yield name + " atoms", lambda: lib.calchem_xc_evaluate_rks_atoms(
            gid, 2, prec, p(P), p(e), p(ne), p(sh), p(v)), (e, ne, sh, v)
        yield name + " shares", lambda: lib.calchem_xc_evaluate_rks_atoms(
            gid, 2, prec, p(P), p(e), p(ne), p(sh), None), (e, ne, sh)
        yield name + " gradient", lambda: lib.calchem_xc_nuclear_gradient(  # (fills its output with zeros first)
            gid, 2, prec, 3, p(z), p(xyz), p(grid.raw_weight), p(grid.host_atom), len(grid), p(P), None, p(g)), (g,)
        eng.close()
        fxc = FxcKernel(basis, grid, "pbe", P, name)
        yield name + " fxc", lambda: lib.calchem_xc_fxc_contract_ex(fxc.grid_id, 0, prec, p(P), 1, p(v)), (v,)
        fxc.close()
    d, _ = dropin(basis, grid)
    rg, wv, wxc, f = out(d.n_pts, 4), np.zeros((d.n_pts, 4)), np.zeros((d.n_pts, 8)), out(3, 3)
    yield "rho", lambda: lib.calchem_cuda_vxc_eval_rho(d.grid_id, p(P), p(rg), d.n_pts, n), (rg,)
    yield "accum", lambda: lib.calchem_cuda_vxc_accum(d.grid_id, p(wv), p(v), d.n_pts, n), (v,)
    yield "force", lambda: lib.calchem_cuda_vxc_grad_force(d.grid_id, p(P), p(P), 1, p(wxc), p(f), d.n_pts, n, 3, 0), (f,)


def check_outputs_stay_as_they_were_when_a_wait_expired(fake):
    """-7: the status word is read before anything is copied to the caller."""
    for name, call, outputs in host_calls():
        before = [o.copy() for o in outputs]
        assert call() == 0, name
        for o, b in zip(outputs, before):
            o[...] = b
        fake.fake_status(1)
        assert call() == -7, name
        fake.fake_status(0)
        for o, b in zip(outputs, before):
            assert np.array_equal(o, b), name


def check_errors_leave_no_copy_under_way(fake):
    """-5 from any copy, clear, launch or wait: nothing still reads or writes the caller's memory afterwards."""
    for name, call, _ in host_calls():
        assert call() == 0, name  # (scratch and caches are there)
        for f in (b"cudaMemcpyAsync", b"cudaMemsetAsync", b"cudaLaunchKernel", b"cudaStreamSynchronize"):
            for nth in range(1, 40):
                fake.fake_fail(f, nth)
                rc = call()
                assert fake.fake_host_copies() == 0, (name, f, nth)
                if rc == 0:
                    break
                assert rc == -5, (name, f, nth, rc)
            fake.fake_fail(f, 0)


def check_allowing_the_ao_cache_again_changes_nothing(fake):
    """set_ao_cache(1) where the caller did not switch it off: what is cached or captured stays, also after the FP64
    form found no room for a cache of its own; and that form asks again at its next evaluation."""
    lib = _native.load()
    _, basis, grid, P = molecule()
    eng = RksVxcEngine(basis, grid, precision="mixed", tile=64)
    eng.evaluate(basis, grid, "pbe", P)
    size = eng.ao_cache_bytes()
    assert size > 0
    d = np.zeros(basis.n_ao ** 2 + 2)
    _native.check("capture", lib.calchem_xc_graph_capture(eng.grid_id, 0, 2, 1, _native.ptr(d), None, _native.ptr(d),
                                                          _native.ptr(d), None))
    os.environ["CALCHEM_MAX_AO_GRID_BYTES"] = "0"
    eng.evaluate(basis, grid, "pbe", P, precision="fp64")  # no cache
    del os.environ["CALCHEM_MAX_AO_GRID_BYTES"]
    used = fake.fake_used()
    eng.set_ao_cache(True)
    assert eng.ao_cache_bytes() == size and lib.calchem_xc_graph_launch(eng.grid_id, None) == 0
    eng.evaluate(basis, grid, "pbe", P, precision="fp64")
    assert fake.fake_used() > used and eng.ao_cache_bytes() == size
    eng.set_ao_cache(False)
    assert eng.ao_cache_bytes() == 0 and lib.calchem_xc_graph_launch(eng.grid_id, None) == -1
    eng.evaluate(basis, grid, "pbe", P)
    assert eng.ao_cache_bytes() == 0
    eng.set_ao_cache(True)
    eng.evaluate(basis, grid, "pbe", P)
    assert eng.ao_cache_bytes() == size


class Budgeted:
    """The molecule uploaded with a memory budget; least() is the smallest that its upload accepts."""

    ids = 10 ** 6

    def __init__(self, limit):
        self.lib = _native.load()
        _, basis, grid, self.P = molecule()
        sh, pr, co = basis.gpu_arrays()
        Budgeted.ids += 1
        self.id = Budgeted.ids
        p = _native.ptr
        self.rc = self.lib.calchem_xc_upload_points_spatial(p(sh), len(sh), p(pr), len(pr), p(co), len(co), p(grid.xyzw),
                                                           len(grid), basis.n_ao, 128, self.id, int(limit))

    @staticmethod
    def least():
        lo, hi = 0, 1 << 34
        while hi - lo > 1:
            mid = (lo + hi) // 2
            b = Budgeted(mid)
            lo, hi = (lo, mid) if b.rc == 0 else (mid, hi)
            b.release()
        return hi

    def launches(self, precision):
        """One evaluation: 3 launches on the tensor cores (prepare, quadrature, finish), 2 in the FP64 SIMT form."""
        e, ne, v = np.zeros(1), np.zeros(2), np.zeros_like(self.P)
        p = _native.ptr
        _native.check("rks", self.lib.calchem_xc_evaluate_rks(self.id, 2, precision, p(self.P), p(e), p(ne), p(v)))
        return self.lib.calchem_xc_last_launch_count(self.id)

    def cache(self):
        out = (ctypes.c_size_t * 1)()
        _native.check("set_ao_cache", self.lib.calchem_xc_set_ao_cache(self.id, -1, out))
        return int(out[0])

    def gradient(self, precision):
        mol, _, grid, P = molecule()
        z, xyz, g = np.array(mol.z, dtype=np.int32), np.ascontiguousarray(mol.coords_bohr), np.zeros((3, 3))
        p = _native.ptr
        return self.lib.calchem_xc_nuclear_gradient(self.id, 2, precision, 3, p(z), p(xyz), p(grid.raw_weight),
                                                    p(grid.host_atom), len(grid), p(P), None, p(g))

    def release(self):
        self.lib.calchem_cuda_vxc_release(self.id)


def check_a_budget_is_charged_with_what_is_allocated(fake):
    """A grid's memory budget: the tensor-core form's cache gets all that the workspace leaves as long as the FP64 form
    has not been used, and that form takes its scratch from what is left then."""
    least = Budgeted.least()
    b = Budgeted(1 << 40)
    assert b.launches(1) == 3
    whole = b.cache()
    assert whole > 0 and b.launches(0) == 3  # (no limit that matters: both forms on the tensor cores)
    b.release()
    b = Budgeted(least + whole)
    assert b.launches(1) == 3 and b.cache() == whole
    assert b.launches(0) == 2  # nothing left
    b.release()
    b = Budgeted(least + whole)
    assert b.launches(0) == 3 and b.launches(1) == 3 and b.cache() < whole
    b.release()
    b = Budgeted(least)
    assert b.launches(0) == 2 and b.launches(1) == 3 and b.cache() == 0
    b.release()


def check_the_fp64_form_asks_again_for_scratch(fake):
    """Device memory too short for the tensor-core form's scratch is no decision for the grid's life."""
    b = Budgeted(1 << 40)
    b.launches(1)
    fake.fake_set_memory(ctypes.c_size_t(fake.fake_used() + 4096))
    assert b.launches(0) == 2
    fake.fake_set_memory(ctypes.c_size_t(280 << 30))
    assert b.launches(0) == 3


def check_a_gradients_buffers_stay_within_the_budget(fake):
    """They are kept for the next gradient where the grid's budget holds them, given back where it does not, and never
    keep a cache or another form's scratch from what it would get without them."""
    least = Budgeted.least()
    for precision in (0, 1):
        b = Budgeted(1 << 40)
        b.launches(1)
        whole = b.cache()
        before = fake.fake_used()
        assert b.gradient(precision) == 0
        kept = fake.fake_used() - before
        assert kept > 0
        n = fake.fake_calls(b"cudaMalloc")
        assert b.gradient(precision) == 0 and fake.fake_calls(b"cudaMalloc") == n
        b.release()

        b = Budgeted(least + whole)  # (the buffers are kept only where the limit allows it)
        b.launches(1)
        assert b.cache() == whole
        before = fake.fake_used()
        assert b.gradient(precision) == 0
        assert fake.fake_used() - before < 20000  # (the order of the points stays: 4 B each)
        b.release()

        b = Budgeted(least + max(whole, kept))
        assert b.gradient(precision) == 0  # first, into the budget that the cache asks for next
        assert b.launches(1) == 3 and b.cache() == whole
        b.release()


def check_a_force_call_keeps_no_more_than_its_limit(fake):
    """calchem_cuda_vxc_grad_force: neither its own buffers nor those of a gradient before it take more device memory
    than the limit it is given, and the limit it refuses does not depend on them."""
    lib = _native.load()
    mol, basis, grid, P = molecule()
    d, wq = dropin(basis, grid)
    w, f = np.zeros((d.n_pts, 8)), np.zeros((3, 3))
    p = _native.ptr

    def force(limit):
        return lib.calchem_cuda_vxc_grad_force(d.grid_id, p(P), p(P), 1, p(w), p(f), d.n_pts, basis.n_ao, 3,
                                               ctypes.c_size_t(limit))

    def least():
        lo, hi = 1, 1 << 34
        while hi - lo > 1:
            mid = (lo + hi) // 2
            rc = force(mid)
            assert rc in (0, -3)
            lo, hi = (lo, mid) if rc == 0 else (mid, hi)
        return hi
    empty = fake.fake_used()
    limit = least()
    assert fake.fake_used() - empty <= limit + 20 * 1024  # (each of some twenty buffers starts on a multiple of 1 KB)
    _native.check("weights", lib.calchem_xc_set_weights(d.grid_id, p(wq), len(wq)))
    z, xyz = np.array(mol.z, dtype=np.int32), np.ascontiguousarray(mol.coords_bohr)
    host = np.zeros(d.n_pts, np.int32)
    assert lib.calchem_xc_nuclear_gradient(d.grid_id, 2, 1, 3, p(z), p(xyz), p(wq), p(host), d.n_pts, p(P), None,
                                           p(f)) == 0
    assert fake.fake_used() - empty > limit + 20 * 1024
    assert least() == limit
    assert fake.fake_used() - empty <= limit + 20 * 1024


def check_kept_memory_makes_way_for_what_a_call_needs(fake):
    """As many grids fit the device as their uploads and workspaces allow: caches, scratch and gradient buffers that
    were allocated where there was room are given back when there is none, except those that a graph holds."""
    lib = _native.load()
    os.environ["CALCHEM_MAX_AO_GRID_BYTES"] = "0"
    b = Budgeted(1 << 40)
    before = fake.fake_used()
    b.release()
    empty = fake.fake_used()
    b = Budgeted(1 << 40)
    b.launches(1)  # (uses the workspace, and nothing else without a cache)
    each = fake.fake_used() - empty
    assert before - empty < each
    b.release()
    del os.environ["CALCHEM_MAX_AO_GRID_BYTES"]
    many = 30
    fake.fake_set_memory(ctypes.c_size_t(empty + many * each + (32 << 20)))
    first = Budgeted(1 << 40)
    assert first.launches(0) == 3
    d = np.zeros_like(first.P)
    p = _native.ptr
    _native.check("capture", lib.calchem_xc_graph_capture(first.id, 0, 2, 0, p(d), None, p(d), p(d), None))
    held = fake.fake_used() - empty
    assert each < held < each + (32 << 20)
    rest = []
    for _ in range(many - 1):
        rest.append(Budgeted(1 << 40))
        assert rest[-1].rc == 0
        assert rest[-1].launches(0) in (2, 3) and rest[-1].launches(1) == 3
        assert rest[-1].gradient(0) == 0
    assert all(r.launches(0) in (2, 3) for r in rest)
    n = fake.fake_calls(b"cudaMalloc")
    assert first.launches(0) == 3 and lib.calchem_xc_graph_launch(first.id, None) == 0
    assert fake.fake_calls(b"cudaMalloc") == n  # the graph's grid kept its own


def nothing_reached(basis):
    """A reference-layout upload whose points all are in batches without candidate shells."""
    pts = np.zeros(300, dtype=_native.GRID_PT)
    pts["x"] = 300.0
    pts["batch_id"] = np.arange(300) // 100
    off = np.array([0, 0, 0, 0, 1], np.int32)
    return GpuVxcGrid.upload(*basis.gpu_arrays(), pts, off, np.zeros(1, np.int32), basis.n_ao)


def check_a_grid_that_no_shell_reaches(fake):
    """Every call on it succeeds (each in a process that a division by zero would end)."""
    lib = _native.load()
    mol, basis, _, P = molecule()
    g = nothing_reached(basis)
    n, p = basis.n_ao, _native.ptr
    g.eval_rho_grad(P)
    g.accumulate_vxc(np.ones((300, 4)))
    g.eval_grad_force(P, P, True, np.ones((300, 8)), 3)
    w, host, f = np.ones(300), np.zeros(300, np.int32), np.zeros((3, 3))
    _native.check("weights", lib.calchem_xc_set_weights(g.grid_id, p(w), 300))
    z, xyz = np.array(mol.z, dtype=np.int32), np.ascontiguousarray(mol.coords_bohr)
    e, ne, v = np.zeros(1), np.zeros(2), np.zeros((n, n))
    for precision in (0, 1):
        assert lib.calchem_xc_evaluate_rks(g.grid_id, 2, precision, p(P), p(e), p(ne), p(v)) == 0
        assert lib.calchem_xc_nuclear_gradient(g.grid_id, 2, precision, 3, p(z), p(xyz), p(w), p(host), 300, p(P), None,
                                               p(f)) == 0


CHECKS = {k[len("check_"):]: v for k, v in list(globals().items()) if k.startswith("check_")}

if __name__ == "__main__":
    runtime = ctypes.CDLL(sys.argv[1])
    runtime.fake_used.restype = ctypes.c_size_t
    CHECKS[sys.argv[2]](runtime)
