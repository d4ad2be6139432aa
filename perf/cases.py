"""The workloads this library's speed is judged by: whole calls through the public entry points, over the
range of systems, bases, grids, functionals and precisions an electronic-structure program uses.

A case is one call that such a program makes over and over: the Vxc build of an SCF iteration (closed or
open shell, the FP64 engine that is the default or the tensor-core one), a group of molecules replayed as
one CUDA graph, the XC nuclear gradient of a geometry step, the TD-DFT kernel contraction of a Davidson
step, and the reference's own two-call interface (densities out, potential back).  The geometry and the
engine built on it are what the program keeps between calls; the density matrices are what changes, and
they come from the seed.

``exact`` evaluates the same quadrature in plain FP64 torch: Gaussian AOs, the published forms of the
functionals with their derivatives by autograd, and dense matrix products.
"""

import functools
import math

import numpy as np
import torch

from calchem_gb300 import (BasisSet, FxcKernel, GpuVxcGrid, GridLevel, MolecularGrid, RksVxcEngine, UksVxcEngine,
                           VxcGroup, plan_points, workloads)
from calchem_gb300 import _native

LEVELS = {"coarse": GridLevel.COARSE, "medium": GridLevel.MEDIUM, "fine": GridLevel.FINE}
BASES = ("sto-3g", "6-31g", "6-31g(d)", "6-31g(d,p)")
FUNCS = ("svwn5", "b3lyp", "pbe", "pbe0")


def listed():
    def case(name, kind, mol, size, basis, func, level, precision, n_mats=1):
        return {"name": name, "kind": kind, "mol": mol, "size": size, "basis": basis, "func": func, "level": level,
                "precision": precision, "n_mats": n_mats}
    return [
        # one SCF iteration of the smallest job: latency and launches
        case("water_svwn5_fp64", "rks", "water", 1, "6-31g(d)", "svwn5", "fine", "fp64"),
        # one SCF iteration of an ordinary organic molecule, the default engine and the tensor-core one
        case("octane_b3lyp_fp64", "rks", "alkane", 8, "6-31g(d,p)", "b3lyp", "fine", "fp64"),
        case("octane_b3lyp_mixed", "rks", "alkane", 8, "6-31g(d,p)", "b3lyp", "fine", "mixed"),
        # one SCF iteration of a solvent cluster in the default engine
        case("waters24_b3lyp_fp64", "rks", "waters", 24, "6-31g(d)", "b3lyp", "medium", "fp64"),
        # one SCF iteration of the largest system, 183 atoms and 1159 AOs
        case("waters61_b3lyp_mixed", "rks", "waters", 61, "6-31g(d)", "b3lyp", "medium", "mixed"),
        # open shells: a small triplet in the default engine, the C54H18 triplet in the tensor-core one
        case("hexane_pbe_uks_fp64", "uks", "alkane", 6, "6-31g(d)", "pbe", "medium", "fp64"),
        case("c54h18_pbe0_uks_mixed", "uks", "flake", 1, "6-31g(d)", "pbe0", "coarse", "mixed"),
        # many small molecules in one launch (screening, data generation), device buffers, graph replay
        case("clusters_pbe_graph_mixed", "graph", "clusters", 8, "6-31g(d)", "pbe", "medium", "mixed", 16),
        # the gradient of a geometry step
        case("waters8_b3lyp_gradient_fp64", "gradient", "waters", 8, "6-31g(d)", "b3lyp", "medium", "fp64"),
        case("octane_b3lyp_gradient_mixed", "gradient", "alkane", 8, "6-31g(d,p)", "b3lyp", "fine", "mixed"),
        # a Davidson step of TD-DFT: several trial matrices
        case("hexane_b3lyp_fxc_fp64", "fxc", "alkane", 6, "6-31g(d,p)", "b3lyp", "coarse", "fp64", 4),
        # the reference's two-call interface on its own batches (densities out, potential back)
        case("octane_ffi_fp64", "ffi", "alkane", 8, "6-31g(d)", "b3lyp", "coarse", "fp64"),
    ]


def draw(rng):
    """A case of the same ranges: any kind, molecule, basis, functional, grid level and precision, sizes
    spread over their logarithm, its contraction work no more than the largest listed case's."""
    while True:
        kind = rng.choice(("rks", "rks", "rks", "uks", "uks", "graph", "gradient", "fxc", "ffi"))
        mol = "clusters" if kind == "graph" else rng.choice(("alkane", "waters"))
        top = 8 if kind == "graph" else 12 if mol == "alkane" else 32
        low = 2 if mol == "alkane" else 1
        c = {"kind": kind, "mol": mol, "size": int(round(math.exp(rng.uniform(math.log(low), math.log(top))))),
             "basis": rng.choice(BASES), "func": rng.choice(FUNCS), "level": rng.choice(tuple(LEVELS)),
             "precision": "fp64" if kind == "ffi" else rng.choice(("fp64", "mixed")),
             "n_mats": rng.randint(2, 12) if kind == "graph" else rng.randint(1, 8) if kind == "fxc" else 1}
        atoms = 3 * c["size"] if mol == "waters" else 3 * c["size"] + 2
        work = atoms * {"coarse": 1.3, "medium": 5.6, "fine": 16.2}[c["level"]]  # thousands of points
        work *= {"graph": 0.6 * c["n_mats"], "fxc": 2.0 * c["n_mats"], "gradient": 3.0, "uks": 2.0}.get(kind, 1.0)
        if work * (1.0 if c["precision"] == "mixed" else 3.0) <= 3000.0:
            return c


# ---- inputs ------------------------------------------------------------------------------------------

def _molecules(case):
    kind, size = case["mol"], case["size"]
    if kind == "clusters":
        return [workloads.water_cluster(k, 1000 + i) for i, k in
                enumerate(workloads.cluster_batch_sizes(case["n_mats"], 2024, size))]
    mol = {"water": lambda: workloads.water(), "alkane": lambda: workloads.alkane(size),
           "waters": lambda: workloads.water_cluster(size, size), "flake": lambda: workloads.circumcoronene()}[kind]()
    if case["kind"] == "uks":
        mol.multiplicity = 3
    return [mol]


def _densities(case, mol, basis, seed):
    """(total,) or (alpha, beta): S-orthonormal random orbitals with the molecule's electron counts."""
    S = basis.overlap()
    if case["kind"] == "uks":
        na, nb = mol.n_alpha_beta()
        return workloads.seeded_density_uks(S, min(na, basis.n_ao), min(nb, basis.n_ao), seed, seed + 1)
    return (workloads.seeded_density_rks(S, min(mol.nelectron() // 2, basis.n_ao), seed),)


def _inputs(case, seed):
    """[(molecule, basis, grid, densities)] of the case's molecules."""
    out = []
    for i, mol in enumerate(_molecules(case)):
        basis = BasisSet.from_name(case["basis"], mol)
        grid = MolecularGrid.build_for_basis(mol, basis, LEVELS[case["level"]])
        out.append((mol, basis, grid, _densities(case, mol, basis, 1000003 * (seed % 99991) + 7 * i)))
    return out


def _trials(case, n, seed):
    rng = np.random.Generator(np.random.PCG64(seed + 17))
    mats = rng.standard_normal((case["n_mats"], n, n)) * 0.02
    return [0.5 * (m + m.T) for m in mats]


def _reference_batches(basis, grid):
    """What CalChem's engine uploads: chunks of 128 consecutive points (|w| < 1e-24 left out) and, per
    chunk, the shells whose cut-off sphere meets the sphere around the chunk's box."""
    sh, pr, co = basis.gpu_arrays()
    centers, rcut = np.asarray(sh["center"]), np.sqrt(sh["r2_cutoff"])
    pts, keep_w, offsets, cand = [], [], [0], []
    for s in range(0, len(grid.xyzw), 128):
        rows = np.arange(s, min(s + 128, len(grid.xyzw)))
        rows = rows[np.abs(grid.xyzw[rows, 3]) >= 1e-24]
        if len(rows) == 0:
            continue
        lo, hi = grid.xyzw[rows, :3].min(axis=0), grid.xyzw[rows, :3].max(axis=0)
        mid = 0.5 * (lo + hi)
        hit = np.where(((centers - mid) ** 2).sum(axis=1) <= (np.sqrt(((hi - mid) ** 2).sum()) + rcut) ** 2)[0]
        if len(hit) == 0:
            continue
        p = np.zeros(len(rows), dtype=_native.GRID_PT)
        p["x"], p["y"], p["z"] = grid.xyzw[rows, 0], grid.xyzw[rows, 1], grid.xyzw[rows, 2]
        p["batch_id"], p["host_atom"] = len(offsets) - 1, grid.host_atom[rows]
        pts.append(p)
        keep_w.append(grid.xyzw[rows, 3])
        cand.extend(int(k) for k in hit)
        offsets.append(len(cand))
    return (sh, pr, co, np.concatenate(pts), np.concatenate(keep_w), np.array(offsets, np.int32),
            np.array(cand, np.int32))


def _ffi_inputs(case, seed):
    """The two-call interface's inputs: batches, density, and per-point potential coefficients of a
    promolecule (w v / 2 and w u), as the caller's own functional code would hand back."""
    (mol, basis, grid, (P,)), = _inputs(case, seed)
    sh, pr, co, pts, w, off, cand = _reference_batches(basis, grid)
    xyz = np.stack([pts["x"], pts["y"], pts["z"]], axis=1)
    scale = 1.0 + 0.1 * np.random.Generator(np.random.PCG64(seed + 29)).random(len(mol.z))
    rho, grad = np.zeros(len(xyz)), np.zeros((len(xyz), 3))
    for z, x, s in zip(mol.z, mol.coords_bohr, scale):
        d = xyz - x
        r = np.sqrt((d ** 2).sum(axis=1))
        e = s * z * np.exp(-2.0 * r)
        rho += e
        grad -= (2.0 * e / np.maximum(r, 1e-12))[:, None] * d
    v = -0.9847450218426965 * np.cbrt(rho)
    u = -0.005 / np.maximum(rho, 1e-10) ** (4.0 / 3.0) * np.exp(-1e-3 / np.maximum(rho, 1e-10))
    wv = np.concatenate([(0.5 * w * v)[:, None], (w * u)[:, None] * grad], axis=1)
    return basis, P, (sh, pr, co, pts, off, cand), xyz, wv


def prepare(case, seed):
    kind, prec = case["kind"], case["precision"]
    if kind == "ffi":
        basis, P, (sh, pr, co, pts, off, cand), _, wv = _ffi_inputs(case, seed)
        return {"kind": kind, "grid": GpuVxcGrid.upload(sh, pr, co, pts, off, cand, basis.n_ao), "P": P, "wv": wv}
    members = _inputs(case, seed)
    mol, basis, grid, dens = members[0]
    st = {"kind": kind, "mol": mol, "basis": basis, "grid": grid, "dens": dens, "func": case["func"]}
    if kind == "rks":
        st["engine"] = RksVxcEngine.new_with_gpu(basis, grid, True, prec)
    elif kind == "uks":
        st["engine"] = UksVxcEngine.new_with_gpu(basis, grid, True, prec)
    elif kind == "gradient":
        st["engine"] = RksVxcEngine.new_with_gpu(basis, grid, True, prec)
        st["half"] = 0.5 * dens[0]
    elif kind == "fxc":
        st["kernel"] = FxcKernel(basis, grid, case["func"], dens[0], prec)
        st["trials"] = _trials(case, basis.n_ao, seed)
    else:  # graph: the group's densities, results and potentials in device buffers
        group = VxcGroup([(b, g) for _, b, g, _ in members], prec)
        st["P"] = torch.from_numpy(group.pack([d[0] for _, _, _, d in members])).cuda()
        st["result"] = torch.zeros(2 * group.n_mols, dtype=torch.float64, device="cuda")
        st["v"] = torch.zeros(group.packed_size, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        group.capture_rks(case["func"], st["P"].data_ptr(), st["result"].data_ptr(), st["v"].data_ptr())
        st["group"] = group
    return st


def run(state):
    kind = state["kind"]
    if kind == "ffi":
        return {"rho_grad": state["grid"].eval_rho_grad(state["P"]), "v": state["grid"].accumulate_vxc(state["wv"])}
    if kind == "rks":
        exc, v = state["engine"].evaluate(state["basis"], state["grid"], state["func"], state["dens"][0])
        return {"sums": np.array([exc, state["engine"].last_nelec]), "v": v}
    if kind == "uks":
        exc, va, vb = state["engine"].evaluate(state["basis"], state["grid"], state["func"], *state["dens"])
        return {"sums": np.array([exc, *state["engine"].last_nelec]), "va": va, "vb": vb}
    if kind == "gradient":
        return {"grad": state["engine"].nuclear_gradient(state["mol"], state["grid"], state["func"], state["half"])}
    if kind == "fxc":
        return {"dv": state["kernel"].contract_batch(state["trials"])}
    state["group"].replay(torch.cuda.current_stream().cuda_stream)
    return {"result": state["result"], "v": state["v"]}


@functools.lru_cache(maxsize=64)
def _plan_work(key):
    """(points, sum over points of the local AO count squared, sum of AO counts squared) of a case."""
    case = dict(key)
    pts = m2n = n2 = 0.0
    for mol in _molecules(case):
        basis = BasisSet.from_name(case["basis"], mol)
        grid = MolecularGrid.build_for_basis(mol, basis, LEVELS[case["level"]])
        pts += len(grid)
        m2n += plan_points(basis, grid)["sum_m2n"]
        n2 += float(basis.n_ao) ** 2
    return pts, m2n, n2


def work(case):
    """The densities read and the potentials written once, the points and weights read once; the two
    contractions over the AOs that reach each point, 4 m^2 flop per point and spin."""
    pts, m2n, n2 = _plan_work(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    spins = {"uks": 2, "fxc": case["n_mats"]}.get(case["kind"], 1)
    per_pt = {"ffi": 32 + 64, "gradient": 44, "fxc": 88}.get(case["kind"], 32)
    return {"bytes": 16.0 * n2 * spins + per_pt * pts, "flops": 4.0 * m2n * spins}


# ---- the same quadrature in plain FP64 torch ---------------------------------------------------------

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _shell_types(basis):
    """Shells of equal angular momentum and primitive count together:
    (l, powers, AO indices [n, funcs], atoms, exponents, weighted norms, component scales, cut-offs)."""
    sh, pr, co = basis.gpu_arrays()
    groups = {}
    for i, s in enumerate(sh):
        groups.setdefault((int(s["n_funcs"]), int(s["n_prims"])), []).append(i)
    d = _dev()
    out = []
    for (nf, n_pr), idx in sorted(groups.items()):
        s = sh[idx]
        pi = s["prim_start"][:, None] + np.arange(n_pr)[None]
        ci = s["comp_start"][:, None] + np.arange(nf)[None]
        powers = [(int(c["lx"]), int(c["ly"]), int(c["lz"])) for c in co[ci[0]]]
        out.append((powers, torch.from_numpy((s["ao_offset"][:, None] + np.arange(nf)[None]).astype(np.int64)).to(d),
                    torch.from_numpy(s["atom_index"].astype(np.int64)).to(d),
                    *(torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(d) for a in
                      (pr["exponent"][pi], pr["weighted_norm"][pi], co["scale"][ci], s["r2_cutoff"]))))
    return out


def _aos(types, centers, xyz):
    """phi and its gradient at the points: [4][points][AOs]; differentiable in centers and xyz."""
    cols = [[] for _ in range(4)]
    index = []
    for powers, ao, atom, exps, norms, scales, cut in types:
        d = [xyz[:, k, None] - centers[atom, k][None] for k in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        r0, r1 = 0.0, 0.0
        for p in range(exps.shape[1]):
            e = norms[None, :, p] * torch.exp(-exps[None, :, p] * r2)
            r0 = r0 + e
            r1 = r1 - 2.0 * exps[None, :, p] * e
        on = (r2 <= cut[None]).to(torch.float64)
        r0, r1 = r0 * on, r1 * on
        pw = [[torch.ones_like(x), x, x * x, x * x * x] for x in d]
        for c, l in enumerate(powers):
            m = pw[0][l[0]] * pw[1][l[1]] * pw[2][l[2]]
            s = scales[None, :, c]
            cols[0].append(s * m * r0)
            for q in range(3):
                g = m * d[q] * r1
                if l[q] > 0:
                    rest = [pw[k][l[k]] for k in range(3) if k != q]
                    g = g + l[q] * pw[q][l[q] - 1] * rest[0] * rest[1] * r0
                cols[q + 1].append(s * g)
            index.append(ao[:, c])
    inv = torch.argsort(torch.cat(index))
    return [torch.cat(c, dim=1)[:, inv] for c in cols]


def _vwn(x, a, x0, b, c):
    X = x * x + b * x + c
    X0 = x0 * x0 + b * x0 + c
    q = math.sqrt(4.0 * c - b * b)
    at = torch.atan(q / (2.0 * x + b))
    return a * (torch.log(x * x / X) + 2.0 * b / q * at -
                b * x0 / X0 * (torch.log((x - x0) ** 2 / X) + 2.0 * (b + 2.0 * x0) / q * at))


def _spin_interp(zeta, e0, e1, ac):
    c2 = 2.0 ** (1.0 / 3.0) - 1.0
    zp, zm = torch.clamp(1.0 + zeta, min=1e-300), torch.clamp(1.0 - zeta, min=1e-300)
    f = (zp ** (4.0 / 3.0) + zm ** (4.0 / 3.0) - 2.0) / (2.0 * c2)
    z4 = zeta ** 4
    return e0 + ac * f * (9.0 * c2 / 4.0) * (1.0 - z4) + (e1 - e0) * f * z4


def _energy_density(func, ra, rb, gaa, gab, gbb):
    rho = ra + rb
    zeta = (ra - rb) / rho
    f = 0.0
    slater = {"svwn5": 1.0, "b3lyp": 0.8}.get(func, 0.0)
    if slater:
        for r in (ra, rb):
            f = f - slater * 0.75 * (6.0 / math.pi) ** (1.0 / 3.0) * r ** (4.0 / 3.0)
    if func == "b3lyp":
        for r, g in ((ra, gaa), (rb, gbb)):
            r43 = r ** (4.0 / 3.0)
            s2 = g / (r43 * r43) + 1e-60
            s = torch.sqrt(s2)
            f = f - 0.72 * r43 * 0.0042 * s2 / (1.0 + 6.0 * 0.0042 * s * torch.asinh(s))
    if func in ("svwn5", "b3lyp"):
        x = torch.sqrt((3.0 / (4.0 * math.pi * rho)) ** (1.0 / 3.0))
        ch = ((-0.10498, 3.72744, 12.9352), (-0.32500, 7.06042, 18.0578), (-0.00475840, 1.13107, 13.0045)) \
            if func == "svwn5" else ((-0.409286, 13.0720, 42.7198), (-0.743294, 20.1231, 101.578),
                                     (-0.228344, 1.06835, 11.4813))
        ec = _spin_interp(zeta, _vwn(x, 0.0310907, *ch[0]), _vwn(x, 0.01554535, *ch[1]),
                          _vwn(x, -0.016886863940389905, *ch[2]))
        f = f + (1.0 if func == "svwn5" else 0.19) * rho * ec
    if func == "b3lyp":  # LYP
        A, B, C, D = 0.04918, 0.132, 0.2533, 0.349
        rm = rho ** (-1.0 / 3.0)
        den = 1.0 + D * rm
        delta = C * rm + D * rm / den
        far = C * rm > 500.0
        omega = torch.where(far, torch.zeros_like(rm), torch.exp(-C * torch.where(far, torch.ones_like(rm), rm)) / den *
                            torch.where(far, torch.ones_like(rm), rho) ** (-11.0 / 3.0))
        cf = 0.3 * (3.0 * math.pi ** 2) ** (2.0 / 3.0)
        stf = 2.0 ** (11.0 / 3.0) * cf * ra * rb * (ra ** (8.0 / 3.0) + rb ** (8.0 / 3.0))
        cg = ra * rb * (47.0 - 7.0 * delta) / 18.0 - 2.0 / 3.0 * rho * rho
        c25, c11 = 2.5 - delta / 18.0, (delta - 11.0) / 9.0
        ea = -ra * rb * c25 - c11 * ra * ra * rb / rho + 2.0 / 3.0 * rho * rho - rb * rb
        eb = -ra * rb * c25 - c11 * ra * rb * rb / rho + 2.0 / 3.0 * rho * rho - ra * ra
        s = stf + (cg + ea) * gaa + 2.0 * cg * gab + (cg + eb) * gbb
        f = f + 0.81 * (-4.0 * A / (rho * den) * ra * rb - A * B * omega * s)
    if func in ("pbe", "pbe0"):
        kappa, mu, beta, gam = 0.804, 0.2195149727645171, 0.06672455060314922, 0.0310906908696549
        for r, g in ((ra, gaa), (rb, gbb)):
            ru, gu = 2.0 * r, 4.0 * g
            s2 = gu / (4.0 * (3.0 * math.pi ** 2 * ru) ** (2.0 / 3.0) * ru * ru)
            ex = -0.75 * (3.0 / math.pi) ** (1.0 / 3.0) * ru ** (4.0 / 3.0)
            f = f + (1.0 if func == "pbe" else 0.75) * 0.5 * ex * (1.0 + kappa - kappa / (1.0 + mu / kappa * s2))
        rs = (3.0 / (4.0 * math.pi * rho)) ** (1.0 / 3.0)
        x = torch.sqrt(rs)

        def pw92(a, a1, b1, b2, b3, b4):
            q1 = 2.0 * a * (b1 * x + b2 * rs + b3 * rs * x + b4 * rs * rs)
            return -2.0 * a * (1.0 + a1 * rs) * torch.log1p(1.0 / q1)
        ec = _spin_interp(zeta, pw92(0.0310907, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294),
                          pw92(0.01554535, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517),
                          -pw92(0.0168869, 0.11125, 10.357, 3.6231, 0.88026, 0.49671))
        phi = 0.5 * (torch.clamp(1.0 + zeta, min=1e-24) ** (2.0 / 3.0) +
                     torch.clamp(1.0 - zeta, min=1e-24) ** (2.0 / 3.0))
        gt = gaa + 2.0 * gab + gbb
        t2 = gt / ((16.0 / math.pi) * (3.0 * math.pi ** 2) ** (1.0 / 3.0) * phi * phi * rho ** (7.0 / 3.0))
        g3 = gam * phi ** 3
        w = -ec / g3
        af = torch.where(w > 100.0, torch.zeros_like(w), beta / gam / torch.expm1(torch.clamp(w, max=100.0)))
        u = af * t2
        h = g3 * torch.log(1.0 + beta / gam * t2 * (1.0 + u) / (1.0 + u + u * u))
        f = f + rho * (ec + h)
    return f


def _functional(func, ra, rb, gaa, gab, gbb):
    """(f, dF/drho_a, dF/drho_b, dF/dgamma_aa, dF/dgamma_ab, dF/dgamma_bb); zero below the density floor."""
    on = ra + rb >= 1e-18
    safe = lambda t, v: torch.where(on, t, torch.full_like(t, v))  # noqa: E731
    x = [safe(torch.clamp(ra, min=1e-30), 1.0), safe(torch.clamp(rb, min=1e-30), 1.0), safe(gaa, 0.0), safe(gab, 0.0),
         safe(gbb, 0.0)]
    x = [t.detach().clone().requires_grad_(True) for t in x]
    f = _energy_density(func, *x)
    d = torch.autograd.grad(f.sum(), x, allow_unused=True)
    zero = torch.zeros_like(f)
    return [torch.where(on, zero if t is None else t.detach(), zero) for t in (f, *d)]


def _exact_vxc(func, basis, xyzw, dens, spins):
    """Exc, electron counts and Vxc per spin for densities `dens` (one: half of the total each spin)."""
    d = _dev()
    P = [torch.from_numpy(np.ascontiguousarray(p)).to(d) for p in dens]
    if not spins:
        P = [0.5 * P[0]]
    types, n = _shell_types(basis), basis.n_ao
    centers = torch.from_numpy(np.stack([s.center for s in basis.shells])).to(d)
    atom_of = np.array([s.atom_index for s in basis.shells])
    at = np.zeros((atom_of.max() + 1, 3))
    at[atom_of] = centers.cpu().numpy()
    centers = torch.from_numpy(at).to(d)
    pts = torch.from_numpy(xyzw).to(d)
    V = [torch.zeros(n, n, dtype=torch.float64, device=d) for _ in P]
    exc, ne = 0.0, [0.0] * len(P)
    step = max(1024, int(4e7 // max(n, 1)))
    for s in range(0, len(pts), step):
        c = pts[s:s + step]
        phi, *grad = _aos(types, centers, c[:, :3])
        rho, g = [], []
        for p in P:
            T = phi @ p.T
            rho.append((phi * T).sum(1))
            g.append([2.0 * (x * T).sum(1) for x in grad])
        a, b = 0, len(P) - 1
        dot = lambda u, v: u[0] * v[0] + u[1] * v[1] + u[2] * v[2]  # noqa: E731
        f, va, vb, vaa, vab, vbb = _functional(func, rho[a], rho[b], dot(g[a], g[a]), dot(g[a], g[b]), dot(g[b], g[b]))
        w = c[:, 3]
        exc += float((w * f).sum())
        on = (rho[a] + rho[b] >= 1e-18).to(torch.float64)
        for k, (v, vself) in enumerate(((va, vaa), (vb, vbb))[:len(P)]):
            ne[k] += float((w * on * rho[k]).sum())
            Z = (0.5 * w * v)[:, None] * phi
            for q in range(3):
                Z = Z + (w * (2.0 * vself * g[k][q] + vab * g[b - k][q]))[:, None] * grad[q]
            M = Z.T @ phi
            V[k] += M + M.T
    return exc, ne, [v.cpu().numpy() for v in V]


RADII = {1: 0.35, 6: 0.70, 8: 0.60}  # Bragg-Slater, Angstrom


def _exact_gradient(func, mol, basis, grid, half):
    """dExc/dR by autograd: points, AO centres and Becke weights move with the atoms, densities fixed."""
    d = _dev()
    P = torch.from_numpy(half).to(d)
    R0 = torch.from_numpy(np.ascontiguousarray(mol.coords_bohr)).to(d)
    R = R0.clone().requires_grad_(True)
    types, n = _shell_types(basis), basis.n_ao
    na = len(mol.z)
    r = np.array([RADII[int(z)] for z in mol.z])
    chi = r[:, None] / r[None]
    u = (chi - 1.0) / (chi + 1.0)
    aij = torch.from_numpy(np.clip(u / (u * u - 1.0), -0.5, 0.5)).to(d)
    eye = torch.eye(na, dtype=torch.float64, device=d)
    xyz = torch.from_numpy(np.ascontiguousarray(grid.xyzw[:, :3])).to(d)
    raw = torch.from_numpy(np.ascontiguousarray(grid.raw_weight)).to(d)
    host = torch.from_numpy(grid.host_atom.astype(np.int64)).to(d)
    step = max(512, int(min(4e6 // n, 1.2e7 // (na * na))))
    for s in range(0, len(xyz), step):
        h = host[s:s + step]
        x = R[h] + (xyz[s:s + step] - R0[h]).detach()
        phi, *grad = _aos(types, R, x)
        T = phi @ P.T
        rho = (phi * T).sum(1)
        g = [2.0 * (q * T).sum(1) for q in grad]
        gam = g[0] * g[0] + g[1] * g[1] + g[2] * g[2]
        on = 2.0 * rho >= 1e-18
        rs, gs = torch.where(on, rho, torch.ones_like(rho)), torch.where(on, gam, torch.zeros_like(gam))
        f = torch.where(on, _energy_density(func, rs, rs, gs, gs, gs), torch.zeros_like(rho))
        dist = torch.sqrt(((x[:, None] - R[None]) ** 2).sum(-1))
        rab = torch.sqrt(((R[:, None] - R[None]) ** 2).sum(-1) + eye)
        m = torch.clamp((dist[:, :, None] - dist[:, None, :]) / rab, -1.0, 1.0)
        m = torch.clamp(m + aij * (1.0 - m * m), -1.0, 1.0)
        for _ in range(3):
            m = 0.5 * m * (3.0 - m * m)
        cell = torch.prod(0.5 * (1.0 - m) * (1.0 - eye) + eye, dim=2)
        wt = raw[s:s + step] * cell.gather(1, h[:, None])[:, 0] / cell.sum(1)
        (wt * f).sum().backward()
    return R.grad.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "fxc":  # the kernel is defined by its finite-difference formula
        return None
    if kind == "ffi":
        basis, P, _, xyz, wv = _ffi_inputs(case, seed)
        d = _dev()
        types, n = _shell_types(basis), basis.n_ao
        at = np.zeros((1 + max(s.atom_index for s in basis.shells), 3))
        for s in basis.shells:
            at[s.atom_index] = s.center
        at, Pt = torch.from_numpy(at).to(d), torch.from_numpy(P).to(d)
        x, w = torch.from_numpy(xyz).to(d), torch.from_numpy(wv).to(d)
        V, rg = torch.zeros(n, n, dtype=torch.float64, device=d), []
        step = max(1024, int(4e7 // n))
        for s in range(0, len(x), step):
            phi, *grad = _aos(types, at, x[s:s + step])
            T = phi @ Pt.T
            rg.append(torch.stack([(phi * T).sum(1)] + [2.0 * (q * T).sum(1) for q in grad], dim=1))
            c = w[s:s + step]
            Z = sum(c[:, k, None] * q for k, q in enumerate((phi, *grad)))
            M = Z.T @ phi
            V += M + M.T
        return {"rho_grad": torch.cat(rg).cpu().numpy(), "v": np.tril(V.cpu().numpy())}
    members = _inputs(case, seed)
    mol, basis, grid, dens = members[0]
    if kind == "gradient":
        return {"grad": _exact_gradient(case["func"], mol, basis, grid, 0.5 * dens[0])}
    if kind == "graph":
        res, vs = [], []
        for _, b, g, p in members:
            e, ne, v = _exact_vxc(case["func"], b, g.xyzw, p, False)
            res += [e, 2.0 * ne[0]]
            vs.append(v[0].ravel())
        return {"result": np.array(res), "v": np.concatenate(vs)}
    e, ne, v = _exact_vxc(case["func"], basis, grid.xyzw, dens, kind == "uks")
    if kind == "uks":
        return {"sums": np.array([e, *ne]), "va": v[0], "vb": v[1]}
    return {"sums": np.array([e, 2.0 * ne[0]]), "v": v[0]}
