"""Workloads of this framework, each through the entry point that a program calls.

A case is a dict of plain values.  Its "kind" names the call:

  call      callTreedriver on host arrays, the reference's own call form: the mesh is
            copied in, the plan is built and used once, the result is copied out
  treecode  device.treecode: the same one-shot call on device arrays
  plan      TreecodePlan.convolve with the plan kept, targets = sources: the
            convolutions of a Green-iteration step (one or many orbitals)
  twomesh   TreecodePlan.convolve with coarse targets and fine sources at degree + 2:
            the convolutions of the two-mesh eigenvalue correction
  systems   Systems.convolve: several molecules in one launch per field pass
  sweep     one captured Green-iteration sweep over all orbitals (source,
            convolution, Harrison update, Gram-Schmidt, residual)
  mgs       weighted Gram-Schmidt of every orbital of a set in order
  interp    two-mesh interpolation, coarse cells to their fine cells
  mesh      two-level quadrature mesh built from cells and nuclei
  mlp       the learned extrapolator's layers, forward and backward, each by its own
            call on its own inputs

Sizes are those of the workloads in bench.py, DESIGN's configurations and the tests,
or lie between them.  A mesh's cells and point count belong to the case; the seed
moves and scales the molecule with its mesh and sets the charges, so inputs of
another seed are other inputs of the same size.
"""
import functools
import importlib
import math

import numpy as np
import torch

PKG = "treecode-accelerated-green-iteration_gb300"
pkg = importlib.import_module(PKG)
dev = importlib.import_module(PKG + ".device")
gi_mod = importlib.import_module(PKG + ".gi")
mesh_mod = importlib.import_module(PKG + ".mesh")
BT = pkg.BaryTreeInterface
KERNEL = {"yukawa": BT.Kernel.YUKAWA, "coulomb": BT.Kernel.COULOMB}
SING = {"subtraction": BT.Singularity.SUBTRACTION, "skipping": BT.Singularity.SKIPPING}
F64 = dict(dtype=torch.float64, device="cuda")


def listed():
    return [
        # the smallest call: a density on a coarse mesh, mixed precision, from host arrays
        dict(name="call_hartree_6k", kind="call", atoms=2, order=5, points=6000, kernel="coulomb", singularity="subtraction",
             degree=7, theta=0.7, leaf=500, precision="mixed"),
        # the reference's CPU-runnable case, one atom: the drop-in at its default precision
        dict(name="call_atom_50k_fp64", kind="call", atoms=1, order=5, points=50112, kernel="yukawa", singularity="subtraction",
             degree=7, theta=0.7, leaf=500, precision="fp64"),
        # the Hartree potential of a molecule, once per SCF iteration, plan included
        dict(name="hartree_1500k", kind="treecode", atoms=4, order=7, points=1500000, kernel="coulomb", singularity="subtraction",
             degree=7, theta=0.7, leaf=2000, precision="mixed"),
        # one orbital at a time over a kept plan, the reference's own loop over orbitals
        dict(name="yukawa_50k_1orb", kind="plan", atoms=2, order=6, points=50000, orbitals=1, kernel="yukawa",
             singularity="subtraction", degree=7, theta=0.7, leaf=500, precision="mixed"),
        # the headline: 32 orbitals of a molecule in one batched call
        dict(name="yukawa_1M_32orb", kind="plan", atoms=3, order=7, points=1000000, orbitals=32, kernel="yukawa",
             singularity="subtraction", degree=7, theta=0.7, leaf=2000, precision="mixed"),
        # the two-mesh correction's convolutions: targets are not the sources, degree 9
        dict(name="twomesh_6orb_deg9", kind="twomesh", spacing=3.0, order=5, level=-2, orbitals=6, kernel="yukawa",
             degree=9, theta=0.55, leaf=1000, precision="mixed"),
        # three molecules of uneven size in one launch, k on the device as a captured loop has it
        dict(name="systems_50k_120k_300k", kind="systems", sizes="50000,120000,300000", orbitals="4,8,8", order=6, degree=7,
             theta=0.7, leaf=1000, precision="mixed"),
        # one sweep of the ring molecule's SCF: 21 occupied orbitals and 3 buffer orbitals
        dict(name="sweep_ring_262k_24orb", kind="sweep", atoms=12, order=7, points=262144, orbitals=24, degree=7, theta=0.7,
             leaf=2000, precision="mixed"),
        # Gram-Schmidt of a whole orbital set after a sweep
        dict(name="mgs_1M_32rows", kind="mgs", points=1000448, rows=32),
        # interpolation of one function to the ring molecule's fine mesh
        dict(name="interp_ring", kind="interp", spacing=1.0, order=7, level=-2),
        # the ring molecule's two-level mesh, built for each geometry
        dict(name="mesh_ring", kind="mesh", spacing=1.0, order=7, level=-2),
        # the extrapolator's layers at 21 orbitals x 512 cells of 8^3 points
        dict(name="mlp_10752_rows", kind="mlp", rows=10752, patch=512, hidden=256),
    ]


# ---------------------------------------------------------------------------------------
# Drawn cases: the same calls over the ranges that the listed ones stand for.
# ---------------------------------------------------------------------------------------
def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw(rng):
    kind = rng.choice(["call", "call", "treecode", "plan", "plan", "twomesh", "systems", "sweep", "mgs", "interp", "mesh", "mlp"])
    order = rng.randint(4, 7)
    tree = dict(degree=rng.randint(4, 8), theta=round(rng.uniform(0.6, 0.8), 3))
    if kind == "call":
        p = rng.choice(["fp64", "mixed"])
        return dict(kind=kind, atoms=rng.randint(1, 8), order=order, points=int(_log(rng, 2500, 50000 if p == "fp64" else 250000)),
                    kernel=rng.choice(["yukawa", "coulomb"]), singularity=rng.choice(["subtraction", "subtraction", "skipping"]),
                    leaf=rng.randint(200, 1000), precision=p, **tree)
    if kind == "treecode":
        return dict(kind=kind, atoms=rng.randint(1, 8), order=order, points=int(_log(rng, 20000, 1500000)),
                    kernel=rng.choice(["yukawa", "coulomb"]), singularity=rng.choice(["subtraction", "subtraction", "skipping"]),
                    leaf=rng.randint(500, 2000), precision="mixed", **tree)
    if kind == "plan":
        p = rng.choice(["mixed", "mixed", "mixed", "fp64"])
        return dict(kind=kind, atoms=rng.randint(1, 8), order=order, points=int(_log(rng, 10000, 1000000)),
                    orbitals=int(_log(rng, 1, 33)), kernel=rng.choice(["yukawa", "yukawa", "coulomb"]),
                    singularity=rng.choice(["subtraction", "subtraction", "skipping"]), leaf=rng.randint(400, 2000), precision=p, **tree)
    if kind == "twomesh":
        return dict(kind=kind, spacing=round(_log(rng, 2.1, 4.9), 3), order=rng.choice([3, 5]), level=-2, orbitals=rng.randint(1, 12),
                    kernel=rng.choice(["yukawa", "yukawa", "coulomb"]), degree=rng.randint(6, 10), theta=round(rng.uniform(0.5, 0.65), 3),
                    leaf=rng.randint(500, 2000), precision="mixed")
    if kind == "systems":
        n = rng.randint(2, 6)
        return dict(kind=kind, sizes=",".join(str(int(_log(rng, 8000, 300000))) for _ in range(n)),
                    orbitals=",".join(str(int(_log(rng, 1, 17))) for _ in range(n)), order=order, leaf=rng.randint(500, 2000),
                    precision="mixed", **tree)
    if kind == "sweep":
        return dict(kind=kind, atoms=rng.choice([1, 2, 4, 12]), order=order, points=int(_log(rng, 20000, 300000)),
                    orbitals=rng.randint(1, 24), leaf=rng.randint(500, 2000), precision="mixed", **tree)
    if kind == "mgs":
        return dict(kind=kind, points=int(_log(rng, 2000, 1200000)), rows=int(_log(rng, 2, 49)))
    if kind in ("interp", "mesh"):
        order = rng.randint(3, 8)
        return dict(kind=kind, spacing=round(_log(rng, 0.9, 4.9), 3), order=order, level=rng.choice([-2, -2, -3]) if order % 2 else -2)
    return dict(kind=kind, rows=int(_log(rng, 400, 24000)), patch=rng.choice([4, 5, 6, 7, 8]) ** 3, hidden=rng.choice([128, 256, 256, 512]))


def draw(rng):
    while True:
        c = _draw(rng)
        w = work(c)
        # FP64 pairs cost a few hundred times a mixed pair; ungrouped orbitals about twice a grouped one
        cost = w["flops"] * (500.0 if c.get("precision") == "fp64" else 1.0)
        if cost <= 1.5e13 and w["bytes"] <= 2.0e10:
            return c


# ---------------------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=16)
def _molecule(atoms, order, points):
    """Points, weights, nuclei and charges of an adaptive mesh of about `points` points."""
    syn = pkg.synthetic
    rng = np.random.default_rng(atoms)
    if atoms == 1:
        nuclei, charges = np.zeros((1, 3)), np.array([4.0])
    elif atoms == 12:
        nuclei, charges = syn.ring_molecule()
    else:
        nuclei, charges = rng.uniform(-2.5, 2.5, (atoms, 3)), rng.choice([1.0, 6.0, 8.0], atoms)
    m = syn.mesh_with_points(nuclei, charges, order, 5 if points <= 60000 else 7, points)
    return np.stack([m.x, m.y, m.z]), m.w, np.asarray(nuclei, float), np.asarray(charges, float)


def _placed(case, seed, points=None):
    """The molecule's mesh moved and scaled by the seed: host coordinates, weights, nuclei, charges."""
    xyz, w, nuclei, charges = _molecule(case.get("atoms", 3), case["order"], points or case["points"])
    rng = np.random.default_rng(seed)
    s, t = 1.0 + 0.05 * rng.uniform(), rng.uniform(-0.5, 0.5, 3)
    return xyz * s + t[:, None], w * s ** 3, nuclei * s + t, charges, rng


def _potential(x, y, z, nuclei, charges, soft=0.01):
    v = torch.zeros_like(x)
    for R, q in zip(nuclei, charges):
        v -= q / torch.sqrt((x - R[0]) ** 2 + (y - R[1]) ** 2 + (z - R[2]) ** 2 + soft)
    return v


def _gaussians(rng, nuclei, n, terms=4):
    """n functions, each a signed sum of Gaussians on the nuclei (exponents 0.1 to 10)."""
    return [[(nuclei[rng.integers(len(nuclei))], math.exp(rng.uniform(math.log(0.1), math.log(10.0))), rng.choice([-1.0, 1.0]))
             for _ in range(terms)] for _ in range(n)]


def _on(mesh, functions):
    x, y, z = mesh
    out = torch.zeros((len(functions), x.numel()), **F64)
    for row, f in zip(out, functions):
        for R, a, c in f:
            row += c * torch.exp(-a * ((x - R[0]) ** 2 + (y - R[1]) ** 2 + (z - R[2]) ** 2))
    return out


def _density(x, y, z, nuclei, charges, rng):
    rho = torch.zeros_like(x)
    for R, q in zip(nuclei, charges):
        for a in np.exp(rng.uniform(math.log(0.1), math.log(10.0), 3)):
            rho += q / 3.0 * (a / math.pi) ** 1.5 * torch.exp(-a * ((x - R[0]) ** 2 + (y - R[1]) ** 2 + (z - R[2]) ** 2))
    return rho


def _charges(case, mesh, nuclei, charges, rng, orbitals):
    """f_i = -2 V psi_i with k_i (Yukawa), or densities with the Gaussian parameter 1 (Coulomb)."""
    x, y, z = mesh
    if case["kernel"] == "coulomb":
        return torch.stack([_density(x, y, z, nuclei, charges, rng) for _ in range(orbitals)]), [1.0] * orbitals
    f = _on(mesh, _gaussians(rng, nuclei, orbitals))
    f *= -2.0 * _potential(x, y, z, nuclei, charges)
    return f, [float(k) for k in rng.uniform(0.4, 3.0, orbitals)]


def _ring_cells(case, seed):
    """Arguments of the two-level mesh of the ring molecule, all lengths scaled by the seed."""
    s = 1.0 + 0.05 * np.random.default_rng(seed).uniform()
    nuclei, charges = pkg.synthetic.ring_molecule()
    h = case["spacing"]
    return dict(XL=20.0 * s, max_side_length=5.01 * s, atoms=nuclei * s, order=case["order"], h=h * s, H=5.5 * s, r=2.0 * s,
                level=float(case["level"])), charges, s


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def _prepare_call(case, seed):
    xyz, w, nuclei, charges, rng = _placed(case, seed)
    mesh = [torch.as_tensor(a, **F64) for a in xyz]
    f, k = _charges(case, mesh, nuclei, charges, rng, 1)
    return dict(kind="call", case=case, x=[np.ascontiguousarray(a) for a in xyz], w=w, f=f[0].cpu().numpy(), k=k)


def _run_call(s):
    c, (x, y, z) = s["case"], s["x"]
    n = len(x)
    return BT.callTreedriver(n, n, x, y, z, s["f"], x, y, z, s["f"], s["w"], KERNEL[c["kernel"]], 1, s["k"], SING[c["singularity"]],
                             BT.Approximation.LAGRANGE, BT.ComputeType.PARTICLE_CLUSTER, True, 0, theta=c["theta"], degree=c["degree"],
                             sourceLeafSize=c["leaf"], targetLeafSize=c["leaf"], precision=c["precision"])


def _on_device(case, seed, orbitals, points=None):
    xyz, w, nuclei, charges, rng = _placed(case, seed, points)
    mesh = [torch.as_tensor(a, **F64).contiguous() for a in xyz]
    f, k = _charges(dict(case, kernel=case.get("kernel", "yukawa")), mesh, nuclei, charges, rng, orbitals)
    return mesh, torch.as_tensor(w, **F64), f, k, nuclei, charges, rng


def _prepare_treecode(case, seed):
    mesh, w, f, k, *_ = _on_device(case, seed, 1)
    return dict(kind="treecode", case=case, mesh=mesh, w=w, f=f[0].contiguous(), k=k)


def _run_treecode(s):
    c, (x, y, z), f = s["case"], s["mesh"], s["f"]
    return dev.treecode(x, y, z, f, x, y, z, f, s["w"], KERNEL[c["kernel"]], s["k"], SING[c["singularity"]], c["theta"], c["degree"],
                        c["leaf"], c["leaf"], precision=c["precision"])


def _prepare_plan(case, seed):
    mesh, w, f, k, *_ = _on_device(case, seed, case["orbitals"])
    plan = dev.TreecodePlan.for_mesh(*mesh, w, theta=case["theta"], degree=case["degree"], source_leaf=case["leaf"],
                                     target_leaf=case["leaf"])
    return dict(kind="plan", case=case, plan=plan, targets=f, sources=f, k=k)


def _prepare_twomesh(case, seed):
    cfg, charges, _ = _ring_cells(case, seed)
    m = mesh_mod.build_mesh(**cfg)
    rng = np.random.default_rng(seed)
    state = rng.bit_generator.state
    tv, k = _charges(case, (m.X, m.Y, m.Z), cfg["atoms"], charges, rng, case["orbitals"])
    rng.bit_generator.state = state
    sv, _ = _charges(case, (m.Xf, m.Yf, m.Zf), cfg["atoms"], charges, rng, case["orbitals"])
    plan = dev.TreecodePlan(m.X, m.Y, m.Z, m.Xf, m.Yf, m.Zf, m.Wf, theta=case["theta"], degree=case["degree"],
                            source_leaf=case["leaf"], target_leaf=case["leaf"])
    return dict(kind="plan", case=dict(case, singularity="subtraction"), plan=plan, targets=tv, sources=sv, k=k)


def _run_plan(s):
    c = s["case"]
    return s["plan"].convolve(s["targets"], s["sources"], KERNEL[c["kernel"]], s["k"], SING[c["singularity"]], precision=c["precision"])


def _systems_of(case, seed):
    sizes = [int(v) for v in case["sizes"].split(",")]
    orbitals = [int(v) for v in case["orbitals"].split(",")]
    return [(_on_device(dict(case, atoms=2 + i), seed + 1000 * i, m, n), m) for i, (n, m) in enumerate(zip(sizes, orbitals))]


def _prepare_systems(case, seed):
    plans, fs, ks, orbitals = [], [], [], []
    for (mesh, w, f, k, *_), m in _systems_of(case, seed):
        plans.append(dev.TreecodePlan.for_mesh(*mesh, w, theta=case["theta"], degree=case["degree"], source_leaf=case["leaf"],
                                               target_leaf=case["leaf"]))
        fs.append(f)
        ks.append(torch.as_tensor(k, **F64))
        orbitals.append(m)
    return dict(kind="systems", systems=dev.Systems(plans, orbitals, precision=case["precision"]), f=fs, k=ks)


def _run_systems(s):
    return s["systems"].convolve(s["f"], s["f"], s["k"])


def _sweep_inputs(case, seed):
    mesh, w, _, _, nuclei, charges, rng = _on_device(case, seed, 0)
    m = case["orbitals"]
    psi = _on(mesh, _gaussians(rng, nuclei, m))
    psi /= torch.sqrt((psi * psi) @ w)[:, None]
    eps = -np.exp(rng.uniform(math.log(0.2), math.log(6.0), m))
    veff = _potential(*mesh, nuclei, charges) - 0.5
    return mesh, w, psi, torch.as_tensor(eps, **F64), veff


def _prepare_sweep(case, seed):
    mesh, w, psi, eps, veff = _sweep_inputs(case, seed)
    plan = dev.TreecodePlan.for_mesh(*mesh, w, theta=case["theta"], degree=case["degree"], source_leaf=case["leaf"],
                                     target_leaf=case["leaf"])
    gi = gi_mod.GreenIteration(plan, w, psi.clone(), eps, veff, precision=case["precision"])
    gi.capture()
    torch.cuda.current_stream().wait_stream(gi.stream)
    return dict(kind="sweep", gi=gi, psi=psi, eps=eps)


def _run_sweep(s):
    gi = s["gi"]
    gi.stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(gi.stream):
        gi.psi.copy_(s["psi"])
        gi.set_eigenvalues(s["eps"])
    gi.step()
    torch.cuda.current_stream().wait_stream(gi.stream)
    return dict(psi=gi.psi, eps=gi.eps, residual=gi.res)


def _mgs_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    conv = torch.randn((case["rows"], case["points"]), generator=g, **F64)
    conv[1:] += 0.3 * conv[:-1]
    return conv, 0.01 + torch.rand(case["points"], generator=g, **F64)


def _prepare_mgs(case, seed):
    conv, w = _mgs_inputs(case, seed)
    return dict(kind="mgs", conv=conv, w=w)


def _run_mgs(s):
    psi = s["conv"] * (1.0 / (4.0 * math.pi))   # the convolution's result, as a sweep scales it
    for m in range(psi.shape[0]):
        dev.mgs(psi, psi[m], s["w"], m)
    return psi


def _prepare_interp(case, seed):
    cfg, _, s = _ring_cells(case, seed)
    m = mesh_mod.build_mesh(**cfg)
    rng = np.random.default_rng(seed)
    f = torch.zeros_like(m.X)
    for R, a in zip(cfg["atoms"], rng.uniform(0.5, 3.0, 12)):
        f += torch.exp(-a * torch.sqrt((m.X - R[0]) ** 2 + (m.Y - R[1]) ** 2 + (m.Z - R[2]) ** 2))
    return dict(kind="interp", m=m, f=f)


def _run_interp(s):
    m = s["m"]
    return dev.interp(m.X, m.Y, m.Z, s["f"], m.PtsPerCellCoarse, m.Xf, m.Yf, m.Zf, m.PtsPerCellFine, m.num_cells, m.order)


def _prepare_mesh(case, seed):
    return dict(kind="mesh", cfg=_ring_cells(case, seed)[0])


_MESH_OUT = ("cellX", "cellY", "cellZ", "cellDX", "cellDY", "cellDZ", "PtsPerCellCoarse", "PtsPerCellFine", "X", "Y", "Z", "W", "Xf", "Yf",
             "Zf", "Wf")


def _run_mesh(s):
    m = mesh_mod.build_mesh(**s["cfg"])
    return {k: getattr(m, k) for k in _MESH_OUT}


def _prepare_mlp(case, seed):
    R, P, H = case["rows"], case["patch"], case["hidden"]
    ldx = (2 * P + 1 + 31) // 32 * 32
    g = torch.Generator(device="cuda").manual_seed(seed)

    def t(*shape, scale=1.0, dtype=torch.bfloat16):
        return (scale * torch.randn(shape, generator=g, device="cuda")).to(dtype)

    s = dict(kind="mlp", R=R, P=P, H=H, ldx=ldx, X=t(R, ldx), W1=t(H, ldx, scale=ldx ** -0.5), W3=t(P, H, scale=H ** -0.5),
             b1=t(H, dtype=torch.float32), b3=t(P, dtype=torch.float32), H2=torch.relu(t(R, H)), dY=t(R, P), dH1=t(R, H))
    s["splits"] = max(1, min(64, (R + 2047) // 2048))
    s["part"] = torch.empty(s["splits"] * H * max(ldx, P), device="cuda")
    s["work"] = torch.empty(int(pkg._native.lib().tagi_mlp_colsum_workspace(R, max(H, P))), device="cuda")
    s["out"] = dict(H1=torch.empty(R, H, dtype=torch.bfloat16, device="cuda"), Y=torch.empty(R, P, device="cuda"),
                    dH2=torch.empty(R, H, dtype=torch.bfloat16, device="cuda"), gW3=torch.empty(P, H, device="cuda"),
                    gW1=torch.empty(H, ldx, device="cuda"), gb1=torch.empty(H, device="cuda"))
    return s


def _run_mlp(s):
    """Layer 1 forward, layer 3 forward, layer 3's data gradient, both weight gradients, a bias gradient."""
    L, check = pkg._native.lib(), pkg._native.check
    R, P, H, ldx, o = s["R"], s["P"], s["H"], s["ldx"], s["out"]
    p = lambda t: t.data_ptr()  # noqa: E731
    q = torch.cuda.current_stream().cuda_stream
    check(L.tagi_mlp_gemm(p(s["X"]), ldx, 1, p(s["W1"]), 1, ldx, R, H, ldx, 1, None, p(o["H1"]), H, p(s["b1"]), None, q))
    check(L.tagi_mlp_gemm(p(s["H2"]), H, 1, p(s["W3"]), 1, H, R, P, H, 3, p(o["Y"]), None, P, p(s["b3"]), None, q))
    check(L.tagi_mlp_gemm(p(s["dY"]), P, 1, p(s["W3"]), H, 1, R, H, P, 2, None, p(o["dH2"]), H, None, p(s["H2"]), q))
    check(L.tagi_mlp_gemm_splitk(p(s["dY"]), 1, P, p(s["H2"]), H, 1, P, H, R, s["splits"], p(s["part"]), p(o["gW3"]), q))
    check(L.tagi_mlp_gemm_splitk(p(s["dH1"]), 1, H, p(s["X"]), ldx, 1, H, ldx, R, s["splits"], p(s["part"]), p(o["gW1"]), q))
    check(L.tagi_mlp_colsum(p(s["dH1"]), 1, R, H, p(o["gb1"]), p(s["work"]), s["work"].numel(), q))
    return o


_PREPARE = dict(call=_prepare_call, treecode=_prepare_treecode, plan=_prepare_plan, twomesh=_prepare_twomesh, systems=_prepare_systems,
                sweep=_prepare_sweep, mgs=_prepare_mgs, interp=_prepare_interp, mesh=_prepare_mesh, mlp=_prepare_mlp)
_RUN = dict(call=_run_call, treecode=_run_treecode, plan=_run_plan, systems=_run_systems, sweep=_run_sweep, mgs=_run_mgs,
            interp=_run_interp, mesh=_run_mesh, mlp=_run_mlp)


# ---------------------------------------------------------------------------------------
# What a pass cannot do without.
# ---------------------------------------------------------------------------------------
def _pairs(targets, sources, leaf, degree):
    """Kernel evaluations of one convolution: the leaves around a target's leaf directly, the rest
    through (degree + 1)^3 proxy points of about 45 clusters a level."""
    levels = max(0.0, math.log(max(sources / leaf, 1.0), 8.0) - 0.5)
    return targets * min(float(sources), 45.0 * leaf + 45.0 * levels * (degree + 1) ** 3)


def _ring_size(case):
    """(coarse points, fine points) of the ring molecule's two-level mesh, roughly."""
    near, far = (27900, 89800), (5000, 15000)
    cells, sub = (5100, near) if case["spacing"] < 1.25 else (1270, far) if case["spacing"] < 2.5 else (624, (1408, 3536))
    p3 = float((case["order"] + 1) ** 3)
    return cells * p3, sub[0 if case["level"] == -2 else 1] * p3


def work(case):
    c, kind = case, case["kind"]
    if kind in ("call", "treecode", "plan"):
        n, m = c["points"], c.get("orbitals", 1)
        return dict(bytes=8.0 * n * (4 + 2 * m), flops=10.0 * m * _pairs(n, n, c["leaf"], c["degree"]))
    if kind == "twomesh":
        nc, nf = _ring_size(c)
        return dict(bytes=8.0 * (3 * nc + 4 * nf + c["orbitals"] * (2 * nc + nf)),
                    flops=10.0 * c["orbitals"] * _pairs(nc, nf, c["leaf"], c["degree"]))
    if kind == "systems":
        sizes, orbitals = ([int(v) for v in c[k].split(",")] for k in ("sizes", "orbitals"))
        return dict(bytes=sum(8.0 * n * (4 + 2 * m) for n, m in zip(sizes, orbitals)),
                    flops=sum(10.0 * m * _pairs(n, n, c["leaf"], c["degree"]) for n, m in zip(sizes, orbitals)))
    if kind == "sweep":
        n, m = c["points"], c["orbitals"]
        return dict(bytes=8.0 * n * (5 + 2 * m), flops=10.0 * m * _pairs(n, n, c["leaf"], c["degree"]) + 2.0 * n * m * m)
    if kind == "mgs":
        n, m = c["points"], c["rows"]
        return dict(bytes=8.0 * n * (1 + 2 * m), flops=2.0 * n * m * (m - 1) + 5.0 * n * m)
    if kind in ("interp", "mesh"):
        nc, nf = _ring_size(c)
        if kind == "mesh":
            return dict(bytes=32.0 * (nc + nf), flops=2.0 * (nc + nf))
        return dict(bytes=32.0 * (nc + nf), flops=6.0 * (c["order"] + 1) * nf)
    R, P, H = c["rows"], c["patch"], c["hidden"]
    ldx = (2 * P + 1 + 31) // 32 * 32
    read = R * ldx + H * ldx + R * H + P * H + R * P + P * H + R * H + R * P + R * H + R * H + R * ldx + R * H
    wrote = 2.0 * R * H + 4.0 * R * P + 2.0 * R * H + 4.0 * P * H + 4.0 * H * ldx
    return dict(bytes=2.0 * read + wrote, flops=2.0 * R * H * (2.0 * ldx + 3.0 * P))


# ---------------------------------------------------------------------------------------
# The same results in 64 bits from torch and numpy alone.
# ---------------------------------------------------------------------------------------
MOST_PAIRS = 9.0e10


def _direct(targets, tv, sources, sv, w, kernel, k, subtract):
    """sum_j G(x_i, y_j) over all pairs, the coincident one left out, with or without subtraction."""
    out = torch.empty_like(tv)
    step = max(1, 8_000_000 // sources[0].numel())
    for a in range(0, tv.numel(), step):
        r2 = None
        for t, s in zip(targets, sources):
            d = t[a:a + step, None] - s[None, :]
            r2 = d * d if r2 is None else r2.addcmul_(d, d)
        zero = r2 == 0.0
        r = torch.sqrt(r2)
        fi = tv[a:a + step, None]
        if kernel == "yukawa":
            g = torch.exp(-k * r).div_(r)
            term = (sv[None, :] - fi) * w * g if subtract else g * (sv * w)
        else:
            e = torch.exp(-k * k * r2).mul_(fi) if subtract else 0.0
            term = (sv[None, :] - e) * w / r
        out[a:a + step] = term.masked_fill_(zero, 0.0).sum(1)
    if subtract:
        out += tv * (4.0 * math.pi / k ** 2 if kernel == "yukawa" else 2.0 * math.pi / k ** 2)
    return out


def _exact_orbitals(case, targets, tv, sources, sv, w, k, subtract):
    return torch.stack([_direct(targets, tv[m], sources, sv[m], w, case["kernel"], k[m], subtract) for m in range(tv.shape[0])])


def exact(case, seed):
    kind = case["kind"]
    sub = case.get("singularity", "subtraction") == "subtraction"
    if kind in ("call", "treecode", "plan"):
        m = case.get("orbitals", 1)
        if float(case["points"]) ** 2 * m > MOST_PAIRS:
            return None
        mesh, w, f, k, *_ = _on_device(case, seed, m)
        out = _exact_orbitals(case, mesh, f, mesh, f, w, k, sub)
        return out if kind == "plan" else out[0].cpu().numpy() if kind == "call" else out[0]
    if kind == "systems":
        n = [int(v) for v in case["sizes"].split(",")]
        if sum(float(a) ** 2 * int(m) for a, m in zip(n, case["orbitals"].split(","))) > MOST_PAIRS:
            return None
        return [_exact_orbitals(dict(case, kernel="yukawa"), mesh, f, mesh, f, w, k, True)
                for (mesh, w, f, k, *_), _m in _systems_of(case, seed)]
    if kind == "sweep":
        return _exact_sweep(case, seed)
    if kind == "mgs":
        conv, w = _mgs_inputs(case, seed)
        return _gram_schmidt(conv * (1.0 / (4.0 * math.pi)), w)
    if kind == "mesh":
        return _exact_mesh(_ring_cells(case, seed)[0])
    if kind == "twomesh":
        return _exact_twomesh(case, seed)
    if kind == "interp":
        return _exact_interp(case, seed)
    return _exact_mlp(case, seed)


def _gram_schmidt(psi, w):
    for m in range(psi.shape[0]):
        u = psi[m].clone()
        if m:
            u -= (psi[:m] @ (u * w)) @ psi[:m]
        psi[m] = u / torch.sqrt((u * u * w).sum())
    return psi


def _exact_sweep(case, seed):
    if float(case["points"]) ** 2 * case["orbitals"] > MOST_PAIRS:
        return None
    mesh, w, psi, eps, veff = _sweep_inputs(case, seed)
    k = torch.sqrt(-2.0 * eps).tolist()
    f = -2.0 * psi * veff
    new = _exact_orbitals(dict(kernel="yukawa"), mesh, f, mesh, f, w, k, True) / (4.0 * math.pi)
    e = eps - (psi * veff * (psi - new)) @ w / ((new * new) @ w)
    e = torch.where(e < 0.0, e, torch.full_like(e, -2.0))
    out = _gram_schmidt(new, w)
    d = out - psi
    return dict(psi=out, eps=e, residual=torch.sqrt((d * d) @ w + (e - eps) ** 2))


def _unit(order):
    n = order + 1
    t = (math.pi - (np.arange(n) + 0.5) * math.pi / n)
    even = np.arange(0, n, 2)
    lam = np.where(even == 0, 1.0, 2.0 / (1.0 - even.astype(float) ** 2))
    return np.cos(t), 2.0 / n * (np.cos(np.outer((np.arange(n) + 0.5) * math.pi / n, even)) * lam).sum(1)


def _leaves(XL, max_side_length, atoms, order, h, H, r, level):
    """Leaf cells (lo, hi) depth first and children per side of each, by the two-level rule."""
    n = int(-((-2 * XL) // max_side_length))
    e = np.linspace(-XL, XL, n + 1)
    i, j, k = (a.ravel() for a in np.meshgrid(*[np.arange(n)] * 3, indexing="ij"))
    lo, hi = np.stack([e[i], e[j], e[k]], 1), np.stack([e[i + 1], e[j + 1], e[k + 1]], 1)
    key = np.arange(n ** 3, dtype=np.int64) << 40
    done = []
    for depth in range(12):
        dist = np.full(len(lo), 10.0 + H)
        for a in atoms:
            inside = ((a > lo) & (a < hi)).all(1)
            far = np.minimum(np.abs(lo - a), np.abs(hi - a))   # the nearest corner
            dist = np.minimum(dist, np.sqrt((far ** 2).sum(1)))
            dist[inside] = 0.0
        side = (hi - lo).max(1)
        div = (side > H) | ((dist < r) & (side > h))
        for near, reach, limit in ((r, r + 2 * h, 2 * h), (r + 2 * h, r + 6 * h, 4 * h), (r + 6 * h, r + 14 * h, 8 * h)):
            div |= (dist >= near) & (dist < reach) & (side > limit)
        m = np.where(dist < 1.5 * r, -int(level) if level < -1 else 1, 1)
        done.append((key[~div], lo[~div], hi[~div], m[~div]))
        if not div.any():
            break
        l, u, kk = lo[div], hi[div], key[div]
        mid = 0.5 * (u + l)
        lo, hi, key = [], [], []
        for q in range(8):
            up = np.array([q >> 2, (q >> 1) & 1, q & 1], bool)
            lo.append(np.where(up, mid, l))
            hi.append(np.where(up, u, mid))
            key.append(kk | (q << (3 * (12 - depth))))
        lo, hi, key = np.concatenate(lo), np.concatenate(hi), np.concatenate(key)
    key, lo, hi, m = (np.concatenate([d[i] for d in done]) for i in range(4))
    at = np.argsort(key, kind="stable")
    return lo[at], hi[at], m[at]


def _points(lo, hi, u, wt):
    hw = 0.5 * (hi - lo)
    p = lo[:, :, None] + hw[:, :, None] * (u + 1.0)
    w = hw[:, :, None] * wt
    n, c = len(u), len(lo)
    shape = (c, n, n, n)
    return [np.broadcast_to(p[:, 0, :, None, None], shape).reshape(-1), np.broadcast_to(p[:, 1, None, :, None], shape).reshape(-1),
            np.broadcast_to(p[:, 2, None, None, :], shape).reshape(-1),
            (w[:, 0, :, None, None] * w[:, 1, None, :, None] * w[:, 2, None, None, :]).reshape(-1)]


def _children(lo, hi, m):
    """Equal children of every cell, cell by cell, x-major."""
    count = m ** 3
    cell = np.repeat(np.arange(len(lo)), count)
    q = np.arange(count.sum()) - np.repeat(np.cumsum(count) - count, count)
    mm = m[cell]
    ijk = np.stack([q // (mm * mm), q // mm % mm, q % mm], 1)
    w = (hi - lo)[cell] / mm[:, None]
    return lo[cell] + w * ijk, np.where(ijk + 1 == mm[:, None], hi[cell], lo[cell] + w * (ijk + 1))


def _exact_mesh(cfg):
    lo, hi, m = _leaves(**cfg)
    u, wt = _unit(cfg["order"])
    p3 = (cfg["order"] + 1) ** 3
    clo, chi = _children(lo, hi, m)
    out = [*(0.5 * (lo + hi)).T, *(hi - lo).T, np.full(len(lo), p3, np.int32), (p3 * m ** 3).astype(np.int32), *_points(lo, hi, u, wt),
           *_points(clo, chi, u, wt)]
    return dict(zip(_MESH_OUT, out))


def _exact_twomesh(case, seed):
    cfg, charges, _ = _ring_cells(case, seed)
    lo, hi, m = _leaves(**cfg)
    u, wt = _unit(case["order"])
    coarse = [torch.as_tensor(a, **F64) for a in _points(lo, hi, u, wt)]
    fine = [torch.as_tensor(a, **F64) for a in _points(*_children(lo, hi, m), u, wt)]
    if float(coarse[0].numel()) * fine[0].numel() * case["orbitals"] > MOST_PAIRS:
        return None
    rng = np.random.default_rng(seed)
    state = rng.bit_generator.state
    tv, k = _charges(case, coarse[:3], cfg["atoms"], charges, rng, case["orbitals"])
    rng.bit_generator.state = state
    sv, _ = _charges(case, fine[:3], cfg["atoms"], charges, rng, case["orbitals"])
    return _exact_orbitals(case, coarse[:3], tv, fine[:3], sv, fine[3], k, True)


def _exact_interp(case, seed):
    cfg, _, _ = _ring_cells(case, seed)
    lo, hi, m = _leaves(**cfg)
    u, wt = _unit(case["order"])
    p1 = case["order"] + 1
    x, y, z, _w = (torch.as_tensor(a, **F64) for a in _points(lo, hi, u, wt))
    f = torch.zeros_like(x)
    for R, a in zip(cfg["atoms"], np.random.default_rng(seed).uniform(0.5, 3.0, 12)):
        f += torch.exp(-a * torch.sqrt((x - R[0]) ** 2 + (y - R[1]) ** 2 + (z - R[2]) ** 2))
    f = f.reshape(-1, p1, p1, p1)
    # the fine nodes on a child's axis, in the cell's own [-1, 1], and their Lagrange rows
    rows = {}
    bw = (-1.0) ** np.arange(p1) * np.sin((2 * np.arange(p1) + 1) * math.pi / (2 * p1))
    for n in (1, -int(case["level"])):
        for i in range(n):
            v = -1.0 + (2.0 * i + u + 1.0) / n
            if n == 1:
                rows[n, i] = torch.eye(p1, **F64)
            else:
                t = bw / (v[:, None] - u[None, :])
                rows[n, i] = torch.as_tensor(t / t.sum(1, keepdims=True), **F64)
    out = torch.empty(int((m ** 3).sum()) * p1 ** 3, **F64).reshape(-1, p1, p1, p1)
    start = np.cumsum(m ** 3) - m ** 3
    for n in set(m.tolist()):
        cells = np.nonzero(m == n)[0]
        fc = f[torch.as_tensor(cells, device="cuda")]
        for q in range(n ** 3):
            i, j, k = q // (n * n), q // n % n, q % n
            v = torch.einsum("ai,bj,ck,nijk->nabc", rows[n, i], rows[n, j], rows[n, k], fc)
            out[torch.as_tensor(start[cells] + q, device="cuda")] = v
    return out.reshape(-1)


def _exact_mlp(case, seed):
    s = _prepare_mlp(case, seed)
    d = {k: v.double() for k, v in s.items() if torch.is_tensor(v)}
    return dict(H1=torch.relu(d["X"] @ d["W1"].T + d["b1"]), Y=d["H2"] @ d["W3"].T + d["b3"],
                dH2=(d["dY"] @ d["W3"]) * (d["H2"] > 0), gW3=d["dY"].T @ d["H2"], gW1=d["dH1"].T @ d["X"], gb1=d["dH1"].sum(0))
