"""Performance cases of the pressure-equation path, through the package's public entry points.

Kinds of work, each as a user's program calls it:

* pressure   one GAMG-PCG pressure solve (solve_ldu on host arrays, solve_ldu_device on resident ones)
* momentum   one PBiCGStab/DILU solve of a convection-diffusion matrix (a momentum predictor component)
* corrector  the pressure-corrector loop on one non-orthogonal mesh, host arrays
* batch      the pressure-corrector loop on a batch of uneven non-orthogonal meshes, resident arrays
* assembly   fvm::laplacian with its non-orthogonal correction, and fvc::grad, host arrays
* cavity     SIMPLE steps of the lid-driven cavity (2D), the serving workload's flow
* tgv        PIMPLE steps of the Taylor-Green vortex
* channel    PIMPLE steps of the LES channel with Van Driest damping and mean-velocity forcing

Meshes are boxes: uniform or graded, with any of their directions periodic, their inner vertices
jittered or not.  Every input follows from the seed.
"""
import math

import numpy as np
import torch

import voluma_b200 as vb
from voluma_b200 import cases as workloads
from voluma_b200 import mesh as vm

DT = 2e-3        # rAUf of the pressure solves (the Taylor-Green workload's time step)
REL_TOL = 1e-8   # relative tolerance of every pressure solve
DEV = "cuda"


# ------------------------------------------------------------------------------ the cases
def _pressure(nx, ny, nz, periodic="", ratio=1.0, jitter=0.0, precision="", memory="device", reproducible=False):
    return dict(kind="pressure", nx=nx, ny=ny, nz=nz, periodic=periodic, ratio=ratio, jitter=jitter,
                precision=precision, memory=memory, reproducible=reproducible)


def listed():
    return [
        # the smallest calls: a drop-in solve of a few hundred cells, where set-up and latency count
        dict(name="solve_small_host", **_pressure(10, 8, 6, jitter=0.2, memory="host")),
        # an ordinary drop-in solve: odd extents, walls all round, graded towards them
        dict(name="solve_walls_host", **_pressure(61, 45, 37, ratio=4.0, memory="host")),
        # a resident solve of middle size in full FP64
        dict(name="solve_periodic_fp64", **_pressure(96, 96, 96, periodic="xyz")),
        # the headline: the Taylor-Green pressure equation at 128^3 with the FP32 V-cycle
        dict(name="solve_tgv128_mixed", **_pressure(128, 128, 128, periodic="xyz", precision="mixed")),
        # bit-reproducible mode (diagonal PCG, exact sums) on a periodic-by-walls box
        dict(name="solve_reproducible", **_pressure(40, 36, 30, periodic="xz", reproducible=True)),
        # a momentum predictor component of a middle-sized transient flow
        dict(name="momentum_dilu", kind="momentum", nx=80, ny=64, nz=48, periodic="xz", courant=0.5),
        # the corrector loop with two non-orthogonal passes, odd extents, host arrays
        dict(name="corrector_jittered", kind="corrector", nx=45, ny=38, nz=33, ratio=3.0, jitter=0.2, passes=3,
             precision=""),
        # a batch of uneven Poisson systems (the batched-systems workload, scaled down)
        dict(name="batch_mixed", kind="batch", systems=24, nmin=16, nmax=48, jitter=0.2, passes=3,
             precision="mixed"),
        # one assembly of a non-orthogonal pressure equation and the gradient of its field
        dict(name="assembly_jittered", kind="assembly", nx=64, ny=56, nz=48, ratio=2.0, jitter=0.2),
        # what one serving request does most of the time: SIMPLE steps of a 2D cavity
        dict(name="flow_cavity64", kind="cavity", n=64, steps=10),
        # transient steps of a periodic 3D flow, mixed-precision pressure
        dict(name="flow_tgv64_mixed", kind="tgv", n=64, steps=4, precision="mixed"),
        # transient LES steps of a wall-bounded flow in FP64
        dict(name="flow_channel_les", kind="channel", nx=96, ny=72, nz=48, steps=2, precision=""),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def even(v):
        return v + (v & 1)

    kind = rng.choice(["pressure", "pressure", "pressure", "momentum", "corrector", "batch", "assembly", "cavity",
                       "tgv", "channel"])
    if kind == "pressure":
        periodic = rng.choice(["", "", "x", "xz", "xyz", "xyz"])
        n = [size(6, 120) for _ in range(3)]
        if rng.random() < 0.7:  # most boxes of a periodic direction have an even extent
            n = [even(v) if d in periodic else v for v, d in zip(n, "xyz")]
        repro = rng.random() < 0.15
        return _pressure(*n, periodic=periodic, ratio=rng.choice([1.0, round(rng.uniform(1.0, 6.0), 2)]),
                         jitter=rng.choice([0.0, 0.0, 0.2]),
                         precision="" if repro else rng.choice(["", "mixed", "mixed", "mixed-dc"]),
                         memory=rng.choice(["host", "device"]), reproducible=repro)
    if kind == "momentum":
        return dict(kind=kind, nx=size(12, 90), ny=size(12, 90), nz=rng.choice([1, size(8, 60)]),
                    periodic=rng.choice(["", "x"]), courant=round(rng.uniform(0.2, 0.8), 2))
    if kind in ("corrector", "assembly"):
        c = dict(kind=kind, nx=size(8, 64), ny=size(8, 64), nz=size(8, 64), ratio=round(rng.uniform(1.0, 6.0), 2),
                 jitter=round(rng.uniform(0.05, 0.2), 2))
        if kind == "corrector":
            c.update(passes=rng.randint(1, 3), precision=rng.choice(["", "mixed"]))
        return c
    if kind == "batch":
        lo = rng.randint(8, 20)
        return dict(kind=kind, systems=rng.randint(4, 32), nmin=lo, nmax=lo + rng.randint(4, 28), jitter=0.2,
                    passes=rng.randint(1, 3), precision=rng.choice(["", "mixed"]))
    if kind == "cavity":
        return dict(kind=kind, n=size(16, 160), steps=rng.randint(4, 10))
    if kind == "tgv":
        return dict(kind=kind, n=even(size(16, 72)), steps=rng.randint(2, 4), precision=rng.choice(["", "mixed"]))
    return dict(kind=kind, nx=even(size(16, 96)), ny=size(16, 72), nz=even(size(12, 48)), steps=2,
                precision=rng.choice(["", "mixed"]))


# ------------------------------------------------------------------------------ inputs
def _box(nx, ny, nz, periodic="", ratio=1.0, jitter=0.0, seed=0):
    """Mesh arrays of a box of near-cubic cells, graded by `ratio` (centre to wall cell
    size) in the directions with walls."""
    n = (nx, ny, nz)
    hi = tuple(v / max(n) for v in n)
    beta = math.acosh(math.sqrt(ratio)) if ratio > 1.0 else 0.0
    betas = tuple(0.0 if d in periodic else beta for d in "xyz")
    flags = tuple(d in periodic for d in "xyz")
    if jitter == 0.0:
        return vb.box_mesh_device(n, hi=hi, periodic=flags, beta=betas, two_d=nz == 1)
    pts = vm.jitter_interior(vm.box_points(n, hi=hi, beta=betas), n, jitter, seed)
    return vb.box_mesh_device(n, periodic=flags, points=pts, two_d=nz == 1)


def _internal_flux(m, seed):
    """Face flux of a seeded sum of 16 Fourier modes on the internal faces (the walls let nothing pass)."""
    nI = m["n_internal_faces"]
    rng = np.random.default_rng(seed)
    X = torch.from_numpy(m["Cf"][:nI]).to(DEV)
    u = torch.zeros_like(X)
    for _ in range(16):
        k = rng.integers(-4, 5, size=3)
        if not k.any():
            k[0] = 1
        a = rng.standard_normal(3) / float((k * k).sum())
        ph = rng.uniform(0, 2 * np.pi)
        c = torch.cos(2 * np.pi * (X[:, 0] * float(k[0]) + X[:, 1] * float(k[1]) + X[:, 2] * float(k[2])) + ph)
        for q in range(3):
            u[:, q] += float(a[q]) * c
    S = torch.from_numpy(m["Sf"][:nI]).to(DEV)
    return (u[:, 0] * S[:, 0] + u[:, 1] * S[:, 1] + u[:, 2] * S[:, 2]).cpu().numpy()


def _cell_sum(m, own_values, nei_values):
    """Per cell, the sum of a value of each internal face it owns and of one of each it neighbours."""
    nI, nC = m["n_internal_faces"], m["n_cells"]
    return (np.bincount(m["owner"][:nI], own_values, nC) + np.bincount(m["neighbour"], nei_values, nC))


def _pressure_system(case, seed):
    m = _box(case["nx"], case["ny"], case["nz"], case["periodic"], case["ratio"], case["jitter"], seed)
    nI = m["n_internal_faces"]
    upper = DT * m["magSf"][:nI] * m["ndc"][:nI]
    diag = -_cell_sum(m, upper, upper)
    diag[0] *= 2.0  # setReference on cell 0
    F = _internal_flux(m, seed)
    return m, diag, upper, _cell_sum(m, F, -F)


def _momentum_system(case, seed):
    """ddt + div(phi, U) - laplacian(nu, U) of one velocity component, central differences."""
    m = _box(case["nx"], case["ny"], case["nz"], case["periodic"], 2.0, 0.0, seed)
    nI = m["n_internal_faces"]
    F = _internal_flux(m, seed)
    h3 = m["V"].mean()
    speed = np.abs(F / m["magSf"][:nI]).max()
    dt = case["courant"] * h3 ** (1.0 / 3.0) / speed
    lap = 0.2 * h3 ** (2.0 / 3.0) / dt * m["magSf"][:nI] * m["ndc"][:nI]
    w = m["w"][:nI]
    lower = -w * F - lap
    upper = (1.0 - w) * F - lap
    diag = m["V"] / dt + _cell_sum(m, -lower, -upper)
    C = m["C"]
    rng = np.random.default_rng(seed + 1)
    u0 = np.sin(6 * C[:, 0] + rng.uniform(0, 6)) * np.cos(6 * C[:, 1]) + 0.05 * rng.standard_normal(m["n_cells"])
    return m, diag, upper, lower, (m["V"] / dt) * u0, u0


def _poisson_system(nx, ny, nz, ratio, jitter, seed):
    """Mesh, face diffusivity and divergence of a projection step on a graded, jittered box."""
    m = _box(nx, ny, nz, "", ratio, jitter, seed)
    F = _internal_flux(m, seed)
    gamma = 1.0 + 0.2 * np.random.default_rng(seed + 2).random(m["n_faces"])
    return m, gamma, _cell_sum(m, F, -F) / m["V"]


def _batch_systems(case, seed):
    sizes = np.random.default_rng(case["systems"] * 10000 + case["nmin"] * 100 + case["nmax"]).integers(
        case["nmin"], case["nmax"] + 1, case["systems"])  # the case's own, whatever the seed
    rng = np.random.default_rng(seed)
    return [_poisson_system(int(n), int(n), int(n), float(rng.uniform(1.0, 8.0)), case["jitter"], seed * 64 + q)
            for q, n in enumerate(sizes)]


def _assembly_inputs(case, seed):
    m = _box(case["nx"], case["ny"], case["nz"], "", case["ratio"], case["jitter"], seed)
    rng = np.random.default_rng(seed + 3)
    C = m["C"]
    psi = np.sin(5 * C[:, 0] + rng.uniform(0, 6)) * np.cos(4 * C[:, 1]) + C[:, 2] ** 2
    gamma = 1.0 + 0.2 * rng.random(m["n_faces"])
    bc_type = np.array([1, 0, 0, 0, 0, 0], np.int32)  # one side held at a value, the others insulated
    bc_value = rng.random(m["n_faces"] - m["n_internal_faces"])
    return m, gamma, psi, bc_type, bc_value


class _Flow:
    """A flow and its mesh, released together."""

    def __init__(self, m, case, steps, dt, U0, model=None, restart=False):
        self.mesh = vb.Mesh.from_arrays(m)
        self.flow = vb.Flow(self.mesh, case)
        if model is not None:
            self.flow.set_model(model)
        self.U0 = np.ascontiguousarray(U0)
        self.p0 = np.zeros(m["n_cells"])
        self.steps, self.dt, self.restart = steps, dt, restart
        self.flow.set_state(self.U0, self.p0)

    def __del__(self):
        self.flow.close()
        self.mesh.close()


# ------------------------------------------------------------------------------ state and pass
def _controls(case):
    return vb.SolverControls("PCG", "GAMG", 0.0, REL_TOL, 2000, precision=case.get("precision", ""),
                             reproducible=case.get("reproducible", False))


def _dev(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).to(DEV) for a in arrays]


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind)
    if kind == "pressure":
        m, diag, upper, b = _pressure_system(case, seed)
        s.update(mesh=vb.Mesh(m["n_cells"], m["owner"], m["neighbour"], m["magSf"], m["ndc"]),
                 ctrl=_controls(case), host=case["memory"] == "host")
        if s["host"]:
            s.update(diag=diag, upper=upper, b=b, x=np.zeros(m["n_cells"]))
        else:
            s["diag"], s["upper"], s["b"], s["x"] = _dev(diag, upper, b, np.zeros(m["n_cells"]))
    elif kind == "momentum":
        m, diag, upper, lower, b, u0 = _momentum_system(case, seed)
        s.update(mesh=vb.Mesh(m["n_cells"], m["owner"], m["neighbour"], m["magSf"], m["ndc"]),
                 ctrl=vb.SolverControls("PBiCGStab", "DILU", 1e-8, 0.0, 1000))
        s["diag"], s["upper"], s["lower"], s["b"], s["u0"], s["x"] = _dev(diag, upper, lower, b, u0, u0)
    elif kind == "corrector":
        m, gamma, div = _poisson_system(case["nx"], case["ny"], case["nz"], case["ratio"], case["jitter"], seed)
        s.update(mesh=vb.Mesh.from_arrays(m), gamma=gamma, div=div, p=np.zeros(m["n_cells"]), ctrl=_controls(case),
                 passes=case["passes"])
    elif kind == "batch":
        systems = _batch_systems(case, seed)
        meshes = [q[0] for q in systems]
        s.update(mesh=vb.Mesh.batch(meshes), ctrl=_controls(case), passes=case["passes"], refs=[0] * len(meshes))
        s["gamma"], s["div"] = _dev(workloads.batch_face_array(meshes, [q[1] for q in systems]),
                                    np.concatenate([q[2] for q in systems]))
        s["p"] = torch.zeros(s["mesh"].n_cells, dtype=torch.float64, device=DEV)
        s["flux"] = torch.zeros(s["mesh"].n_faces, dtype=torch.float64, device=DEV)
    elif kind == "assembly":
        m, gamma, psi, bc_type, bc_value = _assembly_inputs(case, seed)
        s.update(mesh=vb.Mesh.from_arrays(m), gamma=gamma, psi=psi, bc_type=bc_type, bc_value=bc_value)
    elif kind == "cavity":
        rng = np.random.default_rng(seed)
        m, c = workloads.lid_cavity(case["n"], Re=float(rng.uniform(100.0, 1000.0)))
        U0 = np.zeros((m["n_cells"], 3))
        U0[:, :2] = 0.02 * rng.standard_normal((m["n_cells"], 2))
        s["flow"] = _Flow(m, c, case["steps"], 1.0, U0, restart=True)
    elif kind == "tgv":
        m, c, U0 = workloads.taylor_green_flow(case["n"])
        X = 2 * np.pi * np.random.default_rng(seed).random(3) + m["C"]
        U0 += 0.05 * np.stack([np.sin(2 * X[:, 1]), np.sin(2 * X[:, 2]), np.sin(2 * X[:, 0])], 1)
        for key in ("p", "pFinal"):
            c[key] = dict(c[key], precision=case["precision"])
        s["flow"] = _Flow(m, c, case["steps"], DT, U0)
    elif kind == "channel":
        m, c, model, U0, dt = workloads.channel((case["nx"], case["ny"], case["nz"]), seed=seed)
        for key in ("p", "pFinal"):
            c[key] = dict(c[key], precision=case["precision"])
        s["flow"] = _Flow(m, c, case["steps"], dt, U0, model)
    else:
        raise ValueError(kind)
    if kind not in ("cavity", "tgv", "channel"):
        s["stream"] = torch.cuda.ExternalStream(s["mesh"].ctx.stream())
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "pressure":
        if s["host"]:
            s["x"][:] = 0.0
            vb.solve_ldu(s["mesh"], s["diag"], s["upper"], None, s["b"], s["x"], s["ctrl"])
            return s["x"]
        with torch.cuda.stream(s["stream"]):
            s["x"].zero_()
        vb.solve_ldu_device(s["mesh"], s["diag"].data_ptr(), s["upper"].data_ptr(), 0, s["b"].data_ptr(),
                            s["x"].data_ptr(), s["ctrl"])
        return s["x"]
    if kind == "momentum":
        with torch.cuda.stream(s["stream"]):
            s["x"].copy_(s["u0"])
        vb.solve_ldu_device(s["mesh"], s["diag"].data_ptr(), s["upper"].data_ptr(), s["lower"].data_ptr(),
                            s["b"].data_ptr(), s["x"].data_ptr(), s["ctrl"])
        return s["x"]
    if kind == "corrector":
        s["p"][:] = 0.0
        _, flux = vb.pressure_solve(s["mesh"], s["gamma"], s["div"], s["p"], s["ctrl"], n_non_orth=s["passes"] - 1,
                                    grad_scheme=1)
        return {"p": s["p"], "flux": flux}
    if kind == "batch":
        with torch.cuda.stream(s["stream"]):
            s["p"].zero_()
        vb.pressure_solve_device(s["mesh"], s["gamma"].data_ptr(), s["div"].data_ptr(), s["p"].data_ptr(), s["ctrl"],
                                 ref_cell=s["refs"], n_non_orth=s["passes"] - 1, grad_scheme=1,
                                 flux_ptr=s["flux"].data_ptr())
        return {"p": s["p"], "flux": s["flux"]}
    if kind == "assembly":
        eqn = vb.laplacian(s["mesh"], s["gamma"], s["psi"], s["bc_type"], s["bc_value"], grad_scheme=1)
        eqn["grad"] = vb.grad(s["mesh"], s["psi"], s["bc_type"], s["bc_value"], scheme=1)
        return eqn
    f = s["flow"]
    if f.restart:  # a steady request starts from its initial field; a transient flow goes on
        f.flow.set_state(f.U0, f.p0)
    for _ in range(f.steps):
        f.flow.step(f.dt)
    U, p, phi = f.flow.state()
    return {"U": U, "p": p, "phi": phi}


# ------------------------------------------------------------------------------ work and tolerance
def _cells(case):
    if case["kind"] == "batch":
        mid = 0.5 * (case["nmin"] + case["nmax"])
        return case["systems"] * (mid ** 3 + mid * (case["nmax"] - case["nmin"]) ** 2 / 4.0)
    if case["kind"] == "cavity":
        return case["n"] ** 2
    if case["kind"] == "tgv":
        return case["n"] ** 3
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """Inputs once and outputs once (FP64, int32 addressing), F = faces of a box, N = cells; a flow does
    so every step.  Operations: one residual evaluation (a pass cannot know its answer without one)."""
    N = _cells(case)
    F = (2 if case["kind"] == "cavity" or case.get("nz") == 1 else 3) * N
    kind = case["kind"]
    if kind == "pressure":     # diag, b, x out; upper; owner and neighbour
        b = 8 * (3 * N + F) + 8 * F
    elif kind == "momentum":   # diag, b, x in and out; upper and lower; addressing
        b = 8 * (4 * N + 2 * F) + 8 * F
    elif kind in ("corrector", "batch"):  # gamma, geometry (Sf, d, corr, |S|, ndc, w), flux out; div, V, p out
        b = 8 * (3 * N + 14 * F) + 8 * F
    elif kind == "assembly":   # gamma, geometry, upper, ffc; psi, V, diag, source, grad
        b = 8 * (7 * N + 15 * F) + 8 * F
    else:                      # U and p in and out, an old level in 3D; phi in and out, geometry; addressing
        b = case["steps"] * (8 * (12 * N + 9 * F) + 8 * F)
    return {"bytes": b, "flops": case.get("steps", 1) * 2 * (N + 2 * F)}


def tolerance(case):
    """About four times what was measured: a converged solve's distance from the 64-bit solution (6e-8 at
    relTol 1e-8, 7e-9 for the momentum solve at 1e-8), the assembly's from 64-bit sums in another order
    (2.5e-16), a flow's change under a last-bit change of its initial field (1.3e-11 in FP64, 5e-7 with the
    FP32 V-cycle, both in p)."""
    kind = case["kind"]
    if case.get("reproducible"):
        return "exact"  # what the mode promises
    if kind in ("pressure", "corrector", "batch"):
        return {"rel": 2.5e-7}
    if kind == "momentum":
        return {"rel": 3e-8}
    if kind == "assembly":
        return {"rel": 2e-15}
    return {"rel": 2e-6 if case.get("precision") == "mixed" else 1e-10}


# ------------------------------------------------------------------------------ 64-bit answers
def _csr(m, diag, upper, lower):
    nI, n = m["n_internal_faces"], m["n_cells"]
    own, nei = (torch.from_numpy(np.asarray(a[:nI], np.int64)).to(DEV) for a in (m["owner"], m["neighbour"]))
    rng = torch.arange(n, device=DEV)
    i = torch.stack([torch.cat([rng, own, nei]), torch.cat([rng, nei, own])])
    v = torch.cat([torch.from_numpy(diag).to(DEV), torch.from_numpy(upper).to(DEV), torch.from_numpy(lower).to(DEV)])
    return torch.sparse_coo_tensor(i, v, (n, n)).coalesce().to_sparse_csr()


def _neumann_solve(m, upper, b, system=None, count=1, refs=(0,)):
    """x of the symmetric system with zero row sums whose reference cells' diagonals are doubled: the row sums
    give x there exactly, x_ref = sum(b) / (its own diagonal); what is left is singular and solved by
    diagonal CG with each system's mean projected out, to the last digits.  `system`: each cell's system."""
    n = m["n_cells"]
    d0 = -_cell_sum(m, upper, upper)
    A = _csr(m, -d0, -upper, -upper)  # positive semi-definite
    system = torch.zeros(n, dtype=torch.int64, device=DEV) if system is None else system
    refs = torch.tensor(list(refs), device=DEV)
    size = torch.bincount(system, minlength=count).double()

    def per(v):
        return torch.zeros(count, dtype=torch.float64, device=DEV).index_add_(0, system, v)

    def project(v):
        return v - (per(v) / size)[system]

    rhs = -b.clone()
    if count == 1:
        total = torch.tensor([math.fsum(rhs.cpu().tolist())], dtype=torch.float64, device=DEV)
    else:
        total = per(rhs)
    D = torch.from_numpy(-d0).to(DEV)
    xref = total / D[refs]
    rhs[refs] -= total
    rhs = project(rhs)
    x = torch.zeros_like(rhs)
    r = rhs.clone()
    z = project(r / D)
    p, rz = z.clone(), r @ z
    r0 = float(r.norm())
    for k in range(20000):
        Ap = A @ p
        a = rz / (p @ Ap)
        x += a * p
        r -= a * Ap
        if k % 25 == 24 and float(r.norm()) <= 1e-15 * r0:
            break
        z = project(r / D)
        new = r @ z
        p = z + (new / rz) * p
        rz = new
    return x + (xref - x[refs])[system]


def _ls_gradient(m, psi, psi_b, value):
    """Weighted least squares over each cell's faces; `value`: the boundary faces that hold a value, the
    others a zero normal gradient."""
    nI, n = m["n_internal_faces"], m["n_cells"]
    own = torch.from_numpy(m["owner"].astype(np.int64)).to(DEV)
    nei = torch.from_numpy(m["neighbour"].astype(np.int64)).to(DEV)
    d = torch.from_numpy(m["d"]).to(DEV)
    nrm = torch.from_numpy(m["Sf"] / m["magSf"][:, None]).to(DEV)[nI:]
    db = d[nI:]
    nd = torch.maximum((nrm * db).sum(1), 0.05 * db.norm(dim=1))
    vb_ = torch.where(value[:, None], db, nrm * nd[:, None])
    dp_b = torch.where(value, psi_b - psi[own[nI:]], torch.zeros_like(nd))
    rows = torch.cat([own[:nI], nei, own[nI:]])
    v = torch.cat([d[:nI], d[:nI], vb_])
    dpi = psi[nei] - psi[own[:nI]]
    dp = torch.cat([dpi, dpi, dp_b])
    wgt = 1.0 / (v * v).sum(1)
    M = torch.zeros(n, 3, 3, dtype=torch.float64, device=DEV).index_add_(0, rows, v[:, :, None] * v[:, None, :] * wgt[:, None, None])
    if m["two_d"]:
        M[:, m["empty_dir"], m["empty_dir"]] += 1.0
    rhs = torch.zeros(n, 3, dtype=torch.float64, device=DEV).index_add_(0, rows, v * (dp * wgt)[:, None])
    g = (torch.linalg.inv(M) @ rhs[:, :, None])[:, :, 0]
    if m["two_d"]:
        g[:, m["empty_dir"]] = 0.0
    return g


def _laplacian_terms(m, gamma, psi, psi_b, value):
    """upper, diag, source and face correction of fvm::laplacian, and the gradient they use."""
    nI, n = m["n_internal_faces"], m["n_cells"]
    own = torch.from_numpy(m["owner"][:nI].astype(np.int64)).to(DEV)
    nei = torch.from_numpy(m["neighbour"].astype(np.int64)).to(DEV)
    g = _ls_gradient(m, psi, psi_b, value)
    gs = torch.from_numpy(gamma * m["magSf"]).to(DEV)
    w = torch.from_numpy(m["w"][:nI]).to(DEV)[:, None]
    corr = torch.from_numpy(m["corrVecs"][:nI]).to(DEV)
    ffc = torch.zeros(m["n_faces"], dtype=torch.float64, device=DEV)
    ffc[:nI] = gs[:nI] * (corr * (w * g[own] + (1.0 - w) * g[nei])).sum(1)
    upper = gs[:nI] * torch.from_numpy(m["ndc"][:nI]).to(DEV)
    zero = torch.zeros(n, dtype=torch.float64, device=DEV)
    diag = zero.index_add(0, own, -upper).index_add(0, nei, -upper)
    source = zero.index_add(0, own, -ffc[:nI]).index_add(0, nei, ffc[:nI])
    return upper, diag, source, ffc, gs, g


def _union(meshes):
    """One mesh of several: cells in system order, all internal faces before all boundary faces."""
    base = np.cumsum([0] + [q["n_cells"] for q in meshes])
    out = dict(n_cells=int(base[-1]), n_internal_faces=sum(q["n_internal_faces"] for q in meshes),
               n_faces=sum(q["n_faces"] for q in meshes), two_d=False, empty_dir=-1,
               V=np.concatenate([q["V"] for q in meshes]),
               neighbour=np.concatenate([q["neighbour"] + b for q, b in zip(meshes, base)]),
               owner=workloads.batch_face_array(meshes, [q["owner"] + b for q, b in zip(meshes, base)]))
    for key in ("Sf", "magSf", "d", "w", "ndc", "corrVecs"):
        out[key] = workloads.batch_face_array(meshes, [q[key] for q in meshes])
    return out, base


def _exact_corrector(meshes, gammas, divs, passes):
    m, base = _union(meshes)
    nI = m["n_internal_faces"]
    gamma = workloads.batch_face_array(meshes, gammas)
    system = torch.repeat_interleave(torch.arange(len(meshes), device=DEV),
                                     torch.tensor([q["n_cells"] for q in meshes], device=DEV))
    own, nei = (torch.from_numpy(a.astype(np.int64)).to(DEV) for a in (m["owner"], m["neighbour"]))
    vol = torch.from_numpy(m["V"] * np.concatenate(divs)).to(DEV)
    value = torch.zeros(m["n_faces"] - nI, dtype=torch.bool, device=DEV)
    p = torch.zeros(m["n_cells"], dtype=torch.float64, device=DEV)
    for _ in range(passes):
        upper, _, source, ffc, _, _ = _laplacian_terms(m, gamma, p, p[own[nI:]], value)
        p = _neumann_solve(m, upper.cpu().numpy(), source + vol, system, len(meshes), base[:-1].tolist())
    flux = ffc.clone()
    flux[:nI] += upper * (p[nei] - p[own[:nI]])
    return {"p": p, "flux": flux}


def exact(case, seed):
    """The inputs' meshes come from the package; everything computed from them is plain torch in 64 bits.
    The flow steps are None: a step is a sequence of solves whose stopping tests decide its digits."""
    kind = case["kind"]
    if kind == "pressure":
        m, _, upper, b = _pressure_system(case, seed)
        return _neumann_solve(m, upper, torch.from_numpy(b).to(DEV))
    if kind == "momentum":
        m, diag, upper, lower, b, u0 = _momentum_system(case, seed)
        A, D = _csr(m, diag, upper, lower), torch.from_numpy(diag).to(DEV)
        b, x = torch.from_numpy(b).to(DEV), torch.from_numpy(u0).to(DEV)
        for _ in range(400):  # diagonally dominant: Jacobi steps contract to the last digits
            x = x + (b - A @ x) / D
        return x
    if kind == "corrector":
        m, gamma, div = _poisson_system(case["nx"], case["ny"], case["nz"], case["ratio"], case["jitter"], seed)
        return _exact_corrector([m], [gamma], [div], case["passes"])
    if kind == "batch":
        systems = _batch_systems(case, seed)
        return _exact_corrector([q[0] for q in systems], [q[1] for q in systems], [q[2] for q in systems],
                                case["passes"])
    if kind == "assembly":
        m, gamma, psi, bc_type, bc_value = _assembly_inputs(case, seed)
        nI = m["n_internal_faces"]
        held = np.zeros(m["n_faces"] - nI, bool)
        for q, t in enumerate(bc_type):
            a = int(m["patch_start"][q]) - nI
            held[a:a + int(m["patch_size"][q])] = t == 1
        value = torch.from_numpy(held).to(DEV)
        psi_t, val = torch.from_numpy(psi).to(DEV), torch.from_numpy(bc_value).to(DEV)
        own_b = torch.from_numpy(m["owner"][nI:].astype(np.int64)).to(DEV)
        psi_b = torch.where(value, val, psi_t[own_b])
        upper, diag, source, ffc, gs, g = _laplacian_terms(m, gamma, psi_t, psi_b, value)
        gic = torch.where(value, -torch.from_numpy(m["ndc"][nI:]).to(DEV), torch.zeros_like(val))
        return {"diag": diag, "upper": upper, "source": source, "internalCoeffs": gs[nI:] * gic,
                "boundarySource": gs[nI:] * gic * val, "ffc": ffc, "hasFfc": None, "grad": g}
    return None
