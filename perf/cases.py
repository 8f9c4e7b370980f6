"""The work whose time this repository tracks, through its public entry points.

Each case is one timestep, or one spectral solve, as a user's program issues
it: the fused rigid-body engine (FP32 and FP64, one case or many of uneven
sizes), the soft-sphere engine, the drop-in spectral solvers, the drop-in step
loop and the remeshed-particle advection. Grid sizes are those of the
repository's configurations, tests and benchmark (256 x 128 to 2048 x 1024
cells, z by r), with odd ones beside them.

`exact` restates each pass in 64-bit torch: the spectral solve as a cosine or
Fourier transform in z and a tridiagonal elimination in r, the rest as array
expressions.
"""
import math

import numpy as np
import torch

from pyaxisymflow_gb300.engine import RigidBodyCase, RigidEnsemble
from pyaxisymflow_gb300.kernels.advect_particle import advect_vorticity_via_particles
from pyaxisymflow_gb300.kernels.FastDiagonalisationStokesSolver import (
    FastDiagonalisationStokesSolver)
from pyaxisymflow_gb300.simulation import RigidSphereSimulation, SoftCase, SoftSphereEngine

NEUMANN = "homogenous_neumann_along_z_and_r"
PERIODIC_Z = "homogenous_neumann_along_r_and_periodic_along_z"
EPS = float(np.finfo(float).eps)


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def listed():
    return [
        # one body on the smallest grid that is served: latency and launches
        dict(name="rigid_f32_256x128", kind="rigid", precision="f32", grids="256x128",
             sediment=False, dense=False),
        # a handful of requests of uneven size and shape (sphere, spheroid, torus) advanced together
        dict(name="rigid_f32_mixed5", kind="rigid", precision="f32",
             grids="256x128,512x256*2,768x384,1024x512", sediment=False, dense=False),
        # the 64 freely sedimenting spheres of the benchmark
        dict(name="sediment_f32_64", kind="rigid", precision="f32",
             grids="256x128*14,512x256*14,768x384*12,1024x512*24", sediment=True, dense=False),
        # a grid without a cosine-transform plan: dense z products
        dict(name="rigid_f32_500x252", kind="rigid", precision="f32", grids="500x252",
             sediment=False, dense=False),
        # plain FP64 flow past a sphere, the configuration the CPU reference runs
        dict(name="rigid_f64_512x256", kind="rigid", precision="f64", grids="512x256",
             sediment=False, dense=False),
        # the same flow with the reference's own eigenvector products in z
        dict(name="rigid_f64_dense_512x256", kind="rigid", precision="f64", grids="512x256",
             sediment=False, dense=True),
        # a plain FP64 ensemble of sedimenting spheres
        dict(name="sediment_f64_8", kind="rigid", precision="f64",
             grids="256x128*2,512x256*2,768x384*2,1024x512*2", sediment=True, dense=False),
        # the soft sphere of the reference's example on that example's grid
        dict(name="soft_f64_256x128", kind="soft", nz=256, nr=128, r_ball=0.15, dct=False),
        # the soft sphere in oscillatory streaming at the configured size
        dict(name="soft_f64_1024x512", kind="soft", nz=1024, nr=512, r_ball=0.1, dct=False),
        # isolated mixed-precision stream-function solves, periodic in z
        dict(name="solve_f32_2048x1024", kind="solve", precision="f32", nz=2048, nr=1024,
             bc=PERIODIC_Z),
        # the reference's driver loop through the drop-in callables, odd radial size
        dict(name="dropin_f64_384x201", kind="dropin", nz=384, nr=201),
        # vorticity advection by remeshed particles
        dict(name="remesh_f64_1024x512", kind="remesh", nz=1024, nr=512),
    ]


def _log_int(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / multiple)) * multiple))


def _cosine_nz(rng):
    """An nz with a cosine-transform plan between 128 and 1024."""
    return rng.choice([128, 144, 192, 216, 256, 288, 324, 384, 432, 512, 576, 648, 768, 864, 972,
                       1024])


def draw(rng):
    kind = rng.choice(["rigid_f32", "rigid_f32", "rigid_f32", "rigid_f32_odd", "rigid_f64",
                       "rigid_f64", "soft", "solve_f32", "solve_f64", "solve_f64", "dropin",
                       "remesh"])
    if kind in ("rigid_f32", "rigid_f64"):
        n = _log_int(rng, 1, 24 if kind == "rigid_f32" else 4)
        grids = []
        for _ in range(n):
            nz = _cosine_nz(rng)
            grids.append("%dx%d" % (nz, max(64, nz // 2 // 4 * 4 + rng.choice([0, 0, 0, 4, -4]))))
        return dict(kind="rigid", precision=kind[-3:], grids=",".join(grids),
                    sediment=rng.random() < 0.5,
                    dense=kind == "rigid_f64" and rng.random() < 0.5)
    if kind == "rigid_f32_odd":
        n = _log_int(rng, 1, 6)
        grids = ["%dx%d" % (_log_int(rng, 132, 1000, 4), _log_int(rng, 64, 500, 4))
                 for _ in range(n)]
        return dict(kind="rigid", precision="f32", grids=",".join(grids),
                    sediment=rng.random() < 0.5, dense=True)
    if kind == "soft":
        nr = _log_int(rng, 64, 384, 4)
        return dict(kind="soft", nz=2 * nr, nr=nr, r_ball=round(rng.uniform(0.1, 0.15), 4),
                    dct=False)
    if kind == "solve_f32":
        return dict(kind="solve", precision="f32", nz=_log_int(rng, 128, 1400, 4),
                    nr=_log_int(rng, 64, 700, 4), bc=rng.choice([NEUMANN, PERIODIC_Z]))
    if kind == "solve_f64":
        return dict(kind="solve", precision="f64", nz=_log_int(rng, 100, 1024),
                    nr=_log_int(rng, 50, 512), bc=rng.choice([NEUMANN, PERIODIC_Z]))
    if kind == "dropin":
        return dict(kind="dropin", nz=_log_int(rng, 64, 700), nr=_log_int(rng, 40, 400))
    return dict(kind="remesh", nz=_log_int(rng, 100, 1400), nr=_log_int(rng, 50, 700))


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

def _grids(text):
    out = []
    for part in text.split(","):
        size, _, count = part.partition("*")
        nz, nr = (int(x) for x in size.split("x"))
        out += [(nz, nr)] * int(count or 1)
    return out


def _rings(nr, nz, dx, seed, strength, n=8):
    """Seeded axisymmetric Gaussian vortex rings plus small noise (float64, on
    the host): odd in r like a vorticity field."""
    rng = np.random.default_rng(seed)
    z = (np.arange(nz) + 0.5) * dx
    r = (np.arange(nr) + 0.5) * dx
    rad = rng.uniform(0.06, 0.2, n) * nr * dx
    zc, rc = rng.uniform(0.1, 0.9, n) * nz * dx, rng.uniform(0.2, 0.8, n) * nr * dx
    amp = strength * rng.standard_normal(n)
    fz = np.exp(-((z[None, :] - zc[:, None]) / rad[:, None]) ** 2)
    fr = (amp / rc)[:, None] * r[None, :] * np.exp(-((r[None, :] - rc[:, None])
                                                     / rad[:, None]) ** 2)
    return fr.T @ fz + 1e-6 * strength * rng.standard_normal((nr, nz))


def _bodies(case, seed):
    """The rigid bodies of a case (RigidBodyCase) and their initial vorticity."""
    rng = np.random.default_rng(seed)
    cases, w0 = [], []
    for k, (nz, nr) in enumerate(_grids(case["grids"])):
        dx = 2.0 / nz
        radius = float(rng.uniform(0.08, 0.12))
        if case["sediment"]:
            c = RigidBodyCase(nz=nz, nr=nr, dx=dx, r_sphere=radius, z_cm=1.5, U0=0.0,
                              ramp=False, sediment=True,
                              Re=float(np.exp(rng.uniform(np.log(10.0), np.log(500.0)))),
                              rho_s=float(rng.uniform(1.5, 4.0)))
        else:
            body = ("sphere", "spheroid", "torus")[k % 3]
            c = RigidBodyCase(nz=nz, nr=nr, dx=dx, r_sphere=radius, z_cm=0.5, ramp=False,
                              Re=float(np.exp(rng.uniform(np.log(10.0), np.log(500.0)))),
                              body=body, aspect=float(rng.uniform(0.5, 2.0)),
                              torus_R=0.25 if body == "torus" else 0.0)
        cases.append(c)
        w0.append(_rings(nr, nz, dx, seed * 1000 + k, 2.0))
    return cases, w0


def _soft_case(case):
    """Oscillatory streaming around a soft sphere, U(t) = 0.1 cos(2 pi t), shear
    modulus 1e-3, on z in [0, 1]."""
    omega = 2 * math.pi
    r = case["r_ball"]
    e = 0.1 / (r * omega)
    return SoftCase(nz=case["nz"], nr=case["nr"], dx=1.0 / case["nz"], z_cm=0.5, r_ball=r,
                    freq=1.0, e=e, cauchy=e * (r * omega) ** 2 / 1e-3)


def _sphere(case, seed):
    nz = case["nz"]
    rng = np.random.default_rng(seed)
    return RigidBodyCase(nz=nz, nr=case["nr"], dx=2.0 / nz, ramp=False, z_cm=0.5,
                         r_sphere=float(rng.uniform(0.08, 0.12)))


_solvers = {}


def _solver(case):
    """A program solves on one grid many times: one solver per grid is kept."""
    key = (case["nr"], case["nz"], case["bc"], case["precision"])
    if key not in _solvers:
        _solvers.clear()
        _solvers[key] = FastDiagonalisationStokesSolver(
            case["nr"], case["nz"], 1.0 / case["nr"], bc_type=case["bc"],
            real_dtype=np.float32 if case["precision"] == "f32" else np.float64)
    return _solvers[key]


def _cuda(a):
    return torch.tensor(np.asarray(a), dtype=torch.float64, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "rigid":
        cases, w0 = _bodies(case, seed)
        ens = RigidEnsemble(cases, precision=case["precision"], initial_vorticity=w0,
                            dct=False if case["dense"] else None)
        ens.capture()
        if len(cases) > 15:
            # the vorticity of every case; the other fields are recomputed from it each step
            out = {"vorticity": ens.omega_arena}
        else:
            out = {n: [f[n] for f in ens.fields] for n in ("omega", "psi", "u_z", "u_r")}
        if case["precision"] == "f64":
            out["t_dt_cd_steps"] = ens.state[:, :4]
        return dict(kind=kind, ens=ens, out=out)
    if kind == "soft":
        eng = SoftSphereEngine(_soft_case(case))
        eng.vorticity.copy_(_cuda(_rings(case["nr"], case["nz"], 1.0 / case["nz"], seed, 0.02)))
        eng.capture()
        out = {n: getattr(eng, n) for n in ("vorticity", "psi", "u_z", "u_r", "eta1", "eta2",
                                            "ball_phi", "ball_char_func")}
        out["state"] = eng.state[:3]
        return dict(kind=kind, eng=eng, out=out)
    if kind == "solve":
        solver = _solver(case)
        rhs = _cuda(_rings(case["nr"], case["nz"], 1.0 / case["nr"], seed, 1.0, n=32))
        return dict(kind=kind, solver=solver, rhs=rhs, psi=torch.zeros_like(rhs))
    if kind == "dropin":
        c = _sphere(case, seed)
        return dict(kind=kind, sim=RigidSphereSimulation(
            c, vorticity=_rings(c.nr, c.nz, c.dx, seed, 2.0)))
    dx, w, uz, ur = _remesh_inputs(case, seed)
    z = (np.arange(case["nz"]) + 0.5) * dx
    r = (np.arange(2 * case["nr"]) + 0.5) * dx
    Z, R = (_cuda(a) for a in np.meshgrid(z, r))
    return dict(kind=kind, zp=Z.clone(), rp=R.clone(), vp=torch.zeros_like(Z), w=_cuda(w), Z=Z,
                R=R, nr=case["nr"], uz=_cuda(uz), ur=_cuda(ur), dx=dx, dt=0.5 * dx)


def _remesh_inputs(case, seed):
    """Vorticity and a velocity with |u| dt <= 0.5 dx, as under a CFL limit."""
    nr, nz = case["nr"], case["nz"]
    dx = 1.0 / nz
    rng = np.random.default_rng(seed)
    w = _rings(nr, nz, dx, seed, 1.0)
    uz, ur = (np.clip(_rings(nr, nz, dx, seed + q, 0.5), -1, 1) + rng.uniform(-0.01, 0.01)
              for q in (1, 2))
    return dx, w, np.clip(uz, -1, 1), np.clip(ur, -1, 1)


def run(state):
    kind = state["kind"]
    if kind == "rigid":
        state["ens"].replay()
        return state["out"]
    if kind == "soft":
        state["eng"].replay()
        return state["out"]
    if kind == "solve":
        state["solver"].solve(state["psi"], state["rhs"])
        return state["psi"]
    if kind == "dropin":
        s = state["sim"]
        s.step()
        return dict(vorticity=s.vorticity, psi=s.psi, u_z=s.u_z, u_r=s.u_r, dt=s.dt, Cd=s.Cd)
    s = state
    advect_vorticity_via_particles(s["zp"], s["rp"], s["vp"], s["w"], s["Z"], s["R"], s["nr"],
                                   s["uz"], s["ur"], s["dx"], s["dt"])
    return s["w"]


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------

def _fft_flops(n):
    return 2.5 * n * math.log2(n)


def work(case):
    kind = case["kind"]
    if kind == "rigid":
        b = 8 if case["precision"] == "f64" else 4
        total_b = total_f = 0.0
        bases = set()
        for nz, nr in _grids(case["grids"]):
            n = nr * nz
            # omega, psi (a float pair in FP32) in and out, u_z, u_r out, the
            # body mask in (and out where the body moves), 1 / eigenvalues
            words = (2 + (4 if b == 4 else 2) + 2 + 1 + (1 if case["sediment"] else 0) + 1)
            total_b += words * b * n
            z = 2 * nr * _fft_flops(nz) if not case["dense"] and _cosine(nz) else 4.0 * n * nz
            # radial products, z transforms or products, about 150 per cell of stencils
            total_f += 4.0 * n * nr + z + 150.0 * n
            if (nz, nr) not in bases:
                bases.add((nz, nr))
                total_b += 2 * b * nr * nr
        return dict(bytes=total_b, flops=total_f)
    nz, nr = case["nz"], case["nr"]
    n = nr * nz
    if kind == "soft":
        # omega, eta1, eta2, level set in and out, psi, u_z, u_r, masks out,
        # 1 / eigenvalues; the four products and about 500 per cell
        return dict(bytes=8.0 * n * 14 + 16.0 * (nr * nr + nz * nz),
                    flops=4.0 * n * (nr + nz) + 500.0 * n)
    if kind == "solve":
        e = 4 if case["precision"] == "f32" else 8
        return dict(bytes=16.0 * n + e * (n + 2.0 * nr * nr + 2.0 * nz * nz),
                    flops=4.0 * n * (nr + nz) * (2 if case["precision"] == "f32" else 1))
    if kind == "dropin":
        return dict(bytes=8.0 * n * 7 + 16.0 * (nr * nr + nz * nz),
                    flops=4.0 * n * (nr + nz) + 150.0 * n)
    return dict(bytes=8.0 * n * 4 + 16.0 * 2 * n * 2, flops=400.0 * n)


def _cosine(nz):
    for f in (2, 3):
        while nz % f == 0:
            nz //= f
    return nz == 1


# --------------------------------------------------------------------------
# the same passes in 64 bits
# --------------------------------------------------------------------------

def _coords(nr, nz, dx):
    z = (torch.arange(nz, dtype=torch.float64, device="cuda") + 0.5) * dx
    r = (torch.arange(nr, dtype=torch.float64, device="cuda") + 0.5) * dx
    return z.view(1, nz).expand(nr, nz), r.view(nr, 1).expand(nr, nz)


def _x_stokes(w, dx, periodic):
    """psi of -psi_rr - psi_zz + psi_r / r = r w, Neumann at the outer r edge
    (psi = 0 on the axis), Neumann or periodic in z."""
    nr, nz = w.shape
    r = (torch.arange(nr, dtype=torch.float64, device=w.device) + 0.5) * dx
    rhs = w * r.view(nr, 1)
    k = torch.arange(nz, dtype=torch.float64, device=w.device)
    if periodic:
        lam = (2 - 2 * torch.cos(2 * math.pi * k / nz)) / dx ** 2
        f = torch.view_as_real(torch.fft.fft(rhs, dim=1)).movedim(-1, 0).contiguous()
    else:
        # the products of k and 2 j + 1 reduced modulo 4 nz, so that the angles are exact
        kj = torch.outer(torch.arange(nz), 2 * torch.arange(nz) + 1) % (4 * nz)
        basis = torch.cos(math.pi / (2 * nz) * kj.double()).to(w.device) * math.sqrt(2 / nz)
        basis[0] *= math.sqrt(0.5)
        lam = (2 - 2 * torch.cos(math.pi * k / nz)) / dx ** 2
        f = (rhs @ basis.T).unsqueeze(0)
    lo = -1 / dx ** 2 - 0.5 / dx / r     # psi_{i-1}
    up = -1 / dx ** 2 + 0.5 / dx / r     # psi_{i+1}
    di = torch.full((nr,), 2 / dx ** 2, dtype=torch.float64, device=w.device)
    di[-1] = 1 / dx ** 2
    lo[-1] = -1 / dx ** 2
    lo, up, di = lo.tolist(), up.tolist(), di.tolist()
    cp, sol = [], []
    for i in range(nr):
        if i == 0:
            den = lam + di[0]
            sol.append(f[:, 0] / den)
        else:
            den = (lam + di[i]) - lo[i] * cp[-1]
            sol.append((f[:, i] - lo[i] * sol[-1]) / den)
        cp.append(up[i] / den)
    for i in range(nr - 2, -1, -1):
        sol[i] = sol[i] - cp[i] * sol[i + 1]
    y = torch.stack(sol, dim=1)
    if periodic:
        return torch.fft.ifft(torch.view_as_complex(y.movedim(0, -1).contiguous()), dim=1).real
    return y[0] @ basis


def _x_velocity(psi, R, dx):
    uz, ur = torch.empty_like(psi), torch.empty_like(psi)
    uz[1:-1] = (psi[2:] - psi[:-2])
    uz[0] = -psi[2] + 4 * psi[1] - 3 * psi[0]
    uz[-1] = psi[-3] - 4 * psi[-2] + 3 * psi[-1]
    ur[:, 1:-1] = -(psi[:, 2:] - psi[:, :-2])
    ur[:, 0] = psi[:, 2] - 4 * psi[:, 1] + 3 * psi[:, 0]
    ur[:, -1] = -(psi[:, -3] - 4 * psi[:, -2] + 3 * psi[:, -1])
    return uz / (2 * dx) / R, ur / (2 * dx) / R


def _x_kill(w, Z, R, width, dx):
    def taper(x):
        return torch.sin(math.pi * (x - 0.5 * dx) / 2 / (width - 1) / dx)
    w[:, :width] = taper(Z[:, :width]) * w[:, width - 1].clone().view(-1, 1)
    w[:, -width:] = taper(1 - Z[:, -width:]) * w[:, -width].clone().view(-1, 1)
    w[-width:] = taper(1 - R[-width:]) * w[-width].clone()
    w[0] = 0.0


def _x_heaviside(phi, width):
    blend = 0.5 * (1 + phi / width + torch.sin(math.pi * phi / width) / math.pi)
    return torch.where(phi >= width, 1.0, torch.where(phi.abs() < width, blend, 0.0))


def _x_penalise(w, uz, ur, chi, lam_dt, target, dx):
    """Penalised velocities; adds the vorticity of the change to w."""
    pz = (uz + lam_dt * chi * target) / (1 + lam_dt * chi)
    pr = ur / (1 + lam_dt * chi)
    dz, dr = pz - uz, pr - ur
    w[1:-1, 1:-1] += ((dr[1:-1, 2:] - dr[1:-1, :-2]) - (dz[2:, 1:-1] - dz[:-2, 1:-1])) / (2 * dx)
    return pz, pr


def _x_advect(w, uz, ur, dt, dx):
    """One conservative third-order upwind step on the domain mirrored at the axis."""
    nr, nz = w.shape
    g = 2

    def mirrored(f, sign):
        return torch.cat([sign * f[:g + 1].flip(0), f])

    def faces(q, u):
        # faces between cells 1|2, 2|3, ... along axis 1
        left = q[:, 2:-1] / 3 + 5 * q[:, 1:-2] / 6 - q[:, :-3] / 6
        right = q[:, 1:-2] / 3 + 5 * q[:, 2:-1] / 6 - q[:, 3:] / 6
        return torch.where(u[:, 1:-2] > -u[:, 2:-1], left, right)

    fx = faces(w * uz, uz)
    m, mu = mirrored(w, -1.0), mirrored(ur, -1.0)
    fy = faces((m * mu).T, mu.T).T
    div = torch.zeros_like(w)
    div[:, g:-g] = fx[:, 1:] - fx[:, :-1]
    dy = (fy[1:] - fy[:-1])[1:]
    div[:-g, g:-g] += dy[:, g:-g]
    div[-g:] = 0
    w -= dt / dx * div


def _x_diffuse(w, R, nu, dt, dx):
    def op(f):
        c = f[1:-1, 1:-1]
        return ((f[2:, 1:-1] + f[:-2, 1:-1] + f[1:-1, 2:] + f[1:-1, :-2] - 4 * c) / dx ** 2
                + (f[2:, 1:-1] - f[:-2, 1:-1]) / (2 * dx) / R[1:-1, 1:-1]
                - c / R[1:-1, 1:-1] ** 2)
    mid = w.clone()
    mid[1:-1, 1:-1] += 0.5 * nu * dt * op(w)
    w[1:-1, 1:-1] += nu * dt * op(mid)


def _x_rigid_step(c, w0):
    """The first step of a rigid-body case: (vorticity, psi, u_z, u_r, [t, dt, Cd, steps])."""
    dx = c.dx
    Z, R = _coords(c.nr, c.nz, dx)
    w = _cuda(w0)
    chi = _x_heaviside(_cuda(c.level_set(Z.cpu().numpy(), R.cpu().numpy())), dx * 2 ** 0.5)
    _x_kill(w, Z, R, c.kill_width, dx)
    psi = _x_stokes(w, dx, False)
    uz, ur = _x_velocity(psi, R, dx)
    uz = uz + c.U0
    umax = float((uz.abs() + ur.abs()).max())
    dt = min(0.9 * dx ** 2 / 4 / c.nu, c.cfl * dx / (umax + EPS))
    pz, pr = _x_penalise(w, uz, ur, chi, c.lam * dt, 0.0, dx)
    cd = (2 * 2 * math.pi * dx * dx * c.lam * float((R * chi * pz).sum())
          / (math.pi * c.r_sphere ** 2))
    _x_advect(w, pz, pr, dt, dx)
    _x_diffuse(w, R, c.nu, dt, dx)
    return w, psi, pz, pr, [dt, dt, cd, 1.0]


def _x_remesh(case, seed):
    dx, w, uz, ur = _remesh_inputs(case, seed)
    nr, nz = case["nr"], case["nz"]
    w, uz, ur = _cuda(w), _cuda(uz), _cuda(ur)
    dt = 0.5 * dx
    cat = torch.cat
    wd, ud, vd = (cat([s * f.flip(0), f]) for f, s in ((w, -1.0), (uz, 1.0), (ur, -1.0)))
    # displacements in cells, then each particle's 4 x 4 stencil
    jx = torch.arange(nz, device="cuda", dtype=torch.float64).view(1, nz) + ud * dt / dx
    iy = torch.arange(2 * nr, device="cuda", dtype=torch.float64).view(-1, 1) + vd * dt / dx

    def mp4(t):
        t = t.abs()
        return torch.where(t < 1, 1 - 2.5 * t ** 2 + 1.5 * t ** 3,
                           torch.where(t < 2, 0.5 * (2 - t) ** 2 * (1 - t), 0.0))
    x0, y0 = jx.floor(), iy.floor()
    out = torch.zeros(2 * nr * nz, dtype=torch.float64, device="cuda")
    for a in range(-1, 3):
        for b in range(-1, 3):
            gy, gx = y0 + a, x0 + b
            val = wd * mp4(iy - gy) * mp4(jx - gx)
            ok = (gy >= 0) & (gy < 2 * nr) & (gx >= 0) & (gx < nz)
            out.index_add_(0, (gy * nz + gx)[ok].long(), val[ok])
    return out.view(2 * nr, nz)[nr:].clone()


def exact(case, seed):
    kind = case["kind"]
    if kind == "rigid":
        cases, w0 = _bodies(case, seed)
        got = [_x_rigid_step(c, w) for c, w in zip(cases, w0)]
        if len(cases) > 15:
            out = {"vorticity": torch.cat([g[0].reshape(-1) for g in got])}
        else:
            out = {n: [g[q] for g in got] for q, n in enumerate(("omega", "psi", "u_z", "u_r"))}
        if case["precision"] == "f64":
            out["t_dt_cd_steps"] = torch.tensor([g[4] for g in got], dtype=torch.float64)
        return out
    if kind == "soft":
        # the fluid half of the step; the fields behind the elastic stress have no short restatement
        c = _soft_case(case)
        Z, R = _coords(c.nr, c.nz, c.dx)
        w = _cuda(_rings(c.nr, c.nz, c.dx, seed, 0.02))
        _x_kill(w, Z, R, c.kill_width, c.dx)
        psi = _x_stokes(w, c.dx, False)
        uz, ur = _x_velocity(psi, R, c.dx)
        umax = float((uz.abs() + ur.abs()).max())
        dt = min(c.cfl * c.dx / math.sqrt(c.G / c.rho_f), c.cfl * c.dx / (umax + EPS),
                 0.9 * c.dx ** 2 / 4 / c.nu)
        chi = _x_heaviside(c.zeta * c.r_ball - torch.sqrt((Z - c.z_cm) ** 2 + R ** 2),
                           c.moll_zone)
        pz, pr = _x_penalise(w, uz, ur, chi, c.lam * dt, c.U0, c.dx)
        return dict(vorticity=None, psi=psi, u_z=pz, u_r=pr, eta1=None, eta2=None, ball_phi=None,
                    ball_char_func=None, state=torch.tensor([dt, dt, 1.0], dtype=torch.float64))
    if kind == "solve":
        return _x_stokes(_cuda(_rings(case["nr"], case["nz"], 1.0 / case["nr"], seed, 1.0, n=32)),
                         1.0 / case["nr"], case["bc"] == PERIODIC_Z)
    if kind == "dropin":
        c = _sphere(case, seed)
        w, psi, uz, ur, (_, dt, cd, _) = _x_rigid_step(c, _rings(c.nr, c.nz, c.dx, seed, 2.0))
        return dict(vorticity=w, psi=psi, u_z=uz, u_r=ur, dt=dt, Cd=cd)
    return _x_remesh(case, seed)
