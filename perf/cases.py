"""Performance cases of the library: what its users run, at the sizes they run.

Each case is a dict of plain values with a ``kind``:

* ``step``   -- one whole aerodynamic timestep of a moving-body simulation
  (``step.DeviceStepper``): uvort with the pressure equation's particle term,
  assembly, pressure equation, solve, FMM with the element sums.
* ``wing``   -- one timestep of the vortex-lattice wing with its panel wake and
  particle shedding (``step.WakeStepper``), in the developed state where as
  many particles leave the particle box as are shed.
* ``fmm``    -- a standalone wake FMM evaluation
  (``Octree.apply_multipole_device``) of the vortex ring with background.
* ``uvort``  -- the particles' and end vortices' direct sum at panel centres
  (``dust_points_uvort_device``; with ``pressure`` the fused call).
* ``linsys`` -- assembly and solve of a moving-body panel system (rotor over a
  fuselage) from host geometry (``Linsys.assemble_linsys``/``solve_linsys``).
* ``dense``  -- the standalone dense solve (``linsys.dense_solve_device``).
* ``net``    -- loss and gradient (forward and backward pass) of the learned
  preconditioner on a stored system (``Precond.loss_grad``).

Results of the FP32C precision mode carry FP32 accuracy, so a program that
selects it keeps its fields in single precision: those cases return FP32
copies.  FP64 modes return the FP64 arrays.
"""
import ctypes as C
import math

import numpy as np
import torch

from dust_b200 import abi, linsys, octree, precond, synth
from dust_b200._lib import check, lib
from dust_b200.params import FmmParams
from dust_b200.step import DeviceStepper, WakeStepper

F64 = torch.float64
MODES = {"lu64": abi.DUST_SOLVE_LU64, "mixed": abi.DUST_SOLVE_MIXED,
         "gmres": abi.DUST_SOLVE_GMRES_NN}


def listed():
    return [
        # The small named configuration: 400-panel wing, its wake shedding 40
        # particles a step; about 12,800 live particles when developed.  Small
        # kernels in a long chain: launch and host latency count.
        dict(name="wing_step_400", kind="wing", n_span=40, n_chord=10, wake_steps=320),
        # The smallest FMM a program evaluates (the size of the test and smoke
        # calls; the first steps of any simulation).
        dict(name="fmm_3k_p4", kind="fmm", n=3000, degree=4, f32=False),
        # A wake of the usual workstation size, plain FP64, default order.
        dict(name="fmm_110k_p4", kind="fmm", n=110000, degree=4, f32=False),
        # The higher order of the standalone-FMM configuration at an odd size.
        dict(name="fmm_40k_p6", kind="fmm", n=40009, degree=6, f32=False),
        # The standalone-FMM configuration at its full size, FP32C.
        dict(name="fmm_1100k_p4_f32c", kind="fmm", n=1100000, degree=4, f32=True),
        # Wake velocity at the panels of a mid-size model, odd sizes, FP64.
        dict(name="uvort_7k_x_50k", kind="uvort", n_pts=7001, n=50021, f32=False, pressure=False),
        # A small full step in the plain FP64 form: an early step of the
        # rotors-and-wing model on a coarse wing.
        dict(name="step_plain_60k", kind="step", n=60000, wing_span=30, wing_around=40, levels=5,
             f32=False),
        # The headline workload: the full step with 2M particles and 13,920
        # panels in the mixed-precision form.
        dict(name="step_mixed_2m", kind="step", n=2000000, wing_span=98, wing_around=120, levels=7,
             f32=True),
        # One step's system of the rotor-over-fuselage configuration (6,954
        # unknowns, 960 of them moving): assembly and the plain LU solve.
        dict(name="linsys_rotor_7k", kind="linsys", n_fus=6000, n_span=30, mode="lu64"),
        # The ellipsoid configuration: 16,384 unknowns, 64 right-hand sides,
        # mixed-precision LU refined to FP64.
        dict(name="dense_16k_mixed", kind="dense", n=16384, nrhs=64, mode="mixed"),
        # A small plain LU solve of odd size with one right-hand side.
        dict(name="dense_3k_lu64", kind="dense", n=3001, nrhs=1, mode="lu64"),
        # Training direction of the learned preconditioner.
        dict(name="net_gradient_7k", kind="net", n_fus=6000, n_span=30),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["wing", "fmm", "fmm", "fmm", "uvort", "uvort", "step", "step", "linsys",
                       "dense", "dense", "net"])
    if kind == "wing":
        return dict(kind=kind, n_span=rng.randint(20, 60), n_chord=rng.randint(4, 10),
                    wake_steps=rng.randint(40, 320))
    if kind == "fmm":
        degree, hi = rng.choice([(4, 1000000), (4, 1000000), (2, 1000000), (6, 200000), (8, 30000)])
        return dict(kind=kind, n=_log_int(rng, 1000, hi), degree=degree, f32=rng.random() < 0.5)
    if kind == "uvort":
        return dict(kind=kind, n_pts=_log_int(rng, 200, 14000), n=_log_int(rng, 3000, 400000),
                    f32=rng.random() < 0.5, pressure=rng.random() < 0.5)
    if kind == "step":
        n = _log_int(rng, 30000, 600000)
        return dict(kind=kind, n=n, wing_span=rng.randint(20, 70),
                    wing_around=2 * rng.randint(15, 45),
                    levels=int(round(7 + math.log2(n / 2e6) / 2.3)), f32=rng.random() < 0.5)
    if kind == "linsys":
        return dict(kind=kind, n_fus=_log_int(rng, 800, 6000), n_span=rng.randint(10, 30),
                    mode=rng.choice(["lu64", "mixed", "gmres"]))
    if kind == "dense":
        return dict(kind=kind, n=_log_int(rng, 500, 12000), nrhs=_log_int(rng, 1, 64),
                    mode=rng.choice(["lu64", "mixed"]))
    return dict(kind=kind, n_fus=_log_int(rng, 800, 6000), n_span=rng.randint(10, 30))


# ------------------------------------------------------------------ helpers
def _ptr(t, ctype=C.c_double):
    return C.cast(C.c_void_p(t.data_ptr()), C.POINTER(ctype))


def _gpu(a, dtype=F64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")


def _out(f32, *tensors):
    return [t.float() for t in tensors] if f32 else list(tensors)


def _ring(case, seed):
    """The ring workload (1/11 of the particles in the background, core 0.02)."""
    n_bg = case["n"] // 11
    return synth.ring_particles(case["n"] - n_bg, n_bg, seed=seed)


def _ring_levels(n):
    """Levels that keep the finest cells of the ring at <= 64 particles: the
    peak density of its Gaussian cross-section (0.1) with a margin for the
    fluctuation of the fullest cell."""
    rho = 1.4 * n / (2 * math.pi) ** 2 / 0.01
    return max(3, 1 + math.ceil(math.log2(4.0 / (64.0 / rho) ** (1 / 3))))


def _ring_params(case):
    return FmmParams(box_length=4.0, origin=(-2.0, -2.0, -2.0),
                     n_octree_levels=_ring_levels(case["n"]), min_octree_part=8,
                     multipole_degree=case["degree"], rankine_rad=0.02,
                     precision=abi.DUST_PREC_FP32C if case["f32"] else abi.DUST_PREC_FP64)


# ------------------------------------------------------------------ prepare
def _prepare_fmm(case, seed):
    cen, dir_, mag = _ring(case, seed)
    n = mag.shape[0]
    empty = lambda: torch.empty((n, 3), dtype=F64, device="cuda")
    return dict(oc=octree.initialize_octree(_ring_params(case)), cen=_gpu(cen), dir=_gpu(dir_),
                mag=_gpu(mag), rv=torch.full((n,), 0.02, dtype=F64, device="cuda"), vel=empty(),
                str=empty(), rot=empty(), stream=torch.cuda.Stream())


def _run_fmm(case, s):
    with torch.cuda.stream(s["stream"]):
        s["oc"].apply_multipole_device(s["cen"], s["dir"], s["mag"], s["rv"], s["vel"], s["str"],
                                       s["rot"], stream=s["stream"].cuda_stream, sync=False)
        return _out(case["f32"], s["vel"], s["str"], s["rot"])


def _uvort_arrays(case, seed):
    """Panel centres of an ellipsoid (semi-axes 4, 1, 0.5) and a wake behind it."""
    rng = np.random.default_rng(seed)
    u = rng.standard_normal((case["n_pts"], 3))
    pts = u / np.linalg.norm(u, axis=1)[:, None] * np.array([4.0, 1.0, 0.5])
    n = case["n"]
    cen = np.stack([rng.uniform(-3.0, 9.0, n), rng.uniform(-3.0, 3.0, n),
                    0.2 * rng.standard_normal(n)], axis=1)
    dir_ = rng.standard_normal((n, 3))
    dir_ /= np.linalg.norm(dir_, axis=1)[:, None]
    mag = np.abs(1e-3 + 2e-4 * rng.standard_normal(n))
    a = np.stack([np.full(64, 4.2), np.linspace(-1.0, 1.0, 65)[:-1], np.zeros(64)], axis=1)
    b = a + np.array([0.0, 2.0 / 64, 0.0])
    return dict(pts=pts, cen=cen, dir=dir_, mag=mag, rv=np.full(n, 0.04),
                vel=rng.standard_normal((n, 3)), lver=np.stack([a, b], axis=1),
                lmag=0.05 * rng.standard_normal(64))


def _uvort_params(case):
    return FmmParams(box_length=8.0, n_box=(2, 1, 1), origin=(-5.0, -4.0, -4.0), rankine_rad=0.1,
                     precision=abi.DUST_PREC_FP32C if case["f32"] else abi.DUST_PREC_FP64)


def _prepare_uvort(case, seed):
    s = {k: _gpu(v) for k, v in _uvort_arrays(case, seed).items()}
    s["uv"] = torch.empty((case["n_pts"], 3), dtype=F64, device="cuda")
    s["pterm"] = torch.empty(case["n_pts"], dtype=F64, device="cuda")
    s["prm"] = _uvort_params(case).struct()
    s["stream"] = torch.cuda.Stream()
    return s


def _run_uvort(case, s):
    lines = abi.Lines(int(s["lmag"].shape[0]), _ptr(s["lver"]), _ptr(s["lmag"]))
    st = C.c_void_p(s["stream"].cuda_stream)
    with torch.cuda.stream(s["stream"]):
        if case["pressure"]:
            check(lib().dust_points_uvort_pressure_device(
                C.byref(s["prm"]), case["n_pts"], _ptr(s["pts"]), case["n"], _ptr(s["cen"]),
                _ptr(s["dir"]), _ptr(s["mag"]), _ptr(s["rv"]), _ptr(s["vel"]), C.byref(lines),
                _ptr(s["uv"]), _ptr(s["pterm"]), st), "dust_points_uvort_pressure_device")
            return _out(case["f32"], s["uv"], s["pterm"])
        check(lib().dust_points_uvort_device(
            C.byref(s["prm"]), case["n_pts"], _ptr(s["pts"]), case["n"], _ptr(s["cen"]),
            _ptr(s["dir"]), _ptr(s["mag"]), _ptr(s["rv"]), C.byref(lines), _ptr(s["uv"]), st),
            "dust_points_uvort_device")
        return _out(case["f32"], s["uv"])


def _prepare_step(case, seed):
    """A running simulation: its handles, and the previous step done (its
    particle velocities enter the pressure equation)."""
    c = synth.FullStepCase(n_particles=case["n"], seed=seed, wing_span=case["wing_span"],
                           wing_around=case["wing_around"])
    prm = FmmParams(box_length=c.box_length, n_box=c.n_box, origin=c.origin,
                    n_octree_levels=case["levels"], min_octree_part=8, multipole_degree=4,
                    rankine_rad=0.1, cutoff_rad=0.001, u_inf=tuple(c.u_inf),
                    precision=abi.DUST_PREC_FP32C if case["f32"] else abi.DUST_PREC_FP64)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        st = DeviceStepper(c, prm, abi.DUST_SOLVE_MIXED if case["f32"] else abi.DUST_SOLVE_LU64)
        st.step()
    stream.synchronize()
    return dict(st=st, stream=stream)


def _run_step(case, s):
    st = s["st"]
    with torch.cuda.stream(s["stream"]):
        st.step()
        return _out(case["f32"], st.res, st.res_pres, st.euv, st.vel, st.str, st.rot)


def _prepare_wing(case, seed):
    """A developed wake: one row of particles per stripe and past step, trailing
    vorticity of an elliptic loading, slightly scattered."""
    ns, steps, dt = case["n_span"], case["wake_steps"], 0.05
    c = synth.WingWakeCase(n_span=ns, n_chord=case["n_chord"], dt=dt, n_wake_panels=1,
                           n_wake_particles=int(ns * (1.25 * steps + 20)),
                           box_max=(max(2.0, steps * dt), 8.0, 8.0))
    st = WakeStepper(c, c.fmm_params(levels=6))
    rng = np.random.default_rng(seed)
    rows = int((c.box_max[0] - 1.1) / dt)
    edge = np.linspace(-5.0, 5.0, ns + 1)
    load = 0.2 * np.sqrt(np.maximum(0.0, 1.0 - (edge / 5.0) ** 2))
    y = 0.5 * (edge[1:] + edge[:-1])
    n = rows * ns
    cen = np.empty((rows, ns, 3))
    cen[..., 0] = 1.05 + dt * np.arange(rows)[:, None]
    cen[..., 1] = y[None, :]
    cen[..., 2] = -0.09 - 0.02 * dt * np.arange(rows)[:, None]
    cen = cen.reshape(n, 3) + 0.01 * rng.standard_normal((n, 3))
    trail = np.tile(-np.diff(load) * dt, rows) * (1.0 + 0.1 * rng.standard_normal(n))
    dir_ = np.zeros((n, 3))
    dir_[:, 0] = np.where(trail < 0, -1.0, 1.0)
    st.S["cen"][:n], st.S["dir"][:n] = _gpu(cen), _gpu(dir_)
    st.S["mag"][:n], st.S["rv"][:n] = _gpu(np.abs(trail)), 0.1
    st.free[:n] = 0
    return dict(st=st)


def _run_wing(case, s):
    st = s["st"]
    st.step()
    return [st.res, st.S["cen"], st.S["dir"], st.S["mag"], st.S["vel"], st.S["str"], st.free]


def _rotor_case(case, seed):
    rc = synth.RotorFuselageCase(n_fus=case["n_fus"], n_span=case["n_span"])
    return rc, rc.system(seed)


def _add_sample(pc, ls, els, seed):
    ls.assemble_linsys(els)
    x, _ = ls.solve_linsys(abi.DUST_SOLVE_LU64)
    ls.assemble_linsys(els)
    pc.add_sample(ls, x, seed=seed)


def _prepare_linsys(case, seed):
    rc, els = _rotor_case(case, seed)
    ls = linsys.initialize_linsys(rc.fmm_params(), rc.rank, rc.nstatic, els)
    s = dict(ls=ls, els=els)
    if case["mode"] == "gmres":
        s["pc"] = precond.Precond(precond._centres(els), k=8, seed=0)
        for q in range(4):
            _add_sample(s["pc"], ls, rc.system(1000 + q), q)
        s["pc"].train(100, 2e-3)
        s["pc"].attach(ls)
    return s


def _run_linsys(case, s):
    s["ls"].assemble_linsys(s["els"])
    return s["ls"].solve_linsys(MODES[case["mode"]])[0]


def _dense_system(case, seed):
    """Doublet influence matrix of a closed ellipsoid of nearly equal panels in
    a random rotation (solid angle of each panel at every other centre, the
    self term -2 pi less the rest's deviation from the closed-body sum), and
    right-hand sides of random freestream directions."""
    n = case["n"]
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    k = torch.arange(n, dtype=F64, device="cuda") + 0.5
    ph, z = k * (math.pi * (3.0 - math.sqrt(5.0))), 1.0 - 2.0 * k / n
    r = torch.sqrt(1.0 - z * z)
    u = torch.stack([r * torch.cos(ph), r * torch.sin(ph), z], dim=1)
    ax = torch.tensor([4.0, 1.0, 0.5], dtype=F64, device="cuda")
    q, _ = torch.linalg.qr(torch.randn((3, 3), generator=g, dtype=F64, device="cuda"))
    x, w = (u * ax) @ q.T, (u / ax * ax.prod() * 4 * math.pi / n) @ q.T  # centres, area vectors
    at = torch.empty((n, n), dtype=F64, device="cuda")  # at[j, i] = A(i, j)
    grad = torch.empty((n, 3), dtype=F64, device="cuda")
    for j in range(0, n, 1024):
        d = x[None, :, :] - x[j:j + 1024, None, :]
        r2 = (d * d).sum(dim=2) + w[j:j + 1024].norm(dim=1)[:, None]
        at[j:j + 1024] = (d * w[j:j + 1024, None, :]).sum(dim=2) * r2 ** -1.5
        grad[j:j + 1024] = (w[None, :, :] / torch.sqrt(r2)[:, :, None]).sum(dim=1)
    at.diagonal().copy_(-2 * math.pi * (1.0 + 0.02 * torch.rand(n, generator=g, dtype=F64,
                                                                device="cuda")))
    dirs = torch.randn((case["nrhs"], 3), generator=g, dtype=F64, device="cuda")
    bt = (dirs / dirs.norm(dim=1)[:, None]) @ grad.T  # bt[c, i] = B(i, c)
    return at, bt.contiguous()


def _prepare_dense(case, seed):
    at, bt = _dense_system(case, seed)
    return dict(at=at, bt=bt, xt=torch.empty_like(bt), stream=torch.cuda.Stream())


def _run_dense(case, s):
    linsys.dense_solve_device(s["at"], s["bt"], s["xt"], MODES[case["mode"]], 1e-12,
                              stream=s["stream"].cuda_stream)
    return s["xt"]


def _prepare_net(case, seed):
    rc, els = _rotor_case(case, seed)
    ls = linsys.initialize_linsys(rc.fmm_params(), rc.rank, rc.nstatic, els)
    pc = precond.Precond(precond._centres(els), k=8, seed=0)
    rng = np.random.default_rng(7)
    pc.set_params(pc.get_params() + 0.02 * rng.standard_normal(pc.num_params()).astype(np.float32))
    _add_sample(pc, ls, els, seed)
    return dict(pc=pc)


def _run_net(case, s):
    loss, grad = s["pc"].loss_grad(0)
    return [loss, grad]


def prepare(case, seed):
    s = globals()["_prepare_" + case["kind"]](case, seed)
    torch.cuda.synchronize()
    s["case"] = case
    return s


def run(state):
    case = state["case"]
    return globals()["_run_" + case["kind"]](case, state)


# --------------------------------------------------------------------- work
def _fmm_flops(n, degree, particles_per_leaf=16):
    """Near field over 27 leaves (95 flop a pair) and, per leaf, about 60
    occupied interaction cells translated (three scalar sums)."""
    nm = (degree + 1) * (degree + 2) * (degree + 3) // 6
    nj = (degree + 3) * (degree + 4) * (degree + 5) // 6
    return n * 27 * particles_per_leaf * 95.0 + n / particles_per_leaf * 60 * 6.0 * nm * nj


def work(case):
    k = case["kind"]
    if k == "fmm":
        return dict(bytes=case["n"] * 8 * (8 + 9), flops=_fmm_flops(case["n"], case["degree"]))
    if k == "uvort":
        pairs = float(case["n"]) * case["n_pts"]
        return dict(bytes=8 * (8 * case["n"] + 6 * case["n_pts"]),
                    flops=pairs * (34 if case["pressure"] else 27))
    if k == "step":
        stat = case["wing_around"] * (case["wing_span"] + 2)
        mov = 1920
        rank = stat + mov
        flops = (case["n"] * float(rank) * (34 + 31) + _fmm_flops(case["n"], 4)
                 + 2.0 * stat * stat * mov + 2.0 * mov * mov * stat + 2.0 / 3.0 * mov ** 3)
        return dict(bytes=case["n"] * 8 * 17 + 8.0 * rank * rank, flops=flops)
    if k == "wing":
        n, rank = case["n_span"] * case["wake_steps"], case["n_span"] * case["n_chord"]
        return dict(bytes=n * 8 * 17 + 8.0 * rank * rank,
                    flops=n * float(rank) * 27 * 2 + _fmm_flops(n, 4))
    if k in ("linsys", "net"):
        mov = 4 * 8 * case["n_span"]
        stat = case["n_fus"]
        if k == "net":
            return dict(bytes=(stat + mov) * 9 * 64 * 4.0, flops=(stat + mov) * 3 * 6 * 25413.0)
        return dict(bytes=8.0 * (stat + mov) ** 2,
                    flops=2.0 * stat * mov * (stat + mov) + 2.0 / 3.0 * mov ** 3)
    n, m = float(case["n"]), case["nrhs"]
    return dict(bytes=8.0 * (n * n + 2 * n * m), flops=2.0 / 3.0 * n ** 3 + 2.0 * n * n * m)


# -------------------------------------------------------------------- exact
def _exact_fmm(case, seed):
    """The sum over all particle pairs that the FMM approximates."""
    cen, dir_, mag = _ring(case, seed)
    x, a = _gpu(cen), _gpu(dir_ * mag[:, None])
    n, s2, nu = x.shape[0], 0.02 ** 2, 1.8e-5 / 1.225
    vel, st, rot = (torch.empty((n, 3), dtype=F64, device="cuda") for _ in range(3))
    for i in range(0, n, 256):
        m = min(256, n - i)
        d = x[i:i + m, None, :] - x[None, :, :]
        r2 = (d * d).sum(dim=2)
        other = torch.ones((m, n), dtype=F64, device="cuda")
        other[torch.arange(m), torch.arange(i, i + m)] = 0.0
        c = -other * (r2 + s2) ** -1.5 / (4 * math.pi)
        e = -3.0 * c / (r2 + s2)
        aq, ap = a[None, :, :].expand(m, n, 3), a[i:i + m, None, :].expand(m, n, 3)
        vel[i:i + m] = (c[:, :, None] * torch.linalg.cross(d, aq)).sum(dim=1)
        v = torch.linalg.cross(ap, aq)
        w = nu * 17.5 / s2 * (1.0 + r2 / s2) ** -4.5
        st[i:i + m] = (-c[:, :, None] * v - (e * (d * v).sum(dim=2))[:, :, None] * d
                       + w[:, :, None] * (aq - ap)).sum(dim=1)
        rot[i:i + m] = ((-2.0 * c - e * r2)[:, :, None] * aq
                        + (e * (d * aq).sum(dim=2))[:, :, None] * d).sum(dim=1)
    return [vel, st, rot]


def _exact_uvort(case, seed):
    s = {k: _gpu(v) for k, v in _uvort_arrays(case, seed).items()}
    a = s["dir"] * s["mag"][:, None]
    av = torch.linalg.cross(s["dir"], s["vel"]) * s["mag"][:, None]
    uv = torch.empty((case["n_pts"], 3), dtype=F64, device="cuda")
    pt = torch.empty(case["n_pts"], dtype=F64, device="cuda")
    chunk = max(1, 20_000_000 // case["n"])
    for i in range(0, case["n_pts"], chunk):
        d = s["pts"][i:i + chunk, None, :] - s["cen"][None, :, :]
        w = ((d * d).sum(dim=2) + s["rv"][None, :] ** 2) ** -1.5
        uv[i:i + chunk] = (-w[:, :, None] / (4 * math.pi)
                           * torch.linalg.cross(d, a[None].expand_as(d))).sum(dim=1)
        pt[i:i + chunk] = -(w * (d * av[None]).sum(dim=2)).sum(dim=1)
    uv += _exact_lines(s)
    return [uv, pt] if case["pressure"] else [uv]


def _exact_lines(s):
    """Straight segments (the points lie outside every segment's core)."""
    p, a, b = s["pts"][:, None, :], s["lver"][None, :, 0, :], s["lver"][None, :, 1, :]
    r1, r2 = p - a, p - b
    t = (b - a) / (b - a).norm(dim=2, keepdim=True)
    al = (r1 * t).sum(dim=2)
    h = r1 - al[:, :, None] * t
    c = (al / r1.norm(dim=2) - (r2 * t).sum(dim=2) / r2.norm(dim=2)) / (h * h).sum(dim=2)
    w = s["lmag"][None, :] * c / (4 * math.pi)
    return (w[:, :, None] * torch.linalg.cross(t.expand_as(h), h)).sum(dim=1)


def exact(case, seed):
    if case["kind"] == "fmm" and case["n"] <= 120000:
        return _exact_fmm(case, seed)
    if case["kind"] == "uvort" and case["n_pts"] * case["n"] <= 1_500_000_000:
        return _exact_uvort(case, seed)
    if case["kind"] == "dense":
        at, bt = _dense_system(case, seed)
        return torch.linalg.solve(at.T, bt.T).T.contiguous()
    return None
