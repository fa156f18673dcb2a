"""The workloads this framework's speed is measured on.

Each case is one thing that a program built on the framework has it do, called
through the public entry points, with the sizes of the repository's own
configurations (64x32x32, 88x44x44, 128x64x48, 256x128x96, 512x256x160):

* ``steps``: a stretch of a welding job.  The twin is set to a stored state
  (a plate with a bead behind the torch and a molten pool under it), then
  ``WAAMTwin.step`` follows the torch path.  Options cover what a job
  switches on: heat source, wetting / surface tension / gravity, heat losses,
  16-bit populations, temperature tables with the remelt / freeze tail, wire
  droplets, the Lorentz force, the operator-by-operator driver.
* ``adjoint``: loss and gradient of a calibration problem (probe temperatures
  and pool width) through ``CoupledStepLoss``.
* ``flow``: collision and streaming operators on a force-driven channel, as the
  flow validation runs them.
* ``heat``: the thermal operators on a heated block, as the diffusion and
  solidification validations run them.

``exact`` restates the same physics in float64 torch operations.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from waam_solver_b200 import WAAMTwin
from waam_solver_b200 import kernels
from waam_solver_b200.adjoint import AdjointProblem, CoupledStepLoss
from waam_solver_b200.materials import MaterialTables, build_sahoo_dgamma_table, from_constants
from waam_solver_b200.physics import lbm, phase_change, thermal
from waam_solver_b200.physics.arc import goldak_from_job_mm

FLUID, SOLID, GAS, IFACE = 0, 1, 2, 4
EX = (0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0)
EY = (0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1)
EZ = (0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1)
OPP = (0, 2, 1, 4, 3, 6, 5, 8, 7, 10, 9, 12, 11, 14, 13, 16, 15, 18, 17)
W = (1.0 / 3.0,) + (1.0 / 18.0,) * 6 + (1.0 / 36.0,) * 12

STEEL = dict(k=30.0, rho=7800.0, cp=680.0, T_solidus=1723.0, T_liquidus=1783.0, L_fusion=2.7e5,
             gamma_0=1.8, dgamma_dT=-4.3e-4, mu=0.0065, beta_T=1.2e-4)
GOLDAK_MM = dict(a_front_mm=3.0, a_rear_mm=9.0, b_mm=3.0, c_mm=3.0, ff=0.6, fr=1.4)
TRAVEL = 0.008          # m/s
T_AMB = 300.0


# ---- the cases ----------------------------------------------------------------

def _steps(**kw):
    c = dict(kind="steps", nx=64, ny=32, nz=32, dx=2.5e-4, source="goldak", power=3500.0, steps=25,
             storage="float32", wet=False, srt=False, heat_loss=False, tables=False, drops=False,
             lorentz=False, driver="fused")
    c.update(kw)
    return c


def listed():
    return [
        # the smallest job: parameter studies on coarse grids, where launches decide
        _steps(name="small", nx=64, ny=32, nz=32, dx=2.5e-4, source="gaussian2d", power=3000.0,
               steps=25),
        # a coarse validation-matrix bead with an odd grid, SRT, heat losses and all forces
        _steps(name="ragged", nx=87, ny=45, nz=43, dx=2e-4, wet=True, srt=True, heat_loss=True,
               steps=25),
        # temperature-dependent steel with the remelt / trailing-freeze tail (multi-layer jobs)
        _steps(name="tables", nx=131, ny=67, nz=50, dx=2e-4, wet=True, heat_loss=True, tables=True,
               steps=20),
        # the ordinary production bead: wire droplets, wetting, surface tension, gravity
        _steps(name="standard", nx=256, ny=128, nz=96, dx=2e-4, power=4000.0, wet=True, drops=True,
               steps=250),
        # the same bead with half-size populations, without wire
        _steps(name="standard_f16", nx=256, ny=128, nz=96, dx=2e-4, power=4000.0, wet=True,
               storage="float16", steps=50),
        # the largest job: fine two-layer grid with the welding current's force
        _steps(name="large_lorentz", nx=512, ny=256, nz=160, dx=1.5e-4, power=4000.0, wet=True,
               heat_loss=True, lorentz=True, storage="float16", steps=16),
        # a host program that interleaves operators of its own: the reference's call sequence
        _steps(name="operators", nx=128, ny=64, nz=48, dx=2.5e-4, wet=True, heat_loss=True,
               driver="operators", steps=10),
        # calibration: loss and gradient over a stretch of the path
        dict(name="adjoint", kind="adjoint", nx=128, ny=64, nz=48, dx=2.5e-4, steps=64),
        # flow validation: forced channel, SRT and central-moment collision
        dict(name="channel", kind="flow", nx=192, ny=96, nz=66, srt=True, steps=20),
        dict(name="channel_mrt", kind="flow", nx=101, ny=61, nz=43, srt=False, steps=20),
        # heat validation: diffusion, advection and solidification on a block
        dict(name="heat_block", kind="heat", nx=96, ny=96, nz=96, steps=20),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps"] * 6 + ["adjoint", "flow", "flow", "heat"])
    nx, ny, nz = _size(rng, 56, 320), _size(rng, 28, 160), _size(rng, 30, 110)
    if kind == "adjoint":
        return dict(kind=kind, nx=min(nx, 160), ny=min(ny, 80), nz=min(nz, 60), dx=2.5e-4,
                    steps=rng.randrange(30, 80))
    if kind == "flow":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, srt=rng.random() < 0.5,
                    steps=rng.randrange(8, 24))
    if kind == "heat":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=rng.randrange(8, 24))
    tables = rng.random() < 0.2
    ops = not tables and rng.random() < 0.2
    wet = rng.random() < 0.75
    lorentz = not tables and not ops and rng.random() < 0.2
    return _steps(nx=nx, ny=ny, nz=nz, dx=rng.choice([1.5e-4, 2e-4, 2.5e-4]),
                  source=rng.choice(["goldak", "goldak", "gaussian2d"]),
                  power=float(rng.randrange(2800, 4100, 100)), steps=rng.randrange(10, 40),
                  storage="float32" if ops or tables else rng.choice(
                      ["float32", "float32", "float16", "bfloat16"]),
                  wet=wet, srt=rng.random() < 0.25, heat_loss=rng.random() < 0.5, tables=tables,
                  lorentz=lorentz, driver="operators" if ops else "fused")


# ---- the job a program has in hand ---------------------------------------------

def _table_knots():
    m, Tl = STEEL, STEEL["T_liquidus"]
    return dict(cp=[(300.0, 0.95 * m["cp"]), (1000.0, m["cp"]), (Tl, 1.06 * m["cp"])],
                k=[(300.0, 0.93 * m["k"]), (1000.0, m["k"]), (Tl, 1.13 * m["k"])],
                mu=[(300.0, 1.15 * m["mu"]), (Tl, m["mu"]), (Tl + 200.0, 0.85 * m["mu"])],
                dgamma_dT=[(float(np.float32(t)), float(np.float32(v))) for t, v in
                           build_sahoo_dgamma_table(28.0, Tl, max(Tl + 800.0, 2600.0), n=8)])


def _twin(case):
    mat = from_constants("steel", STEEL, contact_angle_deg=30.0)
    if case["tables"]:
        mat.tables = MaterialTables(**_table_knots())
    tw = WAAMTwin(material=mat, nx=case["nx"], ny=case["ny"], nz=case["nz"], dx=case["dx"],
                  arc_power_W=case["power"], arc_efficiency=0.78, arc_sigma_mm=2.0,
                  heat_source=case["source"], use_srt=case["srt"], enable_vof=True,
                  enable_wetting=case["wet"], contact_angle_deg=30.0,
                  enable_csf_tension=case["wet"], enable_hydrostatic_gravity=case["wet"],
                  enable_heat_loss=case["heat_loss"], enable_lorentz=case["lorentz"],
                  welding_current_A=140.0, droplet_freq_hz=200.0 if case["drops"] else 0.0,
                  enable_substrate_growth=case["tables"], enable_bead_freeze=case["tables"],
                  wire_diameter_mm=1.2, travel_speed_m_s=TRAVEL, max_tracers=1024,
                  population_dtype=case["storage"], step_mode=case["driver"])
    if case["drops"]:
        tw.wire_feed_m_s = 0.1
        tw.droplet_transfer_mode = "pulsed"
        tw.pulse_frequency_hz = 200.0
        tw.droplet_size_jitter = 0.0
    if case["source"] == "goldak":
        tw.arc_source = goldak_from_job_mm(tw, GOLDAK_MM)
    return tw


def _start_of_path(case, seed):
    """Torch position [cells] at the start of the stretch."""
    r = np.random.default_rng(seed)
    return (case["nx"] * r.uniform(0.38, 0.5), case["ny"] * r.uniform(0.46, 0.54))


def _noise(shape, gen, scale):
    return (torch.rand(shape, generator=gen, device=gen.device) * 2.0 - 1.0) * scale


def _pool_state(case, seed, nz_solid, device):
    """A plate with a bead behind the torch and a molten pool under it, as
    float32 fields: tanh interface, hot spot with a tail, swirling melt and
    populations near equilibrium."""
    nx, ny, nz, dx = case["nx"], case["ny"], case["nz"], case["dx"]
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    ti, tj = _start_of_path(case, seed)
    f32 = dict(dtype=torch.float32, device=device)
    i = torch.arange(nx, **f32).view(nx, 1, 1)
    j = torch.arange(ny, **f32).view(1, ny, 1)
    k = torch.arange(nz, **f32).view(1, 1, nz)
    mm = 1e-3 / dx                                   # cells per millimetre
    height = min(1.5 * mm, 0.2 * (nz - nz_solid))
    width = min(2.5 * mm, 0.2 * ny)
    track = torch.sigmoid((ti - i) / 2.0) * torch.exp(-((j - tj) / width) ** 2)
    top = (nz_solid - 0.5) + height * track + 0.4 * torch.sin(0.7 * i + 0.1 * seed)
    phi = 0.5 * (1.0 - torch.tanh((k - top) / 0.8))
    phi = torch.where(k < nz_solid, torch.ones_like(phi), phi)
    phi = torch.where(phi < 0.01, torch.zeros_like(phi), phi)
    # hot spot at the torch, a tail behind it
    s = max(3.0, min(2.2 * mm, 0.25 * ny))
    back = torch.where(i < ti, torch.full_like(i, 2.0), torch.ones_like(i))
    r2 = ((i - ti) / back) ** 2 + (j - tj) ** 2 + (k - nz_solid - 0.5 * height) ** 2
    T = T_AMB + 2100.0 * torch.exp(-r2 / (2.0 * s * s)) + 60.0 + _noise((nx, ny, nz), gen, 20.0)
    m = STEEL
    cp_rho, L_rho = m["rho"] * m["cp"], m["rho"] * m["L_fusion"]
    if case.get("tables"):
        cp_rho = m["rho"] * _interp(T, _table_knots()["cp"])
    Ts, Tl = m["T_solidus"], m["T_liquidus"]
    fl = ((T - Ts) / (Tl - Ts)).clamp(0.0, 1.0)
    gas = phi < 0.05
    T = torch.where(gas, torch.full_like(T, T_AMB), T)
    fl = torch.where(gas, torch.zeros_like(fl), fl)
    cp_gas = m["rho"] * m["cp"]
    H = torch.where(gas, torch.full_like(T, T_AMB * cp_gas),
                    cp_rho * torch.minimum(T, torch.full_like(T, Ts)) + fl * L_rho +
                    cp_rho * (T - Tl).clamp(min=0.0))
    fl = torch.where((k < nz_solid), torch.zeros_like(fl), fl)
    flags = torch.full((nx, ny, nz), IFACE, dtype=torch.int32, device=device)
    flags[phi < 0.05] = GAS
    flags[(phi > 0.55) & (fl > 0.1)] = FLUID
    flags[(phi > 0.85) & (fl < 0.05)] = SOLID
    flags[:, :, :nz_solid] = SOLID
    liquid = (fl > 0.0) & (flags != GAS) & (flags != SOLID)
    live = liquid.to(torch.float32)
    u = [(0.01 * torch.sin(a * i + b * j + c * k) + _noise((nx, ny, nz), gen, 1e-3)) * live
         for a, b, c in ((0.21, 0.35, 0.4), (0.3, 0.25, 0.5), (0.27, 0.4, 0.3))]
    rho = 1.0 + _noise((nx, ny, nz), gen, 1e-3)
    f = torch.empty((19, nx, ny, nz), **f32)
    u2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    for q in range(19):
        eu = EX[q] * u[0] + EY[q] * u[1] + EZ[q] * u[2]
        f[q] = W[q] * rho * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * u2)
    if case.get("storage", "float32") != "float32":     # values the storage can hold
        kind = getattr(torch, case["storage"])
        w = torch.tensor(W, **f32).view(19, 1, 1, 1)
        f = (f - w).to(kind).float() + w
    z = torch.zeros((nx, ny, nz), **f32)
    st = dict(f_a=f, f_b=f, rho=rho, ux=u[0], uy=u[1], uz=u[2], T=T, H=H, f_l=fl, phi=phi,
              flags=flags, T_max=T, T_prev=T, dT_dt=z, time_above_800_s=z, time_above_1100_s=z,
              time_above_solidus_s=z, Fx=z, Fy=z, Fz=z, read_is_a=True)
    if case.get("tables"):
        st.update(_properties(T, flags, case, dtype=torch.float32))
    return st


STATE_OUT = ("T", "H", "f_l", "phi", "flags", "rho", "ux", "uy", "uz", "T_max", "dT_dt",
             "time_above_800_s", "time_above_solidus_s", "Fx", "Fy", "Fz", "f_src", "f_dst")


def _positions(case, seed, dt):
    ti, tj = _start_of_path(case, seed)
    dx = case["dx"]
    return [(ti * dx + s * dt * TRAVEL, tj * dx) for s in range(case["steps"])]


def prepare(case, seed):
    """The twin of a running job (its first steps behind it), a stored state to
    start from and the torch path; or the grid and fields of a validation."""
    device = torch.device("cuda", torch.cuda.current_device())
    if case["kind"] == "flow":
        return _prepare_flow(case, seed, device)
    if case["kind"] == "heat":
        return _prepare_heat(case, seed, device)
    if case["kind"] == "adjoint":
        return _prepare_adjoint(case, seed, device)
    tw = _twin(case)
    tw.reset()
    g = tw.grid
    state = _pool_state(case, seed, tw.nz_solid, device)
    path = _positions(case, seed, g.dt)
    # the job is under way: with droplets, half a droplet period into it
    warm = 125 if case["drops"] else 3
    g.load_state(state)
    for _ in range(warm):
        tw.step(path[0][0], path[0][1], True)
    if case["lorentz"]:
        # the next solves start from the last potential, as in a running job
        state["phi_elec"] = g.phi_elec.clone()
        state["phi_elec_tmp"] = torch.zeros_like(state["phi_elec"])
    return dict(case=case, twin=tw, state=state, path=path)


def run(s):
    case = s["case"]
    if case["kind"] == "flow":
        return _run_flow(s)
    if case["kind"] == "heat":
        return _run_heat(s)
    if case["kind"] == "adjoint":
        return _run_adjoint(s)
    tw = s["twin"]
    g = tw.grid
    g.load_state(s["state"])
    for x, y in s["path"]:
        tw.step(x, y, True)
    out = {name: getattr(g, name) for name in STATE_OUT}
    if case["lorentz"]:
        for name in ("phi_elec", "Jx", "Jy", "Jz", "Bx", "By", "Bz"):
            out[name] = getattr(g, name)
    if case["drops"]:
        # the job's monitor: pool size, temperatures and mass balance
        t = tw.get_telemetry()
        out["telemetry"] = {k: t[k] for k in ("peak_temp_K", "n_liquid_cells", "pool_width_mm",
                                              "pool_length_mm", "total_enthalpy_J")}
    return out


def _adjoint_case(case):
    return _steps(**{k: case[k] for k in ("nx", "ny", "nz", "dx", "steps")}, power=3000.0,
                  heat_loss=True)


def _adjoint_probes(case, seed, nz_solid):
    r = np.random.default_rng(seed + 1)
    ti, tj = _start_of_path(case, seed)
    out = []
    for _ in range(8):
        side = 1 if r.random() < 0.5 else -1
        off = r.uniform(2e-3, 6e-3) / case["dx"] * side
        out.append((int(ti + r.uniform(-8.0, 12.0)), int(min(max(tj + off, 1), case["ny"] - 2)),
                    nz_solid - 1))
    return out


def _prepare_adjoint(case, seed, device):
    full = _adjoint_case(case)
    tw = _twin(full)
    tw.reset()
    tw.grid.load_state(_pool_state(full, seed, tw.nz_solid, device))
    path = _positions(full, seed, tw.grid.dt)
    probes = _adjoint_probes(case, seed, tw.nz_solid)
    # measured traces: the pool cools along them, the width a little over the run's
    r = np.random.default_rng(seed + 2)
    T0 = np.array([float(tw.grid.T[p]) for p in probes])
    target = T0[None, :] + r.uniform(2.0, 10.0, len(probes))[None, :] * \
        np.linspace(0.1, 1.0, case["steps"])[:, None]
    prob = AdjointProblem(tw, path, probes, T_target=target, W_target=6.0, w_T=1e-3, w_W=10.0)
    return dict(case=case, problem=prob, theta=torch.tensor(prob.theta, dtype=torch.float64))


def _run_adjoint(s):
    theta = s["theta"].clone().requires_grad_(True)
    loss = CoupledStepLoss.apply(theta, s["problem"])
    loss.backward()
    return dict(loss=loss.detach(), grad=theta.grad, probes=s["problem"].T_probe,
                f_l=s["problem"].fl_final)


# ---- the operator cases ---------------------------------------------------------

CHANNEL_TAU, CHANNEL_FX = 0.8, 1e-5


def _channel_start(case, seed, device):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    f32 = dict(dtype=torch.float32, device=device)
    j = torch.arange(ny, **f32).view(1, ny, 1)
    k = torch.arange(nz, **f32).view(1, 1, nz)
    i = torch.arange(nx, **f32).view(nx, 1, 1)
    wall = ((j == 0) | (j == ny - 1) | (k == 0) | (k == nz - 1)).expand(nx, ny, nz)
    flags = torch.where(wall, SOLID, FLUID).to(torch.int32).contiguous()
    u = [0.02 * torch.sin(2 * math.pi * (i / nx + a * j / ny + b * k / nz)) +
         _noise((nx, ny, nz), gen, 2e-3) for a, b in ((1, 2), (2, 1), (1, 1))]
    rho = 1.0 + _noise((nx, ny, nz), gen, 1e-3)
    u2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    f = torch.empty((19, nx, ny, nz), **f32)
    for q in range(19):
        eu = EX[q] * u[0] + EY[q] * u[1] + EZ[q] * u[2]
        f[q] = W[q] * rho * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * u2)
    return f, flags


def _prepare_flow(case, seed, device):
    tw = WAAMTwin(material=from_constants("steel", STEEL), nx=case["nx"], ny=case["ny"],
                  nz=case["nz"], dx=3e-4, C_darcy=0.0, max_tracers=16)
    g = tw.grid
    f, flags = _channel_start(case, seed, device)
    g.flags.copy_(flags)
    g.f_l.fill_(1.0)
    g.phi.fill_(1.0)
    return dict(case=case, twin=tw, f=f)


def _run_flow(s):
    case, tw = s["case"], s["twin"]
    g = tw.grid
    g.load_state(dict(f_a=s["f"], f_b=s["f"], read_is_a=True))
    om = 1.0 / CHANNEL_TAU
    kernels.set_uniform_Fx(g.Fx, g.Fy, g.Fz, CHANNEL_FX, g.flags, g.FLAG_FLUID)
    for _ in range(case["steps"]):
        a, b = g.f_src, g.f_dst
        if case["srt"]:
            lbm.collide_srt(a, b, g.rho, g.ux, g.uy, g.uz, g.Fx, g.Fy, g.Fz, g.f_l, g.flags,
                            CHANNEL_TAU, om, 1.0, 0.0, g.FLAG_SOLID, g.FLAG_GAS, g.nx, g.ny, g.nz)
        else:
            lbm.collide_mrt(a, b, g.rho, g.ux, g.uy, g.uz, g.Fx, g.Fy, g.Fz, g.f_l, g.flags, g.ex,
                            g.ey, g.ez, g.w, g.opp, om, om, 0.0, g.FLAG_SOLID, g.FLAG_GAS, g.nx,
                            g.ny, g.nz)
        lbm.stream(b, a, g.flags, g.FLAG_SOLID, g.FLAG_GAS, g.nx, g.ny, g.nz)
        g.swap_buffers()
    return dict(f_src=g.f_src, f_dst=g.f_dst, rho=g.rho, ux=g.ux, uy=g.uy, uz=g.uz)


HEAT_DX = 3e-4


def _heat_case(case):
    return _steps(nx=case["nx"], ny=case["ny"], nz=case["nz"], dx=HEAT_DX, steps=case["steps"],
                  heat_loss=True)


def _prepare_heat(case, seed, device):
    tw = _twin(_heat_case(case))
    tw.reset()
    return dict(case=case, twin=tw, state=_pool_state(_heat_case(case), seed, tw.nz_solid, device))


def _run_heat(s):
    case, tw = s["case"], s["twin"]
    g, m = tw.grid, tw.mat
    g.load_state(s["state"])
    H, T = g.H, g.T
    for _ in range(case["steps"]):
        thermal.advect_diffuse_temperature(H, T, g.ux, g.uy, g.uz, g.flags, tw.alpha_lu, 1.0,
                                           g.FLAG_SOLID, g.FLAG_GAS, tw.cp_rho, g.nx, g.ny, g.nz)
        thermal.apply_boundary_losses(H, T, g.flags, tw.T_amb, tw.h_conv, tw.eps_rad, 1, 1,
                                      tw.cp_rho, g.dt, g.dx, tw.sigma_sb, g.FLAG_SOLID,
                                      g.FLAG_GAS, g.nx, g.ny, g.nz)
        phase_change.update_phase(H, T, g.f_l, tw.cp_rho, tw.L_rho, m.T_solidus, m.T_liquidus)
        thermal.update_T_max(T, g.T_max, g.flags, g.FLAG_GAS)
        thermal.update_cooling_rate(T, g.T_prev, g.dT_dt, g.flags, g.dt, g.FLAG_GAS)
    return dict(H=H, T=T, f_l=g.f_l, T_max=g.T_max, T_prev=g.T_prev, dT_dt=g.dT_dt)


# ---- what a pass cannot do without ------------------------------------------------

def work(case):
    n, steps = case["nx"] * case["ny"] * case["nz"], case["steps"]
    nz_solid = max(1, min(case["nz"] // 5, case["nz"] - max(6, case["nz"] // 4)))
    open_cells = n * (case["nz"] - nz_solid) / case["nz"]
    if case["kind"] == "flow":
        # per iteration: collision reads and writes 19 populations, reads F, f_l,
        # flags, writes rho and u; the stream reads and writes 19 and the flags
        return dict(bytes=n * steps * (4 * 76 + 20 + 16 + 4), flops=n * steps * 350)
    if case["kind"] == "heat":
        # H, T, f_l, T_max, T_prev, dT_dt, u and flags, once per iteration
        return dict(bytes=n * steps * (4 * 5 + 4 * 6 + 4 * 4), flops=n * steps * 120)
    metal = n - 0.9 * open_cells
    # per step: the stream reads and writes 19 populations of every cell that is
    # not SOLID; H, T, phi, f_l, flags are read and written, the histories of
    # the metal cells too
    pop = 2 if case.get("storage", "float32") != "float32" else 4
    per = open_cells * 2 * 19 * pop + n * 40 + metal * 24
    if case.get("lorentz"):
        per += n * (2 + 6) * 4          # sigma, source, J and B written
    if case.get("tables"):
        per += n * 16                   # the four property fields
    if case["kind"] == "adjoint":
        # the forward step, its repetition with a tape, and the reverse step
        # (adjoint populations of two buffers, H, T, f_l and u)
        per = 2 * per + open_cells * 4 * 76 + n * 80
    return dict(bytes=per * steps, flops=metal * steps * 150)


def tolerance(case):
    # Rounding alone, about four times what the paths show against the float64
    # restatement.  The cooling rate is a difference of two temperatures a step
    # apart; at a flat interface the direction of the surface tension is a
    # quotient of two rounding errors; 16-bit populations round by 1e-3.
    if case["kind"] == "flow":
        return dict(rel=2e-5, max=1e-2)
    if case["kind"] == "heat":
        return dict(rel=6e-4, max=1e-1)
    if case["kind"] == "adjoint":
        return dict(rel=1e-3, max=0.1)
    if case["wet"] or case["storage"] != "float32":
        return dict(rel=2e-2, max=0.9, differ=1e-5)
    return dict(rel=5e-4, max=0.5, differ=1e-5)


# ---- the same in float64 ----------------------------------------------------------

def exact(case, seed):
    """run() in float64, or None: the droplet's cells are placed one after
    another, each depending on the last (minutes in array operations), and a
    Lorentz job starts from the potential that its own earlier steps left,
    thousands of sweeps of the largest grid."""
    device = torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() \
        else torch.device("cpu")
    if case["kind"] == "flow":
        return _exact_flow(case, seed, device)
    if case["kind"] == "heat":
        return _exact_heat(case, seed, device)
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed, device)
    if case["drops"] or case["lorentz"]:
        return None
    e = _Exact(case, seed, device)
    for x, y in _positions(case, seed, e.dt):
        e.step(x, y)
    out = {name: e.out(name) for name in STATE_OUT}
    if case["wet"]:
        # no exact value: see tolerance() on flat interfaces
        out.update(Fx=None, Fy=None, Fz=None)
    return out


def _shift(a, axis, d, wrap=False):
    """a at the neighbour d cells along axis (clamped, or periodic)."""
    n = a.shape[axis]
    at = torch.arange(n, device=a.device) + d
    at = at % n if wrap else at.clamp(0, n - 1)
    return a.index_select(axis, at)


def _interp(T, knots):
    t = torch.tensor([a for a, _ in knots], dtype=T.dtype, device=T.device)
    v = torch.tensor([b for _, b in knots], dtype=T.dtype, device=T.device)
    at = torch.searchsorted(t, T.contiguous()).clamp(1, len(knots) - 1)
    x = ((T - t[at - 1]) / (t[at] - t[at - 1])).clamp(0.0, 1.0)
    return v[at - 1] + x * (v[at] - v[at - 1])


def _properties(T, flags, case, dtype=torch.float64):
    """rho cp, alpha, dgamma and tau of each cell from the temperature tables."""
    m, dx = STEEL, case["dx"]
    dt = dx * 0.1
    scale = dt ** 2 / (m["rho"] * dx ** 2) / dx
    kn = _table_knots()
    T = T.double()
    fixed = (flags == SOLID) | (flags == GAS)
    cp, k, mu, dg = (_interp(T, kn[name]) for name in ("cp", "k", "mu", "dgamma_dT"))
    to_lu = dt / dx ** 2
    const = dict(cp_rho_field=m["rho"] * m["cp"], alpha_lu_field=m["k"] / (m["rho"] * m["cp"]) * to_lu,
                 dgamma_lu_field=m["dgamma_dT"] * scale, tau_field=3 * m["mu"] / m["rho"] * to_lu + 0.5)
    cell = dict(cp_rho_field=m["rho"] * cp, alpha_lu_field=k / (m["rho"] * cp) * to_lu,
                dgamma_lu_field=dg * scale, tau_field=3 * mu / m["rho"] * to_lu + 0.5)
    return {name: torch.where(fixed, torch.full_like(v, const[name]), v).to(dtype)
            for name, v in cell.items()}


def _advect_diffuse(H, T, u, flags, cp_alpha):
    gas = flags == GAS

    def masked(f, axis, d, fallback):
        return torch.where(_shift(gas, axis, d), fallback, _shift(f, axis, d))

    lap = -6.0 * T
    for axis in range(3):
        lap = lap + masked(T, axis, 1, T) + masked(T, axis, -1, T)
    adv = torch.zeros_like(H)
    for axis in range(3):
        m, p = masked(H, axis, -1, H), masked(H, axis, 1, H)
        mm, pp = masked(H, axis, -2, m), masked(H, axis, 2, p)
        up = u[axis] > 0.0
        d1 = torch.where(up, H - m, p - H)
        d2 = torch.where(up, 0.5 * (3 * H - 4 * m + mm), 0.5 * (-3 * H + 4 * p - pp))
        grad = torch.where(d1 * d2 > 0, torch.where(d1.abs() < d2.abs(), d1, d2),
                           torch.zeros_like(H))
        adv = adv + u[axis] * grad
    dH = cp_alpha * lap - torch.where(flags == SOLID, torch.zeros_like(adv), adv)
    return torch.where(gas, H, H + dH)


def _boundary_losses(H, T, flags, h_conv, eps_rad, conv, rad, dt, dx):
    gas = flags == GAS
    faces = torch.zeros_like(H)
    for axis, d in ((2, 1), (1, 1), (1, -1), (0, 1), (0, -1)):
        at = torch.arange(H.shape[axis], device=H.device) + d
        inside = ((at >= 0) & (at < H.shape[axis])).view([-1 if a == axis else 1 for a in range(3)])
        faces = faces + (_shift(gas, axis, d) & inside)
    Te = T.clamp(max=2500.0)
    q = torch.zeros_like(H)
    if conv:
        q = q + h_conv * (Te - T_AMB)
    if rad:
        q = q + eps_rad * 5.670374419e-8 * (Te ** 4 - T_AMB ** 4)
    return torch.where(gas, H, H - q * faces * dt / dx)


def _phase(H, cp_rho, L_rho, H_sol, Ts, Tl):
    fl = ((H - H_sol) / L_rho).clamp(0.0, 1.0)
    T = torch.where(H <= H_sol, H / cp_rho, torch.where(
        H >= H_sol + L_rho, Tl + (H - H_sol - L_rho) / cp_rho, Ts + fl * (Tl - Ts)))
    return T, fl


def _moments(f):
    r = f.sum(0)
    j = [sum(e[q] * f[q] for q in range(1, 19) if e[q]) for e in (EX, EY, EZ)]
    return r, j


def _collide(f, F, fl, omega, C_darcy, srt):
    """Collided populations, density and velocity of a list of cells (19, n)."""
    r, j = _moments(f)
    om = 1.0 - fl
    ck = 1.0 + C_darcy * om * om / (fl ** 3 + 1e-6)
    u = [(a + 0.5 * b) / (r + 1e-6) / ck for a, b in zip(j, F)]
    u2 = sum(a * a for a in u)
    uF = sum(a * b for a, b in zip(u, F))
    out = torch.empty_like(f)
    if not srt:
        E = (EX, EY, EZ)
        P = {(a, b): sum(E[a][q] * E[b][q] * f[q] for q in range(19) if E[a][q] * E[b][q])
             for a in range(3) for b in range(a, 3)}
        kap = {ab: P[ab] - r * u[ab[0]] * u[ab[1]] for ab in P}
        km = (kap[0, 0] + kap[1, 1] + kap[2, 2]) / 3.0
        kmp = km - omega * (km - r / 3.0)
        post = {(a, b): (kmp + (1.0 - omega) * (kap[a, a] - km) - r / 3.0) if a == b
                else (1.0 - omega) * kap[a, b] for a, b in kap}
    for q in range(19):
        e = (EX[q], EY[q], EZ[q])
        eu = sum(e[a] * u[a] for a in range(3))
        Fe = sum(e[a] * F[a] for a in range(3))
        feq = r * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * u2)
        S = W[q] * (1.0 - 0.5 * omega) * (3.0 * Fe + 9.0 * eu * Fe - 3.0 * uF)
        if srt:
            out[q] = f[q] - omega * (f[q] - W[q] * feq) + S
        else:
            K = sum(e[a] * e[b] * post[a, b] * (1.0 if a == b else 2.0)
                    for a, b in post if e[a] * e[b])
            out[q] = W[q] * (feq + 4.5 * K) + S
    return out, r, u


def _stream(src, dst, flags):
    solid, gas = flags == SOLID, flags == GAS
    for q in range(19):
        def pull(a):
            a = _shift(a, 0, -EX[q], wrap=True) if EX[q] else a
            a = _shift(a, 1, -EY[q]) if EY[q] else a
            return _shift(a, 2, -EZ[q]) if EZ[q] else a
        v = torch.where(pull(solid) & ~gas, src[OPP[q]], pull(src[q]))
        dst[q] = torch.where(solid, dst[q], v)


class _Exact:
    """The coupled step in float64 array operations, from the stored state."""

    def __init__(self, case, seed, device):
        self.c = case
        nz = case["nz"]
        self.nz_solid = max(1, min(nz // 5, nz - max(6, nz // 4)))
        st = _pool_state(case, seed, self.nz_solid, device)
        self.flags = st.pop("flags")
        st.pop("read_is_a")
        self.s = {k: v.double() for k, v in st.items()}
        self.src, self.dst = self.s.pop("f_a").clone(), self.s.pop("f_b").clone()
        m, dx = STEEL, case["dx"]
        self.dt = dx * 0.1
        self.cp_rho, self.L_rho = m["rho"] * m["cp"], m["rho"] * m["L_fusion"]
        self.to_lu = self.dt / dx ** 2
        self.alpha = m["k"] / self.cp_rho * self.to_lu
        self.omega = 1.0 / (3 * m["mu"] / m["rho"] * self.to_lu + 0.5)
        self.scale = self.dt ** 2 / (m["rho"] * dx ** 2) / dx
        self.g_lu = 9.81 * self.dt ** 2 / dx
        self.cp_ts = m["cp"]
        if case["tables"]:
            self.cp_ts = float(_interp(torch.tensor([m["T_solidus"]], dtype=torch.float64),
                                       _table_knots()["cp"]))
        self.H_sol = m["rho"] * self.cp_ts * m["T_solidus"]
        self.H_liq = self.H_sol + self.L_rho
        nx, ny = case["nx"], case["ny"]
        f64 = dict(dtype=torch.float64, device=device)
        self.i = torch.arange(nx, **f64).view(nx, 1, 1)
        self.j = torch.arange(ny, **f64).view(1, ny, 1)
        self.k = torch.arange(nz, **f64).view(1, 1, nz)

    def out(self, name):
        if name == "flags":
            return self.flags
        if name in ("f_src", "f_dst"):
            f = self.src if name == "f_src" else self.dst
            if self.c["storage"] != "float32":      # the buffers hold f_q - w_q
                f = f - torch.tensor(W, dtype=f.dtype, device=f.device).view(19, 1, 1, 1)
            return f
        return self.s[name]

    def _ceiling(self, H, cp_rho):
        m, cap = STEEL, 3200.0
        top = torch.where(H > self.H_liq, self.H_liq + cp_rho * (cap - m["T_liquidus"]),
                          cp_rho * cap + torch.zeros_like(H))
        return torch.where(self.flags == GAS, H, torch.minimum(H, top))

    def _inject(self, arc, cp_rho):
        c, s = self.c, self.s
        di, dj, dk = self.i - arc[0], self.j - arc[1], self.k - arc[2]
        dx = c["dx"]
        if c["source"] == "goldak":
            cell = {k: v * 1e-3 / dx for k, v in GOLDAK_MM.items() if k.endswith("_mm")}
            a = torch.where(di >= 0, cell["a_front_mm"], cell["a_rear_mm"]).double()
            frac = torch.where(di >= 0, GOLDAK_MM["ff"], GOLDAK_MM["fr"]).double()
            shape = frac * torch.exp(-3.0 * (di * di / (a * a + 1e-6) +
                                             dj * dj / (cell["b_mm"] ** 2 + 1e-6) +
                                             dk * dk / (cell["c_mm"] ** 2 + 1e-6)))
        else:
            sig = 2e-3 / dx
            shape = torch.exp(-(di * di + dj * dj + 0.25 * dk * dk) / (2 * sig * sig))
        dz = arc[2] - self.k
        depth = torch.where(dz < -0.5, torch.zeros_like(dz),
                            torch.exp(-dz.clamp(min=0.0) / (2e-3 / dx + 1e-6)))
        wd = torch.where(s["f_l"] > 0.55, torch.ones_like(s["f_l"]), depth.expand_as(s["f_l"]))
        w = torch.where((self.flags == GAS) | (wd < 1e-6), torch.zeros_like(wd), shape * wd)
        return self._ceiling(s["H"] + c["power"] * 0.78 * self.dt / (w.sum() * dx ** 3) * w, cp_rho)

    def _vof(self):
        s, flags = self.s, self.flags
        solid, gas, phi = flags == SOLID, flags == GAS, s["phi"]
        div = torch.zeros_like(phi)
        for axis, name in ((0, "ux"), (1, "uy"), (2, "uz")):
            wrap = axis == 0
            u = torch.where(gas | solid, torch.zeros_like(phi), s[name])
            up = _shift(u, axis, 1, wrap)
            uf = 0.5 * (u + up)
            flux = uf * torch.where(uf > 0, phi, _shift(phi, axis, 1, wrap))   # east / north / top face
            flux = torch.where(solid | _shift(solid, axis, 1, wrap), torch.zeros_like(flux), flux)
            n = phi.shape[axis]
            if not wrap:
                flux.index_fill_(axis, torch.tensor([n - 1], device=phi.device), 0.0)
            low = _shift(flux, axis, -1, wrap)
            if not wrap:
                low = low.index_fill(axis, torch.tensor([0], device=phi.device), 0.0)
            div = div + (flux - low)
        phi = torch.where(solid, torch.ones_like(phi), (phi - div))
        phi = torch.where(gas, torch.where(phi < 1e-6, torch.zeros_like(phi), phi.clamp(max=1.0)),
                          phi.clamp(0.0, 1.0))
        if self.c["wet"]:
            phi = self._wetting(phi)
        fl, k = s["f_l"], self.k.expand_as(phi)
        new = torch.full_like(flags, IFACE)
        new[phi < 0.05] = GAS
        new[(phi > 0.55) & (fl > 0.1)] = FLUID
        new[(phi > 0.85) & (fl < 0.05)] = SOLID
        new[k < self.nz_solid] = SOLID
        s["phi"], self.flags = phi, new
        s["f_l"] = torch.where((new == GAS) | (new == SOLID) | (phi < 0.05), torch.zeros_like(fl), fl)

    def _wetting(self, phi):
        """Contact angle, cell after cell up each column."""
        old, phi = phi, phi.clone()
        flags, th = self.flags, math.radians(30.0)
        sin_t = math.sin(th)
        film = 0.5 * (1.0 - math.cos(th))
        spread = film * (0.85 + 0.15 * sin_t)
        metal = old > 0.55
        near = torch.zeros_like(metal)
        near[1:] |= metal[:-1]
        near[:-1] |= metal[1:]
        near[:, 1:] |= metal[:, :-1]
        near[:, :-1] |= metal[:, 1:]
        nz = phi.shape[2]
        for k in range(nz):
            flag, p = flags[:, :, k], phi[:, :, k]
            opn, gas = flag != SOLID, flag == GAS
            on_solid = (flags[:, :, k - 1] == SOLID) & opn if k else torch.zeros_like(opn)
            p = torch.where(on_solid & gas, p.clamp(min=film), p)
            if k + 1 < nz:
                up = on_solid & (p > 0.55) & (flags[:, :, k + 1] == GAS)
                ghost = torch.maximum(phi[:, :, k + 1], (p - sin_t).clamp(max=0.98).clamp(min=film))
                phi[:, :, k + 1] = torch.where(up, ghost, phi[:, :, k + 1])
            if k:
                below = phi[:, :, k - 1]
                t = (below - sin_t).clamp(max=0.95).clamp(min=film)
                p = torch.where(gas & (below > 0.55), torch.maximum(p, t), p)
            p = torch.where(opn & (p < 0.45) & near[:, :, k], p.clamp(min=spread), p)
            p = torch.where(on_solid & (p > 0.2), p.clamp(min=0.65), p)
            phi[:, :, k] = p
        return phi

    def _forces(self, arc, dgamma):
        c, s, flags = self.c, self.s, self.flags
        phi, T, fl = s["phi"], s["T"], s["f_l"]
        active = (flags == FLUID) | (flags == IFACE)
        zero = torch.zeros_like(phi)
        dp = [0.5 * (_shift(phi, a, 1) - _shift(phi, a, -1)) for a in range(3)]
        g = (dp[0] ** 2 + dp[1] ** 2 + dp[2] ** 2).sqrt()
        some = g >= 1e-6
        nrm = [torch.where(some, a / g.clamp(min=1e-30), zero) for a in dp]
        F = [zero, zero, zero]
        if c["wet"]:
            div = zero
            for a in range(3):
                hi = torch.where(_shift(some, a, 1), _shift(nrm[a], a, 1), nrm[a])
                lo = torch.where(_shift(some, a, -1), _shift(nrm[a], a, -1), nrm[a])
                div = div + 0.5 * (hi - lo)
            tension = -STEEL["gamma_0"] * self.scale * div
            inner = torch.zeros_like(active)
            inner[1:-1, 1:-1, 1:-1] = True
            csf = [tension * a for a in self._wall_gradient(dp, nrm, g)]
            F = [torch.where(inner & some, a, zero) for a in csf]
        dT = [0.5 * (_shift(T, a, 1) - _shift(T, a, -1)) for a in range(3)]
        nd = sum(a * b for a, b in zip(nrm, dT))
        wet = some & (fl >= 0.05)
        F = [a + torch.where(wet, dgamma * g * (t - nd * n), zero) for a, t, n in zip(F, dT, nrm)]
        sig = 2e-3 / c["dx"]
        Flu = 500.0 / (STEEL["rho"] * c["dx"]) * self.dt ** 2 / c["dx"]
        r2 = (self.i - arc[0]) ** 2 + (self.j - arc[1]) ** 2 + 0.1 * (self.k - arc[2]) ** 2
        press = -Flu * torch.exp(-r2 / (2 * sig * sig + 1e-6))
        F[2] = F[2] + torch.where((2.0 * dp[2]).abs() > 0.05, press, zero)
        if c["wet"]:
            F[2] = F[2] - self.g_lu * fl
        F[2] = F[2] + self.g_lu * STEEL["beta_T"] * (T - STEEL["T_liquidus"]) * fl
        F = [torch.where(active, a, zero) for a in F]
        mag = (F[0] ** 2 + F[1] ** 2 + F[2] ** 2).sqrt()
        cut = torch.where(mag > 0.05, 0.05 / (mag + 1e-12), torch.ones_like(mag))
        return [a * cut for a in F], active

    def _wall_gradient(self, dp, nrm, g):
        """grad phi, turned to the contact angle at cells that touch a wall."""
        solid = self.flags == SOLID
        th = math.radians(30.0)
        wall = []
        for a in range(3):
            lo, hi = _shift(solid, a, -1).clone(), _shift(solid, a, 1).clone()
            lo.select(a, 0).fill_(False)
            hi.select(a, solid.shape[a] - 1).fill_(False)
            wall.append((lo, hi))
        touches = sum(lo.int() + hi.int() for lo, hi in wall) > 0
        w = [lo.double() - hi.double() for lo, hi in wall]
        wm = sum(a * a for a in w).sqrt()
        w = [torch.where(wm > 1e-8, a / wm.clamp(min=1e-30), a) for a in w]
        dot = sum(a * b for a, b in zip(nrm, w))
        t = [a - dot * b for a, b in zip(nrm, w)]
        tm = sum(a * a for a in t).sqrt()
        along = tm > 1e-8
        turned = [math.cos(th) * b + math.sin(th) * a / tm.clamp(min=1e-30) for a, b in zip(t, w)]
        up, side = w[2].abs() > 0.5, w[0].abs() > 0.5
        ct, st = torch.full_like(g, math.cos(th)), torch.full_like(g, math.sin(th))
        zero = torch.zeros_like(g)
        bare = [torch.where(up, st, torch.where(side, ct, ct * w[0] + st)),
                torch.where(up, zero, torch.where(side, st, ct * w[1])),
                torch.where(up, ct, torch.where(side, zero, ct * w[2]))]
        nc = [torch.where(along, a, b) for a, b in zip(turned, bare)]
        cm = sum(a * a for a in nc).sqrt()
        nc = [torch.where(cm > 1e-8, a / cm.clamp(min=1e-30), a) for a in nc]
        return [torch.where(touches, a * g, b) for a, b in zip(nc, dp)]

    def step(self, x, y):
        c, s, m = self.c, self.s, STEEL
        dx, tables = c["dx"], c["tables"]
        ai, aj = x / dx, y / dx
        col = (min(max(int(np.float32(ai)), 0), c["nx"] - 1), min(max(int(np.float32(aj)), 0), c["ny"] - 1))
        metal = (self.flags[col] != GAS) & (s["phi"][col] > 0.05)
        top = int(metal.nonzero().max()) if bool(metal.any()) else max(1, self.nz_solid - 1)
        arc = (ai, aj, float(top if top >= 1 else max(1, self.nz_solid - 1)))
        Ts, Tl = m["T_solidus"], m["T_liquidus"]
        s["H"] = self._inject(arc, s["cp_rho_field"] if tables else self.cp_rho)
        cp_rho, alpha, dgamma = self.cp_rho, self.alpha, m["dgamma_dT"] * self.scale
        if tables:
            s.update(_properties(s["T"], self.flags, c))
            cp_rho, alpha, dgamma = s["cp_rho_field"], s["alpha_lu_field"], s["dgamma_lu_field"]
        H = _advect_diffuse(s["H"], s["T"], (s["ux"], s["uy"], s["uz"]), self.flags, cp_rho * alpha)
        gas = self.flags == GAS
        if c["heat_loss"]:
            H = _boundary_losses(H, s["T"], self.flags, 25.0, 0.3, True, False, self.dt, dx)
            H = torch.where(gas, H, torch.maximum(H, cp_rho * T_AMB + torch.zeros_like(H)))
        H = self._ceiling(H, cp_rho)
        T, fl = _phase(H, cp_rho, self.L_rho, self.H_sol, Ts, Tl)
        s["H"], s["T"], s["f_l"] = H, T, fl
        s["T_max"] = torch.where(gas, s["T_max"], torch.maximum(s["T_max"], T))
        s["dT_dt"] = torch.where(gas, s["dT_dt"], (T - s["T_prev"]) / (self.dt + 1e-12))
        s["T_prev"] = torch.where(gas, s["T_prev"], T)
        self._vof()
        F, active = self._forces(arc, dgamma)
        s["Fx"], s["Fy"], s["Fz"] = F
        at = active.reshape(-1).nonzero().squeeze(1)
        pick = lambda a: a.reshape(-1)[at]  # noqa: E731
        omega = self.omega
        if tables:
            omega = 1.0 / (pick(s["tau_field"]) + 1e-6)
        f, r, u = _collide(self.src.view(19, -1)[:, at], [pick(a) for a in F], pick(s["f_l"]), omega,
                           1.6e5, tables or c["srt"])
        self.dst.view(19, -1)[:, at] = f
        mag = sum(a * a for a in u).sqrt()
        cut = torch.where(mag > 0.08, 0.08 / (mag + 1e-12), torch.ones_like(mag))
        for name, v in zip(("rho", "ux", "uy", "uz"), [r] + [a * cut for a in u]):
            s[name] = s[name].reshape(-1).index_copy(0, at, v).view_as(s[name])
        _stream(self.dst, self.src, self.flags)
        self.src, self.dst = self.dst, self.src
        warm = self.flags != GAS
        for name, T0 in (("time_above_800_s", 1073.15), ("time_above_1100_s", 1373.15),
                         ("time_above_solidus_s", Ts)):
            s[name] = s[name] + self.dt * (warm & (s["T"] >= T0))
        if tables:
            self._tail(arc)

    def _tail(self, arc):
        """Remelt hot solid, freeze the pool's tail, solidify cooled metal."""
        s, m = self.s, STEEL
        Ts, Tl, cp = m["T_solidus"], m["T_liquidus"], s["cp_rho_field"]
        melt = (self.flags == SOLID) & (s["T"] > Ts + 5.0)
        fl = ((s["T"] - Ts) / (Tl - Ts + 1e-6)).clamp(max=1.0)
        full = s["T"] >= Tl
        fl = torch.where(full, torch.ones_like(fl), fl)
        h = torch.where(full, cp * s["T"] + self.L_rho, cp * Ts + fl * self.L_rho)
        s["H"] = torch.where(melt, h, s["H"])
        s["f_l"] = torch.where(melt, fl, s["f_l"])
        s["phi"] = torch.where(melt, torch.ones_like(h), s["phi"])
        self.flags = torch.where(melt, torch.full_like(self.flags, FLUID), self.flags)
        behind = (self.i - arc[0]) <= -max(2.0, 2.5e-3 / self.c["dx"])
        freeze = (self.flags != GAS) & (s["phi"] >= 0.85) & (s["f_l"] >= 0.05) & behind & \
            (s["T"] < Tl + 35.0)
        s["H"] = torch.where(freeze, cp * (Ts - 1.0), s["H"])
        s["T"] = torch.where(freeze, torch.full_like(h, Ts - 1.0), s["T"])
        s["f_l"] = torch.where(freeze, torch.zeros_like(h), s["f_l"])
        cold = freeze | ((self.flags != GAS) & (s["phi"] >= 0.85) & (s["f_l"] < 0.02) & (s["T"] < Ts))
        self.flags = torch.where(cold, torch.full_like(self.flags, SOLID), self.flags)
        s["phi"] = torch.where(cold, torch.ones_like(h), s["phi"])
        for name in ("f_l", "ux", "uy", "uz"):
            s[name] = torch.where(cold, torch.zeros_like(h), s[name])


def _exact_flow(case, seed, device):
    f, flags = _channel_start(case, seed, device)
    src, dst = f.double(), f.double().clone()
    at = (flags == FLUID).reshape(-1).nonzero().squeeze(1)
    n = flags.numel()
    F = [torch.full((len(at),), v, dtype=torch.float64, device=device) for v in (CHANNEL_FX, 0.0, 0.0)]
    one = torch.ones_like(F[0])
    for _ in range(case["steps"]):
        g, r, u = _collide(src.view(19, n)[:, at], F, one, 1.0 / CHANNEL_TAU, 0.0, case["srt"])
        dst.view(19, n)[:, at] = g
        _stream(dst, src, flags)
        src, dst = dst, src
    # walls keep the zeros that the grid was made with
    out = {name: torch.zeros(n, dtype=torch.float64, device=device).index_copy(0, at, v).view(flags.shape)
           for name, v in zip(("rho", "ux", "uy", "uz"), [r] + u)}
    return dict(out, f_src=src, f_dst=dst)


def _exact_heat(case, seed, device):
    full = _heat_case(case)
    e = _Exact(full, seed, device)
    s, m = e.s, STEEL
    gas = e.flags == GAS
    for _ in range(case["steps"]):
        H = _advect_diffuse(s["H"], s["T"], (s["ux"], s["uy"], s["uz"]), e.flags, e.cp_rho * e.alpha)
        s["H"] = _boundary_losses(H, s["T"], e.flags, 25.0, 0.3, True, True, e.dt, full["dx"])
        s["T"], s["f_l"] = _phase(s["H"], e.cp_rho, e.L_rho, e.H_sol, m["T_solidus"], m["T_liquidus"])
        s["T_max"] = torch.where(gas, s["T_max"], torch.maximum(s["T_max"], s["T"]))
        s["dT_dt"] = torch.where(gas, s["dT_dt"], (s["T"] - s["T_prev"]) / (e.dt + 1e-12))
        s["T_prev"] = torch.where(gas, s["T_prev"], s["T"])
    return {name: s[name] for name in ("H", "T", "f_l", "T_max", "T_prev", "dT_dt")}


def _exact_adjoint(case, seed, device):
    """The forward half; the gradient's kernels are the adjoint of the float32
    trajectory (its branches frozen), which has no float64 value of its own."""
    full = _adjoint_case(case)
    e = _Exact(full, seed, device)
    probes = _adjoint_probes(case, seed, e.nz_solid)
    rows = []
    for x, y in _positions(full, seed, e.dt):
        e.step(x, y)
        rows.append([float(e.s["T"][p]) for p in probes])
    return dict(loss=None, grad=None, probes=np.array(rows), f_l=e.s["f_l"])
