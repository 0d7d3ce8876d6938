"""The framework's work as its users have it done, case by case, through the public entry points.

Every case is one of six kinds of call:

  solve     one velocity solve (solve_DIVA) of a geometry held on the device, from a cold start: the saved
            initial state restored, the solve, and the velocities the caller reads downloaded
  restart   a solve whose inputs come from host buffers, from approximate velocities (a learned guess, a
            restart file without viscosity, observations): uploads, data model, rheology, state completion,
            solve, SIA velocities, downloads
  ensemble  the members of an ensemble solved by one persistent batch
  step      time steps of the predictor/corrector scheme with the heat equation, from a saved model state
  sia       the shallow-ice velocities of a changed geometry: upload, data model, rheology, solve_SIA
  net       the warm-start network on device buffers: inference, or one training step

Geometries are the package's seeded synthetic ones (marine channel, ice cap, continental sheet); their sizes
follow from the grid spacing.  The caps and the sheet end on land (the sea stands below their bed) and have a
stronger friction, the channels have the floating ice and at least 50 m of ice on their walls: ponds of
free-floating, frictionless ice, ice that vanishes against a wall, or flow that runs into the velocity limit give
systems whose answer two correct solvers, or two builds of one, agree on to a few digits only.
"""
import copy
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """imau-ice_b200/ (a folder name with a hyphen) as the module imau_ice_b200."""
    if "imau_ice_b200" not in sys.modules:
        d = os.path.join(ROOT, "imau-ice_b200")
        spec = importlib.util.spec_from_file_location("imau_ice_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["imau_ice_b200"] = mod
        spec.loader.exec_module(mod)


_package()
from imau_ice_b200 import diva, dynamics, learned, synth  # noqa: E402

GEOMETRY = {"channel": synth.marine_channel, "icecap": synth.ice_cap, "sheet": synth.ice_sheet}
# points along each direction: 1 + 2 floor(half width / dx)
HALF = {"channel": (320e3, 40e3), "icecap": (800e3, 1400e3), "sheet": (3000e3, 3000e3)}
NZ = 15
VELOCITIES = ["u_vav_cx", "v_vav_cy", "u_surf_cx", "v_surf_cy", "u_base_cx", "v_base_cy"]
INPUTS = ["Hi_a", "Hb_a", "SL_a", "dHb_dt_a", "Ti_a", "beta_sq_a"]
RESTART_OUT = ["u_vav_cx", "v_vav_cy", "u_surf_cx", "v_surf_cy", "u_base_cx", "v_base_cy", "u_3D_cx", "v_3D_cy"]
SIA_OUT = ["u_vav_cx", "v_vav_cy", "u_surf_cx", "v_surf_cy"]
STEP_OUT = ["Hi_a", "u_vav_cx", "v_vav_cy", "Ti_a"]


def _points(geometry, dx):
    return tuple(1 + 2 * int(math.floor(h / dx + 1e-9)) for h in HALF[geometry])


def listed():
    return [
        # the smallest grid of the benchmark configurations (129 x 17) at the reference's default step-norm
        # tolerance: hundreds of kernels that take microseconds each, as in a calibration over many channel runs
        dict(name="solve_channel", kind="solve", geometry="channel", dx=5e3, stop="default", precision="fp64",
             anderson=0, margin="infinite_slab", friction=2.0),
        # a calving front with the stress boundary rows to the nonlinear residual, at the finer channel spacing
        dict(name="solve_front", kind="solve", geometry="channel", dx=2.5e3, stop="relres", precision="fp64",
             anderson=0, margin="BC", friction=1.0),
        # a coarse continental run at the reference's default step-norm tolerance, odd sizes
        dict(name="solve_cap_18km", kind="solve", geometry="icecap", dx=18e3, stop="default", precision="fp64",
             anderson=0, margin="infinite_slab", friction=4.0),
        # the benchmark's ice cap (321 x 561 x 15) in plain FP64 with the reference's relaxed iteration
        dict(name="solve_cap_5km", kind="solve", geometry="icecap", dx=5e3, stop="relres", precision="fp64",
             anderson=0, margin="infinite_slab", friction=4.0),
        # the same size in mixed precision under the configuration's step norm and linear tolerance: the
        # linear solves dominate
        dict(name="solve_cap_5km_mixed", kind="solve", geometry="icecap", dx=5e3, stop="norm", precision="mixed",
             anderson=0, margin="infinite_slab", friction=4.0),
        # end to end from host buffers and a velocity guess, with Anderson mixing, as after a learned prediction
        dict(name="restart_cap_5km", kind="restart", geometry="icecap", dx=5e3, stop="relres", precision="fp64",
             anderson=3, margin="infinite_slab", friction=4.0),
        # the largest grid (1501 x 1501 x 15): a continental sheet at 4 km, where memory bandwidth counts
        dict(name="solve_sheet_4km", kind="solve", geometry="sheet", dx=4e3, stop="norm", precision="fp64",
             anderson=0, margin="infinite_slab", friction=4.0),
        # a calibration ensemble: channels of two spacings with a front, and ice caps, all loops in one graph
        dict(name="ensemble_8", kind="ensemble", channels=5, caps=3, cap_dx=20e3, precision="fp64", anderson=3),
        # the model's time step: predictor, warm-started solve, corrector, heat equation, thickness update
        dict(name="step_cap_10km", kind="step", geometry="icecap", dx=10e3, steps=2, integration="explicit",
             friction=4.0),
        # shallow-ice velocities of a large sheet, the cheapest dynamics a long run uses
        dict(name="sia_sheet_6km", kind="sia", geometry="sheet", dx=6e3),
        # inference of the warm-start network for one ice cap, as before each solve
        dict(name="net_predict", kind="net", train=False, ny=561, nx=321, batch=1),
        # one training step at the default minibatch
        dict(name="net_train", kind="net", train=True, ny=561, nx=321, batch=8),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "restart", "ensemble", "step", "sia", "net", "net"])
    if kind == "solve":
        geometry = rng.choice(["channel", "icecap", "icecap", "sheet"])
        c = dict(kind="solve", geometry=geometry, precision="fp64", anderson=0, margin="infinite_slab",
                 friction=2.0 if geometry == "channel" else 4.0)
        if geometry == "channel":
            c.update(dx=round(_log(rng, 2.4e3, 8e3), 1), stop="default")
            if rng.random() < 0.6:   # the front's ragged cells want the finer channels
                c.update(dx=min(c["dx"], 5e3), margin="BC", stop="relres", friction=1.0)
        elif geometry == "icecap":
            c.update(dx=round(_log(rng, 5e3, 40e3), 1), stop=rng.choice(["norm", "relres", "default"]))
            if c["stop"] == "relres":
                c.update(anderson=rng.choice([0, 3]))
            elif c["stop"] == "norm":
                c.update(precision=rng.choice(["fp64", "mixed"]))
        else:
            c.update(dx=round(_log(rng, 4.5e3, 25e3), 1), stop=rng.choice(["norm", "relres"]))
        return c
    if kind == "restart":
        return dict(kind="restart", geometry="icecap", dx=round(_log(rng, 5e3, 25e3), 1), stop="relres",
                    precision="fp64", anderson=3, margin="infinite_slab", friction=4.0)
    if kind == "ensemble":
        return dict(kind="ensemble", channels=rng.randint(1, 6), caps=rng.randint(1, 3),
                    cap_dx=round(_log(rng, 14e3, 40e3), 1), precision="fp64", anderson=3)
    if kind == "step":
        return dict(kind="step", geometry="icecap", dx=round(_log(rng, 7e3, 30e3), 1), steps=rng.randint(1, 3),
                    integration=rng.choice(["explicit", "semi-implicit"]), friction=4.0)
    if kind == "sia":
        geometry = rng.choice(["icecap", "sheet"])
        return dict(kind="sia", geometry=geometry, dx=round(_log(rng, 5e3, 30e3), 1))
    ny, nx = (int(round(_log(rng, 30, 561))) for _ in range(2))
    return dict(kind="net", train=rng.random() < 0.6, ny=ny, nx=min(nx, 400), batch=rng.randint(1, 8))


# ---- inputs -------------------------------------------------------------------------------------------------
def _fields(case, seed):
    """The geometry of a case: its grid, the configuration and the host fields."""
    kw = dict(calving_front=True) if case.get("margin") == "BC" else {}
    g, cfg, f = GEOMETRY[case["geometry"]](seed=seed, dx=case["dx"], **kw)
    f = dict(f)
    f["beta_sq_a"] = np.asfortranarray(f["beta_sq_a"] * case.get("friction", 1.0))
    ny, nx = f["Hi_a"].shape
    if case["geometry"] != "channel":
        f["SL_a"] = np.full((ny, nx), -600.0, order="F")
    elif case.get("margin") != "BC":
        f["Hi_a"] = np.maximum(f["Hi_a"], 50.0)
    return g, cfg, f


def _settings(case):
    """The solver settings of a case, as the benchmark and the integration notes give them."""
    s = dict(precision=case.get("precision", "fp64"))
    if case.get("margin") == "BC":
        s["choice_ice_margin"] = "BC"
    if case.get("stop") == "default":   # the reference's own tolerances, its linear solves ten times tighter
        s.update(DIVA_visc_it_norm_dUV_tol=1e-2, DIVA_visc_it_nit=50, lin_rtol=1e-3)
    elif case.get("stop") == "relres":
        m = case.get("anderson", 0)
        s.update(picard_stop="relres", picard_relres_tol=1e-6, DIVA_visc_it_nit=500, lin_adaptive=1, lin_rtol=1e-10,
                 picard_anderson_m=m, lin_adaptive_eta=0.1 if m else 0.5, picard_stall_its=30)
    return s


def _data_model(ctx):
    ctx.update_general_ice_model_data()
    ctx.calc_pressure_melting_point()
    ctx.calc_ice_rheology()
    ctx.update_general_ice_model_data()


def _context(g, cfg, f):
    ctx = diva.Context(diva.Grid(**g), cfg)
    ctx.upload(f)
    _data_model(ctx)
    return ctx


def _pinned(a):
    """A pinned, Fortran-ordered host copy of an array; the tensor keeps the memory alive."""
    a = np.asarray(a)
    t = torch.empty(a.shape[::-1], dtype=torch.float64 if a.dtype == np.float64 else torch.int32, pin_memory=True)
    h = t.numpy().T
    h[...] = a
    return h, t


def _out(ctx, names):
    keep, out = [], {}
    for n in names:
        out[n], t = _pinned(ctx.empty(n))
        keep.append(t)
    return out, keep


def prepare(case, seed):
    return {"solve": _prepare_solve, "restart": _prepare_restart, "ensemble": _prepare_ensemble,
            "step": _prepare_step, "sia": _prepare_sia, "net": _prepare_net}[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_solve(case, seed):
    g, cfg, f = _fields(case, seed)
    ctx = _context(g, dict(cfg, **_settings(case)), f)
    ctx.state_save()
    out, keep = _out(ctx, VELOCITIES)
    return dict(run=_run_solve, ctx=ctx, out=out, keep=keep)


def _run_solve(s):
    s["ctx"].state_restore()
    s["ctx"].solve_DIVA()
    return s["ctx"].download(VELOCITIES, out=s["out"])


def _prepare_restart(case, seed):
    g, cfg, f = _fields(case, seed)
    # the guess: a loosely converged solution of the same geometry with a smooth 10 % error
    ctx = _context(g, dict(cfg, DIVA_visc_it_norm_dUV_tol=3e-2, lin_rtol=1e-6), f)
    ctx.solve_DIVA()
    guess = ctx.download(["u_vav_cx", "v_vav_cy"])
    rng = np.random.default_rng(seed + 2)
    for n, a in guess.items():
        p = rng.uniform(0, 2 * np.pi, 2)
        yy, xx = np.meshgrid(np.linspace(0, 1, a.shape[0]), np.linspace(0, 1, a.shape[1]), indexing="ij")
        guess[n] = np.asfortranarray(a * (1.0 + 0.1 * np.sin(9 * xx + p[0]) * np.cos(7 * yy + p[1])))
    ctx.set_config(dict(cfg, **_settings(case)))
    keep, inputs = [], {}
    for n in INPUTS:
        inputs[n], t = _pinned(f[n])
        keep.append(t)
    for n in ("taub_cx", "taub_cy", "visc_eff_3D_a"):   # no viscosity yet: the completion forms it
        inputs[n], t = _pinned(ctx.empty(n))
        keep.append(t)
    for n, a in guess.items():
        inputs[n], t = _pinned(a)
        keep.append(t)
    out, more = _out(ctx, RESTART_OUT)
    return dict(run=_run_restart, ctx=ctx, inputs=inputs, out=out, keep=keep + more)


def _run_restart(s):
    ctx = s["ctx"]
    ctx.upload(s["inputs"])
    _data_model(ctx)
    ctx.complete_state(10)
    ctx.solve_DIVA()
    ctx.calc_sia_3d_velocities()
    return ctx.download(RESTART_OUT, out=s["out"])


def _prepare_ensemble(case, seed):
    rng = np.random.default_rng(seed)
    ctxs = []
    for k in range(case["channels"] + case["caps"]):
        cap = k >= case["channels"]
        c = dict(geometry="icecap" if cap else "channel", dx=case["cap_dx"] if cap else (5e3, 4e3)[k % 2],
                 stop="relres", precision=case["precision"], anderson=case["anderson"],
                 margin="infinite_slab" if cap else "BC",
                 friction=float(np.exp(rng.uniform(np.log(4.0), np.log(8.0)))) if cap else 1.0)
        g, cfg, f = _fields(c, seed + 1 + k)
        fa = float(np.exp(rng.uniform(np.log(0.5), np.log(1.0))))
        ctx = _context(g, dict(cfg, m_enh_sheet=fa, m_enh_shelf=fa, **_settings(c)), f)
        ctx.state_save()
        ctxs.append(ctx)
    outs = [_out(c, ["u_vav_cx", "v_vav_cy"]) for c in ctxs]
    return dict(run=_run_ensemble, batch=diva.Batch(ctxs), ctxs=ctxs, outs=[o for o, _ in outs],
                keep=[k for _, k in outs])


def _run_ensemble(s):
    for c in s["ctxs"]:
        c.state_restore()
    s["batch"].solve_DIVA()
    return [c.download(["u_vav_cx", "v_vav_cy"], out=o) for c, o in zip(s["ctxs"], s["outs"])]


def _prepare_step(case, seed):
    g, cfg, f = _fields(case, seed)
    ny, nx = f["Hi_a"].shape
    f["SMB_a"] = np.asfortranarray(np.full((ny, nx), 0.2))
    f["T_surf_annual_a"] = np.asfortranarray(np.asarray(f["Ti_a"])[0])
    f["GHF_a"] = np.asfortranarray(np.full((ny, nx), 1.7e6))
    cfg = dict(cfg, **_settings(dict(case, stop="relres")), dt_thermo=0.02,
               choice_ice_integration_method=case["integration"])
    ctx = _context(g, cfg, f)
    ctx.upload({"mask_ice_a_prev": ctx.download(["mask_ice_a"])["mask_ice_a"]})
    ctx.determine_floating_margin_fraction()
    pc = dynamics.PCTimeStepper(ctx, 0.0, 1e5, thermo=True)
    pc.step()
    pc.step()
    ctx.state_save()
    out, keep = _out(ctx, STEP_OUT)
    return dict(run=_run_step, ctx=ctx, pc=pc, steps=case["steps"], out=out, keep=keep)


def _run_step(s):
    s["ctx"].state_restore()
    pc = copy.copy(s["pc"])
    pc.reports = []
    for _ in range(s["steps"]):
        pc.step()
    return s["ctx"].download(STEP_OUT, out=s["out"])


def _prepare_sia(case, seed):
    g, cfg, f = _fields(case, seed)
    ctx = _context(g, dict(cfg, choice_ice_dynamics="SIA"), f)
    Hi, t = _pinned(f["Hi_a"])
    out, keep = _out(ctx, SIA_OUT)
    return dict(run=_run_sia, ctx=ctx, Hi=Hi, out=out, keep=keep + [t])


def _run_sia(s):
    ctx = s["ctx"]
    ctx.upload({"Hi_a": s["Hi"]})
    _data_model(ctx)
    ctx.solve_SIA()
    return ctx.download(SIA_OUT, out=s["out"])


def _net_tensors(case, seed):
    """Features and targets of one minibatch: smooth fields of the inputs' and the state's magnitudes."""
    n, ny, nx = case["batch"], case["ny"], case["nx"]
    Hp, Wp = (ny + 3) // 4 * 4, (nx + 3) // 4 * 4
    gen = torch.Generator(device="cuda").manual_seed(seed)
    coarse = torch.randn(n, learned.IN_C + learned.N_OUT, max(2, Hp // 8), max(2, Wp // 8), generator=gen,
                         device="cuda")
    x = torch.nn.functional.interpolate(coarse, size=(Hp, Wp), mode="bilinear", align_corners=False)
    x = x.permute(0, 2, 3, 1)
    feat = x[..., :learned.IN_C].clone()
    feat[..., 8:] = 0.0
    feat[:, ny:] = 0.0
    feat[:, :, nx:] = 0.0
    return feat.to(torch.bfloat16).contiguous(), x[..., learned.IN_C:].contiguous()


def _prepare_net(case, seed):
    net = learned.WarmStartNet(diva.Grid(case["nx"], case["ny"], 5e3), batch=case["batch"], capacity=0, seed=seed)
    feat, tgt = _net_tensors(case, seed)
    s = dict(net=net, feat=feat, n=case["batch"])
    if case["train"]:
        return dict(s, run=_run_train, tgt=tgt)
    return dict(s, run=_run_forward, out=torch.empty(tgt.shape, device="cuda"))


def _run_forward(s):
    s["net"].forward(s["feat"].data_ptr(), s["out"].data_ptr(), s["n"])
    return s["out"]


def _run_train(s):
    loss = s["net"].train_step(s["feat"].data_ptr(), s["tgt"].data_ptr(), s["n"], 1e-4)
    return dict(loss=loss, grads=s["net"].grads(), weights=s["net"].get_weights())


# ---- the work a pass cannot do without ----------------------------------------------------------------------
def _bytes(names, nx, ny):
    three = {"Ti_a", "u_3D_cx", "v_3D_cy", "visc_eff_3D_a"}
    return sum(8.0 * nx * ny * (NZ if n in three else 1) for n in names)


def work(case):
    if case["kind"] == "net":
        n, Hp, Wp = case["batch"], (case["ny"] + 3) // 4 * 4, (case["nx"] + 3) // 4 * 4
        lvl = {"e1a": 0, "e1b": 0, "e2a": 1, "e2b": 1, "ba": 2, "bb": 2, "d2a": 1, "d2b": 1, "d1a": 0, "d1b": 0}
        flops = sum(2.0 * 9 * ci * co * n * (Hp >> lvl[k]) * (Wp >> lvl[k]) for k, ci, co in learned.LAYERS)
        flops += 2.0 * learned.HEAD_C * learned.N_OUT * n * Hp * Wp
        weights = 4.0 * learned.weight_layout()[1]
        size = n * Hp * Wp * (2.0 * learned.IN_C + 4.0 * learned.N_OUT)
        return dict(bytes=size + (6 if case["train"] else 1) * weights, flops=flops * (3 if case["train"] else 1))
    if case["kind"] == "ensemble":
        members = [("channel", (5e3, 4e3)[k % 2]) for k in range(case["channels"])]
        members += [("icecap", case["cap_dx"])] * case["caps"]
    else:
        members = [(case["geometry"], case["dx"])]
    total = flops = 0.0
    for geometry, dx in members:
        nx, ny = _points(geometry, dx)
        if case["kind"] == "sia":
            total += _bytes(INPUTS + SIA_OUT, nx, ny)
            flops += 60.0 * NZ * nx * ny
        elif case["kind"] == "step":
            total += case["steps"] * _bytes(INPUTS + STEP_OUT, nx, ny)
            flops += case["steps"] * 2000.0 * NZ * nx * ny
        else:
            # the inputs read and the velocities written once; of the arithmetic, one evaluation of the
            # coefficients and one of the operator for each of the 20 iterations that no solve does without
            total += _bytes(INPUTS + (RESTART_OUT if case["kind"] == "restart" else VELOCITIES), nx, ny)
            flops += 20.0 * (60.0 * NZ + 60.0) * nx * ny
    return dict(bytes=total, flops=flops)


# ---- the same in 64 bits ------------------------------------------------------------------------------------
def exact(case, seed):
    """The network's and the shallow-ice velocities' values.  The other kinds return the iterate at which a stop
    test ended a nonlinear iteration: no formula gives it, and the converged state differs from it by far more
    than 64-bit arithmetic does."""
    if case["kind"] == "net":
        return _exact_net(case, seed)
    if case["kind"] == "sia":
        return _exact_sia(case, seed)
    return None


def _initial_weights(seed, total, layers):
    """The network's initial weights: He-normal by Box-Muller from a splitmix64 stream, zero biases."""
    s, mask = seed & (2 ** 64 - 1), 2 ** 64 - 1
    count = sum(9 * ci * co for _, ci, co in layers) + learned.N_OUT * learned.HEAD_C
    st = (np.uint64(s) + np.uint64(0x9E3779B97F4A7C15) * np.arange(1, 2 * count + 1, dtype=np.uint64)) & np.uint64(mask)
    z = (st ^ (st >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    z = z ^ (z >> np.uint64(31))
    u = ((z >> np.uint64(11)).astype(np.float64) + 0.5) / 9007199254740992.0
    normal = np.sqrt(-2.0 * np.log(u[0::2])) * np.cos(2.0 * np.pi * u[1::2])
    w, at, off = np.zeros(total, np.float32), 0, 0
    for _, ci, co in layers:
        m = 9 * ci * co
        w[off:off + m] = math.sqrt(2.0 / (9.0 * ci)) * normal[at:at + m]
        at, off = at + m, off + m + co
    m = learned.N_OUT * learned.HEAD_C
    w[off:off + m] = math.sqrt(1.0 / learned.HEAD_C) * normal[at:at + m]
    return w


def _exact_net(case, seed):
    F = torch.nn.functional
    layout, total = learned.weight_layout()
    w0 = torch.as_tensor(_initial_weights(seed, total, learned.LAYERS), device="cuda").double()
    w = w0.clone().requires_grad_(case["train"])
    feat, tgt = _net_tensors(case, seed)

    def part(name):
        wo, shape, bo, nb = layout[name]
        t = w[wo:wo + int(np.prod(shape))].reshape(shape)
        if name != "head":
            t = t.permute(1, 2, 0).reshape(shape[1], shape[2], 3, 3)
        return t, w[bo:bo + nb]

    def conv(name, t):
        k, b = part(name)
        return F.relu(F.conv2d(t, k, b, padding=1))

    def up(t):
        return F.interpolate(t, scale_factor=2, mode="nearest")

    with torch.set_grad_enabled(case["train"]):
        e1 = conv("e1b", conv("e1a", feat.double().permute(0, 3, 1, 2)))
        e2 = conv("e2b", conv("e2a", F.avg_pool2d(e1, 2)))
        b = conv("bb", conv("ba", F.avg_pool2d(e2, 2)))
        d2 = conv("d2b", conv("d2a", torch.cat([up(b), e2], 1)))
        d1 = conv("d1b", conv("d1a", torch.cat([up(d2), e1], 1)))
        wh, bh = part("head")
        out = torch.einsum("oc,nchw->nhwo", wh, d1) + bh
    if not case["train"]:
        return out
    ny, nx = case["ny"], case["nx"]
    valid = torch.zeros(out.shape[1:], dtype=torch.float64, device="cuda")
    valid[:ny, :nx - 1, 0] = valid[:ny, :nx - 1, 2] = 1.0
    valid[:ny - 1, :nx, 1] = valid[:ny - 1, :nx, 3] = 1.0
    valid[:ny, :nx, 4:4 + NZ] = 1.0
    e = (out - tgt.double()) * valid
    loss = (e * e).sum() / (valid.sum() * out.shape[0])
    loss.backward()
    g = w.grad
    # Adam's first step (beta1 0.9, beta2 0.999, eps 1e-8): the bias-corrected moments are g and g^2
    w1 = w0 - 1e-4 * g / (g.abs() + 1e-8)
    return dict(loss=float(loss), grads=g.cpu().numpy(), weights=w1.cpu().numpy())


def _exact_sia(case, seed):
    """Glen's-law shallow-ice velocities on the cx and cy faces: vertical averages and surface values."""
    g, _, f = _fields(case, seed)
    rho, rho_sw, grav, R = 910.0, 1028.0, 9.81, 8.314
    dx = g["dx"]
    z = torch.as_tensor(np.asarray(g["zeta"]), device="cuda")
    H, b, SL, T = (torch.as_tensor(np.ascontiguousarray(f[n]), device="cuda") for n in ("Hi_a", "Hb_a", "SL_a", "Ti_a"))
    Hs = H + torch.maximum(SL - rho / rho_sw * H, b)
    ice = H > 0
    floating = (H < (SL - b) * rho_sw / rho).double()[None, None]
    ocean = floating.clone()
    ocean[..., 1:-1, 1:-1] = 0.0
    while True:   # the ocean: floating cells 8-connected to one at the domain's edge
        grown = torch.nn.functional.max_pool2d(ocean, 3, stride=1, padding=1) * floating
        if torch.equal(grown, ocean):
            break
        ocean = grown
    sheet = ice & (ocean[0, 0] == 0)
    T = torch.where(ice, T, torch.full_like(T, 263.15 - 1e-9))
    A = torch.where(T < 263.15, 1.14e-5 * torch.exp(-6.0e4 / (R * T)), 5.47e10 * torch.exp(-13.9e4 / (R * T)))
    A = torch.where(ice, A, torch.full_like(A, 1.14e-5 * math.exp(-6.0e4 / (R * 263.15))))

    def faces(H, Hs, A, sheet):
        """The velocities on the faces between neighbours along the last axis."""
        Hc, Ac = 0.5 * (H[:, :-1] + H[:, 1:]), 0.5 * (A[:, :, :-1] + A[:, :, 1:])
        along = (Hs[:, 1:] - Hs[:, :-1]) / dx
        s = Hs[:, :-1] + Hs[:, 1:]
        across = torch.empty_like(along)
        across[1:-1] = (s[2:] - s[:-2]) / (4 * dx)
        across[0], across[-1] = (s[1] - s[0]) / (2 * dx), (s[-1] - s[-2]) / (2 * dx)
        D0 = (rho * grav * Hc) ** 3 * (along ** 2 + across ** 2)
        q = Ac * (z ** 3)[:, None, None]
        piece = 0.5 * (q[1:] + q[:-1]) * (z[1:] - z[:-1])[:, None, None]
        u = torch.zeros_like(Ac)
        u[:-1] = -torch.flip(torch.cumsum(torch.flip(piece, [0]), 0), [0])
        u = torch.clamp(D0 * 2.0 * Hc * u, min=-1e5) * along
        u = torch.where(sheet[:, :-1] | sheet[:, 1:], u, torch.zeros_like(u))
        mean = (0.5 * (u[1:] + u[:-1]) * (z[1:] - z[:-1])[:, None, None]).sum(0)
        return mean.cpu().numpy(), u[0].cpu().numpy()

    uv, us = faces(H, Hs, A, sheet)
    vv, vs = faces(H.T, Hs.T, A.transpose(1, 2), sheet.T)
    return dict(u_vav_cx=uv, v_vav_cy=vv.T, u_surf_cx=us, v_surf_cy=vs.T)
