"""Performance cases: the work that users of the framework have it do.

Each case is one pass through the public entry points (``phd_gb300.izem``,
``phd_gb300.surrogate``) as a driver program makes it: the state goes from
pinned host memory to the device, the block is advanced, the state comes
back.  Sizes are those of the repository's workloads (``phd_gb300.ics``), of
its tests, or ragged ones between them.

Kinds of case:

``sod``       2-D O2/N2 shock tube, WENO7 (the reference's own test case): the
              smallest block in use, bound by latency and launches.
``tgv``       Taylor-Green vortex, fitted transport, WENO5.
``mix``       temporal H2/air mixing layer, 9 species: time step, RK3 and (with
              chem) the Strang chemistry half steps, by BDF or learned.
``jet``       planar H2/air jet with the jet faces and the LES closure.
``euler``     the three convective sweeps alone on a perturbed layer some of
              whose faces take the nonlinear weights.
``reactors``  independent reactors of a mixing layer's window (the labelling
              of a surrogate's training set), in host or in device arrays.
``forward``, ``train``  the surrogate network: inference, and one epoch of
              its training.

The chemistry cases hold gas in its induction phase (the mixing layer's and
the jet's window), where the integrator's answer is determined to rounding.
Burning and burnt gas is left out on purpose: there an adaptive integrator
with RTOL = 1e-6 amplifies a last-bit change of the rate expressions by ten
orders of magnitude (the table-walking and the generated right-hand side,
equal expressions that the compiler contracts differently, differ by up to
2e-4 of T over the batched-reactor distribution), so two correct builds can
be compared within the integrator's tolerance only, which the tests do.
"""
import math

import numpy as np
import torch

from phd_gb300 import ics, izem, surrogate
from phd_gb300.capi import (BC_EXTRAPOLATION, BC_INFLOWJET, BC_NSCBC_OUT, BC_PERIODIC, IzemJet)
from phd_gb300.mech import h2_mechanism
from phd_gb300.thd import adi_struct, constants, eglib_link, load_species, thd_init

F64 = torch.float64
DX = (12e-3 / 256, 12e-3 / 255, 6e-3 / 128)   # the 256 x 256 x 128 mixing layer's spacing


def listed():
    return [
        # the reference's Sod run: a small 2-D block, WENO7, many short steps
        {"name": "sod_400x11", "kind": "sod", "nx": 400, "ny": 11, "ng": 4, "steps": 20},
        # the plain-method configuration: 64^3, 20 steps
        {"name": "tgv_64", "kind": "tgv", "nx": 64, "ny": 64, "nz": 64, "steps": 20},
        # a ragged block of the same flow with the Fourier time-step criteria
        {"name": "tgv_90x73x41", "kind": "tgv", "nx": 90, "ny": 73, "nz": 41, "steps": 4, "vis_dt": True},
        # a small ragged reacting block, EGLIB, BDF chemistry: one rank's block of a decomposed run
        {"name": "mix_33x40x21", "kind": "mix", "nx": 33, "ny": 40, "nz": 21, "steps": 2, "eglib": True, "chem": "bdf"},
        # the reacting DNS configuration at its full size, one driver step
        {"name": "mix_256x256x128", "kind": "mix", "nx": 256, "ny": 256, "nz": 128, "steps": 1, "eglib": True,
         "chem": "bdf"},
        # the same layer with the learned chemistry and BDF fallback, on a ragged block
        {"name": "mix_learned_144x130x66", "kind": "mix", "nx": 144, "ny": 130, "nz": 66, "steps": 1, "eglib": True,
         "chem": "mlp"},
        # the reacting LES jet: jet faces, Smagorinsky closure, BDF chemistry
        {"name": "jet_les_160x128x64", "kind": "jet", "nx": 160, "ny": 128, "nz": 64, "steps": 1},
        # the convective sweeps alone, linear and nonlinear faces
        {"name": "euler_61x50x38", "kind": "euler", "nx": 61, "ny": 50, "nz": 38},
        # reactors of one small window, host arrays in and out
        {"name": "reactors_500", "kind": "reactors", "n": 500, "device": False},
        # a training set's labels, device arrays
        {"name": "reactors_262144", "kind": "reactors", "n": 262144, "device": True},
        # surrogate inference on host rows
        {"name": "forward_100003", "kind": "forward", "n": 100003},
        # one training epoch
        {"name": "train_65536", "kind": "train", "n": 65536, "batch": 4096},
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sod", "tgv", "mix", "mix", "mix", "jet", "euler", "reactors", "forward", "train"])
    if kind == "sod":
        return {"kind": kind, "nx": _between(rng, 40, 1200), "ny": rng.randint(9, 24), "ng": rng.choice([3, 4]),
                "steps": rng.randint(2, 24)}
    if kind == "tgv":
        return {"kind": kind, "nx": _between(rng, 12, 130), "ny": _between(rng, 12, 130), "nz": _between(rng, 12, 130),
                "steps": rng.randint(1, 6), "vis_dt": rng.random() < 0.3}
    if kind == "mix":
        chem = rng.choice(["", "bdf", "bdf", "skip", "mlp"])
        c = {"kind": kind, "nx": _between(rng, 16, 200), "ny": _between(rng, 16, 200), "nz": _between(rng, 16, 100),
             "steps": 1 if chem else rng.randint(1, 3), "eglib": rng.random() < 0.7, "chem": chem}
        opt = rng.choice(["", "", "les", "vis_dt", "ducros", "weno7"])
        if opt:
            c[opt] = True
        return c
    if kind == "jet":
        return {"kind": kind, "nx": _between(rng, 24, 200), "ny": _between(rng, 24, 160), "nz": _between(rng, 16, 80),
                "steps": 1}
    if kind == "euler":
        return {"kind": kind, "nx": _between(rng, 12, 90), "ny": _between(rng, 12, 90), "nz": _between(rng, 12, 60)}
    if kind == "reactors":
        return {"kind": kind, "n": _between(rng, 1, 400000), "device": rng.random() < 0.5}
    if kind == "forward":
        return {"kind": kind, "n": _between(rng, 1, 300000)}
    return {"kind": kind, "n": _between(rng, 5000, 150000), "batch": rng.choice([256, 1000, 4096])}


# ------------------------------------------------------------------- states
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _pinned(shape, dtype):
    """A pinned Fortran-ordered numpy array of the given shape."""
    return torch.empty(tuple(reversed(shape)), dtype=dtype, pin_memory=True).numpy().transpose()


def _buffers(cfg):
    g = (cfg.nx + 2 * cfg.ng, cfg.ny + 2 * cfg.ng, cfg.nz + 2 * cfg.ng)
    b = {k: _pinned(g, F64) for k in ("T", "W_i", "cp")}
    b["v"] = _pinned(g + (5 + cfg.nrv,), F64)
    b["ha"] = _pinned(g + (cfg.nrv,), F64)
    b["shock_sensor"] = _pinned(g, torch.uint8)
    return b


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device="cuda")


def _fill(buf, cfg, thd, a, rho, u, T, Y):
    """Writes the raw ghosted state of dimensional primitives into buf.
    rho, u[0..2], T and Y[k] are device tensors that broadcast to the
    interior (nz, ny, nx); ghosts by zero-gradient extension."""
    shp = (cfg.nz, cfg.ny, cfg.nx)
    idx = [torch.clamp(torch.arange(n + 2 * cfg.ng, device="cuda") - cfg.ng, 0, n - 1)
           for n in (cfg.nx, cfg.ny, cfg.nz)]
    Wc_i = [thd.Wc_i[k] for k in range(cfg.nrv)]
    rho = rho / a["rho_ref"]
    W_i = sum(Y[k] * Wc_i[k] for k in range(cfg.nrv))
    T = T / a["t_ref"]
    P = rho * T * W_i
    u = [x / a["u_ref"] for x in u]
    # species enthalpies at the (few) distinct temperatures of the state
    h = _dev(ics.ha_code(thd, T.cpu().numpy()))
    hm = sum(h[..., k] * Y[k] for k in range(cfg.nrv))
    cons = [rho, rho * u[0], rho * u[1], rho * u[2],
            rho * hm - P + 0.5 * rho * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])] + [rho * Y[k] for k in range(cfg.nrv)]

    def put(dst, x):
        x = x.expand(shp)[idx[2]][:, idx[1]][:, :, idx[0]]
        torch.from_numpy(dst.transpose()).copy_(x)

    for q, x in enumerate(cons):
        put(buf["v"][..., q], x)
    put(buf["T"], T)
    for k in ("W_i", "cp", "ha", "shock_sensor"):
        buf[k][...] = 0


def _block(case, seed):
    """cfg, species data, scales, metrics and the raw initial state."""
    a = constants()
    kind = case["kind"]
    ng = case.get("ng", 4 if case.get("weno7") else 3)
    gen = _gen(seed)
    nx, ny, nz = case["nx"], case["ny"], case.get("nz", 1)
    sp = load_species({"sod": "o2n2", "tgv": "air2"}.get(kind, "h2air9"))
    thd = thd_init(sp, a)
    nrv, names = thd.nspc, sp["names"]
    W = np.array(sp["W_gmol"][:nrv]) * 1e-3
    ex = {"jet": None, "lx": 0.0, "coords": None}
    per = (BC_PERIODIC,) * 6
    zero = torch.zeros((1, 1, 1), dtype=F64, device="cuda")

    def normal():
        return torch.randn((nz, ny, nx), generator=gen, dtype=F64, device="cuda")

    if kind == "tgv":
        T0, p0 = 300.0, 101325.0
        Rm = a["r_ref"] / W[0]
        U0 = 0.1 * math.sqrt(1.4 * Rm * T0)
        rho0 = p0 / (Rm * T0)
        ce = sp["cofeta"][0]
        L0 = 1600.0 * math.exp(ce[0] + ce[1] * math.log(T0)) * 0.1 / (rho0 * U0)
        xs = [np.arange(n) * (2.0 * math.pi * L0 / n) for n in (nx, ny, nz)]
        ph = 2.0 * math.pi * torch.rand(3, generator=gen, dtype=F64, device="cuda")   # the vortex's seeded offset
        X = _dev(xs[0] / L0)[None, None, :] + ph[0]
        Yc = _dev(xs[1] / L0)[None, :, None] + ph[1]
        Z = _dev(xs[2] / L0)[:, None, None] + ph[2]
        u = [U0 * torch.sin(X) * torch.cos(Yc) * torch.cos(Z), -U0 * torch.cos(X) * torch.sin(Yc) * torch.cos(Z), zero]
        p = p0 + rho0 * U0 * U0 / 16.0 * (torch.cos(2 * X) + torch.cos(2 * Yc)) * (torch.cos(2 * Z) + 2.0)
        Y = [zero + 0.5, zero + 0.5]
        cfg = ics.make_cfg(nx, ny, nz, nrv, bc=per, vis_dt=int(case.get("vis_dt", False)))
        state = (p / (Rm * T0), u, zero + T0, Y)
    elif kind == "sod":
        xs = [np.linspace(0.0, 1.0, nx), np.arange(ny) * (1.0 / (nx - 1)), np.zeros(1)]
        left = _dev(xs[0] < 0.5)[None, None, :]
        X = np.array([0.233, 0.767])
        Yk = X * W / (X * W).sum()
        wi = (Yk / W).sum()
        amp = 1.0 + 0.02 * torch.rand(1, generator=gen, dtype=F64, device="cuda")   # seeded driver pressure
        p = 101325.0 * (left * amp + (1.0 - left) * 0.1)
        T = 300.0 * (left + (1.0 - left) * 0.8)
        Y = [zero + Yk[0], zero + Yk[1]]
        # no z neighbours in 2-D: z ghosts from the plane itself
        cfg = ics.make_cfg(nx, ny, 1, nrv, bc=(BC_EXTRAPOLATION,) * 2 + (BC_PERIODIC,) * 2 + (BC_EXTRAPOLATION,) * 2)
        cfg.ndim = 2
        state = (p / (a["r_ref"] * wi * T), [zero, zero, zero], T, Y)
    elif kind == "jet":
        dx, width, u_jet, u_co, T_jet, T_co, yf, turb = 47e-6, 2e-3, 300.0, 10.0, 1000.0, 1200.0, 0.5, 0.02
        xs = [np.arange(nx) * dx, (np.arange(ny) - 0.5 * (ny - 1)) * dx, np.arange(nz) * dx]
        th = torch.tanh((_dev(xs[1]).abs() - 0.5 * width) / (0.04 * width))[None, :, None]
        Yd = {"H2": 0.5 * (yf - yf * th), "O2": 0.5 * (0.233 + 0.233 * th),
              "N2": 0.5 * ((1.0 - yf + 0.767) - (1.0 - yf - 0.767) * th)}
        Y = [Yd.get(nm, zero) for nm in names]
        T = 0.5 * ((T_jet + T_co) - (T_jet - T_co) * th)
        amp = turb * u_jet * 0.5 * (1.0 - th)
        u = [0.5 * ((u_jet + u_co) - (u_jet - u_co) * th) + amp * (2.0 * torch.rand((nz, ny, nx), generator=gen,
                                                                                   dtype=F64, device="cuda") - 1.0)]
        u += [amp * (2.0 * torch.rand((nz, ny, nx), generator=gen, dtype=F64, device="cuda") - 1.0) for _ in range(2)]
        cfg = ics.make_cfg(nx, ny, nz, nrv, bc=(BC_INFLOWJET, BC_NSCBC_OUT, BC_EXTRAPOLATION, BC_EXTRAPOLATION,
                                                BC_PERIODIC, BC_PERIODIC), eglib=1, reaction=1)
        L = a["l_ref"]
        ex = {"coords": [c / L for c in xs], "lx": (xs[0][-1] - xs[0][0]) / L,
              "jet": IzemJet(width=width, ramp=0.0, T_jet=T_jet, T_co=T_co, p_jet=101325.0, p_co=101325.0, u_jet=u_jet,
                             u_co=u_co, y_fuel=yf, p_far=101325.0, turb=turb, planar=1, reserved=0, seed=int(seed))}
        wi = sum(Y[k] / W[k] for k in range(nrv))
        state = (101325.0 / (a["r_ref"] * wi * T), u, T, Y)
    else:   # the mixing layer
        delta, dU = 0.5e-3, 100.0
        xs = [np.arange(nx) * DX[0], (np.arange(ny) - 0.5 * (ny - 1)) * DX[1], np.arange(nz) * DX[2]]
        t = torch.tanh(_dev(xs[1]) / delta)[None, :, None]
        f = 0.5 * (1.0 + t)
        Yd = {"H2": 0.5 * (1.0 - f), "O2": 0.233 * f, "N2": 0.5 * (1.0 - f) + 0.767 * f}
        Y = [Yd.get(nm, zero) for nm in names]
        T = 1000.0 * (1.0 - f) + 1200.0 * f
        u = [0.5 * dU * t + 0.01 * dU * normal(), 0.01 * dU * normal(), 0.01 * dU * normal()]
        cfg = ics.make_cfg(nx, ny, nz, nrv, bc=(BC_PERIODIC, BC_PERIODIC, BC_EXTRAPOLATION, BC_EXTRAPOLATION,
                                                BC_PERIODIC, BC_PERIODIC),
                           eglib=int(case.get("eglib", False)), reaction=int(bool(case.get("chem"))),
                           vis_dt=int(case.get("vis_dt", False)))
        wi = sum(Y[k] / W[k] for k in range(nrv))
        state = (101325.0 / (a["r_ref"] * wi * T), u, T, Y)
    cfg.ng = ng
    dxi = [ics.grid_dxi(x, ng, a, izem.metrics_dscalar) if len(x) > 2 * ng
           else np.full(len(x) + 2 * ng, a["l_ref"]) for x in xs]
    return cfg, thd, a, dxi, state, ex, names


def _networks(g, mech, dt, seed):
    """Two residual networks for a block's window, normalised on its own
    reactors, and their gate: random weights whose output scale is a hundredth
    of the explicit increments', so that the gate keeps most cells."""
    T, rho, Y, dtp = surrogate.window_reactors(g, dt)
    pick = np.random.Generator(np.random.PCG64(seed)).choice(len(T), size=min(len(T), 1 << 14), replace=False)
    T, rho, Y, dtp = T[pick].copy(), rho[pick].copy(), np.ascontiguousarray(Y[pick]), dtp[pick].copy()
    X = surrogate.features(T, rho, Y, dtp, np.array([mech.wt[k] for k in range(9)]))
    E = surrogate.explicit_increment(mech, T, rho, Y, dtp)
    norm = np.concatenate([X.mean(0), X.std(0) + 1e-6, 0.0 * E.mean(0), 0.01 * E.std(0) + 1e-30]).astype(np.float32)
    nets = []
    for q in range(2):
        s = surrogate.Surrogate(seed=seed + 1000 * (q + 1))
        s.set_residual(True)
        s.set_norm(norm)
        nets.append(s)
    gate = list(surrogate.flow_gate(X, E, 0.05))
    gate[0], gate[1], gate[2], gate[3] = 300.0, 3500.0, 0.5 * float(dtp[0]), 2.0 * float(dtp[0])
    return nets, gate


def _rows(n, seed, width):
    return np.random.Generator(np.random.PCG64(seed)).standard_normal((n, width)).astype(np.float32)


def _window(n, seed):
    """n reactors as a mixing layer's window holds them: unburnt H2/N2 and
    air in all proportions, 1 atm, the layer's time step."""
    rng = np.random.Generator(np.random.PCG64(seed))
    sp = load_species("h2air9")
    W, nm = np.array(sp["W_gmol"]), sp["names"]
    f = 0.5 * (1.0 + np.tanh(rng.uniform(-6.0, 6.0, n)))
    T = (1000.0 * (1.0 - f) + 1200.0 * f) * (1.0 + 0.002 * rng.standard_normal(n))
    Y = np.zeros((n, 9))
    Y[:, nm.index("H2")] = 0.5 * (1.0 - f)
    Y[:, nm.index("O2")] = 0.233 * f
    Y[:, nm.index("N2")] = 0.5 * (1.0 - f) + 0.767 * f
    rho = 101325.0 / (8.314510 * T) / (Y / (W * 1e-3)).sum(1) * 1e-3
    dt = 5e-9 * 10.0 ** rng.uniform(-0.5, 0.5, n)
    return T, rho, Y, dt


# ---------------------------------------------------------------- interface
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("forward", "train"):
        s = surrogate.Surrogate(seed=seed)
        x = _rows(case["n"], seed, 12)
        if kind == "forward":
            return {"kind": kind, "net": s, "x": x}
        t = np.tanh(x[:, :10] * x[:, 2:12]).astype(np.float32)
        return {"kind": kind, "net": s, "x": x, "t": t, "batch": case["batch"]}
    if kind == "reactors":
        arr = _window(case["n"], seed)
        if case["device"]:
            arr = tuple(torch.tensor(x, device="cuda") for x in arr)
        return {"kind": kind, "arr": arr, "mech": h2_mechanism(), "device": case["device"]}
    cfg, thd, a, dxi, raw, ex, names = _block(case, seed)
    g = izem.IzemGPU(cfg, thd, adi_struct(a))
    g.set_grid(*dxi)
    st = {"kind": kind, "g": g, "in": _buffers(cfg), "out": _buffers(cfg), "steps": case.get("steps", 1)}
    if cfg.eglib:
        g.set_eglib(eglib_link(load_species("h2air9")))
    if kind == "jet":
        g.set_coords(*ex["coords"], ex["lx"])
        g.set_jet(ex["jet"])
        g.set_les(mu_sgs_factor=0.17)
    if case.get("les"):
        g.set_les(mu_sgs_factor=0.05)
    if case.get("ducros"):
        g.set_shock_sensor("DUCROS")
    _fill(st["in"], cfg, thd, a, *raw)
    g.upload(**st["in"])
    g.finalize_ic()
    g.download(out=st["in"])
    st["chem"] = case.get("chem", "bdf" if kind == "jet" else "")
    st["mode"] = izem.CHEM_MLP if st["chem"] == "mlp" else izem.CHEM_BDF
    if st["chem"]:
        st["mech"] = h2_mechanism()
        g.set_mechanism(st["mech"])
        if st["chem"] == "skip":
            yf, yo = np.zeros(9), np.zeros(9)
            yf[names.index("H2")] = yf[names.index("N2")] = 0.5
            yo[names.index("O2")], yo[names.index("N2")] = 0.233, 0.767
            g.set_chem_skip(yf, yo, names.index("H2"), names.index("N2"))
        if st["chem"] == "mlp":
            st["nets"], gate = _networks(g, st["mech"], 0.5 * g.timestep()[1], seed)
            g.set_surrogate(st["nets"][0], st["nets"][1], gate)
    if kind == "euler":
        # some faces with the nonlinear weights: flags, and noise for them to see
        gen = _gen(seed + 17)
        shp = tuple(reversed(g.shape))
        flags = (torch.rand(shp, generator=gen, device="cuda") < 0.01).to(torch.uint8)
        noise = 1.0 + 0.02 * torch.randn(shp, generator=gen, dtype=F64, device="cuda")
        torch.from_numpy(st["in"]["shock_sensor"].transpose()).copy_(flags)
        v = torch.from_numpy(st["in"]["v"].transpose())
        v.copy_(v.cuda() * noise)
        g.upload(v=st["in"]["v"], shock_sensor=st["in"]["shock_sensor"])
    return st


def run(state):
    kind = state["kind"]
    if kind == "forward":
        return state["net"].forward(state["x"])
    if kind == "train":
        losses = state["net"].train(state["x"], state["t"], epochs=1, batch=state["batch"])
        W, b = state["net"].get_params()
        return {"losses": losses, "W": W, "b": b}
    if kind == "reactors":
        if state["device"]:
            T, rho, Y, dt = state["arr"]
            T, Y = T.clone(), Y.clone()
            torch.cuda.current_stream().synchronize()   # psr_batch_device's contract: the caller's work is complete
            izem.psr_batch_device(state["mech"], T.numel(), T, rho, Y, dt)
        else:
            T, rho, Y, dt = state["arr"]
            T, Y = T.copy(), Y.copy()
            izem.psr_batch(state["mech"], T, rho, Y, dt)
        return {"T": T, "Y": Y}
    g = state["g"]
    if kind == "euler":
        g.euler_LLF_x()
        g.euler_LLF_y()
        g.euler_LLF_z()
        return g.flux()
    g.upload(**state["in"])
    loop = izem.TimeLoop(g, bool(state["chem"]), chem_mode=state["mode"])
    dts = [loop.step() for _ in range(state["steps"])]
    return {"dt": dts, **g.download(out=state["out"])}


def work(case):
    """Bytes: inputs read once, outputs written once.  Flops: the arithmetic
    of the method per unit (faces, points, reactors, network rows), with a
    transcendental function counted as ten."""
    kind = case["kind"]
    if kind == "forward":
        return {"bytes": case["n"] * 88.0, "flops": case["n"] * 404480.0}
    if kind == "train":
        return {"bytes": case["n"] * 88.0, "flops": case["n"] * 3 * 404480.0}
    if kind == "reactors":
        return {"bytes": case["n"] * 176.0, "flops": case["n"] * 16000.0}
    nrv = {"sod": 2, "tgv": 2}.get(kind, 9)
    ng = case.get("ng", 4 if case.get("weno7") else 3)
    n = case["nx"] * case["ny"] * case.get("nz", 1)
    cells = (case["nx"] + 2 * ng) * (case["ny"] + 2 * ng) * (case.get("nz", 1) + 2 * ng)
    face = 60.0 * (5 + nrv)
    if kind == "euler":
        return {"bytes": cells * 8.0 * (8 + 2 * nrv + 14), "flops": n * 3 * face}
    eg = case.get("eglib") or kind == "jet"
    point = (5500.0 if eg else 900.0 if nrv == 9 else 300.0) + 14.0 * (12 + 3 * nrv)
    stage = face * (2 if kind == "sod" else 3) + point + 60.0 * nrv
    chem = 2 * 16000.0 if case.get("chem", "bdf" if kind == "jet" else "") else 0.0
    return {"bytes": cells * (2.0 * 8 * (8 + 2 * nrv) + 2), "flops": n * case.get("steps", 1) * (3 * stage + chem)}


# --------------------------------------------------------------- 64-bit values
def exact(case, seed):
    if case["kind"] == "euler":
        return _euler_exact(case, seed)
    if case["kind"] == "forward":
        return _forward_exact(case, seed)
    if case["kind"] == "reactors":
        return _reactors_exact(case, seed)
    return None   # whole steps and training


def _forward_exact(case, seed):
    """The network in 64 bits: 12 -> 4 x 256 (GELU, tanh form) -> 10, He
    initialisation from the seed, zero biases."""
    rng = np.random.Generator(np.random.PCG64(seed))
    y = _dev(_rows(case["n"], seed, 12))
    for layer in range(5):
        fan = 12 if layer == 0 else 256
        w = (rng.standard_normal((fan, 10 if layer == 4 else 256)) * np.sqrt(2.0 / fan)).astype(np.float32)
        y = y @ _dev(w)
        if layer < 4:
            y = 0.5 * y * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (y + 0.044715 * y ** 3)))
    return y


def _reactors_exact(case, seed):
    """The constant-volume reactors' solution by the classical fourth-order
    Runge-Kutta method, 100 steps: over these induction times its error is
    far below rounding."""
    m = h2_mechanism()
    T, rho, Y, dt = (_dev(x) for x in _window(case["n"], seed))
    wt = _dev([m.wt[k] for k in range(9)])
    pick = [[m.nuk[i][s] for s in range(6)] for i in range(m.ii)]
    nus = [[m.nu[i][s] for s in range(6)] for i in range(m.ii)]

    def arrhenius(p, T):
        return p[0] * torch.exp(p[1] * torch.log(T) - p[2] / T)

    def rhs(T, Y):
        C = rho[:, None] * Y / wt
        w = torch.zeros_like(C)
        for i in range(m.ii):
            kf = arrhenius(m.par[i], T)
            kr = arrhenius(m.rpar[i], T) if m.rev[i] == 2 else torch.zeros_like(T)
            M = C.sum(1) + sum((m.eff[i][k] - 1.0) * C[:, k] for k in range(9)) if m.thb[i] else torch.ones_like(T)
            if m.fall[i]:
                pr = arrhenius(m.low[i], T) * M / kf
                cor = pr / (1.0 + pr)
                if m.fall[i] > 2:
                    t = m.troe[i]
                    fc = (1.0 - t[0]) * torch.exp(-T / t[1]) + t[0] * torch.exp(-T / t[2])
                    if m.fall[i] == 4:
                        fc = fc + torch.exp(-t[3] / T)
                    lf, lp = torch.log10(fc), torch.log10(pr)
                    x = lp - (0.4 + 0.67 * lf)
                    cor = cor * 10.0 ** (lf / (1.0 + (x / (0.75 - 1.27 * lf - 0.14 * x)) ** 2))
                kf, kr, M = kf * cor, kr * cor, 1.0
            kf, kr = kf * M, kr * M
            for s in range(6):
                if pick[i][s] >= 0:
                    for _ in range(abs(nus[i][s])):
                        if s < 3:
                            kf = kf * C[:, pick[i][s]]
                        else:
                            kr = kr * C[:, pick[i][s]]
            for s in range(6):
                if pick[i][s] >= 0:
                    w[:, pick[i][s]] += nus[i][s] * (kf - kr)
        cv, e = torch.zeros_like(T), torch.zeros_like(T)
        for k in range(9):
            hi = (T > m.tmid[k]).to(F64)
            a = [m.a[k][0][j] * (1.0 - hi) + m.a[k][1][j] * hi for j in range(6)]
            cv += Y[:, k] * m.ru / wt[k] * (a[0] - 1.0 + T * (a[1] + T * (a[2] + T * (a[3] + T * a[4]))))
            u = m.ru * (T * (a[0] - 1.0 + T * (a[1] / 2 + T * (a[2] / 3 + T * (a[3] / 4 + T * a[4] / 5)))) + a[5])
            e += u * w[:, k]
        return -e / (rho * cv), w * wt / rho[:, None]

    steps = 100
    h = dt / steps
    H = h[:, None]
    for _ in range(steps):
        a = rhs(T, Y)
        b = rhs(T + 0.5 * h * a[0], Y + 0.5 * H * a[1])
        c = rhs(T + 0.5 * h * b[0], Y + 0.5 * H * b[1])
        d = rhs(T + h * c[0], Y + H * c[1])
        T = T + h / 6.0 * (a[0] + 2.0 * b[0] + 2.0 * c[0] + d[0])
        Y = Y + H / 6.0 * (a[1] + 2.0 * b[1] + 2.0 * c[1] + d[1])
    return {"T": T, "Y": Y}


def _euler_exact(case, seed):
    """The local Lax-Friedrichs characteristic WENO5 flux differences of the
    three sweeps: dense eigenvector products on every stencil point."""
    st = prepare(case, seed)
    g, thd = st["g"], st["g"].thd
    ng, nrv, n = 3, 9, (case["nx"], case["ny"], case["nz"])
    t = {k: torch.from_numpy(np.ascontiguousarray(st["in"][k].transpose())).cuda() for k in st["in"]}
    v, T, W_i, cp, ha, flag = t["v"], t["T"], t["W_i"], t["cp"], t["ha"], t["shock_sensor"] != 0
    g.close()
    Wc_i = _dev([thd.Wc_i[k] for k in range(nrv)])
    rho = v[0]
    vel = v[1:4] / rho
    P = rho * T * W_i
    c = torch.sqrt(P / rho / (1.0 - thd.gam2 * W_i / cp))
    Y = v[5:] / rho
    ht = (ha * Y).sum(0) + 0.5 * (vel * vel).sum(0)
    et = v[4] / rho
    out = torch.zeros((14,) + n[::-1], dtype=F64, device="cuda")
    axis = {0: 2, 1: 1, 2: 0}   # axis of (z, y, x)
    for d in range(3):
        ax = axis[d]

        def at(x, s):
            """x at the points s cells right of the left cell of every face 0..n."""
            lead = x.dim() - 3
            sl = [slice(None)] * lead + [slice(ng, -ng)] * 3
            sl[lead + ax] = slice(ng - 1 + s, ng - 1 + s + n[d] + 1)
            return x[tuple(sl)]

        r = torch.sqrt(at(rho, 1) / at(rho, 0))
        mean = lambda x: (r * at(x, 1) + at(x, 0)) / (r + 1.0)   # noqa: E731
        u, Yc, H, E = mean(vel), mean(Y), mean(ht), mean(et)
        Wm = (Yc * Wc_i[:, None, None, None]).sum(0)
        Tc = (H - E) / Wm
        hk, cpk = _nasa(thd, Tc)
        gam = 1.0 / (1.0 - thd.gam2 * Wm / (Yc * cpk).sum(0))
        cs = torch.sqrt(gam * Tc * Wm)
        psi = -hk + (gam / (gam - 1.0)) * Tc * Wc_i[:, None, None, None]
        q = 0.5 * (u * u).sum(0)
        b2 = (gam - 1.0) / (cs * cs)
        b1, xi, un = b2 * q, b2 * q - b2 * H, u[d]
        t1, t2 = [k for k in range(3) if k != d]
        w = torch.stack([at(v, s - 2) for s in range(6)])                          # stencil, variable, face
        us = torch.stack([at(vel[d], s - 2) for s in range(6)])
        ps = torch.stack([at(P, s - 2) for s in range(6)])
        cc = torch.stack([at(c, s - 2) for s in range(6)])
        f = w * us[:, None]
        f[:, 1 + d] += ps
        f[:, 4] += us * ps

        def left(x):
            sx = (psi[None] * x[:, 5:]).sum(1)
            mom = (u[None] * x[:, 1:4]).sum(1)
            common = b1 * x[:, 0] - b2 * mom + b2 * x[:, 4] + b2 * sx
            ac = (un * x[:, 0] - x[:, 1 + d]) / cs
            rows = [0.5 * (common + ac), x[:, 0] - common, 0.5 * (common - ac), x[:, 1 + t1] - u[t1] * x[:, 0],
                    x[:, 1 + t2] - u[t2] * x[:, 0],
                    (1.0 + xi) * (q * x[:, 0] - mom + x[:, 4]) + xi * sx]
            rows += [x[:, 5 + s] - Yc[s] * common for s in range(nrv - 1)]
            return torch.stack(rows, 1)

        lam = torch.stack([(us - cc).abs().amax(0), us.abs().amax(0), (us + cc).abs().amax(0)] +
                          [us.abs().amax(0)] * 11)
        pw, pf = left(w), left(f)
        gp = 0.5 * (pf + lam * pw)
        gm = pf - gp
        lin = ((-3.0 * gp[0] + 27.0 * gp[1] + 47.0 * gp[2] - 13.0 * gp[3] + 2.0 * gp[4]) +
               (2.0 * gm[1] - 13.0 * gm[2] + 47.0 * gm[3] + 27.0 * gm[4] - 3.0 * gm[5])) / 60.0
        nl = _weno5(gp[0], gp[1], gp[2], gp[3], gp[4]) + _weno5(gm[5], gm[4], gm[3], gm[2], gm[1])
        shk = torch.stack([at(flag, s - 2) for s in range(6)]).any(0)
        gh = torch.where(shk, nl, lin)
        fh = [gh[0] + gh[1] + gh[2], None, None, None,
              (H - un * cs) * gh[0] + q * gh[1] + (H + un * cs) * gh[2] + u[t1] * gh[3] + u[t2] * gh[4] + gh[5]]
        fh[1 + d] = (un - cs) * gh[0] + un * gh[1] + (un + cs) * gh[2]
        fh[1 + t1] = u[t1] * fh[0] + gh[3]
        fh[1 + t2] = u[t2] * fh[0] + gh[4]
        fh += [Yc[s] * (gh[0] + gh[2]) + gh[6 + s] for s in range(nrv - 1)]
        fh.append(Yc[nrv - 1] * (gh[0] + gh[2]) - (gh[5] + (psi[:nrv - 1] * gh[6:]).sum(0)) / psi[nrv - 1])
        fh = torch.stack(fh)
        out += torch.diff(fh, dim=1 + ax) * (constants()["l_ref"] / DX[d])   # uniform spacing
    return out.cpu().numpy().transpose(3, 2, 1, 0)


def _weno5(a, b, c, d, e):
    """Nonlinear WENO5 value right of c from the points a .. e (eps 1e-10)."""
    q = [(2.0 * c + 5.0 * d - e) / 6.0, (-b + 5.0 * c + 2.0 * d) / 6.0, (2.0 * a - 7.0 * b + 11.0 * c) / 6.0]
    be = [13.0 / 12.0 * (c - 2.0 * d + e) ** 2 + 0.25 * (3.0 * c - 4.0 * d + e) ** 2,
          13.0 / 12.0 * (b - 2.0 * c + d) ** 2 + 0.25 * (b - d) ** 2,
          13.0 / 12.0 * (a - 2.0 * b + c) ** 2 + 0.25 * (a - 4.0 * b + 3.0 * c) ** 2]
    al = [w / (1e-10 + x) ** 2 for w, x in zip((0.3, 0.6, 0.1), be)]
    return (al[0] * q[0] + al[1] * q[1] + al[2] * q[2]) / (al[0] + al[1] + al[2])


def _nasa(thd, T):
    """Species enthalpies and heat capacities (code units) at T."""
    h, cp = [], []
    for k in range(thd.nspc):
        t = T * thd.tinf
        hi = (t >= thd.tpolylim[k]).to(F64)
        a = [thd.heatcap[k][0][j] * (1.0 - hi) + thd.heatcap[k][1][j] * hi for j in range(7)]
        tc = t.clamp(thd.tpolymin[k], thd.tpolymax[k])
        c = a[0] + tc * (a[1] + tc * (a[2] + tc * (a[3] + tc * a[4])))
        dc = a[1] + tc * (2.0 * a[2] + tc * (3.0 * a[3] + tc * 4.0 * a[4]))
        hk = tc * (a[0] + tc * (a[1] / 2 + tc * (a[2] / 3 + tc * (a[3] / 4 + tc * a[4] / 5)))) + a[5]
        h.append((hk + c * (t - tc)) * thd.Wc_i[k] / thd.tinf)
        cp.append((c + dc * (t - tc)) * thd.gam2 * thd.Wc_i[k])
    return torch.stack(h), torch.stack(cp)
