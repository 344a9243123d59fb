"""Performance cases of the control-step library: what a racing program calls, at the sizes
it calls it with.

A case is one pass through the package's public entry points. Kinds:

  mppi    one control step of one or more MPPI controllers (strategic race or gate race),
          `via` one controller's getControl, a batch stepped with host buffers, or a batch
          stepped with device-resident inputs
  pr      one control step of one or more PR-MPPI controllers
  engine  one pass of the simulation engine's loop: control step, true-dynamics step,
          prediction streaming
  grad    forward and backward pass of the differentiable rollout objective

The states are drawn in mid-race: both agents on the track and moving, the opponent a few
metres ahead (or behind), a belief that is neither certain nor flat.
"""
from __future__ import annotations

import ctypes as C
import importlib
import importlib.util
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]


def _package():
    """The package (its directory name has a hyphen, so it is loaded by path)."""
    if "drone_race_b200" not in sys.modules:
        pkg = ROOT / "drone-race_b200"
        spec = importlib.util.spec_from_file_location("drone_race_b200", pkg / "__init__.py", submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["drone_race_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["drone_race_b200"]


# FP32 operations of one environment step of one rollout (each distinct operation once):
# rollout and verification steps of the strategic race and the gate race, and a PR-MPPI step.
STEP_FLOPS = {"strat": (442.0, 233.7), "gate": (189.7, 117.8)}
PR_STEP_FLOPS = {"strat": 411.7, "gate": 189.7}


def listed() -> list[dict]:
    return [
        # One small drone brain in its own control loop: the smallest MPPI call, all latency.
        dict(name="gate_one_small", kind="mppi", race="gate", via="one", agents=1, K=512, T=40, V=1024, n_theta=2, splines=False, gates=2),
        # A single agent with the settings of the small single-agent race (8-point ellipse).
        dict(name="one_agent", kind="mppi", race="ellipse", via="one", agents=1, K=1024, T=50, V=4096, n_theta=2, splines=False),
        # The simulation engine's loop with its front-end's own settings (spline controls, 2^16 samples).
        dict(name="engine_front_end", kind="engine", race="round", agents=1, K=65536, T=80, V=131072, n_theta=2, splines=True),
        # The benchmark's four-agent race, inputs and results resident on the device.
        dict(name="four_agents", kind="mppi", race="circle", via="device", agents=4, K=4096, T=64, V=131072, n_theta=2, splines=False),
        # The same race with a quarter of the samples and a gradient step after each update.
        dict(name="four_agents_refined", kind="mppi", race="circle", via="device", agents=4, K=1024, T=64, V=131072, n_theta=2, splines=False, refine=1),
        # Many opponent hypotheses (a branch plan for each) at sizes that fill no tile evenly.
        dict(name="eight_branches_odd", kind="mppi", race="circle", via="batch", agents=2, K=3001, T=61, V=20011, n_theta=8, splines=False),
        # A server of many races: agents of very different sizes in one batch, spline controls.
        dict(name="uneven_races", kind="mppi", race="circle", via="batch", agents=24, K=16384, T=96, V=4096, n_theta=2, splines=True, uneven=True),
        # The benchmark's PR-MPPI race: eight hypotheses, host buffers.
        dict(name="pr_four_agents", kind="pr", race="circle", via="batch", agents=4, K=2048, T=64, P=8, n_theta=8),
        # One PR-MPPI agent with the front-end's own settings.
        dict(name="pr_front_end", kind="pr", race="round", via="one", agents=1, K=65536, T=60, P=9, n_theta=2),
        # The gate race at the benchmark's size, host buffers.
        dict(name="gate_four_agents", kind="mppi", race="gate", via="batch", agents=4, K=4096, T=64, V=131072, n_theta=2, splines=False, gates=8),
        # One PR-MPPI agent in the gate race.
        dict(name="gate_pr_one", kind="pr", race="gate", via="one", agents=1, K=2048, T=64, P=8, n_theta=2, gates=8),
        # Training through the rollout: objective and gradients at a set of start points.
        dict(name="gradient", kind="grad", race="circle", n=64, T=64, n_theta=2),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    """A case of the ranges that the listed ones stand for, at most as large as their largest."""
    kind = rng.choice(["mppi", "mppi", "mppi", "pr", "pr", "engine", "grad"])
    if kind == "grad":
        return dict(kind="grad", race="circle", n=_log_int(rng, 1, 128), T=rng.randint(24, 80), n_theta=rng.choice([2, 2, 4]))
    T = rng.randint(30, 96)
    K = _log_int(rng, 256, 65536)
    if kind == "engine":
        c = dict(kind="engine", race=rng.choice(["round", "circle"]), agents=1, K=K, T=T, V=_log_int(rng, 1024, 131072), n_theta=2,
                 splines=rng.choice([True, False]))
    elif kind == "pr":
        race = rng.choice(["circle", "circle", "round", "gate"])
        c = dict(kind="pr", race=race, via="batch" if race == "circle" else "one", agents=rng.randint(1, 6) if race == "circle" else 1, K=K, T=T,
                 P=rng.randint(2, 10), n_theta=rng.choice([2, 4, 8]) if race == "circle" else 2)
    else:
        race = rng.choice(["circle", "circle", "ellipse", "gate"])
        via = rng.choice(["one", "batch", "device"])
        c = dict(kind="mppi", race=race, via=via, agents=1 if via == "one" else rng.randint(1, 8), K=min(K, 16384), T=T, V=_log_int(rng, 1024, 131072),
                 n_theta=rng.choice([1, 2, 2, 4, 8]) if race == "circle" else 2, splines=rng.choice([True, False]))
        if race == "circle" and rng.random() < 0.25:
            c["refine"] = rng.randint(1, 3)
    if c["race"] == "gate":
        c["gates"] = rng.randint(2, 12)
    most = 0.5 * max(work(x)["flops"] for x in listed())
    while work(c)["flops"] > most:
        if c["agents"] > 1:
            c["agents"] = (c["agents"] + 1) // 2
        else:
            c["K"] = c["K"] * 2 // 3
            if "V" in c:
                c["V"] = max(1024, c["V"] * 2 // 3)
    return c


def _sizes(case: dict) -> list[tuple[int, int]]:
    """(K, T) of each agent: the case's own, or uneven ones (log-uniform samples up to K,
    horizons of a third of T up to T) fixed by the case."""
    if not case.get("uneven"):
        return [(case["K"], case["T"])] * case["agents"]
    r = random.Random(case["agents"] * 1000 + case["K"])
    return [(_log_int(r, 256, case["K"]), max(32, case["T"] * r.choice([2, 3, 4, 6]) // 6)) for _ in range(case["agents"])]


def work(case: dict) -> dict:
    """Environment steps that the path cannot do without, in FP32 operations; bytes: inputs,
    plans and results, each once (the samples' perturbations are drawn, not read)."""
    nth, T = case["n_theta"], case["T"]
    grids = 512 * 7 * 4
    if case["kind"] == "grad":
        knots = case["n"] * (nth + 1) * T * 2 * 4
        # a forward step and the reverse step's products (about three times the forward's)
        return {"bytes": grids + 2 * knots + case["n"] * (1 + 2 * 6) * 4, "flops": 4 * case["n"] * nth * T * STEP_FLOPS["strat"][0]}
    race = "gate" if case["race"] == "gate" else "strat"
    if case["kind"] == "pr":
        steps = case["agents"] * T * case["P"] * (2 * case["K"] + 4)
        return {"bytes": case["agents"] * (grids + 4 * T * 2 * 4 + 256), "flops": steps * PR_STEP_FLOPS[race]}
    roll, ver = STEP_FLOPS[race]
    flops = bts = 0.0
    for K, t in _sizes(case):
        flops += K * nth * t * roll + 2 * case["V"] * min(40, t) * ver
        bts += grids + 3 * (nth + 1) * t * 2 * 4 + 256
    return {"bytes": bts, "flops": flops}


# ---- scenarios -----------------------------------------------------------------------------


def _moving_state(sc, rng: np.random.Generator):
    """Both agents on the track in mid-race: the opponent 1.5 to 8 m of arc from the ego,
    ahead of it four times out of five, each within its lane, at racing speed."""
    drb = _package()
    g, e = sc.grids, sc.env
    per = g.track_length / 512
    s = drb.abi.dr_sim_state()
    ego = int(rng.integers(0, 512))
    gap = rng.uniform(1.5, 8.0) * (1 if rng.uniform() < 0.8 else -1)
    for a, i in enumerate((ego, (ego + int(round(gap / per))) % 512)):
        lat = float(rng.uniform(-0.4, 0.4)) * (float(e.track_width) - float(e.drone_radius))
        v = float(rng.uniform(0.4, 1.0)) * float(e.max_speed[a])
        t0, t1 = float(g.t_grid[i, 0]), float(g.t_grid[i, 1])
        s.pos[2 * a] = float(g.p_grid[i, 0]) - lat * t1
        s.pos[2 * a + 1] = float(g.p_grid[i, 1]) + lat * t0
        s.vel[2 * a], s.vel[2 * a + 1] = v * t0, v * t1
        s.S[a] = float(np.float32(i / 512 * g.track_length))
        s.lat_dist[a] = lat
    return s


def _gate_state(sc, n_gates: int, rng: np.random.Generator):
    drb = _package()
    ego = float(rng.uniform(0.0, 0.9))
    u = [ego, ego + float(rng.uniform(0.02, 0.08))]
    last = [(int(math.ceil(x * n_gates)) % n_gates - 1) % n_gates for x in u]
    return drb.scenarios.gate_state(sc.track, u, 0, last, speed=float(rng.uniform(1.0, 4.0)))


def _belief(n: int, rng: np.random.Generator) -> np.ndarray:
    b = rng.dirichlet(np.full(n, 3.0)).astype(np.float32)
    return b / b.sum(dtype=np.float32)


def _scenarios(case: dict, seed: int):
    """One scenario per agent, each with a mid-race state, and their beliefs."""
    S = _package().scenarios
    rng = np.random.default_rng([seed, 17])
    nth, track = case["n_theta"], int(rng.integers(1 << 20))
    scs = []
    for a, (K, T) in enumerate(_sizes(case)):
        sd = int(rng.integers(1 << 30))
        spl, V, P = case.get("splines", False), case.get("V", 0), case.get("P", 0)
        if case["race"] == "gate":
            sc = S.gate_race(agent=a, seed=sd, K=K, T=T, use_splines=spl, n_verif=max(V, 1), n_gates=case["gates"])
            if P:
                sc.prmppi = S.make_prmppi(K=K, T=T, P=P)
            sc.state = _gate_state(sc, case["gates"], rng)
        else:
            if P and case["race"] == "circle":
                sc = S.robust_race(agent=a, seed=track, K=K, T=T, P=P, n_theta=nth)
            elif case["race"] == "circle":
                sc = S.circle_race(agent=a, seed=track, K=K, T=T, use_splines=spl, n_theta=nth, n_verif=max(V, 1))
            elif case["race"] == "ellipse":
                sc = S.ellipse_race(seed=track, K=K, T=T, use_splines=spl, n_verif=max(V, 1))
            else:
                sc = S.strat_race(use_pr=bool(P), use_splines=spl, K=K, T=T, n_configs=nth, n_verif=max(V, 1))
                if P:
                    sc.prmppi = S.make_prmppi(K=K, T=T, P=P)
            sc.state = _moving_state(sc, rng)
            sc.seed = sd
        scs.append(sc)
    return scs, np.stack([_belief(nth, rng) for _ in scs])


_control_stream = None


def _stream() -> int:
    """The one CUDA stream of the program's control loop."""
    global _control_stream
    if _control_stream is None:
        _control_stream = torch.cuda.Stream()
    return _control_stream.cuda_stream


def _fields(infos) -> dict:
    """A view of an array of info records by field."""
    a = np.frombuffer(infos, dtype=np.dtype(type(infos)._type_))
    return {n: a[n] for n in a.dtype.names}


def prepare(case: dict, seed: int):
    drb = _package()
    ctl, abi = drb.controllers, drb.abi
    if case["kind"] == "grad":
        return _prepare_grad(case, seed)
    scs, beliefs = _scenarios(case, seed)
    if case["kind"] == "pr":
        cs = [ctl.PRMPPIController(sc.env, sc.prmppi, sc.seed, stream=_stream()) for sc in scs]
    else:
        cs = [ctl.MPPIController(sc.env, sc.mppi, sc.seed, stream=_stream()) for sc in scs]
        for c in cs:
            if case.get("refine"):
                c.set_grad_refine(case["refine"])
    for c, b in zip(cs, beliefs):
        c.engine = True  # the object that drives the controller
        c.h_belief = b.copy()
    s = dict(case=case, scs=scs, beliefs=beliefs)
    if case["kind"] == "engine" or case["via"] == "one":
        s["ctl"] = cs[0]
        return s
    batch = (ctl.PRMPPIBatch if case["kind"] == "pr" else ctl.MPPIBatch)(cs, stream=_stream())
    s["batch"] = batch
    s["states"] = [sc.state for sc in scs]
    if case["via"] == "device":
        n, dev = len(scs), "cuda"
        raw = b"".join(bytes(sc.state) for sc in scs)
        s["d_states"] = torch.frombuffer(bytearray(raw), dtype=torch.uint8).to(dev)
        bel = np.zeros((n, abi.DR_MAX_THETA), np.float32)
        bel[:, : beliefs.shape[1]] = beliefs
        s["d_beliefs"] = torch.from_numpy(bel).to(dev)
        s["d_actions"] = torch.zeros((n, 2), dtype=torch.float32, device=dev)
        info = torch.zeros((n, C.sizeof(abi.dr_mppi_info)), dtype=torch.uint8, device=dev)
        s["d_infos"] = info
        # the records' fields, as views: counts and choices, bounds, costs and temperature
        i32, f64, f32 = info.view(torch.int32), info.view(torch.float64), info.view(torch.float32)
        s["d_fields"] = dict(counts=i32[:, 0:2], bounds=f64[:, 1:4], branch=i32[:, 8], costs=f32[:, 9:12], status=i32[:, 12:14], refine=f32[:, 14:16],
                             best_step=i32[:, 16])
        torch.cuda.current_stream().synchronize()
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "grad":
        return _run_grad(s)
    if case["kind"] == "engine":
        return _run_engine(s)
    if case["via"] == "device":
        s["batch"].step_device(s["d_states"].data_ptr(), s["d_beliefs"].data_ptr(), s["d_actions"].data_ptr(), s["d_infos"].data_ptr())
        return dict(actions=s["d_actions"], **s["d_fields"])
    if case["via"] == "batch":
        b = s["batch"]
        out = dict(actions=b.step(s["states"], s["beliefs"]), **_fields(b.infos))
        if case["kind"] == "mppi":  # the plan that each controller holds now
            out["plans"] = np.concatenate([c.h_nominal for c in b.ctls])
        else:
            out["plans"] = np.concatenate([p for c in b.ctls for p in c.nominals()])
        return out
    c = s["ctl"]
    out = dict(action=c.getControl(s["scs"][0].state), **_fields((type(c.info) * 1).from_buffer(c.info)))
    if case["kind"] == "pr":
        out["nominal"], out["robust"] = c.nominals()
    else:
        out.update(plan=c.h_nominal, failed_new=c.failCountNew, failed_old=c.failCountOld)
    return out


def _run_engine(s):
    """The engine's loop body: the controller's action, the race advanced by it under the
    true hypothesis, the controller's predictions from there."""
    drb = _package()
    c, sc = s["ctl"], s["scs"][0]
    step = c.step_index
    action = c.getControl(sc.state)
    state = drb.abi.dr_sim_state.from_buffer_copy(sc.state)
    belief = np.zeros(drb.abi.DR_MAX_THETA, np.float32)
    belief[: sc.n_theta] = c.h_belief
    term = drb.controllers.env_step(sc.env, sc.true_theta, action, state, belief, True, sc.seed, step)
    pred = c.predict(state, belief[: sc.n_theta])
    return dict(action=action, plan=c.h_nominal, failed_new=c.failCountNew, failed_old=c.failCountOld, term=term, belief=belief,
                pos=np.array(state.pos), vel=np.array(state.vel), arc=np.array(state.S), lat=np.array(state.lat_dist), laps=np.array(state.laps),
                predicted=pred, **_fields((type(c.info) * 1).from_buffer(c.info)))


# ---- the differentiable objective -----------------------------------------------------------


def _grad_case(case: dict, seed: int):
    scs, beliefs = _scenarios(dict(case, agents=1, K=256, V=1024, kind="mppi", via="one"), seed)
    g = torch.Generator().manual_seed(seed)
    sc, n, nth = scs[0], case["n"], case["n_theta"]
    U = torch.randn((n, nth + 1, case["T"], 2), generator=g) * 1.5
    w = torch.tensor([float(getattr(sc.mppi, k)) for k in _WEIGHTS])
    W = w * torch.exp(0.3 * torch.randn((n, 6), generator=g))
    return sc, beliefs[0], U, W


_WEIGHTS = ("boundary_cost", "outside_cost", "win_cost", "opp_win_cost", "final_adv_weight", "final_opp_adv_weight")


def _prepare_grad(case: dict, seed: int):
    drb = _package()
    sc, belief, U, W = _grad_case(case, seed)
    c = drb.controllers.MPPIController(sc.env, sc.mppi, sc.seed)
    return dict(case=case, sc=sc, ctl=c, belief=torch.from_numpy(belief), U=U.cuda().requires_grad_(), W=W.cuda().requires_grad_(),
                G=importlib.import_module("drone_race_b200.grad"))


def _run_grad(s):
    s["U"].grad = s["W"].grad = None
    J = s["G"].nominal_cost(s["ctl"], s["sc"].state, s["belief"], s["U"], s["W"])
    J.sum().backward()
    return dict(J=J.detach(), dU=s["U"].grad, dW=s["W"].grad)


def exact(case: dict, seed: int):
    """The objective and its gradients in 64 bits. A control step has no such value: it is an
    estimate from the library's own random draws, whose samples cross the model's thresholds
    (branch, collision, lap) one way or the other."""
    if case["kind"] != "grad":
        return None
    sc, belief, U, W = _grad_case(case, seed)
    U, W = U.double().requires_grad_(), W.double().requires_grad_()
    J = _objective(sc, torch.from_numpy(belief).double(), U, W)
    J.sum().backward()
    return dict(J=J.detach(), dU=U.grad, dW=W.grad)


def _objective(sc, belief0, U, W):
    """The noise-free rollout of the dense controls U (n, n_theta + 1, T, 2) under every
    hypothesis, costed with the weights W (n, 6) and averaged over the belief: one opponent,
    plain torch, all start points and hypotheses side by side. Decisions (projection
    windows, clamps, branches, endings) are taken on the values."""
    e, c, nth, T = sc.env, sc.mppi, sc.n_theta, U.shape[2]
    f = lambda x: float(np.float32(x))
    n = U.shape[0]
    shape = (n, nth)
    L, dt, rad, width, kV = f(e.track_length), f(e.dt), f(e.drone_radius), f(e.track_width), f(e.kV)
    vmax, amax = [f(v) for v in e.max_speed], [f(v) for v in e.max_accel]
    opp = lambda name: torch.tensor([f(getattr(e.opp_configs[h], name)[0]) for h in range(nth)], dtype=torch.float64)
    s1, s2, s3, speed, noise = opp("s1"), opp("s2"), opp("s3"), opp("speed_scale"), opp("action_noise")
    grid = lambda a: torch.from_numpy(np.asarray(a, np.float64))
    P, Tg, Kp = grid(sc.grids.p_grid), grid(sc.grids.t_grid), grid(sc.grids.kappa_grid)
    where, sqrt0 = torch.where, lambda x: torch.where(x > 0, torch.sqrt(torch.where(x > 0, x, torch.ones_like(x))), 0.0 * x)
    norm2 = lambda v: (v * v).sum(-1)
    cross = lambda a, b: a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]

    def place(S):
        x = S / L
        x = (x - torch.floor(x.detach())) * 512
        i = x.detach().long()
        return i % 512, (i + 1) % 512, x - i

    def along(grid2, q):
        i, j, t = q
        return (1 - t)[..., None] * grid2[i] + t[..., None] * grid2[j]

    def tangent(q):
        t = along(Tg, q)
        return t / torch.sqrt(norm2(t))[..., None]

    def curvature(q):
        return (1 - q[2]) * Kp[q[0]] + q[2] * Kp[q[1]]

    def arc_speed(tg, kap, lat, vel):
        m = 1 - kap * lat
        return (tg * vel).sum(-1) / where(m.abs() < 1e-12, torch.copysign(torch.full_like(m, 1e-12), m), m)

    def project(pos, S):
        i = place(S)[0]
        win = (i[..., None] + torch.arange(-10, 11)) % 512
        near = torch.gather(win, -1, norm2(P[win] - pos.detach()[..., None, :]).argmin(-1, keepdim=True))[..., 0]
        best = None
        for seg in (-1, 0):
            a = (near + seg) % 512
            A = P[a]
            ab = P[(a + 1) % 512] - A
            t = (((pos - A) * ab).sum(-1) / norm2(ab)).clamp(0.0, 1.0)
            foot = A + t[..., None] * ab
            cand = (norm2(pos - foot), (a + t) / 512 * L, foot)
            if best is None:
                best = cand
            else:
                less = cand[0] < best[0]
                best = (where(less, cand[0], best[0]), where(less, cand[1], best[1]), where(less[..., None], cand[2], best[2]))
        d2, S, foot = best
        side = cross(along(Tg, place(S)), (pos - foot).detach())
        d = sqrt0(d2)
        return S, where(side.detach() < 0, -d, d)

    def cap(v, most):
        q = norm2(v)
        return v * where(q > most * most, most / torch.sqrt(where(q > most * most, q, torch.ones_like(q))), torch.ones_like(q))[..., None]

    def policy(pos, vel, S, lat, geo, h):
        """The opponent's action under hypothesis h (columns of shape (n, nth))."""
        (tg0, _, sd0), (tg, kap, sd) = geo
        d = S[0] - S[1]
        goal = (speed[h] * vmax[1]).expand(shape)
        base, aim = goal, torch.zeros(shape, dtype=torch.float64)
        dE = lat[0] - lat[1]
        for ahead in (False, True):
            dS = where(d < 0, d + L, d) if ahead else where(d > 0, d - L, d)
            tol = vmax[0] * 0.3
            block = (dS < 0) & (dS > -L * 0.25) & (sd0 + tol > sd)
            over = (sd > sd0) & (dE.abs() < s1[h])
            near = torch.exp(-s2[h] * dS * dS)
            aim = aim + where(block, lat[0] * (1 - torch.exp(where(block, -s3[h] * (sd0 + tol - sd), 0.0 * dS))) * near, 0.0 * dS)
            aim = aim + where(over, (lat[0] - torch.copysign(s1[h].expand(shape), dE.detach())) * near, 0.0 * dS)
            ego_long = (vel[0] * tg0).sum(-1)
            close = over & (dS < 3 * rad)
            mid = over & ~close & (dS < 6 * rad) & bool(s1[h] > 1e-6)
            goal = where(close, torch.minimum(goal, 0.7 * ego_long), goal)
            lf = dE.abs() / s1[h].clamp_min(1e-30)
            goal = where(mid, torch.minimum(goal, lf * ego_long + (1 - lf) * base), goal)
        most = width - rad * f(e.max_opp_lat_dist_fact)
        aim = aim.clamp(-most, most)
        nrm = torch.stack([-tg[..., 1], tg[..., 0]], -1)
        e_n = ((pos[1] - along(P, place(S[1]))) * nrm).sum(-1)
        v_t, v_n = (vel[1] * tg).sum(-1), (vel[1] * nrm).sum(-1)
        e_max = width - rad * 1.2
        m = 1 - kap * e_n
        m = where(m.abs() < 1e-6, torch.copysign(torch.full_like(m, 1e-6), m), m)
        a_c = v_t * v_t * kap / m
        a_lat = torch.clamp_min(amax[1] - a_c.abs(), amax[1] * 0.2)
        aim = aim.clamp(-e_max, e_max)
        err = aim - e_n
        room = torch.clamp_min(e_max - e_n, 0.001), torch.clamp_min(e_max + e_n, 0.001)
        kp = a_lat / 0.02
        hold = kp * err - 2 * torch.sqrt(kp) * v_n
        hold = torch.maximum(-a_lat, torch.minimum(a_lat, hold))
        toward = ((err > 0) & (v_n > 0)) | ((err < 0) & (v_n < 0))
        slow = toward & (v_n * v_n / (2 * a_lat) >= err.abs() * 0.95)
        bang = where((err > 0) ^ slow, a_lat, -a_lat)
        nxt = v_n + bang * dt
        safe = torch.sqrt(2 * a_lat * where(nxt > 0, room[0], room[1]))
        bang = where((nxt > 0) & (nxt > safe), (safe - v_n) / dt, where((nxt <= 0) & (-nxt > safe), (-safe - v_n) / dt, bang))
        a_n = where(err.abs() < 0.02, hold, bang)
        a_n = where((v_n < 0) & (v_n * v_n > 1.8 * a_lat * room[1]), a_lat, a_n)
        a_n = where((v_n > 0) & (v_n * v_n > 1.8 * a_lat * room[0]), -a_lat, a_n)
        a_tot = (a_n + a_c).clamp(-amax[1], amax[1])
        a_t_max = sqrt0(torch.clamp_min(amax[1] ** 2 - a_tot * a_tot, 0.0))
        k_eff = kap / (1 - kap * aim + 1e-6)
        path = torch.minimum(goal, torch.sqrt(amax[1] / torch.clamp_min(k_eff.abs(), 1e-12)))
        path = where(a_n.abs() > a_lat * 0.5, path * torch.clamp_min(1.5 - a_n.abs() / a_lat, 0.4), path)
        a_t = kV * (path - v_t) - v_n * kap * v_t / m
        a_t = torch.maximum(-a_t_max, torch.minimum(a_t_max, a_t))
        return a_t[..., None] * tg + a_tot[..., None] * nrm

    st = sc.state
    col = lambda v: torch.full(shape, f(v), dtype=torch.float64)
    pos = [torch.stack([col(st.pos[2 * a]), col(st.pos[2 * a + 1])], -1) for a in range(2)]
    vel = [torch.stack([col(st.vel[2 * a]), col(st.vel[2 * a + 1])], -1) for a in range(2)]
    S, lat = [col(st.S[a]) for a in range(2)], [col(st.lat_dist[a]) for a in range(2)]
    laps = [torch.full(shape, int(st.laps[a])) for a in range(2)]
    conf = f(c.min_confidence)
    sure = lambda b: where((b > conf).any(-1), (b > conf).int().argmax(-1) + 1, 0)
    bel = belief0.expand(n, nth, nth).clone()  # [start point, true hypothesis, hypothesis]
    branch = sure(bel)
    counted = (branch == 0) | (branch == torch.arange(nth) + 1)
    origin, run_on = torch.zeros(shape, dtype=torch.long), counted.clone()
    cost, decay = torch.zeros(shape, dtype=torch.float64), 1.0
    rows, cols = torch.arange(n)[:, None].expand(shape), torch.arange(nth).expand(shape)
    keep = lambda new, old: where(run_on.reshape(shape + (1,) * (new.dim() - 2)), new, old)
    for t in range(T):
        if not bool(run_on.any()):
            break
        act0 = cap(U[rows, branch, t - origin], amax[0])
        geo = []
        for a in range(2):
            q = place(S[a])
            tg, kap = tangent(q), curvature(q)
            geo.append((tg, kap, arc_speed(tg, kap, lat[a], vel[a])))
        plans = torch.stack([policy(pos, vel, S, lat, geo, h) for h in range(nth)], 2)
        act1 = cap(plans[rows, cols, cols], amax[1])
        now = []
        for a, act in ((0, act0), (1, act1)):
            p, v = pos[a] + dt * vel[a], cap(vel[a] + dt * act, vmax[a])
            s_new, l_new = project(p, S[a] + dt * geo[a][2])
            lap = laps[a] + (s_new < S[a] - L * 0.5).long() - (s_new > S[a] + L * 0.5).long()
            now.append((p, v, s_new, l_new, lap))
        sig = f(0.2) ** 2 + noise * noise
        like = -0.5 * norm2(act1[:, :, None] - cap(plans, amax[1])) / sig - math.log(2 * math.pi) - torch.log(sig)
        b_new = bel * torch.exp(like)
        total = b_new.sum(-1, keepdim=True)
        b_new = where(total < 1e-20, torch.full_like(b_new, 1.0 / nth), b_new / total.clamp_min(1e-300))
        for a in range(2):
            pos[a], vel[a], S[a], lat[a], laps[a] = (keep(x, y) for x, y in zip(now[a], (pos[a], vel[a], S[a], lat[a], laps[a])))
        bel = keep(b_new, bel)
        takes = run_on & (branch == 0) & (sure(bel) != 0)
        branch, origin = where(takes, sure(bel), branch), where(takes, t + 1, origin)
        bd = torch.minimum(torch.sqrt(norm2(pos[1] - pos[0])) - rad, width - lat[0].abs())
        lost_to, won = laps[1] >= e.n_win_laps, (laps[0] >= e.n_win_laps) | (lat[1].abs() > width - rad)
        w = W[:, None, :].expand(n, nth, 6)
        step = where(bd < f(c.boundary_threshold_factor) * rad, w[..., 0] * (bd / rad) ** 2, 0.0 * bd)
        step = step + where(bd < rad * f(c.coll_dist_factor), w[..., 1], 0.0 * bd) + where(lost_to, w[..., 3], 0.0 * bd) - where(won, w[..., 2], 0.0 * bd)
        cost = cost + where(run_on, step * decay, 0.0 * step)
        decay *= f(0.97)
        run_on = run_on & ~(lost_to | (bd < rad) | won)
    w = W[:, None, :].expand(n, nth, 6)
    cost = cost - w[..., 4] * (S[0] / L + laps[0]) + w[..., 5] * (S[1] / L + laps[1])
    share = where(counted, belief0.expand(shape), torch.zeros(shape, dtype=torch.float64))
    return (where(counted, cost, 0.0 * cost) * share).sum(-1) / share.sum(-1)
