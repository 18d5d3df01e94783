"""Performance cases: what programs that use this package have it do.

Every case goes through a public entry point: ``core.run_simulations`` (the
drop-in call behind ``SimGroup.run``: host arrays in, BOLD / FC / FCD / states
out), ``core.run_batch`` (groups of different networks in one call),
``grad.run_device`` (BOLD left on the GPU, as the fit harness evaluates its
candidates), ``grad.RWWProblem`` + ``grad.rww_fit_loss`` (one step of a gradient
fit) and ``utils.gof`` (scores of a finished batch).

Networks, parameter ranges, delays and batch shapes are those of ``bench.py``
and of the GPU tests (G x w_p x J_N grid, SC at 10-30 %, tract lengths in a 70-mm
sphere at 6 m/s, noise sigma 0.01).  Only the simulated time is shorter than the
60-900 s of a study, so that a pass stays below two seconds; the time loop does
the same work in every simulated second.  Volumes and windows are scaled with
it.  Wilson-Cowan G stays where trajectories are not chaotic (on these networks
they are above about 2), so that two correct programs can be compared.

``precision`` "fp32" integrates the node states in FP32 (the Balloon-Windkessel
state in FP64); a program that asks for it keeps the results in that width.
"""
import math

import numpy as np
import torch

from cubnm_b200 import core, grad, synthetic, utils

NOISE_S = 4          # noise segment, repeated with shuffles (SimGroup's noise_segment_length)


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one parameter point on a parcellated connectome, default precision: a user trying a model out
        {"name": "one_point_fp64", "kind": "run", "model": "rWW", "precision": "fp64", "nodes": 68, "sims": 1,
         "seconds": 5, "density": 0.3, "velocity": 0.0, "fic": 0},
        # the README grid with SimGroup's defaults (FP64, analytical FIC)
        {"name": "grid_fp64_fic", "kind": "run", "model": "rWW", "precision": "fp64", "nodes": 100, "sims": 100,
         "seconds": 8, "density": 0.3, "velocity": 0.0, "fic": 1},
        # a large random search in the default precision
        {"name": "search_fp64", "kind": "run", "model": "rWW", "precision": "fp64", "nodes": 100, "sims": 1000,
         "seconds": 6, "density": 0.3, "velocity": 0.0, "fic": 0},
        # one generation of an evolutionary fit in FP32
        {"name": "generation_fp32", "kind": "run", "model": "rWW", "precision": "fp32", "nodes": 100, "sims": 512,
         "seconds": 8, "density": 0.3, "velocity": 0.0, "fic": 0},
        # the headline workload: thousands of simulations on one SC, BOLD kept on the GPU for a loss
        {"name": "sweep_fp32_device", "kind": "device", "model": "rWW", "precision": "fp32", "nodes": 100,
         "sims": 8192, "seconds": 16, "density": 0.3, "velocity": 0.0, "fic": 0},
        # another model, ragged node and simulation counts, dense connectome
        {"name": "wc_ragged_fp32", "kind": "run", "model": "WC", "precision": "fp32", "nodes": 83, "sims": 1499,
         "seconds": 9, "density": 0.8, "velocity": 0.0, "fic": 0},
        # the 200-node fit network without gradients
        {"name": "rww_200_nodes_fp32", "kind": "run", "model": "rWW", "precision": "fp32", "nodes": 200, "sims": 512,
         "seconds": 6, "density": 0.25, "velocity": 0.0, "fic": 0},
        # conduction delays in the default precision
        {"name": "delays_fp64", "kind": "run", "model": "rWW", "precision": "fp64", "nodes": 100, "sims": 200,
         "seconds": 4, "density": 0.2, "velocity": 6.0, "fic": 0},
        # the large sparse network: Wilson-Cowan, 1,000 nodes, SC at 10 %, delays
        {"name": "wc_1000_nodes_delays", "kind": "run", "model": "WC", "precision": "fp32", "nodes": 1000,
         "sims": 150, "seconds": 1, "density": 0.1, "velocity": 6.0, "fic": 0},
        # the uneven batch: four parcellations x two durations, delays, one call
        {"name": "uneven_batch_delays", "kind": "batch", "model": "rWW", "precision": "fp32", "nodes": 400, "sims": 48,
         "seconds": 2, "density": 0.2, "velocity": 6.0, "fic": 0},
        # one gradient of the 200-node fit: forward, loss, backward
        {"name": "gradient_200_nodes", "kind": "grad", "model": "rWW", "precision": "fp32", "nodes": 200, "sims": 64,
         "seconds": 2, "density": 0.25, "velocity": 0.0, "fic": 0},
        # scoring a generation against the empirical FC / FCD
        {"name": "score_generation", "kind": "gof", "model": "rWW", "precision": "fp64", "nodes": 100, "sims": 128,
         "seconds": 60, "density": 0.3, "velocity": 0.0, "fic": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges, its simulated time and then its batch cut to a
    cost below the largest listed case's."""
    kind = rng.choice(["run", "run", "run", "run", "delay", "delay", "delay", "device", "grad", "gof", "batch"])
    if kind == "gof":
        return {"kind": "gof", "model": "rWW", "precision": "fp64", "nodes": rng.randint(20, 200),
                "sims": _log_int(rng, 8, 500), "seconds": rng.randint(40, 120), "density": 0.3, "velocity": 0.0,
                "fic": 0}
    if kind == "grad":
        return {"kind": "grad", "model": "rWW", "precision": "fp32", "nodes": rng.randint(30, 220),
                "sims": _log_int(rng, 4, 96), "seconds": rng.choice([1, 2]), "density": round(rng.uniform(0.1, 0.5), 2),
                "velocity": 0.0, "fic": 0}
    if kind == "batch":
        return {"kind": "batch", "model": "rWW", "precision": "fp32", "nodes": rng.randint(120, 400),
                "sims": _log_int(rng, 8, 48), "seconds": rng.choice([1, 2]), "density": round(rng.uniform(0.1, 0.3), 2),
                "velocity": round(rng.uniform(4.0, 10.0), 1), "fic": 0}
    delayed = kind == "delay"
    model = rng.choice(["rWW", "rWW", "rWW", "WC", "rWWEx", "JR"])
    precision = "fp32" if kind == "device" else rng.choice(["fp64", "fp32"])
    nodes = _log_int(rng, 20, 400)
    density = round(rng.uniform(0.1, 0.3) if delayed else rng.choice([rng.uniform(0.1, 0.4), rng.uniform(0.6, 1.0)]), 2)
    sims = _log_int(rng, 1, 4000 if kind == "device" else 1500)
    # JR oscillations are compared over a few seconds only
    seconds = rng.choice([1, 2, 3]) if delayed or model == "JR" else rng.choice([2, 4, 6, 9])
    # node-steps x (fan-in + update), weighted by what a step of the path costs
    weight = (24.0 if delayed else 1.0) * (2.0 if precision == "fp64" else 1.0) * (2.0 if nodes > 128 else 1.0)
    cost = nodes * (nodes * density + 60.0) * seconds * 1e4 * weight
    sims = max(1, min(sims, int(2.0e12 / cost)))
    return {"kind": "device" if kind == "device" else "run", "model": model, "precision": precision, "nodes": nodes,
            "sims": sims, "seconds": seconds, "density": density,
            "velocity": round(rng.uniform(4.0, 10.0), 1) if delayed else 0.0,
            "fic": 1 if model == "rWW" and not delayed and rng.random() < 0.3 else 0}


# ---------------------------------------------------------------- inputs
G_RANGE = {"rWW": (0.001, 10.0), "WC": (0.05, 1.5), "JR": (0.05, 1.0), "rWWEx": (0.05, 2.0)}
REGIONAL = {"rWW": 4, "WC": 8, "JR": 6, "rWWEx": 3}
STATES = {"rWW": 6, "WC": 2, "JR": 8, "rWWEx": 3}


def _timing(seconds):
    """(TR in ms, seconds of BOLD dropped, window, step in volumes)."""
    tr = 100 if seconds <= 2 else 250 if seconds <= 5 else 500
    return tr, seconds // 4, 6, 2


def _run_args(c, seed):
    """The 22 arguments of core.run_simulations for a case."""
    n, N = c["nodes"], c["sims"]
    rng = np.random.default_rng(seed)
    lo, hi = G_RANGE[c["model"]]
    tr, remove, window, step = _timing(c["seconds"])
    a = list(synthetic.synthetic_args(
        c["model"], N=N, nodes=n, duration_s=c["seconds"], seed=seed % 100003, density=c["density"],
        G=rng.uniform(lo, hi, N), w_p=rng.uniform(0, 2, N), J_N=rng.uniform(0.001, 0.5, N), do_fic=c["fic"],
        precision=c["precision"], window_size=window, window_step=step, bold_remove_s=remove))
    a[7] = dict(a[7], noise_time_steps=str(NOISE_S * 1000))
    a[17] = a[18] = tr
    reg = a[5].reshape(REGIONAL[c["model"]], N, n)
    if c["model"] == "rWW":  # w_p follows a regional map, as in map-parameterised fits
        reg[0] += rng.uniform(-0.3, 0.3, N)[:, None] * rng.standard_normal(n)[None, :]
    elif c["model"] == "WC":
        reg[6] = reg[7] = 0.01
    elif c["model"] == "rWWEx":
        reg[2] = 0.01
    if c["velocity"] > 0:
        a[3] = np.ascontiguousarray(synthetic.synthetic_lengths(n, seed % 100003).ravel())
        a[6] = np.full(N, c["velocity"])
        a[11] = True
    return a


def _batch_cases(c):
    """Groups of the uneven batch: four parcellations up to the case's, two durations."""
    return [dict(c, nodes=max(10, int(round(c["nodes"] * f))), seconds=c["seconds"] * d)
            for f in (0.17, 0.25, 0.5, 1.0) for d in (1, 2)]


def _fcd_sizes(c):
    vols = c["seconds"]
    windows = len(grad.window_bounds(vols, 0, 10, 2))
    return c["nodes"] * (c["nodes"] - 1) // 2, windows * (windows - 1) // 2


def _gradient_inputs(c, seed):
    n, N = c["nodes"], c["sims"]
    rng = np.random.default_rng(seed)
    emp = synthetic.synthetic_emp_bold(n, 40, seed % 100003)
    tr, remove, window, step = _timing(c["seconds"])
    return {"sc": synthetic.synthetic_sc(n, c["density"], seed % 100003), "G": rng.uniform(0.5, 3, N),
            "w_p": 1.0 + 0.2 * rng.standard_normal((N, n)), "J_N": np.repeat(rng.uniform(0.1, 0.3, (N, 1)), n, axis=1),
            "emp_fc": utils.calculate_fc(emp), "emp_fcd": utils.calculate_fcd(emp, window, step), "tr": tr,
            "remove": remove * 1000 // tr, "window": window, "step": step}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("run", "device"):
        return {"case": case, "args": _run_args(case, seed)}
    if kind == "batch":
        return {"case": case, "groups": [_run_args(g, seed + 17 * i) for i, g in enumerate(_batch_cases(case))]}
    if kind == "grad":
        x = _gradient_inputs(case, seed)
        dev = torch.device("cuda", 0)
        t = lambda v, g=False: torch.tensor(v, dtype=torch.float32, device=dev, requires_grad=g)  # noqa: E731
        N, n = case["sims"], case["nodes"]
        return {"case": case, "x": x,
                "problem": grad.RWWProblem(x["sc"], n, case["seconds"], bold_tr=x["tr"], noise_segment_s=NOISE_S),
                "G": t(x["G"], True), "w_p": t(x["w_p"], True), "J_N": t(x["J_N"], True), "wIE": t(np.ones((N, n))),
                "sigma": t(np.full((N, n), 0.01)),
                "emp_fc": torch.tensor(x["emp_fc"], device=dev), "emp_fcd": torch.tensor(x["emp_fcd"], device=dev)}
    # scores of a finished batch: correlated FC rows and FCD values, as a run returns them (host arrays)
    rng = np.random.default_rng(seed)
    P, M = _fcd_sizes(case)
    emp_fc = np.tanh(0.4 * rng.standard_normal(P))
    mix = rng.uniform(0, 1, (case["sims"], 1))
    return {"case": case, "emp_fc": emp_fc, "emp_fcd": np.tanh(0.3 + 0.4 * rng.standard_normal(M + 30)),
            "sim_fc": np.tanh(mix * np.arctanh(emp_fc)[None] + (1 - mix) * 0.4 * rng.standard_normal((case["sims"], P))),
            "sim_fcd": np.tanh(mix + 0.4 * rng.standard_normal((case["sims"], M)))}


# ---------------------------------------------------------------- one pass
def _results(out, args, case):
    """What the call returned, in the width of its precision."""
    width = np.float32 if case["precision"] == "fp32" else np.float64
    res = {k: out[k].astype(width, copy=False) for k in ("sim_bold", "sim_fc_trils", "sim_fcd_trils", "_sim_states")}
    if case["model"] == "rWW":
        res["bools"], res["ints"] = out["_global_bools"], out["_global_ints"]
        if case["fic"]:
            res["wIE"] = args[5][2].copy()  # solved by the call, in place
    return res


def run(state):
    c = state["case"]
    if c["kind"] == "run":
        return _results(core.run_simulations(*state["args"]), state["args"], c)
    if c["kind"] == "device":
        return {"sim_bold": grad.run_device(state["args"]).float()}
    if c["kind"] == "batch":
        outs = core.run_batch(state["groups"])
        return [_results(o, a, c) for o, a in zip(outs, state["groups"])]
    if c["kind"] == "grad":
        x = state["x"]
        for p in (state["G"], state["w_p"], state["J_N"]):
            p.grad = None
        bold = state["problem"].bold(state["G"], state["w_p"], state["J_N"], state["wIE"], state["sigma"])
        loss = grad.rww_fit_loss(bold, state["emp_fc"], state["emp_fcd"], x["remove"], x["window"], x["step"])
        loss.sum().backward()
        return {"loss": loss.detach().float(), "bold": bold.detach().float(), "G": state["G"].grad,
                "w_p": state["w_p"].grad, "J_N": state["J_N"].grad}
    return utils.gof(state["sim_fc"], state["emp_fc"], state["sim_fcd"], state["emp_fcd"])


# ---------------------------------------------------------------- what a pass cannot do without
UPDATE_FLOPS = {"rWW": 46, "WC": 40, "JR": 70, "rWWEx": 24}  # node update, an exp counted once
BW_FLOPS = 40                                                # Balloon-Windkessel step, once per ms


def _run_work(c):
    n, N, s = c["nodes"], c["sims"], c["seconds"]
    steps = s * 10000
    nnz = n * n * c["density"]
    flops = N * steps * (2.0 * nnz + n * UPDATE_FLOPS[c["model"]]) + N * s * 1000.0 * n * BW_FLOPS
    tr, remove, window, step = _timing(s)
    vols = s * 1000 // tr
    P = n * (n - 1) // 2
    W = len(grad.window_bounds(vols, remove * 1000 // tr, window, step))
    values = N * (vols * n + (REGIONAL[c["model"]] + STATES[c["model"]]) * n)
    if c["kind"] != "device":
        values += N * (P + W * (W - 1) // 2)
    flops += N * P * (2.0 * vols + 2.0 * W * (window + 1) + W * (W - 1))
    return 8.0 * (values + n * n + min(NOISE_S, s) * 10000 * n * 2), flops


def work(case):
    if case["kind"] == "gof":
        P, M = _fcd_sizes(case)
        return {"bytes": 8.0 * case["sims"] * (P + M), "flops": case["sims"] * (8.0 * P + 20.0 * M)}
    if case["kind"] == "batch":
        parts = [_run_work(g) for g in _batch_cases(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    b, f = _run_work(case)
    return {"bytes": b, "flops": 3.0 * f if case["kind"] == "grad" else f}  # backward: about twice a forward


# ---------------------------------------------------------------- the same numbers in 64 bits
def _noise(n, steps_bw, n_noise, bw_it, seed=0):
    """std::mt19937 + libstdc++ normal_distribution<double>, then the node and time shuffles."""
    count = n * steps_bw * 10 * n_noise
    bg = np.random.MT19937()
    bg._legacy_seeding(seed)
    need, got, used, parts = (count + 1) // 2, 0, 0, []
    while got < need:
        m = int((need - got) * 1.3) + 64
        u = bg.random_raw(4 * m).astype(np.float64)
        x = 2.0 * ((u[0::4] + u[1::4] * 2.0**32) / 2.0**64) - 1.0
        y = 2.0 * ((u[2::4] + u[3::4] * 2.0**32) / 2.0**64) - 1.0
        r2 = x * x + y * y
        at = np.flatnonzero((r2 <= 1.0) & (r2 != 0.0))[:need - got]
        f = np.sqrt(-2.0 * np.log(r2[at]) / r2[at])
        parts.append(np.stack([y[at] * f, x[at] * f], axis=1).ravel())
        got += at.size
        used += m if got < need else int(at[-1]) + 1
    noise = np.concatenate(parts)[:count].reshape(steps_bw, 10, n, n_noise)
    bg = np.random.MT19937()
    bg._legacy_seeding(seed)
    bg.random_raw(4 * used, output=False)  # the generator goes on after the last accepted pair
    repeats = -(-bw_it // steps_bw)

    def bounded(top):
        span = top + 1
        scale = 0xFFFFFFFF // span
        while True:
            r = int(bg.random_raw())
            if r < span * scale:
                return r // scale

    def shuffle(v):
        i = 1
        if len(v) % 2 == 0:
            j = bounded(1)
            v[1], v[j] = v[j], v[1]
            i = 2
        while i < len(v):
            x = bounded((i + 1) * (i + 2) - 1)
            for k in (x // (i + 2), x % (i + 2)):
                v[i], v[k] = v[k], v[i]
                i += 1
        return v

    nodes, times = list(range(n)), list(range(steps_bw))
    sh_n = [list(shuffle(nodes)) for _ in range(repeats)]
    sh_t = [list(shuffle(times)) for _ in range(repeats)]
    return noise, sh_n, sh_t


def _model(name, r):
    """(initial states, coupled state, BOLD state, step(s, in_, n0, n1) -> outputs and new states)."""
    dt, sq = 0.1, math.sqrt(0.1)
    clamp = lambda v: v.clamp(0.0, 1.0)  # noqa: E731
    G, r = r
    if name == "rWW":
        w_p, J, wIE, sig = r

        def step(s, q, n0, n1):
            IE = 0.382 + w_p * J * s[4] + q * G * J - wIE * s[5]
            II = 0.7 * 0.382 + J * s[4] - s[5]
            xE, xI = 310 * IE - 125, 615 * II - 177
            rE, rI = xE / (1 - torch.exp(-0.16 * xE)), xI / (1 - torch.exp(-0.087 * xI))
            dE = n0 * sig * sq + dt * (0.641 / 1000) * ((1 - s[4]) * rE) - dt / 100 * s[4]
            dI = n1 * sig * sq + dt / 1000 * rI - dt / 10 * s[5]
            return [IE, II, rE, rI, clamp(s[4] + dE), clamp(s[5] + dI)]
        return [0.0, 0.0, 0.0, 0.0, 0.001, 0.001], 4, 4, step
    if name == "WC":
        cEE, cIE, cEI, cII, PE, PI, sE, sI = r

        def step(s, q, n0, n1):
            SE = 1 / (1 + torch.exp(-1.5 * (cEE * s[0] - cIE * s[1] + G * q + PE - 3)))
            SI = 1 / (1 + torch.exp(-1.5 * (cEI * s[0] - cII * s[1] + PI - 3)))
            dE, dI = (-s[0] + (1 - s[0]) * SE) / 2.5, (-s[1] + (1 - s[1]) * SI) / 3.75
            return [clamp(s[0] + dt * dE + sq * n0 * sE), clamp(s[1] + dt * dI + sq * n1 * sI)]
        return [0.001, 0.001], 0, 0, step
    if name == "rWWEx":
        w, I0, sig = r

        def step(s, q, n0, n1):
            x = w * 0.2609 * s[2] + G * 0.2609 * q + I0
            v = 270 * x - 108
            rate = v / (1 - torch.exp(-0.154 * v))
            return [x, rate, clamp(s[2] + dt * (0.641 / 1000) * ((1 - s[2]) * rate) - dt / 100 * s[2] + n0 * sq * sig)]
        return [0.0, 0.0, 0.001], 2, 2, step
    J, a1, a2, a3, a4, sig = r
    A, B, a, b, v0, nu, rr, mu = 3.25, 22.0, 0.1, 0.05, 6.0, 0.0025, 0.56, 0.22
    sg = lambda v: 2 * nu / (1 + torch.exp(rr * (v0 - v)))  # noqa: E731

    def step(s, q, n0, n1):
        p0, p1, p2 = sg(s[1] - s[2]), sg(a1 * J * s[0]), sg(a3 * J * s[0])
        d3 = A * a * p0 - 2 * a * s[3] - a * a * s[0]
        d4 = A * a * (mu + a2 * J * p1 + G * q) - 2 * a * s[4] - a * a * s[1]
        d5 = B * b * (a4 * J * p2) - 2 * b * s[5] - b * b * s[2]
        y = [s[0] + dt * s[3], s[1] + dt * s[4], s[2] + dt * s[5], s[3] + dt * d3 + sq * n0 * sig, s[4] + dt * d4,
             s[5] + dt * d5]
        v = y[1] - y[2]
        return y + [v, 0.005 / (1 + torch.exp(rr * (6.0 - v)))]
    return [0.0] * 8, 7, 6, step


def _corr(x):
    """Pearson r of the columns of x [..., T, m], lower triangle."""
    x = x - x.mean(-2, keepdims=True)
    x = x / np.sqrt((x * x).sum(-2, keepdims=True))
    r = np.swapaxes(x, -1, -2) @ x
    i, j = np.tril_indices(x.shape[-1], -1)
    return r[..., i, j]


def _exact_run(c, seed):
    n, N, steps = c["nodes"], c["sims"], c["seconds"] * 10000
    delayed = c["velocity"] > 0
    # seconds on a GPU: launches, state traffic, gathered couplings
    est = steps * (1.6e-4 + N * n * 3e-10 + (N * n * n * 4e-11 if delayed else 0.0))
    if c["fic"] or est > 15.0:
        return None  # the FIC root is where the bracketing stops, not a 64-bit value; long runs take too long
    a = _run_args(c, seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    t = lambda v: torch.tensor(v, dtype=torch.float64, device=dev)  # noqa: E731
    sc = t(a[1].reshape(n, n))
    bw_it, tr = c["seconds"] * 1000, a[17]
    noise, sh_n, sh_t = _noise(n, NOISE_S * 1000, 2 if c["model"] in ("rWW", "WC") else 1, bw_it)
    noise, sh_n = t(noise), torch.tensor(sh_n, device=dev)
    reg = [t(v.reshape(N, n)) for v in a[5]]
    init, conn, boldv, step = _model(c["model"], (t(a[4].reshape(N, 1)), reg))
    s = [torch.full((N, n), v, dtype=torch.float64, device=dev) for v in init]
    x, f, nu, q = (torch.full((N, n), v, dtype=torch.float64, device=dev) for v in (0.0, 1.0, 1.0, 1.0))
    rows = torch.zeros_like(noise[0])  # this millisecond's noise [10, n, n_noise]
    if delayed:
        d = np.maximum(np.rint(np.float32(a[3].reshape(n, n) / (c["velocity"] * 0.1))).astype(np.int64), 1)
        d = np.tril(d, -1) + np.tril(d, -1).T
        D = int(d.max())
        src, dst = np.nonzero(np.asarray(a[1]).reshape(n, n))
        order = np.argsort(dst, kind="stable")
        src, dst = src[order], dst[order]
        lag = torch.tensor(d[src, dst], device=dev)
        wgt = sc[src, dst].reshape(-1, 1)
        src, dst = torch.tensor(src, device=dev), torch.tensor(dst, device=dev)
        hist = s[conn].T.reshape(1, n, N).repeat(D, 1, 1).reshape(D * n, N).contiguous()
        now = torch.zeros((), dtype=torch.int64, device=dev)

    def ms():
        for i in range(10):
            if delayed:
                at = ((now - lag) % D) * n + src
                inp = torch.zeros((n, N), dtype=torch.float64, device=dev).index_add_(0, dst, hist[at] * wgt).T
            else:
                inp = s[conn] @ sc
            new = step(s, inp, rows[i, :, 0], rows[i, :, -1])
            for old, v in zip(s, new):
                old.copy_(v)
            if delayed:
                hist.index_copy_(0, (now % D) * n + torch.arange(n, device=dev), s[conn].T.contiguous())
                now.add_(1)
        xn = x + 0.001 * (s[boldv] - x / 0.65 - (f - 1) / 0.41)
        fn = f + 0.001 * xn
        nun = nu + 0.001 / 0.98 * (f - nu ** (1 / 0.32))
        qn = q + 0.001 / 0.98 * (f * (1 - 0.66 ** (1 / f)) / 0.34 - nun ** (1 / 0.32) * q / nun)
        for old, v in ((x, xn), (f, fn), (nu, nun), (q, qn)):
            old.copy_(v)

    go = ms
    if dev.type == "cuda":
        keep = [v.clone() for v in s + [x, f, nu, q] + ([hist, now] if delayed else [])]
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            ms()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            ms()
        for v, k in zip(s + [x, f, nu, q] + ([hist, now] if delayed else []), keep):
            v.copy_(k)
        go = graph.replay
    bold, sums, kept = [], [torch.zeros_like(v) for v in s], 0
    remove = int(a[7]["bold_remove_s"]) * 1000 // tr
    for b in range(bw_it):
        rep, off = divmod(b, NOISE_S * 1000)
        rows.copy_(noise[sh_t[rep][off]][:, sh_n[rep]])
        go()
        if (b + 1) % tr == 0:
            bold.append(2.0 * (7 * 0.34 * (1 - q) + 2.0 * (1 - q / nu) + (2 * 0.34 - 0.2) * (1 - nu)))
            if len(bold) > remove:
                kept += 1
                for u, v in zip(sums, s):
                    u.add_(v)
    bold = torch.stack(bold, dim=1).cpu().numpy()
    if c["kind"] == "device":
        return {"sim_bold": bold}
    wins = grad.window_bounds(bold.shape[1], remove, int(a[7]["window_size"]), int(a[7]["window_step"]))
    wfc = np.stack([_corr(bold[:, lo:hi + 1]) for lo, hi in wins], axis=2)
    return {"sim_bold": bold.reshape(N, -1), "sim_fc_trils": _corr(bold[:, remove:]), "sim_fcd_trils": _corr(wfc),
            "_sim_states": torch.stack([u / kept for u in sums]).cpu().numpy()}


def _exact_gof(case, seed):
    s = prepare(case, seed)
    fc, e = s["sim_fc"], s["emp_fc"]
    xc, ec = fc - fc.mean(1, keepdims=True), e - e.mean()
    emp, ks = np.sort(s["emp_fcd"]), []
    for row in np.sort(s["sim_fcd"], axis=1):
        v = np.concatenate([row, emp])
        ks.append(np.abs(np.searchsorted(row, v, "right") / row.size - np.searchsorted(emp, v, "right") / emp.size).max())
    return {"fc_corr": (xc @ ec) / np.sqrt((xc * xc).sum(1) * (ec @ ec)), "fc_diff": np.abs(fc.mean(1) - e.mean()),
            "fc_normec": np.sqrt(((fc - e) ** 2).sum(1)) / (2 * math.sqrt(e.size)), "fcd_ks": np.array(ks)}


def exact(case, seed):
    if case["kind"] == "gof":
        return _exact_gof(case, seed)
    if case["kind"] in ("run", "device"):
        return _exact_run(case, seed)
    return None  # a batch is its groups' runs; gradients in 64 bits take a tape of every step
