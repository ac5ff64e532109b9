"""The solver's work as a user's program asks for it, one case per kind of call.

Every case goes through the public Python binding (annealing_gb300): a resident plan run again with
its seed, one blocking solve from host couplings, a batch of uneven instances, a burst of served
requests, an SQA anneal, an NMFA anneal. Couplings are drawn on the device from the seed alone with
the distributions of the solver's workloads: complete or Erdos-Renyi +-1 graphs, integers in
[-jmax, jmax], or N(0, 1/n) reals with N(0, 0.1) fields. The instance sizes of a batch or a burst are
part of the case (spread over its range), so that another seed gives other couplings of the same sizes.
"""
import math

import numpy as np
import torch

import annealing_gb300 as sb

DEV = "cuda" if torch.cuda.is_available() else "cpu"
VARIANT = {"asb": sb.ASB, "bsb": sb.BSB, "dsb": sb.DSB}


def listed():
    return [
        # the smallest anneal a program repeats: 128 spins, one trajectory; launch latency and the
        # exchange between steps are all there is
        {"name": "dsb-128-r1", "kind": "plan", "variant": "dsb", "n": 128, "replicas": 1, "steps": 100,
         "jmax": 1, "density": 1.0, "fields": False, "state": True},
        # the reference program's own run (one aSB trial of 100 steps on a 2000-spin graph), the whole
        # call from host couplings to spins, as a caller that solves one graph makes it
        {"name": "asb-solve-2000-r1", "kind": "solve", "variant": "asb", "n": 2000, "replicas": 1, "steps": 100,
         "jmax": 1, "density": 1.0, "fields": False, "state": True},
        # the reference's published figures: 100 trials of 20 steps at N = 2048
        {"name": "asb-2048-r100", "kind": "plan", "variant": "asb", "n": 2048, "replicas": 100, "steps": 20,
         "jmax": 1, "density": 1.0, "fields": False, "state": True},
        # one long trajectory on the 2000-spin complete graph
        {"name": "dsb-2000-r1", "kind": "plan", "variant": "dsb", "n": 2000, "replicas": 1, "steps": 1000,
         "jmax": 1, "density": 1.0, "fields": False, "state": True},
        # the headline: 1024 trajectories of the same graph, 2000 steps; a caller keeps the best
        # spins and every trajectory's energy
        {"name": "dsb-2000-r1024", "kind": "plan", "variant": "dsb", "n": 2000, "replicas": 1024, "steps": 2000,
         "jmax": 1, "density": 1.0, "fields": False, "state": False},
        # a ragged instance with weights and fields: tiles are padded in both directions
        {"name": "dsb-1111-r300-fields", "kind": "plan", "variant": "dsb", "n": 1111, "replicas": 300, "steps": 1000,
         "jmax": 3, "density": 0.5, "fields": True, "state": True},
        # real couplings and fields, 256 trajectories: the split-operand contraction streams J from HBM
        {"name": "bsb-8192-r256-real", "kind": "plan", "variant": "bsb", "n": 8192, "replicas": 256, "steps": 200,
         "jmax": 0, "density": 1.0, "fields": True, "state": True},
        # many instances at once, sizes spread over [64, 4096], 64 trajectories each
        {"name": "batch-96", "kind": "batch", "count": 96, "nmin": 64, "nmax": 4096, "replicas": 64, "steps": 300,
         "jmax": 1},
        # a burst of served requests (J in {-8..8}, 32 trajectories, each its own step budget)
        {"name": "serve-16", "kind": "serve", "count": 16, "nmin": 128, "nmax": 4096, "replicas": 32, "smin": 500,
         "smax": 2000, "jmax": 8},
        # simulated quantum annealing at the reference program's size
        {"name": "sqa-4096-m64-r304", "kind": "sqa", "n": 4096, "trotter": 64, "replicas": 304, "steps": 8,
         "jmax": 1, "rng": "hash"},
        # the reference's NMFA call: one sample, N = 1024, 100 stages
        {"name": "nmfa-1024-s1", "kind": "nmfa", "n": 1024, "samples": 1, "stages": 100},
        # many samples of the same
        {"name": "nmfa-1024-s1024", "kind": "nmfa", "n": 1024, "samples": 1024, "stages": 100},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["plain", "plain", "tensor", "tensor", "real", "batch", "serve", "sqa", "nmfa"])
    if kind == "plain":  # few trajectories: the FP32 field
        variant = rng.choice(["asb", "bsb", "dsb"])
        jmax = 1 if variant == "asb" else rng.choice([0, 1, 1, 6])
        return {"kind": rng.choice(["plan", "plan", "solve"]), "variant": variant, "n": log(40, 3000),
                "replicas": log(1, 12), "steps": 20 if variant == "asb" else log(50, 1000), "jmax": jmax,
                "density": round(rng.uniform(0.1, 1.0), 3), "fields": variant != "asb" and rng.random() < 0.5,
                "state": True}
    if kind == "tensor":  # many trajectories, integer couplings
        n, r = log(65, 4096), log(32, 1024)
        while n * r > 1200000:
            n, r = log(65, 4096), log(32, 1024)
        return {"kind": "plan", "variant": "dsb", "n": n, "replicas": r, "steps": log(200, 2000),
                "jmax": rng.choice([1, 1, 4, 16, 100]), "density": round(rng.uniform(0.1, 1.0), 3),
                "fields": rng.random() < 0.5, "state": rng.random() < 0.5}
    if kind == "real":  # many trajectories, real couplings
        return {"kind": "plan", "variant": "bsb", "n": log(200, 6000), "replicas": log(32, 256), "steps": log(5, 12),
                "jmax": 0, "density": 1.0, "fields": rng.random() < 0.5, "state": True}
    if kind == "batch":
        return {"kind": "batch", "count": log(2, 48), "nmin": 64, "nmax": log(300, 4096), "replicas": log(8, 100),
                "steps": log(100, 300), "jmax": rng.choice([1, 1, 3, 9])}
    if kind == "serve":
        return {"kind": "serve", "count": log(2, 16), "nmin": 128, "nmax": log(300, 4096), "replicas": 32,
                "smin": 200, "smax": 1000, "jmax": rng.choice([1, 8])}
    if kind == "sqa":
        m = log(4, 64)
        return {"kind": "sqa", "n": log(150, 4096), "trotter": m, "replicas": log(4, 304), "steps": log(4, 8),
                "jmax": rng.choice([1, 1, 3]), "rng": rng.choice(["hash", "reference"])}
    return {"kind": "nmfa", "n": log(60, 1500), "samples": log(1, 1024), "stages": log(10, 100)}


# ---- inputs ----

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _couplings(n, jmax, density, seed):
    """Symmetric J with a zero diagonal, on the device: +-1 (jmax 1), integers in [-jmax, jmax], or
    N(0, 1/n) reals (jmax 0), each pair kept with probability density."""
    g = _generator(seed)
    if jmax == 0:
        w = torch.randn((n, n), generator=g, device=DEV) / math.sqrt(n)
    elif jmax == 1:
        w = (torch.randint(0, 2, (n, n), generator=g, device=DEV) * 2 - 1).float()
    else:
        w = torch.randint(-jmax, jmax + 1, (n, n), generator=g, device=DEV).float()
    if density < 1.0:
        w = w * (torch.rand((n, n), generator=g, device=DEV) < density)
    w = torch.triu(w, 1)
    return w + w.T


def _fields(n, jmax, seed):
    g = _generator(seed + 1000003)
    if jmax == 0:
        return torch.randn(n, generator=g, device=DEV) * math.sqrt(0.1)
    return torch.randint(-jmax, jmax + 1, (n,), generator=g, device=DEV).float()


def _problem(n, jmax, density, seed, fields=False):
    J = _couplings(n, jmax, density, seed).cpu().numpy()
    h = _fields(n, jmax, seed).cpu().numpy() if fields else None
    return sb.Problem.wrap(n, J.ctypes.data, h.ctypes.data if fields else 0, keepalive=(J, h))


def _nmfa_couplings(n, seed):
    """Edge probability 1/2, weight uniform in {-1, 0, +1}: the NMFA test graph's distribution."""
    g = _generator(seed)
    w = torch.randint(-1, 2, (n, n), generator=g, device=DEV).float()
    w = torch.triu(w * (torch.rand((n, n), generator=g, device=DEV) < 0.5), 1)
    return w + w.T


def _sizes(case):
    """(n, density, steps) of each instance: batch sizes spread evenly over [nmin, nmax], a burst's
    over their logarithm, densities and step budgets over their ranges, in a scattered order."""
    c = case["count"]
    out = []
    for k in range(c):
        u, v, w = (k + 0.5) / c, (k * 0.618034) % 1.0, (k * 0.754878) % 1.0
        if case["kind"] == "batch":
            out.append((int(case["nmin"] + u * (case["nmax"] - case["nmin"])), 0.05 + 0.95 * v, case["steps"]))
        else:
            n = int(case["nmin"] * (case["nmax"] / case["nmin"]) ** u)
            out.append((n, 0.01 + 0.99 * v, int(case["smin"] + w * (case["smax"] - case["smin"]))))
    return [out[(k * 7) % c] if c % 7 else out[k] for k in range(c)]


def prepare(case, seed):
    kind = case["kind"]
    # the context works on its own stream, as a program without one gives it
    ctx = sb.Context(0)
    s = {"case": case, "ctx": ctx}
    if kind in ("plan", "solve"):
        s["problem"] = _problem(case["n"], case["jmax"], case["density"], seed, case["fields"])
        init = sb.INIT_REFERENCE if case["variant"] == "asb" else sb.INIT_UNIFORM
        s["params"] = sb.Params.default(VARIANT[case["variant"]], steps=case["steps"], replicas=case["replicas"],
                                        seed=seed, init_mode=init)
        if kind == "plan":
            s["plan"] = ctx.plan(s["problem"], s["params"], want_state=case["state"])
    elif kind == "batch":
        s["params"] = sb.Params.default(sb.DSB, steps=case["steps"], replicas=case["replicas"], seed=seed)
        probs = [_problem(n, case["jmax"], d, seed * 1009 + k) for k, (n, d, _) in enumerate(_sizes(case))]
        s["batch"] = ctx.batch(probs, s["params"])
    elif kind == "serve":
        s["requests"] = []
        for k, (n, d, steps) in enumerate(_sizes(case)):
            prm = sb.Params.default(sb.DSB, steps=steps, replicas=case["replicas"], seed=seed + k)
            s["requests"].append((_problem(n, case["jmax"], d, seed * 1009 + k), prm))
    elif kind == "sqa":
        s["problem"] = _problem(case["n"], case["jmax"], 1.0, seed)
        mode = sb.SQA_RNG_HASH if case["rng"] == "hash" else sb.SQA_RNG_REFERENCE
        s["params"] = sb.SqaParams.default(trotter=case["trotter"], steps=case["steps"], replicas=case["replicas"],
                                           rng_mode=mode, seed=seed)
    else:
        J = _nmfa_couplings(case["n"], seed).cpu().numpy()
        s["problem"] = sb.Problem.wrap(case["n"], J.ctypes.data, keepalive=J)
        s["params"] = sb.NmfaParams.default(samples=case["samples"], stages=case["stages"], seed=seed & 0x7FFFFFFF)
    return s


# ---- one pass ----

def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind in ("plan", "solve"):
        r = state["plan"].run() if kind == "plan" else ctx.solve(state["problem"], state["params"],
                                                                want_state=case["state"])
        out = {"best_spins": r.best_spins, "energies": r.replica_energies, "best_energy": r.best_energy}
        if case["state"]:
            out["x"], out["y"] = r.final_x, r.final_y
        return out
    if kind == "batch":
        res = state["batch"].run()
        return {"best_spins": np.concatenate([r.best_spins for r in res]),
                "energies": np.stack([r.replica_energies for r in res])}
    if kind == "serve":
        tickets = [ctx.submit(p, prm) for p, prm in state["requests"]]
        res = [ctx.poll(t, p.n, prm, wait_ms=-1) for t, (p, prm) in zip(tickets, state["requests"])]
        return {"best_spins": np.concatenate([r.best_spins for r in res]),
                "energies": np.stack([r.replica_energies for r in res])}
    if kind == "sqa":
        r = ctx.sqa_solve(state["problem"], state["params"], want_spins=False)
        return {"best_spins": r.best_spins, "energies": r.replica_energies}
    r = ctx.nmfa_solve(state["problem"], state["params"], want_states=True)
    return {"samples": r.samples, "energies": r.energies, "states": r.states}


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        sizes = _sizes(case)
        r = case["replicas"]
        return {"bytes": sum(4.0 * n * n + n + 8 * r for n, _, _ in sizes),
                "flops": sum(2.0 * n * n * r * steps for n, _, steps in sizes)}
    n = case["n"]
    if kind == "sqa":
        updates = case["replicas"] * case["trotter"] * (n + case["trotter"] - 1.0) * case["steps"]
        return {"bytes": 4.0 * n * n + n + 8 * case["replicas"], "flops": 2.0 * n * updates}
    if kind == "nmfa":
        r = case["samples"]
        return {"bytes": 4.0 * n * n + (5.0 * n + 8) * r, "flops": 2.0 * n * n * r * 2 * case["stages"]}
    r = case["replicas"]
    return {"bytes": 4.0 * n * n + n + 8 * r + (8.0 * n * r if case["state"] else 0),
            "flops": 2.0 * n * n * r * case["steps"]}


# ---- 64-bit values ----

def _uniform_start(n, r, seed):
    """x, y uniform in [-0.1, 0.1) from the counter hash of (seed, trajectory, spin)."""
    e = np.arange(2 * n * r, dtype=np.uint64)
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + np.uint64(0x9E3779B97F4A7C15) * (e + np.uint64(1))
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
    f = (z >> np.uint64(40)).astype(np.float32) * np.float32(2.0 ** -24)
    v = ((f * np.float32(2) - np.float32(1)) * np.float32(0.1)).astype(np.float64).reshape(r, n, 2)
    return v[..., 0].copy(), v[..., 1].copy()


def _trial_start(n, r):
    """The reference's start: per-spin xorshift32 seeded with the spin's index, values in [0, 0.1)."""
    st = np.arange(n, dtype=np.uint32)
    out = []
    for _ in range(2 * r):
        st = st ^ (st << np.uint32(13))
        st = st ^ (st >> np.uint32(17))
        st = st ^ (st << np.uint32(5))
        out.append((st.astype(np.float32) / np.float32(4294967296.0)).astype(np.float64) / 10.0)
    v = np.stack(out).astype(np.float32).astype(np.float64).reshape(r, 2, n)
    return v[:, 0].copy(), v[:, 1].copy()


def _energies(J, h, s):
    e = -0.5 * (s * (s @ J)).sum(1)
    return e if h is None else e - s @ h


def _exact_sb(case, seed):
    n, r, steps = case["n"], case["replicas"], case["steps"]
    J = _couplings(n, case["jmax"], case["density"], seed).double()
    h = _fields(n, case["jmax"], seed).double() if case["fields"] else None
    asb = case["variant"] == "asb"
    x, y = (torch.from_numpy(v).to(DEV) for v in (_trial_start(n, r) if asb else _uniform_start(n, r, seed)))
    if asb:
        kick = 0.01565
        for t in range(steps):
            p = t / steps
            for _ in range(2):
                x = x + y * 0.5
                y = y - 0.5 * (x * x * x + (1.0 - p) * x)
            y = y + kick * (x @ J)
    else:
        cnt = n * (n - 1.0)
        mean = J.sum().item() / cnt
        std = math.sqrt(max((J * J).sum().item() / cnt - mean * mean, 0.0))
        c0 = 0.5 / (math.sqrt(n) * (std if std > 0 else 1.0))
        for t in range(steps):
            f = x @ J
            if h is not None:
                f = f + h
            y = y + 1.25 * (c0 * f - (1.0 - t / steps) * x)
            x = x + 1.25 * y
            out = x.abs() > 1.0
            x = torch.where(out, torch.sign(x), x)
            y = torch.where(out, torch.zeros_like(y), y)
    e = _energies(J, h, torch.where(x > 0, 1.0, -1.0).double())
    res = {"best_spins": None, "energies": e, "best_energy": e.min().item()}
    if case["state"]:
        res["x"], res["y"] = x, y
    return res


def _exact_nmfa(case, seed):
    n, r, stages = case["n"], case["samples"], case["stages"]
    mask = 0xFFFFFFFF
    J = _nmfa_couplings(n, seed).double()
    rows = J.abs().sum(1)
    norm = torch.where(rows > 0, -1.0 / torch.sqrt(rows.clamp(min=1e-300)), torch.zeros_like(rows))
    idx = (torch.arange(r, device=DEV)[:, None] * n + torch.arange(n, device=DEV)[None, :] + (seed & 0x7FFFFFFF)) & mask
    w, t = [], idx
    for _ in range(4):
        t = t ^ ((t << 13) & mask)
        t = t ^ (t >> 17)
        t = t ^ ((t << 5) & mask)
        w.append(t)
    count = 0

    def word():
        nonlocal w, count
        t = w[3]
        t = t ^ (t >> 2)
        t = t ^ ((t << 1) & mask)
        t = t ^ w[0] ^ ((w[0] << 4) & mask)
        w = [t, w[0], w[1], w[2]]
        count = (count + 362437) & mask
        return (t + count) & mask

    s = torch.zeros((r, n), dtype=torch.float64, device=DEV)
    beta, step = np.float32(1 / 16), np.float32((8 - 1 / 16) / stages)
    for _ in range(stages):
        a, b = word().double(), word().double()
        rad = torch.sqrt(-2.0 * torch.log(a / 2.0 ** 32)) * 0.15
        ang = 2 * math.pi * b / 2.0 ** 32
        for z in (torch.sin(ang) * rad, torch.cos(ang) * rad):
            s = 0.85 * s + 0.15 * torch.tanh(float(beta) * ((s @ J) * norm + z))
        beta = np.float32(beta + step)
    e = -_energies(J, None, torch.where(s > 0, 1.0, -1.0).double())
    return {"samples": None, "energies": e, "states": s}


def exact(case, seed):
    """64-bit values where the trajectory is short enough to follow one: real-valued SB of few steps
    and NMFA. Longer SB trajectories (and every dSB and SQA one) decide signs at each step, so that a
    64-bit run is another trajectory: theirs is checked by equal spins and energies instead."""
    if case["kind"] == "nmfa":
        return _exact_nmfa(case, seed)
    if case["kind"] in ("plan", "solve") and case["steps"] <= {"asb": 24, "bsb": 12, "dsb": 0}[case["variant"]]:
        return _exact_sb(case, seed)
    return None
