"""The work that users of the propagator have it do, as cases for timing.

A case names a family (which public entry point is called) and its sizes:

  call       propagateGPUAtomic, the reference's Python call: host arrays in,
             lists out, everything uploaded and freed in the call
  once       gdp.propagate: the same work, numpy arrays in and out
  resident   Context.propagate: the matrix stays on the GPU, bounds in host memory
  device     Context.propagate_device: the bounds are device tensors too
  nodes      Batch.nodes: branch-and-bound children of one problem's fixpoint
  instances  Batch.instances: many problems at once
  chains     Batch.instances on chain MIPs, which take thousands of rounds
  noalloc    propagate_noalloc: every array is a device tensor of the caller
  forward    Mlp.forward: scores of row features
  train      Mlp.train: a marking model from traces of propagations

Infinite bounds are +-inf, as read_mps gives them. Propagations return the
bounds, the round count and the verdict.
"""
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "gpu-domain-propagator_gb300"))

import gdp  # noqa: E402
import gdpgen  # noqa: E402

CHAIN_ROUNDS = 10_000  # round cap of chain MIPs: every member reaches its fixpoint
PROPAGATIONS = ("call", "once", "resident", "device", "nodes", "instances", "chains", "noalloc")


def listed():
    return [
        # the smallest call: a solver's subproblem through the reference's interface (its default driver)
        {"name": "call_tiny", "family": "call", "gen": "small", "m": 100, "driver": gdp.CPU_LOOP},
        # one-shot propagation of an ordinary MIP from host arrays
        {"name": "once_ordinary", "family": "once", "gen": "powerlaw", "m": 100_000, "driver": gdp.MEGAKERNEL},
        # repeated propagation of a small resident MIP: a tree search's node after node
        {"name": "resident_small", "family": "resident", "gen": "small", "m": 2_000, "driver": gdp.MEGAKERNEL},
        # an ordinary resident MIP with the library's default driver (host loop), odd sizes
        {"name": "device_host_loop", "family": "device", "gen": "powerlaw", "m": 60_001, "driver": gdp.CPU_LOOP},
        # covering / knapsack rows, binaries mostly, few rounds, the graph driver
        {"name": "device_cover", "family": "device", "gen": "cover", "m": 110_000, "driver": gdp.GPU_LOOP},
        # the benchmark's MIP: 2M rows, 48M non-zeros, rows of up to 100,000
        {"name": "device_large", "family": "device", "gen": "powerlaw", "m": 2_000_000, "driver": gdp.MEGAKERNEL},
        # a frontier of branch-and-bound nodes of one MIP
        {"name": "nodes_frontier", "family": "nodes", "m": 50_000, "members": 64},
        # a mixed bag of MIPs, as a benchmark set or a restart portfolio gives
        {"name": "instances_mixed", "family": "instances", "m": 60_000, "members": 24},
        # chains: thousands of rounds with little work each
        {"name": "chains_long", "family": "chains", "m": 25_000, "members": 8},
        # a caller with its own memory pool: nothing is allocated, rows of up to 20,000 non-zeros
        {"name": "noalloc_ordinary", "family": "noalloc", "gen": "powerlaw", "m": 100_000},
        # scores of the rows of a large MIP
        {"name": "mlp_forward", "family": "forward", "samples": 1_000_000},
        # the marking model's training run on traced rows, minibatches of 8,192
        {"name": "mlp_train", "family": "train", "samples": 200_000, "batch": 8_192, "epochs": 4},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    family = rng.choice(PROPAGATIONS + ("forward", "train"))
    driver = rng.choice((gdp.CPU_LOOP, gdp.GPU_LOOP, gdp.MEGAKERNEL))
    gen = rng.choice(("small", "powerlaw", "powerlaw", "cover"))
    if family == "call":
        return {"family": family, "gen": gen, "m": _log(rng, 40, 20_000), "driver": driver}
    if family == "once":
        return {"family": family, "gen": gen, "m": _log(rng, 1_000, 500_000), "driver": driver}
    if family == "resident":
        return {"family": family, "gen": gen, "m": _log(rng, 40, 300_000), "driver": driver}
    if family == "device":
        return {"family": family, "gen": gen, "m": _log(rng, 1_000, 1_500_000), "driver": driver}
    if family == "nodes":
        return {"family": family, "m": _log(rng, 2_000, 100_000), "members": rng.randint(4, 96)}
    if family == "instances":
        return {"family": family, "m": _log(rng, 2_000, 200_000), "members": rng.randint(2, 32)}
    if family == "chains":
        return {"family": family, "m": _log(rng, 2_000, 50_000), "members": rng.randint(1, 12)}
    if family == "noalloc":
        return {"family": family, "gen": gen, "m": _log(rng, 200, 400_000)}
    if family == "forward":
        return {"family": family, "samples": _log(rng, 500, 2_000_000)}
    return {"family": family, "samples": _log(rng, 2_000, 300_000), "batch": _log(rng, 512, 16_384),
            "epochs": rng.randint(1, 6)}


# ---- inputs ------------------------------------------------------------------

def _infinite(mip):
    for a in (mip.lb, mip.ub, mip.lhs, mip.rhs):
        a[a >= 1e20] = np.inf
        a[a <= -1e20] = -np.inf
    return mip


def _generate(gen, m, seed):
    if gen == "cover":  # ten covering rows to one knapsack row
        knap = max(1, m // 11)
        return _infinite(gdpgen.cover_knapsack(m - knap, knap, max(70, 8 * m // 11), max(70, m // 11), seed=seed))
    n = max(30, 3 * m // 4)
    if gen == "small":
        return _infinite(gdpgen.random_mip(0, seed=seed, m=m, n=n))
    dense = 32 if m >= 1_000_000 else 0
    return _infinite(gdpgen.random_mip(1, seed=seed, m=m, n=n, n_dense_rows=dense))


def _members(case, seed):
    """The MIPs of an instance batch: row counts spread over a factor of 50 (chains: of 4) below case["m"],
    the same for every seed."""
    k, rng = case["members"], np.random.default_rng(case["m"])
    if case["family"] == "chains":
        ms = case["m"] * np.exp(-rng.random(k) * np.log(4.0))
        return [_infinite(gdpgen.chains(int(m), chain_max=2_000, seed=seed * 1000 + i)) for i, m in enumerate(ms)]
    ms = case["m"] * np.exp(-rng.random(k) * np.log(50.0))
    return [_generate("powerlaw", int(m), seed * 1000 + i) for i, m in enumerate(ms)]


def _node_bounds(mip, lb, ub, count, seed):
    """Children of the fixpoint (lb, ub): up to 50 integer variables fixed to a value of their domain."""
    rng = np.random.default_rng(seed)
    ints = np.flatnonzero((mip.vartype != 3) & (ub - lb >= 1) & (np.abs(lb) < 1e19) & (np.abs(ub) < 1e19))
    lbs, ubs = [], []
    for _ in range(count):
        l, u = lb.copy(), ub.copy()
        fix = rng.choice(ints, size=min(len(ints), int(rng.integers(1, 51))), replace=False)
        l[fix] = u[fix] = np.minimum(np.floor(l[fix] + rng.random(len(fix)) * (u[fix] - l[fix] + 1)), u[fix])
        lbs.append(l)
        ubs.append(u)
    return lbs, ubs


def _features(case, seed):
    """Row features as traces hold them: lengths, slacks, flags and ages in [0, 1], and labels that depend on them."""
    n, rng = case["samples"], np.random.default_rng(seed)
    x = rng.random((n, gdp.MLP_FEATURES), dtype=np.float32)
    x[:, 0] = np.log2(1.0 + np.minimum(rng.zipf(1.8, n), 20_000)) / 16.0
    x[:, 5:8] = x[:, 5:8] < 0.3
    x[:, 13:16] = x[:, 13:16] < 0.5
    y = (x[:, 3] + 0.5 * x[:, 8] - x[:, 0] + 0.3 * rng.standard_normal(n, dtype=np.float32) > 0.6).astype(np.float32)
    return x, y, np.where(y > 0.5, 2.0, 0.7).astype(np.float32)


def _parameters(seed):
    """He-uniform weights of the 16-64-64-1 model, in the library's parameter order."""
    rng = np.random.default_rng(seed)
    u = lambda count, fan: rng.uniform(-1, 1, count) * np.sqrt(6.0 / fan)  # noqa: E731
    return np.concatenate([u(64 * 16, 16), np.zeros(64), u(64 * 64, 64), np.zeros(64), u(64, 64),
                           np.zeros(1)]).astype(np.float32)


def prepare(case, seed):
    family = case["family"]
    if family in ("forward", "train"):
        x, y, w = _features(case, seed)
        model = gdp.Mlp(seed=1)
        p = _parameters(seed)
        model.params = p
        return {"case": case, "model": model, "params": p, "x": x, "y": y, "w": w}
    if family in ("instances", "chains"):
        mips = _members(case, seed)
        batch = gdp.Batch.instances(mips, max_rounds=CHAIN_ROUNDS if family == "chains" else 0)
        return {"case": case, "batch": batch, "lbs": [p.lb for p in mips], "ubs": [p.ub for p in mips]}
    if family == "nodes":
        mip = _generate("powerlaw", case["m"], seed)
        ctx = gdp.Context(mip, sync_type=gdp.MEGAKERNEL)
        lb, ub, _ = ctx.propagate()
        lbs, ubs = _node_bounds(mip, lb, ub, case["members"], seed)
        return {"case": case, "ctx": ctx, "batch": gdp.Batch.nodes(ctx, case["members"]), "lbs": lbs, "ubs": ubs}
    mip = _generate(case["gen"], case["m"], seed)
    if family in ("call", "once"):
        return {"case": case, "mip": mip}
    if family == "resident":
        return {"case": case, "mip": mip, "ctx": gdp.Context(mip, sync_type=case["driver"])}
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    state = {"case": case, "lb0": dev(mip.lb), "ub0": dev(mip.ub), "lb": dev(mip.lb), "ub": dev(mip.ub)}
    if family == "device":
        return {**state, "ctx": gdp.Context(mip, sync_type=case["driver"])}
    return {**state, "sizes": (mip.m, mip.n, mip.nnz), "col": dev(mip.col), "row_ptr": dev(mip.row_ptr),
            "val": dev(mip.val), "lhs": dev(mip.lhs), "rhs": dev(mip.rhs), "vartype": dev(mip.vartype)}


# ---- one pass ------------------------------------------------------------------

def _answer(lb, ub, st):
    return {"lb": lb, "ub": ub, "rounds": int(st["rounds"]), "infeasible": int(bool(st["infeasible"]))}


def run(state):
    case = state["case"]
    family = case["family"]
    if family == "call":
        p = state["mip"]
        lb, ub = gdp.propagateGPUAtomic(p.n, p.m, p.nnz, p.col, p.row_ptr, p.val, p.lhs, p.rhs, p.lb, p.ub,
                                        p.vartype, case["driver"])
        return {"lb": np.array(lb), "ub": np.array(ub)}
    if family == "once":
        return _answer(*gdp.propagate(state["mip"], sync_type=case["driver"]))
    if family == "resident":
        return _answer(*state["ctx"].propagate())
    if family in ("nodes", "instances", "chains"):
        lbs, ubs, sts, _ = state["batch"].propagate(state["lbs"], state["ubs"])
        return {"lb": np.concatenate(lbs), "ub": np.concatenate(ubs),
                "rounds": np.array([s["rounds"] for s in sts]), "infeasible": np.array([s["infeasible"] for s in sts])}
    if family == "forward":
        return state["model"].forward(state["x"])
    if family == "train":
        model = state["model"]
        model.params = state["params"]
        loss = model.train(state["x"], state["y"], state["w"], epochs=case["epochs"], batch=case["batch"], lr=2e-3,
                           seed=3)
        return {"params": model.params, "loss": loss}
    lb, ub = state["lb"].copy_(state["lb0"]), state["ub"].copy_(state["ub0"])
    stream = torch.cuda.current_stream().cuda_stream
    if family == "device":
        return _answer(lb, ub, state["ctx"].propagate_device(lb.data_ptr(), ub.data_ptr(), stream))
    at = [state[k].data_ptr() for k in ("col", "row_ptr", "val", "lhs", "rhs", "lb", "ub", "vartype")]
    return _answer(lb, ub, gdp.propagate_noalloc(*state["sizes"], *at, stream=stream))


# ---- what a pass cannot do without ----------------------------------------------

def _pass_work(m, n, nnz):
    """The CSR and the row sides once, the bounds in and out and the types; the activities of every row once."""
    return 12.0 * nnz + 20.0 * m + 36.0 * n, 4.0 * nnz


def work(case):
    family = case["family"]
    if family == "forward":
        n = case["samples"]
        return {"bytes": 68.0 * n, "flops": 2.0 * n * (16 * 64 + 64 * 64 + 64)}
    if family == "train":
        n = case["samples"]
        return {"bytes": 72.0 * n, "flops": 6.0 * n * case["epochs"] * (16 * 64 + 64 * 64 + 64)}
    if family in ("instances", "chains"):
        each = [_pass_work(p.m, p.n, p.nnz) for p in _members(case, 0)]
        return {"bytes": sum(e[0] for e in each), "flops": sum(e[1] for e in each)}
    p = _generate(case.get("gen", "powerlaw"), case["m"], 0)
    b, f = _pass_work(p.m, p.n, p.nnz)
    if family == "nodes":  # one matrix; the bounds of every node in and out, and the difference to the root read
        b += 48.0 * p.n * (case["members"] - 1)
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits ---------------------------------------------------------

EPS, INF, FEASTOL = 1e-9, 1e20, 1e-6


def _eps_max(d):
    """The largest term as a sequential scan finds it that takes a term only when it is larger by more than EPS."""
    best = 0.0
    for v in d:
        if v - best > EPS:
            best = v
    return best


def _crossed(lb, ub):
    return bool(np.any(lb - ub > FEASTOL * np.maximum(1.0, np.maximum(np.abs(lb), np.abs(ub)))))


def _beyond(act, count, side, sign):
    ok = (count == 0) & np.isfinite(side) & (np.abs(side) < INF)
    tol = FEASTOL * np.maximum(1.0, np.maximum(np.abs(act[ok]), np.abs(side[ok])))
    return bool(np.any(sign * (act[ok] - side[ok]) > tol))


@np.errstate(invalid="ignore", over="ignore")
def _fixpoint(mip, lb, ub, max_rounds=100):
    """Rounds of bound propagation from (lb, ub), each from the round-start bounds of the one before."""
    lb, ub = lb.copy(), ub.copy()
    m, col, a = mip.m, mip.col, mip.val
    rp = mip.row_ptr.astype(np.int64)
    filled = np.flatnonzero(np.diff(rp))
    rows = np.repeat(np.arange(m), np.diff(rp))
    cont, pos, gt0 = (mip.vartype == 3)[col], a > EPS, a > 0
    rounds, bad, change = 0, _crossed(lb, ub), True
    while change and not bad and rounds < max_rounds:
        rounds += 1
        l, u = lb[col], ub[col]
        lo, hi = l <= -INF, u >= INF
        imin, imax = np.where(pos, lo, hi), np.where(pos, hi, lo)
        minact = np.bincount(rows, np.where(imin, 0.0, a * np.where(gt0, l, u)), m)
        maxact = np.bincount(rows, np.where(imax, 0.0, a * np.where(gt0, u, l)), m)
        nmin, nmax = np.bincount(rows, imin, m).astype(int), np.bincount(rows, imax, m).astype(int)
        delta = np.abs(a) * (u - l)
        top = np.zeros(m)
        top[filled] = np.maximum(np.maximum.reduceat(delta, rp[:-1][filled]), 0.0)
        slack = np.minimum(mip.rhs - minact, maxact - mip.lhs)
        go = np.where(top < INF, top - slack > EPS, True)
        for r in np.flatnonzero(go & (top < INF) & (top - slack <= 2.1e-9)):
            go[r] = _eps_max(delta[rp[r]:rp[r + 1]]) - slack[r] > EPS
        go &= ~((nmin > 1) & (nmax > 1)) & (np.diff(rp) > 0)
        bad = _beyond(minact, nmin, mip.rhs, 1.0) or _beyond(maxact, nmax, mip.lhs, -1.0)
        e = np.flatnonzero(go[rows])
        r, c, ae, le, ue, up = rows[e], col[e], a[e], l[e], u[e], gt0[e]
        s_hi, s_lo = (mip.rhs - minact)[r], (mip.lhs - maxact)[r]
        rhs_side = (mip.rhs[r] < INF) & (minact[r] > -INF) & (delta[e] - s_hi > EPS)
        lhs_side = (mip.lhs[r] > -INF) & (maxact[r] < INF) & (delta[e] + s_lo > EPS)
        nu, nl = np.where(up, nmin[r], nmax[r]), np.where(up, nmax[r], nmin[r])
        new_u = np.where(up, s_hi, s_lo) / ae + np.where(nu == 0, le, 0.0)
        new_l = np.where(up, s_lo, s_hi) / ae + np.where(nl == 0, ue, 0.0)
        new_u = np.where(cont[e], new_u, np.floor(new_u + EPS))
        new_l = np.where(cont[e], new_l, np.ceil(new_l - EPS))
        tu = np.where(up, rhs_side, lhs_side) & ((nu == 0) | ((nu == 1) & (le <= -INF))) & (new_u - ue < -EPS)
        tl = np.where(up, lhs_side, rhs_side) & ((nl == 0) | ((nl == 1) & (ue >= INF))) & (new_l - le > EPS)
        change = bool(tu.any() or tl.any())
        np.minimum.at(ub, c[tu], new_u[tu])
        np.maximum.at(lb, c[tl], new_l[tl])
        bad = bad or _crossed(lb, ub)
    return lb, ub, {"rounds": rounds, "infeasible": bad}


def _logits(x, p):
    """Pre-activations and activations of the model in 64 bits."""
    w1, b1, w2, b2 = p[:1024].view(64, 16), p[1024:1088], p[1088:5184].view(64, 64), p[5184:5248]
    a1 = x @ w1.T + b1
    a2 = a1.clamp(min=0) @ w2.T + b2
    return a1, a2, a2.clamp(min=0) @ p[5248:5312] + p[5312]


def _splitmix(s):
    mask = (1 << 64) - 1
    s = (s + 0x9E3779B97F4A7C15) & mask
    z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
    return s, z ^ (z >> 31)


def _trained(case, x, y, w, p):
    """Adam over the shuffled minibatches of Mlp.train."""
    n, batch, s = len(y), case["batch"], 3
    perm = list(range(n))
    for i in range(n - 1, 0, -1):
        s, z = _splitmix(s)
        j = z % (i + 1)
        perm[i], perm[j] = perm[j], perm[i]
    order = torch.tensor(perm, device=x.device)
    x, y, w = x[order], y[order], w[order]
    m1, m2, step, nb = torch.zeros_like(p), torch.zeros_like(p), 0, (n + batch - 1) // batch
    for _ in range(case["epochs"]):
        s, z = _splitmix(s)
        rot, loss = z % nb, 0.0
        for b in range(nb):
            part = slice((b + rot) % nb * batch, min(n, ((b + rot) % nb + 1) * batch))
            xb, yb, wb = x[part], y[part], w[part]
            q = p.clone().requires_grad_()
            each = torch.nn.functional.binary_cross_entropy_with_logits(_logits(xb, q)[2], yb, reduction="none")
            total = (wb * each).sum()
            g, = torch.autograd.grad(total / wb.sum(), q)
            loss += float(total)
            step += 1
            m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
            p = p - 2e-3 * (m1 / (1 - 0.9 ** step)) / ((m2 / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return {"params": p.cpu().numpy(), "loss": loss / float(w.sum())}


def exact(case, seed):
    family = case["family"]
    if family in ("forward", "train"):
        x, y, w = (torch.from_numpy(a).cuda().double() for a in _features(case, seed))
        p = torch.from_numpy(_parameters(seed)).cuda().double()
        return _logits(x, p)[2].cpu().numpy() if family == "forward" else _trained(case, x, y, w, p)
    if family == "chains":
        return None  # thousands of rounds
    if family == "instances":
        mips = _members(case, seed)
        if sum(p.nnz for p in mips) > 1_500_000:
            return None
        got = [_fixpoint(p, p.lb, p.ub) for p in mips]
    else:
        mip = _generate(case.get("gen", "powerlaw"), case["m"], seed)
        if mip.nnz * case.get("members", 1) > 1_500_000:
            return None
        got = [_fixpoint(mip, mip.lb, mip.ub)]
        if family == "nodes":
            got = [_fixpoint(mip, l, u) for l, u in zip(*_node_bounds(mip, *got[0][:2], case["members"], seed))]
    if family in ("nodes", "instances"):
        return {"lb": np.concatenate([g[0] for g in got]), "ub": np.concatenate([g[1] for g in got]),
                "rounds": np.array([g[2]["rounds"] for g in got]),
                "infeasible": np.array([int(g[2]["infeasible"]) for g in got])}
    lb, ub, st = got[0]
    return {"lb": lb, "ub": ub} if family == "call" else _answer(lb, ub, st)
