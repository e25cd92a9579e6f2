"""Work that users of the framework have it do, as cases that can be timed and compared.

Every case is one pass through public entry points:

run        a whole simulation on a plain field: objects set from device
           records, lazy_update, `steps` steps, the read buffer read back
frame      one step of a running flock and its state (a program that shows or
           couples every step)
agents     what one rank of a flock spread over column strips does per step:
           records set, lazy_update, read buffer, next states of its agents
neighbors  a program with its own agents asks for the neighbours of many points
sweep      an exploration: a batch of replicas made, stepped and read back
serve      a group of requests through the continuous-batching server

Flocks are seeded and synthetic: uniform, or Gaussian clusters.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import krabmaga_gb300 as kg

DEV = "cuda"
ARITH = {"fast": kg.KB_ARITH_FAST, "strict": kg.KB_ARITH_STRICT}
QUERY = {"relax": kg.KB_QUERY_RELAX, "exact": kg.KB_QUERY_EXACT}
SIGMA = 40.0  # of a cluster, as the clustered benchmark flock has it


def _flock(kind, n, steps=1, density=0.025, ratio=1.5, arith="fast", query="relax", clusters=0):
    """ratio: the neighbour radius (10) over the bag size: 1.5 in the benchmark's
    flocks, 20 with the model's own default bag of 0.5."""
    return {"kind": kind, "n": n, "steps": steps, "density": density, "ratio": ratio, "arith": arith,
            "query": query, "clusters": clusters}


def listed():
    return [
        # the smallest call: one step of the reference's 1,000-bird flock (fast
        # arithmetic) and its state, as a viewer asks for it
        {"name": "frame_1k", **_flock("frame", 1000)},
        # the reference's 1,000-bird run of 200 steps, with the default (strict) arithmetic
        {"name": "run_1k_strict", **_flock("run", 1000, 200, arith="strict")},
        # the same flock as Flocker makes it by default: bags of 0.5, so a query
        # spans 41 x 41 bags and a move may cross more than one
        {"name": "run_1k_small_bags", **_flock("run", 1000, 50, ratio=20.0, arith="strict")},
        # an ordinary flock, an odd number of birds
        {"name": "run_20k", **_flock("run", 20011, 100)},
        # the exact distance query in strict arithmetic
        {"name": "run_65k_exact", **_flock("run", 65537, 50, arith="strict", query="exact")},
        # the headline flock: 1,048,576 birds, density 0.025
        {"name": "run_1m", **_flock("run", 1 << 20, 100)},
        # the headline flock in the default arithmetic, a short run
        {"name": "run_1m_strict", **_flock("run", 1 << 20, 20, arith="strict")},
        # the largest: 4,194,304 birds in 256 clusters (torus side 12952)
        {"name": "clustered_4m", **_flock("run", 1 << 22, 10, clusters=256)},
        # one rank's part of a flock spread over ranks
        {"name": "agents_262k", **_flock("agents", 262147)},
        # neighbour lists of 200,000 points in a 1M flock
        {"name": "neighbors_200k", **_flock("neighbors", 1 << 20, query="exact"), "points": 200003},
        # an exploration of 64 replicas, 500 steps each
        {"name": "sweep_64", "kind": "sweep", "nrep": 64, "n_min": 1024, "n_max": 65536, "steps": 500},
        # a group of 32 requests of the served stream
        {"name": "serve_32", "kind": "serve", "requests": 32, "n_min": 1024, "n_max": 65536,
         "steps_min": 100, "steps_max": 400},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "frame", "agents", "neighbors", "sweep", "serve"])
    arith = rng.choice(["fast", "fast", "strict"])
    query = rng.choice(["relax", "relax", "relax", "exact"])
    density = round(math.exp(rng.uniform(math.log(0.01), math.log(0.06))), 4)
    if kind == "run":
        shape = rng.choice(["uniform", "uniform", "uniform", "clustered", "fine"])
        if shape == "fine":  # small bags: wide rings of them, or rings of three
            ratio = rng.choice([3.0, 20.0])
            return _flock(kind, _log(rng, 500, 20000), rng.randint(10, 50), density, ratio, arith, query)
        if shape == "clustered":
            n = _log(rng, 30000, 1 << 20)
            return _flock(kind, n, rng.randint(4, 10), clusters=max(1, n // 16384), arith=arith, query=query)
        n = _log(rng, 300, 1 << 20)
        return _flock(kind, n, rng.randint(10, 100 if n < 300000 else 40), density, 1.5, arith, query)
    if kind == "frame":
        return _flock(kind, _log(rng, 300, 1 << 18), 1, density, 1.5, arith, query)
    if kind == "agents":
        return _flock(kind, _log(rng, 3000, 1 << 20), 1, density, 1.5, arith, query)
    if kind == "neighbors":
        n = _log(rng, 10000, 1 << 20)
        return {**_flock(kind, n, 1, density, 1.5, arith, query), "points": _log(rng, 1000, 200000)}
    if kind == "sweep":
        return {"kind": "sweep", "nrep": rng.randint(8, 64), "n_min": _log(rng, 256, 2048),
                "n_max": _log(rng, 8192, 65536), "steps": rng.randint(100, 500)}
    return {"kind": "serve", "requests": rng.randint(4, 32), "n_min": _log(rng, 512, 2048),
            "n_max": _log(rng, 8192, 65536), "steps_min": rng.randint(50, 100), "steps_max": rng.randint(150, 400)}


# ---------------------------------------------------------------- inputs
def _geometry(case):
    """Torus side and bag size of a flock case, as f32 values."""
    n = case["n"]
    if case["clusters"]:
        side = 12952.0 * math.sqrt(n / (1 << 22))
    else:
        side = math.sqrt(n / case["density"])
    return float(np.float32(side)), float(np.float32(10.0) / np.float32(case["ratio"]))


def _birds(case, seed):
    """(ids int32, records float32 [n, 4] {x, y, dx, dy}) on the GPU."""
    n = case["n"]
    side, _ = _geometry(case)
    g = torch.Generator(device=DEV).manual_seed(1_000_003 * (seed % 1_000_003) + 17)
    if case["clusters"]:
        c = torch.rand((case["clusters"], 2), generator=g, device=DEV) * side
        of = torch.randint(case["clusters"], (n,), generator=g, device=DEV)
        xy = torch.remainder(c[of] + SIGMA * torch.randn((n, 2), generator=g, device=DEV), side)
    else:
        xy = torch.rand((n, 2), generator=g, device=DEV) * side
    xy = xy.clamp_(0.0, side * (1.0 - 1e-6))
    a = torch.rand((n,), generator=g, device=DEV) * (2.0 * math.pi)
    st = torch.cat([xy, torch.cos(a)[:, None], torch.sin(a)[:, None]], 1).contiguous()
    return torch.arange(n, dtype=torch.int32, device=DEV), st


def _params(case, seed):
    return kg.FlockParams(seed=seed, arith=ARITH[case["arith"]], query_mode=QUERY[case["query"]])


def _mean_n(case):
    lo, hi = case["n_min"], max(case["n_max"], case["n_min"] + 1)
    return (hi - lo) / math.log(hi / lo)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        # the benchmark's table (sizes, weights, radii), the flocks from the seed
        replicas = kg.sweep_replicas(case["nrep"], case["n_min"], case["n_max"])
        for i, r in enumerate(replicas):
            r.params.seed = 1000 * seed + i
            r.state = kg.gen_uniform(r.n, r.width, r.height, r.params.seed, 1.0)
        return {"kind": kind, "steps": case["steps"], "replicas": replicas}
    if kind == "serve":
        # the first requests of the benchmark's stream, their flocks from the seed
        stream = kg.request_stream(200.0, 0.02 * case["requests"] + 1.0, case["n_min"], case["n_max"],
                                   case["steps_min"], case["steps_max"])
        requests = [r for _, r in stream[: case["requests"]]]
        for i, r in enumerate(requests):
            r.init_seed = r.params.seed = 1000 * seed + i
        return {"kind": kind, "requests": requests,
                "server": kg.Server(max_slots=64, hbm_budget_bytes=8 << 30, quantum_steps=50,
                                    max_request_boids=case["n_max"])}
    side, d = _geometry(case)
    ids, st = _birds(case, seed)
    s = {"kind": kind, "steps": case["steps"], "params": _params(case, seed), "ids": ids, "st": st, "step": 0,
         "field": kg.Field2D(side, side, d, True, capacity_hint=case["n"])}
    if kind in ("frame", "neighbors"):
        s["field"].set_states_device(ids, st)
        s["field"].lazy_update()
    if kind == "neighbors":
        r = np.random.default_rng(seed)
        s["query"] = QUERY[case["query"]]
        s["points"] = (r.random((case["points"], 2), dtype=np.float32) * np.float32(side * (1 - 1e-6)))
        s["lists"] = np.zeros(int(1.25 * case["points"] * _pairs(case)) + 1000, np.uint32)  # the program's own table
    return s


# ---------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "sweep":
        with kg.Batch(state["replicas"]) as b:
            b.step(0, state["steps"], graph_launches=100)
            moments = b.moments()
            parts = [b.get_replica(r) for r in range(b.nrep)]
        return moments, np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])
    if kind == "serve":
        server, requests = state["server"], state["requests"]
        tickets = [server.submit(r) for r in requests]
        server.wait_idle()
        parts = [server.result(t, r.nboids) for t, r in zip(tickets, requests)]
        for t in tickets:
            server.release(t)
        return np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])
    f = state["field"]
    if kind == "neighbors":
        counts, ids = f.neighbor_lists(state["query"], 10.0, state["points"])
        state["lists"][: len(ids)] = ids
        return counts, state["lists"]
    if kind == "frame":
        f.flock_step(state["params"], state["step"], 1)
        state["step"] += 1
        return f.read_buffer_device()
    f.set_states_device(state["ids"], state["st"])
    f.lazy_update()
    if kind == "run":
        f.flock_step(state["params"], 0, state["steps"])
        return f.read_buffer_device()
    ids, st = f.read_buffer_device()
    return ids, st, f.next_states_device(state["params"], 0, ids, st)


# ---------------------------------------------------------------- necessary work
def _pairs(case):
    """Expected candidates of one bird: those of its bags (relaxed query), or
    those within the radius (exact)."""
    density = case["density"]
    if case["clusters"]:
        density = case["n"] / case["clusters"] / (4.0 * math.pi * SIGMA * SIGMA)
    if case["query"] == "exact":
        return density * math.pi * 100.0
    ring = 2 * int(math.floor(case["ratio"])) + 1
    return density * (ring * 10.0 / case["ratio"]) ** 2


def work(case):
    """A step reads and writes each bird's record (16 B each way) and one offset
    per bag; a pair takes about 15 operations, a bird about 150 beside its pairs.
    Setting and reading a flock moves each record and id once each way."""
    if case["kind"] in ("sweep", "serve"):
        n = _mean_n(case) * (case["nrep"] if case["kind"] == "sweep" else case["requests"])
        steps = case["steps"] if case["kind"] == "sweep" else 0.5 * (case["steps_min"] + case["steps_max"])
        cells = n / 0.025 / (20.0 / 3.0) ** 2
        return {"bytes": n * 40 + steps * (32 * n + 8 * cells), "flops": steps * n * (150 + 15 * 10.0)}
    n, side = case["n"], _geometry(case)[0]
    if case["kind"] == "neighbors":
        p, found = case["points"], case["points"] * _pairs(case)
        return {"bytes": p * 12 + found * 12, "flops": 8 * found}
    cells = (side * case["ratio"] / 10.0 + 1.0) ** 2
    step = 32 * n + 8 * cells
    moved = {"run": 40 * n, "frame": 20 * n, "agents": 60 * n}[case["kind"]]
    return {"bytes": moved + case["steps"] * step, "flops": case["steps"] * n * (150 + 15 * _pairs(case))}


# ---------------------------------------------------------------- 64-bit values
def _philox(ids, step, seed):
    """Philox4x32-10 (Salmon et al., SC'11) words 0 and 1 at (id, step, 0, 0) under the key `seed`."""
    m = np.uint64(0xFFFFFFFF)
    c = [ids.astype(np.uint64) & m, np.full(len(ids), step & 0xFFFFFFFF, np.uint64),
         np.full(len(ids), step >> 32, np.uint64), np.zeros(len(ids), np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c[0], c[1]


def _bags(x, d):
    """floor(x / d) as the f32 quotient gives it (the bag of a coordinate is a 32-bit decision)."""
    return torch.floor(x.float() / torch.tensor(d, device=DEV)).long()


def _offsets(key, cells):
    return torch.cat([torch.zeros(1, dtype=torch.long, device=DEV), torch.cumsum(torch.bincount(key, minlength=cells), 0)])


def _one_step(case, seed, ids, st):
    """The next states of every bird of a read buffer (in its order), in 64 bits."""
    side, d = _geometry(case)
    lines = int(np.ceil(np.float32(side) / np.float32(d))) + 1
    dd = int(np.floor(np.float32(10.0) / np.float32(d)))
    cx, cy = _bags(st[:, 0], d), _bags(st[:, 1], d)
    start = _offsets(cx * lines + cy, lines * lines)
    me = st.double()
    n = len(ids)
    slot = torch.arange(n, device=DEV)
    sums = torch.zeros((6, n), dtype=torch.float64, device=DEV)
    count = torch.zeros(n, dtype=torch.float64, device=DEV)
    lo, hi = (cy - dd).clamp(min=0), (cy + dd).clamp(max=lines - 2)
    for k in range(-dd, dd + 1):
        col = cx + k
        valid = (col >= 0) & (col <= lines - 2)
        base = col.clamp(0, lines - 2) * lines
        s = start[base + lo]
        e = torch.where(valid, start[base + hi + 1], s)
        for f in range(int((e - s).max()) if n else 0):
            p = (s + f).clamp(max=n - 1)
            o = me[p]
            dx, dy = me[:, 0] - o[:, 0], me[:, 1] - o[:, 1]
            sq = dx * dx + dy * dy
            on = ((s + f) < e) & (p != slot)
            if case["query"] == "exact":
                on &= sq.sqrt() <= 10.0
            w = on.double()
            q = sq * sq + 1.0
            sums += w * torch.stack([dx / q, dy / q, dx, dy, o[:, 2], o[:, 3]])
            count += w
    c = count.clamp(min=1.0)
    avo, coh, con = 400.0 * sums[0:2] / c, -sums[2:4] / c / 10.0, sums[4:6] / c / c
    u0, u1 = _philox(ids.cpu().numpy(), 0, seed)
    r = torch.from_numpy(np.stack([(u >> np.uint64(8)).astype(np.float64) * 2.0 ** -24 * 2.0 - 1.0 for u in (u0, u1)])).to(DEV)
    rnd = float(np.float32(0.05)) * r / r.square().sum(0).sqrt()
    v = coh + avo + con + rnd + me[:, 2:4].T
    v = v / v.square().sum(0).sqrt() * float(np.float32(0.7))
    xy = torch.remainder(me[:, 0:2].T + v, side)
    return torch.cat([xy, v]).T.contiguous()


def exact(case, seed):
    """The single-step cases. A longer run has none: a flock's steps amplify any
    rounding, and the order that birds are kept in follows their positions."""
    if case["kind"] not in ("frame", "agents") or case["clusters"] or case["query"] == "exact":
        return None  # the exact query's whole-bag rule is a matter of 32-bit comparisons
    side, d = _geometry(case)
    lines = int(np.ceil(np.float32(side) / np.float32(d))) + 1
    ids, st = _birds(case, seed)
    order = torch.argsort(_bags(st[:, 0], d) * lines + _bags(st[:, 1], d), stable=True)
    ids, st = ids[order], st[order]
    nxt = _one_step(case, seed, ids, st)
    if case["kind"] == "agents":
        return None, st.double(), nxt
    order = torch.argsort(_bags(nxt[:, 0], d) * lines + _bags(nxt[:, 1], d), stable=True)
    return None, nxt[order]
