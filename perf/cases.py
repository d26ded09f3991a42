"""Timed cases of the library: what its users call, from the smallest call to the largest.

Each case is a dict of plain values; `prepare` makes from a seed what a caller has in hand,
`run` is one call through the public binding, `work` the bytes and operations of that call
that no implementation can do without, and `exact` the float results in 64 bits.

Counts, node totals and pool sizes are whole numbers: they are the library's results and equal
the reference's, so `exact` covers only the cost model.
"""
import importlib.util
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The binding in gpu-n-queens_b200/ (the directory's name is no Python identifier)."""
    name = "gpu_n_queens_b200"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, os.path.join(ROOT, "gpu-n-queens_b200", "__init__.py"))
        module = importlib.util.module_from_spec(spec)
        sys.modules[name] = module
        spec.loader.exec_module(module)
    return sys.modules[name]


nqb = _package()
FORMS = {"plain": nqb.FORM_PLAIN, "batched": nqb.FORM_BATCHED}

# Search nodes of a full count (placements below the pool rows; they hardly depend on the pool
# depth) and pool sizes at depths 2..7: only `work` and `draw` use them.
NODES = {8: 1.0e3, 9: 4.7e3, 10: 1.77e4, 11: 9.13e4, 12: 4.28e5, 13: 2.53e6, 14: 1.37e7, 15: 9.19e7, 16: 6.1e8,
         17: 4.28e9, 18: 2.97e10, 19: 2.45e11, 20: 1.88e12, 21: 1.70e13}
POOL = {8: [21, 70, 163, 209, 147, 80], 9: [31, 129, 396, 796, 929, 573], 10: [36, 182, 697, 1872, 3239, 3179],
        11: [49, 291, 1337, 4516, 10788, 16387], 12: [55, 378, 2040, 8408, 25974, 54894],
        13: [71, 553, 3432, 16592, 62224, 171759], 14: [78, 682, 4816, 27034, 120638, 412951],
        15: [97, 939, 7432, 47460, 244887, 997736], 16: [105, 1118, 9844, 70906, 419408, 1998119],
        17: [127, 1473, 14272, 114434, 762380, 4151425], 18: [136, 1710, 18132, 160850, 1199146, 7409150],
        19: [161, 2179, 25080, 243742, 2009553, 13876054], 20: [171, 2482, 30880, 327274, 2967560, 22781426],
        21: [199, 3081, 41176, 472328, 4670527, 39430182]}
OPS_PER_NODE = 15  # integer operations of one placement: the count the roofline figures use
PARAMS = 112 * 128 + 128 + 128 * 128 + 128 + 128 + 1


def listed():
    return [
        # the smallest call: a first try, a test, or one of many small boards; its time is latency
        {"name": "count_n8", "kind": "count", "n": 8, "depth": 2, "depths": 2, "form": "plain"},
        # an everyday full count with the default options
        {"name": "count_n14", "kind": "count", "n": 14, "depth": 4, "depths": 2, "form": "plain"},
        # a full count in the batched form from a fine pool
        {"name": "count_n18_batched", "kind": "count", "n": 18, "depth": 6, "depths": 2, "form": "batched"},
        # the largest everyday count with the default options
        {"name": "count_n19_plain", "kind": "count", "n": 19, "depth": 6, "depths": 2, "form": "plain"},
        # a count from a shallow pool: few, very uneven items
        {"name": "count_n18_coarse", "kind": "count", "n": 18, "depth": 3, "depths": 2, "form": "batched"},
        # a shard of the headline N=21 pool, resident on the GPU, through the launch entry point
        {"name": "resident_n21_shard", "kind": "resident", "n": 21, "depth": 7, "share": 16, "form": "batched"},
        # a chunk of a state file solved from host memory with the default options
        {"name": "chunk_n17", "kind": "chunk", "n": 17, "depth": 6, "share": 4, "form": "plain"},
        # a handful of small partial boards, one count each
        {"name": "boards_small", "kind": "boards", "boards": 256, "n_lo": 8, "n_hi": 12, "d_lo": 2, "d_hi": 5},
        # a batch of uneven partial boards, queue in the order given
        {"name": "boards_uneven", "kind": "boards", "boards": 8192, "n_lo": 16, "n_hi": 20, "d_lo": 3, "d_hi": 7},
        # the same board set solved again and again: a captured plan ordered by the cost model
        {"name": "plan_uneven", "kind": "plan", "boards": 4096, "n_lo": 15, "n_hi": 18, "d_lo": 3, "d_hi": 7},
        # the cost model's forward pass over a pool's worth of states
        {"name": "predict_300k", "kind": "predict", "boards": 300000, "n_lo": 18, "n_hi": 18, "d_lo": 4, "d_hi": 8},
        # the cost model's training: forward, backward and update
        {"name": "train_64k", "kind": "train", "boards": 65536, "n_lo": 18, "n_hi": 18, "d_lo": 4, "d_hi": 8,
         "batch": 4096, "epochs": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        case = _draw(rng)
        if case not in known:
            return case


def _draw(rng):
    kind = rng.choice(["count", "count", "count", "chunk", "resident", "boards", "boards", "plan", "predict", "train"])
    if kind == "count":
        n = rng.randint(8, 19)
        if rng.random() < 0.25 and n >= 12:  # shallow pools
            return {"kind": kind, "n": min(n, 18), "depth": rng.choice([2, 3]), "depths": rng.choice([2, 3]),
                    "form": "batched"}
        lo = 2 if n < 12 else 4 if n < 16 else 5 if n < 18 else 6
        case = {"kind": kind, "n": n, "depth": lo + (n < 18) * rng.randint(0, 1), "depths": 2}
        if rng.random() < 0.5:
            return dict(case, form="batched")
        return dict(case, form="plain", unit=rng.random() < 0.3)  # also the split into unit and branch placements
    if kind == "chunk":
        n = rng.randint(12, 18)
        return {"kind": kind, "n": n, "depth": 4 if n < 15 else 6, "share": _log_int(rng, 2, 64),
                "form": rng.choice(["plain", "batched"])}
    if kind == "resident":
        n = rng.randint(15, 21)
        lo = 16 if n == 21 else 3 if n == 20 else 2
        return {"kind": kind, "n": n, "depth": 5 if n < 17 else 6 if n < 19 else 7, "share": _log_int(rng, lo, 500),
                "form": "batched" if n > 19 else rng.choice(["plain", "batched", "batched"])}
    if kind == "boards":
        n_lo = rng.randint(8, 17)
        d_lo = rng.randint(2, 4)
        return {"kind": kind, "boards": _log_int(rng, 16, 8192), "n_lo": n_lo, "n_hi": rng.randint(n_lo, min(n_lo + 4, 20)),
                "d_lo": d_lo if n_lo < 15 else max(3, d_lo), "d_hi": rng.randint(d_lo + 1, 7)}
    if kind == "plan":
        n_lo = rng.randint(10, 16)
        return {"kind": kind, "boards": _log_int(rng, 64, 4096), "n_lo": n_lo, "n_hi": n_lo + rng.randint(0, 2), "d_lo": 3,
                "d_hi": rng.randint(4, 7)}
    n = rng.randint(14, 20)
    if kind == "predict":
        return {"kind": kind, "boards": _log_int(rng, 100, 1000000), "n_lo": n, "n_hi": n, "d_lo": 4, "d_hi": 8}
    return {"kind": kind, "boards": _log_int(rng, 2000, 130000), "n_lo": n, "n_hi": n, "d_lo": 4, "d_hi": 8,
            "batch": _log_int(rng, 500, 8192), "epochs": rng.randint(1, 3)}


# ---- inputs ------------------------------------------------------------------------------


def _chunk(case, seed):
    """A share of the pool: one state drawn from each run of `share` states, in pool order."""
    pool = nqb.generate_pool(case["n"], case["depth"])
    k = case["share"]
    at = np.arange(len(pool) // k, dtype=np.int64) * k
    return pool[at + np.random.default_rng(seed).integers(0, k, len(at))]


def _boards(case, seed):
    """Random valid partial boards: n and depth uniform in their ranges, each row's column uniform
    among its free ones; a board that runs dry is drawn anew."""
    rng = np.random.default_rng(seed)
    count = case["boards"]
    out = np.zeros(count, dtype=nqb.STATE_DTYPE)
    n = rng.integers(case["n_lo"], case["n_hi"] + 1, count).astype(np.uint32)
    d = rng.integers(case["d_lo"], case["d_hi"] + 1, count)
    out["n"], out["row"], out["weight"] = n, d, 1
    todo = np.arange(count)
    bits = np.arange(32, dtype=np.uint32)
    while len(todo):
        mask = (np.uint32(1) << n[todo]) - np.uint32(1)
        cols, left, right = (np.zeros(len(todo), dtype=np.uint32) for _ in range(3))
        dry = np.zeros(len(todo), dtype=bool)
        for r in range(int(case["d_hi"])):
            on = (d[todo] > r) & ~dry
            free = mask & ~(cols | left | right)
            dry |= on & (free == 0)
            on &= free != 0
            key = rng.random((len(todo), 32), dtype=np.float32) * ((free[:, None] >> bits) & np.uint32(1))
            b = np.where(on, np.uint32(1) << np.argmax(key, 1).astype(np.uint32), np.uint32(0))
            cols |= b
            left = np.where(on, (left | b) << np.uint32(1), left)
            right = np.where(on, (right | b) >> np.uint32(1), right)
        ok = ~dry
        out["cols"][todo[ok]], out["ldiag"][todo[ok]], out["rdiag"][todo[ok]] = cols[ok], left[ok], right[ok]
        todo = todo[dry]
    return out


def _bit_count(v):
    v = v - ((v >> np.uint32(1)) & np.uint32(0x55555555))
    v = (v & np.uint32(0x33333333)) + ((v >> np.uint32(2)) & np.uint32(0x33333333))
    v = (v + (v >> np.uint32(4))) & np.uint32(0x0F0F0F0F)
    return ((v.astype(np.uint64) * 0x01010101) >> np.uint64(24)).astype(np.int64) & 0xFF


def _rows(boards):
    """Free columns, and the free cells of each of the next 32 rows (0 past the last row)."""
    n, row = boards["n"].astype(np.int64), boards["row"].astype(np.int64)
    free = ((np.uint32(1) << n.astype(np.uint32)) - np.uint32(1)) & ~boards["cols"]
    cells = np.zeros((len(boards), 32))
    for k in range(32):
        left = (boards["ldiag"].astype(np.uint64) << np.uint64(k)).astype(np.uint32)
        open_cells = _bit_count(free & ~(left | (boards["rdiag"] >> np.uint32(k))))
        cells[:, k] = np.where(k < n - row, open_cells, 0)
    return free, cells


def _labels(boards, seed):
    """Regression targets of the size and spread that log2 node counts have."""
    _, cells = _rows(boards)
    noise = np.random.default_rng(seed + 1).normal(0.0, 0.3, len(boards))
    return (0.5 * np.log2(1.0 + cells).sum(1) + noise).astype(np.float32)


def _weights(seed):
    """Freshly initialised network parameters (Glorot uniform, no bias)."""
    rng = np.random.default_rng(seed + 2)
    p = np.zeros(PARAMS, dtype=np.float32)
    for at, n_in, n_out in ((0, 112, 128), (112 * 128 + 128, 128, 128), (PARAMS - 129, 128, 1)):
        a = (6.0 / (n_in + n_out)) ** 0.5
        p[at:at + n_in * n_out] = rng.uniform(-a, a, n_in * n_out)
    return p


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case)
    if kind == "count":  # the caller chooses how deep a pool to build
        state["depth"] = case["depth"] + seed % case["depths"]
    elif kind == "chunk":
        state["states"] = _chunk(case, seed)
    elif kind == "resident":
        states = _chunk(case, seed)
        state["count"] = len(states)
        state["items"] = torch.from_numpy(states.view(np.uint8)).to("cuda")
        state["out"] = torch.zeros(4, dtype=torch.int64, device="cuda")
        state["scratch"] = torch.zeros(nqb.BATCHED_SCRATCH_BYTES, dtype=torch.uint8, device="cuda")
    elif kind == "boards":
        state["boards"] = _boards(case, seed)
    elif kind == "plan":
        boards = _boards(case, seed)
        model = nqb.Model()
        sample = dict(case, boards=4096)
        known = _boards(sample, seed + 3)
        model.train(known, _labels(known, seed + 3), epochs=4, batch=512, lr=2e-3)
        state["model"] = model
        state["plan"] = nqb.BatchPlan(boards, model=model)
    else:
        state["states"] = _boards(case, seed)
        state["model"] = nqb.Model()
        state["weights"] = _weights(seed)
        state["model"].set_params(state["weights"])
        if kind == "train":
            state["labels"] = _labels(state["states"], seed)
    return state


# ---- the calls ---------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "count":
        unit = state.get("unit", False)
        count, stats = nqb.count_ex(state["n"], state["depth"], form=FORMS[state["form"]], count_unit_nodes=unit)
        return {"count": count, "nodes": stats["nodes"], "states": stats["states"],
                "unit_nodes": stats["unit_nodes"] if unit else None}
    if kind == "chunk":
        total, stats = nqb.solve_states(state["states"], form=FORMS[state["form"]])
        return {"total": total, "nodes": stats["nodes"]}
    if kind == "resident":
        out, items = state["out"], state["items"]
        depth = state["n"] - state["depth"] - 1
        stream = torch.cuda.current_stream().cuda_stream
        out.zero_()
        if state["form"] == "plain":
            nqb.plain_launch(items.data_ptr(), state["count"], out.data_ptr(), stack_depth=depth, stream=stream)
        else:
            scratch = state["scratch"]
            scratch.zero_()
            nqb.batched_launch_ex(items.data_ptr(), state["count"], scratch.data_ptr(), scratch.numel(),
                                  out.data_ptr(), stack_depth=depth, stream=stream)
        return out
    if kind == "boards":
        counts, stats = nqb.solve_batch(state["boards"], form=nqb.FORM_BATCHED)
        return {"counts": counts, "nodes": stats["nodes"]}
    if kind == "plan":
        counts, stats = state["plan"].run()
        return {"counts": counts, "nodes": stats["nodes"]}
    model = state["model"]
    if kind == "predict":
        return model.predict(state["states"])
    model.set_params(state["weights"])  # training starts from the same weights in every pass
    losses = model.train(state["states"], state["labels"], epochs=state["epochs"], batch=state["batch"], lr=2e-3)
    return {"losses": losses, "weights": model.get_params()}


# ---- what a call cannot do without ----------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "count":  # the pool is the call's own: no input, a few words of output
        return {"bytes": 64.0, "flops": OPS_PER_NODE * NODES[case["n"]]}
    if kind in ("chunk", "resident"):
        states = POOL[case["n"]][case["depth"] - 2] // case["share"]
        return {"bytes": 16.0 * states + 32, "flops": OPS_PER_NODE * NODES[case["n"]] / case["share"]}
    if kind in ("boards", "plan"):
        per = [NODES[n] / POOL[n][d - 2] for n in range(case["n_lo"], case["n_hi"] + 1)
               for d in range(case["d_lo"], case["d_hi"] + 1)]
        nodes = case["boards"] * sum(per) / len(per)
        return {"bytes": 24.0 * case["boards"], "flops": OPS_PER_NODE * nodes}
    forward = 2.0 * (112 * 128 + 128 * 128 + 128) * case["boards"]
    if kind == "predict":
        return {"bytes": 20.0 * case["boards"] + 4 * PARAMS, "flops": forward}
    backward = 2.0 * (2 * 128 * 128 + 112 * 128 + 2 * 128) * case["boards"]
    return {"bytes": 20.0 * case["boards"] + 8 * PARAMS, "flops": case["epochs"] * (forward + backward)}


# ---- 64-bit results of the cost model ---------------------------------------------------------


def _features(boards):
    free, cells = _rows(boards)
    n, row = boards["n"].astype(np.int64), boards["row"].astype(np.int64)
    shift = (16 - (n >> 1)).astype(np.uint32)
    bits = np.arange(32, dtype=np.uint32)
    candidates = free & ~(boards["ldiag"] | boards["rdiag"])
    x = np.zeros((len(boards), 112))
    x[:, :32] = cells / 32
    x[:, 32:64] = ((free << shift)[:, None] >> bits) & np.uint32(1)
    x[:, 64:96] = ((candidates << shift)[:, None] >> bits) & np.uint32(1)
    x[:, 96], x[:, 97], x[:, 98] = (n - row) / 32, _bit_count(free) / 32, _bit_count(candidates) / 32
    x[:, 99], x[:, 100], x[:, 101] = n / 32, row / 32, cells.sum(1) / 256
    return x


def _unpack(p):
    a, b, c, d = 112 * 128, 112 * 128 + 128, 112 * 128 + 128 + 128 * 128, PARAMS - 129
    return p[:a].view(112, 128), p[a:b], p[b:c].view(128, 128), p[c:d], p[d:d + 128], p[PARAMS - 1]


def _forward(p, x):
    w1, b1, w2, b2, w3, b3 = _unpack(p)
    h = torch.nn.functional.gelu(x @ w1 + b1, approximate="tanh")
    h = torch.nn.functional.gelu(h @ w2 + b2, approximate="tanh")
    return h @ w3 + b3


def _shuffled(perm, rng):
    """Fisher-Yates over splitmix64, the order in which training takes its samples."""
    wrap = (1 << 64) - 1
    for i in range(len(perm) - 1, 0, -1):
        rng = (rng + 0x9E3779B97F4A7C15) & wrap
        z = ((rng ^ (rng >> 30)) * 0xBF58476D1CE4E5B9) & wrap
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & wrap
        j = (z ^ (z >> 31)) % (i + 1)
        perm[i], perm[j] = perm[j], perm[i]
    return rng


def exact(case, seed):
    if case["kind"] not in ("predict", "train"):
        return None
    boards = _boards(case, seed)
    x = torch.from_numpy(_features(boards))
    p = torch.from_numpy(_weights(seed).astype(np.float64))
    if case["kind"] == "predict":
        return _forward(p, x).numpy()
    t = torch.from_numpy(_labels(boards, seed).astype(np.float64))
    p.requires_grad_(True)
    adam = torch.optim.Adam([p], lr=float(np.float32(2e-3)), betas=(0.9, 0.999), eps=1e-8)
    perm, rng, losses = list(range(len(boards))), (0x9E3779B97F4A7C15 + 1) & ((1 << 64) - 1), []
    for _ in range(case["epochs"]):
        rng = _shuffled(perm, rng)
        total = 0.0
        for at in range(0, len(perm), case["batch"]):
            rows = perm[at:at + case["batch"]]
            adam.zero_grad()
            e2 = (_forward(p, x[rows]) - t[rows]).square()
            e2.mean().backward()
            adam.step()
            total += float(e2.detach().sum())
        losses.append(total / len(perm))
    return {"losses": np.array(losses), "weights": p.detach().numpy()}
