"""Timed workloads of the Monte Carlo framework, each through the entry points
a user's program calls.

The work of this framework comes in four forms:

* passes: a fault tree sampled and tallied over some sample words, by an
  engine the program keeps, by a manager that takes the steps of a
  convergence loop, or by one ``compute_tallies`` call from a PDAG;
* batches: many instances of many trees in one call (uncertainty draws, the
  time points of a probability curve);
* importance sampling: one rare-event tree, or many joined into one graph,
  with per-sample likelihood ratios in 64 bits;
* the proposal network: its training and its gradient.

Tree shapes, probability ranges, words and row counts are those of the
repository's workloads (mcscram_b200/synth.py, bench.py) and of its tests.
The structure of a case's tree follows from the case alone; the seed gives
the probabilities, the proposals and the network's rows, as a program that
analyses one model again and again with new data has it.
"""
from __future__ import annotations

import math

import numpy as np

from mcscram_b200 import _capi, host, importance, synth, uncertainty
from mcscram_b200.graph import AND, ATLEAST, NAND, NOR, NOT, OR, XOR, probability_threshold

# Gate mixes and probability ranges of the repository's synthetic trees.
FAMILIES = {
    # 50/50 AND/OR, 20 % of the events shared (the 200-event tree, the uncertainty trees)
    "andor": dict(mix={AND: 0.5, OR: 0.5}, p_range=(1e-3, 1e-1), share_be_frac=0.2),
    # every connective, 30 % of the nodes shared (the 5,000-event tree)
    "mixed": dict(mix={AND: 0.45, OR: 0.40, ATLEAST: 0.10, NOT: 0.025, XOR: 0.025}, p_range=(1e-5, 1e-2),
                  share_node_frac=0.3),
    # rare top events, read-once
    "rare": dict(mix={AND: 0.6, OR: 0.3, ATLEAST: 0.1}, p_range=(1e-6, 1e-3), atleast_n=(3, 5)),
    # rare top events, 20 % of the events read by two gates
    "rare-shared": dict(mix={AND: 0.6, OR: 0.3, ATLEAST: 0.1}, p_range=(1e-6, 1e-3), atleast_n=(3, 5),
                        share_be_frac=0.2, share_scope=1),
}

# Uncertainty draws go up to this probability (bench.py's ua workload).
CLIP = 0.5


def listed():
    return [
        # One step of a convergence loop on a small model: latency and launches are all there is.
        dict(name="step-60be", kind="step", family="andor", events=60, gates=32, layers=0, tree=7, words=4096),
        # One step on the large model with short passes: a launch that does not fill the chip.
        dict(name="step-5000be", kind="step", family="mixed", events=5000, gates=3000, layers=20, tree=11,
             words=1 << 15),
        # The whole analysis call, from the PDAG to every gate's statistics, at a fixed trial budget.
        dict(name="converge-200be", kind="converge", family="andor", events=200, gates=100, layers=7, tree=372,
             words=1 << 16, passes=16),
        # One pass of an engine as Engine() makes it, on the 200-event tree, all gates tallied, a ragged length.
        dict(name="pass-200be", kind="pass", mode="fused", family="andor", events=200, gates=100, layers=7, tree=372,
             words=(1 << 18) + 77),
        # The two-phase pipeline on a middle-sized tree with odd sizes, the top event only.
        dict(name="pass-1003be", kind="pass", mode="staged", family="rare", events=1003, gates=601, layers=10,
             tree=49, words=300001, tally="top"),
        # The headline pass (5,000 events, 3,000 gates, every gate tallied), a sixteenth of its length.
        dict(name="pass-5000be", kind="pass", mode="strip", family="mixed", events=5000, gates=3000, layers=20,
             tree=11, words=1 << 20),
        # Uncertainty analysis: lognormal draws of every tree's probabilities, all instances in one launch.
        dict(name="ua-16x16", kind="ua", trees=16, draws=16, tree=3, words=1 << 14),
        # A probability curve: the time points of one tree as instances, an odd number of them.
        dict(name="curve-200be", kind="curve", family="andor", events=200, gates=100, layers=7, tree=372, points=101,
             words=4096),
        # One round of importance sampling on one rare tree, with the cross-entropy numerators.
        dict(name="is-500be", kind="is", family="rare", events=500, gates=300, layers=8, tree=49, words=2048),
        # One cross-entropy round over many rare trees with shared events: main proposal and cut-set component.
        dict(name="bis-16", kind="bis", family="rare-shared", trees=16, tree=5, words=1 << 11),
        # Training of the shared proposal network.
        dict(name="mlp-train-250k", kind="train", rows=250000, steps=40),
        # One gradient of the network over the rows of a single tree, an odd number of them.
        dict(name="mlp-grad-2001", kind="grad", rows=2001),
    ]


def draw(rng):
    """One more case of the listed ones' ranges (sizes spread over their logarithms)."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "converge", "pass", "pass", "pass", "ua", "curve", "is", "bis", "train", "grad"])
    seed = rng.randrange(1 << 20)
    if kind in ("step", "converge", "pass"):
        family = rng.choice(["andor", "mixed", "rare"])
        events = log(200, 5000) if family == "mixed" else log(30, 5000)
        c = dict(kind=kind, family=family, events=events, gates=max(8, int(events * rng.uniform(0.5, 0.6))), layers=0,
                 tree=seed)
        budget = 2_000_000_000 // events  # basic-event words of a case stay below the largest listed one's
        if kind == "step":
            c["words"] = 1 << rng.randrange(8, 17)
        elif kind == "converge":
            c["words"] = 1 << rng.randrange(10, 17)
            c["passes"] = max(2, min(32, budget // c["words"]))
        else:
            c["mode"] = rng.choice(["fused", "staged", "strip", "auto"])
            c["words"] = min(log(1000, 1 << 20), budget)
            c["tally"] = rng.choice(["gates", "top"])
        return c
    if kind == "ua":
        return dict(kind=kind, trees=log(2, 16), draws=log(3, 24), tree=seed, words=log(256, 8192))
    if kind == "curve":
        events = log(30, 2000)
        return dict(kind=kind, family="andor", events=events, gates=events // 2, layers=0, tree=seed,
                    points=log(5, 200), words=log(256, 8192))
    if kind == "is":
        events = log(60, 4000)
        return dict(kind=kind, family="rare", events=events, gates=int(events * 0.6), layers=0, tree=seed,
                    words=log(500, 40000))
    if kind == "bis":
        return dict(kind=kind, family=rng.choice(["rare", "rare-shared"]), trees=log(1, 16), tree=seed,
                    words=log(256, 2048))
    if kind == "train":
        return dict(kind=kind, rows=log(200, 250000), steps=log(5, 40))
    return dict(kind=kind, rows=log(50, 200000))


# --- inputs -------------------------------------------------------------------


def _generate(family, events, gates, layers, seed):
    for k in range(64):  # a shape that the generator cannot fill with this seed is tried with the next
        try:
            return synth.generate(synth.TreeSpec(n_be=events, n_gates=gates, n_layers=layers or None,
                                                 seed=seed + 1000003 * k, **FAMILIES[family]))
        except ValueError:
            continue
    raise RuntimeError("no tree of this shape")


def _with_probabilities(g, rng, p_range):
    p = np.exp(rng.uniform(math.log(p_range[0]), math.log(p_range[1]), g.n_be))
    out = g.with_thresholds(probability_threshold(p))
    out.be_prob = p
    return out


def _one_tree(case, rng):
    g = _generate(case["family"], case["events"], case["gates"], case["layers"], case["tree"])
    return _with_probabilities(g, rng, FAMILIES[case["family"]]["p_range"])


def _rare_tree(g, rng):
    """g with log-uniform probabilities p, taken to a power p**c that puts the top event's probability (in the
    independence approximation) near a target in [1e-10, 1e-5], and every event's conditional probability given the
    top event, which is what a learned proposal tends to."""
    target = rng.uniform(math.log(1e-10), math.log(1e-5))
    p0 = np.exp(rng.uniform(math.log(1e-6), math.log(1e-3), g.n_be))
    low, high, c, last = 0.0, 4.0, 0.5, None
    for _ in range(24):
        p = np.clip(p0 ** c, 1e-9, 0.5)
        out = g.with_thresholds(probability_threshold(p))
        node, cond = importance.approximate_importance(out)
        f = (math.log(node[g.root]) if node[g.root] > 0 else -800.0) - target
        if abs(f) < 0.5:
            break
        low, high = (c, high) if f > 0 else (low, c)
        step = None if last is None or last[1] == f else c - f * (c - last[0]) / (f - last[1])
        last = c, f
        c = step if step is not None and low < step < high else 0.5 * (low + high)
    out.be_prob = p
    return out, cond


def _proposal(cond, rng, cap=0.5):
    return np.clip(cond * np.exp(rng.uniform(-0.3, 0.3, cond.size)), 1e-7, cap)


def _is_inputs(case, rng):
    """A rare tree and a proposal under which the top event fires in a share of the samples, as the rounds of the
    cross-entropy method have it: the conditional probabilities, flattened until the top event has 2 %."""
    g, cond = _rare_tree(_generate(case["family"], case["events"], case["gates"], case["layers"], case["tree"]), rng)
    c = 1.0
    while c > 0.1:
        q = _proposal(cond ** c, rng, 0.97)
        thr = np.clip(np.floor(q * 2.0**32), 1, 2.0**32 - 1).astype(np.uint64)
        if importance.approximate_importance(g.with_thresholds(thr))[0][g.root] >= 0.02:
            break
        c *= 0.8
    return g, q, thr


def _ua_shapes(case):
    """Gate counts log-uniform in [20, 5,000], 1.6 events a gate, as in the repository's uncertainty trees."""
    r = np.random.default_rng(case["tree"])
    return [(int(round(1.6 * g)), g, int(r.integers(1 << 30)))
            for g in (int(round(math.exp(r.uniform(math.log(20), math.log(5000))))) for _ in range(case["trees"]))]


def _bis_shapes(case):
    """Events log-uniform in [50, 10,000], 1.6 events a gate, as in the batched rare-event set."""
    r = np.random.default_rng(case["tree"])
    return [(b, max(4, int(round(b / 1.6))), int(r.integers(1 << 30)))
            for b in (int(round(math.exp(r.uniform(math.log(50), math.log(10000))))) for _ in range(case["trees"]))]


def _rows(case, rng):
    feats = rng.uniform(-0.5, 1.5, (case["rows"], importance.N_FEATURES)).astype(np.float32)
    targets = np.exp(rng.uniform(math.log(1e-6), math.log(0.5), case["rows"])).astype(np.float32)
    weights = rng.uniform(0.1, 2.0, case["rows"]).astype(np.float32)
    return feats, targets, weights


def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed)
    s = {"case": case}
    if kind == "step":
        g = _one_tree(case, rng)
        pdag = host.Pdag.from_flat(g)
        s["manager"] = host.LayerManager(pdag, 1 << 40, [int(g.gate_pdag_idx[g.root - g.n_be])],
                                         max_words_per_iteration=case["words"])
    elif kind == "converge":
        g = _one_tree(case, rng)
        s["pdag"] = host.Pdag.from_flat(g)
        s["watch"] = [int(i) for i in g.gate_pdag_idx[: min(g.n_gates - 1, 100)]]
        s["settings"] = host.Settings.default(num_trials=64 * case["words"] * case["passes"], early_stop=0,
                                              max_words_per_iteration=case["words"])
    elif kind == "pass":
        g = _one_tree(case, rng)
        nodes = [g.root] if case.get("tally") == "top" else np.arange(g.n_be, g.n_nodes)
        s["engine"] = _capi.Engine(g.with_tallies(nodes), mode=_capi.MODES[case["mode"]],
                                   layered_max_words=1 << 17, tune_pass_words=case["words"])
        s["pass"] = 0
    elif kind == "ua":
        trees = [_generate("andor", *shape[:2], 0, shape[2]) for shape in _ua_shapes(case)]
        trees = [g.with_tallies([g.root]) for g in trees]
        s["base"] = [np.exp(rng.uniform(math.log(1e-3), math.log(1e-1), g.n_be)) for g in trees]
        s["batch"], s["seed"] = uncertainty.Batch(trees), int(seed) & 0x7FFFFFFF
    elif kind == "curve":
        g = _one_tree(case, rng)
        rate = np.exp(rng.uniform(math.log(1e-6), math.log(1e-4), g.n_be))
        hours = np.linspace(0.0, 8760.0, case["points"])
        s["thresholds"] = [probability_threshold(-np.expm1(-rate * t)) for t in hours]
        s["batch"] = uncertainty.Batch([g.with_tallies([g.root])])
    elif kind == "is":
        g, q, _ = _is_inputs(case, rng)
        s["sampler"] = importance.ImportanceSampler(g)
        s["thresholds"] = s["sampler"].proposal_thresholds(q)
        s["pass"] = 1
    elif kind == "bis":
        trees = [_rare_tree(_generate(case["family"], *shape[:2], 0, shape[2]), rng) for shape in _bis_shapes(case)]
        s["sampler"] = importance.BatchedImportanceSampler([g for g, _ in trees],
                                                            chunk_words=(case["words"] + 255) // 256 * 256)
        cond = np.concatenate([c for _, c in trees])
        s["thresholds"] = s["sampler"].proposal_thresholds(_proposal(cond, rng))
        s["cutset"] = s["sampler"].proposal_thresholds(np.clip(cond, 1e-7, 0.9))
        s["pass"] = 1
    else:
        s["rows"] = _rows(case, rng)
        s["mlp"] = importance.ProposalMLP(seed=int(seed) & 0x7FFFFFFF)
    return s


# --- passes -------------------------------------------------------------------


def _counts(tallies):
    return [np.array([t[k] for t in tallies], dtype=np.int64) for k in ("num_one_bits", "total_bits")] + [
        np.array([t[k] for t in tallies]) for k in ("mean", "std_err")]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        return _counts(state["manager"].pass_wait_collect(1).values())
    if kind == "converge":
        return _counts(host.compute_tallies(state["pdag"], state["settings"], state["watch"])[0])
    if kind == "pass":
        state["pass"] += 1  # a new pass has new random numbers
        e = state["engine"]
        e.reset_tallies()
        e.run(state["pass"], 1, 0, case["words"])
        ones, total = e.tallies()
        return ones.astype(np.int64), total
    if kind == "ua":
        p_top, stats, _, thr = state["batch"].uncertainty(
            state["base"], draws_per_tree=case["draws"], clip_max=CLIP, seed=state["seed"],
            words_per_instance=case["words"], return_thresholds=True)
        return p_top, np.array([[t["mean"], t["sigma"]] for t in stats]), thr.astype(np.int64)
    if kind == "curve":
        ones = state["batch"].run([0] * case["points"], state["thresholds"], words_per_instance=case["words"])
        return ones.astype(np.int64)
    if kind == "is":
        r = state["sampler"].run(state["thresholds"], iteration=state["pass"], word_count=case["words"], ce=True)
        state["pass"] += 1
        return [np.array([r["sum_w"], r["sum_w2"], r["max_log_w"]]), r["ce_num"], r["hits"]]
    if kind == "bis":
        r = state["sampler"].run(state["thresholds"], iteration=state["pass"], word_count=case["words"], ce=True,
                                 words_cutset=case["words"] * 3 // 10, q_cutset=state["cutset"])
        state["pass"] += 1
        return [r["sum_w"], r["sum_w2"], r["max_log_w"], r["ce_num"], r["hits"]]
    feats, targets, weights = state["rows"]
    if kind == "train":
        loss = state["mlp"].train(feats, targets, weights, steps=case["steps"])
        return [state["mlp"].params(), loss]
    grad, loss = state["mlp"].grad(feats, targets, weights)
    return [grad, loss, state["mlp"].forward(feats)]


# --- what a pass cannot do without -------------------------------------------

# The reference's counter layout fixes the random numbers: a basic-event word
# is 16 generator calls of ten rounds with two 32x32 -> 64-bit products.  The
# products that depend only on the event or only on the word are shared, which
# leaves 242 (two 32-bit multiplies each); every output is compared once.
WORD_OPS = 242 * 2 + 64


def work(case):
    kind = case["kind"]
    if kind in ("step", "converge", "pass"):
        passes = case.get("passes", 1)
        words = float(case["events"]) * case["words"] * passes
        return {"bytes": 24.0 * case["events"] + 32.0 * case["gates"], "flops": words * WORD_OPS}
    if kind == "ua":  # the draws of a tree share their generator calls, not their comparisons
        events = float(sum(b for b, _, _ in _ua_shapes(case)))
        return {"bytes": 8.0 * events * case["draws"],
                "flops": events * case["words"] * (242 * 2 + 64 * case["draws"])}
    if kind == "curve":
        return {"bytes": 8.0 * case["events"] * case["points"],
                "flops": float(case["events"]) * case["words"] * (242 * 2 + 64 * case["points"])}
    if kind == "is":
        return {"bytes": 32.0 * case["events"], "flops": float(case["events"]) * case["words"] * WORD_OPS}
    if kind == "bis":
        events = float(sum(b for b, _, _ in _bis_shapes(case)))
        return {"bytes": 32.0 * events, "flops": events * case["words"] * WORD_OPS}
    forward = 2.0 * (16 * 64 + 64 * 64 + 64)
    if kind == "train":
        return {"bytes": 72.0 * case["rows"], "flops": 3.0 * forward * case["rows"] * case["steps"]}
    return {"bytes": 76.0 * case["rows"], "flops": 4.0 * forward * case["rows"]}


# --- what the outputs are in 64 bits -----------------------------------------


def _philox(x0, x1, x2, x3):
    """Philox4x32-10 (Salmon et al., Random123) under the reference's fixed key, on uint64 arrays of 32-bit words."""
    lo32, k0, k1 = np.uint64(0xFFFFFFFF), 382307844, 293830103
    for _ in range(10):
        a, b = x0 * np.uint64(0xD2511F53), x2 * np.uint64(0xCD9E8D57)
        x0, x1, x2, x3 = ((b >> np.uint64(32)) ^ x1 ^ np.uint64(k0), b & lo32,
                          (a >> np.uint64(32)) ^ x3 ^ np.uint64(k1), a & lo32)
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return x0, x1, x2, x3


def _samples(g, thr, iteration, words):
    """Every node's value in every sample: [n_nodes, 64 * words] booleans."""
    x = np.zeros((g.n_nodes, words * 64), dtype=bool)
    w = np.repeat(np.arange(1, words + 1, dtype=np.uint64), 16)
    t = np.tile(np.arange(16, dtype=np.uint64) + np.uint64((iteration + 1) << 6), words)
    for e in range(g.n_be):
        out = _philox(np.full(w.size, int(g.be_pdag_idx[e]) + 1, np.uint64),
                      np.full(w.size, int(g.be_event_idx[e]) + 1, np.uint64), w, t)
        x[e] = (np.stack(out, axis=1) < np.uint64(thr[e])).reshape(-1)
    for j in range(g.n_gates):
        v = x[g.gate_inputs(j)]
        v = np.concatenate([v[: v.shape[0] - int(g.gate_neg_count[j])], ~v[v.shape[0] - int(g.gate_neg_count[j]):]])
        op = int(g.gate_op[j])
        r = (v.all(axis=0) if op in (AND, NAND) else v.any(axis=0) if op in (OR, NOR) else
             v.sum(axis=0) >= int(g.gate_k[j]) if op == ATLEAST else (v.sum(axis=0) % 2).astype(bool) if op == XOR
             else v[-1])
        x[g.n_be + j] = ~r if op in (NAND, NOR, NOT) else r
    return x


def _exact_is(case, seed):
    g, _, thr = _is_inputs(case, np.random.default_rng(seed))
    x = _samples(g, thr, 1, case["words"])
    p, q = g.quantised_probabilities(), thr.astype(np.float64) / 2.0**32
    hit = np.nonzero(x[g.root])[0]
    ev = x[: g.n_be, hit].astype(np.float64)
    step = np.log(p / q) - (np.log1p(-p) - np.log1p(-q))
    log_w = float(np.sum(np.log1p(-p) - np.log1p(-q))) + step @ ev
    w = np.exp(log_w)
    return [np.array([w.sum(), (w * w).sum(), log_w.max() if hit.size else -np.inf]), ev @ w, int(hit.size)]


def _exact_network(case, seed):
    """Gradient, loss and outputs of the network in 64 bits.  The initial parameters are the handle's own."""
    feats, targets, weights = (a.astype(np.float64) for a in _rows(case, np.random.default_rng(seed)))
    mlp = importance.ProposalMLP(seed=int(seed) & 0x7FFFFFFF)
    v = mlp.params().astype(np.float64)
    mlp.close()
    w1, v = v[:1024].reshape(16, 64), v[1024:]
    b1, v = v[:64], v[64:]
    w2, v = v[:4096].reshape(64, 64), v[4096:]
    b2, w3, b3 = v[:64], v[64:128], v[128]
    h1 = np.maximum(feats @ w1 + b1, 0.0)
    h2 = np.maximum(h1 @ w2 + b2, 0.0)
    q = 1.0 / (1.0 + np.exp(-(h2 @ w3 + b3)))
    c, u = np.clip(q, 1e-7, 1.0 - 1e-7), weights / weights.sum()
    loss = -float(np.sum(u * (targets * np.log(c) + (1.0 - targets) * np.log(1.0 - c))))
    dz = u * (q - targets)
    d2 = dz[:, None] * w3[None, :] * (h2 > 0)
    d1 = (d2 @ w2.T) * (h1 > 0)
    grad = np.concatenate([(feats.T @ d1).reshape(-1), d1.sum(0), (h1.T @ d2).reshape(-1), d2.sum(0), h2.T @ dz,
                           [dz.sum()]])
    return [grad, loss, q]


def exact(case, seed):
    if case["kind"] == "is" and case["events"] * case["words"] <= 1_100_000:
        return _exact_is(case, seed)
    if case["kind"] == "grad":
        return _exact_network(case, seed)
    return None
