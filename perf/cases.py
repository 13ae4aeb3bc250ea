"""Workloads of the EDDY permutation test, each one call a user's program makes.

A case names an entry point (`entry`), the shape of its inputs and the test's
options:

  labellings  Context.run_labellings: explicit labellings of one gene set
  unit        unit_noalloc: one labelling through the entry point that
              allocates no device memory
  resident    Context.run_permutations: permutations of a set that stays on
              the device (the counter stream draws the labellings there)
  test        the whole test as the command line runs it: matrix loaded, sets
              added, every permutation run, results (JS values, fit, networks,
              edge lists) read back

Inputs are ternary expression matrices (per-gene tertiles).  `loading` is each
gene's weight on a latent factor shared by the genes of a set: co-expressed
genes, whose pair tests lie near the edge threshold; with loading 0 the genes
are independent but for `planted` ones that depend on others in class A only.
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "eddy-gpu_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "eddy-gpu_gb300"))

import eddy_gpu  # noqa: E402

ALPHA, LAMBDA, WEIGHT = 0.05, 2.0, 0.5

# One key per property of a case; what a listed case leaves out is as here.
DEFAULT = dict(
    entry="test",
    matrix=0,         # rows of the matrix (0: the genes of the one set)
    samples=200,
    first=100,        # samples of class A
    sets=1,
    smallest=20,      # genes per set: smallest to largest, spread over the
    largest=20,       # logarithm (spread "log") or evenly ("even")
    spread="log",
    labellings=1,     # labellings per call, or permutations (-r) per set
    parents=3,        # -mp
    bonferroni=True,  # False: -rawp
    prior_share=0.0,  # share of the sets with prior-knowledge edges
    prior_pairs=0,    # and the most of them per set
    stream="counter",
    networks=True,    # keep iteration 0's networks for the output files
    loading=0.0,
    planted=0,        # genes with class-A-only dependencies
    missing=0.0,      # share of values that are neither -1, 0 nor 1
    goes_on=1.0,      # share of the sets whose test goes past iteration 0
)


def full(case):
    return {**DEFAULT, **case}


def listed():
    """One of each use; sizes are the workload generator's, the tests' or odd
    ones between them."""
    return [
        # The smallest calls: one labelling of a small pathway (a notebook, a
        # service that asks for one labelling at a time).
        dict(name="one_labelling_20x200", entry="labellings", loading=0.8),
        dict(name="one_unit_no_alloc_48x300", entry="unit", samples=300, first=120, smallest=48,
             largest=48, parents=4, loading=0.7),
        # The command line on one set, as the reference's users run it (its
        # own glibc stream): the two small shapes of the workload generator.
        dict(name="test_20x200_r100", first=100, labellings=100, stream="glibc", planted=6,
             loading=0.6),
        dict(name="test_40x400_r200_priors", samples=400, first=150, smallest=40, largest=40,
             labellings=200, stream="glibc", prior_share=1.0, prior_pairs=30, planted=10,
             loading=0.6),
        # Explicit labellings (a blocked or stratified scheme of the user's),
        # with missing values, at odd sizes.
        dict(name="labellings_91x451_missing", entry="labellings", samples=451, first=187,
             smallest=91, largest=91, labellings=48, parents=2, loading=0.6, missing=0.01),
        # Permutations of a resident set: ragged sizes, a set above the
        # reference's 200 genes, and the precision-stress shape in full.
        dict(name="resident_137x777_r999", entry="resident", samples=777, first=300, smallest=137,
             largest=137, labellings=999, loading=0.66),
        dict(name="resident_387x600_r301", entry="resident", samples=600, first=300, smallest=387,
             largest=387, labellings=301, loading=0.7),
        dict(name="resident_200x1000_r10000", entry="resident", samples=1000, first=400,
             smallest=200, largest=200, labellings=10000, parents=4, loading=0.65, planted=40),
        # The same shape as one whole test, networks and edge list read back.
        dict(name="test_200x1000_r2000", samples=1000, first=400, smallest=200, largest=200,
             labellings=2000, parents=4, loading=0.65, planted=40),
        # Sweeps over many sets of uneven size: the two sparse ones of the
        # workload generator (most sets stop at iteration 0), and one of
        # co-expressed sets, which run all their permutations.
        dict(name="sweep_500_sets_r1000", matrix=5000, samples=600, first=300, sets=500,
             smallest=10, largest=150, spread="even", labellings=1000, prior_share=0.2,
             prior_pairs=20, planted=100, networks=False, goes_on=0.18),
        dict(name="sweep_2000_sets_r1000", matrix=20000, samples=1000, first=500, sets=2000,
             smallest=5, largest=300, labellings=1000, prior_share=0.97, prior_pairs=30,
             networks=False, goes_on=0.16),
        dict(name="sweep_150_coexpressed_r500", matrix=6000, samples=500, first=230, sets=150,
             smallest=8, largest=250, labellings=500, prior_share=0.3, prior_pairs=25,
             loading=0.6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _limit(case):
    """Work bound of drawn cases, well under the largest listed one's."""
    return work(case)["flops"] <= 0.07 * max(work(c)["flops"] for c in listed())


def draw(rng):
    while True:
        entry = rng.choice(["labellings", "unit", "resident", "resident", "test", "test"])
        n = _log(rng, 60, 2000)
        case = dict(entry=entry, samples=n, first=max(2, min(n - 2, int(n * rng.uniform(0.3, 0.6)))),
                    parents=rng.choice([1, 2, 3, 3, 4]), bonferroni=rng.random() < 0.8,
                    missing=rng.choice([0.0, 0.0, 0.0, 0.01]))
        if entry == "unit":
            g = _log(rng, 6, 64)
        elif entry == "labellings":
            g = _log(rng, 6, 400)
            case["labellings"] = _log(rng, 1, 400)
        elif entry == "resident":
            g = _log(rng, 6, 400)
            case["labellings"] = _log(rng, 60, 12000)
        else:
            g = _log(rng, 8, 300)
            case["labellings"] = _log(rng, 50, 2000)
            case["sets"] = _log(rng, 1, 120)
            case["stream"] = "counter" if case["sets"] > 4 else rng.choice(["counter", "glibc"])
            case["prior_share"] = rng.choice([0.0, 0.4])
            case["prior_pairs"] = rng.randint(5, 30) if case["prior_share"] else 0
        # co-expression that puts the pair tables about the edge threshold
        rho = math.sqrt(min(0.6, 65 / n * rng.uniform(0.5, 1.5)))
        case["loading"] = round(math.sqrt(rho / (1 - rho)), 3)
        case["largest"] = g
        case["smallest"] = g if case.get("sets", 1) == 1 else max(5, g // 8)
        if case.get("sets", 1) > 1:
            case["matrix"] = 3000
        if _limit(case):
            return case


# ------------------------------------------------------------------ inputs
def _sizes(c):
    """Genes per set: the user's pathway file, the same for every matrix."""
    if c["sets"] == 1:
        return [c["largest"]]
    rng = np.random.default_rng([c["sets"], c["largest"]])
    if c["spread"] == "even":
        return [int(v) for v in rng.integers(c["smallest"], c["largest"] + 1, c["sets"])]
    lo, hi = math.log(c["smallest"]), math.log(c["largest"])
    # log-normal about the middle of the range, clipped to it
    v = np.exp(rng.normal((lo + hi) / 2, (hi - lo) / 5, c["sets"]))
    return [int(x) for x in np.clip(np.round(v), c["smallest"], c["largest"])]


def inputs(case, seed):
    """data (genes x samples int8), labels (0 = class A), sets [(gene rows,
    prior matrix or None)]: host arrays, as the entry points take them."""
    c = full(case)
    rng = np.random.default_rng([seed, 20240])
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    sizes = _sizes(c)
    rows = c["matrix"] or max(sizes)
    n, nA = c["samples"], c["first"]
    x = torch.randn((rows, n), generator=gen, device=dev)
    sets = []
    if c["sets"] == 1:
        sets = [np.arange(sizes[0], dtype=np.int32)]
    elif c["loading"]:
        # pathways of co-expressed genes: each set takes a run of the rows
        sets = [np.arange(s, s + g, dtype=np.int32)
                for g, s in ((g, int(rng.integers(0, rows - g + 1))) for g in sizes)]
    else:
        sets = [np.sort(rng.choice(rows, g, replace=False, shuffle=False)).astype(np.int32)
                for g in sizes]
    if c["loading"]:
        block = rows if c["sets"] == 1 else 400
        z = torch.randn(((rows + block - 1) // block, n), generator=gen, device=dev)
        x += c["loading"] * z.repeat_interleave(block, 0)[:rows]
    if c["planted"]:
        target = rng.choice(rows, c["planted"], replace=False)
        source = rng.choice(np.setdiff1d(np.arange(rows), target), c["planted"])
        x[torch.from_numpy(target).to(dev), :nA] += 0.6 * x[torch.from_numpy(source).to(dev), :nA]
    # tertiles per gene, ties low
    s = x.sort(dim=1).values
    t1 = s[:, math.ceil(n / 3) - 1][:, None]
    t2 = s[:, math.ceil(2 * n / 3) - 1][:, None]
    data = ((x > t1).to(torch.int8) + (x > t2).to(torch.int8) - 1)
    if c["missing"]:
        gone = torch.rand((rows, n), generator=gen, device=dev) < c["missing"]
        data[gone] = 2
    labels = np.concatenate([np.zeros(nA, np.uint8), np.ones(n - nA, np.uint8)])
    out = []
    for genes in sets:
        prior = None
        g = len(genes)
        if c["prior_pairs"] and rng.random() < c["prior_share"]:
            prior = np.zeros((g, g), np.uint8)
            k = int(rng.integers(1, c["prior_pairs"] + 1))
            i, j = rng.integers(0, g, k), rng.integers(0, g, k)
            prior[i[i != j], j[i != j]] = 1
            prior |= prior.T
        out.append((genes, prior))
    return data.cpu().numpy(), labels, out


def _labellings(c, seed, labels):
    """The labellings of an explicit scheme, the unpermuted one first."""
    rng = np.random.default_rng([seed, 77])
    lab = np.tile(labels, (c["labellings"], 1))
    return np.concatenate([lab[:1], rng.permuted(lab[1:], axis=1)])


STREAM = dict(glibc=eddy_gpu.RNG_GLIBC, counter=eddy_gpu.RNG_COUNTER)


def prepare(case, seed):
    c = full(case)
    data, labels, sets = inputs(case, seed)
    state = dict(case=c, data=data, labels=labels, sets=sets)
    alpha_prior = 1 - (1 - ALPHA) * WEIGHT ** (1 / LAMBDA)
    if c["entry"] == "unit":
        state["opts"] = eddy_gpu.Opts(c["parents"], ALPHA, alpha_prior, int(c["bonferroni"]), 1,
                                      eddy_gpu.RNG_EXTERNAL, 0, 0, 0)
        return state
    rng = eddy_gpu.RNG_EXTERNAL if c["entry"] == "labellings" else STREAM[c["stream"]]
    ctx = eddy_gpu.Context(max_parents=c["parents"], alpha_edge=ALPHA, prior_weight=WEIGHT,
                           lam=LAMBDA, bonferroni=c["bonferroni"], permutations=c["labellings"],
                           rng=rng, seed=seed, keep_networks=c["networks"])
    state["ctx"] = ctx
    if c["entry"] == "test":
        state["out"], state["end"] = _room(c), {}
    else:
        ctx.load_matrix(data, labels)
        state["set"] = ctx.add_set(*sets[0])
    if c["entry"] == "labellings":
        state["labellings"] = _labellings(c, seed, labels)
    return state


# --------------------------------------------------------------------- run
def run(state):
    c = state["case"]
    if c["entry"] == "unit":
        js, unique = eddy_gpu.unit_noalloc(state["opts"], state["data"], state["labels"],
                                           state["sets"][0][1])
        return dict(js=np.array([js]), unique=unique)
    ctx = state["ctx"]
    if c["entry"] == "labellings":
        js, unique = ctx.run_labellings(state["set"], state["labellings"])
        return dict(js=js, unique=unique)
    if c["entry"] == "resident":
        js, unique = ctx.run_permutations(state["set"], 0, c["labellings"])
        return dict(js=js, unique=unique)
    ctx.clear_sets()
    ctx.load_matrix(state["data"], state["labels"])
    ids = [ctx.add_set(genes, prior) for genes, prior in state["sets"]]
    ctx.run()
    out = state["out"]
    at = dict.fromkeys(out, 0)

    def put(name, values):
        values = np.asarray(values).reshape(-1)
        out[name][at[name]:at[name] + values.size] = values
        at[name] += values.size

    for k in ids:
        s = ctx.summary(k)
        js, unique = ctx.js(k)
        row = slice(k * c["labellings"], k * c["labellings"] + len(js))
        out["js"][row], out["unique"][row] = js, unique
        out["iterations"][k], out["unique0"][k] = s["iterations"], s["unique0"]
        out["alpha"][k], out["beta"][k], out["pddn"][k] = s["alpha"], s["beta"], s["pddn"]
        # the output files are written for the sets whose test ran through
        if c["networks"] and not s["failed"]:
            net, lists = ctx.networks(k), ctx.edge_list(k)
            put("network_ids", net["ids"])
            put("network_nodes", net["nodes"])
            put("network_edges", net["edges"])
            put("likelihoods", net["lval"])
            put("list_nodes", lists["nodes"])
            put("list_edges", lists["edges"])
    for name, end in state["end"].items():  # what an earlier pass left behind
        out[name][at[name]:end] = -1
    state["end"] = at
    return out


def _room(c):
    """Buffers for a test's results: JS values and counts per set and
    iteration (NaN and 0 where a test stopped), then the networks and edge
    lists of the sets one after the other (-1 after the last)."""
    sizes, nets = _sizes(c), c["samples"] + 2
    k, genes, pairs = len(sizes), sum(sizes), sum(g * (g - 1) // 2 for g in sizes)
    room = dict(js=np.full(k * c["labellings"], np.nan), alpha=np.full(k, np.nan),
                beta=np.full(k, np.nan), pddn=np.full(k, np.nan),
                unique=np.zeros(k * c["labellings"], np.int32), iterations=np.zeros(k, np.int32),
                unique0=np.zeros(k, np.int32))
    if c["networks"]:
        room["likelihoods"] = np.full(2 * k * nets, np.nan)
        for name, most in (("network_ids", k * nets), ("network_nodes", genes * nets),
                           ("network_edges", genes * nets * c["parents"]),
                           ("list_nodes", 2 * genes), ("list_edges", 2 * pairs)):
            room[name] = np.full(most, -1, np.int32)
    return room


def work(case):
    """Bytes: inputs read and results written once.  Operations per labelling:
    the class-A tables of every pair (four cells of nine, the others follow
    from the genes' counts), the chi-square of the ten tables that a pair has
    per class (full, and one sample less in each cell), and one pass over the
    samples per node for the scores of the two full networks."""
    c = full(case)
    n = c["samples"]
    sizes = _sizes(c)
    flops = 0.0
    units = 0.0
    for g in sizes:
        pairs = g * (g - 1) / 2
        one = 2 * 4 * pairs * c["first"] + 2 * 10 * 40 * pairs + 2 * 4 * g * n
        k = 1 if c["entry"] == "unit" else c["labellings"]
        k = 1 + (k - 1) * c["goes_on"]
        flops += one * k
        units += k
    rows = c["matrix"] or max(sizes)
    given = n * c["labellings"] if c["entry"] == "labellings" else n
    return dict(bytes=float(rows * n + given + 4 * sum(sizes) + 12 * units), flops=float(flops))


# ------------------------------------------------- the same in 64 bits
LIMIT_S = 11.0


def exact(case, seed):
    c = full(case)
    if c["sets"] != 1:
        return None
    g, n = c["largest"], c["samples"]
    units = 1 if c["entry"] == "unit" else c["labellings"]
    if units * ((n + 2) * g * g * 3e-8 + g * 6e-4 + n * 2e-5) > LIMIT_S:
        return None
    data, labels, sets = inputs(case, seed)
    genes, prior = sets[0]
    if c["entry"] == "unit":
        lab = labels[None]
    elif c["entry"] == "labellings":
        lab = _labellings(c, seed, labels)
    elif c["stream"] == "glibc":
        lab = _glibc_stream(c, labels)
    else:
        lab = _counter_stream(c, seed, labels)
    unit = Unit(data[genes], prior, c)
    js, lval = [], None
    for k, one in enumerate(lab):
        j, lv = unit(one)
        lval = lv if k == 0 else lval
        js.append(j)
        if c["entry"] == "test" and k == 0 and math.isnan(j):
            break  # the test stops there
    if c["entry"] == "unit":
        return dict(js=np.array(js), unique=None)
    js = np.array(js)
    if c["entry"] != "test":
        return dict(js=js, unique=None)
    through = not np.isnan(js).any()
    mean = js.mean() if through else np.nan
    var = ((js - mean) ** 2).mean() if through else np.nan
    with np.errstate(all="ignore"):
        a = ((1 - mean) / var - 1 / mean) * mean ** 2
        b = a * (1 / mean - 1)
    out = dict.fromkeys(_room(c))
    out.update(js=np.full(units, np.nan), alpha=np.array([a]), beta=np.array([b]))
    out["js"][:len(js)] = js
    if c["networks"]:
        out["likelihoods"] = np.full(2 * (n + 2), np.nan)
        if through:
            out["likelihoods"][:lval.size] = lval.reshape(-1)
    return out


def _counter_stream(c, seed, labels):
    """Labelling p of the counter stream: sample s's key is word s mod 4 of
    Philox-4x32-10 of the counter (s / 4, p, set, 0) under the key `seed`; the
    class-A samples are those with the smallest (key, s)."""
    n, nA, R = c["samples"], c["first"], c["labellings"]
    mask = np.uint64(0xFFFFFFFF)
    quads = (n + 3) // 4
    perm = np.arange(R, dtype=np.uint64)[:, None]
    x = [np.broadcast_to(np.arange(quads, dtype=np.uint64), (R, quads)),
         np.broadcast_to(perm, (R, quads)), np.zeros((R, quads), np.uint64),
         np.zeros((R, quads), np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = x[0] * np.uint64(0xD2511F53), x[2] * np.uint64(0xCD9E8D57)
        x = [(p1 >> np.uint64(32)) ^ x[1] ^ np.uint64(k0), p1 & mask,
             (p0 >> np.uint64(32)) ^ x[3] ^ np.uint64(k1), p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    key = np.stack(x, 2).reshape(R, 4 * quads)[:, :n]
    first = np.argsort(key, axis=1, kind="stable")[:, :nA]
    lab = np.ones((R, n), np.uint8)
    np.put_along_axis(lab, first, 0, axis=1)
    lab[0] = labels
    return lab


def _glibc_stream(c, labels):
    """The reference's labellings: per iteration n discarded draws of libc's
    rand() from its initial state, then the first n distinct rand() % n."""
    n, nA = c["samples"], c["first"]
    libc = ctypes.CDLL("libc.so.6")
    libc.srand(1)
    lab = np.ones((c["labellings"], n), np.uint8)
    for k in range(c["labellings"]):
        for _ in range(n):
            libc.rand()
        order, seen = [], set()
        while len(order) < n:
            v = libc.rand() % n
            if v not in seen:
                seen.add(v)
                order.append(v)
        lab[k, order[:nA]] = 0
    lab[0] = labels
    return lab


class Unit:
    """JS divergence and normalised likelihoods of one labelling, network by
    network: every class's network with all its samples and with each sample
    left out, their BDeu scores, and the divergence of the two classes'
    likelihoods over the distinct networks."""

    def __init__(self, data, prior, c):
        self.state = np.where((data >= -1) & (data <= 1), data + 1, 3)  # 3: not counted
        self.g, self.n = data.shape
        self.cap = c["parents"]
        self.row, self.col = np.tril_indices(self.g, -1)
        self.factor = len(self.row) if c["bonferroni"] else 1
        self.alpha = np.full(len(self.row), ALPHA)
        if prior is not None:
            self.alpha[prior[self.row, self.col] == 1] = 1 - (1 - ALPHA) * WEIGHT ** (1 / LAMBDA)
        self.lg = {}

    def loggamma(self, d):
        if d not in self.lg:
            a = 4.0 / d
            self.lg[d] = np.array([math.lgamma(m + a) - math.lgamma(a) for m in range(self.n + 1)])
        return self.lg[d]

    def edges(self, t):
        """Whether each table (..., 3, 3) holds an edge: chi-square with Yates'
        correction where an expected count of the support is below 5, and a
        series for its tail that gives up (p = 1) below 1e-37."""
        t = t.astype(np.float64)
        r, k, total = t.sum(-1), t.sum(-2), t.sum((-1, -2))
        with np.errstate(all="ignore"):
            e = r[..., :, None] * k[..., None, :] / total[..., None, None]
            live = (r[..., :, None] > 0) & (k[..., None, :] > 0)
            y = 0.5 * ((e < 5) & live).any((-1, -2))
            chi = np.where(live, (np.abs(t - e) - y[..., None, None]) ** 2 / e, 0.0).sum((-1, -2))
            dof = ((k > 0).sum(-1) - 1) * ((r > 0).sum(-1) - 1)
            x, p = chi / 2, dof / 2
            tail = torch.special.gammaincc(torch.from_numpy(np.maximum(p, 0.5)),
                                           torch.from_numpy(x)).numpy()
            norm = np.array([math.lgamma(d / 2 + 1) for d in range(5)])[np.clip(dof, 0, 4)]
            floor = p * np.log(x) - norm - x
        none = (x <= 0) | (dof <= 0) | (floor < math.log(1e-37))
        # the series behind the test's p (AS 147) stops at a term below 1e-9
        # of its sum: followed where that can decide
        adjusted = tail * self.factor
        near = ~none & (np.abs(adjusted / self.alpha[:, None] - 1) < 1e-2)
        xs, ps = x[near], p[near]
        term, total, step, on = np.ones_like(xs), np.ones_like(xs), ps.copy(), np.ones(xs.shape, bool)
        while on.any():
            step += 1
            term = np.where(on, term * xs / step, term)
            total = np.where(on, total + term, total)
            on &= term > 1e-9 * total
        adjusted[near] = (1.0 - total * np.exp(floor[near])) * self.factor
        return np.where(none, 1.0, np.minimum(adjusted, 1.0)) < self.alpha[:, None]

    def score(self, t, parents, cls, seen):
        """BDeu of a node (its first three parents) over a class's states."""
        idx = [t, *parents[:3]]
        ok = (cls[idx] < 3).all(0)
        code = np.zeros(int(ok.sum()), np.int64)
        for i in idx:
            code = code * 3 + cls[i][ok]
        cell = np.bincount(code, minlength=3 ** len(idx)).reshape(3, -1)
        r = int(seen[t])
        q = int(np.prod(seen[idx[1:]])) if len(idx) > 1 else 1
        if r == 0 or q == 0:
            return 0.0
        return float(self.loggamma(q * r)[cell].sum() - self.loggamma(q)[cell.sum(0)].sum())

    def __call__(self, labels):
        nets, classes = [], []
        for k in (0, 1):
            cls = self.state[:, labels == k]
            hot = np.stack([cls == a for a in range(3)], 1).reshape(3 * self.g, -1).astype(float)
            gram = (hot @ hot.T).reshape(self.g, 3, self.g, 3).transpose(0, 2, 1, 3)
            table = gram[self.row, self.col]
            less = np.stack([table] + [table - np.eye(9)[j].reshape(3, 3) for j in range(9)], 1)
            bits = self.edges(np.maximum(less, 0))
            bits[:, 1:] = np.where(table.reshape(-1, 9) > 0, bits[:, 1:], bits[:, :1])
            a, b = cls[self.row], cls[self.col]
            pick = np.where((a < 3) & (b < 3), 1 + 3 * a + b, 0)
            edge = np.take_along_axis(bits, pick, 1).T
            edge = np.concatenate([bits[None, :, 0], edge] if k == 0 else [edge, bits[None, :, 0]])
            full_ = np.zeros((len(edge), self.g, self.g), bool)
            full_[:, self.row, self.col] = edge
            nets.append(full_ & (np.cumsum(full_, 2, dtype=np.int16) <= self.cap))
            classes.append((cls, np.array([(hot[3 * i:3 * i + 3].sum(1) > 0).sum()
                                           for i in range(self.g)])))
        nets = np.concatenate(nets)
        first = {}
        for s, bits in enumerate(np.packbits(nets.reshape(len(nets), -1), axis=1)):
            first.setdefault(bits.tobytes(), s)
        known, dist = {}, np.zeros((2, len(first)))
        base = None
        for u, s in enumerate(first.values()):
            net = nets[s]
            if base is None:
                base, todo, was = net, range(self.g), None
            else:
                todo = np.nonzero((net != base).any(1))[0]
            total = [0.0, 0.0] if was is None else list(was)
            for t in todo:
                for sign, from_ in ((1, net), (-1, base)):
                    if was is None and sign < 0:
                        continue
                    parents = np.nonzero(from_[t])[0]
                    key = (t, *parents[:3].tolist())
                    if key not in known:
                        known[key] = [self.score(t, parents, *cl) for cl in classes]
                    total = [total[k] + sign * known[key][k] for k in (0, 1)]
            if was is None:
                was = tuple(total)
            dist[:, u] = total
        with np.errstate(all="ignore"):
            lik = np.exp((dist - dist.mean(1, keepdims=True)) * 10 /
                         (dist.max(1) - dist.min(1))[:, None])
            lik /= lik.sum(1, keepdims=True)
            mid = lik.mean(0)
            terms = np.where((lik > 0) & (mid > 0), lik * np.log(lik / mid), 0.0)
            js = terms.sum() / 2 / math.log(2.0)
        if (dist.max(1) == dist.min(1)).any():
            js = math.nan
            lik[:] = np.nan
        return js, lik
