"""The cases whose time and outputs this repository is measured by.

Each case is one call (or the calls of one step) that a user's program makes on the public
entry points: the FP64 path one problem at a time (the reference's own way of working), the
FP32 path over batches (its throughput way), posterior marginals, internal-branch problems
(subtree re-threading) and one ARG-sampling step. Sizes are those of the benchmark's
configurations and of the tests, odd ones among them. Problems are seeded DSMC ARGs (10 bp
per column, N = 1e4, r = 1.6e-8, mu = 1.8e-8), the workload of the benchmark.
"""

from __future__ import annotations

import concurrent.futures as cf
import math
import os

import numpy as np

from argweaver_gb300 import api, refapi
from argweaver_gb300.sim import simulate

# kinds:
#   fp64_path   FP64 forward table, log-likelihood and sampled path of n problems
#   fp64_post   FP64 posterior marginals of n problems
#   fp32_table  FP32 forward table, log-likelihood and sampled path
#   fp32_path   FP32 log-likelihood and sampled path (the table stays on the device)
#   fp32_post   FP32 posterior marginals, kept in single precision
#   internal    fp32_path on internal-branch problems
#   step        one ARG-sampling step: a sequence threaded into the ARG, and the joint
#               probability of the ARG it is threaded into


def listed():
    return [
        # the smallest call: a toy region of the tests' size, where launches and host count
        dict(name="fp64_k8_1k", kind="fp64_path", n=1, k0=8, k1=8, l0=1000, l1=1000, ntimes=20,
             missing=0.0),
        # 8 haplotypes over 100 kb, one problem per call: the drop-in configuration
        dict(name="fp64_k8_10k", kind="fp64_path", n=1, k0=8, k1=8, l0=10000, l1=10000, ntimes=20,
             missing=0.0),
        # an ordinary drop-in call at the benchmark's largest haplotype count, odd length
        dict(name="fp64_k64_6007", kind="fp64_path", n=1, k0=64, k1=64, l0=6007, l1=6007, ntimes=20,
             missing=0.005),
        # posterior marginals in FP64 (forward and backward), fewer time points
        dict(name="fp64_post_k21_t16", kind="fp64_post", n=1, k0=21, k1=21, l0=3001, l1=3001,
             ntimes=16, missing=0.01),
        # one threading step of an ARG sampler (arg-sample's inner loop) and its joint probability
        dict(name="step_k12_2k", kind="step", n=1, k0=12, k1=12, l0=2000, l1=2000, ntimes=20,
             missing=0.0),
        # a forward table in FP32, a few small ragged problems in one call
        dict(name="fp32_table_4", kind="fp32_table", n=4, k0=8, k1=32, l0=801, l1=2999, ntimes=20,
             missing=0.005),
        # posterior marginals in FP32 of a small batch
        dict(name="fp32_post_8", kind="fp32_post", n=8, k0=8, k1=64, l0=500, l1=2500, ntimes=20,
             missing=0.005),
        # one long chromosome region at 100 haplotypes (the large-instance configuration's
        # per-column work over a tenth of its length)
        dict(name="fp32_k100_100k", kind="fp32_path", n=1, k0=100, k1=100, l0=100003, l1=100003,
             ntimes=20, missing=0.0),
        # many haplotypes at the finest time grid: over a thousand states per column
        dict(name="fp32_k200_t32", kind="fp32_path", n=2, k0=150, k1=200, l0=9001, l1=12001,
             ntimes=32, missing=0.005),
        # a served mix of requests (the serving configuration's haplotypes, shorter regions)
        dict(name="fp32_mix_24", kind="fp32_path", n=24, k0=8, k1=200, l0=5000, l1=40000, ntimes=16,
             missing=0.005),
        # subtree re-threading of a batch: internal-branch problems, cut along a removal path
        dict(name="internal_32", kind="internal", n=32, k0=50, k1=50, l0=20000, l1=40000, ntimes=20,
             missing=0.01),
        # the headline: 256 problems, 8..64 haplotypes, 100 kb .. 1 Mb
        dict(name="fp32_batch_256", kind="fp32_path", n=256, k0=8, k1=64, l0=10000, l1=100000,
             ntimes=20, missing=0.005),
    ]


def draw(rng):
    """One more case of the listed ranges: the same kinds, sizes over their whole range."""
    lu = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    kind = rng.choice(["fp64_path", "fp64_path", "fp64_post", "fp32_table", "fp32_path", "fp32_path",
                       "fp32_path", "fp32_post", "internal", "step"])
    ntimes = rng.choice([16, 20, 20, 32])
    missing = rng.choice([0.0, 0.005, 0.01])
    if kind == "fp64_path":
        k = lu(8, 64)
        L = lu(1000, 10000)
        if k > 24:
            L = min(L, 6007)
        return dict(kind=kind, n=1, k0=k, k1=k, l0=L, l1=L, ntimes=ntimes, missing=missing)
    if kind in ("fp64_post", "step"):
        k = lu(8, 32)
        L = lu(1000, 3500)
        return dict(kind=kind, n=1, k0=k, k1=k, l0=L, l1=L, ntimes=ntimes, missing=missing)
    if kind in ("fp32_table", "fp32_post"):
        n = lu(1, 8)
        return dict(kind=kind, n=n, k0=8, k1=lu(9, 64), l0=lu(300, 900), l1=lu(1000, 2500),
                    ntimes=ntimes, missing=missing)
    if kind == "internal":
        n = lu(4, 32)
        return dict(kind=kind, n=n, k0=lu(16, 30), k1=lu(31, 50), l0=lu(5000, 20000),
                    l1=lu(20001, 40000), ntimes=20, missing=missing)
    n = lu(1, 200)
    k1 = lu(16, 200) if n <= 24 else lu(16, 64)
    l1 = lu(8000, 40000) if k1 > 100 else lu(8000, 80000)
    return dict(kind=kind, n=n, k0=8, k1=k1, l0=5000, l1=l1, ntimes=ntimes, missing=missing)


# ---- inputs


def _specs(case):
    """(haplotypes, columns, ARG seed) of the case's problems. A case's ARGs are its own, as a
    program's are while it resamples them; the sequences' calls and the draws are the seed's."""
    sizes = [int(case[x]) for x in ("n", "k0", "k1", "l0", "l1", "ntimes")]
    rng = np.random.default_rng(sizes)
    n, k0, k1, l0, l1 = sizes[:5]
    if k1 > 100 and n > 4:  # a served mix: haplotypes spread over their logarithm
        ks = np.exp(rng.uniform(math.log(k0), math.log(k1 + 1), size=n)).astype(int)
        ls = np.exp(rng.uniform(math.log(l0), math.log(l1 + 1), size=n)).astype(int)
    else:
        ks = rng.integers(k0, k1 + 1, size=n)
        ls = rng.integers(l0, l1 + 1, size=n)
    seeds = rng.integers(1, 2**62, size=n)
    return [(int(k), int(L), int(s)) for k, L, s in zip(ks, ls, seeds)]


def _calls(seqs, rng):
    """The calls of one run of sequencing: private variants of single haplotypes at 0.4% of the
    columns, on top of the simulated mutations and missing calls."""
    n, L = seqs.shape
    m = int(rng.poisson(0.004 * L))
    rows, cols = rng.integers(0, n, size=m), rng.integers(0, L, size=m)
    base = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, size=m)]
    seqs[rows, cols] = np.where(seqs[rows, cols] == ord("N"), seqs[rows, cols], base)


def _problems(case, seed):
    specs, rng = _specs(case), np.random.default_rng(seed)
    internal = case["kind"] == "internal"

    def one(spec):
        k, L, s = spec
        return simulate(k if internal else k - 1, L, s, compress=10, ntimes=case["ntimes"],
                        maxtime=200e3, popsize=1e4, rho=1.6e-8, mu=1.8e-8,
                        missing=case["missing"], add_thread=not internal)

    with cf.ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
        probs = list(ex.map(one, specs))
    if internal:  # each ARG cut along a uniform removal path, as subtree re-threading cuts
        out = []
        for p, spec in zip(probs, specs):
            refapi.srand(spec[2] % 2**31)
            path, _ = refapi.sample_arg_removal_path_uniform(p)
            out.append(refapi.as_problem(p, refapi.remove_arg_thread_path(p, path), internal=True))
        probs = out
    for p in probs:
        _calls(p.seqs, rng)
    return probs, rng


def prepare(case, seed):
    probs, rng = _problems(case, seed)
    uniforms = [rng.random(p.seqlen) for p in probs]
    return {"case": case, "problems": probs, "uniforms": uniforms, "seed": int(seed) % 2**31}


def run(state):
    kind, probs, u = state["case"]["kind"], state["problems"], state["uniforms"]
    cat = lambda rows: rows[0] if len(rows) == 1 else np.concatenate(rows)  # noqa: E731
    if kind == "step":
        p = probs[0]
        joint = refapi.arghmm_joint_prob(p)
        refapi.srand(state["seed"])
        q = refapi.arghmm_sample_thread(p)
        # the new ARG as the genealogy of each column
        return {"joint": joint, "parents": np.repeat(q.ptrees, q.blocklens, axis=0),
                "ages": np.repeat(q.ages, q.blocklens, axis=0)}
    if kind == "fp64_post":
        r = api.run_batch(probs, precision="fp64", want_forward=False, want_posterior=True)
        return {"posterior": cat([x.posterior for x in r])}
    if kind == "fp32_post":
        r = api.run_batch(probs, precision="fp32", want_forward=False, want_posterior=True)
        return {"posterior": cat([x.posterior.astype(np.float32) for x in r])}
    table = kind in ("fp64_path", "fp32_table")
    r = api.run_batch(probs, precision="fp64" if kind == "fp64_path" else "fp32",
                      want_forward=table, want_path=True, uniforms=u)
    # the FP32 path's log-likelihood is good to single precision
    ll = np.array([x.loglik for x in r], np.float64 if kind == "fp64_path" else np.float32)
    out = {"path": cat([x.path for x in r]), "loglik": ll}
    if table:
        out["forward"] = cat([x.forward for x in r])
    return out


def _states_per_column(k, ntimes):
    # states of a local tree of k - 1 leaves, per column: about 8 per leaf and (at 20 time
    # points) a constant of 20
    return (7.4 * (k - 1) + ntimes) * (ntimes / 20.0) ** 0.4


def work(case):
    """The table's cells written once (and read once by the traceback, or by the backward
    pass, which writes the marginals), and the sequences and trees read. A column needs
    about 8 multiply-adds a state (same-branch moves, stay, inflow, emission, scaling) and
    the ntimes^2 of the moves between times."""
    specs = _specs(case)
    kind = case["kind"]
    size = 8 if kind in ("fp64_path", "fp64_post", "step") else 4
    cells = cols = seqs = 0.0
    for k, L, _s in specs:
        s = 17.0 if kind == "internal" else _states_per_column(k, case["ntimes"])
        cells += s * L
        cols += L
        seqs += k * L
    tables = 3 if kind in ("fp64_post", "fp32_post") else 2
    flops = (2 if tables == 3 else 1) * (16.0 * cells + 2.0 * case["ntimes"] ** 2 * cols)
    return {"bytes": tables * size * cells + seqs + 12.0 * cols, "flops": flops}


# ---- the same results in 64 bits, in plain numpy


def _levels(parent):
    """Nodes with children before parents."""
    n = len(parent)
    depth = np.zeros(n, int)
    for v in range(n):
        u = v
        while parent[u] >= 0:
            u = parent[u]
            depth[v] += 1
    return np.argsort(-depth, kind="stable")


class _Tree:
    def __init__(self, parent, age, T):
        n = len(parent)
        self.parent, self.age, self.n = parent, age, n
        self.kids = [[] for _ in range(n)]
        for v in range(n):
            if parent[v] >= 0:
                self.kids[parent[v]].append(v)
        self.root = int(np.nonzero(parent < 0)[0][0])
        node, time = [], []
        for v in range(n):
            top = T - 2 if v == self.root else int(age[parent[v]])
            for t in range(int(age[v]), top + 1):
                node.append(v)
                time.append(t)
        self.node, self.time = np.array(node), np.array(time)
        self.index = {(a, b): i for i, (a, b) in enumerate(zip(node, time))}
        nb, nr = np.zeros(T), np.zeros(T)
        for v in range(n):
            top = T - 2 if v == self.root else int(age[parent[v]])
            nb[age[v]:top] += 1
            nr[age[v]:top + 1] += 1
            if v == self.root:
                nb[top] += 1
        nb[T - 1] = 1
        self.nbranch, self.nrecomb, self.ncoal = nb, nr, nr.copy()

    def sibling(self, v):
        a, b = self.kids[self.parent[v]]
        return b if a == v else a


class _Model:
    def __init__(self, p):
        self.times, self.T, self.rho, self.mu = p.times, len(p.times), p.rho, p.mu
        t = p.times
        self.pop = p.popsizes
        self.step = np.append(np.diff(t), np.inf)
        mid = [math.sqrt((t[i] + 1.0) * (t[i + 1] + 1.0)) for i in range(self.T - 1)]
        cs = np.zeros(2 * self.T)
        for i in range(self.T - 1):
            cs[2 * i] = mid[i] - t[i]
            cs[2 * i + 1] = t[i + 1] - mid[i]
        cs[2 * self.T - 2] = cs[2 * self.T - 1] = np.inf
        self.cstep = cs
        self.mintime = t[1] * 0.1


def _transition(tr, m):
    """P(j -> k) of one tree, S x S."""
    T, t, ts = m.T, m.times, m.step
    nb, nr, nc = tr.nbranch, tr.nrecomb, tr.ncoal
    root = int(tr.age[tr.root])
    length = sum(t[tr.age[tr.parent[v]]] - t[tr.age[v]] for v in range(tr.n) if v != tr.root)
    b = np.arange(T - 1)
    rate = m.cstep[:2 * T - 2] * np.repeat(nb[:T - 1], 2) / np.repeat(2.0 * m.pop[:T - 1], 2)
    C = np.concatenate([[0.0, 0.0], np.cumsum(rate)])       # C[i + 2] = sum of rate[..i]
    len2 = length + t[:T - 1] + np.where(b > root, t[:T - 1] - t[root], 0.0)
    len2b = len2 + np.where(b > root, ts[:T - 1], ts[root])
    grow = np.exp(C[2 * b + 1])                              # exp(C[2b - 1])
    last = b < T - 2
    hit = np.where(last, -np.expm1(-rate[2 * b] - np.where(b > 0, rate[2 * b - 1], 0.0)), 1.0)
    here = np.where(last, -np.expm1(-rate[2 * b]), 1.0)
    E2 = np.exp(-C[2 * b]) * hit
    share = ts[:T - 1] * (nb[:T - 1] + 1.0) / (nr[:T - 1] + 1.0)
    own = ts[:T - 1] * nb[:T - 1] / (nr[:T - 1] + 1.0 + (b < root))
    B = np.cumsum(grow * share)
    N = grow * (share - own)
    D = -np.expm1(-m.rho * len2) / len2b
    E = 1.0 / nc[:T - 1]
    stay = np.exp(-np.maximum(m.rho * len2, m.rho))
    Bm = np.concatenate([[0.0], B[:-1]])
    X = np.where(b[:, None] < b[None, :], E2[None, :] * (B - N)[:, None],
                 (E2 * Bm)[None, :] + np.where(b[:, None] == b[None, :], (here * own)[None, :],
                                               (here * share)[None, :]))
    a_, b_ = tr.time[:, None], tr.time[None, :]
    DE = D[a_] * E[b_]
    P = DE * X[a_, b_]
    c = tr.age[tr.node]
    cterm = E2[tr.time] * np.where(c > 0, B[np.maximum(c - 1, 0)], 0.0)
    same = tr.node[:, None] == tr.node[None, :]
    P = P + np.where(same, DE * (X[a_, b_] - cterm[None, :]), 0.0)
    P[np.arange(len(c)), np.arange(len(c))] += stay[tr.time]
    return P


def _move(last, m, spr, node, time, parent_age, length, coal_time=None):
    """Probability that the thread at (node, time) leaves the breakpoint's recombination and
    coalescence as they are."""
    k, j, a = int(spr[1]), int(spr[3] if coal_time is None else coal_time), time
    t, ts, nb, cs = m.times, m.step, last.nbranch, m.cstep
    root = int(last.age[last.root])
    ln = length + t[a] + (t[a] - t[root] if node == last.root else 0.0)
    lb = ln + (ts[a] if node == last.root else ts[root])
    nbk = nb[k] + (k < a)
    nrk = last.nrecomb[k] + (k <= a) + (k == a) - (k >= max(root, a))
    p = nbk * ts[k] / (nrk * lb) * -math.expm1(-max(m.rho * ln, m.rho))
    s = 0.0
    for q in range(2 * k, 2 * j - 1):
        h = q // 2
        s += cs[q] * (nb[h] - (h < parent_age) + (h < a)) / (2.0 * m.pop[h])
    nbj = nb[j] - (j < parent_age) + (j < a)
    ncj = last.ncoal[j] - (j <= parent_age) - (j == parent_age) + (j <= a) + (j == a)
    q = 1.0 / ncj
    if j < m.T - 2:
        z = 0.0
        if j > k:
            z = cs[2 * j - 1] * (nb[j - 1] - (j - 1 < parent_age) + (j - 1 < a)) / (2.0 * m.pop[j - 1])
        q *= -math.expm1(-cs[2 * j] * nbj / (2.0 * m.pop[j]) - z)
    return p * math.exp(-s) * q


def _switch(tr, last, m, spr, mapping):
    """P(state of the last tree -> state of this tree) at a breakpoint, dense."""
    rn, rt, cn, ct = (int(x) for x in spr)
    t = m.times
    S1, S2 = len(last.node), len(tr.node)
    P = np.zeros((S1, S2))
    length = sum(t[last.age[last.parent[v]]] - t[last.age[v]] for v in range(last.n) if v != last.root)
    broken = int(last.parent[rn])
    page = int(last.age[broken])
    other = last.sibling(rn)
    after = int(tr.parent[mapping[other]] if other == cn else mapping[other])
    cache = {}

    def usual(node, time):
        key = (node == last.root, time)
        if key not in cache:
            cache[key] = _move(last, m, spr, node, time, page, length)
        return cache[key]

    mrec, mcoal = int(mapping[rn]), int(mapping[cn])
    for i in range(S1):
        v, a = int(last.node[i]), int(last.time[i])
        if (v, a) == (rn, rt):  # the recombination may sit on either side of the thread
            x = tr.index.get((mrec, rt))
            if x is not None:
                P[i, x] += _move(last, m, spr, v, a, page, length)
            x = tr.index.get((after, page))
            if x is not None:
                P[i, x] = _move(last, m, spr, v, a, a, length)
            continue
        if (v, a) == (cn, ct):  # the coalescence may be on the thread, above or below it
            n3 = int(mapping[last.sibling(rn)] if broken == v else mapping[v])
            top = int(tr.parent[mrec])
            for x in range(S2):
                w, b = int(tr.node[x]), int(tr.time[x])
                if (w == mrec and b >= rt) or (b == a and w in (n3, top)):
                    P[i, x] = _move(last, m, spr, v, a, page, length, coal_time=b)
            continue
        if v != rn:
            disrupt = bool(last.kids[v]) and rn in last.kids[v]
            w = int(mapping[last.sibling(rn)] if disrupt else mapping[v])
            if ct < a and (cn == v or mcoal == w) or disrupt and mcoal == w and ct <= a:
                w = int(tr.parent[w])
            x = tr.index.get((w, a))
            if x is not None:
                P[i, x] = usual(v, a)
        elif rt > a:
            x = tr.index.get((mrec, a))
            if x is not None:
                P[i, x] = usual(v, a)
        else:
            x = tr.index.get((after, page))
            if x is not None:
                P[i, x] = _move(last, m, spr, v, a, a, length)
    return P


def _emissions(tr, m, seqs):
    """Emission of every state at the tree's columns, columns x S."""
    ncol, mu, t, mint = seqs.shape[1], m.mu, m.times, m.mintime
    S = len(tr.node)
    same = (seqs == seqs[0]).all(axis=0)
    masked = same & (seqs[0] == ord("N"))
    inner_len = sum(max(t[tr.age[tr.parent[v]]] - t[tr.age[v]], mint) for v in range(tr.n) if v != tr.root)
    coal, low = t[tr.time], t[tr.age[tr.node]]
    ln = inner_len + np.maximum(coal, mint) + np.where(tr.node == tr.root, np.maximum(coal - t[tr.age[tr.root]], mint), 0.0)
    e = np.ones((ncol, S))
    e[same & ~masked] = 0.25 * np.exp(-mu * np.maximum(ln, mint))
    var = np.nonzero(~same)[0]
    if not len(var):
        return e
    code = np.full(256, -1)
    for i, ch in enumerate("ACGT"):
        code[ord(ch)] = code[ord(ch.lower())] = i
    lk = np.concatenate([np.eye(4), np.ones((1, 4))])        # row -1: unknown

    def along(x, d):  # Jukes-Cantor along a branch of length d, x: columns x 4
        f = np.exp(-4.0 / 3.0 * mu * d)
        return x * (0.25 * (1.0 + 3.0 * f)) + (x.sum(-1, keepdims=True) - x) * (0.25 * (1.0 - f))

    dist = [0.0 if v == tr.root else max(t[tr.age[tr.parent[v]]] - t[tr.age[v]], mint) for v in range(tr.n)]
    order = _levels(tr.parent)
    inn, up, out = [None] * tr.n, [None] * tr.n, [None] * tr.n
    for v in order:
        if tr.kids[v]:
            inn[v] = up[tr.kids[v][0]] * up[tr.kids[v][1]]
        else:
            inn[v] = lk[code[seqs[v, var]]]
        if v != tr.root:
            up[v] = along(inn[v], dist[v])
    out[tr.root] = np.ones((len(var), 4))
    for v in order[::-1]:
        if v == tr.root:
            continue
        q = int(tr.parent[v])
        s = up[tr.sibling(v)]
        out[v] = s if q == tr.root else s * along(out[q], dist[q])
    new = lk[code[seqs[(tr.n + 1) // 2, var]]]
    I = np.stack(inn)[tr.node]                                # S x columns x 4
    O = np.stack(out)[tr.node]
    top = np.array([0.0 if v == tr.root else t[tr.age[tr.parent[v]]] for v in tr.node])
    d = lambda x: np.maximum(x, mint)[:, None, None]          # noqa: E731
    p = along(new[None], d(coal)) * along(I, d(coal - low))
    at_root = (tr.node == tr.root)[:, None, None]
    p = np.where(at_root, p, p * along(O, d(top - coal)))
    e[var] = 0.25 * p.sum(-1).T
    return e


def _prior(tr, m):
    nb, cs = tr.nbranch, m.cstep
    out = np.zeros(len(tr.node))
    for b in range(m.T - 1):
        s = sum(cs[q] * nb[q // 2] / (2.0 * m.pop[q // 2]) for q in range(2 * b - 1))
        v = math.exp(-s) / tr.ncoal[b] if tr.ncoal[b] else 0.0
        if b < m.T - 2:
            z = cs[2 * b - 1] * nb[b - 1] / (2.0 * m.pop[b - 1]) if b else 0.0
            v *= -math.expm1(-cs[2 * b] * nb[b] / (2.0 * m.pop[b]) - z)
        out[tr.time == b] = v
    return out


def _hmm(p, posterior):
    """(forward table, log-likelihood, posterior or None) of one external problem."""
    m = _Model(p)
    trees = []
    start, last, x, ll, fw = 0, None, None, 0.0, []
    for i in range(p.ntrees):
        tr = _Tree(p.ptrees[i], p.ages[i], m.T)
        P = _transition(tr, m)
        L = int(p.blocklens[i])
        e = _emissions(tr, m, p.seqs[:, start:start + L])
        W = None
        rows = np.empty((L, len(tr.node)))
        for c in range(L):
            if c == 0 and last is None:
                rows[0] = x = _prior(tr, m)
                continue
            if c == 0:
                W = _switch(tr, last, m, p.sprs[i], p.mapping[i])
                x = (x @ W) * e[0]
            else:
                x = (x @ P) * e[c]
            s = x.sum()
            ll += math.log(s)
            x = x / s
            rows[c] = x
        fw.append(rows)
        if posterior:
            trees.append((P, W, e))
        last = tr
        start += L
    table = np.concatenate([r.ravel() for r in fw])
    if not posterior:
        return table, ll, None
    post = [None] * len(fw)
    b = np.ones(fw[-1].shape[1])
    for i in range(len(fw) - 1, -1, -1):
        P, W, e = trees[i]
        q = np.empty_like(fw[i])
        for c in range(len(q) - 1, -1, -1):
            z = fw[i][c] * b
            q[c] = z / z.sum()
            y = e[c] * b
            if c:
                b = P @ y
            elif W is not None:
                b = W @ y
            b = b / b.sum()
        post[i] = q
    return table, ll, np.concatenate([r.ravel() for r in post])


def exact(case, seed):
    """Tables, marginals and log-likelihoods; a sampled path has no such value. None for
    internal-branch problems, for an ARG-sampling step and where it would take too long."""
    kind = case["kind"]
    if kind in ("internal", "step"):
        return None
    specs = _specs(case)
    # a pass over a column costs about S^2 multiply-adds, over a tree about that of ten columns
    if sum(L * (30.0 + 0.05 * k) + (0.35 * k + 8) * L * 1e-3 * (500 + 12 * k + k * k) for k, L, _ in specs) > 4e6:
        return None
    probs, _ = _problems(case, seed)
    r = [_hmm(p, "post" in kind) for p in probs]
    cat = lambda rows: rows[0] if len(rows) == 1 else np.concatenate(rows)  # noqa: E731
    if "post" in kind:
        return {"posterior": cat([x[2] for x in r])}
    out = {"path": None, "loglik": np.array([x[1] for x in r])}
    if kind in ("fp64_path", "fp32_table"):
        out["forward"] = cat([x[0] for x in r])
    return out
