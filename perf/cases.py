"""The framework's work as a set of cases: whole partitions, finetunes, merges, graph ingest, scoring, the batched and
the learned partitioner, each through the Python binding a user's program calls.

Graphs are seeded directed degree-corrected block models of the law in dcsbm.py (power-law degrees, within-block
fraction w, popularity-weighted targets), drawn on the GPU with integer weights so that a seed always gives the same
edge list.  A finetune or merge starts from the planted partition split into the wanted number of blocks with a tenth
of the vertices moved to random blocks, as a level of the golden-section search meets it.
"""
import importlib
import math
import os
import sys

import numpy as np
import torch

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hybrid-stochastic-block-partitioning_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)
S = importlib.import_module("sbp_b200")


def listed():
    return [
        # The smallest whole call: the 1,000-vertex graph (suite graph 1).  Short batches in many sweeps: latency,
        # launches and host work count.
        dict(name="partition_gibbs_1k", kind="partition", algorithm="async_gibbs", V=1000, K=11, w=0.8, kmax=100,
             batches=10, approximate=True),
        # The headline use: a complete asynchronous-Gibbs partition, B = V down to the planted blocks.
        dict(name="partition_gibbs_100k", kind="partition", algorithm="async_gibbs", V=100_000, K=53, w=0.7, kmax=100,
             batches=10, approximate=True),
        # The end of a search on the 200,000-vertex bench graph: few blocks, the bracket's finetunes.
        dict(name="gibbs_200k_b71", kind="finetune", algorithm="async_gibbs", V=200_000, K=71, w=0.7, kmax=100, split=1,
             batches=10, sweeps=10),
        # The middle of its first descent.
        dict(name="gibbs_200k_b11770", kind="finetune", algorithm="async_gibbs", V=200_000, K=71, w=0.7, kmax=100,
             split=166, batches=10, sweeps=10),
        # The top of the descent of a graph whose block matrix is row-hashed (more blocks than dense storage takes).
        dict(name="gibbs_600k_hashed", kind="finetune", algorithm="async_gibbs", V=600_000, K=101, w=0.7, kmax=100,
             split=1450, batches=10, sweeps=2),
        # Sequential Metropolis-Hastings on the 20,000-vertex graph at its final block count.
        dict(name="mh_20k_b32", kind="finetune", algorithm="metropolis_hastings", V=20_000, K=32, w=0.6, kmax=100,
             split=1, batches=10, sweeps=3),
        # The hybrid schedule in mid-descent: Metropolis-Hastings over the high-degree 15 %, Gibbs over the rest.
        dict(name="hybrid_200k_b1560", kind="finetune", algorithm="hybrid_mcmc", V=200_000, K=71, w=0.7, kmax=100,
             split=22, batches=10, sweeps=2),
        # The first merge of a partition: every vertex its own block, half of the blocks merged away.
        dict(name="merge_200k_first", kind="merge", V=200_000, K=71, w=0.7, kmax=100, split=0, approximate=True),
        # Building the device graph from a host edge list with duplicates and self loops.
        dict(name="ingest_200k", kind="ingest", V=200_000, K=71, w=0.7, kmax=100),
        # Scoring a given partition and probing moves against it (no state changes): the smallest device calls.
        dict(name="score_5k_b40", kind="score", V=5_000, K=40, w=0.6, kmax=60, split=1, n=1500),
        # Many small graphs at once.
        dict(name="batched_16_graphs", kind="batched", V=1000, K=8, w=0.7, kmax=100, graphs=16, vmax=4000),
        # The learned proposal's partition (network weights as a user would load them, plain fallback at 5 %).
        dict(name="learned_partition_20k", kind="learned", V=20_000, K=32, w=0.6, kmax=100, batches=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["partition", "gibbs", "gibbs", "gibbs", "mh", "hybrid", "merge", "ingest", "score", "batched",
                       "learned"])
    w = round(rng.uniform(0.5, 0.85), 3)
    kmax = rng.choice([50, 100, 100, 200])
    if kind == "partition":
        algorithm = rng.choice(["async_gibbs", "async_gibbs", "hybrid_mcmc", "metropolis_hastings"])
        V = _log_int(rng, 700, 60_000 if algorithm == "async_gibbs" else 2500)
        return dict(kind=kind, algorithm=algorithm, V=V, K=max(4, int(1.2 * V ** 0.35)), w=w, kmax=kmax,
                    batches=rng.choice([4, 10, 10, 16]), approximate=rng.random() < 0.8 or V > 5000)
    if kind in ("gibbs", "mh", "hybrid"):
        algorithm = dict(gibbs="async_gibbs", mh="metropolis_hastings", hybrid="hybrid_mcmc")[kind]
        V = _log_int(rng, 3000, dict(gibbs=400_000, mh=20_000, hybrid=100_000)[kind])
        K = max(4, int(1.2 * V ** 0.35))
        split = max(1, int(_log_int(rng, K, V // 4) / K))
        return dict(kind="finetune", algorithm=algorithm, V=V, K=K, w=w, kmax=kmax, split=split,
                    batches=rng.choice([1, 4, 10, 10, 17]), sweeps=rng.randint(2, 8) if kind == "gibbs" else 2)
    if kind == "merge":
        V = _log_int(rng, 3000, 200_000)
        K = max(4, int(1.2 * V ** 0.35))
        split = rng.choice([0, max(1, int(_log_int(rng, 2 * K, V // 4) / K))])
        B = V if split == 0 else K * split
        return dict(kind=kind, V=V, K=K, w=w, kmax=kmax, split=split, approximate=rng.random() < 0.8 or B > 2000)
    if kind == "ingest":
        V = _log_int(rng, 2000, 300_000)
        return dict(kind=kind, V=V, K=max(4, int(1.2 * V ** 0.35)), w=w, kmax=kmax)
    if kind == "score":
        V = _log_int(rng, 1000, 50_000)
        K = max(4, int(1.2 * V ** 0.35))
        return dict(kind=kind, V=V, K=K, w=w, kmax=kmax, split=rng.randint(1, 6), n=rng.randint(300, 1500))
    if kind == "batched":
        return dict(kind=kind, V=700, K=8, w=w, kmax=100, graphs=rng.randint(5, 20), vmax=_log_int(rng, 1500, 6000))
    V = _log_int(rng, 3000, 30_000)
    return dict(kind="learned", V=V, K=max(4, int(1.2 * V ** 0.35)), w=w, kmax=kmax, batches=10)


def _edges(V, K, w, kmax, seed):
    """Host edge arrays and the planted block of every vertex."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 7919 + V)
    kmin = 10

    def uniform(n):
        return torch.rand(n, generator=gen, device=dev, dtype=torch.float64)

    def power_law(n):
        k = np.arange(kmin, kmax + 1, dtype=np.float64)
        cdf = np.cumsum(k ** -2.5)
        cdf = torch.from_numpy(cdf / cdf[-1]).to(dev)
        return (kmin + torch.searchsorted(cdf, uniform(n), right=True)).clamp_(kmin, kmax)

    # block sizes: every block at least V / (4 K), the rest by seeded proportions
    share = np.random.default_rng(seed).dirichlet(np.full(K, 2.0))
    bound = np.concatenate([[0], np.cumsum(V // (4 * K) + share * (V - K * (V // (4 * K))))]).astype(np.int64)
    bound[-1] = V
    bound = torch.from_numpy(bound).to(dev)
    perm = torch.randperm(V, generator=gen, device=dev)   # position in block order -> vertex id
    block_at = torch.searchsorted(bound, torch.arange(V, device=dev), right=True) - 1
    theta = power_law(V)   # popularity by position
    cum = torch.cumsum(theta, 0)
    before = torch.cat([torch.zeros(1, dtype=cum.dtype, device=dev), cum])
    src_pos = torch.repeat_interleave(torch.arange(V, device=dev), power_law(V))
    n = len(src_pos)
    within = uniform(n) < w
    lo, hi = before[bound[:-1]], before[bound[1:]]
    sb = block_at[src_pos]
    a = torch.where(within, lo[sb], torch.zeros_like(sb))
    span = torch.where(within, hi[sb] - lo[sb], before[-1].expand(n))
    x = a + (uniform(n) * span.double()).long().clamp_max(span - 1)
    dst_pos = torch.searchsorted(cum, x, right=True)
    order = torch.randperm(n, generator=gen, device=dev)   # edge lists come in no particular order
    src, dst = perm[src_pos][order], perm[dst_pos][order]
    truth = torch.empty(V, dtype=torch.int64, device=dev)
    truth[perm] = block_at
    return src.int().cpu().numpy(), dst.int().cpu().numpy(), truth.cpu().numpy()


def _start(truth, split, seed):
    """Starting assignment: each planted block in `split` parts (0: every vertex alone), a tenth of the vertices with
    their blocks shuffled among them; no block is empty."""
    V = len(truth)
    if split == 0:
        return V, np.arange(V, dtype=np.int32)
    rng = np.random.default_rng(seed + 1)
    order = np.argsort(truth, kind="stable")
    sizes = np.bincount(truth)
    part = np.arange(V) - np.repeat(np.cumsum(sizes) - sizes, sizes)   # rank of the vertex in its planted block
    a = np.empty(V, np.int64)
    a[order] = truth[order] * split + part % split
    moved = rng.permutation(V)[:V // 10]
    a[moved] = a[rng.permutation(moved)]
    return len(sizes) * split, a.astype(np.int32)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, seed=seed)
    if kind == "batched":
        s["graphs"] = []
        for i in range(case["graphs"]):
            V = int(round(case["V"] * (case["vmax"] / case["V"]) ** ((i + 0.5) / case["graphs"])))
            src, dst, _ = _edges(V, int(round(1.2 * V ** 0.35)), case["w"], case["kmax"], seed * 64 + i)
            s["graphs"].append(S.Graph(V, src, dst))
        return s
    src, dst, truth = _edges(case["V"], case["K"], case["w"], case["kmax"], seed)
    if kind == "ingest":
        s.update(src=src, dst=dst)
        return s
    s["graph"] = S.Graph(case["V"], src, dst)
    if kind in ("finetune", "merge", "score"):
        s["B"], s["start"] = _start(truth, case["split"], seed)
    if kind == "score":
        rng = np.random.default_rng(seed + 2)
        s["vertices"] = rng.permutation(case["V"])[:case["n"]].astype(np.int32)
        s["records"] = rng.integers(0, 2**32, size=(len(s["vertices"]), 4), dtype=np.uint64).astype(np.uint32)
    if kind == "learned":
        s["mlp"] = S.Mlp(seed=seed)
    return s


_COUNTS = ("visits", "proposals_moved", "accepted", "sweeps", "num_blocks")


def _result(assignment, stats):
    return dict(assignment=assignment, counts=np.array([stats[k] for k in _COUNTS]), mdl=stats["mdl"])


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "partition":
        return _result(*S.sbp.stochastic_block_partition(s["graph"], case["algorithm"], batches=case["batches"],
                                                         approximate=case["approximate"], seed=s["seed"]))
    if kind == "finetune":
        bm = S.Blockmodel(s["graph"], s["B"], s["start"])
        st = S.finetune.run(bm, S.ALGORITHMS[case["algorithm"]], batches=case["batches"], seed=s["seed"], call=1,
                            max_sweeps=case["sweeps"])
        return dict(_result(bm.block_assignment(), st), degrees=list(bm.degrees_all()))
    if kind == "merge":
        bm = S.Blockmodel(s["graph"], s["B"], s["start"])
        bm.setNum_blocks_to_merge(s["B"] // 2)
        got = S.block_merge.merge_blocks(bm, approximate=case["approximate"], seed=s["seed"], call=0)
        return dict(best=got["best"], dS=got["dS"], assignment=bm.block_assignment(), degrees=list(bm.degrees_all()),
                    avoided=got["merge_avoided"])
    if kind == "ingest":
        g = S.Graph(case["V"], s["src"], s["dst"])
        high, low = g.split()
        return dict(edges=g.E, high=high, low=low)
    if kind == "score":
        bm = S.Blockmodel(s["graph"], s["B"], s["start"])
        proposal, dS, H, accepted = bm.evaluate_vertices(s["vertices"], s["records"])
        return dict(mdl=S.entropy.mdl(bm), proposal=proposal, dS=dS, hastings=H, accepted=accepted)
    if kind == "batched":
        outs, stats, _ = S.batched.stochastic_block_partition(s["graphs"], batches=10, seed=s["seed"])
        return dict(assignments=outs, counts=np.array([[st[k] for k in _COUNTS] for st in stats]),
                    mdl=np.array([st["mdl"] for st in stats]))
    out, st = S.learned.stochastic_block_partition(s["graph"], s["mlp"], batches=case["batches"], seed=s["seed"],
                                                   fallback_acceptance=0.05)
    return _result(out, st)


def _mean_degree(kmax):
    k = np.arange(10, kmax + 1, dtype=np.float64)
    return float((k ** -1.5).sum() / (k ** -2.5).sum())


def work(case):
    """Bytes and operations of one pass: a visit reads its CSR offsets and block (12 bytes) and each neighbour's id and
    block (8 bytes, out and in), about 40 operations a neighbour; a partition's search runs the cap of 100 sweeps at
    every halving level of its first descent; ingest reads the edges once and writes both directions' lists."""
    V, kind = case["V"], case["kind"]
    E = V * _mean_degree(case["kmax"])
    visit_bytes, visit_flops = 12 * V + 16 * E, 80 * E
    levels = max(1.0, math.log2(max(2.0, V / case["K"])))
    if kind == "finetune":
        n = case["sweeps"]
    elif kind == "partition":
        n = 100 * levels
    elif kind == "learned":
        n = 10 * levels
    elif kind == "batched":
        mean = case["graphs"] * (case["vmax"] - V) / math.log(case["vmax"] / V) / V   # in units of V
        n = 100 * mean * levels
    elif kind == "merge":
        return dict(bytes=16 * E + 4 * V + 24 * V, flops=10 * 80 * E)
    elif kind == "ingest":
        return dict(bytes=8 * E + 12 * E + 9 * V, flops=2 * E)
    else:
        return dict(bytes=12 * E + 4 * V + case["n"] * (12 + 16 * _mean_degree(case["kmax"])) + 28 * case["n"],
                    flops=40 * E + 80 * case["n"] * _mean_degree(case["kmax"]))
    return dict(bytes=n * visit_bytes, flops=n * visit_flops)


def exact(case, seed):
    """Scoring in 64 bits: MDL, and proposal, delta-MDL, Hastings factor and accept decision of the probed vertices.
    The chains of the other cases are whole numbers that plain arrays cannot give in reasonable time."""
    if case["kind"] != "score":
        return None
    V = case["V"]
    src, dst, truth = _edges(V, case["K"], case["w"], case["kmax"], seed)
    B, b = _start(truth, case["split"], seed)
    b = b.astype(np.int64)
    rng = np.random.default_rng(seed + 2)
    vertices = rng.permutation(V)[:case["n"]]
    records = rng.integers(0, 2**32, size=(len(vertices), 4), dtype=np.uint64)
    _, first = np.unique(src.astype(np.int64) * V + dst, return_index=True)   # first occurrence of each edge
    first.sort()
    src, dst = src[first].astype(np.int64), dst[first].astype(np.int64)
    E = len(src)
    M = np.zeros((B, B), np.int64)
    np.add.at(M, (b[src], b[dst]), 1)
    d_out, d_in = M.sum(1), M.sum(0)

    def xlogx(x):   # differences of nearly equal terms follow, hence the longer type
        x = np.asarray(x, np.longdouble)
        return x * np.log(np.maximum(x, 1.0))

    def likelihood(M, d_out, d_in):
        return xlogx(M).sum() - xlogx(d_out).sum() - xlogx(d_in).sum()

    x = float(B) ** 2 / E
    mdl = E * ((1 + x) * np.log(1 + x) - x * np.log(x)) + V * np.log(B) - likelihood(M, d_out, d_in)
    by_out, by_in = np.argsort(src, kind="stable"), np.argsort(dst, kind="stable")
    out_at, in_at = np.searchsorted(src[by_out], np.arange(V + 1)), np.searchsorted(dst[by_in], np.arange(V + 1))
    d = d_out + d_in - np.diag(M)
    n = len(vertices)
    proposal, accepted = np.zeros(n, np.int32), np.zeros(n, bool)
    dS, hastings = np.zeros(n), np.ones(n)
    for i, (v, rec) in enumerate(zip(vertices, records)):
        r = int(b[v])
        out = dst[by_out[out_at[v]:out_at[v + 1]]]
        inn = src[by_in[in_at[v]:in_at[v + 1]]]
        inn = inn[inn != v]
        self_loop = int((out == v).sum())
        k_out, k_in = len(out), len(inn)
        k = k_out + k_in
        pick = (int(rec[0]) * k) >> 32
        t = int(b[out[pick]] if pick < k_out else b[inn[pick - k_out]])
        target = (int(rec[1]) * int(d_out[t] + d_in[t])) >> 32
        line = M[t] if target < d_out[t] else M[:, t]
        s = int(np.searchsorted(np.cumsum(line), target if target < d_out[t] else target - d_out[t], side="right"))
        proposal[i] = s
        if s == r:
            continue
        co = np.bincount(b[out[out != v]], minlength=B)
        ci = np.bincount(b[inn], minlength=B)
        delta = np.zeros((4, B), np.int64)   # rows r and s, columns r and s of the change
        N = M[[r, s], :].copy()
        C = M[:, [r, s]].copy()
        delta[0], delta[1], delta[2], delta[3] = -co, co, -ci, ci
        N += delta[:2]
        C += delta[2:].T
        N[:, r] += delta[2, [r, s]]
        N[:, s] += delta[3, [r, s]]
        N[0, r] -= self_loop
        N[1, s] += self_loop
        C[r] = N[0, [r, s]]
        C[s] = N[1, [r, s]]
        rest = np.ones(B, bool)
        rest[[r, s]] = False
        cells = (xlogx(M[[r, s], :]) - xlogx(N)).sum() + (xlogx(M[rest][:, [r, s]]) - xlogx(C[rest])).sum()
        do, di = k_out, k_in + self_loop
        degrees = (xlogx(d_out[r]) + xlogx(d_out[s]) - xlogx(d_out[r] - do) - xlogx(d_out[s] + do)
                   + xlogx(d_in[r]) + xlogx(d_in[s]) - xlogx(d_in[r] - di) - xlogx(d_in[s] + di))
        change = cells - degrees
        # a present Delta cell (r,s) / (s,r) with net change 0 and a non-zero count counts twice
        if (co[s] or ci[r]) and N[0, s] == M[r, s] > 0:
            change += M[r, s] * (np.log1p(di / d_in[s]) + np.log1p(-do / d_out[r]))
        if (co[r] or ci[s]) and N[1, r] == M[s, r] > 0:
            change += M[s, r] * (np.log1p(-di / d_in[r]) + np.log1p(do / d_out[s]))
        u = np.unique(np.concatenate([b[out], b[inn]]))
        c = (co + ci)[u] + np.where(u == r, self_loop, 0)
        fwd = (c * (M[s, u] + M[u, s] + 1.0) / (d[u] + B)).sum()
        after = d.copy().astype(np.float64)   # the reference leaves the in-side self loop out of r's and s's new degree
        after[r] = (d_out[r] - k_out) + (d_in[r] - k_in) - N[0, r]
        after[s] = (d_out[s] + k_out) + (d_in[s] + k_in) - N[1, s]
        bwd = (c * (N[0, u] + C[u, 0] + 1.0) / (after[u] + B)).sum()
        dS[i] = change
        hastings[i] = bwd / fwd
        accept_u = ((int(rec[2]) << 21) | (int(rec[3]) >> 11)) / 9007199254740992.0
        accepted[i] = accept_u <= min(1.0, math.exp(min(700.0, -3.0 * change)) * hastings[i])
    return dict(mdl=float(mdl), proposal=proposal, dS=dS, hastings=hastings, accepted=accepted)
