"""The finetune kernels at the sizes where their splits change, against the CPU oracle: vertex degrees on both sides of
what a lane, a group of 8, 16 or 32 lanes and a warp hold, batches of 128 and 129 vertices (one cluster or the whole
device), block counts on both sides of the walk's levels (none up to 128 blocks, sums of 64, sums of 64 of those), and
the row-hashed storage.  Integer state is equal; the MDL is stored as a float on both sides (relative 1e-7)."""
import numpy as np
import pytest

from conftest import random_assignment, random_graph
from test_gpu_parity import assert_same_state

pytestmark = pytest.mark.gpu

# out + in degrees of the first vertices, one each
DEGREES = [0, 1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 300, 511, 513, 700]


def graph_of_degrees(V, seed):
    """Vertex i < len(DEGREES) has DEGREES[i] edges (about half each way, no two alike) to the vertices after a third
    of the rest, which have a few edges among themselves; some vertices have a self loop and some edges come twice."""
    rng = np.random.default_rng(seed)
    h = len(DEGREES)
    src, dst = [], []
    for i, k in enumerate(DEGREES):
        out = k // 2
        src += [i] * out
        dst += rng.choice(np.arange(h, V), out, replace=False).tolist()
        dst += [i] * (k - out)
        src += rng.choice(np.arange(h, V), k - out, replace=False).tolist()
    n = 5 * V
    src += rng.integers(h, V, n).tolist()
    dst += (h + (rng.integers(0, V - h, n) * rng.random(n)).astype(int)).tolist()
    src += [3, 20, h + 5] + src[:40]
    dst += [3, 20, h + 5] + dst[:40]
    return np.array(src, np.int32), np.array(dst, np.int32)


def run_both(S, O, V, s, d, B, seed, algo, batches, sweeps):
    a = random_assignment(V, B, seed)
    g, og = S.Graph(V, s, d), O.Graph(V, s, d)
    assert g.E == og.E
    bm, obm = S.Blockmodel(g, B, a), O.Blockmodel(og, B, a)
    st = S.finetune.run(bm, algo, batches=batches, seed=seed, call=1, max_sweeps=sweeps)
    ost = obm.finetune(algo, batches=batches, seed=seed, call=1, max_sweeps=sweeps)
    assert_same_state(bm, obm)
    for k in ("sweeps", "visits", "accepted", "proposals_moved"):
        assert st[k] == ost[k], k
    assert st["mdl"] == pytest.approx(ost["mdl"], rel=1e-7)


@pytest.mark.parametrize("algo", [0, 1, 2])
@pytest.mark.parametrize("B", [2, 127, 128, 129, 500])
@pytest.mark.parametrize("storage", ["dense", "hashed"])
def test_degrees_and_blocks(S, O, storage, B, algo):
    V = 1200
    s, d = graph_of_degrees(V, B)
    S.set_option("dense_max_blocks", 131072 if storage == "dense" else 1)
    try:
        run_both(S, O, V, s, d, B, B + algo, algo, 5, 3)
    finally:
        S.set_option("dense_max_blocks", 131072)


@pytest.mark.parametrize("B", [40, 300])
def test_regrown_rows_count_self_loops(S, O, B):
    """Tight hashed rows run out of room; they are recounted from the out-lists, the in-lists and the self loops."""
    V = 1200
    s, d = graph_of_degrees(V, B)
    loops = np.arange(0, V, 3, dtype=np.int32)
    S.set_option("dense_max_blocks", 1)
    S.set_option("hashed_row_factor", 2)
    try:
        run_both(S, O, V, np.concatenate([s, loops]), np.concatenate([d, loops]), B, B, 1, 4, 4)
    finally:
        S.set_option("hashed_row_factor", 4)
        S.set_option("dense_max_blocks", 131072)


@pytest.mark.parametrize("algo", [0, 1])
@pytest.mark.parametrize("B", [4095, 4096, 4097])   # 64 sums of 64 columns; beyond, a second level
def test_walk_levels(S, O, B, algo):
    V = 4600
    s, d = graph_of_degrees(V, B)
    run_both(S, O, V, s, d, B, B, algo, 3, 2)


@pytest.mark.parametrize("per_batch", [1, 127, 128, 129])
@pytest.mark.parametrize("device_sweeps", [1, 0])
def test_batch_sizes(S, O, per_batch, device_sweeps):
    batches = 4
    V = per_batch * batches if per_batch > 1 else 60
    V, s, d, _ = random_graph(V, 4, per_batch)
    S.set_option("graph_sweeps", device_sweeps)
    try:
        run_both(S, O, V, s, d, min(30, V // 2), per_batch, 1, batches if per_batch > 1 else V, 5)
    finally:
        S.set_option("graph_sweeps", 1)


@pytest.mark.parametrize("group", [0, 1, 2])
def test_group_widths(S, O, group):
    V = 1200
    s, d = graph_of_degrees(V, 3)
    S.set_option("group_kernel", group)
    try:
        for B in (40, 300):
            run_both(S, O, V, s, d, B, 5, 1, 4, 3)
    finally:
        S.set_option("group_kernel", 1)


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 12289])   # edges a pass of the sort takes: 4,096
def test_ingest_sorts(S, O, n):
    """Duplicates and self loops in, in any order; the graph the oracle builds."""
    rng = np.random.default_rng(n)
    V = max(2, n // 6)
    s, d = rng.integers(0, V, n).astype(np.int32), rng.integers(0, V, n).astype(np.int32)
    g, og = S.Graph(V, s, d), O.Graph(V, s, d)
    assert g.E == og.E
    a = random_assignment(V, min(V, 20), n)
    assert_same_state(S.Blockmodel(g, min(V, 20), a), O.Blockmodel(og, min(V, 20), a))


@pytest.mark.parametrize("B", [2, 33, 1200])
@pytest.mark.parametrize("storage", ["dense", "hashed"])
def test_merge_scores(S, O, storage, B):
    """Scores are rounded to 2^-20 on both sides: equal, or one step apart where the sums' last bits fall on either
    side of a rounding boundary."""
    V = 1200
    s, d = graph_of_degrees(V, B)
    a = random_assignment(V, B, B) if B < V else np.arange(V, dtype=np.int32)
    S.set_option("dense_max_blocks", 131072 if storage == "dense" else 1)
    try:
        bm, obm = S.Blockmodel(S.Graph(V, s, d), B, a), O.Blockmodel(O.Graph(V, s, d), B, a)
        got = S.block_merge.merge_blocks(bm, seed=2)
        ref = obm.merge_blocks(seed=2)
    finally:
        S.set_option("dense_max_blocks", 131072)
    assert np.abs(got["dS"] - ref["dS"]).max() <= 2.0**-20
    assert (got["best"] == ref["best"]).mean() > 0.99


def test_batched_many_moves(S):
    """Batches in which more vertices move than the CTA that ends a stage finishes by itself (2,048)."""
    V, s, d, _ = random_graph(9000, 6, 8)
    graphs = [S.Graph(V, s, d) for _ in range(2)]
    outs, stats, info = S.batched.stochastic_block_partition(graphs, batches=2, seed=3)
    assert info["batched_finetunes"] > 0
    one, st = S.sbp.stochastic_block_partition(graphs[0], batches=2, seed=3)
    for a, sb in zip(outs, stats):
        assert np.array_equal(a, one)
        for k in ("num_blocks", "mdl", "sweeps", "accepted"):
            assert sb[k] == st[k], k


@pytest.mark.parametrize("first,last", [(0, 3000), (0, 40), (2960, 3000), (1500, 1501), (0, 0)])
@pytest.mark.parametrize("storage", ["dense", "hashed"])
def test_runs_of_empty_rows(S, O, storage, first, last):
    """Blocks with edges only from first to last: the offsets of the empty rows around them, in the storage's rows and
    in the merge's."""
    V = 3000
    rng = np.random.default_rng(last)
    n = 4000 if last > first else 0
    s, d = (rng.integers(first, max(last, 1), n).astype(np.int32) for _ in range(2))
    a = np.arange(V, dtype=np.int32)
    S.set_option("dense_max_blocks", 131072 if storage == "dense" else 1)
    try:
        bm, obm = S.Blockmodel(S.Graph(V, s, d), V, a), O.Blockmodel(O.Graph(V, s, d), V, a)
        assert_same_state(bm, obm)
        if n:
            got, ref = S.block_merge.merge_blocks(bm, seed=1), obm.merge_blocks(seed=1)
            assert np.array_equal(got["best"], ref["best"])
            assert_same_state(bm, obm)
    finally:
        S.set_option("dense_max_blocks", 131072)


@pytest.mark.parametrize("top", [384, 385, 768, 769, 1536, 1537, 3200])   # distinct neighbour blocks a share takes
@pytest.mark.parametrize("storage", ["dense", "hashed"])
def test_shares_of_heavy_vertices(S, O, storage, top):
    """Every vertex its own block, so a vertex has as many neighbour blocks as neighbours; 20 of them heavy."""
    V = 3300
    rng = np.random.default_rng(top)
    s, d = rng.integers(20, V, 3 * V), rng.integers(20, V, 3 * V)
    for i in range(20):
        k = max(257, top - 37 * i)
        u = rng.choice(np.arange(20, V), k, replace=False)
        out = rng.random(k) < 0.5
        s, d = np.concatenate([s, np.where(out, i, u)]), np.concatenate([d, np.where(out, u, i)])
    s, d = s.astype(np.int32), d.astype(np.int32)
    S.set_option("dense_max_blocks", 131072 if storage == "dense" else 1)
    try:
        g, og = S.Graph(V, s, d), O.Graph(V, s, d)
        bm, obm = S.Blockmodel(g, V, np.arange(V)), O.Blockmodel(og, V, np.arange(V))
        S.finetune.run(bm, 1, batches=3, seed=1, call=1, max_sweeps=2)
        obm.finetune(1, batches=3, seed=1, call=1, max_sweeps=2)
        assert_same_state(bm, obm)
    finally:
        S.set_option("dense_max_blocks", 131072)


def carried_out(best, dS, merges):
    """Blockmodel::carry_out_best_merges of one vertex a block: block pairs by score, equal scores by index."""
    name = np.arange(len(best))
    groups = {i: [i] for i in range(len(best))}
    for x in np.argsort(dS, kind="stable"):
        if merges == 0:
            break
        to = name[best[x]]
        if best[x] >= 0 and to != x:
            moved = groups.pop(x, [])
            name[moved] = to
            groups[to] = groups.get(to, []) + moved
            merges -= 1
    return np.unique(name, return_inverse=True)[1]


@pytest.mark.parametrize("hub", [3, 900, 2500])   # merges of two hubs of 2,500 neighbours score beyond +-2,048
def test_order_of_the_carried_out_merges(S, hub):
    V, hubs = 50_040, 40
    rng = np.random.default_rng(hub)
    s = np.repeat(np.arange(hubs), hub).astype(np.int32)
    d = np.concatenate([hubs + rng.permutation(V - hubs)[:hub] for _ in range(hubs)]).astype(np.int32)
    bm = S.Blockmodel(S.Graph(V, s, d), V, np.arange(V))
    got = S.block_merge.merge_blocks(bm, seed=1)
    assert (got["dS"].max() > 2048) == (hub == 2500)
    assert np.array_equal(bm.block_assignment(), carried_out(got["best"], got["dS"], V - bm.B))


@pytest.mark.parametrize("split,moved", [(1, 0.0), (1, 0.1), (12, 0.0), (12, 0.5), (60, 0.1)])
def test_widths_of_metropolis_hastings_rounds(S, O, split, moved):
    """Few and many accepted moves: rounds of 64, 32 and 16 positions, with histograms by block and with hash tables."""
    V, s, d, truth = random_graph(5000, 12, split, kmin=6, kmax=60)
    rng = np.random.default_rng(split)
    a = truth * split + rng.integers(0, split, V)
    some = rng.random(V) < moved
    a[some] = rng.integers(0, 12 * split, some.sum())
    a = np.unique(a, return_inverse=True)[1].astype(np.int32)
    B = int(a.max()) + 1
    bm, obm = S.Blockmodel(S.Graph(V, s, d), B, a), O.Blockmodel(O.Graph(V, s, d), B, a)
    st = S.finetune.run(bm, 0, seed=1, call=1, max_sweeps=4)
    ost = obm.finetune(0, seed=1, call=1, max_sweeps=4)
    assert_same_state(bm, obm)
    for k in ("sweeps", "visits", "accepted", "proposals_moved"):
        assert st[k] == ost[k], k


@pytest.mark.parametrize("B", [300, 600, 900])   # rows that start with few cells
def test_regrown_rows_do_regrow(S, O, B):
    V = 1200
    s, d = graph_of_degrees(V, B)
    loops = np.arange(0, V, 3, dtype=np.int32)
    s, d = np.concatenate([s, loops]), np.concatenate([d, loops])
    a = random_assignment(V, B, B)
    S.set_option("dense_max_blocks", 1)
    S.set_option("hashed_row_factor", 2)
    try:
        bm, obm = S.Blockmodel(S.Graph(V, s, d), B, a), O.Blockmodel(O.Graph(V, s, d), B, a)
        st = S.finetune.run(bm, 1, batches=4, seed=B, call=1, max_sweeps=4)
        obm.finetune(1, batches=4, seed=B, call=1, max_sweeps=4)
        assert st["overflow_rebuilds"] > 0
        assert_same_state(bm, obm)
    finally:
        S.set_option("hashed_row_factor", 4)
        S.set_option("dense_max_blocks", 131072)


def test_batched_degree_step_as_a_stage(S):
    """Batches of which more than 2,048 vertices move, so that the degree step is a stage of its own."""
    V, s, d, _ = random_graph(20_000, 6, 8)
    g = S.Graph(V, s, d)
    first = S.Blockmodel(g, V, np.arange(V))   # the partition's first round
    S.block_merge.merge_blocks(first, seed=3)
    assert S.finetune.run(first, 1, batches=2, seed=3, max_sweeps=1)["accepted"] > 2 * 2048
    outs, stats, info = S.batched.stochastic_block_partition([g, S.Graph(V, s, d)], batches=2, seed=3)
    assert info["batched_finetunes"] > 0
    one, st = S.sbp.stochastic_block_partition(g, batches=2, seed=3)
    for a, sb in zip(outs, stats):
        assert np.array_equal(a, one)
        for k in ("num_blocks", "mdl", "sweeps", "accepted"):
            assert sb[k] == st[k], k


@pytest.mark.parametrize("storage,algo", [("dense", 0), ("dense", 1), ("hashed", 1)])   # (hashed, 0): refused, the degrees
@pytest.mark.parametrize("share", [(0.5, 0.5), (0.55, 0.4, 0.03, 0.02)])   # corners alone, cells beside them
def test_counts_beyond_the_table(S, O, storage, share, algo):
    """Six million edges between a few blocks: counts and degrees beyond the 2^20 entries of the x log x table."""
    V, B = 3000, len(share)
    rng = np.random.default_rng(B)
    s, d = (x.astype(np.int32) for x in np.nonzero(rng.random((V, V)) < 0.67))
    a = rng.choice(B, V, p=share).astype(np.int32)
    S.set_option("dense_max_blocks", 131072 if storage == "dense" else 1)
    try:
        bm, obm = S.Blockmodel(S.Graph(V, s, d), B, a), O.Blockmodel(O.Graph(V, s, d), B, a)
        M = bm.blockmatrix()
        assert M[0, 1] > 1 << 20
        st = S.finetune.run(bm, algo, batches=4, seed=1, call=1, max_sweeps=1)
        ost = obm.finetune(algo, batches=4, seed=1, call=1, max_sweeps=1)
        assert st["accepted"] == ost["accepted"] > 0
        assert_same_state(bm, obm)
    finally:
        S.set_option("dense_max_blocks", 131072)
