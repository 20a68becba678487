"""Several calls on one blockmodel: what a call leaves behind in the blockmodel's scratch must not reach the next one,
whichever kernels the calls take.  A dense asynchronous-Gibbs finetune is one persistent kernel; hybrid and learned
finetunes, collected moves, host-driven sweeps and row-hashed rounds are launches per batch."""
import threading

import numpy as np
import pytest

from conftest import random_assignment, random_graph, random_records
from test_gpu_parity import assert_same_state

pytestmark = pytest.mark.gpu

HYBRID, GIBBS = 2, 1


def fresh(S, bm, g):
    """A blockmodel of the same state that no call has touched."""
    new = S.Blockmodel(g, bm.B, bm.block_assignment())
    S.set_degrees(new, bm.degrees())
    return new


def same(a, b):
    assert np.array_equal(a.block_assignment(), b.block_assignment())
    assert np.array_equal(a.blockmatrix(), b.blockmatrix())
    for x, y in zip(a.degrees_all(), b.degrees_all()):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("batches", [1, 10])   # 1,001 vertices in ten batches: nine of 101, so an odd number of steps
@pytest.mark.parametrize("B", [40, 300])
def test_finetunes_of_both_kinds_in_turn(S, O, B, batches):
    V, s, d, _ = random_graph(1001, 8, B)
    a = random_assignment(V, B, 1)
    g, og = S.Graph(V, s, d), O.Graph(V, s, d)
    bm, obm = S.Blockmodel(g, B, a), O.Blockmodel(og, B, a)
    for call, algo in enumerate([HYBRID, GIBBS, HYBRID, GIBBS, GIBBS, HYBRID, HYBRID, GIBBS, HYBRID]):
        st = S.finetune.run(bm, algo, batches=batches, seed=3, call=call, max_sweeps=1)
        ost = obm.finetune(algo, batches=batches, seed=3, call=call, max_sweeps=1)
        assert st["accepted"] == ost["accepted"] > 0
        assert_same_state(bm, obm)


@pytest.mark.parametrize("batches", [1, 10])
def test_host_driven_and_device_driven_sweeps_in_turn(S, O, batches):
    V, s, d, _ = random_graph(1001, 8, 2)
    a = random_assignment(V, 60, 1)
    bm, obm = S.Blockmodel(S.Graph(V, s, d), 60, a), O.Blockmodel(O.Graph(V, s, d), 60, a)
    try:
        for call, device in enumerate([0, 1, 0, 0, 1, 1, 0]):
            S.set_option("graph_sweeps", device)
            S.finetune.run(bm, GIBBS, batches=batches, seed=5, call=call, max_sweeps=1)
            obm.finetune(GIBBS, batches=batches, seed=5, call=call, max_sweeps=1)
            assert_same_state(bm, obm)
    finally:
        S.set_option("graph_sweeps", 1)


@pytest.mark.parametrize("kind", ["learned", "collect"])
def test_learned_calls_around_a_plain_finetune(S, kind):
    V, s, d, _ = random_graph(1001, 8, 4)
    g = S.Graph(V, s, d)
    bm = S.Blockmodel(g, 50, random_assignment(V, 50, 1))
    net = S.Mlp(seed=1)

    def step(m, call):
        if kind == "collect":
            ds = S.Dataset(4 * V)
            S.learned.collect_moves(m, ds, batches=10, sweeps=1, seed=7, call=call)
            return len(ds)
        return S.learned.finetune(m, net, batches=10, seed=7, call=call, max_sweeps=1)["accepted"]

    for call in range(0, 8, 2):
        other = fresh(S, bm, g)
        assert step(bm, call) == step(other, call) > 0
        same(bm, other)
        other = fresh(S, bm, g)
        for m in (bm, other):
            S.finetune.run(m, GIBBS, batches=10, seed=7, call=call + 1, max_sweeps=1)
        same(bm, other)


@pytest.mark.parametrize("dense_max", [60, 250])
@pytest.mark.parametrize("algo", [GIBBS, HYBRID])
def test_partition_whose_search_crosses_the_storages(S, O, algo, dense_max):
    V, s, d, _ = random_graph(1001, 8, 6)
    S.set_option("dense_max_blocks", dense_max)
    try:
        out, st = S.sbp.stochastic_block_partition(S.Graph(V, s, d), algorithm=algo, batches=10, seed=11)
    finally:
        S.set_option("dense_max_blocks", 131072)
    ref, ost = O.sbp(O.Graph(V, s, d), algo=algo, batches=10, seed=11)
    assert np.array_equal(out, ref)
    for k in ("num_blocks", "visits", "accepted"):
        assert st[k] == ost[k], k


def test_finetune_after_one_that_reported_an_error(S):
    """A replay stream that ends early: the call fails after its sweeps; the blockmodel keeps their state."""
    V, s, d, _ = random_graph(1500, 8, 9)
    g = S.Graph(V, s, d)
    bm = S.Blockmodel(g, 80, random_assignment(V, 80, 1))
    for call in range(3):
        with pytest.raises(S.SbpError) as e:
            S.finetune.run(bm, GIBBS, batches=5, replay=random_records(V + V // 2, call), max_sweeps=2)
        assert e.value.code == 4
        other = fresh(S, bm, g)
        for m in (bm, other):
            S.finetune.run(m, GIBBS, batches=5, seed=2, call=call, max_sweeps=3)
        same(bm, other)


def test_a_barrier_wait_that_runs_out(S):
    """Failure detection without a GPU fault: with the shortest limit the first CTAs at a barrier of the persistent
    finetune give up, every CTA leaves, the call fails and the blockmodel is left sound."""
    V, s, d, _ = random_graph(20_000, 12, 3)
    g = S.Graph(V, s, d)
    bm = S.Blockmodel(g, 500, random_assignment(V, 500, 1))
    for call in range(3):
        S.set_option("sweep_wait_limit", 1)
        try:
            with pytest.raises(S.SbpError) as e:
                S.finetune.run(bm, GIBBS, batches=4, seed=1, call=call, max_sweeps=5)
        finally:
            S.set_option("sweep_wait_limit", 1 << 23)
        assert e.value.code == 5 and "grid barrier wait" in str(e.value)
        other = S.Blockmodel(g, 500, bm.block_assignment())
        same(bm, other)
        for algo in (GIBBS, HYBRID):
            for m in (bm, other):
                S.finetune.run(m, algo, batches=4, seed=2, call=call, max_sweeps=2)
            same(bm, other)


@pytest.mark.parametrize("algo", [GIBBS, HYBRID])
def test_finetunes_of_two_threads(S, algo):
    """Threads with handles of their own: states and counts are those of the calls one after the other."""
    def build():
        out = []
        for V, B, seed in ((20_000, 300, 1), (1001, 40, 2), (6_000, 130, 3)):
            V, s, d, _ = random_graph(V, 8, seed)
            out.append(S.Blockmodel(S.Graph(V, s, d), B, random_assignment(V, B, seed)))
        return out

    def work(bm, got):
        for call in range(8):
            st = S.finetune.run(bm, algo, batches=10, seed=4, call=call, max_sweeps=2)
            got.append([st[k] for k in ("visits", "accepted", "proposals_moved", "sweeps", "mdl")])

    alone, together = build(), build()
    want, got = [[] for _ in alone], [[] for _ in alone]
    for bm, w in zip(alone, want):
        work(bm, w)
    threads = [threading.Thread(target=work, args=x) for x in zip(together, got)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == want
    for a, b in zip(alone, together):
        same(a, b)


@pytest.mark.parametrize("B", [100, 300, 4096, 4200])   # no sums, one level of them, two
def test_a_copy_finetunes_as_its_source(S, B):
    V, s, d, _ = random_graph(4600, 8, 5)
    g = S.Graph(V, s, d)
    bm = S.Blockmodel(g, B, random_assignment(V, B, 1))
    S.finetune.run(bm, GIBBS, batches=3, seed=1, call=1, max_sweeps=1)
    twin = bm.copy()
    same(bm, twin)
    for m in (bm, twin):
        S.finetune.run(m, GIBBS, batches=3, seed=1, call=2, max_sweeps=2)
        S.finetune.run(m, 0, seed=1, call=3, max_sweeps=1)
    same(bm, twin)


@pytest.mark.parametrize("B", [1, 2, 63, 64, 65, 128, 129])
def test_block_matrix_readback(S, B):
    V, s, d, _ = random_graph(400, 5, 2)
    a = random_assignment(V, B, 1)
    pairs = np.unique(s.astype(np.int64) * V + d)
    M = np.zeros((B, B), np.int32)
    np.add.at(M, (a[pairs // V], a[pairs % V]), 1)
    assert np.array_equal(S.Blockmodel(S.Graph(V, s, d), B, a).blockmatrix(), M)
