"""The learned proposal's kernels at the sizes where their splits change: more distinct neighbour blocks than a warp has
lanes, row counts that leave half a warp or a tile partly empty, and more tiles than the device has CTAs."""
import numpy as np
import pytest

import learned_oracle as LO
from conftest import random_assignment, random_graph, random_records
from test_gpu_finetune_edges import graph_of_degrees
from test_gpu_learned import oracle_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [5, 33, 400])   # degrees up to 700: up to 400 distinct blocks
def test_slots_of_many_blocks(S, B):
    V = 1200
    s, d = graph_of_degrees(V, B)
    g = S.Graph(V, s, d)
    bm = S.Blockmodel(g, B, random_assignment(V, B, B))
    go = LO.Graph(V, s, d)
    b, d_out, d_in = oracle_state(bm, go)
    verts = np.arange(60, dtype=np.int32)
    F, slots, nv = S.learned.vertex_features(bm, verts)
    for v in verts:
        f, sl, *_ = LO.vertex_features(go, b, bm.B, d_out, d_in, v)
        assert nv[v] == len(sl)
        assert slots[v, :nv[v]].tolist() == [x[0] for x in sl]
        assert np.all(np.abs(F[v] - f) <= 2.0**-7 * np.abs(f) + 1e-12)   # one BF16 step (log1pf's last bit)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 129])   # eight rows a CTA of the draw
def test_draw_of_part_of_a_block(S, n):
    """Each row's draw, q and decision are those of the row among all others."""
    V, s, d, _ = random_graph(300, 6, 4)
    bm = S.Blockmodel(S.Graph(V, s, d), 20, random_assignment(V, 20, 4))
    mlp = S.Mlp(seed=2)
    verts, rec = np.arange(V, dtype=np.int32), random_records(V, 9)
    every = S.learned.evaluate(bm, mlp, verts, rec)
    some = S.learned.evaluate(bm, mlp, verts[:n], rec[:n])
    for a, b in zip(every, some):
        assert np.array_equal(a[:n], b)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 18_944, 18_945, 40_000])   # 128 rows a tile, one CTA an SM
def test_network_rows_are_independent(S, n):
    mlp = S.Mlp(seed=5)
    X = np.random.default_rng(n).normal(size=(n, 64)).astype(np.float32)
    got = mlp.forward(X)
    for i in range(0, n, max(1, n // 5)):
        assert np.array_equal(got[i:i + 100], mlp.forward(X[i:i + 100]))
    assert np.array_equal(got[-1:], mlp.forward(X[-1:]))
