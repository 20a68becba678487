"""The arithmetic of the vertex-move delta-MDL for g(a) - g(b), g(x) = x log x, of integer counts (dxlogx_int in
csrc/sbp_device.cuh): a table of g as (hi, lo) doubles and (hi_a - hi_b) + (lo_a - lo_b).  On the CPU the formula is
restated over 40-digit decimals; on the GPU the device's own table is checked through the delta-MDL of evaluated moves."""
import decimal

import numpy as np
import pytest

from conftest import random_graph, random_records

TABLE = 1 << 20
decimal.getcontext().prec = 45


def g_exact(x):
    return decimal.Decimal(x) * decimal.Decimal(x).ln() if x > 1 else decimal.Decimal(0)


def table_entry(x):
    g = g_exact(x)
    hi = float(g)
    return hi, float(g - decimal.Decimal(hi))


def pairs():
    rng = np.random.default_rng(7)
    a = np.concatenate([np.arange(0, 40), rng.integers(0, 300, 600), rng.integers(0, 30_000, 600),
                        rng.integers(0, TABLE, 600), [TABLE - 1, TABLE - 2, 1, 0, 2, 1]])
    d = np.concatenate([rng.integers(-3, 4, 40), rng.integers(-200, 201, 1200), rng.integers(-3000, 3001, 600),
                        [-1, 1, -1, 1, -2, 1]])
    ok = (a + d >= 0) & (a + d < TABLE) & (d != 0)
    return a[ok], (a + d)[ok]


def test_difference_of_table_entries_is_accurate():
    worst = 0.0
    for a, b in zip(*(x.tolist() for x in pairs())):
        (ha, la), (hb, lb) = table_entry(a), table_entry(b)
        got = (ha - hb) + (la - lb)
        ref = g_exact(a) - g_exact(b)
        if ref == 0:
            assert got == 0.0   # g(0) = g(1)
            continue
        worst = max(worst, abs(float((decimal.Decimal(got) - ref) / ref)))
    # half an ulp each for the difference of the high parts and the final sum, and the low parts' rounding
    assert worst <= 2.3e-16


@pytest.mark.gpu
@pytest.mark.parametrize("B", [2, 7, 128, 129, 400])
def test_device_table_through_delta_mdl(S, B):
    """delta-MDL of evaluated moves against 45-digit decimals: within the rounding of a sum of its terms."""
    V, src, dst, _ = random_graph(1500, 5, 31)
    assignment = np.random.default_rng(3).integers(0, B, V).astype(np.int32)
    assignment[:B] = np.arange(B)
    bm = S.Blockmodel(S.Graph(V, src, dst), B, assignment)
    M = bm.blockmatrix().astype(np.int64)
    keep = np.unique(src.astype(np.int64) * V + dst)
    src, dst = keep // V, keep % V
    do, di = M.sum(1), M.sum(0)
    vs = np.random.default_rng(4).permutation(V)[:60].astype(np.int32)
    s, dS, _, _ = bm.evaluate_vertices(vs, random_records(60, 5))
    for v, sv, got in zip(vs, s, dS):
        r = assignment[v]
        if sv == r:
            continue
        out, inn = assignment[dst[(src == v) & (dst != v)]], assignment[src[(dst == v) & (src != v)]]
        self_loop = int(((src == v) & (dst == v)).any())
        cells = {}
        for row, col, n in ([(r, u, -1) for u in out] + [(sv, u, 1) for u in out] + [(u, r, -1) for u in inn]
                            + [(u, sv, 1) for u in inn] + [(r, r, -self_loop), (sv, sv, self_loop)]):
            cells[row, col] = cells.get((row, col), 0) + n
        # a present (r,s) / (s,r) entry with net change 0 and a count is counted twice: skip those moves here
        if any(cells.get(x) == 0 and M[x] > 0 for x in ((r, sv), (sv, r))):
            continue
        k_out, k_in = len(out) + self_loop, len(inn) + self_loop
        terms = [g_exact(int(M[x])) - g_exact(int(M[x] + n)) for x, n in cells.items()]
        terms += [g_exact(int(d[x]) + n) - g_exact(int(d[x])) for d, k in ((do, k_out), (di, k_in))
                  for x, n in ((r, -k), (sv, k))]
        ref, scale = sum(terms), sum(abs(t) for t in terms)
        # each term to 2^-52, a tree of at most 12 additions
        assert abs(decimal.Decimal(float(got)) - ref) <= scale * decimal.Decimal(13 * 2.0 ** -52)
