// Metropolis-Hastings over a vertex list with exact sequential semantics on a dense block matrix
// (finetune::metropolis_hastings, src/finetune.cpp:412-444), one CTA, in rounds:
//   * the groups evaluate the next W vertices of the list against the current state, all at once;
//   * every accepted vertex up to the first one that depends on an earlier accepted vertex of the
//     round commits, and the list position moves there; the rest is evaluated again next round.
// Random records depend only on (vertex, sweep), so evaluating again changes nothing and the chain
// is the sequential one.
//
// What a commit c changes: cells in rows and columns r_c, s_c towards its neighbour blocks, the
// degrees of r_c and s_c, and its own assignment (a neighbour that moved leaves r_c in the table of
// the vertex that saw it).  Vertex w read its neighbours' blocks, row and column t_w, cells towards
// r_w, s_w and its neighbour blocks, and their degrees.  So w is independent of c when r_c, s_c
// are none of r_w, s_w, t_w and not in w's table, and t_w, r_w, s_w are not in c's table.  All
// accepted vertices before the first dependent one commit, so that one is found without a scan:
// every group tests itself against the accepted ones before it, a lane each.
//
// A round is one chain of dependent loads (a few microseconds) whatever its width, and a pass is
// the rounds its accepted moves force: the round's width W = warps * 32 / G trades against the
// length of the chain, which grows as a group has fewer lanes.  G is chosen round by round from how far
// recent rounds got before a dependence stopped them.  The commit issues atomics and stores only; every
// value it needs was read by the evaluation.
#include "sbp_engine.cuh"
#include "sbp_group.cuh"
#include "sbp_steps.cuh"

#include <limits>

namespace sbpb {
namespace {

constexpr int kMhWarps = 16;
constexpr int kMhMaxWidth = kMhWarps * 4;

struct MhArgs {
  GraphView g;
  BlockView bm;
  const int4* recs;     // vertex records in list order
  int n;
  RngParams rng;
  int sweep;
  int region;           // table slots of a warp
  float m16, m8;        // groups of 16 (8) lanes from this many positions between dependences on
  double* out;          // [0] visits [1] proposals moved [2] accepted [3] sum of accepted delta-MDL in list order
  int* status;
};

template <bool kDirect>
__global__ void __launch_bounds__(kMhWarps * 32, 1) k_mh_dense(const __grid_constant__ MhArgs a) {
  extern __shared__ int smem[];
  __shared__ int s_r[kMhMaxWidth], s_s[kMhMaxWidth], s_t[kMhMaxWidth];
  __shared__ double s_dS[kMhMaxWidth];
  __shared__ unsigned s_acc[kMhWarps], s_moved[kMhWarps];   // a bit per group of the warp
  __shared__ int s_first[kMhWarps];                         // the warp's first invalid or dependent position
  const GraphView& g = a.g;
  const BlockView& bm = a.bm;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int slots = warps * a.region;
  group_tabs_init<kDirect>(smem, slots);
  __syncthreads();
  long long visits = 0, moved = 0, accepted = 0;   // warp 0; sum_dS its first lane
  double sum_dS = 0.0;
  float decided = 16.f, stops = 1.f;   // of recent rounds: positions got through, dependences met
  bool whole_warp = false;   // the next vertex does not fit a smaller group's table
  for (int pos = 0; pos < a.n;) {
    const int G = whole_warp || decided < a.m16 * stops ? 32 : decided < a.m8 * stops ? 16 : 8;
    const Lanes L(G, lane);
    const int lg = G == 32 ? 0 : G == 16 ? 1 : 2, per = 1 << lg, W = warps * per;   // groups of a warp, of the CTA
    const int w = warp * per + (lane >> (5 - lg));
    const int share = a.region >> lg;
    auto tab = [&](int x) { return group_tab<kDirect>(smem, slots, x * share, share); };   // group x's
    const GroupTab<kDirect> T = tab(w);
    int4 rec = make_int4(0, 0, 0, 0);
    bool valid = pos + w < a.n;
    if (valid) rec = __ldg(a.recs + pos + w);
    if (!kDirect && valid && G < 32 && min(rec.z + (rec.w >> 1), bm.B) * 4 > share * 3) valid = false;
    uint4 x = make_uint4(0, 0, 0, 0);
    if (valid)
      x = draw_record(a.rng, (uint32_t)rec.x, (uint32_t)a.sweep, 0u, (long long)a.sweep * g.V + rec.x, a.status);
    const GroupEval e = group_evaluate<kDirect, Store::kDense>(g, bm, T, valid, rec, a.rng.moves != 0, x, L, a.status);
    if (L.gl == 0) {
      s_r[w] = e.r;
      s_s[w] = e.s;
      s_t[w] = e.t;
      s_dS[w] = e.dS;
    }
    const unsigned firsts = G == 32 ? 1u : G == 16 ? 0x10001u : 0x1010101u;   // the groups' first lanes
    auto squeeze = [&](unsigned m) {   // one bit per group, from the bits of their first lanes
      m &= firsts;
      return (m | m >> (G - 1) | (G == 8 ? m >> (2 * (G - 1)) | m >> (3 * (G - 1)) : 0u)) & (unsigned)((1 << per) - 1);
    };
    const unsigned acc_w = squeeze(__ballot_sync(kFull, e.accepted));
    const unsigned moved_w = squeeze(__ballot_sync(kFull, valid && e.s != e.r));
    if (lane == 0) {
      s_acc[warp] = acc_w;
      s_moved[warp] = moved_w;
    }
    __syncthreads();
    auto gather = [&](const unsigned* bits) {   // the warps' bits as one mask over the round's positions
      const unsigned m = lane < warps ? bits[lane] : 0u;
      const unsigned long long x = (unsigned long long)m << (lane < warps ? lane * per : 0);
      return (unsigned long long)__reduce_or_sync(kFull, (unsigned)(x >> 32)) << 32 | __reduce_or_sync(kFull, (unsigned)x);
    };
    const unsigned long long acc = gather(s_acc);
    bool halt = !valid;
    if (valid) {
      for (int c = L.gl; c < w; c += G) {
        if (!(acc >> c & 1ull)) continue;
        const GroupTab<kDirect> Tc = tab(c);
        const int rc = s_r[c], sc = s_s[c], tw = e.t >= 0 ? e.t : e.r;
        const int p0 = Tc.peek(e.r), p1 = Tc.peek(e.s), p2 = Tc.peek(tw), p3 = T.peek(rc), p4 = T.peek(sc);
        halt |= (rc == e.r) | (rc == e.s) | (rc == e.t) | (sc == e.r) | (sc == e.s) | (sc == e.t) | Tc.holds(e.r, p0) |
                Tc.holds(e.s, p1) | Tc.holds(tw, p2) | T.holds(rc, p3) | T.holds(sc, p4);
      }
    }
    const unsigned halted = __ballot_sync(kFull, halt);
    if (lane == 0) s_first[warp] = halted ? warp * per + ((__ffs(halted) - 1) >> (5 - lg)) : kMhMaxWidth;
    __syncthreads();
    const int stop = min(W, (int)__reduce_min_sync(kFull, (unsigned)(lane < warps ? s_first[lane] : kMhMaxWidth)));
    if (warp == 0) {
      const unsigned long long below = stop >= 64 ? ~0ull : (1ull << stop) - 1ull;
      const unsigned long long mv = gather(s_moved);
      unsigned long long done = acc & below;
      visits += stop;
      moved += __popcll(mv & below);
      accepted += __popcll(done);
      if (lane == 0)
        for (; done; done &= done - 1ull) sum_dS += s_dS[__ffsll((long long)done) - 1];   // in list order
    }
    if (e.accepted && w < stop) {
      // Blockmodel::move_vertex (src/blockmodel/blockmodel.cpp:344-360): lanes take the non-corner
      // cells, lane 0 the corners, the assignment and the degrees
      const int r = e.r, s = e.s;
      const int co_r = e.wr & kCountMask, ci_r = (e.wr >> kInShift) & kCountMask;
      const int co_s = e.ws & kCountMask, ci_s = (e.ws >> kInShift) & kCountMask;
      for (int j = L.gl; j < e.n; j += G) {
        const int slot = T.list[j];
        const int u = T.key_of(slot);
        if (u == r || u == s) continue;
        const unsigned wu = T.w[slot];
        const int co = wu & kCountMask, ci = (wu >> kInShift) & kCountMask;
        if (co) {
          cell_add<Store::kDense>(bm, r, u, -co);
          cell_add<Store::kDense>(bm, s, u, co);
        }
        if (ci) {
          cell_add<Store::kDense>(bm, u, r, -ci);
          cell_add<Store::kDense>(bm, u, s, ci);
        }
      }
      if (L.gl == 0) {
        const int d_rr = -co_r - ci_r - e.self, d_rs = -co_s + ci_r;
        const int d_sr = co_r - ci_s, d_ss = co_s + ci_s + e.self;
        if (d_rr) cell_add<Store::kDense>(bm, r, r, d_rr);
        if (d_rs) cell_add<Store::kDense>(bm, r, s, d_rs);
        if (d_sr) cell_add<Store::kDense>(bm, s, r, d_sr);
        if (d_ss) cell_add<Store::kDense>(bm, s, s, d_ss);
        bm.b[e.v] = s;
        const int kin_self = e.k_in + e.self;
        const int out_r = e.dout_r - e.k_out, out_s = e.dout_s + e.k_out;
        const int in_r = e.din_r - kin_self, in_s = e.din_s + kin_self;
        bm.d_out[r] = out_r;
        bm.d_out[s] = out_s;
        bm.d_in[r] = in_r;
        bm.d_in[s] = in_s;
        // move_vertex reads the already-updated diagonal and adds the delta again
        set_degree(bm, r, out_r + in_r - (e.M_rr + 2 * d_rr));
        set_degree(bm, s, out_s + in_s - (e.M_ss + 2 * d_ss));
      }
    }
    T.clear(e.n, L);
    __syncthreads();
    whole_warp = stop == 0;   // only a vertex that did not fit stops a round at its start
    decided = 0.9375f * decided + (float)stop;
    stops = 0.9375f * stops + (stop < W ? 1.f : 0.f);
    pos += stop;
  }
  if (threadIdx.x == 0) {
    a.out[0] = (double)visits;
    a.out[1] = (double)moved;
    a.out[2] = (double)accepted;
    a.out[3] = sum_dS;
  }
}

}  // namespace

MhResult mh_pass_dense(SbpBlockmodel& bm, const SbpGraph& g, const VertexList& list, const RngParams& rng, int sweep) {
  Context& c = Context::get();
  MhArgs a;
  a.g = g.view();
  a.bm = bm.view();
  a.recs = list.recs;
  a.n = list.n;
  a.rng = rng;
  a.sweep = sweep;
  a.out = c.mh_out;
  a.status = c.status;
  const bool direct = bm.B <= kSmallB;
  if (!direct) mh_cap(list.max_k);   // the degree limit of the row-hashed and the learned pass
  // a whole warp's table holds every distinct neighbour block of the largest vertex
  const int distinct = std::min(list.max_k, bm.B) + 1;
  a.region = direct ? kRegionSlots : std::max(kRegionSlots, pow2_at_least(distinct + distinct / 3));
  const int warps = (int)std::min<size_t>(kMhWarps, kSmemBudget / group_smem_bytes(direct, a.region));
  if (warps < 1) throw Error(SBP_ERR_UNSUPPORTED, "vertex degree too large for the Metropolis-Hastings kernel");
  // Microseconds of a round, to about a fifth (graphs of 2,000 to 20,000 vertices, 4 to 200 neighbours, 8 to
  // 1,900 blocks): a fixed part, a part per four neighbours of a lane, and what the dependence tests of
  // 64 or 32 positions add, more with hash tables, whose look-ups are chains.  With 300 blocks and 20
  // neighbours 16.3, 8.7 and 6.9; taken for equal, as they were, widths that dependences did not let
  // commit were evaluated: two sweeps of 20,000 vertices at 129 blocks 174 ms against 70.
  const int kref = std::max(1, (int)std::ceil(1.5 * list.mean_k));   // typical degree of the list
  const float wide[3] = {direct ? 2.6f : 9.f, direct ? 0.9f : 3.f, 0.f};
  float cost[3];   // groups of 8, 16 and 32 lanes
  for (int i = 0; i < 3; ++i) {
    const int four_g = 4 * (8 << i);
    cost[i] = 5.f + (direct ? 1.f : 2.5f) * (float)((kref + four_g - 1) / four_g) + wide[i];
  }
  // When a dependence comes after m positions on average, a round of width W gets through m (1 - exp(-W / m))
  // of them: the wider round is the better one from some m on.
  auto from = [&](int i, int j) {
    for (float m = 1.f; m < 4096.f; m *= 1.05f)
      if ((1.f - std::exp(-(float)(warps << (2 - i)) / m)) * cost[j] >
          (1.f - std::exp(-(float)(warps << (2 - j)) / m)) * cost[i])
        return m;
    return std::numeric_limits<float>::infinity();
  };
  a.m16 = std::min(from(1, 2), from(0, 2));
  a.m8 = std::max(from(0, 1), from(0, 2));
  if (g_group_kernel == 0) a.m16 = std::numeric_limits<float>::infinity();
  const size_t smem = group_smem_bytes(direct, a.region * warps);
  const auto k = direct ? k_mh_dense<true> : k_mh_dense<false>;
  set_smem_limit((const void*)k, smem);
  k<<<1, warps * 32, smem, c.stream>>>(a);
  SBP_CHECK_LAUNCH();
  double out[4];
  SBP_CUDA(SBP_COPY_ASYNC(out, c.mh_out, sizeof(out), cudaMemcpyDeviceToHost, c.stream));
  c.sync();
  MhResult res;
  res.visits = (long long)out[0];
  res.moved = (long long)out[1];
  res.accepted = (long long)out[2];
  res.sum_dS = out[3];
  return res;
}

}  // namespace sbpb
