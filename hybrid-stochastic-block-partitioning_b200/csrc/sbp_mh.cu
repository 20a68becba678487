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
// length of the chain, which grows as a group has fewer lanes.  G is chosen round by round from the
// positions that recent rounds got through.  The commit issues atomics and stores only; every
// value it needs was read by the evaluation.
#include "sbp_engine.cuh"
#include "sbp_group.cuh"
#include "sbp_steps.cuh"

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
  int kref;             // typical degree of the list
  int min_lanes;        // smallest group
  double* out;          // [0] visits [1] proposals moved [2] accepted [3] sum of accepted delta-MDL in list order
  int* status;
};

// Lanes per vertex for the next round: most positions decided per unit of time, when a round is
// expected to get through `expect` positions and its chain is a fixed part and a part per four
// neighbours of a lane (measured at 32 blocks: about 4 to 1).
__device__ __forceinline__ int mh_group_lanes(float expect, int warps, int kref) {
  int best = 32;
  float rate = 0.f;
#pragma unroll
  for (int G = 8; G <= 32; G *= 2) {
    const float passes = (float)((kref + 4 * G - 1) / (4 * G));
    const float r = fminf(expect, (float)(warps * (32 / G))) / (4.f + passes);
    if (r > rate) {
      rate = r;
      best = G;
    }
  }
  return best;
}

template <bool kDirect>
__global__ void __launch_bounds__(kMhWarps * 32, 1) k_mh_dense(const __grid_constant__ MhArgs a) {
  extern __shared__ int smem[];
  __shared__ int s_r[kMhMaxWidth], s_s[kMhMaxWidth], s_t[kMhMaxWidth];
  __shared__ double s_dS[kMhMaxWidth];
  __shared__ unsigned s_acc[2], s_moved[2];
  __shared__ int s_stop;
  const GraphView& g = a.g;
  const BlockView& bm = a.bm;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int slots = warps * a.region;
  group_tabs_init<kDirect>(smem, slots);
  if (threadIdx.x < 2) s_acc[threadIdx.x] = s_moved[threadIdx.x] = 0u;
  if (threadIdx.x == 0) s_stop = kMhMaxWidth;
  __syncthreads();
  long long visits = 0, moved = 0, accepted = 0;   // thread 0
  double sum_dS = 0.0;
  float expect = 16.f;
  bool whole_warp = false;   // the next vertex does not fit a smaller group's table
  for (int pos = 0; pos < a.n;) {
    const int G = whole_warp ? 32 : max(a.min_lanes, mh_group_lanes(expect, warps, a.kref));
    const Lanes L(G, lane);
    const int per = 32 / G, W = warps * per;
    const int w = warp * per + lane / G;
    const int share = a.region / per;
    auto tab = [&](int x) { return group_tab<kDirect>(smem, slots, (x / per) * a.region + (x % per) * share, share); };
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
      if (e.accepted) atomicOr(&s_acc[w >> 5], 1u << (w & 31));
      if (valid && e.s != e.r) atomicOr(&s_moved[w >> 5], 1u << (w & 31));
      if (!valid) atomicMin(&s_stop, w);
    }
    __syncthreads();
    const unsigned long long acc = (unsigned long long)s_acc[1] << 32 | s_acc[0];
    if (valid) {
      bool dep = false;
      for (int c = L.gl; c < w; c += G) {
        if (!(acc >> c & 1ull)) continue;
        const GroupTab<kDirect> Tc = tab(c);
        const int rc = s_r[c], sc = s_s[c];
        dep = dep || rc == e.r || rc == e.s || rc == e.t || sc == e.r || sc == e.s || sc == e.t || T.counts_of(rc) ||
              T.counts_of(sc) || (e.t >= 0 && Tc.counts_of(e.t)) || Tc.counts_of(e.r) || Tc.counts_of(e.s);
      }
      if (dep) atomicMin(&s_stop, w);
    }
    __syncthreads();
    const int stop = min(s_stop, W);
    if (threadIdx.x == 0) {
      const unsigned long long below = stop >= 64 ? ~0ull : (1ull << stop) - 1ull;
      visits += stop;
      moved += __popcll(((unsigned long long)s_moved[1] << 32 | s_moved[0]) & below);
      unsigned long long done = acc & below;
      accepted += __popcll(done);
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
          cell_add(bm, r, u, -co);
          cell_add(bm, s, u, co);
        }
        if (ci) {
          cell_add(bm, u, r, -ci);
          cell_add(bm, u, s, ci);
        }
      }
      if (L.gl == 0) {
        const int d_rr = -co_r - ci_r - e.self, d_rs = -co_s + ci_r;
        const int d_sr = co_r - ci_s, d_ss = co_s + ci_s + e.self;
        if (d_rr) cell_add(bm, r, r, d_rr);
        if (d_rs) cell_add(bm, r, s, d_rs);
        if (d_sr) cell_add(bm, s, r, d_sr);
        if (d_ss) cell_add(bm, s, s, d_ss);
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
    __threadfence_block();
    __syncthreads();
    if (threadIdx.x < 2) s_acc[threadIdx.x] = s_moved[threadIdx.x] = 0u;
    if (threadIdx.x == 0) s_stop = kMhMaxWidth;
    __syncthreads();
    whole_warp = stop == 0;   // only a vertex that did not fit stops a round at its start
    if (stop > 0) expect = 0.75f * expect + 0.25f * (stop >= W ? 2.f * (float)W : (float)stop);
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
  a.kref = std::max(1, (int)std::ceil(1.5 * list.mean_k));
  a.min_lanes = g_group_kernel == 0 ? 32 : 8;
  const bool direct = bm.B <= kSmallB;
  if (!direct) mh_cap(list.max_k);   // the degree limit of the row-hashed and the learned pass
  // a whole warp's table holds every distinct neighbour block of the largest vertex
  const int distinct = std::min(list.max_k, bm.B) + 1;
  a.region = direct ? kRegionSlots : std::max(kRegionSlots, pow2_at_least(distinct + distinct / 3));
  const int warps = (int)std::min<size_t>(kMhWarps, kSmemBudget / group_smem_bytes(direct, a.region));
  if (warps < 1) throw Error(SBP_ERR_UNSUPPORTED, "vertex degree too large for the Metropolis-Hastings kernel");
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
