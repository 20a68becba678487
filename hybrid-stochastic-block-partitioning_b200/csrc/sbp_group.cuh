// Evaluation of a vertex move by a group of lanes of a warp (the same proposal, Hastings
// correction, delta-MDL and accept test as evaluate_vertex in sbp_device.cuh; reference
// src/common.cpp:131-192, src/entropy.cpp:296-401, 495-557, src/finetune.cpp:19-29), on either
// storage of the block matrix.
//
// A visit is a chain of about a dozen dependent memory round trips with little work between
// them, so what counts is how many visits are in flight and how few instructions each costs:
//   * a group of G = 8, 16 or 32 lanes evaluates one vertex, so a warp carries 32 / G of them and
//     pays the scalar part of a visit (random record, walk, reductions, accept) once for all;
//   * G is chosen per task from the vertex's degree, at most four neighbours a lane; a group owns 16 G
//     slots of its warp's table region.  Every loop runs to the largest trip count of the warp's
//     groups, so the vertices of a batch are ordered by degree;
//   * a vertex's CSR ranges come as one 16-byte record and its out- and in-neighbours as one list;
//   * the loads of a step are issued together, and what does not depend on the proposal before
//     the walk that picks it.
// Summation orders differ from evaluate_vertex, so delta-MDL and the Hastings factor agree with it
// to rounding; every integer input is the same.
#pragma once
#include "sbp_device.cuh"

namespace sbpb {

// One batch of an asynchronous-Gibbs plan: its light vertices, by degree descending, and its
// heavy ones; n32 / n16 of the light ones are too large for a group of 16 / 8 lanes.
struct BatchDesc {
  int light_begin, light_n, heavy_begin, heavy_n;
  int n32, n16;
};

constexpr int kRegionSlots = 512;   // table slots of one warp, shared by its groups
constexpr int kGroupWarps = 8;      // warps per CTA
constexpr int kGroupThreads = 32 * kGroupWarps;
__device__ __forceinline__ double group_sum(double v, const Lanes& L) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    if (o < L.G) v += __shfl_xor_sync(kFull, v, o);
  return v;
}
// Neighbour-block histogram of one group.  Slot words hold out count | in count << 15 | presence <<
// 30; the list holds the slots in use.  kDirect (B <= kSmallB): the slot is the block; otherwise an
// open-addressing table of mask + 1 slots.
constexpr unsigned kInShift = 15;
constexpr unsigned kCountMask = (1u << 15) - 1;
constexpr unsigned kPresent = 1u << 30;

template <bool kDirect>
struct GroupTab {
  int* keys;               // block of each slot, -1 = empty (unused when direct)
  unsigned* w;
  unsigned short* list;
  int mask;
  __device__ __forceinline__ unsigned home(int key) const { return ((unsigned)key * 2654435761u) >> 16 & (unsigned)mask; }
  // Add `delta` to the word of `key`, whose home slot h was tried with the result `k` (the slot's key
  // before the try); returns the slot when this lane made it, else -1.
  __device__ __forceinline__ int finish_add(int key, unsigned h, int k, unsigned delta, int* status) const {
    for (int probe = 0; k != -1 && k != key; ++probe) {
      if (probe == mask) {
        atomicOr(status, kErrTableFull);
        return -1;
      }
      h = (h + 1) & (unsigned)mask;
      k = atomicCAS(keys + h, -1, key);
    }
    atomicAdd(w + h, delta);
    return k == -1 ? (int)h : -1;
  }
  // The same for a key not tried yet.
  __device__ __forceinline__ int add(int key, unsigned delta, int* status) const {
    if constexpr (kDirect) {
      return atomicAdd(w + key, delta) == 0u ? key : -1;
    } else {
      const unsigned h = home(key);
      return finish_add(key, h, atomicCAS(keys + h, -1, key), delta, status);
    }
  }
  __device__ __forceinline__ unsigned counts_of(int key) const {
    if constexpr (kDirect) {
      return w[key];
    } else {
      unsigned h = home(key);
      for (int probe = 0; probe <= mask; ++probe) {
        const int k = keys[h];
        if (k == key) return w[h];
        if (k == -1) return 0u;
        h = (h + 1) & (unsigned)mask;
      }
      return 0u;
    }
  }
  // What the home slot of `key` holds, and from it whether the table holds the key (a slot in use has
  // a nonzero word): apart, so that several look-ups go out together.
  __device__ __forceinline__ int peek(int key) const { return kDirect ? (int)w[key] : keys[home(key)]; }
  __device__ __forceinline__ bool holds(int key, int peeked) const {
    if constexpr (kDirect) return peeked != 0;
    else return peeked == key || (peeked != -1 && counts_of(key) != 0u);
  }
  __device__ __forceinline__ int key_of(int slot) const { return kDirect ? slot : keys[slot]; }
  // Empty the n slots in use.
  __device__ __forceinline__ void clear(int n, const Lanes& L) const {
    __syncwarp();
    for (int j = L.gl; j < n; j += L.G) {
      const int slot = list[j];
      w[slot] = 0u;
      if constexpr (!kDirect) keys[slot] = -1;
    }
    __syncwarp();
  }
};

// Shared memory of a CTA of kGroupWarps warps: one word and one list entry per slot (and a key
// unless direct), `slots` slots in all.
__host__ __device__ inline size_t group_smem_bytes(bool direct, int slots) {
  return (size_t)slots * (direct ? 6 : 10);
}
template <bool kDirect>
__device__ __forceinline__ GroupTab<kDirect> group_tab(int* smem, int slots, int first, int count) {
  GroupTab<kDirect> T;
  T.w = reinterpret_cast<unsigned*>(smem) + first;
  T.keys = kDirect ? nullptr : smem + slots + first;
  T.list = reinterpret_cast<unsigned short*>(smem + (kDirect ? 1 : 2) * slots) + first;
  T.mask = count - 1;
  return T;
}
template <bool kDirect>
__device__ __forceinline__ void group_tabs_init(int* smem, int slots) {
  for (int i = threadIdx.x; i < slots; i += blockDim.x) {
    smem[i] = 0;
    if (!kDirect) smem[slots + i] = -1;
  }
}

// Result of one group's evaluation; every lane of the group holds it.
struct GroupEval {
  int v, r, s, t;        // vertex, its block, proposed block, the proposal's neighbour block (-1: none)
  int k_out, k_in, self;
  int n;                 // table slots in use
  bool valid, accepted;
  double dS;
  // what a commit needs of the state the move was evaluated against (set when s != r)
  unsigned wr, ws;       // histogram words of r and s
  int M_rr, M_ss, dout_r, dout_s, din_r, din_s;
};

// A vertex of a batch: (vertex, first neighbour in the joint list, out-degree incl. the self loop,
// in-degree without it << 1 | self loop).
__device__ __forceinline__ int4 vertex_record(const GraphView& g, int v) {
  const int o0 = g.out_ptr[v], i0 = g.in_ptr[v];
  return make_int4(v, (int)((unsigned)o0 + (unsigned)i0), g.out_ptr[v + 1] - o0,
                   (g.in_ptr[v + 1] - i0) << 1 | (int)g.self[v]);
}

// Row x of M and of its transpose, for look-ups of (M[x, u], M[u, x]): the row of pairs (dense), or
// the two hashed rows with their places and masks read once.
template <Store ST>
struct RowRef {
  const int2* p;
  __device__ __forceinline__ RowRef(const BlockView& bm, int x) : p(bm.P + (size_t)x * bm.ld) {}
  template <int N>   // on[] masks the look-ups; all N in flight together
  __device__ __forceinline__ void get(const BlockView&, const int (&u)[N], const bool (&on)[N], int2 (&m)[N]) const {
#pragma unroll
    for (int h = 0; h < N; ++h) m[h] = on[h] ? ldv<ST>(p + u[h]) : make_int2(0, 0);
  }
};
template <>
struct RowRef<Store::kHashed> {
  long long rb, cb;
  int rm, cm;
  __device__ __forceinline__ RowRef(const BlockView& bm, int x)
      : rb(bm.rbase[x]), cb(bm.cbase[x]), rm(bm.rmask[x]), cm(bm.cmask[x]) {}
  // The count of column u from the first slot probed, e, on.
  static __device__ __forceinline__ int follow(const int2* slot, long long base, int mask, int u, int2 e) {
    unsigned h = slot_hash(u) & (unsigned)mask;
    for (int probe = 0; probe <= mask; ++probe) {
      if (e.x == u) return e.y;
      if (e.x == -1) return 0;
      h = (h + 1) & (unsigned)mask;
      e = slot[base + h];
    }
    return 0;
  }
  template <int N>
  __device__ __forceinline__ void get(const BlockView& bm, const int (&u)[N], const bool (&on)[N], int2 (&m)[N]) const {
    int2 a[N], b[N];
#pragma unroll
    for (int h = 0; h < N; ++h) {
      a[h] = b[h] = make_int2(-1, 0);
      if (on[h]) {
        a[h] = bm.rslot[rb + (slot_hash(u[h]) & (unsigned)rm)];
        b[h] = bm.cslot[cb + (slot_hash(u[h]) & (unsigned)cm)];
      }
    }
#pragma unroll
    for (int h = 0; h < N; ++h)
      m[h] = on[h] ? make_int2(follow(bm.rslot, rb, rm, u[h], a[h]), follow(bm.cslot, cb, cm, u[h], b[h]))
                   : make_int2(0, 0);
  }
};
template <Store ST>
__device__ __forceinline__ int2 row_pair(const RowRef<ST>& row, const BlockView& bm, int u) {
  const int uu[1] = {u};
  const bool on[1] = {true};
  int2 m[1];
  row.get(bm, uu, on, m);
  return m[0];
}

// A difference of table entries that may lie beyond the table, out of line to keep the evaluation's
// code small.
static __device__ __noinline__ double dxlogx_wide(const double2* __restrict__ gt, int a, int b) {
  if ((unsigned)a < (unsigned)kXlogxTable && (unsigned)b < (unsigned)kXlogxTable) {
    const double2 ga = __ldg(gt + a), gb = __ldg(gt + b);
    return (ga.x - gb.x) + (ga.y - gb.y);
  }
  return dxlogx_far(a, b);
}

// Accept test u <= min(1, exp(-3 dS) H), H = bwd / fwd (1 for a vertex without neighbours).  A
// single-precision estimate decides wherever it is further from u than its error (under 1e-4
// relative) can reach; only the rest, about one visit in a thousand, takes the FP64 exponential
// and division, a chain of some 800 cycles.  The decision is the FP64 test's in every case.
static __device__ __noinline__ bool accept_exact(double x, double H, double u) {
  double ap = exp(x) * H;
  ap = ap >= 1.0 ? 1.0 : ap;
  return u <= ap;
}
__device__ __forceinline__ bool accept_move(double dS, double fwd, double bwd, bool alone, double u) {
  const double x = -3.0 * dS;
  const float xf = (float)x, hf = alone ? 1.0f : __fdividef((float)bwd, (float)fwd);
  if (hf > 1e-6f && hf < 1e6f) {
    if (xf < -80.0f) {
      if (u > 1e-20) return false;
    } else if (xf > 80.0f) {
      if (u <= 1.0) return true;
    } else {
      const float af = __expf(xf) * hf, uf = (float)u;
      if (uf > af * 1.001f) return false;
      if (uf < af * 0.999f && u <= 1.0) return true;
    }
  }
  return accept_exact(x, alone ? 1.0 : bwd / fwd, u);
}

// Evaluate the vertex of `rec` (groups with `valid`) against the blockmodel with random record x:
// gather its neighbour blocks into the group's table (left filled: res.n slots; the caller clears
// it), propose, delta-MDL, Hastings, accept.  Every lane of the warp calls it.
//
// A lane holds up to four neighbours, and up to four table entries, at a time, so the loads of a
// step are all in flight together: the classes of group_max_k give a group four neighbours a lane
// at most (a vertex beyond the largest class takes several rounds).  Row r of the entries is
// fetched before the walk, which does not depend on it.
// kAnyB: hash tables with either walk, for a kernel that serves blockmodels of any size.
template <bool kDirect, Store ST, bool kAnyB = false>
__device__ __forceinline__ GroupEval group_evaluate(const GraphView& g, const BlockView& bm, const GroupTab<kDirect>& T,
                                                    bool valid, int4 rec, bool given, uint4 x, const Lanes& L,
                                                    int* status, int* bins = nullptr) {
  const int B = bm.B;
  GroupEval res;
  res.valid = valid;
  res.accepted = false;
  res.dS = 0.0;
  const int v = res.v = rec.x;
  const int k_out = res.k_out = valid ? rec.z : 0, k_in = res.k_in = valid ? rec.w >> 1 : 0;
  const int self = res.self = valid ? rec.w & 1 : 0;
  const int k = k_out + k_in;
  const int* nbr = g.adj + (unsigned)rec.y;
  const bool walk = valid && !given && k > 0;
  // 1. the neighbour-block histogram, and the block of the proposal's neighbour with its degrees
  int r = 0, t = 0, dot = 0, dit = 0, n = 0;
  const int pick = walk ? (int)scale32(x.x, k) : -1;
  const int kmax = (int)__reduce_max_sync(kFull, (unsigned)k);
  for (int e0 = 0; e0 == 0 || e0 < kmax; e0 += 4 * L.G) {
    int u[4], bu[4];
    int ut = -1;
    if (e0 == 0 && walk) ut = __ldg(nbr + pick);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int e = e0 + j * L.G + L.gl;
      u[j] = e < k ? __ldg(nbr + e) : -1;
    }
    if (e0 == 0) {
      if (valid) r = ldv<ST>(bm.b + v);
      if (walk) t = ldv<ST>(bm.b + ut);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) bu[j] = u[j] >= 0 ? ldv<ST>(bm.b + u[j]) : -1;
    if (e0 == 0 && walk) {
      dot = ldv<ST>(bm.d_out + t);
      dit = ldv<ST>(bm.d_in + t);
    }
    // the first probe of all four together: their latencies overlap
    unsigned h[4];
    int first[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int e = e0 + j * L.G + L.gl;
      if (u[j] == v && e < k_out) u[j] = -1;   // the self loop
      if constexpr (!kDirect) {
        h[j] = T.home(bu[j]);
        first[j] = u[j] >= 0 ? atomicCAS(T.keys + h[j], -1, bu[j]) : -1;
      } else {
        first[j] = u[j] >= 0 ? (int)atomicAdd(T.w + bu[j], e < k_out ? 1u : 1u << kInShift) : -1;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (e0 + j * L.G >= kmax) break;   // warp-uniform
      const int e = e0 + j * L.G + L.gl;
      int made = -1;
      if (u[j] >= 0) {
        if constexpr (kDirect) made = first[j] == 0 ? bu[j] : -1;
        else made = T.finish_add(bu[j], h[j], first[j], e < k_out ? 1u : 1u << kInShift, status);
      }
      const unsigned fresh = __ballot_sync(kFull, made >= 0) & L.gmask;
      if (made >= 0) T.list[n + __popc(fresh & ((1u << L.lane) - 1u))] = (unsigned short)made;
      n += __popc(fresh);
    }
  }
  res.r = r;
  if (__any_sync(kFull, self)) {   // the self loop only marks r present
    int made = -1;
    if (self && L.gl == 0) made = T.add(r, kPresent, status);
    const unsigned fresh = __ballot_sync(kFull, made >= 0) & L.gmask;
    if (made >= 0) T.list[n] = (unsigned short)made;
    n += __popc(fresh);
  }
  __syncwarp();
  res.n = n;
  res.t = walk ? t : -1;
  // this lane's first entries and what of them depends on r alone
  const RowRef<ST> Pr(bm, r);
  int u[4];
  unsigned wu[4];
  bool on[4];
  int2 m_ru[4];
  double inv[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const int j = L.gl + h * L.G;
    const int slot = j < n ? T.list[j] : -1;
    u[h] = slot >= 0 ? T.key_of(slot) : r;
    wu[h] = slot >= 0 ? T.w[slot] : 0u;
    on[h] = wu[h] != 0u;
  }
#pragma unroll
  for (int h = 0; h < 4; ++h) inv[h] = on[h] ? ldv<ST>(bm.inv_d + u[h]) : 0.0;
  Pr.get(bm, u, on, m_ru);
  int M_rr = 0, dout_r = 0, din_r = 0;
  if (valid) {
    M_rr = row_pair(Pr, bm, r).x;
    dout_r = ldv<ST>(bm.d_out + r);
    din_r = ldv<ST>(bm.d_in + r);
  }
  const unsigned wr = T.counts_of(r);
  // 2. the proposal: the multinomial over row t of M, then column t (ascending)
  int s = r;
  {
    const long long target = scale32(x.y, (long long)dot + (long long)dit);
    const bool in_col = target >= dot;
    const int tg = (int)(in_col ? target - dot : target);
    int found = -1;
    if constexpr (ST == Store::kHashed) {   // the whole warp walks for its groups in turn
      for (int first = 0; first < 32; first += L.G) {
        if (!__shfl_sync(kFull, walk, first)) continue;
        const int tt = __shfl_sync(kFull, t, first), goal = __shfl_sync(kFull, tg, first);
        const bool cc = __shfl_sync(kFull, in_col, first);
        const int at = warp_select_hashed(cc ? bm.cbase : bm.rbase, cc ? bm.cmask : bm.rmask, cc ? bm.cslot : bm.rslot,
                                          tt, B, goal, L.lane, bins);
        __syncwarp();
        if (L.gbase == first) found = at;
      }
    } else {
      if (kDirect || (kAnyB && B <= kSmallB)) found = walk_row<ST>(bm, t, in_col, tg, walk, L);
      else found = walk_tree<ST>(bm, t, in_col, tg, walk, L);
    }
    if (walk) {
      s = found;
      if (s < 0 || s >= B) {
        if (L.gl == 0) atomicOr(status, kErrScan);
        s = r;
      }
    } else if (valid && given) {
      s = (int)x.x;
      if (s < 0 || s >= B) {   // a visit the stream has no proposal for
        if (L.gl == 0) atomicOr(status, kErrReplay);
        s = r;
      }
    } else if (valid) {
      s = random_block(r, B, x.y);
    }
  }
  res.s = s;
  const bool active = valid && s != r;
  if (!__any_sync(kFull, active)) return res;
  // 3. delta-MDL and the Hastings correction of the move r -> s
  const RowRef<ST> Ps(bm, s);
  int2 m_su[4], m_rs = make_int2(0, 0);
  int M_ss = 0, dout_s = 0, din_s = 0;
#pragma unroll
  for (int h = 0; h < 4; ++h) on[h] = on[h] && active;
  Ps.get(bm, u, on, m_su);
  if (active) {
    m_rs = row_pair(Pr, bm, s);
    M_ss = row_pair(Ps, bm, s).x;
    dout_s = ldv<ST>(bm.d_out + s);
    din_s = ldv<ST>(bm.d_in + s);
  }
  const unsigned ws = T.counts_of(s);
  const int co_r = wr & kCountMask, ci_r = (wr >> kInShift) & kCountMask;
  const int co_s = ws & kCountMask, ci_s = (ws >> kInShift) & kCountMask;
  const int M_rs = m_rs.x, M_sr = m_rs.y;
  const int d_rr = -co_r - ci_r - self;
  const int d_rs = -co_s + ci_r;
  const int d_sr = co_r - ci_s;
  const int d_ss = co_s + ci_s + self;
  const int kin_self = k_in + self;
  // every count that changes lies in a row or column of r or s: at most their degrees after the move
  const bool small = dout_r + k < kXlogxTable && dout_s + k < kXlogxTable && din_r + k < kXlogxTable &&
                     din_s + k < kXlogxTable;
  const double2* __restrict__ gt = bm.xlogxt;
  double fwd = 0.0, bwd = 0.0, dS = 0.0;
  // corner cells (r,r) (r,s) (s,r) (s,s), then the out- and in-degrees of r and s
  const int q = L.gl;
  const int qa = q == 0 ? M_rr : q == 1 ? M_rs : q == 2 ? M_sr : q == 3 ? M_ss
               : q == 4 ? dout_r : q == 5 ? dout_s : q == 6 ? din_r : din_s;
  const int qd = q == 0 ? d_rr : q == 1 ? d_rs : q == 2 ? d_sr : q == 3 ? d_ss
               : q == 4 ? -k_out : q == 5 ? k_out : q == 6 ? -kin_self : kin_self;
  const bool corner_term = active && q < 8 && qd;
  const bool in_table = (unsigned)qa < (unsigned)kXlogxTable && (unsigned)(qa + qd) < (unsigned)kXlogxTable;
  const double2 c0 = __ldg(gt + (corner_term && in_table ? qa : 0));   // consumed after the entries
  const double2 c1 = __ldg(gt + (corner_term && in_table ? qa + qd : 0));
  if (active && q < 2) {
    // the backward terms of neighbours in r (lane 0) and s (lane 1), whose degrees change
    const int c = q == 0 ? co_r + ci_r + self : co_s + ci_s;
    const int nd = q == 0 ? (dout_r - k_out) + (din_r - k_in) - (M_rr + d_rr)
                          : (dout_s + k_out) + (din_s + k_in) - (M_ss + d_ss);
    const double bw = q == 0 ? (double)(M_rr + d_rr) + (double)(M_rr + d_rr) + 1.0
                             : (double)(M_rs + d_rs) + (double)(M_sr + d_sr) + 1.0;
    if (c) bwd += (double)c * bw * (1.0 / ((double)nd + (double)B));
    // the double count of a present net-zero (r,s) / (s,r) Delta cell
    const bool zero = q == 0 ? (co_s > 0 || ci_r > 0) && d_rs == 0 && M_rs > 0
                             : (co_r > 0 || ci_s > 0) && d_sr == 0 && M_sr > 0;
    if (zero)
      dS += q == 0 ? net_zero_term(M_rs, kin_self, din_s, -k_out, dout_r)
                   : net_zero_term(M_sr, -kin_self, din_r, k_out, dout_s);
  }
  const int nent = active ? n : 0;
  const int nmax = (int)__reduce_max_sync(kFull, (unsigned)nent);
  for (int j0 = 0;;) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      if (j0 + h * L.G >= nmax) break;   // warp-uniform
      const int co = active ? wu[h] & kCountMask : 0, ci = active ? (wu[h] >> kInShift) & kCountMask : 0;
      const bool is_r = u[h] == r, corner = is_r || u[h] == s;
      const int c = co + ci;
      const double cf = (double)(c + (is_r && wu[h] ? self : 0)), cb = corner ? 0.0 : (double)c;
      fwd += cf * ((double)m_su[h].x + (double)m_su[h].y + 1.0) * inv[h];
      bwd += cb * ((double)(m_ru[h].x - co) + (double)(m_ru[h].y - ci) + 1.0) * inv[h];
      // cells (r,u) (s,u) for out-edges to u, (u,r) (u,s) for in-edges; the corners are terms of their own
      const bool out = co != 0;
      const int d = corner || !small ? 0 : out ? co : ci;
      const int ar = small ? (out ? m_ru[h].x : m_ru[h].y) : 0, as = small ? (out ? m_su[h].x : m_su[h].y) : 0;
      const double2 g0 = __ldg(gt + ar), g1 = __ldg(gt + ar - d), g2 = __ldg(gt + as), g3 = __ldg(gt + as + d);
      dS += ((g0.x - g1.x) + (g0.y - g1.y)) + ((g2.x - g3.x) + (g2.y - g3.y));
      if (d && co && ci) {
        const double2 h0 = __ldg(gt + m_ru[h].y), h1 = __ldg(gt + m_ru[h].y - ci);
        const double2 h2 = __ldg(gt + m_su[h].y), h3 = __ldg(gt + m_su[h].y + ci);
        dS += ((h0.x - h1.x) + (h0.y - h1.y)) + ((h2.x - h3.x) + (h2.y - h3.y));
      }
    }
    j0 += 4 * L.G;
    if (j0 >= nmax) break;
#pragma unroll
    for (int h = 0; h < 4; ++h) {   // the next entries of a vertex of more than 4 G distinct blocks
      const int j = j0 + L.gl + h * L.G;
      const int slot = j < nent ? T.list[j] : -1;
      u[h] = slot >= 0 ? T.key_of(slot) : r;
      wu[h] = slot >= 0 ? T.w[slot] : 0u;
      on[h] = wu[h] != 0u;
      inv[h] = on[h] ? ldv<ST>(bm.inv_d + u[h]) : 0.0;
    }
    Pr.get(bm, u, on, m_ru);
    Ps.get(bm, u, on, m_su);
  }
  if (!small) {   // counts beyond the table: the same terms once more, one entry at a time
#pragma unroll 1
    for (int j = L.gl; j < nent; j += L.G) {
      const int slot = T.list[j], uu = T.key_of(slot);
      const int co = T.w[slot] & kCountMask, ci = (T.w[slot] >> kInShift) & kCountMask;
      if (uu == r || uu == s) continue;
      const int2 a = row_pair(Pr, bm, uu), b = row_pair(Ps, bm, uu);
      if (co) dS += dxlogx_wide(gt, a.x, a.x - co) + dxlogx_wide(gt, b.x, b.x + co);
      if (ci) dS += dxlogx_wide(gt, a.y, a.y - ci) + dxlogx_wide(gt, b.y, b.y + ci);
    }
  }
  if (corner_term) {
    const double y = in_table ? (c0.x - c1.x) + (c0.y - c1.y) : dxlogx_far(qa, qa + qd);
    dS += q < 4 ? y : -y;
  }
  fwd = group_sum(fwd, L);
  bwd = group_sum(bwd, L);
  dS = group_sum(dS, L);
  const bool snap = active && maybe_zero_delta(dS, dout_r, dout_s, din_r, din_s, k, g.log_E);
  if (__any_sync(kFull, snap)) {   // the integer scale of the zero snap, as in move_delta
    double Tz = 0.0;               // a sum of integers below 2^53: exact
    if (snap) {
      for (int j = L.gl; j < nent; j += L.G) {
        const int slot = T.list[j];
        const int uu = T.key_of(slot);
        const unsigned w = T.w[slot];
        if (uu == r || uu == s) continue;
        const int2 a = row_pair(Pr, bm, uu), b = row_pair(Ps, bm, uu);
        if (w & kCountMask) Tz += 2.0 * ((double)a.x + (double)b.x);
        if ((w >> kInShift) & kCountMask) Tz += 2.0 * ((double)a.y + (double)b.y);
      }
      if (q < 4 && qd) Tz += 2.0 * (double)qa + (double)qd;
      if (q >= 4 && q < 8) Tz += 2.0 * (double)qa;
    }
    Tz = group_sum(Tz, L);
    if (snap && fabs(dS) <= 0x1p-40 * Tz * g.log_E) dS = 0.0;
  }
  if (active) {
    res.accepted = accept_move(dS, fwd, bwd, k == 0, given ? record_uniform(x) : u53(x.z, x.w));
    res.dS = dS;
    res.wr = wr;
    res.ws = ws;
    res.M_rr = M_rr;
    res.M_ss = M_ss;
    res.dout_r = dout_r;
    res.dout_s = dout_s;
    res.din_r = din_r;
    res.din_s = din_s;
  }
  return res;
}

// Largest degree of the class of G lanes: four neighbours a lane, a quarter of its slots.
__host__ __device__ constexpr int group_max_k(int G) { return 4 * G; }

// Tasks of a batch: one warp each, 32 / G vertices of one class, the largest degrees first; with
// groups of at least gmin lanes.
struct GroupTask {
  int lg;           // log2 of the vertices of the task
  int first, end;   // its vertices from `first`, those below `end` of the batch's light (heavy) list
};
__host__ __device__ inline int group_tasks(const BatchDesc& b, int gmin) {
  const int n = b.light_n;
  const int c32 = gmin >= 32 ? n : b.n32, c16 = gmin >= 32 ? 0 : gmin >= 16 ? n - c32 : b.n16;
  return c32 + ((c16 + 1) >> 1) + ((n - c32 - c16 + 3) >> 2);
}
__device__ __forceinline__ GroupTask group_task(const BatchDesc& b, int gmin, int task, bool light) {
  const int n = b.light_n;
  const int c32 = gmin >= 32 ? n : b.n32, c16 = gmin >= 32 ? 0 : gmin >= 16 ? n - c32 : b.n16;
  const int t16 = (c16 + 1) >> 1;
  GroupTask k;
  k.lg = !light || task < c32 ? 0 : task < c32 + t16 ? 1 : 2;
  k.first = k.lg == 0 ? task : k.lg == 1 ? c32 + 2 * (task - c32) : c32 + c16 + 4 * (task - c32 - t16);
  k.end = !light ? b.heavy_n : k.lg == 0 ? c32 : k.lg == 1 ? c32 + c16 : n;
  return k;
}

}  // namespace sbpb
