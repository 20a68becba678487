// Device-side building blocks of the B200 stochastic block partitioning engine:
// counter-based random numbers, warp primitives, the per-warp neighbour-block table, and the
// warp-cooperative vertex-move evaluation (proposal, Hastings correction, delta-MDL, accept).
//
// Semantics follow the reference (vtsynergy/Hybrid-Stochastic-Block-Partitioning):
//   proposal          src/common.cpp:131-192  (canonical row-then-column multinomial order)
//   hastings          src/entropy.cpp:495-557 (new degree of r/s ignores the in-side self edge)
//   delta-MDL         src/entropy.cpp:296-401 (a present Delta cell with net change 0 and a
//                     non-zero count at (r,s) or (s,r) is counted twice, as the reference's
//                     "unchanged cell" loops do)
//   accept            src/finetune.cpp:19-29
// Log terms are FP64. delta-MDL uses the closed form
//   dS = sum_changed [g(M)-g(M')] - sum_{x in r,s} [g(d_out x)-g(d_out' x)] - [same for d_in] + Q
// with g(x) = x log x, which equals the reference's per-cell sum over rows/cols r,s.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace sbpb {

constexpr int kWarp = 32;
constexpr unsigned kFull = 0xffffffffu;

// Error bits written to the device status word (never trap).
enum : int {
  kErrTableFull = 1,      // neighbour-block table overflow
  kErrScan = 2,           // multinomial walk ran off the row (inconsistent counts)
  kErrReplay = 4,         // replay record index out of range
  kErrBounds = 8,         // block or vertex id out of range
  kErrGridWait = 32,      // a barrier of a persistent kernel gave up waiting
};

// ------------------------------------------------------------------------------------------
// Philox4x32-10 (Salmon et al., SC'11). Counter (a, b, call, tag), key = seed.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int i = 0; i < 10; ++i) {
    const uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
    const uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
    c = make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return c;
}

struct RngParams {
  uint64_t seed;
  const uint4* replay;      // optional host-supplied stream (device copy)
  long long replay_records;
  uint32_t call;
  int moves = 0;            // 1: replay records are proposals (s, 0, u_hi, u_lo), not random words
};

// The accept uniform of a proposal record: the bits of a double in [0, 1).
__device__ __forceinline__ double record_uniform(uint4 x) {
  return __hiloint2double((int)x.z, (int)x.w);
}

// Record for (a, b, tag); replay records are indexed by `slot`.
__device__ __forceinline__ uint4 draw_record(const RngParams& p, uint32_t a, uint32_t b, uint32_t tag,
                                             long long slot, int* status) {
  if (p.replay) {
    if (slot < 0 || slot >= p.replay_records) {
      atomicOr(status, kErrReplay);
      return make_uint4(0, 0, 0, 0xffffffffu);   // u_acc ~ 1: never accepts
    }
    return p.replay[slot];
  }
  return philox4x32_10(make_uint4(a, b, p.call, tag), (uint32_t)p.seed, (uint32_t)(p.seed >> 32));
}

__device__ __forceinline__ long long scale32(uint32_t x, long long n) {
  return (long long)(((unsigned long long)x * (unsigned long long)n) >> 32);
}
__device__ __forceinline__ double u53(uint32_t hi, uint32_t lo) {
  const unsigned long long m = ((unsigned long long)hi << 21) | (unsigned long long)(lo >> 11);
  return (double)m * (1.0 / 9007199254740992.0);
}
// common::propose_random_block with a scaled 32-bit draw.
__device__ __forceinline__ int random_block(int r, int B, uint32_t x) {
  int p = (int)scale32(x, (long long)B - 1);
  return p >= r ? p + 1 : p;
}

// ------------------------------------------------------------------------------------------
// FP64 helpers: g(x) = x log x and accurate differences g(a) - g(b).
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ double xlogx(double x) { return x > 0.0 ? x * log(x) : 0.0; }
// g(a) - g(b) = (a - b) log a + b (log a - log b) for a, b >= 0 without branches: a zero side
// is replaced by 1 inside the logs, which leaves exactly the other side's g term; a == b gives 0.
__device__ __forceinline__ double dxlogx(double a, double b) {
  const double sa = a > 0.0 ? a : 1.0, sb = b > 0.0 ? b : 1.0;
  return (a - b) * log(sa) + b * log1p((sa - sb) / sb);
}

// g(a) - g(b) for integer counts a, b >= 0 from a table of g(x) = hi + lo (hi = g rounded, lo the
// rest, about 104 bits in all; g(0) = g(1) = 0): (hi_a - hi_b) + (lo_a - lo_b).  hi_a - hi_b is
// exact when the two are within a factor of two (Sterbenz) and otherwise within half an ulp of a
// difference of the size of the larger, so the result keeps a relative error near 2^-53 whether
// the counts are close or not (measured worst 1.9e-16; the (a - b) log a + b log(a / b) form
// from a table of logs that it replaced: 3e-16).  Two loads and three additions: that form's
// division, series and two-sided branch were most of the FP64 instructions of a visit.  Counts
// beyond the table go through dxlogx (a call: inline at five places it was most of the code of the
// kernels that evaluate one vertex a warp).
constexpr int kXlogxTable = 1 << 20;
static __device__ __noinline__ double dxlogx_far(int a, int b) { return dxlogx((double)a, (double)b); }
__device__ __forceinline__ double dxlogx_int(const double2* __restrict__ gt, int a, int b) {
  if ((unsigned)a < (unsigned)kXlogxTable && (unsigned)b < (unsigned)kXlogxTable) {
    const double2 ga = __ldg(gt + a), gb = __ldg(gt + b);
    return (ga.x - gb.x) + (ga.y - gb.y);
  }
  return dxlogx_far(a, b);
}

// Merge delta-MDLs are rounded to a multiple of 2^-20 (about 1e-6) before merges are ranked:
// values that are equal but for the rounding of different summation orders then compare equal
// on every implementation, and equal values rank by proposal order and block index, as the
// reference's loops rank exact ties.  (rint: round half to even, the same as the host's
// nearbyint in the default rounding mode.)
__host__ __device__ __forceinline__ double merge_score(double dS) { return rint(dS * 1048576.0) / 1048576.0; }

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}
__device__ __forceinline__ int warp_sum_int(int v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}
__device__ __forceinline__ long long warp_incl_scan(long long v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    long long n = __shfl_up_sync(kFull, v, o);
    if (lane >= o) v += n;
  }
  return v;
}

// ------------------------------------------------------------------------------------------
// Device views of the graph and the blockmodel.
// ------------------------------------------------------------------------------------------
struct GraphView {
  int V;
  long long E;
  double log_E;           // log(max(E, 2)), the zero-snap scale of a delta-MDL
  const int* out_ptr;     // [V+1]
  const int* out_idx;     // out-neighbours incl. self loop, first-occurrence order
  const int* in_ptr;      // [V+1]
  const int* in_idx;      // in-neighbours, self loop removed
  const int* adj;         // both lists of a vertex joined, its out-list first, from out_ptr[v] + in_ptr[v]
  const unsigned char* self;
};

constexpr int kRowPad = 128;   // rows of P are padded to a multiple of this many pairs
// Sums kept per row and column of M for the multinomial walk when B > kSmallB: of chunks of kChunk
// cells and, beyond kFan chunks, of spans of kFan chunks.  Every level of the walk is then one
// load of at most 256 bytes (with chunks of 128 cells and one level of sums a walk at 50,000
// blocks read 2.5 KB in six dependent steps and took a third of a visit).
constexpr int kChunk = 64;
constexpr int kFan = 64;
constexpr int kMaxDense = kChunk * kFan * kFan;   // blocks that three levels reach (their matrix: 550 GB)
constexpr int kSmallB = 128;   // up to this many blocks: no sums, and direct-indexed histograms

struct BlockView {
  int B;
  int sparse;             // 0: dense pairs below; 1: row-hashed regions (large B)
  // row-hashed storage: row r of M lives in rslot[rbase[r] .. rbase[r] + rmask[r]], slots
  // (col, count), col = -1 for an empty slot; MT likewise in cslot.  Keys are never removed
  // (a count can drop to 0).  An insertion that finds its row full sets overflow[0] and the
  // row's flag: overflow[1 + row] for a row of M, overflow[1 + B + row] for a row of MT.
  const long long* rbase;
  const int* rmask;
  int2* rslot;
  const long long* cbase;
  const int* cmask;
  int2* cslot;
  int* overflow;
  int ld;                 // row stride of P (multiple of kRowPad pairs)
  int nch;                // chunks per row = ceil(B / kChunk)
  int ncs;                // row stride of CS and CST: nch rounded up to kFan, the rest zero
  int nss;                // row stride of SS and SST: kFan; 0 up to kFan chunks
  int* CS;                // [B*ncs] CS[row*ncs+c] = sum of M[row, c*kChunk .. c*kChunk+kChunk)
  int* CST;               // [B*ncs] the same over the columns of M
  int* SS;                // [B*nss] sums of kFan chunk sums of CS
  int* SST;               // [B*nss] of CST
  int* b;                 // [V] assignment
  // [B*ld] counts of both directions side by side: P[row*ld+col] = (M[row, col], M[col, row]).
  // A visit needs M[r,u] with M[u,r] and M[s,u] with M[u,s]: one 8-byte load and one 32-byte
  // sector each, where M and a separate transpose took two (200,000 vertices, 11,770 blocks: see
  // the evaluation kernels); the walk gets row t and column t from the same lines.
  int2* P;
  int* d_out;             // [B]
  int* d_in;              // [B]
  int* d;                 // [B] block degrees as the reference maintains them
  double* inv_d;          // [B] 1 / (d + B), the Hastings weight of a block: kept with d, so that a
                          // visit loads it where it took a conversion and a division per entry
  const double2* xlogxt;  // [kXlogxTable] x log x = hi + lo for integer x
};

__device__ __forceinline__ void set_degree(const BlockView& bm, int x, int value) {
  bm.d[x] = value;
  bm.inv_d[x] = 1.0 / ((double)value + (double)bm.B);
}

// ---- row-hashed storage ------------------------------------------------------------------
__device__ __forceinline__ unsigned slot_hash(int key) { return (unsigned)key * 2654435761u; }

__device__ __forceinline__ int hashed_get(const long long* base, const int* mask, const int2* slot, int row, int col) {
  const long long b0 = base[row];
  const int m = mask[row];
  unsigned h = slot_hash(col) & (unsigned)m;
  for (int probe = 0; probe <= m; ++probe) {
    const int2 e = slot[b0 + h];
    if (e.x == col) return e.y;
    if (e.x == -1) return 0;
    h = (h + 1) & (unsigned)m;
  }
  return 0;
}

__device__ __forceinline__ void hashed_add(const long long* base, const int* mask, int2* slot, int row, int col,
                                           int delta, int* overflow, int* row_full) {
  const long long b0 = base[row];
  const int m = mask[row];
  unsigned h = slot_hash(col) & (unsigned)m;
  for (int probe = 0; probe <= m; ++probe) {
    int* key = &slot[b0 + h].x;
    int k = *(volatile int*)key;
    if (k == -1) {
      const int prev = atomicCAS(key, -1, col);
      k = prev == -1 ? col : prev;
    }
    if (k == col) {
      atomicAdd(&slot[b0 + h].y, delta);
      return;
    }
    h = (h + 1) & (unsigned)m;
  }
  atomicOr(overflow, 1);
  row_full[row] = 1;
}

// M[row, col] and MT[row, col] = M[col, row] in either representation.
// Storage of the block matrix as a compile-time choice (kAny: decided by bm.sparse at run time).
// Kernels instantiated for one storage carry no code for the other.
enum class Store { kAny, kDense, kHashed, kDenseFrozen };
// kDenseFrozen: dense storage that no thread of the launch writes (the evaluation half of an
// asynchronous-Gibbs batch), read through the read-only data cache.
template <Store S>
__device__ __forceinline__ int ldi(const int* p) {
  if constexpr (S == Store::kDenseFrozen) return __ldg(p);
  else return *p;
}
template <Store S, class T>
__device__ __forceinline__ T ldv(const T* p) {
  if constexpr (S == Store::kDenseFrozen) return __ldg(p);
  else return *p;
}

// (M[row, col], M[col, row])
template <Store S = Store::kAny>
__device__ __forceinline__ int2 bm_pair(const BlockView& bm, int row, int col) {
  const bool hashed = S == Store::kHashed || (S == Store::kAny && bm.sparse);
  if constexpr (S != Store::kDense && S != Store::kDenseFrozen) {
    if (hashed)
      return make_int2(hashed_get(bm.rbase, bm.rmask, bm.rslot, row, col),
                       hashed_get(bm.cbase, bm.cmask, bm.cslot, row, col));
  }
  if constexpr (S != Store::kHashed) return ldv<S>(bm.P + (size_t)row * bm.ld + col);
  return make_int2(0, 0);
}
// M[row, col]
template <Store S = Store::kAny>
__device__ __forceinline__ int bm_get(const BlockView& bm, int row, int col) {
  if constexpr (S == Store::kDense || S == Store::kDenseFrozen) return ldi<S>(&bm.P[(size_t)row * bm.ld + col].x);
  else if constexpr (S == Store::kHashed) return hashed_get(bm.rbase, bm.rmask, bm.rslot, row, col);
  else return bm.sparse ? hashed_get(bm.rbase, bm.rmask, bm.rslot, row, col) : bm.P[(size_t)row * bm.ld + col].x;
}

// M[col, row]
template <Store S = Store::kAny>
__device__ __forceinline__ int bm_getT(const BlockView& bm, int row, int col) {
  if constexpr (S == Store::kDense || S == Store::kDenseFrozen) return ldi<S>(&bm.P[(size_t)row * bm.ld + col].y);
  else if constexpr (S == Store::kHashed) return hashed_get(bm.cbase, bm.cmask, bm.cslot, row, col);
  else return bm.sparse ? hashed_get(bm.cbase, bm.cmask, bm.cslot, row, col) : bm.P[(size_t)row * bm.ld + col].y;
}

// Walk of a hashed row in ascending column order: the first column whose running count
// exceeds `target`, found digit by digit (5 bits of the column at a time, most significant
// first).  Each pass sums the row's counts of the columns left in range into 32 bins (`bins`:
// 32 ints of the warp's shared memory), scans the bins and keeps the one that holds the target.
// Same result as the dense walks.
__device__ __forceinline__ int warp_select_hashed(const long long* base, const int* mask, const int2* slot, int row,
                                                  int B, long long target, int lane, int* bins) {
  const long long b0 = base[row];
  const int cap = mask[row] + 1;
  int bits = 0;
  while ((1 << bits) < B) ++bits;
  int lo = 0;
  for (int shift = ((bits + 4) / 5) * 5 - 5; shift >= 0; shift -= 5) {
    bins[lane] = 0;
    __syncwarp();
    const long long span = 32LL << shift;
    for (int i = lane; i < cap; i += kWarp) {
      const int2 e = slot[b0 + i];
      if (e.x >= lo && (long long)e.x < lo + span && e.y > 0) atomicAdd(&bins[(e.x - lo) >> shift], e.y);
    }
    __syncwarp();
    const long long v = bins[lane];
    const long long incl = warp_incl_scan(v, lane);
    const unsigned hit = __ballot_sync(kFull, incl > target);
    if (!hit) return -1;
    const int sel = __ffs(hit) - 1;
    target -= __shfl_sync(kFull, incl - v, sel);
    lo += sel << shift;
    __syncwarp();
  }
  return lo;
}

// The sums that cell (row, col) belongs to.
__device__ __forceinline__ void chunks_add(const BlockView& bm, int row, int col, int delta) {
  if (bm.B <= kSmallB) return;
  atomicAdd(bm.CS + (size_t)row * bm.ncs + col / kChunk, delta);
  atomicAdd(bm.CST + (size_t)col * bm.ncs + row / kChunk, delta);
  if (bm.nss) {
    atomicAdd(bm.SS + (size_t)row * bm.nss + col / (kChunk * kFan), delta);
    atomicAdd(bm.SST + (size_t)col * bm.nss + row / (kChunk * kFan), delta);
  }
}

// The calling lane's place in a group of G = 8, 16 or 32 lanes of its warp.
struct Lanes {
  int G, gl, lane, gbase;
  unsigned gmask;
  __device__ __forceinline__ Lanes(int group, int lane_) : G(group), lane(lane_) {
    gl = lane & (G - 1);
    gbase = lane & ~(G - 1);
    gmask = G == 32 ? kFull : ((1u << G) - 1u) << gbase;
  }
};

// ------------------------------------------------------------------------------------------
// The multinomial walk over row t of M (column t when `col`), ascending: the first index whose
// running count exceeds tg.  One group per walk, of which the first eight lanes read; every lane of
// the warp calls it; groups with !on get -1.
// ------------------------------------------------------------------------------------------
// One level: lane g8 holds the N sums v[] of entries [N g8, N g8 + N).  Finds the entry of the
// running count tg, leaves the count before it taken off tg; *ok cleared when there is none.
template <int N>
__device__ __forceinline__ int walk_level(const int (&v)[N], int* tg, bool* ok, const Lanes& L) {
  const int g8 = L.lane & 7;
  int sum = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) sum += v[j];
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const int y = __shfl_up_sync(kFull, incl, o);
    if (g8 >= o) incl += y;
  }
  const unsigned hit = __ballot_sync(kFull, *ok && L.gl < 8 && incl > *tg) & L.gmask;
  const int src = hit ? __ffs(hit) - 1 : L.gbase;
  int rest = *tg - (incl - sum), at = N * g8, run = 0, base = 0;   // meaningful on lane src
#pragma unroll
  for (int j = 0; j < N - 1; ++j) {
    run += v[j];
    if (rest >= run) {
      at = N * g8 + j + 1;
      base = run;
    }
  }
  *ok = *ok && hit;
  *tg = __shfl_sync(kFull, rest - base, src);
  return __shfl_sync(kFull, at, src);
}

template <Store ST>
__device__ __forceinline__ int walk_sums(const int* sums, int* tg, bool* ok, const Lanes& L) {   // kFan sums
  const bool rd = *ok && L.gl < 8;
  const int4* p = reinterpret_cast<const int4*>(sums + 8 * (L.lane & 7));
  const int4 a = rd ? ldv<ST>(p) : make_int4(0, 0, 0, 0), b = rd ? ldv<ST>(p + 1) : make_int4(0, 0, 0, 0);
  const int v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  return walk_level<8>(v, tg, ok, L);
}

// B > kSmallB: through the spans (if any), the chunks of one span, the cells of one chunk.
template <Store ST>
__device__ __forceinline__ int walk_tree(const BlockView& bm, int t, bool col, int tg, bool on, const Lanes& L) {
  bool ok = on;
  int span = 0;
  if (bm.nss) span = walk_sums<ST>((col ? bm.SST : bm.SS) + (size_t)t * bm.nss, &tg, &ok, L);
  const int chunk = span * kFan + walk_sums<ST>((col ? bm.CST : bm.CS) + (size_t)t * bm.ncs + (ok ? span : 0) * kFan,
                                                &tg, &ok, L);
  ok = ok && chunk < bm.nch;
  const bool rd = ok && L.gl < 8;
  constexpr int kPer = kChunk / 8;   // cells a lane
  const int4* p =
      reinterpret_cast<const int4*>(bm.P + (size_t)t * bm.ld + (size_t)(ok ? chunk : 0) * kChunk + kPer * (L.lane & 7));
  int v[kPer];
#pragma unroll
  for (int j = 0; j < kPer / 2; ++j) {
    const int4 a = rd ? ldv<ST>(p + j) : make_int4(0, 0, 0, 0);
    v[2 * j] = col ? a.y : a.x;
    v[2 * j + 1] = col ? a.w : a.z;
  }
  const int at = walk_level<kPer>(v, &tg, &ok, L);
  return ok ? chunk * kChunk + at : -1;
}

// B <= kSmallB: the whole row in up to eight coalesced steps of 16 cells; a transposing reduction
// leaves step q's total on lane q, and the step picked is read again (from L1) two cells a lane.
template <Store ST>
__device__ __forceinline__ int walk_row(const BlockView& bm, int t, bool col, int tg, bool on, const Lanes& L) {
  bool ok = on;
  const int g8 = L.lane & 7;
  const bool rd = ok && L.gl < 8;
  const int2* row = bm.P + (size_t)t * bm.ld;
  int v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int c = 16 * q + 2 * g8;
    const int4 x = (rd && c < bm.B) ? ldv<ST>(reinterpret_cast<const int4*>(row + c)) : make_int4(0, 0, 0, 0);
    v[q] = col ? x.y + x.w : x.x + x.z;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const bool up = g8 & 4;
    const int give = up ? v[q] : v[q + 4], keep = up ? v[q + 4] : v[q];
    v[q] = keep + __shfl_xor_sync(kFull, give, 4);
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const bool up = g8 & 2;
    const int give = up ? v[q] : v[q + 2], keep = up ? v[q + 2] : v[q];
    v[q] = keep + __shfl_xor_sync(kFull, give, 2);
  }
  const bool up = g8 & 1;
  const int give = up ? v[0] : v[1], keep = up ? v[1] : v[0];
  const int total[1] = {keep + __shfl_xor_sync(kFull, give, 1)};
  const int step = walk_level<1>(total, &tg, &ok, L);
  int4 x = make_int4(0, 0, 0, 0);
  if (ok && L.gl < 8) x = ldv<ST>(reinterpret_cast<const int4*>(row + 16 * step + 2 * g8));
  const int two[2] = {col ? x.y : x.x, col ? x.w : x.z};
  const int at = walk_level<2>(two, &tg, &ok, L);
  return ok ? 16 * step + at : -1;
}

// Same walk over a compressed list (idx[i], val[i]), i in [0, n).
__device__ __forceinline__ int warp_select_sparse(const int* __restrict__ idx, const int* __restrict__ val, int n,
                                                  int target, int skip, int lane) {
  for (int base = 0; base < n; base += kWarp) {
    const int i = base + lane;
    int c = -1, incl = 0;   // a row's counts sum to at most E < 2^31
    if (i < n) {
      c = idx[i];
      incl = c != skip ? val[i] : 0;
    }
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
      const int y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    const int tot = __shfl_sync(kFull, incl, 31);
    if (target < tot) {
      const unsigned hit = __ballot_sync(kFull, incl > target);
      return __shfl_sync(kFull, c, __ffs(hit) - 1);
    }
    target -= tot;
  }
  return -1;
}

// ------------------------------------------------------------------------------------------
// Per-warp neighbour-block table in shared memory: open addressing on block id, with a
// compact list of used slots so reset and enumeration cost O(distinct blocks).
// ------------------------------------------------------------------------------------------
struct WarpTable {
  int* keys;   // [cap], -1 = empty
  int* cout;   // [cap] out-neighbour counts (self loop excluded)
  int* cin;    // [cap] in-neighbour counts (self loop excluded)
  int* list;   // [cap] used slots
  int* nlist;  // [1]
  int mask;    // cap - 1 (cap power of two)
};

__device__ __forceinline__ int table_slot(const WarpTable& t, int key, int* status) {
  unsigned h = ((unsigned)key * 2654435761u) & (unsigned)t.mask;
  for (int probe = 0; probe <= t.mask; ++probe) {
    const int k = t.keys[h];
    if (k == key) return (int)h;
    if (k == -1) {
      const int prev = atomicCAS(&t.keys[h], -1, key);
      if (prev == -1) {
        t.list[atomicAdd(t.nlist, 1)] = (int)h;
        return (int)h;
      }
      if (prev == key) return (int)h;
    }
    h = (h + 1) & (unsigned)t.mask;
  }
  atomicOr(status, kErrTableFull);
  return -1;
}

__device__ __forceinline__ int table_find(const WarpTable& t, int key) {
  unsigned h = ((unsigned)key * 2654435761u) & (unsigned)t.mask;
  for (int probe = 0; probe <= t.mask; ++probe) {
    const int k = t.keys[h];
    if (k == key) return (int)h;
    if (k == -1) return -1;
    h = (h + 1) & (unsigned)t.mask;
  }
  return -1;
}

// Warp-aggregated insertion: lanes holding the same key add their multiplicity once.
__device__ __forceinline__ void table_add(const WarpTable& t, int key, bool valid, bool incoming, int* status) {
  const int k = valid ? key : -2;
  const unsigned peers = __match_any_sync(kFull, k);
  const int lane = threadIdx.x & 31;
  if (valid && (__ffs(peers) - 1) == lane) {
    const int slot = table_slot(t, key, status);
    if (slot >= 0) atomicAdd(incoming ? &t.cin[slot] : &t.cout[slot], __popc(peers));
  }
}

// Per-warp table of `cap` slots carved from a CTA's dynamic shared memory (table_ints(cap) ints per warp).
__device__ __forceinline__ WarpTable carve_table(int* base, int cap, int warp) {
  int* p = base + (size_t)warp * (4 * cap + 64);
  WarpTable t;
  t.keys = p;
  t.cout = p + cap;
  t.cin = p + 2 * cap;
  t.list = p + 3 * cap;
  t.nlist = p + 4 * cap;
  t.mask = cap - 1;
  return t;
}

__device__ __forceinline__ void init_table(const WarpTable& t, int lane) {
  const int cap = t.mask + 1;
  for (int i = lane; i < cap; i += kWarp) {
    t.keys[i] = -1;
    t.cout[i] = 0;
    t.cin[i] = 0;
  }
  if (lane == 0) *t.nlist = 0;
  __syncwarp();
}

__device__ __forceinline__ void table_reset(const WarpTable& t, int lane) {
  __syncwarp();
  const int n = *t.nlist;
  for (int i = lane; i < n; i += kWarp) {
    const int h = t.list[i];
    t.keys[h] = -1;
    t.cout[h] = 0;
    t.cin[h] = 0;
  }
  __syncwarp();
  if (lane == 0) *t.nlist = 0;
  __syncwarp();
}

// Build the table for vertex v from the current assignment (self loop excluded; block r is
// inserted when v has a self loop so the Hastings sum sees it).
__device__ __forceinline__ void build_table(const GraphView& g, const BlockView& bm, int v, int r, const WarpTable& t,
                                            int lane, int* status) {
  const int o0 = g.out_ptr[v], o1 = g.out_ptr[v + 1];
  for (int e0 = o0; e0 < o1; e0 += kWarp) {
    const int e = e0 + lane;
    int key = -1;
    bool valid = false;
    if (e < o1) {
      const int u = __ldg(g.out_idx + e);
      if (u != v) { key = bm.b[u]; valid = true; }
    }
    table_add(t, key, valid, false, status);
  }
  const int i0 = g.in_ptr[v], i1 = g.in_ptr[v + 1];
  for (int e0 = i0; e0 < i1; e0 += kWarp) {
    const int e = e0 + lane;
    int key = -1;
    bool valid = false;
    if (e < i1) { key = bm.b[__ldg(g.in_idx + e)]; valid = true; }
    table_add(t, key, valid, true, status);
  }
  if (lane == 0 && g.self[v]) table_slot(t, r, status);
  __syncwarp();
}

struct EvalResult {
  int t;          // block of the proposal's neighbour (-1: no neighbour, uniform proposal)
  int s;          // proposed block
  int accepted;   // 1 if accepted (s != r)
  double dS;      // delta MDL (0 when s == r)
  double H;       // Hastings correction
};

struct MoveCounts {   // self-loop-free neighbour counts by block for the four corner blocks
  int co_r, co_s, ci_r, ci_s;
};

__device__ __forceinline__ MoveCounts corner_counts(const WarpTable& t, int r, int s) {
  MoveCounts mc;
  const int hr = table_find(t, r), hs = table_find(t, s);
  mc.co_r = hr >= 0 ? t.cout[hr] : 0;
  mc.ci_r = hr >= 0 ? t.cin[hr] : 0;
  mc.co_s = hs >= 0 ? t.cout[hs] : 0;
  mc.ci_s = hs >= 0 ? t.cin[hs] : 0;
  return mc;
}

// Warp-aggregated insertion of one element per lane; lanes holding the same block add their
// out- and in-multiplicities once.
__device__ __forceinline__ void table_add_dir(const WarpTable& t, int key, bool valid, bool incoming, int* status) {
  const int k = valid ? key : -2;
  const unsigned peers = __match_any_sync(kFull, k);
  const unsigned in_mask = __ballot_sync(kFull, valid && incoming);
  const int lane = threadIdx.x & 31;
  if (valid && (__ffs(peers) - 1) == lane) {
    const int slot = table_slot(t, key, status);
    if (slot >= 0) {
      const int nin = __popc(peers & in_mask), nout = __popc(peers) - nin;
      if (nout) atomicAdd(&t.cout[slot], nout);
      if (nin) atomicAdd(&t.cin[slot], nin);
    }
  }
}

// One pass over v's virtual neighbour list (out list incl. the self loop, then in list without
// it) gathers every neighbour's block into the table (self loop excluded from the counts, its
// block r inserted with zero counts).  Returns the block of neighbour element `idx` (-1 when
// idx is out of range), the proposal's neighbour of src/common.cpp:11-26.
template <Store ST = Store::kAny>
__device__ __forceinline__ int gather_neighbour_blocks(const GraphView& g, const BlockView& bm, int v, int r, int o0,
                                                       int k_out, int i0, int k, int self, int idx,
                                                       const WarpTable& t, int lane, int* status) {
  int tblk = -1;
  for (int base = 0; base < k; base += 2 * kWarp) {   // two elements per lane in flight
    const int e0 = base + lane, e1 = base + kWarp + lane;
    int u0 = -1, u1 = -1;
    if (e0 < k) u0 = e0 < k_out ? __ldg(g.out_idx + o0 + e0) : __ldg(g.in_idx + i0 + (e0 - k_out));
    if (e1 < k) u1 = e1 < k_out ? __ldg(g.out_idx + o0 + e1) : __ldg(g.in_idx + i0 + (e1 - k_out));
    const int b0 = u0 >= 0 ? ldi<ST>(bm.b + u0) : -1;
    const int b1 = u1 >= 0 ? ldi<ST>(bm.b + u1) : -1;
    if (idx >= base && idx < base + kWarp) tblk = __shfl_sync(kFull, b0, idx - base);
    if (idx >= base + kWarp && idx < base + 2 * kWarp) tblk = __shfl_sync(kFull, b1, idx - base - kWarp);
    table_add_dir(t, b0, u0 >= 0 && u0 != v, e0 >= k_out, status);
    table_add_dir(t, b1, u1 >= 0 && u1 != v, e1 >= k_out, status);
  }
  if (lane == 0 && self) table_slot(t, r, status);
  return tblk;
}

// Loads of move_delta that do not depend on the proposed block s: issued right after the
// neighbour table is built, so that they overlap the multinomial walk that picks s.
struct NbPrefetch {
  int u, co, ci, M_ru, M_ur;   // this lane's first table entry (u = -1: none)
  double inv;
  int M_rr, dout_r, din_r;
};

template <Store ST = Store::kAny>
__device__ __forceinline__ void prefetch_nb(const BlockView& bm, int r, const WarpTable& t, int lane, NbPrefetch* p) {
  __syncwarp();
  const int n = *t.nlist;
  p->u = -1;
  p->co = p->ci = p->M_ru = p->M_ur = 0;
  p->inv = 0.0;
  if (lane < n) {
    const int h = t.list[lane];
    const int u = t.keys[h];
    p->u = u;
    p->co = t.cout[h];
    p->ci = t.cin[h];
    const int2 m = bm_pair<ST>(bm, r, u);
    p->M_ru = m.x;
    p->M_ur = m.y;
    p->inv = ldv<ST>(bm.inv_d + u);
  }
  p->M_rr = bm_get<ST>(bm, r, r);
  p->dout_r = ldi<ST>(bm.d_out + r);
  p->din_r = ldi<ST>(bm.d_in + r);
}

// Whether the zero snap (below) can apply: the integer scale T of the changed cells and degrees is
// at most six times the block degrees of r and s plus four times the vertex's, as every changed
// cell lies in a row or column of r or s.  In single precision, with room for its rounding.
__device__ __forceinline__ bool maybe_zero_delta(double dS, int dout_r, int dout_s, int din_r, int din_s, int k,
                                                 double log_E) {
  const float bound = 6.0f * ((float)dout_r + (float)dout_s + (float)din_r + (float)din_s) + 4.0f * (float)k + 4.0f;
  return fabsf((float)dS) <= 0x1.1p-40f * bound * (float)log_E;
}

// The double count of a net-zero Delta cell, m (log1p(a / b) + log1p(c / d)); rare, so out of line.
static __device__ __noinline__ double net_zero_term(int m, int a, int b, int c, int d) {
  return (double)m * (log1p((double)a / (double)b) + log1p((double)c / (double)d));
}

// Delta-MDL of moving v from r to s (s != r) against the current state, with the gathered
// table of v's neighbour blocks, and the reference's Hastings correction (*H).
//  - One load round over the distinct neighbour blocks (lane i: table entries i, i+32, ...)
//    gives the Hastings sums and the changed cells; the lane that loaded a cell adds its FP64
//    term: (r,u) and (s,u) for v's out-edges to u, (u,r) and (u,s) for its in-edges from u.
//  - Eight lanes add the corner-cell and degree terms.
//  - The double count of a present net-zero (r,s) / (s,r) Delta cell is added by the lanes
//    that hold it, and only then.
// Every lane returns the same values.
template <Store ST = Store::kAny>
__device__ __forceinline__ double move_delta(const GraphView& g, const BlockView& bm, int r, int s, int k_out,
                                             int k_in, int self, const WarpTable& t, int lane, double* H,
                                             const NbPrefetch* pre = nullptr) {
  __syncwarp();
  const MoveCounts mc = corner_counts(t, r, s);
  const int B = bm.B;
  const int d_rr = -mc.co_r - mc.ci_r - self;
  const int d_rs = -mc.co_s + mc.ci_r;
  const int d_sr = mc.co_r - mc.ci_s;
  const int d_ss = mc.co_s + mc.ci_s + self;
  const int2 m_rs = bm_pair<ST>(bm, r, s);
  const int M_rr = pre ? pre->M_rr : bm_get<ST>(bm, r, r), M_rs = m_rs.x;
  const int M_sr = m_rs.y, M_ss = bm_get<ST>(bm, s, s);
  const int dout_r = pre ? pre->dout_r : ldi<ST>(bm.d_out + r), dout_s = ldi<ST>(bm.d_out + s);
  const int din_r = pre ? pre->din_r : ldi<ST>(bm.d_in + r), din_s = ldi<ST>(bm.d_in + s);
  const int kin_self = k_in + self;

  double fwd = 0.0, bwd = 0.0, dS = 0.0;
  const int n = *t.nlist;
  for (int i = lane; i < n; i += kWarp) {
    int u, co, ci, M_ru, M_ur;
    double inv;   // 1 / (d[u] + B): a non-corner block's degree is unchanged
    if (pre && i < kWarp) {
      u = pre->u;
      co = pre->co;
      ci = pre->ci;
      M_ru = pre->M_ru;
      M_ur = pre->M_ur;
      inv = pre->inv;
    } else {
      const int h = t.list[i];
      u = t.keys[h];
      co = t.cout[h];
      ci = t.cin[h];
      const int2 m = bm_pair<ST>(bm, r, u);
      M_ru = m.x;
      M_ur = m.y;
      inv = ldv<ST>(bm.inv_d + u);
    }
    const int2 m_su = bm_pair<ST>(bm, s, u);
    const int M_su = m_su.x, M_us = m_su.y;
    const bool is_r = (u == r), is_s = (u == s);
    const double c = (double)(co + ci + (is_r ? self : 0));
    fwd += c * (M_su + M_us + 1.0) * inv;
    if (is_r || is_s) {
      const int nd = is_r ? (dout_r - k_out) + (din_r - k_in) - (M_rr + d_rr)
                          : (dout_s + k_out) + (din_s + k_in) - (M_ss + d_ss);
      const double bw = is_r ? (double)(M_rr + d_rr) + (double)(M_rr + d_rr) + 1.0
                             : (double)(M_rs + d_rs) + (double)(M_sr + d_sr) + 1.0;
      bwd += c * bw * (1.0 / ((double)nd + (double)B));
    } else {   // changed non-corner cells (r,u) (s,u) (u,r) (u,s); the corner cells are added below
      bwd += c * ((double)(M_ru - co) + (double)(M_ur - ci) + 1.0) * inv;
      if (co) dS += dxlogx_int(bm.xlogxt, M_ru, M_ru - co) + dxlogx_int(bm.xlogxt, M_su, M_su + co);
      if (ci) dS += dxlogx_int(bm.xlogxt, M_ur, M_ur - ci) + dxlogx_int(bm.xlogxt, M_us, M_us + ci);
    }
  }
  if (lane < 8) {   // corner cells (r,r) (r,s) (s,r) (s,s), then the out- and in-degrees of r and s
    const int a = lane == 0 ? M_rr : lane == 1 ? M_rs : lane == 2 ? M_sr : lane == 3 ? M_ss
                : lane == 4 ? dout_r : lane == 5 ? dout_s : lane == 6 ? din_r : din_s;
    const int d = lane == 0 ? d_rr : lane == 1 ? d_rs : lane == 2 ? d_sr : lane == 3 ? d_ss
                : lane == 4 ? -k_out : lane == 5 ? k_out : lane == 6 ? -kin_self : kin_self;
    if (d) {
      const double x = dxlogx_int(bm.xlogxt, a, a + d);
      dS += lane < 4 ? x : -x;
    }
  }
  {
    // the double count of a present net-zero (r,s) / (s,r) Delta cell (lanes 8 and 9)
    const bool q_rs = (mc.co_s > 0 || mc.ci_r > 0) && d_rs == 0 && M_rs > 0;
    const bool q_sr = (mc.co_r > 0 || mc.ci_s > 0) && d_sr == 0 && M_sr > 0;
    const int qm = lane == 8 ? (q_rs ? M_rs : 0) : lane == 9 ? (q_sr ? M_sr : 0) : 0;
    if (qm)
      dS += net_zero_term(qm, lane == 8 ? kin_self : -kin_self, lane == 8 ? din_s : din_r,
                          lane == 8 ? -k_out : k_out, lane == 8 ? dout_r : dout_s);
  }
  fwd = warp_sum(fwd);
  bwd = warp_sum(bwd);
  dS = warp_sum(dS);
  // A mathematically zero change reads as exactly 0 whatever the summation order: the
  // Metropolis-Hastings early stop tests `delta == 0.0` (src/finetune.cpp:147).  T, the integer
  // scale of the snap, takes a second pass over the cells and is formed only when it can matter.
  if (maybe_zero_delta(dS, dout_r, dout_s, din_r, din_s, k_out + k_in, g.log_E)) {   // warp-uniform
    long long T = 0;
    for (int i = lane; i < n; i += kWarp) {
      const int h = t.list[i];
      const int u = t.keys[h];
      if (u == r || u == s) continue;
      const int2 a = bm_pair<ST>(bm, r, u), b = bm_pair<ST>(bm, s, u);
      T += (t.cout[h] ? 2LL * (a.x + b.x) : 0LL) + (t.cin[h] ? 2LL * (a.y + b.y) : 0LL);
    }
    if (lane < 8) {
      const int a = lane == 0 ? M_rr : lane == 1 ? M_rs : lane == 2 ? M_sr : lane == 3 ? M_ss
                  : lane == 4 ? dout_r : lane == 5 ? dout_s : lane == 6 ? din_r : din_s;
      const int d = lane == 0 ? d_rr : lane == 1 ? d_rs : lane == 2 ? d_sr : lane == 3 ? d_ss : 0;
      T += lane < 4 ? (d ? 2LL * a + d : 0LL) : 2LL * a;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) T += __shfl_xor_sync(kFull, T, o);
    if (fabs(dS) <= 0x1p-40 * (double)T * g.log_E) dS = 0.0;
  }
  *H = bwd / fwd;
  return dS;
}

// Full evaluation of vertex v against the current state, table left filled on return
// (caller resets it). Every lane returns the same result.
//  1. gather_neighbour_blocks; the proposal's neighbour (element floor(x0 * k)) is one of the
//     gathered elements, so its block comes from the same pass;
//  2. the multinomial walk over M[t,:] + M[:,t] picks s;
//  3. move_delta gives delta-MDL and the Hastings correction.
//
// `given`: x is a proposal record (s, 0, u_hi, u_lo) of a replayed stream: the proposal is x.x
// and the accept uniform the double of (x.z, x.w); steps 1 (without the neighbour pick) and 3.
template <Store ST = Store::kAny>
__device__ __forceinline__ EvalResult evaluate_vertex(const GraphView& g, const BlockView& bm, int v, uint4 x,
                                                      const WarpTable& t, int lane, int* status, int* r_out,
                                                      int* k_out_out, int* k_in_out, bool given = false) {
  EvalResult res;
  const int r = ldi<ST>(bm.b + v);
  const int o0 = g.out_ptr[v], o1 = g.out_ptr[v + 1];
  const int i0 = g.in_ptr[v], i1 = g.in_ptr[v + 1];
  const int self = g.self[v];
  const int k_out = o1 - o0, k_in = i1 - i0, k = k_out + k_in;
  *r_out = r;
  *k_out_out = k_out;
  *k_in_out = k_in;
  res.accepted = 0;
  res.dS = 0.0;
  res.H = 1.0;
  const int idx = (k > 0 && !given) ? (int)scale32(x.x, k) : -1;
  const int tblk = gather_neighbour_blocks<ST>(g, bm, v, r, o0, k_out, i0, k, self, idx, t, lane, status);
  res.t = (k > 0 && !given) ? tblk : -1;

  NbPrefetch pre;
  prefetch_nb<ST>(bm, r, t, lane, &pre);

  int s;
  if (given) {
    s = (int)x.x;
    if (s < 0 || s >= bm.B) {   // a visit the stream has no proposal for
      if (lane == 0) atomicOr(status, kErrReplay);
      s = r;
    }
  } else if (k == 0) {
    s = random_block(r, bm.B, x.y);
  } else {
    const bool hashed = ST == Store::kHashed || (ST == Store::kAny && bm.sparse);
    if (ST != Store::kDense && hashed) {
      const int dot = bm.d_out[tblk];
      const long long target = scale32(x.y, (long long)dot + (long long)bm.d_in[tblk]);
      int* bins = t.nlist + 32;   // the 32 ints after the table's list count
      if (target < dot) s = warp_select_hashed(bm.rbase, bm.rmask, bm.rslot, tblk, bm.B, target, lane, bins);
      else s = warp_select_hashed(bm.cbase, bm.cmask, bm.cslot, tblk, bm.B, target - dot, lane, bins);
    } else if (ST != Store::kHashed) {
      const int dot = ldi<ST>(bm.d_out + tblk), dit = ldi<ST>(bm.d_in + tblk);
      const long long target = scale32(x.y, (long long)dot + (long long)dit);
      const bool in_col = target >= dot;
      const int tg = (int)(in_col ? target - dot : target);
      const Lanes L(32, lane);
      if (bm.B <= kSmallB) s = walk_row<ST>(bm, tblk, in_col, tg, true, L);
      else s = walk_tree<ST>(bm, tblk, in_col, tg, true, L);
    } else {
      s = -1;
    }
    if (s < 0) {
      if (lane == 0) atomicOr(status, kErrScan);
      s = r;
    }
  }
  res.s = s;
  if (s == r) return res;
  double Hp;
  const double dS = move_delta<ST>(g, bm, r, s, k_out, k_in, self, t, lane, &Hp, &pre);
  const double H = (k == 0) ? 1.0 : Hp;
  double ap = exp(-3.0 * dS) * H;
  ap = ap >= 1.0 ? 1.0 : ap;
  res.dS = dS;
  res.H = H;
  res.accepted = ((given ? record_uniform(x) : u53(x.z, x.w)) <= ap) ? 1 : 0;
  return res;
}

}  // namespace sbpb
