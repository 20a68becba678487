// Device-wide primitives for the sparse block matrix: a stable LSD radix sort of 64-bit keys,
// a multi-CTA exclusive scan of ints and run-length encoding of sorted keys.  Written for this
// engine (no library sort); used to rebuild the block matrix from the edge list when B is large.
#include "sbp_sort.cuh"

namespace sbpb {

constexpr int kSortThreads = 256;
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;

// Per-CTA digit histogram of a contiguous tile; hist is digit-major: hist[d * G + cta].
__global__ void k_radix_hist(const unsigned long long* __restrict__ keys, long long n, long long tile, int shift,
                             unsigned* hist) {
  __shared__ unsigned h[kRadix];
  for (int i = threadIdx.x; i < kRadix; i += blockDim.x) h[i] = 0;
  __syncthreads();
  const long long b0 = (long long)blockIdx.x * tile, b1 = min(n, b0 + tile);
  for (long long i = b0 + threadIdx.x; i < b1; i += blockDim.x) atomicAdd(&h[(keys[i] >> shift) & (kRadix - 1)], 1u);
  __syncthreads();
  for (int i = threadIdx.x; i < kRadix; i += blockDim.x) hist[(size_t)i * gridDim.x + blockIdx.x] = h[i];
}

// Stable scatter: elements of a tile keep their order inside each digit.  A CTA takes 4,096 elements
// at a time, 512 consecutive ones a warp, all loaded before the first is ranked; a warp ranks its
// elements 32 at a time in order (match_any, running counts per warp), then the counts become
// offsets per digit across the warps and across the digits, and the elements go through shared
// memory into digit order, so that a digit's run (16 elements on average) is written as whole
// lines.  Bound by the ranking and the scattered lines: 12 million keys 247 us at 256 elements and
// five barriers a round before (78 us of reads and writes at the copy rate).
constexpr int kSortItems = 16;
constexpr int kSortChunk = kSortThreads * kSortItems;

__global__ void __launch_bounds__(kSortThreads)
    k_radix_scatter(const unsigned long long* __restrict__ in, unsigned long long* __restrict__ out, long long n,
                    long long tile, int shift, const unsigned* __restrict__ offsets) {
  __shared__ unsigned long long buf[kSortChunk];
  __shared__ unsigned wcount[kSortThreads / 32][kRadix];
  __shared__ unsigned base[kRadix], start[kRadix];
  __shared__ unsigned wtot[kSortThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  base[threadIdx.x] = offsets[(size_t)threadIdx.x * gridDim.x + blockIdx.x];   // kRadix == kSortThreads
  const long long b0 = (long long)blockIdx.x * tile, b1 = min(n, b0 + tile);
  for (long long c0 = b0; c0 < b1; c0 += kSortChunk) {
    for (int i = lane; i < kRadix; i += 32) wcount[w][i] = 0;
    __syncwarp();
    const long long seg = c0 + (long long)w * (32 * kSortItems) + lane;
    unsigned long long key[kSortItems];
    unsigned rank[kSortItems];
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) key[j] = seg + 32 * j < b1 ? __ldcs(in + seg + 32 * j) : 0ull;
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
      const bool valid = seg + 32 * j < b1;
      const int d = valid ? (int)((key[j] >> shift) & (kRadix - 1)) : kRadix;
      const unsigned peers = __match_any_sync(0xffffffffu, d);
      const unsigned before = valid ? wcount[w][d] : 0u;
      rank[j] = before + __popc(peers & below);
      __syncwarp();
      if (valid && (peers & below) == 0) wcount[w][d] = before + __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    {   // thread = digit: exclusive counts over the warps, then over the digits
      unsigned run = 0;
#pragma unroll
      for (int ww = 0; ww < kSortThreads / 32; ++ww) {
        const unsigned c = wcount[ww][threadIdx.x];
        wcount[ww][threadIdx.x] = run;
        run += c;
      }
      unsigned incl = run;
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) wtot[w] = incl;
      __syncthreads();
      unsigned pre = 0;
      for (int ww = 0; ww < w; ++ww) pre += wtot[ww];
      start[threadIdx.x] = pre + incl - run;
      __syncthreads();
#pragma unroll
      for (int j = 0; j < kSortItems; ++j)
        if (seg + 32 * j < b1) {
          const int d = (int)((key[j] >> shift) & (kRadix - 1));
          buf[start[d] + wcount[w][d] + rank[j]] = key[j];
        }
      __syncthreads();
      const int count = (int)min((long long)kSortChunk, b1 - c0);
      for (int i = threadIdx.x; i < count; i += kSortThreads) {
        const unsigned long long k = buf[i];
        const int d = (int)((k >> shift) & (kRadix - 1));
        out[base[d] + (unsigned)i - start[d]] = k;
      }
      __syncthreads();
      base[threadIdx.x] += run;
    }
  }
}

// Exclusive scan of digit-major histograms (and of any unsigned array) in three phases.
__global__ void k_scan_partials(const unsigned* __restrict__ in, long long n, long long tile,
                                unsigned long long* partial) {
  __shared__ unsigned long long red[32];
  const long long b0 = (long long)blockIdx.x * tile, b1 = min(n, b0 + tile);
  unsigned long long acc = 0;
  for (long long i = b0 + threadIdx.x; i < b1; i += blockDim.x) acc += in[i];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int j = 0; j < (int)(blockDim.x >> 5); ++j) t += red[j];
    partial[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(1024) k_scan_top(unsigned long long* partial, int g) {   // one CTA
  __shared__ unsigned long long wsum[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long carry = 0;
  for (int c0 = 0; c0 < g; c0 += 1024) {
    const int i = c0 + threadIdx.x;
    const unsigned long long v = i < g ? partial[i] : 0;
    unsigned long long incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    unsigned long long pre = carry, all = carry;
    for (int ww = 0; ww < 32; ++ww) {
      if (ww < w) pre += wsum[ww];
      all += wsum[ww];
    }
    if (i < g) partial[i] = pre + incl - v;
    carry = all;
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[g] = carry;
}

// out[i] = partial[cta] + exclusive prefix inside the tile (tile-serial chunks of blockDim).
// in and out may be the same array (the radix sort scans its histogram in place): every
// element is read by the thread that later writes it, so neither pointer is __restrict__.
template <class OutT>
__global__ void k_scan_down(const unsigned* in, OutT* out, long long n, long long tile,
                            const unsigned long long* __restrict__ partial) {
  __shared__ unsigned long long wsum[32];
  __shared__ unsigned long long carry;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = partial[blockIdx.x];
  __syncthreads();
  const long long b0 = (long long)blockIdx.x * tile, b1 = min(n, b0 + tile);
  for (long long c0 = b0; c0 < b1; c0 += blockDim.x) {
    const long long i = c0 + threadIdx.x;
    const unsigned long long v = i < b1 ? in[i] : 0;
    unsigned long long incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    if (w == 0) {
      unsigned long long t = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += y;
      }
      wsum[lane] = t;
    }
    __syncthreads();
    const unsigned long long before = carry + (w > 0 ? wsum[w - 1] : 0);
    if (i < b1) out[i] = (OutT)(before + incl - v);
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = before + incl;
    __syncthreads();
  }
}

// Run-length encoding of sorted keys: head flags.
__global__ void k_rle_flags(const unsigned long long* __restrict__ keys, long long n, unsigned* flags) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    flags[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1u : 0u;
}

// Unique keys and their counts: run j spans [head_j, head_{j+1}).
__global__ void k_rle_emit(const unsigned long long* __restrict__ keys, long long n, const unsigned* __restrict__ flags,
                           const long long* __restrict__ pos, unsigned long long* ukeys, long long* heads) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    if (flags[i]) {
      ukeys[pos[i]] = keys[i];
      heads[pos[i]] = i;
    }
}

static int scan_grid(long long n, int sms) {
  long long g = (n + 4095) / 4096;
  if (g < 1) g = 1;
  if (g > 4LL * sms) g = 4LL * sms;
  return (int)g;
}

void exclusive_scan_u32(const unsigned* in, long long* out, long long n, unsigned long long* partial, int sms,
                        cudaStream_t s) {
  const int g = scan_grid(n, sms);
  const long long tile = (n + g - 1) / g;
  k_scan_partials<<<g, 256, 0, s>>>(in, n, tile, partial);
  k_scan_top<<<1, 1024, 0, s>>>(partial, g);
  k_scan_down<long long><<<g, 256, 0, s>>>(in, out, n, tile, partial);
}

long long scan_partial_capacity(int sms) { return 4LL * sms + 1; }

void radix_sort_u64(unsigned long long* keys, unsigned long long* tmp, long long n, int low, int bits, unsigned* hist,
                    unsigned long long* partial, int sms, cudaStream_t s, unsigned long long** result) {
  unsigned long long* a = keys;
  unsigned long long* b = tmp;
  const int g = (int)std::min<long long>(std::max<long long>((n + 8191) / 8192, 1), 2LL * sms);
  const long long tile = (n + g - 1) / g;
  for (int shift = low; shift < low + bits; shift += kRadixBits) {
    k_radix_hist<<<g, kSortThreads, 0, s>>>(a, n, tile, shift, hist);
    const long long hn = (long long)kRadix * g;
    const int sg = scan_grid(hn, sms);
    const long long stile = (hn + sg - 1) / sg;
    k_scan_partials<<<sg, 256, 0, s>>>(hist, hn, stile, partial);
    k_scan_top<<<1, 1024, 0, s>>>(partial, sg);
    k_scan_down<unsigned><<<sg, 256, 0, s>>>(hist, hist, hn, stile, partial);
    k_radix_scatter<<<g, kSortThreads, 0, s>>>(a, b, n, tile, shift, hist);
    std::swap(a, b);
  }
  *result = a;
}

long long radix_hist_capacity(long long n, int sms) {
  const long long g = std::min<long long>(std::max<long long>((n + 8191) / 8192, 1), 2LL * sms);
  return (long long)kRadix * g;
}

void rle(const unsigned long long* keys, long long n, unsigned* flags, long long* pos, unsigned long long* ukeys,
         long long* heads, unsigned long long* partial, int sms, cudaStream_t s) {
  const int g = (int)std::min<long long>(std::max<long long>((n + 255) / 256, 1), 8LL * sms);
  k_rle_flags<<<g, 256, 0, s>>>(keys, n, flags);
  exclusive_scan_u32(flags, pos, n, partial, sms, s);
  k_rle_emit<<<g, 256, 0, s>>>(keys, n, flags, pos, ukeys, heads);
}

}  // namespace sbpb
