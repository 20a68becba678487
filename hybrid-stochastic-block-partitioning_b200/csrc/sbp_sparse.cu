// Kernels of the row-hashed (sparse) block matrix used when B is large: rebuild from the edge
// list (Blockmodel::initialize_edge_counts, src/blockmodel/blockmodel.cpp:187-255, through a
// sort of (b_src, b_dst) keys), and the repair steps after a hashed row ran out of room.
#include "sbp_kernels.cuh"

namespace sbpb {

// (b[src], b[dst]) and (b[dst], b[src]) keys of every edge: row << bits | column.
__global__ void k_edge_keys(GraphView g, const int* __restrict__ b, const int* __restrict__ out_src, int bits,
                            unsigned long long* keys, unsigned long long* keysT) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < g.E; e += stride) {
    const unsigned long long bs = (unsigned)b[__ldg(out_src + e)], bd = (unsigned)b[__ldg(g.out_idx + e)];
    keys[e] = bs << bits | bd;
    keysT[e] = bd << bits | bs;
  }
}

// First unique key of every row, by a search of the sorted keys: neighbouring rows search nearly the same
// places.  (A thread a key that writes the offsets of the rows it opens leaves a run of empty rows to one
// thread: a blockmodel of 600,000 blocks of which 570,000 have no edge took 6.4 ms to create, with the search
// 1.25; 10 million keys and no empty row: the same.)  rowptr has B + 1 entries.
__global__ void k_unique_rows(const unsigned long long* __restrict__ ukeys, long long n, int B, int bits,
                              long long* rowptr) {
  const int stride = gridDim.x * blockDim.x;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < B; r += stride) {
    const unsigned long long first = (unsigned long long)r << bits;
    long long lo = 0, hi = n;
    while (lo < hi) {
      const long long mid = (lo + hi) >> 1;
      if (ukeys[mid] < first) lo = mid + 1;
      else hi = mid;
    }
    rowptr[r] = lo;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) rowptr[B] = n;
}

// Row capacity: a power of two of at least factor * cells + 4 factor slots (room to grow: at
// large B most moves add cells, and a full row has to be regrown).  Rows of more than 128
// cells get at most factor 2: the hashed walk reads a row's whole region, and for long rows
// that costs more than the occasional regrowth.
__global__ void k_row_caps(const long long* __restrict__ rowptr, int B, unsigned factor, unsigned* cap, int* mask) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < B; r += gridDim.x * blockDim.x) {
    const unsigned cells = (unsigned)(rowptr[r + 1] - rowptr[r]);
    const unsigned f = cells > 128u && factor > 2u ? 2u : factor;
    unsigned want = f * cells + 4u * f, c = 8u;
    while (c < want) c <<= 1;
    cap[r] = c;
    mask[r] = (int)c - 1;
  }
}

__global__ void k_fill_empty(int2* slot, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    slot[i] = make_int2(-1, 0);
}

// One thread per cell: its entry of the compressed (sorted) row and, with slots given, its hashed
// slot (a cell's key is its own, so the thread whose compare-and-swap takes a free slot owns it; the
// row's capacity is at least twice its cells and 8).  Where a cell sits in its row depends on the
// order of arrival, which no result does.  (One thread per row, its insertions one after another,
// took 1.2 ms for 10 million cells.)
__global__ void k_fill_rows(const long long* __restrict__ rowptr, const unsigned long long* __restrict__ ukeys,
                            const long long* __restrict__ heads, long long nu, long long nedges, int B, int bits,
                            const long long* __restrict__ base, const int* __restrict__ mask, int2* slot,
                            int* csr_ptr, int* csr_idx, int* csr_val) {
  const long long stride = (long long)gridDim.x * blockDim.x, first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (long long r = first; r <= B; r += stride) csr_ptr[r] = (int)rowptr[r];
  for (long long j = first; j < nu; j += stride) {
    const unsigned long long key = ukeys[j];
    const int row = (int)(key >> bits), col = (int)(key & ((1ull << bits) - 1ull));
    const int cnt = (int)((j + 1 < nu ? heads[j + 1] : nedges) - heads[j]);
    csr_idx[j] = col;
    csr_val[j] = cnt;
    if (!slot) continue;
    const long long b0 = base[row];
    const int m = mask[row];
    unsigned h = slot_hash(col) & (unsigned)m;
    for (int probe = 0; probe <= m; ++probe) {
      if (atomicCAS(&slot[b0 + h].x, -1, col) == -1) {
        slot[b0 + h].y = cnt;
        break;
      }
      h = (h + 1) & (unsigned)m;
    }
  }
}

// Regrowth of the hashed rows that ran out of room (one side: rows of M or of MT).  A flagged
// row x gets a region of the power of two at least twice its old room and at least
// 2 min(deg[x], B) + 16 slots, taken after the `top` slots in use; with no room left below
// `limit` the step reports it and changes nothing for that row.
__global__ void k_regrow_alloc(const int* __restrict__ full, const int* __restrict__ deg, int B, long long top,
                               long long limit, unsigned long long* used, unsigned long long* nrows, long long* base,
                               int* mask, int* list, unsigned long long* no_room) {
  for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < B; x += gridDim.x * blockDim.x) {
    if (!full[x]) continue;
    const long long need = 2LL * (long long)min(deg[x], B) + 16;
    long long cap = 2LL * ((long long)mask[x] + 1);
    while (cap < need) cap <<= 1;
    const unsigned long long off = atomicAdd(used, (unsigned long long)cap);
    if (cap > (1LL << 30) || top + (long long)off + cap > limit) {
      atomicOr(no_room, 1ull);
      continue;
    }
    base[x] = top + (long long)off;
    mask[x] = (int)(cap - 1);
    list[atomicAdd(nrows, 1ull)] = x;
  }
}

// Empty slots in the new regions (one CTA per listed row).
__global__ void k_regrow_clear(const int* __restrict__ list, int n, const long long* __restrict__ base,
                               const int* __restrict__ mask, int2* slot) {
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int x = list[i];
    const long long b0 = base[x];
    const int cap = mask[x] + 1;
    for (int j = threadIdx.x; j < cap; j += blockDim.x) slot[b0 + j] = make_int2(-1, 0);
  }
}

// Recount the regrown rows: every edge (b_src, b_dst) adds one to row b_src of M when that row
// is flagged and to row b_dst of MT when that one is (the new regions cannot run out of room).
// Few rows are flagged, so a lane asks for its vertex's block whether it has edges to add, and the
// warp then walks the lists of those that have.  (Every edge asking for both its ends took 114 us
// for 12 million edges, once a batch.)
__global__ void k_regrow_fill(GraphView g, BlockView bm) {
  const int* full_r = bm.overflow + 1;
  const int* full_c = bm.overflow + 1 + bm.B;
  const int lane = threadIdx.x & 31;
  const int step = gridDim.x * blockDim.x;
  for (int base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; base < g.V; base += step) {
    const int v = base + lane;
    const int b = v < g.V ? bm.b[v] : 0;
    unsigned rows = __ballot_sync(kFull, v < g.V && full_r[b]), cols = __ballot_sync(kFull, v < g.V && full_c[b]);
    for (; rows; rows &= rows - 1) {
      const int l = __ffs(rows) - 1, x = base + l, bx = __shfl_sync(kFull, b, l);
      for (int e = g.out_ptr[x] + lane; e < g.out_ptr[x + 1]; e += kWarp)
        hashed_add(bm.rbase, bm.rmask, bm.rslot, bx, bm.b[__ldg(g.out_idx + e)], 1, bm.overflow, bm.overflow + 1);
    }
    for (; cols; cols &= cols - 1) {   // in-lists leave the self loop out
      const int l = __ffs(cols) - 1, x = base + l, bx = __shfl_sync(kFull, b, l);
      for (int e = g.in_ptr[x] + lane; e < g.in_ptr[x + 1]; e += kWarp)
        hashed_add(bm.cbase, bm.cmask, bm.cslot, bx, bm.b[__ldg(g.in_idx + e)], 1, bm.overflow, bm.overflow + 1 + bm.B);
      if (lane == 0 && g.self[x])
        hashed_add(bm.cbase, bm.cmask, bm.cslot, bx, bx, 1, bm.overflow, bm.overflow + 1 + bm.B);
    }
  }
}

// Block degrees from the vertices (out-degree; in-degree with the self loop).
__global__ void k_block_degrees(GraphView g, const int* __restrict__ b, int* d_out, int* d_in) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < g.V; v += gridDim.x * blockDim.x) {
    const int bv = b[v];
    atomicAdd(d_out + bv, g.out_ptr[v + 1] - g.out_ptr[v]);
    atomicAdd(d_in + bv, (g.in_ptr[v + 1] - g.in_ptr[v]) + g.self[v]);
  }
}

// Gibbs batch whose apply overflowed a row: move the assignment now (keeping the old block),
// so the rows can be rebuilt from it before the degree step.
__global__ void k_recover_assign(int* b, const int* moved, const int* n_moved, const int* prop, int* old_block) {
  const int n = *n_moved;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int v = moved[i];
    old_block[v] = b[v];
    b[v] = prop[v];
  }
}

// The degree step of k_apply_finish on the rebuilt rows.
__global__ void k_recover_finish(BlockView bm, const int* moved_list, const int* n_moved, int* next_n_moved,
                                 int* prop, const int* old_block, const int* qr, const int* qs,
                                 const unsigned long long* last, unsigned gen) {
  const int n = *n_moved;
  if (blockIdx.x == 0 && threadIdx.x == 0) *next_n_moved = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int v = moved_list[i];
    const int r = old_block[v], s = prop[v];
    const unsigned long long key = ((unsigned long long)gen << 32) | (unsigned)v;
    if (last[r] == key) set_degree(bm, r, bm.d_out[r] + bm.d_in[r] - bm_get(bm, r, r) - qr[v]);
    if (last[s] == key) set_degree(bm, s, bm.d_out[s] + bm.d_in[s] - bm_get(bm, s, s) - qs[v]);
    prop[v] = -1;
  }
}

// d[r], d[s] of one move (Blockmodel::move_vertex) after its rows were rebuilt.
__global__ void k_fix_move_degrees(BlockView bm, int r, int s, int d_rr, int d_ss) {
  if (threadIdx.x || blockIdx.x) return;
  set_degree(bm, r, bm.d_out[r] + bm.d_in[r] - (bm_get(bm, r, r) + d_rr));
  set_degree(bm, s, bm.d_out[s] + bm.d_in[s] - (bm_get(bm, s, s) + d_ss));
}

// Dense dump of the hashed rows of M (for sbp_get_block_matrix): one thread per slot.
__global__ void k_hashed_to_dense(const long long* __restrict__ base, const int* __restrict__ mask,
                                  const int2* __restrict__ slot, int B, int row0, int rows, int* dense) {
  for (int r = row0 + blockIdx.x; r < row0 + rows && r < B; r += gridDim.x) {
    const long long b0 = base[r];
    const int cap = mask[r] + 1;
    for (int i = threadIdx.x; i < cap; i += blockDim.x) {
      const int2 e = slot[b0 + i];
      if (e.x >= 0) dense[(size_t)(r - row0) * B + e.x] = e.y;
    }
  }
}

}  // namespace sbpb
