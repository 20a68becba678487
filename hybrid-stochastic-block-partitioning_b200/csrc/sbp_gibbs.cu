// Asynchronous Gibbs (finetune::asynchronous_gibbs, src/finetune.cpp:31-89): the evaluation of one
// batch as a kernel of its own, on either storage, and a whole finetune call on a dense block matrix
// -- every sweep's batches, the MDL and the early stop -- as one persistent kernel.
#include "sbp_engine.cuh"
#include "sbp_group.cuh"
#include "sbp_steps.cuh"

namespace sbpb {
namespace {

struct EvalCounts {
  unsigned visit = 0, moved = 0, acc = 0;
};

// Everything one batch's evaluation needs.  Accepted moves go to `moved` (vertex ids) or, where it is
// given, to `moves`: the vertex's record, then (r, s, -, -), so that the apply and the degree step
// find all they need in one load by position.
struct EvalArgs {
  GraphView g;
  BlockView bm;
  const int4* recs;      // vertex records in plan order
  RngParams rng;
  int* prop;
  int* moved;
  int4* moves;           // [2 * batch] or null
  int* status;
  int gmin;              // smallest group
  int slots;             // table slots of the CTA (kGroupWarps regions, or more for a heavy vertex)
  int heavy;             // those of a heavy vertex: a warp's region, twice that, ..., all of them
};

template <bool kDirect, Store ST>
__device__ __forceinline__ void eval_task(const EvalArgs& a, const GroupTab<kDirect>& T, int4 rec, bool valid, int sweep,
                                          int* n_moved, const Lanes& L, EvalCounts& cnt, int* bins) {
  uint4 x = make_uint4(0, 0, 0, 0);
  if (valid)
    x = draw_record(a.rng, (uint32_t)rec.x, (uint32_t)sweep, 0u, (long long)sweep * a.g.V + rec.x, a.status);
  const GroupEval e = group_evaluate<kDirect, ST>(a.g, a.bm, T, valid, rec, a.rng.moves != 0, x, L, a.status, bins);
  if (valid && L.gl == 0) {
    cnt.visit++;
    if (e.s != e.r) cnt.moved++;
    if (e.accepted) {
      cnt.acc++;
      a.prop[e.v] = e.s;
      const int i = atomicAdd(n_moved, 1);
      if (a.moves) {
        a.moves[2 * i] = rec;
        a.moves[2 * i + 1] = make_int4(e.r, e.s, 0, 0);
      } else {
        a.moved[i] = e.v;
      }
    }
  }
  T.clear(e.n, L);
}

// The record of this lane's vertex in task `task` of a batch (zeros: none).
__device__ __forceinline__ int4 task_record(const EvalArgs& a, const BatchDesc& b, const GroupTask& k, int light,
                                            int lane, bool* valid) {
  const int i = k.first + (lane >> (5 - k.lg));
  *valid = i < k.end;
  return *valid ? __ldg(a.recs + (light ? b.light_begin : b.heavy_begin) + i) : make_int4(0, 0, 0, 0);
}

// One batch: tasks of 32 / G vertices, a warp each, the largest degrees first.  Strided over the
// grid, so with the batch ordered by degree every warp gets a similar share.
template <bool kDirect, Store ST>
__device__ __forceinline__ void eval_batch(const EvalArgs& a, BatchDesc b, int sweep, int* n_moved, int* smem,
                                           EvalCounts& cnt) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wid = blockIdx.x * kGroupWarps + warp;
  // Two passes over one body: the heavy vertices, a warp each, then the light ones.  As many warps of a
  // CTA take heavy ones as its table has shares large enough for any of them (with a histogram by block:
  // all); few as they are, they go to all CTAs before a second warp takes one.
#pragma unroll 1
  for (int light = b.heavy_n > 0 ? 0 : 1; light < 2; ++light) {
    const int at_once = kDirect || light ? kGroupWarps : min(kGroupWarps, a.slots / a.heavy);
    const int tasks = light ? group_tasks(b, a.gmin) : b.heavy_n;
    const int first_task = light ? wid : warp < at_once ? warp * (int)gridDim.x + (int)blockIdx.x : tasks;
#pragma unroll 1
    for (int task = first_task; task < tasks; task += at_once * (int)gridDim.x) {
      const GroupTask k = group_task(b, a.gmin, task, light);
      const Lanes L(32 >> k.lg, lane);
      const int sub = lane >> (5 - k.lg), share = kDirect || light ? kRegionSlots >> k.lg : a.heavy;
      const GroupTab<kDirect> T =
          group_tab<kDirect>(smem, a.slots, warp * (kDirect || light ? kRegionSlots : a.heavy) + sub * share, share);
      bool valid;
      const int4 rec = task_record(a, b, k, light, lane, &valid);
      eval_task<kDirect, ST>(a, T, rec, valid, sweep, n_moved, L, cnt,
                             smem + group_smem_bytes(kDirect, a.slots) / sizeof(int) + 32 * warp);
    }
    if (!kDirect && !light) __syncthreads();   // the shares lie across the regions
  }
}

__device__ __forceinline__ void add_counts(EvalCounts c, unsigned long long* counters) {
  const unsigned v = __reduce_add_sync(kFull, c.visit), m = __reduce_add_sync(kFull, c.moved),
                 x = __reduce_add_sync(kFull, c.acc);
  if ((threadIdx.x & 31) == 0 && v) {
    atomicAdd(counters + 0, (unsigned long long)v);
    atomicAdd(counters + 1, (unsigned long long)m);
    atomicAdd(counters + 2, (unsigned long long)x);
  }
}

template <bool kDirect, Store ST>
__global__ void __launch_bounds__(kGroupThreads, 2)
    k_gibbs_eval(const __grid_constant__ EvalArgs a, BatchDesc b, int sweep, int* n_moved, unsigned long long* counters) {
  extern __shared__ int smem[];
  group_tabs_init<kDirect>(smem, a.slots);
  __syncthreads();
  EvalCounts cnt;
  eval_batch<kDirect, ST>(a, b, sweep, n_moved, smem, cnt);
  add_counts(cnt, counters);
}

// ------------------------------------------------------------------------------------------
// A whole finetune call in one kernel.  Per batch: evaluation, apply, degree step, each over the
// whole grid and separated by a barrier over the grid; per sweep: the MDL's partial sums, then
// every CTA forms the same total and takes the same early-stop decision
// (src/finetune.cpp:144-162), so no CTA waits for another's.  As launches (three per batch, replayed
// by a CUDA graph) the same work paid a launch gap and a ramp-up and tail per step.
//
// The barrier is the cluster's where the grid is one cluster (small batches), else a counter in
// global memory, for which the kernel is launched cooperatively: every CTA is resident.  A wait
// gives up after an iteration limit: the CTA that gives up sets the status word and the abort flag
// and every CTA leaves at its next barrier.
// Loads of state that another phase writes are plain loads: the barrier's acquire makes them
// coherent.  Only what no phase writes goes through the read-only cache.
// ------------------------------------------------------------------------------------------
struct SweepsArgs {
  EvalArgs e;
  const BatchDesc* batches;
  int nbatches;
  int max_sweeps;
  int bracket;
  int mdl_cells;
  int mdl_ctas;
  int cluster;              // 1: the grid is one cluster
  unsigned gen0;            // batch generation before the call
  unsigned wait_limit;      // polls of a barrier before it gives up
  unsigned long long* last;
  const int* out_src;
  double* partial;
  unsigned long long* counters;
  int* n_moved;             // three slots taken in turn, zero at launch
  unsigned* bar;            // [0] arrivals (0 at launch), [1] abort flag (0 at launch)
  SweepsResult* result;
};

// Barrier over the grid; false when a wait gave up (the same for every thread of the CTA).
__device__ __forceinline__ bool sync_grid(const SweepsArgs& a, unsigned* target, int* s_abort) {
  if (a.cluster) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    return true;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    *target += gridDim.x;
    atomicAdd(a.bar, 1u);
    unsigned polls = 0, seen;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.bar) : "memory");
      if ((int)(seen - *target) >= 0) break;
      ++polls;
      if ((polls & 1023u) == 0 && *(volatile unsigned*)(a.bar + 1)) {
        *s_abort = 1;
        break;
      }
      if (polls > a.wait_limit) {
        atomicOr(a.e.status, kErrGridWait);
        atomicExch(a.bar + 1, 1u);
        *s_abort = 1;
        break;
      }
    }
    __threadfence();
  }
  __syncthreads();
  return *(volatile int*)s_abort == 0;
}

template <bool kDirect>
__global__ void __launch_bounds__(kGroupThreads, 2) k_gibbs_sweeps(const __grid_constant__ SweepsArgs a) {
  extern __shared__ int smem[];
  __shared__ double red[32];
  __shared__ int s_abort, s_stop;
  const GraphView& g = a.e.g;
  const BlockView& bm = a.e.bm;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wid = blockIdx.x * kGroupWarps + warp, nw = gridDim.x * kGroupWarps;
  group_tabs_init<kDirect>(smem, a.e.slots);
  if (tid == 0) s_abort = 0;
  unsigned target = 0;
  EvalCounts cnt;
  double constant = 0.0, initial = 0.0, mdl = 0.0, d1 = 0.0, d2 = 0.0;   // thread 0: MDL terms, the last two deltas
  if (tid == 0) constant = mdl_constant(g.V, g.E, bm.B);
  unsigned gen = a.gen0;
  int slot = 0;
  int count = 0;
  for (int it = -1;; ++it) {
    if (it >= 0) {
      for (int bt = 0; bt < a.nbatches; ++bt) {
        const BatchDesc b = a.batches[bt];
        int* n_cur = a.n_moved + slot;
        slot = slot == 2 ? 0 : slot + 1;
        if (blockIdx.x == 0 && tid == 0) a.n_moved[slot] = 0;   // the next batch's; last read two barriers ago
        eval_batch<kDirect, Store::kDense>(a.e, b, it, n_cur, smem, cnt);
        if (!sync_grid(a, &target, &s_abort)) return;
        const int n = *(volatile int*)n_cur;
        ++gen;
        if (n == 0) continue;   // the same for the whole grid
        // A batch accepts far fewer moves than there are warps (183 to 454 of 10,000 vertices on the
        // 100,000-vertex graph, against 2,368 warps), and the longest neighbour lists decide the
        // phase: up to four warps share a move.
        const int parts = min(4, max(1, nw / n));
        for (int q = wid; q < n * parts; q += nw) {
          const int part = q / n, i = q - part * n;
          const int4 rec = a.e.moves[2 * i], mv = a.e.moves[2 * i + 1];
          if (part > 0 && part * 2 * kWarp >= rec.z + (rec.w >> 1)) continue;
          const MoveQuirks m =
              apply_moved_record<Store::kDense>(g, bm, rec, mv.x, mv.y, a.e.prop, a.last, gen, lane, part, parts);
          if (lane == 0) {   // zero until here (eval_task)
            atomicAdd(&a.e.moves[2 * i + 1].z, m.qr);
            atomicAdd(&a.e.moves[2 * i + 1].w, m.qs);
          }
        }
        if (!sync_grid(a, &target, &s_abort)) return;
        for (int i = blockIdx.x * kGroupThreads + tid; i < n; i += gridDim.x * kGroupThreads) {
          const int v = a.e.moves[2 * i].x;
          const int4 mv = a.e.moves[2 * i + 1];
          finish_move<Store::kDense>(bm, v, mv.x, mv.y, {mv.z, mv.w}, a.e.prop, a.last, gen);
        }
        if (!sync_grid(a, &target, &s_abort)) return;
      }
    }
    // entropy::mdl over the virtual grid of every other path
    for (int vc = blockIdx.x; vc < a.mdl_ctas; vc += gridDim.x) {
      const double t = a.mdl_cells ? mdl_cells_part(bm, vc, a.mdl_ctas, red)
                                   : mdl_edges_part<Store::kDense>(g, bm, a.out_src, vc, a.mdl_ctas, red);
      if (tid == 0) a.partial[vc] = t;
    }
    if (!sync_grid(a, &target, &s_abort)) return;
    const double L = mdl_total(a.partial, a.mdl_ctas, red);
    if (tid == 0) {
      mdl = constant - L;
      bool stop = false;
      if (it < 0) {
        initial = (double)(float)mdl;   // the reference stores the entropy as float
      } else {
        const double d0 = mdl - initial;   // last_iteration_entropy is never updated
        if (d0 == 0.0) {
          stop = true;
        } else if (it >= 3) {
          double average = d0 + d1 + d2;
          average /= -3.0;
          stop = average < (a.bracket ? 1e-4 * initial : 5e-4 * initial);
        }
        d2 = d1;
        d1 = d0;
        if (it + 1 >= a.max_sweeps) stop = true;
      }
      s_stop = stop ? 1 : 0;
    }
    __syncthreads();
    count = it + 1;
    if (s_stop) break;
    __syncthreads();
  }
  add_counts(cnt, a.counters);
  if (blockIdx.x == 0 && tid == 0) {
    a.result->mdl = mdl;
    a.result->sweeps = count;
  }
}

constexpr int kMaxCluster = 16;
constexpr int kClusterBatch = 128;   // largest batch run on one cluster: a warp for every vertex

EvalArgs eval_args(const SbpGraph& g, SbpBlockmodel& bm, const BatchPlan& plan, const RngParams& rng) {
  EvalArgs a;
  a.g = g.view();
  a.bm = bm.view();
  a.recs = plan.recs.p;
  a.rng = rng;
  a.prop = bm.prop.p;
  a.moved = bm.moved.p;
  a.moves = nullptr;
  a.status = Context::get().status;
  // a heavy vertex needs a slot for each of its distinct neighbour blocks, of which there are at
  // most B; twice that many while they fit
  const int distinct = std::min(g.max_k, bm.B);
  a.slots = std::max(kGroupWarps * kRegionSlots, std::min(kMaxCap, pow2_at_least(2 * distinct)));
  // A share for a heavy vertex: at most three quarters full, or all there is.  6,000 vertices of 670
  // neighbours, three sweeps: 1.15 ms at 300 blocks (a share a warp), 1.38 at 500 (four a CTA), 2.66 at
  // 3,000 (two), where one warp a CTA with the whole table took 3.30, 2.23 and 2.87.
  a.heavy = std::min(a.slots, std::max(kRegionSlots, pow2_at_least(distinct + (distinct + 2) / 3)));
  a.gmin = 8;
  return a;
}

// After a kernel that gave up somewhere in a batch: moves without their apply, counts half updated,
// generations begun.  The assignment is sound at every moment (a vertex changes block by one store), so
// the state is that assignment with everything else made anew.
void recover(SbpBlockmodel& bm, const SbpGraph& g) {
  bm.init_vertex_scratch(bm.V);
  SBP_CUDA(cudaMemsetAsync(bm.last.p, 0, sizeof(unsigned long long) * bm.B, Context::get().stream));
  rebuild(bm, g);
}

// Smallest group for a batch: eight lanes a vertex once that still gives every resident warp a
// task, else as many lanes as the idle warps allow -- a visit's chain gets shorter with more lanes.
int group_min(int batch, int warps) {
  if (g_group_kernel == 0) return 32;
  if (g_group_kernel == 2) return 8;
  return batch >= 4 * warps / 2 ? 8 : batch >= warps ? 16 : 32;
}

}  // namespace

void launch_gibbs_eval(const SbpGraph& g, SbpBlockmodel& bm, const BatchPlan& plan, int bt, const RngParams& rng,
                       int sweep, int* n_moved) {
  Context& c = Context::get();
  EvalArgs a = eval_args(g, bm, plan, rng);
  const BatchDesc& d = plan.desc[bt];
  const int n = d.light_n + d.heavy_n;
  const bool direct = !bm.sparse && bm.B <= kSmallB;
  a.gmin = group_min(n, 2 * kGroupWarps * c.num_sms);
  const size_t smem = group_smem_bytes(direct, a.slots) + (bm.sparse ? 32 * kGroupWarps * sizeof(int) : 0);   // walk bins
  const auto k = bm.sparse ? k_gibbs_eval<false, Store::kHashed>
                 : direct  ? k_gibbs_eval<true, Store::kDenseFrozen>
                           : k_gibbs_eval<false, Store::kDenseFrozen>;
  set_smem_limit((const void*)k, smem);
  k<<<grid_for((long long)n * a.gmin, 32 * kGroupWarps, 64 * c.num_sms), kGroupThreads, smem, c.stream>>>(
      a, d, sweep, n_moved, c.counters);
}

SweepsResult gibbs_sweeps(SbpBlockmodel& bm, const SbpGraph& g, const BatchPlan& plan, const RngParams& rng,
                          int max_sweeps, bool bracket) {
  Context& c = Context::get();
  SweepsArgs a;
  a.e = eval_args(g, bm, plan, rng);
  bm.moves.reserve(2 * (size_t)plan.max_batch);
  a.e.moves = bm.moves.p;
  a.batches = plan.desc_dev.p;
  a.nbatches = (int)plan.desc.size();
  a.max_sweeps = max_sweeps;
  a.bracket = bracket ? 1 : 0;
  a.mdl_cells = mdl_cell_form(bm, g) ? 1 : 0;
  a.mdl_ctas = mdl_grid(bm, g);
  a.gen0 = bm.gen;
  a.wait_limit = (unsigned)g_sweep_wait_limit;
  a.last = bm.last.p;
  a.out_src = g.out_src.p;
  a.partial = c.partial;
  a.counters = c.counters;
  a.n_moved = c.sweeps->n_moved;
  a.bar = c.sweeps->bar;
  a.result = &c.sweeps->result;
  const bool direct = bm.B <= kSmallB;
  const size_t smem = group_smem_bytes(direct, a.e.slots);
  const auto k = direct ? k_gibbs_sweeps<true> : k_gibbs_sweeps<false>;
  set_smem_limit((const void*)k, smem);
  int per_sm = 0;
  SBP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kGroupThreads, smem));
  if (per_sm < 1) throw Error(SBP_ERR_UNSUPPORTED, "vertex degree too large for the finetune kernel");
  // Small batches: one cluster of up to 16 CTAs, whose hardware barrier takes 0.3 us against 1 us
  // through global memory (three of them in a batch of some 12 us).  Only while every vertex gets a
  // warp: at 250 vertices a batch the second round of evaluations costs more than the barriers
  // (1,000 vertices in ten batches: 69 ms a partition against 80; 2,500: 127 against 110).
  int cluster = 0;
  if (plan.max_batch <= kClusterBatch) {
    a.e.gmin = group_min(plan.max_batch, kMaxCluster * kGroupWarps);
    cluster = std::min(kMaxCluster, grid_for((long long)plan.max_batch * a.e.gmin, 32 * kGroupWarps, kMaxCluster));
    cluster = pow2_at_least(cluster);
    if (cluster > 8 && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      cluster = 8;
    }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kGroupThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c.stream;
  cudaLaunchAttribute at[1];
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cluster > 0) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(cluster);
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, k, &cfg) != cudaSuccess || fit < 1) {
      cudaGetLastError();
      cluster = 0;
    }
  }
  a.cluster = cluster > 0 ? 1 : 0;
  if (!cluster) {
    const int resident = per_sm * c.num_sms;
    a.e.gmin = group_min(plan.max_batch, resident * kGroupWarps);
    const int wanted = (int)std::max<long long>(
        ((long long)plan.max_batch * a.e.gmin / 32 + kGroupWarps - 1) / kGroupWarps, a.mdl_ctas);
    cfg.gridDim = dim3(std::max(1, std::min(resident, wanted)));
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  SBP_CUDA(cudaMemsetAsync(c.sweeps, 0, sizeof(SweepsState), c.stream));
  SBP_CUDA(cudaLaunchKernelEx(&cfg, k, a));
  SBP_CHECK_LAUNCH();
  SweepsResult r;
  SBP_CUDA(SBP_COPY_ASYNC(&r, a.result, sizeof r, cudaMemcpyDeviceToHost, c.stream));
  c.sync();
  // Before any error is thrown: bm.last holds the generations of the batches that ran.  They counted in
  // words of their own, so the slot that the next launch per batch takes, gen & 1 of bm.n_moved, has to
  // be the one it would have taken before this call: that one is zero, the other keeps the last such
  // batch's count.
  bm.gen += ((unsigned)(a.nbatches * r.sweeps) + 1u) & ~1u;
  if (r.sweeps == 0) recover(bm, g);
  c.check_status();   // before the result is used: a kernel that gave up leaves none
  return r;
}

}  // namespace sbpb
