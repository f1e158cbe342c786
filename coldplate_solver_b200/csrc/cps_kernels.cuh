// The persistent kernels.  Their instantiations are compiled in translation
// units of their own (cps_grid_*.cu, cps_batch_*.cu), side by side: together in
// one they take minutes.
#pragma once
#include "cps_device.cuh"

// Monitor: the outer loop's pressure-drop monitor and gate compiled in (a
// separate instantiation: compiling it into the plain kernel slowed every
// outer iteration by 60 % on B200).  Pseudo: the pseudo-transient term and the
// CFL controllers compiled in (their registers spill the plain kernel's).
// Carry: the PCG forms and options compiled in (cps::Carries).
template <typename T, bool Monitor, bool Pseudo, int Carry>
__global__ void __launch_bounds__(cps::kThreads, Carry == cps::kCluster ? 1 : CPS_MIN_BLOCKS) cps_grid_kernel(cps::DesignView d, cps::RunControl rc,
                                                                cps::GridBarrier* bar, double* red) {
  __shared__ double smem[(Monitor ? cps::kPlaneSums : cps::kRedWidth) * 8];
  __shared__ cps::PseudoRun s_pr;
  __shared__ double out[8];
  extern __shared__ __align__(128) char tile_smem[];
  if ((int)blockIdx.x >= rc.ctas) return;
  cps::GridGroup g{bar, red, rc.status, blockIdx.x, (unsigned)rc.ctas, 0u, 0ull};
  if (!cps::tile_buffer_fits(tile_smem, cps::kernel_smem_bytes<T, Carry, Monitor>(), rc.status)) return;
  cps::tma_barriers_init();
  cps::load_pseudo(d, s_pr);
  __syncthreads();
  const bool clustered = Carry == cps::kCluster && blockIdx.x < cps::kClusterCtas;  // the cluster that runs the PCG
  if (clustered) cps::cluster_enter();
  cps::SweepHint hint{2, 2};
  for (int it = 0; it < rc.n_outer; ++it) {
    const int r = cps::outer_iteration<T, cps::GridGroup, Monitor, Pseudo, Carry>(
        d, g, smem, tile_smem, out, it + 1 == rc.n_outer, rc.stop_on_conv != 0, rc.eps, rc.iter0 + it,
        rc.dplog ? rc.dplog + (size_t)4 * it : nullptr, rc.dp_converged, &s_pr, &hint);
    if (r < 0) {
      if (clustered && r != cps::kLeft) cps::cluster_leave(true);
      return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      for (int k = 0; k < 8; ++k) rc.hist[(size_t)it * 8 + k] = out[k];
      *rc.n_done = it + 1;
    }
    if (r == 1) break;
  }
  if (clustered) cps::cluster_leave(false);
}

// Batched solves: each cluster takes the next design from the queue and runs
// its outer iterations to convergence or to the item's budget.
template <typename T, bool Options, int Carry>
__global__ void __launch_bounds__(cps::kThreads) cps_cluster_kernel(const cps::BatchItem* __restrict__ items,
                                                                   const int* __restrict__ order, int n_items,
                                                                   int* queue, cps::BatchResult* results) {
  __shared__ double smem[cps::kRedWidth * 8];
  __shared__ double redbuf[2 * cps::kRedWidth];
  __shared__ __align__(16) cps::BatchItem s_item;
  __shared__ cps::PseudoRun s_pr;
  __shared__ int s_next;
  __shared__ double out[8];
  extern __shared__ __align__(128) char tile_smem[];
  cps::cg::cluster_group cl = cps::cg::this_cluster();
  cps::ClusterGroup g{redbuf, nullptr, cl.block_rank(), cl.num_blocks(), 0u, 0u, false};
  if (!cps::tile_buffer_fits(tile_smem, cps::tile_smem_bytes<T>(), &results[0].status)) return;
  if (threadIdx.x == 0) cps::s_cluster_leave = cps::kStay;
  cps::tma_barriers_init();
  for (;;) {
    if (g.rank == 0 && threadIdx.x == 0) s_next = atomicAdd(queue, 1);
    g.sync();
    const int idx = *cl.map_shared_rank(&s_next, 0);
    if (idx >= n_items) break;
    const int id = order[idx];
    {
      const int* src = reinterpret_cast<const int*>(items + id);
      int* dst = reinterpret_cast<int*>(&s_item);
      for (int k = threadIdx.x; k < (int)(sizeof(cps::BatchItem) / sizeof(int)); k += blockDim.x) dst[k] = src[k];
    }
    __syncthreads();
    const cps::BatchItem& item = s_item;
    cps::load_pseudo(item.view, s_pr);
    __syncthreads();
    cps::BatchResult* res = results + id;
    g.status = &res->status;
    if (threadIdx.x < 8) out[threadIdx.x] = 0.0;
    int done = 0;
    cps::SweepHint hint{2, 2};
    for (int it = 0; it < item.n_outer; ++it) {
      const int r = cps::outer_iteration<T, cps::ClusterGroup, false, Options, Carry>(
          item.view, g, smem, tile_smem, out, it + 1 == item.n_outer, item.stop_on_conv != 0, item.eps, item.iter0 + it,
          nullptr, nullptr, &s_pr, &hint);
      if (r < 0) {  // a bounded wait expired here or in another CTA; the design's status says so
        if (!g.left) cps::cluster_leave(true, g.barriers + 1);
        return;
      }
      done = it + 1;
      if (g.rank == 0 && threadIdx.x == 0 && item.hist && it < item.hist_cap)
        for (int k = 0; k < 8; ++k) item.hist[(size_t)it * 8 + k] = out[k];
      if (r != 0) break;
    }
    if (g.rank == 0 && threadIdx.x == 0) {
      res->n_done = done;
      const double conv = cps::maxd(cps::maxd(out[0], out[1]), out[3]);
      res->converged = (done > 0 && conv <= item.eps) ? 1 : 0;
      for (int k = 0; k < 8; ++k) res->last[k] = out[k];
    }
    if (!g.sync()) return;  // s_item, s_next and the reduction ring are reused next round
  }
  cl.sync();    // no CTA leaves while another may still read its shared memory
}

// Batched solves on groups of CTAs inside one cooperative launch: CTAs
// [g*K, (g+1)*K) form group g, which takes designs from the queue one at a
// time and runs each with the bounded software barrier of its own counter.
// The group count sets how many designs are in flight (and so the in-flight
// working set against the 126 MB L2); K sets how many CTAs share one design.
template <typename T, bool Options, int Carry>
__global__ void __launch_bounds__(cps::kThreads, CPS_MIN_BLOCKS) cps_group_kernel(const cps::BatchItem* __restrict__ items,
                                                                    const int* __restrict__ order, int n_items,
                                                                    int* queue, cps::BatchResult* results,
                                                                    cps::GridBarrier* bars, double* rings,
                                                                    int* slots, int group_ctas) {
  __shared__ double smem[cps::kRedWidth * 8];
  __shared__ __align__(16) cps::BatchItem s_item;
  __shared__ cps::PseudoRun s_pr;
  __shared__ double out[8];
  extern __shared__ __align__(128) char tile_smem[];
  const unsigned grp = blockIdx.x / group_ctas;
  int* slot = slots + 2 * grp;  // [0] next queue index, [1] group status before a design is assigned
  cps::GridGroup g{bars + grp, rings + (size_t)grp * cps::kRedSlots * group_ctas * cps::kRedWidth, slot + 1,
                   blockIdx.x % group_ctas, (unsigned)group_ctas, 0u, 0ull};
  if (!cps::tile_buffer_fits(tile_smem, cps::tile_smem_bytes<T>(), &results[0].status)) return;
  cps::tma_barriers_init();
  for (;;) {
    g.status = slot + 1;
    if (g.rank == 0 && threadIdx.x == 0) slot[0] = atomicAdd(queue, 1);
    if (!g.sync()) return;
    const int idx = __ldcg(slot);
    if (!g.sync()) return;  // every CTA has read the index before the leader takes the next one
    if (idx >= n_items) return;
    const int id = order[idx];
    {
      const int* src = reinterpret_cast<const int*>(items + id);
      int* dst = reinterpret_cast<int*>(&s_item);
      for (int k = threadIdx.x; k < (int)(sizeof(cps::BatchItem) / sizeof(int)); k += blockDim.x) dst[k] = src[k];
    }
    __syncthreads();
    const cps::BatchItem& item = s_item;
    cps::load_pseudo(item.view, s_pr);
    __syncthreads();
    cps::BatchResult* res = results + id;
    g.status = &res->status;
    if (threadIdx.x < 8) out[threadIdx.x] = 0.0;
    int done = 0;
    cps::SweepHint hint{2, 2};
    for (int it = 0; it < item.n_outer; ++it) {
      const int r = cps::outer_iteration<T, cps::GridGroup, false, Options, Carry>(
          item.view, g, smem, tile_smem, out, it + 1 == item.n_outer, item.stop_on_conv != 0, item.eps, item.iter0 + it,
          nullptr, nullptr, &s_pr, &hint);
      if (r < 0) return;  // a bounded wait expired; the design's status says so
      done = it + 1;
      if (g.rank == 0 && threadIdx.x == 0 && item.hist && it < item.hist_cap)
        for (int k = 0; k < 8; ++k) item.hist[(size_t)it * 8 + k] = out[k];
      if (r != 0) break;
    }
    if (g.rank == 0 && threadIdx.x == 0) {
      res->n_done = done;
      const double conv = cps::maxd(cps::maxd(out[0], out[1]), out[3]);
      res->converged = (done > 0 && conv <= item.eps) ? 1 : 0;
      for (int k = 0; k < 8; ++k) res->last[k] = out[k];
    }
    __syncthreads();  // s_item is reloaded next round
  }
}

// Batched solves in waves: one design per group, groups sized to their
// designs.  CTAs [first[g], first[g+1]) form group g and run design which[g]
// to convergence or to its budget with the bounded software barrier of their
// own counter; their reduction ring starts at first[g] ring rows.
template <typename T, bool Options, int Carry>
__global__ void __launch_bounds__(cps::kThreads, CPS_MIN_BLOCKS) cps_wave_kernel(const cps::BatchItem* __restrict__ items,
                                                                   const int* __restrict__ first,
                                                                   const int* __restrict__ which, int groups,
                                                                   cps::BatchResult* results,
                                                                   cps::GridBarrier* bars, double* rings) {
  __shared__ double smem[cps::kRedWidth * 8];
  __shared__ __align__(16) cps::BatchItem s_item;
  __shared__ cps::PseudoRun s_pr;
  __shared__ double out[8];
  extern __shared__ __align__(128) char tile_smem[];
  if (!cps::tile_buffer_fits(tile_smem, cps::tile_smem_bytes<T>(), &results[which[0]].status)) return;
  cps::tma_barriers_init();
  int lo = 0, hi = groups;  // first[lo] <= blockIdx.x < first[lo + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (first[mid] <= (int)blockIdx.x) lo = mid; else hi = mid;
  }
  const int grp = lo, K = first[grp + 1] - first[grp], id = which[grp];
  {
    const int* src = reinterpret_cast<const int*>(items + id);
    int* dst = reinterpret_cast<int*>(&s_item);
    for (int k = threadIdx.x; k < (int)(sizeof(cps::BatchItem) / sizeof(int)); k += blockDim.x) dst[k] = src[k];
  }
  __syncthreads();
  const cps::BatchItem& item = s_item;
  cps::load_pseudo(item.view, s_pr);
  __syncthreads();
  cps::BatchResult* res = results + id;
  cps::GridGroup g{bars + grp, rings + (size_t)first[grp] * cps::kRedSlots * cps::kRedWidth, &res->status,
                   blockIdx.x - (unsigned)first[grp], (unsigned)K, 0u, 0ull};
  if (threadIdx.x < 8) out[threadIdx.x] = 0.0;
  int done = 0;
  cps::SweepHint hint{2, 2};
  for (int it = 0; it < item.n_outer; ++it) {
    const int r = cps::outer_iteration<T, cps::GridGroup, false, Options, Carry>(
        item.view, g, smem, tile_smem, out, it + 1 == item.n_outer, item.stop_on_conv != 0, item.eps, item.iter0 + it,
        nullptr, nullptr, &s_pr, &hint);
    if (r < 0) return;  // a bounded wait expired; the design's status says so
    done = it + 1;
    if (g.rank == 0 && threadIdx.x == 0 && item.hist && it < item.hist_cap)
      for (int k = 0; k < 8; ++k) item.hist[(size_t)it * 8 + k] = out[k];
    if (r != 0) break;
  }
  if (g.rank == 0 && threadIdx.x == 0) {
    res->n_done = done;
    const double conv = cps::maxd(cps::maxd(out[0], out[1]), out[3]);
    res->converged = (done > 0 && conv <= item.eps) ? 1 : 0;
    for (int k = 0; k < 8; ++k) res->last[k] = out[k];
  }
}

// Every instantiation the library launches, storage type T.  A batch carries
// the on-chip PCG form its designs need, all forms when one of them needs more
// (kForms), and with Options the pseudo-transient term, the CFL controllers
// and the options of cps::kOptions too.
#define CPS_GRID_KERNEL(PRE, T, MONITOR, PSEUDO, CARRY)                                                             \
  PRE template __global__ void cps_grid_kernel<T, MONITOR, PSEUDO, CARRY>(cps::DesignView, cps::RunControl,         \
                                                                          cps::GridBarrier*, double*);
#define CPS_GRID_KERNELS(PRE, T)                                                                                    \
  CPS_GRID_KERNEL(PRE, T, false, false, cps::kFew)                                                                  \
  CPS_GRID_KERNEL(PRE, T, false, false, cps::kMany)                                                                 \
  CPS_GRID_KERNEL(PRE, T, false, false, cps::kLarge)                                                                \
  CPS_GRID_CLUSTER_KERNELS(PRE, T)
#if CPS_TILE_J == 32  // the cluster form is written for 8 x 32 tiles
#define CPS_GRID_CLUSTER_KERNELS(PRE, T) CPS_GRID_KERNEL(PRE, T, false, false, cps::kCluster)
#else
#define CPS_GRID_CLUSTER_KERNELS(PRE, T)
#endif
#define CPS_GRID_OPTION_KERNELS_OF(PRE, T, MONITOR)                                                                 \
  CPS_GRID_KERNEL(PRE, T, MONITOR, true, cps::kFew | cps::kOptions)                                                 \
  CPS_GRID_KERNEL(PRE, T, MONITOR, true, cps::kMany | cps::kOptions)                                                \
  CPS_GRID_KERNEL(PRE, T, MONITOR, true, cps::kLarge | cps::kOptions)
#define CPS_GRID_OPTION_KERNELS(PRE, T) CPS_GRID_OPTION_KERNELS_OF(PRE, T, false)
#define CPS_GRID_MONITOR_KERNELS(PRE, T) CPS_GRID_OPTION_KERNELS_OF(PRE, T, true)
#define CPS_BATCH_KERNELS_OF(PRE, T, OPTIONS, CARRY)                                                                \
  PRE template __global__ void cps_cluster_kernel<T, OPTIONS, CARRY>(const cps::BatchItem*, const int*, int, int*,  \
                                                                     cps::BatchResult*);                            \
  PRE template __global__ void cps_group_kernel<T, OPTIONS, CARRY>(const cps::BatchItem*, const int*, int, int*,    \
                                                                   cps::BatchResult*, cps::GridBarrier*, double*,   \
                                                                   int*, int);                                      \
  PRE template __global__ void cps_wave_kernel<T, OPTIONS, CARRY>(const cps::BatchItem*, const int*, const int*,    \
                                                                  int, cps::BatchResult*, cps::GridBarrier*, double*);
#define CPS_BATCH_KERNELS(PRE, T)                                                                                   \
  CPS_BATCH_KERNELS_OF(PRE, T, false, cps::kFew)                                                                    \
  CPS_BATCH_KERNELS_OF(PRE, T, false, cps::kMany)                                                                   \
  CPS_BATCH_KERNELS_OF(PRE, T, false, cps::kForms)
#define CPS_BATCH_OPTION_KERNELS(PRE, T) CPS_BATCH_KERNELS_OF(PRE, T, true, cps::kAll)
