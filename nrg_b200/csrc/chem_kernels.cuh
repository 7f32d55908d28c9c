// Kernel templates of the chemistry step (included by the per-variant
// translation units chem_k_*.cu, which instantiate them).
//
//   k_chem_pass   -- one thread per cell in passes (chem_pass.cuh): analytic
//                    Jacobian.
//   k_chem_plain  -- one thread per cell, grid covers all cells.
//   k_chem_queue  -- persistent grid; every lane pulls cells from a device
//                    work queue and is refilled as soon as its cell reaches
//                    t = dt, so lanes never wait for the slowest cell of a
//                    warp.  Block size, blocks per SM and the number of cells
//                    a lane reserves per queue fetch are autotuned on the host.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "chem_bdf.cuh"
#include "chem_kernels.hpp"
#include "chem_pass.cuh"
#include "chem_warp.cuh"

namespace nrg {

namespace cg = cooperative_groups;

// Counter slots (unsigned long long): cells integrated, steps, RHS
// evaluations, Jacobians, linear solves, cells not ok.
enum { kCntCells = 0, kCntSteps, kCntRhs, kCntJac, kCntSolve, kCntBad, kCntSlots };

__device__ __forceinline__ void block_flush_counters(unsigned long long* counters,
                                                     unsigned long long v[kCntSlots]) {
  __shared__ unsigned long long s_cnt[kCntSlots];
  if (threadIdx.x < kCntSlots) s_cnt[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kCntSlots; ++i) {
    unsigned long long x = v[i];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0 && x) atomicAdd(&s_cnt[i], x);
  }
  __syncthreads();
  if (threadIdx.x < kCntSlots && s_cnt[threadIdx.x]) atomicAdd(&counters[threadIdx.x], s_cnt[threadIdx.x]);
}

template <int N, int R, int JAC, typename LUT, int BS, int NF, int SPEC>
__global__ void __launch_bounds__(BS, 1) k_chem_plain(StepArgs a, unsigned long long* counters) {
  extern __shared__ __align__(16) char smem[];
  const long li = (long)blockIdx.x * BS + threadIdx.x;
  const long nl = a.cell_list ? (long)(a.n_list_dev ? *a.n_list_dev : a.n_list) : a.n;
  const long cid = (a.cell_list && li < nl) ? (long)a.cell_list[li] : li;
  unsigned long long v[kCntSlots] = {0, 0, 0, 0, 0, 0};
  CellState<N, R, LUT, BS, NF, SPEC> c;
  c.bind(smem, threadIdx.x);
  if (li < nl) {
    if (cell_begin<N, R, JAC>(c, a, cid)) {
      int st;
      while ((st = cell_advance<N, R, JAC, LUT>(c, a.mxstep)) == 0) {
      }
      cell_finish<N, JAC>(c, a, cid, st);
      v[kCntCells] = 1;
      v[kCntSteps] = c.nstep;
      v[kCntRhs] = c.nfe;
      v[kCntJac] = c.nje;
      v[kCntSolve] = c.nsolve;
      v[kCntBad] = st != kCellOk;
    }
  }
  if (counters) block_flush_counters(counters, v);
}

template <int N, int R, int JAC, typename LUT, int BS, int NF, int SPEC>
__global__ void __launch_bounds__(BS, 1) k_chem_queue(StepArgs a, int* queue, int chunk,
                                                       unsigned long long* counters) {
  extern __shared__ __align__(16) char smem[];
  unsigned long long v[kCntSlots] = {0, 0, 0, 0, 0, 0};
  CellState<N, R, LUT, BS, NF, SPEC> c;
  c.bind(smem, threadIdx.x);
  long cur = 0, left = 0, cid = 0;  // logical index, cells still reserved, cell id
  const long nl = a.cell_list ? (long)(a.n_list_dev ? *a.n_list_dev : a.n_list) : a.n;
  bool have = false;
  for (;;) {
    if (!have) {
      if (left == 0) {
        // warp-aggregated reservation of `chunk` cells per requesting lane
        cg::coalesced_group g = cg::coalesced_threads();
        long base = 0;
        if (g.thread_rank() == 0) base = (long)atomicAdd(queue, (int)(g.size() * chunk));
        base = g.shfl(base, 0);
        cur = base + (long)g.thread_rank() * chunk;
        left = chunk;
      } else {
        ++cur;
      }
      --left;
      if (cur >= nl) break;
      cid = a.cell_list ? (long)a.cell_list[cur] : cur;
      have = cell_begin<N, R, JAC>(c, a, cid);
      if (!have) continue;
    }
    const int st = cell_advance<N, R, JAC, LUT>(c, a.mxstep);
    if (st) {
      cell_finish<N, JAC>(c, a, cid, st);
      v[kCntCells] += 1;
      v[kCntSteps] += c.nstep;
      v[kCntRhs] += c.nfe;
      v[kCntJac] += c.nje;
      v[kCntSolve] += c.nsolve;
      v[kCntBad] += st != kCellOk;
      have = false;
    }
  }
  if (counters) block_flush_counters(counters, v);
}

// Blocks of a work-queue launch: no more than have a cell to start with, and
// few enough that the reservations past the end (up to 64 cells from each of 64
// lanes a block) leave the int queue head far from overflow.
static int queue_blocks(int grid, const StepArgs& a, int cells_per_block) {
  const long nl = a.cell_list ? (long)a.n_list : a.n;
  return (int)std::max<long>(1, std::min<long>({(long)grid, (nl + cells_per_block - 1) / cells_per_block, 65536L}));
}

template <int N, int R, int JAC, typename LUT, int BS, int NF, int SPEC>
static cudaError_t launch_bs(const StepArgs& a, const LaunchCfg& cfg, int* queue,
                             unsigned long long* counters, cudaStream_t s) {
  const size_t smem = (size_t)BS * SmemStore<N, R, LUT, BS>::kBytesPerThread;
  cudaError_t e;
  if (cfg.kernel == kKernelThreadQueue) {
    e = cudaFuncSetAttribute(k_chem_queue<N, R, JAC, LUT, BS, NF, SPEC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    if (e != cudaSuccess) return e;
    const int grid = queue_blocks(cfg.grid > 0 ? cfg.grid : 148, a, BS);
    k_chem_queue<N, R, JAC, LUT, BS, NF, SPEC><<<grid, BS, smem, s>>>(a, queue, cfg.chunk, counters);
  } else {
    e = cudaFuncSetAttribute(k_chem_plain<N, R, JAC, LUT, BS, NF, SPEC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    if (e != cudaSuccess) return e;
    const long nl = a.cell_list ? (long)a.n_list : a.n;
    const long grid = (nl + BS - 1) / BS;
    if (grid > 0) k_chem_plain<N, R, JAC, LUT, BS, NF, SPEC><<<(unsigned)grid, BS, smem, s>>>(a, counters);
  }
  return cudaGetLastError();
}


// One cell per thread, integrated in passes (chem_pass.cuh).  LOCK: the warps of
// the block go through the passes together, so that the loop's 50 to 80 KB of
// code are fetched once for all of them.  QUEUE: the warps pull groups of 32
// cells from the work queue; else the grid covers the cells.
// TM: the cells' rate constants in tensor memory (lockstep blocks of 128 threads:
// warp w has lanes 32 w).
template <int N, int R, typename LUT, int BS, int NF, int SPEC, bool LOCK, bool QUEUE, bool TM>
__global__ void __launch_bounds__(BS, BS > 128 ? 1 : 256 / BS) k_chem_pass(StepArgs a, int* queue, int chunk,
                                                            unsigned long long* counters) {
  static_assert(!(LOCK && QUEUE), "the work queue serves warps on their own");
  static_assert(!TM || (LOCK && BS == 128), "one warp per quarter of the tensor memory's lanes");
  extern __shared__ __align__(16) char smem[];
  const long nl = a.cell_list ? (long)(a.n_list_dev ? *a.n_list_dev : a.n_list) : a.n;
  if (!QUEUE && (long)blockIdx.x * BS >= nl) return;
  unsigned long long v[kCntSlots] = {0, 0, 0, 0, 0, 0};
  using Store = PassStore<N, RateSlots<R, SPEC>::value, LUT, SPEC == 0, TM>;
  Store st;
  st.bind(smem, threadIdx.x);
  __shared__ uint32_t tslot;
  if constexpr (TM) {
    if (threadIdx.x < 32) tc::tmem_alloc(tc::smem_u32(&tslot), Store::kTmCols);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    st.tm = tslot + ((threadIdx.x & ~31u) << 16);
  }
  const int lane = threadIdx.x & 31;
  long base = ((long)blockIdx.x * BS + threadIdx.x) & ~31L;
  int left = 0;
  for (;;) {
    if (QUEUE) {
      if (left == 0) {
        int b = 0;
        if (lane == 0) b = atomicAdd(queue, chunk);
        base = 32L * __shfl_sync(0xffffffffu, b, 0);
        left = chunk;
      } else {
        base += 32;
      }
      --left;
      if (base >= nl) break;
    }
    const long li = base + lane;
    const bool have = li < nl;
    const long cid = have ? (a.cell_list ? (long)a.cell_list[li] : li) : 0;
    PassResult<N, NF> res;
#pragma unroll
    for (int i = 0; i < N; ++i) res.y[i] = 0.0;
    res.tout = a.dt;
    bool live = false;
    if (have) {
      live = pass_begin<N, R, NF>(st, a, cid, res.y);
      if (a.dt_cells) res.tout = a.dt_cells[cid];
    }
    if constexpr (TM) pass_rates_to_tm<N>(st);
    else __syncwarp();  // the set-up scratch covers other lanes' factors when these are floats
    const int status = pass_integrate<N, R, NF, SPEC, LOCK>(st, a, live, res.tout, res.y, v);
    if (live) {
      cell_finish<N, kJacAnalytic>(res, a, cid, status);
      v[kCntCells] += 1;
      v[kCntBad] += status != kCellOk;
    }
    if (!QUEUE) break;
    __syncwarp();  // the factors of this group, before the next group's set-up scratch
  }
  if constexpr (TM) {
    __syncthreads();
    if (threadIdx.x < 32) tc::tmem_dealloc(tslot, Store::kTmCols);
  }
  if (counters) block_flush_counters(counters, v);
}

template <int N, int R, typename LUT, int BS, int NF, int SPEC, bool LOCK, bool QUEUE, bool TM = false>
static cudaError_t launch_pass_bs(const StepArgs& a, long grid, int* queue, int chunk, unsigned long long* counters,
                                  cudaStream_t s) {
  const auto kern = k_chem_pass<N, R, LUT, BS, NF, SPEC, LOCK, QUEUE, TM>;
  const int smem = BS * PassStore<N, RateSlots<R, SPEC>::value, LUT, SPEC == 0, TM>::kBytesPerThread;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  // larger mechanisms spill part of the Nordsieck array: what shared memory the
  // blocks of an SM leave goes to the L1 cache (KONNOV flame of 196,608 cells in
  // lockstep 26.9 -> 22.8 ms; 9,472 random cells on their own 5.71 -> 4.84 ms).
  // Above 10 species (1 KB and more a thread) two blocks, though a third of
  // ACETYLENE's fits (flame of 18,944 cells 3.31 -> 2.59 ms, random cells 9.46 ->
  // 8.12 ms).
  const int fit = std::max(1, 232448 / (smem + 1024));
  const int used = (smem + 1024) * (N > 10 ? std::min(fit, 2) : fit);
  const int carveout = N > 8 ? (100 * used + 233471) / 233472 : 100;
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, carveout);
  if (e != cudaSuccess) return e;
  if (grid > 0) kern<<<(unsigned)grid, BS, smem, s>>>(a, queue, chunk, counters);
  return cudaGetLastError();
}

// Up to 8 integrated species with generated code: blocks of 128 threads in
// lockstep from kLockstepCells cells on, the places of two such blocks on each
// of 148 SMs (a list counts with its capacity, which the host knows); below,
// 64-thread blocks whose warps run on their own: the cells then spread over more
// SMs and nothing waits for another warp.  KEROMNES (880 B a cell, two blocks
// fit): 37,888 random cells 1.90 ms on their own and 1.48 ms in lockstep, 196,608
// 9.18 and 6.47 ms, a flame of 196,608 2.36 and 2.10 ms; 4,096 random cells 1.15
// and 1.29 ms.  ZHANG (976 B, one block fits): 37,888 random cells 2.95 and 2.48
// ms, a flame of 196,608 3.41 and 3.22 ms.
//
// Table walks are bound by the latency of their dependent reads, which more
// warps of their own hide better: 64-thread blocks at any size (KEROMNES, three
// fit: 196,608 random cells 26.5 ms against 29.9 ms in lockstep, a flame 8.0
// against 10.2; 32-thread blocks above 8 species).
constexpr long kLockstepCells = 148L * 2 * 128;

template <int N, int R, typename LUT, int NF, int SPEC>
static cudaError_t launch_pass(const StepArgs& a, const LaunchCfg& cfg, int* queue, unsigned long long* counters,
                               cudaStream_t s) {
  if constexpr (N <= 8) {
    if (cfg.kernel == kKernelThreadQueue)
      return launch_pass_bs<N, R, LUT, 64, NF, SPEC, false, true>(a, queue_blocks(cfg.grid > 0 ? cfg.grid : 148, a, 64),
                                                                  queue, cfg.chunk, counters, s);
  }
  const long nl = a.cell_list ? (long)a.n_list : a.n;
  if constexpr (N <= 8) {
    if constexpr (SPEC != 0) {
      if (nl >= kLockstepCells)
        return launch_pass_bs<N, R, LUT, 128, NF, SPEC, true, false>(a, (nl + 127) / 128, queue, 0, counters, s);
    }
    return launch_pass_bs<N, R, LUT, 64, NF, SPEC, false, false>(a, (nl + 63) / 64, queue, 0, counters, s);
  } else {
    if constexpr (SPEC != 0) {
      // W: the warps of a SM's shared memory, at most two above 10 species, whose
      // spilled state the L1 cache then holds.  More fit in blocks of 128 threads
      // with the rate constants in tensor memory for KONNOV (2 -> 4) and TEREZA (5 ->
      // 8): these from one more cell than the W warps take at once (KONNOV, 9,472
      // random cells 4.88 ms on their own and 5.37 ms, 14,208 7.86 and 5.42 ms;
      // TEREZA, 23,680 cells 2.83 and 2.95 ms, 28,416 4.15 and 3.12 ms).  Otherwise
      // (ACETYLENE) W warps in lockstep from there on: 18,944 random cells 7.76 ms on
      // their own and 6.42 ms, a flame of them 2.53 and 2.60 ms, of 196,608 18.4 and
      // 15.9 ms.  Its three warps that fit took 14.6 ms there, but 66.3 against 57.5
      // ms for random cells, and 3.70 against 2.57 ms for a flame of 4,096 cells,
      // which a large field with few hot cells comes to.
      constexpr int RS = RateSlots<R, SPEC>::value;
      constexpr int kWarpBytes = 32 * PassStore<N, RS, LUT, false>::kBytesPerThread;
      constexpr int W = std::min(232448 / kWarpBytes, N > 10 ? 2 : 8);
      constexpr int kTmBytes = 128 * PassStore<N, RS, LUT, false, true>::kBytesPerThread;
      constexpr int kTmWarps = kTmBytes > 232448 ? 0 : kTmBytes > 115000 ? 4 : 8;
      if constexpr (kTmWarps > W) {
        if (nl > 148L * 32 * W)
          return launch_pass_bs<N, R, LUT, 128, NF, SPEC, true, false, true>(a, (nl + 127) / 128, queue, 0, counters, s);
      } else if (nl > 148L * 32 * W) {
        return launch_pass_bs<N, R, LUT, 32 * W, NF, SPEC, true, false>(a, (nl + 32 * W - 1) / (32 * W), queue, 0,
                                                                        counters, s);
      }
    }
    return launch_pass_bs<N, R, LUT, 32, NF, SPEC, false, false>(a, (nl + 31) / 32, queue, 0, counters, s);
  }
}

__host__ __device__ constexpr size_t warp_tables_bytes() { return (sizeof(DevMech) + 15) / 16 * 16; }

// Warp-per-cell persistent kernel: every warp pulls `chunk` cells at a time
// from the work queue and integrates them one after the other.
template <int N, int R, int JAC, typename LUT, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 4 ? 4 : 1) k_chem_warp(StepArgs a, int* queue, int chunk,
                                                         unsigned long long* counters) {
  // dynamic shared memory: the mechanism tables, then one scratch per warp
  extern __shared__ __align__(16) char wsmem[];
  DevMech& sM = *reinterpret_cast<DevMech*>(wsmem);
  WarpSmem<N, R, LUT>* sm = reinterpret_cast<WarpSmem<N, R, LUT>*>(wsmem + warp_tables_bytes());
  {
    // lanes read per-reaction and per-species entries at different addresses,
    // which __constant__ memory would serialize: work from a shared copy
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(a.mech);
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(&sM);
    for (int i = threadIdx.x; i < (int)(sizeof(DevMech) / 8); i += WARPS * 32) dst[i] = src[i];
    __syncthreads();
  }
  unsigned long long v[kCntSlots] = {0, 0, 0, 0, 0, 0};
  WarpCell<N, R, LUT> c;
  c.M = &sM;
  c.lane = threadIdx.x & 31;
  c.sm = &sm[threadIdx.x >> 5];
  const long nl = a.cell_list ? (long)(a.n_list_dev ? *a.n_list_dev : a.n_list) : a.n;
  long cur = 0, left = 0;
  for (;;) {
    if (left == 0) {
      int base = 0;
      if (c.lane == 0) base = atomicAdd(queue, chunk);
      cur = __shfl_sync(kFullMask, base, 0);
      left = chunk;
    } else {
      ++cur;
    }
    --left;
    if (cur >= nl) break;
    const long cid = a.cell_list ? (long)a.cell_list[cur] : cur;
    if (!warp_cell_begin(c, a, cid)) continue;
    int st;
    while ((st = warp_cell_advance<N, R, JAC>(c, a.mxstep)) == 0) {
    }
    warp_cell_finish(c, a, cid, st);
    if (c.lane == 0) {
      v[kCntCells] += 1;
      v[kCntSteps] += c.nstep;
      v[kCntRhs] += c.nfe;
      v[kCntJac] += c.nje;
      v[kCntSolve] += c.nsolve;
      v[kCntBad] += st != kCellOk;
    }
  }
  if (counters) block_flush_counters(counters, v);
}

template <int N, int R, int JAC, typename LUT, int WARPS>
static cudaError_t launch_warp(const StepArgs& a, const LaunchCfg& cfg, int* queue,
                               unsigned long long* counters, cudaStream_t s) {
  const size_t smem = warp_tables_bytes() + WARPS * sizeof(WarpSmem<N, R, LUT>);
  cudaError_t e = cudaFuncSetAttribute(k_chem_warp<N, R, JAC, LUT, WARPS>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int grid = cfg.grid;
  if (grid <= 0) {
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_chem_warp<N, R, JAC, LUT, WARPS>, WARPS * 32, smem);
    grid = sms * (per_sm > 0 ? per_sm : 1);
  }
  grid = queue_blocks(grid, a, WARPS);
  k_chem_warp<N, R, JAC, LUT, WARPS><<<grid, WARPS * 32, smem, s>>>(a, queue, cfg.chunk, counters);
  return cudaGetLastError();
}

// The thread-per-cell kernels: in passes for the analytic Jacobian (these choose
// their blocks themselves; above 8 species part of the Nordsieck array spills
// to the L1 cache), routine by routine for the reference mode and for mechanisms
// of nine species that all react, which no generated code covers.
template <int NF, int NI, int R, int JAC, typename LUT, int SPEC>
static cudaError_t launch_thread(const StepArgs& a, const LaunchCfg& cfg, int* queue, unsigned long long* counters,
                                 cudaStream_t s) {
  if constexpr (integrates_in_passes(JAC, NI)) {
    return launch_pass<NI, R, LUT, NF, SPEC>(a, cfg, queue, counters, s);
  } else {
    switch (cfg.block) {
      case 32: return launch_bs<NI, R, JAC, LUT, 32, NF, SPEC>(a, cfg, queue, counters, s);
      case 64: return launch_bs<NI, R, JAC, LUT, 64, NF, SPEC>(a, cfg, queue, counters, s);
      default: return cudaErrorInvalidValue;
    }
  }
}

// Launches one (JAC, LUT) variant: cfg.kernel selects thread-per-cell (grid
// or work queue, 32- or 64-thread blocks) or warp-per-cell (128- or 256-thread
// blocks).  With 32-thread blocks every warp is its own block, so an SM slot
// is handed to a new block as soon as the warp's cells are done instead of
// waiting for the slowest warp of a larger block.  NF mechanism species, NI of
// them integrated by the thread-per-cell kernels (the translation unit's
// tables are numbered over those NI); the warp kernel integrates all NF from
// the full tables it copies to shared memory.  SPEC != 0: the thread kernels
// use that generated mechanism-specialised RHS and iteration matrix.
template <int NF, int NI, int R, int JAC, typename LUT, int SPEC>
static cudaError_t launch_variant(const StepArgs& a, const LaunchCfg& cfg, int* queue,
                                  unsigned long long* counters, cudaStream_t s) {
  if (cfg.kernel == kKernelWarpQueue) {
    switch (cfg.block) {
      case 128: return launch_warp<NF, R, JAC, LUT, 4>(a, cfg, queue, counters, s);
      case 256: return launch_warp<NF, R, JAC, LUT, 8>(a, cfg, queue, counters, s);
      default: return cudaErrorInvalidValue;
    }
  }
  return launch_thread<NF, NI, R, JAC, LUT, SPEC>(a, cfg, queue, counters, s);
}

// The thread-per-cell grid kernel only (the shape used for the mechanisms
// other than the default one, which get no queue / warp variants).
template <int NF, int NI, int R, int JAC, typename LUT, int SPEC = 0>
static cudaError_t launch_grid(const StepArgs& a, const LaunchCfg& cfg, int* queue, unsigned long long* counters,
                               cudaStream_t s) {
  if (cfg.kernel != kKernelThreadGrid) return cudaErrorNotSupported;
  return launch_thread<NF, NI, R, JAC, LUT, SPEC>(a, cfg, queue, counters, s);
}

}  // namespace nrg
