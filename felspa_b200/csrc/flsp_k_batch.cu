// flsp_k_batch.cu — batched problems: many independent 2D level-set
// problems (their own meshes, degrees 1..3, velocities and clocks) advance
// in ONE launch per RK stage (and one per reinit pseudo-step and limiter pass)
// per degree.  A block serves a work item (problem, tile) of one degree with
// the same per-tile bodies as the single-problem kernels (adv_tab_tile,
// hjs_tile, weno_tile); each degree has its own instantiation, so its registers, shared memory and
// occupancy are its own, not those of the most demanding degree in the batch.
#include <string>
#include <type_traits>

#include "flsp_advtab.cuh"
#include "flsp_clock.cuh"
#include "flsp_hjs.cuh"
#include "flsp_launch.h"
#include "flsp_tables.h"
#include "flsp_weno.cuh"

namespace flsp {

int upload_tables_batch() {
  cudaError_t e = upload_tables_here();
  if (e != cudaSuccess) return set_error(FLSP_ERR_CUDA, std::string("tables: ") + cudaGetErrorString(e));
  return FLSP_OK;
}

namespace {

// an item's mesh, copied from the problem's descriptor by the whole block
// (every thread reads it, like a plain launch's kernel parameters)
__device__ __forceinline__ void copy_mesh(MeshArgs* dst, const MeshArgs& src) {
  static_assert(sizeof(MeshArgs) % 4 == 0, "copied in words");
  for (int i = threadIdx.x; i < (int)(sizeof(MeshArgs) / 4); i += blockDim.x)
    reinterpret_cast<int*>(dst)[i] = reinterpret_cast<const int*>(&src)[i];
}

// one block per (problem, tile): the stage of the problem's own velocity table
template <typename T, int P>
__global__ void __launch_bounds__(HjsTile<2>::N * (P + 2), advtab_min_blocks<2, P, T>())
    batch_adv_kernel(const BatchProb* __restrict__ probs, const int2* __restrict__ items, int ix, int in_n, int iout,
                     int step, int stage, int combine) {
  __shared__ AdvTabArgs<T> a;
  const int2 w = items[blockIdx.x];
  const BatchProb& pr = probs[w.x];
  copy_mesh(&a.m, pr.m_adv);
  if (threadIdx.x == 0) {
    a.tab = reinterpret_cast<const T*>(pr.tab);
    a.phi_s = reinterpret_cast<const T*>(pr.buf[ix]);
    a.phi_n = reinterpret_cast<const T*>(pr.buf[in_n]);
    a.out = reinterpret_cast<T*>(pr.buf[iout]);
    a.step = pr.steps + step;
    a.stage = stage;
    a.combine = combine;
    a.err = pr.err;
  }
  __syncthreads();
  adv_tab_tile<2, P, false, T>(a, w.y);
}

template <typename T, int P>
__global__ void __launch_bounds__(HjsTile<2>::N * (P + 2), hjs_min_blocks<2, P, T>())
    batch_hj_kernel(const BatchProb* __restrict__ probs, const int2* __restrict__ items, int isrc, int idst,
                    int mode, int rk, double cfl_max, int k) {
  __shared__ HJArgs<T> a;
  const int2 w = items[blockIdx.x];
  const BatchProb& pr = probs[w.x];
  copy_mesh(&a.m, pr.m_hj);
  if (threadIdx.x == 0) {
    a.phi = reinterpret_cast<const T*>(pr.buf[isrc]);
    a.out = idst >= 0 ? reinterpret_cast<T*>(pr.buf[idst]) : nullptr;
    a.clk = pr.clk;
    a.mode = mode;
    a.rk = rk;
    a.step.cfl_max = cfl_max;
    a.step.scale = pr.adv_scale;
    a.step.shift = 0.0;
    a.step.k = k;
    a.rdiff = nullptr;
    a.stab = reinterpret_cast<T*>(pr.stab);
    a.err = pr.err;
  }
  __syncthreads();
  hjs_tile<2, P, T>(a, w.y);
}

// two blocks per (problem, tile)
template <typename T, int P>
__global__ void __launch_bounds__(WenoBlock::N)
    batch_weno_kernel(const BatchProb* __restrict__ probs, const int2* __restrict__ items, int iin, int iout) {
  __shared__ WenoArgs<T> a;
  const int2 w = items[blockIdx.x / 2];
  const BatchProb& pr = probs[w.x];
  copy_mesh(&a.m, pr.m_weno);
  if (threadIdx.x == 0) {
    a.in = reinterpret_cast<const T*>(pr.buf[iin]);
    a.out = reinterpret_cast<T*>(pr.buf[iout]);
    a.count = nullptr;
    a.err = pr.err;
  }
  __syncthreads();
  weno_tile<P, false, T>(a, w.y, (int)blockIdx.x % 2);
}

// clocks
__global__ void batch_clock_kernel(const BatchProb* __restrict__ probs, int n, int what) {
  chain_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const BatchProb& pr = probs[i];
  if (what == kBatchAdvHorizon) adv_clock_horizon_body(pr.clk, __longlong_as_double(0x7ff0000000000000LL));
  else hj_clock_reset_body(pr.clk);
}
// a warp per problem
__global__ void batch_clock_steps_kernel(const BatchProb* __restrict__ probs, int n_steps, int commit) {
  chain_wait();
  const BatchProb& pr = probs[blockIdx.x];
  adv_clock_steps_body(pr.clk, pr.ca, pr.steps, n_steps, commit != 0);
}

}  // namespace

int launch_batch_clock(cudaStream_t s, const BatchProb* probs, int n, int what) {
  return launch_chained("batch_clock_kernel", batch_clock_kernel, (unsigned)(n + 127) / 128, 128, 0, s, probs, n, what);
}

int launch_batch_clock_steps(cudaStream_t s, const BatchProb* probs, int n, int n_steps, bool commit) {
  return launch_chained("batch_clock_steps_kernel", batch_clock_steps_kernel, (unsigned)n, 32, 0, s, probs, n_steps,
                        commit ? 1 : 0);
}

// f(integral_constant<int, p>) for the degree p in 1..3
template <typename F>
int with_degree(int p, F&& f) {
  switch (p) {
    case 1: return f(std::integral_constant<int, 1>());
    case 2: return f(std::integral_constant<int, 2>());
    case 3: return f(std::integral_constant<int, 3>());
  }
  return set_error(FLSP_ERR_UNSUPPORTED, "batched problems: degree 1..3");
}

int batch_prepare(int kind, int prec, int p, int n_items, size_t* smem, int* threads, int* grid) {
  return with_degree(p, [&](auto PC) -> int {
    constexpr int P = decltype(PC)::value;
    cudaError_t e = cudaSuccess;
    auto go = [&](auto tz) {
      using T = decltype(tz);
      auto attr = [&](auto kern) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
      };
      *threads = HjsTile<2>::N * (P + 2);
      *grid = n_items;   // a block per item
      if (kind == kBatchKindAdv) {
        *smem = AdvTabPlan<2, P, false, T>::BYTES;
        attr(batch_adv_kernel<T, P>);
      } else if (kind == kBatchKindHJ) {
        *smem = HjsPlan<2, P, T>::BYTES;
        attr(batch_hj_kernel<T, P>);
      } else {
        *smem = WenoPlan<P, false, T>::BYTES;
        *threads = WenoBlock::N;
        *grid = 2 * n_items;
        attr(batch_weno_kernel<T, P>);
      }
    };
    if (prec == FLSP_FP64) go((double)0);
    else go((float)0);
    if (e != cudaSuccess) return set_error(FLSP_ERR_CUDA, std::string("batch attr: ") + cudaGetErrorString(e));
    return FLSP_OK;
  });
}

int launch_batch_adv(cudaStream_t s, int prec, int p, const BatchProb* probs, const int2* items,
                     int grid, int threads, size_t smem, int ix, int in_n, int iout, int step, int stage, int combine) {
  return with_degree(p, [&](auto PC) -> int {
    constexpr int P = decltype(PC)::value;
    return launch_chained("batch_adv_kernel", prec == FLSP_FP64 ? batch_adv_kernel<double, P> : batch_adv_kernel<float, P>,
                          (unsigned)grid, threads, smem, s, probs, items, ix, in_n, iout, step, stage, combine);
  });
}

int launch_batch_hj(cudaStream_t s, int prec, int p, const BatchProb* probs, const int2* items,
                    int grid, int threads, size_t smem, int isrc, int idst, int mode, int rk, double cfl_max, int k) {
  return with_degree(p, [&](auto PC) -> int {
    constexpr int P = decltype(PC)::value;
    return launch_chained("batch_hj_kernel", prec == FLSP_FP64 ? batch_hj_kernel<double, P> : batch_hj_kernel<float, P>,
                          (unsigned)grid, threads, smem, s, probs, items, isrc, idst, mode, rk, cfl_max, k);
  });
}

int launch_batch_weno(cudaStream_t s, int prec, int p, const BatchProb* probs, const int2* items,
                      int grid, int threads, size_t smem, int iin, int iout) {
  return with_degree(p, [&](auto PC) -> int {
    constexpr int P = decltype(PC)::value;
    return launch_chained("batch_weno_kernel",
                          prec == FLSP_FP64 ? batch_weno_kernel<double, P> : batch_weno_kernel<float, P>, (unsigned)grid,
                          threads, smem, s, probs, items, iin, iout);
  });
}

}  // namespace flsp
