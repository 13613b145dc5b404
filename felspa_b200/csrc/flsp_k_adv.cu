// flsp_k_adv.cu — advection stage kernels (instantiations + launchers).
#include <algorithm>
#include <cstring>

#include "flsp_advect.cuh"
#include "flsp_advtab.cuh"
#include "flsp_launch.h"
#include "flsp_tables.h"

namespace flsp {

int upload_tables_adv() {
  cudaError_t e = upload_tables_here();
  if (e != cudaSuccess) return set_error(FLSP_ERR_CUDA, std::string("tables: ") + cudaGetErrorString(e));
  return FLSP_OK;
}

static int sep_unit(int what, const Ctx& c, const VelDev* v, const int* tile, size_t* bytes,
                    const void* in = nullptr, const void* phin = nullptr, void* out = nullptr,
                    const AdvStep* step = nullptr, int stage = 0, int combine = 0, double ct = 0.0) {
  if (c.dim == 2) return sep2_call(what, c, v, tile, bytes, in, phin, out, step, stage, combine, ct);
  return sep3_call(what, c, v, tile, bytes, in, phin, out, step, stage, combine, ct);
}

// the table kernel's fixed tile
static void tab_tile(const Ctx& c, int* tile) {
  tile[0] = c.dim == 2 ? HjsTile<2>::X : HjsTile<3>::X;
  tile[1] = c.dim == 2 ? HjsTile<2>::Y : HjsTile<3>::Y;
  tile[2] = c.dim == 2 ? HjsTile<2>::Z : HjsTile<3>::Z;
}

int adv_default_tile(const Ctx& c, const VelDev& v, int* tile) {
  if (use_sep_kernel(v)) {
    // the tiles that measured fastest, or within 1.5 % of it (us a stage):
    // 2D FP32 16x8 (1200x1193 Q2: 54.0; 32x8 58.1, 8x8 60.8), FP64 8x8
    // (1200x1193 Q3: 341, 32x8 422; 233x190 Q3: 14.7, 32x8 22.8: few tiles);
    // 3D Q2 8x8x4 (128^3 FP32: 290; 8x4x4 314, 4x4x4 328; 96^3 FP64: 313;
    // 329 with 4x4x4, which takes over when the larger tiles are fewer than
    // the SMs: 24^3 12.2 against 14.4), otherwise FP32 8x4x4 (112^3 P2: 110;
    // 8x8x4 139) and FP64 4x4x4 (128^3 Q1: 254; 8x8x4 329), P1 8x4x4 (191; 207)
    const bool f32 = c.prec == FLSP_FP32, q = c.basis == FLSP_BASIS_Q;
    static const int t2[2][3] = {{8, 8, 1}, {16, 8, 1}};
    static const int t3[3][3] = {{4, 4, 4}, {8, 4, 4}, {8, 8, 4}};
    int k = f32 ? 1 : 0;
    if (c.dim == 3) {
      MeshArgs m = c.m;
      set_tile(m, 3, t3[2]);
      if (q && c.p == 2 && (f32 || nblocks(m) >= 148)) k = 2;
      else if (!q && c.p == 1) k = 1;
    }
    const int* t = c.dim == 2 ? t2[k] : t3[k];
    for (int d = 0; d < 3; ++d) tile[d] = t[d];
    return FLSP_OK;
  }
  if (v.tab) {
    tab_tile(c, tile);
    return FLSP_OK;
  }
  static const int c2[][3] = {{32, 8, 1}, {16, 16, 1}, {16, 8, 1}, {8, 8, 1}};
  static const int c3[][3] = {{8, 8, 4}, {8, 4, 4}, {4, 4, 4}, {4, 4, 2}};
  return dispatch(c, [&](auto D, auto PP, auto tz) -> int {
    constexpr int DIM = decltype(D)::value, P = decltype(PP)::value;
    using T = decltype(tz);
    const int(*cq)[3] = DIM == 2 ? c2 : c3;
    int i = 0;
    for (; i < 3; ++i)
      if (adv_smem_bytes<DIM, P, T>(cq[i], std::max(v.n_terms, 1)) <= 200 * 1024) break;
    tile[0] = cq[i][0];
    tile[1] = cq[i][1];
    tile[2] = cq[i][2];
    return FLSP_OK;
  });
}

int adv_tile_candidates(const Ctx& c, const VelDev& v, int (*out)[3], int* n) {
  if (!use_sep_kernel(v) && v.tab) {
    tab_tile(c, out[0]);
    *n = 1;
    return FLSP_OK;
  }
  static const int c2[][3] = {{32, 8, 1}, {16, 16, 1}, {16, 8, 1}, {8, 8, 1}};
  static const int c3s[][3] = {{8, 8, 4}, {8, 4, 4}, {4, 4, 4}};
  static const int c3q[][3] = {{8, 8, 4}, {8, 4, 4}, {4, 4, 4}, {4, 4, 2}};
  const int(*cand)[3] = c.dim == 2 ? c2 : (use_sep_kernel(v) ? c3s : c3q);
  *n = c.dim == 2 ? 4 : (use_sep_kernel(v) ? 3 : 4);
  for (int i = 0; i < *n; ++i)
    for (int d = 0; d < 3; ++d) out[i][d] = cand[i][d];
  return FLSP_OK;
}

int adv_prepare(const Ctx& c, const VelDev& v, const int* tile) {
  if (use_sep_kernel(v)) return sep_unit(1, c, &v, tile, nullptr);
  return dispatch(c, [&](auto D, auto PP, auto tz) -> int {
    constexpr int DIM = decltype(D)::value, P = decltype(PP)::value;
    using T = decltype(tz);
    if (v.tab) {
      int t[3];
      tab_tile(c, t);
      if (t[0] != tile[0] || t[1] != tile[1] || (DIM > 2 && t[2] != tile[2]))
        return set_error(FLSP_ERR_BAD_ARG, "the velocity-table stage kernel has a fixed tile");
      cudaError_t e = cudaSuccess;
      auto attr = [&](auto kern, size_t smem) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
      };
      if (c.basis == FLSP_BASIS_Q) attr(adv_tab_kernel<DIM, P, false, T>, AdvTabPlan<DIM, P, false, T>::BYTES);
      else attr(adv_tab_kernel<DIM, P, true, T>, AdvTabPlan<DIM, P, true, T>::BYTES);
      if (e != cudaSuccess) return set_error(FLSP_ERR_CUDA, std::string("adv attr: ") + cudaGetErrorString(e));
      return FLSP_OK;
    }
    const size_t smem = adv_smem_bytes<DIM, P, T>(tile, std::max(v.n_terms, 1));
    if (smem > 227 * 1024) return set_error(FLSP_ERR_BAD_ARG, "advection tile too large for shared memory");
    auto kern = adv_stage_kernel<DIM, P, T>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e != cudaSuccess) return set_error(FLSP_ERR_CUDA, std::string("adv attr: ") + cudaGetErrorString(e));
    return FLSP_OK;
  });
}

int launch_adv_stage(const Ctx& c, const VelDev& v, const void* in, const void* phin, void* out,
                     const AdvStep* step, int stage, int combine, double ct_explicit,
                     const int* tile) {
  if (use_sep_kernel(v)) {
    int t[3];
    if (tile) { t[0] = tile[0]; t[1] = tile[1]; t[2] = tile[2]; }
    else {
      const int st = adv_default_tile(c, v, t);
      if (st) return st;
    }
    return sep_unit(2, c, &v, t, nullptr, in, phin, out, step, stage, combine, ct_explicit);
  }
  return dispatch(c, [&](auto D, auto PP, auto tz) -> int {
    constexpr int DIM = decltype(D)::value, P = decltype(PP)::value;
    using T = decltype(tz);
    if (v.tab) {
      AdvTabArgs<T> a;
      std::memset(&a, 0, sizeof(a));
      a.m = c.m;
      int t[3];
      tab_tile(c, t);
      set_tile(a.m, DIM, t);
      a.tab = reinterpret_cast<const T*>(v.tab);
      a.phi_s = reinterpret_cast<const T*>(in);
      a.phi_n = reinterpret_cast<const T*>(phin);
      a.out = reinterpret_cast<T*>(out);
      a.step = step;
      a.stage = stage;
      a.combine = combine;
      a.ct_explicit = ct_explicit;
      a.err = v.err;
      const int threads = HjsTile<DIM>::N * (P + 2);
      const bool q = c.basis == FLSP_BASIS_Q;
      return launch_chained("adv_tab_kernel", q ? adv_tab_kernel<DIM, P, false, T> : adv_tab_kernel<DIM, P, true, T>,
                            (unsigned)nblocks(a.m), threads,
                            q ? AdvTabPlan<DIM, P, false, T>::BYTES : AdvTabPlan<DIM, P, true, T>::BYTES, c.stream, a);
    }
    AdvArgs<T> a;
    std::memset(&a, 0, sizeof(a));
    a.m = c.m;
    int t[3];
    if (tile) { t[0] = tile[0]; t[1] = tile[1]; t[2] = tile[2]; }
    else adv_default_tile(c, v, t);
    set_tile(a.m, DIM, t);
    a.v.vtab = reinterpret_cast<const T*>(v.vtab);
    a.v.n_terms = v.n_terms;
    a.v.nmax = v.nmax;
    a.v.npt = v.npt;
    for (int k = 0; k < v.n_terms; ++k) a.v.comp[k] = v.comp[k];
    term_ranges(a.v.comp, v.n_terms, a.v.cstart);
    a.phi_s = reinterpret_cast<const T*>(in);
    a.phi_n = reinterpret_cast<const T*>(phin);
    a.out = reinterpret_cast<T*>(out);
    a.step = step;
    a.stage = stage;
    a.combine = combine;
    a.ct_explicit = ct_explicit;
    const size_t smem = adv_smem_bytes<DIM, P, T>(a.m.tile, std::max(v.n_terms, 1));
    adv_stage_kernel<DIM, P, T><<<(unsigned)nblocks(a.m), t[0] * t[1] * t[2], smem, c.stream>>>(a);
    return launch_status("adv_stage_kernel");
  });
}

}  // namespace flsp
