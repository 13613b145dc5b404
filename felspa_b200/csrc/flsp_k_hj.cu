// flsp_k_hj.cu — reinitialisation pseudo-step kernels (instantiations + launchers).
#include <algorithm>
#include <cstring>

#include "flsp_hj.cuh"
#include "flsp_hjp.cuh"
#include "flsp_hjs.cuh"
#include "flsp_ldg.cuh"
#include "flsp_launch.h"
#include "flsp_tables.h"

namespace flsp {

int upload_tables_hj() {
  cudaError_t e = upload_tables_here();
  if (e != cudaSuccess) return set_error(FLSP_ERR_CUDA, std::string("tables: ") + cudaGetErrorString(e));
  return FLSP_OK;
}

// tile of the reinitialisation launches: the kernels' block of cells; in the
// P basis several blocks together (the unit the narrow band lists: a sweep's
// frozen margin, and with it its result, depends on it)
int hj_default_tile(const Ctx& c, int* tile) {
  return dispatch(c, [&](auto D, auto PP, auto tz) -> int {
    constexpr int DIM = decltype(D)::value, P = decltype(PP)::value;
    using T = decltype(tz);
    tile[0] = HjsTile<DIM>::X;
    tile[1] = HjsTile<DIM>::Y;
    tile[2] = HjsTile<DIM>::Z;
    if (c.basis == FLSP_BASIS_Q) return FLSP_OK;
    if (DIM == 2) tile[0] = tile[1] = 16;
    else if (P == 1) tile[0] = tile[1] = 8;
    else if (sizeof(T) == 4) tile[0] = 8;
    return FLSP_OK;
  });
}

int hj_prepare(const Ctx& c, const int* tile) {
  return dispatch(c, [&](auto D, auto PP, auto tz) -> int {
    constexpr int DIM = decltype(D)::value, P = decltype(PP)::value;
    using T = decltype(tz);
    using TL = HjsTile<DIM>;
    const bool tq = c.basis == FLSP_BASIS_Q;
    if (tile[0] % TL::X || tile[1] % TL::Y || (DIM > 2 && tile[2] % TL::Z) ||
        (tq && (tile[0] != TL::X || tile[1] != TL::Y || (DIM > 2 && tile[2] != TL::Z))))
      return set_error(FLSP_ERR_BAD_ARG, "the reinit kernels have a fixed tile");
    constexpr size_t bytes[2] = {HjsPlan<DIM, P, T>::BYTES, HjpPlan<DIM, P, T>::BYTES};
    static_assert(bytes[0] <= 227 * 1024 && bytes[1] <= 227 * 1024, "reinit tile too large for shared memory");
    cudaError_t e = cudaSuccess;
    auto attr = [&](auto k, size_t smem) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    };
    if (tq) attr(hjs_kernel<DIM, P, T>, bytes[0]);
    else attr(hjp_kernel<DIM, P, T>, bytes[1]);
    attr(hj_gradient_kernel<DIM, P, T>, hjg_smem_bytes<DIM, P, T>());
    if (e != cudaSuccess) return set_error(FLSP_ERR_CUDA, std::string("hj attr: ") + cudaGetErrorString(e));
    return FLSP_OK;
  });
}

int hj_table_bytes(const Ctx& c, const int* tile, size_t* bytes) {
  return dispatch(c, [&](auto D, auto PP, auto tz) -> int {
    constexpr int DIM = decltype(D)::value, P = decltype(PP)::value;
    using T = decltype(tz);
    MeshArgs m = c.m;
    set_tile(m, DIM, tile);
    const long long nt = (long long)m.tile[0] * m.tile[1] * m.tile[2];
    *bytes = (size_t)nblocks(m) * hjs_ns<DIM, P>() * nt * sizeof(T);
    return FLSP_OK;
  });
}

int ldg_prepare(const Ctx& c) {
  return dispatch(c, [&](auto D, auto PP, auto tz) -> int {
    constexpr int DIM = decltype(D)::value, P = decltype(PP)::value;
    using T = decltype(tz);
    cudaError_t e = cudaSuccess;
    auto attr = [&](auto k, size_t smem) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    };
    if (c.basis == FLSP_BASIS_Q) attr(ldg_kernel<DIM, P, false, T>, LdgPlan<DIM, P, false, T>::BYTES);
    else attr(ldg_kernel<DIM, P, true, T>, LdgPlan<DIM, P, true, T>::BYTES);
    if (e != cudaSuccess) return set_error(FLSP_ERR_CUDA, std::string("ldg attr: ") + cudaGetErrorString(e));
    return FLSP_OK;
  });
}

int launch_ldg(const Ctx& c, const void* in, void* out, double nu) {
  return dispatch(c, [&](auto D, auto PP, auto tz) -> int {
    constexpr int DIM = decltype(D)::value, P = decltype(PP)::value;
    using T = decltype(tz);
    using TL = LdgTile<DIM>;
    LdgArgs<T> a;
    std::memset(&a, 0, sizeof(a));
    a.m = c.m;
    const int* t = DIM == 2 ? kLdgTile2 : kLdgTile3;
    static_assert(kLdgTile2[0] % LdgTile<2>::X == 0 && kLdgTile2[1] % LdgTile<2>::Y == 0 &&
                      kLdgTile3[0] % LdgTile<3>::X == 0 && kLdgTile3[1] % LdgTile<3>::Y == 0 &&
                      kLdgTile3[2] % LdgTile<3>::Z == 0,
                  "the band's unit is whole blocks");
    set_tile(a.m, DIM, t);
    apply_band(c, kNbLdg, a.m);
    a.listed = a.m.tiles ? c.nb_ldg_listed : nullptr;
    a.in = reinterpret_cast<const T*>(in);
    a.out = reinterpret_cast<T*>(out);
    a.nu = nu;
    a.err = c.err;
    const long long blocks = nblocks(a.m) * (t[0] / TL::X) * (t[1] / TL::Y) * (t[2] / TL::Z);
    const bool q = c.basis == FLSP_BASIS_Q;
    return launch_chained("ldg_kernel", q ? ldg_kernel<DIM, P, false, T> : ldg_kernel<DIM, P, true, T>, (unsigned)blocks,
                          TL::N * DIM, q ? LdgPlan<DIM, P, false, T>::BYTES : LdgPlan<DIM, P, true, T>::BYTES, c.stream,
                          a);
  });
}

int launch_hj(const Ctx& c, const void* phi, const void* phi0, void* out, DevClock* clk, int mode,
              int rk, const HjClockArgs* step, long long block, const int* tile, const void* rdiff) {
  return dispatch(c, [&](auto D, auto PP, auto tz) -> int {
    constexpr int DIM = decltype(D)::value, P = decltype(PP)::value;
    using T = decltype(tz);
    HJArgs<T> a;
    std::memset(&a, 0, sizeof(a));
    a.m = c.m;
    int t[3];
    if (tile) { t[0] = tile[0]; t[1] = tile[1]; t[2] = tile[2]; }
    else hj_default_tile(c, t);
    set_tile(a.m, DIM, t);
    a.phi = reinterpret_cast<const T*>(phi);
    a.out = reinterpret_cast<T*>(out);
    a.clk = clk;
    a.mode = mode;
    a.rk = rk;
    if (step) a.step = *step;
    a.block = block;
    a.rdiff = reinterpret_cast<const T*>(rdiff);
    if (mode == kHJGradients) {   // the export, every cell
      static const int tg[3] = {HjgTile<DIM>::X, HjgTile<DIM>::Y, HjgTile<DIM>::Z};
      set_tile(a.m, DIM, tg);
      a.grad = reinterpret_cast<double*>(out);
      hj_gradient_kernel<DIM, P, T>
          <<<(unsigned)nblocks(a.m), tg[0] * tg[1] * tg[2], hjg_smem_bytes<DIM, P, T>(), c.stream>>>(a);
      return launch_status("hj_gradient_kernel");
    }
    apply_band(c, kNbHJ, a.m);
    // the smooth-sign table is filled by the sweep's kHJCflOnly launch,
    // which evaluates phi0 as phi
    if (!c.hj_stab || !clk || (mode == kHJStep && !step))
      return set_error(FLSP_ERR_BAD_ARG, "reinit sign table or clock missing");
    if (mode == kHJCflOnly && phi != phi0)
      return set_error(FLSP_ERR_BAD_ARG, "the sign-table launch needs phi == phi0");
    using TL = HjsTile<DIM>;
    if (a.m.tile[0] % TL::X || a.m.tile[1] % TL::Y || a.m.tile[2] % TL::Z ||
        (c.basis == FLSP_BASIS_Q && (a.m.tile[0] != TL::X || a.m.tile[1] != TL::Y || a.m.tile[2] != TL::Z)))
      return set_error(FLSP_ERR_BAD_ARG, "the reinit kernels have a fixed tile");
    a.stab = reinterpret_cast<T*>(c.hj_stab);
    a.err = c.err;
    const int threads = TL::N * (P + 2);
    if (c.basis == FLSP_BASIS_Q) {
      return launch_chained("hjs_kernel", hjs_kernel<DIM, P, T>, (unsigned)nblocks(a.m), threads,
                            HjsPlan<DIM, P, T>::BYTES, c.stream, a);
    }
    const long long parts = (long long)(a.m.tile[0] / TL::X) * (a.m.tile[1] / TL::Y) * (a.m.tile[2] / TL::Z);
    return launch_chained("hjp_kernel", hjp_kernel<DIM, P, T>, (unsigned)(nblocks(a.m) * parts), threads,
                          HjpPlan<DIM, P, T>::BYTES, c.stream, a);
  });
}

}  // namespace flsp
