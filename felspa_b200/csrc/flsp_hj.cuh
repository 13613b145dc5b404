// flsp_hj.cuh — what the Hamilton-Jacobi reinitialisation kernels share, and
// the export of the LDG one-sided gradients.
//
// The pseudo-step kernels (hjs_kernel, flsp_hjs.cuh: tensor-product basis, the
// batched problems too; hjp_kernel, flsp_hjp.cuh: total-degree basis) replace,
// per pseudo-step
// (src/pde/hamilton_jacobi.cc:514-551):
//   local_left_right_gradients  (hamilton_jacobi.cc:462-511; LDG integrators
//                                src/pde/ldg.cc:355-376, 510-740)
//   ReinitOperator::cell_values (src/level_set/reinit.cc:267-301: smooth sign
//                                :121-133, Lax-Friedrichs H :136-191)
//   HJAssemblerWorkStream       (hamilton_jacobi.cc:730-745)
//   the mass solve and the RK update,
// and the characteristic-speed CFL estimate the next pseudo-step uses
// (ReinitOperator::cell_velocities reinit.cc:304-328, characteristic_velocity
// :235-264, CFLEstimator at QTrapezoid vertices).
//
// The LDG one-sided gradients are computed modally and exactly: for the
// orthonormal Legendre basis, QGauss(p+1) integrates every LDG term without
// error, so  g^L_e = (1/h_e) [ -A c + L(1) (x) T_up - L(0) (x) T_lo^left ]
// along each line of axis e (A_ab = int L_a' L_b, T the face traces, the
// left/right flux taking the trace of the lower/upper cell, the interior
// trace on the boundary).  In the P basis the padded Q modes are masked.
#pragma once
#include "flsp_device.cuh"

namespace flsp {

template <typename T>
struct HJArgs {
  MeshArgs m;
  const T* __restrict__ phi;    // phi^k (read with halo)
  T* __restrict__ out;          // phi^{k+1}
  double* __restrict__ grad;    // gradient blocks (the export)
  DevClock* clk;
  int mode;
  int rk;                       // reinit RK order (all stages see the same L)
  HjClockArgs step;             // pseudo-step sizes
  long long block;              // gradient block stride (ncell * nb)
  const T* __restrict__ rdiff;  // LDG diffusion RHS per unit volume (nu > 0) or null
  T* stab;                      // smooth-sign table of the tensor-product kernel (hjs_kernel)
  int* err;                     // the problem's error word
};

// tile of the gradient export
template <int DIM>
struct HjgTile {
  static constexpr int X = DIM == 2 ? 16 : 8, Y = DIM == 2 ? 16 : 4, Z = DIM == 2 ? 1 : 4;
};
template <int DIM, int P, typename T>
constexpr size_t hjg_smem_bytes() {
  using TL = HjgTile<DIM>;
  return (size_t)(TL::X + 2) * (TL::Y + 2) * (DIM > 2 ? TL::Z + 2 : 1) * ipow(P + 1, DIM) * sizeof(T);
}

// RK combinations of ReinitSimulatorLDG::advance_time with the reference's
// operation order; explicit_time_derivative ignores its argument
// (hamilton_jacobi.cc:514-551), so every stage uses the same L.
template <typename T>
__device__ __forceinline__ T hj_combine(int rk, T phi, T L, T dt) {
  if (rk <= 1) { T s = L * dt; return s + phi; }
  if (rk == 2) { T s = phi; s += dt * L; s += dt * L; s += phi; return s * T(0.5); }
  T s = phi;
  s += dt * L; s += dt * L; s += T(3.0) * phi; s *= T(0.25);
  s += dt * L; s *= T(2.0); s += phi;
  return s * (T(1.0) / T(3.0));
}

// left gradient blocks (one per axis), then the right ones, of every cell
// (HJSimulator::local_left_right_gradients): an export, one thread per cell
template <int DIM, int P, typename T>
__global__ void __launch_bounds__(256) hj_gradient_kernel(const HJArgs<T> a) {
  constexpr int N1 = P + 1, NM = ipow(N1, DIM);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const MeshArgs& m = a.m;
  T* box = reinterpret_cast<T*>(smem_raw);
  const Tab1D<T>& tb = tab<T>(P);
  const TileCoord tc = tile_coord(m, DIM);
  load_box<DIM, NM>(m, a.phi, box, tc.ox, tc.oy, tc.oz, true);
  cp_async_wait_all();
  __syncthreads();
  if (!tc.valid) return;
  const int st[3] = {1, N1, N1 * N1};
  const long long cell = (long long)tc.gx + (long long)m.n[0] * (tc.gy + (long long)m.n[1] * tc.gz);
  const T* c = box + (size_t)box_index(m, DIM, tc.lx, tc.ly, tc.lz) * NM;
#pragma unroll
  for (int e = 0; e < DIM; ++e) {
    const T ih = T(1.0 / m.h[e]);
    int nl[3] = {tc.lx, tc.ly, tc.lz}, nu[3] = {tc.lx, tc.ly, tc.lz};
    int gg[3] = {tc.gx, tc.gy, tc.gz};
    nl[e] -= 1;
    nu[e] += 1;
    const bool has_lo = gg[e] > 0, has_hi = gg[e] + 1 < m.n[e];
    T glo = T(0), ghi = T(0);
    const bool dlo = !has_lo && bc_dirichlet<DIM>(m, e, 0, gg, glo);
    const bool dhi = !has_hi && bc_dirichlet<DIM>(m, e, 1, gg, ghi);
    const T* cL = box + (size_t)box_index(m, DIM, nl[0], nl[1], nl[2]) * NM;
    const T* cU = box + (size_t)box_index(m, DIM, nu[0], nu[1], nu[2]) * NM;
    // lines along axis e: enumerate the other two mode indices
#pragma unroll
    for (int li = 0; li < NM / N1; ++li) {
      const int i0 = li % N1, i1 = li / N1;
      int base;
      if (e == 0) base = i0 * st[1] + i1 * st[2];
      else if (e == 1) base = i0 * st[0] + i1 * st[2];
      else base = i0 * st[0] + i1 * st[1];
      if constexpr (DIM == 2) { base = (e == 0) ? i0 * st[1] : i0 * st[0]; }
      T tup = T(0), tlo = T(0), tnl = T(0), tnu = T(0);
#pragma unroll
      for (int b = 0; b < N1; ++b) {
        const T cb = c[base + b * st[e]];
        tup += tb.L1[b] * cb;
        tlo += tb.L0[b] * cb;
        if (has_lo) tnl += tb.L1[b] * cL[base + b * st[e]];
        if (has_hi) tnu += tb.L0[b] * cU[base + b * st[e]];
      }
      // domain boundary: the Dirichlet value of the face (constant mode
      // only) where it carries one, else the interior trace
      if (!has_lo) tnl = dlo ? (li == 0 ? glo : T(0)) : tlo;
      if (!has_hi) tnu = dhi ? (li == 0 ? ghi : T(0)) : tup;
#pragma unroll
      for (int aa = 0; aa < N1; ++aa) {
        const int k = m.q2g[base + aa * st[e]];
        if (k < 0) continue;
        T bs = T(0);
#pragma unroll
        for (int b = 0; b < N1; ++b) bs -= tb.A[aa][b] * c[base + b * st[e]];
        a.grad[(long long)e * a.block + cell * m.nb + k] = (bs + tb.L1[aa] * tup - tb.L0[aa] * tnl) * ih;
        a.grad[(long long)(DIM + e) * a.block + cell * m.nb + k] = (bs + tb.L1[aa] * tnu - tb.L0[aa] * tlo) * ih;
      }
    }
  }
}

}  // namespace flsp
