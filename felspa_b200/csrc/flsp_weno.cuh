// flsp_weno.cuh — 2D minmod troubled-cell detector + WENO limiter, one pass.
//
// Replaces dg::apply_weno_limiter (include/felspa/pde/src/pde_tools.implement.h:977-1004):
// MinmodShockDetector::cell_has_shock (:277-376, beta = 1 + dim) flags cells
// from the state before limiting, then WENOLimiter::apply_limiting_to_cell
// (:557-706) rebuilds each flagged cell from the old copy of the state
// (gamma_neighbour = 0.001, eps = 1e-6, smoothness up to min(2, p)
// derivatives).  Both read only the pre-limit state, so a CTA reads `in` (tile
// + face halo in shared memory) and writes `out`.  The smoothness indicator
// keeps the reference's indexing of the Hessian (hessians[i][j] with
// i, j < dim indexes the quadrature point i, :545-547) and scales neighbour
// terms by the neighbour's cell measure (:524).
//
// Everything the reference integrates with QGauss(p+2) is a polynomial that
// rule integrates exactly, so it is taken from the coefficients: a cell's
// average is its mode 0 (L_0 = 1); a neighbour's polynomial over the home cell
// has the coefficients S c, S_ab = int L_a(x) L_b(x + 1) (by parity also for
// the other side); int |grad p|^2 is the norm of the derivative's
// coefficients; the new polynomial's projection is the weighted sum of
// coefficients.  That leaves ~400 (degree 2) instructions for a troubled
// cell, few enough for the cell's own thread.
// What bounds it: latency (one load of the tile, then dependent sums).
// Against point-wise averages at (p+2)^2 points of five cells per cell and a
// second pass over a list of troubled cells, a warp each: 256^2 Q2 FP32
// 33.4 -> 4.7 us, 233x190 Q3 FP64 111.5 -> 9.3, 128^2 P1 FP64 26.5 -> 4.2.
#pragma once
#include "flsp_stage.cuh"

namespace flsp {

template <typename T>
struct WenoArgs {
  MeshArgs m;
  const T* __restrict__ in;
  T* __restrict__ out;
  unsigned int* count;   // troubled-cell counter (may be null)
  int* err;              // the problem's error word
};

// a CTA's cells: half of a limiter tile (kWenoTile; the unit the narrow band
// lists)
struct WenoBlock {
  static constexpr int X = 16, Y = 8, N = X * Y;
};

template <int P, bool PB, typename T>
struct WenoPlan {
  static constexpr int N1 = P + 1, NM = N1 * N1, NBG = PB ? (P + 1) * (P + 2) / 2 : NM;
  static constexpr int NMB = NBG * (int)sizeof(T), NROWS = WenoBlock::Y + 2;
  static constexpr int SLOT = (((WenoBlock::X + 2) * NMB + 30) + 15) / 16 * 16;
  static constexpr size_t OFF_BOX = 16;
  static constexpr size_t OFF_SB = OFF_BOX + (size_t)NROWS * SLOT;   // results [cell][NBG]
  static constexpr size_t BYTES = OFF_SB + (size_t)WenoBlock::N * NBG * sizeof(T);
};

// smoothness indicator of a polynomial from its coefficients on the home cell
template <int P, typename T>
__device__ __forceinline__ T weno_smoothness(const Tab1D<T>& tb, const T* c, T ihx, T ihy, T vol) {
  constexpr int N1 = P + 1;
  T sx = T(0), sy = T(0);
#pragma unroll
  for (int b = 0; b < N1; ++b)
#pragma unroll
    for (int a = 0; a < P; ++a) {   // derivative coefficients: A[a'][a] = int L_a' ' L_a, a' > a, a' - a odd
      T gx = T(0), gy = T(0);
#pragma unroll
      for (int k = a + 1; k < N1; k += 2) {
        gx += tb.A[k][a] * c[k + N1 * b];
        gy += tb.A[k][a] * c[b + N1 * k];
      }
      sx += gx * gx;
      sy += gy * gy;
    }
  T beta = (sx * (ihx * ihx) + sy * (ihy * ihy)) * (vol * vol);
  if constexpr (P >= 2) {
    // second derivatives at the home points 0 and 1
    T xx = T(0), xy = T(0), yy = T(0), xy1 = T(0), yy1 = T(0);
#pragma unroll
    for (int a = 0; a < N1; ++a) {
      T v = c[a], d = T(0), h = T(0);
#pragma unroll
      for (int b = 1; b < N1; ++b) {
        v += c[a + N1 * b] * tb.Lq[b][0];
        d += c[a + N1 * b] * tb.Dq[b][0];
        if (b > 1) h += c[a + N1 * b] * tb.Hq[b][0];
      }
      if (a > 1) xx += tb.Hq[a][0] * v;
      if (a > 0) xy += tb.Dq[a][0] * d;
      if (a > 0) xy1 += tb.Dq[a][1] * d;
      yy += tb.Lq[a][0] * h;
      yy1 += tb.Lq[a][1] * h;
    }
    xx *= ihx * ihx;
    xy *= ihx * ihy;
    yy *= ihy * ihy;
    xy1 *= ihx * ihy;
    yy1 *= ihy * ihy;
    const T ls = xx * xx + xy * xy + xy * xy + yy * yy + xy1 * xy1 + yy1 * yy1;
    beta += ls * vol * (vol * vol * vol);
  }
  return beta;
}

// coefficients on the home cell of the neighbour polynomial cn on side S
// (0: lower, 1: upper) of axis E, Q layout
template <int P, bool PB, int E, int S, typename T>
__device__ __forceinline__ void weno_shift(const Tab1D<T>& tb, const T* __restrict__ cn, T* c) {
  constexpr int N1 = P + 1;
#pragma unroll
  for (int b = 0; b < N1; ++b)
#pragma unroll
    for (int a = 0; a < N1; ++a) {
      T s = T(0);
#pragma unroll
      for (int k = a; k < N1; ++k) {   // S is upper triangular, S_aa = 1
        if (!mode_in<P, PB>(k + b)) continue;
        const T x = cn[cell_index<2, P, PB>(E == 0 ? k + N1 * b : b + N1 * k)];
        if (k == a) s += x;
        else if (S == 1 && (k - a) % 2) s -= tb.S[a][k] * x;
        else s += tb.S[a][k] * x;
      }
      c[E == 0 ? a + N1 * b : b + N1 * a] = s;
    }
}

// block `part` (0, 1) of a limiter tile; launch slot as in the other kernels
template <int P, bool PB, typename T>
__device__ __forceinline__ void weno_tile(const WenoArgs<T>& a, int slot, int part) {
  using PL = WenoPlan<P, PB, T>;
  constexpr int N1 = PL::N1, NM = PL::NM, NBG = PL::NBG, NMB = PL::NMB;
  constexpr int TX = WenoBlock::X, TY = WenoBlock::Y;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem_raw);
  unsigned char* boxb = smem_raw + PL::OFF_BOX;
  T* sb = reinterpret_cast<T*>(smem_raw + PL::OFF_SB);
  const MeshArgs& m = a.m;
  const Tab1D<T>& tb = tab<T>(P);
  if (threadIdx.x == 0) mbar_init(bar, 32);
  __syncthreads();
  chain_wait();
  if (tile_inactive(m, slot)) return;
  const int tile = m.tiles ? m.tiles[slot] : slot;
  const int ox = (tile % m.ntile[0]) * m.tile[0], oy = (tile / m.ntile[0]) * m.tile[1] + part * TY;
  if (oy >= m.n[1]) return;
  if (threadIdx.x < 32) bulk_box_rows<2, TX, TY, 1, NMB, PL::SLOT>(m, a.in, boxb, ox, oy, 0, bar);
  const int lx = (int)threadIdx.x % TX, ly = (int)threadIdx.x / TX;
  const int gx = ox + lx, gy = oy + ly, gx0 = max(ox - 1, 0);
  const bool valid = gx < m.n[0] && gy < m.n[1];
  auto cellp = [&](int x, int y) -> const T* {
    const unsigned phase = (((unsigned)m.n[0] * (unsigned)(oy + y) + (unsigned)gx0) * (unsigned)NMB) & 15u;
    return reinterpret_cast<const T*>(boxb + (size_t)(y + 1) * PL::SLOT + phase + (ox + x - gx0) * NMB);
  };
  if (!mbar_wait(bar, 0u, 1 << 22)) {
    if (threadIdx.x == 0 && a.err) atomicOr(a.err, kErrCopyTimeout);
    mbar_wait(bar, 0u, 1 << 22);   // give copies in flight a last chance to land
  }

  bool troubled = false;
  if (valid) {
    T c[NM];
    {
      const T* own = cellp(lx, ly);
#pragma unroll
      for (int q = 0; q < NM; ++q) {
        const int gi = cell_index<2, P, PB>(q);
        c[q] = gi >= 0 ? own[gi] : T(0);
      }
    }
    const bool ok[4] = {gx > 0, gx + 1 < m.n[0], gy > 0, gy + 1 < m.n[1]};
    // ---------------- minmod detection ----------------
    const T avg = c[0];
    T dn[4];   // neighbour averages minus the own one (face order x-, x+, y-, y+)
#pragma unroll
    for (int f = 0; f < 4; ++f)
      dn[f] = ok[f] ? cellp(lx + (f == 1) - (f == 0), ly + (f == 3) - (f == 2))[0] - avg : T(0);
    // vertex values minus the average
    T lo[N1], hi[N1];
#pragma unroll
    for (int b = 0; b < N1; ++b) {
      T x[N1];
#pragma unroll
      for (int aa = 0; aa < N1; ++aa) x[aa] = aa + b == 0 ? T(0) : c[aa + N1 * b];
      end_values<N1, 1, T>(tb, x, lo[b], hi[b]);
    }
    T vv[4];
    end_values<N1, 1, T>(tb, lo, vv[0], vv[2]);
    end_values<N1, 1, T>(tb, hi, vv[1], vv[3]);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int f0 = v & 1, f1 = 2 + (v >> 1);
      if (!ok[f0] || !ok[f1]) continue;
      // directional coefficients (c_nb - c).(v - c) / |c_nb - c|^2 = 1/2 on a
      // uniform Cartesian mesh, beta = 1 + dim
      const T aa = vv[v], bb = T(3) * (T(0.5) * dn[f0] + T(0.5) * dn[f1]);
      const int sa = (aa > T(0)) - (aa < T(0)), sg = (bb > T(0)) - (bb < T(0));
      const T mm = (sa == sg) ? T(sa) * fmin(fabs(aa), fabs(bb)) : T(0);
      troubled = troubled || aa != mm;
    }
    // ---------------- WENO reconstruction ----------------
    if (troubled) {
      const T ihx = T(1.0 / m.h[0]), ihy = T(1.0 / m.h[1]), vol = T(m.vol);
      const T gamma_nb = T(0.001), eps = T(1.0e-6);
      T acc = T(0);
#pragma unroll
      for (int f = 0; f < 4; ++f)
        if (ok[f]) acc += gamma_nb;
      T den = eps + weno_smoothness<P, T>(tb, c, ihx, ihy, vol);
      T w = (T(1) - acc) / den / den;
      T wsum = w;
#pragma unroll
      for (int q = 0; q < NM; ++q) c[q] *= w;
      // neighbour order: faces 0..3 (find_neighbor_cells, :482-508)
      auto add = [&](auto EC, auto SC) {
        constexpr int E = decltype(EC)::value, S = decltype(SC)::value;
        if (!ok[2 * E + S]) return;
        T n[NM];
        weno_shift<P, PB, E, S, T>(tb, cellp(lx + (E == 0 ? 2 * S - 1 : 0), ly + (E == 1 ? 2 * S - 1 : 0)), n);
        const T dl = eps + weno_smoothness<P, T>(tb, n, ihx, ihy, vol);
        const T wl = gamma_nb / dl / dl;
        wsum += wl;
#pragma unroll
        for (int q = 1; q < NM; ++q) c[q] += wl * n[q];
      };
      add(std::integral_constant<int, 0>(), std::integral_constant<int, 0>());
      add(std::integral_constant<int, 0>(), std::integral_constant<int, 1>());
      add(std::integral_constant<int, 1>(), std::integral_constant<int, 0>());
      add(std::integral_constant<int, 1>(), std::integral_constant<int, 1>());
      // every polynomial is shifted to the home average: mode 0 stays
      c[0] = avg;
#pragma unroll
      for (int q = 1; q < NM; ++q) c[q] /= wsum;
    }
#pragma unroll
    for (int q = 0; q < NM; ++q) {
      const int gi = cell_index<2, P, PB>(q);
      if (gi >= 0) sb[(size_t)threadIdx.x * NBG + gi] = c[q];
    }
  }
  if (a.count) {
    const int n = __syncthreads_count(troubled);
    if (threadIdx.x == 0 && n) atomicAdd(a.count, (unsigned)n);
  } else {
    __syncthreads();
  }
  chain_release();
  store_cells<2, TX, TY, 1, NBG, T>(m, sb, a.out, ox, oy, 0);
}

template <int P, bool PB, typename T>
__global__ void __launch_bounds__(WenoBlock::N) weno_kernel(const WenoArgs<T> a) {
  weno_tile<P, PB, T>(a, (int)blockIdx.x / 2, (int)blockIdx.x % 2);
}

}  // namespace flsp
