// flsp_ldg.cuh — LDG artificial viscosity of the reinitialisation (nu > 0).
//
// Replaces LDGDiffusionTerm::compute_diffusion_term (src/pde/ldg.cc:249-298):
// the alternating-flux gradient q (LDGGradientAssembler<alternating>,
// ldg.cc:383-504, with beta renormalised to (1,..,1)/sqrt(dim),
// ldg.implement.h:304-313) followed by the diffusion RHS
// (LDGDiffusionAssembler<alternating>, ldg.cc:750-838; no boundary term).
// Every integral is of polynomial products integrated exactly by the
// reference's QGauss(p+1), so the kernel works modally, one line of modes
// along each axis d at a time (faces normal to d are the only ones with
// n_d != 0).  Along an axis, with kp = 1/2 + 1/sqrt(dim), km = 1/2 - 1/sqrt(dim)
// and the traces x(0), x(1) of a line at its ends:
//   phi^ = km left(1) + kp right(0)     (at the domain boundary the cell's own trace)
//   q    = (1/h) [ -A c + L(1) phi^_up - L(0) phi^_lo ]
//   F    = kp qleft(1) + km qright(0)   (none at the domain boundary)
//   R    = (nu/h) [ -A q + L(1) F_up - L(0) F_lo ]
// all per unit cell volume.  R of a cell needs q of its own line and one trace
// of each neighbour's, and that is a dot product: with L_a(1) = (-1)^a L_a(0) =
// sqrt(2a+1), A_ab = 2 L_a(1) L_b(1) for a > b, a - b odd (else 0), and modes
// 0..K of the line in use,
//   q(1) = (1/h) [ -s1 + (K+1)^2 phi^_up - (-1)^K (K+1) phi^_lo ],
//   q(0) = (1/h) [ -s0 + (-1)^K (K+1) phi^_up - (K+1)^2 phi^_lo ],
//   s1 = sum_b W_b c_b,  s0 = -sum_b (-1)^b W_b c_b,
//   W_b = 2 L_b(1) sum_{b < a <= K, a - b odd} (2a + 1).
// So one pass over phi with a halo of two cells does what a gradient launch, DIM
// blocks of q in memory and a second launch did (256^2 Q2 FP32 2 x 9.2 us, a run
// of 30 pseudo-steps 3.03 -> 2.66 ms; 29x31x33 Q2 FP64, 20: 5.61 -> 4.02 with the
// other kernels' steps).  A thread per (cell, axis); the axes' sums meet in the
// coalesced store.  Bound by latency at these sizes (2 state vectors of traffic).
// In a narrow band q exists in the listed tiles only (LdgArgs::listed): a
// neighbour outside them gives no flux, as when q was kept in a zeroed vector.
#pragma once
#include "flsp_device.cuh"

namespace flsp {

template <typename T>
struct LdgArgs {
  MeshArgs m;              // m.tile: the narrow band's unit, a multiple of LdgTile
  const T* __restrict__ in;    // phi
  T* __restrict__ out;         // R_diff
  const int* listed;       // narrow band: 1 for each tile that is listed (else null)
  double nu;
  int* err;                // the problem's error word
};

// block of cells
template <int DIM>
struct LdgTile {
  static constexpr int X = DIM == 2 ? 16 : 4, Y = DIM == 2 ? 8 : 4, Z = DIM == 2 ? 1 : 4;
  static constexpr int N = X * Y * Z;
};

template <int DIM, int P, bool PB, typename T>
struct LdgPlan {
  using TL = LdgTile<DIM>;
  static constexpr int NBG = PB ? (DIM == 2 ? (P + 1) * (P + 2) / 2 : (P + 1) * (P + 2) * (P + 3) / 6) : ipow(P + 1, DIM);
  static constexpr int NMB = NBG * (int)sizeof(T), BY = TL::Y + 4, NROWS = BY * (DIM > 2 ? TL::Z + 4 : 1);
  static constexpr int SLOT = (((TL::X + 4) * NMB + 30) + 15) / 16 * 16;
  static constexpr int NS = NBG | 1;   // stride of a cell's sums: odd, no bank conflicts
  static constexpr size_t OFF_BOX = 16, BOX = (size_t)NROWS * SLOT;
  static constexpr size_t SUMS = (size_t)DIM * TL::N * NS * sizeof(T);   // over the box
  static constexpr size_t BYTES = OFF_BOX + (BOX > SUMS ? BOX : SUMS);
};

// one thread's axis E of the cell at local l, global g: R into r (HBM order)
template <int DIM, int P, bool PB, int E, typename T, typename CellP>
__device__ __forceinline__ void ldg_axis(const LdgArgs<T>& a, const CellP& cellp, const int* l, const int* g, T* r) {
  constexpr int N1 = P + 1, t0 = E == 0 ? 1 : 0, t1 = E == 2 ? 1 : 2;
  constexpr int st[3] = {1, N1, N1 * N1};
  const MeshArgs& m = a.m;
  const Tab1D<T>& tb = tab<T>(P);
  const T kp = T(0.5 + 1.0 / sqrt((double)DIM)), km = T(0.5 - 1.0 / sqrt((double)DIM));
  const T ih = T(1.0 / m.h[E]), nu = T(a.nu);
  auto at = [&](int o) { return cellp(l[0] + (E == 0 ? o : 0), l[1] + (E == 1 ? o : 0), l[2] + (E == 2 ? o : 0)); };
  const bool h1 = g[E] > 0, h2 = g[E] > 1, u1 = g[E] + 1 < m.n[E], u2 = g[E] + 2 < m.n[E];
  // a neighbour outside the band's tiles has no q
  bool q1 = h1, q2 = u1;
  if (a.listed) {
    auto in_band = [&](int o) {
      const int x = (g[0] + (E == 0 ? o : 0)) / m.tile[0], y = (g[1] + (E == 1 ? o : 0)) / m.tile[1];
      const int z = DIM > 2 ? (g[2] + (E == 2 ? o : 0)) / m.tile[2] : 0;
      return a.listed[x + m.ntile[0] * (y + (long long)m.ntile[1] * z)] != 0;
    };
    q1 = h1 && in_band(-1);
    q2 = u1 && in_band(1);
  }
  const T *c0 = at(0), *cl1 = at(-1), *cl2 = at(-2), *cu1 = at(1), *cu2 = at(2);
#pragma unroll
  for (int m1 = 0; m1 < (DIM > 2 ? N1 : 1); ++m1)
#pragma unroll
    for (int m0 = 0; m0 < N1; ++m0) {
      if (PB && m0 + m1 > P) continue;
      const int K = PB ? P - m0 - m1 : P, base = m0 * st[t0] + (DIM > 2 ? m1 * st[t1] : 0);
      auto line = [&](const T* c, T* x) {
#pragma unroll
        for (int b = 0; b < N1; ++b)
          if (b <= K) x[b] = c[PB ? q2g_ct<DIM, P>(base + b * st[E]) : base + b * st[E]];
      };
      // the line's traces
      auto ends = [&](const T* x, T& lo, T& hi) {
        T e = x[0], o = T(0);
#pragma unroll
        for (int b = 1; b < N1; ++b)
          if (b <= K) (b % 2 ? o : e) += tb.L1[b] * x[b];
        lo = e - o;
        hi = e + o;
      };
      // s0, s1 of the line
      auto ends_of_a = [&](const T* x, T& s0, T& s1) {
        T e = T(0), o = T(0);
#pragma unroll
        for (int b = 0; b < N1; ++b) {
          int w = 0;
#pragma unroll
          for (int aa = b + 1; aa < N1; aa += 2)
            if (aa <= K) w += 2 * (2 * aa + 1);
          if (w > 0) (b % 2 ? o : e) += T(w) * tb.L1[b] * x[b];
        }
        s0 = o - e;
        s1 = e + o;
      };
      auto minus_a = [&](const T* x, int aa) {   // -(A x)_aa
        T s = T(0);
#pragma unroll
        for (int b = 0; b < N1; ++b)
          if (b < aa && (aa - b) % 2) s -= tb.A[aa][b] * x[b];
        return s;
      };
      const T k2 = T((K + 1) * (K + 1)), k1 = T(K % 2 ? -(K + 1) : K + 1);
      T x[N1], y[N1], lo, hi, ylo = T(0), yhi = T(0), fa, fb, flo = T(0), fup = T(0);
      line(c0, x);
      ends(x, lo, hi);
      fa = lo;
      fb = hi;
      T prev = T(0);   // the lower neighbour's q(1)
      if (h1) {
        line(cl1, y);
        ends(y, ylo, yhi);
        fa = km * yhi + kp * lo;
        if (q1) {
          T s0, s1, f2 = ylo;
          ends_of_a(y, s0, s1);
          if (h2) {
            T z[N1], zlo, zhi;
            line(cl2, z);
            ends(z, zlo, zhi);
            f2 = km * zhi + kp * ylo;
          }
          prev = ih * (k2 * fa - k1 * f2 - s1);
        }
      }
      T next = T(0);   // the upper neighbour's q(0)
      if (u1) {
        line(cu1, y);
        ends(y, ylo, yhi);
        fb = km * hi + kp * ylo;
        if (q2) {
          T s0, s1, f3 = yhi;
          ends_of_a(y, s0, s1);
          if (u2) {
            T z[N1], zlo, zhi;
            line(cu2, z);
            ends(z, zlo, zhi);
            f3 = km * yhi + kp * zlo;
          }
          next = ih * (k1 * f3 - k2 * fb - s0);
        }
      }
      T q[N1];
#pragma unroll
      for (int aa = 0; aa < N1; ++aa)
        if (aa <= K) q[aa] = ih * (minus_a(x, aa) + tb.L1[aa] * (aa % 2 ? fb + fa : fb - fa));
      ends(q, lo, hi);
      if (h1) flo = kp * prev + km * lo;
      if (u1) fup = kp * hi + km * next;
#pragma unroll
      for (int aa = 0; aa < N1; ++aa)
        if (aa <= K) {
          const int q0 = base + aa * st[E];
          r[PB ? q2g_ct<DIM, P>(q0) : q0] = nu * ih * (minus_a(q, aa) + tb.L1[aa] * (aa % 2 ? fup + flo : fup - flo));
        }
    }
}

template <int DIM, int P, bool PB, typename T>
__global__ void __launch_bounds__(LdgTile<DIM>::N * DIM) ldg_kernel(const LdgArgs<T> a) {
  using PL = LdgPlan<DIM, P, PB, T>;
  using TL = LdgTile<DIM>;
  constexpr int TX = TL::X, TY = TL::Y, TZ = TL::Z, NT = TL::N, NBG = PL::NBG, NMB = PL::NMB, NS = PL::NS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem_raw);
  unsigned char* boxb = smem_raw + PL::OFF_BOX;
  T* sums = reinterpret_cast<T*>(boxb);   // [DIM][NT][NS]
  const MeshArgs& m = a.m;
  if (threadIdx.x == 0) mbar_init(bar, 32);
  __syncthreads();
  chain_wait();
  const int sx = m.tile[0] / TX, sy = m.tile[1] / TY, parts = sx * sy * (DIM > 2 ? m.tile[2] / TZ : 1);
  const int slot = (int)blockIdx.x / parts, part = (int)blockIdx.x % parts;
  if (tile_inactive(m, slot)) return;
  int o[3];
  {
    int b = m.tiles ? m.tiles[slot] : slot;
    o[0] = (b % m.ntile[0]) * m.tile[0] + (part % sx) * TX;
    b /= m.ntile[0];
    o[1] = (b % m.ntile[1]) * m.tile[1] + (part / sx) % sy * TY;
    o[2] = DIM > 2 ? (b / m.ntile[1]) * m.tile[2] + part / (sx * sy) * TZ : 0;
  }
  if (o[0] >= m.n[0] || o[1] >= m.n[1] || o[2] >= m.n[2]) return;   // a part past the mesh
  if (threadIdx.x < 32) bulk_box_rows<DIM, TX, TY, TZ, NMB, PL::SLOT, 2>(m, a.in, boxb, o[0], o[1], o[2], bar);
  const int cl = (int)threadIdx.x % NT, d = (int)threadIdx.x / NT;   // cell, axis (uniform per warp)
  const int l[3] = {cl % TX, (cl / TX) % TY, DIM > 2 ? cl / (TX * TY) : 0};
  const int g[3] = {o[0] + l[0], o[1] + l[1], o[2] + l[2]};
  const bool valid = g[0] < m.n[0] && g[1] < m.n[1] && (DIM < 3 || g[2] < m.n[2]);
  const int gx0 = max(o[0] - 2, 0);
  auto cellp = [&](int lx, int ly, int lz) -> const T* {
    const int rr = (ly + 2) + PL::BY * (DIM > 2 ? lz + 2 : 0);
    const unsigned rowcell = (unsigned)m.n[0] * (unsigned)((o[1] + ly) + m.n[1] * (DIM > 2 ? o[2] + lz : 0));
    const unsigned phase = ((rowcell + (unsigned)gx0) * (unsigned)NMB) & 15u;
    return reinterpret_cast<const T*>(boxb + (ptrdiff_t)rr * PL::SLOT + phase + (ptrdiff_t)(o[0] + lx - gx0) * NMB);
  };
  if (!mbar_wait(bar, 0u, 1 << 22)) {
    if (threadIdx.x == 0 && a.err) atomicOr(a.err, kErrCopyTimeout);
    mbar_wait(bar, 0u, 1 << 22);   // give copies in flight a last chance to land
  }
  T r[NBG];
  if (valid) {
    if (d == 0) ldg_axis<DIM, P, PB, 0, T>(a, cellp, l, g, r);
    else if (d == 1) ldg_axis<DIM, P, PB, 1, T>(a, cellp, l, g, r);
    else if constexpr (DIM > 2) ldg_axis<DIM, P, PB, 2, T>(a, cellp, l, g, r);
  }
  __syncthreads();   // the box becomes the sums
  if (valid)
#pragma unroll
    for (int k = 0; k < NBG; ++k) sums[(size_t)(d * NT + cl) * NS + k] = r[k];
  __syncthreads();
  chain_release();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = min(TX, m.n[0] - o[0]) * NBG;
  for (int row = warp; row < TY * TZ; row += NT * DIM / 32) {
    const int gy = o[1] + row % TY, gz = o[2] + row / TY;
    if (gy >= m.n[1] || gz >= m.n[2]) continue;
    T* dst = a.out + ((long long)m.n[0] * (gy + (long long)m.n[1] * gz) + o[0]) * NBG;
#pragma unroll
    for (int e = lane; e < TX * NBG; e += 32) {
      if (e >= n) continue;
      const T* s = sums + (size_t)(TX * row + e / NBG) * NS + e % NBG;
      T v = s[0] + s[(size_t)NT * NS];
      if constexpr (DIM > 2) v += s[(size_t)2 * NT * NS];
      dst[e] = v;
    }
  }
}

}  // namespace flsp
