// flsp_hjp.cuh — Hamilton-Jacobi reinitialisation pseudo-step, total-degree
// (FE_DGP) basis.
//
// The operator and the frame of hjs_kernel (flsp_hjs.cuh: NQ threads per
// cell, thread k on Gauss plane k of the last axis, the smooth sign from the
// sweep's table), for fields in P space, where the one-sided gradients are
// the strong derivative plus the lifted face jumps *projected onto P*, so
// that the nodal shortcut of the tensor basis does not apply:
//   (1) one work item per (axis, cell) forms the modal gradients of that
//       axis: mean (l + r) / 2 and half difference (l - r) / 2, NBG modes
//       each (LDG left / right gradients, ldg.cc:355-376, :510-740);
//   (2) per Gauss plane the three means and the sum of the half differences
//       (the Lax-Friedrichs H needs no more, reinit.cc:136-191) are summed
//       mode by mode over the modes P space has: a 3D degree-2 field takes
//       4 + 12 + 24 instructions for the 16 points of a plane;
//   (3) the planes' projections meet in shared memory, as in hjs_kernel.
// What bounds it: issue and latency, as hjs_kernel; 60^3 degree 2 FP32 took
// 1636 us in the point-by-point kernel this one replaces (every field value
// a sum over all 27 padded modes, 255 registers), and takes 64 us here;
// FP64 3998 -> 113 us, 128^2 degree 1 FP64 16.4 -> 6.2 us.
//
// The launch's tiles (m.tile) may hold several HjsTile blocks of cells: block
// b serves part b % NS of tile b / NS.  The narrow band lists whole tiles,
// and which cells it sweeps is part of its result, so the tiles keep their
// shapes (hj_default_tile, flsp_k_hj.cu).
#pragma once
#include "flsp_hjs.cuh"

namespace flsp {

template <int DIM, int P, typename T>
struct HjpPlan {
  using TL = HjsTile<DIM>;
  static constexpr int N1 = P + 1, NQ = P + 2, NQF = ipow(NQ, DIM - 1);
  static constexpr int NBG = DIM == 2 ? (P + 1) * (P + 2) / 2 : (P + 1) * (P + 2) * (P + 3) / 6;
  static constexpr int NBY = TL::Y + 2, NBZ = DIM > 2 ? TL::Z + 2 : 1, NROWS = NBY * NBZ;
  static constexpr int NMB = NBG * (int)sizeof(T);
  static constexpr int SLOT = (((TL::X + 2) * NMB + 30) + 15) / 16 * 16;
  static constexpr int NS = ipow(NQ, DIM) + (1 << DIM);
  static constexpr size_t TAB_BYTES = (size_t)NS * TL::N * sizeof(T);
  static constexpr size_t OFF_BOX = 32;   // mbarrier, CFL maximum, pseudo-step
  static constexpr size_t OFF_GR = OFF_BOX + (size_t)NROWS * SLOT;
  // modal gradients [mean, half difference][axis][mode][cell]; the results'
  // staging at the end
  static constexpr size_t OFF_TAB = (OFF_GR + (size_t)2 * DIM * NBG * TL::N * sizeof(T) + 15) / 16 * 16;
  static constexpr size_t BYTES = OFF_TAB + TAB_BYTES;
};

// 80 (3D FP32) registers hold three CTAs per SM
template <int DIM, int P, typename T>
constexpr int hjp_min_blocks() {
  return DIM == 3 && sizeof(T) == 4 ? 3 : 1;
}

// modal gradients of axis E of the tile's cell cl at local l, global g
template <int DIM, int P, int E, typename T, typename CellP>
__device__ __forceinline__ void hjp_gradient(const MeshArgs& m, const CellP& cellp, const int* l, const int* g, T* gr,
                                             int cl) {
  constexpr int N1 = P + 1, NT = HjsTile<DIM>::N, NBG = HjpPlan<DIM, P, T>::NBG;
  constexpr int t0 = E == 0 ? 1 : 0, t1 = E == 2 ? 1 : 2;
  constexpr int st[3] = {1, N1, N1 * N1};
  const Tab1D<T>& tb = tab<T>(P);
  const T ih = T(1.0 / m.h[E]);
  const bool has_lo = g[E] > 0, has_hi = g[E] + 1 < m.n[E];
  T glo = T(0), ghi = T(0);
  const bool dlo = !has_lo && bc_dirichlet<DIM>(m, E, 0, g, glo);
  const bool dhi = !has_hi && bc_dirichlet<DIM>(m, E, 1, g, ghi);
  const T* c = cellp(l[0], l[1], l[2]);
  const T* cL = cellp(l[0] - (E == 0), l[1] - (E == 1), l[2] - (E == 2));
  const T* cU = cellp(l[0] + (E == 0), l[1] + (E == 1), l[2] + (E == 2));
#pragma unroll
  for (int m1 = 0; m1 < (DIM > 2 ? N1 : 1); ++m1)
#pragma unroll
    for (int m0 = 0; m0 + m1 < N1; ++m0) {
      const int lim = P - m0 - m1;   // modes a = 0 .. lim along axis E
      const int base = m0 * st[t0] + (DIM > 2 ? m1 * st[t1] : 0);
      T v[N1], ev = T(0), od = T(0), tnl = T(0), tnu = T(0);
#pragma unroll
      for (int a = 0; a < N1; ++a) {
        if (a > lim) continue;
        const int gi = q2g_ct<DIM, P>(base + a * st[E]);
        v[a] = c[gi];
        if (a % 2) od += v[a] * tb.L1[a];
        else ev += v[a] * tb.L1[a];
        if (has_lo) tnl += cL[gi] * tb.L1[a];
        if (has_hi) tnu += cU[gi] * tb.L0[a];
      }
      const T tlo = ev - od, tup = ev + od;
      const bool c0 = m0 + m1 == 0;
      // halves of the jumps; a face without a neighbour has none, or that to
      // its Dirichlet value (a constant)
      const T jlo = T(0.5) * (has_lo ? tlo - tnl : (dlo ? tlo - (c0 ? glo : T(0)) : T(0)));
      const T jhi = T(0.5) * (has_hi ? tnu - tup : (dhi ? (c0 ? ghi : T(0)) - tup : T(0)));
#pragma unroll
      for (int a = 0; a < N1; ++a) {
        if (a > lim) continue;
        const int gi = q2g_ct<DIM, P>(base + a * st[E]);
        T d = T(0);   // strong derivative: int L_a L_b' = A[b][a], zero unless b > a, b - a odd
#pragma unroll
        for (int b = 0; b < N1; ++b)
          if (b > a && b <= lim && (b - a) % 2) d += tb.A[b][a] * v[b];
        const T wl = tb.L0[a] * jlo, wh = tb.L1[a] * jhi;
        gr[(size_t)(E * NBG + gi) * NT + cl] = (d + wl + wh) * ih;
        gr[(size_t)((DIM + E) * NBG + gi) * NT + cl] = (wl - wh) * ih;
      }
    }
}

template <int DIM, int P, typename T>
__global__ void __launch_bounds__(HjsTile<DIM>::N * (P + 2), hjp_min_blocks<DIM, P, T>()) hjp_kernel(const HJArgs<T> a) {
  using PL = HjpPlan<DIM, P, T>;
  constexpr int N1 = PL::N1, NQ = PL::NQ, NBG = PL::NBG, NQF = PL::NQF, NS = PL::NS, NMB = PL::NMB;
  constexpr int NV = 1 << DIM, NQV = ipow(NQ, DIM);
  using TL = HjsTile<DIM>;
  constexpr int TX = TL::X, TY = TL::Y, TZ = TL::Z, NT = TL::N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem_raw);
  MaxSlot<T>* cfl = reinterpret_cast<MaxSlot<T>*>(smem_raw + 16);
  double* sdt = reinterpret_cast<double*>(smem_raw + 24);   // the pseudo-step
  unsigned char* boxb = smem_raw + PL::OFF_BOX;
  T* gr = reinterpret_cast<T*>(smem_raw + PL::OFF_GR);    // [2][DIM][NBG][NT]
  T* stl = reinterpret_cast<T*>(smem_raw + PL::OFF_TAB);  // table slice [NS][NT]
  T* ub = stl;   // plane projections, over the entries of the thread's own plane
  const MeshArgs& m = a.m;
  const Tab1D<T>& tb = tab<T>(P);
  // part of the launch's tile
  const int sx = m.tile[0] / TX, sy = m.tile[1] / TY, sz = DIM > 2 ? m.tile[2] / TZ : 1;
  const int slot = (int)blockIdx.x / (sx * sy * sz), part = (int)blockIdx.x % (sx * sy * sz);
  const bool step = a.mode == kHJStep, fill = !step;
  const bool first = blockIdx.x == 0;
  double vd = 0.0;   // thread 0: the running CFL maximum before this step
  chain_wait();
  if (tile_inactive(m, slot)) {
    if (step && first && threadIdx.x == 0) hj_clock_step(a.clk, a.step, true, vd);
    return;
  }
  const int tile = m.tiles ? m.tiles[slot] : slot;
  int o[3];
  {
    int b = tile;
    o[0] = (b % m.ntile[0]) * m.tile[0] + (part % sx) * TX;
    b /= m.ntile[0];
    o[1] = (b % m.ntile[1]) * m.tile[1] + (part / sx) % sy * TY;
    o[2] = DIM > 2 ? (b / m.ntile[1]) * m.tile[2] + part / (sx * sy) * TZ : 0;
  }
  if (o[0] >= m.n[0] || o[1] >= m.n[1] || o[2] >= m.n[2]) return;   // a part past the mesh
  T* const tabp = a.stab + ((size_t)tile * (sx * sy * sz) + part) * NS * NT;
  if (threadIdx.x == 0) {
    mbar_init(bar, 32 + (step ? 1 : 0));
    *cfl = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (step) {
      mbar_arrive_expect_tx(bar, (unsigned)PL::TAB_BYTES);
      bulk_g2s(stl, tabp, (unsigned)PL::TAB_BYTES, bar);
      *sdt = hj_clock_step(a.clk, a.step, first, vd);
    }
  }
  if (threadIdx.x < 32) bulk_box_rows<DIM, TX, TY, TZ, NMB, PL::SLOT>(m, a.phi, boxb, o[0], o[1], o[2], bar);
  const int cl = (int)threadIdx.x % NT, k = (int)threadIdx.x / NT;   // cell, Gauss plane
  const int l[3] = {cl % TX, (cl / TX) % TY, DIM > 2 ? cl / (TX * TY) : 0};
  const int g[3] = {o[0] + l[0], o[1] + l[1], o[2] + l[2]};
  const bool valid = g[0] < m.n[0] && g[1] < m.n[1] && (DIM < 3 || g[2] < m.n[2]);
  const int gx0 = max(o[0] - 1, 0);
  auto cellp = [&](int lx, int ly, int lz) -> const T* {
    const int rr = (ly + 1) + PL::NBY * (DIM > 2 ? lz + 1 : 0);
    const unsigned rowcell = (unsigned)m.n[0] * (unsigned)((o[1] + ly) + m.n[1] * (DIM > 2 ? o[2] + lz : 0));
    const unsigned phase = ((rowcell + (unsigned)gx0) * (unsigned)NMB) & 15u;
    return reinterpret_cast<const T*>(boxb + (size_t)rr * PL::SLOT + phase + (o[0] + lx - gx0) * NMB);
  };
  const T hmin = T(m.min_diam);
  T Lk[N1], Dk[N1];   // this thread's Gauss plane
#pragma unroll
  for (int b = 0; b < N1; ++b) {
    Lk[b] = tb.Lq[b][k];
    Dk[b] = tb.Dq[b][k];
  }
  if (!mbar_wait(bar, 0u, 1 << 22)) {
    if (threadIdx.x == 0 && a.err) atomicOr(a.err, kErrCopyTimeout);
    mbar_wait(bar, 0u, 1 << 22);   // give copies in flight a last chance to land
  }

  // -------- (1) modal gradients: axis k of the thread's cell (whole warps per axis)
  if (valid) {
    if (k == 0) hjp_gradient<DIM, P, 0, T>(m, cellp, l, g, gr, cl);
    else if (k == 1) hjp_gradient<DIM, P, 1, T>(m, cellp, l, g, gr, cl);
    else if constexpr (DIM > 2) {
      if (k == 2) hjp_gradient<DIM, P, 2, T>(m, cellp, l, g, gr, cl);
    }
  }
  __syncthreads();

  const T* c = cellp(l[0], l[1], l[2]);
  T vmax = T(0);
  if (valid) {
    // -------- sign table of this cell's Gauss plane (phi == phi0)
    T cr[ipow(N1, DIM)];   // Q layout, only for the table
    if (fill) {
      const T ih[3] = {T(1.0 / m.h[0]), T(1.0 / m.h[1]), T(DIM > 2 ? 1.0 / m.h[2] : 1.0)};
      T* srow = tabp + cl;
#pragma unroll
      for (int q = 0; q < ipow(N1, DIM); ++q) cr[q] = q2g_ct<DIM, P>(q) >= 0 ? c[q2g_ct<DIM, P>(q)] : T(0);
      for (int j = 0; j < NQF; ++j) {
        const int qx = j % NQ, qy = DIM > 2 ? j / NQ : k;
        T p0 = T(0), g0[3] = {T(0), T(0), T(0)};
#pragma unroll
        for (int q = 0; q < ipow(N1, DIM); ++q) {
          if (q2g_ct<DIM, P>(q) < 0) continue;
          const int i0 = q % N1, i1 = (q / N1) % N1, i2 = q / (N1 * N1);
          const T lx = tb.Lq[i0][qx], ly = DIM > 2 ? tb.Lq[i1][qy] : Lk[i1], lz = DIM > 2 ? Lk[i2] : T(1);
          const T dy = DIM > 2 ? tb.Dq[i1][qy] : Dk[i1];
          p0 += cr[q] * (lx * ly * lz);
          g0[0] += cr[q] * (tb.Dq[i0][qx] * ly * lz);
          g0[1] += cr[q] * (lx * dy * lz);
          if constexpr (DIM > 2) g0[2] += cr[q] * (lx * ly * Dk[i2]);
        }
        T g2 = T(0);
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          const T gg = g0[d] * ih[d];
          g2 += gg * gg;
        }
        T w = tb.wq[qx] * tb.wq[k];
        if constexpr (DIM > 2) w *= tb.wq[qy];
        const T gn = sqrt(g2);
        srow[(size_t)(k * NQF + j) * NT] = w * (p0 / sqrt(p0 * p0 + hmin * hmin * gn * gn));
      }
    }

    // -------- vertex CFL estimate for the next pseudo-step: x-lines of
    // vertices ln = k, k + NQ, ... (corner bits vy = ln & 1, vz = ln >> 1)
#pragma unroll 1
    for (int ln = k; ln < NV / 2; ln += NQ) {
      const int vy = ln & 1, vz = ln >> 1;
      T Y[N1], Z[N1];
#pragma unroll
      for (int b = 0; b < N1; ++b) {
        Y[b] = vy ? tb.L1[b] : tb.L0[b];
        Z[b] = vz ? tb.L1[b] : tb.L0[b];
      }
      T S[2];
      if (fill) {
        T val[2], dphi[2][3];
        hjs_line<DIM, N1, T>(cr, tb, vy, vz, val, dphi);
#pragma unroll
        for (int vx = 0; vx < 2; ++vx) {
          T g2 = T(0);
#pragma unroll
          for (int d = 0; d < DIM; ++d) {
            const T gg = dphi[vx][d] * T(1.0 / m.h[d]);
            g2 += gg * gg;
          }
          const T gn = sqrt(g2);
          S[vx] = val[vx] / sqrt(val[vx] * val[vx] + hmin * hmin * gn * gn);
          tabp[(size_t)(NQV + vx + 2 * ln) * NT + cl] = S[vx];
        }
      } else {
        S[0] = stl[(size_t)(NQV + 2 * ln) * NT + cl];
        S[1] = stl[(size_t)(NQV + 2 * ln + 1) * NT + cl];
      }
      T lft[2][DIM], rgt[2][DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        T av[2], hd[2];
#pragma unroll
        for (int f = 0; f < 2; ++f) {
          T V[N1];
#pragma unroll
          for (int aa = 0; aa < N1; ++aa) {
            V[aa] = T(0);
#pragma unroll
            for (int b = 0; aa + b < N1; ++b) {
              T w = T(0);
#pragma unroll
              for (int cc = 0; cc < (DIM > 2 ? N1 : 1); ++cc) {
                if (aa + b + cc > P) continue;
                const T v = gr[(size_t)((f * DIM + d) * NBG + q2g_ct<DIM, P>(aa + N1 * (b + N1 * cc))) * NT + cl];
                w += cc == 0 ? v : v * Z[cc];
              }
              V[aa] += b == 0 ? w : w * Y[b];
            }
          }
          end_values<N1, 1, T>(tb, V, f ? hd[0] : av[0], f ? hd[1] : av[1]);
        }
#pragma unroll
        for (int vx = 0; vx < 2; ++vx) {
          lft[vx][d] = av[vx] + hd[vx];
          rgt[vx][d] = av[vx] - hd[vx];
        }
      }
      vmax = fmax(vmax, hjs_speed<DIM, T>(S[0], lft[0], rgt[0]));
      vmax = fmax(vmax, hjs_speed<DIM, T>(S[1], lft[1], rgt[1]));
    }
  }
  slot_max(cfl, vmax);
  if (!step) {
    __syncthreads();
    if (threadIdx.x == 0) atomic_max_pos(&a.clk->hj_vd[0], slot_value(cfl) / m.diam);
    return;
  }

  // -------- (2) H at this plane's Gauss points, projected onto the modes of
  // the other axes
  auto mode = [&](int f, int d, int q) -> T {
    return gr[(size_t)((f * DIM + d) * NBG + q2g_ct<DIM, P>(q)) * NT + cl];
  };
  auto hfun = [&](int j, const T* avg, T dif) -> T {
    T a2 = T(0);
#pragma unroll
    for (int d = 0; d < DIM; ++d) a2 += avg[d] * avg[d];
    const T S = stl[(size_t)(k * NQF + j) * NT + cl];   // w_q S
    return S * (sqrt(a2) - T(1)) + fabs(S) * dif;
  };
  if (valid) {
    constexpr int NF = DIM + 1;   // the means, then the sum of the half differences
    constexpr int NB = DIM > 2 ? N1 : 1;
    T V[NF][NB][N1];              // plane modes (b, a), a + b <= P
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int aa = 0; aa + b < N1; ++aa) {
#pragma unroll
        for (int f = 0; f < NF; ++f) V[f][b][aa] = T(0);
#pragma unroll
        for (int cc = 0; cc < N1; ++cc) {
          if (aa + b + cc > P) continue;
          const int q = DIM > 2 ? aa + N1 * (b + N1 * cc) : aa + N1 * cc;
          T hs = T(0);
#pragma unroll
          for (int d = 0; d < DIM; ++d) {
            const T v = mode(0, d, q);
            V[d][b][aa] += cc == 0 ? v : v * Lk[cc];
            hs += mode(1, d, q);
          }
          V[DIM][b][aa] += cc == 0 ? hs : hs * Lk[cc];
        }
      }
    T U[NB][N1];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int aa = 0; aa < N1; ++aa) U[b][aa] = T(0);
#pragma unroll
    for (int qy = 0; qy < (DIM > 2 ? NQ : 1); ++qy) {
      T v[NF][NQ], f[NQ], X[N1];
#pragma unroll
      for (int i = 0; i < NF; ++i) {
        T x[N1];
#pragma unroll
        for (int aa = 0; aa < N1; ++aa) {
          x[aa] = V[i][0][aa];
          if constexpr (DIM > 2) {
#pragma unroll
            for (int b = 1; b < NB; ++b)
              if (aa + b < N1) x[aa] += V[i][b][aa] * tb.Lq[b][qy];
          }
        }
        gauss_values<N1, NQ, 1, T>(tb, x, v[i]);
      }
#pragma unroll
      for (int qx = 0; qx < NQ; ++qx) {
        T avg[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) avg[d] = v[d][qx];
        f[qx] = hfun(DIM > 2 ? qx + NQ * qy : qx, avg, v[DIM][qx]);
      }
#pragma unroll
      for (int aa = 0; aa < N1; ++aa) X[aa] = T(0);
      gauss_project<N1, NQ, 1, T>(tb, f, X);
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int aa = 0; aa + b < N1; ++aa) {
          if (DIM > 2 && b > 0) U[b][aa] += X[aa] * tb.Lq[b][qy];
          else U[b][aa] += X[aa];
        }
    }
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int aa = 0; aa + b < N1; ++aa) ub[(size_t)(k * NQF + aa + N1 * b) * NT + cl] = U[b][aa];
  }
  __syncthreads();   // planes done: the gradients become the store staging
  if (threadIdx.x == 0) {   // the running maximum of the next step (the first block has put this one's)
    const double bm = slot_value(cfl) / m.diam;
    if (bm > vd) atomic_max_pos(&a.clk->hj_vd[(a.step.k + 1) % 3], bm);
  }
  const T dt = T(*sdt);

  // -------- (3) columns (a, b) of modes, dealt to the threads of a cell:
  // project over the planes, update, stage
  T* sb = gr;   // [NT][NBG]
  if (valid) {
    const long long cell = (long long)g[0] + (long long)m.n[0] * (g[1] + (long long)m.n[1] * g[2]);
    int turn = 0;
#pragma unroll
    for (int b = 0; b < (DIM > 2 ? N1 : 1); ++b)
#pragma unroll
      for (int aa = 0; aa + b < N1; ++aa) {
        if (turn++ % NQ != k) continue;
        T f[NQ], R[N1];
#pragma unroll
        for (int kk = 0; kk < NQ; ++kk) f[kk] = ub[(size_t)(kk * NQF + aa + N1 * b) * NT + cl];
#pragma unroll
        for (int cc = 0; cc < N1; ++cc) R[cc] = T(0);
        gauss_project<N1, NQ, 1, T>(tb, f, R);
#pragma unroll
        for (int cc = 0; cc < N1; ++cc) {
          if (aa + b + cc > P) continue;
          const int gi = q2g_ct<DIM, P>(DIM > 2 ? aa + N1 * (b + N1 * cc) : aa + N1 * cc);
          T r = -R[cc];
          if (a.rdiff) r += a.rdiff[cell * NBG + gi];
          sb[(size_t)cl * NBG + gi] = hj_combine<T>(a.rk, c[gi], r, dt);
        }
      }
  }
  __syncthreads();
  chain_release();
  store_cells<DIM, TX, TY, TZ, NBG, T>(m, sb, a.out, o[0], o[1], o[2]);
}

}  // namespace flsp
