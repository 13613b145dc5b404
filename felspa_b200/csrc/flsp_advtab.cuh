// flsp_advtab.cuh — DG advection stage kernel for a velocity given at the
// quadrature points (sums of separable terms; the velocity of a coupled FE
// simulator; every problem of a batch).
//
// The operator of AdvectAssembler (include/felspa/pde/src/
// advection.implement.h:617-744) on QGauss(p+2) cell and face rules.  One
// CTA serves an HjsTile of cells with NQ threads per cell; its halo box
// arrives by bulk copies.
//   (1) every face of the tile is one work item: the upwind trace at the
//       face's points times the table, projected onto the face modes, into
//       the face's slot; only where the velocity changes sign over the face
//       are both traces interpolated;
//   (2) thread k of a cell sums Gauss plane k of the last axis: phi at the
//       plane's points (by parity), the three products with the table,
//       their projections on the other axes, in shared memory;
//   (3) the columns of modes along the last axis are dealt to the threads of
//       a cell: projection over the planes, the lifted faces, and the RK
//       combination in the coalesced store.
// Table (VelTabLayout): per tile, w_q u_d / h_d at the cells' points
// [comp][point][cell], then w_q u_E / h_E at the tile's faces [point][slot]
// (faces of two tiles twice), so every load of a warp is contiguous and the
// weights cost nothing.
// In 2D the tile's slice comes to shared memory by one bulk copy, issued before
// the kernel before has finished; in 3D (64 KB at Q2 FP32) it would cost the
// CTAs that hide its latency, and the threads read it from L2 or HBM.
// What bounds it: in 3D the table, 1.06 KB per cell and stage (Q2 FP32), and
// latency; in 2D latency.  Against one thread per cell with every point summed
// from all modes (128 registers, 16 warps per SM): 48^3 Q2 FP32 131 -> 43 us a
// stage, 256^2 11.6 -> 8.2.  A batched stage of 16 degree-3 problems (248,000
// cells, FP32), where the long-scoreboard stall was the largest: 85 us with the
// table read by the threads, 20 warps per SM; see advtab_min_blocks.
#pragma once
#include "flsp_hjs.cuh"
#include "flsp_stage.cuh"

namespace flsp {

template <typename T>
struct AdvTabArgs {
  MeshArgs m;                    // m.tile: HjsTile
  const T* __restrict__ tab;     // VelTabLayout
  const T* __restrict__ phi_s;   // stage input (read with halo)
  const T* __restrict__ phi_n;   // phi^n for the combinations
  T* __restrict__ out;
  const AdvStep* step;           // the substep (null: explicit)
  int stage;                     // index into step->ct
  int combine;                   // CombineMode
  double ct_explicit, dt_explicit;   // when step == nullptr
  int* err;                      // the problem's error word
};

template <int DIM, int P, bool PB, typename T>
struct AdvTabPlan {
  using TL = HjsTile<DIM>;
  using LY = VelTabLayout<DIM>;
  static constexpr int N1 = P + 1, NQ = P + 2, NQF = ipow(NQ, DIM - 1), NU = ipow(N1, DIM - 1);
  static constexpr int NBG = PB ? (DIM == 2 ? (P + 1) * (P + 2) / 2 : (P + 1) * (P + 2) * (P + 3) / 6) : ipow(N1, DIM);
  static constexpr int NF = PB ? (DIM == 2 ? N1 : (P + 1) * (P + 2) / 2) : ipow(N1, DIM - 1);   // face modes
  static constexpr int NROWS = (TL::Y + 2) * (DIM > 2 ? TL::Z + 2 : 1);
  static constexpr int NMB = NBG * (int)sizeof(T);
  static constexpr int SLOT = (((TL::X + 2) * NMB + 30) + 15) / 16 * 16;
  static constexpr size_t OFF_BOX = 16;
  static constexpr size_t OFF_FL = OFF_BOX + (size_t)NROWS * SLOT;                          // [NF][NFT]
  static constexpr size_t OFF_UB = (OFF_FL + (size_t)NF * LY::NFT * sizeof(T) + 15) / 16 * 16;   // [NQ][2][NU][N]
  static constexpr size_t OFF_SB = OFF_UB + (size_t)NQ * 2 * NU * TL::N * sizeof(T);        // [N][NBG]
  static constexpr size_t OFF_TB = (OFF_SB + (size_t)TL::N * NBG * sizeof(T) + 15) / 16 * 16;
  // 2D: the tile's table slice (15.7 KB at Q3 FP32) is brought into shared memory
  static constexpr bool STAGED = DIM == 2;
  static constexpr unsigned TBYTES = LY::entries(NQ) * sizeof(T);
  // 3D FP64, one CTA per SM: the slice (129 KB at Q2) asked into the L2 ahead, 48^3
  // Q2 110.8 -> 102.9 us a stage, 32^3 31.1 -> 31.0; with FP32's three CTAs it
  // takes their bandwidth (48^3 42.2 -> 44.8)
  static constexpr bool PREFETCH = DIM == 3 && sizeof(T) == 8;
  static_assert(TBYTES % 16 == 0, "bulk copies move 16-byte pieces");
  static constexpr size_t BYTES = OFF_TB + (STAGED ? TBYTES : 0);
};

// CTAs per SM the registers are held to.  3D FP32: three (24 warps).  2D: as
// many as cost no spills worth the name (P = 3 FP32: 64 -> 48 registers with 8
// bytes spilled, 20 -> 40 warps per SM; P = 2: 52 -> 40, 32 -> 48 warps; FP64
// P = 3: 106 -> 96, 10 -> 20 warps, P = 2: 76 -> 64, 24 -> 32 warps): with the
// table in shared memory 48 uneven problems of degrees 1..3 took 22.4 ms without
// the bounds, 20.7 with them, in FP64 (20 steps) 26.8 and 23.3.
template <int DIM, int P, typename T>
constexpr int advtab_min_blocks() {
  if (DIM == 3) return sizeof(T) == 4 ? 3 : 1;
  return sizeof(T) == 4 ? (P == 3 ? 4 : P == 2 ? 6 : 8) : (P == 3 ? 2 : P == 2 ? 4 : 1);
}

// one tile of a stage; every thread of the block calls it
template <int DIM, int P, bool PB, typename T>
__device__ __forceinline__ void adv_tab_tile(const AdvTabArgs<T>& a, int tile) {
  using PL = AdvTabPlan<DIM, P, PB, T>;
  using LY = VelTabLayout<DIM>;
  using TL = HjsTile<DIM>;
  constexpr int N1 = PL::N1, NQ = PL::NQ, NQF = PL::NQF, NU = PL::NU, NBG = PL::NBG, NMB = PL::NMB;
  constexpr int TX = TL::X, TY = TL::Y, TZ = TL::Z, NT = TL::N, NQD = ipow(NQ, DIM);
  constexpr int BY = TY + 2, NB1 = DIM > 2 ? N1 : 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem_raw);
  unsigned char* boxb = smem_raw + PL::OFF_BOX;
  T* fl = reinterpret_cast<T*>(smem_raw + PL::OFF_FL);
  T* ub = reinterpret_cast<T*>(smem_raw + PL::OFF_UB);
  T* sb = reinterpret_cast<T*>(smem_raw + PL::OFF_SB);
  const MeshArgs& m = a.m;
  const Tab1D<T>& tb = tab<T>(P);
  int o[3];
  {
    int b = tile;
    o[0] = (b % m.ntile[0]) * TX;
    b /= m.ntile[0];
    o[1] = (b % m.ntile[1]) * TY;
    o[2] = DIM > 2 ? (b / m.ntile[1]) * TZ : 0;
  }
  if (threadIdx.x == 0) mbar_init(bar, 32 + (PL::STAGED ? 1 : 0));
  __syncthreads();
  // the table does not change during a run; the field does
  const T* tabg = a.tab + (size_t)tile * LY::template entries<NQ>();
  if (PL::STAGED && threadIdx.x == 0) {
    mbar_arrive_expect_tx(bar, PL::TBYTES);
    bulk_g2s(smem_raw + PL::OFF_TB, tabg, PL::TBYTES, bar);
  }
  if (PL::PREFETCH && threadIdx.x == 0) bulk_prefetch_l2(tabg, PL::TBYTES);
  chain_wait();
  if (threadIdx.x < 32) bulk_box_rows<DIM, TX, TY, TZ, NMB, PL::SLOT>(m, a.phi_s, boxb, o[0], o[1], o[2], bar);
  const int cl = (int)threadIdx.x % NT, k = (int)threadIdx.x / NT;   // cell, Gauss plane
  const int l[3] = {cl % TX, (cl / TX) % TY, DIM > 2 ? cl / (TX * TY) : 0};
  const int g[3] = {o[0] + l[0], o[1] + l[1], o[2] + l[2]};
  const bool valid = g[0] < m.n[0] && g[1] < m.n[1] && (DIM < 3 || g[2] < m.n[2]);
  const int gx0 = max(o[0] - 1, 0);
  auto cellp = [&](int lx, int ly, int lz) -> const T* {
    const int rr = (ly + 1) + BY * (DIM > 2 ? lz + 1 : 0);
    const unsigned rowcell = (unsigned)m.n[0] * (unsigned)((o[1] + ly) + m.n[1] * (DIM > 2 ? o[2] + lz : 0));
    const unsigned phase = ((rowcell + (unsigned)gx0) * (unsigned)NMB) & 15u;
    return reinterpret_cast<const T*>(boxb + (size_t)rr * PL::SLOT + phase + (o[0] + lx - gx0) * NMB);
  };
  const T ct = a.step ? T(a.step->ct[a.stage]) : T(a.ct_explicit);
  const T dt = a.step ? T(a.step->dt) : T(a.dt_explicit);
  const bool active = a.step ? (a.step->active != 0) : true;
  const T* tabc = PL::STAGED ? reinterpret_cast<const T*>(smem_raw + PL::OFF_TB) : tabg;   // the tile's cells
  const T* tabf = tabc + (size_t)DIM * NQD * NT;                                           // and faces
  auto entry = [](const T* p) -> T {
    if constexpr (PL::STAGED) return *p;
    else return __ldg(p);
  };
  T Lk[N1];
#pragma unroll
  for (int b = 0; b < N1; ++b) Lk[b] = tb.Lq[b][k];
  if (!mbar_wait(bar, 0u, 1 << 22)) {
    if (threadIdx.x == 0 && a.err) atomicOr(a.err, kErrCopyTimeout);
    mbar_wait(bar, 0u, 1 << 22);   // give copies in flight a last chance to land
  }

  // ===== (1) face fluxes
  auto face_item = [&](auto EC, int r) {
    constexpr int E = decltype(EC)::value;
    constexpr int EX = TX + (E == 0), EY = TY + (E == 1);
    const int lx = r % EX, ly = (r / EX) % EY, lz = DIM > 2 ? r / (EX * EY) : 0;
    const int gc[3] = {o[0] + lx, o[1] + ly, o[2] + lz};
    if ((E != 0 && gc[0] >= m.n[0]) || (E != 1 && gc[1] >= m.n[1]) || (DIM > 2 && E != 2 && gc[2] >= m.n[2])) return;
    const int gE = gc[E];
    const bool has_m = gE >= 1 && gE - 1 < m.n[E], has_p = gE < m.n[E];
    if (!has_m && !has_p) return;
    T u[NQF];
    const T* uf = tabf + LY::off(E) + r;
#pragma unroll
    for (int q = 0; q < NQF; ++q) u[q] = entry(uf + (size_t)q * LY::NFT);
    // which side is upwind at the points (the time factor's sign with it)
    bool some_m = false, some_p = false;
#pragma unroll
    for (int q = 0; q < NQF; ++q) {
      const bool up = u[q] * ct > T(0);
      some_m = some_m || up;
      some_p = some_p || !up;
    }
    T gd = T(0);
    bool dir = false;
    if (!has_m) dir = bc_dirichlet<DIM>(m, E, 0, gc, gd);
    else if (!has_p) {
      const int gl[3] = {gc[0] - (E == 0), gc[1] - (E == 1), gc[2] - (E == 2)};
      dir = bc_dirichlet<DIM>(m, E, 1, gl, gd);
    }
    // the trace from below (side 0) or above (1): a missing one is the
    // face's Dirichlet value, or without one the other side's (zero Neumann)
    auto trace = [&](int side, T* tr) {
      const bool have = side == 0 ? has_m : has_p;
      if (!have && dir) {
#pragma unroll
        for (int f = 0; f < PL::NF; ++f) tr[f] = f == 0 ? gd : T(0);
        return;
      }
      const bool lower = have ? side == 0 : side != 0;
      face_trace_ct<DIM, P, PB, E, T>(lower ? cellp(lx - (E == 0), ly - (E == 1), lz - (E == 2)) : cellp(lx, ly, lz),
                                      lower ? tb.L1 : tb.L0, tr);
    };
    auto nodal = [&](const T* tr, T* v) {
      if constexpr (DIM == 2) {
        gauss_values<N1, NQ, 1, T>(tb, tr, v);
      } else {
#pragma unroll
        for (int q1 = 0; q1 < NQ; ++q1) {
          T x[N1];
#pragma unroll
          for (int m0 = 0; m0 < N1; ++m0) {
            x[m0] = tr[face_index<P, PB>(m0, 0)];
#pragma unroll
            for (int m1 = 1; m1 < N1; ++m1)
              if (mode_in<P, PB>(m0 + m1)) x[m0] += tr[face_index<P, PB>(m0, m1)] * tb.Lq[m1][q1];
          }
          gauss_values<N1, NQ, 1, T>(tb, x, v + NQ * q1);
        }
      }
    };
    T tr[PL::NF], v[NQF];
    trace(some_m ? 0 : 1, tr);
    nodal(tr, v);
    if (some_m && some_p) {
      T w[NQF];
      trace(1, tr);
      nodal(tr, w);
#pragma unroll
      for (int q = 0; q < NQF; ++q) v[q] = u[q] * ct > T(0) ? v[q] : w[q];
    }
#pragma unroll
    for (int q = 0; q < NQF; ++q) v[q] *= u[q];
    T* fs = fl + LY::off(E) + r;
    if constexpr (DIM == 2) {
      T X[N1];
#pragma unroll
      for (int m0 = 0; m0 < N1; ++m0) X[m0] = T(0);
      gauss_project<N1, NQ, 1, T>(tb, v, X);
#pragma unroll
      for (int m0 = 0; m0 < N1; ++m0) fs[(size_t)m0 * LY::NFT] = ct * X[m0];
    } else {
      T F[N1][N1];   // [m1][m0]
#pragma unroll
      for (int m1 = 0; m1 < N1; ++m1)
#pragma unroll
        for (int m0 = 0; m0 < N1; ++m0) F[m1][m0] = T(0);
#pragma unroll
      for (int q1 = 0; q1 < NQ; ++q1) {
        T X[N1];
#pragma unroll
        for (int m0 = 0; m0 < N1; ++m0) X[m0] = T(0);
        gauss_project<N1, NQ, 1, T>(tb, v + NQ * q1, X);
#pragma unroll
        for (int m1 = 0; m1 < N1; ++m1)
#pragma unroll
          for (int m0 = 0; m0 < N1; ++m0)
            if (mode_in<P, PB>(m0 + m1)) F[m1][m0] += m1 == 0 ? X[m0] : X[m0] * tb.Lq[m1][q1];
      }
#pragma unroll
      for (int m1 = 0; m1 < N1; ++m1)
#pragma unroll
        for (int m0 = 0; m0 < N1; ++m0)
          if (mode_in<P, PB>(m0 + m1)) fs[(size_t)face_index<P, PB>(m0, m1) * LY::NFT] = ct * F[m1][m0];
    }
  };
  if (active) {
    // each axis' items start on a warp boundary: no warp runs two axes' code
    constexpr int W0 = (LY::S0 + 31) / 32 * 32, W1 = W0 + (LY::S1 + 31) / 32 * 32;
    for (int i = threadIdx.x; i < W1 + LY::S2; i += NT * NQ) {
      if (i < W0) {
        if (i < LY::S0) face_item(std::integral_constant<int, 0>(), i);
      } else if (i < W1) {
        if (i < W0 + LY::S1) face_item(std::integral_constant<int, 1>(), i - W0);
      } else if constexpr (DIM > 2) {
        face_item(std::integral_constant<int, 2>(), i - W1);
      }
    }
  }

  // ===== (2) the cell's Gauss plane k
  const bool work = valid && active;
  if (work) {
    const T* c = cellp(l[0], l[1], l[2]);
    T V[NB1][N1];   // (b, a): the plane's modes of the other axes
#pragma unroll
    for (int b = 0; b < NB1; ++b)
#pragma unroll
      for (int aa = 0; aa < N1; ++aa) {
        if (!mode_in<P, PB>(aa + b)) continue;
        T s = T(0);
#pragma unroll
        for (int cc = 0; cc < N1; ++cc) {
          if (!mode_in<P, PB>(aa + b + cc)) continue;
          const T x = c[cell_index<DIM, P, PB>(DIM > 2 ? aa + N1 * (b + N1 * cc) : aa + N1 * cc)];
          s += cc == 0 ? x : x * Lk[cc];
        }
        V[b][aa] = s;
      }
    T Uv[NB1][N1], Ud[NB1][N1];   // projections: with L along the last axis, with its derivative
#pragma unroll
    for (int b = 0; b < NB1; ++b)
#pragma unroll
      for (int aa = 0; aa < N1; ++aa) Uv[b][aa] = Ud[b][aa] = T(0);
#pragma unroll
    for (int qy = 0; qy < (DIM > 2 ? NQ : 1); ++qy) {
      T x[N1], ph[NQ], f0[NQ], f1[NQ], f2[NQ];
      const T* tq = tabc + (size_t)((DIM > 2 ? NQ * qy + NQF * k : NQ * k)) * NT + cl;
#pragma unroll
      for (int qx = 0; qx < NQ; ++qx) {
        f0[qx] = entry(tq + (size_t)qx * NT);
        f1[qx] = entry(tq + (size_t)(NQD + qx) * NT);
        if constexpr (DIM > 2) f2[qx] = entry(tq + (size_t)(2 * NQD + qx) * NT);
      }
#pragma unroll
      for (int aa = 0; aa < N1; ++aa) {
        x[aa] = V[0][aa];
#pragma unroll
        for (int b = 1; b < NB1; ++b)
          if (mode_in<P, PB>(aa + b)) x[aa] += V[b][aa] * tb.Lq[b][qy];
      }
      gauss_values<N1, NQ, 1, T>(tb, x, ph);
#pragma unroll
      for (int qx = 0; qx < NQ; ++qx) {
        f0[qx] *= ph[qx];
        f1[qx] *= ph[qx];
        if constexpr (DIM > 2) f2[qx] *= ph[qx];
      }
      T X0[N1], X1[N1], X2[N1];
#pragma unroll
      for (int aa = 0; aa < N1; ++aa) X0[aa] = X1[aa] = X2[aa] = T(0);
      gauss_project_derivative<N1, NQ, T>(tb, f0, X0);
      gauss_project<N1, NQ, 1, T>(tb, f1, X1);
      if constexpr (DIM == 2) {
#pragma unroll
        for (int aa = 0; aa < N1; ++aa) {
          Uv[0][aa] = X0[aa];
          Ud[0][aa] = X1[aa];
        }
      } else {
        gauss_project<N1, NQ, 1, T>(tb, f2, X2);
#pragma unroll
        for (int aa = 0; aa < N1; ++aa) {
          if (aa > 0) Uv[0][aa] += X0[aa];
          Ud[0][aa] += X2[aa];
#pragma unroll
          for (int b = 1; b < N1; ++b) {
            if (!mode_in<P, PB>(aa + b)) continue;
            if (aa > 0) Uv[b][aa] += X0[aa] * tb.Lq[b][qy];
            Uv[b][aa] += X1[aa] * tb.Dq[b][qy];
            Ud[b][aa] += X2[aa] * tb.Lq[b][qy];
          }
        }
      }
    }
#pragma unroll
    for (int b = 0; b < NB1; ++b)
#pragma unroll
      for (int aa = 0; aa < N1; ++aa) {
        if (!mode_in<P, PB>(aa + b)) continue;
        ub[(size_t)((2 * k) * NU + aa + N1 * b) * NT + cl] = Uv[b][aa];
        ub[(size_t)((2 * k + 1) * NU + aa + N1 * b) * NT + cl] = Ud[b][aa];
      }
  }
  __syncthreads();

  // ===== (3) columns (a, b) of modes along the last axis
  if (work) {
    constexpr int SY = TX, SZ = TX * TY;   // the upper face's slot beside the lower one's
    const int s0 = LY::off(0) + l[0] + (TX + 1) * (l[1] + TY * l[2]);
    const int s1 = LY::off(1) + l[0] + TX * (l[1] + (TY + 1) * l[2]);
    const int s2 = LY::off(2) + l[0] + TX * (l[1] + TY * l[2]);
    // even modes along the face's axis take L_a(1) times lower minus upper
    // flux, odd ones minus L_a(1) times their sum
    auto lift = [&](int slot, int up, int f, int md) -> T {
      const T lo = fl[(size_t)f * LY::NFT + slot], hi = fl[(size_t)f * LY::NFT + slot + up];
      return md % 2 ? -tb.L1[md] * (lo + hi) : (md == 0 ? lo - hi : tb.L1[md] * (lo - hi));
    };
    int turn = 0;
#pragma unroll
    for (int b = 0; b < NB1; ++b)
#pragma unroll
      for (int aa = 0; aa < N1; ++aa) {
        if (!mode_in<P, PB>(aa + b)) continue;
        if (turn++ % NQ != k) continue;
        T fv[NQ], fd[NQ], R[N1];
#pragma unroll
        for (int kk = 0; kk < NQ; ++kk) {
          fv[kk] = ub[(size_t)((2 * kk) * NU + aa + N1 * b) * NT + cl];
          fd[kk] = ub[(size_t)((2 * kk + 1) * NU + aa + N1 * b) * NT + cl];
        }
#pragma unroll
        for (int cc = 0; cc < N1; ++cc) R[cc] = T(0);
        gauss_project<N1, NQ, 1, T>(tb, fv, R);
        gauss_project_derivative<N1, NQ, T>(tb, fd, R);
#pragma unroll
        for (int cc = 0; cc < N1; ++cc) {
          if (!mode_in<P, PB>(aa + b + cc)) continue;
          T r = ct * R[cc];
          if constexpr (DIM == 2) {
            r += lift(s0, 1, cc, aa);
            r += lift(s1, SY, aa, cc);
          } else {
            r += lift(s0, 1, face_index<P, PB>(b, cc), aa);
            r += lift(s1, SY, face_index<P, PB>(aa, cc), b);
            r += lift(s2, SZ, face_index<P, PB>(aa, b), cc);
          }
          sb[(size_t)cl * NBG + cell_index<DIM, P, PB>(DIM > 2 ? aa + N1 * (b + N1 * cc) : aa + N1 * cc)] = r;
        }
      }
  }
  __syncthreads();
  chain_release();
  combine_rows<DIM, TX, TY, TZ, NBG, NT * NQ / 32, T>(m, cellp, sb, a.phi_n, a.out, a.combine, dt, active, o[0], o[1],
                                                      o[2]);
}

template <int DIM, int P, bool PB, typename T>
__global__ void __launch_bounds__(HjsTile<DIM>::N * (P + 2), advtab_min_blocks<DIM, P, T>())
    adv_tab_kernel(const AdvTabArgs<T> a) {
  adv_tab_tile<DIM, P, PB, T>(a, (int)blockIdx.x);
}

}  // namespace flsp
