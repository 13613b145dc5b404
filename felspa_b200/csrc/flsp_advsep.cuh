// flsp_advsep.cuh — DG advection stage kernel for a separable velocity.
//
// Same operator as adv_stage_kernel (AdvectAssembler cell, face and
// boundary terms, include/felspa/pde/src/advection.implement.h:617-744,
// on QGauss(p+2) cell and face rules), evaluated for a velocity whose
// component d is ONE separable term u_d = c(t) g_d0(x) g_d1(y) g_d2(z)
// (coefficient folded into g_d0).  The tensor-product Gauss sum of a
// separable integrand is the product of 1D Gauss sums, so the quadrature
// sums factor exactly into per-axis operators (no approximation):
//
//   cell, component d:  R += c(t)/h_d (A_d0 (x) A_d1 (x) A_d2) phi
//     A_de[a][b] = sum_q w_q g_de(x_q) L_b(x_q) (e == d ? L_a'(x_q) : L_a(x_q))
//   face normal E (flux in +e_E, traces T- of the lower, T+ of the upper cell):
//     u_E phi_upwind = u_E (T- + T+)/2 + |u_E| (T- - T+)/2
//     F = c g_EE (A_Et0 (x) A_Et1) (T- + T+)/2
//       + |c g_EE| (B_Et0 (x) B_Et1) (T- - T+)/2,   B_de = A_de with |g_de|
//   (|u_E| = |c g_EE| |g_Et0| |g_Et1| is separable too; on the domain
//   boundary the missing trace is the Dirichlet value of the face, or the
//   own trace (zero-Neumann inflow), when the second term vanishes);
//   R- -= L(1) F / h_E, R+ += L(0) F / h_E.
//
// The CTA's halo box (one bulk copy per row of cells, each row keeping its
// 16-byte phase from HBM so that 27-value cells need no splitting) and its
// operator rows arrive by TMA bulk copies on one mbarrier.  Every face of
// the tile is then one work item of a single routine (runtime axis), its
// flux kept in shared memory; each cell adds its cell term and lifts its
// faces' fluxes; the RK combination is fused into a coalesced store that
// prefetches phi^n into registers (float4 rows where FP32 alignment
// allows).  Tile shapes are compile-time.
//
// The per-axis operators are tabulated once per velocity on the host in
// FP64 (optab, one row per component d, axis e and cell index i:
// A_de then, at element BOFF, B_de, or for e == d A_dd then g_dd(0),
// g_dd(1)).  Per cell that
// is ~1.5k FMA for Q2 in 3D instead of the ~4k of point-wise quadrature.
#pragma once
#include <type_traits>

#include "flsp_stage.cuh"

namespace flsp {

// row layout: two (P+1)^2 blocks, each with one spare element and padded to
// a multiple of 4 elements so that every block starts on a 16-byte boundary
// (FP32 and FP64).  The spare element of the A block of a row with e != d
// holds the sign of g_de over the cell's Gauss points (+1 / -1 if it keeps
// one sign, 0 if it changes sign).
template <int P>
__host__ __device__ constexpr int sep_boff() {
  return (((P + 1) * (P + 1) + 1 + 3) / 4) * 4;
}
template <int P>
__host__ __device__ constexpr int sep_opw() {
  return 2 * sep_boff<P>();
}

template <typename T>
struct AdvSepArgs {
  MeshArgs m;
  const T* __restrict__ optab;   // [(d*3 + e) * nmax + i][OPW]
  int nmax;                      // row stride per (d, e): >= n[e] + kOpRowPad (a tile's
                                 // bulk copy of its rows never leaves the table)
  int* err;                      // the problem's error word
  const T* __restrict__ phi_s;
  const T* __restrict__ phi_n;
  T* __restrict__ out;
  const AdvStep* step;           // the substep (null: explicit)
  int stage;                     // index into step->ct
  int combine;
  double ct_explicit;
  double dt_explicit;
};

// Shared-memory plan of the separable stage kernel for a compile-time tile
// TX x TY x TZ (TZ = 1 in 2D): mbarrier | halo box rows | operator rows |
// face fluxes (reused for the tile's R).  Box rows: (TY+2)(TZ+2) slots of
// SLOT bytes, each holding the row's cells x in [ox-1, ox+TX] from the
// 16-byte-aligned address at or below the first one.
template <int DIM, int P, bool PB, int TX, int TY, int TZ, typename T>
struct SepPlan {
  static constexpr int N1 = P + 1, NM = ipow(N1, DIM);
  static constexpr int NF = PB ? (DIM == 2 ? N1 : (P + 1) * (P + 2) / 2) : ipow(N1, DIM - 1);   // face modes
  static constexpr int NBG = PB ? (DIM == 2 ? (P + 1) * (P + 2) / 2 : (P + 1) * (P + 2) * (P + 3) / 6) : NM;
  static constexpr int OPW = sep_opw<P>();
  static constexpr int NT = TX * TY * TZ;
  static constexpr int BY = DIM > 1 ? TY + 2 : 1, BZ = DIM > 2 ? TZ + 2 : 1;
  static constexpr int NROWS = BY * BZ;
  static constexpr int NMB = NBG * (int)sizeof(T);           // bytes per cell in HBM
  static constexpr int SLOT = (((TX + 2) * NMB + 30) + 15) / 16 * 16;
  static constexpr int SPAN = TX + TY + (DIM > 2 ? TZ : 0);
  static constexpr int SL0 = (TX + 1) * TY * TZ, SL1 = TX * (TY + 1) * TZ,
                       SL2 = DIM > 2 ? TX * TY * (TZ + 1) : 0;
  static constexpr int FLN = NF * (SL0 + SL1 + SL2);
  static constexpr int FLE = FLN > NT * NBG ? FLN : NT * NBG;  // elements
  static constexpr size_t OFF_BOX = 16;
  static constexpr size_t OFF_OPS = OFF_BOX + (size_t)NROWS * SLOT;
  static constexpr size_t OFF_FL = OFF_OPS + (size_t)DIM * SPAN * OPW * sizeof(T);
  static constexpr size_t BYTES = OFF_FL + (size_t)FLE * sizeof(T);
};

// N1 x N1 operator block from shared memory (16-byte aligned)
template <int N1, typename T>
__device__ __forceinline__ void load_op(const T* __restrict__ src, T (&M)[N1][N1]) {
  constexpr int NN = N1 * N1;
  T v[NN];
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int k = 0; k + 4 <= NN; k += 4) {
      const float4 f = *reinterpret_cast<const float4*>(src + k);
      v[k] = f.x; v[k + 1] = f.y; v[k + 2] = f.z; v[k + 3] = f.w;
    }
#pragma unroll
    for (int k = (NN / 4) * 4; k < NN; ++k) v[k] = src[k];
  } else {
#pragma unroll
    for (int k = 0; k + 2 <= NN; k += 2) {
      const double2 f = *reinterpret_cast<const double2*>(src + k);
      v[k] = f.x; v[k + 1] = f.y;
    }
#pragma unroll
    for (int k = (NN / 2) * 2; k < NN; ++k) v[k] = src[k];
  }
#pragma unroll
  for (int a = 0; a < N1; ++a)
#pragma unroll
    for (int b = 0; b < N1; ++b) M[a][b] = v[a * N1 + b];
}

// F = s1 (A0 (x) A1) S + s2 (B0 (x) B1) D on the face modes in use;
// in 2D only A0 / B0; the B blocks start BOFF elements after the A blocks
template <int DIM, int P, bool PB, int BOFF, typename T>
__device__ __forceinline__ void face_apply(const T* __restrict__ rowA0, const T* __restrict__ rowA1,
                                           const T* S, const T* D, T s1, T s2, bool upwind, T* F) {
  constexpr int N1 = P + 1, NH = DIM > 2 ? N1 : 1;
  auto apply = [&](const T* r0, const T* r1, const T* x, T s, bool acc_into) {
    T M0[N1][N1], u[N1][NH];   // u: [a0][b1]
    load_op<N1, T>(r0, M0);
#pragma unroll
    for (int a0 = 0; a0 < N1; ++a0)
#pragma unroll
      for (int b1 = 0; b1 < NH; ++b1) {
        T acc = T(0);
#pragma unroll
        for (int b0 = 0; b0 < N1; ++b0)
          if (mode_in<P, PB>(b0 + b1)) acc += M0[a0][b0] * x[face_index<P, PB>(b0, b1)];
        u[a0][b1] = acc;
      }
    T M1[N1][N1];
    if constexpr (DIM > 2) load_op<N1, T>(r1, M1);
#pragma unroll
    for (int a1 = 0; a1 < NH; ++a1)
#pragma unroll
      for (int a0 = 0; a0 < N1; ++a0) {
        if (!mode_in<P, PB>(a0 + a1)) continue;
        T acc = T(0);
        if constexpr (DIM > 2) {
#pragma unroll
          for (int b1 = 0; b1 < N1; ++b1) acc += M1[a1][b1] * u[a0][b1];
        } else {
          acc = u[a0][0];
        }
        const int f = face_index<P, PB>(a0, a1);
        F[f] = acc_into ? F[f] + s * acc : s * acc;
      }
  };
  apply(rowA0, rowA1, S, s1, false);
  if (upwind) apply(rowA0 + BOFF, rowA1 + BOFF, D, s2, true);
}

// R += s (M0 (x) M1 (x) M2) c for component D (Q layout, index a0 + N1 a1 +
// N1^2 a2), contracted one z-slab of c at a time; M2 read from its
// shared-memory row.  The operator of axis D holds L_a', so its row a = 0
// vanishes and the modes a_D = 0 get nothing.
template <int DIM, int P, bool PB, int D, typename T>
__device__ __forceinline__ void apply_sep_reg(const T* __restrict__ m0row, const T* __restrict__ m1row,
                                              const T* __restrict__ m2row, const T* c, T* R, T s) {
  constexpr int N1 = P + 1, NZ = DIM > 2 ? N1 : 1;
  T M0[N1][N1], M1[N1][N1];
  load_op<N1, T>(m0row, M0);
  load_op<N1, T>(m1row, M1);
#pragma unroll
  for (int a0 = D == 0 ? 1 : 0; a0 < N1; ++a0)
#pragma unroll
    for (int b0 = 0; b0 < N1; ++b0) M0[a0][b0] *= s;
#pragma unroll
  for (int b2 = 0; b2 < NZ; ++b2) {
    T u[N1][N1];   // [a0][b1]
#pragma unroll
    for (int a0 = D == 0 ? 1 : 0; a0 < N1; ++a0)
#pragma unroll
      for (int b1 = 0; b1 < N1; ++b1) {
        if (!mode_in<P, PB>(b1 + b2)) continue;
        T acc = T(0);
#pragma unroll
        for (int b0 = 0; b0 < N1; ++b0)
          if (mode_in<P, PB>(b0 + b1 + b2)) acc += M0[a0][b0] * c[b0 + N1 * (b1 + N1 * b2)];
        u[a0][b1] = acc;
      }
    T m2c[N1];   // column b2 of M2
    if constexpr (DIM > 2) {
#pragma unroll
      for (int a2 = D == 2 ? 1 : 0; a2 < N1; ++a2) m2c[a2] = m2row[a2 * N1 + b2];
    }
#pragma unroll
    for (int a1 = D == 1 ? 1 : 0; a1 < N1; ++a1)
#pragma unroll
      for (int a0 = D == 0 ? 1 : 0; a0 < N1; ++a0) {
        if (!mode_in<P, PB>(a0 + a1)) continue;
        T v = T(0);
#pragma unroll
        for (int b1 = 0; b1 < N1; ++b1)
          if (mode_in<P, PB>(b1 + b2)) v += M1[a1][b1] * u[a0][b1];
        if constexpr (DIM == 2) {
          R[a0 + N1 * a1] += v;
        } else {
#pragma unroll
          for (int a2 = D == 2 ? 1 : 0; a2 < N1; ++a2)
            if (mode_in<P, PB>(a0 + a1 + a2)) R[a0 + N1 * (a1 + N1 * a2)] += m2c[a2] * v;
        }
      }
  }
}

// What bounds it: issue and latency, 16 warps per SM at Q2 3D (128 registers).
// 64^3 Q2 FP32 51.4 -> 39.5 us, 128^3 372 -> 290, 60^3 P2 FP32 48.9 -> 22.4,
// FP64 72 -> 36, 45x37x50 Q2 FP64 43.8 -> 38.3 against the version with the
// zero rows, the padded modes, a mode switch per stored value and 8 instead
// of 5 instructions per lifted face mode.
//
// FP32 tiles fit two CTAs per SM (<= 128 registers); an FP64 tile takes most
// of an SM's shared memory, so FP64 gets the full register file.
//
// Phases: (1) every face of the tile (interior, tile boundary, domain
// boundary) is a work item: traces of its two box cells, the separable
// upwind flux, written to the face's slot, so each face's flux is computed
// once per CTA by one routine whatever the tiling;
// (2) every cell: the cell term (one direction at a time) and the lifting of
// its 2 dim face fluxes from the slots; (3) the RK combination fused into
// the coalesced store.  BC: the mesh may carry Dirichlet faces.
template <int DIM, int P, bool PB, int TX, int TY, int TZ, typename T, bool BC>
__global__ void __launch_bounds__(TX * TY * TZ, sizeof(T) == 4 ? 2 : 1)
    adv_sep_kernel(const AdvSepArgs<T> a) {
  using PL = SepPlan<DIM, P, PB, TX, TY, TZ, T>;
  constexpr int N1 = PL::N1, NM = PL::NM, NF = PL::NF, OPW = PL::OPW, BOFF = sep_boff<P>();
  constexpr int NBG = PL::NBG;
  constexpr int NT = PL::NT, NMB = PL::NMB, SPAN = PL::SPAN;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem_raw);
  unsigned char* boxb = smem_raw + PL::OFF_BOX;
  T* ops = reinterpret_cast<T*>(smem_raw + PL::OFF_OPS);
  T* fl = reinterpret_cast<T*>(smem_raw + PL::OFF_FL);
  const MeshArgs& m = a.m;
  const Tab1D<T>& tb = tab<T>(P);

  // tile and cell coordinates
  int b = blockIdx.x;
  const int ox = (b % m.ntile[0]) * TX;
  b /= m.ntile[0];
  const int oy = DIM > 1 ? (b % m.ntile[1]) * TY : 0;
  const int oz = DIM > 2 ? (b / m.ntile[1]) * TZ : 0;
  const int l[3] = {(int)threadIdx.x % TX, ((int)threadIdx.x / TX) % TY, DIM > 2 ? (int)threadIdx.x / (TX * TY) : 0};
  const int g[3] = {ox + l[0], oy + l[1], oz + l[2]};
  const bool valid = g[0] < m.n[0] && g[1] < m.n[1] && (DIM < 3 || g[2] < m.n[2]);
  const int gx0 = max(ox - 1, 0), gx1 = min(ox + TX + 1, m.n[0]);

  // address of the box copy of the cell at local coordinates (lx, ly, lz)
  auto cellp = [&](int lx, int ly, int lz) -> const T* {
    const int rr = DIM > 2 ? (ly + 1) + PL::BY * (lz + 1) : ly + 1;
    const unsigned rowcell = (unsigned)m.n[0] * (unsigned)((oy + ly) + m.n[1] * (DIM > 2 ? oz + lz : 0));
    const unsigned phase = ((rowcell + (unsigned)gx0) * (unsigned)NMB) & 15u;
    return reinterpret_cast<const T*>(boxb + (size_t)rr * PL::SLOT + phase + (ox + lx - gx0) * NMB);
  };
  // operator row of component d, axis e, tile cell le along e
  auto rowp = [&](int d, int e, int le) -> const T* {
    const int roff = e == 0 ? 0 : (e == 1 ? TX : TX + TY);
    return ops + (size_t)(d * SPAN + roff + le) * OPW;
  };

  // ---- staging on one mbarrier: the box rows by bulk copies issued by the
  // lanes of warp 0, the operator rows by thread 0
  if (threadIdx.x == 0) mbar_init(bar, 33);
  __syncthreads();
  if (threadIdx.x == 0) {
    constexpr unsigned kRowBytes = OPW * sizeof(T);
    mbar_arrive_expect_tx(bar, DIM * SPAN * kRowBytes);
#pragma unroll
    for (int d = 0; d < DIM; ++d)
#pragma unroll
      for (int e = 0; e < DIM; ++e)
        bulk_g2s(const_cast<T*>(rowp(d, e, 0)),
                 a.optab + ((size_t)(d * 3 + e) * a.nmax + (e == 0 ? ox : (e == 1 ? oy : oz))) * OPW,
                 (e == 0 ? TX : (e == 1 ? TY : TZ)) * kRowBytes, bar);
  }
  // the operator rows do not change during a run; the field does
  chain_wait();
  if (threadIdx.x < 32) bulk_box_rows<DIM, TX, TY, TZ, NMB, PL::SLOT>(m, a.phi_s, boxb, ox, oy, oz, bar);
  if (!mbar_wait(bar, 0, 1 << 22)) {
    if (threadIdx.x == 0 && a.err) atomicOr(a.err, kErrCopyTimeout);
    mbar_wait(bar, 0, 1 << 22);   // give copies in flight a last chance to land
  }

  const T ct = a.step ? T(a.step->ct[a.stage]) : T(a.ct_explicit);
  const T dt = a.step ? T(a.step->dt) : T(a.dt_explicit);
  const bool active = a.step ? (a.step->active != 0) : true;
  const int cl = threadIdx.x;
  const T ih[3] = {T(1.0 / m.h[0]), T(1.0 / m.h[1]), T(DIM > 2 ? 1.0 / m.h[2] : 1.0)};
  const bool work = valid && active;
  constexpr int SL[3] = {PL::SL0, PL::SL1, PL::SL2};
  constexpr int FLO[3] = {0, NF * PL::SL0, NF * (PL::SL0 + PL::SL1)};

  // ===== (1) face fluxes, one work item per face of the tile.  The faces
  // normal to E form a block (TX + (E==0)) x (TY + (E==1)) x (TZ + (E==2))
  // in slot order, x fastest (consecutive lanes read consecutive cells of a
  // box row); the three blocks start on warp boundaries when their sizes are
  // multiples of 32, so a warp serves one axis
  auto face_item = [&](auto EC, int r) {
    constexpr int E = decltype(EC)::value;
    constexpr int t0 = E == 0 ? 1 : 0, t1 = E == 2 ? 1 : 2;
    constexpr int EX = TX + (E == 0), EY = TY + (E == 1);
    const int lx = r % EX, ly = (r / EX) % EY, lz = DIM > 2 ? r / (EX * EY) : 0;
    const int lc[3] = {lx, ly, lz};
    const int gc[3] = {ox + lx, oy + ly, oz + lz};
    if ((E != 0 && gc[0] >= m.n[0]) || (E != 1 && gc[1] >= m.n[1]) || (DIM > 2 && E != 2 && gc[2] >= m.n[2])) return;
    const int f = lc[E], gE = gc[E];
    const bool has_m = gE >= 1 && gE - 1 < m.n[E], has_p = gE < m.n[E];
    if (!has_m && !has_p) return;
    const T* cp = cellp(lx, ly, lz);
    const T* cm = cellp(lx - (E == 0), ly - (E == 1), lz - (E == 2));
    T gd = T(0);
    bool dir = false;
    if constexpr (BC) {
      if (!has_m) dir = bc_dirichlet<DIM>(m, E, 0, gc, gd);
      else if (!has_p) {
        const int gl[3] = {gc[0] - (E == 0), gc[1] - (E == 1), gc[2] - (E == 2)};
        dir = bc_dirichlet<DIM>(m, E, 1, gl, gd);
      }
    }
    // tangential operator rows and the normal factor g_EE at the face: the
    // upper cell's xi = 0 value where that cell is a tile cell of the mesh,
    // else the lower cell's xi = 1 value (the same number, tabulated from
    // one expression; rows past the mesh hold no face values)
    const T* r0 = rowp(E, t0, lc[t0]);
    const T* r1 = DIM > 2 ? rowp(E, t1, lc[t1]) : nullptr;
    const T fe = (f < (E == 0 ? TX : (E == 1 ? TY : TZ)) && has_p) ? rowp(E, E, f)[BOFF] : rowp(E, E, f - 1)[BOFF + 1];
    const T s1 = ct * fe * ih[E];   // the flux is kept per unit length
    T F[NF];
    // tangential factors of one sign over the face: |u_E| = sigma u_E, so
    // the flux is u_E times the upwind trace alone
    const T sigma = DIM > 2 ? r0[N1 * N1] * r1[N1 * N1] : r0[N1 * N1];
    if (sigma != T(0)) {
      const bool flow_up = s1 * sigma > T(0);   // upwind: the lower cell
      T W[NF];
      if (dir && !(flow_up ? has_m : has_p)) {
#pragma unroll
        for (int mf = 0; mf < NF; ++mf) W[mf] = mf == 0 ? gd : T(0);
      } else {
        const bool up_m = flow_up ? has_m : !has_p;
        face_trace_ct<DIM, P, PB, E, T>(up_m ? cm : cp, up_m ? tb.L1 : tb.L0, W);
      }
      face_apply<DIM, P, PB, BOFF, T>(r0, r1, W, W, s1, T(0), false, F);
    } else {
      T S[NF], D[NF];   // traces Tm / Tp, then their mean / half jump in place
      if (has_m) face_trace_ct<DIM, P, PB, E, T>(cm, tb.L1, S);
      if (has_p) face_trace_ct<DIM, P, PB, E, T>(cp, tb.L0, D);
#pragma unroll
      for (int mf = 0; mf < NF; ++mf) {
        const T ghost = dir ? (mf == 0 ? gd : T(0)) : T(0);
        const T tm = has_m ? S[mf] : (dir ? ghost : D[mf]), tp = has_p ? D[mf] : (dir ? ghost : S[mf]);
        S[mf] = T(0.5) * (tm + tp);
        D[mf] = T(0.5) * (tm - tp);
      }
      face_apply<DIM, P, PB, BOFF, T>(r0, r1, S, D, s1, s1 < T(0) ? -s1 : s1, (has_m && has_p) || dir, F);
    }
    const int sl = lx + EX * (ly + EY * lz);
#pragma unroll
    for (int mf = 0; mf < NF; ++mf) fl[FLO[E] + mf * SL[E] + sl] = F[mf];
  };
  if (active) {
    constexpr int TOT = PL::SL0 + PL::SL1 + PL::SL2;
    for (int it = threadIdx.x; it < TOT; it += NT) {
      if (it < SL[0]) face_item(std::integral_constant<int, 0>(), it);
      else if (it < SL[0] + SL[1]) face_item(std::integral_constant<int, 1>(), it - SL[0]);
      else if constexpr (DIM > 2) face_item(std::integral_constant<int, 2>(), it - SL[0] - SL[1]);
    }
  }
  __syncthreads();

  // ===== (2) cell term and the lifting of the cell's face fluxes
  T R[NM];
#pragma unroll
  for (int q = 0; q < NM; ++q) R[q] = T(0);
  if (work) {
    // the cell's coefficients in registers (Q layout)
    T c[NM];
    {
      const T* cme = cellp(l[0], l[1], l[2]);
#pragma unroll
      for (int q = 0; q < NM; ++q) {
        constexpr int kOut = -1;
        const int gi = cell_index<DIM, P, PB>(q);
        c[q] = gi != kOut ? cme[gi] : T(0);
      }
    }
    const T* m2[3] = {nullptr, nullptr, nullptr};
    if constexpr (DIM > 2) {
#pragma unroll
      for (int d = 0; d < DIM; ++d) m2[d] = rowp(d, 2, l[2]);
    }
    apply_sep_reg<DIM, P, PB, 0, T>(rowp(0, 0, l[0]), rowp(0, 1, l[1]), m2[0], c, R, ct * ih[0]);
    apply_sep_reg<DIM, P, PB, 1, T>(rowp(1, 0, l[0]), rowp(1, 1, l[1]), m2[1], c, R, ct * ih[1]);
    if constexpr (DIM > 2) apply_sep_reg<DIM, P, PB, 2, T>(rowp(2, 0, l[0]), rowp(2, 1, l[1]), m2[2], c, R, ct * ih[2]);
    // R += L(0) F_lower - L(1) F_upper: by parity (L_a(0) = (-1)^a L_a(1)) the
    // even modes along E take L_a(1) times the difference, the odd ones
    // minus L_a(1) times the sum
    auto lift = [&](auto EC) {
      constexpr int E = decltype(EC)::value;
      constexpr int t0 = E == 0 ? 1 : 0, t1 = E == 2 ? 1 : 2;
      constexpr int st[3] = {1, N1, N1 * N1};
      const int slo = l[0] + (TX + (E == 0)) * (l[1] + (TY + (E == 1)) * l[2]);
      const int sup = slo + (E == 0 ? 1 : (E == 1 ? TX : (TX * (TY + 0)) ));
#pragma unroll
      for (int m1 = 0; m1 < (DIM > 2 ? N1 : 1); ++m1)
#pragma unroll
        for (int m0 = 0; m0 < N1; ++m0) {
          if (!mode_in<P, PB>(m0 + m1)) continue;
          const int f = FLO[E] + face_index<P, PB>(m0, m1) * SL[E];
          const T flo = fl[f + slo], fup = fl[f + sup];
          const T dif = flo - fup, sum = flo + fup;
          const int base = m0 * st[t0] + (DIM > 2 ? m1 * st[t1] : 0);
          R[base] += dif;
#pragma unroll
          for (int a = 1; a < N1; ++a) {
            if (!mode_in<P, PB>(m0 + m1 + a)) continue;
            if (a % 2) R[base + a * st[E]] -= tb.L1[a] * sum;
            else R[base + a * st[E]] += tb.L1[a] * dif;
          }
        }
    };
    lift(std::integral_constant<int, 0>());
    lift(std::integral_constant<int, 1>());
    if constexpr (DIM == 3) lift(std::integral_constant<int, 2>());
  }
  __syncthreads();   // face fluxes consumed: the region now holds R [cell][NBG], HBM order
  T* rbuf = fl;
  if (work) {
#pragma unroll
    for (int q = 0; q < NM; ++q) {
      const int gi = cell_index<DIM, P, PB>(q);
      if (gi >= 0) rbuf[(size_t)cl * NBG + gi] = R[q];
    }
  }
  __syncthreads();

  // 2D FP64: without an early release (233x190 Q3 run 4.10 against 4.27 ms with
  // it, 128^2 P1 the same within 1 %)
  if constexpr (DIM == 3 || sizeof(T) == 4) chain_release();
  combine_rows<DIM, TX, TY, TZ, NBG, NT / 32, T>(m, cellp, rbuf, a.phi_n, a.out, a.combine, dt, active, ox, oy, oz);
}

}  // namespace flsp
