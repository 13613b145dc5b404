// flsp_hjs.cuh — Hamilton-Jacobi reinitialisation pseudo-step, tensor-
// product (FE_DGQLegendre) basis, with the work of a cell split over its
// Gauss planes.
//
// The point-wise operator (the reference functions it replaces are listed in
// flsp_hj.cuh), restated for throughput:
//  * the smooth sign S(phi0) (src/level_set/reinit.cc:121-133) depends on
//    phi0 alone, which stays fixed through a reinitialisation sweep.  The
//    sweep's first launch (mode kHJCflOnly, phi == phi0) evaluates it at the
//    cell Gauss points and at the CFL vertices into a per-tile table; every
//    pseudo-step reads it from there instead of evaluating phi0 and its
//    gradient again (the same expression on the same inputs);
//  * NQ threads per cell: thread k of a cell owns the Gauss plane k of the
//    last axis (z in 3D, y in 2D).  Its partial projection onto the modes
//    goes through shared memory, and each thread finishes every NQ-th mode
//    of the cell (the sums over planes keep their order);
//  * the face jumps are formed once per face, not once per cell side;
//  * the sums over modes and points go by parity (gauss_values and its
//    neighbours), the Hamiltonian takes the mean and half the difference of
//    the one-sided gradients, and the plane projections overwrite the sign
//    table entries of the thread's own plane.
// What bounds it: issue and latency (64^3 Q2 FP32: 61.5 M warp instructions,
// 58 % issue active, 24 warps per SM; the loads, barriers and store alone take
// 47 us).  64^3 Q2 FP32 135 -> 98 us, 128^3 996 -> 708, 45x37x50 Q2 FP64
// 129 -> 101, 256^2 Q2 FP32 14.4 -> 10.3 against the kernel with plain sums
// and a two-pass copy issue.
//
// Table layout: stab[(tile * NS + j) * nt + c], c the cell within the tile;
// j < NQ^dim: the Gauss point qx + NQ (qy + NQ qz), holding w_q S (the
// quadrature weight folded in: w_q H = H with S replaced by w_q S, as
// w_q > 0); j = NQ^dim + v: S at the vertex v (x bit 0, y bit 1, z bit 2).  Tiles are the launch's tiles (the
// narrow band selects among them; the tile index is the global one).
#pragma once
#include "flsp_device.cuh"
#include "flsp_clock.cuh"
#include "flsp_hj.cuh"

namespace flsp {

// table entries per cell
template <int DIM, int P>
__host__ __device__ constexpr int hjs_ns() {
  return ipow(P + 2, DIM) + (1 << DIM);
}

// shared-memory plan: the halo box as rows of cells along x, each row a
// bulk copy from a 16-byte aligned global address (the row's data starts at
// its slot + the address phase), then the face jumps, the corner jumps,
// the plane projections and the block reduction
template <int DIM, int P, typename T>
struct HjsPlan {
  using TL = HjsTile<DIM>;
  static constexpr int N1 = P + 1, NQ = P + 2, NM = ipow(N1, DIM), NQF = ipow(NQ, DIM - 1);
  static constexpr int NC = 1 << (DIM - 1), NU = ipow(N1, DIM - 1);
  static constexpr int BY = TL::Y + 2, BZ = DIM > 2 ? TL::Z + 2 : 1, NROWS = BY * BZ;
  static constexpr int NMB = NM * (int)sizeof(T);   // bytes per cell
  static constexpr int SLOT = (((TL::X + 2) * NMB + 30) + 15) / 16 * 16;
  static constexpr size_t OFF_BOX = 32;   // mbarrier, CFL maximum, pseudo-step
  static constexpr size_t OFF_JN = OFF_BOX + (size_t)NROWS * SLOT;
  static constexpr size_t OFF_JV = OFF_JN + (size_t)2 * DIM * NQF * TL::N * sizeof(T);
  // the tile's slice of the sign table (pseudo-steps: staged with the box);
  // a thread's plane projections overwrite the entries of its own plane
  static constexpr int NS = ipow(NQ, DIM) + (1 << DIM);
  static constexpr size_t TAB_BYTES = (size_t)NS * TL::N * sizeof(T);
  static constexpr size_t UB_BYTES = (size_t)NQ * NU * TL::N * sizeof(T);
  static constexpr size_t OFF_UB = (OFF_JV + (size_t)2 * DIM * NC * TL::N * sizeof(T) + 15) / 16 * 16;
  static constexpr size_t BYTES = OFF_UB + (TAB_BYTES > UB_BYTES ? TAB_BYTES : UB_BYTES);
};

// CTAs per SM the registers are held to: FP32 3D, as many as the shared
// memory admits (80 registers, 24 warps: left to itself the compiler takes
// 105 and two CTAs, and the kernel is no faster than before it lost a third
// of its instructions).  2D P = 3 one more than its registers would allow
// (FP32 72 -> 64 registers, 20 -> 30 warps; FP64 116 -> 96, 10 -> 20 warps:
// inviscid 233x190 run 4.07 -> 3.89 ms, band reinit of 256x240 6.4 -> 5.7);
// P = 2 spills when held (256^2 run 3.00 -> 3.02 ms) and is left alone.
template <int DIM, int P, typename T>
constexpr int hjs_min_blocks() {
  if (DIM == 2) return P == 3 ? (sizeof(T) == 4 ? 3 : 2) : 1;
  return sizeof(T) == 4 ? (P == 1 ? 4 : 3) : 1;
}

// smooth sign from phi0's value and (scaled) gradient at a point, with the
// pseudo-step kernels' operation sequence
template <typename T>
__device__ __forceinline__ T hjs_sign(T p0, T g2, T hmin) {
  if constexpr (sizeof(T) == 4) {
    return p0 * rsqrtf(p0 * p0 + hmin * hmin * g2);
  } else {
    const T gn = sqrt(g2);
    return p0 / sqrt(p0 * p0 + hmin * hmin * gn * gn);
  }
}

// the jump phi_upper - phi_lower on the faces normal to E (one face per
// call, lower cell at local lc with lc[E] = f - 1), times 1/h_E, written
// nodal at the face Gauss points and at the face corners for both adjacent
// tile cells
template <int DIM, int P, int E, typename T, typename CellP>
__device__ __forceinline__ void hjs_face(const MeshArgs& m, const CellP& cellp, T* jn, T* jv, const int* o,
                                         int r) {
  constexpr int N1 = P + 1, NQ = P + 2, NF = ipow(N1, DIM - 1), NQF = ipow(NQ, DIM - 1), NC = 1 << (DIM - 1);
  constexpr int t0 = E == 0 ? 1 : 0, t1 = E == 2 ? 1 : 2;
  constexpr int st[3] = {1, N1, N1 * N1};
  const Tab1D<T>& tb = tab<T>(P);
  using TL = HjsTile<DIM>;
  constexpr int nt = TL::N, tl[3] = {TL::X, TL::Y, TL::Z};
  const int f = r % (tl[E] + 1);
  const int rest = r / (tl[E] + 1);
  int lu[3];
  lu[E] = f;
  lu[t0] = rest % tl[t0];
  lu[t1] = DIM > 2 ? rest / tl[t0] : 0;
  if (o[t0] + lu[t0] >= m.n[t0] || (DIM > 2 && o[t1] + lu[t1] >= m.n[t1])) return;
  int ll[3] = {lu[0], lu[1], lu[2]};
  ll[E] = f - 1;
  const bool inside = o[E] + f - 1 >= 0 && o[E] + f < m.n[E];
  T J[NF];
  // a domain-boundary face with a Dirichlet value: the missing side's trace
  // is that constant (LDG left / right boundary terms, ldg.cc:551-620,
  // :686-740); without one the jump is zero (interior trace)
  T gd = T(0);
  bool dir = false;
  if (!inside && (o[E] + f == 0 || o[E] + f == m.n[E])) {
    int gcell[3] = {o[0] + lu[0], o[1] + lu[1], o[2] + lu[2]};
    gcell[E] = o[E] + f == 0 ? 0 : m.n[E] - 1;
    dir = bc_dirichlet<DIM>(m, E, o[E] + f == 0 ? 0 : 1, gcell, gd);
  }
  if (dir) {
    const bool lower = o[E] + f == 0;   // the domain's lower side: the cell is above the face
    const T* cc = lower ? cellp(lu[0], lu[1], lu[2]) : cellp(ll[0], ll[1], ll[2]);
#pragma unroll
    for (int mf = 0; mf < NF; ++mf) {
      const int m0 = mf % N1, m1 = mf / N1;
      const int base = m0 * st[t0] + (DIM > 2 ? m1 * st[t1] : 0);
      T tr = T(0);
#pragma unroll
      for (int b = 0; b < N1; ++b) tr += (lower ? tb.L0[b] : tb.L1[b]) * cc[base + b * st[E]];
      const T ghost = mf == 0 ? gd : T(0);
      J[mf] = lower ? tr - ghost : ghost - tr;
    }
  } else if (inside) {
    const T* cu = cellp(lu[0], lu[1], lu[2]);
    const T* cd = cellp(ll[0], ll[1], ll[2]);
#pragma unroll
    for (int mf = 0; mf < NF; ++mf) {
      const int m0 = mf % N1, m1 = mf / N1;
      const int base = m0 * st[t0] + (DIM > 2 ? m1 * st[t1] : 0);
      T j = cu[base] - cd[base];   // L_0 = 1
#pragma unroll
      for (int b = 1; b < N1; ++b) j += tb.L0[b] * cu[base + b * st[E]] - tb.L1[b] * cd[base + b * st[E]];
      J[mf] = j;
    }
  } else {
#pragma unroll
    for (int mf = 0; mf < NF; ++mf) J[mf] = T(0);
  }
  // the upper cell sees this face as its lower side (slot 2E), the lower
  // cell as its upper side (slot 2E + 1)
  const int cu_l = f < tl[E] ? lu[0] + tl[0] * (lu[1] + tl[1] * lu[2]) : -1;
  const int cd_l = f >= 1 ? ll[0] + tl[0] * (ll[1] + tl[1] * ll[2]) : -1;
  const T ihE = T(1.0 / m.h[E]);
#pragma unroll
  for (int mf = 0; mf < NF; ++mf) J[mf] *= ihE;
  auto put = [&](int q, T v, bool corner) {
    const int base = corner ? 2 * E * NC : 2 * E * NQF, stride = corner ? NC : NQF;
    T* dst = corner ? jv : jn;
    if (cu_l >= 0) dst[(size_t)(base + q) * nt + cu_l] = v;
    if (cd_l >= 0) dst[(size_t)(base + stride + q) * nt + cd_l] = v;
  };
  if constexpr (DIM == 2) {
    T v[NQ], lo, hi;
    gauss_values<N1, NQ, 1, T>(tb, J, v);
#pragma unroll
    for (int q0 = 0; q0 < NQ; ++q0) put(q0, v[q0], false);
    end_values<N1, 1, T>(tb, J, lo, hi);
    put(0, lo, true);
    put(1, hi, true);
  } else {
    T Pq[N1][NQ], Pl[N1], Ph[N1];   // [m1][q0], and at the ends of axis t0
#pragma unroll
    for (int m1 = 0; m1 < N1; ++m1) {
      gauss_values<N1, NQ, 1, T>(tb, J + N1 * m1, Pq[m1]);
      end_values<N1, 1, T>(tb, J + N1 * m1, Pl[m1], Ph[m1]);
    }
#pragma unroll
    for (int q0 = 0; q0 < NQ; ++q0) {
      T v[NQ];
      gauss_values<N1, NQ, NQ, T>(tb, &Pq[0][q0], v);
#pragma unroll
      for (int q1 = 0; q1 < NQ; ++q1) put(q0 + NQ * q1, v[q1], false);
    }
    T c0, c1, c2, c3;
    end_values<N1, 1, T>(tb, Pl, c0, c2);
    end_values<N1, 1, T>(tb, Ph, c1, c3);
    put(0, c0, true);
    put(1, c1, true);
    put(2, c2, true);
    put(3, c3, true);
  }
}

// values and gradients (reference-cell derivatives) of the modal field c
// at the two vertices (vx = 0, 1) of the x-line with corner bits (vy, vz):
// the y/z reductions are shared by both ends of the line.  The odd modes
// change sign between the two ends of an axis, L_0 = 1, D_0 = 0.
template <int DIM, int N1, typename T>
__device__ __forceinline__ void hjs_line(const T* c, const Tab1D<T>& tb, int vy, int vz, T* val, T (*gr)[3]) {
  T Y[N1], Yd[N1], Z[N1], Zd[N1];
#pragma unroll
  for (int b = 1; b < N1; ++b) {
    Y[b] = vy ? tb.L1[b] : tb.L0[b];
    Yd[b] = vy ? tb.D1[b] : tb.D0[b];
    Z[b] = vz ? tb.L1[b] : tb.L0[b];
    Zd[b] = vz ? tb.D1[b] : tb.D0[b];
  }
  T V[N1], Vy[N1], Vz[N1];
#pragma unroll
  for (int a = 0; a < N1; ++a) {
    T W[N1], Wd[N1];
#pragma unroll
    for (int b = 0; b < N1; ++b) {
      W[b] = c[a + N1 * b];
      Wd[b] = T(0);
      if constexpr (DIM > 2) {
#pragma unroll
        for (int cc = 1; cc < N1; ++cc) {
          W[b] += c[a + N1 * (b + N1 * cc)] * Z[cc];
          Wd[b] += c[a + N1 * (b + N1 * cc)] * Zd[cc];
        }
      }
    }
    T s0 = W[0], s1 = T(0), s2 = Wd[0];
#pragma unroll
    for (int b = 1; b < N1; ++b) {
      s0 += W[b] * Y[b];
      s1 += W[b] * Yd[b];
      if constexpr (DIM > 2) s2 += Wd[b] * Y[b];
    }
    V[a] = s0;
    Vy[a] = s1;
    Vz[a] = s2;
  }
  end_values<N1, 1, T>(tb, V, val[0], val[1]);
  end_values<N1, 1, T>(tb, Vy, gr[0][1], gr[1][1]);
  if constexpr (DIM > 2) end_values<N1, 1, T>(tb, Vz, gr[0][2], gr[1][2]);
  T ge = V[1] * tb.D1[1], go = T(0);   // L_a' is even for odd a
  if constexpr (N1 > 3) ge += V[3] * tb.D1[3];
  if constexpr (N1 > 2) go = V[2] * tb.D1[2];
  gr[0][0] = ge - go;
  gr[1][0] = ge + go;
}

// the characteristic speed at a vertex (ReinitOperator::
// characteristic_velocity, reinit.cc:235-264) from the upwind parts of the
// one-sided gradients: their unit vector times S, i.e. |S| unless every
// part vanishes (then the vanishing norm itself).  A norm that overflows
// or is NaN gives NaN, which the maxima ignore.
template <int DIM, typename T>
__device__ __forceinline__ T hjs_speed(T S, const T* left, const T* right) {
  T n2 = T(0);
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const T l = S >= T(0) ? left[d] : -left[d], r = S >= T(0) ? -right[d] : right[d];
    const T g = fmax(fmax(l, T(0)), fmax(r, T(0)));
    n2 += g * g;
  }
  constexpr T eps2 = T(2.220446049250313e-16) * T(2.220446049250313e-16);
  return n2 > eps2 ? fabs(S) + (n2 - n2) : sqrt(n2);
}

// One block serves one HjsTile of cells (launch slot blockIdx.x) with NQ
// threads per cell (blockDim = cells * NQ); its halo box arrives by bulk
// copies on one mbarrier.  Modes: kHJCflOnly (phi == phi0: fills the sign
// table, CFL estimate of the first pseudo-step) and kHJStep (one pseudo-
// step from the table, CFL estimate of the next).
template <int DIM, int P, typename T>
__device__ __forceinline__ void hjs_tile(const HJArgs<T>& a, int slot) {
  using PL = HjsPlan<DIM, P, T>;
  constexpr int N1 = P + 1, NQ = P + 2, NM = ipow(N1, DIM), NV = 1 << DIM;
  constexpr int NQF = ipow(NQ, DIM - 1), NC = 1 << (DIM - 1);
  constexpr int NU = ipow(N1, DIM - 1), NQV = ipow(NQ, DIM), NS = NQV + NV;
  using TL = HjsTile<DIM>;
  constexpr int TX = TL::X, TY = TL::Y, TZ = TL::Z, NT = TL::N, NMB = PL::NMB;
  static_assert(NM <= 2 * DIM * NQF, "the store staging reuses the face-jump area");
  static_assert(NU <= NQF, "a plane's projection fits its table entries");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem_raw);
  unsigned char* boxb = smem_raw + PL::OFF_BOX;
  T* jn = reinterpret_cast<T*>(smem_raw + PL::OFF_JN);   // [2*DIM*NQF][NT]
  T* jv = reinterpret_cast<T*>(smem_raw + PL::OFF_JV);   // [2*DIM*NC][NT]
  MaxSlot<T>* cfl = reinterpret_cast<MaxSlot<T>*>(smem_raw + 16);
  double* sdt = reinterpret_cast<double*>(smem_raw + 24);   // the pseudo-step
  T* stl = reinterpret_cast<T*>(smem_raw + PL::OFF_UB);   // table slice [NS][NT] (pseudo-steps)
  T* ub = stl;                                            // plane projections [NQ][NQF][NT] (u < NU used)
  const MeshArgs& m = a.m;
  const Tab1D<T>& tb = tab<T>(P);
  const bool step = a.mode == kHJStep;
  double vd = 0.0;   // thread 0: the running CFL maximum before this step
  chain_wait();
  if (tile_inactive(m, slot)) {
    if (step && slot == 0 && threadIdx.x == 0) hj_clock_step(a.clk, a.step, true, vd);
    return;
  }

  auto origin = [&](int slot, int* o) {
    int b = m.tiles ? m.tiles[slot] : slot;
    o[0] = (b % m.ntile[0]) * TX;
    b /= m.ntile[0];
    o[1] = DIM > 1 ? (b % m.ntile[1]) * TY : 0;
    o[2] = DIM > 2 ? (b / m.ntile[1]) * TZ : 0;
  };
  const int cl = (int)threadIdx.x % NT, k = (int)threadIdx.x / NT;   // cell, Gauss plane
  const int l[3] = {cl % TX, (cl / TX) % TY, DIM > 2 ? cl / (TX * TY) : 0};
  const T ih[3] = {T(1.0 / m.h[0]), T(1.0 / m.h[1]), T(DIM > 2 ? 1.0 / m.h[2] : 1.0)};
  const T hmin = T(m.min_diam);
  const bool fill = a.mode == kHJCflOnly;
  // this thread's Gauss plane (uniform per warp): its 1D table entries
  T Lk[N1], Dk[N1];
#pragma unroll
  for (int b = 0; b < N1; ++b) {
    Lk[b] = tb.Lq[b][k];
    Dk[b] = tb.Dq[b][k];
    if (step) Dk[b] *= ih[DIM - 1];   // the pseudo-steps' plane derivative, per unit length
  }
  T vmax = T(0);

  int o[3];
  origin(slot, o);
  const int tile = m.tiles ? m.tiles[slot] : slot;
  // the tile's slice of the sign table by one bulk copy, the halo box by row
  // copies of the first warp's lanes
  if (threadIdx.x == 0) {
    mbar_init(bar, 32 + (step ? 1 : 0));
    *cfl = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (step) {
      mbar_arrive_expect_tx(bar, (unsigned)PL::TAB_BYTES);
      bulk_g2s(stl, a.stab + (size_t)tile * NS * NT, (unsigned)PL::TAB_BYTES, bar);
      *sdt = hj_clock_step(a.clk, a.step, slot == 0, vd);
    }
  }
  if (threadIdx.x < 32) bulk_box_rows<DIM, TX, TY, TZ, NMB, PL::SLOT>(m, a.phi, boxb, o[0], o[1], o[2], bar);
  const int g[3] = {o[0] + l[0], o[1] + l[1], o[2] + l[2]};
  const bool valid = g[0] < m.n[0] && g[1] < m.n[1] && (DIM < 3 || g[2] < m.n[2]);
  const int gx0 = max(o[0] - 1, 0);
  // box copy of the cell at local coordinates (lx, ly, lz)
  auto cellp = [&](int lx, int ly, int lz) -> const T* {
    const int rr = (ly + 1) + PL::BY * (DIM > 2 ? lz + 1 : 0);
    const unsigned rowcell = (unsigned)m.n[0] * (unsigned)((o[1] + ly) + m.n[1] * (DIM > 2 ? o[2] + lz : 0));
    const unsigned phase = ((rowcell + (unsigned)gx0) * (unsigned)NMB) & 15u;
    return reinterpret_cast<const T*>(boxb + (size_t)rr * PL::SLOT + phase + (o[0] + lx - gx0) * NMB);
  };
  if (!mbar_wait(bar, 0u, 1 << 22)) {
    if (threadIdx.x == 0 && a.err) atomicOr(a.err, kErrCopyTimeout);
    mbar_wait(bar, 0u, 1 << 22);   // give copies in flight a last chance to land
  }

  // -------- face jumps, one work item per face of the tile
  {
    constexpr int C0 = (TX + 1) * (NT / TX), C1 = (TY + 1) * (NT / TY);
    constexpr int C2 = DIM > 2 ? (TZ + 1) * (NT / TZ) : 0;
    // each axis' items start on a warp boundary: no warp runs two axes' code
    constexpr int W0 = (C0 + 31) / 32 * 32, W1 = W0 + (C1 + 31) / 32 * 32;
    for (int i = threadIdx.x; i < W1 + C2; i += NT * NQ) {
      if (i < W0) {
        if (i < C0) hjs_face<DIM, P, 0, T>(m, cellp, jn, jv, o, i);
      } else if (i < W1) {
        if (i < W0 + C1) hjs_face<DIM, P, 1, T>(m, cellp, jn, jv, o, i - W0);
      } else if constexpr (DIM > 2) {
        hjs_face<DIM, P, 2, T>(m, cellp, jn, jv, o, i - W1);
      }
    }
  }
  __syncthreads();

  T* srow = a.stab + (size_t)tile * NS * NT + cl;   // this cell's table column, stride NT
  // the cell's modes projected on this thread's Gauss plane of the last
  // axis: value (PL0) and derivative (PL1) tables, in the modes of the others
  T PL0[NU], PL1[NU];
  const T* c = cellp(l[0], l[1], l[2]);   // the cell's modes (box copy)
  if (valid) {
    T cr[NM];
#pragma unroll
    for (int q = 0; q < NM; ++q) cr[q] = c[q];
    // -------- sign table of this cell's Gauss plane (phi == phi0)
    if (fill) {
      if constexpr (DIM == 2) {
        T P0y[N1], P0dy[N1];
#pragma unroll
        for (int aa = 0; aa < N1; ++aa) {
          T s3 = T(0), s4 = T(0);
#pragma unroll
          for (int b = 0; b < N1; ++b) {
            const T c0v = cr[aa + N1 * b];
            s3 += c0v * Lk[b];
            s4 += c0v * Dk[b];
          }
          P0y[aa] = s3;
          P0dy[aa] = s4;
        }
#pragma unroll
        for (int qx = 0; qx < NQ; ++qx) {
          T p0 = T(0), g0x = T(0), g0y = T(0);
#pragma unroll
          for (int aa = 0; aa < N1; ++aa) {
            p0 += P0y[aa] * tb.Lq[aa][qx];
            g0x += P0y[aa] * tb.Dq[aa][qx];
            g0y += P0dy[aa] * tb.Lq[aa][qx];
          }
          g0x *= ih[0];
          g0y *= ih[1];
          const T g2 = g0x * g0x + g0y * g0y;
          srow[(size_t)(k * NQF + qx) * NT] = tb.wq[qx] * tb.wq[k] * hjs_sign<T>(p0, g2, hmin);
        }
      } else {
        T P0z[N1][N1], D0z[N1][N1];
#pragma unroll
        for (int aa = 0; aa < N1; ++aa)
#pragma unroll
          for (int b = 0; b < N1; ++b) {
            T s3 = T(0), s4 = T(0);
#pragma unroll
            for (int cc = 0; cc < N1; ++cc) {
              const T c0v = cr[aa + N1 * (b + N1 * cc)];
              s3 += c0v * Lk[cc];
              s4 += c0v * Dk[cc];
            }
            P0z[aa][b] = s3;
            D0z[aa][b] = s4;
          }
#pragma unroll
        for (int qy = 0; qy < NQ; ++qy) {
          T P0y[N1], P0dy[N1], D0zy[N1];
#pragma unroll
          for (int aa = 0; aa < N1; ++aa) {
            T s4 = T(0), s5 = T(0), s6 = T(0);
#pragma unroll
            for (int b = 0; b < N1; ++b) {
              s4 += P0z[aa][b] * tb.Lq[b][qy];
              s5 += P0z[aa][b] * tb.Dq[b][qy];
              s6 += D0z[aa][b] * tb.Lq[b][qy];
            }
            P0y[aa] = s4;
            P0dy[aa] = s5;
            D0zy[aa] = s6;
          }
#pragma unroll
          for (int qx = 0; qx < NQ; ++qx) {
            T p0 = T(0), g0x = T(0), g0y = T(0), g0z = T(0);
#pragma unroll
            for (int aa = 0; aa < N1; ++aa) {
              p0 += P0y[aa] * tb.Lq[aa][qx];
              g0x += P0y[aa] * tb.Dq[aa][qx];
              g0y += P0dy[aa] * tb.Lq[aa][qx];
              g0z += D0zy[aa] * tb.Lq[aa][qx];
            }
            g0x *= ih[0];
            g0y *= ih[1];
            g0z *= ih[2];
            T g2 = g0x * g0x + g0y * g0y;
            g2 += g0z * g0z;
            srow[(size_t)(k * NQF + qx + NQ * qy) * NT] =
                tb.wq[qx] * tb.wq[qy] * tb.wq[k] * hjs_sign<T>(p0, g2, hmin);
          }
        }
      }
    }

    // -------- vertex CFL estimate for the next pseudo-step: x-lines of
    // vertices ln = k, k + NQ, ... (corner bits vy = ln & 1, vz = ln >> 1)
#pragma unroll 1
    for (int ln = k; ln < NV / 2; ln += NQ) {
      T vals[2], grs[2][3];
      hjs_line<DIM, N1, T>(cr, tb, ln & 1, ln >> 1, vals, grs);
#pragma unroll
      for (int vx = 0; vx < 2; ++vx) {
      const int v = vx + 2 * ln;
      const int vb[3] = {vx, ln & 1, ln >> 1};
      const T val = vals[vx];
      const T* dphi = grs[vx];
      T S;
      if (fill) {
        T g2 = T(0);
#pragma unroll
        for (int d = 0; d < DIM; ++d) { const T gg = dphi[d] * ih[d]; g2 += gg * gg; }
        const T gn = sqrt(g2);
        S = val / sqrt(val * val + hmin * hmin * gn * gn);
        srow[(size_t)(NQV + v) * NT] = S;
      } else {
        S = stl[(size_t)(NQV + v) * NT + cl];
      }
      T lft[DIM], rgt[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        const int t0 = d == 0 ? 1 : 0, t1 = d == 2 ? 1 : 2;
        const int cr = vb[t0] + (DIM > 2 ? 2 * vb[t1] : 0);
        const T gd = dphi[d] * ih[d];
        lft[d] = gd + tb.K0v[vb[d]] * jv[(size_t)(2 * d * NC + cr) * NT + cl];
        rgt[d] = gd + tb.K1v[vb[d]] * jv[(size_t)((2 * d + 1) * NC + cr) * NT + cl];
      }
      vmax = fmax(vmax, hjs_speed<DIM, T>(S, lft, rgt));
      }
    }
    if (!fill) {
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        T s1 = cr[u], s2 = T(0);
#pragma unroll
        for (int cc = 1; cc < N1; ++cc) {
          const T cv = cr[u + NU * cc];
          s1 += cv * Lk[cc];
          s2 += cv * Dk[cc];
        }
        PL0[u] = s1;
        PL1[u] = s2;
      }
    }
  }
  slot_max(cfl, vmax);
  if (!step) {
    __syncthreads();
    if (threadIdx.x == 0) atomic_max_pos(&a.clk->hj_vd[0], slot_value(cfl) / m.diam);
    return;
  }

  // -------- pseudo-step: H at this plane's Gauss points, projected onto
  // the modes of the other axes.  With the half jumps p = K0 jl / 2 and
  // q = K1 jh / 2 of an axis the one-sided gradients are g + 2 p and
  // g + 2 q: their mean is g + p + q, half their difference p - q.
  auto jnv = [&](int d, int side, int qf) -> T { return jn[(size_t)((2 * d + side) * NQF + qf) * NT + cl]; };
  auto hfun = [&](T S, const T* avg, T dif) -> T {
    T avg2 = T(0);
#pragma unroll
    for (int d = 0; d < DIM; ++d) avg2 += avg[d] * avg[d];
    T nrm;
    if constexpr (sizeof(T) == 4) nrm = avg2 * rsqrt_normal(fmaxf(avg2, 1e-30f));
    else nrm = sqrt(avg2);
    return S * (nrm - T(1)) + fabs(S) * dif;
  };
  if (valid) {
    const T hK0k = T(0.5) * tb.K0q[k], hK1k = T(0.5) * tb.K1q[k];
    // PL1 already carries 1/h of the plane's axis (Dk)
    if constexpr (DIM == 2) {
      const int qy = k;
      const T jlx = T(0.5) * jnv(0, 0, qy), jhx = T(0.5) * jnv(0, 1, qy);
      T gx[NQ], gy[NQ], f[NQ], X[N1];
#pragma unroll
      for (int aa = 1; aa < N1; ++aa) PL0[aa] *= ih[0];
      gauss_derivatives<N1, NQ, 1, T>(tb, PL0, gx);
      gauss_values<N1, NQ, 1, T>(tb, PL1, gy);
#pragma unroll
      for (int qx = 0; qx < NQ; ++qx) {
        const T jly = jnv(1, 0, qx), jhy = jnv(1, 1, qx);
        const T avg[2] = {gx[qx] + tb.K0q[qx] * jlx + tb.K1q[qx] * jhx, gy[qx] + hK0k * jly + hK1k * jhy};
        T dif = tb.K0q[qx] * jlx;
        dif += hK0k * jly;
        dif -= tb.K1q[qx] * jhx;
        dif -= hK1k * jhy;
        f[qx] = hfun(stl[(size_t)(k * NQF + qx) * NT + cl], avg, dif);   // w_q H
      }
#pragma unroll
      for (int aa = 0; aa < N1; ++aa) X[aa] = T(0);
      gauss_project<N1, NQ, 1, T>(tb, f, X);
#pragma unroll
      for (int aa = 0; aa < N1; ++aa) ub[(size_t)(k * NQF + aa) * NT + cl] = X[aa];
    } else {
      T PLy[N1][N1];   // [aa][b >= 1], for the y derivative
#pragma unroll
      for (int aa = 0; aa < N1; ++aa)
#pragma unroll
        for (int b = 1; b < N1; ++b) PLy[aa][b] = PL0[aa + N1 * b] * ih[1];
#pragma unroll
      for (int aa = 1; aa < N1; ++aa)
#pragma unroll
        for (int b = 0; b < N1; ++b) PL0[aa + N1 * b] *= ih[0];
      T jly[NQ], jhy[NQ];
#pragma unroll
      for (int qx = 0; qx < NQ; ++qx) {
        jly[qx] = T(0.5) * jnv(1, 0, qx + NQ * k);
        jhy[qx] = T(0.5) * jnv(1, 1, qx + NQ * k);
      }
      T U[N1][N1];
#pragma unroll
      for (int aa = 0; aa < N1; ++aa)
#pragma unroll
        for (int b = 0; b < N1; ++b) U[aa][b] = T(0);
      auto line = [&](int qy, const T* Py, const T* Pdy, const T* Dzy) {
        T gx[NQ], gy[NQ], gz[NQ], f[NQ], X[N1];
        gauss_derivatives<N1, NQ, 1, T>(tb, Py, gx);
        gauss_values<N1, NQ, 1, T>(tb, Pdy, gy);
        gauss_values<N1, NQ, 1, T>(tb, Dzy, gz);
        const T jlx = T(0.5) * jnv(0, 0, qy + NQ * k), jhx = T(0.5) * jnv(0, 1, qy + NQ * k);
#pragma unroll
        for (int qx = 0; qx < NQ; ++qx) {
          const T jlz = jnv(2, 0, qx + NQ * qy), jhz = jnv(2, 1, qx + NQ * qy);
          const T avg[3] = {gx[qx] + tb.K0q[qx] * jlx + tb.K1q[qx] * jhx,
                            gy[qx] + tb.K0q[qy] * jly[qx] + tb.K1q[qy] * jhy[qx], gz[qx] + hK0k * jlz + hK1k * jhz};
          T dif = tb.K0q[qx] * jlx;
          dif += tb.K0q[qy] * jly[qx];
          dif += hK0k * jlz;
          dif -= tb.K1q[qx] * jhx;
          dif -= tb.K1q[qy] * jhy[qx];
          dif -= hK1k * jhz;
          f[qx] = hfun(stl[(size_t)(k * NQF + qx + NQ * qy) * NT + cl], avg, dif);   // w_q H
        }
#pragma unroll
        for (int aa = 0; aa < N1; ++aa) X[aa] = T(0);
        gauss_project<N1, NQ, 1, T>(tb, f, X);
#pragma unroll
        for (int aa = 0; aa < N1; ++aa) {
          U[aa][0] += X[aa];
#pragma unroll
          for (int b = 1; b < N1; ++b) U[aa][b] += X[aa] * tb.Lq[b][qy];
        }
      };
      T Py[N1][NQ], Pdy[N1][NQ], Dzy[N1][NQ];
#pragma unroll
      for (int aa = 0; aa < N1; ++aa) {
        if (aa > 0) gauss_values<N1, NQ, N1, T>(tb, PL0 + aa, Py[aa]);
        gauss_derivatives<N1, NQ, 1, T>(tb, PLy[aa], Pdy[aa]);
        gauss_values<N1, NQ, N1, T>(tb, PL1 + aa, Dzy[aa]);
      }
#pragma unroll
      for (int qy = 0; qy < NQ; ++qy) {
        T py[N1], pdy[N1], dzy[N1];
#pragma unroll
        for (int aa = 0; aa < N1; ++aa) {
          py[aa] = aa > 0 ? Py[aa][qy] : T(0);
          pdy[aa] = Pdy[aa][qy];
          dzy[aa] = Dzy[aa][qy];
        }
        line(qy, py, pdy, dzy);
      }
#pragma unroll
      for (int b = 0; b < N1; ++b)
#pragma unroll
        for (int aa = 0; aa < N1; ++aa) ub[(size_t)(k * NQF + aa + N1 * b) * NT + cl] = U[aa][b];
    }
  }
  __syncthreads();   // planes done: the face-jump area becomes the store staging
  if (threadIdx.x == 0) {   // the running maximum of the next step (the first block has put this one's)
    const double bm = slot_value(cfl) / m.diam;
    if (bm > vd) atomic_max_pos(&a.clk->hj_vd[(a.step.k + 1) % 3], bm);
  }
  const T dt = T(*sdt);

  // -------- columns u = k, k + NQ, ... of modes: project over the planes,
  // update, stage
  {
  T* sb = jn;   // [NT][NM]
  if (valid) {
    const long long cell = (long long)g[0] + (long long)m.n[0] * (g[1] + (long long)m.n[1] * g[2]);
#pragma unroll
    for (int u0 = 0; u0 < NU; u0 += NQ) {
      const int u = u0 + k;
      if (u < NU) {
        T f[NQ], R[N1];
#pragma unroll
        for (int kk = 0; kk < NQ; ++kk) f[kk] = ub[(size_t)(kk * NQF + u) * NT + cl];
#pragma unroll
        for (int cz = 0; cz < N1; ++cz) R[cz] = T(0);
        gauss_project<N1, NQ, 1, T>(tb, f, R);
#pragma unroll
        for (int cz = 0; cz < N1; ++cz) {
          const int q = u + NU * cz;
          T r = -R[cz];
          if (a.rdiff) r += a.rdiff[cell * NM + q];
          sb[(size_t)cl * NM + q] = hj_combine<T>(a.rk, c[q], r, dt);
        }
      }
    }
  }
  __syncthreads();
  chain_release();
  store_cells<DIM, TX, TY, TZ, NM, T>(m, sb, a.out, o[0], o[1], o[2]);
  }
}

template <int DIM, int P, typename T>
__global__ void __launch_bounds__(HjsTile<DIM>::N * (P + 2), hjs_min_blocks<DIM, P, T>())
    hjs_kernel(const HJArgs<T> a) {
  hjs_tile<DIM, P, T>(a, (int)blockIdx.x);
}

}  // namespace flsp
