// flsp_device.cuh — device-side building blocks shared by every kernel of
// libflsp_dg.so: 1D Legendre/Gauss tables in constant memory, the device
// clock, parameter blocks, small reduction helpers.
//
// Data layout in HBM: one array of n_cells * nb coefficients per state
// vector, cells lexicographic (x fastest), nb DoFs of a cell contiguous in
// deal.II order (FE_DGQLegendre lexicographic, FE_DGP total-degree order).
// Inside a CTA every cell is expanded to the Q layout of (p+1)^dim modes
// (zero where the P space has no mode), so one code path serves both bases.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace flsp {

constexpr int kMaxP = 3;
constexpr int kMaxN1 = kMaxP + 1;   // modes per axis
constexpr int kMaxNQ = kMaxP + 2;   // Gauss points per axis (p+2 rule)
constexpr int kMaxTerms = 24;
constexpr int kMaxFeVel = 3;        // largest degree of an FE velocity field

__host__ __device__ constexpr int ipow(int b, int e) { return e == 0 ? 1 : b * ipow(b, e - 1); }

// In-cell DoF index (HBM order) of Q-layout mode q for FE_DGP
// (PolynomialSpace order: c outer, b, a inner with a + b + c <= P), -1 for a
// mode outside P-space
template <int DIM, int P>
__host__ __device__ constexpr int q2g_ct(int q) {
  const int N1 = P + 1;
  const int a = q % N1, b = (q / N1) % N1, c = DIM > 2 ? q / (N1 * N1) : 0;
  if (a + b + c > P) return -1;
  int idx = 0;
  for (int cc = 0; cc < c; ++cc)
    for (int bb = 0; bb <= P - cc; ++bb) idx += P - bb - cc + 1;
  for (int bb = 0; bb < b; ++bb) idx += P - bb - c + 1;
  return idx + a;
}

// block of cells of the kernels that give a cell NQ threads (one per Gauss
// plane): fixed per dimension so that every shared-memory and table offset is
// a compile-time constant; a multiple of 32 cells keeps each warp on one plane
template <int DIM>
struct HjsTile {
  static constexpr int X = DIM == 2 ? 8 : 4, Y = DIM == 2 ? 8 : 4, Z = DIM == 2 ? 1 : 4;
  static constexpr int N = X * Y * Z;
};

// Velocity table of a problem (adv_tab_tile, flsp_advtab.cuh): per HjsTile,
// w_q u_d / h_d at the cells' QGauss(p+2) points, entry (d NQ^DIM + q) N +
// cell, then w_q u_E / h_E at the tile's faces' points, entry q NFT + off(E) +
// slot; faces normal to E in slots lx + EX (ly + EY lz) of a block with one
// more face than cells along E.
template <int DIM>
struct VelTabLayout {
  using TL = HjsTile<DIM>;
  static constexpr int S0 = (TL::X + 1) * TL::Y * TL::Z, S1 = TL::X * (TL::Y + 1) * TL::Z;
  static constexpr int S2 = DIM > 2 ? TL::X * TL::Y * (TL::Z + 1) : 0, NFT = S0 + S1 + S2;
  __host__ __device__ static constexpr int off(int E) { return E == 0 ? 0 : (E == 1 ? S0 : S0 + S1); }
  // entries of a tile
  __host__ __device__ static constexpr int entries(int nq) {
    return DIM * ipow(nq, DIM) * TL::N + ipow(nq, DIM - 1) * NFT;
  }
  template <int NQ>
  __host__ __device__ static constexpr int entries() { return entries(NQ); }
};

// 1D tables for one polynomial degree p (entries beyond p unused)
template <typename T>
struct Tab1D {
  T xq[kMaxNQ], wq[kMaxNQ];            // Gauss (p+2) points/weights on [0,1]
  T Lq[kMaxN1][kMaxNQ];                 // L_a(xq)
  T Dq[kMaxN1][kMaxNQ];                 // L_a'(xq)
  T Hq[kMaxN1][kMaxNQ];                 // L_a''(xq)
  T L0[kMaxN1], L1[kMaxN1];             // L_a(0), L_a(1)
  T D0[kMaxN1], D1[kMaxN1];             // L_a'(0), L_a'(1)
  T H0[kMaxN1], H1[kMaxN1];             // L_a''(0), L_a''(1)
  T A[kMaxN1][kMaxN1];                  // int_0^1 L_a' L_b
  T S[kMaxN1][kMaxN1];                  // int_0^1 L_a(x) L_b(x + 1)
  T xl[kMaxN1], wl[kMaxN1];             // Gauss (p+1) points/weights
  T Ll[kMaxN1][kMaxN1];                 // L_a(xl)
  T Dl[kMaxN1][kMaxN1];                 // L_a'(xl)
  // LDG lifting kernels K_s(x) = sum_a L_a(x) L_a(s), s = 0, 1, at the
  // Gauss (p+2) points and at x = 0, 1
  T K0q[kMaxNQ], K1q[kMaxNQ];
  T K0v[2], K1v[2];
};

// Every translation unit of the library holds its own copy of the tables
// (no relocatable device code); flsp_upload_tables_<unit>() fills it.
static __constant__ Tab1D<double> c_tab_d[kMaxP + 1];
static __constant__ Tab1D<float> c_tab_f[kMaxP + 1];

template <typename T> __device__ __forceinline__ const Tab1D<T>& tab(int p);
template <> __device__ __forceinline__ const Tab1D<double>& tab<double>(int p) { return c_tab_d[p]; }
template <> __device__ __forceinline__ const Tab1D<float>& tab<float>(int p) { return c_tab_f[p]; }

// ---------------------------------------------------------------------
// 1D Legendre sums by parity.  About the interval's centre L_a and the
// Gauss rule are even / odd (L_a(1 - x) = (-1)^a L_a(x), L_0 = 1, L_1'
// constant), so the points q and NQ-1-q share the even and the odd part of
// a sum: 3 modes to 4 points take 6 instructions instead of 12, their
// derivatives 5 instead of 12, 4 modes to 5 points 11 instead of 20.
// ---------------------------------------------------------------------
// v[q] = sum_a c[a S] L_a(x_q)
template <int N1, int NQ, int S, typename T>
__device__ __forceinline__ void gauss_values(const Tab1D<T>& tb, const T* c, T* v) {
  constexpr int H = NQ / 2;
#pragma unroll
  for (int q = 0; q < H; ++q) {
    T e = c[0];
    if constexpr (N1 > 2) e += c[2 * S] * tb.Lq[2][q];
    if constexpr (N1 > 3) {
      const T o = c[S] * tb.Lq[1][q] + c[3 * S] * tb.Lq[3][q];
      v[q] = e + o;
      v[NQ - 1 - q] = e - o;
    } else {
      v[q] = e + c[S] * tb.Lq[1][q];
      v[NQ - 1 - q] = e - c[S] * tb.Lq[1][q];
    }
  }
  if constexpr (NQ % 2) {
    T e = c[0];
    if constexpr (N1 > 2) e += c[2 * S] * tb.Lq[2][H];
    v[H] = e;
  }
}
// v[q] = sum_a c[a S] L_a'(x_q); c[0] is not read
template <int N1, int NQ, int S, typename T>
__device__ __forceinline__ void gauss_derivatives(const Tab1D<T>& tb, const T* c, T* v) {
  constexpr int H = NQ / 2;
  const T c1 = c[S] * tb.Dq[1][0];
#pragma unroll
  for (int q = 0; q < H; ++q) {
    T e = c1;
    if constexpr (N1 > 3) e += c[3 * S] * tb.Dq[3][q];
    if constexpr (N1 > 2) {
      v[q] = e + c[2 * S] * tb.Dq[2][q];
      v[NQ - 1 - q] = e - c[2 * S] * tb.Dq[2][q];
    } else {
      v[q] = e;
      v[NQ - 1 - q] = e;
    }
  }
  if constexpr (NQ % 2) {
    T e = c1;
    if constexpr (N1 > 3) e += c[3 * S] * tb.Dq[3][H];
    v[H] = e;
  }
}
// X[a S] += sum_q f[q] L_a(x_q), a < NA
template <int NA, int NQ, int S, typename T>
__device__ __forceinline__ void gauss_project(const Tab1D<T>& tb, const T* f, T* X) {
  constexpr int H = NQ / 2;
#pragma unroll
  for (int q = 0; q < H; ++q) {
    const T s = f[q] + f[NQ - 1 - q];
    X[0] += s;
    if constexpr (NA > 1) {
      const T d = f[q] - f[NQ - 1 - q];
      X[S] += d * tb.Lq[1][q];
      if constexpr (NA > 3) X[3 * S] += d * tb.Lq[3][q];
    }
    if constexpr (NA > 2) X[2 * S] += s * tb.Lq[2][q];
  }
  if constexpr (NQ % 2) {
    X[0] += f[H];
    if constexpr (NA > 2) X[2 * S] += f[H] * tb.Lq[2][H];
  }
}
// X[a] += sum_q f[q] L_a'(x_q), 1 <= a < NA
template <int NA, int NQ, typename T>
__device__ __forceinline__ void gauss_project_derivative(const Tab1D<T>& tb, const T* f, T* X) {
  constexpr int H = NQ / 2;
  T s1 = T(0);
#pragma unroll
  for (int q = 0; q < H; ++q) {
    const T s = f[q] + f[NQ - 1 - q];
    s1 += s;
    if constexpr (NA > 3) X[3] += s * tb.Dq[3][q];
    if constexpr (NA > 2) X[2] += (f[q] - f[NQ - 1 - q]) * tb.Dq[2][q];
  }
  if constexpr (NQ % 2) {
    s1 += f[H];
    if constexpr (NA > 3) X[3] += f[H] * tb.Dq[3][H];
  }
  X[1] += s1 * tb.Dq[1][0];
}
// the values at the interval's ends 0 and 1
template <int N1, int S, typename T>
__device__ __forceinline__ void end_values(const Tab1D<T>& tb, const T* c, T& lo, T& hi) {
  T e = c[0], o = T(0);
  if constexpr (N1 > 2) e += c[2 * S] * tb.L1[2];
  if constexpr (N1 > 3) {
    o = c[S] * tb.L1[1] + c[3 * S] * tb.L1[3];
    lo = e - o;
    hi = e + o;
  } else {
    lo = e - c[S] * tb.L1[1];
    hi = e + c[S] * tb.L1[1];
  }
}

// ---------------------------------------------------------------------
// Programmatic dependent launch (launch_chained, flsp_launch.h): a kernel of
// a chain touches nothing an earlier kernel writes, and leaves no block,
// before chain_wait: that returns once the kernel before has finished, and
// with it all before that.  chain_release, before a block's final stores, lets
// the next kernel's blocks start once every block has come so far; its launch
// latency and set-up then overlap the tail of this one.  (Released first thing
// instead, the waiting blocks of several kernels pile up beside the running
// one: a 256^2 Q2 FP32 run took 4.0 ms; 3.1 so, 3.4 without a chain.)
// ---------------------------------------------------------------------
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---------------------------------------------------------------------
// device clock: simulation time and CFL state live on the GPU so that a
// whole reinit period can be replayed from a CUDA graph without host
// synchronisation.  All fields in double (clocks are FP64 in both modes).
// ---------------------------------------------------------------------
struct DevClock {
  double t;          // time at the start of the current substep
  double dt;         // current substep
  double vd_run;     // running max of (max vertex |u|)/diam (never reset:
                     // the reference CFLEstimator keeps its maximum)
  double vd_static;  // max over vertices of |u_spatial| / diam
  int n_substeps;    // executed substeps
  // reinitialisation
  double hj_dt;      // last pseudo-step
  double hj_cum;     // accumulated pseudo-time
  // running maxima of the CFL estimate (atomicMax on the bit patterns):
  // pseudo-step k reads slot k % 3, accumulates slot (k + 1) % 3 and clears
  // slot (k + 2) % 3
  unsigned long long hj_vd[3];
  double scratch[2]; // length of the advance call, cumulative time in it
};

// one substep of the advection clock, computed ahead of its stages (the
// velocity is known in advance, so the clock needs nothing from the field)
struct AdvStep {
  double ct[3];      // velocity time factor at the RK stage times
  double dt, t;      // substep and its start time
  int active;        // the substep is non-zero
  int pad;
};
constexpr int kClockSteps = 32;   // substeps one clock launch computes at most

// stage combinations of the SSP-RK schemes (time_integration.implement.h:141-234)
enum CombineMode : int {
  kRhsOnly = 0,     // out = phidot
  kRK1 = 1,         // out = phidot*dt + phi
  kRK2a = 2,        // out = phi + dt*phidot
  kRK2b = 3,        // out = (phi1 + dt*phidot + phin) * 0.5
  kRK3a = 4,        // out = phi + dt*phidot
  kRK3b = 5,        // out = (phi1 + dt*phidot + 3 phin) * 0.25
  kRK3c = 6         // out = ((phi2 + dt*phidot) * 2 + phin) * (1/3)
};

// modes of the reinitialisation kernel
enum HJMode : int { kHJCflOnly = 0, kHJStep = 1, kHJGradients = 2 };

// advection clock parameters (scale = AdvectSimulator::cfl_scaling(p))
struct AdvClockArgs {
  double cfl_max, scale;
  int tkind;
  double ta, tb;
  int step_count;   // 1: a step-count run (the horizon only caps the time)
};

// reinitialisation clock: pseudo-step k of size cfl_max / (scale vd + shift),
// vd the running maximum of the CFL estimate
struct HjClockArgs {
  double cfl_max, scale, shift;
  int k;
};

// time factor kinds (flsp_time_kind)
__device__ __forceinline__ double time_factor(int kind, double a, double b, double t) {
  switch (kind) {
    case 1: return cos(a * t + b);
    case 2: return cospi(a * t + b);
    case 3: return 1.0 - exp(-a * t);
    default: return 1.0;
  }
}

// positive doubles compare like their bit patterns
__device__ __forceinline__ void atomic_max_pos(unsigned long long* slot, double v) {
  if (!(v > 0.0)) return;
  atomicMax(slot, (unsigned long long)__double_as_longlong(v));
}

// 1 / sqrt(x) for x >= 1e-30 by the PTX instruction rsqrt.approx.ftz.f32: relative
// error at most 2^-22.9 over the positive finite numbers (PTX ISA, rsqrt); .ftz takes
// a subnormal input as zero, which the caller's range excludes.  rsqrtf gave the same
// bits in every run compared and took longer: 64^3 Q2 FP32 run 22.97 against 22.81 ms,
// band reinitialisation of 56 x 64 x 48 6.84 against 6.77.
__device__ __forceinline__ float rsqrt_normal(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

template <typename T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// max of a non-negative value over a warp, NaN counting as zero; into the
// shared slot of the block (atomics on the bit patterns), which starts at 0
__device__ __forceinline__ void slot_max(unsigned int* slot, float v) {
  const unsigned int u = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(v, 0.f)));
  if ((threadIdx.x & 31) == 0) atomicMax(slot, u);
}
__device__ __forceinline__ void slot_max(unsigned long long* slot, double v) {
  v = warp_max(fmax(v, 0.0));
  if ((threadIdx.x & 31) == 0) atomicMax(slot, (unsigned long long)__double_as_longlong(v));
}
__device__ __forceinline__ double slot_value(const unsigned int* slot) { return (double)__uint_as_float(*slot); }
__device__ __forceinline__ double slot_value(const unsigned long long* slot) {
  return __longlong_as_double((long long)*slot);
}
template <typename T>
using MaxSlot = std::conditional_t<sizeof(T) == 4, unsigned int, unsigned long long>;

// block-wide max of a non-negative double, result valid in thread 0
__device__ __forceinline__ double block_max(double v, double* red) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    double x = l < nw ? red[l] : 0.0;
    x = warp_max(x);
    if (l == 0) red[0] = x;
  }
  __syncthreads();
  return red[0];
}

// ---------------------------------------------------------------------
// mesh / tile description passed by value to every stencil kernel
// ---------------------------------------------------------------------
struct MeshArgs {
  int n[3];          // cells per axis (1 for unused axes)
  long long ncell;
  double lo[3], h[3];
  double vol, diam, min_diam;
  int nb;            // DoFs per cell in HBM
  signed char q2g[64];  // Q-layout mode -> in-cell DoF index (-1: absent)
  signed char g2q[64];  // in-cell DoF index -> Q-layout mode
  int tile[3];       // CTA tile in cells
  int ntile[3];      // tiles per axis
  // compute-restricted narrow band: block b serves tile tiles[b]; blocks
  // at or past *n_tiles have no tile (null: block b serves tile b)
  const int* tiles;
  const int* n_tiles;
  // Dirichlet value of every domain-boundary face (NaN: none, the face
  // keeps the zero-Neumann interior trace); null: no Dirichlet face.
  // Faces side by side (x-, x+, y-, y+, z-, z+), each side's faces
  // lexicographic in the other axes (lower axis fastest).
  const double* bc_face;
};

// boundary faces on the sides before side (E, S) and within it
template <int DIM>
__host__ __device__ __forceinline__ long long bc_side_faces(const MeshArgs& m, int E) {
  const int t0 = E == 0 ? 1 : 0, t1 = E == 2 ? 1 : 2;
  return (long long)m.n[t0] * (DIM > 2 ? m.n[t1] : 1);
}

// Dirichlet value g on the domain-boundary face on side S (0: lower, 1:
// upper) of axis E of the cell at lattice position c, when the face's
// boundary id carries one: the exterior trace there is the constant g, a
// face polynomial with g in the constant mode and zeros elsewhere
// (inflow of advection.implement.h:719-741; LDG left / right gradients,
// ldg.cc:551-620 and :686-740).  False: zero-Neumann (interior trace).
template <int DIM, typename T>
__device__ __forceinline__ bool bc_dirichlet(const MeshArgs& m, int E, int S, const int* c, T& g) {
  if (!m.bc_face) return false;
  long long off = 0;
#pragma unroll
  for (int e = 0; e < DIM; ++e)
    if (e < E) off += 2 * bc_side_faces<DIM>(m, e);
  const int t0 = E == 0 ? 1 : 0, t1 = E == 2 ? 1 : 2;
  off += S * bc_side_faces<DIM>(m, E) + c[t0] + (DIM > 2 ? (long long)m.n[t0] * c[t1] : 0);
  const double v = m.bc_face[off];
  if (v != v) return false;   // NaN: no Dirichlet value on this face
  g = T(v);
  return true;
}

// separable velocity: vtab[((k*3 + axis) * nmax + i) * npt + j]
// j < NQ: Gauss (p+2) point j of cell i; j == NQ: xi = 0; j == NQ+1: xi = 1
template <typename T>
struct VelArgs {
  const T* vtab;
  int n_terms;
  int nmax;
  int npt;
  int comp[kMaxTerms];
  int cstart[4];   // terms of component c: [cstart[c], cstart[c+1]) (terms sorted by component)
};

// first term of each component in a component-sorted term list
__host__ __device__ inline void term_ranges(const int* comp, int n_terms, int* cstart) {
  for (int c = 0; c < 4; ++c) {
    int k = 0;
    while (k < n_terms && comp[k] < c) ++k;
    cstart[c] = k;
  }
}

// next 16-byte aligned address at or after p (shared-memory sub-buffers)
template <typename U>
__device__ __forceinline__ U* align16(void* p) {
  return reinterpret_cast<U*>((reinterpret_cast<uintptr_t>(p) + 15) & ~uintptr_t(15));
}

// local (tile) coordinates of the thread's cell
struct TileCoord {
  int lx, ly, lz;     // in [0, tile)
  int gx, gy, gz;     // global lattice coordinates
  bool valid;
  int ox, oy, oz;     // tile origin
};

// a launch slot (the block index of a plain launch, a work item of a
// persistent one) with no tile to serve in a narrow-band launch (uniform per block)
__device__ __forceinline__ bool tile_inactive(const MeshArgs& m, int slot) {
  return m.tiles != nullptr && slot >= *m.n_tiles;
}

// tile of launch slot `slot` and this thread's cell in it
__device__ __forceinline__ TileCoord tile_coord(const MeshArgs& m, int dim, int slot) {
  TileCoord c;
  int b = m.tiles ? m.tiles[slot] : slot;
  const int bx = b % m.ntile[0];
  b /= m.ntile[0];
  const int by = dim > 1 ? b % m.ntile[1] : 0;
  const int bz = dim > 2 ? b / m.ntile[1] : 0;
  c.ox = bx * m.tile[0];
  c.oy = by * m.tile[1];
  c.oz = bz * m.tile[2];
  int t = threadIdx.x;
  c.lx = t % m.tile[0];
  t /= m.tile[0];
  c.ly = dim > 1 ? t % m.tile[1] : 0;
  c.lz = dim > 2 ? t / m.tile[1] : 0;
  c.gx = c.ox + c.lx;
  c.gy = c.oy + c.ly;
  c.gz = c.oz + c.lz;
  c.valid = (int)threadIdx.x < m.tile[0] * m.tile[1] * m.tile[2] && c.gx < m.n[0] &&
            c.gy < m.n[1] && c.gz < m.n[2];
  return c;
}

__device__ __forceinline__ bool tile_inactive(const MeshArgs& m) { return tile_inactive(m, (int)blockIdx.x); }
__device__ __forceinline__ TileCoord tile_coord(const MeshArgs& m, int dim) { return tile_coord(m, dim, (int)blockIdx.x); }

// padded smem box (tile + 1 halo layer per axis, edge/corner slots unused)
__device__ __forceinline__ int box_index(const MeshArgs& m, int dim, int lx, int ly, int lz) {
  const int bx = m.tile[0] + 2, by = dim > 1 ? m.tile[1] + 2 : 1;
  return (lx + 1) + bx * ((dim > 1 ? ly + 1 : 0) + by * (dim > 2 ? lz + 1 : 0));
}

__device__ __forceinline__ int box_cells(const MeshArgs& m, int dim) {
  return (m.tile[0] + 2) * (dim > 1 ? m.tile[1] + 2 : 1) * (dim > 2 ? m.tile[2] + 2 : 1);
}

// Store of a compile-time tile's cells from [cell][NE] smem to NE DoFs per
// cell in HBM, one warp per row of cells.
template <int DIM, int TX, int TY, int TZ, int NE, typename T>
__device__ __forceinline__ void store_cells(const MeshArgs& m, const T* __restrict__ sm, T* __restrict__ g, int ox,
                                            int oy, int oz) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int n = min(TX, m.n[0] - ox) * NE;
  for (int r = warp; r < TY * TZ; r += nw) {
    const int gy = oy + r % TY, gz = oz + r / TY;
    if (gy >= m.n[1] || gz >= m.n[2]) continue;
    T* dst = g + ((long long)m.n[0] * (gy + (long long)m.n[1] * gz) + ox) * NE;
    const T* src = sm + (size_t)TX * r * NE;
#pragma unroll
    for (int e = lane; e < TX * NE; e += 32)
      if (e < n) dst[e] = src[e];
  }
}

// ---------------------------------------------------------------------
// asynchronous global -> shared copies (cp.async, one element each): a
// thread issues all of its copies before waiting, so the latency of every
// row of a tile overlaps instead of serialising row by row
// ---------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void cp_async_elem(T* smem, const T* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  if constexpr (sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Load of the tile and its face halo (no edges/corners) from a cell-major
// vector into the smem box, expanded to the Q layout.  One warp per row of
// cells along x (contiguous in HBM), lanes over the row's elements.  Slots
// of cells outside the domain are not written (boundary faces never read
// them).  Completes with cp_async_wait_all() + __syncthreads() by the caller.
template <int DIM, int NM, typename T>
__device__ __forceinline__ void load_box(const MeshArgs& m, const T* __restrict__ g,
                                         T* __restrict__ sm, int ox, int oy, int oz,
                                         bool with_halo) {
  const int tx = m.tile[0], ty = DIM > 1 ? m.tile[1] : 1, tz = DIM > 2 ? m.tile[2] : 1;
  const int h = with_halo ? 1 : 0;
  const int nry = ty + 2 * (DIM > 1 ? h : 0), nrz = tz + 2 * (DIM > 2 ? h : 0);
  const int ly0 = DIM > 1 ? -h : 0, lz0 = DIM > 2 ? -h : 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const bool dense = m.nb == NM;   // Q basis: smem row == HBM row
  for (int r = warp; r < nry * nrz; r += nw) {
    const int ly = ly0 + r % nry, lz = lz0 + r / nry;
    const bool yout = ly < 0 || ly >= ty, zout = lz < 0 || lz >= tz;
    if (yout && zout) continue;
    const int gy = oy + ly, gz = oz + lz;
    if (gy < 0 || gy >= m.n[1] || gz < 0 || gz >= m.n[2]) continue;
    const int lx0 = (!yout && !zout) ? -h : 0;
    const int lx1 = (!yout && !zout) ? tx + h : tx;
    const int gx0 = max(ox + lx0, 0), gx1 = min(ox + lx1, m.n[0]);
    if (gx1 <= gx0) continue;
    const long long rowcell = (long long)m.n[0] * (gy + (long long)m.n[1] * gz);
    T* dst = sm + (size_t)box_index(m, DIM, gx0 - ox, ly, lz) * NM;
    const int count = (gx1 - gx0) * NM;
    if (dense) {
      const T* src = g + (rowcell + gx0) * NM;
      for (int e = lane; e < count; e += 32) cp_async_elem(dst + e, src + e);
    } else {
      const T* src = g + (rowcell + gx0) * m.nb;
      for (int e = lane; e < count; e += 32) {
        const int cx = e / NM, q = e - cx * NM;
        const int gi = m.q2g[q];
        if (gi >= 0) cp_async_elem(dst + e, src + (long long)cx * m.nb + gi);
        else dst[e] = T(0);
      }
    }
  }
}

// Load of the tile's own cells (no halo) into [cell][NM] (stride = NM) or,
// with transposed = true, into [NM][ld] (column = tile cell index).
template <int DIM, int NM, typename T>
__device__ __forceinline__ void load_tile(const MeshArgs& m, const T* __restrict__ g,
                                          T* __restrict__ sm, int ox, int oy, int oz,
                                          bool transposed, int ld) {
  const int tx = m.tile[0], ty = DIM > 1 ? m.tile[1] : 1, tz = DIM > 2 ? m.tile[2] : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int r = warp; r < ty * tz; r += nw) {
    const int ly = r % ty, lz = r / ty;
    const int gy = oy + ly, gz = oz + lz;
    const int nx = min(tx, m.n[0] - ox);
    const int cl0 = tx * r;
    const int count = nx * NM;
    if (gy >= m.n[1] || gz >= m.n[2] || nx <= 0) {
      for (int e = lane; e < tx * NM; e += 32) {
        const int cx = e / NM, q = e - cx * NM;
        if (transposed) sm[(size_t)q * ld + cl0 + cx] = T(0);
        else sm[(size_t)(cl0 + cx) * NM + q] = T(0);
      }
      continue;
    }
    const T* src = g + ((long long)m.n[0] * (gy + (long long)m.n[1] * gz) + ox) * m.nb;
    for (int e = lane; e < count; e += 32) {
      const int cx = e / NM, q = e - cx * NM;
      const int gi = m.q2g[q];
      T* d = transposed ? sm + (size_t)q * ld + cl0 + cx : sm + (size_t)(cl0 + cx) * NM + q;
      if (gi >= 0) cp_async_elem(d, src + (long long)cx * m.nb + gi);
      else *d = T(0);
    }
    for (int e = count + lane; e < tx * NM; e += 32) {   // cells past the domain edge
      const int cx = e / NM, q = e - cx * NM;
      if (transposed) sm[(size_t)q * ld + cl0 + cx] = T(0);
      else sm[(size_t)(cl0 + cx) * NM + q] = T(0);
    }
  }
}

// Store of the tile's own cells from [cell][NM] smem to HBM (nb DoFs per
// cell, g2q maps them to the Q slots), one warp per row.
template <int DIM, int NM, typename T>
__device__ __forceinline__ void store_tile(const MeshArgs& m, const T* __restrict__ sm,
                                           T* __restrict__ g, int ox, int oy, int oz) {
  const int tx = m.tile[0], ty = DIM > 1 ? m.tile[1] : 1, tz = DIM > 2 ? m.tile[2] : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const bool dense = m.nb == NM;
  for (int r = warp; r < ty * tz; r += nw) {
    const int ly = r % ty, lz = r / ty;
    const int gy = oy + ly, gz = oz + lz;
    const int nx = min(tx, m.n[0] - ox);
    if (gy >= m.n[1] || gz >= m.n[2] || nx <= 0) continue;
    T* dst = g + ((long long)m.n[0] * (gy + (long long)m.n[1] * gz) + ox) * m.nb;
    const T* src = sm + (size_t)tx * r * NM;
    if (dense) {
      for (int e = lane; e < nx * NM; e += 32) dst[e] = src[e];
    } else {
      for (int e = lane; e < nx * m.nb; e += 32) {
        const int cx = e / m.nb, k = e - cx * m.nb;
        dst[e] = src[(size_t)cx * NM + m.g2q[k]];
      }
    }
  }
}

// ---------------------------------------------------------------------
// Bulk asynchronous copies (TMA engine, cp.async.bulk) completing on a
// shared-memory mbarrier.  Copies are plain global -> own-CTA shared
// memory: no cluster multicast.  Both addresses 16-byte aligned, size a
// multiple of 16.
// ---------------------------------------------------------------------
constexpr int kErrCopyTimeout = 1;   // bit of a problem's error word: a bulk-copy wait ran out
constexpr int kOpRowPad = 32;        // operator-table rows past the mesh per (d, e) block
constexpr int kStatePad = 256;       // bytes past the end of every state buffer

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
// one arrival that also announces the bytes the phase waits for
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// 16-byte aligned address, size a multiple of 16
__device__ __forceinline__ void bulk_prefetch_l2(const void* src, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(src), "r"(bytes) : "memory");
}
// Halo box of the TX x TY x TZ tile at (ox, oy, oz), HL cells wide, as rows of
// cells along x: row (ly, lz) holds cells [max(ox - HL, 0), min(ox + TX + HL, n))
// of NMB bytes from the 16-byte aligned address at or below the first, in slot
// (ly + HL) + BY (lz + HL) of SLOT bytes; rows outside the mesh and edge rows
// are left out.  One bulk copy per row, issued by the lanes of one warp: 32
// arrivals on the barrier, each announcing its lane's bytes.
template <int DIM, int TX, int TY, int TZ, int NMB, int SLOT, int HL = 1>
__device__ __forceinline__ void bulk_box_rows(const MeshArgs& m, const void* g, unsigned char* box, int ox, int oy,
                                              int oz, unsigned long long* bar) {
  constexpr int BY = TY + 2 * HL, NROWS = BY * (DIM > 2 ? TZ + 2 * HL : 1);
  const char* src = reinterpret_cast<const char*>(g);
  const int hx0 = max(ox - HL, 0), hx1 = min(ox + TX + HL, m.n[0]);
  unsigned bytes = 0;
  for (int rr = threadIdx.x & 31; rr < NROWS; rr += 32) {
    const int ly = rr % BY - HL, lz = DIM > 2 ? rr / BY - HL : 0;
    const bool yout = ly < 0 || ly >= TY, zout = DIM > 2 && (lz < 0 || lz >= TZ);
    if (yout && zout) continue;
    const int gy = oy + ly, gz = oz + lz;
    if (gy < 0 || gy >= m.n[1] || (DIM > 2 && (gz < 0 || gz >= m.n[2]))) continue;
    const long long rowcell = (long long)m.n[0] * (gy + (long long)m.n[1] * (DIM > 2 ? gz : 0));
    const long long a0 = ((rowcell + hx0) * NMB) & ~15LL, a1 = ((rowcell + hx1) * NMB + 15) & ~15LL;
    bulk_g2s(box + (size_t)rr * SLOT, src + a0, (unsigned)(a1 - a0), bar);
    bytes += (unsigned)(a1 - a0);
  }
  mbar_arrive_expect_tx(bar, bytes);
}
// Wait for phase `parity` of the barrier, at most max_iter polls (each
// try_wait may itself suspend for a while); false when it ran out.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, int max_iter) {
  const unsigned a = smem_u32(bar);
  for (int it = 0; it < max_iter; ++it) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

}  // namespace flsp
