// flsp_misc.cuh — small kernels around the two stencil kernels: device
// clocks, host<->device DoF order, initial-condition projection, FP64
// diagnostics reductions, the static part of the advection CFL.
#pragma once
#include "flsp_clock.cuh"
#include "flsp_device.cuh"
#include "flsp_dg.h"

namespace flsp {

constexpr double kPiD = 3.14159265358979323846;
constexpr double kEpsD = 2.220446049250313e-16;

// ---------------------------------------------------------------------
// clocks
// ---------------------------------------------------------------------

// clock kernels (the updates are in flsp_clock.cuh)
// the next n substeps (one warp); horizon >= 0 starts an advance call of that
// length first
__global__ void adv_clock_steps(DevClock* c, const AdvClockArgs a, AdvStep* st, int n, int commit, double horizon) {
  chain_wait();
  if (horizon >= 0.0 && threadIdx.x == 0) adv_clock_horizon_body(c, horizon);
  adv_clock_steps_body(c, a, st, n, commit != 0);
}
__global__ void adv_clock_horizon(DevClock* c, double time_step) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  adv_clock_horizon_body(c, time_step);
}
__global__ void hj_clock_reset(DevClock* c) {
  chain_wait();
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  hj_clock_reset_body(c);
}
// ---------------------------------------------------------------------
// host DoF order <-> device layout (optional cell permutation)
// ---------------------------------------------------------------------
// count: the non-finite values written
template <typename T>
__global__ void scatter_state(const double* __restrict__ src, T* __restrict__ dst,
                              const int64_t* __restrict__ perm, long long ncell, int nb, unsigned int* count) {
  const long long n = ncell * nb;
  unsigned int bad = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    long long o = i;
    if (perm) {
      const long long k = i / nb;
      o = perm[k] * nb + (i - k * nb);
    }
    const T v = T(src[i]);
    if (!isfinite((double)v)) ++bad;
    dst[o] = v;
  }
  if (bad) atomicAdd(count, bad);
}

template <typename T>
__global__ void gather_state(const T* __restrict__ src, double* __restrict__ dst,
                             const int64_t* __restrict__ perm, long long ncell, int nb) {
  const long long n = ncell * nb;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    long long o = i;
    if (perm) {
      const long long k = i / nb;
      o = perm[k] * nb + (i - k * nb);
    }
    dst[i] = double(src[o]);
  }
}

// ---------------------------------------------------------------------
// initial conditions (src/level_set/geometry.cc:17-235, geometry.h:80-160)
// nodes are evaluated in index order; children precede their parents
// ---------------------------------------------------------------------
__device__ inline double ic_eval(const flsp_ic_desc* ic, int dim, const double* x) {
  double val[FLSP_MAX_IC_NODES];
  for (int k = 0; k < ic->n_nodes; ++k) {
    const flsp_ic_node& nd = ic->nodes[k];
    double r = 0.0;
    switch (nd.kind) {
      case FLSP_IC_SPHERE: {
        double s = 0.0;
        for (int d = 0; d < dim; ++d) { const double e = x[d] - nd.p[d]; s += e * e; }
        r = sqrt(s) - nd.p[3];
        break;
      }
      case FLSP_IC_RECT: {
        double out2 = 0.0;
        bool inside = true;
        for (int d = 0; d < dim; ++d) {
          double e = 0.0;
          if (x[d] < nd.p[d]) { e = x[d] - nd.p[d]; inside = false; }
          else if (x[d] > nd.p[3 + d]) { e = x[d] - nd.p[3 + d]; inside = false; }
          out2 += e * e;
        }
        if (!inside) { r = sqrt(out2); break; }
        double mm = -1e300;
        for (int d = 0; d < dim; ++d) {
          mm = fmax(mm, nd.p[d] - x[d]);
          mm = fmax(mm, x[d] - nd.p[3 + d]);
        }
        r = mm;
        break;
      }
      case FLSP_IC_HEIGHT: {
        const int ax = (int)nd.p[0];
        int u = -1, v = -1;
        for (int d = 0; d < dim; ++d)
          if (d != ax) { if (u < 0) u = d; else v = d; }
        double hgt = nd.p[1];
        for (int w = 0; w < ic->n_waves; ++w) {
          double arg = ic->waves[w][1] * x[u];
          if (v >= 0) arg += ic->waves[w][2] * x[v];
          hgt += ic->waves[w][0] * cos(2.0 * kPiD * arg + ic->waves[w][3]);
        }
        r = x[ax] - hgt;
        break;
      }
      case FLSP_IC_UNION: r = fmin(val[nd.a], val[nd.b]); break;
      case FLSP_IC_DIFF: r = fmax(val[nd.a], -val[nd.b]); break;
      case FLSP_IC_INTERSECT: r = fmax(val[nd.a], val[nd.b]); break;
    }
    val[k] = r;
  }
  return val[ic->root];
}

// evaluate the DG function of one cell at reference point (table columns)
template <int DIM, int P>
__device__ __forceinline__ double eval_modal(const double* c, const double* bx, const double* by,
                                             const double* bz) {
  constexpr int N1 = P + 1;
  double s = 0.0;
  if constexpr (DIM == 2) {
#pragma unroll
    for (int b = 0; b < N1; ++b) {
      double r = 0.0;
#pragma unroll
      for (int a = 0; a < N1; ++a) r += c[a + N1 * b] * bx[a];
      s += r * by[b];
    }
  } else {
#pragma unroll
    for (int cc = 0; cc < N1; ++cc)
#pragma unroll
      for (int b = 0; b < N1; ++b) {
        double r = 0.0;
#pragma unroll
        for (int a = 0; a < N1; ++a) r += c[a + N1 * (b + N1 * cc)] * bx[a];
        s += r * by[b] * bz[cc];
      }
  }
  return s;
}

// L2 projection with QGauss(p+2) (advection.cc:145-161); always in FP64
template <int DIM, int P, typename T>
__global__ void project_ic_kernel(const MeshArgs m, const flsp_ic_desc* __restrict__ ic,
                                  T* __restrict__ out) {
  constexpr int N1 = P + 1, NQ = P + 2, NM = ipow(N1, DIM);
  const Tab1D<double>& tb = c_tab_d[P];
  const long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (cell >= m.ncell) return;
  const int gx = (int)(cell % m.n[0]);
  const int gy = (int)((cell / m.n[0]) % m.n[1]);
  const int gz = DIM > 2 ? (int)(cell / ((long long)m.n[0] * m.n[1])) : 0;
  const double x0[3] = {m.lo[0] + gx * m.h[0], m.lo[1] + gy * m.h[1], DIM > 2 ? m.lo[2] + gz * m.h[2] : 0.0};
  double R[NM];
#pragma unroll
  for (int q = 0; q < NM; ++q) R[q] = 0.0;
  const int nqz = DIM > 2 ? NQ : 1;
  for (int qz = 0; qz < nqz; ++qz)
    for (int qy = 0; qy < NQ; ++qy)
      for (int qx = 0; qx < NQ; ++qx) {
        double x[3] = {x0[0] + m.h[0] * tb.xq[qx], x0[1] + m.h[1] * tb.xq[qy],
                       DIM > 2 ? x0[2] + m.h[2] * tb.xq[qz] : 0.0};
        double f = ic_eval(ic, DIM, x);
        double w = tb.wq[qx] * tb.wq[qy];
        if (DIM > 2) w *= tb.wq[qz];
        const double fw = f * w;
#pragma unroll
        for (int q = 0; q < NM; ++q) {
          const int i0 = q % N1, i1 = (q / N1) % N1, i2 = q / (N1 * N1);
          double bw = tb.Lq[i0][qx] * tb.Lq[i1][qy];
          if (DIM > 2) bw *= tb.Lq[i2][qz];
          R[q] += fw * bw;
        }
      }
  for (int k = 0; k < m.nb; ++k) out[cell * m.nb + k] = T(R[m.g2q[k]]);
}

// ---------------------------------------------------------------------
// static CFL part: max over cells and vertices of |u_spatial| / diam
// (CFLEstimator::local_estimate, pde_tools.implement.h:44-57)
// ---------------------------------------------------------------------
template <int DIM>
__global__ void static_cfl_kernel(const MeshArgs m, const VelArgs<double> v, DevClock* clk) {
  __shared__ double red[32];
  const long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  double best = 0.0;
  if (cell < m.ncell) {
    const int g[3] = {(int)(cell % m.n[0]), (int)((cell / m.n[0]) % m.n[1]),
                      DIM > 2 ? (int)(cell / ((long long)m.n[0] * m.n[1])) : 0};
    const int NQ = v.npt - 2;
    for (int vv = 0; vv < (1 << DIM); ++vv) {
      double u[3] = {0.0, 0.0, 0.0};
      for (int k = 0; k < v.n_terms; ++k) {
        double tv = 1.0;
        for (int d = 0; d < DIM; ++d) {
          const int j = NQ + ((vv >> d) & 1);
          tv *= v.vtab[((size_t)(k * 3 + d) * v.nmax + g[d]) * v.npt + j];
        }
        u[v.comp[k]] += tv;
      }
      double s = 0.0;
      for (int d = 0; d < DIM; ++d) s += u[d] * u[d];
      best = fmax(best, sqrt(s));
    }
    best /= m.diam;
  }
  const double bm = block_max(best, red);
  if (threadIdx.x == 0) {
    unsigned long long* slot = reinterpret_cast<unsigned long long*>(&clk->vd_static);
    atomic_max_pos(slot, bm);
  }
}

// the same estimate for an FE velocity lattice of degree pv (fe_n* nodes per
// axis, FP64): a cell's vertex velocities are its corner nodes
template <int DIM>
__global__ void fe_static_cfl_kernel(const MeshArgs m, const double* __restrict__ u, int pv, int nx, int ny,
                                     int nz, DevClock* clk) {
  __shared__ double red[32];
  const long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  double best = 0.0;
  if (cell < m.ncell) {
    const int g[3] = {(int)(cell % m.n[0]), (int)((cell / m.n[0]) % m.n[1]),
                      DIM > 2 ? (int)(cell / ((long long)m.n[0] * m.n[1])) : 0};
    const size_t nn = (size_t)nx * ny * nz;
    for (int vv = 0; vv < (1 << DIM); ++vv) {
      const int x = pv * (g[0] + (vv & 1)), y = pv * (g[1] + ((vv >> 1) & 1));
      const int z = DIM > 2 ? pv * (g[2] + ((vv >> 2) & 1)) : 0;
      const size_t node = ((size_t)z * ny + y) * nx + x;
      double s = 0.0;
      for (int d = 0; d < DIM; ++d) s += u[d * nn + node] * u[d * nn + node];
      best = fmax(best, sqrt(s));
    }
    best /= m.diam;
  }
  const double bm = block_max(best, red);
  if (threadIdx.x == 0) {
    unsigned long long* slot = reinterpret_cast<unsigned long long*>(&clk->vd_static);
    atomic_max_pos(slot, bm);
  }
}

struct VelTerms {
  int cstart[4];
};

// position of entry i of a velocity table (VelTabLayout): a cell's point
// (component d, point q, cell g) or a face's (component d = E, point q, face
// index g over the n + e_E faces); false for entries past the mesh
template <int DIM>
__device__ __forceinline__ bool vel_tab_entry(const MeshArgs& m, int nq, long long i, bool& face, int& d, int& q,
                                              int* g) {
  using LY = VelTabLayout<DIM>;
  using TL = HjsTile<DIM>;
  const int nqd = DIM > 2 ? nq * nq * nq : nq * nq, per = LY::entries(nq);
  const long long tile = i / per;
  int r = (int)(i - tile * per);
  const int ntx = (m.n[0] + TL::X - 1) / TL::X, nty = (m.n[1] + TL::Y - 1) / TL::Y;
  const int o[3] = {(int)(tile % ntx) * TL::X, (int)((tile / ntx) % nty) * TL::Y,
                    DIM > 2 ? (int)(tile / ((long long)ntx * nty)) * TL::Z : 0};
  face = r >= DIM * nqd * TL::N;
  int ex = TL::X, ey = TL::Y, s;
  if (!face) {
    s = r % TL::N;
    q = (r / TL::N) % nqd;
    d = r / (TL::N * nqd);
  } else {
    r -= DIM * nqd * TL::N;
    s = r % LY::NFT;
    q = r / LY::NFT;
    d = s < LY::S0 ? 0 : (s < LY::S0 + LY::S1 ? 1 : 2);
    s -= LY::off(d);
    ex += d == 0;
    ey += d == 1;
  }
  g[0] = o[0] + s % ex;
  g[1] = o[1] + (s / ex) % ey;
  g[2] = DIM > 2 ? o[2] + s / (ex * ey) : 0;
  bool in = true;
#pragma unroll
  for (int e = 0; e < DIM; ++e) in = in && g[e] < m.n[e] + (face && d == e);
  return in;
}

// the table of a sum of separable terms: ((coeff f0) f1) f2 of the term
// tables' entries, the component's terms in order, times the quadrature weight
// over h, in FP64, stored in T; a face from its lower cell's upper-face entries
// (the first face: the upper cell's lower-face entries, the same face
// coordinate bit for bit)
template <int DIM, typename T>
__global__ void vel_tabulate(const MeshArgs m, const double* __restrict__ vtab, int nmax, int npt, const VelTerms vt,
                             int nq, long long total, T* __restrict__ out) {
  const double* wq = tab<double>(nq - 2).wq;
  auto row = [&](int k, int ax, int i) { return vtab + ((size_t)(k * 3 + ax) * nmax + i) * npt; };
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    bool face;
    int d, q, g[3];
    if (!vel_tab_entry<DIM>(m, nq, i, face, d, q, g)) continue;
    int j[3] = {0, 0, 0};
    double w = 1.0 / m.h[d];
#pragma unroll
    for (int e = 0; e < DIM; ++e) {
      if (face && e == d) {
        if (g[e] > 0) { g[e] -= 1; j[e] = nq + 1; }
        else j[e] = nq;
        continue;
      }
      j[e] = q % nq;
      q /= nq;
      w *= wq[j[e]];
    }
    double u = 0.0;
    for (int k = vt.cstart[d]; k < vt.cstart[d + 1]; ++k) {
      double v = row(k, 0, g[0])[j[0]] * row(k, 1, g[1])[j[1]];
      if (DIM == 3) v = v * row(k, 2, g[2])[j[2]];
      u += v;
    }
    out[i] = T(u * w);
  }
}

struct FeBasis {
  double b[kMaxFeVel + 1][kMaxNQ + 2];   // Lagrange basis a at Gauss point q
};

// The table of an FE velocity of degree PV, sums over the nodes factorised,
// FP64, stored in T.  Cells: one thread per (component, plane of points,
// cell), the plane's sum over the nodes along the last axis, then line by
// line; a coupled run makes the table anew every outer step (48^3 Q2 FP32,
// degree 2: 47 us for the cells; 367 us point by point).
template <int DIM, int P, int PV, typename T>
__global__ void fe_tabulate_cells(const MeshArgs m, const double* __restrict__ u, const FeBasis fb,
                                  long long total, T* __restrict__ out) {
  using LY = VelTabLayout<DIM>;
  using TL = HjsTile<DIM>;
  constexpr int NQ = P + 2, NQD = ipow(NQ, DIM), NQF = ipow(NQ, DIM - 1), NB = DIM > 2 ? PV + 1 : 1;
  const double* wq = tab<double>(P).wq;
  const int nx = PV * m.n[0] + 1, ny = PV * m.n[1] + 1, nz = DIM > 2 ? PV * m.n[2] + 1 : 1;
  const size_t nn = (size_t)nx * ny * nz;
  const int ntx = (m.n[0] + TL::X - 1) / TL::X, nty = (m.n[1] + TL::Y - 1) / TL::Y;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int cl = (int)(i % TL::N), k = (int)(i / TL::N % NQ), d = (int)(i / (TL::N * NQ) % DIM);
    const long long tile = i / ((long long)TL::N * NQ * DIM);
    const int g[3] = {(int)(tile % ntx) * TL::X + cl % TL::X, (int)(tile / ntx % nty) * TL::Y + cl / TL::X % TL::Y,
                      DIM > 2 ? (int)(tile / ((long long)ntx * nty)) * TL::Z + cl / (TL::X * TL::Y) : 0};
    if (g[0] >= m.n[0] || g[1] >= m.n[1] || (DIM > 2 && g[2] >= m.n[2])) continue;
    const double* un = u + d * nn + ((size_t)(PV * g[2]) * ny + PV * g[1]) * nx + PV * g[0];
    const size_t sl = DIM > 2 ? (size_t)ny * nx : nx;   // node stride along the last axis
    double V[NB][PV + 1];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int a = 0; a <= PV; ++a) {
        double s = 0.0;
#pragma unroll
        for (int c = 0; c <= PV; ++c) s += un[c * sl + (size_t)b * nx + a] * fb.b[c][k];
        V[b][a] = s;
      }
    const double wk = wq[k] / m.h[d];
    T* o = out + (size_t)tile * LY::template entries<NQ>() + ((size_t)d * NQD + (size_t)k * NQF) * TL::N + cl;
#pragma unroll
    for (int qy = 0; qy < (DIM > 2 ? NQ : 1); ++qy) {
      double x[PV + 1];
#pragma unroll
      for (int a = 0; a <= PV; ++a) {
        x[a] = V[0][a];
        if constexpr (DIM > 2) {
          x[a] *= fb.b[0][qy];
#pragma unroll
          for (int b = 1; b < NB; ++b) x[a] += V[b][a] * fb.b[b][qy];
        }
      }
      const double w = DIM > 2 ? wk * wq[qy] : wk;
#pragma unroll
      for (int qx = 0; qx < NQ; ++qx) {
        double s = 0.0;
#pragma unroll
        for (int a = 0; a <= PV; ++a) s += x[a] * fb.b[a][qx];
        o[(size_t)(qx + NQ * qy) * TL::N] = T(s * (w * wq[qx]));
      }
    }
  }
}

// the normal component at every face's quadrature points, from the face's
// own nodes (the basis of the others vanishes on it): the same value in both
// tiles of a face
template <int DIM, int P, int PV, typename T>
__global__ void fe_tabulate_faces(const MeshArgs m, const double* __restrict__ u, const FeBasis fb,
                                  long long total, T* __restrict__ out) {
  using LY = VelTabLayout<DIM>;
  using TL = HjsTile<DIM>;
  constexpr int NQ = P + 2, NQD = ipow(NQ, DIM), N1B = DIM > 2 ? PV + 1 : 1;
  const double* wq = tab<double>(P).wq;
  const int nx = PV * m.n[0] + 1, ny = PV * m.n[1] + 1, nz = DIM > 2 ? PV * m.n[2] + 1 : 1;
  const size_t nn = (size_t)nx * ny * nz;
  const size_t st[3] = {1, (size_t)nx, (size_t)nx * ny};
  const int ntx = (m.n[0] + TL::X - 1) / TL::X, nty = (m.n[1] + TL::Y - 1) / TL::Y;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    int s = (int)(i % LY::NFT);
    const int q1 = (int)(i / LY::NFT % (DIM > 2 ? NQ : 1));
    const long long tile = i / ((long long)LY::NFT * (DIM > 2 ? NQ : 1));
    T* o = out + (size_t)tile * LY::template entries<NQ>() + (size_t)DIM * NQD * TL::N + (size_t)NQ * q1 * LY::NFT + s;
    const int E = s < LY::S0 ? 0 : (s < LY::S0 + LY::S1 ? 1 : 2);
    s -= LY::off(E);
    const int ex = TL::X + (E == 0), ey = TL::Y + (E == 1);
    const int g[3] = {(int)(tile % ntx) * TL::X + s % ex, (int)(tile / ntx % nty) * TL::Y + s / ex % ey,
                      DIM > 2 ? (int)(tile / ((long long)ntx * nty)) * TL::Z + s / (ex * ey) : 0};
    bool in = true;
#pragma unroll
    for (int e = 0; e < DIM; ++e) in = in && g[e] < m.n[e] + (E == e);
    if (!in) continue;
    const int t0 = E == 0 ? 1 : 0, t1 = E == 2 ? 1 : 2;
    const double* un = u + E * nn + PV * (g[0] * st[0] + g[1] * st[1] + g[2] * st[2]);
    const double w = DIM > 2 ? wq[q1] / m.h[E] : 1.0 / m.h[E];
    double x[PV + 1];
#pragma unroll
    for (int a = 0; a <= PV; ++a) {
      x[a] = 0.0;
#pragma unroll
      for (int b = 0; b < N1B; ++b) x[a] += un[a * st[t0] + b * st[t1]] * (DIM > 2 ? fb.b[b][q1] : 1.0);
    }
#pragma unroll
    for (int q0 = 0; q0 < NQ; ++q0) {
      double v = 0.0;
#pragma unroll
      for (int a = 0; a <= PV; ++a) v += x[a] * fb.b[a][q0];
      o[(size_t)q0 * LY::NFT] = T(v * (w * wq[q0]));
    }
  }
}

// ---------------------------------------------------------------------
// FP64 reductions (level_set.implement.h:215-295, 356-380, 957-993;
// advection.cc:452-484; reinit.cc:491-526).  Two levels, fixed order.
// ---------------------------------------------------------------------
__device__ __forceinline__ double heaviside_sine(double x, double eps) {
  if (x > eps) return 1.0;
  if (x < -eps) return 0.0;
  const double val = 0.5 * (1.0 + x / eps + sin(x * kPiD / eps) / kPiD);
  if (fabs(val) < kEpsD) return 0.0;
  if (fabs(val - 1.0) < kEpsD) return 1.0;
  return val;
}
__device__ __forceinline__ double heaviside_sharp(double x) {
  return x > 0.0 ? 1.0 : (x < 0.0 ? 0.0 : 0.5);
}

template <typename T>
struct RedArgs {
  MeshArgs m;
  const T* phi;
  const T* ref;
  const flsp_ic_desc* ic;
  int which;
  double* partial;   // [gridDim.x][2]
};

template <int DIM, int P, typename T>
__global__ void reduce_kernel(const RedArgs<T> a) {
  constexpr int N1 = P + 1, NQ = P + 2, NM = ipow(N1, DIM);
  __shared__ double red[2][32];
  const MeshArgs& m = a.m;
  const Tab1D<double>& tb = c_tab_d[P];
  const long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  double s0 = 0.0, s1 = 0.0;
  if (cell < m.ncell) {
    double c[NM], r[NM];
#pragma unroll
    for (int q = 0; q < NM; ++q) {
      const int gi = m.q2g[q];
      c[q] = gi >= 0 ? double(a.phi[cell * m.nb + gi]) : 0.0;
      r[q] = (gi >= 0 && a.ref) ? double(a.ref[cell * m.nb + gi]) : 0.0;
    }
    const int g[3] = {(int)(cell % m.n[0]), (int)((cell / m.n[0]) % m.n[1]),
                      DIM > 2 ? (int)(cell / ((long long)m.n[0] * m.n[1])) : 0};
    const double eps = 1.5 * m.min_diam;
    const int w = a.which;
    if (w == FLSP_RED_MEAN_ABS_DIFF) {
      for (int k = 0; k < m.nb; ++k) s0 += fabs(double(a.phi[cell * m.nb + k]) - double(a.ref[cell * m.nb + k]));
    } else if (w == FLSP_RED_MAX_ABS) {
      for (int k = 0; k < m.nb; ++k) s0 = fmax(s0, fabs(double(a.phi[cell * m.nb + k])));
    } else {
      const bool gauss_p1 = (w == FLSP_RED_MASS || w == FLSP_RED_MASS_ERROR ||
                             w == FLSP_RED_GRAD_DEVIATION || w == FLSP_RED_L2_ERROR_IC);
      const int nq = gauss_p1 ? N1 : NQ;
      const int nqz = DIM > 2 ? nq : 1;
      double cellacc = 0.0;
      for (int qz = 0; qz < nqz; ++qz)
        for (int qy = 0; qy < nq; ++qy)
          for (int qx = 0; qx < nq; ++qx) {
            const int qq[3] = {qx, qy, qz};
            double bx[N1], by[N1], bz[N1], dx[N1], dy[N1], dz[N1], xx[3], wgt = 1.0;
            for (int d = 0; d < 3; ++d) xx[d] = 0.0;
            for (int i = 0; i < N1; ++i) {
              bx[i] = gauss_p1 ? tb.Ll[i][qx] : tb.Lq[i][qx];
              by[i] = gauss_p1 ? tb.Ll[i][qy] : tb.Lq[i][qy];
              bz[i] = DIM > 2 ? (gauss_p1 ? tb.Ll[i][qz] : tb.Lq[i][qz]) : 1.0;
              dx[i] = gauss_p1 ? tb.Dl[i][qx] : tb.Dq[i][qx];
              dy[i] = gauss_p1 ? tb.Dl[i][qy] : tb.Dq[i][qy];
              dz[i] = DIM > 2 ? (gauss_p1 ? tb.Dl[i][qz] : tb.Dq[i][qz]) : 1.0;
            }
            for (int d = 0; d < DIM; ++d) {
              const double xi = gauss_p1 ? tb.xl[qq[d]] : tb.xq[qq[d]];
              xx[d] = (m.lo[d] + g[d] * m.h[d]) + m.h[d] * xi;
              wgt *= gauss_p1 ? tb.wl[qq[d]] : tb.wq[qq[d]];
            }
            const double jxw = wgt * m.vol;
            const double val = eval_modal<DIM, P>(c, bx, by, bz);
            if (w == FLSP_RED_MASS || w == FLSP_RED_MASS_ERROR) {
              s0 += heaviside_sine(-val, eps) * jxw;
              if (w == FLSP_RED_MASS_ERROR) s1 += heaviside_sine(-ic_eval(a.ic, DIM, xx), eps) * jxw;
            } else if (w == FLSP_RED_MASS_SHARP) {
              s0 += heaviside_sharp(-val) * jxw;
            } else if (w == FLSP_RED_L1_INTERFACE) {
              s0 += fabs(heaviside_sharp(-val) - heaviside_sharp(-eval_modal<DIM, P>(r, bx, by, bz))) * jxw;
            } else if (w == FLSP_RED_L1_INTERFACE_IC) {
              s0 += fabs(heaviside_sharp(-val) - heaviside_sharp(-ic_eval(a.ic, DIM, xx))) * jxw;
            } else if (w == FLSP_RED_L2_ERROR_IC) {
              const double diff = val - ic_eval(a.ic, DIM, xx);
              cellacc += diff * diff * jxw;
            } else if (w == FLSP_RED_GRAD_DEVIATION) {
              const double gxv = eval_modal<DIM, P>(c, dx, by, bz) / m.h[0];
              const double gyv = eval_modal<DIM, P>(c, bx, dy, bz) / m.h[1];
              const double gzv = DIM > 2 ? eval_modal<DIM, P>(c, bx, by, dz) / m.h[2] : 0.0;
              const double g2 = gxv * gxv + gyv * gyv + gzv * gzv;
              s0 += fabs(sqrt(g2) - 1.0) * jxw;
            }
          }
      if (w == FLSP_RED_L2_ERROR_IC) s0 += cellacc;
      if (w == FLSP_RED_GRAD_DEVIATION) s1 += m.vol;
    }
  }
  if (a.which == FLSP_RED_MAX_ABS) {
    const double bm = block_max(s0, red[0]);
    if (threadIdx.x == 0) { a.partial[2 * blockIdx.x] = bm; a.partial[2 * blockIdx.x + 1] = 0.0; }
    return;
  }
  s0 = warp_sum(s0);
  s1 = warp_sum(s1);
  const int wi = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { red[0][wi] = s0; red[1][wi] = s1; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t0 = 0.0, t1 = 0.0;
    const int nw = (blockDim.x + 31) >> 5;
    for (int i = 0; i < nw; ++i) { t0 += red[0][i]; t1 += red[1][i]; }
    a.partial[2 * blockIdx.x] = t0;
    a.partial[2 * blockIdx.x + 1] = t1;
  }
}

__global__ void reduce_final(const double* __restrict__ partial, int n, int is_max, double* out) {
  __shared__ double red[2][32];
  double s0 = 0.0, s1 = 0.0;
  // fixed assignment of partials to threads -> deterministic
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    if (is_max) s0 = fmax(s0, partial[2 * i]);
    else { s0 += partial[2 * i]; s1 += partial[2 * i + 1]; }
  }
  if (is_max) {
    const double bm = block_max(s0, red[0]);
    if (threadIdx.x == 0) { out[0] = bm; out[1] = 0.0; }
    return;
  }
  s0 = warp_sum(s0);
  s1 = warp_sum(s1);
  const int wi = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { red[0][wi] = s0; red[1][wi] = s1; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t0 = 0.0, t1 = 0.0;
    for (int i = 0; i < (int)((blockDim.x + 31) >> 5); ++i) { t0 += red[0][i]; t1 += red[1][i]; }
    out[0] = t0;
    out[1] = t1;
  }
}

// finite check of a state vector: counts non-finite entries
template <typename T>
__global__ void nonfinite_kernel(const T* __restrict__ x, long long n, unsigned int* count) {
  unsigned int local = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    if (!isfinite((double)x[i])) ++local;
  if (local) atomicAdd(count, local);
}

}  // namespace flsp
