// flsp_stage.cuh — what the advection stage kernels share: the SSP-RK stage
// combination and its coalesced store, the modes in use, face traces.
#pragma once
#include "flsp_device.cuh"

namespace flsp {

// stage combination: v = phi + dt L (L itself for kRhsOnly), then phi^n's share.
// FP32: the weighted sum (v + b phi^n) f, its products and sums in the order
// CombineMode states (kRK3c as (v + phi^n / 2) (2/3): the same bits, both factors
// moved by a power of two).  A narrow band and a learned reinitialisation compare
// cell means with a threshold, so the last bits decide which cells they take, and an
// FP32 mean is near enough to it for that to happen: the order is part of the
// result.  v + w (phi^n - v) leaves out the constant's scaling by up to 1 + 3e-8 a
// step and ends 3 to 5 times nearer the 64-bit field, but it moved the means at the
// edge of a 6-cell band by 1.3e-7 in 60 steps (this order: 9e-9, an ulp), and 2 of 26
// band runs by 5.8e-4 and 1.3e-3 of the field in the cells that changed sides.  They
// cost the same in 3D (64^3 Q2 run 22.95 and 22.97 ms), the sum 0.7 % of a 256^2 run.
// FP64: v + w (phi^n - v); 120 steps of a rotation end 7e-16 from extended
// precision, with the weighted sum 6.5e-15.
template <typename T>
struct Combine {
  static constexpr bool SUM = sizeof(T) == 4;
  T dt, w, f;
  bool rhs;
  __device__ __forceinline__ Combine(int mode, T step) : dt(mode == kRhsOnly ? T(1) : step), rhs(mode == kRhsOnly) {
    if constexpr (SUM) {
      w = mode == kRK2b ? T(1) : mode == kRK3b ? T(3) : mode == kRK3c ? T(0.5) : T(0);
      f = mode == kRK2b ? T(0.5) : mode == kRK3b ? T(0.25) : T(2) * (T(1) / T(3));
    } else {
      w = mode == kRK2b ? T(0.5) : mode == kRK3b ? T(0.75) : mode == kRK3c ? T(1) / T(3) : T(0);
    }
  }
  __device__ __forceinline__ T operator()(T phi, T phin, T L) const {
    if constexpr (SUM) {
      const T v = fma(dt, L, rhs ? T(0) : phi);
      return w != T(0) ? fma(w, phin, v) * f : v;
    } else {
      const T v = (rhs ? T(0) : phi) + dt * L;
      return w != T(0) ? v + w * (phin - v) : v;
    }
  }
};

// Modes in use: every (a, b, c) of the Q layout, or with PB those of the P
// space, a + b + c <= P; sums and results outside it are left out at compile
// time (3D degree 2: 10 of 27 modes).
template <int P, bool PB>
__host__ __device__ constexpr bool mode_in(int sum) {
  return !PB || sum <= P;
}
// index of the face mode (m0, m1) among those in use
template <int P, bool PB>
__host__ __device__ constexpr int face_index(int m0, int m1) {
  int i = m0;
  for (int k = 0; k < m1; ++k) i += PB ? P + 1 - k : P + 1;
  return i;
}
// index of mode (a, b, c) in a cell's HBM order
template <int DIM, int P, bool PB>
__host__ __device__ constexpr int cell_index(int q) {
  return PB ? q2g_ct<DIM, P>(q) : q;
}

// trace of a box cell (HBM order) on its face normal to E, in face modes
// (side values Ls = L(0) or L(1); L_0 = 1)
template <int DIM, int P, bool PB, int E, typename T>
__device__ __forceinline__ void face_trace_ct(const T* __restrict__ src, const T* Ls, T* tr) {
  constexpr int N1 = P + 1;
  constexpr int t0 = E == 0 ? 1 : 0, t1 = E == 2 ? 1 : 2;
  constexpr int st[3] = {1, N1, N1 * N1};
#pragma unroll
  for (int m1 = 0; m1 < (DIM > 2 ? N1 : 1); ++m1)
#pragma unroll
    for (int m0 = 0; m0 < N1; ++m0) {
      if (!mode_in<P, PB>(m0 + m1)) continue;
      const int base = m0 * st[t0] + (DIM > 2 ? m1 * st[t1] : 0);
      T s = src[cell_index<DIM, P, PB>(base)];
#pragma unroll
      for (int aa = 1; aa < N1; ++aa)
        if (mode_in<P, PB>(m0 + m1 + aa)) s += Ls[aa] * src[cell_index<DIM, P, PB>(base + aa * st[E])];
      tr[face_index<P, PB>(m0, m1)] = s;
    }
}

// The stage combination of a TX x TY x TZ tile's cells, fused into the
// coalesced store: stage input from the box copies (cellp), R from rbuf
// ([cell][NBG], HBM order), phi^n from HBM.  NW warps, one per row of cells
// along x; inactive (a zero-length substep): the stage input passes through.
template <int DIM, int TX, int TY, int TZ, int NBG, int NW, typename T, typename CellP>
__device__ __forceinline__ void combine_rows(const MeshArgs& m, const CellP& cellp, const T* __restrict__ rbuf,
                                             const T* __restrict__ phi_n, T* __restrict__ out, int combine, T dt,
                                             bool active, int ox, int oy, int oz) {
  // ---- RK combination fused into the coalesced store: one warp per row of
  // cells along x; stage input from the box, phi^n from HBM, all of a
  // lane's phi^n loads issued before the first use.  Plain loads: the kernel
  // before may still write phi^n when this one starts (chain_wait), which the
  // read-only path does not allow for
  const Combine<T> comb(combine, dt);
  const bool need_n = combine == kRK2b || combine == kRK3b || combine == kRK3c;
  constexpr int NROW = TY * TZ, ROWE = TX * NBG;
  constexpr int RPW = (NROW + NW - 1) / NW, KPR = (ROWE + 31) / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nx = min(TX, m.n[0] - ox);
  // FP32 rows of whole tiles start on 16-byte boundaries in HBM, in the box
  // copy (same 16-byte phase) and in the R buffer when TX * NBG and the row
  // pitch n[0] * NM are multiples of 4: float4 loads and stores
  constexpr bool VEC = sizeof(T) == 4 && (TX * NBG) % 4 == 0;
  const bool vec_ok = VEC && nx == TX && ((long long)m.n[0] * NBG) % 4 == 0 &&
                      ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(phi_n)) & 15) == 0;
  if (VEC && vec_ok) {
    constexpr int RV = TX * NBG / 4, KV = (RV + 31) / 32;   // float4 per row, per lane
    constexpr int CV = RPW;                                 // rows with loads in flight together
#pragma unroll
    for (int j0 = 0; j0 < RPW; j0 += CV) {
      float4 pn[CV][KV];
#pragma unroll
      for (int jj = 0; jj < CV; ++jj) {
        const int r = warp + NW * (j0 + jj);
        const int ly = r % TY, lz = r / TY;
        const bool rok = j0 + jj < RPW && r < NROW && oy + ly < m.n[1] && (DIM < 3 || oz + lz < m.n[2]);
        const long long gbase =
            ((long long)m.n[0] * ((oy + ly) + (long long)m.n[1] * (DIM > 2 ? oz + lz : 0)) + ox) * NBG;
        const float4* src = reinterpret_cast<const float4*>(phi_n + (rok ? gbase : 0));
#pragma unroll
        for (int k = 0; k < KV; ++k) {
          const int e = lane + 32 * k;
          pn[jj][k] = (need_n && active && rok && e < RV) ? src[e] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
#pragma unroll
      for (int jj = 0; jj < CV; ++jj) {
        const int r = warp + NW * (j0 + jj);
        const int ly = r % TY, lz = r / TY;
        if (!(j0 + jj < RPW && r < NROW && oy + ly < m.n[1] && (DIM < 3 || oz + lz < m.n[2]))) continue;
        const long long gbase =
            ((long long)m.n[0] * ((oy + ly) + (long long)m.n[1] * (DIM > 2 ? oz + lz : 0)) + ox) * NBG;
        const float4* cs = reinterpret_cast<const float4*>(cellp(0, ly, lz));
        const float4* rs = reinterpret_cast<const float4*>(rbuf + (size_t)TX * r * NBG);
        float4* dst = reinterpret_cast<float4*>(out + gbase);
#pragma unroll
        for (int k = 0; k < KV; ++k) {
          const int e = lane + 32 * k;
          if (e >= RV) continue;
          const float4 cv = cs[e];
          float4 o = cv;
          if (active) {
            const float4 rv = rs[e], nv = pn[jj][k];
            o.x = comb(cv.x, nv.x, rv.x);
            o.y = comb(cv.y, nv.y, rv.y);
            o.z = comb(cv.z, nv.z, rv.z);
            o.w = comb(cv.w, nv.w, rv.w);
          }
          dst[e] = o;
        }
      }
    }
  } else {
    // rows in chunks of CH, a chunk's phi^n loads all in flight together
    constexpr int CH = RPW * KPR > 16 ? (RPW > 2 ? 2 : RPW) : RPW;
#pragma unroll
    for (int j0 = 0; j0 < RPW; j0 += CH) {
      T pn[CH][KPR];
#pragma unroll
      for (int jj = 0; jj < CH; ++jj) {
        const int r = warp + NW * (j0 + jj);
        const int ly = r % TY, lz = r / TY;
        const bool rok = j0 + jj < RPW && r < NROW && oy + ly < m.n[1] && (DIM < 3 || oz + lz < m.n[2]);
        const long long gbase =
            ((long long)m.n[0] * ((oy + ly) + (long long)m.n[1] * (DIM > 2 ? oz + lz : 0)) + ox) * NBG;
#pragma unroll
        for (int k = 0; k < KPR; ++k) {
          const int e = lane + 32 * k;
          pn[jj][k] = (need_n && active && rok && e < nx * NBG) ? phi_n[gbase + e] : T(0);
        }
      }
#pragma unroll
      for (int jj = 0; jj < CH; ++jj) {
        const int r = warp + NW * (j0 + jj);
        const int ly = r % TY, lz = r / TY;
        if (!(j0 + jj < RPW && r < NROW && oy + ly < m.n[1] && (DIM < 3 || oz + lz < m.n[2]))) continue;
        const long long gbase =
            ((long long)m.n[0] * ((oy + ly) + (long long)m.n[1] * (DIM > 2 ? oz + lz : 0)) + ox) * NBG;
        const T* cs = cellp(0, ly, lz);
        const T* rs = rbuf + (size_t)TX * r * NBG;
#pragma unroll
        for (int k = 0; k < KPR; ++k) {
          const int e = lane + 32 * k;
          if (e >= nx * NBG) continue;
          const T cv = cs[e];
          out[gbase + e] = active ? comb(cv, pn[jj][k], rs[e]) : cv;
        }
      }
    }
  }
}

}  // namespace flsp
