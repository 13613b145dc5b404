// flsp_clock.cuh — the device clocks' updates (shared by the single-problem
// clock kernels and the batched ones).
#pragma once
#include "flsp_device.cuh"

namespace flsp {

constexpr double kClockEps = 2.220446049250313e-16;

// AdvectSimulator::advance_time substep set-up (advection.cc:396-404) of the
// next n substeps: CFL estimate at the substep's time (running maximum, the
// estimator never resets), substep = min(cfl_max / estimate, remaining), stage
// time factors.  A warp's work: the chain of times on lane 0, the stage factors
// dealt to the lanes.  commit: the clock moves on past the n substeps.
__device__ __forceinline__ void adv_clock_steps_body(DevClock* c, const AdvClockArgs& a, AdvStep* st, int n,
                                                     bool commit) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) {
    double t = c->t, vd_run = c->vd_run, cum = c->scratch[1], dt = c->dt;
    int done = 0;
    for (int k = 0; k < n; ++k) {
      const double ctn = time_factor(a.tkind, a.ta, a.tb, t);
      vd_run = fmax(vd_run, fabs(ctn) * c->vd_static);
      double suggest = a.cfl_max / (vd_run * a.scale);
      const double remaining = c->scratch[0] - cum;   // time_step - cumulative
      // a velocity whose time factor vanishes (e.g. 1 - exp(-t) at t = 0) gives
      // an infinite CFL substep.  A call for a time step (the reference rule)
      // then takes the remaining time; a step-count run, whose horizon only
      // caps the time, falls back to the estimate of the spatial field alone
      // (|time factor| = 1)
      if (a.step_count && !isfinite(suggest) && c->vd_static > 0.0) suggest = a.cfl_max / (c->vd_static * a.scale);
      dt = fmin(suggest, remaining);
      if (!isfinite(dt) && c->vd_static > 0.0) dt = a.cfl_max / (c->vd_static * a.scale);
      const bool active = !(fabs(dt) <= kClockEps);   // TempoIntegrator skips zero steps
      st[k].ct[0] = ctn;
      st[k].dt = dt;
      st[k].t = t;
      st[k].active = active ? 1 : 0;
      if (active) {
        t += dt;
        ++done;
      }
      cum += dt;
    }
    c->vd_run = vd_run;
    if (commit) {
      c->t = t;
      c->dt = dt;
      c->scratch[1] = cum;   // cumulative time of this advance call
      c->n_substeps += done;
    }
  }
  __syncwarp();
  for (int i = lane; i < 2 * n; i += 32) {
    AdvStep& s = st[i / 2];
    if (i % 2) s.ct[2] = time_factor(a.tkind, a.ta, a.tb, s.t + 0.5 * s.dt);
    else s.ct[1] = time_factor(a.tkind, a.ta, a.tb, s.t + s.dt);
  }
}

// start an advance call of length time_step (scratch[0]); +inf = unclamped
__device__ __forceinline__ void adv_clock_horizon_body(DevClock* c, double time_step) {
  c->scratch[0] = time_step;
  c->scratch[1] = 0.0;
}

__device__ __forceinline__ void hj_clock_reset_body(DevClock* c) {
  c->hj_dt = 0.0;
  c->hj_cum = 0.0;
  for (int k = 0; k < 3; ++k) c->hj_vd[k] = 0ull;
}

// Size of pseudo-step a.k (ReinitSimulatorLDG::advance_time, reinit.cc:396-408,
// with HJSimulator::cfl_scaling, hamilton_jacobi.cc:554-580), from the running
// maximum the launch before left; one thread of every block computes it, the
// launch's first block moves the clock on.
__device__ __forceinline__ double hj_clock_step(DevClock* c, const HjClockArgs& a, bool first, double& vd) {
  vd = __longlong_as_double((long long)c->hj_vd[a.k % 3]);
  const double dt = a.cfl_max / (a.scale * vd + a.shift);
  if (first) {
    c->hj_dt = dt;
    c->hj_cum += dt;
    c->hj_vd[(a.k + 2) % 3] = 0ull;
    atomic_max_pos(&c->hj_vd[(a.k + 1) % 3], vd);
  }
  return dt;
}

}  // namespace flsp
