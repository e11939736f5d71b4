// The accept/reject and PI step-size update of one adaptive attempt, shared by
// the single-solve controller kernel (csrc/imex.cu) and the batched controller
// (csrc/imex_batch.cu).
#pragma once

#include "spectral.cuh"

namespace mjx {

// What bounds the update: one dependent chain of FP64 instructions of a single warp, ~64 cycles
// each whatever its active lanes.  With two pow calls, six divisions and three-comparison
// min/max the controller took 15 us of a 139 us attempt at 1024^2.  The step factor
//   (1/e)^kI (e_prev/e)^kP = exp(kP log e_prev - (kI + kP) log e)
// now takes one log and one exp, both on the size of a rounding error in dt, log e_prev is kept
// from the attempt that set it, the quotients that do not change are formed on the host, and
// the square root runs beside the logarithm: 15.1 -> 7.1 us.

// NaN test on the bits: an FP64 comparison would take an FP64 issue slot
__device__ __forceinline__ bool jnan(double a) {
  const unsigned hi = (unsigned)__double2hiint(a) & 0x7fffffffu;
  return hi > 0x7ff00000u || (hi == 0x7ff00000u && __double2loint(a) != 0);
}
// NaN-propagating min/max (jnp.minimum/maximum semantics)
__device__ __forceinline__ double jmax(double a, double b) { return (jnan(a) || a > b) ? a : b; }
__device__ __forceinline__ double jmin(double a, double b) { return (jnan(a) || a < b) ? a : b; }
__device__ __forceinline__ double jclip(double x, double lo, double hi) { return jmin(jmax(x, lo), hi); }

// log max(e, 1e-10) of the error norm e = sqrt(q), and the step factor before the safety
// factor: propose_dt_imex (dt_policy.py:544-610) over pid_controller_dt (178-227) for e <= 1
// and handle_rejected_step (230-268) above
__device__ __forceinline__ double ctl_log(double q) { return jmax(0.5 * log(q), -23.025850929940456840); }
__device__ __forceinline__ double ctl_factor(const CtlGain& G, bool small, double le, double lprev) {
  // x^0 is 1 for every x, also where the norm has overflowed or is NaN: without an integral gain a
  // rejected step shrinks by the safety factor
  return exp(small ? G.kP * lprev - (G.kI + G.kP) * le : (G.kI == 0.0 ? 0.0 : -G.kI * jmax(le, 0.0)));
}

// e = max(sqrt(tot / n_dof), 1e-10) with tot the sum over every degree of freedom of
// (err / (atol + rtol |y_new|))^2, le = ctl_log, fac = ctl_factor; bad: any non-finite value.
// Applies moljax/core/stepping.py:1246-1359 (the accept and reject branches, the loop stop and
// final status) to st and returns whether the run continues.  hist_t / hist_dt may be null.
__device__ __forceinline__ bool ctl_apply(DevState* st, double e, double le, double fac, int bad,
                                          const mjx_pid_params& P, double* hist_t, double* hist_dt) {
  const double dtc = st->dtc;
  const int finite = !bad;
  const bool small = e <= 1.0;
  const bool accept = small && finite;
  fac = jclip(P.safety * fac, P.min_factor, small ? P.max_factor : 1.0);
  const double dt_a = jclip(dtc * fac, P.dt_min, P.dt_max);
  const double dt_new = jclip(jmin(dt_a, st->dt_cfl), P.dt_min, P.dt_max);
  st->err_last = e;
  st->save_slot = -1;
  if (accept) {  // stepping.py:1271-1309
    if (st->n_acc % st->save_every == 0) {
      if (hist_t) hist_t[st->write_idx] = st->t + dtc;
      if (hist_dt) hist_dt[st->write_idx - 1] = dtc;
      st->save_slot = st->write_idx;
      st->write_idx += 1;
    }
    st->t = st->t + dtc;
    st->cur = 1 - st->cur;
    st->dt = dt_new;
    st->prev_err = e;
    st->lprev = le;
    st->dt_last_accepted = dtc;
    st->n_acc += 1;
  } else {  // stepping.py:1311-1334
    const double dtr = jmax(dt_new * 0.5, P.dt_min);
    st->dt = dtr;
    if (dtr <= P.dt_min * 1.1) st->status = MJX_STATUS_DT_TOO_SMALL_CODE;
    st->n_rej += 1;
  }
  if (!finite) { st->status = MJX_STATUS_NON_FINITE_CODE; st->finite = 0; }
  st->attempts += 1;
  const bool running = st->status == MJX_STATUS_RUNNING_CODE && st->t < st->t_end &&
                       st->write_idx < st->max_saves && st->attempts < st->max_attempts;
  if (running) {
    st->dtc = jmin(st->dt, st->t_end - st->t);
  } else {
    st->done = 1;
    if (st->t >= st->t_end) st->status = MJX_STATUS_SUCCESS_CODE;             // 1351-1359
    else if (st->write_idx >= st->max_saves) st->status = MJX_STATUS_MAX_STEPS_CODE;
    else if (st->status == MJX_STATUS_RUNNING_CODE) st->status = MJX_STATUS_MAX_STEPS_CODE;
  }
  return running;
}

// the whole update by one thread
__device__ __forceinline__ bool ctl_update(DevState* st, double tot, int bad, const CtlGain& G,
                                           const mjx_pid_params& P, double* hist_t, double* hist_dt) {
  const double q = tot * G.inv_n, e = jmax(sqrt(q), 1e-10), le = ctl_log(q);
  return ctl_apply(st, e, le, ctl_factor(G, e <= 1.0, le, st->lprev), bad, P, hist_t, hist_dt);
}

}  // namespace mjx
