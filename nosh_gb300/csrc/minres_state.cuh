// MINRES recurrence state (device memory) and its device-side update.
#pragma once

#include <cstddef>

#include "common.cuh"

namespace nosh {

struct MinresScalars {
  double beta1, beta, oldb, alfa, dbar, epsln, oldeps, phibar, phi, cs, sn, gamma, delta;
  double zu, rz;  // reduction results: <z, J z>, <r, M r>
  double ibeta, ioldb;  // 1 / beta, 1 / oldb (0 before the second step)
  double rtol;
  int itn, maxit;
  int done;        // 0 running, 1 converged in the last update, 2 frozen
  int flag;        // NOSH_OK / NOSH_ERR_NOT_CONVERGED / _NAN / _BREAKDOWN
  int wx_pending;  // the w/x update of the last Lanczos step is still due
  // per-element coefficients, computed once per step by the single thread
  // that owns the recurrence (FP64 division is slow on GB300: element
  // kernels only load these):
  //   lanczos: r_new = la[0] u - la[1] r_old - la[2] r_cur
  //   w/x:     w = (z wx[0] - wx[1] w2 - wx[2] w) wx[3];  x += wx[4] w
  double la64[3], wx64[5];
  float la32[3], wx32[5];
};

template <typename T>
__device__ __forceinline__ const T *lanczos_coef(const MinresScalars *s);
template <>
__device__ __forceinline__ const float *lanczos_coef<float>(const MinresScalars *s) {
  return s->la32;
}
template <>
__device__ __forceinline__ const double *lanczos_coef<double>(const MinresScalars *s) {
  return s->la64;
}
template <typename T>
__device__ __forceinline__ const T *wx_coef(const MinresScalars *s);
template <>
__device__ __forceinline__ const float *wx_coef<float>(const MinresScalars *s) {
  return s->wx32;
}
template <>
__device__ __forceinline__ const double *wx_coef<double>(const MinresScalars *s) {
  return s->wx64;
}

// Both updates run on one warp at the end of a launch, so they are a chain of
// FP64 instructions, 64 cycles of its scheduler each, and nothing else.  The
// lanes share them: even lanes hold one of a pair of values and odd lanes the
// other, so that a pair costs one instruction (delta and gbar, the two
// reciprocal square roots, cs and sn, phi and phibar).  Reciprocals come from
// the square roots of the step before instead of divisions, and the Givens
// rotation's radius is sqrt(gbar^2 + rz) (beta^2 is rz itself).  `head` is the
// state up to wx_pending, in shared memory or *sp itself; whole warps call.
// The launches that end in them, with the state's fetch ahead of the sum
// (grid_reduce), on the 65^2 square: J z 7.2 -> 6.7 us in FP64 and 6.4 -> 5.5 in
// FP32, last smoothing step 9.4 -> 8.3 and 8.2 -> 6.5 (one thread, one value an
// instruction, before).
constexpr int kMinresHeadWords = (int)((offsetof(MinresScalars, wx_pending) + 4 + 7) / 8);

__device__ __forceinline__ double flip_sign(double v) {
  return __hiloint2double(__double2hiint(v) ^ 0x80000000, __double2loint(v));
}

// Lanczos coefficients once <z, J z> (zu) is known.  After convergence
// (done == 1) the launch has applied the last deferred w/x update, and the
// recurrence is frozen (done = 2): the remaining launches of the chunk return
// at once.
__device__ __forceinline__ void minres_lanczos_coefs(MinresScalars *sp, const double *head, double zu) {
  const MinresScalars &s = *reinterpret_cast<const MinresScalars *>(head);
  const int lane = threadIdx.x & 31;
  if (s.done) {
    __syncwarp();
    if (lane == 0) {
      sp->done = 2;
      sp->wx_pending = 0;
    }
    return;
  }
  const double ibeta = s.ibeta, alfa = zu * (ibeta * ibeta);
  // 1 / beta, beta / oldb, alfa / beta
  double c = (lane == 1 ? s.beta : alfa) * (lane == 1 ? s.ioldb : ibeta);
  if (lane == 0) c = ibeta;
  __syncwarp();
  if (lane == 0) {
    sp->zu = zu;
    sp->alfa = alfa;
  }
  if (lane < 3) {
    sp->la64[lane] = c;
    sp->la32[lane] = (float)c;
  }
}

// One step of the Paige-Saunders Givens recurrence after <r_new, M r_new>
// (rz) is known; scipy / Paige-Saunders variable names.
__device__ __forceinline__ void minres_advance(MinresScalars *sp, const double *head, double rz) {
  const MinresScalars &s = *reinterpret_cast<const MinresScalars *>(head);
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const bool odd = lane & 1;
  const double alfa = s.alfa;
  const bool nan_alfa = isnan(alfa), bad_rz = !(rz >= 0.0) || isinf(rz);
  if (s.done || bad_rz || nan_alfa) {
    const int done = s.done;
    __syncwarp();
    if (lane == 0) {
      sp->rz = rz;
      sp->done = 2;
      sp->wx_pending = 0;
      if (!done) {
        sp->oldb = s.beta;
        sp->ioldb = s.ibeta;
        sp->flag = isnan(rz) || isinf(rz) || nan_alfa ? NOSH_ERR_NAN : NOSH_ERR_BREAKDOWN;
      }
    }
    return;
  }
  const double oldb = s.beta, ioldb = s.ibeta, oldeps = s.epsln, phibar0 = s.phibar, beta1 = s.beta1, rtol = s.rtol;
  const int itn = s.itn + 1, maxit = s.maxit;
  const double a = odd ? s.sn : s.cs, b = odd ? flip_sign(s.cs) : s.sn;
  const double d = a * s.dbar + b * alfa;  // delta, gbar
  const double delta = __shfl_sync(kAll, d, 0), gbar = __shfl_sync(kAll, d, 1);
  const double g2 = gbar * gbar + rz, q = odd ? g2 : rz;
  const double iq = rsqrt(q), rq = q * iq;  // 1 / beta and beta (infinite and 0 for rz = 0), 1 / gamma and gamma
  const double ibeta = __shfl_sync(kAll, iq, 0);
  double nb = __shfl_sync(kAll, rq, 0), ig = __shfl_sync(kAll, iq, 1), gamma = __shfl_sync(kAll, rq, 1);
  if (rz == 0.0) nb = 0.0;
  if (!(g2 > 1e-280 && g2 < 1e280)) {  // the squares leave the normal range
    gamma = hypot(gbar, nb);
    if (gamma == 0.0) gamma = 2.2e-16;
    ig = 1.0 / gamma;
  }
  const double eps = b * nb;  // even: epsln = sn nb; odd: dbar = -cs nb
  const double rot = (odd ? nb : gbar) * ig;  // cs, sn
  const double ph = rot * phibar0;            // phi, phibar
  const double phi = __shfl_sync(kAll, ph, 0), phibar = __shfl_sync(kAll, ph, 1);
  const bool conv = phibar <= rtol * beta1 || nb == 0.0;
  double w = ioldb;
  if (lane == 1) w = oldeps;
  if (lane == 2) w = delta;
  if (lane == 3) w = ig;
  if (lane == 4) w = phi;
  __syncwarp();
  if (lane < 5) {
    sp->wx64[lane] = w;
    sp->wx32[lane] = (float)w;
  }
  if (lane == 0) {
    sp->rz = rz;
    sp->oldb = oldb;
    sp->ioldb = ioldb;
    sp->beta = nb;
    sp->ibeta = ibeta;
    sp->oldeps = oldeps;
    sp->epsln = eps;
    sp->cs = rot;
    sp->phi = ph;
    sp->delta = delta;
    sp->itn = itn;
    sp->wx_pending = 1;
    if (conv) {
      sp->done = 1;
    } else if (itn >= maxit) {
      sp->done = 1;
      sp->flag = NOSH_ERR_NOT_CONVERGED;
    }
  }
  if (lane == 1) {
    sp->dbar = eps;
    sp->sn = rot;
    sp->phibar = ph;
    sp->gamma = gamma;
  }
}

// The deferred w/x update of one Lanczos step for element i:
// w_new = (z/oldb - oldeps w2 - delta w) / gamma (over the w1 buffer),
// x += phi w_new.
template <typename T>
__device__ __forceinline__ void minres_wx_elem(const T *c, int64_t i, const T *z, T *wa, const T *wb,
                                               const T *wc, T *x) {
  const T w = (z[i] * c[0] - c[1] * wb[i] - c[2] * wc[i]) * c[3];
  wa[i] = w;
  x[i] += c[4] * w;
}

}  // namespace nosh
