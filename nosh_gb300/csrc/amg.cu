// Aggregation AMG preconditioner for the regularised KEO
// (keo_regularized, src/keo_regularized.cpp).  The reference applies one
// MueLu SA-AMG V-cycle with 2 equations per node (:292-336); this is a
// GB300-native aggregation AMG with the same role:
//
//  * structure (aggregates, coarse graphs, Galerkin plans) is built on the
//    host at the first rebuild and reused afterwards (MueLu "reuse: full"
//    keeps the hierarchy too); every rebuild refreshes all numeric values on
//    the GPU from the current K_reg;
//  * plain (unsmoothed) aggregation with 2x2-block identity prolongation:
//    every level keeps the fine level's compact format -- one complex value
//    per off-diagonal block plus a symmetric 2x2 diagonal block -- and the
//    Galerkin product P^T A P is a deterministic segmented sum;
//  * block-Jacobi Chebyshev smoothing (same polynomial before and after the
//    coarse correction, so the V-cycle is a fixed SPD operator as MINRES
//    requires); Gershgorin bound for lambda_max(D^-1 A);
//  * coarsest level: dense inverse (Gauss-Jordan) applied as a matvec.
#include <algorithm>
#include <cmath>
#include <complex>
#include <numeric>
#include <type_traits>

#include "amg.cuh"
#include "spmv.cuh"

namespace nosh {

using namespace dev;

namespace {

// The largest level that the resident V-cycle starts on, and the largest mesh
// that it takes whole.  Measured per MINRES iteration, whole against from
// level 1 on: 17^2 25 / 36 us (FP64) and 21 / 30 (mixed), 45^2 41 / 45 and
// 30 / 35, 11^3 cubes 35 / 43 and 23 / 30; a 65^2 square's rows (265 a CTA)
// are more than one pass of the CTA.  Levels of 2048 and 4096 nodes in it gained
// nothing on 32^3 and 48^3 (their SpMVs fill the grid by then).
constexpr int64_t kTailMax = 1024;
constexpr int64_t kResidentMax = 2048;

struct HostLevel {
  int64_t n = 0;
  std::vector<int32_t> rp, ci;  // off-diagonal CSR
  std::vector<std::complex<double>> off;  // values (strength / next level)
  std::vector<double> dia;                // 3 per node
  // transfer to the next level
  std::vector<int32_t> agg;               // n
  std::vector<int32_t> mem_ptr, mem_idx;  // coarse node -> fine nodes
  std::vector<int32_t> seg_ptr, seg_idx;  // coarse nonzero -> fine nonzeros
  std::vector<int32_t> intra_ptr, intra_idx;  // coarse node -> fine intra nnz
  // independent systems (batched solves): nodes of system s are
  // [soff[s], soff[s+1]); a single system has soff = {0, n}
  std::vector<int64_t> soff;
};

int64_t max_block(const HostLevel &L) {
  int64_t m = 0;
  for (size_t s = 0; s + 1 < L.soff.size(); s++) m = std::max(m, L.soff[s + 1] - L.soff[s]);
  return m;
}

// Greedy aggregation on the strong graph (deterministic, vertex order):
// 1) a vertex whose strong neighbours are all free roots an aggregate with
//    them; 2) every remaining vertex joins the aggregate it is most strongly
//    connected to; 3) isolated leftovers become singletons.
int64_t aggregate(const HostLevel &L, std::vector<int32_t> &agg, double theta) {
  const int64_t n = L.n;
  std::vector<double> scale(n);
  for (int64_t i = 0; i < n; i++) scale[i] = std::max(0.5 * (L.dia[3 * i] + L.dia[3 * i + 1]), 1e-300);
  auto strong = [&](int64_t i, int64_t k) {
    const int64_t j = L.ci[k];
    return std::abs(L.off[k]) >= theta * std::sqrt(scale[i] * scale[j]);
  };
  agg.assign(n, -1);
  int64_t na = 0;
  for (int64_t i = 0; i < n; i++) {
    if (agg[i] >= 0) continue;
    bool free = true;
    for (int64_t k = L.rp[i]; k < L.rp[i + 1] && free; k++)
      if (strong(i, k) && agg[L.ci[k]] >= 0) free = false;
    if (!free) continue;
    agg[i] = (int32_t)na;
    for (int64_t k = L.rp[i]; k < L.rp[i + 1]; k++)
      if (strong(i, k)) agg[L.ci[k]] = (int32_t)na;
    na++;
  }
  std::vector<int32_t> agg1 = agg;  // phase 2 reads phase-1 state only
  for (int64_t i = 0; i < n; i++) {
    if (agg1[i] >= 0) continue;
    double best = -1.0;
    int32_t to = -1;
    for (int64_t k = L.rp[i]; k < L.rp[i + 1]; k++) {
      const int32_t a = agg1[L.ci[k]];
      if (a >= 0 && std::abs(L.off[k]) > best) {
        best = std::abs(L.off[k]);
        to = a;
      }
    }
    agg[i] = to;
  }
  for (int64_t i = 0; i < n; i++)
    if (agg[i] < 0) agg[i] = (int32_t)na++;
  return na;
}

// Coarse graph + Galerkin plans for plain aggregation, and the coarse values
// (host copy, used for the next level's strength test).
void coarsen(HostLevel &F, HostLevel &C, double theta) {
  const int64_t n = F.n;
  const int64_t na = aggregate(F, F.agg, theta);
  C.n = na;
  // aggregates never cross systems (no edges between them); number them
  // system by system so every level keeps contiguous system ranges
  {
    const int64_t ns = (int64_t)F.soff.size() - 1;
    std::vector<int32_t> asys(na, 0);
    for (int64_t sy = 0; sy < ns; sy++)
      for (int64_t i = F.soff[sy]; i < F.soff[sy + 1]; i++) asys[F.agg[i]] = (int32_t)sy;
    std::vector<int32_t> order(na);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return asys[a] < asys[b]; });
    std::vector<int32_t> renum(na);
    for (int64_t q = 0; q < na; q++) renum[order[q]] = (int32_t)q;
    for (int64_t i = 0; i < n; i++) F.agg[i] = renum[F.agg[i]];
    C.soff.assign(ns + 1, 0);
    for (int64_t a = 0; a < na; a++) C.soff[asys[order[a]] + 1]++;
    for (int64_t sy = 0; sy < ns; sy++) C.soff[sy + 1] += C.soff[sy];
  }
  // members
  F.mem_ptr.assign(na + 1, 0);
  for (int64_t i = 0; i < n; i++) F.mem_ptr[F.agg[i] + 1]++;
  for (int64_t a = 0; a < na; a++) F.mem_ptr[a + 1] += F.mem_ptr[a];
  F.mem_idx.resize(n);
  {
    std::vector<int32_t> fill(F.mem_ptr.begin(), F.mem_ptr.end() - 1);
    for (int64_t i = 0; i < n; i++) F.mem_idx[fill[F.agg[i]]++] = (int32_t)i;
  }
  // coarse rows: unique neighbour aggregates
  C.rp.assign(na + 1, 0);
  std::vector<std::vector<int32_t>> rows(na);
  for (int64_t a = 0; a < na; a++) {
    auto &r = rows[a];
    for (int32_t q = F.mem_ptr[a]; q < F.mem_ptr[a + 1]; q++) {
      const int32_t i = F.mem_idx[q];
      for (int32_t k = F.rp[i]; k < F.rp[i + 1]; k++) {
        const int32_t b = F.agg[F.ci[k]];
        if (b != a) r.push_back(b);
      }
    }
    std::sort(r.begin(), r.end());
    r.erase(std::unique(r.begin(), r.end()), r.end());
    C.rp[a + 1] = C.rp[a] + (int32_t)r.size();
  }
  C.ci.resize(C.rp[na]);
  for (int64_t a = 0; a < na; a++) std::copy(rows[a].begin(), rows[a].end(), C.ci.begin() + C.rp[a]);
  // plans: each fine nonzero goes either to one coarse nonzero or to the
  // coarse diagonal of its aggregate
  const int64_t nzc = C.rp[na];
  std::vector<int32_t> target(F.rp[n]);
  std::vector<int32_t> cnt(nzc + 1, 0), icnt(na + 1, 0);
  for (int64_t i = 0; i < n; i++) {
    const int32_t a = F.agg[i];
    for (int32_t k = F.rp[i]; k < F.rp[i + 1]; k++) {
      const int32_t b = F.agg[F.ci[k]];
      if (b == a) {
        target[k] = -1;
        icnt[a + 1]++;
      } else {
        const int32_t *rb = C.ci.data() + C.rp[a], *re = C.ci.data() + C.rp[a + 1];
        const int32_t t = (int32_t)(std::lower_bound(rb, re, b) - C.ci.data());
        target[k] = t;
        cnt[t + 1]++;
      }
    }
  }
  for (int64_t t = 0; t < nzc; t++) cnt[t + 1] += cnt[t];
  for (int64_t a = 0; a < na; a++) icnt[a + 1] += icnt[a];
  F.seg_ptr = cnt;
  F.intra_ptr = icnt;
  F.seg_idx.resize(cnt[nzc]);
  F.intra_idx.resize(icnt[na]);
  {
    std::vector<int32_t> fs(cnt.begin(), cnt.end() - 1), fi(icnt.begin(), icnt.end() - 1);
    for (int64_t i = 0; i < n; i++)
      for (int32_t k = F.rp[i]; k < F.rp[i + 1]; k++) {
        if (target[k] >= 0) F.seg_idx[fs[target[k]]++] = k;
        else F.intra_idx[fi[F.agg[i]]++] = k;
      }
  }
  // coarse values (host, same arithmetic as the GPU refresh)
  C.off.assign(nzc, 0.0);
  for (int64_t t = 0; t < nzc; t++)
    for (int32_t q = F.seg_ptr[t]; q < F.seg_ptr[t + 1]; q++) C.off[t] += F.off[F.seg_idx[q]];
  C.dia.assign(3 * na, 0.0);
  for (int64_t a = 0; a < na; a++) {
    for (int32_t q = F.mem_ptr[a]; q < F.mem_ptr[a + 1]; q++) {
      const int32_t i = F.mem_idx[q];
      for (int c = 0; c < 3; c++) C.dia[3 * a + c] += F.dia[3 * i + c];
    }
    for (int32_t q = F.intra_ptr[a]; q < F.intra_ptr[a + 1]; q++) {
      const double re = F.off[F.intra_idx[q]].real();
      C.dia[3 * a] += re;
      C.dia[3 * a + 1] += re;
    }
  }
}

// ------------------------------------------------------------- kernels
// coarse off-diagonal values: sum of the fine nonzeros of each segment
template <typename T>
__global__ void rap_offdiag(int64_t nzc, const int32_t *__restrict__ ptr,
                            const int32_t *__restrict__ idx, const C2<T> *__restrict__ fine,
                            C2<T> *__restrict__ coarse) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nzc) return;
  T sr = 0, si = 0;
  for (int32_t q = ptr[t]; q < ptr[t + 1]; q++) {
    const C2<T> v = fine[idx[q]];
    sr += v.x;
    si += v.y;
  }
  coarse[t] = C2<T>{sr, si};
}

// coarse diagonal blocks: member diagonal blocks + real parts of the
// intra-aggregate couplings (their imaginary parts cancel pairwise)
template <typename T>
__global__ void rap_diag(int64_t na, const int32_t *__restrict__ mptr,
                         const int32_t *__restrict__ midx, const int32_t *__restrict__ iptr,
                         const int32_t *__restrict__ iidx, const T *__restrict__ fdia,
                         const C2<T> *__restrict__ foff, T *__restrict__ cdia) {
  const int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (a >= na) return;
  T d0 = 0, d1 = 0, d2 = 0;
  for (int32_t q = mptr[a]; q < mptr[a + 1]; q++) {
    const int32_t i = midx[q];
    d0 += fdia[3 * i];
    d1 += fdia[3 * i + 1];
    d2 += fdia[3 * i + 2];
  }
  for (int32_t q = iptr[a]; q < iptr[a + 1]; q++) {
    const T re = foff[iidx[q]].x;
    d0 += re;
    d1 += re;
  }
  cdia[3 * a] = d0;
  cdia[3 * a + 1] = d1;
  cdia[3 * a + 2] = d2;
}

// sum_j |a_ij| per row (the loop dinv_gershgorin runs without rowabs)
template <typename T>
__global__ void row_abs_sums(int64_t n, const int32_t *__restrict__ rp, const C2<T> *__restrict__ off,
                             T *__restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  T s = 0;
  for (int32_t k = rp[i]; k < rp[i + 1]; k++) {
    const C2<T> v = off[k];
    s += sqrt(v.x * v.x + v.y * v.y);
  }
  out[i] = s;
}

// The smoother's Chebyshev polynomial on [lmax / ratio, 1.1 lmax]: its
// centre and half width are multiples of lmax, so everything but 1 / lmax is
// a constant of the degree and the ratio: coef[0] = c0 / lmax, then per step
// k >= 1 the pair (p[k] = rho_k rho_{k-1}, q[k] / lmax = 2 rho_k / delta).
constexpr int kMaxDegree = 8;  // of the smoother (nosh_nls_set_amg_options)
struct ChebSpec {
  int deg;
  double c0, p[kMaxDegree], q[kMaxDegree];
  static ChebSpec of(int deg, double ratio) {
    ChebSpec s{};
    s.deg = deg;
    const double lmin = 1.0 / (1.1 * ratio), theta = 0.5 * (1.0 + lmin), delta = 0.5 * (1.0 - lmin);
    const double sigma = theta / delta;
    double rho = 1.0 / sigma;
    s.c0 = 1.0 / theta;
    for (int k = 1; k < deg; k++) {
      const double rn = 1.0 / (2.0 * sigma - rho);
      s.p[k] = rn * rho;
      s.q[k] = 2.0 * rn / delta;
      rho = rn;
    }
    return s;
  }
};

__device__ __forceinline__ void inv3(double det, double a, double d, double b, double *o) {
  const double r = 1.0 / det;  // one FP64 division instead of three
  o[0] = d * r;
  o[1] = a * r;
  o[2] = -b * r;
}
__device__ __forceinline__ void inv3(float det, float a, float d, float b, float *o) {
  o[0] = d / det;
  o[1] = a / det;
  o[2] = -b / det;
}

// Inverse diagonal blocks and the Gershgorin bound of lambda_max(D^-1 A),
// 1 + ||D_i^-1||_2 sum_j |a_ij| reduced by max over rows (arithmetic in T;
// rowabs: the rows' sums of |a_ij| when known, else summed here); the last
// CTA to finish turns it into the level's Chebyshev coefficients.  The bound
// is compared as the bits of a non-negative double, which order alike: an
// FP64 maximum would be FP64 instructions.  *lmax_bits and *arrive are zero
// between launches.
template <typename T>
__global__ void dinv_gershgorin(int64_t n, const int32_t *__restrict__ rp, const C2<T> *__restrict__ off,
                                const T *__restrict__ dia, T *__restrict__ dinv, unsigned long long *lmax_bits,
                                unsigned *arrive, int *err, const T *__restrict__ rowabs, ChebSpec spec, T *coef) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  unsigned long long v = 0;
  if (i < n) {
    const T a = dia[3 * i], d = dia[3 * i + 1], b = dia[3 * i + 2];
    const T det = a * d - b * b;
    inv3(det, a, d, b, dinv + 3 * i);
    const T lmin = (T)0.5 * (a + d) - sqrt((T)0.25 * (a - d) * (a - d) + b * b);
    T s = 0;
    if (rowabs) {
      s = rowabs[i];
    } else {
      for (int32_t k = rp[i]; k < rp[i + 1]; k++) {
        const C2<T> w = off[k];
        s += sqrt(w.x * w.x + w.y * w.y);
      }
    }
    const double bound = (lmin > 0 && det > 0) ? 1.0 + (double)(s / lmin) : 1e300;
    v = (unsigned long long)__double_as_longlong(bound);
    // a diagonal block that is not positive definite: the operator is not
    // SPD (a g < 0 regularisation), so neither is the V-cycle
    if (!(lmin > 0 && det > 0)) atomicOr(err, 32);
  }
  __shared__ unsigned long long sm[32];
  auto warp_max = [](unsigned long long u) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) u = max(u, __shfl_xor_sync(0xffffffffu, u, o));
    return u;
  };
  v = warp_max(v);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  v = warp_max(threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0ull);
  if (threadIdx.x != 0) return;
  atomicMax(lmax_bits, v);
  if (arrive_acq_rel(arrive) != gridDim.x - 1) return;
  const double il = 1.0 / (1.1 * __longlong_as_double((long long)atomicExch(lmax_bits, 0ull)));
  *arrive = 0u;
  coef[0] = (T)(spec.c0 * il);
  for (int k = 1; k < spec.deg; k++) {
    coef[2 * k] = (T)spec.p[k];
    coef[2 * k + 1] = (T)(spec.q[k] * il);
  }
}

// ---- smoother building blocks (shared by the grid kernels and the tail)
// d = c0 D^-1 b, x = d  (first Chebyshev step from x = 0)
template <typename T>
__device__ __forceinline__ void cheb_first_elem(int64_t i, const T *dinv, T c0, C2<T> bi, C2<T> *d,
                                                C2<T> *x) {
  const T a = dinv[3 * i], e = dinv[3 * i + 1], f = dinv[3 * i + 2];
  const C2<T> di{c0 * (a * bi.x + f * bi.y), c0 * (f * bi.x + e * bi.y)};
  d[i] = di;
  x[i] = di;
}

// Chebyshev step k given (sr, si) = (offdiag A x_in)_i:
// r = D^-1 (b - A x_in), d = c1 d + c2 r (d = c0 r for k == 0), x_out = x_in + d
template <typename T>
struct ChebPre {
  C2<T> xi, bi, dold;
  T d0r, d0i, d1b, a, e, f;
};
template <typename T>
__device__ __forceinline__ ChebPre<T> cheb_load(int64_t i, int k, const T *dia, const T *dinv, const C2<T> *b,
                                                const C2<T> *xin, const C2<T> *d) {
  ChebPre<T> p;
  p.xi = xin[i];
  p.bi = b[i];
  p.d0r = dia[3 * i];
  p.d0i = dia[3 * i + 1];
  p.d1b = dia[3 * i + 2];
  p.a = dinv[3 * i];
  p.e = dinv[3 * i + 1];
  p.f = dinv[3 * i + 2];
  p.dold = k == 0 ? C2<T>{0, 0} : d[i];
  return p;
}
template <typename T>
__device__ __forceinline__ C2<T> cheb_apply(int64_t i, int k, T sr, T si, const ChebPre<T> &p, const T *coef,
                                            C2<T> *d, C2<T> *xout) {
  const T rr = p.bi.x - (sr + p.d0r * p.xi.x + p.d1b * p.xi.y);
  const T ri = p.bi.y - (si + p.d1b * p.xi.x + p.d0i * p.xi.y);
  const T zr = p.a * rr + p.f * ri, zi = p.f * rr + p.e * ri;
  C2<T> dn;
  if (k == 0) {
    dn = C2<T>{coef[0] * zr, coef[0] * zi};
  } else {
    const T c1 = coef[2 * k], c2 = coef[2 * k + 1];
    dn = C2<T>{c1 * p.dold.x + c2 * zr, c1 * p.dold.y + c2 * zi};
  }
  d[i] = dn;
  const C2<T> xo{p.xi.x + dn.x, p.xi.y + dn.y};
  xout[i] = xo;
  return xo;
}

template <typename T>
__global__ void cheb_first(int64_t n, const T *__restrict__ dinv, const T *__restrict__ coef,
                           const C2<T> *__restrict__ b, C2<T> *__restrict__ d,
                           C2<T> *__restrict__ x) {
  dep_sync();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  cheb_first_elem<T>(i, dinv, coef[0], b[i], d, x);
}

// MINRES head fused with the first Chebyshev step of the fine level:
// r_new = J z / beta - (beta/oldb) r_old - (alfa/beta) r_cur over r_old, then
// d = c0 D^-1 r_new, x = d
template <typename T>
__global__ void lanczos_first(int64_t n, const MinresScalars *__restrict__ s,
                              const C2<T> *__restrict__ u, C2<T> *__restrict__ r_old,
                              const C2<T> *__restrict__ r_cur, const T *__restrict__ dinv,
                              const T *__restrict__ coef, C2<T> *__restrict__ d, C2<T> *__restrict__ x) {
  dep_sync();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n || s->done >= 2) return;
  const T *la = lanczos_coef<T>(s);
  const T a = la[0], bb = la[1], c = la[2];
  const C2<T> ui = u[i], ro = r_old[i], rc = r_cur[i];
  const C2<T> bi{a * ui.x - bb * ro.x - c * rc.x, a * ui.y - bb * ro.y - c * rc.y};
  r_old[i] = bi;
  cheb_first_elem<T>(i, dinv, coef[0], bi, d, x);
}

// The same for a union of systems: each vertex takes its system's
// coefficients, a frozen system's new vector is zero.
template <typename T>
__global__ void lanczos_first_sys(int64_t n, const int32_t *__restrict__ vsys, const MinresScalars *__restrict__ sc,
                                  const C2<T> *__restrict__ u, C2<T> *__restrict__ r_old,
                                  const C2<T> *__restrict__ r_cur, const T *__restrict__ dinv,
                                  const T *__restrict__ coef, C2<T> *__restrict__ d, C2<T> *__restrict__ x,
                                  const int *halt) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const MinresScalars *s = sc + (i < n ? vsys[i] : 0);
  dep_sync();
  if (i >= n || (halt && *halt >= 2)) return;
  const C2<T> ui = u[i], ro = r_old[i], rc = r_cur[i];
  const T *la = lanczos_coef<T>(s);
  const T a = la[0], bb = la[1], c = la[2];
  C2<T> bi{a * ui.x - bb * ro.x - c * rc.x, a * ui.y - bb * ro.y - c * rc.y};
  if (s->done >= 2) bi = C2<T>{0, 0};
  r_old[i] = bi;
  cheb_first_elem<T>(i, dinv, coef[0], bi, d, x);
}

// Chebyshev step with SpMV (grid kernel epilogue)
template <typename T>
struct ChebOp {
  static constexpr bool kReduce = false;
  const T *dia, *dinv, *coef;
  int step;
  const C2<T> *b, *xin;
  C2<T> *d, *xout;
  const int *halt = nullptr;
  using Pre = ChebPre<T>;
  __device__ Pre load(int i) const { return cheb_load<T>(i, step, dia, dinv, b, xin, d); }
  __device__ double finish(int i, T sr, T si, const Pre &p) const {
    cheb_apply<T>(i, step, sr, si, p, coef, d, xout);
    return 0.0;
  }
};

// Last post-smoothing step of the fine level inside MINRES: also reduces
// <r_new, z_new> and, in the finishing thread, advances the Givens recurrence.
template <typename T>
struct ChebMinresOp {
  static constexpr bool kReduce = true;
  static constexpr bool kHook = true;
  const T *dia, *dinv, *coef;
  int step;
  const C2<T> *b, *xin;
  C2<T> *d, *xout;
  MinresScalars *s;
  const int *halt = nullptr;
  using Pre = ChebPre<T>;
  __device__ Pre load(int i) const { return cheb_load<T>(i, step, dia, dinv, b, xin, d); }
  __device__ double finish(int i, T sr, T si, const Pre &p) const {
    const C2<T> z = cheb_apply<T>(i, step, sr, si, p, coef, d, xout);
    return (double)p.bi.x * (double)z.x + (double)p.bi.y * (double)z.y;
  }
  static constexpr int kHeadWords = kMinresHeadWords;
  __device__ const double *head() const { return reinterpret_cast<const double *>(s); }
  __device__ void hook(double total, const double *state) const { minres_advance(s, state, total); }
};

// The fine level's last step of a batch: also rowdot[i] = <b_i, x_i>.
template <typename T>
struct ChebRowDotOp {
  static constexpr bool kReduce = false;
  const T *dia, *dinv, *coef;
  int step;
  const C2<T> *b, *xin;
  C2<T> *d, *xout;
  double *rowdot;
  const int *halt = nullptr;
  using Pre = ChebPre<T>;
  __device__ Pre load(int i) const { return cheb_load<T>(i, step, dia, dinv, b, xin, d); }
  __device__ double finish(int i, T sr, T si, const Pre &p) const {
    const C2<T> z = cheb_apply<T>(i, step, sr, si, p, coef, d, xout);
    rowdot[i] = (double)p.bi.x * (double)z.x + (double)p.bi.y * (double)z.y;
    return 0.0;
  }
};

// res = b - A x
template <typename T>
struct ResidOp {
  static constexpr bool kReduce = false;
  const T *dia;
  const C2<T> *b, *x;
  C2<T> *res;
  const int *halt = nullptr;
  bool trigger = false;
  struct Pre {
    C2<T> xi, bi;
    T d0r, d0i, d1b;
  };
  __device__ Pre load(int i) const { return Pre{x[i], b[i], dia[3 * i], dia[3 * i + 1], dia[3 * i + 2]}; }
  __device__ double finish(int i, T sr, T si, const Pre &p) const {
    res[i] = C2<T>{p.bi.x - (sr + p.d0r * p.xi.x + p.d1b * p.xi.y),
                   p.bi.y - (si + p.d1b * p.xi.x + p.d0i * p.xi.y)};
    return 0.0;
  }
};

// Restriction: aggregate sums of the finer level's residual, LN lanes per
// aggregate and then a shuffle tree, so the coarse levels' few thousand
// aggregates spread over the whole GPU instead of a few dozen CTAs each
// walking its members serially.  In FP32 a lane takes every LN-th member, both
// components.  In FP64 the launch's time is that of its additions, and a lane
// pair takes the two components of every LN / 2-th member: half the additions
// of the tree.  The two restrictions of a cycle over 226 K vertices of
// triangle meshes 9.0 -> 6.3 us each; 6.1 us at 32^3 tetrahedral, where 4 lanes
// with both components took 8.6.
template <typename T, int LN>
__device__ __forceinline__ C2<T> aggregate_sum(int64_t a, int64_t na, int li, const int32_t *__restrict__ mptr,
                                               const int32_t *__restrict__ midx, const C2<T> *__restrict__ r) {
  if (sizeof(T) == 8) {
    const T *rc = reinterpret_cast<const T *>(r) + (li & 1);
    T s = 0;
    if (a < na)
      for (int32_t q = mptr[a] + (li >> 1); q < mptr[a + 1]; q += LN / 2) s += rc[2 * (int64_t)midx[q]];
#pragma unroll
    for (int o = LN / 2; o > 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return C2<T>{s, __shfl_xor_sync(0xffffffffu, s, 1)};
  }
  T sr = 0, si = 0;
  if (a < na)
    for (int32_t q = mptr[a] + li; q < mptr[a + 1]; q += LN) {
      const C2<T> v = r[midx[q]];
      sr += v.x;
      si += v.y;
    }
#pragma unroll
  for (int o = LN / 2; o > 0; o >>= 1) {
    sr += __shfl_xor_sync(0xffffffffu, sr, o);
    si += __shfl_xor_sync(0xffffffffu, si, o);
  }
  return C2<T>{sr, si};
}
// Lanes per aggregate: half of them where an aggregate has few members (of a
// triangle mesh some 9, of a tetrahedral one some 25) and the sums are FP64.
template <typename T>
inline bool few_members(int64_t n, int64_t na) {
  return sizeof(T) == 8 && n <= 14 * na;
}

template <typename T, int LN>
__global__ void restrict_kernel(int64_t na, const int32_t *__restrict__ mptr,
                                const int32_t *__restrict__ midx, const C2<T> *__restrict__ r,
                                C2<T> *__restrict__ rc, const int *halt) {
  dep_sync();
  if (halt && *halt >= 2) return;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t a = t / LN;
  const int li = (int)(t % LN);
  const C2<T> b = aggregate_sum<T, LN>(a, na, li, mptr, midx, r);
  if (a < na && li == 0) rc[a] = b;
}

// restriction fused with the coarse level's first Chebyshev step
template <typename T, int LN>
__global__ void restrict_first(int64_t na, const int32_t *__restrict__ mptr,
                               const int32_t *__restrict__ midx, const C2<T> *__restrict__ r,
                               C2<T> *__restrict__ rc, const T *__restrict__ dinv,
                               const T *__restrict__ coef, C2<T> *__restrict__ d,
                               C2<T> *__restrict__ x, const int *halt) {
  dep_sync();
  if (halt && *halt >= 2) return;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t a = t / LN;
  const int li = (int)(t % LN);
  const C2<T> b = aggregate_sum<T, LN>(a, na, li, mptr, midx, r);
  if (a < na && li == 0) {
    rc[a] = b;
    cheb_first_elem<T>(a, dinv, coef[0], b, d, x);
  }
}

template <typename T>
__global__ void prolong_kernel(int64_t n, const int32_t *__restrict__ agg,
                               const C2<T> *__restrict__ xc, C2<T> *__restrict__ x, const int *halt) {
  dep_sync();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n || (halt && *halt >= 2)) return;
  const C2<T> c = xc[agg[i]];
  C2<T> v = x[i];
  v.x += c.x;
  v.y += c.y;
  x[i] = v;
}

// Dense real matrix (m = 2n) of the coarsest level from its compact form.
template <typename T>
__global__ void coarse_dense(int64_t n, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                             const C2<T> *__restrict__ off, const T *__restrict__ dia,
                             const int32_t *__restrict__ bstart, const int64_t *__restrict__ rowoff,
                             const int32_t *__restrict__ bdim, double *A) {
  // the coarsest level is block diagonal (one block per system): node i's
  // two real rows live in its block's packed dense matrix
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t m = bdim[2 * i];
  const int64_t s0 = bstart[2 * i];  // first real row of the block
  double *r0 = A + rowoff[2 * i], *r1 = A + rowoff[2 * i + 1];
  for (int64_t j = 0; j < m; j++) {
    r0[j] = 0.0;
    r1[j] = 0.0;
  }
  const int64_t li = 2 * i - s0;
  r0[li] = dia[3 * i];
  r0[li + 1] = dia[3 * i + 2];
  r1[li] = dia[3 * i + 2];
  r1[li + 1] = dia[3 * i + 1];
  for (int32_t k = rp[i]; k < rp[i + 1]; k++) {
    const int64_t lj = 2 * (int64_t)ci[k] - s0;
    const C2<T> v = off[k];  // block [[re, -im], [im, re]]
    r0[lj] = v.x;
    r0[lj + 1] = -v.y;
    r1[lj] = v.y;
    r1[lj + 1] = v.x;
  }
}

// Gauss-Jordan inversion of the coarsest level's SPD blocks (no pivoting
// needed), kPivots pivots a launch, in FP64.  A CTA owns kPivotCols columns of
// a block: it inverts the pivot block P (every CTA does), takes R = P^-1 times
// its columns' pivot rows and subtracts the pivot columns times R from the
// other rows; a column of the pivot block itself starts from the identity.  It
// reads src and writes dst, since every CTA reads the pivot columns.  After the
// last launch the FP32 copy is written as well.
//
// Most of a launch's 13 us in FP64 is the chain of 16 reciprocals and updates
// of P.  One CTA a block was bound by the FP64 pipe of its multiprocessor, m^3
// multiply-adds: 661 -> 104 us for a block of 128 rows, 35 -> 26 us for one of
// 32 (an FP64 continuation at 32^3 with two of the former 16.2 -> 14.8 ms).
constexpr int kPivots = 16, kPivotCols = 2, kPivotThreads = 128;
__global__ void __launch_bounds__(kPivotThreads)
    gauss_jordan_step(const int64_t *__restrict__ boff, const int32_t *__restrict__ bd, int k0, int last,
                      const double *__restrict__ src, double *__restrict__ dst, float *__restrict__ Afg, int *err) {
  const int m = bd[blockIdx.x], j0 = blockIdx.y * kPivotCols;
  if (j0 >= m) return;
  const double *A = src + boff[blockIdx.x];
  double *B = dst + boff[blockIdx.x];
  float *Af = last ? Afg + boff[blockIdx.x] : nullptr;
  const int nc = min(kPivotCols, m - j0), nk = min(kPivots, m - k0);
  dep_sync();
  if (nk <= 0) {  // a smaller block, inverted by an earlier launch
    for (int q = threadIdx.x; q < m * kPivotCols; q += kPivotThreads) {
      const int jj = q % kPivotCols;
      const int64_t at = (int64_t)(q / kPivotCols) * m + j0 + jj;
      if (jj >= nc) continue;
      B[at] = A[at];
      if (last) Af[at] = (float)A[at];
    }
    return;
  }
  __shared__ double P[2][kPivots][kPivots + 1], Y[kPivots][kPivotCols], R[kPivots][kPivotCols];
  const int r = threadIdx.x / (kPivots / 2), c = threadIdx.x % (kPivots / 2) * 2;
#pragma unroll
  for (int q = 0; q < 2; q++) P[0][r][c + q] = r < nk && c + q < nk ? A[(int64_t)(k0 + r) * m + k0 + c + q] : 0.0;
  if (threadIdx.x < kPivots * kPivotCols) {
    const int l = threadIdx.x / kPivotCols, jj = threadIdx.x % kPivotCols;
    Y[l][jj] = l < nk && jj < nc ? A[(int64_t)(k0 + l) * m + j0 + jj] : 0.0;
  }
  __syncthreads();
  for (int k = 0; k < nk; k++) {
    const double(*S)[kPivots + 1] = P[k & 1];
    const double piv = S[k][k];
    if (threadIdx.x == 0 && blockIdx.y == 0 && !(piv > 0.0)) atomicOr(err, 16);
    const double ip = 1.0 / piv;
    const double f = r == k ? ip : -S[r][k] * ip;
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const double a = c + q == k ? 0.0 : S[r][c + q], pk = c + q == k ? 1.0 : S[k][c + q];
      P[(k & 1) ^ 1][r][c + q] = r == k ? pk * f : a + f * pk;
    }
    __syncthreads();
  }
  const double(*S)[kPivots + 1] = P[nk & 1];
  if (threadIdx.x < kPivots * kPivotCols) {
    const int l = threadIdx.x / kPivotCols, jj = threadIdx.x % kPivotCols, jp = j0 + jj - k0;
    double v = 0;
    if (jp >= 0 && jp < nk) {
      v = l < nk ? S[l][jp] : 0.0;
    } else {
#pragma unroll
      for (int q = 0; q < kPivots; q++) v += S[l][q] * Y[q][jj];
    }
    R[l][jj] = v;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < m; i += kPivotThreads) {
    const int ip = i - k0;
    const bool pivot_row = ip >= 0 && ip < nk;
    double v[kPivotCols];
#pragma unroll
    for (int jj = 0; jj < kPivotCols; jj++) {
      const int jp = j0 + jj - k0;
      v[jj] = pivot_row ? R[ip][jj] : jj >= nc || (jp >= 0 && jp < nk) ? 0.0 : A[(int64_t)i * m + j0 + jj];
    }
    if (!pivot_row)
#pragma unroll
      for (int q = 0; q < kPivots; q++) {
        const double a = q < nk ? A[(int64_t)i * m + k0 + q] : 0.0;
#pragma unroll
        for (int jj = 0; jj < kPivotCols; jj++) v[jj] -= a * R[q][jj];
      }
#pragma unroll
    for (int jj = 0; jj < kPivotCols; jj++)
      if (jj < nc) {
        B[(int64_t)i * m + j0 + jj] = v[jj];
        if (last) Af[(int64_t)i * m + j0 + jj] = (float)v[jj];
      }
  }
}
// The same in FP32 on the mixed path, one CTA a block of up to kDenseFp32 rows
// in shared memory (43 us for 54 rows, bound by its barriers); larger blocks
// are inverted in FP64 there too.  An FP64 solve that follows on the handle
// works with this inverse until its own refresh, and the rounding of the
// elimination shows in its iterates: by blocks of pivots (20 us) they moved by
// 1e-10 to 1e-9 relative, so the mixed path keeps this order.
constexpr int kDenseFp32 = 128;
__global__ void gauss_jordan_fp32(const int64_t *__restrict__ boff, const int32_t *__restrict__ bd, double *Ag,
                                  float *Afg, int *err) {
  // one CTA per diagonal block of the coarsest level
  const int m = bd[blockIdx.x];
  double *A = Ag + boff[blockIdx.x];
  float *Af = Afg + boff[blockIdx.x];
  extern __shared__ __align__(16) unsigned char gj_raw[];
  float *S = reinterpret_cast<float *>(gj_raw);
  __shared__ float ip_s;
  for (int q = threadIdx.x; q < m * m; q += blockDim.x) S[q] = (float)A[q];
  __syncthreads();
  for (int k = 0; k < m; k++) {
    if (threadIdx.x == 0) {
      const float piv = S[k * m + k];
      if (!(piv > 0.f)) atomicOr(err, 16);
      ip_s = 1.f / piv;
    }
    __syncthreads();
    const float ip = ip_s;
    for (int j = threadIdx.x; j < m; j += blockDim.x) S[k * m + j] = (j == k) ? ip : S[k * m + j] * ip;
    __syncthreads();
    for (int q = threadIdx.x; q < m * m; q += blockDim.x) {
      const int i = q / m, j = q % m;
      if (i == k || j == k) continue;
      S[q] -= S[i * m + k] * S[k * m + j];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += blockDim.x)
      if (i != k) S[i * m + k] = -S[i * m + k] * ip;
    __syncthreads();
  }
  for (int q = threadIdx.x; q < m * m; q += blockDim.x) {
    A[q] = (double)S[q];
    Af[q] = S[q];
  }
}

// Packed block-diagonal dense inverse: real row i of the coarsest level is
// row rowoff[i] of the packed array, its block starts at real row bstart[i]
// and has bdim[i] columns.
struct DenseMap {
  const int64_t *rowoff;
  const int32_t *bstart, *bdim;
};
// x = Ainv b, a half-warp per real row (a batch's coarsest level, or a
// hierarchy of one level)
constexpr int kDenseLanes = 16;
template <typename T>
__global__ void dense_matvec(int m, const T *__restrict__ Ainv, DenseMap D, const T *__restrict__ b,
                             T *__restrict__ x, const int *halt) {
  dep_sync();
  if (halt && *halt >= 2) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x, i = t / kDenseLanes, li = t % kDenseLanes;
  T s = 0;
  if (i < m) {
    const T *a = Ainv + D.rowoff[i], *bb = b + D.bstart[i];
    const int n = D.bdim[i];
#pragma unroll 4
    for (int j = li; j < n; j += kDenseLanes) s = fma(a[j], bb[j], s);
  }
#pragma unroll
  for (int o = kDenseLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (i < m && li == 0) x[i] = s;
}

// ---- the resident V-cycle: every level from `lt` down, in one launch of one
// thread-block cluster.
//
// The coarse levels are latency: a few hundred to a thousand rows, five SpMVs
// each.  A launch per step costs about 3 us; one CTA for all of them left the
// FP64 pipe of a single SM as the bound (a 737-node level of the 65^2 square:
// 65 us a cycle, 79 % of that pipe).  Here the rows of a level are spread over
// the CTAs of a cluster (16, which needs the opt-in above the portable 8) and
// each level's vectors live in shared memory, replicated in every CTA: a row's
// result is sent to all CTAs by asynchronous stores that complete on the
// phase's mbarrier in the receiving CTA, and every gather is a local shared-
// memory read.  A CTA goes on as soon as it has the whole vector; a cluster
// barrier per phase instead measured 1000-1400 cycles of each phase's 2800.
// Each CTA's rows of the operators are staged in its shared memory while the
// predecessor (which triggers this launch at its start) runs.
//
// A vector may be overwritten by other CTAs as soon as they have the vector
// of the phase that reads it: each sends its rows of that phase only after
// its own reads, and nobody goes on without all rows.
//
// The waits are bounded.  A thread whose wait runs out flags it to the host,
// waits for nothing more and goes through the remaining phases all the same
// (their results are invalid), so every CTA sends all that the others expect.
// At the end it waits once more, with a bound, for all of it: no store is to
// land in the shared memory of a CTA that has left.
//
// A row is summed by LN lanes: even lanes its real component, odd lanes its
// imaginary one (two FMAs a nonzero each, no reduction between the two), and
// LN/2 parts of the row.  FP64 takes just enough lanes for a warp on each of
// the SM's four FP64 pipes, since idle lanes of a warp cost as much as busy
// ones and every shuffle step of a wider split is more FP64 adds; FP32 splits
// up to sixteen ways.
constexpr int kTailThreads = 512;
constexpr int kTailSmem = 200 * 1024;  // shared memory of one CTA, at most

template <typename T>
struct LevelDesc {
  int n, rw;   // rows, rows per CTA (CTA r owns [r rw, (r + 1) rw))
  int lnb;     // log2 of the lanes per row
  const int32_t *rp, *ci;
  const C2<T> *off;
  const T *dia, *dinv, *coef;
  const int32_t *agg, *mem_ptr, *mem_idx;  // transfer to the next level
  // shared-memory byte offsets: two replicated vectors, the own rows' right-
  // hand side and Chebyshev direction, the own rows of the operator (row
  // pointers, columns, values, diagonal blocks and their inverses), this
  // level's aggregates, the own members of this level's nodes (a list over
  // the finer level)
  uint32_t xa, xb, b, d, s_rp, s_ci, s_off, s_dia, s_agg, s_mp, s_mi;
};

enum TailHead { kHeadRestrict = 0, kHeadVector = 1, kHeadLanczos = 2 };
enum TailOut { kOutProlong = 0, kOutVector = 1, kOutMinres = 2 };

// Where the resident cycle starts and ends: the finer level's residual,
// iterate and aggregates (restriction in, prolongation out), or a vector in
// and out (the whole V-cycle, lt = 0), the MINRES step's Lanczos vector in and
// its Givens step out.
template <typename T>
struct TailArgs {
  int head, out;
  const C2<T> *f_res;
  C2<T> *f_x;
  const int32_t *f_agg, *f_mp, *f_mi;
  int64_t f_n;
  const C2<T> *b;      // kHeadVector; kHeadLanczos: J z
  C2<T> *r_old;        // kHeadLanczos: r_old in, the new Lanczos vector out
  const C2<T> *r_cur;
  C2<T> *z;            // kOutVector, kOutMinres
  MinresScalars *ms;
  unsigned *fail;           // (pinned host memory) set when a wait for a phase's vector gives up
  const unsigned *counter;  // kStageWaitSlot: diagnostic override of the waits' bound
};

// The coarsest level's dense inverse in shared memory (byte offsets): the own
// real rows, packed as in global memory, and their (offset, first column,
// columns); staged when it fits.
struct TailDense {
  uint32_t s_bd, s_xd, s_a, s_map;
  int staged;
};

// phases of a level: the first step, deg - 1 pre-smoothing steps, the
// residual, deg post-smoothing steps; two for the coarsest level
__host__ __device__ constexpr int tail_phases(int levels, int deg) { return (levels - 1) * (2 * deg + 1) + 2; }

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory"); }
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, int rank) {
  uint32_t ra;
  asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(addr), "r"(rank));
  return ra;
}
// store to another CTA's shared memory, completing on its mbarrier
__device__ __forceinline__ void st_async(uint32_t addr, uint32_t bar, int rank, C2<float> v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];\n" ::"r"(
                   map_rank(addr, rank)),
               "f"(v.x), "f"(v.y), "r"(map_rank(bar, rank))
               : "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, uint32_t bar, int rank, C2<double> v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];\n" ::"r"(
                   map_rank(addr, rank)),
               "d"(v.x), "d"(v.y), "r"(map_rank(bar, rank))
               : "memory");
}

// sign flip by the sign bit (a select between a value and its negative costs
// an FP64 instruction otherwise)
__device__ __forceinline__ float flip(float v, unsigned mask) { return __uint_as_float(__float_as_uint(v) ^ mask); }
__device__ __forceinline__ double flip(double v, unsigned mask) {
  return __hiloint2double(__double2hiint(v) ^ (int)mask, __double2loint(v));
}

extern __shared__ __align__(16) unsigned char tail_sm[];
template <typename V>
__device__ __forceinline__ V &tail_at(uint32_t o, int i = 0) {
  return *(reinterpret_cast<V *>(tail_sm + o) + i);
}

// The cluster as one thread sees it.
struct TailTeam {
  uint32_t sm_addr, bars;
  int rank, nct;  // CTA of the cluster, CTAs in it
  int lane, warp;
  unsigned *fail;
  uint32_t polls;  // bound of a wait; 0 once one has run out
  bool lost;       // one has
  template <typename T>
  __device__ __forceinline__ int rows_of(const LevelDesc<T> &A) const {
    return max(0, min(A.rw, A.n - rank * A.rw));
  }
  // the value of row `row`, component c in v, to the replicated vector at byte
  // offset o of every CTA (phase ph); the row's lanes share the CTAs
  template <typename T>
  __device__ __forceinline__ void spread(int ph, uint32_t o, int row, int li, int LN, T v, bool ok) const {
    const T other = __shfl_xor_sync(0xffffffffu, v, 1);
    const C2<T> w = (li & 1) ? C2<T>{other, v} : C2<T>{v, other};
    if (!ok) return;
    const uint32_t at = sm_addr + o + row * (uint32_t)sizeof(C2<T>), bar = bars + 8u * ph;
    for (int q = li; q < nct; q += LN) st_async(at, bar, q, w);
  }
  // polls until phase ph's vector is here or the bound is reached
  __device__ __forceinline__ bool arrived(int ph, uint32_t &bound) const {
    const uint32_t a = bars + 8u * ph;
    for (; bound > 0; bound--) {
      uint32_t done;
      asm volatile(
          "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n"
          " selp.u32 %0, 1, 0, p;\n}\n"
          : "=r"(done)
          : "r"(a)
          : "memory");
      if (done) return true;
    }
    return false;
  }
  // the whole vector of phase ph has arrived here
  __device__ __forceinline__ void wait(int ph) {
    uint32_t bound = polls;
    if (arrived(ph, bound) || lost) return;
    *(volatile unsigned *)fail = 1u;
    lost = true;
    polls = 0;
  }
  // all that is under way to this CTA has landed: the vectors of the n phases
  // but `unused` (at most the default bound, over all of them)
  __device__ __forceinline__ void drain(int n, int unused) const {
    uint32_t bound = kStageWaitPolls;
    for (int ph = 0; ph < n && bound > 0; ph++)
      if (ph != unused) arrived(ph, bound);
  }
};

// This thread's part of a level: one component of part p of one own row (a
// level has at most kTailRows rows a CTA, so one pass covers them).  The first
// kLaneNz nonzeros and the row's diagonal blocks are held in registers for the
// phases of one visit to the level: a phase is a chain of dependent
// instructions on a few warps, and loading them anew in each took half of it.
// Warps without a row do nothing; the spare lanes of a warp with one repeat
// its last row without storing, so that every lane takes part in the shuffles.
constexpr int kTailRows = kTailThreads / 2;
constexpr int kLaneNz = 8;
template <typename T>
struct TailLane {
  bool act, ok;  // the warp has a row; this lane's is its own
  int i, row, li, LN, c, P;
  uint32_t xo[kLaneNz];  // byte offsets into a replicated vector
  T vr[kLaneNz], vi[kLaneNz];  // the value; its imaginary part with the component's sign
  int k, e;              // nonzeros past the registers (staged, step P)
  int used;              // register slots that any lane of the warp fills
  T dd, df, id, jf;      // diagonal block and inverse: own component, coupling
  __device__ __forceinline__ void place(const TailTeam &R, const LevelDesc<T> &A) {
    const int m = R.rows_of(A);
    LN = 1 << A.lnb;
    P = LN >> 1;
    li = R.lane & (LN - 1);
    c = li & 1;
    const int i0 = R.warp << (5 - A.lnb);
    act = i0 < m;
    const int at = i0 + (R.lane >> A.lnb);
    ok = at < m;
    i = ok ? at : m - 1;
    row = R.rank * A.rw + i;
  }
  __device__ __forceinline__ void load(const LevelDesc<T> &A) {
    if (!act) return;
    const unsigned sg = c ? 0u : 0x80000000u;
    e = tail_at<int32_t>(A.s_rp, i + 1);
    k = tail_at<int32_t>(A.s_rp, i) + (li >> 1);
    used = __reduce_max_sync(0xffffffffu, (e - k + P - 1) >> (A.lnb - 1));
#pragma unroll
    for (int u = 0; u < kLaneNz; u++) {
      xo[u] = (uint32_t)row * (uint32_t)sizeof(C2<T>);  // (times zero: the row's own value)
      vr[u] = vi[u] = 0;
      if (k < e) {
        xo[u] = (uint32_t)tail_at<int32_t>(A.s_ci, k) * (uint32_t)sizeof(C2<T>);
        const C2<T> v = tail_at<C2<T>>(A.s_off, k);
        vr[u] = v.x;
        vi[u] = flip(v.y, sg);
        k += P;
      }
    }
    dd = tail_at<T>(A.s_dia, 3 * i + c);
    df = tail_at<T>(A.s_dia, 3 * i + 2);
    id = tail_at<T>(A.s_dia, 3 * A.rw + 3 * i + c);
    jf = tail_at<T>(A.s_dia, 3 * A.rw + 3 * i + 2);
  }
  __device__ __forceinline__ T parts_sum(T v) const {
    for (int o = 2; o < LN; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  }
  // component c of the off-diagonal row sum over the vector at offset x
  __device__ __forceinline__ T row_sum(const LevelDesc<T> &A, uint32_t x) const {
    // FP64: pairs of slots that no lane fills are branched over (their FMAs
    // would take the pipe all the same; a level of 100 rows fills one or two of
    // the eight): Newton on the 65^2 square 5.28 -> 5.09 ms
    constexpr int kStep = sizeof(T) == 8 ? 2 : kLaneNz;
    C2<T> xv[kLaneNz];
#pragma unroll
    for (int u = 0; u < kLaneNz; u++) xv[u] = tail_at<C2<T>>(x + xo[u]);
    T s0 = 0, s1 = 0;
#pragma unroll
    for (int g = 0; g < kLaneNz; g += kStep)
      if (g == 0 || g < used) {
#pragma unroll
        for (int u = g; u < g + kStep; u++) {
          s0 = fma(vr[u], c ? xv[u].y : xv[u].x, s0);
          s1 = fma(vi[u], c ? xv[u].x : xv[u].y, s1);
        }
      }
    const unsigned sg = c ? 0u : 0x80000000u;
    for (int q = k; q < e; q += P) {
      const C2<T> v = tail_at<C2<T>>(A.s_off, q), y = tail_at<C2<T>>(x, tail_at<int32_t>(A.s_ci, q));
      s0 = fma(v.x, c ? y.y : y.x, s0);
      s1 = fma(flip(v.y, sg), c ? y.x : y.y, s1);
    }
    return parts_sum(s0 + s1);
  }
  // component c of the own node's sum over its members (lists at A.s_mp,
  // A.s_mi) of the finer vector `at(j)` gives
  template <class F>
  __device__ __forceinline__ T members(const LevelDesc<T> &A, F &&at) const {
    T acc = 0;
    const int last = tail_at<int32_t>(A.s_mp, i + 1);
    constexpr int U = 8;  // loads under way at once
    for (int k0 = tail_at<int32_t>(A.s_mp, i) + (li >> 1); k0 < last; k0 += U * P) {
      T v[U];
#pragma unroll
      for (int u = 0; u < U; u++) v[u] = at(tail_at<int32_t>(A.s_mi, min(k0 + u * P, last - 1)));
#pragma unroll
      for (int u = 0; u < U; u++)
        if (k0 + u * P < last) acc += v[u];
    }
    return parts_sum(acc);
  }
};

// own rows of a level's operator (and its lists) into shared memory; the
// members of its nodes over the finer level (mp, mi: null for the first)
template <typename T>
__device__ __forceinline__ void tail_stage(const TailTeam &R, const LevelDesc<T> &A, bool matrix,
                                           const int32_t *mp, const int32_t *mi, int t, int st) {
  const int r0 = R.rank * A.rw, m = R.rows_of(A);
  if (matrix)
    for (int q = t; q < A.n; q += st) tail_at<int32_t>(A.s_agg, q) = A.agg[q];
  if (m == 0) return;
  const int mb = mp ? mp[r0] : 0, me = mp ? mp[r0 + m] : 0;
  const int b = matrix ? A.rp[r0] : 0, e = matrix ? A.rp[r0 + m] : 0;
  if (mp)
    for (int q = t; q <= m; q += st) tail_at<int32_t>(A.s_mp, q) = mp[r0 + q] - mb;
  for (int q = t; q < me - mb; q += st) tail_at<int32_t>(A.s_mi, q) = mi[mb + q];
  if (!matrix) return;
  for (int q = t; q <= m; q += st) tail_at<int32_t>(A.s_rp, q) = A.rp[r0 + q] - b;
  for (int q = t; q < e - b; q += st) {
    tail_at<int32_t>(A.s_ci, q) = A.ci[b + q];
    tail_at<C2<T>>(A.s_off, q) = A.off[b + q];
  }
  for (int q = t; q < 3 * m; q += st) {
    tail_at<T>(A.s_dia, q) = A.dia[3 * (int64_t)r0 + q];
    tail_at<T>(A.s_dia, 3 * A.rw + q) = A.dinv[3 * (int64_t)r0 + q];
  }
}

// Chebyshev step k of the lane's row: the iterate at offset x -> its new
// value (component c), d the direction, b the right-hand side
template <typename T>
__device__ __forceinline__ T tail_cheb(const TailLane<T> &Q, const LevelDesc<T> &A, const T *coef, int k, uint32_t x,
                                       T b, T &d) {
  const C2<T> xi = tail_at<C2<T>>(x, Q.row);
  const T xc = Q.c ? xi.y : xi.x, xo = Q.c ? xi.x : xi.y;
  const T rc = (b - (Q.dd * xc + Q.df * xo)) - Q.row_sum(A, x);
  const T ro = __shfl_xor_sync(0xffffffffu, rc, 1);
  const T z = Q.id * rc + Q.jf * ro;
  d = k == 0 ? coef[0] * z : coef[2 * k] * d + coef[2 * k + 1] * z;
  return xc + d;
}

template <typename T>
__global__ void __launch_bounds__(kTailThreads)
    resident_vcycle(const LevelDesc<T> *__restrict__ lv_g, int lt, int L, int deg, const T *__restrict__ Ainv,
                    DenseMap D, TailDense td, uint32_t s_bar, TailArgs<T> a, const int *halt) {
  __shared__ LevelDesc<T> lv[16];
  __shared__ T s_coef[16][2 * kMaxDegree];
  __shared__ double s_dot[16];
  __shared__ double s32[32];
  TailTeam R;
  R.sm_addr = smem_addr(tail_sm);
  R.bars = R.sm_addr + s_bar;
  R.fail = a.fail;
  {
    const unsigned o = __ldcg(a.counter + kStageWaitSlot);
    R.polls = o ? o - 1 : kStageWaitPolls;
    R.lost = false;
  }
  {
    unsigned r, n;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
    R.rank = (int)r;
    R.nct = (int)n;
  }
  R.lane = threadIdx.x & 31;
  R.warp = threadIdx.x >> 5;
  {
    const int nw = (int)(sizeof(LevelDesc<T>) / 4) * (L - lt);
    const uint32_t *src = reinterpret_cast<const uint32_t *>(lv_g + lt);
    for (int q = threadIdx.x; q < nw; q += blockDim.x) reinterpret_cast<uint32_t *>(lv + lt)[q] = src[q];
  }
  __syncthreads();
  const int per = 2 * deg + 1, nph = tail_phases(L - lt, deg);
  // every phase's mbarrier expects its whole vector
  for (int q = threadIdx.x; q < nph; q += blockDim.x) {
    uint64_t *bar = &tail_at<uint64_t>(s_bar, q);
    const int l = q < nph - 2 ? lt + q / per : L - 1;
    mbar_init(bar);
    mbar_expect_tx(bar, (uint32_t)(lv[l].n * (int)sizeof(C2<T>)));
  }
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  cluster_arrive();  // (waited for below) every CTA's mbarriers are ready before any store to it
  // the operators and lists were written before the launch this one follows:
  // staged while that one runs
  for (int l = lt; l < L; l++) {
    const int32_t *mp = l > lt ? lv[l - 1].mem_ptr : a.f_mp, *mi = l > lt ? lv[l - 1].mem_idx : a.f_mi;
    // (the first level by three quarters of the warps, the others by the rest)
    constexpr int kFirst = kTailThreads / 4 * 3;
    const int t = (int)threadIdx.x - (l > lt ? kFirst : 0);
    if (t >= 0 && (l > lt || t < kFirst))
      tail_stage<T>(R, lv[l], l < L - 1, mp, mi, t, l > lt ? kTailThreads - kFirst : kFirst);
  }
  for (int q = threadIdx.x; q < (L - 1 - lt) * 2 * deg; q += blockDim.x) {
    const int l = lt + q / (2 * deg);
    s_coef[l][q % (2 * deg)] = lv[l].coef[q % (2 * deg)];
  }
  if (td.staged) {
    const LevelDesc<T> &C = lv[L - 1];
    const int i0 = 2 * R.rank * C.rw, m2 = 2 * R.rows_of(C);
    if (m2 > 0) {
      const int64_t o0 = D.rowoff[i0], o1 = D.rowoff[i0 + m2 - 1] + D.bdim[i0 + m2 - 1];
      for (int q = threadIdx.x; q < m2; q += blockDim.x) {
        tail_at<int32_t>(td.s_map, 3 * q) = (int32_t)(D.rowoff[i0 + q] - o0);
        tail_at<int32_t>(td.s_map, 3 * q + 1) = D.bstart[i0 + q];
        tail_at<int32_t>(td.s_map, 3 * q + 2) = D.bdim[i0 + q];
      }
      for (int q = threadIdx.x; q < (int)(o1 - o0); q += blockDim.x) tail_at<T>(td.s_a, q) = Ainv[o0 + q];
    }
  }
  cluster_wait();
  dep_sync();
  __syncthreads();
  const int done = halt ? *halt : 0;  // (looked at below, with the first loads under way)
  TailLane<T> Q{};
  // The start of level l from its right-hand side's component bc: the first
  // Chebyshev step (x = c0 D^-1 b) is spread; b and d stay with the row.
  auto start_level = [&](int l, T bc) {
    const LevelDesc<T> &A = lv[l];
    if (l == L - 1) {
      R.spread<T>(nph - 2, td.s_bd, Q.row, Q.li, Q.LN, bc, Q.ok);
      return;
    }
    const T bo = __shfl_xor_sync(0xffffffffu, bc, 1);
    const T x = s_coef[l][0] * (tail_at<T>(A.s_dia, 3 * A.rw + 3 * Q.i + Q.c) * bc +
                                tail_at<T>(A.s_dia, 3 * A.rw + 3 * Q.i + 2) * bo);
    if (Q.ok && Q.li < 2) {
      tail_at<T>(A.b, 2 * Q.i + Q.c) = bc;
      tail_at<T>(A.d, 2 * Q.i + Q.c) = x;
    }
    R.spread<T>((l - lt) * per, deg % 2 == 1 ? A.xb : A.xa, Q.row, Q.li, Q.LN, x, Q.ok);
    __syncwarp();
  };
  {
    const LevelDesc<T> &A = lv[lt];
    Q.place(R, A);
    T bc = 0;
    if (Q.act) {
      if (a.head == kHeadRestrict) {
        const T *res = reinterpret_cast<const T *>(a.f_res);
        bc = Q.members(A, [&](int j) { return res[2 * (int64_t)j + Q.c]; });
      } else {
        const int64_t e = 2 * (int64_t)Q.row + Q.c;
        bc = reinterpret_cast<const T *>(a.b)[e];
        if (a.head == kHeadLanczos) {
          const T *la = lanczos_coef<T>(a.ms);
          T *ro = reinterpret_cast<T *>(a.r_old);
          bc = la[0] * bc - la[1] * ro[e] - la[2] * reinterpret_cast<const T *>(a.r_cur)[e];
          __syncwarp();  // every part has read r_old
          if (Q.ok && Q.li < 2 && done < 2) ro[e] = bc;
        }
      }
    }
    // the recurrence has ended: every CTA leaves alike, before any store to
    // another
    if (done >= 2) return;
    if (Q.act) start_level(lt, bc);
  }
  for (int l = lt; l < L - 1; l++) {
    const LevelDesc<T> &A = lv[l];
    int ph = (l - lt) * per;
    uint32_t cur = deg % 2 == 1 ? A.xb : A.xa, oth = deg % 2 == 1 ? A.xa : A.xb;
    T b = 0, d = 0;
    Q.load(A);
    if (Q.act) {
      b = tail_at<T>(A.b, 2 * Q.i + Q.c);
      d = tail_at<T>(A.d, 2 * Q.i + Q.c);
    }
    for (int k = 1; k < deg; k++, ph++) {
      R.wait(ph);
      if (Q.act) {
        const T x = tail_cheb<T>(Q, A, s_coef[l], k, cur, b, d);
        R.spread<T>(ph + 1, oth, Q.row, Q.li, Q.LN, x, Q.ok);
      }
      const uint32_t t = cur;
      cur = oth;
      oth = t;
    }
    // the residual over xa (the pre-smoothed iterate is xb)
    R.wait(ph++);
    if (Q.act) {
      const C2<T> xi = tail_at<C2<T>>(A.xb, Q.row);
      const T t = b - (Q.dd * (Q.c ? xi.y : xi.x) + Q.df * (Q.c ? xi.x : xi.y));
      R.spread<T>(ph, A.xa, Q.row, Q.li, Q.LN, t - Q.row_sum(A, A.xb), Q.ok);
    }
    const LevelDesc<T> &C = lv[l + 1];
    Q.place(R, C);
    R.wait(ph);
    if (Q.act) start_level(l + 1, Q.members(C, [&](int j) {
      const C2<T> v = tail_at<C2<T>>(A.xa, j);
      return Q.c ? v.y : v.x;
    }));
  }
  // the coarsest level: its dense inverse, real rows split over 16 lanes
  {
    const LevelDesc<T> &C = lv[L - 1];
    const int m2 = 2 * R.rows_of(C), li = R.lane & 15;
    R.wait(nph - 2);
    for (int base = 2 * R.warp; base < m2; base += 2 * (kTailThreads / 32)) {
      const int i = base + (R.lane >> 4);  // a warp holds both components of a node
      const int row = 2 * R.rank * C.rw + i;
      T s = 0;
      if (td.staged) {
        const int o = tail_at<int32_t>(td.s_map, 3 * i), bs = tail_at<int32_t>(td.s_map, 3 * i + 1),
                  m = tail_at<int32_t>(td.s_map, 3 * i + 2);
#pragma unroll 4
        for (int j = li; j < m; j += 16) s = fma(tail_at<T>(td.s_a, o + j), tail_at<T>(td.s_bd, bs + j), s);
      } else {
        const T *av = Ainv + D.rowoff[row];
        const int bs = D.bstart[row], m = D.bdim[row];
#pragma unroll 4
        for (int j = li; j < m; j += 16) s = fma(av[j], tail_at<T>(td.s_bd, bs + j), s);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const T other = __shfl_xor_sync(0xffffffffu, s, 16);
      const C2<T> w = R.lane < 16 ? C2<T>{s, other} : C2<T>{other, s};
      if (R.lane < R.nct)
        st_async(R.sm_addr + td.s_xd + (uint32_t)(row >> 1) * (uint32_t)sizeof(C2<T>), R.bars + 8u * (nph - 1),
                 R.lane, w);
    }
    R.wait(nph - 1);
  }
  uint32_t xc = td.s_xd;
  double part = 0.0;
  // the first of this thread's fine elements that the result is added to,
  // loaded ahead
  const int64_t j0 = (int64_t)R.rank * blockDim.x + threadIdx.x;
  int32_t ag0 = 0;
  C2<T> fx0{0, 0};
  if (a.out == kOutProlong && j0 < a.f_n) {
    ag0 = a.f_agg[j0];
    fx0 = a.f_x[j0];
  }
  for (int l = L - 2; l >= lt; l--) {
    const LevelDesc<T> &A = lv[l];
    int ph = (l - lt) * per + deg + 1;  // the first post-smoothing step's
    T b = 0, d = 0;
    Q.place(R, A);
    Q.load(A);
    if (Q.act) b = tail_at<T>(A.b, 2 * Q.i + Q.c);
    // coarse correction on the CTA's own copy of the whole vector (a CTA
    // without rows here sends none, so others may already be overwriting its
    // copy: it reads the result only)
    if (R.rows_of(A) > 0)
      for (int j = threadIdx.x; j < A.n; j += blockDim.x) {
        const C2<T> e = tail_at<C2<T>>(xc, tail_at<int32_t>(A.s_agg, j));
        C2<T> &x = tail_at<C2<T>>(A.xb, j);
        x = C2<T>{x.x + e.x, x.y + e.y};
      }
    __syncthreads();
    uint32_t in = A.xb, out = A.xa;
    for (int k = 0; k < deg; k++, ph++) {
      const bool fin = l == lt && k == deg - 1 && a.out != kOutProlong;
      if (Q.act) {
        const T x = tail_cheb<T>(Q, A, s_coef[l], k, in, b, d);
        if (!fin) {
          R.spread<T>(ph, out, Q.row, Q.li, Q.LN, x, Q.ok);
        } else if (Q.ok && Q.li < 2) {
          reinterpret_cast<T *>(a.z)[2 * (int64_t)Q.row + Q.c] = x;
          part = (double)b * (double)x;
        }
      }
      if (!fin) R.wait(ph);
      const uint32_t t = in;
      in = out;
      out = t;
    }
    xc = in;
  }
  // (no CTA leaves while others may still send to it)
  if (a.out == kOutProlong) {
    cluster_arrive();
    for (int64_t j = j0; j < a.f_n; j += (int64_t)R.nct * blockDim.x) {
      const C2<T> e = tail_at<C2<T>>(xc, j == j0 ? ag0 : a.f_agg[j]);
      const C2<T> v = j == j0 ? fx0 : a.f_x[j];
      a.f_x[j] = C2<T>{v.x + e.x, v.y + e.y};
    }
    cluster_wait();
  } else if (a.out == kOutMinres) {
    // <r, z>: the CTAs' sums in CTA order, then the Givens step
    const double s = block_sum(part, s32);
    if (threadIdx.x == 0)
      asm volatile("st.shared::cluster.f64 [%0], %1;\n" ::"r"(map_rank(smem_addr(&s_dot[R.rank]), 0)), "d"(s)
                   : "memory");
    cluster_arrive();
    cluster_wait();
    if (R.rank == 0 && threadIdx.x < 32) {
      dep_trigger();
      double t = 0.0;
      for (int q = 0; q < R.nct; q++) t += s_dot[q];
      minres_advance(a.ms, reinterpret_cast<const double *>(a.ms), t);
    }
  } else {
    cluster_arrive();
    cluster_wait();
  }
  // (the first level's last step goes to memory unless it is prolonged)
  if (R.lost) R.drain(nph, a.out == kOutProlong ? -1 : per - 1);
}

// plain MINRES pieces for the single-level case
template <typename T>
__global__ void lanczos_only(int64_t n, const MinresScalars *__restrict__ s, const C2<T> *__restrict__ u,
                             C2<T> *__restrict__ r_old, const C2<T> *__restrict__ r_cur) {
  dep_sync();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const T *la = lanczos_coef<T>(s);
  const T a = la[0], bb = la[1], c = la[2];
  const C2<T> ui = u[i], ro = r_old[i], rc = r_cur[i];
  r_old[i] = C2<T>{a * ui.x - bb * ro.x - c * rc.x, a * ui.y - bb * ro.y - c * rc.y};
}

template <typename T>
__global__ void dot_advance(int64_t n, const C2<T> *__restrict__ a, const C2<T> *__restrict__ b,
                            double *partials, unsigned *counter, MinresScalars *s) {
  dep_sync();
  double v = 0.0;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) v = (double)a[i].x * b[i].x + (double)a[i].y * b[i].y;
  double total = 0.0;
  if (grid_reduce(v, partials, counter, &s->rz, &total))
    minres_advance(s, reinterpret_cast<const double *>(s), total);
}

// the longest 4-aligned range of nonzeros of a block of kRows rows
int longest_block(const std::vector<int32_t> &rp, int64_t n) {
  int32_t mx = 0;
  for (int64_t r0 = 0; r0 < n; r0 += kRows) mx = std::max(mx, rp[std::min<int64_t>(n, r0 + kRows)] - (rp[r0] & ~3));
  return mx;
}

}  // namespace

// ------------------------------------------------------------ structures
struct AmgLevel {
  int64_t n = 0, nnz = 0;
  const int32_t *rp = nullptr, *ci = nullptr;  // level 0: the mesh graph
  DevBuf<int32_t> rp_own, ci_own;
  int block_nnz = 0;  // longest_block
  bool warp32 = false, warp64 = false;  // SpMV schedule (tuned on the first refresh)
  bool tuned32 = false, tuned64 = false;
  // transfer to the next level
  DevBuf<int32_t> agg, mem_ptr, mem_idx, seg_ptr, seg_idx, intra_ptr, intra_idx;
  // host copies for the resident cycle's layout (levels and transfers small
  // enough for it)
  std::vector<int32_t> h_rp, h_mem_ptr;
};

// One layout of the resident V-cycle: its first level, the level descriptors
// and the shared memory of a CTA.
template <typename T>
struct TailPlan {
  int lt = -1;  // -1: none
  size_t smem = 0;
  TailDense dense{};
  uint32_t s_bar = 0;
  DevBuf<LevelDesc<T>> desc;
};

template <typename T>
struct AmgVals {
  bool ready = false;
  int64_t refreshes = 0;  // numeric refreshes so far
  int64_t built = -1;     // the rebuild (NlsImpl::reg_builds) the last one followed
  std::vector<DevBuf<C2<T>>> off;  // level >= 1
  std::vector<DevBuf<T>> dia;      // level >= 1
  std::vector<DevBuf<T>> dinv, coef;
  std::vector<DevBuf<C2<T>>> b, x, x2, d, res;
  // the resident V-cycle's layouts: [0] in use, [1] the one that keeps the
  // fine level on the grid (kernel timing of a mesh that [0] takes whole)
  TailPlan<T> plan[2];
  // row sums of |K_ij| on the fine level for its Gershgorin bound, computed
  // once: |K_ij| = |alpha_ij| does not depend on mu (the phase factor has
  // modulus one), so only the diagonal blocks change between refreshes
  DevBuf<T> rowabs0;
  bool rowabs_ready = false;
};

struct Amg::Impl {
  NlsImpl &nls;
  AmgOptions opt;
  std::vector<AmgLevel> lev;
  int lt = 1;  // first level handled by the coarse-level tail
  AmgVals<float> vf;
  AmgVals<double> vd;
  // per level, zero between refreshes: the Gershgorin bound's bits, arrivals
  DevBuf<unsigned long long> lmax_bits;
  DevBuf<unsigned> arrive;
  ChebSpec cheb;
  // The coarsest level's inverse, FP64 (2n)^2 and FP32: of the operators of the
  // precision inverse_of (in bytes) that was refreshed in full last.  A solve
  // takes it as it is (any SPD inverse preconditions), an apply of the V-cycle
  // by itself has its own formed first (ensure).
  DevBuf<double> dense;
  size_t inverse_of = 0;
  DevBuf<double> dense2;  // the inversion's other buffer
  DevBuf<float> densef;
  // packed block-diagonal coarsest inverse: per block (offset, dim), per real
  // row (offset, block start, dim)
  DevBuf<int64_t> blk_off, row_off;
  DevBuf<int32_t> blk_dim, row_start, row_dim;
  int nblk = 0, max_dim = 0;
  DenseMap dmap() const { return DenseMap{row_off.p, row_start.p, row_dim.p}; }
  DevBuf<int> err;
  Impl(NlsImpl &s, const AmgOptions &o) : nls(s), opt(o) {}
  template <typename T> AmgVals<T> &vals();
  template <typename T> void ensure_vals();
  template <typename T> void invert_coarsest();
  template <typename T> const C2<T> *off(int l);
  template <typename T> const T *dia(int l);
  template <typename T> const T *dense_inv();
  template <typename T, class Op> void rows(int l, const C2<T> *x, const Op &op);
  template <typename T>
  void descend_ascend(int l, const C2<T> *b, C2<T> *x, MinresScalars *ms, double *rowdot = nullptr);
  // the MINRES state's `done` while a MINRES V-cycle is being issued: its
  // launches return at once once the solve has converged
  const int *halt = nullptr;
  template <typename T> void prime();
  void choose_cluster();
  int tail_ctas = 1;        // CTAs of the resident cycle's cluster
  bool grid_coarse = false;  // coarsest level too large for it: dense kernel on the grid
  template <typename T> size_t tail_layout(int first, std::vector<LevelDesc<T>> *desc, TailPlan<T> *P);
  template <typename T> void build_plan(TailPlan<T> &P, int first);
  template <typename T> const TailPlan<T> &plan() {
    AmgVals<T> &V = vals<T>();
    return V.plan[V.plan[1].lt >= 0 && (nls.timers[0].on || nls.timers[1].on) ? 1 : 0];
  }
  template <typename T> void launch_tail(const TailPlan<T> &P, TailArgs<T> a, bool overlap);
  // V-cycle launches overlap their predecessors (launch_dep) unless the
  // handle turned that off or times kernels with events between launches
  bool ovl() const { return nls.overlap_launches && !nls.timers[0].on && !nls.timers[1].on; }
};

template <> AmgVals<float> &Amg::Impl::vals<float>() { return vf; }
template <> AmgVals<double> &Amg::Impl::vals<double>() { return vd; }
template <> const C2<float> *Amg::Impl::off<float>(int l) {
  return l == 0 ? nls.d_keo32.p : vf.off[l].p;
}
template <> const C2<double> *Amg::Impl::off<double>(int l) {
  return l == 0 ? nls.d_keo64.p : vd.off[l].p;
}
template <> const float *Amg::Impl::dia<float>(int l) { return l == 0 ? nls.d_rd32.p : vf.dia[l].p; }
template <> const double *Amg::Impl::dia<double>(int l) { return l == 0 ? nls.d_rd64.p : vd.dia[l].p; }
template <> const float *Amg::Impl::dense_inv<float>() { return densef.p; }
template <> const double *Amg::Impl::dense_inv<double>() { return dense.p; }

Amg::Amg(NlsImpl &s, const AmgOptions &o) : impl(new Impl(s, o)) {
  Impl &I = *impl;
  cudaStream_t st = s.stream;
  MeshImpl &m = *s.mesh;
  // host copy of the current fine operator (strength tests)
  std::vector<HostLevel> H(1);
  H[0].n = m.N;
  H[0].rp = m.rp();
  H[0].ci = m.ci();
  {
    std::vector<C2<double>> off(2 * m.E);
    s.d_keo64.download(off.data(), 2 * m.E, st);
    H[0].dia.resize(3 * m.N);
    s.d_rd64.download(H[0].dia.data(), 3 * m.N, st);
    s.sync();
    H[0].off.resize(2 * m.E);
    for (int64_t k = 0; k < 2 * m.E; k++) H[0].off[k] = {off[k].x, off[k].y};
  }
  if (s.sys_off.empty())
    H[0].soff = {0, (int64_t)m.N};
  else
    H[0].soff = s.sys_off;
  // coarsen until every system's coarsest block is small (one system: the
  // whole level)
  while ((int)H.size() < o.max_levels && max_block(H.back()) > o.coarse_size) {
    HostLevel C;
    coarsen(H.back(), C, o.strength_threshold);
    if (C.n >= H.back().n) {  // no coarsening progress: stop here
      H.back().agg.clear();
      break;
    }
    H.push_back(std::move(C));
  }
  NOSH_CHECK(max_block(H.back()) <= 512, NOSH_ERR_INVALID,
             "AMG coarsening stalled at " + std::to_string(max_block(H.back())) + " nodes per system");
  const int L = (int)H.size();
  I.lev.resize(L);
  for (int l = 0; l < L; l++) {
    AmgLevel &A = I.lev[l];
    HostLevel &h = H[l];
    A.n = h.n;
    A.nnz = h.rp[h.n];
    if (l == 0) {
      A.rp = m.d_rp.p;
      A.ci = m.d_ci.p;
    } else {
      A.rp_own.upload(h.rp, st);
      A.ci_own.alloc(h.ci.size() + kPad);
      A.ci_own.zero(st);
      if (!h.ci.empty())
        NOSH_CUDA(cudaMemcpyAsync(A.ci_own.p, h.ci.data(), h.ci.size() * 4, cudaMemcpyHostToDevice, st));
      A.rp = A.rp_own.p;
      A.ci = A.ci_own.p;
    }
    A.block_nnz = longest_block(h.rp, h.n);
    if (l + 1 < L) {
      A.agg.upload(h.agg, st);
      A.mem_ptr.upload(h.mem_ptr, st);
      A.mem_idx.upload(h.mem_idx, st);
      A.seg_ptr.upload(h.seg_ptr, st);
      A.seg_idx.upload(h.seg_idx, st);
      A.intra_ptr.upload(h.intra_ptr, st);
      A.intra_idx.upload(h.intra_idx, st);
    }
  }
  for (int l = 0; l < L; l++) {
    if (H[l].n <= std::max(kTailMax, kResidentMax)) I.lev[l].h_rp = H[l].rp;
    if (l + 1 < L && H[l + 1].n <= std::max(kTailMax, kResidentMax)) I.lev[l].h_mem_ptr = H[l].mem_ptr;
  }
  // The resident cycle starts on the first level small enough for it whose
  // vectors, with those of the levels below, fit a CTA's shared memory in
  // FP64; the levels above it run on the whole grid.
  I.choose_cluster();
  I.lt = L - 1;
  I.grid_coarse = L < 2;
  for (int l = 0; l < L; l++) {
    if (I.lev[l].n > (l == 0 ? kResidentMax : kTailMax)) {
      if (l == L - 1) I.grid_coarse = true;
      continue;
    }
    if (I.tail_layout<double>(l, nullptr, nullptr) <= (size_t)kTailSmem) {
      I.lt = l;
      break;
    }
    if (l == L - 1) I.grid_coarse = true;
  }
  I.lmax_bits.alloc(L);
  I.lmax_bits.zero(st);
  I.arrive.alloc(L);
  I.arrive.zero(st);
  I.cheb = ChebSpec::of(std::max(o.smooth_degree, 1), o.cheb_ratio);
  {
    // the coarsest level's dense inverse: one packed block per system
    const HostLevel &Hc = H.back();
    const int64_t ns = (int64_t)Hc.soff.size() - 1;
    std::vector<int64_t> boff, roff;
    std::vector<int32_t> bdim, rstart, rdim;
    int64_t total = 0;
    for (int64_t sy = 0; sy < ns; sy++) {
      const int64_t n0 = Hc.soff[sy], nb = Hc.soff[sy + 1] - n0;
      if (nb == 0) continue;
      const int32_t m = (int32_t)(2 * nb);
      boff.push_back(total);
      bdim.push_back(m);
      for (int32_t r = 0; r < m; r++) {
        roff.push_back(total + (int64_t)r * m);
        rstart.push_back((int32_t)(2 * n0));
        rdim.push_back(m);
      }
      total += (int64_t)m * m;
      I.max_dim = std::max<int>(I.max_dim, m);
    }
    I.nblk = (int)boff.size();
    I.blk_off.upload(boff, st);
    I.blk_dim.upload(bdim, st);
    I.row_off.upload(roff, st);
    I.row_start.upload(rstart, st);
    I.row_dim.upload(rdim, st);
    I.dense.alloc(total);
    I.densef.alloc(total);
    I.dense2.alloc(total);
  }
  I.err.alloc(1);
  I.err.zero(st);
  NOSH_CUDA(cudaFuncSetAttribute(gauss_jordan_fp32, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kDenseFp32 * kDenseFp32 * (int)sizeof(float)));
  s.sync();
}

Amg::~Amg() = default;

int Amg::num_levels() const { return (int)impl->lev.size(); }
int64_t Amg::level_size(int l) const { return impl->lev[l].n; }
int Amg::tail_level() const { return impl->lt; }

const int *Amg::error_flag_ptr() const { return impl->err.p; }

void Amg::clear_error() {
  // the coarse operators that failed the pivot check are replaced by the
  // next refresh, which is made a full Galerkin one
  NOSH_CUDA(cudaMemsetAsync(impl->err.p, 0, sizeof(int), impl->nls.stream));
  impl->vf.refreshes = 0;
  impl->vd.refreshes = 0;
}

int Amg::error_flag() {
  int herr = 0;
  impl->err.download(&herr, 1, impl->nls.stream);
  impl->nls.sync();
  return herr;
}

template <typename T>
void Amg::Impl::ensure_vals() {
  AmgVals<T> &V = vals<T>();
  if (V.ready) return;
  const int L = (int)lev.size();
  V.off.resize(L);
  V.dia.resize(L);
  V.dinv.resize(L);
  V.coef.resize(L);
  V.b.resize(L);
  V.x.resize(L);
  V.x2.resize(L);
  V.d.resize(L);
  V.res.resize(L);
  for (int l = 0; l < L; l++) {
    const int64_t n = lev[l].n;
    if (l > 0) {
      V.off[l].alloc(lev[l].nnz + kPad);
      V.off[l].zero(nls.stream);
      V.dia[l].alloc(3 * n);
    }
    V.dinv[l].alloc(3 * n);
    V.coef[l].alloc(2 * std::max(opt.smooth_degree, 1) + 2);
    // (levels inside the resident cycle keep their vectors in shared memory)
    if (l > 0 && l >= lt && !grid_coarse) continue;
    V.b[l].alloc(n);
    V.x[l].alloc(n);
    V.x2[l].alloc(n);
    V.d[l].alloc(n);
    V.res[l].alloc(n);
  }
  if (!grid_coarse) {
    build_plan<T>(V.plan[0], lt);
    if (lt == 0) build_plan<T>(V.plan[1], 1);
  }
  nls.sync();
  prime<T>();
  V.ready = true;
}

// Numeric refresh from the current regularised KEO; stream-ordered, no host
// synchronisation (the pivot check is read later through error_flag()).
template <typename T>
void Amg::refresh() {
  Impl &I = *impl;
  if (sizeof(T) == 4) I.nls.ensure_keo32();
  I.ensure_vals<T>();
  AmgVals<T> &V = I.vals<T>();
  cudaStream_t st = I.nls.stream;
  const int L = (int)I.lev.size();
  // (counted where it is done: after a failure on the way the hierarchy, the
  // coarsest inverse above all, may be half formed, and the next is full again)
  const bool partial = I.opt.reuse_period > 1 && L > 1 && V.refreshes % I.opt.reuse_period != 0;
  const int64_t done = std::exchange(V.refreshes, 0) + 1;
  V.built = -1;
  if (!V.rowabs_ready) {
    V.rowabs0.alloc(I.lev[0].n);
    row_abs_sums<T><<<div_up(I.lev[0].n, 256), 256, 0, st>>>(I.lev[0].n, I.lev[0].rp, I.off<T>(0), V.rowabs0.p);
    ++I.nls.launch_count;
    V.rowabs_ready = true;
  }
  if (partial) {
    // hierarchy reuse (MueLu "reuse: type full", src/keo_regularized.cpp:
    // 298-330): the fine level reads the current operator directly; only its
    // block-Jacobi inverse and Chebyshev bounds follow it, the coarse
    // operators keep their last Galerkin values (SPD, so the V-cycle stays
    // an SPD preconditioner)
    dinv_gershgorin<T><<<div_up(I.lev[0].n, 256), 256, 0, st>>>(I.lev[0].n, I.lev[0].rp, I.off<T>(0), I.dia<T>(0),
                                                                V.dinv[0].p, I.lmax_bits.p, I.arrive.p, I.err.p,
                                                                V.rowabs0.p, I.cheb, V.coef[0].p);
    ++I.nls.launch_count;
    NOSH_CUDA(cudaGetLastError());
    V.refreshes = done;
    V.built = I.nls.reg_builds;
    return;
  }
  for (int l = 0; l < L; l++) {
    AmgLevel &A = I.lev[l];
    if (l > 0) {
      AmgLevel &F = I.lev[l - 1];
      rap_offdiag<T><<<div_up(std::max<int64_t>(A.nnz, 1), 256), 256, 0, st>>>(
          A.nnz, F.seg_ptr.p, F.seg_idx.p, I.off<T>(l - 1), V.off[l].p);
      ++I.nls.launch_count;
      rap_diag<T><<<div_up(A.n, 256), 256, 0, st>>>(A.n, F.mem_ptr.p, F.mem_idx.p, F.intra_ptr.p,
                                                     F.intra_idx.p, I.dia<T>(l - 1), I.off<T>(l - 1),
                                                     V.dia[l].p);
      ++I.nls.launch_count;
    }
    if (l < L - 1) {  // the coarsest level is solved directly
      dinv_gershgorin<T><<<div_up(A.n, 256), 256, 0, st>>>(
          A.n, A.rp, I.off<T>(l), I.dia<T>(l), V.dinv[l].p, I.lmax_bits.p + l, I.arrive.p + l, I.err.p,
          l == 0 ? (const T *)V.rowabs0.p : nullptr, I.cheb, V.coef[l].p);
      ++I.nls.launch_count;
    }
  }
  // SpMV schedule per coarse level, once (needs the level's values)
  for (int l = 1; l < L; l++) {
    AmgLevel &A = I.lev[l];
    bool &tuned = sizeof(T) == 4 ? A.tuned32 : A.tuned64;
    if (tuned) continue;
    bool &warp = sizeof(T) == 4 ? A.warp32 : A.warp64;
    if (I.nls.spmv_schedule == 0)
      warp = pick_warp_schedule<T>((int)A.n, A.rp, A.ci, I.off<T>(l), A.block_nnz,
                                   I.nls.red.partials.p, I.nls.red.counter.p, st);
    else
      warp = I.nls.spmv_schedule == 2;
    tuned = true;
  }
  I.invert_coarsest<T>();
  V.refreshes = done;
  V.built = I.nls.reg_builds;
}

// The dense inverse of the coarsest level's operators of precision T.
template <typename T>
void Amg::Impl::invert_coarsest() {
  const AmgLevel &C = lev.back();
  const bool fp32 = sizeof(T) == 4 && max_dim <= kDenseFp32;
  const int L = (int)lev.size();
  cudaStream_t st = nls.stream;
  const int steps = fp32 ? 0 : div_up(max_dim, kPivots);
  double *buf[2] = {dense.p, dense2.p};  // the last step writes the first
  coarse_dense<T><<<div_up(C.n, 128), 128, 0, st>>>(C.n, C.rp, C.ci, off<T>(L - 1), dia<T>(L - 1),
                                                     row_start.p, row_off.p, row_dim.p, buf[steps & 1]);
  if (fp32)
    gauss_jordan_fp32<<<nblk, 1024, (size_t)max_dim * max_dim * sizeof(float), st>>>(
        blk_off.p, blk_dim.p, dense.p, densef.p, err.p);
  for (int k = 0; k < steps; k++)
    launch_dep(ovl(), gauss_jordan_step, dim3(nblk, div_up(max_dim, kPivotCols)), dim3(kPivotThreads), 0, st,
               blk_off.p, blk_dim.p, k * kPivots, (int)(k == steps - 1), (const double *)buf[(steps - k) & 1],
               buf[(steps - k - 1) & 1], densef.p, err.p);
  nls.launch_count += 1 + (fp32 ? 1 : steps);
  NOSH_CUDA(cudaGetLastError());
  inverse_of = sizeof(T);
}

template <typename T>
void Amg::ensure() {
  if (impl->vals<T>().built != impl->nls.reg_builds) refresh<T>();
  if (impl->inverse_of != sizeof(T)) impl->invert_coarsest<T>();
}

template <typename T>
void Amg::Impl::prime() {
  // shared-memory opt-in of every row kernel instantiation, set before any
  // stream capture
  allow_staging<T, ChebOp<T>>();
  allow_staging<T, ChebMinresOp<T>>();
  allow_staging<T, ChebRowDotOp<T>>();
  allow_staging<T, ResidOp<T>>();
}

// The cluster's size: 16 CTAs (above the portable 8) when the device runs
// them at the layouts' largest shared memory, else 8, else one.
void Amg::Impl::choose_cluster() {
  auto fits = [&](int c, const void *k) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = kTailSmem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    const bool ok = cudaOccupancyMaxActiveClusters(&n, k, &cfg) == cudaSuccess && n > 0;
    cudaGetLastError();
    return ok;
  };
  const void *ks[2] = {(const void *)resident_vcycle<float>, (const void *)resident_vcycle<double>};
  for (const void *k : ks) {
    NOSH_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmem));
    NOSH_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  }
  tail_ctas = 1;
  for (int c : {16, 8})
    if (fits(c, ks[0]) && fits(c, ks[1])) {
      tail_ctas = c;
      break;
    }
}

// Shared-memory layout of a resident cycle that starts on level `first`;
// returns its bytes (the dense inverse's rows are staged when they fit too).
template <typename T>
size_t Amg::Impl::tail_layout(int first, std::vector<LevelDesc<T>> *desc, TailPlan<T> *P) {
  const int L = (int)lev.size(), C = tail_ctas;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o += (bytes + 15) / 16 * 16;
    return (uint32_t)at;
  };
  // the longest of the CTAs' ranges of a CSR's entries
  auto longest = [&](const std::vector<int32_t> &ptr, int n, int rw) {
    int m = 0;
    for (int r = 0; r * rw < n; r++) m = std::max(m, ptr[std::min(n, (r + 1) * rw)] - ptr[r * rw]);
    return (size_t)m;
  };
  std::vector<LevelDesc<T>> D(L);
  for (int l = first; l < L; l++) {
    LevelDesc<T> &A = D[l];
    A = LevelDesc<T>{};
    A.n = (int)lev[l].n;
    A.rw = (A.n + C - 1) / C;
    const int cap = sizeof(T) == 8 ? 128 : kTailThreads;
    if (A.rw > kTailRows) o += kTailSmem;  // more rows than a pass covers: does not fit
    A.lnb = 1;  // (see the kernel's note on lanes)
    while (A.lnb < 4 && (A.rw << (A.lnb + 1)) <= cap) ++A.lnb;
    if (l > first || first > 0) {
      A.s_mp = take(4 * (size_t)(A.rw + 1));
      A.s_mi = take(4 * longest(lev[l - 1].h_mem_ptr, A.n, A.rw));
    }
    if (l == L - 1) break;
    A.xa = take(sizeof(C2<T>) * (size_t)A.n);
    A.xb = take(sizeof(C2<T>) * (size_t)A.n);
    A.b = take(sizeof(C2<T>) * (size_t)A.rw);
    A.d = take(sizeof(C2<T>) * (size_t)A.rw);
    A.s_agg = take(4 * (size_t)A.n);
    const size_t nz = longest(lev[l].h_rp, A.n, A.rw);
    A.s_rp = take(4 * (size_t)(A.rw + 1));
    A.s_ci = take(4 * nz);
    A.s_off = take(sizeof(C2<T>) * nz);
    A.s_dia = take(6 * sizeof(T) * (size_t)A.rw);
  }
  const uint32_t bd = take(sizeof(C2<T>) * (size_t)D[L - 1].n), xd = take(sizeof(C2<T>) * (size_t)D[L - 1].n);
  const uint32_t bar = take(8 * (size_t)tail_phases(L - first, std::max(opt.smooth_degree, 1)));
  if (!desc) return o;
  P->dense = TailDense{bd, xd, 0, 0, 0};
  P->s_bar = bar;
  AmgVals<T> &V = vals<T>();
  for (int l = first; l < L; l++) {
    LevelDesc<T> &A = D[l];
    A.rp = lev[l].rp;
    A.ci = lev[l].ci;
    A.off = off<T>(l);
    A.dia = dia<T>(l);
    A.dinv = V.dinv[l].p;
    A.coef = V.coef[l].p;
    A.agg = lev[l].agg.p;
    A.mem_ptr = lev[l].mem_ptr.p;
    A.mem_idx = lev[l].mem_idx.p;
  }
  {
    // the dense inverse's own rows
    const int rw2 = 2 * D[L - 1].rw;
    const size_t before = o;
    P->dense.s_map = take(12 * (size_t)rw2);
    P->dense.s_a = take(sizeof(T) * (size_t)rw2 * max_dim);
    if (o <= (size_t)kTailSmem) P->dense.staged = 1;
    else o = before;
  }
  *desc = std::move(D);
  return o;
}

template <typename T>
void Amg::Impl::build_plan(TailPlan<T> &P, int first) {
  std::vector<LevelDesc<T>> d;
  P.smem = tail_layout<T>(first, &d, &P);
  P.desc.upload(d, nls.stream);
  nls.sync();
  P.lt = first;
}

template <typename T>
void Amg::Impl::launch_tail(const TailPlan<T> &P, TailArgs<T> a, bool overlap) {
  a.fail = nls.h_stage_err + 1;
  a.counter = nls.red.counter.p;
  launch_cluster_dep(overlap, tail_ctas, resident_vcycle<T>, dim3(kTailThreads), P.smem, nls.stream,
                     (const LevelDesc<T> *)P.desc.p, P.lt, (int)lev.size(), std::max(opt.smooth_degree, 1),
                     dense_inv<T>(), dmap(), P.dense, P.s_bar, a, halt);
  ++nls.launch_count;
}

template <typename T, class Op>
void Amg::Impl::rows(int l, const C2<T> *x, const Op &op) {
  const AmgLevel &A = lev[l];
  const bool warp = l == 0 ? (sizeof(T) == 4 ? nls.warp32 : nls.warp64) : (sizeof(T) == 4 ? A.warp32 : A.warp64);
  launch_spmv<T, Op>(warp, (int)A.n, A.rp, A.ci, off<T>(l), x, A.block_nnz, op, nls.red.partials.p, nls.red.counter.p,
                     Op::kReduce ? &nls.red.out.p[32] : nullptr, nls.stream, ovl());
  ++nls.launch_count;
}

// Level l of the V-cycle after its first Chebyshev step: finish the
// pre-smoothing (its result ends in x), coarse correction, post-smoothing.
// With ms != nullptr the fine level's last step also advances MINRES, with
// rowdot != nullptr it writes each vertex's <b, x>.
template <typename T>
void Amg::Impl::descend_ascend(int l, const C2<T> *b, C2<T> *x, MinresScalars *ms, double *rowdot) {
  AmgVals<T> &V = vals<T>();
  AmgLevel &A = lev[l];
  cudaStream_t st = nls.stream;
  const int L = (int)lev.size();
  const int deg = std::max(opt.smooth_degree, 1);
  const int B = 256;
  const T *dv = dia<T>(l);
  C2<T> *cur = (deg % 2 == 1) ? x : V.x2[l].p;
  C2<T> *oth = (deg % 2 == 1) ? V.x2[l].p : x;
  KernelTimer *tm = l == 0 ? &nls.timers[NOSH_KERNEL_SMOOTHER] : nullptr;
  // values per vertex: a Chebyshev step reads x, b, the diagonal block and
  // its inverse and the previous direction d, and writes d and x (16; the
  // first step of a sweep reads no d: 14); the residual reads x, b and the
  // diagonal block and writes the residual (9)
  const int vb = (int)sizeof(T);
  const double cheb_bytes = nls.spmv_bytes(2 * vb, 16 * vb);
  const double cheb0_bytes = nls.spmv_bytes(2 * vb, 14 * vb);
  const double res_bytes = nls.spmv_bytes(2 * vb, 9 * vb);
  // timed as one event pair around the consecutive fine-level launches of
  // the pre-smoothing and the residual (and of the post-smoothing below)
  if (tm) tm->begin(st);
  for (int k = 1; k < deg; k++) {
    ChebOp<T> op{dv, V.dinv[l].p, V.coef[l].p, k, b, cur, V.d[l].p, oth, halt};
    rows<T>(l, cur, op);
    std::swap(cur, oth);
  }
  // (the resident cycle stages its operators under the residual's launch)
  ResidOp<T> rop{dv, b, x, V.res[l].p, halt, !grid_coarse && l + 1 == plan<T>().lt && ovl()};
  rows<T>(l, x, rop);
  if (tm) tm->end(st, (deg - 1) * cheb_bytes + res_bytes, deg);
  const AmgLevel &Cl = lev[l + 1];
  const TailPlan<T> &P = plan<T>();
  if (!grid_coarse && l + 1 == P.lt) {
    TailArgs<T> a{};
    a.head = kHeadRestrict;
    a.out = kOutProlong;
    a.f_res = V.res[l].p;
    a.f_x = x;
    a.f_agg = A.agg.p;
    a.f_mp = A.mem_ptr.p;
    a.f_mi = A.mem_idx.p;
    a.f_n = A.n;
    launch_tail<T>(P, a, ovl());
  } else {
    const bool few = few_members<T>(A.n, Cl.n);
    if (l + 1 < L - 1) {
      // restriction + first step of level l+1, whose pre-smoothing must end
      // in its x buffer
      C2<T> *first = (deg % 2 == 1) ? V.x[l + 1].p : V.x2[l + 1].p;
      launch_dep(ovl(), few ? restrict_first<T, 8> : restrict_first<T, 16>, dim3(div_up(Cl.n * (few ? 8 : 16), B)),
                 dim3(B), 0, st, Cl.n, A.mem_ptr.p, A.mem_idx.p, V.res[l].p, V.b[l + 1].p, V.dinv[l + 1].p,
                 V.coef[l + 1].p, V.d[l + 1].p, first, halt);
      ++nls.launch_count;
      descend_ascend<T>(l + 1, V.b[l + 1].p, V.x[l + 1].p, nullptr);
    } else {
      launch_dep(ovl(), few ? restrict_kernel<T, 8> : restrict_kernel<T, 16>,
                 dim3(div_up(Cl.n * (few ? 8 : 16), B)), dim3(B), 0, st, Cl.n, A.mem_ptr.p, A.mem_idx.p, V.res[l].p,
                 V.b[l + 1].p, halt);
      const int m = (int)(2 * Cl.n);
      launch_dep(ovl(), dense_matvec<T>, dim3(div_up(m * kDenseLanes, B)), dim3(B), 0, st, m, dense_inv<T>(), dmap(),
                 (const T *)V.b[l + 1].p, (T *)V.x[l + 1].p, halt);
      nls.launch_count += 2;
    }
    launch_dep(ovl(), prolong_kernel<T>, dim3(div_up(A.n, B)), dim3(B), 0, st, A.n, A.agg.p, V.x[l + 1].p, x, halt);
    ++nls.launch_count;
  }
  cur = x;
  oth = V.x2[l].p;
  if (tm) tm->begin(st);
  for (int k = 0; k < deg; k++) {
    if (ms && k == deg - 1) {
      ChebMinresOp<T> op{dv, V.dinv[l].p, V.coef[l].p, k, b, cur, V.d[l].p, oth, ms, halt};
      rows<T>(l, cur, op);
    } else if (rowdot && k == deg - 1) {
      ChebRowDotOp<T> op{dv, V.dinv[l].p, V.coef[l].p, k, b, cur, V.d[l].p, oth, rowdot, halt};
      rows<T>(l, cur, op);
    } else {
      ChebOp<T> op{dv, V.dinv[l].p, V.coef[l].p, k, b, cur, V.d[l].p, oth, halt};
      rows<T>(l, cur, op);
    }
    std::swap(cur, oth);
  }
  if (tm) tm->end(st, cheb0_bytes + (deg - 1) * cheb_bytes, deg);
  if (cur != x) {
    NOSH_CUDA(cudaMemcpyAsync(x, cur, A.n * sizeof(C2<T>), cudaMemcpyDeviceToDevice, st));
  }
}

// z = V-cycle(r)
template <typename T>
void Amg::apply(const T *r, T *z) {
  Impl &I = *impl;
  AmgVals<T> &V = I.vals<T>();
  cudaStream_t st = I.nls.stream;
  const int L = (int)I.lev.size();
  const AmgLevel &A = I.lev[0];
  if (L == 1) {
    const int m2 = (int)(2 * A.n);
    launch_dep(I.ovl(), dense_matvec<T>, dim3(div_up(m2 * kDenseLanes, 256)), dim3(256), 0, st, m2,
               I.dense_inv<T>(), I.dmap(), r, z, (const int *)nullptr);
    ++I.nls.launch_count;
    NOSH_CUDA(cudaGetLastError());
    return;
  }
  if (const TailPlan<T> &P = I.plan<T>(); P.lt == 0) {
    // the whole cycle resident; no overlap: it stages the block inverses,
    // which the refresh before it may have written
    TailArgs<T> a{};
    a.head = kHeadVector;
    a.out = kOutVector;
    a.b = (const C2<T> *)r;
    a.z = (C2<T> *)z;
    I.launch_tail<T>(P, a, false);
    NOSH_CUDA(cudaGetLastError());
    return;
  }
  const int deg = std::max(I.opt.smooth_degree, 1);
  C2<T> *first = (deg % 2 == 1) ? (C2<T> *)z : V.x2[0].p;
  launch_dep(I.ovl(), cheb_first<T>, dim3(div_up(A.n, 256)), dim3(256), 0, st, A.n, V.dinv[0].p, V.coef[0].p,
             (const C2<T> *)r, V.d[0].p, first);
  ++I.nls.launch_count;
  I.descend_ascend<T>(0, (const C2<T> *)r, (C2<T> *)z, nullptr);
  NOSH_CUDA(cudaGetLastError());
}

// The fine level's pre-smoothing sweep alone, from x = 0: the first
// Chebyshev step, then degree - 1 SpMV steps (as in descend_ascend).
template <typename T>
void Amg::presmooth(const T *b, T *x) {
  Impl &I = *impl;
  NOSH_CHECK(I.lev.size() >= 2, NOSH_ERR_INVALID, "the hierarchy has one level: no smoother");
  AmgVals<T> &V = I.vals<T>();
  cudaStream_t st = I.nls.stream;
  const AmgLevel &A = I.lev[0];
  const int deg = std::max(I.opt.smooth_degree, 1);
  C2<T> *cur = (deg % 2 == 1) ? (C2<T> *)x : V.x2[0].p;
  C2<T> *oth = (deg % 2 == 1) ? V.x2[0].p : (C2<T> *)x;
  launch_dep(I.ovl(), cheb_first<T>, dim3(div_up(A.n, 256)), dim3(256), 0, st, A.n, V.dinv[0].p, V.coef[0].p,
             (const C2<T> *)b, V.d[0].p, cur);
  ++I.nls.launch_count;
  for (int k = 1; k < deg; k++) {
    ChebOp<T> op{I.dia<T>(0), V.dinv[0].p, V.coef[0].p, k, (const C2<T> *)b, cur, V.d[0].p, oth, nullptr};
    I.rows<T>(0, cur, op);
    std::swap(cur, oth);
  }
  NOSH_CUDA(cudaGetLastError());
}

// One MINRES Lanczos step around the V-cycle:
//   r_old <- J z / beta - (beta/oldb) r_old - (alfa/beta) r_cur  (= r_new)
//   z_out <- V-cycle(r_new),  <r_new, z_out> and the Givens recurrence.
template <typename T>
void Amg::apply_minres(MinresScalars *ms, const T *u, T *r_old, const T *r_cur, T *z_out) {
  Impl &I = *impl;
  AmgVals<T> &V = I.vals<T>();
  cudaStream_t st = I.nls.stream;
  const int L = (int)I.lev.size();
  const AmgLevel &A = I.lev[0];
  if (L == 1) {
    launch_dep(I.ovl(), lanczos_only<T>, dim3(div_up(A.n, 256)), dim3(256), 0, st, A.n, ms, (const C2<T> *)u,
               (C2<T> *)r_old, (const C2<T> *)r_cur);
    apply<T>(r_old, z_out);
    launch_dep(I.ovl(), dot_advance<T>, dim3(div_up(A.n, 256)), dim3(256), 0, st, A.n, (const C2<T> *)r_old,
               (const C2<T> *)z_out, I.nls.red.partials.p, I.nls.red.counter.p, ms);
    I.nls.launch_count += 2;
    NOSH_CUDA(cudaGetLastError());
    return;
  }
  I.halt = &ms->done;
  if (const TailPlan<T> &P = I.plan<T>(); P.lt == 0) {
    TailArgs<T> a{};
    a.head = kHeadLanczos;
    a.out = kOutMinres;
    a.b = (const C2<T> *)u;
    a.r_old = (C2<T> *)r_old;
    a.r_cur = (const C2<T> *)r_cur;
    a.z = (C2<T> *)z_out;
    a.ms = ms;
    I.launch_tail<T>(P, a, I.ovl());
    I.halt = nullptr;
    NOSH_CUDA(cudaGetLastError());
    return;
  }
  const int deg = std::max(I.opt.smooth_degree, 1);
  // the fine level's right-hand side is r_new itself: point b[0] at r_old
  C2<T> *first = (deg % 2 == 1) ? (C2<T> *)z_out : V.x2[0].p;
  launch_dep(I.ovl(), lanczos_first<T>, dim3(div_up(A.n, 256)), dim3(256), 0, st, A.n, ms, (const C2<T> *)u,
             (C2<T> *)r_old, (const C2<T> *)r_cur, V.dinv[0].p, V.coef[0].p, V.d[0].p, first);
  ++I.nls.launch_count;
  I.descend_ascend<T>(0, (const C2<T> *)r_old, (C2<T> *)z_out, ms);
  I.halt = nullptr;
  NOSH_CUDA(cudaGetLastError());
}

template <typename T>
bool Amg::apply_batch(const int32_t *vsys, const MinresScalars *sc, const int *halt, const T *u, T *r_old,
                      const T *r_cur, T *z_out, double *rowdot) {
  Impl &I = *impl;
  AmgVals<T> &V = I.vals<T>();
  if (I.lev.size() == 1 || I.plan<T>().lt == 0) return false;
  const AmgLevel &A = I.lev[0];
  const int deg = std::max(I.opt.smooth_degree, 1);
  C2<T> *first = (deg % 2 == 1) ? (C2<T> *)z_out : V.x2[0].p;
  I.halt = halt;
  launch_dep(I.ovl(), lanczos_first_sys<T>, dim3(div_up(A.n, 256)), dim3(256), 0, I.nls.stream, A.n, vsys, sc,
             (const C2<T> *)u, (C2<T> *)r_old, (const C2<T> *)r_cur, V.dinv[0].p, V.coef[0].p, V.d[0].p, first, halt);
  ++I.nls.launch_count;
  I.descend_ascend<T>(0, (const C2<T> *)r_old, (C2<T> *)z_out, nullptr, rowdot);
  I.halt = nullptr;
  NOSH_CUDA(cudaGetLastError());
  return true;
}

template void Amg::refresh<float>();
template void Amg::refresh<double>();
template void Amg::ensure<float>();
template void Amg::ensure<double>();
template void Amg::apply<float>(const float *, float *);
template void Amg::apply<double>(const double *, double *);
template void Amg::presmooth<float>(const float *, float *);
template void Amg::presmooth<double>(const double *, double *);
template bool Amg::apply_batch<float>(const int32_t *, const MinresScalars *, const int *, const float *, float *,
                                      const float *, float *, double *);
template bool Amg::apply_batch<double>(const int32_t *, const MinresScalars *, const int *, const double *, double *,
                                       const double *, double *, double *);
template void Amg::apply_minres<float>(MinresScalars *, const float *, float *, const float *, float *);
template void Amg::apply_minres<double>(MinresScalars *, const double *, double *, const double *, double *);

}  // namespace nosh
