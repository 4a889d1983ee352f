// Row-block SpMV over the off-diagonal KEO graph with a fused per-vertex
// epilogue (diagonal 2x2 block, residual nonlinearity, reductions).
//
// One CTA = 128 threads on consecutive rows, 1 to 8 threads a row (row_lanes),
// persistent over row blocks.  A row block's nonzeros [rp[r0], rp[r1]) are
// contiguous: one thread stages them into shared memory with two bulk
// asynchronous copies (TMA, cp.async.bulk: column ids and complex values)
// completing on an mbarrier; the several CTAs of an SM overlap one another's
// copies and arithmetic (stage_ctas).  The threads of a row then reduce its
// nonzeros out of shared memory and gather x through the read-only path.  A
// row block whose nonzeros exceed the staging capacity reads them directly.
#pragma once

#include <utility>

#include <type_traits>

#include "common.cuh"

namespace nosh {
namespace dev {

// Arrival at a grid reduction: counter += 1 with acquire-release semantics
// at GPU scope, returning the old value.  The release publishes the CTA's
// partial written before it; the acquire, in the CTA that arrives last,
// orders the partials read after it (behind the CTA barrier that follows)
// after every other CTA's write.  It takes the place of a full fence on
// either side of a relaxed atomic.
__device__ __forceinline__ unsigned arrive_acq_rel(unsigned *counter) {
  unsigned old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;\n" : "=r"(old) : "l"(counter) : "memory");
  return old;
}

constexpr int kRows = 128;  // rows of a row block at one thread a row, and threads of a CTA
// Threads per row of the staged schedule (adjacent lanes, each taking every
// n-th nonzero; a row block then has kRows / n rows), as a power of two: the
// most that still fit one CTA on every multiprocessor and leave a lane
// kLaneNnz nonzeros, up to 8.  One thread walks a long row of a small matrix
// while most multiprocessors idle, and its row blocks may exceed the staging
// buffer: the 1331 rows of some 27 nonzeros of a 32^3 hierarchy take 4.2
// instead of 5.4 us a smoothing step (continuation there 16.4 -> 15.7 ms;
// V-cycles at 48^3, 4913 such rows, 619 -> 607 us; 4 or 6 nonzeros a lane do
// equally, 8 gains a tenth of it).  Short rows lose by the longer fold: 4225
// rows of 6, 4.0 -> 4.5 us with four lanes.  In a grid that is full anyway two
// lanes measured 4 % slower (FP32 smoother at 64^3).
constexpr int kLaneNnz = 6;
inline int row_lanes_log2(int64_t n, int block_nnz) {
  int lr = 0;
  while (lr < 3 && (n << (lr + 1)) <= (int64_t)kRows * kNumSMs && (block_nnz >> (lr + 1)) >= kLaneNnz * kRows) lr++;
  return lr;
}

template <typename T>
struct Acc;  // accumulator type per value type
template <> struct Acc<float> { using type = float; };
template <> struct Acc<double> { using type = double; };

// Grid-wide deterministic sum of one double per thread: block partials, then
// the last CTA to arrive adds them in fixed order and stores *out.  Returns
// true in the first warp of that last CTA, with the sum in *total of all its
// lanes, so callers can continue with scalar work on the result.  That work's
// state (`words` <= 32 doubles at `head`) is fetched into s_head beside the
// partials, whose loads are all under way before the first is added: their
// latencies are the tail of the launch.
__device__ __forceinline__ bool grid_reduce(double v, double *partials, unsigned *counter, double *out,
                                            double *total = nullptr, const double *head = nullptr,
                                            double *s_head = nullptr, int words = 0) {
  __shared__ double s32[32];
  __shared__ bool last;
  const double b = block_sum(v, s32);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = b;
    const unsigned t = arrive_acq_rel(counter);
    last = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return false;
  dep_trigger();
  const unsigned G = gridDim.x, st = blockDim.x, tid = threadIdx.x;
  const int hl = (int)tid - 32;
  const double h = hl >= 0 && hl < words ? __ldcg(head + hl) : 0.0;
  double a = 0.0;
  for (unsigned j0 = 0; j0 < G; j0 += 4 * st) {
    double t[4];
#pragma unroll
    for (int k = 0; k < 4; k++) t[k] = j0 + k * st + tid < G ? __ldcg(partials + j0 + k * st + tid) : 0.0;
    a += t[0];
    if (j0 + st < G) a += t[1];
    if (j0 + 2 * st < G) a += t[2];
    if (j0 + 3 * st < G) a += t[3];
  }
  if (hl >= 0 && hl < words) s_head[hl] = h;
  double s = block_sum(a, s32);  // (its barriers also publish s_head)
  if (tid >= 32) return false;
  s = __shfl_sync(0xffffffffu, s, 0);
  if (tid == 0) {
    *out = s;
    *counter = 0u;
  }
  if (total) *total = s;
  return true;
}

// The same for m <= K values at once (v[0..m-1], partials in columns
// partials + k gridDim.x, one arrival counter): one pass of block sums and
// one arrival instead of m successive grid_reduce calls, each with its own
// barriers, fence and atomic.  The sums are bitwise those of m grid_reduce
// calls (the same block and final summation orders).  Writes out[0..m-1]
// in the last CTA; returns true in exactly one thread.
template <int K>
__device__ __forceinline__ bool grid_reduce_n(const double (&v)[K], int m, double *partials, unsigned *counter,
                                              double *out) {
  __shared__ double sw[32 * K];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double r[K];
#pragma unroll
  for (int k = 0; k < K; k++) r[k] = k < m ? warp_sum(v[k]) : 0.0;
  __syncthreads();
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < K; k++)
      if (k < m) sw[w * K + k] = r[k];
  }
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (k < m) {
        double t = lane < nw ? sw[lane * K + k] : 0.0;
        t = warp_sum(t);
        if (lane == 0) partials[(size_t)k * gridDim.x + blockIdx.x] = t;
      }
    }
  }
  if (threadIdx.x == 0) {
    const unsigned t = arrive_acq_rel(counter);
    last = (t == gridDim.x - 1);
  }
  __syncthreads();
  bool finisher = false;
  if (last) {
    dep_trigger();
    const unsigned G = gridDim.x, st = blockDim.x;
    double acc[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      acc[k] = 0.0;
      if (k < m) {
        const double *pk = partials + (size_t)k * G;
        double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
        unsigned j = threadIdx.x;
        for (; j + 3 * st < G; j += 4 * st) {
          a0 += __ldcg(pk + j);
          a1 += __ldcg(pk + j + st);
          a2 += __ldcg(pk + j + 2 * st);
          a3 += __ldcg(pk + j + 3 * st);
        }
        for (; j < G; j += st) a0 += __ldcg(pk + j);
        acc[k] = warp_sum((a0 + a1) + (a2 + a3));
      }
    }
    __syncthreads();
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < K; k++)
        if (k < m) sw[w * K + k] = acc[k];
    }
    __syncthreads();
    if (w == 0) {
#pragma unroll
      for (int k = 0; k < K; k++) {
        if (k < m) {
          double t = lane < nw ? sw[lane * K + k] : 0.0;
          t = warp_sum(t);
          if (lane == 0) out[k] = t;
        }
      }
    }
    if (threadIdx.x == 0) {
      *counter = 0u;
      finisher = true;
    }
  }
  return finisher;
}

// The type a launch accumulates the epilogues' partials in: the SpMV's
// accumulator type unless the Op asks for FP64 (`using Part = double`).
template <class Op, class A, class = void>
struct PartOf {
  using type = A;
};
template <class Op, class A>
struct PartOf<Op, A, decltype((void)sizeof(typename Op::Part), void())> {
  using type = typename Op::Part;
};

// One nonzero of a row sum: (sr, si) += v x (complex).  In FP64 each component
// is two chained FMAs: GB300's FP64 pipe takes 16 cycles of an SM per warp
// instruction and bounds these kernels, so four instructions a nonzero
// instead of the six that adding the rounded product takes (mul, fma, add
// per component), with one rounding less.  In FP32 the pipe is not the
// bound; the product is formed first.
__device__ __forceinline__ void row_mac(float &sr, float &si, const C2<float> &v, const C2<float> &x) {
  sr += v.x * x.x - v.y * x.y;
  si += v.x * x.y + v.y * x.x;
}
__device__ __forceinline__ void row_mac(double &sr, double &si, const C2<double> &v, const C2<double> &x) {
  sr = fma(v.x, x.x, sr);
  si = fma(v.x, x.y, si);
  sr = fma(-v.y, x.y, sr);
  si = fma(v.y, x.x, si);
}

// Op must provide:
//   static constexpr bool kReduce;
//   struct Pre;                                  -- the row's epilogue operands
//   __device__ Pre load(int row)                 -- issued before the row's
//                                                   nonzeros arrive, so the
//                                                   epilogue loads overlap the
//                                                   staging and the gathers
//   __device__ double finish(int row, acc sr, acc si, const Pre &)
//                                                -- writes y[row], returns the
//                                                   thread's partial
// and, when kReduce, may provide kHook + hook(total, state): scalar work done
// by one warp once the grid sum is known, on kHeadWords doubles from head().
template <class Op, class = void>
struct HasHook {
  static constexpr bool value = false;
};
template <class Op>
struct HasHook<Op, decltype((void)Op::kHook, void())> {
  static constexpr bool value = Op::kHook;
};
template <class Op>
__device__ __forceinline__ void reduce_rows(const Op &op, double part, double *partials, unsigned *counter,
                                            double *red_out) {
  if constexpr (HasHook<Op>::value) {
    __shared__ double s_head[32];
    double total = 0.0;
    if (grid_reduce(part, partials, counter, red_out, &total, op.head(), s_head, Op::kHeadWords))
      op.hook(total, s_head);
  } else {
    grid_reduce(part, partials, counter, red_out);
  }
}
// An Op may also carry `const int *halt`: when it points at a value >= 2
// the whole launch returns at once (MINRES iterations of a captured chunk
// that follow convergence).
template <class Op, class = void>
struct HasHalt {
  static constexpr bool value = false;
};
template <class Op>
struct HasHalt<Op, decltype((void)std::declval<Op>().halt, void())> {
  static constexpr bool value = true;
};
template <class Op>
__device__ __forceinline__ bool halted(const Op &op) {
  if constexpr (HasHalt<Op>::value) {
    return op.halt != nullptr && *op.halt >= 2;
  } else {
    return false;
  }
}
// The same test before dep_sync(), read from L2: the flag only rises within
// a solve and is reset several launches before the solve's first iteration,
// so a true answer is final, while a false one may be stale (the kernel this
// launch follows may have raised it without its write being visible yet).
template <class Op>
__device__ __forceinline__ bool halted_early(const Op &op) {
  if constexpr (HasHalt<Op>::value) {
    return op.halt != nullptr && __ldcg(op.halt) >= 2;
  } else {
    return false;
  }
}
// An Op may carry `bool trigger`: the launch then lets its successor start as
// soon as all its own CTAs run, for a successor that has work to do before
// its dep_sync() and leaves room on the SMs (the resident coarse cycle).
template <class Op, class = void>
struct HasTrigger {
  static constexpr bool value = false;
};
template <class Op>
struct HasTrigger<Op, decltype((void)std::declval<Op>().trigger, void())> {
  static constexpr bool value = true;
};
template <class Op>
__device__ __forceinline__ void early_trigger(const Op &op) {
  if constexpr (HasTrigger<Op>::value) {
    if (op.trigger) dep_trigger();
  }
}
// ---- bulk-copy staging (TMA + mbarrier) ------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_addr(bar)));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}
// global -> shared bulk copy; dst, src 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}
// Default bound of a staging wait, in polls of mbarrier.try_wait.
constexpr uint32_t kStageWaitPolls = 1u << 20;
// Bounded wait for the phase with the given parity; false after `limit`
// polls (at once for a limit of 0).
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, uint32_t limit = kStageWaitPolls) {
  const uint32_t a = smem_addr(bar);
  for (uint32_t it = 0; it < limit; it++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Shared memory of a CTA's staging buffer (column ids, then complex values)
// for a capacity of cap nonzeros (a multiple of 4).
template <typename T>
__host__ __device__ constexpr size_t stage_bytes(int cap) {
  return (size_t)cap * (sizeof(int32_t) + sizeof(C2<T>));
}
// CTAs per SM the staged kernel is compiled for (its register budget).  A CTA
// has one buffer, and the other CTAs of its SM run under its copies: two
// buffers left room for fewer CTAs, and the gathers, whose latency bounds the
// FP32 kernel, and the FP64 pipe, which bounds the other, waited.
// FP64, a tetrahedral mesh: two buffers (72 KB) fit three CTAs, one fits four
// (the smoother's step, 110 registers) or five (the residual, 95).  J rebuild +
// apply at 160^3 776 -> 699 us, V-cycles at 48^3 925 -> 868 us; six CTAs (80
// registers) gained 1 % more there and lost 3 % on a 32^3 continuation.
// FP32: two buffers with 16 gathers in flight a row (88 registers) fit five
// CTAs, one with 8 gathers seven (the Jacobian, 70 registers) or eight (the
// smoother's step, 64).  A mixed continuation step at
// 64^3 73.3 -> 70.5 ms; one buffer with 16 gathers and five or six CTAs 71.1
// and 71.9, with 8 gathers and all held to eight CTAs 71.2.
template <typename T>
__host__ __device__ constexpr int stage_ctas() {
  return sizeof(T) == 4 ? 7 : 4;
}
// Largest staging capacity of one buffer: 48 KB.
template <typename T>
__host__ __device__ constexpr int stage_limit() {
  return (int)((48 * 1024) / (sizeof(int32_t) + sizeof(C2<T>))) & ~3;
}
// Slots of the reduction counters that hold the address of the host's failure
// word (pinned memory, read after every synchronisation): a bounded wait that
// gave up sets it.
constexpr int kStageErrorSlot = 12;
__device__ __forceinline__ void stage_fail(const unsigned *counter) {
  unsigned *const *p = reinterpret_cast<unsigned *const *>(counter + kStageErrorSlot);
  if (*p) **reinterpret_cast<volatile unsigned *const *>(p) = 1u;
}
// Slot holding a diagnostic override of the staging-wait bound: 0 = the
// default kStageWaitPolls, v > 0 = v - 1 polls.  Read only by launches that
// stage (cap > 0).
constexpr int kStageWaitSlot = 14;

template <typename T, class Op, bool Lanes = false>
__global__ void __launch_bounds__(kRows, stage_ctas<T>())
    row_block_apply(int N, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                    const C2<T> *__restrict__ val, const C2<T> *__restrict__ x, int cap,
                    Op op, double *partials, unsigned *counter, double *red_out, int log2_lanes) {
  using A = typename Acc<T>::type;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar;
  const int lr = Lanes ? log2_lanes : 0;
  const int R = 1 << lr, rows = kRows >> lr;  // lanes of a row, rows of a block
  const int nblocks = (N + rows - 1) / rows;
  if (threadIdx.x == 0) {
    mbar_init(&bar);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  __syncthreads();
  // row block -> its aligned nonzero range; staged when it fits
  auto range = [&](int rb, int &ks, int &n) {
    const int r0 = rb * rows, r1 = min(N, r0 + rows);
    const int k0 = __ldg(rp + r0), k1 = __ldg(rp + r1);
    ks = k0 & ~3;  // 16-byte aligned start for both arrays
    n = k1 - ks;
  };
  auto issue = [&](int rb) {
    int ks, n;
    range(rb, ks, n);
    if (n > 0 && n <= cap) {
      const uint32_t cb = (uint32_t)(((n + 3) >> 2) * 16);                   // column ids
      const uint32_t vb = (uint32_t)(((size_t)n * sizeof(C2<T>) + 15) / 16 * 16);  // values
      mbar_expect_tx(&bar, cb + vb);
      bulk_g2s(smem_raw, ci + ks, cb, &bar);
      bulk_g2s(smem_raw + (size_t)cap * sizeof(int32_t), val + ks, vb, &bar);
    }
  };
  // The first row block's copy is issued before dep_sync(): the matrix (row
  // pointers, column ids, values) is never written by the kernel that a
  // launch with overlap follows, so the copy is in flight while the launch
  // waits for that kernel's completion.
  // row blocks blockIdx.x, + gridDim.x, ... (strided: consecutive row blocks,
  // which share x gathers, run at the same time on different SMs; contiguous
  // chunks per CTA measured 5 % slower at 64^3)
  const int rb0 = blockIdx.x, rb_end = nblocks;
  auto nxt = [&](int rb) { return rb + (int)gridDim.x; };
  const bool skip = halted_early(op);
  if (!skip && threadIdx.x == 0 && rb0 < rb_end) issue(rb0);
  dep_sync();
  early_trigger(op);
  if (halted(op)) {
    // let the copy issued above land before the CTA leaves
    if (!skip && threadIdx.x == 0 && rb0 < rb_end) {
      int ks, n;
      range(rb0, ks, n);
      if (n > 0 && n <= cap && !mbar_wait(&bar, 0u)) stage_fail(counter);
    }
    return;
  }
  typename PartOf<Op, A>::type part = 0;
  uint32_t parity = 0u;
  bool ok = true;
  bool staged = false;  // the current row block's copy was issued
  uint32_t limit = kStageWaitPolls;
  if (cap > 0) {
    const unsigned o = __ldcg(counter + kStageWaitSlot);
    if (o != 0u) limit = o - 1u;
  }
  for (int rb = rb0; rb < rb_end; rb = nxt(rb)) {
    int ks, n;
    range(rb, ks, n);
    const int row = rb * rows + ((int)threadIdx.x >> lr), lane_r = (int)threadIdx.x & (R - 1);
    typename Op::Pre pre{};
    if (row < N && lane_r == 0) pre = op.load(row);
    const int b = row < N ? __ldg(rp + row) : 0, e = row < N ? __ldg(rp + row + 1) : 0;
    staged = n > 0 && n <= cap;
    const bool arrived = staged ? mbar_wait(&bar, parity, limit) : true;
    if (__syncthreads_or(!arrived)) {  // the CTA leaves together
      ok = false;
      break;
    }
    if (staged) parity ^= 1u;
    const int32_t *s_col = reinterpret_cast<const int32_t *>(smem_raw);
    const C2<T> *s_val = reinterpret_cast<const C2<T> *>(smem_raw + (size_t)cap * sizeof(int32_t));
    A sr = 0, si = 0;
    if (staged) {
      // batches of kBatch nonzeros per lane (the row's lanes take every R-th
      // one): all gathers of a batch are issued before the first is used (a
      // row of the mesh graph is one or two); the values are read from shared
      // memory when used, so only the gathered x of a batch occupies registers
      // An FP64 instruction whose lanes are all off still takes the pipe, so a
      // batch goes by pairs of nonzeros, and a branch that the whole warp takes
      // skips those beyond its longest row: rows of 14 paid for 16, rows of 6
      // for 8.  J rebuild + apply at 160^3 643 -> 565 us, V-cycles at 48^3 611
      // -> 563 us, 24 squares of 97^2 16.0 -> 14.9 ms.  FP32 predicates each
      // nonzero (in pairs three products at 64^3 lost 2 %).
      constexpr int kBatch = 8, kPair = sizeof(T) == 8 ? 2 : 1;
      const int k0 = b - ks + lane_r, cnt = row < N ? (e - ks - k0 + R - 1) >> lr : 0;
      const int most = __reduce_max_sync(0xffffffffu, cnt);
      for (int q = 0; q < most; q += kBatch) {
        C2<T> xv[kBatch];
#pragma unroll
        for (int g = 0; g < kBatch; g += kPair)
          if (g == 0 || q + g < most) {
#pragma unroll
            for (int u = g; u < g + kPair; u++)
              if (q + u < cnt) xv[u] = ldg(x + s_col[k0 + ((q + u) << lr)]);
          }
#pragma unroll
        for (int g = 0; g < kBatch; g += kPair)
          if (g == 0 || q + g < most) {
#pragma unroll
            for (int u = g; u < g + kPair; u++)
              if (q + u < cnt) row_mac(sr, si, s_val[k0 + ((q + u) << lr)], xv[u]);
          }
      }
    } else if (row < N) {
      for (int k = b + lane_r; k < e; k += R) {
        const C2<T> v = ldg(val + k);
        const C2<T> xv = ldg(x + __ldg(ci + k));
        row_mac(sr, si, v, xv);
      }
    }
    // the row's lanes are adjacent: fold their partial sums into lane 0, one
    // component on the even lanes and the other on the odd ones
    if (Lanes) {
      const bool odd = lane_r & 1;
      A v = odd ? si : sr;
      v += __shfl_xor_sync(0xffffffffu, odd ? sr : si, 1);
      for (int o = R / 2; o > 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      sr = v;
      si = __shfl_xor_sync(0xffffffffu, v, 1);
    }
    if (row < N && lane_r == 0) part += (typename PartOf<Op, A>::type)op.finish(row, sr, si, pre);
    __syncthreads();  // the buffer's readers are done: it may be refilled
    if (threadIdx.x == 0 && nxt(rb) < rb_end) issue(nxt(rb));
  }
  if (!ok) {
    // a wait gave up: record it, give the copy still in flight a last wait at
    // the default bound, so that it does not land in shared memory after the
    // CTA has left, and leave (the results of this launch are invalid)
    if (threadIdx.x == 0) stage_fail(counter);
    if (staged) mbar_wait(&bar, parity);
    return;
  }
  if constexpr (Op::kReduce) reduce_rows(op, (double)part, partials, counter, red_out);
}

// Warp-cooperative schedule of the same SpMV + epilogue (no staging): a
// warp owns 32 consecutive rows and walks them in 16 pairs, a half-warp per
// row, each lane loading one nonzero (coalesced: a row's nonzeros are
// contiguous) and gathering its x; half-warp shuffles reduce the row and
// hand the sum to the row's own lane, so the epilogue runs on all 32 lanes
// with coalesced accesses.  Few registers and no shared memory: high
// occupancy for latency hiding.  kWarpThreads threads per CTA, persistent.
constexpr int kWarpThreads = 256;
template <typename T, class Op>
__global__ void __launch_bounds__(kWarpThreads)
    row_warp_apply(int N, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                   const C2<T> *__restrict__ val, const C2<T> *__restrict__ x, Op op, double *partials,
                   unsigned *counter, double *red_out) {
  using A = typename Acc<T>::type;
  dep_sync();
  early_trigger(op);
  if (halted(op)) return;
  const int lane = threadIdx.x & 31, hl = lane & 15, half = lane >> 4;
  const int nwb = (N + 31) / 32;
  const int wpb = kWarpThreads / 32;
  typename PartOf<Op, A>::type part = 0;
  for (int wb = blockIdx.x * wpb + (threadIdx.x >> 5); wb < nwb; wb += gridDim.x * wpb) {
    const int r0 = wb * 32;
    const int row = r0 + lane;
    typename Op::Pre pre{};
    if (row < N) pre = op.load(row);
    // row pointers of the 32 rows and the block end
    const int beg = __ldg(rp + min(row, N));
    const int bend = __ldg(rp + min(r0 + 32, N));
    A msr = 0, msi = 0;
    // two batches of 8 row pairs: the column ids and values of a batch are
    // loaded together, then all its x gathers, so a batch costs two memory
    // round trips; rows longer than 16 nonzeros finish in a tail loop
#pragma unroll
    for (int p0 = 0; p0 < 16; p0 += 8) {
      int k[8], e[8];
      int32_t c[8];
      C2<T> v[8], xv[8];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const int rr = 2 * (p0 + q) + half;
        const int b = __shfl_sync(0xffffffffu, beg, rr);
        const int e1 = __shfl_sync(0xffffffffu, beg, (rr + 1) & 31);
        e[q] = rr < 31 ? e1 : bend;
        k[q] = b + hl;
      }
#pragma unroll
      for (int q = 0; q < 8; q++) {
        c[q] = 0;
        v[q] = C2<T>{0, 0};
        if (k[q] < e[q]) {
          c[q] = __ldg(ci + k[q]);
          v[q] = ldg(val + k[q]);
        }
      }
#pragma unroll
      for (int q = 0; q < 8; q++) xv[q] = k[q] < e[q] ? ldg(x + c[q]) : C2<T>{0, 0};
#pragma unroll
      for (int q = 0; q < 8; q++) {
        A sr = v[q].x * xv[q].x - v[q].y * xv[q].y;
        A si = v[q].x * xv[q].y + v[q].y * xv[q].x;
        for (int kk = k[q] + 16; kk < e[q]; kk += 16) {
          const C2<T> vv = ldg(val + kk);
          const C2<T> xx = ldg(x + __ldg(ci + kk));
          row_mac(sr, si, vv, xx);
        }
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) {
          sr += __shfl_xor_sync(0xffffffffu, sr, off);
          si += __shfl_xor_sync(0xffffffffu, si, off);
        }
        // lanes 2p and 2p+1 take the sums of halves 0 and 1
        const A tr = __shfl_sync(0xffffffffu, sr, (lane & 1) << 4);
        const A ti = __shfl_sync(0xffffffffu, si, (lane & 1) << 4);
        if ((lane >> 1) == p0 + q) {
          msr = tr;
          msi = ti;
        }
      }
    }
    if (row < N) part += (typename PartOf<Op, A>::type)op.finish(row, msr, msi, pre);
  }
  if constexpr (Op::kReduce) reduce_rows(op, (double)part, partials, counter, red_out);
}

// Resident CTAs of row_warp_apply on the device, capped by the work.
int warp_grid(const void *kernel, int64_t n_rows);

// Grid for a persistent row kernel of `threads` threads per CTA: the
// resident capacity of the device for this kernel and shared-memory size,
// capped by the number of row blocks n_blocks.
int row_grid(const void *kernel, int threads, size_t smem, int64_t n_blocks);

// Opts the staged kernels of Op into the largest staging buffer (done ahead of
// a capture where the first launch may be in one).
template <typename T, class Op>
void allow_staging() {
  for (auto *k : {row_block_apply<T, Op, false>, row_block_apply<T, Op, true>})
    NOSH_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)stage_bytes<T>(stage_limit<T>())));
}

// Launch the SpMV + epilogue over an off-diagonal CSR with one of the two
// schedules (warp: row_warp_apply, else the staged row_block_apply); block_nnz:
// the longest 4-aligned range of nonzeros of a block of kRows rows.
//
// With `overlap` the launch may start while the previous kernel of the stream
// finishes (launch_dep); the staged schedule then copies its first row block
// before waiting for it, so the previous kernel must not write this matrix.
template <typename T, class Op>
void launch_spmv(bool warp, int N, const int32_t *rp, const int32_t *ci, const C2<T> *val, const C2<T> *x,
                 int block_nnz, const Op &op, double *partials, unsigned *counter, double *red_out,
                 cudaStream_t st, bool overlap = false) {
  if (warp) {
    const int grid = warp_grid((const void *)row_warp_apply<T, Op>, N);
    launch_dep(overlap, row_warp_apply<T, Op>, dim3(grid), dim3(kWarpThreads), 0, st, N, rp, ci, val, x, op,
               partials, counter, red_out);
  } else {
    const int lr = row_lanes_log2(N, block_nnz);
    const auto kernel = lr > 0 ? row_block_apply<T, Op, true> : row_block_apply<T, Op, false>;
    static bool attr_set = false;  // per instantiation
    if (!attr_set) {
      allow_staging<T, Op>();
      attr_set = true;
    }
    const int cap = std::min((block_nnz + 3) & ~3, stage_limit<T>());
    const size_t smem = stage_bytes<T>(cap);
    // (kernels of one lane a row are compiled apart: with the lanes a parameter
    // the FP32 ones lost 3 %)
    launch_dep(overlap, kernel, dim3(row_grid((const void *)kernel, kRows, smem, div_up((int64_t)N << lr, kRows))),
               dim3(kRows), smem, st, N, rp, ci, val, x, cap, op, partials, counter, red_out, lr);
  }
  NOSH_CUDA(cudaGetLastError());
}

// The faster schedule for one matrix: both are timed once (CUDA events,
// after a warm-up) on y = A x + D x with <x, y> reduced, when the matrix
// structure is set up.
template <typename T>
bool pick_warp_schedule(int N, const int32_t *rp, const int32_t *ci, const C2<T> *val, int block_nnz, double *partials,
                        unsigned *counter, cudaStream_t st);

// ---- epilogues --------------------------------------------------------
// y = K x : diagonal K_ii = sum of incident alpha (real)
template <typename T>
struct KeoOp {
  static constexpr bool kReduce = false;
  const T *kdiag;
  const C2<T> *x;
  C2<T> *y;
  struct Pre {
    C2<T> xi;
    T d;
  };
  __device__ Pre load(int i) const { return Pre{x[i], kdiag[i]}; }
  __device__ double finish(int i, T sr, T si, const Pre &p) const {
    y[i] = C2<T>{sr + p.d * p.xi.x, si + p.d * p.xi.y};
    return 0.0;
  }
};

// y = sum (no diagonal): dK/dp
template <typename T>
struct PlainOp {
  static constexpr bool kReduce = false;
  C2<T> *y;
  struct Pre {};
  __device__ Pre load(int) const { return Pre{}; }
  __device__ double finish(int i, T sr, T si, const Pre &) const {
    y[i] = C2<T>{sr, si};
    return 0.0;
  }
};

// y = K_offdiag x + [[d0r, d1b], [d1b, d0i]] x_i (Jacobian or regularised
// KEO; the diagonal blocks include K_ii); optionally sum_i <x_i, y_i>.
template <typename T, bool kDot, typename Out = T>
struct BlockDiagOp {
  static constexpr bool kReduce = kDot;
  const T *d;  // 3 per vertex
  const C2<T> *x;
  C2<Out> *y;
  struct Pre {
    C2<T> xi;
    T d0r, d0i, d1b;
  };
  __device__ Pre load(int i) const { return Pre{x[i], d[3 * i], d[3 * i + 1], d[3 * i + 2]}; }
  __device__ double finish(int i, T sr, T si, const Pre &p) const {
    const T yr = sr + p.d0r * p.xi.x + p.d1b * p.xi.y;
    const T yi = si + p.d1b * p.xi.x + p.d0i * p.xi.y;
    y[i] = C2<Out>{(Out)yr, (Out)yi};
    return kDot ? (double)p.xi.x * (double)yr + (double)p.xi.y * (double)yi : 0.0;
  }
};

// F = K psi + cv t (V + g|psi|^2) psi (FP64), optionally ||F||^2; with soff,
// also the off-diagonal sums (K psi)_i - K_ii psi_i (the base of a later
// ResidualUpdateOp)
template <bool kNorm>
struct ResidualOp {
  static constexpr bool kReduce = kNorm;
  const double *kdiag, *cvt, *V;
  double g;
  const C2<double> *x;
  C2<double> *y;
  C2<double> *soff = nullptr;
  struct Pre {
    C2<double> p;
    double kd, ct, v;
  };
  __device__ Pre load(int i) const { return Pre{x[i], kdiag[i], cvt[i], V[i]}; }
  __device__ double finish(int i, double sr, double si, const Pre &q) const {
    if (soff) soff[i] = C2<double>{sr, si};
    const double a = q.kd + q.ct * (q.v + g * (q.p.x * q.p.x + q.p.y * q.p.y));
    const double fr = sr + a * q.p.x, fi = si + a * q.p.y;
    y[i] = C2<double>{fr, fi};
    return kNorm ? fr * fr + fi * fi : 0.0;
  }
};

// F of psi + dx from the off-diagonal sums of K psi (soff, FP64) and the
// FP32 SpMV of the update: soff += K dx (in place), F = soff + cv t (V +
// g|psi+dx|^2)(psi+dx) with the updated state `x` (FP64), ||F||^2 summed in
// FP64.  K is linear and the nonlinearity is per vertex, so this is F itself;
// the FP32 part is the product of the small update only, whose rounding
// (~1e-7 of |K dx|) lies far below the FP64 rounding of the O(1) sums.
struct ResidualUpdateOp {
  static constexpr bool kReduce = true;
  using Part = double;
  const double *kdiag, *cvt, *V;
  double g;
  const C2<double> *x;
  C2<double> *y;
  C2<double> *soff;
  struct Pre {
    C2<double> p, s;
    double kd, ct, v;
  };
  __device__ Pre load(int i) const { return Pre{x[i], soff[i], kdiag[i], cvt[i], V[i]}; }
  __device__ double finish(int i, float sr, float si, const Pre &q) const {
    const double s_r = q.s.x + (double)sr, s_i = q.s.y + (double)si;
    soff[i] = C2<double>{s_r, s_i};
    const double a = q.kd + q.ct * (q.v + g * (q.p.x * q.p.x + q.p.y * q.p.y));
    const double fr = s_r + a * q.p.x, fi = s_i + a * q.p.y;
    y[i] = C2<double>{fr, fi};
    return fr * fr + fi * fi;
  }
};

}  // namespace dev
}  // namespace nosh
