// Mesh set-up on the GPU: edges, KEO graph and edge -> nonzero scatter map
// from the cells, then the geometry in FP64 (edge coefficients, covolumes,
// control volumes).
//
// Reference: nosh::mesh + mesh_tri / mesh_tetra (src/mesh.cpp,
// src/mesh_tri.cpp, src/mesh_tetra.cpp).  Edge order: the reference takes
// MOAB's entity order, which is not reproducible without MOAB; here edges are
// the canonical sorted pairs (v0 < v1) in lexicographic order, and the KEO
// graph (sorted columns per row) is identical to Tpetra's after fillComplete.
//
// The integer work is a vertex -> cell incidence (counting, scan, scatter),
// then a warp per vertex that sorts its incident cells (so that every later
// sum runs in cell order, whatever order the scatter left) and its neighbours.
// At 64^3 (1.57 M tetrahedra) 0.65 ms on the device, 60 of the 75 ms of the
// whole mesh on the host's cores; the mesh now takes 4.9 ms, half of them the
// copies of its description.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

#include "mesh.cuh"

namespace nosh {

namespace {

// local edge k of a simplex joins local vertices (pair0(k), pair1(k)):
// triangles (0,1),(0,2),(1,2); tetrahedra (0,1),(0,2),(0,3),(1,2),(1,3),(2,3).
// constexpr so that unrolled loops index register arrays statically.
template <int nvc>
__host__ __device__ constexpr int pair0(int k) {
  return nvc == 3 ? (k < 2 ? 0 : 1) : (k < 3 ? 0 : (k < 5 ? 1 : 2));
}
template <int nvc>
__host__ __device__ constexpr int pair1(int k) {
  return nvc == 3 ? (k == 0 ? 1 : 2) : (k < 3 ? k + 1 : (k == 3 ? 2 : 3));
}
// the local edge of local vertices a != b
template <int nvc>
__device__ __forceinline__ constexpr int edge_of(int a, int b) {
  const int lo = a < b ? a : b, hi = a < b ? b : a;
  return nvc == 3 ? lo + hi - 1 : (lo == 0 ? hi - 1 : lo + hi);
}

// ------------------------------------------------------------- topology
__global__ void count_incident(int64_t n, const int32_t *__restrict__ cells, int32_t *cnt) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
    atomicAdd(cnt + cells[k], 1);
}
__global__ void scatter_incident(int64_t n, const int32_t *__restrict__ cells, int32_t *cur, int32_t *vc) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
    vc[atomicAdd(cur + cells[k], 1)] = (int32_t)k;
}

// Exclusive scan of n counts (in: int32, out: n + 1 int64 prefix sums stored as
// V), in tiles of 1024: tile sums, their scan by one CTA, then the tiles.
constexpr int kScanTile = 1024;
__device__ __forceinline__ int64_t block_scan(int64_t v, int64_t *sm) {
  // inclusive over 1024 threads
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) sm[w] = v;
  __syncthreads();
  if (w == 0) {
    int64_t t = sm[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t u = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += u;
    }
    sm[lane] = t;
  }
  __syncthreads();
  return v + (w ? sm[w - 1] : 0);
}
__global__ void __launch_bounds__(kScanTile) scan_tiles(int64_t n, const int32_t *__restrict__ in, int64_t *tile) {
  __shared__ int64_t sm[32];
  const int64_t i = blockIdx.x * (int64_t)kScanTile + threadIdx.x;
  const int64_t s = block_scan(i < n ? in[i] : 0, sm);
  if (threadIdx.x == kScanTile - 1) tile[blockIdx.x] = s;
}
__global__ void __launch_bounds__(kScanTile) scan_sums(int64_t nt, int64_t *tile) {
  __shared__ int64_t sm[32];
  int64_t carry = 0;
  for (int64_t t0 = 0; t0 < nt; t0 += kScanTile) {
    const int64_t t = t0 + threadIdx.x;
    const int64_t v = t < nt ? tile[t] : 0;
    const int64_t s = block_scan(v, sm);
    const int64_t total = sm[31];
    if (t < nt) tile[t] = carry + s - v;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) tile[nt] = carry;
}
__global__ void __launch_bounds__(kScanTile) scan_write(int64_t n, const int32_t *__restrict__ in,
                                                        const int64_t *__restrict__ tile, int32_t *out) {
  __shared__ int64_t sm[32];
  const int64_t i = blockIdx.x * (int64_t)kScanTile + threadIdx.x;
  const int64_t v = i < n ? in[i] : 0;
  const int64_t s = block_scan(v, sm) + tile[blockIdx.x];
  if (i < n) out[i] = (int32_t)(s - v);
  if (i == n - 1) out[n] = (int32_t)s;
}

// A warp per vertex: its incident (cell, slot) codes sorted in place, and its
// neighbours (the other vertices of those cells) sorted and without
// repetition at nb + (nvc - 1) ptr[v], their number and how many are above v.
// Ranks by counting in shared memory: a vertex of a tetrahedral mesh has some
// 24 cells and 72 candidates.  Vertices with more than kMaxIncident cells are
// left to the host, listed in `hubs`.  Bound by the counting loops (0.49 ms at
// 64^3).
constexpr int kMaxIncident = 84;  // 3 x 84 candidates
constexpr int kNbWarps = 4;
template <int nvc>
__global__ void __launch_bounds__(32 * kNbWarps)
    neighbour_kernel(int64_t N, const int32_t *__restrict__ cells, const int32_t *__restrict__ ptr, int32_t *vc,
                     int32_t *nb, int32_t *deg, int32_t *up, int32_t *hubs, int *nhubs) {
  constexpr int kCand = kMaxIncident * 3;
  __shared__ int32_t s_code[kNbWarps][kMaxIncident], s_cand[kNbWarps][kCand];
  __shared__ uint8_t s_first[kNbWarps][kCand + 4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int64_t v = blockIdx.x * (int64_t)kNbWarps + w; v < N; v += (int64_t)gridDim.x * kNbWarps) {
    const int b = ptr[v], d = ptr[v + 1] - b;
    if (d > kMaxIncident) {
      if (lane == 0) hubs[atomicAdd(nhubs, 1)] = (int32_t)v;
      continue;
    }
    int32_t *code = s_code[w], *cand = s_cand[w];
    uint8_t *first = s_first[w];
    __syncwarp();
    for (int q = lane; q < d; q += 32) code[q] = vc[b + q];
    __syncwarp();
    for (int q = lane; q < d; q += 32) {
      const int32_t c = code[q];
      int r = 0;
      for (int j = 0; j < d; j++) r += code[j] < c;
      vc[b + r] = c;
      const int64_t cell = c / nvc;
      int o = 0;
#pragma unroll
      for (int k = 0; k < nvc; k++) {
        const int32_t u = cells[nvc * cell + k];
        if (u != (int32_t)v) cand[(nvc - 1) * q + o++] = u;
      }
    }
    __syncwarp();
    const int m = (nvc - 1) * d;
    for (int q = lane; q < m; q += 32) {
      const int32_t c = cand[q];
      bool f = true;
      for (int j = 0; j < q; j++) f = f && cand[j] != c;
      first[q] = f;
    }
    __syncwarp();
    int above = 0, uniq = 0;
    for (int q = lane; q < m; q += 32) {
      if (!first[q]) continue;
      const int32_t c = cand[q];
      int r = 0;
      for (int j = 0; j < m; j++) r += first[j] && cand[j] < c;
      nb[(int64_t)(nvc - 1) * b + r] = c;
      uniq++;
      above += c > (int32_t)v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      uniq += __shfl_xor_sync(0xffffffffu, uniq, o);
      above += __shfl_xor_sync(0xffffffffu, above, o);
    }
    if (lane == 0) {
      deg[v] = uniq;
      up[v] = above;
    }
  }
}

// rows of the graph and the edges, half a warp per vertex (the upper
// neighbours of each vertex are its edges, in lexicographic order)
__global__ void graph_rows(int64_t N, int nvc, const int32_t *__restrict__ ptr, const int32_t *__restrict__ nb,
                           const int32_t *__restrict__ rp, const int32_t *__restrict__ up,
                           const int32_t *__restrict__ ebase, int32_t *ci, int32_t *edges, int32_t *pos_fwd,
                           int32_t *nz_edge) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, v = t >> 4;
  if (v >= N) return;
  const int b = rp[v], d = rp[v + 1] - b, low = d - up[v];
  const int32_t *src = nb + (int64_t)(nvc - 1) * ptr[v];
  for (int q = (int)(t & 15); q < d; q += 16) {
    const int32_t c = src[q];
    ci[b + q] = c;
    if (q >= low) {
      const int e = ebase[v] + q - low;
      edges[2 * (int64_t)e] = (int32_t)v;
      edges[2 * (int64_t)e + 1] = c;
      pos_fwd[e] = b + q;
      nz_edge[b + q] = e;
    }
  }
}
// the nonzero of (v1, v0) of each edge, by bisection of row v1; and the row
// lengths that the SpMV's staging wants
__global__ void graph_back(int64_t E, const int32_t *__restrict__ edges, const int32_t *__restrict__ rp,
                           const int32_t *__restrict__ ci, int32_t *pos_bwd, int32_t *nz_edge) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= E) return;
  const int32_t v = edges[2 * e], w = edges[2 * e + 1];
  int lo = rp[w], hi = rp[w + 1];
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (ci[mid] < v) lo = mid + 1;
    else hi = mid;
  }
  pos_bwd[e] = lo;
  nz_edge[lo] = ~(int32_t)e;
}
__global__ void row_extents(int64_t N, const int32_t *__restrict__ rp, int *out) {
  const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int row = 0, block = 0;
  if (v < N) {
    row = rp[v + 1] - rp[v];
    if (v % 128 == 0) block = rp[min(N, v + 128)] - (rp[v] & ~3);
  }
  row = __reduce_max_sync(0xffffffffu, row);
  block = __reduce_max_sync(0xffffffffu, block);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(out, row);
    if (block > 0) atomicMax(out + 1, block);
  }
}

// ------------------------------------------------------------- geometry
struct V3 {
  double x, y, z;
};
__device__ __forceinline__ V3 ld3(const double *p) { return V3{p[0], p[1], p[2]}; }
__device__ __forceinline__ V3 operator-(V3 a, V3 b) { return V3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 operator+(V3 a, V3 b) { return V3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V3 operator*(double s, V3 a) { return V3{s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ double dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 cross(V3 a, V3 b) {
  return V3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ double norm(V3 a) { return sqrt(dot(a, a)); }

// In-place Cholesky solve of the SPD system A c = r (lower triangle of A, n <=
// 6), fully unrolled, the pivots' reciprocal roots instead of divisions.  The
// edge-coefficient matrix A_ij = (e_i . e_j)^2 is the Gram matrix of the
// rank-one tensors e_i e_i^T, SPD for a non-degenerate simplex.
template <int n>
__device__ __forceinline__ bool chol_solve(double (&A)[n][n], double (&r)[n]) {
  bool ok = true;
#pragma unroll
  for (int j = 0; j < n; j++) {
    double d = A[j][j];
#pragma unroll
    for (int k = 0; k < j; k++) d -= A[j][k] * A[j][k];
    ok = ok && d > 0.0;
    const double inv = rsqrt(d);
    A[j][j] = inv;
#pragma unroll
    for (int i = j + 1; i < n; i++) {
      double s = A[i][j];
#pragma unroll
      for (int k = 0; k < j; k++) s -= A[i][k] * A[j][k];
      A[i][j] = s * inv;
    }
  }
#pragma unroll
  for (int i = 0; i < n; i++) {
    double s = r[i];
#pragma unroll
    for (int k = 0; k < i; k++) s -= A[i][k] * r[k];
    r[i] = s * A[i][i];
  }
#pragma unroll
  for (int i = n - 1; i >= 0; i--) {
    double s = r[i];
#pragma unroll
    for (int k = i + 1; k < n; k++) s -= A[k][i] * r[k];
    r[i] = s * A[i][i];
  }
  return ok;
}

// Per simplex: edge coefficients (src/mesh_tri.cpp:107-151,
// src/mesh_tetra.cpp:107-160) times edge length, one value per local edge,
// and the control-volume share of each local vertex (circumcentric
// splitting, src/mesh.cpp:931-1027, src/mesh_tetra.cpp:196-331).
//
// The kernel is bound by FP64 instructions, so every quantity comes from the
// inner products of the edges.  In a triangle the signed distance
// of the circumcentre from edge e is |e| / 2 times the cotangent of the
// opposite angle, so an edge's share is |e|^2 cot / 8 to either end.  In a
// tetrahedron the piece of the dual face of edge e that lies in face F is the
// triangle of the edge's midpoint, F's circumcentre and the cell's: half of
// (|e| / 2) cot_F(e) times the signed height h_F of the cell's circumcentre
// over F, and with cot = (a . b) / |N|, h = (w . N) / |N| (N = F's normal,
// twice its area, towards the opposite vertex; w from F to the circumcentre)
// no square root is left: a share of |e|^2 / 24 (a . b) (w . N) / |N|^2 to
// either end.  486 FP64 instructions a warp, 1.37 ms at 64^3 (81 % of the FP64
// pipe's rate); with every circumcentre, norm and cross product formed as such
// 1962 and 5.46 ms.
template <int nvc>
__global__ void cell_geometry_kernel(int64_t T, const int32_t *__restrict__ cells, const double *__restrict__ x,
                                     double *__restrict__ coef_len, double *__restrict__ cv_part, int *err) {
  constexpr int ne = nvc == 3 ? 3 : 6;
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= T) return;
  V3 v[nvc];
#pragma unroll
  for (int k = 0; k < nvc; k++) v[k] = ld3(x + 3 * (int64_t)cells[nvc * c + k]);
  // edge vectors and their inner products (lower triangle); the first nvc - 1
  // edges are those at vertex 0
  V3 r[ne];
  double g[ne][ne];
#pragma unroll
  for (int i = 0; i < ne; i++) r[i] = v[pair1<nvc>(i)] - v[pair0<nvc>(i)];
#pragma unroll
  for (int i = 0; i < ne; i++)
#pragma unroll
    for (int j = 0; j <= i; j++) g[i][j] = dot(r[i], r[j]);
  // (v_a - v_b) . (v_a - v_c)
  auto ip = [&](int a, int b, int c) {
    const int p = edge_of<nvc>(a, b), q = edge_of<nvc>(a, c);
    const double d = g[p > q ? p : q][p > q ? q : p];
    return (a < b) == (a < c) ? d : -d;
  };
  double l2[ne];  // squared edge lengths
#pragma unroll
  for (int k = 0; k < ne; k++) l2[k] = g[k][k];
  double len[ne];
#pragma unroll
  for (int k = 0; k < ne; k++) len[k] = sqrt(l2[k]);
  double vol, t = 0.0, nn = 0.0;
  V3 n12, n20, n01;
  if (nvc == 3) {
    const V3 cr = cross(r[0], r[1]);
    nn = dot(cr, cr);
    vol = 0.5 * sqrt(nn);
    // degenerate triangle (the reference tests |omega| < 1e-10 absolutely,
    // src/mesh.cpp:917-927; a scale-free test keeps fine meshes valid)
    if (!(2.0 * nn > 1.0e-20 * (l2[0] * l2[2]))) atomicOr(err, 1);
  } else {
    n12 = cross(r[1], r[2]);
    n20 = cross(r[2], r[0]);
    n01 = cross(r[0], r[1]);
    t = dot(r[0], n12);
    // local edges 0,1,2 share local vertex 0: never coplanar
    if (fabs(t) / (len[0] * len[1] * len[2]) < 1.0e-5) atomicOr(err, 2);
    if (!(2.0 * fabs(t) > 1.0e-10 * (len[0] * len[1] * len[2]))) atomicOr(err, 8);
    vol = fabs(t) * (1.0 / 6.0);
  }
  double share[nvc];
#pragma unroll
  for (int k = 0; k < nvc; k++) share[k] = 0.0;
  if (nvc == 3) {
    // |e|^2 cot / 8, cot = (x_0 - o) . (x_1 - o) / (2 area)
    const double q = 0.125 / (2.0 * vol);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int e0 = pair0<3>(k), e1 = pair1<3>(k), o = 3 - e0 - e1;
      const double s = q * (l2[k] * ip(o, e0, e1));
      share[e0] += s;
      share[e1] += s;
    }
  } else {
    // circumcentre - v_0 (src/mesh_tetra.cpp:377-415)
    const double h = 0.5 / t;
    const V3 w = (g[0][0] * h) * n12 + (g[1][1] * h) * n20 + (g[2][2] * h) * n01;
    const double sg = t > 0.0 ? 1.0 : -1.0;
#pragma unroll
    for (int f = 0; f < 4; f++) {
      // face opposite vertex f, its normal towards f (t = r_0 . n12 > 0 for
      // the orientation below), w relative to one of its vertices
      V3 N;
      double wn;
      if (f == 0) {
        N = V3{-(n12.x + n20.x + n01.x), -(n12.y + n20.y + n01.y), -(n12.z + n20.z + n01.z)};
        wn = dot(w, N) + t;  // (w - r_0) . N, r_0 . N = -t
      } else {
        N = f == 1 ? n12 : f == 2 ? n20 : n01;
        wn = dot(w, N);
      }
      const double n2 = dot(N, N);
      const double q = sg * wn / (24.0 * n2);
      const int a = f == 0 ? 1 : 0, b = f <= 1 ? 2 : 1, d = f <= 2 ? 3 : 2;
      // edges (a,b), (a,d), (b,d) with the angles at d, b, a
      const double lab = l2[a == 0 ? b - 1 : a + b], lad = l2[a == 0 ? d - 1 : a + d], lbd = l2[b + d];
      if (!(2.0 * n2 > 1.0e-20 * (lbd * fmax(lab, lad)))) atomicOr(err, 1);
      const double sab = q * (lab * ip(d, a, b)), sad = q * (lad * ip(b, a, d)), sbd = q * (lbd * ip(a, b, d));
      share[a] += sab + sad;
      share[b] += sab + sbd;
      share[d] += sad + sbd;
    }
  }
#pragma unroll
  for (int k = 0; k < nvc; k++) cv_part[nvc * c + k] = share[k];
  double A[ne][ne], rhs[ne];
#pragma unroll
  for (int i = 0; i < ne; i++) {
    rhs[i] = vol * l2[i];
#pragma unroll
    for (int j = 0; j <= i; j++) A[i][j] = g[i][j] * g[i][j];
  }
  if (!chol_solve<ne>(A, rhs)) atomicOr(err, 4);
#pragma unroll
  for (int k = 0; k < ne; k++) coef_len[ne * c + k] = rhs[k] * len[k];
}

// Covolume of each edge: the coefficients of the cells around it, found among
// the cells incident to its end with fewer of them, in cell order (the order
// in which the reference accumulates; deterministic).  Bound by the latency of
// the cells' gathers: 0.34 ms at 64^3, without the lists of cells of each edge
// that the host took 25 ms to make.
template <int nvc>
__global__ void edge_covolumes(int64_t E, const int32_t *__restrict__ edges, const int32_t *__restrict__ cells,
                               const int32_t *__restrict__ ptr, const int32_t *__restrict__ vc,
                               const double *__restrict__ coef_len, double *__restrict__ covol) {
  constexpr int ne = nvc == 3 ? 3 : 6;
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= E) return;
  int32_t v = edges[2 * e], w = edges[2 * e + 1];
  if (ptr[w + 1] - ptr[w] < ptr[v + 1] - ptr[v]) {
    const int32_t t = v;
    v = w, w = t;
  }
  double s = 0.0;
  for (int j = ptr[v]; j < ptr[v + 1]; j++) {
    const int32_t k = vc[j], c = k / nvc, a = k - c * nvc;
#pragma unroll
    for (int b = 0; b < nvc; b++)
      if (cells[(int64_t)nvc * c + b] == w) s += coef_len[(int64_t)ne * c + edge_of<nvc>(a, b)];
  }
  covol[e] = s;
}

// out[v] = sum of the vertex's shares in cell order
__global__ void vertex_sum(int64_t N, const int32_t *__restrict__ ptr, const int32_t *__restrict__ vc,
                           const double *__restrict__ src, double *__restrict__ out) {
  const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (v >= N) return;
  double s = 0.0;
  for (int j = ptr[v]; j < ptr[v + 1]; j++) s += src[vc[j]];
  out[v] = s;
}

__global__ void edge_length_kernel(int64_t E, const int32_t *__restrict__ edges,
                                   const double *__restrict__ x,
                                   double *__restrict__ len) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= E) return;
  const V3 d = ld3(x + 3 * (int64_t)edges[2 * e]) - ld3(x + 3 * (int64_t)edges[2 * e + 1]);
  len[e] = norm(d);
}

}  // namespace

// ------------------------------------------------------------------------
void MeshImpl::validate(int64_t n_vertices, const int32_t *cells, int64_t n_cells,
                        int verts_per_cell) {
  NOSH_CHECK(verts_per_cell == 3 || verts_per_cell == 4, NOSH_ERR_INVALID,
             "verts_per_cell must be 3 (triangles) or 4 (tetrahedra)");
  NOSH_CHECK(n_vertices > 0 && n_cells > 0, NOSH_ERR_INVALID, "empty mesh");
  NOSH_CHECK(n_cells * verts_per_cell < (int64_t)1 << 31 && n_vertices < (int64_t)1 << 30,
             NOSH_ERR_INVALID, "mesh too large for 32-bit indices");
  const int nvc = verts_per_cell;
  // one pass without branches over everything, on the host's cores when the
  // mesh is large; only a bad mesh is gone through again for its first fault
  std::atomic<int> bad{0};
  parallel_ranges(n_cells, 1 << 17, [&](int64_t b, int64_t e) {
    unsigned f = 0;
    for (int64_t k = nvc * b; k < nvc * e; k++) f |= (unsigned)((uint32_t)cells[k] >= (uint32_t)n_vertices);
    if (nvc == 3) {
      for (int64_t c = b; c < e; c++) {
        const int32_t *q = cells + 3 * c;
        f |= (unsigned)((q[0] == q[1]) | (q[0] == q[2]) | (q[1] == q[2]));
      }
    } else {
      for (int64_t c = b; c < e; c++) {
        const int32_t *q = cells + 4 * c;
        f |= (unsigned)((q[0] == q[1]) | (q[0] == q[2]) | (q[0] == q[3]) | (q[1] == q[2]) | (q[1] == q[3]) |
                        (q[2] == q[3]));
      }
    }
    if (f) bad.store(1);
  });
  if (!bad.load()) return;
  for (int64_t k = 0; k < nvc * n_cells; k++)
    NOSH_CHECK(cells[k] >= 0 && cells[k] < n_vertices, NOSH_ERR_INVALID,
               "cell vertex index out of range at entry " + std::to_string(k));
  for (int64_t c = 0; c < n_cells; c++)
    for (int a = 0; a < nvc; a++)
      for (int b = a + 1; b < nvc; b++)
        NOSH_CHECK(cells[nvc * c + a] != cells[nvc * c + b], NOSH_ERR_MESH,
                   "cell " + std::to_string(c) + " repeats a vertex");
}

MeshImpl::MeshImpl(const double *coords, int64_t n_vertices, const int32_t *cells_in,
                   int64_t n_cells, int verts_per_cell) {
  // the description has passed validate() (nosh_mesh_create runs it before
  // it looks for a device): one pass over the cells, not two
  nvc = verts_per_cell;
  ne = nvc == 3 ? 3 : 6;
  N = n_vertices;
  T = n_cells;
  NOSH_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
  try {
    build(coords, cells_in);
  } catch (...) {
    // a throwing constructor runs no destructor: release the stream here
    // (the device buffers free themselves)
    cudaStreamSynchronize(stream);
    cudaStreamDestroy(stream);
    stream = nullptr;
    throw;
  }
}

MeshImpl::~MeshImpl() {
  if (stream) cudaStreamDestroy(stream);
}

namespace {
// exclusive scan of in[0..n) into out[0..n] on the stream; the total is left
// in tile[number of tiles]
int64_t scan(int64_t n, const int32_t *in, int32_t *out, int64_t *tile, cudaStream_t s) {
  const int64_t nt = div_up(n, kScanTile);
  scan_tiles<<<(unsigned)nt, kScanTile, 0, s>>>(n, in, tile);
  scan_sums<<<1, kScanTile, 0, s>>>(nt, tile);
  scan_write<<<(unsigned)nt, kScanTile, 0, s>>>(n, in, tile, out);
  return nt;
}
inline int wide_grid(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>(div_up(n, 256), 16 * kNumSMs)); }

// The vertices with too many cells for the warp kernel: their codes are sorted
// and their neighbours found on the host's cores, all hubs in one copy out and
// one back.  A mesh of 10000 fans of 100 triangles 6.2 ms; 350 with the hubs one
// after the other, each with copies and waits of its own, and 45 with all of the
// topology on the host's cores.  One fan 0.39 ms (0.35).
struct Hubs {
  DevBuf<int32_t> off, codes, nb, deg, up;  // hub h: codes [off[h], off[h + 1])
};
__global__ void hub_sizes(int64_t nh, const int32_t *__restrict__ hubs, const int32_t *__restrict__ ptr,
                          int32_t *size) {
  const int64_t h = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (h < nh) size[h] = ptr[hubs[h] + 1] - ptr[hubs[h]];
}
// a CTA per hub
__global__ void hub_gather(const int32_t *__restrict__ hubs, const int32_t *__restrict__ ptr,
                           const int32_t *__restrict__ vc, const int32_t *__restrict__ off, int32_t *codes) {
  const int b = ptr[hubs[blockIdx.x]], o = off[blockIdx.x], d = off[blockIdx.x + 1] - o;
  for (int q = threadIdx.x; q < d; q += blockDim.x) codes[o + q] = vc[b + q];
}
__global__ void hub_scatter(int nvc, const int32_t *__restrict__ hubs, const int32_t *__restrict__ ptr,
                            const int32_t *__restrict__ off, const int32_t *__restrict__ codes,
                            const int32_t *__restrict__ hub_nb, const int32_t *__restrict__ hub_deg,
                            const int32_t *__restrict__ hub_up, int32_t *vc, int32_t *nb, int32_t *deg, int32_t *up) {
  const int v = hubs[blockIdx.x], b = ptr[v], o = off[blockIdx.x], d = off[blockIdx.x + 1] - o, m = hub_deg[blockIdx.x];
  for (int q = threadIdx.x; q < d; q += blockDim.x) vc[b + q] = codes[o + q];
  for (int q = threadIdx.x; q < m; q += blockDim.x)
    nb[(int64_t)(nvc - 1) * b + q] = hub_nb[(int64_t)(nvc - 1) * o + q];
  if (threadIdx.x == 0) {
    deg[v] = m;
    up[v] = hub_up[blockIdx.x];
  }
}
void solve_hubs(int nvc, const int32_t *cells, int nh, const DevBuf<int32_t> &hubs, const DevBuf<int32_t> &ptr,
                DevBuf<int32_t> &vc, DevBuf<int32_t> &nb, DevBuf<int32_t> &deg, DevBuf<int32_t> &up, cudaStream_t s) {
  std::vector<int32_t> hv(nh), off(nh + 1, 0), h_deg(nh), h_up(nh);
  Hubs D;
  D.deg.alloc(nh);
  D.up.alloc(nh);
  D.off.alloc(nh + 1);
  hub_sizes<<<div_up(nh, 256), 256, 0, s>>>(nh, hubs.p, ptr.p, D.deg.p);
  NOSH_CUDA(cudaGetLastError());
  hubs.download(hv.data(), nh, s);
  D.deg.download(off.data() + 1, nh, s);
  NOSH_CUDA(cudaStreamSynchronize(s));
  for (int h = 0; h < nh; h++) off[h + 1] += off[h];  // (at most the codes of all vertices: 32 bits)
  const int64_t total = off[nh];
  std::vector<int32_t> codes(total), adj((nvc - 1) * total);
  D.codes.alloc(total);
  D.nb.alloc((nvc - 1) * total);
  D.off.upload(off, s);
  hub_gather<<<nh, 128, 0, s>>>(hubs.p, ptr.p, vc.p, D.off.p, D.codes.p);
  NOSH_CUDA(cudaGetLastError());
  D.codes.download(codes.data(), total, s);
  NOSH_CUDA(cudaStreamSynchronize(s));
  parallel_ranges(nh, 16, [&](int64_t h0, int64_t h1) {
    for (int64_t h = h0; h < h1; h++) {
      const int32_t v = hv[h];
      std::sort(codes.begin() + off[h], codes.begin() + off[h + 1]);
      int32_t *u = adj.data() + (int64_t)(nvc - 1) * off[h], *e = u;
      for (int32_t k = off[h]; k < off[h + 1]; k++)
        for (int q = 0; q < nvc; q++) {
          const int32_t w = cells[(int64_t)(codes[k] / nvc) * nvc + q];
          if (w != v) *e++ = w;
        }
      std::sort(u, e);
      e = std::unique(u, e);
      h_deg[h] = (int32_t)(e - u);
      h_up[h] = (int32_t)(e - std::upper_bound(u, e, v));
    }
  });
  D.codes.upload(codes, s);
  D.nb.upload(adj, s);
  D.deg.upload(h_deg, s);
  D.up.upload(h_up, s);
  hub_scatter<<<nh, 128, 0, s>>>(nvc, hubs.p, ptr.p, D.off.p, D.codes.p, D.nb.p, D.deg.p, D.up.p, vc.p, nb.p, deg.p,
                                 up.p);
  NOSH_CUDA(cudaGetLastError());
  NOSH_CUDA(cudaStreamSynchronize(s));
}
}  // namespace

void MeshImpl::build(const double *coords, const int32_t *cells) {
  cudaStream_t s = stream;
  const int64_t nk = nvc * T;
  slab_vertices.want(d_x, 3 * N);
  slab_vertices.want(d_rp, N + 1);
  slab_vertices.want(d_cv, N);
  slab_vertices.commit();
  DevBuf<double> coef_len, cv_part;
  DevBuf<int> flags;  // geometry errors, hubs, longest row, longest row block
  DevBuf<int32_t> d_cells, cnt, ptr, vc, nb, deg, up, hubs, ebase;
  DevBuf<int64_t> tile;
  DevSlab tmp;
  tmp.want(coef_len, ne * T);
  tmp.want(cv_part, nk);
  tmp.want(flags, 4);
  tmp.want(d_cells, nk);
  for (DevBuf<int32_t> *b : {&cnt, &deg, &up, &hubs}) tmp.want(*b, N);
  for (DevBuf<int32_t> *b : {&ptr, &ebase}) tmp.want(*b, N + 1);
  tmp.want(vc, nk);
  tmp.want(nb, (nvc - 1) * nk);
  tmp.want(tile, div_up(N, kScanTile) + 1);
  tmp.commit();
  d_cells.upload(cells, nk, s);
  d_x.upload(coords, 3 * N, s);
  // geometry of the cells
  flags.zero(s);
  const int B = 128;
  if (nvc == 3)
    cell_geometry_kernel<3><<<div_up(T, B), B, 0, s>>>(T, d_cells.p, d_x.p, coef_len.p, cv_part.p, flags.p);
  else
    cell_geometry_kernel<4><<<div_up(T, B), B, 0, s>>>(T, d_cells.p, d_x.p, coef_len.p, cv_part.p, flags.p);
  // vertex -> (cell, slot) incidence and neighbours
  cnt.zero(s);
  count_incident<<<wide_grid(nk), 256, 0, s>>>(nk, d_cells.p, cnt.p);
  scan(N, cnt.p, ptr.p, tile.p, s);
  NOSH_CUDA(cudaMemcpyAsync(cnt.p, ptr.p, N * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
  scatter_incident<<<wide_grid(nk), 256, 0, s>>>(nk, d_cells.p, cnt.p, vc.p);
  const int ng = (int)std::min<int64_t>(div_up(N, kNbWarps), 1 << 20);
  if (nvc == 3)
    neighbour_kernel<3><<<ng, 32 * kNbWarps, 0, s>>>(N, d_cells.p, ptr.p, vc.p, nb.p, deg.p, up.p, hubs.p,
                                                     flags.p + 1);
  else
    neighbour_kernel<4><<<ng, 32 * kNbWarps, 0, s>>>(N, d_cells.p, ptr.p, vc.p, nb.p, deg.p, up.p, hubs.p,
                                                     flags.p + 1);
  NOSH_CUDA(cudaGetLastError());
  int h[4] = {0, 0, 0, 0};
  flags.download(h, 2, s);
  NOSH_CUDA(cudaStreamSynchronize(s));
  NOSH_CHECK(h[0] == 0, NOSH_ERR_MESH, "degenerate cell(s) in the mesh (flags " + std::to_string(h[0]) + ")");
  if (h[1] > 0) solve_hubs(nvc, cells, h[1], hubs, ptr, vc, nb, deg, up, s);
  // row pointers and first edges
  int64_t total[2];
  NOSH_CUDA(cudaMemcpyAsync(&total[0], tile.p + scan(N, deg.p, d_rp.p, tile.p, s), sizeof(int64_t),
                            cudaMemcpyDeviceToHost, s));
  NOSH_CUDA(cudaMemcpyAsync(&total[1], tile.p + scan(N, up.p, ebase.p, tile.p, s), sizeof(int64_t),
                            cudaMemcpyDeviceToHost, s));
  row_extents<<<div_up(N, 256), 256, 0, s>>>(N, d_rp.p, flags.p + 2);
  flags.download(h, 4, s);
  NOSH_CUDA(cudaStreamSynchronize(s));
  NOSH_CHECK(total[0] < (int64_t)1 << 31, NOSH_ERR_INVALID, "too many edges");
  E = total[1];
  max_row = h[2];
  max_block = h[3];
  // column indices padded by kPad entries so that 128-bit staged loads of a
  // row block may run past its end
  slab_edges.want(d_ci, 2 * E + kPad);
  slab_edges.want(d_edges, 2 * E);
  slab_edges.want(d_pos_fwd, E);
  slab_edges.want(d_pos_bwd, E);
  slab_edges.want(d_nz_edge, 2 * E);
  slab_edges.want(d_len, E);
  slab_edges.want(d_covol, E);
  slab_edges.commit();
  NOSH_CUDA(cudaMemsetAsync(d_ci.p + 2 * E, 0, kPad * sizeof(int32_t), s));
  graph_rows<<<div_up(16 * N, 256), 256, 0, s>>>(N, nvc, ptr.p, nb.p, d_rp.p, up.p, ebase.p, d_ci.p, d_edges.p,
                                                 d_pos_fwd.p, d_nz_edge.p);
  graph_back<<<div_up(E, 256), 256, 0, s>>>(E, d_edges.p, d_rp.p, d_ci.p, d_pos_bwd.p, d_nz_edge.p);
  edge_length_kernel<<<div_up(E, 256), 256, 0, s>>>(E, d_edges.p, d_x.p, d_len.p);
  if (nvc == 3)
    edge_covolumes<3><<<div_up(E, 256), 256, 0, s>>>(E, d_edges.p, d_cells.p, ptr.p, vc.p, coef_len.p, d_covol.p);
  else
    edge_covolumes<4><<<div_up(E, 256), 256, 0, s>>>(E, d_edges.p, d_cells.p, ptr.p, vc.p, coef_len.p, d_covol.p);
  vertex_sum<<<div_up(N, 256), 256, 0, s>>>(N, ptr.p, vc.p, cv_part.p, d_cv.p);
  NOSH_CUDA(cudaGetLastError());
  NOSH_CUDA(cudaStreamSynchronize(s));
}

void MeshImpl::complex_graph(int32_t *row_ptr, int32_t *cols) {
  const std::vector<int32_t> &rp = this->rp(), &ci = this->ci();
  row_ptr[0] = 0;
  for (int64_t v = 0; v < N; v++) {
    const int64_t b = rp[v], e = rp[v + 1], o = row_ptr[v];
    int64_t k = 0;
    bool placed = false;
    for (int64_t q = b; q < e; q++) {
      if (!placed && ci[q] > v) {
        cols[o + k++] = (int32_t)v;
        placed = true;
      }
      cols[o + k++] = ci[q];
    }
    if (!placed) cols[o + k++] = (int32_t)v;
    row_ptr[v + 1] = (int32_t)(o + k);
  }
}

}  // namespace nosh
