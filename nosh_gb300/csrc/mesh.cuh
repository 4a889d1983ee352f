// Mesh handle: device geometry and KEO graph, host copies on demand.
#pragma once

#include <mutex>

#include "common.cuh"

namespace nosh {

struct MeshImpl {
  int nvc = 0, ne = 0;  // vertices / edges per cell
  int64_t N = 0, E = 0, T = 0;
  cudaStream_t stream = nullptr;
  // the longest row of the off-diagonal KEO graph, and the longest 4-aligned
  // range of nonzeros of 128 consecutive rows from a multiple of 128
  int max_row = 0, max_block = 0;

  DevSlab slab_vertices, slab_edges;  // memory of the buffers below
  // device: coordinates, edges (v0 < v1, lexicographic), geometry, the
  // off-diagonal KEO graph (row v: its sorted neighbours), each nonzero's edge
  // (~e if the row is v1), the nonzeros of (v0, v1) and (v1, v0) of each edge
  DevBuf<double> d_x, d_len, d_covol, d_cv;
  DevBuf<int32_t> d_edges;
  DevBuf<int32_t> d_rp, d_ci, d_nz_edge, d_pos_fwd, d_pos_bwd;

  // expects a description that validate() accepted
  MeshImpl(const double *coords, int64_t n_vertices, const int32_t *cells,
           int64_t n_cells, int verts_per_cell);
  ~MeshImpl();
  // host-only checks of a mesh description (sizes, cell type, every vertex
  // index in range, no cell repeating a vertex); throws nosh::Error
  static void validate(int64_t n_vertices, const int32_t *cells, int64_t n_cells,
                       int verts_per_cell);
  MeshImpl(const MeshImpl &) = delete;
  MeshImpl &operator=(const MeshImpl &) = delete;

  // host copies, fetched from the device on first use (a mesh may serve
  // several handles and threads)
  const std::vector<int32_t> &edges() { return fetch(h_edges_, d_edges, 2 * E); }
  const std::vector<int32_t> &rp() { return fetch(h_rp_, d_rp, N + 1); }
  const std::vector<int32_t> &ci() { return fetch(h_ci_, d_ci, 2 * E); }
  const std::vector<double> &len() { return fetch(h_len_, d_len, E); }
  // a caller's own copy
  template <typename V>
  void read(V *out, const DevBuf<V> &d, int64_t n) {
    NOSH_CUDA(cudaMemcpyAsync(out, d.p, n * sizeof(V), cudaMemcpyDeviceToHost, stream));
    NOSH_CUDA(cudaStreamSynchronize(stream));
  }

  // complex graph with the diagonal (row_ptr[N+1], cols[N+2E])
  void complex_graph(int32_t *row_ptr, int32_t *cols);

 private:
  std::mutex fetch_mtx_;
  std::vector<int32_t> h_edges_, h_rp_, h_ci_;
  std::vector<double> h_len_;
  template <typename V>
  const std::vector<V> &fetch(std::vector<V> &h, const DevBuf<V> &d, int64_t n) {
    std::lock_guard<std::mutex> lock(fetch_mtx_);
    if ((int64_t)h.size() != n) {
      std::vector<V> v(n);
      read(v.data(), d, n);
      h.swap(v);
    }
    return h;
  }
  void build(const double *coords, const int32_t *cells);
};

}  // namespace nosh
