// ogs_scatter.cuh -- Scatter in node order.
//
// v[n] = gv[row(n)] (ogsOperator.cpp:206-238) is a copy, so it needs no row
// lists: a warp takes consecutive nodes, finds each node's row and writes the
// nodes as one run.  Rows are numbered by first member (ogs_setup), so the
// rows of the first members among 32 nodes are consecutive: a bit word and one
// row number give them all, and only the other members carry a row number of
// their own.  Against writing through the rows' column lists this reads 4
// bytes for each of the nnz - R other members and half a byte a node instead
// of 4 (nnz + R) bytes, and the field's stores fill whole sectors.  What bounds
// it is bandwidth: 24^3 p=7 fp64 moves 38.6 MB of gathered values, 56.6 MB of
// field and 11 MB of rows and words in 20.9 us (28.3 us through the column
// lists), p=15 875 MB in 152 us (257), 32x32x16 p=5 permuted fp32 k=3 13.3 us
// (20.5).  k is a constant: with k from 5 up as a number given at the launch,
// every word took eight runs and a division, 20^3 p=7 fp64 k=5 82.7 us and k=8
// 111.6 against 58.4 and 79.6 through the column lists; now 24^3 p=7 k=5 85.0
// (101.6 through the lists) and k=8 130.1 (133.8).
#pragma once

#include <cstdint>

#include "ogs_kernels.cuh"

namespace ogsgb {

// Threads of a CTA: 256, or 64 where that makes fewer than kScatterCtas CTAs
// (3.4 an SM), since a small mesh leaves SMs idle and CTAs of 64 for 7 M nodes
// take as long as 55 k CTAs need to start.  CTAs of 256 / of 64 / through the
// column lists, us: fp64 k=2 10^3 p=3 (64 k nodes) 3.00 / 2.85 / 2.87, k=4 2.96 /
// 2.75 / 2.69, k=1 2.97 / 2.90 / 2.87, 24^3 p=3 4.23 / 4.16 / 4.64; the other
// way fp32 k=1 24^3 p=7 10.8 / 14.7, k=3 16^3 p=3 (512 CTAs) 2.75 / 2.87, 24^3
// p=7 34.9 / 56.5.
constexpr int kScatterBlock = 256, kScatterSmallBlock = 64;
constexpr int64_t kScatterCtas = 512;

// Words of 32 nodes a warp takes for K components, all their loads in flight at
// once: about eight runs of 32 values.
OGS_HD constexpr int scatter_words(int K) { return K == 1 ? 8 : K == 2 ? 4 : K <= 4 ? 2 : 1; }

// The 32 nodes of a word hold 32 K consecutive values: a lane first finds the
// row of one node, then writes values lane, lane + 32, ... with the rows of
// their nodes from the other lanes.  NONLY: writes N members only (Trans).
template <typename T, int K, bool NONLY, int BLOCK>
__global__ void __launch_bounds__(BLOCK) ogs_scatter_kernel(const DevNodes m, T* v, const T* gv, const int32_t nrows,
                                                            unsigned int* err, const int release) {
  constexpr int W = scatter_words(K);
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int64_t w0 = (static_cast<int64_t>(blockIdx.x) * (BLOCK / 32) + (threadIdx.x >> 5)) * W;
  if (w0 >= m.nwords) {
    grid_wait(release);
    return;
  }
  NodeWord w[W];
#pragma unroll
  for (int j = 0; j < W; ++j) w[j] = m.words[w0 + j];  // (padded to whole items)
  int32_t r[W];  // -1: takes no part
#pragma unroll
  for (int j = 0; j < W; ++j) {
    const uint32_t bit = 1u << lane;
    r[j] = -1;
    if (w[j].first & bit) r[j] = w[j].row0 + __popc(w[j].first & (bit - 1u));
    else if (w[j].other & bit) r[j] = __ldg(m.orow + w[j].other0 + __popc(w[j].other & (bit - 1u)));
    if (r[j] >= 0) r[j] = checked_id(r[j], nrows, err);
    if (NONLY && !((m.nmem[w0 + j] >> lane) & 1u)) r[j] = -1;
  }
  grid_wait(release);
  T x[W][K];
  int32_t row[W][K];
#pragma unroll
  for (int j = 0; j < W; ++j)
#pragma unroll
    for (int q = 0; q < K; ++q) {
      const uint32_t u = static_cast<uint32_t>(q * 32 + lane);
      const uint32_t n = u / K;
      row[j][q] = K == 1 ? r[j] : __shfl_sync(0xffffffffu, r[j], n & 31);
      if (row[j][q] >= 0) x[j][q] = gv[static_cast<int64_t>(row[j][q]) * K + (u - n * K)];
    }
#pragma unroll
  for (int j = 0; j < W; ++j)
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (row[j][q] >= 0) v[(w0 + j) * 32 * K + q * 32 + lane] = x[j][q];
}

template <int K>
inline int64_t scatter_ctas(int64_t nwords, int block) {
  const int64_t per_block = scatter_words(K) * (block / 32);
  return (nwords + per_block - 1) / per_block;
}

template <typename T, int K, bool NONLY, int BLOCK>
inline cudaError_t launch_scatter_block(const DevMaps& m, const FieldArgs& f, cudaStream_t s) {
  const dim3 grid(static_cast<unsigned>(scatter_ctas<K>(m.nodes.nwords, BLOCK)));
  launch_overlapped(ogs_scatter_kernel<T, K, NONLY, BLOCK>, grid, BLOCK, 0, s, f.overlap, m.nodes, static_cast<T*>(f.v),
                    static_cast<const T*>(f.gv), m.b[1].nrows, m.b[1].err, f.overlap);
  return cudaGetLastError();
}

template <typename T, int K, bool NONLY>
inline cudaError_t launch_scatter_as(const DevMaps& m, const FieldArgs& f, cudaStream_t s) {
  if (scatter_ctas<K>(m.nodes.nwords, kScatterBlock) < kScatterCtas)
    return launch_scatter_block<T, K, NONLY, kScatterSmallBlock>(m, f, s);
  return launch_scatter_block<T, K, NONLY, kScatterBlock>(m, f, s);
}

// The instantiation of f.K components, from K down.
template <typename T, bool NONLY, int K>
inline cudaError_t launch_scatter_k(const DevMaps& m, const FieldArgs& f, cudaStream_t s) {
  if constexpr (K > 1) {
    if (f.K < K) return launch_scatter_k<T, NONLY, K - 1>(m, f, s);
  }
  return launch_scatter_as<T, K, NONLY>(m, f, s);
}

template <typename T>
inline cudaError_t launch_scatter(const DevMaps& m, const FieldArgs& f, const Pattern& pat, cudaStream_t s) {
  constexpr int K = scatter_max_k(sizeof(T));
  return pat.scatter_n ? launch_scatter_k<T, true, K>(m, f, s) : launch_scatter_k<T, false, K>(m, f, s);
}

}  // namespace ogsgb
