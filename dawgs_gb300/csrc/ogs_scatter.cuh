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
// field and 11 MB of rows and words in 21.5 us (28.7 us through the column
// lists), p=15 875 MB in 152 us (257), 32x32x16 p=5 permuted fp32 k=3 13.3 us
// (20.5).
#pragma once

#include <cstdint>

#include "ogs_kernels.cuh"

namespace ogsgb {

constexpr int kScatterBlock = 256;

// Words of 32 nodes a warp takes for KC components (0: any number), all their
// loads in flight at once: about eight runs of 32 values.
OGS_HD constexpr int scatter_words(int KC) { return KC == 1 ? 8 : KC == 2 ? 4 : KC == 0 ? 1 : 2; }

// KC: the components when they are few, else 0.  The 32 nodes of a word hold
// 32 K consecutive values: a lane first finds the row of one node, then
// writes values lane, lane + 32, ... with the rows of their nodes from the
// other lanes.  NONLY: writes N members only (Trans).
template <typename T, int KC, bool NONLY>
__global__ void __launch_bounds__(kScatterBlock) ogs_scatter_kernel(const DevNodes m, T* v, const T* gv,
                                                                    const int K_in, const uint32_t kmagic,
                                                                    const int32_t nrows, unsigned int* err) {
  constexpr int W = scatter_words(KC);
  constexpr int B = KC ? KC : 8;  // runs of a word in flight
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int64_t w0 = (static_cast<int64_t>(blockIdx.x) * (kScatterBlock / 32) + (threadIdx.x >> 5)) * W;
  grid_release();
  if (w0 >= m.nwords) {
    grid_wait();
    return;
  }
  const int K = KC ? KC : K_in;
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
  grid_wait();
  for (int p0 = 0; p0 < K; p0 += B) {
    T x[W][B];
    int32_t row[W][B];
#pragma unroll
    for (int j = 0; j < W; ++j)
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const uint32_t u = static_cast<uint32_t>(p0 + q) * 32u + static_cast<uint32_t>(lane);
        uint32_t n = u;
        if (KC == 0) n = kmagic ? __umulhi(u, kmagic) : u / static_cast<uint32_t>(K);
        else if (KC > 1) n = u / KC;
        row[j][q] = KC == 1 ? r[j] : __shfl_sync(0xffffffffu, r[j], n & 31);
        if (KC == 0 && p0 + q >= K) row[j][q] = -1;
        if (row[j][q] >= 0) x[j][q] = gv[static_cast<int64_t>(row[j][q]) * K + (u - n * K)];
      }
#pragma unroll
    for (int j = 0; j < W; ++j)
#pragma unroll
      for (int q = 0; q < B; ++q)
        if (row[j][q] >= 0) v[(w0 + j) * 32 * K + (p0 + q) * 32 + lane] = x[j][q];
  }
}

// Whether a Scatter runs in node order: wherever the handle has the node words
// (rows numbered by first member).  It was faster at every size and k measured
// (24^3 p=3 k=8 permuted 13.8 us against 15.9, 48^3 p=2 permuted 11.3 against
// 15.3) but the smallest, where both are one chain of loads (10^3 p=3: 4.1
// against 3.6 us, at a timer step of 0.5).  Operators over caller maps and the
// slices of host-buffer calls keep the tile kernels.
inline bool scatter_applies(const DevMaps& m, const FieldArgs& f, const Pattern& pat) {
  return m.nodes.nwords > 0 && !f.is_many && !pat.gslib && pat.scatter_n <= 1;
}

template <typename T, int KC, bool NONLY>
inline cudaError_t launch_scatter_as(const DevMaps& m, const FieldArgs& f, cudaStream_t s) {
  constexpr int64_t per_block = scatter_words(KC) * (kScatterBlock / 32);
  const unsigned grid = static_cast<unsigned>((m.nodes.nwords + per_block - 1) / per_block);
  // division by K as a multiply-high, exact while (32 K) K < 2^32
  const uint32_t kmagic = f.K < 11585 ? 0xFFFFFFFFu / static_cast<uint32_t>(f.K) + 1u : 0u;
  return launch_overlapped(ogs_scatter_kernel<T, KC, NONLY>, dim3(grid), kScatterBlock, 0, s, f.overlap, m.nodes,
                           static_cast<T*>(f.v), static_cast<const T*>(f.gv), f.K, kmagic, m.b[1].nrows, m.b[1].err);
}

template <typename T, bool NONLY>
inline cudaError_t launch_scatter_k(const DevMaps& m, const FieldArgs& f, cudaStream_t s) {
  switch (f.K) {
    case 1: return launch_scatter_as<T, 1, NONLY>(m, f, s);
    case 2: return launch_scatter_as<T, 2, NONLY>(m, f, s);
    case 3: return launch_scatter_as<T, 3, NONLY>(m, f, s);
    case 4: return launch_scatter_as<T, 4, NONLY>(m, f, s);
    default: return launch_scatter_as<T, 0, NONLY>(m, f, s);
  }
}

template <typename T>
inline cudaError_t launch_scatter(const DevMaps& m, const FieldArgs& f, const Pattern& pat, cudaStream_t s) {
  return pat.scatter_n ? launch_scatter_k<T, true>(m, f, s) : launch_scatter_k<T, false>(m, f, s);
}

}  // namespace ogsgb
