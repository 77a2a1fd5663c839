// ogs_wide.cuh -- rows above degree 8, a lane a row.
//
// The reference folds such a row like any other (ogsOperator.cpp:60-97,
// 206-238, 311-360), in ascending member order.  What bounds it is latency and
// the requests of members that lie in as many sectors.  The column ids of 32
// consecutive rows are laid out member by member (a coalesced load each), a
// lane has up to 24 members in flight, and k components are split over a
// tile's k parts as in ogs_async.cuh.  Before, a CTA took up to 256 rows
// through their CSR lists, a thread a row and one load after the other, all
// components in turn.  GatherScatter fp64, vertices of degree 24, us a call
// before and now: 64^3 cells of six p=1 tetrahedra 72.0 -> 59.3, 20x20x16 of
// p=3 with k=3 26.0 -> 15.1, 24^3 of p=2 in 4 arrays 43.0 -> 31.2, 32x32x24 of
// p=3 25.5 -> 24.8.  Slower forms: four lanes a row with the members passed by
// shuffles (an fp64 add costs a warp 16 cycles of its pipe whatever lanes take
// part), and the tiles at the head of the launch of the exact-degree rows (28-34
// us in the last case, and that kernel 3 % slower where there are none).
#pragma once

#include <algorithm>
#include <cstdint>

#include "ogs_kernels.cuh"

namespace ogsgb {

// Members a lane has in flight: 24, or 12 where the general rows have up to 12 on
// average (DevMaps::wide_short).  With 24, 2,432 tiles run at once and more of
// them take turns; with 12 it is 4,256.  1 M nodes in rows of one degree, us with
// a thread a row as before this kernel / with 24 / with 12, fp64 k=1, the members
// drawn at random and from as many blocks of nodes: degree 9 12.5 / 17.0 / 9.9 and
// 6.3 / 9.6 / 5.6, degree 12 11.9 / 17.0 / 9.8 and 6.4 / 9.1 / 5.3, degree 13 12.1
// / 12.1 / 12.3 and 6.7 / 6.8 / 7.3, degree 25 13.8 / 14.5 / 13.9 and 8.8 / 8.3 /
// 7.2, degree 48 15.7 / 13.5 / 14.5 and 11.1 / 7.5 / 8.4, degree 128 24.6 / 22.5 /
// 23.8 and 21.1 / 15.5 / 16.6; the vertices of p=3 tetrahedra 18.8 / 18.0 / 18.4,
// of p=1 11.9 / 11.1 / 12.6.  (Rows of 1,000 drawn at random stay slower than with
// a thread a row, 142 us against 130; from blocks 104 against 139.)
constexpr int kWideLong = 24, kWideShort = 12;
constexpr int kWideBlock = 64;  // small CTAs, so that a few hundred tiles reach every SM

// The ids of B members from q0 on of a row, none past the tile's degree d.
template <int B>
__device__ __forceinline__ void load_wide_ids(const uint32_t* ids, int q0, int d, uint32_t (&id)[B]) {
#pragma unroll
  for (int q = 0; q < B; ++q) id[q] = q0 + q < d ? __ldg(ids + (q0 + q) * 32) : kNoWideId;
}

// One work item: component k of row rl of wide tile `t`, B members in flight.
template <typename T, int OP, int MODE, int B>
__device__ __forceinline__ void wide_tile(const DevMaps& m, const FieldArgs& f, const Pattern& pat, int t, int rl,
                                          int k, int K, int64_t stride) {
  const Tile w = m.wide[t];
  if (rl >= w.count || (pat.limit_n && w.begin + rl >= m.g.nP)) return;
  const uint32_t* ids = m.wide_ids + static_cast<int64_t>(w.first_row) * 32 + rl;
  const int d = w.bucket;
  const int64_t r = MODE == kModeGS ? 0 : checked_id(__ldg(m.g.rows + w.begin + rl), m.g.nrows, m.g.err);
  T a;
  if (MODE == kModeScatter) {
    a = static_cast<const T*>(f.gv)[r * K + k];
  } else {
    const T* src = field_base<T>(f, k);
    a = op_init<T, OP>();
    uint32_t id[B], nxt[B];
    load_wide_ids<B>(ids, 0, d, id);
    for (int q0 = 0; q0 < d; q0 += B) {
      T x[B];
      if (B == kWideLong && q0) load_wide_ids<B>(ids, q0, d, id);
#pragma unroll
      for (int q = 0; q < B; ++q) {
        if (pat.gather_n && !(id[q] >> 31)) id[q] = kNoWideId;
        if (id[q] != kNoWideId)
          x[q] = src[static_cast<int64_t>(checked_id(id[q] & 0x7FFFFFFFu, m.g.nnodes, m.g.err)) * stride];
      }
      // (the short form has registers left for the ids of the next batch)
      if (B == kWideShort && q0 + B < d) load_wide_ids<B>(ids, q0 + B, d, nxt);
#pragma unroll
      for (int q = 0; q < B; ++q)
        if (id[q] != kNoWideId) op_apply<T, OP>(a, x[q]);
      if (B == kWideShort) {
#pragma unroll
        for (int q = 0; q < B; ++q) id[q] = nxt[q];
      }
    }
  }
  if (MODE == kModeGather) {
    static_cast<T*>(f.gv)[r * K + k] = a;
  } else {
    T* dst = field_base<T>(f, k);
    for (int q0 = 0; q0 < d; q0 += B) {
      uint32_t id[B];
      load_wide_ids<B>(ids, q0, d, id);
#pragma unroll
      for (int q = 0; q < B; ++q)
        if (id[q] != kNoWideId && (!pat.scatter_n || (id[q] >> 31)))
          dst[static_cast<int64_t>(checked_id(id[q] & 0x7FFFFFFFu, m.g.nnodes, m.g.err)) * stride] = a;
    }
  }
}

// All wide tiles: a warp an item, (tile, part) or (array, tile); see KLayout for
// the parts of k > 1 interleaved.
template <typename T, int OP, int MODE, int KL, int B>
__global__ void __launch_bounds__(kWideBlock, B == kWideLong ? 8 : 14)
    ogs_wide_kernel(const DevMaps m, const FieldArgs f, const Pattern pat) {
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int K = KL == kK1 ? 1 : f.K;
  const int64_t n = static_cast<int64_t>(m.nwide) * K;
  const int64_t W = static_cast<int64_t>(gridDim.x) * (kWideBlock / 32);
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * (kWideBlock / 32) + (threadIdx.x >> 5); i < n; i += W) {
    if (KL == kKInterleaved) {
      const int64_t t = i / K;
      const uint32_t u = static_cast<uint32_t>(i - t * K) * 32u + static_cast<uint32_t>(lane);
      const uint32_t rl = u / static_cast<uint32_t>(K);
      wide_tile<T, OP, MODE, B>(m, f, pat, static_cast<int>(t), static_cast<int>(rl), static_cast<int>(u - rl * K), K, K);
    } else {
      const int64_t a = KL == kKMany ? i / m.nwide : 0;
      wide_tile<T, OP, MODE, B>(m, f, pat, static_cast<int>(i - a * m.nwide), lane, static_cast<int>(a), K, 1);
    }
  }
}

template <typename T, int OP, int MODE, int KL>
inline void launch_wide(const DevMaps& m, const FieldArgs& f, Pattern pat, cudaStream_t s) {
  const int64_t items = static_cast<int64_t>(m.nwide) * f.K;
  const unsigned grid =
      static_cast<unsigned>(std::min<int64_t>((items + kWideBlock / 32 - 1) / (kWideBlock / 32), 1 << 20));
  if (m.wide_short) ogs_wide_kernel<T, OP, MODE, KL, kWideShort><<<grid, kWideBlock, 0, s>>>(m, f, pat);
  else ogs_wide_kernel<T, OP, MODE, KL, kWideLong><<<grid, kWideBlock, 0, s>>>(m, f, pat);
}

// The general rows of a call: as wide tiles or, for handles without them and
// gslib's rules, on the direct kernel.
template <typename T, int OP, int MODE>
inline cudaError_t launch_general(const DevMaps& m, const FieldArgs& f, Pattern pat, cudaStream_t s) {
  if (m.ngtiles == 0) return cudaSuccess;
  if (m.nwide == 0 || pat.gslib || pat.scatter_n > 1) {
    DevMaps g = m;
    g.tiles = m.gtiles;
    g.ntiles = m.ngtiles;
    return launch_direct<T, OP, MODE>(g, f, pat, s);
  }
  if (f.is_many) launch_wide<T, OP, MODE, kKMany>(m, f, pat, s);
  else if (f.K == 1) launch_wide<T, OP, MODE, kK1>(m, f, pat, s);
  else launch_wide<T, OP, MODE, kKInterleaved>(m, f, pat, s);
  return cudaGetLastError();
}

}  // namespace ogsgb
