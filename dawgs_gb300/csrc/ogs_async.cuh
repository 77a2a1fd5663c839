// ogs_async.cuh -- the warp pipeline with its value gathers staged through
// shared memory by cp.async.
//
// Same work items, arithmetic and stores as ogs_warp_kernel (ogs_warp.cuh;
// the reference fold is ogsOperator.cpp:60-97, 206-238, 311-360).  What
// changes is how many loads a warp keeps in flight.  The register pipeline
// holds one item's values and the next item's column ids; its registers cap
// it there, and the kernel is latency-bound (ncu: DRAM well under half busy,
// long-scoreboard stalls first).  Here the value gathers of an item are
// cp.async copies into a per-warp ring of shared memory, which hold no
// registers while in flight, so each warp keeps two items' values and a
// third item's column ids in flight:
//
//   iteration for item i:  issue gathers of item i+W into stage (s+1) % 2
//                          issue column-id loads of item i+2W (registers)
//                          wait for the gathers of item i (stage s)
//                          fold item i from shared memory, store
//
// Every lane gathers and later folds its own entries only, so no barrier of
// any kind is needed: cp.async.wait_group makes a thread's own completed
// copies visible to it.  Two stages suffice: the stage an iteration refills
// is the one the previous iteration read, and every value read there was
// consumed by the fold (in-order issue, and the asm's memory clobber keeps
// the compiler from moving the reads) before this iteration's cp.async
// issues.  A third stage only takes shared memory from L1 (measured slower).
#pragma once

#include <cstdint>

#include "ogs_warp.cuh"

#ifndef OGS_ASYNC
#define OGS_ASYNC 1
#endif

namespace ogsgb {

#ifndef OGS_ASYNC_STAGES
#define OGS_ASYNC_STAGES 2
#endif
constexpr int kAsyncStages = OGS_ASYNC_STAGES;
// k > 1 interleaved: split a tile's (row lane, component) units across its k
// parts so neighbouring threads take one node's neighbouring values (1), or
// give part j component j of every row lane (0).
// Resident CTAs per SM of the grid (0: as many as fit).
#ifndef OGS_ASYNC_CTAS
#define OGS_ASYNC_CTAS 0
#endif
#ifndef OGS_KI_SPLIT
#define OGS_KI_SPLIT 1
#endif

template <typename T>
__device__ __forceinline__ void cp_async_elem(T* smem, const T* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  if (sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// `lane` picks the tile rows (rows lane, lane + 32, ...); entry e of the
// thread lives at stage[e * 32 + slot], slot = the thread's own lane.
template <typename T, int MODE, int D, typename S>
__device__ __forceinline__ void async_issue_vals(const WarpState& s, const T* src, const T* gv, S stride, int K,
                                                 int k, bool gmask, int lane, int slot, T* stage) {
  constexpr int RPT = warp_rows_per_lane(D);
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
    if (j * 32 + lane < s.cnt) {
      if (MODE == kModeScatter) {
        cp_async_elem(stage + j * 32 + slot, gv + static_cast<int64_t>(s.R[j]) * K + k);
      } else {
#pragma unroll
        for (int q = 0; q < D; ++q)
          if (!gmask || ((s.emask >> (j * D + q)) & 1u))
            cp_async_elem(stage + (j * D + q) * 32 + slot, value_at(src, s.I[j * D + q], stride));
      }
    }
  }
}

template <typename T, int MODE, int D>
__device__ __forceinline__ void async_read_vals(const WarpState& s, bool gmask, int lane, int slot, const T* stage,
                                                T (&V)[kWarpSlots]) {
  constexpr int RPT = warp_rows_per_lane(D);
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
    if (j * 32 + lane < s.cnt) {
      if (MODE == kModeScatter) {
        V[j] = stage[j * 32 + slot];
      } else {
#pragma unroll
        for (int q = 0; q < D; ++q)
          if (!gmask || ((s.emask >> (j * D + q)) & 1u)) V[j * D + q] = stage[(j * D + q) * 32 + slot];
      }
    }
  }
}

// ---- lone tiles: 256 consecutive nodes, of which a byte per lane says which
// are their row's only member.  Their values come in 16-byte vectors, without
// column ids, and go back only if the fold from the identity changes their
// bits.  The degree-1 tiles of a mesh of high degree cost 4 of every 12 bytes a
// node moved and gathers of eight lines each: 24^3 p=15 fp64 185.7 -> 158.0 us.

// Whether identity (+) x has x's bits for every x: integer Add and Min, and
// Mul of every type (the fold starts from the member).  Lone tiles then have
// nothing to do.
template <typename T, int OP>
OGS_HD constexpr bool lone_is_noop() {
  return OP == OGS_MUL || (std::is_integral<T>::value && (OP == OGS_ADD || OP == OGS_MIN));
}

// Whether identity (+) x may differ from x: -0 under Add, infinities and NaN
// under Max and Min, by their bits (a compare of 8-byte floats costs a warp 16
// cycles of their pipe; 20^3 p=11 fp64 Max 45 us a call with it).
template <typename T, int OP>
__device__ __forceinline__ bool lone_suspect(const T x) {
  if constexpr (std::is_floating_point<T>::value) {
    using U = typename std::conditional<sizeof(T) == 8, unsigned long long, unsigned int>::type;
    constexpr U sign = U(1) << (8 * sizeof(T) - 1);
    constexpr U expo = sizeof(T) == 8 ? U(0x7FF0000000000000ull) : U(0x7F800000u);
    U b;
    memcpy(&b, &x, sizeof(T));
    return OP == OGS_ADD ? b == sign : (b & expo) == expo;
  } else {
    return x < -type_max<T>();  // Max starts there
  }
}

template <typename T>
__device__ __forceinline__ void lone_load_state(const DevMaps& m, const Tile& t, int lane, WarpState& s) {
  s.I[0] = t.begin;
  const uint32_t mask = __ldg((sizeof(T) == 8 ? m.lmask8 : m.lmask4) + static_cast<int64_t>(t.count) * 32 + lane);
  s.emask = checked_lone_mask(mask, t.begin, lane, 16 / sizeof(T), m.b[1].nnodes, m.b[1].err);
}

template <typename T, int OP>
__device__ __forceinline__ void lone_issue(const WarpState& s, const T* src, int N, int lane, T* stage) {
  if (lone_is_noop<T, OP>()) return;
  constexpr int VEC = 16 / sizeof(T);
#pragma unroll
  for (int j = 0; j < 8 / VEC; ++j) {
    const int at = (j * 32 + lane) * VEC;
    if (!((s.emask >> (j * VEC)) & ((1u << VEC) - 1u))) continue;
    if (lone_vector_in(s.I[0], at, VEC, N)) {
      const unsigned to = static_cast<unsigned>(__cvta_generic_to_shared(stage + at));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(to), "l"(src + s.I[0] + at) : "memory");
    } else {  // the field's last vector
#pragma unroll
      for (int i = 0; i < VEC; ++i)
        if (lone_vector_in(s.I[0], at + i, 1, N)) cp_async_elem(stage + at + i, src + s.I[0] + at + i);
    }
  }
}

template <typename T, int OP>
__device__ __forceinline__ void lone_fold_store(const WarpState& s, T* dst, int lane, const T* stage) {
  if (lone_is_noop<T, OP>()) return;
  constexpr int VEC = 16 / sizeof(T);
#pragma unroll
  for (int j = 0; j < 8 / VEC; ++j) {
    const int at = (j * 32 + lane) * VEC;
    alignas(16) T x[VEC];
    *reinterpret_cast<uint4*>(x) = *reinterpret_cast<const uint4*>(stage + at);
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      if (!lone_suspect<T, OP>(x[i]) || !((s.emask >> (j * VEC + i)) & 1u)) continue;
      T a;
      if constexpr (OP == OGS_ADD || OP == OGS_MUL) {
        a = fold_from_first<T, OP, 1>(x, i);
      } else {
        a = op_init<T, OP>();
        op_apply<T, OP>(a, x[i]);
      }
      if (!same_bits(a, x[i])) dst[s.I[0] + at + i] = a;
    }
  }
}

template <typename T>
constexpr size_t async_smem_bytes() {
  return static_cast<size_t>(kBlock / 32) * kAsyncStages * kWarpSlots * 32 * sizeof(T);
}

// PLAIN: every member takes part and receives the result (Pattern all zero:
// GatherScatter Sym, Gather/Scatter through the T map) -- the member-mask,
// store-mode and gslib branches drop out at compile time.
// LONE: the tiles are DevMaps::ltiles (plain GatherScatter, k = 1 or separate
// arrays on 16-byte boundaries).
template <typename T, int OP, int MODE, int KL, bool PLAIN, bool LONE>
__global__ void __launch_bounds__(kBlock, OGS_WARP_MINB) ogs_async_kernel(const DevMaps m, const FieldArgs f,
                                                                          const Pattern pat_in) {
  const Pattern pat = PLAIN ? Pattern{0, 0, 0, 0} : pat_in;
  extern __shared__ __align__(16) unsigned char async_smem[];
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int warp = static_cast<int>(threadIdx.x) >> 5;
  T* ring = reinterpret_cast<T*>(async_smem) + static_cast<size_t>(warp) * kAsyncStages * kWarpSlots * 32;
  const int64_t W = static_cast<int64_t>(gridDim.x) * (kBlock / 32);
  const int K = KL == kK1 ? 1 : f.K;
  const int64_t nw = m.nwtiles;
  const int64_t nitems = nw * K;
  const int64_t wid = static_cast<int64_t>(blockIdx.x) * (kBlock / 32) + warp;
  // Warp w takes items w, w+W, w+2W, ...: the grid sweeps the mesh front to
  // back.  k > 1 interleaved: item = (tile, part), tile-major, parts 0..k-1.
  // A tile's 32 row lanes times k components are 32k (row lane, component)
  // units, and part j takes units 32j .. 32j+31: thread t of part j works row
  // lane (32j+t) / k, component (32j+t) % k.  Neighbouring threads then read
  // the k neighbouring values of one node in the same instruction, so a
  // gather touches the sectors of about 32/k nodes instead of 32 (with OGS_KI_SPLIT
  // = 0, part j is component j for all 32 row lanes, and the k warps of a
  // tile meet each node's sectors only through L1).  Separate arrays: item =
  // (array, tile), array-major, so one array and the column ids stay in L2
  // while the grid sweeps it.  (A warp running a contiguous run of (tile,
  // component) items, loading each tile's column ids once, was measured much
  // slower: 83 vs 62 us for k = 3 on 3.5 M permuted nodes.)  Items are
  // followed as (tile, part) pairs, advanced by W without division.
  const int64_t i0 = wid;
  // Plain k = 1 reads descriptors and column ids before it waits for the work
  // ahead (grid_wait).  With components the wait in the middle costs more
  // registers than it hides: 32x32x16 p=5 permuted k=3 fp32 27.3 us a call
  // against 26.4 with the wait up here, Gather 23.0 against 18.6.
  constexpr bool kLate = PLAIN && KL == kK1;
  if (!kLate || i0 >= nitems) grid_wait(f.overlap);
  if (i0 >= nitems) return;
  int64_t i = i0;
  const int64_t step = W, iend = nitems;
  // item = outer * M + inner; interleaved: (tile, comp), M = K; many: (comp, tile), M = nw
  const int M = KL == kKMany ? static_cast<int>(nw) : (KL == kKInterleaved ? K : 1);
  const int Wi = static_cast<int>(W);
  const int Wq = KL == kK1 ? Wi : Wi / M, Wr = KL == kK1 ? 0 : Wi % M;
  const int o0 = KL == kK1 ? static_cast<int>(i0) : static_cast<int>(i0 / M);
  const int n0 = KL == kK1 ? 0 : static_cast<int>(i0 - static_cast<int64_t>(o0) * M);
  int tcur = KL == kKMany ? n0 : o0;
  int ccur = KL == kKMany ? o0 : n0;
  const bool use_mask = !PLAIN && (pat.gather_n || pat.scatter_n) && m.signed_maps;
  const bool gmask = !PLAIN && pat.gather_n != 0;
  const int smode = PLAIN ? 0 : pat.scatter_n;
  const bool gslib = !PLAIN && pat.gslib != 0;
  const ByteStride stride{(KL == kKInterleaved ? static_cast<uint32_t>(K) : 1u) * static_cast<uint32_t>(sizeof(T))};
  // the item W after (t, c)
  auto advance = [&](int t, int c, int& tn, int& cn) {
    if (KL == kK1) {
      tn = t + Wi;
      cn = 0;
    } else if (KL == kKInterleaved) {
      cn = c + Wr;
      tn = t + Wq;
      if (cn >= M) { cn -= M; tn += 1; }
    } else {
      tn = t + Wr;
      cn = c + Wq;
      if (tn >= M) { tn -= M; cn += 1; }
    }
  };
  T* gv = static_cast<T*>(f.gv);
  // The thread's row lane and component in item part c, recomputed where
  // needed rather than carried through the pipeline (registers).  Division by
  // k as a multiply-high by ceil(2^32 / k), exact while (32k) * k < 2^32.
  const bool split = KL == kKInterleaved && OGS_KI_SPLIT;
  const uint32_t kmagic = split && K > 1 ? 0xFFFFFFFFu / static_cast<uint32_t>(K) + 1u : 0u;
  const bool kmagic_ok = K < 11585;
  auto unit = [&](int c, int& rl, int& comp) {
    if (split) {
      const uint32_t u = static_cast<uint32_t>(c) * 32u + static_cast<uint32_t>(lane);
      rl = static_cast<int>(kmagic_ok ? __umulhi(u, kmagic) : u / static_cast<uint32_t>(K));
      comp = static_cast<int>(u) - rl * K;
    } else {
      rl = lane;
      comp = c;
    }
  };
  int rcur, kcur;
  unit(ccur, rcur, kcur);

  // prologue: the descriptors of items i, i+1 step, i+2 steps in one round
  // trip, the column ids of the first two in the next, then the gathers of
  // item i; the loop's first pass issues the gathers of the next item at once
  int tnxt = 0, cnxt = 0, tnn = 0, cnn = 0;
  const bool has1 = i + step < iend;
  Tile cur = m.wtiles[tcur];
  Tile nxt{}, nn{};
  if (has1) {
    advance(tcur, ccur, tnxt, cnxt);
    nxt = m.wtiles[tnxt];
    if (i + 2 * step < iend) {
      advance(tnxt, cnxt, tnn, cnn);
      nn = m.wtiles[tnn];
    }
  }
  WarpState scur, snxt;
#define OGS_A_LOAD(D, TILE, TI, RL, S) warp_load_state<MODE, D>(m.b[D], TILE, m.wemask, TI, use_mask, pat, RL, S)
#define OGS_A_LOAD_CUR(D) OGS_A_LOAD(D, cur, tcur, rcur, scur)
  if (LONE && cur.bucket == kLoneBucket) lone_load_state<T>(m, cur, lane, scur);
  else OGS_DEGREE_SWITCH(cur.bucket, OGS_A_LOAD_CUR)
#undef OGS_A_LOAD_CUR
  if (has1) {
    int rnxt, knxt;
    unit(cnxt, rnxt, knxt);
#define OGS_A_LOAD_NXT(D) OGS_A_LOAD(D, nxt, tnxt, rnxt, snxt)
    if (LONE && nxt.bucket == kLoneBucket) lone_load_state<T>(m, nxt, lane, snxt);
    else OGS_DEGREE_SWITCH(nxt.bucket, OGS_A_LOAD_NXT)
#undef OGS_A_LOAD_NXT
  }
  if (kLate) grid_wait(f.overlap);  // the first access to the field follows
  {
    const T* src = (MODE == kModeScatter) ? nullptr : field_base<T>(f, kcur);
#define OGS_A_ISSUE0(D) async_issue_vals<T, MODE, D>(scur, src, gv, stride, K, kcur, gmask, rcur, lane, ring)
    if (LONE && cur.bucket == kLoneBucket) lone_issue<T, OP>(scur, src, m.b[1].nnodes, lane, ring);
    else OGS_DEGREE_SWITCH(cur.bucket, OGS_A_ISSUE0)
#undef OGS_A_ISSUE0
  }
  cp_async_commit();

  int stage = 0;
  for (;;) {
    const bool more1 = i + step < iend;
    const bool more2 = i + 2 * step < iend;
    const int nstage = stage == kAsyncStages - 1 ? 0 : stage + 1;
    if (more1) {
      int rnxt, knxt;
      unit(cnxt, rnxt, knxt);
      const T* src1 = (MODE == kModeScatter) ? nullptr : field_base<T>(f, knxt);
      T* st1 = ring + nstage * (kWarpSlots * 32);
#define OGS_A_ISSUE1(D) async_issue_vals<T, MODE, D>(snxt, src1, gv, stride, K, knxt, gmask, rnxt, lane, st1)
      if (LONE && nxt.bucket == kLoneBucket) lone_issue<T, OP>(snxt, src1, m.b[1].nnodes, lane, st1);
      else OGS_DEGREE_SWITCH(nxt.bucket, OGS_A_ISSUE1)
#undef OGS_A_ISSUE1
    }
    cp_async_commit();
    WarpState snn;
    Tile n3{};
    int tn3 = 0, cn3 = 0;
    if (more2) {
      int rnn, knn;
      unit(cnn, rnn, knn);
#define OGS_A_LOAD_NN(D) OGS_A_LOAD(D, nn, tnn, rnn, snn)
      if (LONE && nn.bucket == kLoneBucket) lone_load_state<T>(m, nn, lane, snn);
      else OGS_DEGREE_SWITCH(nn.bucket, OGS_A_LOAD_NN)
#undef OGS_A_LOAD_NN
      if (i + 3 * step < iend) {
        advance(tnn, cnn, tn3, cn3);
        n3 = m.wtiles[tn3];
      }
    }
    cp_async_wait<1>();  // the gathers of item i are in
    {
      unit(ccur, rcur, kcur);
      T* dst = (MODE == kModeGather) ? nullptr : field_base<T>(f, kcur);
      const T* st0 = ring + stage * (kWarpSlots * 32);
      T V[kWarpSlots];
#define OGS_A_FOLD(D)                                                                              \
  do {                                                                                             \
    async_read_vals<T, MODE, D>(scur, gmask, rcur, lane, st0, V);                                  \
    warp_fold_store<T, OP, MODE, D>(scur, dst, gv, stride, K, kcur, gmask, smode, gslib, rcur, V); \
  } while (0)
      if (LONE && cur.bucket == kLoneBucket) lone_fold_store<T, OP>(scur, dst, lane, st0);
      else OGS_DEGREE_SWITCH(cur.bucket, OGS_A_FOLD)
#undef OGS_A_FOLD
    }
    if (!more1) break;
    i += step;
    stage = nstage;
    cur = nxt;
    scur = snxt;
    tcur = tnxt;
    ccur = cnxt;
    nxt = nn;
    snxt = snn;
    tnxt = tnn;
    cnxt = cnn;
    nn = n3;
    tnn = tn3;
    cnn = cn3;
  }
  cp_async_wait<0>();
#undef OGS_A_LOAD
}

template <typename T, int OP, int MODE, int KL, bool PLAIN, bool LONE>
inline int async_grid(int64_t nitems) {
  static DeviceCache cache;
  int dev = 0;
  cudaGetDevice(&dev);
  const int cached = cache.get(dev, [dev] {
    int bps = 0, sms = 0;
    // above 48 KB (more entries per lane) the dynamic shared memory must be opted into
    if (async_smem_bytes<T>() > 48 * 1024)
      cudaFuncSetAttribute(ogs_async_kernel<T, OP, MODE, KL, PLAIN, LONE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(async_smem_bytes<T>()));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, ogs_async_kernel<T, OP, MODE, KL, PLAIN, LONE>, kBlock,
                                                  async_smem_bytes<T>());
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
#if OGS_ASYNC_CTAS > 0
    if (bps > OGS_ASYNC_CTAS) bps = OGS_ASYNC_CTAS;
#endif
    return (bps > 0 ? bps : 1) * (sms > 0 ? sms : 1);
  });
  const int64_t need = (nitems + (kBlock / 32) - 1) / (kBlock / 32);
  return static_cast<int>(need < cached ? need : cached);
}

template <typename T, int OP, int MODE, int KL, bool PLAIN, bool LONE>
inline void launch_async_as(const DevMaps& m, const FieldArgs& f, Pattern pat, cudaStream_t s) {
  const int grid = async_grid<T, OP, MODE, KL, PLAIN, LONE>(static_cast<int64_t>(m.nwtiles) * (KL == kK1 ? 1 : f.K));
  launch_overlapped(ogs_async_kernel<T, OP, MODE, KL, PLAIN, LONE>, dim3(grid), kBlock, async_smem_bytes<T>(), s,
                    f.overlap, m, f, pat);
}

template <typename T, int OP, int MODE, int KL>
inline void launch_async_kl(const DevMaps& m, const FieldArgs& f, Pattern pat, cudaStream_t s) {
  const bool plain = !pat.gather_n && !pat.scatter_n && !pat.limit_n && !pat.gslib;
  if constexpr (MODE == kModeGS && KL != kKInterleaved) {
    constexpr bool cheap = OP == OGS_MAX || OP == OGS_MIN || lone_is_noop<T, OP>();
    bool lone = plain && lone_folds(m, sizeof(T), cheap);
    for (int k = 0; lone && k < (KL == kKMany ? f.K : 1); ++k)
      lone = (reinterpret_cast<uintptr_t>(KL == kKMany ? f.many[k] : f.v) & 15) == 0;
    if (lone) {
      DevMaps l = m;
      l.wtiles = m.ltiles;
      l.nwtiles = m.nltiles;
      return launch_async_as<T, OP, MODE, KL, true, true>(l, f, pat, s);
    }
  }
  if (plain) launch_async_as<T, OP, MODE, KL, true, false>(m, f, pat, s);
  else launch_async_as<T, OP, MODE, KL, false, false>(m, f, pat, s);
}

// Exact-degree tiles on the async pipeline, general rows in a launch of their own.
template <typename T, int OP, int MODE>
inline cudaError_t launch_async(const DevMaps& m, const FieldArgs& f, Pattern pat, cudaStream_t s) {
  if (m.nwtiles > 0) {
    if (f.is_many) launch_async_kl<T, OP, MODE, kKMany>(m, f, pat, s);
    else if (f.K == 1) launch_async_kl<T, OP, MODE, kK1>(m, f, pat, s);
    else launch_async_kl<T, OP, MODE, kKInterleaved>(m, f, pat, s);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return launch_general<T, OP, MODE>(m, f, pat, s);
}

}  // namespace ogsgb
