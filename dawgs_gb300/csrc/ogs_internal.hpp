// ogs_internal.hpp -- shared definitions of the GB300 gather-scatter library:
// the device layout of one mesh's maps, the work tiles, and the launch
// interface between the C ABI (ogs_capi.cpp) and the per-type kernel units
// (ogs_kern_*.cu).
#pragma once

#include <atomic>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include <cuda_runtime_api.h>

#include "ogs_c.h"

#ifdef __CUDACC__
#define OGS_HD __host__ __device__
#else
#define OGS_HD
#endif

namespace ogsgb {

// A launch figure per device (CTAs per SM, SM count), computed on first use.
// Concurrent first uses compute the same value, so filling it without a lock
// is safe; the atomics keep the sharing well defined.
struct DeviceCache {
  static constexpr int kDevices = 64;
  std::atomic<int> v[kDevices];
  template <typename F>
  int get(int dev, F compute) {
    if (dev < 0 || dev >= kDevices) return compute();
    int x = v[dev].load(std::memory_order_acquire);
    if (x == 0) {
      x = compute();
      v[dev].store(x, std::memory_order_release);
    }
    return x;
  }
};

// Checked builds (-DOGS_CHECK_BOUNDS=1, for tests): every column id and row
// id a kernel loads from the maps is compared with the handle's node and row
// counts before a value is read or written through it; an id out of range
// is counted in the handle's error word and replaced by 0, so the access
// stays inside the field.  Default builds compile the checks out.
#ifndef OGS_CHECK_BOUNDS
#define OGS_CHECK_BOUNDS 0
#endif

// Rows of exact degree 1..kDmax are stored in fixed-width buckets; rows of a
// larger degree go to one general CSR bucket.
constexpr int kDmax = 8;
// Entries (row members) per work tile.  A 256-thread CTA handles one tile:
// every thread owns kTileNnz/256 = 8 entries, i.e. 8/d rows of degree d.
constexpr int kBlock = 256;
constexpr int kTileNnz = 2048;
constexpr int kEntriesPerThread = kTileNnz / kBlock;
// General-bucket tiles hold at most one row per thread.
constexpr int kGeneralRowsPerTile = kBlock;
// Slices of the host-buffer pipeline (ogs_gather_scatter_host) and whether
// the pipeline is captured into a CUDA graph and replayed on later calls with
// the same host buffer.
#ifndef OGS_HOST_PHASES
#define OGS_HOST_PHASES 8
#endif
#ifndef OGS_HOST_GRAPH
#define OGS_HOST_GRAPH 0
#endif
// With 6 or more slices, the first and last two take 1/4 and 1/2 of the
// others' share of tiles: the first copy in and the last copy out run with
// nothing beside them, so they are kept short.
#ifndef OGS_HOST_TAPER
#define OGS_HOST_TAPER 1
#endif
// Separate arrays handled by one launch of the *_many entry points.
constexpr int kMaxMany = 16;
// Member entries per lane of a warp tile (ogs_warp.cuh): lane l owns
// kWarpEntries/d rows of degree d (at least one); the per-lane arrays hold up
// to kWarpSlots entries.
#ifndef OGS_WARP_ENTRIES
#define OGS_WARP_ENTRIES 8
#endif
constexpr int kWarpEntries = OGS_WARP_ENTRIES;
constexpr int kWarpSlots = kWarpEntries > kDmax ? kWarpEntries : kDmax;

// Rows of degree d that one thread handles in a tile (at least one).
OGS_HD inline constexpr int rows_per_thread(int d) {
  return (kEntriesPerThread / d) > 0 ? (kEntriesPerThread / d) : 1;
}
OGS_HD inline constexpr int rows_per_tile(int d) {
  return d >= 1 && d <= kDmax ? kBlock * rows_per_thread(d) : kGeneralRowsPerTile;
}
OGS_HD inline constexpr int warp_rows_per_lane(int d) {
  return (kWarpEntries / d) > 0 ? (kWarpEntries / d) : 1;
}
OGS_HD inline constexpr int warp_rows_per_tile(int d) { return 32 * warp_rows_per_lane(d); }

// One bucket of rows of exact degree d, rows in ascending row order.
// Arrays are padded (stride = n rounded up to 4 rows, masks to 16 bytes) so
// that every tile's chunk starts on a 16-byte boundary and may be copied with
// its length rounded up, as the bulk (TMA) copies require.
struct DevBucket {
  const int32_t* cols;   // [d][stride]: member j of bucket row i at cols[j*stride + i]
  const int32_t* rows;   // [stride] row ids (ascending)
  const uint8_t* nmask;  // [stride rounded to 16] bit j: member j is in the N map (Signed only)
  int32_t n;             // rows in the bucket
  int32_t nP;            // rows with row id < NrowsN, a prefix of the bucket
  int32_t stride;        // n rounded up to a multiple of 4
  int32_t nnodes;        // local nodes: column ids lie in [0, nnodes)
  int32_t nrows;         // rows of the T map: row ids lie in [0, nrows)
  unsigned int* err;     // ids found out of range (checked builds); may be null
};

// Rows of degree > kDmax, CSR relative to the bucket.
struct DevGeneral {
  const int32_t* rows;     // [n]
  const int32_t* startsT;  // [n+1]
  const int32_t* colsT;
  const int32_t* startsN;  // [n+1] (alias startsT when Unsigned)
  const int32_t* colsN;
  int32_t n, nP;
  int32_t nnodes, nrows;   // as in DevBucket
  unsigned int* err;
};

// A tile: `count` consecutive rows of one bucket, starting at `begin`.
// bucket 0 = general, 1..kDmax = exact degree.  Tiles are ordered by the row
// id of their first row so that concurrently running CTAs touch nearby nodes.
struct Tile {
  int32_t bucket;
  int32_t begin;
  int32_t count;
  int32_t first_row;
};

// One warp tile as a self-contained 32-byte record, for launches that walk
// the tiles of several meshes (ogs_batch.cuh).
struct WarpRec {
  const int32_t* cols;   // the bucket's column ids (member q of row i at cols[q*stride + i])
  const int32_t* rows;   // the bucket's row ids
  int32_t begin;         // first bucket row of the tile
  int32_t bucket_count;  // degree << 16 | rows in the tile
  int32_t stride;        // the bucket's stride
  int32_t nP;            // bucket rows below NrowsN
};
static_assert(sizeof(WarpRec) == 32, "WarpRec is 32 bytes");

// One entry of a batched launch, in device memory.
struct BatchEntry {
  const WarpRec* recs;     // the handle's warp records
  const uint8_t* wemask;   // the handle's per-lane N masks (Signed only)
  void* v;                 // field, K interleaved components per node
  int32_t K, op;
  int32_t gather_n, scatter_n, limit_n, use_mask;
  uint32_t kmagic;         // ceil(2^32 / K) for 1 < K < 11585 (division by K as a multiply-high), else 0
  int32_t reserved;
};
// The multiply-high divisor of a batch entry's K: floor(u / K) ==
// umulhi(u, ceil(2^32 / K)) for every u < 32 K when (32 K) K < 2^32.
inline bool batch_plain(const BatchEntry& e) {
  return !e.gather_n && !e.scatter_n && !e.limit_n && !e.use_mask;
}
inline uint32_t batch_kmagic(int K) { return K > 1 && K < 11585 ? 0xFFFFFFFFu / static_cast<uint32_t>(K) + 1u : 0u; }
// Work items of a batched launch: each (warp record, component) pair of each
// entry; starts[e] = first item of entry e, records of an entry in order with
// their K components adjacent.


// 32 consecutive nodes of a handle whose rows are numbered by first member
// (ogs_scatter.cuh): which of them are their row's first member -- their rows
// are row0, row0 + 1, ... -- and which another, whose rows are listed from
// orow[other0] on.
struct alignas(16) NodeWord {
  uint32_t first, other;
  int32_t row0, other0;
};
struct DevNodes {
  const NodeWord* words;  // padded with empty words to a multiple of kNodeWordPad
  const uint32_t* nmem;   // bit per node: in the N map (padded alike)
  const int32_t* orow;
  int64_t nwords;         // 0: the handle has none
  int32_t scatter;        // whether a Scatter runs over them (scatter_share)
};
constexpr int kNodeWordPad = 16;
inline int64_t node_words(int64_t N) { return (N + 31) / 32; }
inline int64_t node_words_padded(int64_t N) { return (node_words(N) + kNodeWordPad - 1) / kNodeWordPad * kNodeWordPad; }

// Lone nodes (their row's only member) of kLoneNodes consecutive nodes, as a
// tile of the exact-degree rows' launch (ogs_async.cuh): bucket kLoneBucket,
// begin the first node, count the tile's row of the masks.
constexpr int kLoneNodes = 256;
constexpr int kLoneBucket = kDmax + 1;
// Bit q of lane l's byte stands for node ((q / v) * 32 + l) * v + q % v of the
// tile, v = 2 or 4 values of 8 or 4 bytes in a 16-byte vector, or 1.
OGS_HD inline int lone_node(int l, int q, int v) { return ((q / v) * 32 + l) * v + q % v; }
// Whether the v values from place `at` of a lone tile on lie in a field of N
// nodes.  (begin + at + v passes 2^31 in the last tile of 2^31 - 1 nodes.)
OGS_HD inline bool lone_vector_in(int32_t begin, int at, int v, int32_t N) {
  return static_cast<uint32_t>(begin) + static_cast<uint32_t>(at + v) <= static_cast<uint32_t>(N);
}

// Member of a wide tile's row: node | N member << 31, or none.
constexpr uint32_t kNoWideId = 0xFFFFFFFFu;
constexpr int kWideRows = 32;  // rows of a wide tile

struct DevMaps {
  DevBucket b[kDmax + 1];  // b[0] unused
  DevGeneral g;
  const Tile* tiles;       // CTA tiles of every bucket, ordered by first row (direct kernel)
  int32_t ntiles;
  int32_t signed_maps;     // N maps differ from T maps
  int32_t ngtiles;         // general-bucket CTA tiles, ordered by first row
  const Tile* gtiles;
  const Tile* wtiles;      // exact-degree warp tiles (ogs_warp.cuh), ordered by first row
  const uint8_t* wemask;   // [nwtiles][32] per-lane entry masks of the N map (Signed only)
  int32_t nwtiles;
  const WarpRec* wrecs;    // [nwtiles] the warp tiles as records (batched launches)
  DevNodes nodes;
  // The general rows, kWideRows a tile (ogs_wide.cuh): bucket = the longest
  // row's degree, begin and count in the general bucket, member q of the
  // tile's row j at wide_ids[(first_row + q) * 32 + j].
  const Tile* wide;
  const uint32_t* wide_ids;
  int32_t nwide;           // 0: the general rows run as CTA tiles
  int32_t wide_short;      // the rows are of degree 12 and less on average
  // The warp tiles of degree 2 and up with lone tiles in place of the degree-1
  // ones, in node order, for handles that are mostly lone nodes (wants_lone).
  const Tile* ltiles;
  const uint8_t* lmask8;   // [lone tiles][32] for 8-byte values
  const uint8_t* lmask4;   // ... for 4-byte values
  const uint8_t* lmask1;   // ... a node at a time (handles with node words)
  int32_t nltiles;         // 0: the handle has none
};

// Which members take part, per ogsOperator.cpp:60-97, 206-238, 311-360.
struct Pattern {
  int32_t gather_n;   // fold only members of the N map
  int32_t scatter_n;  // 1: write only members of the N map; 2: those, or member 0
                      //    when the row has none (gslib transpose 1)
  int32_t limit_n;    // process rows < NrowsN only
  int32_t gslib = 0;  // gslib rules: fold from the first member taking part,
                      //    integer Max starting at INT_MIN (gs_defs.h:44-52)
};

enum Mode : int { kModeGS = 0, kModeGather = 1, kModeScatter = 2 };

// Field operands of one launch.  Interleaved: component c of node n at
// base[0][c + n*K].  Many: component c of node n at base[c][n].
struct FieldArgs {
  void* v;                  // interleaved local vector (GS, Gather input, Scatter output)
  void* gv;                 // interleaved gathered vector (Gather output, Scatter input)
  void* many[kMaxMany];     // separate arrays (GS many)
  int32_t K;
  int32_t is_many;
  int32_t overlap = 0;      // programmatic stream serialization (grid_wait)
};

// Whether the pipelines and the wide tiles take a call of K components: they
// number a tile's 32 K (row lane, component) units in 32 bits.  The direct kernel
// (ogs_kernels.cuh) steps through components in 64.
inline bool units_fit(int K, bool is_many) { return is_many || K <= (1 << 27); }

// Whether a plain GatherScatter of values of `bytes` bytes runs over the lone
// tiles, and a plain Gather: from kLoneBytes a field on, where the column ids and
// gathers that they save come out of DRAM, a quarter of L2 with the ids beside.
// Below, a GatherScatter does from 65 % lone nodes on, or where the fold of a lone
// node is the dearest (8-byte Max and Min of floats, a compare of 16 cycles) or
// nothing (integers and Mul: `cheap`).  Us a call without / with them, Add: fp64
// p=10 (55 %) 12^3 7.0 / 7.2, 14^3 (29 MB) 9.9 / 10.8, 16^3 (44 MB) 16.4 / 15.7,
// 20^3 34.8 / 31.8; p=15 (67 %) 8^3 6.9 / 6.7, 12^3 (57 MB) 20.3 / 18.4; fp32 p=10
// 14^3 7.9 / 8.8, 20^3 (43 MB) 26.4 / 22.7, p=13 (63 %) 12^3 (19 MB) 9.0 / 9.6,
// 16^3 (45 MB) 25.2 / 21.5; four arrays of fp64 p=10 10^3 14.2 / 15.5, 24^3 243.7 /
// 226.4.  Max fp64 p=10 10^3 6.1 / 5.3.  Gather fp64 p=10 14^3 9.3 / 10.1, 16^3
// 15.8 / 13.6, p=15 8^3 6.6 / 6.9, fp32 p=10 16^3 (22 MB) 9.6 / 10.6, 20^3 26.5 /
// 22.5.
constexpr int64_t kLoneBytes = 30 << 20;
inline bool lone_folds(const DevMaps& m, int bytes, bool cheap) {
  const int64_t N = m.b[1].nnodes;
  return m.nltiles > 0 && (N * bytes >= kLoneBytes || int64_t{20} * m.b[1].n >= 13 * N || (cheap && bytes == 8));
}
inline bool lone_gathers(const DevMaps& m, int bytes) {
  return m.nltiles > 0 && m.nodes.nwords > 0 && int64_t{m.b[1].nnodes} * bytes >= kLoneBytes;
}

// Whether a Scatter runs in node order (ogs_scatter.cuh): where the handle has
// node words (rows numbered by first member) and most of its nodes take part
// (scatter_share), for components of up to kScatterNodeBytes a node: 8 of 8 bytes,
// 16 of 4.  A warp takes every component of a word, so more of them leave a small
// mesh with few warps that each go through many rounds (eight runs a round: 1,000
// nodes k=1000 117 us against 3.9 through the column lists, 64 nodes k=20000
// 2,459 against 7.9, 20^3 p=7 k=64 fp64 93 against 78).  Through the column lists
// / in node order, us: fp64 k=8 10^3 p=7 8.5 / 7.4, 24^3 p=7 134.8 / 130.1, 40^3
// p=3 permuted 80.5 / 82.5, k=5 24^3 p=7 101.4 / 86.2; fp32 k=8 20^3 p=7 56.2 /
// 43.9, k=14 10^3 p=7 11.0 / 8.5 and 20^3 p=7 87.4 / 86.8, k=16 12.1 / 9.5, 105.8 /
// 114.0 and 40^3 p=3 permuted 109.1 / 120.9.  Operators over caller maps and the
// slices of host-buffer calls keep the tile kernels.
constexpr int kScatterNodeBytes = 64;
OGS_HD constexpr int scatter_max_k(int bytes) { return kScatterNodeBytes / bytes; }
inline bool scatter_applies(const DevMaps& m, const FieldArgs& f, const Pattern& pat, int bytes) {
  return m.nodes.scatter && f.K <= scatter_max_k(bytes) && !f.is_many && !pat.gslib && pat.scatter_n <= 1;
}

// A slice of the warp and general tiles for the host-buffer pipeline: its
// kernels read and write local nodes in [lo, hi]; its host->device chunk is
// [h0, h1) and once it has run, local nodes [d0, d1) are final and go back.
struct Phase {
  int32_t w0, w1;  // warp tiles
  int32_t g0, g1;  // general tiles
  int64_t lo, hi;
  int64_t h0, h1, d0, d1;
  // rows: the gathered vector's rows [r0, r1) are final once this slice has
  // run (no later slice writes a row below r1); rows [0, rn) hold every row
  // this slice or an earlier one reads (host-buffer Gather and Scatter)
  int64_t r0, r1, rn;
};

// Host-side copy of everything built at setup.
struct HostLayout {
  std::vector<int32_t> cols[kDmax + 1];
  std::vector<int32_t> rows[kDmax + 1];
  std::vector<uint8_t> nmask[kDmax + 1];
  int32_t nP[kDmax + 1] = {0};
  int32_t n[kDmax + 1] = {0};
  std::vector<int32_t> g_rows, g_startsT, g_colsT, g_startsN, g_colsN;
  int32_t g_nP = 0;
  std::vector<Tile> tiles;   // CTA tiles, all buckets, by first row
  std::vector<Tile> gtiles;  // general CTA tiles, by first row
  std::vector<Tile> wtiles;  // exact-degree warp tiles, by first row
  std::vector<uint8_t> wemask;
  std::vector<NodeWord> nwords;  // host path only: see DevNodes
  std::vector<uint32_t> nmem;
  std::vector<int32_t> orow;
  std::vector<Tile> ltiles;        // see DevMaps
  std::vector<uint8_t> lmask8, lmask4, lmask1;  // host path only
  std::vector<Tile> wide;          // see DevMaps
  int64_t wide_units = 0;          // 32 ids each
  std::vector<Phase> phases;
  int64_t g_n = 0, g_nnzT = 0;  // general-bucket rows and T entries
  // lowest and highest local node each warp tile / general tile touches
  std::vector<int64_t> wlo, whi, glo, ghi;
};

}  // namespace ogsgb

struct ogs_handle_s {
  int64_t N = 0;
  int kind = 0;
  int unique = 0;
  int gather_defined = 0;
  int64_t NlocalP = 0, NlocalT = 0, Ngather = 0, NgatherGlobal = 0;
  int64_t nnzT = 0, nnzN = 0;
  int32_t max_degree = 0;
  bool host_only = false;
  bool covers_all = false;  // every local node is in the T map (no zero ids)
  bool gslib = false;       // maps in gslib's member order (ogs_gslib.cpp)
  bool from_maps = false;   // an operator over caller-built maps (ogs_maps.cpp)
  bool overlap = true;      // calls may start before the work ahead of them has ended
  bool distinct_cols = true;  // no local node in two rows (GatherScatter/Scatter need it)

  std::vector<int32_t> rowStartsT, colIdsT, rowStartsN, colIdsN;  // N empty when Unsigned
  ogsgb::HostLayout lay;

  int device = -1;
  void* arena = nullptr;  // one device allocation for all maps
  size_t arena_bytes = 0;
  ogsgb::DevMaps dmaps{};

  std::mutex host_mu;     // serialises the _host entry points (they share `stage`)
  void* stage = nullptr;  // device staging for the _host entry points
  size_t stage_bytes = 0;
  void* copy_in = nullptr;   // cudaStream_t: host->device chunks of the host pipeline
  void* copy_out = nullptr;  // cudaStream_t: device->host chunks
  void* capture = nullptr;   // cudaStream_t: the pipeline is captured on it
  std::vector<void*> events; // cudaEvent_t: [0] start, 2 per phase, then 2 joins
  struct HostGraph {         // captured host-buffer pipelines, most recent first
    void* host;
    int k, type, op, trans;
    void* exec;              // cudaGraphExec_t
  };
  std::vector<HostGraph> host_graphs;
};

namespace ogsgb {

// Host setup (ogs_setup.cpp).
ogs_status build_host_maps(ogs_handle_s* h, int64_t N, int64_t* ids, int kind, int unique);
// The same maps built on the current device (ogs_dsetup.cu).
ogs_status build_device_maps(ogs_handle_s* h, int64_t N, int64_t* ids, int kind, int unique, bool layout);
void build_layout(ogs_handle_s* h);
ogs_status upload_layout(ogs_handle_s* h);
void release_device(ogs_handle_s* h);
void build_phases(ogs_handle_s* h, int max_phases);  // needs the tiles and their lo/hi
// Whether a handle gets node words: Scatter is defined and every row has a
// positive member, so that rows are numbered by first member.
inline bool wants_node_words(const ogs_handle_s* h) {
  return h->kind == OGS_SIGNED && h->gather_defined && !h->from_maps && !h->gslib && h->NlocalT > 0 &&
         h->NlocalP == h->NlocalT;
}
// Whether enough nodes take part for a Scatter to go through all of them: three
// quarters.  In 10 M nodes of which the first part takes part, pairs of
// neighbours, fp64 k=3, through the column lists / in node order: 1/2 37.0 /
// 43.8 us, 5/8 45.1 / 49.1, 3/4 53.0 / 54.2, 7/8 60.7 / 59.0; 1/1000 of 7 M
// nodes 2.5 / 15.4.  (Parts that lie between the others do better: 1/2 89.4 /
// 81.0.)
inline bool scatter_share(const ogs_handle_s* h) { return h->nnzT * 4 >= h->N * 3; }
// Wide tiles of general rows with the given row starts; the units of 32 ids
// they take.  None where rows of very different degree are neighbours and the
// padding would outweigh the rows.
int64_t wide_layout(const int32_t* starts, int64_t rows, std::vector<Tile>& wide);
// Fills m.wide_ids from the general rows on `stream` (ogs_dsetup.cu); a cudaError_t value.
int launch_wide_ids(const DevMaps& m, void* stream);
// Whether a handle gets lone tiles for its n1 rows of degree 1 (the rows being
// numbered by first member): from 55 % of its nodes on; which calls run over them
// is up to lone_folds and lone_gathers.  Us a call without and with them, boxes of
// 24^3: GatherScatter fp64 p=9 (51 %) 47.7 and 49.0, p=10 (55 %) 58.2 and 58.5,
// four arrays 243.7 and 226.4, p=11 (58 %) 75.2 and 74.3, p=15 (67 %) 185.1 and
// 157.1; fp32 p=7 (42 %) 17.5 and 19.1, p=11 59.1 and 56.5, p=15 134.8 and 108.8.
// Gather fp64 p=7 25.1 and 24.6, p=9 46.6 and 44.5, p=11 77.2 and 71.7, p=15 187.6
// and 161.5; fp32 p=7 13.3 and 14.8, p=11 54.9 and 53.8.
inline bool wants_lone(const ogs_handle_s* h, int64_t n1) {
  return !h->gslib && !h->from_maps && h->NlocalP == h->NlocalT && n1 * 20 >= h->N * 11;
}
// The lone tiles of N nodes; and HostLayout::ltiles (needs the warp tiles and the
// lowest node of each).
inline int64_t lone_tiles(int64_t N) { return (N + kLoneNodes - 1) / kLoneNodes; }
void lone_layout(ogs_handle_s* h);
// DevMaps restricted to the general rows.
DevMaps general_maps(const DevMaps& m);
// DevMaps restricted to the tiles of one phase.
DevMaps phase_maps(const DevMaps& m, const Phase& p);
// The id ranges and error word of every bucket (both setup paths).
void set_id_bounds(const ogs_handle_s* h, DevMaps& m, unsigned int* err);

// Per-type launchers (ogs_kern_*.cu; which kernels: ogs_launch.cuh).  Return a
// cudaError_t value.
int launch_f32(const DevMaps& m, const FieldArgs& f, int mode, int op, Pattern pat, void* stream);
int launch_f64(const DevMaps& m, const FieldArgs& f, int mode, int op, Pattern pat, void* stream);
int launch_i32(const DevMaps& m, const FieldArgs& f, int mode, int op, Pattern pat, void* stream);
int launch_i64(const DevMaps& m, const FieldArgs& f, int mode, int op, Pattern pat, void* stream);

// Batched launch over `n` entries (ogs_batch.cuh); grid <= 0 = one full wave;
// block = 128 or 256 threads per CTA; occ = 2 or 3 (register budget: 256-thread
// CTAs per SM); pipe = 0 register pipeline, 1 cp.async ring (256 threads);
// plain = 1 when no entry has N masks, a store mode or a row limit
// (batch_plain), which selects kernels without those branches.
int launch_batch_f32(const BatchEntry* E, const int64_t* starts, int n, int64_t nitems, int grid, int block,
                     int occ, int pipe, int plain, void* stream);
int launch_batch_f64(const BatchEntry* E, const int64_t* starts, int n, int64_t nitems, int grid, int block,
                     int occ, int pipe, int plain, void* stream);
int launch_batch_i32(const BatchEntry* E, const int64_t* starts, int n, int64_t nitems, int grid, int block,
                     int occ, int pipe, int plain, void* stream);
int launch_batch_i64(const BatchEntry* E, const int64_t* starts, int n, int64_t nitems, int grid, int block,
                     int occ, int pipe, int plain, void* stream);

// Device and page-locked host allocations (ogs_alloc.cpp): counted, and made
// to fail on demand by ogs_debug_fail_alloc.  Every allocation of the library
// goes through these.
cudaError_t dev_malloc_raw(void** p, size_t bytes);
void dev_free(void* p);
cudaError_t host_malloc_raw(void** p, size_t bytes);
void host_free(void* p);
template <typename T>
inline cudaError_t dev_malloc(T** p, size_t bytes) {
  return dev_malloc_raw(reinterpret_cast<void**>(p), bytes);
}
template <typename T>
inline cudaError_t host_malloc(T** p, size_t bytes) {
  return host_malloc_raw(reinterpret_cast<void**>(p), bytes);
}

// Load the batched kernel the server launches (256 threads, 2 CTAs per SM)
// ahead of its first use.
int preload_batch_f32();
int preload_batch_f64();
int preload_batch_i32();
int preload_batch_i64();

// Thread-local error message (ogs_capi.cpp).
ogs_status set_error(ogs_status s, const std::string& msg);

// Argument checks and member patterns shared by the entry points (ogs_capi.cpp).
size_t type_size(int type);
// handle usable on the current device, k >= 1, known type and transpose; refuses
// host-only handles and handles made by ogs_gslib_setup
ogs_status check_common(ogs_handle h, int k, int type, int trans, const char* fn);
// GatherScatter and Scatter write every member: no local node in two rows
ogs_status check_writes(ogs_handle h, const char* fn);
ogs_status check_op(int op, const char* fn);
// members read and written for (kind, mode, transpose), ogsOperator.cpp:71-79, 214-222, 321-339
Pattern pattern_for(const ogs_handle_s* h, int mode, int trans);

}  // namespace ogsgb
