// Scratch layout of one frame and small host helpers shared by the stage launchers.
#pragma once
#include <algorithm>
#include <cstdio>
#include <cstdarg>
#include <utility>
#include "common.cuh"

namespace mlpsp {

// Rows handled by one evaluator work item (one tensor-core M tile), and by an item of the small-group list.
constexpr int kRowsPerItem = 128;
constexpr int kRowsPerSmallItem = 32;
// counters[] slots (device int32)
enum Counter {
  kCtrRecords = 0,   // records appended by the hit pass of the current wave
  kCtrWaveTiles = 1, // tiles on the current wave's list (of all views of a batch)
  kCtrWorkNext = 2,  // dynamic work cursor of the evaluator
  kCtrActive0 = 3,   // active tile count, list 0
  kCtrActive1 = 4,   // active tile count, list 1
  kCtrPairs = 5,     // total candidate pairs (binning)
  kCtrScratch = 6,   // four words (record export, cursors of the sort)
  kCtrWaveRecords = 10, // records of the current wave
  kCtrLongTiles = 11, // tiles on the sort's list of long ones
  kCtrWork = 12,     // evaluator work items of the current wave, and, as the upper half of the same 64-bit word,
  kCtrWorkSmall = 13, // small-group work items
  kNumCounters = 16
};

// One evaluator input record (32 bytes): encoded-input vector, decay and the compositing slot.
struct __align__(16) RecIn {
  float rdx, rdy, rdz, dx;
  float dy, dz, decay;
  uint32_t slot;
};

struct Scratch {
  int32_t* tile_cnt;     // [T+1]
  int32_t* tile_diff;    // [(nty+1)*(ntx+1)] rectangle corners of the count pass (2-D difference array)
  int32_t* tile_fill;    // [T] pairs written per tile; in the fused path, which counts in tile_len, the list of long tiles
  uint2* rect;           // [n]  (x0 | x1<<16, y0 | y1<<16); x0 > x1 marks "culled"
  int32_t* scan_blk;     // block sums of the multi-block scans
  float4* px_state;      // [P] (C.r, C.g, C.b, transmittance)
  float2* px_depth;      // [P] (sum w t, sum w)
  uint32_t* masks32;     // [2*max_pairs] evaluated-hit mask halves per pair
  uint32_t* pair_base;   // [max_pairs] first compositing slot of the pair
  int32_t* prim_cnt;     // [2][n] records per primitive in the current wave (even waves use the first half, odd the second)
  int32_t* prim_pos;     // [n] where the primitive's next record of the current wave goes
  int4* work;            // [max_work] (primitive, first record, rows, 0)
  int4* work_small;      // [max_work_small] the same for items of at most kRowsPerSmallItem rows
  RecIn* rec_in;         // [max_records] primitive-major, reused by every wave
  float4* rec_out;       // [max_records] (R,G,B,alpha) at compositing slots (slots are unique per frame)
  float* rec_t;          // [max_records] t* at compositing slots
  float4* rec_gate;      // [max_records] feature gates at compositing slots
  float* rec_w;          // [max_records] compositing weight trans*alpha of consumed records
  float* rec_tr;         // [max_records] transmittance before the record (record export)
  float4* rec_ext;       // [max_records] (sigma_raw, sigma_logit, relu mask 1, relu mask 2) (record export)
  int32_t* px_cnt;       // [P+2] per-pixel record counts (record export)
  int32_t* px_off;       // [P+2] their exclusive prefix
  uint32_t* used32;      // [2*max_pairs] consumed-record mask halves per pair (when the caller gives none)
  int32_t* active[2];    // [T] each
  FramePlane* plane;     // tangent plane of the frame, and
  float4* tile_rect;     // [T] every tile's rectangle in it (tile pre-test of the fused frame path)
  char* dir_table;       // encoded ray directions (images whose table is at most kDirTableMax)
  int32_t* tile_len;     // [T] candidates per tile that the wave kernels traverse
  int32_t* counters;     // [kNumCounters]
  int64_t max_work;
  int64_t max_work_small;
  int64_t bytes;
};

inline int64_t align_up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

inline int num_tiles(int W, int H, int ts) { return ((W + ts - 1) / ts) * ((H + ts - 1) / ts); }

constexpr int kScanItems = 4096;  // elements per block of the multi-block scans
constexpr int kPrimScanItems = 1024;   // primitives per block of the per-primitive scan (256 threads, four each)

// Used while the table fits beside the frame's other streams in the 126 MB L2: every record then reads 80 bytes of it
constexpr int64_t kDirTableMax = 96ll << 20;
inline int64_t dir_table_bytes(int W, int H) { return 5120ll * (((W + 7) / 8) * (int64_t)((H + 7) / 8)); }

// Carve the scratch block.  base may be null (size query).
inline Scratch carve_scratch(void* base, int n, int W, int H, int ts, int64_t max_pairs, int64_t max_records) {
  Scratch s;
  char* p = static_cast<char*>(base);
  int64_t off = 0;
  const int64_t T = num_tiles(W, H, ts);
  const int64_t P = (int64_t)W * H;
  auto take = [&](int64_t bytes) { char* r = p ? p + off : nullptr; off += align_up(bytes, 256); return r; };
  s.tile_cnt = (int32_t*)take(4 * (T + 1));
  s.tile_diff = (int32_t*)take(4 * (int64_t)((W + ts - 1) / ts + 1) * ((H + ts - 1) / ts + 1));
  s.tile_fill = (int32_t*)take(4 * T);
  s.rect = (uint2*)take(8 * (int64_t)n);
  s.scan_blk = (int32_t*)take(4 * ((std::max<int64_t>(T, P + 1) + kScanItems - 1) / kScanItems + 2));
  s.px_state = (float4*)take(16 * P);
  s.px_depth = (float2*)take(8 * P);
  s.masks32 = (uint32_t*)take(8 * max_pairs);
  s.pair_base = (uint32_t*)take(4 * max_pairs);
  s.prim_cnt = (int32_t*)take(4 * 2 * ((int64_t)n + 4));
  s.prim_pos = (int32_t*)take(4 * (int64_t)n);
  s.max_work = (int64_t)n + max_records / kRowsPerItem + 2;
  s.work = (int4*)take(16 * s.max_work);
  s.max_work_small = 2 * (int64_t)n + 2;
  s.work_small = (int4*)take(16 * s.max_work_small);
  s.rec_in = (RecIn*)take(32 * max_records);
  s.rec_out = (float4*)take(16 * max_records);
  s.rec_t = (float*)take(4 * max_records);
  s.rec_gate = (float4*)take(16 * max_records);
  s.rec_w = (float*)take(4 * max_records);
  s.rec_tr = (float*)take(4 * max_records);
  s.rec_ext = (float4*)take(16 * max_records);
  s.px_cnt = (int32_t*)take(4 * (P + 2));
  s.px_off = (int32_t*)take(4 * (P + 2));
  s.used32 = (uint32_t*)take(8 * max_pairs);
  s.active[0] = (int32_t*)take(4 * T);
  s.active[1] = (int32_t*)take(4 * T);
  s.counters = (int32_t*)take(4 * kNumCounters);
  s.plane = (FramePlane*)take(sizeof(FramePlane));
  s.tile_rect = (float4*)take(16 * T);
  s.tile_len = (int32_t*)take(4 * T);
  s.dir_table = dir_table_bytes(W, H) <= kDirTableMax ? (char*)take(dir_table_bytes(W, H)) : nullptr;
  s.bytes = off;
  return s;
}

// Programmatic dependent launch.  The kernels of a frame form one dependent chain of some thirty launches; with the
// launch attribute below the next kernel of the chain is set up and its CTAs take their places while the previous
// kernel's last CTAs are still running, instead of after the previous grid has drained.  Every kernel launched this
// way begins with chain_wait(), which returns once the previous grid has completed and its writes are visible (so
// the stream's order is kept exactly), and then lets its own successor be set up (chain_release()).  On a kernel
// launched without the attribute both are no-ops.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgs, typename... Args>
inline cudaError_t launch_chained(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(std::forward<Args>(args))...);
}

// A launch serves up to kViewsPerLaunch views of a batch, a row of CTAs each (blockIdx.y): launched view by view, the later waves of
// a batch, a few microseconds of work per view, were mostly launches, and each view ended in a tail of its own (four 500k views of
// 1200 x 680: 4,006 -> 3,720 us, three 200k views of 640 x 480: 1,830 -> 1,687).  Arguments travel by value, 300 bytes a view.
constexpr int kViewsPerLaunch = 8;
template <typename A, int V>
struct Views { A v[V]; int count; };
template <int V> __device__ __forceinline__ int view_of_cta() { return V == 1 ? 0 : (int)blockIdx.y; }

// one launch for the views args[0 .. count)
template <int V, typename A, typename... KArgs, typename... Args>
inline cudaError_t launch_views(void (*kernel)(Views<A, V>, KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A* args,
                                int count, const Args&... rest) {
  Views<A, V> b = {};
  b.count = count;
  for (int v = 0; v < count; ++v) b.v[v] = args[v];
  grid.y = (unsigned)count;
  return launch_chained(kernel, grid, block, smem, st, b, rest...);
}

// Kernel classes for the launch counter and the optional per-class device timing.
enum KernelClass { kKBin = 0, kKSort, kKHits, kKScan, kKFill, kKMlp, kKComposite, kKMisc, kNumKernelClasses };

// RAII marker around the launches of one class: counts them and, when timing is enabled,
// brackets them with CUDA events on the launching stream.
struct LaunchScope {
  LaunchScope(KernelClass k, int launches, cudaStream_t st);
  ~LaunchScope();
  int slot;
  cudaStream_t st;
};

// last-error text (thread-local) for the negative return codes
void set_error(const char* fmt, ...);
int cuda_check(cudaError_t e, const char* what);

#define MLPSP_CUDA_OK(call)                                         \
  do {                                                              \
    int rc__ = ::mlpsp::cuda_check((call), #call);                  \
    if (rc__ != 0) return rc__;                                     \
  } while (0)

#define MLPSP_REQUIRE(cond, code, ...)                              \
  do {                                                              \
    if (!(cond)) { ::mlpsp::set_error(__VA_ARGS__); return (code); }\
  } while (0)

// SMs of the current device (asked once per device)
int sm_count();

// Per-device "first use" marker for settings that CUDA keeps per device (the opt-in dynamic shared-memory
// size of a kernel, for one): a process that drives several GPUs must apply them once on each.  The caller
// keeps one DeviceOnce per setting; first() answers true the first time it is asked with a given device current.
struct DeviceOnce {
  bool seen[64] = {false};
  bool first() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return true;   // unknown device: apply every time
    if (seen[dev]) return false;
    seen[dev] = true;
    return true;
  }
};

// A few words of page-locked host memory that kernels write directly, and an event to wait for the kernel that does so:
// a finding reaches the host without a copy, and without waiting for whatever was launched behind it.  One per host
// thread (and, for the event, device), so calls of different threads do not meet; released with the thread.
struct HostWords {
  static constexpr int kWords = 16;
  int32_t* word = nullptr;
  cudaEvent_t event[64] = {nullptr};
  int open(cudaEvent_t* ev) {
    int dev = 0;
    MLPSP_CUDA_OK(cudaGetDevice(&dev));
    MLPSP_REQUIRE(dev >= 0 && dev < 64, MLPSP_E_LIMIT, "device ordinal %d beyond 63", dev);
    if (!word) MLPSP_CUDA_OK(cudaHostAlloc((void**)&word, 4 * kWords, cudaHostAllocPortable | cudaHostAllocMapped));
    if (!event[dev]) MLPSP_CUDA_OK(cudaEventCreateWithFlags(&event[dev], cudaEventDisableTiming));
    *ev = event[dev];
    return MLPSP_OK;
  }
  ~HostWords() {
    if (word) cudaFreeHost(word);
    for (cudaEvent_t e : event) if (e) cudaEventDestroy(e);
  }
};
HostWords& host_words();

// stage launchers (defined in the .cu files)
// order_lists = false leaves every tile list in scatter order for a following launch_sort(unordered_input = true).
// pretest: write only the (tile, primitive) pairs that some ray of the tile can hit; s.tile_len receives the
// number kept per tile (they sit at the front of the tile's span), tile_offsets stay those of the full lists.
// Pre-tested binning works on what launch_frame_begin has prepared.  view_dev / proj_dev: the matrices in device memory,
// in place of the frame's host matrices.
int launch_bin(const mlpsp_scene* sc, const mlpsp_frame* fr, const Scratch& s, cudaStream_t st, bool order_lists = true,
               bool pretest = false, const float* view_dev = nullptr, const float* proj_dev = nullptr);
// the count pass adds rectangle corners (the corner array fits one CTA's shared memory: frames to about 3,500 x 3,500)
bool bin_uses_corners(const mlpsp_frame* fr);
// everything the fused path reads of a frame or of a batch's views, in one launch for eight of them (see k_frame_begin)
int launch_frame_begin(const mlpsp_scene* sc, const mlpsp_frame* frs, const Scratch* ss, int views, const float* const* rays_raw,
                       bool reset_status, cudaStream_t st);
// launch_bin and launch_sort for the views of a batch that launch_frame_begin has prepared (bin_uses_corners, at least one
// primitive, lists in scatter order), one launch for eight of them
int launch_bin_batch(const mlpsp_scene* sc, const mlpsp_frame* frs, const Scratch* ss, int views, cudaStream_t st);
int launch_sort_batch(const mlpsp_scene* sc, const mlpsp_frame* frs, const Scratch* ss, int views, cudaStream_t st);
int launch_bin_mosaic(const mlpsp_scene* sc, const mlpsp_frame* fr, const Scratch& s, const int32_t* tile_view,
                      const float* views_host, int num_views, cudaStream_t st);
int launch_bin_raycone(const mlpsp_scene* sc, const mlpsp_frame* fr, const Scratch& s, cudaStream_t st);
// cursors [2]: device scratch, the tile cursors of the two sort kernels
// prepared (optional): the scratch of a pre-tested binning, which knows the candidates actually present at the front of every
// tile's span (the rest of the span is filled with -1 in sorted_prims) and lists the long tiles
int launch_sort(const mlpsp_scene* sc, const mlpsp_frame* fr, float* keys_out, cudaStream_t st, bool unordered_input,
                int32_t* cursors, const Scratch* prepared = nullptr);
// lists longer than this are sorted by a CTA
constexpr int kWarpSortMax = 256;
int launch_hit_masks(const mlpsp_scene* sc, const mlpsp_frame* fr, uint64_t* mask_geo, cudaStream_t st);
// lists_refined: launch_frame_begin has prepared the frame and s.tile_len holds the traversal length of every tile
int launch_render_sorted(const mlpsp_scene* sc, const mlpsp_frame* fr, const Scratch& s, cudaStream_t st,
                         bool lists_refined = false);
// rec_ext (optional): per record (sigma_raw, sigma_logit, layer-1 ReLU bitmask, layer-2 ReLU bitmask)
// grid_cap > 0 limits the number of CTAs (a wave that is expected to be idle)
int launch_mlp_f32(const mlpsp_scene* sc, const RecIn* rec_in, const int4* work,
                   const int32_t* counters, float4* rec_out, float4* rec_ext, int out_mode, int32_t* status,
                   cudaStream_t st, int grid_cap = 0);
// bf16: bfloat16 operands (sc->wbf16) instead of binary16 (sc->w16)
// work_small: the wave's small-group list (launch_prim_scan with split_small), or null when every item is on `work`
int launch_mlp_f16(const mlpsp_scene* sc, const RecIn* rec_in, const int4* work,
                   const int32_t* counters, float4* rec_out, float4* rec_ext, int out_mode, int32_t* status,
                   cudaStream_t st, bool bf16 = false, int grid_cap = 0, const int4* work_small = nullptr,
                   const char* dir_table = nullptr);
// The encoded ray directions of a frame (5,120 bytes per tile), for records that name their pixel instead of carrying its
// direction (launch_fill with the table flag; not together with a small-group list or record export).
int launch_encode_directions(const mlpsp_scene* sc, const mlpsp_frame* fr, char* table, cudaStream_t st);
int launch_scan_i32(const int32_t* in, int64_t n, int32_t* blk, int32_t* out, cudaStream_t st);
// counted: the per-pixel counts and their prefix are those of the call before; writes the rows only
int launch_export_records(const mlpsp_scene* sc, const mlpsp_frame* fr, const Scratch& s, int64_t* offsets, int32_t* ids,
                          float* x6, float* raw, int32_t* relu_masks, float* gates, int64_t max_out, int32_t max_hits,
                          int64_t* total_host, int32_t* worst_host, bool counted, cudaStream_t st);

// evaluator output modes
constexpr int kOutAlpha = 0;     // (R,G,B, 1-exp(-softplus(o3)*decay)) scattered to rec.slot
constexpr int kOutSigmaRaw = 1;  // (R,G,B, softplus(o3)) scattered to rec.slot

// feature compositing on the tensor cores (feature_tc.cu): whether this scene's attributes qualify (a binary16 copy,
// 128 / 256 / 384 / 512 channels, 1, 4 or 5 slots), and the launch for a rendered frame (consumed masks in used32)
bool feature_tc_supported(const mlpsp_scene* sc);
int launch_feature_tc(const mlpsp_scene* sc, const mlpsp_frame* fr, const Scratch& s, const uint32_t* used32, cudaStream_t st);

// distance in elements between the count arrays of even and odd waves (keeps the second one 16-byte aligned)
__host__ __device__ inline size_t prim_cnt_stride(int n) { return ((size_t)n + 3) & ~(size_t)3; }
int launch_render_batch(const mlpsp_scene* sc, const mlpsp_frame* frs, const Scratch* ss, int V, cudaStream_t st, bool lists_refined);
int scan_launches(int64_t n);   // kernels launch_scan_i32 launches for n items
// positions of the primitives' records and the evaluator's work items from the per-primitive counts (or from fixed)
// split_small: remainders of at most kRowsPerSmallItem records go to the small-group list (s.work_small)
int launch_prim_scan(const Scratch& s, int n, const int64_t* fixed, int32_t* status, cudaStream_t st, bool split_small, int wave);

}  // namespace mlpsp
