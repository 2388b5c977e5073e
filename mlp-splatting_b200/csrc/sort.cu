// Per-tile depth sort: key = t* of the tile-centre ray against each candidate
// (scannet/cuda/np_tile_kernels.cu:483-518), stable ascending order (1914-1990).
// Keys are positive floats (or the 1e30 sentinel), so their bit patterns order like the values and the
// sort runs on the raw bits of the 64-bit composite (key bits, tie-break).  Lists of up to 256 candidates are sorted by one
// warp (eight tiles per CTA), a bitonic network in registers over 32-bit words that stand for the composites, whose order
// it then corrects; longer lists by a whole CTA, through buckets of their keys.
#include "frame.cuh"

namespace mlpsp {

constexpr int kSortCap = 2048;

// Composite of one candidate: (depth key bits << 32) | tie-break.  FROM_SCATTER: the list comes straight
// from the binning scatter in arbitrary order and holds distinct ids, so the id itself is the tie-break
// (the result is the stable sort of the ascending-id list) and the id is read back from the sorted
// composite.  Otherwise the tie-break is the position in the caller's list (stable sort of that list).
template <bool FROM_SCATTER>
__device__ __forceinline__ unsigned long long make_composite(const float4* __restrict__ geom, int n, int p, int i, V3 o,
                                                             V3 d, int key_mode) {
  float key = MLPSP_SENTINEL_KEY;
  if (p >= 0 && p < n) {
    // key_mode 2 (per-pixel ordering): the pixels sort their own hits later and fall back on the list order for
    // equal hit distances (rays that start inside several primitives meet them all at t = 0), so the list keeps
    // the order it was given, or ascending ids when it comes from the binning scatter.  Bit 2 (value 4) asks for the
    // tile-centre key in the reference kernels' arithmetic (frame.hit_arith = 1).
    if (key_mode == 4) {
      key = tile_key_ref(load_geom_ref(geom, p), o, d);
    } else {
      const Geom g = load_geom(geom, p);
      key = (key_mode & 3) == 2 ? 0.f : ((key_mode & 3) ? tile_key_euclid(g, o, d) : tile_key(g, o, d));
    }
  }
  return ((unsigned long long)__float_as_uint(key) << 32) | (unsigned long long)(uint32_t)(FROM_SCATTER ? p : i);
}

// sorted_prims[s .. s + len) = the sorted list; [s + len, s + span) = -1 (span > len only after a
// pre-tested binning, whose dropped pairs leave the end of the tile's span unused)
template <bool FROM_SCATTER>
__device__ __forceinline__ void write_sorted(const unsigned long long* buf, const int32_t* tile_prims,
                                             int32_t* __restrict__ sorted_prims, float* __restrict__ keys_out, int s,
                                             int len, int span, int first, int step) {
  for (int i = first; i < span; i += step) {
    if (i < len) {
      const unsigned long long kv = buf[i];
      sorted_prims[s + i] = FROM_SCATTER ? (int32_t)(uint32_t)kv : tile_prims[s + (int)(uint32_t)kv];
      if (keys_out) keys_out[s + i] = __uint_as_float((uint32_t)(kv >> 32));
    } else {
      sorted_prims[s + i] = -1;
    }
  }
}

constexpr int kTilesPerCta = 8;
constexpr int kLongDraw = 4;
constexpr int kLongCtas = 6;            // CTAs of k_sort_long per SM
constexpr int kFixPasses = 8;
constexpr int kBucketMax = 128;         // candidates in one bucket of a list that is sorted by buckets

// ---- warp-level bitonic sort in registers: lane l holds the elements r * 32 + l, r < PER ----
// A compare-exchange at distance j >= 32 pairs two registers of the same lane; at distance j < 32 it pairs the same
// register of the lanes l and l ^ j, one shuffle each way.  Ascending where the element index has bit k clear.
// No shared memory and no barrier: the stages of a tile follow one another at the latency of a shuffle.
__device__ __forceinline__ unsigned long long shfl_xor_u64(unsigned long long v, int j) {
  const uint32_t lo = __shfl_xor_sync(0xffffffffu, (uint32_t)v, j);
  const uint32_t hi = __shfl_xor_sync(0xffffffffu, (uint32_t)(v >> 32), j);
  return ((unsigned long long)hi << 32) | lo;
}

__device__ __forceinline__ unsigned long long shfl_xor_any(unsigned long long v, int j) { return shfl_xor_u64(v, j); }
__device__ __forceinline__ uint32_t shfl_xor_any(uint32_t v, int j) { return __shfl_xor_sync(0xffffffffu, v, j); }

template <int PER, typename T>
__device__ __forceinline__ void warp_bitonic_regs(T (&v)[PER], int lane) {
  constexpr int N = PER * 32;
#pragma unroll
  for (int k = 2; k <= N; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
        const int jr = j >> 5;
#pragma unroll
        for (int r = 0; r < PER; ++r) {
          if ((r & jr) == 0) {
            const bool up = ((r * 32) & k) == 0;          // k >= 64 here: the lane bits do not reach it
            const T mn = min(v[r], v[r | jr]), mx = max(v[r], v[r | jr]);
            v[r] = up ? mn : mx;
            v[r | jr] = up ? mx : mn;
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < PER; ++r) {
          const T a = v[r], b = shfl_xor_any(a, j);
          const bool up = ((r * 32 + lane) & k) == 0;
          const bool lower = (lane & j) == 0;
          v[r] = lower == up ? min(a, b) : max(a, b);
        }
      }
    }
  }
}

// The CTA sorts s_buf[0 .. len) by a bitonic network in shared memory, two of its stages (distances j and j / 2) per pass: the
// way of lists whose keys crowd into few buckets.  Loops and not an unrolled network in registers, so that it adds neither
// registers nor code to the kernel around it.  In passes at distances up to 64 a warp's exchanges stay among the same
// 128 elements, and only the warp has to keep step.
template <int THREADS>
__device__ __forceinline__ void cta_bitonic_shared(unsigned long long* s_buf, int len) {
  int n = 128;
  while (n < len) n <<= 1;
  for (int e = len + (int)threadIdx.x; e < n; e += THREADS) s_buf[e] = ~0ull;
  __syncthreads();
  auto exchange = [](unsigned long long& x, unsigned long long& y, bool up) {
    const unsigned long long lo = min(x, y), hi = max(x, y);
    x = up ? lo : hi;
    y = up ? hi : lo;
  };
#pragma unroll 1
  for (int k = 2; k <= n; k <<= 1) {
#pragma unroll 1
    for (int j = k >> 1; j > 0; j >>= 2) {
      const int q = max(j >> 1, 1);
#pragma unroll 1
      for (int i = threadIdx.x; i < n / 4; i += THREADS) {
        unsigned long long* p = s_buf + ((i & ~(q - 1)) << 2 | (i & (q - 1)));
        const int e = (int)(p - s_buf);
        unsigned long long v0 = p[0], v1 = p[q], v2 = p[2 * q], v3 = p[3 * q];
        const bool up = (e & k) == 0;
        if (j > 1) { exchange(v0, v2, up); exchange(v1, v3, up); }
        exchange(v0, v1, up);
        exchange(v2, v3, ((e + 2 * q) & k) == 0);
        p[0] = v0; p[q] = v1; p[2 * q] = v2; p[3 * q] = v3;
      }
      if (max(j, j >> 2 ? j >> 2 : k) > 64) __syncthreads();
      else __syncwarp();
    }
  }
}

// One tile's list (len <= PER * 32) sorted by one warp in registers and written out; buf: 256 composites of shared memory.
// The network runs on 32-bit words -- the key's distance from the list's smallest, cut to 24 bits, and the element's place --
// which costs a third of the instructions of 64-bit ones; the composites then move once, and neighbours that the cut has left
// out of order are exchanged.  Lists with long runs of equal keys (more than kFixPasses exchanges deep) fall back on the
// 64-bit network.
template <int PER, bool FROM_SCATTER>
__device__ __forceinline__ void sort_tile_in_registers(const float4* __restrict__ geom, int n, const int32_t* tile_prims,
                                                       int32_t* __restrict__ sorted_prims, float* __restrict__ keys_out,
                                                       int s, int len, int span, V3 o, V3 d, int key_mode, int lane,
                                                       unsigned long long* buf) {
  unsigned long long c[PER];
  uint32_t v[PER], kmin = 0xffffffffu, kmax = 0u;
#pragma unroll
  for (int r = 0; r < PER; ++r) {
    const int e = r * 32 + lane;
    c[r] = e < len ? make_composite<FROM_SCATTER>(geom, n, tile_prims[s + e], e, o, d, key_mode) : ~0ull;
    if (e < len) {
      buf[e] = c[r];
      const uint32_t key = (uint32_t)(c[r] >> 32);
      kmin = min(kmin, key);
      if (key != __float_as_uint(MLPSP_SENTINEL_KEY)) kmax = max(kmax, key);
    }
  }
  kmin = __reduce_min_sync(0xffffffffu, kmin);
  kmax = __reduce_max_sync(0xffffffffu, kmax);
  const int cut = max(0, 8 - __clz((int)(kmax >= kmin ? kmax - kmin : 0u)));
#pragma unroll
  for (int r = 0; r < PER; ++r) {
    const int e = r * 32 + lane;
    v[r] = e < len ? (min(((uint32_t)(c[r] >> 32) - kmin) >> cut, 0xffffffu) << 8) | (uint32_t)e : 0xffffffffu;
  }
  warp_bitonic_regs<PER>(v, lane);
  __syncwarp();
#pragma unroll
  for (int r = 0; r < PER; ++r) c[r] = r * 32 + lane < len ? buf[v[r] & 255u] : ~0ull;
  for (int pass = 0;; ++pass) {
    __syncwarp();
#pragma unroll
    for (int r = 0; r < PER; ++r) if (r * 32 + lane < len) buf[r * 32 + lane] = c[r];
    __syncwarp();
    bool wrong = false;
#pragma unroll
    for (int r = 0; r < PER; ++r) if (r * 32 + lane + 1 < len) wrong = wrong || c[r] > buf[r * 32 + lane + 1];
    if (!__any_sync(0xffffffffu, wrong)) break;
    if (pass == kFixPasses) {
      warp_bitonic_regs<PER>(c, lane);
      break;
    }
    for (int parity = 0; parity < 2; ++parity) {
      for (int e = 2 * lane + parity; e < len - 1; e += 64) {
        const unsigned long long a = buf[e], b = buf[e + 1];
        if (a > b) { buf[e] = b; buf[e + 1] = a; }
      }
      __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < PER; ++r) if (r * 32 + lane < len) c[r] = buf[r * 32 + lane];
  }
#pragma unroll
  for (int r = 0; r < PER; ++r) {
    const int e = r * 32 + lane;
    if (e < len) {
      sorted_prims[s + e] = FROM_SCATTER ? (int32_t)(uint32_t)c[r] : tile_prims[s + (int)(uint32_t)c[r]];
      if (keys_out) keys_out[s + e] = __uint_as_float((uint32_t)(c[r] >> 32));
    }
  }
  for (int i = len + lane; i < span; i += 32) sorted_prims[s + i] = -1;
  __syncwarp();
}

// end of k_sort_tiles: the grid may not complete before the grid it was launched behind has
__device__ __forceinline__ void sort_tiles_done() {
  if ((threadIdx.x & 31) == 0) chain_wait();
}

// Short lists: one warp per tile, eight tiles per CTA.  Tiles with more than kWarpSortMax candidates are left to
// k_sort_long, which gives each of them a CTA of its own.
// cursors: [0] of k_sort_long, [1] of k_sort_tiles.  long_tiles, long_count: the tiles of k_sort_long, or null
struct SortArgs {
  const float* rays_o; const float* rays_d; const int32_t* tile_offsets; const int32_t* tile_prims; int32_t* sorted_prims; float* keys_out;
  int32_t* cursors; const int32_t* list_len; const int32_t* long_tiles; const int32_t* long_count; int32_t* status;
};
struct SortShape { int W, H, ts, ntx, T, key_mode; };

template <bool IDSORT, int V>
__global__ void __launch_bounds__(256, 6) k_sort_tiles(const __grid_constant__ Views<SortArgs, V> views, const float4* __restrict__ geom, int n,
                                                       const SortShape shape, int cap) {
  const SortArgs& a = views.v[view_of_cta<V>()];
  const float* __restrict__ rays_o = a.rays_o; const float* __restrict__ rays_d = a.rays_d;
  const int32_t* __restrict__ tile_offsets = a.tile_offsets; const int32_t* tile_prims = a.tile_prims;
  int32_t* __restrict__ sorted_prims = a.sorted_prims; float* __restrict__ keys_out = a.keys_out;
  int32_t* __restrict__ cursor = a.cursors + 1;
  const int32_t* __restrict__ list_len = a.list_len;
  int32_t* __restrict__ status = a.status;
  const int W = shape.W, H = shape.H, ts = shape.ts, ntx = shape.ntx, T = shape.T, key_mode = shape.key_mode;
  __shared__ unsigned long long s_buf[8][kWarpSortMax];
  // Launched behind k_sort_long as its programmatic dependent WITHOUT waiting for it here: the two kernels sort
  // disjoint tiles and run side by side.  What this kernel reads (the binned lists, the status word) was complete
  // before k_sort_long's CTAs got past their own wait, and none of this kernel's CTAs starts before all of them
  // have.  The wait is at the end instead (sort_tiles_done), so that this grid's completion implies the other's.
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) { sort_tiles_done(); return; }
  const int lane = threadIdx.x & 31;
  // warps draw tiles from a shared cursor: list lengths differ by two orders of magnitude, and
  // a fixed deal would leave most warps of a CTA waiting for the one with the longest list
  for (;;) {
  int tile = 0;
  if (lane == 0) tile = atomicAdd(cursor, 1);
  tile = __shfl_sync(0xffffffffu, tile, 0);
  if (tile >= T) { sort_tiles_done(); return; }
  const int s = tile_offsets[tile];
  const int span = min(tile_offsets[tile + 1] - s, cap);
  const int len = list_len ? min(list_len[tile], span) : span;
  if (list_len && lane == 0 && len > 0) atomicAdd(status + MLPSP_ST_PAIRS_KEPT, len);
  if (len > kWarpSortMax) continue;      // k_sort_long's
  if (len <= 0) {
    for (int i = lane; i < span; i += 32) sorted_prims[s + i] = -1;
    continue;
  }
  const int tx = tile % ntx, ty = tile / ntx;
  const int cx = min(tx * ts + (ts >> 1), W - 1), cy = min(ty * ts + (ts >> 1), H - 1);
  const int64_t pc = (int64_t)cy * W + cx;
  const V3 o = load3(rays_o, pc), d = load3(rays_d, pc);
  if (len <= 32) sort_tile_in_registers<1, IDSORT>(geom, n, tile_prims, sorted_prims, keys_out, s, len, span, o, d, key_mode, lane, s_buf[threadIdx.x >> 5]);
  else if (len <= 64) sort_tile_in_registers<2, IDSORT>(geom, n, tile_prims, sorted_prims, keys_out, s, len, span, o, d, key_mode, lane, s_buf[threadIdx.x >> 5]);
  else if (len <= 128) sort_tile_in_registers<4, IDSORT>(geom, n, tile_prims, sorted_prims, keys_out, s, len, span, o, d, key_mode, lane, s_buf[threadIdx.x >> 5]);
  else sort_tile_in_registers<8, IDSORT>(geom, n, tile_prims, sorted_prims, keys_out, s, len, span, o, d, key_mode, lane, s_buf[threadIdx.x >> 5]);
  }
}

// One tile's list (len <= PER * THREADS) sorted by the CTA and written out.  The keys' range is cut into CAP buckets: a
// candidate draws its place in its bucket with one atomic in shared memory, a prefix over the buckets gives their starts, the
// composites move there, and each one's place inside the bucket, of a handful, is the number of smaller ones.  A list
// with more than kBucketMax candidates in one bucket (an outlier that stretches the range of many equal keys) takes the
// network.  (A place costs a read per candidate of the bucket, the network some 36 passes over all: lists of a thin wall with
// another behind it, sort of a 400,000-primitive view, network beyond 32 in a bucket 141 us, beyond 64, 128, 200: 102, 101, 100.)
// s_buf: CAP composites, s_bucket: CAP words, s_range: a word pair per warp.
template <int PER, int THREADS, int CAP, bool IDSORT>
__device__ __forceinline__ void sort_tile_by_cta(const float4* __restrict__ geom, int n, const int32_t* tile_prims,
                                                 int32_t* __restrict__ sorted_prims, float* __restrict__ keys_out, int s, int len, int span,
                                                 V3 o, V3 d, int key_mode, unsigned long long* s_buf, uint32_t* s_bucket, uint2* s_range) {
  constexpr int OWN = CAP / THREADS;                  // buckets per thread in the prefix
  static_assert(OWN % 4 == 0, "buckets are read four at a time");
  const int tid = threadIdx.x, lane = tid & 31;
  unsigned long long c[PER];
  uint32_t kmin = 0xffffffffu, kmax = 0u;
  for (int i = tid; i < CAP / 4; i += THREADS) reinterpret_cast<uint4*>(s_bucket)[i] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int r = 0; r < PER; ++r) {
    const int i = r * THREADS + tid;
    c[r] = ~0ull;
    if (i < len) {
      c[r] = make_composite<IDSORT>(geom, n, tile_prims[s + i], i, o, d, key_mode);
      const uint32_t key = (uint32_t)(c[r] >> 32);
      kmin = min(kmin, key);
      if (key != __float_as_uint(MLPSP_SENTINEL_KEY)) kmax = max(kmax, key);
    }
  }
  kmin = __reduce_min_sync(0xffffffffu, kmin);
  kmax = __reduce_max_sync(0xffffffffu, kmax);
  if (lane == 0) s_range[tid >> 5] = make_uint2(kmin, kmax);
  __syncthreads();
#pragma unroll
  for (int w = 0; w < THREADS / 32; ++w) { kmin = min(kmin, s_range[w].x); kmax = max(kmax, s_range[w].y); }
  // the map from composites to buckets is monotone: each of its operations is.  Where all keys but sentinels are equal (lists
  // for per-pixel ordering), the tie-breaks take the keys' place, and sentinels the last bucket
  const bool equal = kmax <= kmin;
  const float scale = (float)(CAP - 1) / (float)(equal ? (IDSORT ? n : len) : (int)(kmax - kmin));
  auto bucket_of = [&](unsigned long long v) {
    const uint32_t key = (uint32_t)(v >> 32);
    const float x = equal ? (key == kmin ? (float)(uint32_t)v : (float)CAP * 4294967296.f) : (float)(key - kmin);
    return (uint32_t)fminf(x * scale, (float)(CAP - 1));
  };
  uint32_t place[(PER + 3) / 4] = {};                 // in its bucket, a byte each (deeper buckets take the network)
  static_assert(kBucketMax < 255, "places of a byte");
#pragma unroll
  for (int r = 0; r < PER; ++r)
    if (r * THREADS + tid < len)
      place[r >> 2] |= min(atomicAdd(s_bucket + bucket_of(c[r]), 1u), 255u) << (r & 3) * 8;
  __syncthreads();
  uint32_t sum = 0u, deepest = 0u;
  uint4* own_s = reinterpret_cast<uint4*>(s_bucket) + tid * (OWN / 4);
  uint4 own[OWN / 4];
#pragma unroll
  for (int j = 0; j < OWN / 4; ++j) {
    const uint4 q = own[j] = own_s[j];
    deepest = max(max(max(deepest, q.x), q.y), max(q.z, q.w));
    sum += q.x + q.y + q.z + q.w;
  }
  uint32_t upto = sum;
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, upto, k);
    if (lane >= k) upto += u;
  }
  if (lane == 31) s_range[tid >> 5].x = upto;         // (all have read the ranges before the barrier above)
  if (__syncthreads_or(deepest > kBucketMax)) {
#pragma unroll
    for (int r = 0; r < PER; ++r) if (r * THREADS + tid < len) s_buf[r * THREADS + tid] = c[r];
    cta_bitonic_shared<THREADS>(s_buf, len);
    write_sorted<IDSORT>(s_buf, tile_prims, sorted_prims, keys_out, s, len, span, tid, THREADS);
    __syncthreads();
    return;
  }
  uint32_t start = upto - sum;
  for (int w = 0; w < (tid >> 5); ++w) start += s_range[w].x;
#pragma unroll
  for (int j = 0; j < OWN / 4; ++j) {
    const uint4 q = own[j];
    own_s[j] = make_uint4(start, start + q.x, start + q.x + q.y, start + q.x + q.y + q.z);
    start += q.x + q.y + q.z + q.w;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < PER; ++r)
    if (r * THREADS + tid < len) s_buf[s_bucket[bucket_of(c[r])] + (place[r >> 2] >> (r & 3) * 8 & 0xffu)] = c[r];
  __syncthreads();
  for (int e = tid; e < span; e += THREADS) {
    if (e >= len) { sorted_prims[s + e] = -1; continue; }
    const unsigned long long v = s_buf[e];
    const uint32_t b = bucket_of(v);
    const int lo = (int)s_bucket[b], hi = b + 1 < CAP ? (int)s_bucket[b + 1] : len;
    int at = s + lo;
    for (int j = lo; j < hi; ++j) at += s_buf[j] < v ? 1 : 0;
    sorted_prims[at] = IDSORT ? (int32_t)(uint32_t)v : tile_prims[s + (int)(uint32_t)v];
    if (keys_out) keys_out[at] = __uint_as_float((uint32_t)(v >> 32));
  }
  __syncthreads();
}

// Long lists (more than kWarpSortMax candidates): one CTA per such tile.  Launched before k_sort_tiles, which runs beside it.
// Bound: the gathers of the candidates' geometry and shared memory.  Both kernels on the 100k frame, a 500k view and four of
// them in one batch: the bitonic network in registers on every list, 64 registers a thread, 61, 77 and 311 us; five CTAs per SM
// drawing from the list of long tiles 60, 72 and 279; buckets 55, 58 and 208; six CTAs per SM (40 registers, of which the
// network in registers, as the way of crowded lists, spilled 380 bytes) 52, 58 and 198; that network in shared memory, by
// loops (spills 40 bytes), 52, 56 and 196.  Given lists, 3,456 of 12,750 longer than 256: 112 -> 88, all keys equal 175 -> 63.
template <int THREADS, int CAP, bool IDSORT, int V>
__global__ void __launch_bounds__(THREADS, kLongCtas) k_sort_long(const __grid_constant__ Views<SortArgs, V> views, const float4* __restrict__ geom, int n,
                                                       const SortShape shape) {
  const SortArgs& a = views.v[view_of_cta<V>()];
  const float* __restrict__ rays_o = a.rays_o; const float* __restrict__ rays_d = a.rays_d;
  const int32_t* __restrict__ tile_offsets = a.tile_offsets; const int32_t* tile_prims = a.tile_prims;
  int32_t* __restrict__ sorted_prims = a.sorted_prims; float* __restrict__ keys_out = a.keys_out;
  int32_t* __restrict__ cursor = a.cursors;
  const int32_t* __restrict__ list_len = a.list_len;
  const int32_t* __restrict__ status = a.status;
  const int W = shape.W, H = shape.H, ts = shape.ts, ntx = shape.ntx, T = shape.T, key_mode = shape.key_mode;
  __shared__ __align__(16) unsigned long long s_buf[CAP];
  __shared__ __align__(16) uint32_t s_bucket[CAP];
  __shared__ uint2 s_range[THREADS / 32];
  static_assert(CAP == 2048, "places of eleven bits");
  __shared__ int s_draw;
  __shared__ int4 s_list[kLongDraw];           // tile, start, span, length
  chain_wait();
  chain_release();
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  // CTAs draw tiles from a shared cursor.  The pre-tested binning lists the long ones as their fill passes the limit, the
  // densest first, so that every draw is one sort and the last ones are short.  Without that list a draw is
  // kLongDraw tiles a band of the image apart, since long lists cluster in its dense part.
  const int bands = (T + kLongDraw - 1) / kLongDraw;
  const int32_t* __restrict__ long_tiles = a.long_tiles;
  const int draws = long_tiles ? *a.long_count : bands, per_draw = long_tiles ? 1 : kLongDraw;
  int draw = 0;
  if (threadIdx.x == 0) draw = atomicAdd(cursor, 1);
  for (;;) {
    if (threadIdx.x == 0) { s_draw = draw; draw = atomicAdd(cursor, 1); }
    __syncthreads();
    if (s_draw >= draws) return;
    if (threadIdx.x < per_draw) {
      const int tile = long_tiles ? long_tiles[s_draw] : s_draw + threadIdx.x * bands;
      int4 e = make_int4(tile, 0, 0, 0);
      if (tile < T) {
        e.y = tile_offsets[tile];
        e.z = min(tile_offsets[tile + 1] - e.y, CAP);
        e.w = list_len ? min(list_len[tile], e.z) : e.z;
      }
      s_list[threadIdx.x] = e;
    }
    __syncthreads();
    for (int u = 0; u < per_draw; ++u) {
    const int tile = s_list[u].x, s = s_list[u].y, span = s_list[u].z, len = s_list[u].w;
    if (len <= kWarpSortMax) continue;        // k_sort_tiles' (uniform over the CTA)
    const int tx = tile % ntx, ty = tile / ntx;
    const int cx = min(tx * ts + (ts >> 1), W - 1), cy = min(ty * ts + (ts >> 1), H - 1);
    const int64_t pc = (int64_t)cy * W + cx;
    const V3 o = load3(rays_o, pc), d = load3(rays_d, pc);
    if (len <= CAP / 4) sort_tile_by_cta<CAP / 4 / THREADS, THREADS, CAP, IDSORT>(geom, n, tile_prims, sorted_prims, keys_out, s, len, span, o, d, key_mode, s_buf, s_bucket, s_range);
    else if (len <= CAP / 2) sort_tile_by_cta<CAP / 2 / THREADS, THREADS, CAP, IDSORT>(geom, n, tile_prims, sorted_prims, keys_out, s, len, span, o, d, key_mode, s_buf, s_bucket, s_range);
    else sort_tile_by_cta<CAP / THREADS, THREADS, CAP, IDSORT>(geom, n, tile_prims, sorted_prims, keys_out, s, len, span, o, d, key_mode, s_buf, s_bucket, s_range);
    }
  }
}

template <bool IDSORT, int V>
static void launch_sort_kernels(const mlpsp_scene* sc, const mlpsp_frame* fr, const SortArgs* args, int views, cudaStream_t st) {
  const int T = num_tiles(fr->width, fr->height, fr->tile), ntx = (fr->width + fr->tile - 1) / fr->tile, sms = sm_count();
  // k_sort_tiles runs beside k_sort_long, whose CTAs must all have started for that: they share the SMs between the views
  const int grid = std::min((T + kTilesPerCta - 1) / kTilesPerCta, sms * 6);
  const int grid_long = std::min(T, (sms * kLongCtas + views - 1) / views);
  // the reference kernels' arithmetic exists for the tile-centre key only (sort_key 0)
  const int key_mode = fr->sort_key | ((fr->hit_arith == 1 && fr->sort_key == 0) ? 4 : 0);
  const SortShape shape = {fr->width, fr->height, fr->tile, ntx, T, key_mode};
  const float4* geom = (const float4*)sc->geom;
  launch_views<V>(k_sort_long<256, kSortCap, IDSORT, V>, dim3(grid_long), dim3(256), 0, st, args, views, geom, sc->n, shape);
  launch_views<V>(k_sort_tiles<IDSORT, V>, dim3(grid), dim3(256), 0, st, args, views, geom, sc->n, shape, kSortCap);
}

int launch_sort_batch(const mlpsp_scene* sc, const mlpsp_frame* frs, const Scratch* ss, int views, cudaStream_t st) {
  constexpr int N = kViewsPerLaunch;
  LaunchScope scope(kKSort, 2 * ((views + N - 1) / N), st);
  for (int v0 = 0; v0 < views; v0 += N) {
    SortArgs a[N];
    const int count = std::min(N, views - v0);
    for (int q = 0; q < count; ++q) {
      const mlpsp_frame* fr = frs + v0 + q;
      const Scratch& s = ss[v0 + q];
      a[q] = {fr->rays_o, fr->rays_d, fr->tile_offsets, fr->tile_prims, fr->sorted_prims, nullptr, s.counters + kCtrScratch + 2, s.tile_len,
              s.tile_fill, s.counters + kCtrLongTiles, fr->status};
    }
    launch_sort_kernels<true, N>(sc, frs, a, count, st);
  }
  return cuda_check(cudaGetLastError(), "sort_tiles");
}

int launch_sort(const mlpsp_scene* sc, const mlpsp_frame* fr, float* keys_out, cudaStream_t st, bool unordered_input,
                int32_t* cursors, const Scratch* prepared) {
  MLPSP_REQUIRE(fr->tile_capacity > 0 && fr->tile_capacity <= kSortCap, MLPSP_E_LIMIT,
                "tile_capacity must be in [1, %d]", kSortCap);
  MLPSP_REQUIRE(cursors, MLPSP_E_ARG, "sort: scratch for the tile cursors missing");
  // a frame that k_frame_begin prepared starts with both cursors at zero
  if (!prepared) MLPSP_CUDA_OK(cudaMemsetAsync(cursors, 0, 8, st));
  LaunchScope scope(kKSort, 2, st);
  const SortArgs a = {fr->rays_o, fr->rays_d, fr->tile_offsets, fr->tile_prims, fr->sorted_prims, keys_out, cursors,
                      prepared ? prepared->tile_len : nullptr, prepared ? prepared->tile_fill : nullptr,
                      prepared ? prepared->counters + kCtrLongTiles : nullptr, fr->status};
  if (unordered_input) launch_sort_kernels<true, 1>(sc, fr, &a, 1, st);
  else launch_sort_kernels<false, 1>(sc, fr, &a, 1, st);
  return cuda_check(cudaGetLastError(), "sort_tiles");
}

}  // namespace mlpsp
