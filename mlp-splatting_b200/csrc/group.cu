// Record grouping helpers that mirror scannet/primitive_csr.py:23-29 (group_records: stable sort of
// record ids by primitive + bincount + cumsum) and scannet/primitive_gemm.py:186-203
// (prepare_groups: fixed-size segments of every primitive's record range).
//
// group_records is a device-wide stable LSD radix sort of (primitive id, record index) pairs with digits of up to
// eight bits (two passes up to 65,535 primitives, three beyond).  A block owns 4,096 consecutive items, a warp 512 of
// them in order.  Per pass: the blocks' digit counts, one scan per digit over the blocks, and the scatter, which ranks
// the items of a warp with match.any against per-warp digit counters, orders the block's items by digit in shared
// memory and writes them out in runs, so equal ids keep their record order; the last pass writes the permutation and, when
// rows are to be moved, its inverse.  The last kernel writes the CSR offsets (by binary search in the sorted keys: no
// counting pass) and the caller's record rows in the new order.
#include "frame.cuh"

namespace mlpsp {

int launch_scan_i32(const int32_t* in, int64_t n, int32_t* blk, int32_t* out, cudaStream_t st);

constexpr int kGsThreads = 256, kGsRounds = 16, kGsItems = kGsThreads * kGsRounds, kGsWarps = kGsThreads / 32;
constexpr int kGsBins = 256;

// an id outside [0, nprim) sorts behind every primitive, as key nprim
__device__ __forceinline__ uint32_t gs_key(int32_t id, int nprim) { return (uint32_t)id < (uint32_t)nprim ? (uint32_t)id : (uint32_t)nprim; }

// digit counts of every block, digit-major: ghist[digit * nblocks + block]
template <bool FIRST>
__global__ void __launch_bounds__(kGsThreads) k_gs_hist(const uint32_t* __restrict__ keys, int64_t n, int nprim, int shift,
                                                        int dbits, int nblocks, int32_t* __restrict__ ghist) {
  chain_wait();
  chain_release();
  __shared__ int h[kGsBins];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kGsItems;
  const uint32_t dmask = (1u << dbits) - 1u;
#pragma unroll
  for (int r = 0; r < kGsRounds; ++r) {
    const int64_t i = base + r * kGsThreads + threadIdx.x;
    if (i < n) {
      const uint32_t k = FIRST ? gs_key((int32_t)keys[i], nprim) : keys[i];
      atomicAdd(&h[(k >> shift) & dmask], 1);
    }
  }
  __syncthreads();
  if (threadIdx.x < (1u << dbits)) ghist[(size_t)threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

// block = one digit: exclusive prefix of its counts over the blocks, in place, and its total
__global__ void __launch_bounds__(kGsThreads) k_gs_scan(int nblocks, int32_t* __restrict__ ghist, int32_t* __restrict__ dtot) {
  chain_wait();
  chain_release();
  __shared__ int warp_sums[32];
  int32_t* row = ghist + (size_t)blockIdx.x * nblocks;
  int run = 0;
  for (int b0 = 0; b0 < nblocks; b0 += kGsThreads) {
    const int b = b0 + threadIdx.x;
    const int v = b < nblocks ? row[b] : 0;
    int total;
    const int ex = block_exclusive_scan(v, warp_sums, total);
    if (b < nblocks) row[b] = run + ex;
    run += total;
  }
  if (threadIdx.x == 0) dtot[blockIdx.x] = run;
}

// LAST: order and inverse (where given) instead of vals_out
template <bool FIRST, bool LAST>
__global__ void __launch_bounds__(kGsThreads) k_gs_scatter(
    const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals, int64_t n, int nprim, int shift, int dbits, int nblocks,
    const int32_t* __restrict__ ghist, const int32_t* __restrict__ dtot, uint32_t* __restrict__ keys_out,
    uint32_t* __restrict__ vals_out, int64_t* __restrict__ order, uint32_t* __restrict__ inverse) {
  chain_wait();
  chain_release();
  __shared__ int s_cnt[kGsWarps][kGsBins];   // running digit counts per warp, then each warp's first position of a digit
  __shared__ int s_dst[kGsBins];             // global position of the block's first item of a digit, minus its position here
  __shared__ uint2 s_item[kGsItems];
  __shared__ int warp_sums[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t base = (int64_t)blockIdx.x * kGsItems;
  const uint32_t dmask = (1u << dbits) - 1u, lt = (1u << lane) - 1u;
  for (int i = lane; i < kGsBins; i += 32) s_cnt[warp][i] = 0;
  __syncwarp();
  uint32_t key[kGsRounds];
  int rank[kGsRounds];
#pragma unroll
  for (int r = 0; r < kGsRounds; ++r) {
    const int64_t i = base + warp * (kGsRounds * 32) + r * 32 + lane;
    key[r] = i < n ? (FIRST ? gs_key((int32_t)keys[i], nprim) : keys[i]) : 0xffffffffu;
  }
#pragma unroll
  for (int r = 0; r < kGsRounds; ++r) {
    const bool valid = base + warp * (kGsRounds * 32) + r * 32 + lane < n;
    const uint32_t d = valid ? ((key[r] >> shift) & dmask) : 0x1000u;
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    const int before = valid ? s_cnt[warp][d] : 0;
    rank[r] = before + __popc(peers & lt);
    __syncwarp();
    if (valid && (peers & lt) == 0u) s_cnt[warp][d] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // thread = digit: the warps' first positions inside the digit, the digit's first position in the block and in the output
  int mine = 0;
#pragma unroll
  for (int w = 0; w < kGsWarps; ++w) { const int c = s_cnt[w][tid]; s_cnt[w][tid] = mine; mine += c; }
  int total;
  const int local = block_exclusive_scan(mine, warp_sums, total);
  const bool live = tid < (1 << dbits);
  int unused;
  const int global = block_exclusive_scan(live ? dtot[tid] : 0, warp_sums, unused);
  s_dst[tid] = live ? global + ghist[(size_t)tid * nblocks + blockIdx.x] - local : 0;
#pragma unroll
  for (int w = 0; w < kGsWarps; ++w) s_cnt[w][tid] += local;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kGsRounds; ++r) {
    const int64_t i = base + warp * (kGsRounds * 32) + r * 32 + lane;
    if (i < n) {
      const uint32_t d = (key[r] >> shift) & dmask;
      s_item[s_cnt[warp][d] + rank[r]] = make_uint2(key[r], FIRST ? (uint32_t)i : vals[i]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kGsRounds; ++r) {
    const int j = r * kGsThreads + tid;
    if (j < total) {
      const uint2 it = s_item[j];
      const int dst = s_dst[(it.x >> shift) & dmask] + j;
      keys_out[dst] = it.x;
      if (!LAST) vals_out[dst] = it.y;
      else {
        order[dst] = (int64_t)it.y;
        if (inverse) inverse[it.y] = (uint32_t)dst;
      }
    }
  }
}

// CSR offsets and, where given, the records' rows in primitive-major order.  Rows are read in the order they come in and
// written to their places: a primitive's records come from neighbouring pixels, a few hundred kilobytes apart at most, so
// the pieces of a line meet in L2 and memory sees whole lines both ways.  (The other way round, whole lines written and
// rows fetched, memory delivers 64 bytes for each 8, 16 or 24.)  Bound: memory; 4.3 M records of 48 bytes 365 -> 182 us, the
// scattered order of the last pass (31 us more) included.
// Three consecutive threads move the three 8-byte words of an x6 row.
__global__ void __launch_bounds__(256) k_gs_finish(
    const uint32_t* __restrict__ keys, const uint32_t* __restrict__ inverse, int64_t n, int nprim,
    int64_t* __restrict__ offsets, const float2* __restrict__ x6, const float4* __restrict__ d4, const int2* __restrict__ masks,
    float2* __restrict__ x6_out, float4* __restrict__ d4_out, int2* __restrict__ masks_out) {
  chain_wait();
  chain_release();
  __shared__ uint32_t s_dst[256];
  const int64_t base = (int64_t)blockIdx.x * 256;
  const int64_t i = base + threadIdx.x;
  const int rows = (int)max((int64_t)0, min((int64_t)256, n - base));
  if (i <= nprim) {      // first position whose key is not below i
    int64_t lo = 0, hi = n;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (__ldg(keys + mid) < (uint32_t)i) lo = mid + 1; else hi = mid;
    }
    offsets[i] = lo;
  }
  if (!inverse) return;
  if (i < n) {
    const uint32_t v = inverse[i];
    s_dst[threadIdx.x] = v;
    if (d4) d4_out[v] = __ldg(d4 + i);
    if (masks) masks_out[v] = __ldg(masks + i);
  }
  if (!x6) return;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 3; ++u) {
    const int w = u * 256 + threadIdx.x;
    if (w < rows * 3) x6_out[(size_t)s_dst[w / 3] * 3 + w % 3] = __ldg(x6 + base * 3 + w);
  }
}

// total64 (zeroed by the caller) receives the exact number of groups: the per-primitive counts and their
// prefix are 32-bit, and the host rejects a layout whose total does not fit
__global__ void k_groups_count(const int64_t* __restrict__ offsets, int n, int64_t seg, int32_t* __restrict__ cnt,
                               unsigned long long* __restrict__ total64) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  long long c = 0;
  if (i < n) {
    c = (offsets[i + 1] - offsets[i] + seg - 1) / seg;
    if (c < 0) c = 0;
    cnt[i] = (int32_t)(c > 2147483647LL ? 2147483647LL : c);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0 && c > 0) atomicAdd(total64, (unsigned long long)c);
}

__global__ void k_groups_fill(const int64_t* __restrict__ offsets, int n, int64_t seg, const int32_t* __restrict__ goff32,
                              int64_t* __restrict__ group_offsets, int64_t* __restrict__ primitives,
                              int64_t* __restrict__ starts, int64_t max_groups) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n) return;
  group_offsets[i] = goff32[i];
  if (i == n || !primitives || !starts) return;
  const int g0 = goff32[i], g1 = goff32[i + 1];
  for (int g = g0; g < g1; ++g)
    if (g < max_groups) { primitives[g] = i; starts[g] = offsets[i] + (int64_t)(g - g0) * seg; }
}

// digits of the primitive ids (and of the key that stands for an invalid one): equal passes of at most eight bits
struct GsPlan { int passes, dbits, nblocks; };
static GsPlan gs_plan(int64_t R, int n) {
  int bits = 1;
  while (bits < 31 && (1ll << bits) <= (int64_t)n) ++bits;      // keys 0 .. n
  GsPlan g;
  g.passes = (bits + 7) / 8;
  g.dbits = (bits + g.passes - 1) / g.passes;
  g.nblocks = (int)((R + kGsItems - 1) / kGsItems);
  return g;
}

// scratch: digit totals | block counts | 2 x keys | 2 x indices
struct GsLayout { int64_t dtot, hist, key[2], val[2], bytes; };
static GsLayout gs_layout(int64_t R) {
  GsLayout L;
  int64_t off = 0;
  auto take = [&](int64_t bytes) { int64_t o = off; off += align_up(bytes, 256); return o; };
  L.dtot = take(4 * kGsBins);
  L.hist = take(4 * kGsBins * std::max<int64_t>((R + kGsItems - 1) / kGsItems, 1));
  for (int i = 0; i < 2; ++i) { L.key[i] = take(4 * R); L.val[i] = take(4 * R); }
  L.bytes = off;
  return L;
}

static int group_rows(const int32_t* ids, int64_t R, int n, int64_t* offsets, int64_t* order, const float* x6, const float* d4,
                      const int32_t* masks, float* x6_out, float* d4_out, int32_t* masks_out, void* scratch,
                      int64_t scratch_bytes, cudaStream_t st, const char* who) {
  MLPSP_REQUIRE(R >= 0 && n >= 0 && offsets, MLPSP_E_ARG, "%s: bad arguments", who);
  MLPSP_REQUIRE(R < (1ll << 31), MLPSP_E_LIMIT, "%s: more than 2^31-1 records", who);
  MLPSP_REQUIRE(R == 0 || (ids && order), MLPSP_E_ARG, "%s: null pointer", who);
  MLPSP_REQUIRE((!x6 || x6_out) && (!d4 || d4_out) && (!masks || masks_out), MLPSP_E_ARG, "%s: null pointer", who);
  const GsLayout L = gs_layout(R);
  MLPSP_REQUIRE(scratch && scratch_bytes >= L.bytes, MLPSP_E_SCRATCH, "%s: scratch needs %lld bytes", who, (long long)L.bytes);
  if (R == 0) return cuda_check(cudaMemsetAsync(offsets, 0, 8 * ((size_t)n + 1), st), who);
  const GsPlan g = gs_plan(R, n);
  LaunchScope scope(kKMisc, 3 * g.passes + 1, st);
  char* b = (char*)scratch;
  int32_t* dtot = (int32_t*)(b + L.dtot);
  int32_t* hist = (int32_t*)(b + L.hist);
  const uint32_t* k_in = reinterpret_cast<const uint32_t*>(ids);
  const uint32_t* v_in = nullptr;
  uint32_t* inverse = nullptr;
  for (int pass = 0; pass < g.passes; ++pass) {
    const int shift = pass * g.dbits;
    const bool first = pass == 0, last = pass == g.passes - 1;
    uint32_t* k_out = (uint32_t*)(b + L.key[pass & 1]);
    uint32_t* v_out = (uint32_t*)(b + L.val[pass & 1]);          // the last pass writes no values: their place takes the inverse
    if (last && (x6 || d4 || masks)) inverse = v_out;
    launch_chained(first ? k_gs_hist<true> : k_gs_hist<false>, dim3(g.nblocks), dim3(kGsThreads), 0, st, k_in, R, n, shift, g.dbits, g.nblocks, hist);
    launch_chained(k_gs_scan, dim3(1 << g.dbits), dim3(kGsThreads), 0, st, g.nblocks, hist, dtot);
    auto* scatter = first ? (last ? k_gs_scatter<true, true> : k_gs_scatter<true, false>) : (last ? k_gs_scatter<false, true> : k_gs_scatter<false, false>);
    launch_chained(scatter, dim3(g.nblocks), dim3(kGsThreads), 0, st, k_in, v_in, R, n, shift, g.dbits, g.nblocks, hist, dtot, k_out, v_out,
                   order, inverse);
    k_in = k_out;
    v_in = v_out;
  }
  const int64_t span = std::max<int64_t>(inverse ? R : 0, (int64_t)n + 1);
  launch_chained(k_gs_finish, dim3((unsigned)((span + 255) / 256)), dim3(256), 0, st, k_in, inverse, R, n, offsets,
                 reinterpret_cast<const float2*>(x6), reinterpret_cast<const float4*>(d4), reinterpret_cast<const int2*>(masks),
                 reinterpret_cast<float2*>(x6_out), reinterpret_cast<float4*>(d4_out), reinterpret_cast<int2*>(masks_out));
  return cuda_check(cudaGetLastError(), who);
}

}  // namespace mlpsp

using namespace mlpsp;

extern "C" int64_t mlpsp_group_records_scratch_bytes(int64_t num_records, int32_t n) {
  if (num_records < 0 || n < 0) return -1;
  return gs_layout(num_records).bytes;
}

extern "C" int mlpsp_group_records(const int32_t* primitive_ids, int64_t num_records, int32_t n, int64_t* offsets,
                                   int64_t* order, void* scratch, int64_t scratch_bytes, void* stream) {
  return group_rows(primitive_ids, num_records, n, offsets, order, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, scratch,
                    scratch_bytes, (cudaStream_t)stream, "mlpsp_group_records");
}

extern "C" int mlpsp_group_rows(const int32_t* primitive_ids, int64_t num_records, int32_t n, const float* x6,
                                const float* grad4, const int32_t* relu_masks, int64_t* offsets, int64_t* order,
                                float* x6_out, float* grad4_out, int32_t* masks_out, void* scratch, int64_t scratch_bytes,
                                void* stream) {
  MLPSP_REQUIRE(((reinterpret_cast<uintptr_t>(x6) | reinterpret_cast<uintptr_t>(x6_out) | reinterpret_cast<uintptr_t>(relu_masks) |
                  reinterpret_cast<uintptr_t>(masks_out)) & 7) == 0 &&
                    ((reinterpret_cast<uintptr_t>(grad4) | reinterpret_cast<uintptr_t>(grad4_out)) & 15) == 0,
                MLPSP_E_ARG, "mlpsp_group_rows: x6 and masks must be 8-byte aligned, grad4 16-byte aligned");
  return group_rows(primitive_ids, num_records, n, offsets, order, x6, grad4, relu_masks, x6_out, grad4_out, masks_out, scratch,
                    scratch_bytes, (cudaStream_t)stream, "mlpsp_group_rows");
}

extern "C" int mlpsp_prepare_groups(const int64_t* offsets, int32_t n, int64_t segment_size, int64_t* group_offsets,
                                    int64_t* primitives, int64_t* starts, int64_t max_groups,
                                    int64_t* num_groups_host, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  MLPSP_REQUIRE(offsets && group_offsets && n >= 0, MLPSP_E_ARG, "mlpsp_prepare_groups: null pointer");
  MLPSP_REQUIRE(segment_size > 0, MLPSP_E_ARG, "segment_size must be a positive integer");
  // three small work arrays in one allocation: counts | prefix | scan blocks | 64-bit total
  const size_t bytes = (size_t)align_up(4 * ((int64_t)n + 2), 256);
  const size_t blk_bytes = (size_t)align_up(4 * ((int64_t)n / kScanItems + 4), 256);
  char* work = nullptr;
  MLPSP_CUDA_OK(cudaMallocAsync(&work, 2 * bytes + blk_bytes + 256, st));
  int32_t* cnt = reinterpret_cast<int32_t*>(work);
  int32_t* goff = reinterpret_cast<int32_t*>(work + bytes);
  int32_t* blk = reinterpret_cast<int32_t*>(work + 2 * bytes);
  unsigned long long* total64 = reinterpret_cast<unsigned long long*>(work + 2 * bytes + blk_bytes);
  int32_t G = 0;
  unsigned long long total = 0;
  // the allocation is released on every path; the first error wins
  int rc = cuda_check(cudaMemsetAsync(goff, 0, bytes + blk_bytes + 256, st), "prepare_groups");
  if (!rc && n > 0) k_groups_count<<<(n + 255) / 256, 256, 0, st>>>(offsets, n, segment_size, cnt, total64);
  if (!rc) rc = launch_scan_i32(cnt, n, blk, goff, st);
  if (!rc) {
    k_groups_fill<<<(n + 256) / 256, 256, 0, st>>>(offsets, n, segment_size, goff, group_offsets, primitives, starts, max_groups);
    rc = cuda_check(cudaMemcpyAsync(&G, goff + n, 4, cudaMemcpyDeviceToHost, st), "prepare_groups");
  }
  if (!rc) rc = cuda_check(cudaMemcpyAsync(&total, total64, 8, cudaMemcpyDeviceToHost, st), "prepare_groups");
  if (!rc) rc = cuda_check(cudaStreamSynchronize(st), "prepare_groups");
  cudaFreeAsync(work, st);
  if (rc) return rc;
  MLPSP_REQUIRE(total <= 2147483647ull, MLPSP_E_LIMIT,
                "mlpsp_prepare_groups: %llu groups exceed the 32-bit group index (raise segment_size)", total);
  if (num_groups_host) *num_groups_host = G;
  return cuda_check(cudaGetLastError(), "prepare_groups");
}

// ------------------------------------------------------------------------------------------
// prepare_groups for callers that must not allocate.
//
// mlpsp_prepare_groups above takes its three small work arrays from cudaMallocAsync.  Some hosts of
// this library cannot do that: a renderer plugin whose embedding engine owns all device memory and
// forbids driver allocations after start-up, or a frame loop that must not hit the implicit device
// synchronisation and the latency of cudaMalloc/cudaFree.  For them the same computation runs on a
// fixed scratch area that is part of the library image: a file-scope __device__ array, present on
// every GPU that loads the library until the process exits (about 4 MiB).
//
// The array's name is only a host-side handle in host code, not a device address, so the device
// address is looked up once per device with cudaGetSymbolAddress (with that device current) and
// cached; kernels receive that pointer.  The first call on a device performs this look-up, so make
// that first call outside any stream capture.  All calls share the one array and it keeps the
// previous call's contents: the part that must start at zero is cleared on every call, and two
// calls that overlap on the GPU (different streams or threads) would race on it, so serialise them.
namespace mlpsp {

constexpr int kStaticGroupsMaxPrims = MLPSP_STATIC_GROUPS_MAX_PRIMITIVES;
constexpr int64_t kSgCntBytes = (4ll * (kStaticGroupsMaxPrims + 2) + 255) / 256 * 256;
constexpr int64_t kSgBlkBytes = (4ll * (kStaticGroupsMaxPrims / kScanItems + 4) + 255) / 256 * 256;
constexpr int64_t kSgBytes = 2 * kSgCntBytes + kSgBlkBytes + 256;   // counts | prefix | scan blocks | 64-bit total

static __device__ __align__(256) unsigned char g_static_groups_scratch[kSgBytes];
static void* g_static_groups_ptr[64] = {nullptr};   // device address of the array, per device ordinal

static int static_groups_scratch(char** out) {
  int dev = -1;
  MLPSP_CUDA_OK(cudaGetDevice(&dev));
  MLPSP_REQUIRE(dev >= 0 && dev < 64, MLPSP_E_LIMIT, "mlpsp_prepare_groups_static: device ordinal %d beyond 63", dev);
  if (!g_static_groups_ptr[dev]) {
    void* p = nullptr;
    MLPSP_CUDA_OK(cudaGetSymbolAddress(&p, g_static_groups_scratch));
    MLPSP_REQUIRE(p != nullptr, MLPSP_E_CUDA, "mlpsp_prepare_groups_static: no device address for the scratch array");
    g_static_groups_ptr[dev] = p;
  }
  *out = static_cast<char*>(g_static_groups_ptr[dev]);
  return MLPSP_OK;
}

}  // namespace mlpsp

extern "C" int mlpsp_prepare_groups_static(const int64_t* offsets, int32_t n, int64_t segment_size,
                                           int64_t* group_offsets, int64_t* primitives, int64_t* starts,
                                           int64_t max_groups, int64_t* num_groups_host, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  MLPSP_REQUIRE(offsets && group_offsets && n >= 0, MLPSP_E_ARG, "mlpsp_prepare_groups_static: null pointer");
  MLPSP_REQUIRE(segment_size > 0, MLPSP_E_ARG, "segment_size must be a positive integer");
  MLPSP_REQUIRE(n <= kStaticGroupsMaxPrims, MLPSP_E_LIMIT,
                "mlpsp_prepare_groups_static: %d primitives exceed the built-in scratch capacity of %d "
                "(MLPSP_STATIC_GROUPS_MAX_PRIMITIVES); use mlpsp_prepare_groups", n, kStaticGroupsMaxPrims);
  char* base = nullptr;
  int rc = static_groups_scratch(&base);
  if (rc) return rc;
  int32_t* cnt = reinterpret_cast<int32_t*>(base);
  int32_t* goff = reinterpret_cast<int32_t*>(base + kSgCntBytes);
  int32_t* blk = reinterpret_cast<int32_t*>(base + 2 * kSgCntBytes);
  unsigned long long* total64 = reinterpret_cast<unsigned long long*>(base + 2 * kSgCntBytes + kSgBlkBytes);
  // the prefix array must read zero where the scan does not write (n == 0) and must not show the
  // previous call's totals; the 64-bit group total starts at zero as well
  MLPSP_CUDA_OK(cudaMemsetAsync(goff, 0, 4 * ((size_t)n + 2), st));
  MLPSP_CUDA_OK(cudaMemsetAsync(total64, 0, 8, st));
  if (n > 0) k_groups_count<<<(n + 255) / 256, 256, 0, st>>>(offsets, n, segment_size, cnt, total64);
  rc = launch_scan_i32(cnt, n, blk, goff, st);
  if (rc) return rc;
  k_groups_fill<<<(n + 256) / 256, 256, 0, st>>>(offsets, n, segment_size, goff, group_offsets, primitives, starts, max_groups);
  int32_t G = 0;
  unsigned long long total = 0;
  MLPSP_CUDA_OK(cudaMemcpyAsync(&G, goff + n, 4, cudaMemcpyDeviceToHost, st));
  MLPSP_CUDA_OK(cudaMemcpyAsync(&total, total64, 8, cudaMemcpyDeviceToHost, st));
  MLPSP_CUDA_OK(cudaStreamSynchronize(st));
  MLPSP_REQUIRE(total <= 2147483647ull, MLPSP_E_LIMIT,
                "mlpsp_prepare_groups_static: %llu groups exceed the 32-bit group index (raise segment_size)", total);
  if (num_groups_host) *num_groups_host = G;
  return cuda_check(cudaGetLastError(), "prepare_groups_static");
}
