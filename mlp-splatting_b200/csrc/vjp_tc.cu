// Per-primitive weight gradients of the 72-32-32-4 MLP on the 5th-generation tensor cores (tcgen05, sm_100a):
// the mixed-precision modes of grouped_weight_gradients (scannet/primitive_gemm.py:101-166: binary16 or bfloat16
// operands, FP32 accumulation over the whole segment, adjoints scaled before the cast and unscaled in FP32).
//
// The launch is persistent: a CTA walks the planned segments (VjpItem, backward.cu) round-robin in blocks of 128
// records (thread = record).  All operand tiles of a block live in shared memory as chunks of [128 records][8 elements]
// (16 bytes per record, 2,048 bytes per chunk).  That one layout serves two kinds of product:
//   * record-major products (rows of D = records), the tile is the K-major A operand as in the evaluator:
//       H1 = relu(E W1^T + b1), H2 = relu(H1 W2^T + b2), D1 = (D2 W2) * mask1
//     (W2 is stored once: K-major for layer 2, the same bytes MN-major for D1);
//   * the weight gradients contract over the records, so the same bytes are read as MN-major operands
//     (eight records x eight elements = one 128-byte core matrix with the element dimension contiguous):
//       dW1^T [72 x 32] += E^T D1,   [H1 | H2]^T [D2 | D3]: dW2^T [32 x 32] and dW3^T [32 x 4] are two blocks of it
//     with M = 128 rows of the tensor core over the element dimension (rows past the operand's width read the
//     chunks that follow and land in accumulator lanes nobody looks at), K = 16 records per MMA, as many K steps as the
//     block has records.  A chunk of ones directly behind E, H1 and H2 makes the bias gradients the next accumulator
//     lane -- FP32 sums of the rounded adjoints, as primitive_gemm.py:157-160 takes them.
// D2 = (D3 W3) * mask2 has K = 4 and is done by the threads from the rounded operands.
// The gradient accumulators stay in tensor memory for the whole segment and are written, divided by the scale, to the
// primitive's gradient tensors, or -- for a primitive of several segments -- to the segment's partial row.
//
// What bounds it: the chain of a block (operand tile complete -> fence -> CTA barrier -> one thread issues and commits ->
// everyone waits on the mbarrier, bounded): 7,300 cycles with three CTAs per SM, 6,700 with one, of which 1,700 are the issue of
// the MMAs (47 cycles each, the time their operands take out of shared memory) and the rest instructions of the twelve warps;
// bytes (weights in, gradients out, 48 B per record) would take a third of the time.  So the chain is kept short: with saved
// masks the adjoint chain does not depend on the forward one, D1 rides with layer 1 and dW1 with layer 2, three round trips per
// block; the last one (dW2, dW3) overlaps the next block's encoding, a finished segment's gradients leave and the next block's
// records and weights arrive while layer 1 runs.  5.5 M records of 15,000 primitives, 35,000 more without records: 598 us with
// dW1 in the last round trip, the gradients written between two blocks and weights loaded a row per lane, 546 so.  (Two threads
// per record, 256 per CTA: 840, by spills, and 855 with two CTAs per SM.)
#include "frame.cuh"
#include "tc.cuh"
#include "vjp.cuh"

namespace mlpsp {

constexpr int kVjpRows = kVjpBlock, kVjpChunk = kVjpRows * 16;
// chunk indices of the operand tiles
constexpr int kVcE = 0, kVcOneE = 9, kVcH1 = 10, kVcOneH1 = 14, kVcH2 = 15, kVcOneH2 = 19, kVcD1 = 20, kVcD2 = 24,
              kVcD3 = 28, kVcEnd = 30;
// weight operands ([K / 8 chunks][32 rows][8 elements]); a chunk is 512 bytes and 16 more, so that the lanes of a warp, which
// hold consecutive k of a row or two, store into different banks
constexpr int kVjpWChunk = 528;
constexpr int kVoW1 = kVcEnd * kVjpChunk;          // W1[h][j], 10 chunks (the last one zero: it meets the ones behind E)
constexpr int kVoW2 = kVoW1 + 10 * kVjpWChunk;     // W2[q][h], 4 chunks
constexpr int kVoW3 = kVoW2 + 4 * kVjpWChunk;      // W3[c][h], rounded to the operand format, as FP32: [4][32]
constexpr int kVoBias = kVoW3 + 512;               // b1[32], b2[32] as FP32
constexpr int kVoBar = kVoBias + 256;
constexpr int kVjpSmem = kVoBar + 16;
// tensor memory: 128 columns: [0,32) layers, [32,64) dW1^T, [64,112) dW2^T | dW3^T; and 32 of their own: D1
constexpr int kVjpTmemCols = 128, kVjpTmemColsD1 = 32, kVtG1 = 32, kVtG2 = 64;
constexpr int kVjpCtas = 3;
static_assert((kVcH1 + 16) * kVjpChunk <= kVoW1, "an M = 128 window from any tile start stays inside the tiles");
static_assert(kVjpCtas * (kVjpSmem + 1024) <= 227 * 1024 && kVjpCtas * (kVjpTmemCols + kVjpTmemColsD1) <= 512, "resident CTAs");

// bits 15 / 16 of the instruction descriptor: A / B is MN-major
constexpr uint32_t kMnA = 1u << 15, kMnB = 1u << 16;

template <bool BF16>
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  return make_uint4(pack_h2<BF16>(v[0], v[1]), pack_h2<BF16>(v[2], v[3]), pack_h2<BF16>(v[4], v[5]), pack_h2<BF16>(v[6], v[7]));
}
// the two values of a packed word, as FP32
template <bool BF16>
__device__ __forceinline__ float2 unpack_h2(uint32_t w) {
  if (BF16) return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}

// ReLU + rounding of 32 accumulator columns (+ FP32 bias) into a hidden tile; returns the sign mask
template <bool BF16>
__device__ __forceinline__ uint32_t vjp_hidden(const uint32_t (&acc)[32], const float4* __restrict__ bias, char* dst) {
  uint32_t sign = 0u;
#pragma unroll
  for (int kc = 0; kc < 4; ++kc) {
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; q += 2) {
      const int j = kc * 8 + q * 2;
      const float4 b = bias[j / 4];
      const float v0 = __uint_as_float(acc[j]) + b.x, v1 = __uint_as_float(acc[j + 1]) + b.y;
      const float v2 = __uint_as_float(acc[j + 2]) + b.z, v3 = __uint_as_float(acc[j + 3]) + b.w;
      sign |= (v0 > 0.f ? 1u : 0u) << j;
      sign |= (v1 > 0.f ? 1u : 0u) << (j + 1);
      sign |= (v2 > 0.f ? 1u : 0u) << (j + 2);
      sign |= (v3 > 0.f ? 1u : 0u) << (j + 3);
      w[q] = pack_h2_relu<BF16>(v0, v1);
      w[q + 1] = pack_h2_relu<BF16>(v2, v3);
    }
    *reinterpret_cast<uint4*>(dst + kc * kVjpChunk) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  return sign;
}

// N accumulator columns (N / 8 chunks of an adjoint tile), masked and rounded; m holds the mask bits of these columns
template <bool BF16, int N>
__device__ __forceinline__ void vjp_adjoint(const uint32_t (&acc)[N], uint32_t m, char* dst) {
#pragma unroll
  for (int kc = 0; kc < N / 8; ++kc) {
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int j = kc * 8 + q * 2;
      const float v0 = ((m >> j) & 1u) ? __uint_as_float(acc[j]) : 0.f;
      const float v1 = ((m >> (j + 1)) & 1u) ? __uint_as_float(acc[j + 1]) : 0.f;
      w[q] = pack_h2<BF16>(v0, v1);
    }
    *reinterpret_cast<uint4*>(dst + kc * kVjpChunk) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// pairs of FP32 values: two IEEE operations in one instruction
__device__ __forceinline__ uint64_t pair_of(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ uint64_t pair_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t pair_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// D2 = (D3 W3) * mask2 of one record, from the rounded operands
template <bool BF16>
__device__ __forceinline__ void vjp_d2(uint32_t d01, uint32_t d23, uint32_t m2, const float* __restrict__ w3, char* dst) {
  const float2 a = unpack_h2<BF16>(d01), b = unpack_h2<BF16>(d23);
  const uint64_t d[4] = {pair_of(a.x, a.x), pair_of(a.y, a.y), pair_of(b.x, b.x), pair_of(b.y, b.y)};
#pragma unroll
  for (int kc = 0; kc < 4; ++kc) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; i += 4) {
      ulonglong2 w = *reinterpret_cast<const ulonglong2*>(w3 + 3 * kGH + kc * 8 + i);
      uint64_t s0 = pair_mul(d[3], w.x), s1 = pair_mul(d[3], w.y);
#pragma unroll
      for (int c = 2; c >= 0; --c) {
        w = *reinterpret_cast<const ulonglong2*>(w3 + c * kGH + kc * 8 + i);
        s0 = pair_fma(d[c], w.x, s0);
        s1 = pair_fma(d[c], w.y, s1);
      }
      asm("mov.b64 {%0, %1}, %2;" : "=f"(v[i]), "=f"(v[i + 1]) : "l"(s0));
      asm("mov.b64 {%0, %1}, %2;" : "=f"(v[i + 2]), "=f"(v[i + 3]) : "l"(s1));
#pragma unroll
      for (int u = 0; u < 4; ++u) v[i + u] = ((m2 >> (kc * 8 + i + u)) & 1u) ? v[i + u] : 0.f;
    }
    *reinterpret_cast<uint4*>(dst + kc * kVjpChunk) = pack8<BF16>(v);
  }
}

// MASKS: the records carry saved ReLU masks.  Without them the signs come from the recomputed layers, the adjoint chain
// has to follow the forward one, and a block takes four round trips.  vec: rows may be loaded in 16- and 8-byte pieces.
template <bool BF16, bool MASKS>
__global__ void __launch_bounds__(kVjpRows, kVjpCtas) k_grouped_vjp_tc(
    const float* __restrict__ x6, const float* __restrict__ d4, const int32_t* __restrict__ masks,
    const VjpItem* __restrict__ items, int64_t max_items, const VjpItem* __restrict__ multi, int n, int aligned, int32_t* __restrict__ counters,
    const float* __restrict__ freq, const float* __restrict__ att, const float* __restrict__ W1, const float* __restrict__ b1, const float* __restrict__ W2,
    const float* __restrict__ b2, const float* __restrict__ W3, int vec, float scale, VjpOut out, float* __restrict__ partial) {
  chain_wait();
  chain_release();
  extern __shared__ __align__(128) char smem[];
  const VjpList list(items, max_items, counters);
  const int G = list.total, E = vjp_planned(counters, kVpEmpty);
  const int idx = blockIdx.x;
  const int tid = threadIdx.x, warp = warp_of_cta();
  // primitives without records, one between two waits; the number of the next one is on its way
  int empty = blockIdx.x, empty_prim = empty < E ? __ldg(&multi[n - 1 - empty].prim) : 0;
  auto zero_next = [&]() {
    if (empty >= E) return;
    const int prim = empty_prim;
    empty += (int)gridDim.x;
    if (empty < E) empty_prim = __ldg(&multi[n - 1 - empty].prim);
    if (!aligned) {
      vjp_zero(out, prim, aligned, tid, kVjpRows);
      return;
    }
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4* w1 = reinterpret_cast<float4*>(out.W1 + prim * out.sW1) + tid;
    float4* w2 = reinterpret_cast<float4*>(out.W2 + prim * out.sW2) + tid;
#pragma unroll
    for (int i = 0; i < 4; ++i) w1[i * kVjpRows] = zero;
#pragma unroll
    for (int i = 0; i < 2; ++i) w2[i * kVjpRows] = zero;
    if (tid < 64) {
      w1[4 * kVjpRows] = zero;
    } else if (tid < 96) {
      reinterpret_cast<float4*>(out.W3 + prim * out.sW3)[tid - 64] = zero;
    } else {
      const int i = tid - 96;
      if (i < 8) reinterpret_cast<float4*>(out.b1 + prim * out.sb1)[i] = zero;
      else if (i < 16) reinterpret_cast<float4*>(out.b2 + prim * out.sb2)[i - 8] = zero;
      else if (i == 16) *reinterpret_cast<float4*>(out.b3 + prim * out.sb3) = zero;
    }
  };
  if (idx >= G) {
    while (empty < E) zero_next();
    return;
  }
  uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + kVoBar);
  uint32_t* s_misc = reinterpret_cast<uint32_t*>(s_bar + 1);
  float* s_bias = reinterpret_cast<float*>(smem + kVoBias);
  float* s_w3 = reinterpret_cast<float*>(smem + kVoW3);
  const uint32_t sb = smem_u32(smem), bar = smem_u32(s_bar);
  if (tid == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {      // together three CTAs' allocations fit an SM, so neither waits for good while the first is held
    tmem_alloc(smem_u32(&s_misc[0]), kVjpTmemCols, true);
    tmem_alloc(smem_u32(&s_misc[1]), kVjpTmemColsD1);
  }
  // segments differ tenfold in length, so a CTA takes its first by its number and the others from a counter, two ahead
  __shared__ int s_next;
  auto draw = [&]() { if (tid == 0) s_next = (int)gridDim.x + atomicAdd(counters + kVpNext, 1); };
  draw();
  // tiles: zeros, except the three chunks of ones; W1's last chunk stays zero
  {
    const uint32_t one2 = BF16 ? 0x3f803f80u : 0x3c003c00u;
    for (int i = tid; i < kVcEnd * kVjpRows; i += kVjpRows) {
      const int chunk = i >> 7;
      const uint32_t v = (chunk == kVcOneE || chunk == kVcOneH1 || chunk == kVcOneH2) ? one2 : 0u;
      *reinterpret_cast<uint4*>(smem + (size_t)i * 16) = make_uint4(v, v, v, v);
    }
    if (tid < 32) *reinterpret_cast<uint4*>(smem + kVoW1 + 9 * kVjpWChunk + tid * 16) = make_uint4(0u, 0u, 0u, 0u);
  }
  float mult[6];
#pragma unroll
  for (int f = 0; f < 6; ++f) mult[f] = __ldg(freq + f) * __ldg(att + f);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_misc[0], tmem_d1 = s_misc[1];
  const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16), trow_d1 = tmem_d1 + ((uint32_t)(warp * 32) << 16);

  constexpr uint32_t idesc_h = instr_desc(kVjpRows, 32, BF16), idesc_d1 = instr_desc(kVjpRows, 32, BF16) | kMnB,
                     idesc_g1 = instr_desc(kVjpRows, 32, BF16) | kMnA | kMnB, idesc_g2 = instr_desc(kVjpRows, 48, BF16) | kMnA | kMnB;
  auto tile = [&](int chunk) { return sb + (uint32_t)chunk * kVjpChunk; };
  // record-major A operand (K-major): K chunks a chunk apart, groups of eight records 128 bytes apart
  auto a_rows = [&](int chunk) { return smem_desc(tile(chunk), kVjpChunk, 128); };
  // MN-major operand: groups of eight elements a chunk apart, groups of eight records 128 bytes apart
  auto mn = [&](int chunk) { return smem_desc(tile(chunk), 128, kVjpChunk); };
  auto adv = [](uint64_t desc, int bytes) { return desc + (uint64_t)(bytes >> 4); };
  const uint64_t w1_desc = smem_desc(sb + kVoW1, kVjpWChunk, 128), w2_desc = smem_desc(sb + kVoW2, kVjpWChunk, 128);
  const uint64_t w2t_desc = smem_desc(sb + kVoW2, 128, kVjpWChunk);      // N = h (a chunk per eight), K = q (128 bytes per eight)

  char* my = smem + tid * 16;
  uint32_t ph = 0u;
  bool ok = true;
  // tile writes visible to the tensor core, tensor-memory reads retired, then one thread (of the warp that has no part in
  // emit) issues and commits; false in all threads when a wait has given up in one
  constexpr int kIssueWarp = 3;
  auto issue_phase = [&](auto issue) -> bool {
    fence_async_smem();
    tc_fence_before();
    if (!__syncthreads_and(ok)) return false;
    if (warp == kIssueWarp) {
      tc_fence_after();
      if (elect_one()) {
        issue();
        mma_commit(bar);
      }
      __syncwarp();
    }
    return true;
  };
  // every thread waits for itself: what it touches next is its own (tile rows, tensor-memory lanes), and the barrier of the
  // next issue_phase is the one that tells the CTA of a wait that gave up
  auto wait_phase = [&]() {
    ok = __all_sync(0xffffffffu, mbar_wait(bar, ph & 1u)) && ok;
    ++ph;
    tc_fence_after();
  };

  // ---- a step's inputs in registers: one record per thread, and with a new primitive its weights ----
  float rx[6];
  float4 rg;
  uint32_t rm1 = 0u, rm2 = 0u;
  auto load_rec = [&](const VjpItem& it, int sub) {
#pragma unroll
    for (int c = 0; c < 6; ++c) rx[c] = 0.f;
    rg = make_float4(0.f, 0.f, 0.f, 0.f);
    rm1 = rm2 = 0u;
    if (sub + tid < it.rows) {
      const int64_t r = it.start + sub + tid;
      if (vec) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float2 v = __ldg(reinterpret_cast<const float2*>(x6) + r * 3 + c);
          rx[2 * c] = v.x; rx[2 * c + 1] = v.y;
        }
      } else {
#pragma unroll
        for (int c = 0; c < 6; ++c) rx[c] = __ldg(x6 + r * 6 + c);
      }
      rg = __ldg(reinterpret_cast<const float4*>(d4) + r);
      if (MASKS) { rm1 = (uint32_t)__ldg(masks + r * 2); rm2 = (uint32_t)__ldg(masks + r * 2 + 1); }
    }
  };
  // W1 as 576 groups of four consecutive k of one row, W2 as 256, both in the order of memory, W3 and the biases one value per
  // thread (eight k of a row per thread, a row per lane, took 32 cycles of the load unit per load instead of four)
  float4 wv[7];
  float wr3 = 0.f, wrb = 0.f;
  auto load4 = [&](const float* p) {
    return vec ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
  };
  auto load_weights = [&](int prim) {
    const float* w1 = W1 + (size_t)prim * (kGH * kGIN);
#pragma unroll
    for (int u = 0; u < 5; ++u) {
      const int g = u * kVjpRows + tid;
      if (u < 4 || g < 576) wv[u] = load4(w1 + 4 * g);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) wv[5 + u] = load4(W2 + (size_t)prim * (kGH * kGH) + 4 * (u * kVjpRows + tid));
    wr3 = __ldg(W3 + (size_t)prim * (4 * kGH) + tid);
    if (tid < 64) wrb = __ldg((tid < 32 ? b1 : b2) + (size_t)prim * kGH + (tid & 31));
  };
  auto store_weights = [&]() {
    auto put4 = [&](int off, int h, int k, const float4& v) {
      *reinterpret_cast<uint2*>(smem + off + (k >> 3) * kVjpWChunk + h * 16 + (k & 4) * 2) = make_uint2(pack_h2<BF16>(v.x, v.y), pack_h2<BF16>(v.z, v.w));
    };
#pragma unroll
    for (int u = 0; u < 5; ++u) {
      const int g = u * kVjpRows + tid, h = g / (kGIN / 4);
      if (u < 4 || g < 576) put4(kVoW1, h, 4 * (g - h * (kGIN / 4)), wv[u]);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int g = u * kVjpRows + tid;
      put4(kVoW2, g / (kGH / 4), 4 * (g % (kGH / 4)), wv[5 + u]);
    }
    s_w3[tid] = unpack_h2<BF16>(pack_h2<BF16>(wr3, 0.f)).x;
    if (tid < 64) s_bias[tid] = wrb;
  };
  // the gradients of a finished segment: accumulator lane = input of the layer (its ones lane: the bias), column = output
  const float inv = 1.f / scale;
  bool bad = false;
  auto emit = [&](const VjpItem& it) {
    const VjpOut o = vjp_row(out, partial, it);
    uint32_t acc[32];
    auto put = [&](float* p, uint32_t v) {
      const float g = __uint_as_float(v) * inv;
      bad |= !(fabsf(g) <= 3.4028235e38f);
      *p = g;
    };
    if (warp < 3) {
      tmem_ld32(trow + kVtG1, acc);
      if (tid < 72) {
#pragma unroll
        for (int h = 0; h < 32; ++h) put(o.W1 + h * 72 + tid, acc[h]);
      } else if (tid == 72) {
#pragma unroll
        for (int h = 0; h < 32; ++h) put(o.b1 + h, acc[h]);
      }
    }
    if (warp < 2) {
      tmem_ld32(trow + kVtG2, acc);
      if (tid < 32) {
#pragma unroll
        for (int q = 0; q < 32; ++q) put(o.W2 + q * 32 + tid, acc[q]);
      } else if (tid == 32) {
#pragma unroll
        for (int q = 0; q < 32; ++q) put(o.b2 + q, acc[q]);
      }
    }
    if (warp == 1 || warp == 2) {      // the H2 rows of the window follow H1's four chunks and its ones
      uint32_t o3[4];
      tmem_ld4(trow + kVtG2 + 32, o3);
      if (tid >= 40 && tid < 72) {
#pragma unroll
        for (int c = 0; c < 4; ++c) put(o.W3 + c * 32 + tid - 40, o3[c]);
      } else if (tid == 72) {
#pragma unroll
        for (int c = 0; c < 4; ++c) put(o.b3 + c, o3[c]);
      }
    }
  };

  VjpItem it = list.at(idx), it_n = it, it_p = it;
  bool has_n = s_next < G;
  if (has_n) it_n = list.at(s_next);
  __syncthreads();                 // before the next draw
  load_weights(it.prim);
  load_rec(it, 0);
  int sub = 0;
  bool pending = false, finished = false;      // gradient MMAs in flight; they complete segment it_p

  for (;;) {
    // ---- encoding (index c * 6 + f holds sin, 36 + c * 6 + f holds cos: scannet/cumodel.py:183-195) and D3,
    //      into registers while the previous block's gradient MMAs finish ----
    //      (rows past the segment's end encode zeros; their adjoints are zero, so they add nothing to a gradient)
    uint32_t ew[36];                                            // 32-bit word = two consecutive encoding entries
#pragma unroll
    for (int c = 0; c < 6; ++c) {
#pragma unroll
      for (int g = 0; g < 3; ++g) {
        float s0, c0, s1, c1;
        __sincosf(rx[c] * mult[2 * g], &s0, &c0);
        __sincosf(rx[c] * mult[2 * g + 1], &s1, &c1);
        ew[3 * c + g] = pack_h2<BF16>(s0, s1);
        ew[18 + 3 * c + g] = pack_h2<BF16>(c0, c1);
      }
    }
    const uint32_t d01 = pack_h2<BF16>(rg.x * scale, rg.y * scale), d23 = pack_h2<BF16>(rg.z * scale, rg.w * scale);
    uint32_t m1 = rm1, m2 = rm2;
    if (pending) {
      wait_phase();
    }
    if (sub == 0) store_weights();
#pragma unroll
    for (int kc = 0; kc < 9; ++kc)
      *reinterpret_cast<uint4*>(my + (kVcE + kc) * kVjpChunk) = make_uint4(ew[4 * kc], ew[4 * kc + 1], ew[4 * kc + 2], ew[4 * kc + 3]);
    *reinterpret_cast<uint4*>(my + kVcD3 * kVjpChunk) = make_uint4(d01, d23, 0u, 0u);
    if (MASKS) {
      if (sub == 0) __syncthreads();                            // W3 of the new primitive
      vjp_d2<BF16>(d01, d23, m2, s_w3, my + kVcD2 * kVjpChunk);
    }
    if (sub == 0) draw();                                       // read after the barrier of this layer, at the segment's last block
    // ---- layer 1: K = 80 (the ones behind E meet the zero chunk of W1); with masks the first half of D1 ----
    ok = issue_phase([&]() {
      const uint64_t a = a_rows(kVcE);
#pragma unroll
      for (int ks = 0; ks < 5; ++ks) mma_f16(tmem, adv(a, ks * 2 * kVjpChunk), adv(w1_desc, ks * 2 * kVjpWChunk), idesc_h, ks > 0);
      if (MASKS) {
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) mma_f16(tmem_d1, adv(a_rows(kVcD2), ks * 2 * kVjpChunk), adv(w2t_desc, ks * 256), idesc_d1, ks > 0);
      }
    });
    if (!ok) break;
    // ---- the finished segment's gradients, while layer 1 runs ----
    if (pending && finished && ok) emit(it_p);
    // ---- the next step's loads, in flight from here on ----
    const int cnt = min(kVjpRows, it.rows - sub);
    const bool last = sub + kVjpRows >= it.rows;
    const VjpItem it_c = it;
    const int sub_c = sub;
    bool more = true;
    if (!last) {
      sub += kVjpRows;
      load_rec(it, sub);
    } else if (has_n) {
      it = it_n;
      sub = 0;
      load_rec(it, 0);
      load_weights(it.prim);
      has_n = s_next < G;
      if (has_n) it_n = list.at(s_next);
    } else {
      more = false;
    }
    zero_next();
    wait_phase();
    {
      uint32_t acc[32];
      tmem_ld32(trow, acc);
      const uint32_t sign = vjp_hidden<BF16>(acc, reinterpret_cast<const float4*>(s_bias), my + kVcH1 * kVjpChunk);
      if (!MASKS) m1 = sign;
    }
    if (MASKS) {
      uint32_t acc[32];
      tmem_ld32(trow_d1, acc);
      vjp_adjoint<BF16, 32>(acc, m1, my + kVcD1 * kVjpChunk);
    }
    // ---- layer 2; with masks dW1 behind it, contracting over the block's records, 16 per MMA ----
    auto grad1 = [&]() {
      const uint64_t e = mn(kVcE), d1 = mn(kVcD1);
      const int steps = (cnt + 15) >> 4;
      for (int ks = 0; ks < steps; ++ks) mma_f16(tmem + kVtG1, adv(e, ks * 256), adv(d1, ks * 256), idesc_g1, (sub_c > 0 || ks > 0) ? 1u : 0u);
    };
    ok = issue_phase([&]() {
      const uint64_t a = a_rows(kVcH1);
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) mma_f16(tmem, adv(a, ks * 2 * kVjpChunk), adv(w2_desc, ks * 2 * kVjpWChunk), idesc_h, ks > 0);
    });
    if (MASKS && ok && warp == kIssueWarp) {                             // not waited for before the last phase
      if (elect_one()) grad1();
      __syncwarp();
    }
    if (!ok) break;
    wait_phase();
    {
      uint32_t acc[32];
      tmem_ld32(trow, acc);
      const uint32_t sign = vjp_hidden<BF16>(acc, reinterpret_cast<const float4*>(s_bias + 32), my + kVcH2 * kVjpChunk);
      if (!MASKS) m2 = sign;
    }
    if (!MASKS) {
      vjp_d2<BF16>(d01, d23, m2, s_w3, my + kVcD2 * kVjpChunk);
      ok = issue_phase([&]() {
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) mma_f16(tmem, adv(a_rows(kVcD2), ks * 2 * kVjpChunk), adv(w2t_desc, ks * 256), idesc_d1, ks > 0);
      });
      if (!ok) break;
      wait_phase();
      uint32_t acc[32];
      tmem_ld32(trow, acc);
      vjp_adjoint<BF16, 32>(acc, m1, my + kVcD1 * kVjpChunk);
    }
    // ---- dW2 and dW3 (without masks dW1 too) ----
    ok = issue_phase([&]() {
      if (!MASKS) grad1();
      const uint64_t h = mn(kVcH1), d23t = mn(kVcD2);
      const int steps = (cnt + 15) >> 4;
      for (int ks = 0; ks < steps; ++ks) mma_f16(tmem + kVtG2, adv(h, ks * 256), adv(d23t, ks * 256), idesc_g2, (sub_c > 0 || ks > 0) ? 1u : 0u);
    });
    if (!ok) break;
    pending = true;
    finished = last;
    it_p = it_c;
    if (!more) break;
  }
  if (ok) {
    while (empty < E) zero_next();
    wait_phase();
    if (ok) emit(it_p);
  }
  if (bad) atomicOr(counters + kVpFlag, 1);
  if (!ok && tid == 0) atomicOr(counters + kVpFlag, 2);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tmem_free(tmem, kVjpTmemCols);
    tmem_free(tmem_d1, kVjpTmemColsD1);
  }
}

int launch_grouped_vjp_tc(bool bf16, const float* x6, const float* d4, const int32_t* masks, const VjpItem* items,
                          int64_t max_items, const VjpItem* multi, int32_t* counters, const mlpsp_scene* sc, float scale,
                          const VjpOut& out, float* partial, cudaStream_t st) {
  static DeviceOnce attr_once;
  if (attr_once.first()) {
    MLPSP_CUDA_OK(cudaFuncSetAttribute(k_grouped_vjp_tc<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kVjpSmem));
    MLPSP_CUDA_OK(cudaFuncSetAttribute(k_grouped_vjp_tc<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kVjpSmem));
    MLPSP_CUDA_OK(cudaFuncSetAttribute(k_grouped_vjp_tc<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kVjpSmem));
    MLPSP_CUDA_OK(cudaFuncSetAttribute(k_grouped_vjp_tc<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kVjpSmem));
  }
  auto* kernel = bf16 ? (masks ? k_grouped_vjp_tc<true, true> : k_grouped_vjp_tc<true, false>)
                      : (masks ? k_grouped_vjp_tc<false, true> : k_grouped_vjp_tc<false, false>);
  const int vec = ((reinterpret_cast<uintptr_t>(sc->W1) | reinterpret_cast<uintptr_t>(sc->W2)) & 15) == 0 &&
                  (reinterpret_cast<uintptr_t>(x6) & 7) == 0;
  const int grid = (int)std::min<int64_t>(std::max<int64_t>(max_items, sc->n), (int64_t)sm_count() * kVjpCtas);     // CTAs without segments write zeros
  return cuda_check(launch_chained(kernel, dim3(grid), dim3(kVjpRows), kVjpSmem, st, x6, d4, masks, items, max_items, multi, sc->n, vjp_aligned(out), counters,
                                   sc->freq, sc->att,
                                   sc->W1, sc->b1, sc->W2, sc->b2, sc->W3, vec, scale, out, partial),
                    "grouped_vjp_tc");
}

}  // namespace mlpsp
