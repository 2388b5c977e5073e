// Gated feature compositing as a contraction on the 5th-generation tensor cores (tcgen05, sm_100a).
//
//   out_feat[pix, :] = sum over the pixel's composited records of w * mix(p, gates)          (np_tile_kernels.cu:6036-6075)
// with mix = sum_s g_s attr[p, s, :] (S = 4), attr[p, 0, :] + sum_s g_s attr[p, 1+s, :] (S = 5) or attr[p, 0, :] (S = 1).
// The reference adds C values to global memory per hit.  Per tile this is a product
//   D^T [C x 64 pixels] = Attr^T [C x K] . Coef [K x 64 pixels],   K = (touched primitives of the tile) x S,
// where Coef holds w * g_s of the consumed (pixel, primitive) records and zeros elsewhere.  One CTA owns one
// (tile, block of up to 512 channels) and walks the tile's touched primitives 8 or 16 at a time:
//   * the attribute rows (binary16, the reference's inference storage format, scannet/checkpoints.py:358-359) are
//     gathered from this GPU's memory with cp.async into the MN-major core-matrix layout (eight K rows of eight
//     channels = 128 bytes) that tcgen05.mma reads as its A operand: the channel dimension is M, so all 128 rows
//     of the tensor core carry channels;
//   * every thread turns two or four (pixel, primitive) cells into coefficients: weight and gates of the record when
//     the pixel composited the primitive, zero otherwise, split into a binary16 head and a binary16 tail so that the
//     two products together carry 22 mantissa bits (the attributes themselves are exact);
//   * one thread issues the MMAs of the stage (128 x 64 x 16 each, FP32 accumulators in tensor memory) and commits
//     them to the mbarrier that guards the stage's buffers; the other stage is filled meanwhile.
// The copies and the record loads of the next stage are in flight while a stage is finished.
// Afterwards each warp reads its 32 channels x 64 pixels from tensor memory and writes 128-byte lines of the map.
//
// Bound: issue slots and the latency of the gather (each (tile, primitive) pair reads S * C * 2 bytes, from L2 for the most
// part); the map's own writes take 0.25 ms of a 1200 x 680 x 512 frame.  With scalar coefficient code, addresses made for every
// copy and two CTAs per SM, that frame (250k primitives) took 1.10 ms here, now 0.80; a 957 x 541 x 128 one 0.26, now 0.16.
//
// Every wait on an mbarrier is bounded (MLPSP_ST_TIMEOUT), copies in flight are waited for, tensor memory is freed.
#include "frame.cuh"
#include "tc.cuh"

namespace mlpsp {

constexpr int kFtThreads = 256;
constexpr int kFtListMax = 2048;      // candidates of a tile the kernel looks at (kWinMax of the wave kernels)
constexpr int kFtMeta = 256;          // touched primitives whose masks and bases are held in shared memory at a time

// what the kernel needs of one touched (tile, primitive) pair
struct __align__(8) FtMeta {
  int32_t prim;
  uint32_t base;     // compositing slot of the pair's first record
  uint32_t u0, u1;   // pixels that composited the primitive
  uint32_t m0, m1;   // pixels whose hit was evaluated (the record's slot is its rank among them)
};
static_assert(sizeof(FtMeta) == 24, "shared-memory plan");

__device__ __forceinline__ void ft_cp_async16(uint32_t dst, const void* src, bool valid) {
  const uint32_t n = valid ? 16u : 0u;   // source size 0: the 16 bytes are written as zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void ft_cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// instruction descriptor: D = F32, A = B = F16, A MN-major (bit 15), B K-major, dense
__host__ __device__ constexpr uint32_t ft_instr_desc(int M, int N) {
  return (1u << 4) | (1u << 15) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// shared memory of one stage: A [K/8 groups of eight K rows][CB/8 groups of eight channels][8 rows][8 halves],
// then the coefficient heads and tails [K/8 chunks][64 pixels][8 halves] each
// for PR primitives of S slots
template <int S, int PR>
struct FtPlan {
  static constexpr int K = PR * S;
  static_assert(K % 16 == 0, "whole MMA steps");
  __host__ __device__ static constexpr int a_bytes(int CB) { return K * CB * 2; }
  static constexpr int kCoefBytes = 64 * K * 2;
  __host__ __device__ static constexpr int stage_bytes(int CB) { return a_bytes(CB) + 2 * kCoefBytes; }
  __host__ __device__ static constexpr int smem_bytes(int CB) { return 2 * stage_bytes(CB) + 2 * kFtListMax + kFtMeta * 24 + 64; }
};

template <int S, int PR>
__global__ void __launch_bounds__(kFtThreads, PR == 8 ? 4 : 2) k_feature_tc(
    const int32_t* __restrict__ tile_offsets, const int32_t* __restrict__ tile_len, const int32_t* __restrict__ sorted_prims,
    int W, int H, int ntx, const uint32_t* __restrict__ used32, const uint32_t* __restrict__ masks32,
    const uint32_t* __restrict__ pair_base, const float* __restrict__ rec_w, const float4* __restrict__ rec_gate,
    const __half* __restrict__ feat16, int C, int CB, float* __restrict__ out_feat, int32_t* __restrict__ status) {
  using P = FtPlan<S, PR>;
  constexpr int K = P::K, NC = PR / 4;              // NC cells per thread and stage
  extern __shared__ __align__(128) char smem[];
  __shared__ int warp_sums[32];
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int tile = blockIdx.x, c0 = blockIdx.y * CB;
  const int tid = threadIdx.x, lane = tid & 31, warp = warp_of_cta();
  const int stage_bytes = P::stage_bytes(CB);
  uint16_t* s_idx = reinterpret_cast<uint16_t*>(smem + 2 * stage_bytes);            // touched candidates of the tile
  FtMeta* s_meta = reinterpret_cast<FtMeta*>(smem + 2 * stage_bytes + 2 * kFtListMax);
  uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + 2 * stage_bytes + 2 * kFtListMax + kFtMeta * 24);   // [0..1] MMAs of a stage buffer done
  uint32_t* s_misc = reinterpret_cast<uint32_t*>(s_bar + 2);                        // [0] tmem base
  const uint32_t sb = smem_u32(smem);
  const uint32_t bar0 = smem_u32(&s_bar[0]);
  const int nb128 = CB / 128;
  const uint32_t tmem_cols = nb128 > 2 ? 256u : (uint32_t)nb128 * 64u;
  if (tid == 0) {
    mbar_init(bar0, 1);
    mbar_init(bar0 + 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(smem_u32(&s_misc[0]), tmem_cols);

  // ---- the tile's touched candidates (some pixel composited the primitive), in list order ----
  const int s = tile_offsets[tile];
  const int len = min(tile_len[tile], kFtListMax);
  int nt = 0;
  for (int j0 = 0; j0 < len; j0 += kFtThreads) {
    const int j = j0 + tid;
    bool touched = false;
    if (j < len) {
      const uint2 u = *reinterpret_cast<const uint2*>(used32 + 2 * (size_t)(s + j));
      touched = (u.x | u.y) != 0u;
    }
    int total;
    const int pos = block_exclusive_scan(touched ? 1 : 0, warp_sums, total);
    if (touched) s_idx[nt + pos] = (uint16_t)j;
    nt += total;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_misc[0];
  const int a_bytes = P::a_bytes(CB);
  const uint32_t lbo_a = (uint32_t)CB * 16u;      // between groups of eight K rows
  const uint32_t idesc = ft_instr_desc(128, 64);
  bool ok = true;
  int gs = 0;                                     // stages issued so far: buffer = gs & 1, use of that buffer = gs >> 1
  const int half = warp & 1, px = half * 32 + lane, pl0 = (warp >> 1) * NC;     // this thread's cells of a stage: primitives pl0.. of pixel px

  // the MMAs that last read the buffer of stage g (two stages earlier) have finished
  auto buffer_free = [&](int g) {
    if (g >= 2) ok = mbar_wait(bar0 + 8 * (g & 1), (uint32_t)((g >> 1) - 1) & 1u) && ok;
  };
  // Attribute rows of the PR primitives from touched index l0 of the batch on: a warp copies eight K rows x four channel
  // groups at a time, so that eight lanes fill one 128-byte core matrix (no bank conflicts) and four lanes read 64
  // contiguous bytes; its rows stay, so the next copy is 64 bytes on.  One cp.async group per stage.
  auto issue_copies = [&](int g, int l0, int nb) {
    constexpr int KG = K / 8, parts = KG < kFtThreads / 32 ? kFtThreads / 32 / KG : 1;     // row groups; warps that share one
    const int gq_n = CB / 32 / parts;
    for (int task = warp; task < KG * parts; task += kFtThreads / 32) {
      const int kg = task % KG, grp = (task / KG) * gq_n * 4 + (lane >> 3);
      const int k = kg * 8 + (lane & 7), pl = k / S, sl = k - pl * S;
      const bool valid = l0 + pl < nb;
      const int prim = valid ? s_meta[l0 + pl].prim : 0;
      const __half* src = feat16 + ((size_t)prim * S + sl) * C + c0 + grp * 8;
      uint32_t dst = sb + (g & 1) * stage_bytes + kg * lbo_a + grp * 128 + (lane & 7) * 16;
#pragma unroll 4
      for (int gq = 0; gq < gq_n; ++gq) {
        ft_cp_async16(dst, src, valid);
        src += 32;
        dst += 512;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // weight and gates of this thread's cells of a stage; zero where the pixel did not composite the primitive
  auto load_cells = [&](int l0, int nb, float (&cw)[NC], float4 (&cg)[NC]) {
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const int l = l0 + pl0 + i;
      cw[i] = 0.f;
      cg[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (l < nb) {
        const FtMeta& m = s_meta[l];
        if (((half ? m.u1 : m.u0) >> lane) & 1u) {
          const uint32_t slot = m.base + (half ? __popc(m.m0) : 0) + __popc((half ? m.m1 : m.m0) & ((1u << lane) - 1u));
          cw[i] = __ldg(rec_w + slot);
          if (S > 1) cg[i] = __ldg(rec_gate + slot);
        }
      }
    }
  };
  // two coefficients -> packed heads and tails
  auto split2 = [](float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
  };
  // coefficients of the cells, head + tail in binary16; K index of slot sl of the stage's primitive pl is pl * S + sl,
  // element (pixel, k) sits at (k / 8) * 1024 + pixel * 16 + (k % 8) * 2
  auto write_coefs = [&](int g, const float (&cw)[NC], const float4 (&cg)[NC]) {
    char* coef_hi = smem + (g & 1) * stage_bytes + a_bytes;
    char* coef_lo = coef_hi + P::kCoefBytes;
    if (S == 4) {                                       // two primitives fill the pixel's 16 bytes of one K group
#pragma unroll
      for (int i = 0; i < NC; i += 2) {
        uint32_t h[4], l[4];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          split2(cw[i + j] * cg[i + j].x, cw[i + j] * cg[i + j].y, h[2 * j], l[2 * j]);
          split2(cw[i + j] * cg[i + j].z, cw[i + j] * cg[i + j].w, h[2 * j + 1], l[2 * j + 1]);
        }
        const int off = ((pl0 + i) >> 1) * 1024 + px * 16;
        *reinterpret_cast<uint4*>(coef_hi + off) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4*>(coef_lo + off) = make_uint4(l[0], l[1], l[2], l[3]);
      }
    } else if (S == 1) {                                // four primitives: eight of the sixteen bytes
      uint32_t h[2], l[2];
      split2(cw[0], cw[1], h[0], l[0]);
      split2(cw[NC > 2 ? 2 : 0], cw[NC > 3 ? 3 : 0], h[1], l[1]);
      const int off = (pl0 >> 3) * 1024 + px * 16 + (pl0 & 7) * 2;
      *reinterpret_cast<uint2*>(coef_hi + off) = make_uint2(h[0], h[1]);
      *reinterpret_cast<uint2*>(coef_lo + off) = make_uint2(l[0], l[1]);
    } else {
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        const float cf[5] = {cw[i], cw[i] * cg[i].x, cw[i] * cg[i].y, cw[i] * cg[i].z, cw[i] * cg[i].w};
#pragma unroll
        for (int sl = 0; sl < S; ++sl) {
          const int k = (pl0 + i) * S + sl, off = (k >> 3) * 1024 + px * 16 + (k & 7) * 2;
          const __half hi = __float2half_rn(cf[sl]);
          *reinterpret_cast<__half*>(coef_hi + off) = hi;
          *reinterpret_cast<__half*>(coef_lo + off) = __float2half_rn(cf[sl] - __half2float(hi));
        }
      }
    }
  };

  for (int b0 = 0; b0 < nt && ok; b0 += kFtMeta) {
    const int nb = min(kFtMeta, nt - b0);
    // ---- the batch's primitives, consumed masks, hit masks and record bases ----
    __syncthreads();
    for (int l = tid; l < nb; l += kFtThreads) {
      const size_t pi = (size_t)(s + s_idx[b0 + l]);
      const uint2 u = *reinterpret_cast<const uint2*>(used32 + 2 * pi), m = *reinterpret_cast<const uint2*>(masks32 + 2 * pi);
      FtMeta e;
      e.prim = __ldg(sorted_prims + pi); e.base = __ldg(pair_base + pi); e.u0 = u.x; e.u1 = u.y; e.m0 = m.x; e.m1 = m.y;
      s_meta[l] = e;
    }
    __syncthreads();
    // ---- stages of PR primitives; the copies and the record loads of stage l+1 are in flight while stage l is
    // finished and handed to the tensor cores ----
    const int nsb = (nb + PR - 1) / PR;
    float cw[NC];
    float4 cg[NC];
    buffer_free(gs);
    issue_copies(gs, 0, nb);
    load_cells(0, nb, cw, cg);
    for (int ls = 0; ls < nsb; ++ls) {
      const int g = gs + ls;
      const bool more = ls + 1 < nsb;
      if (more) {
        buffer_free(g + 1);
        issue_copies(g + 1, (ls + 1) * PR, nb);
      }
      write_coefs(g, cw, cg);
      if (more) load_cells((ls + 1) * PR, nb, cw, cg);
      if (more) asm volatile("cp.async.wait_group 1;" ::: "memory");
      else asm volatile("cp.async.wait_group 0;" ::: "memory");
      fence_async_smem();
      tc_fence_before();
      if (!__syncthreads_and(ok)) { ok = false; break; }
      if (warp == 0) tc_fence_after();
      if (warp == 0 && elect_one()) {
        const uint32_t a_s = sb + (g & 1) * stage_bytes;
        const uint32_t hi_s = a_s + a_bytes, lo_s = hi_s + P::kCoefBytes;
        const uint64_t bh_desc = smem_desc(hi_s, 1024, 128), bl_desc = smem_desc(lo_s, 1024, 128);
        for (int h = 0; h < nb128; ++h) {
          // A: MN-major, 128 channels = 16 groups of eight (128 bytes apart), K groups of eight lbo_a apart
          const uint64_t a_desc = smem_desc(a_s + h * 2048, lbo_a, 128);
#pragma unroll
          for (int ks = 0; ks < K / 16; ++ks) {
            const uint64_t a_k = a_desc + (uint64_t)((ks * 2 * lbo_a) >> 4);
            mma_f16(tmem + h * 64, a_k, bh_desc + (uint64_t)((ks * 2 * 1024) >> 4), idesc, (g > 0 || ks > 0) ? 1u : 0u);
            mma_f16(tmem + h * 64, a_k, bl_desc + (uint64_t)((ks * 2 * 1024) >> 4), idesc, 1u);
          }
        }
        mma_commit(bar0 + 8 * (g & 1));
      }
    }
    gs += nsb;
  }
  const int nst = gs;

  // ---- the last stage's MMAs (tensor-core instructions complete in order) ----
  if (ok && nst > 0) {
    const int last = nst - 1;
    ok = mbar_wait(bar0 + 8 * (last & 1), (uint32_t)(last >> 1) & 1u);
  }
  ok = __all_sync(0xffffffffu, ok);
  tc_fence_after();
  // ---- epilogue: warp = 32 channels of one 128-channel half, thread = channel, 64 pixels from tensor memory ----
  const int q = warp & 3;
  const int x0 = (tile % ntx) * 8, y0 = (tile / ntx) * 8;
  for (int h = warp >> 2; h < nb128; h += 2) {
    float* dst = out_feat + ((size_t)y0 * W + x0) * C + c0 + h * 128 + q * 32 + lane;
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
      uint32_t v[32];
      if (ok && nst > 0) {
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + h * 64 + part * 32, v);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = 0u;
      }
      // streaming stores: the map is not read again here, the attributes in L2 are
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int y = part * 4 + r;
        if (y0 + y >= H) break;
        float* row = dst + (size_t)y * W * C;
#pragma unroll
        for (int x = 0; x < 8; ++x)
          if (x0 + x < W) __stcs(row + (size_t)x * C, __uint_as_float(v[r * 8 + x]));
      }
    }
  }
  if (!ok) {
    if (tid == 0) atomicOr(status + MLPSP_ST_BITS, MLPSP_ST_TIMEOUT);
    ft_cp_async_wait_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, tmem_cols);
}

// binary16 copy of the attributes [n, S, C]; raises MLPSP_ST_FEAT_INEXACT when a value does not survive the round trip
__global__ void k_pack_features(const float* __restrict__ attr, int64_t count, __half* __restrict__ out, int32_t* __restrict__ status) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  bool inexact = false;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
    const float v = attr[i];
    const __half hv = __float2half_rn(v);
    out[i] = hv;
    inexact |= !(__half2float(hv) == v);
  }
  if (inexact && status) atomicOr(status + MLPSP_ST_BITS, MLPSP_ST_FEAT_INEXACT);
}

bool feature_tc_supported(const mlpsp_scene* sc) {
  return sc->feat16 != nullptr && sc->feat_dim >= 128 && sc->feat_dim <= 512 && sc->feat_dim % 128 == 0 &&
         (sc->feat_slots == 1 || sc->feat_slots == 4 || sc->feat_slots == 5) &&
         (reinterpret_cast<uintptr_t>(sc->feat16) & 15) == 0;
}

// Primitives per stage and channels per CTA.  Four slots: eight primitives (two whole K steps) and up to 256 channels, so that
// three CTAs or more stay on an SM: 957 x 541 x 128 0.24 -> 0.16 ms against stages of 16, 1200 x 680 x 512 0.80 ms with 256
// and with 512 channels a CTA.  One and five slots need 16 primitives for whole steps (K = 16, 80).
template <int S, int PR>
static int launch_ft(const mlpsp_scene* sc, const mlpsp_frame* fr, const Scratch& s, const uint32_t* used32, int T, int ntx, int CB,
                     cudaStream_t st) {
  const int smem = FtPlan<S, PR>::smem_bytes(CB);
  static DeviceOnce attr_once;
  if (attr_once.first())
    MLPSP_CUDA_OK(cudaFuncSetAttribute(k_feature_tc<S, PR>, cudaFuncAttributeMaxDynamicSharedMemorySize, 113 * 1024));
  const dim3 grid(T, sc->feat_dim / CB);
  k_feature_tc<S, PR><<<grid, kFtThreads, smem, st>>>(fr->tile_offsets, s.tile_len, fr->sorted_prims, fr->width, fr->height, ntx, used32,
                                                      s.masks32, s.pair_base, s.rec_w, s.rec_gate, (const __half*)sc->feat16, sc->feat_dim, CB,
                                                      fr->feat, fr->status);
  return cuda_check(cudaGetLastError(), "feature_tc");
}

int launch_feature_tc(const mlpsp_scene* sc, const mlpsp_frame* fr, const Scratch& s, const uint32_t* used32, cudaStream_t st) {
  const int T = num_tiles(fr->width, fr->height, 8), ntx = (fr->width + 7) / 8;
  const int C = sc->feat_dim;
  if (sc->feat_slots == 1) return launch_ft<1, 16>(sc, fr, s, used32, T, ntx, C, st);
  if (sc->feat_slots == 5) return launch_ft<5, 16>(sc, fr, s, used32, T, ntx, 128, st);
  return launch_ft<4, 8>(sc, fr, s, used32, T, ntx, C % 256 == 0 ? 256 : C, st);
}

}  // namespace mlpsp

using namespace mlpsp;

extern "C" int mlpsp_pack_features_f16(const mlpsp_scene* sc, void* feat16_out, int32_t* status, void* stream) {
  MLPSP_REQUIRE(sc && feat16_out, MLPSP_E_ARG, "mlpsp_pack_features_f16: null pointer");
  MLPSP_REQUIRE(sc->feat_attr && sc->feat_dim > 0 && sc->feat_slots > 0 && sc->n >= 0, MLPSP_E_ARG,
                "mlpsp_pack_features_f16: the scene has no feature attributes");
  const int64_t count = (int64_t)sc->n * sc->feat_slots * sc->feat_dim;
  if (count == 0) return MLPSP_OK;
  cudaStream_t st = (cudaStream_t)stream;
  LaunchScope scope(kKMisc, 1, st);
  const int blocks = (int)std::min<int64_t>((count + 255) / 256, 148 * 32);
  k_pack_features<<<blocks, 256, 0, st>>>(sc->feat_attr, count, (__half*)feat16_out, status);
  return cuda_check(cudaGetLastError(), "mlpsp_pack_features_f16");
}
