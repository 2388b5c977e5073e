// Scalar FP32 per-primitive evaluator: positional encoding + 12F -> H -> H -> 4 MLP in the
// operation order of the reference's scalar kernels (scannet/cuda/np_tile_kernels.cu:2047-2103):
// layer 1 starts from the bias and accumulates (sin weight, cos weight) per (component, frequency);
// layers 2 and 3 start from the bias and accumulate over ascending input index.
// One CTA per work item (primitive, up to 128 of its records); the primitive's FP32 weights are
// staged once in shared memory.  k_mlp_f32_pair (hidden 32) gives a thread up to four records of half the units,
// k_mlp_f32_wide (hidden 64) register tiles, and k_mlp_f32, for every other shape, one record.
#include "frame.cuh"
#include "tc.cuh"

namespace mlpsp {

template <int HMAX>
__global__ void __launch_bounds__(kRowsPerItem) k_mlp_f32(
    const float* __restrict__ W1, const float* __restrict__ b1, const float* __restrict__ W2,
    const float* __restrict__ b2, const float* __restrict__ W3, const float* __restrict__ b3,
    const float* __restrict__ freq, const float* __restrict__ att, int F, int H,
    const RecIn* __restrict__ rec_in, const int4* __restrict__ work,
    int32_t* __restrict__ counters, float4* __restrict__ rec_out, float4* __restrict__ rec_ext, int out_mode,
    const int32_t* __restrict__ status) {
  extern __shared__ float sW[];
  __shared__ int s_item;
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int IN = 12 * F, half = 6 * F;
  float* sW1 = sW;
  float* sb1 = sW1 + H * IN;
  float* sW2 = sb1 + H;
  float* sb2 = sW2 + H * H;
  float* sW3 = sb2 + H;
  float* sb3 = sW3 + 4 * H;
  float* sfa = sb3 + 4;  // freq[f]*att is NOT pre-multiplied: the product is v*freq*att left to right
  const int tid = threadIdx.x;
  const int G = counters[kCtrWork];
  for (;;) {
    if (tid == 0) s_item = atomicAdd(counters + kCtrWorkNext, 1);
    __syncthreads();
    const int item = s_item;
    if (item >= G) break;
    const int4 wk = work[item];
    const int p = wk.x;
    for (int i = tid; i < H * IN; i += kRowsPerItem) sW1[i] = W1[(size_t)p * H * IN + i];
    for (int i = tid; i < H * H; i += kRowsPerItem) sW2[i] = W2[(size_t)p * H * H + i];
    for (int i = tid; i < 4 * H; i += kRowsPerItem) sW3[i] = W3[(size_t)p * 4 * H + i];
    for (int i = tid; i < H; i += kRowsPerItem) { sb1[i] = b1[(size_t)p * H + i]; sb2[i] = b2[(size_t)p * H + i]; }
    if (tid < 4) sb3[tid] = b3[(size_t)p * 4 + tid];
    if (tid < F) { sfa[tid] = freq[tid]; sfa[F + tid] = att[tid]; }
    __syncthreads();
    if (tid < wk.z) {
      const RecIn r = rec_in[wk.y + tid];
      const float v6[6] = {r.rdx, r.rdy, r.rdz, r.dx, r.dy, r.dz};
      float h1[HMAX];
#pragma unroll
      for (int h = 0; h < HMAX; ++h) h1[h] = (h < H) ? sb1[h] : 0.f;
      for (int c = 0; c < 6; ++c) {
        for (int f = 0; f < F; ++f) {
          const float ph = v6[c] * sfa[f] * sfa[F + f];
          const float sn = __sinf(ph), cs = __cosf(ph);
          const int j = c * F + f;
#pragma unroll
          for (int h = 0; h < HMAX; ++h) {
            if (h < H) {
              h1[h] = fmaf(sW1[h * IN + j], sn, h1[h]);
              h1[h] = fmaf(sW1[h * IN + j + half], cs, h1[h]);
            }
          }
        }
      }
      uint32_t m1 = 0u, m2 = 0u;
#pragma unroll
      for (int h = 0; h < HMAX; ++h) {
        if (h < 32 && h1[h] > 0.f) m1 |= 1u << h;
        h1[h] = fmaxf(h1[h], 0.f);
      }
      float o0 = sb3[0], o1 = sb3[1], o2 = sb3[2], o3 = sb3[3];
      for (int q = 0; q < H; ++q) {
        float a = sb2[q];
#pragma unroll
        for (int h = 0; h < HMAX; ++h) if (h < H) a = fmaf(sW2[q * H + h], h1[h], a);
        if (q < 32 && a > 0.f) m2 |= 1u << q;
        a = fmaxf(a, 0.f);
        // layer 3 accumulates over ascending hidden index, which is this loop's order
        o0 = fmaf(sW3[0 * H + q], a, o0); o1 = fmaf(sW3[1 * H + q], a, o1);
        o2 = fmaf(sW3[2 * H + q], a, o2); o3 = fmaf(sW3[3 * H + q], a, o3);
      }
      const float sigma_raw = softplus_fast(o3);
      float4 out;
      out.x = sigmoid_fast(o0); out.y = sigmoid_fast(o1); out.z = sigmoid_fast(o2);
      out.w = (out_mode == kOutAlpha) ? (1.f - __expf(-(sigma_raw * r.decay))) : sigma_raw;
      rec_out[r.slot] = out;
      if (rec_ext) rec_ext[r.slot] = make_float4(sigma_raw, o3, __uint_as_float(m1), __uint_as_float(m2));
    }
    __syncthreads();
  }
}

constexpr int kTIN = 72, kTF = 6;         // six frequencies

__device__ __forceinline__ unsigned long long pack_f32x2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack_f32x2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma_f32x2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// The 72 -> 32 -> 32 -> 4 network: 64 threads per work item.  A thread owns up to four records of sixteen units (the other
// half-warp the other sixteen), the sums in registers as packed pairs of units (fma.rn.f32x2: two IEEE multiply-adds, so
// every sum keeps the order and the bits described at the top of this file).  The weights lie transposed in shared memory
// ([input][unit]): four broadcast 16-byte reads per input, whose halves are the packed operands, feed 64 multiply-adds.  The
// half-warps exchange the hidden units through shared memory, in the place of the first layer's weights and the records.
// The weights are copied asynchronously and transposed on the way; six CTAs per SM (three warps on each scheduler) cover one
// another's copies, and take their items from a counter.
// Bound: FP32 multiply-adds, 3,456 per record -- 36 G on the 100k frame, 1.0 ms at the chip's rate, 1.2 with the rows that
// fill up an item's last 32.  One record per thread with scalar multiply-adds, bounded by the broadcast reads (two cycles
// each), took 2.75 ms; two records of all units per thread 2.26; this 1.86 (five CTAs of two buffers and a fixed order of
// the items 2.31, seven or eight CTAs of 128 registers 2.08 and 1.97).
struct PairBuf {
  static constexpr int kRow = 36;          // floats per row of weights: 16-byte aligned, conflict-free transposing copies
  static constexpr int kRecRow = 12;       // floats per record: 16-byte aligned, neighbouring records on different banks
  static constexpr int kW1 = 0, kRec = kW1 + kTIN * kRow, kW2 = kRec + kRowsPerItem * kRecRow, kW3 = kW2 + 32 * kRow, kB1 = kW3 + 128,
                       kB2 = kB1 + 32, kB3 = kB2 + 32, kFloats = kB3 + 4;
  static constexpr int kHid = 0, kHidWarp = 32 * 64;      // hidden units of a warp's records, after layer 1
  static_assert(2 * kHidWarp <= kW2, "the hidden units take the place of W1 and the records");
  static_assert(kRec % 4 == 0 && kW2 % 4 == 0 && kFloats % 4 == 0, "16-byte accesses");
};
constexpr int kPairThreads = 64, kPairCtas = 6;

__device__ __forceinline__ void cp_async4(uint32_t dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// one row of sixteen weights onto the sums of R records
template <int R>
__device__ __forceinline__ void row_fma(unsigned long long (&acc)[R][8], const float* row, const float (&x)[R]) {
  unsigned long long xx[R];
#pragma unroll
  for (int r = 0; r < R; ++r) xx[r] = pack_f32x2(x[r], x[r]);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(row + 4 * k);
#pragma unroll
    for (int r = 0; r < R; ++r) { fma_f32x2(acc[r][2 * k], w.x, xx[r]); fma_f32x2(acc[r][2 * k + 1], w.y, xx[r]); }
  }
}
template <int R>
__device__ __forceinline__ void row_start(unsigned long long (&acc)[R][8], const float* bias) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(bias + 4 * k);
#pragma unroll
    for (int r = 0; r < R; ++r) { acc[r][2 * k] = b.x; acc[r][2 * k + 1] = b.y; }
  }
}
// R values of a lane as one vector of V >= R floats (V = 1, 2, 4)
template <int R, int V>
__device__ __forceinline__ void put_vec(float* p, const float (&x)[R]) {
  if (V == 4) *reinterpret_cast<float4*>(p) = make_float4(x[0], x[R > 1 ? 1 : 0], x[R > 2 ? 2 : 0], x[R > 3 ? 3 : 0]);
  else if (V == 2) *reinterpret_cast<float2*>(p) = make_float2(x[0], x[R > 1 ? 1 : 0]);
  else *p = x[0];
}
template <int R, int V>
__device__ __forceinline__ void get_vec(const float* p, float (&x)[R]) {
  float v[4];
  if (V == 4) { const float4 q = *reinterpret_cast<const float4*>(p); v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w; }
  else if (V == 2) { const float2 q = *reinterpret_cast<const float2*>(p); v[0] = q.x; v[1] = q.y; }
  else v[0] = *p;
#pragma unroll
  for (int r = 0; r < R; ++r) x[r] = v[r];
}
// ReLU of the sums to the warp's exchange area; bit u of mask: this half's unit u is positive
template <int R, int V>
__device__ __forceinline__ void relu_put(const unsigned long long (&acc)[R][8], float* hid, int lane, uint32_t (&mask)[R], bool want) {
  const int half = lane >> 4, l16 = lane & 15;
#pragma unroll
  for (int r = 0; r < R; ++r) mask[r] = 0u;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    float a[R], b[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float2 v = unpack_f32x2(acc[r][k]);
      if (want) mask[r] |= ((v.x > 0.f ? 1u : 0u) | (v.y > 0.f ? 2u : 0u)) << (2 * k);
      a[r] = fmaxf(v.x, 0.f);
      b[r] = fmaxf(v.y, 0.f);
    }
    put_vec<R, V>(hid + (half * 16 + 2 * k) * (16 * V) + l16 * V, a);
    put_vec<R, V>(hid + (half * 16 + 2 * k + 1) * (16 * V) + l16 * V, b);
  }
}

// R * 32 records of an item; record r of a lane is warp * 16 R + 16 r + lane % 16
template <int R>
__device__ __forceinline__ void pair_eval(float* sm, const float* s_freq, int warp, int lane, int rows, float4* __restrict__ rec_out,
                                          float4* __restrict__ rec_ext, int out_mode) {
  using B = PairBuf;
  constexpr int V = R == 3 ? 4 : R, NF = (R + 1) / 2;       // NF records finished per lane: those with r % 2 == half
  const int half = lane >> 4, l16 = lane & 15, rec0 = warp * 16 * R + l16;
  unsigned long long acc[R][8];
  uint32_t m1[R], m2[R];
  float decay[NF];
  uint32_t slot[NF];
#pragma unroll
  for (int q = 0; q < NF; ++q) {
    const int rec = rec0 + 16 * min(2 * q + half, R - 1);
    decay[q] = sm[B::kRec + rec * B::kRecRow + 6];
    slot[q] = __float_as_uint(sm[B::kRec + rec * B::kRecRow + 7]);
  }
  row_start<R>(acc, sm + B::kB1 + half * 16);
#pragma unroll 1
  for (int c = 0; c < 6; ++c) {
    float v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = sm[B::kRec + (rec0 + 16 * r) * B::kRecRow + c];
    const float* row = sm + B::kW1 + c * kTF * B::kRow + half * 16;
#pragma unroll
    for (int f = 0; f < kTF; ++f) {
      const float2 fa = *reinterpret_cast<const float2*>(s_freq + 2 * f);
      float sn[R], cs[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float ph = v[r] * fa.x * fa.y;
        sn[r] = __sinf(ph);
        cs[r] = __cosf(ph);
      }
      row_fma<R>(acc, row + f * B::kRow, sn);
      row_fma<R>(acc, row + (f + kTIN / 2) * B::kRow, cs);
    }
  }
  __syncthreads();                         // W1 and the records have been read
  float* hid = sm + B::kHid + warp * B::kHidWarp;
  relu_put<R, V>(acc, hid, lane, m1, rec_ext != nullptr);
  __syncwarp();
  row_start<R>(acc, sm + B::kB2 + half * 16);
#pragma unroll 4
  for (int k = 0; k < 32; ++k) {
    float x[R];
    get_vec<R, V>(hid + k * (16 * V) + l16 * V, x);
    row_fma<R>(acc, sm + B::kW2 + k * B::kRow + half * 16, x);
  }
  __syncwarp();
  relu_put<R, V>(acc, hid, lane, m2, rec_ext != nullptr);
  __syncwarp();
  // outputs 2 * half and 2 * half + 1 of all R records
  unsigned long long o[R];
#pragma unroll
  for (int r = 0; r < R; ++r) o[r] = *reinterpret_cast<const unsigned long long*>(sm + B::kB3 + 2 * half);
#pragma unroll 8
  for (int k = 0; k < 32; ++k) {
    float x[R];
    get_vec<R, V>(hid + k * (16 * V) + l16 * V, x);
    const unsigned long long w = *reinterpret_cast<const unsigned long long*>(sm + B::kW3 + 4 * k + 2 * half);
#pragma unroll
    for (int r = 0; r < R; ++r) fma_f32x2(o[r], w, pack_f32x2(x[r], x[r]));
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, o[r], 16);
    if (rec_ext) {
      const uint32_t a = __shfl_xor_sync(0xffffffffu, m1[r], 16), b = __shfl_xor_sync(0xffffffffu, m2[r], 16);
      m1[r] = half ? (m1[r] << 16) | a : m1[r] | (a << 16);
      m2[r] = half ? (m2[r] << 16) | b : m2[r] | (b << 16);
    }
    const int rec = rec0 + 16 * r;
    if ((r & 1) != half || rec >= rows) continue;
    const float2 lo = unpack_f32x2(half ? other : o[r]), hi = unpack_f32x2(half ? o[r] : other);
    const float sigma_raw = softplus_fast(hi.y);
    float4 out;
    out.x = sigmoid_fast(lo.x); out.y = sigmoid_fast(lo.y); out.z = sigmoid_fast(hi.x);
    out.w = (out_mode == kOutAlpha) ? (1.f - __expf(-(sigma_raw * decay[r / 2]))) : sigma_raw;
    rec_out[slot[r / 2]] = out;
    if (rec_ext) rec_ext[slot[r / 2]] = make_float4(sigma_raw, hi.y, __uint_as_float(m1[r]), __uint_as_float(m2[r]));
  }
}

__global__ void __launch_bounds__(kPairThreads, kPairCtas) k_mlp_f32_pair(
    const float* __restrict__ W1, const float* __restrict__ b1, const float* __restrict__ W2,
    const float* __restrict__ b2, const float* __restrict__ W3, const float* __restrict__ b3,
    const float* __restrict__ freq, const float* __restrict__ att, const RecIn* __restrict__ rec_in,
    const int4* __restrict__ work, const int32_t* __restrict__ counters, int32_t* __restrict__ cursor, float4* __restrict__ rec_out,
    float4* __restrict__ rec_ext, int out_mode, const int32_t* __restrict__ status) {
  using B = PairBuf;
  chain_wait();
  chain_release();
  extern __shared__ __align__(16) float sm[];
  __shared__ __align__(8) float s_freq[2 * kTF];
  __shared__ int s_next;
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int tid = threadIdx.x, warp = warp_of_cta(), lane = tid & 31;
  const int G = counters[kCtrWork];
  const int item = blockIdx.x;
  if (item >= G) return;
  if (tid < kTF) { s_freq[2 * tid] = __ldg(freq + tid); s_freq[2 * tid + 1] = __ldg(att + tid); }
  const uint32_t s0 = smem_u32(sm);
  // A warp copies eight inputs of four units at a time: whole 32-byte sectors, 32 different banks.
  const int jl = lane & 7, hl = lane >> 3;
  auto copy = [&](const int4& w) {
    const uint32_t d = s0;
    const size_t p = (size_t)w.x;
    const float* w1 = W1 + p * (kTIN * 32) + (warp * 16 + hl) * kTIN + jl;
    const float* w2 = W2 + p * (32 * 32) + (warp * 16 + hl) * 32 + jl;
    const uint32_t d1 = d + 4u * (uint32_t)(B::kW1 + jl * B::kRow + warp * 16 + hl), d2 = d1 + 4u * (uint32_t)(B::kW2 - B::kW1);
#pragma unroll
    for (int hb = 0; hb < 4; ++hb) {
#pragma unroll
      for (int jb = 0; jb < kTIN / 8; ++jb) cp_async4(d1 + 4u * (uint32_t)(jb * 8 * B::kRow + hb * 4), w1 + hb * 4 * kTIN + jb * 8);
#pragma unroll
      for (int jb = 0; jb < 4; ++jb) cp_async4(d2 + 4u * (uint32_t)(jb * 8 * B::kRow + hb * 4), w2 + hb * 4 * 32 + jb * 8);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int j = (2 * warp + u) * 8 + jl;
      cp_async4(d + 4u * (uint32_t)(B::kW3 + j * 4 + hl), W3 + p * 128 + hl * 32 + j);
    }
    cp_async4(d + 4u * (uint32_t)(B::kB1 + tid), tid < 32 ? b1 + p * 32 + tid : b2 + p * 32 + tid - 32);
    if (tid < 4) cp_async4(d + 4u * (uint32_t)(B::kB3 + tid), b3 + p * 4 + tid);
    const char* rec = reinterpret_cast<const char*>(rec_in + w.y);
    for (int c = tid; c < 2 * w.z; c += kPairThreads)    // the item's records, 32 bytes each
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 4u * (uint32_t)(B::kRec + (c >> 1) * B::kRecRow + (c & 1) * 4)),
                   "l"(rec + 16 * (size_t)c) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto ahead = [&](const int4& w) {
    const char* w1 = reinterpret_cast<const char*>(W1 + (size_t)w.x * (kTIN * 32));
    const char* w2 = reinterpret_cast<const char*>(W2 + (size_t)w.x * (32 * 32));
    const char* rec = reinterpret_cast<const char*>(rec_in + w.y);
    for (int l = tid; l < kTIN + 32 + 32; l += kPairThreads) {         // 128-byte lines of W1, W2 and the records
      const char* q = l < kTIN ? w1 + l * 128 : (l < kTIN + 32 ? w2 + (l - kTIN) * 128 : rec + (l - kTIN - 32) * 128);
      if (l < kTIN + 32 || (l - kTIN - 32) * 4 < w.z) asm volatile("prefetch.global.L2 [%0];" ::"l"(q));
    }
  };
  int4 wn = make_int4(0, 0, 0, 0);
  // The items come from a counter: the warps of an SM's four schedulers do not all get on at the same pace.  The next item's
  // number is fetched and its lines are brought into L2 while the current one is computed.
  int4 wk = __ldg(work + item);
  for (;;) {
    copy(wk);
    int next = G;
    if (tid == 0) s_next = next = (int)gridDim.x + atomicAdd(cursor, 1);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    next = s_next;
    const bool more = next < G;
    if (more) {
      wn = __ldg(work + next);
      ahead(wn);
    }
    // rows past the item's last record are computed from what the buffer holds and dropped
    switch ((wk.z + 31) >> 5) {
      case 1: pair_eval<1>(sm, s_freq, warp, lane, wk.z, rec_out, rec_ext, out_mode); break;
      case 2: pair_eval<2>(sm, s_freq, warp, lane, wk.z, rec_out, rec_ext, out_mode); break;
      case 3: pair_eval<3>(sm, s_freq, warp, lane, wk.z, rec_out, rec_ext, out_mode); break;
      default: pair_eval<4>(sm, s_freq, warp, lane, wk.z, rec_out, rec_ext, out_mode);
    }
    if (!more) break;
    __syncthreads();                       // the buffer has been read
    wk = wn;
  }
}

// The 72 -> 64 -> 64 -> 4 network, whose sums do not fit a thread's registers, as register-tiled products.  A work item's
// records lie transposed in shared memory ([quantity][record], rows of 132 floats), the weights as [input][unit], and a
// thread owns eight records of four units: per input three 16-byte reads feed 32 multiply-adds.  The next item's weights and
// records are loaded into registers while the current one is computed.  Bound: FP32 multiply-adds, 9,216 per record; a
// thread per record with scalar reads of its weights took 21.0 ms where this takes 5.1 (100k frame of 64-wide
// layers).
struct WideNet {
  static constexpr int kH = 64, kThreads = 256, kWRow = kH + 4, kTRow = kRowsPerItem + 4;
  static constexpr int kE = 0, kH1 = kE + kTIN * kTRow, kW1T = kH1 + kH * kTRow, kW2T = kW1T + kTIN * kWRow, kW3T = kW2T + kH * kWRow,
                       kB1 = kW3T + 4 * kH, kB2 = kB1 + kH, kB3 = kB2 + kH, kFloats = kB3 + 4;
  static constexpr int kCtas = 2;
  static_assert(kH <= kTIN, "the second hidden layer takes the encoding's place");
  static_assert(kCtas * (kFloats * 4 + 1024) <= 228 * 1024, "resident CTAs");
};

__global__ void __launch_bounds__(WideNet::kThreads, WideNet::kCtas) k_mlp_f32_wide(
    const float* __restrict__ W1, const float* __restrict__ b1, const float* __restrict__ W2,
    const float* __restrict__ b2, const float* __restrict__ W3, const float* __restrict__ b3,
    const float* __restrict__ freq, const float* __restrict__ att, const RecIn* __restrict__ rec_in,
    const int4* __restrict__ work, const int32_t* __restrict__ counters, float4* __restrict__ rec_out,
    int out_mode, const int32_t* __restrict__ status) {
  using N = WideNet;
  constexpr int H = N::kH, kTRow = N::kTRow, kT = N::kThreads, kL1 = kTIN * H / kT, kL2 = H * H / kT;      // weights per thread
  chain_wait();
  chain_release();
  extern __shared__ __align__(16) float sm[];
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int tid = threadIdx.x;
  const int G = counters[kCtrWork];
  int item = blockIdx.x;
  if (item >= G) return;
  float fr[kTF], at[kTF];
#pragma unroll
  for (int f = 0; f < kTF; ++f) { fr[f] = __ldg(freq + f); at[f] = __ldg(att + f); }
  const int rec = tid & (kRowsPerItem - 1), part = tid / kRowsPerItem;       // two threads encode a record
  const int h4 = (tid % (H / 4)) * 4, r8 = (tid / (H / 4)) * 8;

  float w1[kL1], w2[kL2], w3, bias = 0.f;
  float4 q0, q1;
  auto load = [&](const int4& w) {
    const size_t p = (size_t)w.x;
#pragma unroll
    for (int u = 0; u < kL1; ++u) w1[u] = __ldg(W1 + p * (kTIN * H) + u * kT + tid);
#pragma unroll
    for (int u = 0; u < kL2; ++u) w2[u] = __ldg(W2 + p * (H * H) + u * kT + tid);
    w3 = __ldg(W3 + p * (4 * H) + tid);
    if (tid < H) bias = __ldg(b1 + p * H + tid);
    else if (tid < 2 * H) bias = __ldg(b2 + p * H + tid - H);
    else if (tid < 2 * H + 4) bias = __ldg(b3 + p * 4 + tid - 2 * H);
    q0 = q1 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (rec < w.z) {
      const float4* src = reinterpret_cast<const float4*>(rec_in) + 2 * (size_t)(w.y + rec);
      q0 = __ldg(src);
      q1 = __ldg(src + 1);
    }
  };
  // acc[u][v] += w[k][h4 + u] * x[k][r8 + 2 v .. + 1]
  unsigned long long acc[4][4];
  auto step = [&](int x_off, int k, int w_off) {
    const ulonglong2 xa = *reinterpret_cast<const ulonglong2*>(sm + x_off + k * kTRow + r8);
    const ulonglong2 xb = *reinterpret_cast<const ulonglong2*>(sm + x_off + k * kTRow + r8 + 4);
    const float4 w = *reinterpret_cast<const float4*>(sm + w_off + k * N::kWRow + h4);
    const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const unsigned long long ww = pack_f32x2(wv[u], wv[u]);
      fma_f32x2(acc[u][0], xa.x, ww); fma_f32x2(acc[u][1], xa.y, ww);
      fma_f32x2(acc[u][2], xb.x, ww); fma_f32x2(acc[u][3], xb.y, ww);
    }
  };
  auto start = [&](int b_off) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float b = sm[b_off + h4 + u];
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[u][v] = pack_f32x2(b, b);
    }
  };
  auto relu_store = [&](int off) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float2 a = unpack_f32x2(acc[u][0]), b = unpack_f32x2(acc[u][1]), c = unpack_f32x2(acc[u][2]), d = unpack_f32x2(acc[u][3]);
      float* dst = sm + off + (h4 + u) * kTRow + r8;
      *reinterpret_cast<float4*>(dst) = make_float4(fmaxf(a.x, 0.f), fmaxf(a.y, 0.f), fmaxf(b.x, 0.f), fmaxf(b.y, 0.f));
      *reinterpret_cast<float4*>(dst + 4) = make_float4(fmaxf(c.x, 0.f), fmaxf(c.y, 0.f), fmaxf(d.x, 0.f), fmaxf(d.y, 0.f));
    }
  };

  int4 wk = __ldg(work + item);
  load(wk);
  for (;;) {
    const int rows = wk.z;
    const float decay = q1.z;
    const uint32_t slot = __float_as_uint(q1.w);
    __syncthreads();                       // the previous item's layers have been read
#pragma unroll
    for (int u = 0; u < kL1; ++u) { const int i = u * kT + tid; sm[N::kW1T + (i % kTIN) * N::kWRow + i / kTIN] = w1[u]; }
#pragma unroll
    for (int u = 0; u < kL2; ++u) { const int i = u * kT + tid; sm[N::kW2T + (i % H) * N::kWRow + i / H] = w2[u]; }
    sm[N::kW3T + (tid % H) * 4 + tid / H] = w3;
    if (tid < 2 * H + 4) sm[N::kB1 + tid] = bias;
    {
      const float v6[6] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y};
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        if ((c < 3) != (part == 0)) continue;
#pragma unroll
        for (int f = 0; f < kTF; ++f) {
          const float ph = v6[c] * fr[f] * at[f];
          sm[N::kE + (c * kTF + f) * kTRow + rec] = __sinf(ph);
          sm[N::kE + (36 + c * kTF + f) * kTRow + rec] = __cosf(ph);
        }
      }
    }
    const int next = item + (int)gridDim.x;
    const bool more = next < G;
    if (more) { wk = __ldg(work + next); load(wk); }
    __syncthreads();
    const bool live = r8 < rows;
    if (live) {
      start(N::kB1);
#pragma unroll 4
      for (int j = 0; j < kTIN / 2; ++j) { step(N::kE, j, N::kW1T); step(N::kE, kTIN / 2 + j, N::kW1T); }
      relu_store(N::kH1);
    }
    __syncthreads();
    if (live) {
      start(N::kB2);
#pragma unroll 8
      for (int k = 0; k < H; ++k) step(N::kH1, k, N::kW2T);
      relu_store(N::kE);                   // the encoding has been read
    }
    __syncthreads();
    if (tid < rows) {
      float o0 = sm[N::kB3], o1 = sm[N::kB3 + 1], o2 = sm[N::kB3 + 2], o3 = sm[N::kB3 + 3];
#pragma unroll 8
      for (int q = 0; q < H; ++q) {
        const float a = sm[N::kE + q * kTRow + tid];
        const float4 w = *reinterpret_cast<const float4*>(sm + N::kW3T + q * 4);
        o0 = fmaf(w.x, a, o0); o1 = fmaf(w.y, a, o1); o2 = fmaf(w.z, a, o2); o3 = fmaf(w.w, a, o3);
      }
      const float sigma_raw = softplus_fast(o3);
      float4 out;
      out.x = sigmoid_fast(o0); out.y = sigmoid_fast(o1); out.z = sigmoid_fast(o2);
      out.w = (out_mode == kOutAlpha) ? (1.f - __expf(-(sigma_raw * decay))) : sigma_raw;
      rec_out[slot] = out;
    }
    if (!more) break;
    item = next;
  }
}

int launch_mlp_f32(const mlpsp_scene* sc, const RecIn* rec_in, const int4* work,
                   const int32_t* counters, float4* rec_out, float4* rec_ext, int out_mode, int32_t* status,
                   cudaStream_t st, int grid_cap) {
  const int H = sc->hidden, F = sc->num_freq;
  MLPSP_REQUIRE(H >= 1 && H <= 64 && F >= 1 && F <= 8, MLPSP_E_LIMIT, "FP32 evaluator needs 1<=H<=64, 1<=F<=8");
  MLPSP_REQUIRE(sc->W1 && sc->b1 && sc->W2 && sc->b2 && sc->W3 && sc->b3 && sc->freq && sc->att, MLPSP_E_ARG,
                "FP32 evaluator needs the FP32 weight arrays");
  const int IN = 12 * F;
  const size_t smem = sizeof(float) * (size_t)(H * IN + H + H * H + H + 4 * H + 4 + 2 * F);
  const int sms = sm_count();
  const int grid = grid_cap > 0 ? std::min(grid_cap, sms * 8) : sms * 8;
  int32_t* ctr = const_cast<int32_t*>(counters);
  LaunchScope scope(kKMlp, 1, st);
  if (F == kTF && H == 32) {
    static_assert(sizeof(float) * PairBuf::kFloats <= 48 * 1024, "no opt-in needed");
    const int want = sms * kPairCtas;
    return cuda_check(launch_chained(k_mlp_f32_pair, dim3(grid_cap > 0 ? std::min(grid_cap, want) : want), dim3(kPairThreads),
                                     sizeof(float) * PairBuf::kFloats, st, sc->W1, sc->b1, sc->W2, sc->b2, sc->W3, sc->b3, sc->freq, sc->att,
                                     rec_in, work, ctr, ctr + kCtrWorkNext, rec_out, rec_ext, out_mode, status),
                      "mlp_f32");
  }
  if (F == kTF && H == 64 && !rec_ext) {
    using N = WideNet;
    static DeviceOnce attr_once;
    if (attr_once.first())
      MLPSP_CUDA_OK(cudaFuncSetAttribute(k_mlp_f32_wide, cudaFuncAttributeMaxDynamicSharedMemorySize, N::kFloats * 4));
    const int want = sms * N::kCtas;
    return cuda_check(launch_chained(k_mlp_f32_wide, dim3(grid_cap > 0 ? std::min(grid_cap, want) : want), dim3(N::kThreads), N::kFloats * 4, st,
                                     sc->W1, sc->b1, sc->W2, sc->b2, sc->W3, sc->b3, sc->freq, sc->att, rec_in, work, ctr, rec_out, out_mode, status),
                      "mlp_f32");
  }
  if (H <= 32) {
    k_mlp_f32<32><<<grid, kRowsPerItem, smem, st>>>(sc->W1, sc->b1, sc->W2, sc->b2, sc->W3, sc->b3, sc->freq, sc->att,
                                                   F, H, rec_in, work, ctr, rec_out, rec_ext, out_mode, status);
  } else {
    k_mlp_f32<64><<<grid, kRowsPerItem, smem, st>>>(sc->W1, sc->b1, sc->W2, sc->b2, sc->W3, sc->b3, sc->freq, sc->att,
                                                   F, H, rec_in, work, ctr, rec_out, rec_ext, out_mode, status);
  }
  return cuda_check(cudaGetLastError(), "mlp_f32");
}

}  // namespace mlpsp
