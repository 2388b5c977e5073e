// Per-primitive MLP evaluator on the 5th-generation tensor cores (tcgen05, sm_100a).
//
// What the reference does per (tile, primitive) with warp-level wmma on 64 rays
// (scannet/cuda/rgb_wmma.cuh:75-223) is done here per (primitive, 128 of its records):
//   * the primitive's weight image (packed once per scene in the canonical K-major core-matrix
//     layout, biases included) arrives in shared memory in three pieces, one per layer, each by a TMA
//     bulk copy (cp.async.bulk) that signals its own mbarrier;
//   * each of the 128 worker threads of a group owns one record (row): it encodes the record (sin / cos of 36 phases),
//     rounds to the operand format and stores the first 32 of the 80 K elements into a K-major tile in shared memory, the
//     others into tensor memory;
//   * layer 1 (128x80 . 80xH), layer 2 (128xH . HxH) and layer 3 (128xH . Hx16, 4 columns used) are
//     tcgen05.mma.kind::f16 instructions issued by one lane of the group's fifth warp, FP32 accumulators in tensor memory.
//     The biases ride in the same instructions, split into up to eight operand-format terms, so no thread ever
//     adds a bias: those of layer 1 meet a chunk of ones that fills its last K step, layers 2 and 3 (and layer 1
//     where records are kept) take one extra K step against a constant row of ones (eight rows of shared memory,
//     broadcast to all 128 by a zero row stride);
//   * between layers every thread pulls its accumulator row back with tcgen05.ld, applies ReLU while
//     rounding to the operand format and writes the next layer's A operand into tensor memory (tcgen05.st); the
//     epilogue applies sigmoid / softplus (and 1-exp(-sigma*decay)) and scatters one float4 per record to its
//     compositing slot.
// The three layers of item i, the encoding of item i+1 and the output of item i-1 are software-pipelined:
// every wait for a group of MMAs is preceded by independent work of a neighbouring item.
//
// What bounds it: the chain of an item, 5,000 to 6,000 cycles, most of them instructions of its five warps at 60 % of the issue
// slots; no other unit is half used.  So groups per SM and instructions count.  First wave of a 100,000-primitive frame at 1200 x
// 680 (6.9 M records in windows of 40): 223 us with a CTA per group, six per SM, the whole layer-1 operand in shared memory; the
// same with five per SM and most of it in tensor memory; 219 as six groups of one CTA; 188 with instructions taken out (warp
// number known to be uniform, no zeroing of absent records, one check of the outputs for layer 2's overflow, selections in
// softplus).  2, 3, 4, 5 groups: 432, 310, 255, 224.  As one CTA the groups' issue warps spread over the SM's four schedulers;
// in CTAs of their own all are fifth warps and share one (a warp's number decides).
//
// Numerics follow the reference's tensor-core contract: operands and hidden activations rounded
// to binary16 / bfloat16 (RN), FP32 accumulation from zero.
//
// Every wait on an mbarrier is bounded; when one gives up the CTA raises MLPSP_ST_TIMEOUT, waits
// (bounded) for its own copies, frees its tensor memory and returns.
#include <type_traits>
#include "frame.cuh"
#include "tc.cuh"

namespace mlpsp {

constexpr int kRows = kRowsPerItem;      // 128 = MMA M
constexpr int kChunk = kRows * 16;       // bytes of one K chunk of an A tile: [128 rows][8 halves]
constexpr int kN3 = 16, kOut = 4;        // the outputs, and the smallest N that holds them
constexpr int kA1Chunks = 10;            // 72 encoded inputs and a constant chunk that meets the bias terms
// of these in shared memory, and the columns of the others in tensor memory (two K elements each)
constexpr int kA1SmemChunks = 4, kA1TmemCols = (kA1Chunks - kA1SmemChunks) * 4;

// ---- packed weight image (per primitive) and shared-memory plan for F = 6, hidden width H = 32 or 64 ----
// piece 1: W1 as [10 chunks][H rows][8 halves]: K = 0..71 in the order of enc_k(), then the eight terms of b1[h];
// piece 2: W2 as [H/8 + 1 chunks][H][8], the last one the terms of b2;
// piece 3: W3 as [H/8 + 1 chunks][4][8], the last one the terms of b3.  The MMA has N = 16: its rows 4..7 are the next
//          chunk's rows, its rows 8..15 rows 0..7 again (a row-group stride of zero); nobody looks at their columns.
// With W3 padded to 16 rows an image took 8,960 / 21,760 bytes, and six small-group CTAs of 64-wide layers an SM's shared
// memory; seven fit now (four views of a million primitives: that kernel 2.84 -> 2.64 ms).
template <int H>
struct Net {
  static_assert(H == 32 || H == 64, "hidden width of the tensor-core evaluator");
  static constexpr int kWChunk = H * 16;
  static constexpr int kW3Chunk = kOut * 16;
  static constexpr int kOffW1 = 0;
  static constexpr int kBytesW1 = kA1Chunks * kWChunk;
  static constexpr int kOffW2 = kOffW1 + kBytesW1;
  static constexpr int kBytesW2 = (H / 8 + 1) * kWChunk;
  static constexpr int kOffW3 = kOffW2 + kBytesW2;
  static constexpr int kBytesW3 = (H / 8 + 1) * kW3Chunk;
  static constexpr int kWeightBytes = kOffW3 + kBytesW3;          // 8,000 (H = 32) / 20,032 (H = 64)
  // shared memory: weight image | zeros | eight rows of ones, eight rows of zeros | layer-1 A tile | barriers.  The second chunk
  // of a bias K step on the weight side is "whatever follows" (the next piece, or the zeros and constants after the image,
  // kWChunk bytes from the start of W3 on), always finite, and meets the zero rows on the A side.
  static constexpr int kOffConst = kOffW3 + (kBytesW3 + kW3Chunk > kWChunk ? (kBytesW3 + kW3Chunk + 127) / 128 * 128 : kWChunk);
  static_assert(kOffConst % 128 == 0 && kOffConst >= kOffW3 + kWChunk && kOffConst >= kWeightBytes + kW3Chunk, "what the MMAs read behind the image");
  static constexpr int kOffA1 = kOffConst + 256;                   // chunks 0..3 of the layer-1 operand; the others lie in tensor memory
  static constexpr int kOffBar = kOffA1 + kA1SmemChunks * kChunk;
  static constexpr int kSmemBytes = kOffBar + 96;                  // 16,736 / 29,024
  // tensor memory of a group: D1 and, once it has been read, D2 | the outputs | the hidden layers' operand (H / 2 columns, two
  // elements each) | chunks 4..9 of the layer-1 operand.  D3 begins in the last eight columns of D2, which has been read by then:
  // its columns 8..11 are the outputs again (see W3 above), past D2's end.
  static constexpr int kTmemCols = H == 32 ? 80 : 128;
  static constexpr int kD1 = 0, kD2 = 0, kD3 = H - 8, kOutputs = H, kA2 = H + 8, kA1 = kA2 + H / 2;
  // groups of a CTA, which has an SM to itself: by tensor memory (and H = 32 by registers, 64 a thread)
  static constexpr int kGroups = H == 32 ? 6 : 4, kGroupBytes = (kSmemBytes + 127) / 128 * 128;
  static constexpr int kThreads = kGroups * (kRows + 32);
  static_assert(kA1 + kA1TmemCols <= kTmemCols && kGroups * kTmemCols <= 512 && kGroups * kGroupBytes <= 227 * 1024, "plans");
  static_assert(kWeightBytes % 16 == 0 && kBytesW1 % 16 == 0 && kBytesW2 % 16 == 0 && kBytesW3 % 16 == 0, "bulk-copy granularity");
};

// Position of an encoded input inside the K dimension of layer 1.  The reference orders K as
// [sin(c,f) for c, f][cos(c,f) for c, f] (np_tile_kernels.cu:329-343); a dot product does not care, so
// the A tile and the packed W1 rows both use an order in which the six (sin, cos) pairs of one input
// coordinate are contiguous (six 32-bit words per coordinate):
//   k' = 12 c + 4 (f / 2) + 2 is_cos + (f % 2).
// The ray direction's 36 inputs fill the chunks 0..3 and the first half of chunk 4, the offset's the rest.
__host__ __device__ constexpr int enc_k(int c, int f, int is_cos) { return 12 * c + 4 * (f >> 1) + 2 * is_cos + (f & 1); }
__host__ __device__ constexpr int enc_k_of_reference(int k) { return enc_k((k % 36) / 6, (k % 36) % 6, k / 36); }
constexpr int kBiasChunk = 9;            // the terms of the layer-1 bias

// The six words of one input coordinate.  mult[f] is freq[f] * att[f].  LADDER: every band is exactly twice the
// one before, so the phases are exact doublings of the first and sin / cos of the higher bands follow from the
// double-angle identities (2 special-function evaluations per coordinate instead of 12).
template <bool LADDER, bool BF16>
__device__ __forceinline__ void encode_coord(float v, const float (&mult)[6], uint32_t (&w)[6]) {
  float sn[6], cs[6];
  if (LADDER) {
    __sincosf(v * mult[0], &sn[0], &cs[0]);
#pragma unroll
    for (int f = 1; f < 6; ++f) {
      const float t = sn[f - 1] + sn[f - 1];
      sn[f] = t * cs[f - 1];
      cs[f] = fmaf(-t, sn[f - 1], 1.0f);
    }
  } else {
#pragma unroll
    for (int f = 0; f < 6; ++f) __sincosf(v * mult[f], &sn[f], &cs[f]);
  }
#pragma unroll
  for (int g = 0; g < 3; ++g) {
    w[g * 2] = pack_h2<BF16>(sn[2 * g], sn[2 * g + 1]);
    w[g * 2 + 1] = pack_h2<BF16>(cs[2 * g], cs[2 * g + 1]);
  }
}

// A finite input gives finite phases (freq * att <= 101).  A NaN passes here: its sines and cosines make every activation of the
// first layer one, which that layer's check finds.
__device__ __forceinline__ bool too_large(float x, float y, float z) { return fmaxf(fmaxf(fabsf(x), fabsf(y)), fabsf(z)) >= 1.0e30f; }

template <bool BF16>
constexpr uint32_t kOnes2 = BF16 ? 0x3f803f80u : 0x3c003c00u;

// Three coordinates into this thread's row of the layer-1 A tile, the ray direction (OFF = false) or the offset (row =
// generic pointer to the row's 16 bytes inside chunk 0; kChunk = bytes between the K chunks), the first two and the third.
template <bool LADDER, bool BF16, bool OFF, int kChunk = mlpsp::kChunk>
__device__ __forceinline__ void encode_two(float x, float y, const float (&mult)[6], char* row) {
  uint32_t a[6], b[6];
  encode_coord<LADDER, BF16>(x, mult, a);
  encode_coord<LADDER, BF16>(y, mult, b);
  if (OFF) {
    *reinterpret_cast<uint2*>(row + 4 * kChunk + 8) = make_uint2(a[0], a[1]);
    *reinterpret_cast<uint4*>(row + 5 * kChunk) = make_uint4(a[2], a[3], a[4], a[5]);
    *reinterpret_cast<uint4*>(row + 6 * kChunk) = make_uint4(b[0], b[1], b[2], b[3]);
    *reinterpret_cast<uint2*>(row + 7 * kChunk) = make_uint2(b[4], b[5]);
  } else {
    *reinterpret_cast<uint4*>(row) = make_uint4(a[0], a[1], a[2], a[3]);
    *reinterpret_cast<uint4*>(row + kChunk) = make_uint4(a[4], a[5], b[0], b[1]);
    *reinterpret_cast<uint4*>(row + 2 * kChunk) = make_uint4(b[2], b[3], b[4], b[5]);
  }
}
template <bool LADDER, bool BF16, bool OFF, int kChunk = mlpsp::kChunk>
__device__ __forceinline__ void encode_one(float z, const float (&mult)[6], char* row) {
  uint32_t a[6];
  encode_coord<LADDER, BF16>(z, mult, a);
  if (OFF) {
    *reinterpret_cast<uint2*>(row + 7 * kChunk + 8) = make_uint2(a[0], a[1]);
    *reinterpret_cast<uint4*>(row + 8 * kChunk) = make_uint4(a[2], a[3], a[4], a[5]);
  } else {
    *reinterpret_cast<uint4*>(row + 3 * kChunk) = make_uint4(a[0], a[1], a[2], a[3]);
    *reinterpret_cast<uint2*>(row + 4 * kChunk) = make_uint2(a[4], a[5]);
  }
}
template <bool BF16, bool OFF, int kChunk = mlpsp::kChunk>
__device__ __forceinline__ void encode_three(bool ladder, float x, float y, float z, const float (&mult)[6], char* row) {
  if (ladder) {
    encode_two<true, BF16, OFF, kChunk>(x, y, mult, row);
    encode_one<true, BF16, OFF, kChunk>(z, mult, row);
  } else {
    encode_two<false, BF16, OFF, kChunk>(x, y, mult, row);
    encode_one<false, BF16, OFF, kChunk>(z, mult, row);
  }
}

// The same for the operand that lies half in shared, half in tensor memory: the first sixteen words of a direction go to the
// row's chunks 0..3, the other two (w_rest) and the eighteen of an offset to the columns of chunks 4..8.
template <bool LADDER, bool BF16>
__device__ __forceinline__ bool split_direction(float x, float y, float z, const float (&mult)[6], char* row, uint32_t (&w_rest)[2]) {
  uint32_t a[6], b[6], c[6];
  encode_coord<LADDER, BF16>(x, mult, a);
  encode_coord<LADDER, BF16>(y, mult, b);
  encode_coord<LADDER, BF16>(z, mult, c);
  *reinterpret_cast<uint4*>(row) = make_uint4(a[0], a[1], a[2], a[3]);
  *reinterpret_cast<uint4*>(row + kChunk) = make_uint4(a[4], a[5], b[0], b[1]);
  *reinterpret_cast<uint4*>(row + 2 * kChunk) = make_uint4(b[2], b[3], b[4], b[5]);
  *reinterpret_cast<uint4*>(row + 3 * kChunk) = make_uint4(c[0], c[1], c[2], c[3]);
  w_rest[0] = c[4]; w_rest[1] = c[5];
  return too_large(x, y, z);
}
template <bool LADDER, bool BF16>
__device__ __forceinline__ void split_offset_two(float x, float y, const float (&mult)[6], uint32_t col) {
  uint32_t a[6], b[6];
  encode_coord<LADDER, BF16>(x, mult, a);
  tmem_st2(col + 2, a[0], a[1]);
  tmem_st4(col + 4, a[2], a[3], a[4], a[5]);
  encode_coord<LADDER, BF16>(y, mult, b);
  tmem_st4(col + 8, b[0], b[1], b[2], b[3]);
  tmem_st2(col + 12, b[4], b[5]);
}
template <bool LADDER, bool BF16>
__device__ __forceinline__ void split_offset_one(float z, const float (&mult)[6], uint32_t col) {
  uint32_t a[6];
  encode_coord<LADDER, BF16>(z, mult, a);
  tmem_st2(col + 14, a[0], a[1]);
  tmem_st4(col + 16, a[2], a[3], a[4], a[5]);
}

// The encodings of the ray directions of a frame, in the operand format: per tile [5 chunks][64 pixels][16 bytes] (of the last
// one 8 bytes are used), so that
// the pixels of one tile -- neighbouring records of a primitive, mostly -- lie together in every chunk.
constexpr int kDirTileBytes = 5 * 64 * 16, kDirChunk = 64 * 16;

template <bool BF16>
__global__ void __launch_bounds__(256) k_encode_directions(const float* __restrict__ rays_d, int W, int H, int ntx, int T,
                                                           const float* __restrict__ freq, const float* __restrict__ att,
                                                           char* __restrict__ table) {
  chain_wait();
  chain_release();
  float mult[6];
  bool ladder = true;
#pragma unroll
  for (int f = 0; f < 6; ++f) mult[f] = __ldg(freq + f) * __ldg(att + f);
#pragma unroll
  for (int f = 1; f < 6; ++f) ladder = ladder && mult[f] == 2.0f * mult[f - 1];
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < (int64_t)T * 64; i += (int64_t)gridDim.x * 256) {
    const TilePix tp = tile_pixel((int)(i >> 6), (int)(i & 63), ntx, W, H);
    if (!tp.valid) continue;
    const V3 d = load3(rays_d, tp.pix);
    encode_three<BF16, false, kDirChunk>(ladder, d.x, d.y, d.z, mult, table + (i >> 6) * kDirTileBytes + (i & 63) * 16);
  }
}

// hidden layer epilogue: ReLU, operand format (RN), write this thread's row of the hidden A tile.  The biases are
// already in the accumulators.  Returns true when an activation rounded to +inf.  The FP32 sums themselves are
// finite for finite operands (rgb_wmma.cuh:179-181 checks for a non-finite or overflowing activation per element).
template <bool KEEP, bool BF16, int kChunk = mlpsp::kChunk>
__device__ __forceinline__ bool hidden_to_smem(const uint32_t (&acc)[32], char* a2, int row, uint32_t& relu_mask) {
  // running maximum of the packed activations (they are >= 0 after the ReLU, so for both formats the bit
  // patterns order like the values and one unsigned 16-bit-lane maximum serves either)
  uint32_t top = 0u;
  relu_mask = 0u;
#pragma unroll
  for (int kc = 0; kc < 4; ++kc) {
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int j = kc * 8 + q * 2;
      const float v0 = __uint_as_float(acc[j]), v1 = __uint_as_float(acc[j + 1]);
      if (KEEP) {
        relu_mask |= (v0 > 0.f ? 1u : 0u) << j;
        relu_mask |= (v1 > 0.f ? 1u : 0u) << (j + 1);
      }
      w[q] = pack_h2_relu<BF16>(v0, v1);
      top = __vmaxu2(top, w[q]);
    }
    *reinterpret_cast<uint4*>(a2 + kc * kChunk + row * 16) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  // +inf (or the canonical NaN a non-finite sum converts to) in either lane
  const uint32_t inf16 = BF16 ? 0x7f80u : 0x7c00u;
  return (top & 0xffffu) >= inf16 || (top >> 16) >= inf16;
}

// the same for 16 columns, into the operand's columns of tensor memory (taddr: first column, this warp's lanes)
template <bool KEEP, bool BF16, bool CHECK>
__device__ __forceinline__ uint32_t hidden_to_tmem(const uint32_t (&acc)[16], uint32_t taddr, int col, uint32_t& relu_mask) {
  uint32_t top = 0u, w[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const float v0 = __uint_as_float(acc[2 * q]), v1 = __uint_as_float(acc[2 * q + 1]);
    if (KEEP) {
      relu_mask |= (v0 > 0.f ? 1u : 0u) << (col + 2 * q);
      relu_mask |= (v1 > 0.f ? 1u : 0u) << (col + 2 * q + 1);
    }
    w[q] = pack_h2_relu<BF16>(v0, v1);
    if (CHECK) top = __vmaxu2(top, w[q]);
  }
  tmem_st8(taddr, w);
  return top;
}
template <bool BF16>
__device__ __forceinline__ bool overflowed(uint32_t top) {
  const uint32_t inf16 = BF16 ? 0x7f80u : 0x7c00u;
  return (top & 0xffffu) >= inf16 || (top >> 16) >= inf16;
}

// One work item = (primitive, first record, rows <= 128).  Items are dealt to CTAs, then groups, round-robin
// (item = blockIdx.x + (group + k * kGroups) * gridDim.x): all items cost about the same, and a fixed deal lets a group
// fetch the next items' descriptors, records and weight pieces while the current item is in flight.
//
// A CTA takes a whole SM and is kGroups groups of four worker warps (one record per thread) and an issue warp; the issue warps
// are the last ones.  Groups share nothing but the allocation of tensor memory, and nothing in the steady state is a CTA-wide
// barrier: the workers tell their issue warp that an operand tile is complete through an mbarrier that counts one arrival per
// worker warp, the issue warp (one lane) waits for that and for the layer's weight piece, issues the layer's MMAs and commits
// them to the mbarrier the workers wait on.  It also refills each weight piece as soon as the MMAs that read it have finished.  A
// worker warp, item i ("|" = while the MMAs run):
//   layer-1 tile of i complete -> arrive | output of i-1 (its layer-3 MMAs have finished by now)
//   wait layer 1: hidden tile 1 of i written -> arrive | first part of the encoding of i+1
//   wait layer 2: hidden tile 2 of i written -> arrive | second part of the encoding of i+1
// TAB: the records name their pixel, whose encoded direction is copied from the frame's table (k_encode_directions) into
// the A tile by cp.async: half of the 72 sines and cosines of a record are those of its ray, and a pixel has about a dozen
// records.  The record is then (offset, decay | slot, pixel); without it (direction, offset, decay, slot).
template <bool KEEP, bool BF16, int H, bool TAB>
__global__ void __launch_bounds__(Net<H>::kThreads, 1) k_mlp_tc(
    const char* __restrict__ w16, const float* __restrict__ freq, const float* __restrict__ att,
    const char* __restrict__ dir_table, const float4* __restrict__ rec_in, const int4* __restrict__ work,
    const int32_t* __restrict__ counters, float4* __restrict__ rec_out, float4* __restrict__ rec_ext, int out_mode,
    int32_t* __restrict__ status) {
  using N = Net<H>;
  static_assert(!KEEP || H == 32, "the record export keeps 32-bit ReLU masks");
  chain_wait();       // the work list and the records come from the previous kernels of the frame
  chain_release();
  extern __shared__ __align__(128) char smem_all[];
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int G = counters[kCtrWork];
  if ((int)blockIdx.x >= G) return;          // more CTAs than work: leave before touching tensor memory
  const int warp = warp_of_cta(), lane = threadIdx.x & 31;
  const bool issuer = warp >= 4 * N::kGroups;
  const int group = issuer ? warp - 4 * N::kGroups : warp >> 2, wrow = warp & 3, tid = wrow * 32 + lane;      // tid: a worker's row
  char* smem = smem_all + group * N::kGroupBytes;
  // [0..2] weight pieces landed, [3..5] operand tile of layer 1 / 2 / 3 complete, [6] layer-1 MMAs done, [7] layer-2 / 3 MMAs done
  uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + N::kOffBar);
  uint32_t* s_misc = reinterpret_cast<uint32_t*>(s_bar + 8);          // [0] tmem base (the first group's), [1] a wait gave up
  int item = group * (int)gridDim.x + (int)blockIdx.x;
  const int stride = N::kGroups * (int)gridDim.x;
  const uint32_t wb = smem_u32(smem), cst = wb + N::kOffConst, a1 = wb + N::kOffA1;
  const uint32_t bar_w0 = smem_u32(&s_bar[0]), bar_r0 = smem_u32(&s_bar[3]), bar_a = smem_u32(&s_bar[6]), bar_b = smem_u32(&s_bar[7]);
  if (issuer) {
    if (lane == 0) {
#pragma unroll
      for (int b = 0; b < 3; ++b) { mbar_init(bar_w0 + 8 * b, 1); mbar_init(bar_r0 + 8 * b, kRows / 32); }
      mbar_init(bar_a, 1);
      mbar_init(bar_b, 1);
      s_misc[1] = 0u;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (group == 0) tmem_alloc(smem_u32(&s_misc[0]), 512);
  } else {
    if (tid < 16) {
      const uint32_t v = tid < 8 ? kOnes2<BF16> : 0u;
      *reinterpret_cast<uint4*>(smem + N::kOffConst + tid * 16) = make_uint4(v, v, v, v);
    }
    if (tid < (N::kOffConst - N::kWeightBytes) / 16) *reinterpret_cast<uint4*>(smem + N::kWeightBytes + tid * 16) = make_uint4(0u, 0u, 0u, 0u);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_all = *reinterpret_cast<const uint32_t*>(smem_all + N::kOffBar + 64);
  const uint32_t tmem = tmem_all + group * N::kTmemCols, a1t = tmem + N::kA1;
  bool ok = true;

  if (item >= G) {
    // fewer items than groups
  } else if (issuer) {
    // ------------------------------------------------------------------ issue warp ----
    const uint32_t idesc_h = instr_desc(kRows, H, BF16), idesc_o = instr_desc(kRows, kN3, BF16);
    // Operand descriptors are built once; a K step only moves the start address, which sits in the low bits in
    // units of 16 bytes (shared-memory addresses stay below 2^18, so the sum never carries out of the field).
    const uint64_t a1_desc = smem_desc(a1, kChunk, 128);
    const uint64_t ones_desc = smem_desc(cst, 128, 0);     // rows of ones, then rows of zeros; every row group the same
    const uint64_t w1_desc = smem_desc(wb + N::kOffW1, N::kWChunk, 128), w2_desc = smem_desc(wb + N::kOffW2, N::kWChunk, 128);
    const uint64_t w3_desc = smem_desc(wb + N::kOffW3, N::kW3Chunk, 0);
    auto step = [](uint64_t desc, int bytes) { return desc + (uint64_t)(bytes >> 4); };
    auto request = [&](int piece, int prim) {
      const int off = piece == 0 ? N::kOffW1 : (piece == 1 ? N::kOffW2 : N::kOffW3);
      const int bytes = piece == 0 ? N::kBytesW1 : (piece == 1 ? N::kBytesW2 : N::kBytesW3);
      mbar_expect_tx(bar_w0 + 8 * piece, bytes);
      bulk_g2s(wb + off, w16 + (size_t)prim * N::kWeightBytes + off, bytes, bar_w0 + 8 * piece);
    };
    // every lane waits, one issues
    auto both = [&](uint32_t x, uint32_t y, uint32_t parity) {
      return __all_sync(0xffffffffu, mbar_wait(x, parity) && mbar_wait(y, parity)) != 0;
    };
    auto done = [&](uint32_t x, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(x, parity)) != 0; };
    int prim = __ldg(work + item).x;
    uint32_t pend = 7u;                    // weight pieces requested and not yet waited for
    if (elect_one()) { request(0, prim); request(1, prim); request(2, prim); }
    uint32_t li = 0u;
    for (;;) {
      const uint32_t par = li & 1u;
      const int next = item + stride;
      const bool has_next = next < G;
      int prim_n = 0;
      if (has_next) prim_n = __ldg(work + next).x;
      // ---- layer 1: D1[128xH] = A1[128x80] . W1^T, the biases included ----
      ok = both(bar_r0, bar_w0, par);
      pend &= ~1u;
      // The second chunk of a bias K step (layers 2 and 3) reads the start of the next piece's region as don't-care data
      // (it meets zeros), which must still be finite: before the first item all three pieces have to be in place,
      // afterwards the regions always hold the previous or the incoming image.
      if (ok && li == 0u) ok = both(bar_w0 + 8, bar_w0 + 16, 0u);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < kA1Chunks / 2; ++ks) {
          const uint64_t w = step(w1_desc, ks * 2 * N::kWChunk);
          if (ks < kA1SmemChunks / 2) mma_f16(tmem + N::kD1, step(a1_desc, ks * 2 * kChunk), w, idesc_h, ks > 0);
          else mma_f16_ta(tmem + N::kD1, a1t + (ks - kA1SmemChunks / 2) * 8, w, idesc_h, 1u);
        }
        if (KEEP) mma_f16(tmem + N::kD1, ones_desc, step(w1_desc, kBiasChunk * N::kWChunk), idesc_h, 1u);
        mma_commit(bar_a);
      }
      __syncwarp();
      if (!(ok = done(bar_a, par))) break;
      if (has_next) {                                            // W1 is no longer read
        if (elect_one()) request(0, prim_n);
        pend |= 1u;
      }
      // ---- layer 2: D2[128xH] = H1[128xH] . W2^T + b2 ----
      ok = both(bar_r0 + 8, bar_w0 + 8, par);
      pend &= ~2u;
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < H / 16; ++ks)
          mma_f16_ta(tmem + N::kD2, tmem + N::kA2 + ks * 8, step(w2_desc, ks * 2 * N::kWChunk), idesc_h, ks > 0);
        mma_f16(tmem + N::kD2, ones_desc, step(w2_desc, (H / 8) * N::kWChunk), idesc_h, 1u);
        mma_commit(bar_b);
      }
      __syncwarp();
      if (!(ok = done(bar_b, 0u))) break;
      if (has_next) {
        if (elect_one()) request(1, prim_n);
        pend |= 2u;
      }
      // ---- layer 3: D3[128x16] = H2[128xH] . W3^T + b3 (of 16 columns the first four are looked at) ----
      ok = both(bar_r0 + 16, bar_w0 + 16, par);
      pend &= ~4u;
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < H / 16; ++ks)
          mma_f16_ta(tmem + N::kD3, tmem + N::kA2 + ks * 8, step(w3_desc, ks * 2 * N::kW3Chunk), idesc_o, ks > 0);
        mma_f16(tmem + N::kD3, ones_desc, step(w3_desc, (H / 8) * N::kW3Chunk), idesc_o, 1u);
        mma_commit(bar_b);
      }
      __syncwarp();
      if (!(ok = done(bar_b, 1u))) break;
      if (!has_next) break;
      if (elect_one()) request(2, prim_n);
      pend |= 4u;
      item = next;
      prim = prim_n;
      ++li;
    }
    if (!ok) {
      if (lane == 0) s_misc[1] = 1u;
      // our own bulk copies may still be in flight: give them a bounded chance to land before the CTA's
      // shared memory is released
      for (int b = 0; b < 3; ++b)
        if (pend & (1u << b)) mbar_wait(bar_w0 + 8 * b, li & 1u);
    }
    __syncwarp();
  } else {
    // ---------------------------------------------------------------- worker warps ----
    const uint32_t trow = tmem + ((uint32_t)(wrow * 32) << 16), a1row = a1t + ((uint32_t)(wrow * 32) << 16);   // this warp's 32 lanes
    // the constant chunk of layer 1: ones, so that the bias rides in its last K step; with KEEP zeros, and the bias a step of its
    // own as in layers 2 and 3 (the order of the sums decides saved ReLU signs of values next to zero)
    {
      const uint32_t v = KEEP ? 0u : kOnes2<BF16>;
      tmem_st4(a1row + (kBiasChunk - kA1SmemChunks) * 4, v, v, v, v);
    }
    // phase multipliers freq[f] * att[f]; when every band is exactly twice the one before (equal
    // attenuation: FourierFeatureEncoding's bands, cumodel.py:163) the encoder takes the double-angle route
    float mult[6];
    bool ladder = true;
#pragma unroll
    for (int f = 0; f < 6; ++f) mult[f] = __ldg(freq + f) * __ldg(att + f);
#pragma unroll
    for (int f = 1; f < 6; ++f) ladder = ladder && mult[f] == 2.0f * mult[f - 1];
    int4 wk = __ldg(work + item);
    int4 wk_n = __ldg(work + min(item + stride, G - 1));       // (past the list's end: any item, and nobody encodes it)
    auto load_rec = [&](const int4& w, float4& r0, float4& r1) {     // rows past the end keep their last record and store nothing
      if (tid < w.z) { r0 = __ldg(rec_in + 2 * (size_t)(w.y + tid)); r1 = __ldg(rec_in + 2 * (size_t)(w.y + tid) + 1); }
    };
    auto rec_decay = [](const float4& r0, const float4& r1) { return TAB ? r0.w : r1.z; };
    auto rec_slot = [](const float4& r1) { return TAB ? __float_as_uint(r1.x) : __float_as_uint(r1.w); };
    // the pixel's encoded direction on its way to this thread's row of the A tile; its last two words
    auto copy_direction = [&](const float4& r1) {
      const uint32_t pixel = __float_as_uint(r1.y);
      const char* src = dir_table + (size_t)(pixel >> 6) * kDirTileBytes + (pixel & 63u) * 16;
      const uint32_t dst = a1 + tid * 16;
#pragma unroll
      for (int c = 0; c < 4; ++c) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + c * kChunk), "l"(src + c * kDirChunk) : "memory");
      return __ldg(reinterpret_cast<const uint2*>(src + 4 * kDirChunk));
    };
    auto direction_landed = [&]() { asm volatile("cp.async.wait_all;" ::: "memory"); };
    char* my_row = smem + N::kOffA1 + tid * 16;
    // a hidden layer of the warp's rows: accumulator columns from d on -> operand
    // (check: the first layer.  An infinite activation there may leave the second only sums of minus infinity, which its ReLU
    // hides; one of the second makes every output infinite or not a number, which emit_output looks at.)
    auto hidden = [&](uint32_t d, uint32_t& relu_mask, auto check) {
      uint32_t top = 0u;
      relu_mask = 0u;
#pragma unroll
      for (int part = 0; part < H / 16; ++part) {
        uint32_t acc[16];
        tmem_ld16(trow + d + part * 16, acc);
        const uint32_t t = hidden_to_tmem<KEEP, BF16, decltype(check)::value>(acc, trow + N::kA2 + part * 8, part * 16, relu_mask);
        top = __vmaxu2(top, t);
      }
      return overflowed<BF16>(top);
    };
    // the warp's rows of an operand tile are complete (and its reads of tensor memory have retired); in_smem: some of
    // it was written to shared memory
    auto tile_done = [&](uint32_t bar, bool in_smem = false) {
      tmem_st_wait();
      if (in_smem) fence_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
    };
    bool bad = false;
    uint2 rest = make_uint2(0u, 0u);           // the last two words of the next record's direction
    auto direction = [&](float x, float y, float z) {
      uint32_t w[2];
      bad |= ladder ? split_direction<true, BF16>(x, y, z, mult, my_row, w) : split_direction<false, BF16>(x, y, z, mult, my_row, w);
      rest = make_uint2(w[0], w[1]);
    };
    auto offset_two = [&](float x, float y) {
      if (ladder) split_offset_two<true, BF16>(x, y, mult, a1row); else split_offset_two<false, BF16>(x, y, mult, a1row);
    };
    auto offset_one = [&](float x, float y, float z) {       // (x, y: for the check)
      bad |= too_large(x, y, z);
      if (ladder) split_offset_one<true, BF16>(z, mult, a1row); else split_offset_one<false, BF16>(z, mult, a1row);
      tmem_st2(a1row, rest.x, rest.y);
    };
    // ---- prologue: the first item's record, encoded in full ----
    float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0;
    load_rec(wk, q0, q1);
    // MMA rows are independent and rows past the end of the primitive's records are never stored, so a
    // warp whose 32 rows are all past the end skips the encoding and the epilogues (its rows of the
    // operand tiles keep whatever they held) and only reports its tiles complete
    if (wrow * 32 < wk.z) {
      if (TAB) {
        rest = copy_direction(q1);
        offset_two(q0.x, q0.y);
        offset_one(q0.x, q0.y, q0.z);
        direction_landed();
      } else {
        direction(q0.x, q0.y, q0.z);
        offset_two(q0.w, q1.x);
        offset_one(q0.w, q1.x, q1.y);
      }
    }
    tile_done(bar_r0, true);
    float decay_c = rec_decay(q0, q1);
    uint32_t slot_c = rec_slot(q1);
    load_rec(wk_n, q0, q1);                    // the second item's record

    bool have_prev = false, live_p = false, valid_p = false;
    float decay_p = 0.f;
    uint32_t slot_p = 0u, relu1 = 0u, relu2 = 0u, relu1_p = 0u, relu2_p = 0u;
    uint32_t li = 0u;                          // items this group has started: parity of the once-per-item barriers

    auto emit_output = [&]() {
      // output of the item whose layer-3 MMAs have just finished: (decay_p, slot_p), accumulator columns [H, H + 4)
      if (!live_p) return;
      uint32_t o[4];
      tmem_ld4(trow + N::kOutputs, o);
      if (valid_p) {
        const float o0 = __uint_as_float(o[0]), o1 = __uint_as_float(o[1]), o2 = __uint_as_float(o[2]), o3 = __uint_as_float(o[3]);
        const float sigma_raw = softplus_fast(o3);
        bad |= !(fabsf((o0 + o1) + (o2 + o3)) < 3.0e38f);
        float4 out;
        out.x = sigmoid_fast(o0); out.y = sigmoid_fast(o1); out.z = sigmoid_fast(o2);
        out.w = (out_mode == kOutAlpha) ? (1.f - __expf(-(sigma_raw * decay_p))) : sigma_raw;
        rec_out[slot_p] = out;
        if (KEEP) rec_ext[slot_p] = make_float4(sigma_raw, o3, __uint_as_float(relu1_p), __uint_as_float(relu2_p));
      }
    };

    for (;;) {
      const int nrows = wk.z;
      const bool valid = tid < nrows;
      const bool warp_live = wrow * 32 < nrows;
      const int next = item + stride;
      const bool has_next = next < G;
      const bool next_live = has_next && wrow * 32 < wk_n.z;
      const uint32_t par = li & 1u;
      // descriptor of the item after the next one
      const int next2 = next + stride;
      const int4 wk_n2 = __ldg(work + min(next2, G - 1));
      // ---- output of the previous item while layer 1 of this one runs ----
      if (have_prev) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar_b, 1u) && ok);   // warp-uniform: tcgen05.ld is .sync.aligned
        tc_fence_after();
        if (!ok) break;
        emit_output();
      }
      ok = __all_sync(0xffffffffu, mbar_wait(bar_a, par) && ok);
      tc_fence_after();
      if (!ok) break;
      // layer 1 no longer reads the A tile: the next item's directions are in flight over two round trips
      if (TAB && next_live) rest = copy_direction(q1);
      // the record this thread will load at the end of this item (for the item after the next) is asked into L2 now (with the
      // table of directions L2 is busy enough: 100k frame 816 us, without 811)
      if (!TAB && tid < wk_n2.z) asm volatile("prefetch.global.L2 [%0];" ::"l"(rec_in + 2 * (size_t)(wk_n2.y + tid)));
      if (warp_live) bad |= hidden(N::kD1, relu1, std::true_type{}) && valid;
      tile_done(bar_r0 + 8);
      // ---- first part of the next item's encoding while layer 2 runs ----
      if (next_live) {
        if (!TAB) direction(q0.x, q0.y, q0.z);
        else offset_two(q0.x, q0.y);
      }
      ok = __all_sync(0xffffffffu, mbar_wait(bar_b, 0u) && ok);
      tc_fence_after();
      if (!ok) break;
      if (warp_live) hidden(N::kD2, relu2, std::false_type{});
      tile_done(bar_r0 + 16);
      // ---- second part of the next item's encoding while layer 3 runs ----
      if (next_live) {
        if (!TAB) {
          offset_two(q0.w, q1.x);
          offset_one(q0.w, q1.x, q1.y);
        } else {
          offset_one(q0.x, q0.y, q0.z);
          direction_landed();
        }
      }
      // this item becomes the one whose output is pending; the next one becomes current
      have_prev = true;
      live_p = warp_live; valid_p = valid; decay_p = decay_c; slot_p = slot_c; relu1_p = relu1; relu2_p = relu2;
      if (!has_next) break;
      tile_done(bar_r0, true);
      decay_c = rec_decay(q0, q1);
      slot_c = rec_slot(q1);
      item = next;
      wk = wk_n;
      wk_n = wk_n2;
      load_rec(wk_n, q0, q1);
      ++li;
    }
    if (ok && have_prev) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar_b, 1u) && ok);
      tc_fence_after();
      if (ok) emit_output();
    }
    if (!ok && lane == 0) s_misc[1] = 1u;
    if (bad) atomicOr(status + MLPSP_ST_BITS, MLPSP_ST_NUMERIC);
  }
  tc_fence_before();
  __syncthreads();
  if (issuer && lane == 0 && s_misc[1]) atomicOr(status + MLPSP_ST_BITS, MLPSP_ST_TIMEOUT);
  if (issuer && group == 0) tmem_free(tmem_all, 512);
}

// ------------------------------------------------------------------ small groups ----
// Work items of at most 32 records (the remainder of a primitive's records when it is small: most primitives of a
// scene with millions of primitives own a few records per wave).  A 128-row item would carry one live warp and
// three idle ones through the same chain of MMA round trips, and only six (H = 64: four) of them fit an SM.  Here one warp IS
// the CTA: the operand tiles hold 32 rows (chunk stride 512 bytes; the MMA still has M = 128 and reads, as rows
// 32..127, whatever follows -- those accumulator rows are never looked at), the accumulators of the three layers
// share 32 (H = 64: 64) columns of tensor memory, lane 0 issues the MMAs between __syncwarp()s, and 12 (7) such
// CTAs fit an SM.  Same weight pieces, same bias folding, same arithmetic as k_mlp_tc.
constexpr int kMiniRows = kRowsPerSmallItem;
constexpr int kMiniChunk = kMiniRows * 16;

template <int H>
struct MiniNet {
  using N = Net<H>;
  static constexpr int kOffConst = N::kOffConst;
  static constexpr int kOffA1 = kOffConst + 256;
  static constexpr int kOffA2 = kOffA1 + kA1Chunks * kMiniChunk;
  static constexpr int kOffPad = kOffA2 + (H / 8) * kMiniChunk;     // rows 32..127 of the last hidden chunk land here (with the
  static constexpr int kOffBar = kOffPad + (kRows - kMiniRows) * 16;  // weight image there instead an item takes 15 % longer)
  static constexpr int kSmemBytes = kOffBar + 64;                   // 17,216 (H = 32) / 31,552 (H = 64)
  static constexpr int kTmemCols = H;
  static constexpr int kCtas = H == 32 ? 12 : 7;
  static_assert(kCtas * (kSmemBytes + 1024) <= 228 * 1024 && kCtas * kTmemCols <= 512, "resident CTAs");
};

template <bool BF16, int H>
__global__ void __launch_bounds__(kMiniRows, MiniNet<H>::kCtas) k_mlp_tc_mini(
    const char* __restrict__ w16, const float* __restrict__ freq, const float* __restrict__ att,
    const float4* __restrict__ rec_in, const int4* __restrict__ work, const int32_t* __restrict__ counters,
    float4* __restrict__ rec_out, int out_mode, int32_t* __restrict__ status) {
  using N = Net<H>;
  using M = MiniNet<H>;
  chain_wait();
  chain_release();
  extern __shared__ __align__(128) char smem[];
  char* s_a1 = smem + M::kOffA1;
  char* s_a2 = smem + M::kOffA2;
  uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + M::kOffBar);   // [0..2] weight pieces, [3] MMAs of a layer done
  uint32_t* s_misc = reinterpret_cast<uint32_t*>(s_bar + 4);
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int lane = threadIdx.x;
  const int G = counters[kCtrWorkSmall];
  int item = blockIdx.x;
  if (item >= G) return;
  const int stride = (int)gridDim.x;
  const uint32_t wb = smem_u32(smem), a1 = wb + M::kOffA1, a2 = wb + M::kOffA2;
  const uint32_t bar_w0 = smem_u32(&s_bar[0]), bar_m = smem_u32(&s_bar[3]);
  if (lane == 0) {
#pragma unroll
    for (int b = 0; b < 4; ++b) mbar_init(bar_w0 + 8 * b, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tmem_alloc(smem_u32(&s_misc[0]), M::kTmemCols);
  if (lane < 16) {
    const uint32_t v = lane < 8 ? kOnes2<BF16> : 0u;
    *reinterpret_cast<uint4*>(smem + M::kOffConst + lane * 16) = make_uint4(v, v, v, v);
  }
  if (lane < (N::kOffConst - N::kWeightBytes) / 16) *reinterpret_cast<uint4*>(smem + N::kWeightBytes + lane * 16) = make_uint4(0u, 0u, 0u, 0u);
  *reinterpret_cast<uint4*>(s_a1 + kBiasChunk * kMiniChunk + lane * 16) = make_uint4(kOnes2<BF16>, kOnes2<BF16>, kOnes2<BF16>, kOnes2<BF16>);
  fence_async_smem();
  tc_fence_before();
  __syncwarp();
  tc_fence_after();
  const uint32_t tmem = s_misc[0];
  float mult[6];
  bool ladder = true;
#pragma unroll
  for (int f = 0; f < 6; ++f) mult[f] = __ldg(freq + f) * __ldg(att + f);
#pragma unroll
  for (int f = 1; f < 6; ++f) ladder = ladder && mult[f] == 2.0f * mult[f - 1];
  const uint64_t ones_desc = smem_desc(wb + M::kOffConst, 128, 0);
  const uint32_t idesc_h = instr_desc(kRows, H, BF16), idesc_o = instr_desc(kRows, kN3, BF16);
  const uint64_t a1_desc = smem_desc(a1, kMiniChunk, 128), a2_desc = smem_desc(a2, kMiniChunk, 128);
  const uint64_t w1_desc = smem_desc(wb + N::kOffW1, N::kWChunk, 128), w2_desc = smem_desc(wb + N::kOffW2, N::kWChunk, 128);
  const uint64_t w3_desc = smem_desc(wb + N::kOffW3, N::kW3Chunk, 0);
  auto step = [](uint64_t desc, int bytes) { return desc + (uint64_t)(bytes >> 4); };
  auto request = [&](int piece, int prim) {
    const int off = piece == 0 ? N::kOffW1 : (piece == 1 ? N::kOffW2 : N::kOffW3);
    const int bytes = piece == 0 ? N::kBytesW1 : (piece == 1 ? N::kBytesW2 : N::kBytesW3);
    mbar_expect_tx(bar_w0 + 8 * piece, bytes);
    bulk_g2s(wb + off, w16 + (size_t)prim * N::kWeightBytes + off, bytes, bar_w0 + 8 * piece);
  };
  auto load_rec = [&](const int4& w, float4& r0, float4& r1) {       // rows past the end keep their last record and store nothing
    if (lane < w.z) { r0 = __ldg(rec_in + 2 * (size_t)(w.y + lane)); r1 = __ldg(rec_in + 2 * (size_t)(w.y + lane) + 1); }
  };
  // the warp's writes to an operand tile are visible to the tensor core, its reads of tensor memory have retired
  auto tile_done = [&]() {
    fence_async_smem();
    tc_fence_before();
    __syncwarp();
  };
  int4 wk = __ldg(work + item);
  int4 wk_n = __ldg(work + min(item + stride, G - 1));
  uint32_t pend = 0u;
  if (elect_one()) { request(0, wk.x); request(1, wk.x); request(2, wk.x); }
  pend = 7u;
  char* my_row = s_a1 + lane * 16;
  bool bad = false, ok = true;
  float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0;
  load_rec(wk, q0, q1);
  auto direction = [&]() {
    encode_three<BF16, false, kMiniChunk>(ladder, q0.x, q0.y, q0.z, mult, my_row);
    bad |= too_large(q0.x, q0.y, q0.z);
  };
  auto offset = [&]() {
    encode_three<BF16, true, kMiniChunk>(ladder, q0.w, q1.x, q1.y, mult, my_row);
    bad |= too_large(q0.w, q1.x, q1.y);
  };
  direction();
  offset();
  float decay_c = q1.z;
  uint32_t slot_c = __float_as_uint(q1.w);
  load_rec(wk_n, q0, q1);
  uint32_t li = 0u, ph = 0u, relu_unused = 0u;   // ph: phases of the MMA barrier completed so far
  const uint32_t trow = tmem;   // warp 0 of the CTA: lanes 0..31

  for (;;) {
    const bool valid = lane < wk.z;
    const int next = item + stride;
    const bool has_next = next < G;
    const uint32_t par = li & 1u;
    const int next2 = next + stride;
    const int4 wk_n2 = __ldg(work + min(next2, G - 1));
    // ---- layer 1 ----
    tile_done();
    bool landed = mbar_wait(bar_w0, par);
    if (li == 0u) landed = landed && mbar_wait(bar_w0 + 8, 0u) && mbar_wait(bar_w0 + 16, 0u);   // see k_mlp_tc
    pend &= ~1u;
    ok = __all_sync(0xffffffffu, landed) != 0;
    if (!ok) break;
    tc_fence_after();
    if (elect_one()) {
#pragma unroll
      for (int ks = 0; ks < kA1Chunks / 2; ++ks)
        mma_f16(tmem, step(a1_desc, ks * 2 * kMiniChunk), step(w1_desc, ks * 2 * N::kWChunk), idesc_h, ks > 0);
      mma_commit(bar_m);
    }
    __syncwarp();
    if (lane < wk_n2.z) asm volatile("prefetch.global.L2 [%0];" ::"l"(rec_in + 2 * (size_t)(wk_n2.y + lane)));
    ok = __all_sync(0xffffffffu, mbar_wait(bar_m, ph++ & 1u) && ok);   // one completion per layer
    tc_fence_after();
    if (!ok) break;
    if (has_next) {
      if (elect_one()) request(0, wk_n.x);
      pend |= 1u;
    }
#pragma unroll
    for (int part = 0; part < H / 32; ++part) {
      uint32_t acc[32];
      tmem_ld32(trow + part * 32, acc);
      bad |= hidden_to_smem<false, BF16, kMiniChunk>(acc, s_a2 + part * 4 * kMiniChunk, lane, relu_unused) && valid;
    }
    // ---- layer 2 (its accumulator takes the columns of layer 1) ----
    tile_done();
    ok = __all_sync(0xffffffffu, mbar_wait(bar_w0 + 8, par)) != 0;
    pend &= ~2u;
    if (!ok) break;
    tc_fence_after();
    if (elect_one()) {
#pragma unroll
      for (int ks = 0; ks < H / 16; ++ks)
        mma_f16(tmem, step(a2_desc, ks * 2 * kMiniChunk), step(w2_desc, ks * 2 * N::kWChunk), idesc_h, ks > 0);
      mma_f16(tmem, ones_desc, step(w2_desc, (H / 8) * N::kWChunk), idesc_h, 1u);
      mma_commit(bar_m);
    }
    __syncwarp();
    // first part of the next item's encoding while layer 2 runs (the layer-1 tile is free)
    if (has_next) direction();
    ok = __all_sync(0xffffffffu, mbar_wait(bar_m, ph++ & 1u) && ok);
    tc_fence_after();
    if (!ok) break;
    if (has_next) {
      if (elect_one()) request(1, wk_n.x);
      pend |= 2u;
    }
#pragma unroll
    for (int part = 0; part < H / 32; ++part) {
      uint32_t acc[32];
      tmem_ld32(trow + part * 32, acc);
      hidden_to_smem<false, BF16, kMiniChunk>(acc, s_a2 + part * 4 * kMiniChunk, lane, relu_unused);      // (checked at the outputs, see k_mlp_tc)
    }
    // ---- layer 3 ----
    tile_done();
    ok = __all_sync(0xffffffffu, mbar_wait(bar_w0 + 16, par)) != 0;
    pend &= ~4u;
    if (!ok) break;
    tc_fence_after();
    if (elect_one()) {
#pragma unroll
      for (int ks = 0; ks < H / 16; ++ks)
        mma_f16(tmem, step(a2_desc, ks * 2 * kMiniChunk), step(w3_desc, ks * 2 * N::kW3Chunk), idesc_o, ks > 0);
      mma_f16(tmem, ones_desc, step(w3_desc, (H / 8) * N::kW3Chunk), idesc_o, 1u);
      mma_commit(bar_m);
    }
    __syncwarp();
    if (has_next) offset();
    ok = __all_sync(0xffffffffu, mbar_wait(bar_m, ph++ & 1u) && ok);
    tc_fence_after();
    if (!ok) break;
    if (has_next) {
      if (elect_one()) request(2, wk_n.x);
      pend |= 4u;
    }
    {
      uint32_t o[4];
      tmem_ld4(trow, o);
      if (valid) {
        const float o0 = __uint_as_float(o[0]), o1 = __uint_as_float(o[1]), o2 = __uint_as_float(o[2]), o3 = __uint_as_float(o[3]);
        const float sigma_raw = softplus_fast(o3);
        bad |= !(fabsf((o0 + o1) + (o2 + o3)) < 3.0e38f);
        float4 out;
        out.x = sigmoid_fast(o0); out.y = sigmoid_fast(o1); out.z = sigmoid_fast(o2);
        out.w = (out_mode == kOutAlpha) ? (1.f - __expf(-(sigma_raw * decay_c))) : sigma_raw;
        rec_out[slot_c] = out;
      }
    }
    if (!has_next) break;
    decay_c = q1.z;
    slot_c = __float_as_uint(q1.w);
    item = next;
    wk = wk_n;
    wk_n = wk_n2;
    load_rec(wk_n, q0, q1);
    ++li;
  }
  if (!ok) {
    if (lane == 0) atomicOr(status + MLPSP_ST_BITS, MLPSP_ST_TIMEOUT);
    for (int b = 0; b < 3; ++b)
      if (pend & (1u << b)) mbar_wait(bar_w0 + 8 * b, li & 1u);
  }
  if (bad) atomicOr(status + MLPSP_ST_BITS, MLPSP_ST_NUMERIC);
  tc_fence_before();
  __syncwarp();
  tmem_free(tmem, M::kTmemCols);
}

// ------------------------------------------------------------------------------ packing ----
template <bool BF16>
__device__ __forceinline__ uint16_t to_lp(float x, bool& bad) {
  if (BF16) {
    const __nv_bfloat16 v = __float2bfloat16_rn(x);
    bad |= __hisinf(v) || __hisnan(v);
    return *reinterpret_cast<const uint16_t*>(&v);
  }
  const __half v = __float2half_rn(x);
  bad |= __hisinf(v) || __hisnan(v);
  return *reinterpret_cast<const uint16_t*>(&v);
}
template <bool BF16>
__device__ __forceinline__ float from_lp(uint16_t u) {
  if (BF16) return __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(&u));
  return __half2float(*reinterpret_cast<const __half*>(&u));
}

// A bias as a sum of up to eight operand-format terms (greedy: each term is the remainder clamped to the
// format's range and rounded): three terms carry every FP32 mantissa bit, the others serve biases beyond the
// format's range (8 x 65504 for binary16).  A bias that does not fit is reported.
template <bool BF16>
__device__ __forceinline__ void bias_terms(float b, uint16_t* dst /* [8] */, bool& bad) {
  const float lim = BF16 ? 3.3e38f : 65504.f;
  float rem = b;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    bool ignore = false;
    const uint16_t t = to_lp<BF16>(fminf(fmaxf(rem, -lim), lim), ignore);
    dst[j] = (rem == rem) ? t : (uint16_t)0;
    if (rem == rem) rem -= from_lp<BF16>(t);
  }
  bad |= !(fabsf(rem) <= 1e-6f * fabsf(b) + 1e-7f);
}

// One CTA per primitive: its image is put together in shared memory and written in 16-byte pieces.  Bound: memory (13.8 KB
// in, 8,000 bytes out at H = 32).  Two-byte stores straight to memory took 192 us for 20,000 primitives, this 103.
constexpr int kPackThreads = 128;
template <bool BF16, int H>
__global__ void __launch_bounds__(kPackThreads) k_pack_weights(
    const float* __restrict__ W1, const float* __restrict__ b1, const float* __restrict__ W2, const float* __restrict__ b2,
    const float* __restrict__ W3, const float* __restrict__ b3, int n, char* __restrict__ out, int32_t* __restrict__ status) {
  using N = Net<H>;
  static_assert(N::kWeightBytes % 16 == 0 && H * 72 % kPackThreads == 0 && H * H % kPackThreads == 0 && 4 * H % kPackThreads == 0, "whole rounds");
  __shared__ __align__(16) char img[N::kWeightBytes];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t p = blockIdx.x;
  uint16_t* w1 = reinterpret_cast<uint16_t*>(img + N::kOffW1);
  uint16_t* w2 = reinterpret_cast<uint16_t*>(img + N::kOffW2);
  uint16_t* w3 = reinterpret_cast<uint16_t*>(img + N::kOffW3);
  bool bad = false;
#pragma unroll 9
  for (int u = 0; u < H * 72 / kPackThreads; ++u) {
    const int i = u * kPackThreads + tid, h = i / 72, kk = enc_k_of_reference(i - h * 72);
    w1[(kk >> 3) * (H * 8) + h * 8 + (kk & 7)] = to_lp<BF16>(__ldg(W1 + p * (H * 72) + i), bad);
  }
#pragma unroll 8
  for (int u = 0; u < H * H / kPackThreads; ++u) {
    const int i = u * kPackThreads + tid, h = i / H, k = i % H;
    w2[(k >> 3) * (H * 8) + h * 8 + (k & 7)] = to_lp<BF16>(__ldg(W2 + p * (H * H) + i), bad);
  }
#pragma unroll
  for (int u = 0; u < kOut * H / kPackThreads; ++u) {
    const int i = u * kPackThreads + tid, h = i / H, k = i % H;
    w3[(k >> 3) * (kOut * 8) + h * 8 + (k & 7)] = to_lp<BF16>(__ldg(W3 + p * (kOut * H) + i), bad);
  }
  // the biases, a warp or two each
  for (int h = lane; h < H; h += 32) {
    if (warp == 0) {
      bias_terms<BF16>(__ldg(b1 + p * H + h), w1 + kBiasChunk * (H * 8) + h * 8, bad);
    } else if (warp == 1) {
      bias_terms<BF16>(__ldg(b2 + p * H + h), w2 + (H / 8) * (H * 8) + h * 8, bad);
    }
  }
  if (warp == 2 && lane < kOut) bias_terms<BF16>(__ldg(b3 + p * kOut + lane), w3 + (H / 8) * (kOut * 8) + lane * 8, bad);
  __syncthreads();
  uint4* dst = reinterpret_cast<uint4*>(out + p * N::kWeightBytes);
  for (int i = tid; i < N::kWeightBytes / 16; i += kPackThreads) dst[i] = reinterpret_cast<const uint4*>(img)[i];
  if (bad && status) atomicOr(status + MLPSP_ST_BITS, MLPSP_ST_NUMERIC);
}

template <bool KEEP, bool BF16, int H, bool TAB>
static int launch_one(const char* image, const mlpsp_scene* sc, const char* dir_table, const RecIn* rec_in, const int4* work,
                      const int32_t* counters, float4* rec_out, float4* rec_ext, int out_mode, int32_t* status, cudaStream_t st, int grid) {
  using N = Net<H>;
  static DeviceOnce attr_once;
  if (attr_once.first())
    MLPSP_CUDA_OK(cudaFuncSetAttribute(k_mlp_tc<KEEP, BF16, H, TAB>, cudaFuncAttributeMaxDynamicSharedMemorySize, N::kGroups * N::kGroupBytes));
  launch_chained(k_mlp_tc<KEEP, BF16, H, TAB>, dim3(grid), dim3(N::kThreads), N::kGroups * N::kGroupBytes, st, image, sc->freq, sc->att, dir_table,
                 reinterpret_cast<const float4*>(rec_in), work, counters, rec_out, rec_ext, out_mode, status);
  return MLPSP_OK;
}

template <bool BF16, int H>
static int launch_mini(const char* image, const mlpsp_scene* sc, const RecIn* rec_in, const int4* work_small,
                       const int32_t* counters, float4* rec_out, int out_mode, int32_t* status, cudaStream_t st, int grid) {
  using M = MiniNet<H>;
  static DeviceOnce attr_once;
  if (attr_once.first())
    MLPSP_CUDA_OK(cudaFuncSetAttribute(k_mlp_tc_mini<BF16, H>, cudaFuncAttributeMaxDynamicSharedMemorySize, M::kSmemBytes));
  launch_chained(k_mlp_tc_mini<BF16, H>, dim3(grid), dim3(kMiniRows), M::kSmemBytes, st, image, sc->freq, sc->att, reinterpret_cast<const float4*>(rec_in),
                                                                work_small, counters, rec_out, out_mode, status);
  return MLPSP_OK;
}

template <int H>
static int launch_tc(const mlpsp_scene* sc, const char* image, const char* dir_table, const RecIn* rec_in, const int4* work, const int4* work_small,
                     const int32_t* counters, float4* rec_out, float4* rec_ext, int out_mode, int32_t* status, cudaStream_t st,
                     bool bf16, int grid_cap) {
  const int sms = sm_count();
  const int grid = grid_cap > 0 ? std::min(sms, grid_cap) : sms;
  LaunchScope scope(kKMlp, (work_small && !rec_ext) ? 2 : 1, st);
  int rc;
  if (rec_ext) {
    if (H != 32) {
      set_error("record export needs hidden width 32 (32-bit ReLU masks)");
      return MLPSP_E_LIMIT;
    }
    rc = bf16 ? launch_one<true, true, 32, false>(image, sc, nullptr, rec_in, work, counters, rec_out, rec_ext, out_mode, status, st, grid)
              : launch_one<true, false, 32, false>(image, sc, nullptr, rec_in, work, counters, rec_out, rec_ext, out_mode, status, st, grid);
  } else if (dir_table) {
    rc = bf16 ? launch_one<false, true, H, true>(image, sc, dir_table, rec_in, work, counters, rec_out, rec_ext, out_mode, status, st, grid)
              : launch_one<false, false, H, true>(image, sc, dir_table, rec_in, work, counters, rec_out, rec_ext, out_mode, status, st, grid);
  } else {
    rc = bf16 ? launch_one<false, true, H, false>(image, sc, nullptr, rec_in, work, counters, rec_out, rec_ext, out_mode, status, st, grid)
              : launch_one<false, false, H, false>(image, sc, nullptr, rec_in, work, counters, rec_out, rec_ext, out_mode, status, st, grid);
  }
  if (rc) return rc;
  if (work_small && !rec_ext) {
    // the wave's small groups (at most 32 records) on their own kernel: one warp per item, twelve (seven) items per SM
    int grid_s = sms * MiniNet<H>::kCtas;
    if (grid_cap > 0) grid_s = std::min(grid_s, grid_cap);
    rc = bf16 ? launch_mini<true, H>(image, sc, rec_in, work_small, counters, rec_out, out_mode, status, st, grid_s)
              : launch_mini<false, H>(image, sc, rec_in, work_small, counters, rec_out, out_mode, status, st, grid_s);
    if (rc) return rc;
  }
  return cuda_check(cudaGetLastError(), "mlp_f16");
}

int launch_encode_directions(const mlpsp_scene* sc, const mlpsp_frame* fr, char* table, cudaStream_t st) {
  const int T = num_tiles(fr->width, fr->height, 8), ntx = (fr->width + 7) / 8;
  LaunchScope scope(kKMlp, 1, st);
  auto* kernel = fr->precision == MLPSP_PRECISION_BF16 ? k_encode_directions<true> : k_encode_directions<false>;
  return cuda_check(launch_chained(kernel, dim3((unsigned)std::min<int64_t>(((int64_t)T * 64 + 255) / 256, (int64_t)sm_count() * 64)), dim3(256), 0, st,
                                   fr->rays_d, fr->width, fr->height, ntx, T, sc->freq, sc->att, table),
                    "encode_directions");
}

int launch_mlp_f16(const mlpsp_scene* sc, const RecIn* rec_in, const int4* work,
                   const int32_t* counters, float4* rec_out, float4* rec_ext, int out_mode, int32_t* status,
                   cudaStream_t st, bool bf16, int grid_cap, const int4* work_small, const char* dir_table) {
  MLPSP_REQUIRE((sc->hidden == 32 || sc->hidden == 64) && sc->num_freq == 6, MLPSP_E_LIMIT,
                "the tensor-core evaluator is built for 72->H->H->4 networks with H = 32 or 64 (6 frequencies)");
  const char* image = (const char*)(bf16 ? sc->wbf16 : sc->w16);
  MLPSP_REQUIRE(image && sc->freq && sc->att, MLPSP_E_ARG, "%s evaluator needs the packed weight image",
                bf16 ? "bf16" : "fp16");
  MLPSP_REQUIRE((reinterpret_cast<uintptr_t>(image) & 15) == 0, MLPSP_E_ARG, "the packed weight image must be 16-byte aligned");
  if (sc->hidden == 64)
    return launch_tc<64>(sc, image, dir_table, rec_in, work, work_small, counters, rec_out, rec_ext, out_mode, status, st, bf16, grid_cap);
  return launch_tc<32>(sc, image, dir_table, rec_in, work, work_small, counters, rec_out, rec_ext, out_mode, status, st, bf16, grid_cap);
}

}  // namespace mlpsp

using namespace mlpsp;

extern "C" int64_t mlpsp_packed_weight_bytes(int32_t hidden, int32_t num_freq) {
  if (num_freq != 6) return 0;
  return hidden == 32 ? Net<32>::kWeightBytes : (hidden == 64 ? Net<64>::kWeightBytes : 0);
}

static int pack_weights(const mlpsp_scene* sc, void* out, int32_t* status, void* stream, bool bf16, const char* who) {
  MLPSP_REQUIRE(sc && out, MLPSP_E_ARG, "%s: null pointer", who);
  MLPSP_REQUIRE((sc->hidden == 32 || sc->hidden == 64) && sc->num_freq == 6, MLPSP_E_LIMIT,
                "%s: only 72->H->H->4 networks with H = 32 or 64 have a packed image", who);
  MLPSP_REQUIRE(sc->W1 && sc->b1 && sc->W2 && sc->b2 && sc->W3 && sc->b3, MLPSP_E_ARG, "%s: FP32 weights missing", who);
  if (sc->n == 0) return MLPSP_OK;
  cudaStream_t st = (cudaStream_t)stream;
  LaunchScope scope(kKMisc, 1, st);
#define MLPSP_PACK(BF, HH)                                                                                         \
  k_pack_weights<BF, HH><<<sc->n, kPackThreads, 0, st>>>(sc->W1, sc->b1, sc->W2, sc->b2, sc->W3, sc->b3, sc->n, (char*)out, status)
  if (sc->hidden == 64) { if (bf16) MLPSP_PACK(true, 64); else MLPSP_PACK(false, 64); }
  else { if (bf16) MLPSP_PACK(true, 32); else MLPSP_PACK(false, 32); }
#undef MLPSP_PACK
  return cuda_check(cudaGetLastError(), who);
}

extern "C" int mlpsp_pack_weights_f16(const mlpsp_scene* sc, void* w16_out, int32_t* status, void* stream) {
  return pack_weights(sc, w16_out, status, stream, false, "mlpsp_pack_weights_f16");
}

extern "C" int mlpsp_pack_weights_bf16(const mlpsp_scene* sc, void* wbf16_out, int32_t* status, void* stream) {
  return pack_weights(sc, wbf16_out, status, stream, true, "mlpsp_pack_weights_bf16");
}
