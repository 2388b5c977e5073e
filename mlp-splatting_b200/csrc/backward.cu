// The backward side of the record path: reverse compositing over saved records and the per-primitive
// weight gradients of the grouped MLP.
//
// mlpsp_records_reverse computes what primitive_records_reverse_kernel computes (scannet/cuda/primitive_records.cuh:3-49):
// the image adjoints become the adjoint of every record's four pre-activation MLP outputs plus position /
// log-scale / quaternion gradients accumulated per primitive; see "records reverse" below for how the work is split.
//
// mlpsp_grouped_weight_gradients computes what scannet/primitive_gemm.py:101-279 computes with Triton
// (grouped_weight_gradients, FP32 operand mode) and scannet/primitive_csr.py:33-58 states in PyTorch:
// per primitive, with its records' encoded inputs E, saved ReLU masks and output adjoints D3,
//   D2 = (D3 W3) * mask2,  D1 = (D2 W2) * mask1,
//   dW3 = D3^T H2, db3 = sum D3, dW2 = D2^T H1, db2 = sum D2, dW1 = D1^T E, db1 = sum D1.
// A segment (at most segment_size records of one primitive) is summed by one CTA.  A primitive with one segment, the
// usual case, gets its gradients straight from that CTA; the partial 3,524-vectors of the others are added in segment
// order by a second kernel, so the result does not depend on scheduling.  mlpsp_weight_gradients plans the segments from
// the offsets, mlpsp_grouped_weight_gradients takes the caller's.
#include "frame.cuh"
#include "vjp.cuh"

namespace mlpsp {

// ------------------------------------------------------------------ quaternion helpers ----
// rotate v by the unit quaternion (w, x, y, z): v + w t + u x t with t = 2 (u x v), u = (x, y, z)
__device__ __forceinline__ V3 rot_quat(float qw, float qx, float qy, float qz, V3 v) {
  const float tx = 2.f * (qy * v.z - qz * v.y), ty = 2.f * (qz * v.x - qx * v.z), tz = 2.f * (qx * v.y - qy * v.x);
  V3 r;
  r.x = v.x + qw * tx + (qy * tz - qz * ty);
  r.y = v.y + qw * ty + (qz * tx - qx * tz);
  r.z = v.z + qw * tz + (qx * ty - qy * tx);
  return r;
}

// Chain rule from the adjoint G of the rotation matrix R(q) (row-major 3x3) to the quaternion
// (np_tile_kernels.cu:439-480).  With R = I + 2 w [u]x + 2 [u]x^2 the partial derivatives are
//   dR/dw = 2 [u]x,   dR/du_k = 2 w [e_k]x + 2 ([e_k]x [u]x + [u]x [e_k]x).
__device__ __forceinline__ void quat_adjoint(float w, float x, float y, float z, const float (&G)[9], float (&gq)[4]) {
  const float u[3] = {x, y, z};
  // [a]x as a row-major matrix
  auto cross_m = [](const float a[3], float M[9]) {
    M[0] = 0.f;   M[1] = -a[2]; M[2] = a[1];
    M[3] = a[2];  M[4] = 0.f;   M[5] = -a[0];
    M[6] = -a[1]; M[7] = a[0];  M[8] = 0.f;
  };
  float U[9];
  cross_m(u, U);
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < 9; ++i) acc += G[i] * 2.f * U[i];
  gq[0] = acc;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float e[3] = {0.f, 0.f, 0.f};
    e[k] = 1.f;
    float E[9];
    cross_m(e, E);
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        float eu = 0.f, ue = 0.f;
#pragma unroll
        for (int m = 0; m < 3; ++m) { eu += E[r * 3 + m] * U[m * 3 + c]; ue += U[r * 3 + m] * E[m * 3 + c]; }
        s += G[r * 3 + c] * (2.f * w * E[r * 3 + c] + 2.f * (eu + ue));
      }
    gq[1 + k] = s;
  }
}

// ------------------------------------------------------------------- records reverse ----
// The reference walks a pixel's records backwards in one thread and issues ten (warp-aggregated) global atomics per
// record from inside that walk (primitive_records.cuh:3-49).  Here the walk is reduced to what is sequential -- the
// recurrence of the colour that lies behind a record -- and everything else runs record-parallel afterwards:
//   k_reverse_check     the argument checks of the caller (offsets, ids) as one status word;
//   k_reverse_pixels    thread = pixel: the recurrence, the four adjoints of every record and
//                       k = g_sigma * sigma_raw * decay, the weight of the record's geometry terms;
//   k_reverse_geometry  decay = exp(-1/2 q^T M q) with q = R^T d, M = diag(exp(-2 ls)): the position, log-scale and
//                       quaternion gradients of a primitive are linear in the nine sums of k q and k q q^T over its
//                       records, so only those are accumulated, a chunk of records at a time (records that follow one
//                       another belong to neighbouring pixels, which mostly see the same primitives);
//   k_reverse_finish    thread = primitive: the gradients from the nine sums.
constexpr int kRevAcc = 12;          // floats per primitive: k q (3), k q q^T (6), padding to three 16-byte reductions

__global__ void __launch_bounds__(256) k_reverse_check(const int32_t* __restrict__ ids, int64_t total, int n,
                                                       const int64_t* __restrict__ offsets, int64_t pixels,
                                                       int32_t* __restrict__ bad, volatile int32_t* bad_host) {
  chain_wait();
  chain_release();
  int b = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x, t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t i = t; i < total; i += stride) b |= (uint32_t)__ldg(ids + i) >= (uint32_t)n ? MLPSP_REVERSE_BAD_IDS : 0;
  for (int64_t i = t; i < pixels; i += stride) b |= __ldg(offsets + i + 1) < __ldg(offsets + i) ? MLPSP_REVERSE_BAD_OFFSETS : 0;
  if (t == 0 && (offsets[0] != 0 || offsets[pixels] != total)) b |= MLPSP_REVERSE_BAD_OFFSETS;
  if (b) { atomicOr(bad, b); if (bad_host) atomicOr_system(const_cast<int32_t*>(bad_host), b); }
}

// A block's pixels own one run of records.  It is brought into shared memory in whole lines, from its end on, kRevStage
// records at a time; a thread walks those of its pixel among them, the outputs take the records' places and leave the same
// way.  Bound: memory, 52 bytes per record; 4.3 M records in 480,000 pixels read and written by the walk itself: 167 us,
// staged: 74.
constexpr int kRevPixels = 128, kRevStage = 1024;
__global__ void __launch_bounds__(kRevPixels) k_reverse_pixels(const int64_t* __restrict__ offsets, const float* __restrict__ raw,
                                 const float* __restrict__ grgb, const float* __restrict__ gt, int64_t pixels,
                                 float* __restrict__ d4, float* __restrict__ kw, const int32_t* __restrict__ bad) {
  chain_wait();
  chain_release();
  __shared__ __align__(16) float4 s_raw[2 * kRevStage];
  if (*bad) return;
  const int tid = threadIdx.x;
  const int64_t p0 = (int64_t)blockIdx.x * kRevPixels, p1 = min(p0 + kRevPixels, pixels), pix = p0 + tid;
  const int64_t base = offsets[p0], end = offsets[p1];
  const float4* raw4 = reinterpret_cast<const float4*>(raw);
  float gr = 0.f, gg = 0.f, gb = 0.f, behind = 0.f;
  int64_t first = 0, last = -1;
  if (pix < pixels) {
    gr = grgb[pix * 3]; gg = grgb[pix * 3 + 1]; gb = grgb[pix * 3 + 2];
    behind = gt[pix];   // adjoint of the transmittance that reaches whatever lies behind the current record
    first = offsets[pix];
    last = offsets[pix + 1] - 1;
  }
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_raw);
  for (int64_t hi = end; hi > base;) {
    const int64_t lo = max(base, hi - kRevStage);
    const int run = (int)(hi - lo);
    for (int i = tid; i < 2 * run; i += kRevPixels)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * (uint32_t)i), "l"(raw4 + 2 * lo + i) : "memory");
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int q = (int)(min(last, hi - 1) - lo), q0 = (int)max(first - lo, (int64_t)0); q >= q0; --q) {
      const float4 a = s_raw[2 * q], c = s_raw[2 * q + 1];  // R, G, B, sigma_raw; trans before, alpha, decay, sigma logit
      const float colour = gr * a.x + gg * a.y + gb * a.z;
      const float g_alpha = c.x * (colour - behind);
      behind = behind * (1.f - c.y) + colour * c.y;
      const float g_sigma = g_alpha * __expf(-a.w * c.z);   // d alpha / d (sigma_raw * decay) = 1 - alpha
      const float w = c.x * c.y, parked = g_sigma * c.z;
      s_raw[2 * q] = make_float4(gr * w * a.x * (1.f - a.x), gg * w * a.y * (1.f - a.y), gb * w * a.z * (1.f - a.z),
                                 parked * sigmoid_fast(c.w));                               // softplus' = sigmoid
      s_raw[2 * q + 1].x = parked * a.w;                    // g_decay * decay
    }
    __syncthreads();
    for (int i = tid; i < run; i += kRevPixels) {
      *reinterpret_cast<float4*>(d4 + (lo + i) * 4) = s_raw[2 * i];
      kw[lo + i] = s_raw[2 * i + 1].x;
    }
    hi = lo;
    if (hi > base) __syncthreads();
  }
}

constexpr int kRevThreads = 256, kRevPer = 8;
constexpr int kRevChunk = kRevThreads * kRevPer;      // records per CTA
constexpr int kRevTable = 1024;      // rows of the chunk's table of primitives (a power of two)
constexpr int kRevProbe = 16;        // probes before a record goes to global memory directly
constexpr int kRevPiece = 16;        // records that one thread adds up
constexpr int kRevUnits = kRevTable + kRevChunk / kRevPiece;
constexpr int kRevSmem = (kRevChunk + 3 * kRevThreads) * 16;
static_assert(kRevChunk <= 2048 && kRevPiece <= 32 && kRevTable <= 1024, "packing of a unit: start 11 bits, count - 1 5 bits, row 10 bits");

__device__ __forceinline__ void red_add4(float* dst, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// A chunk's records are ordered by primitive in shared memory -- a hash table of the primitives that counts its rows, a
// prefix over the rows -- and a thread adds up to kRevPiece records of one primitive in registers; the sums leave three
// 16-byte reductions at a time, a primitive's by neighbouring lanes.  Bound: the reductions in L2 and the record's 44 bytes.
// With nine floating-point additions per record in shared memory (each a loop of compare-and-swap, on rows that
// neighbouring pixels share) 4.3 M records took 246 us and 0.7 M 141; this takes 71 and about 40.
__device__ __forceinline__ void reverse_terms(const float4 qt, float dx, float dy, float dz, float k, float (&v)[9]) {
  const V3 q = rot_conj_fast(qt.x, qt.y, qt.z, qt.w, V3{dx, dy, dz});
  const float kx = k * q.x, ky = k * q.y, kz = k * q.z;
  v[0] += kx; v[1] += ky; v[2] += kz;
  v[3] += kx * q.x; v[4] += ky * q.y; v[5] += kz * q.z;
  v[6] += kx * q.y; v[7] += kx * q.z; v[8] += ky * q.z;
}

__global__ void __launch_bounds__(kRevThreads, 3) k_reverse_geometry(
    const int32_t* __restrict__ ids, const float* __restrict__ x6, const float* __restrict__ kw,
    const float* __restrict__ quats, int64_t total, float* __restrict__ acc, const int32_t* __restrict__ bad) {
  chain_wait();
  chain_release();
  extern __shared__ __align__(16) float4 s_rec[];      // [kRevChunk] offset and weight, by primitive; then the sums of a round
  __shared__ int s_key[kRevTable], s_cnt[kRevTable];   // primitive, records (later: first record)
  __shared__ uint32_t s_unit[kRevUnits];
  __shared__ int warp_sums[32];
  float4 (*s_sum)[3] = reinterpret_cast<float4(*)[3]>(s_rec + kRevChunk);
  if (*bad) return;
  const int tid = threadIdx.x;
  for (int i = tid; i < kRevTable; i += kRevThreads) { s_key[i] = -1; s_cnt[i] = 0; }
  const int64_t r0 = (int64_t)blockIdx.x * kRevChunk;
  float4 rec[kRevPer];
  int place[kRevPer];              // row << 16 | rank in it; -1: none
#pragma unroll
  for (int u = 0; u < kRevPer; ++u) {
    const int64_t r = r0 + u * kRevThreads + tid;
    place[u] = r < total ? ids[r] : -1;
    rec[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < total) rec[u] = make_float4(x6[r * 6 + 3], x6[r * 6 + 4], x6[r * 6 + 5], kw[r]);      // centre - foot point
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kRevPer; ++u) {
    const int p = place[u];
    if (p < 0) continue;
    // the primitive's row of the table: linear probing from a multiplicative hash
    int row = (int)(((uint32_t)p * 2654435761u) >> 22) & (kRevTable - 1);
    bool placed = false;
    for (int probe = 0; probe < kRevProbe && !placed; ++probe) {
      int seen = s_key[row];
      if (seen == -1) seen = atomicCAS(&s_key[row], -1, p);
      if (seen == -1 || seen == p) placed = true;
      else row = (row + 1) & (kRevTable - 1);
    }
    if (placed) {
      place[u] = (row << 16) | atomicAdd(&s_cnt[row], 1);
    } else {
      place[u] = -1;
      float v[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      reverse_terms(__ldg(reinterpret_cast<const float4*>(quats) + p), rec[u].x, rec[u].y, rec[u].z, rec[u].w, v);
      float* dst = acc + (size_t)p * kRevAcc;
      red_add4(dst, v[0], v[1], v[2], v[3]);
      red_add4(dst + 4, v[4], v[5], v[6], v[7]);
      red_add4(dst + 8, v[8], 0.f, 0.f, 0.f);
    }
  }
  __syncthreads();
  // rows -> first records and pieces (a thread has kRevTable / kRevThreads rows in order)
  constexpr int kRows = kRevTable / kRevThreads;
  int cnt[kRows], mine = 0;
#pragma unroll
  for (int j = 0; j < kRows; ++j) {
    cnt[j] = s_cnt[tid * kRows + j];
    mine += (cnt[j] << 16) + (cnt[j] + kRevPiece - 1) / kRevPiece;
  }
  int all;
  const int before = block_exclusive_scan(mine, warp_sums, all);
  int start = before >> 16, unit = before & 0xffff;
  const int units = all & 0xffff;
#pragma unroll
  for (int j = 0; j < kRows; ++j) {
    s_cnt[tid * kRows + j] = start;
    for (int c = 0; c < cnt[j]; c += kRevPiece)
      s_unit[unit++] = (uint32_t)(start + c) | ((uint32_t)(min(kRevPiece, cnt[j] - c) - 1) << 11) | ((uint32_t)(tid * kRows + j) << 16);
    start += cnt[j];
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kRevPer; ++u)
    if (place[u] >= 0) s_rec[s_cnt[place[u] >> 16] + (place[u] & 0xffff)] = rec[u];
  __syncthreads();
  for (int b = 0; b < units; b += kRevThreads) {
    if (b + tid < units) {
      const uint32_t w = s_unit[b + tid];
      const float4 qt = __ldg(reinterpret_cast<const float4*>(quats) + s_key[w >> 16]);
      float v[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      const int from = w & 2047, to = from + 1 + ((w >> 11) & 31);
      for (int i = from; i < to; ++i) {
        const float4 e = s_rec[i];
        reverse_terms(qt, e.x, e.y, e.z, e.w, v);
      }
      s_sum[tid][0] = make_float4(v[0], v[1], v[2], v[3]);
      s_sum[tid][1] = make_float4(v[4], v[5], v[6], v[7]);
      s_sum[tid][2] = make_float4(v[8], 0.f, 0.f, 0.f);
    }
    __syncthreads();
    const int pieces = 3 * min(kRevThreads, units - b);
    for (int i = tid; i < pieces; i += kRevThreads) {
      const float4 e = s_sum[i / 3][i % 3];
      red_add4(acc + (size_t)s_key[s_unit[b + i / 3] >> 16] * kRevAcc + (i % 3) * 4, e.x, e.y, e.z, e.w);
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(128) k_reverse_finish(const float* __restrict__ acc, const float* __restrict__ logs,
                                                        const float* __restrict__ quats, int n, float* __restrict__ gp,
                                                        float* __restrict__ gs, float* __restrict__ gq, int gq_vec) {
  chain_wait();
  chain_release();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const float4 a = *reinterpret_cast<const float4*>(acc + (size_t)p * kRevAcc);
  const float4 b = *reinterpret_cast<const float4*>(acc + (size_t)p * kRevAcc + 4);
  const float syz = acc[(size_t)p * kRevAcc + 8];
  const float S[9] = {a.w, b.z, b.w, b.z, b.x, syz, b.w, syz, b.y};        // sum of k q q^T
  const float4 qt = __ldg(reinterpret_cast<const float4*>(quats) + p);
  const float m[3] = {__expf(-2.f * logs[(size_t)p * 3]), __expf(-2.f * logs[(size_t)p * 3 + 1]), __expf(-2.f * logs[(size_t)p * 3 + 2])};
  // adjoint of q is -k M q; of d (hence of the centre) R times that; of R, with q = R^T d, d (-k M q)^T
  const V3 gd = rot_quat(qt.x, qt.y, qt.z, qt.w, V3{-m[0] * a.x, -m[1] * a.y, -m[2] * a.z});
  gp[(size_t)p * 3] = gd.x; gp[(size_t)p * 3 + 1] = gd.y; gp[(size_t)p * 3 + 2] = gd.z;
  gs[(size_t)p * 3] = m[0] * S[0]; gs[(size_t)p * 3 + 1] = m[1] * S[4]; gs[(size_t)p * 3 + 2] = m[2] * S[8];
  float Gm[9];
#pragma unroll
  for (int j = 0; j < 3; ++j) {      // column j of sum d gl^T = R (-m_j S_.j)
    const V3 c = rot_quat(qt.x, qt.y, qt.z, qt.w, V3{-m[j] * S[j], -m[j] * S[3 + j], -m[j] * S[6 + j]});
    Gm[j] = c.x; Gm[3 + j] = c.y; Gm[6 + j] = c.z;
  }
  float gquat[4];
  quat_adjoint(qt.x, qt.y, qt.z, qt.w, Gm, gquat);
  if (gq_vec) {                      // the caller's rows are 16-byte aligned
    *reinterpret_cast<float4*>(gq + (size_t)p * 4) = make_float4(gquat[0], gquat[1], gquat[2], gquat[3]);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) gq[(size_t)p * 4 + i] = gquat[i];
  }
}

// --------------------------------------------------------- grouped weight gradients ----
// Segments of the launch, planned on the device (no count travels to the host): the order of the items does not matter,
// a primitive of several segments owns consecutive partial rows and an entry of the multi list, a primitive without
// records (its gradients are zero) an entry at the other end of that list.
// The lists are sized from the record count, the segments counted from the offsets: offsets that descend or leave
// [0, records] set a flag bit, on which the kernels behind this one do nothing, and no item is written past the list.
// (With every range ascending inside [0, records] the counts add up to no more than the records, and the lists hold them.)
__global__ void __launch_bounds__(256) k_vjp_plan(const int64_t* __restrict__ offsets, int n, int64_t records, int segment_size,
                                                  VjpItem* __restrict__ items, int64_t max_items, VjpItem* __restrict__ multi,
                                                  int32_t* __restrict__ counters) {
  chain_wait();
  chain_release();
  __shared__ int warp_sums[32];
  __shared__ int base[5];
  const int p = blockIdx.x * 256 + threadIdx.x;
  int64_t start = 0, count = 0;
  if (p < n) {
    start = offsets[p];
    const int64_t end = offsets[p + 1];
    if (start < 0 || end < start || end > records) atomicOr(counters + kVpFlag, kVpBadPlan);
    else count = end - start;
  }
  const int segs = count > 0 ? (int)((count + segment_size - 1) / segment_size) : 0;
  const int rows = segs > 1 ? segs : 0, listed = segs > 1, empty = p < n && segs == 0;
  const int full = (int)(count / segment_size), part = segs - full;      // full segments, and a shorter last one
  int ts, tp, tr, tm, te;
  const int es = block_exclusive_scan(full, warp_sums, ts);
  const int ep = block_exclusive_scan(part, warp_sums, tp);
  const int er = block_exclusive_scan(rows, warp_sums, tr);
  const int em = block_exclusive_scan(listed, warp_sums, tm);
  const int ee = block_exclusive_scan(empty, warp_sums, te);
  if (threadIdx.x == 0) {
    base[0] = ts ? atomicAdd(counters + kVpItems, ts) : 0;
    base[1] = tr ? atomicAdd(counters + kVpRows, tr) : 0;
    base[2] = tm ? atomicAdd(counters + kVpMulti, tm) : 0;
    base[3] = te ? atomicAdd(counters + kVpEmpty, te) : 0;
    base[4] = tp ? atomicAdd(counters + kVpParts, tp) : 0;
  }
  __syncthreads();
  for (int g = 0; g < segs; ++g) {
    VjpItem it = {};
    it.start = start + (int64_t)g * segment_size;
    it.rows = (int)min((int64_t)segment_size, count - (int64_t)g * segment_size);
    it.prim = p;
    it.dest = segs > 1 ? base[1] + er + g : -1;
    const uint32_t at = (uint32_t)(g < full ? base[0] + es + g : base[4] + ep);
    if (at < max_items) items[g < full ? at : max_items - 1 - at] = it;
  }
  if (listed) {
    VjpItem it = {};
    it.start = base[1] + er;
    it.rows = rows;
    it.prim = p;
    multi[base[2] + em] = it;
  }
  if (empty) multi[n - 1 - (base[3] + ee)].prim = p;
}

// The same lists from a layout that the caller has prepared: segment g is item g and, unless it is its primitive's only
// one, partial row g.  A segment outside its primitive's records or list refuses the plan.
__global__ void __launch_bounds__(256) k_vjp_plan_layout(const int64_t* __restrict__ offsets, int n, int segment_size,
                                                         const int64_t* __restrict__ seg_prim, const int64_t* __restrict__ seg_start,
                                                         const int64_t* __restrict__ seg_offsets, int G, VjpItem* __restrict__ items,
                                                         VjpItem* __restrict__ multi, int32_t* __restrict__ counters) {
  chain_wait();
  chain_release();
  __shared__ int warp_sums[32];
  __shared__ int base[2];
  const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
  bool ok = true;
  if (t < G) {
    const int64_t p = seg_prim[t], start = seg_start[t];
    ok = p >= 0 && p < n;
    if (ok) {
      const int64_t begin = offsets[p], end = offsets[p + 1], g0 = seg_offsets[p], g1 = seg_offsets[p + 1];
      ok = begin >= 0 && start >= begin && start < end && g0 <= t && t < g1;
      VjpItem it = {};
      it.start = start;
      it.rows = (int)min((int64_t)segment_size, end - start);
      it.prim = (int)p;
      it.dest = g1 - g0 > 1 ? (int)t : -1;
      items[t] = it;
    }
  }
  VjpItem it = {};
  it.prim = (int)t;
  int listed = 0, empty = 0;
  if (t < n) {
    const int64_t g0 = seg_offsets[t], g1 = seg_offsets[t + 1];
    if (g0 < 0 || g1 < g0 || g1 > G) {
      ok = false;
    } else {
      it.start = g0;
      it.rows = (int)(g1 - g0);
      listed = it.rows > 1;
      empty = it.rows == 0;
    }
  }
  int tm, te;
  const int em = block_exclusive_scan(listed, warp_sums, tm), ee = block_exclusive_scan(empty, warp_sums, te);
  if (threadIdx.x == 0) {
    base[0] = tm ? atomicAdd(counters + kVpMulti, tm) : 0;
    base[1] = te ? atomicAdd(counters + kVpEmpty, te) : 0;
    if (blockIdx.x == 0) counters[kVpItems] = G;
  }
  __syncthreads();
  if (listed) multi[base[0] + em] = it;
  if (empty) multi[n - 1 - (base[1] + ee)] = it;
  if (!ok) atomicOr(counters + kVpFlag, kVpBadPlan);
}

// IEEE FP32 on the CUDA cores, sums in record order over each half of the blocks.  A CTA of 128 threads takes 64 records at a
// time; everything per record lies transposed in shared memory ([quantity][record], rows of 68 floats), so that the record-major
// products (layers, adjoints) give a thread a tile of four records x four units and the contractions over the records (the
// gradients) 4 x 9 + 4 x 4 + 2 sums in registers over 32 of the records, both fed by 16-byte reads.  Bound: what goes from shared
// memory into registers, 128 bytes a cycle whether lanes read the same bytes or not (a tile of a x b costs a + b floats for a b
// multiply-adds), then issue: load unit 74 %, issue slots 65, multiply-adds 49.  With 2 x 9 + 2 x 4 + 1 sums over all 64 records
// per thread, hidden rows that share banks, weights loaded one by one and all of a thread's sincosf in a row (a third of the
// instruction cache), 5.5 M records of 15,000 primitives took 3,930 us, so 3,090; 0.8 M of 9,800 887 and 718.  A warp per
// segment with tiles of 4 x 8 (38 KB, six warps per SM) 3,880 and 957, of 8 x 8 (52 KB, four) 4,920 and 1,160: too few warps.
constexpr int kGfRec = 64, kGfThreads = 128, kGfRow = kGfRec + 4, kGfCtas = 3;
constexpr int kGfE = 0, kGfH1 = kGfE + kGIN * kGfRow, kGfH2 = kGfH1 + kGH * kGfRow, kGfD1 = kGfH2 + kGH * kGfRow,
              kGfD2 = kGfD1 + kGH * kGfRow, kGfD3 = kGfD2 + kGH * kGfRow, kGfMask = kGfD3 + 4 * kGfRow,
              kGfW1T = kGfMask + 2 * kGfRec, kGfW2T = kGfW1T + kGIN * kGH, kGfW2 = kGfW2T + kGH * kGH, kGfW2Row = kGH + 4,
              kGfW3 = kGfW2 + kGH * kGfW2Row, kGfB = kGfW3 + 4 * kGH, kGfFloats = kGfB + 2 * kGH;
constexpr int kGradSmem = kGfFloats * 4;
static_assert(kGfCtas * (kGradSmem + 1024) <= 228 * 1024, "resident CTAs");

// Where the records r .. r + 3 lie in a row of a hidden tile: every eight rows the records begin four places further on, so that
// neither the eight rows that a tile of units is written to nor the eight that a gradient is read from share banks.
__device__ __forceinline__ int gf_turn(int r, int row) { return (r + 4 * (row >> 3)) & (kGfRec - 1); }
__device__ __forceinline__ void fma4(float4& a, float s, const float4 v) {
  a.x = fmaf(s, v.x, a.x); a.y = fmaf(s, v.y, a.y); a.z = fmaf(s, v.z, a.z); a.w = fmaf(s, v.w, a.w);
}
// acc + the products of four consecutive records, in record order
__device__ __forceinline__ float dot4(float acc, const float4 a, const float4 b) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}

__global__ void __launch_bounds__(kGfThreads, kGfCtas) k_grouped_vjp(
    const float* __restrict__ x6, const float* __restrict__ d4, const int32_t* __restrict__ masks,
    const VjpItem* __restrict__ items, int64_t max_items, int32_t* __restrict__ counters, const float* __restrict__ freq,
    const float* __restrict__ att, const float* __restrict__ W1, const float* __restrict__ b1, const float* __restrict__ W2,
    const float* __restrict__ b2, const float* __restrict__ W3, int vec, float scale, VjpOut out, float* __restrict__ partial) {
  chain_wait();
  chain_release();
  extern __shared__ __align__(16) float sm[];
  const VjpList list(items, max_items, counters);
  const int tid = threadIdx.x;
  const int hg = tid & 7, rg = tid >> 3;         // units 4 hg .. + 3 of records 4 rg .. + 3
  // gradients: rows 4 gq .. + 3, inputs hg + 8 i, over the records of one half of a block
  const int half = tid >> 6, gq = (tid >> 3) & 7, th = tid & 63;
  const float inv = 1.f / scale;
  bool bad = false;
  uint32_t* sMask = reinterpret_cast<uint32_t*>(sm + kGfMask);
  float fr[6], at[6];
#pragma unroll
  for (int f = 0; f < 6; ++f) { fr[f] = __ldg(freq + f); at[f] = __ldg(att + f); }
  __shared__ int s_next;
  for (int idx = blockIdx.x; idx < list.total; idx = s_next) {   // (read behind the barriers of the item's blocks)
    const VjpItem it = list.at(idx);
    const size_t p = (size_t)it.prim;
    __syncthreads();                             // the previous item's last block has been consumed
    if (tid == 0) s_next = (int)gridDim.x + atomicAdd(counters + kVpNext, 1);
    // lane = row of W1 and W2, four consecutive inputs a time; the transposed stores are conflict-free (inputs one by one cost the
    // load unit 32 cycles each)
    auto row4 = [&](const float* w) {
      return vec ? __ldg(reinterpret_cast<const float4*>(w)) : make_float4(__ldg(w), __ldg(w + 1), __ldg(w + 2), __ldg(w + 3));
    };
    const int wr = tid & 31;
    auto put_t = [&](int off, int k, const float4& v) {
      sm[off + k * kGH + wr] = v.x; sm[off + (k + 1) * kGH + wr] = v.y; sm[off + (k + 2) * kGH + wr] = v.z; sm[off + (k + 3) * kGH + wr] = v.w;
    };
    float4 w1v[5], w2v[2];
#pragma unroll
    for (int u = 0; u < 5; ++u) {
      const int k = (u * 4 + (tid >> 5)) * 4;
      if (u < 4 || k < kGIN) w1v[u] = row4(W1 + p * (kGH * kGIN) + wr * kGIN + k);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) w2v[u] = row4(W2 + p * (kGH * kGH) + wr * kGH + (u * 4 + (tid >> 5)) * 4);
#pragma unroll
    for (int u = 0; u < 5; ++u) {
      const int k = (u * 4 + (tid >> 5)) * 4;
      if (u < 4 || k < kGIN) put_t(kGfW1T, k, w1v[u]);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int k = (u * 4 + (tid >> 5)) * 4;
      put_t(kGfW2T, k, w2v[u]);
      *reinterpret_cast<float4*>(sm + kGfW2 + wr * kGfW2Row + k) = w2v[u];
    }
    sm[kGfW3 + tid] = __ldg(W3 + p * (4 * kGH) + tid);
    if (tid < 2 * kGH) sm[kGfB + tid] = tid < kGH ? __ldg(b1 + p * kGH + tid) : __ldg(b2 + p * kGH + tid - kGH);
    float g1[4][9], g2[4][4], g3[2] = {0.f, 0.f}, gb = 0.f, gb3 = 0.f;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
#pragma unroll
      for (int i = 0; i < 9; ++i) g1[a][i] = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) g2[a][i] = 0.f;
    }
    for (int sub = 0; sub < it.rows; sub += kGfRec) {
      const int cnt = min(kGfRec, it.rows - sub);
      if (sub > 0) __syncthreads();              // the previous block's rows have been consumed
      {
        // encoding as scannet/cumodel.py:183-195: index c*F + f holds sin, + 36 holds cos; a thread takes three coordinates
        const int rec = tid & (kGfRec - 1), part = tid >> 6;
        const bool valid = rec < cnt;
        const int64_t r = it.start + sub + rec;
        float xs[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) xs[c] = valid ? __ldg(x6 + r * 6 + part * 3 + c) : 0.f;
#pragma unroll 1
        for (int c = 0; c < 3; ++c) {             // (a loop: eighteen sincosf in a row take a third of the instruction cache)
          const int cc = part * 3 + c;
          const float v = c == 0 ? xs[0] : (c == 1 ? xs[1] : xs[2]);
#pragma unroll
          for (int f = 0; f < 6; ++f) {
            float sn, cs;
            sincosf(v * fr[f] * at[f], &sn, &cs);
            sm[kGfE + (cc * 6 + f) * kGfRow + rec] = valid ? sn : 0.f;
            sm[kGfE + (36 + cc * 6 + f) * kGfRow + rec] = valid ? cs : 0.f;
          }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
          sm[kGfD3 + (part * 2 + c) * kGfRow + rec] = valid ? __ldg(d4 + r * 4 + part * 2 + c) * scale : 0.f;
        if (masks) sMask[part * kGfRec + rec] = valid ? (uint32_t)__ldg(masks + r * 2 + part) : 0u;
      }
      __syncthreads();
      const int r4 = rg * 4, h4 = hg * 4;
      uint32_t m1[4], m2[4];
      if (masks) {
#pragma unroll
        for (int j = 0; j < 4; ++j) { m1[j] = sMask[r4 + j] >> h4; m2[j] = sMask[kGfRec + r4 + j] >> h4; }
      }
      // a tile acc[u] = (four records) of unit h4 + u; gate: the records' mask bits of that unit
      float4 acc[4];
      auto product8 = [&](int x_off, int K, int w_off, int w_row, int r) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const float4 x = *reinterpret_cast<const float4*>(sm + x_off + k * kGfRow + r);
          const float4 w = *reinterpret_cast<const float4*>(sm + w_off + k * w_row + h4);
          fma4(acc[0], w.x, x); fma4(acc[1], w.y, x); fma4(acc[2], w.z, x); fma4(acc[3], w.w, x);
        }
      };
      auto product = [&](int x_off, int K, int w_off, int w_row, bool turned) {
#pragma unroll 1
        for (int k = 0; k < K; k += 8)
          product8(x_off + k * kGfRow, 8, w_off + k * w_row, w_row, turned ? gf_turn(r4, k) : r4);
      };
      auto hidden = [&](int dst, uint32_t (&m)[4]) {
        if (!masks) { m[0] = m[1] = m[2] = m[3] = 0u; }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          float4 a = acc[u];
          if (!masks) {
            m[0] |= (a.x > 0.f ? 1u : 0u) << u; m[1] |= (a.y > 0.f ? 1u : 0u) << u;
            m[2] |= (a.z > 0.f ? 1u : 0u) << u; m[3] |= (a.w > 0.f ? 1u : 0u) << u;
          }
          a.x = a.x > 0.f ? a.x : 0.f; a.y = a.y > 0.f ? a.y : 0.f; a.z = a.z > 0.f ? a.z : 0.f; a.w = a.w > 0.f ? a.w : 0.f;
          *reinterpret_cast<float4*>(sm + dst + (h4 + u) * kGfRow + gf_turn(r4, h4)) = a;
        }
      };
      auto adjoint = [&](int dst, const uint32_t (&m)[4]) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          float4 a = acc[u];
          a.x = ((m[0] >> u) & 1u) ? a.x : 0.f; a.y = ((m[1] >> u) & 1u) ? a.y : 0.f;
          a.z = ((m[2] >> u) & 1u) ? a.z : 0.f; a.w = ((m[3] >> u) & 1u) ? a.w : 0.f;
          *reinterpret_cast<float4*>(sm + dst + (h4 + u) * kGfRow + gf_turn(r4, h4)) = a;
        }
      };
      auto start = [&](const float* bias) {
#pragma unroll
        for (int u = 0; u < 4; ++u) { const float b = bias ? bias[h4 + u] : 0.f; acc[u] = make_float4(b, b, b, b); }
      };
      start(sm + kGfB);
      product(kGfE, kGIN, kGfW1T, kGH, false);
      hidden(kGfH1, m1);
      __syncthreads();
      start(sm + kGfB + kGH);
      product(kGfH1, kGH, kGfW2T, kGH, true);
      hidden(kGfH2, m2);
      start(nullptr);
      product8(kGfD3, 4, kGfW3, kGH, r4);
      adjoint(kGfD2, m2);
      __syncthreads();
      start(nullptr);
      product(kGfD2, kGH, kGfW2, kGfW2Row, true);
      adjoint(kGfD1, m1);
      __syncthreads();
      // ---- sums over the records of the thread's half of the block, four at a time (rows past the last record hold zero adjoints) ----
      const int gr = gq * 4, r_end = min(cnt, (half + 1) * (kGfRec / 2));
      for (int r = half * (kGfRec / 2); r < r_end; r += 4) {
        auto at4 = [&](int off, int row) { return *reinterpret_cast<const float4*>(sm + off + row * kGfRow + r); };
        auto turned4 = [&](int off, int row, int turn) { return *reinterpret_cast<const float4*>(sm + off + row * kGfRow + gf_turn(r, turn)); };
        auto sum4 = [](float s, const float4 v) { return ((s + v.x) + v.y) + v.z + v.w; };
        {
          float4 d[4];
#pragma unroll
          for (int a = 0; a < 4; ++a) d[a] = turned4(kGfD1, gr + a, gr);
#pragma unroll
          for (int i = 0; i < 9; ++i) {
            const float4 e = at4(kGfE, hg + 8 * i);
#pragma unroll
            for (int a = 0; a < 4; ++a) g1[a][i] = dot4(g1[a][i], d[a], e);
          }
        }
        {
          float4 d[4];
#pragma unroll
          for (int a = 0; a < 4; ++a) d[a] = turned4(kGfD2, gr + a, gr);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 e = turned4(kGfH1, hg + 8 * i, 8 * i);
#pragma unroll
            for (int a = 0; a < 4; ++a) g2[a][i] = dot4(g2[a][i], d[a], e);
          }
        }
        {
          const float4 h = turned4(kGfH2, th & 31, th & 31);
#pragma unroll
          for (int c = 0; c < 2; ++c) g3[c] = dot4(g3[c], at4(kGfD3, (th >> 5) * 2 + c), h);
        }
        gb = sum4(gb, turned4(th < 32 ? kGfD1 : kGfD2, th & 31, th & 31));
        if (th < 4) gb3 = sum4(gb3, at4(kGfD3, th));
      }
    }
    // the halves' sums meet in shared memory: the first half adds and writes
    {
      auto each = [&](auto f) {
        int j = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
#pragma unroll
          for (int i = 0; i < 9; ++i) f(g1[a][i], j++);
#pragma unroll
          for (int i = 0; i < 4; ++i) f(g2[a][i], j++);
        }
        f(g3[0], j++); f(g3[1], j++); f(gb, j++); f(gb3, j++);
      };
      static_assert(56 * 64 <= kGfH1 - kGfE, "room for one half's sums in the encoding's tile");
      __syncthreads();                           // the last block's rows have been consumed
      if (half == 1) each([&](float& v, int j) { sm[kGfE + j * 64 + th] = v; });
      __syncthreads();
      if (half == 1) continue;
      each([&](float& v, int j) { v += sm[kGfE + j * 64 + th]; });
    }
    const VjpOut o = vjp_row(out, partial, it);
    auto put = [&](float* dst, float v) {
      const float g = v * inv;
      bad |= !(fabsf(g) <= 3.4028235e38f);
      *dst = g;
    };
#pragma unroll
    for (int a = 0; a < 4; ++a) {
#pragma unroll
      for (int i = 0; i < 9; ++i) put(o.W1 + (gq * 4 + a) * kGIN + hg + 8 * i, g1[a][i]);
#pragma unroll
      for (int i = 0; i < 4; ++i) put(o.W2 + (gq * 4 + a) * kGH + hg + 8 * i, g2[a][i]);
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) put(o.W3 + ((th >> 5) * 2 + c) * kGH + (th & 31), g3[c]);
    put(th < 32 ? o.b1 + th : o.b2 + th - 32, gb);
    if (th < 4) put(o.b3 + th, gb3);
  }
  if (bad) atomicOr(counters + kVpFlag, 1);
}

// The gradients of the primitives on the multi list, their partial rows in segment order; and, unless the tensor-core
// kernel has done it between its waits, the zeros of the primitives without records.
__global__ void __launch_bounds__(256) k_vjp_reduce(const VjpItem* __restrict__ multi, const float* __restrict__ partial,
                                                    VjpOut out, int n, int zeros, int aligned, int32_t* __restrict__ counters) {
  chain_wait();
  chain_release();
  const int M = vjp_planned(counters, kVpMulti), E = zeros ? vjp_planned(counters, kVpEmpty) : 0;
  bool bad = false;
  for (int e = blockIdx.x; e < E; e += gridDim.x) vjp_zero(out, __ldg(&multi[n - 1 - e].prim), aligned, threadIdx.x, 256);
  for (int e = blockIdx.x; e < M; e += gridDim.x) {
    VjpItem it = load_item(multi + e);
    it.dest = -1;
    const VjpOut o = vjp_row(out, nullptr, it);
    for (int i = threadIdx.x; i < kGradLen; i += 256) {
      float acc = 0.f;
      for (int g = 0; g < it.rows; ++g) acc += partial[(size_t)(it.start + g) * kGradLen + i];
      float* dst = i < kOb1 ? o.W1 + i : i < kOW2 ? o.b1 + i - kOb1 : i < kOb2 ? o.W2 + i - kOW2 : i < kOW3 ? o.b2 + i - kOb2
                   : i < kOb3 ? o.W3 + i - kOW3 : o.b3 + i - kOb3;
      *dst = acc;
      bad |= !(fabsf(acc) <= 3.4028235e38f);
    }
  }
  if (bad) atomicOr(counters + kVpFlag, 1);
}

int launch_grouped_vjp_tc(bool bf16, const float* x6, const float* d4, const int32_t* masks, const VjpItem* items,
                          int64_t max_items, const VjpItem* multi, int32_t* counters, const mlpsp_scene* sc, float scale,
                          const VjpOut& out, float* partial, cudaStream_t st);

// scratch of a launch: counters | items | multi list | partial rows
struct VjpScratch { int64_t items, multi, partial, bytes, max_items, max_rows; };
static VjpScratch vjp_scratch(int64_t R, int n, int segment_size) {
  VjpScratch s;
  s.max_items = R / segment_size + std::min<int64_t>(n, R);
  s.max_rows = std::min<int64_t>(2 * (R / segment_size), s.max_items);     // a primitive of c > 1 segments owns more than c / 2 of them in full
  int64_t off = 256;
  auto take = [&](int64_t bytes) { const int64_t o = off; off += align_up(bytes, 256); return o; };
  s.items = take((int64_t)sizeof(VjpItem) * s.max_items);
  s.multi = take((int64_t)sizeof(VjpItem) * n);
  s.partial = take(4ll * kGradLen * s.max_rows);
  s.bytes = off + 256;
  return s;
}

// the kernels behind a plan: at most max_items segments, their partial rows added up
static int run_vjp_plan(const mlpsp_scene* sc, const float* x6, const float* d4, const int32_t* masks, const VjpItem* items,
                        int64_t max_items, const VjpItem* multi, int32_t* counters, int precision, float loss_scale,
                        const VjpOut& out, float* partial, cudaStream_t st) {
  const bool tc = max_items > 0 && precision != MLPSP_PRECISION_F32;
  if (tc) {
    const int rc = launch_grouped_vjp_tc(precision == MLPSP_PRECISION_BF16, x6, d4, masks, items, max_items, multi, counters, sc, loss_scale,
                                         out, partial, st);
    if (rc) return rc;
  } else if (max_items > 0) {
    static DeviceOnce attr_once;
    if (attr_once.first())
      MLPSP_CUDA_OK(cudaFuncSetAttribute(k_grouped_vjp, cudaFuncAttributeMaxDynamicSharedMemorySize, kGradSmem));
    const int vec = ((reinterpret_cast<uintptr_t>(sc->W1) | reinterpret_cast<uintptr_t>(sc->W2)) & 15) == 0;
    launch_chained(k_grouped_vjp, dim3((unsigned)std::min<int64_t>(max_items, (int64_t)sm_count() * kGfCtas)), dim3(kGfThreads), kGradSmem, st,
                   x6, d4, masks, items, max_items, counters, sc->freq, sc->att, sc->W1, sc->b1, sc->W2, sc->b2, sc->W3, vec, loss_scale, out, partial);
  }
  launch_chained(k_vjp_reduce, dim3((unsigned)std::min(sc->n, sm_count() * 8)), dim3(256), 0, st, multi, partial, out, sc->n, tc ? 0 : 1,
                 vjp_aligned(out), counters);
  return cuda_check(cudaGetLastError(), "weight_gradients");
}

static int weight_gradients(const mlpsp_scene* sc, const int64_t* offsets, const float* x6, const float* d4, const int32_t* masks,
                            int64_t R, int segment_size, int precision, float loss_scale, const VjpOut& out, void* scratch,
                            int64_t scratch_bytes, int32_t* flag_host, cudaStream_t st) {
  const VjpScratch L = vjp_scratch(R, sc->n, segment_size);
  MLPSP_REQUIRE(scratch && scratch_bytes >= L.bytes, MLPSP_E_SCRATCH, "mlpsp_weight_gradients: scratch needs %lld bytes", (long long)L.bytes);
  // segment_size is a hint.  Segments cut long primitives for the CTAs to share; where the records alone make more than
  // sixteen full segments per CTA, longer ones leave fewer partial rows to write and add, and fewer ragged ends (their sums
  // stay in one accumulator all the same).  512 against the rule's length: 5.9 M records of a 50,000-primitive scene (17,806
  // segments, 12,593 of 1,024) 773 and 717 us, 9.5 M (24,337; 11,182 of 2,048) 1,093 and 973, 7.3 M of 100,000 primitives 1,036
  // and 974, 4.3 M in primitives of 860 516 and 416, of 8,600 494 and 440; the same where no primitive has two segments; slower
  // nowhere.  Below sixteen a doubling is no sure gain: 1.0 M records in primitives of 860 181 and 166 us, of 2,150 182 and 191.
  if (precision != MLPSP_PRECISION_F32)
    while (segment_size < 4096 && R / segment_size > (int64_t)sm_count() * 3 * 16) segment_size *= 2;
  char* base = reinterpret_cast<char*>(align_up((int64_t)reinterpret_cast<uintptr_t>(scratch), 256));
  int32_t* counters = reinterpret_cast<int32_t*>(base);
  VjpItem* items = reinterpret_cast<VjpItem*>(base + L.items);
  VjpItem* multi = reinterpret_cast<VjpItem*>(base + L.multi);
  float* partial = reinterpret_cast<float*>(base + L.partial);
  LaunchScope scope(kKMisc, R > 0 ? 3 : 2, st);
  MLPSP_CUDA_OK(cudaMemsetAsync(counters, 0, 4 * kVpCounters, st));
  launch_chained(k_vjp_plan, dim3((sc->n + 255) / 256), dim3(256), 0, st, offsets, sc->n, R, segment_size, items, L.max_items,
                 multi, counters);
  const int rc = run_vjp_plan(sc, x6, d4, masks, items, L.max_items, multi, counters, precision, loss_scale, out, partial, st);
  if (rc) return rc;
  HostWords& hw = host_words();
  cudaEvent_t ev = nullptr;
  const int opened = hw.open(&ev);
  if (opened) return opened;
  MLPSP_CUDA_OK(cudaMemcpyAsync(hw.word, counters + kVpFlag, 4, cudaMemcpyDeviceToHost, st));
  MLPSP_CUDA_OK(cudaEventRecord(ev, st));
  MLPSP_CUDA_OK(cudaEventSynchronize(ev));
  *flag_host = *static_cast<volatile int32_t*>(hw.word);
  return cuda_check(cudaGetLastError(), "weight_gradients");
}

}  // namespace mlpsp

using namespace mlpsp;

// scratch: findings of the argument checks | the nine sums of every primitive | one weight per record
extern "C" int64_t mlpsp_records_reverse_scratch_bytes(int64_t total_records, int32_t n) {
  if (total_records < 0 || n < 0) return -1;
  return 256 + align_up(4ll * kRevAcc * n, 256) + align_up(4 * total_records, 256) + 256;
}

extern "C" int mlpsp_records_reverse_checked(const int32_t* ids, const int64_t* offsets, const float* x6, const float* raw,
                                             const float* log_scales, const float* quats, const float* grad_rgb,
                                             const float* grad_t, int64_t pixels, int64_t total_records, int32_t n, float* d4,
                                             float* grad_pos, float* grad_log_scales, float* grad_quats, void* scratch,
                                             int64_t scratch_bytes, int32_t* findings_host, void* stream) {
  MLPSP_REQUIRE(pixels >= 0 && n >= 0 && total_records >= 0, MLPSP_E_ARG, "mlpsp_records_reverse: negative size");
  MLPSP_REQUIRE(offsets && (n == 0 || (log_scales && quats && grad_pos && grad_log_scales && grad_quats)) &&
                    (pixels == 0 || (grad_rgb && grad_t)) && (total_records == 0 || (ids && x6 && raw && d4 && quats)),
                MLPSP_E_ARG, "mlpsp_records_reverse: null pointer");
  MLPSP_REQUIRE(((reinterpret_cast<uintptr_t>(raw) | reinterpret_cast<uintptr_t>(d4) | reinterpret_cast<uintptr_t>(quats)) & 15) == 0,
                MLPSP_E_ARG, "mlpsp_records_reverse: raw, d4 and quats must be 16-byte aligned");
  MLPSP_REQUIRE(scratch && scratch_bytes >= mlpsp_records_reverse_scratch_bytes(total_records, n), MLPSP_E_SCRATCH,
                "mlpsp_records_reverse: scratch too small");
  cudaStream_t st = (cudaStream_t)stream;
  char* base = reinterpret_cast<char*>(align_up((int64_t)reinterpret_cast<uintptr_t>(scratch), 256));
  int32_t* bad = reinterpret_cast<int32_t*>(base);          // cleared together with the sums behind it
  float* acc = reinterpret_cast<float*>(base + 256);
  float* kw = reinterpret_cast<float*>(base + 256 + align_up(4ll * kRevAcc * n, 256));
  HostWords& hw = host_words();
  cudaEvent_t ev = nullptr;
  if (findings_host) {
    const int rc = hw.open(&ev);
    if (rc) return rc;
    hw.word[0] = 0;
  }
  LaunchScope scope(kKMisc, 4, st);
  MLPSP_CUDA_OK(cudaMemsetAsync(base, 0, 256 + 4ll * kRevAcc * n, st));
  const int64_t most = std::max(total_records, pixels);
  launch_chained(k_reverse_check, dim3((unsigned)std::min<int64_t>(148 * 8, most / 1024 + 1)), dim3(256), 0, st, ids, total_records, n, offsets,
                 pixels, bad, findings_host ? hw.word : nullptr);
  if (findings_host) MLPSP_CUDA_OK(cudaEventRecord(ev, st));
  if (pixels > 0 && total_records > 0) {
    static DeviceOnce attr_once;
    if (attr_once.first())
      MLPSP_CUDA_OK(cudaFuncSetAttribute(k_reverse_geometry, cudaFuncAttributeMaxDynamicSharedMemorySize, kRevSmem));
    launch_chained(k_reverse_pixels, dim3((unsigned)((pixels + kRevPixels - 1) / kRevPixels)), dim3(kRevPixels), 0, st, offsets, raw, grad_rgb, grad_t, pixels, d4, kw, bad);
    launch_chained(k_reverse_geometry, dim3((unsigned)((total_records + kRevChunk - 1) / kRevChunk)), dim3(kRevThreads),
                   kRevSmem, st, ids, x6, kw, quats,
                   total_records, acc, bad);
  }
  if (n > 0) launch_chained(k_reverse_finish, dim3((n + 127) / 128), dim3(128), 0, st, acc, log_scales, quats, n, grad_pos, grad_log_scales, grad_quats,
                            (reinterpret_cast<uintptr_t>(grad_quats) & 15) == 0 ? 1 : 0);
  MLPSP_CUDA_OK(cudaGetLastError());
  if (findings_host) {
    MLPSP_CUDA_OK(cudaEventSynchronize(ev));
    *findings_host = *static_cast<volatile int32_t*>(hw.word);
  }
  return MLPSP_OK;
}

extern "C" int mlpsp_records_reverse(const int32_t* ids, const int64_t* offsets, const float* x6, const float* raw,
                                     const float* log_scales, const float* quats, const float* grad_rgb,
                                     const float* grad_t, int64_t pixels, int64_t total_records, int32_t n, float* d4,
                                     float* grad_pos, float* grad_log_scales, float* grad_quats, void* stream) {
  MLPSP_REQUIRE(pixels >= 0 && n >= 0, MLPSP_E_ARG, "mlpsp_records_reverse: negative size");
  MLPSP_REQUIRE(offsets && grad_pos && grad_log_scales && grad_quats, MLPSP_E_ARG, "mlpsp_records_reverse: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  if (pixels == 0) {             // nothing is read: zero gradients
    MLPSP_CUDA_OK(cudaMemsetAsync(grad_pos, 0, sizeof(float) * 3 * (size_t)n, st));
    MLPSP_CUDA_OK(cudaMemsetAsync(grad_log_scales, 0, sizeof(float) * 3 * (size_t)n, st));
    return cuda_check(cudaMemsetAsync(grad_quats, 0, sizeof(float) * 4 * (size_t)n, st), "records_reverse");
  }
  MLPSP_REQUIRE(ids && x6 && raw && log_scales && quats && grad_rgb && grad_t && d4, MLPSP_E_ARG, "mlpsp_records_reverse: null pointer");
  MLPSP_REQUIRE(total_records >= 0, MLPSP_E_ARG, "mlpsp_records_reverse: negative record count");
  // the variant with the caller's scratch, which this signature has no room for: taken from the stream's pool
  const int64_t bytes = mlpsp_records_reverse_scratch_bytes(total_records, n);
  char* work = nullptr;
  MLPSP_CUDA_OK(cudaMallocAsync(&work, bytes, st));
  const int rc = mlpsp_records_reverse_checked(ids, offsets, x6, raw, log_scales, quats, grad_rgb, grad_t, pixels, total_records, n,
                                               d4, grad_pos, grad_log_scales, grad_quats, work, bytes, nullptr, stream);
  cudaFreeAsync(work, st);
  return rc;
}

extern "C" int64_t mlpsp_grouped_gradient_floats(void) { return kGradLen; }

static int check_gradient_args(const mlpsp_scene* sc, int64_t segment_size, int precision, float loss_scale, const char* who) {
  MLPSP_REQUIRE(sc->hidden == kGH && sc->num_freq == 6, MLPSP_E_LIMIT,
                "grouped backward requires the 72->32->32->4 architecture");
  MLPSP_REQUIRE(sc->W1 && sc->b1 && sc->W2 && sc->b2 && sc->W3 && sc->freq && sc->att, MLPSP_E_ARG,
                "%s: FP32 weights missing", who);
  MLPSP_REQUIRE(loss_scale > 0.f && segment_size > 0, MLPSP_E_ARG, "%s: bad loss scale, segment size or segment count", who);
  MLPSP_REQUIRE(precision == MLPSP_PRECISION_F32 || precision == MLPSP_PRECISION_F16 || precision == MLPSP_PRECISION_BF16,
                MLPSP_E_ARG, "%s: unsupported operand precision %d", who, precision);
  return MLPSP_OK;
}
static int check_gradient_rows(const float* d4, int precision, const char* who) {
  MLPSP_REQUIRE(precision == MLPSP_PRECISION_F32 || (reinterpret_cast<uintptr_t>(d4) & 15) == 0, MLPSP_E_ARG,
                "%s: d4 must be 16-byte aligned", who);
  return MLPSP_OK;
}

extern "C" int64_t mlpsp_weight_gradients_scratch_bytes(int64_t num_records, int32_t n, int32_t segment_size) {
  if (num_records < 0 || n < 0 || segment_size <= 0) return -1;
  return vjp_scratch(num_records, n, segment_size).bytes;
}

extern "C" int mlpsp_weight_gradients(const mlpsp_scene* sc, const int64_t* offsets, const float* x6, const float* d4,
                                      const int32_t* relu_masks, int64_t num_records, int32_t segment_size, int32_t precision,
                                      float loss_scale, float* dW1, float* db1, float* dW2, float* db2, float* dW3, float* db3,
                                      void* scratch, int64_t scratch_bytes, int32_t* nonfinite_host, void* stream) {
  MLPSP_REQUIRE(sc && offsets && nonfinite_host && num_records >= 0, MLPSP_E_ARG, "mlpsp_weight_gradients: null pointer");
  int rc = check_gradient_args(sc, segment_size, precision, loss_scale, "mlpsp_weight_gradients");
  if (!rc) rc = check_gradient_rows(d4, precision, "mlpsp_weight_gradients");
  if (rc) return rc;
  *nonfinite_host = 0;
  if (sc->n == 0) return MLPSP_OK;
  MLPSP_REQUIRE(dW1 && db1 && dW2 && db2 && dW3 && db3 && (num_records == 0 || (x6 && d4)), MLPSP_E_ARG,
                "mlpsp_weight_gradients: null pointer");
  MLPSP_REQUIRE(num_records / segment_size + sc->n < (1ll << 31), MLPSP_E_LIMIT, "mlpsp_weight_gradients: too many segments");
  const VjpOut out = {dW1, db1, dW2, db2, dW3, db3, kGH * kGIN, kGH, kGH * kGH, kGH, 4 * kGH, 4};
  return weight_gradients(sc, offsets, x6, d4, relu_masks, num_records, segment_size, precision, loss_scale, out, scratch,
                          scratch_bytes, nonfinite_host, (cudaStream_t)stream);
}

extern "C" int mlpsp_grouped_weight_gradients(const mlpsp_scene* sc, const int64_t* offsets, const float* x6,
                                              const float* d4, const int32_t* relu_masks, const int64_t* seg_prim,
                                              const int64_t* seg_start, const int64_t* seg_offsets, int64_t num_segments,
                                              int32_t segment_size, int32_t precision, float loss_scale, float* partial,
                                              float* result, int32_t* nonfinite, void* stream) {
  MLPSP_REQUIRE(sc && offsets && result && nonfinite, MLPSP_E_ARG, "mlpsp_grouped_weight_gradients: null pointer");
  int rc = check_gradient_args(sc, segment_size, precision, loss_scale, "mlpsp_grouped_weight_gradients");
  if (rc) return rc;
  MLPSP_REQUIRE(num_segments >= 0 && num_segments < (1ll << 31), MLPSP_E_ARG,
                "mlpsp_grouped_weight_gradients: bad loss scale, segment size or segment count");
  // every pointer a launch below reads is checked before the first CUDA call
  MLPSP_REQUIRE(sc->n == 0 || num_segments == 0 || (x6 && d4 && seg_prim && seg_start && seg_offsets && partial),
                MLPSP_E_ARG, "mlpsp_grouped_weight_gradients: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  MLPSP_CUDA_OK(cudaMemsetAsync(nonfinite, 0, 4, st));
  if (sc->n == 0) return MLPSP_OK;
  if (num_segments == 0)       // no records at all: every primitive's gradient row is zero
    return cuda_check(cudaMemsetAsync(result, 0, sizeof(float) * (size_t)sc->n * kGradLen, st), "grouped_weight_gradients");
  rc = check_gradient_rows(d4, precision, "mlpsp_grouped_weight_gradients");
  if (rc) return rc;
  // the work lists, 32 bytes per segment and primitive, have no room in this signature: they come from the stream's pool
  const int64_t item_bytes = align_up((int64_t)sizeof(VjpItem) * num_segments, 256);
  char* work = nullptr;
  MLPSP_CUDA_OK(cudaMallocAsync(&work, 256 + item_bytes + (int64_t)sizeof(VjpItem) * sc->n, st));
  int32_t* counters = reinterpret_cast<int32_t*>(work);
  VjpItem* items = reinterpret_cast<VjpItem*>(work + 256);
  VjpItem* multi = reinterpret_cast<VjpItem*>(work + 256 + item_bytes);
  float* r = result;
  const VjpOut out = {r + kOW1, r + kOb1, r + kOW2, r + kOb2, r + kOW3, r + kOb3, kGradLen, kGradLen, kGradLen, kGradLen, kGradLen, kGradLen};
  LaunchScope scope(kKMisc, 3, st);
  rc = cuda_check(cudaMemsetAsync(counters, 0, 4 * kVpCounters, st), "grouped_weight_gradients");
  if (!rc)
    rc = cuda_check(launch_chained(k_vjp_plan_layout, dim3((unsigned)((std::max<int64_t>(num_segments, sc->n) + 255) / 256)), dim3(256), 0,
                                   st, offsets, sc->n, segment_size, seg_prim, seg_start, seg_offsets, (int)num_segments, items, multi,
                                   counters), "grouped_weight_gradients");
  if (!rc)
    rc = run_vjp_plan(sc, x6, d4, relu_masks, items, num_segments, multi, counters, precision, loss_scale, out, partial, st);
  if (!rc) rc = cuda_check(cudaMemcpyAsync(nonfinite, counters + kVpFlag, 4, cudaMemcpyDeviceToDevice, st), "grouped_weight_gradients");
  cudaFreeAsync(work, st);
  return rc;
}
