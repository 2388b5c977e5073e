// Hit masks, primitive-major record construction (CSR), and front-to-back compositing.
//
// The reference walks a tile's sorted list serially and evaluates the MLP inside that walk
// (scannet/cuda/np_tile_kernels.cu:2110-2117).  Here the walk is cut into waves of consecutive
// list positions.  Per wave:
//   k_hits       every still-active pixel is tested against the wave's candidates
//                (hit_and_features_rot, np_tile_kernels.cu:659-711); one 64-bit mask per
//                (tile, candidate) pair, record slots reserved tile-major
//   prim scan    per-primitive record counts -> CSR offsets + evaluator work items
//   k_fill       (pixel, primitive) records written primitive-major: the 6-vector fed to the
//                encoder, decay, and the slot compositing will read
//   evaluator    per-primitive MLP over its records (mlp_f32.cu / mlp_tc.cu)
//   k_composite  per pixel, in list order, only while transmittance >= 1e-3
//                (np_tile_kernels.cu:2025-2136); tiles with a live pixel and candidates left go
//                on the next wave's list
// A record evaluated in a wave but reached after its pixel terminated inside the same wave is
// skipped by compositing, so results do not depend on the wave schedule.
#include <algorithm>
#include <climits>
#include <cmath>
#include "frame.cuh"

namespace mlpsp {

constexpr int kWinMax = 2048;

// squared bounding radius in units of the largest scale, with the 2 % margin surely_misses() relies on
static inline float miss_bound2(float thr) { return (float)(-2.0 * log((double)thr) * 1.02); }
// threshold of the quadratic form, -2 ln thr; 0 (no form) where decay could underflow before it reaches thr
static inline float form_threshold(float thr) { const double k = -2.0 * log((double)thr); return k > 0.0 && k < 170.0 ? (float)k : 0.f; }

// -------------------------------------------------------------------------- frame init ----
// One launch prepares a frame whose lists come from the caller (k_frame_begin prepares the fused path): pixel state and the output image, the list of live tiles and the wave counters,
// and the per-primitive counts and cursors of the first wave.
// tile_len = the length of the caller's list.
__global__ void k_init_frame(int64_t P, float4* __restrict__ px_state, float2* __restrict__ px_depth,
                             float* __restrict__ rgb, float* __restrict__ alpha, float* __restrict__ depth_t,
                             float bgr, float bgg, float bgb, int T, int32_t* __restrict__ active0,
                             int32_t* __restrict__ counters, const int32_t* __restrict__ tile_offsets,
                             int32_t* __restrict__ tile_len, int n, int32_t* __restrict__ prim_cnt) {
  chain_wait();
  chain_release();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < P) {
    px_state[i] = make_float4(0.f, 0.f, 0.f, 1.f);
    px_depth[i] = make_float2(0.f, 0.f);
    rgb[i * 3] = bgr; rgb[i * 3 + 1] = bgg; rgb[i * 3 + 2] = bgb;
    alpha[i] = 0.f;
    if (depth_t) depth_t[i] = 0.f;
  }
  if (i < T) {
    active0[i] = (int)i;
    tile_len[i] = tile_offsets[i + 1] - tile_offsets[i];
  }
  if (i < n) { prim_cnt[i] = 0; prim_cnt[prim_cnt_stride(n) + i] = 0; }   // the counts of even and odd waves
  if (i == 0) {
    counters[kCtrRecords] = 0;
    counters[kCtrActive0] = T; counters[kCtrActive1] = 0;
  }
}

// consumed-record masks of the pairs the tiles will traverse
__global__ void __launch_bounds__(256) k_clear_used(const int32_t* __restrict__ tile_offsets, const int32_t* __restrict__ tile_len,
                                                    int T, uint2* __restrict__ used, const int32_t* __restrict__ status) {
  chain_wait();
  chain_release();
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int tile = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (tile >= T) return;
  const int s = tile_offsets[tile], len = tile_len[tile];
  for (int i = threadIdx.x & 31; i < len; i += 32) used[s + i] = make_uint2(0u, 0u);
}

// ------------------------------------------------------------------------- frame begin ----
// The fused frame path starts with one launch that prepares everything the chain behind it reads: unit ray directions
// (from the caller's raw ones, when given), the tiles' rectangles in the tangent plane for the binning pre-test, pixel state and output
// image, the per-primitive counts, the binning's corner array and fill counters, the tile lists' cursors and the wave
// counters, the status block.  (One warp per tile, two pixels per lane; the flat arrays by all threads.)  It replaces a
// normalising launch, two preparing launches and four memsets.
struct BeginArgs {
  const float* rays_o; const float* rays_raw; float* rays_d;   // rays_raw null: rays_d already holds unit directions
  int W, H, ntx, T;
  FramePlane* plane; float4* tile_rect; int32_t* fill; int32_t* zero; int64_t zero_words;     // corner array (or tile counts) of the binning
  float4* px_state; float2* px_depth; float* rgb; float* alpha; float* depth_t; float bgr, bgg, bgb;
  int32_t* active0; int32_t* counters; int64_t cnt_words; int32_t* prim_cnt;
  int32_t* status;                                             // null: the caller has reset it
};

template <int V>
__global__ void __launch_bounds__(256) k_frame_begin(const __grid_constant__ Views<BeginArgs, V> b) {
  chain_wait();
  chain_release();
  const BeginArgs& a = b.v[view_of_cta<V>()];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t gid = (int64_t)blockIdx.x * 256 + threadIdx.x, gn = (int64_t)gridDim.x * 256;
  for (int64_t i = gid; i * 4 < a.cnt_words; i += gn) *reinterpret_cast<int4*>(a.prim_cnt + i * 4) = make_int4(0, 0, 0, 0);
  for (int64_t i = gid; i < a.zero_words; i += gn) a.zero[i] = 0;
  if (blockIdx.x == 0 && threadIdx.x < kNumCounters)
    a.counters[threadIdx.x] = threadIdx.x == kCtrActive0 ? a.T : 0;
  if (a.status && blockIdx.x == 0 && threadIdx.x < MLPSP_STATUS_WORDS) a.status[threadIdx.x] = 0;
  // the tangent plane (every thread computes the same one): around the central ray, u along the central image row
  FramePlane f;
  {
    const int64_t row = (int64_t)(a.H / 2) * a.W;
    const float* rays = a.rays_raw ? a.rays_raw : a.rays_d;
    auto ray = [&](int x) {
      const V3 d = {rays[(row + x) * 3], rays[(row + x) * 3 + 1], rays[(row + x) * 3 + 2]};
      const float r = rsqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
      return V3{d.x * r, d.y * r, d.z * r};
    };
    const V3 o = load3(a.rays_o, row + a.W / 2), c = ray(a.W / 2), lft = ray(0), rgt = ray(a.W - 1);
    float ux = rgt.x - lft.x, uy = rgt.y - lft.y, uz = rgt.z - lft.z;
    if (!(ux * ux + uy * uy + uz * uz > 1e-10f)) {      // a column of pixels: any axis
      ux = fabsf(c.x) < 0.57f ? 1.f : 0.f; uy = fabsf(c.x) < 0.57f ? 0.f : 1.f; uz = 0.f;
    }
    const float ua = ux * c.x + uy * c.y + uz * c.z;
    ux -= ua * c.x; uy -= ua * c.y; uz -= ua * c.z;
    const float r = rsqrtf(ux * ux + uy * uy + uz * uz);
    f.ox = o.x; f.oy = o.y; f.oz = o.z; f.ax = c.x; f.ay = c.y; f.az = c.z;
    f.ux = ux * r; f.uy = uy * r; f.uz = uz * r;
    f.vx = f.ay * f.uz - f.az * f.uy; f.vy = f.az * f.ux - f.ax * f.uz; f.vz = f.ax * f.uy - f.ay * f.ux;
    f.pad0 = f.pad1 = f.pad2 = f.pad3 = 0.f;
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.plane = f;
  }
  for (int tile = blockIdx.x * 8 + warp; tile < a.T; tile += gridDim.x * 8) {
    const int tx = tile % a.ntx, ty = tile / a.ntx;
    bool same = true;
    float a0 = 3e38f, a1 = -3e38f, b0 = 3e38f, b1 = -3e38f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = h * 32 + lane;
      const int x = tx * 8 + (k & 7), y = ty * 8 + (k >> 3);
      if (x >= a.W || y >= a.H) continue;
      const int64_t pix = (int64_t)y * a.W + x;
      const V3 o = load3(a.rays_o, pix);
      V3 d;
      if (a.rays_raw) {
        d = load3(a.rays_raw, pix);
        const float nrm = fmaxf(__fsqrt_rn(ffma(d.z, d.z, ffma(d.y, d.y, fmul(d.x, d.x)))), 1e-12f);
        d = V3{fdiv(d.x, nrm), fdiv(d.y, nrm), fdiv(d.z, nrm)};
        a.rays_d[pix * 3] = d.x; a.rays_d[pix * 3 + 1] = d.y; a.rays_d[pix * 3 + 2] = d.z;
      } else {
        d = V3{a.rays_d[pix * 3], a.rays_d[pix * 3 + 1], a.rays_d[pix * 3 + 2]};
      }
      const float da = d.x * f.ax + d.y * f.ay + d.z * f.az, len2 = d.x * d.x + d.y * d.y + d.z * d.z;
      const float al = (d.x * f.ux + d.y * f.uy + d.z * f.uz) / da, be = (d.x * f.vx + d.y * f.vy + d.z * f.vz) / da;
      same = same && o.x == f.ox && o.y == f.oy && o.z == f.oz && da * rsqrtf(len2) > 0.26f && fabsf(al) < 1e3f && fabsf(be) < 1e3f;
      a0 = fminf(a0, al); a1 = fmaxf(a1, al); b0 = fminf(b0, be); b1 = fmaxf(b1, be);
      a.px_state[pix] = make_float4(0.f, 0.f, 0.f, 1.f);
      a.rgb[pix * 3] = a.bgr; a.rgb[pix * 3 + 1] = a.bgg; a.rgb[pix * 3 + 2] = a.bgb;
      a.alpha[pix] = 0.f;
      if (a.depth_t) { a.depth_t[pix] = 0.f; a.px_depth[pix] = make_float2(0.f, 0.f); }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      a0 = fminf(a0, __shfl_xor_sync(0xffffffffu, a0, off)); a1 = fmaxf(a1, __shfl_xor_sync(0xffffffffu, a1, off));
      b0 = fminf(b0, __shfl_xor_sync(0xffffffffu, b0, off)); b1 = fmaxf(b1, __shfl_xor_sync(0xffffffffu, b1, off));
    }
    same = __all_sync(0xffffffffu, same);
    if (lane == 0) {
      // inflate the rectangle: rounding of the coordinates and of the plane's frame
      const float pa = 2e-6f * (1.f + fabsf(a0) + fabsf(a1)) * (1.f + fabsf(a0) + fabsf(a1) + fabsf(b0) + fabsf(b1)) + 1e-3f * (a1 - a0);
      const float pb = 2e-6f * (1.f + fabsf(b0) + fabsf(b1)) * (1.f + fabsf(a0) + fabsf(a1) + fabsf(b0) + fabsf(b1)) + 1e-3f * (b1 - b0);
      const float nan = __int_as_float(0x7fc00000);
      a.tile_rect[tile] = same ? make_float4(a0 - pa, a1 + pa, b0 - pb, b1 + pb) : make_float4(nan, nan, nan, nan);
      a.fill[tile] = 0;
      a.active0[tile] = tile;
    }
  }
}

static BeginArgs begin_args(const mlpsp_scene* sc, const mlpsp_frame* fr, const Scratch& s, const float* rays_raw, bool reset_status,
                            int32_t* prim_cnt) {
  BeginArgs a;
  a.rays_o = fr->rays_o; a.rays_raw = rays_raw; a.rays_d = const_cast<float*>(fr->rays_d);
  a.W = fr->width; a.H = fr->height; a.ntx = (fr->width + 7) / 8; a.T = num_tiles(fr->width, fr->height, 8);
  a.plane = s.plane; a.tile_rect = s.tile_rect; a.fill = s.tile_len;
  const bool corners = bin_uses_corners(fr);
  a.zero = corners ? s.tile_diff : s.tile_cnt;
  a.zero_words = corners ? (int64_t)(a.ntx + 1) * ((fr->height + 7) / 8 + 1) : a.T + 1;
  a.px_state = s.px_state; a.px_depth = s.px_depth; a.rgb = fr->rgb; a.alpha = fr->alpha; a.depth_t = fr->depth_t;
  a.bgr = a.bgg = a.bgb = 0.f;
  if (fr->bg_color) { a.bgr = fr->bg_color[0]; a.bgg = fr->bg_color[1]; a.bgb = fr->bg_color[2]; }
  a.active0 = s.active[0]; a.counters = s.counters;
  a.prim_cnt = prim_cnt; a.cnt_words = prim_cnt ? 2 * (int64_t)prim_cnt_stride(sc->n) : 0;
  a.status = reset_status ? fr->status : nullptr;
  return a;
}

int launch_frame_begin(const mlpsp_scene* sc, const mlpsp_frame* frs, const Scratch* ss, int views, const float* const* rays_raw,
                       bool reset_status, cudaStream_t st) {
  LaunchScope scope(kKMisc, (views + kViewsPerLaunch - 1) / kViewsPerLaunch, st);
  cudaError_t e = cudaSuccess;
  for (int v0 = 0; v0 < views && e == cudaSuccess; v0 += kViewsPerLaunch) {
    BeginArgs a[kViewsPerLaunch];
    const int count = std::min(kViewsPerLaunch, views - v0);
    // the per-primitive counts are the first view's
    for (int q = 0; q < count; ++q)
      a[q] = begin_args(sc, frs + v0 + q, ss[v0 + q], rays_raw ? rays_raw[v0 + q] : nullptr, reset_status && v0 + q == 0,
                        v0 + q == 0 ? ss[0].prim_cnt : nullptr);
    const dim3 grid(std::max((a[0].T + 7) / 8, (int)std::min<int64_t>(sm_count() * 8, (a[0].cnt_words / 4 + 255) / 256)));
    if (count == 1) e = launch_views<1>(k_frame_begin<1>, grid, dim3(256), 0, st, a, 1);
    else e = launch_views<kViewsPerLaunch>(k_frame_begin<kViewsPerLaunch>, grid, dim3(256), 0, st, a, count);
  }
  return cuda_check(e, "frame_begin");
}

// --------------------------------------------------------------------------- hit pass ----
// The exact decision (hit_test) costs about 130 FP32 operations per pixel and candidate.  Almost every decision is far
// from the threshold, and for a candidate and the rays of one tile, which leave one origin, it is the sign of a quadratic
// form: with the rays as a + alpha u + beta v up to scale (an orthonormal frame of the tile) and x, e the primitive-frame
// offset and direction divided by its scales, decay > thr <=> |x cross e|^2 < K |e|^2 with K = -2 ln thr -- six
// coefficients per (tile, candidate), computed by one lane, and five multiply-adds per pixel.  The pixel's value decides
// when it is further from zero than the candidate's tolerance; the few pixels in between are decided by hit_test itself,
// so every decision is hit_test's.
//
// Tolerance, relative to |e|^2 (u = 2^-24, S = |c - o| + |o|, im = largest inverse scale): building x and e from rounded
// matrices costs |x cross e| at most 45 u S im |e| (frame and ray rounding included), hence the form 90 u sqrt(K) S im =
// 5.4e-6 sqrt(K) S im near the threshold; hit_test's own foot point p = o + t d is off by u S per axis, 6 u sqrt(K) S im;
// its relative errors (r^2, the exponential, the rounded threshold) stay below 20 u K, and those of |e| below
// 12 u K im / |e|; evaluating the polynomial adds 10 u times the sum M of its terms' magnitudes.  The constants below are
// above the sum of these.  t > 0 is decided for the whole tile from x . e with a margin of 1e-3 |x||e| (rounding is below
// 10 u im (|c - o||e| + |x|)); a candidate that is neither surely in front nor surely behind, or not finite, is left to
// hit_test altogether.
struct RayFrame {
  V3 o, a, u, v;           // common origin and frame
  float A, B;              // largest |alpha|, |beta| of the tile
  bool fast;               // the tile has such a frame
};

__device__ __forceinline__ void hit_form(const Geom& g, const RayFrame& f, float K, float4& q0, float4& q1) {
  const float kAll = __int_as_float(0x7f800000);
  const PrimWhiten pw = make_whiten(g);
  const float vx = g.cx - f.o.x, vy = g.cy - f.o.y, vz = g.cz - f.o.z;
  const V3 x = whiten(pw, vx, vy, vz);
  const V3 e0 = whiten(pw, f.a.x, f.a.y, f.a.z), e1 = whiten(pw, f.u.x, f.u.y, f.u.z), e2 = whiten(pw, f.v.x, f.v.y, f.v.z);
  const V3 w0 = {x.y * e0.z - x.z * e0.y, x.z * e0.x - x.x * e0.z, x.x * e0.y - x.y * e0.x};
  const V3 w1 = {x.y * e1.z - x.z * e1.y, x.z * e1.x - x.x * e1.z, x.x * e1.y - x.y * e1.x};
  const V3 w2 = {x.y * e2.z - x.z * e2.y, x.z * e2.x - x.x * e2.z, x.x * e2.y - x.y * e2.x};
  auto dot = [](const V3& p, const V3& q) { return p.x * q.x + p.y * q.y + p.z * q.z; };
  const float e00 = dot(e0, e0), e11 = dot(e1, e1), e22 = dot(e2, e2);
  const float c0 = dot(w0, w0) - K * e00;
  const float b1 = 2.f * (dot(w0, w1) - K * dot(e0, e1)), b2 = 2.f * (dot(w0, w2) - K * dot(e0, e2));
  const float a11 = dot(w1, w1) - K * e11, a22 = dot(w2, w2) - K * e22, a12 = 2.f * (dot(w1, w2) - K * dot(e1, e2));
  const float M = dot(w0, w0) + K * e00 + f.A * (fabsf(b1) + f.A * fabsf(a11) + f.B * fabsf(a12)) + f.B * (fabsf(b2) + f.B * fabsf(a22));
  const float emax = sqrtf(e00) + f.A * sqrtf(e11) + f.B * sqrtf(e22);
  const float dist = fabsf(vx) + fabsf(vy) + fabsf(vz), S = dist + fabsf(f.o.x) + fabsf(f.o.y) + fabsf(f.o.z);
  float tol = ((8e-6f * sqrtf(K) * S * pw.ismax + 1e-4f * K) * emax + 1e-6f * K * pw.ismax) * emax + 1e-6f * M;
  const float xn = sqrtf(dot(x, x)), mid = dot(x, e0), var = f.A * fabsf(dot(x, e1)) + f.B * fabsf(dot(x, e2));
  const float margin = 1e-3f * xn * emax + 3e-6f * pw.ismax * (dist * emax + xn);
  if (!(e00 > 1e-14f) || !(mid - var > margin)) tol = kAll;
  q0 = make_float4(c0, b1, b2, tol);
  q1 = make_float4(a11, a12, a22, 0.f);
  if (mid + var < -margin && e00 > 1e-14f) { q0 = make_float4(1.f, 0.f, 0.f, 0.f); q1 = make_float4(0.f, 0.f, 0.f, 0.f); }   // behind every ray's origin
  if (!f.fast) q0.w = kAll;
}

// A warp's view of a tile: lane l owns the pixels l and 32 + l.
struct HitPixels {
  RayFrame f;
  float al[2], be[2];
  int pix[2];
  uint32_t act[2];         // live pixels of the two halves
};

__device__ __forceinline__ HitPixels hit_pixels(const float* __restrict__ rays_o, const float* __restrict__ rays_d,
                                                const float4* __restrict__ px_state, int tile, int ntx, int W, int H, bool allow) {
  HitPixels h;
  const int lane = threadIdx.x & 31;
  V3 o[2], d[2];
  bool valid[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const TilePix tp = tile_pixel(tile, k * 32 + lane, ntx, W, H);
    valid[k] = tp.valid;
    h.pix[k] = tp.pix;
    o[k] = d[k] = V3{0.f, 0.f, 0.f};
    bool live = false;
    if (tp.valid) {
      o[k] = load3(rays_o, tp.pix);
      d[k] = load3(rays_d, tp.pix);
      live = px_state[tp.pix].w >= MLPSP_TERM;
    }
    h.act[k] = __ballot_sync(0xffffffffu, live);
  }
  // the frame around one of the central rays (pixel (3, 3), or the tile's first at the image's border)
  const uint32_t v0 = __ballot_sync(0xffffffffu, valid[0]);
  const int src = (v0 >> 27) & 1u ? 27 : 0;
  h.f.o = V3{__shfl_sync(0xffffffffu, o[0].x, src), __shfl_sync(0xffffffffu, o[0].y, src), __shfl_sync(0xffffffffu, o[0].z, src)};
  h.f.a = V3{__shfl_sync(0xffffffffu, d[0].x, src), __shfl_sync(0xffffffffu, d[0].y, src), __shfl_sync(0xffffffffu, d[0].z, src)};
  V3 a = h.f.a;
  const float ra = rsqrtf(a.x * a.x + a.y * a.y + a.z * a.z);
  a.x *= ra; a.y *= ra; a.z *= ra;
  V3 u = fabsf(a.x) < 0.6f ? V3{0.f, a.z, -a.y} : V3{-a.z, 0.f, a.x};
  const float ru = rsqrtf(u.x * u.x + u.y * u.y + u.z * u.z);
  u.x *= ru; u.y *= ru; u.z *= ru;
  h.f.a = a; h.f.u = u;
  h.f.v = V3{a.y * u.z - a.z * u.y, a.z * u.x - a.x * u.z, a.x * u.y - a.y * u.x};
  bool same = allow;
  float A = 0.f, B = 0.f;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float da = d[k].x * a.x + d[k].y * a.y + d[k].z * a.z;
    const float r = __fdividef(1.f, da);
    h.al[k] = (d[k].x * u.x + d[k].y * u.y + d[k].z * u.z) * r;
    h.be[k] = (d[k].x * h.f.v.x + d[k].y * h.f.v.y + d[k].z * h.f.v.z) * r;
    if (!valid[k]) { h.al[k] = h.be[k] = 0.f; continue; }
    const float dd = d[k].x * d[k].x + d[k].y * d[k].y + d[k].z * d[k].z;
    same = same && o[k].x == h.f.o.x && o[k].y == h.f.o.y && o[k].z == h.f.o.z && da > 0.7f && dd < 1.01f;
    A = fmaxf(A, fabsf(h.al[k])); B = fmaxf(B, fabsf(h.be[k]));
  }
  h.f.fast = __all_sync(0xffffffffu, same);
  h.f.A = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(A)));
  h.f.B = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(B)));
  return h;
}

template <bool REF>
__device__ __noinline__ bool hit_exact(const float* __restrict__ rays_o, const float* __restrict__ rays_d, const float4* __restrict__ geom,
                                       int p, int pix, float thr, float bound2) {
  const V3 o = load3(rays_o, pix), d = load3(rays_d, pix);
  const Geom g = load_geom(geom, p);
  if (surely_misses(g, o, d, bound2)) return false;
  Hit h;
  return REF ? hit_test_ref(load_geom_ref(geom, p), o, d, thr, h) : hit_test(g, o, d, thr, h);
}

// Hit masks (m0, m1: the tile's two pixel halves) of the candidate ids p_lane of a chunk of cnt <= 32 candidates, lane l
// holding the l-th; s_q: the warp's 64 float4 of shared memory.
template <bool REF>
__device__ __forceinline__ void hit_chunk(const HitPixels& h, const float* __restrict__ rays_o, const float* __restrict__ rays_d,
                                          const float4* __restrict__ geom, int n, int p_lane, int cnt, float K, float thr,
                                          float bound2, float4* s_q, uint32_t& m0, uint32_t& m1) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  if (lane < cnt) {
    float4 q0 = make_float4(1.f, 0.f, 0.f, 0.f), q1 = make_float4(0.f, 0.f, 0.f, 0.f);     // misses
    if (p_lane >= 0 && p_lane < n) hit_form(load_geom(geom, p_lane), h.f, K, q0, q1);
    s_q[2 * lane] = q0;
    s_q[2 * lane + 1] = q1;
  }
  __syncwarp();
  m0 = m1 = 0u;
  const bool live0 = (h.act[0] >> lane) & 1u, live1 = (h.act[1] >> lane) & 1u;
#pragma unroll 2
  for (int t = 0; t < cnt; ++t) {
    const float4 q0 = s_q[2 * t], q1 = s_q[2 * t + 1];
    const float f0 = fmaf(fmaf(q1.x, h.al[0], fmaf(q1.y, h.be[0], q0.y)), h.al[0], fmaf(fmaf(q1.z, h.be[0], q0.z), h.be[0], q0.x));
    const float f1 = fmaf(fmaf(q1.x, h.al[1], fmaf(q1.y, h.be[1], q0.y)), h.al[1], fmaf(fmaf(q1.z, h.be[1], q0.z), h.be[1], q0.x));
    bool hit0 = f0 < -q0.w, hit1 = f1 < -q0.w;
    const bool amb0 = live0 && !(fabsf(f0) > q0.w), amb1 = live1 && !(fabsf(f1) > q0.w);
    if (__any_sync(0xffffffffu, amb0 || amb1)) {
      const int p = __shfl_sync(0xffffffffu, p_lane, t);
      if (amb0) hit0 = hit_exact<REF>(rays_o, rays_d, geom, p, h.pix[0], thr, bound2);
      if (amb1) hit1 = hit_exact<REF>(rays_o, rays_d, geom, p, h.pix[1], thr, bound2);
    }
    const uint32_t b0 = __ballot_sync(0xffffffffu, hit0) & h.act[0], b1 = __ballot_sync(0xffffffffu, hit1) & h.act[1];
    if (lane == t) { m0 = b0; m1 = b1; }
  }
}

struct HitArgs {
  const float* rays_o; const float* rays_d; const float4* geom; int n;
  const int32_t* tile_offsets; const int32_t* tile_len; const int32_t* sorted_prims; int W, H, ntx;
  float thr, bound2, K;            // K <= 0: no quadratic form (thresholds the exponential underflows at)
  const int32_t* active; const int32_t* active_count; int lo, hi;
  const float4* px_state; uint2* masks; uint32_t* pair_base; int32_t* prim_cnt; int32_t* counters; int64_t max_records;
  int32_t* status; int32_t* next_count; int add_tiles;      // add_tiles: a launch for a batch that is not its first
};

// the wave's counters start at zero, and the lists its compositing pass will append to start empty
template <int V>
__device__ __forceinline__ void reset_wave(const Views<HitArgs, V>& b) {
  const HitArgs& a = b.v[0];
  int tiles = a.add_tiles ? a.counters[kCtrWaveTiles] : 0;
  for (int v = 0; v < (V == 1 ? 1 : b.count); ++v) {
    *b.v[v].next_count = 0;
    tiles += *b.v[v].active_count;
  }
  a.counters[kCtrWaveTiles] = tiles;
  a.counters[kCtrWork] = 0; a.counters[kCtrWorkSmall] = 0; a.counters[kCtrWorkNext] = 0; a.counters[kCtrWaveRecords] = 0;
}

__device__ __forceinline__ int warp_inclusive_scan(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  return v;
}

// One warp per (tile, part of its window): every parts-th chunk of 32 candidates, nothing shared between warps; a chunk's
// record slots are one reservation.  The later a wave, the wider its window and the fewer its tiles, so windows of up to
// kHitParts chunks are cut into chunks and longer ones into kHitParts parts (LOOP; registers for the loop would cost the
// others occupancy): a part prepares its tile's rays again, a tenth of a chunk's work.  A warp per tile for windows up to 128
// and a CTA per tile beyond took 72 us of a 60k-primitive 639 x 477 frame and 1,454 of four 1M views at 1920 x 1080, this
// 58 and 1,374.
constexpr int kHitWarps = 4, kHitParts = 8;
template <bool REF, bool LOOP, int V>
__global__ void __launch_bounds__(32 * kHitWarps) k_hits(const __grid_constant__ Views<HitArgs, V> b, int parts) {
  chain_wait();
  chain_release();
  __shared__ float4 s_q[kHitWarps][64];
  const HitArgs& a = b.v[view_of_cta<V>()];
  if (a.status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) reset_wave<V>(b);
  const int lane = threadIdx.x & 31, warp = warp_of_cta(), wpb = blockDim.x >> 5;
  const int units = *a.active_count * parts;
  for (int unit = blockIdx.x * wpb + warp; unit < units; unit += gridDim.x * wpb) {
    const int slot_i = parts == 1 ? unit : unit / parts, part = unit - slot_i * parts;
    const int tile = a.active[slot_i];
    const int s = a.tile_offsets[tile], len = a.tile_len[tile];
    const int wlo = min(a.lo, len), nwin = min(a.hi, len) - wlo;
    if (part * 32 >= nwin) continue;
    const HitPixels h = hit_pixels(a.rays_o, a.rays_d, a.px_state, tile, a.ntx, a.W, a.H, a.K > 0.f);
    int j0 = part * 32;
    do {
      const int j = j0 + lane;
      const size_t pair = (size_t)(s + wlo) + j;
      const int p = j < nwin ? a.sorted_prims[pair] : -1;
      uint32_t m0, m1;
      hit_chunk<REF>(h, a.rays_o, a.rays_d, a.geom, a.n, p, min(32, nwin - j0), a.K, a.thr, a.bound2, s_q[warp], m0, m1);
      const int c = __popc(m0) + __popc(m1);
      if (c > 0) atomicAdd(a.prim_cnt + p, c);
      const int inc = warp_inclusive_scan(c);
      int base = 0;
      if (lane == 31 && inc > 0) {
        base = atomicAdd(a.counters + kCtrRecords, inc);
        if ((int64_t)base + inc > a.max_records) atomicOr(a.status + MLPSP_ST_BITS, MLPSP_ST_RECORD_OVERFLOW);
      }
      base = __shfl_sync(0xffffffffu, base, 31);
      if (j < nwin) {
        a.masks[pair] = make_uint2(m0, m1);
        a.pair_base[pair] = (uint32_t)(base + inc - c);
      }
    } while (LOOP && (j0 += parts * 32) < nwin);
  }
}

static int launch_hits(const HitArgs* args, int views, bool ref_arith, int tiles, int sms, bool idle_tail, cudaStream_t st) {
  const HitArgs& a = args[0];
  const int parts = std::min((a.hi - a.lo + 31) / 32, kHitParts);
  // small images spread their tiles over the SMs one warp at a time
  const int64_t units = (int64_t)tiles * parts;
  const int wpb = units * views >= sms * 2 * kHitWarps ? kHitWarps : 1;
  const dim3 grid((unsigned)std::min<int64_t>((units + wpb - 1) / wpb, idle_tail ? sms : sms * 16)), block(32 * wpb);
  const bool loop = (a.hi - a.lo + 31) / 32 > parts;
  cudaError_t e = cudaSuccess;
  if (views == 1) {
    auto* kernel = ref_arith ? (loop ? k_hits<true, true, 1> : k_hits<true, false, 1>) : (loop ? k_hits<false, true, 1> : k_hits<false, false, 1>);
    e = launch_views<1>(kernel, grid, block, 0, st, args, 1, parts);
  } else {
    constexpr int N = kViewsPerLaunch;
    auto* kernel = ref_arith ? (loop ? k_hits<true, true, N> : k_hits<true, false, N>) : (loop ? k_hits<false, true, N> : k_hits<false, false, N>);
    e = launch_views<N>(kernel, grid, block, 0, st, args, views, parts);
  }
  return cuda_check(e, "hits");
}

// Geometric hit masks of all pairs (no transmittance state): the superset the waves draw from.
__global__ void __launch_bounds__(256) k_hit_masks_all(
    const float* __restrict__ rays_o, const float* __restrict__ rays_d, const float4* __restrict__ geom, int n,
    const int32_t* __restrict__ tile_offsets, const int32_t* __restrict__ sorted_prims, int W, int H, int ntx,
    float thr, float bound2, uint32_t* __restrict__ masks32, int ref_arith, const int32_t* __restrict__ status) {
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int tile = blockIdx.x;
  const int s = tile_offsets[tile];
  const int len = tile_offsets[tile + 1] - s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = warp & 1;
  const TilePix tp = tile_pixel(tile, half * 32 + lane, ntx, W, H);
  V3 o = {0.f, 0.f, 0.f}, d = {0.f, 0.f, 0.f};
  if (tp.valid) { o = load3(rays_o, tp.pix); d = load3(rays_d, tp.pix); }
  for (int i = (warp >> 1); i < len; i += 4) {
    const int p = sorted_prims[s + i];
    bool hit = false;
    if (tp.valid && p >= 0 && p < n) {
      const Geom g = load_geom(geom, p);
      if (!surely_misses(g, o, d, bound2)) {
        Hit h;
        hit = ref_arith ? hit_test_ref(load_geom_ref(geom, p), o, d, thr, h) : hit_test(g, o, d, thr, h);
      }
    }
    const uint32_t m = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) masks32[2 * (size_t)(s + i) + half] = m;
  }
}

// ------------------------------------------------------- per-primitive scan + work items ----
// A primitive's records of the wave become evaluator work items: blocks of 128 rows, and -- when the evaluator has
// a kernel for small groups (split) -- a remainder of at most 32 records becomes an item on a list of its own
// instead of a 128-row block that would be three quarters empty.  (Two small items for a remainder of 33..64
// measured slower than one block.)
__device__ __forceinline__ int items_of(int cnt, int split) {
  if (!split) return (cnt + kRowsPerItem - 1) / kRowsPerItem;
  const int rem = cnt % kRowsPerItem;
  return cnt / kRowsPerItem + (rem > kRowsPerSmallItem ? 1 : 0);
}
__device__ __forceinline__ int small_items_of(int cnt, int split) {
  if (!split) return 0;
  const int rem = cnt % kRowsPerItem;
  return (rem > 0 && rem <= kRowsPerSmallItem) ? 1 : 0;
}

// One launch per wave: every block scans its own 1,024 counts, reserves its share of the wave's record range and work
// lists with one atomic each (their order among the blocks does not matter: a primitive's records only have to be
// contiguous), writes the primitives' first positions and work items, and clears the counts the NEXT wave will add to
// (waves alternate between two count arrays, so nothing this launch reads is written by it).  An exclusive scan over
// the blocks, which this replaces, took two dependent launches (18 -> 8 us per wave at 100,000 primitives).
// fixed (optional): the primitives' first positions are given (records already lie in primitive order).
__global__ void __launch_bounds__(kPrimScanItems / 4) k_prim_alloc(
    const int32_t* __restrict__ prim_cnt, int32_t* __restrict__ prim_cnt_next, const int64_t* __restrict__ fixed, int n, int split,
    int32_t* __restrict__ prim_pos, int4* __restrict__ work, int64_t max_work, int4* __restrict__ work_small,
    int64_t max_work_small, int32_t* __restrict__ counters, int32_t* __restrict__ status) {
  chain_wait();
  chain_release();
  __shared__ int warp_sums[32];
  __shared__ int s_base[3];
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) {
    // after a record overflow, leave the size the wave asked for so the caller can grow its scratch
    if (blockIdx.x == 0 && threadIdx.x == 0 && (status[MLPSP_ST_BITS] & MLPSP_ST_RECORD_OVERFLOW))
      atomicMax(status + MLPSP_ST_WAVE_RECORDS, counters[kCtrRecords]);
    return;
  }
  const int64_t base = (int64_t)blockIdx.x * kPrimScanItems + (int64_t)threadIdx.x * 4;
  int c[4] = {0, 0, 0, 0}, a = 0, b = 0, m = 0;
  if (fixed) {
#pragma unroll
    for (int j = 0; j < 4; ++j) if (base + j < n) c[j] = (int)(fixed[base + j + 1] - fixed[base + j]);
  } else if (base < n) {     // both count arrays start 16-byte aligned and are padded to a multiple of four
    const int4 v = *reinterpret_cast<const int4*>(prim_cnt + base);
    c[0] = v.x; c[1] = base + 1 < n ? v.y : 0; c[2] = base + 2 < n ? v.z : 0; c[3] = base + 3 < n ? v.w : 0;
    *reinterpret_cast<int4*>(prim_cnt_next + base) = make_int4(0, 0, 0, 0);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) { a += c[j]; b += items_of(c[j], split); m += small_items_of(c[j], split); }
  int ta, tb, tm = 0;
  int ea = block_exclusive_scan(a, warp_sums, ta);
  if (ta == 0) {           // no records here: positions that nobody will use
    return;
  }
  int eb = block_exclusive_scan(b, warp_sums, tb);
  int em = split ? block_exclusive_scan(m, warp_sums, tm) : 0;
  if (threadIdx.x == 0) {
    const int r0 = atomicAdd(counters + kCtrWaveRecords, ta);
    // both work lists in one 64-bit word, so that the last block to come sees the totals of both
    const unsigned long long w0 = atomicAdd(reinterpret_cast<unsigned long long*>(counters + kCtrWork),
                                            (unsigned long long)(uint32_t)tb | ((unsigned long long)(uint32_t)tm << 32));
    s_base[0] = r0;
    s_base[1] = (int)(uint32_t)w0;
    s_base[2] = (int)(w0 >> 32);
    if ((int64_t)s_base[1] + tb > max_work || (int64_t)s_base[2] + tm > max_work_small)
      atomicOr(status + MLPSP_ST_BITS, MLPSP_ST_RECORD_OVERFLOW);
    atomicAdd((unsigned long long*)(status + MLPSP_ST_RECORDS_LO), (unsigned long long)ta);
    atomicMax(status + MLPSP_ST_WAVE_RECORDS, r0 + ta);
    atomicMax(status + MLPSP_ST_WORK_ITEMS, s_base[1] + tb + s_base[2] + tm);
    if (tb + tm) atomicAdd(status + MLPSP_ST_WORK_TOTAL, tb + tm);
    if (tm) atomicAdd(status + MLPSP_ST_WORK_SMALL, tm);
    if (r0 == 0) {
      atomicAdd(status + MLPSP_ST_WAVES, 1);
      status[MLPSP_ST_LAST_TILES] = counters[kCtrWaveTiles];
    }
  }
  __syncthreads();
  ea += s_base[0]; eb += s_base[1]; em += s_base[2];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (c[j] > 0) {
      const int first = fixed ? (int)fixed[base + j] : ea;
      if (prim_pos) prim_pos[base + j] = first;
      const int it = items_of(c[j], split);
      for (int q = 0; q < it; ++q)
        if ((int64_t)eb + q < max_work)
          work[eb + q] = make_int4((int)(base + j), first + q * kRowsPerItem, min(kRowsPerItem, c[j] - q * kRowsPerItem), 0);
      if (small_items_of(c[j], split)) {                      // the remainder starts behind the full blocks
        const int rem = c[j] % kRowsPerItem;
        if ((int64_t)em < max_work_small) work_small[em] = make_int4((int)(base + j), first + c[j] - rem, rem, 0);
        ++em;
      }
      ea += c[j]; eb += it;
    }
  }
}

int launch_prim_scan(const Scratch& s, int n, const int64_t* fixed, int32_t* status, cudaStream_t st, bool split_small, int wave) {
  const int nblk = (n + kPrimScanItems - 1) / kPrimScanItems;
  if (nblk == 0) return MLPSP_OK;
  LaunchScope scope(kKScan, 1, st);
  const int split = split_small && s.work_small ? 1 : 0;
  int32_t* cnt = s.prim_cnt + (size_t)(wave & 1) * prim_cnt_stride(n);
  int32_t* cnt_next = s.prim_cnt + (size_t)((wave & 1) ^ 1) * prim_cnt_stride(n);
  return cuda_check(launch_chained(k_prim_alloc, dim3(nblk), dim3(kPrimScanItems / 4), 0, st, cnt, cnt_next, fixed, n, split, s.prim_pos, s.work,
                                   s.max_work, s.work_small, s.max_work_small, s.counters, status),
                    "prim_scan");
}

// -------------------------------------------------------------------------- fill pass ----
// Feature gates (semantic_tetra_gates, np_tile_kernels.cu:97-124).  What depends on the primitive alone, the reciprocals
// of beta * scale + 1e-6, is a function of its own: the fill pass prepares it once per candidate.
__device__ __forceinline__ V3 gate_scales(const float4 ls, float beta) {
  return {1.f / (beta * det_exp(ls.x) + 1e-6f), 1.f / (beta * det_exp(ls.y) + 1e-6f), 1.f / (beta * det_exp(ls.z) + 1e-6f)};
}
__device__ __forceinline__ float4 tetra_gates(const Hit& h, V3 inv_s, float tau) {
  const float ux = fminf(1.f, fmaxf(-1.f, h.qx * inv_s.x));
  const float uy = fminf(1.f, fmaxf(-1.f, h.qy * inv_s.y));
  const float uz = fminf(1.f, fmaxf(-1.f, h.qz * inv_s.z));
  const float l0 = tau * (ux + uy + uz), l1 = tau * (ux - uy - uz);
  const float l2 = tau * (-ux + uy - uz), l3 = tau * (-ux - uy + uz);
  const float lm = fmaxf(fmaxf(l0, l1), fmaxf(l2, l3));
  const float e0 = __expf(l0 - lm), e1 = __expf(l1 - lm), e2 = __expf(l2 - lm), e3 = __expf(l3 - lm);
  const float inv = __fdividef(1.f, fmaxf(e0 + e1 + e2 + e3, 1e-8f));
  return make_float4(e0 * inv, e1 * inv, e2 * inv, e3 * inv);
}

// Transpose of the 32 x 32 bit matrix whose row l is lane l's word.
__device__ __forceinline__ uint32_t transpose32(uint32_t w) {
  const int lane = threadIdx.x & 31;
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int s = 16; s; s >>= 1) {
    const uint32_t other = __shfl_xor_sync(0xffffffffu, w, s);
    w = (lane & s) ? (w & ~m) | ((other & ~m) >> s) : (w & m) | ((other & m) << s);
    m ^= m << (s >> 1);
  }
  return w;
}

// One warp per chunk of 32 candidates of an active tile; nothing is shared between warps.  A candidate's lane reserves its
// records' primitive-major range (one atomic per pair with a hit) and prepares its geometry once: rotation, M R^T v and v
// for the tile's common origin.  The records of the chunk are then listed (pixel lanes walk their own hits, as in
// compositing: the masks transposed) and dealt to the lanes, so every lane computes a record whatever the hits' pattern,
// and neighbouring lanes write neighbouring records.  About 100 instructions per record where a search for the record's
// pair and pixel, and the full geometry per record, took 350 (100k frame, 10.6 M records: 193 -> 135 us).
// MODE 0: values only (no decision hangs on them: hardware reciprocal and exponential); 1: hit_test's own values, for the
// feature gates, which divide the local offset by the scales, and for per-pixel ordering, which sorts by t (geometry and
// gate scales staged per candidate as well: 270 -> 208 us of a 250k feature frame); 2: the
// reference kernels' arithmetic.
constexpr int kFillWarps = 8;
struct FillSmem { float4 geo[32][5]; float4 ray[32]; uint16_t list[1024]; };

struct FillArgs {
  const float* rays_o; const float* rays_d; const float4* geom;
  const int32_t* tile_offsets; const int32_t* tile_len; const int32_t* sorted_prims; int W, H, ntx; float thr;
  const int32_t* active; const int32_t* active_count; int lo, hi;
  const uint2* masks; const uint32_t* pair_base; int32_t* prim_pos; float4* rec_in; float* rec_t; float4* rec_gate;
  float beta, tau; int plain, table; const int32_t* status;      // plain: MODE 0 without the shared per-candidate geometry; table: see below
  int width, chunks, halves;                              // candidates per unit, units per window and half, 2: a unit is one half
};

template <int MODE, int V>
__global__ void __launch_bounds__(32 * kFillWarps, 4) k_fill(const __grid_constant__ Views<FillArgs, V> b) {
  chain_wait();
  chain_release();
  __shared__ FillSmem s_all[kFillWarps];
  const FillArgs& a = b.v[view_of_cta<V>()];
  if (a.status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int lane = threadIdx.x & 31, warp = warp_of_cta(), wpb = blockDim.x >> 5;
  FillSmem& sm = s_all[warp];
  const uint32_t lt = (1u << lane) - 1u;
  const int per_tile = a.chunks * a.halves, units = *a.active_count * per_tile;
  for (int unit = blockIdx.x * wpb + warp; unit < units; unit += gridDim.x * wpb) {
    const int slot_i = per_tile == 1 ? unit : unit / per_tile;
    const int part = unit - slot_i * per_tile, ch = a.halves == 2 ? part >> 1 : part;
    const int h0 = a.halves == 2 ? part & 1 : 0, h1 = a.halves == 2 ? h0 + 1 : 2;
    const int tile = a.active[slot_i];
    const int s = a.tile_offsets[tile], len = a.tile_len[tile];
    const int j0 = min(a.lo, len) + ch * a.width, whi = min(min(a.hi, len), j0 + a.width);
    if (j0 >= whi) continue;
    uint2 m = make_uint2(0u, 0u);
    int p = 0, c = 0, q0 = 0;
    uint32_t first = 0u;
    if (j0 + lane < whi) {
      m = a.masks[(size_t)s + j0 + lane];
      first = a.pair_base[(size_t)s + j0 + lane];
      c = (h0 == 0 ? __popc(m.x) : 0) + (h1 == 2 ? __popc(m.y) : 0);
      if (c > 0) {
        p = a.sorted_prims[s + j0 + lane];
        q0 = atomicAdd(a.prim_pos + p, c);
      }
    }
    if (!__any_sync(0xffffffffu, c > 0)) continue;
    // rays of the tile's two halves; one origin is the usual case
    V3 o[2], d[2];
    bool same = true;
    V3 o0 = {0.f, 0.f, 0.f};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const TilePix tp = tile_pixel(tile, h * 32 + lane, a.ntx, a.W, a.H);
      o[h] = d[h] = V3{0.f, 0.f, 0.f};
      if (tp.valid) { o[h] = load3(a.rays_o, tp.pix); d[h] = load3(a.rays_d, tp.pix); }
      if (h == 0) o0 = V3{__shfl_sync(0xffffffffu, o[0].x, 0), __shfl_sync(0xffffffffu, o[0].y, 0), __shfl_sync(0xffffffffu, o[0].z, 0)};
      same = same && (!tp.valid || (o[h].x == o0.x && o[h].y == o0.y && o[h].z == o0.z));
    }
    const bool uni = MODE != 2 && !(MODE == 0 && a.plain) && __all_sync(0xffffffffu, same);
    __syncwarp();
    if (MODE == 1 && c > 0) {
      // centre, quaternion, scales and, for a common origin, the local offset: hit_test's operands, so its bits
      const Geom g = load_geom(a.geom, p);
      const V3 vl = local_offset(g, o0);
      V3 is = {0.f, 0.f, 0.f};
      if (a.rec_gate) is = gate_scales(__ldg(a.geom + (size_t)p * 4 + 3), a.beta);
      sm.geo[lane][0] = make_float4(g.cx, g.cy, g.cz, g.qw);
      sm.geo[lane][1] = make_float4(g.qx, g.qy, g.qz, vl.x);
      sm.geo[lane][2] = make_float4(vl.y, vl.z, is.x, is.y);
      sm.geo[lane][3] = make_float4(g.mx, g.my, g.mz, 0.f);
      sm.geo[lane][4] = make_float4(is.z, 0.f, 0.f, 0.f);
    }
    if (MODE == 0 && uni && c > 0) {
      const Geom g = load_geom(a.geom, p);
      // rows of R^T: R^T applied to the axes gives its columns
      const V3 c0 = rot_conj_fast(g.qw, g.qx, g.qy, g.qz, V3{1.f, 0.f, 0.f}), c1 = rot_conj_fast(g.qw, g.qx, g.qy, g.qz, V3{0.f, 1.f, 0.f}),
               c2 = rot_conj_fast(g.qw, g.qx, g.qy, g.qz, V3{0.f, 0.f, 1.f});
      const V3 v = {g.cx - o0.x, g.cy - o0.y, g.cz - o0.z};
      const V3 vl = rot_conj_fast(g.qw, g.qx, g.qy, g.qz, v);
      sm.geo[lane][0] = make_float4(c0.x, c1.x, c2.x, vl.x * g.mx);
      sm.geo[lane][1] = make_float4(c0.y, c1.y, c2.y, vl.y * g.my);
      sm.geo[lane][2] = make_float4(c0.z, c1.z, c2.z, vl.z * g.mz);
      sm.geo[lane][3] = make_float4(g.mx, g.my, g.mz, 0.f);
      sm.geo[lane][4] = make_float4(v.x, v.y, v.z, 0.f);
    }
    int before = 0;                                       // this unit's records of the candidate in the first half
    for (int h = h0; h < h1; ++h) {
      const uint32_t mine = h ? m.y : m.x;
      const int inc = warp_inclusive_scan(__popc(mine));
      const int total = __shfl_sync(0xffffffffu, inc, 31), pref = inc - __popc(mine);
      if (total == 0) continue;
      // positions of this half's records behind the entries of the list
      __syncwarp();
      sm.geo[lane][3].w = __int_as_float(q0 + before - pref);
      sm.geo[lane][4].w = __int_as_float((int)first + (h ? __popc(m.x) : 0) - pref);
      before += __popc(mine);
      const V3 dh = h ? d[1] : d[0], oh = h ? o[1] : o[0];
      sm.ray[lane] = make_float4(dh.x, dh.y, dh.z, 0.f);
      uint32_t todo = transpose32(mine);
      while (__any_sync(0xffffffffu, todo != 0u)) {
        const int j = todo ? __ffs(todo) - 1 : lane;
        const uint32_t mj = __shfl_sync(0xffffffffu, mine, j);
        const int pj = __shfl_sync(0xffffffffu, pref, j);
        if (todo) sm.list[pj + __popc(mj & lt)] = (uint16_t)(j | (lane << 5));
        todo &= todo - 1u;
      }
      __syncwarp();
      for (int r = lane; r - lane < total; r += 32) {
        const bool on = r < total;
        const int e = on ? sm.list[r] : 0;
        const int j = e & 31, px = e >> 5;
        V3 oo = o0;
        int pj = 0;
        if (!uni) {        // a warp-wide exchange, so before the lanes part
          oo = V3{__shfl_sync(0xffffffffu, oh.x, px), __shfl_sync(0xffffffffu, oh.y, px), __shfl_sync(0xffffffffu, oh.z, px)};
          pj = __shfl_sync(0xffffffffu, p, j);
        }
        if (!on) continue;
        const float4 ray = sm.ray[px];
        const float4 g3 = sm.geo[j][3], g4 = sm.geo[j][4];
        const int pos = __float_as_int(g3.w) + r;
        const uint32_t slot = (uint32_t)(__float_as_int(g4.w) + r);
        Hit ht;
        V3 is = {0.f, 0.f, 0.f};
        if (MODE == 0 && uni) {
          const float4 g0 = sm.geo[j][0], g1 = sm.geo[j][1], g2 = sm.geo[j][2];
          const float lx = g0.x * ray.x + g0.y * ray.y + g0.z * ray.z, ly = g1.x * ray.x + g1.y * ray.y + g1.z * ray.z,
                      lz = g2.x * ray.x + g2.y * ray.y + g2.z * ray.z;
          const float denom = lx * lx * g3.x + ly * ly * g3.y + lz * lz * g3.z;
          const float numer = lx * g0.w + ly * g1.w + lz * g2.w;
          ht.t = __fdividef(numer, denom);
          ht.dx = g4.x - ht.t * ray.x; ht.dy = g4.y - ht.t * ray.y; ht.dz = g4.z - ht.t * ray.z;
          const float qx = g0.x * ht.dx + g0.y * ht.dy + g0.z * ht.dz, qy = g1.x * ht.dx + g1.y * ht.dy + g1.z * ht.dz,
                      qz = g2.x * ht.dx + g2.y * ht.dy + g2.z * ht.dz;
          ht.decay = __expf(-0.5f * (qx * qx * g3.x + qy * qy * g3.y + qz * qz * g3.z));
        } else {
          const V3 dd = {ray.x, ray.y, ray.z};
          if (MODE == 2) hit_test_ref(load_geom_ref(a.geom, pj), oo, dd, a.thr, ht);
          else if (MODE == 1) {
            const float4 g0 = sm.geo[j][0], g1 = sm.geo[j][1], g2 = sm.geo[j][2];
            Geom g;
            g.cx = g0.x; g.cy = g0.y; g.cz = g0.z; g.qw = g0.w; g.qx = g1.x; g.qy = g1.y; g.qz = g1.z;
            g.mx = g3.x; g.my = g3.y; g.mz = g3.z; g.smax = 0.f;
            is = V3{g2.z, g2.w, g4.x};
            if (uni) hit_test_t<true>(g, oo, dd, V3{g1.w, g2.x, g2.y}, a.thr, ht);
            else hit_test(g, oo, dd, a.thr, ht);
          } else hit_values_fast(load_geom(a.geom, pj), oo, dd, ht);
        }
        // the record's 32 bytes in one store: a full sector.  (direction, offset, decay, slot), or, for an evaluator that
        // looks the encoded direction up (table), (offset, decay, slot, pixel)
        const float sl = __uint_as_float(slot), pixel = __uint_as_float((uint32_t)(tile * 64 + h * 32 + px));
        float v[8] = {ray.x, ray.y, ray.z, ht.dx, ht.dy, ht.dz, ht.decay, sl};
        if (a.table) { v[0] = ht.dx; v[1] = ht.dy; v[2] = ht.dz; v[3] = ht.decay; v[4] = sl; v[5] = pixel; }
        asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(a.rec_in + 2 * (size_t)pos), "f"(v[0]), "f"(v[1]),
                     "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
        if (a.rec_t) a.rec_t[slot] = ht.t;
        if (MODE != 0 && a.rec_gate) {
          if (MODE == 2) is = gate_scales(__ldg(a.geom + (size_t)pj * 4 + 3), a.beta);
          a.rec_gate[slot] = tetra_gates(ht, is, a.tau);
        }
      }
      __syncwarp();
    }
  }
}

static int launch_fill(FillArgs* args, int views, bool exact, bool ref_arith, int tiles, int sms, bool idle_tail, cudaStream_t st) {
  // 16 candidates per warp balance best on large frames (32: 957, 16: 939, 8: 1,000 us for the whole 100k frame); with few
  // tiles the window is cut finer, so that the SMs get more and shorter warps
  const int window = args[0].hi - args[0].lo;
  const bool small = (int64_t)tiles * views * ((window + 15) / 16) < (int64_t)sms * 8;
  const int width = small ? 8 : 16, halves = small ? 2 : 1, chunks = (window + width - 1) / width;
  for (int v = 0; v < views; ++v) { args[v].width = width; args[v].halves = halves; args[v].chunks = chunks; }
  const int64_t units = (int64_t)tiles * chunks * halves;
  const int wpb = units * views >= sms * 2 * kFillWarps ? kFillWarps : 1;
  const dim3 grid((unsigned)std::min<int64_t>((units + wpb - 1) / wpb, idle_tail ? sms : sms * 32)), block(32 * wpb);
  cudaError_t e = cudaSuccess;
  if (views == 1) {
    e = launch_views<1>(ref_arith ? k_fill<2, 1> : (exact ? k_fill<1, 1> : k_fill<0, 1>), grid, block, 0, st, args, 1);
  } else {
    constexpr int N = kViewsPerLaunch;
    e = launch_views<N>(ref_arith ? k_fill<2, N> : (exact ? k_fill<1, N> : k_fill<0, N>), grid, block, 0, st, args, views);
  }
  return cuda_check(e, "fill");
}

// --------------------------------------------------------------------------- composite ----
// 64 threads per tile; each warp owns 32 pixels and stops as soon as none of them is live.
struct PrimStats {
  const float* gt_rgb; const int32_t* sorted_prims;
  float* sum_w; float* max_w; int32_t* hits; float* sum_werr; int32_t* contrib;
};

struct CompositeArgs {
  PrimStats ps;
  const int32_t* tile_offsets; const int32_t* tile_len; int W, H, ntx; const int32_t* active; const int32_t* active_count; int lo, hi;
  const uint32_t* masks32; const uint32_t* pair_base; const float4* rec_out; const float* rec_t; float4* px_state; float2* px_depth;
  float* rgb; float* alpha; float* depth_t; uint32_t* mask_used32; float* rec_w; float* rec_tr; float bgr, bgg, bgb; int has_bg;
  int32_t* next_active; int32_t* next_count; int32_t* status;
};

template <bool STATS, int V>
__global__ void __launch_bounds__(64) k_composite(const __grid_constant__ Views<CompositeArgs, V> views) {
  chain_wait();
  chain_release();
  const CompositeArgs& a = views.v[view_of_cta<V>()];
  const PrimStats& ps = a.ps;
  const int32_t* __restrict__ tile_offsets = a.tile_offsets; const int32_t* __restrict__ tile_len = a.tile_len;
  const int W = a.W, H = a.H, ntx = a.ntx, lo = a.lo, hi = a.hi, has_bg = a.has_bg;
  const int32_t* __restrict__ active = a.active; const int32_t* __restrict__ active_count = a.active_count;
  const uint32_t* __restrict__ masks32 = a.masks32; const uint32_t* __restrict__ pair_base = a.pair_base;
  const float4* __restrict__ rec_out = a.rec_out; const float* __restrict__ rec_t = a.rec_t;
  float4* __restrict__ px_state = a.px_state; float2* __restrict__ px_depth = a.px_depth;
  float* __restrict__ rgb = a.rgb; float* __restrict__ alpha = a.alpha; float* __restrict__ depth_t = a.depth_t;
  uint32_t* __restrict__ mask_used32 = a.mask_used32; float* __restrict__ rec_w = a.rec_w; float* __restrict__ rec_tr = a.rec_tr;
  const float bgr = a.bgr, bgg = a.bgg, bgb = a.bgb;
  int32_t* __restrict__ next_active = a.next_active; int32_t* __restrict__ next_count = a.next_count; int32_t* __restrict__ status = a.status;
  __shared__ int s_live[2];
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int n_active = *active_count;
  for (int slot_i = blockIdx.x; slot_i < n_active; slot_i += gridDim.x) {
  const int tile = active[slot_i];
  const int s = tile_offsets[tile];
  const int len = tile_len[tile];
  const int wlo = min(lo, len), whi = min(hi, len);
  const int lane = threadIdx.x & 31, half = warp_of_cta();
  const TilePix tp = tile_pixel(tile, half * 32 + lane, ntx, W, H);
  float4 st = make_float4(0.f, 0.f, 0.f, 0.f);
  float2 dp = make_float2(0.f, 0.f);
  if (tp.valid) { st = px_state[tp.pix]; if (depth_t) dp = px_depth[tp.pix]; }
  bool act = tp.valid && st.w >= MLPSP_TERM;
  const uint32_t lt = (1u << lane) - 1u;
  int used = 0;
  float gtr = 0.f, gtg = 0.f, gtb = 0.f;
  if (STATS && tp.valid) { gtr = ps.gt_rgb[(size_t)tp.pix * 3]; gtg = ps.gt_rgb[(size_t)tp.pix * 3 + 1]; gtb = ps.gt_rgb[(size_t)tp.pix * 3 + 2]; }
  if (!STATS) {
    for (int i0 = wlo; i0 < whi && __any_sync(0xffffffffu, act); i0 += 32) {
      const int idx = i0 + lane;
      uint32_t mine = 0u, first = 0u;       // pair i0 + lane: this half's hit mask and the slot of its first record
      if (idx < whi) {
        const uint2 mm = *reinterpret_cast<const uint2*>(masks32 + 2 * (size_t)(s + idx));
        mine = half ? mm.y : mm.x;
        first = pair_base[s + idx] + (half ? __popc(mm.x) : 0);
      }
      // A pixel meets about one candidate in eight, so every lane walks its own hits (bit j of todo: pair i0 + j) instead of
      // the warp walking the pairs: four of a lane's records are requested at a time, whether its pixel will still be live or
      // not, then blended in list order.
      uint32_t todo = transpose32(mine), taken = 0u;
      if (!act) todo = 0u;
      while (__any_sync(0xffffffffu, todo != 0u)) {
        float4 rr[4];
        uint32_t slot4[4], bit4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = todo ? __ffs(todo) - 1 : lane;
          bit4[u] = todo & (0u - todo);
          todo &= todo - 1u;
          const uint32_t mj = __shfl_sync(0xffffffffu, mine, j), fj = __shfl_sync(0xffffffffu, first, j);
          slot4[u] = fj + __popc(mj & lt);
          rr[u] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (bit4[u]) rr[u] = rec_out[slot4[u]];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool take = act && bit4[u];
          if (take) {
            const float4 r = rr[u];
            const float w = st.w * r.w;
            st.x = fmaf(w, r.x, st.x); st.y = fmaf(w, r.y, st.y); st.z = fmaf(w, r.z, st.z);
            if (depth_t) { dp.x = fmaf(w, rec_t[slot4[u]], dp.x); dp.y += w; }
            if (rec_w) rec_w[slot4[u]] = w;
            if (rec_tr) rec_tr[slot4[u]] = st.w;
            st.w *= (1.f - r.w);
            act = st.w >= MLPSP_TERM;
            taken |= bit4[u];
          }
        }
        if (!act) todo = 0u;
      }
      used += __popc(taken);
      if (mask_used32) {
        const uint32_t um = transpose32(taken);
        if (um) mask_used32[2 * (size_t)(s + idx) + half] = um;
      }
    }
    used = __reduce_add_sync(0xffffffffu, used);
  } else {
    // statistics: the warp walks the pairs together, so that a pair's contributions are summed before they go to memory
    for (int i0 = wlo; i0 < whi && __any_sync(0xffffffffu, act); i0 += 32) {
      const int idx = i0 + lane;
      uint2 mm = make_uint2(0u, 0u);
      uint32_t bb = 0;
      if (idx < whi) {
        mm = *reinterpret_cast<const uint2*>(masks32 + 2 * (size_t)(s + idx));
        bb = pair_base[s + idx];
      }
      const int cnt = min(32, whi - i0);
      bool stop = false;
      // four pairs at a time: the records a lane may need are requested first (whether its pixel is still live or
      // not), then blended in list order, so the gathers of a batch overlap instead of forming a chain
      for (int j0 = 0; j0 < cnt && !stop; j0 += 4) {
        float4 rr[4];
        uint32_t slot4[4], mine4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = min(j0 + u, 31);
          const uint32_t m0 = __shfl_sync(0xffffffffu, mm.x, j), m1 = __shfl_sync(0xffffffffu, mm.y, j);
          const uint32_t b = __shfl_sync(0xffffffffu, bb, j);
          const uint32_t mine = (j0 + u < cnt) ? (half ? m1 : m0) : 0u;
          mine4[u] = mine;
          slot4[u] = b + (half ? __popc(m0) : 0) + __popc(mine & lt);
          rr[u] = make_float4(0.f, 0.f, 0.f, 0.f);
          if ((mine >> lane) & 1u) rr[u] = rec_out[slot4[u]];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = j0 + u;
          const uint32_t mine = mine4[u];
          if (stop || mine == 0u) continue;
          const bool take = act && ((mine >> lane) & 1u);
          float sw = 0.f, swerr = 0.f;
          if (take) {
            const uint32_t slot = slot4[u];
            const float4 r = rr[u];
            const float w = st.w * r.w;
            st.x = fmaf(w, r.x, st.x); st.y = fmaf(w, r.y, st.y); st.z = fmaf(w, r.z, st.z);
            sw = w;
            if (w > 1e-1f) swerr = w * (fabsf(st.x - gtr) + fabsf(st.y - gtg) + fabsf(st.z - gtb));
            if (depth_t) { dp.x = fmaf(w, rec_t[slot], dp.x); dp.y += w; }
            if (rec_w) rec_w[slot] = w;
            if (rec_tr) rec_tr[slot] = st.w;
            st.w *= (1.f - r.w);
            act = st.w >= MLPSP_TERM;
          }
          const uint32_t um = __ballot_sync(0xffffffffu, take);
          if (um) {
            // this half-tile's share of the pair's statistics: one atomic per array
            const int n_hit = __popc(__ballot_sync(0xffffffffu, sw > 1e-8f));
            const int n_con = __popc(__ballot_sync(0xffffffffu, sw > 1e-1f));
            float tsum = sw, tmax = sw, terr = swerr;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
              tsum += __shfl_xor_sync(0xffffffffu, tsum, o);
              tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
              terr += __shfl_xor_sync(0xffffffffu, terr, o);
            }
            if (lane == 0) {
              const int p = ps.sorted_prims[s + i0 + j];
              atomicAdd(ps.sum_w + p, tsum);
              atomicMax(reinterpret_cast<int*>(ps.max_w + p), __float_as_int(tmax));   // w >= 0: bit order = value order
              if (n_hit) atomicAdd(ps.hits + p, n_hit);
              if (n_con) { atomicAdd(ps.contrib + p, n_con); atomicAdd(ps.sum_werr + p, terr); }
            }
          }
          if (um) {
            if (lane == 0) { used += __popc(um); if (mask_used32) mask_used32[2 * (size_t)(s + i0 + j) + half] = um; }
            if (!__any_sync(0xffffffffu, act)) stop = true;
          }
        }
      }
    }
  }
  if (tp.valid) {
    px_state[tp.pix] = st;
    const float a = 1.f - st.w;
    float r = st.x, g = st.y, b = st.z;
    if (has_bg) {
      const float k = fminf(fmaxf(1.f - a, 0.f), 1.f);
      r += k * bgr; g += k * bgg; b += k * bgb;
    }
    rgb[(size_t)tp.pix * 3] = r; rgb[(size_t)tp.pix * 3 + 1] = g; rgb[(size_t)tp.pix * 3 + 2] = b;
    alpha[tp.pix] = a;
    if (depth_t) { px_depth[tp.pix] = dp; depth_t[tp.pix] = dp.x / ((dp.y > 1e-8f) ? dp.y : 1.f); }
  }
  const bool live = __any_sync(0xffffffffu, act);
  if (lane == 0) {
    s_live[half] = live;
    if (used) atomicAdd((unsigned long long*)(status + MLPSP_ST_USED_LO), (unsigned long long)used);
  }
  __syncthreads();
  if (threadIdx.x == 0 && (s_live[0] | s_live[1]) && whi < len) next_active[atomicAdd(next_count, 1)] = tile;
  __syncthreads();
  }
}

// --------------------------------------------------------------- per-pixel exact ordering ----
// render_tiles_kernel_with_sort (np_tile_kernels.cu:714-926): every pixel sorts its own hits by its own hit
// distance and blends them front to back.  Here the hits of all pixels have been found and evaluated in one
// wave (no pixel is gated by transmittance, as the order is not known yet); a thread per pixel collects its
// (t, record slot) pairs in list order -- at most kPixelHits, one more raises MLPSP_ST_PIXEL_HITS and the pixel
// blends what it has, as the reference's kernel does before its wrapper raises -- sorts them with the
// reference's stable insertion sort (ties keep list order) and blends until the transmittance falls below 1e-3.
// With a feature map (render_tiles_kernel_with_sort_and_feat) the consumed records and their weights are left for
// k_feature_composite, whose sum does not depend on the order.
constexpr int kPixelHits = 256;
__global__ void __launch_bounds__(64) k_composite_per_pixel(
    const int32_t* __restrict__ tile_offsets, const int32_t* __restrict__ tile_len, int T, int W, int H, int ntx,
    const uint32_t* __restrict__ masks32, const uint32_t* __restrict__ pair_base, const float4* __restrict__ rec_out,
    const float* __restrict__ rec_t, float* __restrict__ rgb, float* __restrict__ alpha, float bgr, float bgg, float bgb,
    int has_bg, uint32_t* __restrict__ used32, float* __restrict__ rec_w, int32_t* __restrict__ status) {
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int lane = threadIdx.x & 31, half = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  for (int tile = blockIdx.x; tile < T; tile += gridDim.x) {
    const int s = tile_offsets[tile], len = tile_len[tile];
    const TilePix tp = tile_pixel(tile, half * 32 + lane, ntx, W, H);
    float key[kPixelHits];
    uint32_t slot[kPixelHits];
    uint16_t pair[kPixelHits];               // position in the tile's list (< 2048), for the consumed masks
    int cnt = 0;
    bool over = false;
    int used = 0;
    for (int i = 0; i < len && !over; ++i) {
      const uint32_t m0 = masks32[2 * (size_t)(s + i)], m1 = masks32[2 * (size_t)(s + i) + 1];
      const uint32_t mine = half ? m1 : m0;
      if (tp.valid && ((mine >> lane) & 1u)) {
        if (cnt < kPixelHits) {
          const uint32_t sl = pair_base[s + i] + (half ? __popc(m0) : 0) + __popc(mine & lt);
          key[cnt] = rec_t[sl];
          slot[cnt] = sl;
          pair[cnt] = (uint16_t)i;
          ++cnt;
        } else {
          over = true;
        }
      }
    }
    if (over) atomicOr(status + MLPSP_ST_BITS, MLPSP_ST_PIXEL_HITS);
    for (int i = 1; i < cnt; ++i) {
      const float kt = key[i];
      const uint32_t ks = slot[i];
      const uint16_t kp = pair[i];
      int j = i - 1;
      while (j >= 0 && key[j] > kt) { key[j + 1] = key[j]; slot[j + 1] = slot[j]; pair[j + 1] = pair[j]; --j; }
      key[j + 1] = kt;
      slot[j + 1] = ks;
      pair[j + 1] = kp;
    }
    float cr = 0.f, cg = 0.f, cb = 0.f, trans = 1.f;
    for (int i = 0; i < cnt; ++i) {
      const float4 r = rec_out[slot[i]];
      const float w = trans * r.w;
      cr = fmaf(w, r.x, cr); cg = fmaf(w, r.y, cg); cb = fmaf(w, r.z, cb);
      if (rec_w) {
        // the feature pass adds w * (gated attributes) for every consumed record, whatever their order
        rec_w[slot[i]] = w;
        atomicOr(used32 + 2 * (size_t)(s + pair[i]) + half, 1u << lane);
      }
      trans *= (1.f - r.w);
      ++used;
      if (trans < MLPSP_TERM) break;
    }
    if (tp.valid) {
      const float a = 1.f - trans;
      if (has_bg) {
        const float k = fminf(fmaxf(1.f - a, 0.f), 1.f);
        cr += k * bgr; cg += k * bgg; cb += k * bgb;
      }
      rgb[(size_t)tp.pix * 3] = cr; rgb[(size_t)tp.pix * 3 + 1] = cg; rgb[(size_t)tp.pix * 3 + 2] = cb;
      alpha[tp.pix] = a;
    }
    for (int o = 16; o > 0; o >>= 1) used += __shfl_xor_sync(0xffffffffu, used, o);
    if (lane == 0 && used) atomicAdd((unsigned long long*)(status + MLPSP_ST_USED_LO), (unsigned long long)used);
  }
}

// ------------------------------------------------------------------- feature compositing ----
// out_feat[pix, :] = sum over the pixel's composited records of w * mix(p, gates)  with
//   S = 4: mix = sum_s g_s * attr[p, s, :]      S = 5: mix = attr[p, 0, :] + sum_s g_s * attr[p, 1+s, :]
//   S = 1: mix = attr[p, 0, :]                                     (np_tile_kernels.cu:6036-6075)
// One CTA per tile after the last wave.  The 64 x C accumulator tile lives in shared memory; for
// every pair that composited at least one record, the consumed pixels and their coefficients
// w * g_s are compacted into shared memory and every thread adds its channels' contribution.
constexpr int kFeatThreads = 256;
constexpr int kFeatBatch = 256;    // consumed records staged per barrier (one per thread)
constexpr int kFeatChan = 256;     // channels per CTA: (tile, channel block) pairs make the grid

// Shared memory: [64][CB] accumulators, then the tile's consumed masks and their record prefix.
template <bool VEC4>
__global__ void __launch_bounds__(kFeatThreads) k_feature_composite(
    const int32_t* __restrict__ tile_offsets, const int32_t* __restrict__ tile_len, const int32_t* __restrict__ sorted_prims, int W, int H, int ntx,
    const uint32_t* __restrict__ used32, const uint32_t* __restrict__ masks32, const uint32_t* __restrict__ pair_base,
    const float* __restrict__ rec_w, const float4* __restrict__ rec_gate, const float* __restrict__ feat_attr,
    int S, int C, int CB, float* __restrict__ out_feat, const int32_t* __restrict__ status) {
  extern __shared__ float s_acc[];                 // [64][CB]
  __shared__ uint32_t s_u[2][kWinMax];             // consumed masks of the tile's pairs
  __shared__ int32_t s_pref[kWinMax + 1];          // records before pair i
  __shared__ __align__(16) float s_cw[kFeatBatch][8];   // per staged record: base weight + 4 gated weights (+ padding)
  __shared__ int s_px[kFeatBatch];                 // its pixel
  __shared__ int s_pr[kFeatBatch];                 // its primitive
  __shared__ int s_run[kFeatBatch + 1];            // first staged record of every run of equal primitives
  __shared__ int s_nruns;
  __shared__ int warp_sums[32];
  if (status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int tile = blockIdx.x, c0 = blockIdx.y * CB;
  const int nc = min(CB, C - c0);
  // VEC4 (launched for maps of at least 256 channels, a multiple of 4): full 256-channel blocks take the
  // four-channels-per-thread path; narrower blocks measured no faster with it and keep the leaner kernel
  const bool vec4 = VEC4 && nc == kFeatChan;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < 64 * CB; i += kFeatThreads) s_acc[i] = 0.f;
  const int s = tile_offsets[tile];
  const int len = min(tile_len[tile], kWinMax);
  int running = 0;
  for (int j0 = 0; j0 < len; j0 += kFeatThreads) {
    const int j = j0 + tid;
    uint32_t u0 = 0u, u1 = 0u;
    if (j < len) { u0 = used32[2 * (size_t)(s + j)]; u1 = used32[2 * (size_t)(s + j) + 1]; s_u[0][j] = u0; s_u[1][j] = u1; }
    int total;
    const int ex = block_exclusive_scan(__popc(u0) + __popc(u1), warp_sums, total);
    if (j < len) s_pref[j] = running + ex;
    running += total;
  }
  if (tid == 0) s_pref[len] = running;
  __syncthreads();
  const int n_tot = running;
  for (int b0 = 0; b0 < n_tot; b0 += kFeatBatch) {
    const int n = min(kFeatBatch, n_tot - b0);
    if (tid < n) {
      const int r = b0 + tid;
      int a = 0, b = len - 1;                  // largest pair index with s_pref <= r (see k_fill)
      while (a < b) {
        const int mid = (a + b + 1) >> 1;
        if (s_pref[mid] <= r) a = mid; else b = mid - 1;
      }
      const int k = r - s_pref[a];
      const uint32_t u0 = s_u[0][a], u1 = s_u[1][a];
      const int cu0 = __popc(u0);
      const int px = (k < cu0) ? nth_set_bit(u0, k) : 32 + nth_set_bit(u1, k - cu0);
      const uint32_t m0 = masks32[2 * (size_t)(s + a)], m1 = masks32[2 * (size_t)(s + a) + 1];
      const uint32_t slot = pair_base[s + a] +
                            (px < 32 ? __popc(m0 & ((1u << px) - 1u)) : __popc(m0) + __popc(m1 & ((1u << (px - 32)) - 1u)));
      const float w = rec_w[slot];
      float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
      if (S > 1) g = rec_gate[slot];
      s_px[tid] = px;
      const int prim = sorted_prims[s + a];
      s_pr[tid] = prim;
      s_cw[tid][0] = w; s_cw[tid][1] = w * g.x; s_cw[tid][2] = w * g.y; s_cw[tid][3] = w * g.z; s_cw[tid][4] = w * g.w;
      // the first record of a pair asks L2 for the pair's attribute rows of this channel block
      if (k == 0 || tid == 0) {
        const char* rows = reinterpret_cast<const char*>(feat_attr + (size_t)prim * S * C + c0);
        for (int sl = 0; sl < S; ++sl)
          for (int b = 0; b < nc * 4; b += 128)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(rows + (size_t)sl * C * 4 + b));
      }
    }
    __syncthreads();
    // runs of equal primitives (block-wide compaction of the run heads)
    {
      const bool head = tid < n && (tid == 0 || s_pr[tid] != s_pr[tid - 1]);
      int total;
      const int pos = block_exclusive_scan(head ? 1 : 0, warp_sums, total);
      if (head) s_run[pos] = tid;
      if (tid == 0) { s_run[total] = n; s_nruns = total; }
    }
    __syncthreads();
    const int nruns = s_nruns;
    // A thread owns one channel; with fewer than 256 channels in the block, RL threads of a warp share a channel
    // and split the records of a run between them (one primitive touches a pixel at most once, so the records
    // of a run hit distinct accumulator cells; runs follow one another in warp lockstep).  The attribute rows
    // of run r + 2 are requested before run r is accumulated, so their latency overlaps two runs of arithmetic.
    if (vec4) {
      // four adjacent channels per thread: one 16-byte accumulator update serves four channels, and the record
      // coefficients are read once for them (same operations per channel as below, so the same bits)
      const int ng = nc >> 2;
      int RL = 1;
      while (RL < 32 && 2 * RL * ng <= kFeatThreads) RL *= 2;
      const int CPW = 32 / RL, rl = lane / CPW;
      uint32_t wmask = 0xffffffffu;
      for (int g = warp * CPW + lane % CPW;; g += (kFeatThreads / 32) * CPW) {
        wmask = __ballot_sync(wmask, g < ng);
        if (g >= ng) break;
        const int c = g * 4;
        const int C4 = C >> 2;
        auto load_rows = [&](int r, float4 (&a)[5]) {
          a[0] = a[1] = a[2] = a[3] = a[4] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (r >= nruns) return;
          const float4* src = reinterpret_cast<const float4*>(feat_attr + (size_t)s_pr[s_run[r]] * S * C + c0 + c);
          a[0] = __ldg(src);
          if (S >= 4) { a[1] = __ldg(src + C4); a[2] = __ldg(src + 2 * C4); a[3] = __ldg(src + 3 * C4); }
          if (S == 5) a[4] = __ldg(src + 4 * C4);
        };
        float4 a_cur[5], a_n1[5], a_n2[5];
        load_rows(0, a_cur);
        load_rows(1, a_n1);
        for (int r = 0; r < nruns; ++r) {
          load_rows(r + 2, a_n2);
          const int j0 = s_run[r], j1 = s_run[r + 1];
          auto mix = [&](const float (&cw)[5], float a0, float a1, float a2, float a3, float a4) {
            float v;
            if (S == 4) {
              v = cw[1] * a0;
              v = fmaf(cw[2], a1, v); v = fmaf(cw[3], a2, v); v = fmaf(cw[4], a3, v);
            } else if (S == 5) {
              v = cw[0] * a0;
              v = fmaf(cw[1], a1, v); v = fmaf(cw[2], a2, v); v = fmaf(cw[3], a3, v); v = fmaf(cw[4], a4, v);
            } else {
              v = cw[0] * a0;
            }
            return v;
          };
          auto contribution = [&](int j) {
            const float4 c03 = *reinterpret_cast<const float4*>(&s_cw[j][0]);
            const float cw[5] = {c03.x, c03.y, c03.z, c03.w, s_cw[j][4]};
            return make_float4(mix(cw, a_cur[0].x, a_cur[1].x, a_cur[2].x, a_cur[3].x, a_cur[4].x),
                               mix(cw, a_cur[0].y, a_cur[1].y, a_cur[2].y, a_cur[3].y, a_cur[4].y),
                               mix(cw, a_cur[0].z, a_cur[1].z, a_cur[2].z, a_cur[3].z, a_cur[4].z),
                               mix(cw, a_cur[0].w, a_cur[1].w, a_cur[2].w, a_cur[3].w, a_cur[4].w));
          };
          int j = j0 + rl;
          for (; j + RL < j1; j += 2 * RL) {
            float4* q0 = reinterpret_cast<float4*>(s_acc + s_px[j] * CB + c);
            float4* q1 = reinterpret_cast<float4*>(s_acc + s_px[j + RL] * CB + c);
            const float4 v0 = contribution(j), v1 = contribution(j + RL);
            const float4 x0 = *q0, x1 = *q1;
            *q0 = make_float4(x0.x + v0.x, x0.y + v0.y, x0.z + v0.z, x0.w + v0.w);
            *q1 = make_float4(x1.x + v1.x, x1.y + v1.y, x1.z + v1.z, x1.w + v1.w);
          }
          for (; j < j1; j += RL) {
            float4* q0 = reinterpret_cast<float4*>(s_acc + s_px[j] * CB + c);
            const float4 v0 = contribution(j), x0 = *q0;
            *q0 = make_float4(x0.x + v0.x, x0.y + v0.y, x0.z + v0.z, x0.w + v0.w);
          }
          if (RL > 1) __syncwarp(wmask);
#pragma unroll
          for (int q = 0; q < 5; ++q) { a_cur[q] = a_n1[q]; a_n1[q] = a_n2[q]; }
        }
      }
      __syncthreads();
      continue;
    }
    int RL = 1;
    while (RL < 32 && 2 * RL * nc <= kFeatThreads) RL *= 2;
    const int CPW = 32 / RL, rl = lane / CPW;
    uint32_t wmask = 0xffffffffu;              // lanes of this warp that still own a channel
    for (int c = warp * CPW + lane % CPW;; c += (kFeatThreads / 32) * CPW) {
      wmask = __ballot_sync(wmask, c < nc);
      if (c >= nc) break;
      auto load_rows = [&](int r, float (&a)[5]) {
        a[0] = a[1] = a[2] = a[3] = a[4] = 0.f;
        if (r >= nruns) return;
        const float* src = feat_attr + (size_t)s_pr[s_run[r]] * S * C + c0 + c;
        a[0] = __ldg(src);
        if (S >= 4) { a[1] = __ldg(src + C); a[2] = __ldg(src + 2 * C); a[3] = __ldg(src + 3 * C); }
        if (S == 5) a[4] = __ldg(src + 4 * C);
      };
      float a_cur[5], a_n1[5], a_n2[5];
      load_rows(0, a_cur);
      load_rows(1, a_n1);
      for (int r = 0; r < nruns; ++r) {
        load_rows(r + 2, a_n2);
        const int j0 = s_run[r], j1 = s_run[r + 1];
        auto contribution = [&](int j) {
          float v;
          if (S == 4) {
            v = s_cw[j][1] * a_cur[0];
            v = fmaf(s_cw[j][2], a_cur[1], v); v = fmaf(s_cw[j][3], a_cur[2], v); v = fmaf(s_cw[j][4], a_cur[3], v);
          } else if (S == 5) {
            v = s_cw[j][0] * a_cur[0];
            v = fmaf(s_cw[j][1], a_cur[1], v); v = fmaf(s_cw[j][2], a_cur[2], v);
            v = fmaf(s_cw[j][3], a_cur[3], v); v = fmaf(s_cw[j][4], a_cur[4], v);
          } else {
            v = s_cw[j][0] * a_cur[0];
          }
          return v;
        };
        int j = j0 + rl;
        // records of one pair touch distinct pixels: four accumulator cells are loaded together
        for (; j + 3 * RL < j1; j += 4 * RL) {
          float* q0 = s_acc + s_px[j] * CB + c; float* q1 = s_acc + s_px[j + RL] * CB + c;
          float* q2 = s_acc + s_px[j + 2 * RL] * CB + c; float* q3 = s_acc + s_px[j + 3 * RL] * CB + c;
          const float v0 = contribution(j), v1 = contribution(j + RL), v2 = contribution(j + 2 * RL), v3 = contribution(j + 3 * RL);
          const float x0 = *q0, x1 = *q1, x2 = *q2, x3 = *q3;
          *q0 = x0 + v0; *q1 = x1 + v1; *q2 = x2 + v2; *q3 = x3 + v3;
        }
        for (; j < j1; j += RL) s_acc[s_px[j] * CB + c] += contribution(j);
        if (RL > 1) __syncwarp(wmask);
#pragma unroll
        for (int q = 0; q < 5; ++q) { a_cur[q] = a_n1[q]; a_n1[q] = a_n2[q]; }
      }
    }
    __syncthreads();
  }
  for (int k = warp; k < 64; k += kFeatThreads / 32) {
    const TilePix tp = tile_pixel(tile, k, ntx, W, H);
    if (!tp.valid) continue;
    for (int c = lane; c < nc; c += 32) out_feat[(size_t)tp.pix * C + c0 + c] = s_acc[k * CB + c];
  }
}

// ------------------------------------------------------------------------------ driver ----
// after the tile pre-test a tile's list rarely holds more than a few hundred candidates, and few tiles
// need more than the first hundred: the tail wave takes whatever is left
static const int kDefaultWaves[] = {32, 32, 64, 128, 256, INT_MAX};

// A schedule for the size of the work (for hosts that can give a frame more records when it asks for them; kDefaultWaves is
// what num_waves = 0 means).  A wave costs some 25 us of dependent launches and, where primitives own few records, another
// fetch of their weight images; a longer window costs records of pixels that end inside it.  So the first window is
//     a = 70 (318,000 / P)^(1/3) (4 / r)^e,   P pixels, r pixels per primitive (at most 9), e = 0.4, or 0.55 for r < 4
// (smaller primitives: fewer of a window's candidates hit a pixel), twice that where the lists come from the caller and have
// not been through the tile pre-test, 65 for 70 in FP32; for a batch of views e = 0.8 for r < 4, and again times H / 32 (the
// images' bytes).  Then a, 2a, 4a, or, on large images, two of a/2 (binary16: at least 32) for the a, and the rest; the smallest
// frames take one window.
// Whole frames, 32, 32, 64, 128, 256, rest against this, us:
//     pixels  primitives  binary16     FP32             pixels  primitives   binary16        FP32
//      5,696       3,560  284 -> 145   279 -> 163      318,159     198,849    806 -> 708   2,080 -> 1,981
//     14,000       8,750  316 -> 182   358 -> 282      318,159      79,539    559 -> 502   1,475 -> 1,353
//     35,840       8,960  247 -> 190   394 -> 354      318,159      10,605    440 -> 414   1,043 -> 1,041
//     80,640      50,400  426 -> 313   750 -> 676      504,000     126,000    745 -> 712   2,187 -> 2,008
//     80,640       2,688  214 -> 169   347 -> 303      808,640     202,160  1,071 -> 1,027 3,355 -> 3,125
//    161,500      16,150  344 -> 322   731 -> 707      808,640      26,954    859 -> 825   2,565 -> 2,400
// a record frame of 320 x 240 and 20,000 primitives 394 -> 296; four views at 1200 x 680 of 500,000 4,486 -> 4,251, at
// 1920 x 1080 of 1,000,000 64-wide ones 10,867 -> 10,408.
//
// How many of a window's candidates hit a pixel is not known here, since it follows from the splats' sizes.  The rows above
// are scenes with 6 to 12 composited records per pixel; where splats are large or stand in deep stacks, windows of this length
// evaluate several times what is composited.  So a caller that reads the counts of a frame can ask for windows halved `finer`
// times (one window: first the several of its size), and lists that the caller gave tell their mean length beforehand: one
// window is for up to 100,000 candidates (FP32 30,000) in all.  Evaluated and composited records per pixel, us, of one
// window and of 104, 104, 208, 416, rest, binary16:
//     200 x 150: own lists  24 / 11  178 | 185,  49 / 13  209 | 183,  67 / 16  216 | 167,  95 / 23  262 | 205
//     200 x 150: given, of 68,000 24 / 11  188 | 219,  105,000 49 / 13  215 | 215,  117,000 67 / 16  234 | 205,  135,000 269 | 220
//     128 x 96:  own lists   6 / 6  107 | 128,  23 / 12  125 | 144,  33 / 15  128 | 137
// and of 72, 72, 144, 288, rest against 32, 32, 64, 128, 256, rest at 320 x 240 in FP32: 33 / 18  584 | 517,  43 / 23  733 | 608.
static int wave_schedule(int32_t n, int32_t width, int32_t height, int32_t hidden, int32_t precision, int32_t views,
                         int64_t list_pairs, int32_t tile_capacity, int32_t finer, int32_t* wave_len) {
  const double P = (double)width * height, r = std::min(9.0, P / std::max(n, 1));
  const bool f32 = precision == MLPSP_PRECISION_F32;
  int count = 0;
  if (P <= (f32 ? 16000.0 : 30000.0) && list_pairs <= (f32 ? 30000 : 100000) && tile_capacity <= kWinMax) {
    if (finer == 0) {
      wave_len[count++] = tile_capacity;
      return count;
    }
    --finer;
  }
  double a = (f32 ? 65.0 : 70.0) * std::cbrt(318000.0 / P) * std::pow(4.0 / r, r >= 4.0 ? 0.4 : (views > 1 ? 0.8 : 0.55));
  if (list_pairs >= 0) a *= 2.0;
  if (views > 1) a *= std::max(1.0, hidden / 32.0);
  a = std::ldexp(a, -std::min(finer, 16));
  const int first = (int)std::min(512.0, std::max(32.0, 8.0 * std::floor(a / 8.0 + 0.5)));
  const bool halves = P >= (f32 ? 250000.0 : 450000.0);
  int lo = 0;
  auto add = [&](int len) {
    len = std::min(std::min(len, kWinMax), tile_capacity - lo);
    if (len > 0) { wave_len[count++] = len; lo += len; }
  };
  add(first);
  const int second = halves ? std::max(first / 2, f32 ? 16 : 32) : first;
  add(second);
  if (halves) add(second);
  add(2 * first);
  add(4 * first);
  while (lo < tile_capacity && count < MLPSP_MAX_WAVES) add(kWinMax);
  return count;
}

extern "C" int mlpsp_wave_schedule(int32_t n, int32_t width, int32_t height, int32_t hidden, int32_t precision, int32_t views,
                                   int32_t caller_lists, int32_t tile_capacity, int32_t* wave_len) {
  MLPSP_REQUIRE(n >= 0 && width > 0 && height > 0 && views > 0 && tile_capacity > 0 && wave_len, MLPSP_E_ARG,
                "mlpsp_wave_schedule: bad argument");
  return wave_schedule(n, width, height, hidden, precision, views, caller_lists ? 0 : -1, tile_capacity, 0, wave_len);
}

extern "C" int mlpsp_wave_schedule_finer(int32_t n, int32_t width, int32_t height, int32_t hidden, int32_t precision, int32_t views,
                                         int64_t list_pairs, int32_t tile_capacity, int32_t finer, int32_t* wave_len) {
  MLPSP_REQUIRE(n >= 0 && width > 0 && height > 0 && views > 0 && list_pairs >= -1 && tile_capacity > 0 && finer >= 0 && wave_len,
                MLPSP_E_ARG, "mlpsp_wave_schedule_finer: bad argument");
  return wave_schedule(n, width, height, hidden, precision, views, list_pairs, tile_capacity, finer, wave_len);
}

int launch_hit_masks(const mlpsp_scene* sc, const mlpsp_frame* fr, uint64_t* mask_geo, cudaStream_t st) {
  const int T = num_tiles(fr->width, fr->height, fr->tile);
  const int ntx = (fr->width + 7) / 8;
  LaunchScope scope(kKHits, 1, st);
  k_hit_masks_all<<<T, 256, 0, st>>>(fr->rays_o, fr->rays_d, (const float4*)sc->geom, sc->n, fr->tile_offsets,
                                     fr->sorted_prims, fr->width, fr->height, ntx, fr->threshold,
                                     miss_bound2(fr->threshold), (uint32_t*)mask_geo, fr->hit_arith == 1 ? 1 : 0, fr->status);
  return cuda_check(cudaGetLastError(), "hit_masks");
}

int launch_render_sorted(const mlpsp_scene* sc, const mlpsp_frame* fr, const Scratch& s, cudaStream_t st,
                         bool lists_refined) {
  const int W = fr->width, H = fr->height;
  const int T = num_tiles(W, H, 8);
  const int ntx = (W + 7) / 8;
  const int64_t P = (int64_t)W * H;
  const int n = sc->n;
  float bg[3] = {0.f, 0.f, 0.f};
  const int has_bg = fr->bg_color != nullptr;
  if (has_bg) { bg[0] = fr->bg_color[0]; bg[1] = fr->bg_color[1]; bg[2] = fr->bg_color[2]; }
  const bool want_t = fr->depth_t != nullptr;
  const bool want_feat = fr->feat != nullptr;
  if (want_feat) {
    MLPSP_REQUIRE(sc->feat_attr && sc->feat_dim > 0 && sc->feat_dim <= 512, MLPSP_E_ARG,
                  "feature rendering needs feat_attr with 1..512 channels");
    MLPSP_REQUIRE(sc->feat_slots == 1 || sc->feat_slots == 4 || sc->feat_slots == 5, MLPSP_E_ARG,
                  "feature slots must be 1, 4 or 5");
  }
  const bool keep = fr->keep_records == 1;
  const bool want_stats = fr->stat_sum_w != nullptr;
  const bool per_pixel = fr->sort_key == MLPSP_ORDER_PER_PIXEL;
  if (per_pixel) {
    MLPSP_REQUIRE(!keep && !want_stats && !fr->mask_used && !want_t, MLPSP_E_ARG,
                  "per-pixel ordering renders rgb, alpha and the feature map only");
    MLPSP_REQUIRE(fr->tile_capacity <= kWinMax, MLPSP_E_LIMIT, "per-pixel ordering needs tile_capacity <= %d", kWinMax);
  }
  if (want_stats)
    MLPSP_REQUIRE(fr->gt_rgb && fr->stat_max_w && fr->stat_hits && fr->stat_sum_werr && fr->stat_contrib, MLPSP_E_ARG,
                  "contribution statistics need gt_rgb and all five per-primitive arrays");
  const PrimStats pstats = {fr->gt_rgb, fr->sorted_prims, fr->stat_sum_w, fr->stat_max_w, fr->stat_hits,
                            fr->stat_sum_werr, fr->stat_contrib};
  // record export reads the consumed masks from the scratch copy, so a caller-owned mask buffer is
  // filled by a device copy afterwards
  uint32_t* used32 = (keep || want_feat) ? s.used32 : (uint32_t*)fr->mask_used;
  if (!lists_refined) {
    LaunchScope scope(kKMisc, 1, st);
    const int64_t span = std::max<int64_t>(std::max<int64_t>(P, T), n);
    launch_chained(k_init_frame, dim3((unsigned)((span + 255) / 256)), dim3(256), 0, st, P, s.px_state, s.px_depth, fr->rgb, fr->alpha, fr->depth_t, bg[0], bg[1],
                                                                bg[2], T, s.active[0], s.counters, fr->tile_offsets, s.tile_len,
                                                                n, s.prim_cnt);
  }
  if (used32 && fr->mask_used) {
    MLPSP_CUDA_OK(cudaMemsetAsync(used32, 0, 8 * (size_t)fr->max_pairs, st));     // the caller sees all of it
  } else if (used32) {
    LaunchScope scope(kKMisc, 1, st);
    launch_chained(k_clear_used, dim3((T + 7) / 8), dim3(256), 0, st, fr->tile_offsets, s.tile_len, T, reinterpret_cast<uint2*>(used32), fr->status);
  }
  if (n == 0) {
    if (want_feat) MLPSP_CUDA_OK(cudaMemsetAsync(fr->feat, 0, 4 * (size_t)P * sc->feat_dim, st));
    return cuda_check(cudaGetLastError(), "render_sorted");
  }
  const bool tc_path = fr->precision == MLPSP_PRECISION_F16 || fr->precision == MLPSP_PRECISION_BF16;
  const bool ref_arith = fr->hit_arith == 1;
  // Small groups get their own work list and kernel when the tensor-core evaluator runs and the scene is one whose
  // primitives own few records each: a frame evaluates about a dozen records per pixel, so with more than one
  // primitive per three pixels the typical primitive has fewer than 40 records per frame.  With fewer primitives the
  // extra launch per wave costs more than the few remainders gain (measured: 250,000 primitives on 816,000 pixels
  // lose 4 % of evaluator time with the second list, 500,000 gain 2 %, 2,000,000 with 64 hidden units gain 21 %).  (Record export keeps one list.)
  const bool split_small = tc_path && !keep && (int64_t)n * 3 > P;
  // Encoded ray directions from a table where a primitive owns many records: the table takes half of the special functions
  // off the evaluator and adds 80 bytes per record to what it draws from L2, and a launch.  With few records per weight image
  // L2 is the scarcer of the two, and a small image has too few records to pay for the launch.  Whole frames with the table
  // against without, 32-wide layers, by pixels per primitive:
  //     320 x 240: 10 to 26 +4 %;  400 x 300: 7.1 +1 %, 40 +3 %;  480 x 360: 7.1 0, 11 -1.5 %, 40 -1 %;
  //     639 x 477: 3.4 +6 %, 5.1 +1 %, 7.1 -1 %, 16 -4 %;  800 x 600: 7.1 -2.5 %, 16 -5.5 %;
  //     1200 x 680: 3.3 +17 %, 5.8 +2.5 %, 7.0 +0.5 %, 8.2 -0.5 %, 16 -5 %, 40 -6 %
  // and 64-wide ones, whose image is 2.5 times as large:
  //     480 x 360: 11 to 150 +1 to +6 %;  639 x 477: 16 0, 25 to 150 +1 to +2 %;  800 x 600: 11 0, 16 -1 %, 60 -1.3 %;
  //     1200 x 680: 8.2 +3.3 %, 11 +1.5 %, 16 0, 25 -1 %, 60 -1.3 %.
  const bool wide = sc->hidden > 32;
  const bool table = tc_path && !keep && (int64_t)n * (wide ? 20 : 7) <= P && P >= (wide ? 400000 : 150000) && s.dir_table &&
                     sc->num_freq == 6;
  if (table) {
    const int rc_dir = launch_encode_directions(sc, fr, s.dir_table, st);
    if (rc_dir) return rc_dir;
  }
  const int sms = sm_count();
  // per-pixel ordering: one wave over the whole lists, every pixel live
  const int nw = per_pixel ? 1 : (fr->num_waves > 0 ? fr->num_waves : (int)(sizeof(kDefaultWaves) / sizeof(int)));
  int lo = 0;
  for (int w = 0; w < nw && lo < fr->tile_capacity; ++w) {
    const int wl = per_pixel ? fr->tile_capacity : (fr->num_waves > 0 ? fr->wave_len[w] : kDefaultWaves[w]);
    MLPSP_REQUIRE(wl > 0, MLPSP_E_ARG, "wave_len[%d] must be positive", w);
    int hi = (wl >= fr->tile_capacity - lo || w == nw - 1) ? fr->tile_capacity : lo + wl;
    MLPSP_REQUIRE(hi - lo <= kWinMax, MLPSP_E_LIMIT, "wave window beyond %d candidates", kWinMax);
    const int cur = w & 1, nxt = cur ^ 1;
    // a last wave the caller expects to be idle: one CTA per SM walks whatever is left
    const bool idle_tail = fr->tail_hint == 1 && hi == fr->tile_capacity && w > 0;
    const int grid_comp = idle_tail ? sms : std::min(T, sms * 32);
    const int cap_mlp = idle_tail ? sms : 0;
    const int32_t* act = s.active[cur];
    const int32_t* act_n = s.counters + kCtrActive0 + cur;
    int rc;
    {
      LaunchScope scope(kKHits, 1, st);
      const HitArgs ha = {fr->rays_o, fr->rays_d, (const float4*)sc->geom, n, fr->tile_offsets, s.tile_len, fr->sorted_prims, W, H, ntx,
                          fr->threshold, miss_bound2(fr->threshold), form_threshold(fr->threshold), act, act_n, lo, hi, s.px_state,
                          reinterpret_cast<uint2*>(s.masks32), s.pair_base, s.prim_cnt + (size_t)(w & 1) * prim_cnt_stride(n), s.counters,
                          fr->max_records, fr->status, s.counters + kCtrActive0 + nxt, 0};
      rc = launch_hits(&ha, 1, ref_arith, T, sms, idle_tail, st);
      if (rc) return rc;
    }
    rc = launch_prim_scan(s, n, nullptr, fr->status, st, split_small, w);
    if (rc) return rc;
    {
      LaunchScope scope(kKFill, 1, st);
      float4* gate = (want_feat && sc->feat_slots > 1) ? s.rec_gate : nullptr;
      FillArgs fa = {fr->rays_o, fr->rays_d, (const float4*)sc->geom, fr->tile_offsets, s.tile_len, fr->sorted_prims, W, H, ntx,
                           fr->threshold, act, act_n, lo, hi, reinterpret_cast<const uint2*>(s.masks32), s.pair_base,
                           s.prim_pos, reinterpret_cast<float4*>(s.rec_in), (want_t || per_pixel) ? s.rec_t : nullptr, gate,
                           sc->gate_beta, sc->gate_tau, keep ? 1 : 0, table ? 1 : 0, fr->status, 0, 0, 0};
      rc = launch_fill(&fa, 1, gate || per_pixel, ref_arith, T, sms, idle_tail, st);
      if (rc) return rc;
    }
    if (tc_path)
      rc = launch_mlp_f16(sc, s.rec_in, s.work, s.counters, s.rec_out, keep ? s.rec_ext : nullptr, kOutAlpha,
                          fr->status, st, fr->precision == MLPSP_PRECISION_BF16, cap_mlp, split_small ? s.work_small : nullptr,
                          table ? s.dir_table : nullptr);
    else
      rc = launch_mlp_f32(sc, s.rec_in, s.work, s.counters, s.rec_out, keep ? s.rec_ext : nullptr, kOutAlpha,
                          fr->status, st, cap_mlp);
    if (rc) return rc;
    if (per_pixel) {
      LaunchScope scope(kKComposite, 1, st);
      k_composite_per_pixel<<<std::min(T, sms * 32), 64, 0, st>>>(fr->tile_offsets, s.tile_len, T, W, H, ntx, s.masks32, s.pair_base,
                                                                 s.rec_out, s.rec_t, fr->rgb, fr->alpha, bg[0], bg[1], bg[2],
                                                                 has_bg, want_feat ? used32 : nullptr,
                                                                 want_feat ? s.rec_w : nullptr, fr->status);
      break;
    }
    {
      LaunchScope scope(kKComposite, 1, st);
      const CompositeArgs ca = {pstats, fr->tile_offsets, s.tile_len, W, H, ntx, act, act_n, lo, hi, s.masks32, s.pair_base,
                                s.rec_out, want_t ? s.rec_t : nullptr, s.px_state, s.px_depth, fr->rgb, fr->alpha, fr->depth_t, used32,
                                want_feat ? s.rec_w : nullptr, keep ? s.rec_tr : nullptr, bg[0], bg[1], bg[2], has_bg,
                                s.active[nxt], s.counters + kCtrActive0 + nxt, fr->status};
      launch_views<1>(want_stats ? k_composite<true, 1> : k_composite<false, 1>, dim3(grid_comp), dim3(64), 0, st, &ca, 1);
    }
    lo = hi;
  }
  if (fr->mask_used && used32 != (uint32_t*)fr->mask_used)
    MLPSP_CUDA_OK(cudaMemcpyAsync(fr->mask_used, used32, 8 * (size_t)fr->max_pairs, cudaMemcpyDeviceToDevice, st));
  if (want_feat && feature_tc_supported(sc)) {
    // binary16 attributes and a channel count the tensor-core kernel takes: the contraction runs on tcgen05
    LaunchScope scope(kKComposite, 1, st);
    const int rc_ft = launch_feature_tc(sc, fr, s, used32, st);
    if (rc_ft) return rc_ft;
  } else if (want_feat) {
    static DeviceOnce attr_once;
    const int CB = std::min(sc->feat_dim, kFeatChan);
    const size_t smem = sizeof(float) * 64 * (size_t)CB;
    if (attr_once.first()) {
      MLPSP_CUDA_OK(cudaFuncSetAttribute(k_feature_composite<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * kFeatChan * 4));
      MLPSP_CUDA_OK(cudaFuncSetAttribute(k_feature_composite<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * kFeatChan * 4));
    }
    LaunchScope scope(kKComposite, 1, st);
    const dim3 grid(T, (sc->feat_dim + CB - 1) / CB);
    const bool vec = sc->feat_dim >= kFeatChan && (sc->feat_dim & 3) == 0 && (reinterpret_cast<uintptr_t>(sc->feat_attr) & 15) == 0;
    if (vec)
      k_feature_composite<true><<<grid, kFeatThreads, smem, st>>>(fr->tile_offsets, s.tile_len, fr->sorted_prims, W, H, ntx, used32, s.masks32,
                                                                 s.pair_base, s.rec_w, s.rec_gate, sc->feat_attr, sc->feat_slots,
                                                                 sc->feat_dim, CB, fr->feat, fr->status);
    else
      k_feature_composite<false><<<grid, kFeatThreads, smem, st>>>(fr->tile_offsets, s.tile_len, fr->sorted_prims, W, H, ntx, used32, s.masks32,
                                                                  s.pair_base, s.rec_w, s.rec_gate, sc->feat_attr, sc->feat_slots,
                                                                  sc->feat_dim, CB, fr->feat, fr->status);
  }
  return cuda_check(cudaGetLastError(), "render_sorted");
}

// ----------------------------------------------------------------------- view batches ----
// Several views of one scene rendered together (rgb and alpha only).  Binning, sorting, hit masks, record fill and
// compositing run per view on the view's own scratch; what is shared is everything per primitive: the record
// counts, the CSR offsets, the work list and the record arrays live in the first frame's scratch, compositing
// slots are numbered across the views, and ONE evaluator launch per wave serves all views.  A primitive's weight
// image is then fetched once per wave for the records of all views, which is what bounds many-primitive scenes
// (a few records per primitive and view).  Every record goes through the same arithmetic as in a frame rendered
// alone, so the images are bit-identical.
int launch_render_batch(const mlpsp_scene* sc, const mlpsp_frame* frs, const Scratch* ss, int V, cudaStream_t st,
                        bool lists_refined) {
  const mlpsp_frame* f0 = frs;
  const Scratch& lead = ss[0];
  const int W = f0->width, H = f0->height;
  const int T = num_tiles(W, H, 8);
  const int ntx = (W + 7) / 8;
  const int64_t P = (int64_t)W * H;
  const int n = sc->n;
  const PrimStats no_stats = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  if (!lists_refined) {
    LaunchScope scope(kKMisc, V, st);
    for (int v = 0; v < V; ++v) {
      const mlpsp_frame* fr = frs + v;
      float bg[3] = {0.f, 0.f, 0.f};
      if (fr->bg_color) { bg[0] = fr->bg_color[0]; bg[1] = fr->bg_color[1]; bg[2] = fr->bg_color[2]; }
      const int nv = v == 0 ? n : 0;     // the per-primitive arrays are the first frame's
      const int64_t span = std::max<int64_t>(std::max<int64_t>(P, T), nv);
      launch_chained(k_init_frame, dim3((unsigned)((span + 255) / 256)), dim3(256), 0, st, P, ss[v].px_state, ss[v].px_depth, fr->rgb, fr->alpha, nullptr, bg[0], bg[1],
                                                                  bg[2], T, ss[v].active[0], ss[v].counters, fr->tile_offsets,
                                                                  ss[v].tile_len, nv, lead.prim_cnt);
    }
  }
  if (n == 0) return cuda_check(cudaGetLastError(), "render_batch");
  const bool tc_path = f0->precision == MLPSP_PRECISION_F16 || f0->precision == MLPSP_PRECISION_BF16;
  const bool ref_arith = f0->hit_arith == 1;
  // the second work list costs one launch per wave and batch, not per view, so it pays earlier than for one frame
  // (measured with and without: fourview_500k in one batch of 4 views 2.51 -> 2.31 ms, stress_2m in batches of 16
  // views 72.2 -> 65.8 ms of evaluator time)
  const bool split_small = tc_path && (int64_t)n * 20 > P * V;
  const int sms = sm_count(), groups = (V + kViewsPerLaunch - 1) / kViewsPerLaunch;
  const int nw = f0->num_waves > 0 ? f0->num_waves : (int)(sizeof(kDefaultWaves) / sizeof(int));
  int lo = 0;
  for (int w = 0; w < nw && lo < f0->tile_capacity; ++w) {
    const int wl = f0->num_waves > 0 ? f0->wave_len[w] : kDefaultWaves[w];
    MLPSP_REQUIRE(wl > 0, MLPSP_E_ARG, "wave_len[%d] must be positive", w);
    const int hi = (wl >= f0->tile_capacity - lo || w == nw - 1) ? f0->tile_capacity : lo + wl;
    MLPSP_REQUIRE(hi - lo <= kWinMax, MLPSP_E_LIMIT, "wave window beyond %d candidates", kWinMax);
    const int cur = w & 1, nxt = cur ^ 1;
    const bool idle_tail = f0->tail_hint == 1 && hi == f0->tile_capacity && w > 0;
    const int grid_comp = idle_tail ? sms : std::min(T, sms * 32);
    const int cap_mlp = idle_tail ? sms : 0;
    int32_t* cnt = lead.prim_cnt + (size_t)(w & 1) * prim_cnt_stride(n);
    int rc = MLPSP_OK;
    {
      LaunchScope scope(kKHits, groups, st);
      HitArgs ha[kViewsPerLaunch];
      for (int v = 0; v < V; ++v) {
        const mlpsp_frame* fr = frs + v;
        const Scratch& s = ss[v];
        const int q = v % kViewsPerLaunch;
        ha[q] = {fr->rays_o, fr->rays_d, (const float4*)sc->geom, n, fr->tile_offsets, s.tile_len, fr->sorted_prims, W, H, ntx,
                            f0->threshold, miss_bound2(f0->threshold), form_threshold(f0->threshold), s.active[cur],
                            s.counters + kCtrActive0 + cur, lo, hi, s.px_state, reinterpret_cast<uint2*>(s.masks32), s.pair_base, cnt,
                            lead.counters, f0->max_records, f0->status, s.counters + kCtrActive0 + nxt, v > 0 ? 1 : 0};
        if (q + 1 < kViewsPerLaunch && v + 1 < V) continue;
        rc = launch_hits(ha, q + 1, ref_arith, T, sms, idle_tail, st);
        if (rc) return rc;
      }
    }
    rc = launch_prim_scan(lead, n, nullptr, f0->status, st, split_small, w);
    if (rc) return rc;
    {
      // (no table of ray directions: the records of a launch come from all views, and would have to name theirs)
      LaunchScope scope(kKFill, groups, st);
      FillArgs fa[kViewsPerLaunch];
      for (int v = 0; v < V; ++v) {
        const mlpsp_frame* fr = frs + v;
        const Scratch& s = ss[v];
        const int q = v % kViewsPerLaunch;
        fa[q] = {fr->rays_o, fr->rays_d, (const float4*)sc->geom, fr->tile_offsets, s.tile_len, fr->sorted_prims, W, H, ntx,
                             f0->threshold, s.active[cur], s.counters + kCtrActive0 + cur, lo, hi,
                             reinterpret_cast<const uint2*>(s.masks32), s.pair_base, lead.prim_pos, reinterpret_cast<float4*>(lead.rec_in),
                             nullptr, nullptr, sc->gate_beta, sc->gate_tau, 0, 0, f0->status, 0, 0, 0};
        if (q + 1 < kViewsPerLaunch && v + 1 < V) continue;
        rc = launch_fill(fa, q + 1, false, ref_arith, T, sms, idle_tail, st);
        if (rc) return rc;
      }
    }
    if (tc_path)
      rc = launch_mlp_f16(sc, lead.rec_in, lead.work, lead.counters, lead.rec_out, nullptr, kOutAlpha, f0->status, st,
                          f0->precision == MLPSP_PRECISION_BF16, cap_mlp, split_small ? lead.work_small : nullptr);
    else
      rc = launch_mlp_f32(sc, lead.rec_in, lead.work, lead.counters, lead.rec_out, nullptr, kOutAlpha, f0->status, st, cap_mlp);
    if (rc) return rc;
    {
      LaunchScope scope(kKComposite, groups, st);
      CompositeArgs ca[kViewsPerLaunch];
      for (int v = 0; v < V; ++v) {
        const mlpsp_frame* fr = frs + v;
        const Scratch& s = ss[v];
        float bg[3] = {0.f, 0.f, 0.f};
        const int has_bg = fr->bg_color != nullptr;
        if (has_bg) { bg[0] = fr->bg_color[0]; bg[1] = fr->bg_color[1]; bg[2] = fr->bg_color[2]; }
        const int q = v % kViewsPerLaunch;
        ca[q] = {no_stats, fr->tile_offsets, s.tile_len, W, H, ntx, s.active[cur], s.counters + kCtrActive0 + cur, lo, hi, s.masks32,
                 s.pair_base, lead.rec_out, nullptr, s.px_state, s.px_depth, fr->rgb, fr->alpha, nullptr, nullptr, nullptr, nullptr,
                 bg[0], bg[1], bg[2], has_bg, s.active[nxt], s.counters + kCtrActive0 + nxt, f0->status};
        if (q + 1 < kViewsPerLaunch && v + 1 < V) continue;
        if (q == 0) launch_views<1>(k_composite<false, 1>, dim3(grid_comp), dim3(64), 0, st, ca, 1);
        else launch_views<kViewsPerLaunch>(k_composite<false, kViewsPerLaunch>, dim3(grid_comp), dim3(64), 0, st, ca, q + 1);
      }
    }
    lo = hi;
  }
  return cuda_check(cudaGetLastError(), "render_batch");
}

// ----------------------------------------------------------------------- record export ----
// Pixel-major records in compositing order (np_tile_kernels.cu:3138-3154; training_wmma.cuh:223-256),
// rebuilt after the frame from the consumed masks, the evaluator outputs kept per compositing slot
// and a recomputed hit test.  Like the reference: count per pixel, prefix, emit.  A pixel's lane walks the pairs it consumed (the
// masks of 32 pairs transposed); in the emitting walk it leaves each record's slot and pixel in the record's own row, and a
// thread per record then makes the row of it, so that the walk's uneven tiles carry no arithmetic and rows are written whole.
// (Without ids and rows of the records to leave them in, the walk emits.)  Bound: the latency of the walk's and the rows'
// gathers; 0.7 M records (320 x 240): a walk over the pairs that any pixel of a warp consumed, emitting, took 218 us, each
// pixel's own walk 152, with the records of a warp listed first 115, this 58.
struct ExportArgs {
  const float* rays_o; const float* rays_d; const float4* geom;
  const int32_t* tile_offsets; const int32_t* tile_len; const int32_t* sorted_prims; int W, H, ntx; float thr, beta, tau;
  const uint32_t* used32; const uint32_t* masks32; const uint32_t* pair_base; const float4* rec_out; const float4* rec_ext; const float* rec_tr;
  const float4* px_state; int32_t* px_cnt; const int32_t* px_off; int max_hits; int32_t* worst;
  int32_t* ids; float* x6; float* raw; int32_t* relu_masks; float* gates; int64_t max_out; int ref_arith, vec, place; const int32_t* status;
};

// one record: slot of its evaluation, primitive, pixel, place in the output
__device__ __forceinline__ void export_row(const ExportArgs& a, uint32_t slot, int p, int pix, int64_t r) {
  const float4 ro = __ldg(a.rec_out + slot), re = __ldg(a.rec_ext + slot);
  const float tr = a.raw ? __ldg(a.rec_tr + slot) : 0.f;
  const V3 o = load3(a.rays_o, pix), d = load3(a.rays_d, pix);
  Hit h;
  if (a.ref_arith) hit_test_ref(load_geom_ref(a.geom, p), o, d, a.thr, h);
  else hit_test(load_geom(a.geom, p), o, d, a.thr, h);
  if (a.ids && !a.place) a.ids[r] = p;
  if (a.x6) {
    if (a.vec) {
      float2* q = reinterpret_cast<float2*>(a.x6) + r * 3;
      q[0] = make_float2(d.x, d.y); q[1] = make_float2(d.z, h.dx); q[2] = make_float2(h.dy, h.dz);
    } else {
      float* q = a.x6 + r * 6; q[0] = d.x; q[1] = d.y; q[2] = d.z; q[3] = h.dx; q[4] = h.dy; q[5] = h.dz;
    }
  }
  if (a.raw) {
    if (a.vec) {
      float4* q = reinterpret_cast<float4*>(a.raw) + r * 2;
      q[0] = make_float4(ro.x, ro.y, ro.z, re.x); q[1] = make_float4(tr, ro.w, h.decay, re.y);
    } else {
      float* q = a.raw + r * 8;
      q[0] = ro.x; q[1] = ro.y; q[2] = ro.z; q[3] = re.x; q[4] = tr; q[5] = ro.w; q[6] = h.decay; q[7] = re.y;
    }
  }
  if (a.relu_masks) {
    const int2 m = make_int2((int32_t)__float_as_uint(re.z), (int32_t)__float_as_uint(re.w));
    if (a.vec) reinterpret_cast<int2*>(a.relu_masks)[r] = m;
    else { a.relu_masks[r * 2] = m.x; a.relu_masks[r * 2 + 1] = m.y; }
  }
  if (a.gates) {
    const float4 g = tetra_gates(h, gate_scales(__ldg(a.geom + (size_t)p * 4 + 3), a.beta), a.tau);
    if (a.vec) reinterpret_cast<float4*>(a.gates)[r] = g;
    else { float* q = a.gates + r * 4; q[0] = g.x; q[1] = g.y; q[2] = g.z; q[3] = g.w; }
  }
}

template <bool EMIT>
__global__ void __launch_bounds__(64) k_export(const ExportArgs a) {
  if (a.status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int tile = blockIdx.x;
  const int s = a.tile_offsets[tile], e = s + a.tile_len[tile];
  const int lane = threadIdx.x & 31, half = threadIdx.x >> 5;
  const TilePix tp = tile_pixel(tile, half * 32 + lane, a.ntx, a.W, a.H);
  const int64_t out0 = EMIT && tp.valid ? a.px_off[tp.pix] : 0;
  const uint32_t lt = (1u << lane) - 1u;
  int cnt = 0;
  for (int i0 = s; i0 < e; i0 += 32) {
    const int idx = i0 + lane;
    uint32_t mine = 0u, hitm = 0u, first = 0u;       // pair idx: this half's consumed and hit pixels, the slot of its first record
    int prim = 0;
    if (idx < e) {
      const uint2 uu = *reinterpret_cast<const uint2*>(a.used32 + 2 * (size_t)idx);
      mine = half ? uu.y : uu.x;
      if (EMIT && mine) {
        const uint2 mm = *reinterpret_cast<const uint2*>(a.masks32 + 2 * (size_t)idx);
        hitm = half ? mm.y : mm.x;
        first = a.pair_base[idx] + (half ? __popc(mm.x) : 0);
        prim = a.sorted_prims[idx];
      }
    }
    if (!__any_sync(0xffffffffu, mine != 0u)) continue;
    uint32_t todo = transpose32(mine);               // the pairs that this lane's pixel consumed
    if (!EMIT) {
      cnt += __popc(todo);
      continue;
    }
    while (__any_sync(0xffffffffu, todo != 0u)) {
      const int j = todo ? __ffs(todo) - 1 : lane;
      const uint32_t hj = __shfl_sync(0xffffffffu, hitm, j), fj = __shfl_sync(0xffffffffu, first, j);
      const int p = __shfl_sync(0xffffffffu, prim, j);
      if (!todo) continue;
      todo &= todo - 1u;
      const uint32_t slot = fj + __popc(hj & lt);
      const int64_t r = out0 + cnt++;
      if (r >= a.max_out) continue;
      if (a.place) {
        a.ids[r] = p;
        *reinterpret_cast<int2*>(a.raw + r * 8) = make_int2((int)slot, tp.pix);
      } else {
        export_row(a, slot, p, tp.pix, r);
      }
    }
  }
  if (!EMIT && tp.valid) {
    a.px_cnt[tp.pix] = cnt;
    atomicMax(a.worst, cnt);
    const bool live = a.px_state[tp.pix].w >= MLPSP_TERM;
    if (a.max_hits > 0 && cnt >= a.max_hits && (cnt > a.max_hits || live)) atomicOr(a.worst + 1, 1);
  }
}

// the rows of the records that k_export has placed: no more than the frame has, whatever total the caller gives
__global__ void __launch_bounds__(256) k_export_rows(const ExportArgs a, int64_t total) {
  if (a.status[MLPSP_ST_BITS] & MLPSP_ST_FATAL) return;
  const int64_t r = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (r >= total || r >= a.px_off[(size_t)a.W * a.H]) return;
  const int2 at = *reinterpret_cast<const int2*>(a.raw + r * 8);
  export_row(a, (uint32_t)at.x, a.ids[r], at.y, r);
}

__global__ void k_widen_i32(const int32_t* __restrict__ in, int64_t n, int64_t* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = in[i];
}

int launch_export_records(const mlpsp_scene* sc, const mlpsp_frame* fr, const Scratch& s, int64_t* offsets, int32_t* ids,
                          float* x6, float* raw, int32_t* relu_masks, float* gates, int64_t max_out, int32_t max_hits,
                          int64_t* total_host, int32_t* worst_host, bool counted, cudaStream_t st) {
  const int W = fr->width, H = fr->height, T = num_tiles(W, H, 8), ntx = (W + 7) / 8;
  const int64_t P = (int64_t)W * H;
  int32_t* worst = s.counters + kCtrScratch;     // [0] largest per-pixel count, [1] capacity flag
  const bool outputs = ids || x6 || raw || relu_masks || gates;
  int64_t total = max_out;                       // counted: the caller holds this frame's total
  const int vec = (reinterpret_cast<uintptr_t>(x6) & 7) == 0 && (reinterpret_cast<uintptr_t>(relu_masks) & 7) == 0 &&
                  ((reinterpret_cast<uintptr_t>(raw) | reinterpret_cast<uintptr_t>(gates)) & 15) == 0;
  ExportArgs a = {fr->rays_o, fr->rays_d, (const float4*)sc->geom, fr->tile_offsets, s.tile_len, fr->sorted_prims, W, H, ntx, fr->threshold,
                  sc->gate_beta, sc->gate_tau, s.used32, s.masks32, s.pair_base, s.rec_out, s.rec_ext, s.rec_tr, s.px_state, s.px_cnt, s.px_off,
                  max_hits, worst, ids, x6, raw, relu_masks, gates, max_out, fr->hit_arith == 1 ? 1 : 0, vec, 0, fr->status};
  if (!counted) {
    LaunchScope scope(kKMisc, 2 + scan_launches(P), st);
    HostWords& hw = host_words();
    cudaEvent_t ev = nullptr;
    int rc = hw.open(&ev);
    if (rc) return rc;
    MLPSP_CUDA_OK(cudaMemsetAsync(worst, 0, 8, st));
    k_export<false><<<T, 64, 0, st>>>(a);
    rc = launch_scan_i32(s.px_cnt, P, s.scan_blk, s.px_off, st);
    if (rc) return rc;
    k_widen_i32<<<(unsigned)((P + 1 + 255) / 256), 256, 0, st>>>(s.px_off, P + 1, offsets);
    MLPSP_CUDA_OK(cudaMemcpyAsync(hw.word, s.px_off + P, 4, cudaMemcpyDeviceToHost, st));
    MLPSP_CUDA_OK(cudaMemcpyAsync(hw.word + 1, worst, 8, cudaMemcpyDeviceToHost, st));
    MLPSP_CUDA_OK(cudaEventRecord(ev, st));
    MLPSP_CUDA_OK(cudaEventSynchronize(ev));
    const volatile int32_t* h = hw.word;
    total = h[0];
    if (total_host) *total_host = h[0];
    if (worst_host) *worst_host = h[2] ? -h[1] : h[1];
  }
  if (outputs && max_out >= total && total > 0) {
    a.place = ids && raw && vec ? 1 : 0;
    LaunchScope scope(kKMisc, a.place ? 2 : 1, st);
    k_export<true><<<T, 64, 0, st>>>(a);
    if (a.place) k_export_rows<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(a, total);
  }
  return cuda_check(cudaGetLastError(), "export_records");
}

}  // namespace mlpsp
