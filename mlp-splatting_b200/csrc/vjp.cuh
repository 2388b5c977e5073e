// What the FP32 and the tensor-core weight-gradient kernels share: the plan of a launch and where gradients go.
#pragma once
#include <cstdint>

namespace mlpsp {

constexpr int kVjpBlock = 128;      // records a CTA takes at a time

// One segment of one primitive: dest < 0 = it is the primitive's only one and goes to the gradient tensors, else the row
// of the partial sums it goes to.
struct __align__(16) VjpItem { int64_t start; int32_t rows, prim, dest, pad[3]; };

__device__ __forceinline__ VjpItem load_item(const VjpItem* p) {
  const int4 a = __ldg(reinterpret_cast<const int4*>(p));
  VjpItem v;
  v.start = (int64_t)((uint64_t)(uint32_t)a.x | ((uint64_t)(uint32_t)a.y << 32));
  v.rows = a.z;
  v.prim = a.w;
  v.dest = __ldg(&p->dest);
  return v;
}

// W1[32,72] b1[32] W2[32,32] b2[32] W3[4,32] b3[4]: base and floats from one primitive to the next of each tensor
struct VjpOut { float* W1; float* b1; float* W2; float* b2; float* W3; float* b3; int64_t sW1, sb1, sW2, sb2, sW3, sb3; };

constexpr int kGH = 32, kGIN = 72;
constexpr int kOW1 = 0, kOb1 = kOW1 + kGH * kGIN, kOW2 = kOb1 + kGH, kOb2 = kOW2 + kGH * kGH, kOW3 = kOb2 + kGH,
              kOb3 = kOW3 + 4 * kGH, kGradLen = kOb3 + 4;   // 3,524 = the reference's packed gradient row
static_assert(kGradLen == 3524, "gradient row layout");

// plan counters (device int32); the flag word holds the bits that mlpsp.h gives for *nonfinite
enum VjpCounter { kVpItems = 0, kVpRows = 1, kVpMulti = 2, kVpFlag = 3, kVpEmpty = 4, kVpNext = 5, kVpParts = 6, kVpCounters = 7 };
constexpr int kVpBadPlan = 4;
// a counter of the plan, 0 when the offsets were refused: a list that may be cut short or point past the records is not read
__device__ __forceinline__ int vjp_planned(const int32_t* counters, int which) {
  return (counters[kVpFlag] & kVpBadPlan) ? 0 : counters[which];
}

// The list of segments: kVpItems from the front of the array and kVpParts from its end backwards.  A plan puts the full segments
// in front, so that CTAs end on the shorter remainders (with both in the primitives' order the last CTAs of 5.5 M records worked
// 62 us after the first had run out).
struct VjpList {
  const VjpItem* items; const VjpItem* end; int front, total;
  __device__ __forceinline__ VjpList(const VjpItem* items_, int64_t max_items, const int32_t* counters)
      : items(items_), end(items_ + max_items), front(vjp_planned(counters, kVpItems)), total(front + vjp_planned(counters, kVpParts)) {}
  __device__ __forceinline__ VjpItem at(int i) const { return load_item(i < front ? items + i : end - 1 - (i - front)); }
};

// zero gradients of one primitive, by nthr threads (rows of 16-byte multiples; b = the tensors' bases aligned)
__device__ __forceinline__ void vjp_zero(const VjpOut& o, int prim, int aligned, int t, int nthr) {
  auto fill = [&](float* p, int64_t stride, int len) {
    p += prim * stride;
    if (aligned) {
      for (int i = t; i < len / 4; i += nthr) reinterpret_cast<float4*>(p)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
      for (int i = t; i < len; i += nthr) p[i] = 0.f;
    }
  };
  fill(o.W1, o.sW1, kGH * kGIN); fill(o.b1, o.sb1, kGH); fill(o.W2, o.sW2, kGH * kGH); fill(o.b2, o.sb2, kGH);
  fill(o.W3, o.sW3, 4 * kGH); fill(o.b3, o.sb3, 4);
}
inline int vjp_aligned(const VjpOut& o) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(o.W1) | reinterpret_cast<uintptr_t>(o.b1) | reinterpret_cast<uintptr_t>(o.W2) |
                      reinterpret_cast<uintptr_t>(o.b2) | reinterpret_cast<uintptr_t>(o.W3) | reinterpret_cast<uintptr_t>(o.b3);
  return (a & 15) == 0 && ((o.sW1 | o.sb1 | o.sW2 | o.sb2 | o.sW3 | o.sb3) & 3) == 0;
}

__device__ __forceinline__ VjpOut vjp_row(const VjpOut& o, float* partial, const VjpItem& it) {
  VjpOut r;
  if (it.dest >= 0) {
    float* p = partial + (size_t)it.dest * kGradLen;
    r.W1 = p + kOW1; r.b1 = p + kOb1; r.W2 = p + kOW2; r.b2 = p + kOb2; r.W3 = p + kOW3; r.b3 = p + kOb3;
  } else {
    r.W1 = o.W1 + it.prim * o.sW1; r.b1 = o.b1 + it.prim * o.sb1; r.W2 = o.W2 + it.prim * o.sW2;
    r.b2 = o.b2 + it.prim * o.sb2; r.W3 = o.W3 + it.prim * o.sW3; r.b3 = o.b3 + it.prim * o.sb3;
  }
  return r;
}

}  // namespace mlpsp
