// fp32_copy.cuh -- asynchronous copies of FP32 operand panels into shared memory
// (the CUDA-core SGEMM and the grouped GEMM's FP32 tiles).
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace b2 {
namespace f32copy {

constexpr int PK = 16;    // k per panel
constexpr int NT = 256;   // threads that copy it

// `bytes` (0 .. 4 or 16) of one copy, the rest of it zero; the _full ones all of it.
#ifdef __CUDACC__
__device__ __forceinline__ void copy16(uint32_t dst, const float *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void copy4(uint32_t dst, const float *src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void copy16_full(uint32_t dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src));
}
__device__ __forceinline__ void copy4_full(uint32_t dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src));
}
#else  // host compilers check the index arithmetic: dst, src, size, bytes
void host_copy(uint32_t, const void *, int, int);
inline void copy16(uint32_t dst, const float *src, int bytes) { host_copy(dst, src, 16, bytes); }
inline void copy4(uint32_t dst, const float *src, int bytes) { host_copy(dst, src, 4, bytes); }
inline void copy16_full(uint32_t dst, const float *src) { host_copy(dst, src, 16, 16); }
inline void copy4_full(uint32_t dst, const float *src) { host_copy(dst, src, 4, 4); }
#endif

// An operand panel of OUTER outer indices x 16 k lies in shared memory as
// [k][LD].  KCONT: element (o, k) at g[o*ld + k] in memory, else g[k*ld + o].
//
// Place of element (k, o) of a K-contiguous operand's panel.  From k = 8 on the
// pairs of a group of four outer indices are swapped: the stores of 16 k x 2 o
// then fall on 32 different banks (LD = 4 mod 32: 4 k + o repeats from k = 8),
// and a 16-byte read of a group only has its halves exchanged.
template <int LD>
__device__ __forceinline__ int panel_at(int k, int o) {
  static_assert(LD % 32 == 4, "bank pattern");
  return k * LD + (o ^ ((k >> 3) << 1));
}

// A thread's first element and its place: K-contiguous operands 16 k x 2 outer
// indices per warp, 4 bytes each; others along the outer index, 16 bytes each
// (VEC: base and ld allow it) or 4.
template <int OUTER, bool KCONT, bool VEC>
__device__ __forceinline__ void slot(int tid, int &o, int &k) {
  if (KCONT) {
    k = tid & 15;
    o = tid >> 4;
  } else if (VEC) {
    k = tid / (OUTER / 4);
    o = tid % (OUTER / 4) * 4;
  } else {
    k = tid / OUTER;
    o = tid % OUTER;
  }
}
// Copies per thread, and from one to the next: outer indices (KCONT) or k.
template <int OUTER, bool KCONT, bool VEC>
struct Steps {
  static constexpr int COUNT = OUTER * PK / NT / (!KCONT && VEC ? 4 : 1);
  static constexpr int STEP = KCONT ? NT / PK : NT * (VEC ? 4 : 1) / OUTER;
  static_assert(COUNT >= 1, "panel smaller than one copy per thread");
};
template <int OUTER, int LD, bool KCONT, bool VEC>
__device__ __forceinline__ uint32_t run_dst(int tid) {
  int o, k;
  slot<OUTER, KCONT, VEC>(tid, o, k);
  return (uint32_t)(KCONT ? panel_at<LD>(k, o) : k * LD + o) * 4u;
}
template <int OUTER, bool KCONT, bool VEC>
__device__ __forceinline__ size_t run_offset(int o0, int k0, int ld, int tid) {
  int o, k;
  slot<OUTER, KCONT, VEC>(tid, o, k);
  return KCONT ? (size_t)(o0 + o) * ld + (k0 + k) : (size_t)(k0 + k) * ld + (o0 + o);
}

// One panel at outer index o0 (zero from olim on) and k0 (zero from klim on).
template <int OUTER, int LD, bool KCONT, bool VEC>
__device__ __forceinline__ void load_panel(uint32_t dst, const float *__restrict__ g, int ld,
                                           int o0, int k0, int olim, int klim, int tid) {
  using S = Steps<OUTER, KCONT, VEC>;
  int o, k;
  slot<OUTER, KCONT, VEC>(tid, o, k);
  const float *p = g + run_offset<OUTER, KCONT, VEC>(o0, k0, ld, tid);
  const uint32_t d = dst + run_dst<OUTER, LD, KCONT, VEC>(tid);
#pragma unroll
  for (int e = 0; e < S::COUNT; ++e) {
    const int oe = o0 + o + (KCONT ? S::STEP * e : 0), ke = k0 + k + (KCONT ? 0 : S::STEP * e);
    const uint32_t de = d + (uint32_t)(S::STEP * e * (KCONT ? 1 : LD)) * 4u;
    const float *q = p + (size_t)(S::STEP * e) * ld;
    const int have = ke < klim ? olim - oe : 0;
    if constexpr (VEC && !KCONT) copy16(de, have > 0 ? q : g, have >= 4 ? 16 : have > 0 ? 4 * have : 0);
    else copy4(de, have > 0 ? q : g, have > 0 ? 4 : 0);
  }
}

// The same panel when it lies wholly inside the operand: from the thread's
// running pointer p, to its place d (run_dst added).
template <int OUTER, int LD, bool KCONT, bool VEC>
__device__ __forceinline__ void run_panel(uint32_t d, const float *p, int ld) {
  using S = Steps<OUTER, KCONT, VEC>;
  const size_t step = (size_t)S::STEP * ld;
#pragma unroll
  for (int e = 0; e < S::COUNT; ++e) {
    const uint32_t de = d + (uint32_t)(S::STEP * e * (KCONT ? 1 : LD)) * 4u;
    if constexpr (VEC && !KCONT) copy16_full(de, p);
    else copy4_full(de, p);
    p += step;
  }
}

}  // namespace f32copy
}  // namespace b2
