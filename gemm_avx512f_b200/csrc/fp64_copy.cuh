// fp64_copy.cuh -- asynchronous copies of FP64 operand tiles into shared memory
// (the plain FP64 GEMM and the grouped GEMM's FP64 tiles).
#pragma once

#include <stdint.h>

namespace b2 {
namespace f64copy {

#ifdef __CUDACC__
template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void *src, int src_bytes) {
  if constexpr (BYTES == 16) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src),
                 "r"(src_bytes));
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src),
                 "r"(src_bytes));
  }
}
template <int BYTES>
__device__ __forceinline__ void cp_async_full(uint32_t dst, const void *src) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}
#else  // host compilers check the index arithmetic: dst, src, size, bytes
void host_copy(uint32_t, const void *, int, int);
template <int BYTES>
inline void cp_async(uint32_t dst, const void *src, int src_bytes) {
  host_copy(dst, src, BYTES, src_bytes);
}
template <int BYTES>
inline void cp_async_full(uint32_t dst, const void *src) {
  host_copy(dst, src, BYTES, BYTES);
}
#endif

// Operand tiles are copied as 16-byte chunks (two elements) of the rows that are
// contiguous in memory.  SH: the operand's base or leading dimension is odd, so
// rows may start 8 bytes off a 16-byte boundary; such a row is copied from one
// element earlier (one chunk more) and sits one element later in its shared
// row, whose padding has room for both.  Tiles start at even elements, so a
// row's shift is row_shift(p0, ld, row), and the row distances between one
// thread's chunks, and between its fragment reads, are even: the shift is a
// constant of the thread.  Odd leading dimensions took twice the copies, of 8
// bytes, before: 2501x1777x1999 671 -> 647 us on B200 (578 with even ones: the
// shifted rows' shared reads meet 2-way bank conflicts).
__device__ __forceinline__ int row_shift(const double *g, int ld, int row) {
  return (int)(((reinterpret_cast<uintptr_t>(g) >> 3) + (unsigned)row * (unsigned)ld) & 1u);
}

// Chunk i of an OUTER x BK operand tile.  Element (o, k) of the operand lives
// at g[o*ld + k] when KCONT (k contiguous in memory) else g[k*ld + o].  Shared
// layout: KCONT -> [o][BK+4], else [k][OUTER+4].
template <int OUTER, int BK, int NT>
__host__ __device__ constexpr int tile_chunks() {
  static_assert(OUTER * BK / 2 % NT == 0, "tile/thread mismatch");
  return OUTER * BK / 2 / NT;
}
// One bounds-checked chunk: elements e0, e0 + 1 (e0 may be -1: not needed) of
// row `row`, zero beyond the row's lim elements and for rows >= rows.
template <bool SH>
__device__ __forceinline__ void copy_pair(uint32_t dst, const double *__restrict__ g, int ld,
                                          int row, int rows, int e0, int lim) {
  int valid = row < rows ? min(2, lim - e0) : 0;
  valid = valid < 0 ? 0 : valid;
  if (SH && e0 < 0 && row == 0) {  // the element before the operand's first is not read
    cp_async<8>(dst + 8, g, valid > 1 ? 8 : 0);
    return;
  }
  const double *none = reinterpret_cast<const double *>(reinterpret_cast<uintptr_t>(g) &
                                                        ~(uintptr_t)15);
  cp_async<16>(dst, valid ? g + (size_t)row * ld + e0 : none, valid * 8);
}
template <int OUTER, int BK, bool KCONT, bool SH, int NT>
__device__ __forceinline__ void load_chunk(uint32_t sbase, const double *__restrict__ g, int ld,
                                           int o0, int k0, int olim, int klim, int tid, int i,
                                           int sh) {
  const int c = tid + i * NT;
  constexpr int CPR = (KCONT ? BK : OUTER) / 2;
  const int hi = c / CPR, lo = (c % CPR) * 2;
  const uint32_t dst = sbase + (uint32_t)(hi * (KCONT ? BK + 4 : OUTER + 4) + lo) * 8u;
  if (KCONT) copy_pair<SH>(dst, g, ld, o0 + hi, olim, k0 + lo - sh, klim);
  else copy_pair<SH>(dst, g, ld, k0 + hi, klim, o0 + lo - sh, olim);
}
// The chunk past the end of each shifted row (its first element is the row's last).
template <int OUTER, int BK, bool KCONT, int NT>
__device__ __forceinline__ void load_tails(uint32_t sbase, const double *__restrict__ g, int ld,
                                           int o0, int k0, int olim, int klim, int tid) {
  constexpr int ROWS = KCONT ? OUTER : BK, LEN = KCONT ? BK : OUTER;
  static_assert(ROWS <= NT, "one tail per thread");
  const int row = (KCONT ? o0 : k0) + tid;
  if (tid >= ROWS || !row_shift(g, ld, row)) return;
  const uint32_t dst = sbase + (uint32_t)(tid * (LEN + 4) + LEN) * 8u;
  if (KCONT) copy_pair<true>(dst, g, ld, row, olim, k0 + LEN - 1, klim);
  else copy_pair<true>(dst, g, ld, row, klim, o0 + LEN - 1, olim);
}

// The same map for tiles without an edge: element offset of the thread's chunk
// 0 in the operand, its shared-memory byte offset, and the distances from one
// chunk to the next.
template <int OUTER, int BK, bool KCONT>
__device__ __forceinline__ size_t run_offset(int o0, int k0, int ld, int tid) {
  constexpr int CPR = (KCONT ? BK : OUTER) / 2;
  const int hi = tid / CPR, lo = (tid % CPR) * 2;
  return KCONT ? (size_t)(o0 + hi) * ld + (k0 + lo) : (size_t)(k0 + hi) * ld + (o0 + lo);
}
template <int OUTER, int BK, bool KCONT>
__device__ __forceinline__ uint32_t run_dst(int tid) {
  constexpr int CPR = (KCONT ? BK : OUTER) / 2;
  return (uint32_t)((tid / CPR) * (KCONT ? BK + 4 : OUTER + 4) + (tid % CPR) * 2) * 8u;
}
template <int OUTER, int BK, bool KCONT, int NT>
__device__ __forceinline__ size_t run_step(int ld) {
  constexpr int CPR = (KCONT ? BK : OUTER) / 2;
  static_assert(NT % CPR == 0 && (NT / CPR) % 2 == 0, "an even number of whole rows per step");
  return (size_t)(NT / CPR) * ld;
}
template <int OUTER, int BK, bool KCONT, int NT>
__host__ __device__ constexpr uint32_t run_dst_step() {
  return (uint32_t)(NT / ((KCONT ? BK : OUTER) / 2) * (KCONT ? BK + 4 : OUTER + 4)) * 8u;
}

// A tile that reaches past the operand's outer limit, K block inside: a chunk's
// copies from the same running pointers need only its byte count, from the
// thread's rows left (KCONT) or its pair's place on the row.
template <int OUTER, int BK, bool KCONT, int NT>
__device__ __forceinline__ int edge_bytes(int o0, int olim, int tid, int sh, int c) {
  constexpr int CPR = (KCONT ? BK : OUTER) / 2;
  if (KCONT) return c * (NT / CPR) < olim - o0 - tid / CPR ? 16 : 0;
  const int have = olim - (o0 + (tid % CPR) * 2 - sh);
  return have >= 2 ? 16 : have == 1 ? 8 : 0;
}
__device__ __forceinline__ void cp_async_edge(uint32_t dst, const double *src, const double *g,
                                              int bytes) {
  const double *none = reinterpret_cast<const double *>(reinterpret_cast<uintptr_t>(g) &
                                                        ~(uintptr_t)15);
  cp_async<16>(dst, bytes ? src : none, bytes);
}

// Operand offset and shared byte offset of the chunk past the end of row tid.
template <int OUTER, int BK, bool KCONT>
__device__ __forceinline__ size_t run_tail(int o0, int k0, int ld, int tid) {
  return KCONT ? (size_t)(o0 + tid) * ld + (k0 + BK - 1) : (size_t)(k0 + tid) * ld + (o0 + OUTER - 1);
}
template <int OUTER, int BK, bool KCONT>
__device__ __forceinline__ uint32_t run_tail_dst(int tid) {
  constexpr int LEN = KCONT ? BK : OUTER;
  return (uint32_t)(tid * (LEN + 4) + LEN) * 8u;
}

}  // namespace f64copy
}  // namespace b2
