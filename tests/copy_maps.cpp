// CPU check of the operand copies of csrc/fp32_copy.cuh and csrc/fp64_copy.cuh, compiled
// from those headers: every copy is aligned and reads inside the operand, and every
// element that a fragment reads lies where the fragment looks for it, zero beyond the
// matrix.  Prints the first violation and exits 1.
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <vector>

#define __device__
#define __host__
#define __forceinline__ inline
#define __restrict__
using std::min;
#include "fp32_copy.cuh"
#include "fp64_copy.cuh"

static unsigned char g_smem[1 << 20];
static const unsigned char *g_lo, *g_hi;  // the operand
static const char *g_what = "";
static void fail(const char *why, long a, long b) {
  printf("%s: %s (%ld, %ld)\n", g_what, why, a, b);
  exit(1);
}
static void copy(uint32_t dst, const void *src, int size, int bytes) {
  const unsigned char *p = (const unsigned char *)src;
  if (dst % size || (uintptr_t)p % size) fail("misaligned copy", dst, (long)((uintptr_t)p % 64));
  if (bytes < 0 || bytes > size || dst + size > sizeof(g_smem)) fail("copy size", bytes, dst);
  if (bytes && (p < g_lo || p + bytes > g_hi)) fail("read outside the operand", p - g_lo, bytes);
  memset(g_smem + dst, 0, size);
  memcpy(g_smem + dst, p, bytes);
}
namespace b2 {
namespace f32copy {
void host_copy(uint32_t d, const void *s, int size, int bytes) { copy(d, s, size, bytes); }
}  // namespace f32copy
namespace f64copy {
void host_copy(uint32_t d, const void *s, int size, int bytes) { copy(d, s, size, bytes); }
}  // namespace f64copy
}  // namespace b2

// An operand of `outer` x `kn` in memory of its own, `off` elements off a 64-byte
// boundary; element (o, k) holds o * 4096 + k + 1.
template <typename T>
struct Operand {
  std::vector<T> buf;
  T *g;
  int ld;
  Operand(int outer, int kn, bool kcont, int off, int pad) : buf() {
    const int len = kcont ? kn : outer, rows = kcont ? outer : kn;
    ld = len + pad;
    buf.assign((size_t)ld * rows + off + 64, (T)-1);
    T *base = (T *)(((uintptr_t)buf.data() + 63) & ~(uintptr_t)63);
    g = base + off;
    for (int o = 0; o < outer; ++o)
      for (int k = 0; k < kn; ++k)
        g[kcont ? (size_t)o * ld + k : (size_t)k * ld + o] = (T)(o * 4096 + k + 1);
    g_lo = (const unsigned char *)g;
    g_hi = (const unsigned char *)(g + (size_t)(rows - 1) * ld + len);
  }
};
static double want(int o, int k, int olim, int klim) {
  return o < olim && k < klim ? o * 4096 + k + 1 : 0;
}

template <int OUTER, bool KCONT, bool VEC>
void check32(int outer, int kn, int off, int pad) {
  using namespace b2::f32copy;
  constexpr int LD = OUTER + 4;
  Operand<float> A(outer, kn, KCONT, off, pad);
  if (VEC && ((uintptr_t)A.g % 16 || A.ld % 4)) return;  // not chosen by the kernels
  for (int o0 = 0; o0 < outer; o0 += OUTER)
    for (int k0 = 0; k0 < kn; k0 += PK)
      for (int run = 0; run < 2; ++run) {
        if (run && (o0 + OUTER > outer || k0 + PK > kn)) continue;  // inside tiles only
        memset(g_smem, 0xff, sizeof(g_smem));
        for (int tid = 0; tid < NT; ++tid) {
          if (run)
            run_panel<OUTER, LD, KCONT, VEC>(run_dst<OUTER, LD, KCONT, VEC>(tid),
                                             A.g + run_offset<OUTER, KCONT, VEC>(o0, k0, A.ld, tid),
                                             A.ld);
          else load_panel<OUTER, LD, KCONT, VEC>(0, A.g, A.ld, o0, k0, outer, kn, tid);
        }
        const float *sm = (const float *)g_smem;
        for (int k = 0; k < PK; ++k)
          for (int o = 0; o < OUTER; ++o) {
            // what the kernels read: groups of four, halves exchanged from k = 8 on
            const int at = k * LD + (o & ~3) + ((o & 3) ^ (KCONT && k >= 8 ? 2 : 0));
            if (sm[at] != (float)want(o0 + o, k0 + k, outer, kn)) fail("fp32 panel", o0 + o, k0 + k);
          }
      }
}

// One FP64 operand's stages as the kernels choose their copies (load_stage, Op64).
template <int OUTER, bool KCONT, int NT>
void check64(int outer, int kn, int off, int pad) {
  using namespace b2::f64copy;
  constexpr int BK = 16, LEN = KCONT ? BK : OUTER, ROWS = KCONT ? OUTER : BK, PITCH = LEN + 4;
  constexpr int CPR = LEN / 2, CH = tile_chunks<OUTER, BK, NT>();
  Operand<double> A(outer, kn, KCONT, off, pad);
  const double *g = A.g;
  const int ld = A.ld;
  for (int kbeg = 0; kbeg < kn; kbeg += 32)
    for (int o0 = 0; o0 < outer; o0 += OUTER) {
      const int kend = std::min(kn, kbeg + 32);
      for (int k0 = kbeg; k0 < kend; k0 += BK)
        for (int form = 0; form < 3; ++form) {  // bounds-checked, edge, whole
          const bool full = k0 + BK <= kend, inside = o0 + OUTER <= outer;
          const bool first = k0 == kbeg && (KCONT ? o0 : kbeg) == 0 && ((uintptr_t)g & 8);
          if (form == 1 && (!full || first)) continue;
          if (form == 2 && (!full || first || !inside)) continue;
          memset(g_smem, 0xff, sizeof(g_smem));
          for (int tid = 0; tid < NT; ++tid) {
            const int r0 = KCONT ? o0 : k0, sh = row_shift(g, ld, r0 + tid / CPR);
            const double *p = g + run_offset<OUTER, BK, KCONT>(o0, k0, ld, tid) - sh;
            const uint32_t d = run_dst<OUTER, BK, KCONT>(tid);
            for (int c = 0; c < CH; ++c) {
              const uint32_t dc = d + c * run_dst_step<OUTER, BK, KCONT, NT>();
              const double *pc = p + c * run_step<OUTER, BK, KCONT, NT>(ld);
              if (form == 2) cp_async_full<16>(dc, pc);
              else if (form == 1)
                cp_async_edge(dc, pc, g, edge_bytes<OUTER, BK, KCONT, NT>(o0, outer, tid, sh, c));
              else
                load_chunk<OUTER, BK, KCONT, true, NT>(0, g, ld, o0, k0, outer, kend, tid, c, sh);
            }
            if (form == 2) {
              if (tid < ROWS && row_shift(g, ld, r0 + tid))
                cp_async<16>(run_tail_dst<OUTER, BK, KCONT>(tid),
                             g + run_tail<OUTER, BK, KCONT>(o0, k0, ld, tid),
                             (KCONT ? k0 + BK < kend : o0 + OUTER < outer) ? 16 : 8);
            } else {
              load_tails<OUTER, BK, KCONT, NT>(0, g, ld, o0, k0, outer, kend, tid);
            }
          }
          const double *sm = (const double *)g_smem;
          for (int o = 0; o < OUTER; ++o)
            for (int k = 0; k < BK; ++k) {
              const int r = KCONT ? o : k, c = KCONT ? k : o;
              const int fs = row_shift(g, ld, r);  // a fragment's: its row within the tile
              if (sm[r * PITCH + c + fs] != want(o0 + o, k0 + k, outer, kend))
                fail("fp64 tile", o0 + o, k0 + k);
            }
        }
    }
}

int main() {
  const int sizes[][2] = {{1, 1}, {63, 15}, {64, 16}, {65, 17}, {128, 32}, {130, 47}, {257, 64}, {31, 33}};
  for (auto &s : sizes)
    for (int off = 0; off < 5; ++off)
      for (int pad = 0; pad < 5; ++pad) {
        const int o = s[0], k = s[1];
        g_what = "fp32 128";
        check32<128, true, false>(o, k, off, pad), check32<128, false, false>(o, k, off, pad);
        check32<128, true, true>(o, k, off, pad), check32<128, false, true>(o, k, off, pad);
        g_what = "fp32 64";
        check32<64, true, false>(o, k, off, pad), check32<64, false, false>(o, k, off, pad);
        check32<64, true, true>(o, k, off, pad), check32<64, false, true>(o, k, off, pad);
        g_what = "fp64 64 x 16, 128 threads";
        check64<64, true, 128>(o, k, off, pad), check64<64, false, 128>(o, k, off, pad);
        g_what = "fp64 32 x 16, 128 threads";
        check64<32, true, 128>(o, k, off, pad), check64<32, false, 128>(o, k, off, pad);
        g_what = "fp64 64 x 16, 256 threads";
        check64<64, true, 256>(o, k, off, pad), check64<64, false, 256>(o, k, off, pad);
        g_what = "fp64 128 x 16, 256 threads";
        check64<128, true, 256>(o, k, off, pad), check64<128, false, 256>(o, k, off, pad);
      }
  printf("ok\n");
  return 0;
}
