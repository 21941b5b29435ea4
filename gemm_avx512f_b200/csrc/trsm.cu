// trsm.cu -- blocked triangular solve on the GPU (dtrsm_).
//
// The reference ships DTRSM solve kernels for packed panels
// (OpenBLAS-like_implementation/dtrsm_16x4/dtrsm_kernel_16x4_skylakex.S:1863-2536,
// semantics in dtrsm_kernel_16x4_tester.c:66-199: add the incoming GEMM update,
// solve against the triangle whose diagonal is stored inverted, write X back),
// driven by an OpenBLAS trsm driver.  Here the driver is a recursive split of
// the triangle: solve the leading part, update the trailing right-hand sides
// with one large GEMM (plain FP64 DMMA or the INT8 Ozaki emulation), solve the
// trailing part.  The 128x128 diagonal blocks of op(A) are inverted up front in
// one batched launch (trtri_batched_kernel, the diagonal inverted first, the
// reference kernels' convention), and a leaf of the recursion -- up to 512 rows
// -- is one launch (trsm_leaf_kernel) whose CTAs each take a strip of right-hand
// sides through the leaf's blocks: X_k = inv(T_kk)(Z_k - sum_j T_kj X_j).
// Trailing updates use the INT8 Ozaki GEMM when requested and the product is
// large enough to amortise its slicing passes, plain FP64 otherwise.
//
// Side 'R' is solved as its transpose: X op(A) = B is op(A)^T X^T = B^T, so T
// below is op(A) (side 'L') or its transpose (side 'R'), T(i, j) = A[i*rs + j*cs]
// with one of rs, cs 1 and the other lda, and right-hand side r is column r or
// row r of B.
#include <type_traits>

#include "b2_methods.cuh"
#include "b2_profile.cuh"

namespace b2 {
namespace {

constexpr int TB = 128;        // diagonal block order
constexpr int TB_LD = TB + 2;  // shared column stride (2-way conflicts at most for all reads of it)
constexpr int TI_NT = 512;     // threads of the inversion
constexpr int TI_K = 16;       // rows it solves at a time
constexpr int TI_PLD = TB + 4; // stride of the copied columns (conflict-free DMMA fragments)

// Invert every diagonal block T_b = T[kb:kb+bs, kb:kb+bs] (lower or upper, unit
// or not); block b goes to Tinv + b*TB*TB (column-major, ld TB, zero outside the
// triangle and beyond bs, and on the diagonal, whose inverse goes to dinv + b*TB; a
// block of order up to keep_diag keeps it).
// An upper block is inverted as the lower one it is
// with both indices reversed.  Substitution against the identity in shared
// memory, in place, 16 columns of T at a time (copied aside as [k][row]): the 16
// rows of their diagonal block are solved, one thread per column, and taken off
// the sums of all later rows, which replace T as its columns are used up.
// Each element is the same chain as plain substitution column by column, k
// ascending from the column's own index: a zero of the triangle is never
// multiplied (it would turn an infinity or a NaN of T into NaN in columns that
// do not depend on it), and nothing is lost to products of inverses (inversion
// by doubling: 1.5-2x the backward error on LU factors).
// Bound: FP64 latency of one CTA per block, about 2.3 us for 16 rows.  A solve of
// order 128 for 8 right-hand sides takes 31 us, with inversion by doubling 28, with
// one thread per column of the block 198; of order 16, 11 against 24 and 24 (B200).
using Yes = std::integral_constant<bool, true>;
using No = std::integral_constant<bool, false>;
__device__ __forceinline__ double &tel(double *T, int i, int j) { return T[j * TB_LD + i]; }

__global__ void __launch_bounds__(TI_NT)
    trtri_batched_kernel(const double *__restrict__ A, long long rs, long long cs, int n, int lower,
                         int unit, int keep_diag, double *__restrict__ Tinv,
                         double *__restrict__ dinv) {
  extern __shared__ __align__(16) double tsm[];
  double *T = tsm;                      // T(i, j) at [j*TB_LD + i], then sums, then the inverse
  double *pan = tsm + TB * TB_LD;       // 16 columns of T, [k][row], this step's and the next's
  double *inv = pan + 2 * TI_K * TI_PLD;  // inverted diagonal
  const int kb = blockIdx.x * TB, bs = min(TB, n - kb), tid = threadIdx.x;
  // lower triangle of the (index-reversed if upper) block, identity beyond bs,
  // zeros above the diagonal
  for (int base = tid; base < TB * TB; base += 16 * TI_NT) {
    double v[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      // consecutive threads along the contiguous dimension of A
      const int idx = base + e * TI_NT, u = idx % TB, w = idx / TB;
      const int i = rs == 1 ? u : w, j = rs == 1 ? w : u;
      v[e] = i == j ? 1.0 : 0.0;
      if (i < bs && j < bs && i >= j) {
        const int gi = lower ? i : bs - 1 - i, gj = lower ? j : bs - 1 - j;
        if (i != j || !unit) v[e] = A[(kb + gi) * rs + (kb + gj) * cs];
      }
    }
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const int idx = base + e * TI_NT, u = idx % TB, w = idx / TB;
      tel(T, rs == 1 ? u : w, rs == 1 ? w : u) = v[e];
    }
  }
  __syncthreads();
  const int rows = (bs + TI_K - 1) / TI_K * TI_K;  // those beyond bs are the identity's
  const int lane = tid & 31, warp = tid >> 5;
  auto panel = [&](int k0) { return pan + (k0 / TI_K & 1) * TI_K * TI_PLD; };
  auto copy_panel = [&](int k0, int t0, int nt) {
    double *p = panel(k0);
    for (int idx = t0; idx < TI_K * TB; idx += nt)
      if (idx % TB >= k0) p[idx / TB * TI_PLD + idx % TB] = tel(T, idx % TB, k0 + idx / TB);
  };
  // rows k0 .. k0 + 15 of column tid < k0 + 16 (the columns after it are zero);
  // EDGE: the warp has columns of the diagonal 16 x 16
  auto solve = [&](auto edge, int k0) {
    constexpr bool EDGE = decltype(edge)::value;
    const double *p = panel(k0);
    double x[TI_K];
    const int own = tid - k0;  // of the diagonal 16 x 16: the rows before it are zero
#pragma unroll
    for (int r = 0; r < TI_K; ++r)
      x[r] = !EDGE || own < 0 ? tel(T, k0 + r, tid) : r == own ? 1.0 : 0.0;
#pragma unroll
    for (int r = 0; r < TI_K; ++r) {
      if (!EDGE || r >= own) {
        x[r] *= inv[k0 + r];
#pragma unroll
        for (int q = r + 1; q < TI_K; ++q) x[q] = fma(-p[r * TI_PLD + k0 + q], x[r], x[q]);
      }
    }
#pragma unroll
    for (int r = 0; r < TI_K; ++r) tel(T, k0 + r, tid) = x[r];
  };
  // takes rows k0 .. k0 + 15 off the sums of rows [r0, r1), warps w0 to the last:
  // 16 x 8 outputs at a time on DMMA (a chain of multiply-adds, k ascending), the
  // columns of the diagonal 16 x 16, whose first sums start at their own index, one
  // column and 8 rows per lane
  auto update = [&](int k0, int r0, int r1, int w0) {
    const double *p = panel(k0);
    const int rblocks = (r1 - r0) / 16, items = rblocks * (k0 / 8 + 1);
    for (int it = warp - w0; it < items; it += TI_NT / 32 - w0) {
      const int i0 = r0 + it % rblocks * 16, c = it / rblocks;
      if (c == 0) {
        const int i = i0 + (lane >> 4) * 8, j = k0 + (lane & 15);
        double acc[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r] = 0.0;
#pragma unroll
        for (int k = 0; k < TI_K; ++k) {
          const double x = tel(T, k0 + k, j);
          const double2 *t2 = reinterpret_cast<const double2 *>(p + k * TI_PLD + i);
          if (k0 + k >= j) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              const double2 t = t2[r];
              acc[2 * r] = fma(-t.x, x, acc[2 * r]);
              acc[2 * r + 1] = fma(-t.y, x, acc[2 * r + 1]);
            }
          }
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) tel(T, i + r, j) = acc[r];
      } else {
        const int g = lane >> 2, t = lane & 3, j0 = (c - 1) * 8;
        double acc[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[v] = tel(T, i0 + g + 8 * (v >> 1), j0 + 2 * t + (v & 1));
#pragma unroll
        for (int k = 0; k < TI_K; k += 4) {
          const double a0 = -p[(k + t) * TI_PLD + i0 + g], a1 = -p[(k + t) * TI_PLD + i0 + g + 8];
          const double b = tel(T, k0 + k + t, j0 + g);
          asm volatile(
              "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
              "{%0,%1,%2,%3};\n"
              : "+d"(acc[0]), "+d"(acc[1]), "+d"(acc[2]), "+d"(acc[3])
              : "d"(a0), "d"(a1), "d"(b));
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) tel(T, i0 + g + 8 * (v >> 1), j0 + 2 * t + (v & 1)) = acc[v];
      }
    }
  };
  if (tid < TB) inv[tid] = 1.0 / tel(T, tid, tid);
  copy_panel(0, tid, TI_NT);
  __syncthreads();
  if (tid < TI_K) solve(Yes{}, 0);
  __syncthreads();
  // the next 16 rows' sums, then those rows beside the sums of the rows after them
  for (int k0 = 0, k1 = TI_K; k1 < rows; k0 = k1, k1 += TI_K) {
    update(k0, k1, k1 + TI_K, 0);
    copy_panel(k1, tid, TI_NT);
    __syncthreads();
    if (tid >= TB) update(k0, k1 + TI_K, rows, 4);
    else if (warp * 32 + 32 <= k1) solve(No{}, k1);
    else if (tid < k1 + TI_K) solve(Yes{}, k1);
    __syncthreads();
  }
  double *out = Tinv + (long long)blockIdx.x * TB * TB;
  for (int idx = tid; idx < TB * TB; idx += TI_NT) {
    const int i = idx % TB, j = idx / TB;  // element (i, j) of the stored inverse
    double v = 0.0;
    if (i < bs && j < bs) {
      const int li = lower ? i : bs - 1 - i, lj = lower ? j : bs - 1 - j;
      if (li > lj || (li == lj && bs <= keep_diag)) v = tel(T, li, lj);
    }
    out[idx] = v;
  }
  if (tid < TB) dinv[blockIdx.x * TB + tid] = tid < bs ? inv[lower ? tid : bs - 1 - tid] : 0.0;
}

// ------------------------------------------------------------------ leaf --
// Rows [0, nr) of a leaf for W right-hand sides per CTA, on DMMA m16n8k4: the
// strip lives in shared memory as Z[rhs][row] through all of the leaf's steps,
// each a 128 x W x 128 product of a block of T (or an inverted diagonal block)
// and 128 solved rows.  A warp owns 16 rows of the product and brings its own
// rows of T, 32 columns at a time, through a private cp.async ring (no barrier
// of the CTA; the copies run ahead across steps, since T does not depend on the
// solution).  Lane (g, t) uses the 2 x 2 element blocks at rows 2g, 2g + 1 and
// columns 8s + 2t, + 1 -- the MMA's rows g, g + 8 and the k = t of two K steps
// -- so that either orientation of T is copied and read 16 bytes at a time, and
// Z two rows at a time.
// Bound: L2 -> SM (128 KB of T per step, 64 bytes per clock: 1.07 us) and, wider
// than 8, the FP64 pipe; reached: 25, 41 and 76 us for 512 rows at 8, 16 and 32
// (B200; 24, 37 and 70 with one chain of additions through a step).  Each 128-row block
// as its own memset, GEMM, reduction and copy, with the updates between them as further
// launches, took 68 us for 512 rows and 1024 right-hand sides; dtrsm 4096 x 1024
// 1374 -> 755 us in all.
constexpr int LEAF_BLOCKS = 4;  // 512 rows
constexpr int LEAF_COLS = 32;   // columns of T per ring stage
template <int W>
struct LeafSmem {
  static constexpr int STAGES = W == 8 ? 6 : W == 16 ? 5 : 3;
  static constexpr int P = LEAF_BLOCKS * TB + 8;  // Z[r * P + i]
  static constexpr int WARP_STAGE = 16 * LEAF_COLS;  // doubles
  static constexpr int BYTES = (W * P + 8 * STAGES * WARP_STAGE) * (int)sizeof(double);
};
// Shared offset (doubles) of element (row, col) of a warp's stage: T columns (or
// rows, by_row) contiguous, 16-byte chunks swizzled so that the lanes' 16-byte
// reads meet no bank conflict.
template <bool BY_ROW>
__device__ __forceinline__ int leaf_at(int row, int col) {
  return BY_ROW ? row * LEAF_COLS + ((((col >> 1) ^ (((row >> 1) & 1) << 2)) << 1) | (col & 1))
                : col * 16 + ((((row >> 1) ^ (((col >> 1) & 3) << 1)) << 1) | (row & 1));
}

// ROWS: T's rows are contiguous in A (cs = 1); the inverted blocks' columns are.
template <int W, bool ROWS>
__global__ void __launch_bounds__(256, 1)
    trsm_leaf_kernel(const double *__restrict__ A, long long rs, long long cs, int forward, int nr,
                     const double *__restrict__ Tinv, const double *__restrict__ dinv,
                     double *__restrict__ B, long long si, long long sr, int nrhs) {
  using L = LeafSmem<W>;
  constexpr int P = L::P, STAGES = L::STAGES, NT = W / 8;
  extern __shared__ __align__(16) double Z[];
  const int nb = (nr + TB - 1) / TB;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3, wm = warp * 16;
  const int r0 = blockIdx.x * W;
  double *ring = Z + W * P + warp * STAGES * L::WARP_STAGE;
  const uint32_t ring_u = (uint32_t)__cvta_generic_to_shared(ring);

  // The steps in order: for each block k (ascending when forward), the blocks j
  // solved before it, then its inverse (j = k).  q-th block: forward ? q : nb-1-q.
  const int stages = nb * (nb + 1) / 2 * (TB / LEAF_COLS);
  // 16-byte copies of T: its columns' (rows') starts are 16-byte aligned
  const bool vec = (reinterpret_cast<uintptr_t>(A) & 15) == 0 && ((rs == 1 ? cs : rs) & 1) == 0;
  int pk = 0, pj = 0, ph = 0, pslot = 0, issued = 0;  // next stage to copy
  auto copy_block = [&](auto by, const double *p, long long ld, uint32_t dst, bool whole, int rlim,
                        int clim) {
    constexpr bool BY = decltype(by)::value;  // ld: from one contiguous line to the next
    if (whole) {
      const int line = BY ? lane >> 4 : lane >> 3, at = (BY ? lane & 15 : lane & 7) * 2;
      const double *q = p + (wm * (BY ? ld : 1) + line * ld + at);
#pragma unroll
      for (int e = 0; e < 8; ++e)  // 256 chunks of two elements
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                         dst + (uint32_t)(BY ? leaf_at<true>(line + 2 * e, at)
                                             : leaf_at<false>(at, line + 4 * e)) * 8u),
                     "l"(q + (BY ? 2 : 4) * e * ld));
    } else {
#pragma unroll 4
      for (int e = 0; e < 16; ++e) {
        const int c = lane + 32 * e;
        const int row = BY ? c >> 5 : c & 15, col = BY ? c & 31 : c >> 4;
        const bool in = wm + row < rlim && col < clim;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(
                         dst + (uint32_t)leaf_at<BY>(row, col) * 8u),
                     "l"(in ? p + (BY ? (wm + row) * ld + col : wm + row + col * ld) : A),
                     "r"(in ? 8 : 0));
      }
    }
  };
  auto copy_stage = [&]() {
    if (issued < stages) {
      const int k = forward ? pk : nb - 1 - pk, j = forward ? pj : nb - 1 - pj;
      const uint32_t dst = ring_u + (uint32_t)(pslot * L::WARP_STAGE) * 8u;
      const int c0 = ph * LEAF_COLS;
      if (pk == pj) {
        copy_block(No{}, Tinv + (long long)k * TB * TB + c0 * TB, (long long)TB, dst, true, 0, 0);
      } else {
        const int rlim = nr - k * TB, clim = nr - j * TB;
        copy_block(std::integral_constant<bool, ROWS>{},
                   A + k * TB * rs + (long long)(j * TB + c0) * cs, ROWS ? rs : cs, dst,
                   vec && rlim >= TB && clim >= TB, rlim, clim - c0);
      }
      ++issued;
      if (++pslot == STAGES) pslot = 0;
      if (++ph == TB / LEAF_COLS) {
        ph = 0;
        if (pj == pk) ++pk, pj = 0;
        else ++pj;
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) copy_stage();

  for (int idx = tid; idx < nb * TB * W; idx += 256) {
    // consecutive threads along B's contiguous dimension
    const int i = si == 1 ? idx % (nb * TB) : idx / W, r = si == 1 ? idx / (nb * TB) : idx % W;
    Z[r * P + i] = (i < nr && r0 + r < nrhs) ? B[i * si + (r0 + r) * sr] : 0.0;
  }
  // A DMMA waits for the one before it on the same accumulator: four
  // independent chains (K steps dealt out in turn).  Every 16 k a chain goes to the
  // sum: the error of a product of 128 is 3.6 u, not the 8 u of one chain (the slices of
  // a GEMM of that size are no longer either).
  constexpr int SETS = NT >= 4 ? 1 : 4 / NT;
  double acc[SETS][NT][4], sum[NT][4];
  auto end_chains = [&]() {
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        double x = acc[0][n][v];
#pragma unroll
        for (int c = 1; c < SETS; ++c) x += acc[c][n][v];
        sum[n][v] += x;
#pragma unroll
        for (int c = 0; c < SETS; ++c) acc[c][n][v] = 0.0;
      }
  };
  // Element (n, v) of a warp's fragment: row wm + 2g + (v >> 1), rhs 8n + 2t + (v & 1)
  __syncthreads();
  int slot = 0;
  for (int kq = 0; kq < nb; ++kq) {
    const int k = forward ? kq : nb - 1 - kq;
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        sum[n][v] = 0.0;
#pragma unroll
        for (int c = 0; c < SETS; ++c) acc[c][n][v] = 0.0;
      }
    double *zk = Z + k * TB + wm + 2 * g;
    const double d[2] = {dinv[k * TB + wm + 2 * g], dinv[k * TB + wm + 2 * g + 1]};
    for (int jq = 0; jq <= kq; ++jq) {
      const bool diag = jq == kq;
      if (diag && kq > 0) {  // all updates of block k are in: Z_k -= their sum
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            zk[(8 * n + 2 * t + (v & 1)) * P + (v >> 1)] -= sum[n][v];
            sum[n][v] = 0.0;
          }
        __syncthreads();
      }
      const double *zb = Z + (forward ? jq : nb - 1 - jq) * TB + 2 * t + g * P;
      auto mac_block = [&](auto by) {
        constexpr bool BY = decltype(by)::value;
        for (int h = 0; h < TB / LEAF_COLS; ++h) {
          asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
          __syncwarp();  // this stage is in; every lane is done with the slot refilled next
          const double *f = ring + slot * L::WARP_STAGE;
          // rows 2g, 2g + 1 x columns 8s + 2t, + 1 (BY: the two rows; else the two columns)
          double2 lo[LEAF_COLS / 8], hi[LEAF_COLS / 8];
#pragma unroll
          for (int s = 0; s < LEAF_COLS / 8; ++s) {
            lo[s] = *reinterpret_cast<const double2 *>(f + leaf_at<BY>(2 * g, 8 * s + 2 * t));
            hi[s] = *reinterpret_cast<const double2 *>(
                f + (BY ? leaf_at<BY>(2 * g + 1, 8 * s + 2 * t) : leaf_at<BY>(2 * g, 8 * s + 2 * t + 1)));
          }
          copy_stage();
#pragma unroll
          for (int s = 0; s < LEAF_COLS / 8; ++s) {
            const double a00 = lo[s].x, a10 = BY ? hi[s].x : lo[s].y;
            const double a01 = BY ? lo[s].y : hi[s].x, a11 = hi[s].y;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
              const double2 b =
                  *reinterpret_cast<const double2 *>(zb + n * 8 * P + h * LEAF_COLS + 8 * s);
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                double(&c)[4] = acc[(2 * s + e) % SETS][n];
                asm volatile(
                    "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, "
                    "{%6}, {%0,%1,%2,%3};\n"
                    : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                    : "d"(e ? a01 : a00), "d"(e ? a11 : a10), "d"(e ? b.y : b.x));
              }
            }
            // 8 k a step of s, over SETS chains
            if (SETS == 1 && (s & 1)) end_chains();
          }
          if (SETS == 2 || (SETS == 4 && (h & 1))) end_chains();
          if (++slot == STAGES) slot = 0;
        }
      };
      if (ROWS && !diag) mac_block(Yes{});
      else mac_block(No{});
    }
    // X_k = inv(T_kk) Z_k replaces Z_k once every warp has read it.  The diagonal's
    // term, which may dwarf the others, is added last: one rounding of its size.
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int r = 8 * n + 2 * t + (v & 1), i = wm + 2 * g + (v >> 1);
        const double z = zk[r * P + (v >> 1)];
        double x = fma(d[v >> 1], z, sum[n][v]);
        if (!isfinite(z)) {  // the zero that stands for the diagonal made a NaN of it
          const double *ti = Tinv + (long long)k * TB * TB + i, *zr = Z + r * P + k * TB;
          x = d[v >> 1] * z;
          for (int j = 0; j < TB; ++j)
            if (j != i) x = fma(ti[j * TB], zr[j], x);
        }
        sum[n][v] = x;
      }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int v = 0; v < 4; ++v) zk[(8 * n + 2 * t + (v & 1)) * P + (v >> 1)] = sum[n][v];
    __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  for (int idx = tid; idx < nb * TB * W; idx += 256) {
    const int i = si == 1 ? idx % (nb * TB) : idx / W, r = si == 1 ? idx / (nb * TB) : idx % W;
    if (i < nr && r0 + r < nrhs) B[i * si + (r0 + r) * sr] = Z[r * P + i];
  }
}

__global__ void fill_zero_kernel(int M, int N, double *__restrict__ B, int ldb) {
  const long long total = (long long)M * N;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x)
    B[(idx / M) * ldb + idx % M] = 0.0;
}

struct TrsmPlan {
  bool left, upper, trans, unit;
  int m, n;
  const double *A;
  int lda;
  double *B;
  int ldb;
  int method;
  int leaf;
  cudaStream_t s;
  double *tinv;            // inverted diagonal blocks of T, TB x TB each, zero diagonal
  double *dinv;            // their diagonals
  double *tmp;             // small_solve's product
  int sm_count;
  bool forward;            // T is lower: blocks are solved in ascending order
  long long rs, cs;        // T(i, j) = A[i*rs + j*cs]
};

// Trailing-update GEMM: the INT8 emulation only where its slicing passes are
// amortised (measured: below ~2^33 multiply-adds or K < 1024 plain FP64 wins).
int update_gemm(const TrsmPlan &p, char ta, char tb, int m, int n, int k, const double *A,
                int lda, const double *B, int ldb, double *C, int ldc) {
  int meth = p.method;
  if (meth != B2_METHOD_FP64 && ((double)m * n * k < 8.6e9 || k < 1024)) meth = B2_METHOD_FP64;
  return dgemm_device(ta, tb, m, n, k, -1.0, A, lda, B, ldb, 1.0, C, ldc, meth, 0, p.s);
}

template <int W>
int launch_leaf(const TrsmPlan &p, int k0, int nr) {
  const int nrhs = p.left ? p.n : p.m;
  constexpr int smem = LeafSmem<W>::BYTES;
  static_assert(smem <= 232448, "shared memory of one CTA");
  auto kern = p.rs == 1 ? trsm_leaf_kernel<W, false> : trsm_leaf_kernel<W, true>;
  B2_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  B2_PROF("trsm_leaf", p.s);
  kern<<<(nrhs + W - 1) / W, 256, smem, p.s>>>(
      p.A + (long long)k0 * (p.rs + p.cs), p.rs, p.cs, p.forward ? 1 : 0, nr,
      p.tinv + (long long)(k0 / TB) * TB * TB, p.dinv + k0, p.B + (p.left ? k0 : (long long)k0 * p.ldb),
      p.left ? 1 : p.ldb, p.left ? p.ldb : 1, nrhs);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

// A triangle of order up to SMALL against so many right-hand sides that the leaf kernel
// would take its widest strips: the inverse times all of them as one GEMM, copied back.
// A leaf takes a step of 128 rows whatever the order, one CTA per SM.  B200, us, whole
// solves, leaf / GEMM: order 16 by 1000 12.0 / 11.4, by 4096 18.3 / 13.0, by 100000
// 229 / 39; order 64 by 4096 25.3 / 22.1, by 100000 235 / 86; order 96 by 8192 41.7 /
// 41.7.
constexpr int SMALL = 64;
bool small_many(int nr, int nrhs, int sms) { return nr <= SMALL && nrhs > 16 * sms; }

int small_solve(const TrsmPlan &p, int k0, int nr) {
  const double *Ti = p.tinv + (long long)(k0 / TB) * TB * TB;
  const int rows = p.left ? nr : p.m, cols = p.left ? p.n : nr;
  double *Bk = p.B + (p.left ? k0 : (long long)k0 * p.ldb);
  // (beta = 0 multiplies what the product's place holds)
  B2_CUDA_TRY(cudaMemsetAsync(p.tmp, 0, (size_t)rows * cols * sizeof(double), p.s));
  const int rc = p.left ? dgemm_device('N', 'N', nr, p.n, nr, 1.0, Ti, TB, Bk, p.ldb, 0.0, p.tmp,
                                       nr, B2_METHOD_FP64, 0, p.s)
                        : dgemm_device('N', 'T', p.m, nr, nr, 1.0, Bk, p.ldb, Ti,
                                       TB, 0.0, p.tmp, p.m, B2_METHOD_FP64, 0, p.s);
  if (rc != B2_OK) return rc;
  B2_CUDA_TRY(cudaMemcpy2DAsync(Bk, (size_t)p.ldb * sizeof(double), p.tmp,
                                (size_t)rows * sizeof(double), (size_t)rows * sizeof(double), cols,
                                cudaMemcpyDeviceToDevice, p.s));
  return B2_OK;
}

// Strips of 8, 16 or 32 right-hand sides: the narrowest that one wave of CTAs
// (one per SM) can take; wider ones lengthen every step (leaf times above).
int leaf_solve(const TrsmPlan &p, int k0, int nr) {
  const int nrhs = p.left ? p.n : p.m;
  if (nr <= SMALL && p.tmp) return small_solve(p, k0, nr);
  if (nrhs <= 8 * p.sm_count) return launch_leaf<8>(p, k0, nr);
  if (nrhs <= 16 * p.sm_count) return launch_leaf<16>(p, k0, nr);
  return launch_leaf<32>(p, k0, nr);
}

// Solve the order-nr diagonal part starting at k0 (rows of B for side 'L',
// columns for side 'R').
int solve_range(const TrsmPlan &p, int k0, int nr) {
  if (nr <= p.leaf) return leaf_solve(p, k0, nr);
  int n1 = (nr / 2 + p.leaf - 1) / p.leaf * p.leaf;
  if (n1 >= nr) n1 = nr - p.leaf;
  const int n2 = nr - n1;
  const int k1 = k0 + n1;
  const bool opA_lower = (!p.upper && !p.trans) || (p.upper && p.trans);
  const char tA = p.trans ? 'T' : 'N';
  // op(A)[r, c] block pointer for a GEMM operand: op(A)(i,j) = A[i,j] (N) or A[j,i] (T)
  auto opA_block = [&](int r0, int c0) -> const double * {
    return p.trans ? p.A + c0 + (long long)r0 * p.lda : p.A + r0 + (long long)c0 * p.lda;
  };
  int rc;
  if (p.left) {
    if (opA_lower) {  // forward: solve top, B2 -= op(A)21 X1, solve bottom
      rc = solve_range(p, k0, n1);
      if (rc != B2_OK) return rc;
      rc = update_gemm(p, tA, 'N', n2, p.n, n1, opA_block(k1, k0), p.lda, p.B + k0, p.ldb,
                       p.B + k1, p.ldb);
      if (rc != B2_OK) return rc;
      return solve_range(p, k1, n2);
    }
    // backward: solve bottom, B1 -= op(A)12 X2, solve top
    rc = solve_range(p, k1, n2);
    if (rc != B2_OK) return rc;
    rc = update_gemm(p, tA, 'N', n1, p.n, n2, opA_block(k0, k1), p.lda, p.B + k1, p.ldb,
                     p.B + k0, p.ldb);
    if (rc != B2_OK) return rc;
    return solve_range(p, k0, n1);
  }
  // side 'R': X op(A) = B over column blocks
  if (!opA_lower) {  // op(A) upper: forward over columns
    rc = solve_range(p, k0, n1);
    if (rc != B2_OK) return rc;
    rc = update_gemm(p, 'N', tA, p.m, n2, n1, p.B + (long long)k0 * p.ldb, p.ldb,
                     opA_block(k0, k1), p.lda, p.B + (long long)k1 * p.ldb, p.ldb);
    if (rc != B2_OK) return rc;
    return solve_range(p, k1, n2);
  }
  rc = solve_range(p, k1, n2);  // op(A) lower: backward over columns
  if (rc != B2_OK) return rc;
  rc = update_gemm(p, 'N', tA, p.m, n1, n2, p.B + (long long)k1 * p.ldb, p.ldb,
                   opA_block(k1, k0), p.lda, p.B + (long long)k0 * p.ldb, p.ldb);
  if (rc != B2_OK) return rc;
  return solve_range(p, k0, n1);
}

}  // namespace

int dtrsm_device(char side, char uplo, char transa, char diag, int m, int n, double alpha,
                 const double *A, int lda, double *B, int ldb, int method, int block,
                 cudaStream_t s) {
  if (m <= 0 || n <= 0) return B2_OK;
  Ctx *cx = ctx();
  if (!cx) return B2_ERR_NO_DEVICE;
  if (alpha == 0.0) {  // BLAS: B := 0
    const long long total = (long long)m * n;
    const int blocks = (int)((total + 255) / 256 > 4096 ? 4096 : (total + 255) / 256);
    B2_PROF("trsm_zero", s);
    fill_zero_kernel<<<blocks, 256, 0, s>>>(m, n, B, ldb);
    B2_CUDA_TRY(cudaGetLastError());
    return B2_OK;
  }
  if (alpha != 1.0) {
    const int rc = scale_matrix_d(m, n, alpha, B, ldb, s);
    if (rc != B2_OK) return rc;
  }
  TrsmPlan p;
  p.left = (side == 'L' || side == 'l');
  p.upper = (uplo == 'U' || uplo == 'u');
  p.trans = !(transa == 'N' || transa == 'n');
  p.unit = (diag == 'U' || diag == 'u');
  p.m = m;
  p.n = n;
  p.A = A;
  p.lda = lda;
  p.B = B;
  p.ldb = ldb;
  p.method = method == B2_METHOD_DEFAULT ? B2_METHOD_FP64 : method;
  (void)block;  // leaves are up to LEAF_BLOCKS diagonal blocks of order TB
  p.leaf = LEAF_BLOCKS * TB;
  p.s = s;
  const bool opA_lower = (!p.upper && !p.trans) || (p.upper && p.trans);
  p.forward = p.left == opA_lower;  // T is op(A), or its transpose for side 'R'
  p.rs = (p.left != p.trans) ? 1 : lda;
  p.cs = (p.left != p.trans) ? lda : 1;
  const int na = p.left ? m : n;
  const int nblk = (na + TB - 1) / TB;
  p.tinv = (double *)workspace(cx, WS_TRSM_INV, (size_t)nblk * TB * (TB + 1) * sizeof(double));
  if (!p.tinv) return B2_ERR_NOMEM;
  p.dinv = p.tinv + (size_t)nblk * TB * TB;
  p.sm_count = cx->sm_count;
  // the last leaf may be a small triangle against many right-hand sides
  const int last = (na - 1) % p.leaf + 1, nrhs = p.left ? n : m;
  p.tmp = small_many(last, nrhs, cx->sm_count)
              ? (double *)workspace(cx, WS_TRSM_TMP, (size_t)last * nrhs * sizeof(double))
              : nullptr;  // (no scratch: the leaf kernel)
  {
    const int smem = (TB * TB_LD + 2 * TI_K * TI_PLD + TB) * (int)sizeof(double);
    B2_CUDA_TRY(cudaFuncSetAttribute(trtri_batched_kernel,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    B2_PROF("trsm_trtri", s);
    trtri_batched_kernel<<<nblk, TI_NT, smem, s>>>(A, p.rs, p.cs, na, p.forward ? 1 : 0,
                                                   p.unit ? 1 : 0, p.tmp ? SMALL : 0, p.tinv,
                                                   p.dinv);
    B2_CUDA_TRY(cudaGetLastError());
  }
  return solve_range(p, 0, na);
}

}  // namespace b2
