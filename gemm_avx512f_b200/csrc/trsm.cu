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
constexpr int TB_LD = TB + 1;  // shared row stride
constexpr int TI_NT = 256;     // threads of the inversion

// Invert every diagonal block T_b = T[kb:kb+bs, kb:kb+bs] (lower or upper, unit
// or not); block b goes to Tinv + b*TB*TB (column-major, ld TB, zero outside the
// triangle and beyond bs).  An upper block is inverted as the lower one it is
// with both indices reversed.  In shared memory, in place: the eight 16x16
// diagonal blocks by substitution against the identity (one thread per column),
// then three doublings, M21 <- -inv(M22) M21 inv(M11) for every pair of
// s x s blocks, s = 16, 32, 64, as two register-tiled products.
// Bound: FP64 latency of one CTA per block; one thread per column of the whole
// block (8192 dependent FMAs) took 232 us at order 4096, this 28 us (B200).
__device__ __forceinline__ double &tel(double *T, int i, int j) { return T[j * TB_LD + i]; }

template <int S>
__device__ __forceinline__ void trtri_double(double *T, double *tmp, int tid) {
  // pairs p: M11 at 2Sp, M22 at 2Sp + S; outputs per pair S x S, all pairs: 64 S.
  // Each thread: CELLS consecutive columns of one row.
  constexpr int PAIRS = TB / (2 * S), CELLS = PAIRS * S * S / TI_NT;
  const int row = tid % S, cg = (tid / S) % (S / CELLS), pair = tid / (S * (S / CELLS));
  const int o1 = 2 * S * pair, o2 = o1 + S, c0 = cg * CELLS;
  double acc[CELLS];
  // tmp = M21 inv(M11): columns c of inv(M11) are zero above c
#pragma unroll
  for (int c = 0; c < CELLS; ++c) acc[c] = 0.0;
#pragma unroll 4
  for (int k = c0; k < S; ++k) {
    const double a = tel(T, o2 + row, o1 + k);
#pragma unroll
    for (int c = 0; c < CELLS; ++c)  // inv(M11)(k, c0 + c): the upper part holds zeros
      acc[c] = fma(a, tel(T, o1 + k, o1 + c0 + c), acc[c]);
  }
#pragma unroll
  for (int c = 0; c < CELLS; ++c) tmp[(c0 + c) * (TB / 2 + 1) + pair * S + row] = acc[c];
  __syncthreads();
  // M21 = -inv(M22) tmp
#pragma unroll
  for (int c = 0; c < CELLS; ++c) acc[c] = 0.0;
#pragma unroll 4
  for (int k = 0; k < S; ++k) {  // (zero beyond the row)
    const double a = tel(T, o2 + row, o2 + k);
#pragma unroll
    for (int c = 0; c < CELLS; ++c)
      acc[c] = fma(a, tmp[(c0 + c) * (TB / 2 + 1) + pair * S + k], acc[c]);
  }
#pragma unroll
  for (int c = 0; c < CELLS; ++c) tel(T, o2 + row, o1 + c0 + c) = -acc[c];
  __syncthreads();
}

__global__ void __launch_bounds__(TI_NT)
    trtri_batched_kernel(const double *__restrict__ A, long long rs, long long cs, int n, int lower,
                         int unit, double *__restrict__ Tinv) {
  extern __shared__ double tsm[];
  double *T = tsm;                  // T(i, j) at [j*TB_LD + i]
  double *tmp = tsm + TB * TB_LD;   // up to 64 columns x 64 rows
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
  double *inv = tmp;  // inverted diagonal
  if (tid < TB) inv[tid] = 1.0 / tel(T, tid, tid);
  __syncthreads();
  // 16x16 diagonal blocks: thread 16 b + j forms column j of block b's inverse
  if (tid < TB) {
    const int o = tid & ~15, j = tid & 15;
    double x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      double acc = i == j ? 1.0 : 0.0;
#pragma unroll
      for (int k = 0; k < i; ++k) acc = fma(-tel(T, o + i, o + k), x[k], acc);
      x[i] = i < j ? 0.0 : acc * inv[o + i];
    }
    __syncwarp();  // a half-warp owns a block: all of it is read before it is written
#pragma unroll
    for (int i = 0; i < 16; ++i) tel(T, o + i, o + j) = x[i];
  }
  __syncthreads();
  trtri_double<16>(T, tmp, tid);
  trtri_double<32>(T, tmp, tid);
  trtri_double<64>(T, tmp, tid);
  double *out = Tinv + (long long)blockIdx.x * TB * TB;
  for (int idx = tid; idx < TB * TB; idx += TI_NT) {
    const int i = idx % TB, j = idx / TB;  // element (i, j) of the stored inverse
    double v = 0.0;
    if (i < bs && j < bs) {
      const int li = lower ? i : bs - 1 - i, lj = lower ? j : bs - 1 - j;
      if (li >= lj) v = tel(T, li, lj);
    }
    out[idx] = v;
  }
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
// than 8, the FP64 pipe; reached: 24, 37 and 70 us for 512 rows at 8, 16 and 32
// (B200).  Each 128-row block as its own memset, GEMM, reduction and copy, with
// the updates between them as further launches, took 68 us for 512 rows and 1024
// right-hand sides, 24 now; dtrsm 4096 x 1024 1747 -> 796 us in all.
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
                     const double *__restrict__ Tinv, double *__restrict__ B, long long si,
                     long long sr, int nrhs) {
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
  using Yes = std::integral_constant<bool, true>;
  using No = std::integral_constant<bool, false>;
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
  // independent chains (K steps dealt out in turn), added at a step's end.
  constexpr int SETS = NT >= 4 ? 1 : 4 / NT;
  double acc[SETS][NT][4];
  // Element (n, v) of a warp's fragment: row wm + 2g + (v >> 1), rhs 8n + 2t + (v & 1)
  __syncthreads();
  int slot = 0;
  for (int kq = 0; kq < nb; ++kq) {
    const int k = forward ? kq : nb - 1 - kq;
#pragma unroll
    for (int c = 0; c < SETS; ++c)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[c][n][v] = 0.0;
    double *zk = Z + k * TB + wm + 2 * g;
    for (int jq = 0; jq <= kq; ++jq) {
      const bool diag = jq == kq;
      if (diag && kq > 0) {  // all updates of block k are in: Z_k -= their sum
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            double x = acc[0][n][v];
#pragma unroll
            for (int c = 1; c < SETS; ++c) x += acc[c][n][v];
            zk[(8 * n + 2 * t + (v & 1)) * P + (v >> 1)] -= x;
#pragma unroll
            for (int c = 0; c < SETS; ++c) acc[c][n][v] = 0.0;
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
          }
          if (++slot == STAGES) slot = 0;
        }
      };
      if (ROWS && !diag) mac_block(Yes{});
      else mac_block(No{});
    }
    // X_k = inv(T_kk) Z_k replaces Z_k once every warp has read it
    __syncthreads();
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        double x = acc[0][n][v];
#pragma unroll
        for (int c = 1; c < SETS; ++c) x += acc[c][n][v];
        zk[(8 * n + 2 * t + (v & 1)) * P + (v >> 1)] = x;
      }
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
  double *tinv;            // inverted diagonal blocks of T, TB x TB each
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
      p.tinv + (long long)(k0 / TB) * TB * TB, p.B + (p.left ? k0 : (long long)k0 * p.ldb),
      p.left ? 1 : p.ldb, p.left ? p.ldb : 1, nrhs);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

// Strips of 8, 16 or 32 right-hand sides: the narrowest that one wave of CTAs
// (one per SM) can take; wider ones lengthen every step (leaf times above).
int leaf_solve(const TrsmPlan &p, int k0, int nr) {
  const int nrhs = p.left ? p.n : p.m;
  if (nrhs <= 8 * 148) return launch_leaf<8>(p, k0, nr);
  if (nrhs <= 16 * 148) return launch_leaf<16>(p, k0, nr);
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
  p.tinv = (double *)workspace(cx, WS_TRSM_INV, (size_t)nblk * TB * TB * sizeof(double));
  if (!p.tinv) return B2_ERR_NOMEM;
  {
    const int smem = (TB * TB_LD + (TB / 2) * (TB / 2 + 1)) * (int)sizeof(double);
    B2_CUDA_TRY(cudaFuncSetAttribute(trtri_batched_kernel,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    B2_PROF("trsm_trtri", s);
    trtri_batched_kernel<<<nblk, TI_NT, smem, s>>>(A, p.rs, p.cs, na, p.forward ? 1 : 0,
                                                   p.unit ? 1 : 0, p.tinv);
    B2_CUDA_TRY(cudaGetLastError());
  }
  return solve_range(p, 0, na);
}

}  // namespace b2
