// dgemm_fp64.cu -- plain FP64 GEMM on the sm_100 FP64 tensor-core path.
//
// Replaces the reference's cache-blocked AVX-512 DGEMM (src/gemm_driver.c:116-195
// driving the 24x8 register tile of src/kernel/gemm_kernel.S:822-1213, and the
// OpenBLAS-like 16x2 / 4x8 / 8x8 kernels).  tcgen05 has no f64 kind, so the
// FP64 tensor path on sm_100 is the warp-level DMMA instruction
// mma.sync.aligned.m16n8k{4,8,16}.row.col.f64 with accumulators in registers.
//
// Design:
//  * CTA tile BM x BN (128x128 / 128x64 / 64x64 / 32x32), warp tile 64x32,
//    32x32 or 16x16;
//    fragments double-buffered in registers (DMMA K 4 and 8).
//  * op(A)/op(B) tiles streamed global->shared with 16-byte cp.async (rows off
//    a 16-byte boundary shifted by one element) through a STAGES-deep ring;
//    the reference's packing (src/gemm_copy.c) disappears: the smem tile keeps
//    the global orientation, padded so every DMMA fragment load is
//    bank-conflict free for both orientations (+4 doubles per row).
//  * alpha/beta are applied once in the epilogue (the reference folds alpha
//    into packed B, src/gemm_copy.c:64, and pre-scales C, :131).
//  * Optional split-K: each z-slice writes an FP64 partial into workspace and
//    a reduction kernel adds them in slice order (deterministic) and applies
//    alpha/beta.  Measured on B200 against an in-kernel fixup (the tile's last
//    slice to arrive adds the partials): the separate reduction is faster on
//    every shape tried, 14 us against 66 us at 128x128x1024 with 8 slices and
//    83 us against 118 us at 1024^3 with 4.
#include <type_traits>

#include "b2_internal.cuh"
#include "b2_profile.cuh"
#include "fp64_copy.cuh"

namespace b2 {
namespace {

using namespace f64copy;

template <int MMAK>
__device__ __forceinline__ void dmma(double (&c)[4], const double *a, const double *b) {
  if constexpr (MMAK == 4) {
    asm volatile(
        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
        "{%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(b[0]));
  } else if constexpr (MMAK == 8) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
  } else {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, "
        "{%4,%5,%6,%7,%8,%9,%10,%11}, {%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]),
          "d"(a[7]), "d"(b[0]), "d"(b[1]), "d"(b[2]), "d"(b[3]));
  }
}

// A_KCONT = transA (op(A)(m,k) = A[m*lda+k]); B_KCONT = !transB (op(B)(k,n) = B[n*ldb+k]).
// Output: when P != nullptr the raw product of this CTA's K range is written to
// P + z*ldp*N (split-K partial); otherwise C = alpha*acc + beta*C (beta==1: C += alpha*acc).
// FOLD > 0: the sums of every `fold` blocks of K are chains of their own, added in
// order.  The chains' sum is held in registers (2, at most four CTAs per SM) or, so that
// five CTAs of the 32x32 tile fit an SM, in local memory (1: 64 bytes a thread, which
// stay in L1).  B200: 1024^3 70.4 us in one chain, 72.5 in four with the sum in local
// memory, 84 with registers bounded to five CTAs; 128x4096x128 in eight chains 9.1 with
// it in registers, 11 in local memory.
template <int BM, int BN, int BK, int WM, int WN, int STAGES, int MMAK, bool A_KCONT,
          bool B_KCONT, bool SH, int FOLD>
__global__ void __launch_bounds__(WM *WN * 32, FOLD == 2                          ? 4
                                               : BM * BN <= 64 * 64 && MMAK == 4 ? 3
                                                                                 : 1)
    dgemm_dmma_kernel(int M, int N, int K, int kchunk, int fold, double alpha,
                      const double *__restrict__ A, int lda, const double *__restrict__ B,
                      int ldb, double beta, double *__restrict__ C, int ldc,
                      double *__restrict__ P, int ldp) {
  constexpr int NT = WM * WN * 32;
  constexpr int TM = BM / WM, TN = BN / WN;  // warp tile
  constexpr int MT = TM / 16, NTL = TN / 8;
  constexpr int A_ST = A_KCONT ? BM * (BK + 4) : BK * (BM + 4);
  constexpr int B_ST = B_KCONT ? BN * (BK + 4) : BK * (BN + 4);
  static_assert(TM % 16 == 0 && TN % 8 == 0 && BK % MMAK == 0, "bad tile");

  extern __shared__ __align__(16) double smem[];
  double *sA = smem;
  double *sB = smem + STAGES * A_ST;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint32_t sA_u = (uint32_t)__cvta_generic_to_shared(sA);
  const uint32_t sB_u = (uint32_t)__cvta_generic_to_shared(sB);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm0 = (warp / WN) * TM, wn0 = (warp % WN) * TN;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int kbeg = blockIdx.z * kchunk;
  const int kend = min(K, kbeg + kchunk);
  const int KT = (kend - kbeg + BK - 1) / BK;

  double acc[MT][NTL][4];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NTL; ++j)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[i][j][v] = 0.0;

  constexpr int A_CH = tile_chunks<BM, BK, NT>(), B_CH = tile_chunks<BN, BK, NT>();
  // row shifts of this thread's chunks and of its fragment reads (A rows are k
  // or m: the fragments' rows are t or g plus even numbers)
  const int sha = SH ? row_shift(A, lda, (A_KCONT ? m0 : kbeg) + tid / ((A_KCONT ? BK : BM) / 2)) : 0;
  const int shb = SH ? row_shift(B, ldb, (B_KCONT ? n0 : kbeg) + tid / ((B_KCONT ? BK : BN) / 2)) : 0;
  const int fsa = SH ? row_shift(A, lda, A_KCONT ? g : t) : 0;
  const int fsb = SH ? row_shift(B, ldb, B_KCONT ? g : t) : 0;
  // An operand's tile that lies wholly inside it is copied from running
  // pointers (a few instructions per copy); an edge tile, a last short K block
  // and, when shifted, whatever touches the start of the operand's first row
  // take the bounds-checked form.
  const bool in_a = m0 + BM <= M, in_b = n0 + BN <= N;
  const bool a_first = SH && (A_KCONT ? m0 : kbeg) == 0, b_first = SH && (B_KCONT ? n0 : kbeg) == 0;
  const bool tail_a = SH && tid < (A_KCONT ? BM : BK) && row_shift(A, lda, (A_KCONT ? m0 : kbeg) + tid);
  const bool tail_b = SH && tid < (B_KCONT ? BN : BK) && row_shift(B, ldb, (B_KCONT ? n0 : kbeg) + tid);
  const double *pa = A + run_offset<BM, BK, A_KCONT>(m0, kbeg, lda, tid) - sha;
  const double *pb = B + run_offset<BN, BK, B_KCONT>(n0, kbeg, ldb, tid) - shb;
  const uint32_t da = sA_u + run_dst<BM, BK, A_KCONT>(tid);
  const uint32_t db = sB_u + run_dst<BN, BK, B_KCONT>(tid);
  const size_t ia = run_step<BM, BK, A_KCONT, NT>(lda);  // chunk to chunk
  const size_t ib = run_step<BN, BK, B_KCONT, NT>(ldb);
  const size_t ka = A_KCONT ? (size_t)BK : (size_t)BK * lda;  // stage to stage
  const size_t kb = B_KCONT ? (size_t)BK : (size_t)BK * ldb;
  // Copies stage kt (called once per kt, in order) into ring slot st.
  auto load_stage = [&](int st, int kt) {
    const int k0 = kbeg + kt * BK;
    const bool full = k0 + BK <= kend;
    if (full && in_a && !(a_first && kt == 0)) {
#pragma unroll
      for (int c = 0; c < A_CH; ++c)
        cp_async_full<16>(da + st * (A_ST * 8) + c * run_dst_step<BM, BK, A_KCONT, NT>(),
                          pa + c * ia);
      // (the element after the tile is in the row, or is not read)
      if (SH && tail_a)
        cp_async<16>(sA_u + st * (A_ST * 8) + run_tail_dst<BM, BK, A_KCONT>(tid),
                     A + run_tail<BM, BK, A_KCONT>(m0, k0, lda, tid),
                     (A_KCONT ? k0 + BK < kend : m0 + BM < M) ? 16 : 8);
    } else if (full && !(a_first && kt == 0)) {
#pragma unroll
      for (int c = 0; c < A_CH; ++c)
        cp_async_edge(da + st * (A_ST * 8) + c * run_dst_step<BM, BK, A_KCONT, NT>(),
                      pa + c * ia, A, edge_bytes<BM, BK, A_KCONT, NT>(m0, M, tid, sha, c));
      if (SH) load_tails<BM, BK, A_KCONT, NT>(sA_u + st * A_ST * 8, A, lda, m0, k0, M, kend, tid);
    } else {
#pragma unroll
      for (int c = 0; c < A_CH; ++c)
        load_chunk<BM, BK, A_KCONT, SH, NT>(sA_u + st * A_ST * 8, A, lda, m0, k0, M, kend, tid, c,
                                            sha);
      if (SH) load_tails<BM, BK, A_KCONT, NT>(sA_u + st * A_ST * 8, A, lda, m0, k0, M, kend, tid);
    }
    if (full && in_b && !(b_first && kt == 0)) {
#pragma unroll
      for (int c = 0; c < B_CH; ++c)
        cp_async_full<16>(db + st * (B_ST * 8) + c * run_dst_step<BN, BK, B_KCONT, NT>(),
                          pb + c * ib);
      if (SH && tail_b)
        cp_async<16>(sB_u + st * (B_ST * 8) + run_tail_dst<BN, BK, B_KCONT>(tid),
                     B + run_tail<BN, BK, B_KCONT>(n0, k0, ldb, tid),
                     (B_KCONT ? k0 + BK < kend : n0 + BN < N) ? 16 : 8);
    } else if (full && !(b_first && kt == 0)) {
#pragma unroll
      for (int c = 0; c < B_CH; ++c)
        cp_async_edge(db + st * (B_ST * 8) + c * run_dst_step<BN, BK, B_KCONT, NT>(),
                      pb + c * ib, B, edge_bytes<BN, BK, B_KCONT, NT>(n0, N, tid, shb, c));
      if (SH) load_tails<BN, BK, B_KCONT, NT>(sB_u + st * B_ST * 8, B, ldb, n0, k0, N, kend, tid);
    } else {
#pragma unroll
      for (int c = 0; c < B_CH; ++c)
        load_chunk<BN, BK, B_KCONT, SH, NT>(sB_u + st * B_ST * 8, B, ldb, n0, k0, N, kend, tid, c,
                                            shb);
      if (SH) load_tails<BN, BK, B_KCONT, NT>(sB_u + st * B_ST * 8, B, ldb, n0, k0, N, kend, tid);
    }
    pa += ka;
    pb += kb;
  };

#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < KT) load_stage(s, s);
    cp_async_commit();
  }

  // Bound: the FP64 pipe (0.533 us per 64x64x16 block and SM at 1.92 GHz).
  // Fragments are double-buffered in registers: the next K step's shared loads
  // (across a stage's edge too, so the barrier sits before the last step's
  // DMMAs) are in flight while the current step's DMMAs issue.  With the
  // running copy pointers and DMMA K 4 (whose fragments leave three CTAs per
  // SM) a block takes 0.553 us where it took 0.597 (K = 4096, 10 tiles per SM;
  // 4096^3 4228 -> 3886 us); one CTA alone on an SM 0.72 instead of 1.0.
  // Edge tiles copy from running pointers too (bounds checked element by element
  // they cost a lone CTA 1.34 us a block, now 0.90: 424x39x1600 21.3 -> 16.0 us).
  // Copies placed one by one between the DMMAs were slower (0.70).
  constexpr int KS = BK / MMAK;
  // (DMMA K 16 has one step per stage and twice the fragments: single-buffered.)
  constexpr bool PIPE = KS % 2 == 0;
  double af[PIPE ? 2 : 1][MT][MMAK / 2], bf[PIPE ? 2 : 1][NTL][MMAK / 4];
  auto load_frags = [&](int buf, int st, int kk) {
    const double *As = sA + st * A_ST + fsa;
    const double *Bs = sB + st * B_ST + fsb;
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int v1 = 0; v1 < MMAK / 4; ++v1)
#pragma unroll
        for (int v0 = 0; v0 < 2; ++v0) {
          const int m = wm0 + i * 16 + g + 8 * v0, k = kk + t + 4 * v1;
          af[buf][i][v0 + 2 * v1] = A_KCONT ? As[m * (BK + 4) + k] : As[k * (BM + 4) + m];
        }
#pragma unroll
    for (int j = 0; j < NTL; ++j)
#pragma unroll
      for (int v = 0; v < MMAK / 4; ++v) {
        const int n = wn0 + j * 8 + g, k = kk + t + 4 * v;
        bf[buf][j][v] = B_KCONT ? Bs[n * (BK + 4) + k] : Bs[k * (BN + 4) + n];
      }
  };
  using Tot = std::conditional_t<FOLD == 1, volatile double, double>;  // (volatile: local)
  Tot tot[FOLD ? MT * NTL * 4 : 1];
  auto end_chain = [&](bool first) {
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NTL; ++j)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          Tot &t = tot[(i * NTL + j) * 4 + v];
          t = first ? acc[i][j][v] : t + acc[i][j][v];
          acc[i][j][v] = 0.0;
        }
  };
  cp_async_wait<STAGES - 2>();
  __syncthreads();
  if (PIPE) load_frags(0, 0, 0);
  int st = 0, st_fill = STAGES - 1;  // stage being multiplied, stage refilled next
  for (int kt = 0; kt < KT;) {
    const int chain_end = FOLD ? min(KT, kt + fold) : KT;
    for (; kt < chain_end; ++kt) {
      const int st_next = st + 1 == STAGES ? 0 : st + 1;
      // every warp has issued its last reads of stage kt - 1, which is refilled here
      const bool fill = kt + STAGES - 1 < KT;
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        const int cur = PIPE ? (ks & 1) : 0;
        if (!PIPE) load_frags(0, st, ks * MMAK);
        if (PIPE && ks + 1 < KS) load_frags(cur ^ 1, st, (ks + 1) * MMAK);
        if (ks == 0 && fill) load_stage(st_fill, kt + STAGES - 1);
        if (ks + 1 == KS) {
          cp_async_commit();
          cp_async_wait<STAGES - 2>();
          __syncthreads();
          if (PIPE && kt + 1 < KT) load_frags(cur ^ 1, st_next, 0);
        }
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int j = 0; j < NTL; ++j) dmma<MMAK>(acc[i][j], af[cur][i], bf[cur][j]);
      }
      st = st_next;
      st_fill = st_fill + 1 == STAGES ? 0 : st_fill + 1;
    }
    if (FOLD && kt < KT) end_chain(kt == fold);
  }
  cp_async_wait<0>();
  if constexpr (FOLD) {  // (a slice of one chain has none before it)
    if (KT > fold) {
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NTL; ++j)
#pragma unroll
          for (int v = 0; v < 4; ++v) acc[i][j][v] = tot[(i * NTL + j) * 4 + v] + acc[i][j][v];
    }
  }

  // Epilogue.  Fragment (i, j, v): row g + 8*(v>>1), column 2t + (v&1).
  if (P != nullptr) {
    double *Pz = P + (size_t)blockIdx.z * ldp * N;
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NTL; ++j)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int m = m0 + wm0 + i * 16 + g + 8 * (v >> 1);
          const int n = n0 + wn0 + j * 8 + 2 * t + (v & 1);
          if (m < M && n < N) Pz[(size_t)n * ldp + m] = acc[i][j][v];
        }
    return;
  }
  // C is read before any of it is written, 16 rows of the warp tile at a
  // time: interleaved with the stores, each load would wait for the one before
  // it (the compiler keeps their order), 32 round trips to memory in a row --
  // 8 us of the 11 us of a 64x64x64 product on B200.
  const bool beta_one = (beta == 1.0);
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    double c_old[NTL][4];
#pragma unroll
    for (int j = 0; j < NTL; ++j)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int m = m0 + wm0 + i * 16 + g + 8 * (v >> 1);
        const int n = n0 + wn0 + j * 8 + 2 * t + (v & 1);
        c_old[j][v] = (m < M && n < N) ? C[(size_t)n * ldc + m] : 0.0;
      }
#pragma unroll
    for (int j = 0; j < NTL; ++j)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int m = m0 + wm0 + i * 16 + g + 8 * (v >> 1);
        const int n = n0 + wn0 + j * 8 + 2 * t + (v & 1);
        if (m < M && n < N)
          C[(size_t)n * ldc + m] = beta_one ? fma(alpha, acc[i][j][v], c_old[j][v])
                                            : fma(alpha, acc[i][j][v], beta * c_old[j][v]);
      }
  }
}

// C = alpha * (sum of the slices' partials, in slice order) + beta * C: one row
// pair per thread along x, columns along y.  Launched as a programmatic
// dependent of the GEMM: its blocks start while the GEMM's last ones finish and
// wait here for its writes.
__global__ void __launch_bounds__(256)
    splitk_reduce_kernel(int M, int N, int splits, const double *__restrict__ P, int ldp,
                         double alpha, double beta, double *__restrict__ C, int ldc) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int pairs = (M + 1) / 2;
  const long long total = (long long)pairs * N;
  const size_t plane = (size_t)ldp * N;
  const bool cvec = (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (ldc & 1) == 0;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int n = (int)(idx / pairs), m = (int)(idx - (long long)n * pairs) * 2;
    const double *p = P + (size_t)n * ldp + m;  // ldp is even: 16-byte aligned
    double *q = C + (size_t)n * ldc + m;
    const bool two = m + 1 < M;
    double2 c;
    if (two && cvec) c = *reinterpret_cast<const double2 *>(q);
    else c = make_double2(q[0], two ? q[1] : 0.0);
    double s0 = 0.0, s1 = 0.0;
    for (int z = 0; z < splits; z += 4) {
      double2 x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (z + u < splits) x[u] = *reinterpret_cast<const double2 *>(p + (size_t)(z + u) * plane);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (z + u < splits) s0 += x[u].x, s1 += x[u].y;
    }
    c.x = (beta == 1.0) ? fma(alpha, s0, c.x) : fma(alpha, s0, beta * c.x);
    c.y = (beta == 1.0) ? fma(alpha, s1, c.y) : fma(alpha, s1, beta * c.y);
    if (two && cvec) *reinterpret_cast<double2 *>(q) = c;
    else {
      q[0] = c.x;
      if (two) q[1] = c.y;
    }
  }
}

template <typename T>
__global__ void scale_kernel(int M, int N, T beta, T *__restrict__ C, int ldc) {
  const size_t total = (size_t)M * N;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int m = (int)(idx % M), n = (int)(idx / M);
    C[(size_t)n * ldc + m] *= beta;
  }
}

struct LaunchArgs {
  int M, N, K, kchunk;
  int fold;  // K blocks of 16 per chain (32x32 tile), 0: one chain
  bool few;  // at most four CTAs per SM
  double alpha;
  const double *A;
  int lda;
  const double *B;
  int ldb;
  double beta;
  double *C;
  int ldc;
  double *P;
  int ldp;
  int splits;
};

template <int BM, int BN, int BK, int WM, int WN, int STAGES, int MMAK, bool AK, bool BKc,
          bool SH, int FOLD>
cudaError_t launch_one(const LaunchArgs &a, cudaStream_t s) {
  constexpr int A_ST = AK ? BM * (BK + 4) : BK * (BM + 4);
  constexpr int B_ST = BKc ? BN * (BK + 4) : BK * (BN + 4);
  constexpr size_t SMEM = (size_t)STAGES * (A_ST + B_ST) * sizeof(double);
  auto kern = dgemm_dmma_kernel<BM, BN, BK, WM, WN, STAGES, MMAK, AK, BKc, SH, FOLD>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)SMEM);
  if (e != cudaSuccess) return e;
  dim3 grid((a.M + BM - 1) / BM, (a.N + BN - 1) / BN, a.splits);
  // A programmatic dependent: it is set up while the kernel before it ends and
  // waits for that one's writes before it touches memory (48x40x64 in a row of
  // calls 8.5 -> 7.9 us, 1024^3 79.9 -> 77.8).
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = grid;
  lc.blockDim = dim3(WM * WN * 32);
  lc.dynamicSmemBytes = SMEM;
  lc.stream = s;
  lc.attrs = attr;
  lc.numAttrs = 1;
  B2_PROF("dgemm_dmma", s);
  e = cudaLaunchKernelEx(&lc, kern, a.M, a.N, a.K, a.kchunk, a.fold, a.alpha, a.A, a.lda, a.B,
                         a.ldb, a.beta, a.C, a.ldc, a.P, a.ldp);
  return e != cudaSuccess ? e : cudaGetLastError();
}

template <int BM, int BN, int WM, int WN, int STAGES, int MMAK, bool SH, int FOLD = 0>
cudaError_t launch_layout(bool ak, bool bk, const LaunchArgs &a, cudaStream_t s) {
  // 64x64, both operands K-contiguous: 80 KB in four stages would leave two
  // CTAs per SM; three stages keep three
  constexpr int ST_TN = BM * BN <= 64 * 64 ? 3 : STAGES;
  if (ak && bk) return launch_one<BM, BN, 16, WM, WN, ST_TN, MMAK, true, true, SH, FOLD>(a, s);
  if (ak && !bk) return launch_one<BM, BN, 16, WM, WN, STAGES, MMAK, true, false, SH, FOLD>(a, s);
  if (!ak && bk) return launch_one<BM, BN, 16, WM, WN, STAGES, MMAK, false, true, SH, FOLD>(a, s);
  return launch_one<BM, BN, 16, WM, WN, STAGES, MMAK, false, false, SH, FOLD>(a, s);
}

template <int MMAK, bool SH>
cudaError_t launch_tile(int tile, bool ak, bool bk, const LaunchArgs &a, cudaStream_t s) {
  switch (tile) {
    case 0: return launch_layout<128, 128, 2, 4, 4, MMAK, SH>(ak, bk, a, s);
    case 1: return launch_layout<128, 64, 2, 2, 4, MMAK, SH>(ak, bk, a, s);
    case 3:  // fp64_call_cfg's, DMMA K 4 only
      if constexpr (MMAK == 4)
        return !a.fold  ? launch_layout<32, 32, 2, 2, 4, 4, SH>(ak, bk, a, s)
               : a.few ? launch_layout<32, 32, 2, 2, 4, 4, SH, 2>(ak, bk, a, s)
                        : launch_layout<32, 32, 2, 2, 4, 4, SH, 1>(ak, bk, a, s);
      else return cudaErrorInvalidValue;
    default: return launch_layout<64, 64, 2, 2, 4, MMAK, SH>(ak, bk, a, s);
  }
}

inline bool is_notrans(char c) { return c == 'N' || c == 'n'; }

}  // namespace

namespace {

// K slices of a product on 64x64 tiles: as many as keep 8 of K each, up to 8, and at
// most 1024 units (32 MB of partials).  They fill the SMs, and they bound the length
// of a chain of additions: 512^3 has a relative error of 3.0e-16 in eight chains added
// up, 7.8e-16 in one.  chain_k is the length that they give, for every form.
int slices64(int m, int n, int k) {
  const long long tiles = (long long)((m + 63) / 64) * ((n + 63) / 64);
  int s = 1;
  if (tiles < 1024)
    while (s < 8 && k / (2 * s) >= 8 && tiles * s * 2 <= 1024) s *= 2;
  return s;
}
int slice_k(int k, int slices) { return ((k + slices - 1) / slices + 15) / 16 * 16; }
int chain_k(int m, int n, int k) {
  const int s = slices64(m, n, k);
  return s > 1 ? slice_k(k, s) : k;
}

// Model of the 64x64 tile's time in us in its K slices.
// q = work units (tiles x slices) per SM, each of `kit` K blocks of 16
// that take the FP64 pipe 0.53 us; a lone CTA per SM reaches 74 % of that rate,
// up to four 91 %, more 95 %; 3 us to fill and drain, 1 us per further wave of
// three; rows off a 16-byte boundary cost 9 % (shared-memory conflicts).  A
// split adds a second launch (1.5 us on the device and 2 on the host, which bounds
// a run of small calls: 128x128x128 8.2 us a call in two launches, 6.0
// in one) and 64 KB of partials per unit, written and read at about 8 TB/s
// (they stay in L2).  Measured (B200, us, graph replays):
//   128x4096x128   S=1 9.2  2 12.4  4 13.0  8 16.2     512^3  26.4 17.1 15.7 17.6
//   512x1024x512   26.6 26.6 27.3 27.3     2048^3  504 541 551 588
double model64(int m, int n, int k, int sms, bool shifted) {
  const int s = slices64(m, n, k);
  const long long units = (long long)((m + 63) / 64) * ((n + 63) / 64) * s;
  const long long q = (units + sms - 1) / sms;
  const int kit = ((k + s - 1) / s + 15) / 16;
  const double rate = q == 1 ? 0.74 : q <= 4 ? 0.91 : 0.95;
  double us = (double)q * kit * 0.53 / rate * (shifted ? 1.09 : 1.0) + 3.0 +
              (double)((q + 2) / 3 - 1);
  if (s > 1) us += 3.5 + (double)units * 65536.0 / 8e6;
  return us;
}

// The same for the 32x32 tile, S = 1, 2, 4, 8 and the best S in *sk: up to five CTAs
// per SM, 0.24 us per K block for
// one CTA alone on an SM, 0.33 for two, 0.148 each from three on (0.139 a
// quarter of a 64x64 tile), 0.8 us per further wave of five, 16 KB of partials
// per unit; 5 % for tiles past an edge, 20 % for shifted rows (40 % for a lone
// CTA, whose copies are on its critical path).
double model32(int m, int n, int k, int sms, bool shifted, int *sk) {
  const long long tm = (m + 31) / 32, tn = (n + 31) / 32;
  double best = 1e300;
  for (int s = 1; s <= 8 && tn <= 65535; s *= 2) {
    if (s > 1 && (k < 8 * s || ((tm + 1) / 2) * ((tn + 1) / 2) * s > 1024)) break;  // as slices64
    const long long units = tm * tn * s, qc = (units + sms - 1) / sms;
    const double q = qc <= 6 ? (double)qc : (double)units / sms;
    const int kit = ((k + s - 1) / s + 15) / 16;
    const double block = qc == 1 ? 0.24 : qc == 2 ? 0.33 : 0.148 * q;
    double us = kit * block * (!shifted ? 1.0 : qc == 1 ? 1.4 : 1.2) *
                    (m % 32 || n % 32 ? 1.05 : 1.0) + 2.2 +
                0.8 * (double)((qc + 4) / 5 - 1);
    if (s > 1) us += 3.5 + (double)units * 16384.0 / 8e6;
    if (us < best) best = us, *sk = s;
  }
  return best;
}

}  // namespace

// The 64x64 tile (three CTAs per SM) is the best of the three tiles of the
// tuner's list from 1024^3 to 8192^3 and in the exhaustive sweep over M, N, K in
// [16, 1024].
Fp64Cfg fp64_default_cfg(int m, int n, int k, int sm_count) {
  (void)sm_count;
  Fp64Cfg c;
  c.tile = 2;
  c.mmak = 4;
  c.split_k = slices64(m, n, k);
  return c;
}

// A call's own choice (no configuration asked for): the 32x32 tile where the
// models find it faster.  Four times the tiles fill the SMs where 64x64 ones
// leave them one chain of K blocks or an uneven last wave, in fewer slices, whose
// chains it adds up itself (64x64 has no registers for that); from about 2048^3 on
// its extra shared reads lose.  B200, us, 64x64 / 32x32 in the better S of each:
//   48x40x64 3.7 / 3.0     128x4096x128 15.9 / 9.1    424x39x1600 15.0 / 8.8
//   512^3 17.1 / 13.3      900^3 65.9 / 59.1          1024^3 75.9 / 72.5
//   1536x1024x2048 231 / 212    2048^3 504 / 525      4096^3 3896 / 4083
static Fp64Cfg fp64_call_cfg(int m, int n, int k, int sm_count, bool shifted) {
  const int sms = sm_count > 0 ? sm_count : 148;
  Fp64Cfg c;
  c.mmak = 4;
  int s32 = 1;
  const bool small = model32(m, n, k, sms, shifted, &s32) < model64(m, n, k, sms, shifted);
  c.tile = small ? 3 : 2;
  c.split_k = small ? s32 : slices64(m, n, k);
  c.chain = small ? chain_k(m, n, k) : 0;
  return c;
}

Fp64Cfg &fp64_override_cfg() {
  static thread_local Fp64Cfg cfg;
  return cfg;
}

int scale_matrix_d(int m, int n, double beta, double *C, int ldc, cudaStream_t s) {
  if (m <= 0 || n <= 0) return B2_OK;
  const size_t total = (size_t)m * n;
  const int blocks = (int)((total + 255) / 256 > 8192 ? 8192 : (total + 255) / 256);
  B2_PROF("scale_matrix", s);
  scale_kernel<double><<<blocks, 256, 0, s>>>(m, n, beta, C, ldc);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

int scale_matrix_s(int m, int n, float beta, float *C, int ldc, cudaStream_t s) {
  if (m <= 0 || n <= 0) return B2_OK;
  const size_t total = (size_t)m * n;
  const int blocks = (int)((total + 255) / 256 > 8192 ? 8192 : (total + 255) / 256);
  B2_PROF("scale_matrix", s);
  scale_kernel<float><<<blocks, 256, 0, s>>>(m, n, beta, C, ldc);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

int dgemm_fp64(char ta, char tb, int m, int n, int k, double alpha, const double *A, int lda,
               const double *B, int ldb, double beta, double *C, int ldc, cudaStream_t s,
               const Fp64Cfg *cfg_in) {
  if (m <= 0 || n <= 0) return B2_OK;
  Ctx *cx = ctx();
  if (!cx) return B2_ERR_NO_DEVICE;
  if (k <= 0 || alpha == 0.0) return beta == 1.0 ? B2_OK : scale_matrix_d(m, n, beta, C, ldc, s);
  const bool ak = !is_notrans(ta);  // transposed A: k contiguous
  const bool bk = is_notrans(tb);   // plain B: k contiguous
  const bool vec2 = (lda % 2 == 0) && (ldb % 2 == 0) && (((uintptr_t)A & 15) == 0) &&
                    (((uintptr_t)B & 15) == 0);
  Fp64Cfg cfg = cfg_in            ? *cfg_in
                : cx->fp64_override ? fp64_override_cfg()
                                    : fp64_call_cfg(m, n, k, cx->sm_count, !vec2);
  LaunchArgs a{m, n, k, k, 0, false, alpha, A, lda, B, ldb, beta, C, ldc, nullptr, 0, 1};
  int splits = cfg.split_k < 1 ? 1 : cfg.split_k;
  if (splits > 1) {
    const int chunk = slice_k(k, splits);
    splits = (k + chunk - 1) / chunk;
    a.kchunk = chunk;
    a.splits = splits;
    if (splits > 1) {
      const int ldp = (m + 1) & ~1;  // even: 16-byte row pairs in the reduction
      const size_t bytes = (size_t)splits * ldp * n * sizeof(double);
      double *P = (double *)workspace(cx, WS_MISC, bytes);
      if (!P) return B2_ERR_NOMEM;
      a.P = P;
      a.ldp = ldp;
    } else {
      a.kchunk = k;
    }
  }
  if (cfg.chain > 0 && cfg.chain < a.kchunk) {
    a.fold = cfg.chain / 16;
    a.few = (long long)((m + 31) / 32) * ((n + 31) / 32) * a.splits <= 4ll * cx->sm_count;
  }
  cudaError_t e;
  const int mk = cfg.mmak;
  if (vec2) {
    e = mk == 16 ? launch_tile<16, false>(cfg.tile, ak, bk, a, s)
        : mk == 8 ? launch_tile<8, false>(cfg.tile, ak, bk, a, s)
                  : launch_tile<4, false>(cfg.tile, ak, bk, a, s);
  } else {
    e = mk == 16 ? launch_tile<16, true>(cfg.tile, ak, bk, a, s)
        : mk == 8 ? launch_tile<8, true>(cfg.tile, ak, bk, a, s)
                  : launch_tile<4, true>(cfg.tile, ak, bk, a, s);
  }
  if (e != cudaSuccess) return cuda_fail(e, "dgemm_dmma_kernel");
  if (a.P) {
    const long long total = (long long)((m + 1) / 2) * n;
    const long long want = (total + 255) / 256;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)(want > 8192 ? 8192 : want));
    lc.blockDim = dim3(256);
    lc.stream = s;
    lc.attrs = attr;
    lc.numAttrs = 1;
    B2_PROF("dgemm_splitk_reduce", s);
    B2_CUDA_TRY(cudaLaunchKernelEx(&lc, splitk_reduce_kernel, m, n, a.splits, (const double *)a.P,
                                   a.ldp, alpha, beta, C, ldc));
    B2_CUDA_TRY(cudaGetLastError());
  }
  return B2_OK;
}

}  // namespace b2

extern "C" int b2_set_fp64_config(int tile, int mmak, int split_k) {
  b2::Ctx *c = b2::ctx();
  if (!c) return B2_ERR_NO_DEVICE;
  if (tile < 0) {
    c->fp64_override = 0;
    return B2_OK;
  }
  if (tile > 2 || !(mmak == 4 || mmak == 8 || mmak == 16) || split_k < 1 || split_k > 64)
    return B2_ERR_ARG;
  b2::Fp64Cfg &o = b2::fp64_override_cfg();
  o.tile = tile;
  o.mmak = mmak;
  o.split_k = split_k;
  c->fp64_override = 1;
  return B2_OK;
}
