// gemm3m.cu -- complex GEMM by the 3M method.
//
// zgemm3m runs in ONE fused launch (zgemm3m_dmma_kernel, FP64 DMMA) below 2^35
// multiply-adds and as three FP64 DMMA GEMMs between a pre-add pass and a
// combine pass above; cgemm3m runs in one fused FFMA launch below 2^24
// multiply-adds and otherwise as a batch of three 3xTF32 tensor-core products
// (cgemm3m_tensor, sgemm_tc.cu).
//
// Replaces the OpenBLAS gemm3m driver + the reference's 3M kernels
// (zgemm3m_kernel_2x8_skylakex.c:336-351, zgemm3m_kernel_8x4_skylakex.c:309-334,
// cgemm3m_kernel_16x4_skylakex.c:415-440).  The reference kernels compute
// C_cplx += (alpha_r + i alpha_i) (A_real_packed . B_real_packed) and are called
// three times by the driver on pre-added panels.  Here every CTA owns one tile
// of C and forms all three real products from the same staged tiles:
//     P1 = Ar Br,  P2 = Ai Bi,  P3 = (Ar + Ai)(Br + Bi)
//     Re(AB) = P1 - P2,  Im(AB) = P3 - P1 - P2
// The pre-additions (and conjugation for 'C'/'R') are made on operand fragments
// in registers (zgemm3m_kernel, for operands off a 16-byte boundary: while its
// tiles are de-interleaved into shared memory); the post-additions and the
// complex alpha/beta happen in the epilogue.  beta follows the reference
// drivers (C scaled whenever beta != 1, src/gemm_driver.c:131).
//   zgemm3m: FP64 DMMA (mma.sync.m16n8k4.f64), 32x32 tile, 4 warps of 16x16.
//   cgemm3m: FP32 FFMA, 32x32 tile, four groups of 64 threads of 4x4 outputs
//   splitting each panel's k.
#include <stdlib.h>

#include "b2_methods.cuh"
#include "b2_profile.cuh"
#include "umma.cuh"

namespace b2 {
namespace {

constexpr int G_BM = 64, G_BN = 64, G_BK = 16, G_PAD = 4;
constexpr int G_LD = G_BM + G_PAD;  // [k][m] / [k][n] row stride (68 = 4 mod 16 doubles)

__host__ __device__ __forceinline__ bool tr_is_t(char c) {
  return !(c == 'N' || c == 'n' || c == 'R' || c == 'r');
}
__host__ __device__ __forceinline__ bool tr_is_conj(char c) {
  return c == 'C' || c == 'c' || c == 'R' || c == 'r';
}

// Stage one BK-deep complex K panel of op(A) (G_BM rows) and op(B) (G_BN
// columns) into registers.  Element (m,k) of op(A) is A[m*lda+k] when
// transposed, else A[k*lda+m] (complex units); element (k,n) of op(B) is
// B[k*ldb+n] when transposed, else B[n*ldb+k].
template <typename T, int NT>
struct Stage3M {
  static constexpr int PER = G_BM * G_BK / NT;  // complex elements per thread per operand
  T ar[PER], ai[PER], br[PER], bi[PER];
  __device__ __forceinline__ void load(const T *A, int lda, const T *B, int ldb, int M, int N,
                                       int K, int m0, int n0, int k0, bool tA, bool tB,
                                       T sa, T sb, int tid) {
#pragma unroll
    for (int e = 0; e < PER; ++e) {
      const int idx = tid + NT * e;
      int mm, kk;
      if (tA) { kk = idx % G_BK; mm = idx / G_BK; } else { mm = idx % G_BM; kk = idx / G_BM; }
      const int gm = m0 + mm, gk = k0 + kk;
      T re = 0, im = 0;
      if (gm < M && gk < K) {
        const T *p = A + 2 * (tA ? ((long long)gm * lda + gk) : ((long long)gk * lda + gm));
        re = p[0];
        im = sa * p[1];
      }
      ar[e] = re;
      ai[e] = im;
      int nn;
      if (tB) { nn = idx % G_BN; kk = idx / G_BN; } else { kk = idx % G_BK; nn = idx / G_BK; }
      const int gn = n0 + nn, gk2 = k0 + kk;
      re = 0;
      im = 0;
      if (gn < N && gk2 < K) {
        const T *p = B + 2 * (tB ? ((long long)gk2 * ldb + gn) : ((long long)gn * ldb + gk2));
        re = p[0];
        im = sb * p[1];
      }
      br[e] = re;
      bi[e] = im;
    }
  }
  // shared layout: [3][BK][G_LD] for A (r, i, r+i) and the same for B
  __device__ __forceinline__ void store(T *sA, T *sB, bool tA, bool tB, int tid) const {
#pragma unroll
    for (int e = 0; e < PER; ++e) {
      const int idx = tid + NT * e;
      int mm, kk;
      if (tA) { kk = idx % G_BK; mm = idx / G_BK; } else { mm = idx % G_BM; kk = idx / G_BM; }
      sA[(0 * G_BK + kk) * G_LD + mm] = ar[e];
      sA[(1 * G_BK + kk) * G_LD + mm] = ai[e];
      sA[(2 * G_BK + kk) * G_LD + mm] = ar[e] + ai[e];
      int nn;
      if (tB) { nn = idx % G_BN; kk = idx / G_BN; } else { kk = idx % G_BK; nn = idx / G_BK; }
      sB[(0 * G_BK + kk) * G_LD + nn] = br[e];
      sB[(1 * G_BK + kk) * G_LD + nn] = bi[e];
      sB[(2 * G_BK + kk) * G_LD + nn] = br[e] + bi[e];
    }
  }
};

template <typename T>
__device__ __forceinline__ void epilogue3m(T *C, int ldc, int m, int n, T p1, T p2, T p3,
                                           T ar, T ai, T br, T bi) {
  const T re = p1 - p2, im = p3 - p1 - p2;
  T *c = C + 2 * ((long long)n * ldc + m);
  T cr = c[0], ci = c[1];
  if (!(br == (T)1 && bi == (T)0)) {
    const T tr = br * cr - bi * ci, ti = br * ci + bi * cr;
    cr = tr;
    ci = ti;
  }
  c[0] = cr + (ar * re - ai * im);
  c[1] = ci + (ar * im + ai * re);
}

// ---------------------------------------------------- zgemm3m: FP64 DMMA --
__global__ void __launch_bounds__(256)
    zgemm3m_kernel(int M, int N, int K, const double *__restrict__ A, int lda,
                   const double *__restrict__ B, int ldb, double *__restrict__ C, int ldc,
                   double ar, double ai, double br, double bi, char transa, char transb) {
  extern __shared__ __align__(16) double zsm[];  // [2][3*BK*LD] A, then [2][3*BK*LD] B
  double *sA[2] = {zsm, zsm + 3 * G_BK * G_LD};
  double *sB[2] = {zsm + 6 * G_BK * G_LD, zsm + 9 * G_BK * G_LD};
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm0 = (warp >> 2) * 32, wn0 = (warp & 3) * 16;
  const int m0 = blockIdx.x * G_BM, n0 = blockIdx.y * G_BN;
  const bool tA = tr_is_t(transa), tB = tr_is_t(transb);
  const double sa = tr_is_conj(transa) ? -1.0 : 1.0, sb = tr_is_conj(transb) ? -1.0 : 1.0;
  double acc[3][2][2][4];
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[p][i][j][v] = 0.0;

  Stage3M<double, 256> st;
  const int KT = (K + G_BK - 1) / G_BK;
  st.load(A, lda, B, ldb, M, N, K, m0, n0, 0, tA, tB, sa, sb, tid);
  st.store(sA[0], sB[0], tA, tB, tid);
  __syncthreads();
  for (int kt = 0; kt < KT; ++kt) {
    const int buf = kt & 1;
    if (kt + 1 < KT) st.load(A, lda, B, ldb, M, N, K, m0, n0, (kt + 1) * G_BK, tA, tB, sa, sb, tid);
    const double *As = sA[buf], *Bs = sB[buf];
#pragma unroll
    for (int kk = 0; kk < G_BK; kk += 4) {
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        double af[2][2], bf[2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int v = 0; v < 2; ++v)
            af[i][v] = As[(p * G_BK + kk + t) * G_LD + wm0 + i * 16 + g + 8 * v];
#pragma unroll
        for (int j = 0; j < 2; ++j) bf[j] = Bs[(p * G_BK + kk + t) * G_LD + wn0 + j * 8 + g];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j)
            asm volatile(
                "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, "
                "{%6}, {%0,%1,%2,%3};\n"
                : "+d"(acc[p][i][j][0]), "+d"(acc[p][i][j][1]), "+d"(acc[p][i][j][2]),
                  "+d"(acc[p][i][j][3])
                : "d"(af[i][0]), "d"(af[i][1]), "d"(bf[j]));
      }
    }
    if (kt + 1 < KT) {
      st.store(sA[buf ^ 1], sB[buf ^ 1], tA, tB, tid);
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int m = m0 + wm0 + i * 16 + g + 8 * (v >> 1);
        const int n = n0 + wn0 + j * 8 + 2 * t + (v & 1);
        if (m < M && n < N)
          epilogue3m<double>(C, ldc, m, n, acc[0][i][j][v], acc[1][i][j][v], acc[2][i][j][v],
                             ar, ai, br, bi);
      }
}

// ---------------------------------------------------- cgemm3m: FP32 FFMA --
// Products below 2^24 multiply-adds: a few CTAs, so what bounds them is the
// chain of K panels of one CTA.  CTA tile 32 x 32 complex outputs, 256 threads:
// four groups of 64 take every fourth k of a panel of 16, each thread 4 x 4
// outputs (rows 2 tx + {0, 1} and 16 further, columns likewise with ty) of the
// three products; the groups' sums meet in shared memory at the end, each group
// storing one of a thread's four rows.  The complex panels go through a
// four-stage cp.async ring as they are, the pre-adds are made in registers.
// With 64 x 64 tiles, panels of three real planes staged through registers and
// no split, B200 us: 64^3 17.9, 200x100x300 70.1, 255^3 60.4, 2000x1000x8 28.0;
// this way 4.8, 15.6, 13.6 and 19.7.  (From 2^24 multiply-adds on the
// tensor-core products, 3xTF32, take over: their rounding differs, so the line
// stays where it was.)
constexpr int C_T = 32, C_K = 16, C_LD = 34;  // tile edge, k per panel, [k][.] pitch
constexpr int C_STAGES = 4;
constexpr int C_PANEL = C_K * C_LD;  // complex elements of one operand's panel
constexpr int C_SMEM = 4 * 48 * 64 * 4;  // the groups' sums
static_assert(C_STAGES * 2 * C_PANEL * 8 <= C_SMEM, "the ring fits where the sums go");

// Panel of 32 outer indices x 16 k at [k][C_LD], two elements per thread, as 8
// bytes or (operand off an 8-byte boundary) 4 + 4.  KC: K is contiguous in
// memory; a half-warp then stores 8 k x 2 outer indices, 32 different banks.
template <bool KC>
__device__ __forceinline__ void c3m_copy(uint32_t dst, const float2 *__restrict__ g, int ld, int o0,
                                         int k0, int olim, int K, bool al8, int tid) {
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int o = KC ? tid >> 3 : tid & 31, k = (KC ? tid & 7 : tid >> 5) + 8 * e;
    const bool in = o0 + o < olim && k0 + k < K;
    const float2 *p = in ? g + (KC ? (long long)(o0 + o) * ld + (k0 + k)
                                   : (long long)(k0 + k) * ld + (o0 + o))
                         : g;
    const uint32_t d = dst + (uint32_t)(k * C_LD + o) * 8u;
    if (al8) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(p),
                   "r"(in ? 8 : 0));
    } else {
      const float *q = reinterpret_cast<const float *>(p);
#pragma unroll
      for (int h = 0; h < 2; ++h)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d + 4 * h),
                     "l"(q + h), "r"(in ? 4 : 0));
    }
  }
}

template <bool AK, bool BK>
__global__ void __launch_bounds__(256)
    cgemm3m_kernel(int M, int N, int K, const float2 *__restrict__ A, int lda,
                   const float2 *__restrict__ B, int ldb, float *__restrict__ C, int ldc, float ar,
                   float ai, float br, float bi, float sa, float sb, int tiles_m, bool al8a,
                   bool al8b) {
  extern __shared__ __align__(16) float2 csm[];
  const int tid = threadIdx.x, lane = tid & 31, grp = tid >> 6, t64 = tid & 63;
  const int tx = lane & 7, ty = t64 >> 3;
  const int m0 = (int)(blockIdx.x % tiles_m) * C_T, n0 = (int)(blockIdx.x / tiles_m) * C_T;
  const uint32_t smu = (uint32_t)__cvta_generic_to_shared(csm);
  float acc[3][4][4];
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[p][i][j] = 0.f;
  const int KT = (K + C_K - 1) / C_K;
  auto load_stage = [&](int st, int kt) {
    const uint32_t d = smu + (uint32_t)(st * 2 * C_PANEL) * 8u;
    c3m_copy<AK>(d, A, lda, m0, kt * C_K, M, K, al8a, tid);
    c3m_copy<BK>(d + C_PANEL * 8u, B, ldb, n0, kt * C_K, N, K, al8b, tid);
  };
#pragma unroll
  for (int i = 0; i < C_STAGES - 1; ++i) {
    if (i < KT) load_stage(i, i);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  int st = 0, fill = C_STAGES - 1;
  for (int kt = 0; kt < KT; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(C_STAGES - 2));
    __syncthreads();  // panel kt is in; every thread is done with the one refilled here
    if (kt + C_STAGES - 1 < KT) load_stage(fill, kt + C_STAGES - 1);
    asm volatile("cp.async.commit_group;\n" ::);
    const float2 *As = csm + st * 2 * C_PANEL + 2 * tx, *Bs = csm + st * 2 * C_PANEL + C_PANEL + 2 * ty;
    st = st + 1 == C_STAGES ? 0 : st + 1;
    fill = fill + 1 == C_STAGES ? 0 : fill + 1;
#pragma unroll
    for (int kq = 0; kq < C_K / 4; ++kq) {
      const int kk = (kq * 4 + grp) * C_LD;
      float a[3][4], b[3][4];  // re, im, re + im (conjugated: im negated)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 u = *reinterpret_cast<const float4 *>(As + kk + 16 * h);
        const float4 v = *reinterpret_cast<const float4 *>(Bs + kk + 16 * h);
        a[0][2 * h] = u.x, a[1][2 * h] = sa * u.y, a[0][2 * h + 1] = u.z, a[1][2 * h + 1] = sa * u.w;
        b[0][2 * h] = v.x, b[1][2 * h] = sb * v.y, b[0][2 * h + 1] = v.z, b[1][2 * h + 1] = sb * v.w;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[2][i] = a[0][i] + a[1][i];
        b[2][i] = b[0][i] + b[1][i];
      }
#pragma unroll
      for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[p][i][j] = fmaf(a[p][i], b[p][j], acc[p][i][j]);
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  // group g finishes row g of each thread's four; C's reads before its writes
  const int m = m0 + 2 * tx + (grp & 1) + 16 * (grp >> 1);
  float *c[4];
  float old[4][2];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int n = n0 + 2 * ty + (j & 1) + 16 * (j >> 1);
    const bool in = m < M && n < N;
    c[j] = in ? C + 2 * ((long long)n * ldc + m) : nullptr;
    old[j][0] = in ? c[j][0] : 0.f;
    old[j][1] = in ? c[j][1] : 0.f;
  }
  float *red = reinterpret_cast<float *>(csm);  // [p][i][j][group][64]
  __syncthreads();  // every thread is done with the last panel
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) red[((p * 4 + i) * 4 + j) * 256 + tid] = acc[p][i][j];
  __syncthreads();
  const bool one = br == 1.f && bi == 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float s[3];
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const float *r = red + ((p * 4 + grp) * 4 + j) * 256 + t64;
      s[p] = (r[0] + r[64]) + (r[128] + r[192]);
    }
    if (c[j] == nullptr) continue;
    const float re = s[0] - s[1], im = s[2] - s[0] - s[1];
    float cr = old[j][0], ci = old[j][1];
    if (!one) {
      const float tr = br * cr - bi * ci, ti = br * ci + bi * cr;
      cr = tr;
      ci = ti;
    }
    c[j][0] = cr + (ar * re - ai * im);
    c[j][1] = ci + (ar * im + ai * re);
  }
}

template <bool AK, bool BK>
int launch_cgemm3m(int m, int n, int k, const float *A, int lda, const float *B, int ldb, float *C,
                   int ldc, float ar, float ai, float br, float bi, float sa, float sb,
                   cudaStream_t s) {
  const int tm = (m + C_T - 1) / C_T, tn = (n + C_T - 1) / C_T;
  B2_PROF("cgemm3m_fused", s);
  cgemm3m_kernel<AK, BK><<<(unsigned)tm * (unsigned)tn, 256, C_SMEM, s>>>(
      m, n, k, reinterpret_cast<const float2 *>(A), lda, reinterpret_cast<const float2 *>(B), ldb,
      C, ldc, ar, ai, br, bi, sa, sb, tm, ((uintptr_t)A & 7) == 0, ((uintptr_t)B & 7) == 0);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

// --------------------------------------- zgemm3m: one-launch FP64 DMMA --
// The fused 3M product for complex128, on the FP64 tensor path
// (mma.sync.m16n8k4.f64; tcgen05 has no f64 kind).  CTA tile 32 x 32 complex
// outputs, 4 warps of 16 x 16, three CTAs per SM; K in blocks of 16 complex
// elements streamed global -> shared by cp.async (one 16-byte complex element
// per copy, zero filled outside the matrix) through a 3-deep ring.  The smem
// tile keeps the interleaved (re, im) pairs, so one 16-byte shared load gives a
// fragment element's real and imaginary part; per K step every warp issues
//     P1 += Ar Br,   P2 += Ai Bi,   P3 += (Ar + sa Ai)(Br + sb Bi)
// with the pre-additions made on the fragments in registers (sa, sb = -1 for
// conjugated operands), and the epilogue forms
//     Re = P1 - sa sb P2,   Im = P3 - P1 - sa sb P2
// and applies the complex alpha and beta (beta != 1 scales C, as the
// reference drivers do: src/gemm_driver.c:131).  Padding: +4 complex per row
// when K is contiguous, +2 otherwise, so both orientations' 16-byte fragment
// loads are conflict free.
// Bound: the FP64 pipe.  As in the real kernel (dgemm_fp64.cu) the next step's
// fragments are loaded, across a stage's edge too, before the current step's
// DMMAs issue, and tiles inside the matrices copy from running pointers.  The
// earlier form (one 512-thread CTA of 64 x 64 per SM, fragments loaded at
// their use) kept the pipe 75 % busy: 2048^3 1886 -> 1680 us on B200 (84 % busy).
// A 64 x 32 tile (two CTAs per SM) is no faster there and leaves small products
// with few CTAs and uneven last waves: 48^3 6.5 us against 4.6, 255^3 23.9 / 16.0,
// 1000^3 257 / 225, 1500^3 732 / 682, 2048^3 1679 / 1678.
constexpr int Z_BM = 32, Z_BN = 32, Z_BK = 16, Z_WM = 2, Z_WN = 2, Z_STAGES = 3;
constexpr int Z_NT = Z_WM * Z_WN * 32;

template <bool KC>
__host__ __device__ constexpr int z_pitch(int outer) {
  return KC ? Z_BK + 4 : outer + 2;
}
template <bool KC>
__host__ __device__ constexpr int z_stage_elems(int outer) {
  return (KC ? outer : Z_BK) * z_pitch<KC>(outer);
}

// Chunk i (one complex element per thread) of an OUTER x BK tile; element
// (o, k) at g[o*ld + k] when KC (K contiguous) else g[k*ld + o] (complex
// units).  Shared: KC -> [o][BK+4], else [k][OUTER+2].
template <int OUTER, bool KC>
__device__ __forceinline__ void z_load_chunk(uint32_t sbase, const double2 *__restrict__ g, int ld,
                                             int o0, int k0, int olim, int klim, int tid, int i) {
  constexpr int CPR = KC ? Z_BK : OUTER;
  const int c = tid + i * Z_NT, hi = c / CPR, lo = c % CPR;
  const int go = o0 + (KC ? hi : lo), gk = k0 + (KC ? lo : hi);
  const bool ok = go < olim && gk < klim;
  const double2 *src = ok ? g + (KC ? (size_t)go * ld + gk : (size_t)gk * ld + go) : g;
  const uint32_t dst = sbase + (uint32_t)(hi * z_pitch<KC>(OUTER) + lo) * 16u;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src),
               "r"(ok ? 16 : 0));
}

__device__ __forceinline__ void z_mma(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

template <bool A_KC, bool B_KC>
__global__ void __launch_bounds__(Z_NT, 3)
    zgemm3m_dmma_kernel(int M, int N, int K, const double2 *__restrict__ A, int lda,
                        const double2 *__restrict__ B, int ldb, double2 *__restrict__ C, int ldc,
                        double ar, double ai, double br, double bi, double sa, double sb) {
  constexpr int A_ST = z_stage_elems<A_KC>(Z_BM), B_ST = z_stage_elems<B_KC>(Z_BN);
  constexpr int A_LD = z_pitch<A_KC>(Z_BM), B_LD = z_pitch<B_KC>(Z_BN);
  extern __shared__ __align__(16) double2 zsh[];
  double2 *sA = zsh;
  double2 *sB = zsh + Z_STAGES * A_ST;
  const uint32_t sA_u = (uint32_t)__cvta_generic_to_shared(sA);
  const uint32_t sB_u = (uint32_t)__cvta_generic_to_shared(sB);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm0 = (warp / Z_WN) * 16, wn0 = (warp % Z_WN) * 16;
  const unsigned col0 = (blockIdx.z * gridDim.y + blockIdx.y) * Z_BN;
  if (col0 >= (unsigned)N) return;  // past the last tile, where column tiles fill several planes
  const int m0 = blockIdx.x * Z_BM, n0 = (int)col0;
  const int KT = (K + Z_BK - 1) / Z_BK;

  double acc[3][2][4];
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[p][j][v] = 0.0;

  constexpr int A_CPR = A_KC ? Z_BK : Z_BM, B_CPR = B_KC ? Z_BK : Z_BN;
  constexpr int A_CH = Z_BM * Z_BK / Z_NT, B_CH = Z_BN * Z_BK / Z_NT;
  static_assert(Z_NT % A_CPR == 0 && Z_NT % B_CPR == 0, "whole rows per chunk");
  const bool in_a = m0 + Z_BM <= M, in_b = n0 + Z_BN <= N;
  const double2 *pa = A + (A_KC ? (size_t)(m0 + tid / A_CPR) * lda + tid % A_CPR
                                : (size_t)(tid / A_CPR) * lda + m0 + tid % A_CPR);
  const double2 *pb = B + (B_KC ? (size_t)(n0 + tid / B_CPR) * ldb + tid % B_CPR
                                : (size_t)(tid / B_CPR) * ldb + n0 + tid % B_CPR);
  const uint32_t da = sA_u + (uint32_t)((tid / A_CPR) * A_LD + tid % A_CPR) * 16u;
  const uint32_t db = sB_u + (uint32_t)((tid / B_CPR) * B_LD + tid % B_CPR) * 16u;
  const size_t ia = (size_t)(Z_NT / A_CPR) * lda, ib = (size_t)(Z_NT / B_CPR) * ldb;
  const size_t ka = A_KC ? (size_t)Z_BK : (size_t)Z_BK * lda;
  const size_t kb = B_KC ? (size_t)Z_BK : (size_t)Z_BK * ldb;
  // Copies stage kt (called once per kt, in order) into ring slot st.
  auto load_stage = [&](int st, int kt) {
    const bool full = (kt + 1) * Z_BK <= K;
#pragma unroll
    for (int c = 0; c < A_CH; ++c) {
      if (full && in_a)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                         da + (uint32_t)(st * A_ST + c * (Z_NT / A_CPR) * A_LD) * 16u),
                     "l"(pa + c * ia));
      else
        z_load_chunk<Z_BM, A_KC>(sA_u + st * A_ST * 16, A, lda, m0, kt * Z_BK, M, K, tid, c);
    }
#pragma unroll
    for (int c = 0; c < B_CH; ++c) {
      if (full && in_b)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                         db + (uint32_t)(st * B_ST + c * (Z_NT / B_CPR) * B_LD) * 16u),
                     "l"(pb + c * ib));
      else
        z_load_chunk<Z_BN, B_KC>(sB_u + st * B_ST * 16, B, ldb, n0, kt * Z_BK, N, K, tid, c);
    }
    pa += ka;
    pb += kb;
  };
  // Fragments of K step kk (4 complex k) of stage st: A rows g, g + 8, B
  // columns g of the two 8-column blocks, k = kk + t.
  double2 af[2][2], bf[2][2];
  auto load_frags = [&](int buf, int st, int kk) {
    const double2 *As = sA + st * A_ST, *Bs = sB + st * B_ST;
    const int k = kk + t;
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int m = wm0 + g + 8 * v, n = wn0 + g + 8 * v;
      af[buf][v] = A_KC ? As[m * A_LD + k] : As[k * A_LD + m];
      bf[buf][v] = B_KC ? Bs[n * B_LD + k] : Bs[k * B_LD + n];
    }
  };

#pragma unroll
  for (int st = 0; st < Z_STAGES - 1; ++st) {
    if (st < KT) load_stage(st, st);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  asm volatile("cp.async.wait_group %0;\n" ::"n"(Z_STAGES - 2));
  __syncthreads();
  load_frags(0, 0, 0);
  int st = 0, st_fill = Z_STAGES - 1;
  for (int kt = 0; kt < KT; ++kt) {
    const int st_next = st + 1 == Z_STAGES ? 0 : st + 1;
#pragma unroll
    for (int ks = 0; ks < Z_BK / 4; ++ks) {
      const int cur = ks & 1;
      if (ks + 1 < Z_BK / 4) load_frags(cur ^ 1, st, 4 * (ks + 1));
      // every warp has issued its last reads of stage kt - 1, which is refilled here
      if (ks == 0 && kt + Z_STAGES - 1 < KT) load_stage(st_fill, kt + Z_STAGES - 1);
      if (ks + 1 == Z_BK / 4) {
        asm volatile("cp.async.commit_group;\n" ::);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(Z_STAGES - 2));
        __syncthreads();
        if (kt + 1 < KT) load_frags(cur ^ 1, st_next, 0);
      }
      const double2 a0 = af[cur][0], a1 = af[cur][1];
#pragma unroll
      for (int j = 0; j < 2; ++j) z_mma(acc[0][j], a0.x, a1.x, bf[cur][j].x);
#pragma unroll
      for (int j = 0; j < 2; ++j) z_mma(acc[1][j], a0.y, a1.y, bf[cur][j].y);
      const double s0 = fma(sa, a0.y, a0.x), s1 = fma(sa, a1.y, a1.x);
#pragma unroll
      for (int j = 0; j < 2; ++j)
        z_mma(acc[2][j], s0, s1, fma(sb, bf[cur][j].y, bf[cur][j].x));
    }
    st = st_next;
    st_fill = st_fill + 1 == Z_STAGES ? 0 : st_fill + 1;
  }
  asm volatile("cp.async.wait_group 0;\n" ::);

  // Fragment (j, v): row g + 8 (v >> 1), column 2t + (v & 1) of the warp tile.
  // All of C is read before any of it is written (a load between two stores
  // would wait for the one before it).
  const double s2 = sa * sb;
  const bool beta_one = br == 1.0 && bi == 0.0;
  double2 cv[2][4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int m = m0 + wm0 + g + 8 * (v >> 1), n = n0 + wn0 + j * 8 + 2 * t + (v & 1);
      cv[j][v] = (m < M && n < N) ? C[(size_t)n * ldc + m] : make_double2(0.0, 0.0);
    }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int m = m0 + wm0 + g + 8 * (v >> 1);
      const int n = n0 + wn0 + j * 8 + 2 * t + (v & 1);
      if (m < M && n < N) {
        const double p1 = acc[0][j][v], p2 = s2 * acc[1][j][v], p3 = acc[2][j][v];
        const double re = p1 - p2, im = p3 - p1 - p2;
        double2 c = cv[j][v];
        if (!beta_one) c = make_double2(br * c.x - bi * c.y, br * c.y + bi * c.x);
        C[(size_t)n * ldc + m] =
            make_double2(c.x + (ar * re - ai * im), c.y + (ar * im + ai * re));
      }
    }
}

template <bool AK, bool BKc>
int launch_zgemm3m_dmma(int m, int n, int k, const double *A, int lda, const double *B, int ldb,
                        double *C, int ldc, double ar, double ai, double br, double bi, double sa,
                        double sb, cudaStream_t s) {
  constexpr size_t SMEM =
      (size_t)Z_STAGES * (z_stage_elems<AK>(Z_BM) + z_stage_elems<BKc>(Z_BN)) * 16;
  auto kern = zgemm3m_dmma_kernel<AK, BKc>;
  B2_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM));
  // Column tiles over y and, from N = 2097121 on, z: y ends at 65535.  (One flat
  // dimension divided by the row tiles in the kernel: 2048^3 1679 -> 1692 us on B200.)
  const unsigned tn = (unsigned)((n + Z_BN - 1) / Z_BN), planes = (tn + 65534) / 65535;
  dim3 grid((unsigned)((m + Z_BM - 1) / Z_BM), (tn + planes - 1) / planes, planes);
  B2_PROF("zgemm3m_dmma", s);
  kern<<<grid, Z_NT, SMEM, s>>>(m, n, k, reinterpret_cast<const double2 *>(A), lda,
                                reinterpret_cast<const double2 *>(B), ldb,
                                reinterpret_cast<double2 *>(C), ldc, ar, ai, br, bi, sa, sb);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

template <typename T>
__global__ void cscale_kernel(int M, int N, T br, T bi, T *__restrict__ C, int ldc) {
  const long long total = (long long)M * N;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int m = (int)(idx % M), n = (int)(idx / M);
    T *c = C + 2 * ((long long)n * ldc + m);
    const T cr = c[0], ci = c[1];
    c[0] = br * cr - bi * ci;
    c[1] = br * ci + bi * cr;
  }
}

}  // namespace

// ------------------------------------------ large products: 3 real GEMMs --
// Real and imaginary parts of op(X) (R x Cc, element (r, c) at
// X[2*(r*ld + c)] when transposed, else X[2*(c*ld + r)]; imaginary part times
// sgn for conjugation) and their sum, column-major with leading dimension R.
template <typename T>
__global__ void prep3m_kernel(const T *__restrict__ X, int ld, bool trans, T sgn, int R, int Cc,
                              T *__restrict__ outr, T *__restrict__ outi, T *__restrict__ outs) {
  const long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (r >= R) return;
  for (long long c = blockIdx.y; c < Cc; c += gridDim.y) {
    const T *p = X + 2 * (trans ? r * ld + c : c * ld + r);
    const T re = p[0], im = sgn * p[1];
    const long long o = r + c * (long long)R;
    outr[o] = re;
    outi[o] = im;
    outs[o] = re + im;
  }
}

// C = alpha (P1 - P2 + i (P3 - P1 - P2)) + beta C, beta applied when != 1.
template <typename T>
__global__ void combine3m_kernel(const T *__restrict__ P, long long plane, int M, int N, T ar,
                                 T ai, T br, T bi, T *__restrict__ C, int ldc) {
  const long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (m >= M) return;
  for (long long n = blockIdx.y; n < N; n += gridDim.y) {
    const long long o = m + n * M;
    const T p1 = P[o], p2 = P[plane + o], p3 = P[2 * plane + o];
    epilogue3m(C, ldc, (int)m, (int)n, p1, p2, p3, ar, ai, br, bi);
  }
}

// Large zgemm3m products: the three real products run as the library's own
// FP64 DMMA GEMMs between one pre-add pass and one post-combination pass --
// both HBM-bound.  (cgemm3m: cgemm3m_tensor.)
int zgemm3m_three_gemms(char ta, char tb, int m, int n, int k, double ar, double ai, double br,
                        double bi, const double *A, int lda, const double *B, int ldb, double *C,
                        int ldc, cudaStream_t s) {
  using T = double;
  Ctx *cx = ctx();
  if (!cx) return B2_ERR_NO_DEVICE;
  const bool tA = !(ta == 'N' || ta == 'n' || ta == 'R' || ta == 'r');
  const bool tB = !(tb == 'N' || tb == 'n' || tb == 'R' || tb == 'r');
  const T sA = (ta == 'C' || ta == 'c' || ta == 'R' || ta == 'r') ? (T)-1 : (T)1;
  const T sB = (tb == 'C' || tb == 'c' || tb == 'R' || tb == 'r') ? (T)-1 : (T)1;
  const long long pa = (long long)m * k, pb = (long long)k * n, pc = (long long)m * n;
  T *W = (T *)workspace(cx, WS_3M, (size_t)(3 * pa + 3 * pb + 3 * pc) * sizeof(T));
  if (!W) return B2_ERR_NOMEM;
  T *Ar = W, *Ai = Ar + pa, *As = Ai + pa;
  T *Br = As + pa, *Bi = Br + pb, *Bs = Bi + pb;
  T *P = Bs + pb;
  {
    B2_PROF("gemm3m_prep", s);
    dim3 ga((unsigned)((m + 255) / 256), (unsigned)(k < 4096 ? k : 4096));
    prep3m_kernel<T><<<ga, 256, 0, s>>>(A, lda, tA, sA, m, k, Ar, Ai, As);
    dim3 gb((unsigned)((k + 255) / 256), (unsigned)(n < 4096 ? n : 4096));
    prep3m_kernel<T><<<gb, 256, 0, s>>>(B, ldb, tB, sB, k, n, Br, Bi, Bs);
    B2_CUDA_TRY(cudaGetLastError());
  }
  // beta = 0 still multiplies the output (reference semantics): start at zero
  B2_CUDA_TRY(cudaMemsetAsync(P, 0, (size_t)(3 * pc) * sizeof(T), s));
  const T *X[3] = {Ar, Ai, As}, *Y[3] = {Br, Bi, Bs};
  for (int t = 0; t < 3; ++t) {
    const int st =
        dgemm_fp64('N', 'N', m, n, k, 1.0, X[t], m, Y[t], k, 0.0, P + t * pc, m, s, nullptr);
    if (st != B2_OK) return st;
  }
  B2_PROF("gemm3m_combine", s);
  dim3 gc((unsigned)((m + 255) / 256), (unsigned)(n < 4096 ? n : 4096));
  combine3m_kernel<T><<<gc, 256, 0, s>>>(P, pc, m, n, ar, ai, br, bi, C, ldc);
  B2_CUDA_TRY(cudaGetLastError());
  return B2_OK;
}

// cgemm3m in ONE tensor-core GEMM launch: the three real products of the 3M
// method run as 3xTF32 on the single-CTA tcgen05 engine in its three-
// accumulator mode -- each work unit is a 128 x 128 tile of C that multiplies
// batch 0 (Br, Ar), 1 (Bi, Ai) and 2 (Br + Bi, Ar + Ai) of the split operands
// into three TMEM accumulators of 128 columns, and the epilogue forms
// Re = P1 - P2, Im = P3 - P1 - P2 and C = alpha (Re + i Im) + beta C from
// them, so P1/P2/P3 never leave the SM.  The pre-adds (and conjugation /
// transposition) and the TF32 big/small splits stay passes in front.
constexpr int C3M_BN = 128, C3M_STAGES = 6;  // 128 x 128 tiles, one accumulator set

struct C3MEpi {
  float *C;
  int ldc;
  int M, N;  // C is M x N; the engine's P runs over N, Q over M
  float ar, ai, br, bi;
  __device__ __forceinline__ void operator()(int p, int q0, const uint32_t (&v0)[32],
                                             const uint32_t (&v1)[32],
                                             const uint32_t (&v2)[32]) const {
    if (p >= N || q0 >= M) return;
    const int nq = min(32, M - q0);
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < nq)
        epilogue3m<float>(C, ldc, q0 + j, p, __uint_as_float(v0[j]), __uint_as_float(v1[j]),
                          __uint_as_float(v2[j]), ar, ai, br, bi);
  }
};

int cgemm3m_fused_tc(char ta, char tb, int m, int n, int k, float ar, float ai, float br,
                     float bi, const float *A, int lda, const float *B, int ldb, float *C,
                     int ldc, cudaStream_t s) {
  Ctx *cx = ctx();
  if (!cx) return B2_ERR_NO_DEVICE;
  const bool tA = !(ta == 'N' || ta == 'n' || ta == 'R' || ta == 'r');
  const bool tB = !(tb == 'N' || tb == 'n' || tb == 'R' || tb == 'r');
  const float sA = (ta == 'C' || ta == 'c' || ta == 'R' || ta == 'r') ? -1.f : 1.f;
  const float sB = (tb == 'C' || tb == 'c' || tb == 'R' || tb == 'r') ? -1.f : 1.f;
  const long long pa = (long long)m * k, pb = (long long)k * n;
  float *W = (float *)workspace(cx, WS_3M, (size_t)(3 * pa + 3 * pb) * sizeof(float));
  if (!W) return B2_ERR_NOMEM;
  float *Ar = W, *Ai = Ar + pa, *As = Ai + pa;
  float *Br = As + pa, *Bi = Br + pb, *Bs = Bi + pb;
  {
    B2_PROF("gemm3m_prep", s);
    dim3 ga((unsigned)((m + 255) / 256), (unsigned)(k < 4096 ? k : 4096));
    prep3m_kernel<float><<<ga, 256, 0, s>>>(A, lda, tA, sA, m, k, Ar, Ai, As);
    dim3 gb((unsigned)((k + 255) / 256), (unsigned)(n < 4096 ? n : 4096));
    prep3m_kernel<float><<<gb, 256, 0, s>>>(B, ldb, tB, sB, k, n, Br, Bi, Bs);
    B2_CUDA_TRY(cudaGetLastError());
  }
  // split planes: Y[t] = rows of op(A) parts (m x [big|small]), X[t] = columns
  // of op(B) parts (n x [big|small]), t = 0, 1, 2 the three products
  const int kp = (int)((k + 31) / 32 * 32);
  const long long ks = 2LL * kp;
  float *Yp = (float *)workspace(cx, WS_SPLIT_Y, (size_t)(3 * m * ks) * sizeof(float));
  float *Xp = (float *)workspace(cx, WS_SPLIT_X, (size_t)(3 * n * ks) * sizeof(float));
  if (!Yp || !Xp) return B2_ERR_NOMEM;
  const float *Ya[3] = {Ar, Ai, As}, *Xb[3] = {Br, Bi, Bs};
  for (int t = 0; t < 3; ++t) {
    int rc = sgemm_split_tf32x3(Ya[t], 1, m, m, k, kp, Yp + t * m * ks, s);
    if (rc == B2_OK) rc = sgemm_split_tf32x3(Xb[t], k, 1, n, k, kp, Xp + t * n * ks, s);
    if (rc != B2_OK) return rc;
  }
  CUtensorMap tmX, tmY;
  int rc = umma::make_kmajor_map(&tmX, umma::KIND_TF32, Xp, ks, n, 3, ks * 4, (long long)n * ks * 4,
                                 umma::BM);
  if (rc == B2_OK)
    rc = umma::make_kmajor_map(&tmY, umma::KIND_TF32, Yp, ks, m, 3, ks * 4, (long long)m * ks * 4,
                               C3M_BN);
  if (rc != B2_OK) return rc;
  // three-term interleave as in the 3xTF32 SGEMM: terms (Bb, Ab), (Bs, Ab), (Bb, As)
  const int seg_kb = kp * 4 / umma::KBLOCK_BYTES;
  C3MEpi epi{C, ldc, m, n, ar, ai, br, bi};
  return umma::launch<umma::KIND_TF32, C3M_BN, C3M_STAGES, C3MEpi, 3>(tmX, tmY, n, m, 3LL * kp, 3, epi,
                                                         cx->sm_count, cx->derr, s,
                                                         "cgemm3m_umma", 0, nullptr, 1, seg_kb,
                                                         0x2u, 0x4u);
}

template <typename T>
int gemm3m_device(char ta, char tb, int m, int n, int k, const T *alpha, const T *A, int lda,
                  const T *B, int ldb, const T *beta, T *C, int ldc, cudaStream_t s) {
  if (m <= 0 || n <= 0) return B2_OK;
  const T ar = alpha[0], ai = alpha[1], br = beta[0], bi = beta[1];
  if (k <= 0 || (ar == (T)0 && ai == (T)0)) {
    if (br == (T)1 && bi == (T)0) return B2_OK;
    const long long total = (long long)m * n;
    const int blocks = (int)((total + 255) / 256 > 4096 ? 4096 : (total + 255) / 256);
    B2_PROF("gemm3m_scale", s);
    cscale_kernel<T><<<blocks, 256, 0, s>>>(m, n, br, bi, C, ldc);
    B2_CUDA_TRY(cudaGetLastError());
    return B2_OK;
  }
  if constexpr (sizeof(T) == 8) {
    // complex128: the one-launch DMMA kernel (16-byte aligned operands, the
    // normal case; an odd-aligned pointer takes the other paths) below 2^35
    // multiply-adds, 2048^3 included: the pre-adds, the three products and
    // the combination never leave the SM, and no intermediate planes are
    // allocated (the three-GEMM form needs 3 (m k + k n + m n) doubles of
    // workspace, 302 MB at 2048^3).  It runs 2 % below the three DMMA GEMMs
    // there (40.8 against 41.6 TFLOPS effective).  The three GEMMs take over
    // from 2^35: at 4096^3 they run at 45.1 TFLOPS effective against 41.5 for
    // the one launch.  B2_Z3M_FUSED_MAX (multiply-adds)
    // moves the limit.
    static const double fused_max = [] {
      const char *e = getenv("B2_Z3M_FUSED_MAX");
      return e ? atof(e) : 34359738368.0;
    }();
    const bool al16 = (((uintptr_t)A | (uintptr_t)B | (uintptr_t)C) & 15) == 0;
    if (al16 && (double)m * n * k < fused_max) {
      const bool tA = !(ta == 'N' || ta == 'n' || ta == 'R' || ta == 'r');
      const bool tB = !(tb == 'N' || tb == 'n' || tb == 'R' || tb == 'r');
      const double sA = (ta == 'C' || ta == 'c' || ta == 'R' || ta == 'r') ? -1.0 : 1.0;
      const double sB = (tb == 'C' || tb == 'c' || tb == 'R' || tb == 'r') ? -1.0 : 1.0;
      const bool ak = tA, bk = !tB;  // K contiguous in memory
      if (ak && bk)
        return launch_zgemm3m_dmma<true, true>(m, n, k, A, lda, B, ldb, C, ldc, ar, ai, br, bi, sA, sB, s);
      if (ak)
        return launch_zgemm3m_dmma<true, false>(m, n, k, A, lda, B, ldb, C, ldc, ar, ai, br, bi, sA, sB, s);
      if (bk)
        return launch_zgemm3m_dmma<false, true>(m, n, k, A, lda, B, ldb, C, ldc, ar, ai, br, bi, sA, sB, s);
      return launch_zgemm3m_dmma<false, false>(m, n, k, A, lda, B, ldb, C, ldc, ar, ai, br, bi, sA, sB, s);
    }
  }
  if ((double)m * n * k >= 16777216.0) {
    if constexpr (sizeof(T) == 4) {
      // One tensor-core launch (cgemm3m_fused_tc) when B2_C3M_FUSED=1 and its
      // 128 x 128 tiles fill the SMs.  Off by default: at 2048^3 it takes 0.577 ms
      // against 0.308 of the batched products (4096^3: 3.12 against 1.66 ms), and its
      // full-K FP32 accumulation gives 2.1e-5 relative error against 3.8e-6.
      static const bool fused_on = [] {
        const char *e = getenv("B2_C3M_FUSED");
        return e && e[0] == '1';
      }();
      Ctx *cx = ctx();
      const long long tiles = (long long)((n + 127) / 128) * ((m + C3M_BN - 1) / C3M_BN);
      if (fused_on && cx && tiles >= cx->sm_count)
        return cgemm3m_fused_tc(ta, tb, m, n, k, ar, ai, br, bi, A, lda, B, ldb, C, ldc, s);
    }
    if constexpr (sizeof(T) == 4)
      return cgemm3m_tensor(ta, tb, m, n, k, ar, ai, br, bi, A, lda, B, ldb, C, ldc, s);
    else
      return zgemm3m_three_gemms(ta, tb, m, n, k, ar, ai, br, bi, A, lda, B, ldb, C, ldc, s);
  }
  if constexpr (sizeof(T) == 8) {
    dim3 grid((m + G_BM - 1) / G_BM, (n + G_BN - 1) / G_BN);
    const int smem = (int)(12 * G_BK * G_LD * sizeof(T));
    B2_CUDA_TRY(cudaFuncSetAttribute(zgemm3m_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    B2_PROF("zgemm3m_fused", s);
    zgemm3m_kernel<<<grid, 256, smem, s>>>(m, n, k, A, lda, B, ldb, C, ldc, ar, ai, br, bi, ta, tb);
    B2_CUDA_TRY(cudaGetLastError());
    return B2_OK;
  } else {
    const bool ak = tr_is_t(ta), bk = !tr_is_t(tb);  // K contiguous in memory
    const float sa = tr_is_conj(ta) ? -1.f : 1.f, sb = tr_is_conj(tb) ? -1.f : 1.f;
    if (ak && bk)
      return launch_cgemm3m<true, true>(m, n, k, A, lda, B, ldb, C, ldc, ar, ai, br, bi, sa, sb, s);
    if (ak)
      return launch_cgemm3m<true, false>(m, n, k, A, lda, B, ldb, C, ldc, ar, ai, br, bi, sa, sb, s);
    if (bk)
      return launch_cgemm3m<false, true>(m, n, k, A, lda, B, ldb, C, ldc, ar, ai, br, bi, sa, sb, s);
    return launch_cgemm3m<false, false>(m, n, k, A, lda, B, ldb, C, ldc, ar, ai, br, bi, sa, sb, s);
  }
}

template int gemm3m_device<double>(char, char, int, int, int, const double *, const double *, int,
                                   const double *, int, const double *, double *, int,
                                   cudaStream_t);
template int gemm3m_device<float>(char, char, int, int, int, const float *, const float *, int,
                                  const float *, int, const float *, float *, int, cudaStream_t);

}  // namespace b2
