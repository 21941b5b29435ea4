// sgemm.cu -- SGEMM methods.
//
// Native FP32 replaces the reference's AVX-512 SGEMM (src/gemm_driver.c:116
// built without -DDOUBLE driving the 48x8 tile of src/kernel/gemm_kernel.S,
// and the m16 x n24 tiles of OpenBLAS-like_implementation/sgemm.c:366-412):
// a CUDA-core kernel of paired FP32 FMAs (fma.rn.f32x2) with a 128x128 CTA
// tile, 8x8 outputs per thread in registers, K panels in a cp.async ring, and a
// 64x64 form for products that leave SMs idle.  The tensor-core forms (TF32, 3xTF32, 3xBF16) run on the tcgen05
// engine (sgemm_tc.cu).
#include "b2_methods.cuh"
#include "b2_profile.cuh"
#include "fp32_copy.cuh"

namespace b2 {
namespace {

// ----------------------------------------------------------------------
// Paired-FMA FP32 kernel (sm_100 fma.rn.f32x2: two FP32 FMAs per issued
// instruction, so the FFMA pipe, not instruction issue, is the limit).
// CTA tile 128 x 128, K blocks of 16, 256 threads of 8 x 8 outputs, K panels
// copied by cp.async through a 3-deep ring as [k][m] and [k][n] (16 bytes at a
// time where the operand is contiguous that way and aligned, else 4: a panel
// staged through registers needs 16 of the 128, which spilled).  Thread (tx, ty) owns rows
// 4 tx + {0..3} + 64 h' and columns 4 ty + {0..3} + 64 h (h', h = 0, 1): per
// K step it reads two 16-byte A vectors and two 16-byte B vectors (64 bytes
// for 64 FMAs -- the shared-memory rate of 128 bytes per clock per SM then
// matches the 128 FMAs per clock) and forms the broadcast pairs (a, a) in
// registers.  Storing A duplicated in shared memory instead (one 16-byte load
// giving two pairs) cost 96 bytes per 64 FMAs and made the kernel
// shared-memory bound (ncu at 4096^3: L1 84 % busy, FMA pipe 55 %).  Two CTAs
// per SM (128 registers, a few bytes spilled) beat one CTA with 150 registers:
// 54.4 against 51.3 TFLOPS at 8192^3, 52.6 against 49.0 at 4096^3.
constexpr int S2_M = 128, S2_N = 128, S2_K = 16, S2_APAD = 4, S2_BPAD = 4;
constexpr int S2_ALD = S2_M + S2_APAD;  // floats per k row of the A panel
constexpr int S2_BLD = S2_N + S2_BPAD;
constexpr int S2_STAGES = 3;
constexpr int S2_STAGE = S2_K * (S2_ALD + S2_BLD);  // floats per stage: A panel, B panel
constexpr int S2_SMEM = S2_STAGES * S2_STAGE * 4;

__device__ __forceinline__ unsigned long long dup2(float a) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(a));
  return d;
}

__device__ __forceinline__ void ffma2(unsigned long long &c, unsigned long long a,
                                      unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

// MODE 0: tiles [tile0, tile0 + gridDim.x) of C in full; MODE 1: K slice
// blockIdx.z of a split-K product, its raw sums to P + z*plane (ld ldp); MODE 2:
// K slice blockIdx.z of tile tile0 + blockIdx.x, the raw sums of its 128 x 128
// outputs to P + (z*gridDim.x + blockIdx.x)*128*128.  Tiles run down the columns.
// dependents: the launch after this one (MODE 2, other tiles) may start as these
// blocks leave.
template <bool TA, bool TB, bool VEC, int MODE>
__global__ void __launch_bounds__(256, 2)
    sgemm_ffma2_kernel(int M, int N, int K, float alpha, const float *__restrict__ A, int lda,
                       const float *__restrict__ B, int ldb, float beta, float *__restrict__ C,
                       int ldc, int kchunk, float *__restrict__ P, long long plane, int ldp,
                       int tiles_m, int tile0, int dependents) {
  constexpr bool SPLIT = MODE != 0;
  if (dependents) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  extern __shared__ __align__(16) float s2mem[];  // stages of [S2_K][S2_ALD], [S2_K][S2_BLD]
  const uint32_t smem_u = (uint32_t)__cvta_generic_to_shared(s2mem);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int tile = tile0 + (int)blockIdx.x;
  const int m0 = tile % tiles_m * S2_M, n0 = tile / tiles_m * S2_N;
  // K range of this CTA (kchunk a multiple of S2_K)
  const int kbeg = SPLIT ? blockIdx.z * kchunk : 0;
  const int kend = SPLIT ? min(K, kbeg + kchunk) : K;

  unsigned long long acc[8][4];  // row r: 4tx + (r&3) + 64(r>>2); column pair c
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0ull;

  const int KT = (kend - kbeg + S2_K - 1) / S2_K;
  const bool in_a = m0 + S2_M <= M, in_b = n0 + S2_N <= N;
  constexpr bool KA = TA, KB = !TB;  // K contiguous
  const float *pa = A + f32copy::run_offset<S2_M, KA, VEC>(m0, kbeg, lda, tid);
  const float *pb = B + f32copy::run_offset<S2_N, KB, VEC>(n0, kbeg, ldb, tid);
  const uint32_t da = smem_u + f32copy::run_dst<S2_M, S2_ALD, KA, VEC>(tid);
  const uint32_t db = smem_u + S2_K * S2_ALD * 4u + f32copy::run_dst<S2_N, S2_BLD, KB, VEC>(tid);
  // Copies stage kt (called once per kt, in order) into ring slot st.
  auto load_stage = [&](int st, int kt) {
    const int k0 = kbeg + kt * S2_K;
    const bool full = k0 + S2_K <= kend;
    const uint32_t d = (uint32_t)(st * S2_STAGE) * 4u;
    if (full && in_a) f32copy::run_panel<S2_M, S2_ALD, KA, VEC>(da + d, pa, lda);
    else f32copy::load_panel<S2_M, S2_ALD, KA, VEC>(smem_u + d, A, lda, m0, k0, M, kend, tid);
    if (full && in_b) f32copy::run_panel<S2_N, S2_BLD, KB, VEC>(db + d, pb, ldb);
    else
      f32copy::load_panel<S2_N, S2_BLD, KB, VEC>(smem_u + d + S2_K * S2_ALD * 4u, B, ldb, n0, k0, N,
                                                 kend, tid);
    pa += KA ? (size_t)S2_K : (size_t)S2_K * lda;
    pb += KB ? (size_t)S2_K : (size_t)S2_K * ldb;
  };
#pragma unroll
  for (int i = 0; i < S2_STAGES - 1; ++i) {
    if (i < KT) load_stage(i, i);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  int st = 0, st_fill = S2_STAGES - 1;
  for (int kt = 0; kt < KT; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(S2_STAGES - 2));
    __syncthreads();  // stage kt is in, and every thread is done with the one refilled here
    if (kt + S2_STAGES - 1 < KT) load_stage(st_fill, kt + S2_STAGES - 1);
    asm volatile("cp.async.commit_group;\n" ::);
    const float *as = s2mem + st * S2_STAGE;
    const float *bs = as + S2_K * S2_ALD;
    st = st + 1 == S2_STAGES ? 0 : st + 1;
    st_fill = st_fill + 1 == S2_STAGES ? 0 : st_fill + 1;
#pragma unroll
    for (int kk = 0; kk < S2_K; ++kk) {
      float av[8];  // rows 4tx + i + 64h'
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const float4 v = *reinterpret_cast<const float4 *>(as + kk * S2_ALD + 64 * hh + 4 * tx);
        const int sw = TA && kk >= 8 ? 2 : 0;  // panel_at's order
        av[4 * hh + sw] = v.x;
        av[4 * hh + 1 + sw] = v.y;
        av[4 * hh + (2 ^ sw)] = v.z;
        av[4 * hh + (3 ^ sw)] = v.w;
      }
      ulonglong2 b2[2];  // columns 64h + 4ty .. 64h + 4ty + 3
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const ulonglong2 v =
            *reinterpret_cast<const ulonglong2 *>(bs + kk * S2_BLD + 64 * h + 4 * ty);
        const bool sw = !TB && kk >= 8;
        b2[h] = make_ulonglong2(sw ? v.y : v.x, sw ? v.x : v.y);
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const unsigned long long a = dup2(av[r]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          ffma2(acc[r][2 * h], a, b2[h].x);
          ffma2(acc[r][2 * h + 1], a, b2[h].y);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  // Output element (r, c, e): row 4tx + (r & 3) + 64 (r >> 2), column
  // 64 (c >> 1) + 4ty + 2 (c & 1) + e.
  auto value = [&](int r, int col) {  // col = 2c + e
    const float2 v = *reinterpret_cast<const float2 *>(&acc[r][col >> 1]);
    return (col & 1) ? v.y : v.x;
  };
  auto column = [&](int col) { return 64 * (col >> 2) + 4 * ty + (col & 3); };
  if (MODE == 2) {
    float *T = P + ((long long)blockIdx.z * gridDim.x + blockIdx.x) * (S2_M * S2_N);
#pragma unroll
    for (int col = 0; col < 8; ++col)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float4 *>(T + column(col) * S2_M + 64 * h + 4 * tx) =
            make_float4(value(4 * h, col), value(4 * h + 1, col), value(4 * h + 2, col),
                        value(4 * h + 3, col));
    // this launch ends only after the one it overlaps
    asm volatile("griddepcontrol.wait;" ::: "memory");
    return;
  }
  if (MODE == 1) {
#pragma unroll
    for (int col = 0; col < 8; ++col) {
      const int n = n0 + column(col);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int m = m0 + 4 * tx + (r & 3) + 64 * (r >> 2);
        if (m < M && n < N) P[blockIdx.z * plane + (long long)n * ldp + m] = value(r, col);
      }
    }
    return;
  }
  // C two columns at a time, all of their reads before their writes (between
  // two writes each read would wait for the one before it)
  const bool beta_one = (beta == 1.f);
  const bool cvec = (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (ldc & 3) == 0;
  const bool inside = m0 + S2_M <= M && n0 + S2_N <= N;
#pragma unroll
  for (int q = 0; q < 8; q += 2) {
    float old[2][8];
    if (cvec && inside) {
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 v = *reinterpret_cast<const float4 *>(
              C + (size_t)(n0 + column(q + u)) * ldc + m0 + 64 * h + 4 * tx);
          old[u][4 * h] = v.x, old[u][4 * h + 1] = v.y;
          old[u][4 * h + 2] = v.z, old[u][4 * h + 3] = v.w;
        }
    } else {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int n = n0 + column(q + u);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const int m = m0 + 4 * tx + (r & 3) + 64 * (r >> 2);
          old[u][r] = (m < M && n < N) ? C[(size_t)n * ldc + m] : 0.f;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float x = value(r, q + u);
        old[u][r] = beta_one ? fmaf(alpha, x, old[u][r]) : fmaf(alpha, x, beta * old[u][r]);
      }
    if (cvec && inside) {
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          *reinterpret_cast<float4 *>(C + (size_t)(n0 + column(q + u)) * ldc + m0 + 64 * h +
                                      4 * tx) =
              make_float4(old[u][4 * h], old[u][4 * h + 1], old[u][4 * h + 2], old[u][4 * h + 3]);
    } else {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int n = n0 + column(q + u);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const int m = m0 + 4 * tx + (r & 3) + 64 * (r >> 2);
          if (m < M && n < N) C[(size_t)n * ldc + m] = old[u][r];
        }
      }
    }
  }
}

// C = alpha * (sum of the K slices of tiles tile0 .. tile0 + tiles - 1, in FP64
// and slice order) + beta * C; 16 blocks per tile, four rows per thread.
__global__ void __launch_bounds__(256)
    ffma2_tail_reduce_kernel(const float *__restrict__ P, int tiles, int S, int M, int N,
                             float alpha, float beta, float *__restrict__ C, int ldc, int tiles_m,
                             int tile0) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int lt = blockIdx.x >> 4, idx = ((blockIdx.x & 15) * 256 + threadIdx.x) * 4;
  const int tile = tile0 + lt;
  const int m = tile % tiles_m * S2_M + idx % S2_M, n = tile / tiles_m * S2_N + idx / S2_M;
  if (m >= M || n >= N) return;
  const float *p = P + (long long)lt * (S2_M * S2_N) + idx;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
  for (int z = 0; z < S; ++z) {
    const float4 x =
        *reinterpret_cast<const float4 *>(p + (long long)z * tiles * (S2_M * S2_N));
    acc[0] += (double)x.x, acc[1] += (double)x.y, acc[2] += (double)x.z, acc[3] += (double)x.w;
  }
  float *c = C + (size_t)n * ldc + m;
  float old[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) old[e] = m + e < M ? c[e] : 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float a = (float)acc[e];
    if (m + e < M) c[e] = (beta == 1.f) ? fmaf(alpha, a, old[e]) : fmaf(alpha, a, beta * old[e]);
  }
}

// K slices for a grid of `tiles` CTAs at two per SM: 1 when the tiles fill
// the slots, else the count (at most 8, each slice >= 32 K blocks of 16)
// whose work units best fill whole waves of 2 * sms.  8192 x 256 x 8192 has
// 128 tiles for the 296 slots of 148 SMs; 2 slices fill them 86 %.
int ffma2_ksplit(long long tiles, int kblocks, int sms) {
  const long long slots = 2ll * sms;
  if (tiles >= slots) return 1;
  int best = 1;
  double best_eff = (double)tiles / slots;
  for (int S = 2; S <= 8 && S * 32 <= kblocks; ++S) {
    const long long units = tiles * S, waves = (units + slots - 1) / slots;
    const double eff = (double)units / (double)(waves * slots);
    if (eff > best_eff + 0.02) {
      best = S;
      best_eff = eff;
    }
  }
  return best;
}

// ----------------------------------------------------------------------
// Small products: 64 x 64 tiles, so that four times the CTAs share them, and
// four groups of 64 threads of 8 x 8 outputs that take every fourth k of a panel
// (a chain of K panels bounds a call that leaves SMs idle, and a panel is 0.4 us
// here against 1.7 for a lone 128 x 128 CTA).  Shared reads and paired FMAs are
// in the big tile's proportion.  The groups exchange column pairs of their sums
// through shared memory; group g finishes pair g of each thread's four.
// Slices of K (blockIdx.z) write their raw sums to P (plane, ldp); else C.
constexpr int S4_T = 64, S4_K = 16, S4_LD = S4_T + 4, S4_STAGES = 4;
constexpr int S4_PANEL = S4_K * S4_LD;
constexpr int S4_SMEM = 3 * 16 * 256 * 4;  // the exchange; 48 KB
static_assert(S4_STAGES * 2 * S4_PANEL * 4 <= S4_SMEM, "the ring fits where the exchange goes");

template <bool TA, bool TB, bool VEC>
__global__ void __launch_bounds__(256, 2)
    sgemm_small_kernel(int M, int N, int K, float alpha, const float *__restrict__ A, int lda,
                       const float *__restrict__ B, int ldb, float beta, float *__restrict__ C,
                       int ldc, int kchunk, float *__restrict__ P, long long plane, int ldp,
                       int tiles_m) {
  constexpr bool KA = TA, KB = !TB;  // K contiguous in memory
  constexpr bool VA = VEC && !KA, VB = VEC && !KB;
  extern __shared__ __align__(16) float s4m[];
  const uint32_t smu = (uint32_t)__cvta_generic_to_shared(s4m);
  const int tid = threadIdx.x, lane = tid & 31, grp = tid >> 6, t64 = tid & 63;
  const int rm = (lane & 7) * 4, cn = (t64 >> 3) * 4;
  const int m0 = (int)(blockIdx.x % tiles_m) * S4_T, n0 = (int)(blockIdx.x / tiles_m) * S4_T;
  const int kbeg = blockIdx.z * kchunk, kend = min(K, kbeg + kchunk);
  const int KT = (kend - kbeg + S4_K - 1) / S4_K;
  unsigned long long acc[8][4];  // row 4 tx + i (+ 32 from i = 4), column pairs
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  const bool in_a = m0 + S4_T <= M, in_b = n0 + S4_T <= N;
  const float *pa = A + f32copy::run_offset<S4_T, KA, VA>(m0, kbeg, lda, tid);
  const float *pb = B + f32copy::run_offset<S4_T, KB, VB>(n0, kbeg, ldb, tid);
  const uint32_t da = f32copy::run_dst<S4_T, S4_LD, KA, VA>(tid);
  const uint32_t db = f32copy::run_dst<S4_T, S4_LD, KB, VB>(tid) + S4_PANEL * 4u;
  auto load_stage = [&](int st, int kt) {
    const int k0 = kbeg + kt * S4_K;
    const uint32_t d = smu + (uint32_t)(st * 2 * S4_PANEL) * 4u;
    const bool full = k0 + S4_K <= kend;
    if (full && in_a) f32copy::run_panel<S4_T, S4_LD, KA, VA>(d + da, pa, lda);
    else f32copy::load_panel<S4_T, S4_LD, KA, VA>(d, A, lda, m0, k0, M, kend, tid);
    if (full && in_b) f32copy::run_panel<S4_T, S4_LD, KB, VB>(d + db, pb, ldb);
    else f32copy::load_panel<S4_T, S4_LD, KB, VB>(d + S4_PANEL * 4u, B, ldb, n0, k0, N, kend, tid);
    pa += KA ? (size_t)S4_K : (size_t)S4_K * lda;
    pb += KB ? (size_t)S4_K : (size_t)S4_K * ldb;
  };
#pragma unroll
  for (int i = 0; i < S4_STAGES - 1; ++i) {
    if (i < KT) load_stage(i, i);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  int st = 0, fill = S4_STAGES - 1;
  for (int kt = 0; kt < KT; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(S4_STAGES - 2));
    __syncthreads();  // panel kt is in; every thread is done with the one refilled here
    if (kt + S4_STAGES - 1 < KT) load_stage(fill, kt + S4_STAGES - 1);
    asm volatile("cp.async.commit_group;\n" ::);
    const float *As = s4m + st * 2 * S4_PANEL + grp * S4_LD + rm;
    const float *Bs = s4m + st * 2 * S4_PANEL + S4_PANEL + grp * S4_LD + cn;
    st = st + 1 == S4_STAGES ? 0 : st + 1;
    fill = fill + 1 == S4_STAGES ? 0 : fill + 1;
#pragma unroll
    for (int kq = 0; kq < S4_K / 4; ++kq) {  // k = 4 kq + grp
      const bool sa = KA && kq >= 2, sb = KB && kq >= 2;  // panel_at's order
      unsigned long long bv[4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const ulonglong2 b2 = *reinterpret_cast<const ulonglong2 *>(&Bs[4 * kq * S4_LD + 32 * h]);
        bv[2 * h] = sb ? b2.y : b2.x;
        bv[2 * h + 1] = sb ? b2.x : b2.y;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 a4 = *reinterpret_cast<const float4 *>(&As[4 * kq * S4_LD + 32 * h]);
        const float av[4] = {sa ? a4.z : a4.x, sa ? a4.w : a4.y, sa ? a4.x : a4.z,
                             sa ? a4.y : a4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const unsigned long long ai = dup2(av[i]);
#pragma unroll
          for (int j = 0; j < 4; ++j) ffma2(acc[4 * h + i][j], ai, bv[j]);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();  // every thread is done with the last panel
  unsigned long long *xch = reinterpret_cast<unsigned long long *>(s4m);  // [3][8][256]
#pragma unroll
  for (int r = 1; r < 4; ++r) {
    const int q = (grp + r) & 3;  // the group that finishes pair q
#pragma unroll
    for (int i = 0; i < 8; ++i)
      xch[((r - 1) * 8 + i) * 256 + tid] = q == 0   ? acc[i][0]
                                           : q == 1 ? acc[i][1]
                                           : q == 2 ? acc[i][2]
                                                    : acc[i][3];
  }
  const int n = n0 + cn + (grp >> 1) * 32 + (grp & 1) * 2;
  float old[8][2];  // all of C's reads before its writes
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int m = m0 + rm + i + (i >> 2) * 28;
      old[i][j] = (P == nullptr && m < M && n + j < N) ? C[(size_t)(n + j) * ldc + m] : 0.f;
    }
  __syncthreads();
  const bool one = beta == 1.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const unsigned long long mine = grp == 0   ? acc[i][0]
                                    : grp == 1 ? acc[i][1]
                                    : grp == 2 ? acc[i][2]
                                               : acc[i][3];
    float2 v = *reinterpret_cast<const float2 *>(&mine);
#pragma unroll
    for (int r = 1; r < 4; ++r) {
      const unsigned long long o = xch[((r - 1) * 8 + i) * 256 + ((grp - r) & 3) * 64 + t64];
      const float2 w = *reinterpret_cast<const float2 *>(&o);
      v.x += w.x;
      v.y += w.y;
    }
    const int m = m0 + rm + i + (i >> 2) * 28;
    const float x[2] = {v.x, v.y};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if (m >= M || n + j >= N) continue;
      if (P != nullptr) P[blockIdx.z * plane + (size_t)(n + j) * ldp + m] = x[j];
      else
        C[(size_t)(n + j) * ldc + m] =
            one ? fmaf(alpha, x[j], old[i][j]) : fmaf(alpha, x[j], beta * old[i][j]);
    }
  }
}

template <bool TA, bool TB, bool VEC>
int launch_small(int m, int n, int k, float alpha, const float *A, int lda, const float *B,
                 int ldb, float beta, float *C, int ldc, int S, Ctx *cx, cudaStream_t s) {
  const int tm = (m + S4_T - 1) / S4_T, tn = (n + S4_T - 1) / S4_T;
  const int kblocks = (k + S4_K - 1) / S4_K, ldp = (m + 3) & ~3;
  const long long plane = (long long)n * ldp;
  int kchunk = (kblocks + S - 1) / S * S4_K;
  S = (k + kchunk - 1) / kchunk;
  float *P = S > 1 ? (float *)workspace(cx, WS_F32, (size_t)plane * S * sizeof(float)) : nullptr;
  if (P == nullptr) S = 1, kchunk = k;  // no scratch for the slices: one
  {
    B2_PROF("sgemm_simt", s);
    sgemm_small_kernel<TA, TB, VEC><<<dim3((unsigned)tm * (unsigned)tn, 1, S), 256, S4_SMEM, s>>>(
        m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, kchunk, P, plane, ldp, tm);
    B2_CUDA_TRY(cudaGetLastError());
  }
  if (S == 1) return B2_OK;
  return sgemm_splitk_reduce(P, plane, ldp, S, m, n, alpha, beta, C, ldc, s);
}

// K slices of the small-tile kernel for a product whose 128 x 128 tiles leave
// slots empty, or 0 where those (in S slices) are modelled faster.  Both models:
// K panels of 16 in a row times a panel's time at q work units per SM, the ends,
// and for slices a second launch (1.5 us on the device, 2 on the host) and the
// partials at 8 TB/s.  128 x 128: 1.47 us a panel alone on an SM, 1.37 a unit
// from two on (4-byte copies 12 % more); 64 x 64: 0.46 and 0.43 (20 %).  B200, us,
// 128 x 128 / 64 x 64: 128^3 15.3 / 7.0, 256^3 27.0 / 8.0, 512^3 47.3 / 13.4, 700^3
// 74.3 / 27.8, 384x240x848 90.8 / 12.4, 128x128x8192 115 / 24.9; 1024^3 54.3 / 60.7,
// 1500^3 145 / 173, 2048x1024x512 50.7 / 62.3.
int small_slices(int m, int n, int kblocks, long long tiles, int S, bool vec, int sms,
                 bool slices) {
  const auto ends = [](int s, long long units, double bytes) {
    return s > 1 ? 3.5 + (double)units * bytes / 8e6 : 0.0;
  };
  const long long ub = tiles * S, qb = (ub + sms - 1) / sms;
  double best = 3.5 + (kblocks + S - 1) / S * (qb == 1 ? 1.47 : 1.37 * qb) * (vec ? 1.0 : 1.12) +
                ends(S, ub, 131072.0);
  int pick = 0;
  const long long t64 = (long long)((m + S4_T - 1) / S4_T) * ((n + S4_T - 1) / S4_T);
  for (const int s : {1, 2, 3, 4, 6, 8, 16}) {
    if (s > 1 && (!slices || kblocks < 4 * s)) break;
    const long long u = t64 * s, q = (u + sms - 1) / sms;
    const double us = 4.4 + (kblocks + s - 1) / s * (q == 1 ? 0.46 : 0.43 * q) * (vec ? 1.0 : 1.2) +
                      ends(s, u, 32768.0);
    if (us < best) best = us, pick = s;
  }
  return pick;
}

template <bool TA, bool TB, bool VEC>
int launch_ffma2(int m, int n, int k, float alpha, const float *A, int lda, const float *B,
                 int ldb, float beta, float *C, int ldc, cudaStream_t s) {
  auto kern = sgemm_ffma2_kernel<TA, TB, VEC, 0>;
  auto kern_split = sgemm_ffma2_kernel<TA, TB, VEC, 1>;
  Ctx *cx = ctx();
  if (!cx) return B2_ERR_NO_DEVICE;
  const int gx = (m + S2_M - 1) / S2_M, gy = (n + S2_N - 1) / S2_N;
  const long long tiles = (long long)gx * gy, slots = 2ll * cx->sm_count;
  if (tiles > 0x7fffffffll) return B2_ERR_ARG;
  const int kblocks = (k + S2_K - 1) / S2_K;
  const int S = ffma2_ksplit(tiles, kblocks, cx->sm_count);
  // Slices of the 64 x 64 form and of the last wave are for calls that run now: a
  // captured one would hold scratch that a larger call may replace.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) (void)cudaGetLastError();
  const bool capturing = cap != cudaStreamCaptureStatusNone;
  if (tiles < slots) {
    const int Ss = small_slices(m, n, kblocks, tiles, S, VEC, cx->sm_count, !capturing);
    if (Ss > 0)
      return launch_small<TA, TB, VEC>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, Ss, cx, s);
  }
  if (S == 1) {
    // The tiles of whole waves run in full; the rest, when it would leave half
    // or more of the CTA slots empty, is cut into K slices that fill them, as a
    // launch of its own (a programmatic dependent: it starts while the last
    // whole wave ends).  4096^3: 1024 tiles are 3 waves of 296 and 136 tiles,
    // 2388 -> 2360 us with the rest in 2 slices (B200).
    // From 12 waves on the last one runs in full: there is little left to win (0.5 to
    // 2 %: 7680 x 7680 x 1024, 12.2 waves, 2134 against 2089 us).
    const int rest = (int)(tiles % slots);
    int St = rest > 0 ? (int)(slots / rest) : 1;
    if (St > 8) St = 8;
    while (St > 1 && kblocks / St < 16) --St;
    bool tail = !capturing && tiles > slots && tiles < 12 * slots && St >= 2;
    float *P = nullptr;
    int kchunk = k;
    if (tail) {
      kchunk = (kblocks + St - 1) / St * S2_K;
      St = (k + kchunk - 1) / kchunk;
      P = (float *)workspace(cx, WS_F32, (size_t)St * rest * S2_M * S2_N * sizeof(float));
      if (!P) tail = false;  // no scratch: the last wave in full
    }
    const int whole = (int)(tail ? tiles - rest : tiles);
    B2_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S2_SMEM));
    {
      B2_PROF("sgemm_simt", s);
      kern<<<whole, 256, S2_SMEM, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, k, nullptr, 0,
                                       0, gx, 0, tail ? 1 : 0);
      B2_CUDA_TRY(cudaGetLastError());
    }
    if (!tail) return B2_OK;
    auto kern_tail = sgemm_ffma2_kernel<TA, TB, VEC, 2>;
    B2_CUDA_TRY(
        cudaFuncSetAttribute(kern_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, S2_SMEM));
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)rest, 1, (unsigned)St);
    lc.blockDim = dim3(256);
    lc.dynamicSmemBytes = S2_SMEM;
    lc.stream = s;
    lc.attrs = attr;
    lc.numAttrs = 1;
    {
      B2_PROF("sgemm_simt", s);
      B2_CUDA_TRY(cudaLaunchKernelEx(&lc, kern_tail, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc,
                                     kchunk, P, 0ll, 0, gx, whole, 0));
    }
    lc.gridDim = dim3((unsigned)rest * 16);
    lc.dynamicSmemBytes = 0;
    B2_PROF("sgemm_splitk_reduce", s);
    B2_CUDA_TRY(cudaLaunchKernelEx(&lc, ffma2_tail_reduce_kernel, (const float *)P, rest, St, m, n,
                                   alpha, beta, C, ldc, gx, whole));
    return B2_OK;
  }
  // Split-K: S raw partial products of K ranges (multiples of S2_K), then one
  // reduction adding them in K order (FP64 sums, rounded once) into C.
  const int kchunk = (kblocks + S - 1) / S * S2_K;
  const int S_used = (k + kchunk - 1) / kchunk;
  const int ldp = (m + 3) & ~3;
  const long long plane = (long long)n * ldp;
  float *P = (float *)workspace(cx, WS_MISC, (size_t)plane * S_used * sizeof(float));
  if (!P) return B2_ERR_NOMEM;
  {
    B2_CUDA_TRY(
        cudaFuncSetAttribute(kern_split, cudaFuncAttributeMaxDynamicSharedMemorySize, S2_SMEM));
    B2_PROF("sgemm_simt", s);
    kern_split<<<dim3((unsigned)tiles, 1, S_used), 256, S2_SMEM, s>>>(
        m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, kchunk, P, plane, ldp, gx, 0, 0);
    B2_CUDA_TRY(cudaGetLastError());
  }
  return sgemm_splitk_reduce(P, plane, ldp, S_used, m, n, alpha, beta, C, ldc, s);
}

}  // namespace

int sgemm_simt(char ta, char tb, int m, int n, int k, float alpha, const float *A, int lda,
               const float *B, int ldb, float beta, float *C, int ldc, cudaStream_t s) {
  if (m <= 0 || n <= 0) return B2_OK;
  if (k <= 0 || alpha == 0.f) return beta == 1.f ? B2_OK : scale_matrix_s(m, n, beta, C, ldc, s);
  const bool TA = !(ta == 'N' || ta == 'n');
  const bool TB = !(tb == 'N' || tb == 'n');
  // 16-byte loads need 16-byte aligned bases and leading dimensions of 4k floats
  const bool vec = (lda % 4 == 0) && (ldb % 4 == 0) && (((uintptr_t)A & 15) == 0) &&
                   (((uintptr_t)B & 15) == 0);
  if (vec) {
    if (TA && TB) return launch_ffma2<true, true, true>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
    if (TA) return launch_ffma2<true, false, true>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
    if (TB) return launch_ffma2<false, true, true>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
    return launch_ffma2<false, false, true>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
  }
  if (TA && TB) return launch_ffma2<true, true, false>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
  if (TA) return launch_ffma2<true, false, false>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
  if (TB) return launch_ffma2<false, true, false>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
  return launch_ffma2<false, false, false>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
}

int sgemm_dispatch(char ta, char tb, int m, int n, int k, float alpha, const float *A, int lda,
                   const float *B, int ldb, float beta, float *C, int ldc, int method,
                   cudaStream_t s) {
  switch (method) {
    case B2_METHOD_FP32:
    case B2_METHOD_DEFAULT:
      return sgemm_simt(ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
    case B2_METHOD_TF32:
    case B2_METHOD_TF32X3:
    case B2_METHOD_BF16X3:
      return sgemm_tensor(ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, method, s);
    default:
      return B2_ERR_UNSUPPORTED;
  }
}

}  // namespace b2
