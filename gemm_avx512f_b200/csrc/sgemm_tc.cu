// sgemm_tc.cu -- SGEMM on the tcgen05 tensor cores with FP32 accumulation.
//
// Replaces the reference's AVX-512 SGEMM (src/gemm_driver.c:116 built without
// -DDOUBLE, OpenBLAS-like_implementation/sgemm.c:366-412) by three tensor-core
// forms, all with FP32 accumulators in TMEM:
//   TF32    1 product:  C = tf32(A) tf32(B)                     (kind::tf32)
//   TF32X3  3 products: A = Ab + As, B = Bb + Bs (each TF32),
//                       C = Ab Bb + Ab Bs + As Bb                (kind::tf32)
//   BF16X3  3 products: A = Ah + Al, B = Bh + Bl (each BF16),
//                       C = Ah Bh + Ah Bl + Al Bh                (kind::f16, bf16 in)
// Every method is ONE GEMM on the engine in umma.cuh; the split/convert kernel
// is the only extra pass.  For three terms each operand stores two segments,
// [big | small], each padded with zeros to a 128-byte K block, and a stage of
// the engine holds both segments of a K block of A and B: its MMAs add
// Ab Bb + Ab Bs + As Bb, so every segment is loaded once.
#include <cuda_bf16.h>

#include <type_traits>

#include "b2_methods.cuh"
#include "b2_profile.cuh"
#include "umma.cuh"

namespace b2 {
namespace {

__device__ __forceinline__ float tf32_round(float x) {  // round to nearest, ties away
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// One operand of a split pass: R rows of K elements, element (r, k) at
// X[r + k*ld] (rowcont) or X[r*ld + k]; vec: 16-byte loads are legal (X 16-byte
// aligned, ld a multiple of 4).
struct SplitOp {
  const float *X;
  long long ld;
  int R, rowcont, vec;
  void *out;
};

// Writes every row of both operands as [big | small] (segs = 2) or [big]
// segments of kp elements of type T, zero beyond K: out[r][segs*kp].  One
// block turns 64 rows x 64 k around in shared memory; blocks that follow each
// other read neighbouring memory.
// Bound: HBM, 4 bytes read and segs*sizeof(T) written per element: 8192x8192
// to two bfloat16 segments in 83 us, 6.4 TB/s (32x64 blocks with two loads in
// flight per thread, k blocks first: 125 us).
template <typename T>
__global__ void __launch_bounds__(256)
    split_kernel(const SplitOp a, const SplitOp b, unsigned blocks_a, int K, int kp, int segs) {
  __shared__ float tile[64][65];
  umma::grid_dependency_wait();
  const bool second = blockIdx.x >= blocks_a;
  const float *X = second ? b.X : a.X;
  const long long ld = second ? b.ld : a.ld;
  const int R = second ? b.R : a.R;
  const bool rowcont = second ? b.rowcont : a.rowcont, vec = second ? b.vec : a.vec;
  T *out = (T *)(second ? b.out : a.out);
  const unsigned id = second ? blockIdx.x - blocks_a : blockIdx.x;
  const unsigned kt = (unsigned)(kp + 63) / 64, rt = (unsigned)(R + 63) / 64;
  const int r0 = (int)(rowcont ? id % rt : id / kt) * 64;
  const int k0 = (int)(rowcont ? id / rt : id % kt) * 64;
  const int tid = threadIdx.x;
  if (vec) {
    float v[4][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int idx = tid + 256 * e;
      const int hi = idx >> 4, lo = (idx & 15) * 4;  // lo along the contiguous dimension
      const int rr = rowcont ? lo : hi, kk = rowcont ? hi : lo;
      const int r = r0 + rr, k = k0 + kk;
      const int left = rowcont ? (k < K ? R - r : 0) : (r < R ? K - k : 0);
      const float *src = X + (rowcont ? r + k * ld : r * ld + k);
      if (left >= 4) {
        const float4 q = __ldg(reinterpret_cast<const float4 *>(src));
        v[e][0] = q.x, v[e][1] = q.y, v[e][2] = q.z, v[e][3] = q.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[e][j] = j < left ? __ldg(src + j) : 0.f;
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int idx = tid + 256 * e;
      const int hi = idx >> 4, lo = (idx & 15) * 4;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (rowcont) tile[lo + j][hi] = v[e][j];
        else tile[hi][lo + j] = v[e][j];
      }
    }
  } else {
    float v[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const int idx = tid + 256 * e, hi = idx >> 6, lo = idx & 63;
      const int r = r0 + (rowcont ? lo : hi), k = k0 + (rowcont ? hi : lo);
      v[e] = (r < R && k < K) ? __ldg(X + (rowcont ? r + k * ld : r * ld + k)) : 0.f;
    }
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const int idx = tid + 256 * e, hi = idx >> 6, lo = idx & 63;
      if (rowcont) tile[lo][hi] = v[e];
      else tile[hi][lo] = v[e];
    }
  }
  __syncthreads();
  // 16-byte stores: 4 floats or 8 bfloat16 of one row; kp is a multiple of 32
  // (float) or 64 (bfloat16) elements, and the tile is zero beyond K.
  constexpr int GW = 16 / (int)sizeof(T), GPR = 64 / GW;
#pragma unroll
  for (int e = 0; e < 64 * GPR / 256; ++e) {
    const int idx = tid + 256 * e, rr = idx / GPR, kl = (idx % GPR) * GW;
    const int r = r0 + rr;
    if (r >= R || k0 + kl >= kp) continue;
    T *dst = out + (long long)r * segs * kp + k0 + kl;
    if constexpr (sizeof(T) == 4) {
      float big[4], small[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float x = tile[rr][kl + j];
        big[j] = tf32_round(x);
        small[j] = tf32_round(x - big[j]);
      }
      *reinterpret_cast<float4 *>(dst) = make_float4(big[0], big[1], big[2], big[3]);
      if (segs == 2)
        *reinterpret_cast<float4 *>(dst + kp) = make_float4(small[0], small[1], small[2], small[3]);
    } else {
      uint32_t hw[4], lw[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t h2 = 0, l2 = 0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float x = tile[rr][kl + 2 * j + i];
          const __nv_bfloat16 h = __float2bfloat16_rn(x);
          const __nv_bfloat16 l = __float2bfloat16_rn(x - __bfloat162float(h));
          h2 |= (uint32_t)__bfloat16_as_ushort(h) << (16 * i);
          l2 |= (uint32_t)__bfloat16_as_ushort(l) << (16 * i);
        }
        hw[j] = h2;
        lw[j] = l2;
      }
      *reinterpret_cast<uint4 *>(dst) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
      if (segs == 2)
        *reinterpret_cast<uint4 *>(dst + kp) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
    }
  }
}

// FP32 epilogue: lane p = row m of C, v[j] = column q0 + j: a warp reads and
// writes 32 consecutive rows of a column, all of C's reads before its writes.
struct F32Epi {
  float *C;
  int ldc;
  int M, N;
  float alpha, beta;
  static constexpr bool PARTIAL = false;
  __device__ __forceinline__ bool wide() const { return false; }
  // Brings the warp's 32 rows x NC columns of C (rows from p0) into L2 while
  // the product is formed: one line per lane and column.
  template <int NC>
  __device__ __forceinline__ void prefetch(int p0, int lane, int q0) const {
#pragma unroll
    for (int i = 0; i < NC / 32; ++i) {
      const int q = q0 + 32 * i + lane;
      if (p0 < M && q < N) umma::prefetch_l2(C + (long long)q * ldc + p0);
    }
  }
  __device__ __forceinline__ void operator()(int, int p, int q0, const float (&v)[16]) const {
    if (p >= M || q0 >= N) return;
    // (the volatile asms keep the compiler from holding the addresses of many
    // columns at once beside the 128 sums, which spills)
    long long ld = ldc;
    asm volatile("" : "+l"(ld));
    float *c = C + q0 * ld + p;
    const int nq = min(16, N - q0);
    float old[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      old[j] = j < nq ? *c : 0.f;
      c += ld;
    }
    asm volatile("" : "+l"(ld));
    c -= 16 * ld;
    const bool one = (beta == 1.f);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      if (j < nq) *c = one ? fmaf(alpha, v[j], old[j]) : fmaf(alpha, v[j], beta * old[j]);
      c += ld;
    }
  }
};

// Split-K epilogue: the partial of unit ks (the engine's batch index) to
// W[ks][n][ldw]: one accumulator, FP32, or (pairs) the sum of several with its rounding
// error, both at 1/16; sgemm_splitk_reduce_kernel adds the units in a fixed order.
struct PartialEpi {
  void *W;
  long long plane;
  int ldw;
  int M, N;
  bool pairs;
  static constexpr bool PARTIAL = true;
  __device__ __forceinline__ bool wide() const { return pairs; }
  template <int NC>
  __device__ __forceinline__ void prefetch(int, int, int) const {}
  template <typename T>  // float or float2
  __device__ __forceinline__ void operator()(int ks, int p, int q0, const T (&v)[16]) const {
    if (p >= M || q0 >= N) return;
    T *w = (T *)W + ks * plane + (long long)q0 * ldw + p;
    const int nq = min(16, N - q0);
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (j < nq) w[(long long)j * ldw] = v[j];
  }
};

// One partial in FP64 (an infinity's error is a NaN: it is itself).
__device__ __forceinline__ double partial(float x) { return (double)x; }
__device__ __forceinline__ double partial(float2 x) {
  const double s = (double)x.x, r = s + (double)x.y;
  return 16.0 * (r == r ? r : s);
}
__device__ __forceinline__ void add4(double (&acc)[4], const float *w) {
  const float4 x = *reinterpret_cast<const float4 *>(w);
  acc[0] += (double)x.x, acc[1] += (double)x.y, acc[2] += (double)x.z, acc[3] += (double)x.w;
}
__device__ __forceinline__ void add4(double (&acc)[4], const float2 *w) {
  const float4 x = *reinterpret_cast<const float4 *>(w);
  const float4 y = *reinterpret_cast<const float4 *>(w + 2);
  acc[0] += partial(make_float2(x.x, x.y)), acc[1] += partial(make_float2(x.z, x.w));
  acc[2] += partial(make_float2(y.x, y.y)), acc[3] += partial(make_float2(y.z, y.w));
}

// C(m, n) = alpha * sum_ks W[ks][n][m] + beta C (beta != 1 multiplies), the
// partials summed in FP64 in K order and rounded once.
// Four rows per thread; launched as a programmatic dependent of the GEMM, whose
// writes it waits for.  W is 16-byte aligned and ldw a multiple of 4.
template <typename T>
__global__ void __launch_bounds__(256)
    sgemm_splitk_reduce_kernel(const T *__restrict__ W, long long plane, int ldw, int S, int M,
                               int N, float alpha, float beta, float *__restrict__ C, int ldc) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const unsigned quads = (unsigned)(M + 3) / 4;
  const unsigned long long total = (unsigned long long)quads * (unsigned)N;
  const bool cvec = (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (ldc & 3) == 0;
  for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < total;
       i += gridDim.x * 256ull) {
    const int n = (int)(i / quads), m = (int)(i - (unsigned long long)n * quads) * 4;
    float *c = C + (long long)n * ldc + m;
    const T *w = W + (long long)n * ldw + m;
    const int left = M - m;
    float old[4];
    if (cvec && left >= 4) {
      const float4 q = *reinterpret_cast<const float4 *>(c);
      old[0] = q.x, old[1] = q.y, old[2] = q.z, old[3] = q.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) old[e] = e < left ? c[e] : 0.f;
    }
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
    for (int ks = 0; ks < S; ++ks) add4(acc, w + ks * plane);
    float r[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float a = (float)acc[e];
      r[e] = (beta == 1.f) ? fmaf(alpha, a, old[e]) : fmaf(alpha, a, beta * old[e]);
    }
    if (cvec && left >= 4) {
      *reinterpret_cast<float4 *>(c) = make_float4(r[0], r[1], r[2], r[3]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < left) c[e] = r[e];
    }
  }
}

// K ranges for a product of `tiles` output tiles and `kblocks` K blocks: 1
// when the tiles already fill the SMs, else the count (at most 16, >= 8 K
// blocks per range) that best fills whole waves of `sms` CTAs.
int choose_ksplit(long long tiles, int kblocks, int sms) {
  if (tiles >= sms) return 1;
  int best = 1;
  double best_eff = (double)tiles / sms;
  for (int S = 2; S <= 16 && S * 8 <= kblocks; ++S) {
    const long long units = tiles * S;
    const long long waves = (units + sms - 1) / sms;
    const double eff = (double)units / (double)(waves * sms);
    if (eff > best_eff + 0.02) {
      best_eff = eff;
      best = S;
    }
  }
  return best;
}

inline long long round_up(long long x, long long a) { return (x + a - 1) / a * a; }

// Tile of an engine (rows m x columns n), CTAs or pairs that run at once, and time of
// a term block (us: measured; with one term a 128 x 128 tile waits for its copies).
struct Engine {
  int tile_p, tile_q, slots;
  double t_tb;
};
Engine engine(int eng, int terms, int sms) {  // of SgCfg
  switch (eng) {
    case 1: return Engine{umma::BM, 128, sms, terms == 1 ? 0.31 : 0.21};
    case 2: return Engine{256, 256, sms / 2, 0.28};
    default: return Engine{umma::BM, 256, sms, 0.28};
  }
}

// How a product is run: engine, partials per tile, term blocks per unit and per
// accumulated range; pairs: the partials are sums with their errors.
struct Ranges {
  int eng, E, unit_tb, range_tb;
  bool pairs;
  size_t bytes() const { return pairs ? sizeof(float2) : sizeof(float); }  // of a partial
};

// K is accumulated in S ranges of tbs term blocks (a K block of a three-term product is
// three: its MMAs add Ab Bb, Ab Bs and As Bb in turn): `split` of them (0: chosen for
// the engine's tiles).  Ranges are as short as separate launches per range would have
// them: the tensor core's accumulation error grows with a chain's length (ranges of
// whole K blocks, 3xTF32 with K = 64: 3.8e-7 instead of 1.1e-7).  Either each range is
// a unit of its own, on engine `eng`, and S partials per tile go through memory; or a
// unit takes `per` consecutive ranges of its tile and adds them in its epilogue, on
// engine 1: 64 sums and their rounding errors are what a thread has registers for.
// (128 of them, for tiles of 256 columns, spill, and the spills leave for L2: 12 us a
// launch.  A pair's tile of 256 x 128 takes 0.23 us a term block, limited by its
// copies, against 0.21 for half of it on engine 1.)
// Modelled time (us): waves of units, each t_tb per term block but at least 1 us a
// range, which is what adding an accumulator to the sums takes; fill, drain and the
// gaps between waves; partials written and read, in L2 below 64 MB, and a second
// launch.  nprod: products of that shape in one launch.  Measured (B200, us, whole
// calls, partials of each range / the best sums): 3xTF32 512^3 11.9 / 12.9, 1024^3
// 26.7 / 24.5 (4 ranges a unit), 2048^3 117 / 100, 8192x256x8192 272 / 291; 3xBF16
// 2048^3 89.6 / 61.4; cgemm3m 2048^3 381 / 300, 1900x1300x2100 201 / 205.
Ranges choose_ranges(int eng, int split, int terms, int kblocks, int m, int n, int nprod,
                     int sms) {
  const int tblocks = terms * kblocks;
  auto tiles = [&](const Engine &g) {
    return ((m + g.tile_p - 1) / g.tile_p) * (long long)((n + g.tile_q - 1) / g.tile_q);
  };
  const Engine base = engine(eng, terms, sms), adder = engine(1, terms, sms);
  int S = split > 0 ? split : choose_ksplit(tiles(base), tblocks, base.slots);
  if (S > tblocks) S = tblocks > 0 ? tblocks : 1;
  const int tbs = (tblocks + S - 1) / S;
  S = (tblocks + tbs - 1) / tbs;
  Ranges best{};
  double best_us = 1e300;
  for (int per = 1; per <= S; ++per) {
    const int E = (S + per - 1) / per;
    if (per > 1 && (S + per - 2) / (per - 1) == E) continue;  // more even with per - 1
    const bool pairs = E > 1 && per > 1;
    if (pairs && 2 * E > S) continue;  // no more scratch than one FP32 partial per range
    const Engine &g = per > 1 ? adder : base;
    const long long waves = (nprod * tiles(g) * E + g.slots - 1) / g.slots;
    const int tb = per * tbs < tblocks ? per * tbs : tblocks;
    const double work = tb * g.t_tb, drains = 1.0 * ((tb + tbs - 1) / tbs);
    double us = (double)waves * (work > drains ? work : drains) + 4.0 + 0.7 * (double)(waves - 1);
    if (E > 1) {
      const double bytes = (double)E * m * n * nprod * (pairs ? 16.0 : 8.0);
      us += 2.0 + bytes / (bytes < 64e6 ? 12e6 : 6e6);
    }
    if (us < best_us) best_us = us, best = Ranges{per > 1 ? 1 : eng, E, per * tbs, tbs, pairs};
  }
  return best;
}

// One SGEMM product (or nbatch of them).
template <class Epi>
int run_engine(bool bf16, int terms, const CUtensorMap &tmX, const CUtensorMap &tmY, int m,
               int n, int kp, int nbatch, int seg_kb, const Ranges &rg, const Epi &epi, Ctx *cx,
               cudaStream_t s) {
  const char *nm = bf16 ? "sgemm_umma_bf16" : "sgemm_umma_tf32";
  // TERMS = 3 stages hold four operand tiles: 64 KB (pair and 128x128), 96 KB
  auto pair = [&](auto kd, auto t3) {
    constexpr int T = decltype(t3)::value;
    return umma::launch_pair<decltype(kd)::value, 256, T == 3 ? 3 : 6, Epi, true, T>(
        tmX, tmY, m, n, kp, nbatch, epi, cx->device, cx->derr, s, nm, nullptr, rg.E, seg_kb,
        rg.unit_tb, rg.range_tb);
  };
  auto single = [&](auto kd, auto bn, auto t3) {
    constexpr int T = decltype(t3)::value, BN = decltype(bn)::value;
    constexpr int ST = BN == 256 ? (T == 3 ? 2 : 4) : (T == 3 ? 3 : 6);
    return umma::launch<decltype(kd)::value, BN, ST, Epi, 1, true, T>(
        tmX, tmY, m, n, kp, nbatch, epi, cx->sm_count, cx->derr, s, nm, 0, nullptr, rg.E, seg_kb, 0,
        0, rg.unit_tb, rg.range_tb);
  };
  using BF = std::integral_constant<int, umma::KIND_BF16>;
  using TF = std::integral_constant<int, umma::KIND_TF32>;
  using I1 = std::integral_constant<int, 1>;
  using I3 = std::integral_constant<int, 3>;
  using I128 = std::integral_constant<int, 128>;
  using I256 = std::integral_constant<int, 256>;
  if (rg.eng == 2)
    return bf16 ? pair(BF{}, I3{}) : terms == 3 ? pair(TF{}, I3{}) : pair(TF{}, I1{});
  if (rg.eng == 1)
    return bf16         ? single(BF{}, I128{}, I3{})
           : terms == 3 ? single(TF{}, I128{}, I3{})
                        : single(TF{}, I128{}, I1{});
  return bf16         ? single(BF{}, I256{}, I3{})
         : terms == 3 ? single(TF{}, I256{}, I3{})
                      : single(TF{}, I256{}, I1{});
}

// Rows of Y in one TMA box: a CTA's.
int y_box(int eng) { return eng == 0 ? 256 : 128; }

// Launch as a programmatic dependent of the kernel before it in the stream
// (the kernel waits for that one's writes with griddepcontrol.wait).
template <typename... KArgs, typename... Args>
cudaError_t launch_dependent(void (*kern)(KArgs...), unsigned blocks, int threads, cudaStream_t s,
                             Args... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(blocks);
  lc.blockDim = dim3((unsigned)threads);
  lc.stream = s;
  lc.attrs = attr;
  lc.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&lc, kern, args...);
  return e != cudaSuccess ? e : cudaGetLastError();
}

template <typename T>
int splitk_reduce(const T *W, long long plane, int ldw, int S, int m, int n, float alpha,
                  float beta, float *C, int ldc, cudaStream_t s) {
  const long long blocks = ((long long)((m + 3) / 4) * n + 255) / 256;
  B2_PROF("sgemm_splitk_reduce", s);
  // 8 blocks on each of 148 SMs
  B2_CUDA_TRY(launch_dependent(sgemm_splitk_reduce_kernel<T>,
                               (unsigned)(blocks < 1184 ? blocks : 1184), 256, s, W, plane, ldw, S,
                               m, n, alpha, beta, C, ldc));
  return B2_OK;
}

SplitOp split_op(const float *X, long long sr, long long sk, int R, void *out) {
  SplitOp o;
  o.X = X;
  o.rowcont = sr == 1;
  o.ld = o.rowcont ? sk : sr;
  o.R = R;
  o.vec = ((uintptr_t)X & 15) == 0 && o.ld % 4 == 0;
  o.out = out;
  return o;
}

// Split pass over one or two operands (b.R = 0: one).
template <typename T>
int run_split(const SplitOp &a, const SplitOp &b, int K, int kp, int segs, cudaStream_t s) {
  const unsigned kt = (unsigned)(kp + 63) / 64;
  const unsigned ba = kt * ((unsigned)(a.R + 63) / 64), bb = kt * ((unsigned)(b.R + 63) / 64);
  B2_PROF("sgemm_split", s);
  B2_CUDA_TRY(launch_dependent(split_kernel<T>, ba + bb, 256, s, a, b, ba, K, kp, segs));
  return B2_OK;
}

// ------------------------------------------------- complex64 3M products --
// One complex operand of a 3M product: R rows of K complex elements, element
// (r, k) at complex index r + k*ld (rowcont) or r*ld + k; sgn = -1 conjugates.
struct Split3Op {
  const float *X;
  long long ld;
  int R, rowcont, pairs;  // pairs: 8-byte loads are legal
  float sgn;
  float *out;
};

// Writes the real part, the imaginary part and their sum of every row of both
// operands as [big | small] TF32 segments: out[t][r][2*kp], t = 0, 1, 2 (the
// operands of P1, P2, P3), or only part t = `only` (>= 0), to out[0].  One block
// turns 64 rows x 32 k around.
// Bound: HBM, 8 bytes read and 24 written per element.  The pre-adds and the
// splits were passes of their own (20 + 36 bytes per element): 110 -> 31 us at
// 1900x1300x2100 on B200, the whole product 367 -> 199.
__global__ void __launch_bounds__(256)
    split3m_kernel(const Split3Op a, const Split3Op b, unsigned blocks_a, int K, int kp, int only) {
  __shared__ float tr[64][33], ti[64][33];
  umma::grid_dependency_wait();
  const bool second = blockIdx.x >= blocks_a;
  const float *X = second ? b.X : a.X;
  const long long ld = second ? b.ld : a.ld;
  const int R = second ? b.R : a.R;
  const bool rowcont = second ? b.rowcont : a.rowcont, pairs = second ? b.pairs : a.pairs;
  const float sgn = second ? b.sgn : a.sgn;
  float *out = second ? b.out : a.out;
  const unsigned id = second ? blockIdx.x - blocks_a : blockIdx.x;
  const unsigned kt = (unsigned)kp / 32, rt = (unsigned)(R + 63) / 64;
  const int r0 = (int)(rowcont ? id % rt : id / kt) * 64;
  const int k0 = (int)(rowcont ? id / rt : id % kt) * 32;
  const int tid = threadIdx.x;
  float2 v[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int idx = tid + 256 * e;
    const int rr = rowcont ? idx & 63 : idx >> 5, kk = rowcont ? idx >> 6 : idx & 31;
    const int r = r0 + rr, k = k0 + kk;
    v[e] = make_float2(0.f, 0.f);
    if (r < R && k < K) {
      const float *p = X + 2 * (rowcont ? r + k * ld : r * ld + k);
      if (pairs) v[e] = __ldg(reinterpret_cast<const float2 *>(p));
      else v[e] = make_float2(__ldg(p), __ldg(p + 1));
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int idx = tid + 256 * e;
    const int rr = rowcont ? idx & 63 : idx >> 5, kk = rowcont ? idx >> 6 : idx & 31;
    tr[rr][kk] = v[e].x;
    ti[rr][kk] = sgn * v[e].y;
  }
  __syncthreads();
  const long long plane = (long long)R * 2 * kp;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int idx = tid + 256 * e, rr = idx >> 3, kl = (idx & 7) * 4;
    const int r = r0 + rr;
    if (r >= R) continue;
    float *dst = out + (long long)r * 2 * kp + k0 + kl;
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      if (only >= 0 && t != only) continue;
      float *to = dst + (only >= 0 ? 0 : t) * plane;
      float big[4], small[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float re = tr[rr][kl + j], im = ti[rr][kl + j];
        const float x = t == 0 ? re : t == 1 ? im : re + im;
        big[j] = tf32_round(x);
        small[j] = tf32_round(x - big[j]);
      }
      *reinterpret_cast<float4 *>(to) = make_float4(big[0], big[1], big[2], big[3]);
      *reinterpret_cast<float4 *>(to + kp) = make_float4(small[0], small[1], small[2], small[3]);
    }
  }
}

// C = alpha (P1 - P2 + i (P3 - P1 - P2)) + beta C from the E partials of each
// product (plane t*E + e of W), summed in FP64 and rounded once.
template <typename T>
__global__ void __launch_bounds__(256)
    combine3m_tc_kernel(const T *__restrict__ W, long long plane, int ldw, int E, int M, int N,
                        float ar, float ai, float br, float bi, float *__restrict__ C, int ldc) {
  umma::grid_dependency_wait();
  const bool beta_one = br == 1.f && bi == 0.f;
  const unsigned long long total = (unsigned long long)(unsigned)M * (unsigned)N;
  for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < total;
       i += gridDim.x * 256ull) {
    const int n = (int)(i / (unsigned)M), m = (int)(i - (unsigned long long)n * (unsigned)M);
    const T *w = W + (long long)n * ldw + m;
    float *c = C + 2 * ((long long)n * ldc + m);
    float cr = c[0], ci = c[1], p[3];
    if (E == 1) {
#pragma unroll
      for (int t = 0; t < 3; ++t) p[t] = (float)partial(w[t * plane]);
    } else {
      double acc[3] = {0.0, 0.0, 0.0};
      for (int e = 0; e < E; ++e)
#pragma unroll
        for (int t = 0; t < 3; ++t) acc[t] += partial(w[(t * E + e) * plane]);
#pragma unroll
      for (int t = 0; t < 3; ++t) p[t] = (float)acc[t];
    }
    const float re = p[0] - p[1], im = p[2] - p[0] - p[1];
    if (!beta_one) {
      const float tr = br * cr - bi * ci, ti = br * ci + bi * cr;
      cr = tr;
      ci = ti;
    }
    c[0] = cr + (ar * re - ai * im);
    c[1] = ci + (ar * im + ai * re);
  }
}

Split3Op split3_op(const float *X, int ld, bool rowcont, bool conj, int R, float *out) {
  return Split3Op{X, ld, R, rowcont ? 1 : 0, ((uintptr_t)X & 7) == 0 ? 1 : 0, conj ? -1.f : 1.f,
                  out};
}

}  // namespace

// cgemm3m on the tensor cores in three launches: one pass writes the three
// products' split operands, one GEMM launch runs P1, P2 and P3 (3xTF32) as a
// batch, one pass combines them into C.
int cgemm3m_tensor(char ta, char tb, int m, int n, int k, float ar, float ai, float br, float bi,
                   const float *A, int lda, const float *B, int ldb, float *C, int ldc,
                   cudaStream_t s) {
  Ctx *cx = ctx();
  if (!cx) return B2_ERR_NO_DEVICE;
  const bool tA = !(ta == 'N' || ta == 'n' || ta == 'R' || ta == 'r');
  const bool tB = !(tb == 'N' || tb == 'n' || tb == 'R' || tb == 'r');
  const bool cA = ta == 'C' || ta == 'c' || ta == 'R' || ta == 'r';
  const bool cB = tb == 'C' || tb == 'c' || tb == 'R' || tb == 'r';
  const int kp = (int)round_up(k, 32);
  const long long ks = 2LL * kp;
  // engine and K ranges as for one 3xTF32 SGEMM of this shape
  const SgCfg cfg = sgemm_pick_cfg('N', 'N', m, n, k, 1, B2_METHOD_TF32X3);
  const int seg_kb = kp * 4 / umma::KBLOCK_BYTES;
  Ranges rg = choose_ranges((cfg.engine >= 0 && cfg.engine <= 2) ? cfg.engine : 0, cfg.split, 3,
                            seg_kb, m, n, 3, cx->sm_count);
  const int ldw = (int)round_up(m, 32);
  const long long plane = (long long)n * ldw;
  // The split segments of both operands, then the products' sums.  Where there is no
  // room for those of all three products, one after another: a set of segments that
  // they share, and one plane each.
  auto scratch = [&](int sets) {
    const size_t seg = (size_t)((m + (long long)n) * ks) * sizeof(float);
    return (float *)workspace(cx, WS_3M, sets * seg + (size_t)(plane * 3 * rg.E) * rg.bytes());
  };
  bool batch = true;
  float *Xp = scratch(3);
  if (!Xp) {
    batch = false;
    if (rg.E > 1) rg = Ranges{1, 1, 3 * seg_kb, rg.range_tb, false};
    Xp = scratch(1);
  }
  if (!Xp) return B2_ERR_NOMEM;
  const int sets = batch ? 3 : 1, E = rg.E;
  float *Yp = Xp + sets * m * ks, *W = Yp + sets * n * ks;
  CUtensorMap tmX, tmY;
  int rc = umma::make_kmajor_map(&tmX, umma::KIND_TF32, Xp, ks, m, sets, ks * 4,
                                 (long long)m * ks * 4, umma::BM);
  if (rc == B2_OK)
    rc = umma::make_kmajor_map(&tmY, umma::KIND_TF32, Yp, ks, n, sets, ks * 4,
                               (long long)n * ks * 4, y_box(rg.eng));
  for (int t = 0; t < 3 && rc == B2_OK; t += sets) {
    const unsigned kt = (unsigned)kp / 32;
    const unsigned ba = kt * ((unsigned)(m + 63) / 64), bb = kt * ((unsigned)(n + 63) / 64);
    {
      B2_PROF("gemm3m_prep", s);
      B2_CUDA_TRY(launch_dependent(split3m_kernel, ba + bb, 256, s,
                                   split3_op(A, lda, !tA, cA, m, Xp),
                                   split3_op(B, ldb, tB, cB, n, Yp), ba, k, kp, batch ? -1 : t));
    }
    rc = run_engine(false, 3, tmX, tmY, m, n, kp, sets, seg_kb, rg,
                    PartialEpi{W + t * plane, plane, ldw, m, n, rg.pairs}, cx, s);
  }
  if (rc != B2_OK) return rc;
  const long long blocks = ((long long)m * n + 255) / 256;
  B2_PROF("gemm3m_combine", s);
  const unsigned grid = (unsigned)(blocks < 2368 ? blocks : 2368);
  B2_CUDA_TRY(rg.pairs ? launch_dependent(combine3m_tc_kernel<float2>, grid, 256, s,
                                          (const float2 *)W, plane, ldw, E, m, n, ar, ai, br, bi,
                                          C, ldc)
                       : launch_dependent(combine3m_tc_kernel<float>, grid, 256, s,
                                          (const float *)W, plane, ldw, E, m, n, ar, ai, br, bi, C,
                                          ldc));
  return B2_OK;
}

int sgemm_split_tf32x3(const float *X, long long sr, long long sk, int R, int K, int kp,
                       float *out, cudaStream_t s) {
  return run_split<float>(split_op(X, sr, sk, R, out), SplitOp{}, K, kp, 2, s);
}

// Tensor-core engine of an SGEMM call: 0 = single CTA, 128 x 256 tile; 1 = single
// CTA, 128 x 128 tile; 2 = CTA pair, 256 x 256 tile; 4, 6 and 6 stages, 2, 3 and 3 of
// both segments with three terms.  split: K ranges (0 = chosen from the tile count).
int sgemm_tensor_cfg(char ta, char tb, int m, int n, int k, float alpha, const float *A, int lda,
                     const float *B, int ldb, float beta, float *C, int ldc, int method,
                     const SgCfg &cfg, cudaStream_t s);

// Without selector weights: up to 1024 the 128 x 128 engine with 8 K ranges, for
// its short chains.  On 260 shapes with M, N, K log-uniform in [16, 1024] (B200) its
// mean regret against the best of the 12 configurations of a shape is 8.0 % (TF32),
// 10.9 % (TF32x3) and 14.5 % (BF16x3); the fastest single ones have chains two or eight
// times as long (4 ranges 7.1 and 10.2 %, one 7.0 %).  Larger products run on the CTA
// pair with the wave-fitting split: at 4096^3 and 8192^3 it is the fastest engine of
// every method (8192^3: TF32 787, TF32x3 279, BF16x3 485 TFLOPS, against 689 / 230 /
// 411 for the single-CTA 128 x 256 engine).
SgCfg sgemm_default_cfg(int m, int n, int k, int method) {
  (void)method;
  if (m <= 1024 && n <= 1024 && k <= 1024) return SgCfg{1, 8};
  return SgCfg{2, 0};
}

int sgemm_tensor(char ta, char tb, int m, int n, int k, float alpha, const float *A, int lda,
                 const float *B, int ldb, float beta, float *C, int ldc, int method,
                 cudaStream_t s) {
  return sgemm_tensor_cfg(ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, method,
                          sgemm_pick_cfg(ta, tb, m, n, k, beta == 0.f, method), s);
}

int sgemm_tensor_cfg(char ta, char tb, int m, int n, int k, float alpha, const float *A, int lda,
                     const float *B, int ldb, float beta, float *C, int ldc, int method,
                     const SgCfg &cfg, cudaStream_t s) {
  if (m <= 0 || n <= 0) return B2_OK;
  Ctx *cx = ctx();
  if (!cx) return B2_ERR_NO_DEVICE;
  if (k <= 0 || alpha == 0.f) return beta == 1.f ? B2_OK : scale_matrix_s(m, n, beta, C, ldc, s);
  const bool tA = !(ta == 'N' || ta == 'n');
  const bool tB = !(tb == 'N' || tb == 'n');
  const long long asr = tA ? lda : 1, ask = tA ? 1 : lda;   // op(A) rows m
  const long long bsr = tB ? 1 : ldb, bsk = tB ? ldb : 1;   // op(B) columns n
  const bool bf16 = (method == B2_METHOD_BF16X3);
  const int terms = (method == B2_METHOD_TF32) ? 1 : 3;
  const int esz = bf16 ? 2 : 4;
  const int kp = (int)round_up(k, 128 / esz);
  const int segs = terms == 3 ? 2 : 1;                      // stored segments per row
  const long long ks_ = (long long)segs * kp;
  void *Xp = workspace(cx, WS_SPLIT_X, (size_t)m * ks_ * esz);
  void *Yp = workspace(cx, WS_SPLIT_Y, (size_t)n * ks_ * esz);
  if (!Yp || !Xp) return B2_ERR_NOMEM;
  // The engine's X (accumulator lanes) is op(A): a warp's 32 lanes are then 32
  // consecutive rows of a column of C.  Stored segments: [big] or [big, small].
  const SplitOp oa = split_op(A, asr, ask, m, Xp), ob = split_op(B, bsr, bsk, n, Yp);
  int rc = bf16 ? run_split<__nv_bfloat16>(oa, ob, k, kp, segs, s)
                : run_split<float>(oa, ob, k, kp, segs, s);
  if (rc != B2_OK) return rc;
  const int kind = bf16 ? umma::KIND_BF16 : umma::KIND_TF32;
  const int seg_kb = terms == 3 ? (int)((long long)kp * esz / umma::KBLOCK_BYTES) : 0;
  const int kblocks = (int)(((long long)kp * esz + umma::KBLOCK_BYTES - 1) / umma::KBLOCK_BYTES);
  const Ranges rg = choose_ranges((cfg.engine >= 0 && cfg.engine <= 2) ? cfg.engine : 0, cfg.split,
                                  terms, kblocks, m, n, 1, cx->sm_count);
  const int E = rg.E;  // partials per tile
  CUtensorMap tmX, tmY;
  rc = umma::make_kmajor_map(&tmX, kind, Xp, ks_, m, 1, ks_ * esz, (long long)m * ks_ * esz,
                             umma::BM);
  if (rc == B2_OK)
    rc = umma::make_kmajor_map(&tmY, kind, Yp, ks_, n, 1, ks_ * esz, (long long)n * ks_ * esz,
                               y_box(rg.eng));
  if (rc != B2_OK) return rc;
  if (E == 1)
    return run_engine(bf16, terms, tmX, tmY, m, n, kp, 1, seg_kb, rg,
                      F32Epi{C, ldc, m, n, alpha, beta}, cx, s);
  // E partial products of K ranges, then one fixed-order reduction.
  const int ldw = (int)round_up(m, 32);
  const long long plane = (long long)n * ldw;
  void *W = workspace(cx, WS_MISC, (size_t)plane * E * rg.bytes());
  if (!W) return B2_ERR_NOMEM;
  rc = run_engine(bf16, terms, tmX, tmY, m, n, kp, 1, seg_kb, rg,
                  PartialEpi{W, plane, ldw, m, n, rg.pairs}, cx, s);
  if (rc != B2_OK) return rc;
  return rg.pairs ? splitk_reduce((const float2 *)W, plane, ldw, E, m, n, alpha, beta, C, ldc, s)
                 : splitk_reduce((const float *)W, plane, ldw, E, m, n, alpha, beta, C, ldc, s);
}

int sgemm_splitk_reduce(const float *W, long long plane, int ldw, int S, int m, int n,
                        float alpha, float beta, float *C, int ldc, cudaStream_t s) {
  return splitk_reduce(W, plane, ldw, S, m, n, alpha, beta, C, ldc, s);
}

}  // namespace b2
