// out[M,N] (+)= A[M,K] * W[N,K]^T with 32-bit FMA on CUDA cores.
//
// This is the matrix product of the true 32-bit path (no tensor cores, hence no
// reduced-precision matrix mode) and the cross-check of the tcgen05 kernel.  Each
// output element is one sequential fused-multiply-add chain over k in both kernels
// below, so a row's result depends neither on which other rows are in the batch nor
// on the kernel or tile that computes it.  The reference's counterparts are its GEMV
// kernels (matmul infer.cu:234-248 and the fused variants infer.cu:250-337), which
// also convert each weight to 32 bits and accumulate in 32 bits.
#include "api.h"
#include "common.cuh"
#include "scan.cuh"

namespace yalm {

// ------------------------------------------------------------------ many rows
// Bound by the FMA pipe and by what shared memory delivers to registers (128 bytes a clock,
// counted per thread).  256 threads; a thread of the largest tile computes 8 x 8 outputs, 64
// multiply-adds for 64 bytes, with packed fma.rn.f32x2 (two chains per instruction, each
// rounded like fmaf), on operand tiles that lie k-major in shared memory.  The next 16 k's are
// loaded into registers under this tile's products and stored, transposed, into the other
// buffer: one barrier per 16 k's.  A warp takes 4 x 8 threads; a thread's rows and columns come
// in runs of four, a run of all threads apart.
// Measured (us, before: 64 x 64 tiles, scalar loads, one buffer): 600 x 2,048 over 8,192 k's 1,738
// -> 930, 600 x 16,384 over 2,048 1,910 -> 972, 2,048 x 16,384 over 2,048 5,855 -> 2,635 (52 TFLOP/s).
constexpr int SG_BK = 16;

// Four neighbouring k's of a row, zeros beyond K and where the row is not `live`.  VEC: K % 4 == 0 and an
// aligned base.  (Without a branch around them the loads stay in flight until `store` reads them.)
template <bool VEC, typename T>
__device__ __forceinline__ void load_four(const T* __restrict__ row, int k, int K, bool live, float* x) {
  if constexpr (VEC) {
    live = live && k < K;
    if constexpr (sizeof(T) == 4) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (live) v = *reinterpret_cast<const float4*>(row + k);
      x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    } else {
      uint2 v = make_uint2(0u, 0u);
      if (live) v = *reinterpret_cast<const uint2*>(row + k);
      const T* t = reinterpret_cast<const T*>(&v);
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = to_float(t[j]);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = live && k + j < K ? to_float(row[k + j]) : 0.f;
  }
}

template <typename TA, typename TW, typename TO, int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__(BM * BN / (TM * TN), TM * TN == 64 ? 2 : 1)
gemm_simt_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TO* __restrict__ out, int M,
                 int N, int K, int accumulate) {
  constexpr int TX = BN / TN, TY = BM / TM, THREADS = TX * TY;
  constexpr int PA = BM + 4, PW = BN + 4;
  constexpr int LA = BM * SG_BK / 4 / THREADS, LW = BN * SG_BK / 4 / THREADS;
  static_assert(TX % 8 == 0 && TY % 4 == 0 && TM % 4 == 0 && TN % 4 == 0 && LA * THREADS * 4 == BM * SG_BK &&
                    LW * THREADS * 4 == BN * SG_BK, "tile");
  __shared__ __align__(16) float As[2][SG_BK][PA];
  __shared__ __align__(16) float Ws[2][SG_BK][PW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = (warp % (TX / 8)) * 8 + (lane & 7), ty = (warp / (TX / 8)) * 4 + (lane >> 3);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  f2 acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0;

  float ra[LA][4], rw[LW][4];
  auto fetch_w = [&](int k0) {
#pragma unroll
    for (int i = 0; i < LW; ++i) {
      const int idx = tid + i * THREADS, n = n0 + (idx >> 2);
      load_four<VEC>(W + (size_t)(n < N ? n : 0) * K, k0 + (idx & 3) * 4, K, n < N, rw[i]);
    }
  };
  auto fetch_a = [&](int k0) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int idx = tid + i * THREADS, m = m0 + (idx >> 2);
      load_four<VEC>(A + (size_t)(m < M ? m : 0) * K, k0 + (idx & 3) * 4, K, m < M, ra[i]);
    }
  };
  auto store = [&](int b) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int idx = tid + i * THREADS;
#pragma unroll
      for (int j = 0; j < 4; ++j) As[b][(idx & 3) * 4 + j][idx >> 2] = ra[i][j];
    }
#pragma unroll
    for (int i = 0; i < LW; ++i) {
      const int idx = tid + i * THREADS;
#pragma unroll
      for (int j = 0; j < 4; ++j) Ws[b][(idx & 3) * 4 + j][idx >> 2] = rw[i][j];
    }
  };

  pdl_launch_dependents();
  fetch_w(0);                               // weights: nothing in a step writes them
  pdl_wait();
  fetch_a(0);
  store(0);
  __syncthreads();
  int b = 0;
  for (int k0 = 0; k0 < K; k0 += SG_BK, b ^= 1) {
    const bool more = k0 + SG_BK < K;
    if (more) {
      fetch_a(k0 + SG_BK);
      fetch_w(k0 + SG_BK);
    }
#pragma unroll
    for (int k = 0; k < SG_BK; ++k) {
      float a[TM];
      f2 w[TN / 2];
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(&As[b][k][i * TY + ty * 4]);
        a[i] = v.x; a[i + 1] = v.y; a[i + 2] = v.z; a[i + 3] = v.w;
      }
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&Ws[b][k][j * TX + tx * 4]);
        w[j / 2] = v.x; w[j / 2 + 1] = v.y;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const f2 aa = pack_f2(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = fma_f2(aa, w[j], acc[i][j]);
      }
    }
    if (more) store(b ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + (i / 4) * 4 * TY + ty * 4 + i % 4;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; j += 2) {
      const int gn = n0 + (j / 4) * 4 * TX + tx * 4 + j % 4;
      float v[2];
      unpack_f2(acc[i][j / 2], v[0], v[1]);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (gn + c >= N) continue;
        const size_t o = (size_t)gm * N + gn + c;
        float x = v[c];
        if (accumulate) x += to_float(out[o]);
        out[o] = from_float<TO>(x);
      }
    }
  }
}

// ------------------------------------------------------------------- few rows
// Up to FEW_ROWS rows (decode steps): bound by the weights' bytes, and by the length of a chain where
// the weights are few.  A block of 128 threads takes 16 weight rows and up to eight rows of A through
// an eight-stage cp.async ring of 64 k's (52 KB: four blocks and 112 KB of weights in flight per
// SM); a thread owns one output and reads both operands k-contiguously, four k's per 16-byte
// read.  A row pitch of 68 floats puts the eight weight rows that a warp reads together into
// different banks.  (One row of 16,384 x 2,048 weights 418 -> 53 us, of 2,048 x 8,192 621 -> 75; the tiles
// above take 66 and 320 us from 17 rows on.)
constexpr int FEW_ROWS = 16;
constexpr int FR_M = 8, FR_N = 16, FR_K = 64, FR_STAGES = 8, FR_PITCH = FR_K + 4;
constexpr int FR_SMEM = FR_STAGES * (FR_M + FR_N) * FR_PITCH * 4;

__device__ __forceinline__ void fr_copy(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

template <typename TO>
__global__ void __launch_bounds__(128)
gemm_simt_few_kernel(const float* __restrict__ A, const float* __restrict__ W, TO* __restrict__ out, int M,
                     int N, int K, int accumulate) {
  extern __shared__ __align__(16) float fr_smem[];
  float (*Ws)[FR_N][FR_PITCH] = reinterpret_cast<float (*)[FR_N][FR_PITCH]>(fr_smem);
  float (*As)[FR_M][FR_PITCH] =
      reinterpret_cast<float (*)[FR_M][FR_PITCH]>(fr_smem + FR_STAGES * FR_N * FR_PITCH);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n0 = blockIdx.x * FR_N, m0 = blockIdx.y * FR_M;
  const int nt = (K + FR_K - 1) / FR_K;
  // a thread copies 16 bytes of a row at a time: rows tid / 16 (+ 8), k's 4 (tid % 16)
  const int r = tid >> 4, c = (tid & 15) * 4;
  auto load_w = [&](int t) {
    const int k = t * FR_K + c;
#pragma unroll
    for (int i = 0; i < FR_N / 8; ++i) {
      const int n = n0 + r + i * 8;
      const bool on = n < N && k < K;
      fr_copy(&Ws[t % FR_STAGES][r + i * 8][c], on ? W + (size_t)n * K + k : W, on ? 16 : 0);
    }
  };
  auto load_a = [&](int t) {
    const int k = t * FR_K + c, m = m0 + r;
    const bool on = m < M && k < K;
    fr_copy(&As[t % FR_STAGES][r][c], on ? A + (size_t)m * K + k : A, on ? 16 : 0);
  };
  pdl_launch_dependents();
#pragma unroll
  for (int t = 0; t < FR_STAGES - 1; ++t)
    if (t < nt) load_w(t);                       // weights: before the previous kernel has ended
  pdl_wait();
#pragma unroll
  for (int t = 0; t < FR_STAGES - 1; ++t) {
    if (t < nt) load_a(t);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const int nx = (warp & 1) * 8 + (lane & 7), my = (warp >> 1) * 4 + (lane >> 3);
  float acc = 0.f;
  for (int t = 0; t < nt; ++t) {
    asm volatile("cp.async.wait_group %0;" ::"n"(FR_STAGES - 2) : "memory");
    __syncthreads();
    const float* ap = &As[t % FR_STAGES][my][0];
    const float* wp = &Ws[t % FR_STAGES][nx][0];
    const int next = t + FR_STAGES - 1;          // into the stage that every thread left before the barrier above
    if (next < nt) {
      load_w(next);
      load_a(next);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
    for (int k = 0; k < FR_K; k += 4) {
      const float4 a = *reinterpret_cast<const float4*>(ap + k);
      const float4 w = *reinterpret_cast<const float4*>(wp + k);
      acc = fmaf(a.x, w.x, acc);
      acc = fmaf(a.y, w.y, acc);
      acc = fmaf(a.z, w.z, acc);
      acc = fmaf(a.w, w.w, acc);
    }
  }
  const int gm = m0 + my, gn = n0 + nx;
  if (gm >= M || gn >= N) return;
  const size_t o = (size_t)gm * N + gn;
  if (accumulate) acc += to_float(out[o]);
  out[o] = from_float<TO>(acc);
}

constexpr int SG_SMS = 148;

template <typename TA, typename TW, typename TO, int BM, int BN, int TM, int TN>
static int launch_tile(const void* A, const void* W, void* out, int M, int N, int K, int accumulate,
                       cudaStream_t stream) {
  const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM), block(BM * BN / (TM * TN));
  if (grid.y > 65535) return -4;
  const bool vec = K % 4 == 0 && (uintptr_t)A % (4 * sizeof(TA)) == 0 && (uintptr_t)W % (4 * sizeof(TW)) == 0;
  auto kernel = vec ? gemm_simt_kernel<TA, TW, TO, BM, BN, TM, TN, true> : gemm_simt_kernel<TA, TW, TO, BM, BN, TM, TN, false>;
  // No more large tiles than SMs: one block per SM (the shared memory that it asks for keeps a second one out).
  // While the previous kernel drains, blocks would otherwise pair up on the SMs that are free first and
  // take 1.75 times as long there (1,024 x 2,048 outputs over 2,048 k's: 379 against 216 us).
  int alone = 0;
  if (TM * TN >= 32 && (long long)grid.x * grid.y <= SG_SMS) {
    alone = 100 * 1024;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, alone);
    if (e != cudaSuccess) return (int)e;
  }
  launch_pdl(kernel, grid, block, alone, stream, (const TA*)A, (const TW*)W, (TO*)out, M, N, K, accumulate);
  YALM_LAUNCH_CHECK();
  return 0;
}

// The tile shape for an [M, N] product of 32-bit operands, by estimated time.  Measured at K = 2,048, us: a
// block of 128 x 128 alone on its SM 216, two of them 380; of 64 x 128 140 and 250; 32 x 64 tiles 0.27 each
// over the whole device, and no less than 66.  0: 128 x 128, 1: 64 x 128, 2: 32 x 64.
constexpr long long SIMT_MAX_ROWS = 65535LL * 64;             // (a grid has up to 65,535 rows of blocks)
static int simt_tile(int M, int N) {
  auto blocks = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
  auto rounds = [](long long b, double one, double two) {
    const long long left = b % (2 * SG_SMS);
    return (double)(b / (2 * SG_SMS)) * two + (left == 0 ? 0.0 : left <= SG_SMS ? one : two);
  };
  const double t128 = rounds(blocks(128, 128), 216, 380), t64 = rounds(blocks(64, 128), 140, 250);
  const double small = 0.27 * (double)blocks(32, 64) + 20, t32 = small > 66 ? small : 66;
  const bool can32 = M <= 65535LL * 32;
  return t128 <= t64 && (t128 <= t32 || !can32) ? 0 : t64 <= t32 || !can32 ? 1 : 2;
}

template <typename TA, typename TW, typename TO>
static int launch_simt_out(const void* A, const void* W, void* out, int M, int N, int K, int accumulate,
                           cudaStream_t stream) {
  if constexpr (sizeof(TA) == 4 && sizeof(TW) == 4) {
    if (M <= FEW_ROWS && K % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0) {
      const cudaError_t e =
          cudaFuncSetAttribute(gemm_simt_few_kernel<TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, FR_SMEM);
      if (e != cudaSuccess) return (int)e;
      launch_pdl(gemm_simt_few_kernel<TO>, dim3((N + FR_N - 1) / FR_N, (M + FR_M - 1) / FR_M), dim3(128), FR_SMEM,
                 stream, (const float*)A, (const float*)W, (TO*)out, M, N, K, accumulate);
      YALM_LAUNCH_CHECK();
      return 0;
    }
    switch (simt_tile(M, N)) {
      case 0: return launch_tile<TA, TW, TO, 128, 128, 8, 8>(A, W, out, M, N, K, accumulate, stream);
      case 1: return launch_tile<TA, TW, TO, 64, 128, 4, 8>(A, W, out, M, N, K, accumulate, stream);
      default: return launch_tile<TA, TW, TO, 32, 64, 4, 4>(A, W, out, M, N, K, accumulate, stream);
    }
  }
  // 16-bit or mixed operands: a matrix stored in 32 bits under 16-bit compute, and cross-checks
  return launch_tile<TA, TW, TO, 64, 64, 4, 4>(A, W, out, M, N, K, accumulate, stream);
}

template <typename TA, typename TW>
static int launch_simt(const void* A, const void* W, void* out, int out_dtype, int M, int N, int K,
                       int accumulate, cudaStream_t stream) {
  if (out_dtype == DT_F32) return launch_simt_out<TA, TW, float>(A, W, out, M, N, K, accumulate, stream);
  if (out_dtype == DT_BF16) return launch_simt_out<TA, TW, __nv_bfloat16>(A, W, out, M, N, K, accumulate, stream);
  if (out_dtype == DT_F16) return launch_simt_out<TA, TW, __half>(A, W, out, M, N, K, accumulate, stream);
  return -3;
}

}  // namespace yalm

using namespace yalm;

extern "C" int yalm_gemm_simt(const void* A, int a_dtype, const void* W, int w_dtype, void* out,
                              int out_dtype, int M, int N, int K, int accumulate,
                              cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return -2;
  if (M > SIMT_MAX_ROWS) return -4;
  if (a_dtype == DT_F32 && w_dtype == DT_F32)
    return launch_simt<float, float>(A, W, out, out_dtype, M, N, K, accumulate, stream);
  if (a_dtype == DT_BF16 && w_dtype == DT_BF16)
    return launch_simt<__nv_bfloat16, __nv_bfloat16>(A, W, out, out_dtype, M, N, K, accumulate,
                                                     stream);
  if (a_dtype == DT_F32 && w_dtype == DT_BF16)
    return launch_simt<float, __nv_bfloat16>(A, W, out, out_dtype, M, N, K, accumulate, stream);
  if (a_dtype == DT_BF16 && w_dtype == DT_F32)
    return launch_simt<__nv_bfloat16, float>(A, W, out, out_dtype, M, N, K, accumulate, stream);
  if (a_dtype == DT_F16 && w_dtype == DT_F16)
    return launch_simt<__half, __half>(A, W, out, out_dtype, M, N, K, accumulate, stream);
  if (a_dtype == DT_F32 && w_dtype == DT_F16)
    return launch_simt<float, __half>(A, W, out, out_dtype, M, N, K, accumulate, stream);
  if (a_dtype == DT_F16 && w_dtype == DT_F32)
    return launch_simt<__half, float>(A, W, out, out_dtype, M, N, K, accumulate, stream);
  return -3;
}

// The tile that more than FEW_ROWS rows of 32-bit operands run on: its rows times 1,000 plus its columns.
extern "C" int yalm_gemm_simt_tile(int M, int N) {
  const int t = simt_tile(M, N);
  return t == 0 ? 128128 : t == 1 ? 64128 : 32064;
}
