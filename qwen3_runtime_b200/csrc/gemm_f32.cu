// C[M, N] = A[M, K] * W[N, K]^T in true fp32 on the FMA pipes: no tensor cores, no
// TF32 (large weights: gemm_f32_split.cuh, on the tensor cores in three bfloat16 parts).
// Every output element is one accumulator that takes its K products in ascending k
// order, so a row of C does not depend on M, on the tile shape chosen for M, or on
// where the row sits in the batch.  This is the matrix product of the
// engine's 32-bit path (the reference's fp32 path is torch on the CPU,
// qwen3_runtime/engine/factory.py:136-137).
//
// What bounds it: with many rows the FMA pipes (62 TFLOP/s for products of three registers, measured alone), with few
// the weights' bytes.  Rows of both operands stay k-contiguous in shared memory (no transposition: cp.async moves 16
// bytes at a time through a ring of stages), a thread reads four k-values of a row with one 16-byte load and uses each TM
// or TN times.  A thread's rows and columns are (BM / TM) and (BN / TN) apart, so that a load touches neighbouring rows,
// whose stride of BK + 4 floats spreads them over all banks.  A 16-byte load takes two cycles of shared memory if lanes
// that differ in bit 0, or those that differ in bit 1, read the same address, and four otherwise (measured): columns come
// from lane bits 0, 2, 3 and rows from bits 1, 4, so that both operands' loads are of the first kind (32 x 32 tiles 26 ->
// 35 TFLOP/s, 32 x 64 40 -> 42).  Long slices of k in two or three stages beat short ones in four or more (64 x 64: 742 ->
// 696 us at 300 x 2560 -> 19456), and tiles of 128 rows or columns are nowhere the fastest.  Since K may not be cut, an
// output too small for large tiles gets smaller ones (SHAPES).
#include "common.cuh"
#include "gemm_f32_split.cuh"

#include <stdint.h>

namespace {

__device__ __forceinline__ void copy16(void* dst, const float* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void copy4(void* dst, const float* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 4 : 0)
               : "memory");
}

// VEC: rows start at 16-byte boundaries and K is a multiple of 4; else single floats are copied.  What lies outside the
// matrices is zero: products of zeros leave an accumulator as it is.
template <int BM, int BN, int BK, int TM, int TN, int STAGES, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ C, int ldc,
                int M, int N, int K) {
  constexpr int TX = BN / TN, TY = BM / TM, THREADS = TX * TY, LD = BK + 4;
  static_assert(TX % 8 == 0 && TY % 4 == 0, "a warp is 4 x 8 threads");
  extern __shared__ __align__(16) float smem[];  // [STAGES][BM + BN][LD]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // columns from lane bits 0, 2, 3 and rows from bits 1, 4 (see above)
  const int tx = ((lane & 1) | ((lane >> 1) & 6)) + 8 * (warp % (TX / 8));
  const int ty = (((lane >> 1) & 1) | ((lane >> 3) & 2)) + 4 * (warp / (TX / 8));
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int steps = (K + BK - 1) / BK;
  // a thread copies the same columns of rows PER apart in every step
  constexpr int W4 = VEC ? 4 : 1, CHUNKS = BK / W4, PER = THREADS / CHUNKS;
  static_assert(THREADS % CHUNKS == 0 && BM % PER == 0 && BN % PER == 0, "whole rows per turn");
  const int r0 = tid / CHUNKS, kc = (tid % CHUNKS) * W4;
  const float* a_src = A + (long)(m0 + r0) * lda + kc;
  const float* w_src = W + (long)(n0 + r0) * ldw + kc;
  auto load = [&](int s) {  // one commit group per call, also when empty
    if (s < steps) {
      float* dst = smem + (s % STAGES) * (BM + BN) * LD + r0 * LD + kc;
      const bool k_in = s * BK + kc < K;
#pragma unroll
      for (int i = 0; i < BM / PER; ++i) {
        const bool in = k_in && m0 + r0 + i * PER < M;
        const float* src = in ? a_src + (long)(i * PER) * lda : A;
        if (VEC) copy16(dst + i * PER * LD, src, in); else copy4(dst + i * PER * LD, src, in);
      }
#pragma unroll
      for (int i = 0; i < BN / PER; ++i) {
        const bool in = k_in && n0 + r0 + i * PER < N;
        const float* src = in ? w_src + (long)(i * PER) * ldw : W;
        if (VEC) copy16(dst + (BM + i * PER) * LD, src, in); else copy4(dst + (BM + i * PER) * LD, src, in);
      }
      a_src += BK;
      w_src += BK;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) load(s);
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();  // step s has landed for every thread; step s - 1 has been used up
    load(s + STAGES - 1);
    const float* as = smem + (s % STAGES) * (BM + BN) * LD + ty * LD;
    const float* ws = smem + (s % STAGES) * (BM + BN) * LD + (BM + tx) * LD;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      float4 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * TY * LD + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float4 b = *reinterpret_cast<const float4*>(ws + j * TX * LD + k);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
          acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
          acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty + i * TY;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx + j * TX;
      if (gn < N) C[(long)gm * ldc + gn] = acc[i][j];
    }
  }
}

template <int BM, int BN, int BK, int TM, int TN, int STAGES>
int launch_tile(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K, bool vec,
                cudaStream_t stream) {
  constexpr size_t smem = (size_t)STAGES * (BM + BN) * (BK + 4) * sizeof(float);
  static bool configured_on[Q3_MAX_DEVICES];
  bool& configured = configured_on[q3_current_device()];
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_f32_kernel<BM, BN, BK, TM, TN, STAGES, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess ||
        cudaFuncSetAttribute(gemm_f32_kernel<BM, BN, BK, TM, TN, STAGES, false>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return Q3_ERR_LAUNCH;
    configured = true;
  }
  const dim3 block((BM / TM) * (BN / TN));
  constexpr int MOST = 65535 * BM;  // rows of one launch: a grid has at most 65535 blocks along y
  for (int m0 = 0;; m0 += MOST) {
    const int rows = M - m0 < MOST ? M - m0 : MOST;
    const dim3 grid((N + BN - 1) / BN, (rows + BM - 1) / BM);
    const float* a = A + (long)m0 * lda;
    float* c = C + (long)m0 * ldc;
    if (vec)
      gemm_f32_kernel<BM, BN, BK, TM, TN, STAGES, true><<<grid, block, smem, stream>>>(a, lda, W, ldw, c, ldc, rows, N, K);
    else
      gemm_f32_kernel<BM, BN, BK, TM, TN, STAGES, false><<<grid, block, smem, stream>>>(a, lda, W, ldw, c, ldc, rows, N, K);
    if (rows == M - m0) break;
  }
  return q3_launch_status();
}

// Time of a product on a tile shape, about ns per k-value: `first` where every SM has one tile at most, `more` for each
// further one.  Fitted to the choice, not to the times: over 147 products of 1..1000 rows at the Qwen3-4B and 8B sizes and
// one of 2048 -> 1024 the shape chosen is 0.1 % slower than the best one on average and 4 % at most.  Measured (us; one
// shape of 128 x 128 with single-float loads took 2045 for both products of 300 rows): 300 x 2560 -> 19456: 700, 300 x 9728
// -> 2560: 414, 1000 rows 48 TFLOP/s, one row 84 and 88.
struct Shape {
  int bm, bn;
  float first, more;
};
constexpr Shape SHAPES[] = {{16, 32, 3.91f, 4.4f}, {64, 64, 21.7f, 11.8f}, {32, 64, 13.0f, 6.7f},
                            {32, 32, 6.6f, 6.5f}, {16, 64, 12.9f, 4.3f},  {16, 16, 0.f, 3.5f}};
constexpr int NUM_SHAPES = sizeof(SHAPES) / sizeof(SHAPES[0]);

}  // namespace

// Leading dimensions are in elements.  tile: -1, or which of the tile shapes computes it (every one gives the same bits).
Q3_EXPORT int q3_gemm_f32(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N,
                          int K, int tile, cudaStream_t stream) {
  if (!A || !W || !C || N < 1 || K < 1 || lda < K || ldw < K || ldc < N || tile >= NUM_SHAPES) return Q3_ERR_ARGUMENT;
  if (M == 0) return Q3_OK;
  if (tile < 0) {
    static int sms_on[Q3_MAX_DEVICES];
    const int device = q3_current_device();
    if (!sms_on[device] &&
        cudaDeviceGetAttribute(&sms_on[device], cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
      return Q3_ERR_LAUNCH;
    float best = 0.f;
    for (int x = 0; x < NUM_SHAPES; ++x) {
      const long tiles = (long)((M + SHAPES[x].bm - 1) / SHAPES[x].bm) * ((N + SHAPES[x].bn - 1) / SHAPES[x].bn);
      const long per_sm = (tiles + sms_on[device] - 1) / sms_on[device];
      const float cost = SHAPES[x].first + (float)(per_sm - 1) * SHAPES[x].more;
      if (tile < 0 || cost < best) {
        tile = x;
        best = cost;
      }
    }
  }
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
  switch (tile) {
    case 0: return launch_tile<16, 32, 64, 2, 4, 4>(A, lda, W, ldw, C, ldc, M, N, K, vec, stream);
    case 1: return launch_tile<64, 64, 32, 8, 4, 3>(A, lda, W, ldw, C, ldc, M, N, K, vec, stream);
    case 2: return launch_tile<32, 64, 64, 4, 4, 2>(A, lda, W, ldw, C, ldc, M, N, K, vec, stream);
    case 3: return launch_tile<32, 32, 64, 2, 4, 3>(A, lda, W, ldw, C, ldc, M, N, K, vec, stream);
    case 4: return launch_tile<16, 64, 64, 4, 4, 3>(A, lda, W, ldw, C, ldc, M, N, K, vec, stream);
    default: return launch_tile<16, 16, 64, 2, 1, 7>(A, lda, W, ldw, C, ldc, M, N, K, vec, stream);
  }
}
