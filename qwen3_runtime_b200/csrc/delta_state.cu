// The gated delta rule with a decay per key channel, on a matrix state S [D, Dv] per (sequence, head):
//
//   S <- diag(g_t) S;   u = beta_t (v_t - S^T k_t);   S <- S + k_t u^T;   o_t = S^T q_t
//
// and what surrounds it: a short causal convolution with silu on every channel of q, k and v, unit vectors for q
// and k per head, g = exp(neg_a_h * softplus(z + dt_bias)), beta = sigmoid(b).  q and k have G heads, v and the
// state H = a multiple of G; head h reads q/k head h / (H / G).  The state, decays, steps, unit vectors and all
// sums are fp32.
//
// The convolution's past inputs live in a ring of `taps` rows per state slot (fp32 [taps, C]; the input of
// position p sits in row p mod taps), so a step that brings one token writes its row beside the rows that are
// still read.  Rows of positions before the sequence's start are never read: they count as zeros.
//
//   delta_prepare    every token of a step: convolution, silu, unit vectors, decays and steps as rows in memory
//   ring_update      the last rows of every sequence's portion into the ring (after delta_prepare has read it)
//   delta_scan       the recurrence over every sequence's tokens of the step, from delta_prepare's rows
//   delta_chunk_*    the same in chunks of 16 tokens, for prompts
//   delta_step       all of it for steps in which every sequence brings one token, with the decay's and the
//                    gate's second low-rank products and the heads' output norm and gate: one kernel
#include "common.cuh"
#include "split_mma.cuh"

#define DELTA_MAX_TAPS 16
#define UNIT_EPS 1e-6f

static inline bool ds_aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

__device__ __forceinline__ float softplus_f(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + expf(-x)); }

// E (1 or 8) consecutive channels' convolution at token t of the step, n rows into its sequence's portion, at
// position p; ring: the slot's rows.  w: fp32 [taps, C].
template <typename T, int E>
__device__ __forceinline__ void conv_silu(const T* __restrict__ xrow, long x_stride, const float* __restrict__ w,
                                          int taps, const float* __restrict__ ring, int C, int n, int p, int c,
                                          float (&y)[E]) {
#pragma unroll
  for (int e = 0; e < E; ++e) y[e] = 0.f;
#pragma unroll 4
  for (int j = 0; j < taps; ++j) {
    const int back = taps - 1 - j;
    if (p - back < 0) continue;
    float u[E], wv[E];
    if constexpr (E == 8) {
      if (n - back >= 0) load8(xrow - (long)back * x_stride + c, u);
      else load8(ring + (long)((p - back) % taps) * C + c, u);
      load8(w + (long)j * C + c, wv);
    } else {
      u[0] = n - back >= 0 ? to_f32(xrow[-(long)back * x_stride + c]) : ring[(long)((p - back) % taps) * C + c];
      wv[0] = w[(long)j * C + c];
    }
#pragma unroll
    for (int e = 0; e < E; ++e) y[e] = fmaf(wv[e], u[e], y[e]);
  }
#pragma unroll
  for (int e = 0; e < E; ++e) y[e] = y[e] * sigmoid_f(y[e]);
}

// Warps of a block take the token's work items: groups of q and k heads (a warp holds 32 / lph heads, lph lanes of E
// elements each and, for E = 1, up to 8 strided elements), then groups of 32 * E value channels, then groups of
// 32 * E decays, then the steps.  v is kept in the activation type; q and k are normalised from the convolution's
// fp32 values.
template <typename T, int E>
__global__ void __launch_bounds__(256)
delta_prepare_kernel(const T* __restrict__ x, long x_stride, const float* __restrict__ w, int taps,
                     const float* __restrict__ ring, const int* __restrict__ positions,
                     const int* __restrict__ token_seq, const int* __restrict__ cu_seqlens,
                     const int* __restrict__ state_slots, const float* __restrict__ z, const float* __restrict__ dt_bias,
                     const float* __restrict__ neg_a, const T* __restrict__ b, long b_stride, float q_scale,
                     float* __restrict__ qn, float* __restrict__ kn, T* __restrict__ vc, float* __restrict__ g,
                     float* __restrict__ beta, int G, int H, int D, int Dv, int lph) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, lane = threadIdx.x & 31;
  int item = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int seq = token_seq[t], p = positions[t], n = t - cu_seqlens[seq];
  const int C = 2 * G * D + H * Dv;
  const T* xrow = x + (long)t * x_stride;
  const float* rows = taps > 1 ? ring + (long)state_slots[seq] * taps * C : nullptr;
  const int per_warp = 32 / lph;
  const int qk_items = (2 * G + per_warp - 1) / per_warp, v_items = (H * Dv + 32 * E - 1) / (32 * E),
            g_items = (H * D + 32 * E - 1) / (32 * E);
  if (item < qk_items) {
    const int head = item * per_warp + lane / lph;  // q heads, then k heads
    const bool live_head = head < 2 * G;
    constexpr int M = E == 8 ? 1 : 8;               // strided groups of a lane (E = 1: elements lane + 32 m)
    float y[M][E];
    float ss = 0.f;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int d = E == 8 ? (lane % lph) * 8 : lane + 32 * m;
#pragma unroll
      for (int e = 0; e < E; ++e) y[m][e] = 0.f;
      if (live_head && d < D) conv_silu<T, E>(xrow, x_stride, w, taps, rows, C, n, p, head * D + d, y[m]);
#pragma unroll
      for (int e = 0; e < E; ++e) ss += y[m][e] * y[m][e];
    }
    for (int o = lph >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (!live_head) return;
    const float inv = rsqrtf(ss + UNIT_EPS) * (head < G ? q_scale : 1.f);
    float* dst = head < G ? qn + ((long)t * G + head) * D : kn + ((long)t * G + head - G) * D;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int d = E == 8 ? (lane % lph) * 8 : lane + 32 * m;
      if (d >= D) continue;
#pragma unroll
      for (int e = 0; e < E; ++e) y[m][e] *= inv;
      if constexpr (E == 8) store8(dst + d, y[m]); else dst[d] = y[m][0];
    }
    return;
  }
  item -= qk_items;
  if (item < v_items) {
    const int c = (item * 32 + lane) * E;
    if (c >= H * Dv) return;
    float y[E];
    conv_silu<T, E>(xrow, x_stride, w, taps, rows, C, n, p, 2 * G * D + c, y);
    T* dst = vc + (long)t * H * Dv + c;
    if constexpr (E == 8) store8(dst, y); else dst[0] = from_f32<T>(y[0]);
    return;
  }
  item -= v_items;
  if (item < g_items) {
    const int c = (item * 32 + lane) * E;
    if (c >= H * D) return;
    float zz[E], bb[E];
    if constexpr (E == 8) {
      load8(z + (long)t * H * D + c, zz);
      load8(dt_bias + c, bb);
    } else {
      zz[0] = z[(long)t * H * D + c];
      bb[0] = dt_bias[c];
    }
    const float a = neg_a[c / D];
#pragma unroll
    for (int e = 0; e < E; ++e) zz[e] = expf(a * softplus_f(zz[e] + bb[e]));
    float* dst = g + (long)t * H * D + c;
    if constexpr (E == 8) store8(dst, zz); else dst[0] = zz[0];
    return;
  }
  item -= g_items;
  const int h = item * 32 + lane;
  if (h < H) beta[(long)t * H + h] = sigmoid_f(to_f32(b[(long)t * b_stride + h]));
}

// x: [T, C] rows (q heads | k heads | v heads), w fp32 [taps, C], ring fp32 [slots, taps, C]; z fp32 [T, H * D];
// neg_a fp32 [H] (-exp of the stored logarithm); b [T, H] rows b_stride apart; qn, kn fp32 [T, G, D]; vc [T, H, Dv];
// g fp32 [T, H, D]; beta fp32 [T, H].
Q3_EXPORT int q3_delta_prepare(int dtype, const void* x, long x_stride, const float* w, int taps, const float* ring,
                               const int* positions, const int* token_seq, const int* cu_seqlens,
                               const int* state_slots, const float* z, const float* dt_bias, const float* neg_a,
                               const void* b, long b_stride, float q_scale, float* qn, float* kn, void* vc, float* g,
                               float* beta, int num_tokens, int G, int H, int D, int Dv, cudaStream_t stream) {
  if (!x || !w || !positions || !token_seq || !cu_seqlens || !state_slots || !z || !dt_bias || !neg_a || !b || !qn || !kn ||
      !vc || !g || !beta)
    return Q3_ERR_ARGUMENT;
  if (G < 1 || H < 1 || H % G || D < 1 || Dv < 1 || taps < 1 || (taps > 1 && !ring)) return Q3_ERR_ARGUMENT;
  if (D > 256 || taps > DELTA_MAX_TAPS) return Q3_ERR_UNSUPPORTED;
  if (num_tokens == 0) return Q3_OK;
  const bool vec = D % 8 == 0 && Dv % 8 == 0 && x_stride % 8 == 0 && ds_aligned(x) && ds_aligned(w) && ds_aligned(ring) &&
                   ds_aligned(z) && ds_aligned(dt_bias) && ds_aligned(qn) && ds_aligned(kn) && ds_aligned(vc) &&
                   ds_aligned(g);
  const int E = vec ? 8 : 1;
  int lph = 32;
  if (vec) {
    lph = 1;
    while (lph * 8 < D) lph <<= 1;
  }
  const int items = (2 * G + 32 / lph - 1) / (32 / lph) + (H * Dv + 32 * E - 1) / (32 * E) +
                    (H * D + 32 * E - 1) / (32 * E) + (H + 31) / 32;
  const dim3 grid(num_tokens, (items + 7) / 8);
  if (grid.y > 65535) return Q3_ERR_UNSUPPORTED;
  cudaError_t e;
#define Q3_DELTA_PREPARE(T, EE)                                                                                      \
  e = launch_pdl(delta_prepare_kernel<T, EE>, grid, dim3(256), 0, stream, (const T*)x, x_stride, w, taps, ring, positions, \
                 token_seq, cu_seqlens, state_slots, z, dt_bias, neg_a, (const T*)b, b_stride, q_scale, qn, kn, (T*)vc, g, \
                 beta, G, H, D, Dv, lph)
  if (dtype == Q3_DTYPE_F32) {
    if (vec) Q3_DELTA_PREPARE(float, 8); else Q3_DELTA_PREPARE(float, 1);
  } else if (dtype == Q3_DTYPE_BF16) {
    if (vec) Q3_DELTA_PREPARE(bf16, 8); else Q3_DELTA_PREPARE(bf16, 1);
  } else {
    return Q3_ERR_ARGUMENT;
  }
#undef Q3_DELTA_PREPARE
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}

// The last taps rows of every sequence's portion into its ring (rows of earlier positions stay where they are).
template <typename T>
__global__ void ring_update_kernel(const T* __restrict__ x, long x_stride, float* __restrict__ ring,
                                   const int* __restrict__ positions, const int* __restrict__ cu_seqlens,
                                   const int* __restrict__ state_slots, int taps, int C, long total) {
  pdl_wait();
  pdl_launch_dependents();
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int seq = (int)(idx / C), c = (int)(idx - (long)seq * C);
  const int t0 = cu_seqlens[seq], t1 = cu_seqlens[seq + 1];
  float* rows = ring + (long)state_slots[seq] * taps * C;
  for (int t = max(t0, t1 - taps); t < t1; ++t) rows[(long)(positions[t] % taps) * C + c] = to_f32(x[(long)t * x_stride + c]);
}

Q3_EXPORT int q3_ring_update(int dtype, const void* x, long x_stride, float* ring, const int* positions,
                             const int* cu_seqlens, const int* state_slots, int taps, int C, int num_seqs,
                             cudaStream_t stream) {
  if (!x || !ring || !positions || !cu_seqlens || !state_slots || C < 1 || taps < 1) return Q3_ERR_ARGUMENT;
  const long total = (long)num_seqs * C;
  if (total == 0) return Q3_OK;
  const unsigned blocks = (unsigned)((total + 255) / 256);
  cudaError_t e;
  if (dtype == Q3_DTYPE_F32)
    e = launch_pdl(ring_update_kernel<float>, dim3(blocks), dim3(256), 0, stream, (const float*)x, x_stride, ring,
                   positions, cu_seqlens, state_slots, taps, C, total);
  else if (dtype == Q3_DTYPE_BF16)
    e = launch_pdl(ring_update_kernel<bf16>, dim3(blocks), dim3(256), 0, stream, (const bf16*)x, x_stride, ring, positions,
                   cu_seqlens, state_slots, taps, C, total);
  else
    return Q3_ERR_ARGUMENT;
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}

// ---- the recurrence, token by token ------------------------------------------------------------------
// One block per (VT value columns, head, sequence).  A thread owns R key rows of one value column of the state in
// registers; the RG row groups of a column are neighbouring lanes of a warp, so the two sums a token needs -- the
// decayed state times k and times q -- are shuffle sums that run side by side: with them and k . q,
// o = (g S)^T q + u (k . q), so the output does not wait for the state's update.  Tokens come CT at a time through a
// double buffer in shared memory whose next half is fetched into registers while this one is worked on.
#define DS_CT 16
template <typename T, int RG, int R, int VT>
__global__ void __launch_bounds__(RG * VT)
delta_scan_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const T* __restrict__ vc,
                  const float* __restrict__ g, const float* __restrict__ beta, float* __restrict__ state,
                  const int* __restrict__ cu_seqlens, const int* __restrict__ state_slots, float* __restrict__ out, int G,
                  int H, int D, int Dv, int longest) {
  constexpr int THREADS = RG * VT, DP = RG * R, CPW = 32 / RG;
  constexpr int EPT = DS_CT * DP / THREADS;
  constexpr int VPT = (DS_CT * VT + THREADS - 1) / THREADS;
  extern __shared__ __align__(16) float ds_smem[];
  float* qs = ds_smem;                           // [2][CT][DP]
  float* ks = qs + 2 * DS_CT * DP;
  float* gs = ks + 2 * DS_CT * DP;
  float* vs = gs + 2 * DS_CT * DP;               // [2][CT][VT]
  float* bs = vs + 2 * DS_CT * VT;               // [2][CT]
  pdl_wait();
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rg = lane % RG, col = warp * CPW + lane / RG;
  const int h = blockIdx.y, seq = blockIdx.z, gh = h / (H / G);
  const int j = blockIdx.x * VT + col;
  const int t0 = cu_seqlens[seq], t1 = cu_seqlens[seq + 1];
  if (t1 <= t0 || t1 - t0 > longest) return;
  float* Sg = state + ((long)state_slots[seq] * H + h) * (long)D * Dv;
  float S[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = rg * R + r;
    S[r] = (i < D && j < Dv) ? Sg[(long)i * Dv + j] : 0.f;
  }
  float qr[EPT], kr[EPT], gr[EPT], br = 0.f;
  float vr[VPT];
  auto fetch = [&](int c0) {
#pragma unroll
    for (int m = 0; m < EPT; ++m) {
      const int x = tid + m * THREADS, c = x / DP, i = x - c * DP;
      const long t = c0 + c;
      const bool live = t < t1 && i < D;
      qr[m] = live ? qn[(t * G + gh) * D + i] : 0.f;
      kr[m] = live ? kn[(t * G + gh) * D + i] : 0.f;
      gr[m] = live ? g[(t * H + h) * D + i] : 0.f;
    }
#pragma unroll
    for (int m = 0; m < VPT; ++m) {
      const int x = tid + m * THREADS, c = x / VT, jj = blockIdx.x * VT + x % VT;
      const long t = c0 + c;
      vr[m] = (x < DS_CT * VT && t < t1 && jj < Dv) ? to_f32(vc[(t * H + h) * Dv + jj]) : 0.f;
    }
    if (tid < DS_CT) br = c0 + tid < t1 ? beta[(long)(c0 + tid) * H + h] : 0.f;
  };
  auto stage = [&](int buf) {
#pragma unroll
    for (int m = 0; m < EPT; ++m) {
      const int x = tid + m * THREADS;
      qs[buf * DS_CT * DP + x] = qr[m];
      ks[buf * DS_CT * DP + x] = kr[m];
      gs[buf * DS_CT * DP + x] = gr[m];
    }
#pragma unroll
    for (int m = 0; m < VPT; ++m) {
      const int x = tid + m * THREADS;
      if (x < DS_CT * VT) vs[buf * DS_CT * VT + x] = vr[m];
    }
    if (tid < DS_CT) bs[buf * DS_CT + tid] = br;
  };
  fetch(t0);
  stage(0);
  __syncthreads();
  int buf = 0;
  for (int c0 = t0; c0 < t1; c0 += DS_CT, buf ^= 1) {
    const int n = min(DS_CT, t1 - c0);
    const bool more = c0 + DS_CT < t1;
    if (more) fetch(c0 + DS_CT);
    for (int c = 0; c < n; ++c) {
      const float* qc = qs + (buf * DS_CT + c) * DP + rg * R;
      const float* kc = ks + (buf * DS_CT + c) * DP + rg * R;
      const float* gc = gs + (buf * DS_CT + c) * DP + rg * R;
      float sk = 0.f, sq = 0.f, kq = 0.f, kk[R];
#pragma unroll
      for (int r = 0; r < R; r += 4) {
        const float4 a = *reinterpret_cast<const float4*>(gc + r);
        const float4 k4 = *reinterpret_cast<const float4*>(kc + r);
        const float4 q4 = *reinterpret_cast<const float4*>(qc + r);
        kk[r] = k4.x; kk[r + 1] = k4.y; kk[r + 2] = k4.z; kk[r + 3] = k4.w;
        S[r] *= a.x; S[r + 1] *= a.y; S[r + 2] *= a.z; S[r + 3] *= a.w;
        sk = fmaf(S[r], k4.x, sk); sq = fmaf(S[r], q4.x, sq); kq = fmaf(k4.x, q4.x, kq);
        sk = fmaf(S[r + 1], k4.y, sk); sq = fmaf(S[r + 1], q4.y, sq); kq = fmaf(k4.y, q4.y, kq);
        sk = fmaf(S[r + 2], k4.z, sk); sq = fmaf(S[r + 2], q4.z, sq); kq = fmaf(k4.z, q4.z, kq);
        sk = fmaf(S[r + 3], k4.w, sk); sq = fmaf(S[r + 3], q4.w, sq); kq = fmaf(k4.w, q4.w, kq);
      }
#pragma unroll
      for (int o = 1; o < RG; o <<= 1) {
        sk += __shfl_xor_sync(0xffffffffu, sk, o);
        sq += __shfl_xor_sync(0xffffffffu, sq, o);
        kq += __shfl_xor_sync(0xffffffffu, kq, o);
      }
      const float u = bs[buf * DS_CT + c] * (vs[(buf * DS_CT + c) * VT + col] - sk);
#pragma unroll
      for (int r = 0; r < R; ++r) S[r] = fmaf(kk[r], u, S[r]);
      if (rg == 0 && j < Dv) out[((long)(c0 + c) * H + h) * Dv + j] = fmaf(u, kq, sq);
    }
    if (more) stage(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = rg * R + r;
    if (i < D && j < Dv) Sg[(long)i * Dv + j] = S[r];
  }
}

template <typename T, int RG, int R, int VT>
static cudaError_t launch_delta_scan(cudaStream_t stream, int num_seqs, const float* qn, const float* kn, const void* vc,
                                     const float* g, const float* beta, float* state, const int* cu_seqlens,
                                     const int* state_slots, float* out, int G, int H, int D, int Dv, int longest) {
  constexpr size_t smem = (size_t)(6 * DS_CT * RG * R + 2 * DS_CT * VT + 2 * DS_CT) * sizeof(float);
  auto kernel = delta_scan_kernel<T, RG, R, VT>;
  if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return launch_pdl(kernel, dim3((Dv + VT - 1) / VT, H, num_seqs), dim3(RG * VT), smem, stream, qn, kn, (const T*)vc, g,
                    beta, state, cu_seqlens, state_slots, out, G, H, D, Dv, longest);
}

// qn, kn, vc, g, beta: delta_prepare's rows; state fp32 [slots, H, D, Dv]; out fp32 [T, H, Dv].  Sequences of more than
// `longest` tokens are left alone.
Q3_EXPORT int q3_delta_scan(int dtype, const float* qn, const float* kn, const void* vc, const float* g,
                            const float* beta, float* state, const int* cu_seqlens, const int* state_slots, float* out,
                            int num_seqs, int G, int H, int D, int Dv, int longest, cudaStream_t stream) {
  if (!qn || !kn || !vc || !g || !beta || !state || !cu_seqlens || !state_slots || !out) return Q3_ERR_ARGUMENT;
  if (G < 1 || H < 1 || H % G || D < 1 || Dv < 1 || H > 65535 || num_seqs > 65535) return Q3_ERR_ARGUMENT;
  if (D > 256 || (dtype != Q3_DTYPE_F32 && dtype != Q3_DTYPE_BF16)) return Q3_ERR_UNSUPPORTED;
  if (num_seqs == 0) return Q3_OK;
  cudaError_t e;
#define Q3_DELTA_SCAN(T, RG, R, VT)                                                                                  \
  e = launch_delta_scan<T, RG, R, VT>(stream, num_seqs, qn, kn, vc, g, beta, state, cu_seqlens, state_slots, out, G, H, \
                                      D, Dv, longest)
#define Q3_DELTA_SIZES(T)                                                                                            \
  if (D <= 16) Q3_DELTA_SCAN(T, 4, 4, 16); else if (D <= 32) Q3_DELTA_SCAN(T, 8, 4, 16);                              \
  else if (D <= 64) Q3_DELTA_SCAN(T, 8, 8, 16); else if (D <= 128) Q3_DELTA_SCAN(T, 16, 8, 16);                       \
  else Q3_DELTA_SCAN(T, 32, 8, 16)
  if (dtype == Q3_DTYPE_F32) { Q3_DELTA_SIZES(float); } else { Q3_DELTA_SIZES(bf16); }
#undef Q3_DELTA_SIZES
#undef Q3_DELTA_SCAN
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}

// ---- the recurrence in chunks of 16 tokens ------------------------------------------------------------
// With G_i the product of a chunk's decays up to token i and S the state before the chunk, the recurrence is, in
// matrices whose rows are the chunk's tokens (the WY form of a product of rank-one updates):
//   A_ij = sum_d k_i k_j prod_(j < m <= i) g_m  (j < i)        B_ij = sum_d q_i k_j prod_(j < m <= i) g_m  (j <= i)
//   P = (I + diag(beta) A)^(-1) diag(beta) (G k)                U0 = (I + diag(beta) A)^(-1) diag(beta) V
//   Q = G q - B P                                              O0 = B U0
//   U = U0 - P S      O = O0 + Q S      S <- G_last S + sum_j (prod_(m > j) g_m k_j) u_j^T
// P, Q, U0 and O0 do not depend on the state, so only two products are left in the chain from chunk to chunk.  A row of P
// is beta_i k_i times a product of contractions and no longer than beta_i |k_i|.  Only products of decays occur, never
// quotients, so strong decays lose nothing.
//
// Products of matrices run on mma.sync with every operand as the sum of three bfloat16 (split_mma.cuh) and the six
// products of parts that matter, the largest alone and added last; what a product adds to the state is summed from zero and
// added to it in fp32, once per chunk.  Everything else is fp32 FMA.  Against float64 (700 + 300 tokens, 16 heads of 128,
// mean decays of 0.95 / 0.9997 a token): outputs 1.2e-7 / 2.2e-7, state 1.0e-7 / 2.2e-7; with FMA throughout 1.3e-7 / 3.4e-7
// and 1.0e-7 / 3.6e-7.
//
// delta_chunk_rows: everything that does not depend on the state.  A record of DC_REC words per (chunk, head), operands in
// three parts in the order of the products' fragments: P, Q and the decayed-to-the-end keys [DP / 16][3][32 lanes][4], G_last
// [DP] in fp32; U0 in rows of its own, O0 where the output will be.  Chunks of sequence b start at place cu_seqlens[b] / 16 + b;
// tokens beyond a portion's end are k = q = 0, g = 1, beta = 0.
// delta_chunk_scan: one block per (16 value columns, head, sequence); the state's columns stay in registers, the next chunks'
// records are on their way while one is worked on.
// 1500 + 548 tokens of 16 heads, rows and scan: 41 + 225 us with FMA, four barriers a chunk and W, B in the chain; 56 + 114 us
// now.  (The scan on FMA without W and B in the chain 144 us, on mma.sync with both halves' work in all warps 159, with the
// parts made in the scan instead of stored 125; the rows with substitutions for every column on FMA 68.)
#define DC_C 16
#define DC_REC(DP) ((DP) * 73)

// Element (i, its column) of a product with a lower triangular matrix of tokens, whose parts lie at `left` in the order of a left
// operand, from rows 0 .. i of the right operand only (at(j): row j's element of the column).
template <typename F>
__device__ __forceinline__ float ds_own_rows(const uint32_t* left, int i, F at) {
  float sum = 0.f;
  for (int j = 0; j <= i; ++j) {
    const int place = ((i & 7) * 4 + ((j & 7) >> 1)) * 4 + (i >> 3) + 2 * (j >> 3), shift = j & 1 ? 0 : 16;
    float w = 0.f;
    for (int m = 2; m >= 0; --m) w += __uint_as_float((left[m * 128 + place] << shift) & 0xffff0000u);
    sum = fmaf(w, at(j), sum);
  }
  return sum;
}
// A warp's share of a record once more where keys or values are not finite: W and B W hold zeros behind a row's own token, which in
// the products make a NaN of an earlier token's row.  Behind everything else, so that the products' registers are free.
template <typename T, int DP>
__device__ __forceinline__ void delta_own_rows(uint32_t* rec, const uint32_t* w, const uint32_t* bw, const float* gk, const float* gq,
                                            int pitch, const T* v, float* u0, float* out, long row, int n, int Dv) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, t4 = lane & 3;
  for (int x = 0; x < 2; ++x)
    for (int i = 0; i < 2; ++i) {
      const int c = gr + 8 * i;
      if (warp < DP / 16) {
        const int d = warp * 16 + 8 * x + 2 * t4, at = warp * 384 + lane * 4 + 2 * i + x;
        float p[2], q[2];
        for (int e = 0; e < 2; ++e) {
          p[e] = ds_own_rows(w, c, [&](int j) { return gk[j * pitch + d + e]; });
          q[e] = gq[c * pitch + d + e] - ds_own_rows(bw, c, [&](int j) { return gk[j * pitch + d + e]; });
        }
        uint32_t p3[3], q3[3];
        ds_split(p[0], p[1], p3);
        ds_split(q[0], q[1], q3);
        for (int m = 0; m < 3; ++m) {
          rec[m * 128 + at] = p3[m];
          rec[24 * DP + m * 128 + at] = q3[m];
        }
      }
      for (int col = warp * 16 + 8 * x + 2 * t4; col < Dv; col += 128)
        for (int e = 0; e < 2 && c < n && col + e < Dv; ++e) {
          const T* column = v + col + e;
          u0[c * row + col + e] = ds_own_rows(w, c, [&](int j) { return to_f32(column[j * row]); });
          out[c * row + col + e] = ds_own_rows(bw, c, [&](int j) { return to_f32(column[j * row]); });
        }
    }
}

// A block makes one record.  Loads; the pairs' sums A and B; then, side by side, the decayed keys and queries (warps 4 up, in
// place) and the 16 x 16 matrices W = (I + diag(beta) A)^(-1) diag(beta) and B W by substitution, a lane per column (warps 0
// and 1); then a warp makes 16 channels of P = W (G k) and Q = G q - (B W) (G k) and 16 value columns of U0 = W V and O0 =
// (B W) V on the tensor cores, whose accumulators are the fragments that the scan reads.  What bounds it is the number of its
// instructions (14 000 a block, issued in half of the cycles).
template <typename T, int DP>
__global__ void __launch_bounds__(256, 3)
delta_chunk_rows_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const T* __restrict__ vc,
                        const float* __restrict__ g, const float* __restrict__ beta, const int* __restrict__ cu_seqlens,
                        int num_seqs, uint32_t* __restrict__ records, float* __restrict__ u0, float* __restrict__ out,
                        int G, int H, int D, int Dv, int shortest) {
  constexpr int PITCH = DP + 4;  // tokens two apart lie 8 banks apart
  __shared__ __align__(16) float ks[DC_C][PITCH], qs[DC_C][PITCH], gs[DC_C][PITCH];  // later: keys to the end, G q, G k
  __shared__ __align__(16) float at[DC_C][DC_C], bt[DC_C][DC_C];                      // A and B, transposed
  __shared__ __align__(16) uint32_t tp[2][3 * 128];                                   // W and B W as left operands
  __shared__ float be[DC_C];
  pdl_wait();
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gr = lane >> 2, t4 = lane & 3;
  const int place = blockIdx.x, h = blockIdx.y, gh = h / (H / G);
  int n = 0;
  long t0 = 0;
  for (int b0 = 0; b0 < num_seqs; b0 += 32) {  // whose chunk this is, every warp for itself, 32 sequences at a time
    const int b = b0 + lane;
    int first = 0, left = 0;
    bool found = false;
    if (b < num_seqs) {
      const int c0 = cu_seqlens[b], c1 = cu_seqlens[b + 1], base = c0 / DC_C + b;
      found = place >= base && place < c1 / DC_C + b + 1;
      first = c0 + (place - base) * DC_C;
      left = c1 - c0 < shortest ? 0 : min(c1 - first, DC_C);
    }
    const uint32_t who = __ballot_sync(0xffffffffu, found);
    if (who) {
      t0 = __shfl_sync(0xffffffffu, first, __ffs(who) - 1);
      n = __shfl_sync(0xffffffffu, left, __ffs(who) - 1);
      break;
    }
  }
  if (n <= 0) return;
  // (whole 16 bytes where rows are made of them)
  const bool vec = D % 4 == 0 && (((uintptr_t)qn | (uintptr_t)kn | (uintptr_t)g) & 15) == 0;
#pragma unroll
  for (int x = tid * 4; x < DC_C * DP; x += 1024) {
    const int c = x / DP, i = x - c * DP;
    const long gi = ((t0 + c) * G + gh) * D + i, hi = ((t0 + c) * H + h) * D + i;
    const bool live = c < n && i < D;
    if (live && vec) {
      ds_copy16(&ks[c][i], kn + gi);
      ds_copy16(&qs[c][i], qn + gi);
      ds_copy16(&gs[c][i], g + hi);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const bool in = live && i + e < D;
        ks[c][i + e] = in ? kn[gi + e] : 0.f;
        qs[c][i + e] = in ? qn[gi + e] : 0.f;
        gs[c][i + e] = in ? g[hi + e] : 1.f;
      }
    }
  }
  if (tid < DC_C) be[tid] = tid < n ? beta[(t0 + tid) * H + h] : 0.f;
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  // this lane's values of the first 128 columns: tokens 2 t4, 2 t4 + 1, 2 t4 + 8, 2 t4 + 9 of columns 16 warp + gr (+ 8)
  T vr[2][4];
  auto values = [&](int col) {
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int c = 2 * t4 + (x & 1) + 4 * (x & 2);
      const T* src = vc + ((t0 + c) * H + h) * Dv + col;
      vr[0][x] = c < n && col < Dv ? src[0] : from_f32<T>(0.f);
      vr[1][x] = c < n && col + 8 < Dv ? src[8] : from_f32<T>(0.f);
    }
  };
  values(warp * 16 + gr);
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  {  // rows 15 - warp and warp of A and B, 17 pairs of tokens for every warp; the lanes share the channels
    constexpr int E = DP / 32;
    float v[48];  // row 15 - warp: A_ij, then B_ij, by i - j; row warp: the same
    auto row = [&](const float* from, float(&to)[E]) {
      if constexpr (E == 4) {
        const float4 x = *reinterpret_cast<const float4*>(from + lane * 4);
        to[0] = x.x; to[1] = x.y; to[2] = x.z; to[3] = x.w;
      } else {
        const float2 x = *reinterpret_cast<const float2*>(from + lane * 2);
        to[0] = x.x; to[1] = x.y;
      }
    };
    auto pairs = [&](int i, int most, int at_a, int at_b) {
      float wk[E], wq[E];
      row(ks[i], wk);
      row(qs[i], wq);
#pragma unroll
      for (int r = 0; r < most; ++r) {
        float a = 0.f, b = 0.f;
        if (r <= i) {
          float kj[E], gj[E];
          row(ks[i - r], kj);
          row(gs[i - r], gj);
#pragma unroll
          for (int e = 0; e < E; ++e) {
            a = fmaf(wk[e], kj[e], a);
            b = fmaf(wq[e], kj[e], b);
            wk[e] *= gj[e];
            wq[e] *= gj[e];
          }
        }
        v[at_a + r] = a;  // (A's diagonal is not used)
        v[at_b + r] = b;
      }
    };
    pairs(DC_C - 1 - warp, 16, 0, 16);
    pairs(warp, 8, 32, 40);
    // the sums over the lanes: a lane gives half of its values away at each step and has three of them in the end
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int half = 24 >> s;
      const bool up = (lane >> s) & 1;
#pragma unroll
      for (int x = 0; x < half; ++x) {
        const float give = up ? v[x] : v[x + half];
        v[x] = (up ? v[x + half] : v[x]) + __shfl_xor_sync(0xffffffffu, give, 1 << s);
      }
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) v[x] += __shfl_xor_sync(0xffffffffu, v[x], 16);
    if (lane < 16) {
      const int first = (lane & 1) * 24 + (lane & 2) * 6 + (lane & 4) / 4 * 6 + (lane & 8) / 8 * 3;
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        const int at_v = first + x;
        const int i = at_v < 32 ? DC_C - 1 - warp : warp, r = at_v < 32 ? at_v & 15 : at_v & 7;
        const bool is_b = at_v < 32 ? at_v >= 16 : at_v >= 40;
        if (r <= i) (is_b ? bt : at)[i - r][i] = v[x];
      }
    }
  }
  __syncthreads();
  uint32_t* rec = records + ((long)place * H + h) * DC_REC(DP);
  if (warp < 2) {  // column c of W (warp 0) or of B W (warp 1), in two lanes
    const int c = lane & 15;
    float x[DC_C], y[DC_C];
#pragma unroll
    for (int i = 0; i < DC_C; ++i) x[i] = i == c ? 1.f : 0.f, y[i] = 0.f;
#pragma unroll
    for (int j = 0; j < DC_C; ++j) {
      x[j] *= be[j];
#pragma unroll
      for (int i4 = j / 4 * 4; i4 < DC_C; i4 += 4) {
        const float4 a4 = *reinterpret_cast<const float4*>(&at[j][i4]);
        const float4 b4 = *reinterpret_cast<const float4*>(&bt[j][i4]);
        const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          if (i4 + m > j) x[i4 + m] = fmaf(-av[m], x[j], x[i4 + m]);
          if (i4 + m >= j) y[i4 + m] = fmaf(bv[m], x[j], y[i4 + m]);
        }
      }
    }
    // a lane's rows are eight, and two lanes make pairs of columns: the even one those of even rows
    const int half = lane >> 4;
    const bool odd = c & 1;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      float r[2];
#pragma unroll
      for (int e = 0; e < 2; ++e)
        r[e] = warp ? (half ? y[2 * m + e + 8] : y[2 * m + e]) : (half ? x[2 * m + e + 8] : x[2 * m + e]);
      const float other = __shfl_xor_sync(0xffffffffu, odd ? r[0] : r[1], 1);
      uint32_t p[3];
      ds_split(odd ? other : r[0], odd ? r[1] : other, p);
#pragma unroll
      for (int i = 0; i < 3; ++i)
        tp[warp][i * 128 + ((2 * m + odd) * 4 + ((c & 7) >> 1)) * 4 + half + 2 * (c >> 3)] = p[i];
    }
  } else if (tid >= 128 && tid - 128 < DP) {  // decays from the chunk's start and to its end
    const int d = tid - 128;
    float run = 1.f, gd[DC_C], kd[DC_C];
#pragma unroll
    for (int i = 0; i < DC_C; ++i) {
      gd[i] = gs[i][d];
      kd[i] = ks[i][d];
      run *= gd[i];
      gs[i][d] = run * kd[i];
      qs[i][d] *= run;
    }
    rec[72 * DP + d] = __float_as_uint(run);
    run = 1.f;
#pragma unroll
    for (int i = DC_C - 1; i >= 0; --i) {
      ks[i][d] = run * kd[i];
      run *= gd[i];
    }
  }
  __syncthreads();
  uint32_t w3[3][4], bw3[3][4];
  ds_parts(w3, tp[0], lane);
  ds_parts(bw3, tp[1], lane);
  // becomes NaN where a right operand of this warp's is not finite (its first part tells)
  __nv_bfloat162 none = __floats2bfloat162_rn(0.f, 0.f);
  auto watch = [&](uint32_t first) {
    none = __hfma2(*reinterpret_cast<__nv_bfloat162*>(&first), __floats2bfloat162_rn(0.f, 0.f), none);
  };
  // tokens 2 t4, 2 t4 + 1, 2 t4 + 8, 2 t4 + 9 of channels 16 warp + gr (+ 8), in parts
  auto right = [&](const float(*from)[PITCH], uint32_t(&to)[3][4]) {
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float* f = &from[2 * t4 + 8 * (x & 1)][warp * 16 + gr + 4 * (x & 2)];
      uint32_t p[3];
      ds_split(f[0], f[PITCH], p);
#pragma unroll
      for (int m = 0; m < 3; ++m) to[m][x] = p[m];
    }
  };
  auto store = [&](uint32_t* to, const uint32_t (&p)[3][4]) {
#pragma unroll
    for (int m = 0; m < 3; ++m)
      *reinterpret_cast<uint4*>(to + m * 128 + lane * 4) = make_uint4(p[m][0], p[m][1], p[m][2], p[m][3]);
  };
  if (warp < DP / 16) {
    uint32_t gk[3][4];
    float acc[2][4];
    // accumulators (rows gr, gr + 8; channels 2 t4, 2 t4 + 1 of two tiles) as two tiles of eight rows of the scan's right operand
    auto record = [&](uint32_t* to) {
      uint32_t r[3][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          uint32_t p[3];
          ds_split(acc[x][2 * i], acc[x][2 * i + 1], p);
#pragma unroll
          for (int m = 0; m < 3; ++m) r[m][2 * i + x] = p[m];
        }
      store(to + warp * 384, r);
    };
    right(gs, gk);
#pragma unroll
    for (int x = 0; x < 4; ++x) watch(gk[0][x]);
    ds_products(acc, w3, gk);
    record(rec);
    ds_products(acc, bw3, gk);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const float2 q = *reinterpret_cast<const float2*>(&qs[gr + 8 * i][warp * 16 + 8 * x + 2 * t4]);
        acc[x][2 * i] = q.x - acc[x][2 * i];
        acc[x][2 * i + 1] = q.y - acc[x][2 * i + 1];
      }
    record(rec + 24 * DP);
    right(ks, gk);
    store(rec + 48 * DP + warp * 384, gk);
  }
  for (int col = warp * 16; col < Dv; col += 128) {
    if (col >= 128) values(col + gr);
    uint32_t v3[3][4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      uint32_t p[3];
      ds_split(to_f32(vr[x >> 1][2 * (x & 1)]), to_f32(vr[x >> 1][2 * (x & 1) + 1]), p);
      watch(p[0]);
#pragma unroll
      for (int m = 0; m < 3; ++m) v3[m][x] = p[m];
    }
    auto rows_out = [&](float* to, const uint32_t (&left)[3][4]) {
      float acc[2][4];
      ds_products<sizeof(T) == 2>(acc, left, v3);
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int c = gr + 4 * (j & 2), i = col + 8 * x + 2 * t4 + (j & 1);
          if (c < n && i < Dv) to[((t0 + c) * H + h) * Dv + i] = acc[x][j];
        }
    };
    rows_out(u0, w3);
    rows_out(out, bw3);
  }
  if (__any_sync(0xffffffffu, __hisnan(none.x) || __hisnan(none.y)))
    delta_own_rows<T, DP>(rec, tp[0], tp[1], gs[0], qs[0], PITCH, vc + (t0 * H + h) * Dv, u0 + (t0 * H + h) * Dv,
                          out + (t0 * H + h) * Dv, (long)H * Dv, n, Dv);
}

// The state is held transposed, as the accumulators of its update (rows: the 16 value columns; columns: a warp's 16
// channels), which is also the layout of the left operand of the products with it.  Half of the warps are the chain: P S
// (the warps' parts are added through shared memory), U, the update, two barriers a chunk.  The other half fetches the
// records and makes O from the state's parts, which the chain leaves in shared memory, while the chain goes on.  What bounds
// it is the chain's latency, 1.0 us a chunk (products 0.2, shared memory two thirds busy).  `out` holds O0.
template <int DP>
__global__ void __launch_bounds__(4 * DP, 2)
delta_chunk_scan_kernel(const float* __restrict__ records, const float* __restrict__ u0, float* __restrict__ state,
                        const int* __restrict__ cu_seqlens, const int* __restrict__ state_slots, float* out, int num_seqs,
                        int H, int D, int Dv, int shortest) {
  constexpr int VT = 16, REC = DC_REC(DP), NT = 4 * DP, WARPS = DP / 16;
  extern __shared__ __align__(16) uint32_t dc_smem[];                    // two records, then
  float2* part = reinterpret_cast<float2*>(dc_smem + 2 * REC);           // [P, Q][WARPS][2 tiles][2 column halves][32]
  uint32_t* ss = reinterpret_cast<uint32_t*>(part + 2 * WARPS * 128);    // the state's parts: [WARPS][3][32][4]
  uint32_t* us = ss + WARPS * 384;                                       // U's: [3][32][4]
  pdl_wait();
  pdl_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const bool chain = tid < NT / 2;
  const int wtid = chain ? tid : tid - NT / 2, warp = wtid >> 5;
  const int h = blockIdx.y, col0 = blockIdx.x * VT;
  int b = blockIdx.z;
  if (shortest > 1) {  // the blockIdx.z-th sequence of at least that many tokens
    int before = 0;
    b = -1;
    for (int b0 = 0; b0 < num_seqs && b < 0; b0 += 32) {
      const bool in = b0 + lane < num_seqs && cu_seqlens[b0 + lane + 1] - cu_seqlens[b0 + lane] >= shortest;
      const uint32_t found = __ballot_sync(0xffffffffu, in);
      if (before + __popc(found) > (int)blockIdx.z) b = b0 + (int)__fns(found, 0, (int)blockIdx.z - before + 1);
      before += __popc(found);
    }
    if (b < 0) return;
  }
  const int t0 = cu_seqlens[b], t1 = cu_seqlens[b + 1];
  if (t1 <= t0) return;
  const int chunks = (t1 - t0 + DC_C - 1) / DC_C;
  // A thread's sums (the first four warps of a half): tile of eight rows, half of the columns, lane of the fragment: two tokens
  // of a column.
  const int o_col = col0 + ((wtid & 31) >> 2) + ((wtid >> 2) & 8), o_tok = ((wtid >> 3) & 8) + 2 * (wtid & 3);
  const bool sums = wtid < 128 && o_col < Dv;
  float x_next = 0.f, y_next = 0.f;
  auto base_value = [&](const float* rows, int c) {
    const int t = t0 + c * DC_C + o_tok;
    const float* p = rows + ((long)t * H + h) * Dv + o_col;
    x_next = sums && t < t1 ? p[0] : 0.f;
    y_next = sums && t + 1 < t1 ? p[(long)H * Dv] : 0.f;
  };
  auto sum_parts = [&](const float2* from) {
    float2 s = from[wtid];
#pragma unroll
    for (int w = 1; w < WARPS; ++w) {
      const float2 p = from[w * 128 + wtid];
      s.x += p.x;
      s.y += p.y;
    }
    return s;
  };
  auto write_part = [&](float2* to, const float(&acc)[2][4]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      to[warp * 128 + i * 64 + lane] = make_float2(acc[i][0], acc[i][1]);
      to[warp * 128 + i * 64 + 32 + lane] = make_float2(acc[i][2], acc[i][3]);
    }
  };
  if (!chain) {
    // P is needed a barrier before the rest of its record: its next one is asked for as soon as the last one has been read
    const uint32_t* rec0 = reinterpret_cast<const uint32_t*>(records) + ((long)(t0 / DC_C + b) * H + h) * REC;
    auto load = [&](int c, int what) {  // what: 1 for P, 2 for the rest
      if (c < chunks) {
        const uint32_t* src = rec0 + (long)c * H * REC + wtid * 4;
        uint32_t* dst = dc_smem + (c & 1) * REC + wtid * 4;
        if (what & 1) {
#pragma unroll
          for (int x = 0; x < 3; ++x) ds_copy16(dst + x * 2 * NT, src + x * 2 * NT);  // 24 DP words
        }
        if (what & 2) {
#pragma unroll
          for (int x = 3; x < 9; ++x) ds_copy16(dst + x * 2 * NT, src + x * 2 * NT);
          if (wtid < DP / 4) ds_copy16(dst + 18 * NT, src + 18 * NT);
        }
      }
    };
    load(0, 3);
    load(1, 1);
    asm volatile("cp.async.commit_group;\n" ::);
    base_value(out, 0);
    asm volatile("cp.async.wait_group 0;\n" ::);
    asm volatile("bar.sync 2, %0;" ::"n"(NT) : "memory");  // the first record is there
    for (int c = 0; c < chunks; ++c) {
      asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");  // the state's parts are there; P and the last record have been read
      asm volatile("cp.async.wait_group 0;\n" ::);
      load(c + 1, 2);
      load(c + 2, 1);
      asm volatile("cp.async.commit_group;\n" ::);
      uint32_t a[3][4], q[3][4];
      ds_parts(a, ss + warp * 384, lane);
      asm volatile("bar.sync 3, %0;" ::"n"(NT / 2) : "memory");  // everyone's copies of the group before have arrived
      asm volatile("bar.arrive 2, %0;" ::"n"(NT) : "memory");  // the next P is there, the state's parts are read
      ds_parts(q, dc_smem + (c & 1) * REC + 24 * DP + warp * 384, lane);
      float acc[2][4];
      ds_products(acc, a, q);
      write_part(part + WARPS * 128, acc);
      asm volatile("bar.sync 3, %0;" ::"n"(NT / 2) : "memory");
      if (wtid < 128) {
        const float2 s = sum_parts(part + WARPS * 128);
        const int t = t0 + c * DC_C + o_tok;
        float* p = out + ((long)t * H + h) * Dv + o_col;
        if (sums && t < t1) p[0] = x_next + s.x;
        if (sums && t + 1 < t1) p[(long)H * Dv] = y_next + s.y;
        base_value(out, c + 1);
      }
    }
    return;
  }
  float* Sg = state + ((long)state_slots[b] * H + h) * (long)D * Dv;
  float S[2][4];  // channel 16 warp + 8 i + 2 t4 + (j & 1), value column g + 8 (j >> 1)
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int d = warp * 16 + 8 * i + 2 * t4 + (j & 1), col = col0 + g + 8 * (j >> 1);
      S[i][j] = d < D && col < Dv ? Sg[(long)d * Dv + col] : 0.f;
    }
  base_value(u0, 0);
  auto state_product = [&](const uint32_t* rec) {
    uint32_t a[3][4], p[3][4];
    ds_parts(p, rec + warp * 384, lane);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t w[3];
      ds_split(S[i >> 1][2 * (i & 1)], S[i >> 1][2 * (i & 1) + 1], w);
#pragma unroll
      for (int m = 0; m < 3; ++m) a[m][i] = w[m];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
      *reinterpret_cast<uint4*>(ss + warp * 384 + i * 128 + lane * 4) = make_uint4(a[i][0], a[i][1], a[i][2], a[i][3]);
    float acc[2][4];
    ds_products(acc, a, p);
    write_part(part, acc);
  };
  asm volatile("bar.sync 2, %0;" ::"n"(NT) : "memory");
  state_product(dc_smem);
  for (int c = 0; c < chunks; ++c) {
    asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
    if (wtid < 128) {
      const float2 s = sum_parts(part);
      uint32_t p[3];
      ds_split(x_next - s.x, y_next - s.y, p);
#pragma unroll
      for (int i = 0; i < 3; ++i) us[i * 128 + (wtid & 31) * 4 + (wtid >> 5)] = p[i];
      base_value(u0, c + 1);
    }
    asm volatile("bar.sync 2, %0;" ::"n"(NT) : "memory");
    const uint32_t* rec = dc_smem + (c & 1) * REC;
    uint32_t a[3][4], k[3][4];
    ds_parts(k, rec + 48 * DP + warp * 384, lane);
    ds_parts(a, us, lane);
    float acc[2][4];
    ds_products(acc, a, k);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float2 gl = *reinterpret_cast<const float2*>(rec + 72 * DP + warp * 16 + 8 * i + 2 * t4);
#pragma unroll
      for (int j = 0; j < 4; ++j) S[i][j] = fmaf(j & 1 ? gl.y : gl.x, S[i][j], acc[i][j]);
    }
    state_product(dc_smem + ((c + 1) & 1) * REC);  // (behind the last chunk: nobody reads what this makes)
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int d = warp * 16 + 8 * i + 2 * t4 + (j & 1), col = col0 + g + 8 * (j >> 1);
      if (d < D && col < Dv) Sg[(long)d * Dv + col] = S[i][j];
    }
}

template <typename T, int DP>
static int launch_delta_chunks(cudaStream_t stream, int num_tokens, int num_seqs, int num_long, const float* qn, const float* kn,
                               const void* vc, const float* g, const float* beta, float* records, float* u0, float* state,
                               const int* cu_seqlens, const int* state_slots, float* out, int G, int H, int D, int Dv) {
  const int places = num_tokens / DC_C + num_seqs;
  const int shortest = num_long < num_seqs ? 2 : 1;
  constexpr size_t smem = sizeof(float) * (2 * DC_REC(DP) + DP * 32 + DP * 24 + 3 * 128);
  auto rows = delta_chunk_rows_kernel<T, DP>;
  auto scan = delta_chunk_scan_kernel<DP>;
  static bool configured_on[Q3_MAX_DEVICES];
  bool& configured = configured_on[q3_current_device()];
  if (!configured) {
    if (cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return Q3_ERR_LAUNCH;
    configured = true;
  }
  if (launch_pdl(rows, dim3(places, H), dim3(256), 0, stream, qn, kn, (const T*)vc, g, beta, cu_seqlens, num_seqs,
                 reinterpret_cast<uint32_t*>(records), u0, out, G, H, D, Dv, shortest) != cudaSuccess)
    return Q3_ERR_LAUNCH;
  // Not as a dependent launch: its blocks would start between the last blocks of the kernel before, two of the longest
  // sequence's on some SMs while others have none.  No block for a one-token sequence either where num_long says so: with
  // more blocks than SMs the first ones are no longer dealt out one to an SM (128 long blocks and 512 others: six SMs got two
  // long ones).
  scan<<<dim3((Dv + 15) / 16, H, num_long), dim3(4 * DP), smem, stream>>>(records, u0, state, cu_seqlens, state_slots, out,
                                                                      num_seqs, H, D, Dv, shortest);
  return q3_launch_status();
}

// The same as q3_delta_scan for key sizes up to 128, in chunks.  num_long: num_seqs, or the number of sequences of two tokens
// and more, which are then the only ones served; records: (num_tokens / 16 + num_seqs) * H * 73 * DP
// words with DP = 64 (D <= 64) or 128; u0: scratch of the output's size.
Q3_EXPORT int q3_delta_chunk_scan(int dtype, const float* qn, const float* kn, const void* vc, const float* g,
                                  const float* beta, float* records, float* u0, float* state,
                                  const int* cu_seqlens, const int* state_slots, float* out, int num_tokens, int num_seqs, int num_long, int G,
                                  int H, int D, int Dv, cudaStream_t stream) {
  if (!qn || !kn || !vc || !g || !beta || !records || !u0 || !state || !cu_seqlens || !state_slots || !out) return Q3_ERR_ARGUMENT;
  if (G < 1 || H < 1 || H % G || D < 1 || Dv < 1 || H > 65535 || num_seqs > 65535 || num_long > num_seqs) return Q3_ERR_ARGUMENT;
  if (D > 128 || (dtype != Q3_DTYPE_F32 && dtype != Q3_DTYPE_BF16) || !ds_aligned(records)) return Q3_ERR_UNSUPPORTED;
  if (num_long < 1 || num_tokens == 0) return Q3_OK;
#define Q3_DELTA_CHUNKS(T, DP)                                                                                       \
  return launch_delta_chunks<T, DP>(stream, num_tokens, num_seqs, num_long, qn, kn, vc, g, beta, records, u0, state,   \
                                    cu_seqlens, state_slots, out, G, H, D, Dv)
  if (dtype == Q3_DTYPE_F32) {
    if (D <= 64) Q3_DELTA_CHUNKS(float, 64);
    Q3_DELTA_CHUNKS(float, 128);
  }
  if (D <= 64) Q3_DELTA_CHUNKS(bf16, 64);
  Q3_DELTA_CHUNKS(bf16, 128);
#undef Q3_DELTA_CHUNKS
}

// ---- steps in which every sequence brings one token, in one kernel ------------------------------------
// One block per (head, sequence).  The head's state is fetched into registers before the projection it waits for is
// finished; then the block convolves its q, k and v channels (and writes the token's inputs into the ring), makes the
// decays and the output gate from the low-rank products' first halves, updates the state, norms and gates the head's
// output.  A thread holds up to 32 key rows of one value column; the NT / DVP row groups of a column meet in shared
// memory.  DVP: the value size rounded up to a power of two (32 at least).
template <typename T>
__global__ void __launch_bounds__(512)
delta_step_kernel(const T* __restrict__ x, long x_stride, const float* __restrict__ w, int taps, float* ring,
                  const int* __restrict__ positions, const int* __restrict__ cu_seqlens,
                  const int* __restrict__ state_slots, const T* __restrict__ low_a, const T* __restrict__ low_g,
                  const T* __restrict__ a2, int a_rank, const T* __restrict__ g2, int g_rank,
                  const float* __restrict__ dt_bias, const float* __restrict__ neg_a, const T* __restrict__ b,
                  float q_scale, float* state, const float* __restrict__ norm_w, float eps, T* __restrict__ out,
                  long out_stride, int G, int H, int D, int Dv, int dvp_shift) {
  extern __shared__ __align__(16) float st_smem[];
  const int NT = blockDim.x, tid = threadIdx.x, DVP = 1 << dvp_shift, RG = NT >> dvp_shift;
  const int RP = (((D + RG - 1) / RG) + 3) & ~3;  // rows of a thread: at most 32
  const int DP = (RP * RG + 3) & ~3;
  float* qs = st_smem;              // [DP] q, then k, then decays; zero beyond D
  float* ks = qs + DP;
  float* gs = ks + DP;
  float* vs = gs + DP;              // [Dv] values, then gates
  float* gate = vs + ((Dv + 3) & ~3);
  float* la = gate + ((Dv + 3) & ~3);  // low-rank rows
  float* lg = la + ((a_rank + 3) & ~3);
  float* part = lg + ((g_rank + 3) & ~3);  // [2][RG][DVP]
  __shared__ float red[33], sums[3];
  const int h = blockIdx.x, seq = blockIdx.y, rep = H / G, gh = h / rep;
  const int j = tid & (DVP - 1), rg = tid >> dvp_shift, i0 = rg * RP;
  const int slot = state_slots[seq];
  float* Sg = state + ((long)slot * H + h) * (long)D * Dv;
  float S[32];
#pragma unroll
  for (int r = 0; r < 32; ++r) S[r] = (r < RP && i0 + r < D && j < Dv) ? Sg[(long)(i0 + r) * Dv + j] : 0.f;
  pdl_wait();
  pdl_launch_dependents();
  const int t = cu_seqlens[seq], p = positions[t];
  const T* xrow = x + (long)t * x_stride;
  const int C = 2 * G * D + H * Dv;
  float* rows = taps > 1 ? ring + (long)slot * taps * C : nullptr;
  for (int c = tid; c < a_rank; c += NT) la[c] = to_f32(low_a[(long)t * x_stride + c]);
  for (int c = tid; c < g_rank; c += NT) lg[c] = to_f32(low_g[(long)t * x_stride + c]);
  for (int c = tid; c < 2 * D + Dv; c += NT) {
    const int ch = c < D ? gh * D + c : (c < 2 * D ? G * D + gh * D + c - D : 2 * G * D + h * Dv + c - 2 * D);
    float y[1];
    conv_silu<T, 1>(xrow, x_stride, w, taps, rows, C, 0, p, ch, y);
    (c < D ? qs[c] : (c < 2 * D ? ks[c - D] : vs[c - 2 * D])) = y[0];
    if (rows && (c >= 2 * D || h == gh * rep)) rows[(long)(p % taps) * C + ch] = to_f32(xrow[ch]);
  }
  for (int i = D + tid; i < DP; i += NT) qs[i] = ks[i] = gs[i] = 0.f;
  __syncthreads();
  // decays (outputs 0 .. D - 1) and gates (D ..): four lanes an output
  {
    const int lane4 = tid & 3;
    for (int o0 = 0; o0 < D + Dv; o0 += NT >> 2) {
      const int o = o0 + (tid >> 2);
      const bool live = o < D + Dv, is_a = o < D;
      const int rank = is_a ? a_rank : g_rank;
      const T* wr = live ? (is_a ? a2 + ((long)h * D + o) * a_rank : g2 + ((long)h * Dv + o - D) * g_rank) : a2;
      const float* lo = is_a ? la : lg;
      float acc = 0.f;
      if (live) {
        if ((rank & 7) == 0) {
          for (int r = lane4 * 8; r < rank; r += 32) {
            float v8[8];
            load8(wr + r, v8);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc = fmaf(v8[e], lo[r + e], acc);
          }
        } else {
          for (int r = lane4; r < rank; r += 4) acc = fmaf(to_f32(wr[r]), lo[r], acc);
        }
      }
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      if (live && lane4 == 0) {
        if (is_a) gs[o] = expf(neg_a[h] * softplus_f(acc + dt_bias[h * D + o]));
        else gate[o - D] = sigmoid_f(acc);
      }
    }
  }
  if (tid < 96) {  // |q|^2, |k|^2 and k . q, a warp each
    const float* p1 = tid < 32 ? qs : ks;
    const float* p2 = tid < 32 || tid >= 64 ? qs : ks;
    float acc = 0.f;
    for (int i = tid & 31; i < D; i += 32) acc = fmaf(p1[i], p2[i], acc);
    acc = warp_sum(acc);
    if ((tid & 31) == 0) sums[tid >> 5] = acc;
  }
  __syncthreads();
  const float inv_q = rsqrtf(sums[0] + UNIT_EPS) * q_scale, inv_k = rsqrtf(sums[1] + UNIT_EPS);
  const float kq = sums[2] * inv_q * inv_k;
  float sk = 0.f, sq = 0.f;
#pragma unroll
  for (int r = 0; r < 32; r += 4) {
    if (r < RP) {
      const float4 a = *reinterpret_cast<const float4*>(gs + i0 + r);
      const float4 k4 = *reinterpret_cast<const float4*>(ks + i0 + r);
      const float4 q4 = *reinterpret_cast<const float4*>(qs + i0 + r);
      S[r] *= a.x; S[r + 1] *= a.y; S[r + 2] *= a.z; S[r + 3] *= a.w;
      sk = fmaf(S[r], k4.x, sk); sq = fmaf(S[r], q4.x, sq);
      sk = fmaf(S[r + 1], k4.y, sk); sq = fmaf(S[r + 1], q4.y, sq);
      sk = fmaf(S[r + 2], k4.z, sk); sq = fmaf(S[r + 2], q4.z, sq);
      sk = fmaf(S[r + 3], k4.w, sk); sq = fmaf(S[r + 3], q4.w, sq);
    }
  }
  part[rg * DVP + j] = sk;
  part[(RG + rg) * DVP + j] = sq;
  __syncthreads();
  sk = sq = 0.f;
  for (int r = 0; r < RG; ++r) sk += part[r * DVP + j];
  const float beta = sigmoid_f(to_f32(b[(long)t * x_stride + h]));
  const float u = j < Dv ? beta * (vs[j] - sk * inv_k) : 0.f;
  const float uk = u * inv_k;
#pragma unroll
  for (int r = 0; r < 32; ++r)
    if (r < RP && i0 + r < D && j < Dv) Sg[(long)(i0 + r) * Dv + j] = fmaf(ks[i0 + r], uk, S[r]);
  float o = 0.f;
  if (rg == 0 && j < Dv) {
    for (int r = 0; r < RG; ++r) sq += part[(RG + r) * DVP + j];
    o = fmaf(u, kq, sq * inv_q);
  }
  const float rstd = rsqrtf(block_sum(o * o, red) / (float)Dv + eps);
  if (rg == 0 && j < Dv) out[(long)t * out_stride + (long)h * Dv + j] = from_f32<T>((o * rstd) * norm_w[j] * gate[j]);
}

// x, low_a, low_g and b are columns of one product: rows x_stride apart.  ring fp32 [slots, taps, C] (or null with one
// tap); a2 [H * D, a_rank], g2 [H * Dv, g_rank] of the activation type; norm_w fp32 [Dv]; out rows out_stride apart,
// head h at column h * Dv.  Value sizes up to 256 with D * (Dv rounded up to a power of two) at most 16384.
Q3_EXPORT int q3_delta_step(int dtype, const void* x, long x_stride, const float* w, int taps, float* ring,
                            const int* positions, const int* cu_seqlens, const int* state_slots, const void* low_a,
                            const void* low_g, const void* a2, int a_rank, const void* g2, int g_rank,
                            const float* dt_bias, const float* neg_a, const void* b, float q_scale, float* state,
                            const float* norm_w, float eps, void* out, long out_stride, int num_seqs, int G, int H, int D,
                            int Dv, cudaStream_t stream) {
  if (!x || !w || !positions || !cu_seqlens || !state_slots || !low_a || !low_g || !a2 || !g2 || !dt_bias || !neg_a || !b ||
      !state || !norm_w || !out)
    return Q3_ERR_ARGUMENT;
  if (G < 1 || H < 1 || H % G || D < 1 || Dv < 1 || taps < 1 || (taps > 1 && !ring) || a_rank < 1 || g_rank < 1)
    return Q3_ERR_ARGUMENT;
  int shift = 5;
  while ((1 << shift) < Dv) ++shift;
  const int DVP = 1 << shift;
  if (D > 256 || DVP > 256 || D * DVP > 16384 || taps > DELTA_MAX_TAPS || num_seqs > 65535) return Q3_ERR_UNSUPPORTED;
  if (((a_rank & 7) == 0 && !ds_aligned(a2)) || ((g_rank & 7) == 0 && !ds_aligned(g2))) return Q3_ERR_UNSUPPORTED;
  if (num_seqs == 0) return Q3_OK;
  int NT = 128;
  while (NT < 512 && (long)NT * 32 < (long)D * DVP) NT <<= 1;
  if (NT < DVP) NT = DVP;
  const int RG = NT / DVP, RP = (((D + RG - 1) / RG) + 3) & ~3;
  if (RP > 32) return Q3_ERR_UNSUPPORTED;
  const size_t smem = sizeof(float) * (size_t)(3 * ((RP * RG + 3) & ~3) + 2 * ((Dv + 3) & ~3) + ((a_rank + 3) & ~3) +
                                               ((g_rank + 3) & ~3) + 2 * RG * DVP);
  if (smem > 48 * 1024) return Q3_ERR_UNSUPPORTED;
  cudaError_t e;
#define Q3_DELTA_STEP(T)                                                                                               e = launch_pdl(delta_step_kernel<T>, dim3(H, num_seqs), dim3(NT), smem, stream, (const T*)x, x_stride, w, taps, ring,                  positions, cu_seqlens, state_slots, (const T*)low_a, (const T*)low_g, (const T*)a2, a_rank,                          (const T*)g2, g_rank, dt_bias, neg_a, (const T*)b, q_scale, state, norm_w, eps, (T*)out, out_stride, G, H,                  D, Dv, shift)
  if (dtype == Q3_DTYPE_F32) Q3_DELTA_STEP(float);
  else if (dtype == Q3_DTYPE_BF16) Q3_DELTA_STEP(bf16);
  else return Q3_ERR_ARGUMENT;
#undef Q3_DELTA_STEP
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}
