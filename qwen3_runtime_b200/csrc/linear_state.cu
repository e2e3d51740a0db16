// Linear attention with a decayed matrix state per (sequence, head), kept in fp32 in a state slot:
//
//   S_t = diag(a_t) S_(t-1) + k_t v_t^T        o_t = S_t^T q_t        S: [D, Dv]
//
// a_t is a decay per key channel.  It comes either from logits, a_t[i] = sigmoid(z_t[i] + b[i])^(1 / tau)
// (gated linear attention), or is one constant per head (retention).  q and k may be rotated first
// (pairs (i, i + pairs) of a head turn by position * inv_freq[i]) and are multiplied by q_scale and
// k_scale; decays, angles, the state and the products with it are fp32, q, k, v and z arrive in the
// activation type.  Further forms of the same recurrence: the decay exp(-exp(z_t[i] + b[i])) per key
// channel (decay_mode 1); a decay and a factor on k given per (token, head) as fp32 numbers (gates worked
// out beforehand); a last value column whose value is 1 for every token (ones_col: the state then also
// carries the decayed sum of the keys, and o's last column is that sum times q); and a bonus u per key
// channel with which the present token counts while the state is read before its update,
//   o_t = (S_(t-1) + diag(u) k_t v_t^T)^T q_t        S_t = diag(a_t) S_(t-1) + k_t v_t^T.
//
// stabilised_gates: the gates of a matrix memory with exponential input and forget gates, kept in range
// by a running maximum m per (sequence, head) (fp32, in a state slot, 0 at the start):
//   li = cap tanh((zi + bi) / cap)   lf = logsigmoid(cap tanh((zf + bf) / cap))   m_t = max(lf + m_(t-1), li)
//   decay_t = exp(lf + m_(t-1) - m_t)        k_scale_t = exp(li - m_t)
//
// decayed_state_scan: one block per (32 value columns, head, sequence).  A thread owns eight key
// rows of one value column of the state and keeps them in registers from the sequence's first token
// of the step to its last; the row groups of a column are neighbouring lanes of one warp, so a
// token's output is a shuffle sum over them (a fixed tree) and warps never wait for one another
// inside a chunk.  Tokens come 16 at a time: while the threads run the updates of one chunk from
// shared memory (q, k and decay rows as fp32, already rotated and scaled), the next chunk's raw
// values are already on their way into registers; they are turned into fp32 rows in the other half
// of the double buffer afterwards.  A token's arithmetic does not depend on where the step's portion
// starts or ends, so the result has the same bits however a prompt is cut.
//
// Segments: the same recurrence for prompts in bfloat16.  The scan above is a chain over a sequence's tokens, 0.21 us each, with
// one block per (head, 16 columns): 2048 tokens of 16 heads took 430 us with the SMs mostly idle.  Here a sequence is cut
// into segments of `seg` tokens: (1) every segment but a sequence's last works out the state it would leave behind if it
// began with zeros, and the product of its decays; (2) the segments' first states follow one from another,
// S <- diag(product) S + left behind; (3) every segment runs from its first state and writes its outputs, a sequence's last
// one the slot.  All decays are at most one, so nothing grows, and every sum is fp32 as before.  Within a segment 16 tokens are
// one step of matrix products (below): token by token the two passes and the rows took 133 us for 2048 tokens of 16 heads of
// 64 x 128 and 229 for 128 x 128, in chunks 83 and 134.  When this is the faster scan, and with which `seg`, is worked out from
// the sequences' lengths (ops/cuda.py, decayed_scan_segment, chunk_segment).
//
// head_norm_gate: y[t, h, :] = o / sqrt(mean(o^2) + eps) * w * silu(g[t, h, :]) * out_scale, one warp
// per (token, head); w may be absent.
#include "common.cuh"
#include "split_mma.cuh"

#define SCAN_CT 16  // tokens per chunk

// SCAN_R key rows per thread, SCAN_VT value columns per block; RGP2: row groups per value column (a
// power of two, 4..32): the block holds RGP2 * SCAN_R >= D key rows.  Four rows a thread and 16
// columns a block (key sizes up to 128) make four times as many warps as eight and 32 do: a single
// prompt's scan is a chain of dependent steps whose latencies only other warps can fill.
template <typename T, int RGP2, int SCAN_R, int SCAN_VT, bool BONUS>
__global__ void __launch_bounds__(SCAN_VT * RGP2)
decayed_state_scan_kernel(const T* __restrict__ q, long q_stride, const T* __restrict__ k, long k_stride,
                          const T* __restrict__ v, long v_stride, const T* __restrict__ z, long z_stride,
                          const float* __restrict__ z_bias, float inv_tau, const float* __restrict__ head_decay,
                          const float* __restrict__ inv_freq, int rot_pairs, const int* __restrict__ positions,
                          float q_scale, float k_scale, float* __restrict__ state,
                          const int* __restrict__ cu_seqlens, const int* __restrict__ state_slots,
                          float* __restrict__ out, int H, int D, int Dv, int decay_mode,
                          const float* __restrict__ tok_decay, const float* __restrict__ tok_kscale, int ones_col,
                          const float* __restrict__ bonus) {
  constexpr int THREADS = SCAN_VT * RGP2, DP = RGP2 * SCAN_R, CPW = 32 / RGP2;  // columns per warp
  constexpr int EPT = SCAN_CT * DP / THREADS;                              // row elements per thread and chunk: 4
  constexpr int VPT = (SCAN_CT * SCAN_VT + THREADS - 1) / THREADS;         // value elements per thread and chunk
  extern __shared__ __align__(16) float scan_smem[];
  typedef float (*Rows)[SCAN_CT][DP];
  typedef float (*Vals)[SCAN_CT][SCAN_VT];
  Rows qs = reinterpret_cast<Rows>(scan_smem);                    // [2][CT][DP]
  Rows ks = reinterpret_cast<Rows>(scan_smem + 2 * SCAN_CT * DP);
  Rows as = reinterpret_cast<Rows>(scan_smem + 4 * SCAN_CT * DP);
  Vals vs = reinterpret_cast<Vals>(scan_smem + 6 * SCAN_CT * DP);  // [2][CT][VT]
  float (*os)[SCAN_VT] = reinterpret_cast<float (*)[SCAN_VT]>(scan_smem + 6 * SCAN_CT * DP + 2 * SCAN_CT * SCAN_VT);
  pdl_wait();
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rg = lane % RGP2, col = warp * CPW + lane / RGP2;
  const int h = blockIdx.y, b = blockIdx.z;
  const int j = blockIdx.x * SCAN_VT + col;
  const int t0 = cu_seqlens[b], t1 = cu_seqlens[b + 1];
  const long slot = state_slots[b];
  float* Sg = state + ((slot * H + h) * (long)D) * Dv;
  float S[SCAN_R];
#pragma unroll
  for (int r = 0; r < SCAN_R; ++r) {
    const int i = rg * SCAN_R + r;
    S[r] = (i < D && j < Dv) ? Sg[(long)i * Dv + j] : 0.f;
  }
  const float decay_h = head_decay ? head_decay[h] : 1.f;
  const int Dvin = Dv - ones_col;  // value columns that v brings; the column after them holds ones
  float U[SCAN_R];
#pragma unroll
  for (int r = 0; r < SCAN_R; ++r) {
    const int i = rg * SCAN_R + r;
    U[r] = (BONUS && i < D) ? bonus[h * D + i] : 0.f;
  }

  // what a thread fetches of a chunk: EPT elements of the q, k (and logit) rows, their rotation
  // partners, VPT values
  T qr[EPT], kr[EPT], zr[EPT], qo[EPT], ko[EPT], vr[VPT];
  auto fetch = [&](int c0) {
#pragma unroll
    for (int m = 0; m < EPT; ++m) {
      const int x = tid + m * THREADS, c = x / DP, i = x - c * DP;
      const long t = c0 + c;
      const bool live = t < t1 && i < D;
      qr[m] = live ? q[t * q_stride + h * D + i] : from_f32<T>(0.f);
      kr[m] = live ? k[t * k_stride + h * D + i] : from_f32<T>(0.f);
      zr[m] = (live && z) ? z[t * z_stride + h * D + i] : from_f32<T>(0.f);
      if (live && i < 2 * rot_pairs) {
        const int other = i < rot_pairs ? i + rot_pairs : i - rot_pairs;
        qo[m] = q[t * q_stride + h * D + other];
        ko[m] = k[t * k_stride + h * D + other];
      }
    }
#pragma unroll
    for (int m = 0; m < VPT; ++m) {
      const int x = tid + m * THREADS, c = x / SCAN_VT, jj = blockIdx.x * SCAN_VT + (x % SCAN_VT);
      const long t = c0 + c;
      vr[m] = (x < SCAN_CT * SCAN_VT && t < t1 && jj < Dvin) ? v[t * v_stride + h * Dvin + jj]
                                                            : from_f32<T>((t < t1 && jj < Dv) ? 1.f : 0.f);
    }
  };
  // turn what was fetched into the fp32 rows of buffer `buf`: rows beyond D and tokens beyond the
  // portion are zero (their state stays zero and adds nothing)
  auto stage = [&](int c0, int buf) {
#pragma unroll
    for (int m = 0; m < EPT; ++m) {
      const int x = tid + m * THREADS, c = x / DP, i = x - c * DP;
      const long t = c0 + c;
      float qv = 0.f, kv = 0.f, av = 0.f;
      if (t < t1 && i < D) {
        qv = to_f32(qr[m]);
        kv = to_f32(kr[m]);
        if (i < 2 * rot_pairs) {
          const int pair = i < rot_pairs ? i : i - rot_pairs;
          float sn, cs;
          sincosf((float)positions[t] * inv_freq[pair], &sn, &cs);
          const float qp = to_f32(qo[m]), kp = to_f32(ko[m]);
          // first of a pair: u cos - v sin; second: v cos + u sin
          qv = i < rot_pairs ? qv * cs - qp * sn : qv * cs + qp * sn;
          kv = i < rot_pairs ? kv * cs - kp * sn : kv * cs + kp * sn;
        }
        qv *= q_scale;
        kv *= k_scale;
        if (tok_kscale) kv *= tok_kscale[t * H + h];
        if (z) {
          const float zz = to_f32(zr[m]) + (z_bias ? z_bias[h * D + i] : 0.f);
          if (decay_mode == 1) {
            av = expf(-expf(zz));
          } else {
            const float log_sig = fminf(zz, 0.f) - log1pf(expf(-fabsf(zz)));
            av = expf(log_sig * inv_tau);
          }
        } else {
          av = tok_decay ? tok_decay[t * H + h] : decay_h;
        }
      }
      qs[buf][c][i] = qv;
      ks[buf][c][i] = kv;
      as[buf][c][i] = av;
    }
#pragma unroll
    for (int m = 0; m < VPT; ++m) {
      const int x = tid + m * THREADS;
      if (x < SCAN_CT * SCAN_VT) vs[buf][x / SCAN_VT][x % SCAN_VT] = to_f32(vr[m]);
    }
  };

  fetch(t0);
  stage(t0, 0);
  __syncthreads();
  int buf = 0;
  for (int c0 = t0; c0 < t1; c0 += SCAN_CT, buf ^= 1) {
    const int n = min(SCAN_CT, t1 - c0);
    const bool more = c0 + SCAN_CT < t1;
    if (more) fetch(c0 + SCAN_CT);  // in flight while this chunk is computed
    const int i0 = rg * SCAN_R;
    // one token's update of this thread's rows; returns its share of the token's output
    auto update = [&](int c) -> float {
      const float vj = vs[buf][c][col];
      const float4* a4 = reinterpret_cast<const float4*>(&as[buf][c][i0]);
      const float4* k4 = reinterpret_cast<const float4*>(&ks[buf][c][i0]);
      const float4* q4 = reinterpret_cast<const float4*>(&qs[buf][c][i0]);
      float acc0 = 0.f, acc1 = 0.f;
#pragma unroll
      for (int g = 0; g < SCAN_R / 4; ++g) {
        const float4 a = a4[g], kk = k4[g], qq = q4[g];
        if (BONUS) {  // the output reads the state before its update, the present token through the bonus
          const float p0 = kk.x * vj, p1 = kk.y * vj, p2 = kk.z * vj, p3 = kk.w * vj;
          acc0 = fmaf(fmaf(U[4 * g + 0], p0, S[4 * g + 0]), qq.x, acc0);
          acc1 = fmaf(fmaf(U[4 * g + 1], p1, S[4 * g + 1]), qq.y, acc1);
          acc0 = fmaf(fmaf(U[4 * g + 2], p2, S[4 * g + 2]), qq.z, acc0);
          acc1 = fmaf(fmaf(U[4 * g + 3], p3, S[4 * g + 3]), qq.w, acc1);
          S[4 * g + 0] = fmaf(a.x, S[4 * g + 0], p0);
          S[4 * g + 1] = fmaf(a.y, S[4 * g + 1], p1);
          S[4 * g + 2] = fmaf(a.z, S[4 * g + 2], p2);
          S[4 * g + 3] = fmaf(a.w, S[4 * g + 3], p3);
          continue;
        }
        S[4 * g + 0] = fmaf(a.x, S[4 * g + 0], kk.x * vj);
        S[4 * g + 1] = fmaf(a.y, S[4 * g + 1], kk.y * vj);
        S[4 * g + 2] = fmaf(a.z, S[4 * g + 2], kk.z * vj);
        S[4 * g + 3] = fmaf(a.w, S[4 * g + 3], kk.w * vj);
        acc0 = fmaf(S[4 * g + 0], qq.x, acc0);
        acc1 = fmaf(S[4 * g + 1], qq.y, acc1);
        acc0 = fmaf(S[4 * g + 2], qq.z, acc0);
        acc1 = fmaf(S[4 * g + 3], qq.w, acc1);
      }
      return acc0 + acc1;
    };
    int c = 0;
    for (; c + 4 <= n; c += 4) {  // four tokens' sums over the row groups side by side: their shuffles overlap
      float acc[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[u] = update(c + u);
#pragma unroll
      for (int o = 1; o < RGP2; o <<= 1) {
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], o);
      }
      if (rg == 0) {
#pragma unroll
        for (int u = 0; u < 4; ++u) os[c + u][col] = acc[u];
      }
    }
    for (; c < n; ++c) {
      float acc = update(c);
#pragma unroll
      for (int o = 1; o < RGP2; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (rg == 0) os[c][col] = acc;
    }
    __syncthreads();  // the chunk's outputs are complete; nobody reads this half of the buffers any more
    for (int x = tid; x < n * SCAN_VT; x += THREADS) {
      const int c = x / SCAN_VT, jj = blockIdx.x * SCAN_VT + (x % SCAN_VT);
      if (jj < Dv) out[((long)(c0 + c) * H + h) * Dv + jj] = os[c][x % SCAN_VT];
    }
    if (more) stage(c0 + SCAN_CT, buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < SCAN_R; ++r) {
    const int i = rg * SCAN_R + r;
    if (i < D && j < Dv) Sg[(long)i * Dv + j] = S[r];
  }
}

template <typename T, int RGP2, int SCAN_R, int SCAN_VT, bool BONUS>
static cudaError_t launch_scan(cudaStream_t stream, int num_seqs, const void* q, long q_stride, const void* k,
                               long k_stride, const void* v, long v_stride, const void* z, long z_stride,
                               const float* z_bias, float inv_tau, const float* head_decay, const float* inv_freq,
                               int rot_pairs, const int* positions, float q_scale, float k_scale, float* state,
                               const int* cu_seqlens, const int* state_slots, float* out, int H, int D, int Dv,
                               int decay_mode, const float* tok_decay, const float* tok_kscale, int ones_col,
                               const float* bonus) {
  constexpr size_t smem = (size_t)(6 * SCAN_CT * RGP2 * SCAN_R + 3 * SCAN_CT * SCAN_VT) * sizeof(float);
  auto kernel = decayed_state_scan_kernel<T, RGP2, SCAN_R, SCAN_VT, BONUS>;
  if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const dim3 grid((Dv + SCAN_VT - 1) / SCAN_VT, H, num_seqs);
  return launch_pdl(kernel, grid, dim3(SCAN_VT * RGP2), smem, stream, (const T*)q, q_stride,
                    (const T*)k, k_stride, (const T*)v, v_stride, (const T*)z, z_stride, z_bias, inv_tau, head_decay,
                    inv_freq, rot_pairs, positions, q_scale, k_scale, state, cu_seqlens, state_slots, out, H, D, Dv,
                    decay_mode, tok_decay, tok_kscale, ones_col, bonus);
}

// ---- the same in segments ------------------------------------------------------------------------------
struct ScanArgs {
  const void *q, *k, *v, *z;
  long q_stride, k_stride, v_stride, z_stride;
  const float* z_bias;
  float inv_tau;
  const float *head_decay, *inv_freq;
  int rot_pairs;
  const int* positions;
  float q_scale, k_scale;
  float* state;
  const int *cu_seqlens, *state_slots;
  float* out;
  int num_seqs, H, D, Dv, decay_mode;
  const float *tok_decay, *tok_kscale;
  int ones_col;
  const float* bonus;
  int seg;          // tokens per segment
  int lo, hi;       // the tokens that this launch runs: the others' sequences are empty or shorter
  float* ends;      // [segments, H, D, Dv]: what a segment leaves behind, then the segments' first states
  float* products;  // [segments, H, D]
};

// the first token of sequence b among this launch's (of num_seqs: their end)
__device__ __forceinline__ int first_token(const ScanArgs& a, int b) { return min(max(a.cu_seqlens[b], a.lo), a.hi); }
__device__ __forceinline__ int segments_of(const ScanArgs& a, int b) {
  return (first_token(a, b + 1) - first_token(a, b) + a.seg - 1) / a.seg;
}

// Channel i < D of a token's key (turned, scaled), decay and query (turned, scaled) of a head, from its raw values.
__device__ __forceinline__ void scan_element(const ScanArgs& a, long t, int h, int i, float& kv, float& av, float& qv, float zz) {
  if (i < 2 * a.rot_pairs) {
    const bf16 *q = (const bf16*)a.q + t * a.q_stride + h * a.D, *k = (const bf16*)a.k + t * a.k_stride + h * a.D;
    const bool front = i < a.rot_pairs;
    const int pair = front ? i : i - a.rot_pairs, other = front ? i + a.rot_pairs : pair;
    float sn, cs;
    sincosf((float)a.positions[t] * a.inv_freq[pair], &sn, &cs);
    const float qp = to_f32(q[other]), kp = to_f32(k[other]);
    qv = front ? qv * cs - qp * sn : qv * cs + qp * sn;
    kv = front ? kv * cs - kp * sn : kv * cs + kp * sn;
  }
  qv *= a.q_scale;
  kv *= a.k_scale;
  if (a.tok_kscale) kv *= a.tok_kscale[t * a.H + h];
  if (a.z) {
    av = a.decay_mode == 1 ? expf(-expf(zz)) : expf((fminf(zz, 0.f) - log1pf(expf(-fabsf(zz)))) * a.inv_tau);
  } else {
    av = a.tok_decay ? a.tok_decay[t * a.H + h] : a.head_decay[h];
  }
}

// The sequence that this block's segment (blockIdx.x) belongs to (-1: none), the number of that sequence's first segment and
// how many it has.  Every warp for itself, 32 sequences at a time.
__device__ __forceinline__ int segment_owner(const ScanArgs& a, int& first, int& count) {
  const int lane = threadIdx.x & 31;
  int at = 0;
  for (int b0 = 0; b0 < a.num_seqs; b0 += 32) {
    const int n = b0 + lane < a.num_seqs ? segments_of(a, b0 + lane) : 0;
    int sum = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += x;
    }
    const uint32_t beyond = __ballot_sync(0xffffffffu, at + sum > (int)blockIdx.x);
    if (beyond) {
      const int l = __ffs(beyond) - 1;
      count = __shfl_sync(0xffffffffu, n, l);
      first = at + __shfl_sync(0xffffffffu, sum, l) - count;
      return b0 + l;
    }
    at += __shfl_sync(0xffffffffu, sum, 31);
  }
  return -1;
}

// Step 2: one thread per element of the state; what the segments left behind becomes their first states.
__global__ void __launch_bounds__(256)
segment_join_kernel(const __grid_constant__ ScanArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  const int h = blockIdx.y, seq = blockIdx.z, D = a.D, Dv = a.Dv;
  const int x = blockIdx.x * 256 + threadIdx.x;
  const int count = segments_of(a, seq);
  if (count < 2) return;
  int first = 0;  // segments of the sequences before: a warp counts 32 of them at a time
  for (int b0 = 0; b0 < seq; b0 += 32) {
    int n = b0 + (int)(threadIdx.x & 31) < seq ? segments_of(a, b0 + (int)(threadIdx.x & 31)) : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    first += n;
  }
  if (x >= D * Dv) return;
  const int i = x / Dv;
  float S = a.state[((long)a.state_slots[seq] * a.H + h) * D * Dv + x];
  constexpr int AHEAD = 6;  // segments whose numbers are read together: the chain is one multiply-add a segment
  for (int m0 = 0; m0 < count; m0 += AHEAD) {
    float left[AHEAD], product[AHEAD];
#pragma unroll
    for (int e = 0; e < AHEAD; ++e) {
      const long at = ((long)(first + m0 + e) * a.H + h) * D;
      const bool live = m0 + e < count - 1;
      left[e] = live ? a.ends[at * Dv + x] : 0.f;
      product[e] = live ? a.products[at + i] : 0.f;
    }
#pragma unroll
    for (int e = 0; e < AHEAD; ++e) {
      if (m0 + e < count) a.ends[((long)(first + m0 + e) * a.H + h) * D * Dv + x] = S;
      S = fmaf(product[e], S, left[e]);
    }
  }
}

// ---- a segment in chunks of 16 tokens ------------------------------------------------------------------
// With G_i the product of a chunk's decays up to token i and S the state before the chunk, in matrices whose rows are the
// chunk's tokens:
//   B_ij = sum_d q_i k_j prod_(j < m <= i) a_m  (j <= i)      O = B V + (G q) S
//   S <- G_last S + sum_j (prod_(m > j) a_m k_j) v_j^T
// (with a bonus u, which reads the state before its update: prod_(j < m < i), G_(i - 1), and B_ii = sum_d q_i u k_i).  Only
// products of decays occur, never quotients, and nothing in the state's chain but one multiply-add per chunk depends on the chunk
// before.  The products run on mma.sync, fp32 operands in three bfloat16 parts (split_mma.cuh), values as they are; what is added
// to the state is summed from zero.
//
// scan_chunk_rows, a block per (chunk, head): a record of SC_REC words, namely B, G q and the keys decayed to the chunk's end as
// parts in the order of the scan's fragments, [3][32 lanes][4] for every 16 channels, G_last [DP], whether values are not finite;
// behind it the values in that order, 128 words for 16 columns.  Chunks of sequence b start at place first_token / 16 + b (tokens
// counted from this launch's first); tokens beyond a portion's end are k = q = v = 0, a = 1.  Bound by instructions (2.5 a cycle; the decays' exponentials, the pairs'
// sums): 38 us for 2048 tokens of 16 heads of 64 x 128, 30 with the loads' addresses worked out once and 8 blocks an SM.
// scan_chunk_states, a block per (segment, 32 value columns, head): the state transposed in registers as in delta_state.cu, a
// warp 16 channels; the warps' parts of (G q) S meet in shared memory, one barrier a chunk, and are added a chunk later.  The same
// prompt, us: 20 + 59 with values and B V read and written beside the records, 13 + 29 so (two stages, so that 4 blocks fit an
// SM; 11 + 35 with three).  What is left waits for shared memory and the MMAs' results.
#define SC_C 16
#define SC_TILES 2  // of 16 value columns, in a block
#define SC_STAGES 2
#define SC_REC(DP) (416 + (DP) * 49)  // a record before its values, whole lines of 128 bytes
#define SC_VALUES(Dv) (((Dv) + 16 * SC_TILES - 1) / (16 * SC_TILES) * SC_TILES * 128)

template <int DP>
__global__ void __launch_bounds__(2 * DP, 512 / DP)
scan_chunk_rows_kernel(const __grid_constant__ ScanArgs a, uint32_t* __restrict__ records) {
  constexpr int PITCH = DP + 4, WARPS = DP / 16, NT = 2 * DP, E = DP / 32;
  __shared__ __align__(16) float ks[SC_C][PITCH], qs[SC_C][PITCH], gs[SC_C][PITCH];  // later: keys to the end, G q
  __shared__ __align__(16) float bs[SC_C][SC_C + 4];                                  // B
  pdl_wait();
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gr = lane >> 2, t4 = lane & 3;
  const int place = blockIdx.x, h = blockIdx.y, H = a.H, Dv = a.Dv, Dvin = Dv - a.ones_col;
  int n = 0;
  long t0 = 0;
  for (int b0 = 0; b0 < a.num_seqs; b0 += 32) {  // whose chunk this is, every warp for itself, 32 sequences at a time
    const int b = b0 + lane;
    int first = 0, left = 0;
    bool found = false;
    if (b < a.num_seqs) {
      const int c0 = first_token(a, b), c1 = first_token(a, b + 1), base = (c0 - a.lo) / SC_C + b;
      found = place >= base && place < (c1 - a.lo) / SC_C + b + 1;
      first = c0 + (place - base) * SC_C;
      left = min(c1 - first, SC_C);
    }
    const uint32_t who = __ballot_sync(0xffffffffu, found);
    if (who) {
      t0 = __shfl_sync(0xffffffffu, first, __ffs(who) - 1);
      n = __shfl_sync(0xffffffffu, left, __ffs(who) - 1);
      break;
    }
  }
  if (n <= 0) return;
  {  // a thread one channel of every other token; all of its loads in flight together
    const int i = tid % DP, c0 = tid / DP;
    const long t = t0 + c0;
    const bf16 *q = (const bf16*)a.q + t * a.q_stride + h * a.D + i, *k = (const bf16*)a.k + t * a.k_stride + h * a.D + i;
    const bf16* z = (const bf16*)a.z + t * a.z_stride + h * a.D + i;
    const bool channel = i < a.D, logits = a.z && channel;
    float qv[8], kv[8], zv[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const bool live = channel && c0 + 2 * e < n;
      qv[e] = live ? to_f32(*q) : 0.f;
      kv[e] = live ? to_f32(*k) : 0.f;
      zv[e] = live && logits ? to_f32(*z) : 0.f;
      q += 2 * a.q_stride, k += 2 * a.k_stride, z += 2 * a.z_stride;
    }
    const float zb = logits && a.z_bias ? a.z_bias[h * a.D + i] : 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int c = c0 + 2 * e;
      float av = 1.f;
      if (channel && c < n) scan_element(a, t + 2 * e, h, i, kv[e], av, qv[e], zv[e] + zb);
      ks[c][i] = kv[e];
      gs[c][i] = av;
      qs[c][i] = qv[e];
    }
  }
  float bonus[E];
#pragma unroll
  for (int e = 0; e < E; ++e) bonus[e] = a.bonus && lane + 32 * e < a.D ? a.bonus[h * a.D + lane + 32 * e] : 0.f;
  __syncthreads();
  for (int w = warp; w < 8; w += WARPS) {  // rows 15 - w and w of B, 17 pairs of tokens; the lanes share the channels
    float v[24];  // row 15 - w by i - j, then row w
    auto pairs = [&](int i, int most, int at) {
      float wq[E], b = 0.f;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        wq[e] = qs[i][lane + 32 * e];
        b = fmaf(wq[e], a.bonus ? bonus[e] * ks[i][lane + 32 * e] : ks[i][lane + 32 * e], b);
        if (!a.bonus) wq[e] *= gs[i][lane + 32 * e];
      }
      v[at] = b;
#pragma unroll
      for (int r = 1; r < most; ++r) {
        b = 0.f;
        if (r <= i) {
#pragma unroll
          for (int e = 0; e < E; ++e) {
            b = fmaf(wq[e], ks[i - r][lane + 32 * e], b);
            wq[e] *= gs[i - r][lane + 32 * e];
          }
        }
        v[at + r] = b;
      }
    };
    pairs(SC_C - 1 - w, 16, 0);
    pairs(w, 8, 16);
    // the sums over the lanes: a lane gives half of its values away in each of three steps and has three of them in the end
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const int half = 12 >> s;
      const bool up = (lane >> s) & 1;
#pragma unroll
      for (int x = 0; x < half; ++x) {
        const float give = up ? v[x] : v[x + half];
        v[x] = (up ? v[x + half] : v[x]) + __shfl_xor_sync(0xffffffffu, give, 1 << s);
      }
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      v[x] += __shfl_xor_sync(0xffffffffu, v[x], 8);
      v[x] += __shfl_xor_sync(0xffffffffu, v[x], 16);
    }
    if (lane < 8) {
      const int first = (lane & 1) * 12 + (lane & 2) * 3 + (lane & 4) / 4 * 3;
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        const int at = first + x, i = at < 16 ? SC_C - 1 - w : w, r = at & (at < 16 ? 15 : 7);
        if (r <= i) bs[i][i - r] = v[x];
      }
    }
  }
  for (int x = tid; x < SC_C * SC_C; x += NT)
    if (x % SC_C > x / SC_C) bs[x / SC_C][x % SC_C] = 0.f;
  __syncthreads();
  uint32_t* rec = records + ((long)place * H + h) * (SC_REC(DP) + SC_VALUES(Dv));
  if (tid < DP) {  // decays from the chunk's start and to its end
    float run = 1.f, gd[SC_C];
#pragma unroll
    for (int i = 0; i < SC_C; ++i) {
      gd[i] = gs[i][tid];
      const float before = run;
      run *= gd[i];
      qs[i][tid] *= a.bonus ? before : run;
    }
    rec[384 + 48 * DP + tid] = __float_as_uint(run);
    run = 1.f;
#pragma unroll
    for (int i = SC_C - 1; i >= 0; --i) {
      ks[i][tid] *= run;
      run *= gd[i];
    }
  }
  __syncthreads();
  auto store = [&](uint32_t* to, const uint32_t (&w)[3][4]) {
#pragma unroll
    for (int m = 0; m < 3; ++m)
      *reinterpret_cast<uint4*>(to + m * 128 + lane * 4) = make_uint4(w[m][0], w[m][1], w[m][2], w[m][3]);
  };
  uint32_t w3[3][4];
  auto put = [&](int x, float lo, float hi) {
    uint32_t p[3];
    ds_split(lo, hi, p);
#pragma unroll
    for (int m = 0; m < 3; ++m) w3[m][x] = p[m];
  };
  if (warp == 0) {  // of tokens gr (+ 8), the weights of tokens 2 t4, 2 t4 + 1 (+ 8)
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float2 f = *reinterpret_cast<const float2*>(&bs[gr + 4 * (x & 2)][2 * t4 + 8 * (x & 1)]);
      put(x, f.x, f.y);
    }
    store(rec, w3);
  }
#pragma unroll
  for (int x = 0; x < 4; ++x) {  // tokens gr (+ 8) of channels 2 t4, 2 t4 + 1 (+ 8)
    const float2 f = *reinterpret_cast<const float2*>(&qs[gr + 4 * (x & 2)][warp * 16 + 2 * t4 + 8 * (x & 1)]);
    put(x, f.x, f.y);
  }
  store(rec + 384 + warp * 384, w3);
#pragma unroll
  for (int x = 0; x < 4; ++x) {  // tokens 2 t4, 2 t4 + 1 (+ 8) of channels gr (+ 8)
    const float* f = &ks[2 * t4 + 8 * (x & 1)][warp * 16 + gr + 4 * (x & 2)];
    put(x, f[0], f[PITCH]);
  }
  store(rec + 384 + 24 * DP + warp * 384, w3);
  const bf16 *v = (const bf16*)a.v + t0 * a.v_stride + h * Dvin, one = from_f32<bf16>(1.f), none = from_f32<bf16>(0.f);
  int odd = 0;  // values that are not finite
  for (int w = warp; w < SC_VALUES(Dv) / 128; w += WARPS) {  // transposed: columns gr (+ 8), tokens 2 t4, 2 t4 + 1 (+ 8)
    uint32_t word[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int c = 2 * t4 + 4 * (x & 2), j = 16 * w + gr + 8 * (x & 1);
      const bf16 beyond = j < Dv ? one : none;
      __nv_bfloat162 pair;
      pair.x = c >= n ? none : j < Dvin ? v[c * a.v_stride + j] : beyond;
      pair.y = c + 1 >= n ? none : j < Dvin ? v[(c + 1) * a.v_stride + j] : beyond;
      word[x] = *reinterpret_cast<uint32_t*>(&pair);
    }
    *reinterpret_cast<uint4*>(rec + SC_REC(DP) + w * 128 + lane * 4) = make_uint4(word[0], word[1], word[2], word[3]);
#pragma unroll
    for (int x = 0; x < 4; ++x) odd |= (word[x] & 0x7f80u) == 0x7f80u || (word[x] & 0x7f800000u) == 0x7f800000u;
  }
  odd = __syncthreads_or(odd);
  if (tid == 0) rec[384 + 49 * DP] = odd;
}

// The chunk's own share of an output (element x of a thread's eight, as ds_products orders them) where values are not finite: a
// weight of zero is no reason to touch an earlier token's output.  rec: the weights' parts; v: the column tile's values.
__device__ __noinline__ float own_token(const uint32_t* rec, const uint32_t* v, int x) {
  const int lane = threadIdx.x & 31, t = 8 * (x >> 2) + 2 * (lane & 3) + (x & 1), col = (lane >> 2) + 4 * (x & 2);
  float sum = 0.f;
  for (int j = 0; j <= t; ++j) {
    const int at = (((t & 7) * 4 + ((j & 7) >> 1)) << 2) + 2 * (t >> 3) + (j >> 3), shift = j & 1 ? 0 : 16;
    float w = 0.f;
    for (int m = 2; m >= 0; --m) w += __uint_as_float((rec[m * 128 + at] << shift) & 0xffff0000u);
    const uint32_t pair = v[(((col & 7) * 4 + ((j & 7) >> 1)) << 2) + 2 * (j >> 3) + (col >> 3)];
    sum = fmaf(w, __uint_as_float((pair << shift) & 0xffff0000u), sum);
  }
  return sum;
}

template <int DP, bool OUT>
__global__ void __launch_bounds__(2 * DP, DP == 64 ? 4 : 2)
scan_chunk_states_kernel(const __grid_constant__ ScanArgs a, const uint32_t* __restrict__ records) {
  constexpr int NC = SC_TILES, VT = 16 * NC, NT = 2 * DP, WARPS = DP / 16, PITCH = VT + 4, N = SC_C * VT / NT;
  constexpr int SKIP = OUT ? 0 : 384 + 24 * DP, HEAD = SC_REC(DP) - SKIP, REC = HEAD + NC * 128;  // what is read of a record
  constexpr int Q0 = 384, K0 = 384 + 24 * DP - SKIP, GL = K0 + 24 * DP;
  extern __shared__ __align__(16) uint32_t sc_smem[];                 // the records' ring, then
  float* part = reinterpret_cast<float*>(sc_smem + SC_STAGES * REC);  // [2][WARPS][SC_C][PITCH]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gr = lane >> 2, t4 = lane & 3;
  const int col0 = blockIdx.y * VT, h = blockIdx.z;
  const int H = a.H, D = a.D, Dv = a.Dv;
  int first, count;
  pdl_wait();
  pdl_launch_dependents();
  const int b = segment_owner(a, first, count);
  if (b < 0) return;
  const int mine = blockIdx.x - first;  // the segment's number in its sequence
  const bool last = mine == count - 1;
  if (!OUT && last) return;
  const int seq0 = first_token(a, b), t0 = seq0 + mine * a.seg, t1 = min(first_token(a, b + 1), t0 + a.seg);
  const int chunks = (t1 - t0 + SC_C - 1) / SC_C;
  const long rec_size = SC_REC(DP) + SC_VALUES(Dv);
  const uint32_t* rec0 = records + ((long)((seq0 - a.lo) / SC_C + b + mine * (a.seg / SC_C)) * H + h) * rec_size;
  auto load = [&](int c) {
    if (c < chunks) {
      const uint32_t* src = rec0 + (long)c * H * rec_size;
      uint32_t* dst = sc_smem + (c % SC_STAGES) * REC;
#pragma unroll
      for (int x = 0; x < (REC / 4 + NT - 1) / NT; ++x) {
        const int at = (tid + x * NT) * 4;
        if (at < REC) ds_copy16(dst + at, src + (at < HEAD ? SKIP + at : SC_REC(DP) + blockIdx.y * NC * 128 + at - HEAD));
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);  // also when empty: one group per call
  };
#pragma unroll
  for (int c = 0; c < SC_STAGES - 1; ++c) load(c);
  const long tile = ((long)blockIdx.x * H + h) * D;
  float* Sg = a.state + ((long)a.state_slots[b] * H + h) * (long)D * Dv;
  const float* from = count > 1 ? a.ends + tile * Dv : Sg;
  float S[NC][2][4], P[2][2];  // channel 16 warp + 8 i + 2 t4 + (j & 1), value column 16 w + gr + 8 (j >> 1)
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    P[i][0] = P[i][1] = 1.f;
#pragma unroll
    for (int w = 0; w < NC; ++w)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int d = warp * 16 + 8 * i + 2 * t4 + (j & 1), col = col0 + 16 * w + gr + 8 * (j >> 1);
        S[w][i][j] = OUT && d < D && col < Dv ? from[(long)d * Dv + col] : 0.f;
      }
  }
  const int o_tok = tid / (VT / N), o_col = tid % (VT / N) * N;  // this thread's outputs: N columns of a token
  const bool whole = Dv % N == 0;
  auto finish = [&](int c) {  // chunk c's outputs
    const float* from = part + ((c & 1) * WARPS * SC_C + o_tok) * PITCH + o_col;
    float sum[N];
#pragma unroll
    for (int w = 0; w < WARPS; ++w)
#pragma unroll
      for (int x = 0; x < N; x += 2) {
        const float2 f = *reinterpret_cast<const float2*>(from + w * SC_C * PITCH + x);
        sum[x] = w ? sum[x] + f.x : f.x;
        sum[x + 1] = w ? sum[x + 1] + f.y : f.y;
      }
    const int t = t0 + c * SC_C + o_tok, col = col0 + o_col;
    if (t >= t1) return;
    float* p = a.out + ((long)t * H + h) * Dv + col;
    if (whole && col < Dv) {
      if constexpr (N == 4) *reinterpret_cast<float4*>(p) = make_float4(sum[0], sum[1], sum[2], sum[3]);
      else *reinterpret_cast<float2*>(p) = make_float2(sum[0], sum[1]);
    } else {
#pragma unroll
      for (int x = 0; x < N; ++x)
        if (col + x < Dv) p[x] = sum[x];
    }
  };
  for (int c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(SC_STAGES - 2));
    __syncthreads();  // the record is there, the last one read; the parts of chunk c - 1 are there, those of c - 2 read
    load(c + SC_STAGES - 1);
    const uint32_t* rec = sc_smem + (c % SC_STAGES) * REC;
    uint32_t v3[NC][3][4], r[3][4];
#pragma unroll
    for (int w = 0; w < NC; ++w) {
      const uint4 word = *reinterpret_cast<const uint4*>(rec + HEAD + w * 128 + lane * 4);
      v3[w][0][0] = word.x, v3[w][0][1] = word.y, v3[w][0][2] = word.z, v3[w][0][3] = word.w;
#pragma unroll
      for (int x = 0; x < 4; ++x) v3[w][1][x] = v3[w][2][x] = 0u;
    }
    if (OUT) {
      ds_parts(r, rec + Q0 + warp * 384, lane);
#pragma unroll
      for (int w = 0; w < NC; ++w) {
        uint32_t s3[3][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t p[3];
          ds_split(S[w][i >> 1][2 * (i & 1)], S[w][i >> 1][2 * (i & 1) + 1], p);
#pragma unroll
          for (int m = 0; m < 3; ++m) s3[m][i] = p[m];
        }
        float acc[2][4];
        ds_products(acc, s3, r);
        if (warp == w) {  // this warp's share has the chunk's own tokens too
          uint32_t b3[3][4];
          float own[2][4];
          ds_parts(b3, rec, lane);
          ds_products<false, true>(own, v3[w], b3);
          if (rec[GL + DP]) {
#pragma unroll
            for (int x = 0; x < 8; ++x) own[x >> 2][x & 3] = own_token(rec, rec + HEAD + w * 128, x);
          }
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] += own[i][j];
        }
        float* to = part + (((c & 1) * WARPS + warp) * SC_C + 2 * t4) * PITCH + 16 * w + gr;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) to[(8 * i + (j & 1)) * PITCH + 8 * (j >> 1)] = acc[i][j];
      }
    }
    ds_parts(r, rec + K0 + warp * 384, lane);
    float2 gl[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      gl[i] = *reinterpret_cast<const float2*>(rec + GL + warp * 16 + 8 * i + 2 * t4);
      P[i][0] *= gl[i].x;
      P[i][1] *= gl[i].y;
    }
#pragma unroll
    for (int w = 0; w < NC; ++w) {
      float acc[2][4];
      ds_products<false, true>(acc, v3[w], r);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) S[w][i][j] = fmaf(j & 1 ? gl[i].y : gl[i].x, S[w][i][j], acc[i][j]);
    }
    if (OUT && c > 0) finish(c - 1);
  }
  if (OUT) {
    __syncthreads();
    finish(chunks - 1);
  }
  float* dst = OUT ? Sg : a.ends + tile * Dv;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int d0 = warp * 16 + 8 * i + 2 * t4;
    if (!OUT || last) {
#pragma unroll
      for (int w = 0; w < NC; ++w)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int d = d0 + (j & 1), col = col0 + 16 * w + gr + 8 * (j >> 1);
          if (d < D && col < Dv) dst[(long)d * Dv + col] = S[w][i][j];
        }
    }
    if (!OUT && blockIdx.y == 0 && gr == 0) {
      if (d0 < D) a.products[tile + d0] = P[i][0];
      if (d0 + 1 < D) a.products[tile + d0 + 1] = P[i][1];
    }
  }
}

template <int DP>
static cudaError_t launch_segments(const ScanArgs& a, int segments, bool cut, uint32_t* records, cudaStream_t stream) {
  constexpr size_t ends_smem = sizeof(uint32_t) * SC_STAGES * (25 * DP + 32 + SC_TILES * 128);
  constexpr size_t smem = sizeof(uint32_t) * (SC_STAGES * (SC_REC(DP) + SC_TILES * 128) + 2 * DP / 16 * SC_C * (16 * SC_TILES + 4));
  auto ends = scan_chunk_states_kernel<DP, false>, scan = scan_chunk_states_kernel<DP, true>;
  static bool configured_on[Q3_MAX_DEVICES];
  bool& configured = configured_on[q3_current_device()];
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(ends, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ends_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  const dim3 grid((unsigned)segments, (unsigned)((a.Dv + 16 * SC_TILES - 1) / (16 * SC_TILES)), (unsigned)a.H), block(2 * DP);
  cudaError_t e = launch_pdl(scan_chunk_rows_kernel<DP>, dim3((unsigned)((a.hi - a.lo) / SC_C + a.num_seqs), (unsigned)a.H),
                             dim3(2 * DP), 0, stream, a, records);
  if (e != cudaSuccess) return e;
  // Neither pass is a dependent launch: its blocks would start between those of the kernel before and crowd some SMs while others
  // stay empty (a prompt of 2048 tokens, 16 heads of 64 x 128, segments of 1024: the second pass 101 us).  Unless they are few and
  // short (16 prompts of 16 tokens, 4 heads of 32 x 32, lengths unknown: 20.4 us instead of 23.5).
  const bool dependent = cut && a.seg <= 64 && (long)grid.x * grid.y * grid.z <= 512;
  if (cut) {
    if (dependent) {
      e = launch_pdl(ends, grid, block, ends_smem, stream, a, (const uint32_t*)records);
    } else {
      ends<<<grid, block, ends_smem, stream>>>(a, records);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess)
      e = launch_pdl(segment_join_kernel, dim3((unsigned)((a.D * a.Dv + 255) / 256), (unsigned)a.H, (unsigned)a.num_seqs),
                     dim3(256), 0, stream, a);
    if (e != cudaSuccess) return e;
  }
  if (dependent) return launch_pdl(scan, grid, block, smem, stream, a, (const uint32_t*)records);
  scan<<<grid, block, smem, stream>>>(a, records);
  return cudaGetLastError();
}

// The same arguments as q3_decayed_state_scan, bfloat16, key sizes up to 128: tokens lo .. hi - 1 of the step in segments of `seg`
// tokens, a multiple of 16.  (A step whose records are too many runs in several calls over tokens one after another; a sequence's
// state carries over.  cu_seqlens and state_slots may start at the first sequence that has tokens in the call.)  segments: the number
// of them, sum over the sequences of ceil(tokens / seg), or more; cut: whether a sequence may have more than one; scratch: 32-bit
// words, 16-byte aligned, ((hi - lo) / 16 + num_seqs) * H * (416 + 49 * DP + 256 * ceil(Dv / 32)) with DP = 64 (D <= 64) or 128, and
// if cut segments * H * D * (Dv + 1) more.
Q3_EXPORT int q3_decayed_segment_scan(int dtype, const void* q, long q_stride, const void* k, long k_stride, const void* v,
                                      long v_stride, const void* z, long z_stride, const float* z_bias, float inv_tau,
                                      const float* head_decay, const float* inv_freq, int rot_pairs, const int* positions,
                                      float q_scale, float k_scale, float* state, const int* cu_seqlens,
                                      const int* state_slots, float* out, int num_seqs, int H, int D, int Dv,
                                      int decay_mode, const float* tok_decay, const float* tok_kscale, int ones_col,
                                      const float* bonus, int seg, int segments, int cut, float* scratch,
                                      int lo, int hi, cudaStream_t stream) {
  if (!q || !k || !v || !state || !cu_seqlens || !state_slots || !out || !scratch || seg < 1 || seg % SC_C || segments < 1 ||
      lo < 0 || hi < lo || ((uintptr_t)scratch & 15))
    return Q3_ERR_ARGUMENT;
  if (!z && !head_decay && !tok_decay) return Q3_ERR_ARGUMENT;
  if (decay_mode < 0 || decay_mode > 1 || ones_col < 0 || ones_col > 1 || Dv - ones_col < 1) return Q3_ERR_ARGUMENT;
  if (rot_pairs < 0 || 2 * rot_pairs > D || (rot_pairs && (!inv_freq || !positions))) return Q3_ERR_ARGUMENT;
  if (H < 1 || D < 1 || Dv < 1 || H > 65535 || num_seqs > 65535) return Q3_ERR_ARGUMENT;
  if (D > 128 || dtype != Q3_DTYPE_BF16) return Q3_ERR_UNSUPPORTED;
  if (num_seqs == 0 || hi == lo) return Q3_OK;
  const int DP = D <= 64 ? 64 : 128;
  float* ends = scratch + ((long)(hi - lo) / SC_C + num_seqs) * H * (SC_REC(DP) + SC_VALUES(Dv));
  uint32_t* records = reinterpret_cast<uint32_t*>(scratch);
  const ScanArgs a = {q, k, v, z, q_stride, k_stride, v_stride, z_stride, z_bias, inv_tau, head_decay, inv_freq, rot_pairs,
                      positions, q_scale, k_scale, state, cu_seqlens, state_slots, out, num_seqs, H, D, Dv, decay_mode,
                      tok_decay, tok_kscale, ones_col, bonus, seg, lo, hi, ends, ends + (long)segments * H * D * Dv};
  const cudaError_t e = DP == 64 ? launch_segments<64>(a, segments, cut, records, stream)
                                 : launch_segments<128>(a, segments, cut, records, stream);
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}

// q, k: head h of token t at [t * stride + h * D]; v at [t * v_stride + h * (Dv - ones_col)]; z (decay
// logits, or null) like q, z_bias fp32 [H * D] or null; decay_mode 0: exp(logsigmoid(z + b) * inv_tau), 1:
// exp(-exp(z + b)); head_decay fp32 [H] or tok_decay fp32 [T, H] (one of them when z is null); tok_kscale
// fp32 [T, H] or null; bonus fp32 [H * D] or null; inv_freq fp32 [rot_pairs] with positions, or
// rot_pairs = 0; state fp32 [slots, H, D, Dv]; out fp32 [T, H, Dv]; Dv counts the column of ones.
Q3_EXPORT int q3_decayed_state_scan(int dtype, const void* q, long q_stride, const void* k, long k_stride,
                                    const void* v, long v_stride, const void* z, long z_stride, const float* z_bias,
                                    float inv_tau, const float* head_decay, const float* inv_freq, int rot_pairs,
                                    const int* positions, float q_scale, float k_scale, float* state,
                                    const int* cu_seqlens, const int* state_slots, float* out, int num_seqs, int H,
                                    int D, int Dv, int decay_mode, const float* tok_decay, const float* tok_kscale,
                                    int ones_col, const float* bonus, cudaStream_t stream) {
  if (!q || !k || !v || !state || !cu_seqlens || !state_slots || !out) return Q3_ERR_ARGUMENT;
  if (!z && !head_decay && !tok_decay) return Q3_ERR_ARGUMENT;
  if (decay_mode < 0 || decay_mode > 1 || ones_col < 0 || ones_col > 1 || Dv - ones_col < 1) return Q3_ERR_ARGUMENT;
  if (rot_pairs < 0 || 2 * rot_pairs > D || (rot_pairs && (!inv_freq || !positions))) return Q3_ERR_ARGUMENT;
  if (H < 1 || D < 1 || Dv < 1 || H > 65535 || num_seqs > 65535) return Q3_ERR_ARGUMENT;
  if (D > 256 || (dtype != Q3_DTYPE_F32 && dtype != Q3_DTYPE_BF16)) return Q3_ERR_UNSUPPORTED;
  if (num_seqs == 0) return Q3_OK;
  cudaError_t e;
#define Q3_SCAN_B(T, RGP2, R, VT, B)                                                                                 \
  e = launch_scan<T, RGP2, R, VT, B>(stream, num_seqs, q, q_stride, k, k_stride, v, v_stride, z, z_stride, z_bias,   \
                                     inv_tau, head_decay, inv_freq, rot_pairs, positions, q_scale, k_scale, state,   \
                                     cu_seqlens, state_slots, out, H, D, Dv, decay_mode, tok_decay, tok_kscale,      \
                                     ones_col, bonus)
#define Q3_SCAN(T, RGP2, R, VT)                                                                                      \
  do { if (bonus) Q3_SCAN_B(T, RGP2, R, VT, true); else Q3_SCAN_B(T, RGP2, R, VT, false); } while (0)
#define Q3_SCAN_SIZES(T)                                                                                             \
  if (D <= 16) Q3_SCAN(T, 4, 4, 16); else if (D <= 32) Q3_SCAN(T, 8, 4, 16); else if (D <= 64) Q3_SCAN(T, 16, 4, 16); \
  else if (D <= 128) Q3_SCAN(T, 32, 4, 16); else Q3_SCAN(T, 32, 8, 32)
  if (dtype == Q3_DTYPE_F32) { Q3_SCAN_SIZES(float); } else { Q3_SCAN_SIZES(bf16); }
#undef Q3_SCAN_SIZES
#undef Q3_SCAN
#undef Q3_SCAN_B
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}

// ---- gates of a matrix memory with a running maximum ---------------------------------------------------
// One warp per (sequence, head), 32 tokens at a time: every lane works out its token's two log gates, the
// running maximum then goes through the 32 tokens in order (an add and a max per token, on values handed
// round by shuffles, so the chain is exactly the sequential one wherever a portion starts), and every
// lane turns its token's maximum and its predecessor's into the decay and the key factor.
template <typename T>
__global__ void stabilised_gates_kernel(const T* __restrict__ zi, const T* __restrict__ zf, long z_stride,
                                        const float* __restrict__ bi, const float* __restrict__ bf, float cap,
                                        float* __restrict__ m_state, const int* __restrict__ cu_seqlens,
                                        const int* __restrict__ state_slots, float* __restrict__ decay,
                                        float* __restrict__ kscale, float* __restrict__ m_run, int H, int pairs) {
  pdl_wait();
  pdl_launch_dependents();
  const int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (item >= pairs) return;
  const int b = item / H, h = item - b * H;
  const int t0 = cu_seqlens[b], t1 = cu_seqlens[b + 1];
  if (t1 <= t0) return;
  float* mslot = m_state + (long)state_slots[b] * H + h;
  float m = *mslot;
  const float bih = bi ? bi[h] : 0.f, bfh = bf ? bf[h] : 0.f, inv_cap = 1.f / cap;
  for (int c0 = t0; c0 < t1; c0 += 32) {
    const int t = c0 + lane, n = min(32, t1 - c0);
    float li = 0.f, lf = 0.f;
    if (t < t1) {
      li = cap * tanhf((to_f32(zi[t * z_stride + h]) + bih) * inv_cap);
      const float x = cap * tanhf((to_f32(zf[t * z_stride + h]) + bfh) * inv_cap);
      lf = fminf(x, 0.f) - log1pf(expf(-fabsf(x)));
    }
    float m_before = 0.f, m_after = 0.f;
    for (int s = 0; s < n; ++s) {
      const float lis = __shfl_sync(0xffffffffu, li, s), lfs = __shfl_sync(0xffffffffu, lf, s);
      const float next = fmaxf(lfs + m, lis);
      if (lane == s) { m_before = m; m_after = next; }
      m = next;
    }
    if (t < t1) {
      decay[(long)t * H + h] = expf(lf + m_before - m_after);
      kscale[(long)t * H + h] = expf(li - m_after);
      m_run[(long)t * H + h] = m_after;
    }
  }
  if (lane == 0) *mslot = m;
}

// zi, zf: [T, H] rows z_stride apart (the two gates' pre-activations); bi, bf: fp32 [H] or null; m_state:
// fp32 [slots, H]; decay, kscale, m_run: fp32 [T, H].
Q3_EXPORT int q3_stabilised_gates(int dtype, const void* zi, const void* zf, long z_stride, const float* bi,
                                  const float* bf, float cap, float* m_state, const int* cu_seqlens,
                                  const int* state_slots, float* decay, float* kscale, float* m_run, int num_seqs,
                                  int H, cudaStream_t stream) {
  if (!zi || !zf || !m_state || !cu_seqlens || !state_slots || !decay || !kscale || !m_run || H < 1 || !(cap > 0.f))
    return Q3_ERR_ARGUMENT;
  if (num_seqs == 0) return Q3_OK;
  const int pairs = num_seqs * H;
  const unsigned blocks = (unsigned)((pairs + 3) / 4);
  cudaError_t e;
  if (dtype == Q3_DTYPE_F32)
    e = launch_pdl(stabilised_gates_kernel<float>, dim3(blocks), dim3(128), 0, stream, (const float*)zi,
                   (const float*)zf, z_stride, bi, bf, cap, m_state, cu_seqlens, state_slots, decay, kscale, m_run, H,
                   pairs);
  else if (dtype == Q3_DTYPE_BF16)
    e = launch_pdl(stabilised_gates_kernel<bf16>, dim3(blocks), dim3(128), 0, stream, (const bf16*)zi, (const bf16*)zf,
                   z_stride, bi, bf, cap, m_state, cu_seqlens, state_slots, decay, kscale, m_run, H, pairs);
  else
    return Q3_ERR_ARGUMENT;
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}

// head_norm_gate: every head's fp32 output divided by its root mean square, times a weight (one per value
// channel, shared by the heads or one per head and channel), times act(gate) and out_scale, rounded once.
// gate_act 0: silu, 1: sigmoid.  With m_run (fp32 [T, H]) a row of o has one more column, c = o[Dv], and the
// values are first divided by max(|c|, exp(-m_run)) + 1e-6 (the normaliser of a memory whose gates are kept
// in range by a running maximum).
__device__ __forceinline__ float gate_value(float g, int gate_act) {
  const float sg = 1.f / (1.f + expf(-g));
  return gate_act == 1 ? sg : g * sg;
}

template <typename T>
__global__ void head_norm_gate_kernel(const float* __restrict__ o, int o_stride, const float* __restrict__ m_run,
                                      const float* __restrict__ w, int w_per_head, float eps,
                                      const T* __restrict__ g, long g_stride, T* __restrict__ y, long y_stride,
                                      float out_scale, int gate_act, long items, int H, int Dv) {
  pdl_wait();
  pdl_launch_dependents();
  const long item = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (item >= items) return;
  const long t = item / H;
  const int h = (int)(item - t * H);
  const float* orow = o + item * o_stride;
  const float den = m_run ? fmaxf(fabsf(orow[Dv]), expf(-m_run[item])) + 1e-6f : 1.f;
  float ss = 0.f;
  for (int d = lane; d < Dv; d += 32) {
    const float x = m_run ? orow[d] / den : orow[d];
    ss += x * x;
  }
  const float rstd = rsqrtf(warp_sum(ss) / (float)Dv + eps);
  const T* grow = g + t * g_stride + (long)h * Dv;
  T* yrow = y + t * y_stride + (long)h * Dv;
  const float* wrow = w ? (w_per_head ? w + (long)h * Dv : w) : nullptr;
  for (int d = lane; d < Dv; d += 32) {
    float val = (m_run ? orow[d] / den : orow[d]) * rstd;
    if (wrow) val *= wrow[d];
    yrow[d] = from_f32<T>(val * gate_value(to_f32(grow[d]), gate_act) * out_scale);
  }
}

// The same with 16-byte accesses for value sizes up to 256 that are multiples of 8 (rows 16-byte
// aligned): a lane keeps its eight values in registers between the sum of squares and the store, and a
// warp takes as many (token, head) items as fit (`lph` lanes per item, a power of two >= Dv / 8).  Rows of
// o with the extra column are not aligned and are read value by value.
template <typename T>
__global__ void head_norm_gate_vec_kernel(const float* __restrict__ o, int o_stride, const float* __restrict__ m_run,
                                          const float* __restrict__ w, int w_per_head, float eps,
                                          const T* __restrict__ g, long g_stride, T* __restrict__ y, long y_stride,
                                          float out_scale, int gate_act, long items, int H, int Dv, int lph) {
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, per_warp = 32 / lph;
  const long item = ((long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per_warp + lane / lph;
  const int d = (lane % lph) * 8;
  const bool live = item < items && d < Dv;
  const long t = live ? item / H : 0;
  const int h = live ? (int)(item - t * H) : 0;
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, gate[8];
  float ss = 0.f;
  if (live) {
    const float* orow = o + item * o_stride;
    if (m_run) {
      const float den = fmaxf(fabsf(orow[Dv]), expf(-m_run[item])) + 1e-6f;
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = orow[d + e] / den;
    } else {
      load8(orow + d, v);
    }
    load8(g + t * g_stride + (long)h * Dv + d, gate);
#pragma unroll
    for (int e = 0; e < 8; ++e) ss += v[e] * v[e];
  }
  for (int off = lph >> 1; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
  if (!live) return;
  const float rstd = rsqrtf(ss / (float)Dv + eps);
  float wv[8];
  if (w) load8(w + (w_per_head ? (long)h * Dv : 0) + d, wv);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    float val = v[e] * rstd;
    if (w) val *= wv[e];
    v[e] = val * gate_value(gate[e], gate_act) * out_scale;
  }
  store8(y + t * y_stride + (long)h * Dv + d, v);
}

static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// o: fp32 [T, H, Dv] (with m_run: [T, H, Dv + 1] and m_run fp32 [T, H]); w: fp32 [Dv] shared by the heads
// or [H, Dv] (w_per_head), or null; g, y: head h of token t at [t * stride + h * Dv].
Q3_EXPORT int q3_head_norm_gate(int dtype, const float* o, const float* m_run, const float* w, int w_per_head,
                                float eps, const void* g, long g_stride, void* y, long y_stride, float out_scale,
                                int gate_act, int num_tokens, int H, int Dv, cudaStream_t stream) {
  if (!o || !g || !y || H < 1 || Dv < 1 || gate_act < 0 || gate_act > 1) return Q3_ERR_ARGUMENT;
  const long items = (long)num_tokens * H;
  if (items == 0) return Q3_OK;
  const int o_stride = Dv + (m_run ? 1 : 0);
  const unsigned blocks = (unsigned)((items + 7) / 8);
  cudaError_t e;
  const bool vec = Dv % 8 == 0 && Dv <= 256 && g_stride % 8 == 0 && y_stride % 8 == 0 && (m_run || aligned16(o)) &&
                   aligned16(g) && aligned16(y) && (!w || aligned16(w));
  int lph = 1;  // lanes per (token, head) item
  while (lph * 8 < Dv) lph <<= 1;
  const long per_block = 8 * (32 / (lph > 32 ? 32 : lph));
  const unsigned vblocks = (unsigned)((items + per_block - 1) / per_block);
  if (vec && dtype == Q3_DTYPE_F32)
    e = launch_pdl(head_norm_gate_vec_kernel<float>, dim3(vblocks), dim3(256), 0, stream, o, o_stride, m_run, w,
                   w_per_head, eps, (const float*)g, g_stride, (float*)y, y_stride, out_scale, gate_act, items, H, Dv,
                   lph);
  else if (vec && dtype == Q3_DTYPE_BF16)
    e = launch_pdl(head_norm_gate_vec_kernel<bf16>, dim3(vblocks), dim3(256), 0, stream, o, o_stride, m_run, w,
                   w_per_head, eps, (const bf16*)g, g_stride, (bf16*)y, y_stride, out_scale, gate_act, items, H, Dv,
                   lph);
  else if (dtype == Q3_DTYPE_F32)
    e = launch_pdl(head_norm_gate_kernel<float>, dim3(blocks), dim3(256), 0, stream, o, o_stride, m_run, w, w_per_head,
                   eps, (const float*)g, g_stride, (float*)y, y_stride, out_scale, gate_act, items, H, Dv);
  else if (dtype == Q3_DTYPE_BF16)
    e = launch_pdl(head_norm_gate_kernel<bf16>, dim3(blocks), dim3(256), 0, stream, o, o_stride, m_run, w, w_per_head,
                   eps, (const bf16*)g, g_stride, (bf16*)y, y_stride, out_scale, gate_act, items, H, Dv);
  else
    return Q3_ERR_ARGUMENT;
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}
