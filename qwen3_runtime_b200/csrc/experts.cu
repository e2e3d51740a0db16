// Routed experts: router scores and choice, grouping of (token, choice) slots by expert on the
// device, the experts' two products over their own slots on the FMA pipes (float32, and bfloat16 of sizes
// that experts_tcgen05.cu refuses), and the per-token sum.
//
//   route_top      z = W_router h in fp32, the `top` largest z (the order of their sigmoids; lowest
//                  index on a tie) with sigmoid(z) as weights (optionally divided by their sum), or
//                  with the softmax over the chosen z as weights
//   group_slots    slots sorted by expert: offsets[E + 1], order[S], and for the products the
//                  first row tile of each expert, tile_offsets[E + 1] (tiles of `bm` slots)
//   expert_gate_up mid[slot] = glu(W_gate_e x, W_up_e x), x = h[token] * weight (rounded to the
//                  operand type) when the weight multiplies the expert's input
//                  glu: g = min(g, limit), u = clamp(u, -limit, limit), g * sigmoid(alpha g) * (u + off)
//   expert_up      mid[slot] = relu(W_up_e h[token])^2: the first product of an expert without a gate
//   expert_down    y[slot] = W_down_e mid[slot]
//   combine        out[t] = sum over the token's slots of y (times the weight when it multiplies
//                  the output), plus the shared expert's result (times the sigmoid of a gate logit, if
//                  one is given), summed in fp32 in slot order
//
// Products accumulate in fp32 on the FMA pipes, each output one accumulator over ascending k, so a
// token's result does not depend on which other tokens chose the same expert.  Nothing here reads
// a count back on the host: grids are sized for the worst case and surplus blocks leave at once.
#include "common.cuh"
#include "split_mma.cuh"

constexpr int EXPERT_BM = 32;  // slots per row tile of the FMA products

// ---- router ------------------------------------------------------------------------------------
// Logits, then the choice.  A token's logits are the same bits in every batch.
//   bfloat16 tokens (route_logits_mma): mma.sync with the router's float32 as the sum of three bfloat16 (split_mma.cuh).  A block's
//   eight warps share the width in equal runs of 32-value slices; a slice's six products are one chain, smallest first, its result
//   is added to float32 sums; the warps' sums are added in order.  Blocks of 32 tokens x 32 experts where there are enough of
//   them, else 16 x 8: the bits do not depend on it.  What is NaN is worked out once more with FMAs, as parts of infinities have
//   no sum.  With the choice, us, FMAs (the float32 form) / here: 2048 tokens x 64 experts x 2048 31.2 / 14.3, 8 tokens 8.3 / 5.5,
//   2048 x 32 x 4096 29.8 / 21.0, 2048 x 256 x 2048 80 / 42; relative error against float64 1.6e-7 .. 2.1e-7 / 1.0e-7 .. 1.1e-7.
//   float32 tokens: lane l adds the products of k = 4 l .. 4 l + 3, then of those + 128, and so on; the lanes' sums are added by
//   halving.  Few tokens (route_logits): a block stages 2 tokens' rows in shared memory, each of its eight warps streams one
//   expert's router row for them.  Many tokens (route_logits_tile): a warp keeps 8 tokens x 8 experts in registers and reads
//   operands straight from L1.
// Three kernels choose, one warp per token: the `top` largest logits -- the choice is made on the logits, which order the
// experts as their sigmoids do but do not collapse into ties where the sigmoid saturates; lowest index on an exact tie, NaN
// after every number -- with logits in registers (route_pick_regs, up to 256 outputs) or in memory (route_pick), and the choice
// on a softmax over all outputs (route_pick_softmax_all).
constexpr int ROUTE_TT = 8;

__global__ void __launch_bounds__(256)
route_logits_kernel(const float* __restrict__ h, long h_stride, const float* __restrict__ router, int num_tokens, int E,
                    int W, int tt, int vec, float* __restrict__ logits) {
  extern __shared__ float route_rows[];  // [tt][W], tt <= ROUTE_TT tokens per block
  pdl_wait();
  pdl_launch_dependents();
  const int t0 = blockIdx.x * tt;
  const int nt = min(tt, num_tokens - t0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int t = 0; t < nt; ++t) {
    const float* src = h + (long)(t0 + t) * h_stride;
    if (vec) {
      for (int i = threadIdx.x * 8; i < W; i += 256 * 8) {
        float v[8];
        load8(src + i, v);
        store8(route_rows + t * W + i, v);
      }
    } else {
      for (int i = threadIdx.x; i < W; i += 256) route_rows[t * W + i] = src[i];
    }
  }
  __syncthreads();
  const int e = blockIdx.y * 8 + warp;
  if (e >= E) return;
  const float* wr = router + (long)e * W;
  float acc[ROUTE_TT];
#pragma unroll
  for (int t = 0; t < ROUTE_TT; ++t) acc[t] = 0.f;
  if ((W & 3) == 0) {
#pragma unroll 2
    for (int i = lane * 4; i < W; i += 128) {
      const float4 w4 = *reinterpret_cast<const float4*>(wr + i);
#pragma unroll
      for (int t = 0; t < ROUTE_TT; ++t) {
        if (t < nt) {
          const float4 x4 = *reinterpret_cast<const float4*>(route_rows + t * W + i);
          acc[t] = fmaf(x4.x, w4.x, fmaf(x4.y, w4.y, fmaf(x4.z, w4.z, fmaf(x4.w, w4.w, acc[t]))));
        }
      }
    }
  } else {
    for (int i = lane; i < W; i += 32) {
      const float w1 = wr[i];
#pragma unroll
      for (int t = 0; t < ROUTE_TT; ++t)
        if (t < nt) acc[t] = fmaf(route_rows[t * W + i], w1, acc[t]);
    }
  }
#pragma unroll
  for (int t = 0; t < ROUTE_TT; ++t) {
    if (t < nt) {
      const float v = warp_sum(acc[t]);
      if (lane == 0) logits[(long)(t0 + t) * E + e] = v;
    }
  }
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }

constexpr int ROUTE_EPW = 8;  // experts per warp

// WT, WE: warps of a block along tokens and along experts
template <int WT, int WE>
__global__ void __launch_bounds__(32 * WT * WE, 3)
route_logits_tile_kernel(const float* __restrict__ h, long h_stride, const float* __restrict__ router, int num_tokens, int E,
                         int W, float* __restrict__ logits) {
  pdl_wait();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int t0 = (blockIdx.x * WT + warp / WE) * ROUTE_TT;
  int e0 = (blockIdx.y * WE + warp % WE) * ROUTE_EPW;
  if (t0 >= num_tokens || e0 >= E) return;
  // a last group that would pass the end starts earlier: its first logits are computed twice, with the same bits
  t0 = min(t0, num_tokens - ROUTE_TT);
  e0 = min(e0, E - ROUTE_EPW);
  const float* x = h + (long)t0 * h_stride + lane * 4;
  const float* w = router + (long)e0 * W + lane * 4;
  float acc[ROUTE_TT][ROUTE_EPW];
#pragma unroll
  for (int t = 0; t < ROUTE_TT; ++t)
#pragma unroll
    for (int e = 0; e < ROUTE_EPW; ++e) acc[t][e] = 0.f;
  for (int i = 0; i < W - lane * 4; i += 128) {
    float4 w4[ROUTE_EPW];
#pragma unroll
    for (int e = 0; e < ROUTE_EPW; ++e) w4[e] = load4(w + (long)e * W + i);
#pragma unroll
    for (int t = 0; t < ROUTE_TT; ++t) {
      const float4 x4 = load4(x + t * h_stride + i);
#pragma unroll
      for (int e = 0; e < ROUTE_EPW; ++e)
        acc[t][e] = fmaf(x4.x, w4[e].x, fmaf(x4.y, w4[e].y, fmaf(x4.z, w4[e].z, fmaf(x4.w, w4[e].w, acc[t][e]))));
    }
  }
#pragma unroll
  for (int t = 0; t < ROUTE_TT; ++t)
#pragma unroll
    for (int e = 0; e < ROUTE_EPW; ++e) {
      const float v = warp_sum(acc[t][e]);
      if (lane == 0) logits[(long)(t0 + t) * E + e0 + e] = v;
    }
}

// MT x 16 tokens and NT x 8 experts a block.  Lane (g, t4) = (lane / 4, lane % 4) of a fragment holds rows g (and g + 8) and, of a
// slice, k = 8 t4 .. 8 t4 + 7, half of them for each of two MMAs: the order of k within a slice is the same for both operands.
// VEC: values that a load takes, as far as strides, addresses and the width allow: 8 (tokens 16 bytes, the router 2 x 16), 4 or 1.
constexpr int ROUTE_SLICE = 32, ROUTE_WARPS = 8;
template <int MT, int NT, int VEC>
__global__ void __launch_bounds__(32 * ROUTE_WARPS)
route_logits_mma_kernel(const bf16* __restrict__ h, long h_stride, const float* __restrict__ router, int num_tokens, int E,
                        int W, float* __restrict__ logits) {
  __shared__ float parts[ROUTE_WARPS][MT * 16][NT * 8 + 1];
  pdl_wait();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int t0 = blockIdx.x * (16 * MT), e0 = blockIdx.y * (8 * NT);
  const bf16* x[MT][2];  // (what lies beyond the last token or expert is read as that one, and not stored)
  const float* w[NT];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int r = 0; r < 2; ++r) x[m][r] = h + (long)min(t0 + m * 16 + r * 8 + g, num_tokens - 1) * h_stride;
#pragma unroll
  for (int n = 0; n < NT; ++n) w[n] = router + (long)min(e0 + n * 8 + g, E - 1) * W;
  uint4 a[MT][2];
  float b[NT][8];
  auto load = [&](int slice) {
    const int k = slice * ROUTE_SLICE + 8 * t4;
    if (VEC > 1) {
      const bool in = k < W, on = VEC == 8 ? in : k + 4 < W;  // (of 4 values a load, the second may be beyond the end)
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          if (VEC == 8) {
            a[m][r] = in ? __ldg(reinterpret_cast<const uint4*>(x[m][r] + k)) : make_uint4(0, 0, 0, 0);
          } else {
            const uint2 lo = in ? __ldg(reinterpret_cast<const uint2*>(x[m][r] + k)) : make_uint2(0, 0);
            const uint2 hi = on ? __ldg(reinterpret_cast<const uint2*>(x[m][r] + k + 4)) : make_uint2(0, 0);
            a[m][r] = make_uint4(lo.x, lo.y, hi.x, hi.y);
          }
        }
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 8; i += 4) {
          const float4 v = (i ? on : in) ? __ldg(reinterpret_cast<const float4*>(w[n] + k + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
          b[n][i] = v.x, b[n][i + 1] = v.y, b[n][i + 2] = v.z, b[n][i + 3] = v.w;
        }
    } else {
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          uint32_t p[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const bf16 lo = k + 2 * i < W ? x[m][r][k + 2 * i] : from_f32<bf16>(0.f);
            const bf16 hi = k + 2 * i + 1 < W ? x[m][r][k + 2 * i + 1] : from_f32<bf16>(0.f);
            p[i] = (uint32_t)__bfloat16_as_ushort(lo) | (uint32_t)__bfloat16_as_ushort(hi) << 16;
          }
          a[m][r] = make_uint4(p[0], p[1], p[2], p[3]);
        }
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 8; ++i) b[n][i] = k + i < W ? w[n][k + i] : 0.f;
    }
  };
  float sum[MT][NT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[m][n][j] = 0.f;
  const int slices = (W + ROUTE_SLICE - 1) / ROUTE_SLICE, per = (slices + ROUTE_WARPS - 1) / ROUTE_WARPS;
  const int last = min(slices, (warp + 1) * per);
  int slice = warp * per;
  if (slice < last) load(slice);
  for (; slice < last; ++slice) {
    uint32_t left[MT][2][4], right[NT][2][2][3];  // by MMA; right: pairs of k, parts
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const uint32_t lo[4] = {a[m][0].x, a[m][0].y, a[m][0].z, a[m][0].w}, hi[4] = {a[m][1].x, a[m][1].y, a[m][1].z, a[m][1].w};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        left[m][i][0] = lo[2 * i];
        left[m][i][1] = hi[2 * i];
        left[m][i][2] = lo[2 * i + 1];
        left[m][i][3] = hi[2 * i + 1];
      }
    }
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) ds_split(b[n][2 * i], b[n][2 * i + 1], right[n][i >> 1][i & 1]);
    if (slice + 1 < last) load(slice + 1);  // on its way while this one is multiplied
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        float acc[4];
        ds_mma_zero(acc, left[m][0], right[n][0][0][2], right[n][0][1][2]);
        mma_bf16(acc, left[m][1], right[n][1][0][2], right[n][1][1][2]);
#pragma unroll
        for (int part = 1; part >= 0; --part)
#pragma unroll
          for (int i = 0; i < 2; ++i) mma_bf16(acc, left[m][i], right[n][i][0][part], right[n][i][1][part]);
#pragma unroll
        for (int j = 0; j < 4; ++j) sum[m][n][j] += acc[j];
      }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int j = 0; j < 4; ++j) parts[warp][m * 16 + g + 4 * (j & 2)][n * 8 + 2 * t4 + (j & 1)] = sum[m][n][j];
  __syncthreads();
  constexpr int OUT = MT * 16 * NT * 8;
#pragma unroll 1
  for (int i = threadIdx.x; i - lane < OUT; i += 32 * ROUTE_WARPS) {  // (whole warps)
    const int t = i / (NT * 8), e = i - t * (NT * 8);
    const bool live = i < OUT && t0 + t < num_tokens && e0 + e < E;
    float v = 0.f;
    if (live) {
      v = parts[0][t][e];
#pragma unroll
      for (int p = 1; p < ROUTE_WARPS; ++p) v += parts[p][t][e];
    }
    for (uint32_t none = __ballot_sync(0xffffffffu, v != v); none; none &= none - 1) {
      const int from = i - lane + __ffs(none) - 1, ft = from / (NT * 8), fe = from - ft * (NT * 8);
      const bf16* xr = h + (long)(t0 + ft) * h_stride;
      const float* wr = router + (long)(e0 + fe) * W;
      float again = 0.f;
      for (int k = lane; k < W; k += 32) again = fmaf(to_f32(xr[k]), wr[k], again);
      again = warp_sum(again);
      if (lane == __ffs(none) - 1) v = again;
    }
    if (live) logits[(long)(t0 + t) * E + e0 + e] = v;
  }
}

// The same choice as route_pick_kernel for up to 32 * PICK_REGS outputs: a token's logits are read once, all loads in
// flight together, and wait in registers (one warp per token; lane l holds outputs l, l + 32, ...) as whole numbers of their order,
// so that a choice is two reductions over the warp.  (2048 tokens, 6 of 64: with ten shuffles a choice 8.3 us; logits and choice
// 18.7 -> 14.3.)
constexpr int PICK_REGS = 8;

// 0 for NaN; else larger for a larger number, the same for both zeros
__device__ __forceinline__ uint32_t order_of(float x) {
  const uint32_t b = __float_as_uint(x + 0.f);
  return x != x ? 0u : b & 0x80000000u ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float number_of(uint32_t order) {
  return order ? __uint_as_float(order & 0x80000000u ? order & 0x7fffffffu : ~order) : -INFINITY;
}

template <int REGS>
__global__ void route_pick_regs_kernel(const float* __restrict__ logits, int num_tokens, int E, int top, int mode,
                                       float scale, int* __restrict__ chosen, float* __restrict__ weights) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= num_tokens) return;
  const float* z = logits + (long)t * E;
  float v[REGS];
  uint32_t order[REGS], open = 0;  // open: outputs of this lane that exist and have not been taken
#pragma unroll
  for (int r = 0; r < REGS; ++r) v[r] = lane + 32 * r < E ? z[lane + 32 * r] : 0.f;
#pragma unroll
  for (int r = 0; r < REGS; ++r) {
    order[r] = order_of(v[r]);
    open |= (lane + 32 * r < E ? 1u : 0u) << r;
  }
  float mine[REGS];  // lane k % 32 keeps the logit of choice k, then its score
  int index[REGS];
#pragma unroll
  for (int r = 0; r < REGS; ++r) mine[r] = 0.f, index[r] = 0;
  float first = 0.f;
  for (int k = 0; k < top; ++k) {
    uint32_t best = 0;
    int at = 0x7fffffff;  // (where nothing but NaN is left: the lowest open output)
#pragma unroll
    for (int r = REGS - 1; r >= 0; --r)
      if ((open >> r & 1u) && order[r] >= best) {
        best = order[r];
        at = lane + 32 * r;
      }
    const uint32_t most = __reduce_max_sync(0xffffffffu, best);
    at = (int)__reduce_min_sync(0xffffffffu, best == most ? (uint32_t)at : 0x7fffffffu);
    if ((at & 31) == lane) open &= ~(1u << (at >> 5));
    if (k == 0) first = number_of(most);  // the largest logit: the softmax's reference point
#pragma unroll
    for (int r = 0; r < REGS; ++r)
      if (k == lane + 32 * r) mine[r] = number_of(most), index[r] = at;
  }
#pragma unroll
  for (int r = 0; r < REGS; ++r) mine[r] = mode == 2 ? expf(mine[r] - first) : 1.f / (1.f + expf(-mine[r]));
  float total = 0.f;
  if (mode)
#pragma unroll
    for (int r = 0; r < REGS; ++r)
      for (int k = 32 * r; k < min(top, 32 * r + 32); ++k) total += __shfl_sync(0xffffffffu, mine[r], k & 31);
#pragma unroll
  for (int r = 0; r < REGS; ++r) {
    const int k = lane + 32 * r;
    if (k < top) {
      chosen[(long)t * top + k] = index[r];
      weights[(long)t * top + k] = (mode ? mine[r] / total : mine[r]) * scale;
    }
  }
}

// mode 0: weights are the chosen logits' sigmoids; 1: those divided by their sum; 2: the softmax over
// the chosen logits only; all times `scale`.
__global__ void route_pick_kernel(float* __restrict__ logits, int num_tokens, int E, int top, int mode,
                                  float scale, int* __restrict__ chosen, float* __restrict__ weights) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= num_tokens) return;
  float* z = logits + (long)t * E;
  float total = 0.f, first = 0.f;
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int at = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      const float v = z[e];
      if (v > best || (v == best && e < at)) {
        best = v;
        at = e;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oa = __shfl_xor_sync(0xffffffffu, at, o);
      if (ob > best || (ob == best && oa < at)) {
        best = ob;
        at = oa;
      }
    }
    if (at >= E) {  // nothing but NaN is left: the lowest output not chosen yet, one of the first k + 1
      int low = 0x7fffffff;
      for (int e = lane; e <= k && low > e; e += 32) {
        bool open = true;
        for (int c = 0; c < k; ++c) open = open && chosen[(long)t * top + c] != e;
        if (open) low = e;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) low = min(low, __shfl_xor_sync(0xffffffffu, low, o));
      at = low;
    }
    if (k == 0) first = best;  // the largest logit: the softmax's reference point
    const float score = mode == 2 ? expf(best - first) : 1.f / (1.f + expf(-best));
    if (lane == 0) {
      chosen[(long)t * top + k] = at;
      weights[(long)t * top + k] = score;
      z[at] = NAN;  // taken: compares false with everything
    }
    total += score;
    __syncwarp();
  }
  if (mode || scale != 1.f)
    for (int k = lane; k < top; k += 32) {
      const float w = weights[(long)t * top + k];
      weights[(long)t * top + k] = (mode ? w / total : w) * scale;
    }
}

// mode 3: s = softmax over all E logits; the choice is made on c = s + correction (correction null: on s)
// among the outputs of the `keep` best of `count` equal groups of neighbours (a group's score: its largest
// c; count <= 1: no groups), lowest index on a tie; the weights are the chosen s, divided by their sum +
// 1e-20 when `renorm`, times `scale`.  One warp per token; c and the groups' scores wait in shared memory.
__global__ void route_pick_softmax_all_kernel(const float* __restrict__ logits, int num_tokens, int E, int top,
                                              const float* __restrict__ correction, int count, int keep, int renorm,
                                              float scale, int* __restrict__ chosen, float* __restrict__ weights) {
  extern __shared__ float pick_smem[];  // per warp: c[E], group scores[count]
  pdl_wait();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * (blockDim.x >> 5) + warp;
  if (t >= num_tokens) return;
  const int groups = count > 1 ? count : 0;
  float* c = pick_smem + (long)warp * (E + groups);
  float* gs = c + E;
  const float* z = logits + (long)t * E;
  float zmax = -INFINITY;
  for (int e = lane; e < E; e += 32) zmax = fmaxf(zmax, z[e]);
  zmax = warp_max(zmax);
  float den = 0.f;
  for (int e = lane; e < E; e += 32) den += expf(z[e] - zmax);
  den = warp_sum(den);
  for (int e = lane; e < E; e += 32) c[e] = expf(z[e] - zmax) / den + (correction ? correction[e] : 0.f);
  __syncwarp();
  if (groups) {
    const int per = E / groups;
    for (int g = lane; g < groups; g += 32) {
      float best = -INFINITY;
      for (int e = g * per; e < (g + 1) * per; ++e) best = fmaxf(best, c[e]);
      gs[g] = best;
    }
    __syncwarp();
    // a group stays if fewer than `keep` groups come before it (larger score, or equal and lower index)
    for (int g = lane; g < groups; g += 32) {
      const float mine = gs[g];
      int before = 0;
      for (int o = 0; o < groups; ++o) before += gs[o] > mine || (gs[o] == mine && o < g);
      if (before >= keep)
        for (int e = g * per; e < (g + 1) * per; ++e) c[e] = -INFINITY;
    }
    __syncwarp();
  }
  float total = 0.f;
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int at = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      const float v = c[e];
      if (v > best || (v == best && e < at)) {
        best = v;
        at = e;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oa = __shfl_xor_sync(0xffffffffu, at, o);
      if (ob > best || (ob == best && oa < at)) {
        best = ob;
        at = oa;
      }
    }
    if (at >= E) at = k;  // nothing left to choose from (more choices than open outputs): never read
    const float score = expf(z[at] - zmax) / den;
    if (lane == 0) {
      chosen[(long)t * top + k] = at;
      weights[(long)t * top + k] = score;
      c[at] = NAN;  // taken: compares false with everything
    }
    total += score;
    __syncwarp();
  }
  if (renorm || scale != 1.f)
    for (int k = lane; k < top; k += 32) {
      const float w = weights[(long)t * top + k];
      weights[(long)t * top + k] = (renorm ? w / (total + 1e-20f) : w) * scale;
    }
}

static int sm_count() {
  static int count_on[Q3_MAX_DEVICES];
  int& count = count_on[q3_current_device()];
  int device = 0;
  if (!count && (cudaGetDevice(&device) != cudaSuccess ||
                 cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess))
    count = 0;
  return count;
}

// logits: fp32 scratch [num_tokens, E].
// scale: a factor on all weights.  mode 3 takes correction (fp32 [E] or null), count and keep (groups) and renorm; the other modes ignore them.
Q3_EXPORT int q3_route_top(int dtype, const void* h, long h_stride, const float* router, int num_tokens, int E, int W,
                           int top, int mode, float* logits, int* chosen, float* weights, const float* correction,
                           int count, int keep, int renorm, float scale, cudaStream_t stream) {
  if (!h || !router || !logits || !chosen || !weights || E < 1 || W < 1 || top < 1 || top > E) return Q3_ERR_ARGUMENT;
  if (mode == 3 && count > 1 && (E % count || keep < 1 || keep > count || top > keep * (E / count)))
    return Q3_ERR_ARGUMENT;
  if (num_tokens == 0) return Q3_OK;
  if (reinterpret_cast<uintptr_t>(router) & 15) return Q3_ERR_UNSUPPORTED;
  if (dtype != Q3_DTYPE_F32 && dtype != Q3_DTYPE_BF16) return Q3_ERR_ARGUMENT;
  cudaError_t e;
  if (dtype == Q3_DTYPE_BF16) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(h) | (uintptr_t)(2 * h_stride) | (uintptr_t)(2 * W);
    const int vec = (at & 15) == 0 ? 8 : (at & 7) == 0 ? 4 : 1;
    const dim3 large((num_tokens + 31) / 32, (E + 31) / 32), small((num_tokens + 15) / 16, (E + 7) / 8);
#define Q3_ROUTE_MMA(MT_, NT_, VEC_, grid_)                                                                              \
  e = launch_pdl(route_logits_mma_kernel<MT_, NT_, VEC_>, grid_, dim3(32 * ROUTE_WARPS), 0, stream, (const bf16*)h, h_stride, \
                 router, num_tokens, E, W, logits)
    // large blocks from where they fill half of the SMs, and where 32 experts are not mostly none (8 x 512, 4096 tokens: 13.7 us
    // with the choice, 6.1 with small blocks).  Rows at 8-byte places (2048 tokens x 64 experts x 2052 with
    // the choice): single loads in small blocks 45.5, FMAs 35.7, loads of 4 in large ones 16.8.
    const bool wide = vec > 1 && E > 16 && 2l * large.x * large.y >= sm_count() && large.y <= 65535;
    if (!wide && small.y > 65535) return Q3_ERR_UNSUPPORTED;
    if (wide && vec == 8) Q3_ROUTE_MMA(2, 4, 8, large);
    else if (wide) Q3_ROUTE_MMA(2, 4, 4, large);
    else if (vec == 8) Q3_ROUTE_MMA(1, 1, 8, small);
    else if (vec == 4) Q3_ROUTE_MMA(1, 1, 4, small);
    else Q3_ROUTE_MMA(1, 1, 1, small);
#undef Q3_ROUTE_MMA
  } else {
    // both kernels give the same bits; the tile kernel needs about 64 tokens to fill the SMs
    const bool tile = num_tokens > 64 && E >= ROUTE_EPW && W % 4 == 0 && h_stride % 4 == 0 &&
                      (reinterpret_cast<uintptr_t>(h) & 15) == 0;
    // a block's four warps all have experts: 8 experts x 1024, 4096 tokens 23 us, with three idle warps a block 30
    const int we = E > 2 * ROUTE_EPW ? 4 : E > ROUTE_EPW ? 2 : 1;
    const int te = we * ROUTE_EPW, tokens = 4 / we * ROUTE_TT;
    if (tile && (E + te - 1) / te <= 65535) {
      const dim3 grid((num_tokens + tokens - 1) / tokens, (E + te - 1) / te);
#define Q3_ROUTE_TILE(WT_, WE_)                                                                                          \
  e = launch_pdl(route_logits_tile_kernel<WT_, WE_>, grid, dim3(32 * WT_ * WE_), 0, stream, (const float*)h, h_stride, \
                 router, num_tokens, E, W, logits)
      if (we == 4) Q3_ROUTE_TILE(1, 4); else if (we == 2) Q3_ROUTE_TILE(2, 2); else Q3_ROUTE_TILE(4, 1);
#undef Q3_ROUTE_TILE
    } else {
      int tt = num_tokens > 64 ? ROUTE_TT : 2;
      while (tt > 1 && (size_t)tt * W * sizeof(float) > 128 * 1024) tt >>= 1;  // fewer where their rows would not fit
      const size_t smem = (size_t)tt * W * sizeof(float);
      if (smem > 200 * 1024 || (E + 7) / 8 > 65535) return Q3_ERR_UNSUPPORTED;
      const dim3 grid((num_tokens + tt - 1) / tt, (E + 7) / 8);
      const int vec = W % 8 == 0 && h_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(h) & 15) == 0;
      if (smem > 48 * 1024)
        cudaFuncSetAttribute(route_logits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      e = launch_pdl(route_logits_kernel, grid, dim3(256), smem, stream, (const float*)h, h_stride, router,
                     num_tokens, E, W, tt, vec, logits);
    }
  }
  if (e != cudaSuccess) return Q3_ERR_LAUNCH;
  if (mode == 3) {
    const size_t pick = (size_t)4 * (E + (count > 1 ? count : 0)) * sizeof(float);
    if (pick > 48 * 1024) return Q3_ERR_UNSUPPORTED;
    e = launch_pdl(route_pick_softmax_all_kernel, dim3((num_tokens + 3) / 4), dim3(128), pick, stream,
                   (const float*)logits, num_tokens, E, top, correction, count, keep, renorm, scale, chosen, weights);
    return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
  }
#define Q3_PICK(REGS_)                                                                                                  \
  e = launch_pdl(route_pick_regs_kernel<REGS_>, dim3((num_tokens + 3) / 4), dim3(128), 0, stream, (const float*)logits,  \
                 num_tokens, E, top, mode, scale, chosen, weights)
  if (E <= 64) Q3_PICK(2);
  else if (E <= 32 * PICK_REGS) Q3_PICK(PICK_REGS);
#undef Q3_PICK
  else
    e = launch_pdl(route_pick_kernel, dim3((num_tokens + 3) / 4), dim3(128), 0, stream, logits, num_tokens, E, top,
                   mode, scale, chosen, weights);
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}

// ---- slots grouped by expert ----------------------------------------------------------------------
// One block, for a few slots and experts.  Slots of one expert keep their order (slot s before slot
// s' > s).
__global__ void group_slots_kernel(const int* __restrict__ chosen, int S, int E, int bm, int* __restrict__ offsets,
                                   int* __restrict__ tile_offsets, int* __restrict__ order, int* __restrict__ place) {
  extern __shared__ int sm[];  // counts[E], cursor[E]
  int* counts = sm;
  int* cursor = sm + E;
  pdl_wait();
  pdl_launch_dependents();
  for (int e = threadIdx.x; e < E; e += blockDim.x) counts[e] = 0;
  __syncthreads();
  for (int s = threadIdx.x; s < S; s += blockDim.x) atomicAdd(&counts[chosen[s]], 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    int at = 0, tiles = 0;
    for (int e = 0; e < E; ++e) {
      offsets[e] = at;
      tile_offsets[e] = tiles;
      cursor[e] = at;
      at += counts[e];
      tiles += (counts[e] + bm - 1) / bm;
    }
    offsets[E] = at;
    tile_offsets[E] = tiles;
  }
  __syncthreads();
  // a slot's place in its expert's group is the number of earlier slots with the same expert
  for (int s = threadIdx.x; s < S; s += blockDim.x) {
    const int e = chosen[s];
    int rank = 0;
    for (int r = 0; r < s; ++r) rank += chosen[r] == e;
    if (order) order[cursor[e] + rank] = s;
    if (place) place[s] = cursor[e] + rank;
  }
}

// The same for many slots, in two kernels of a block per 1024 slots (the order inside an expert's group may differ from
// run to run; every slot's result is computed on its own, so the outputs do not).  count_slots: a slot's rank among its
// block's slots of the same expert and the block's counts; place_slots: every block adds up the counts of the blocks
// before it and of all blocks.  What bounds this is the latency of the atomics on a few counters; one block for all
// slots took 13 us for 12,288 slots of 64 experts, these two 8.
constexpr int GROUP_THREADS = 1024;
__global__ void __launch_bounds__(GROUP_THREADS)
count_slots_kernel(const int* __restrict__ chosen, int S, int E, int* __restrict__ ranks, int* __restrict__ counts) {
  extern __shared__ int sm[];
  const int tid = threadIdx.x, s = blockIdx.x * GROUP_THREADS + tid;
  for (int e = tid; e < E; e += GROUP_THREADS) sm[e] = 0;
  pdl_wait();
  pdl_launch_dependents();
  const int e = s < S ? chosen[s] : -1;
  __syncthreads();
  if (e >= 0) ranks[s] = atomicAdd(&sm[e], 1);
  __syncthreads();
  for (int x = tid; x < E; x += GROUP_THREADS) counts[(long)blockIdx.x * E + x] = sm[x];
}

__global__ void __launch_bounds__(GROUP_THREADS)
place_slots_kernel(const int* __restrict__ chosen, int S, int E, int bm, const int* __restrict__ ranks,
                   const int* __restrict__ counts, int* __restrict__ offsets, int* __restrict__ tile_offsets,
                   int* __restrict__ order, int* __restrict__ place) {
  extern __shared__ int sm[];
  int* total = sm;       // slots per expert; then the expert's first slot
  int* before = sm + E;  // slots of the expert in earlier blocks
  const int tid = threadIdx.x, s = blockIdx.x * GROUP_THREADS + tid;
  pdl_wait();
  pdl_launch_dependents();
  const int e = s < S ? chosen[s] : -1;
  const int rank = s < S ? ranks[s] : 0;
  for (int x = tid; x < E; x += GROUP_THREADS) {
    int sum = 0, mine = 0;
#pragma unroll 8
    for (int b = 0; b < (int)gridDim.x; ++b) {
      const int c = counts[(long)b * E + x];
      if (b < (int)blockIdx.x) mine += c;
      sum += c;
    }
    total[x] = sum;
    before[x] = mine;
  }
  __syncthreads();
  if (tid < 32) {
    int at = 0, tiles = 0;  // sums over the experts before this batch of 32
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int x = e0 + tid;
      const int n = x < E ? total[x] : 0, m = (n + bm - 1) / bm;
      int n_sum = n, m_sum = m;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, n_sum, o), b = __shfl_up_sync(0xffffffffu, m_sum, o);
        if (tid >= o) {
          n_sum += a;
          m_sum += b;
        }
      }
      if (x < E) {
        total[x] = at + n_sum - n;
        if (blockIdx.x == 0) {
          offsets[x] = at + n_sum - n;
          tile_offsets[x] = tiles + m_sum - m;
        }
      }
      at += __shfl_sync(0xffffffffu, n_sum, 31);
      tiles += __shfl_sync(0xffffffffu, m_sum, 31);
    }
    if (tid == 0 && blockIdx.x == 0) {
      offsets[E] = at;
      tile_offsets[E] = tiles;
    }
  }
  __syncthreads();
  if (e >= 0) {
    const int at = total[e] + before[e] + rank;
    if (order) order[at] = s;
    if (place) place[s] = at;
  }
}

// bm: slots per row tile of the products that will use tile_offsets (EXPERT_BM for the FMA kernels).  order: int32 [S], the
// slots in the grouped order, or null.  place: int32 [S],
// the position of every slot in the grouped order, or null.  scratch: int32 [S + ceil(S / 1024) * E] for the two kernels, or
// null for the one block (512 slots at most).
Q3_EXPORT int q3_group_slots(const int* chosen, int S, int E, int bm, int* offsets, int* tile_offsets, int* order,
                             int* place, int* scratch, cudaStream_t stream) {
  if (!chosen || !offsets || !tile_offsets || E < 1 || S < 0 || bm < 1) return Q3_ERR_ARGUMENT;
  if (E > 8192) return Q3_ERR_UNSUPPORTED;
  const size_t smem = 2 * (size_t)E * sizeof(int);
  cudaError_t e;
  if (!scratch) {
    if (S > 512) return Q3_ERR_ARGUMENT;
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(group_slots_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    e = launch_pdl(group_slots_kernel, dim3(1), dim3(512), smem, stream, chosen, S, E, bm, offsets, tile_offsets,
                   order, place);
  } else {
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(place_slots_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const dim3 grid((S + GROUP_THREADS - 1) / GROUP_THREADS);
    e = launch_pdl(count_slots_kernel, grid, dim3(GROUP_THREADS), smem / 2, stream, chosen, S, E, scratch, scratch + S);
    if (e == cudaSuccess)
      e = launch_pdl(place_slots_kernel, grid, dim3(GROUP_THREADS), smem, stream, chosen, S, E, bm,
                     (const int*)scratch, (const int*)(scratch + S), offsets, tile_offsets, order, place);
  }
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}

// ---- the experts' products ------------------------------------------------------------------------
__device__ __forceinline__ int expert_of_tile(const int* __restrict__ tile_offsets, int E, int tile) {
  int lo = 0, hi = E;  // the last e with tile_offsets[e] <= tile
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (tile_offsets[mid] <= tile) lo = mid; else hi = mid;
  }
  return lo;
}

// GATE_UP: A rows are h[token(slot)] (times the slot's weight when scale_input), B is the expert's
// [2F, W] (gate rows, then up rows), the result mid[slot, F].  Else: A rows are A[slot / top] (top = 1:
// a row per slot, the second product; top = the choices per token: the token's row, a first product
// without a gate), B is the expert's [N, K], the result C[slot, N]; scale_input then stands for the
// activation: 0 none, 1 the squared ReLU of the rounded product.
template <typename T, bool GATE_UP>
__global__ void __launch_bounds__(256)
expert_gemm_kernel(const T* __restrict__ A, long a_stride, const T* __restrict__ B, T* __restrict__ C, int N, int K,
                   const int* __restrict__ offsets, const int* __restrict__ tile_offsets,
                   const int* __restrict__ order, const float* __restrict__ weights, int E, int top,
                   int scale_input, float limit, float alpha, float up_offset) {
  constexpr int BM = EXPERT_BM, BN = 64, BK = 16, TM = 2, TN = 4, THREADS = 256;
  constexpr int NB = GATE_UP ? 2 : 1;
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[NB][BK][BN + 4];
  __shared__ int slot_of[BM];
  __shared__ float scale_of[BM];
  pdl_wait();
  pdl_launch_dependents();
  const int tile = blockIdx.y;
  if (tile >= tile_offsets[E]) return;
  const int e = expert_of_tile(tile_offsets, E, tile);
  const int row0 = offsets[e] + (tile - tile_offsets[e]) * BM;
  const int rows = min(BM, offsets[e + 1] - row0);
  const int tid = threadIdx.x;
  if (tid < BM) {
    const int slot = tid < rows ? order[row0 + tid] : -1;
    slot_of[tid] = slot;
    scale_of[tid] = (slot >= 0 && GATE_UP && scale_input) ? weights[slot] : 1.f;
  }
  __syncthreads();
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  const int n0 = blockIdx.x * BN;
  const T* Be = B + (long)e * (GATE_UP ? 2 : 1) * N * K;
  float acc[NB][TM][TN];
#pragma unroll
  for (int b = 0; b < NB; ++b)
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[b][i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += BK) {
    for (int x = tid; x < BM * BK; x += THREADS) {
      const int r = x / BK, c = x % BK;
      const int slot = slot_of[r], gk = k0 + c;
      float a = 0.f;
      if (slot >= 0 && gk < K) {
        const long arow = slot / top;
        a = to_f32(A[arow * a_stride + gk]);
        if (GATE_UP && scale_input) a = to_f32(from_f32<T>(a * scale_of[r]));
      }
      As[c][r] = a;
    }
    for (int x = tid; x < NB * BN * BK; x += THREADS) {
      const int b = x / (BN * BK), y = x % (BN * BK);
      const int r = y / BK, c = y % BK;
      const int gn = n0 + r, gk = k0 + c;
      Ws[b][c][r] = (gn < N && gk < K) ? to_f32(Be[((long)b * N + gn) * K + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        float w[TN];
#pragma unroll
        for (int j = 0; j < TN; ++j) w[j] = Ws[b][kk][tx * TN + j];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[b][i][j] = fmaf(a[i], w[j], acc[b][i][j]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int slot = slot_of[ty * TM + i];
    if (slot < 0) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx * TN + j;
      if (gn >= N) continue;
      if (GATE_UP) {
        // both products are rounded to the operand type before the gated unit, as two separate
        // products followed by an activation kernel would
        const float g = fminf(to_f32(from_f32<T>(acc[0][i][j])), limit);
        const float u = fminf(fmaxf(to_f32(from_f32<T>(acc[NB - 1][i][j])), -limit), limit);
        C[(long)slot * N + gn] = from_f32<T>((g / (1.f + expf(-alpha * g))) * (u + up_offset));
      } else if (scale_input) {
        const float r = fmaxf(to_f32(from_f32<T>(acc[0][i][j])), 0.f);
        C[(long)slot * N + gn] = from_f32<T>(r * r);
      } else {
        C[(long)slot * N + gn] = from_f32<T>(acc[0][i][j]);
      }
    }
  }
}

// h: [T, W] rows h_stride apart; gate_up: [E, 2F, W]; mid: [S, F]; S = T * top slots.
Q3_EXPORT int q3_expert_gate_up(int dtype, const void* h, long h_stride, const void* gate_up, void* mid, int S, int E,
                                int F, int W, int top, const int* offsets, const int* tile_offsets, const int* order,
                                const float* weights, int scale_input, float limit, float alpha, float up_offset,
                                cudaStream_t stream) {
  if (!h || !gate_up || !mid || !offsets || !tile_offsets || !order || !weights) return Q3_ERR_ARGUMENT;
  if (E < 1 || F < 1 || W < 1 || top < 1) return Q3_ERR_ARGUMENT;
  if (S == 0) return Q3_OK;
  const int tiles = S / EXPERT_BM + (E < S ? E : S);
  if (tiles > 65535) return Q3_ERR_UNSUPPORTED;
  const dim3 grid((F + 63) / 64, tiles);
  cudaError_t e;
  if (dtype == Q3_DTYPE_F32)
    e = launch_pdl(expert_gemm_kernel<float, true>, grid, dim3(256), 0, stream, (const float*)h, h_stride,
                   (const float*)gate_up, (float*)mid, F, W, offsets, tile_offsets, order, weights, E, top, scale_input,
                   limit, alpha, up_offset);
  else if (dtype == Q3_DTYPE_BF16)
    e = launch_pdl(expert_gemm_kernel<bf16, true>, grid, dim3(256), 0, stream, (const bf16*)h, h_stride,
                   (const bf16*)gate_up, (bf16*)mid, F, W, offsets, tile_offsets, order, weights, E, top, scale_input,
                   limit, alpha, up_offset);
  else
    return Q3_ERR_ARGUMENT;
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}

// mid: [S, F]; down: [E, W, F]; y: [S, W].
Q3_EXPORT int q3_expert_down(int dtype, const void* mid, const void* down, void* y, int S, int E, int F, int W,
                             const int* offsets, const int* tile_offsets, const int* order, cudaStream_t stream) {
  if (!mid || !down || !y || !offsets || !tile_offsets || !order || E < 1 || F < 1 || W < 1) return Q3_ERR_ARGUMENT;
  if (S == 0) return Q3_OK;
  const int tiles = S / EXPERT_BM + (E < S ? E : S);
  if (tiles > 65535) return Q3_ERR_UNSUPPORTED;
  const dim3 grid((W + 63) / 64, tiles);
  cudaError_t e;
  if (dtype == Q3_DTYPE_F32)
    e = launch_pdl(expert_gemm_kernel<float, false>, grid, dim3(256), 0, stream, (const float*)mid, (long)F,
                   (const float*)down, (float*)y, W, F, offsets, tile_offsets, order, (const float*)nullptr, E, 1, 0,
                   0.f, 0.f, 0.f);
  else if (dtype == Q3_DTYPE_BF16)
    e = launch_pdl(expert_gemm_kernel<bf16, false>, grid, dim3(256), 0, stream, (const bf16*)mid, (long)F,
                   (const bf16*)down, (bf16*)y, W, F, offsets, tile_offsets, order, (const float*)nullptr, E, 1, 0, 0.f,
                   0.f, 0.f);
  else
    return Q3_ERR_ARGUMENT;
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}

// An expert's first product without a gate: mid[slot] = act(W_up_e h[token(slot)]); up: [E, F, W].
// act 1: the squared ReLU.
Q3_EXPORT int q3_expert_up(int dtype, const void* h, long h_stride, const void* up, void* mid, int S, int E, int F,
                           int W, int top, const int* offsets, const int* tile_offsets, const int* order, int act,
                           cudaStream_t stream) {
  if (!h || !up || !mid || !offsets || !tile_offsets || !order || E < 1 || F < 1 || W < 1 || top < 1)
    return Q3_ERR_ARGUMENT;
  if (S == 0) return Q3_OK;
  const int tiles = S / EXPERT_BM + (E < S ? E : S);
  if (tiles > 65535) return Q3_ERR_UNSUPPORTED;
  const dim3 grid((F + 63) / 64, tiles);
  cudaError_t e;
  if (dtype == Q3_DTYPE_F32)
    e = launch_pdl(expert_gemm_kernel<float, false>, grid, dim3(256), 0, stream, (const float*)h, h_stride,
                   (const float*)up, (float*)mid, F, W, offsets, tile_offsets, order, (const float*)nullptr, E, top,
                   act, 0.f, 0.f, 0.f);
  else if (dtype == Q3_DTYPE_BF16)
    e = launch_pdl(expert_gemm_kernel<bf16, false>, grid, dim3(256), 0, stream, (const bf16*)h, h_stride,
                   (const bf16*)up, (bf16*)mid, F, W, offsets, tile_offsets, order, (const float*)nullptr, E, top, act,
                   0.f, 0.f, 0.f);
  else
    return Q3_ERR_ARGUMENT;
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}

// ---- per-token sum ----------------------------------------------------------------------------------
// VEC values of one token per thread (8: 16-byte accesses, rows of a multiple of 8; what bounds it is memory: 2048
// tokens x 2048 of 6 slots took 105 us with one value per thread, 18 us with 8).  place: the row of y that holds a slot
// (null: the slot's own number).
template <typename T, int VEC>
__global__ void combine_kernel(const T* __restrict__ y, const float* __restrict__ weights, const T* __restrict__ shared,
                               const T* __restrict__ shared_gate, long gate_stride, T* __restrict__ out, long total,
                               int W, int top, const int* __restrict__ chosen, int stored, const T* __restrict__ h,
                               long h_stride, const int* __restrict__ place) {
  pdl_wait();
  pdl_launch_dependents();
  const long idx = ((long)blockIdx.x * blockDim.x + threadIdx.x) * VEC;
  if (idx >= total) return;
  const long t = idx / W;
  const int i = (int)(idx - t * W);
  auto load = [](const T* p, float (&v)[VEC]) {
    if constexpr (VEC == 8) load8(p, v); else v[0] = to_f32(*p);
  };
  float sum[VEC];
#pragma unroll
  for (int x = 0; x < VEC; ++x) sum[x] = 0.f;
#pragma unroll 4
  for (int k = 0; k < top; ++k) {
    const long slot = t * top + k;
    // a choice beyond the stored experts stands for an expert that returns its input
    const bool same = chosen && chosen[slot] >= stored;
    float v[VEC];
    load(same ? h + t * h_stride + i : y + (place ? (long)place[slot] : slot) * W + i, v);
    const float w = weights ? weights[slot] : 1.f;
#pragma unroll
    for (int x = 0; x < VEC; ++x) sum[x] += weights ? v[x] * w : v[x];
  }
  if (shared) {
    float v[VEC];
    load(shared + idx, v);
    const float gate = shared_gate ? 1.f + expf(-to_f32(shared_gate[t * gate_stride])) : 1.f;
#pragma unroll
    for (int x = 0; x < VEC; ++x) sum[x] += shared_gate ? v[x] / gate : v[x];
  }
  if constexpr (VEC == 8) store8(out + idx, sum); else out[idx] = from_f32<T>(sum[0]);
}

// y: [T * top, W]; weights: fp32 [T * top] or null (the weight was applied to the input);
// shared: [T, W] or null; shared_gate: one logit per token, gate_stride elements apart, or null: the
// shared expert's result is multiplied by the logit's sigmoid; out: [T, W].  chosen (int32 [T * top], with
// h [T, W] rows h_stride apart, or null): a slot whose choice is >= `stored` takes the token's row of h in
// place of y.  place (int32 [T * top] or null): the row of y of every slot.
Q3_EXPORT int q3_expert_combine(int dtype, const void* y, const float* weights, const void* shared,
                                const void* shared_gate, long gate_stride, void* out, int num_tokens, int W, int top,
                                const int* chosen, int stored, const void* h, long h_stride, const int* place,
                                cudaStream_t stream) {
  if (!y || !out || W < 1 || top < 1 || (chosen && !h)) return Q3_ERR_ARGUMENT;
  const long total = (long)num_tokens * W;
  if (total == 0) return Q3_OK;
  const bool vec = W % 8 == 0 && (!chosen || h_stride % 8 == 0) &&
                   (((uintptr_t)y | (uintptr_t)shared | (uintptr_t)out | (chosen ? (uintptr_t)h : 0)) & 15) == 0;
  const unsigned blocks = (unsigned)((total / (vec ? 8 : 1) + 255) / 256);
  cudaError_t e;
#define Q3_COMBINE(T_, VEC_)                                                                                       \
  e = launch_pdl(combine_kernel<T_, VEC_>, dim3(blocks), dim3(256), 0, stream, (const T_*)y, weights,              \
                 (const T_*)shared, (const T_*)shared_gate, gate_stride, (T_*)out, total, W, top, chosen, stored,   \
                 (const T_*)h, h_stride, place)
  if (dtype == Q3_DTYPE_F32) {
    if (vec) Q3_COMBINE(float, 8); else Q3_COMBINE(float, 1);
  } else if (dtype == Q3_DTYPE_BF16) {
    if (vec) Q3_COMBINE(bf16, 8); else Q3_COMBINE(bf16, 1);
  } else {
    return Q3_ERR_ARGUMENT;
  }
#undef Q3_COMBINE
  return e == cudaSuccess ? Q3_OK : Q3_ERR_LAUNCH;
}
