// C[M, N] = A[M, K] * W[N, K]^T of float32 matrices on the tensor cores, every operand as the sum of three bfloat16 (8 + 8 + 8
// bits: nothing is lost, see split_mma.cuh) and the six products of parts that matter; the other three are below 2^-24 of a
// product together (2^-25 each for the larger two).
//
// The accumulators of tcgen05.mma round towards zero at every step (products of 2560 values: 2.7e-6 off, 7e-6 if all are
// positive; one chain of fp32 FMA 9e-7 and 7e-7, this kernel 1.2e-7 and 1.0e-7), so a chain is never longer than a slice of 64
// k-values: its 20 small products first, which cost no digits of the sum, then the 4 large ones; the slice's result is added to
// fp32 registers, rounded to nearest, in ascending k.  K may be cut into segments, whose sums are added in order by a second
// kernel; how many depends on N and K only.  So a row of C does not depend on M, on the tile chosen for M, or on where the row
// sits in the batch, and lies nearer to the exact product than the FMA chain (split_matrix and the kernel below; K from 1024:
// see the dispatch).
//
// A pair of blocks (one per SM, tcgen05 cta_group::2) is persistent over items of (2 x 128 weight rows, segment, token tile), token
// tiles of the same weights side by side.  Weights are the rows of an MMA, 128 in each block, tokens its 16 to 160 columns; a
// block's shared memory holds half of the tokens' parts only, and the weights' parts lie in tensor memory as the left operand.
// Roles of a block:
//   warp 0        TMA: its half of the tokens' three parts (made beforehand by split_matrix), four slices ahead
//   warp 1        MMA issuer (the leader's, for both)
//   warp 2        TMA: its weights as they are, three to eight slices ahead
//   warps 4..11   read them (half a row a thread), split them and write the parts to tensor memory, two to four slices ahead
//   warps 12..19  sums: the accumulators of a slice (two of them in tensor memory) are added to registers, a row and half of the
//                 columns a thread; at the item's end they are stored
// Few tokens: an item has 48 to 128 rows a block, whichever fills the rounds over the pairs.
// What bounds it: shared memory and the way from L2 to the SMs were what a slice waited for as long as one block read all of the
// tokens' parts and wrote the weights' to shared memory (160 tokens: 3700 cycles a slice, 24 products take 1900).  Now it takes
// 2050 to 2300; what is left is rounds that are not full (300 tokens of 19456 x 2560: 5 for 4.1) and the stores between items
// (about 4000 cycles; the accumulators hide two slices of it).  With up to 32 tokens the weights' bytes: 5.3 TB/s.
// us of this kernel alone, one block at a time with parts in shared memory / now: 300 tokens 19456 x 2560 199 / 145, 8192 x 2560
// 85 / 64; 160 tokens 123 / 95; one token 59 / 53; calls behind one another, split and sums included: 2560 x 9728 300 tokens 103 /
// 82, 33 tokens 45 / 35; 24576 x 4096 366 / 282, 148 / 101, one token 107 / 99; 151936 x 2560 one token 353 / 294.
// (An arrival at the leader's barrier that is released to the cluster takes its warp 1000 cycles: 300 tokens 204 us with it, 173
// without; the weights' loads from global memory into registers, two slices ahead, 211.)
#include "async_tiles.cuh"
#include "split_mma.cuh"

namespace split {

constexpr int ROWS = 128, SLICE = 64, MOST_TOKENS = 160;
constexpr int X_STAGES = 4, MOST_RAW = 8;  // slices of the tokens' parts, and of the weights, on their way
constexpr int W_STAGES = 4, W_COLUMNS = 96;  // slices of the weights' parts: at most four, where two accumulators leave room
constexpr int THREADS = 20 * 32;
constexpr int smem_bytes(int rows, int tokens, int raw) { return X_STAGES * 192 * tokens + raw * rows * SLICE * 4 + 1024; }
constexpr int MOST_SMEM = 231936;

// x [M, K], rows ldx apart, as three dense bfloat16 matrices one behind the other; K a multiple of 8
template <bool VEC>
__global__ void __launch_bounds__(256)
split_matrix(const float* __restrict__ x, long ldx, uint4* __restrict__ to, int M, int K) {
  const long at = (long)blockIdx.x * 256 + threadIdx.x, per_row = K / 8;
  if (at >= M * per_row) return;
  const long m = at / per_row;
  const float* src = x + m * ldx + (at - m * per_row) * 8;
  float v[8];
  if (VEC) {
    load8(src, v);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = src[i];
  }
  uint32_t p[4][3];
#pragma unroll
  for (int i = 0; i < 4; ++i) ds_split(v[2 * i], v[2 * i + 1], p[i]);
#pragma unroll
  for (int i = 0; i < 3; ++i) to[i * M * per_row + at] = make_uint4(p[0][i], p[1][i], p[2][i], p[3][i]);
}

struct Args {
  const float *a, *w;  // the float32 operands
  long lda, ldw;
  float* out;          // [segments][M][ldc]
  long ldc, plane;
  int M, N, K, segments, slices_per_segment, tokens, token_tiles, items;
  int rows, raw, w_stages;  // a block's weight rows of an item, a multiple of 16 up to 128; slots of the weights' rings
  int* error_word;
};

__device__ __forceinline__ float4 load_shared4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void tmem_load8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

// Registers of a warpgroup's threads from here on.  What the warpgroups ask for together stays below what the block is launched
// with (gemm_f32_split_kernel: 96 x 640; 128 x (32 + 2 x 80 + 2 x 128)): those that take more wait for those that give some back.
template <int N>
__device__ __forceinline__ void set_registers_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void set_registers_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }

// Results of a warp's 32 rows from row0 on that are NaN: parts of infinities, and of what rounds up to one, have no sum, so these
// results are worked out once more in fp32, by the warp together, 32 k-values at a time.  A NaN among the token's values, or
// among the sums so far, is the answer, and nothing more is read.  out: row0's result for token t0.  (Out of line: eighty copies
// of it behind the sums took 15 us an item to be fetched and jumped over.)  300 rows of 19456 x 2560: all NaN 0.55 ms, 77
// with a chain of K values per thread and result; one row of NaN 0.36 (0.83), one infinity 0.69 (0.83), finite values 0.25.
__device__ __noinline__ void as_float32(const Args& p, float* out, bool open, int row0, int t0, int tokens, int k0, int k1) {
  constexpr int AT_ONCE = 8;  // values of a lane whose loads are in flight together
  const int lane = threadIdx.x & 31;
  for (int i = 0; i < tokens; ++i) {
    float* dst = out + (long)i * p.ldc;
    const float y = open ? dst[lane] : 0.f;
    uint32_t rows = __ballot_sync(0xffffffffu, y != y);
    const float* a = p.a + (long)(t0 + i) * p.lda;
    for (int k = k0 + lane; rows && k - lane < k1; k += 32 * AT_ONCE) {
      bool none = false;
#pragma unroll
      for (int e = 0; e < AT_ONCE; ++e) {
        const float x = k + 32 * e < k1 ? a[k + 32 * e] : 0.f;
        none |= x != x;
      }
      if (__any_sync(0xffffffffu, none)) rows = 0;
    }
    for (; rows; rows &= rows - 1) {
      const int r = __ffs(rows) - 1;
      const float* w = p.w + (long)(row0 + r) * p.ldw;
      float sum = 0.f;
      for (int k = k0 + lane; k - lane < k1; k += 32 * AT_ONCE) {
        float x[AT_ONCE], v[AT_ONCE];
#pragma unroll
        for (int e = 0; e < AT_ONCE; ++e) {
          const bool in = k + 32 * e < k1;
          x[e] = in ? a[k + 32 * e] : 0.f;
          v[e] = in ? w[k + 32 * e] : 0.f;
        }
#pragma unroll
        for (int e = 0; e < AT_ONCE; ++e) sum = fmaf(x[e], v[e], sum);
        if (__any_sync(0xffffffffu, sum != sum)) break;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) dst[r] = sum;
    }
  }
}

__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                      const __grid_constant__ Args p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t x_part = (uint32_t)p.tokens * 64, x_stage = 3 * x_part;
  const uint32_t x_s = smem_addr(base);             // X_STAGES x [3 parts][tokens / 2][128 B]
  const uint32_t raw_s = x_s + X_STAGES * x_stage;  // p.raw x [2 halves of k][rows][128 B]: the weights as they are
  const uint32_t raw_half = (uint32_t)p.rows * 128;
  enum { D_FULL = 0, D_EMPTY = 2, W_FULL = 4, W_EMPTY = W_FULL + W_STAGES, X_FULL = W_EMPTY + W_STAGES, X_EMPTY = X_FULL + X_STAGES,
         RAW_FULL = X_EMPTY + X_STAGES, RAW_EMPTY = RAW_FULL + MOST_RAW, DRAINED = RAW_EMPTY + MOST_RAW, BARS };
  __shared__ __align__(8) unsigned long long bars[BARS];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const uint32_t bar0 = smem_addr(&bars[0]);
  auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
  int issued = 0;  // slices whose boxes this thread has asked for
  if (tid == 0) {
    abort_flag = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(D_FULL + i), 1);
      mbar_init(bar(D_EMPTY + i), 16);  // the sums' warps of both blocks (used in the leader)
    }
    for (int i = 0; i < W_STAGES; ++i) {
      mbar_init(bar(W_FULL + i), 16);  // the weights' warps of both blocks (used in the leader)
      mbar_init(bar(W_EMPTY + i), 1);
    }
    for (int i = 0; i < X_STAGES; ++i) {
      mbar_init(bar(X_FULL + i), 1);
      mbar_init(bar(X_EMPTY + i), 1);
    }
    for (int i = 0; i < p.raw; ++i) {
      mbar_init(bar(RAW_FULL + i), 1);
      mbar_init(bar(RAW_EMPTY + i), 8);  // the weights' warps
    }
    mbar_init(bar(DRAINED), 1);
    mbar_init_fence();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_addr(&tmem_base_s)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before anything arrives on them
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;
  const int slices = (p.K + SLICE - 1) / SLICE;
  struct Item {
    int row0, token0, segment, first, count;  // this block's rows; slices first .. first + count - 1
  };
  auto item_at = [&](int i) {
    Item it;
    const int rest = i / p.token_tiles;
    it.token0 = (i - rest * p.token_tiles) * p.tokens;
    const int tile = rest / p.segments;
    it.segment = rest - tile * p.segments;
    it.row0 = (tile * 2 + (int)rank) * p.rows;
    it.first = it.segment * p.slices_per_segment;
    it.count = min(p.slices_per_segment, slices - it.first);
    return it;
  };

  const int warp_u = __shfl_sync(0xffffffffu, warp, 0);
  if (warp_u < 4) set_registers_down<32>();
  if (warp == 0) {  // ---- this block's half of the tokens' parts ----
    if (lane == 0) {
      const uint32_t leader_full = map_to_cta(bar(X_FULL), 0);
      int st = 0;
      uint32_t phase = 1;
      bool ok = true;
      for (int i = pair; i < p.items && ok; i += pairs) {
        const Item it = item_at(i);
        for (int c = 0; c < it.count; ++c) {
          ok = mbar_wait(bar(X_EMPTY + st), phase, &abort_flag);
          if (!ok) break;
          if (rank == 0) mbar_expect_tx(bar(X_FULL + st), 2 * x_stage);  // this block's boxes and the peer's
#ifndef Q3_TEST_WITHHOLD_A_BOX  // (a test build leaves the tokens' boxes out: the stage never fills, a wait runs out)
          for (int q = 0; q < 3; ++q)
            tma_load_3d_pair(x_s + st * x_stage + q * x_part, &xmap, leader_full + 8 * st, (it.first + c) * SLICE,
                             it.token0 + (int)rank * (p.tokens / 2), q);
#endif
          ++issued;
          if (++st == X_STAGES) st = 0, phase ^= 1;
        }
      }
    }
  } else if (warp_u == 1) {  // ---- products, issued by the leader ----
    if (rank == 0) {
      const bool leader = elect_one();
      const uint32_t idesc = umma_idesc(2 * ROWS, p.tokens);
      const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
      int s = 0, xs = 0, ws = 0;
      uint32_t x_phase = 0, w_phase = 0;
      bool ok = true;
      for (int i = pair; i < p.items && ok; i += pairs) {
        const int count = item_at(i).count;
        for (int c = 0; c < count; ++c, ++s) {
          const int st = s & 1;
          const uint32_t phase = (s >> 1) & 1;
          // (the three at once: one after the other they would cost three times the wait's latency)
          const bool d = mbar_try_wait_cluster(bar(D_EMPTY + st), phase ^ 1), f = mbar_try_wait_cluster(bar(W_FULL + ws), w_phase),
                     t = mbar_try_wait_cluster(bar(X_FULL + xs), x_phase);
          if (!__all_sync(0xffffffffu, d & f & t))
            ok = __all_sync(0xffffffffu, mbar_wait_cluster(bar(D_EMPTY + st), phase ^ 1, &abort_flag) &&
                                             mbar_wait_cluster(bar(W_FULL + ws), w_phase, &abort_flag) &&
                                             mbar_wait_cluster(bar(X_FULL + xs), x_phase, &abort_flag));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t xd = umma_desc(x_s + xs * x_stage);
          const uint32_t acc = tmem_u + st * p.tokens, w = tmem_u + 2 * p.tokens + ws * W_COLUMNS, xp = x_part >> 4;
          if (leader) {
            auto product = [&](int wq, int xq, bool first) {  // 16 k-values are 32 bytes: 2 descriptor units
#pragma unroll
              for (int k = 0; k < SLICE / 16; ++k)
                umma_pair_tmem(acc, w + wq * 32 + 8 * k, xd + xq * xp + 2 * k, idesc, first && k == 0 ? 0u : 1u);
            };
            product(2, 0, true);
            product(0, 2, false);
            product(1, 1, false);
            product(1, 0, false);
            product(0, 1, false);
            product(0, 0, false);
            umma_commit_pair(bar(X_EMPTY + xs));
            umma_commit_pair(bar(W_EMPTY + ws));
            umma_commit_pair(bar(D_FULL + st));
          }
          __syncwarp();
          if (++xs == X_STAGES) xs = 0, x_phase ^= 1;
          if (++ws == p.w_stages) ws = 0, w_phase ^= 1;
        }
      }
    }
  } else if (warp_u == 2) {  // ---- this block's weights ----
    if (lane == 0) {
      int s = 0, st = 0;
      uint32_t phase = 1;
      bool ok = true;
      for (int i = pair; i < p.items && ok; i += pairs) {
        const Item it = item_at(i);
        for (int c = 0; c < it.count; ++c, ++s) {
          ok = mbar_wait(bar(RAW_EMPTY + st), phase, &abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar(RAW_FULL + st), 2 * raw_half);
          for (int half = 0; half < 2; ++half)
            tma_load_2d(raw_s + (2 * st + half) * raw_half, &wmap, bar(RAW_FULL + st),
                        (it.first + c) * SLICE + half * (SLICE / 2), it.row0);
          if (++st == p.raw) st = 0, phase ^= 1;
        }
      }
      // the last boxes may still be in flight when the others have given up
      for (int b = max(0, s - p.raw); b < s; ++b) mbar_wait_drain(bar(RAW_FULL + b % p.raw), (b / p.raw) & 1);
    }
  } else if (warp_u >= 4 && warp_u < 12) {  // ---- weights ----
    set_registers_down<80>();
    // a thread makes half of the slice of one row (beyond an item's rows: of its last one; these are not stored)
    const int row = min((warp_u & 3) * 32 + lane, p.rows - 1), half = (warp_u - 4) >> 2;
    const uint32_t leader_w_full = map_to_cta(bar(W_FULL), 0);
    const uint32_t raw = raw_s + half * raw_half + row * 128;
    const uint32_t to = tmem + ((uint32_t)(warp_u & 3) << 21) + 2 * p.tokens + half * 16;
    int total = 0, raw_st = 0, ws = 0;
    uint32_t raw_phase = 0, w_phase = 1;
    for (int x = pair; x < p.items; x += pairs) total += item_at(x).count;
    for (int s = 0; s < total; ++s) {
      const bool ok = mbar_wait(bar(RAW_FULL + raw_st), raw_phase, &abort_flag) &&
                      mbar_wait(bar(W_EMPTY + ws), w_phase, &abort_flag);
      if (!__all_sync(0xffffffffu, ok)) break;
      float4 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = load_shared4(raw + raw_st * 2 * raw_half + ((i ^ (row & 7)) * 16));
      uint32_t parts[3][16];  // two k-values a column
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint32_t lo[3], hi[3];
        ds_split(v[i].x, v[i].y, lo);
        ds_split(v[i].z, v[i].w, hi);
#pragma unroll
        for (int q = 0; q < 3; ++q) parts[q][2 * i] = lo[q], parts[q][2 * i + 1] = hi[q];
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) tmem_store16(to + ws * W_COLUMNS + q * 32, parts[q]);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        remote_arrive_relaxed(leader_w_full + 8 * ws);
        // (given back behind the stores of what they became: an arrival does not wait for loads that are still on their way)
        mbar_arrive(bar(RAW_EMPTY + raw_st));
      }
      if (++raw_st == p.raw) raw_st = 0, raw_phase ^= 1;
      if (++ws == p.w_stages) ws = 0, w_phase ^= 1;
    }
  } else if (warp_u >= 12) {  // ---- sums ----
    set_registers_up<128>();
    const int quarter = warp_u & 3, cols = p.tokens / 2, col0 = ((warp_u - 12) >> 2) * cols;
    const uint32_t from = tmem + ((uint32_t)(quarter * 32) << 16) + col0;
    const uint32_t leader_d_empty = map_to_cta(bar(D_EMPTY), 0);
    float sum[MOST_TOKENS / 2];
    int s = 0;
    bool ok = true;
    for (int x = pair; x < p.items && ok; x += pairs) {
      const Item it = item_at(x);
#pragma unroll
      for (int i = 0; i < MOST_TOKENS / 2; ++i) sum[i] = 0.f;
      for (int c = 0; c < it.count; ++c, ++s) {
        const int st = s & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(bar(D_FULL + st), (s >> 1) & 1, &abort_flag));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int g = 0; g < MOST_TOKENS / 2; g += 32) {
          if (g < cols) {
            uint32_t r[4][8];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (g + 8 * i < cols) tmem_load8(from + st * p.tokens + g + 8 * i, r[i]);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (g + 8 * i >= MOST_TOKENS / 2 || g + 8 * i >= cols) break;
#pragma unroll
              for (int e = 0; e < 8; ++e) sum[g + 8 * i + e] += __uint_as_float(r[i][e]);
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) remote_arrive_relaxed(leader_d_empty + 8 * st);
      }
      if (!ok) break;
      const int row0 = it.row0 + quarter * 32, t0 = it.token0 + col0;
      float* out = p.out + it.segment * p.plane + (long)t0 * p.ldc + row0;
      const int live = quarter * 32 + lane < p.rows && row0 + lane < p.N ? min(cols, p.M - t0) : 0;
      float* dst = out + lane;
      bool none = false;
#pragma unroll
      for (int i = 0; i < MOST_TOKENS / 2; ++i) {
        if (i < live) {
          *dst = sum[i];
          none |= sum[i] != sum[i];
        }
        dst += p.ldc;
      }
      if (__any_sync(0xffffffffu, none))
        as_float32(p, out, none, row0, t0, min(cols, p.M - t0), it.first * SLICE, min(p.K, (it.first + it.count) * SLICE));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_flag && rank == 0) {
    // given up: the boxes of the last X_STAGES slices (both blocks' complete on the leader's barriers) and every MMA issued so far
    // finish before tensor memory is freed and shared memory left
    if (warp == 0 && lane == 0)
      for (int j = issued > X_STAGES ? issued - X_STAGES : 0; j < issued; ++j)
        mbar_wait_drain(bar(X_FULL + j % X_STAGES), (j / X_STAGES) & 1);
    if (warp == 1 && lane == 0) {
      umma_commit_pair(bar(DRAINED));
      mbar_wait_drain(bar(DRAINED), 0);
    }
  }
  __syncthreads();
  cluster_sync_all();  // nobody leaves while the other still reads its shared memory or signals its barriers
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
  if (tid == 0 && abort_flag && p.error_word) atomicExch(p.error_word, 2);
}

// the segments' sums, in order
__global__ void __launch_bounds__(256)
add_segments(const float* __restrict__ planes, long plane, int segments, float* __restrict__ out, long ldc, int M, int N) {
  const long at = ((long)blockIdx.x * 256 + threadIdx.x) * 4;
  const long m = at / N, n = at - m * N;
  if (m >= M) return;
  float4 sum = *reinterpret_cast<const float4*>(planes + at);
  for (int s = 1; s < segments; ++s) {
    const float4 v = *reinterpret_cast<const float4*>(planes + s * plane + at);
    sum.x += v.x;
    sum.y += v.y;
    sum.z += v.z;
    sum.w += v.w;
  }
  float* dst = out + m * ldc + n;
  dst[0] = sum.x;
  dst[1] = sum.y;
  dst[2] = sum.z;
  dst[3] = sum.w;
}

// Segments of K for N features: the fewest slices one after another on 148 SMs at one token tile, against the sums that every
// segment writes and a second kernel reads.  300 tokens, us when this was chosen (for single blocks; pairs make the same rounds),
// with 1, 2, 3, 4, 6, 8 segments (the choice behind the sizes): 19456 x 2560 (2) 249, 236, 241, 253, 284, 300; 24576 x 4096 (3)
// 398, 425, 400, 431, 464, 490; 4096 x 12288 (4) 286, 212, 232, 220, 230, 238; 2560 x 9728 (7: 120) 222, 144, 124, 151, 134, 146.
// Of N and K only, whatever the device: the bits depend on it.
static inline int segments_of(int N, int K) {
  const int tiles = (N + ROWS - 1) / ROWS, slices = (K + SLICE - 1) / SLICE;
  int best = 1, best_cost = 0;
  for (int n = 1; n <= 8 && (n == 1 || n <= slices / 8); ++n) {
    const int cost = 25 * ((tiles * n + 147) / 148) * ((slices + n - 1) / n) + n * tiles;
    if (n == 1 || cost < best_cost) best = n, best_cost = cost;
  }
  return best;
}

}  // namespace split

// Segments the product's K is cut into; 0: not a product for this kernel.  The tokens must have no say in it, so the line is
// where few tokens do not lose: weights of 20 M values (one token, us, here, parts and sums included / FMA: 8192 x 2560 32 / 38,
// 7680 x 2688 32 / 39, 12288 x 2048 36 / 41, 5120 x 5120 35 / 62, 2560 x 9728 34 / 84, 24576 x 4096 83 / 125; 33 tokens of the first 33
// / 84).  (It was drawn for the single blocks, for which the first three were level; a line further down would change the bits.)
Q3_EXPORT int q3_gemm_f32_split_segments(int N, int K) {
  return N < 256 || N % 4 || K < 1024 || K % 8 || (long)N * K < 20000000 ? 0 : split::segments_of(N, K);
}

// As q3_gemm_f32.  parts: scratch of 3 * M * K bfloat16; planes: scratch of segments * M * N floats where there is more than one
// segment.  W: rows at 16-byte boundaries.  error_word: device int set to 2 if a wait inside the kernel expired.
Q3_EXPORT int q3_gemm_f32_split(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                                void* parts, float* planes, int* error_word, cudaStream_t stream) {
  using namespace split;
  const int segments = q3_gemm_f32_split_segments(N, K);
  if (!A || !W || !C || !parts || !error_word || lda < K || ldw < K || ldc < N || segments < 1 || (segments > 1 && !planes))
    return Q3_ERR_ARGUMENT;
  if (ldw % 4 || ((uintptr_t)W & 15) || ((uintptr_t)parts & 15) || ((uintptr_t)planes & 15)) return Q3_ERR_UNSUPPORTED;
  if (M == 0) return Q3_OK;
  static int pairs_on[Q3_MAX_DEVICES];  // pairs of SMs that the device runs at once with this kernel
  int& pairs = pairs_on[q3_current_device()];
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(THREADS);
  cfg.stream = stream;
  cudaLaunchAttribute cluster;
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = 2;
  cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
  cfg.attrs = &cluster;
  cfg.numAttrs = 1;
  if (!pairs) {
    int device = 0, sms = 0, n = 0;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaFuncSetAttribute(gemm_f32_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST_SMEM) != cudaSuccess)
      return Q3_ERR_LAUNCH;
    cfg.gridDim = dim3(sms / 2 * 2);
    cfg.dynamicSmemBytes = MOST_SMEM;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_f32_split_kernel, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      return Q3_ERR_UNSUPPORTED;
    }
    pairs = n < sms / 2 ? n : sms / 2;
  }
  const long work = (long)M * (K / 8);
  const unsigned blocks = (unsigned)((work + 255) / 256);
  if (lda % 4 == 0 && ((uintptr_t)A & 15) == 0)
    split_matrix<true><<<blocks, 256, 0, stream>>>(A, lda, (uint4*)parts, M, K);
  else
    split_matrix<false><<<blocks, 256, 0, stream>>>(A, lda, (uint4*)parts, M, K);
  // The token tile and a block's weight rows: whichever make the rounds over the pairs times a slice's cycles the fewest.  Those
  // are its products' (half a cycle a token and MMA), or the weights' way.
  int best = 0, rows = ROWS;
  double best_cost = 0;
  for (int n = (M + MOST_TOKENS - 1) / MOST_TOKENS, tries = 0; tries < 4; ++n, ++tries) {
    const int t = ((M + n - 1) / n + 15) / 16 * 16;
    for (int r = ROWS; r >= 48; r -= 16) {
      const long items = (long)((N + 2 * r - 1) / (2 * r)) * segments * ((M + t - 1) / t);
      const int products = 12 * t + 300, way = 11 * r > 1000 ? 11 * r : 1000;
      const double cost = (double)((items + pairs - 1) / pairs) * (products > way ? products : way);
      if (!best || cost < best_cost) best = t, rows = r, best_cost = cost;
    }
  }
  const int tiles = (N + 2 * rows - 1) / (2 * rows);
  Args p = {A, W, lda, ldw, segments > 1 ? planes : C, segments > 1 ? N : ldc, (long)M * N, M, N, K, segments, 0, best, 0, 0,
            rows, 0, 0, error_word};
  const int slices = (K + SLICE - 1) / SLICE;
  p.slices_per_segment = (slices + segments - 1) / segments;
  p.token_tiles = (M + best - 1) / best;
  p.items = tiles * segments * p.token_tiles;
  CUtensorMap map, wmap;
  Q3EncodeTiledFn encode = q3_encode_tiled();
  if (!encode) return Q3_ERR_LAUNCH;
  const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)M, 3};
  const cuuint64_t strides[2] = {(cuuint64_t)K * 2, (cuuint64_t)M * K * 2};
  const cuuint32_t box[3] = {SLICE, (cuuint32_t)best / 2, 1}, es[3] = {1, 1, 1};
  if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, parts, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return Q3_ERR_LAUNCH;
  const cuuint64_t wdims[2] = {(cuuint64_t)K, (cuuint64_t)N}, wstrides[1] = {(cuuint64_t)ldw * 4};
  const cuuint32_t wbox[2] = {SLICE / 2, (cuuint32_t)rows};
  if (encode(&wmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(W), wdims, wstrides, wbox, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return Q3_ERR_LAUNCH;
  p.raw = (MOST_SMEM - smem_bytes(rows, best, 0)) / (rows * SLICE * 4);
  if (p.raw > MOST_RAW) p.raw = MOST_RAW;
  p.w_stages = (512 - 2 * best) / W_COLUMNS < W_STAGES ? (512 - 2 * best) / W_COLUMNS : W_STAGES;
  cfg.gridDim = dim3(2 * (p.items < pairs ? p.items : pairs));
  cfg.dynamicSmemBytes = smem_bytes(rows, best, p.raw);
  if (cudaLaunchKernelEx(&cfg, gemm_f32_split_kernel, map, wmap, p) != cudaSuccess) return Q3_ERR_LAUNCH;
  if (segments > 1)
    add_segments<<<(unsigned)(((long)M * N / 4 + 255) / 256), 256, 0, stream>>>(planes, (long)M * N, segments, C, ldc, M, N);
  return q3_launch_status();
}
