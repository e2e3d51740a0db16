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
// Weights are the 128 rows of an MMA, tokens its 16 to 160 columns.  Roles of a block (one per SM, persistent over items of
// (128 weight rows, segment, token tile), token tiles of the same weights side by side):
//   warp 0       TMA: the tokens' three parts (made beforehand by split_matrix) of a slice, one box of 64 columns per part
//   warp 1       MMA issuer
//   warps 2..9   weights: 16 bytes of float32 per lane from global memory, a slice ahead in registers, split and written in the
//                128-byte swizzle; and sums: the accumulators of the slice before (two buffers in tensor memory) into
//                registers, a row and half of the columns a thread; at the item's end they are stored
// Up to 32 tokens (kernel of its own, the same sums): where few products follow, the weights' loads a slice ahead, 2600 cycles under
// load, were what a slice waited for.
//   warp 10      TMA: the weights' slices as they are, up to eight ahead in what shared memory the few tokens leave
//   warps 2..9   read them from there; an item has 48 to 128 rows, whichever fills the rounds over the SMs
// What bounds it: with 160 tokens a slice takes 2700 cycles, its 24 products 1900 of them, the sums and the weights' way (wait,
// split, write, hand-over) the rest; with up to 32 tokens and 128 rows 1800, the weights' way, which is 4.5 TB/s.  us, on the FMA
// pipes / here: 300 tokens 19456 x 2560 701 / 218, 2560 x 9728 412 / 112; one token 19456 x 2560 82 / 73 (105 without that kernel),
// 24576 x 4096 129 / 105 (145), 151936 x 2560 383 / 345 (495), 4096 x 12288 111 / 64 (82).
#include "async_tiles.cuh"
#include "split_mma.cuh"

namespace split {

constexpr int ROWS = 128, SLICE = 64, MOST_TOKENS = 160, FEW_TOKENS = 32;
constexpr int AHEAD = 4;  // slices
constexpr int W_PART = ROWS * 128, W_STAGE = 3 * W_PART;
constexpr int MOST_RAW = 8;  // few tokens: slices of weights as they are, on their way
constexpr int threads(int most) { return (most == FEW_TOKENS ? 11 : 10) * 32; }
constexpr int smem_bytes(int rows, int tokens, int raw) { return 768 * (rows + tokens) + raw * rows * SLICE * 4 + 1024; }
constexpr int MOST_SMEM = 231936;
enum { BAR_W_FULL = 0, BAR_X_FULL = 2, BAR_EMPTY = 4, BAR_D_FULL = 6, BAR_D_EMPTY = 8, BAR_END = 10, BAR_RAW_FULL = 11,
       BAR_RAW_EMPTY = BAR_RAW_FULL + MOST_RAW, NUM_BARS = BAR_RAW_EMPTY + MOST_RAW };

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
  int rows, raw;  // weight rows of an item: 128, with few tokens a multiple of 16 up to it; slots of the weights' ring
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

// MOST: tokens that there are registers for.  FEW_TOKENS: the weights come by TMA (warp 10) into a ring of their own.
template <int MOST>
__global__ void __launch_bounds__(threads(MOST), 1)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                      const __grid_constant__ Args p) {
  constexpr bool FEW = MOST == FEW_TOKENS;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t x_part = (uint32_t)p.tokens * 128, x_stage = 3 * x_part;
  // (an MMA reads 128 rows: behind the item's own it finds what follows in shared memory, and makes rows that are not stored)
  const uint32_t w_part = FEW ? (uint32_t)p.rows * 128 : W_PART, w_stage = 3 * w_part, raw_stage = (uint32_t)p.rows * SLICE * 4;
  unsigned char* w_s = base;                       // 2 x [3 parts][rows][128 B]
  const uint32_t x_s = smem_addr(base) + 2 * w_stage;  // 2 x [3 parts][tokens][128 B]
  const uint32_t raw_s = x_s + 2 * x_stage;            // FEW: p.raw x [rows][256 B]
  __shared__ __align__(8) unsigned long long bars[NUM_BARS];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t bar0 = smem_addr(&bars[0]);
  auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
  if (tid == 0) {
    abort_flag = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(BAR_W_FULL + i), 8);   // the weights' warps
      mbar_init(bar(BAR_X_FULL + i), 1);
      mbar_init(bar(BAR_EMPTY + i), 1);
      mbar_init(bar(BAR_D_FULL + i), 1);
      mbar_init(bar(BAR_D_EMPTY + i), 8);  // the sums' warps
    }
    mbar_init(bar(BAR_END), 1);
    for (int i = 0; FEW && i < p.raw; ++i) {
      mbar_init(bar(BAR_RAW_FULL + i), 1);
      mbar_init(bar(BAR_RAW_EMPTY + i), 8);  // the weights' warps
    }
    mbar_init_fence();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_addr(&tmem_base_s)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;
  const int slices = (p.K + SLICE - 1) / SLICE;
  struct Item {
    int row0, token0, segment, first, count;  // slices first .. first + count - 1
  };
  auto item_at = [&](int i) {
    Item it;
    const int rest = i / p.token_tiles;
    it.token0 = (i - rest * p.token_tiles) * p.tokens;
    const int tile = rest / p.segments;
    it.segment = rest - tile * p.segments;
    it.row0 = tile * p.rows;
    it.first = it.segment * p.slices_per_segment;
    it.count = min(p.slices_per_segment, slices - it.first);
    return it;
  };

  const int warp_u = __shfl_sync(0xffffffffu, warp, 0);
  if (warp == 0) {  // ---- the tokens' parts ----
    int s = 0;
    bool ok = true;
    for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
      const Item it = item_at(i);
      for (int c = 0; c < it.count; ++c, ++s) {
        const int st = s & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(bar(BAR_EMPTY + st), ((s >> 1) & 1) ^ 1, &abort_flag));
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(bar(BAR_X_FULL + st), x_stage);
#ifndef Q3_TEST_WITHHOLD_A_BOX  // (a test build leaves the tokens' boxes out: the stage never fills, a wait runs out)
          for (int q = 0; q < 3; ++q)
            tma_load_3d(x_s + st * x_stage + q * x_part, &xmap, bar(BAR_X_FULL + st), (it.first + c) * SLICE, it.token0, q);
#endif
        }
      }
    }
    // the last boxes may still be in flight when the others have given up
    if (lane == 0)
      for (int b = max(0, s - 2); b < s; ++b) mbar_wait_drain(bar(BAR_X_FULL + (b & 1)), (b >> 1) & 1);
  } else if (FEW && warp_u == 10) {  // ---- few tokens: the weights ----
    int s = 0, st = 0;
    uint32_t phase = 1;
    bool ok = true;
    for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
      const Item it = item_at(i);
      for (int c = 0; c < it.count; ++c, ++s) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar(BAR_RAW_EMPTY + st), phase, &abort_flag));
        if (!ok) break;
        if (lane == 0) {
          mbar_expect_tx(bar(BAR_RAW_FULL + st), raw_stage);
          tma_load_2d(raw_s + st * raw_stage, &wmap, bar(BAR_RAW_FULL + st), (it.first + c) * SLICE, it.row0);
        }
        if (++st == p.raw) st = 0, phase ^= 1;
      }
    }
    if (lane == 0)
      for (int b = max(0, s - p.raw); b < s; ++b) mbar_wait_drain(bar(BAR_RAW_FULL + b % p.raw), (b / p.raw) & 1);
  } else if (warp_u == 1) {  // ---- products ----
    // (one lane chosen by elect.sync, in a warp that runs as a whole: descriptors then stay in uniform registers, and an MMA is
    // issued every 37 cycles; chosen by its number 60 to 78)
    const bool leader = elect_one();
    const uint32_t idesc = umma_idesc(ROWS, p.tokens);
    const uint32_t w_addr = smem_addr(w_s), tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
    int s = 0;
    bool ok = true;
    for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
      const int count = item_at(i).count;
      for (int c = 0; c < count; ++c, ++s) {
        const int st = s & 1;
        const uint32_t phase = (s >> 1) & 1;
        // (the three at once: one after the other they would cost three times the wait's latency)
        const bool d = mbar_try_wait(bar(BAR_D_EMPTY + st), phase ^ 1), w = mbar_try_wait(bar(BAR_W_FULL + st), phase),
                   t = mbar_try_wait(bar(BAR_X_FULL + st), phase);
        if (!__all_sync(0xffffffffu, d & w & t))
          ok = __all_sync(0xffffffffu, mbar_wait(bar(BAR_D_EMPTY + st), phase ^ 1, &abort_flag) &&
                                           mbar_wait(bar(BAR_W_FULL + st), phase, &abort_flag) &&
                                           mbar_wait(bar(BAR_X_FULL + st), phase, &abort_flag));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t wd = umma_desc(w_addr + st * w_stage), xd = umma_desc(x_s + st * x_stage);
        const uint32_t acc = tmem_u + st * 256, xp = x_part >> 4;
        if (leader) {
          auto product = [&](int wq, int xq, bool first) {  // 16 k-values are 32 bytes: 2 descriptor units
#pragma unroll
            for (int k = 0; k < SLICE / 16; ++k)
              umma_bf16(acc, wd + wq * (w_part >> 4) + 2 * k, xd + xq * xp + 2 * k, idesc, first && k == 0 ? 0u : 1u);
          };
          product(2, 0, true);
          product(0, 2, false);
          product(1, 1, false);
          product(1, 0, false);
          product(0, 1, false);
          product(0, 0, false);
          umma_commit(bar(BAR_EMPTY + st));
          umma_commit(bar(BAR_D_FULL + st));
        }
        __syncwarp();
      }
    }
    if (leader) {  // nothing of this block's is in flight any more when the tensor memory is freed
      umma_commit(bar(BAR_END));
      mbar_wait_drain(bar(BAR_END), 0);
    }
    __syncwarp();
  } else {  // ---- weights and sums ----
    const int worker = warp - 2, quarter = warp & 3, cols = p.tokens / 2, col0 = (worker >> 2) * cols;
    const uint32_t from = tmem + ((uint32_t)(quarter * 32) << 16) + col0;
    // the 16 threads of a row are neighbours; a thread's rows are r0 + STEP i
    constexpr int STEP = FEW ? 16 : 2;
    const int r0 = (FEW ? worker * 2 : worker * 16) + (lane >> 4), kl = (lane & 15) * 4;
    unsigned char* const w_dst = w_s + r0 * 128 + (lane & 1) * 8;
    const uint32_t raw = raw_s + r0 * 256 + (lane & 15) * 16;
    float4 v[8];  // rows r0 + STEP i, k-values kl .. kl + 3 of the slice that is split next
    const float* w_row = p.w;  // the first of those rows
    int rows_left = 0;         // (rows from N on are read as that row, and not stored)
    auto item_rows = [&](const Item& it) {
      w_row = p.w + (long)min(it.row0 + r0, p.N - 1) * p.ldw + kl;
      rows_left = p.N - it.row0 - r0;
    };
    auto load = [&](int slice) {
      const float* src = w_row + slice * SLICE;
      const bool in = slice * SLICE + kl < p.K;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[i] = in ? __ldg(reinterpret_cast<const float4*>(src)) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (2 * i + 2 < rows_left) src += 2 * p.ldw;
      }
    };
    // Into L2 ahead of the loads: a slice is 128 rows of two lines, one a thread.
    auto ahead = [&](const Item& it, int slice) {
      const int row = it.row0 + (tid - 64 >> 1), k = slice * SLICE + (tid & 1) * 32;
      if (row < p.N && k < p.K) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.w + (long)row * p.ldw + k));
    };
    int raw_st = 0;  // FEW: the ring's slot that is read next
    uint32_t raw_phase = 0;
    auto load_raw = [&]() -> bool {
      if (!__all_sync(0xffffffffu, mbar_wait(bar(BAR_RAW_FULL + raw_st), raw_phase, &abort_flag))) return false;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i * 16 < p.rows) v[i] = load_shared4(raw + raw_st * raw_stage + i * 16 * 256);
      return true;
    };
    float sum[MOST / 2];
    auto add = [&](int s) -> bool {  // the accumulators of stage s
      const int st = s & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(bar(BAR_D_FULL + st), (s >> 1) & 1, &abort_flag))) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int g = 0; g < MOST / 2; g += 16) {
        if (g < cols) {
          uint32_t r[2][8];
          tmem_load8(from + st * 256 + g, r[0]);
          if (g + 8 < cols) tmem_load8(from + st * 256 + g + 8, r[1]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int e = 0; e < 8; ++e) sum[g + e] += __uint_as_float(r[0][e]);
          if (g + 8 < cols) {
#pragma unroll
            for (int e = 0; e < 8; ++e) sum[g + 8 + e] += __uint_as_float(r[1][e]);
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(BAR_D_EMPTY + st));
      return true;
    };
    bool ok = true;
    if (FEW) {
      ok = load_raw();
    } else {
      const Item it = item_at(blockIdx.x);
      item_rows(it);
      load(it.first);
      for (int c = 1; c < AHEAD && c < it.count; ++c) ahead(it, it.first + c);
    }
    int s = 0;
    for (int x = blockIdx.x; x < p.items && ok; x += gridDim.x) {
      const Item it = item_at(x);
      const int after = x + (int)gridDim.x;
      const Item nx = item_at(after < p.items ? after : x);
#pragma unroll
      for (int i = 0; i < MOST / 2; ++i) sum[i] = 0.f;
      for (int c = 0; c < it.count && ok; ++c, ++s) {
        const int st = s & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(bar(BAR_EMPTY + st), ((s >> 1) & 1) ^ 1, &abort_flag));
        if (!ok) break;
        unsigned char* dst = w_dst + st * w_stage;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (FEW && i * 16 >= p.rows) break;  // (rows beyond stay as they are: a result depends on its own row only)
          uint32_t lo[3], hi[3];
          ds_split(v[i].x, v[i].y, lo);
          ds_split(v[i].z, v[i].w, hi);
          const int at = i * STEP * 128 + ((((lane & 15) >> 1) ^ ((r0 + STEP * i) & 7)) * 16);
#pragma unroll
          for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(dst + q * w_part + at) = make_uint2(lo[q], hi[q]);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(BAR_W_FULL + st));
        if (FEW) {
          // (given back behind the stores of what they became: an arrival does not wait for loads that are still on their way)
          if (lane == 0) mbar_arrive(bar(BAR_RAW_EMPTY + raw_st));
          if (++raw_st == p.raw) raw_st = 0, raw_phase ^= 1;
          if ((c + 1 < it.count || after < p.items) && !(ok = load_raw())) break;
        } else {
          if (c + 1 < it.count) {
            load(it.first + c + 1);
          } else if (after < p.items) {
            item_rows(nx);
            load(nx.first);
          }
          if (c + AHEAD < it.count) ahead(it, it.first + c + AHEAD);
          else if (after < p.items && c + AHEAD - it.count < nx.count) ahead(nx, nx.first + c + AHEAD - it.count);
        }
        if (c > 0) ok = add(s - 1);  // while this slice's products run
      }
      if (ok) ok = add(s - 1);
      if (!ok) break;
      const int row0 = it.row0 + quarter * 32, t0 = it.token0 + col0;
      float* out = p.out + it.segment * p.plane + (long)t0 * p.ldc + row0;
      bool none = false;
      if (quarter * 32 + lane < p.rows && row0 + lane < p.N) {
#pragma unroll
        for (int i = 0; i < MOST / 2; ++i) {
          if (i < cols && t0 + i < p.M) {
            out[(long)i * p.ldc + lane] = sum[i];
            none |= sum[i] != sum[i];
          }
        }
      }
      if (__any_sync(0xffffffffu, none))
        as_float32(p, out, none, row0, t0, min(cols, p.M - t0), it.first * SLICE, min(p.K, (it.first + it.count) * SLICE));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
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
// segment writes and a second kernel reads.  300 tokens, us when this was chosen, with 1, 2, 3, 4, 6, 8 segments (the choice behind
// the sizes): 19456 x 2560 (2) 249, 236, 241, 253, 284, 300; 24576 x 4096 (3) 398, 425, 400, 431, 464, 490; 4096 x 12288 (4) 286,
// 212, 232, 220, 230, 238; 2560 x 9728 (7: 120) 222, 144, 124, 151, 134, 146.  Of N and K only, whatever the device: the bits
// depend on it.
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
// where few tokens do not lose: weights of 20 M values (one token, us, here / FMA: 8192 x 2560 38 / 41, 7680 x 2688 38 / 43,
// 12288 x 2048 44 / 43, 5120 x 5120 44 / 64, 2560 x 9728 42 / 88).
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
  static int sms_on[Q3_MAX_DEVICES];
  const int device = q3_current_device();
  if (!sms_on[device]) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaFuncSetAttribute(gemm_f32_split_kernel<MOST_TOKENS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem_bytes(ROWS, MOST_TOKENS, 0)) != cudaSuccess ||
        cudaFuncSetAttribute(gemm_f32_split_kernel<FEW_TOKENS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             MOST_SMEM) != cudaSuccess)
      return Q3_ERR_LAUNCH;
    sms_on[device] = sms;
  }
  const int sms = sms_on[device];
  const long work = (long)M * (K / 8);
  const unsigned blocks = (unsigned)((work + 255) / 256);
  if (lda % 4 == 0 && ((uintptr_t)A & 15) == 0)
    split_matrix<true><<<blocks, 256, 0, stream>>>(A, lda, (uint4*)parts, M, K);
  else
    split_matrix<false><<<blocks, 256, 0, stream>>>(A, lda, (uint4*)parts, M, K);
  // The token tile: rounds over the SMs times a slice's time, which is that of shared memory (a token's parts are read by 24
  // products and written once, the weights' read and written) or of the weights' bytes.
  int best = 0, rows = ROWS;
  double best_cost = 0;
  if (M <= FEW_TOKENS) {
    // One token tile, and the rows of an item whichever make the rounds times a slice's cycles (its products', or its weights' way)
    // the fewest.  One token, us with 128 / 112 / 96 / 80 rows: 19456 x 2560 79 / 75 / 73 / 87, 24576 x 4096 106 / 118 / 130 / 142,
    // 8192 x 2560 40 / 38 / 54 / 52, 151936 x 2560 345 / 372 / 386 / 429.
    best = M <= 16 ? 16 : 32;
    for (int r = ROWS; r >= 48; r -= 16) {
      const long items = (long)((N + r - 1) / r) * segments;
      const double cost = (double)((items + sms - 1) / sms) * (600 + 15 * r / 2 < 1040 ? 1040 : 600 + 15 * r / 2);
      if (r == ROWS || cost < best_cost) rows = r, best_cost = cost;
    }
  }
  const int tiles = (N + rows - 1) / rows;
  for (int n = (M + MOST_TOKENS - 1) / MOST_TOKENS, tries = 0; M > FEW_TOKENS && tries < 4; ++n, ++tries) {
    const int t = ((M + n - 1) / n + 15) / 16 * 16;
    const long items = (long)tiles * segments * ((M + t - 1) / t);
    const double slice = 24 * (4096 + 32 * t) + W_STAGE + 384 * t;
    const double cost = (double)((items + sms - 1) / sms) * (slice < 180000 ? 180000 : slice);
    if (!best || cost < best_cost) best = t, best_cost = cost;
  }
  Args p = {A, W, lda, ldw, segments > 1 ? planes : C, segments > 1 ? N : ldc, (long)M * N, M, N, K, segments, 0, best, 0, 0, rows, 0,
            error_word};
  const int slices = (K + SLICE - 1) / SLICE;
  p.slices_per_segment = (slices + segments - 1) / segments;
  p.token_tiles = (M + best - 1) / best;
  p.items = tiles * segments * p.token_tiles;
  CUtensorMap map, wmap;
  Q3EncodeTiledFn encode = q3_encode_tiled();
  if (!encode) return Q3_ERR_LAUNCH;
  const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)M, 3};
  const cuuint64_t strides[2] = {(cuuint64_t)K * 2, (cuuint64_t)M * K * 2};
  const cuuint32_t box[3] = {SLICE, (cuuint32_t)best, 1}, es[3] = {1, 1, 1};
  if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, parts, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return Q3_ERR_LAUNCH;
  const cuuint64_t wdims[2] = {(cuuint64_t)K, (cuuint64_t)N}, wstrides[1] = {(cuuint64_t)ldw * 4};
  const cuuint32_t wbox[2] = {SLICE, (cuuint32_t)rows};
  if (best <= FEW_TOKENS &&
      encode(&wmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(W), wdims, wstrides, wbox, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return Q3_ERR_LAUNCH;  // (many tokens: not used)
  const int grid = p.items < sms ? p.items : sms;
  if (best <= FEW_TOKENS) {
    p.raw = (MOST_SMEM - smem_bytes(rows, best, 0)) / (rows * SLICE * 4);
    if (p.raw > MOST_RAW) p.raw = MOST_RAW;
    gemm_f32_split_kernel<FEW_TOKENS><<<grid, threads(FEW_TOKENS), smem_bytes(rows, best, p.raw), stream>>>(map, wmap, p);
  } else {
    gemm_f32_split_kernel<MOST_TOKENS><<<grid, threads(MOST_TOKENS), smem_bytes(rows, best, 0), stream>>>(map, wmap, p);
  }
  if (segments > 1)
    add_segments<<<(unsigned)(((long)M * N / 4 + 255) / 256), 256, 0, stream>>>(planes, (long)M * N, segments, C, ldc, M, N);
  return q3_launch_status();
}
