// Products of up to 128 tokens on the 5th-generation tensor cores:  out[M, N] = x[M, K] W[N, K]^T, bfloat16 operands.
//
// What bounds them: the weights' stream from memory (100 MB of gate_up take 15 us at the copy rate; 48 tokens' products a
// quarter of that), as long as every SM has the same share of it and the tokens' rows, which every SM reads from L2, stay a
// fraction of what arrives there.  Hence:
//  * the weights are the row operand, the tokens the column operand; a pair of SMs (tcgen05 cta_group::2) takes 2 h weight rows,
//    h <= 128 in each of the two, and each reads half of the tokens' rows only;
//  * h is not the instruction's 128 but what deals the rows out evenly over the pairs (19,456 rows: 2 rounds of 2 x 66); the box
//    has h rows, and the instruction's other rows are worked out from whatever lies there and dropped;
//  * where the caller takes partial sums, K is cut as well (2560 rows of 9728 values: 7 ranges of 10 x 2 x 128 rows);
//  * a ring as deep as shared memory allows (some 200 KB in flight an SM), in stages of two or four k-slices: a stage costs its
//    issuers some 300 cycles whatever it holds (2560 rows of 4096 values in 2 x 18 rows: 16.7 us by single slices, 13.0 by two,
//    11.3 by four; the output head, whose slices are 20 KB: 122 / 121 / 126).
// 48 tokens, us, the library / this (partial sums and gated: with the kernel that takes them): head of 151,936 x 2560 136 / 121
// (6.4 TB/s), x 4096 211 / 193; 7 or fewer ranges of 2560 x 9728 16.9 / 13.6, 4096 x 12288 24.7 / 22.8; gated 2 x 25600 x 5120
// 99.8 / 87.6.  Finished products of a few thousand rows stay the library's (6144 x 2560 8.3 / 9.9): one round, whose ends count.
// Sums of up to 16 tokens: the accumulators round towards zero at every instruction, so one chain over 2560 values is 2.7e-6 off,
// and the streaming kernels, which add 16 chains of a sixteenth, 1.6e-7.  Here half a k-slice (two instructions) has an accumulator
// of its own, eight to a buffer; the epilogue adds eight, then those sums, rounded to nearest: 8.7e-8, and 5.0e-8 .. 1.3e-7 from 64 to
// 25,600 values (those kernels 5.0e-8 .. 9.5e-6, and never less).  8 tokens, us, one chain / this: 151936 x 2560 115.6 / 115.6, x 4096
// 188.3 / 189.2, gated 2 x 11008 x 4096 30.7 / 32.2, 2 x 25600 x 5120 77.9 / 79.3, 10240 x 5120 20.4 / 21.0, 4096 x 12288 in parts
// 19.3 / 19.9.  (A buffer for every slice: 125, 201, 42, 85, 30, 22 us: its way to the epilogue and back takes some 600 cycles.)
// From 17 tokens on one chain, as in the library's products.
// Before the kernel ahead is waited for the first ring's worth of weights is asked for into L2 (not into shared memory: that
// kernel may be the one that writes them).
//
// Persistent, one CTA per SM: warp 0 TMA producer, warp 1 MMA issuer (leader only; both with their lane chosen by elect.sync),
// warps 2..5 epilogue; two buffers in tensor memory.  Every wait is bounded; on expiry the waiter raises the block's abort
// flag and the error word, every role leaves its loop, and what is in flight is waited for (bounded again) before tensor memory
// is freed.  No load uses cluster multicast.
#include "async_tiles.cuh"

namespace {

enum { OUT_BF16 = 0, OUT_F32 = 1, OUT_SILU = 2, OUT_GELU = 3 };
constexpr int MAX_KS = 4;                            // k-slices of 64 values a stage, at most
constexpr int BK = 64, THREADS = 192, MAX_STAGES = 24, MAX_ROWS = 128, MAX_TOKENS = 128;
constexpr int ACC_COLS = 128;                        // columns of a buffer of one accumulator; two buffers
constexpr int FEW = 16, SUMS = 8, SLICE_SUMS = 2;    // up to 16 tokens: SUMS accumulators of 32 columns, two for every k-slice
constexpr int OUT_STRIDE = 132;                      // floats per token in the gated unit's buffer
constexpr int RING_BYTES = 204 * 1024;
constexpr int KS_BYTES = 14 * 1024;                 // slices up to this size go four a stage, larger ones two

struct Maps {
  CUtensorMap w, x;
};
struct Plan {
  int rows;    // h: weight rows (gated: of gate and of up each) of a CTA's tile
  int parts;   // ranges of K
  int per;     // k-slices of a range
  int tiles;   // of 2 h rows
};

template <int MODE, bool FEW_SUMS>
__global__ void __launch_bounds__(THREADS, 1)
few_tokens_kernel(const __grid_constant__ Maps maps, void* __restrict__ out, long out_ld, int M, int N, int num_kb, Plan plan,
                  int n, int ks, int stages, int* __restrict__ error_word) {
  constexpr bool GATED = MODE >= OUT_SILU;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) unsigned long long bars[2 * MAX_STAGES + 5];
  __shared__ float staged[GATED ? 32 * OUT_STRIDE : 1];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_flag;
  int issued = 0;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1, items = plan.tiles * plan.parts;
  const int a_rows = GATED ? 2 * plan.rows : plan.rows;
  const uint32_t a_bytes = (uint32_t)(a_rows * BK * 2 + 1023) & ~1023u, slice_bytes = a_bytes + n / 2 * BK * 2;
  const uint32_t full0 = smem_addr(&bars[0]), empty0 = smem_addr(&bars[MAX_STAGES]);
  const uint32_t acc_full0 = smem_addr(&bars[2 * MAX_STAGES]), acc_empty0 = smem_addr(&bars[2 * MAX_STAGES + 2]);
  const uint32_t drained = smem_addr(&bars[2 * MAX_STAGES + 4]);
  const int group = FEW_SUMS ? SUMS / SLICE_SUMS : plan.per;  // k-slices of a buffer
  constexpr int BUF_COLS = FEW_SUMS ? 32 * SUMS : ACC_COLS, TMEM_COLS = 2 * BUF_COLS;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full0 + 8 * b, 1);
      mbar_init(acc_empty0 + 8 * b, 8);  // one arrival per epilogue warp of both CTAs (used in the leader)
    }
    mbar_init(drained, 1);
    mbar_init_fence();
  }
  if (warp == 0) {
    if (elect_one() && pair < items) {
      const int tile = pair % plan.tiles, kb0 = pair / plan.tiles * plan.per;
      for (int s = 0; s < ks * stages && s < plan.per && kb0 + s < num_kb; ++s)
        asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(&maps.w),
                     "r"((kb0 + s) * BK), "r"((2 * tile + (int)rank) * plan.rows), "r"(0)
                     : "memory");
    }
    __syncwarp();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_s)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before anything arrives on them
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_s;
  pdl_wait();
  pdl_launch_dependents();

  if (warp == 0) {  // ---- TMA producer ---------------------------------------------------------------------------------
    const bool chosen = elect_one();
    const uint32_t leader_full0 = __shfl_sync(0xffffffffu, map_to_cta(full0, 0), 0), tiles0 = smem_addr(tiles);
    const uint32_t bytes = (uint32_t)(a_rows + n / 2) * BK * 2;
    int s = 0;
    uint32_t phase = 1;
    bool ok = true;
    for (int item = pair; item < items && ok; item += num_pairs) {
      const int part = item / plan.tiles, tile = item - part * plan.tiles;
      const int kb0 = part * plan.per, kb1 = min(num_kb, kb0 + plan.per), w_row = (2 * tile + (int)rank) * plan.rows;
      for (int kb = kb0; kb < kb1; kb += ks) {
        ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, phase, &abort_flag));
        if (!ok) break;
        const uint32_t dst = tiles0 + (uint32_t)(s * ks) * slice_bytes;
        const int slices = min(ks, kb1 - kb);
        if (chosen) {
          if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * slices * bytes);  // this CTA's boxes and the peer's
#pragma unroll
          for (int j = 0; j < MAX_KS; ++j) {
            if (j >= slices) break;
            tma_load_3d_pair(dst + j * slice_bytes, &maps.w, leader_full0 + 8 * s, (kb + j) * BK, w_row, 0);
#ifdef Q3_TEST_WITHHOLD_A_BOX  // (a test build leaves the tokens' boxes of a pair's last item out: its stages never fill)
            if (item + num_pairs >= items) continue;
#endif
            tma_load_2d_pair(dst + j * slice_bytes + a_bytes, &maps.x, leader_full0 + 8 * s, (kb + j) * BK, (int)rank * (n / 2));
          }
        }
        ++issued;
        if (++s == stages) s = 0, phase ^= 1;
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {  // ---- MMA issuer of the pair ---------------------------------------------------------------------
      const bool chosen = elect_one();
      const uint32_t acc0 = __shfl_sync(0xffffffffu, tmem_base, 0), tiles0 = smem_addr(tiles);
      const uint32_t idesc = umma_idesc(256, n);
      int s = 0, buf = 0;
      uint32_t phase = 0, acc_phase = 1;
      bool ok = true;
      for (int item = pair; item < items && ok; item += num_pairs) {
        const int kb0 = item / plan.tiles * plan.per, kb1 = min(num_kb, kb0 + plan.per);
        for (int g0 = kb0; g0 < kb1; g0 += group) {
          const int g1 = min(kb1, g0 + group);
          ok = __all_sync(0xffffffffu, mbar_wait_cluster(acc_empty0 + 8 * buf, acc_phase, &abort_flag));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t acc = acc0 + buf * BUF_COLS;
          for (int kb = g0; kb < g1; kb += ks) {  // (ks divides the group)
            ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, phase, &abort_flag));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a_addr = tiles0 + (uint32_t)(s * ks) * slice_bytes;
            const int slices = min(ks, g1 - kb);
            if (chosen) {
#pragma unroll
              for (int j = 0; j < MAX_KS; ++j) {
                if (j >= slices) break;
                const uint64_t a_desc = umma_desc(a_addr + j * slice_bytes), b_desc = umma_desc(a_addr + j * slice_bytes + a_bytes);
                const uint32_t to = FEW_SUMS ? acc + 32 * SLICE_SUMS * (kb - g0 + j) : acc;
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                  umma_pair(FEW_SUMS ? to + 32 * (k / 2) : to, a_desc + 2 * k, b_desc + 2 * k, idesc,
                            (FEW_SUMS ? k % 2 > 0 : kb > g0 || j > 0 || k > 0) ? 1u : 0u);
              }
              umma_commit_pair(empty0 + 8 * s);
            }
            __syncwarp();
            if (++s == stages) s = 0, phase ^= 1;
          }
          if (!ok) break;
          if (chosen) umma_commit_pair(acc_full0 + 8 * buf);
          __syncwarp();
          buf ^= 1, acc_phase ^= buf ^ 1;
        }
      }
    }
  } else {  // ---- epilogue: warp w reads TMEM lanes 32 * (w % 4) .. + 31 of this CTA ---------------------------------------
    const int quarter = warp & 3, row = quarter * 32 + lane, et = threadIdx.x - 64;
    const uint32_t leader_acc_empty0 = map_to_cta(acc_empty0, 0);
    int buf = 0;
    uint32_t phase = 0;
    for (int item = pair; item < items; item += num_pairs) {
      const int part = item / plan.tiles, tile = item - part * plan.tiles;
      const int f0 = (2 * tile + (int)rank) * plan.rows;
      uint32_t lane_addr = 0;
      float v[32] = {};  // of this row: all tokens' sums, or the next 32 tokens'
      bool lost = false;
      const int per = min(plan.per, num_kb - part * plan.per);
      for (int done = 0; done < per; done += group) {
        lost = !__all_sync(0xffffffffu, mbar_wait(acc_full0 + 8 * buf, phase, &abort_flag));
        if (lost) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        lane_addr = tmem_base + buf * BUF_COLS + ((uint32_t)(quarter * 32) << 16);
        if constexpr (!FEW_SUMS) {
          break;
        } else {
          uint32_t r[SUMS][FEW];
#pragma unroll
          for (int g = 0; g < SUMS; ++g) tmem_load16(lane_addr + 32 * g, r[g]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          if (lane == 0) remote_arrive_relaxed(leader_acc_empty0 + 8 * buf);
          buf ^= 1, phase ^= buf ^ 1;
#pragma unroll
          for (int c = 0; c < FEW; ++c) {
            float f[SUMS];
#pragma unroll
            for (int g = 0; g < SUMS; ++g) f[g] = done + g / SLICE_SUMS < per ? __uint_as_float(r[g][c]) : 0.f;
            v[c] += ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
          }
        }
      }
      if (any_gave_up(1, 128, lost)) break;
#pragma unroll 1
      for (int c0 = 0; c0 < n; c0 += 32) {
        if (!FEW_SUMS) {
          uint32_t acc[32];
          tmem_load32(lane_addr + c0, acc);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (c0 + 32 >= n) {  // the last of this buffer is in registers: hand it back to the MMA issuer
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (lane == 0) remote_arrive_relaxed(leader_acc_empty0 + 8 * buf);
            buf ^= 1, phase ^= buf ^ 1;
          }
#pragma unroll
          for (int c = 0; c < 32; ++c) v[c] = __uint_as_float(acc[c]);
        }
        if (GATED) {  // (the products go to the unit in fp32)
#pragma unroll
          for (int c = 0; c < 32; ++c) staged[c * OUT_STRIDE + row] = v[c];
          asm volatile("bar.sync 1, 128;" ::: "memory");
          const int tokens = min(32, M - c0);
          for (int j = et; j < tokens * plan.rows; j += 128) {
            const int c = j / plan.rows, f = j - c * plan.rows;
            const float* src = staged + c * OUT_STRIDE + f;
            if (f0 + f < N)
              static_cast<bf16*>(out)[(c0 + c) * out_ld + f0 + f] =
                  from_f32<bf16>(gated_unit(src[0], src[plan.rows], MODE == OUT_GELU));
          }
          asm volatile("bar.sync 1, 128;" ::: "memory");  // the buffer is free again
        } else if (row < plan.rows && f0 + row < N) {
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            if (c0 + c >= M) break;
            if (MODE == OUT_F32)
              static_cast<float*>(out)[(part * (long)M + c0 + c) * out_ld + f0 + row] = v[c];
            else
              static_cast<bf16*>(out)[(c0 + c) * out_ld + f0 + row] = from_f32<bf16>(v[c]);
          }
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_flag && rank == 0) {
    // given up: the boxes of the last ring's k-slices (both CTAs' complete on the leader's barriers) and every MMA issued so far
    // finish before tensor memory is freed and shared memory left
    if (warp == 0 && lane == 0)
      for (int j = issued > stages ? issued - stages : 0; j < issued; ++j)
        mbar_wait_drain(full0 + 8 * (j % stages), (j / stages) & 1);
    if (warp == 1 && lane == 0) {
      umma_commit_pair(drained);
      mbar_wait_drain(drained, 0);
    }
  }
  __syncthreads();
  cluster_sync_all();  // nobody leaves while the other still reads its shared memory or signals its barriers
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
  if (threadIdx.x == 0 && abort_flag && error_word) atomicExch(error_word, 1);
}

int tokens_padded(int M) { return (M + 31) / 32 * 32; }  // the epilogue takes 32 columns at a time

// Rounds, rows and ranges that leave an SM with the fewest bytes to take in: weights, half as much for the tokens' rows (they come
// from L2), what partial sums cost on their way out and back in, and 8 KB an item for its ends.
// (the padded token count decides, not M)
Plan plan_of(int n, int N, int K, bool gated, int most_parts, int pairs) {
  const int num_kb = (K + BK - 1) / BK, cap = gated ? MAX_ROWS / 2 : MAX_ROWS;
  Plan best = {0, 1, num_kb, 0};
  double least = 0;
  for (int parts = 1; parts <= most_parts && parts <= num_kb; ++parts) {
    const int per = (num_kb + parts - 1) / parts;
    if ((num_kb + per - 1) / per != parts) continue;
    for (int rounds = 1, options = 0; options < 3; ++rounds) {
      const int most_tiles = pairs * rounds / parts;
      if (most_tiles < 1) continue;
      const int rows = (N + 2 * most_tiles - 1) / (2 * most_tiles);
      if (rows > cap) continue;
      ++options;
      const double bytes = rounds * ((double)per * BK * 2 * (rows * (gated ? 2 : 1) + 0.5 * (n / 2)) + 8192) +
                           (parts > 1 ? 8.0 * parts * n * N / (2 * pairs) : 0.0);
      if (!best.rows || bytes < least) {
        best = {rows, parts, per, (N + 2 * rows - 1) / (2 * rows)};
        least = bytes;
      }
    }
  }
  return best;
}

template <int MODE, bool FEW_SUMS>
int pairs_of() {  // pairs of SMs the device runs at once with this kernel
  static int pairs_on[Q3_MAX_DEVICES];
  int& pairs = pairs_on[q3_current_device()];
  if (!pairs) {
    int device = 0, sms = 0, n = 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = RING_BYTES;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaFuncSetAttribute(few_tokens_kernel<MODE, FEW_SUMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_BYTES) != cudaSuccess)
      return 0;
    cfg.gridDim = dim3(sms / 2 * 2);
    if (cudaOccupancyMaxActiveClusters(&n, few_tokens_kernel<MODE, FEW_SUMS>, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      return 0;
    }
    pairs = n < sms / 2 ? n : sms / 2;
  }
  return pairs;
}

template <int MODE, bool FEW_SUMS>
int launch_as(const void* x, long x_ld, const void* w, long w_ld, void* out, long out_ld, int parts, int M, int N, int K,
           int* error_word, cudaStream_t stream) {
  constexpr bool GATED = MODE >= OUT_SILU;
  const int pairs = pairs_of<MODE, FEW_SUMS>();
  if (!pairs) return Q3_ERR_UNSUPPORTED;
  // (given parts: the caller's planes are of that many)
  const int n = tokens_padded(M);
  const Plan plan = plan_of(n, N, K, GATED, parts, pairs);
  if (!plan.rows || (parts > 1 && plan.parts != parts)) return Q3_ERR_UNSUPPORTED;
  const int a_rows = GATED ? 2 * plan.rows : plan.rows;
  Maps maps;
  const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)N, GATED ? 2u : 1u};
  const cuuint64_t strides[2] = {(cuuint64_t)w_ld * 2, (cuuint64_t)w_ld * 2 * N};
  const cuuint32_t box[3] = {BK, (cuuint32_t)plan.rows, GATED ? 2u : 1u}, es[3] = {1, 1, 1};
  Q3EncodeTiledFn encode = q3_encode_tiled();
  if (!encode ||
      encode(&maps.w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(w), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS ||
      !q3_bf16_map(&maps.x, x, M, K, x_ld, n / 2))
    return Q3_ERR_LAUNCH;
  const int slice_bytes = ((a_rows * BK * 2 + 1023) & ~1023) + n / 2 * BK * 2, ks = slice_bytes <= KS_BYTES ? 4 : 2,
            stage_bytes = ks * slice_bytes;
  // (the instruction reads 128 rows from a slice's first byte on, also of the ring's last slice)
  const int room = RING_BYTES - 1024 - (slice_bytes < 16384 ? 16384 - slice_bytes : 0);
  const int stages = room / stage_bytes < MAX_STAGES ? room / stage_bytes : MAX_STAGES;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  const int items = plan.tiles * plan.parts;
  cfg.gridDim = dim3(2 * (items < pairs ? items : pairs));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = RING_BYTES;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = q3_pdl_enabled() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, few_tokens_kernel<MODE, FEW_SUMS>, maps, out, out_ld, M, N, (K + BK - 1) / BK, plan, n, ks, stages,
                            error_word) == cudaSuccess
             ? Q3_OK
             : Q3_ERR_LAUNCH;
}

template <int MODE>
int launch(const void* x, long x_ld, const void* w, long w_ld, void* out, long out_ld, int parts, int M, int N, int K,
           int* error_word, cudaStream_t stream) {
  return M <= FEW ? launch_as<MODE, true>(x, x_ld, w, w_ld, out, out_ld, parts, M, N, K, error_word, stream)
                  : launch_as<MODE, false>(x, x_ld, w, w_ld, out, out_ld, parts, M, N, K, error_word, stream);
}

}  // namespace

// How many planes of partial sums the product is best cut into, at most most_parts (1: none).
Q3_EXPORT int q3_gemm_few_parts(int M, int N, int K, int most_parts) {
  if (M < 1 || M > MAX_TOKENS || N < 1 || K < 1 || most_parts < 1) return 1;
  const int pairs = pairs_of<OUT_F32, false>();
  if (!pairs) return 1;
  // (found again when it is asked for as the most there may be: the least of fewer is the same)
  return plan_of(tokens_padded(M), N, K, false, most_parts, pairs).parts;
}

// mode 0: out bf16 [M, N]; 1: fp32, with parts > 1 that many planes [parts, M, N] whose sum is the product; 2, 3: w [2N, K] (gate
// rows, then up rows), out bf16 [M, N] = silu(gate) * up (3: gelu, tanh form).
// 1 <= M <= 128; K, x_ld and w_ld multiples of 8, x and w 16-byte aligned.
Q3_EXPORT int q3_gemm_few_tokens(int mode, const void* x, long x_ld, const void* w, long w_ld, void* out, long out_ld, int parts,
                                 int M, int N, int K, int* error_word, cudaStream_t stream) {
  if (!x || !w || !out || M < 0 || N < 1 || K < 1 || parts < 1 || (parts > 1 && mode != OUT_F32)) return Q3_ERR_ARGUMENT;
  if (M == 0) return Q3_OK;
  if (M > MAX_TOKENS || K % 8 || x_ld % 8 || w_ld % 8 || x_ld < K || w_ld < K || (((uintptr_t)x | (uintptr_t)w) & 15))
    return Q3_ERR_UNSUPPORTED;
  switch (mode) {
    case OUT_BF16: return launch<OUT_BF16>(x, x_ld, w, w_ld, out, out_ld, parts, M, N, K, error_word, stream);
    case OUT_F32: return launch<OUT_F32>(x, x_ld, w, w_ld, out, out_ld, parts, M, N, K, error_word, stream);
    case OUT_SILU: return launch<OUT_SILU>(x, x_ld, w, w_ld, out, out_ld, parts, M, N, K, error_word, stream);
    case OUT_GELU: return launch<OUT_GELU>(x, x_ld, w, w_ld, out, out_ld, parts, M, N, K, error_word, stream);
    default: return Q3_ERR_ARGUMENT;
  }
}
