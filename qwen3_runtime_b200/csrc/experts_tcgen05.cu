// The routed experts' products for prompt portions, in bfloat16 on the 5th-generation tensor cores.
//
//   gather      xs[place(slot)] = h[token(slot)] (times the slot's weight where it multiplies the expert's input,
//               rounded to bfloat16): the slots' rows side by side, grouped by expert
//   gate_up     mid[r] = glu(W_gate_e xs[r], W_up_e xs[r])   (or relu(W_up_e xs[r])^2 without a gate)
//   down        y[r] = W_down_e mid[r]
//
// What bounds them: with a few hundred slots per expert the weights' bytes and the products' operations
// take about the same time (64 experts of 2 x 1408 x 2048, 12,288 slots: 113 us of HBM reads for gate_up against 86 us
// of MMAs at the measured peak), so every weight has to be read from memory once only and MMAs must not
// be spent on padding.  Hence the weights are the row operand and the slots the column operand: one tile is 256
// weight rows x up to 256 slots of ONE expert, the instruction's N is the slots there are (a multiple of 32, not of
// 128), and an expert with at most 256 slots has its weights read by one tile only.  A tile runs on a pair of SMs
// (tcgen05 cta_group::2): per 16 k-values a CTA's shared memory takes in and gives out 4 KB of weights and at most
// 4 KB of slots, where one CTA alone would need twice the slots and fall behind its tensor pipe.
// For the gated unit each CTA's 128 rows are 64 gate rows and the 64 up rows of the same features, so that both
// halves of a feature meet in one CTA's epilogue.
//
// Persistent, one CTA per SM, three roles as in gemm_tcgen05.cu: warp 0 TMA producer (6 stages of 16 KB weights + at most 16 KB
// slots), warp 1 MMA issuer (leader only), warps 2..9 epilogue in two groups (accumulators double-buffered in tensor memory; 32
// slots at a time through shared memory as bfloat16, so that a slot's features are stored side by side).
// What held it back beside the bytes: the issue of up to six boxes a k-slice by one lane (60 to 80 cycles each; two boxes now,
// their lane chosen by elect.sync) and the gated unit in four warps (26,000 cycles a tile of 192 slots, its MMAs 12,300).  2048
// tokens, us, gate_up / down: 64 experts of 2 x 1408 x 2048, top 6: 180 / 94, two boxes 170 / 92, two groups 158 / 90; 32 of 2 x
// 2048 x 4096, top 4: 330 / 168, 268 / 137, 262 / 136.  512 tokens of the first: 146 / 84 -> 139 / 82 (5.3 TB/s of weights).
// Feature tiles of a chunk are neighbours in the tile order: the pairs share its slots' rows in L2.
//
// Every wait is bounded; on expiry the waiter raises the block's abort flag and the error word, every role leaves its
// loop, what is in flight is waited for (bounded again) before tensor memory is freed.  No load uses cluster multicast.
#include "async_tiles.cuh"

namespace {

enum { UNIT_NONE = 0, UNIT_RELU2 = 1, UNIT_GLU = 2 };
constexpr int BK = 64;
constexpr int STAGES = 6;
constexpr int THREADS = 64 + 2 * 128;     // two groups of four epilogue warps
constexpr int A_BYTES = 128 * BK * 2;     // this CTA's 128 weight rows
constexpr int B_ROWS = 32, B_MAPS = 4;    // slots per TMA box: 32, 64, 96 or 128, a tensor map for each
constexpr int B_BYTES = 128 * BK * 2;     // at most 128 slots per CTA
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int MAX_SLOTS = 256;            // slots per tile
constexpr int ACC_COLS = 256, TMEM_COLS = 512;
constexpr int OUT_STRIDE = 160;           // bfloat16 per slot in a group's buffer: 128 rows; two slots cover all banks

struct Tile {
  int expert, row0, rows, n, f;  // slots row0 .. row0 + rows of the grouped order; n: rows rounded up to 32; f: feature tile
};

__device__ __forceinline__ Tile tile_at(int tile, int ftiles, const int* __restrict__ offsets,
                                        const int* __restrict__ tile_offsets, int E) {
  Tile t;
  const int chunk = tile / ftiles;
  t.f = tile - chunk * ftiles;
  int lo = 0, hi = E;  // the last expert with tile_offsets[e] <= chunk
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (tile_offsets[mid] <= chunk) lo = mid; else hi = mid;
  }
  t.expert = lo;
  const int first = offsets[lo], count = offsets[lo + 1] - first;
  const int chunks = (count + MAX_SLOTS - 1) / MAX_SLOTS;
  const int size = ((count + chunks - 1) / chunks + 31) & ~31;  // an expert's slots in equal chunks, 256 at most
  t.row0 = first + (chunk - tile_offsets[lo]) * size;
  t.rows = min(size, first + count - t.row0);
  t.n = (t.rows + 31) & ~31;
  return t;
}

// The tensor maps of a product: weights as [2E][N][K] (gated: a box is 64 rows of a gate and the 64 of its up matrix) or
// [E * N][K], and the slots' rows with every height of a box.
struct Maps {
  CUtensorMap w, x[B_MAPS];
};

template <int UNIT>
__global__ void __launch_bounds__(THREADS, 1)
expert_tcgen05_kernel(const __grid_constant__ Maps maps, bf16* __restrict__ out, int N, int K, int E,
                      const int* __restrict__ offsets, const int* __restrict__ tile_offsets, float limit, float alpha,
                      float up_offset, int* __restrict__ error_word) {
  constexpr int TILE_F = UNIT == UNIT_GLU ? 128 : 256;  // features per tile; half of them in each CTA
  extern __shared__ unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  bf16* stage_out = reinterpret_cast<bf16*>(tiles + (size_t)STAGES * STAGE_BYTES);  // [2 groups][32 slots][OUT_STRIDE]
  __shared__ __align__(8) unsigned long long bars[2 * STAGES + 5];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_flag;
  int issued = 0;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int num_kb = (K + BK - 1) / BK;
  const int ftiles = (N + TILE_F - 1) / TILE_F;
  const uint32_t full0 = smem_addr(&bars[0]), empty0 = smem_addr(&bars[STAGES]);
  const uint32_t acc_full0 = smem_addr(&bars[2 * STAGES]), acc_empty0 = smem_addr(&bars[2 * STAGES + 2]);
  const uint32_t drained = smem_addr(&bars[2 * STAGES + 4]);

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full0 + 8 * b, 1);
      mbar_init(acc_empty0 + 8 * b, 16);  // one arrival per epilogue warp of both CTAs (used in the leader)
    }
    mbar_init(drained, 1);
    mbar_init_fence();
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
  pdl_wait();  // the grouping and the slots' rows come from the kernels before
  pdl_launch_dependents();
  const int num_tiles = tile_offsets[E] * ftiles;

  if (warp == 0) {  // ---- TMA producer: one lane chosen by elect.sync, two boxes a k-slice ---------------------------
    const bool chosen = elect_one();
    const uint32_t leader_full0 = __shfl_sync(0xffffffffu, map_to_cta(full0, 0), 0), tiles0 = smem_addr(tiles);
    int s = 0;
    uint32_t phase = 1;
    bool ok = true;
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      const Tile t = tile_at(tile, ftiles, offsets, tile_offsets, E);
      const int w_row = (UNIT == UNIT_GLU ? 0 : t.expert * N) + t.f * TILE_F + (TILE_F / 2) * (int)rank;
      const int w_mat = UNIT == UNIT_GLU ? 2 * t.expert : 0;
      const int half = t.n / 2, box = (half + B_ROWS - 1) / B_ROWS;
      const int x0 = t.row0 + (int)rank * half;
      const uint32_t bytes = A_BYTES + box * (B_ROWS * BK * 2);
      const CUtensorMap* xmap = &maps.x[box - 1];
      for (int kb = 0; kb < num_kb; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, phase, &abort_flag));
        if (!ok) break;
        const uint32_t dst = tiles0 + (uint32_t)s * STAGE_BYTES;
        if (chosen) {
          if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * bytes);  // this CTA's boxes and the peer's
          tma_load_3d_pair(dst, &maps.w, leader_full0 + 8 * s, kb * BK, w_row, w_mat);
#ifdef Q3_TEST_WITHHOLD_A_BOX  // (a test build leaves the slots' boxes of a pair's last tile out: its stages never fill)
          if (tile + num_pairs < num_tiles)
#endif
          tma_load_2d_pair(dst + A_BYTES, xmap, leader_full0 + 8 * s, kb * BK, x0);
        }
        ++issued;
        if (++s == STAGES) s = 0, phase ^= 1;
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {  // ---- MMA issuer of the pair, one lane chosen by elect.sync ------------------------------------
      const bool chosen = elect_one();
      const uint32_t acc0 = __shfl_sync(0xffffffffu, tmem_base, 0), tiles0 = smem_addr(tiles);
      int s = 0, i = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, ++i) {
        const Tile t = tile_at(tile, ftiles, offsets, tile_offsets, E);
        const uint32_t idesc = umma_idesc(256, t.n);
        const int buf = i & 1;
        // both epilogues have drained it
        ok = __all_sync(0xffffffffu, mbar_wait_cluster(acc_empty0 + 8 * buf, ((i >> 1) & 1) ^ 1, &abort_flag));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = acc0 + buf * ACC_COLS;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, phase, &abort_flag));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_addr = tiles0 + (uint32_t)s * STAGE_BYTES;
          const uint64_t a_desc = umma_desc(a_addr), b_desc = umma_desc(a_addr + A_BYTES);
          if (chosen) {
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              umma_pair(acc, a_desc + 2 * k, b_desc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            umma_commit_pair(empty0 + 8 * s);
          }
          __syncwarp();
          if (++s == STAGES) s = 0, phase ^= 1;
        }
        if (ok && chosen) umma_commit_pair(acc_full0 + 8 * buf);
        __syncwarp();
      }
    }
  } else {  // ---- epilogue: warp w reads TMEM lanes 32 * (w % 4) .. + 31 of this CTA, a group every other 32 slots -------
    const int group = (warp - 2) >> 2, quarter = warp & 3, et = (threadIdx.x - 64) & 127;
    const int slot_in = et >> 2, part = et & 3;  // second half: four threads per slot
    const uint32_t leader_acc_empty0 = map_to_cta(acc_empty0, 0);
    bf16* const staged = stage_out + group * 32 * OUT_STRIDE;
    auto meet = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory"); };
    int i = 0;
    for (int tile = pair; tile < num_tiles; tile += num_pairs, ++i) {
      const Tile t = tile_at(tile, ftiles, offsets, tile_offsets, E);
      const int buf = i & 1;
      const int f0 = t.f * TILE_F + (int)rank * (TILE_F / 2);
      // (a group without slots in a tile meets nowhere else in it)
      const bool lost = !__all_sync(0xffffffffu, mbar_wait(acc_full0 + 8 * buf, (i >> 1) & 1, &abort_flag));
      if (any_gave_up(group + 1, 128, lost)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t lane_addr = tmem_base + buf * ACC_COLS + ((uint32_t)(quarter * 32) << 16);
      if (group * 32 >= t.n && lane == 0) remote_arrive_relaxed(leader_acc_empty0 + 8 * buf);  // nothing here for this group
#pragma unroll 1
      for (int c0 = group * 32; c0 < t.n; c0 += 64) {
        uint32_t acc[32];
        tmem_load32(lane_addr + c0, acc);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + 64 >= t.n) {  // the last of this buffer for this group is in registers: hand it back to the MMA issuer
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          if (lane == 0) remote_arrive_relaxed(leader_acc_empty0 + 8 * buf);
        }
        // (whatever follows takes the products rounded to bfloat16, as separate kernels would)
#pragma unroll
        for (int c = 0; c < 32; ++c) staged[c * OUT_STRIDE + quarter * 32 + lane] = from_f32<bf16>(__uint_as_float(acc[c]));
        meet();
        if (c0 + slot_in < t.rows) {
          bf16* row = out + (long)(t.row0 + c0 + slot_in) * N;
          const bf16* src = staged + slot_in * OUT_STRIDE;
#pragma unroll
          for (int j = 0; j < TILE_F / 64; ++j) {
            const int f = 8 * (part + 4 * j);
            if (f0 + f >= N) continue;  // N is a multiple of 8
            if (UNIT != UNIT_NONE) {
              float a[8], v[8];
              load8(src + f, a);
              if (UNIT == UNIT_GLU) {
                float b[8];
                load8(src + 64 + f, b);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                  const float gt = fminf(a[e], limit), up = fminf(fmaxf(b[e], -limit), limit);
                  v[e] = (gt / (1.f + expf(-alpha * gt))) * (up + up_offset);
                }
              } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                  const float r = fmaxf(a[e], 0.f);
                  v[e] = r * r;
                }
              }
              store8(row + f0 + f, v);
            } else {
              *reinterpret_cast<uint4*>(row + f0 + f) = *reinterpret_cast<const uint4*>(src + f);
            }
          }
        }
        meet();  // the buffer is free again
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_flag && rank == 0) {
    // given up: the boxes of the last STAGES k-slices (both CTAs' complete on the leader's barriers) and every MMA
    // issued so far finish before tensor memory is freed and shared memory left
    if (warp == 0 && lane == 0)
      for (int j = issued > STAGES ? issued - STAGES : 0; j < issued; ++j)
        mbar_wait_drain(full0 + 8 * (j % STAGES), (j / STAGES) & 1);
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

// One block per token: its row is read once and written to the places of its slots; 16 bytes per thread and turn.
// Slots whose choice is no stored expert have no row.
__global__ void gather_slots_kernel(const bf16* __restrict__ h, long h_stride, const float* __restrict__ weights,
                                    const int* __restrict__ chosen, const int* __restrict__ place, int E, int W, int top,
                                    bf16* __restrict__ xs) {
  pdl_wait();
  pdl_launch_dependents();
  const long t = blockIdx.x;
  const bf16* src = h + t * h_stride;
  for (int i = threadIdx.x * 8; i < W; i += blockDim.x * 8) {
    const uint4 raw = *reinterpret_cast<const uint4*>(src + i);
    const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw);
    for (int k = 0; k < top; ++k) {
      const long slot = t * top + k;
      if (chosen[slot] >= E) continue;
      bf16* dst = xs + (long)place[slot] * W + i;
      if (weights) {
        const float w = weights[slot];
        float v[8];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const float2 f = __bfloat1622float2(pairs[x]);
          v[2 * x] = f.x * w;
          v[2 * x + 1] = f.y * w;
        }
        store8(dst, v);
      } else {
        *reinterpret_cast<uint4*>(dst) = raw;
      }
    }
  }
}

constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + 2 * 32 * OUT_STRIDE * sizeof(bf16) + 1024;

template <int UNIT>
int launch(const void* w, long w_rows, const void* x, void* out, int S, int E, int N, int K, const int* offsets,
           const int* tile_offsets, float limit, float alpha, float up_offset, int* error_word, cudaStream_t stream) {
  Maps maps;
  const bool glu = UNIT == UNIT_GLU;
  const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)(glu ? N : w_rows), (cuuint64_t)(glu ? 2 * E : 1)};
  const cuuint64_t strides[2] = {(cuuint64_t)K * 2, (cuuint64_t)K * 2 * dims[1]};
  const cuuint32_t box[3] = {BK, glu ? 64u : 128u, glu ? 2u : 1u}, es[3] = {1, 1, 1};
  Q3EncodeTiledFn encode = q3_encode_tiled();
  if (!encode ||
      encode(&maps.w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(w), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return Q3_ERR_LAUNCH;
  for (int i = 0; i < B_MAPS; ++i)
    if (!q3_bf16_map(&maps.x[i], x, S, K, K, B_ROWS * (i + 1))) return Q3_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  static int pairs_on[Q3_MAX_DEVICES];  // pairs of SMs the device runs at once with this kernel
  int& pairs = pairs_on[q3_current_device()];
  if (!pairs) {
    int device = 0, sms = 0, n = 0;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaFuncSetAttribute(expert_tcgen05_kernel<UNIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) != cudaSuccess)
      return Q3_ERR_LAUNCH;
    cfg.gridDim = dim3(sms / 2 * 2);
    if (cudaOccupancyMaxActiveClusters(&n, expert_tcgen05_kernel<UNIT>, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      return Q3_ERR_UNSUPPORTED;
    }
    pairs = n < sms / 2 ? n : sms / 2;
  }
  if (q3_pdl_enabled()) cfg.numAttrs = 2;
  constexpr int TILE_F = UNIT == UNIT_GLU ? 128 : 256;
  const long most = ((long)S / MAX_SLOTS + (E < S ? E : S)) * ((N + TILE_F - 1) / TILE_F);
  cfg.gridDim = dim3((unsigned)(2 * (most < pairs ? most : pairs)));
  return cudaLaunchKernelEx(&cfg, expert_tcgen05_kernel<UNIT>, maps, (bf16*)out, N, K, E, offsets, tile_offsets, limit,
                            alpha, up_offset, error_word) == cudaSuccess
             ? Q3_OK
             : Q3_ERR_LAUNCH;
}

}  // namespace

// xs [T * top, W] bf16: row place[slot] is the token's row of every slot with chosen[slot] < E (times weights[slot],
// fp32, if given).
Q3_EXPORT int q3_expert_gather(const void* h, long h_stride, const float* weights, const int* chosen, const int* place,
                               int num_tokens, int E, int W, int top, void* xs, cudaStream_t stream) {
  if (!h || !chosen || !place || !xs || num_tokens < 0 || E < 1 || W < 1 || top < 1) return Q3_ERR_ARGUMENT;
  if (W % 8 || h_stride % 8 || (((uintptr_t)h | (uintptr_t)xs) & 15)) return Q3_ERR_UNSUPPORTED;
  if (num_tokens == 0) return Q3_OK;
  const int threads = W >= 2048 ? 256 : W >= 1024 ? 128 : 64;
  return launch_pdl(gather_slots_kernel, dim3(num_tokens), dim3(threads), 0, stream, (const bf16*)h, h_stride, weights,
                    chosen, place, E, W, top, (bf16*)xs) == cudaSuccess
             ? Q3_OK
             : Q3_ERR_LAUNCH;
}

// One product of every stored expert over its slots: x [S, K] and out [S, N] in the grouped order; offsets [E + 1] the
// experts' first slots, tile_offsets [E + 1] their first chunk of at most 256 slots.  unit 0: w [E, N, K], out = W x;
// 1: the squared ReLU of that (rounded to bf16 first); 2: w [E, 2N, K] (gate rows, then up rows), out =
// g * sigmoid(alpha g) * (u + up_offset) with g = min(W_gate x, limit), u = clamp(W_up x, -limit, limit).
// K and N are multiples of 8, all bases 16-byte aligned.
Q3_EXPORT int q3_expert_tcgen05(int unit, const void* w, const void* x, void* out, int S, int E, int N, int K,
                                const int* offsets, const int* tile_offsets, float limit, float alpha, float up_offset,
                                int* error_word, cudaStream_t stream) {
  if (!w || !x || !out || !offsets || !tile_offsets || S < 0 || E < 1 || N < 1 || K < 1) return Q3_ERR_ARGUMENT;
  if (N % 8 || K % 8 || (((uintptr_t)w | (uintptr_t)x | (uintptr_t)out) & 15)) return Q3_ERR_UNSUPPORTED;
  const long w_rows = (long)E * N * (unit == UNIT_GLU ? 2 : 1);
  if (w_rows > 0x7fffffffL) return Q3_ERR_UNSUPPORTED;  // TMA coordinates are 32-bit
  if (S == 0) return Q3_OK;
  if (unit == UNIT_GLU)
    return launch<UNIT_GLU>(w, w_rows, x, out, S, E, N, K, offsets, tile_offsets, limit, alpha, up_offset, error_word, stream);
  if (unit == UNIT_RELU2)
    return launch<UNIT_RELU2>(w, w_rows, x, out, S, E, N, K, offsets, tile_offsets, 0.f, 0.f, 0.f, error_word, stream);
  if (unit == UNIT_NONE)
    return launch<UNIT_NONE>(w, w_rows, x, out, S, E, N, K, offsets, tile_offsets, 0.f, 0.f, 0.f, error_word, stream);
  return Q3_ERR_ARGUMENT;
}
