// Causal attention of prompt portions on the 5th-generation tensor cores: S = Q K^T and O += P V are tcgen05.mma
// with accumulators in tensor memory; Q, K and V tiles arrive by TMA (128-byte swizzle).  bfloat16; three forms:
//   PAGED    heads of 128 over the paged cache, straight from the QKV buffer and the pages (group size a divisor of 128,
//            page size 8/16/32/64); options: a chunked mask, turned values, sinks;
//   MAPS     differential attention: a head is two maps of 64 side by side in its 128 columns, over one value of 128;
//            options: a chunked mask or a window;
//   DENSE    keys of 192 = 128 of the head's own + 64 shared by the heads, values of 128, one key head per query head,
//            from matrices that hold the keys and values of the step's sequences one after another (attention through
//            a latent whose keys and values were expanded); options: a window, sinks.
// The mma.sync kernels serve everything else.
//
// Work item: (sequence, kv head, two row blocks A and B of 128 rows); rows are the (query token, head of the group) pairs in
// token-major order, so one 3-D TMA box [128/G tokens, G heads, 64] is 64 columns of a Q tile and the group's heads share
// every K/V tile.  PAGED and DENSE: A and B are consecutive blocks; MAPS: A and B are the two maps of the same rows.
// Keys come in tiles of 64 (PAGED, MAPS: 64/page_size pages, one TMA box per page and 64 columns), and each tile is used
// by both row blocks.  Per 64-key tile a row block's chain is long (TMEM load, exp2 on the special-function unit, TMEM
// store, fences, barrier round trips) and leaves the tensor core and the exp2 unit idle for much of the time; two blocks in
// flight hide each other's chain.  Sixteen warps:
//   warps 0..3       : TMA producers, keys and values, 64 columns each, through rings of stages (the fourth one brings Q of
//                      both blocks first);
//   warps 4..7, 8..11: softmax of block A and of block B, one thread per row: reads S_j from TMEM and gives its place back at
//                      once, masks, online softmax in fp32 (exp2, scale folded in), writes P_j as bf16 into one of two
//                      buffers in TMEM, where the PV MMA reads it as its A operand; O stays in TMEM (the MMAs accumulate
//                      into it) and is rescaled there only when a row's maximum has grown by more than 2^8; finally stores
//                      O / l.  MAPS: block B's threads leave lambda O_B / l_B in shared memory, block A's subtract it, divide
//                      by the root mean square and store;
//   warps 12, 13     : MMA issuers of S for block A and B: S_(j+1) as soon as S_j is in registers;
//   warps 14, 15     : MMA issuers of PV for block A and B: PV_j when P_j is written.
// Tensor memory: all 512 columns, per block S [0,64), P_0 and P_1 [64,128), O [128,256).
// What bounds it: the softmax warps, and behind them the products (S with 64 columns is bound by its reads of shared memory,
// 47 cycles per 16 k-values) and the keys' and values' way from L2 (32 KB a step and SM).  A step of both blocks takes 1520
// cycles where the exp2 unit alone needs 1024.  What counted was code, not arithmetic: 32 heads over 8, 8192 tokens, one layer,
// us (2048 tokens: 48 -> 43; forms of this code that differ only in what stands beside the loops lie 4 % apart, so time both sizes):
//   554  one issuer per block (PV_j before S_(j+2): its waits, commits and products took longer than the softmax of a tile), one
//        producer, S twice and P over S
//   550  S issued before PV by warps of their own, four producers
//   512  tiles that all rows see as a whole without the masks' branches; waits with their slow part out of line
//   457  the reference point moved without a branch, the rescaling out of line
//   451  the issuers' lane chosen by elect.sync (an MMA of 64 columns every 47 cycles instead of 60 to 78)
// Not kept: 128 keys a step (830: the chain of a block twice as long), turns of the two blocks at the exponentials (482),
// S_(j+1) loaded beside the exponentials of tile j with 192 registers a thread (585), waits that try again without looking at
// the clock (512 -> 562).  Forms: differential attention, 16 heads over 4, 2333 + 419 tokens 60 -> 54 us (mma.sync: 247);
// latent, 16 heads, 2048 tokens, window 1024: 34 -> 31 us and 26 us for the expansion (in the latent space on mma.sync: 481).
// V is the B operand of PV in MN-major form (rows = keys): descriptor with the halves of D
// 8 KB apart (leading offset) and 8-key groups 1 KB apart (stride offset); 16 keys = 2 KB.
// Keys past a block's last position are zeroed in shared memory before PV (stale or poisoned
// page contents must not meet a zero probability).  Every mbarrier wait is bounded; on expiry
// the block raises its abort flag and the global error word, frees TMEM and returns.
#include <type_traits>

#include "async_tiles.cuh"

namespace {

enum { PAGED = 0, MAPS = 1, DENSE = 2 };
constexpr int D = 128;  // value size, and query/key size of PAGED and of both maps together
constexpr int BLOCK_M = 128;
constexpr int BLOCK_N = 64;
constexpr int THREADS = 512;
constexpr int HALF_Q = BLOCK_M * 128;           // 64 columns of a Q tile: [128 rows][128 B]
constexpr int HALF_KV = BLOCK_N * 128;          // 64 columns of a K or V tile: [64 rows][128 B]
constexpr int V_BYTES = 2 * HALF_KV;
constexpr int TMEM_COLS = 512;                  // per row block: S [0,64), P [64,128) (two buffers), O [128,256)
constexpr int TMEM_BLOCK = 256, TMEM_P = 64, TMEM_O = 128;

template <int MODE>
struct Sizes {
  static constexpr int DK = MODE == DENSE ? 192 : 128;
  static constexpr int Q_BYTES = DK / 64 * HALF_Q;
  static constexpr int K_BYTES = DK / 64 * HALF_KV;
  static constexpr int STAGES = MODE == DENSE ? 3 : 4;  // key tiles and value tiles in flight
  static constexpr int SMEM = 2 * Q_BYTES + STAGES * (K_BYTES + V_BYTES) + 1024;
};

struct Params {
  const int* block_table;
  int max_pages;
  const int *kv_lens, *cu_seqlens;
  bf16* out;
  int num_seqs, num_work, nq, nkv, ps;
  float scale_log2;
  int skip_single, chunk, window;
  const float *turns, *sinks;
  const int* kv_base;             // DENSE: key j of sequence s is row kv_base[s] + j
  float lambda, eps, out_scale;   // MAPS
  int* error_word;
};

// 2^x in one instruction (exp2f adds range fix-ups around the same instruction; results
// below 2^-126 become zero here, which is what a probability that small is worth)
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// A wait that is one instruction and a branch that is not taken where the barrier is complete, or becomes so while the
// instruction holds the warp; the rest is out of line.  (Branches are what the softmax warps stumble over.)
__device__ __noinline__ bool wait_on(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return mbar_wait(bar, parity, abort_flag);
}
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (__builtin_expect(mbar_try_wait(bar, parity), 1)) return true;
  return wait_on(bar, parity, abort_flag);
}
// a row's D accumulators in tensor memory times `corr`; rare, and out of line for the same reason
__device__ __noinline__ void rescale_rows(uint32_t o_addr, float corr) {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
  for (int c0 = 0; c0 < D; c0 += 32) {
    uint32_t ov[32];
    tmem_load32(o_addr + c0, ov);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int c = 0; c < 32; ++c) ov[c] = __float_as_uint(__uint_as_float(ov[c]) * corr);
    tmem_store32(o_addr + c0, ov);
  }
}
__device__ __forceinline__ void arrive_if(bool yes, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}"
      ::"r"(bar), "r"((uint32_t)yes)
      : "memory");
}

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
prefill_attention_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                            const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_r,
                            const __grid_constant__ Params p) {
  typedef Sizes<MODE> Z;
  constexpr int KV_STAGES = Z::STAGES, Q_BYTES = Z::Q_BYTES, K_BYTES = Z::K_BYTES, DK = Z::DK;
  enum { BAR_Q = 0, BAR_K_FULL = 1, BAR_K_EMPTY = BAR_K_FULL + KV_STAGES, BAR_V_FULL = BAR_K_EMPTY + KV_STAGES,
         BAR_V_EMPTY = BAR_V_FULL + KV_STAGES, BAR_S_FULL = BAR_V_EMPTY + KV_STAGES,  // [block], like the rest
         BAR_S_EMPTY = BAR_S_FULL + 2, BAR_P_FULL = BAR_S_EMPTY + 2, BAR_PV_FULL = BAR_P_FULL + 2,
         BAR_END = BAR_PV_FULL + 2, NUM_BARS = BAR_END + 4 };
  const int *block_table = p.block_table, *cu_seqlens = p.cu_seqlens;
  const int max_pages = p.max_pages, nq = p.nq, nkv = p.nkv, ps = p.ps, chunk = p.chunk, window = p.window;
  const float scale_log2 = p.scale_log2;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* q_s = base;                         // 2 blocks x [DK / 64][128 rows][128 B]
  unsigned char* k_s = q_s + 2 * Q_BYTES;            // KV_STAGES x [DK / 64][64 rows][128 B]
  unsigned char* v_s = k_s + KV_STAGES * K_BYTES;    // KV_STAGES x [2 halves][64 rows][128 B]
  __shared__ __align__(8) unsigned long long bars[NUM_BARS];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int abort_flag;
  __shared__ int s_item[2];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // heavy items first over the whole grid: all kv heads of the heaviest item, then the next ...
  const int kvh = blockIdx.x % nkv;
  const int G = nq / nkv;
  const uint32_t bar0 = smem_addr(&bars[0]);
  auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };

  if (tid == 0) {
    abort_flag = 0;
    // heavy work (late rows of long prompts) first: walk the work list from its end
    int acc = 0, found = -1, rb = 0;
    const int w = p.num_work - 1 - (int)(blockIdx.x / nkv);
    for (int s = 0; s < p.num_seqs; ++s) {
      const int ql = cu_seqlens[s + 1] - cu_seqlens[s];
      if (ql <= 0 || (p.skip_single && ql == 1)) continue;
      int nb = (ql * G + BLOCK_M - 1) / BLOCK_M;  // row blocks
      if (MODE != MAPS) nb = (nb + 1) / 2;        // pairs of them
      if (w < acc + nb) {
        found = s;
        rb = w - acc;
        break;
      }
      acc += nb;
    }
    s_item[0] = found;
    s_item[1] = rb;
    mbar_init(bar(BAR_Q), 1);
    for (int i = 0; i < KV_STAGES; ++i) {
      mbar_init(bar(BAR_K_FULL + i), 2);   // two producers
      mbar_init(bar(BAR_K_EMPTY + i), 2);  // both issuers
      mbar_init(bar(BAR_V_FULL + i), 2);
      mbar_init(bar(BAR_V_EMPTY + i), 2);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(BAR_S_FULL + i), 1);
      mbar_init(bar(BAR_S_EMPTY + i), 4);  // a block's softmax warps
      mbar_init(bar(BAR_P_FULL + i), 4);
      mbar_init(bar(BAR_PV_FULL + i), 1);
    }
    for (int i = 0; i < 4; ++i) mbar_init(bar(BAR_END + i), 1);  // the issuers
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 12) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_s)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;
  const int seq = s_item[0];

  if (seq >= 0) {
    const int tok0 = cu_seqlens[seq];
    const int q_len = cu_seqlens[seq + 1] - tok0;
    const int kv_len = p.kv_lens[seq];
    const int rows = q_len * G;
    const int base_pos = kv_len - q_len;
    // row blocks A and B of this item; B may not exist (odd number of blocks)
    int row0[2], p_max[2], tiles[2];
    // under a chunked mask or a window the item's first visible key is that of its first row; tiles count from the tile
    // it is in
    const int p_first = base_pos + (MODE == MAPS ? 1 : 2) * s_item[1] * BLOCK_M / G;
    const int k_lo = chunk > 0 ? p_first / chunk * chunk : (window > 0 ? max(0, p_first - window + 1) : 0);
    const int tile0 = k_lo / BLOCK_N;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      row0[x] = (MODE == MAPS ? s_item[1] : 2 * s_item[1] + x) * BLOCK_M;
      const bool live = row0[x] < rows;
      const int last_row = min(rows, row0[x] + BLOCK_M) - 1;
      p_max[x] = live ? base_pos + last_row / G : -1;
      tiles[x] = live ? p_max[x] / BLOCK_N + 1 - tile0 : 0;
    }
    const int num_tiles = max(tiles[0], tiles[1]);  // B lies after A, so this is B's count when B exists
    const int p_last = max(p_max[0], p_max[1]);
    const int* bt = MODE == DENSE ? nullptr : block_table + (long)seq * max_pages;
    const int pages_per_tile = MODE == DENSE ? 0 : BLOCK_N / ps;

    if (warp < 4) {  // ---- TMA producers: keys and values, 64 columns each ----
      const int part = warp;  // keys: 0, 1; values: 2, 3
      const int half = part & 1;
      if (part == 3 && lane == 0) {
        constexpr int BOXES = MODE == MAPS ? 1 : DK / 64;  // of a block; MAPS: map x is columns 64 x .. of the head
        mbar_expect_tx(bar(BAR_Q), (tiles[1] ? 2 : 1) * BOXES * HALF_Q);
        for (int x = 0; x < 2; ++x) {
          if (!tiles[x]) continue;
          for (int c = 0; c < BOXES; ++c) {
            const bool turned = MODE == DENSE && c == 2;
            tma_load_3d(smem_addr(q_s) + x * Q_BYTES + c * HALF_Q, turned ? &tmap_r : &tmap_q, bar(BAR_Q),
                        turned ? 0 : 64 * (MODE == MAPS ? x : c), kvh * G, tok0 + row0[x] / G);
          }
        }
      }
      // PAGED, MAPS: a tile is 64 / ps pages, one box per page; each lane holds a page of the next tile.  DENSE: boxes of 64
      // rows (keys: two of the head's own columns, one of the shared ones; the values lie beside the keys, behind those of all
      // heads).
      const int row_base = MODE == DENSE ? p.kv_base[seq] : 0;
      const uint32_t full = bar(part < 2 ? BAR_K_FULL : BAR_V_FULL), empty = bar(part < 2 ? BAR_K_EMPTY : BAR_V_EMPTY);
      const uint32_t stage_bytes = part < 2 ? K_BYTES : V_BYTES;
      const uint32_t dst0 = smem_addr(part < 2 ? k_s : v_s) + half * HALF_KV;
      const CUtensorMap* map = MODE == DENSE || part < 2 ? &tmap_k : &tmap_v;
      auto page_of = [&](int j) -> int {  // pages of tile j that exist in the block table (the rest of the tile is masked)
        const int pi = (tile0 + j) * pages_per_tile + lane;
        const bool in = lane < pages_per_tile && j < num_tiles && pi < max_pages && pi * ps <= p_last && (pi + 1) * ps > k_lo;
        return in ? bt[pi] : -1;
      };
      int next = MODE == DENSE ? 0 : page_of(0);
      int st = 0, j = 0;
      uint32_t phase = 1;
      for (; j < num_tiles; ++j) {
        const int page = next;
        const uint32_t dst = dst0 + st * stage_bytes;
        uint32_t bytes = HALF_KV + (MODE == DENSE && part == 1 ? HALF_KV : 0);
        if (MODE != DENSE) {
          bytes = __popc(__ballot_sync(0xffffffffu, page >= 0)) * (uint32_t)ps * 128u;
          next = page_of(j + 1);
        }
        if (!__all_sync(0xffffffffu, mbar_wait(empty + 8 * st, phase, &abort_flag))) break;
        if (lane == 0) mbar_expect_tx(full + 8 * st, bytes);
#ifdef Q3_TEST_WITHHOLD_A_BOX  // (a test build leaves one half of the keys' boxes out: the stage never fills, a wait runs out)
        if (part != 1)
#endif
        if (MODE == DENSE) {
          if (lane == 0) {
            const int y = row_base + (tile0 + j) * BLOCK_N;
            tma_load_2d(dst, map, full + 8 * st, (part < 2 ? kvh : nkv + kvh) * D + half * 64, y);
            if (part == 1) tma_load_2d(dst + HALF_KV, &tmap_v, full + 8 * st, 0, y);
          }
        } else {
          for (int u = 0; u < pages_per_tile; ++u) {
            const int pg = __shfl_sync(0xffffffffu, page, u);
            if (lane == 0 && pg >= 0) tma_load_2d(dst + u * ps * 128, map, full + 8 * st, half * 64, (pg * nkv + kvh) * ps);
          }
        }
        if (++st == KV_STAGES) st = 0, phase ^= 1;
      }
      // The last boxes may still be in flight when the others have given up.  (Then a stage that the other producer did not come to
      // any more is waited for until the limit.)
      if (lane == 0) {
        if (part == 3) mbar_wait_drain(bar(BAR_Q), 0);
        for (int i = max(0, j - KV_STAGES); i < j; ++i) mbar_wait_drain(full + 8 * (i % KV_STAGES), (i / KV_STAGES) & 1);
      }
    } else if (warp > 11) {
      // ---- MMA issuers: warps 12 and 13 for S of block A and B, warps 14 and 15 for PV ---------
      // Issuing is work too (descriptors, barrier round trips of a hundred cycles each, a queue in front of the tensor
      // core): one thread that issued both products of a block needed longer for a tile than the softmax.  The warps run as
      // a whole (an arrival and its wait, there and back, take 511 cycles between single lanes and 247 between warps).  Both
      // blocks use every K and V tile: its "empty" barrier counts two arrivals, a commit from an issuer that multiplied with
      // the tile and a plain arrival (after the tile's "full") from one that had no use for it.
      const int role = __shfl_sync(0xffffffffu, warp, 0), x = role & 1;
      const int mine = __shfl_sync(0xffffffffu, tiles[x], 0), all = __shfl_sync(0xffffffffu, num_tiles, 0);
      const uint32_t tmem_x = __shfl_sync(0xffffffffu, tmem, 0) + x * TMEM_BLOCK;
      const bool leader = elect_one();
      auto wait_all = [&](int b, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar(b), parity, &abort_flag)); };
      int st = 0;
      uint32_t phase = 0;
      if (role < 14) {
        constexpr uint32_t idesc = umma_idesc(BLOCK_M, BLOCK_N, 0);  // S = Q K^T: N = 64 keys
        const uint32_t q_addr = smem_addr(q_s) + x * Q_BYTES;
        bool ok = mine == 0 || wait_all(BAR_Q, 0);
        for (int j = 0; j < all && ok; ++j) {
          // S_j as soon as the softmax has S_(j-1) in its registers
          ok = (j == 0 || j >= mine || wait_all(BAR_S_EMPTY + x, (j - 1) & 1)) && wait_all(BAR_K_FULL + st, phase);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (leader) {
            if (j < mine) {
              const uint32_t k_addr = smem_addr(k_s) + st * K_BYTES;
#pragma unroll
              for (int k = 0; k < (MODE == MAPS ? 64 : DK) / 16; ++k) {
                const uint32_t half = (k >> 2), sub = (k & 3) * 2;  // 4 steps of 32 bytes per 64 columns
                umma_bf16(tmem_x, umma_desc(q_addr + half * HALF_Q) + sub,
                     umma_desc(k_addr + (MODE == MAPS ? x : half) * HALF_KV) + sub, idesc, k > 0 ? 1u : 0u);
              }
              umma_commit(bar(BAR_S_FULL + x));    // S_j is in TMEM
              umma_commit(bar(BAR_K_EMPTY + st));  // this block is done with the key tile
            } else {
              mbar_arrive(bar(BAR_K_EMPTY + st));
            }
          }
          __syncwarp();
          if (++st == KV_STAGES) st = 0, phase ^= 1;
        }
      } else {
        constexpr uint32_t idesc = umma_idesc(BLOCK_M, D, 1);  // PV: N = 128, V MN-major
        bool ok = true;
        for (int j = 0; j < all && ok; ++j) {
          ok = (j >= mine || wait_all(BAR_P_FULL + x, j & 1)) && wait_all(BAR_V_FULL + st, phase);  // P_j written, O at rest
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (leader) {
            if (j < mine) {
              const uint32_t v_addr = smem_addr(v_s) + st * V_BYTES;
#pragma unroll
              for (int k = 0; k < BLOCK_N / 16; ++k)  // 16 keys: 8 columns of P, 2 KB down V's rows
                umma_bf16_tmem(tmem_x + TMEM_O, tmem_x + TMEM_P + (j & 1) * (BLOCK_N / 2) + 8 * k,
                     umma_desc_mn_major(v_addr + k * 2048, HALF_KV), idesc, (j > 0 || k > 0) ? 1u : 0u);
              umma_commit(bar(BAR_PV_FULL + x));
              umma_commit(bar(BAR_V_EMPTY + st));
            } else {
              mbar_arrive(bar(BAR_V_EMPTY + st));
            }
          }
          __syncwarp();
          if (++st == KV_STAGES) st = 0, phase ^= 1;
        }
      }
      if (elect_one()) {  // (the same lane again) nothing of this issuer's is in flight any more when the tensor memory is freed
        umma_commit(bar(BAR_END + role - 12));
        mbar_wait_drain(bar(BAR_END + role - 12), 0);
      }
      __syncwarp();
    } else {  // ---- softmax: one thread per row; warps 4..7 block A, warps 8..11 block B -------------
      const int x = (warp - 4) >> 2;
      const int quarter = warp & 3;
      const int r = quarter * 32 + lane;  // row of the tile = TMEM lane
      const int R = row0[x] + r;
      const bool row_ok = R < rows;
      const int pos = row_ok ? base_pos + R / G : -1;
      // the row's first visible key
      const int lo = !row_ok ? 0 : (chunk > 0 ? pos / chunk * chunk : (window > 0 ? max(0, pos - window + 1) : 0));
      const int my_tiles = tiles[x];
      const uint32_t lane_base = tmem + x * TMEM_BLOCK + ((uint32_t)(quarter * 32) << 16);
      const uint32_t o_addr = lane_base + TMEM_O;
      // O stays in TMEM and the MMAs accumulate into it.  The reference point of the exponentials
      // (m_ref) is only moved when a row's maximum exceeds it by more than 2^8 after scaling; then
      // O and l are rescaled.  Probabilities may therefore reach 2^8, which bf16 and fp32 hold easily,
      // and the final O / l is unchanged.
      const float slack = fminf(8.f / scale_log2, 1e38f);
      float m_ref = -INFINITY, l_run = 0.f;
      const float2 scale2 = make_float2(scale_log2, scale_log2);
      // One tile.  EDGE: some row of the block does not see all of its keys, or some of them lie outside of what the item reads;
      // the others have no branch but the rare one for a new reference point, so that loads, maxima and exponentials
      // are scheduled as one run of instructions.
      auto step = [&](int j, auto edge) -> bool {
        constexpr bool EDGE = decltype(edge)::value;
        const int key0 = (tile0 + j) * BLOCK_N;
        if (!wait(bar(BAR_S_FULL + x), j & 1, &abort_flag)) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t sa[32], sb[32];
        tmem_load32(lane_base, sa);
        tmem_load32(lane_base + 32, sb);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        arrive_if(lane == 0, bar(BAR_S_EMPTY + x));  // S_(j+1) may come
        if constexpr (EDGE) {
          if (key0 + BLOCK_N - 1 > pos) {  // the tile crosses this row's diagonal
#pragma unroll
            for (int c = 0; c < 32; ++c) {
              if (key0 + c > pos) sa[c] = 0xff800000u;  // -inf
              if (key0 + 32 + c > pos) sb[c] = 0xff800000u;
            }
          }
          if (key0 < lo) {  // keys of an earlier chunk, or before the window
#pragma unroll
            for (int c = 0; c < 32; ++c) {
              if (key0 + c < lo) sa[c] = 0xff800000u;
              if (key0 + 32 + c < lo) sb[c] = 0xff800000u;
            }
          }
        }
        float mx;
        {  // eight independent running maxima: a single chain of 64 would expose its latency
          float part[8];
#pragma unroll
          for (int c = 0; c < 8; ++c) part[c] = fmaxf(__uint_as_float(sa[c]), __uint_as_float(sb[c]));
#pragma unroll
          for (int c = 8; c < 32; ++c)
            part[c & 7] = fmaxf(part[c & 7], fmaxf(__uint_as_float(sa[c]), __uint_as_float(sb[c])));
          mx = fmaxf(fmaxf(fmaxf(part[0], part[1]), fmaxf(part[2], part[3])),
                     fmaxf(fmaxf(part[4], part[5]), fmaxf(part[6], part[7])));
        }
        const float m_old = m_ref;
        m_ref = mx > m_ref + slack ? mx : m_ref;  // (also from -infinity)
        const bool moved = __any_sync(0xffffffffu, m_ref != m_old);
        const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
        // probabilities, rounded to bf16 as the MMA will see them, into tensor memory; the scaling and the row sum run on
        // pairs of elements (packed fp32 instructions)
        float2 sums[4] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
        uint32_t w[32];
        const float2 neg2 = make_float2(-m_use * scale_log2, -m_use * scale_log2);
#pragma unroll
        for (int ch = 0; ch < 8; ++ch) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int c = ch * 8 + 2 * e;
            const float2 s2 = make_float2(__uint_as_float(c < 32 ? sa[c & 31] : sb[c & 31]),
                                          __uint_as_float(c < 32 ? sa[(c + 1) & 31] : sb[(c + 1) & 31]));
            const float2 t2 = __ffma2_rn(s2, scale2, neg2);
            const float2 x2 = make_float2(ex2(t2.x), ex2(t2.y));
            sums[e] = __fadd2_rn(sums[e], x2);
            w[ch * 4 + e] = pack2(x2.x, x2.y);
          }
        }
        tmem_store32(lane_base + TMEM_P + (j & 1) * (BLOCK_N / 2), w);
        {
          const float2 a = __fadd2_rn(sums[0], sums[1]), b = __fadd2_rn(sums[2], sums[3]);
          const float2 c = __fadd2_rn(a, b);
          const float corr = m_ref == m_old ? 1.f : exp2f((m_old - m_ref) * scale_log2);  // 0 from -infinity
          l_run = l_run * corr + (c.x + c.y);
        }
        // PV_(j-1) must be finished before P_j is signalled: it keeps this barrier from running a phase ahead of the waiters,
        // P_(j+1) goes where P_(j-1) was, and O must be at rest if it has to be rescaled
        if (!EDGE || j > 0) {
          if (!wait(bar(BAR_PV_FULL + x), (j - 1) & 1, &abort_flag)) return false;
          if (__builtin_expect(moved, 0)) {
            rescale_rows(o_addr, m_ref == m_old ? 1.f : exp2f((m_old - m_ref) * scale_log2));
          }
        }
        // keys of this tile past the item's last position hold whatever the page held, keys before its first
        // visible one may not have been loaded at all: zero their value rows before PV reads them (both blocks
        // do, each before its own PV; keys between the blocks' last positions are real and only masked)
        if constexpr (EDGE) {
          if (key0 + BLOCK_N - 1 > p_last || key0 < k_lo) {
            const int vst = j % KV_STAGES;
            if (!wait(bar(BAR_V_FULL + vst), (j / KV_STAGES) & 1, &abort_flag)) return false;
            const int vrow = r & 63, half = r >> 6;
            if (key0 + vrow > p_last || key0 + vrow < k_lo) {
              uint4* dst = reinterpret_cast<uint4*>(v_s + vst * V_BYTES + half * HALF_KV + vrow * 128);
#pragma unroll
              for (int ch = 0; ch < 8; ++ch) dst[ch] = make_uint4(0, 0, 0, 0);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // zeroed V visible to the MMA
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        arrive_if(lane == 0, bar(BAR_P_FULL + x));
        return true;
      };
      // tiles that every row of the block sees as a whole: from the last row's first key on, up to the first row's position
      const int row_first = row0[x], row_last = min(rows, row0[x] + BLOCK_M) - 1;
      const int pos_first = base_pos + row_first / G, pos_last = base_pos + row_last / G;
      const int lo_last = chunk > 0 ? pos_last / chunk * chunk : (window > 0 ? max(0, pos_last - window + 1) : 0);
      // (What rows that are none see in a last block has no say: nothing of theirs is stored.  A last block that goes through tiles with
      // masks only is the longest of its sequence: 32 heads over 8, 500 tokens behind 3000, 78 us; so 64.)
      int whole0 = 1, whole1 = 0;  // such tiles behind the first one
      if (row0[x] < rows) {
        whole0 = max(1, (max(lo_last, k_lo) + BLOCK_N - 1) / BLOCK_N - tile0);
        whole1 = min(my_tiles, (pos_first + 1) / BLOCK_N - tile0);
      }
      bool ok = true;
      for (int j = 0; j < my_tiles && ok; ++j) {
        if (j < whole0 || j >= whole1) {
          ok = step(j, std::true_type());
        } else {
          while (step(j, std::false_type()) && ++j < whole1) {}
          ok = j-- == whole1;
        }
      }
      if (ok && my_tiles) ok = wait(bar(BAR_PV_FULL + x), (my_tiles - 1) & 1, &abort_flag);
      __syncwarp();
      if constexpr (MODE == MAPS) {
        // out = o / sqrt(mean(o^2) + eps) * out_scale, o = O_A / l_A - lambda O_B / l_B.  A row's 128 values pass from
        // B's thread to A's through the Q tiles' shared memory (both blocks' products with Q are finished), 16 bytes at a
        // time in places that differ between neighbouring rows.  All threads come here, also after an expired wait.
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const float inv = (x ? p.lambda : 1.f) / l_run;
        float4* mine = reinterpret_cast<float4*>(q_s + r * 512);
        asm volatile("bar.sync 2, 256;" ::: "memory");
        if (x == 1) {
#pragma unroll 1
          for (int c0 = 0; c0 < D; c0 += 32) {
            uint32_t ov[32];
            tmem_load32(o_addr + c0, ov);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int c = 0; c < 32; c += 4)
              mine[((c0 + c) >> 2) ^ (r & 31)] =
                  make_float4(__uint_as_float(ov[c]) * inv, __uint_as_float(ov[c + 1]) * inv,
                              __uint_as_float(ov[c + 2]) * inv, __uint_as_float(ov[c + 3]) * inv);
          }
        }
        asm volatile("bar.sync 2, 256;" ::: "memory");
        if (x == 0) {
          float ss = 0.f;
#pragma unroll 1
          for (int c0 = 0; c0 < D; c0 += 32) {
            uint32_t ov[32];
            tmem_load32(o_addr + c0, ov);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int c = 0; c < 32; c += 4) {
              float4* at = mine + (((c0 + c) >> 2) ^ (r & 31));
              const float4 b = *at;
              const float4 o = make_float4(__uint_as_float(ov[c]) * inv - b.x, __uint_as_float(ov[c + 1]) * inv - b.y,
                                           __uint_as_float(ov[c + 2]) * inv - b.z, __uint_as_float(ov[c + 3]) * inv - b.w);
              ss += o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w;
              *at = o;
            }
          }
          const float rstd = rsqrtf(ss / (float)D + p.eps) * p.out_scale;
          if (ok && row_ok) {
            bf16* dst = p.out + ((long)(tok0 + R / G) * nq + kvh * G + R % G) * D;
#pragma unroll 4
            for (int c = 0; c < D; c += 8) {
              const float4 a = mine[(c >> 2) ^ (r & 31)], b = mine[((c >> 2) + 1) ^ (r & 31)];
              const float v8[8] = {a.x * rstd, a.y * rstd, a.z * rstd, a.w * rstd, b.x * rstd, b.y * rstd, b.z * rstd, b.w * rstd};
              store8(dst + c, v8);
            }
          }
        }
      } else if (ok && my_tiles) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // a head's sink: one more term in the denominator, in the units of the row's reference point
        if (p.sinks && row_ok) l_run += exp2f(p.sinks[kvh * G + R % G] * LOG2_E - m_ref * scale_log2);
        const float inv = 1.f / l_run;
        const float* turns = MODE == PAGED ? p.turns : nullptr;
        bf16* dst = row_ok ? p.out + ((long)(tok0 + R / G) * nq + kvh * G + R % G) * D : nullptr;
        if (turns) {  // turned values: the sum is turned back, element c with element c + D / 2
          const float* cs = row_ok ? turns + (long)(tok0 + R / G) * D : nullptr;  // cos (D / 2), sin (D / 2)
#pragma unroll 1
          for (int c0 = 0; c0 < D / 2; c0 += 32) {
            uint32_t ua[32], ub[32];
            tmem_load32(o_addr + c0, ua);
            tmem_load32(o_addr + D / 2 + c0, ub);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (row_ok) {
#pragma unroll
              for (int c = 0; c < 32; c += 8) {
                float co[8], sn[8], x8[8], y8[8];
                load8(cs + c0 + c, co);
                load8(cs + D / 2 + c0 + c, sn);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                  const float u = __uint_as_float(ua[c + e]) * inv, v = __uint_as_float(ub[c + e]) * inv;
                  x8[e] = u * co[e] + v * sn[e];
                  y8[e] = v * co[e] - u * sn[e];
                }
                store8(dst + c0 + c, x8);
                store8(dst + D / 2 + c0 + c, y8);
              }
            }
          }
        }
#pragma unroll 1
        for (int c0 = 0; c0 < D && !turns; c0 += 32) {
          uint32_t ov[32];
          tmem_load32(o_addr + c0, ov);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (row_ok) {
#pragma unroll
            for (int c = 0; c < 32; c += 8) {
              float v8[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) v8[e] = __uint_as_float(ov[c + e]) * inv;
              store8(dst + c0 + c, v8);
            }
          }
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 12) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
  if (tid == 0 && abort_flag && p.error_word) atomicExch(p.error_word, 2);
}

template <int MODE>
int launch(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tr, const Params& p,
           cudaStream_t stream) {
  static bool configured_on[Q3_MAX_DEVICES];
  bool& configured = configured_on[q3_current_device()];
  if (!configured) {
    if (cudaFuncSetAttribute(prefill_attention_tc_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             Sizes<MODE>::SMEM) != cudaSuccess)
      return Q3_ERR_LAUNCH;
    configured = true;
  }
  prefill_attention_tc_kernel<MODE><<<dim3((unsigned)p.num_work * p.nkv), THREADS, Sizes<MODE>::SMEM, stream>>>(tq, tk, tv, tr, p);
  return q3_launch_status();
}

// Q as [tokens][heads][columns]: boxes of 128 / G tokens x G heads x 64 columns
bool q_map(CUtensorMap* map, const void* q, int cols, int nq, long num_tokens, long q_stride, int G) {
  Q3EncodeTiledFn fn = q3_encode_tiled();
  if (!fn) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)nq, (cuuint64_t)num_tokens};
  const cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)q_stride * 2};
  const cuuint32_t box[3] = {64, (cuuint32_t)G, (cuuint32_t)(BLOCK_M / G)};
  const cuuint32_t es[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool paged_ok(const void* q, int q_stride, const void* kpages, const void* vpages, int nq, int nkv, int ps) {
  return BLOCK_M % (nq / nkv) == 0 && (ps == 8 || ps == 16 || ps == 32 || ps == 64) && q_stride % 8 == 0 && nkv <= 65535 &&
         (((uintptr_t)q | (uintptr_t)kpages | (uintptr_t)vpages) & 15) == 0;
}

}  // namespace

// q: the QKV buffer, [num_tokens, *] bf16 with row stride q_stride (elements), head h at column
// h * 128.  kpages / vpages: [num_rows_kv / (nkv * ps), nkv, ps, 128] bf16 of one layer, num_rows_kv
// rows of 128 in all.  num_work = sum over served sequences of ceil(ceil(q_len * (nq / nkv) / 128) / 2).
// Returns Q3_ERR_UNSUPPORTED for shapes this kernel does not take (the caller then uses the
// mma.sync kernel).  chunk > 0: a token sees the keys of its own chunk of that many tokens only.  turns: null, or
// fp32 [num_tokens, 2, 64], cos then sin per pair (m, m + 64): the cached values are turned by their positions and a
// head's result is turned back by its token's angles.  sinks: null, or fp32 [nq], per head a score without a value in the
// softmax's denominator.  error_word: device int set to 2 if a wait inside the kernel expired.
Q3_EXPORT int q3_paged_attention_prefill_tc(const void* q, int q_stride, int num_tokens, const void* kpages,
                                            const void* vpages, long num_rows_kv, const int* block_table,
                                            int max_pages, const int* kv_lens, const int* cu_seqlens, void* out,
                                            int num_seqs, int num_work, int nq, int nkv, int head_dim, int ps,
                                            float scale, int skip_single, int chunk, const float* turns,
                                            const float* sinks, int* error_word, cudaStream_t stream) {
  if (chunk < 0 || ((uintptr_t)turns & 15)) return Q3_ERR_ARGUMENT;
  if (!q || !kpages || !vpages || !block_table || !kv_lens || !cu_seqlens || !out) return Q3_ERR_ARGUMENT;
  if (nq < 1 || nkv < 1 || nq % nkv) return Q3_ERR_ARGUMENT;
  if (head_dim != D || !paged_ok(q, q_stride, kpages, vpages, nq, nkv, ps)) return Q3_ERR_UNSUPPORTED;
  if (num_work == 0) return Q3_OK;
  CUtensorMap tq, tk, tv;
  // pages as a matrix [rows of all pages and kv heads][D], read in boxes of one page x 64 dims
  if (!q_map(&tq, q, D, nq, num_tokens, q_stride, nq / nkv) ||
      !q3_bf16_map(&tk, kpages, num_rows_kv, D, D, ps, CU_TENSOR_MAP_L2_PROMOTION_L2_128B) ||
      !q3_bf16_map(&tv, vpages, num_rows_kv, D, D, ps, CU_TENSOR_MAP_L2_PROMOTION_L2_128B))
    return Q3_ERR_LAUNCH;
  const Params p = {block_table, max_pages, kv_lens, cu_seqlens, (bf16*)out, num_seqs, num_work, nq, nkv, ps,
                    scale * LOG2_E, skip_single, chunk, 0, turns, sinks, nullptr, 0.f, 0.f, 0.f, error_word};
  return launch<PAGED>(tq, tk, tv, tq, p, stream);
}

// Differential attention of every sequence of the step: query head h is [map 1 (64) | map 2 (64)] at column h * 128, key
// pages hold both maps side by side, value pages the values of 128; out [num_tokens, nq, 128]: (a1 - lambda a2) divided by
// its root mean square (eps inside the root), times out_scale.  num_work = sum over sequences of ceil(q_len * (nq / nkv) /
// 128).  window or chunk > 0: the mask (not both).
Q3_EXPORT int q3_diff_attention_prefill_tc(const void* q, int q_stride, int num_tokens, const void* kpages,
                                           const void* vpages, long num_rows_kv, const int* block_table, int max_pages,
                                           const int* kv_lens, const int* cu_seqlens, void* out, int num_seqs, int num_work,
                                           int nq, int nkv, int ps, float scale, int window, int chunk, float lambda,
                                           float eps, float out_scale, int* error_word, cudaStream_t stream) {
  if (chunk < 0 || window < 0 || (chunk && window)) return Q3_ERR_ARGUMENT;
  if (!q || !kpages || !vpages || !block_table || !kv_lens || !cu_seqlens || !out) return Q3_ERR_ARGUMENT;
  if (nq < 1 || nkv < 1 || nq % nkv) return Q3_ERR_ARGUMENT;
  if (!paged_ok(q, q_stride, kpages, vpages, nq, nkv, ps) || ((uintptr_t)out & 15)) return Q3_ERR_UNSUPPORTED;
  if (num_work == 0) return Q3_OK;
  CUtensorMap tq, tk, tv;
  if (!q_map(&tq, q, D, nq, num_tokens, q_stride, nq / nkv) ||
      !q3_bf16_map(&tk, kpages, num_rows_kv, D, D, ps, CU_TENSOR_MAP_L2_PROMOTION_L2_128B) ||
      !q3_bf16_map(&tv, vpages, num_rows_kv, D, D, ps, CU_TENSOR_MAP_L2_PROMOTION_L2_128B))
    return Q3_ERR_LAUNCH;
  const Params p = {block_table, max_pages, kv_lens, cu_seqlens, (bf16*)out, num_seqs, num_work, nq, nkv, ps,
                    scale * LOG2_E, 0, chunk, window, nullptr, nullptr, nullptr, lambda, eps, out_scale, error_word};
  return launch<MAPS>(tq, tk, tv, tq, p, stream);
}

// Attention over expanded keys and values: q [num_tokens, heads, q_cols] with row stride q_stride, of which the first 128
// columns of a head are read; q_turned [num_tokens, heads, 64] dense: a head's part for the keys' shared columns; kv
// [rows, 2 * heads * 128]: the heads' own 128 key columns, then the heads' values; shared [rows, *] with row stride
// shared_stride: the 64 key columns that all heads share; key j of sequence s is row kv_base[s] + j (tiles of 64 keys are
// read from multiples of 64 on, the first one that holds the sequence's first visible key).  out [num_tokens, heads, 128].
// num_work = sum over sequences of ceil(ceil(q_len / 128) / 2).
Q3_EXPORT int q3_dense_attention_prefill_tc(const void* q, int q_cols, int q_stride, const void* q_turned, int num_tokens,
                                            const void* kv, const void* shared, long rows, long shared_stride,
                                            const int* kv_base, const int* kv_lens, const int* cu_seqlens, void* out,
                                            int num_seqs, int num_work, int heads, float scale, int window,
                                            const float* sinks, int* error_word, cudaStream_t stream) {
  if (!q || !q_turned || !kv || !shared || !kv_base || !kv_lens || !cu_seqlens || !out || heads < 1 || window < 0 || rows < 1 ||
      q_cols < D)
    return Q3_ERR_ARGUMENT;
  if (q_cols % 8 || q_stride % 8 || shared_stride % 8 ||
      (((uintptr_t)q | (uintptr_t)q_turned | (uintptr_t)kv | (uintptr_t)shared | (uintptr_t)out) & 15))
    return Q3_ERR_UNSUPPORTED;
  if (num_work == 0) return Q3_OK;
  const long cols = 2L * heads * D;
  CUtensorMap tq, tk, tv, tr;
  if (!q_map(&tq, q, q_cols, heads, num_tokens, q_stride, 1) || !q_map(&tr, q_turned, 64, heads, num_tokens, 64L * heads, 1) ||
      !q3_bf16_map(&tk, kv, rows, cols, cols, BLOCK_N, CU_TENSOR_MAP_L2_PROMOTION_L2_128B) ||
      !q3_bf16_map(&tv, shared, rows, 64, shared_stride, BLOCK_N, CU_TENSOR_MAP_L2_PROMOTION_L2_128B))
    return Q3_ERR_LAUNCH;
  const Params p = {nullptr, 0, kv_lens, cu_seqlens, (bf16*)out, num_seqs, num_work, heads, heads, BLOCK_N,
                    scale * LOG2_E, 0, 0, window, nullptr, sinks, kv_base, 0.f, 0.f, 0.f, error_word};
  return launch<DENSE>(tq, tk, tv, tr, p, stream);
}
