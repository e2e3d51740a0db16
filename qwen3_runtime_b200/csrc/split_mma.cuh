// fp32 products of small matrices on mma.sync with every operand as the sum of three bfloat16 and the six products of parts that
// matter (the other three are below 2^-24 of a product together); shared by the chunked scans of delta_state.cu and
// linear_state.cu.  The split also by gemm_f32_split.cuh.
//
// Three bfloat16 hold 24 bits, so nothing of a value is lost as long as its third part is one: from about 2^-110 on.  Below, the parts
// end at the smallest bfloat16, 2^-133, and the value is off by 2^-134 at most (2^-118: 9e-6 of it, 2^-126: 2e-3).  Infinities,
// and what rounds up to one in bfloat16 (from 3.396e38 on), have no parts: their sum is NaN.
#pragma once
#include "mma_tiles.cuh"

__device__ __forceinline__ void ds_copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(dst)), "l"(src));
}

// (x, y) as the sum of three bfloat16 pairs
__device__ __forceinline__ void ds_split(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p[i]) : "f"(y), "f"(x));
    x -= __uint_as_float(p[i] << 16);
    y -= __uint_as_float(p[i] & 0xffff0000u);
  }
}

// four words of each of the three parts: a left operand, or two tiles of a right one
__device__ __forceinline__ void ds_parts(uint32_t (&p)[3][4], const uint32_t* from, int lane) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const uint4 w = *reinterpret_cast<const uint4*>(from + i * 128 + lane * 4);
    p[i][0] = w.x;
    p[i][1] = w.y;
    p[i][2] = w.z;
    p[i][3] = w.w;
  }
}
__device__ __forceinline__ void ds_mma_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// acc = a b over 16 channels (or tokens) for two tiles of eight rows (or channels), operands in three parts.  The largest
// product stands alone and is added last, rounded to nearest; the tiles' chains run side by side.
// EXACT_A, EXACT_B: that operand is bfloat16 as it is (its first part).
template <bool EXACT_B = false, bool EXACT_A = false>
__device__ __forceinline__ void ds_products(float (&acc)[2][4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][4]) {
  float small[2][4], mid[2][4];
  auto set = [&](float(&sum)[2][4], int i, int j) {
#pragma unroll
    for (int n = 0; n < 2; ++n) ds_mma_zero(sum[n], a[i], b[j][2 * n], b[j][2 * n + 1]);
  };
  auto add = [&](float(&sum)[2][4], int i, int j) {
#pragma unroll
    for (int n = 0; n < 2; ++n) mma_bf16(sum[n], a[i], b[j][2 * n], b[j][2 * n + 1]);
  };
  if constexpr (EXACT_A) {
    set(small, 0, 2);
    set(mid, 0, 1);
    set(acc, 0, 0);
  } else if constexpr (EXACT_B) {
    set(small, 2, 0);
    set(mid, 1, 0);
    set(acc, 0, 0);
  } else {
    set(small, 2, 0);
    set(mid, 0, 1);
    set(acc, 0, 0);
    add(small, 0, 2);
    add(mid, 1, 0);
    add(small, 1, 1);
  }
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[n][j] += mid[n][j] + small[n][j];
}
