// Rotation of one thread's share of a head by the angles of one position, shared by the kernel
// that rotates every token of a step (rope_kv.cu) and by the decode-attention kernel that makes
// the newest token's q and k itself (attention_decode.cu), so that both give the same bits.
//
// A head of D elements (D a multiple of 16, rotation over the whole head) is handled by D/16
// threads; thread c holds a[] = elements [8c, 8c+8) and b[] = elements [D/2 + 8c, D/2 + 8c + 8).
// `cos_row` / `sin_row` point at the D/2 angles of the token's position.
//   pairing 0 ("half"):        pair i = (i, i + D/2)  -- a[e] rotates with b[e], angle 8c + e
//   pairing 1 ("interleaved"): pair i = (2i, 2i + 1)  -- neighbours inside a[] (angles 4c ..)
//                                                        and inside b[] (angles D/4 + 4c ..)
#pragma once
#include "common.cuh"

struct Angles {
  float cs[8], sn[8];  // pairing 0: of elements 8c + e; 1: pairs 4c + 0..3 of a[], then of b[]
};
__device__ __forceinline__ Angles load_angles(const float* __restrict__ cos_row, const float* __restrict__ sin_row, int c, int half,
                                              int pairing) {
  Angles y;
  const int first = pairing ? 4 * c : 8 * c, second = pairing ? half / 2 + 4 * c : 8 * c + 4;
  const float4 ca = *reinterpret_cast<const float4*>(cos_row + first), cb = *reinterpret_cast<const float4*>(cos_row + second);
  const float4 sa = *reinterpret_cast<const float4*>(sin_row + first), sb = *reinterpret_cast<const float4*>(sin_row + second);
  y.cs[0] = ca.x, y.cs[1] = ca.y, y.cs[2] = ca.z, y.cs[3] = ca.w, y.cs[4] = cb.x, y.cs[5] = cb.y, y.cs[6] = cb.z, y.cs[7] = cb.w;
  y.sn[0] = sa.x, y.sn[1] = sa.y, y.sn[2] = sa.z, y.sn[3] = sa.w, y.sn[4] = sb.x, y.sn[5] = sb.y, y.sn[6] = sb.z, y.sn[7] = sb.w;
  return y;
}
__device__ __forceinline__ void rotate_by(float (&a)[8], float (&b)[8], const Angles& y, int pairing) {
  if (!pairing) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float ya = a[e], yb = b[e];
      a[e] = ya * y.cs[e] - yb * y.sn[e];
      b[e] = yb * y.cs[e] + ya * y.sn[e];
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float a0 = a[2 * j], a1 = a[2 * j + 1], b0 = b[2 * j], b1 = b[2 * j + 1];
    a[2 * j] = a0 * y.cs[j] - a1 * y.sn[j];
    a[2 * j + 1] = a1 * y.cs[j] + a0 * y.sn[j];
    b[2 * j] = b0 * y.cs[4 + j] - b1 * y.sn[4 + j];
    b[2 * j + 1] = b1 * y.cs[4 + j] + b0 * y.sn[4 + j];
  }
}
__device__ __forceinline__ void rotate_chunks(float (&a)[8], float (&b)[8], const float* __restrict__ cos_row,
                                              const float* __restrict__ sin_row, int c, int half, int pairing) {
  rotate_by(a, b, load_angles(cos_row, sin_row, c, half, pairing), pairing);
}
