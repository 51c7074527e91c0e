// In-register DFT butterflies of radix 2, 3, 4, 5, 8 and 16.
//
// Forward uses W = exp(-2 pi i / R); INV flips the sign of every imaginary
// unit. Outputs are in natural order: v[m] <- sum_q v[q] W^{q m}. Constants
// are the exact values of cos/sin at the DFT angles.
//
// The passes are bound by the instructions they issue, so both components of
// a complex value go through one packed instruction (add, multiply, FMA on
// two FP32 values) wherever they meet the same operation; a rotation by +-i,
// which crosses the components, is folded into the additions after it. Every
// operation is spelled out (no expression that the compiler may contract into
// an FMA or not), so each kernel that runs the same transform rounds alike:
// the schedules of a solver give the same bits. A 16-point DFT is 106
// instructions instead of 164. Measured (iterations of all starts in one
// launch per pass, one component an instruction -> here): 16 starts of
// 480 x 480 52.7 -> 47.9 us, 16 of 240 x 240 18.2 -> 17.3, 4 of 128^3
// 111 -> 108 (bound by memory), 32 of 256 x 256 22.8 -> 22.0.
#pragma once

#include "common.cuh"

namespace qpb {

// a + W_4 d and a - W_4 d, W_4 = -i forward, +i inverse.
template <bool INV>
__device__ __forceinline__ float2 cadd_w4(float2 a, float2 d) {
  return INV ? float2{__fsub_rn(a.x, d.y), __fadd_rn(a.y, d.x)}
             : float2{__fadd_rn(a.x, d.y), __fsub_rn(a.y, d.x)};
}
template <bool INV>
__device__ __forceinline__ float2 csub_w4(float2 a, float2 d) {
  return cadd_w4<!INV>(a, d);
}

// a + s W_4 d and a - s W_4 d.
template <bool INV>
__device__ __forceinline__ float2 cfma_w4(float s, float2 d, float2 a) {
  return INV ? float2{fmaf(-s, d.y, a.x), fmaf(s, d.x, a.y)}
             : float2{fmaf(s, d.y, a.x), fmaf(-s, d.x, a.y)};
}

template <bool INV>
__device__ __forceinline__ void bfly2(float2& a, float2& b) {
  const float2 t = a;
  a = cadd(t, b);
  b = csub(t, b);
}

template <bool INV>
__device__ __forceinline__ void bfly4(float2& v0, float2& v1, float2& v2, float2& v3) {
  const float2 t0 = cadd(v0, v2);
  const float2 t1 = csub(v0, v2);
  const float2 t2 = cadd(v1, v3);
  const float2 t3 = csub(v1, v3);
  v0 = cadd(t0, t2);
  v2 = csub(t0, t2);
  v1 = cadd_w4<INV>(t1, t3);
  v3 = csub_w4<INV>(t1, t3);
}

// bfly4 of (v0, v1, W_4 v2, v3).
template <bool INV>
__device__ __forceinline__ void bfly4_w4(float2& v0, float2& v1, float2& v2, float2& v3) {
  const float2 t0 = cadd_w4<INV>(v0, v2);
  const float2 t1 = csub_w4<INV>(v0, v2);
  const float2 t2 = cadd(v1, v3);
  const float2 t3 = csub(v1, v3);
  v0 = cadd(t0, t2);
  v2 = csub(t0, t2);
  v1 = cadd_w4<INV>(t1, t3);
  v3 = csub_w4<INV>(t1, t3);
}

template <bool INV>
__device__ __forceinline__ void bfly3(float2& v0, float2& v1, float2& v2) {
  constexpr float kS = 0.86602540378443864676f;  // sin(2 pi / 3)
  const float2 t = cadd(v1, v2);
  const float2 m = cfma(-0.5f, t, v0);
  const float2 d = csub(v1, v2);
  v0 = cadd(v0, t);
  v1 = cfma_w4<INV>(kS, d, m);
  v2 = cfma_w4<INV>(-kS, d, m);
}

template <bool INV>
__device__ __forceinline__ void bfly5(float2& v0, float2& v1, float2& v2, float2& v3, float2& v4) {
  constexpr float c1 = 0.30901699437494742410f;   // cos(2 pi / 5)
  constexpr float c2 = -0.80901699437494742410f;  // cos(4 pi / 5)
  constexpr float s1 = 0.95105651629515357212f;   // sin(2 pi / 5)
  constexpr float s2 = 0.58778525229247312917f;   // sin(4 pi / 5)
  const float2 a1 = cadd(v1, v4);
  const float2 a2 = cadd(v2, v3);
  const float2 b1 = csub(v1, v4);
  const float2 b2 = csub(v2, v3);
  const float2 r1 = cfma(c2, a2, cfma(c1, a1, v0));
  const float2 r2 = cfma(c1, a2, cfma(c2, a1, v0));
  // forward X1 = r1 - i (s1 b1 + s2 b2), X2 = r2 - i (s2 b1 - s1 b2)
  const float2 q1 = cfma(s2, b2, cscale(b1, s1));
  const float2 q2 = cfma(-s1, b2, cscale(b1, s2));
  v0 = cadd(v0, cadd(a1, a2));
  v1 = cadd_w4<INV>(r1, q1);
  v4 = csub_w4<INV>(r1, q1);
  v2 = cadd_w4<INV>(r2, q2);
  v3 = csub_w4<INV>(r2, q2);
}

// sqrt(2) W_8^1 a, W_8^1 = (1 - i)/sqrt(2) forward, (1 + i)/sqrt(2) inverse.
template <bool INV>
__device__ __forceinline__ float2 mul_w8_root2(float2 a) {
  return cadd_w4<INV>(a, a);
}

// -sqrt(2) W_8^3 a, W_8^3 = (-1 - i)/sqrt(2) forward, (-1 + i)/sqrt(2) inverse.
template <bool INV>
__device__ __forceinline__ float2 mul_w8_3_root2(float2 a) {
  return csub_w4<INV>(a, a);
}

// v[0..7] in natural order.
template <bool INV>
__device__ __forceinline__ void bfly8(float2* v) {
  constexpr float r = 0.70710678118654752440f;
  // even / odd 4-point DFTs
  float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
  float2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  bfly4<INV>(e0, e1, e2, e3);
  bfly4<INV>(o0, o1, o2, o3);
  o1 = mul_w8_root2<INV>(o1);
  o3 = mul_w8_3_root2<INV>(o3);
  v[0] = cadd(e0, o0);
  v[4] = csub(e0, o0);
  v[1] = cfma(r, o1, e1);
  v[5] = cfma(-r, o1, e1);
  v[2] = cadd_w4<INV>(e2, o2);
  v[6] = csub_w4<INV>(e2, o2);
  v[3] = cfma(-r, o3, e3);
  v[7] = cfma(r, o3, e3);
}

// a (c, -s) forward, a (c, s) inverse, for constants c and s.
template <bool INV>
__device__ __forceinline__ float2 cmul_constant(float2 a, float c, float s) {
  return cfma_w4<INV>(s, a, cscale(a, c));
}

// v[0..15] in natural order: 4 x 4 with W_16 twiddles between the two levels.
template <bool INV>
__device__ __forceinline__ void bfly16(float2* v) {
  constexpr float c1 = 0.92387953251128675613f;  // cos(pi / 8)
  constexpr float s1 = 0.38268343236508977173f;  // sin(pi / 8)
  constexpr float r = 0.70710678118654752440f;
  // Level 1: for each n1 in 0..3, a 4-point DFT over v[n1 + 4 n2].
#pragma unroll
  for (int n1 = 0; n1 < 4; ++n1) bfly4<INV>(v[n1], v[n1 + 4], v[n1 + 8], v[n1 + 12]);
  // Twiddles W_16^{n1 k2} on v[n1 + 4 k2]; W^4 (v[10]) in its 4-point DFT.
  v[5] = cmul_constant<INV>(v[5], c1, s1);                   // W^1
  v[9] = cscale(mul_w8_root2<INV>(v[9]), r);                 // W^2
  v[13] = cmul_constant<INV>(v[13], s1, c1);                 // W^3
  v[6] = cscale(mul_w8_root2<INV>(v[6]), r);                 // W^2
  v[14] = cscale(mul_w8_3_root2<INV>(v[14]), -r);            // W^6
  v[7] = cmul_constant<INV>(v[7], s1, c1);                   // W^3
  v[11] = cscale(mul_w8_3_root2<INV>(v[11]), -r);            // W^6
  v[15] = cmul_constant<INV>(v[15], -c1, -s1);               // W^9 = -W^1
  // Level 2: for each k2, a 4-point DFT over n1: v[4 k2 + n1] lives at v[n1 + 4 k2].
  bfly4<INV>(v[0], v[1], v[2], v[3]);
  bfly4<INV>(v[4], v[5], v[6], v[7]);
  bfly4_w4<INV>(v[8], v[9], v[10], v[11]);
  bfly4<INV>(v[12], v[13], v[14], v[15]);
  // Output X[k2 + 4 k1] sits at v[4 k2 + k1]: transpose the 4x4 block.
  float2 t[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) t[i] = v[i];
#pragma unroll
  for (int k2 = 0; k2 < 4; ++k2) {
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) v[k2 + 4 * k1] = t[4 * k2 + k1];
  }
}

}  // namespace qpb
