// Packed FP32 arithmetic on two neighbouring columns (float2): the fma.f32x2 family of
// sm_100 issues both halves at once and rounds each as the scalar instruction does.
#pragma once
#include "lens_common.cuh"

LENS_HD float2 f2(float v) { return make_float2(v, v); }
LENS_HD float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
LENS_HD float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
LENS_HD float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
LENS_HD float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, f2(-1.f), a); }  // a - b, rounded once
LENS_HD float2 sel2(bool x, bool y, float2 a, float2 b) { return make_float2(x ? a.x : b.x, y ? a.y : b.y); }

// psi' = b psi + c d, the first product fused
LENS_HD float2 cell_psi(float2 b, float2 psi, float2 c, float2 d) { return fma2(b, psi, mul2(c, d)); }
