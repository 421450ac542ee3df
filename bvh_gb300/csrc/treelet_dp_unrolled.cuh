// treelet_dp_unrolled.cuh -- generated by gen_treelet_dp.py; do not edit.
//
// The LBVH+ subset DP (src/cuda/lbvh_plus_builder.cu:119-165) for N = 4..7 treelet leaves as
// straight-line code: subset costs in registers; this lane's shared-memory column A (stride 32)
// holds the subsets' areas and receives their costs.  Returns the full set's best split, 0 where
// no split is finite.
#pragma once

namespace bvhgb {

// 4 leaves: 25 split evaluations.
__device__ __forceinline__ uint32_t dp_unrolled_4(float* __restrict__ A) {
  const float c1 = 0.0f;
  A[1 * 32] = 0.0f;
  const float c2 = 0.0f;
  A[2 * 32] = 0.0f;
  const float c3 = __fadd_rn(fminf(kTlInf, __fadd_rn(c2, c1)), A[3 * 32]);
  A[3 * 32] = c3;
  const float c4 = 0.0f;
  A[4 * 32] = 0.0f;
  const float c5 = __fadd_rn(fminf(kTlInf, __fadd_rn(c4, c1)), A[5 * 32]);
  A[5 * 32] = c5;
  const float c6 = __fadd_rn(fminf(kTlInf, __fadd_rn(c4, c2)), A[6 * 32]);
  A[6 * 32] = c6;
  const float c7 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c5), __fadd_rn(c4, c3), __fadd_rn(c6, c1))), A[7 * 32]);
  A[7 * 32] = c7;
  const float c8 = 0.0f;
  A[8 * 32] = 0.0f;
  const float c9 = __fadd_rn(fminf(kTlInf, __fadd_rn(c8, c1)), A[9 * 32]);
  A[9 * 32] = c9;
  const float c10 = __fadd_rn(fminf(kTlInf, __fadd_rn(c8, c2)), A[10 * 32]);
  A[10 * 32] = c10;
  const float c11 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c9), __fadd_rn(c8, c3), __fadd_rn(c10, c1))), A[11 * 32]);
  A[11 * 32] = c11;
  const float c12 = __fadd_rn(fminf(kTlInf, __fadd_rn(c8, c4)), A[12 * 32]);
  A[12 * 32] = c12;
  const float c13 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c9), __fadd_rn(c8, c5), __fadd_rn(c12, c1))), A[13 * 32]);
  A[13 * 32] = c13;
  const float c14 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c10), __fadd_rn(c8, c6), __fadd_rn(c12, c2))), A[14 * 32]);
  A[14 * 32] = c14;
  float b = kTlInf, b2 = kTlInf, v, v2;
  uint32_t bp = 0u, bp2 = 0u;
  v = __fadd_rn(c2, c13);
  if (v < b) { b = v; bp = 2u; }
  v2 = __fadd_rn(c10, c5);
  if (v2 < b2) { b2 = v2; bp2 = 10u; }
  v = __fadd_rn(c4, c11);
  if (v < b) { b = v; bp = 4u; }
  v2 = __fadd_rn(c12, c3);
  if (v2 < b2) { b2 = v2; bp2 = 12u; }
  v = __fadd_rn(c6, c9);
  if (v < b) { b = v; bp = 6u; }
  v2 = __fadd_rn(c14, c1);
  if (v2 < b2) { b2 = v2; bp2 = 14u; }
  v = __fadd_rn(c8, c7);
  if (v < b) { b = v; bp = 8u; }
  return b2 < b ? bp2 : bp;
}

// 5 leaves: 90 split evaluations.
__device__ __forceinline__ uint32_t dp_unrolled_5(float* __restrict__ A) {
  const float c1 = 0.0f;
  A[1 * 32] = 0.0f;
  const float c2 = 0.0f;
  A[2 * 32] = 0.0f;
  const float c3 = __fadd_rn(fminf(kTlInf, __fadd_rn(c2, c1)), A[3 * 32]);
  A[3 * 32] = c3;
  const float c4 = 0.0f;
  A[4 * 32] = 0.0f;
  const float c5 = __fadd_rn(fminf(kTlInf, __fadd_rn(c4, c1)), A[5 * 32]);
  A[5 * 32] = c5;
  const float c6 = __fadd_rn(fminf(kTlInf, __fadd_rn(c4, c2)), A[6 * 32]);
  A[6 * 32] = c6;
  const float c7 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c5), __fadd_rn(c4, c3), __fadd_rn(c6, c1))), A[7 * 32]);
  A[7 * 32] = c7;
  const float c8 = 0.0f;
  A[8 * 32] = 0.0f;
  const float c9 = __fadd_rn(fminf(kTlInf, __fadd_rn(c8, c1)), A[9 * 32]);
  A[9 * 32] = c9;
  const float c10 = __fadd_rn(fminf(kTlInf, __fadd_rn(c8, c2)), A[10 * 32]);
  A[10 * 32] = c10;
  const float c11 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c9), __fadd_rn(c8, c3), __fadd_rn(c10, c1))), A[11 * 32]);
  A[11 * 32] = c11;
  const float c12 = __fadd_rn(fminf(kTlInf, __fadd_rn(c8, c4)), A[12 * 32]);
  A[12 * 32] = c12;
  const float c13 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c9), __fadd_rn(c8, c5), __fadd_rn(c12, c1))), A[13 * 32]);
  A[13 * 32] = c13;
  const float c14 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c10), __fadd_rn(c8, c6), __fadd_rn(c12, c2))), A[14 * 32]);
  A[14 * 32] = c14;
  const float c15 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c13), __fadd_rn(c4, c11), __fadd_rn(c6, c9)), min3f(__fadd_rn(c8, c7), __fadd_rn(c10, c5), __fadd_rn(c12, c3)), __fadd_rn(c14, c1))), A[15 * 32]);
  A[15 * 32] = c15;
  const float c16 = 0.0f;
  A[16 * 32] = 0.0f;
  const float c17 = __fadd_rn(fminf(kTlInf, __fadd_rn(c16, c1)), A[17 * 32]);
  A[17 * 32] = c17;
  const float c18 = __fadd_rn(fminf(kTlInf, __fadd_rn(c16, c2)), A[18 * 32]);
  A[18 * 32] = c18;
  const float c19 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c17), __fadd_rn(c16, c3), __fadd_rn(c18, c1))), A[19 * 32]);
  A[19 * 32] = c19;
  const float c20 = __fadd_rn(fminf(kTlInf, __fadd_rn(c16, c4)), A[20 * 32]);
  A[20 * 32] = c20;
  const float c21 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c17), __fadd_rn(c16, c5), __fadd_rn(c20, c1))), A[21 * 32]);
  A[21 * 32] = c21;
  const float c22 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c18), __fadd_rn(c16, c6), __fadd_rn(c20, c2))), A[22 * 32]);
  A[22 * 32] = c22;
  const float c23 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c21), __fadd_rn(c4, c19), __fadd_rn(c6, c17)), min3f(__fadd_rn(c16, c7), __fadd_rn(c18, c5), __fadd_rn(c20, c3)), __fadd_rn(c22, c1))), A[23 * 32]);
  A[23 * 32] = c23;
  const float c24 = __fadd_rn(fminf(kTlInf, __fadd_rn(c16, c8)), A[24 * 32]);
  A[24 * 32] = c24;
  const float c25 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c17), __fadd_rn(c16, c9), __fadd_rn(c24, c1))), A[25 * 32]);
  A[25 * 32] = c25;
  const float c26 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c18), __fadd_rn(c16, c10), __fadd_rn(c24, c2))), A[26 * 32]);
  A[26 * 32] = c26;
  const float c27 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c25), __fadd_rn(c8, c19), __fadd_rn(c10, c17)), min3f(__fadd_rn(c16, c11), __fadd_rn(c18, c9), __fadd_rn(c24, c3)), __fadd_rn(c26, c1))), A[27 * 32]);
  A[27 * 32] = c27;
  const float c28 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c20), __fadd_rn(c16, c12), __fadd_rn(c24, c4))), A[28 * 32]);
  A[28 * 32] = c28;
  const float c29 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c25), __fadd_rn(c8, c21), __fadd_rn(c12, c17)), min3f(__fadd_rn(c16, c13), __fadd_rn(c20, c9), __fadd_rn(c24, c5)), __fadd_rn(c28, c1))), A[29 * 32]);
  A[29 * 32] = c29;
  const float c30 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c26), __fadd_rn(c8, c22), __fadd_rn(c12, c18)), min3f(__fadd_rn(c16, c14), __fadd_rn(c20, c10), __fadd_rn(c24, c6)), __fadd_rn(c28, c2))), A[30 * 32]);
  A[30 * 32] = c30;
  float b = kTlInf, b2 = kTlInf, v, v2;
  uint32_t bp = 0u, bp2 = 0u;
  v = __fadd_rn(c2, c29);
  if (v < b) { b = v; bp = 2u; }
  v2 = __fadd_rn(c18, c13);
  if (v2 < b2) { b2 = v2; bp2 = 18u; }
  v = __fadd_rn(c4, c27);
  if (v < b) { b = v; bp = 4u; }
  v2 = __fadd_rn(c20, c11);
  if (v2 < b2) { b2 = v2; bp2 = 20u; }
  v = __fadd_rn(c6, c25);
  if (v < b) { b = v; bp = 6u; }
  v2 = __fadd_rn(c22, c9);
  if (v2 < b2) { b2 = v2; bp2 = 22u; }
  v = __fadd_rn(c8, c23);
  if (v < b) { b = v; bp = 8u; }
  v2 = __fadd_rn(c24, c7);
  if (v2 < b2) { b2 = v2; bp2 = 24u; }
  v = __fadd_rn(c10, c21);
  if (v < b) { b = v; bp = 10u; }
  v2 = __fadd_rn(c26, c5);
  if (v2 < b2) { b2 = v2; bp2 = 26u; }
  v = __fadd_rn(c12, c19);
  if (v < b) { b = v; bp = 12u; }
  v2 = __fadd_rn(c28, c3);
  if (v2 < b2) { b2 = v2; bp2 = 28u; }
  v = __fadd_rn(c14, c17);
  if (v < b) { b = v; bp = 14u; }
  v2 = __fadd_rn(c30, c1);
  if (v2 < b2) { b2 = v2; bp2 = 30u; }
  v = __fadd_rn(c16, c15);
  if (v < b) { b = v; bp = 16u; }
  return b2 < b ? bp2 : bp;
}

// 6 leaves: 301 split evaluations.
__device__ __forceinline__ uint32_t dp_unrolled_6(float* __restrict__ A) {
  const float c1 = 0.0f;
  A[1 * 32] = 0.0f;
  const float c2 = 0.0f;
  A[2 * 32] = 0.0f;
  const float c3 = __fadd_rn(fminf(kTlInf, __fadd_rn(c2, c1)), A[3 * 32]);
  A[3 * 32] = c3;
  const float c4 = 0.0f;
  A[4 * 32] = 0.0f;
  const float c5 = __fadd_rn(fminf(kTlInf, __fadd_rn(c4, c1)), A[5 * 32]);
  A[5 * 32] = c5;
  const float c6 = __fadd_rn(fminf(kTlInf, __fadd_rn(c4, c2)), A[6 * 32]);
  A[6 * 32] = c6;
  const float c7 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c5), __fadd_rn(c4, c3), __fadd_rn(c6, c1))), A[7 * 32]);
  A[7 * 32] = c7;
  const float c8 = 0.0f;
  A[8 * 32] = 0.0f;
  const float c9 = __fadd_rn(fminf(kTlInf, __fadd_rn(c8, c1)), A[9 * 32]);
  A[9 * 32] = c9;
  const float c10 = __fadd_rn(fminf(kTlInf, __fadd_rn(c8, c2)), A[10 * 32]);
  A[10 * 32] = c10;
  const float c11 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c9), __fadd_rn(c8, c3), __fadd_rn(c10, c1))), A[11 * 32]);
  A[11 * 32] = c11;
  const float c12 = __fadd_rn(fminf(kTlInf, __fadd_rn(c8, c4)), A[12 * 32]);
  A[12 * 32] = c12;
  const float c13 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c9), __fadd_rn(c8, c5), __fadd_rn(c12, c1))), A[13 * 32]);
  A[13 * 32] = c13;
  const float c14 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c10), __fadd_rn(c8, c6), __fadd_rn(c12, c2))), A[14 * 32]);
  A[14 * 32] = c14;
  const float c15 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c13), __fadd_rn(c4, c11), __fadd_rn(c6, c9)), min3f(__fadd_rn(c8, c7), __fadd_rn(c10, c5), __fadd_rn(c12, c3)), __fadd_rn(c14, c1))), A[15 * 32]);
  A[15 * 32] = c15;
  const float c16 = 0.0f;
  A[16 * 32] = 0.0f;
  const float c17 = __fadd_rn(fminf(kTlInf, __fadd_rn(c16, c1)), A[17 * 32]);
  A[17 * 32] = c17;
  const float c18 = __fadd_rn(fminf(kTlInf, __fadd_rn(c16, c2)), A[18 * 32]);
  A[18 * 32] = c18;
  const float c19 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c17), __fadd_rn(c16, c3), __fadd_rn(c18, c1))), A[19 * 32]);
  A[19 * 32] = c19;
  const float c20 = __fadd_rn(fminf(kTlInf, __fadd_rn(c16, c4)), A[20 * 32]);
  A[20 * 32] = c20;
  const float c21 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c17), __fadd_rn(c16, c5), __fadd_rn(c20, c1))), A[21 * 32]);
  A[21 * 32] = c21;
  const float c22 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c18), __fadd_rn(c16, c6), __fadd_rn(c20, c2))), A[22 * 32]);
  A[22 * 32] = c22;
  const float c23 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c21), __fadd_rn(c4, c19), __fadd_rn(c6, c17)), min3f(__fadd_rn(c16, c7), __fadd_rn(c18, c5), __fadd_rn(c20, c3)), __fadd_rn(c22, c1))), A[23 * 32]);
  A[23 * 32] = c23;
  const float c24 = __fadd_rn(fminf(kTlInf, __fadd_rn(c16, c8)), A[24 * 32]);
  A[24 * 32] = c24;
  const float c25 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c17), __fadd_rn(c16, c9), __fadd_rn(c24, c1))), A[25 * 32]);
  A[25 * 32] = c25;
  const float c26 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c18), __fadd_rn(c16, c10), __fadd_rn(c24, c2))), A[26 * 32]);
  A[26 * 32] = c26;
  const float c27 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c25), __fadd_rn(c8, c19), __fadd_rn(c10, c17)), min3f(__fadd_rn(c16, c11), __fadd_rn(c18, c9), __fadd_rn(c24, c3)), __fadd_rn(c26, c1))), A[27 * 32]);
  A[27 * 32] = c27;
  const float c28 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c20), __fadd_rn(c16, c12), __fadd_rn(c24, c4))), A[28 * 32]);
  A[28 * 32] = c28;
  const float c29 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c25), __fadd_rn(c8, c21), __fadd_rn(c12, c17)), min3f(__fadd_rn(c16, c13), __fadd_rn(c20, c9), __fadd_rn(c24, c5)), __fadd_rn(c28, c1))), A[29 * 32]);
  A[29 * 32] = c29;
  const float c30 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c26), __fadd_rn(c8, c22), __fadd_rn(c12, c18)), min3f(__fadd_rn(c16, c14), __fadd_rn(c20, c10), __fadd_rn(c24, c6)), __fadd_rn(c28, c2))), A[30 * 32]);
  A[30 * 32] = c30;
  const float c31 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c29), __fadd_rn(c4, c27), __fadd_rn(c6, c25)), min3f(__fadd_rn(c8, c23), __fadd_rn(c10, c21), __fadd_rn(c12, c19)), min3f(__fadd_rn(c14, c17), __fadd_rn(c16, c15), __fadd_rn(c18, c13))), min3f(__fadd_rn(c20, c11), __fadd_rn(c22, c9), __fadd_rn(c24, c7)), min3f(__fadd_rn(c26, c5), __fadd_rn(c28, c3), __fadd_rn(c30, c1)))), A[31 * 32]);
  A[31 * 32] = c31;
  const float c32 = 0.0f;
  A[32 * 32] = 0.0f;
  const float c33 = __fadd_rn(fminf(kTlInf, __fadd_rn(c32, c1)), A[33 * 32]);
  A[33 * 32] = c33;
  const float c34 = __fadd_rn(fminf(kTlInf, __fadd_rn(c32, c2)), A[34 * 32]);
  A[34 * 32] = c34;
  const float c35 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c33), __fadd_rn(c32, c3), __fadd_rn(c34, c1))), A[35 * 32]);
  A[35 * 32] = c35;
  const float c36 = __fadd_rn(fminf(kTlInf, __fadd_rn(c32, c4)), A[36 * 32]);
  A[36 * 32] = c36;
  const float c37 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c33), __fadd_rn(c32, c5), __fadd_rn(c36, c1))), A[37 * 32]);
  A[37 * 32] = c37;
  const float c38 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c34), __fadd_rn(c32, c6), __fadd_rn(c36, c2))), A[38 * 32]);
  A[38 * 32] = c38;
  const float c39 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c37), __fadd_rn(c4, c35), __fadd_rn(c6, c33)), min3f(__fadd_rn(c32, c7), __fadd_rn(c34, c5), __fadd_rn(c36, c3)), __fadd_rn(c38, c1))), A[39 * 32]);
  A[39 * 32] = c39;
  const float c40 = __fadd_rn(fminf(kTlInf, __fadd_rn(c32, c8)), A[40 * 32]);
  A[40 * 32] = c40;
  const float c41 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c33), __fadd_rn(c32, c9), __fadd_rn(c40, c1))), A[41 * 32]);
  A[41 * 32] = c41;
  const float c42 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c34), __fadd_rn(c32, c10), __fadd_rn(c40, c2))), A[42 * 32]);
  A[42 * 32] = c42;
  const float c43 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c41), __fadd_rn(c8, c35), __fadd_rn(c10, c33)), min3f(__fadd_rn(c32, c11), __fadd_rn(c34, c9), __fadd_rn(c40, c3)), __fadd_rn(c42, c1))), A[43 * 32]);
  A[43 * 32] = c43;
  const float c44 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c36), __fadd_rn(c32, c12), __fadd_rn(c40, c4))), A[44 * 32]);
  A[44 * 32] = c44;
  const float c45 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c41), __fadd_rn(c8, c37), __fadd_rn(c12, c33)), min3f(__fadd_rn(c32, c13), __fadd_rn(c36, c9), __fadd_rn(c40, c5)), __fadd_rn(c44, c1))), A[45 * 32]);
  A[45 * 32] = c45;
  const float c46 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c42), __fadd_rn(c8, c38), __fadd_rn(c12, c34)), min3f(__fadd_rn(c32, c14), __fadd_rn(c36, c10), __fadd_rn(c40, c6)), __fadd_rn(c44, c2))), A[46 * 32]);
  A[46 * 32] = c46;
  const float c47 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c45), __fadd_rn(c4, c43), __fadd_rn(c6, c41)), min3f(__fadd_rn(c8, c39), __fadd_rn(c10, c37), __fadd_rn(c12, c35)), min3f(__fadd_rn(c14, c33), __fadd_rn(c32, c15), __fadd_rn(c34, c13))), min3f(__fadd_rn(c36, c11), __fadd_rn(c38, c9), __fadd_rn(c40, c7)), min3f(__fadd_rn(c42, c5), __fadd_rn(c44, c3), __fadd_rn(c46, c1)))), A[47 * 32]);
  A[47 * 32] = c47;
  const float c48 = __fadd_rn(fminf(kTlInf, __fadd_rn(c32, c16)), A[48 * 32]);
  A[48 * 32] = c48;
  const float c49 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c16, c33), __fadd_rn(c32, c17), __fadd_rn(c48, c1))), A[49 * 32]);
  A[49 * 32] = c49;
  const float c50 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c16, c34), __fadd_rn(c32, c18), __fadd_rn(c48, c2))), A[50 * 32]);
  A[50 * 32] = c50;
  const float c51 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c49), __fadd_rn(c16, c35), __fadd_rn(c18, c33)), min3f(__fadd_rn(c32, c19), __fadd_rn(c34, c17), __fadd_rn(c48, c3)), __fadd_rn(c50, c1))), A[51 * 32]);
  A[51 * 32] = c51;
  const float c52 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c16, c36), __fadd_rn(c32, c20), __fadd_rn(c48, c4))), A[52 * 32]);
  A[52 * 32] = c52;
  const float c53 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c49), __fadd_rn(c16, c37), __fadd_rn(c20, c33)), min3f(__fadd_rn(c32, c21), __fadd_rn(c36, c17), __fadd_rn(c48, c5)), __fadd_rn(c52, c1))), A[53 * 32]);
  A[53 * 32] = c53;
  const float c54 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c50), __fadd_rn(c16, c38), __fadd_rn(c20, c34)), min3f(__fadd_rn(c32, c22), __fadd_rn(c36, c18), __fadd_rn(c48, c6)), __fadd_rn(c52, c2))), A[54 * 32]);
  A[54 * 32] = c54;
  const float c55 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c53), __fadd_rn(c4, c51), __fadd_rn(c6, c49)), min3f(__fadd_rn(c16, c39), __fadd_rn(c18, c37), __fadd_rn(c20, c35)), min3f(__fadd_rn(c22, c33), __fadd_rn(c32, c23), __fadd_rn(c34, c21))), min3f(__fadd_rn(c36, c19), __fadd_rn(c38, c17), __fadd_rn(c48, c7)), min3f(__fadd_rn(c50, c5), __fadd_rn(c52, c3), __fadd_rn(c54, c1)))), A[55 * 32]);
  A[55 * 32] = c55;
  const float c56 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c16, c40), __fadd_rn(c32, c24), __fadd_rn(c48, c8))), A[56 * 32]);
  A[56 * 32] = c56;
  const float c57 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c8, c49), __fadd_rn(c16, c41), __fadd_rn(c24, c33)), min3f(__fadd_rn(c32, c25), __fadd_rn(c40, c17), __fadd_rn(c48, c9)), __fadd_rn(c56, c1))), A[57 * 32]);
  A[57 * 32] = c57;
  const float c58 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c8, c50), __fadd_rn(c16, c42), __fadd_rn(c24, c34)), min3f(__fadd_rn(c32, c26), __fadd_rn(c40, c18), __fadd_rn(c48, c10)), __fadd_rn(c56, c2))), A[58 * 32]);
  A[58 * 32] = c58;
  const float c59 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c57), __fadd_rn(c8, c51), __fadd_rn(c10, c49)), min3f(__fadd_rn(c16, c43), __fadd_rn(c18, c41), __fadd_rn(c24, c35)), min3f(__fadd_rn(c26, c33), __fadd_rn(c32, c27), __fadd_rn(c34, c25))), min3f(__fadd_rn(c40, c19), __fadd_rn(c42, c17), __fadd_rn(c48, c11)), min3f(__fadd_rn(c50, c9), __fadd_rn(c56, c3), __fadd_rn(c58, c1)))), A[59 * 32]);
  A[59 * 32] = c59;
  const float c60 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c8, c52), __fadd_rn(c16, c44), __fadd_rn(c24, c36)), min3f(__fadd_rn(c32, c28), __fadd_rn(c40, c20), __fadd_rn(c48, c12)), __fadd_rn(c56, c4))), A[60 * 32]);
  A[60 * 32] = c60;
  const float c61 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c4, c57), __fadd_rn(c8, c53), __fadd_rn(c12, c49)), min3f(__fadd_rn(c16, c45), __fadd_rn(c20, c41), __fadd_rn(c24, c37)), min3f(__fadd_rn(c28, c33), __fadd_rn(c32, c29), __fadd_rn(c36, c25))), min3f(__fadd_rn(c40, c21), __fadd_rn(c44, c17), __fadd_rn(c48, c13)), min3f(__fadd_rn(c52, c9), __fadd_rn(c56, c5), __fadd_rn(c60, c1)))), A[61 * 32]);
  A[61 * 32] = c61;
  const float c62 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c4, c58), __fadd_rn(c8, c54), __fadd_rn(c12, c50)), min3f(__fadd_rn(c16, c46), __fadd_rn(c20, c42), __fadd_rn(c24, c38)), min3f(__fadd_rn(c28, c34), __fadd_rn(c32, c30), __fadd_rn(c36, c26))), min3f(__fadd_rn(c40, c22), __fadd_rn(c44, c18), __fadd_rn(c48, c14)), min3f(__fadd_rn(c52, c10), __fadd_rn(c56, c6), __fadd_rn(c60, c2)))), A[62 * 32]);
  A[62 * 32] = c62;
  float b = kTlInf, b2 = kTlInf, v, v2;
  uint32_t bp = 0u, bp2 = 0u;
  v = __fadd_rn(c2, c61);
  if (v < b) { b = v; bp = 2u; }
  v2 = __fadd_rn(c34, c29);
  if (v2 < b2) { b2 = v2; bp2 = 34u; }
  v = __fadd_rn(c4, c59);
  if (v < b) { b = v; bp = 4u; }
  v2 = __fadd_rn(c36, c27);
  if (v2 < b2) { b2 = v2; bp2 = 36u; }
  v = __fadd_rn(c6, c57);
  if (v < b) { b = v; bp = 6u; }
  v2 = __fadd_rn(c38, c25);
  if (v2 < b2) { b2 = v2; bp2 = 38u; }
  v = __fadd_rn(c8, c55);
  if (v < b) { b = v; bp = 8u; }
  v2 = __fadd_rn(c40, c23);
  if (v2 < b2) { b2 = v2; bp2 = 40u; }
  v = __fadd_rn(c10, c53);
  if (v < b) { b = v; bp = 10u; }
  v2 = __fadd_rn(c42, c21);
  if (v2 < b2) { b2 = v2; bp2 = 42u; }
  v = __fadd_rn(c12, c51);
  if (v < b) { b = v; bp = 12u; }
  v2 = __fadd_rn(c44, c19);
  if (v2 < b2) { b2 = v2; bp2 = 44u; }
  v = __fadd_rn(c14, c49);
  if (v < b) { b = v; bp = 14u; }
  v2 = __fadd_rn(c46, c17);
  if (v2 < b2) { b2 = v2; bp2 = 46u; }
  v = __fadd_rn(c16, c47);
  if (v < b) { b = v; bp = 16u; }
  v2 = __fadd_rn(c48, c15);
  if (v2 < b2) { b2 = v2; bp2 = 48u; }
  v = __fadd_rn(c18, c45);
  if (v < b) { b = v; bp = 18u; }
  v2 = __fadd_rn(c50, c13);
  if (v2 < b2) { b2 = v2; bp2 = 50u; }
  v = __fadd_rn(c20, c43);
  if (v < b) { b = v; bp = 20u; }
  v2 = __fadd_rn(c52, c11);
  if (v2 < b2) { b2 = v2; bp2 = 52u; }
  v = __fadd_rn(c22, c41);
  if (v < b) { b = v; bp = 22u; }
  v2 = __fadd_rn(c54, c9);
  if (v2 < b2) { b2 = v2; bp2 = 54u; }
  v = __fadd_rn(c24, c39);
  if (v < b) { b = v; bp = 24u; }
  v2 = __fadd_rn(c56, c7);
  if (v2 < b2) { b2 = v2; bp2 = 56u; }
  v = __fadd_rn(c26, c37);
  if (v < b) { b = v; bp = 26u; }
  v2 = __fadd_rn(c58, c5);
  if (v2 < b2) { b2 = v2; bp2 = 58u; }
  v = __fadd_rn(c28, c35);
  if (v < b) { b = v; bp = 28u; }
  v2 = __fadd_rn(c60, c3);
  if (v2 < b2) { b2 = v2; bp2 = 60u; }
  v = __fadd_rn(c30, c33);
  if (v < b) { b = v; bp = 30u; }
  v2 = __fadd_rn(c62, c1);
  if (v2 < b2) { b2 = v2; bp2 = 62u; }
  v = __fadd_rn(c32, c31);
  if (v < b) { b = v; bp = 32u; }
  return b2 < b ? bp2 : bp;
}

// 7 leaves: 966 split evaluations.
__device__ __forceinline__ uint32_t dp_unrolled_7(float* __restrict__ A) {
  const float c1 = 0.0f;
  A[1 * 32] = 0.0f;
  const float c2 = 0.0f;
  A[2 * 32] = 0.0f;
  const float c3 = __fadd_rn(fminf(kTlInf, __fadd_rn(c2, c1)), A[3 * 32]);
  A[3 * 32] = c3;
  const float c4 = 0.0f;
  A[4 * 32] = 0.0f;
  const float c5 = __fadd_rn(fminf(kTlInf, __fadd_rn(c4, c1)), A[5 * 32]);
  A[5 * 32] = c5;
  const float c6 = __fadd_rn(fminf(kTlInf, __fadd_rn(c4, c2)), A[6 * 32]);
  A[6 * 32] = c6;
  const float c7 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c5), __fadd_rn(c4, c3), __fadd_rn(c6, c1))), A[7 * 32]);
  A[7 * 32] = c7;
  const float c8 = 0.0f;
  A[8 * 32] = 0.0f;
  const float c9 = __fadd_rn(fminf(kTlInf, __fadd_rn(c8, c1)), A[9 * 32]);
  A[9 * 32] = c9;
  const float c10 = __fadd_rn(fminf(kTlInf, __fadd_rn(c8, c2)), A[10 * 32]);
  A[10 * 32] = c10;
  const float c11 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c9), __fadd_rn(c8, c3), __fadd_rn(c10, c1))), A[11 * 32]);
  A[11 * 32] = c11;
  const float c12 = __fadd_rn(fminf(kTlInf, __fadd_rn(c8, c4)), A[12 * 32]);
  A[12 * 32] = c12;
  const float c13 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c9), __fadd_rn(c8, c5), __fadd_rn(c12, c1))), A[13 * 32]);
  A[13 * 32] = c13;
  const float c14 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c10), __fadd_rn(c8, c6), __fadd_rn(c12, c2))), A[14 * 32]);
  A[14 * 32] = c14;
  const float c15 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c13), __fadd_rn(c4, c11), __fadd_rn(c6, c9)), min3f(__fadd_rn(c8, c7), __fadd_rn(c10, c5), __fadd_rn(c12, c3)), __fadd_rn(c14, c1))), A[15 * 32]);
  A[15 * 32] = c15;
  const float c16 = 0.0f;
  A[16 * 32] = 0.0f;
  const float c17 = __fadd_rn(fminf(kTlInf, __fadd_rn(c16, c1)), A[17 * 32]);
  A[17 * 32] = c17;
  const float c18 = __fadd_rn(fminf(kTlInf, __fadd_rn(c16, c2)), A[18 * 32]);
  A[18 * 32] = c18;
  const float c19 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c17), __fadd_rn(c16, c3), __fadd_rn(c18, c1))), A[19 * 32]);
  A[19 * 32] = c19;
  const float c20 = __fadd_rn(fminf(kTlInf, __fadd_rn(c16, c4)), A[20 * 32]);
  A[20 * 32] = c20;
  const float c21 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c17), __fadd_rn(c16, c5), __fadd_rn(c20, c1))), A[21 * 32]);
  A[21 * 32] = c21;
  const float c22 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c18), __fadd_rn(c16, c6), __fadd_rn(c20, c2))), A[22 * 32]);
  A[22 * 32] = c22;
  const float c23 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c21), __fadd_rn(c4, c19), __fadd_rn(c6, c17)), min3f(__fadd_rn(c16, c7), __fadd_rn(c18, c5), __fadd_rn(c20, c3)), __fadd_rn(c22, c1))), A[23 * 32]);
  A[23 * 32] = c23;
  const float c24 = __fadd_rn(fminf(kTlInf, __fadd_rn(c16, c8)), A[24 * 32]);
  A[24 * 32] = c24;
  const float c25 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c17), __fadd_rn(c16, c9), __fadd_rn(c24, c1))), A[25 * 32]);
  A[25 * 32] = c25;
  const float c26 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c18), __fadd_rn(c16, c10), __fadd_rn(c24, c2))), A[26 * 32]);
  A[26 * 32] = c26;
  const float c27 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c25), __fadd_rn(c8, c19), __fadd_rn(c10, c17)), min3f(__fadd_rn(c16, c11), __fadd_rn(c18, c9), __fadd_rn(c24, c3)), __fadd_rn(c26, c1))), A[27 * 32]);
  A[27 * 32] = c27;
  const float c28 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c20), __fadd_rn(c16, c12), __fadd_rn(c24, c4))), A[28 * 32]);
  A[28 * 32] = c28;
  const float c29 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c25), __fadd_rn(c8, c21), __fadd_rn(c12, c17)), min3f(__fadd_rn(c16, c13), __fadd_rn(c20, c9), __fadd_rn(c24, c5)), __fadd_rn(c28, c1))), A[29 * 32]);
  A[29 * 32] = c29;
  const float c30 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c26), __fadd_rn(c8, c22), __fadd_rn(c12, c18)), min3f(__fadd_rn(c16, c14), __fadd_rn(c20, c10), __fadd_rn(c24, c6)), __fadd_rn(c28, c2))), A[30 * 32]);
  A[30 * 32] = c30;
  const float c31 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c29), __fadd_rn(c4, c27), __fadd_rn(c6, c25)), min3f(__fadd_rn(c8, c23), __fadd_rn(c10, c21), __fadd_rn(c12, c19)), min3f(__fadd_rn(c14, c17), __fadd_rn(c16, c15), __fadd_rn(c18, c13))), min3f(__fadd_rn(c20, c11), __fadd_rn(c22, c9), __fadd_rn(c24, c7)), min3f(__fadd_rn(c26, c5), __fadd_rn(c28, c3), __fadd_rn(c30, c1)))), A[31 * 32]);
  A[31 * 32] = c31;
  const float c32 = 0.0f;
  A[32 * 32] = 0.0f;
  const float c33 = __fadd_rn(fminf(kTlInf, __fadd_rn(c32, c1)), A[33 * 32]);
  A[33 * 32] = c33;
  const float c34 = __fadd_rn(fminf(kTlInf, __fadd_rn(c32, c2)), A[34 * 32]);
  A[34 * 32] = c34;
  const float c35 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c33), __fadd_rn(c32, c3), __fadd_rn(c34, c1))), A[35 * 32]);
  A[35 * 32] = c35;
  const float c36 = __fadd_rn(fminf(kTlInf, __fadd_rn(c32, c4)), A[36 * 32]);
  A[36 * 32] = c36;
  const float c37 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c33), __fadd_rn(c32, c5), __fadd_rn(c36, c1))), A[37 * 32]);
  A[37 * 32] = c37;
  const float c38 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c34), __fadd_rn(c32, c6), __fadd_rn(c36, c2))), A[38 * 32]);
  A[38 * 32] = c38;
  const float c39 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c37), __fadd_rn(c4, c35), __fadd_rn(c6, c33)), min3f(__fadd_rn(c32, c7), __fadd_rn(c34, c5), __fadd_rn(c36, c3)), __fadd_rn(c38, c1))), A[39 * 32]);
  A[39 * 32] = c39;
  const float c40 = __fadd_rn(fminf(kTlInf, __fadd_rn(c32, c8)), A[40 * 32]);
  A[40 * 32] = c40;
  const float c41 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c33), __fadd_rn(c32, c9), __fadd_rn(c40, c1))), A[41 * 32]);
  A[41 * 32] = c41;
  const float c42 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c34), __fadd_rn(c32, c10), __fadd_rn(c40, c2))), A[42 * 32]);
  A[42 * 32] = c42;
  const float c43 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c41), __fadd_rn(c8, c35), __fadd_rn(c10, c33)), min3f(__fadd_rn(c32, c11), __fadd_rn(c34, c9), __fadd_rn(c40, c3)), __fadd_rn(c42, c1))), A[43 * 32]);
  A[43 * 32] = c43;
  const float c44 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c36), __fadd_rn(c32, c12), __fadd_rn(c40, c4))), A[44 * 32]);
  A[44 * 32] = c44;
  const float c45 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c41), __fadd_rn(c8, c37), __fadd_rn(c12, c33)), min3f(__fadd_rn(c32, c13), __fadd_rn(c36, c9), __fadd_rn(c40, c5)), __fadd_rn(c44, c1))), A[45 * 32]);
  A[45 * 32] = c45;
  const float c46 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c42), __fadd_rn(c8, c38), __fadd_rn(c12, c34)), min3f(__fadd_rn(c32, c14), __fadd_rn(c36, c10), __fadd_rn(c40, c6)), __fadd_rn(c44, c2))), A[46 * 32]);
  A[46 * 32] = c46;
  const float c47 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c45), __fadd_rn(c4, c43), __fadd_rn(c6, c41)), min3f(__fadd_rn(c8, c39), __fadd_rn(c10, c37), __fadd_rn(c12, c35)), min3f(__fadd_rn(c14, c33), __fadd_rn(c32, c15), __fadd_rn(c34, c13))), min3f(__fadd_rn(c36, c11), __fadd_rn(c38, c9), __fadd_rn(c40, c7)), min3f(__fadd_rn(c42, c5), __fadd_rn(c44, c3), __fadd_rn(c46, c1)))), A[47 * 32]);
  A[47 * 32] = c47;
  const float c48 = __fadd_rn(fminf(kTlInf, __fadd_rn(c32, c16)), A[48 * 32]);
  A[48 * 32] = c48;
  const float c49 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c16, c33), __fadd_rn(c32, c17), __fadd_rn(c48, c1))), A[49 * 32]);
  A[49 * 32] = c49;
  const float c50 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c16, c34), __fadd_rn(c32, c18), __fadd_rn(c48, c2))), A[50 * 32]);
  A[50 * 32] = c50;
  const float c51 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c49), __fadd_rn(c16, c35), __fadd_rn(c18, c33)), min3f(__fadd_rn(c32, c19), __fadd_rn(c34, c17), __fadd_rn(c48, c3)), __fadd_rn(c50, c1))), A[51 * 32]);
  A[51 * 32] = c51;
  const float c52 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c16, c36), __fadd_rn(c32, c20), __fadd_rn(c48, c4))), A[52 * 32]);
  A[52 * 32] = c52;
  const float c53 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c49), __fadd_rn(c16, c37), __fadd_rn(c20, c33)), min3f(__fadd_rn(c32, c21), __fadd_rn(c36, c17), __fadd_rn(c48, c5)), __fadd_rn(c52, c1))), A[53 * 32]);
  A[53 * 32] = c53;
  const float c54 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c50), __fadd_rn(c16, c38), __fadd_rn(c20, c34)), min3f(__fadd_rn(c32, c22), __fadd_rn(c36, c18), __fadd_rn(c48, c6)), __fadd_rn(c52, c2))), A[54 * 32]);
  A[54 * 32] = c54;
  const float c55 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c53), __fadd_rn(c4, c51), __fadd_rn(c6, c49)), min3f(__fadd_rn(c16, c39), __fadd_rn(c18, c37), __fadd_rn(c20, c35)), min3f(__fadd_rn(c22, c33), __fadd_rn(c32, c23), __fadd_rn(c34, c21))), min3f(__fadd_rn(c36, c19), __fadd_rn(c38, c17), __fadd_rn(c48, c7)), min3f(__fadd_rn(c50, c5), __fadd_rn(c52, c3), __fadd_rn(c54, c1)))), A[55 * 32]);
  A[55 * 32] = c55;
  const float c56 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c16, c40), __fadd_rn(c32, c24), __fadd_rn(c48, c8))), A[56 * 32]);
  A[56 * 32] = c56;
  const float c57 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c8, c49), __fadd_rn(c16, c41), __fadd_rn(c24, c33)), min3f(__fadd_rn(c32, c25), __fadd_rn(c40, c17), __fadd_rn(c48, c9)), __fadd_rn(c56, c1))), A[57 * 32]);
  A[57 * 32] = c57;
  const float c58 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c8, c50), __fadd_rn(c16, c42), __fadd_rn(c24, c34)), min3f(__fadd_rn(c32, c26), __fadd_rn(c40, c18), __fadd_rn(c48, c10)), __fadd_rn(c56, c2))), A[58 * 32]);
  A[58 * 32] = c58;
  const float c59 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c57), __fadd_rn(c8, c51), __fadd_rn(c10, c49)), min3f(__fadd_rn(c16, c43), __fadd_rn(c18, c41), __fadd_rn(c24, c35)), min3f(__fadd_rn(c26, c33), __fadd_rn(c32, c27), __fadd_rn(c34, c25))), min3f(__fadd_rn(c40, c19), __fadd_rn(c42, c17), __fadd_rn(c48, c11)), min3f(__fadd_rn(c50, c9), __fadd_rn(c56, c3), __fadd_rn(c58, c1)))), A[59 * 32]);
  A[59 * 32] = c59;
  const float c60 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c8, c52), __fadd_rn(c16, c44), __fadd_rn(c24, c36)), min3f(__fadd_rn(c32, c28), __fadd_rn(c40, c20), __fadd_rn(c48, c12)), __fadd_rn(c56, c4))), A[60 * 32]);
  A[60 * 32] = c60;
  const float c61 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c4, c57), __fadd_rn(c8, c53), __fadd_rn(c12, c49)), min3f(__fadd_rn(c16, c45), __fadd_rn(c20, c41), __fadd_rn(c24, c37)), min3f(__fadd_rn(c28, c33), __fadd_rn(c32, c29), __fadd_rn(c36, c25))), min3f(__fadd_rn(c40, c21), __fadd_rn(c44, c17), __fadd_rn(c48, c13)), min3f(__fadd_rn(c52, c9), __fadd_rn(c56, c5), __fadd_rn(c60, c1)))), A[61 * 32]);
  A[61 * 32] = c61;
  const float c62 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c4, c58), __fadd_rn(c8, c54), __fadd_rn(c12, c50)), min3f(__fadd_rn(c16, c46), __fadd_rn(c20, c42), __fadd_rn(c24, c38)), min3f(__fadd_rn(c28, c34), __fadd_rn(c32, c30), __fadd_rn(c36, c26))), min3f(__fadd_rn(c40, c22), __fadd_rn(c44, c18), __fadd_rn(c48, c14)), min3f(__fadd_rn(c52, c10), __fadd_rn(c56, c6), __fadd_rn(c60, c2)))), A[62 * 32]);
  A[62 * 32] = c62;
  const float c63 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(min3f(__fadd_rn(c2, c61), __fadd_rn(c4, c59), __fadd_rn(c6, c57)), min3f(__fadd_rn(c8, c55), __fadd_rn(c10, c53), __fadd_rn(c12, c51)), min3f(__fadd_rn(c14, c49), __fadd_rn(c16, c47), __fadd_rn(c18, c45))), min3f(min3f(__fadd_rn(c20, c43), __fadd_rn(c22, c41), __fadd_rn(c24, c39)), min3f(__fadd_rn(c26, c37), __fadd_rn(c28, c35), __fadd_rn(c30, c33)), min3f(__fadd_rn(c32, c31), __fadd_rn(c34, c29), __fadd_rn(c36, c27))), min3f(min3f(__fadd_rn(c38, c25), __fadd_rn(c40, c23), __fadd_rn(c42, c21)), min3f(__fadd_rn(c44, c19), __fadd_rn(c46, c17), __fadd_rn(c48, c15)), min3f(__fadd_rn(c50, c13), __fadd_rn(c52, c11), __fadd_rn(c54, c9)))), min3f(__fadd_rn(c56, c7), __fadd_rn(c58, c5), __fadd_rn(c60, c3)), __fadd_rn(c62, c1))), A[63 * 32]);
  A[63 * 32] = c63;
  const float c64 = 0.0f;
  A[64 * 32] = 0.0f;
  const float c65 = __fadd_rn(fminf(kTlInf, __fadd_rn(c64, c1)), A[65 * 32]);
  A[65 * 32] = c65;
  const float c66 = __fadd_rn(fminf(kTlInf, __fadd_rn(c64, c2)), A[66 * 32]);
  A[66 * 32] = c66;
  const float c67 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c2, c65), __fadd_rn(c64, c3), __fadd_rn(c66, c1))), A[67 * 32]);
  A[67 * 32] = c67;
  const float c68 = __fadd_rn(fminf(kTlInf, __fadd_rn(c64, c4)), A[68 * 32]);
  A[68 * 32] = c68;
  const float c69 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c65), __fadd_rn(c64, c5), __fadd_rn(c68, c1))), A[69 * 32]);
  A[69 * 32] = c69;
  const float c70 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c4, c66), __fadd_rn(c64, c6), __fadd_rn(c68, c2))), A[70 * 32]);
  A[70 * 32] = c70;
  const float c71 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c69), __fadd_rn(c4, c67), __fadd_rn(c6, c65)), min3f(__fadd_rn(c64, c7), __fadd_rn(c66, c5), __fadd_rn(c68, c3)), __fadd_rn(c70, c1))), A[71 * 32]);
  A[71 * 32] = c71;
  const float c72 = __fadd_rn(fminf(kTlInf, __fadd_rn(c64, c8)), A[72 * 32]);
  A[72 * 32] = c72;
  const float c73 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c65), __fadd_rn(c64, c9), __fadd_rn(c72, c1))), A[73 * 32]);
  A[73 * 32] = c73;
  const float c74 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c66), __fadd_rn(c64, c10), __fadd_rn(c72, c2))), A[74 * 32]);
  A[74 * 32] = c74;
  const float c75 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c73), __fadd_rn(c8, c67), __fadd_rn(c10, c65)), min3f(__fadd_rn(c64, c11), __fadd_rn(c66, c9), __fadd_rn(c72, c3)), __fadd_rn(c74, c1))), A[75 * 32]);
  A[75 * 32] = c75;
  const float c76 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c8, c68), __fadd_rn(c64, c12), __fadd_rn(c72, c4))), A[76 * 32]);
  A[76 * 32] = c76;
  const float c77 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c73), __fadd_rn(c8, c69), __fadd_rn(c12, c65)), min3f(__fadd_rn(c64, c13), __fadd_rn(c68, c9), __fadd_rn(c72, c5)), __fadd_rn(c76, c1))), A[77 * 32]);
  A[77 * 32] = c77;
  const float c78 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c74), __fadd_rn(c8, c70), __fadd_rn(c12, c66)), min3f(__fadd_rn(c64, c14), __fadd_rn(c68, c10), __fadd_rn(c72, c6)), __fadd_rn(c76, c2))), A[78 * 32]);
  A[78 * 32] = c78;
  const float c79 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c77), __fadd_rn(c4, c75), __fadd_rn(c6, c73)), min3f(__fadd_rn(c8, c71), __fadd_rn(c10, c69), __fadd_rn(c12, c67)), min3f(__fadd_rn(c14, c65), __fadd_rn(c64, c15), __fadd_rn(c66, c13))), min3f(__fadd_rn(c68, c11), __fadd_rn(c70, c9), __fadd_rn(c72, c7)), min3f(__fadd_rn(c74, c5), __fadd_rn(c76, c3), __fadd_rn(c78, c1)))), A[79 * 32]);
  A[79 * 32] = c79;
  const float c80 = __fadd_rn(fminf(kTlInf, __fadd_rn(c64, c16)), A[80 * 32]);
  A[80 * 32] = c80;
  const float c81 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c16, c65), __fadd_rn(c64, c17), __fadd_rn(c80, c1))), A[81 * 32]);
  A[81 * 32] = c81;
  const float c82 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c16, c66), __fadd_rn(c64, c18), __fadd_rn(c80, c2))), A[82 * 32]);
  A[82 * 32] = c82;
  const float c83 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c81), __fadd_rn(c16, c67), __fadd_rn(c18, c65)), min3f(__fadd_rn(c64, c19), __fadd_rn(c66, c17), __fadd_rn(c80, c3)), __fadd_rn(c82, c1))), A[83 * 32]);
  A[83 * 32] = c83;
  const float c84 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c16, c68), __fadd_rn(c64, c20), __fadd_rn(c80, c4))), A[84 * 32]);
  A[84 * 32] = c84;
  const float c85 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c81), __fadd_rn(c16, c69), __fadd_rn(c20, c65)), min3f(__fadd_rn(c64, c21), __fadd_rn(c68, c17), __fadd_rn(c80, c5)), __fadd_rn(c84, c1))), A[85 * 32]);
  A[85 * 32] = c85;
  const float c86 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c82), __fadd_rn(c16, c70), __fadd_rn(c20, c66)), min3f(__fadd_rn(c64, c22), __fadd_rn(c68, c18), __fadd_rn(c80, c6)), __fadd_rn(c84, c2))), A[86 * 32]);
  A[86 * 32] = c86;
  const float c87 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c85), __fadd_rn(c4, c83), __fadd_rn(c6, c81)), min3f(__fadd_rn(c16, c71), __fadd_rn(c18, c69), __fadd_rn(c20, c67)), min3f(__fadd_rn(c22, c65), __fadd_rn(c64, c23), __fadd_rn(c66, c21))), min3f(__fadd_rn(c68, c19), __fadd_rn(c70, c17), __fadd_rn(c80, c7)), min3f(__fadd_rn(c82, c5), __fadd_rn(c84, c3), __fadd_rn(c86, c1)))), A[87 * 32]);
  A[87 * 32] = c87;
  const float c88 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c16, c72), __fadd_rn(c64, c24), __fadd_rn(c80, c8))), A[88 * 32]);
  A[88 * 32] = c88;
  const float c89 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c8, c81), __fadd_rn(c16, c73), __fadd_rn(c24, c65)), min3f(__fadd_rn(c64, c25), __fadd_rn(c72, c17), __fadd_rn(c80, c9)), __fadd_rn(c88, c1))), A[89 * 32]);
  A[89 * 32] = c89;
  const float c90 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c8, c82), __fadd_rn(c16, c74), __fadd_rn(c24, c66)), min3f(__fadd_rn(c64, c26), __fadd_rn(c72, c18), __fadd_rn(c80, c10)), __fadd_rn(c88, c2))), A[90 * 32]);
  A[90 * 32] = c90;
  const float c91 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c89), __fadd_rn(c8, c83), __fadd_rn(c10, c81)), min3f(__fadd_rn(c16, c75), __fadd_rn(c18, c73), __fadd_rn(c24, c67)), min3f(__fadd_rn(c26, c65), __fadd_rn(c64, c27), __fadd_rn(c66, c25))), min3f(__fadd_rn(c72, c19), __fadd_rn(c74, c17), __fadd_rn(c80, c11)), min3f(__fadd_rn(c82, c9), __fadd_rn(c88, c3), __fadd_rn(c90, c1)))), A[91 * 32]);
  A[91 * 32] = c91;
  const float c92 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c8, c84), __fadd_rn(c16, c76), __fadd_rn(c24, c68)), min3f(__fadd_rn(c64, c28), __fadd_rn(c72, c20), __fadd_rn(c80, c12)), __fadd_rn(c88, c4))), A[92 * 32]);
  A[92 * 32] = c92;
  const float c93 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c4, c89), __fadd_rn(c8, c85), __fadd_rn(c12, c81)), min3f(__fadd_rn(c16, c77), __fadd_rn(c20, c73), __fadd_rn(c24, c69)), min3f(__fadd_rn(c28, c65), __fadd_rn(c64, c29), __fadd_rn(c68, c25))), min3f(__fadd_rn(c72, c21), __fadd_rn(c76, c17), __fadd_rn(c80, c13)), min3f(__fadd_rn(c84, c9), __fadd_rn(c88, c5), __fadd_rn(c92, c1)))), A[93 * 32]);
  A[93 * 32] = c93;
  const float c94 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c4, c90), __fadd_rn(c8, c86), __fadd_rn(c12, c82)), min3f(__fadd_rn(c16, c78), __fadd_rn(c20, c74), __fadd_rn(c24, c70)), min3f(__fadd_rn(c28, c66), __fadd_rn(c64, c30), __fadd_rn(c68, c26))), min3f(__fadd_rn(c72, c22), __fadd_rn(c76, c18), __fadd_rn(c80, c14)), min3f(__fadd_rn(c84, c10), __fadd_rn(c88, c6), __fadd_rn(c92, c2)))), A[94 * 32]);
  A[94 * 32] = c94;
  const float c95 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(min3f(__fadd_rn(c2, c93), __fadd_rn(c4, c91), __fadd_rn(c6, c89)), min3f(__fadd_rn(c8, c87), __fadd_rn(c10, c85), __fadd_rn(c12, c83)), min3f(__fadd_rn(c14, c81), __fadd_rn(c16, c79), __fadd_rn(c18, c77))), min3f(min3f(__fadd_rn(c20, c75), __fadd_rn(c22, c73), __fadd_rn(c24, c71)), min3f(__fadd_rn(c26, c69), __fadd_rn(c28, c67), __fadd_rn(c30, c65)), min3f(__fadd_rn(c64, c31), __fadd_rn(c66, c29), __fadd_rn(c68, c27))), min3f(min3f(__fadd_rn(c70, c25), __fadd_rn(c72, c23), __fadd_rn(c74, c21)), min3f(__fadd_rn(c76, c19), __fadd_rn(c78, c17), __fadd_rn(c80, c15)), min3f(__fadd_rn(c82, c13), __fadd_rn(c84, c11), __fadd_rn(c86, c9)))), min3f(__fadd_rn(c88, c7), __fadd_rn(c90, c5), __fadd_rn(c92, c3)), __fadd_rn(c94, c1))), A[95 * 32]);
  A[95 * 32] = c95;
  const float c96 = __fadd_rn(fminf(kTlInf, __fadd_rn(c64, c32)), A[96 * 32]);
  A[96 * 32] = c96;
  const float c97 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c32, c65), __fadd_rn(c64, c33), __fadd_rn(c96, c1))), A[97 * 32]);
  A[97 * 32] = c97;
  const float c98 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c32, c66), __fadd_rn(c64, c34), __fadd_rn(c96, c2))), A[98 * 32]);
  A[98 * 32] = c98;
  const float c99 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c2, c97), __fadd_rn(c32, c67), __fadd_rn(c34, c65)), min3f(__fadd_rn(c64, c35), __fadd_rn(c66, c33), __fadd_rn(c96, c3)), __fadd_rn(c98, c1))), A[99 * 32]);
  A[99 * 32] = c99;
  const float c100 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c32, c68), __fadd_rn(c64, c36), __fadd_rn(c96, c4))), A[100 * 32]);
  A[100 * 32] = c100;
  const float c101 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c97), __fadd_rn(c32, c69), __fadd_rn(c36, c65)), min3f(__fadd_rn(c64, c37), __fadd_rn(c68, c33), __fadd_rn(c96, c5)), __fadd_rn(c100, c1))), A[101 * 32]);
  A[101 * 32] = c101;
  const float c102 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c4, c98), __fadd_rn(c32, c70), __fadd_rn(c36, c66)), min3f(__fadd_rn(c64, c38), __fadd_rn(c68, c34), __fadd_rn(c96, c6)), __fadd_rn(c100, c2))), A[102 * 32]);
  A[102 * 32] = c102;
  const float c103 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c101), __fadd_rn(c4, c99), __fadd_rn(c6, c97)), min3f(__fadd_rn(c32, c71), __fadd_rn(c34, c69), __fadd_rn(c36, c67)), min3f(__fadd_rn(c38, c65), __fadd_rn(c64, c39), __fadd_rn(c66, c37))), min3f(__fadd_rn(c68, c35), __fadd_rn(c70, c33), __fadd_rn(c96, c7)), min3f(__fadd_rn(c98, c5), __fadd_rn(c100, c3), __fadd_rn(c102, c1)))), A[103 * 32]);
  A[103 * 32] = c103;
  const float c104 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c32, c72), __fadd_rn(c64, c40), __fadd_rn(c96, c8))), A[104 * 32]);
  A[104 * 32] = c104;
  const float c105 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c8, c97), __fadd_rn(c32, c73), __fadd_rn(c40, c65)), min3f(__fadd_rn(c64, c41), __fadd_rn(c72, c33), __fadd_rn(c96, c9)), __fadd_rn(c104, c1))), A[105 * 32]);
  A[105 * 32] = c105;
  const float c106 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c8, c98), __fadd_rn(c32, c74), __fadd_rn(c40, c66)), min3f(__fadd_rn(c64, c42), __fadd_rn(c72, c34), __fadd_rn(c96, c10)), __fadd_rn(c104, c2))), A[106 * 32]);
  A[106 * 32] = c106;
  const float c107 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c105), __fadd_rn(c8, c99), __fadd_rn(c10, c97)), min3f(__fadd_rn(c32, c75), __fadd_rn(c34, c73), __fadd_rn(c40, c67)), min3f(__fadd_rn(c42, c65), __fadd_rn(c64, c43), __fadd_rn(c66, c41))), min3f(__fadd_rn(c72, c35), __fadd_rn(c74, c33), __fadd_rn(c96, c11)), min3f(__fadd_rn(c98, c9), __fadd_rn(c104, c3), __fadd_rn(c106, c1)))), A[107 * 32]);
  A[107 * 32] = c107;
  const float c108 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c8, c100), __fadd_rn(c32, c76), __fadd_rn(c40, c68)), min3f(__fadd_rn(c64, c44), __fadd_rn(c72, c36), __fadd_rn(c96, c12)), __fadd_rn(c104, c4))), A[108 * 32]);
  A[108 * 32] = c108;
  const float c109 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c4, c105), __fadd_rn(c8, c101), __fadd_rn(c12, c97)), min3f(__fadd_rn(c32, c77), __fadd_rn(c36, c73), __fadd_rn(c40, c69)), min3f(__fadd_rn(c44, c65), __fadd_rn(c64, c45), __fadd_rn(c68, c41))), min3f(__fadd_rn(c72, c37), __fadd_rn(c76, c33), __fadd_rn(c96, c13)), min3f(__fadd_rn(c100, c9), __fadd_rn(c104, c5), __fadd_rn(c108, c1)))), A[109 * 32]);
  A[109 * 32] = c109;
  const float c110 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c4, c106), __fadd_rn(c8, c102), __fadd_rn(c12, c98)), min3f(__fadd_rn(c32, c78), __fadd_rn(c36, c74), __fadd_rn(c40, c70)), min3f(__fadd_rn(c44, c66), __fadd_rn(c64, c46), __fadd_rn(c68, c42))), min3f(__fadd_rn(c72, c38), __fadd_rn(c76, c34), __fadd_rn(c96, c14)), min3f(__fadd_rn(c100, c10), __fadd_rn(c104, c6), __fadd_rn(c108, c2)))), A[110 * 32]);
  A[110 * 32] = c110;
  const float c111 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(min3f(__fadd_rn(c2, c109), __fadd_rn(c4, c107), __fadd_rn(c6, c105)), min3f(__fadd_rn(c8, c103), __fadd_rn(c10, c101), __fadd_rn(c12, c99)), min3f(__fadd_rn(c14, c97), __fadd_rn(c32, c79), __fadd_rn(c34, c77))), min3f(min3f(__fadd_rn(c36, c75), __fadd_rn(c38, c73), __fadd_rn(c40, c71)), min3f(__fadd_rn(c42, c69), __fadd_rn(c44, c67), __fadd_rn(c46, c65)), min3f(__fadd_rn(c64, c47), __fadd_rn(c66, c45), __fadd_rn(c68, c43))), min3f(min3f(__fadd_rn(c70, c41), __fadd_rn(c72, c39), __fadd_rn(c74, c37)), min3f(__fadd_rn(c76, c35), __fadd_rn(c78, c33), __fadd_rn(c96, c15)), min3f(__fadd_rn(c98, c13), __fadd_rn(c100, c11), __fadd_rn(c102, c9)))), min3f(__fadd_rn(c104, c7), __fadd_rn(c106, c5), __fadd_rn(c108, c3)), __fadd_rn(c110, c1))), A[111 * 32]);
  A[111 * 32] = c111;
  const float c112 = __fadd_rn(fminf(kTlInf, min3f(__fadd_rn(c32, c80), __fadd_rn(c64, c48), __fadd_rn(c96, c16))), A[112 * 32]);
  A[112 * 32] = c112;
  const float c113 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c16, c97), __fadd_rn(c32, c81), __fadd_rn(c48, c65)), min3f(__fadd_rn(c64, c49), __fadd_rn(c80, c33), __fadd_rn(c96, c17)), __fadd_rn(c112, c1))), A[113 * 32]);
  A[113 * 32] = c113;
  const float c114 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c16, c98), __fadd_rn(c32, c82), __fadd_rn(c48, c66)), min3f(__fadd_rn(c64, c50), __fadd_rn(c80, c34), __fadd_rn(c96, c18)), __fadd_rn(c112, c2))), A[114 * 32]);
  A[114 * 32] = c114;
  const float c115 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c2, c113), __fadd_rn(c16, c99), __fadd_rn(c18, c97)), min3f(__fadd_rn(c32, c83), __fadd_rn(c34, c81), __fadd_rn(c48, c67)), min3f(__fadd_rn(c50, c65), __fadd_rn(c64, c51), __fadd_rn(c66, c49))), min3f(__fadd_rn(c80, c35), __fadd_rn(c82, c33), __fadd_rn(c96, c19)), min3f(__fadd_rn(c98, c17), __fadd_rn(c112, c3), __fadd_rn(c114, c1)))), A[115 * 32]);
  A[115 * 32] = c115;
  const float c116 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c16, c100), __fadd_rn(c32, c84), __fadd_rn(c48, c68)), min3f(__fadd_rn(c64, c52), __fadd_rn(c80, c36), __fadd_rn(c96, c20)), __fadd_rn(c112, c4))), A[116 * 32]);
  A[116 * 32] = c116;
  const float c117 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c4, c113), __fadd_rn(c16, c101), __fadd_rn(c20, c97)), min3f(__fadd_rn(c32, c85), __fadd_rn(c36, c81), __fadd_rn(c48, c69)), min3f(__fadd_rn(c52, c65), __fadd_rn(c64, c53), __fadd_rn(c68, c49))), min3f(__fadd_rn(c80, c37), __fadd_rn(c84, c33), __fadd_rn(c96, c21)), min3f(__fadd_rn(c100, c17), __fadd_rn(c112, c5), __fadd_rn(c116, c1)))), A[117 * 32]);
  A[117 * 32] = c117;
  const float c118 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c4, c114), __fadd_rn(c16, c102), __fadd_rn(c20, c98)), min3f(__fadd_rn(c32, c86), __fadd_rn(c36, c82), __fadd_rn(c48, c70)), min3f(__fadd_rn(c52, c66), __fadd_rn(c64, c54), __fadd_rn(c68, c50))), min3f(__fadd_rn(c80, c38), __fadd_rn(c84, c34), __fadd_rn(c96, c22)), min3f(__fadd_rn(c100, c18), __fadd_rn(c112, c6), __fadd_rn(c116, c2)))), A[118 * 32]);
  A[118 * 32] = c118;
  const float c119 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(min3f(__fadd_rn(c2, c117), __fadd_rn(c4, c115), __fadd_rn(c6, c113)), min3f(__fadd_rn(c16, c103), __fadd_rn(c18, c101), __fadd_rn(c20, c99)), min3f(__fadd_rn(c22, c97), __fadd_rn(c32, c87), __fadd_rn(c34, c85))), min3f(min3f(__fadd_rn(c36, c83), __fadd_rn(c38, c81), __fadd_rn(c48, c71)), min3f(__fadd_rn(c50, c69), __fadd_rn(c52, c67), __fadd_rn(c54, c65)), min3f(__fadd_rn(c64, c55), __fadd_rn(c66, c53), __fadd_rn(c68, c51))), min3f(min3f(__fadd_rn(c70, c49), __fadd_rn(c80, c39), __fadd_rn(c82, c37)), min3f(__fadd_rn(c84, c35), __fadd_rn(c86, c33), __fadd_rn(c96, c23)), min3f(__fadd_rn(c98, c21), __fadd_rn(c100, c19), __fadd_rn(c102, c17)))), min3f(__fadd_rn(c112, c7), __fadd_rn(c114, c5), __fadd_rn(c116, c3)), __fadd_rn(c118, c1))), A[119 * 32]);
  A[119 * 32] = c119;
  const float c120 = __fadd_rn(fminf(kTlInf, min3f(min3f(__fadd_rn(c16, c104), __fadd_rn(c32, c88), __fadd_rn(c48, c72)), min3f(__fadd_rn(c64, c56), __fadd_rn(c80, c40), __fadd_rn(c96, c24)), __fadd_rn(c112, c8))), A[120 * 32]);
  A[120 * 32] = c120;
  const float c121 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c8, c113), __fadd_rn(c16, c105), __fadd_rn(c24, c97)), min3f(__fadd_rn(c32, c89), __fadd_rn(c40, c81), __fadd_rn(c48, c73)), min3f(__fadd_rn(c56, c65), __fadd_rn(c64, c57), __fadd_rn(c72, c49))), min3f(__fadd_rn(c80, c41), __fadd_rn(c88, c33), __fadd_rn(c96, c25)), min3f(__fadd_rn(c104, c17), __fadd_rn(c112, c9), __fadd_rn(c120, c1)))), A[121 * 32]);
  A[121 * 32] = c121;
  const float c122 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c8, c114), __fadd_rn(c16, c106), __fadd_rn(c24, c98)), min3f(__fadd_rn(c32, c90), __fadd_rn(c40, c82), __fadd_rn(c48, c74)), min3f(__fadd_rn(c56, c66), __fadd_rn(c64, c58), __fadd_rn(c72, c50))), min3f(__fadd_rn(c80, c42), __fadd_rn(c88, c34), __fadd_rn(c96, c26)), min3f(__fadd_rn(c104, c18), __fadd_rn(c112, c10), __fadd_rn(c120, c2)))), A[122 * 32]);
  A[122 * 32] = c122;
  const float c123 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(min3f(__fadd_rn(c2, c121), __fadd_rn(c8, c115), __fadd_rn(c10, c113)), min3f(__fadd_rn(c16, c107), __fadd_rn(c18, c105), __fadd_rn(c24, c99)), min3f(__fadd_rn(c26, c97), __fadd_rn(c32, c91), __fadd_rn(c34, c89))), min3f(min3f(__fadd_rn(c40, c83), __fadd_rn(c42, c81), __fadd_rn(c48, c75)), min3f(__fadd_rn(c50, c73), __fadd_rn(c56, c67), __fadd_rn(c58, c65)), min3f(__fadd_rn(c64, c59), __fadd_rn(c66, c57), __fadd_rn(c72, c51))), min3f(min3f(__fadd_rn(c74, c49), __fadd_rn(c80, c43), __fadd_rn(c82, c41)), min3f(__fadd_rn(c88, c35), __fadd_rn(c90, c33), __fadd_rn(c96, c27)), min3f(__fadd_rn(c98, c25), __fadd_rn(c104, c19), __fadd_rn(c106, c17)))), min3f(__fadd_rn(c112, c11), __fadd_rn(c114, c9), __fadd_rn(c120, c3)), __fadd_rn(c122, c1))), A[123 * 32]);
  A[123 * 32] = c123;
  const float c124 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(__fadd_rn(c8, c116), __fadd_rn(c16, c108), __fadd_rn(c24, c100)), min3f(__fadd_rn(c32, c92), __fadd_rn(c40, c84), __fadd_rn(c48, c76)), min3f(__fadd_rn(c56, c68), __fadd_rn(c64, c60), __fadd_rn(c72, c52))), min3f(__fadd_rn(c80, c44), __fadd_rn(c88, c36), __fadd_rn(c96, c28)), min3f(__fadd_rn(c104, c20), __fadd_rn(c112, c12), __fadd_rn(c120, c4)))), A[124 * 32]);
  A[124 * 32] = c124;
  const float c125 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(min3f(__fadd_rn(c4, c121), __fadd_rn(c8, c117), __fadd_rn(c12, c113)), min3f(__fadd_rn(c16, c109), __fadd_rn(c20, c105), __fadd_rn(c24, c101)), min3f(__fadd_rn(c28, c97), __fadd_rn(c32, c93), __fadd_rn(c36, c89))), min3f(min3f(__fadd_rn(c40, c85), __fadd_rn(c44, c81), __fadd_rn(c48, c77)), min3f(__fadd_rn(c52, c73), __fadd_rn(c56, c69), __fadd_rn(c60, c65)), min3f(__fadd_rn(c64, c61), __fadd_rn(c68, c57), __fadd_rn(c72, c53))), min3f(min3f(__fadd_rn(c76, c49), __fadd_rn(c80, c45), __fadd_rn(c84, c41)), min3f(__fadd_rn(c88, c37), __fadd_rn(c92, c33), __fadd_rn(c96, c29)), min3f(__fadd_rn(c100, c25), __fadd_rn(c104, c21), __fadd_rn(c108, c17)))), min3f(__fadd_rn(c112, c13), __fadd_rn(c116, c9), __fadd_rn(c120, c5)), __fadd_rn(c124, c1))), A[125 * 32]);
  A[125 * 32] = c125;
  const float c126 = __fadd_rn(fminf(kTlInf, min3f(min3f(min3f(min3f(__fadd_rn(c4, c122), __fadd_rn(c8, c118), __fadd_rn(c12, c114)), min3f(__fadd_rn(c16, c110), __fadd_rn(c20, c106), __fadd_rn(c24, c102)), min3f(__fadd_rn(c28, c98), __fadd_rn(c32, c94), __fadd_rn(c36, c90))), min3f(min3f(__fadd_rn(c40, c86), __fadd_rn(c44, c82), __fadd_rn(c48, c78)), min3f(__fadd_rn(c52, c74), __fadd_rn(c56, c70), __fadd_rn(c60, c66)), min3f(__fadd_rn(c64, c62), __fadd_rn(c68, c58), __fadd_rn(c72, c54))), min3f(min3f(__fadd_rn(c76, c50), __fadd_rn(c80, c46), __fadd_rn(c84, c42)), min3f(__fadd_rn(c88, c38), __fadd_rn(c92, c34), __fadd_rn(c96, c30)), min3f(__fadd_rn(c100, c26), __fadd_rn(c104, c22), __fadd_rn(c108, c18)))), min3f(__fadd_rn(c112, c14), __fadd_rn(c116, c10), __fadd_rn(c120, c6)), __fadd_rn(c124, c2))), A[126 * 32]);
  A[126 * 32] = c126;
  float b = kTlInf, b2 = kTlInf, v, v2;
  uint32_t bp = 0u, bp2 = 0u;
  v = __fadd_rn(c2, c125);
  if (v < b) { b = v; bp = 2u; }
  v2 = __fadd_rn(c66, c61);
  if (v2 < b2) { b2 = v2; bp2 = 66u; }
  v = __fadd_rn(c4, c123);
  if (v < b) { b = v; bp = 4u; }
  v2 = __fadd_rn(c68, c59);
  if (v2 < b2) { b2 = v2; bp2 = 68u; }
  v = __fadd_rn(c6, c121);
  if (v < b) { b = v; bp = 6u; }
  v2 = __fadd_rn(c70, c57);
  if (v2 < b2) { b2 = v2; bp2 = 70u; }
  v = __fadd_rn(c8, c119);
  if (v < b) { b = v; bp = 8u; }
  v2 = __fadd_rn(c72, c55);
  if (v2 < b2) { b2 = v2; bp2 = 72u; }
  v = __fadd_rn(c10, c117);
  if (v < b) { b = v; bp = 10u; }
  v2 = __fadd_rn(c74, c53);
  if (v2 < b2) { b2 = v2; bp2 = 74u; }
  v = __fadd_rn(c12, c115);
  if (v < b) { b = v; bp = 12u; }
  v2 = __fadd_rn(c76, c51);
  if (v2 < b2) { b2 = v2; bp2 = 76u; }
  v = __fadd_rn(c14, c113);
  if (v < b) { b = v; bp = 14u; }
  v2 = __fadd_rn(c78, c49);
  if (v2 < b2) { b2 = v2; bp2 = 78u; }
  v = __fadd_rn(c16, c111);
  if (v < b) { b = v; bp = 16u; }
  v2 = __fadd_rn(c80, c47);
  if (v2 < b2) { b2 = v2; bp2 = 80u; }
  v = __fadd_rn(c18, c109);
  if (v < b) { b = v; bp = 18u; }
  v2 = __fadd_rn(c82, c45);
  if (v2 < b2) { b2 = v2; bp2 = 82u; }
  v = __fadd_rn(c20, c107);
  if (v < b) { b = v; bp = 20u; }
  v2 = __fadd_rn(c84, c43);
  if (v2 < b2) { b2 = v2; bp2 = 84u; }
  v = __fadd_rn(c22, c105);
  if (v < b) { b = v; bp = 22u; }
  v2 = __fadd_rn(c86, c41);
  if (v2 < b2) { b2 = v2; bp2 = 86u; }
  v = __fadd_rn(c24, c103);
  if (v < b) { b = v; bp = 24u; }
  v2 = __fadd_rn(c88, c39);
  if (v2 < b2) { b2 = v2; bp2 = 88u; }
  v = __fadd_rn(c26, c101);
  if (v < b) { b = v; bp = 26u; }
  v2 = __fadd_rn(c90, c37);
  if (v2 < b2) { b2 = v2; bp2 = 90u; }
  v = __fadd_rn(c28, c99);
  if (v < b) { b = v; bp = 28u; }
  v2 = __fadd_rn(c92, c35);
  if (v2 < b2) { b2 = v2; bp2 = 92u; }
  v = __fadd_rn(c30, c97);
  if (v < b) { b = v; bp = 30u; }
  v2 = __fadd_rn(c94, c33);
  if (v2 < b2) { b2 = v2; bp2 = 94u; }
  v = __fadd_rn(c32, c95);
  if (v < b) { b = v; bp = 32u; }
  v2 = __fadd_rn(c96, c31);
  if (v2 < b2) { b2 = v2; bp2 = 96u; }
  v = __fadd_rn(c34, c93);
  if (v < b) { b = v; bp = 34u; }
  v2 = __fadd_rn(c98, c29);
  if (v2 < b2) { b2 = v2; bp2 = 98u; }
  v = __fadd_rn(c36, c91);
  if (v < b) { b = v; bp = 36u; }
  v2 = __fadd_rn(c100, c27);
  if (v2 < b2) { b2 = v2; bp2 = 100u; }
  v = __fadd_rn(c38, c89);
  if (v < b) { b = v; bp = 38u; }
  v2 = __fadd_rn(c102, c25);
  if (v2 < b2) { b2 = v2; bp2 = 102u; }
  v = __fadd_rn(c40, c87);
  if (v < b) { b = v; bp = 40u; }
  v2 = __fadd_rn(c104, c23);
  if (v2 < b2) { b2 = v2; bp2 = 104u; }
  v = __fadd_rn(c42, c85);
  if (v < b) { b = v; bp = 42u; }
  v2 = __fadd_rn(c106, c21);
  if (v2 < b2) { b2 = v2; bp2 = 106u; }
  v = __fadd_rn(c44, c83);
  if (v < b) { b = v; bp = 44u; }
  v2 = __fadd_rn(c108, c19);
  if (v2 < b2) { b2 = v2; bp2 = 108u; }
  v = __fadd_rn(c46, c81);
  if (v < b) { b = v; bp = 46u; }
  v2 = __fadd_rn(c110, c17);
  if (v2 < b2) { b2 = v2; bp2 = 110u; }
  v = __fadd_rn(c48, c79);
  if (v < b) { b = v; bp = 48u; }
  v2 = __fadd_rn(c112, c15);
  if (v2 < b2) { b2 = v2; bp2 = 112u; }
  v = __fadd_rn(c50, c77);
  if (v < b) { b = v; bp = 50u; }
  v2 = __fadd_rn(c114, c13);
  if (v2 < b2) { b2 = v2; bp2 = 114u; }
  v = __fadd_rn(c52, c75);
  if (v < b) { b = v; bp = 52u; }
  v2 = __fadd_rn(c116, c11);
  if (v2 < b2) { b2 = v2; bp2 = 116u; }
  v = __fadd_rn(c54, c73);
  if (v < b) { b = v; bp = 54u; }
  v2 = __fadd_rn(c118, c9);
  if (v2 < b2) { b2 = v2; bp2 = 118u; }
  v = __fadd_rn(c56, c71);
  if (v < b) { b = v; bp = 56u; }
  v2 = __fadd_rn(c120, c7);
  if (v2 < b2) { b2 = v2; bp2 = 120u; }
  v = __fadd_rn(c58, c69);
  if (v < b) { b = v; bp = 58u; }
  v2 = __fadd_rn(c122, c5);
  if (v2 < b2) { b2 = v2; bp2 = 122u; }
  v = __fadd_rn(c60, c67);
  if (v < b) { b = v; bp = 60u; }
  v2 = __fadd_rn(c124, c3);
  if (v2 < b2) { b2 = v2; bp2 = 124u; }
  v = __fadd_rn(c62, c65);
  if (v < b) { b = v; bp = 62u; }
  v2 = __fadd_rn(c126, c1);
  if (v2 < b2) { b2 = v2; bp2 = 126u; }
  v = __fadd_rn(c64, c63);
  if (v < b) { b = v; bp = 64u; }
  return b2 < b ? bp2 : bp;
}

}  // namespace bvhgb
