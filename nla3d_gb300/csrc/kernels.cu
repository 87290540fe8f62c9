// Assembly kernels for sm_103a: SOLID81 (FP64 and mixed), its Jacobian
// precompute, TETRA0 / QUADTH, the fixed-order CSR gather and the rigid-body
// MPC rows.
//
// SOLID81 algebra (reference: SOLID81.cpp:29-82, 85-115):
//   B = 2 (B_L + Omega B_NL) is 2 * Bh, where for node a, displacement
//   component i and Voigt row (jk):  Bh[(jk)][i] = F_ij G_ak + F_ik G_aj
//   (j != k), F_ij G_aj (j == k);  F = I + O, G_a = dN_a/dX.
//   Kuu(a,i; b,k) += w * (Bh_a^T Dd' Bh_b)[i][k] + w * delta_ik G_a . S G_b
//       with Dd' = 2 * Dd (the reference halves Dd, materials_hyperelastic.cpp:124,
//       and scales B^T Dd B by w/2 with B = 2 Bh);
//   Fu_a   += -w * (F S G_a)              ( = -w/2 B^T S,  SOLID81.cpp:73 )
//   Kup_a  +=  w * (cof(F) G_a)           ( = w/2 B^T J C^-1, since J F C^-1 = cof F )
//   Fp     += -(J - 1 - p/k) w ;  Kpp += -w / k
// Writing Bh out, both Kuu terms are one contraction with a symmetric 9x9
// tensor per Gauss point,
//   Kuu(a,i; b,k) += sum_{L,N} G_aL A[iL][kN] G_bN,
//   A[iL][kN] = sum_{J,M} F_iJ wDd'[(JL)][(MN)] F_kM + delta_ik w S_LN.
// The mixed kernel forms A and h_a[ik] = A^T G_a per node (i <= k: A is
// symmetric) and 3 FMA per Kuu entry and Gauss point.  The FP64 kernel writes
// the same contraction in the element's reference coordinates and sums over
// the Gauss points first (see solid81_fp64_kernel).  These are the
// reference's products with the structural zeros of B, B_NL and Omega removed
// and the sums regrouped; they agree with the reference to rounding (the
// tests bound the difference at 1e-12 relative).
#include <atomic>
#include <cmath>
#include <cstdio>
#include <mutex>
#include <type_traits>

#include "kernels.cuh"

namespace nla3d_gpu {

namespace {

constexpr int kWarpsPerBlock = 4;  // default launch shape
constexpr int kEPW = 4;                              // elements per warp
constexpr int kKuuPerElem = 300;
constexpr int kOwned = (kEPW * kKuuPerElem + 31) / 32;  // Kuu entries per lane (38)
constexpr double kGaussA = 0.5773502691896258;        // isoparametric.h:127

// Position in assemble3 order (SOLID81.h:62-74) of the Kuu entry that
// D[(i,k), a, b] = K(a,i; b,k) (i <= k) stands for, at [(a * 6 +
// hblock(i,k)) * 8 + b]: K(a,i; b,k) when a <= b, K(b,k; a,i) when a > b;
// 0xFFFF where a > b and i == k (the same entry as D[(i,i), b, a]).
constexpr int kDpos = 8 * 6 * 8;
constexpr size_t kDposBytes = kDpos * sizeof(uint16_t);
__constant__ uint16_t c_dpos[kDpos];

// the (i, k) blocks of h that are formed: i <= k, packed (6 blocks)
__host__ __device__ constexpr int hblock(int i, int k) {  // i <= k
  return 3 * i - (i * (i - 1)) / 2 + (k - i);
}

// Mixed kernel: -w F S (float pairs) and w cof F (FP64: the pressure
// coupling K_up keeps FP64) are only needed between phase 1 and the residual
// / coupling pass that precedes the Gauss point loop, so they share their
// bytes with the staging buffer of the Kuu write after that loop.  Per
// (element q, Gauss point g) they sit at slot g * 4 + q, so the pass's
// broadcast reads of one Gauss point hit four consecutive words.  h stays in
// registers (each lane keeps its own node's).
struct MixedSmem {
  float A[45][32];
  union {
    float stage[4 * 300];   // the quad's Kuu entries in assemble3 order, for the write
    struct {
      float2 wP[9][32];     // -w F S, float pairs
      double wCof[9][32];   // w cof F, FP64
      float wCofF[9][32];   // the same from the float F (for G's low part)
    };
  };
  float G[3][32];
};

__device__ __forceinline__ int sym6(int r, int s) {  // packed upper index, r <= s
  return 6 * r - ((r - 1) * r) / 2 + (s - r);
}

__device__ __forceinline__ int sym6u(int r, int s) { return r <= s ? sym6(r, s) : sym6(s, r); }

__device__ __forceinline__ int sym9(int p, int c) {  // packed upper 9x9, any order
  return p <= c ? 9 * p - ((p - 1) * p) / 2 + (c - p) : 9 * c - ((c - 1) * c) / 2 + (p - c);
}

// Voigt index of the symmetric pair (J, L): xx xy xz yy yz zz
__device__ __forceinline__ int voigt(int J, int L) {
  return J == L ? (J == 0 ? 0 : (J == 1 ? 3 : 5)) : (J + L == 1 ? 1 : (J + L == 2 ? 2 : 4));
}

__device__ __forceinline__ void flag_element(ElementStatus* st, uint32_t el1) {
  atomicAdd(&st->count, 1u);
  atomicMax(&st->first_inv, ~el1);
}

// w * 2 Dd, packed upper Voigt, from the coefficient form
//   A (x) P + B (x) Q + Ci (x) R + sIIt * IIt + sI * (I (x) I - II)
// with P = wk11 A - wk1 Ci, Q = -wk2 Ci, R = -wk1 A - wk2 B + wc0 Ci
// (materials_hyperelastic.cpp:64-129 with the reference's /2 taken out).
template <typename TT>
__device__ __forceinline__ void tangent_from_coefficients(const TT At[6], const TT Bt[6],
                                                          const TT Ct[6], TT wk11, TT wk1,
                                                          TT wk2, TT wc0, TT sIIt, TT sI,
                                                          TT wD[21]) {
  TT P[6], Q[6], R[6];
#pragma unroll
  for (int i = 0; i < 6; i++) {
    P[i] = wk11 * At[i] - wk1 * Ct[i];
    Q[i] = -wk2 * Ct[i];
    R[i] = -wk1 * At[i] - wk2 * Bt[i] + wc0 * Ct[i];
  }
  // IIt (materials_hyperelastic.cpp:97-108): -sym(Ci (x) Ci), packed upper
  const TT c_xx = Ct[0], c_xy = Ct[1], c_xz = Ct[2], c_yy = Ct[3], c_yz = Ct[4], c_zz = Ct[5];
  const TT h = (TT)0.5;
  const TT IIt[21] = {
      -c_xx * c_xx, -c_xx * c_xy, -c_xx * c_xz, -c_xy * c_xy, -c_xy * c_xz, -c_xz * c_xz,
      -h * (c_xx * c_yy + c_xy * c_xy), -h * (c_xx * c_yz + c_xz * c_xy), -c_xy * c_yy,
      -h * (c_xy * c_yz + c_xz * c_yy), -c_xz * c_yz,
      -h * (c_xx * c_zz + c_xz * c_xz), -c_xy * c_yz, -h * (c_xy * c_zz + c_xz * c_yz),
      -c_xz * c_zz,
      -c_yy * c_yy, -c_yy * c_yz, -c_yz * c_yz,
      -h * (c_yy * c_zz + c_yz * c_yz), -c_yz * c_zz,
      -c_zz * c_zz};
  // I (x) I - II, packed upper: +1 at (0,3),(0,5),(3,5); -1/2 at (1,1),(2,2),(4,4)
  int idx = 0;
#pragma unroll
  for (int r = 0; r < 6; r++)
#pragma unroll
    for (int s = r; s < 6; s++, idx++) {
      TT v = At[r] * P[s] + Bt[r] * Q[s] + Ct[r] * R[s] + sIIt * IIt[idx];
      const bool plus = (r == 0 && (s == 3 || s == 5)) || (r == 3 && s == 5);
      const bool minus = (r == s) && (r == 1 || r == 2 || r == 4);
      if (plus) v += sI;
      if (minus) v -= h * sI;
      wD[idx] = v;
    }
}

// ---------------------------------------------------------------------------
// Float-pair ("double-word") arithmetic for the mixed path's residual.
//
// On this part the FP64 pipe runs at 1/64 of the FP32 rate, so the mixed
// kernel computes the residual chain (displacement gradient, C, the
// material's S and J, -w F S G_a, the pressure terms) with pairs of floats
// x = h + l, |l| <= ulp(h) / 2, instead of doubles.  The building blocks are
// the error-free transformations TwoSum (Knuth) and TwoProd by FMA, and the
// compensated dot product Dot2 (Ogita, Rump, Oishi, "Accurate sum and dot
// product", SIAM J. Sci. Comput. 26, 2005); the pair operations follow the
// double-word algorithms analysed by Joldes, Muller and Popescu ("Tight and
// rigorous error bounds for basic building blocks of double-word
// arithmetic", ACM TOMS 44, 2017).  Each operation's error is a few units of
// 2^-48 relative to its operands, so the residual agrees with the FP64 path
// to ~1e-14 relative (the tests bound it at 1e-12).  The float exponent range
// applies: the mixed path needs |values| well inside 1e-30 .. 1e30.
// The intrinsics (__fadd_rn, __fmul_rn, __fmaf_rn) keep the compiler from
// contracting the transformations' separate roundings into FMAs.
struct dw {
  float h, l;
};

__device__ __forceinline__ dw two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return {s, e};
}

__device__ __forceinline__ dw fast_two_sum(float a, float b) {  // |a| >= |b| (or a == 0)
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}

__device__ __forceinline__ dw two_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return {p, __fmaf_rn(a, b, -p)};
}

__device__ __forceinline__ dw dw_neg(dw x) { return {-x.h, -x.l}; }
__device__ __forceinline__ dw dw_scale2(dw x, float p2) {  // p2 a power of two: exact
  return {x.h * p2, x.l * p2};
}

// x + y with error ~2^-47 (|x| + |y|)
__device__ __forceinline__ dw dw_add(dw x, dw y) {
  const dw s = two_sum(x.h, y.h);
  return fast_two_sum(s.h, __fadd_rn(s.l, __fadd_rn(x.l, y.l)));
}

__device__ __forceinline__ dw dw_addf(dw x, float y) {
  const dw s = two_sum(x.h, y);
  return fast_two_sum(s.h, __fadd_rn(s.l, x.l));
}

__device__ __forceinline__ dw dw_mul(dw x, dw y) {
  const dw p = two_prod(x.h, y.h);
  return fast_two_sum(p.h, __fmaf_rn(x.h, y.l, __fmaf_rn(x.l, y.h, p.l)));
}

__device__ __forceinline__ dw dw_mulf(dw x, float y) {
  const dw p = two_prod(x.h, y);
  return fast_two_sum(p.h, __fmaf_rn(x.l, y, p.l));
}

// Dot2 accumulator: value s + c, c collects the rounding errors unnormalised
struct dacc {
  float s, c;
};

__device__ __forceinline__ void acc_prod(dacc& a, dw x, dw y) {
  const dw p = two_prod(x.h, y.h);
  const float e = __fmaf_rn(x.h, y.l, __fmaf_rn(x.l, y.h, p.l));
  const dw t = two_sum(a.s, p.h);
  a.s = t.h;
  a.c = __fadd_rn(a.c, __fadd_rn(t.l, e));
}

__device__ __forceinline__ void acc_add(dacc& a, dw x) {
  const dw t = two_sum(a.s, x.h);
  a.s = t.h;
  a.c = __fadd_rn(a.c, __fadd_rn(t.l, x.l));
}

__device__ __forceinline__ dw acc_val(dacc a) { return two_sum(a.s, a.c); }

__device__ __forceinline__ dw dw_of(float2 v) { return {v.x, v.y}; }

// float -> double, exact, with integer operations only: on this part the
// conversion instruction runs on the FP64 pipe, at its 1/64 rate, while a
// normal float widens by re-biasing the exponent (127 -> 1023) and shifting
// the mantissa on the integer pipe.  A subnormal is scaled by 2^64 first (an
// exact FP32 product); infinities and NaNs take the exponent 2047.  A
// conversion instruction kept for these values is issued for every value (the
// compiler selects instead of branching): 700 of the mixed kernel's 1,840
// FP64-pipe instructions per element, and 1.09 ms at 216,000 elements for
// 0.93 ms with integers alone.
__device__ __forceinline__ double f2d(float f) {
  const uint32_t sign = __float_as_uint(f) & 0x80000000u;
  const uint32_t mag = __float_as_uint(f) & 0x7FFFFFFFu;
  const bool tiny = mag < 0x00800000u;
  const uint32_t m = tiny ? __float_as_uint(__uint_as_float(mag) * 18446744073709551616.0f) : mag;
  const uint32_t bias = mag >= 0x7F800000u ? 1792u : tiny ? 832u : 896u;
  const uint32_t hi = mag ? (m >> 3) + (bias << 20) : 0u;
  return __hiloint2double((int)(sign | hi), (int)(m << 29));
}

// The same with the rare values behind a real branch (the empty asm keeps the
// compiler from selecting): five integer operations for a normal float, and
// the tangent's FP32 sums around it stay in the blocks they were in, so that
// they round as they did.
__device__ __forceinline__ double f2d_branch(float f) {
  const uint32_t b = __float_as_uint(f);
  const uint32_t mag = b & 0x7FFFFFFFu;
  const uint32_t e = b & 0x7F800000u;
  const uint32_t sign = b & 0x80000000u;
  if (mag != 0u && (e == 0u || e == 0x7F800000u)) {
    double d = f2d(f);
    asm volatile("" : "+d"(d));
    return d;
  }
  const uint32_t hi = mag ? (sign | ((mag >> 3) + (896u << 20))) : sign;
  const uint32_t lo = mag ? (b << 29) : 0u;
  return __hiloint2double((int)hi, (int)lo);
}

__device__ __forceinline__ dw dw_from_double(double v) {
  const float h = __double2float_rn(v);
  return {h, __double2float_rn(v - f2d(h))};
}

__device__ __forceinline__ double dw_to_double(dw x) { return f2d_branch(x.h) + f2d_branch(x.l); }

// sqrt(d): the float root refined by one Newton step on the pair
__device__ __forceinline__ dw dw_sqrt(dw d) {
  const float y = __fsqrt_rn(d.h);
  const dw yy = two_prod(y, y);
  const float r = __fadd_rn(__fsub_rn(__fsub_rn(d.h, yy.h), yy.l), d.l);  // d - y^2
  return fast_two_sum(y, __fdiv_rn(r, 2.0f * y));
}

// 1 / d: the float reciprocal refined by one Newton step
__device__ __forceinline__ dw dw_rcp(dw d) {
  const float y = __frcp_rn(d.h);
  const dw p = two_prod(d.h, y);
  const float r = __fsub_rn(__fsub_rn(1.0f, p.h), __fmaf_rn(d.l, y, p.l));  // 1 - d y
  return fast_two_sum(y, __fmul_rn(y, r));
}

// x^(-1/3): the float estimate refined by Newton steps on f(x) = x^-3 - J,
//   x' = x + x (1 - J x^3) / 3,   relative error e -> 2 e^2,
// two steps, since one leaves 2 (2^-23)^2 ~ 3e-14 from a 1-ulp estimate.
__device__ __forceinline__ dw dw_rcbrt(dw J) {
  const float x0 = rcbrtf(J.h);
  const dw t0 = dw_mul(J, dw_mulf(two_prod(x0, x0), x0));
  const float u0 = __fsub_rn(__fsub_rn(1.0f, t0.h), t0.l);  // 1 - J x^3 (t.h ~ 1: exact)
  const dw x1 = fast_two_sum(x0, __fmul_rn(x0, __fmul_rn(u0, 1.0f / 3.0f)));
  const dw t1 = dw_mul(J, dw_mul(dw_mul(x1, x1), x1));
  const float u1 = __fsub_rn(__fsub_rn(1.0f, t1.h), t1.l);
  return dw_add(x1, dw_mulf(x1, __fmul_rn(u1, 1.0f / 3.0f)));
}

// constants as pairs (the low parts folded at compile time)
#define NLA3D_DW_CONST(name, value) \
  constexpr float name##_h = (float)(value); \
  constexpr float name##_l = (float)((value) - (double)name##_h);
NLA3D_DW_CONST(kThird, 1.0 / 3.0)
NLA3D_DW_CONST(kTwoThirds, 2.0 / 3.0)
NLA3D_DW_CONST(kFourThirds, 4.0 / 3.0)
NLA3D_DW_CONST(kEightThirds, 8.0 / 3.0)
#undef NLA3D_DW_CONST

// a b - c d
__device__ __forceinline__ dw dw_diff_prod(dw a, dw b, dw c, dw d) {
  dacc t{0.0f, 0.0f};
  acc_prod(t, a, b);
  acc_prod(t, dw_neg(c), d);
  return acc_val(t);
}

// Material response at one Gauss point (materials_hyperelastic.cpp:30-129,
// 135-204) from C (Voigt), p_state (for S) and p_cur (for the tangent): the state
// (S, J) in pairs, the tangent coefficients rounded to float.
__device__ __forceinline__ void material_mixed(int mat_id, const float2* mcd, const dw C[6],
                                               dw p_state, dw p_cur, dw w, dw S[6], dw& Jout,
                                               float wD[21]) {
  const dw I1 = dw_add(dw_add(C[0], C[3]), C[5]);
  dacc t2{0.0f, 0.0f};
  acc_prod(t2, C[0], C[3]);
  acc_prod(t2, C[3], C[5]);
  acc_prod(t2, C[0], C[5]);
  acc_prod(t2, dw_neg(C[1]), C[1]);
  acc_prod(t2, dw_neg(C[4]), C[4]);
  acc_prod(t2, dw_neg(C[2]), C[2]);
  const dw I2 = acc_val(t2);
  // cofactors of the symmetric C: Ci = cof / det C
  dw cf[6];
  cf[0] = dw_diff_prod(C[3], C[5], C[4], C[4]);
  cf[1] = dw_diff_prod(C[2], C[4], C[1], C[5]);
  cf[2] = dw_diff_prod(C[1], C[4], C[2], C[3]);
  cf[3] = dw_diff_prod(C[0], C[5], C[2], C[2]);
  cf[4] = dw_diff_prod(C[1], C[2], C[0], C[4]);
  cf[5] = dw_diff_prod(C[0], C[3], C[1], C[1]);
  dacc td{0.0f, 0.0f};
  acc_prod(td, C[0], cf[0]);
  acc_prod(td, C[1], cf[1]);
  acc_prod(td, C[2], cf[2]);
  const dw detC = acc_val(td);
  const dw J = dw_sqrt(detC);
  const dw rc = dw_rcbrt(J);
  const dw pp = dw_mul(rc, rc);      // J^(-2/3)
  const dw pppp = dw_mul(pp, pp);    // J^(-4/3)
  const dw oo = dw_rcp(detC);        // 1 / J^2
  dw Ci[6];
#pragma unroll
  for (int i = 0; i < 6; i++) Ci[i] = dw_mul(oo, cf[i]);
  const dw t13 = dw_mul(I1, dw{kThird_h, kThird_l});
  const dw t23 = dw_mul(I2, dw{kTwoThirds_h, kTwoThirds_l});
  dw a1, a2{0.0f, 0.0f}, a11{0.0f, 0.0f};
  if (mat_id == 1) {
    a1 = dw_scale2(dw_of(mcd[0]), 0.5f);
  } else if (mat_id == 2) {
    const dw d = dw_addf(dw_mul(I1, pp), -3.0f);
    const dw m1 = dw_of(mcd[1]), m2 = dw_of(mcd[2]);
    dacc ta{0.0f, 0.0f};
    acc_add(ta, dw_of(mcd[0]));
    acc_prod(ta, dw_scale2(m1, 2.0f), d);
    acc_prod(ta, dw_mulf(m2, 3.0f), dw_mul(d, d));
    a1 = acc_val(ta);
    a2 = dw_of(mcd[3]);
    a11 = dw_add(dw_scale2(m1, 2.0f), dw_mul(dw_mulf(m2, 6.0f), d));
  } else {
    a1 = dw_of(mcd[0]);
    a2 = dw_of(mcd[1]);
  }
  const float I6[6] = {1.0f, 0.0f, 0.0f, 1.0f, 0.0f, 1.0f};
  dw A[6], B[6];
#pragma unroll
  for (int i = 0; i < 6; i++) {
    A[i] = dw_addf(dw_neg(dw_mul(t13, Ci[i])), I6[i]);
    dacc tb{0.0f, 0.0f};
    acc_add(tb, dw_neg(C[i]));
    acc_prod(tb, dw_neg(t23), Ci[i]);
    if (I6[i] != 0.0f) acc_add(tb, I1);
    B[i] = acc_val(tb);
  }
  const dw ko1 = dw_scale2(dw_mul(a1, pp), 2.0f), ko2 = dw_scale2(dw_mul(a2, pppp), 2.0f);
  const dw pJs = dw_mul(p_state, J);
#pragma unroll
  for (int i = 0; i < 6; i++) {
    dacc ts{0.0f, 0.0f};
    acc_prod(ts, ko1, A[i]);
    acc_prod(ts, ko2, B[i]);
    acc_prod(ts, pJs, Ci[i]);
    S[i] = acc_val(ts);
  }
  Jout = J;
  // tangent coefficients (Dd before the reference's /2, times w), in float
  const dw k11 = dw_scale2(dw_mul(a11, pppp), 4.0f);
  const dw k1 = dw_mul(dw_mul(a1, pp), dw{kFourThirds_h, kFourThirds_l});
  const dw k2 = dw_mul(dw_mul(a2, pppp), dw{kEightThirds_h, kEightThirds_l});
  const dw pj = dw_mul(p_cur, J);
  dacc tc0{0.0f, 0.0f};
  acc_add(tc0, pj);
  acc_prod(tc0, dw_neg(k1), t13);
  acc_prod(tc0, dw_neg(k2), t23);
  const dw c0 = acc_val(tc0);
  dacc tst{0.0f, 0.0f};
  acc_add(tst, dw_scale2(pj, 2.0f));
  acc_prod(tst, dw_neg(k1), I1);
  acc_prod(tst, dw_neg(k2), I2);
  const float wf = w.h;
  const float sIIt = wf * acc_val(tst).h;
  const float sI = wf * 1.5f * k2.h;
  float At[6], Bt[6], Ct[6];
#pragma unroll
  for (int i = 0; i < 6; i++) {
    At[i] = A[i].h;
    Bt[i] = B[i].h;
    Ct[i] = Ci[i].h;
  }
  tangent_from_coefficients<float>(At, Bt, Ct, wf * k11.h, wf * k1.h, wf * k2.h, wf * c0.h, sIIt,
                                   sI, wD);
}

// ---------------------------------------------------------------------------
// FP64 kernel.  The FP64 pipe is what bounds it (1/64 of the FP32 rate: about
// 59 clocks per warp instruction and scheduler), so the algebra is arranged
// for the fewest FP64 instructions:
//
//  - Everything is written in the element's reference coordinates xi_p, where
//    the shape gradients at the 2 x 2 x 2 Gauss points are constants: with
//    sigma_d = +-1 the sign of coordinate d at a node b or a Gauss point g and
//    s = 1/sqrt(3),
//      dN_b/dxi_p (g) = 1/8 sum_{P not containing p} s^|P| phi_{P+p}(b) chi_P(g),
//    phi_S(b), chi_S(g) = prod_{d in S} sigma_d (P, S subsets of the three
//    coordinates).  The deformation gradient F = I + O itself is formed in the
//    global axes, O_ij = du_i/dxi_p dxi_p/dX_j, and so are J = det F, b = F F^T
//    and the invariants; only F and cof F then take xi components, FI_ip = F_ij
//    dxi_p/dX_j and V_ip = (F^-T)_ij dxi_p/dX_j.  (With dx_i/dxi_p and FI = dx/dxi g
//    the condition of dX/dxi entered twice: on an element sheared by 100 K_uu lost
//    four digits and F_u at 1e-4 strain five, for 5% fewer FP64 instructions.)
//    With the metric g^{pq} = (dxi_p/dX . dxi_q/dX) in the place of I:
//      C^-1 -> V^T V,  F A = FI - I1/3 V,  F B = I1 FI - b FI - 2 I2/3 V,
//      w F S = ko1 F A + ko2 F B + p J V,  w cof(F) dN/dX -> cof(F) dN/dxi,
//    and the tangent tensor is a sum of products of those 3 x 3 matrices
//      A[ip][kq] = V_ip X_kq + X_ip V_kq - sIIt/2 V_iq V_kp + k11 FA_ip FA_kq
//                  + sI (FI_ip FI_kq - FI_iq FI_kp / 2 - b_ik g^{pq} / 2)
//                  + delta_ik (S^{pq} - sIIt/2 C^-1^{pq})       (times w),
//    X = -k1 FA - k2 FB + c0/2 V: 2 or 3 FMA per entry instead of 6 and the
//    21 Voigt entries of D.
//  - Sum over the Gauss points: the products chi_P chi_Q make it a
//    Walsh-Hadamard transform of each tensor entry over the 8 points (24 adds
//    each for 45 entries of A, 9 of w F S, 9 of cof F), instead of h_a and 3
//    FMA per Kuu entry and Gauss point.
//  - Kuu(a,i; b,k) is then a sum of those over the (P, p), (Q, q) of both
//    sides: for each of the 7 modes P+p, seven sums over the modes Q+q and
//    their butterfly to the 8 nodes b (22 adds / FMA), then for each b the
//    butterfly over the modes to the 8 nodes a.
//  9,732 FP64 instructions per element (Mooney-Rivlin, counted by ncu) where
//  the form with h_a and 231 accumulated entries took 16,723.  Element launch
//  at 1e6 elements, Mooney-Rivlin: 28.9 -> 19.1 ms; at 216,000: 4.18 ms, and
//  3.27 ms Neo-Hookean.  The FP64 pipe is 87% busy; what is left is the two
//  warps per scheduler that shared memory allows waiting at the exchanges
//  (short scoreboard).
//
// One warp per four elements.  Lane = (element, node) for the displacements'
// butterfly to modes (exact differences to node 0 first), (element, Gauss
// point) for the material, (tensor entry, element) for the transforms, then
// (block (i, k), element) and (element, node b).  All exchange is through the
// warp's shared memory (25 KB: eight warps per SM).

// warp scratch, in doubles: 63 tensor rows of 4 elements x (8 points + pad);
// the mode-to-node sums T reuse the rows of w F S and cof F, the finished
// entries' stage the rows of A
constexpr int kFRow = 36, kFElem = 9;
constexpr int kFRowsA = 45;                      // A by (i, k) block: 6 or 9 entries
constexpr int kFRowP = kFRowsA, kFRowCof = kFRowsA + 9, kFRows = kFRowsA + 18;
// T: for each mode of the a side, 24 (block, element) x 8 nodes (+ pad).  The
// one-coordinate modes come last: they are written while w F S and cof F,
// which the four other blocks overwrite, are still read
constexpr int kFTMode = 24 * 9;
constexpr int kFT = kFRowsA * kFRow;
__host__ __device__ constexpr int f64_T(int mode) {
  return kFT + kFTMode * (mode == 3 ? 0 : mode == 5 ? 1 : mode == 6 ? 2 : mode == 7 ? 3
                          : mode == 1 ? 4 : mode == 2 ? 5 : 6);
}
constexpr int kFModes = kFRows * kFRow;          // modal positions: 3 x 32, before T exists
constexpr int kFWarp = kFT + 7 * kFTMode;
constexpr size_t kHead64Bytes = (kDposBytes + sizeof(uint16_t) * kFRows + 15) / 16 * 16;
static_assert(kFModes + 96 <= kFWarp && 4 * kKuuPerElem <= kFT, "scratch layout");
static_assert(kFT + 4 * kFTMode >= kFRows * kFRow, "one-coordinate modes beyond the F rows");

// first A row of block (i, k), i <= k (hblock order), and the entry within it
__device__ __forceinline__ constexpr int f64_block_row(int ik) {
  return ik == 0 ? 0 : ik == 1 ? 6 : ik == 2 ? 15 : ik == 3 ? 24 : ik == 4 ? 30 : 39;
}
__host__ __device__ constexpr int sym3(int p, int q) {
  return p <= q ? 3 * p - p * (p - 1) / 2 + (q - p) : 3 * q - q * (q - 1) / 2 + (p - q);
}
// node with the sign bits `mask` (bit d set: +1 in coordinate d), and back
__host__ __device__ constexpr int hex_corner(int mask) {
  return (mask & 2) ? (mask ^ 1) : mask;
}

// The butterfly of an element's eight lanes from corner values to shape modes
// (lane sub holds corner hex_corner(sub), then mode sub; not divided by 8), and
// a field's gradient in xi at the lane's Gauss point from its seven modes m.
__device__ __forceinline__ double corners_to_mode(double v, int sub) {
  v -= __shfl_sync(0xFFFFFFFFu, v, threadIdx.x & 24);
#pragma unroll
  for (int d = 1; d < 8; d <<= 1) {
    const double o = __shfl_xor_sync(0xFFFFFFFFu, v, d);
    v = (sub & d) ? __dsub_rn(v, o) : __dadd_rn(v, o);
  }
  return v;
}

struct GaussSigns {
  double x, y, z, xy, xz, yz;   // sigma_d / sqrt(3), and their products
};

__device__ __forceinline__ GaussSigns gauss_signs(int g) {
  GaussSigns s;
  s.x = (g & 1) ? kGaussA : -kGaussA;
  s.y = (g & 2) ? kGaussA : -kGaussA;
  s.z = (g & 4) ? kGaussA : -kGaussA;
  s.xy = __dmul_rn(s.x, s.y);
  s.xz = __dmul_rn(s.x, s.z);
  s.yz = __dmul_rn(s.y, s.z);
  return s;
}

__device__ __forceinline__ void mode_gradient(const double m[8], const GaussSigns& s, double F[3]) {
  F[0] = fma(s.yz, m[7], fma(s.z, m[5], fma(s.y, m[3], m[1])));
  F[1] = fma(s.xz, m[7], fma(s.z, m[6], fma(s.x, m[3], m[2])));
  F[2] = fma(s.xy, m[7], fma(s.y, m[6], fma(s.x, m[5], m[4])));
}

__device__ __forceinline__ double minor2(double a, double b, double c, double d) {
  return fma(a, b, -__dmul_rn(c, d));   // a b - c d
}

// cof F (F^-T det F) and det F
__device__ __forceinline__ double cofactors(const double F[9], double cof[9]) {
  cof[0] = minor2(F[4], F[8], F[5], F[7]);
  cof[1] = minor2(F[5], F[6], F[3], F[8]);
  cof[2] = minor2(F[3], F[7], F[4], F[6]);
  cof[3] = minor2(F[2], F[7], F[1], F[8]);
  cof[4] = minor2(F[0], F[8], F[2], F[6]);
  cof[5] = minor2(F[1], F[6], F[0], F[7]);
  cof[6] = minor2(F[1], F[5], F[2], F[4]);
  cof[7] = minor2(F[2], F[3], F[0], F[5]);
  cof[8] = minor2(F[0], F[4], F[1], F[3]);
  return fma(F[2], cof[2], fma(F[1], cof[1], __dmul_rn(F[0], cof[0])));
}

// v / 8, by the exponent (an integer subtraction, not an FP64 multiply)
__device__ __forceinline__ double eighth(double v) {
  const int hi = __double2hiint(v);
  if ((hi & 0x7FF00000) <= (3 << 20) || (hi & 0x7FF00000) == 0x7FF00000) return 0.125 * v;
  return __hiloint2double(hi - (3 << 20), __double2loint(v));
}

// J^(-1/3): the float estimate x0 improved by one third-order Householder step
// for x^-3 = J: with e = 1 - J x0^3, J^(-1/3) = x0 (1 - e)^(-1/3)
// = x0 (1 + e/3 + 2 e^2/9 + O(e^3)), |e| < 2^-20; rcbrt() outside the floats'
// comfortable range
__device__ __forceinline__ double inv_cbrt(double J) {
  if (!(J > 1e-30 && J < 1e30)) return rcbrt(J);
  const double x0 = (double)rcbrtf((float)J);
  const double e = fma(-J, x0 * x0 * x0, 1.0);
  return fma(x0 * e, fma(2.0 / 9.0, e, 1.0 / 3.0), x0);
}

// o[mask of b] = sum over the modes of c_mode phi_mode(b) M_mode, c = 1, s, s^2
// for one, two, three coordinates
__device__ __forceinline__ void modes_to_nodes(const double M[8], double o[8]) {
  constexpr double s = kGaussA;
#pragma unroll
  for (int x = 0; x < 2; x++) {
    const double sx = x ? s : -s;
    const double p2 = fma(sx, M[3], M[2]), p4 = fma(sx, M[5], M[4]), p6 = fma(sx, M[7], M[6]);
    const double m1 = x ? M[1] : -M[1];
    const double xy[2] = {m1 - p2, m1 + p2};
    const double z[2] = {fma(-s, p6, p4), fma(s, p6, p4)};
#pragma unroll
    for (int y = 0; y < 2; y++) {
      o[x + 2 * y] = xy[y] - z[y];
      o[x + 2 * y + 4] = xy[y] + z[y];
    }
  }
}

template <int WPB>
__global__ void __launch_bounds__(WPB * 32)
    solid81_fp64_kernel(const Solid81Args a) {
  if (a.skip && *a.skip) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint16_t* dpos = reinterpret_cast<uint16_t*>(smem_raw);  // [kDpos]
  // first double of the tensor rows: the 27 entries with p != q, then the 36
  // that need four characters, p = 0, 1, 2 in turn
  uint16_t* rows = dpos + kDpos;
  double* sm = reinterpret_cast<double*>(smem_raw + kHead64Bytes) + kFWarp * (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  for (int v = threadIdx.x; v < kDpos; v += blockDim.x) dpos[v] = c_dpos[v];
  if (threadIdx.x < 6) {
    const int ik = threadIdx.x;
    const bool diag = ik == 0 || ik == 3 || ik == 5;
    // entries p != q before this block: 3 per i = k block, 6 per i < k block
    int n = ik == 0 ? 0 : ik == 1 ? 3 : ik == 2 ? 9 : ik == 3 ? 15 : ik == 4 ? 18 : 24;
    for (int p = 0; p < 3; p++)
      for (int r = diag ? p : 0; r < 3; r++) {
        const int row = kFRow * (f64_block_row(ik) + (diag ? sym3(p, r) : 3 * p + r));
        if (p == r) rows[27 + 3 * ik + p] = (uint16_t)row;
        else rows[n++] = (uint16_t)row;
      }
  } else if (threadIdx.x < 24) {
    const int c = threadIdx.x - 6;   // the 18 rows of w F S and cof F
    rows[27 + 18 + c] = (uint16_t)(kFRow * (kFRowP + c));
  }
  __syncthreads();

  const uint32_t E = a.n_elems;  // end of this launch's element range
  const uint64_t E8 = (uint64_t)(a.n_total ? a.n_total : E) * 8;
  const uint64_t n_quads = (E + kEPW - 1) / kEPW;
  const uint64_t warp_global = (uint64_t)blockIdx.x * WPB + (threadIdx.x >> 5);
  const uint64_t warp_stride = (uint64_t)gridDim.x * WPB;
  const int q = lane >> 3, sub = lane & 7;
  const GaussSigns sg = gauss_signs(sub);

  for (uint64_t quad = a.e_begin / kEPW + warp_global; quad < n_quads; quad += warp_stride) {
    const uint32_t e0 = (uint32_t)(quad * kEPW);
    const uint32_t e = e0 + q;
    const bool valid = e < E;
    const uint32_t ec = valid ? e : E - 1;
    const uint64_t tg = (uint64_t)ec * 8 + sub;

    // ---- modal displacements, lane = (element, node), then mode ----
    double um[3] = {0.0, 0.0, 0.0};
    if (a.have_state) {
      const uint32_t nid = __ldg(a.conn + (uint64_t)ec * 8 + hex_corner(sub));
      const uint4 eq = __ldg(reinterpret_cast<const uint4*>(a.node_eq3) + (nid - 1));
      const double u[3] = {a.U_state[eq.x - 1], a.U_state[eq.y - 1], a.U_state[eq.z - 1]};
#pragma unroll
      for (int i = 0; i < 3; i++) um[i] = 0.125 * corners_to_mode(u[i], sub);
    }
#pragma unroll
    for (int i = 0; i < 3; i++) sm[kFModes + 32 * i + lane] = um[i];   // (mode 0 is not read)
    const double w = __ldg(a.wdet + tg);
    double Xi[9], g[6];   // dxi_p/dX_i at 3 i + p, and the metric
#pragma unroll
    for (int c = 0; c < 9; c++) Xi[c] = __ldg(a.geo + c * E8 + tg);
#pragma unroll
    for (int c = 0; c < 6; c++) g[c] = __ldg(a.geo + (9 + c) * E8 + tg);
    const double pc = a.U_cur[a.p_eq[ec] - 1];
    const double ps = a.have_state ? a.U_state[a.p_eq[ec] - 1] : 0.0;
    int mat_id = a.mat_id;
    const double* mc = a.mc;
    double inv_kb = a.inv_kb;
    if (a.elem_mesh) {
      const double* mm = a.mesh_mat + 8 * (uint64_t)__ldg(a.elem_mesh + ec);
      mat_id = (int)mm[0];
      mc = mm + 1;
      inv_kb = mm[7];
    }
    __syncwarp();

    // ---- material, lane = (element, Gauss point) ----
    double Fp_part, Kpp_part;
    {
      double F[9], cof[9];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        double du[3];   // du_i/dxi_p
        mode_gradient(sm + kFModes + 32 * i + 8 * q, sg, du);
#pragma unroll
        for (int k = 0; k < 3; k++) {
          const double O = fma(du[2], Xi[3 * k + 2], fma(du[1], Xi[3 * k + 1], du[0] * Xi[3 * k]));
          F[3 * i + k] = i == k ? 1.0 + O : O;
        }
      }
      const double detF = cofactors(F, cof);
      // J as sqrt(det C) gives it; an inverted element (det F <= 0, or w <= 0:
      // numbered left-handed) is flagged and keeps the reference's values
      const double J = fabs(detF);
      const bool bad = valid && !(J > 0.0 && isfinite(J) && detF > 0.0 && w > 0.0);
      const unsigned ballot = __ballot_sync(0xFFFFFFFFu, bad);
      if (sub == 0 && ((ballot >> (q * 8)) & 0xFFu)) flag_element(a.status, e + 1);
      Kpp_part = -inv_kb * w;
      Fp_part = fma(1.0 - J, w, -pc * Kpp_part);   // -(J - 1 - p / K) w
      const double rc = inv_cbrt(J);
      const double pp = rc * rc;       // J^(-2/3)
      // 1 / det F, the cube's three roundings taken out (F A is a difference: it
      // shows them at small strains)
      const double id0 = pp * rc;
      const double id = copysign(fma(id0, fma(-J, id0, 1.0), id0), detF);
      // F and cof F in xi components.  At rest (or translated) F = I exactly, and
      // so V = FI, I1 = 3 and F A = F B = 0, as the reference finds them
      double V[9], FI[9];
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int p = 0; p < 3; p++) {
          FI[3 * i + p] = fma(F[3 * i + 2], Xi[6 + p], fma(F[3 * i + 1], Xi[3 + p], F[3 * i] * Xi[p]));
          const double c = fma(cof[3 * i + 2], Xi[6 + p],
                               fma(cof[3 * i + 1], Xi[3 + p], cof[3 * i] * Xi[p]));
          V[3 * i + p] = c * id;
          sm[(kFRowCof + 3 * i + p) * kFRow + kFElem * q + sub] = w * c;
        }
      double I1 = F[0] * F[0];
#pragma unroll
      for (int c = 1; c < 9; c++) I1 = fma(F[c], F[c], I1);
      const double t13 = (1.0 / 3.0) * I1;
      const double pj = pc * J, pJs = ps * J;
      const double w64 = w * 0.015625;   // the two factors 1/8 of dN/dxi
      double FA[9];
#pragma unroll
      for (int c = 0; c < 9; c++) FA[c] = fma(-t13, V[c], FI[c]);
      double CI[6];
#pragma unroll
      for (int p = 0; p < 3; p++)
#pragma unroll
        for (int r = p; r < 3; r++)
          CI[sym3(p, r)] = V[p] * V[r] + V[3 + p] * V[3 + r] + V[6 + p] * V[6 + r];
      auto store_A = [&](int i, int k, int p, int r, double v) {
        const int row = f64_block_row(hblock(i, k)) + (i == k ? sym3(p, r) : 3 * p + r);
        sm[row * kFRow + kFElem * q + sub] = v;
      };
      // (warp-uniform: the general form serves every lane of a mixed warp)
      const bool general = __any_sync(0xFFFFFFFFu, mat_id != 1);
      double X[9], hV[9];
      if (!general) {
        const double a1 = 0.5 * mc[0];
        const double ko1 = a.have_state ? 2 * a1 * pp : 0.0;
        const double k1 = (4.0 / 3.0) * a1 * pp;
        const double c0 = pj - k1 * t13;
        const double h = -0.5 * w64 * (2.0 * pj - k1 * I1);
        const double pk = -w * ko1, pv = -w * pJs;
#pragma unroll
        for (int c = 0; c < 9; c++)
          sm[(kFRowP + c) * kFRow + kFElem * q + sub] = fma(pk, FA[c], pv * V[c]);
        const double xk = -w64 * k1, xv = 0.5 * w64 * c0;
        const double eg = w64 * ko1, ec2 = w64 * (pJs - ko1 * t13) + h;
        double Ed[6];
#pragma unroll
        for (int c = 0; c < 6; c++) Ed[c] = fma(ec2, CI[c], eg * g[c]);
#pragma unroll
        for (int c = 0; c < 9; c++) {
          X[c] = fma(xk, FA[c], xv * V[c]);
          hV[c] = h * V[c];
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
          // i = k: the two V V terms join in Y = X + h V
          double Y[3];
#pragma unroll
          for (int p = 0; p < 3; p++) Y[p] = X[3 * i + p] + hV[3 * i + p];
#pragma unroll
          for (int p = 0; p < 3; p++)
#pragma unroll
            for (int r = p; r < 3; r++)
              store_A(i, i, p, r,
                      fma(V[3 * i + p], Y[r], fma(X[3 * i + p], V[3 * i + r], Ed[sym3(p, r)])));
#pragma unroll
          for (int k = i + 1; k < 3; k++)
#pragma unroll
            for (int p = 0; p < 3; p++)
#pragma unroll
              for (int r = 0; r < 3; r++)
                store_A(i, k, p, r,
                        fma(V[3 * i + p], X[3 * k + r],
                            fma(X[3 * i + p], V[3 * k + r], hV[3 * i + r] * V[3 * k + p])));
        }
      } else {
        const double pppp = pp * pp;     // J^(-4/3)
        double b[6];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
          for (int k = i; k < 3; k++)
            b[sym3(i, k)] = F[3 * i] * F[3 * k] + F[3 * i + 1] * F[3 * k + 1] +
                            F[3 * i + 2] * F[3 * k + 2];
        const double I2 = b[0] * b[3] + b[3] * b[5] + b[0] * b[5] - b[1] * b[1] - b[4] * b[4] -
                          b[2] * b[2];
        const double t23 = (2.0 / 3.0) * I2;
        // W derivatives at (I1 J^-2/3, I2 J^-4/3) (materials_hyperelastic.cpp:135-204)
        double a1, a2 = 0.0, a11 = 0.0;
        if (mat_id == 1) {
          a1 = 0.5 * mc[0];
        } else if (mat_id == 2) {
          const double d = I1 * pp - 3.0;
          a1 = mc[0] + 2 * mc[1] * d + 3 * mc[2] * d * d;
          a2 = mc[3];
          a11 = 2 * mc[1] + 6 * mc[2] * d;
        } else {
          a1 = mc[0];
          a2 = mc[1];
        }
        const double st = a.have_state ? 1.0 : 0.0;
        const double ko1 = st * (2 * a1 * pp), ko2 = st * (2 * a2 * pppp);
        const double k11 = 4.0 * a11 * pppp, k1 = (4.0 / 3.0) * a1 * pp, k2 = (8.0 / 3.0) * a2 * pppp;
        const double c0 = pj - k1 * t13 - k2 * t23;
        const double h = -0.5 * w64 * (2.0 * pj - k1 * I1 - k2 * I2);
        const double sI = 1.5 * w64 * k2;
        const double pk = -w * ko1, pb = -w * ko2, pv = -w * pJs;
        const double xk = -w64 * k1, xb = -w64 * k2, xv = 0.5 * w64 * c0;
        const double w11 = w64 * k11;
        const bool biderman = __any_sync(0xFFFFFFFFu, a11 != 0.0);
#pragma unroll
        for (int c = 0; c < 9; c++) {
          const int i = c / 3, p = c % 3;
          const double fc = b[sym3(i, 0)] * FI[p] + b[sym3(i, 1)] * FI[3 + p] +
                            b[sym3(i, 2)] * FI[6 + p];
          const double FB = fma(-t23, V[c], fma(I1, FI[c], -fc));
          sm[(kFRowP + c) * kFRow + kFElem * q + sub] = fma(pk, FA[c], fma(pb, FB, pv * V[c]));
          X[c] = fma(xk, FA[c], fma(xb, FB, xv * V[c]));
          hV[c] = h * V[c];
        }
        // S^{pq} = (ko1 + ko2 I1) g - ko2 C^{pq} + (p J - ko1 I1/3 - ko2 2 I2/3) C^-1
        const double eg = w64 * (ko1 + ko2 * I1), ecc = -w64 * ko2;
        const double ec2 = w64 * (pJs - ko1 * t13 - ko2 * t23) + h;
        const double hI = 0.5 * sI;
        double Ed[6];
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
          for (int r = p; r < 3; r++) {
            const int c = sym3(p, r);
            const double C = FI[p] * FI[r] + FI[3 + p] * FI[3 + r] + FI[6 + p] * FI[6 + r];
            Ed[c] = fma(ecc, C, fma(ec2, CI[c], eg * g[c]));
          }
#pragma unroll
        for (int i = 0; i < 3; i++) {
          double Y[3], Z[3], Z2[3], W3[3];
          const double bi = -hI * b[sym3(i, i)];
#pragma unroll
          for (int p = 0; p < 3; p++) {
            Y[p] = X[3 * i + p] + hV[3 * i + p];
            Z[p] = hI * FI[3 * i + p];
            if (i < 2) Z2[p] = sI * FI[3 * i + p];
            if (biderman) W3[p] = w11 * FA[3 * i + p];
          }
#pragma unroll
          for (int p = 0; p < 3; p++)
#pragma unroll
            for (int r = p; r < 3; r++) {
              double v = fma(bi, g[sym3(p, r)], Ed[sym3(p, r)]);
              v = fma(Z[p], FI[3 * i + r], v);
              v = fma(V[3 * i + p], Y[r], fma(X[3 * i + p], V[3 * i + r], v));
              if (biderman) v = fma(W3[p], FA[3 * i + r], v);
              store_A(i, i, p, r, v);
            }
#pragma unroll
          for (int k = i + 1; k < 3; k++) {
            const double bk = -hI * b[sym3(i, k)];
            double bg[6];
#pragma unroll
            for (int c = 0; c < 6; c++) bg[c] = bk * g[c];
#pragma unroll
            for (int p = 0; p < 3; p++)
#pragma unroll
              for (int r = 0; r < 3; r++) {
                double v = fma(-Z[r], FI[3 * k + p], bg[sym3(p, r)]);
                v = fma(Z2[p], FI[3 * k + r], v);
                v = fma(hV[3 * i + r], V[3 * k + p], v);
                v = fma(V[3 * i + p], X[3 * k + r], fma(X[3 * i + p], V[3 * k + r], v));
                if (biderman) v = fma(W3[p], FA[3 * k + r], v);
                store_A(i, k, p, r, v);
              }
          }
        }
      }
    }
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) {
      Fp_part += __shfl_xor_sync(0xFFFFFFFFu, Fp_part, off);
      Kpp_part += __shfl_xor_sync(0xFFFFFFFFu, Kpp_part, off);
    }
    __syncwarp();

    // ---- sums over the Gauss points: the rows' transforms, in place ----
    // An entry (p, q) with p = q, and every entry (i, p) of w F S and cof F,
    // is read only at the characters without coordinate p: its two halves in
    // p are added and four points transformed (12 adds instead of 24).
#pragma unroll 2
    for (int r = 0; r < 4; r++) {
      const int t = lane + 32 * r;   // 27 entries p != q x 4 elements
      if (t >= 27 * kEPW) break;
      double* W = sm + rows[t >> 2] + kFElem * (t & 3);
      double v[8];
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = W[j];
#pragma unroll
      for (int d = 1; d < 8; d <<= 1)
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (!(j & d)) {
            const double lo = v[j], hi = v[j | d];
            v[j] = lo + hi;
            v[j | d] = hi - lo;
          }
#pragma unroll
      for (int j = 0; j < 8; j++) W[j] = v[j];
    }
#pragma unroll 2
    for (int r = 0; r < 5; r++) {
      const int t = lane + 32 * r;   // 36 entries x 4 elements
      if (t >= 36 * kEPW) break;
      const int n = t >> 2;
      const int p = n % 3;
      double* W = sm + rows[27 + n] + kFElem * (t & 3);
      const int mp = 1 << p, ma = p == 0 ? 2 : 1, mb = p == 2 ? 2 : 4;
      const double v0 = W[0] + W[mp], va = W[ma] + W[ma + mp], vb = W[mb] + W[mb + mp],
                   vab = W[ma + mb] + W[7];
      const double s0 = v0 + va, d0 = va - v0, s1 = vb + vab, d1 = vab - vb;
      W[0] = s0 + s1;
      W[ma] = d0 + d1;
      W[mb] = s1 - s0;
      W[ma + mb] = d1 - d0;
    }
    __syncwarp();

    // destination of contribution idx: slot-ordered (kpos) or element-ordered
    auto kdst = [&](uint64_t idx) -> uint64_t { return a.kpos ? (uint64_t)__ldg(a.kpos + idx) : idx; };
    auto fdst = [&](uint64_t idx) -> uint64_t { return a.fpos ? (uint64_t)__ldg(a.fpos + idx) : idx; };

    // ---- modes of both sides, the b side to nodes ----
    // lanes 0 .. 23 = (block (i, k), element), one mode of the a side per
    // round; F_u and K_up (six components x four elements) have the form of a
    // one-coordinate mode and take the eight lanes left in those three rounds
    {
      const bool spare = lane >= 24;
      const int ik = spare ? 0 : lane >> 2, el = lane & 3;
      const bool diag = ik == 0 || ik == 3 || ik == 5;
      const double* W = sm + (spare ? kFRowP : f64_block_row(ik)) * kFRow + kFElem * el;
      int off[3][3];
#pragma unroll
      for (int p = 0; p < 3; p++)
#pragma unroll
        for (int r = 0; r < 3; r++)
          off[p][r] = kFRow * (spare ? 3 * (2 * p + ((lane >> 2) & 1)) + r
                                     : diag ? sym3(p, r) : 3 * p + r);
#pragma unroll
      for (int round = 0; round < 7; round++) {
        const int al = round == 0 ? 1 : round == 1 ? 2 : round == 2 ? 4 : round == 3 ? 3
                     : round == 4 ? 5 : round == 5 ? 6 : 7;
        if (round == 3) {
          __syncwarp();
          if (spare) break;
        }
        double M[8], o[8];
#pragma unroll
        for (int be = 1; be < 8; be++) {
          double v = 0.0;
          bool first = true;
#pragma unroll
          for (int p = 0; p < 3; p++) {
            if (!(al >> p & 1)) continue;
#pragma unroll
            for (int r = 0; r < 3; r++) {
              if (!(be >> r & 1)) continue;
              const double x = W[off[p][r] + ((al ^ (1 << p)) ^ (be ^ (1 << r)))];
              v = first ? x : v + x;
              first = false;
            }
          }
          M[be] = v;
        }
        modes_to_nodes(M, o);
        if (!spare) {
          double* T = sm + f64_T(al) + 9 * lane;
#pragma unroll
          for (int b = 0; b < 8; b++) T[b] = o[b];
        } else {
          const int c = 2 * round + ((lane >> 2) & 1);   // c < 3: F_u, else K_up
          const uint32_t ee = e0 + el;
          if (ee < E) {
#pragma unroll
            for (int b = 0; b < 8; b++) {
              const int n = hex_corner(b);
              const double v = eighth(o[b]);
              if (c < 3) a.contribF[fdst((uint64_t)ee * kSolidFc + 3 * n + c)] = v;
              else a.contribK[kdst((uint64_t)ee * kSolidKc + 300 + 3 * n + c - 3)] = v;
            }
          }
        }
      }
    }
    __syncwarp();

    // ---- the a side to nodes: lane = (element, node b), block by block ----
    {
      const int nb = hex_corner(sub);
#pragma unroll
      for (int ik = 0; ik < 6; ik++) {
        double M[8], o[8];
#pragma unroll
        for (int al = 1; al < 8; al++) M[al] = sm[f64_T(al) + 9 * (ik * 4 + q) + sub];
        modes_to_nodes(M, o);
#pragma unroll
        for (int m = 0; m < 8; m++) {
          const uint32_t pos = dpos[(hex_corner(m) * 6 + ik) * 8 + nb];
          if (pos != 0xFFFFu) sm[q * kKuuPerElem + pos] = o[m];
        }
      }
    }
    __syncwarp();
#pragma unroll 4
    for (int m = 0; m < kOwned; m++) {
      const int x = lane + 32 * m;
      if (x < kEPW * kKuuPerElem) {
        const int qq = x / kKuuPerElem, t = x - qq * kKuuPerElem;
        const uint32_t ee = e0 + qq;
        if (ee < E) a.contribK[kdst((uint64_t)ee * kSolidKc + t)] = sm[x];
      }
    }
    if (valid && sub == 0) {
      a.contribK[kdst((uint64_t)e * kSolidKc + 324)] = Kpp_part;
      a.contribF[fdst((uint64_t)e * kSolidFc + 24)] = Fp_part;
    }
    __syncwarp();
  }
}

template <int WPB>
__global__ void __launch_bounds__(WPB * 32)
    solid81_mixed_kernel(const Solid81Args a) {
  if (a.skip && *a.skip) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // block header: the D -> assemble3 position table
  uint16_t* dpos = reinterpret_cast<uint16_t*>(smem_raw);  // [kDpos]
  MixedSmem* sm = reinterpret_cast<MixedSmem*>(smem_raw + kDposBytes) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;

  for (int v = threadIdx.x; v < kDpos; v += blockDim.x) dpos[v] = c_dpos[v];
  __syncthreads();

  const uint32_t E = a.n_elems;  // end of this launch's element range
  const uint64_t E8 = (uint64_t)(a.n_total ? a.n_total : E) * 8;
  const uint64_t n_quads = (E + kEPW - 1) / kEPW;
  const uint64_t warp_global = (uint64_t)blockIdx.x * WPB + (threadIdx.x >> 5);
  const uint64_t warp_stride = (uint64_t)gridDim.x * WPB;

  for (uint64_t quad = a.e_begin / kEPW + warp_global; quad < n_quads; quad += warp_stride) {
    const uint32_t e0 = (uint32_t)(quad * kEPW);
    const int q = lane >> 3;
    const int sub = lane & 7;  // Gauss point in phase 1, node in phase 2
    const uint32_t e = e0 + q;
    const bool valid = e < E;
    const uint32_t ec = valid ? e : E - 1;

    // ---------------- phase 1: lane = (element q, Gauss point g) ----------------
    double Fp_part = 0.0, Kpp_part = 0.0;  // FP64
    {
      const int g = sub;
      const uint64_t tg = (uint64_t)ec * 8 + g;
      float Fm[9], wS[6], wD[21];
      bool bad;
      {
        // the residual chain in float pairs, the tangent inputs rounded to float
        const dw w = dw_of(__ldg(a.wdf + tg));
        const dw pc = dw_from_double(a.U_cur[a.p_eq[ec] - 1]);
        dw O[9];
        dw C[6];
        dw ps{0.0f, 0.0f};
        if (a.have_state) {
          // O = sum_n (u_n - u_0) G_n (the shape gradients sum to zero): the
          // displacements relative to the element's node 0 are formed in FP64,
          // so the pairs carry the small differences, not |u| (which can be
          // ~1/h times larger, and would cost that factor in accuracy).
          // Lane (q, g) forms node g's difference; the others read it by shuffle.
          const uint32_t* cn = a.conn + (uint64_t)ec * 8;
          const uint4 eq0 = __ldg(reinterpret_cast<const uint4*>(a.node_eq3) + (__ldg(cn) - 1));
          const uint4 eqg = __ldg(reinterpret_cast<const uint4*>(a.node_eq3) + (__ldg(cn + g) - 1));
          const dw dx = dw_from_double(a.U_state[eqg.x - 1] - a.U_state[eq0.x - 1]);
          const dw dy = dw_from_double(a.U_state[eqg.y - 1] - a.U_state[eq0.y - 1]);
          const dw dz = dw_from_double(a.U_state[eqg.z - 1] - a.U_state[eq0.z - 1]);
          dw G[24];
#pragma unroll
          for (int c = 0; c < 24; c++) G[c] = dw_of(__ldg(a.Gdf + c * E8 + tg));
          dacc Oa[9];
#pragma unroll
          for (int c = 0; c < 9; c++) Oa[c] = dacc{0.0f, 0.0f};
          const int base = lane & ~7;
#pragma unroll
          for (int n = 1; n < 8; n++) {
            const dw ux{__shfl_sync(0xFFFFFFFFu, dx.h, base + n), __shfl_sync(0xFFFFFFFFu, dx.l, base + n)};
            const dw uy{__shfl_sync(0xFFFFFFFFu, dy.h, base + n), __shfl_sync(0xFFFFFFFFu, dy.l, base + n)};
            const dw uz{__shfl_sync(0xFFFFFFFFu, dz.h, base + n), __shfl_sync(0xFFFFFFFFu, dz.l, base + n)};
#pragma unroll
            for (int j = 0; j < 3; j++) {
              acc_prod(Oa[0 + j], ux, G[3 * n + j]);
              acc_prod(Oa[3 + j], uy, G[3 * n + j]);
              acc_prod(Oa[6 + j], uz, G[3 * n + j]);
            }
          }
#pragma unroll
          for (int c = 0; c < 9; c++) O[c] = acc_val(Oa[c]);
          ps = dw_from_double(a.U_state[a.p_eq[ec] - 1]);
          // C = F^T F = I + O + O^T + O^T O (SOLID81.cpp:105-110)
          const int dg[3] = {0, 4, 8};
          const int cj[6] = {0, 0, 0, 1, 1, 2}, cl[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
          for (int v = 0; v < 6; v++) {
            const int J = cj[v], L = cl[v];
            dacc t{J == L ? 1.0f : 0.0f, 0.0f};
            if (J == L) {
              acc_add(t, dw_scale2(O[dg[J]], 2.0f));
            } else {
              acc_add(t, O[3 * J + L]);
              acc_add(t, O[3 * L + J]);
            }
#pragma unroll
            for (int i = 0; i < 3; i++) acc_prod(t, O[3 * i + J], O[3 * i + L]);
            C[v] = acc_val(t);
          }
        } else {
#pragma unroll
          for (int c = 0; c < 9; c++) O[c] = dw{0.0f, 0.0f};
          C[0] = C[3] = C[5] = dw{1.0f, 0.0f};
          C[1] = C[2] = C[4] = dw{0.0f, 0.0f};
        }
        int mat_id = a.mat_id;
        const float2* mcd = a.mcd;
        if (a.elem_mesh) {
          const uint32_t mi = __ldg(a.elem_mesh + ec);
          mat_id = (int)a.mesh_mat[8 * (uint64_t)mi];
          mcd = a.mesh_mat_df + 8 * (uint64_t)mi + 1;
        }
        dw S[6], J;
        material_mixed(mat_id, mcd, C, ps, pc, w, S, J, wD);
        if (!a.have_state) {
#pragma unroll
          for (int i = 0; i < 6; i++) S[i] = dw{0.0f, 0.0f};
        }
        dw F[9];
#pragma unroll
        for (int c = 0; c < 9; c++) F[c] = (c == 0 || c == 4 || c == 8) ? dw_addf(O[c], 1.0f) : O[c];
        const int sv[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
          for (int k = 0; k < 3; k++) {
            dacc t{0.0f, 0.0f};
#pragma unroll
            for (int J2 = 0; J2 < 3; J2++) acc_prod(t, F[3 * i + J2], S[sv[3 * J2 + k]]);
            const dw wp = dw_mul(w, acc_val(t));
            // slot g * 4 + q: the four elements' pairs of one Gauss point
            // fall in different bank pairs when phase 2 reads them
            sm->wP[3 * i + k][g * 4 + q] = make_float2(-wp.h, -wp.l);
          }
#pragma unroll
        for (int c = 0; c < 9; c++) Fm[c] = F[c].h;
#pragma unroll
        for (int c = 0; c < 6; c++) wS[c] = w.h * S[c].h;
        // The volumetric terms in FP64: F (the pair O widened exactly, plus
        // I), cof F, J = det F, and from them Fp = -(J - 1 - p / K) w,
        // Kpp = -w / K (SOLID81.cpp:78-79) and w cof F = w J F^-T, whose
        // products with G_a are K_up (D_p = J C^-1, materials_hyperelastic.cpp:127).
        double Fd[9];
#pragma unroll
        for (int c = 0; c < 9; c++) {
          const double o = dw_to_double(O[c]);
          Fd[c] = (c == 0 || c == 4 || c == 8) ? 1.0 + o : o;
        }
        const double cofd[9] = {Fd[4] * Fd[8] - Fd[5] * Fd[7], Fd[5] * Fd[6] - Fd[3] * Fd[8],
                                Fd[3] * Fd[7] - Fd[4] * Fd[6], Fd[2] * Fd[7] - Fd[1] * Fd[8],
                                Fd[0] * Fd[8] - Fd[2] * Fd[6], Fd[1] * Fd[6] - Fd[0] * Fd[7],
                                Fd[1] * Fd[5] - Fd[2] * Fd[4], Fd[2] * Fd[3] - Fd[0] * Fd[5],
                                Fd[0] * Fd[4] - Fd[1] * Fd[3]};
        const double wd = a.wdet[tg];
#pragma unroll
        for (int c = 0; c < 9; c++) sm->wCof[c][g * 4 + q] = wd * cofd[c];
        {
          const float cf[9] = {Fm[4] * Fm[8] - Fm[5] * Fm[7], Fm[5] * Fm[6] - Fm[3] * Fm[8],
                               Fm[3] * Fm[7] - Fm[4] * Fm[6], Fm[2] * Fm[7] - Fm[1] * Fm[8],
                               Fm[0] * Fm[8] - Fm[2] * Fm[6], Fm[1] * Fm[6] - Fm[0] * Fm[7],
                               Fm[1] * Fm[5] - Fm[2] * Fm[4], Fm[2] * Fm[3] - Fm[0] * Fm[5],
                               Fm[0] * Fm[4] - Fm[1] * Fm[3]};
#pragma unroll
          for (int c = 0; c < 9; c++) sm->wCofF[c][g * 4 + q] = w.h * cf[c];
        }
        const double Jd = Fd[0] * cofd[0] + Fd[1] * cofd[1] + Fd[2] * cofd[2];
        const double inv_kbd =
            a.elem_mesh ? a.mesh_mat[8 * (uint64_t)__ldg(a.elem_mesh + ec) + 7] : a.inv_kb;
        const double pcd = a.U_cur[a.p_eq[ec] - 1];
        Fp_part = -(Jd - 1 - pcd * inv_kbd) * wd;
        Kpp_part = -inv_kbd * wd;
        bad = valid && !(Jd > 0.0 && isfinite(Jd) && J.h > 0.0f && isfinite(J.h) && wd > 0.0);
      }
      // A[iL][kN] = sum_J F_iJ (sum_M wD[(JL)][(MN)] F_kM) + delta_ik w S_LN,
      // one row (i, L) at a time
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int L = 0; L < 3; L++) {
          float T6[6];
#pragma unroll
          for (int t = 0; t < 6; t++)
            T6[t] = Fm[3 * i + 0] * wD[sym6u(voigt(0, L), t)] +
                    Fm[3 * i + 1] * wD[sym6u(voigt(1, L), t)] +
                    Fm[3 * i + 2] * wD[sym6u(voigt(2, L), t)];
#pragma unroll
          for (int k = 0; k < 3; k++)
#pragma unroll
            for (int N = 0; N < 3; N++) {
              if (3 * k + N < 3 * i + L) continue;
              float v = T6[voigt(0, N)] * Fm[3 * k + 0] + T6[voigt(1, N)] * Fm[3 * k + 1] +
                     T6[voigt(2, N)] * Fm[3 * k + 2];
              if (i == k) v += wS[voigt(L, N)];
              sm->A[sym9(3 * i + L, 3 * k + N)][lane] = v;
            }
        }
      const unsigned ballot = __ballot_sync(0xFFFFFFFFu, bad);
      if (sub == 0 && ((ballot >> (q * 8)) & 0xFFu)) flag_element(a.status, e + 1);
    }
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) {
      Fp_part += __shfl_xor_sync(0xFFFFFFFFu, Fp_part, off);
      Kpp_part += __shfl_xor_sync(0xFFFFFFFFu, Kpp_part, off);
    }
    __syncwarp();

    // destination of contribution idx: slot-ordered (kpos) or element-ordered
    auto kdst = [&](uint64_t idx) -> uint64_t { return a.kpos ? (uint64_t)__ldg(a.kpos + idx) : idx; };
    auto fdst = [&](uint64_t idx) -> uint64_t { return a.fpos ? (uint64_t)__ldg(a.fpos + idx) : idx; };

    {
      // Residual and pressure coupling, lane = (element q, node a), before the
      // Gauss point loop reuses the scratch that holds -w F S and w cof F:
      //   F_u(a, i) = sum_g sum_L (-w F S)_g[iL] G_g[aL]   (float pairs),
      //   K_up(a, i) = sum_g sum_L (w cof F)_g[iL] G_g[aL]  (FP64),
      // G = G_hi + G_lo its pair.  The K_up products with G_hi are FP64 FMAs
      // (two accumulators, even and odd Gauss points, to halve the dependent
      // chain); the products with G_lo, 2^-24 of the total, are summed in
      // FP32 (their error, 2^-48 of the total, is that of the pair itself)
      // and added in FP64 at the end.  The pair arithmetic of F_u keeps the
      // FP32 pipes busy while the FP64 FMAs drain.  Kpp and Fp are written
      // here too.
      double Kupd[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
      float Kupl[3] = {0.0f, 0.0f, 0.0f};
      dacc Fua[3] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
#pragma unroll 2
      for (int g = 0; g < 8; g++) {
        const uint64_t tg = (uint64_t)ec * 8 + g;
        const float2 p0 = __ldg(a.Gdf + (3 * sub + 0) * E8 + tg);
        const float2 p1 = __ldg(a.Gdf + (3 * sub + 1) * E8 + tg);
        const float2 p2 = __ldg(a.Gdf + (3 * sub + 2) * E8 + tg);
        const double G0 = f2d(p0.x), G1 = f2d(p1.x), G2 = f2d(p2.x);
        const int sp = g * 4 + q;
#pragma unroll
        for (int i = 0; i < 3; i++) {
          double& kd = Kupd[g & 1][i];
          kd = fma(sm->wCof[3 * i + 0][sp], G0, kd);
          kd = fma(sm->wCof[3 * i + 1][sp], G1, kd);
          kd = fma(sm->wCof[3 * i + 2][sp], G2, kd);
          Kupl[i] += sm->wCofF[3 * i + 0][sp] * p0.y + sm->wCofF[3 * i + 1][sp] * p1.y +
                     sm->wCofF[3 * i + 2][sp] * p2.y;
          acc_prod(Fua[i], dw_of(sm->wP[3 * i + 0][sp]), dw_of(p0));
          acc_prod(Fua[i], dw_of(sm->wP[3 * i + 1][sp]), dw_of(p1));
          acc_prod(Fua[i], dw_of(sm->wP[3 * i + 2][sp]), dw_of(p2));
        }
      }
      if (valid) {
        const uint64_t kb = (uint64_t)e * kSolidKc, fb = (uint64_t)e * kSolidFc;
#pragma unroll
        for (int i = 0; i < 3; i++) {
          a.contribK[kdst(kb + 300 + 3 * sub + i)] = (Kupd[0][i] + Kupd[1][i]) + f2d(Kupl[i]);
          a.contribF[fdst(fb + 3 * sub + i)] = dw_to_double(acc_val(Fua[i]));
        }
        if (sub == 0) {
          a.contribK[kdst(kb + 324)] = Kpp_part;
          a.contribF[fdst(fb + 24)] = Fp_part;
        }
      }
      __syncwarp();
    }

    // ---------------- phases 2 + 3 per Gauss point ----------------
    {
      // Lane (q, a) keeps h_a[ik] (i <= k, its own node) in registers and
      // accumulates D[(ik), a, b] = sum_g h_a[ik] . G_b for all 8 nodes b:
      // 48 sums of 3 FMA per Gauss point from 3 shared loads per node b.
      // The 48 cover the element's 300 Kuu entries (the 84 D[(ii), a, b],
      // a > b, repeat D[(ii), b, a] and are not written).
      float acc[6][8];
#pragma unroll
      for (int c = 0; c < 6; c++)
#pragma unroll
        for (int b = 0; b < 8; b++) acc[c][b] = 0.0f;
      for (int g = 0; g < 8; g++) {
        const int s1 = q * 8 + g;
        const uint64_t tg = (uint64_t)ec * 8 + g;
        // phase 2: the tangent uses the high parts of G
        const float g0 = __ldg(a.Gdf + (3 * sub + 0) * E8 + tg).x;
        const float g1 = __ldg(a.Gdf + (3 * sub + 1) * E8 + tg).x;
        const float g2 = __ldg(a.Gdf + (3 * sub + 2) * E8 + tg).x;
        float h[6][3];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
          for (int k = i; k < 3; k++)
#pragma unroll
            for (int N = 0; N < 3; N++)
              h[hblock(i, k)][N] = g0 * sm->A[sym9(3 * i + 0, 3 * k + N)][s1] +
                                   g1 * sm->A[sym9(3 * i + 1, 3 * k + N)][s1] +
                                   g2 * sm->A[sym9(3 * i + 2, 3 * k + N)][s1];
        sm->G[0][lane] = g0;
        sm->G[1][lane] = g1;
        sm->G[2][lane] = g2;
        __syncwarp();
        // phase 3
#pragma unroll
        for (int b = 0; b < 8; b++) {
          const float b0 = sm->G[0][q * 8 + b], b1 = sm->G[1][q * 8 + b],
                      b2 = sm->G[2][q * 8 + b];
#pragma unroll
          for (int c = 0; c < 6; c++) {
            float v = acc[c][b];
            v = fmaf(h[c][0], b0, v);
            v = fmaf(h[c][1], b1, v);
            v = fmaf(h[c][2], b2, v);
            acc[c][b] = v;
          }
        }
        __syncwarp();
      }
      // stage the quad's 4 x 300 entries in assemble3 order, then write them
      // coalesced (the stage shares its bytes with -w F S / w cof F, dead now)
#pragma unroll
      for (int c = 0; c < 6; c++)
#pragma unroll
        for (int b = 0; b < 8; b++) {
          const uint32_t pos = dpos[(sub * 6 + c) * 8 + b];
          if (pos != 0xFFFFu) sm->stage[q * kKuuPerElem + pos] = acc[c][b];
        }
      __syncwarp();
#pragma unroll 4
      for (int m = 0; m < kOwned; m++) {
        const int x = lane + 32 * m;
        if (x < kEPW * kKuuPerElem) {
          const int qq = x / kKuuPerElem, t = x - qq * kKuuPerElem;
          const uint32_t ee = e0 + qq;
          if (ee < E) a.contribK[kdst((uint64_t)ee * kSolidKc + t)] = f2d(sm->stage[x]);
        }
      }
      __syncwarp();
    }
  }
}

// The FP64 kernel's element geometry, one thread per Gauss point: the shape
// modes of the positions, and from them w = det dX/dxi, dxi_p/dX_i and the metric
// dxi_p/dX . dxi_q/dX.  The modes start from the differences along the edges: no
// digits are lost to the element's distance from the origin, nor a thin element's
// thickness to its length.
__global__ void __launch_bounds__(256) solid81_geometry_kernel(const JacobianArgs a) {
  if (a.skip && *a.skip) return;
  const uint64_t E8 = (uint64_t)a.n_elems * 8;
  const uint64_t t = (uint64_t)blockIdx.x * 256 + threadIdx.x;
  if (t >= E8) return;
  const int sub = threadIdx.x & 7;
  const uint32_t* cn = a.conn + (t & ~7ull);
  const GaussSigns sg = gauss_signs(sub);
  double F[9], cof[9];
  for (int i = 0; i < 3; i++) {
    double x[8], m[8], ex[4], ey[4], ez[4];   // corners by mask
    for (int b = 0; b < 8; b++) x[b] = a.xyz[(uint64_t)(cn[hex_corner(b)] - 1) * 3 + i];
    for (int k = 0; k < 4; k++) {
      const int y0 = (k & 1) | (k & 2) << 1;
      ex[k] = x[2 * k + 1] - x[2 * k];
      ey[k] = x[y0 + 2] - x[y0];
      ez[k] = x[k + 4] - x[k];
    }
    m[1] = (ex[0] + ex[1]) + (ex[2] + ex[3]);
    m[2] = (ey[0] + ey[1]) + (ey[2] + ey[3]);
    m[4] = (ez[0] + ez[1]) + (ez[2] + ez[3]);
    m[3] = (ex[1] - ex[0]) + (ex[3] - ex[2]);
    m[5] = (ex[2] - ex[0]) + (ex[3] - ex[1]);
    m[6] = (ey[2] - ey[0]) + (ey[3] - ey[1]);
    m[7] = (ex[3] - ex[2]) - (ex[1] - ex[0]);
    for (int b = 1; b < 8; b++) m[b] *= 0.125;
    mode_gradient(m, sg, F + 3 * i);
  }
  const double det = cofactors(F, cof);
  const double r = 1.0 / det;
  for (int c = 0; c < 9; c++) {
    cof[c] *= r;   // dxi_p/dX_i
    a.geo[c * E8 + t] = cof[c];
  }
  for (int p = 0; p < 3; p++)
    for (int s = p; s < 3; s++) {
      double v = 0.0;
      for (int i = 0; i < 3; i++) v += cof[3 * i + p] * cof[3 * i + s];
      a.geo[(9 + sym3(p, s)) * E8 + t] = v;
    }
  a.wdet[t] = det;
  // isoparametric.cpp:177 logs det < 1e-20; here it is an element status
  if (!(det >= 1.0e-20) && sub == 0) flag_element(a.status, (uint32_t)(t >> 3) + 1);
}

__global__ void solid81_jacobian_kernel(const JacobianArgs a) {
  if (a.skip && *a.skip) return;
  const uint64_t E8 = (uint64_t)a.n_elems * 8;
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= E8) return;
  const uint32_t e = (uint32_t)(t >> 3);
  const int g = (int)(t & 7);
  // Gauss point of ElementIsoParamHEXAHEDRON, order 2 (isoparametric.h:126-136)
  const double r = (g & 1) ? kGaussA : -kGaussA;
  const double s = (g & 2) ? kGaussA : -kGaussA;
  const double u = (g & 4) ? kGaussA : -kGaussA;
  // formFuncDeriv (isoparametric.cpp:211-221)
  const double dN[24] = {
      -0.125 * (1.0 - s) * (1.0 - u), -0.125 * (1.0 - r) * (1.0 - u), -0.125 * (1.0 - r) * (1.0 - s),
      +0.125 * (1.0 - s) * (1.0 - u), -0.125 * (1.0 + r) * (1.0 - u), -0.125 * (1.0 + r) * (1.0 - s),
      +0.125 * (1.0 + s) * (1.0 - u), +0.125 * (1.0 + r) * (1.0 - u), -0.125 * (1.0 + r) * (1.0 + s),
      -0.125 * (1.0 + s) * (1.0 - u), +0.125 * (1.0 - r) * (1.0 - u), -0.125 * (1.0 - r) * (1.0 + s),
      -0.125 * (1.0 - s) * (1.0 + u), -0.125 * (1.0 - r) * (1.0 + u), +0.125 * (1.0 - r) * (1.0 - s),
      +0.125 * (1.0 - s) * (1.0 + u), -0.125 * (1.0 + r) * (1.0 + u), +0.125 * (1.0 + r) * (1.0 - s),
      +0.125 * (1.0 + s) * (1.0 + u), +0.125 * (1.0 + r) * (1.0 + u), +0.125 * (1.0 + r) * (1.0 + s),
      -0.125 * (1.0 + s) * (1.0 + u), +0.125 * (1.0 - r) * (1.0 + u), +0.125 * (1.0 - r) * (1.0 + s)};
  double J[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int n = 0; n < 8; n++) {
    const uint32_t nid = a.conn[(uint64_t)e * 8 + n];
    const double* X = a.xyz + (uint64_t)(nid - 1) * 3;
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) J[3 * i + j] += dN[3 * n + i] * X[j];
  }
  // Mat<3,3>::det / inv (Mat.cpp:23-46)
  const double det = J[0] * (J[4] * J[8] - J[5] * J[7]) - J[1] * (J[3] * J[8] - J[5] * J[6]) +
                     J[2] * (J[3] * J[7] - J[4] * J[6]);
  const double sc = 1.0 / det;
  const double Ji[9] = {(J[4] * J[8] - J[5] * J[7]) * sc, (J[2] * J[7] - J[1] * J[8]) * sc,
                        (J[1] * J[5] - J[2] * J[4]) * sc, (J[6] * J[5] - J[3] * J[8]) * sc,
                        (J[0] * J[8] - J[2] * J[6]) * sc, (J[3] * J[2] - J[0] * J[5]) * sc,
                        (J[3] * J[7] - J[4] * J[6]) * sc, (J[1] * J[6] - J[0] * J[7]) * sc,
                        (J[0] * J[4] - J[1] * J[3]) * sc};
  for (int n = 0; n < 8; n++)
    for (int i = 0; i < 3; i++) {
      double v = 0.0;
      for (int j = 0; j < 3; j++) v += Ji[3 * i + j] * dN[3 * n + j];
      const dw p = dw_from_double(v);
      a.Gdf[(uint64_t)(3 * n + i) * E8 + t] = make_float2(p.h, p.l);
    }
  a.wdet[t] = 1.0 * det;
  const dw pw = dw_from_double(1.0 * det);
  a.wdf[t] = make_float2(pw.h, pw.l);
  // isoparametric.cpp:177 logs det < 1e-20; here it is an element status
  if (!(det >= 1.0e-20) && g == 0) flag_element(a.status, e + 1);
}

// K[s] = sum of its contributions in ascending contribution order (the
// reference's element-ascending accumulation order), starting from 0.
//
// The sums are FP64 adds, and on this part the FP64 pipe is the scarce unit:
// a warp pays for an add whenever any of its lanes needs one.  Slots have
// 1..8 contributions (a hexahedral mesh: 8 on a node's own diagonal, 4/2/1
// off it, 1 for every pressure coupling), so a warp of consecutive slots pays
// for 8 adds where its slots need ~2.2 on average.  Each block therefore
// first sorts its slots by contribution count (a counting sort in shared
// memory; which thread sums a slot does not change the slot's sum), so the
// warps see nearly uniform counts and stop adding at their own maximum.
// Up to kBatch loads of a slot are issued before the first add; the adds keep
// the ascending order, and 0 + c1 is taken as c1 with -0 turned into +0, so
// the result is bitwise the plain sequential loop's.
constexpr int kBatch = 8;
constexpr int kCountClasses = kBatch + 2;  // counts 0..kBatch, and more than kBatch
constexpr int kMaxGatherBlock = 1024;

__device__ __forceinline__ double plus_zero_sum(double x) {
  // 0.0 + x without an FP64 add: x, except -0.0 -> +0.0
  const long long b = __double_as_longlong(x);
  return __longlong_as_double(b == (long long)0x8000000000000000ull ? 0ll : b);
}

template <bool kIds>
__device__ __forceinline__ void gather_block(const uint64_t block, const uint64_t s_begin,
                                             const uint64_t n_slots,
                                             const uint32_t* __restrict__ ptr,
                                             const uint32_t* __restrict__ ids,
                                             const double* __restrict__ contrib,
                                             double* __restrict__ out) {
  __shared__ uint32_t s_beg[kMaxGatherBlock];
  __shared__ uint32_t s_end[kMaxGatherBlock];
  __shared__ uint16_t s_slot[kMaxGatherBlock];
  __shared__ uint32_t s_wcnt[kMaxGatherBlock / 32][kCountClasses];
  __shared__ uint32_t s_total[kCountClasses];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_warps = blockDim.x >> 5;
  const uint64_t base = s_begin + block * blockDim.x;
  const uint64_t s = base + tid;
  uint32_t b = 0, e = 0;
  if (s < n_slots) {
    b = __ldg(ptr + s);
    e = __ldg(ptr + s + 1);
  }
  s_beg[tid] = b;
  s_end[tid] = e;
  const uint32_t n = e - b;
  const int cls = n > (uint32_t)kBatch ? kBatch + 1 : (int)n;
  // rank within (warp, class), and per-warp class counts
  if (lane < kCountClasses) s_wcnt[warp][lane] = 0;
  __syncwarp();
  const unsigned same = __match_any_sync(0xFFFFFFFFu, cls);
  const uint32_t rank = __popc(same & ((1u << lane) - 1u));
  if (rank == 0) s_wcnt[warp][cls] = __popc(same);
  __syncthreads();
  // exclusive prefix over warps, per class (one thread per class)
  if (tid < kCountClasses) {
    uint32_t run = 0;
    for (int w = 0; w < n_warps; w++) {
      const uint32_t t = s_wcnt[w][tid];
      s_wcnt[w][tid] = run;
      run += t;
    }
    s_total[tid] = run;
  }
  __syncthreads();
  uint32_t pos = s_wcnt[warp][cls] + rank;
  for (int c = 0; c < cls; c++) pos += s_total[c];
  s_slot[pos] = (uint16_t)tid;
  __syncthreads();

  const int lt = s_slot[tid];
  const uint64_t slot = base + lt;
  const uint32_t sb = s_beg[lt], se = s_end[lt];
  const uint32_t sn = se - sb;
  unsigned nmax = __reduce_max_sync(0xFFFFFFFFu, slot < n_slots ? sn : 0u);
  if (slot >= n_slots) return;
  double x[kBatch];
#pragma unroll
  for (int j = 0; j < kBatch; j++) {
    x[j] = 0.0;
    if ((uint32_t)j < sn) x[j] = kIds ? __ldg(contrib + __ldg(ids + sb + j)) : __ldg(contrib + sb + j);
  }
  double v = plus_zero_sum(x[0]);
#pragma unroll
  for (int j = 1; j < kBatch; j++) {
    if ((unsigned)j >= nmax) break;  // warp-uniform
    const double t = v + x[j];
    v = (uint32_t)j < sn ? t : v;
  }
  for (uint32_t k = sb + kBatch; k < se; k++) v += kIds ? contrib[ids[k]] : contrib[k];
  out[slot] = v;
}

template <bool kIds>
__global__ void __launch_bounds__(kMaxGatherBlock)
    gather_sorted_kernel(const uint64_t s_begin, const uint64_t n_slots,
                         const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ ids,
                         const double* __restrict__ contrib, double* __restrict__ out,
                         const uint32_t* __restrict__ skip) {
  if (skip && *skip) return;  // the same word for every thread: a uniform exit
  gather_block<kIds>(blockIdx.x, s_begin, n_slots, ptr, ids, contrib, out);
}

// K and F in one launch, F's blocks after K's: a small model's assembly is as
// long as its launches (1,000 elements: 28.7 -> 27.8 us a call with this,
// one memset of the status instead of two, and the launch shape looked up once
// per device)
template <bool kIds>
__global__ void __launch_bounds__(kMaxGatherBlock)
    gather_pair_kernel(const GatherArgs k, const GatherArgs f, const uint32_t k_blocks) {
  if (blockIdx.x < k_blocks)
    gather_block<kIds>(blockIdx.x, k.s_begin, k.n_slots, k.ptr, k.ids, k.contrib, k.out);
  else
    gather_block<kIds>(blockIdx.x - k_blocks, f.s_begin, f.n_slots, f.ptr, f.ids, f.contrib, f.out);
}

// Sparse block products of the Newton iteration (FESolver.cpp:454-466):
// one thread per output entry walks its precomputed list in the reference's
// order; explicit _rn operations keep (K x) coef and the running sum from
// being fused, so each entry is the reference's value bit for bit (structural
// zeros, which the reference's symmetric product also visits, add +-0 there
// and are not visited here).  The walk is a chain of two dependent loads per
// entry: kMvBatch entries' indices, then their values and products, are in
// flight before the ordered adds.  A row of more than kMvLong entries (a
// rigid-body master couples to every slave) would still hold its warp for its
// length: the warp forms such rows' products together, kMvChunk entries of up
// to kMvRows rows at a time, and their own threads only add them (K(2) of a 9
// x 11 x 43 bar, 20,103 rows, the longest 360 entries: 108 -> 49 us).  The skip
// test and a coefficient of +-1 stay off the FP64 pipe; a skipped product is
// -0, which changes no sum.
constexpr int kMvBatch = 16;
constexpr uint32_t kMvLong = 96;
constexpr int kMvChunk = 64, kMvRows = 8, kMvThreads = 128;

// |x| > 1e-20 (false for a NaN), on the bits
__device__ __forceinline__ bool mv_counts(double x) {
  const long long v = __double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFll;
  return v > __double_as_longlong(1e-20) && v <= 0x7FF0000000000000ll;
}

__global__ void __launch_bounds__(kMvThreads) block_mv_kernel(const BlockMvArgs a) {
  __shared__ double prod[kMvThreads / 32][kMvRows][kMvChunk + 1];
  const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool in = r < a.n_out;
  double acc = in ? a.y[r] : 0.0;
  const uint32_t beg = in ? __ldg(a.ptr + r) : 0u, end = in ? __ldg(a.ptr + r + 1) : 0u;
  const int unit = a.coef == 1.0 ? 1 : a.coef == -1.0 ? -1 : 0;
  auto product = [&](double kv, double x) {
    const double p = __dmul_rn(kv, x);
    // (multiplying by +-1 rounds nothing; a NaN's sign is immaterial)
    const double q = unit == 1 ? p : unit == -1 ? -p : __dmul_rn(p, a.coef);
    return !a.sym || mv_counts(x) ? q : -0.0;
  };
  const bool is_long = end - beg > kMvLong;
  for (uint32_t k = beg; k < end && !is_long; k += kMvBatch) {
    uint32_t xi[kMvBatch], slot[kMvBatch];
#pragma unroll
    for (int u = 0; u < kMvBatch; u++) {
      xi[u] = k + u < end ? __ldg(a.xi + k + u) : 0u;
      slot[u] = k + u < end ? __ldg(a.slot + k + u) : 0u;
    }
    double x[kMvBatch], p[kMvBatch];
#pragma unroll
    for (int u = 0; u < kMvBatch; u++) {
      x[u] = k + u < end ? a.x[xi[u]] : 0.0;
      p[u] = k + u < end ? __ldg(a.K + slot[u]) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kMvBatch; u++) p[u] = product(p[u], x[u]);
#pragma unroll
    for (int u = 0; u < kMvBatch; u++)
      if (k + u < end) acc = __dadd_rn(acc, p[u]);
  }
  __syncwarp();
  for (uint32_t todo = __ballot_sync(0xFFFFFFFFu, is_long); todo;) {
    // the next kMvRows long rows of the warp
    uint32_t rb[kMvRows], re[kMvRows];
    int mine = -1;
    uint32_t longest = 0;
#pragma unroll
    for (int i = 0; i < kMvRows; i++) {
      const int l = todo ? __ffs(todo) - 1 : 0;
      rb[i] = __shfl_sync(0xFFFFFFFFu, beg, l);
      re[i] = __shfl_sync(0xFFFFFFFFu, end, l);
      if (!todo) re[i] = rb[i];
      else if (l == lane) mine = i;
      longest = max(longest, re[i] - rb[i]);
      todo &= todo - 1;
    }
    for (uint32_t o = 0; o < longest; o += kMvChunk) {
#pragma unroll
      for (int h = 0; h < kMvChunk / 32; h++) {
        uint32_t xi[kMvRows], slot[kMvRows];
        const uint32_t j = o + lane + 32 * h;
#pragma unroll
        for (int i = 0; i < kMvRows; i++) {
          xi[i] = rb[i] + j < re[i] ? __ldg(a.xi + rb[i] + j) : 0u;
          slot[i] = rb[i] + j < re[i] ? __ldg(a.slot + rb[i] + j) : 0u;
        }
        double x[kMvRows], p[kMvRows];
#pragma unroll
        for (int i = 0; i < kMvRows; i++) {
          x[i] = rb[i] + j < re[i] ? a.x[xi[i]] : 0.0;
          p[i] = rb[i] + j < re[i] ? __ldg(a.K + slot[i]) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < kMvRows; i++)
          prod[warp][i][lane + 32 * h] = rb[i] + j < re[i] ? product(p[i], x[i]) : -0.0;
      }
      __syncwarp();
      if (mine >= 0)
#pragma unroll 8
        for (int j = 0; j < kMvChunk; j++) acc = __dadd_rn(acc, prod[warp][mine][j]);
      __syncwarp();
    }
  }
  if (in) a.y[r] = acc;
}

__global__ void linear_mpc_kernel(const LinearMpcArgs a) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= a.n) return;
  a.F[a.eq[k] - 1] = a.b[k];
  for (uint32_t t = a.ptr[k]; t < a.ptr[k + 1]; t++) a.K[a.slot[t]] += a.coef[t];
}

// Rigid-body MPC rows (RigidBodyMpc::update, Mpc.cpp:70-164, and
// FEStorage.cpp:51-61): one thread per MPC equation.
__global__ void mpc_kernel(const MpcArgs a) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= a.n_mpc) return;
  const uint32_t* me = a.master_eq6 + (uint64_t)k * 6;
  const double w0[3] = {a.U[me[0] - 1], a.U[me[1] - 1], a.U[me[2] - 1]};
  const double th[3] = {a.U[me[3] - 1], a.U[me[4] - 1], a.U[me[5] - 1]};
  const double tn = sqrt(th[0] * th[0] + th[1] * th[1] + th[2] * th[2]);
  double c1, c2, c3, c4;
  if (tn < 1.0e-3) {
    c1 = 1.0;
    c2 = 0.5;
    c3 = -1.0 / 3.0;
    c4 = -1.0 / 12.0;
  } else {
    const double sn = sin(tn), cs = cos(tn);
    c1 = sn / tn;
    c2 = (1.0 - cs) / (tn * tn);
    c3 = (tn * cs - sn) / (tn * tn * tn);
    c4 = (tn * sn - 2.0 + 2.0 * cs) / (tn * tn * tn * tn);
  }
  // Levi-Civita e_{i m j} with the reference's table (solidmech.h:24-33)
  auto lc = [](int i, int m, int j) -> double {
    if (i == m || m == j || i == j) return 0.0;
    return ((i == 0 && m == 1 && j == 2) || (i == 1 && m == 2 && j == 0) ||
            (i == 2 && m == 0 && j == 1))
               ? 1.0
               : -1.0;
  };
  const int i = a.slave_dof[k];
  const double ct = cos(tn);
  double Crow[3];
  for (int j = 0; j < 3; j++) {
    const double tm = lc(i, 0, j) * th[0] + lc(i, 1, j) * th[1] + lc(i, 2, j) * th[2];
    Crow[j] = ct * (i == j ? 1.0 : 0.0) + c1 * tm + c2 * th[i] * th[j];
  }
  const double* mp = a.xyz + (uint64_t)(a.master[k] - 1) * 3;
  const double* sp = a.xyz + (uint64_t)(a.slave[k] - 1) * 3;
  const double pq[3] = {sp[0] - mp[0], sp[1] - mp[1], sp[2] - mp[2]};
  double cD[3][3];
  for (int j = 0; j < 3; j++)
    for (int l = 0; l < 3; l++) {
      const double Iij = i == j ? 1.0 : 0.0, Iil = i == l ? 1.0 : 0.0, Ijl = j == l ? 1.0 : 0.0;
      cD[j][l] = Iij * (-c1) * th[l] +
                 c3 * th[l] * (lc(i, 0, j) * th[0] + lc(i, 1, j) * th[1] + lc(i, 2, j) * th[2]) +
                 c1 * lc(i, l, j) + c4 * th[l] * th[i] * th[j] + c2 * (Iil * th[j] + th[i] * Ijl);
    }
  const double b = w0[i] + (Crow[0] - (i == 0)) * pq[0] + (Crow[1] - (i == 1)) * pq[1] +
                   (Crow[2] - (i == 2)) * pq[2] - a.U[a.slave_eq[k] - 1];
  const uint32_t* sl = a.slot + (uint64_t)k * 5;
  a.K[sl[0]] += 1.0;
  a.K[sl[1]] += -1.0;
  for (int l = 0; l < 3; l++)
    a.K[sl[2 + l]] += -(cD[0][l] * pq[0] + cD[1][l] * pq[1] + cD[2][l] * pq[2]);
  a.F[a.eq[k] - 1] = b;
}

// TETRA0 (TETRA0.cpp:18-78, 110-199) and QUADTH (QUADTH.cpp:22-49): one
// thread per element; contributions in Element::assembleK order.
__device__ double det4_lu(double* m) {
  double det = 1.0;
  for (int k = 0; k < 4; k++) {
    int p = k;
    double best = fabs(m[k * 4 + k]);
    for (int i = k + 1; i < 4; i++) {
      const double v = fabs(m[i * 4 + k]);
      if (v > best) {
        best = v;
        p = i;
      }
    }
    if (best == 0.0) return 0.0;
    if (p != k) {
      for (int j = 0; j < 4; j++) {
        const double t = m[k * 4 + j];
        m[k * 4 + j] = m[p * 4 + j];
        m[p * 4 + j] = t;
      }
      det = -det;
    }
    const double piv = m[k * 4 + k];
    det *= piv;
    for (int i = k + 1; i < 4; i++) {
      const double f = m[i * 4 + k] / piv;
      for (int j = k + 1; j < 4; j++) m[i * 4 + j] -= f * m[k * 4 + j];
    }
  }
  return det;
}

__global__ void linear_kernel(const LinearArgs a) {
  const uint32_t e = a.e_begin + blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.n_elems) return;
  const uint32_t* c = a.conn + (uint64_t)e * 4;
  double P[4][3];
  for (int n = 0; n < 4; n++)
    for (int d = 0; d < 3; d++) P[n][d] = a.xyz[(uint64_t)(c[n] - 1) * 3 + d];
  if (a.etype == 3) {
    double S[16];
    for (int n = 0; n < 4; n++) {
      S[n * 4 + 0] = 1.0;
      S[n * 4 + 1] = P[n][0];
      S[n * 4 + 2] = P[n][1];
      S[n * 4 + 3] = P[n][2];
    }
    const double vol = det4_lu(S) / 6.0;
    if (!(vol > 0.0)) flag_element(a.status, e + 1);
    const double Em = a.eparams[kEparamStride * (uint64_t)e];
    const double my = a.eparams[kEparamStride * (uint64_t)e + 1];
    const double Ac = Em / ((1. + my) * (1. - 2. * my));
    // C (6x6, makeC) as dense
    double Cm[6][6] = {};
    Cm[0][0] = Cm[1][1] = Cm[2][2] = (1. - my) * Ac;
    Cm[0][1] = Cm[1][0] = Cm[0][2] = Cm[2][0] = Cm[1][2] = Cm[2][1] = my * Ac;
    Cm[3][3] = Cm[4][4] = Cm[5][5] = (1. / 2. - my) * Ac;
    // makeB: b, c, d coefficients
    auto X = [&](int n, int d) { return P[n][d]; };
    const double x12 = X(0, 0) - X(1, 0), x13 = X(0, 0) - X(2, 0), x14 = X(0, 0) - X(3, 0);
    const double x23 = X(1, 0) - X(2, 0), x24 = X(1, 0) - X(3, 0), x34 = X(2, 0) - X(3, 0);
    const double y12 = X(0, 1) - X(1, 1), y13 = X(0, 1) - X(2, 1), y14 = X(0, 1) - X(3, 1);
    const double y23 = X(1, 1) - X(2, 1), y24 = X(1, 1) - X(3, 1), y34 = X(2, 1) - X(3, 1);
    const double z12 = X(0, 2) - X(1, 2), z13 = X(0, 2) - X(2, 2), z14 = X(0, 2) - X(3, 2);
    const double z23 = X(1, 2) - X(2, 2), z24 = X(1, 2) - X(3, 2), z34 = X(2, 2) - X(3, 2);
    const double x21 = -x12, x31 = -x13, x32 = -x23, x42 = -x24, x43 = -x34;
    const double y21 = -y12, y31 = -y13, y32 = -y23, y42 = -y24, y43 = -y34;
    const double z21 = -z12, z31 = -z13, z32 = -z23, z42 = -z24, z43 = -z34;
    const double bb[4] = {y42 * z32 - y32 * z42, y31 * z43 - y34 * z13, y24 * z14 - y14 * z24,
                          y13 * z21 - y12 * z31};
    const double cc[4] = {x32 * z42 - x42 * z32, x43 * z31 - x13 * z34, x14 * z24 - x24 * z14,
                          x21 * z13 - x31 * z12};
    const double dd[4] = {x42 * y32 - x32 * y42, x31 * y43 - x34 * y13, x24 * y14 - x14 * y24,
                          x13 * y21 - x12 * y31};
    const double Af = -1. / 6. / vol;
    double B[6][12] = {};
    for (int i = 0; i < 4; i++) {
      B[0][3 * i + 0] = bb[i] * Af;
      B[1][3 * i + 1] = cc[i] * Af;
      B[2][3 * i + 2] = dd[i] * Af;
      B[3][3 * i + 0] = cc[i] * Af;
      B[3][3 * i + 1] = bb[i] * Af;
      B[4][3 * i + 1] = dd[i] * Af;
      B[4][3 * i + 2] = cc[i] * Af;
      B[5][3 * i + 0] = dd[i] * Af;
      B[5][3 * i + 2] = bb[i] * Af;
    }
    int idx = 0;
    for (int r = 0; r < 12; r++)
      for (int col = r; col < 12; col++, idx++) {
        double v = 0.0;
        for (int k = 0; k < 6; k++) {
          double cb = 0.0;
          for (int l = 0; l < 6; l++) cb += Cm[k][l] * B[l][col];
          v += B[k][r] * cb;
        }
        const uint64_t i = (uint64_t)e * 78 + idx;
        a.contribK[a.kpos ? a.kpos[i] : i] = v * vol;
      }
  } else {
    // QUADTH: 2x2 Gauss (isoparametric.h:80-85), conduction k and volume flux
    // (QUADTH.cpp:22-49), capacity rho c for transient analysis (:51-67)
    const double* ep = a.eparams + kEparamStride * (uint64_t)e;
    const double kc = ep[0], vflux = ep[1], rho = ep[2], cap = ep[3];
    double Ke[10] = {}, Ce[10] = {}, Fe[4] = {};
    for (int g = 0; g < 4; g++) {
      const double r = (g & 1) ? kGaussA : -kGaussA;
      const double s = (g & 2) ? kGaussA : -kGaussA;
      const double dN[4][2] = {{-0.25 * (1.0 - s), -0.25 * (1.0 - r)},
                               {+0.25 * (1.0 - s), -0.25 * (1.0 + r)},
                               {+0.25 * (1.0 + s), +0.25 * (1.0 + r)},
                               {-0.25 * (1.0 + s), +0.25 * (1.0 - r)}};
      const double N[4] = {0.25 * (1.0 - r) * (1.0 - s), 0.25 * (1.0 + r) * (1.0 - s),
                           0.25 * (1.0 + r) * (1.0 + s), 0.25 * (1.0 - r) * (1.0 + s)};
      double J[2][2] = {};
      for (int n = 0; n < 4; n++)
        for (int i = 0; i < 2; i++)
          for (int j = 0; j < 2; j++) J[i][j] += dN[n][i] * P[n][j];
      const double det = J[0][0] * J[1][1] - J[0][1] * J[1][0];
      if (!(det >= 1.0e-20)) flag_element(a.status, e + 1);
      const double s1 = 1.0 / det;
      const double Ji[2][2] = {{J[1][1] * s1, -J[0][1] * s1}, {-J[1][0] * s1, J[0][0] * s1}};
      double G[4][2];
      for (int n = 0; n < 4; n++)
        for (int i = 0; i < 2; i++) G[n][i] = Ji[i][0] * dN[n][0] + Ji[i][1] * dN[n][1];
      const double w = 1.0 * det;
      int idx = 0;
      for (int i = 0; i < 4; i++)
        for (int j = i; j < 4; j++, idx++) {
          Ke[idx] += (G[i][0] * kc * G[j][0] + G[i][1] * kc * G[j][1]) * w;
          Ce[idx] = __dadd_rn(Ce[idx], __dmul_rn(N[i] * N[j] * rho * cap, w));
        }
      if (vflux != 0.0)
        for (int i = 0; i < 4; i++) Fe[i] = __dadd_rn(Fe[i], __dmul_rn(N[i], vflux * w));
    }
    for (int i = 0; i < 10; i++) {
      const uint64_t k = (uint64_t)e * 10 + i;
      a.contribK[a.kpos ? a.kpos[k] : k] = Ke[i];
      if (a.contribC) a.contribC[a.kpos ? a.kpos[k] : k] = Ce[i];
    }
    for (int i = 0; i < 4; i++) {
      const uint64_t k = (uint64_t)e * 4 + i;
      a.contribF[a.fpos ? a.fpos[k] : k] = Fe[i];
    }
  }
}

// SurfaceLINETH::buildK (QUADTH.cpp:86-121): 2-point Gauss on the line
// (isoparametric.h:47-50), w = det = length / 2 (isoparametric.cpp:12-26);
// flux: F += N flux w; convection: K += N N^T htc w and F += (N N^T htc w) T_env.
__global__ void line_kernel(const LineArgs a) {
  const uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= a.n_lines) return;
  const uint32_t na = a.conn[2 * (uint64_t)l], nb = a.conn[2 * (uint64_t)l + 1];
  double d2 = 0.0;
  for (int k = 0; k < 3; k++) {
    const double d = a.xyz[(uint64_t)(nb - 1) * 3 + k] - a.xyz[(uint64_t)(na - 1) * 3 + k];
    d2 += d * d;
  }
  const double det = sqrt(d2) * 0.5;
  if (!(det > 0.0)) flag_element(a.status, a.first_elem + l);
  const double* par = a.par + 4 * (uint64_t)l;
  const double htc = par[0], flux = par[1], t0 = par[2], t1 = par[3];
  double Ke[3] = {0.0, 0.0, 0.0}, Fe[2] = {0.0, 0.0};
  const double w = 1.0 * det;
  // the flux loop runs over both points before the convection loop, and F
  // takes each product separately (matBVprod, Mat.h), as the reference adds
  if (flux != 0.0)
    for (int g = 0; g < 2; g++) {
      const double r = g ? kGaussA : -kGaussA;
      const double N0 = 0.5 * (1.0 - r), N1 = 0.5 * (1.0 + r);
      Fe[0] = __dadd_rn(Fe[0], __dmul_rn(N0, flux * w));
      Fe[1] = __dadd_rn(Fe[1], __dmul_rn(N1, flux * w));
    }
  if (htc != 0.0)
    for (int g = 0; g < 2; g++) {
      const double r = g ? kGaussA : -kGaussA;
      const double N0 = 0.5 * (1.0 - r), N1 = 0.5 * (1.0 + r);
      const double k00 = N0 * N0 * htc * w, k01 = N0 * N1 * htc * w, k11 = N1 * N1 * htc * w;
      Ke[0] += k00;
      Ke[1] += k01;
      Ke[2] += k11;
      Fe[0] = __dadd_rn(Fe[0], __dmul_rn(k00, t0));
      Fe[0] = __dadd_rn(Fe[0], __dmul_rn(k01, t1));
      Fe[1] = __dadd_rn(Fe[1], __dmul_rn(k01, t0));
      Fe[1] = __dadd_rn(Fe[1], __dmul_rn(k11, t1));
    }
  for (int i = 0; i < 3; i++) {
    const uint64_t k = a.k_off + 3 * (uint64_t)l + i;
    a.contribK[a.kpos ? a.kpos[k] : k] = Ke[i];
  }
  for (int i = 0; i < 2; i++) {
    const uint64_t k = a.f_off + 2 * (uint64_t)l + i;
    a.contribF[a.fpos ? a.fpos[k] : k] = Fe[i];
  }
}

// FMA throughput probe: 8 independent chains per thread, enough warps per SM
// to cover the pipe latency; every result is folded into one store so the
// chains cannot be removed.
template <typename T>
__global__ void fma_probe_kernel(T* out, int iters, T a, T b) {
  T x[8];
#pragma unroll
  for (int k = 0; k < 8; k++) x[k] = (T)(threadIdx.x + k);
  for (int i = 0; i < iters; i++)
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = x[k] * a + b;
  T s = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) s += x[k];
  if (s == (T)-12345.0) out[0] = s;
}

// One ready flag per device: the table is uploaded once per device (a
// synchronous copy), under a lock so that threads on different devices
// neither race on the flags nor repeat the upload.
constexpr int kMaxTableDevices = 64;
std::atomic<bool> g_tables_ready[kMaxTableDevices];
std::mutex g_tables_mutex;

cudaError_t ensure_tables() {
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  if (dev < 0 || dev >= kMaxTableDevices) return cudaErrorInvalidDevice;
  if (g_tables_ready[dev].load(std::memory_order_acquire)) return cudaSuccess;
  std::lock_guard<std::mutex> lock(g_tables_mutex);
  if (g_tables_ready[dev].load(std::memory_order_relaxed)) return cudaSuccess;
  // assemble3's order of the entries (a, i, b, k) (SOLID81.h:62-74)
  int tpos[8][3][8][3];
  int t = 0;
  for (int i = 0; i < 8; i++)
    for (int di = 0; di < 3; di++)
      for (int j = i; j < 8; j++)
        for (int dj = 0; dj < 3; dj++) {
          if (i == j && dj < di) continue;
          tpos[i][di][j][dj] = t++;
        }
  // D[(i,k), a, b] -> assemble3 position (see c_dpos)
  uint16_t dp[kDpos];
  for (int a = 0; a < 8; a++)
    for (int i = 0; i < 3; i++)
      for (int k = i; k < 3; k++)
        for (int b = 0; b < 8; b++) {
          const int at = (a * 6 + hblock(i, k)) * 8 + b;
          if (a <= b) dp[at] = (uint16_t)tpos[a][i][b][k];
          else dp[at] = i == k ? (uint16_t)0xFFFF : (uint16_t)tpos[b][k][a][i];
        }
  err = cudaMemcpyToSymbol(c_dpos, dp, sizeof(dp));
  if (err == cudaSuccess) g_tables_ready[dev].store(true, std::memory_order_release);
  return err;
}

}  // namespace

size_t solid81_smem_bytes_wpb(bool mixed, int wpb) {
  return mixed ? kDposBytes + wpb * sizeof(MixedSmem) : kHead64Bytes + wpb * kFWarp * sizeof(double);
}

using Solid81Kernel = void (*)(Solid81Args);

Solid81Kernel solid81_fn(bool mixed, int wpb) {
  switch (wpb) {
    case 2: return mixed ? solid81_mixed_kernel<2> : solid81_fp64_kernel<2>;
    case 8: return mixed ? solid81_mixed_kernel<8> : solid81_fp64_kernel<8>;
    default: return mixed ? solid81_mixed_kernel<4> : solid81_fp64_kernel<4>;
  }
}

cudaError_t prepare_device_tables() { return ensure_tables(); }

namespace {
// resident blocks per SM of each kernel and shape, + 1 (0: not asked yet); per
// device, as the tables
std::atomic<int> g_blocks_per_sm[kMaxTableDevices][2][3];
}  // namespace

int solid81_max_blocks_per_sm(bool mixed, int wpb) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::atomic<int>* known = dev >= 0 && dev < kMaxTableDevices
                                ? &g_blocks_per_sm[dev][mixed][wpb == 2 ? 0 : wpb == 8 ? 2 : 1]
                                : nullptr;
  if (known)
    if (const int v = known->load(std::memory_order_acquire)) return v - 1;
  const void* fn = reinterpret_cast<const void*>(solid81_fn(mixed, wpb));
  const size_t smem = solid81_smem_bytes_wpb(mixed, wpb);
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return 0;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, wpb * 32, smem) != cudaSuccess)
    return 0;
  if (known) known->store(per_sm + 1, std::memory_order_release);
  return per_sm;
}

cudaError_t launch_solid81_shaped(const Solid81Args& a, bool mixed, Solid81Shape shape,
                                  cudaStream_t s) {
  if (a.n_elems <= a.e_begin) return cudaSuccess;  // empty element range
  const int wpb = (shape.warps_per_block == 2 || shape.warps_per_block == 8)
                      ? shape.warps_per_block : 4;
  cudaError_t err = ensure_tables();
  if (err != cudaSuccess) return err;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t smem = solid81_smem_bytes_wpb(mixed, wpb);
  const int max_per_sm = solid81_max_blocks_per_sm(mixed, wpb);
  if (max_per_sm < 1) return cudaErrorInvalidConfiguration;
  int per_sm = shape.blocks_per_sm;
  if (per_sm <= 0 || per_sm > max_per_sm) per_sm = max_per_sm;
  const uint64_t quads = ((uint64_t)a.n_elems + kEPW - 1) / kEPW - a.e_begin / kEPW;
  uint64_t blocks = (uint64_t)sms * per_sm;
  const uint64_t need = (quads + wpb - 1) / wpb;
  if (blocks > need) blocks = need;
  const dim3 grid((unsigned)blocks), block(wpb * 32);
  solid81_fn(mixed, wpb)<<<grid, block, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_solid81_jacobian(const JacobianArgs& a, cudaStream_t s) {
  const uint64_t n = (uint64_t)a.n_elems * 8;
  if (n == 0) return cudaSuccess;
  const int bs = 256;
  const unsigned blocks = (unsigned)((n + bs - 1) / bs);
  if (a.geo) solid81_geometry_kernel<<<blocks, bs, 0, s>>>(a);
  else solid81_jacobian_kernel<<<blocks, bs, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_solid81(const Solid81Args& a, bool mixed, int blocks_per_sm_hint,
                           cudaStream_t s) {
  Solid81Shape shape;
  shape.warps_per_block = kWarpsPerBlock;
  shape.blocks_per_sm = blocks_per_sm_hint;
  return launch_solid81_shaped(a, mixed, shape, s);
}

cudaError_t probe_fma_peak(bool fp64, double* flops) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  void* buf = nullptr;
  cudaError_t e = cudaMalloc(&buf, 16);
  if (e != cudaSuccess) return e;
  const int threads = 512, blocks = sms * 4;
  const int iters = fp64 ? 4096 : 65536;
  cudaEvent_t t0, t1;
  cudaEventCreate(&t0);
  cudaEventCreate(&t1);
  float best = 1e30f;
  for (int rep = 0; rep < 4; rep++) {
    cudaEventRecord(t0);
    if (fp64)
      fma_probe_kernel<double><<<blocks, threads>>>((double*)buf, iters, 0.999999, 1e-7);
    else
      fma_probe_kernel<float><<<blocks, threads>>>((float*)buf, iters, 0.9999f, 1e-7f);
    cudaEventRecord(t1);
    e = cudaEventSynchronize(t1);
    if (e != cudaSuccess) break;
    float ms = 0;
    cudaEventElapsedTime(&ms, t0, t1);
    if (rep > 0 && ms < best) best = ms;
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  cudaEventDestroy(t0);
  cudaEventDestroy(t1);
  cudaFree(buf);
  *flops = 2.0 * 8.0 * (double)iters * threads * blocks / (best * 1e-3);
  return e;
}

cudaError_t launch_gather_bs(const GatherArgs& a, int bs, cudaStream_t s) {
  if (a.n_slots <= a.s_begin) return cudaSuccess;
  if (bs != 128 && bs != 256 && bs != 512 && bs != 1024) bs = 256;
  gather_sorted_kernel<true><<<(unsigned)((a.n_slots - a.s_begin + bs - 1) / bs), bs, 0, s>>>(
      a.s_begin, a.n_slots, a.ptr, a.ids, a.contrib, a.out, a.skip);
  return cudaGetLastError();
}

cudaError_t launch_gather_pair(const GatherArgs& k, const GatherArgs& f, int bs, cudaStream_t s) {
  if (bs != 128 && bs != 256 && bs != 512 && bs != 1024) bs = 256;
  const uint64_t nk = k.n_slots > k.s_begin ? (k.n_slots - k.s_begin + bs - 1) / bs : 0;
  const uint64_t nf = f.n_slots > f.s_begin ? (f.n_slots - f.s_begin + bs - 1) / bs : 0;
  if (nk + nf == 0) return cudaSuccess;
  if (k.ids)
    gather_pair_kernel<true><<<(unsigned)(nk + nf), bs, 0, s>>>(k, f, (uint32_t)nk);
  else
    gather_pair_kernel<false><<<(unsigned)(nk + nf), bs, 0, s>>>(k, f, (uint32_t)nk);
  return cudaGetLastError();
}

cudaError_t launch_gather(const GatherArgs& a, cudaStream_t s) { return launch_gather_bs(a, 256, s); }

cudaError_t launch_segsum(const SegSumArgs& a, int bs, cudaStream_t s) {
  if (a.n_slots <= a.s_begin) return cudaSuccess;
  if (bs != 128 && bs != 256 && bs != 512 && bs != 1024) bs = 256;
  gather_sorted_kernel<false><<<(unsigned)((a.n_slots - a.s_begin + bs - 1) / bs), bs, 0, s>>>(
      a.s_begin, a.n_slots, a.ptr, nullptr, a.contrib, a.out, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_block_mv(const BlockMvArgs& a, cudaStream_t s) {
  if (a.n_out == 0) return cudaSuccess;
  const int bs = kMvThreads;
  block_mv_kernel<<<(unsigned)((a.n_out + bs - 1) / bs), bs, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_linear_mpc(const LinearMpcArgs& a, cudaStream_t s) {
  if (a.n == 0) return cudaSuccess;
  const int bs = 128;
  linear_mpc_kernel<<<(a.n + bs - 1) / bs, bs, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_mpc(const MpcArgs& a, cudaStream_t s) {
  if (a.n_mpc == 0) return cudaSuccess;
  const int bs = 128;
  mpc_kernel<<<(a.n_mpc + bs - 1) / bs, bs, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_lines(const LineArgs& a, cudaStream_t s) {
  if (a.n_lines == 0) return cudaSuccess;
  const int bs = 128;
  line_kernel<<<(a.n_lines + bs - 1) / bs, bs, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_linear(const LinearArgs& a, cudaStream_t s) {
  if (a.n_elems <= a.e_begin) return cudaSuccess;
  const int bs = 128;
  linear_kernel<<<(a.n_elems - a.e_begin + bs - 1) / bs, bs, 0, s>>>(a);
  return cudaGetLastError();
}

// PLANE41 algebra (PLANE41.cpp:29-101): with B = B_L + Omega B_omega (3x8),
//   Kuu += (2 B^T Dd B + B_omega^T S4 B_omega) w,  Kup += B^T Dp w,
//   Kpp -= w / k,  Qe += B^T S w,  Fp += (J - 1 - p/k) w,
// Dd and Dp the (XX, YY, XY) part of getDdDp_UP with C_zz = 1; K and F take
// -Qe, -Fp and the entries in ElementPLANE41::assembleK order (PLANE41.h:54-95).
//
// The FP64 pipe bounds it, so it runs the FP64 SOLID81 kernel's algebra (see
// solid81_fp64_kernel) in two dimensions, one thread per element: 2 x 2
// components (the third direction contributes its 1 to I1, I2 and C),
// the characters of the four Gauss points accumulated point by point, modes
// x, y, xy to nodes at the end.  Some 1,500 FP64 instructions per element
// where forming B, Dd B and every Kuu entry per Gauss point took about 2,900
// and spilled: 39,963 elements 277 -> 164 us (ncu, cold).  As there, F is formed
// in the global axes: with F from dx/dxi (4% faster) K_uu of an element sheared
// by 100 lost four digits.
struct Mode2 {
  double x, y, xy;
};

// o[mask of b] = sigma_x Mx + sigma_y My + sigma_x sigma_y Mxy / sqrt(3)
__device__ __forceinline__ void modes2_to_nodes(const Mode2& M, double o[4]) {
#pragma unroll
  for (int x = 0; x < 2; x++) {
    const double p = fma(x ? kGaussA : -kGaussA, M.xy, M.y), m = x ? M.x : -M.x;
    o[x] = m - p;
    o[x + 2] = m + p;
  }
}

__device__ __forceinline__ Mode2 corners_to_modes2(const double v[4]) {   // v by mask; not / 4
  const double d1 = __dsub_rn(v[1], v[0]), d3 = __dsub_rn(v[3], v[2]);
  const double e2 = __dsub_rn(v[2], v[0]), e3 = __dsub_rn(v[3], v[1]);
  return {__dadd_rn(d1, d3), __dadd_rn(e2, e3), __dsub_rn(d3, d1)};
}

// One warp per block: with some 210 registers an SM holds nine, and warps of
// 32 elements spread evenly over the SMs' FP64 pipes (in blocks of 128 the
// last of them ran alone: 131 -> 125 us a call).
constexpr int kPlaneThreads = 32;
__global__ void __launch_bounds__(kPlaneThreads) plane41_kernel(const Plane41Args a) {
  const uint32_t e = a.e_begin + blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.n_elems) return;
  const uint32_t* cn = a.conn + (uint64_t)e * 4;
  const uint32_t peq = a.p_eq[e];
  const double pc = a.U_cur[peq - 1];
  const double ps = a.have_state ? a.U_state[peq - 1] : 0.0;
  const double st = a.have_state ? 1.0 : 0.0;
  int mat_id = a.mat_id;
  const double* mc = a.mc;
  double kbulk = a.kbulk;
  if (a.elem_mesh) {
    const double* mm = a.mesh_mat + 8 * (uint64_t)a.elem_mesh[e];
    mat_id = (int)mm[0];
    mc = mm + 1;
    kbulk = mm[6];
  }
  // positions and displacements as modes
  Mode2 Xm[2], um[2];
  {
    double X[2][4], u[2][4] = {};
#pragma unroll
    for (int b = 0; b < 4; b++) {
      const uint64_t n = cn[hex_corner(b)] - 1;
#pragma unroll
      for (int i = 0; i < 2; i++) {
        X[i][b] = a.xyz[3 * n + i];
        if (a.have_state) u[i][b] = a.U_state[a.node_eq3[4 * n + i] - 1];
      }
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const Mode2 M = corners_to_modes2(X[i]), d = corners_to_modes2(u[i]);
      Xm[i] = {0.25 * M.x, 0.25 * M.y, 0.25 * M.xy};
      um[i] = {0.25 * d.x, 0.25 * d.y, 0.25 * d.xy};
    }
  }
  // sums over the Gauss points of chi_S A[ip][kq]: S = 0, 1 (xi), 2 (eta), 3.
  // Blocks (0,0), (0,1), (1,1); of an entry p = q only the characters without
  // coordinate p are read, and so for w F S and cof F
  double A00[3][4] = {}, A11[3][4] = {}, A01[4][4] = {};   // sym2 / 2 p + q
  double Pw[2][2][2] = {}, Cw[2][2][2] = {};               // [i][p]: S = 0 and the other coordinate
  double Kpp = 0.0, Fp = 0.0;
  bool bad = false;
  const double inv_kb = 1.0 / kbulk;
#pragma unroll 1
  for (int g = 0; g < 4; g++) {
    const double sx = (g & 1) ? kGaussA : -kGaussA, sy = (g & 2) ? kGaussA : -kGaussA;
    auto gradient = [&](const Mode2 m[2], double F[2][2]) {
#pragma unroll
      for (int i = 0; i < 2; i++) {
        F[i][0] = fma(sy, m[i].xy, m[i].x);
        F[i][1] = fma(sx, m[i].xy, m[i].y);
      }
    };
    double Xg[2][2], du[2][2], F[2][2];
    gradient(Xm, Xg);
    const double w = minor2(Xg[0][0], Xg[1][1], Xg[0][1], Xg[1][0]);
    if (!(w >= 1.0e-20)) bad = true;
    const double rw = 1.0 / w;
    // dxi_p/dX_i, and the metric
    const double Xi[2][2] = {{Xg[1][1] * rw, -Xg[1][0] * rw}, {-Xg[0][1] * rw, Xg[0][0] * rw}};   // [i][p]
    double G[3];
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int r = p; r < 2; r++) G[p + r] = Xi[0][p] * Xi[0][r] + Xi[1][p] * Xi[1][r];
    // F = I + O in the global axes (at rest exactly I)
    gradient(um, du);
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const double O = fma(du[i][1], Xi[k][1], du[i][0] * Xi[k][0]);
        F[i][k] = i == k ? 1.0 + O : O;
      }
    const double detF = minor2(F[0][0], F[1][1], F[0][1], F[1][0]);
    const double J = fabs(detF);
    if (!(J > 0.0 && isfinite(J))) bad = true;
    const double kw = inv_kb * w;
    Fp += fma(J - 1.0, w, -pc * kw);
    Kpp -= kw;
    const double rc = inv_cbrt(J), pp = rc * rc, pppp = pp * pp;
    const double id0 = pp * rc;
    const double id = copysign(fma(id0, fma(-J, id0, 1.0), id0), detF);   // 1 / det F
    // w cof F with the sign of J C^-1 (J = |det F|), a quarter of dN/dxi's factor
    const double ws = signbit(detF) ? -0.25 * w : 0.25 * w;
    double cof[2][2], V[2][2], FI[2][2], FA[2][2];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int p = 0; p < 2; p++) {
        // cof F = (F11 -F10; -F01 F00) by rows
        const double c = i == 0 ? fma(-F[1][0], Xi[1][p], F[1][1] * Xi[0][p])
                                : fma(F[0][0], Xi[1][p], -F[0][1] * Xi[0][p]);
        cof[i][p] = ws * c;
        V[i][p] = c * id;
        FI[i][p] = fma(F[i][1], Xi[1][p], F[i][0] * Xi[0][p]);
      }
    const double b00 = F[0][0] * F[0][0] + F[0][1] * F[0][1];
    const double b01 = F[0][0] * F[1][0] + F[0][1] * F[1][1];
    const double b11 = F[1][0] * F[1][0] + F[1][1] * F[1][1];
    const double tr = b00 + b11;
    const double I1 = tr + 1.0;
    const double I2 = fma(b00, b11, fma(-b01, b01, tr));
    const double t13 = (1.0 / 3.0) * I1, t23 = (2.0 / 3.0) * I2;
    // W derivatives at (I1 J^-2/3, I2 J^-4/3) (materials_hyperelastic.cpp:135-204)
    double a1, a2 = 0.0, a11 = 0.0;
    if (mat_id == 1) {
      a1 = 0.5 * mc[0];
    } else if (mat_id == 2) {
      const double d = I1 * pp - 3.0;
      a1 = mc[0] + 2 * mc[1] * d + 3 * mc[2] * d * d;
      a2 = mc[3];
      a11 = 2 * mc[1] + 6 * mc[2] * d;
    } else {
      a1 = mc[0];
      a2 = mc[1];
    }
    const double ww = 0.0625 * w;   // the two factors 1/4 of dN/dxi
    const double pj = pc * J, pJs = ps * J;
    const double ko1 = st * (2 * a1 * pp), ko2 = st * (2 * a2 * pppp);
    const double k11 = ww * (4.0 * a11 * pppp), k1 = (4.0 / 3.0) * a1 * pp,
                 k2 = (8.0 / 3.0) * a2 * pppp;
    const double h = -0.5 * ww * (2.0 * pj - k1 * I1 - k2 * I2);
    const double sI = 1.5 * ww * k2, hI = 0.5 * sI;
    const double wq = -0.25 * w;
    const double pk = wq * ko1, pb = wq * ko2, pv = wq * pJs;
    const double xk = -ww * k1, xb = -ww * k2, xv = 0.5 * ww * (pj - k1 * t13 - k2 * t23);
    const double chi[2] = {(g & 1) ? 1.0 : -1.0, (g & 2) ? 1.0 : -1.0};
    double X[2][2];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int p = 0; p < 2; p++) {
        FA[i][p] = fma(-t13, V[i][p], FI[i][p]);
        const double fc = i == 0 ? b00 * FI[0][p] + b01 * FI[1][p] : b01 * FI[0][p] + b11 * FI[1][p];
        const double FB = fma(-t23, V[i][p], fma(I1, FI[i][p], -fc));
        const double P = fma(pk, FA[i][p], fma(pb, FB, pv * V[i][p]));
        X[i][p] = fma(xk, FA[i][p], fma(xb, FB, xv * V[i][p]));
        Pw[i][p][0] += P;
        Pw[i][p][1] = fma(chi[1 - p], P, Pw[i][p][1]);
        Cw[i][p][0] += cof[i][p];
        Cw[i][p][1] = fma(chi[1 - p], cof[i][p], Cw[i][p][1]);
      }
    // S^{pq} = (ko1 + ko2 I1) g - ko2 C^{pq} + (p J - ko1 I1/3 - ko2 2 I2/3) C^-1
    const double eg = ww * (ko1 + ko2 * I1), ecc = -ww * ko2;
    const double ec = ww * (pJs - ko1 * t13 - ko2 * t23) + h;
    double E[3];
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int r = p; r < 2; r++) {
        const double CI = V[0][p] * V[0][r] + V[1][p] * V[1][r];
        const double CC = FI[0][p] * FI[0][r] + FI[1][p] * FI[1][r];
        E[p + r] = fma(ecc, CC, fma(ec, CI, eg * G[p + r]));
      }
    const bool biderman = __any_sync(__activemask(), a11 != 0.0);
    auto entry = [&](int i, int k, int p, int r, double base) {
      double v = fma(V[i][p], X[k][r], fma(X[i][p], V[k][r], base));
      v = fma(h * V[i][r], V[k][p], v);
      if (i == k) v = fma(hI * FI[i][p], FI[i][r], v);
      else v = fma(sI * FI[i][p], FI[k][r], fma(-hI * FI[i][r], FI[k][p], v));
      return biderman ? fma(k11 * FA[i][p], FA[k][r], v) : v;
    };
    auto add = [&](double acc[4], int p, int r, double v) {
      acc[0] += v;
      if (p == r) {
        acc[2 - p] = fma(chi[1 - p], v, acc[2 - p]);   // the other coordinate
      } else {
        acc[1] = fma(chi[0], v, acc[1]);
        acc[2] = fma(chi[1], v, acc[2]);
        acc[3] = fma(chi[0] * chi[1], v, acc[3]);
      }
    };
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int r = 0; r < 2; r++) {
        if (r >= p) {
          add(A00[p + r], p, r, entry(0, 0, p, r, fma(-hI * b00, G[p + r], E[p + r])));
          add(A11[p + r], p, r, entry(1, 1, p, r, fma(-hI * b11, G[p + r], E[p + r])));
        }
        add(A01[2 * p + r], p, r, entry(0, 1, p, r, -hI * b01 * G[p + r]));
      }
  }
  if (bad) flag_element(a.status, e + 1);
  const uint64_t kb = (uint64_t)e * 45, fb = (uint64_t)e * 9;
  auto kd = [&](uint64_t i) { return a.kpos ? (uint64_t)a.kpos[i] : i; };
  auto fd = [&](uint64_t i) { return a.fpos ? (uint64_t)a.fpos[i] : i; };
  // position of (i, di; j, dj), i <= j, in assembleK order
  auto pos = [](int i, int di, int j, int dj) {
    int t = 0;
    for (int q = 0; q < i; q++) t += 3 + 4 * (3 - q);
    if (i == j) return t + di * (di + 1) / 2 + dj;   // (0,0) (1,0) (1,1)
    return t + 3 + 4 * (j - i - 1) + 2 * di + dj;
  };
  // block (i, k): modes of both sides to nodes; W(p, r) its four characters
  auto block = [&](const double (*W)[4], bool sym, double K[4][4]) {
    auto at = [&](int p, int r, int S) { return W[sym ? p + r : 2 * p + r][S]; };
    double T[3][4];
    // one mode of the a side: x = (0, 0), y = (1, 0), xy = (0, {1}) + (1, {0});
    // the characters of the two sides multiply (S: xi = 1, eta = 2)
    auto row = [&](int p, int P, Mode2& M) {
      M.x = at(p, 0, P);
      M.y = at(p, 1, P);
      M.xy = at(p, 0, P ^ 2) + at(p, 1, P ^ 1);
    };
    Mode2 M, M2;
    row(0, 0, M);
    modes2_to_nodes(M, T[0]);
    row(1, 0, M);
    modes2_to_nodes(M, T[1]);
    row(0, 2, M);
    row(1, 1, M2);
    M = {M.x + M2.x, M.y + M2.y, M.xy + M2.xy};
    modes2_to_nodes(M, T[2]);
#pragma unroll
    for (int b = 0; b < 4; b++) {
      double o[4];
      modes2_to_nodes(Mode2{T[0][b], T[1][b], T[2][b]}, o);
#pragma unroll
      for (int c = 0; c < 4; c++) K[hex_corner(c)][hex_corner(b)] = o[c];
    }
  };
  double K[4][4];
#pragma unroll
  for (int d = 0; d < 2; d++) {
    block(d == 0 ? A00 : A11, true, K);
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = i; j < 4; j++) a.contribK[kd(kb + pos(i, d, j, d))] = K[i][j];
  }
  block(A01, false, K);
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = i; j < 4; j++) {
      if (i != j) a.contribK[kd(kb + pos(i, 0, j, 1))] = K[i][j];
      a.contribK[kd(kb + pos(i, 1, j, 0))] = K[j][i];
    }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    double o[4];
    modes2_to_nodes(Mode2{Cw[i][0][0], Cw[i][1][0], Cw[i][0][1] + Cw[i][1][1]}, o);
#pragma unroll
    for (int b = 0; b < 4; b++) a.contribK[kd(kb + 36 + 2 * hex_corner(b) + i)] = o[b];
    modes2_to_nodes(Mode2{Pw[i][0][0], Pw[i][1][0], Pw[i][0][1] + Pw[i][1][1]}, o);
#pragma unroll
    for (int b = 0; b < 4; b++) a.contribF[fd(fb + 2 * hex_corner(b) + i)] = o[b];
  }
  a.contribK[kd(kb + 44)] = Kpp;
  a.contribF[fd(fb + 8)] = -Fp;
}

cudaError_t launch_plane41(const Plane41Args& a, cudaStream_t s) {
  if (a.n_elems <= a.e_begin) return cudaSuccess;
  const int bs = kPlaneThreads;
  plane41_kernel<<<(a.n_elems - a.e_begin + bs - 1) / bs, bs, 0, s>>>(a);
  return cudaGetLastError();
}

__global__ void slot_last_range_kernel(uint64_t n_slots, const uint32_t* ptr, const uint32_t* ids,
                                       uint32_t n_kc, const uint32_t* eb, int n, uint8_t* out) {
  const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n_slots) return;
  const uint32_t b = ptr[s], e = ptr[s + 1];
  int r = 0;
  if (e > b) {
    const uint32_t el = ids[e - 1] / n_kc;  // ids ascend within a slot
    while (r + 1 < n && el >= eb[r + 1]) r++;
  }
  out[s] = (uint8_t)r;
}

cudaError_t launch_slot_last_range(uint64_t n_slots, const uint32_t* ptr, const uint32_t* ids,
                                   uint32_t n_kc, const uint32_t* eb, int n, uint8_t* out,
                                   cudaStream_t s) {
  if (n_slots == 0) return cudaSuccess;
  const int bs = 256;
  slot_last_range_kernel<<<(unsigned)((n_slots + bs - 1) / bs), bs, 0, s>>>(n_slots, ptr, ids,
                                                                          n_kc, eb, n, out);
  return cudaGetLastError();
}

}  // namespace nla3d_gpu
