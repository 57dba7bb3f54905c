// The K2 + Kf integrand of the BK right-hand side in its cancellation-free form, shared by
// the quasi-Monte Carlo kernel (k2kf.cu) and the Vegas kernel (k2kf_vegas.cu):
// _nlo_integrand x exp(2 log z + 2 log z') of bk/derivatives.py:322-335 and 490-612, with
// the kernels of bk_kernels/k2.py:8-39 and bk_kernels/kf.py:10-41.  A sample's
// parent-independent quantities (z, z', |z - z'|, their amplitudes, the Jacobian) form a
// record (k2_prepare*); k2_point evaluates one (record, parent) pair, k2_pair_fast two in FP32.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "common.cuh"
#include "sobol.cuh"

namespace nlo {
namespace k2 {

// Per-sample record (r-independent), 20 values.
enum Rec {
    kZ, kZ2, kS1, kS2, kP1, kP2, kU1, kV1, kU2, kV2,
    kQ, kD1, kD2, kDN, kSY, kLmin, kCpt, kDl, kZsq, kZ2sq,
    kRecLen
};

template <typename T>
struct alignas(16) K2Rec {
    T v[kRecLen];
};

template <typename T>
struct K2Box {
    T lower[4], width[4];
    T cpt_scale;  // volume * Nc^2 / (8 pi^4)
};

// atanh(t)/t - 1 = t^2 g(t^2), g(x) = sum_{k>=0} x^k/(2k+3), for t^2 < 1/4: the series in
// FP64; the FP32 pair path (k2_pair_fast) evaluates g by a degree-6 polynomial fitted on
// [0, 1/4] in relative error (least squares at Chebyshev nodes; 8e-8 relative in FP32
// Horner, i.e. FP32 rounding).
template <typename T>
__device__ __forceinline__ T atanh_ratio_m1(T t2);

template <>
__device__ __forceinline__ double atanh_ratio_m1<double>(double t2)
{
    double s = 0.0;
#pragma unroll
    for (int k = 30; k >= 1; --k) s = fma(s, t2, 1.0 / (2.0 * k + 1.0));
    return s * t2;
}

template <>
__device__ __forceinline__ float atanh_ratio_m1<float>(float t2)
{
    float g = fmaf(0.15609439065092748f, t2, 0.04106302733766397f);
    g = fmaf(g, t2, 0.09747851219255123f);
    g = fmaf(g, t2, 0.11051354325642386f);
    g = fmaf(g, t2, 0.1428825580061165f);
    g = fmaf(g, t2, 0.19999959971627077f);
    g = fmaf(g, t2, 0.33333333435159396f);
    return g * t2;
}

// The parent-independent record of one sample at box coordinates x = (log z, log z',
// theta_z, theta_z'); `valid` false gives a record of zero weight.
template <typename T>
__device__ __forceinline__ void k2_prepare_x(const SplineView<T>& s, const K2Box<T>& box, const T* x, bool valid,
                                             T* rec)
{
    const T lz = x[0], lz2 = x[1], th = x[2], th2 = x[3];
    const T z = M<T>::exp_acc(lz), z2 = M<T>::exp_acc(lz2);
    const T sh1 = M<T>::sin((T)0.5 * th), sh2 = M<T>::sin((T)0.5 * th2);
    const T c1 = M<T>::cos(th), c2 = M<T>::cos(th2);
    const T dth = th - th2;
    const T c12 = M<T>::cos(dth), sh12 = M<T>::sin((T)0.5 * dth);
    const T zzsq = (z - z2) * (z - z2) + (T)4 * z * z2 * sh12 * sh12;
    valid = valid && zzsq >= M<T>::tiny_square();
    const T lzz = (T)0.5 * M<T>::log_acc(zzsq);
    const NS<T> Y = eval_s_log(s, lz), Y2 = eval_s_log(s, lz2), ZZ = eval_s_log(s, lzz);
    const T dN = ndiff_s(Y2, Y);  // N_Y2 - N_Y
    rec[kZ] = z;
    rec[kZ2] = z2;
    rec[kS1] = z * (sh1 * sh1);  // z sin^2(theta/2): X^2 = (r - z)^2 + 4 r rec[kS1]
    rec[kS2] = z2 * (sh2 * sh2);
    rec[kP1] = (z2 - z) * (z2 + z);
    rec[kP2] = (T)2 * z * z2 * (z2 * c1 - z * c2);
    rec[kU1] = z2 - z * c12;
    rec[kV1] = z * (z * c2 - z2 * c1);
    rec[kU2] = z - z2 * c12;
    rec[kV2] = z2 * (z2 * c1 - z * c2);
    rec[kQ] = valid ? M<T>::rcp(zzsq) : (T)0;
    // S_Y - S_zz S_Y2 = S_Y N_zz + S_zz (N_Y2 - N_Y);  S_Y2 - S_zz S_Y = S_Y2 N_zz - S_zz (N_Y2 - N_Y)
    rec[kD1] = Y.S * ZZ.N + ZZ.S * dN;
    rec[kD2] = Y2.S * ZZ.N - ZZ.S * dN;
    rec[kDN] = dN;
    rec[kSY] = Y.S;
    rec[kLmin] = M<T>::fmin(M<T>::fmin(lz, lz2), lzz);
    rec[kCpt] = valid ? box.cpt_scale * M<T>::exp_acc((T)2 * lz + (T)2 * lz2) : (T)0;
    rec[kDl] = (T)2 * (lz2 - lz);
    rec[kZsq] = z * z;
    rec[kZ2sq] = z2 * z2;
}

template <typename T>
struct K2Parent {
    T r, r2, lr, two_r;
    T alpha_r;  // the RC_NLO = PARENT_NLO coupling
};

// K2 and Kf contributions of one sample to one parent (already weighted).
template <typename T, bool SYM, typename EvalSpline>
__device__ __forceinline__ void k2_point(const EvalSpline& s, const Phys<T>& ph, const K2Parent<T>& P,
                                         const T* __restrict__ rec, T& k2w, T& kfw)
{
    const T r = P.r;
    const T z = rec[kZ], z2 = rec[kZ2];
    const T Xsq = (r - z) * (r - z) + (T)4 * r * rec[kS1];
    const T X2sq = (r - z2) * (r - z2) + (T)4 * r * rec[kS2];
    const bool valid = Xsq >= M<T>::tiny_square() && X2sq >= M<T>::tiny_square();
    const T lXs = M<T>::log_fast(Xsq), lX2s = M<T>::log_fast(X2sq);
    const PS<T> vX = eval_s_ps(s, (T)0.5 * lXs), vX2 = eval_s_ps(s, (T)0.5 * lX2s);
    // kernels (k2.py, kf.py) in the stable form
    const T a = Xsq * rec[kZ2sq], b = X2sq * rec[kZsq];
    const T sab = a + b;
    const T rs = M<T>::rcp(sab);
    const T d = r * (r * rec[kP1] - rec[kP2]);
    const T t = d * rs;
    const T t2 = t * t;
    T hm1, Ld;
    if (t2 < (T)0.25) {
        hm1 = atanh_ratio_m1<T>(t2);
        Ld = (T)2 * t * ((T)1 + hm1);
    } else {
        Ld = lXs - lX2s + rec[kDl];  // log(a/b)
        hm1 = M<T>::div(Ld, (T)2 * t) - (T)1;
    }
    const T q = rec[kQ];
    const T L = (T)2 * ((T)1 + hm1) * rs;
    const T f = (T)2 * hm1;
    const T fq2 = f * q * q;
    const T r2Lq = P.r2 * L * q;
    const T C0 = fq2 - (T)4 * r2Lq;
    // L r^4/a + log(a/b) r^2 q/a = L r^2 q 2 r B1/(X^2 z'), B1 = r (z' - z c12) + z (z c2 - z' c1)
    const T B1 = r * rec[kU1] + rec[kV1];
    const T B2 = r * rec[kU2] + rec[kV2];
    T k2 = C0 + r2Lq * P.two_r * B1 * M<T>::rcp(Xsq * z2);
    T k2s = C0 + r2Lq * P.two_r * B2 * M<T>::rcp(X2sq * z);
    const T kf = (r2Lq - fq2) * ph.nf_over_nc;
    T dip = vX.S * rec[kD1];
    T dips = vX2.S * rec[kD2];
    if (M<T>::fabs(k2) > (T)1e10 && M<T>::fabs(dip) < (T)1e-10) { k2 = (T)0; dip = (T)0; }
    if (M<T>::fabs(k2s) > (T)1e10 && M<T>::fabs(dips) < (T)1e-10) { k2s = (T)0; dips = (T)0; }
    const T dNX = ndiff_ps(vX, vX2);
    T k2part, fermion;
    if (SYM) {
        k2part = (T)0.5 * (k2 * dip + k2s * dips);
        fermion = (T)0.5 * kf * dNX * rec[kDN];
    } else {
        k2part = k2 * dip;
        fermion = kf * rec[kSY] * dNX;
    }
    if (!(ph.nf > (T)0)) fermion = (T)0;
    const T lmin = M<T>::fmin(M<T>::fmin(rec[kLmin], P.lr), (T)0.5 * M<T>::fmin(lXs, lX2s));
    // _nlo_alpha_s (bk/derivatives.py:615-632): the smallest of the six sizes, or the parent
    const T alpha = ph.nlo_parent ? P.alpha_r : alpha_of_log(lmin, ph);
    const T scale = alpha * alpha * rec[kCpt];
    k2w = k2part * scale;
    kfw = -fermion * scale;
    if (!valid || !M<T>::finite(k2w)) k2w = (T)0;
    if (!valid || !M<T>::finite(kfw)) kfw = (T)0;
}

// The record of Sobol point `index` mapped into the box (explicitly rounded operations, as
// the oracle replays them).
template <typename T>
__device__ __forceinline__ void k2_prepare(const SplineView<T>& s, const K2Box<T>& box, const uint32_t* state,
                                           const uint32_t* shift, uint64_t index, bool valid, T* rec)
{
    T x[4];
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        const T u = sobol_unit<T>(sobol_bits(state + 30 * d, shift[d], index), index);
        x[d] = M<T>::add_rn(box.lower[d], M<T>::mul_rn(box.width[d], u));
    }
    k2_prepare_x<T>(s, box, x, valid, rec);
}

// ---------------------------------------------------------------------------
// FP32 evaluation tuned for instruction count (the kernel is issue-bound).
// Spline values are carried in log2 units; the log S coefficients are stored
// pre-scaled to the unit interval, (a, b h, c h^2, d h^3) * log2(e), so that the
// position u = (log X - x0)/h gives the piece i = floor(u) and t = u - i directly.
// Amplitudes outside the grid are encoded as p2 = 0 (S = 1, below r_min) and
// p2 = -150 (S = 0, above r_max), which lets one branch-free difference formula
// serve every case:  N_A - N_B = S_A (2^(pB-pA) - 1) if pB <= pA, else -S_B (2^(pA-pB) - 1).
__device__ __forceinline__ float ex2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_approx(float x)
{
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_approx(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

struct FastSpline {
    // [n + 1] pre-scaled rows (see above): row 0 is (0, 0, 0, 0), the value below r_min
    // (log2 S = 0, S = 1); rows 1..n-1 are the intervals; row n is (-150, 0, 0, 0), above
    // r_max (S = 0)
    const float4* coef;
    float u_scale;  // (ln 2 / 2) / h : u from log2(X^2)
    float u_off;    // -x0 / h
    float u_top;    // n - 1
};

// The same rows for Vegas, whose grids gather the samples where the integrand cancels: what the
// roundings of the position constants leave out, and the pair for a position from log X itself.
struct FineSpline : FastSpline {
    float u_scale_lo, u_off_lo;
    float l_scale, l_scale_lo;  // 1 / h
};

struct P2S {
    float p2, S;
};

struct K2ParentF {
    float r, r2, lr, two_r, four_r;
    float alpha_r;  // the RC_NLO = PARENT_NLO coupling
};

// COUPLING: 0 smooth freeze, 1 smooth freeze capped at alpha_cap, 2 fixed, 3 any coupling
// of alpha_of_log (flavour thresholds), 4 the parent's coupling (RC_NLO = PARENT_NLO).

// Spline position u = (log X - x0)/h -> (log2 S, S) for a pair of positions.  u is clamped
// to [-1, n-1]; the row floor(u) + 1 of the table with its two edge rows serves every case
// (below the grid, inside, above), so there is no edge select.  floor(u) + 1 comes without
// the XU conversions: u + (2^23 + 1) rounded down holds it in the low mantissa bits.  The
// clamp, floor and fraction run on the packed instructions, the table lookup and the cubic
// per component.
__device__ __forceinline__ void fast_amplitude_pair(const FastSpline& s, f2 u, P2S& ax, P2S& ay)
{
    const f2 uc = make_float2(fminf(fmaxf(u.x, -1.0f), s.u_top), fminf(fmaxf(u.y, -1.0f), s.u_top));
    const f2 shifted = __fadd2_rd(uc, bc2(8388609.0f));  // 2^23 + 1 + floor(uc)
    const f2 t = sub2(uc, sub2(shifted, bc2(8388609.0f)));
    const float4 cx = s.coef[__float_as_int(shifted.x) - 0x4B000000];
    const float4 cy = s.coef[__float_as_int(shifted.y) - 0x4B000000];
    const float px = fmaf(t.x, fmaf(t.x, fmaf(t.x, cx.w, cx.z), cx.y), cx.x);
    const float py = fmaf(t.y, fmaf(t.y, fmaf(t.y, cy.w, cy.z), cy.y), cy.x);
    ax = {px, ex2_approx(px)};
    ay = {py, ex2_approx(py)};
}

// The pair of amplitudes at L = log2(X^2) (scale u_scale) or log X (scale l_scale).  The row comes
// from the rounded position; the fraction t = L scale + offset - row is formed anew from the
// two-part constants: offset - row is exact, the fused product cancels against it with one
// rounding of t, so t is good to 1e-7 where u - floor(u) carries the rounding of u and of both
// constants (1e-5 at u ~ 100, which was the larger part of the FP32 error of Vegas K2+Kf).
__device__ __forceinline__ void fine_amplitude_pair(const FineSpline& s, f2 L, float scale, float scale_lo, P2S& ax,
                                                    P2S& ay)
{
    const float lo = -0.5f, hi = s.u_top + 0.5f;  // below the grid and above it: the edge rows
    const f2 u = fma2(L, bc2(scale), bc2(s.u_off));
    const f2 uc = make_float2(fminf(fmaxf(u.x, lo), hi), fminf(fmaxf(u.y, lo), hi));
    // an L out of range (infinite for X = 0) meets a row without slopes: any finite t will do
    const f2 Lc = make_float2(u.x > lo && u.x < hi ? L.x : 0.0f, u.y > lo && u.y < hi ? L.y : 0.0f);
    const f2 shifted = __fadd2_rd(uc, bc2(8388609.0f));  // 2^23 + 1 + floor(uc)
    const f2 a = sub2(bc2(s.u_off), sub2(shifted, bc2(8388609.0f)));
    const f2 t = add2(fma2(Lc, bc2(scale), a), fma2(Lc, bc2(scale_lo), bc2(s.u_off_lo)));
    const float4 cx = s.coef[__float_as_int(shifted.x) - 0x4B000000];
    const float4 cy = s.coef[__float_as_int(shifted.y) - 0x4B000000];
    const float px = fmaf(t.x, fmaf(t.x, fmaf(t.x, cx.w, cx.z), cx.y), cx.x);
    const float py = fmaf(t.y, fmaf(t.y, fmaf(t.y, cy.w, cy.z), cy.y), cy.x);
    ax = {px, ex2_approx(px)};
    ay = {py, ex2_approx(py)};
}

// ---------------------------------------------------------------------------
// Two samples per call on the packed FP32x2 pipe of sm_100 (FFMA2/FADD2/FMUL2): the
// per-evaluation arithmetic of k2_point_fast, component x for sample 2p and y for 2p+1
// of a pair record (every field of the two samples side by side), so each packed
// instruction does the work of two.  MUFU operations, compares and selects stay scalar.
__device__ __forceinline__ f2 rcp2(f2 a) { return make_float2(rcp_approx(a.x), rcp_approx(a.y)); }
__device__ __forceinline__ f2 lg22(f2 a) { return make_float2(lg2_approx(a.x), lg2_approx(a.y)); }
__device__ __forceinline__ f2 sel2(bool cx, bool cy, f2 a, f2 b) { return make_float2(cx ? a.x : b.x, cy ? a.y : b.y); }

// N_A - N_B from log2 S values, for a pair
__device__ __forceinline__ f2 fast_ndiff2(const P2S& Ax, const P2S& Ay, const P2S& Bx, const P2S& By)
{
    // N_A - N_B = S_B - S_A.  Near each other (|pB - pA| < 1/2 in log2 units) it is
    // S_A (2^(pB-pA) - 1) or -S_B (2^(pA-pB) - 1) with 2^x - 1 = x q(x), q a degree-5
    // polynomial fitted to (2^x - 1)/x on [-1/2, 0] (1.2e-7 relative in FP32); farther
    // apart the plain difference S_B - S_A has no cancellation (the ratio is at least
    // sqrt(2)), and both S are at hand.
    const f2 d = make_float2(Bx.p2 - Ax.p2, By.p2 - Ay.p2);
    const f2 x = make_float2(-fabsf(d.x), -fabsf(d.y));
    f2 q = fma2(bc2(0.0001327910803141678f), x, bc2(0.001321632968973654f));
    q = fma2(q, x, bc2(0.009615099576281485f));
    q = fma2(q, x, bc2(0.05550375169709732f));
    q = fma2(q, x, bc2(0.24022649146109623f));
    q = fma2(q, x, bc2(0.6931471804499034f));
    const f2 S = make_float2(d.x <= 0.0f ? Ax.S : -Bx.S, d.y <= 0.0f ? Ay.S : -By.S);
    const f2 near = mul2(S, mul2(q, x));
    const f2 far = make_float2(Bx.S - Ax.S, By.S - Ay.S);
    return make_float2(x.x > -0.5f ? near.x : far.x, x.y > -0.5f ? near.y : far.y);
}

// Kf and K2 + Kf of the pair, each 0 where the sum is not finite; with a FineSpline (Vegas) Kf and
// K2, each 0 where it is not finite, for the caller to add in FP64.
template <bool SYM, int COUPLING, class Spline>
__device__ __forceinline__ void k2_pair_fast(const Spline& s, const Phys<float>& ph, const K2ParentF& P,
                                             const float4* __restrict__ rec4, f2& kfw, f2& total)
{
    constexpr bool FINE = std::is_same<Spline, FineSpline>::value;
    constexpr float LN2 = 0.69314718055994531f;
    constexpr float L2E = 1.4426950408889634f;
    // pair layout: float4 k holds fields 2k and 2k+1 of (sample x, sample y)
    const float4 w0 = rec4[0], w1 = rec4[1], w2 = rec4[2], w3 = rec4[3], w4 = rec4[4];
    const float4 w5 = rec4[5], w6 = rec4[6], w7 = rec4[7], w8 = rec4[8], w9 = rec4[9];
    const f2 z = make_float2(w0.x, w0.y), z2 = make_float2(w0.z, w0.w);
    const f2 s1 = make_float2(w1.x, w1.y), s2 = make_float2(w1.z, w1.w);
    const f2 P1 = make_float2(w2.x, w2.y), P2 = make_float2(w2.z, w2.w);
    const f2 U1 = make_float2(w3.x, w3.y), V1 = make_float2(w3.z, w3.w);
    const f2 U2 = make_float2(w4.x, w4.y), V2 = make_float2(w4.z, w4.w);
    const f2 q = make_float2(w5.x, w5.y), D1 = make_float2(w5.z, w5.w);
    const f2 D2 = make_float2(w6.x, w6.y), dN = make_float2(w6.z, w6.w);
    const f2 SY = make_float2(w7.x, w7.y), Lmin = make_float2(w7.z, w7.w);
    const f2 cpt = make_float2(w8.x, w8.y), Dl = make_float2(w8.z, w8.w);
    const f2 zsq = make_float2(w9.x, w9.y), z2sq = make_float2(w9.z, w9.w);
    const f2 r = bc2(P.r);
    const f2 rz = sub2(r, z), rz2 = sub2(r, z2);
    const f2 Xsq = fma2(bc2(P.four_r), s1, mul2(rz, rz));  // s1 = z sin^2(theta/2)
    const f2 X2sq = fma2(bc2(P.four_r), s2, mul2(rz2, rz2));
    const f2 L2X = lg22(Xsq), L2X2 = lg22(X2sq);
    P2S vXx, vXy, vX2x, vX2y;
    if constexpr (FINE) {
        fine_amplitude_pair(s, L2X, s.u_scale, s.u_scale_lo, vXx, vXy);
        fine_amplitude_pair(s, L2X2, s.u_scale, s.u_scale_lo, vX2x, vX2y);
    } else {
        const f2 uX = fma2(L2X, bc2(s.u_scale), bc2(s.u_off)), uX2 = fma2(L2X2, bc2(s.u_scale), bc2(s.u_off));
        fast_amplitude_pair(s, uX, vXx, vXy);
        fast_amplitude_pair(s, uX2, vX2x, vX2y);
    }
    // kernels
    // log(a/b)/(a - b) = 2 (1 + hm1)/(a + b), hm1 = atanh(t)/t - 1, t = (a - b)/(a + b): the series
    // in t^2 where |a - b| < (a + b)/2, else log(a/b) directly; each case needs one reciprocal,
    // of a + b or of a - b, and the test needs none
    const f2 a = mul2(Xsq, z2sq), b = mul2(X2sq, zsq);
    const f2 sab = add2(a, b);
    const f2 d = mul2(r, fma2(r, P1, make_float2(-P2.x, -P2.y)));  // a - b
    const bool ser_x = fabsf(d.x) < 0.5f * sab.x, ser_y = fabsf(d.y) < 0.5f * sab.y;
    const f2 rden = rcp2(sel2(ser_x, ser_y, sab, d));
    const f2 t = mul2(d, rden);
    const f2 t2 = mul2(t, t);
    f2 g = fma2(bc2(0.15609439065092748f), t2, bc2(0.04106302733766397f));
    g = fma2(g, t2, bc2(0.09747851219255123f));
    g = fma2(g, t2, bc2(0.11051354325642386f));
    g = fma2(g, t2, bc2(0.1428825580061165f));
    g = fma2(g, t2, bc2(0.19999959971627077f));
    g = fma2(g, t2, bc2(0.33333333435159396f));
    const f2 hm1_series = mul2(g, t2);
    const f2 Ld = fma2(bc2(LN2), sub2(L2X, L2X2), Dl);  // log(a/b)
    // log case: 1 + hm1 = log(a/b) (a + b) / (2 (a - b)) and L = log(a/b) / (a - b)
    const f2 Lr = mul2(Ld, rden);
    const f2 hm1 = sel2(ser_x, ser_y, hm1_series, fma2(mul2(bc2(0.5f), Lr), sab, bc2(-1.0f)));
    const f2 rs2 = add2(rden, rden);
    const f2 L = sel2(ser_x, ser_y, fma2(hm1, rs2, rs2), Lr);
    const f2 r2Lq = mul2(mul2(bc2(P.r2), L), q);
    const f2 fq2 = mul2(add2(hm1, hm1), mul2(q, q));
    const f2 C0 = fma2(bc2(-4.0f), r2Lq, fq2);
    const f2 B1 = fma2(r, U1, V1), B2 = fma2(r, U2, V2);
    const f2 w = mul2(r2Lq, bc2(P.two_r));
    const f2 k2 = fma2(mul2(w, B1), rcp2(mul2(Xsq, z2)), C0);
    const f2 k2s = fma2(mul2(w, B2), rcp2(mul2(X2sq, z)), C0);
    const f2 kf = mul2(sub2(r2Lq, fq2), bc2(ph.nf_over_nc));
    const f2 dip = mul2(make_float2(vXx.S, vXy.S), D1), dips = mul2(make_float2(vX2x.S, vX2y.S), D2);
    // the cut |K2| > 1e10 with |dipole| < 1e-10 sets both factors to zero: zero their product
    const bool cut_x = fabsf(k2.x) > 1e10f && fabsf(dip.x) < 1e-10f;
    const bool cut_y = fabsf(k2.y) > 1e10f && fabsf(dip.y) < 1e-10f;
    const f2 prod = sel2(cut_x, cut_y, bc2(0.0f), mul2(k2, dip));
    const f2 dNX = fast_ndiff2(vXx, vXy, vX2x, vX2y);
    f2 k2part, fermion;
    if (SYM) {  // the factor 1/2 of the symmetrisation is folded into cpt
        const bool cuts_x = fabsf(k2s.x) > 1e10f && fabsf(dips.x) < 1e-10f;
        const bool cuts_y = fabsf(k2s.y) > 1e10f && fabsf(dips.y) < 1e-10f;
        k2part = add2(prod, sel2(cuts_x, cuts_y, bc2(0.0f), mul2(k2s, dips)));
        fermion = mul2(mul2(kf, dNX), dN);
    } else {
        k2part = prod;
        fermion = mul2(mul2(kf, SY), dNX);
    }
    f2 alpha;
    if (COUPLING == 2) {
        alpha = bc2(ph.fixed_as);
    } else if (COUPLING == 4) {
        alpha = bc2(P.alpha_r);
    } else {
        const f2 lmin = make_float2(fminf(fminf(Lmin.x, P.lr), (0.5f * LN2) * fminf(L2X.x, L2X2.x)),
                                    fminf(fminf(Lmin.y, P.lr), (0.5f * LN2) * fminf(L2X.y, L2X2.y)));
        if (COUPLING == 3) {
            alpha = make_float2(alpha_of_log(lmin.x, ph), alpha_of_log(lmin.y, ph));
        } else {
            const f2 right = fma2(bc2(-10.0f), lmin, bc2(5.0f * ph.log_sc));
            const f2 m = make_float2(fmaxf(ph.left, right.x), fmaxf(ph.left, right.y));
            const f2 gap = make_float2(fabsf(ph.left - right.x), fabsf(ph.left - right.y));
            // logaddexp = max + log(1 + e^-gap); beyond gap = 17 the correction is below
            // 4.2e-8 of max >= 9.16 (FP32 rounding), and the warp skips the two MUFU operations
            f2 lae = m;
            if (gap.x < 17.0f || gap.y < 17.0f) {
                const f2 e = make_float2(ex2_approx(-gap.x * L2E), ex2_approx(-gap.y * L2E));
                lae = fma2(bc2(LN2), lg22(add2(bc2(1.0f), e)), m);
            }
            alpha = rcp2(mul2(bc2(ph.b0c), lae));
            if (COUPLING == 1) alpha = make_float2(fminf(alpha.x, ph.alpha_cap), fminf(alpha.y, ph.alpha_cap));
        }
    }
    const f2 scale = mul2(mul2(alpha, alpha), cpt);
    const f2 k2w = mul2(k2part, scale);
    kfw = mul2(make_float2(-fermion.x, -fermion.y), scale);
    if constexpr (FINE) {
        kfw = sel2(fabsf(kfw.x) < INFINITY, fabsf(kfw.y) < INFINITY, kfw, bc2(0.0f));
        total = sel2(fabsf(k2w.x) < INFINITY, fabsf(k2w.y) < INFINITY, k2w, bc2(0.0f));
        return;
    }
    const f2 tot = add2(k2w, kfw);
    // X^2 or X'^2 below the normal range (the oracle's validity cut) gives infinite kernels
    // (the approximate reciprocal flushes denormals), so the finite test covers it
    const bool ok_x = fabsf(tot.x) < INFINITY;
    const bool ok_y = fabsf(tot.y) < INFINITY;
    kfw = sel2(ok_x, ok_y, kfw, bc2(0.0f));
    total = sel2(ok_x, ok_y, tot, bc2(0.0f));
}

// The pre-scaled rows of a FastSpline with its two edge rows, from the FP64 log S block; called by
// all threads of a CTA, before a barrier.
__device__ __forceinline__ void stage_fast_rows(float4* rows, const double* coef, int n, double h)
{
    const double l2e = 1.4426950408889634;
    for (int i = threadIdx.x; i < n - 1; i += blockDim.x) {
        const double* c = coef + 4 * (size_t)i;
        rows[i + 1] = make_float4((float)(c[0] * l2e), (float)(c[1] * h * l2e), (float)(c[2] * h * h * l2e),
                                  (float)(c[3] * h * h * h * l2e));
    }
    if (threadIdx.x == 0) {
        rows[0] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        rows[n] = make_float4(-150.0f, 0.0f, 0.0f, 0.0f);
    }
}

__device__ __forceinline__ FastSpline fast_spline(const float4* rows, int n, double x0, double h)
{
    FastSpline fs;
    fs.coef = rows;
    fs.u_scale = (float)(0.5 * 0.69314718055994531 / h);
    fs.u_off = (float)(-x0 / h);
    fs.u_top = (float)(n - 1);
    return fs;
}

__device__ __forceinline__ FineSpline fine_spline(const float4* rows, int n, double x0, double h)
{
    FineSpline fs;
    static_cast<FastSpline&>(fs) = fast_spline(rows, n, x0, h);
    fs.u_scale_lo = (float)(0.5 * 0.69314718055994531 / h - (double)fs.u_scale);
    fs.u_off_lo = (float)(-x0 / h - (double)fs.u_off);
    fs.l_scale = (float)(1.0 / h);
    fs.l_scale_lo = (float)(1.0 / h - (double)fs.l_scale);
    return fs;
}

// A parent for Vegas: r^2 is that of the rounded r, as in X^2.
__device__ __forceinline__ K2ParentF fine_parent(double r, const Phys<float>& ph)
{
    K2ParentF P;
    P.r = (float)r;
    P.r2 = P.r * P.r;
    P.lr = (float)log(r);
    P.two_r = (float)(2.0 * r);
    P.four_r = (float)(4.0 * r);
    P.alpha_r = alpha_of_log(P.lr, ph);
    return P;
}

// The records of two samples (component x, y) at box coordinates lz = log z, lz2 = log z',
// th, th2, in registers, for a caller that evaluates each record once (Vegas, one parent per
// integral): k2_prepare_x with the amplitudes from the FineSpline rows, z^2 z'^2 for the Jacobian,
// and every cosine as 1 - 2 sin^2 of the half angle with the 1s cancelled by hand, z' - z c12 =
// (z' - z) + 2 z sin^2, so that neighbouring z and z' at small angles, where adapted grids put
// their samples, keep their differences.
__device__ __forceinline__ void k2_prepare_pair(const FineSpline& s, float cpt_scale, f2 lz, f2 lz2, f2 th, f2 th2,
                                                float4 (&rec4)[kRecLen / 2])
{
    constexpr float LN2 = 0.69314718055994531f;
    const f2 z = make_float2(expf(lz.x), expf(lz.y)), z2 = make_float2(expf(lz2.x), expf(lz2.y));
    const f2 sh1 = make_float2(sinf(0.5f * th.x), sinf(0.5f * th.y));
    const f2 sh2 = make_float2(sinf(0.5f * th2.x), sinf(0.5f * th2.y));
    const f2 sh12 = make_float2(sinf(0.5f * (th.x - th2.x)), sinf(0.5f * (th.y - th2.y)));
    const f2 sq1 = mul2(sh1, sh1), sq2 = mul2(sh2, sh2), sq12 = mul2(sh12, sh12);
    const f2 dz = sub2(z, z2);
    const f2 zz2 = mul2(z, z2);
    const f2 zzsq = fma2(mul2(bc2(4.0f), zz2), sq12, mul2(dz, dz));
    const f2 L2ZZ = make_float2(log2f(zzsq.x), log2f(zzsq.y));
    P2S Yx, Yy, Wx, Wy, Zx, Zy;
    fine_amplitude_pair(s, lz, s.l_scale, s.l_scale_lo, Yx, Yy);
    fine_amplitude_pair(s, lz2, s.l_scale, s.l_scale_lo, Wx, Wy);
    fine_amplitude_pair(s, L2ZZ, s.u_scale, s.u_scale_lo, Zx, Zy);
    const f2 NZ = expm1_2(make_float2(LN2 * Zx.p2, LN2 * Zy.p2));  // -N_zz
    const f2 SY = make_float2(Yx.S, Yy.S), SW = make_float2(Wx.S, Wy.S), SZ = make_float2(Zx.S, Zy.S);
    const f2 dN = fast_ndiff2(Wx, Wy, Yx, Yy);  // N_Y2 - N_Y
    const f2 SZdN = mul2(SZ, dN);
    const f2 nSY = make_float2(-SY.x, -SY.y), nSW = make_float2(-SW.x, -SW.y);
    const f2 D1 = fma2(nSY, NZ, SZdN), D2 = fma2(nSW, NZ, make_float2(-SZdN.x, -SZdN.y));
    const bool ok_x = zzsq.x >= M<float>::tiny_square(), ok_y = zzsq.y >= M<float>::tiny_square();
    const f2 q = make_float2(ok_x ? rcp_approx(zzsq.x) : 0.0f, ok_y ? rcp_approx(zzsq.y) : 0.0f);
    const f2 zsq = mul2(z, z), z2sq = mul2(z2, z2);
    f2 cpt = mul2(bc2(cpt_scale), mul2(zsq, z2sq));
    cpt = make_float2(ok_x ? cpt.x : 0.0f, ok_y ? cpt.y : 0.0f);
    const f2 zc = fma2(bc2(2.0f), sub2(mul2(z2, sq1), mul2(z, sq2)), dz);  // z cos th' - z' cos th
    const f2 s1 = mul2(z, sq1), s2 = mul2(z2, sq2);
    const f2 P1 = mul2(sub2(z2, z), add2(z2, z)), P2 = mul2(mul2(bc2(-2.0f), zz2), zc);
    const f2 two12 = add2(sq12, sq12);
    const f2 U1 = fma2(z, two12, make_float2(-dz.x, -dz.y)), V1 = mul2(z, zc);
    const f2 U2 = fma2(z2, two12, dz), V2 = mul2(make_float2(-z2.x, -z2.y), zc);
    const f2 lm = make_float2(fminf(fminf(lz.x, lz2.x), 0.5f * LN2 * L2ZZ.x),
                              fminf(fminf(lz.y, lz2.y), 0.5f * LN2 * L2ZZ.y));
    const f2 Dl = mul2(bc2(2.0f), sub2(lz2, lz));
    auto put = [&](int k, f2 a, f2 b) { rec4[k] = make_float4(a.x, a.y, b.x, b.y); };
    put(0, z, z2);
    put(1, s1, s2);
    put(2, P1, P2);
    put(3, U1, V1);
    put(4, U2, V2);
    put(5, q, D1);
    put(6, D2, dN);
    put(7, SY, lm);
    put(8, cpt, Dl);
    put(9, zsq, z2sq);
}

// Parents of a CTA of the fixed-point kernels; larger grids take several parent tiles.
constexpr int kLaneCap = 448;

// The box at the kernels' precision with the integral's constant factor.
template <typename T>
inline K2Box<T> make_box(const nlo_bk_params& p, const nlo_bk_box& box, bool sym)
{
    K2Box<T> kb;
    double volume = 1.0;
    for (int d = 0; d < 4; ++d) {
        kb.lower[d] = (T)box.lower[d];
        kb.width[d] = (T)box.width[d];
    }
    if (sizeof(T) == sizeof(float)) {
        const float v01 = (float)box.width[0] * (float)box.width[1];
        const float v23 = (float)box.width[2] * (float)box.width[3];
        volume = (double)(v01 * v23);
    } else {
        volume = box.width[0] * box.width[1] * box.width[2] * box.width[3];
    }
    // the FP32 path folds the symmetrisation's 1/2 into the per-sample weight
    const double half = (sizeof(T) == sizeof(float) && sym) ? 0.5 : 1.0;
    kb.cpt_scale = (T)(half * volume * p.nc * p.nc / (8.0 * kPi * kPi * kPi * kPi));
    return kb;
}

// The kernel instantiation of a parameter set: FP64 (one form for every coupling) or the
// FP32 coupling variant; f(T(), SYM, COUPLING) with std::integral_constant tags.
template <class F>
cudaError_t dispatch_variant(const nlo_bk_params& p, F f)
{
    using std::integral_constant;
    const bool sym = p.symmetrize != 0;
    const int coupling = p.fixed_coupling                 ? 2
                         : p.rc_nlo == NLO_RC_NLO_PARENT ? 4
                         : p.nf > 3.0                    ? 3
                         : p.alpha_cap > 0.0             ? 1
                                                         : 0;
#define NLO_K2_VARIANT(T, C)                                                                  \
    (sym ? f(T(), integral_constant<bool, true>(), integral_constant<int, C>())                \
         : f(T(), integral_constant<bool, false>(), integral_constant<int, C>()))
    if (p.precision == NLO_PRECISION_FP64) return NLO_K2_VARIANT(double, 0);
    switch (coupling) {
        case 0: return NLO_K2_VARIANT(float, 0);
        case 1: return NLO_K2_VARIANT(float, 1);
        case 2: return NLO_K2_VARIANT(float, 2);
        case 3: return NLO_K2_VARIANT(float, 3);
        default: return NLO_K2_VARIANT(float, 4);
    }
#undef NLO_K2_VARIANT
}

}  // namespace k2
}  // namespace nlo
