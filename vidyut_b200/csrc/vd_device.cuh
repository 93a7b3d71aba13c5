// vd_device.cuh -- device-side data layout and physics of the explicit species /
// electron-energy update (sm_100a).
//
// The mechanism lives in __constant__ memory (every thread of a warp reads the
// same reaction at the same time, so the constant cache broadcasts it).  Two
// arithmetic flavours share the code:
//   PREC_FP64   all arithmetic in FP64; results agree with the reference CPU build
//               to ~1e-14 (FMA contraction and exp(log) rate evaluation are the
//               only differences);
//   PREC_MIXED  WENO weights, reconstructions, flux arithmetic and mobilities in
//               FP32 (values rescaled by an exact power of two per stencil), rate
//               constants through the FP32 special-function unit, and FP64 for the
//               production/loss sums, the energy-exchange sum and n += dt*dsdt.
#pragma once
#include "vd_types.cuh"

namespace vd {

// The loaded mechanism.  Every translation unit that includes this header has its
// own copy (internal linkage; the library is compiled without relocatable device
// code) and uploads it through its own upload function (upload_mech in
// vd_kernels.cu, which also calls upload_mech_batch in vd_batch_kernels.cu and
// upload_mech_diffusion in vd_diffusion.cu).
static __constant__ VdMechDev c_mech;

// Approximate reciprocal on the special-function unit (rcp.approx.ftz.f32,
// ~1 ulp); arguments are normal positive numbers wherever it is used.
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// 2^x for an FP64 exponent x as an FP32 value: x = i + f with i = rint(x) (exact in
// FP64), 2^f for f in [-1/2, 1/2] on the FP32 special-function unit (exp2f, ~2 ulp)
// and 2^i through the exponent bits.  Relative error ~2.4e-7 whatever |x|;
// results below 2^-126 flush to zero, above 2^127 saturate to infinity.
__device__ __forceinline__ float exp2_split(double x)
{
    const double xi = rint(x);
    const float f = exp2f((float)(x - xi));
    int i = (int)fmax(fmin(xi, 128.0), -127.0);
    if (i <= -127) return 0.0f;
    if (i >= 128) return __int_as_float(0x7f800000);
    return f * __int_as_float((i + 127) << 23);
}

// ---------------------------------------------------------------------------
// Mobility (specMob, test/models/Ar_DC_1d/Chemistry.H:177-202) by model kind.
// FP64: mob_c = -e/me / sqrt(8 kB/(pi me)) (electron) or e/M / sqrt(8 kB/(pi M))
// (ion), so mu = mob_c / (sqrt(T) N sigma): one sqrt and one division.  emag is
// the field magnitude |E| the caller's reference loop passes to specMob (power
// laws in |E|, test/verification/Streamer/Chemistry.H:165-183).
// The He_RF_1d header's models (test/verification/He_RF_1d/Chemistry.H:229-243),
// in its order of operations: the ion form (1 + c0 x^2 + c1 x^4)^p of x = |E|/N,
// and the electron form exp(c0 + c1 ln m + c2/m + c3/m^2 + c4/m^3) of the mean
// energy m = 1.5 Te/eV (the constant factor and the 1/N are the caller's).
__device__ __forceinline__ double mob_en_poly(const double* c, double p, double emag, double N)
{
    const double x = emag / N;
    return pow(1.0 + c[0] * pow(x, 2.0) + c[1] * pow(x, 4.0), p);
}
__device__ __forceinline__ double mob_exp_meane(const double* c, double Te)
{
    const double m = 1.5 * Te / EV;
    return exp(c[0] + c[1] * log(m) + c[2] / m + c[3] / pow(m, 2.0) + c[4] / pow(m, 3.0));
}
// The field-dependent models in FP64, out of line: their pow / exp / log code,
// inlined into the transport tile, would cost every mechanism registers that only
// these models use.
static __device__ __noinline__ double mob_field_fp64(int s, double Te, double N, double emag)
{
    switch (c_mech.mob_kind[s]) {
    case VD_MOB_POW_EMAG: return c_mech.mob_p0[s] * pow(emag, c_mech.mob_p1[s]);
    case VD_MOB_EN_POLY: return c_mech.mob_p0[s] * mob_en_poly(c_mech.fits[c_mech.mob_ref[s]].jc, c_mech.mob_p1[s], emag, N);
    case VD_MOB_EXP_MEANE: return c_mech.mob_p0[s] * mob_exp_meane(c_mech.fits[c_mech.mob_ref[s]].jc, Te) / N;
    default: return 0.0;
    }
}
// velocity basis kinds 3, 4 and 5 of the FP64 transport tile (E times the per-cell
// factor of VD_MOB_POW_EMAG / VD_MOB_EN_POLY / VD_MOB_EXP_MEANE), out of line
static __device__ __noinline__ double basis_field_fp64(int kind, int fit, double pw, double E, double emag, double N,
                                                       double Te)
{
    if (kind == 3) return E * pow(emag, pw);
    if (kind == 4) return E * mob_en_poly(c_mech.fits[fit].jc, pw, emag, N);
    return E * mob_exp_meane(c_mech.fits[fit].jc, Te) / N;
}
__device__ __forceinline__ double mob_base_fp64(int s, double Te, double N, double Tg, double emag)
{
    switch (c_mech.mob_kind[s]) {
    case VD_MOB_ELECTRON: return c_mech.mob_c[s] / (sqrt(Te) * N * c_mech.mob_p0[s]);
    case VD_MOB_ION_TG: return c_mech.mob_c[s] / (sqrt(Tg) * N * c_mech.mob_p0[s]);
    case VD_MOB_CONST_N: return c_mech.mob_p0[s] / N;
    case VD_MOB_CONST: return c_mech.mob_p0[s];
    case VD_MOB_POW_EMAG:
    case VD_MOB_EN_POLY:
    case VD_MOB_EXP_MEANE: return mob_field_fp64(s, Te, N, emag);
    default: return 0.0;
    }
}
__device__ __forceinline__ double mob_fp64(int s, double Te, double N, double Tg, double emag)
{
    if (c_mech.mob_kind[s] == VD_MOB_SCALED)
        return c_mech.mob_p0[s] * mob_base_fp64(c_mech.mob_ref[s], Te, N, Tg, emag);
    return mob_base_fp64(s, Te, N, Tg, emag);
}
// The He_RF_1d models for the mixed path: the polynomial in FP32; the
// mean-energy exponent (about 55, whose FP32 rounding alone would be 4e-6 of the
// mobility) summed in FP64 from an FP32 logarithm and raised by exp2_split.
__device__ __forceinline__ float mob_en_poly_f32(const double* c, float p, float emag, float N)
{
    const float x = emag * rcp_approx(N);
    const float x2 = x * x;
    const float q = fmaf((float)c[1], x2 * x2, fmaf((float)c[0], x2, 1.0f));
    return exp2f(p * log2f(q));
}
__device__ __forceinline__ float mob_exp_meane_f32(const double* c, float Te)
{
    constexpr double LN2 = 0.69314718055994530942, LOG2E = 1.4426950408889634074;
    const double m = 1.5 * (double)Te / EV;
    const double im = 1.0 / m;
    const double sum = fma((double)log2f((float)m), c[1] * LN2, c[0]) + im * fma(im, fma(im, c[4], c[3]), c[2]);
    return exp2_split(sum * LOG2E);
}
// velocity basis kinds 3, 4 and 5 of the mixed transport tile, out of line (as
// basis_field_fp64)
static __device__ __noinline__ float basis_field_f32(int kind, int fit, float pw, float E, float emag, float N,
                                                     float Te)
{
    if (kind == 3) return E * exp2f(pw * log2f(emag));
    if (kind == 4) return E * mob_en_poly_f32(c_mech.fits[fit].jc, pw, emag, N);
    return E * mob_exp_meane_f32(c_mech.fits[fit].jc, Te) * rcp_approx(N);
}
__device__ __forceinline__ float mob_base_f32(int s, float Te, float N, float Tg, float emag)
{
    switch (c_mech.mob_kind[s]) {
    case VD_MOB_ELECTRON: return (float)c_mech.mob_c[s] * rsqrtf(Te) * rcp_approx(N * (float)c_mech.mob_p0[s]);
    case VD_MOB_ION_TG: return (float)c_mech.mob_c[s] * rsqrtf(Tg) * rcp_approx(N * (float)c_mech.mob_p0[s]);
    case VD_MOB_CONST_N: return (float)c_mech.mob_p0[s] * rcp_approx(N);
    case VD_MOB_CONST: return (float)c_mech.mob_p0[s];
    case VD_MOB_POW_EMAG: return (float)c_mech.mob_p0[s] * exp2f((float)c_mech.mob_p1[s] * log2f(emag));
    // the exponential's argument is too large for FP32 (e^55 in the He_RF_1d fit)
    case VD_MOB_EN_POLY:
        return (float)c_mech.mob_p0[s] *
               mob_en_poly_f32(c_mech.fits[c_mech.mob_ref[s]].jc, (float)c_mech.mob_p1[s], emag, N);
    case VD_MOB_EXP_MEANE:
        return (float)c_mech.mob_p0[s] * mob_exp_meane_f32(c_mech.fits[c_mech.mob_ref[s]].jc, Te) * rcp_approx(N);
    default: return 0.0f;
    }
}
__device__ __forceinline__ float mob_f32(int s, float Te, float N, float Tg, float emag)
{
    if (c_mech.mob_kind[s] == VD_MOB_SCALED)
        return (float)c_mech.mob_p0[s] * mob_base_f32(c_mech.mob_ref[s], Te, N, Tg, emag);
    return mob_base_f32(s, Te, N, Tg, emag);
}
// specDiff (test/models/Ar_DC_1d/Chemistry.H:204-239) by model kind; the
// field- and pressure-dependent ones out of line, as mob_field_fp64.
static __device__ __noinline__ double diff_field_fp64(int s, double Te, double N, double Tg, double emag)
{
    switch (c_mech.diff_kind[s]) {
    case VD_DIFF_POW_EMAG: return c_mech.diff_factor[s] * pow(emag, c_mech.diff_p1[s]);
    // P_NTP / (N kB Tg) (test/verification/He_RF_1d/Chemistry.H:270-296)
    case VD_DIFF_PRES: return c_mech.diff_factor[s] * (P_NTP / (N * K_B * Tg));
    case VD_DIFF_TE_PRES: return c_mech.diff_factor[s] * (Te / c_mech.diff_p1[s]) * (P_NTP / (N * K_B * Tg));
    default: return 0.0;
    }
}
__device__ __forceinline__ double diff_base_fp64(int s, double Te, double N, double Tg, double emag)
{
    switch (c_mech.diff_kind[s]) {
    case VD_DIFF_TE_ABSMOB:
        return c_mech.diff_factor[s] * (Te / EV) * fabs(mob_fp64(c_mech.diff_ref[s], Te, N, Tg, emag));
    case VD_DIFF_TG_MOB:
        return c_mech.diff_factor[s] * (Tg / EV) * mob_fp64(c_mech.diff_ref[s], Te, N, Tg, emag);
    case VD_DIFF_CONST: return c_mech.diff_factor[s];
    case VD_DIFF_POW_EMAG:
    case VD_DIFF_PRES:
    case VD_DIFF_TE_PRES: return diff_field_fp64(s, Te, N, Tg, emag);
    default: return 0.0;
    }
}
// specDiff with the scaled model (D = factor * D[ref], the energy's 5/3 of the
// electrons' coefficient in the Streamer and He_RF_1d headers)
__device__ __forceinline__ double diff_fp64(int s, double Te, double N, double Tg, double emag)
{
    if (c_mech.diff_kind[s] == VD_DIFF_SCALED)
        return c_mech.diff_factor[s] * diff_base_fp64(c_mech.diff_ref[s], Te, N, Tg, emag);
    return diff_base_fp64(s, Te, N, Tg, emag);
}
__device__ __forceinline__ float diff_base_f32(int s, float Te, float N, float Tg, float emag, float mu_e)
{
    // mu_e: the electron mobility when s's model refers to it (saves its re-evaluation)
    const int dk = c_mech.diff_kind[s], dr = c_mech.diff_ref[s];
    const float f = (float)c_mech.diff_factor[s];
    switch (dk) {
    case VD_DIFF_TE_ABSMOB:
    case VD_DIFF_TG_MOB: {
        const float mr = dr == c_mech.e_id ? mu_e : mob_f32(dr, Te, N, Tg, emag);
        if (dk == VD_DIFF_TE_ABSMOB) return f * (Te * (float)(1.0 / EV)) * fabsf(mr);
        return f * (Tg * (float)(1.0 / EV)) * mr;
    }
    case VD_DIFF_CONST: return f;
    case VD_DIFF_POW_EMAG: return f * exp2f((float)c_mech.diff_p1[s] * log2f(emag));
    case VD_DIFF_PRES: return f * ((float)P_NTP * rcp_approx(N * (float)K_B * Tg));
    case VD_DIFF_TE_PRES:
        return f * (Te * (float)(1.0 / c_mech.diff_p1[s])) * ((float)P_NTP * rcp_approx(N * (float)K_B * Tg));
    default: return 0.0f;
    }
}
__device__ __forceinline__ float diff_f32(int s, float Te, float N, float Tg, float emag, float mu_e)
{
    if (c_mech.diff_kind[s] == VD_DIFF_SCALED)
        return (float)c_mech.diff_factor[s] * diff_base_f32(c_mech.diff_ref[s], Te, N, Tg, emag, mu_e);
    return diff_base_f32(s, Te, N, Tg, emag, mu_e);
}

// ---------------------------------------------------------------------------
// WENO-5 reconstruction at i+1/2 from (im2, im1, i, ip1, ip2)
// (Source/compute_explicit_flux.H:25-112).  SCHEME 1 JS, 2 M, 3 Z.
template <class R>
__device__ __forceinline__ R gk_map(R wk, R g)
{
    return wk * (g + g * g - R(3) * g * wk + wk * wk) / (g * g + wk * (R(1) - R(2) * g));
}

// One FP32 reconstruction of values already scaled to O(1), from its three 4 beta_k
// and candidate polynomials.  The nonlinear weights are
// rescaled so that no term can overflow and the smoothest stencil always keeps a
// weight of order gamma (the sum never underflows to zero, whatever the spread of
// the smoothness indicators): with q_k = beta_k + eps and m = min_k q_k,
//   WENO-JS  alpha_k ~ gamma_k (m/q_k)^2
//   WENO-Z   alpha_k ~ gamma_k (1 + (tau/q_k)^2)              if tau <= m
//            alpha_k ~ gamma_k ((m/tau)^2 + (m/q_k)^2)        otherwise
// (each a positive multiple of the reference's alpha_k); WENO-M keeps its map.
// The smoothness indicators are kept as 4 beta_k (13/3 and 1 for the reference's
// 13/12 and 1/4) and eps4 is 4 eps: every weight is a ratio of these, and scaling
// by a power of two changes no rounding, so the result is the same and each
// indicator costs one multiply less.
// Two FP32 values in one register pair: Blackwell's packed FP32 arithmetic (one issue
// slot for both halves, each rounded as the scalar operation).
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float x, float y)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void unpack2(F2 a, float& x, float& y)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}
__device__ __forceinline__ F2 both2(float x) { return pack2(x, x); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b) { return fma2(both2(-1.0f), b, a); }  // one rounding, as a - b

// One reconstruction of two fields at once (packed), eps4 the same for both; scheme 3
// WENO-Z, 1 WENO-JS, 2 WENO-M.  The kernel is issue bound (72 % active, FMA 35 %): the
// drift flux and the density of a face go through packed operations side by side, same
// bits (B200: 3-D transport of 24 species on 128^3 1.86 -> 1.80 ms, a batched 2-D
// step 0.295 -> 0.276 ms).
__device__ __forceinline__ F2 weno_weights_f32(F2 b1, F2 b2, F2 b3, F2 p1, F2 p2, F2 p3, int scheme, F2 eps4)
{
    const F2 q1 = add2(b1, eps4), q2 = add2(b2, eps4), q3 = add2(b3, eps4);
    float q1x, q1y, q2x, q2y, q3x, q3y;
    unpack2(q1, q1x, q1y);
    unpack2(q2, q2x, q2y);
    unpack2(q3, q3x, q3y);
    const float mx = fminf(q1x, fminf(q2x, q3x)), my = fminf(q1y, fminf(q2y, q3y));
    const F2 r1 = pack2(rcp_approx(q1x), rcp_approx(q1y)), r2 = pack2(rcp_approx(q2x), rcp_approx(q2y));
    const F2 r3 = pack2(rcp_approx(q3x), rcp_approx(q3y));
    F2 a1, a2, a3;
    if (scheme == 3) {
        float tx, ty;
        unpack2(sub2(b1, b3), tx, ty);
        tx = fabsf(tx);
        ty = fabsf(ty);
        const bool bx = tx > mx, by = ty > my;
        const float cx = bx ? __fmul_rn(mx, rcp_approx(tx)) : 1.0f, cy = by ? __fmul_rn(my, rcp_approx(ty)) : 1.0f;
        const F2 t = pack2(bx ? mx : tx, by ? my : ty), cr = pack2(cx, cy);
        const F2 B1 = mul2(t, r1), B2 = mul2(t, r2), B3 = mul2(t, r3);
        const F2 c2 = mul2(cr, cr);
        a1 = mul2(both2(0.1f), fma2(B1, B1, c2));
        a2 = mul2(both2(0.6f), fma2(B2, B2, c2));
        a3 = mul2(both2(0.3f), fma2(B3, B3, c2));
    } else {
        const F2 m = pack2(mx, my);
        const F2 B1 = mul2(m, r1), B2 = mul2(m, r2), B3 = mul2(m, r3);
        a1 = mul2(both2(0.1f), mul2(B1, B1));
        a2 = mul2(both2(0.6f), mul2(B2, B2));
        a3 = mul2(both2(0.3f), mul2(B3, B3));
        if (scheme == 2) {
            float x, y, ax, ay;
            unpack2(add2(add2(a1, a2), a3), x, y);
            x = rcp_approx(x);
            y = rcp_approx(y);
            unpack2(a1, ax, ay);
            a1 = pack2(gk_map(ax * x, 0.1f), gk_map(ay * y, 0.1f));
            unpack2(a2, ax, ay);
            a2 = pack2(gk_map(ax * x, 0.6f), gk_map(ay * y, 0.6f));
            unpack2(a3, ax, ay);
            a3 = pack2(gk_map(ax * x, 0.3f), gk_map(ay * y, 0.3f));
        }
    }
    float sx, sy;
    unpack2(add2(add2(a1, a2), a3), sx, sy);
    return mul2(fma2(a1, p1, fma2(a2, p2, mul2(a3, p3))), pack2(rcp_approx(sx), rcp_approx(sy)));
}

// Both reconstructions of two fields at a face from their six stencil values x0..x5:
// plus, the left-biased WENO-5 value from x0..x4, and minus, the right-biased one
// from x5..x1 (weno(e,d,c,b,a) of the reference).
// They share two of their three second differences (x1-2x2+x3, x2-2x3+x4) with
// their squared terms, and two of their candidate polynomials (the parabola
// through x1..x3 at x2+1/2 and through x2..x4 at x3+1/2), which are computed once.
__device__ __forceinline__ void weno_pair_f32(const F2* x, int scheme, F2 eps4, F2& plus, F2& minus)
{
    const F2 k2 = both2(-2.0f), k133 = both2(13.0f / 3.0f), k13 = both2(1.0f / 3.0f), k56 = both2(5.0f / 6.0f);
    const F2 k16 = both2(-1.0f / 6.0f), k76 = both2(-7.0f / 6.0f), k116 = both2(11.0f / 6.0f);
    const F2 k3 = both2(3.0f), k4 = both2(-4.0f);
    // second differences and the 13/3 d^2 terms of the windows centred at x1..x4
    const F2 d1 = add2(fma2(k2, x[1], x[0]), x[2]), d2 = add2(fma2(k2, x[2], x[1]), x[3]);
    const F2 d3 = add2(fma2(k2, x[3], x[2]), x[4]), d4 = add2(fma2(k2, x[4], x[3]), x[5]);
    const F2 c2 = mul2(k133, mul2(d2, d2)), c3 = mul2(k133, mul2(d3, d3));
    // the polynomials the two share
    const F2 pm = fma2(k16, x[1], fma2(k56, x[2], mul2(k13, x[3])));
    const F2 pn = fma2(k13, x[2], fma2(k56, x[3], mul2(k16, x[4])));
    {
        const F2 p1 = fma2(k13, x[0], fma2(k76, x[1], mul2(k116, x[2])));
        const F2 t2 = fma2(k3, x[2], fma2(k4, x[1], x[0])), t4 = sub2(x[1], x[3]);
        const F2 t6 = fma2(k3, x[2], fma2(k4, x[3], x[4]));
        const F2 b1 = fma2(k133, mul2(d1, d1), mul2(t2, t2)), b2 = fma2(t4, t4, c2), b3 = fma2(t6, t6, c3);
        plus = weno_weights_f32(b1, b2, b3, p1, pm, pn, scheme, eps4);
    }
    {
        const F2 p1 = fma2(k13, x[5], fma2(k76, x[4], mul2(k116, x[3])));
        const F2 t2 = fma2(k3, x[3], fma2(k4, x[4], x[5])), t4 = sub2(x[4], x[2]);
        const F2 t6 = fma2(k3, x[3], fma2(k4, x[2], x[1]));
        const F2 b1 = fma2(k133, mul2(d4, d4), mul2(t2, t2)), b2 = fma2(t4, t4, c3), b3 = fma2(t6, t6, c2);
        minus = weno_weights_f32(b1, b2, b3, p1, pn, pm, scheme, eps4);
    }
}

// ---------------------------------------------------------------------------
// First-order upwind and second-order WAF-MINBEE flux (compute_flux,
// Source/compute_explicit_flux.H:245-300) from the densities of cells i-2 .. i+1 and
// the velocities of cells i-1 and i; FP64 in both paths.
__device__ __forceinline__ double face_flux_low(double um, double pL, double pR, double up, double vL, double vR,
                                                int hyp_order, double dxmin, double dt)
{
    const double vmid = 0.5 * (vL + vR);
    const double sgn = copysign(1.0, vmid);
    const double fL = pL * vL, fR = pR * vR;
    if (hyp_order == 1) return fL * 0.5 * (1.0 + sgn) + fR * 0.5 * (1.0 - sgn);
    const double dl = pL - um, dm = pR - pL, dr = up - pR;
    const double cfl = vmid * dt / dxmin;
    const double r = (cfl >= 0.0) ? dl / (dm + 1.0e-30) : dr / (dm + 1.0e-30);
    const double lim = (r <= 0.0) ? 1.0 : ((r <= 1.0) ? 1.0 - (1.0 - fabs(cfl)) * r : fabs(cfl));
    return 0.5 * (fL + fR) - 0.5 * sgn * lim * (fR - fL);
}

// Mixed-precision face flux from densities already staged in FP32 (|n| < 3e38).
// The six values are scaled by an exact power of two s = 2^-e chosen from the
// exponent bits of max|u| (so max|u*s| is in [1/2, 1)); eps = 1e-20 is carried
// into the scaled units as 1e-20 s^2, clamped to [1e-30, 1e30] (for tiny fields
// eps dominates the smoothness indicators and the weights become the ideal ones,
// as in FP64).  The flux is unscaled by the exact power of two; the result is
// returned in FP32, which holds it exactly while it is a normal FP32 value (the
// FP64 route serves the one scale, 2^-127, that FP32 cannot hold).
__device__ __forceinline__ float face_flux_mixed32(const float* u, const float* v, int scheme)
{
    const float m = fmaxf(fmaxf(fmaxf(fabsf(u[0]), fabsf(u[1])), fmaxf(fabsf(u[2]), fabsf(u[3]))),
                          fmaxf(fabsf(u[4]), fabsf(u[5])));
    const int eb = (__float_as_int(m) >> 23) & 0xff;  // biased exponent of max|u|
    int e = 0;                                        // scale 2^-e; 0 for zero/denormal/non-finite
    if (eb > 0 && eb < 255) e = eb - 126;             // m in [2^(e-1), 2^e)
    int bs = 127 - e;
    bs = bs < 1 ? 1 : (bs > 254 ? 254 : bs);
    const float s = __int_as_float(bs << 23);
    int b2 = 127 - 2 * e;
    b2 = b2 < 0 ? 0 : (b2 > 255 ? 255 : b2);
    const float s2 = __int_as_float(b2 << 23);        // 2^-2e, 0 or inf at the ends
    const float eps = 4.0f * fminf(fmaxf(1e-20f * s2, 1e-30f), 1e30f);  // the weights take 4 eps
    // the drift flux f = u v in the low half, the density in the high half
    F2 x[6];
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const float us = __fmul_rn(u[q], s);
        x[q] = pack2(__fmul_rn(us, v[q]), us);
    }
    const float lam = fabsf(__fmul_rn(0.5f, __fadd_rn(v[2], v[3])));
    F2 plus, minus;
    weno_pair_f32(x, scheme, both2(eps), plus, minus);
    float fp, fm, up, um;
    unpack2(plus, fp, up);
    unpack2(minus, fm, um);
    const float F = 0.5f * (fmaf(lam, up, fp) + fmaf(-lam, um, fm));
    if (bs < 254) return F * __int_as_float((254 - bs) << 23);  // 2^(127-bs)
    return (float)((double)F * __longlong_as_double((long long)(1150 - bs) << 52));
}

// ---------------------------------------------------------------------------
// WENO-5 around one cell centre, in FP64 and without a division per weight.
//
// The reference reconstructs the right face of cell c as weno(a,b,c,d,e) (the
// left-biased value of that face) and its left face as weno(e,d,c,b,a) (the
// right-biased one) from the values a..e of cells c-2..c+2.  Both use the same three
// smoothness indicators in opposite order, so one triple Y_1..Y_3 per centre serves
// both, alpha_k = gamma_k Y_k at the right face and gamma_k Y_(4-k) at the left one.
// Written with the first differences g (of neighbours) and second differences d:
//   4 beta_1 = 13/3 d_-^2 + (d_- + 2 g_-)^2, 4 beta_2 = 13/3 d_0^2 + (g_- + g_+)^2,
//   4 beta_3 = 13/3 d_+^2 + (d_+ - 2 g_+)^2
// and, with q_k = 4 beta_k + 4 eps and tau = |q_1 - q_3|, the weights up to a common
// factor (every weight is a ratio; multiplied through by q_1^2 q_2^2 q_3^2)
//   WENO-Z   1 + (tau/q_k)^2  ->  Y_k = P + tau^2 P_k,  P_k = prod_(j != k) q_j^2,  P = q_k^2 P_k
//   WENO-JS  1/q_k^2          ->  Y_k = P_k   (M: then the map)
// (Source/compute_explicit_flux.H:38-109).  A reconstruction is then the cell value
// plus a weighted sum of the candidates' offsets from it, with one reciprocal.  Four
// divisions per centre and two reconstructions became two reciprocals.
// Range: the products are of degree 6 in q, so the values are taken scaled by
// kWenoScale = 2^-32 (exact): eps then keeps q above 2e-39 (q^6 > 1e-232, so a weighted
// offset keeps its digits down to differences of 1e-60), and values up to 4e32 keep a
// weighted offset (degree 13) below 1e308.  A larger value overflows to a NaN, and such
// a face is evaluated again with every centre scaled by its own power of two (SAFE;
// weno_y64).
// Every operation is pinned (no contraction left to the compiler), so a centre gives
// the same bits wherever in a run of faces it is evaluated and the tile
// decomposition cannot change a result.
constexpr double kWenoScale = 0x1p-32, kWenoUnscale = 0x1p32;

// 1/d of a normal FP64 number: the hardware's 20-bit approximation and one
// third-order (Householder) iteration r (1 + e + e^2), e = 1 - d r, which leaves
// e^3 < 2^-57 beside the rounding; no branch for the special operands that a
// correctly rounded division serves (zero, NaN and infinity give a NaN).
__device__ __forceinline__ double rcp64(double d)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = __fma_rn(-d, r, 1.0);
    return __fma_rn(r, __fma_rn(e, e, e), r);
}
// n/d by the same iteration on the quotient
__device__ __forceinline__ double div64(double n, double d)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = __fma_rn(-d, r, 1.0);
    const double q = __dmul_rn(n, r);
    return __fma_rn(q, __fma_rn(e, e, e), q);
}
struct WenoY64 {
    double y1, y2, y3;
};
// S: 1 JS, 2 M (unmapped here), 3 Z.  SAFE: the q_k are first scaled by the power of
// two that brings the larger of q_1, q_3 to [1, 2) (q_2 is at most a few times that;
// non-negative numbers order like their high words; a NaN or infinity keeps the scale
// finite and carries itself).
template <int S, bool SAFE>
__device__ __forceinline__ WenoY64 weno_y64(double q1, double q2, double q3)
{
    if constexpr (SAFE) {
        const int m = min(max(__double2hiint(q1), __double2hiint(q3)), 0x7fd00000) & 0x7ff00000;
        const double s = __hiloint2double(0x7fe00000 - m, 0);  // 2^-e
        q1 = __dmul_rn(q1, s);
        q2 = __dmul_rn(q2, s);
        q3 = __dmul_rn(q3, s);
    }
    const double Q1 = __dmul_rn(q1, q1), Q2 = __dmul_rn(q2, q2), Q3 = __dmul_rn(q3, q3);
    WenoY64 y;
    y.y1 = __dmul_rn(Q2, Q3);
    y.y2 = __dmul_rn(Q1, Q3);
    y.y3 = __dmul_rn(Q1, Q2);
    if constexpr (S == 3) {
        const double t = __dsub_rn(q1, q3);
        const double T = __dmul_rn(t, t), P = __dmul_rn(Q1, y.y1);
        y.y1 = __fma_rn(T, y.y1, P);
        y.y2 = __fma_rn(T, y.y2, P);
        y.y3 = __fma_rn(T, y.y3, P);
    }
    return y;
}
// the mapping of WENO-M (Henrick et al.) of a normalised weight
__device__ __forceinline__ double gk_map64(double wk, double g)
{
    const double num = __fma_rn(wk, wk, __fma_rn(-3.0 * g, wk, g + g * g));
    const double den = __fma_rn(wk, 1.0 - 2.0 * g, g * g);
    return div64(__dmul_rn(wk, num), den);
}
// xc + (1/6) sum_k a_k o_k / sum_k a_k with a = (y1, 6 y2, 3 y3) (M: mapped); A2 = 6 y2
template <int S>
__device__ __forceinline__ double weno_value64(double xc, double y1, double A2, double y3, double o1, double o2, double o3)
{
    double a1 = y1, a2 = A2, a3 = __dmul_rn(3.0, y3);
    double D = __dadd_rn(__dadd_rn(a1, a2), a3);
    if constexpr (S == 2) {
        const double r = rcp64(D);
        a1 = gk_map64(__dmul_rn(a1, r), 0.1);
        a2 = gk_map64(__dmul_rn(a2, r), 0.6);
        a3 = gk_map64(__dmul_rn(a3, r), 0.3);
        D = __dadd_rn(__dadd_rn(a1, a2), a3);
    }
    const double N = __fma_rn(a1, o1, __fma_rn(a2, o2, __dmul_rn(a3, o3)));
    return __fma_rn(1.0 / 6.0, div64(N, D), xc);
}
// The sliding window of one field around centre c: value, the differences to its
// neighbours and the second differences d with their 13/3 d^2 + 4 eps.
struct WenoWin64 {
    double xc, xp;          // cells c and c + 1
    double gm, gp;          // x_c - x_(c-1), x_(c+1) - x_c
    double dm, d0, cm, c0;  // second differences at c - 1 and c
};
template <bool SAFE>
__device__ __forceinline__ double weno_c64(double d)
{
    constexpr double eps4 = SAFE ? 4e-20 : 4e-20 * kWenoScale * kWenoScale;
    return __fma_rn(__dmul_rn(13.0 / 3.0, d), d, eps4);
}
// window around centre c from cells c-2 .. c+1
template <bool SAFE>
__device__ __forceinline__ WenoWin64 weno_start64(double xa, double xb, double xc, double xd)
{
    WenoWin64 w;
    w.xc = xc;
    w.xp = xd;
    const double ga = __dsub_rn(xb, xa);
    w.gm = __dsub_rn(xc, xb);
    w.gp = __dsub_rn(xd, xc);
    w.dm = __dsub_rn(w.gm, ga);
    w.d0 = __dsub_rn(w.gp, w.gm);
    w.cm = weno_c64<SAFE>(w.dm);
    w.c0 = weno_c64<SAFE>(w.d0);
    return w;
}
// Both reconstructions around the window's centre, given cell c + 2: `right`, the
// left-biased value at the right face of c, and `left`, the right-biased value at its
// left face (each only when wanted); then the window moves on by one cell.
template <int S, bool SAFE, bool RIGHT, bool LEFT>
__device__ __forceinline__ void weno_step64(WenoWin64& w, double xe, double& right, double& left)
{
    const double gn = __dsub_rn(xe, w.xp);  // x_(c+2) - x_(c+1)
    const double dp = __dsub_rn(gn, w.gp);  // second difference at c + 1
    const double cp = weno_c64<SAFE>(dp);
    const double t1 = __fma_rn(2.0, w.gm, w.dm), t2 = __dadd_rn(w.gm, w.gp), t3 = __fma_rn(-2.0, w.gp, dp);
    const WenoY64 y = weno_y64<S, SAFE>(__fma_rn(t1, t1, w.cm), __fma_rn(t2, t2, w.c0), __fma_rn(t3, t3, cp));
    const double A2 = __dmul_rn(6.0, y.y2);
    // six times the candidates' offsets from x_c
    if (RIGHT)
        right = weno_value64<S>(w.xc, y.y1, A2, y.y3, __fma_rn(2.0, t1, -w.gm), __fma_rn(3.0, w.gp, -w.d0),
                                __fma_rn(3.0, w.gp, -dp));
    if (LEFT)
        left = weno_value64<S>(w.xc, y.y3, A2, y.y1, __fma_rn(2.0, t3, w.gp), __fma_rn(-3.0, w.gm, -w.d0),
                               __fma_rn(-3.0, w.gm, -w.dm));
    w.xc = w.xp;
    w.xp = xe;
    w.gm = w.gp;
    w.gp = gn;
    w.dm = w.d0;
    w.d0 = dp;
    w.cm = w.c0;
    w.c0 = cp;
}
// local Lax-Friedrichs flux of a face from the reconstructions of the drift flux
// (fp, fm) and the density (up, um) and the two cells' velocities
// (Source/compute_explicit_flux.H:300-312)
__device__ __forceinline__ double llf_flux64(double fp, double fm, double up, double um, double vl, double vr)
{
    const double lam = fabs(__dmul_rn(0.5, __dadd_rn(vl, vr)));
    return __dmul_rn(0.5, __fma_rn(lam, __dsub_rn(up, um), __dadd_rn(fp, fm)));
}

// ---------------------------------------------------------------------------
// Face flux from the 6-cell stencil u[0..5] = cells (i-3 .. i+2), velocities v[0..5]
// (compute_flux, Source/compute_explicit_flux.H:245-316), WENO scheme S, for values
// of any size.
template <int S>
__device__ __forceinline__ double face_flux_weno64(const double* u, const double* v)
{
    double up, um, fp, fm, x;
    {
        WenoWin64 w = weno_start64<true>(u[0], u[1], u[2], u[3]);
        weno_step64<S, true, true, false>(w, u[4], up, x);
        weno_step64<S, true, false, true>(w, u[5], x, um);
    }
    {
        double f[6];
#pragma unroll
        for (int q = 0; q < 6; q++) f[q] = __dmul_rn(u[q], v[q]);
        WenoWin64 w = weno_start64<true>(f[0], f[1], f[2], f[3]);
        weno_step64<S, true, true, false>(w, f[4], fp, x);
        weno_step64<S, true, false, true>(w, f[5], x, fm);
    }
    return llf_flux64(fp, fm, up, um, v[2], v[3]);
}
__device__ __forceinline__ double face_flux_fp64(const double* u, const double* v, int hyp_order, int scheme,
                                                 double dxmin, double dt)
{
    if (hyp_order != 5) return face_flux_low(u[1], u[2], u[3], u[4], v[2], v[3], hyp_order, dxmin, dt);
    if (scheme == 3) return face_flux_weno64<3>(u, v);
    if (scheme == 2) return face_flux_weno64<2>(u, v);
    return face_flux_weno64<1>(u, v);
}
// The face of a run whose scaled evaluation was not finite: from its staged (scaled)
// densities pu and velocity basis pb (null: velocity k), `str` apart; scaled result.
static __device__ __noinline__ double face_flux_again64(const double* pu, const double* pb, int str, double k, int scheme)
{
    double u[6], v[6];
    for (int q = 0; q < 6; q++) {
        u[q] = pu[q * str] * kWenoUnscale;
        v[q] = pb ? __dmul_rn(k, pb[q * str]) : k;
    }
    return face_flux_fp64(u, v, 5, scheme, 1.0, 0.0) * kWenoScale;
}

// ---------------------------------------------------------------------------
// Janev / F-fit electron-impact rates (test/Reactor/CO2_H2_Ar_mechanism_reduced/
// Chemistry.H:940-1030): with Te_eV = Te/11595, tep[j] = ln(Te_eV)^j (j = 0..8) and
// itp[j] = Te_eV^-(j+1) (j = 0..3; 1 for Te = 0),
//   Janev  k = jA exp(sum_j jc_j tep[j]) NA,   F-fit  k = fA exp(sum_j fc_j itp[j]) NA,
// the sums accumulated in order.  FP64 takes the powers with pow() as the header
// does; the mixed path by products and the exponential on the FP32 unit.
template <int PREC>
__device__ __forceinline__ void fit_powers(double Te, double* tep, double* itp, double& teev)
{
    teev = Te / TE_FIT_EV;
    const double lte = log(teev);
    const double ite = (Te == 0) ? 1.0 : 1.0 / teev;
    if (PREC == PREC_FP64) {
#pragma unroll
        for (int j = 0; j < 9; j++) tep[j] = pow(lte, (double)j);
#pragma unroll
        for (int j = 0; j < 4; j++) itp[j] = pow(ite, (double)(j + 1));
    } else {
        tep[0] = 1.0;
#pragma unroll
        for (int j = 1; j < 9; j++) tep[j] = tep[j - 1] * lte;
        itp[0] = ite;
#pragma unroll
        for (int j = 1; j < 4; j++) itp[j] = itp[j - 1] * ite;
    }
}
template <int PREC>
__device__ __forceinline__ double fit_rate(int kind, const VdFitDev& F, const double* tep, const double* itp,
                                           double teev)
{
    const bool janev = kind == VD_RATE_JANEV || (kind == VD_RATE_JANEV_FFIT && teev < F.switch_ev);
    // products and sums rounded separately as the header's loop (no contraction):
    // the sums cancel terms up to ~1e5 times larger than the result
    double sum = 0.0;
    if (janev) {
#pragma unroll
        for (int j = 0; j < 9; j++) sum = __dadd_rn(sum, __dmul_rn(F.jc[j], tep[j]));
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++) sum = __dadd_rn(sum, __dmul_rn(F.fc[j], itp[j]));
    }
    if (PREC == PREC_FP64) return (janev ? F.jA : F.fA) * exp(sum) * NA_CE;
    constexpr double LOG2E = 1.4426950408889634074;
    return (double)exp2_split(fma(sum, LOG2E, janev ? F.l2jA : F.l2fA));
}

// Field-driven ionisation rate (test/verification/Streamer/Chemistry.H:266-280):
// alpha = (c0 + c1/E^3) exp(-c2/E), the attachment c3, mu_e = c4 E^c5,
// k = (alpha - c3) mu_e E, in the header's order of operations (FP64 in both paths).
__device__ __forceinline__ double townsend_rate(const double* c, double E)
{
    const double alpha = (c[0] + c[1] / pow(E, 3.0)) * exp(-c[2] / E);
    const double mu_e = c[4] * pow(E, c[5]);
    return (alpha - c[3]) * mu_e * E;
}

// ---------------------------------------------------------------------------
// CKWC for one cell (Source/ScalarSolve.cpp:143-157 + the generated productionRate,
// test/models/Ar_DC_1d/Chemistry.H:315-506).  The thread's species arrays live in
// shared memory with a stride of the block size ([species][thread]): every thread
// of a warp works on the same reaction at the same time, so sc[reac*st + tid] and
// wd[sp*st + tid] are conflict-free rows, and nothing spills to local memory.
// On entry sc[s*st] holds the number density of species s [1/m^3]; on exit
// wd[s*st] holds rxn_s [1/m^3/s]; returns the energy exchange [W/m^3].
template <int PREC>
__device__ __forceinline__ double chem_cell(double* sc, double* wd, const int st, double Te, double Tg, double EN)
{
    const int ns = c_mech.ns;
    const int eid = c_mech.e_id;
    for (int s = 0; s < ns; s++) {
        sc[s * st] = sc[s * st] * 1.0e-6 / N_A * 1.0e6;
        wd[s * st] = 0.0;
    }
    const double sce = sc[eid * st];
    const double ne = sce * NA_CE;
    const double Ue = 1.5 * Te * ne * KB_CE;
    const double mee_na = Ue / ne * NA_CE;
    const double sefact = (tanh((Te - Tg) / 0.5) + 1.0) / 2.0;
    const double dT = Te - Tg;
    double lnTe, lnTg;
    if (PREC == PREC_FP64) {
        lnTe = log(Te);
        lnTg = log(Tg);
    } else {
        lnTe = log2(Te);
        lnTg = log2(Tg);
    }
    const double invTe = 1.0 / Te, invTg = 1.0 / Tg;
    // the powers of ln(Te_eV) and 1/Te_eV the fit rates share
    // (test/Reactor/CO2_H2_Ar_mechanism_reduced/Chemistry.H:945-952)
    double tep[9], itp[4], teev = 0.0;
    if (c_mech.nfits > 0) fit_powers<PREC>(Te, tep, itp, teev);
    // the field magnitude of the field-driven rates: E = EN N 1e-21
    // (test/verification/Streamer/Chemistry.H:262-264)
    double efm = 0.0;
    if (c_mech.need_en) {
        double mix = 0.0;
        for (int s = 0; s < ns; s++) mix += sc[s * st];
        efm = EN * (mix * N_A) * 1e-21;
    }
    double ee = 0.0;
    const int nr = c_mech.nr;
    for (int r = 0; r < nr; r++) {
        const VdRxnDev& R = c_mech.rxn[r];
        double k;
        if (R.kind == VD_RATE_CONST) {
            k = R.A;
        } else if (R.kind == VD_RATE_TOWNSEND) {
            k = townsend_rate(c_mech.fits[R.fit].jc, efm);
        } else if (R.kind >= VD_RATE_JANEV) {
            k = fit_rate<PREC>(R.kind, c_mech.fits[R.fit], tep, itp, teev);
        } else {
            const bool te = (R.kind == VD_RATE_ARRHENIUS_TE);
            const double lT = te ? lnTe : lnTg;
            const double iT = te ? invTe : invTg;
            if (PREC == PREC_FP64) {
                k = exp(fma(R.b, lT, R.lnA) - R.C * iT);
            } else {
                k = (double)exp2_split(fma(R.b, lT, R.l2A) - R.Cl2 * iT);
            }
        }
        double prod = sc[R.reac[0] * st];
        for (int t = 1; t < R.nreac; t++) prod *= sc[R.reac[t] * st];
        const double q = k * prod;
        for (int t = 0; t < R.nterms; t++) {
            double* w = wd + R.sp[t] * st;
            *w = fma(R.coef[t], q, *w);
        }
        if (R.rxntype == VD_RXN_EXCITATION || R.rxntype == VD_RXN_IONIZATION) {
            ee -= R.ex * q * sefact;
        } else if (R.rxntype == VD_RXN_RECOMB || R.rxntype == VD_RXN_ATTACH) {
            ee -= mee_na * q;
        } else if (R.rxntype == VD_RXN_DETACH) {
            ee += mee_na * q;
        } else if (R.rxntype == VD_RXN_ELASTIC) {
            ee -= R.ex * dT * (sce * sc[R.elidx * st] * k) * NA_CE;
        }
    }
    if (c_mech.elastic_loss) {
        double nd = 0.0;
        for (int s = 0; s < ns; s++) nd += sc[s * st] * N_A;
        // |E| = EN N 1e-21 (the He_RF_1d header's CKWC, Chemistry.H:618); the argon
        // headers pass 0 there, with mobilities that do not read it
        double mu = mob_fp64(eid, Te, nd, Tg, EN * nd * 1.0e-21);
        double nu = -ECHARGE / ME / mu;
        ee -= 1.5 * K_B * sce * N_A * dT * nu * c_mech.elastic_coef;
    }
    for (int s = 0; s < ns; s++) wd[s * st] = wd[s * st] * 1.0e-6 * N_A * 1.0e6;
    return ee;
}

}  // namespace vd
