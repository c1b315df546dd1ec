// Device-side lens-equation pieces (per-lens constants and deflection formulas), shared by the
// deflection kernel (deflect.cu) and the persistent batched sweep (sweep.cu). The formulas and
// their reference sources are documented in deflect.cu.
#pragma once

#include "common.cuh"

namespace lentils {

constexpr int kMaxLensesPerLaunch = 8;
constexpr int kSeriesTerms = 20;  // fixed 20-term series (deflect.c:212)
constexpr int kMaxMultipoleOrder = 12;

struct DevLens {
    int type;
    int order;    // multipoles: highest order
    int same_centre;  // centred where the lens before it (of one launch or sample) is
    double x0, y0;
    float x0h, x0l, y0h, y0l;  // the centre as FP32 pairs: x0 = x0h + x0l to ~2^-48 relative
    float gxh, gxl, gyh, gyl;  // batched sweep: its sample's pixel-grid origin minus the centre
    // PEMD: alpha = conj((amp + ampl) * rs2^h * F(u) * rot / z), see pemd_setup. The second parts
    // hold what FP32 drops of amp and q^2: a rounding of a constant moves every point the same
    // way, where the roundings of the points' own values average out.
    float cth, sth, q2, q2l, cx, cy, amp, ampl;
    int nterms;   // series terms (kSeriesTerms: the full series, complex Horner)
    int tail;     // some points have |u| >= 0.75
    float an[kSeriesTerms];
    double an64[kSeriesTerms], cth64, sth64, cx64, cy64;
    // power of the squared radius (PEMD and multipoles): h = h0 + h1; general: outside the
    // range of pow_pos, powf instead
    float h0, h1;
    int general;
    // shear (ssc = ss c2, sss = ss s2, rounded once)
    float ss, c2, s2, ssc, sss, gks, cgka, sgka, gss, cgsa, sgsa;
    // multipoles: radial and tangential coefficients of (cos m th, sin m th) per order
    float rc[kMaxMultipoleOrder + 1], rs[kMaxMultipoleOrder + 1], tc[kMaxMultipoleOrder + 1],
        ts[kMaxMultipoleOrder + 1];
};

struct DevLensSet {
    int n;
    DevLens l[kMaxLensesPerLaunch];
};

// The lens functions take two points at a time, one per half of a float2, so that most of the
// arithmetic is packed FP32x2 instructions (add, mul, fma on both halves): the deflection is
// bound by instruction issue, and a pair costs little more than one point.
__device__ __forceinline__ float2 splat(float a) { return make_float2(a, a); }
// products with -1 (exact): the packed instructions take no negated operand, and a sign flip
// of each half costs two
__device__ __forceinline__ float2 neg2(float2 a) { return __fmul2_rn(a, splat(-1.f)); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b)
{
    return __ffma2_rn(b, splat(-1.f), a);
}

// x - (hi + lo) for FP32 x and a pair (hi, lo), rounded once: Knuth's two-sum gives
// x - hi = s + e exactly, then s + (e - lo). Exact offsets from a lens centre matter near the
// centre, where the angle of the offset sets the direction of the deflection; this keeps the
// FP32 path off the FP64 units, which on GB300 run at a small fraction of the FP32 rate.
__device__ __forceinline__ float2 offset_f32(float2 x, float hi, float lo)
{
    const float2 nh = splat(-hi);
    const float2 s = __fadd2_rn(x, nh);
    const float2 bp = sub2(s, x);
    const float2 e = __fadd2_rn(sub2(x, sub2(s, bp)), sub2(nh, bp));
    return __fadd2_rn(s, __fadd2_rn(e, splat(-lo)));
}

// 1 / x by the hardware approximation and one Newton step
__device__ __forceinline__ float2 recip2(float2 x)
{
    float2 r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(x.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(x.y));
    const float2 e = __ffma2_rn(neg2(x), r, splat(1.f));
    // the residual is not finite where x is 0, infinite or beyond the approximation's range
    const float2 n = __ffma2_rn(e, r, r);
    return make_float2(fabsf(e.x) < 1.f ? n.x : r.x, fabsf(e.y) < 1.f ? n.y : r.y);
}

// x^(h0 + h1) for x > 0 and |h0| <= 1: x = 2^e m with m in [1/sqrt 2, sqrt 2),
// log2 m = f P(f), f = m - 1, the exponent h (e + log2 m) split into an integer n and
// a rest in [-1/2, 1/2] (h e - n by one fma, so it does not lose the low bits of a large
// product), 2^rest by a polynomial, 2^n through the exponent field. The coefficients are minimax fits
// made one after the other from the constant term, each rounded to FP32 before the next: as they
// stand here log2 m = f P(f) is within 1.5e-9 and 2^y within 3.0e-9 (relative), evaluated exactly.
// A fixed error of the power moves all points near a radius the same way, so it is kept below the
// rounding of single points.
__device__ __forceinline__ float2 pow_pos(float2 x, float h0, float h1)
{
    const int ix = __float_as_int(x.x), iy = __float_as_int(x.y);
    const int ex = (ix - 0x3f3504f3) >> 23, ey = (iy - 0x3f3504f3) >> 23;
    const float2 f = __fadd2_rn(make_float2(__int_as_float(ix - (ex << 23)),
                                            __int_as_float(iy - (ey << 23))), splat(-1.f));
    // (float)e through the mantissa of 1.5 * 2^23
    const float2 e = __fadd2_rn(make_float2(__int_as_float(0x4b400000 + ex),
                                            __int_as_float(0x4b400000 + ey)),
                                splat(-12582912.f));
    float2 p = splat(-0.10772465169429779f);
    p = __ffma2_rn(p, f, splat(0.18571536242961884f));
    p = __ffma2_rn(p, f, splat(-0.19199073314666748f));
    p = __ffma2_rn(p, f, splat(0.2048441469669342f));
    p = __ffma2_rn(p, f, splat(-0.23951542377471924f));
    p = __ffma2_rn(p, f, splat(0.28853684663772583f));
    p = __ffma2_rn(p, f, splat(-0.36070021986961365f));
    p = __ffma2_rn(p, f, splat(0.4808996021747589f));
    p = __ffma2_rn(p, f, splat(-0.7213473320007324f));
    p = __ffma2_rn(p, f, splat(1.4426950216293335f));
    const float2 l = __fmul2_rn(p, f);  // log2 m
    const float2 h = splat(h0);
    const float2 c = __ffma2_rn(h, l, __fmul2_rn(splat(h1), __fadd2_rn(e, l)));
    const float2 tm = __fadd2_rn(__ffma2_rn(h, e, c), splat(12582912.f));  // rounds to integers
    const float2 nn = sub2(splat(12582912.f), tm);  // -n
    const float2 y = __fadd2_rn(__ffma2_rn(h, e, nn), c);
    float2 r = splat(0.00015326471475418657f);
    r = __ffma2_rn(r, y, splat(0.0013390806270763278f));
    r = __ffma2_rn(r, y, splat(0.009618505835533142f));
    r = __ffma2_rn(r, y, splat(0.05550359934568405f));
    r = __ffma2_rn(r, y, splat(0.24022647738456726f));
    r = __ffma2_rn(r, y, splat(0.6931471824645996f));
    r = __ffma2_rn(r, y, splat(1.f));
    const float2 sc = make_float2(__int_as_float((__float_as_int(tm.x) << 23) + 0x3f800000),
                                  __int_as_float((__float_as_int(tm.y) << 23) + 0x3f800000));
    return __fmul2_rn(r, sc);
}

__device__ __forceinline__ float2 lens_power(const DevLens &L, float2 r2)
{
    if (L.general) {
        const float h = L.h0 + L.h1;
        return make_float2(powf(r2.x, h), powf(r2.y, h));
    }
    return pow_pos(r2, L.h0, L.h1);
}

// sum_k an[k] u^k over NT real coefficients at complex u, by synthetic division by
// (v - u)(v - conj u) = v^2 - 2 Re(u) v + |u|^2: two real multiply-adds per term where complex
// Horner takes four.
template <int NT, int NP>
__device__ __forceinline__ void series_real(const DevLens &L, const float2 (&ur)[NP],
                                            const float2 (&ui)[NP], float2 (&fr)[NP],
                                            float2 (&fi)[NP])
{
    float2 r[NP], s[NP], b1[NP], b2[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        r[q] = __fadd2_rn(ur[q], ur[q]);
        s[q] = neg2(__ffma2_rn(ur[q], ur[q], __fmul2_rn(ui[q], ui[q])));
        b2[q] = splat(L.an[NT - 1]);
        b1[q] = __ffma2_rn(r[q], b2[q], splat(L.an[NT - 2]));
    }
#pragma unroll
    for (int k = NT - 3; k >= 1; --k) {
        const float2 a = splat(L.an[k]);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const float2 b0 = __ffma2_rn(r[q], b1[q], __ffma2_rn(s[q], b2[q], a));
            b2[q] = b1[q];
            b1[q] = b0;
        }
    }
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        fr[q] = __ffma2_rn(b1[q], ur[q], __ffma2_rn(s[q], b2[q], splat(L.an[0])));
        fi[q] = __fmul2_rn(b1[q], ui[q]);
    }
}

// The full series by complex Horner.
template <int NP>
__device__ __forceinline__ void series_full(const DevLens &L, const float2 (&ur)[NP],
                                            const float2 (&ui)[NP], float2 (&fr)[NP],
                                            float2 (&fi)[NP])
{
    float2 nui[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        nui[q] = neg2(ui[q]);
        fr[q] = splat(L.an[kSeriesTerms - 1]);
        fi[q] = splat(0.f);
    }
#pragma unroll
    for (int n = kSeriesTerms - 2; n >= 0; --n) {
        const float2 a = splat(L.an[n]);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const float2 tr = __ffma2_rn(fr[q], ur[q], __ffma2_rn(fi[q], nui[q], a));
            fi[q] = __ffma2_rn(fr[q], ui[q], __fmul2_rn(fi[q], ur[q]));
            fr[q] = tr;
        }
    }
}

// The series near and beyond |u| = 1 (the tail, q < 0.4), in FP64 from the FP64 offset: there
// the 20 terms amplify a rounding of u up to 20 times. By synthetic division, as series_real.
static __device__ __forceinline__ float2 series_tail(const DevLens &L, double dx, double dy)
{
    const double X = dx * L.cth64 + dy * L.sth64, Y = dy * L.cth64 - dx * L.sth64;
    const double inv = 1.0 / (X * X + Y * Y);
    const double ur = (L.cx64 * X * X + L.cy64 * Y * Y) * inv;
    const double ui = (L.cy64 - L.cx64) * X * Y * inv;
    const double r = 2.0 * ur, s = -(ur * ur + ui * ui);
    double b2 = L.an64[kSeriesTerms - 1], b1 = fma(r, b2, L.an64[kSeriesTerms - 2]);
    for (int k = kSeriesTerms - 3; k >= 1; --k) {
        const double b0 = fma(r, b1, fma(s, b2, L.an64[k]));
        b2 = b1;
        b1 = b0;
    }
    return make_float2((float)fma(b1, ur, fma(s, b2, L.an64[0])), (float)(b1 * ui));
}

// PEMD. With z = X + iY the offset in the rotated frame and r_s^2 = q^2 X^2 + Y^2, the argument
// of the series is u = (1 - sqrt(1 - w^2)) / 2, w^2 = (1 - q^2) / q^2 * r_s^2 / z^2. Since
// z^2 - (1 - q^2) / q^2 r_s^2 = (qX + iY/q)^2 and qX + iY/q has a positive component along z,
// the principal root is (qX + iY/q) / z exactly, so
//   u = (cx X + i cy Y) / z,   cx = (1 - q) / 2, cy = (1 - 1/q) / 2,
// without a complex square root, and |u| <= max(|cx|, |cy|) at every point: the number of
// series terms that FP32 can tell apart follows from q alone (build_lens). The prefactor
// b'^2 / (q z) (b' / r_s)^(t - 2) is amp (r_s^2)^h / z, h = (2 - t) / 2, amp = b'^t / q.
// One reciprocal, of |z|^2, serves both quotients. Gives z, u and a = (amp + ampl)
// (r_s^2)^h / |z|^2. The low parts of amp and q^2 enter by products that are rounded once together
// with the high ones: added to a product rounded before, they would be below half its last place.
__device__ __forceinline__ void pemd_setup(const DevLens &L, float2 dx, float2 dy, float2 ct,
                                           float2 st, float2 ns, float2 &X, float2 &Y,
                                           float2 &ur, float2 &ui, float2 &a)
{
    X = __ffma2_rn(dx, ct, __fmul2_rn(dy, st));  // z = (dx + i dy) (cth - i sth)
    Y = __ffma2_rn(dy, ct, __fmul2_rn(dx, ns));
    const float2 xx = __fmul2_rn(X, X), yy = __fmul2_rn(Y, Y), xy = __fmul2_rn(X, Y);
    const float2 rs2 = __fadd2_rn(__ffma2_rn(splat(L.q2), xx, __fmul2_rn(splat(L.q2l), xx)), yy);
    const float2 pw = lens_power(L, rs2);
    const float2 inv = recip2(__fadd2_rn(xx, yy));
    ur = __fmul2_rn(__ffma2_rn(splat(L.cx), xx, __fmul2_rn(splat(L.cy), yy)), inv);
    ui = __fmul2_rn(__fmul2_rn(splat(L.cy - L.cx), xy), inv);
    a = __fmul2_rn(__ffma2_rn(splat(L.amp), pw, __fmul2_rn(splat(L.ampl), pw)), inv);
}

__device__ __forceinline__ void shear_alpha(const DevLens &L, float sx, float sy, float &ax,
                                            float &ay)
{
    ax = L.ss * (L.c2 * sx + L.s2 * sy);
    ay = L.ss * (L.s2 * sx - L.c2 * sy);
    if (L.gks != 0.f) {
        const float rx = sx * L.cgka + sy * L.sgka;
        const float ry = -sx * L.sgka + sy * L.cgka;
        const float dx = -0.25f * L.gks * (3.f * rx * rx + ry * ry);
        const float dy = -0.5f * L.gks * rx * ry;
        ax += dx * L.cgka - dy * L.sgka;
        ay += dx * L.sgka + dy * L.cgka;
    }
    if (L.gss != 0.f) {
        const float rx = sx * L.cgsa + sy * L.sgsa;
        const float ry = -sx * L.sgsa + sy * L.cgsa;
        const float dx = -0.5f * L.gss * (rx * rx - ry * ry);
        const float dy = L.gss * rx * ry;
        ax += dx * L.cgsa - dy * L.sgsa;
        ay += dx * L.sgsa + dy * L.cgsa;
    }
}

// Multipoles at a point whose squared distance from the centre is not a normal FP32 number: the
// same sums by a scaled offset and the library's functions. Not inlined: rare.
static __device__ __noinline__ float2 multipole_scaled(const DevLens &L, float sx, float sy)
{
    if (L.order < 3) return make_float2(0.f, 0.f);
    const float up = 0x1p+100f, top = fmaxf(fabsf(sx), fabsf(sy));
    const float k = top < 1.f ? up : 1.f / up;
    const float x = sx * k, y = sy * k, r = sqrtf(fmaf(x, x, y * y));
    const float cn = x / r, sn = y / r;
    const float h = 2.f * (L.h0 + L.h1);
    const float rp = powf(r, h) * (k == up ? powf(1.f / up, h) : powf(up, h));
    float cm = cn * cn - sn * sn, sm = 2.f * cn * sn, dr = 0.f, dt = 0.f;
    for (int m = 3; m <= L.order; ++m) {
        const float c = cm * cn - sm * sn;
        sm = cm * sn + sm * cn;
        cm = c;
        dr = fmaf(L.rc[m], cm, fmaf(L.rs[m], sm, dr));
        dt = fmaf(L.tc[m], cm, fmaf(L.ts[m], sm, dt));
    }
    return make_float2(rp * (cn * dr - sn * dt), rp * (sn * dr + cn * dt));
}

// Internal multipoles: with e = (sx + i sy) / r, cos m th and sin m th are the parts of e^m
// (one complex product per order, no angle), and r^(1 - alpha) = (r^2)^h, h = (1 - alpha) / 2.
// A squared radius outside the normal FP32 numbers (r below 1.1e-19 or above 1.8e19) would make the
// reciprocal root 0 or infinite: those points are done again by multipole_scaled.
template <int NP>
__device__ __forceinline__ void multipole_alpha(const DevLens &L, const float2 (&sx)[NP],
                                                const float2 (&sy)[NP], float2 (&ax)[NP],
                                                float2 (&ay)[NP])
{
    float2 rp[NP], cn[NP], sn[NP], nsn[NP], cm[NP], sm[NP], dr[NP], dt[NP];
    auto normal = [](float a, float b) {  // both
        return fminf(a, b) >= 0x1p-126f && fmaxf(a, b) <= 3.402823466e38f;
    };
    bool all = true;
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        const float2 r2 = __ffma2_rn(sx[q], sx[q], __fmul2_rn(sy[q], sy[q]));
        all = all && normal(r2.x, r2.y);
        rp[q] = lens_power(L, r2);
        float2 ri;
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(ri.x) : "f"(r2.x));
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(ri.y) : "f"(r2.y));
        // one Newton step: ri += ri (1 - r2 ri^2) / 2
        const float2 t = __ffma2_rn(neg2(__fmul2_rn(r2, ri)), ri, splat(1.f));
        ri = __ffma2_rn(__fmul2_rn(splat(0.5f), ri), t, ri);
        cn[q] = __fmul2_rn(sx[q], ri);
        sn[q] = __fmul2_rn(sy[q], ri);
        nsn[q] = neg2(sn[q]);
        cm[q] = __ffma2_rn(cn[q], cn[q], __fmul2_rn(nsn[q], sn[q]));
        sm[q] = __fmul2_rn(__fadd2_rn(cn[q], cn[q]), sn[q]);
        dr[q] = dt[q] = splat(0.f);
    }
    for (int m = 3; m <= L.order; ++m) {
        const float2 rc = splat(L.rc[m]), rs = splat(L.rs[m]);
        const float2 tc = splat(L.tc[m]), ts = splat(L.ts[m]);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const float2 c = __ffma2_rn(cm[q], cn[q], __fmul2_rn(sm[q], nsn[q]));
            sm[q] = __ffma2_rn(cm[q], sn[q], __fmul2_rn(sm[q], cn[q]));
            cm[q] = c;
            dr[q] = __ffma2_rn(rc, cm[q], __ffma2_rn(rs, sm[q], dr[q]));
            dt[q] = __ffma2_rn(tc, cm[q], __ffma2_rn(ts, sm[q], dt[q]));
        }
    }
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        ax[q] = __fmul2_rn(rp[q], __ffma2_rn(cn[q], dr[q], __fmul2_rn(nsn[q], dt[q])));
        ay[q] = __fmul2_rn(rp[q], __ffma2_rn(sn[q], dr[q], __fmul2_rn(cn[q], dt[q])));
    }
    if (!all) {
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const float2 r2 = __ffma2_rn(sx[q], sx[q], __fmul2_rn(sy[q], sy[q]));
            if (!normal(r2.x, r2.x)) {
                const float2 a = multipole_scaled(L, sx[q].x, sy[q].x);
                ax[q].x = a.x;
                ay[q].x = a.y;
            }
            if (!normal(r2.y, r2.y)) {
                const float2 a = multipole_scaled(L, sx[q].y, sy[q].y);
                ax[q].y = a.x;
                ay[q].y = a.y;
            }
        }
    }
}

// per-lens constants from the reference's packed parameters (host, FP64)
int build_lens(const lentils_mass_model &m, DevLens &L);

// alpha of one lens at NP pairs of offsets (sx, sy) from its centre; tail(L, q, h): series_tail
// of point h of pair q
template <int NP, class Tail>
__device__ __forceinline__ void lens_alpha(const DevLens &L, const float2 (&sx)[NP],
                                           const float2 (&sy)[NP], Tail tail, float2 (&ax)[NP],
                                           float2 (&ay)[NP])
{
    if (L.type == 0) {
        float2 fr[NP], fi[NP], ur[NP], ui[NP], X[NP], Y[NP], a[NP];
        const float2 ct = splat(L.cth), st = splat(L.sth), ns = splat(-L.sth);
#pragma unroll
        for (int q = 0; q < NP; ++q)
            pemd_setup(L, sx[q], sy[q], ct, st, ns, X[q], Y[q], ur[q], ui[q], a[q]);
        if (L.nterms == 8) {
            series_real<8, NP>(L, ur, ui, fr, fi);
        } else if (L.nterms == 12) {
            series_real<12, NP>(L, ur, ui, fr, fi);
        } else if (L.nterms == 16) {
            series_real<16, NP>(L, ur, ui, fr, fi);
        } else {
            series_full<NP>(L, ur, ui, fr, fi);
            if (L.tail) {
#pragma unroll
                for (int q = 0; q < NP; ++q) {
                    if (!(ur[q].x * ur[q].x + ui[q].x * ui[q].x < 0.5625f)) {
                        const float2 f = tail(L, q, 0);
                        fr[q].x = f.x;
                        fi[q].x = f.y;
                    }
                    if (!(ur[q].y * ur[q].y + ui[q].y * ui[q].y < 0.5625f)) {
                        const float2 f = tail(L, q, 1);
                        fr[q].y = f.x;
                        fi[q].y = f.y;
                    }
                }
            }
        }
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            // alpha = conj(a F conj(z) rot), rot = cth - i sth
            const float2 gr = __fmul2_rn(a[q], __ffma2_rn(fr[q], X[q], __fmul2_rn(fi[q], Y[q])));
            const float2 gn = __fmul2_rn(a[q], __ffma2_rn(fr[q], Y[q],
                                                          neg2(__fmul2_rn(fi[q], X[q]))));
            ax[q] = __ffma2_rn(gr, ct, __fmul2_rn(gn, ns));
            ay[q] = __ffma2_rn(gr, st, __fmul2_rn(gn, ct));
        }
    } else if (L.type == 1) {
        if (L.gks == 0.f && L.gss == 0.f) {
            const float2 sc = splat(L.ssc), s2 = splat(L.sss), nc = splat(-L.ssc);
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                ax[q] = __ffma2_rn(sc, sx[q], __fmul2_rn(s2, sy[q]));
                ay[q] = __ffma2_rn(s2, sx[q], __fmul2_rn(nc, sy[q]));
            }
        } else {
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                shear_alpha(L, sx[q].x, sy[q].x, ax[q].x, ay[q].x);
                shear_alpha(L, sx[q].y, sy[q].y, ax[q].y, ay[q].y);
            }
        }
    } else {
        multipole_alpha<NP>(L, sx, sy, ax, ay);
    }
}

}  // namespace lentils
