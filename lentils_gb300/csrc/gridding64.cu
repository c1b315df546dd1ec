// The FP64 operators (degrid64, grid64) in pairs of FP32 values.
//
// GB300 runs two FP64 multiply-adds per SM and clock against 128 in FP32, so FP64 kernels are
// bound by that pipe whatever else they do: at 2e6 visibilities and 2w = 8 they took 905 us
// (degrid) and 1170 us (grid). Here every FP64 number is an unevaluated sum h + l of two FP32
// values (48 bits), and the window sums run on the FP32 pipe, two components per packed
// instruction:
//   mac:  the high half of a sum carries a bias B = 1.5 * 2^m that keeps it in one binade, so
//         s = fl(w g + r) rounds to the last place of B, s - r is exact, and one more fma gives
//         the product's remainder; that and the cross terms wh gl + wl gh collect in the low
//         half. Six packed instructions per complex tap (a sum without bias takes eleven: the
//         product's own rounding and Knuth's two-sum).
// The bias follows the data, the real and the imaginary part each: in degridding the largest value
// of each row of the visibility's own window, in gridding the sums so far and the largest of the
// next visibilities of the same cell, so the rounding is relative to values that reach the same
// results.
// The weights are fits of degree 11 here, 9 in the FP64 kernels. Largest difference from the
// profile, in units of its peak, beta = 2.34 (2w), degree 11 and 9: w = 1: 3.9e-10 and 4.4e-8; 2:
// 4.0e-11 and 5.0e-9; 3: 4.6e-12 and 5.4e-10; 4: 4.5e-13 and 1.1e-10 (the NUFFT's own beta at padding
// 2 to 4: 2.5e-11 to 4.3e-10, 2.8e-11 to 1.0e-10, 4.0e-12 to 1.7e-11, 4.2e-13 to 3.1e-12). The
// pairs' rounding, about 1e-14 of the result, is below that at every width, so the operators are
// closer to the definition than in FP64 with the shorter fits, though a value has 48 bits for 53.
// F^T F of a 512^2 image with 2e6 visibilities (w = 4): degridding 905 -> 137 us, gridding 1170 ->
// 227 us (the rest of the operator's 2410 -> 495 us is its FFT, 340 -> 130); relative error against
// direct FP64 sums 8.6e-13 -> 2.4e-14.
//
// Range. FP32 exponents do not cover FP64's, so a work item scales its tile (degrid) or its
// visibilities (grid) by the power of two that brings the largest finite one to [1, 2) and the
// result back. A value keeps all 48 bits down to 2^-77 of that largest value. What lies below it
// (far(): subnormals too) does not go through pairs: a tile with such a value is degridded in
// FP64, and such a visibility is added to the grid in FP64, with the same weights. Infinities and
// NaN go through as such: where the high half of a result is not finite it is the result.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "gridding_items.cuh"

namespace lentils {

struct DS {  // two (packed) numbers, each h + l
    float2 h, l;
};

__device__ __forceinline__ float2 minus(float2 a, float2 b)  // a - b in one packed instruction
{
    return __ffma2_rn(b, f2(-1.f), a);
}

// r += (wh + wl) * (gh + gl), r.h biased
__device__ __forceinline__ void ds_mac(float wh, float wl, const DS &g, DS &r)
{
    const float2 w = f2(wh);
    const float2 s = __ffma2_rn(w, g.h, r.h);
    const float2 e = __ffma2_rn(w, g.h, minus(r.h, s));  // what the sum lost of the product
    r.l = __ffma2_rn(f2(wl), g.h, __ffma2_rn(w, g.l, __fadd2_rn(r.l, e)));
    r.h = s;
}

// The bias 1.5 * 2^m with 2^(m - 1) above |bound|, per part.
__device__ __forceinline__ float bias(float bound)
{
    return __int_as_float((((__float_as_int(bound) >> 23) + 2) << 23) | 0x400000);
}
__device__ __forceinline__ float2 bias(float2 bound)
{
    return make_float2(bias(bound.x), bias(bound.y));
}

// Biased exponents of the real and the imaginary part, in the halves of a word (maxima by
// __vmaxu2), and the powers of two above the values of such exponents. The parts are separate sums:
// each has its own bias.
__device__ __forceinline__ unsigned exponents(int re, int im)
{
    return (unsigned)re | (unsigned)im << 16;
}
__device__ __forceinline__ float2 above(unsigned e)
{
    return make_float2(__int_as_float((int)((e & 0xffff) + 1) << 23),
                       __int_as_float((int)((e >> 16) + 1) << 23));
}

__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= 3.402823466e38f; }

// a + b, renormalised (not where the sum is not finite: its low half is NaN)
__device__ __forceinline__ DS ds_add(const DS &a, const DS &b)
{
    const float2 s = __fadd2_rn(a.h, b.h);
    const float2 bb = minus(s, a.h);
    const float2 e = __fadd2_rn(minus(a.h, minus(s, bb)), minus(b.h, bb));
    const float2 l = __fadd2_rn(e, __fadd2_rn(a.l, b.l));
    DS r;
    r.h = __fadd2_rn(s, l);
    r.l = minus(l, minus(r.h, s));
    if (!finite(s.x)) r.h.x = s.x;
    if (!finite(s.y)) r.h.y = s.y;
    return r;
}

// Weights of one axis. Horner steps with the high halves on a fixed grid per tap: the table
// holds each coefficient as cb = c_h + B and c_l, with B = 1.5 * 2^m large enough that every
// partial value stays in B's binade (as in ds_mac): seven packed instructions for two taps.
template <int W2>
__device__ __forceinline__ void ds_weights(const KBPolyDS &kb, uint32_t word, float res,
                                           float (&wh)[W2], float (&wl)[W2])
{
    constexpr int w = W2 / 2;
    // t = 2 frac - 1 + 2 res: the first part is exact in FP32
    const float th = (float)(2 * (int)(word & kFracMask) - (1 << kFracBits)) *
                     (1.0f / (float)(1u << kFracBits));
    const float tl = 2.0f * res;
    const float uh = th * th;
    const float ul = fmaf(2.0f * th, tl, fmaf(th, th, -uh));
    const float2 UH = f2(uh), UL = f2(ul), TH = f2(th), TL = f2(tl);
#pragma unroll
    for (int p = 0; p < (w + 1) / 2; ++p) {
        const float2 nB = kb.nb[p], B = kb.b[p];
        auto horner = [&](const float2 (&cb)[kDsHalf][kMaxDsTaps / 2],
                          const float2 (&cl)[kDsHalf][kMaxDsTaps / 2]) {
            DS e;
            e.h = cb[0][p];  // the leading coefficient, without B
            e.l = cl[0][p];
#pragma unroll
            for (int k = 1; k < kDsHalf; ++k) {
                const float2 s = __ffma2_rn(e.h, UH, cb[k][p]);
                const float2 e1 = __ffma2_rn(e.h, UH, minus(cb[k][p], s));
                e.l = __ffma2_rn(e.l, UH, __ffma2_rn(e.h, UL, __fadd2_rn(e1, cl[k][p])));
                e.h = __fadd2_rn(s, nB);
            }
            return e;
        };
        const DS e = horner(kb.eb, kb.el), o = horner(kb.ob, kb.ol);
        // taps i and 2w-1-i: t o + e and t o - e
        const float2 d = __fadd2_rn(__ffma2_rn(o.h, TH, B), nB);
        const float2 dl = __ffma2_rn(o.h, TL, __ffma2_rn(o.l, TH,
                                                         __ffma2_rn(o.h, TH, minus(f2(0.f), d))));
        const float2 loh = __fadd2_rn(d, e.h), lol = __fadd2_rn(dl, e.l);
        const float2 hih = minus(d, e.h), hil = minus(dl, e.l);
        wh[2 * p] = loh.x;
        wl[2 * p] = lol.x;
        wh[W2 - 1 - 2 * p] = hih.x;
        wl[W2 - 1 - 2 * p] = hil.x;
        if (2 * p + 1 < w) {
            wh[2 * p + 1] = loh.y;
            wl[2 * p + 1] = lol.y;
            wh[W2 - 2 - 2 * p] = hih.y;
            wl[W2 - 2 - 2 * p] = hil.y;
        }
    }
    if (word & kTopOffBit) wh[W2 - 1] = wl[W2 - 1] = 0.f;
}

// -- FP64 <-> scaled pairs, on the integer and FP32 pipes ------------------------------------
__device__ __forceinline__ int exponent_of(double v)  // biased; 0 for zero, subnormal, not finite
{
    const int e = (__double2hiint(v) >> 20) & 0x7ff;
    return e == 0x7ff ? 0 : e;
}

// whether v is too small beside a value of biased exponent emax for a pair to hold its bits
__device__ __forceinline__ bool far(double v, int emax)
{
    const int e = (__double2hiint(v) >> 20) & 0x7ff;
    return e < max(1, emax - 77) && v != 0.0;
}

// v * 2^(1023 - emax) as h + l (emax: biased exponent of the largest value, at least 1)
__device__ __forceinline__ void split(double v, int emax, float &h, float &l)
{
    const int hi = __double2hiint(v), lo = __double2loint(v);
    const int e = (hi >> 20) & 0x7ff;
    const int sign = hi & 0x80000000;
    const int fe = e - emax + 127;
    if (e == 0x7ff) {  // infinity or NaN
        h = __int_as_float(sign | 0x7f800000 | (((hi & 0xfffff) | lo) ? 0x400000 : 0));
        l = 0.f;
        return;
    }
    if (e == 0 || fe <= 0) {
        h = l = 0.f;
        return;
    }
    const int scale = fe << 23;  // 2^(e - emax)
    // 52-bit mantissa: the upper 23 bits and the lower 29
    const int m_hi = ((hi & 0xfffff) << 3) | (int)((unsigned)lo >> 29);
    h = __int_as_float(sign | scale | m_hi);
    const float r = (float)(lo & 0x1fffffff) * (1.0f / 4503599627370496.0f);  // * 2^-52
    l = r * __int_as_float(sign | scale);
}

__device__ __forceinline__ double join(float h, float l, double s1, double s2)
{
    const double v = finite(h) ? (double)h + (double)l : (double)h;
    return v * s1 * s2;
}

__device__ __forceinline__ double pow2(int e)  // |e| <= 1022
{
    return __hiloint2double((e + 1023) << 20, 0);
}

// Largest biased exponent over the CTA (>= 1); red: one int per warp
__device__ __forceinline__ int block_max_exponent(int e, int *red)
{
    e = __reduce_max_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
    __syncthreads();
    int m = 1;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) m = max(m, red[q]);
    return m;
}

// (Both kernels let the next one start when they end, pdl_wait: see fft2d.cu.)
constexpr int kDsThreads = 128;

// Cell (ea, eb) of the extended tile at (a0, b0), through the Hermitian fold.
__device__ __forceinline__ double2 tile_cell(const double2 *__restrict__ grid, const GridGeom &g,
                                             int a0, int b0, int ea, int eb)
{
    int au = wrap_index(a0 + ea, g.nu), bv = wrap_index(b0 + eb, g.nv);
    const bool conj = bv >= g.half_nv;
    if (conj) {
        au = (g.nu - au) % g.nu;
        bv = g.nv - bv;
    }
    double2 v = grid[(long long)au * g.half_nv + bv];
    if (conj) v.y = -v.y;
    return v;
}

// The item of degrid_ds_kernel in FP64, with the same weights: tiles whose values span more than
// the pairs' range. Rare, and not inlined, so that the paired path keeps its registers.
template <int W2>
static __device__ __noinline__ void degrid_far(const double2 *__restrict__ grid,
                                               const uint2 *__restrict__ coords,
                                               const float2 *__restrict__ cres,
                                               double2 *__restrict__ out,
                                               const WorkItem *__restrict__ items,
                                               const KBPolyDS &kb, const GridGeom &g,
                                               const double *__restrict__ vscale,
                                               unsigned char *smraw)
{
    constexpr int w = W2 / 2;
    double2 *sm = reinterpret_cast<double2 *>(smraw);  // as many bytes as the pairs
    const WorkItem it = items[blockIdx.x];
    const int a0 = it.tu * g.T - g.Hu - w, b0 = it.tv * g.T - g.Hv - w, E = g.E, S = g.stride;
    for (int e = threadIdx.x; e < E * E; e += kDsThreads)
        sm[e / E * S + e % E] = tile_cell(grid, g, a0, b0, e / E, e % E);
    __syncthreads();
    for (int k = threadIdx.x; k < it.count; k += kDsThreads) {
        const uint2 c = coords[it.begin + k];
        const float2 rr = cres[it.begin + k];
        const int lu = cell_of(c.x), lv = cell_of(c.y);
        float uh[W2], ul[W2], vh[W2], vl[W2];
        ds_weights<W2>(kb, c.y, rr.y, vh, vl);
        ds_weights<W2>(kb, c.x, rr.x, uh, ul);
        double wv[W2], re = 0.0, im = 0.0;  // wv with scale2: subnormal cells keep their bits
#pragma unroll
        for (int j = 0; j < W2; ++j) wv[j] = ((double)vh[j] + (double)vl[j]) * kb.scale2;
        auto row = [&](double wu, const double2 *p) {
            double tr = 0.0, ti = 0.0;
#pragma unroll
            for (int j = 0; j < W2; ++j) {
                tr = fma(wv[j], p[j].x, tr);
                ti = fma(wv[j], p[j].y, ti);
            }
            re = fma(wu, tr, re);
            im = fma(wu, ti, im);
        };
        const double2 *p = sm + (lu + 1) * S + (lv + 1);
#pragma unroll
        for (int i = 0; i < W2; ++i) row((double)uh[i] + (double)ul[i], p + i * S);
        if (c.x & kExtraTapBit) row(kb.edge, p - S);
        if (c.y & kExtraTapBit) {
            auto column = [&](double wu, const double2 &q) {
                re = fma(wu * kb.edge * kb.scale2, q.x, re);
                im = fma(wu * kb.edge * kb.scale2, q.y, im);
            };
#pragma unroll
            for (int i = 0; i < W2; ++i) column((double)uh[i] + (double)ul[i], p[i * S - 1]);
            if (c.x & kExtraTapBit) column(kb.edge, p[-S - 1]);
        }
        double sc = tap_parity(it, g, lu, lv) ? -1.0 : 1.0;
        if (vscale) sc *= vscale[it.begin + k];
        out[it.begin + k] = make_double2(re * sc, im * sc);
    }
}

// Degridding: one visibility per thread over the staged tile (as degrid_item). Bound by the
// FP32 pipe: about 450 packed instructions for the taps and 630 for the weights of a
// visibility.
template <int W2>
__global__ void __launch_bounds__(kDsThreads, W2 == 6 ? 3 : 4)  // 4 would spill at 2w = 6
    degrid_ds_kernel(const double2 *__restrict__ grid, const uint2 *__restrict__ coords,
                     const float2 *__restrict__ cres, double2 *__restrict__ out,
                     const WorkItem *__restrict__ items, const __grid_constant__ KBPolyDS kb,
                     const __grid_constant__ GridGeom g, const double *__restrict__ vscale)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    float4 *sm = reinterpret_cast<float4 *>(smraw);  // (h.re, h.im, l.re, l.im) per cell
    // largest exponents (biased; real, imaginary) of the 2w cells of a row that a cell's window
    // covers, E x T
    uchar2 *rowmax = reinterpret_cast<uchar2 *>(sm + g.E * g.stride);
    __shared__ int red[kDsThreads / 32];
    constexpr int w = W2 / 2;
    pdl_wait();
    const WorkItem it = items[blockIdx.x];
    const int a0 = it.tu * g.T - g.Hu - w, b0 = it.tv * g.T - g.Hv - w;
    const int E = g.E, S = g.stride;
    int emax = 0;
    for (int e = threadIdx.x; e < E * E; e += kDsThreads) {
        const double2 v = tile_cell(grid, g, a0, b0, e / E, e % E);
        emax = max(emax, max(exponent_of(v.x), exponent_of(v.y)));
    }
    emax = block_max_exponent(emax, red);
    bool out_of_range = false;
    for (int e = threadIdx.x; e < E * E; e += kDsThreads) {
        const int ea = e / E, eb = e - ea * E;
        const double2 v = tile_cell(grid, g, a0, b0, ea, eb);
        out_of_range |= far(v.x, emax) || far(v.y, emax);
        float4 q;
        split(v.x, emax, q.x, q.z);
        split(v.y, emax, q.y, q.w);
        sm[ea * S + eb] = q;
    }
    if (__syncthreads_or(out_of_range)) {
        degrid_far<W2>(grid, coords, cres, out, items, kb, g, vscale, smraw);
        return;
    }
    auto of_cell = [](const float4 &q) {  // 0 where a part is not finite
        const int a = (__float_as_int(q.x) >> 23) & 0xff, b = (__float_as_int(q.y) >> 23) & 0xff;
        return exponents(a == 0xff ? 0 : a, b == 0xff ? 0 : b);
    };
    const int T = g.T;
    for (int e = threadIdx.x; e < E * T; e += kDsThreads) {
        const int ea = e / T, lv = e - ea * T;
        unsigned m = 0;
#pragma unroll
        for (int j = 0; j < W2; ++j) m = __vmaxu2(m, of_cell(sm[ea * S + lv + 1 + j]));
        rowmax[e] = make_uchar2(m & 0xff, m >> 16);
    }
    __syncthreads();
    const int es = emax - 1023;
    const double s1 = pow2(es / 2), s2 = pow2(es - es / 2) * kb.scale2;
    for (int k = threadIdx.x; k < it.count; k += kDsThreads) {
        const uint2 c = coords[it.begin + k];
        const float2 rr = cres[it.begin + k];
        const int lu = cell_of(c.x), lv = cell_of(c.y);
        float uh[W2], ul[W2], vh[W2], vl[W2];
        ds_weights<W2>(kb, c.y, rr.y, vh, vl);
        ds_weights<W2>(kb, c.x, rr.x, uh, ul);
        const float4 *p = sm + (lu + 1) * S + (lv + 1);
        // the cells of a window row are below 2^(e - 126) and the v-weights sum to less than 1;
        // the window's sum is below the sum of the rows' bounds times the u-weights
        const uchar2 *rm = rowmax + (lu + 1) * T + lv;
        auto row_above = [&](int i) { return above(exponents(rm[i * T].x, rm[i * T].y)); };
        float2 bound = f2(0.f);
#pragma unroll
        for (int i = 0; i < W2; ++i) bound = __ffma2_rn(f2(fabsf(uh[i])), row_above(i), bound);
        const float2 BA = bias(bound);
        DS acc{BA, f2(0.f)};
#pragma unroll
        for (int i = 0; i < W2; ++i) {
            // (a row's bound is a power of two: half of it has the bias that its exponent asks for)
            const float2 B = bias(__fmul2_rn(f2(0.5f), row_above(i)));
            DS r{B, f2(0.f)};
#pragma unroll
            for (int j = 0; j < W2; ++j) {
                const float4 q = p[i * S + j];
                ds_mac(vh[j], vl[j], DS{make_float2(q.x, q.y), make_float2(q.z, q.w)}, r);
            }
            r.h = minus(r.h, B);
            ds_mac(uh[i], ul[i], r, acc);
        }
        acc.h = minus(acc.h, BA);
        double re, im;
        if ((c.x | c.y) & kExtraTapBit) {
            // the taps at argument +w, in FP64 (coordinates on a cell boundary only)
            const double eu = (c.x & kExtraTapBit) ? kb.edge : 0.0;
            const double ev = (c.y & kExtraTapBit) ? kb.edge : 0.0;
            const float4 *q = sm + lu * S + lv;
            double tr = 0.0, ti = 0.0;
            auto add = [&](double wt, const float4 &f) {
                tr += wt * ((double)f.x + (double)f.z);
                ti += wt * ((double)f.y + (double)f.w);
            };
            if (eu != 0.0) {
                for (int j = 0; j < W2; ++j) add(eu * ((double)vh[j] + (double)vl[j]), q[j + 1]);
                add(eu * ev, q[0]);
            }
            if (ev != 0.0)
                for (int i = 0; i < W2; ++i)
                    add(ev * ((double)uh[i] + (double)ul[i]), q[(i + 1) * S]);
            re = (join(acc.h.x, acc.l.x, 1.0, 1.0) + tr) * s1 * s2;
            im = (join(acc.h.y, acc.l.y, 1.0, 1.0) + ti) * s1 * s2;
        } else {
            re = join(acc.h.x, acc.l.x, s1, s2);
            im = join(acc.h.y, acc.l.y, s1, s2);
        }
        if (tap_parity(it, g, lu, lv)) {
            re = -re;
            im = -im;
        }
        if (vscale) {
            const double sc = vscale[it.begin + k];
            re *= sc;
            im *= sc;
        }
        out[it.begin + k] = make_double2(re, im);
    }
}

// One visibility's row in the gridding batch, in floats:
//   [vh | vl] (padded to 4 each), (uh, ul) pairs, x (h.re, h.im, l.re, l.im)
template <int W2>
struct DsRow {
    static constexpr int WP = (W2 + 3) & ~3;
    static constexpr int U = 2 * WP;
    static constexpr int X = U + ((2 * W2 + 3) & ~3);
    static constexpr int LEN = X + 4;
    // an odd number of 16-byte words: the rows a group writes side by side fall in distinct
    // bank quads
    static constexpr int STR = ((LEN / 4) % 2) ? LEN : LEN + 4;
    static constexpr int GSTR = W2 * STR + 8;  // rows of one group; groups 8 banks apart
};

template <int W2>
__host__ __device__ inline size_t grid_ds_smem_bytes(const GridGeom &g)
{
    constexpr int NW = kDsThreads / 32;
    return sizeof(float4) * (size_t)NW * g.E * g.stride +
           sizeof(float) * (size_t)NW * (32 / W2) * DsRow<W2>::GSTR;
}

// Gridding with the data flow of the FP32 row-owner kernels: a group of 2w lanes takes a
// contiguous share of the item's sorted visibilities; its lanes produce the rows of 2w of them
// at a time, then lane i sums window row i in registers while the visibilities stay in one
// cell, and adds the sums to the warp's copy of the tile when the cell changes (the groups of a
// warp in turn). The copies are summed once per item and flushed with FP64 atomics through the
// fold.
template <int W2>
__global__ void __launch_bounds__(kDsThreads, 3)
    grid_ds_kernel(const double2 *__restrict__ vis, const uint2 *__restrict__ coords,
                   const float2 *__restrict__ cres, double2 *__restrict__ grid,
                   const WorkItem *__restrict__ items, const __grid_constant__ KBPolyDS kb,
                   const GridGeom g)
{
    using Row = DsRow<W2>;
    constexpr int w = W2 / 2;
    constexpr int NW = kDsThreads / 32;
    constexpr int G = 32 / W2, NG = NW * G;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ int red[NW];
    pdl_wait();
    const WorkItem it = items[blockIdx.x];
    const int E = g.E, S = g.stride;
    float4 *tiles = reinterpret_cast<float4 *>(smraw);
    float *rows = reinterpret_cast<float *>(tiles + NW * E * S);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float4 *mytile = tiles + warp * E * S;
    for (int e = lane; e < E * S; e += 32) mytile[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    int emax = 0;
    for (int k = threadIdx.x; k < it.count; k += kDsThreads) {
        const double2 v = vis[it.begin + k];
        emax = max(emax, max(exponent_of(v.x), exponent_of(v.y)));
    }
    emax = block_max_exponent(emax, red);
    const int es = emax - 1023 - 1;  // with the factor 1/2 of the gridding
    const double s1 = pow2(es / 2), s2 = pow2(es - es / 2) * kb.scale2;
    const double unscaled = 0.5 * kb.scale2;  // the same for values that are not scaled
    const int a0 = it.tu * g.T - g.Hu - w, b0 = it.tv * g.T - g.Hv - w;
    auto to_grid = [&](int ea, int eb, double re, double im) {
        int au = wrap_index(a0 + ea, g.nu), bv = wrap_index(b0 + eb, g.nv);
        if (bv >= g.half_nv) {
            au = (g.nu - au) % g.nu;
            bv = g.nv - bv;
            im = -im;
        } else if (bv == 0) {
            re *= 2.0;
            im *= 2.0;
        }
        double2 *d = grid + (long long)au * g.half_nv + bv;
        atomicAdd(&d->x, re);
        atomicAdd(&d->y, im);
    };

    const bool lane_on = lane < G * W2;
    const int grp = lane_on ? lane / W2 : G - 1;
    const int ri = lane_on ? lane - grp * W2 : 0;
    const int gid = warp * G + grp;
    const int L = (it.count + NG - 1) / NG;
    const int rbeg = min(it.count, gid * L), rend = lane_on ? min(it.count, rbeg + L) : rbeg;
    const int nbatch = (L + W2 - 1) / W2;
    const unsigned gmask = ((1u << W2) - 1u) << (grp * W2);
    float *rowg = rows + gid * Row::GSTR;
    float *myrow = rowg + ri * Row::STR;

    // acc[j].h carries the bias B[j]; |term| <= row_peak * kb.peak[j] * |x|. A batch of sorted
    // visibilities may span several cells, so the bias is chosen for each run of one cell, from
    // that run's own |x|: a strong visibility must not set the rounding of cells that it does not
    // reach. (F^T F of 2e6 visibilities, w = 4: 579 us, and 582 with one bias per batch.)
    const float row_peak = (float)W2 * kb.peak[ri];
    float2 B[W2];
    DS acc[W2];
#pragma unroll
    for (int j = 0; j < W2; ++j) {
        B[j] = bias(f2(0.f));
        acc[j] = DS{B[j], f2(0.f)};
    }
    // xr: largest biased exponents of the run that the sums are for next
    auto flush_to = [&](int cell, unsigned xr) {
        const float2 rx = __fmul2_rn(f2(row_peak), above(xr));
        float4 *p = mytile + ((cell >> 6) + 1 + ri) * S + (cell & 63) + 1;
#pragma unroll
        for (int j = 0; j < W2; ++j) {
            const float4 f = p[j];
            acc[j].h = minus(acc[j].h, B[j]);
            const DS r = ds_add(DS{make_float2(f.x, f.y), make_float2(f.z, f.w)}, acc[j]);
            p[j] = make_float4(r.h.x, r.h.y, r.l.x, r.l.y);
            B[j] = bias(__fmul2_rn(rx, f2(kb.peak[j])));
            acc[j] = DS{B[j], f2(0.f)};
        }
    };
    int plast = -1;  // cell of the group's sums, -1: none
    for (int b = 0; b < nbatch; ++b) {
        __syncwarp();
        const int kv = rbeg + b * W2 + ri;
        const bool valid = kv < rend;
        int key = -1;
        unsigned xe = 0;
        double2 fx = make_double2(0.0, 0.0);  // parts beyond the pairs' range
        if (valid) {
            const uint2 c = coords[it.begin + kv];
            const float2 rr = cres[it.begin + kv];
            const double2 x = vis[it.begin + kv];
            xe = exponents(max(0, exponent_of(x.x) - emax + 127),
                           max(0, exponent_of(x.y) - emax + 127));
            const int lu = cell_of(c.x), lv = cell_of(c.y);
            const float sg = tap_parity(it, g, lu, lv) ? -1.f : 1.f;
            float4 xs;
            split(x.x, emax, xs.x, xs.z);
            split(x.y, emax, xs.y, xs.w);
            if (far(x.x, emax)) {
                fx.x = sg * unscaled * x.x;
                xs.x = xs.z = 0.f;
            }
            if (far(x.y, emax)) {
                fx.y = sg * unscaled * x.y;
                xs.y = xs.w = 0.f;
            }
            key = (lu << 6) | lv;
            float4 *r4 = reinterpret_cast<float4 *>(myrow);
            r4[Row::X / 4] = make_float4(sg * xs.x, sg * xs.y, sg * xs.z, sg * xs.w);
            float vh[Row::WP], vl[Row::WP];
            {
                float h[W2], l[W2];
                ds_weights<W2>(kb, c.y, rr.y, h, l);
#pragma unroll
                for (int j = 0; j < Row::WP; ++j) {
                    vh[j] = j < W2 ? h[j] : 0.f;
                    vl[j] = j < W2 ? l[j] : 0.f;
                }
            }
#pragma unroll
            for (int q = 0; q < Row::WP / 4; ++q) {
                r4[q] = make_float4(vh[4 * q], vh[4 * q + 1], vh[4 * q + 2], vh[4 * q + 3]);
                r4[Row::WP / 4 + q] =
                    make_float4(vl[4 * q], vl[4 * q + 1], vl[4 * q + 2], vl[4 * q + 3]);
            }
            float uh[W2], ul[W2];
            ds_weights<W2>(kb, c.x, rr.x, uh, ul);
#pragma unroll
            for (int q = 0; q < W2 / 2; ++q)
                r4[Row::U / 4 + q] = make_float4(uh[2 * q], ul[2 * q], uh[2 * q + 1], ul[2 * q + 1]);
            if ((c.x | c.y) & kExtraTapBit) {
                // the taps at argument +w (coordinates on a cell boundary only): FP64, straight
                // to the grid
                const double eu = (c.x & kExtraTapBit) ? kb.edge : 0.0;
                const double ev = (c.y & kExtraTapBit) ? kb.edge : 0.0;
                const double xr = sg * unscaled * x.x, xi = sg * unscaled * x.y;
                auto put = [&](int ea, int eb, double wt) { to_grid(ea, eb, wt * xr, wt * xi); };
                if (eu != 0.0) {
                    for (int j = 0; j < W2; ++j)
                        put(lu, lv + 1 + j, eu * ((double)vh[j] + (double)vl[j]));
                    if (ev != 0.0) put(lu, lv, eu * ev);
                }
                if (ev != 0.0)
                    for (int i = 0; i < W2; ++i)
                        put(lu + 1 + i, lv, ev * ((double)uh[i] + (double)ul[i]));
            }
        }
        // visibilities beyond the range: in FP64, straight to the grid, the taps over the lanes
        for (unsigned fm = __ballot_sync(0xffffffffu, fx.x != 0.0 || fx.y != 0.0); fm;
             fm &= fm - 1) {
            __syncwarp();  // the rows are written
            const int src = __ffs(fm) - 1;
            const double xr = __shfl_sync(0xffffffffu, fx.x, src);
            const double xi = __shfl_sync(0xffffffffu, fx.y, src);
            const int cell = __shfl_sync(0xffffffffu, key, src);
            const float *row = rows + (warp * G + src / W2) * Row::GSTR + (src % W2) * Row::STR;
            for (int e = lane; e < W2 * W2; e += 32) {
                const int i = e / W2, j = e % W2;
                const double wt = ((double)row[Row::U + 2 * i] + (double)row[Row::U + 2 * i + 1]) *
                                  ((double)row[j] + (double)row[Row::WP + j]);
                to_grid((cell >> 6) + 1 + i, (cell & 63) + 1 + j, wt * xr, wt * xi);
            }
        }
        const int up = __shfl_up_sync(0xffffffffu, key, 1);
        const int prev = (ri == 0) ? plast : up;
        const unsigned flags = __ballot_sync(0xffffffffu, valid && prev >= 0 && key != prev);
        const unsigned nvalid = __popc(__ballot_sync(0xffffffffu, valid) & gmask);
        const int cell0 = plast;
        const int lastkey = __shfl_sync(0xffffffffu, key, grp * W2 + max((int)nvalid, 1) - 1);
        if (nvalid) plast = lastkey;
        unsigned wm = 0;  // steps at which any group of the warp flushes
#pragma unroll
        for (int q = 0; q < G; ++q) wm |= flags >> (q * W2);
        wm &= (1u << W2) - 1u;
        const unsigned bm = lane_on ? (flags >> (grp * W2)) & ((1u << W2) - 1u) : 0u;
        const int steps = (int)(lane_on ? nvalid : 0);
        // the largest |x| of this lane's run from here on (equal cells are neighbours; lanes of
        // the next group with the same cell may count too)
#pragma unroll
        for (int d = 1; d < W2; d <<= 1) {
            const int ke = __shfl_down_sync(0xffffffffu, key, d);
            const unsigned xo = __shfl_down_sync(0xffffffffu, xe, d);
            if (ke == key) xe = __vmaxu2(xe, xo);
        }
        // Renormalise the sums and choose each tap's bias for what this batch adds to them: above
        // the sum so far plus 2w terms of the largest |x| of the batch's first run, if that is of
        // the sums' cell, and the taps' largest weights. (Without this the low halves would grow
        // past the last place of the high ones.)
        {
            const int k0 = __shfl_sync(0xffffffffu, key, grp * W2);
            const unsigned x0 = __shfl_sync(0xffffffffu, xe, grp * W2);
            const float2 rx = __fmul2_rn(f2(cell0 < 0 || k0 == cell0 ? row_peak : 0.f), above(x0));
#pragma unroll
            for (int j = 0; j < W2; ++j) {
                const float2 v = minus(acc[j].h, B[j]);  // exact
                const float2 s = __fadd2_rn(v, acc[j].l);
                // (a part that is not finite stays what it is whatever its bias)
                const float2 top = make_float2(finite(s.x) ? fabsf(s.x) : 0.f,
                                               finite(s.y) ? fabsf(s.y) : 0.f);
                B[j] = bias(__ffma2_rn(rx, f2(kb.peak[j]), top));
                const float2 h = __fadd2_rn(s, B[j]);
                acc[j].l = __fadd2_rn(minus(acc[j].l, minus(s, v)), minus(s, minus(h, B[j])));
                acc[j].h = h;
            }
        }
        __syncwarp();
#pragma unroll 1
        for (int st = 0; st < W2; ++st) {
            if (wm & (1u << st)) {
                const bool need = (bm >> st) & 1u;
                const int before = __shfl_sync(0xffffffffu, key, grp * W2 + max(st, 1) - 1);
                const int fcell = st > 0 ? before : cell0;
                const unsigned xr = __shfl_sync(0xffffffffu, xe, grp * W2 + st);
                unsigned gm = __ballot_sync(0xffffffffu, need);
                while (gm) {
                    const int g0 = (__ffs(gm) - 1) / W2;
                    if (need && grp == g0) flush_to(fcell, xr);
                    __syncwarp();
                    gm &= ~(((1u << W2) - 1u) << (g0 * W2));
                }
            }
            if (st < steps) {
                const float *row = rowg + st * Row::STR;
                const float4 x = reinterpret_cast<const float4 *>(row + Row::X)[0];
                const float2 u = reinterpret_cast<const float2 *>(row + Row::U)[ri];
                // t = (uh + ul) x
                DS t;
                t.h = __fmul2_rn(f2(u.x), make_float2(x.x, x.y));
                t.l = __ffma2_rn(f2(u.x), make_float2(x.x, x.y), minus(f2(0.f), t.h));
                t.l = __ffma2_rn(f2(u.x), make_float2(x.z, x.w), t.l);
                t.l = __ffma2_rn(f2(u.y), make_float2(x.x, x.y), t.l);
                float vh[Row::WP], vl[Row::WP];
#pragma unroll
                for (int q = 0; q < Row::WP / 4; ++q) {
                    const float4 a = reinterpret_cast<const float4 *>(row)[q];
                    const float4 c = reinterpret_cast<const float4 *>(row + Row::WP)[q];
                    vh[4 * q] = a.x;
                    vh[4 * q + 1] = a.y;
                    vh[4 * q + 2] = a.z;
                    vh[4 * q + 3] = a.w;
                    vl[4 * q] = c.x;
                    vl[4 * q + 1] = c.y;
                    vl[4 * q + 2] = c.z;
                    vl[4 * q + 3] = c.w;
                }
#pragma unroll
                for (int j = 0; j < W2; ++j) ds_mac(vh[j], vl[j], t, acc[j]);
            }
        }
    }
#pragma unroll 1
    for (int g0 = 0; g0 < G; ++g0) {
        if (lane_on && grp == g0 && plast >= 0) flush_to(plast, 0);
        __syncwarp();
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E * E; e += kDsThreads) {
        const int ea = e / E, eb = e - ea * E;
        DS a{f2(0.f), f2(0.f)};
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            const float4 f = tiles[q * E * S + ea * S + eb];
            a = ds_add(a, DS{make_float2(f.x, f.y), make_float2(f.z, f.w)});
        }
        if (a.h.x == 0.f && a.h.y == 0.f) continue;
        to_grid(ea, eb, join(a.h.x, a.l.x, s1, s2), join(a.h.y, a.l.y, s1, s2));
    }
}

// Host: Chebyshev interpolation of the profile at 2 kDsHalf nodes per tap (as kb_poly_build),
// then the pairs.
void kb_ds_build(int w, double beta, KBPolyDS *out)
{
    memset(out, 0, sizeof(*out));
    constexpr int n = 2 * kDsHalf;
    double mono[kMaxDsTaps][n];
    for (int i = 0; i < w; ++i) {
        double f[n], cheb[n];
        for (int j = 0; j < n; ++j) {
            const double t = cos(M_PI * (j + 0.5) / n);
            f[j] = ((i & 1) ? -1.0 : 1.0) / (2.0 * w) *
                   kb_profile(0.5 * (t + 1.0) + w - 1 - i, w, beta);
        }
        for (int k = 0; k < n; ++k) {
            double s = 0.0;
            for (int j = 0; j < n; ++j) s += f[j] * cos(M_PI * k * (j + 0.5) / n);
            cheb[k] = (k ? 2.0 : 1.0) * s / n;
        }
        double a[n] = {1.0}, b[n] = {0.0, 1.0};  // T_0, T_1
        for (int d = 0; d < n; ++d) mono[i][d] = cheb[0] * a[d] + cheb[1] * b[d];
        for (int k = 2; k < n; ++k) {
            double c[n];
            for (int d = 0; d < n; ++d) c[d] = 2.0 * (d ? b[d - 1] : 0.0) - a[d];
            for (int d = 0; d < n; ++d) {
                mono[i][d] += cheb[k] * c[d];
                a[d] = b[d];
                b[d] = c[d];
            }
        }
    }
    // largest sum of an axis' weights, and per tap the largest weight and partial value of the
    // two Horner sums and of t times the odd one
    double sum = 0.0, peak[2 * kMaxDsTaps] = {0.0}, part[kMaxDsTaps] = {0.0};
    for (int q = 0; q <= 512; ++q) {
        const double t = q / 256.0 - 1.0, u = t * t;
        double s = 0.0;
        for (int i = 0; i < w; ++i) {
            double e = 0.0, o = 0.0;
            for (int k = kDsHalf - 1; k >= 0; --k) {
                e = e * u + mono[i][2 * k];
                o = o * u + mono[i][2 * k + 1];
                part[i] = std::max(part[i], std::max(fabs(e), fabs(o)));
            }
            s += fabs(e + t * o) + fabs(e - t * o);
            peak[i] = std::max(peak[i], std::max(fabs(e + t * o), fabs(e - t * o)));
        }
        sum = std::max(sum, s);
    }
    const double factor = (sum > 0.0 && std::isfinite(sum)) ? 0.99 / sum : 1.0;
    out->scale2 = 1.0 / (factor * factor);
    out->edge = -factor * kb_profile((double)w, w, beta) / (2.0 * w);
    for (int i = 0; i < w; ++i) {
        out->peak[i] = out->peak[2 * w - 1 - i] = (float)(1.01 * factor * peak[i]);
        // B = 1.5 * 2^m with 2^(m-1) above every partial value
        int m = -100;
        const double top = 1.02 * factor * part[i];
        if (top > 0.0 && std::isfinite(top)) {
            frexp(top, &m);  // top < 2^m
            m += 1;
        }
        const double B = ldexp(1.5, m), grid = ldexp(1.0, m - 23);
        const int p = i / 2;
        auto set = [&](float2 &dst, double v) {
            if (i & 1) dst.y = (float)v;
            else dst.x = (float)v;
        };
        set(out->b[p], B);
        set(out->nb[p], -B);
        for (int k = 0; k < kDsHalf; ++k) {
            const double ce = mono[i][2 * (kDsHalf - 1 - k)] * factor;
            const double co = mono[i][2 * (kDsHalf - 1 - k) + 1] * factor;
            const double eh = std::nearbyint(ce / grid) * grid;
            const double oh = std::nearbyint(co / grid) * grid;
            set(out->eb[k][p], k ? eh + B : eh);
            set(out->el[k][p], ce - eh);
            set(out->ob[k][p], k ? oh + B : oh);
            set(out->ol[k][p], co - oh);
        }
    }
}

static int ds_smem(const void *kern, size_t smem)
{
    if (smem > 48 * 1024)
        LENTILS_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)smem));
    return LENTILS_OK;
}

// The shared memory of an SM holds two CTAs or more.
constexpr size_t kMaxDsSmem = 100 * 1024;

template <int W2>
static int degrid_ds(const lentils_plan *p, const double2 *grid, double2 *vis, cudaStream_t s,
                     const double *vscale)
{
    const GridGeom &g = p->geom;
    const size_t smem = sizeof(float4) * (size_t)g.E * g.stride + sizeof(uchar2) * (size_t)g.E * g.T;
    if (int st = ds_smem((const void *)degrid_ds_kernel<W2>, smem)) return st;
    LENTILS_CUDA_TRY(pdl_launch(degrid_ds_kernel<W2>, dim3(p->nitems), dim3(kDsThreads), smem, s,
                                grid, (const uint2 *)p->coords, (const float2 *)p->coords_res, vis,
                                (const WorkItem *)p->items, p->kbds, p->geom, vscale));
    LENTILS_CHECK_LAUNCH("degrid_ds_kernel");
    return LENTILS_OK;
}

template <int W2>
static int grid_ds(const lentils_plan *p, const double2 *vis, double2 *grid, cudaStream_t s)
{
    const size_t smem = grid_ds_smem_bytes<W2>(p->geom);
    if (int st = ds_smem((const void *)grid_ds_kernel<W2>, smem)) return st;
    LENTILS_CUDA_TRY(pdl_launch(grid_ds_kernel<W2>, dim3(p->nitems), dim3(kDsThreads), smem, s, vis,
                                (const uint2 *)p->coords, (const float2 *)p->coords_res, grid,
                                (const WorkItem *)p->items, p->kbds, p->geom));
    LENTILS_CHECK_LAUNCH("grid_ds_kernel");
    return LENTILS_OK;
}

// Whether this plan's FP64 operators run as pairs (both directions or neither, so that they stay
// each other's transpose): not for 2w > 8 (the registers of the weights) nor where the warps'
// copies of a tile of 32 or 64 cells leave an SM fewer than two CTAs. Those keep the FP64
// kernels.
bool plan_uses_ds(const lentils_plan *p)
{
    switch (p->geom.w) {
    case 1: return grid_ds_smem_bytes<2>(p->geom) <= kMaxDsSmem;
    case 2: return grid_ds_smem_bytes<4>(p->geom) <= kMaxDsSmem;
    case 3: return grid_ds_smem_bytes<6>(p->geom) <= kMaxDsSmem;
    case 4: return grid_ds_smem_bytes<8>(p->geom) <= kMaxDsSmem;
    }
    return false;
}

int launch_degrid_ds(const lentils_plan *p, const double2 *grid, double2 *vis, cudaStream_t s,
                     const double *vscale)
{
    switch (p->geom.w) {
    case 1: return degrid_ds<2>(p, grid, vis, s, vscale);
    case 2: return degrid_ds<4>(p, grid, vis, s, vscale);
    case 3: return degrid_ds<6>(p, grid, vis, s, vscale);
    }
    return degrid_ds<8>(p, grid, vis, s, vscale);
}

int launch_grid_ds(const lentils_plan *p, const double2 *vis, double2 *grid, cudaStream_t s)
{
    switch (p->geom.w) {
    case 1: return grid_ds<2>(p, vis, grid, s);
    case 2: return grid_ds<4>(p, vis, grid, s);
    case 3: return grid_ds<6>(p, vis, grid, s);
    }
    return grid_ds<8>(p, vis, grid, s);
}

}  // namespace lentils
