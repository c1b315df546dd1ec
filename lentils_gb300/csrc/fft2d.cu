// Real 2-D transforms of a zero-padded image (the uniform FFT of the NUFFT and of the dirty-beam
// convolution) for padded sizes 2^7 ... 2^11.
//
// The padded plane is at least twice the image in each direction, so half of the rows of a
// forward transform are zero and half of those of an inverse one are cropped away. A library
// transform does not know that, and needs a pass that writes the padded plane before it and one
// that crops after it. Here
//   forward: rows     image rows x apodisation, zero-padded in registers, real FFT of two rows as
//                     one complex one; only the nx image rows exist in the scratch
//            columns  nx rows in, nu rows out
//   inverse: columns  nu rows in, only the nx image rows out
//            rows     two rows per complex inverse FFT, crop and apodisation on the way out
// so that a 512^2 image on a 1024^2 plane moves 13 MB per transform instead of 27 and takes two
// launches instead of three (forward) or four (inverse, whose Hermitian-edge pass is the row
// kernel's treatment of columns 0 and nv/2). The planes fit the L2; what bounds these kernels is
// latency: a CTA's load, two or three exchanges through shared memory and its store. So the work
// is cut into many small CTAs: a row pair each, or four columns (32-byte segments) each.
// Measured (sum of a forward and an inverse transform, warm caches): 512^2 image in FP32
// 47 -> 23 us (with the padding, edge and crop passes before), in FP64 345 -> 130 us (bound by
// the FP64 pipe: 78 MFLOP); the dirty-beam convolution of a 256^2 image 31 -> 17 us. Other
// sizes keep the library transform: these kernels' radices are powers of two.
//
// One transform: N/16 threads with 16 values each in registers, passes of radix 16, 16 and
// N/256 (Stockham order), values exchanged through shared memory with one word of padding per
// 16, twiddles from a table rounded from FP64.
#include "fft2d.cuh"

#include <cmath>
#include <vector>

namespace lentils {

// N = 16 * R2 * R3
template <int N>
struct FftShape {
    static constexpr int R2 = N >= 256 ? 16 : N / 16;
    static constexpr int R3 = N / (16 * R2);
    static constexpr int T = N / 16;  // threads per transform
    static constexpr int PAD = N + N / 16;
};

template <typename C>
__device__ __forceinline__ C cadd(C a, C b) { a.x += b.x; a.y += b.y; return a; }
template <typename C>
__device__ __forceinline__ C csub(C a, C b) { a.x -= b.x; a.y -= b.y; return a; }
template <bool INV, typename C>
__device__ __forceinline__ C rot(C a)  // times -i (forward) or i
{
    C r;
    r.x = INV ? -a.y : a.y;
    r.y = INV ? a.x : -a.x;
    return r;
}
template <bool INV, typename C>
__device__ __forceinline__ C twmul(C a, C w)  // a * w, or a * conj(w) for the inverse
{
    C r;
    if (INV) {
        r.x = a.x * w.x + a.y * w.y;
        r.y = a.y * w.x - a.x * w.y;
    } else {
        r.x = a.x * w.x - a.y * w.y;
        r.y = a.y * w.x + a.x * w.y;
    }
    return r;
}

template <bool INV, typename C>
__device__ __forceinline__ void dft4(C &a, C &b, C &c, C &d)
{
    const C s = cadd(a, c), t = csub(a, c), u = cadd(b, d), v = rot<INV>(csub(b, d));
    a = cadd(s, u);
    b = cadd(t, v);
    c = csub(s, u);
    d = csub(t, v);
}

// In-place DFT of v[0], v[ST], ..., v[(R - 1) ST], natural order in and out.
template <int R, int ST, bool INV, typename C>
__device__ __forceinline__ void dft(C *v)
{
    using F = decltype(v[0].x);
    if constexpr (R == 2) {
        const C a = v[0];
        v[0] = cadd(a, v[ST]);
        v[ST] = csub(a, v[ST]);
    } else if constexpr (R == 4) {
        dft4<INV>(v[0], v[ST], v[2 * ST], v[3 * ST]);
    } else if constexpr (R == 8) {
        const F h = (F)0.70710678118654752440;
        C e0 = v[0], e1 = v[2 * ST], e2 = v[4 * ST], e3 = v[6 * ST];
        C o0 = v[ST], o1 = v[3 * ST], o2 = v[5 * ST], o3 = v[7 * ST];
        dft4<INV>(e0, e1, e2, e3);
        dft4<INV>(o0, o1, o2, o3);
        const C r1 = rot<INV>(o1), r3 = rot<INV>(o3);
        o1.x = h * (o1.x + r1.x);  // (1 - i) / sqrt 2 (forward)
        o1.y = h * (o1.y + r1.y);
        o2 = rot<INV>(o2);
        o3.x = h * (r3.x - o3.x);  // (-1 - i) / sqrt 2
        o3.y = h * (r3.y - o3.y);
        v[0] = cadd(e0, o0);
        v[ST] = cadd(e1, o1);
        v[2 * ST] = cadd(e2, o2);
        v[3 * ST] = cadd(e3, o3);
        v[4 * ST] = csub(e0, o0);
        v[5 * ST] = csub(e1, o1);
        v[6 * ST] = csub(e2, o2);
        v[7 * ST] = csub(e3, o3);
    } else if constexpr (R == 16) {
        // cos, sin of 2 pi k / 16
        const F c1 = (F)0.92387953251128675613, s1 = (F)0.38268343236508977173,
                h = (F)0.70710678118654752440;
#pragma unroll
        for (int n = 0; n < 4; ++n)
            dft4<INV>(v[n * ST], v[(n + 4) * ST], v[(n + 8) * ST], v[(n + 12) * ST]);
        // v[(4 k + n) ST] *= w16^(n k)
        auto tw = [&](int i, F c, F s) {
            C w;
            w.x = c;
            w.y = -s;
            v[i * ST] = twmul<INV>(v[i * ST], w);
        };
        tw(5, c1, s1);    // n k = 1
        tw(6, h, h);      // 2
        tw(7, s1, c1);    // 3
        tw(9, h, h);      // 2
        v[10 * ST] = rot<INV>(v[10 * ST]);  // 4
        tw(11, -h, h);    // 6
        tw(13, s1, c1);   // 3
        tw(14, -h, h);    // 6
        tw(15, -c1, -s1); // 9
#pragma unroll
        for (int k = 0; k < 4; ++k)
            dft4<INV>(v[4 * k * ST], v[(4 * k + 1) * ST], v[(4 * k + 2) * ST],
                      v[(4 * k + 3) * ST]);
        // X[k + 4 m] sits at v[4 k + m]
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int m = k + 1; m < 4; ++m) {
                const C t = v[(4 * k + m) * ST];
                v[(4 * k + m) * ST] = v[(4 * m + k) * ST];
                v[(4 * m + k) * ST] = t;
            }
    }
}

// A thread's twiddles. FP32 transforms load them into registers before they wait for the kernel
// before them (the table, and the apodisation factors of the row kernel, do not change), which
// takes a load's latency out of each pass: the normal operator of a 512^2 image (four transform
// kernels) 144 -> 135 us, the dirty-beam one of 256^2 (three) 50 -> 46 us. FP64 ones, whose registers
// would not hold them, load them at their use.
template <int N, typename C>
struct Twiddles {
    using S = FftShape<N>;
    static constexpr bool kHeld = sizeof(C) == 8;
    static constexpr int N2 = (16 / S::R2) * (S::R2 - 1);
    static constexpr int N3 = S::R3 > 1 ? (16 / S::R3) * (S::R3 - 1) : 0;
    C w2[kHeld ? N2 : 1], w3[kHeld && N3 ? N3 : 1];
    const C *tw;
    int t;
    __device__ __forceinline__ Twiddles(const C *__restrict__ table, int t_) : tw(table), t(t_)
    {
        if constexpr (kHeld) {
#pragma unroll
            for (int b = 0; b < 16 / S::R2; ++b)
#pragma unroll
                for (int q = 1; q < S::R2; ++q) w2[b * (S::R2 - 1) + q - 1] = at2(b, q);
            if constexpr (N3 > 0)
#pragma unroll
                for (int b = 0; b < 16 / S::R3; ++b)
#pragma unroll
                    for (int q = 1; q < S::R3; ++q) w3[b * (S::R3 - 1) + q - 1] = at3(b, q);
        }
    }
    __device__ __forceinline__ C at2(int b, int q) const
    {
        return __ldg(tw + q * 16 + ((t + b * S::T) & 15));
    }
    __device__ __forceinline__ C at3(int b, int q) const
    {
        constexpr int Ns = 16 * S::R2;
        return __ldg(tw + Ns + q * Ns + t + b * S::T);
    }
    __device__ __forceinline__ C pass2(int b, int q) const
    {
        if constexpr (kHeld) return w2[b * (S::R2 - 1) + q - 1];
        else return at2(b, q);
    }
    __device__ __forceinline__ C pass3(int b, int q) const
    {
        if constexpr (kHeld) return w3[b * (S::R3 - 1) + q - 1];
        else return at3(b, q);
    }
};

// One transform by the T threads t: in v[q] = x[t + q T], out v[b R + q] = X[at(b, q)] with R the
// last radix. sm(pos) is the shared-memory slot of a position; the CTA's transforms run in step.
template <int N, bool INV, typename C, class Slot>
__device__ __forceinline__ void fft_regs(C (&v)[16], int t, const Twiddles<N, C> &tw, Slot sm)
{
    using S = FftShape<N>;
    constexpr int R2 = S::R2, R3 = S::R3, T = S::T;
    dft<16, 1, INV>(v);
#pragma unroll
    for (int q = 0; q < 16; ++q) sm(t * 16 + q) = v[q];
    __syncthreads();
#pragma unroll
    for (int b = 0; b < 16 / R2; ++b) {
        const int j = t + b * T;
#pragma unroll
        for (int q = 0; q < R2; ++q) {
            v[b * R2 + q] = sm(j + q * (N / R2));
            if (q > 0) v[b * R2 + q] = twmul<INV>(v[b * R2 + q], tw.pass2(b, q));
        }
        dft<R2, 1, INV>(v + b * R2);
    }
    if constexpr (R3 > 1) {
        constexpr int Ns = 16 * R2;
        static_assert(R2 == 16, "three passes: the second is radix 16");
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 16; ++q) sm((t / 16) * Ns + (t & 15) + q * 16) = v[q];
        __syncthreads();
#pragma unroll
        for (int b = 0; b < 16 / R3; ++b) {
            const int j = t + b * T;  // below Ns
#pragma unroll
            for (int q = 0; q < R3; ++q) {
                v[b * R3 + q] = sm(j + q * Ns);
                if (q > 0) v[b * R3 + q] = twmul<INV>(v[b * R3 + q], tw.pass3(b, q));
            }
            dft<R3, 1, INV>(v + b * R3);
        }
    }
}

// Position of the value v[i] after fft_regs.
template <int N>
__device__ __forceinline__ int fft_at(int t, int i)
{
    using S = FftShape<N>;
    constexpr int R = S::R3 > 1 ? S::R3 : S::R2;
    return t + (i / R) * S::T + (i % R) * (N / R);
}

// Programmatic dependent launch. FP32 transforms are latency chains, and let the next kernel start as
// soon as they have all begun. FP64 ones are bound by the FP64 pipe of the SMs that they run on,
// and a kernel that starts while another still holds most SMs has its CTAs packed onto the SMs that
// are free: the row pass of a 512^2 plane (128 CTAs of a warp) took 75 us for 24. So they let the next
// kernel start when their results are ready (fft_end), and a grid of more CTAs than SMs starts on an
// idle GPU (fft_launch). Early start everywhere, late start everywhere, this rule, no early start at
// all, us per call, FP64: F of a 256^2 image with 6e4 visibilities, w = 3: 109, 53, 53, 61; F^T F of
// 512^2 with 2e6, w = 4: 580, 563, 483, 486; of 128^2 with 2e4: 95, 84, 84, 98; the dirty-beam
// convolution of 512^2: 250, 208, 127, 130; of 64^2: 56, 56, 56, 64.
template <typename C>
__device__ __forceinline__ void fft_begin()
{
    if constexpr (sizeof(C) == 8) pdl_entry();
    else pdl_wait();
}
template <typename C>
__device__ __forceinline__ void fft_end()  // before the stores
{
    if constexpr (sizeof(C) == 16) pdl_trigger();
}
template <typename C, class K, class... Args>
static cudaError_t fft_launch(K kern, dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                              Args &&...args)
{
    if (sizeof(C) == 16 && grid.x > kSMs) {
        kern<<<grid, block, smem, s>>>(std::forward<Args>(args)...);
        return cudaGetLastError();
    }
    return pdl_launch(kern, grid, block, smem, s, std::forward<Args>(args)...);
}

template <int N>
constexpr int kRowPairs = FftShape<N>::T >= 32 ? 1 : 32 / FftShape<N>::T;  // per CTA
template <int N>
constexpr int kCols = 4;

// Rows 2p, 2p + 1 of the image -> rows of mid (half values each).
template <typename R, typename C, int N>
__global__ void __launch_bounds__(kRowPairs<N> *FftShape<N>::T)
    fft_rows_forward(const R *__restrict__ img, C *__restrict__ mid, const R *__restrict__ apx,
                     const R *__restrict__ apy, const C *__restrict__ tw, int nx, int ny, int pady)
{
    using S = FftShape<N>;
    __shared__ C smem[kRowPairs<N> * S::PAD];
    const int w = threadIdx.x / S::T, t = threadIdx.x % S::T;
    const int a = 2 * (blockIdx.x * kRowPairs<N> + w), b = a + 1;
    auto sm = [&](int pos) -> C & { return smem[w * S::PAD + pos + (pos >> 4)]; };
    const Twiddles<N, C> tws(tw, t);
    const R fa = a < nx ? (apx ? apx[a] : (R)1) : (R)0, fb = b < nx ? (apx ? apx[b] : (R)1) : (R)0;
    C v[16];
    R f[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const int j = t + q * S::T - pady;
        f[q] = j >= 0 && j < ny ? (apy ? apy[j] : (R)1) : (R)0;
    }
    fft_begin<C>();
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const int j = t + q * S::T - pady;
        v[q].x = v[q].y = (R)0;
        if (j >= 0 && j < ny) {
            if (a < nx) v[q].x = img[(long long)a * ny + j];
            if (b < nx) v[q].y = img[(long long)b * ny + j];
        }
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const int j = t + q * S::T - pady;
        if (j >= 0 && j < ny) {  // not where the factor is 0: an image may hold infinities
            v[q].x = fa * f[q] * v[q].x;
            v[q].y = fb * f[q] * v[q].y;
        }
    }
    fft_regs<N, false>(v, t, tws, sm);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; ++i) sm(fft_at<N>(t, i)) = v[i];
    __syncthreads();
    fft_end<C>();
    // Z = A + iB with A, B Hermitian: A_k = (Z_k + conj Z_-k) / 2, B_k = (Z_k - conj Z_-k) / 2i
    constexpr int half = N / 2 + 1, pitch = fft2d_pitch(N);
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const int k = t + q * S::T;
        if (k >= half) break;  // the ninth: k = N / 2 only
        const C z = sm(k), y = sm((N - k) & (N - 1));
        C ra, rb;
        ra.x = (R)0.5 * (z.x + y.x);
        ra.y = (R)0.5 * (z.y - y.y);
        rb.x = (R)0.5 * (z.y + y.y);
        rb.y = (R)0.5 * (y.x - z.x);
        if (a < nx) mid[(long long)a * pitch + k] = ra;
        if (b < nx) mid[(long long)b * pitch + k] = rb;
    }
}

// Rows 2p, 2p + 1 of mid -> rows of the image.
template <typename R, typename C, int N>
__global__ void __launch_bounds__(kRowPairs<N> *FftShape<N>::T)
    fft_rows_inverse(const C *__restrict__ mid, R *__restrict__ img, const R *__restrict__ apx,
                     const R *__restrict__ apy, const C *__restrict__ tw, int nx, int ny, int pady)
{
    using S = FftShape<N>;
    __shared__ C smem[kRowPairs<N> * S::PAD];
    const int w = threadIdx.x / S::T, t = threadIdx.x % S::T;
    const int a = 2 * (blockIdx.x * kRowPairs<N> + w), b = a + 1;
    auto sm = [&](int pos) -> C & { return smem[w * S::PAD + pos + (pos >> 4)]; };
    constexpr int pitch = fft2d_pitch(N);
    const Twiddles<N, C> tws(tw, t);
    fft_begin<C>();
    // Z_k = A_k + i B_k, Z_-k = conj A_k + i conj B_k; all loads before the first store
    C v[16];
    const C *ma = mid + (long long)a * pitch, *mb = mid + (long long)b * pitch;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        v[2 * q].x = v[2 * q].y = v[2 * q + 1].x = v[2 * q + 1].y = (R)0;
        if (a < nx) v[2 * q] = ma[t + q * S::T];
        if (b < nx) v[2 * q + 1] = mb[t + q * S::T];
    }
    C last;  // k = N / 2: both real
    last.x = last.y = (R)0;
    if (t == 0 && a < nx) last.x = ma[N / 2].x;
    if (t == 0 && b < nx) last.y = mb[N / 2].x;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int k = t + q * S::T;
        C ra = v[2 * q], rb = v[2 * q + 1], z, y;
        if (k == 0) ra.y = rb.y = (R)0;
        z.x = ra.x - rb.y;
        z.y = ra.y + rb.x;
        y.x = ra.x + rb.y;
        y.y = rb.x - ra.y;
        sm(k) = z;
        if (k != 0) sm(N - k) = y;
    }
    if (t == 0) sm(N / 2) = last;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = sm(t + q * S::T);
    __syncthreads();
    fft_regs<N, true>(v, t, tws, sm);
    fft_end<C>();
    const R fa = a < nx ? (apx ? apx[a] : (R)1) : (R)0, fb = b < nx ? (apx ? apx[b] : (R)1) : (R)0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int j = fft_at<N>(t, i) - pady;
        if (j < 0 || j >= ny) continue;
        const R f = apy ? apy[j] : (R)1;
        if (a < nx) img[(long long)a * ny + j] = fa * f * v[i].x;
        if (b < nx) img[(long long)b * ny + j] = fb * f * v[i].y;
    }
}

// Four columns per CTA. MODE 0: mid (nx rows) -> grid (N rows); 1: grid -> mid (inverse), and
// the grid is zero afterwards (the next adjoint accumulates into it without a memset of its
// own); 2: mid -> mid, forward, times spec, inverse.
template <typename C, int N, int MODE>
__global__ void __launch_bounds__(kCols<N> *FftShape<N>::T)
    fft_columns(C *in, C *out, const C *__restrict__ spec,
                const C *__restrict__ tw, int nx, int padx, int half, int pitch)
{
    using S = FftShape<N>;
    constexpr int NC = kCols<N>;
    extern __shared__ __align__(16) unsigned char smraw[];
    C *smem = reinterpret_cast<C *>(smraw);  // PAD x NC
    const int c = threadIdx.x % NC, t = threadIdx.x / NC;
    const int col = blockIdx.x * NC + c;
    const bool on = col < half;
    auto sm = [&](int pos) -> C & { return smem[(pos + (pos >> 4)) * NC + c]; };
    const Twiddles<N, C> tws(tw, t);
    fft_begin<C>();
    C v[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const int p = t + q * S::T, i = MODE == 1 ? p : p - padx;
        v[q].x = v[q].y = 0;
        if (on && (MODE == 1 || (i >= 0 && i < nx)))
            v[q] = in[(long long)i * (MODE == 1 ? half : pitch) + col];
    }
    if (MODE == 1 && on) {
        C zero;
        zero.x = zero.y = 0;
#pragma unroll
        for (int q = 0; q < 16; ++q) in[(long long)(t + q * S::T) * half + col] = zero;
    }
    fft_regs<N, MODE == 1>(v, t, tws, sm);
    if constexpr (MODE == 2) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int p = fft_at<N>(t, i);
            C f;
            f.x = f.y = 0;
            if (on) f = spec[(long long)p * half + col];
            sm(p) = twmul<false>(v[i], f);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = sm(t + q * S::T);
        __syncthreads();
        fft_regs<N, true>(v, t, tws, sm);
    }
    fft_end<C>();
    if (!on) return;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int p = fft_at<N>(t, i), r = MODE == 0 ? p : p - padx;
        if (MODE == 0 || (r >= 0 && r < nx))
            out[(long long)r * (MODE == 0 ? half : pitch) + col] = v[i];
    }
}

constexpr int kFftMin = 128, kFftMax = 2048;

static bool fft_size(int n) { return n >= kFftMin && n <= kFftMax && (n & (n - 1)) == 0; }
bool fft2d_supported(int nu, int nv) { return fft_size(nu) && fft_size(nv); }

// Twiddles of passes 2 and 3 (q Ns + k: exp(-2 pi i k q / (Ns R))); pass 3's start at 16 R2.
template <typename C>
static int upload_twiddles(int n, void **dst, cudaStream_t s)
{
    const int r2 = n >= 256 ? 16 : n / 16, r3 = n / (16 * r2);
    std::vector<C> h(16 * r2 + (r3 > 1 ? n : 0));
    auto set = [&](C &d, int k, int q, int m) {
        const double a = -2.0 * M_PI * (double)k * (double)q / (double)m;
        d.x = (decltype(d.x))cos(a);
        d.y = (decltype(d.y))sin(a);
    };
    for (int q = 0; q < r2; ++q)
        for (int k = 0; k < 16; ++k) set(h[q * 16 + k], k, q, 16 * r2);
    if (r3 > 1)
        for (int q = 0; q < r3; ++q)
            for (int k = 0; k < 16 * r2; ++k) set(h[16 * r2 + q * 16 * r2 + k], k, q, n);
    LENTILS_CUDA_TRY(cudaMalloc(dst, sizeof(C) * h.size()));
    LENTILS_CUDA_TRY(cudaMemcpyAsync(*dst, h.data(), sizeof(C) * h.size(), cudaMemcpyHostToDevice, s));
    LENTILS_CUDA_TRY(cudaStreamSynchronize(s));
    return LENTILS_OK;
}

template <typename C>
int fft2d_init(Fft2d *op, int nx, int ny, int padx, int pady, int nu, int nv, cudaStream_t s)
{
    *op = Fft2d{nx, ny, padx, pady, nu, nv, nv / 2 + 1, fft2d_pitch(nv), nullptr, nullptr};
    if (int st = upload_twiddles<C>(nu, &op->tw_u, s)) return st;
    return upload_twiddles<C>(nv, &op->tw_v, s);
}
template int fft2d_init<float2>(Fft2d *, int, int, int, int, int, int, cudaStream_t);
template int fft2d_init<double2>(Fft2d *, int, int, int, int, int, int, cudaStream_t);

void fft2d_free(Fft2d *op)
{
    cudaFree(op->tw_u);
    cudaFree(op->tw_v);
    op->tw_u = op->tw_v = nullptr;
}

template <typename R, typename C, int N>
static int rows(const Fft2d &op, bool inverse, const void *in, void *out, const R *apx,
                const R *apy, cudaStream_t s)
{
    const dim3 grid((op.nx + 2 * kRowPairs<N> - 1) / (2 * kRowPairs<N>));
    const dim3 block(kRowPairs<N> * FftShape<N>::T);
    const C *tw = (const C *)op.tw_v;
    if (inverse)
        LENTILS_CUDA_TRY(fft_launch<C>(fft_rows_inverse<R, C, N>, grid, block, 0, s, (const C *)in,
                                       (R *)out, apx, apy, tw, op.nx, op.ny, op.pady));
    else
        LENTILS_CUDA_TRY(fft_launch<C>(fft_rows_forward<R, C, N>, grid, block, 0, s, (const R *)in,
                                       (C *)out, apx, apy, tw, op.nx, op.ny, op.pady));
    LENTILS_CHECK_LAUNCH("fft_rows");
    return LENTILS_OK;
}

template <typename C, int N, int MODE>
static int columns(const Fft2d &op, C *in, C *out, const C *spec, cudaStream_t s)
{
    constexpr int NC = kCols<N>;
    const size_t smem = sizeof(C) * FftShape<N>::PAD * NC;
    if (smem > 48 * 1024)
        LENTILS_CUDA_TRY(cudaFuncSetAttribute(fft_columns<C, N, MODE>,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)smem));
    LENTILS_CUDA_TRY(fft_launch<C>(fft_columns<C, N, MODE>, dim3((op.half + NC - 1) / NC),
                                   dim3(NC * FftShape<N>::T), smem, s, in, out, spec,
                                   (const C *)op.tw_u, op.nx, op.padx, op.half, op.pitch));
    LENTILS_CHECK_LAUNCH("fft_columns");
    return LENTILS_OK;
}

template <typename R, typename C>
static int any_rows(const Fft2d &op, bool inverse, const void *in, void *out, const R *apx,
                    const R *apy, cudaStream_t s)
{
    switch (op.nv) {
    case 128: return rows<R, C, 128>(op, inverse, in, out, apx, apy, s);
    case 256: return rows<R, C, 256>(op, inverse, in, out, apx, apy, s);
    case 512: return rows<R, C, 512>(op, inverse, in, out, apx, apy, s);
    case 1024: return rows<R, C, 1024>(op, inverse, in, out, apx, apy, s);
    case 2048: return rows<R, C, 2048>(op, inverse, in, out, apx, apy, s);
    }
    return set_error(LENTILS_ERR_UNSUPPORTED, "fft2d: nv=%d", op.nv);
}

template <typename C, int MODE>
static int any_columns(const Fft2d &op, C *in, C *out, const C *spec, cudaStream_t s)
{
    switch (op.nu) {
    case 128: return columns<C, 128, MODE>(op, in, out, spec, s);
    case 256: return columns<C, 256, MODE>(op, in, out, spec, s);
    case 512: return columns<C, 512, MODE>(op, in, out, spec, s);
    case 1024: return columns<C, 1024, MODE>(op, in, out, spec, s);
    case 2048: return columns<C, 2048, MODE>(op, in, out, spec, s);
    }
    return set_error(LENTILS_ERR_UNSUPPORTED, "fft2d: nu=%d", op.nu);
}

template <typename R, typename C>
int fft2d_forward(const Fft2d &op, const R *img, C *mid, C *grid, const R *apx, const R *apy,
                  cudaStream_t s)
{
    if (int st = any_rows<R, C>(op, false, img, mid, apx, apy, s)) return st;
    return any_columns<C, 0>(op, mid, grid, (const C *)nullptr, s);
}

template <typename R, typename C>
int fft2d_inverse(const Fft2d &op, C *grid, C *mid, R *img, const R *apx, const R *apy,
                  cudaStream_t s)
{
    if (int st = any_columns<C, 1>(op, grid, mid, (const C *)nullptr, s)) return st;
    return any_rows<R, C>(op, true, mid, img, apx, apy, s);
}

template <typename R, typename C>
int fft2d_convolve(const Fft2d &op, const R *img, C *mid, const C *spec, R *out, cudaStream_t s)
{
    if (int st = any_rows<R, C>(op, false, img, mid, (const R *)nullptr, (const R *)nullptr, s))
        return st;
    if (int st = any_columns<C, 2>(op, mid, mid, spec, s)) return st;
    return any_rows<R, C>(op, true, mid, out, (const R *)nullptr, (const R *)nullptr, s);
}

#define LENTILS_FFT2D(R, C)                                                                      \
    template int fft2d_forward<R, C>(const Fft2d &, const R *, C *, C *, const R *, const R *,   \
                                     cudaStream_t);                                              \
    template int fft2d_inverse<R, C>(const Fft2d &, C *, C *, R *, const R *, const R *,   \
                                     cudaStream_t);                                              \
    template int fft2d_convolve<R, C>(const Fft2d &, const R *, C *, const C *, R *, cudaStream_t);
LENTILS_FFT2D(float, float2)
LENTILS_FFT2D(double, double2)

}  // namespace lentils
