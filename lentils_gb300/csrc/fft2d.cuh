// Two-dimensional real transforms between an image and its zero-padded spectrum, for padded
// sizes that are powers of two (fft2d.cu). See there.
#pragma once

#include "common.cuh"

namespace lentils {

// Whether the padded plane (nu, nv) has transforms here.
bool fft2d_supported(int nu, int nv);

// Values per row of the scratch between the passes: nv / 2 + 1 up to whole 32-byte segments of
// FP32 values, so that the column kernels' four columns are one segment.
constexpr int fft2d_pitch(int nv) { return (nv / 2 + 1 + 3) & ~3; }

struct Fft2d {
    int nx, ny, padx, pady;  // image and its offset in the padded plane
    int nu, nv, half;        // padded plane, nv / 2 + 1
    int pitch;               // of the scratch rows
    void *tw_u, *tw_v;       // twiddle tables (device), float2 or double2
};

// Twiddle tables of `op` in FP32 (C = float2) or FP64 (double2), uploaded on s and complete on
// return; free them with fft2d_free.
template <typename C>
int fft2d_init(Fft2d *op, int nx, int ny, int padx, int pady, int nu, int nv, cudaStream_t s);
void fft2d_free(Fft2d *op);

// Image -> half-plane spectrum (nu x half) of the zero-padded image, unnormalised. apx (nx) and
// apy (ny): separable factors of the image (null: 1). mid: nx * pitch values of scratch.
template <typename R, typename C>
int fft2d_forward(const Fft2d &op, const R *img, C *mid, C *grid, const R *apx, const R *apy,
                  cudaStream_t s);
// Half-plane spectrum -> image (crop of the unnormalised inverse, times the factors); the spectrum
// is zero afterwards. The imaginary parts of the self-conjugate columns (0 and nv / 2) of the column
// transforms do not count, as in numpy's irfft2.
template <typename R, typename C>
int fft2d_inverse(const Fft2d &op, C *grid, C *mid, R *img, const R *apx, const R *apy,
                  cudaStream_t s);
// out = crop(inverse(spec * forward(pad(img)))): the two column transforms and the product in one
// kernel, in place on mid.
template <typename R, typename C>
int fft2d_convolve(const Fft2d &op, const R *img, C *mid, const C *spec, R *out, cudaStream_t s);

}  // namespace lentils
