// wg_frame.cuh — what the frame kernels of scenes and of the server share: the palette index
// in FP32 where that decides it, and the tile of pixels a block renders.
//
// A pixel's palette index in FP64 (tanh, log, divisions) is 70 to 130 operations on a pipe that
// retires 1.68 a clock and SM, which bounded every frame: of a 1920x1080 FP32 grid at size 2
// (0.5 Mpixel, with the call and the copy to the host) 77 us for the amplitude and 144 us for the
// log energy, of which the copy is about 10.  Only 256 outcomes exist, so the index is first computed
// in FP32 with a bound on its distance from the FP64 one; where no palette boundary lies within
// twice the bound (all but about one pixel in a thousand) it is the index, and the other pixels
// take the FP64 path.  The frames are the same bytes: 37 and 58 us.  The modes with a running
// sum keep the sum in FP64 (150 to 74 us); the total flux is FP64 throughout (137 us, as before).
#pragma once
#include <cmath>
#include "wg_internal.h"

namespace wg {

// A block renders FT_ROWS x COLS pixels: a warp reads FT_ROWS frame rows of one column i
// (contiguous along j), and the colours go to the frame through shared memory, row by row.
// FT_COLS columns (32 columns a block measured the same on large frames and twice as slow on a 64x32
// one); half as many for the total flux, whose pixels are FP64 throughout and a chain: blocks that fit
// the SMs all at once, 32 registers a thread, and divide among them more evenly (1280x720 at size 2,
// 48 registers and 8 columns: 81 us; now 71 to 72, and 69 with a thread per pixel along i before).
constexpr int FT_ROWS = 32, FT_COLS = 8, FT_COLS_FLUX = 4;
__host__ __device__ inline int frame_tiles_x(int w, int cols = FT_COLS) { return (w + cols - 1) / cols; }
__host__ __device__ inline int frame_tiles_y(int h) { return (h + FT_ROWS - 1) / FT_ROWS; }

struct FrameFast {
    float vshift, vscale, k, range, log_shift, log_scale, flux, inv_t;  // k = slope/scale; range includes the attenuation
    float es2, half, halfb;  // E_SCALE^2 and the energy's gradient factors inside and outside
    float fade, inv_c2, ratio, ratio_b;  // FADE value; 1/COURANT^2, c2/c2 (1, or NaN), (COURANTB/COURANT)^2
    int plain;  // colours are palette bytes as they are: no fade, no obstacle fade
};

inline FrameFast frame_fast(const wg_frame_params &fp, const DevParams &p)
{
    FrameFast f;
    f.vshift = (float)fp.vshift;
    f.vscale = (float)fp.vscale;
    f.k = (float)(fp.slope / fp.scale);
    f.range = (float)(fp.color_range * (fp.attenuation != 0.0 ? exp(-((double)fp.time * fp.attenuation)) : 1.0));
    f.log_shift = (float)fp.log_shift;
    f.log_scale = (float)fp.log_scale;
    f.flux = (float)fp.flux_scale;
    f.inv_t = (float)(1.0 / (double)(fp.time + 1));
    f.es2 = (float)p.e_scale2;
    f.half = (float)p.ehalf_c2;
    f.halfb = (float)p.ehalf_c2b;
    f.fade = (float)fp.fade_value;
    f.inv_c2 = (float)(1.0 / p.c2);  // (the server's kernel, whose scenes differ, uses none of p's)
    f.ratio = (float)(p.c2 / p.c2);
    f.ratio_b = (float)(p.c2b / p.c2);
    f.plain = !fp.fade && !fp.fade_in_obstacle;
    // The error bounds leave out what FP32 loses below its smallest numbers.  That does not matter while
    // the factors of a value are 0 or within 1e-30..1e12; otherwise (k a NaN) every pixel takes FP64.
    const auto fits = [](double v) { return v == 0.0 || (fabs(v) >= 1e-30 && fabs(v) <= 1e12); };
    bool ok = fits(fp.slope / fp.scale) && fits(f.range);
    if (fp.plot == WG_P_AMPLITUDE) ok = ok && fits(fp.vscale);
    else ok = ok && fits(fp.log_scale) && fits(fp.flux_scale) && fits(f.inv_t) && fits(p.e_scale2) && fits(p.ehalf_c2) && fits(p.ehalf_c2b);
    if (!ok) f.k = NAN;
    if (!fits(p.c2b / p.c2)) f.ratio_b = NAN;
    return f;
}

// The palette index of the value v, known to within err (absolute); -1 where the bound leaves
// two indices.  Each FP32 operation is within 2^-23 relative, tanhf within 5e-7.
__device__ __forceinline__ int hue_fast(const FrameFast &f, float v, float err, bool asym)
{
    const float u = v * f.k, th = tanhf(u);
    const float et = fminf(err * fabsf(f.k) + 5e-7f * fabsf(u), 2.f) + 1e-6f;  // of tanh, whose slope is at most 1
    const float amp = f.range * th;
    const float hv = asym ? 256.f * amp : 128.f * (1.f + amp);
    const float m = 2.f * (256.f * (fabsf(f.range) * et + 4e-7f * fabsf(amp)) + 6e-5f);
    const float lo = hv - m, hi = hv + m;
    const int a = lo >= 255.f ? 255 : (lo <= 0.f ? 0 : (int)lo), b = hi >= 255.f ? 255 : (hi <= 0.f ? 0 : (int)hi);
    if (a == b && m < 64.f && hv == hv) return a;
    if (!asym && lo > 127.f && hi < 129.f) {
        // a field at rest, or ahead of a front, lies at the boundary of 127 and 128 itself: there
        // the sign decides, 1 + amp being 1 in FP64 where |amp| < 2^-54
        if (fabsf(f.range * f.k) * (fabsf(v) + err + 1e-37f) < 4e-17f) return 128;
        if (fabsf(v) > 2.f * err && (amp > 0.f || amp < -4e-16f)) return amp > 0.f ? 128 : 127;
    }
    return -1;
}

// The value of P_AMPLITUDE, VSHIFT + VSCALE*x, and its error.
__device__ __forceinline__ float amplitude_fast(const FrameFast &f, float x, float *err)
{
    const float sx = f.vscale * x;
    *err = 4e-7f * (fabsf(f.vshift) + fabsf(sx));
    return f.vshift + sx;
}

// cc/c2 of the obstacle fade, NaN (the colour then takes FP64) where FP32 may have lost digits of cc,
// c2 or the ratio to its smallest numbers.
__device__ __forceinline__ float fade_ratio(float cc, float inv_c2)
{
    const float r = cc * inv_c2;
    return inv_c2 >= 1e-30f && inv_c2 <= 1e30f && (cc == 0.f || (cc >= 1e-30f && r >= 1e-30f)) ? r : NAN;
}

// lut colour times f (known to within a relative rel), rounded, to o; false where the bound
// leaves two values for a byte.
__device__ __forceinline__ bool colour_fast(const uint8_t *lut, int hue, float f, float rel, uint8_t *o)
{
    bool ok = true;
    uint8_t c[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float v = (float)lut[hue * 3 + k] * f, m = (rel + 3e-7f) * fabsf(v) + 1e-6f;
        const int a = (int)(v - m + 0.5f), b = (int)(v + m + 0.5f);
        ok = ok && a == b && v - m > -0.4f && m < 1.f;  // (truncation; a NaN fails)
        c[k] = (uint8_t)(a > 255 ? 255 : a);
    }
    if (ok)
        for (int k = 0; k < 3; k++) o[k] = c[k];
    return ok;
}

// The colour of palette index hue times the optional fades, rounded, in FP64.
static __device__ __noinline__ void frame_colour64(const wg_frame_params &fp, const uint8_t *lut, int hue, double dim,
                                                   double cc, double c2, uint8_t *o)
{
    double f = dim;
    // (1 where cc is c2; NaN, and so black, where COURANT = 0 makes it 0/0)
    if (fp.fade_in_obstacle && !(cc == c2 && c2 > 0.0 && c2 < INFINITY)) f *= pow(cc / c2, 0.1);
    if (fp.fade) f *= fp.fade_value;
    for (int q = 0; q < 3; q++) {
        const double v = (double)lut[hue * 3 + q] * f;
        const int b = (int)(v + 0.5);
        o[q] = (uint8_t)(b > 255 ? 255 : (b < 0 ? 0 : b));
    }
}

// The block's colours, sh[row][3*col..], to the frame (w x h pixels, tile (tx, ty)); call after a
// barrier.
template <int COLS>
struct FrameTile {
    uint8_t c[FT_ROWS][3 * COLS + 4];
};
template <int COLS>
__device__ __forceinline__ void frame_tile_out(const FrameTile<COLS> &sh, uint8_t *out, int w, int h, int tx, int ty)
{
    const int n = 3 * min(COLS, w - tx * COLS), rows = min(FT_ROWS, h - ty * FT_ROWS);
    const int t = threadIdx.y * FT_ROWS + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int q = t + k * FT_ROWS * COLS, row = q / (3 * COLS), b = q - row * 3 * COLS;
        if (row < rows && b < n) out[((size_t)(ty * FT_ROWS + row) * w + (size_t)tx * COLS) * 3 + b] = sh.c[row][b];
    }
}

}  // namespace wg
