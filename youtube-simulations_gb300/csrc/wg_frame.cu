// wg_frame.cu — colour-mapped RGB8 frames of a scene (the serving output).
//
// draw_wave_highres_palette (wave_common.c:1750-1848) with wave_value (wave_common.c:
// 1053-1162) for the C_ONEDIM colour scheme (colors_waves.c:3-22, 161-258;
// colormaps.c:2449-2482) at every size-th cell.  The value of a sampled cell comes
// from the plot mode (phi, compute_energy, compute_energy_flux, and the running sums of
// the mean, exponential-average and total-flux modes, kept per sampled cell);
// amplitude = COLOR_RANGE*tanh(SLOPE*value/scale)*exp(-time*ATTENUATION); palette
// index (int)(256*h) with h = 0.5*(1 + amplitude) (color_scheme_palette) or h =
// amplitude (color_scheme_asym_palette: the energy and flux modes), clamped to 0..255.
// Drawn cells (TWOSPEEDS or xy != 0) get that palette colour times the optional
// factors, other cells black.  The reference hands floats to glColor3f; here the
// palette is the caller's byte table and the faded colour is rounded to bytes.
#include <cmath>
#include <type_traits>
#include "wg_internal.h"
#include "wg_frame.cuh"
#include "wg_scene.h"

namespace wg {

// argument() of sub_wave.c:287-302 with the reference's PI and PID constants.
__device__ __forceinline__ double ref_argument(double x, double y)
{
    const double PI_ = 3.141592654, PID_ = 1.570796327;
    double alph;
    if (x != 0.0) {
        alph = atan(y / x);
        if (x < 0.0) alph += PI_;
    } else {
        alph = PID_;
        if (y < 0.0) alph = PI_ * 1.5;
    }
    return alph;
}

// The sampled cell as it is stored: phi, psi (FP64 fields) or the velocity (FP32), and its
// neighbours' phi, clamped at the edges.
template <class T>
struct FrameRaw {
    T x, y, e, w, n, s;
    int m, j;
};
// The same in FP64; psi of FP32 fields is phi - v (exact in FP64).
struct FrameCell {
    double x, y, e, w, n, s;
    int m, j;
};
template <class T>
__device__ __forceinline__ FrameCell frame_cell(const FrameRaw<T> &r)
{
    const double x = (double)r.x;
    return FrameCell{x, sizeof(T) == 4 ? S_(x, (double)r.y) : (double)r.y, (double)r.e, (double)r.w, (double)r.n, (double)r.s, r.m, r.j};
}

// wave_value (wave_common.c:1053-1162) without the running sums: q is the mode's updated sum.
__device__ double frame_value(const DevParams &p, const wg_frame_params &fp, const FrameCell &c, double q)
{
    double energy;
    switch (fp.plot) {
    case WG_P_AMPLITUDE: return A_(fp.vshift, M_(fp.vscale, c.x));
    case WG_P_ENERGY: return cell_energy(p, c.x, c.y, c.e, c.w, c.n, c.s, c.m);
    case WG_P_MIXED: return (c.j > p.ny / 2) ? c.x : cell_energy(p, c.x, c.y, c.e, c.w, c.n, c.s, c.m);
    case WG_P_MEAN_ENERGY: return D_(q, (double)(fp.time + 1));
    case WG_P_LOG_ENERGY:
        energy = cell_energy(p, c.x, c.y, c.e, c.w, c.n, c.s, c.m);
        if (energy < 1.0e-20) energy = 1.0e-20;
        return A_(fp.log_shift, M_(fp.log_scale, log(energy)));
    case WG_P_LOG_MEAN_ENERGY: return A_(fp.log_shift, M_(fp.log_scale, log(D_(q, (double)(fp.time + 1)))));
    case WG_P_ENERGY_FLUX: {
        const double vel = fabs(S_(c.x, c.y)), gx = S_(c.e, c.w), gy = S_(c.n, c.s);
        const double mod = (c.m || p.twospeeds) ? M_(vel, sqrt(A_(M_(gx, gx), M_(gy, gy)))) : 0.0;
        return M_(mod, fp.flux_scale);
    }
    case WG_P_AVERAGE_ENERGY: return q;
    default:  // WG_P_LOG_AVERAGE_ENERGY
        return (q == 0.0) ? S_(fp.log_shift, M_(10.0, fp.log_scale)) : A_(fp.log_shift, M_(fp.log_scale, log(q)));
    }
}

// The modes drawn by color_scheme_asym_palette.
__device__ __forceinline__ bool frame_asym(int plot)
{
    return plot == WG_P_ENERGY || plot == WG_P_MEAN_ENERGY || plot == WG_P_ENERGY_FLUX || plot == WG_P_AVERAGE_ENERGY;
}

// The palette index in FP64, as the reference computes it.
template <class T>
__device__ __noinline__ int frame_hue64(const DevParams &p, const wg_frame_params &fp, const FrameRaw<T> &c, double q)
{
    double amp = M_(fp.color_range, tanh(D_(M_(fp.slope, frame_value(p, fp, frame_cell(c), q)), fp.scale)));
    if (fp.attenuation != 0.0) amp = M_(amp, exp(-M_((double)fp.time, fp.attenuation)));
    const double hv = M_(256.0, frame_asym(fp.plot) ? amp : M_(0.5, A_(1.0, amp)));
    return hv >= 255.0 ? 255 : (hv <= 0.0 ? 0 : (int)hv);
}

// The index and dimming of WG_P_TOTAL_ENERGY_FLUX, whose sum (mgx, mgy) has been updated.
__device__ __noinline__ int frame_hue_flux(const wg_frame_params &fp, double mgx, double mgy, double *dim)
{
    const double mod = sqrt(A_(M_(mgx, mgx), M_(mgy, mgy)));
    double arg = ref_argument(mgx, mgy);
    if (arg < 0.0) arg = A_(arg, 6.283185307);
    *dim = tanh(M_(mod, fp.flux_scale));
    double hh = M_(fp.slope, D_(arg, 6.283185307));  // C_ONEDIM_LINEAR with scale 1 (colors_waves.c:198-205)
    if (hh > 1.0) hh = S_(hh, 1.0);
    else if (hh < 0.0) hh = A_(hh, 1.0);
    const double hv = M_(256.0, hh);
    return hv >= 255.0 ? 255 : (hv <= 0.0 ? 0 : (int)hv);
}

// value +- err of the modes that need no FP64: LOG_SHIFT + LOG_SCALE*log(q) of q with relative
// error rel and absolute error tiny (FP64 where that is more than half of q: |log(1 - t)| is below
// 2t, the factor hue_fast takes, only for smaller t)
__device__ __forceinline__ float log_fast(const FrameFast &f, float q, float rel, float tiny, float *err)
{
    const float l = logf(q);
    *err = fabsf(f.log_scale) * (rel + tiny / q + 5e-7f * fabsf(l) + 2e-7f) + 3e-7f * (fabsf(f.log_shift) + fabsf(f.log_scale * l));
    if (!(tiny <= 0.5f * q)) *err = INFINITY;
    return f.log_shift + f.log_scale * l;
}

// One block per tile of pixels, a thread per pixel.  The running sums (acc) are kept column by
// column (k = col*h + row), as they are read.
template <class T, int COEF, int COLS>
__global__ void __launch_bounds__(FT_ROWS *COLS, COLS == FT_COLS_FLUX ? 16 : 0) k_frame_rgb8(const __grid_constant__ DevParams p, const T *__restrict__ phi,
                                                       const T *__restrict__ psi, const uint32_t *__restrict__ nz,
                                                       const T *__restrict__ tcc, const uint8_t *__restrict__ lut,
                                                       const __grid_constant__ wg_frame_params fp,
                                                       const __grid_constant__ FrameFast ff, double *__restrict__ acc,
                                                       uint8_t *__restrict__ out, int w, int h)
{
    __shared__ FrameTile<COLS> sh;
    const int row = blockIdx.y * FT_ROWS + threadIdx.x, col = blockIdx.x * COLS + threadIdx.y;
    if (col < w && row < h) {
        const int i = col * fp.size, j = row * fp.size, plot = fp.plot;
        uint8_t *o = &sh.c[threadIdx.x][3 * threadIdx.y];
        const size_t k = (size_t)col * h + row, c = (size_t)i * p.pitch + j;
        const int m = (nz[(size_t)i * p.wpitch + (j >> 5)] >> (j & 31)) & 1u;
        const bool drawn = p.twospeeds || m;
        constexpr bool F32 = sizeof(T) == 4;
        const T tx = phi[c];
        FrameRaw<T> raw{tx, (T)0, (T)0, (T)0, (T)0, (T)0, m, j};
        float value = 0.f, err = INFINITY;  // in FP32, when the mode allows
        double q = 0.0, dim = 1.0;
        int hue = -1;
        if (plot == WG_P_AMPLITUDE) {
            value = amplitude_fast(ff, (float)tx, &err);
        } else {
            const int ip = (i + 1 == p.nx) ? p.nx - 1 : i + 1, im = (i == 0) ? 0 : i - 1;
            const int jp = (j + 1 == p.ny) ? p.ny - 1 : j + 1, jm = (j == 0) ? 0 : j - 1;
            const T te = phi[(size_t)ip * p.pitch + j], tw = phi[(size_t)im * p.pitch + j];
            const T tn = phi[(size_t)i * p.pitch + jp], ts = phi[(size_t)i * p.pitch + jm], ty = psi[c];
            raw = FrameRaw<T>{tx, ty, te, tw, tn, ts, m, j};
            // the velocity and the differences, rounded once to FP32; the energy from them, all of
            // its terms of one sign: 12 roundings.  tiny: psi = phi - v loses what lies below 2^-53 of
            // phi, and squares what lies below the smallest float
            const auto dif = [](T a, T b) { return F32 ? (float)a - (float)b : (float)S_((double)a, (double)b); };
            const float x = (float)tx, v = F32 ? (float)ty : dif(tx, ty);
            const float de = dif(te, tx), dw = dif(tx, tw), dn = dif(tn, tx), ds = dif(tx, ts);
            const float half = m ? ff.half : ff.halfb, es2 = ff.es2;
            const float rel = 1.5e-6f, tiny = es2 * (4.5e-16f * fabsf(x) * fabsf(v) + 5e-32f * x * x + 1e-40f);
            const float en = drawn ? es2 * (v * v + half * ((de * de + dw * dw) + (dn * dn + ds * ds))) : 0.f;
            switch (plot) {
            case WG_P_MIXED:
                if (j > p.ny / 2) {
                    value = x;
                    err = 2e-7f * fabsf(x);
                    break;
                }  // else the energy
            case WG_P_ENERGY:
                value = en;
                err = rel * en + tiny;
                break;
            case WG_P_LOG_ENERGY:
                value = log_fast(ff, fmaxf(en, 1.0e-20f), rel, tiny, &err);
                break;
            case WG_P_ENERGY_FLUX: {
                const float gx = dif(te, tw), gy = dif(tn, ts), g = sqrtf(gx * gx + gy * gy);
                value = drawn ? fabsf(v) * g * ff.flux : 0.f;
                err = rel * fabsf(value) + fabsf(ff.flux) * (g * 4.5e-16f * fabsf(x) + fabsf(v) * 2e-19f) + 1e-37f;
                break;
            }
            case WG_P_TOTAL_ENERGY_FLUX: {
                const FrameCell fc = frame_cell(raw);
                const double vel = fabs(S_(fc.x, fc.y));
                const double fx = drawn ? M_(vel, S_(fc.e, fc.w)) : 0.0, fy = drawn ? M_(vel, S_(fc.n, fc.s)) : 0.0;
                const double mgx = A_(M_(acc[2 * k], 0.99), fx), mgy = A_(M_(acc[2 * k + 1], 0.99), fy);
                acc[2 * k] = mgx;
                acc[2 * k + 1] = mgy;
                if (drawn) hue = frame_hue_flux(fp, mgx, mgy, &dim);
                break;
            }
            default: {  // the modes with a running sum of the energy, kept in FP64
                const FrameCell fc = frame_cell(raw);
                double energy = cell_energy(p, fc.x, fc.y, fc.e, fc.w, fc.n, fc.s, m);
                if (plot == WG_P_AVERAGE_ENERGY || plot == WG_P_LOG_AVERAGE_ENERGY) {
                    q = A_(M_(fp.avrg_e_factor, acc[k]), M_(S_(1.0, fp.avrg_e_factor), energy));
                } else {
                    if (plot == WG_P_LOG_MEAN_ENERGY && energy == 0.0) energy = 1.0e-20;
                    q = A_(acc[k], energy);
                }
                acc[k] = q;
                const float qf = (float)q;
                if (plot == WG_P_MEAN_ENERGY || plot == WG_P_AVERAGE_ENERGY) {
                    value = plot == WG_P_MEAN_ENERGY ? qf * ff.inv_t : qf;
                    err = 4e-7f * fabsf(value) + 1e-37f;
                } else if (qf > 1e-30f) {
                    value = log_fast(ff, plot == WG_P_LOG_MEAN_ENERGY ? qf * ff.inv_t : qf, 4e-7f, 0.f, &err);
                }
                break;
            }
            }
        }
        if (!drawn) {
            o[0] = o[1] = o[2] = 0;
        } else {
            if (hue < 0 && err < 1e30f) hue = hue_fast(ff, value, err, frame_asym(plot));
            if (hue < 0) hue = frame_hue64<T>(p, fp, raw, q);
            if (ff.plain && plot != WG_P_TOTAL_ENERGY_FLUX) {
#pragma unroll
                for (int a = 0; a < 3; a++) o[a] = lut[hue * 3 + a];
            } else {
                double cc = p.c2;
                if (fp.fade_in_obstacle) cc = (COEF == WG_COEF_TABLE) ? (double)tcc[c] : (m ? p.c2 : p.c2b);
                // powf is within 4 ulp, its argument within 3e-7 (a tenth of which counts)
                float ff32 = (float)dim * (fp.fade ? ff.fade : 1.f);
                if (fp.fade_in_obstacle) ff32 *= powf((COEF == WG_COEF_TABLE) ? fade_ratio((float)tcc[c], ff.inv_c2) : (m ? ff.ratio : ff.ratio_b), 0.1f);
                if (!colour_fast(lut, hue, ff32, 8e-7f, o)) frame_colour64(fp, lut, hue, dim, cc, p.c2, o);
            }
        }
    }
    __syncthreads();
    frame_tile_out(sh, out, w, h, blockIdx.x, blockIdx.y);
}

// doubles of running state per sampled cell for a plot mode
static int frame_acc_per_cell(int plot)
{
    switch (plot) {
    case WG_P_MEAN_ENERGY: case WG_P_LOG_MEAN_ENERGY: case WG_P_AVERAGE_ENERGY: case WG_P_LOG_AVERAGE_ENERGY: return 1;
    case WG_P_TOTAL_ENERGY_FLUX: return 2;
    default: return 0;
    }
}

wg_status frame_launch(const DevParams &p, const void *phi, const void *psi, int prec, int coef, const uint32_t *nz,
                       const void *tcc, const uint8_t *lut, const wg_frame_params &fp, double *acc, uint8_t *out,
                       cudaStream_t st)
{
    const int w = p.nx / fp.size, h = p.ny / fp.size;
    const FrameFast ff = frame_fast(fp, p);
    const auto go = [&](auto cols, auto *x, auto *y, auto *t) {
        using T = std::remove_cv_t<std::remove_pointer_t<decltype(x)>>;
        constexpr int COLS = decltype(cols)::value;
        const auto kernel = coef == WG_COEF_TABLE ? k_frame_rgb8<T, WG_COEF_TABLE, COLS> : k_frame_rgb8<T, WG_COEF_MASK, COLS>;
        kernel<<<dim3(frame_tiles_x(w, COLS), frame_tiles_y(h)), dim3(FT_ROWS, COLS), 0, st>>>(p, x, y, nz, t, lut, fp, ff, acc, out, w, h);
    };
    const auto tiled = [&](auto *x, auto *y, auto *t) {
        if (fp.plot == WG_P_TOTAL_ENERGY_FLUX) go(std::integral_constant<int, FT_COLS_FLUX>(), x, y, t);
        else go(std::integral_constant<int, FT_COLS>(), x, y, t);
    };
    if (prec == WG_FP32) tiled((const float *)phi, (const float *)psi, (const float *)tcc);
    else tiled((const double *)phi, (const double *)psi, (const double *)tcc);
    WG_CUDA(cudaGetLastError());
    return WG_OK;
}

wg_status frame_validate(const wg_params &p, const wg_frame_params *fp, const uint8_t *lut)
{
    if (!fp || !lut) { set_error("frame parameters and palette are required"); return WG_ERR_INVALID; }
    if (fp->size < 1 || fp->size > p.nx || fp->size > p.ny) { set_error("frame size (downsampling) out of range"); return WG_ERR_INVALID; }
    if (!(fp->scale != 0.0)) { set_error("frame scale must be non-zero"); return WG_ERR_INVALID; }
    if (fp->plot < WG_P_AMPLITUDE || fp->plot > WG_P_LOG_AVERAGE_ENERGY) { set_error("unknown plot mode %d", fp->plot); return WG_ERR_INVALID; }
    return WG_OK;
}

}  // namespace wg

using namespace wg;

extern "C" wg_status wg_scene_frame_rgb8(wg_scene *s, const wg_frame_params *fp, const uint8_t *lut, uint8_t *rgb_host,
                                         void *rgb_device)
{
    if (!s) { set_error("NULL scene"); return WG_ERR_INVALID; }
    wg_status st = frame_validate(s->prm, fp, lut);
    if (st) return st;
    const size_t bytes = (size_t)(s->prm.nx / fp->size) * (s->prm.ny / fp->size) * 3;
    if (!s->lut) WG_CUDA(cudaMalloc(&s->lut, 768));
    WG_CUDA(cudaMemcpyAsync(s->lut, lut, 768, cudaMemcpyHostToDevice, s->st));
    uint8_t *dst = (uint8_t *)rgb_device;
    if (!dst) {
        if (s->rgb_bytes < bytes) {
            if (s->rgb) cudaFree(s->rgb);
            s->rgb = nullptr;
            s->rgb_bytes = 0;
            WG_CUDA(cudaMalloc(&s->rgb, bytes));
            s->rgb_bytes = bytes;
        }
        dst = s->rgb;
    }
    // running sums of the mean / average / total-flux modes, at frame resolution
    const int per = frame_acc_per_cell(fp->plot);
    if (per) {
        const size_t n = (size_t)(s->prm.nx / fp->size) * (s->prm.ny / fp->size) * per;
        if (!s->facc || s->facc_n != n || s->facc_plot != fp->plot || s->facc_size != fp->size) {
            if (s->facc) cudaFree(s->facc);
            s->facc = nullptr;
            WG_CUDA(cudaMalloc(&s->facc, n * sizeof(double)));
            WG_CUDA(cudaMemsetAsync(s->facc, 0, n * sizeof(double), s->st));
            s->facc_n = n;
            s->facc_plot = fp->plot;
            s->facc_size = fp->size;
        }
    }
    if ((st = frame_launch(s->dp, s->f[s->cur], s->f[1 - s->cur], s->prec, s->coef, s->nz, s->tcc, s->lut, *fp,
                           per ? s->facc : nullptr, dst, s->st)))
        return st;
    s->launches++;
    if (rgb_host) WG_CUDA(cudaMemcpyAsync(rgb_host, dst, bytes, cudaMemcpyDeviceToHost, s->st));
    return scene_check_flag(s);  // synchronises the stream (the image is ready on return)
}

extern "C" wg_status wg_scene_frame_reset(wg_scene *s)
{
    if (!s) { set_error("NULL scene"); return WG_ERR_INVALID; }
    if (s->facc) WG_CUDA(cudaMemsetAsync(s->facc, 0, s->facc_n * sizeof(double), s->st));
    return WG_OK;
}
