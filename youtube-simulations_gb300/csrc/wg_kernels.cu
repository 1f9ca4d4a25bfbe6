// wg_kernels.cu — single-update stepping kernels, Neumann gather, point source,
// energy reductions and small utility kernels for sm_103a.
//
//  k_step64       FP64 update in the reference's operation order, of native scenes (in
//                 place, the new level overwrites psi) and of the drop-in (int16 mask,
//                 tables, three buffers, writes exactly the cells wave_billiard.c:302-610
//                 writes; bit-identical).
//  k_step_bulk    FP32 update, interior rows: 1-bit masks, 16-byte vector loads along j;
//                 phi and velocity, increment form, into the other pair of fields.
//  k_step_edge    FP32, the four boundary lines and the point source.
//  k_neumann      Neumann gather of wave_billiard.c:379-389 for the active records.
//  k_energy_cols  compute_energy (wave_common.c:453-472) per cell, one warp per
//                 column: sums of j < ny/2 and j >= ny/2, box partials per block.
//  k_energy_final total and the six compute_energy_tblr boxes from the partials.
#include <algorithm>
#include <type_traits>
#include "wg_internal.h"
#include "wg_cells.cuh"
#include "wg_step64.cuh"

namespace wg {

// ---------------------------------------------------------------------------
// FP64 updates (scenes and the drop-in)
// ---------------------------------------------------------------------------
int sm_count()
{
    static PerDevice sms;
    return sms.get([] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return std::max(1, n);
    });
}

// One update: blocks of boundary-line cells, then a warp per strip of ST_COLS columns and `rows`
// rows (wg_step64.cuh).  3840x2160 two-medium table, GAMMA = 1e-4: 104 us an update
// (80 Gcell/s, FP64 pipe 75% busy), 166 with every operation on the FP64 pipe and the edge lines
// in a second launch; 1280x720 ellipse, no GAMMA: 10.6 us against 14.2.  16 warps per SM: 128
// registers (96 spill and measured 12% slower on tables).
template <int COEF, bool EXACT, int Z>
__global__ void __launch_bounds__(128, 4) k_step64(const __grid_constant__ DevParams p, const __grid_constant__ Strip64 a,
                                                   int edge_blocks, int strips, int rows, bool few, long long time)
{
    pdl_wait();  // launched by launch_pdl: the previous update has completed
    // The next launch may come from here on where this one leaves SMs free (few: no more blocks than
    // SMs: 71x88, 4.1 to 3.8 us an update), otherwise after the work: its blocks, resident early, would
    // crowd the SMs that this one leaves first, and a launch of less than a wave that is bound by
    // the FP64 pipe would run at their rate (650x2026, an update and an energy: 294 us so, 171 now).
    if (few) pdl_trigger();
    if ((int)blockIdx.x < edge_blocks) {  // a thread per boundary-line cell
        const int q = blockIdx.x * 128 + threadIdx.x;
        if (q < edge64_cells(p)) edge64_cell<COEF, EXACT>(p, a, q, time);
        return;
    }
    const int w = ((int)blockIdx.x - edge_blocks) * 4 + (threadIdx.x >> 5);
    const int chunk = w / strips, base = (w - chunk * strips) * ST_COLS, r0 = 1 + chunk * rows;
    if (r0 >= p.nx - 1) return;  // warp-uniform
    strip64<COEF, EXACT, Z>(p, a, base, r0, min(r0 + rows, p.nx - 1), time);
    if (!few) pdl_trigger();
}

template <int COEF, bool EXACT, int Z>
static void launch_step64_z(const DevParams &p, const Strip64 &a, long long time, cudaStream_t st)
{
    static PerDevice warps_on;
    const int resident = warps_on.get([] {  // warps on the device
        int per = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_step64<COEF, EXACT, Z>, 128, 0);
        return sm_count() * std::max(1, per) * 4;
    });
    // about three waves of warps: fewer leave SMs idle behind strips outside the domain, more
    // unpack too many rows twice (1280x720 ellipse, us an update by rows of a strip: 1: 12.0,
    // 2: 9.9, 3: 9.6 (chosen), 4: 10.1, 7: 10.9; 1920x1080 table: 3: 20.5, 5: 19.9 (chosen), 8: 20.6)
    const int strips = (p.ny + ST_COLS - 1) / ST_COLS;
    const int rows = (int)std::min(256LL, std::max(1LL, ((long long)(p.nx - 2) * strips + 3LL * resident - 1) / (3LL * resident)));
    const long long warps = (long long)strips * ((p.nx - 2 + rows - 1) / rows);
    const int edge_blocks = (edge64_cells(p) + 127) / 128;
    const long long blocks = edge_blocks + (warps + 3) / 4;
    launch_pdl(k_step64<COEF, EXACT, Z>, dim3((unsigned)blocks), dim3(128), 0, st, p, a, edge_blocks, strips, rows,
               blocks <= sm_count(), time);
}

// wave_energy's stepper (wave_energy.c:662-913) on the half domain j < ny/2, with
// its tables built from the mask (wave_energy.c:670-697).  The OSCILLATE_TOPBOT
// branch of that file reads outside its tables and is rejected on the host.
__global__ void __launch_bounds__(256) k_step_exact_energy(DevParams p, const double *__restrict__ phi,
                                                           const double *__restrict__ psi, double *__restrict__ out,
                                                           const int16_t *__restrict__ xy, long long time)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    const int NX = p.nx, jmid = p.ny / 2;
    if (i >= NX || j >= jmid) return;
    const int P = p.pitch;
    auto PHI = [&](int a, int b) { return phi[(size_t)a * P + b]; };
    auto XY = [&](int a, int b) { return (int)xy[(size_t)a * P + b]; };
    auto TCC = [&](int a, int b) { return XY(a, b) ? p.c2 : (p.twospeeds ? p.c2b : 0.0); };
    auto TC = [&](int a, int b) { return XY(a, b) ? p.courant : (p.twospeeds ? p.courantb : 0.0); };
    auto TG = [&](int a, int b) { return XY(a, b) ? p.gam : (p.twospeeds ? p.gamb : 0.0); };
    const size_t c = (size_t)i * P + j;
    const int m = XY(i, j);
    const bool active = p.twospeeds || m != 0;
    const double x = phi[c], y = psi[c];
    double v = 0.0, delta;
    bool w = false;
    if (j == jmid - 1 || j == 0) {
        const int jb = j, jn = (j == 0) ? 1 : jmid - 2, jw = (j == 0) ? jmid - 1 : 0;
        if (i == 0 && j == jmid - 1 && p.osc_left) { v = osc_bc(p, (int)time, j); w = true; }
        if (active) {
            int ip, im;
            switch (p.b_cond) {
            case 0:
                ip = i + 1; if (ip == NX) ip = NX - 1;
                im = i - 1; if (im == -1) im = 0;
                delta = S_(A_(A_(PHI(ip, jb), PHI(im, jb)), PHI(i, jn)), M_(3.0, x));
                v = upd64(x, y, TCC(i, jb), delta, p.kappa, TG(i, jb));
                break;
            case 1:
                ip = (i + 1) % NX; im = (i - 1) % NX; if (im < 0) im += NX;
                delta = S_(A_(A_(A_(PHI(ip, jb), PHI(im, jb)), PHI(i, jn)), PHI(i, jw)), M_(4.0, x));
                v = upd64(x, y, TCC(i, jb), delta, p.kappa, TG(i, jb));
                break;
            case 2:
                v = absorb64(x, y, TC(i, jb), PHI(i, jn), p.kappa_topbot, p.gamma_topbot);
                break;
            default:
                ip = i + 1; if (ip == NX) ip = NX - 1;
                im = i - 1; if (im == -1) im = 0;
                if (i == 0) v = absorb64(x, y, TC(0, jb), PHI(1, jb), p.kappa_sides, p.gamma_sides);
                else {
                    delta = S_(A_(A_(A_(PHI(ip, jb), PHI(im, jb)), PHI(i, jn)), PHI(i, jw)), M_(4.0, x));
                    v = upd64(x, y, TCC(i, jb), delta, p.kappa, TG(i, jb));
                }
                break;
            }
            w = true;
        }
    } else if (i == 0 && p.osc_left) {
        v = osc_bc(p, (int)time, j);
        w = true;
    } else if (i == 0 || i == NX - 1) {
        if (active) {
            const int in = (i == 0) ? 1 : NX - 2, iw = (i == 0) ? NX - 1 : 0;
            switch (p.b_cond) {
            case 0:
                delta = S_(A_(A_(PHI(in, j), PHI(i, j + 1)), PHI(i, j - 1)), M_(3.0, x));
                v = upd64(x, y, TCC(i, j), delta, p.kappa, TG(i, j));
                break;
            case 1:
                delta = S_(A_(A_(A_(PHI(in, j), PHI(iw, j)), PHI(i, j + 1)), PHI(i, j - 1)), M_(4.0, x));
                v = upd64(x, y, TCC(i, j), delta, p.kappa, TG(i, j));
                break;
            default:
                v = absorb64(x, y, TC(i, j), PHI(in, j), p.kappa_sides, p.gamma_sides);
                break;
            }
            w = true;
        }
    } else if (active) {
        delta = S_(A_(A_(A_(PHI(i + 1, j), PHI(i - 1, j)), PHI(i, j + 1)), PHI(i, j - 1)), M_(4.0, x));
        v = upd64(x, y, TCC(i, j), delta, p.kappa, TG(i, j));
        w = true;
    }
    if (p.floor_clamp && m != 0) {
        if (!w) { v = out[c]; w = true; }
        v = floor_clamp(p, v);
    }
    if (w) out[c] = v;
}

__global__ void k_cell_energy(DevParams p, const double *phi, const double *psi, const int16_t *xy, int i, int j,
                              double *out)
{
    const int NX = p.nx, NY = p.ny, P = p.pitch;
    const int ip = (i + 1 == NX) ? NX - 1 : i + 1, im = (i == 0) ? 0 : i - 1;
    const int jp = (j + 1 == NY) ? NY - 1 : j + 1, jm = (j == 0) ? 0 : j - 1;
    const size_t c = (size_t)i * P + j;
    *out = cell_energy(p, phi[c], psi[c], phi[(size_t)ip * P + j], phi[(size_t)im * P + j], phi[(size_t)i * P + jp],
                       phi[(size_t)i * P + jm], xy[c] != 0);
}

// Neumann gather for active records (drop-in form; records pre-validated to lie in
// 1..nx-2 x 1..ny-2 with in-range neighbours).
__global__ void k_neumann_exact(DevParams p, const double *__restrict__ phi, double *__restrict__ out,
                                const int16_t *__restrict__ xy, const wg_neumann_bc *__restrict__ rec, int n)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const wg_neumann_bc r = rec[q];
    if (!r.active) return;
    const size_t c = (size_t)r.i * p.pitch + r.j;
    double v = M_(r.nx, phi[(size_t)r.nbi1 * p.pitch + r.nbj1]);
    v = A_(v, M_(r.ny, phi[(size_t)r.nbi2 * p.pitch + r.nbj2]));
    if (p.floor_clamp && xy[c] != 0) v = floor_clamp(p, v);
    out[c] = v;
}

// vout (FP32 fields): the velocity takes the increment too.
template <class T>
__global__ void k_point_source(DevParams p, T *out, T *vout, long long time)
{
    const size_t c = (size_t)p.src_i * p.pitch + p.src_j;
    const double add = point_source(p, time);
    out[c] = (T)A_((double)out[c], add);
    if (vout) vout[c] = (T)A_((double)vout[c], add);
}

// ---------------------------------------------------------------------------
// Fast native kernel
// ---------------------------------------------------------------------------
// Interior rows 1..nx-2 of one FP32 update: each thread updates four consecutive cells of
// row i with every load (three phi rows, the velocity, tcc, the j-1 / j+4 neighbours, the
// mask word) issued before the first use, the new phi and velocity into the other pair.
// Boundary-line cells (j = 0, j = ny-1) and what padding shares a group of four with column ny-1
// take the rule of an unwritten cell; k_step_edge computes the boundary lines afterwards.  (Over
// the whole pitch, periodic scenes, whose rows hold ghosts, took 3 to 6% longer: 3840x2160
// 25.1 us an update, now 23.8.)
template <int COEF>
__global__ void __launch_bounds__(256) k_step_bulk(const __grid_constant__ DevParams p,
                                                   const __grid_constant__ FastArgs<float> a)
{
    constexpr int V = Vec<float>::n;
    pdl_wait();  // launched by launch_pdl: the previous update has completed
    pdl_trigger();
    const int i = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    const int j0 = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (i >= p.nx - 1 || j0 >= p.ny) return;
    const size_t row = (size_t)i * p.pitch;
    float c[V], y[V], n[V], s[V], cc[V];
    vload(a.phi + row + j0, c);
    vload(a.psi + row + j0, y);
    vload(a.phi + row + p.pitch + j0, n);
    vload(a.phi + row - p.pitch + j0, s);
    if (COEF == WG_COEF_TABLE) vload(a.tcc + row + j0, cc);
    const float wl = (j0 > 0) ? a.phi[row + j0 - 1] : 0.f;
    const float er = (j0 + V < p.pitch) ? a.phi[row + j0 + V] : 0.f;
    const uint32_t word = a.act[(size_t)i * p.wpitch + (j0 >> 5)] >> (j0 & 31);
    uint32_t nzw = 0;
    if (p.floor_clamp && a.has_ghosts) nzw = a.nz[(size_t)i * p.wpitch + (j0 >> 5)] >> (j0 & 31);
    float out[V], vo[V];
#pragma unroll
    for (int k = 0; k < V; k++) {
        const int j = j0 + k;
        const bool act = (word >> k) & 1u;
        const bool upd = j >= 1 && j < p.ny - 1 && (p.twospeeds || act);
        const bool clamp = p.floor_clamp && j >= 1 && j < p.ny - 1 && ((upd && act) || ((nzw >> k) & 1u));
        const float x = c[k];
        const float w = (k == 0) ? wl : c[k - 1];
        const float e = (k == V - 1) ? er : c[k + 1];
        XV r = keep32(x, y[k]);
        if (upd) {
            const float delta = ((n[k] - x) + (s[k] - x)) + ((e - x) + (w - x));
            const float ccv = (COEF == WG_COEF_TABLE) ? cc[k] : (act ? a.c2f : a.c2bf);
            float g;
            if (COEF == WG_COEF_TABLE) g = a.tg ? a.tg[row + j] : a.gamf;
            else g = act ? a.gamf : a.gambf;
            r = upd32(x, y[k], ccv, delta, a.kappaf, g);
        }
        if (clamp) r = clamp32(x, r, a.vmaxf);
        out[k] = r.x;
        vo[k] = r.v;
    }
    vstore(a.out + row + j0, out);
    vstore(a.vout + row + j0, vo);
}

// The four boundary lines of one FP32 update (one thread per cell, reference rules) and,
// in the last thread, the point source when it lies inside; runs after k_step_bulk
// (boundary cells read only phi and their own velocity).
template <int COEF>
__global__ void __launch_bounds__(256) k_step_edge(const __grid_constant__ DevParams p,
                                                   const __grid_constant__ FastArgs<float> a, long long time)
{
    pdl_wait();  // launched by launch_pdl: the bulk kernel of this update has completed
    pdl_trigger();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    const int NX = p.nx, NY = p.ny;
    const int nedge = 2 * NX + 2 * (NY - 2);
    int i, j;
    if (idx < NX) { i = idx; j = 0; }
    else if (idx < 2 * NX) { i = idx - NX; j = NY - 1; }
    else if (idx < 2 * NX + (NY - 2)) { i = 0; j = idx - 2 * NX + 1; }
    else if (idx < nedge) { i = NX - 1; j = idx - 2 * NX - (NY - 2) + 1; }
    else {
        if (idx == nedge && a.do_source && p.src_on && p.src_i > 0 && p.src_i < NX - 1 && p.src_j > 0 &&
            p.src_j < NY - 1) {
            const size_t o = (size_t)p.src_i * p.pitch + p.src_j;
            const double add = point_source(p, time);
            a.out[o] = (float)A_((double)a.out[o], add);
            a.vout[o] = (float)A_((double)a.vout[o], add);
        }
        return;
    }
    const size_t o = (size_t)i * p.pitch + j;
    const bool src = a.do_source && p.src_on && i == p.src_i && j == p.src_j;
    XV r = fast_edge_v<COEF>(p, a, i, j, time);
    if (src) r = source32(r, point_source(p, time));
    a.out[o] = r.x;
    a.vout[o] = r.v;
}

// Native Neumann gather: active records only, from phi (level t) into the new level
// (vout: FP32 fields, the velocity of the gathered value against the cell's phi at level
// t, in FP64).
template <class T>
__global__ void k_neumann_fast(DevParams p, const T *__restrict__ phi, T *__restrict__ out, T *__restrict__ vout,
                               const int4 *__restrict__ idx, const double2 *__restrict__ w, int n)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int4 r = idx[q];       // cell, nb1, nb2 (element offsets), flags (bit0 floor, bit1 inactive)
    if (r.w & 2) return;
    const double2 cw = w[q];
    double v = M_(cw.x, (double)phi[r.y]);
    v = A_(v, M_(cw.y, (double)phi[r.z]));
    if (p.floor_clamp && (r.w & 1)) v = floor_clamp(p, v);
    out[r.x] = (T)v;
    if (vout) vout[r.x] = (T)S_(v, (double)phi[r.x]);
}

// ---------------------------------------------------------------------------
// Energy
// ---------------------------------------------------------------------------
// Error-free FP32 double-word ("double-float") accumulator: h + l carries the running
// sum to about 2^-48 relative.  Every addition is Knuth's TwoSum (the rounding error of
// h + x, recovered exactly, goes into l); merges add the two high words by TwoSum and
// renormalise.  All of it runs on the FP32 pipe: on this GPU an FP64 operation costs
// about 64 FP32 operations, so the FP32 fields' sums stay off the FP64 pipe and are
// converted to FP64 (exactly) only per column.
// An aggregate like Neu: start it as {0.f, 0.f}.
struct DF {
    float h, l;
    __device__ __forceinline__ void add(float x)
    {
        const float s = __fadd_rn(h, x);
        const float bp = __fsub_rn(s, h);
        const float e = __fadd_rn(__fsub_rn(h, __fsub_rn(s, bp)), __fsub_rn(x, bp));
        h = s;
        l = __fadd_rn(l, e);
    }
    __device__ __forceinline__ void merge(const DF &o)
    {
        const float s = __fadd_rn(h, o.h);
        const float bp = __fsub_rn(s, h);
        const float e = __fadd_rn(__fsub_rn(h, __fsub_rn(s, bp)), __fsub_rn(o.h, bp));
        const float t = __fadd_rn(__fadd_rn(l, o.l), e);
        h = __fadd_rn(s, t);                  // Fast2Sum renormalisation (|s| >= |t|)
        l = __fsub_rn(t, __fsub_rn(h, s));
    }
    __device__ __forceinline__ double value() const { return A_((double)h, (double)l); }
};

// compute_energy in FP32 for FP32 fields (same formula and order as cell_energy), with
// the stored velocity v in place of phi - psi.
__device__ __forceinline__ float cell_energy32(float es2, float hc2, float hc2b, int twospeeds, float x, float v,
                                               float e, float w, float n, float s, int m)
{
    float a = e - x, b = x - w, c = n - x, d = x - s;
    float g = (a * a + b * b) + (c * c + d * d);
    if (m) return es2 * (v * v + hc2 * g);
    if (twospeeds) return es2 * (v * v + hc2b * g);
    return 0.0f;
}

// Merges the accumulators of the 32 lanes into lane 0 (value and compensation travel).
__device__ __forceinline__ void warp_merge(Neu &a)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        Neu o = {0.0, 0.0};
        o.s = __shfl_down_sync(0xffffffffu, a.s, off);
        o.c = __shfl_down_sync(0xffffffffu, a.c, off);
        a.merge(o);
    }
}
__device__ __forceinline__ void warp_merge(DF &a)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        DF o = {0.f, 0.f};
        o.h = __shfl_down_sync(0xffffffffu, a.h, off);
        o.l = __shfl_down_sync(0xffffffffu, a.l, off);
        a.merge(o);
    }
}
__device__ __forceinline__ void acc_add(Neu &a, double x) { a.add(x); }
__device__ __forceinline__ void acc_add(DF &a, float x) { a.add(x); }
__device__ __forceinline__ void acc_merge(Neu &a, const Neu &o) { a.merge(o); }
__device__ __forceinline__ void acc_merge(DF &a, const DF &o) { a.merge(o); }

// One warp per column i, eight columns per block.  MASK: 0 = int16 (xy != 0), 1 =
// "nonzero" bit plane.  Per cell compute_energy (wave_common.c:453-472): FP64 for FP64
// fields, FP32 for FP32 fields.  Every reduction is compensated: FP64 fields add their
// cell energies into FP64 Neumaier accumulators; FP32 fields into the error-free FP32
// double-word accumulator DF above.  Lanes merge (value and compensation) into the
// column sums of compute_energy_x (wave_energy.c:292-302); the block merges the six
// boxes of compute_energy_tblr (sub_wave_comp.c:1752-1800) over its columns, and its
// total.  cols[i] = (sum over j < ny/2, sum over j >= ny/2); part[6 b + k] = box k of
// block b (0..2 top left/mid/right, 3..5 bottom); the block's total overwrites
// cols[8 b].y (already folded into the boxes).  FP32 fields: psi is the velocity.
#define ENERGY_COLS_PER_BLOCK 8
template <class T, int MASK>
__global__ void __launch_bounds__(32 * ENERGY_COLS_PER_BLOCK)
    k_energy_cols(const __grid_constant__ DevParams p, const T *__restrict__ phi, const T *__restrict__ psi,
                  const int16_t *__restrict__ xy, const uint32_t *__restrict__ nz, int ileft, int iright,
                  double2 *__restrict__ cols, double *__restrict__ part)
{
    using Acc = typename std::conditional<sizeof(T) == 8, Neu, DF>::type;
    __shared__ Acc sh[ENERGY_COLS_PER_BLOCK][2];
    __shared__ Acc sbx[6];
    __shared__ int sbox[ENERGY_COLS_PER_BLOCK];
    pdl_wait();  // launched by launch_pdl: the update that wrote the fields has completed
    pdl_trigger();
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * ENERGY_COLS_PER_BLOCK + wid;
    Acc ab = {0, 0}, at = {0, 0};  // bottom (j < ny/2) and top halves of the column
    if (i < p.nx) {
        const int NX = p.nx, NY = p.ny, jmid = NY / 2;
        const size_t row = (size_t)i * p.pitch;
        const int ip = (i + 1 == NX) ? NX - 1 : i + 1, im = (i == 0) ? 0 : i - 1;
        const T *re = phi + (size_t)ip * p.pitch, *rw = phi + (size_t)im * p.pitch, *rc = phi + row, *ry = psi + row;
        const float es2 = (float)p.e_scale2, hc2 = (float)p.ehalf_c2, hc2b = (float)p.ehalf_c2b;
        if (sizeof(T) == 4 && MASK == 1) {
            // FP32 fields: four cells per lane and step as 16-byte loads of the rows i-1, i, i+1
            // and the velocity; the j-1 / j+1 neighbours from the adjacent lanes (the row pitch is a
            // multiple of 128 elements, so every load stays in the row)
            const float *fc = (const float *)rc, *fy = (const float *)ry, *fe = (const float *)re,
                        *fw = (const float *)rw;
            const uint32_t *nzr = nz + (size_t)i * p.wpitch;
            for (int base = 0; base < NY; base += 128) {
                const int j0 = base + 4 * lane;
                const float4 c4 = *reinterpret_cast<const float4 *>(fc + j0);
                const float4 y4 = *reinterpret_cast<const float4 *>(fy + j0);
                const float4 e4 = *reinterpret_cast<const float4 *>(fe + j0);
                const float4 w4 = *reinterpret_cast<const float4 *>(fw + j0);
                float left = __shfl_up_sync(0xffffffffu, c4.w, 1), right = __shfl_down_sync(0xffffffffu, c4.x, 1);
                if (lane == 0) left = (j0 > 0) ? fc[j0 - 1] : c4.x;
                if (lane == 31) right = (j0 + 4 < NY) ? fc[j0 + 4] : c4.w;
                const uint32_t bits = (nzr[j0 >> 5] >> (j0 & 31)) & 0xFu;
                const float xs[4] = {c4.x, c4.y, c4.z, c4.w}, ys[4] = {y4.x, y4.y, y4.z, y4.w};
                const float es[4] = {e4.x, e4.y, e4.z, e4.w}, ws[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int j = j0 + k;
                    if (j >= NY) break;
                    float jn = (k < 3) ? xs[k < 3 ? k + 1 : 3] : right;
                    float js = (k > 0) ? xs[k > 0 ? k - 1 : 0] : left;
                    if (j == NY - 1) jn = xs[k];  // clamped at the boundary lines
                    if (j == 0) js = xs[k];
                    const float en = cell_energy32(es2, hc2, hc2b, p.twospeeds, xs[k], ys[k], es[k], ws[k], jn, js,
                                                   (int)((bits >> k) & 1u));
                    acc_add(j < jmid ? ab : at, en);
                }
            }
        } else {
#pragma unroll 4
            for (int j = lane; j < NY; j += 32) {
                const int jp = (j + 1 == NY) ? NY - 1 : j + 1, jm = (j == 0) ? 0 : j - 1;
                int m;
                if (MASK == 0) m = xy[row + j] != 0;
                else m = (nz[(size_t)i * p.wpitch + (j >> 5)] >> (j & 31)) & 1u;
                if (sizeof(T) == 8) {
                    const double en = cell_energy(p, (double)rc[j], (double)ry[j], (double)re[j], (double)rw[j],
                                                  (double)rc[jp], (double)rc[jm], m);
                    acc_add(j < jmid ? ab : at, en);
                } else {
                    const float en = cell_energy32(es2, hc2, hc2b, p.twospeeds, (float)rc[j], (float)ry[j],
                                                   (float)re[j], (float)rw[j], (float)rc[jp], (float)rc[jm], m);
                    acc_add(j < jmid ? ab : at, en);
                }
            }
        }
    }
    warp_merge(ab);
    warp_merge(at);
    if (lane == 0) {
        if (i < p.nx) cols[i] = make_double2(ab.value(), at.value());
        sh[wid][0] = ab;
        sh[wid][1] = at;
        sbox[wid] = (i < ileft) ? 0 : (i < iright ? 1 : 2);
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int k = threadIdx.x, box = k % 3, half = k < 3 ? 1 : 0;  // top boxes sum j >= ny/2
        Acc acc = {0, 0};
#pragma unroll
        for (int w = 0; w < ENERGY_COLS_PER_BLOCK; w++)
            if (sbox[w] == box) acc_merge(acc, sh[w][half]);
        part[(size_t)blockIdx.x * 6 + k] = acc.value();
        sbx[k] = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        Acc t = {0, 0};
#pragma unroll
        for (int k = 0; k < 6; k++) acc_merge(t, sbx[k]);
        cols[(size_t)blockIdx.x * ENERGY_COLS_PER_BLOCK].y = t.value();
    }
}

// One block per output: block k < 6 merges box k over the blocks of k_energy_cols into
// out[1 + k] (top left/mid/right, bottom left/mid/right); block 6 merges the blocks'
// totals into out[0]; all of them copy the first ncols column sums over j < ny/2 into out[7..].
// out may be page-locked host memory; *flag (when not NULL) goes to *hflag beside it.  FP64 Neumaier
// per thread, then merged across the warp and the block.  With one warp per output (480 partial
// sums in a chain of 15 reads) and copies of the sums and of the flag to the host, an energy of an
// FP32 scene took 45 us at 3840x2160 and 26 us at 256x192; 37 and 19 us now.
constexpr int ENERGY_FINAL_WARPS = 8;
__global__ void __launch_bounds__(32 * ENERGY_FINAL_WARPS)
    k_energy_final(int ncols, int nblocks, const double2 *__restrict__ cols, const double *__restrict__ part,
                   double *__restrict__ out, const int *__restrict__ flag, int *__restrict__ hflag)
{
    __shared__ Neu sh[ENERGY_FINAL_WARPS];
    pdl_wait();  // launched by launch_pdl: k_energy_cols has completed
    pdl_trigger();
    constexpr int N = 32 * ENERGY_FINAL_WARPS;
    const int k = blockIdx.x, t = threadIdx.x;
    for (int i = k * N + t; i < ncols; i += 7 * N) out[7 + i] = cols[i].x;
    Neu acc = {0.0, 0.0};
    for (int b = t; b < nblocks; b += N)
        acc.add(k < 6 ? part[(size_t)b * 6 + k] : cols[(size_t)b * ENERGY_COLS_PER_BLOCK].y);
    warp_merge(acc);
    if ((t & 31) == 0) sh[t >> 5] = acc;
    __syncthreads();
    if (t == 0) {
        for (int w = 1; w < ENERGY_FINAL_WARPS; w++) acc.merge(sh[w]);
        out[k < 6 ? 1 + k : 0] = acc.value();
        if (k == 0 && flag) *hflag = *flag;
    }
}

// ---------------------------------------------------------------------------
// Utilities
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_count_nonfinite(int nx, int ny, int pitch, const T *__restrict__ a, unsigned long long *count)
{
    unsigned long long local = 0;
    const size_t total = (size_t)nx * pitch;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < total; c += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)(c % pitch);
        if (j < ny && !isfinite((double)a[c])) local++;
    }
    if (local) atomicAdd(count, local);
}

// Packs the int16 mask into the "active" plane (bulk test xy > 0, boundary-line test
// xy != 0) and the "nonzero" plane (xy != 0).  One thread per 32-bit word.
__global__ void k_pack_mask(int nx, int ny, int wpitch, const int16_t *__restrict__ xy, uint32_t *__restrict__ act,
                            uint32_t *__restrict__ nz)
{
    const int wj = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (wj >= wpitch || i >= nx) return;
    uint32_t a = 0, z = 0;
    for (int b = 0; b < 32; b++) {
        const int j = wj * 32 + b;
        if (j >= ny) break;
        const int m = xy[(size_t)i * ny + j];
        const bool edge = (i == 0 || i == nx - 1 || j == 0 || j == ny - 1);
        if (edge ? (m != 0) : (m > 0)) a |= 1u << b;
        if (m != 0) z |= 1u << b;
    }
    act[(size_t)i * wpitch + wj] = a;
    nz[(size_t)i * wpitch + wj] = z;
}

// Dense FP64 [nx][ny] -> pitched T [nx][pitch] (padding zeroed).
template <class T>
__global__ void k_convert_in(int nx, int ny, int pitch, const double *__restrict__ src, T *__restrict__ dst)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (j >= pitch || i >= nx) return;
    dst[(size_t)i * pitch + j] = (j < ny) ? (T)src[(size_t)i * ny + j] : (T)0;
}
// Dense [nx][ny] rows of the field precision into the pitched layout (padding zeroed).
template <class T>
__global__ void k_repack_in(int nx, int ny, int pitch, const T *__restrict__ src, T *__restrict__ dst)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (j >= pitch || i >= nx) return;
    dst[(size_t)i * pitch + j] = (j < ny) ? src[(size_t)i * ny + j] : (T)0;
}
// a - b of two floats rounded once to FP32, i.e. the FP32 subtraction.  The difference
// computed in FP64 and then rounded to FP32 is the same value (53 >= 2*24 + 2 bits, so the
// double rounding is innocuous for a sum of two floats), without the FP64 pipe.
__device__ __forceinline__ float dif32(float a, float b) { return __fsub_rn(a, b); }

// FP32 state from host (phi, psi) rows, dense [nx][ny] of H = double or float: phi
// rounded once, the velocity phi - psi computed exactly and rounded once (FP64 rows: in
// FP64; FP32 rows: dif32); padding zeroed.  The rows may be the caller's page-locked
// host memory, read in place.
template <class H>
__global__ void k_state_in32(int nx, int ny, int pitch, const H *__restrict__ phi, const H *__restrict__ psi,
                             float *__restrict__ x, float *__restrict__ v)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (j >= pitch || i >= nx) return;
    const size_t o = (size_t)i * pitch + j, c = (size_t)i * ny + j;
    if constexpr (sizeof(H) == 4) {
        const float a = j < ny ? phi[c] : 0.f, b = j < ny ? psi[c] : 0.f;
        x[o] = a;
        v[o] = dif32(a, b);
    } else {
        const double a = j < ny ? phi[c] : 0.0, b = j < ny ? psi[c] : 0.0;
        x[o] = (float)a;
        v[o] = (float)S_(a, b);
    }
}
// The same for FP32 host rows four columns per thread (ny a multiple of 4, so every dense
// row starts on 16 bytes), padding zeroed.
__global__ void k_state_in32_v4(int nx, int ny, int pitch, const float4 *__restrict__ phi,
                                const float4 *__restrict__ psi, float *__restrict__ x, float *__restrict__ v)
{
    const int j = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int i = blockIdx.y;
    if (j >= pitch || i >= nx) return;
    const size_t o = (size_t)i * pitch + j;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (j < ny) {
        const size_t c = ((size_t)i * ny + j) / 4;
        a = phi[c];
        b = psi[c];
    }
    const float4 dv = make_float4(dif32(a.x, b.x), dif32(a.y, b.y), dif32(a.z, b.z), dif32(a.w, b.w));
    *reinterpret_cast<float4 *>(x + o) = a;
    *reinterpret_cast<float4 *>(v + o) = dv;
}

// The same rows into a stage in device memory (launch_state_stage: both on 16 bytes, room for a last
// group of V cells): a thread forms V cells of both, since psi shares phi's read and, in FP64 rows, its
// conversion, which the FP64 pipe does.  With k_state_out a download of an FP32 scene into pageable
// FP64 rows took 841 us at 3840x2160 and 239 at 1920x1080; 768 and 218 so.
template <class T, class H>
__global__ void __launch_bounds__(256)
    k_state_stage(int ny, int pitch, long long n, const T *__restrict__ x0, const T *__restrict__ y0,
                  const T *__restrict__ x1, const T *__restrict__ y1, const int *__restrict__ sel, H *__restrict__ phi,
                  H *__restrict__ psi)
{
    constexpr int V = 16 / sizeof(H);
    const long long e0 = ((long long)blockIdx.x * 256 + threadIdx.x) * V;
    if (e0 >= n) return;
    const bool second = sel && *sel;
    const T *const x = second ? x1 : x0, *const y = second ? y1 : y0;
    const long long i = n < (1ll << 31) ? (long long)((unsigned)e0 / (unsigned)ny) : e0 / ny;
    int j = (int)(e0 - i * ny);
    long long o = i * pitch + j;
    alignas(16) H a[V], b[V];
#pragma unroll
    for (int k = 0; k < V; k++) {
        const bool in = e0 + k < n;
        const T xv = in ? x[o] : (T)0, yv = in && psi ? y[o] : (T)0;
        a[k] = (H)xv;
        if constexpr (sizeof(T) == 8) b[k] = (H)yv;
        else if constexpr (sizeof(H) == 4) b[k] = dif32(xv, yv);
        else b[k] = S_((double)xv, (double)yv);
        o++;
        if (++j == ny) {
            j = 0;
            o += pitch - ny;
        }
    }
    if (phi) *reinterpret_cast<uint4 *>(phi + e0) = *reinterpret_cast<const uint4 *>(a);
    if (psi) *reinterpret_cast<uint4 *>(psi + e0) = *reinterpret_cast<const uint4 *>(b);
}

// State to dense host rows (blockIdx.y 0: phi, 1: psi; either may be NULL): FP32 fields hold phi
// and v, and psi = phi - v is formed exactly and rounded once to H (FP64 rows: in FP64; FP32
// rows: dif32); FP64 fields hold phi and psi.  The rows may be the caller's page-locked host
// memory, written in place.  *sel (when not NULL) chooses the second pair of fields.
//
// A thread writes 16 aligned bytes of the dense rows whatever ny is, and a warp four whole lines
// of 128 bytes, since the host link takes a partial line as slowly as a whole one.  A download
// into page-locked rows, with a block per grid row before: 1920x1080 FP32 110 to 100 us, 1277x717
// FP32 61 to 52 us, 3840x2160 FP64 (by 2D copies) 837 to 702 us, 189 GB/s of the link's 191.
template <class T, class H>
__global__ void __launch_bounds__(256)
    k_state_out(int ny, int pitch, long long n, const T *__restrict__ x0, const T *__restrict__ y0,
                const T *__restrict__ x1, const T *__restrict__ y1, const int *__restrict__ sel, H *__restrict__ phi,
                H *__restrict__ psi)
{
    constexpr int V = 16 / sizeof(H);
    H *const out = blockIdx.y ? psi : phi;
    if (!out) return;
    const int shift = (int)(((unsigned long long)out & 127u) / sizeof(H));  // the first line's missing cells
    const long long e0 = ((long long)blockIdx.x * 256 + threadIdx.x) * V - shift;
    if (e0 >= n || e0 + V <= 0) return;
    const bool second = sel && *sel;
    const T *const x = second ? x1 : x0, *const y = second ? y1 : y0;
    const long long ef = e0 < 0 ? 0 : e0;
    const long long i = n < (1ll << 31) ? (long long)((unsigned)ef / (unsigned)ny) : ef / ny;
    int j = (int)(ef - i * ny);
    long long o = i * pitch + j;
    alignas(16) H r[V];
#pragma unroll
    for (int k = 0; k < V; k++) {
        r[k] = (H)0;
        if (e0 + k < 0 || e0 + k >= n) continue;
        if (blockIdx.y == 0) r[k] = (H)x[o];
        else if constexpr (sizeof(T) == 8) r[k] = (H)y[o];
        else if constexpr (sizeof(H) == 4) r[k] = dif32(x[o], y[o]);
        else r[k] = S_((double)x[o], (double)y[o]);
        o++;
        if (++j == ny) {
            j = 0;
            o += pitch - ny;
        }
    }
    if (e0 >= 0 && e0 + V <= n) {
        *reinterpret_cast<uint4 *>(out + e0) = *reinterpret_cast<const uint4 *>(r);
    } else {
#pragma unroll
        for (int k = 0; k < V; k++)
            if (e0 + k >= 0 && e0 + k < n) out[e0 + k] = r[k];
    }
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
void launch_step_exact(const DevParams &p, const double *phi, const double *psi, double *out, const int16_t *xy,
                       const double *tcc, const double *tc, const double *tg, long long time, int do_source,
                       cudaStream_t st)
{
    const Strip64 a{phi, psi, out, nullptr, nullptr, xy, tcc, tc, tg, 0, do_source};
    if (p.kappa == 0.0) launch_step64_z<WG_COEF_TABLE, true, Z_KAPPA>(p, a, time, st);
    else launch_step64_z<WG_COEF_TABLE, true, 0>(p, a, time, st);
}

void launch_step_exact_energy(const DevParams &p, const double *phi, const double *psi, double *out,
                              const int16_t *xy, long long time, cudaStream_t st)
{
    dim3 blk(64, 4), grd((p.ny / 2 + 63) / 64, (p.nx + 3) / 4);
    k_step_exact_energy<<<grd, blk, 0, st>>>(p, phi, psi, out, xy, time);
}

void launch_cell_energy(const DevParams &p, const double *phi, const double *psi, const int16_t *xy, int i, int j,
                        double *out, cudaStream_t st)
{
    k_cell_energy<<<1, 1, 0, st>>>(p, phi, psi, xy, i, j, out);
}

void launch_neumann_exact(const DevParams &p, const double *phi, double *out, const int16_t *xy,
                          const wg_neumann_bc *rec, int n, cudaStream_t st)
{
    if (n <= 0) return;
    k_neumann_exact<<<(n + 255) / 256, 256, 0, st>>>(p, phi, out, xy, rec, n);
}

template <class T>
void launch_point_source(const DevParams &p, T *out, T *vout, long long time, cudaStream_t st)
{
    k_point_source<T><<<1, 1, 0, st>>>(p, out, vout, time);
}
template void launch_point_source<float>(const DevParams &, float *, float *, long long, cudaStream_t);
template void launch_point_source<double>(const DevParams &, double *, double *, long long, cudaStream_t);

// The FP64 update without the terms whose coefficient is zero on every cell (upd64's Z flags:
// KAPPA = 0; GAMMA = 0 as a uniform value); the values are unchanged.
template <int COEF>
static void launch_step64(const DevParams &p, const FastArgs<double> &f, long long time, cudaStream_t st)
{
    const Strip64 a{f.phi, f.psi, f.out, f.act, f.nz, nullptr, f.tcc, f.tc, f.tg, f.has_ghosts, f.do_source};
    const bool g0 = (COEF == WG_COEF_TABLE) ? (!f.tg && p.gam == 0.0) : (p.gam == 0.0 && p.gamb == 0.0);
    switch ((p.kappa == 0.0 ? Z_KAPPA : 0) | (g0 ? Z_GAMMA : 0)) {
    case Z_KAPPA: launch_step64_z<COEF, false, Z_KAPPA>(p, a, time, st); return;
    case Z_GAMMA: launch_step64_z<COEF, false, Z_GAMMA>(p, a, time, st); return;
    case Z_KAPPA | Z_GAMMA: launch_step64_z<COEF, false, Z_KAPPA | Z_GAMMA>(p, a, time, st); return;
    default: launch_step64_z<COEF, false, 0>(p, a, time, st); return;
    }
}

template <>
int launch_step_fast<double>(const DevParams &p, const FastArgs<double> &a, int coef_mode, long long time, cudaStream_t st)
{
    if (coef_mode == WG_COEF_MASK) launch_step64<WG_COEF_MASK>(p, a, time, st);
    else launch_step64<WG_COEF_TABLE>(p, a, time, st);
    return 1;
}

template <>
int launch_step_fast<float>(const DevParams &p, const FastArgs<float> &a, int coef_mode, long long time, cudaStream_t st)
{
    constexpr int V = Vec<float>::n;
    dim3 blk(64, 4), grd(((p.ny + V - 1) / V + 63) / 64, (p.nx - 2 + 3) / 4);
    const int nedge = 2 * p.nx + 2 * (p.ny - 2) + 1;
    if (coef_mode == WG_COEF_MASK) {
        launch_pdl(k_step_bulk<WG_COEF_MASK>, grd, blk, 0, st, p, a);
        launch_pdl(k_step_edge<WG_COEF_MASK>, dim3((nedge + 255) / 256), dim3(256), 0, st, p, a, time);
    } else {
        launch_pdl(k_step_bulk<WG_COEF_TABLE>, grd, blk, 0, st, p, a);
        launch_pdl(k_step_edge<WG_COEF_TABLE>, dim3((nedge + 255) / 256), dim3(256), 0, st, p, a, time);
    }
    return 2;
}

template <class T>
void launch_neumann_fast(const DevParams &p, const T *phi, T *out, T *vout, const int4 *idx, const double2 *w, int n,
                         cudaStream_t st)
{
    if (n <= 0) return;
    k_neumann_fast<T><<<(n + 255) / 256, 256, 0, st>>>(p, phi, out, vout, idx, w, n);
}
template void launch_neumann_fast<float>(const DevParams &, const float *, float *, float *, const int4 *, const double2 *, int, cudaStream_t);
template void launch_neumann_fast<double>(const DevParams &, const double *, double *, double *, const int4 *, const double2 *, int, cudaStream_t);

template <class T>
void launch_energy(const DevParams &p, const T *phi, const T *psi, const int16_t *xy, const uint32_t *nz,
                   double2 *bot, double2 *top, int ileft, int iright, double *out, int ncols, const int *flag, int *hflag,
                   cudaStream_t st)
{
    // bot: per-column sums; top (2 nx doubles): six box partials per block of 8 columns
    const int nblocks = (p.nx + ENERGY_COLS_PER_BLOCK - 1) / ENERGY_COLS_PER_BLOCK;
    double *part = reinterpret_cast<double *>(top);
    const dim3 g(nblocks), b(32 * ENERGY_COLS_PER_BLOCK);
    if (xy) launch_pdl(k_energy_cols<T, 0>, g, b, 0, st, p, phi, psi, xy, nz, ileft, iright, bot, part);
    else launch_pdl(k_energy_cols<T, 1>, g, b, 0, st, p, phi, psi, xy, nz, ileft, iright, bot, part);
    launch_pdl(k_energy_final, dim3(7), dim3(32 * ENERGY_FINAL_WARPS), 0, st, ncols, nblocks, (const double2 *)bot,
               (const double *)part, out, flag, hflag);
}
template void launch_energy<float>(const DevParams &, const float *, const float *, const int16_t *, const uint32_t *, double2 *, double2 *, int, int,
                                double *, int, const int *, int *, cudaStream_t);
template void launch_energy<double>(const DevParams &, const double *, const double *, const int16_t *, const uint32_t *, double2 *, double2 *, int, int,
                                 double *, int, const int *, int *, cudaStream_t);

template <class T>
void launch_count_nonfinite(int nx, int ny, int pitch, const T *a, unsigned long long *count, cudaStream_t st)
{
    k_count_nonfinite<T><<<4 * sm_count(), 256, 0, st>>>(nx, ny, pitch, a, count);
}
template void launch_count_nonfinite<float>(int, int, int, const float *, unsigned long long *, cudaStream_t);
template void launch_count_nonfinite<double>(int, int, int, const double *, unsigned long long *, cudaStream_t);

void launch_pack_mask(int nx, int ny, int wpitch, const int16_t *xy, uint32_t *act, uint32_t *nz, cudaStream_t st)
{
    dim3 grd((wpitch + 127) / 128, nx);
    k_pack_mask<<<grd, 128, 0, st>>>(nx, ny, wpitch, xy, act, nz);
}

template <class T>
void launch_convert_in(int nx, int ny, int pitch, const double *src, T *dst, cudaStream_t st)
{
    dim3 grd((pitch + 255) / 256, nx);
    k_convert_in<T><<<grd, 256, 0, st>>>(nx, ny, pitch, src, dst);
}
template <class T>
void launch_repack_in(int nx, int ny, int pitch, const T *src, T *dst, cudaStream_t st)
{
    dim3 grd((pitch + 255) / 256, nx);
    k_repack_in<T><<<grd, 256, 0, st>>>(nx, ny, pitch, src, dst);
}
template void launch_repack_in<float>(int, int, int, const float *, float *, cudaStream_t);
template void launch_repack_in<double>(int, int, int, const double *, double *, cudaStream_t);
template void launch_convert_in<float>(int, int, int, const double *, float *, cudaStream_t);
template void launch_convert_in<double>(int, int, int, const double *, double *, cudaStream_t);

// dense FP32 rows of ny % 4 == 0 columns from 16-byte aligned bases take the 4-wide kernels
static bool rows_v4(int ny, const void *a, const void *b)
{
    return ny % 4 == 0 && ((uintptr_t)a & 15) == 0 && ((uintptr_t)b & 15) == 0;
}
template <class H>
void launch_state_in32(int nx, int ny, int pitch, const H *phi, const H *psi, float *x, float *v, cudaStream_t st)
{
    if (sizeof(H) == 4 && rows_v4(ny, phi, psi)) {
        dim3 grd((pitch / 4 + 255) / 256, nx);
        k_state_in32_v4<<<grd, 256, 0, st>>>(nx, ny, pitch, (const float4 *)phi, (const float4 *)psi, x, v);
        return;
    }
    dim3 grd((pitch + 255) / 256, nx);
    k_state_in32<H><<<grd, 256, 0, st>>>(nx, ny, pitch, phi, psi, x, v);
}
template <class T, class H>
void launch_state_out(int nx, int ny, int pitch, const T *x0, const T *y0, const T *x1, const T *y1, const int *sel, H *phi,
                      H *psi, cudaStream_t st)
{
    const long long n = (long long)nx * ny, per = 256 * (16 / sizeof(H));
    const dim3 grd((unsigned)((n + 128 / sizeof(H) + per - 1) / per), 2);
    k_state_out<T, H><<<grd, 256, 0, st>>>(ny, pitch, n, x0, y0, x1, y1, sel, phi, psi);
}
template <class T, class H>
void launch_state_stage(int nx, int ny, int pitch, const T *x0, const T *y0, const T *x1, const T *y1, const int *sel, H *phi,
                        H *psi, cudaStream_t st)
{
    const long long n = (long long)nx * ny, per = 256 * (16 / sizeof(H));
    k_state_stage<T, H><<<(unsigned)((n + per - 1) / per), 256, 0, st>>>(ny, pitch, n, x0, y0, x1, y1, sel, phi, psi);
}
#define WG_STATE_STAGE(T, H) \
    template void launch_state_stage<T, H>(int, int, int, const T *, const T *, const T *, const T *, const int *, H *, H *, cudaStream_t);
WG_STATE_STAGE(float, float)
WG_STATE_STAGE(float, double)
WG_STATE_STAGE(double, double)
#undef WG_STATE_STAGE
template void launch_state_in32<float>(int, int, int, const float *, const float *, float *, float *, cudaStream_t);
template void launch_state_in32<double>(int, int, int, const double *, const double *, float *, float *, cudaStream_t);
template void launch_state_out<float, float>(int, int, int, const float *, const float *, const float *, const float *, const int *, float *,
                                         float *, cudaStream_t);
template void launch_state_out<float, double>(int, int, int, const float *, const float *, const float *, const float *, const int *, double *,
                                         double *, cudaStream_t);
template void launch_state_out<double, double>(int, int, int, const double *, const double *, const double *, const double *, const int *, double *,
                                         double *, cudaStream_t);

}  // namespace wg
