// wg_step64.cuh — one FP64 update of a strip of the grid by one warp (scenes, batches and the
// drop-in).
//
// The strip is ST_COLS columns wide: lane l holds columns base - 2 + 2l and the one after it,
// and lanes 0 and 31 only lend theirs to their neighbours.  The warp marches down the rows with
// the unpacked integers (wg_soft64.h) of rows i-1 and i in registers, unpacks row i+1, and forms
// the Laplacian and x - y of every cell on the integer pipes; the FP64 pipe does the other 3 (no
// KAPPA, no GAMMA) to 7 operations.  Cells whose operands the integer form refuses (about one
// in 150 of a wave field, next to zero crossings; most cells of an exponentially small tail)
// take the FP64 pipe for all of it, in a branch that a warp skips when it has none.
//
// What bounds it: the FP64 pipe's 1.68 operations a clock and SM for table scenes with GAMMA
// (5 of 10 operations left), the integer pipes beside it otherwise.
#pragma once
#include "wg_cells.cuh"
#include "wg_soft64.h"

namespace wg {

constexpr int ST_COLS = 60;  // columns a warp updates
// Where a strip's data comes from.  EXACT = false: native scenes and batches (bit planes, phi
// and psi, the new level over psi).  EXACT = true: the drop-in (int16 mask, tables, a third
// buffer of which only the reference's cells are written).
struct Strip64 {
    const double *phi, *psi;
    double *out;
    const uint32_t *act, *nz;          // native
    const int16_t *xy;                 // drop-in
    const double *tcc, *tc, *tg;       // tables (tg may be null in native scenes: uniform)
    int has_ghosts, do_source;
};

// Whether FLOOR clamps cell k (0, 1) of the lane's pair: xy != 0.
__device__ __forceinline__ bool floor_bit(const DevParams &p, const Strip64 &a, unsigned ac, int k, int i, int c)
{
    if ((ac >> k) & 1u) return true;
    return a.has_ghosts && c >= 0 && c < p.pitch && ((a.nz[(size_t)i * p.wpitch + (c >> 5)] >> ((c & 31) + k)) & 1u);
}

// A boundary-line cell, reference rules, with the point source.
template <int COEF, bool EXACT>
__device__ __noinline__ void edge64(const DevParams &p, const Strip64 &a, int i, int j, long long time)
{
    const size_t c = (size_t)i * p.pitch + j;
    Field<double> PHI{a.phi, p.pitch}, PSI{a.psi, p.pitch};
    double v;
    bool w, nz;
    if (EXACT) {
        CoefTab<double> CF{a.tcc, a.tc, a.tg, p.pitch, 0.0};
        w = edge_cell<double>(p, time, i, j, PHI, PSI, ActI16{a.xy, p.pitch}, CF, &v);
        nz = a.xy[c] != 0;
    } else {
        ActBits ACT{a.act, p.wpitch};
        if (COEF == WG_COEF_TABLE) {
            CoefTab<double> CF{a.tcc, a.tc, a.tg, p.pitch, p.gam};
            w = edge_cell<double>(p, time, i, j, PHI, PSI, ACT, CF, &v);
        } else {
            CoefMask CF{ACT, p.c2, p.c2b, p.gam, p.gamb, p.courant, p.courantb};
            w = edge_cell<double>(p, time, i, j, PHI, PSI, ACT, CF, &v);
        }
        nz = ActBits{a.nz, p.wpitch}(i, j);
    }
    const bool src = a.do_source && p.src_on && i == p.src_i && j == p.src_j;
    if (!w) {
        if (!(p.floor_clamp && nz) && !src) return;  // not written: native fields keep psi there
        v = a.out[c];
    }
    if (p.floor_clamp && nz) v = floor_clamp(p, v);
    if (src) v = A_(v, point_source(p, time));
    a.out[c] = v;
}

// The edge64_cells(p) boundary-line cells by number: they write their own cells only, and read phi
// and their own psi, so they run beside the strips (at the end of the strips that touch them they
// made those the last to finish: a fifth of the time of a 300x300 grid with absorbing edges).
__host__ __device__ __forceinline__ int edge64_cells(const DevParams &p) { return 2 * p.nx + 2 * (p.ny - 2); }
template <int COEF, bool EXACT>
__device__ __forceinline__ void edge64_cell(const DevParams &p, const Strip64 &a, int q, long long time)
{
    const int nx = p.nx, ny = p.ny;
    int i, j;
    if (q < nx) { i = q; j = 0; }
    else if (q < 2 * nx) { i = q - nx; j = ny - 1; }
    else if (q < 2 * nx + (ny - 2)) { i = 0; j = q - 2 * nx + 1; }
    else { i = nx - 1; j = q - 2 * nx - (ny - 2) + 1; }
    edge64<COEF, EXACT>(p, a, i, j, time);
}

// Rows [r0, r1) of 1..nx-2 of the strip whose first column is `base`.  Z: upd64's flags.  The
// drop-in's terms that are an exact zero (KAPPA = 0; GAMMA = 0 on a row of the strip) are left out
// for cells the integer form takes with a finite y: that changes no bit, since r - (+-0) == r but
// for r = -0, and r is -0 only if x is.
template <int COEF, bool EXACT, int Z>
__device__ __forceinline__ void strip64(const DevParams &p, const Strip64 &a, int base, int r0, int r1, long long time)
{
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, c = base - 2 + 2 * lane;
    const int ny = p.ny;
    const bool two = p.twospeeds, floor = p.floor_clamp;
    const double kappa = p.kappa, c2 = p.c2, c2b = p.c2b, gm = p.gam, gmb = p.gamb;
    constexpr bool CT = EXACT || COEF == WG_COEF_TABLE;
    const bool has_tg = EXACT || (COEF == WG_COEF_TABLE && a.tg);
    // the cells of this lane that updates write: bits 0 and 1, of lanes that do not only lend
    // their columns.  Columns outside the rows are read as the nearest ones: only cells that are
    // not written see them.
    const bool core = lane > 0 && lane < 31;
    const unsigned cols = (core && c >= 1 && c < ny - 1 ? 1u : 0u) | (core && c + 1 >= 1 && c + 1 < ny - 1 ? 2u : 0u);
    const long long P = p.pitch, at = r0 * P + min(max(c, 0), p.pitch - 2);
    const double *pn = a.phi + at + P, *py = a.psi + at, *pc = CT ? a.tcc + at : nullptr, *pg = has_tg ? a.tg + at : nullptr;
    double *po = a.out + at;
    const int mc = min(max(c, 0), p.pitch - 2), msh = mc & 31;
    const uint32_t *pm = EXACT ? reinterpret_cast<const uint32_t *>(a.xy + r0 * P + mc)
                               : a.act + ((long long)r0 * p.wpitch + (mc >> 5));
    const long long mstep = EXACT ? P / 2 : p.wpitch;
    const auto ld2 = [](const double *f) { return *reinterpret_cast<const double2 *>(f); };

    double2 s = ld2(pn - 2 * P), x = ld2(pn - P);
    S64 S[2] = {s64_unpack(s.x), s64_unpack(s.y)}, X[2] = {s64_unpack(x.x), s64_unpack(x.y)};
    double2 nn = ld2(pn), yn = ld2(py), cn = make_double2(c2, c2), gn = make_double2(gm, gm);
    if (CT) cn = ld2(pc);
    if (has_tg) gn = ld2(pg);
    unsigned mn = *pm;
#pragma unroll 1
    for (int i = r0; i < r1; i++) {
        const double2 n = nn, y = yn;
        double2 cc = cn, g = gn;
        const unsigned m = mn;
        if (i + 1 < r1) {  // the next row's loads
            pn += P;
            py += P;
            pm += mstep;
            nn = ld2(pn);
            yn = ld2(py);
            if (CT) {
                pc += P;
                cn = ld2(pc);
            }
            if (has_tg) {
                pg += P;
                gn = ld2(pg);
            }
            mn = *pm;
        }
        unsigned ac, up;  // xy != 0, and the cells this update writes
        if (EXACT) {
            const int m0 = (int16_t)(m & 0xFFFFu), m1 = (int16_t)(m >> 16);
            ac = (m0 != 0 ? 1u : 0u) | (m1 != 0 ? 2u : 0u);
            up = (two ? 3u : (m0 > 0 ? 1u : 0u) | (m1 > 0 ? 2u : 0u)) & cols;
        } else {
            ac = (m >> msh) & 3u;
            up = (two ? 3u : ac) & cols;
            if (COEF == WG_COEF_MASK) {
                cc = make_double2(ac & 1u ? c2 : c2b, ac & 2u ? c2 : c2b);
                if (!(Z & Z_GAMMA)) g = make_double2(ac & 1u ? gm : gmb, ac & 2u ? gm : gmb);
            }
        }
        const S64 N[2] = {s64_unpack(n.x), s64_unpack(n.y)};
        if (__any_sync(FULL, up != 0u)) {
            S64 W, E;
            W.m = __shfl_up_sync(FULL, X[1].m, 1);
            W.e = __shfl_up_sync(FULL, X[1].e, 1);
            W.z = __shfl_up_sync(FULL, X[1].z, 1);
            E.m = __shfl_down_sync(FULL, X[0].m, 1);
            E.e = __shfl_down_sync(FULL, X[0].e, 1);
            E.z = __shfl_down_sync(FULL, X[0].z, 1);
            bool ok0, ok1;
            const double d0 = s64_laplacian(N[0], S[0], X[1], W, X[0], ok0);
            const double d1 = s64_laplacian(N[1], S[1], E, X[0], X[1], ok1);
            double v0 = A_(P2_(x.x, y.x), M_(cc.x, d0)), v1 = A_(P2_(x.y, y.y), M_(cc.y, d1));
            if (!(Z & Z_KAPPA)) {
                v0 = S_(v0, M_(kappa, x.x));
                v1 = S_(v1, M_(kappa, x.y));
            }
            // the GAMMA term: not in the kernel, or (drop-in) zero for every cell of the row
            const bool gam = EXACT ? __any_sync(FULL, ((up & 1u) && g.x != 0.0) || ((up & 2u) && g.y != 0.0)) : !(Z & Z_GAMMA);
            if (gam) {
                bool k0, k1;
                v0 = S_(v0, M_(g.x, s64_sub(X[0], s64_unpack(y.x), k0)));
                v1 = S_(v1, M_(g.y, s64_sub(X[1], s64_unpack(y.y), k1)));
                ok0 = ok0 && k0;
                ok1 = ok1 && k1;
            }
            if (EXACT && (!gam || (Z & Z_KAPPA))) {  // a zero term of an infinite value is a NaN
                ok0 = ok0 && (__double2hiint(y.x) & 0x7FF00000) != 0x7FF00000;
                ok1 = ok1 && (__double2hiint(y.y) & 0x7FF00000) != 0x7FF00000;
            }
            const bool f0 = (up & 1u) && !ok0, f1 = (up & 2u) && !ok1;
            if (__any_sync(FULL, f0)) {
                const double h = upd64<EXACT ? 0 : Z>(x.x, y.x, cc.x, L4_(A_(A_(A_(n.x, s.x), x.y), __shfl_up_sync(FULL, x.y, 1)), x.x), kappa, g.x);
                v0 = f0 ? h : v0;
            }
            if (__any_sync(FULL, f1)) {
                const double h = upd64<EXACT ? 0 : Z>(x.y, y.y, cc.y, L4_(A_(A_(A_(n.y, s.y), __shfl_down_sync(FULL, x.x, 1)), x.x), x.y), kappa, g.y);
                v1 = f1 ? h : v1;
            }
            if (floor) {
                if (floor_bit(p, a, ac, 0, i, c)) v0 = floor_clamp(p, v0);
                if (floor_bit(p, a, ac, 1, i, c)) v1 = floor_clamp(p, v1);
            }
            if (up == 3u) {
                *reinterpret_cast<double2 *>(po) = make_double2(v0, v1);
            } else {
                if (up & 1u) po[0] = v0;
                if (up & 2u) po[1] = v1;
            }
        }
        // FLOOR on cells the update does not write: the drop-in's, and a native scene's ghosts
        if (floor && (EXACT || a.has_ghosts)) {
            if ((cols & ~up & 1u) && floor_bit(p, a, ac, 0, i, c)) po[0] = floor_clamp(p, po[0]);
            if ((cols & ~up & 2u) && floor_bit(p, a, ac, 1, i, c)) po[1] = floor_clamp(p, po[1]);
        }
        po += P;
        s = x;
        x = n;
        S[0] = X[0];
        S[1] = X[1];
        X[0] = N[0];
        X[1] = N[1];
    }
    // the point source in the interior, on the finished value
    if (a.do_source && p.src_on && p.src_i >= r0 && p.src_i < r1 && p.src_j >= base && p.src_j < base + ST_COLS &&
        p.src_j > 0 && p.src_j < p.ny - 1) {
        __syncwarp();
        if (lane == 0) {
            double *o = a.out + p.src_i * P + p.src_j;
            *o = A_(*o, point_source(p, time));
        }
    }
}

}  // namespace wg
