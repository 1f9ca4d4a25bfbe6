// wg_tb.cu — temporal blocking of the FP32 leapfrog stepper, and its autotuner.
//
// k_step_tb<COEF>: one CTA owns an extended tile of L rows (i) x W columns (j, W =
// blockDim.x = 128 or 256; L = 16..64), i.e. a core of (L-2K) x (W-2K) cells plus a
// halo of K.  The tile's phi (two levels, alternating) and velocity sit in shared
// memory; K leapfrog updates run on the shrinking region [s, L-s) x [s, W-s) (the new
// phi goes to the other phi level, the velocity is updated in place at the cell itself,
// so a sub-step has no hazards), each thread marching down its column with the i+-1
// neighbours in a register window.  Then the core of phi and the velocity is stored.
// HBM traffic per K updates: one read of phi, the velocity (and the tcc table) over the
// extended tile and one write of both over the core.
//
// The per-cell rules are the reference's (wave_billiard.c:361-590) for the boundary
// conditions whose stencils stay inside the tile: the mirror "Dirichlet" box edges,
// absorbing edges, OSCILLATE_LEFT / OSCILLATE_TOPBOT, FLOOR and the point source.
// Periodic grids take skewed passes in a ghost layout (k_step_wrap); VPER_HABS boundaries
// (which read the opposite side of the grid) and Neumann gathers use the single-step kernel.
#include <algorithm>
#include <type_traits>
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>
#include "wg_scene.h"
#include "wg_batch.h"
#include "wg_tma.cuh"

namespace wg {


constexpr int TB_AW = 12;  // mask words loaded per tile row (covers 256 + 3*32 columns)

struct TbArgs {
    const float *phi, *psi;   // phi(t) and the velocity phi(t) - phi(t-1)
    float *phi_out, *psi_out; // the same after the pass (distinct buffers)
    const uint32_t *act;      // active plane
    const float *tcc, *tc;    // tables (WG_COEF_TABLE)
    float c2, c2b, gam, gamb, kappa, ks, kt, gs, gt, vmax, courant, courantb;
    long long t0;             // step counter before the pass
    const float *osc;         // oscillating_bc values of the pass, [K][ny]
    const double *src;        // point-source increments of the pass, [K]
    int *err;                 // set to 1 when a bounded wait gives up
};

// FP32 phi and velocity of one boundary-line or point-source cell after update t, with
// the reference rules for non-wrapping boundaries (wave_billiard.c:393-590): the mirror
// "Dirichlet" edge and OSCILLATE_TOPBOT rows are the bulk update with the missing
// neighbours replaced by the cell itself, absorbing edges use their inward neighbour,
// oscillating cells take the precomputed oscillating_bc value; keep32 where the
// reference writes nothing.
template <int COEF>
__device__ __forceinline__ XV tb_general(const DevParams &p, const TbArgs &a, int gi, int gj, int s, float x,
                                         float v, float nip, float nim, float njp, float njm, float cc, int act)
{
    const float ccv = (COEF == WG_COEF_TABLE) ? cc : (act ? a.c2 : a.c2b);
    const float g = (COEF == WG_COEF_TABLE) ? a.gam : (act ? a.gam : a.gamb);
    const float tcv = (COEF == WG_COEF_TABLE) ? (a.tc ? a.tc[(size_t)gi * p.pitch + gj] : 0.f)
                                              : (act ? a.courant : a.courantb);
    const Edge32K k{a.kappa, a.ks, a.kt, a.gs, a.gt, a.vmax};
    XV r = edge32<true>(p, gi, gj, x, v, nip, nim, njp, njm, ccv, tcv, g, act != 0, k,
                        [&] { return a.osc[(size_t)(s - 1) * p.ny + gj]; });
    if (p.src_on && gi == p.src_i && gj == p.src_j) r = source32(r, a.src[s - 1]);
    return r;
}

// One sub-step down this thread's column for a tile with no boundary-line or source
// cell: rows [r0, r1), the i+-1 neighbours in a register window, shared-memory
// addressing by constant offsets.  P: phi of the previous level; Q: phi of the new
// level; Vs: the velocity, in place.  ACT: the cell's mask bit selects coefficients and
// whether it is written (otherwise every cell is written with its tcc).
template <int COEF, bool ACT>
__device__ __forceinline__ void tb_rows_interior(const DevParams &p, const TbArgs &a, const float *__restrict__ P,
                                                 float *__restrict__ Q, float *__restrict__ Vs,
                                                 const float *__restrict__ Cs, int Bw, int c, int r0, int r1,
                                                 uint64_t actb)
{
    int idx = r0 * Bw + c;
    float up = P[idx - Bw], mid = P[idx];
    uint64_t am = actb >> r0;
    const int n = r1 - r0;
#pragma unroll 4
    for (int q = 0; q < n; q++, idx += Bw) {
        const float dn = P[idx + Bw], e = P[idx + 1], w = P[idx - 1], y = Vs[idx];
        const float delta = ((dn - mid) + (up - mid)) + ((e - mid) + (w - mid));
        XV r;
        if (!ACT) {
            r = upd32(mid, y, Cs[idx], delta, a.kappa, a.gam);
        } else {
            const bool act = am & 1u;
            am >>= 1;
            const float ccv = (COEF == WG_COEF_TABLE) ? Cs[idx] : (act ? a.c2 : a.c2b);
            const float g = (COEF == WG_COEF_TABLE) ? a.gam : (act ? a.gam : a.gamb);
            r = keep32(mid, y);
            if (p.twospeeds || act) {
                r = upd32(mid, y, ccv, delta, a.kappa, g);
                if (p.floor_clamp && act) r = clamp32(mid, r, a.vmax);
            }
        }
        Q[idx] = r.x;
        Vs[idx] = r.v;
        up = mid;
        mid = dn;
    }
}

// oscillating_bc(t0 + s, j) for s = 1..n (when OSCILLATE_LEFT) and the point-source
// increment of update t0 + s, rounded to FP32, for the passes of one step() call.
__global__ void k_boundary_values(const __grid_constant__ DevParams p, long long t0, int n, float *osc, double *src)
{
    pdl_wait();  // launched by launch_pdl: the previous pass, which read these arrays, has completed
    pdl_trigger();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (p.osc_left && idx < n * p.ny) {
        const int s = idx / p.ny, j = idx % p.ny;
        osc[idx] = (float)osc_bc(p, (int)(t0 + s + 1), j);
    }
    if (p.src_on && idx < n) src[idx] = point_source(p, t0 + idx + 1);
}

// Shared-memory layout of one tile: F0, F1 (phi, alternating levels), Vs (velocity),
// Cs (tcc, table mode), Aw (the active-plane words covering the tile), one mbarrier.
// F0, Vs, Cs and Aw are loaded; F1 is written before it is read.
struct TbLayout {
    int f0, f1, vs, cs, aw, bar, bytes, tma_bytes;
};
__host__ __device__ inline TbLayout tb_layout(int coef, int L, int Bw)
{
    TbLayout t;
    const int fb = L * Bw * 4;
    t.f0 = 0;
    t.f1 = fb;
    t.vs = 2 * fb;
    t.cs = 3 * fb;
    t.aw = (coef == WG_COEF_TABLE ? 4 : 3) * fb;
    t.bar = t.aw + ((L * TB_AW * 4 + 15) / 16) * 16;
    t.bytes = t.bar + 16;
    t.tma_bytes = (coef == WG_COEF_TABLE ? 3 : 2) * fb + L * TB_AW * 4;
    return t;
}

template <int COEF>
__global__ void __launch_bounds__(256) k_step_tb(const __grid_constant__ DevParams p, const __grid_constant__ TbArgs a,
                                                 const __grid_constant__ CUtensorMap m_phi,
                                                 const __grid_constant__ CUtensorMap m_psi,
                                                 const __grid_constant__ CUtensorMap m_tcc,
                                                 const __grid_constant__ CUtensorMap m_act, int K, int Kh, int L)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    const int Bw = blockDim.x;
    const TbLayout lay = tb_layout(COEF, L, Bw);
    float *F0 = (float *)(smem + lay.f0), *F1 = (float *)(smem + lay.f1), *Vs = (float *)(smem + lay.vs),
          *Cs = (float *)(smem + lay.cs);
    const uint32_t *Aw = (const uint32_t *)(smem + lay.aw);
    uint64_t *bar = (uint64_t *)(smem + lay.bar);
    const int c = threadIdx.x;
    const int core_w = Bw - 2 * Kh, core_h = L - 2 * K;
    const int x0 = blockIdx.x * core_w - Kh;   // first column of the tile (a multiple of 4)
    const int gi0 = blockIdx.y * core_h - K;   // first row of the tile
    const int w0 = (x0 >> 5) & ~3;             // first mask word of the tile (a multiple of 4)
    const int gj = x0 + c;
    const bool col_ok = gj >= 0 && gj < p.ny;
    const bool col_special = (gj == 0 || gj == p.ny - 1);

    // TMA destinations must be 128-byte aligned; refuse (flag) rather than issue otherwise
    if (smem_u32(smem) & 127u) {
        if (c == 0) atomicExch(a.err, 2);
        return;
    }
    // TMA: the extended tile of phi, the velocity (tcc) and the mask words, zero outside the grid
    if (c == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (c == 0) {
        mbar_arrive_expect_tx(bar, (unsigned)lay.tma_bytes);
        tma_load_2d(F0, &m_phi, x0, gi0, bar);
        tma_load_2d(Vs, &m_psi, x0, gi0, bar);
        if (COEF == WG_COEF_TABLE) tma_load_2d(Cs, &m_tcc, x0, gi0, bar);
        tma_load_2d((void *)Aw, &m_act, w0, gi0, bar);
    }
    const bool ok = mbar_wait_bounded(bar, 0, 1u << 24);
    if (__syncthreads_or(!ok)) {
        // the copies did not land in time: flag it, let them drain (bounded), leave
        if (c == 0) atomicExch(a.err, 1);
        mbar_wait_bounded(bar, 0, 1u << 24);
        return;
    }

    uint64_t actb = 0;
    if (col_ok) {
        const int wi = (gj >> 5) - w0;
#pragma unroll 8
        for (int r = 0; r < L; r++) actb |= (uint64_t)((Aw[r * TB_AW + wi] >> (gj & 31)) & 1u) << r;
    }

    // a tile with no boundary line and no source cell runs the lean interior loop
    const bool interior_tile = gi0 >= 1 && gi0 + L <= p.nx - 1 && x0 >= 1 && x0 + Bw <= p.ny - 1 &&
                               !(p.src_on && p.src_i >= gi0 && p.src_i < gi0 + L && p.src_j >= x0 && p.src_j < x0 + Bw);
    const bool no_act = COEF == WG_COEF_TABLE && p.twospeeds && !p.floor_clamp;

    for (int s = 1; s <= K; s++) {
        const float *P = (s & 1) ? F0 : F1;  // phi of level t+s-1
        float *Q = (s & 1) ? F1 : F0;        // phi of level t+s-2, becomes level t+s
        const bool in_region = c >= Kh - K + s && c < Bw - Kh + K - s;
        if (interior_tile) {
            if (in_region) {
                if (no_act) tb_rows_interior<COEF, false>(p, a, P, Q, Vs, Cs, Bw, c, s, L - s, actb);
                else tb_rows_interior<COEF, true>(p, a, P, Q, Vs, Cs, Bw, c, s, L - s, actb);
            }
        } else if (col_ok && in_region && !col_special) {
            // a boundary tile, interior column: lean segments between the special rows
            // (gi = 0, gi = nx-1, the source row), the special rows one at a time
            const int lo = max(s, -gi0), hi = min(L - s, p.nx - gi0);
            const int ra = -gi0, rb = p.nx - 1 - gi0;
            const int rs = (p.src_on && gj == p.src_j) ? p.src_i - gi0 : -1;
            int r = lo;
            while (r < hi) {
                if (r == ra || r == rb || r == rs) {
                    const int gi = gi0 + r, o = r * Bw + c;
                    const float cc = (COEF == WG_COEF_TABLE) ? Cs[o] : 0.f;
                    const XV res = tb_general<COEF>(p, a, gi, gj, s, P[o], Vs[o], P[o + Bw], P[o - Bw], P[o + 1],
                                                    P[o - 1], cc, (int)((actb >> r) & 1u));
                    Q[o] = res.x;
                    Vs[o] = res.v;
                    r++;
                } else {
                    int nxt = hi;
                    if (ra > r && ra < nxt) nxt = ra;
                    if (rb > r && rb < nxt) nxt = rb;
                    if (rs > r && rs < nxt) nxt = rs;
                    if (no_act) tb_rows_interior<COEF, false>(p, a, P, Q, Vs, Cs, Bw, c, r, nxt, actb);
                    else tb_rows_interior<COEF, true>(p, a, P, Q, Vs, Cs, Bw, c, r, nxt, actb);
                    r = nxt;
                }
            }
        } else if (col_ok && in_region) {
            int r = s;
            float up = P[(r - 1) * Bw + c], mid = P[r * Bw + c];
#pragma unroll 4
            for (; r < L - s; r++) {
                const float dn = P[(r + 1) * Bw + c];
                const int gi = gi0 + r;
                if (gi >= 0 && gi < p.nx) {
                    const int o = r * Bw + c;
                    const float e = P[o + 1], w = P[o - 1];
                    const float y = Vs[o];
                    const float cc = (COEF == WG_COEF_TABLE) ? Cs[o] : 0.f;
                    const int act = (int)((actb >> r) & 1u);
                    XV res = keep32(mid, y);
                    if (col_special || gi == 0 || gi == p.nx - 1 || (p.src_on && gi == p.src_i && gj == p.src_j)) {
                        res = tb_general<COEF>(p, a, gi, gj, s, mid, y, dn, up, e, w, cc, act);
                    } else if (p.twospeeds || act) {
                        const float ccv = (COEF == WG_COEF_TABLE) ? cc : (act ? a.c2 : a.c2b);
                        const float g = (COEF == WG_COEF_TABLE) ? a.gam : (act ? a.gam : a.gamb);
                        res = upd32(mid, y, ccv, ((dn - mid) + (up - mid)) + ((e - mid) + (w - mid)), a.kappa, g);
                        if (p.floor_clamp && act) res = clamp32(mid, res, a.vmax);
                    }
                    Q[o] = res.x;
                    Vs[o] = res.v;
                }
                up = mid;
                mid = dn;
            }
        }
        __syncthreads();
    }

    // store the core: phi of level t+K and the velocity
    if (col_ok && c >= Kh && c < Bw - Kh) {
        const float *newest = (K & 1) ? F1 : F0;
#pragma unroll 4
        for (int r = K; r < L - K; r++) {
            const int gi = gi0 + r;
            if (gi < p.nx) {
                const size_t o = (size_t)gi * p.pitch + gj;
                a.phi_out[o] = newest[r * Bw + c];
                a.psi_out[o] = Vs[r * Bw + c];
            }
        }
    }
}

// Oscillating values and source increments of a batch's passes, computed at their update
// time (single grids read them from the per-call arrays; both are the same double values,
// rounded the same way).
// Out of line: they are rare, and inlined copies per level would crowd the instruction cache.
__device__ __noinline__ float osc_inl(const DevParams &p, long long t, int j) { return (float)osc_bc(p, (int)t, j); }
__device__ __noinline__ double src_inl(const DevParams &p, long long t) { return point_source(p, t); }

// The update a pass compiles: general (two speeds, FLOOR and the mask tested at run time),
// every cell written with KAPPA = 0 (two speeds, no FLOOR), or masked cells with KAPPA = 0
// (one speed, no FLOOR).  A zero KAPPA leaves out an exact zero: at most the sign of a zero
// result changes.
enum { PL_GEN = 0, PL_ALL = 1, PL_MASKED = 2 };
__host__ __device__ inline int skew_form(int twospeeds, int floor_clamp, double kappa)
{
    return (floor_clamp || kappa != 0.0) ? PL_GEN : (twospeeds ? PL_ALL : PL_MASKED);
}

// Paired FP32 arithmetic: the two-wide add, sub and fma of this GPU (.f32x2) round each
// element exactly as the scalar instruction does, so two cells computed together get the
// same bits as two computed one at a time, for one instruction issued instead of two.  A
// pair is held as one 64-bit value from the load to the store.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float x, float y)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float lo2(f2 a)
{
    float x;
    asm("mov.b64 {%0, _}, %1;" : "=f"(x) : "l"(a));
    return x;
}
__device__ __forceinline__ float hi2(f2 a)
{
    float x;
    asm("mov.b64 {_, %0}, %1;" : "=f"(x) : "l"(a));
    return x;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b)
{
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// cell k (0..3) of a lane's four cells held as the pairs (0, 1) and (2, 3)
template <int k>
__device__ __forceinline__ float el(const f2 (&q)[2])
{
    return k & 1 ? hi2(q[k >> 1]) : lo2(q[k >> 1]);
}
template <int k>
__device__ __forceinline__ void set_el(f2 (&q)[2], float v)
{
    q[k >> 1] = k & 1 ? pk(lo2(q[k >> 1]), v) : pk(v, hi2(q[k >> 1]));
}

// The coefficients of a pass as pairs, kept in registers: -GAMMA, -KAPPA, COURANT^2.
struct SkewK {
    f2 ng, nk, c2;
};

// The update of a pass for the two cells of a pair, with the Laplacian given in
// differences.  Vertical: vert = dn - dp with dn = n - x and dp = x - sv, which
// equals (n - x) + (sv - x) exactly (round to nearest is symmetric, so sv - x == -(x - sv));
// dp is the previous row's dn, so each row's difference is formed once per column.
// Horizontal: hh = he - hw with he = e - x and hw = x - w, (e - x) + (w - x) == he - hw
// exactly, and a lane's four cells share the five differences of their row.  x, y, vert,
// cc: the cells' phi, velocity, vertical part and tcc.  New phi in xo, new velocity in vo:
// upd32_k0 (PL_ALL), the same or the unwritten cell's rule by the mask (PL_MASKED), or
// updkeep32 and clamp32 (PL_GEN), element by element.
template <int COEF, int PL>
__device__ __forceinline__ void skew_inner2(const DevParams &p, const TbArgs &a, const SkewK &k, f2 x, f2 y, f2 vert, f2 hh,
                                            f2 cc, bool act0, bool act1, f2 &xo, f2 &vo)
{
    f2 ccv = COEF == WG_COEF_TABLE ? cc : k.c2, ng = k.ng;
    if (COEF == WG_COEF_MASK && PL != PL_MASKED) {  // masked: the cells it writes are inside
        ccv = pk(act0 ? a.c2 : a.c2b, act1 ? a.c2 : a.c2b);
        ng = pk(act0 ? -a.gam : -a.gamb, act1 ? -a.gam : -a.gamb);
    }
    const f2 lap = add2(vert, hh);
    f2 vn = PL == PL_GEN ? fma2(ccv, lap, fma2(k.nk, x, fma2(ng, y, y)))  // vel32
                         : fma2(ccv, lap, fma2(ng, y, y));
    if (PL != PL_ALL)
        vn = pk((PL == PL_GEN && p.twospeeds) || act0 ? lo2(vn) : -lo2(y), (PL == PL_GEN && p.twospeeds) || act1 ? hi2(vn) : -hi2(y));
    xo = add2(x, vn);
    vo = vn;
    if (PL == PL_GEN && p.floor_clamp) {
        XV r0{lo2(xo), lo2(vo)}, r1{hi2(xo), hi2(vo)};
        if (act0) r0 = clamp32(lo2(x), r0, a.vmax);
        if (act1) r1 = clamp32(hi2(x), r1, a.vmax);
        xo = pk(r0.x, r1.x);
        vo = pk(r0.v, r1.v);
    }
}

// ---------------------------------------------------------------------------
// Time-skewed streaming in a pipeline of warps (k_step_skew, k_batch_skew).  A team of P
// warps (one CTA) owns a tile of 128 columns (four adjacent columns j per lane, held as two
// float2 pairs; a column halo of H = K rounded up to 4) and a chunk of rows, and walks down
// it once, two rows a step.  Warp w computes levels 2w+1 and 2w+2: it takes the rows of
// level 2w from the input ring (w = 0, filled by cp.async) or from the warp before it
// (a double-buffered pair of rows in shared memory), keeps a window of two phi rows, one
// velocity row and one vertical difference per level in registers, and hands the rows of
// level 2w+2 on, or stores them (the last warp; one level only when K is odd).  One CTA
// barrier a step.  At step s warp w takes rows m0 + 2s - 4w and the next one.
//
// Why teams: with all K levels in one warp the loop body was K levels long (126 registers at
// K = 4, spills at 6, instruction-cache misses when unrolled) and 16 warps per SM left row
// chunks of 28 rows with a fill of 2K+1.  Here a warp holds two levels (80-96 registers, 20
// warps per SM), the body is the same for every depth, a pass reads and writes each cell once
// for up to 6 updates, and a tile costs less fill.  3840x2160, two-medium table, absorbing:
// 881 Gcell/s at K = 4 before, 1010 at K = 4 (5.1 TB/s of DRAM) and 1170 at K = 6 now; 640x480
// and smaller grids, where a pass is a chain of dependent steps, 2.3 times as fast.
// What bounds it: at K = 4 DRAM, at K = 6 the latency of a step (half the issue slots are
// used: 210 warp instructions for 4 rows of 128 cells and level, 84 of them arithmetic).
//
// Tiles that reach an edge row or column of the grid or hold the point source (EDGE) take
// the edge rules after the common update; the others have no test for them.
// ---------------------------------------------------------------------------
// Asynchronous global->shared copies of one lane's 16 (or 4) bytes to a 32-bit shared-window
// address.
__device__ __forceinline__ void cp_async16s(unsigned d, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4s(unsigned d, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Shared memory of one team, in floats: the input ring (SK_IN steps of two rows of phi and
// velocity), the hand-over pairs between warps, and rings that every warp reads at its own
// lag: tcc, one active word per lane and row, tc of the lane's edge column.
constexpr int SK_IN = 3;  // 2 and 4 measured slower: fewer steps in flight, or fewer teams per SM
template <int COEF, int PL, int P>
struct SkewShm {
    static constexpr bool NEED_ACT = !(PL == PL_ALL && COEF == WG_COEF_TABLE);  // else the update ignores the mask
    static constexpr int NT = SK_IN + 2 * P - 1;  // steps a lagged ring holds: prefetched ones, and back to warp P-1's
    static constexpr int IN = 0, HAND = IN + SK_IN * 512, TCC = HAND + (P - 1) * 1024,
                         ACT = TCC + (COEF == WG_COEF_TABLE ? NT * 256 : 0), TCE = ACT + (NEED_ACT ? NT * 64 : 0),
                         SIZE = TCE + (COEF == WG_COEF_TABLE ? NT * 64 : 0);
    // single grids with OSCILLATE_LEFT: row 0's values at the tile's columns, per level
    static constexpr int OSC = SIZE;
    static constexpr size_t BYTES = SIZE * sizeof(float), OSC_BYTES = 2 * P * 128 * sizeof(float);
};

// What an edge strip knows.  EDGE of a step: 0 inner; 1 the tile holds column 0 or ny-1 (mirror
// or absorbing); 2 any rule (rows 0 and nx-1, OSCILLATE_LEFT and _TOPBOT, the point source).
struct SkewEdge {
    int m0, m1, m2, m3, m4;  // masks of the horizontal differences: 0 where a mirror edge makes one zero
    int cr;                  // column ny-1's place in its lane's group (the same for every lane)
    bool left, right;        // the tile holds column 0, column ny-1 (warp-uniform)
    bool my_left, my_right;  // this lane holds it
    bool src, absorb;        // the lane holds the point source's column; B_COND is absorbing
    const float *osc;        // OSCILLATE_LEFT's values at the lane's columns, 128 floats a level
};

// Cell k's absorbing rule along j on the lanes of `mine`; d = x - (its inward neighbour).
template <int COEF, int PL, int k>
__device__ __forceinline__ void skew_absorb(const DevParams &p, const TbArgs &a, const f2 (&c)[2], const f2 (&cv)[2], float d,
                                            float tcv, unsigned act, bool mine, f2 (&ox)[2], f2 (&ov)[2])
{
    const float x = el<k>(c), y = el<k>(cv);
    const bool ac = (act >> k) & 1u;
    if (COEF == WG_COEF_MASK) tcv = (PL == PL_MASKED || ac) ? a.courant : a.courantb;
    float vn = -fmaf(a.gt, y, fmaf(a.kt, x, __fmul_rn(tcv, d)));
    if (PL == PL_MASKED && !ac) vn = -y;
    if (PL == PL_GEN && !p.twospeeds && !ac) vn = -y;
    XV n = XV{__fadd_rn(x, vn), vn};
    if (PL == PL_GEN && p.floor_clamp && ac) n = clamp32(x, n, a.vmax);
    set_el<k>(ox, mine ? n.x : el<k>(ox));
    set_el<k>(ov, mine ? n.v : el<k>(ov));
}

// Cell k on rows 0 and nx-1 (absorbing, or the oscillating values of OSCILLATE_LEFT).
template <int COEF, bool INL, int k>
__device__ __forceinline__ void skew_row_edge(const DevParams &p, const TbArgs &a, const SkewEdge &ed, int r, int lv, int gj0,
                                              const f2 (&c)[2], const f2 (&cv)[2], const f2 (&dn)[2], const f2 (&D)[2],
                                              unsigned act, f2 (&ox)[2], f2 (&ov)[2])
{
    const int gj = gj0 + k;
    if (gj < 0 || gj >= p.ny || gj == 0 || gj == p.ny - 1) return;
    const bool ac = (act >> k) & 1u;
    const float x = el<k>(c), y = el<k>(cv);
    XV n;
    if (r == 0 && left_bc(p, gj)) {
        n = set32(x, INL ? osc_inl(p, a.t0 + lv, gj) : ed.osc[(lv - 1) * 128 + k]);
    } else if (ed.absorb && (p.twospeeds || ac)) {
        const float d = r == 0 ? -el<k>(dn) : el<k>(D);
        const float tcv = (COEF == WG_COEF_TABLE) ? (a.tc ? a.tc[(size_t)r * p.pitch + gj] : 0.f)
                                                  : (ac ? a.courant : a.courantb);
        const float vn = -fmaf(a.gs, y, fmaf(a.ks, x, __fmul_rn(tcv, d)));
        n = XV{__fadd_rn(x, vn), vn};
    } else {
        return;
    }
    if (p.floor_clamp && ac) n = clamp32(x, n, a.vmax);
    set_el<k>(ox, n.x);
    set_el<k>(ov, n.v);
}

// Cell k: a corner of OSCILLATE_LEFT, then the point source.
template <bool INL, int k>
__device__ __forceinline__ void skew_corner_src(const DevParams &p, const TbArgs &a, const SkewEdge &ed, int lv, int gj0,
                                                const f2 (&c)[2],
                                                unsigned act, bool corner, bool src, f2 (&ox)[2], f2 (&ov)[2])
{
    const int gj = gj0 + k;
    XV n = XV{el<k>(ox), el<k>(ov)};
    if (corner && gj < p.ny && (gj == 0 || (p.corner2_on && gj == p.nx - 1))) {
        n = set32(el<k>(c), INL ? osc_inl(p, a.t0 + lv, gj) : ed.osc[(lv - 1) * 128 + k]);
        if (p.floor_clamp && ((act >> k) & 1u)) n = clamp32(el<k>(c), n, a.vmax);
    }
    if (src && gj == p.src_j) n = source32(n, INL ? src_inl(p, a.t0 + lv) : a.src[lv - 1]);
    set_el<k>(ox, n.x);
    set_el<k>(ov, n.v);
}

// One level's new row r (phi and velocity) from level lv-1: c, cv its phi and velocity at row
// r, nn its phi at row r+1, D its vertical difference x(r) - x(r-1), replaced by the next; T
// the cells' tcc, tcv the tc of the lane's edge column (table scenes), act the mask bits.
template <int COEF, int PL, int EDGE, bool INL>
__device__ __forceinline__ void skew_level(const DevParams &p, const TbArgs &a, const SkewK &kk, const SkewEdge &ed, int r,
                                           int lv, int gj0, const f2 (&c)[2], const f2 (&cv)[2], const f2 (&nn)[2], f2 (&D)[2],
                                           const f2 (&T)[2], float tcv, unsigned act, f2 (&ox)[2], f2 (&ov)[2])
{
    f2 dn[2] = {sub2(nn[0], c[0]), sub2(nn[1], c[1])};
    if (EDGE == 2) {  // rows 0 and nx-1 mirror: the neighbour outside is the cell itself
        if (r == p.nx - 1) dn[0] = dn[1] = 0;
        if (r == 0) D[0] = D[1] = 0;
    }
    const f2 vt[2] = {sub2(dn[0], D[0]), sub2(dn[1], D[1])};
    const float c0 = lo2(c[0]), c1 = hi2(c[0]), c2 = lo2(c[1]), c3 = hi2(c[1]);
    const float w0 = __shfl_up_sync(0xffffffffu, c3, 1);
    const float e3 = __shfl_down_sync(0xffffffffu, c0, 1);
    float hd[5] = {c0 - w0, c1 - c0, c2 - c1, c3 - c2, e3 - c3};
    if (EDGE) {
        hd[0] = __int_as_float(__float_as_int(hd[0]) & ed.m0);
        hd[1] = __int_as_float(__float_as_int(hd[1]) & ed.m1);
        hd[2] = __int_as_float(__float_as_int(hd[2]) & ed.m2);
        hd[3] = __int_as_float(__float_as_int(hd[3]) & ed.m3);
        hd[4] = __int_as_float(__float_as_int(hd[4]) & ed.m4);
    }
    f2 hh[2] = {pk(hd[1] - hd[0], hd[2] - hd[1]), pk(hd[3] - hd[2], hd[4] - hd[3])};
    // OSCILLATE_TOPBOT: the edge column takes the vertical part only
    const bool topbot = EDGE == 2 && p.osc_topbot && r > 0 && r < p.nx - 1 && r < p.tb_ilim;
    if (EDGE == 2 && topbot) {
        if (ed.my_left || (ed.my_right && ed.cr == 0)) set_el<0>(hh, 0.f);
        if (ed.my_right && ed.cr == 1) set_el<1>(hh, 0.f);
        if (ed.my_right && ed.cr == 2) set_el<2>(hh, 0.f);
        if (ed.my_right && ed.cr == 3) set_el<3>(hh, 0.f);
    }
#pragma unroll
    for (int h = 0; h < 2; h++)
        skew_inner2<COEF, PL>(p, a, kk, c[h], cv[h], vt[h], hh[h], T[h], (act >> (2 * h)) & 1u, (act >> (2 * h + 1)) & 1u,
                              ox[h], ov[h]);
    if (EDGE == 2 && (r == 0 || r == p.nx - 1) && (ed.absorb || (p.osc_left && r == 0))) {
        skew_row_edge<COEF, INL, 0>(p, a, ed, r, lv, gj0, c, cv, dn, D, act, ox, ov);
        skew_row_edge<COEF, INL, 1>(p, a, ed, r, lv, gj0, c, cv, dn, D, act, ox, ov);
        skew_row_edge<COEF, INL, 2>(p, a, ed, r, lv, gj0, c, cv, dn, D, act, ox, ov);
        skew_row_edge<COEF, INL, 3>(p, a, ed, r, lv, gj0, c, cv, dn, D, act, ox, ov);
    }
    if (EDGE && ed.absorb && !topbot) {  // warp-uniform
        // the bottom and top columns, absorbing
        if (ed.left) skew_absorb<COEF, PL, 0>(p, a, c, cv, -hd[1], tcv, act, ed.my_left, ox, ov);
        if (ed.right) {
            switch (ed.cr) {
            case 0: skew_absorb<COEF, PL, 0>(p, a, c, cv, hd[0], tcv, act, ed.my_right, ox, ov); break;
            case 1: skew_absorb<COEF, PL, 1>(p, a, c, cv, hd[1], tcv, act, ed.my_right, ox, ov); break;
            case 2: skew_absorb<COEF, PL, 2>(p, a, c, cv, hd[2], tcv, act, ed.my_right, ox, ov); break;
            default: skew_absorb<COEF, PL, 3>(p, a, c, cv, hd[3], tcv, act, ed.my_right, ox, ov); break;
            }
        }
    }
    if (EDGE == 2) {
        const bool corner = r == 0 && p.osc_left && !p.beam, src = ed.src && r == p.src_i;
        if (corner || src) {
            skew_corner_src<INL, 0>(p, a, ed, lv, gj0, c, act, corner, src, ox, ov);
            skew_corner_src<INL, 1>(p, a, ed, lv, gj0, c, act, corner, src, ox, ov);
            skew_corner_src<INL, 2>(p, a, ed, lv, gj0, c, act, corner, src, ox, ov);
            skew_corner_src<INL, 3>(p, a, ed, lv, gj0, c, act, corner, src, ox, ov);
        }
    }
    D[0] = dn[0];
    D[1] = dn[1];
}

// The window of one warp: per level, X[u] and V[u] alternate between the row in use and the
// next one (phi, velocity), D is the vertical difference of skew_level.
struct SkewWin {
    f2 XA[2][2], VA[2][2], DA[2], XB[2][2], VB[2][2], DB[2];
};

// One step of warp w: its input rows m and m+1 (at `in`), level 2w+1 at rows m-1 and m, level
// 2w+2 at rows m-2 and m-1 (xo, vo); level 2w+1's rows are then in XB[1], VB[1] and XB[0], VB[0].
template <int COEF, int PL, int EDGE, bool INL>
__device__ __forceinline__ void skew_step(const DevParams &p, const TbArgs &a, const SkewK &kk, const SkewEdge &ed, int m, int w,
                                          int gj0, const float *in, const f2 (&T)[3][2],
                                          const float (&te)[3], const unsigned (&act)[3], SkewWin &q, f2 (&xo)[2][2],
                                          f2 (&vo)[2][2])
{
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const ulonglong2 x4 = *reinterpret_cast<const ulonglong2 *>(in + u * 256);
        const ulonglong2 v4 = *reinterpret_cast<const ulonglong2 *>(in + u * 256 + 128);
        q.XA[u ^ 1][0] = x4.x;
        q.XA[u ^ 1][1] = x4.y;
        q.VA[u ^ 1][0] = v4.x;
        q.VA[u ^ 1][1] = v4.y;
        // level 2w+1's row is the next row of level 2w+2's window
        skew_level<COEF, PL, EDGE, INL>(p, a, kk, ed, m + u - 1, 2 * w + 1, gj0, q.XA[u], q.VA[u], q.XA[u ^ 1], q.DA, T[u + 1],
                                        te[u + 1], act[u + 1], q.XB[u ^ 1], q.VB[u ^ 1]);
        skew_level<COEF, PL, EDGE, INL>(p, a, kk, ed, m + u - 2, 2 * w + 2, gj0, q.XB[u], q.VB[u], q.XB[u ^ 1], q.DB, T[u],
                                        te[u], act[u], xo[u], vo[u]);
    }
}

// The team's barrier (warps wait at different places of the code).
__device__ __forceinline__ void team_sync() { asm volatile("bar.sync 0;\n" ::: "memory"); }

// One team's strip: rows [i_s, i_e), the lane's columns gj0..gj0+3, stored for columns
// [lo, hi) (multiples of 4 but for hi = ny).  Rows [rlo, rhi) and columns [clo, chi) exist (a
// periodic scene of a batch holds its wrapped halo outside the grid, its ghosts); a row
// outside is read as the nearest one and a lane outside reads nothing: no stored cell
// depends on either.  K levels, K = 2P or 2P-1.
template <int COEF, int PL, int P, bool EDGE, bool INL>
__device__ __forceinline__ void skew_strip(const DevParams &p, const TbArgs &a, int K, int i_s, int i_e, int gj0, int lane,
                                           int w, float *shm, int lo, int hi, int rlo, int rhi, int clo, int chi)
{
    using SM = SkewShm<COEF, PL, P>;
    const int m0 = i_s - K, half = (i_e - i_s + 1) >> 1;
    const int s_first = 3 * w, s_last = K + w - 1 + half, nsteps = K + P - 1 + half;
    const bool two = P > 1 ? (w < P - 1 || K == 2 * P) : K == 2;
    const bool last = w == P - 1;
    const bool col_ok = gj0 >= clo && gj0 < chi;
    const bool core = gj0 >= lo && gj0 < hi && gj0 >= 0 && gj0 < p.ny;
    SkewEdge ed = {-1, -1, -1, -1, -1, 0, false, false, false, false, false, false, nullptr};
    if (EDGE) {
        const int cr = p.ny - 1 - gj0;  // column ny-1 within the lane's group when 0..3
        const int t0 = gj0 - 4 * lane;
        ed.left = t0 <= 0;
        ed.right = t0 + 128 >= p.ny;
        ed.my_left = gj0 == 0;
        ed.my_right = cr >= 0 && cr <= 3;
        ed.cr = (p.ny - 1) & 3;
        ed.m0 = ed.my_left ? 0 : -1;
        ed.m1 = cr == 0 ? 0 : -1;
        ed.m2 = cr == 1 ? 0 : -1;
        ed.m3 = cr == 2 ? 0 : -1;
        ed.m4 = cr == 3 ? 0 : -1;
        ed.src = p.src_on && p.src_j >= gj0 && p.src_j < gj0 + 4;
        ed.absorb = p.b_cond == WG_BC_ABSORBING;
    }
    const bool need_tce = EDGE && COEF == WG_COEF_TABLE && ed.absorb;
    float *const my4 = shm + 4 * lane;
    const float *const my1 = shm + lane;
    const unsigned base16 = (unsigned)__cvta_generic_to_shared(my4), base4 = (unsigned)__cvta_generic_to_shared(my1);
    const long long pitch = p.pitch;
    if (EDGE && !INL) {
        // Each warp fetches row 0's values of its two levels ahead.  Read where they are used, their
        // latencies, one after the other in every level, made the first rows' strips last longest
        // (1277x717, 50 updates a call: 4.21 to 3.79 us an update).
        ed.osc = my4 + SM::OSC;
        if (p.osc_left && i_s < K) {
#pragma unroll 1
            for (int lv = 2 * w + 1; lv <= min(2 * w + 2, K); lv++)
                for (int k = 0; k < 4; k++)
                    if (gj0 + k >= 0 && gj0 + k < p.ny)
                        cp_async4s(base16 + 4 * (SM::OSC + (lv - 1) * 128 + k), a.osc + ((size_t)(lv - 1) * p.ny + gj0 + k));
            cp_async_commit();
            if (w > 0) cp_async_wait<0>();  // (warp 0: with its first rows)
        }
    }

    // warp 0: copies of the next two rows (row m_in and the one after it) into input slot si and
    // lagged slot ti (in bytes from the rings' start), while the strip has more rows
    int m_in = m0;
    const int m_end = min(m0 + 2 * (s_last + 1), rhi);
    long long off = m0 * pitch + gj0;
    // the group's mask word: floor division, so that the ghost columns left of column 0 read
    // the row's ghost word (index -1)
    const int aw = (gj0 + 32) / 32 - 1;
    const int tce_c = ed.my_left ? 0 : ed.cr;
    unsigned si = 0, ti = 0;
    auto issue = [&]() {
#pragma unroll
        for (int u = 0; u < 2; u++) {
            if (col_ok && m_in + u < m_end && (!EDGE || m_in + u >= rlo)) {
                cp_async16s(base16 + (4 * SM::IN + 1024 * u) + si, a.phi + off);
                cp_async16s(base16 + (4 * SM::IN + 1024 * u + 512) + si, a.psi + off);
                if (COEF == WG_COEF_TABLE) cp_async16s(base16 + (4 * SM::TCC + 512 * u) + 4 * ti, a.tcc + off);
                if (SM::NEED_ACT)
                    cp_async4s(base4 + (4 * SM::ACT + 128 * u) + ti, a.act + ((long long)(m_in + u) * p.wpitch + aw));
                if (need_tce && (ed.my_left || ed.my_right)) cp_async4s(base4 + (4 * SM::TCE + 128 * u) + ti, a.tc + off + tce_c);
            }
            off += pitch;
        }
        m_in += 2;
        si = si == (SK_IN - 1) * 2048 ? 0 : si + 2048;
        ti = ti == (SM::NT - 1) * 256 ? 0 : ti + 256;
        cp_async_commit();
    };
    // the last warp's row r
    auto store = [&](int r, const f2 (&x)[2], const f2 (&v)[2]) {
        if (r < i_s || r >= i_e) return;
        const long long o = r * pitch + gj0;
        if (!EDGE || gj0 + 3 < p.ny) {
            *reinterpret_cast<ulonglong2 *>(a.phi_out + o) = make_ulonglong2(x[0], x[1]);
            *reinterpret_cast<ulonglong2 *>(a.psi_out + o) = make_ulonglong2(v[0], v[1]);
        } else {
            const float xs[4] = {el<0>(x), el<1>(x), el<2>(x), el<3>(x)}, vs[4] = {el<0>(v), el<1>(v), el<2>(v), el<3>(v)};
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (gj0 + k < p.ny) {
                    a.phi_out[o + k] = xs[k];
                    a.psi_out[o + k] = vs[k];
                }
        }
    };
    if (w == 0) {
#pragma unroll 1
        for (int q = 0; q < SK_IN - 1; q++) issue();
    }

    const SkewK kk = {pk(-a.gam, -a.gam), pk(-a.kappa, -a.kappa), pk(a.c2, a.c2)};
    SkewWin q;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        q.XA[0][h] = q.XA[1][h] = q.VA[0][h] = q.VA[1][h] = q.DA[h] = 0;
        q.XB[0][h] = q.XB[1][h] = q.VB[0][h] = q.VB[1][h] = q.DB[h] = 0;
    }
    // the warp's place in its input (the ring, or the hand-over pair of the warp before it) and in
    // the lagged rings: the slot of rows (m, m+1) and of the two rows before them (warp w starts
    // with the rows of step w; before step 0 there is nothing, and nothing stored depends on it)
    const float *const in_lo = my4 + (w == 0 ? SM::IN : SM::HAND + (w - 1) * 1024);
    const float *const in_hi = in_lo + (w == 0 ? SK_IN : 2) * 512;
    const float *in = w == 0 ? in_lo : in_lo + ((s_first - 1) & 1) * 512;
    float *const out_lo = my4 + SM::HAND + w * 1024;
    int out_at = (s_first & 1) * 512;
    int tcur = w * 64, tprev = w == 0 ? (SM::NT - 1) * 64 : (w - 1) * 64;  // in words of the 4-byte rings
    int m = m0 + 2 * s_first - 4 * w;
    if (P > 1)
        for (int s = 0; s < s_first; s++) team_sync();
    const auto step = [&](auto edge) {
        if (w == 0) cp_async_wait<SK_IN - 2>();  // the rows of step s have landed
        unsigned act[3] = {0xFu, 0xFu, 0xFu};  // rows m-2, m-1, m
        f2 T[3][2];
        float te[3] = {0.f, 0.f, 0.f};
        if (SM::NEED_ACT) {
            const unsigned *aw = reinterpret_cast<const unsigned *>(my1) + SM::ACT;
            act[0] = aw[tprev] >> (gj0 & 31);
            act[1] = aw[tprev + 32] >> (gj0 & 31);
            act[2] = aw[tcur] >> (gj0 & 31);
        }
#pragma unroll
        for (int k = 0; k < 3; k++) {
            T[k][0] = T[k][1] = 0;
            if (COEF == WG_COEF_TABLE) {
                const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(my4 + SM::TCC + (k < 2 ? 4 * tprev + k * 128 : 4 * tcur));
                T[k][0] = t.x;
                T[k][1] = t.y;
            }
        }
        if (need_tce) {
            te[0] = my1[SM::TCE + tprev];
            te[1] = my1[SM::TCE + tprev + 32];
            te[2] = my1[SM::TCE + tcur];
        }
        f2 xo[2][2], vo[2][2];
        constexpr int E = decltype(edge)::value;
        if constexpr (E == 3) {
            const bool full = p.osc_topbot || (m >= 0 && m <= 2) || (m >= p.nx - 1 && m <= p.nx + 1) ||
                              (p.src_on && m >= p.src_i && m <= p.src_i + 2);
            if (full) skew_step<COEF, PL, 2, INL>(p, a, kk, ed, m, w, gj0, in, T, te, act, q, xo, vo);
            else skew_step<COEF, PL, 1, INL>(p, a, kk, ed, m, w, gj0, in, T, te, act, q, xo, vo);
        } else {
            skew_step<COEF, PL, E, INL>(p, a, kk, ed, m, w, gj0, in, T, te, act, q, xo, vo);
        }
        if (!last) {
            float *out = out_lo + out_at;
#pragma unroll
            for (int u = 0; u < 2; u++) {
                *reinterpret_cast<ulonglong2 *>(out + u * 256) = make_ulonglong2(xo[u][0], xo[u][1]);
                *reinterpret_cast<ulonglong2 *>(out + u * 256 + 128) = make_ulonglong2(vo[u][0], vo[u][1]);
            }
        } else if (core) {
            if (two) {
                store(m - 2, xo[0], vo[0]);
                store(m - 1, xo[1], vo[1]);
            } else {
                store(m - 1, q.XB[1], q.VB[1]);
                store(m, q.XB[0], q.VB[0]);
            }
        }
        // on to the next step's rows
        in = in + 512 == in_hi ? in_lo : in + 512;
        out_at ^= 512;
        tprev = tcur;
        tcur = tcur == (SM::NT - 1) * 64 ? 0 : tcur + 64;
        if (w == 0) issue();  // into slots that no warp reads any more
        if (P > 1) team_sync();
    };
    if (!EDGE || !INL) {
        // EDGE (3): the full rules only where a step computes row 0, nx-1 or the point source
#pragma unroll 1
        for (int s = s_first; s <= s_last; s++, m += 2) step(std::integral_constant<int, EDGE ? 3 : 0>());
    } else {
        // The same in loops of their own: as branches of one loop the two forms cost a batch's masked
        // strips 1.7 times the inner strip's instructions instead of 1.45 (64 scenes of 1000x120,
        // mirror: 113 to 99 us for 10 updates).  (Single grids' table forms spill more this way:
        // 1172 to 1058 Gcell/s on 3840x2160.)
        const auto next_full = [&](int mm) {
            if (p.osc_topbot) return mm;
            int n = 0x7fffffff;
            if (p.src_on && mm <= p.src_i + 2) n = p.src_i;
            if (mm <= p.nx + 1) n = min(n, p.nx - 1);
            return mm <= 2 ? min(n, 0) : n;
        };
        const int m_last = m + 2 * (s_last - s_first);
        while (m <= m_last) {
            const int mf = min(next_full(m), m_last + 1);
#pragma unroll 1
            for (; m < mf; m += 2) step(std::integral_constant<int, 1>());
            if (m <= m_last && m >= next_full(m)) {
                step(std::integral_constant<int, 2>());
                m += 2;
            }
        }
    }
    if (P > 1)
        for (int s = s_last + 1; s < nsteps; s++) team_sync();
}


// One team per task: column tile t.x, rows [t.y, t.z), whether it is an EDGE strip (t.w).  The task list fills one wave of resident teams.
// Resident teams per SM: 20 or 21 warps (96 registers a thread for P = 2, 80 for P = 3); 24
// warps left 80 registers and measured 3-10% slower, 16 warps 10% slower.
constexpr int skew_min_blocks(int P) { return P == 1 ? 20 : (P == 2 ? 10 : 7); }
template <int COEF, int P, int PL>
__global__ void __launch_bounds__(32 * P, skew_min_blocks(P))
    k_step_skew(const __grid_constant__ DevParams p, const __grid_constant__ TbArgs a, const int4 *__restrict__ tasks, int K)
{
    extern __shared__ float4 skew_smem[];
    const int lane = threadIdx.x & 31, w = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int H = (K + 3) & ~3, step = 128 - 2 * H;
    const int4 t = tasks[blockIdx.x];
    const int lo = t.x * step, hi = lo + step;  // the core columns of tile t.x
    const int gj0 = lo - H + 4 * lane;
    float *shm = reinterpret_cast<float *>(skew_smem);
    // Programmatic dependent launch: this pass may be launched while the previous one is
    // finishing (its blocks take the SMs the previous pass's blocks leave); it reads and
    // writes the fields only after the previous pass has completed and its writes are
    // visible.  The next pass may be launched from here on.
    pdl_wait();
    pdl_trigger();
    if (t.w)
        skew_strip<COEF, PL, P, true, false>(p, a, K, t.y, t.z, gj0, lane, w, shm, lo, hi, 0, p.nx, 0, p.ny);
    else
        skew_strip<COEF, PL, P, false, false>(p, a, K, t.y, t.z, gj0, lane, w, shm, lo, hi, 0, p.nx, 0, p.ny);
}

// The ghost cells that mirror the rows [i_s, i_e) and columns [lo, hi) of a wrapped scene's new
// fields, by the team that stored them: a cell within BATCH_GHOST_COLS of the left or right edge or
// BATCH_GHOST_ROWS of the top or bottom one goes to every place of the extended grid that wraps to
// it, but for the ghost columns of a real row's last group of four, which the team of the last tile
// stores with that group: every cell has one writer.
// A kernel before each pass did this over the whole batch, 22 us with 48 scenes, and
// kept passes from overlapping: 48 scenes of 256 to 960 a side, half of them periodic, 10 updates:
// 224 to 195 us.
__device__ __noinline__ void skew_images(float *f0, float *f1, int nx, int ny, int pitch, int i_s, int i_e, int lo, int hi,
                                         int t0, int nt)
{
    constexpr int GC = BATCH_GHOST_COLS, GX = BATCH_GHOST_COLS_R, GR = BATCH_GHOST_ROWS;
    const int ge = batch_group_end(ny);
    // cells t0, t0 + nt, .. of an nr x nc block whose cell (r, c) is (row(r), col(c)): the loads of
    // four cells before their stores while there are four, then one by one
    const auto cells = [&](auto u, int t, int nc, auto row, auto col) {
        constexpr int U = decltype(u)::value;
        float x[U], v[U];
        int rr[U], cc[U];
#pragma unroll
        for (int k = 0; k < U; k++) {
            const int tk = t + k * nt, r = tk / nc;
            rr[k] = row(r);
            cc[k] = col(tk - r * nc);
            const long long o = (long long)rr[k] * pitch + cc[k];
            x[k] = f0[o];
            v[k] = f1[o];
        }
#pragma unroll
        for (int k = 0; k < U; k++)
            for (int i = rr[k] - nx * ((rr[k] + GR) / nx); i < nx + GR; i += nx)
                for (int j = cc[k] - ny * ((cc[k] + GC) / ny); j < ny + GX; j += ny)
                    if (i != rr[k] || (j != cc[k] && (j < ny || j >= ge))) {
                        f0[(long long)i * pitch + j] = x[k];
                        f1[(long long)i * pitch + j] = v[k];
                    }
    };
    const auto block = [&](int nr, int nc, auto row, auto col) {
        int t = t0;
        for (; t + 3 * nt < nr * nc; t += 4 * nt) cells(std::integral_constant<int, 4>(), t, nc, row, col);
        for (; t < nr * nc; t += nt) cells(std::integral_constant<int, 1>(), t, nc, row, col);
    };
    // the two bands of columns, all rows
    const int wa = max(0, min(hi, GX) - lo), b0 = max(max(lo, ny - GC), lo + wa), wb = max(0, hi - b0), wc = wa + wb;
    if (wc > 0) block(i_e - i_s, wc, [&](int r) { return i_s + r; }, [&](int q) { return q < wa ? lo + q : b0 + q - wa; });
    // the two bands of rows, the columns between
    const int na = max(0, min(i_e, GR) - i_s), r0 = max(max(i_s, nx - GR), i_s + na), nb = max(0, i_e - r0);
    if (hi - lo > wc)
        block(na + nb, hi - lo - wc, [&](int r) { return r < na ? i_s + r : r0 + r - na; }, [&](int q) { return lo + wa + q; });
}

// A pass over a periodic scene in the ghost layout: every tile is inner, reads its wrapped halo as
// ordinary neighbours and writes the ghosts of its cells.  A kernel of its own, so that the strips
// of k_step_skew keep their constants.  Periodic grids took single updates before, at DRAM's rate:
// 3840x2160, table, 31.3 to 7.5 us an update (1105 Gcell/s); 1277x717 7.0 to 2.6; 256x192, where a launch
// bounds the update, 4.9 to 1.8.
template <int COEF, int P, int PL>
__global__ void __launch_bounds__(32 * P, skew_min_blocks(P))
    k_step_wrap(const __grid_constant__ DevParams p, const __grid_constant__ TbArgs a, const int4 *__restrict__ tasks, int K)
{
    extern __shared__ float4 skew_smem[];
    constexpr int GC = BATCH_GHOST_COLS, GR = BATCH_GHOST_ROWS;
    const int lane = threadIdx.x & 31, w = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int H = (K + 3) & ~3, step = 128 - 2 * H;
    const int4 t = tasks[blockIdx.x];
    const int lo = t.x * step, hi = min(lo + step, p.ny);
    pdl_wait();
    pdl_trigger();
    skew_strip<COEF, PL, P, false, false>(p, a, K, t.y, t.z, lo - H + 4 * lane, lane, w, reinterpret_cast<float *>(skew_smem), lo,
                                          hi, -GR, p.nx + GR, -GC, p.ny + GC);
    __syncthreads();  // the last warp's rows
    skew_images(a.phi_out, a.psi_out, p.nx, p.ny, p.pitch, t.y, t.z, lo, hi, threadIdx.x, 32 * P);
}

static bool skew_shape_ok(const DevParams &p, int K, int S)
{
    return K >= 2 && K <= WG_SKEW_MAX_K && S >= 8 && S <= 4096 && p.ny >= 8 && p.nx >= 2;
}

template <int COEF, int P, int PL, bool WRAP>
static int skew_capacity()
{
    const auto kernel = WRAP ? k_step_wrap<COEF, P, PL> : k_step_skew<COEF, P, PL>;
    constexpr size_t smem = SkewShm<COEF, PL, P>::BYTES;
    static PerDevice cap;
    return cap.get([&] {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smem + SkewShm<COEF, PL, P>::OSC_BYTES));
        int nb = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, 32 * P, smem);
        return std::max(1, nb) * sm_count();
    });
}

template <int COEF, int P, int PL>
static int skew_launch(const DevParams &p, const TbArgs *a, int K, const int4 *tasks, int ntasks, cudaStream_t st, bool wrap)
{
    // the capacity sets the shared-memory attribute once
    const int cap = wrap ? skew_capacity<COEF, P, PL, true>() : skew_capacity<COEF, P, PL, false>();
    if (a)
        launch_pdl(wrap ? k_step_wrap<COEF, P, PL> : k_step_skew<COEF, P, PL>, dim3((unsigned)ntasks), dim3(32 * P),
                   SkewShm<COEF, PL, P>::BYTES + (p.osc_left ? SkewShm<COEF, PL, P>::OSC_BYTES : 0), st, p, *a, tasks, K);
    return cap;
}

template <int COEF, int PL>
static int skew_dispatch(const DevParams &p, const TbArgs *a, int K, const int4 *tasks, int ntasks, cudaStream_t st, bool wrap)
{
    switch ((K + 1) / 2) {
    case 1: return skew_launch<COEF, 1, PL>(p, a, K, tasks, ntasks, st, wrap);
    case 2: return skew_launch<COEF, 2, PL>(p, a, K, tasks, ntasks, st, wrap);
    default: return skew_launch<COEF, 3, PL>(p, a, K, tasks, ntasks, st, wrap);
    }
}

// Launches a pass (a != nullptr) and returns the number of resident teams.
static int skew_call(const DevParams &p, const TbArgs *a, int coef, int K, const int4 *tasks, int ntasks, cudaStream_t st, bool wrap)
{
    const int pl = skew_form(p.twospeeds, p.floor_clamp, p.kappa);
    if (coef == WG_COEF_TABLE) {
        if (pl == PL_ALL) return skew_dispatch<WG_COEF_TABLE, PL_ALL>(p, a, K, tasks, ntasks, st, wrap);
        if (pl == PL_MASKED) return skew_dispatch<WG_COEF_TABLE, PL_MASKED>(p, a, K, tasks, ntasks, st, wrap);
        return skew_dispatch<WG_COEF_TABLE, PL_GEN>(p, a, K, tasks, ntasks, st, wrap);
    }
    if (pl == PL_ALL) return skew_dispatch<WG_COEF_MASK, PL_ALL>(p, a, K, tasks, ntasks, st, wrap);
    if (pl == PL_MASKED) return skew_dispatch<WG_COEF_MASK, PL_MASKED>(p, a, K, tasks, ntasks, st, wrap);
    return skew_dispatch<WG_COEF_MASK, PL_GEN>(p, a, K, tasks, ntasks, st, wrap);
}

// Task list of a skewed pass.  Every column tile is cut into row chunks; a chunk costs its
// rows plus the pipeline's fill (skew_fill rows), and an EDGE chunk (a tile that holds column
// 0 or ny-1, rows 0 or nx-1 within K, the point source) SKEW_EDGE_COST times that.  Chunks are
// sized so that all teams carry about the same cost and the list fills the resident teams
// once (chunks of at least min_rows rows).  Tasks are ordered by row band so that the edge
// chunks spread over the SMs.
// shifted = false: tile tj spans columns [tj*step - H, tj*step - H + 128) and stores
// [tj*step, (tj+1)*step).  shifted = true (batches): tile tj starts at column tj*step, so
// the first tile needs no halo on the left and the last none on the right (column 0 and
// ny-1 read no column outside the grid); a scene of 128 columns or fewer is one tile.
constexpr double SKEW_EDGE_COST = 2.0;  // 1.5, 2.3, 2.6 and 3.0 measured slower on 3840x2160
static int skew_fill(int K) { return 2 * K + 2 * ((K + 1) / 2) - 2; }
static std::vector<int4> skew_plan(const DevParams &p, int K, int min_rows, int cap, bool shifted = false)
{
    const int H = (K + 3) & ~3, step = 128 - 2 * H, F = skew_fill(K), sh = shifted ? 0 : H;
    const int nx = p.nx;
    const int tiles_j = shifted ? 1 + std::max(0, (p.ny - 128 + step - 1) / step) : (p.ny + step - 1) / step;
    const auto col_edge = [&](int tj) { return tj * step - sh < 1 || tj * step - sh + 128 > p.ny - 1; };
    const auto form = [&](int tj, int i_s, int i_e) {
        const int t0 = tj * step - sh;
        const bool src = p.src_on && p.src_i >= i_s - K && p.src_i < i_e + K && p.src_j >= t0 && p.src_j < t0 + 128;
        return (i_s < K || i_e + K > nx || src || col_edge(tj)) ? 1 : 0;
    };
    // the chunks of a tile, none of them costing more than `cost` where min_rows allows it: the
    // first and the last (EDGE) shorter, the others of equal length
    const auto cut = [&](int tj, double cost, std::vector<std::pair<int, int>> &out) {
        out.clear();
        const int rm = std::max(min_rows, (int)(cost / (col_edge(tj) ? SKEW_EDGE_COST : 1.0) - F));
        const int re = std::max(std::max(min_rows / 2, 2), (int)(cost / SKEW_EDGE_COST - F));
        if (nx <= re) {
            out.push_back({0, nx});
            return;
        }
        if (nx <= 2 * re + rm / 2) {
            const int n = std::max(2, (nx + re - 1) / re);
            for (int q = 0; q < n; q++) out.push_back({(int)((long long)q * nx / n), (int)((long long)(q + 1) * nx / n)});
            return;
        }
        const int nm = nx - 2 * re, n = std::max(1, (nm + rm - 1) / rm);
        out.push_back({0, re});
        for (int q = 0; q < n; q++) out.push_back({re + (int)((long long)q * nm / n), re + (int)((long long)(q + 1) * nm / n)});
        out.push_back({nx - re, nx});
    };
    std::vector<std::pair<int, int>> ch;
    const auto count = [&](double cost) {
        int n = 0;
        for (int tj = 0; tj < tiles_j; tj++) {  // only the edge tiles differ
            cut(tj, cost, ch);
            n += (int)ch.size();
        }
        return n;
    };
    // the smallest chunk cost whose list fits the resident teams
    double cost_lo = min_rows + F, cost_hi = 2.0 * SKEW_EDGE_COST * (nx + F);
    if (count(cost_lo) > cap) {
        for (int it = 0; it < 24; it++) {
            const double c = 0.5 * (cost_lo + cost_hi);
            (count(c) > cap ? cost_lo : cost_hi) = c;
        }
    } else {
        cost_hi = cost_lo;
    }
    struct T { double key; int4 t; };
    std::vector<T> ts;
    const auto add = [&](int tj, int i_s, int i_e) {
        if (i_s < i_e) ts.push_back({(i_s + i_e) * 0.5 / nx + tj * 1e-9, make_int4(tj, i_s, i_e, form(tj, i_s, i_e))});
    };
    for (int tj = 0; tj < tiles_j; tj++) {
        cut(tj, cost_hi, ch);
        for (auto &c : ch) {
            const int mid = (c.first + c.second) / 2;
            if (!col_edge(tj) && c.first >= K && c.second + K <= nx && form(tj, c.first, c.second)) {
                add(tj, c.first, mid);  // a point source in an inner chunk: two shorter ones
                add(tj, mid, c.second);
            } else {
                add(tj, c.first, c.second);
            }
        }
    }
    std::sort(ts.begin(), ts.end(), [](const T &x, const T &y) { return x.key < y.key; });
    std::vector<int4> out(ts.size());
    for (size_t i = 0; i < ts.size(); i++) out[i] = ts[i].t;
    return out;
}

// The same for a periodic scene: all strips cost the same, so every tile is cut into equal chunks of
// at least min_rows rows, as many as fill the resident teams once.
static std::vector<int4> wrap_plan(const DevParams &p, int K, int min_rows, int cap)
{
    const int step = 128 - 2 * ((K + 3) & ~3), tiles = (p.ny + step - 1) / step;
    const int n = std::max(1, std::min(p.nx / std::max(min_rows, 1), cap / tiles));
    std::vector<int4> out;
    for (int q = 0; q < n; q++)
        for (int tj = 0; tj < tiles; tj++)
            out.push_back(make_int4(tj, (int)((long long)q * p.nx / n), (int)((long long)(q + 1) * p.nx / n), 0));
    return out;
}

// A task list in device memory.  On a scene that is recorded its stream may be recording now: the
// allocation is then made in the capture mode that allows it, and the copy on a stream of its own.
static wg_status device_list(const std::vector<int4> &v, bool recorded, int4 **dev)
{
    const size_t bytes = v.size() * sizeof(int4);
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaStream_t st = nullptr;
    if (recorded) WG_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    int4 *d = nullptr;
    cudaError_t e = cudaMalloc(&d, bytes);
    if (e == cudaSuccess && recorded) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess) {
        e = recorded ? cudaMemcpyAsync(d, v.data(), bytes, cudaMemcpyHostToDevice, st)
                     : cudaMemcpy(d, v.data(), bytes, cudaMemcpyHostToDevice);
        if (e == cudaSuccess && recorded) e = cudaStreamSynchronize(st);
    }
    if (st) cudaStreamDestroy(st);
    if (recorded) cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) {
        if (d) cudaFree(d);
        return cuda_fail(e, "skewed task list");
    }
    *dev = d;
    return WG_OK;
}

// Task list of (depth K, minimum rows L) for this scene, built once and kept on the device.
static wg_status skew_tasks(wg_scene *s, int K, int L, const int4 **tasks, int *ntasks)
{
    if (K < 0 || K > WG_SKEW_MAX_K) { set_error("skewed depth %d outside 0..%d", K, WG_SKEW_MAX_K); return WG_ERR_INVALID; }
    SkewPlanCache &c = s->skew[K];
    if (!c.dev || c.min_rows != L) {
        const int cap = skew_call(s->dp, nullptr, s->coef, K, nullptr, 0, s->st, s->wrap);
        const std::vector<int4> v = s->wrap ? wrap_plan(s->dp, K, L, cap) : skew_plan(s->dp, K, L, cap);
        if (c.dev && s->recorded) s->retired.push_back(c.dev);
        else if (c.dev) cudaFree(c.dev);
        c.dev = nullptr;
        if (wg_status st = device_list(v, s->recorded, &c.dev)) return st;
        c.n = (int)v.size();
        c.min_rows = L;
    }
    *tasks = c.dev;
    *ntasks = c.n;
    return WG_OK;
}

// ---------------------------------------------------------------------------
// Skewed passes over a batch of scenes (mask coefficients, FP32).  Each team takes the task of
// its block, then, from a longer list, tasks by a ticket counter: table entry, first column of the tile (shifted tiling),
// rows i_s | i_e << 16, kind (0 inner, 1 EDGE, 3 periodic in the ghost layout).  The scene's
// parameters are staged in the team's shared memory.  Pass q of a frame reads pair
// (pair ^ q) of the scene and writes the other pair.  Oscillating values and source
// increments are computed inline at update time + toff + level.
//
// The first task goes by block because a pass's blocks are resident early, where the pass before
// left room: taken by ticket, a short list's tasks fell on the SMs unevenly (6 grids of 500x400,
// 10 updates, mirror: 53.5 us by ticket with 15 warps per SM, 70 with 21; 39.1 now).  15 warps
// per SM, the most that 128 registers allow, measured 10-15% slower than 21 on long lists, although
// the general form spills (64 scenes of 1000x896, mirror: 630 to 512 us; 192 scenes of 128 to
// 512 a side, absorbing: 333 to 285 us for 10 updates).
// ---------------------------------------------------------------------------
static_assert(sizeof(DevParams) % 4 == 0, "DevParams is copied as 32-bit words");

template <int P, int PL>
__global__ void __launch_bounds__(32 * P, P == 1 ? 16 : skew_min_blocks(P))
    k_batch_skew(const SlotDev *__restrict__ tab, const SlotDyn *__restrict__ dyn, const int4 *__restrict__ tasks,
                 const int *__restrict__ ntasks, int *__restrict__ ticket, int K, int q, int toff)
{
    extern __shared__ float4 skew_smem[];
    __shared__ DevParams p;
    __shared__ int s_ticket;
    const int lane = threadIdx.x & 31, w = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    float *shm = reinterpret_cast<float *>(skew_smem);
    // The lists and the scenes' parameters do not change within a frame, and the first pass of
    // a frame is not launched early: they are read before the wait for the previous pass.
    const int n = *ntasks, H = (K + 3) & ~3;
    if (n == 0) pdl_wait();  // (so that the pass after this one still waits for the one before)
    int t = blockIdx.x;  // the first tasks by block, so that they spread over the SMs; then by ticket
    for (bool first = true; t < n; first = false) {
        const int4 d = tasks[t];
        const SlotDev &sd = tab[d.x];
        {
            const int *src = reinterpret_cast<const int *>(&sd.p);
            int *dst = reinterpret_cast<int *>(&p);
            for (int k = threadIdx.x; k < (int)(sizeof(DevParams) / 4); k += 32 * P) dst[k] = src[k];
        }
        if (first) {
            pdl_wait();
            pdl_trigger();
        }
        __syncthreads();
        const SlotDyn dy = dyn[sd.slot];
        const int pin = dy.pair ^ (q & 1), pout = pin ^ 1;
        TbArgs a;
        a.phi = (const float *)sd.f[2 * pin];
        a.psi = (const float *)sd.f[2 * pin + 1];
        a.phi_out = (float *)sd.f[2 * pout];
        a.psi_out = (float *)sd.f[2 * pout + 1];
        a.act = sd.act;
        a.tcc = a.tc = nullptr;
        a.c2 = sd.cf[CF_C2];
        a.c2b = sd.cf[CF_C2B];
        a.gam = sd.cf[CF_GAM];
        a.gamb = sd.cf[CF_GAMB];
        a.kappa = sd.cf[CF_KAPPA];
        a.ks = sd.cf[CF_KS];
        a.kt = sd.cf[CF_KT];
        a.gs = sd.cf[CF_GS];
        a.gt = sd.cf[CF_GT];
        a.vmax = sd.cf[CF_VMAX];
        a.courant = sd.cf[CF_COURANT];
        a.courantb = sd.cf[CF_COURANTB];
        a.t0 = dy.time + toff;
        a.osc = nullptr;
        a.src = nullptr;
        a.err = nullptr;
        const int i_s = d.z & 0xFFFF, i_e = (int)((unsigned)d.z >> 16);
        const int gjs = d.y, gj0 = gjs + 4 * lane;
        const bool wrap = d.w == 3;  // a halo on both sides of every tile
        const int lo = wrap ? max(gjs + H, 0) : (gjs <= 0 ? 0 : gjs + H);
        const int hi = wrap ? min(gjs + 128 - H, p.ny) : (gjs + 128 >= p.ny ? p.ny : gjs + 128 - H);
        const int gr = wrap ? BATCH_GHOST_ROWS : 0, gc = wrap ? BATCH_GHOST_COLS : 0;
        if (d.w == 1)
            skew_strip<WG_COEF_MASK, PL, P, true, true>(p, a, K, i_s, i_e, gj0, lane, w, shm, lo, hi, 0, p.nx, 0, p.ny);
        else
            skew_strip<WG_COEF_MASK, PL, P, false, true>(p, a, K, i_s, i_e, gj0, lane, w, shm, lo, hi, -gr, p.nx + gr, -gc,
                                                         p.ny + gc);
        if (wrap) {
            __syncthreads();  // the last warp's rows
            skew_images(a.phi_out, a.psi_out, p.nx, p.ny, p.pitch, i_s, i_e, lo, hi, threadIdx.x, 32 * P);
        }
        if (n <= (int)gridDim.x) break;
        __syncthreads();  // every warp is done with the task
        if (threadIdx.x == 0) s_ticket = (int)gridDim.x + atomicAdd(ticket, 1);
        __syncthreads();
        t = s_ticket;
    }
}

template <int P, int PL>
static int batch_skew_cap_p()
{
    constexpr size_t smem = SkewShm<WG_COEF_MASK, PL, P>::BYTES;
    static PerDevice cap;
    return cap.get([] {
        cudaFuncSetAttribute(k_batch_skew<P, PL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        int nb = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_batch_skew<P, PL>, 32 * P, smem);
        return std::max(1, nb) * sm_count();
    });
}

int batch_skew_form(const wg_params &p)
{
    return skew_form(p.twospeeds, p.floor_clamp, p.kappa) == PL_MASKED ? PL_MASKED : PL_GEN;
}

int batch_skew_fill(int K) { return skew_fill(K); }

int batch_skew_tiles(const DevParams &p, int K)
{
    const int step = 128 - 2 * ((K + 3) & ~3);
    if (p.b_cond == WG_BC_PERIODIC) return (p.ny + step - 1) / step;  // halo on both sides of every tile
    return 1 + std::max(0, (p.ny - 128 + step - 1) / step);
}

int batch_skew_capacity(int K, int form)
{
    if (K < 2 || K > WG_SKEW_MAX_K) return 0;
    if (form == PL_MASKED) return K <= 2 ? batch_skew_cap_p<1, PL_MASKED>() : (K <= 4 ? batch_skew_cap_p<2, PL_MASKED>()
                                                                                     : batch_skew_cap_p<3, PL_MASKED>());
    return K <= 2 ? batch_skew_cap_p<1, PL_GEN>() : (K <= 4 ? batch_skew_cap_p<2, PL_GEN>() : batch_skew_cap_p<3, PL_GEN>());
}

template <int P>
static void launch_batch_skew_p(int form, dim3 g, const SlotDev *tab, const SlotDyn *dyn, const int4 *tasks, const int *ntasks,
                                int *ticket, int K, int q, int toff, cudaStream_t st)
{
    constexpr size_t smem = SkewShm<WG_COEF_MASK, PL_GEN, P>::BYTES;  // the mask forms share a layout
    if (form == PL_MASKED) launch_pdl(k_batch_skew<P, PL_MASKED>, g, dim3(32 * P), smem, st, tab, dyn, tasks, ntasks, ticket, K, q, toff);
    else launch_pdl(k_batch_skew<P, PL_GEN>, g, dim3(32 * P), smem, st, tab, dyn, tasks, ntasks, ticket, K, q, toff);
}

void launch_batch_skew(int K, int form, const SlotDev *tab, const SlotDyn *dyn, const int4 *tasks, const int *ntasks,
                       int *ticket, int q, int toff, cudaStream_t st)
{
    const dim3 g(std::max(1, batch_skew_capacity(K, form)));
    switch ((K + 1) / 2) {
    case 1: launch_batch_skew_p<1>(form, g, tab, dyn, tasks, ntasks, ticket, K, q, toff, st); break;
    case 2: launch_batch_skew_p<2>(form, g, tab, dyn, tasks, ntasks, ticket, K, q, toff, st); break;
    case 3: launch_batch_skew_p<3>(form, g, tab, dyn, tasks, ntasks, ticket, K, q, toff, st); break;
    default: break;
    }
}

bool batch_wrap_ok(const wg_params &p, int prec)
{
    // nx + 2 ghost-row bands within a grid dimension of the mask's ghost kernel (65535)
    return prec == WG_FP32 && p.b_cond == WG_BC_PERIODIC && !p.bc_neumann && !p.src_on && !p.oscillate_left &&
           !p.oscillate_topbot && p.ny >= 8 && p.nx >= 2 && p.nx + 2 * BATCH_GHOST_ROWS <= 0xFFFF;
}

bool batch_skew_ok(const wg_params &p, int prec)
{
    if (batch_wrap_ok(p, prec)) return true;
    return prec == WG_FP32 && (p.b_cond == WG_BC_DIRICHLET || p.b_cond == WG_BC_ABSORBING) && !p.bc_neumann &&
           p.ny >= 8 && p.nx >= 2 && p.nx <= 0xFFFF;
}

void batch_skew_plan(const DevParams &p, int entry, int K, int rows, std::vector<int4> &tasks, std::vector<float> &cost)
{
    const int H = (K + 3) & ~3, step = 128 - 2 * H, F = skew_fill(K);
    if (p.b_cond == WG_BC_PERIODIC) {  // ghost layout: every tile inner (kind 3), rows in chunks of rows..2 rows
        const int tiles_j = (p.ny + step - 1) / step, nl = std::max(1, p.nx / std::max(rows, 1));
        for (int tj = 0; tj < tiles_j; tj++)
            for (int q = 0; q < nl; q++) {
                const int i_s = (int)((long long)q * p.nx / nl), i_e = (int)((long long)(q + 1) * p.nx / nl);
                if (i_s >= i_e) continue;
                tasks.push_back(make_int4(entry, tj * step - H, (int)((unsigned)i_s | ((unsigned)i_e << 16)), 3));
                cost.push_back((float)(i_e - i_s + F));
            }
        return;
    }
    const std::vector<int4> v = skew_plan(p, K, rows, 1 << 30, true);  // inner chunks of rows..2 rows rows
    for (const int4 &t : v) {
        tasks.push_back(make_int4(entry, t.x * step, (int)((unsigned)t.y | ((unsigned)t.z << 16)), t.w));
        cost.push_back((float)((t.z - t.y + F) * (t.w ? SKEW_EDGE_COST : 1.0)));
    }
}

static int tb_halo(int K) { return (K + 3) & ~3; }

static bool tb_shape_ok(int K, int L, int W)
{
    return K >= 2 && K <= 8 && (W == 128 || W == 256) && L >= 16 && L <= 64 && (L % 2 == 0) && L - 2 * K >= 8 &&
           W - 2 * tb_halo(K) >= 32 && tb_layout(WG_COEF_TABLE, L, W).bytes <= 200 * 1024;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no libcuda link)
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)f;
    });
    return fn;
}

// 2-D map over a pitched array of 4-byte elements: dims {cols, rows}, row stride bytes
static bool make_map(CUtensorMap *m, const void *base, bool is_float, uint64_t cols, uint64_t rows, uint64_t stride,
                     uint32_t box_cols, uint32_t box_rows)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {stride};
    cuuint32_t box[2] = {box_cols, box_rows};
    cuuint32_t es[2] = {1, 1};
    return fn(m, is_float ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void *>(base),
              dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct TbMaps {
    CUtensorMap phi, psi, tcc, act;
};

static bool tb_maps(wg_scene *s, const TbArgs &a, int L, int W, TbMaps *m)
{
    const uint64_t stride = (uint64_t)s->pitch * 4;
    bool ok = make_map(&m->phi, a.phi, true, s->prm.ny, s->prm.nx, stride, W, L) &&
              make_map(&m->psi, a.psi, true, s->prm.ny, s->prm.nx, stride, W, L) &&
              make_map(&m->act, s->act, false, s->dp.wpitch, s->prm.nx, (uint64_t)s->dp.wpitch * 4, TB_AW, L);
    if (ok && s->coef == WG_COEF_TABLE) ok = make_map(&m->tcc, a.tcc, true, s->prm.ny, s->prm.nx, stride, W, L);
    else m->tcc = m->phi;
    return ok;
}

static bool launch_tb(wg_scene *s, const TbArgs &a, int K, int L, int W)
{
    if (!tb_shape_ok(K, L, W)) return false;
    const int Kh = tb_halo(K);
    TbMaps m;
    if (!tb_maps(s, a, L, W, &m)) {
        set_error("cuTensorMapEncodeTiled failed");
        return false;
    }
    const DevParams &p = s->dp;
    dim3 grd((p.ny + (W - 2 * Kh) - 1) / (W - 2 * Kh), (p.nx + (L - 2 * K) - 1) / (L - 2 * K));
    const size_t sm = tb_layout(s->coef, L, W).bytes;
    static std::once_flag attr_once;  // raise the dynamic shared-memory limit once per process
    std::call_once(attr_once, [] {
        cudaFuncSetAttribute(k_step_tb<WG_COEF_TABLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(k_step_tb<WG_COEF_MASK>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    });
    if (s->coef == WG_COEF_TABLE)
        k_step_tb<WG_COEF_TABLE><<<grd, W, sm, s->st>>>(p, a, m.phi, m.psi, m.tcc, m.act, K, Kh, L);
    else
        k_step_tb<WG_COEF_MASK><<<grd, W, sm, s->st>>>(p, a, m.phi, m.psi, m.tcc, m.act, K, Kh, L);
    return true;
}

static bool tb_depth_ok(int k) { return k >= 2 && k <= 8; }

bool tb_supported(const wg_scene *s)
{
    return s->prec == WG_FP32 && (s->prm.b_cond == WG_BC_DIRICHLET || s->prm.b_cond == WG_BC_ABSORBING || s->wrap) &&
           s->nrec == 0 && !s->has_ghosts && (s->coef == WG_COEF_MASK || s->tg == nullptr);
}

static wg_status ensure_tb_buffers(wg_scene *s)
{
    for (int k = 0; k < 2; k++)
        if (!s->g[k])
            if (wg_status st = scene_alloc_field(s, &s->g[k])) return st;
    return WG_OK;
}

wg_status tb_prepare(wg_scene *s, int n)
{
    if (s->wrap && !s->mask_ghosts_ok) {
        launch_act_ghosts(s->act, s->dp.wpitch, s->prm.nx, s->prm.ny, s->st);
        if (s->tcc) launch_grid_ghosts((float *)s->tcc, nullptr, s->prm.nx, s->prm.ny, s->pitch, s->st);
        s->launches += s->tcc ? 2 : 1;
        WG_CUDA(cudaGetLastError());
        s->mask_ghosts_ok = true;
    }
    if (!s->prm.oscillate_left && !s->prm.src_on) return WG_OK;
    const size_t need = (size_t)n * (s->prm.oscillate_left ? s->prm.ny : 1);
    if (need > s->bv_cap) {
        if (s->bv_osc) cudaFree(s->bv_osc);
        if (s->bv_src) cudaFree(s->bv_src);
        s->bv_osc = nullptr;
        s->bv_src = nullptr;
        s->bv_cap = 0;
        WG_CUDA(cudaMalloc(&s->bv_osc, need * sizeof(float)));
        WG_CUDA(cudaMalloc(&s->bv_src, need * sizeof(double)));
        s->bv_cap = need;
    }
    s->bv_t0 = s->time;
    const int threads = 256, blocks = (int)((need + threads - 1) / threads);
    launch_pdl(k_boundary_values, dim3(blocks), dim3(threads), 0, s->st, s->dp, s->time, n, s->bv_osc, s->bv_src);
    s->launches++;
    WG_CUDA(cudaGetLastError());
    return WG_OK;
}

static TbArgs tb_args(wg_scene *s)
{
    TbArgs a;
    a.phi = (const float *)s->f[s->cur];
    a.psi = (const float *)s->f[1 - s->cur];
    a.phi_out = (float *)s->g[0];
    a.psi_out = (float *)s->g[1];
    a.act = s->act;
    a.tcc = (const float *)s->tcc;
    a.tc = (const float *)s->tc;
    a.c2 = (float)s->dp.c2;
    a.c2b = (float)s->dp.c2b;
    a.gam = (float)s->dp.gam;
    a.gamb = (float)s->dp.gamb;
    a.kappa = (float)s->dp.kappa;
    a.ks = (float)s->dp.kappa_sides;
    a.kt = (float)s->dp.kappa_topbot;
    a.gs = (float)s->dp.gamma_sides;
    a.gt = (float)s->dp.gamma_topbot;
    a.vmax = (float)s->dp.vmax;
    a.courant = (float)s->dp.courant;
    a.courantb = (float)s->dp.courantb;
    a.t0 = s->time;
    const long long off = s->time - s->bv_t0;
    a.osc = s->bv_osc ? s->bv_osc + off * s->prm.ny : nullptr;
    a.src = s->bv_src ? s->bv_src + off : nullptr;
    a.err = s->dflag;
    return a;
}

template <>
wg_status tb_pass<float>(wg_scene *s, int k)
{
    wg_status st = ensure_tb_buffers(s);
    if (st) return st;
    if (!tb_depth_ok(k)) { set_error("temporal block depth %d outside 2..8", k); return WG_ERR_INVALID; }
    const int W = s->tile_j > 0 ? s->tile_j : 256, L = s->tile_i > 0 ? s->tile_i : 32;
    TbArgs a = tb_args(s);
    if (W == 1) {  // time-skewed streaming strips of L rows
        if (!skew_shape_ok(s->dp, k, L)) {
            set_error("unsupported skewed strip (depth %d of 2..6, %d rows of 8..4096, ny >= 8)", k, L);
            return WG_ERR_INVALID;
        }
        const int4 *tasks = nullptr;
        int ntasks = 0;
        if ((st = skew_tasks(s, k, L, &tasks, &ntasks))) return st;
        if (s->wrap && !s->ghosts_ok) {
            launch_grid_ghosts((float *)s->f[s->cur], (float *)s->f[1 - s->cur], s->prm.nx, s->prm.ny, s->pitch, s->st);
            s->launches++;
        }
        skew_call(s->dp, &a, s->coef, k, tasks, ntasks, s->st, s->wrap);
        s->ghosts_ok = s->wrap;
    } else if (clear_error(), !launch_tb(s, a, k, L, W)) {
        if (wg_last_error()[0] == 0) set_error("unsupported temporal block (depth %d, tile %d x %d)", k, L, W);
        return WG_ERR_INVALID;
    }
    s->launches++;
    // the pass's outputs become the scene's fields; the inputs become the next outputs
    std::swap(s->f[s->cur], s->g[0]);
    std::swap(s->f[1 - s->cur], s->g[1]);
    s->time += k;
    return WG_OK;
}

template <>
wg_status tb_pass<double>(wg_scene *, int)
{
    set_error("temporal blocking is FP32 only");
    return WG_ERR_STATE;
}

// Passes of a call of n updates at depth k, each of n/passes updates, rounded up while they last; 0:
// single updates.  The fewest passes of depth <= k, so that depths are equal to within one (10 updates
// at k = 4: 4, 3, 3, at k = 6: 5, 5; 6 and a single update would be three launches).  parity: an even
// number of passes for an even n, an odd one for an odd n (the last may then be a single update).
int tb_passes(int k, int n, bool parity)
{
    const int m = std::min(k, 8);
    if (m < 2 || n < 2) return 0;
    const int q = (n + m - 1) / m;
    return parity && ((q ^ n) & 1) ? q + 1 : q;
}

// ---------------------------------------------------------------------------
// Autotuner: temporal-block depth and tile width per size class, measured once per
// (size class, coefficient mode) with CUDA events on a copy of the scene's state.
// ---------------------------------------------------------------------------
static std::mutex g_tune_mu;
static std::map<std::tuple<int, int, int, int>, std::tuple<int, int, int>> g_tune;

static std::tuple<int, int, int, int> size_class(const wg_scene *s)
{
    auto lg = [](int v) { int c = 0; while ((1 << (c + 1)) <= v) c++; return c; };
    return {lg(s->prm.nx), lg(s->prm.ny), s->coef, s->prm.b_cond};
}

void autotune_scene(wg_scene *s)
{
    if (!tb_supported(s)) {
        s->tb_k = 1;
        s->tile_i = s->tile_j = 0;
        return;
    }
    const auto key = size_class(s);
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_tune.find(key);
        if (it != g_tune.end()) {
            std::tie(s->tb_k, s->tile_i, s->tile_j) = it->second;
            return;
        }
    }
    // save the state, time the candidates, restore the state
    const size_t fb = s->field_bytes;
    void *save[2] = {nullptr, nullptr};
    bool ok = ensure_tb_buffers(s) == WG_OK;
    for (int k = 0; k < 2 && ok; k++) ok = cudaMalloc(&save[k], fb) == cudaSuccess;
    int best_k = 1, best_l = 0, best_w = 0;
    if (ok) {
        cudaMemcpyAsync(save[0], scene_field_base(s, s->f[0]), fb, cudaMemcpyDeviceToDevice, s->st);
        cudaMemcpyAsync(save[1], scene_field_base(s, s->f[1]), fb, cudaMemcpyDeviceToDevice, s->st);
        const long long t_save = s->time;
        const int cur_save = s->cur;
        void *const bufs[] = {s->f[0], s->f[1], s->g[0], s->g[1]};  // the fields return to their buffers
        const int probes = s->probe_n;  // the probes sample the scene's updates, not these
        s->probe_n = 0;
        cudaEvent_t e0, e1;
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        const int updates = 120;  // a multiple of every depth 2..6; long enough for stable timings
        float best = 1e30f;
        struct Cand { int k, l, w; };
        // single updates, and skewed passes with chunks of at least 16 or 8 rows (the TMA tiles of
        // set_blocking are slower than the passes on every grid tried, by 1.5 to 5 times)
        const Cand cands[] = {{1, 0, 0},  {2, 16, 1}, {3, 16, 1}, {4, 16, 1}, {5, 16, 1},
                              {6, 16, 1}, {3, 8, 1},  {4, 8, 1},  {5, 8, 1},  {6, 8, 1}};
        for (const Cand &c : cands) {
            s->tb_k = c.k;
            s->tile_i = c.l;
            s->tile_j = c.w;
            float ms_best = 1e30f;
            for (int rep = 0; rep < 3; rep++) {
                cudaEventRecord(e0, s->st);
                const wg_status st = scene_step_impl<float>(s, updates);
                cudaEventRecord(e1, s->st);
                if (st != WG_OK) {  // a shape this scene does not take
                    cudaEventSynchronize(e1);
                    clear_error();
                    ms_best = 1e30f;
                    break;
                }
                cudaEventSynchronize(e1);
                float ms = 0.f;
                cudaEventElapsedTime(&ms, e0, e1);
                if (rep > 0) ms_best = std::min(ms_best, ms);
            }
            if (ms_best < best * 0.99f) {  // a later candidate must be faster by more than the noise
                best = ms_best;
                best_k = c.k;
                best_l = c.l;
                best_w = c.w;
            }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        s->cur = cur_save;
        s->probe_n = probes;
        for (int k = 0; k < 2; k++) {
            s->f[k] = bufs[k];
            s->g[k] = bufs[2 + k];
        }
        cudaMemcpyAsync(scene_field_base(s, s->f[0]), save[0], fb, cudaMemcpyDeviceToDevice, s->st);
        cudaMemcpyAsync(scene_field_base(s, s->f[1]), save[1], fb, cudaMemcpyDeviceToDevice, s->st);
        cudaStreamSynchronize(s->st);
        s->time = t_save;
        s->ghosts_ok = false;
    }
    for (void *p : save)
        if (p) cudaFree(p);
    cudaGetLastError();
    s->tb_k = best_k;
    s->tile_i = best_l;
    s->tile_j = best_w;
    if (!ok) return;  // no memory for the copy: single updates for this scene, but not for its class
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune[key] = {best_k, best_l, best_w};
}

}  // namespace wg
