// wg_batch.cu — many scenes of uneven sizes advanced together.
//
// Single updates: every active scene is cut into work items (BT_ROWS rows x 64 threads x 4
// columns in FP32, hdr->rows64 x ST_COLS in FP64); a frame of n updates is n launches of one
// persistent kernel (k_batch_step32, k_batch_step64, sized to fill every SM) whose blocks or
// warps take items from a device-side atomic counter, plus one kernel that advances each
// scene's step counter.  The whole frame is recorded once as a CUDA graph and replayed; the
// scene table, the work counts and the per-scene time and buffer parity live in device
// memory, so admitting or removing scenes changes data, not the graph.
//
// The per-cell arithmetic is the single-scene kernels' (k_step_bulk, strip64, fast_edge_v), so a
// scene advanced in a batch is bit-identical to the same scene advanced alone.  FP64
// scenes update in place (the new level overwrites psi); FP32 scenes (phi and the
// velocity) write each update into their other pair of fields.
//
// FP32 scenes with mirror ("Dirichlet"), absorbing or periodic boundaries (periodic ones
// in the ghost layout of wg_batch.h) take skewed passes instead (k_batch_skew, wg_tb.cu):
// a frame of n updates is a few passes of 2..6 updates
// each, at the depth class tuned for the scene's size class, writing between two buffer
// pairs.  Each depth class runs as its own branch of the frame's graph, beside the chain
// of single updates of the other scenes.  The skewed cells are the single-update cells
// bit for bit, so a batch gives the same fields with and without skewed passes.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>
#include "wg_internal.h"
#include "wg_scene.h"
#include "wg_cells.cuh"
#include "wg_batch.h"
#include "wg_step64.cuh"

namespace wg {

// An FP32 boundary-line cell (reference rules) plus the point source; out of line so that
// the tile loop below stays small.  Its arguments are plain pointers and values: the
// rule's argument block is built here, in registers of this call, not passed by address
// (an address taken across the call would put the block in local memory).
__device__ __noinline__ XV batch_edge_v(const DevParams &p, const float *cf, const float *phi, const float *vel,
                                        const uint32_t *act, const uint32_t *nz, int i, int j, long long time)
{
    FastArgs<float> a;
    a.phi = phi;
    a.psi = vel;
    a.out = nullptr;
    a.vout = nullptr;
    a.act = act;
    a.nz = nz;
    a.tcc = a.tc = a.tg = nullptr;
    a.c2f = cf[CF_C2];  // rounded on the host (a conversion here would run on the FP64 pipe)
    a.c2bf = cf[CF_C2B];
    a.gamf = cf[CF_GAM];
    a.gambf = cf[CF_GAMB];
    a.kappaf = cf[CF_KAPPA];
    a.courantf = cf[CF_COURANT];
    a.courantbf = cf[CF_COURANTB];
    a.ksf = cf[CF_KS];
    a.ktf = cf[CF_KT];
    a.gsf = cf[CF_GS];
    a.gtf = cf[CF_GT];
    a.vmaxf = cf[CF_VMAX];
    a.has_ghosts = 0;
    a.do_source = 1;
    XV r = fast_edge_v<WG_COEF_MASK>(p, a, i, j, time);
    if (p.src_on && i == p.src_i && j == p.src_j) r = source32(r, point_source(p, time));
    return r;
}

// The scene values the bulk update reads, held in registers for a work item (the
// descriptor lives in global memory, which the tile's stores could alias).
struct TileCoef {
    int nx, ny, pitch, wpitch, twospeeds, floor_clamp;
    float c2, c2b, gam, gamb, kappa;
};

// One FP32 work item: phi and the velocity vin; the new phi and velocity go to out and vout.
__device__ __forceinline__ void batch_tile(const DevParams &p, const float *cf, const float *__restrict__ phi,
                                           const float *__restrict__ vin, float *__restrict__ out,
                                           float *__restrict__ vout, const uint32_t *__restrict__ act,
                                           const uint32_t *__restrict__ nz, int i0, int jt, long long time)
{
    constexpr int V = Vec<float>::n;
    const TileCoef k{p.nx, p.ny, p.pitch, p.wpitch, p.twospeeds, p.floor_clamp,
                     cf[CF_C2], cf[CF_C2B], cf[CF_GAM], cf[CF_GAMB], cf[CF_KAPPA]};
    const float vmaxf = cf[CF_VMAX];
    const int j0 = (jt * BT_THREADS + (int)threadIdx.x) * V;
    // interior rows: the bulk rule (boundary columns and padding take the unwritten-cell
    // rule for now)
    for (int rr = threadIdx.y; rr < BT_ROWS; rr += blockDim.y) {
        const int i = i0 + rr;
        if (i >= k.nx - 1 || i == 0 || j0 >= k.pitch) continue;
        const size_t row = (size_t)i * k.pitch;
        float c[V], y[V], n[V], s[V];
        vload(phi + row + j0, c);
        vload(vin + row + j0, y);
        vload(phi + row + k.pitch + j0, n);
        vload(phi + row - k.pitch + j0, s);
        const float wl = (j0 > 0) ? phi[row + j0 - 1] : 0.f;
        const float er = (j0 + V < k.pitch) ? phi[row + j0 + V] : 0.f;
        const uint32_t word = act[(size_t)i * k.wpitch + (j0 >> 5)] >> (j0 & 31);
        float o[V], ov[V];
#pragma unroll
        for (int q = 0; q < V; q++) {
            const int j = j0 + q;
            const bool ac = (word >> q) & 1u;
            const bool upd = j >= 1 && j < k.ny - 1 && (k.twospeeds || ac);
            const float x = c[q];
            const float w = (q == 0) ? wl : c[q - 1];
            const float e = (q == V - 1) ? er : c[q + 1];
            XV r = keep32(x, y[q]);
            if (upd) {
                const float delta = ((n[q] - x) + (s[q] - x)) + ((e - x) + (w - x));
                r = upd32(x, y[q], ac ? k.c2 : k.c2b, delta, k.kappa, ac ? k.gam : k.gamb);
                if (k.floor_clamp && ac) r = clamp32(x, r, vmaxf);
            }
            o[q] = r.x;
            ov[q] = r.v;
        }
        vstore(out + row + j0, o);
        vstore(vout + row + j0, ov);
    }
    // then the boundary lines and the point source, by the threads that stored those
    // cells above (each reads phi and its own cell's velocity)
    const bool col0 = j0 == 0, colr = k.ny - 1 >= j0 && k.ny - 1 < j0 + V;
    const bool srcj = p.src_on && p.src_j >= j0 && p.src_j < j0 + V && p.src_j > 0 && p.src_j < k.ny - 1;
    auto edge = [&](size_t row, int i, int j) {
        const XV r = batch_edge_v(p, cf, phi, vin, act, nz, i, j, time);
        out[row + j] = r.x;
        vout[row + j] = r.v;
    };
    for (int rr = threadIdx.y; rr < BT_ROWS; rr += blockDim.y) {
        const int i = i0 + rr;
        if (i >= k.nx || j0 >= k.pitch) continue;
        const size_t row = (size_t)i * k.pitch;
        if (i == 0 || i == k.nx - 1) {
            for (int q = 0; q < V; q++) {
                const int j = j0 + q;
                if (j >= k.ny) break;
                edge(row, i, j);
            }
            continue;
        }
        if (col0) edge(row, i, 0);
        if (colr) edge(row, i, k.ny - 1);
        if (srcj && i == p.src_i) {
            const double add = point_source(p, time);
            out[row + p.src_j] = (float)A_((double)out[row + p.src_j], add);
            vout[row + p.src_j] = (float)A_((double)vout[row + p.src_j], add);
        }
    }
}

// Persistent blocks take FP32 work items (BT_ROWS rows x one column tile of one scene) from
// a device counter.  Each item's scene entry, first row, column tile and slot come from
// one int4 of the item table built with the scene table.  The ticket of the following
// item is taken while this one runs, and read after it, so its latency is hidden.
// all = 0: only the items of scenes without skewed passes (the first plain_tiles).
__global__ void __launch_bounds__(256, 4) k_batch_step32(const BatchHdr *__restrict__ hdr, const SlotDev *__restrict__ tab,
                                                         const int4 *__restrict__ items, SlotDyn *__restrict__ dyn,
                                                         int *__restrict__ counter, int u, int all)
{
    __shared__ int s_next[2];
    pdl_wait();  // launched by launch_pdl: the previous update has completed
    pdl_trigger();
    const int total = all ? hdr->total_tiles : hdr->plain_tiles;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    if (tid == 0) s_next[0] = atomicAdd(counter + u, 1);
    __syncthreads();
    for (int buf = 0;; buf ^= 1) {
        const int it = s_next[buf];
        if (it >= total) break;
        int next = 0;
        if (tid == 0) next = atomicAdd(counter + u, 1);
        const int4 w = items[it];
        const SlotDev &sd = tab[w.x];
        const SlotDyn d = dyn[w.w];
        const int pin = d.pair ^ (u & 1);  // pair (pair ^ u) -> the other pair
        batch_tile(sd.p, sd.cf, (const float *)sd.f[2 * pin], (const float *)sd.f[2 * pin + 1], (float *)sd.f[2 * (pin ^ 1)],
                   (float *)sd.f[2 * (pin ^ 1) + 1], sd.act, sd.nz, w.y, w.z, d.time + u + 1);
        if (tid == 0) s_next[buf ^ 1] = next;
        __syncthreads();  // the next ticket is visible; s_next[buf] is free again
    }
}

// FP64 items: strips of hdr->rows64 rows x ST_COLS columns (wg_step64.cuh), or 32 cells of the
// boundary lines (first row 0), one warp and one ticket each, in place within pair 0.  The scene's parameters are staged in the warp's shared
// memory.
__global__ void __launch_bounds__(128, 4) k_batch_step64(const BatchHdr *__restrict__ hdr, const SlotDev *__restrict__ tab,
                                                         const int4 *__restrict__ items, SlotDyn *__restrict__ dyn,
                                                         int *__restrict__ counter, int u, int all)
{
    __shared__ DevParams s_p[4];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    DevParams &p = s_p[wid];
    pdl_wait();  // launched by launch_pdl: the previous update has completed
    pdl_trigger();
    const int total = all ? hdr->total_tiles : hdr->plain_tiles;
    int next = 0;
    if (lane == 0) next = atomicAdd(counter + u, 1);
    for (;;) {
        const int it = __shfl_sync(0xffffffffu, next, 0);
        if (it >= total) break;  // warp-uniform
        if (lane == 0) next = atomicAdd(counter + u, 1);  // read after this item: its latency is hidden
        const int4 w = items[it];
        const SlotDev &sd = tab[w.x];
        __syncwarp();  // every lane is done with the previous item's parameters
        {
            const int *src = reinterpret_cast<const int *>(&sd.p);
            int *dst = reinterpret_cast<int *>(&p);
            for (int k = lane; k < (int)(sizeof(DevParams) / 4); k += 32) dst[k] = src[k];
        }
        __syncwarp();
        const SlotDyn d = dyn[w.w];
        const int phase = (d.cur + u) & 1;
        const Strip64 a{(const double *)sd.f[phase], (const double *)sd.f[1 - phase], (double *)sd.f[1 - phase], sd.act, sd.nz,
                        nullptr, nullptr, nullptr, nullptr, 0, 1};
        const int r1 = min(w.y + hdr->rows64, p.nx - 1);
        const long long t = d.time + u + 1;
        if (w.y == 0) {  // 32 boundary-line cells
            const int q = w.z * 32 + lane;
            if (q < edge64_cells(p)) edge64_cell<WG_COEF_MASK, false>(p, a, q, t);
            continue;
        }
        const int z = (p.kappa == 0.0 ? Z_KAPPA : 0) | (p.gam == 0.0 && p.gamb == 0.0 ? Z_GAMMA : 0);
        if (z == (Z_KAPPA | Z_GAMMA)) strip64<WG_COEF_MASK, false, Z_KAPPA | Z_GAMMA>(p, a, w.z * ST_COLS, w.y, r1, t);
        else if (z == Z_KAPPA) strip64<WG_COEF_MASK, false, Z_KAPPA>(p, a, w.z * ST_COLS, w.y, r1, t);
        else strip64<WG_COEF_MASK, false, 0>(p, a, w.z * ST_COLS, w.y, r1, t);
    }
}

// Ghost cells t0, t0 + nt, .. of one grid: each takes the value of the real cell it wraps to, in
// both fields (f1 may be NULL).  Ghost cells are written and real cells read, so blocks need no
// ordering.
__device__ __forceinline__ void ghost_fill(float *f0, float *f1, int nx, int ny, int pitch, long long t0, long long nt)
{
    constexpr int GC = BATCH_GHOST_COLS, GT = GC + BATCH_GHOST_COLS_R, GR = BATCH_GHOST_ROWS;
    const int wide = ny + GT, ncol = GT * nx;
    const long long total = ncol + 2LL * GR * wide;
    for (long long t = t0; t < total; t += nt) {
        int i, j;
        if (t < ncol) {  // the ghost columns of the real rows
            i = (int)t / GT;
            const int g = (int)t - i * GT;
            j = g < GC ? g - GC : ny + g - GC;
        } else {  // the ghost rows, over the extended width
            const long long u = t - ncol;
            const int rg = (int)(u / wide);
            j = (int)(u - (long long)rg * wide) - GC;
            i = rg < GR ? rg - GR : nx + rg - GR;
        }
        const int si = ((i % nx) + nx) % nx, sj = ((j % ny) + ny) % ny;
        const long long d = (long long)i * pitch + j, s = (long long)si * pitch + sj;
        f0[d] = f0[s];
        if (f1) f1[d] = f1[s];
    }
}

// Ghost cells of every wrapped scene's current pair, when its fields do not come from a skewed
// pass (which writes them beside its cells).  Block (x, y): table entry x, a share y of its
// ghost cells.
__global__ void k_batch_ghosts(const BatchHdr *__restrict__ hdr, const SlotDev *__restrict__ tab,
                               const SlotDyn *__restrict__ dyn)
{
    const int e = blockIdx.x;
    if (e >= hdr->nactive) return;
    const SlotDev &sd = tab[e];
    if (!sd.wrap) return;
    const int pair = dyn[sd.slot].pair;
    ghost_fill((float *)sd.f[2 * pair], (float *)sd.f[2 * pair + 1], sd.p.nx, sd.p.ny, sd.p.pitch,
               blockIdx.y * blockDim.x + threadIdx.x, gridDim.y * blockDim.x);
}

// The same of one grid (scenes).
__global__ void k_grid_ghosts(float *f0, float *f1, int nx, int ny, int pitch)
{
    ghost_fill(f0, f1, nx, ny, pitch, blockIdx.x * (long long)blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
}
void launch_grid_ghosts(float *f0, float *f1, int nx, int ny, int pitch, cudaStream_t st)
{
    const long long gt = BATCH_GHOST_COLS + BATCH_GHOST_COLS_R, total = gt * nx + 2LL * BATCH_GHOST_ROWS * (ny + gt);
    k_grid_ghosts<<<(unsigned)std::min(4LL * sm_count(), (total + 127) / 128), 128, 0, st>>>(f0, f1, nx, ny, pitch);
}

// The ghost words and rows of a wrapped scene's active plane: one thread per word of rows
// -BATCH_GHOST_ROWS..nx+BATCH_GHOST_ROWS-1, words -1..(ny+BATCH_GHOST_COLS-1)/32; a bit of a
// real cell keeps its value, a bit of a ghost cell takes the bit of the cell it wraps to.
__global__ void k_act_ghosts(uint32_t *act, int wpitch, int nx, int ny)
{
    constexpr int GC = BATCH_GHOST_COLS, GR = BATCH_GHOST_ROWS;
    const int w = (int)(blockIdx.x * blockDim.x + threadIdx.x) - 1;
    const int i = (int)blockIdx.y - GR;
    if (w > (ny + GC - 1) / 32 || i >= nx + GR) return;
    const bool real_row = i >= 0 && i < nx;
    if (real_row && w >= 0 && 32 * w + 31 < ny) return;  // all real cells
    const long long base = (long long)i * wpitch + w;
    uint32_t v = 0;
    for (int bit = 0; bit < 32; bit++) {
        const int j = 32 * w + bit;
        uint32_t x;
        if (real_row && j >= 0 && j < ny) {
            x = (act[base] >> bit) & 1u;
        } else if (j >= -GC && j < ny + GC) {
            const int si = ((i % nx) + nx) % nx, sj = ((j % ny) + ny) % ny;
            x = (act[(long long)si * wpitch + (sj >> 5)] >> (sj & 31)) & 1u;
        } else {
            x = 0;
        }
        v |= x << bit;
    }
    act[base] = v;
}
void launch_act_ghosts(uint32_t *act, int wpitch, int nx, int ny, cudaStream_t st)
{
    const int words = (ny + BATCH_GHOST_COLS + 31) / 32 + 1, rows = nx + 2 * BATCH_GHOST_ROWS;
    k_act_ghosts<<<dim3((words + 63) / 64, rows), 64, 0, st>>>(act, wpitch, nx, ny);
}

// The work items of the table's scenes, a thread each: (entry, first row, column tile, slot) in FP32,
// and in FP64 first the boundary lines' items (row 0 as their mark), then the interior's strips.
// (Built on the host and copied, up to 9000 items, they were a fifth of wg_batch_add:
// 178 us each for 40 FP64 scenes of 400x300, 149 so.)
__global__ void k_batch_items(const SlotDev *__restrict__ tab, int ntab, int total, int f64, int rows64, int4 *__restrict__ items)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    int lo = 0, hi = ntab - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tab[mid].tile_base <= t) lo = mid; else hi = mid - 1;
    }
    const SlotDev &d = tab[lo];
    const int edges = f64 ? (edge64_cells(d.p) + 31) / 32 : 0, q = t - d.tile_base, ti = (q - edges) / d.tiles_j;
    items[t] = q < edges ? make_int4(lo, 0, q, d.slot)
                         : make_int4(lo, f64 ? 1 + ti * rows64 : ti * BT_ROWS, q - edges - ti * d.tiles_j, d.slot);
}

// skewed: the frame ran the skewed passes of the scenes with a depth class.  pairs: FP32
// scenes, whose single updates also alternate between the pairs.
__global__ void k_batch_advance(const BatchHdr *__restrict__ hdr, const SlotDev *__restrict__ tab,
                                SlotDyn *__restrict__ dyn, int n, int skewed, int pairs)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= hdr->nactive) return;
    SlotDyn &d = dyn[tab[k].slot];
    d.time += n;
    const int P = skewed ? batch_passes(n, tab[k].skew_k) : 0;
    if (P > 0) d.pair ^= P & 1;
    else if (pairs) d.pair ^= n & 1;
    else d.cur = (d.cur + n) & 1;
}

}  // namespace wg

using namespace wg;

namespace wg {

static void batch_drop_graphs(wg_batch *b);

BatchLayout batch_layout(const wg_params &p, int prec)
{
    BatchLayout L;
    const int esz = prec == WG_FP32 ? 4 : 8;
    if (batch_wrap_ok(p, prec)) {  // ghost columns, ghost rows, one ghost mask word per row
        L.pitch = pitch_for(p.ny + 2 * BATCH_GHOST_COLS + 64, esz);
        const size_t rows = (size_t)p.nx + 2 * BATCH_GHOST_ROWS, wpitch = (L.pitch + 31) / 32;
        L.field_bytes = rows * L.pitch * esz;
        L.mask_bytes = rows * wpitch * 4;
        L.field_off = (size_t)BATCH_GHOST_ROWS * L.pitch + BATCH_GHOST_COLS;
        L.mask_off = (size_t)BATCH_GHOST_ROWS * wpitch + 1;
    } else {
        L.pitch = pitch_for(p.ny, esz);
        const size_t wpitch = (L.pitch + 31) / 32;
        L.field_bytes = (size_t)p.nx * L.pitch * esz;
        L.mask_bytes = (size_t)p.nx * wpitch * 4;
        L.field_off = L.mask_off = 0;
    }
    return L;
}

static int entry_skew_k(const wg_batch *b, const BatchSlotHost &h)
{
    if (!h.skew || b->skew_mode == 0) return 0;
    return b->skew_mode > 0 ? b->skew_mode : b->class_k[h.cls];
}

// the kernel form that covers every scene of a list: the masked one, or the general one
static int list_form(const std::vector<const BatchSlotHost *> &hs)
{
    int form = hs.empty() ? 0 : batch_skew_form(hs[0]->prm);
    for (const BatchSlotHost *h : hs)
        if (batch_skew_form(h->prm) != form) return 0;
    return form;
}

// Tasks of the pass depth d for the scenes of depth class K (table entries), largest first
// so that the ticket order balances the warps.  Row chunks: the rows tuned for the scene's
// size class, or (untuned, fixed depth) sized from the whole list's work, about two tasks
// per resident team, so that no single chunk outlasts the rest of the pass; the short top and
// bottom segments fill the end.  A list too small for that (chunks below 32 rows, where the fill
// costs more than the balance) gives each team about one chunk of at least 8 rows, since its time
// is that of a chunk: 6 grids of 500x400, 10 updates: 45.6 us in chunks of 32 rows, 39.1 so.
// force_rows > 0 overrides both.
static void build_skew_tasks(const wg_batch *b, const std::vector<const BatchSlotHost *> &hs,
                             const std::vector<int> &entries, int d, std::vector<int4> &out, int force_rows = 0)
{
    const int F = batch_skew_fill(d);
    double rows = 0.0;
    for (const BatchSlotHost *h : hs) rows += (double)batch_skew_tiles(h->dp, d) * (h->prm.nx + 3 * F);
    const int cap = std::max(1, batch_skew_capacity(d, list_form(hs)));
    const int chunk = rows >= 64.0 * cap ? std::min(4096, (int)(rows / (2.0 * cap)))
                                         : std::max(8, (int)(rows / cap));
    std::vector<int4> t;
    std::vector<float> cost;
    for (size_t k = 0; k < hs.size(); k++) {
        const int tuned = b->skew_mode < 0 ? b->class_rows[hs[k]->cls] : 0;
        batch_skew_plan(hs[k]->dp, entries[k], d, force_rows > 0 ? force_rows : (tuned > 0 ? tuned : chunk), t, cost);
    }
    std::vector<int> ord(t.size());
    for (size_t k = 0; k < ord.size(); k++) ord[k] = (int)k;
    std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return cost[x] > cost[y]; });
    out.resize(t.size());
    for (size_t k = 0; k < ord.size(); k++) out[k] = t[ord[k]];
}

// (re)build the task list of (depth class K, pass depth d) from the current table
static wg_status build_list(wg_batch *b, int K, int d, const std::vector<int> &tab_slot)
{
    auto it = b->lists.find({K, d});
    if (it == b->lists.end()) {
        if ((int)b->lists.size() >= b->skew_n_cap - 1) { set_error("too many skewed task lists"); return WG_ERR_STATE; }
        BatchSkewList L;
        L.index = (int)b->lists.size();
        it = b->lists.emplace(std::make_pair(K, d), L).first;
    }
    BatchSkewList &L = it->second;
    std::vector<const BatchSlotHost *> hs;
    std::vector<int> entries;
    for (size_t e = 0; e < tab_slot.size(); e++) {
        const BatchSlotHost &h = b->slots[tab_slot[e]];
        if (entry_skew_k(b, h) == K) {
            hs.push_back(&h);
            entries.push_back((int)e);
        }
    }
    std::vector<int4> tasks;
    build_skew_tasks(b, hs, entries, d, tasks);
    if ((int)tasks.size() > L.cap) {
        if (L.dev) cudaFree(L.dev);
        L.dev = nullptr;
        const int cap = std::max(1024, (int)tasks.size() * 2);
        WG_CUDA(cudaMalloc(&L.dev, sizeof(int4) * cap));
        L.cap = cap;
        batch_drop_graphs(b);  // the graphs hold the list pointer
    }
    const int form = list_form(hs);
    if (form != L.form) {  // the graphs hold the kernel
        L.form = form;
        batch_drop_graphs(b);
    }
    L.n = (int)tasks.size();
    if (L.n) WG_CUDA(cudaMemcpyAsync(L.dev, tasks.data(), sizeof(int4) * L.n, cudaMemcpyHostToDevice, b->st));
    WG_CUDA(cudaMemcpyAsync(b->d_skew_n + L.index, &L.n, sizeof(int), cudaMemcpyHostToDevice, b->st));
    WG_CUDA(cudaStreamSynchronize(b->st));  // the host vectors above go out of scope
    return WG_OK;
}

wg_status batch_refresh_table(wg_batch *b)
{
    constexpr int V = Vec<float>::n;
    std::vector<SlotDev> tab;
    std::vector<int> tab_slot;
    int base = 0, plain = 0, nskew = 0, nwrap = 0;
    long long cells = 0;
    unsigned sig = 0;
    // FP64: rows of a strip, about three items per resident warp
    int rows64 = BT_ROWS;
    if (b->prec == WG_FP64) {
        long long strip_rows = 0;
        for (const BatchSlotHost &h : b->slots)
            if (h.used) strip_rows += (long long)(h.prm.nx - 2) * ((h.prm.ny + ST_COLS - 1) / ST_COLS);
        const long long warps = 4LL * b->persistent_blocks;
        rows64 = (int)std::min(64LL, std::max(2LL, (strip_rows + 3 * warps - 1) / (3 * warps)));
    }
    // scenes without skewed passes first: their items are the first plain_tiles
    for (int pass = 0; pass < 2; pass++) {
        for (int k = 0; k < (int)b->slots.size(); k++) {
            const BatchSlotHost &h = b->slots[k];
            if (!h.used) continue;
            const int sk = entry_skew_k(b, h);
            if ((sk > 0) != (pass == 1)) continue;
            SlotDev d;
            memset(&d, 0, sizeof d);
            d.p = h.dp;
            for (int q = 0; q < 4; q++) d.f[q] = h.f[q];
            d.act = h.act;
            d.nz = h.nz;
            d.slot = k;
            {
                const double c[12] = {h.dp.c2, h.dp.c2b, h.dp.gam, h.dp.gamb, h.dp.kappa, h.dp.kappa_sides,
                                      h.dp.kappa_topbot, h.dp.gamma_sides, h.dp.gamma_topbot, h.dp.vmax,
                                      h.dp.courant, h.dp.courantb};
                for (int q = 0; q < 12; q++) d.cf[q] = (float)c[q];
            }
            d.skew_k = sk;
            d.wrap = h.wrap ? 1 : 0;
            // its items, as k_batch_items numbers them
            const bool f64 = b->prec == WG_FP64;
            d.tiles_j = f64 ? (h.prm.ny + ST_COLS - 1) / ST_COLS : (h.dp.pitch / V + BT_THREADS - 1) / BT_THREADS;
            const int first = f64 ? 1 : 0, step = f64 ? rows64 : BT_ROWS, tiles_i = (h.prm.nx - 2 * first + step - 1) / step;
            const int edges = f64 ? (edge64_cells(h.dp) + 31) / 32 : 0;
            d.ntiles = edges + tiles_i * d.tiles_j;
            d.tile_base = base;
            base += d.ntiles;
            cells += (long long)h.prm.nx * h.prm.ny;
            if (sk > 0) {
                sig |= 1u << sk;
                nskew++;
                if (h.wrap) nwrap++;
            } else {
                plain = base;
            }
            tab.push_back(d);
            tab_slot.push_back(k);
        }
    }
    if (plain > 0) sig |= 1u;
    if ((int)tab.size() > b->tab_cap) {
        if (b->d_tab) cudaFree(b->d_tab);
        b->d_tab = nullptr;
        const int cap = std::max(64, (int)tab.size() * 2);
        WG_CUDA(cudaMalloc(&b->d_tab, sizeof(SlotDev) * cap));
        b->tab_cap = cap;
        batch_drop_graphs(b);  // the graphs hold the table pointer and size the advance launch by it
    }
    if (base > b->items_cap) {
        if (b->d_items) cudaFree(b->d_items);
        b->d_items = nullptr;
        const int cap = std::max(1024, base * 2);
        WG_CUDA(cudaMalloc(&b->d_items, sizeof(int4) * cap));
        b->items_cap = cap;
        batch_drop_graphs(b);  // the graphs hold the item-table pointer
    }
    if (sig != b->graph_sig) {  // another set of branches: the graphs are recorded again
        batch_drop_graphs(b);
        b->graph_sig = sig;
    }
    if (!tab.empty()) {
        WG_CUDA(cudaMemcpyAsync(b->d_tab, tab.data(), sizeof(SlotDev) * tab.size(), cudaMemcpyHostToDevice, b->st));
        k_batch_items<<<(base + 255) / 256, 256, 0, b->st>>>(b->d_tab, (int)tab.size(), base, b->prec == WG_FP64, rows64, b->d_items);
        WG_CUDA(cudaGetLastError());
        b->launches++;
    }
    BatchHdr h{(int)tab.size(), base, plain, rows64};
    WG_CUDA(cudaMemcpyAsync(b->d_hdr, &h, sizeof h, cudaMemcpyHostToDevice, b->st));
    WG_CUDA(cudaStreamSynchronize(b->st));
    b->nactive = (int)tab.size();
    b->total_cells = cells;
    b->plain_tiles = plain;
    b->skew_scenes = nskew;
    b->wrap_scenes = nwrap;
    b->ghosts_ok = false;  // the table may hold new scenes, or scenes that took single updates
    b->tab_slot = tab_slot;
    // the task lists in use follow the new table
    std::vector<std::pair<int, int>> keys;
    for (auto &kv : b->lists) keys.push_back(kv.first);
    for (auto &key : keys) {
        wg_status st = build_list(b, key.first, key.second, tab_slot);
        if (st) return st;
    }
    return WG_OK;
}

static void batch_drop_graphs(wg_batch *b)
{
    for (auto &g : b->graphs) cudaGraphExecDestroy(g.second);
    b->graphs.clear();
}

// depth classes present in the table (bits 2..6 of graph_sig)
static std::vector<int> batch_groups(const wg_batch *b)
{
    std::vector<int> g;
    for (int K = 2; K <= WG_SKEW_MAX_K; K++)
        if (b->graph_sig & (1u << K)) g.push_back(K);
    return g;
}

// Everything a frame of n updates needs before it is recorded: counters, tickets, the
// task lists of its passes, the branches' streams and events, the kernels' attributes.
static wg_status batch_prepare_frame(wg_batch *b, int n, bool skewed)
{
    if (n > b->counter_cap) {
        if (b->d_counter) cudaFree(b->d_counter);
        b->d_counter = nullptr;
        WG_CUDA(cudaMalloc(&b->d_counter, sizeof(int) * n));
        b->counter_cap = n;
        batch_drop_graphs(b);
    }
    if (!skewed) return WG_OK;
    int tickets = 0;
    for (int K : batch_groups(b)) {
        const int P = batch_passes(n, K);
        tickets += P;
        for (int q = 0; q < P; q++) {
            const int d = batch_pass_depth(n, P, q);
            if (!b->lists.count({K, d})) {
                wg_status st = build_list(b, K, d, b->tab_slot);
                if (st) return st;
            }
            batch_skew_capacity(d, b->lists.at({K, d}).form);  // sets the kernel's shared-memory attribute outside the capture
        }
    }
    if (tickets > b->ticket_cap) {
        if (b->d_ticket) cudaFree(b->d_ticket);
        b->d_ticket = nullptr;
        const int cap = std::max(64, tickets * 2);
        WG_CUDA(cudaMalloc(&b->d_ticket, sizeof(int) * cap));
        b->ticket_cap = cap;
        batch_drop_graphs(b);
    }
    for (int K : batch_groups(b)) {
        if (!b->side[K]) WG_CUDA(cudaStreamCreateWithFlags(&b->side[K], cudaStreamNonBlocking));
        if (!b->ev_join[K]) WG_CUDA(cudaEventCreateWithFlags(&b->ev_join[K], cudaEventDisableTiming));
    }
    if (!b->ev_fork) WG_CUDA(cudaEventCreateWithFlags(&b->ev_fork, cudaEventDisableTiming));
    return WG_OK;
}

template <class T>
static void batch_enqueue_frame(wg_batch *b, int n, bool skewed)
{
    cudaMemsetAsync(b->d_counter, 0, sizeof(int) * n, b->st);
    std::vector<int> groups;
    if (skewed) {
        groups = batch_groups(b);
        int tickets = 0;
        for (int K : groups) tickets += batch_passes(n, K);
        cudaMemsetAsync(b->d_ticket, 0, sizeof(int) * tickets, b->st);
        cudaEventRecord(b->ev_fork, b->st);
        int ti = 0;
        for (int K : groups) {  // one branch per depth class
            cudaStream_t ss = b->side[K];
            cudaStreamWaitEvent(ss, b->ev_fork, 0);
            const int P = batch_passes(n, K);
            int toff = 0;
            for (int q = 0; q < P; q++) {
                const int d = batch_pass_depth(n, P, q);
                const BatchSkewList &L = b->lists.at({K, d});
                launch_batch_skew(d, L.form, b->d_tab, b->d_dyn, L.dev, b->d_skew_n + L.index, b->d_ticket + ti++, q, toff, ss);
                toff += d;
            }
            cudaEventRecord(b->ev_join[K], ss);
        }
    }
    if (!skewed || (b->graph_sig & 1u)) {  // the chain of single updates
        const bool f32 = sizeof(T) == 4;
        for (int u = 0; u < n; u++)
            launch_pdl(f32 ? k_batch_step32 : k_batch_step64, dim3(b->persistent_blocks),
                       f32 ? dim3(BT_THREADS, 4) : dim3(128), 0, b->st, (const BatchHdr *)b->d_hdr,
                       (const SlotDev *)b->d_tab, (const int4 *)b->d_items, b->d_dyn, b->d_counter, u, skewed ? 0 : 1);
    }
    for (int K : groups) cudaStreamWaitEvent(b->st, b->ev_join[K], 0);
    const int cap = std::max(b->tab_cap, 1);
    k_batch_advance<<<(cap + 255) / 256, 256, 0, b->st>>>(b->d_hdr, b->d_tab, b->d_dyn, n, skewed ? 1 : 0,
                                                          sizeof(T) == 4 ? 1 : 0);
}

// Depth and row chunk per size class, in two stages: depths 6..2 with the list-wide
// chunk, then chunks of 32, 64, 128 and 256 rows at the best depth.  Each candidate
// times one skewed pass over the class's scenes (reading their current fields, writing
// the other pair, so the state does not change), best of five after one untimed pass;
// the fastest per update is kept, a later candidate only if 5% faster (classes run side by
// side: timed alone, a shallower pass can look a little better and cost the frame 10%).  Nine
// candidates per class keep the tuning frame of a server tick short.
// Tuned classes are kept for the process, keyed by device, size class and the kinds of
// scene in the class (their boundary conditions, the ghost layout, two speeds): a later
// batch or server whose class holds the same kinds takes that depth and chunk without
// timing them again, so a serving tick pays the tuning of a size class at most once per
// process.  (Keyed by size class alone, the sweep's absorbing scenes took the depth tuned
// for the uneven batch's mirror and periodic ones: 309 against 351 Gcell/s.)
struct TuneCacheEntry {
    int k = 0, rows = 0;
    double ms[8] = {0, 0, 0, 0, 0, 0, 0, 0};
};
static std::mutex g_tune_mu;
static std::map<std::tuple<int, int, unsigned>, TuneCacheEntry> g_tune_cache;  // (device, class, kinds)

static unsigned class_kinds(const wg_batch *b, int c)
{
    unsigned sig = 0;
    for (size_t e = 0; e < b->tab_slot.size(); e++) {
        const BatchSlotHost &h = b->slots[b->tab_slot[e]];
        if (!(h.skew && h.cls == c)) continue;
        sig |= 1u << (h.prm.b_cond & 7);
        if (h.wrap) sig |= 1u << 8;
        if (h.prm.twospeeds) sig |= 1u << 9;
        if (h.prm.oscillate_left || h.prm.oscillate_topbot) sig |= 1u << 10;
        if (h.prm.src_on) sig |= 1u << 11;
        if (batch_skew_form(h.prm) == 0) sig |= 1u << 12;
    }
    return sig;
}

static wg_status batch_autotune(wg_batch *b)
{
    bool tuned = false, ghosts = false;
    int devno = 0;
    WG_CUDA(cudaGetDevice(&devno));
    for (int c = 0; c < BATCH_CLASSES; c++) {
        if (b->class_k[c]) continue;
        {
            std::lock_guard<std::mutex> lk(g_tune_mu);
            const unsigned kinds = class_kinds(b, c);
            if (!kinds) continue;  // no scene of this class takes skewed passes
            auto it = g_tune_cache.find(std::make_tuple(devno, c, kinds));
            if (it != g_tune_cache.end()) {
                if (b->tune_ms.empty()) b->tune_ms.assign(BATCH_CLASSES * 8, 0.0);
                b->class_k[c] = it->second.k;
                b->class_rows[c] = it->second.rows;
                for (int K = 0; K < 8; K++) b->tune_ms[c * 8 + K] = it->second.ms[K];
                tuned = true;
                continue;
            }
        }
        std::vector<const BatchSlotHost *> hs;
        std::vector<int> entries;
        for (size_t e = 0; e < b->tab_slot.size(); e++) {
            const BatchSlotHost &h = b->slots[b->tab_slot[e]];
            if (h.skew && h.cls == c) {
                hs.push_back(&h);
                entries.push_back((int)e);
            }
        }
        if (hs.empty()) continue;
        if (b->tune_ms.empty()) b->tune_ms.assign(BATCH_CLASSES * 8, 0.0);
        if (!ghosts) {  // the wrapped scenes' ghosts of their current pair, read by the timed passes
            k_batch_ghosts<<<dim3(std::max(b->nactive, 1), 8), 256, 0, b->st>>>(b->d_hdr, b->d_tab, b->d_dyn);
            b->launches++;
            ghosts = true;
        }
        cudaEvent_t ev[6];
        for (int q = 0; q < 6; q++) WG_CUDA(cudaEventCreate(&ev[q]));
        int best = 0, best_rows = 0;
        double best_ms = 1e30;
        int4 *dev = nullptr;
        cudaError_t err = cudaSuccess;
        static const int ROWS[] = {32, 64, 128, 256};
        const int ndepth = 5;  // depths 6..2
        for (int cand = 0; cand < ndepth + 4 && err == cudaSuccess; cand++) {
            const int K = cand < ndepth ? 6 - cand : best, R = cand < ndepth ? 0 : ROWS[cand - ndepth];
            std::vector<int4> tasks;
            build_skew_tasks(b, hs, entries, K, tasks, R);
            const int nt = (int)tasks.size();
            err = cudaMallocAsync((void **)&dev, sizeof(int4) * std::max(nt, 1), b->st);
            if (err == cudaSuccess && nt) err = cudaMemcpyAsync(dev, tasks.data(), sizeof(int4) * nt, cudaMemcpyHostToDevice, b->st);
            const int idx = b->skew_n_cap - 1;  // the count slot kept for tuning
            if (err == cudaSuccess) err = cudaMemcpyAsync(b->d_skew_n + idx, &nt, sizeof(int), cudaMemcpyHostToDevice, b->st);
            const int reps = 5;  // one untimed pass, then the best of five
            for (int r = 0; r <= reps && err == cudaSuccess; r++) {
                cudaMemsetAsync(b->d_tune_ticket + r, 0, sizeof(int), b->st);
                launch_batch_skew(K, list_form(hs), b->d_tab, b->d_dyn, dev, b->d_skew_n + idx, b->d_tune_ticket + r, 0, 0, b->st);
                b->launches++;
                err = cudaGetLastError();
                if (err == cudaSuccess) err = cudaEventRecord(ev[r], b->st);
            }
            if (err == cudaSuccess) err = cudaEventSynchronize(ev[reps]);
            float ms = 1e30f;
            for (int r = 1; r <= reps && err == cudaSuccess; r++) {
                float t = 0.f;
                err = cudaEventElapsedTime(&t, ev[r - 1], ev[r]);
                ms = std::min(ms, t);
            }
            if (dev) cudaFreeAsync(dev, b->st);
            dev = nullptr;
            if (err == cudaSuccess) err = cudaStreamSynchronize(b->st);  // tasks outlives its copy
            const double per = ms / K;
            if (R == 0 || per < b->tune_ms[c * 8 + K]) b->tune_ms[c * 8 + K] = per;
            if (per < 0.95 * best_ms) {
                best_ms = per;
                best = K;
                best_rows = R;
            }
        }
        for (int q = 0; q < 6; q++) cudaEventDestroy(ev[q]);
        if (err != cudaSuccess) return cuda_fail(err, "batch autotune");
        b->class_k[c] = best;
        b->class_rows[c] = best_rows;
        {
            std::lock_guard<std::mutex> lk(g_tune_mu);
            TuneCacheEntry &ce = g_tune_cache[std::make_tuple(devno, c, class_kinds(b, c))];
            ce.k = best;
            ce.rows = best_rows;
            for (int K = 0; K < 8; K++) ce.ms[K] = b->tune_ms[c * 8 + K];
        }
        tuned = true;
    }
    if (tuned) return batch_refresh_table(b);
    return WG_OK;
}

}  // namespace wg

extern "C" {

wg_status wg_batch_create(int32_t precision, void *stream, wg_batch **out)
{
    if (!out) { set_error("NULL argument"); return WG_ERR_INVALID; }
    if (precision != WG_FP32 && precision != WG_FP64) { set_error("precision must be WG_FP32 or WG_FP64"); return WG_ERR_INVALID; }
    wg_batch *b = new wg_batch();
    b->prec = precision;
    b->esz = precision == WG_FP32 ? 4 : 8;
    cudaError_t e = cudaSuccess;
    if (stream) b->st = (cudaStream_t)stream;
    else {
        e = cudaStreamCreateWithFlags(&b->st, cudaStreamNonBlocking);
        b->own_stream = true;
    }
    if (e == cudaSuccess) e = cudaMalloc(&b->d_hdr, sizeof(BatchHdr));
    if (e == cudaSuccess) e = cudaMemsetAsync(b->d_hdr, 0, sizeof(BatchHdr), b->st);
    int dev = 0, sms = 0, per = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = (precision == WG_FP32)
                ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_batch_step32, BT_THREADS * 4, 0)
                : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_batch_step64, 128, 0);
    if (e == cudaSuccess) e = cudaHostAlloc(&b->h_out, 16 * sizeof(double), cudaHostAllocDefault);
    b->skew_n_cap = 32;
    if (e == cudaSuccess) e = cudaMalloc(&b->d_skew_n, sizeof(int) * b->skew_n_cap);
    if (e == cudaSuccess) e = cudaMemsetAsync(b->d_skew_n, 0, sizeof(int) * b->skew_n_cap, b->st);
    if (e == cudaSuccess) e = cudaMalloc(&b->d_tune_ticket, sizeof(int) * 8);
    if (e != cudaSuccess) {
        wg_status r = cuda_fail(e, "wg_batch_create");
        wg_batch_destroy(b);
        return r;
    }
    b->persistent_blocks = std::max(1, sms * std::max(per, 1));
    *out = b;
    return WG_OK;
}

wg_status wg_batch_destroy(wg_batch *b)
{
    if (!b) return WG_OK;
    if (b->st) cudaStreamSynchronize(b->st);
    batch_drop_graphs(b);
    for (auto &h : b->slots) {
        if (!h.used) continue;
        void *ptrs[] = {h.mem[0], h.mem[1], h.mem[2], h.mem[3], h.act_mem, h.nz_mem, h.ebot, h.etop};
        for (void *p : ptrs) if (p) cudaFree(p);
    }
    for (auto &kv : b->lists) if (kv.second.dev) cudaFree(kv.second.dev);
    void *ptrs[] = {b->d_tab, b->d_dyn, b->d_hdr, b->d_counter, b->d_items, b->d_skew_n, b->d_ticket, b->d_tune_ticket};
    for (void *p : ptrs) if (p) cudaFree(p);
    for (int k = 0; k < BATCH_GROUPS; k++) {
        if (b->side[k]) cudaStreamDestroy(b->side[k]);
        if (b->ev_join[k]) cudaEventDestroy(b->ev_join[k]);
    }
    if (b->ev_fork) cudaEventDestroy(b->ev_fork);
    if (b->h_out) cudaFreeHost(b->h_out);
    if (b->own_stream && b->st) cudaStreamDestroy(b->st);
    delete b;
    return WG_OK;
}

wg_status wg_batch_add(wg_batch *b, const wg_params *p, const double *phi, const double *psi, const int16_t *xy,
                       int32_t *slot)
{
    if (!b || !p || !phi || !psi || !xy || !slot) { set_error("NULL argument"); return WG_ERR_INVALID; }
    wg_status st = validate_params(*p);
    if (st) return st;
    if (p->bc_neumann) { set_error("batches do not take Neumann records; use a scene"); return WG_ERR_INVALID; }
    const size_t n = (size_t)p->nx * p->ny;
    for (size_t c = 0; c < n; c++)
        if (xy[c] != 0 && xy[c] != 1) { set_error("batch masks take values 0/1"); return WG_ERR_INVALID; }
    int k = 0;
    while (k < (int)b->slots.size() && b->slots[k].used) k++;
    if (k == (int)b->slots.size()) b->slots.emplace_back();
    BatchSlotHost &h = b->slots[k];
    h = BatchSlotHost();
    h.prm = *p;
    h.skew = batch_skew_ok(*p, b->prec);
    h.wrap = batch_wrap_ok(*p, b->prec);
    const BatchLayout L = batch_layout(*p, b->prec);
    const int pitch = L.pitch;
    h.dp = make_dev_params(*p, pitch);
    {
        const double cells = (double)p->nx * p->ny;
        h.cls = std::min(BATCH_CLASSES - 1, std::max(0, (int)std::floor(std::log2(cells)) - 10));
    }
    const size_t fb = L.field_bytes, mb = L.mask_bytes;
    cudaError_t e = cudaSuccess;
    const int nf = b->prec == WG_FP32 ? 4 : 2;  // FP32: the second pair takes every update's output
    for (int q = 0; q < nf && e == cudaSuccess; q++) e = cudaMallocAsync(&h.mem[q], fb, b->st);
    for (int q = (h.wrap ? 0 : 2); q < nf && e == cudaSuccess; q++) e = cudaMemsetAsync(h.mem[q], 0, fb, b->st);
    if (e == cudaSuccess) e = cudaMallocAsync((void **)&h.act_mem, mb, b->st);
    if (e == cudaSuccess) e = cudaMallocAsync((void **)&h.nz_mem, mb, b->st);
    if (e == cudaSuccess && h.wrap) e = cudaMemsetAsync(h.act_mem, 0, mb, b->st);
    for (int q = 0; q < nf; q++) h.f[q] = h.mem[q] ? (char *)h.mem[q] + L.field_off * b->esz : nullptr;
    h.act = h.act_mem ? h.act_mem + L.mask_off : nullptr;
    h.nz = h.nz_mem ? h.nz_mem + L.mask_off : nullptr;
    if (e == cudaSuccess) e = cudaMallocAsync((void **)&h.ebot, p->nx * sizeof(double2), b->st);
    if (e == cudaSuccess) e = cudaMallocAsync((void **)&h.etop, p->nx * sizeof(double2), b->st);
    void *stage = nullptr;
    if (e == cudaSuccess) e = cudaMallocAsync(&stage, 2 * n * sizeof(double), b->st);
    if (e != cudaSuccess) {
        void *ptrs[] = {h.mem[0], h.mem[1], h.mem[2], h.mem[3], h.act_mem, h.nz_mem, h.ebot, h.etop, stage};
        for (void *q : ptrs) if (q) cudaFreeAsync(q, b->st);
        h = BatchSlotHost();
        return cuda_fail(e, "wg_batch_add");
    }
    h.bytes = nf * fb + 2 * mb;
    // mask planes, then the two fields (FP64 host values rounded on the device)
    WG_CUDA(cudaMemcpyAsync(stage, xy, n * sizeof(int16_t), cudaMemcpyHostToDevice, b->st));
    launch_pack_mask(p->nx, p->ny, h.dp.wpitch, (const int16_t *)stage, h.act, h.nz, b->st);
    if (h.wrap) {  // the mask's ghost words and rows, once (the mask does not change)
        launch_act_ghosts(h.act, h.dp.wpitch, p->nx, p->ny, b->st);
        b->launches++;
    }
    double *dstage = (double *)stage;
    WG_CUDA(cudaMemcpyAsync(dstage, phi, n * sizeof(double), cudaMemcpyHostToDevice, b->st));
    WG_CUDA(cudaMemcpyAsync(dstage + n, psi, n * sizeof(double), cudaMemcpyHostToDevice, b->st));
    if (b->prec == WG_FP32) {  // phi and the velocity phi - psi
        launch_state_in32<double>(p->nx, p->ny, pitch, dstage, dstage + n, (float *)h.f[0], (float *)h.f[1], b->st);
    } else {
        launch_convert_in<double>(p->nx, p->ny, pitch, dstage, (double *)h.f[0], b->st);
        launch_convert_in<double>(p->nx, p->ny, pitch, dstage + n, (double *)h.f[1], b->st);
    }
    WG_CUDA(cudaFreeAsync(stage, b->st));
    WG_CUDA(cudaGetLastError());
    // dynamic state: time 0, phi in f[0]
    if (k >= b->dyn_cap) {
        const int cap = std::max(64, 2 * (k + 1));
        SlotDyn *nd = nullptr;
        WG_CUDA(cudaMalloc(&nd, sizeof(SlotDyn) * cap));
        WG_CUDA(cudaMemsetAsync(nd, 0, sizeof(SlotDyn) * cap, b->st));
        if (b->d_dyn) {
            WG_CUDA(cudaMemcpyAsync(nd, b->d_dyn, sizeof(SlotDyn) * b->dyn_cap, cudaMemcpyDeviceToDevice, b->st));
            WG_CUDA(cudaStreamSynchronize(b->st));
            cudaFree(b->d_dyn);
        }
        b->d_dyn = nd;
        b->dyn_cap = cap;
        batch_drop_graphs(b);
    }
    SlotDyn zero{0, 0, 0};
    WG_CUDA(cudaMemcpyAsync(b->d_dyn + k, &zero, sizeof zero, cudaMemcpyHostToDevice, b->st));
    h.used = true;
    const int old_cap = b->tab_cap;
    if ((st = batch_refresh_table(b))) return st;
    if (b->tab_cap != old_cap) batch_drop_graphs(b);
    *slot = k;
    return WG_OK;
}

wg_status wg_batch_remove(wg_batch *b, int32_t slot)
{
    if (!b || slot < 0 || slot >= (int)b->slots.size() || !b->slots[slot].used) {
        set_error("unknown batch slot %d", slot);
        return WG_ERR_NOTFOUND;
    }
    BatchSlotHost &h = b->slots[slot];
    h.used = false;
    wg_status st = batch_refresh_table(b);  // the kernels stop seeing the slot first
    void *ptrs[] = {h.mem[0], h.mem[1], h.mem[2], h.mem[3], h.act_mem, h.nz_mem, h.ebot, h.etop};
    for (void *p : ptrs) if (p) WG_CUDA(cudaFreeAsync(p, b->st));
    h = BatchSlotHost();
    return st;
}

wg_status wg_batch_step(wg_batch *b, int32_t nsteps)
{
    if (!b || nsteps < 0) { set_error("bad arguments"); return WG_ERR_INVALID; }
    if (nsteps == 0 || b->nactive == 0) return WG_OK;
    wg_status st;
    if (b->prec == WG_FP32 && b->skew_mode < 0 && nsteps >= 2 && (st = batch_autotune(b))) return st;
    const bool skewed = b->prec == WG_FP32 && nsteps >= 2 && b->skew_scenes > 0;
    if ((st = batch_prepare_frame(b, nsteps, skewed))) return st;
    auto it = b->graphs.find(nsteps);
    if (it == b->graphs.end()) {
        cudaGraph_t g;
        WG_CUDA(cudaStreamBeginCapture(b->st, cudaStreamCaptureModeThreadLocal));
        if (b->prec == WG_FP32) batch_enqueue_frame<float>(b, nsteps, skewed);
        else batch_enqueue_frame<double>(b, nsteps, skewed);
        WG_CUDA(cudaStreamEndCapture(b->st, &g));
        cudaGraphExec_t ge;
        cudaError_t e = cudaGraphInstantiate(&ge, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGraphInstantiate");
        it = b->graphs.emplace(nsteps, ge).first;
    }
    if (skewed && b->wrap_scenes > 0 && !b->ghosts_ok) {
        k_batch_ghosts<<<dim3(b->nactive, 8), 256, 0, b->st>>>(b->d_hdr, b->d_tab, b->d_dyn);
        WG_CUDA(cudaGetLastError());
        b->launches++;
    }
    WG_CUDA(cudaGraphLaunch(it->second, b->st));
    b->ghosts_ok = skewed;  // (nsteps >= 2: every depth class takes at least one pass)
    long long n = 1;  // the advance kernel
    if (!skewed || (b->graph_sig & 1u)) n += nsteps;
    if (skewed)
        for (int K : batch_groups(b)) n += batch_passes(nsteps, K);
    b->launches += n;
    return WG_OK;
}

wg_status wg_batch_set_skew(wg_batch *b, int32_t mode)
{
    if (!b) { set_error("NULL batch"); return WG_ERR_INVALID; }
    if (!(mode == -1 || mode == 0 || (mode >= 2 && mode <= WG_SKEW_MAX_K))) {
        set_error("skewed depth %d: -1 (tuned per size class), 0 (off) or 2..%d", mode, WG_SKEW_MAX_K);
        return WG_ERR_INVALID;
    }
    WG_CUDA(cudaStreamSynchronize(b->st));
    b->skew_mode = mode;
    batch_drop_graphs(b);
    return batch_refresh_table(b);
}

wg_status wg_batch_skew_depths(wg_batch *b, int32_t *depths, int32_t *chunk_rows, double *ms_per_update)
{
    if (!b || !depths) { set_error("NULL argument"); return WG_ERR_INVALID; }
    for (int c = 0; c < BATCH_CLASSES; c++) {
        depths[c] = b->skew_mode >= 0 ? b->skew_mode : b->class_k[c];
        if (chunk_rows) chunk_rows[c] = b->skew_mode >= 0 ? 0 : b->class_rows[c];
        if (ms_per_update)
            for (int K = 0; K < 8; K++)
                ms_per_update[c * 8 + K] = b->tune_ms.empty() ? 0.0 : b->tune_ms[c * 8 + K];
    }
    return WG_OK;
}

wg_status wg_batch_download(wg_batch *b, int32_t slot, double *phi, double *psi)
{
    if (!b || slot < 0 || slot >= (int)b->slots.size() || !b->slots[slot].used) {
        set_error("unknown batch slot %d", slot);
        return WG_ERR_NOTFOUND;
    }
    BatchSlotHost &h = b->slots[slot];
    const size_t n = (size_t)h.prm.nx * h.prm.ny;
    // Page-locked rows are written in place, others through a stage; the kernel reads which
    // buffers are current, so that the call waits for the device once.  (With a copy of the slot's
    // state, a second wait and a stage each time: 1277x717 114 to 88 us, grids of 240x240 about
    // 41 to 14 us.)
    double *stage = nullptr, *ophi = phi, *opsi = psi;
    const size_t m = state_stage_cells(n);
    const bool mapped = mapped_rows(ophi, opsi, n);
    if (!mapped) {
        WG_CUDA(cudaMallocAsync((void **)&stage, 2 * m * sizeof(double), b->st));
        ophi = phi ? stage : nullptr;
        opsi = psi ? stage + m : nullptr;
    }
    if (b->prec == WG_FP32) {  // phi, and psi = phi - v
        const auto launch = mapped ? launch_state_out<float, double> : launch_state_stage<float, double>;
        launch(h.prm.nx, h.prm.ny, h.dp.pitch, (const float *)h.f[0], (const float *)h.f[1], (const float *)h.f[2],
               (const float *)h.f[3], &b->d_dyn[slot].pair, ophi, opsi, b->st);
    } else {
        const auto launch = mapped ? launch_state_out<double, double> : launch_state_stage<double, double>;
        launch(h.prm.nx, h.prm.ny, h.dp.pitch, (const double *)h.f[0], (const double *)h.f[1], (const double *)h.f[1],
               (const double *)h.f[0], &b->d_dyn[slot].cur, ophi, opsi, b->st);
    }
    if (!mapped) {
        if (phi) WG_CUDA(cudaMemcpyAsync(phi, stage, n * sizeof(double), cudaMemcpyDeviceToHost, b->st));
        if (psi) WG_CUDA(cudaMemcpyAsync(psi, stage + m, n * sizeof(double), cudaMemcpyDeviceToHost, b->st));
        WG_CUDA(cudaFreeAsync(stage, b->st));
    }
    WG_CUDA(cudaGetLastError());
    WG_CUDA(cudaStreamSynchronize(b->st));
    return WG_OK;
}

wg_status wg_batch_energy(wg_batch *b, int32_t slot, double *total)
{
    if (!b || !total || slot < 0 || slot >= (int)b->slots.size() || !b->slots[slot].used) {
        set_error("unknown batch slot %d", slot);
        return WG_ERR_NOTFOUND;
    }
    BatchSlotHost &h = b->slots[slot];
    SlotDyn d;
    WG_CUDA(cudaMemcpyAsync(&d, b->d_dyn + slot, sizeof d, cudaMemcpyDeviceToHost, b->st));
    WG_CUDA(cudaStreamSynchronize(b->st));
    // FP32: phi and the velocity of the current pair; FP64: phi and psi of pair 0
    const void *phi = h.f[2 * d.pair + d.cur], *psi = h.f[2 * d.pair + 1 - d.cur];
    if (b->prec == WG_FP32)
        launch_energy<float>(h.dp, (const float *)phi, (const float *)psi, nullptr, h.nz, h.ebot, h.etop, 0, 0, b->h_out, 0,
                             nullptr, nullptr, b->st);
    else
        launch_energy<double>(h.dp, (const double *)phi, (const double *)psi, nullptr, h.nz, h.ebot, h.etop, 0, 0, b->h_out, 0,
                             nullptr, nullptr, b->st);
    b->launches += 2;
    WG_CUDA(cudaGetLastError());
    WG_CUDA(cudaStreamSynchronize(b->st));
    *total = b->h_out[0];
    return WG_OK;
}

wg_status wg_batch_count(wg_batch *b, int32_t *n_active, int64_t *cells)
{
    if (!b) return WG_ERR_INVALID;
    if (n_active) *n_active = b->nactive;
    if (cells) *cells = b->total_cells;
    return WG_OK;
}

wg_status wg_batch_launch_count(wg_batch *b, int64_t *n)
{
    if (!b || !n) return WG_ERR_INVALID;
    *n = b->launches;
    return WG_OK;
}

}  // extern "C"
