// 2D TMz stepping entirely on chip: one thread-block cluster holds a whole small grid in distributed shared
// memory and runs every step of a tfd_step call without touching HBM between steps.
//
// What bounds it is instruction issue and the two barriers of a step (0.64 us): one lane per cell with the x neighbours by
// shuffle issued 6.2 warp-instructions per cell on 16 SMs and took 7.4 us per step at 320 x 240 cells.
//
// A 320 x 240 TMz grid is about 1.4 MB of fields, inverse permittivity and CPML memories: more than one CTA's
// shared memory, less than a cluster's (8 or 16 CTAs of up to 227 KB on a B200). Each CTA of the cluster owns a
// band of rows [r0, r1) and keeps Ez, Hx, Hy, 1/eps and the CPML memories of its rows in its own shared memory.
// A step is
//   E phase: Ez of every own cell from Hy (same row) and Hx (row y - 1: the CTA below for the first row, read
//            through distributed shared memory), the E-family CPML memories, the E soft sources;
//   cluster barrier;
//   H phase: Hx from Ez (row y + 1: the CTA above for the last row), Hy from Ez (x + 1), the H-family memories,
//            the H soft sources, then the point traces of the step (the owning CTA writes them to HBM);
//   cluster barrier.
// A thread takes 4 consecutive cells of a row (2 in FP64) with 16-byte shared-memory loads; groups that meet an x slab are
// walked after the others, so that a warp runs the x memories or does not: 320 x 240 cells, FP32, 5.4 us per step against
// 7.4 with one cell per thread (2000 steps through the public call 10.8 against 15.9 ms). Each phase
// reads only the other family, so the updates are in place. The arithmetic per cell is that of
// the strip kernels' general path (step2d.cuh: strip_general), so the fields are bitwise the same. The state
// is loaded from the parity the step counter names at the start of the launch and written back, with the
// counter, at the end. Scope: 2D TMz plans without DFT planes (the traces are the only observations).
#pragma once
#include <cooperative_groups.h>

#include "internal.cuh"
#include "step_pass.cuh"

namespace tfd {

namespace cg = cooperative_groups;

constexpr int kCl2dThreads = 1024;               // at most; a launch takes as many as share the groups of a band evenly
constexpr int kCl2dMaxRanks = 16;

struct Cluster2D {
    int ranks;                       // CTAs in the cluster
    int r0[kCl2dMaxRanks + 1];       // band of rank c: rows [r0[c], r0[c + 1])
    int rows_max;                    // the largest band
    int w;                           // shared-memory row width: nx rounded up to a whole group
    int threads;
    PassSplit split[2];              // a row's groups clear of the x slabs of each family, and the others
    int h;                           // rows of the grid (ny): length of the per-row coefficient tables
    int rx_e, rx_h;                  // x-slab memory widths (rows of both x slabs) of the E and H families
    int rye_lo[kCl2dMaxRanks], rye_n[kCl2dMaxRanks];   // per rank: first y-slab memory row of its band, count (E)
    int ryh_lo[kCl2dMaxRanks], ryh_n[kCl2dMaxRanks];   // the same for the H family
    int rye_max, ryh_max;
    int count;                       // steps of this launch
};

// Shared-memory arrays of one rank, at element offsets fixed by the launch (every rank uses the same layout, so
// a neighbour's row sits at the same offset in its shared memory). After the fields and memories: per family f
// and axis a (x: nx entries, y: ny entries) the CPML coefficients b, c, 1/kappa and the metric factor of each
// column / row (tab), and the memory row of each column / row (-1: no CPML term there; slab).
struct Cl2dLayout {
    int ez, hx, hy, ie, pex, pey, phx, phy;
    int tab[2][2];                   // 4 consecutive T arrays (b, c, k, metric) of n[a] entries
    int slab[2][2];                  // int arrays, element offsets from the start of the int region
    int ints;                        // start of the int region (in T elements)
    int total;                       // T elements including the int region
};

__host__ __device__ inline Cl2dLayout cl2d_layout(const Cluster2D &c, int tsize) {
    Cl2dLayout L;
    const int cells = c.rows_max * c.w, align = 16 / tsize;
    auto up = [&](int n) { return (n + align - 1) / align * align; };   // arrays start on 16 bytes
    L.ez = 0;
    L.hx = L.ez + cells;
    L.hy = L.hx + cells;
    L.ie = L.hy + cells;
    L.pey = L.ie + cells;
    L.phy = L.pey + c.rye_max * c.w;
    L.pex = L.phy + c.ryh_max * c.w;
    L.phx = up(L.pex + c.rows_max * c.rx_e);
    int o = up(L.phx + c.rows_max * c.rx_h);
    int io = 0;
    for (int f = 0; f < 2; ++f)
        for (int a = 0; a < 2; ++a) {
            const int n = a == 0 ? c.w : up(c.h);
            L.tab[f][a] = o;
            o += 4 * n;
            L.slab[f][a] = io;
            io += n;
        }
    L.ints = o;
    L.total = o + (io * 4 + tsize - 1) / tsize;
    return L;
}

template <typename T>
__global__ void __launch_bounds__(kCl2dThreads, 1) k_step2d_cluster(const __grid_constant__ Grid<T> g, const __grid_constant__ Cluster2D c,
                                                                   const TraceDev *__restrict__ traces, int n_traces, T *trace_out) {
    extern __shared__ __align__(16) unsigned char cl_raw[];
    T *const sm = reinterpret_cast<T *>(cl_raw);
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const Cl2dLayout L = cl2d_layout(c, (int)sizeof(T));
    const int nx = g.n[0], ny = g.n[1], W = c.w, pitch = g.pitch;
    const int r0 = c.r0[rank], r1 = c.r0[rank + 1], rows = r1 - r0;
    const int tid = threadIdx.x, threads = blockDim.x, hcol = L.tab[0][1] - L.tab[0][0] >> 2, hrow = L.tab[1][0] - L.tab[0][1] >> 2;
    const long long n0 = *g.counter;
    const int par0 = (int)(n0 & 1);
    T *Ez = sm + L.ez, *Hx = sm + L.hx, *Hy = sm + L.hy, *ie = sm + L.ie;
    T *pex = sm + L.pex, *pey = sm + L.pey, *phx = sm + L.phx, *phy = sm + L.phy;
    int *const ints = reinterpret_cast<int *>(sm + L.ints);
    // The neighbours' bands: the last Hx row of the rank below, the first Ez row of the rank above.
    const T *hx_below = rank > 0 ? cluster.map_shared_rank(sm + L.hx, rank - 1) : nullptr;
    const T *ez_above = rank + 1 < c.ranks ? cluster.map_shared_rank(sm + L.ez, rank + 1) : nullptr;
    const int rows_below = rank > 0 ? c.r0[rank] - c.r0[rank - 1] : 0;
    const int RxE = g.rows[0][0], RxH = g.rows[1][0];

    // Load the band (parity par0) and its CPML memories.
    for (int q = tid; q < rows * W; q += threads) {
        const int y = r0 + q / W, x = q % W;
        const bool in = x < nx;                           // the row's padding stays zero (see step_pass.cuh)
        const long long i = (long long)y * pitch + x;
        Ez[q] = in ? g.E[par0][2][i] : T(0);
        Hx[q] = in ? g.H[par0][0][i] : T(0);
        Hy[q] = in ? g.H[par0][1][i] : T(0);
        ie[q] = in ? g.cn * g.inv_eps[2][i] : T(0);     // the update's factor (cn / eps)
    }
    if (RxE) for (int q = tid; q < rows * RxE; q += threads) pex[q] = g.psiE[par0][0][1][(long long)(r0 + q / RxE) * RxE + q % RxE];
    if (RxH) for (int q = tid; q < rows * RxH; q += threads) phx[q] = g.psiH[0][0][(long long)(r0 + q / RxH) * RxH + q % RxH];
    for (int q = tid; q < c.rye_n[rank] * W; q += threads) pey[q] = q % W < nx ? g.psiE[par0][1][1][(long long)(c.rye_lo[rank] + q / W) * pitch + q % W] : T(0);
    for (int q = tid; q < c.ryh_n[rank] * W; q += threads) phy[q] = q % W < nx ? g.psiH[1][0][(long long)(c.ryh_lo[rank] + q / W) * pitch + q % W] : T(0);
    // Coefficient tables. A column / row whose difference the update does not take (E: x = 0, y = 0; H: the last
    // column / row) gets no memory row, so the tables alone decide where CPML terms apply.
    for (int f = 0; f < 2; ++f)
        for (int a = 0; a < 2; ++a) {
            const int len = a == 0 ? nx : ny, room = a == 0 ? hcol : hrow;
            T *tb = sm + L.tab[f][a];
            int *ts = ints + L.slab[f][a];
            const int *rowp = g.row[f][a];
            const T *m = g.metric[f][a];
            for (int i = tid; i < room; i += threads) {
                const bool diff = i < len && (f == 0 ? i > 0 : i < len - 1);
                const int r = (rowp != nullptr && diff) ? rowp[i] : -1;
                ts[i] = r;
                tb[i] = r >= 0 ? g.cb[f][a][i] : T(0);
                tb[room + i] = r >= 0 ? g.cc[f][a][i] : T(0);
                tb[2 * room + i] = r >= 0 ? g.ck[f][a][i] : T(1);
                tb[3 * room + i] = m != nullptr && i < len ? m[i] : T(1);
            }
        }
    // Sources that meet the band (E: its rows; H: its rows), tested once.
    unsigned src_e = 0, src_hx = 0, src_hy = 0;
    for (int t = 0; t < g.n_src; ++t) {
        const SourceTerm &s = g.src[t];
        const bool hit = s.lo[1] < r1 && r0 < s.hi[1];
        if (s.family == 0 && s.comp == 2 && hit) src_e |= 1u << t;
        if (s.family == 1 && s.comp == 0 && hit) src_hx |= 1u << t;
        if (s.family == 1 && s.comp == 1 && hit) src_hy |= 1u << t;
    }
    bool band_traces = false;
    for (int t = 0; t < n_traces; ++t) {
        const int y = (int)(traces[t].offset / pitch);
        band_traces |= y >= r0 && y < r1;
    }
    // Soft sources of a group, one source after the other (ascending index, the order of the strip kernels). Thread t
    // loads term t one step ahead, the barriers in between publish it (a source mask has 32 bits: at most 32 terms).
    __shared__ T src_val[2][32];
    const unsigned src_any = src_e | src_hx | src_hy;
    constexpr int N = Pack<T>::N;
    auto add_sources = [&](unsigned mask, int which, int x, int y, Pack<T> &f) {
        for (; mask; mask &= mask - 1) {
            const int t = __ffs(mask) - 1;
            const SourceTerm &s = g.src[t];
            if (y < s.lo[1] || y >= s.hi[1] || x >= s.hi[0] || x + N <= s.lo[0]) continue;
            const T v = src_val[which][t];
#pragma unroll
            for (int k = 0; k < N; ++k)
                if (x + k >= s.lo[0] && x + k < s.hi[0]) f.v[k] = f.v[k] + v;
        }
    };
    const bool pec_x = g.pec_on[0] != 0, pec_y = g.pec_on[1] != 0;
    const T pneg_x = g.pec_neg[0], pneg_y = g.pec_neg[1], cn = g.cn;
    const bool m_e = g.metric[0][0] != nullptr || g.metric[0][1] != nullptr, m_h = g.metric[1][0] != nullptr || g.metric[1][1] != nullptr;
    const T *const xb_e = sm + L.tab[0][0], *const yb_e = sm + L.tab[0][1];
    const T *const xb_h = sm + L.tab[1][0], *const yb_h = sm + L.tab[1][1];
    const int *const xs_e = ints + L.slab[0][0], *const ys_e = ints + L.slab[0][1];
    const int *const xs_h = ints + L.slab[1][0], *const ys_h = ints + L.slab[1][1];
    // Group q of the band in the order of a family's split: its row and first column.
    auto group_at = [&](const PassSplit &sp, int q, int &yl, int &x) -> bool {
        const int plain = sp.plain * rows;
        int xg;
        const bool slab = q >= plain;
        if (!slab) {
            yl = pass_divide((unsigned)q, (unsigned)sp.plain, sp.magic_plain, xg);
            xg += sp.x_lo;
        } else {
            yl = pass_divide((unsigned)(q - plain), (unsigned)sp.slab, sp.magic_slab, xg);
            if (xg >= sp.x_lo) xg += sp.plain;
        }
        x = xg * N;
        return slab;
    };
    const int groups = (c.split[0].plain + c.split[0].slab) * rows;
    // Point traces: a thread keeps the band-local index of its trace (-1: another band's cell) and the field.
    int tr_e = -1, tr_f = 0;
    if (tid < n_traces) {
        const TraceDev tr = traces[tid];
        const int y = (int)(tr.offset / pitch), x = (int)(tr.offset % pitch);
        if (y >= r0 && y < r1) tr_e = (y - r0) * W + x;
        tr_f = (tr.family == 0 && tr.comp == 2) ? 1 : (tr.family == 1 && tr.comp == 0) ? 2 : (tr.family == 1 && tr.comp == 1) ? 3 : 0;
    }
    long long n = n0;
    if (tid < 32 && ((src_any >> tid) & 1u) && n0 < g.steps) src_val[n0 & 1][tid] = g.src_values[(long long)tid * g.steps + n0];
    cluster.sync();                                       // every band, table and source value loaded before it is read

    for (int k = 0; k < c.count && n < g.steps; ++k, ++n) {
        // The next step's source values, into the other buffer: their latency overlaps this step, its barriers publish them.
        if (tid < 32 && ((src_any >> tid) & 1u) && n + 1 < g.steps) src_val[(n + 1) & 1][tid] = g.src_values[(long long)tid * g.steps + n + 1];
        const int sv = (int)(n & 1);
        // ---- E pass ----
        for (int q = tid; q < groups; q += threads) {
            int yl, x;
            const bool slab = group_at(c.split[0], q, yl, x);
            const int y = r0 + yl, e = yl * W + x;
            const Pack<T> hy = pack_load(Hy + e), hx = pack_load(Hx + e), f = pack_load(ie + e);
            const T left = x > 0 ? Hy[e - 1] : T(0);
            // Hx of the row below: this band's row, the band below (DSMEM), or none at y = 0.
            Pack<T> low{};
            if (yl > 0) low = pack_load(Hx + e - W);
            else if (hx_below != nullptr) low = pack_load(hx_below + (rows_below - 1) * W + x);
            Pack<T> ez = pack_load(Ez + e);
            T dx[N], dy[N];
#pragma unroll
            for (int i = 0; i < N; ++i) {
                dx[i] = hy.v[i] - (i == 0 ? left : hy.v[i == 0 ? 0 : i - 1]);
                dy[i] = hx.v[i] - low.v[i];
            }
            if (x == 0) dx[0] = T(0);
            if (y == 0)
#pragma unroll
                for (int i = 0; i < N; ++i) dy[i] = T(0);
            if (m_e) {
                const T my = yb_e[3 * hrow + y];
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    dx[i] = dx[i] * xb_e[3 * hcol + x + i];
                    dy[i] = dy[i] * my;
                }
            }
            if (slab)
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    const int r = xs_e[x + i];
                    if (r < 0) continue;
                    T *p = pex + yl * RxE + r;
                    const T mem = *p * xb_e[x + i] + xb_e[hcol + x + i] * dx[i];
                    *p = mem;
                    dx[i] = dx[i] * xb_e[2 * hcol + x + i] + mem;
                }
            const int rye = ys_e[y];
            if (rye >= 0) {
                T *p = pey + (rye - c.rye_lo[rank]) * W + x;
                const T b = yb_e[y], cc = yb_e[hrow + y], ck = yb_e[2 * hrow + y];
                Pack<T> mem = pack_load(p);
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    mem.v[i] = mem.v[i] * b + cc * dy[i];
                    dy[i] = dy[i] * ck + mem.v[i];
                }
                pack_store(p, mem);
            }
#pragma unroll
            for (int i = 0; i < N; ++i) {
                T acc = T(0) + dx[i];
                acc = acc + (-dy[i]);
                ez.v[i] = ez.v[i] + f.v[i] * acc;         // the padding's factor is zero ...
            }
            if (x + N > nx)
#pragma unroll
                for (int i = 0; i < N; ++i)
                    if (x + i >= nx) ez.v[i] = T(0);      // ... and its value, whatever its neighbour holds
            if (src_e) add_sources(src_e, sv, x, y, ez);
            pack_store(Ez + e, ez);
        }
        cluster.sync();
        // ---- H pass ----
        for (int q = tid; q < groups; q += threads) {
            int yl, x;
            const bool slab = group_at(c.split[1], q, yl, x);
            const int h = r0 + yl, e = yl * W + x;
            const Pack<T> ez = pack_load(Ez + e);
            const T right = x + N < nx ? Ez[e + N] : T(0);
            // Ez of the row above: this band's row, the band above (DSMEM); none above the last grid row.
            Pack<T> high{};
            if (yl + 1 < rows) high = pack_load(Ez + e + W);
            else if (ez_above != nullptr) high = pack_load(ez_above + x);
            Pack<T> hx = pack_load(Hx + e), hy = pack_load(Hy + e);
            T dx[N], dy[N];
#pragma unroll
            for (int i = 0; i < N; ++i) {
                dx[i] = (i == N - 1 ? right : ez.v[i == N - 1 ? i : i + 1]) - ez.v[i];
                dy[i] = high.v[i] - ez.v[i];
            }
            if (m_h) {
                const T my = yb_h[3 * hrow + h];
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    dx[i] = dx[i] * xb_h[3 * hcol + x + i];
                    dy[i] = dy[i] * my;
                }
            }
            if (x + N >= nx)                              // the row's last cell: the PEC ghost or 0
#pragma unroll
                for (int i = 0; i < N; ++i)
                    if (x + i >= nx - 1) dx[i] = (pec_x && x + i == nx - 1) ? pneg_x * ez.v[i] : T(0);
            if (h == ny - 1)
#pragma unroll
                for (int i = 0; i < N; ++i) dy[i] = pec_y ? pneg_y * ez.v[i] : T(0);
            if (slab)
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    const int r = xs_h[x + i];
                    if (r < 0) continue;
                    T *p = phx + yl * RxH + r;
                    const T mem = *p * xb_h[x + i] + xb_h[hcol + x + i] * dx[i];
                    *p = mem;
                    dx[i] = dx[i] * xb_h[2 * hcol + x + i] + mem;
                }
            const int ryh = ys_h[h];
            if (ryh >= 0) {
                T *p = phy + (ryh - c.ryh_lo[rank]) * W + x;
                const T b = yb_h[h], cc = yb_h[hrow + h], ck = yb_h[2 * hrow + h];
                Pack<T> mem = pack_load(p);
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    mem.v[i] = mem.v[i] * b + cc * dy[i];
                    dy[i] = dy[i] * ck + mem.v[i];
                }
                pack_store(p, mem);
            }
#pragma unroll
            for (int i = 0; i < N; ++i) {
                hx.v[i] = hx.v[i] - cn * (T(0) + dy[i]);
                hy.v[i] = hy.v[i] - cn * (T(0) + (-dx[i]));
            }
            if (src_hx) add_sources(src_hx, sv, x, h, hx);
            if (src_hy) add_sources(src_hy, sv, x, h, hy);
            pack_store(Hx + e, hx);
            pack_store(Hy + e, hy);
        }
        if (band_traces) {
            // Point traces of step n sampled by the rank that owns the cell (a CTA-uniform branch).
            __syncthreads();
            if (tid < n_traces && tr_e >= 0) {
                const T v = tr_f == 1 ? Ez[tr_e] : tr_f == 2 ? Hx[tr_e] : tr_f == 3 ? Hy[tr_e] : T(0);
                trace_out[n * n_traces + tid] = v;
            }
            for (int t = tid + threads; t < n_traces; t += threads) {
                const TraceDev tr = traces[t];
                const int y = (int)(tr.offset / pitch), x = (int)(tr.offset % pitch);
                if (y < r0 || y >= r1) continue;
                const int e = (y - r0) * W + x;
                T v = T(0);
                if (tr.family == 0 && tr.comp == 2) v = Ez[e];
                else if (tr.family == 1 && tr.comp == 0) v = Hx[e];
                else if (tr.family == 1 && tr.comp == 1) v = Hy[e];
                trace_out[n * n_traces + t] = v;
            }
        }
        cluster.sync();
    }
    // Write the band back at the parity of the step count reached, and the counter.
    const int par = (int)(n & 1);
    for (int q = tid; q < rows * W; q += threads) {
        const int y = r0 + q / W, x = q % W;
        if (x >= nx) continue;
        const long long i = (long long)y * pitch + x;
        g.E[par][2][i] = Ez[q];
        g.H[par][0][i] = Hx[q];
        g.H[par][1][i] = Hy[q];
    }
    if (RxE) for (int q = tid; q < rows * RxE; q += threads) g.psiE[par][0][1][(long long)(r0 + q / RxE) * RxE + q % RxE] = pex[q];
    if (RxH) for (int q = tid; q < rows * RxH; q += threads) g.psiH[0][0][(long long)(r0 + q / RxH) * RxH + q % RxH] = phx[q];
    for (int q = tid; q < c.rye_n[rank] * W; q += threads) if (q % W < nx) g.psiE[par][1][1][(long long)(c.rye_lo[rank] + q / W) * pitch + q % W] = pey[q];
    for (int q = tid; q < c.ryh_n[rank] * W; q += threads) if (q % W < nx) g.psiH[1][0][(long long)(c.ryh_lo[rank] + q / W) * pitch + q % W] = phy[q];
    if (rank == 0 && tid == 0) *g.counter = n;
    cluster.sync();                                       // no rank leaves while a neighbour may still read it
}

}  // namespace tfd
