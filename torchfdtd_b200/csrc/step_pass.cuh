// Two-pass step: an E pass and an H pass over the grid, one thread per 16-byte group of cells of a row.
//
// Runs every plan the 2D strip kernels do not take (2D TE and mixed polarizations, periodic 2D grids, TFSF boxes,
// dispersive materials, 3D grids except the largest, see two_pass_3d in api.cu) and is selectable as kernel 'gather'
// for all of them. The E pass computes E_new of its group from the old H and E (and writes the E-family CPML memories);
// the H pass reads E_new back, so no value is recomputed and nothing waits for a neighbour.
//
// Every input of a group is a load of its own, independent of the others: the H rows at y and y - 1, the planes z
// and z - 1, E and 1/eps as 16-byte vectors, the x - 1 value as one scalar, all issued before the first use. What bounds
// it on large grids is DRAM: 76 bytes per cell and step in FP32 (E pass: H, E, 1/eps read, E written; H pass: E, H read,
// H written; 5.1 GB per step at 512 x 512 x 256 cells, and 0.4 GB of CPML memories) in 0.96-0.99 ms (5.5-5.7 TB/s, 86-88 % of the copy rate). The H
// pass walks the planes in the opposite order of the E pass and starts on the E values that the E pass left in L2.
// At 256^3 cells: 0.276-0.281 ms per step against 0.336 ms for the fused marching kernel (its halo recomputation and
// per-row paths issue 11 warp-instructions per cell, these two passes 6.2) and 0.665 ms for one thread per cell with a
// TFSF box. Not kept: the H pass trailing the E pass slab by slab in one launch, or in alternating launches, so that L2
// serves the second reads (1.02-1.4 ms and 1.1-1.7 ms at 512 x 512 x 256: signalling and launch tails cost more than
// the traffic saved).
//
// Arithmetic in the reference operation order (torchfdtd/boundaries.py:363-438, torchfdtd/cuda_kernels.py:186-259,
// 327-347): d = F[i] - F[i-1]; times the metric factor of the updated cell on a nonuniform mesh (periodic wrap
// included, PEC ghost excluded); psi = psi*b + c*d; d = d*(1/kappa) + psi; curl = (0 + s0*d0) + s1*d1;
// E += (cn*inv_eps)*curl; dispersive samples corrected; soft sources added; H -= cn*curl; soft sources added.
//
// Cells of a row's padding (x >= nx) are stored as zero: their inputs are zero and stay so.
#pragma once
#include <cooperative_groups.h>

#include "aux.cuh"
#include "internal.cuh"
#include "persist2d.cuh"

namespace tfd {

constexpr int kPassThreads = 256;
// Blocks per SM: 80 registers in FP32 (the slab path spills; at 128 and two blocks 512 x 512 x 256 cells took 10 % longer),
// 128 in FP64.
template <typename T> constexpr int kPassBlocks = sizeof(T) == 4 ? 3 : 2;

// Groups of a row: those that meet no x slab (`plain` of them from x_lo on) and those that do (the first x_lo and the last
// ones). A plane's groups are walked plain ones first, then the slab ones, so that a warp holds one kind: with both in a
// warp the slab path ran for every warp of a 256-cell row (786 instructions per warp and pass, 256^3 cells: 488 against
// 290 us per step).
struct PassSplit { int plain, x_lo, slab; unsigned magic_plain, magic_slab, plain_total, total; };

// Where the steps of a replay leave what their transposes read: H and the E-family CPML memories after each step, in the
// restart-snapshot layout (element offsets from the slot's start). base: the slot after the launch's first step.
template <typename T>
struct PassSnap {
    T *base;                     // nullptr: no replay
    long long stride;            // elements between slots
    long long sH[3], sPsiE[3][2];
};

template <typename T>
struct PassArgs {
    Grid<T> g;
    int slab[2][3][4];           // per family and axis: lo0, hi0, lo1, hi1 of the two CPML slabs
    int tables;                  // 1: more than two slabs on some axis, slab rows come from the row tables
    PassSplit split[2];          // per family
    // k_pass_steps (PassShape in api.cu): chunks of blockDim.x groups, numbered through the planes (magic_total divides a group's
    // number by split[].total); rotate: CTAs that the chunks move on by from sweep to sweep.
    unsigned chunks, magic_total, rotate;
    PassSnap<T> snap;
};

template <typename T> struct alignas(16) Pack { static constexpr int N = 16 / sizeof(T); T v[N]; };

__device__ __forceinline__ Pack<float> pack_load(const float *p) {
    const float4 q = *reinterpret_cast<const float4 *>(p);
    return Pack<float>{{q.x, q.y, q.z, q.w}};
}
__device__ __forceinline__ Pack<double> pack_load(const double *p) {
    const double2 q = *reinterpret_cast<const double2 *>(p);
    return Pack<double>{{q.x, q.y}};
}
__device__ __forceinline__ void pack_store(float *p, const Pack<float> &q) {
    *reinterpret_cast<float4 *>(p) = make_float4(q.v[0], q.v[1], q.v[2], q.v[3]);
}
__device__ __forceinline__ void pack_store(double *p, const Pack<double> &q) {
    *reinterpret_cast<double2 *>(p) = make_double2(q.v[0], q.v[1]);
}

// Slab row of coordinate c on axis a (family f), or -1.
template <typename T>
__device__ __forceinline__ int pass_row(const PassArgs<T> &A, int f, int a, int c) {
    if (A.tables) return A.g.row[f][a] != nullptr ? A.g.row[f][a][c] : -1;
    const int *b = A.slab[f][a];
    return (c >= b[0] && c < b[1]) ? c - b[0] : (c >= b[2] && c < b[3]) ? (b[1] - b[0]) + (c - b[2]) : -1;
}

// One group: its cells [x, x + N) of row (y, z), the element index of the first one. I: int where the component
// arrays and CPML memories stay below 2^31 elements (one multiply-add per address), else long long.
template <typename I>
struct PassCell { int x, y, z; I i; };

// The x-slab memories of a group (both terms) and their coefficients, each cell in its own slab row (row[k] < 0: none).
// Loaded before anything is stored: a load after a store may alias it for the compiler, which would put the round
// trips of the 2 N memories in a row.
template <typename T, typename I>
struct PassSlab {
    static constexpr int N = Pack<T>::N;
    I at;
    int row[N];
    T old[2][N], b[N], c[N], k[N];
};

template <typename T, int F, typename I>
__device__ __forceinline__ void slab_load(const PassArgs<T> &A, const PassCell<I> &q, const T *old0, const T *old1, PassSlab<T, I> &m) {
    constexpr int N = Pack<T>::N;
    const Grid<T> &g = A.g;
    m.at = ((I)q.z * g.n[1] + q.y) * g.rows[F][0];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const int c = q.x + k;
        m.row[k] = c < g.n[0] ? pass_row(A, F, 0, c) : -1;
        m.old[0][k] = m.old[1][k] = m.b[k] = m.c[k] = m.k[k] = T(0);
        if (m.row[k] >= 0) {
            if (old0 != nullptr) m.old[0][k] = old0[m.at + m.row[k]];
            if (old1 != nullptr) m.old[1][k] = old1[m.at + m.row[k]];
            m.b[k] = g.cb[F][0][c];
            m.c[k] = g.cc[F][0][c];
            m.k[k] = g.ck[F][0][c];
        }
    }
}

// psi <- b psi + c d (stored to out, and to the replay's slot); d <- d/kappa + psi, for term j of the x axis.
template <typename T, typename I>
__device__ __forceinline__ void slab_apply(const PassSlab<T, I> &m, int j, T *out, T *snap, T (&d)[Pack<T>::N]) {
#pragma unroll
    for (int k = 0; k < Pack<T>::N; ++k)
        if (m.row[k] >= 0) {
            const T v = m.old[j][k] * m.b[k] + m.c[k] * d[k];
            out[m.at + m.row[k]] = v;
            if (snap != nullptr) snap[m.at + m.row[k]] = v;
            d[k] = d[k] * m.k[k] + v;
        }
}

// The same for a y or z slab row r >= 0 (axis a) of a group: one memory vector per term.
template <typename T, int F, int a, typename I>
__device__ __forceinline__ void pass_cpml(const PassArgs<T> &A, const PassCell<I> &q, int r, const T *old, T *out, T *snap, T (&d)[Pack<T>::N]) {
    const Grid<T> &g = A.g;
    const int c = a == 1 ? q.y : q.z;
    const I p = a == 1 ? ((I)q.z * g.rows[F][1] + r) * g.pitch + q.x : ((I)r * g.n[1] + q.y) * g.pitch + q.x;
    const T b = g.cb[F][a][c], cc = g.cc[F][a][c], ck = g.ck[F][a][c];
    Pack<T> m = pack_load(old + p);
#pragma unroll
    for (int k = 0; k < Pack<T>::N; ++k) {
        m.v[k] = m.v[k] * b + cc * d[k];
        d[k] = d[k] * ck + m.v[k];
    }
    pack_store(out + p, m);
    if (snap != nullptr) pack_store(snap + p, m);
}

// The cell of an element index of a component array. A plane of a 2D grid may hold 2^31 elements and more.
struct CellAt { int x, y, z; };
__host__ __device__ constexpr CellAt cell_at(long long i, long long plane, int pitch) {
    const long long rest = i % plane;
    const int z = (int)(i / plane);
    if (rest < (1LL << 31)) return CellAt{(int)rest % pitch, (int)rest / pitch, z};       // a fraction of the 64-bit division
    return CellAt{(int)(rest % pitch), (int)(rest / pitch), z};
}
static_assert(cell_at(65000LL * 65536 + 7, 65536LL * 65536, 65536).y == 65000 && cell_at(65000LL * 65536 + 7, 65536LL * 65536, 65536).x == 7,
              "element indices of large planes");

// Dispersive samples (threads j of total): the coupled trapezoidal ADE turns the free update that the E pass stored into
// E_new and advances the pole states, then the soft sources of the cell are added (the E pass leaves dispersive samples
// to this sweep). Reference operation order (torchfdtd/materials.py:67-88).
//
// A sweep of its own, one thread per sample in memory order, because the samples are a small share of the cells but touch
// most warps: inside the E pass every warp that held one sample ran the whole correction for it (201 x 187 x 163 cells,
// 1.2 M samples: 306 us per step, 164 with this sweep).
template <typename T>
__device__ __forceinline__ void pass_ade(const Grid<T> &g, int j, int par, long long n) {
    const long long at = g.ade_at[j];
    const int c = at >= 2 * g.count ? 2 : at >= g.count ? 1 : 0;
    const long long i = at - c * g.count;
    const T old = g.E[par][c][i], free = g.E[par ^ 1][c][i];
    int s = 0;
    while (s + 1 < g.n_ade && j >= g.ade[s + 1].start) ++s;
    const AdeDev<T> &st = g.ade[s];
    const int l = j - st.start, ns = st.samples;
    T e;
    if (st.poles == 1) {
        const T P = st.P[l], Q = st.Q[l];
        const T response = (Q - st.a[0] * P) / st.d[0];
        e = (st.eps * free - st.ksum * old - response) / st.denom;
        const T delta = response + st.k[0] * (e + old);
        st.P[l] = P + delta;
        st.Q[l] = -Q + T(2) * delta;
    } else {
        auto response = [&](int p) -> T { return (st.Q[p * ns + l] - st.a[p] * st.P[p * ns + l]) / st.d[p]; };
        T total = response(0);
        for (int p = 1; p < st.poles; ++p) total = total + response(p);
        e = (st.eps * free - st.ksum * old - total) / st.denom;
        for (int p = 0; p < st.poles; ++p) {
            const T delta = response(p) + st.k[p] * (e + old);
            st.P[p * ns + l] = st.P[p * ns + l] + delta;
            st.Q[p * ns + l] = -st.Q[p * ns + l] + T(2) * delta;
        }
    }
    if (g.n_src > 0) {
        const CellAt cell = cell_at(i, g.plane, g.pitch);
        for (int t = 0; t < g.n_src; ++t) {
            const SourceTerm &q = g.src[t];
            if (q.family == 0 && q.comp == c && cell.x >= q.lo[0] && cell.x < q.hi[0] && cell.y >= q.lo[1] && cell.y < q.hi[1] &&
                cell.z >= q.lo[2] && cell.z < q.hi[2])
                e = e + g.src_values[(long long)t * g.steps + n];
        }
    }
    g.E[par ^ 1][c][i] = e;
}

template <typename T>
__global__ void __launch_bounds__(kPassThreads) k_pass_ade(const __grid_constant__ Grid<T> g, int samples) {
    const long long n = *g.counter;
    if (n >= g.steps) return;
    const int j = blockIdx.x * kPassThreads + threadIdx.x;
    if (j < samples) pass_ade(g, j, (int)(n & 1), n);
}

// Soft sources of a family over a group, one term after the other (ascending index). ADE: dispersive samples are left out.
template <typename T, bool ADE, typename I>
__device__ __forceinline__ void pass_sources(const Grid<T> &g, int family, long long n, const PassCell<I> &q, Pack<T> (&f)[3]) {
    constexpr int N = Pack<T>::N;
    for (int s = 0; s < g.n_src; ++s) {
        const SourceTerm &t = g.src[s];
        if (t.family != family || q.z < t.lo[2] || q.z >= t.hi[2] || q.y < t.lo[1] || q.y >= t.hi[1] || q.x >= t.hi[0] || q.x + N <= t.lo[0])
            continue;
        const T v = g.src_values[(long long)s * g.steps + n];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int k = 0; k < N; ++k)
                if (t.comp == c && q.x + k >= t.lo[0] && q.x + k < t.hi[0] && !(ADE && g.ade_map[c][q.i + k] >= 0)) f[c].v[k] = f[c].v[k] + v;
    }
}

// E_new of a group. ACTIVE: bitmask of advanced components (bit c: E_c, bit 3+c: H_c). XS: the group meets an x slab.
template <typename T, int ACTIVE, bool METRIC, bool ADE, bool XS, typename I>
__device__ __forceinline__ void pass_e(const PassArgs<T> &A, const PassCell<I> &q, int par, long long n, T *slot) {
    constexpr int N = Pack<T>::N;
    const Grid<T> &g = A.g;
    constexpr bool HX = ACTIVE & 8, HY = ACTIVE & 16, HZ = ACTIVE & 32;
    constexpr bool EX = ACTIVE & 1, EY = ACTIVE & 2, EZ = ACTIVE & 4;
    const I i = q.i, plane = (I)g.plane;
    // The -1 neighbours: one period away at a periodic face, the cell itself (unused) at another one.
    const bool xin = q.x > 0 || g.periodic[0], yin = q.y > 0 || g.periodic[1], zin = q.z > 0 || g.periodic[2];
    const I ix = q.x > 0 ? i - 1 : i + (g.periodic[0] ? g.n[0] - 1 : 0);
    const I iy = q.y > 0 ? i - g.pitch : i + (g.periodic[1] ? (I)(g.n[1] - 1) * g.pitch : 0);
    const I iz = q.z > 0 ? i - plane : i + (g.periodic[2] ? (I)(g.n[2] - 1) * plane : 0);
    const T *Hx = g.H[par][0], *Hy = g.H[par][1], *Hz = g.H[par][2];
    Pack<T> hx{}, hy{}, hz{}, hx_y{}, hz_y{}, hx_z{}, hy_z{}, eo[3], ie[3];
    T hy_x = T(0), hz_x = T(0);
    if (HX) hx = pack_load(Hx + i);
    if (HY) hy = pack_load(Hy + i);
    if (HZ) hz = pack_load(Hz + i);
    if (EZ && HX) hx_y = pack_load(Hx + iy);
    if (EX && HZ) hz_y = pack_load(Hz + iy);
    if (EY && HX) hx_z = pack_load(Hx + iz);
    if (EX && HY) hy_z = pack_load(Hy + iz);
    if (EZ && HY) hy_x = Hy[ix];
    if (EY && HZ) hz_x = Hz[ix];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        eo[c] = Pack<T>{};
        ie[c] = Pack<T>{};
        if ((ACTIVE >> c) & 1) {
            eo[c] = pack_load(g.E[par][c] + i);
            if (c == 0 || !((ACTIVE >> 0) & 1) || g.inv_eps[c] != g.inv_eps[0]) ie[c] = pack_load(g.inv_eps[c] + i);
            else ie[c] = ie[0];
        }
    }
    PassSlab<T, I> sx;
    if (XS) slab_load<T, 0>(A, q, g.psiE[par][0][0], g.psiE[par][0][1], sx);
    const int ry = pass_row(A, 0, 1, q.y), rz = pass_row(A, 0, 2, q.z);
    // A row with a missing neighbour or a slab memory leaves the plain difference by one branch per term.
    const bool ycold = !yin || ry >= 0, zcold = !zin || rz >= 0;
    // Metric factors of the updated cells (1 on a uniform axis).
    T mx[N], my = T(1), mz = T(1);
    if (METRIC) {
#pragma unroll
        for (int k = 0; k < N; ++k) mx[k] = g.metric[0][0] != nullptr ? g.metric[0][0][min(q.x + k, g.n[0] - 1)] : T(1);
        if (g.metric[0][1] != nullptr) my = g.metric[0][1][q.y];
        if (g.metric[0][2] != nullptr) mz = g.metric[0][2][q.z];
    }
    auto dx = [&](const Pack<T> &h, T left, int j, T (&d)[N]) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            d[k] = h.v[k] - (k == 0 ? left : h.v[k == 0 ? 0 : k - 1]);
            if (k == 0 && !xin) d[k] = T(0);
            if (METRIC) d[k] = d[k] * mx[k];
        }
        if (XS) slab_apply(sx, j, g.psiE[par ^ 1][0][j], slot ? slot + A.snap.sPsiE[0][j] : nullptr, d);
    };
    auto dy = [&](const Pack<T> &h, const Pack<T> &low, int j, T (&d)[N]) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            d[k] = h.v[k] - low.v[k];
            if (METRIC) d[k] = d[k] * my;
        }
        if (ycold) {
            if (!yin)
#pragma unroll
                for (int k = 0; k < N; ++k) d[k] = T(0);
            if (ry >= 0) pass_cpml<T, 0, 1>(A, q, ry, g.psiE[par][1][j], g.psiE[par ^ 1][1][j], slot ? slot + A.snap.sPsiE[1][j] : nullptr, d);
        }
    };
    auto dz = [&](const Pack<T> &h, const Pack<T> &low, int j, T (&d)[N]) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            d[k] = h.v[k] - low.v[k];
            if (METRIC) d[k] = d[k] * mz;
        }
        if (zcold) {
            if (!zin)
#pragma unroll
                for (int k = 0; k < N; ++k) d[k] = T(0);
            if (rz >= 0) pass_cpml<T, 0, 2>(A, q, rz, g.psiE[par][2][j], g.psiE[par ^ 1][2][j], slot ? slot + A.snap.sPsiE[2][j] : nullptr, d);
        }
    };
    T d0[N], d1[N];
    Pack<T> e[3];
    auto update = [&](int c, bool neg0, bool neg1) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const T acc = (T(0) + (neg0 ? -d0[k] : d0[k])) + (neg1 ? -d1[k] : d1[k]);
            e[c].v[k] = eo[c].v[k] + (g.cn * ie[c].v[k]) * acc;
        }
    };
    if (EX) {
        dy(hz, hz_y, 0, d0);
        dz(hy, hy_z, 0, d1);
        update(0, false, true);
    }
    if (EY) {
        dx(hz, hz_x, 0, d0);
        dz(hx, hx_z, 1, d1);
        update(1, true, false);
    }
    if (EZ) {
        dx(hy, hy_x, 1, d0);
        dy(hx, hx_y, 1, d1);
        update(2, false, true);
    }
    if (ADE && g.ade_map[0] != nullptr) pass_sources<T, true>(g, 0, n, q, e);
    else pass_sources<T, false>(g, 0, n, q, e);
    const bool tail = q.x + N > g.n[0];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        if (!((ACTIVE >> c) & 1)) continue;
        if (tail)
#pragma unroll
            for (int k = 0; k < N; ++k)
                if (q.x + k >= g.n[0]) e[c].v[k] = T(0);
        pack_store(g.E[par ^ 1][c] + i, e[c]);
    }
}

// H_new of a group from the stored E_new.
template <typename T, int ACTIVE, bool METRIC, bool XS, typename I>
__device__ __forceinline__ void pass_h(const PassArgs<T> &A, const PassCell<I> &q, int par, long long n, T *slot) {
    constexpr int N = Pack<T>::N;
    const Grid<T> &g = A.g;
    constexpr bool HX = ACTIVE & 8, HY = ACTIVE & 16, HZ = ACTIVE & 32;
    constexpr bool EX = ACTIVE & 1, EY = ACTIVE & 2, EZ = ACTIVE & 4;
    const I i = q.i, plane = (I)g.plane;
    const int nx = g.n[0];
    const bool last = q.x + N >= nx;                     // the group holds the row's last cell
    const bool yin = q.y < g.n[1] - 1, zin = q.z < g.n[2] - 1;
    const I ix = last ? i - q.x : i + N;                 // the row's first cell: the neighbour at a periodic face
    const I iy = yin ? i + g.pitch : i - (g.periodic[1] ? (I)(g.n[1] - 1) * g.pitch : 0);
    const I iz = zin ? i + plane : i - (g.periodic[2] ? (I)(g.n[2] - 1) * plane : 0);
    const T *Ex = g.E[par ^ 1][0], *Ey = g.E[par ^ 1][1], *Ez = g.E[par ^ 1][2];
    Pack<T> ex{}, ey{}, ez{}, ex_y{}, ez_y{}, ex_z{}, ey_z{}, ho[3];
    T ey_x = T(0), ez_x = T(0);
    if (EX) ex = pack_load(Ex + i);
    if (EY) ey = pack_load(Ey + i);
    if (EZ) ez = pack_load(Ez + i);
    if (HZ && EX) ex_y = pack_load(Ex + iy);
    if (HX && EZ) ez_y = pack_load(Ez + iy);
    if (HY && EX) ex_z = pack_load(Ex + iz);
    if (HX && EY) ey_z = pack_load(Ey + iz);
    if (HZ && EY) ey_x = Ey[ix];
    if (HY && EZ) ez_x = Ez[ix];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        ho[c] = Pack<T>{};
        if ((ACTIVE >> (3 + c)) & 1) ho[c] = pack_load(g.H[par][c] + i);
    }
    PassSlab<T, I> sx;
    if (XS) slab_load<T, 1>(A, q, g.psiH[0][0], g.psiH[0][1], sx);
    const int ry = pass_row(A, 1, 1, q.y), rz = pass_row(A, 1, 2, q.z);
    // A row with a missing neighbour or a slab memory leaves the plain difference by one branch per term.
    const bool ycold = !yin || ry >= 0, zcold = !zin || rz >= 0;
    T mx[N], my = T(1), mz = T(1);
    if (METRIC) {
#pragma unroll
        for (int k = 0; k < N; ++k) mx[k] = g.metric[1][0] != nullptr ? g.metric[1][0][min(q.x + k, nx - 1)] : T(1);
        if (g.metric[1][1] != nullptr) my = g.metric[1][1][q.y];
        if (g.metric[1][2] != nullptr) mz = g.metric[1][2][q.z];
    }
    auto dx = [&](const Pack<T> &f, T right, int j, T (&d)[N]) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            d[k] = (k == N - 1 ? right : f.v[k == N - 1 ? k : k + 1]) - f.v[k];
            if (METRIC) d[k] = d[k] * mx[k];
        }
        if (last)
#pragma unroll
            for (int k = 0; k < N; ++k)
                if (q.x + k == nx - 1) {
                    d[k] = g.periodic[0] ? right - f.v[k] : (g.pec_on[0] ? g.pec_neg[0] * f.v[k] : T(0));
                    if (METRIC && g.periodic[0]) d[k] = d[k] * mx[k];
                }
        if (XS) slab_apply(sx, j, g.psiH[0][j], (T *)nullptr, d);
    };
    auto edge = [&](int a, const Pack<T> &f, T (&d)[N]) {       // no +1 neighbour and no period: the PEC ghost, or 0
#pragma unroll
        for (int k = 0; k < N; ++k) d[k] = g.pec_on[a] ? g.pec_neg[a] * f.v[k] : T(0);
    };
    auto dy = [&](const Pack<T> &f, const Pack<T> &high, int j, T (&d)[N]) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            d[k] = high.v[k] - f.v[k];
            if (METRIC) d[k] = d[k] * my;
        }
        if (ycold) {
            if (!yin && !g.periodic[1]) edge(1, f, d);
            if (ry >= 0) pass_cpml<T, 1, 1>(A, q, ry, g.psiH[1][j], g.psiH[1][j], (T *)nullptr, d);
        }
    };
    auto dz = [&](const Pack<T> &f, const Pack<T> &high, int j, T (&d)[N]) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            d[k] = high.v[k] - f.v[k];
            if (METRIC) d[k] = d[k] * mz;
        }
        if (zcold) {
            if (!zin && !g.periodic[2]) edge(2, f, d);
            if (rz >= 0) pass_cpml<T, 1, 2>(A, q, rz, g.psiH[2][j], g.psiH[2][j], (T *)nullptr, d);
        }
    };
    T d0[N], d1[N];
    Pack<T> h[3];
    auto update = [&](int c, bool neg0, bool neg1) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const T acc = (T(0) + (neg0 ? -d0[k] : d0[k])) + (neg1 ? -d1[k] : d1[k]);
            h[c].v[k] = ho[c].v[k] - g.cn * acc;
        }
    };
    if (HX) {
        dy(ez, ez_y, 0, d0);
        dz(ey, ey_z, 0, d1);
        update(0, false, true);
    }
    if (HY) {
        dx(ez, ez_x, 0, d0);
        dz(ex, ex_z, 1, d1);
        update(1, true, false);
    }
    if (HZ) {
        dx(ey, ey_x, 1, d0);
        dy(ex, ex_y, 1, d1);
        update(2, false, true);
    }
    pass_sources<T, false>(g, 1, n, q, h);
    const bool tail = q.x + N > nx;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        if (!((ACTIVE >> (3 + c)) & 1)) continue;
        if (tail)
#pragma unroll
            for (int k = 0; k < N; ++k)
                if (q.x + k >= nx) h[c].v[k] = T(0);
        pack_store(g.H[par ^ 1][c] + i, h[c]);
        if (slot != nullptr) pack_store(slot + A.snap.sH[c] + i, h[c]);
    }
}

// p / d and the remainder. m: ceil(2^32 / d) (the largest value for d = 1); the quotient it gives is at most one off
// (its error is below p / 2^32).
__device__ __forceinline__ int pass_divide(unsigned p, unsigned d, unsigned m, int &rest) {
    int y = (int)__umulhi(p, m);
    rest = (int)(p - (unsigned)y * d);
    if (rest < 0) {
        --y;
        rest += (int)d;
    } else if (rest >= (int)d) {
        ++y;
        rest -= (int)d;
    }
    return y;
}

// Group p of plane z in the order of a split; slab: whether it meets an x slab.
template <typename I, typename T>
__device__ __forceinline__ PassCell<I> pass_cell(const Grid<T> &g, const PassSplit &s, unsigned p, int z, bool slab) {
    PassCell<I> q;
    int xg;
    if (!slab) {
        q.y = pass_divide(p, (unsigned)s.plain, s.magic_plain, xg);
        xg += s.x_lo;
    } else {
        q.y = pass_divide(p - s.plain_total, (unsigned)s.slab, s.magic_slab, xg);
        if (xg >= s.x_lo) xg += s.plain;
    }
    q.x = xg * Pack<T>::N;
    q.z = z;
    q.i = (I)z * (I)g.plane + (I)q.y * g.pitch + q.x;
    return q;
}

// Group p of plane z in each pass.
template <typename T, int ACTIVE, bool METRIC, bool ADE, typename I>
__device__ __forceinline__ void pass_block_e(const PassArgs<T> &A, unsigned p, int z, int par, long long n, T *slot) {
    if (p >= A.split[0].total) return;
    const bool slab = p >= A.split[0].plain_total;
    const PassCell<I> q = pass_cell<I>(A.g, A.split[0], p, z, slab);
    if (slab) pass_e<T, ACTIVE, METRIC, ADE, true>(A, q, par, n, slot);
    else pass_e<T, ACTIVE, METRIC, ADE, false>(A, q, par, n, slot);
}

template <typename T, int ACTIVE, bool METRIC, typename I>
__device__ __forceinline__ void pass_block_h(const PassArgs<T> &A, unsigned p, int z, int par, long long n, T *slot) {
    if (p >= A.split[1].total) return;
    const bool slab = p >= A.split[1].plain_total;
    const PassCell<I> q = pass_cell<I>(A.g, A.split[1], p, z, slab);
    if (slab) pass_h<T, ACTIVE, METRIC, true>(A, q, par, n, slot);
    else pass_h<T, ACTIVE, METRIC, false>(A, q, par, n, slot);
}

// One launch per pass: blocks of kPassThreads groups of one plane (blockIdx.x), planes on
// blockIdx.y, ascending in the E pass, descending in the H pass.
template <typename T, int ACTIVE, bool METRIC, bool ADE, typename I>
__global__ void __launch_bounds__(kPassThreads, kPassBlocks<T>) k_pass_e(const __grid_constant__ PassArgs<T> A) {
    const long long n = *A.g.counter;
    if (n >= A.g.steps) return;                 // past the plan's last step: a step is a no-op
    for (int z = blockIdx.y; z < A.g.n[2]; z += gridDim.y)
        pass_block_e<T, ACTIVE, METRIC, ADE, I>(A, blockIdx.x * kPassThreads + threadIdx.x, z, (int)(n & 1), n, A.snap.base);
}

// end: nothing follows in the step but point traces, which the block that finishes last records before it advances the step
// counter. A third launch costs about 1 us on small grids (captured TE steps, 400 x 400 cells: 10.8 us with it, 9.8 without; single
// steps 12.5 and 11.7); with many blocks their fences cost more than that (1000 x 1000: 16.9 and 17.7), see pass_ends_step in api.cu.
template <typename T, int ACTIVE, bool METRIC, typename I>
__global__ void __launch_bounds__(kPassThreads, kPassBlocks<T>) k_pass_h(const __grid_constant__ PassArgs<T> A,
                                                                        const __grid_constant__ MonitorArgs<T> m, int end) {
    const long long n = *A.g.counter;
    if (n >= A.g.steps) return;
    for (int z = A.g.n[2] - 1 - (int)blockIdx.y; z >= 0; z -= gridDim.y)
        pass_block_h<T, ACTIVE, METRIC, I>(A, blockIdx.x * kPassThreads + threadIdx.x, z, (int)(n & 1), n, A.snap.base);
    if (!end) return;
    __shared__ int is_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        is_last = atomicAdd(m.done, 1u) == gridDim.x * gridDim.y - 1;
        __threadfence();
    }
    __syncthreads();
    if (!is_last) return;
    const long long shift = ((n + 1) & 1) ? m.count : 0;
    for (int k = threadIdx.x; k < m.n_traces; k += kPassThreads) {
        const TraceDev t = m.traces[k];
        const T *base = m.field[3 * t.family + t.comp];
        m.trace_out[n * m.n_traces + k] = base ? __ldcg(base + shift + t.offset) : T(0);
    }
    if (threadIdx.x == 0) {
        *m.done = 0;
        *A.g.counter = n + 1;
    }
}

// The step counter alone (a replayed step records no observations).
template <typename T>
__global__ void k_pass_advance(const __grid_constant__ Grid<T> g) {
    const long long n = *g.counter;
    if (n < g.steps) *g.counter = n + 1;
}

// ---- many steps in one launch ----------------------------------------------------------------------------------
// Grids whose passes are shorter than a launch (a 200 x 121 TE step: three launches of 3 us each for 24,200 cells)
// run all steps of a tfd_step call in one launch: E pass, barrier, H pass, barrier, the observations of step n - 1 taken
// beside the E pass of step n (they read the parity that step n leaves alone). CLUSTER: one thread-block cluster, hardware
// barrier; else at most one CTA per SM and a counting barrier in global memory. The groups are shared out evenly, a chunk per CTA
// and sweep; the observations start on the CTAs with the fewest chunks.
constexpr int kPassStepThreads = 512;
constexpr int kPassWaitTries = 1 << 22;          // polls of about 0.3 us: about a second

// Arrival of every CTA at barrier number `round` (0, 1, ...) of the launch; bar starts the launch at zero and must not wrap
// (kPassLaunchSteps in api.cu). False (with the status recorded) when the wait runs out.
__device__ __forceinline__ bool pass_grid_barrier(unsigned *bar, unsigned round, int *status) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned target = (round + 1) * gridDim.x;
        int good = 1;
        __threadfence();
        atomicAdd(bar, 1u);
        int it = 0;
        while (ld_acquire_u32(bar) < target)
            if (++it > kPassWaitTries) {
                good = 0;
                atomicExch(status, kStatusBarrierTimeout);
                break;
            }
        __threadfence();
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

template <typename T, int ACTIVE, bool METRIC, bool ADE, bool CLUSTER>
__global__ void __launch_bounds__(kPassStepThreads, 1) k_pass_steps(const __grid_constant__ PassArgs<T> A, const __grid_constant__ MonitorArgs<T> m,
                                                                    int mgx, int mgy, int count, unsigned *bar) {
    const Grid<T> &g = A.g;
    const long long n0 = *g.counter;
    // This thread's group p of plane z in the chunk at CTA position c of a sweep, and the position in the next sweep. FP32 steps
    // from sweep to sweep (on_p groups and on_z planes on; [1]: where c + rotate passes the last CTA); in FP64 the registers for
    // that spill (151 x 133 x 117 cells: 3 % longer), and each chunk divides.
    constexpr bool STEPPED = sizeof(T) == 4;
    const unsigned total = A.split[0].total;
    int p0;
    const int z0 = pass_divide(blockIdx.x * blockDim.x + threadIdx.x, total, A.magic_total, p0);
    unsigned on_p[2], on_z[2];
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        const unsigned by = (A.rotate + (d == 0 ? gridDim.x : 0)) * blockDim.x;
        on_z[d] = by / total;
        on_p[d] = by - on_z[d] * total;
    }
    auto at = [&](unsigned chunk, unsigned &p, unsigned &z) {
        if (STEPPED) return;
        int rest;
        z = (unsigned)pass_divide(chunk * blockDim.x + threadIdx.x, total, A.magic_total, rest);
        p = (unsigned)rest;
    };
    auto next = [&](unsigned &c, unsigned &p, unsigned &z) {
        c += A.rotate;
        const int d = c >= gridDim.x;
        if (d) c -= gridDim.x;
        if (!STEPPED) return;
        p += d ? on_p[1] : on_p[0];
        z += d ? on_z[1] : on_z[0];
        if (p >= total) {
            p -= total;
            ++z;
        }
    };
    // The observations: first on the CTAs at the end of the last sweep, which may have no chunk in it.
    const unsigned sweeps = (A.chunks + gridDim.x - 1) / gridDim.x;
    const int last = (int)(gridDim.x - 1 - (blockIdx.x + (sweeps - 1) * A.rotate) % gridDim.x);
    unsigned round = 0;
    auto barrier = [&]() -> bool {
        if constexpr (CLUSTER) {
            __syncthreads();
            cooperative_groups::this_cluster().sync();
            return true;
        } else {
            return pass_grid_barrier(bar, round++, g.status);
        }
    };
    long long n = n0;
    for (int k = 0; k < count && n < g.steps; ++k, ++n) {
        const int par = (int)(n & 1);
        T *slot = A.snap.base != nullptr ? A.snap.base + k * A.snap.stride : nullptr;
        if (k > 0)
            for (int b = last; b < mgx * mgy; b += gridDim.x) monitor_call(m, b % mgx, b / mgx, n - 1, mgx);
        for (unsigned sweep = 0, c = blockIdx.x, p = p0, z = z0; sweep < A.chunks; sweep += gridDim.x, next(c, p, z)) {
            at(sweep + c, p, z);
            if (sweep + c < A.chunks && z < (unsigned)g.n[2]) pass_block_e<T, ACTIVE, METRIC, ADE, int>(A, p, (int)z, par, n, slot);
        }
        if (!barrier()) return;
        if (ADE) {
            for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < g.ade_samples; j += gridDim.x * blockDim.x) pass_ade(g, j, par, n);
            if (!barrier()) return;
        }
        for (unsigned sweep = 0, c = blockIdx.x, p = p0, z = z0; sweep < A.chunks; sweep += gridDim.x, next(c, p, z)) {
            at(sweep + c, p, z);
            if (sweep + c < A.chunks && z < (unsigned)g.n[2]) pass_block_h<T, ACTIVE, METRIC, int>(A, p, (int)z, par, n, slot);
        }
        if (!barrier()) return;
    }
    if (n > n0)
        for (int b = last; b < mgx * mgy; b += gridDim.x) monitor_call(m, b % mgx, b / mgx, n - 1, mgx);
    if (blockIdx.x == 0 && threadIdx.x == 0) *g.counter = n;
}

}  // namespace tfd
