// Discrete adjoint of one Yee/CPML step: two passes, one thread per 16-byte group of cells of a row.
//
// The forward step n maps the state s_n = (E, H, psi) to s_{n+1}:
//     E' = E + (cn / eps) curl_b(H; psi_E)      then E sources
//     H' = H - cn curl_f(E'; psi_H)             then H sources
// and observations sample s_{n+1}. Its transpose (reference torchfdtd/differentiable.py:489-519,
// _System.transpose_step, with the CPML memory transpose of curl_faces_transpose :369-432) maps the
// adjoint lambda_{n+1} = (e_bar, h_bar, psi_bar) to lambda_n:
//     e_bar += curl_f^T(-cn h_bar)              (psi_H bars: m = psi_bar + v, psi_bar <- b m, v <- v/kappa + c m)
//     dJ/d eps += -cn e_bar curl_b(H_n; psi_E,n) / eps^2
//     h_bar += curl_b^T((cn / eps) e_bar)       (psi_E bars likewise)
// Sources are additive constants and drop out; observation seeds are added to e_bar / h_bar before
// the transpose of the step whose result they sampled. On a nonuniform mesh the forward scales each plain
// difference by the cell's metric factor before its CPML terms, so the transpose scales each D value after
// the CPML memory transpose (reference torchfdtd/differentiable.py:409-418).
//
// curl_f^T is a backward difference of the per-H-cell values D(k) (k = 0..n-2, plus the periodic wrap or
// PEC edge at n-1) and curl_b^T a forward difference of per-E-cell values D(k) (k = 1..n-1, plus the
// periodic edge at 0), so the adjoint step has the forward step's stencil shape and runs like it as two passes, one
// thread per 16-byte group of cells: k_adjoint_e writes e_bar_new (and accumulates the sensitivity), k_adjoint_h reads
// e_bar_new of its own cells and their +x, +y, +z neighbours back and writes h_bar_new. Adjoint fields and both
// families' adjoint CPML memories are double-buffered by reverse-step parity; each memory is written once, by the thread
// that owns its cell. The forward state comes from a snapshot of s_n, so no forward buffer is disturbed.
//
// In FP32 they must move 72 bytes per cell in the E pass (h_bar, the snapshot's H, e_bar and S read, e_bar and S written) and 40
// in the H pass (e_bar, 1/eps and h_bar read, h_bar written): 36 and 20 us at 200 x 200 x 80 cells and the copy rate.
//
// The material sensitivity is accumulated as S_c = sum_n e_bar_c * curl_b(H)_c per component; the host
// forms dJ/d eps = -cn S / eps^2 (summed over components for a per-cell permittivity).
#pragma once
#include "internal.cuh"
#include "step_pass.cuh"

namespace tfd {

// Terms of the curl whose INPUT is component C, in reference CURL_TERMS order (ascending axis):
// {axis, out, sign, j}.
struct RevTerm { int axis, out, sign, j; };
__host__ __device__ constexpr RevTerm rev_of(int in, int k) {
    return in == 0 ? (k == 0 ? RevTerm{1, 2, -1, 1} : RevTerm{2, 1, +1, 1})
         : in == 1 ? (k == 0 ? RevTerm{0, 2, +1, 1} : RevTerm{2, 0, -1, 0})
                   : (k == 0 ? RevTerm{0, 1, -1, 0} : RevTerm{1, 0, +1, 0});
}

template <typename T>
struct AdjArgs {
    Grid<T> g;                   // geometry, CPML tables, 1/eps; its field pointers are not used
    long long sE[3], sH[3];      // element offsets of the snapshot's arrays (-1: absent)
    long long sPsiE[3][2];
    T *eb[2][3], *hb[2][3];      // adjoint fields [parity][component]
    T *pEb[2][3][2], *pHb[2][3][2];   // adjoint CPML memories [parity][axis][term j]
    T *S[3];                     // material sensitivity per E component
    int slab[2][3][4];           // per family and axis: lo0, hi0, lo1, hi1 of the two CPML slabs
    PassSplit split;             // groups of a row away from the x slabs, and the others
};

// Slab row of coordinate c from the (lo, hi) bounds of a (family, axis), or -1: rows of the low slab first.
// The bounds sit in the kernel parameters, so no dependent table load precedes the CPML work.
__device__ __forceinline__ int adj_slab_row(const int *b, int c) {
    return (c >= b[0] && c < b[1]) ? c - b[0] : (c >= b[2] && c < b[3]) ? (b[1] - b[0]) + (c - b[2]) : -1;
}

// Loads through the read-only path: the memories and snapshots a reverse pass reads are not written by its launch, and
// without it every load waits behind the stores before it, which could alias it for the compiler.
__device__ __forceinline__ Pack<float> pack_ldg(const float *p) {
    const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
    return Pack<float>{{q.x, q.y, q.z, q.w}};
}
__device__ __forceinline__ Pack<double> pack_ldg(const double *p) {
    const double2 q = __ldg(reinterpret_cast<const double2 *>(p));
    return Pack<double>{{q.x, q.y}};
}

// CPML transpose of the D values v[] of a group's cells in one y or z slab row r: m = psi_bar + v; psi_bar <- b m (when
// own); v <- v / kappa + c m.
template <typename I, int F, int a, typename T>
__device__ __forceinline__ void adj_slab_row_apply(const AdjArgs<T> &A, int r, int x, int y, int z, const T *old, T *out, bool own,
                                                   T (&v)[Pack<T>::N]) {
    constexpr int N = Pack<T>::N;
    const Grid<T> &g = A.g;
    const int c = a == 1 ? y : z;
    const I p = a == 1 ? ((I)z * g.rows[F][1] + r) * g.pitch + x : ((I)r * g.n[1] + y) * g.pitch + x;
    const T b = __ldg(g.cb[F][a] + c), cc = __ldg(g.cc[F][a] + c), ck = __ldg(g.ck[F][a] + c);
    const Pack<T> m0 = pack_ldg(old + p);
    Pack<T> w;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const T m = m0.v[k] + v[k];
        w.v[k] = b * m;
        v[k] = v[k] * ck + cc * m;
    }
    if (own) pack_store(out + p, w);
}

// The same for one cell of an x slab.
template <typename I, int F, typename T>
__device__ __forceinline__ T adj_slab_x_apply(const AdjArgs<T> &A, int x, int y, int z, const T *old, T *out, bool own, T v) {
    const Grid<T> &g = A.g;
    if (old == nullptr || x < 0 || x >= g.n[0]) return v;
    const int r = adj_slab_row(A.slab[F][0], x);
    if (r < 0) return v;
    const I p = ((I)z * g.n[1] + y) * g.rows[F][0] + r;
    const T m = __ldg(old + p) + v;
    if (own) out[p] = __ldg(g.cb[F][0] + x) * m;
    return v * __ldg(g.ck[F][0] + x) + __ldg(g.cc[F][0] + x) * m;
}

// e_bar_new and the sensitivity of a group. XS: the group or a neighbour of its ends lies in an x slab. YZ: its row may meet
// a y or z slab or face, or the mesh is nonuniform; false (the plain variant) leaves those cases' code out.
// The D values of H-family terms are sign * (-cn h_bar): through the CPML transpose below the last cell, one period away
// or the PEC edge at it; e_bar[c] += D(c - 1), e_bar[c] -= D(c), in the order of the terms.
template <typename T, int ACTIVE, bool XS, bool YZ, typename I>
__device__ __forceinline__ void adj_pass_e(const AdjArgs<T> &A, const T *__restrict__ slot, int q, const PassCell<I> &w) {
    constexpr int N = Pack<T>::N;
    const Grid<T> &g = A.g;
    const I i = w.i, plane = (I)g.plane;
    const int x = w.x, y = w.y, z = w.z, nx = g.n[0], ny = g.n[1], nz = g.n[2];
    const bool last = x + N >= nx;
    const I ix = x > 0 ? i - 1 : i + (g.periodic[0] ? nx - 1 : 0);
    const I iy = !YZ || y > 0 ? i - g.pitch : i + (g.periodic[1] ? (I)(ny - 1) * g.pitch : 0);
    const I iz = !YZ || z > 0 ? i - plane : i + (g.periodic[2] ? (I)(nz - 1) * plane : 0);
    Pack<T> h[3], hy[3], hz[3], f[3], fy[3], fz[3], eb[3], S[3];
    T hx[3], fx[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        h[c] = hy[c] = hz[c] = f[c] = fy[c] = fz[c] = eb[c] = S[c] = Pack<T>{};
        hx[c] = fx[c] = T(0);
        if ((ACTIVE >> (3 + c)) & 1) {
            const T *hb = A.hb[q][c], *sf = slot + A.sH[c];
            h[c] = pack_ldg(hb + i);
            f[c] = pack_ldg(sf + i);
            if (c != 0) { hx[c] = __ldg(hb + ix); fx[c] = __ldg(sf + ix); }
            if (c != 1 && ny > 1) { hy[c] = pack_ldg(hb + iy); fy[c] = pack_ldg(sf + iy); }
            if (c != 2 && nz > 1) { hz[c] = pack_ldg(hb + iz); fz[c] = pack_ldg(sf + iz); }
        }
        if ((ACTIVE >> c) & 1) {
            eb[c] = pack_ldg(A.eb[q][c] + i);
            S[c] = pack_load(A.S[c] + i);
        }
    }
    const bool metric = YZ && (g.metric[0][0] != nullptr || g.metric[0][1] != nullptr || g.metric[0][2] != nullptr);
    auto mt = [&](int fam, int a, int c) -> T { return g.metric[fam][a] != nullptr ? g.metric[fam][a][c] : T(1); };
    Pack<T> e[3];
#pragma unroll
    for (int C = 0; C < 3; ++C) {
        if (!((ACTIVE >> C) & 1)) continue;
        T contrib[N], acc[N];
#pragma unroll
        for (int k = 0; k < N; ++k) contrib[k] = acc[k] = T(0);
#pragma unroll
        for (int t2 = 0; t2 < 2; ++t2) {
            const RevTerm t = rev_of(C, t2);
            const int a = t.axis, o = t.out;
            if (g.n[a] == 1 || !((ACTIVE >> (3 + o)) & 1)) continue;
            // D at the cells below (lo) and at the cells themselves (up).
            T lo[N], up[N];
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const T below = a == 0 ? (k == 0 ? hx[o] : h[o].v[k == 0 ? 0 : k - 1]) : a == 1 ? hy[o].v[k] : hz[o].v[k];
                const T dl = -g.cn * below, du = -g.cn * h[o].v[k];
                lo[k] = t.sign > 0 ? dl : -dl;
                up[k] = t.sign > 0 ? du : -du;
            }
            const T *old = A.pHb[q][a][t.j];
            T *out = A.pHb[q ^ 1][a][t.j];
            // Away from the faces of the axis (the usual case): both values, nothing else.
            if (a == 0 && x > 0 && !last) {
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const int c = x + k;
                    if (XS) {
                        lo[k] = adj_slab_x_apply<I, 1>(A, c - 1, y, z, old, out, false, lo[k]);
                        up[k] = adj_slab_x_apply<I, 1>(A, c, y, z, old, out, true, up[k]);
                    }
                    if (metric) {
                        lo[k] = lo[k] * mt(1, 0, c - 1);
                        up[k] = up[k] * mt(1, 0, c);
                    }
                    contrib[k] = contrib[k] + lo[k];
                    contrib[k] = contrib[k] - up[k];
                }
            } else if (a == 0) {
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const int c = x + k;
                    if (XS) {
                        if (c >= 1) lo[k] = adj_slab_x_apply<I, 1>(A, c - 1, y, z, old, out, false, lo[k]);
                        if (c < nx - 1) up[k] = adj_slab_x_apply<I, 1>(A, c, y, z, old, out, true, up[k]);
                    }
                    if (metric && c < nx) {
                        lo[k] = lo[k] * mt(1, 0, c >= 1 ? c - 1 : nx - 1);
                        if (c < nx - 1 || g.periodic[0]) up[k] = up[k] * mt(1, 0, c);
                    }
                    if (k == 0 && x == 0) {
                        // No cell below: nothing, or the wrap edge, added after the own cell's value.
                        contrib[0] = contrib[0] - up[0];
                        if (g.periodic[0]) contrib[0] = contrib[0] + lo[0];
                        continue;
                    }
                    contrib[k] = contrib[k] + lo[k];
                    if (!last || c < nx - 1) contrib[k] = contrib[k] - up[k];
                    else if (c == nx - 1) {
                        if (g.periodic[0]) contrib[k] = contrib[k] - up[k];
                        else if (g.pec_on[0]) contrib[k] = contrib[k] - (-g.pec_neg[0] * up[k]);
                    }
                }
            } else {
                const int c = a == 1 ? y : z, n = g.n[a];
                if (!YZ) {
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        contrib[k] = contrib[k] + lo[k];
                        contrib[k] = contrib[k] - up[k];
                    }
                    continue;
                }
                if (c >= 1 && old != nullptr) {
                    const int r = adj_slab_row(A.slab[1][a], c - 1);
                    if (r >= 0) {
                        if (a == 1) adj_slab_row_apply<I, 1, 1>(A, r, x, y - 1, z, old, out, false, lo);
                        else adj_slab_row_apply<I, 1, 2>(A, r, x, y, z - 1, old, out, false, lo);
                    }
                }
                if (c < n - 1 && old != nullptr) {
                    const int r = adj_slab_row(A.slab[1][a], c);
                    if (r >= 0) {
                        if (a == 1) adj_slab_row_apply<I, 1, 1>(A, r, x, y, z, old, out, true, up);
                        else adj_slab_row_apply<I, 1, 2>(A, r, x, y, z, old, out, true, up);
                    }
                }
                const T ml = metric ? mt(1, a, c >= 1 ? c - 1 : n - 1) : T(1), mu = metric ? mt(1, a, c) : T(1);
                if (c >= 1 && c < n - 1) {
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        if (metric) {
                            lo[k] = lo[k] * ml;
                            up[k] = up[k] * mu;
                        }
                        contrib[k] = contrib[k] + lo[k];
                        contrib[k] = contrib[k] - up[k];
                    }
                    continue;
                }
                const bool pec = c == n - 1 && !g.periodic[a] && g.pec_on[a], none = c == n - 1 && !g.periodic[a] && !g.pec_on[a];
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    if (metric) {
                        lo[k] = lo[k] * ml;
                        if (!pec) up[k] = up[k] * mu;
                    }
                    if (pec) up[k] = -g.pec_neg[a] * up[k];
                    if (c >= 1) contrib[k] = contrib[k] + lo[k];
                    if (!none) contrib[k] = contrib[k] - up[k];
                    if (c == 0 && g.periodic[a]) contrib[k] = contrib[k] + lo[k];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < N; ++k) e[C].v[k] = eb[C].v[k] + contrib[k];
        // The forward E curl from the snapshot (the arithmetic of the forward E update).
#pragma unroll
        for (int t2 = 0; t2 < 2; ++t2) {
            const Term t = term_of(C, t2);
            const int a = t.axis, in = t.in;
            if (g.n[a] == 1) continue;
            T d[N];
            const int c0 = a == 0 ? x : a == 1 ? y : z;
            const bool live = (a != 0 && !YZ) || c0 > 0 || g.periodic[a];
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const T below = a == 0 ? (k == 0 ? fx[in] : f[in].v[k == 0 ? 0 : k - 1]) : a == 1 ? fy[in].v[k] : fz[in].v[k];
                d[k] = f[in].v[k] - below;
                if ((a != 0 || k == 0) && !live) d[k] = T(0);
                if (metric) d[k] = d[k] * mt(0, a, a == 0 ? min(x + k, nx - 1) : c0);
            }
            if ((a == 0 ? XS : YZ) && A.sPsiE[a][t.j] >= 0) {
                const T *psi = slot + A.sPsiE[a][t.j];
                if (a == 0) {
                    if (XS)
#pragma unroll
                        for (int k = 0; k < N; ++k) {
                            const int c = x + k, r = c < nx ? adj_slab_row(A.slab[0][0], c) : -1;
                            if (c > 0 && r >= 0) {
                                const T m = __ldg(psi + (((I)z * ny + y) * g.rows[0][0] + r)) * __ldg(g.cb[0][0] + c) + __ldg(g.cc[0][0] + c) * d[k];
                                d[k] = d[k] * __ldg(g.ck[0][0] + c) + m;
                            }
                        }
                } else {
                    const int r = c0 > 0 ? adj_slab_row(A.slab[0][a], c0) : -1;
                    if (r >= 0) {
                        const Pack<T> m0 = pack_ldg(psi + (a == 1 ? ((I)z * g.rows[0][1] + r) * g.pitch + x : ((I)r * ny + y) * g.pitch + x));
                        const T b = __ldg(g.cb[0][a] + c0), cc = __ldg(g.cc[0][a] + c0), ck = __ldg(g.ck[0][a] + c0);
#pragma unroll
                        for (int k = 0; k < N; ++k) {
                            const T m = m0.v[k] * b + cc * d[k];
                            d[k] = d[k] * ck + m;
                        }
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < N; ++k) acc[k] = acc[k] + (t.sign > 0 ? d[k] : -d[k]);
        }
#pragma unroll
        for (int k = 0; k < N; ++k) {
            S[C].v[k] = S[C].v[k] + e[C].v[k] * acc[k];
            if (last && x + k >= nx) e[C].v[k] = S[C].v[k] = T(0);
        }
    }
#pragma unroll
    for (int C = 0; C < 3; ++C)
        if ((ACTIVE >> C) & 1) {
            pack_store(A.eb[q ^ 1][C] + i, e[C]);
            pack_store(A.S[C] + i, S[C]);
        }
}

// h_bar_new of a group from the stored e_bar_new. The D values of E-family terms are sign * ((cn / eps) e_bar_new), zero
// at cell 0 without a period; h_bar[c] += D(c), h_bar[c] -= D(c + 1).
template <typename T, int ACTIVE, bool XS, bool YZ, typename I>
__device__ __forceinline__ void adj_pass_h(const AdjArgs<T> &A, int q, const PassCell<I> &w) {
    constexpr int N = Pack<T>::N;
    const Grid<T> &g = A.g;
    const I i = w.i, plane = (I)g.plane;
    const int x = w.x, y = w.y, z = w.z, nx = g.n[0], ny = g.n[1], nz = g.n[2];
    const bool last = x + N >= nx;
    const I ix = last ? i - x : i + N;
    const I iy = !YZ || y < ny - 1 ? i + g.pitch : i - (g.periodic[1] ? (I)(ny - 1) * g.pitch : 0);
    const I iz = !YZ || z < nz - 1 ? i + plane : i - (g.periodic[2] ? (I)(nz - 1) * plane : 0);
    // u = (cn / eps) e_bar_new at the cells and at the +x, +y, +z neighbours.
    Pack<T> u[3], uy[3], uz[3], hb[3];
    T ux[3];
    auto scaled = [&](const Pack<T> &ie, const Pack<T> &eb) {
        Pack<T> r;
#pragma unroll
        for (int k = 0; k < N; ++k) r.v[k] = (g.cn * ie.v[k]) * eb.v[k];
        return r;
    };
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        u[c] = uy[c] = uz[c] = hb[c] = Pack<T>{};
        ux[c] = T(0);
        if ((ACTIVE >> c) & 1) {
            const T *eb = A.eb[q ^ 1][c], *ie = g.inv_eps[c];
            u[c] = scaled(pack_ldg(ie + i), pack_ldg(eb + i));
            if (c != 0) ux[c] = (g.cn * __ldg(ie + ix)) * __ldg(eb + ix);
            if (c != 1 && ny > 1) uy[c] = scaled(pack_ldg(ie + iy), pack_ldg(eb + iy));
            if (c != 2 && nz > 1) uz[c] = scaled(pack_ldg(ie + iz), pack_ldg(eb + iz));
        }
        if ((ACTIVE >> (3 + c)) & 1) hb[c] = pack_ldg(A.hb[q][c] + i);
    }
    const bool metric = YZ && (g.metric[0][0] != nullptr || g.metric[0][1] != nullptr || g.metric[0][2] != nullptr);
    auto mt = [&](int a, int c) -> T { return g.metric[0][a] != nullptr ? g.metric[0][a][c] : T(1); };
#pragma unroll
    for (int C = 0; C < 3; ++C) {
        if (!((ACTIVE >> (3 + C)) & 1)) continue;
        T contrib[N];
#pragma unroll
        for (int k = 0; k < N; ++k) contrib[k] = T(0);
#pragma unroll
        for (int t2 = 0; t2 < 2; ++t2) {
            const RevTerm t = rev_of(C, t2);
            const int a = t.axis, o = t.out;
            if (g.n[a] == 1 || !((ACTIVE >> o) & 1)) continue;
            T at[N], up[N];
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const T above = a == 0 ? (k == N - 1 ? ux[o] : u[o].v[k == N - 1 ? k : k + 1]) : a == 1 ? uy[o].v[k] : uz[o].v[k];
                at[k] = t.sign > 0 ? u[o].v[k] : -u[o].v[k];
                up[k] = t.sign > 0 ? above : -above;
            }
            const T *old = A.pEb[q][a][t.j];
            T *out = A.pEb[q ^ 1][a][t.j];
            if (a == 0 && x > 0 && !last) {
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const int c = x + k;
                    if (XS) {
                        at[k] = adj_slab_x_apply<I, 0>(A, c, y, z, old, out, true, at[k]);
                        up[k] = adj_slab_x_apply<I, 0>(A, c + 1, y, z, old, out, false, up[k]);
                    }
                    if (metric) {
                        at[k] = at[k] * mt(0, c);
                        up[k] = up[k] * mt(0, c + 1);
                    }
                    contrib[k] = contrib[k] + at[k];
                    contrib[k] = contrib[k] - up[k];
                }
            } else if (a == 0) {
                if (last && g.periodic[0]) {             // the last cell's +1 neighbour is the row's first
                    const T first = t.sign > 0 ? ux[o] : -ux[o];
#pragma unroll
                    for (int k = 0; k < N; ++k)
                        if (x + k == nx - 1) up[k] = first;
                }
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const int c = x + k;
                    if (XS) {
                        if (c >= 1) at[k] = adj_slab_x_apply<I, 0>(A, c, y, z, old, out, true, at[k]);
                        if (c + 1 <= nx - 1) up[k] = adj_slab_x_apply<I, 0>(A, c + 1, y, z, old, out, false, up[k]);
                    }
                    if (metric && c < nx) {
                        at[k] = at[k] * mt(0, c);
                        up[k] = up[k] * mt(0, c + 1 <= nx - 1 ? c + 1 : 0);
                    }
                    const bool wrap = g.periodic[0];
                    if (c >= 1 || k > 0) contrib[k] = contrib[k] + at[k];
                    if (!last || c + 1 <= nx - 1) contrib[k] = contrib[k] - up[k];
                    if (k == 0 && x == 0 && wrap) contrib[k] = contrib[k] + at[k];
                    if (last && c == nx - 1 && wrap) contrib[k] = contrib[k] - up[k];
                }
            } else {
                const int c = a == 1 ? y : z, n = g.n[a];
                if (!YZ) {
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        contrib[k] = contrib[k] + at[k];
                        contrib[k] = contrib[k] - up[k];
                    }
                    continue;
                }
                if (c >= 1 && old != nullptr) {
                    const int r = adj_slab_row(A.slab[0][a], c);
                    if (r >= 0) {
                        if (a == 1) adj_slab_row_apply<I, 0, 1>(A, r, x, y, z, old, out, true, at);
                        else adj_slab_row_apply<I, 0, 2>(A, r, x, y, z, old, out, true, at);
                    }
                }
                if (c + 1 <= n - 1 && old != nullptr) {
                    const int r = adj_slab_row(A.slab[0][a], c + 1);
                    if (r >= 0) {
                        if (a == 1) adj_slab_row_apply<I, 0, 1>(A, r, x, y + 1, z, old, out, false, up);
                        else adj_slab_row_apply<I, 0, 2>(A, r, x, y, z + 1, old, out, false, up);
                    }
                }
                const T ma = metric ? mt(a, c) : T(1), mu = metric ? mt(a, c + 1 <= n - 1 ? c + 1 : 0) : T(1);
                if (c >= 1 && c < n - 1) {
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        if (metric) {
                            at[k] = at[k] * ma;
                            up[k] = up[k] * mu;
                        }
                        contrib[k] = contrib[k] + at[k];
                        contrib[k] = contrib[k] - up[k];
                    }
                    continue;
                }
                const bool wrap = g.periodic[a];
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    if (metric) {
                        at[k] = at[k] * ma;
                        up[k] = up[k] * mu;
                    }
                    if (c >= 1) contrib[k] = contrib[k] + at[k];
                    if (c + 1 <= n - 1) contrib[k] = contrib[k] - up[k];
                    if (wrap && c == 0) contrib[k] = contrib[k] + at[k];
                    if (wrap && c == n - 1) contrib[k] = contrib[k] - up[k];
                }
            }
        }
        Pack<T> r;
#pragma unroll
        for (int k = 0; k < N; ++k) r.v[k] = !last || x + k < nx ? hb[C].v[k] + contrib[k] : T(0);
        pack_store(A.hb[q ^ 1][C] + i, r);
    }
}

// Whether row (y, z) takes the YZ variant: a nonuniform mesh, a y or z face, or a slab of either family on rows c - 1 .. c + 1.
template <typename T>
__device__ __forceinline__ bool adj_yz(const AdjArgs<T> &A, int y, int z) {
    const Grid<T> &g = A.g;
    bool near = g.metric[0][0] != nullptr || g.metric[0][1] != nullptr || g.metric[0][2] != nullptr;
#pragma unroll
    for (int a = 1; a < 3; ++a) {
        const int c = a == 1 ? y : z;
        if (g.n[a] == 1) continue;
        near = near || c == 0 || c == g.n[a] - 1;
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            const int *b = A.slab[f][a];
            near = near || (c + 1 >= b[0] && c - 1 < b[1]) || (c + 1 >= b[2] && c - 1 < b[3]);
        }
    }
    return near;
}

// Blocks per SM, us per launch at 200 x 200 x 80 cells, CPML 12, FP32: E pass 112 with two (128 registers), 123 with three;
// H pass 75 with two, 60 with three. (One thread per cell: 180 and 100.) Both are far from the DRAM floor of 36 and 20 us (260
// and 140 MB moved, CPML memories included): half the rows meet a slab, whose terms triple the instructions, and the E pass holds
// 20 input vectors per thread.
//
// Blocks of kPassThreads groups of one plane (blockIdx.x; plain groups first, then those near an x slab), planes on
// blockIdx.y: ascending in the E pass, descending in the H pass. Reads parity q, writes q^1.
template <typename T, int ACTIVE, typename I>
__global__ void __launch_bounds__(kPassThreads, 2) k_adjoint_e(const __grid_constant__ AdjArgs<T> A, const T *__restrict__ slot, int q) {
    const unsigned p = blockIdx.x * kPassThreads + threadIdx.x;
    if (p >= A.split.total) return;
    const bool slab = p >= A.split.plain_total;
    for (int z = blockIdx.y; z < A.g.n[2]; z += gridDim.y) {
        const PassCell<I> w = pass_cell<I>(A.g, A.split, p, z, slab);
        if (slab) adj_pass_e<T, ACTIVE, true, true>(A, slot, q, w);
        else if (adj_yz(A, w.y, w.z)) adj_pass_e<T, ACTIVE, false, true>(A, slot, q, w);
        else adj_pass_e<T, ACTIVE, false, false>(A, slot, q, w);
    }
}

template <typename T, int ACTIVE, typename I>
__global__ void __launch_bounds__(kPassThreads, sizeof(T) == 4 ? 3 : 2) k_adjoint_h(const __grid_constant__ AdjArgs<T> A, int q) {
    const unsigned p = blockIdx.x * kPassThreads + threadIdx.x;
    if (p >= A.split.total) return;
    const bool slab = p >= A.split.plain_total;
    for (int z = A.g.n[2] - 1 - (int)blockIdx.y; z >= 0; z -= gridDim.y) {
        const PassCell<I> w = pass_cell<I>(A.g, A.split, p, z, slab);
        if (slab) adj_pass_h<T, ACTIVE, true, true>(A, q, w);
        else if (adj_yz(A, w.y, w.z)) adj_pass_h<T, ACTIVE, false, true>(A, q, w);
        else adj_pass_h<T, ACTIVE, false, false>(A, q, w);
    }
}

// Observation seeds of one step: bar[family][comp][offset] += seed[k] (observers are distinct cells).
template <typename T>
__global__ void k_adjoint_seed(const __grid_constant__ AdjArgs<T> A, const TraceDev *__restrict__ obs, int n_obs,
                               const T *__restrict__ seed, int q) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n_obs; k += gridDim.x * blockDim.x) {
        const TraceDev o = obs[k];
        T *bar = o.family == 0 ? A.eb[q][o.comp] : A.hb[q][o.comp];
        if (bar != nullptr) bar[o.offset] = bar[o.offset] + seed[k];
    }
}

}  // namespace tfd
