// adjoint.cu -- kernels of the transposed half steps (adjoint.cuh).
#include <cuda_runtime.h>

#include <cstring>

#include "adjoint.cuh"

namespace mittet {

namespace {

// Threads of a CTA and x cells per thread.  ncu, 128x128x96 with 4 shots: 910
// warp instructions a vector (the mean of all boxes; two thirds of the cells
// are in the CPML), 39 % of the cycles issue, L1 is half busy, DRAM moves 3.6
// to 4.5 TB/s, and loads are 69 % of a warp's time.  Two cells at 80 registers
// beat four at twice that, as the boxes of a thin CPML are few vectors wide.
// Milliseconds of the adjoint stage (128x128x96 with 16 shots, 60 steps, and 4,
// 120; 64x64x48 x 4, 256; 108x110x104 x 2, 100; 110x106x108 x 1, 120; FP64
// 53x46x41 x 2, 150): 96.7, 50.0, 18.0, 15.0, 10.1, 5.7; with 6 CTAs of 128
// threads, tap offsets from the tables (the tap loads then wait for them), the
// history through L2 like the rest and both phases in the same order of shots
// 97.7, 50.8, 18.4, 15.3, 10.5, 5.7.  Over thousands of steps of 16 shots, where
// the power cap sets the clock, both take 1.72 ms a step.  20, 16 and 12 warps an
// SM with more registers take 103, 116 and 142 ms of the first; more than 24
// spill and are no faster.  Prefetches, tiles of 8 x 4 x 4 vectors instead of
// vectors in order, loads of the own field or the slabs' taus ahead of the taps,
// and a launch of the interior's own at 64 registers made no step faster.
constexpr int kNT = 64, kVX = 2, kBlocks = 12;

// Indices into the profile of one axis: sh and b of the own field (H phase:
// from H, own E).
template <bool EPH>
struct ProfOf {
    static constexpr int OSH = EPH ? 1 : 0, OB = EPH ? 4 : 2;
};

// Four values of a table row, 16 bytes a load.
__device__ __forceinline__ void ld4(int (&d)[4], const int *p) {
    const int4 v = __ldg(reinterpret_cast<const int4 *>(p));
    d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
}
__device__ __forceinline__ void ld4(double (&d)[4], const double *p) {
    const double2 a = __ldg(reinterpret_cast<const double2 *>(p)), b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
    d[0] = a.x; d[1] = a.y; d[2] = b.x; d[3] = b.y;
}

__device__ __forceinline__ bool in_axis(const DBox &b, int ax, int v) { return v >= b.lo[ax] && v < b.hi[ax]; }

// The y (AX = 1) or z (AX = 2) axis of one vector: adds the transposed
// differences of the weights to acc.  Along y the from field's z
// component A goes into the own x and x (X) into z; along z, y into x and x
// into y.  G: cells general along the axis: coefficients and slab rows come
// from the axis's table, so that no load waits behind a branch; tap offsets are
// clamped to the grid.  GX: lanes may lie outside the update range or the slab.
template <typename T, int VX, bool EPH, int AX, bool G, bool GX>
__device__ __forceinline__ void adj_axis(const AdjArgs<T> &a, int shot, int i0, int j, int k, const double *__restrict__ A,
                                         const double *__restrict__ X, const double (&ac)[VX], const double (&xc)[VX],
                                         double (&acc)[3][VX]) {
    constexpr int W = EPH ? -1 : -2, C = -W, OTH = 3 - AX, INTO = AX == 1 ? 2 : 1;
    const int n = AX == 1 ? a.ny : a.nz, v0 = AX == 1 ? j : k, vo = AX == 1 ? k : j, step = AX == 1 ? a.px : (int)a.plane;
    const DBox &UA = a.fupd[AX == 1 ? 2 : 1], &UX = a.fupd[0];
    const unsigned all = (1u << VX) - 1u;
    const unsigned ma = !in_axis(UA, OTH, vo) ? 0u : GX ? xmask<VX>(i0, UA.lo[0], UA.hi[0]) : all;
    const unsigned mx = !in_axis(UX, OTH, vo) ? 0u : GX ? xmask<VX>(i0, UX.lo[0], UX.hi[0]) : all;
    const AdjTapRow *__restrict__ R = G ? a.taps[AX - 1] + v0 : nullptr;
    double wa[4][VX], wx[4][VX];
    int l[4];
    double qa[4], qx[4];
    if constexpr (G) {
        ld4(l, R->l);
        ld4(qa, R->qa);
        ld4(qx, R->qx);
    }
#pragma unroll
    for (int t = 0; t < 4; t++) {
        int d = W + t;
        if constexpr (G) {
            d = min(max(v0 + d, 0), n - 1) - v0;
        } else {
            qa[t] = a.qk[AX][t];
            qx[t] = -qa[t];
        }
        if (t == C) {
#pragma unroll
            for (int v = 0; v < VX; v++) {
                wa[t][v] = ac[v];
                wx[t][v] = xc[v];
            }
        } else {
            ldv<double, VX>(wa[t], A + d * step);
            ldv<double, VX>(wx[t], X + d * step);
        }
    }
    double sa[VX], sx[VX];
#pragma unroll
    for (int v = 0; v < VX; v++) {
        sa[v] = sx[v] = 0.0;
#pragma unroll
        for (int t = 0; t < 4; t++) {
            sa[v] = fma(qa[t], wa[t][v], sa[v]);
            sx[v] = fma(qx[t], wx[t][v], sx[v]);
        }
        if (!(ma >> v & 1)) sa[v] = 0.0;
        if (!(mx >> v & 1)) sx[v] = 0.0;
    }
    if constexpr (G) {
        const DSlab &S = a.fslab[AX];
        if ((l[0] & l[1] & l[2] & l[3]) >= 0 && in_axis(S.other, OTH, vo)) {  // a tap in the slab
            const T *pa = a.ftau[AX][AX == 1 ? 1 : 0] + shot * a.fpsi[AX], *px = a.ftau[AX][AX == 1 ? 0 : 1] + shot * a.fpsi[AX];
            const unsigned sm = GX ? xmask<VX>(i0, S.other.lo[0], S.other.hi[0]) : all;
            T ta[4][VX], tx[4][VX];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const int lt = l[t] & 0x7fffffff;
                const int po = (AX == 1 ? k * S.width + lt : lt * a.ny + j) * a.px + i0;
                ldv<T, VX>(ta[t], pa + po);
                ldv<T, VX>(tx[t], px + po);
            }
            double qg[4];
            ld4(qg, R->qg);
#pragma unroll
            for (int t = 0; t < 4; t++)
#pragma unroll
                for (int v = 0; v < VX; v++)
                    if (sm >> v & 1) {
                        sa[v] = fma(qg[t], (double)ta[t][v], sa[v]);
                        sx[v] = fma(qg[t], (double)tx[t][v], sx[v]);
                    }
        }
    }
#pragma unroll
    for (int v = 0; v < VX; v++) {
        acc[0][v] += sa[v];
        acc[INTO][v] += sx[v];
    }
}

// The x axis: the from field's z component into the own y and y into z.
template <typename T, int VX, bool EPH, bool G>
__device__ __forceinline__ void adj_xaxis(const AdjArgs<T> &a, int shot, int i0, int j, int k, const double *__restrict__ Y,
                                          const double *__restrict__ Z, const double (&yc)[VX], const double (&zc)[VX],
                                          double (&acc)[3][VX]) {
    constexpr int W = EPH ? -1 : -2;
    constexpr int Q0 = VX + W, Q1 = 2 * VX + W + 3;  // taps of the vector's lanes, of [i0 - VX, i0 + 2 VX)
    const bool hl = !G || i0 >= VX, hr = !G || i0 + VX < a.nx;
    double y[3 * VX], z[3 * VX];
    {
        double l[2][VX], r[2][VX];
        ldv<double, VX>(l[0], Y - (hl ? VX : 0));
        ldv<double, VX>(l[1], Z - (hl ? VX : 0));
        ldv<double, VX>(r[0], Y + (hr ? VX : 0));
        ldv<double, VX>(r[1], Z + (hr ? VX : 0));
#pragma unroll
        for (int v = 0; v < VX; v++) {
            y[v] = l[0][v];
            z[v] = l[1][v];
            y[VX + v] = yc[v];
            z[VX + v] = zc[v];
            y[2 * VX + v] = r[0][v];
            z[2 * VX + v] = r[1][v];
        }
    }
    const DBox &UY = a.fupd[1], &UZ = a.fupd[2];
    const bool uy = in_axis(UY, 1, j) && in_axis(UY, 2, k), uz = in_axis(UZ, 1, j) && in_axis(UZ, 2, k);
    const double *qk = a.qk[0];
    if constexpr (!G) {
#pragma unroll
        for (int v = 0; v < VX; v++) {
            double sy = 0.0, sz = 0.0;
#pragma unroll
            for (int t = 0; t < 4; t++) {
                sz = fma(qk[t], z[VX + v + W + t], sz);
                sy = fma(qk[t], y[VX + v + W + t], sy);
            }
            if (uz) acc[1][v] += sz;
            if (uy) acc[2][v] -= sy;
        }
    } else {
        // weights of the cells (table entries are offset by 8), then psi
        const DSlab &S = a.fslab[0];
        const bool psi = in_axis(S.other, 1, j) && in_axis(S.other, 2, k);
        const long long row = shot * a.fpsi[0] + ((long long)k * a.ny + j) * S.width;
        double ty[3 * VX];  // psi_Hyx has a stencil of its own (cpu_cpml4.f90:400)
        double kz[3 * VX], ky[3 * VX], cg[3 * VX];
        int lx[3 * VX];
#pragma unroll
        for (int u = 0; u < 3; u++) {
            const int o = 8 + i0 + (u - 1) * VX;
            double t0[VX], t1[VX], t2[VX];
            int tl[VX];
            ldv<double, VX>(t0, a.xtab.kz + o);
            ldv<double, VX>(t1, a.xtab.ky + o);
            ldv<double, VX>(t2, a.xtab.cg + o);
            const int2 l2 = __ldg(reinterpret_cast<const int2 *>(a.xtab.l + o));
            tl[0] = l2.x;
            tl[1] = l2.y;
#pragma unroll
            for (int v = 0; v < VX; v++) {
                kz[u * VX + v] = uz ? t0[v] : 0.0;
                ky[u * VX + v] = uy ? t1[v] : 0.0;
                cg[u * VX + v] = t2[v];
                lx[u * VX + v] = tl[v];
            }
        }
#pragma unroll
        for (int q = Q0; q < Q1; q++) {
            const bool on = psi && lx[q] >= 0;
            const double tz = on ? cg[q] * (double)__ldg(a.ftau[0][0] + row + lx[q]) : 0.0;
            ty[q] = on ? cg[q] * (double)__ldg(a.ftau[0][1] + row + lx[q]) : 0.0;
            z[q] = fma(kz[q], z[q], tz);
            y[q] = EPH ? fma(ky[q], y[q], ty[q]) : ky[q] * y[q];
        }
#pragma unroll
        for (int v = 0; v < VX; v++) {
            const int q = VX + v + W;
#pragma unroll
            for (int t = 0; t < 4; t++) {
                acc[1][v] = fma(a.q[t], z[q + t], acc[1][v]);
                acc[2][v] = fma(a.q[t], y[q + t], acc[2][v]);
                if (!EPH) acc[2][v] = fma(t == 2 ? -(double)a.c2t : a.q[t], ty[q + t], acc[2][v]);
            }
        }
    }
}

// One vector of cells.  EPH: the E update's transpose (B from A, window from
// -1), else the H update's (A from B, window from -2).  GM: mask of the axes
// that are general; along the others every tap is interior to both fields.
template <typename T, int VX, bool EPH, int GM>
__device__ __forceinline__ void adj_cells(const AdjArgs<T> &a, int shot, int i0, int j, int k) {
    using P = ProfOf<EPH>;
    constexpr bool GX = (GM & 1) != 0, GY = (GM & 2) != 0, GZ = (GM & 4) != 0;
    const long long sb = (long long)shot * a.fshot;
    const int py = a.px, c = k * (int)a.plane + j * py + i0;
    const double *__restrict__ X = a.from[0] + sb + c, *__restrict__ Y = a.from[1] + sb + c, *__restrict__ Z = a.from[2] + sb + c;
    const T *__restrict__ PR = a.prof;
    const int ps = a.nmax;
    double xc[VX], yc[VX], zc[VX], o[3][VX];
    T m[VX];
    ldv<double, VX>(xc, X);
    ldv<double, VX>(yc, Y);
    ldv<double, VX>(zc, Z);
    if (!EPH || GM) ldv<T, VX>(m, a.m + c);
    // gradient of the E update at these cells, ahead of the stores, so that its
    // loads are in flight with the taps'
    if constexpr (EPH) {
        T e0[3][VX], e1[3][VX];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            ldv_stream<T, VX>(e0[q], a.S0[q] + sb + c);
            ldv_stream<T, VX>(e1[q], a.S1[q] + sb + c);
        }
        double2 *g = reinterpret_cast<double2 *>(a.grad + sb + c);
#pragma unroll
        for (int v = 0; v < VX; v += 2) {
            double2 gv = g[v / 2];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int w = v + u;
                const double s = fma(xc[w], (double)e0[0][w] - (double)e1[0][w],
                                     fma(yc[w], (double)e0[1][w] - (double)e1[1][w],
                                         zc[w] * ((double)e0[2][w] - (double)e1[2][w])));
                (u ? gv.y : gv.x) = fma(s, a.inv2w0dt, u ? gv.y : gv.x);
            }
            g[v / 2] = gv;
        }
    }
    double acc[3][VX];  // transposed curl and psi terms of the own x, y, z component
#pragma unroll
    for (int q = 0; q < 3; q++)
#pragma unroll
        for (int v = 0; v < VX; v++) acc[q][v] = 0.0;
    adj_axis<T, VX, EPH, 1, GY, GX>(a, shot, i0, j, k, Z, X, zc, xc, acc);
    adj_axis<T, VX, EPH, 2, GZ, GX>(a, shot, i0, j, k, Y, X, yc, xc, acc);
    adj_xaxis<T, VX, EPH, GX>(a, shot, i0, j, k, Y, Z, yc, zc, acc);
#pragma unroll
    for (int q = 0; q < 3; q++) ldv_rw<double, VX>(o[q], a.own[q] + sb + c);

    // own <- ca own + cb acc
    T base[VX];
    if constexpr (EPH) {
        if (a.dtmu) {
            ldv<T, VX>(base, a.dtmu + c);
        } else {
#pragma unroll
            for (int v = 0; v < VX; v++) base[v] = a.dtmu0;
        }
    } else {
#pragma unroll
        for (int v = 0; v < VX; v++) base[v] = m[v];
    }
    T shx[VX], shy = T(0), shz = T(0);
    if constexpr (GX) ldv<T, VX>(shx, PR + P::OSH * ps + i0);
    else zerov<T, VX>(shx);
    if constexpr (GY) shy = __ldg(PR + (8 + P::OSH) * ps + j);
    if constexpr (GZ) shz = __ldg(PR + (16 + P::OSH) * ps + k);
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const DBox &U = a.oupd[q];
        unsigned um = (1u << VX) - 1u;
        if constexpr (GM != 0)
            um = in_axis(U, 1, j) && in_axis(U, 2, k) ? (GX ? xmask<VX>(i0, U.lo[0], U.hi[0]) : um) : 0u;
        constexpr int bit[3] = {1, 2, 4};
#pragma unroll
        for (int v = 0; v < VX; v++) {
            T ca = T(1), cb = base[v];
            if (GM & bit[q]) {
                const T sh = q == 0 ? shx[v] : (q == 1 ? shy : shz);
                if (sh != T(0)) {
                    const T h = sh * m[v];
                    const T r = rcp(T(1) + h);
                    if (um >> v & 1) ca = (T(1) - h) * r;
                    cb *= r;
                }
            }
            o[q][v] = fma((double)cb, acc[q][v], (double)ca * o[q][v]);
            if (GX && i0 + v >= a.nx) o[q][v] = 0.0;
        }
    }
    // tau of the own slabs: x (z +, y -), y (x +, z -), z (y +, x -) on E, the
    // other signs on H
    const double so = EPH ? -1.0 : 1.0;
    if constexpr (GX) {
        const DSlab &S = a.oslab[0];
        if (in_axis(S.other, 1, j) && in_axis(S.other, 2, k)) {
            const long long po = shot * a.opsi[0] + ((long long)k * a.ny + j) * S.width;
            T t0[VX], t1[VX], b[VX];
            int l[VX];
#pragma unroll
            for (int v = 0; v < VX; v++) {
                l[v] = slab_local(S, i0 + v);
                t0[v] = l[v] >= 0 ? a.otau[0][0][po + l[v]] : T(0);
                t1[v] = l[v] >= 0 ? a.otau[0][1][po + l[v]] : T(0);
            }
            ldv<T, VX>(b, PR + P::OB * ps + i0);
#pragma unroll
            for (int v = 0; v < VX; v++)
                if (l[v] >= 0) {
                    a.otau[0][0][po + l[v]] = (T)fma((double)b[v], (double)t0[v], so * o[2][v]);
                    a.otau[0][1][po + l[v]] = (T)fma((double)b[v], (double)t1[v], -so * o[1][v]);
                }
        }
    }
    auto own_tau = [&](int ax, long long po, unsigned mk, const double(&plus)[VX], const double(&minus)[VX], double b) {
        if (!mk) return;
        T t0[VX], t1[VX], *p0 = a.otau[ax][0] + po, *p1 = a.otau[ax][1] + po;
        ldv_rw<T, VX>(t0, p0);  // whole vectors: psi rows are padded
        ldv_rw<T, VX>(t1, p1);
#pragma unroll
        for (int v = 0; v < VX; v++) {
            t0[v] = (T)fma(b, (double)t0[v], so * plus[v]);
            t1[v] = (T)fma(b, (double)t1[v], -so * minus[v]);
        }
        st_psi<T, VX>(p0, 0, t0, mk);
        st_psi<T, VX>(p1, 0, t1, mk);
    };
    if constexpr (GY) {
        const DSlab &S = a.oslab[1];
        const int l = slab_local(S, j);
        if (l >= 0 && in_axis(S.other, 2, k))
            own_tau(1, shot * a.opsi[1] + ((long long)k * S.width + l) * py + i0, xmask<VX>(i0, S.other.lo[0], S.other.hi[0]),
                    o[0], o[2], __ldg(PR + (8 + P::OB) * ps + j));
    }
    if constexpr (GZ) {
        const DSlab &S = a.oslab[2];
        const int l = slab_local(S, k);
        if (l >= 0 && in_axis(S.other, 1, j))
            own_tau(2, shot * a.opsi[2] + ((long long)l * a.ny + j) * py + i0, xmask<VX>(i0, S.other.lo[0], S.other.hi[0]),
                    o[1], o[0], __ldg(PR + (16 + P::OB) * ps + k));
    }
#pragma unroll
    for (int q = 0; q < 3; q++) stv<double, VX>(a.own[q] + sb + c, o[q]);

    // gradient of the H update, in profile cells
    if constexpr (!EPH && GM != 0) {
        T fsx[VX], fsy = T(0), fsz = T(0);
        if constexpr (GX) ldv<T, VX>(fsx, PR + ps + i0);
        else zerov<T, VX>(fsx);
        if constexpr (GY) fsy = __ldg(PR + 9 * ps + j);
        if constexpr (GZ) fsz = __ldg(PR + 17 * ps + k);
        bool ax = false;
#pragma unroll
        for (int v = 0; v < VX; v++) ax |= fsx[v] != T(0);
        const bool on[3] = {GX && ax, GY && fsy != T(0), GZ && fsz != T(0)};
        if (on[0] || on[1] || on[2]) {
            double s[VX];
#pragma unroll
            for (int v = 0; v < VX; v++) s[v] = 0.0;
#pragma unroll
            for (int q = 0; q < 3; q++) {
                if (!on[q]) continue;
                T h0[VX], h1[VX];
                ldv<T, VX>(h0, a.S0[q] + sb + c);
                ldv<T, VX>(h1, a.S1[q] + sb + c);
                const DBox &U = a.fupd[q];
                const unsigned um = in_axis(U, 1, j) && in_axis(U, 2, k) ? xmask<VX>(i0, U.lo[0], U.hi[0]) : 0u;
#pragma unroll
                for (int v = 0; v < VX; v++) {
                    const T sh = q == 0 ? fsx[v] : (q == 1 ? fsy : fsz);
                    const double f = q == 0 ? xc[v] : (q == 1 ? yc[v] : zc[v]);
                    const double d = (um >> v & 1) ? (double)h1[v] + (double)h0[v] : (double)h1[v] - (double)h0[v];
                    s[v] = fma(f * d, (double)sh, s[v]);
                }
            }
            double *g = a.grad + sb + c;
#pragma unroll
            for (int v = 0; v < VX; v++) {
                if (GX && i0 + v >= a.nx) continue;
                const double mm = (double)m[v], idm = a.dtmu ? 1.0 / (double)__ldg(a.dtmu + c + v) : a.inv_dtmu0;
                g[v] = fma(s[v], mm * (mm * a.inv2w0dt) * idm, g[v]);
            }
        }
    }
}

// All boxes of one phase in one launch, one vector per thread; the body is
// chosen per CTA.  Corners and edges come first: they take longest.  The E
// phase walks the shots backwards: its first ones are those the H phase left
// in L2, and the reverse at the next step.
template <typename T, bool EPH>
__global__ void __launch_bounds__(kNT, kBlocks)
    adj_phase_kernel(const __grid_constant__ AdjArgs<T> a, const __grid_constant__ AdjBoxes b) {
    constexpr int VX = kVX;
    const int t = (int)blockIdx.x;
    int q = 0;
    for (int w = 1; w < b.nbox; w++)
        if (t >= b.start[w]) q = w;
    const int x = (t - b.start[q]) * kNT + (int)threadIdx.x;
    if (x >= b.vecs[q]) return;
    const int r = x / b.nvx[q], kl = r / b.rows[q];
    const int i0 = b.lo[q][0] + (x - r * b.nvx[q]) * VX, j = b.lo[q][1] + r - kl * b.rows[q], k = b.lo[q][2] + kl;
    const int shot = EPH ? (int)(gridDim.y - 1u - blockIdx.y) : (int)blockIdx.y;
    switch (b.kind[q]) {
        case 0: adj_cells<T, VX, EPH, 0>(a, shot, i0, j, k); break;
        case 1: adj_cells<T, VX, EPH, 1>(a, shot, i0, j, k); break;
        case 2: adj_cells<T, VX, EPH, 2>(a, shot, i0, j, k); break;
        case 4: adj_cells<T, VX, EPH, 4>(a, shot, i0, j, k); break;
        default: adj_cells<T, VX, EPH, 7>(a, shot, i0, j, k); break;
    }
}

// Receivers of one kind: the scaled adjoint and the taus that hold it.
template <typename T, bool E>
__global__ void adj_inject_kernel(const __grid_constant__ AdjInject<T> q, int n) {
    const AdjArgs<T> &a = q.a;
    const int tot = q.nrec * q.nshot;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += gridDim.x * blockDim.x) {
        const int s = e / q.nrec, r = e % q.nrec, comp = q.rec_comp[r];
        if ((comp < 3) != E) continue;
        const int c = (int)q.rec_off[r], w = comp % 3;
        const int k = c / (int)a.plane, rem = c - k * (int)a.plane, j = rem / a.px, i = rem - j * a.px;
        const int p3[3] = {i, j, k};
        T cb = E ? a.m[c] : (a.dtmu ? a.dtmu[c] : a.dtmu0);
        const T sh = a.prof[(w * 8 + (E ? 0 : 1)) * a.nmax + p3[w]];
        if (sh != T(0)) cb *= rcp(T(1) + sh * a.m[c]);
        const double d = (double)cb * q.asrc[(long long)e * q.nt + n];
        atomicAdd(a.own[w] + s * a.fshot + c, d);
        // component x is in tau y0 (+), z1 (-); y in z0 (+), x1 (-); z in x0
        // (+), y1 (-) on E; the other signs on H
        const double so = E ? d : -d;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int ax = u == 0 ? (w + 1) % 3 : (w + 2) % 3;
            const DSlab &S = a.oslab[ax];
            const int l = slab_local(S, p3[ax]);
            bool in = l >= 0;
#pragma unroll
            for (int b = 0; b < 3; b++)
                if (b != ax) in = in && p3[b] >= S.other.lo[b] && p3[b] < S.other.hi[b];
            if (!in) continue;
            const long long po = s * a.opsi[ax] + (ax == 0 ? ((long long)k * a.ny + j) * S.width + l
                                                   : ax == 1 ? ((long long)k * S.width + l) * a.px + i
                                                             : ((long long)l * a.ny + j) * a.px + i);
            atomicAdd(a.otau[ax][u] + po, (T)(u == 0 ? so : -so));
        }
    }
}

// Source terms of adjoint step n for the points of one kind (adjoint.cuh).
template <typename T, bool E>
__global__ void adj_src_kernel(const __grid_constant__ AdjArgs<T> a, const AdjSrc *__restrict__ pts, int npts,
                               const double *__restrict__ wave, int n, int shot0, int shot1) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= npts) return;
    const AdjSrc p = pts[q];
    if ((p.kind == 1) != E || (p.comp < 3) != E || p.shot < shot0 || p.shot >= shot1) return;
    const long long c = (long long)(p.shot - shot0) * a.fshot + p.off;
    const int ax = p.comp % 3, v = ax == 0 ? p.i : (ax == 1 ? p.j : p.k);
    const double m = (double)a.m[p.off], h = (double)a.prof[(ax * 8 + (E ? 0 : 1)) * a.nmax + v] * m;
    if (h == 0.0) return;
    const double f = a.from[ax][c];
    double t;
    if (E) {
        t = f * p.g * ((wave[n] + wave[n + 1]) / 2.0) * h * a.inv2w0dt;
    } else {
        const double dm = a.dtmu ? (double)a.dtmu[p.off] : (double)a.dtmu0;
        const double k = f * h * (m * a.inv2w0dt) / dm;
        t = (in_box(a.fupd[ax], p.i, p.j, p.k) ? k : -k) * (-p.g * wave[n + 1]);
    }
    atomicAdd(a.grad + c, t);
}

}  // namespace

template <typename T>
AdjBoxes adj_boxes(int nx, int ny, int nz, const int lo[3], const int hi[3]) {
    constexpr int VX = kVX;
    AdjBoxes b;
    memset(&b, 0, sizeof(b));
    auto add = [&](int kind, int x0, int y0, int z0, int x1, int y1, int z1) {
        if (x1 <= x0 || y1 <= y0 || z1 <= z0) return;
        const int q = b.nbox++;
        b.kind[q] = kind;
        b.lo[q][0] = x0; b.lo[q][1] = y0; b.lo[q][2] = z0;
        b.hi[q][0] = x1; b.hi[q][1] = y1; b.hi[q][2] = z1;
        b.nvx[q] = (x1 - x0 + VX - 1) / VX;
        b.rows[q] = y1 - y0;
        b.vecs[q] = b.nvx[q] * (y1 - y0) * (z1 - z0);
        b.start[q + 1] = b.start[q] + (b.vecs[q] + kNT - 1) / kNT;
    };
    const int x0 = (lo[0] + VX - 1) / VX * VX, x1 = hi[0] / VX * VX;  // whole vectors
    const bool inner = x1 > x0 && hi[1] > lo[1] && hi[2] > lo[2];
    if (!inner) {
        add(7, 0, 0, 0, nx, ny, nz);
        return b;
    }
    const int y0 = lo[1], y1 = hi[1], z0 = lo[2], z1 = hi[2];
    const int xr[2][2] = {{0, x0}, {x1, nx}}, yr[2][2] = {{0, y0}, {y1, ny}}, zr[2][2] = {{0, z0}, {z1, nz}};
    for (const auto &z : zr) {  // rings around the z faces, edges along z
        add(7, 0, 0, z[0], nx, y0, z[1]);
        add(7, 0, y1, z[0], nx, ny, z[1]);
        add(7, 0, y0, z[0], x0, y1, z[1]);
        add(7, x1, y0, z[0], nx, y1, z[1]);
    }
    for (const auto &x : xr)
        for (const auto &y : yr) add(7, x[0], y[0], z0, x[1], y[1], z1);
    add(1, 0, y0, z0, x0, y1, z1);  // faces
    add(1, x1, y0, z0, nx, y1, z1);
    add(2, x0, 0, z0, x1, y0, z1);
    add(2, x0, y1, z0, x1, ny, z1);
    add(4, x0, y0, 0, x1, y1, z0);
    add(4, x0, y0, z1, x1, y1, nz);
    add(0, x0, y0, z0, x1, y1, z1);
    return b;
}

template <typename T>
void adj_phase_launch(bool e, const AdjArgs<T> &a, const AdjBoxes &b, int nshot, cudaStream_t st) {
    const dim3 grid((unsigned)b.start[b.nbox], (unsigned)nshot);
    if (e) adj_phase_kernel<T, true><<<grid, kNT, 0, st>>>(a, b);
    else adj_phase_kernel<T, false><<<grid, kNT, 0, st>>>(a, b);
}
template <typename T>
void adj_inject_launch(bool e, const AdjInject<T> &q, int n, cudaStream_t st) {
    const int tot = q.nrec * q.nshot;
    if (tot <= 0) return;
    const int grid = tot < 1024 ? (tot + 63) / 64 : 16;
    if (e) adj_inject_kernel<T, true><<<grid, 64, 0, st>>>(q, n);
    else adj_inject_kernel<T, false><<<grid, 64, 0, st>>>(q, n);
}
template <typename T>
void adj_src_launch(bool e, const AdjArgs<T> &a, const AdjSrc *pts, int npts, const double *wave, int n, int shot0,
                    int shot1, cudaStream_t st) {
    if (npts <= 0) return;
    const int grid = (npts + 63) / 64;
    if (e) adj_src_kernel<T, true><<<grid, 64, 0, st>>>(a, pts, npts, wave, n, shot0, shot1);
    else adj_src_kernel<T, false><<<grid, 64, 0, st>>>(a, pts, npts, wave, n, shot0, shot1);
}

#define MITTET_ADJ(T)                                                                                            \
    template AdjBoxes adj_boxes<T>(int, int, int, const int[3], const int[3]);                                  \
    template void adj_phase_launch<T>(bool, const AdjArgs<T> &, const AdjBoxes &, int, cudaStream_t);            \
    template void adj_inject_launch<T>(bool, const AdjInject<T> &, int, cudaStream_t);                           \
    template void adj_src_launch<T>(bool, const AdjArgs<T> &, const AdjSrc *, int, const double *, int, int, int, \
                                    cudaStream_t);
MITTET_ADJ(float)
MITTET_ADJ(double)

}  // namespace mittet
