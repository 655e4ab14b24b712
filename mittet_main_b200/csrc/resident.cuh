// resident.cuh -- a block of time steps with the fields resident in shared
// memory.
//
// A grid of up to about a million FP32 cells (half that in FP64) fits the
// shared memory of the whole GPU: 148 SMs x 227 KB hold its six field
// components.  The stepped path moves those fields through L2 or HBM twice a
// step and launches four to a dozen kernels for it; here one cooperative
// launch keeps one CTA per SM, gives each a tile of rows (all of x, a block of
// y and z), keeps the tile's six components in shared memory for all steps
// of the launch, and exchanges only the rows a neighbouring tile reads.
//
//   per phase: edge rows (they read the neighbours' rows from global memory,
//   L2-coherent, and write their own there for the neighbours) -> raise this
//   tile's flag -> inner rows -> wait for the four neighbours' flags
//
// so the rows and flags travel while the inner rows are computed.  E reads
// offsets -2..+1, H reads -1..+2 along y and z, so the rows a tile exchanges
// after a phase and the rows that need a neighbour in that phase are the same:
// the first two and the last one (E), the first one and the last two (H).  A
// tile overwrites an exchanged row only after its neighbour's next flag, which
// the neighbour raises after all of its rows that read it.
//
// Sources and receivers are done by the tile that owns the cell: electric
// points after the E update, the next step's magnetic points after the H
// update (a receiver on such a cell samples the value before it), samples
// one phase later, while the neighbours are waited for.  Every value is
// formed with the fma forms of stencil.cuh, so a cell's result is the same
// bit for bit as on the stepped path.
//
// The model word, permeability and psi are private to a cell's thread and
// stay in L2; those of a thread's first cells of a phase are loaded before the
// wait.  Shots are independent: with
// G tiles per shot, floor(SMs / G) groups of CTAs each walk their own shots.
//
// What bounds it (ncu, 64^3, one pass of a CTA over its vectors, 10.4 us a
// step): a third of the warps' time goes to the barriers behind the neighbours'
// flags, and the general body issues 1010 instructions per vector of four cells
// and phase, 39 % of the issue slots of the 16 warps an SM holds; DRAM is idle.
// At 96^3 the body is most of the time (38 Gcell/s; the stepped path's 20 is
// launch- and L2-bound there).  Tried and slower: halo rows staged by bulk copies (the
// copies wait for the flags, 8 us a phase at 64^3), and 64-bit words that
// carry data and a message number (every vector polls its own words: 11 us).
//
// The launch is cooperative (every CTA co-resident) and every wait is
// bounded by %globaltimer as in persistent.cuh: bit 2 of the error word.
#pragma once
#include <type_traits>

#include "persistent.cuh"

namespace mittet {

// x cells per thread and threads per CTA.  Measured for FP32 (64^3 in one
// pass, 96^3, 32 shots of 64^3; microseconds per step): 4 x 512 (128
// registers, 48 bytes of spill) 10.7, 26.9, 225; 4 x 384 (168) 13.6, 28.2,
// 238; 2 x 768 (80) 12.5, 29.7, 252; 2 x 512 (128) 11.9, 30.2, 253.  FP64: two
// cells need 232 registers.
template <typename T>
struct ResShape;
template <>
struct ResShape<float> {
    static constexpr int VX = 4, NT = 512;
};
template <>
struct ResShape<double> {
    static constexpr int VX = 2, NT = 256;
};
// Steps of one resident launch: long enough that loading and storing the
// tiles does not show, and by the tiling's own estimate no more than half a
// second for all shots, since nothing else of the process gets the SMs
// meanwhile (64 shots of 101^3 take 2 ms a step).
constexpr int kResidentSteps = 1024;
constexpr double kResidentLaunchUs = 5e5;
constexpr int kResMaxPts = 32;    // points of one shot
constexpr int kResRecCache = 128; // receivers of a tile listed in shared memory
constexpr int kResFlagStride = 32;  // words between flags: one line each
constexpr int kResMaxTiles = 160;  // tiles along one axis, at most the SMs

// A receiver of one tile: offset within a field of the tile, component, index.
struct ResRec {
    int off, comp, rec;
};

template <typename T>
struct ResArgs {
    PhaseArgs<T> e, h;
    int ty, tz;              // tiles along y and z
    int groups;              // shots computed at a time
    int nshot, nsteps, n0;
    int nrow;                // rows of the largest tile
    int pitch, rymax, rzmax; // elements of a shared row (whole vectors); most rows of a tile along y and z
    unsigned short ys[kResMaxTiles + 1], zs[kResMaxTiles + 1];  // first row of each tile
    const SrcPoint *pts;
    int npts;
    const double *wave;
    const ResRec *recs;      // receivers by tile
    const int *rec_start;    // [ty * tz + 1]
    int nrec;
    T *traces;               // [shot][nrec][nt] or nullptr
    int nt;
    T *hist;                 // state after step s at slot s + 1 (nullptr: none)
    long long hist_slot, hist_comp;
    unsigned *flags;         // [CTA] phases done, kResFlagStride words apart, zero at launch
    unsigned expect_more;    // 0; a test asks for a phase that nobody finishes
    int *err;
    unsigned long long wait_ns;
};

struct ResPt {
    double g;
    int off;   // within a field of the tile
    int comp, kind;
    int pad;
};

// One row of the tile in one phase, in the order the rows are computed.
struct __align__(16) ResRow {
    unsigned flags;          // row index, then the kRow bits
    int c;                   // offset of the row in a global field of the shot
    int ox, oy, oz;          // offsets of the row in the psi slabs
    unsigned short jl, kl;   // position in the tile
    unsigned short tap[12];  // shared row of the taps beside the centre: G_z and G_x along y, G_x and G_y along z
};
static_assert(sizeof(ResRow) == 48, "three vector loads");
constexpr unsigned kRowVy = 1u << 16, kRowVz = 1u << 17, kRowU0 = 1u << 18, kRowMx = 1u << 21, kRowMy = 1u << 22,
                   kRowMz = 1u << 23, kRowSy = 1u << 24, kRowSz = 1u << 25;
constexpr unsigned kRowPy = 1u << 26, kRowPz = 1u << 27;  // a neighbour along y, z reads the row
constexpr unsigned short kTapRemote = 0xffff;             // the tap's row is a neighbour's
// One x vector in one phase: four-bit lane masks (update ranges of the three
// components, x slab, x range of the y and z slabs, valid x difference), then
// whether a lane has an x profile and whether every lane is inside every
// update range with a valid difference.
struct __align__(8) ResVec {
    unsigned lanes;
    int lx;                  // x-slab index of lane 0 (may lie outside; lanes in the mask count from it)
};
constexpr unsigned kVecS = 1u << 28, kVecFull = 1u << 29;

// A shot's arrays, in shared memory so that the step loop does not keep
// dozens of addresses in registers.
template <typename T>
struct ResPtrs {
    T *f[6], *psi[2][6], *hist;
};

// Shared memory of a CTA.
template <typename T>
struct ResSmem {
    static constexpr int VX = ResShape<T>::VX;
    static __host__ __device__ size_t a16(size_t n) { return (n + 15) / 16 * 16; }
    static __host__ __device__ size_t rows(int nrow, int pitch) { return a16((size_t)6 * nrow * pitch * sizeof(T)); }
    static __host__ __device__ size_t xprof(int pitch) { return a16((size_t)8 * pitch * sizeof(T)); }
    static __host__ __device__ size_t yzprof(int ry, int rz) { return a16((size_t)8 * (ry + rz) * sizeof(T)); }
    // nrow: rows of the largest tile
    static __host__ __device__ size_t bytes(int nrow, int ry, int rz, int pitch) {
        return rows(nrow, pitch) + xprof(pitch) + yzprof(ry, rz) + (size_t)2 * nrow * sizeof(ResRow) +
               a16((size_t)2 * (pitch / VX) * sizeof(ResVec)) + a16(sizeof(ResPtrs<T>)) + kResMaxPts * sizeof(ResPt) +
               a16(kResMaxPts * sizeof(T)) + a16(kResRecCache * sizeof(ResRec));
    }
};

// Sums and products that the compiler may not contract: what it makes of the
// same terms in stencil.cuh, written out.
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
// The ring's copy of an injected cell, as inject_kernel's old + (T)(-g w)
// rounds: in FP64 the compiler contracts it.
__device__ __forceinline__ float inject_ring(float old, double g, double w) { return add_rn(old, (float)(-mul_rn(g, w))); }
__device__ __forceinline__ double inject_ring(double old, double g, double w) { return fma(-g, w, old); }
// Along an axis with profile sh: cb becomes cb/(1 + h) and e = ca f with
// ca = (1 - h)/(1 + h), h = sh m.
template <typename T>
__device__ __forceinline__ void res_coef(T sh, T m, T &cb, T f, T &e) {
    const T h = mul_rn(sh, m);
    const T r = rcp(add_rn(T(1), h));
    e = mul_rn(mul_rn(add_rn(T(1), -h), r), f);
    cb = mul_rn(cb, r);
}

template <typename T, int VX>
__device__ __forceinline__ void ld_plain(T (&d)[VX], const T *p) {
    using V = typename VecT<T, VX>::type;
    const V v = *reinterpret_cast<const V *>(p);
    const T *s = reinterpret_cast<const T *>(&v);
#pragma unroll
    for (int q = 0; q < VX; q++) d[q] = s[q];
}
// Loads a neighbour's cell vector (L2-coherent) where `on`, without a branch,
// so that all of a thread's loads are in flight at once.
__device__ __forceinline__ void ld_remote(float (&d)[2], const float *p, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];\n\t}"
                 : "+f"(d[0]), "+f"(d[1])
                 : "l"(p), "r"((unsigned)on)
                 : "memory");
}
__device__ __forceinline__ void ld_remote(float (&d)[4], const float *p, bool on) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t@p ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "l"(p), "r"((unsigned)on)
        : "memory");
}
__device__ __forceinline__ void ld_remote(double (&d)[2], const double *p, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];\n\t}"
                 : "+d"(d[0]), "+d"(d[1])
                 : "l"(p), "r"((unsigned)on)
                 : "memory");
}

// What a CTA knows of its tile.
template <typename T>
struct ResTile {
    T *s;                      // shared rows: six fields of rmax rows, then the halo
    const T *xp, *yp, *zp;     // profiles: x [8][pitch], y [2][nry][4], z [2][nrz][4] (sh, 1/kd, b, c/d of E, H)
    const ResRow *rows[2];     // E, H; rows of the exchange first
    const ResVec *vecs[2];
    const ResPtrs<T> *g;
    const ResPt *pts;
    T *pre;                    // H at a magnetic point before its injection
    int rmax, pitch, nvec, nry, nrz, items, edge[2];
    float inv_nvec;            // 1 / nvec
    int npt, shot;
};

// Rows a tile exchanges along one axis after a phase (and that need the
// neighbour in it): E the first two and the last, H the first and the last two.
__device__ __forceinline__ bool res_exchanged(bool eph, int v, int n, bool lo, bool hi) {
    return (lo && v < (eph ? 2 : 1)) || (hi && v >= n - (eph ? 1 : 2));
}

// Row of item x (below 2^20, so that the rounded product is exact enough).
template <typename T>
__device__ __forceinline__ int res_row(const ResTile<T> &t, int x) {
    return (int)(((float)x + 0.5f) * t.inv_nvec);
}

__device__ __forceinline__ unsigned res_lanes(const ResVec &V, int which) { return V.lanes >> (4 * which) & 15u; }

// {sh, 1/kd, b, c/d} of one row and axis.
template <typename T>
struct ResProf {
    T sh, ik, b, g;
};
__device__ __forceinline__ ResProf<float> res_prof(const float *p) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    return {v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ ResProf<double> res_prof(const double *p) {
    const double2 v = *reinterpret_cast<const double2 *>(p), w = *reinterpret_cast<const double2 *>(p + 2);
    return {v.x, v.y, w.x, w.y};
}

// psi of one slab group: the lanes of mk.
template <typename T, int VX>
__device__ __forceinline__ void res_ld_psi(T (&d)[VX], const T *p, unsigned mk) {
    if (mk == (1u << VX) - 1u) {
        ld_plain<T, VX>(d, p);
    } else {
#pragma unroll
        for (int v = 0; v < VX; v++) d[v] = (mk >> v & 1) ? p[v] : T(0);
    }
}

// What a cell vector owns alone, in L2: its model words and psi.
template <typename T, int VX>
struct ResPriv {
    T m[VX], q[6][VX];
};
template <typename T, int VX, bool EPH>
__device__ __forceinline__ void res_private(const PhaseArgs<T> &a, const ResTile<T> &t, const ResRow &R,
                                            const ResVec &V, int i0, ResPriv<T, VX> &pv) {
    T *const *psi = t.g->psi[EPH ? 0 : 1];
    const unsigned mx = (R.flags & kRowMx) ? res_lanes(V, 3) : 0u, my = (R.flags & kRowMy) ? res_lanes(V, 4) : 0u,
                   mz = (R.flags & kRowMz) ? res_lanes(V, 5) : 0u;
    if (EPH || ((V.lanes & kVecS) | (R.flags & (kRowSy | kRowSz)))) ldv<T, VX>(pv.m, a.m + R.c + i0);
    else zerov<T, VX>(pv.m);
#pragma unroll
    for (int w = 0; w < 2; w++) {
        if (mx) {
            const T *p = psi[w] + R.ox + V.lx;
#pragma unroll
            for (int v = 0; v < VX; v++) pv.q[w][v] = (mx >> v & 1) ? p[v] : T(0);
        } else {
            zerov<T, VX>(pv.q[w]);
        }
        if (my) res_ld_psi<T, VX>(pv.q[2 + w], psi[2 + w] + R.oy + i0, my);
        else zerov<T, VX>(pv.q[2 + w]);
        if (mz) res_ld_psi<T, VX>(pv.q[4 + w], psi[4 + w] + R.oz + i0, mz);
        else zerov<T, VX>(pv.q[4 + w]);
    }
}

// One cell vector of a phase.  EPH: E from H, else H from E; both are
//   F = ca F + s cb curl(G) and the psi terms,
// with the window of four taps starting at -2 (E) or -1 (H).  EDGE: rows of
// the exchange.
template <typename T, int VX, bool EPH, bool EDGE>
__device__ __forceinline__ void res_cells(const ResArgs<T> &ra, const PhaseArgs<T> &a, const ResTile<T> &t,
                                          const ResRow &R, const ResVec &V, int vi, int n, int s,
                                          ResPriv<T, VX> &pv) {
    constexpr int W = EPH ? -2 : -1;  // first tap
    constexpr int GB = EPH ? 3 : 0, FB = EPH ? 0 : 3;
    const int pitch = t.pitch, fs = t.rmax * pitch, i0 = vi * VX;
    const int o = (int)(R.flags & 0xffffu) * pitch + i0, c = R.c + i0;
    const T c1 = a.c1, c2 = a.c2;
    const bool vy = R.flags & kRowVy, vz = R.flags & kRowVz;
    const unsigned mx = (R.flags & kRowMx) ? res_lanes(V, 3) : 0u, my = (R.flags & kRowMy) ? res_lanes(V, 4) : 0u,
                   mz = (R.flags & kRowMz) ? res_lanes(V, 5) : 0u;

    T *const *psi = t.g->psi[EPH ? 0 : 1];
    T(&m)[VX] = pv.m;
    T(&q)[6][VX] = pv.q;
    T dm[VX];
    if constexpr (!EPH) {
        if (a.dtmu) {
            ldv<T, VX>(dm, a.dtmu + c);
        } else {
#pragma unroll
            for (int v = 0; v < VX; v++) dm[v] = a.dtmu0;
        }
    }
    const T *const gx = t.s + GB * fs + o, *const gy = gx + fs, *const gz = gy + fs;
    T tap[12][VX];  // G_z, G_x beside the centre along y, then G_x, G_y along z
    if constexpr (EDGE) {
#pragma unroll
        for (int w = 0; w < 12; w++) {
            const int w3 = w % 3, d = W + w3 + (w3 >= -W);  // offset beside 0
            const bool remote = R.tap[w] == kTapRemote;
            if ((w < 6 ? vy : vz) && !remote) ld_plain<T, VX>(tap[w], t.s + i0 + (int)R.tap[w] * pitch);
            else zerov<T, VX>(tap[w]);
            ld_remote(tap[w], t.g->f[GB + (w < 3 ? 2 : (w < 9 ? 0 : 1))] + (c + d * (w < 6 ? a.px : (int)a.plane)), remote);
        }
    } else {
        const int zs = t.nry * pitch;
        if (vy) {
#pragma unroll
            for (int w = 0; w < 3; w++) {
                const int d = (W + w + (w >= -W)) * pitch;
                ld_plain<T, VX>(tap[w], gz + d);
                ld_plain<T, VX>(tap[3 + w], gx + d);
            }
        } else {
#pragma unroll
            for (int w = 0; w < 6; w++) zerov<T, VX>(tap[w]);
        }
        if (vz) {
#pragma unroll
            for (int w = 0; w < 3; w++) {
                const int d = (W + w + (w >= -W)) * zs;
                ld_plain<T, VX>(tap[6 + w], gx + d);
                ld_plain<T, VX>(tap[9 + w], gy + d);
            }
        } else {
#pragma unroll
            for (int w = 6; w < 12; w++) zerov<T, VX>(tap[w]);
        }
    }
    // difference d4(w2, w1, w3, w0) of the window [W .. W + 3]: the centre is
    // w2 on E and w1 on H
    auto diff = [&](T ctr, T t0, T t1, T t2) { return EPH ? d4(c1, c2, ctr, t1, t2, t0) : d4(c1, c2, t1, ctr, t2, t0); };
    const bool xl = i0 >= VX, xr = i0 + VX < a.nx;
    T dyz[VX], dyx[VX], dzx[VX], dzy[VX], dxz[VX], dxy[VX], dxt[VX];
    {
        T g[VX];
        ld_plain<T, VX>(g, gx);
#pragma unroll
        for (int v = 0; v < VX; v++) {
            dyx[v] = vy ? diff(g[v], tap[3][v], tap[4][v], tap[5][v]) : T(0);
            dzx[v] = vz ? diff(g[v], tap[6][v], tap[7][v], tap[8][v]) : T(0);
        }
    }
    auto xwindow = [&](T(&w)[3 * VX], const T *src) {
        T v3[3][VX];
        ld_plain<T, VX>(v3[1], src);
        if (xl) ld_plain<T, VX>(v3[0], src - VX);
        else zerov<T, VX>(v3[0]);
        if (xr) ld_plain<T, VX>(v3[2], src + VX);
        else zerov<T, VX>(v3[2]);
#pragma unroll
        for (int v = 0; v < VX; v++) {
            w[v] = v3[0][v];
            w[VX + v] = v3[1][v];
            w[2 * VX + v] = v3[2][v];
        }
    };
    {
        T w[3 * VX];
        xwindow(w, gz);
#pragma unroll
        for (int v = 0; v < VX; v++) {
            const int xc = VX + v + W;
            dyz[v] = vy ? diff(w[VX + v], tap[0][v], tap[1][v], tap[2][v]) : T(0);
            dxz[v] = d4(c1, c2, w[xc + 2], w[xc + 1], w[xc + 3], w[xc]);
            dxt[v] = dxz[v];
        }
        if constexpr (!EPH)  // psi_Hyx stencil (cpu_cpml4.f90:400)
            if (mx) {
#pragma unroll
                for (int v = 0; v < VX; v++) {
                    const int xc = VX + v + W;
                    dxt[v] = fma(c2, w[xc + 3] - w[xc], fma(c1, w[xc + 2], -(a.c2t * w[xc + 1])));
                }
            }
        xwindow(w, gy);
#pragma unroll
        for (int v = 0; v < VX; v++) {
            const int xc = VX + v + W;
            dzy[v] = vz ? diff(w[VX + v], tap[9][v], tap[10][v], tap[11][v]) : T(0);
            dxy[v] = d4(c1, c2, w[xc + 2], w[xc + 1], w[xc + 3], w[xc]);
        }
    }
    const bool full = (V.lanes & kVecFull) && (R.flags & (7u * kRowU0)) == 7u * kRowU0;
    if (!full) {
        const unsigned vx = res_lanes(V, 6);
#pragma unroll
        for (int v = 0; v < VX; v++)
            if (!(vx >> v & 1)) dxz[v] = dxy[v] = dxt[v] = T(0);
    }

    constexpr int SH = EPH ? 0 : 1, PB = EPH ? 2 : 4, PC = EPH ? 3 : 5, IK = EPH ? 6 : 7;
    const ResProf<T> py = res_prof(t.yp + 4 * ((EPH ? 0 : t.nry) + R.jl)), pz = res_prof(t.zp + 4 * ((EPH ? 0 : t.nrz) + R.kl));
    T ik_x[VX];
    ld_plain<T, VX>(ik_x, t.xp + IK * pitch + i0);
    const T sg = EPH ? a.sgn : -a.sgn;
    T f[3][VX], e[3][VX], cb[3][VX];  // old values, ca times them, cb
#pragma unroll
    for (int w = 0; w < 3; w++) {
        ld_plain<T, VX>(f[w], t.s + (FB + w) * fs + o);
#pragma unroll
        for (int v = 0; v < VX; v++) {
            e[w][v] = f[w][v];
            cb[w][v] = EPH ? m[v] : dm[v];
        }
    }
    if (V.lanes & kVecS) {
        T sh[VX];
        ld_plain<T, VX>(sh, t.xp + SH * pitch + i0);
#pragma unroll
        for (int v = 0; v < VX; v++)
            if (sh[v] != T(0)) res_coef(sh[v], m[v], cb[0][v], f[0][v], e[0][v]);
    }
    if (R.flags & kRowSy) {
#pragma unroll
        for (int v = 0; v < VX; v++) res_coef(py.sh, m[v], cb[1][v], f[1][v], e[1][v]);
    }
    if (R.flags & kRowSz) {
#pragma unroll
        for (int v = 0; v < VX; v++) res_coef(pz.sh, m[v], cb[2][v], f[2][v], e[2][v]);
    }
#pragma unroll
    for (int v = 0; v < VX; v++) {
        e[0][v] = fma(sg * cb[0][v], curl2(dyz[v], py.ik, dzy[v], pz.ik), e[0][v]);
        e[1][v] = fma(sg * cb[1][v], curl2(dzx[v], pz.ik, dxz[v], ik_x[v]), e[1][v]);
        e[2][v] = fma(sg * cb[2][v], curl2(dxy[v], ik_x[v], dyx[v], py.ik), e[2][v]);
    }
    if (!full) {  // cells outside a component's update range keep its value
#pragma unroll
        for (int w = 0; w < 3; w++) {
            const unsigned u = (R.flags & (kRowU0 << w)) ? res_lanes(V, w) : 0u;
#pragma unroll
            for (int v = 0; v < VX; v++)
                if (!(u >> v & 1)) e[w][v] = f[w][v];
        }
    }
    // psi terms: + then - on E, - then + on H
    if (mx) {
        T b[VX], g[VX];
        ld_plain<T, VX>(b, t.xp + PB * pitch + i0);
        ld_plain<T, VX>(g, t.xp + PC * pitch + i0);
        T *p0 = psi[0] + R.ox + V.lx, *p1 = psi[1] + R.ox + V.lx;
#pragma unroll
        for (int v = 0; v < VX; v++)
            if (mx >> v & 1) {
                q[0][v] = fma(b[v], q[0][v], g[v] * dxy[v]);
                q[1][v] = fma(b[v], q[1][v], g[v] * dxt[v]);
                e[2][v] = fma(EPH ? cb[2][v] : -cb[2][v], q[0][v], e[2][v]);
                e[1][v] = fma(EPH ? -cb[1][v] : cb[1][v], q[1][v], e[1][v]);
                p0[v] = q[0][v];
                p1[v] = q[1][v];
            }
    }
    if (my) {
#pragma unroll
        for (int v = 0; v < VX; v++)
            if (my >> v & 1) {
                q[2][v] = fma(py.b, q[2][v], py.g * dyz[v]);
                q[3][v] = fma(py.b, q[3][v], py.g * dyx[v]);
                e[0][v] = fma(EPH ? cb[0][v] : -cb[0][v], q[2][v], e[0][v]);
                e[2][v] = fma(EPH ? -cb[2][v] : cb[2][v], q[3][v], e[2][v]);
            }
        st_psi<T, VX>(psi[2], R.oy + i0, q[2], my);
        st_psi<T, VX>(psi[3], R.oy + i0, q[3], my);
    }
    if (mz) {
#pragma unroll
        for (int v = 0; v < VX; v++)
            if (mz >> v & 1) {
                q[4][v] = fma(pz.b, q[4][v], pz.g * dzx[v]);
                q[5][v] = fma(pz.b, q[5][v], pz.g * dzy[v]);
                e[1][v] = fma(EPH ? cb[1][v] : -cb[1][v], q[4][v], e[1][v]);
                e[0][v] = fma(EPH ? -cb[0][v] : cb[0][v], q[5][v], e[0][v]);
            }
        st_psi<T, VX>(psi[4], R.oz + i0, q[4], mz);
        st_psi<T, VX>(psi[5], R.oz + i0, q[5], mz);
    }
    // the history holds E after its electric points and H before the next
    // step's magnetic points
    T *const hist = ra.hist ? t.g->hist : nullptr;
    if (!EPH && hist) {
#pragma unroll
        for (int w = 0; w < 3; w++)
            stv_stream<T, VX>(hist + (s + 1) * ra.hist_slot + (FB + w) * ra.hist_comp + c, e[w]);
    }
    const bool ringed = EPH && a.ring_k > 0;
    if (ringed) {
#pragma unroll
        for (int w = 0; w < 3; w++)
            if (a.vmask >> w & 1)
                stv_stream<T, VX>(a.ring + ring_index(a.ring_comp, a.ring_k, w, t.shot * a.fshot + c, n % a.ring_k), e[w]);
    }
#pragma unroll 1
    for (int k = 0; k < t.npt; k++) {  // the shot's points in this tile
        const ResPt pt = t.pts[k];
        if (pt.off < o || pt.off >= o + VX || (pt.kind == 1) != EPH) continue;
        if (!EPH && s + 1 >= ra.nsteps) continue;
        const double w = EPH ? (ra.wave[n] + ra.wave[n + 1]) / 2.0 : ra.wave[n + 2];
        const T add = (T)(-mul_rn(pt.g, w));
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
            for (int v = 0; v < VX; v++)
                if (pt.comp == FB + p && pt.off == o + v) {
                    if (!EPH) t.pre[k] = e[p][v];
                    if (ringed && (a.vmask >> p & 1))  // the ring's value of the cell, rounded as inject_kernel rounds it
                        a.ring[ring_index(a.ring_comp, a.ring_k, p, t.shot * a.fshot + c + v, n % a.ring_k)] =
                            inject_ring(e[p][v], pt.g, w);
                    e[p][v] = add_rn(e[p][v], add);
                }
    }
    if (EPH && hist) {
#pragma unroll
        for (int w = 0; w < 3; w++)
            stv_stream<T, VX>(hist + (s + 1) * ra.hist_slot + (FB + w) * ra.hist_comp + c, e[w]);
    }
#pragma unroll
    for (int w = 0; w < 3; w++) stv<T, VX>(t.s + (FB + w) * fs + o, e[w]);
    if constexpr (EDGE) {  // rows the neighbours read: x and z components along y, x and y along z
        if (R.flags & (kRowPy | kRowPz)) stv<T, VX>(t.g->f[FB + 0] + c, e[0]);
        if (R.flags & kRowPz) stv<T, VX>(t.g->f[FB + 1] + c, e[1]);
        if (R.flags & kRowPy) stv<T, VX>(t.g->f[FB + 2] + c, e[2]);
    }
}

// Waits until a neighbour has raised its flag f (null: none) to `target`;
// false when this CTA must leave.
__device__ __forceinline__ bool res_poll(const unsigned *f, unsigned target, int *err, unsigned long long wait_ns) {
    if (!f) return true;
    unsigned long long t0 = 0;
    for (unsigned spin = 0; (int)(ld_acquire_gpu(f) - target) < 0; spin++) {
        if ((spin & 255u) != 255u) continue;
        const unsigned long long now = global_ns();
        if (!t0) t0 = now;
        if (*(volatile int *)err & 4) return false;
        if (now - t0 > wait_ns) {
            atomicOr(err, 4);
            return false;
        }
    }
    return true;
}

// Receiver samples of the components [3 EB, 3 EB + 3) after step n.
template <typename T, bool E>
__device__ __forceinline__ void res_sample(const ResArgs<T> &ra, const ResTile<T> &t, const ResRec *cache,
                                           const ResRec *list, int cnt, int n) {
    for (int q = threadIdx.x; q < cnt; q += ResShape<T>::NT) {
        const ResRec r = q < kResRecCache ? cache[q] : list[q];
        if ((r.comp < 3) != E) continue;
        T v = t.s[r.comp * t.rmax * t.pitch + r.off];
        if (!E)  // the next step's magnetic point is in already: the value before it
            for (int w = t.npt - 1; w >= 0; w--)
                if (t.pts[w].kind == 0 && t.pts[w].comp == r.comp && t.pts[w].off == r.off) v = t.pre[w];
        ra.traces[((long long)t.shot * ra.nrec + r.rec) * ra.nt + n] = v;
    }
}

// How a CTA talks to its neighbours: this tile's flag, the flag this thread
// waits for (null: none) and the phases done.
struct ResLink {
    unsigned *mine;
    const unsigned *nb;
    unsigned ph;
};
__device__ __forceinline__ void res_raise(const ResLink &L) {
    if (threadIdx.x == 0) {
        __threadfence();
        st_release_gpu(L.mine, L.ph + 1u);
    }
}

// This thread's first item of a phase: private values.
template <typename T, bool EPH>
__device__ __forceinline__ void res_first(const PhaseArgs<T> &a, const ResTile<T> &t,
                                          ResPriv<T, ResShape<T>::VX> &pv) {
    constexpr int VX = ResShape<T>::VX, P = EPH ? 0 : 1;
    const int x = threadIdx.x;
    if (x >= t.items) return;
    const int r = res_row(t, x), vi = x - r * t.nvec;
    res_private<T, VX, EPH>(a, t, t.rows[P][r], t.vecs[P][vi], vi * VX, pv);
}

// One phase of the tile: the rows of the exchange, then the inner rows, then
// the wait for the neighbours (before it, the private values of the next
// phase's first cells).  pv: this phase's.  False when this CTA must leave.
template <typename T, bool EPH>
__device__ __forceinline__ bool res_phase(const ResArgs<T> &ra, const ResTile<T> &t, ResLink &L,
                                          ResPriv<T, ResShape<T>::VX> &pv, int n, int s) {
    constexpr int VX = ResShape<T>::VX, NT = ResShape<T>::NT, P = EPH ? 0 : 1;
    const PhaseArgs<T> &a = EPH ? ra.e : ra.h;
    const int edge = t.edge[P];
    bool raised = false;
#pragma unroll 1
    for (int base = 0; base < t.items; base += NT) {
        const int x = base + (int)threadIdx.x;
        if (x < t.items) {
            const int r = res_row(t, x), vi = x - r * t.nvec;
            const ResRow R = t.rows[P][r];
            const ResVec V = t.vecs[P][vi];
            if (base > 0) res_private<T, VX, EPH>(a, t, R, V, vi * VX, pv);
            if (x < edge)
                res_cells<T, VX, EPH, true>(ra, a, t, R, V, vi, n, s, pv);
            else
                res_cells<T, VX, EPH, false>(ra, a, t, R, V, vi, n, s, pv);
        }
        if (!raised && base + NT >= edge) {
            __syncthreads();
            res_raise(L);
            raised = true;
        }
    }
    res_first<T, !EPH>(EPH ? ra.h : ra.e, t, pv);
    const bool ok = res_poll(L.nb, L.ph + 1u + ra.expect_more, ra.err, ra.wait_ns);
    L.ph++;
    return __syncthreads_and(ok) != 0;
}

// The row and vector tables of a tile (rows of the exchange first).
template <typename T>
__device__ __forceinline__ void res_tables(const ResArgs<T> &ra, const ResTile<T> &t, ResRow *rows, ResVec *vecs,
                                           int j0, int k0, bool ylo, bool yhi, bool zlo, bool zhi, int *s_edge) {
    constexpr int VX = ResShape<T>::VX, NT = ResShape<T>::NT;
    const int nrow = t.nry * t.nrz, rmax = t.rmax;
    auto is_edge = [&](bool eph, int r) {
        const int kl = r / t.nry, jl = r - kl * t.nry;
        return res_exchanged(eph, jl, t.nry, ylo, yhi) || res_exchanged(eph, kl, t.nrz, zlo, zhi);
    };
    if (threadIdx.x < 2) s_edge[threadIdx.x] = 0;
    __syncthreads();
    for (int q = threadIdx.x; q < 2 * nrow; q += NT)
        if (is_edge(q < nrow, q < nrow ? q : q - nrow)) atomicAdd(&s_edge[q < nrow ? 0 : 1], 1);
    __syncthreads();
    for (int q = threadIdx.x; q < 2 * nrow; q += NT) {
        const bool eph = q < nrow;
        const PhaseArgs<T> &a = eph ? ra.e : ra.h;
        const int r = eph ? q : q - nrow, kl = r / t.nry, jl = r - kl * t.nry, j = j0 + jl, k = k0 + kl;
        int before = 0;
        for (int w = 0; w < r; w++) before += is_edge(eph, w);
        const int W = eph ? -2 : -1, GB = eph ? 3 : 0;
        const int ly = slab_local(a.slab[1], j), lz = slab_local(a.slab[2], k);
        ResRow R;
        R.flags = (unsigned)r;
        if (j + W >= 0 && j + W + 3 < a.ny) R.flags |= kRowVy;
        if (k + W >= 0 && k + W + 3 < a.nz) R.flags |= kRowVz;
#pragma unroll
        for (int u = 0; u < 3; u++)
            if (j >= a.upd[u].lo[1] && j < a.upd[u].hi[1] && k >= a.upd[u].lo[2] && k < a.upd[u].hi[2])
                R.flags |= kRowU0 << u;
        const DBox &o0 = a.slab[0].other, &o1 = a.slab[1].other, &o2 = a.slab[2].other;
        if (j >= o0.lo[1] && j < o0.hi[1] && k >= o0.lo[2] && k < o0.hi[2]) R.flags |= kRowMx;
        if (ly >= 0 && k >= o1.lo[2] && k < o1.hi[2]) R.flags |= kRowMy;
        if (lz >= 0 && j >= o2.lo[1] && j < o2.hi[1]) R.flags |= kRowMz;
        if (res_exchanged(eph, jl, t.nry, ylo, yhi)) R.flags |= kRowPy;
        if (res_exchanged(eph, kl, t.nrz, zlo, zhi)) R.flags |= kRowPz;
        if (a.prof[(8 + (eph ? 0 : 1)) * a.nmax + j] != T(0)) R.flags |= kRowSy;
        if (a.prof[(16 + (eph ? 0 : 1)) * a.nmax + k] != T(0)) R.flags |= kRowSz;
        R.jl = (unsigned short)jl;
        R.kl = (unsigned short)kl;
        R.c = k * (int)a.plane + j * a.px;
        R.ox = (k * a.ny + j) * a.slab[0].width;
        R.oy = (k * a.slab[1].width + ly) * a.px;
        R.oz = (lz * a.ny + j) * a.px;
        for (int w = 0; w < 12; w++) {
            const int cw = w / 3, comp = GB + (cw == 0 ? 2 : (cw == 3 ? 1 : 0));
            const int d = W + w % 3 + (w % 3 >= -W);  // the offsets beside 0
            const bool along_y = cw < 2;
            const int v = (along_y ? jl : kl) + d, nn = along_y ? t.nry : t.nrz;
            int row;
            if (v >= 0 && v < nn) row = comp * rmax + (along_y ? kl * t.nry + v : v * t.nry + jl);
            else if (!(R.flags & (along_y ? kRowVy : kRowVz))) row = comp * rmax;  // never read
            else row = kTapRemote;
            R.tap[w] = (unsigned short)row;
        }
        rows[(eph ? 0 : rmax) + (is_edge(eph, r) ? before : s_edge[eph ? 0 : 1] + r - before)] = R;
    }
    for (int q = threadIdx.x; q < 2 * t.nvec; q += NT) {
        const bool eph = q < t.nvec;
        const PhaseArgs<T> &a = eph ? ra.e : ra.h;
        const int vi = eph ? q : q - t.nvec, i0 = vi * VX, W = eph ? -2 : -1;
        ResVec V;
        V.lanes = kVecFull;
        V.lx = 0;
        for (int v = 0; v < VX; v++) {
            const int i = i0 + v;
            const int l = slab_local(a.slab[0], i);
            auto set = [&](int which, bool on) { V.lanes |= (unsigned)on << (4 * which + v); };
            auto need = [&](int which, bool on) {
                set(which, on);
                if (!on) V.lanes &= ~kVecFull;
            };
            need(0, i >= a.upd[0].lo[0] && i < a.upd[0].hi[0]);
            need(1, i >= a.upd[1].lo[0] && i < a.upd[1].hi[0]);
            need(2, i >= a.upd[2].lo[0] && i < a.upd[2].hi[0]);
            set(3, l >= 0);
            set(4, i >= a.slab[1].other.lo[0] && i < a.slab[1].other.hi[0]);
            set(5, i >= a.slab[2].other.lo[0] && i < a.slab[2].other.hi[0]);
            need(6, i + W >= 0 && i + W + 3 < a.nx);
            if (i < a.nx && a.prof[(eph ? 0 : 1) * a.nmax + i] != T(0)) V.lanes |= kVecS;
            // lanes of a vector in the slab are consecutive there: the two
            // intervals lie at least four cells apart (2 ncpml + 4 <= nx)
            if (l >= 0) V.lx = l - v;
        }
        vecs[q] = V;
    }
}

template <typename T>
__global__ void __launch_bounds__(ResShape<T>::NT, 1) resident_kernel(const __grid_constant__ ResArgs<T> ra) {
    constexpr int VX = ResShape<T>::VX, NT = ResShape<T>::NT;
    extern __shared__ __align__(16) unsigned char res_smem[];
    __shared__ int s_npt, s_edge[2];
    const PhaseArgs<T> &a = ra.e;
    const int tiles = ra.ty * ra.tz;
    const int group = (int)blockIdx.x / tiles, tile = (int)blockIdx.x - group * tiles;
    const int tyi = tile % ra.ty, tzi = tile / ra.ty;
    const int j0 = ra.ys[tyi], k0 = ra.zs[tzi];
    const bool ylo = tyi > 0, yhi = tyi + 1 < ra.ty, zlo = tzi > 0, zhi = tzi + 1 < ra.tz;
    using S = ResSmem<T>;
    ResTile<T> t;
    t.rmax = ra.nrow;
    t.pitch = ra.pitch;
    t.nvec = (a.nx + VX - 1) / VX;
    t.inv_nvec = 1.0f / (float)t.nvec;
    t.nry = ra.ys[tyi + 1] - j0;
    t.nrz = ra.zs[tzi + 1] - k0;
    t.items = t.nry * t.nrz * t.nvec;
    unsigned char *sp = res_smem;
    auto take = [&](size_t n) {
        unsigned char *q = sp;
        sp += n;
        return q;
    };
    t.s = reinterpret_cast<T *>(take(S::rows(ra.nrow, ra.pitch)));
    T *xp = reinterpret_cast<T *>(take(S::xprof(ra.pitch)));
    T *yp = reinterpret_cast<T *>(take(S::yzprof(ra.rymax, ra.rzmax))), *zp = yp + 8 * t.nry;
    ResRow *rows = reinterpret_cast<ResRow *>(take((size_t)2 * t.rmax * sizeof(ResRow)));
    ResVec *vecs = reinterpret_cast<ResVec *>(take(S::a16((size_t)2 * (ra.pitch / VX) * sizeof(ResVec))));
    ResPtrs<T> *gp = reinterpret_cast<ResPtrs<T> *>(take(S::a16(sizeof(ResPtrs<T>))));
    ResPt *pts = reinterpret_cast<ResPt *>(take(kResMaxPts * sizeof(ResPt)));
    t.pre = reinterpret_cast<T *>(take(S::a16(kResMaxPts * sizeof(T))));
    ResRec *cache = reinterpret_cast<ResRec *>(take(S::a16(kResRecCache * sizeof(ResRec))));
    t.xp = xp;
    t.yp = yp;
    t.zp = zp;
    t.rows[0] = rows;
    t.rows[1] = rows + t.rmax;
    t.vecs[0] = vecs;
    t.vecs[1] = vecs + t.nvec;
    t.g = gp;
    t.pts = pts;

    ResLink L;
    L.mine = ra.flags + (size_t)blockIdx.x * kResFlagStride;
    L.nb = nullptr;
    if (threadIdx.x == 0 && ylo) L.nb = L.mine - kResFlagStride;
    if (threadIdx.x == 1 && yhi) L.nb = L.mine + kResFlagStride;
    if (threadIdx.x == 2 && zlo) L.nb = L.mine - (size_t)ra.ty * kResFlagStride;
    if (threadIdx.x == 3 && zhi) L.nb = L.mine + (size_t)ra.ty * kResFlagStride;
    L.ph = 0;

    res_tables<T>(ra, t, rows, vecs, j0, k0, ylo, yhi, zlo, zhi, s_edge);
    for (int q = threadIdx.x; q < 8 * t.pitch; q += NT) {
        const int w = q / t.pitch, i = q - w * t.pitch;
        xp[q] = i < a.nx ? a.prof[w * a.nmax + i] : T(0);
    }
    // {sh, 1/kd, b, c/d}: profile arrays 0 6 2 3 of E, 1 7 4 5 of H
    for (int q = threadIdx.x; q < 8 * (t.nry + t.nrz); q += NT) {
        const bool y = q < 8 * t.nry;
        const int x = y ? q : q - 8 * t.nry, nn = y ? t.nry : t.nrz;
        const int ph = x / (4 * nn), v = (x - ph * 4 * nn) / 4, w = x & 3;
        const int which = w == 0 ? ph : (w == 1 ? 6 + ph : (w == 2 ? 2 + 2 * ph : 3 + 2 * ph));
        yp[q] = a.prof[((y ? 8 : 16) + which) * a.nmax + (y ? j0 : k0) + v];
    }
    const int r0 = ra.traces ? ra.rec_start[tile] : 0, nr = ra.traces ? ra.rec_start[tile + 1] - r0 : 0;
    for (int q = threadIdx.x; q < nr && q < kResRecCache; q += NT) cache[q] = ra.recs[r0 + q];
    __syncthreads();
    t.edge[0] = s_edge[0] * t.nvec;
    t.edge[1] = s_edge[1] * t.nvec;

    for (int shot = group; shot < ra.nshot; shot += ra.groups) {
        t.shot = shot;
        const long long sb = (long long)shot * a.fshot;
        if (threadIdx.x < 6) {
            gp->f[threadIdx.x] = a.f[threadIdx.x] + sb;
            gp->psi[0][threadIdx.x] = ra.e.psi[threadIdx.x >> 1][threadIdx.x & 1] + shot * ra.e.pshot[threadIdx.x >> 1];
            gp->psi[1][threadIdx.x] = ra.h.psi[threadIdx.x >> 1][threadIdx.x & 1] + shot * ra.h.pshot[threadIdx.x >> 1];
            if (threadIdx.x == 0) gp->hist = ra.hist ? ra.hist + sb : nullptr;
        }
        // the tile's state, and the shot's points that lie in it, in their order
        for (int x = threadIdx.x; x < t.items; x += NT) {
            const int row = x / t.nvec, i0 = (x - row * t.nvec) * VX;
            const int kl = row / t.nry, jl = row - kl * t.nry;
            const long long c = sb + (k0 + kl) * a.plane + (long long)(j0 + jl) * a.px + i0;
#pragma unroll
            for (int f = 0; f < 6; f++) {
                T v[VX];
                ldf<T, VX, true>(v, a.f[f] + c);
                stv<T, VX>(t.s + (f * t.rmax + row) * t.pitch + i0, v);
            }
        }
        if (threadIdx.x < 32) {
            int cnt = 0;
            for (int q0 = 0; q0 < ra.npts; q0 += 32) {
                const int q = q0 + (int)threadIdx.x;
                bool in = false;
                ResPt pt;
                if (q < ra.npts) {
                    const SrcPoint s = ra.pts[q];
                    const long long cell = s.off - sb;
                    if (cell >= 0 && cell < a.fshot) {
                        const int k = (int)(cell / a.plane), rem = (int)(cell - k * a.plane);
                        const int j = rem / a.px, jl = j - j0, kl = k - k0;
                        in = jl >= 0 && jl < t.nry && kl >= 0 && kl < t.nrz;
                        pt.g = s.g;
                        pt.off = (kl * t.nry + jl) * t.pitch + rem - j * a.px;
                        pt.comp = s.comp;
                        pt.kind = s.kind;
                        pt.pad = 0;
                    }
                }
                const unsigned bal = __ballot_sync(0xffffffffu, in);
                const int at = cnt + __popc(bal & ((1u << threadIdx.x) - 1u));
                if (in && at < kResMaxPts) pts[at] = pt;
                cnt += __popc(bal);
            }
            if (threadIdx.x == 0) s_npt = min(cnt, kResMaxPts);
        }
        __syncthreads();
        t.npt = s_npt;
        if (threadIdx.x == 0)  // the first step's magnetic points, for this tile and its neighbours
            for (int q = 0; q < t.npt; q++) {
                const ResPt pt = pts[q];
                if (pt.kind != 0) continue;
                T *cell = t.s + pt.comp * t.rmax * t.pitch + pt.off;
                const T v = add_rn(*cell, (T)(-mul_rn(pt.g, ra.wave[ra.n0 + 1])));
                *cell = v;
                const int row = pt.off / t.pitch, kl = row / t.nry, jl = row - kl * t.nry;
                gp->f[pt.comp][(k0 + kl) * a.plane + (long long)(j0 + jl) * a.px + (pt.off - row * t.pitch)] = v;
            }
        res_raise(L);
        ResPriv<T, VX> pv;
        res_first<T, true>(ra.e, t, pv);
        const bool ok = res_poll(L.nb, L.ph + 1u + ra.expect_more, ra.err, ra.wait_ns);
        L.ph++;
        if (!__syncthreads_and(ok)) return;
#pragma unroll 1
        for (int s = 0; s < ra.nsteps; s++) {
            const int n = ra.n0 + s;
            if (nr > 0 && s > 0) res_sample<T, false>(ra, t, cache, ra.recs + r0, nr, n - 1);
            if (!res_phase<T, true>(ra, t, L, pv, n, s)) return;
            if (nr > 0) res_sample<T, true>(ra, t, cache, ra.recs + r0, nr, n);
            if (!res_phase<T, false>(ra, t, L, pv, n, s)) return;
        }
        if (nr > 0) {
            t.npt = 0;  // the last step leaves the next magnetic points to the next launch
            res_sample<T, false>(ra, t, cache, ra.recs + r0, nr, ra.n0 + ra.nsteps - 1);
        }
        // the rows that the exchange has not left in global memory already
        for (int x = threadIdx.x; x < t.items; x += NT) {
            const int row = x / t.nvec, i0 = (x - row * t.nvec) * VX;
            const int kl = row / t.nry, jl = row - kl * t.nry;
            const int c = (k0 + kl) * (int)a.plane + (j0 + jl) * a.px + i0;
            const bool ey = res_exchanged(true, jl, t.nry, ylo, yhi), ez = res_exchanged(true, kl, t.nrz, zlo, zhi);
            const bool hy = res_exchanged(false, jl, t.nry, ylo, yhi), hz = res_exchanged(false, kl, t.nrz, zlo, zhi);
            const bool done[6] = {ey || ez, ez, ey, hy || hz, hz, hy};
#pragma unroll
            for (int f = 0; f < 6; f++) {
                if (done[f]) continue;
                T v[VX];
                ld_plain<T, VX>(v, t.s + (f * t.rmax + row) * t.pitch + i0);
                stv<T, VX>(gp->f[f] + c, v);
            }
        }
        __syncthreads();
    }
}

// Tiling of one solve; ok = false where the fields do not fit.
struct ResPlan {
    bool ok = false;
    int ty = 0, tz = 0, groups = 0;
    int nrow = 0, ry = 0, rz = 0, pitch = 0;  // rows of the largest tile; most rows along y, z; elements per row
    unsigned short ys[kResMaxTiles + 1], zs[kResMaxTiles + 1];
    size_t smem = 0;                          // bytes
    int steps = 0;                            // most steps of one launch
};

// The tiling for nshot shots on nsm SMs (resident.cu); heavy_y, heavy_z: rows
// whose cells carry a CPML profile or psi.
template <typename T>
ResPlan resident_plan(int nx, int ny, int nz, const unsigned char *heavy_y, const unsigned char *heavy_z, int nshot,
                      int nsm);

// Limits of the launch's waits (resident.cu): MITTET_PERSIST_WAIT_MS, and with
// MITTET_RESIDENT_STALL=1 every wait asks for a phase that nobody finishes, so
// that a test can watch the waits give up.
template <typename T>
void resident_waits(ResArgs<T> *a);

// One cooperative launch of a.nsteps steps (resident.cu).
template <typename T>
cudaError_t resident_launch(const ResArgs<T> &a, const ResPlan &p, cudaStream_t st);

}  // namespace mittet
