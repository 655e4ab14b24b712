// adjoint.cuh -- discrete adjoint of the forward step, for the FWI gradient.
//
// The forward step is linear in the state (E, H, psi_E, psi_H) for a fixed
// model; its transpose is applied step by step in reverse time.  The adjoint
// fields are kept scaled by the update coefficient of their own cell,
//   A = cb lambda_E  (cb = m/(1+h), h = esig m/2, m = 2 w0 dt/sigma),
//   B = db lambda_H  (db = (dt/mu)/(1+h), h = msig m/2),
// and each psi's adjoint as tau, its value before the recurrence factor b of
// the step it came from.  The transposed half steps are then
//   H phase:  A <- ca A + cb sum_a D+_a^T (s ik_a B + g_a tau_H)
//   E phase:  B <- da B + db sum_a D_a^T  (s ik_a A + g_a tau_E)
// with the signs of the curl, tau <- b tau +- the cell's own A or B in the
// slabs, and D+^T = -D, D^T = -D+: the forward's own stencils (2,4), read at
// the neighbours of one cell and written at that cell alone.  One kernel per
// half step, each cell of an adjoint field read and written once, as in the
// forward; storing the weight of every derivative instead (13 arrays, a
// kernel that writes them and one that gathers them) moved 220 bytes per
// interior cell and step in FP32 where this moves 116 (192 with the FP64
// fields below).
//
// The adjoint fields are FP64 whatever the field precision, so that the error
// of an FP32 gradient is that of its forward fields; the taus, which hold
// values of the CPML alone, keep the field precision (in FP64 the errors below
// are the same to all digits).  Against the FP64 gradient, root mean square
// over 7 seeds on 85x102x80 (5 shots), 64x64x48 (2), 96x80x96 (3) and 64^3
// (2): 4.3e-7, 2.1e-7, 4.8e-7, 4.8e-7; with FP32 fields 9.6e-7, 3.0e-7,
// 8.0e-7, 1.1e-6 (stored weights: 8.4e-7, 2.4e-7, 8.4e-7, 1.1e-6).  It costs
// time on grids that do not fit in L2.  Adjoint stage in ms, FP64 fields, FP32
// fields, FP64 taus too, stored weights: 128x128x96, 16 shots, 60 steps 100, 91,
// 104, 86; 4 shots, 120 steps 52, 47, 54, 48; 64x64x48, 4 shots, 256 steps 22.5,
// 21.3, 24.7, 25.8; FP64 53x46x41, 150 steps 5.7 (stored weights 9.9).  Since
// then adjoint.cu has brought the first column to 96.7, 50.0, 18.0 and 5.7.
//
// Adjoint step n (reverse of forward step n):
//   add the receivers' a_H[n] to B;  H phase (A, tau_E; gradient of the H
//   update);  add a_E[n] to A;  source terms;  E phase (B, tau_H; gradient of
//   the E update).
//
// Gradient of the misfit with respect to sigma.  With the scaled fields every
// factor of the E update's derivative cancels but one:
//   E update, every cell, in range or not:  A (E0 - E1) / (2 w0 dt),
//   H update, cells with a magnetic profile: B h/(dm sigma) (H1 +- H0), + in
//   range, - outside, dm = dt/mu,
//   electric source gain: A h g w / (2 w0 dt);  magnetic: the stored H0 is the
//   one before the injection, so its -g w enters the H term.
// The sums are accumulated per shot in FP64.
#pragma once
#include "kernels.cuh"

namespace mittet {

// A row of a general axis, for the taps W .. W + 3 around it (W = -2 in the H
// phase, -1 in the E phase): stencil weight times the curl's sign times 1/kd
// of the tap, zero outside the update range and the grid (qa, qx of the two
// components the axis carries), stencil weight times c/d (qg, zero outside the
// slab) and the tap's row in the slab (the sign bit set where it has none).
struct __align__(16) AdjTapRow {
    double qa[4], qx[4], qg[4];
    int l[4];
};
// Cells along x, one array each (read as vectors, entry 8 is cell 0): signed
// 1/kd of the z and the y component (zero outside their range), c/d, slab
// index (-1: none).
struct AdjXTab {
    const double *kz, *ky, *cg;
    const int *l;
};

// One transposed half step.  "from" is the field whose neighbours are read
// (B in the H phase, A in the E phase), "own" the one that is updated.
template <typename T>
struct AdjArgs {
    const double *from[3];
    double *own[3];             // [shot][cell]
    const T *ftau[3][2];        // tau of the from field's slab groups (axis, which)
    T *otau[3][2];              // tau of the own field's
    long long fpsi[3], opsi[3];  // elements per shot
    DSlab fslab[3], oslab[3];
    DBox fupd[3], oupd[3];
    const T *S0[3], *S1[3];  // the from field's forward values before and after this step's update
    double *grad;          // [shot][cell]
    const T *m, *dtmu;
    T dtmu0;
    const T *prof;
    int nmax;
    int nx, ny, nz, px;
    long long plane, fshot;
    T c2t;                 // centre weight of the psi_Hyx stencil
    double q[4];           // transposed stencil weights c2, c1, -c1, -c2
    double qk[3][4];       // for cells interior along an axis: q times the sign and 1/d of its first component
    const AdjTapRow *taps[2];  // y, z
    AdjXTab xtab;
    double inv2w0dt;       // 1/(2 w0 dt): 1/sigma = m * inv2w0dt
    double inv_dtmu0;      // 1/dtmu0
};

// Boxes of one transposed half step, as the forward's (stencil.cuh TileMap):
// kind = mask of the axes along which a tap may meet a profile, slab or range
// edge of either field; corners and edges first, since they take longest.
struct AdjBoxes {
    int nbox;
    int lo[19][3], hi[19][3], kind[19];
    int start[20];                     // first CTA
    int nvx[19], rows[19], vecs[19];   // vectors of a row, rows of a plane, vectors in all
};

// Adds a[shot][rec][n] to the scaled adjoint of each receiver of one kind.
template <typename T>
struct AdjInject {
    AdjArgs<T> a;          // the phase that last wrote the field: own, otau
    const long long *rec_off;
    const int *rec_comp;
    const double *asrc;
    int nrec, nshot, nt;
};

struct AdjSrc {
    long long off;   // cell offset within the shot (padded layout)
    int shot, comp, kind, i, j, k;
    double g;        // gain (as SrcPoint::g)
};

// adjoint.cu.  e: the phase whose update is transposed (true E, false H).
template <typename T>
void adj_phase_launch(bool e, const AdjArgs<T> &a, const AdjBoxes &b, int nshot, cudaStream_t st);
template <typename T>
AdjBoxes adj_boxes(int nx, int ny, int nz, const int lo[3], const int hi[3]);
template <typename T>
void adj_inject_launch(bool e, const AdjInject<T> &q, int n, cudaStream_t st);
template <typename T>
void adj_src_launch(bool e, const AdjArgs<T> &a, const AdjSrc *pts, int npts, const double *wave, int n, int shot0,
                    int shot1, cudaStream_t st);

// ---------------------------------------------------------------- sources
// Adjoint sources a[shot][rec][n] = sum_f Re(conj(R[shot][rec][f]) W_rf[n]),
// W_rf[n] = hf dt exp((i-1) sqrt(w0 w_f) n dt) with the H factor on H receivers.
static __global__ void adj_source_kernel(const double2 *__restrict__ R, int ntr, int nrec, int nf, int nt,
                                  const double *__restrict__ omega, double dt, double omega0,
                                  const unsigned char *__restrict__ is_h, int hfac, double *__restrict__ out) {
    const long long tot = (long long)ntr * nt;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < tot; e += (long long)gridDim.x * blockDim.x) {
        const int t = (int)(e / nt), n = (int)(e - (long long)t * nt);
        const bool h = hfac && is_h[t % nrec];
        double acc = 0.0;
        for (int f = 0; f < nf; f++) {
            const double xa = sqrt(omega0 * omega[f]) * (double)n * dt;
            double s, cs;
            sincos(xa, &s, &cs);
            const double e0 = exp(-xa) * dt;
            double wr = e0 * cs, wi = e0 * s;
            if (h) {
                const double r = sqrt(2.0 * omega0 / omega[f]) * 0.70710678118654752440;
                const double a2 = wr * r - wi * r, b2 = wr * r + wi * r;
                wr = a2;
                wi = b2;
            }
            const double2 res = R[(long long)t * nf + f];
            acc += res.x * wr + res.y * wi;  // Re(conj(res) * w)
        }
        out[e] = acc;
    }
}

// Copies the six field arrays of a group of shots into one history slot,
// 16 bytes per thread and iteration (len is a multiple of 32 elements, every
// array 16-byte aligned); blockIdx.y is the field.
template <typename T>
__global__ void __launch_bounds__(256) copy_state_kernel(const T *f0, const T *f1, const T *f2, const T *f3,
                                                         const T *f4, const T *f5, T *dst, long long len) {
    constexpr int VX = 16 / sizeof(T);
    using V = typename VecT<T, VX>::type;
    const int c = blockIdx.y;
    const T *src = c == 0 ? f0 : c == 1 ? f1 : c == 2 ? f2 : c == 3 ? f3 : c == 4 ? f4 : f5;
    const V *__restrict__ s = reinterpret_cast<const V *>(src);
    V *__restrict__ d = reinterpret_cast<V *>(dst + c * len);
    const long long nv = len / VX;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nv; e += (long long)gridDim.x * blockDim.x)
        d[e] = __ldcs(s + e);
}

// grad_out[cell] = sum over shots of grad[shot][cell], zero outside the frame
// [ncpml, n-ncpml) on every axis (satan_i calc_gamma, fwi3d_cpu_function_v1.4.c:2359-2361).
static __global__ void grad_reduce_kernel(const double *__restrict__ g, int nshot, long long fshot, int nx, int ny, int nz,
                                   int px, long long plane, int ncpml, double *__restrict__ out) {
    const long long n = (long long)nx * ny * nz;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(e % nx);
        const int j = (int)((e / nx) % ny);
        const int k = (int)(e / ((long long)nx * ny));
        double s = 0.0;
        if (i >= ncpml && i < nx - ncpml && j >= ncpml && j < ny - ncpml && k >= ncpml && k < nz - ncpml) {
            const long long c = (long long)k * plane + (long long)j * px + i;
            for (int q = 0; q < nshot; q++) s += g[(long long)q * fshot + c];
        }
        out[e] = s;
    }
}

// residual R = S - obs and misfit 0.5 sum |R|^2 (one block reduction per launch, atomically added)
static __global__ void residual_kernel(const double2 *__restrict__ S, const double2 *__restrict__ obs, long long n,
                                double2 *__restrict__ R, double *misfit) {
    double acc = 0.0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const double2 r = make_double2(S[e].x - obs[e].x, S[e].y - obs[e].y);
        R[e] = r;
        acc += 0.5 * (r.x * r.x + r.y * r.y);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(misfit, acc);
}

}  // namespace mittet
