// resident.cu -- tiling and launch of the resident time loop (resident.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "resident.cuh"

namespace mittet {

// Cuts n rows into nt runs of about equal weight (a heavy row weighs 1 +
// weight), two rows at least: a tap reaches the next tile at most.
static void split_rows(int n, const unsigned char *heavy, double weight, int nt, unsigned short *first) {
    double total = 0.0;
    for (int v = 0; v < n; v++) total += 1.0 + weight * heavy[v];
    first[0] = 0;
    double sum = 0.0;
    int v = 0;
    for (int q = 1; q < nt; q++) {
        const double goal = total * q / nt;
        const int lo = first[q - 1] + 2, hi = n - 2 * (nt - q);
        while (v < hi && (v < lo || sum + 0.5 * (1.0 + weight * heavy[v]) < goal)) {
            sum += 1.0 + weight * heavy[v];
            v++;
        }
        first[q] = (unsigned short)v;
    }
    first[nt] = (unsigned short)n;
}

template <typename T>
ResPlan resident_plan(int nx, int ny, int nz, const unsigned char *heavy_y, const unsigned char *heavy_z, int nshot,
                      int nsm) {
    constexpr int VX = ResShape<T>::VX, NT = ResShape<T>::NT;
    constexpr size_t kMaxSmem = 227 * 1024 - 1024;  // dynamic, beside the kernel's few static words
    ResPlan best;
    const int nvec = (nx + VX - 1) / VX, pitch = nvec * VX;
    if (ny > 65535 || nz > 65535) return best;
    nsm = std::min(nsm, kResMaxTiles);
    std::vector<int> sum_y(ny + 1, 0), sum_z(nz + 1, 0);  // heavy rows before a row
    for (int j = 0; j < ny; j++) sum_y[j + 1] = sum_y[j] + heavy_y[j];
    for (int k = 0; k < nz; k++) sum_z[k + 1] = sum_z[k] + heavy_z[k];
    double best_t = 0.0;
    ResPlan p;
    p.ok = true;
    p.pitch = pitch;
    for (double weight : {0.0, 0.4})
        for (p.ty = 1; p.ty <= nsm; p.ty++) {
            if (p.ty > 1 && ny < 2 * p.ty) break;
            split_rows(ny, heavy_y, weight, p.ty, p.ys);
            p.ry = 0;
            for (int q = 0; q < p.ty; q++) p.ry = std::max(p.ry, p.ys[q + 1] - p.ys[q]);
            for (p.tz = 1; p.ty * p.tz <= nsm; p.tz++) {
                if (p.tz > 1 && nz < 2 * p.tz) break;
                split_rows(nz, heavy_z, weight, p.tz, p.zs);
                p.rz = 0;
                for (int q = 0; q < p.tz; q++) p.rz = std::max(p.rz, p.zs[q + 1] - p.zs[q]);
                p.nrow = p.ry * p.rz;
                if (6 * p.nrow >= kTapRemote) continue;  // rows are numbered in 16 bits
                p.smem = ResSmem<T>::bytes(p.nrow, p.ry, p.rz, pitch);
                if (p.smem > kMaxSmem) continue;
                p.groups = std::min(nshot, nsm / (p.ty * p.tz));
                const int rounds = (nshot + p.groups - 1) / p.groups;
                // Microseconds per phase: 2.4 for the exchange, 2.2 for each
                // pass of the slowest CTA over its vectors (more where rows
                // are heavy along y, z or both) and 0.7 for a full one;
                // fitted to 4.4 us (32^3 in 64 tiles), 5.3 (64^3, 128 tiles,
                // one pass), 8.7 (144 tiles, two passes), 13.4 (96^3, three),
                // 14.0 (64^3 in 36 tiles, four), all FP32.  An FP64 phase takes
                // 0.47 to 0.63 of it on 16 tilings (a pass 1.95 us, heavy
                // rows or not), which ranks tilings by their passes alike.
                // Of equal ones fewer tiles along y (long in y: 5.3 us, long
                // in z: 6.2).
                // without the heavy rows' part already no better: the tile with
                // the most rows along y and z exists
                const int nmost = p.ry * p.rz * nvec;
                if (best.ok && rounds * (2.4 + 2.2 * ((nmost + NT - 1) / NT) + 0.04 * p.ty) >= best_t) continue;
                double most = 0.0;
                for (int z = 0; z < p.tz; z++)
                    for (int y = 0; y < p.ty; y++) {
                        const int j0 = p.ys[y], j1 = p.ys[y + 1], k0 = p.zs[z], k1 = p.zs[z + 1];
                        const double hy = (double)(sum_y[j1] - sum_y[j0]) / (j1 - j0), hz = (double)(sum_z[k1] - sum_z[k0]) / (k1 - k0);
                        const int items = (j1 - j0) * (k1 - k0) * nvec;
                        most = std::max(most, 2.2 * ((items + NT - 1) / NT) * (1.0 + 0.3 * (hy + hz)) + 0.7 * items / NT);
                    }
                const double t = rounds * (2.4 + most + 0.04 * p.ty);
                if (best.ok && t >= best_t) continue;
                best_t = t;
                best = p;
            }
        }
    best.steps = best.ok ? std::min(kResidentSteps, std::max(1, (int)(kResidentLaunchUs / (2.0 * best_t)))) : 0;
    return best;
}

template <typename T>
void resident_waits(ResArgs<T> *a) {
    const char *stall = std::getenv("MITTET_RESIDENT_STALL"), *wms = std::getenv("MITTET_PERSIST_WAIT_MS");
    a->expect_more = (stall && std::atoi(stall) == 1) ? 1u << 30 : 0u;
    a->wait_ns = (unsigned long long)((wms ? std::max(1.0, std::atof(wms)) : 2000.0) * 1e6);
}

template <typename T>
cudaError_t resident_launch(const ResArgs<T> &a, const ResPlan &p, cudaStream_t st) {
    // an attribute of the current device's function: set for each launch
    cudaError_t e = cudaFuncSetAttribute(resident_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024);
    if (e != cudaSuccess) return e;
    const int ctas = p.groups * p.ty * p.tz;
    e = cudaMemsetAsync(a.flags, 0, (size_t)ctas * kResFlagStride * sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(ResShape<T>::NT);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, resident_kernel<T>, a);
}

template ResPlan resident_plan<float>(int, int, int, const unsigned char *, const unsigned char *, int, int);
template ResPlan resident_plan<double>(int, int, int, const unsigned char *, const unsigned char *, int, int);
template void resident_waits<float>(ResArgs<float> *);
template void resident_waits<double>(ResArgs<double> *);
template cudaError_t resident_launch<float>(const ResArgs<float> &, const ResPlan &, cudaStream_t);
template cudaError_t resident_launch<double>(const ResArgs<double> &, const ResPlan &, cudaStream_t);

}  // namespace mittet
