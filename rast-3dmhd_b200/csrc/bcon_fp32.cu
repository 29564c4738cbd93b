// bcon_fp32.cu - BCON, time-step limits and totals for the FP32-bulk state.
//
// The state is stored as FP32 momenta and FP32 deviations rho' = rho - R(k), T' = T - T0(k);
// these kernels rebuild full values in FP64 (R, T0 from the static polytrope), apply the
// reference formulas in FP64 (src/bcon.cpp:12-141, src/step.cpp:122-229) and store the result
// back as FP32 deviations.
#include <cuda_runtime.h>

#include "bcon_fp32.cuh"
#include "r3d_kernels.h"
#include "stage_common.cuh"

namespace r3dk {

__global__ void __launch_bounds__(256) bcon_fp32_kernel(Geometry g, Physics ph, Lines L, Boundary b,
                                                        Background bg, FieldSet32 fs, Scalars* sc,
                                                        int with_dt) {
    __shared__ double red[5 * 8];
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    const int side = blockIdx.z;  // 0 top, 1 bottom
    double m1 = 1e300, m2 = 1e300, m3 = 1e300, m4 = 1e300, mu = 0.0;
    if (i <= g.npx && j <= g.npy && (side == 0 ? g.top_edge : g.bot_edge))  // a slab's interior face has none
        bcon_column_fp32(g, ph, L, b, bg, fs.xout, side, i, j, with_dt != 0, m1, m2, m3, mu);
    if (with_dt) reduce_dt(red, m1, m2, m3, m4, mu, sc);
}

__global__ void __launch_bounds__(256) dt_full_fp32_kernel(Geometry g, Physics ph, Lines L,
                                                           Background bg, FieldSet32 fs, Scalars* sc,
                                                           int only_refold) {
    __shared__ double red[5 * 8];
    if (only_refold && *(volatile int*)&sc->refold == 0) return;  // uniform over the grid
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    double m1 = 1e300, m2 = 1e300, m3 = 1e300, m4 = 1e300, mu = 0.0;
    if (i <= g.npx && j <= g.npy) {
        const double dxy = (L.ddy[j] < L.ddx[i]) ? L.ddy[j] : L.ddx[i];
        for (int k = 1 + blockIdx.z; k <= g.npz; k += gridDim.z) {
            const int64_t n = (int64_t)k * g.plane + (int64_t)j * g.pitch + i;
            const double dd = (L.ddz[k] < dxy) ? L.ddz[k] : dxy;
            double w1, w2, w3, w4, um;
            dt_terms<false>(ph, fs.xin[0][n], fs.xin[1][n], fs.xin[2][n], bg.r[k] + (double)fs.xin[3][n],
                            bg.t[k] + (double)fs.xin[4][n], 0.0, dd, L.rkapa[k], w1, w2, w3, w4, um);
            m1 = fold_min(m1, w1);
            m2 = fold_min(m2, w2);
            m3 = fold_min(m3, w3);
            mu = fold_max(mu, um);
        }
    }
    reduce_dt(red, m1, m2, m3, m4, mu, sc);
}

__global__ void totals_fp32_kernel(Geometry g, Physics ph, Background bg, FieldSet32 fs, Scalars* sc) {
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    double m = 0.0, e = 0.0;
    if (i <= g.npx && j <= g.npy) {
        for (int k = 1 + blockIdx.z; k <= g.npz; k += gridDim.z) {
            const int64_t n = (int64_t)k * g.plane + (int64_t)j * g.pitch + i;
            const double ru = fs.xin[0][n], rv = fs.xin[1][n], rw = fs.xin[2][n];
            const double ro = bg.r[k] + (double)fs.xin[3][n], tt = bg.t[k] + (double)fs.xin[4][n];
            m += ro;
            e += ro * tt * ph.cv + 0.5 * (ru * ru + rv * rv + rw * rw) / ro;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        m += __shfl_xor_sync(0xffffffffu, m, o);
        e += __shfl_xor_sync(0xffffffffu, e, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&sc->mass, m);
        atomicAdd(&sc->energy, e);
    }
}

cudaError_t launch_bcon_fp32(const Geometry& g, const Physics& ph, const Lines& L, const Boundary& b,
                             const Background& bg, const FieldSet32& fs, Scalars* sc, int with_dt,
                             cudaStream_t st) {
    dim3 block(32, 8, 1), grid((g.npx + 31) / 32, (g.npy + 7) / 8, 2);
    bcon_fp32_kernel<<<grid, block, 0, st>>>(g, ph, L, b, bg, fs, sc, with_dt);
    return cudaGetLastError();
}

cudaError_t launch_dt_full_fp32(const Geometry& g, const Physics& ph, const Lines& L,
                                const Background& bg, const FieldSet32& fs, Scalars* sc, cudaStream_t st,
                                int only_refold) {
    dim3 block(32, 8, 1), grid((g.npx + 31) / 32, (g.npy + 7) / 8, (unsigned)min(g.npz, only_refold ? 2 : 64));
    dt_full_fp32_kernel<<<grid, block, 0, st>>>(g, ph, L, bg, fs, sc, only_refold);
    return cudaGetLastError();
}

cudaError_t launch_totals_fp32(const Geometry& g, const Physics& ph, const Background& bg,
                               const FieldSet32& fs, Scalars* sc, cudaStream_t st) {
    dim3 block(32, 8, 1), grid((g.npx + 31) / 32, (g.npy + 7) / 8, (unsigned)min(g.npz, 64));
    totals_fp32_kernel<<<grid, block, 0, st>>>(g, ph, bg, fs, sc);
    return cudaGetLastError();
}

}  // namespace r3dk
