// bcon_fp32.cuh - BCON of one column of the FP32-bulk state (src/bcon.cpp:12-141): full values
// rebuilt in FP64 from the static background, the result stored as FP32 deviations.
#pragma once

#include "r3d_kernels.h"
#include "stage_common.cuh"

namespace r3dk {

// The domain's top plane (side 0) or bottom plane (side 1), ghost images included; with dt the
// plane's time-step limits (of the stored values) are folded as well.  The state is read past L1
// (a stage kernel's other CTAs may have written it).
__device__ __forceinline__ void bcon_column_fp32(const Geometry& g, const Physics& ph, const Lines& L,
                                                 const Boundary& b, const Background& bg, float* const* x, int side,
                                                 int i, int j, bool dt, double& m1, double& m2, double& m3, double& mu) {
    const double c13 = ph.c13, c23 = ph.c23, c43 = ph.c43;
    const int k = side == 0 ? 1 : g.npz, dk = side == 0 ? 1 : -1;
    const int64_t base = (int64_t)k * g.plane, n = base + (int64_t)j * g.pitch + i;
    const int64_t n1 = n + dk * g.plane, n2 = n1 + dk * g.plane;
    const float *ru = x[0], *rv = x[1], *ro = x[3], *tt = x[4];
    const double ro0 = bg.r[k] + (double)__ldcg(ro + n);
    const double ro1 = bg.r[k + dk] + (double)__ldcg(ro + n1);
    const double ro2 = bg.r[k + 2 * dk] + (double)__ldcg(ro + n2);
    const double u = ro0 * (c43 * (double)__ldcg(ru + n1) / ro1 - c13 * (double)__ldcg(ru + n2) / ro2);
    const double v = ro0 * (c43 * (double)__ldcg(rv + n1) / ro1 - c13 * (double)__ldcg(rv + n2) / ro2);
    const double t1 = bg.t[k + dk] + (double)__ldcg(tt + n1), t2 = bg.t[k + 2 * dk] + (double)__ldcg(tt + n2);
    const int mode = side == 0 ? b.top_mode : (b.bottom_mode == 0 ? 6 : 7);
    const double lin = c43 * t1 - c13 * t2;  // modes 1, 3, 7
    double t;
    if (mode == 2 || mode == 3) {  // plume: * plume_x / hh * plume_y / hh
        double f = (mode == 2 ? 1.0 - b.tpr : b.theta - b.tpr) * L.plume_x[i];
        if (b.hh != 1.0) f = f / b.hh;
        f = f * L.plume_y[j];
        if (b.hh != 1.0) f = f / b.hh;
        t = mode == 2 ? 1.0 - f : lin - c23 * b.dz_top * (b.theta - f);
    } else if (mode == 1) {
        t = lin - c23 * b.dz_top * b.theta;
    } else if (mode == 7) {
        t = lin + c23 * b.dz_bot * b.theta / L.rkapa[k];
    } else {  // constant, constant bottom temperature, half-domain
        t = mode == 0 ? 1.0 : (mode == 6 ? b.tb : ((i <= b.half_nx) ? 1.0 - b.tp : 1.0));
    }
    put_periodic(x[0], base, g, i, j, (float)u);
    put_periodic(x[1], base, g, i, j, (float)v);
    put_periodic(x[2], base, g, i, j, 0.0f);
    put_periodic(x[4], base, g, i, j, (float)(t - bg.t[k]));
    if (dt) {
        const double dd = min_of3(L.ddx[i], L.ddy[j], L.ddz[k]);
        double w1, w2, w3, w4, um;
        dt_terms<false>(ph, (double)(float)u, (double)(float)v, 0.0, ro0, bg.t[k] + (double)(float)(t - bg.t[k]), 0.0,
                        dd, L.rkapa[k], w1, w2, w3, w4, um);
        m1 = fold_min(m1, w1);
        m2 = fold_min(m2, w2);
        m3 = fold_min(m3, w3);
        mu = fold_max(mu, um);
    }
}

}  // namespace r3dk
