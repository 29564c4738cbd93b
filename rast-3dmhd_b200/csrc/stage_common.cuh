// stage_common.cuh - device helpers shared by the stage, BCON and dt kernels.
#pragma once

#include <cuda_runtime.h>

#include "r3d_device.cuh"

namespace r3dk {

// Per-cell time-step limits of src/step.cpp:125-196 for one cell of the finished state:
// returns ww1 = dd/sqrt(c^2), ww2 (conduction), ww3 (viscosity), vv (resistivity, 1e300 without
// LMAG) and the Mach term ogamma*uu/tt.  b2sum = bx^2+by^2+bz^2 (0 without LMAG).
// KC: rkapa == 1 everywhere, where x/rkapa == x exactly and the division is skipped.
template <bool KC = false>
__device__ __forceinline__ void dt_terms(const Physics& ph, double ru, double rv, double rw,
                                         double ro, double tt, double b2sum, double dd,
                                         double rkap, double& w1, double& w2, double& w3,
                                         double& w4, double& um) {
    const double r = __drcp_rn(ro);  // == 1.0/ro
    double uu = (ru * ru + rv * rv + rw * rw) * r * r;
    um = ph.ogamma * uu / tt;
    if (ph.lmag) {
        const double b2 = b2sum * ph.obeta / ro;
        uu = uu + ph.gamma * tt + b2 + 2.0 * sqrt(uu * (ph.gamma * tt + b2));
        w4 = 0.5 * dd * dd * ph.rm;
    } else {
        uu = uu + ph.gamma * tt + 2.0 * sqrt(uu * ph.gamma * tt);
        w4 = 1e300;
    }
    w1 = dd / sqrt(uu);
    w2 = KC ? 0.5 * dd * dd * ph.repr * ph.cv * ro : 0.5 * dd * dd * ph.repr * ph.cv * ro / rkap;
    w3 = 0.375 * dd * dd * ph.re * ro;
}

// std::min(acc, v) / std::max(acc, v): a NaN v never replaces acc.
__device__ __forceinline__ double fold_min(double acc, double v) { return (v < acc) ? v : acc; }
__device__ __forceinline__ double fold_max(double acc, double v) { return (acc < v) ? v : acc; }

// True when x is positive and 2^-30 <= x < 2^31 (one integer compare on the high word): the
// window in which the float estimates below keep their error bound.
__device__ __forceinline__ bool est_window(double x) {
    return (unsigned)__double2hiint(x) - 0x3e100000u < 0x03d00000u;
}

// The plane-independent part of a cell's dd = min(ddx, ddy, ddz) for the filter: min(ddx, ddy)^2 in
// float, 0 (no cell is skipped) when it is outside the window of the estimates.
__device__ __forceinline__ float dd2_est(double dd) {
    return est_window(dd) ? (float)dd * (float)dd : 0.0f;
}

// Fold one cell's time-step limits into running minima m1..m3 and maximum mu, evaluating them (a
// reciprocal, two divisions, two square roots and some fifteen products in FP64) only for cells
// that can matter.  With m = rho u, the limits are
//     Mach term  um = |m|^2 / (gamma T rho^2)
//     CFL        w1 = dd / (|u| + c),  c^2 = gamma T (+ obeta |B|^2 / rho)
//     conduction w2 = 0.5 repr cv dd^2 rho / rkapa,   viscosity  w3 = 0.375 re dd^2 rho
// and (|u| + c)^2 <= (1 + 1/s) |u|^2 + (1 + s) c^2 for any s > 0 (2 |u| c <= |u|^2/s + s c^2; step_begin
// takes s^2 = the Mach term's threshold, where the bound is tight).  So a cell has um < thr_um and
// every limit above its threshold when |m|^2 < u T rho^2, dd^2 rho^2 > a1 |m|^2 + a2 T rho^2 +
// a3 |B|^2 rho and dd^2 rho > max(q2 rkapa, q3) - products and sums of positive quantities, formed in
// float from inputs in 2^-30 .. 2^30, against coefficients that step_begin widens by 2^-10.  From
// correctly rounded inputs both sides have a relative error below 2^-19.  FP32-bulk forms rho and T as
// float(background) + deviation, off by up to 2^-24 of the background and a rounding: where they are
// 2^-8 of the background or more (rlo, tlo), 2^-16 relative, and 2^-13 over the two sides' five factors.
// A non-finite value fails a comparison and the cell is evaluated.  The folded limits over the whole domain are exact whenever the final minima
// are <= and the maximum >= their thresholds (checked by step_end, which requests a full
// re-evaluation otherwise).  The resistive limit depends on the grid alone: the whole-state
// evaluation after an upload leaves its minimum, which no step clears.
// dd2: min(dd2_est(min(ddx, ddy)), dd2_est(ddz)); qk: max(q2 rkapa, q3); dd evaluates min_of3(...).
// rlo, tlo: the smallest rho and T of the estimates.
constexpr float kDtLow = 0x1p-30f;
__device__ __forceinline__ bool dt_skip(const DtBounds& B, float ru, float rv, float rw, float ro, float tt,
                                        float bcfl, float dd2, float qk, float rlo = kDtLow, float tlo = kDtLow) {
    const float msq = ru * ru + rv * rv + rw * rw, r2 = ro * ro, tr2 = tt * r2;
    return ro >= rlo && ro < 0x1p30f && tt >= tlo && tt < 0x1p30f && msq < B.u * tr2 &&
           dd2 * r2 > B.a1 * msq + B.a2 * tr2 + bcfl && dd2 * ro > qk;
}

template <bool KC, bool MHD, class DD>
__device__ __forceinline__ void fold_dt_filtered(const Physics& ph, const DtBounds& B, double ru, double rv, double rw,
                                                 double ro, double tt, double b2sum, float dd2, float qk, DD dd,
                                                 double rkap, double& m1, double& m2, double& m3, double& mu) {
    const float rof = (float)ro;
    if (dt_skip(B, (float)ru, (float)rv, (float)rw, rof, (float)tt, MHD ? B.a3 * ((float)b2sum * rof) : 0.0f, dd2, qk))
        return;
    double w1, w2, w3, w4, um;
    dt_terms<KC>(ph, ru, rv, rw, ro, tt, MHD ? b2sum : 0.0, dd(), rkap, w1, w2, w3, w4, um);
    m1 = fold_min(m1, w1);
    m2 = fold_min(m2, w2);
    m3 = fold_min(m3, w3);
    mu = fold_max(mu, um);
}

// std::min(std::min(a, b), c) with the reference's comparison order.
__device__ __forceinline__ double min_of3(double a, double b, double c) {
    const double m = (b < a) ? b : a;
    return (c < m) ? c : m;
}

// The limit that sets dt, chosen from the four minima's keys as step_begin_kernel does: 0 CFL,
// 1 conduction, 2 viscosity, 3 resistivity; m receives its value.
__device__ __forceinline__ int winning_limit(const unsigned long long* key, int lmag, double& m) {
    int t = 0;
    m = order_value(key[0]);
    const double w1 = order_value(key[1]), w2 = order_value(key[2]), w3 = order_value(key[3]);
    if (w1 < m) { t = 1; m = w1; }
    if (w2 < m) { t = 2; m = w2; }
    if (lmag && w3 < m) { t = 3; m = w3; }
    return t;
}

// Block-wide fold of the running limits, then one atomic per quantity into the scalars.
// red must hold 5 doubles per warp.  Every thread of the block must call it.
__device__ __forceinline__ void reduce_dt(double* red, double w1, double w2, double w3,
                                          double w4, double um, Scalars* sc) {
    const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int nthr = blockDim.x * blockDim.y * blockDim.z;
    const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        w1 = fold_min(w1, __shfl_xor_sync(0xffffffffu, w1, o));
        w2 = fold_min(w2, __shfl_xor_sync(0xffffffffu, w2, o));
        w3 = fold_min(w3, __shfl_xor_sync(0xffffffffu, w3, o));
        w4 = fold_min(w4, __shfl_xor_sync(0xffffffffu, w4, o));
        um = fold_max(um, __shfl_xor_sync(0xffffffffu, um, o));
    }
    __syncthreads();
    if (lane == 0) {
        red[warp * 5 + 0] = w1;
        red[warp * 5 + 1] = w2;
        red[warp * 5 + 2] = w3;
        red[warp * 5 + 3] = w4;
        red[warp * 5 + 4] = um;
    }
    __syncthreads();
    if (tid == 0) {
        const int nw = (nthr + 31) / 32;
        for (int w = 1; w < nw; ++w) {
            w1 = fold_min(w1, red[w * 5 + 0]);
            w2 = fold_min(w2, red[w * 5 + 1]);
            w3 = fold_min(w3, red[w * 5 + 2]);
            w4 = fold_min(w4, red[w * 5 + 3]);
            um = fold_max(um, red[w * 5 + 4]);
        }
        atomicMin(&sc->wmin[0], order_key(w1));
        atomicMin(&sc->wmin[1], order_key(w2));
        atomicMin(&sc->wmin[2], order_key(w3));
        atomicMin(&sc->wmin[3], order_key(w4));
        atomicMax(&sc->umax, order_key(um));
    }
}

// Store v at (i,j) of the plane starting at base, and at its periodic ghost images (the
// one-domain form of the periodic exchange, src/communicate.cpp:108-168).
template <class T>
__device__ __forceinline__ void put_periodic(T* f, int64_t base, const Geometry& g, int i, int j,
                                             T v) {
    f[base + (int64_t)j * g.pitch + i] = v;
    const int gi = (i == 1) ? g.npx + 1 : ((i == g.npx) ? 0 : -1);
    const int gj = (j == 1) ? g.npy + 1 : ((j == g.npy) ? 0 : -1);
    if (gi >= 0) f[base + (int64_t)j * g.pitch + gi] = v;
    if (gj >= 0) f[base + (int64_t)gj * g.pitch + i] = v;
    if (gi >= 0 && gj >= 0) f[base + (int64_t)gj * g.pitch + gi] = v;
}

// BCON (src/bcon.cpp:12-141) of one column on the domain's top plane k = 1 (side 0, src/bcon.cpp:
// 27-98) or bottom plane k = npz (side 1, src/bcon.cpp:104-139), ghost images included; with dt
// the plane's time-step limits are folded as well.  Bound by latency (its loads all go out first, then
// two chains of divisions): one copy of the code serves both sides.  The state is read past L1 (a TAIL
// stage's other CTAs may have written it).
__device__ __forceinline__ void bcon_column(const Geometry& g, const Physics& ph, const Lines& L, const Boundary& b,
                                            double* const* x, int side, int i, int j, bool dt, double& m1, double& m2,
                                            double& m3, double& m4, double& mu) {
    const double c13 = ph.c13, c23 = ph.c23, c43 = ph.c43;
    const int k = side == 0 ? 1 : g.npz;
    const int64_t d = side == 0 ? g.plane : -g.plane;
    const int64_t base = (int64_t)k * g.plane, n = base + (int64_t)j * g.pitch + i;
    const int64_t n1 = n + d, n2 = n1 + d;
    const double *ru = x[0], *rv = x[1], *ro = x[3], *tt = x[4];
    const double ro1 = __ldcg(ro + n), ro2 = __ldcg(ro + n1), ro3 = __ldcg(ro + n2);
    const double u2 = __ldcg(ru + n1), u3 = __ldcg(ru + n2), v2 = __ldcg(rv + n1), v3 = __ldcg(rv + n2);
    const double t1 = __ldcg(tt + n), t2 = __ldcg(tt + n1), t3 = __ldcg(tt + n2);
    const double u = ro1 * (c43 * u2 / ro2 - c13 * u3 / ro3);
    const double v = ro1 * (c43 * v2 / ro2 - c13 * v3 / ro3);
    const int mode = side == 0 ? b.top_mode : (b.bottom_mode == 0 ? 6 : 7);
    const double lin = c43 * t2 - c13 * t3;  // modes 1, 3, 7
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
        t = lin + c23 * b.dz_bot * b.theta / L.rkapa[g.npz];
    } else {
        // constant, itcon 3 (the stage's value stands), half-domain, constant bottom temperature
        t = mode == 0 ? 1.0 : (mode == 5 ? t1 : (mode == 6 ? b.tb : ((i <= b.half_nx) ? 1.0 - b.tp : 1.0)));
    }
    put_periodic(x[0], base, g, i, j, u);
    put_periodic(x[1], base, g, i, j, v);
    put_periodic(x[2], base, g, i, j, 0.0);
    put_periodic(x[4], base, g, i, j, t);
    double b2 = 0.0;
    if (ph.lmag) {
        put_periodic(x[7], base, g, i, j, 0.0);
        const double bx = __ldcg(x[5] + n), by = __ldcg(x[6] + n);
        b2 = bx * bx + by * by + 0.0 * 0.0;
    }
    if (dt) {
        const double dd = min_of3(L.ddx[i], L.ddy[j], L.ddz[k]);
        double w1, w2, w3, w4, um;
        dt_terms(ph, u, v, 0.0, ro1, t, b2, dd, L.rkapa[k], w1, w2, w3, w4, um);
        m1 = fold_min(m1, w1);
        m2 = fold_min(m2, w2);
        m3 = fold_min(m3, w3);
        m4 = fold_min(m4, w4);
        mu = fold_max(mu, um);
    }
}

// The sides (bit 0 top, bit 1 bottom) of its column tile whose BCON this CTA runs, decided when the
// planes kb..ke of its chunk are stored: the plane rewritten and the two inside it lie in one chunk
// (then its own CTA does it) or in up to three, whose last CTA to arrive does it.  Every thread
// of the CTA calls it; s is a shared word.
__device__ __forceinline__ int bcon_sides(const Geometry& g, const StageTail& tail, int kb, int ke, int kchunk,
                                          bool leader, unsigned int* s) {
    const bool top = g.top_edge && kb <= 3, bot = g.bot_edge && ke >= g.npz - 2;
    if (!(tail.flags & kTailBcon) || !(top || bot)) return 0;
    const int nchunks = (g.npz + kchunk - 1) / kchunk;
    const unsigned int ntop = min(nchunks, (2 + kchunk) / kchunk), nbot = nchunks - (g.npz - 3) / kchunk;
    int sides = (top && ntop == 1 ? 1 : 0) | (bot && nbot == 1 ? 2 : 0);
    const bool ct = top && ntop > 1, cb = bot && nbot > 1;
    if (ct || cb) {  // uniform over the CTA
        __threadfence();
        __syncthreads();
        if (leader) {
            unsigned int* cnt = tail.edge_cnt + 2 * (blockIdx.y * gridDim.x + blockIdx.x);
            unsigned int last = 0;
            if (ct && atomicInc(cnt, ntop - 1) == ntop - 1) last |= 1;
            if (cb && atomicInc(cnt + 1, nbot - 1) == nbot - 1) last |= 2;
            __threadfence();
            *s = last;
        }
        __syncthreads();
        sides |= (int)*s;
    }
    return sides;
}

// Start of a step (src/step.cpp:133-141, 224-229): dt = sff*min(...).
__device__ __forceinline__ double step_dt(const Physics& ph, const Scalars* sc) {
    const double w0 = order_value(sc->wmin[0]), w1 = order_value(sc->wmin[1]);
    const double w2 = order_value(sc->wmin[2]), w3 = order_value(sc->wmin[3]);
    double m = (w1 < w0) ? w1 : w0;
    m = (w2 < m) ? w2 : m;
    if (ph.lmag) m = (w3 < m) ? w3 : m;
    return ph.sff * m;
}

// The rest of the start of a step, once per step: dt, umach = sqrt(max(...)) and the thresholds of
// the filtered fold: the previous limits widened by the margin (a margin < 0 forces the
// re-evaluation path; thr_on == 0 skips nothing); a slab takes its own limits, so that its check
// at the step's end makes its own fold exact.
__device__ __forceinline__ void step_begin(const Physics& ph, Scalars* sc) {
    sc->dt = step_dt(ph, sc);
    const double u = order_value(sc->umax);
    sc->umach = sqrt(u);
    double t[3];
    for (int q = 0; q < 3; ++q) {
        t[q] = order_value(sc->thr_local ? sc->wloc[q] : sc->wmin[q]) * (1.0 + sc->thr_margin);
        sc->thr_w[q] = sc->thr_on ? t[q] : 1e308;
    }
    const double tu = (sc->thr_local ? order_value(sc->uloc) : u) * (1.0 - sc->thr_margin);
    sc->thr_um = sc->thr_on ? tu : 0.0;
    DtBounds B{};  // u == 0: every cell is evaluated
    const double s = sqrt(tu), wide = 1.0 + 0x1p-10, t2 = t[0] * t[0] * wide;
    const double q2 = t[1] * wide / (0.5 * ph.repr * ph.cv), q3 = t[2] * wide / (0.375 * ph.re);
    // thresholds far outside the range of any flow (and NaN) would leave float's range
    if (sc->thr_on && tu > 0x1p-40 && tu < 0x1p40 && t[0] > 0x1p-30 && t[0] < 0x1p30 && q2 > 0x1p-60 && q2 < 0x1p60 &&
        q3 > 0x1p-60 && q3 < 0x1p60) {
        B.u = (float)(tu * ph.gamma / wide);
        B.a1 = (float)(t2 * (1.0 + 1.0 / s));
        B.a2 = (float)(t2 * (1.0 + s) * ph.gamma);
        B.a3 = (float)(t2 * (1.0 + s) * ph.obeta);
        B.q2 = (float)q2;
        B.q3 = (float)q3;
    }
    sc->bnd = B;
}

// The limits a step folds anew (all but the resistive one, wmin[3]: it depends on the grid alone).
__device__ __forceinline__ void clear_limits(Scalars* sc) {
    sc->wmin[0] = sc->wmin[1] = sc->wmin[2] = order_key(1e300);
    sc->umax = order_key(0.0);
}

// End of a step: nit, timc, timt (src/step.cpp:254-256).  check != 0 (after a full step on a
// handle with the threshold filter): the skipped cells have limits > thr_w and a Mach term < thr_um,
// so the folded limits are exact iff the minima found are <= thr_w and the maximum >= thr_um;
// otherwise clear them and request the full evaluation (dt_full_kernel with only_refold).  The
// keys are read past L1: a TAIL third stage's other CTAs wrote them.
__device__ __forceinline__ void step_end(Scalars* sc, int check) {
    sc->nit += 1;
    sc->timc += sc->dt;
    sc->timt = sc->timi + sc->timc;
    int refold = 0;
    if (check && sc->thr_on) {
        refold = !(order_value(__ldcg(&sc->umax)) >= sc->thr_um);
        for (int q = 0; q < 3; ++q) refold |= !(order_value(__ldcg(&sc->wmin[q])) <= sc->thr_w[q]);
        if (refold) {
            sc->refolds += 1;
            clear_limits(sc);
        }
    }
    sc->refold = refold;
}

// True for the CTA that ends the launch: every other CTA of the grid has called this before (and
// its stores are visible).  Every thread of the CTA calls it; s is a shared word.
__device__ __forceinline__ bool last_cta(Scalars* sc, bool leader, unsigned int* s) {
    __syncthreads();
    if (leader) {
        const unsigned int n = gridDim.x * gridDim.y * gridDim.z;
        __threadfence();
        *s = atomicInc(&sc->ticket, n - 1) == n - 1;
        __threadfence();
    }
    __syncthreads();
    return *s != 0;
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

}  // namespace r3dk
