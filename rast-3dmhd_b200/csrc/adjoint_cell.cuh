// adjoint_cell.cuh - per-cell arithmetic of the discrete adjoint of one FP64 RK3 step.
//
// The forward step (src/step.cpp:114-257 with src/fluxes.cpp:87-533, src/bcon.cpp:12-141 and,
// with LMAG, golden/fortran/3dmhdsub.f:2146-2650) is, per stage s,
//     Y = Z_s + gam_s dt F(X_s),  X_{s+1} = BCON(Y),  Z_{s+1} = X_{s+1} + zeta_{s+1} dt F(X_s),
// with dt = sff * min over cells of the CFL / diffusion limits of X_0.  Its adjoint runs the
// stages backwards; the one non-trivial piece is the transpose of the flux Jacobian, F'(X)^T.
// Every flux term is a product of point values at the output cell (u, v, w, 1/rho, T, B) and
// first/second differences of u, v, w, T, P = rho*T, B and the momenta, plus the cross
// differences d/dy(du/dx)-type terms of the viscous stress.  F'^T is therefore evaluated in
// two gather passes, with no atomics:
//
//   pass 1 (per output cell c): lambda_F at c, and from it and the forward values the adjoints
//     of the velocity differences du/dx .. dw/dz and of the curl of B at c.  The viscous heating
//     depends on du/dy + dv/dx (and its two companions) as a whole, and the Lorentz force and
//     ohmic heating on the curl, so six arrays (nine with MHD) carry what the heating, the p dV
//     work and the current contribute.  The partials w.r.t. u, v, w, 1/rho, T, B at c itself go
//     through the chain rule here (u = RU/rho, P = rho*T, 1/rho) and wait in the output array.
//   pass 2 (per input cell m): adds the transposed difference stencils, gathered at the neighbours
//     of m (a central difference coef(c)*(f(c+e) - f(c-e)) contributes coef(m-e)*Lambda(m-e) -
//     coef(m+e)*Lambda(m+e) to f's adjoint at m).  Every Lambda not stored is a product of values
//     at one point - lambda_F times u, v, w, 1/rho, B - and is formed where it is gathered; the
//     cross differences of the viscous stress are corner stencils of lambda_F itself.  lambda_Y, the
//     largest term, is added last, so that it is rounded once (128x128x128 hydro vjp, error against
//     64-bit torch 2.9e-17; added in pass 1 1.4e-16).
//
// Bound: the latency of the gathers, then DRAM: one stage moves 106 arrays with MHD, 67 without.  The
// partials in pass 1 keep pass 2 at 128 registers (with them it needs 174 and runs 8 warps per SM).
//
// x and y are periodic: the forward reads ghost cells that are exact images of interior cells,
// so the adjoint works on the npx x npy torus with wrapped neighbour indices and never stores an
// adjoint in a ghost cell.  The z ghost planes are constants of the forward map (zero momenta
// and field there), so adjoints that would land on them are dropped.  The one-sided z stencils
// of the planes k = 1 and k = npz (the continuity flux, src/fluxes.cpp:106-117, and the LMAG
// terms of 3dmhdsub.f 1125/1126, 1391/1392, 1511/1513) transpose to the extra edge terms of
// pass 2's z part.
#pragma once

#include "r3d_device.cuh"

#ifdef __CUDACC__
#define R3D_HD __host__ __device__ __forceinline__
#else
#define R3D_HD inline
#endif

namespace r3dk {

// Intermediate arrays written by pass 1 and read by pass 2 (the last three only with LMAG).
enum {
    Q_SXY, Q_SXZ, Q_SYZ,  // common part of the adjoints of (du/dy, dv/dx), (du/dz, dw/dx), (dv/dz, dw/dy)
    Q_DX, Q_DY, Q_DZ,     // adjoints of du/dx, dv/dy, dw/dz without their cross-difference terms
    kMidHydro,
    Q_KX = kMidHydro, Q_KY, Q_KZ,  // adjoints of the curl components dBz/dy - dBy/dz, ... (up to sign)
    kMidMax
};

enum { F_RU, F_RV, F_RW, F_RO, F_TT, F_BX, F_BY, F_BZ };

// Everything the adjoint passes read or write.  Every pointer is the first field of a set stored
// field after field, fe elements apart, in the padded device layout.
struct AdjArgs {
    Geometry g;
    Physics ph;
    Lines L;
    int64_t fe;
    const double* x;      // forward state X_s
    const double* lam;    // lambda_Y of stage s
    const double* lprev;  // lambda_Y of stage s + 1 (null in the last stage)
    double* a;            // pass 1 out: lambda_F, the adjoint of F(X_s) = (FU FV FW FR FT W1 W2 W3)
    double* mid;          // pass 1 out, pass 2 in
    double* out;          // lambda_X_s: pass 1 leaves the cell's own part, pass 2 adds the rest (may be
                          // lprev, which pass 1 reads at the cell itself only)
    const double* F;      // F(X_s), for d/d(dt)
    const Scalars* sc;    // dt of the step
    double gam, zeta;     // gam_s, zeta_{s+1}
    int ahead;            // blocks by which the L2 prefetch runs ahead
};

struct Nbr {  // neighbour offsets of an interior cell on the x/y torus
    int n, xp, xm, yp, ym, ip, im, jp, jm;
};

R3D_HD Nbr neighbours(const Geometry& g, int i, int j, int k) {
    Nbr b;
    const int P = (int)g.pitch, PL = (int)g.plane;
    b.ip = (i == g.npx) ? 1 : i + 1;
    b.im = (i == 1) ? g.npx : i - 1;
    b.jp = (j == g.npy) ? 1 : j + 1;
    b.jm = (j == 1) ? g.npy : j - 1;
    b.n = k * PL + j * P + i;
    b.xp = k * PL + j * P + b.ip;
    b.xm = k * PL + j * P + b.im;
    b.yp = k * PL + b.jp * P + i;
    b.ym = k * PL + b.jm * P + i;
    return b;
}

R3D_HD double recip(double x) {
#ifdef __CUDA_ARCH__
    return __drcp_rn(x);
#else
    return 1.0 / x;
#endif
}

// An array that its kernel only reads: loads of it may be moved ahead of stores (left in order
// behind them, the gathers of a cell went out one by one and the passes waited on each).
struct In {
    const double* p;
    R3D_HD double operator[](int64_t n) const {
#ifdef __CUDA_ARCH__
        return __ldg(p + n);
#else
        return p[n];
#endif
    }
    R3D_HD In field(int64_t off) const { return In{p + off}; }
};

struct Vel {  // 1/rho and the velocity at one cell
    double r, u, v, w;
};
R3D_HD Vel vel_at(const In& x, int64_t fe, int m) {
    Vel q;
    q.r = recip(x[F_RO * fe + m]);
    q.u = x[F_RU * fe + m] * q.r;
    q.v = x[F_RV * fe + m] * q.r;
    q.w = x[F_RW * fe + m] * q.r;
    return q;
}

// ------------------------------------------------------------------------ pass 1 --------
// lambda_F = gam_s dt lambda_Y(s) + zeta_{s+1} dt lambda_Y(s+1) at the cell, the adjoints of the
// velocity and field differences there that pass 2 gathers at its neighbours, and the cell's own
// part of lambda_X_s; returns <F(X_s), lambda_F> there.
template <bool MHD>
R3D_HD double adj_pass1_cell(const AdjArgs& A, int i, int j, int k) {
    constexpr int NF = MHD ? 8 : 5;
    const Geometry& g = A.g;
    const Physics& ph = A.ph;
    const Lines& L = A.L;
    const Nbr b = neighbours(g, i, j, k);
    const int PL = (int)g.plane, n = b.n, zp = n + PL, zm = n - PL;
    const int64_t fe = A.fe;
    const In x{A.x}, lam{A.lam}, F{A.F};
    const double dt = A.sc->dt, cg = A.gam * dt, cz = A.zeta * dt;
    double a[NF], own[NF], dot = 0.0;
#pragma unroll
    for (int f = 0; f < NF; ++f) a[f] = A.lprev ? A.lprev[f * fe + n] : 0.0;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        own[f] = 0.0;
        a[f] = cg * lam[f * fe + n] + cz * a[f];
        dot += F[f * fe + n] * a[f];
    }
#pragma unroll
    for (int f = 0; f < NF; ++f) A.a[f * fe + n] = a[f];
    // first differences of the velocities at c (central on every plane; planes 1 and npz
    // read the constant z ghost planes, where the momenta vanish)
    const double X1 = ph.hx * L.dxxdx[i], Y1 = L.tmpy[j], Z1 = L.tmpz[k];
    const Vel xp_ = vel_at(x, fe, b.xp), xm_ = vel_at(x, fe, b.xm);
    const Vel yp_ = vel_at(x, fe, b.yp), ym_ = vel_at(x, fe, b.ym);
    const Vel zp_ = vel_at(x, fe, zp), zm_ = vel_at(x, fe, zm);
    const double ux = (xp_.u - xm_.u) * X1, vx = (xp_.v - xm_.v) * X1, wx = (xp_.w - xm_.w) * X1;
    const double uy = (yp_.u - ym_.u) * Y1, vy = (yp_.v - ym_.v) * Y1, wy = (yp_.w - ym_.w) * Y1;
    const double uz = (zp_.u - zm_.u) * Z1, vz = (zp_.v - zm_.v) * Z1, wz = (zp_.w - zm_.w) * Z1;
    // viscous heating and p dV (src/fluxes.cpp:327-514)
    const In tt = x.field(F_TT * fe);
    const double T = tt[n], r = recip(x[F_RO * fe + n]), aT = a[F_TT];
    const double s2 = 2.0 * aT * ph.theat * r, s43 = aT * ph.theat43 * r, pdv = aT * ph.ocv * T;
    A.mid[Q_SXY * fe + n] = s2 * (vx + uy);
    A.mid[Q_SXZ * fe + n] = s2 * (wx + uz);
    A.mid[Q_SYZ * fe + n] = s2 * (wy + vz);
    A.mid[Q_DX * fe + n] = s43 * (2.0 * ux - vy - wz) - pdv;
    A.mid[Q_DY * fe + n] = s43 * (2.0 * vy - ux - wz) - pdv;
    A.mid[Q_DZ * fe + n] = s43 * (2.0 * wz - ux - vy) - pdv;
    own[F_TT] -= aT * ph.ocv * (ux + vy + wz);
    // partials w.r.t. u, v, w and 1/rho: energy advection, conduction (src/fluxes.cpp:229-276), heating
    double Pu, Pv, Pw, Pr;
    {
        const double sx = tt[b.xp] - tt[b.xm], lx = tt[b.xp] - 2.0 * T + tt[b.xm];
        const double sy = tt[b.yp] - tt[b.ym], ly = tt[b.yp] - 2.0 * T + tt[b.ym];
        const double sz = tt[zp] - tt[zm], lz = tt[zp] - 2.0 * T + tt[zm];
        Pu = -aT * X1 * sx;
        Pv = -aT * Y1 * sy;
        Pw = -aT * Z1 * sz;
        const double cond = sx * ph.hx * L.d2xxdx2[i] + lx * ph.h2x * L.dxxdx[i] * L.dxxdx[i] + sy * L.tmpy1[j] +
                            ly * L.tmpy2[j] + sz * L.tmpz1[k] + lz * L.tmpz2[k];
        Pr = ph.tdiff * (L.rkapa[k] * cond + L.dkapa[k] * Z1 * sz) +
             ph.theat * (ph.c43 * ux * ux + vx * vx + wx * wx + uy * uy + 2.0 * uy * vx + uz * uz + vz * vz + wy * wy +
                         2.0 * vz * wy + 2.0 * uz * wx) +
             ph.theat43 * (vy * vy + wz * wz - ux * wz - ux * vy - vy * wz);
    }
    if constexpr (MHD) {  // induction, Lorentz force, ohmic heating (golden/fortran/3dmhdsub.f:2146-2650)
        const In bx = x.field(F_BX * fe), by = x.field(F_BY * fe), bz = x.field(F_BZ * fe);
        const double BX = bx[n], BY = by[n], BZ = bz[n], ob = ph.obeta, c = 2.0 * aT * ph.tmag * r;
        const double aU = a[F_RU], aV = a[F_RV], aW = a[F_RW], a1 = a[F_BX], a2 = a[F_BY], a3 = a[F_BZ];
        const double byx = (by[b.xp] - by[b.xm]) * X1, bzx = (bz[b.xp] - bz[b.xm]) * X1;
        const double bxy = (bx[b.yp] - bx[b.ym]) * Y1, bzy = (bz[b.yp] - bz[b.ym]) * Y1;
        const double bxz = (bx[zp] - bx[zm]) * Z1, byz = (by[zp] - by[zm]) * Z1;
        const double jx = bzy - byz, jy = bxz - bzx, jz = byx - bxy;
        A.mid[Q_KX * fe + n] = ob * (aV * BZ - aW * BY) - c * jx;
        A.mid[Q_KY * fe + n] = ob * (aU * BZ - aW * BX) + c * jy;
        A.mid[Q_KZ * fe + n] = ob * (aU * BY - aV * BX) - c * jz;
        Pu -= a1 * ((bx[b.xp] - bx[b.xm]) * X1) + a2 * byx + a3 * bzx;
        Pv -= a1 * bxy + a2 * ((by[b.yp] - by[b.ym]) * Y1) + a3 * bzy;
        Pw -= a1 * bxz + a2 * byz + a3 * ((bz[zp] - bz[zm]) * Z1);
        Pr += ph.tmag * (jx * jx + jy * jy + jz * jz);
        double wzm = wz;  // 3dmhdsub.f 1125/1126: one-sided on the edge planes
        if (k == 1) wzm = (4.0 * zp_.w - vel_at(x, fe, n + 2 * PL).w) * Z1;
        if (k == g.npz) wzm = (vel_at(x, fe, n - 2 * PL).w - 4.0 * zm_.w) * Z1;
        own[F_BX] += -a1 * (vy + wzm) + a2 * vx + a3 * wx + ob * (aV * jz - aW * jy);
        own[F_BY] += a1 * uy - a2 * (ux + wzm) + a3 * wy + ob * (aW * jx - aU * jz);
        own[F_BZ] += a1 * uz + a2 * vz - a3 * (ux + vy) + ob * (aU * jy - aV * jx);
    }
    // chain rule through u = RU/rho and 1/rho; buoyancy and rotation
    own[F_RU] += r * Pu - ph.omz * a[F_RV];
    own[F_RV] += r * Pv + ph.omz * a[F_RU] - ph.omx * a[F_RW];
    own[F_RW] += r * Pw + ph.omx * a[F_RV];
    own[F_RO] += ph.grav * a[F_RW] - r * r * (aT * Pr + x[F_RU * fe + n] * Pu + x[F_RV * fe + n] * Pv + x[F_RW * fe + n] * Pw);
#pragma unroll
    for (int f = 0; f < NF; ++f) A.out[f * fe + n] = own[f];
    return dot;
}

// ------------------------------------------------------------------------ pass 2 --------
// lambda_X_s at one input cell: the own part of pass 1 plus what the differences at the
// neighbours contribute.
template <bool MHD>
R3D_HD void adj_pass2_cell(const AdjArgs& A, int i, int j, int k) {
    constexpr int NF = MHD ? 8 : 5;
    const Geometry& g = A.g;
    const Physics& ph = A.ph;
    const Lines& L = A.L;
    const Nbr b = neighbours(g, i, j, k);
    const int PL = (int)g.plane, npz = g.npz;
    const int n = b.n, zp = n + PL, zm = n - PL;
    const bool lo = k > 1, hi = k < npz;
    const int64_t fe = A.fe;
    const In x{A.x}, a{A.a}, md{A.mid}, lam{A.lam};
    const In mu = x.field(F_RU * fe), mv = x.field(F_RV * fe), mw = x.field(F_RW * fe), ro = x.field(F_RO * fe);
    const In aU = a.field(F_RU * fe), aV = a.field(F_RV * fe), aW = a.field(F_RW * fe), aR = a.field(F_RO * fe);
    const In aT = a.field(F_TT * fe);
    const In a1 = a.field(F_BX * fe), a2 = a.field(F_BY * fe), a3 = a.field(F_BZ * fe);  // MHD only
    const In bx = x.field(F_BX * fe), by = x.field(F_BY * fe), bz = x.field(F_BZ * fe);
    auto mid = [&](int q, int m) { return md[q * fe + m]; };
    double own[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) own[f] = A.out[f * fe + n];

    const double RU = mu[n], RV = mv[n], RW = mw[n];
    const double r = recip(ro[n]), u = RU * r, v = RV * r, w = RW * r;
    const double U0 = aU[n], V0 = aV[n], W0 = aW[n], T0 = aT[n];
    const double ore = ph.ore, c43 = ph.c43, tB = ph.t13, tk = ph.tdiff, tkr = tk * L.rkapa[k], orm = ph.orm;
    double lu, lv, lw, lP, lT, oU, oV, oW, lB1 = 0.0, lB2 = 0.0, lB3 = 0.0;

    // coefficients live at the output cell: X1m = hx*dxxdx at the column left of this one etc.; a
    // central difference at c transposes to X1m*F(xm) - X1p*F(xp) here
    const double X1m = ph.hx * L.dxxdx[b.im], X1p = ph.hx * L.dxxdx[b.ip];
    const double Y1m = L.tmpy[b.jm], Y1p = L.tmpy[b.jp];
    const double Z1m = lo ? L.tmpz[k - 1] : 0.0, Z1p = hi ? L.tmpz[k + 1] : 0.0;
    {  // ---- x ----
        const int m = b.xm, p = b.xp;
        const double rm = recip(ro[m]), rp = recip(ro[p]), um = mu[m] * rm, up = mu[p] * rp;
        const double X2lm = ph.h2x * L.dxxdx[b.im] * L.dxxdx[b.im], X2lp = ph.h2x * L.dxxdx[b.ip] * L.dxxdx[b.ip];
        const double dm = ph.hx * L.d2xxdx2[b.im] + X2lm, dp = X2lp - ph.hx * L.d2xxdx2[b.ip];
        const double d0 = -2.0 * ph.h2x * L.dxxdx[i] * L.dxxdx[i];
        const double Um = aU[m], Up = aU[p], Vm = aV[m], Vp = aV[p], Wm = aW[m], Wp = aW[p];
        const double gU = X1m * Um - X1p * Up, gV = X1m * Vm - X1p * Vp, gW = X1m * Wm - X1p * Wp;
        lu = X1m * mid(Q_DX, m) - X1p * mid(Q_DX, p) + ore * c43 * (dm * Um + dp * Up + d0 * U0) -
             (RU * gU + RV * gV + RW * gW);
        lv = X1m * mid(Q_SXY, m) - X1p * mid(Q_SXY, p) + ore * (dm * Vm + dp * Vp + d0 * V0);
        lw = X1m * mid(Q_SXZ, m) - X1p * mid(Q_SXZ, p) + ore * (dm * Wm + dp * Wp + d0 * W0);
        lP = -gU;
        oU = -u * gU - (X1m * aR[m] - X1p * aR[p]);
        oV = -u * gV;
        oW = -u * gW;
        lT = aT[m] * (rm * tkr * dm - um * X1m) + aT[p] * (rp * tkr * dp + up * X1p) + T0 * r * tkr * d0;
        if constexpr (MHD) {
            const double m1 = a1[m], p1 = a1[p], m2 = a2[m], p2 = a2[p], m3 = a3[m], p3 = a3[p];
            lu -= X1m * (m2 * by[m] + m3 * bz[m]) - X1p * (p2 * by[p] + p3 * bz[p]);
            lv += X1m * (m2 * bx[m]) - X1p * (p2 * bx[p]);
            lw += X1m * (m3 * bx[m]) - X1p * (p3 * bx[p]);
            lB1 = X1p * (p1 * up) - X1m * (m1 * um) + orm * (dm * m1 + dp * p1 + d0 * a1[n]);
            lB2 = X1p * (p2 * up + mid(Q_KZ, p)) - X1m * (m2 * um + mid(Q_KZ, m)) + orm * (dm * m2 + dp * p2 + d0 * a2[n]);
            lB3 = X1p * (p3 * up + mid(Q_KY, p)) - X1m * (m3 * um + mid(Q_KY, m)) + orm * (dm * m3 + dp * p3 + d0 * a3[n]);
        }
    }
    {  // ---- y ----
        const int m = b.ym, p = b.yp;
        const double rm = recip(ro[m]), rp = recip(ro[p]), vm = mv[m] * rm, vp = mv[p] * rp;
        const double dm = L.tmpy1[b.jm] + L.tmpy2[b.jm], dp = L.tmpy2[b.jp] - L.tmpy1[b.jp], d0 = -2.0 * L.tmpy2[j];
        const double Um = aU[m], Up = aU[p], Vm = aV[m], Vp = aV[p], Wm = aW[m], Wp = aW[p];
        const double gU = Y1m * Um - Y1p * Up, gV = Y1m * Vm - Y1p * Vp, gW = Y1m * Wm - Y1p * Wp;
        lu += Y1m * mid(Q_SXY, m) - Y1p * mid(Q_SXY, p) + ore * (dm * Um + dp * Up + d0 * U0);
        lv += Y1m * mid(Q_DY, m) - Y1p * mid(Q_DY, p) + ore * c43 * (dm * Vm + dp * Vp + d0 * V0) -
              (RU * gU + RV * gV + RW * gW);
        lw += Y1m * mid(Q_SYZ, m) - Y1p * mid(Q_SYZ, p) + ore * (dm * Wm + dp * Wp + d0 * W0);
        lP -= gV;
        oU -= v * gU;
        oV -= v * gV + (Y1m * aR[m] - Y1p * aR[p]);
        oW -= v * gW;
        lT += aT[m] * (rm * tkr * dm - vm * Y1m) + aT[p] * (rp * tkr * dp + vp * Y1p) + T0 * r * tkr * d0;
        if constexpr (MHD) {
            const double m1 = a1[m], p1 = a1[p], m2 = a2[m], p2 = a2[p], m3 = a3[m], p3 = a3[p];
            lu += Y1m * (m1 * by[m]) - Y1p * (p1 * by[p]);
            lv -= Y1m * (m1 * bx[m] + m3 * bz[m]) - Y1p * (p1 * bx[p] + p3 * bz[p]);
            lw += Y1m * (m3 * by[m]) - Y1p * (p3 * by[p]);
            lB1 += Y1m * (mid(Q_KZ, m) - m1 * vm) - Y1p * (mid(Q_KZ, p) - p1 * vp) + orm * (dm * m1 + dp * p1 + d0 * a1[n]);
            lB2 += Y1p * (p2 * vp) - Y1m * (m2 * vm) + orm * (dm * m2 + dp * p2 + d0 * a2[n]);
            lB3 += Y1p * (p3 * vp + mid(Q_KX, p)) - Y1m * (m3 * vm + mid(Q_KX, m)) + orm * (dm * m3 + dp * p3 + d0 * a3[n]);
        }
    }
    {  // ---- z: the neighbours' coefficients are 0 beyond the domain (the ghost planes of a and
       // mid are zero, those of x constant) ----
        const int m = zm, p = zp;
        const double rm = recip(ro[m]), rp = recip(ro[p]), wm = mw[m] * rm, wp = mw[p] * rp;
        const double dm = lo ? L.tmpz1[k - 1] + L.tmpz2[k - 1] : 0.0, dp = hi ? L.tmpz2[k + 1] - L.tmpz1[k + 1] : 0.0;
        const double d0 = -2.0 * L.tmpz2[k];
        // the continuity flux, dw/dz of the B fluxes and the z diffusion of Bx, By are one-sided on
        // the planes 1 and npz: their central form transposes from the inner planes only (coefficients
        // e*), the one-sided forms through the values on those planes (below)
        const bool im = k >= 3, ip = k <= npz - 2, in = lo && hi;
        const double e1m = im ? Z1m : 0.0, e1p = ip ? Z1p : 0.0;
        const double Um = aU[m], Up = aU[p], Vm = aV[m], Vp = aV[p], Wm = aW[m], Wp = aW[p];
        const double gU = Z1m * Um - Z1p * Up, gV = Z1m * Vm - Z1p * Vp, gW = Z1m * Wm - Z1p * Wp;
        lu += Z1m * mid(Q_SXZ, m) - Z1p * mid(Q_SXZ, p) + ore * (dm * Um + dp * Up + d0 * U0);
        lv += Z1m * mid(Q_SYZ, m) - Z1p * mid(Q_SYZ, p) + ore * (dm * Vm + dp * Vp + d0 * V0);
        lw += Z1m * mid(Q_DZ, m) - Z1p * mid(Q_DZ, p) + ore * c43 * (dm * Wm + dp * Wp + d0 * W0) -
              (RU * gU + RV * gV + RW * gW);
        lP -= gW;
        oU -= w * gU;
        oV -= w * gV;
        oW -= w * gW + (e1m * aR[m] - e1p * aR[p]);
        const double rkm = lo ? tk * L.rkapa[k - 1] : 0.0, rkp = hi ? tk * L.rkapa[k + 1] : 0.0;
        const double dkm = lo ? tk * L.dkapa[k - 1] : 0.0, dkp = hi ? tk * L.dkapa[k + 1] : 0.0;
        lT += aT[m] * (rm * (rkm * dm + dkm * Z1m) - wm * Z1m) + aT[p] * (rp * (rkp * dp - dkp * Z1p) + wp * Z1p) +
              T0 * r * tkr * d0;
        if constexpr (MHD) {
            const double edm = im ? dm : 0.0, edp = ip ? dp : 0.0, ed0 = in ? d0 : 0.0;
            const double m1 = a1[m], p1 = a1[p], m2 = a2[m], p2 = a2[p], m3 = a3[m], p3 = a3[p];
            lu += Z1m * (m1 * bz[m]) - Z1p * (p1 * bz[p]);
            lv += Z1m * (m2 * bz[m]) - Z1p * (p2 * bz[p]);
            lw -= e1m * (m1 * bx[m] + m2 * by[m]) - e1p * (p1 * bx[p] + p2 * by[p]);
            lB1 += Z1m * (mid(Q_KY, m) - m1 * wm) - Z1p * (mid(Q_KY, p) - p1 * wp) + orm * (edm * m1 + edp * p1 + ed0 * a1[n]);
            lB2 += Z1m * (mid(Q_KX, m) - m2 * wm) - Z1p * (mid(Q_KX, p) - p2 * wp) + orm * (edm * m2 + edp * p2 + ed0 * a2[n]);
            lB3 += Z1p * (p3 * wp) - Z1m * (m3 * wm) + orm * (dm * m3 + dp * p3 + d0 * a3[n]);
        }
        if (k <= 4 || k >= npz - 3) {
            // transposed one-sided forms: plane 1 reads planes 2, 3 (first difference, weights 4, -1)
            // and 1 .. 4 (second difference); plane npz mirrors it
            const int o1 = k - 1, o2 = npz - k;
            const int c1 = n - o1 * PL, c2 = n + o2 * PL;
            const double f1 = L.tmpz[1] * (o1 == 1 ? 4.0 : (o1 == 2 ? -1.0 : 0.0));
            const double f2 = -L.tmpz[npz] * (o2 == 1 ? 4.0 : (o2 == 2 ? -1.0 : 0.0));
            oW -= f1 * aR[c1] + f2 * aR[c2];
            if constexpr (MHD) {
                lw -= f1 * (a1[c1] * bx[c1] + a2[c1] * by[c1]) + f2 * (a1[c2] * bx[c2] + a2[c2] * by[c2]);
                auto l4 = [](int o) { return o == 0 ? 2.0 : (o == 1 ? -5.0 : (o == 2 ? 4.0 : (o == 3 ? -1.0 : 0.0))); };
                auto s4 = [](int o) { return o == 0 ? -3.0 : (o == 1 ? 4.0 : (o == 2 ? -1.0 : 0.0)); };
                const double q1 = L.tmpz1[1] * s4(o1) + L.tmpz2[1] * l4(o1);
                const double q2 = L.tmpz2[npz] * l4(o2) - L.tmpz1[npz] * s4(o2);
                lB1 += orm * (q1 * a1[c1] + q2 * a1[c2]);
                lB2 += orm * (q1 * a2[c1] + q2 * a2[c2]);
            }
        }
    }
    {  // ---- cross differences of the viscous stress: FU += c13/Re (d/dy dv/dx + d/dx dw/dz) ... ----
        const int dyp = b.yp - n, dym = b.ym - n;
        const int xpyp = b.xp + dyp, xpym = b.xp + dym, xmyp = b.xm + dyp, xmym = b.xm + dym;
        auto gxy = [&](const In& F) {
            return X1m * (Y1m * F[xmym] - Y1p * F[xmyp]) - X1p * (Y1m * F[xpym] - Y1p * F[xpyp]);
        };
        auto gxz = [&](const In& F) {
            return X1m * (Z1m * F[b.xm - PL] - Z1p * F[b.xm + PL]) - X1p * (Z1m * F[b.xp - PL] - Z1p * F[b.xp + PL]);
        };
        auto gyz = [&](const In& F) {
            return Y1m * (Z1m * F[b.ym - PL] - Z1p * F[b.ym + PL]) - Y1p * (Z1m * F[b.yp - PL] - Z1p * F[b.yp + PL]);
        };
        lu += tB * (gxy(aV) + gxz(aW));
        lv += tB * (gxy(aU) + gyz(aW));
        lw += tB * (gxz(aU) + gyz(aV));
    }
    // chain rule through u = RU/rho, P = rho*T
    own[F_RU] += oU + r * lu;
    own[F_RV] += oV + r * lv;
    own[F_RW] += oW + r * lw;
    own[F_RO] += x[F_TT * fe + n] * lP - r * r * (RU * lu + RV * lv + RW * lw);
    own[F_TT] += lT + ro[n] * lP;
    if constexpr (MHD) {
        own[F_BX] += lB1;
        own[F_BY] += lB2;
        own[F_BZ] += lB3;
    }
#pragma unroll
    for (int f = 0; f < NF; ++f) A.out[f * fe + n] = own[f] + lam[f * fe + n];  // the Z path
}

// ------------------------------------------------------------------- BCON^T -------------
// src/bcon.cpp:27-140 on one (i, j) column: the written values (momenta, T, Bz on the planes
// 1 and npz) pass their adjoint to what they were computed from, and their own pre-BCON
// values get none.  x holds the post-BCON state (equal to the pre-BCON state on every value
// BCON reads).
R3D_HD void adj_bcon_column(const Geometry& g, const Physics& ph, const Boundary& bd, const double* const* x,
                            double* const* lam, int nf, int side, int i, int j) {
    const int PL = (int)g.plane;
    const double c13 = ph.c13, c43 = ph.c43;
    const int k = side == 0 ? 1 : g.npz;
    const int d = side == 0 ? PL : -PL;
    const int n = k * PL + j * (int)g.pitch + i, n1 = n + d, n2 = n + 2 * d;
    // every load before the first store, so that they go out together
    const double ro0 = x[F_RO][n], i1 = recip(x[F_RO][n1]), i2 = recip(x[F_RO][n2]);
    double lr0 = lam[F_RO][n], lr1 = lam[F_RO][n1], lr2 = lam[F_RO][n2];
    const double C = lam[F_TT][n], t1 = lam[F_TT][n1], t2 = lam[F_TT][n2];
    double a[2], u1[2], u2[2], l1[2], l2[2];
#pragma unroll
    for (int q = F_RU; q <= F_RV; ++q) {
        a[q] = lam[q][n];
        l1[q] = lam[q][n1];
        l2[q] = lam[q][n2];
        u1[q] = x[q][n1];
        u2[q] = x[q][n2];
    }
#pragma unroll
    for (int q = F_RU; q <= F_RV; ++q) {  // ru = ro0 (c43 ru1/ro1 - c13 ru2/ro2), same for rv
        const double v1 = c43 * u1[q] * i1, v2 = c13 * u2[q] * i2, w = a[q] * ro0;
        lr0 += a[q] * (v1 - v2);
        l1[q] += w * c43 * i1;
        l2[q] -= w * c13 * i2;
        lr1 -= w * v1 * i1;
        lr2 += w * v2 * i2;
    }
#pragma unroll
    for (int q = F_RU; q <= F_RV; ++q) {
        lam[q][n] = 0.0;
        lam[q][n1] = l1[q];
        lam[q][n2] = l2[q];
    }
    lam[F_RO][n] = lr0;
    lam[F_RO][n1] = lr1;
    lam[F_RO][n2] = lr2;
    lam[F_RW][n] = 0.0;
    const bool linear = side == 0 ? (bd.top_mode == 1 || bd.top_mode == 3) : (bd.bottom_mode == 1);
    if (linear) {  // T = c43 T1 - c13 T2 + const
        lam[F_TT][n1] = t1 + c43 * C;
        lam[F_TT][n2] = t2 - c13 * C;
    }
    lam[F_TT][n] = 0.0;
    if (nf == 8) lam[F_BZ][n] = 0.0;  // Bz = 0 at both boundaries (ibcon 0)
}

// ------------------------------------------------------------------- dt^T ---------------
// Partial derivatives of the winning time-step limit at one cell (src/step.cpp:122-229):
// ww1 = dd/sqrt(c2) with c2 = q + s + 2 sqrt(q s), q = |rho u|^2/rho^2, s = gamma T (+ B^2
// obeta/rho); ww2 ~ rho; ww3 ~ rho; vv constant.  At q = 0 (a cell at rest) sqrt(q s) has no
// derivative along the momenta; its symmetric subgradient 0 is used.
R3D_HD void adj_dt_cell(const Physics& ph, int term, double dd, double rkap, const double* xv, int nf,
                        double L, double* gout) {
    for (int f = 0; f < nf; ++f) gout[f] = 0.0;
    const double ro = xv[F_RO], r = 1.0 / ro;
    if (term == 1) {  // 0.5 dd^2 repr cv rho / rkapa
        gout[F_RO] = L * (0.5 * dd * dd * ph.repr * ph.cv / rkap);
        return;
    }
    if (term == 2) {  // 0.375 dd^2 re rho
        gout[F_RO] = L * (0.375 * dd * dd * ph.re);
        return;
    }
    if (term != 0) return;
    const double ru = xv[F_RU], rv = xv[F_RV], rw = xv[F_RW], tt = xv[F_TT];
    const double q = (ru * ru + rv * rv + rw * rw) * r * r;
    double b2 = 0.0, bx = 0.0, by = 0.0, bz = 0.0;
    if (nf == 8) {
        bx = xv[F_BX];
        by = xv[F_BY];
        bz = xv[F_BZ];
        b2 = (bx * bx + by * by + bz * bz) * ph.obeta * r;
    }
    const double s = ph.gamma * tt + b2;
    const double c2 = q + s + 2.0 * sqrt(q * s);
    const double w1 = dd / sqrt(c2);
    const double dw_dc2 = -0.5 * w1 / c2;
    const double dc2_dq = 1.0 + (q > 0.0 ? sqrt(s / q) : 0.0);
    const double dc2_ds = 1.0 + (s > 0.0 ? sqrt(q / s) : 0.0);
    const double gq = L * dw_dc2 * dc2_dq, gs = L * dw_dc2 * dc2_ds;
    gout[F_RU] = gq * 2.0 * ru * r * r;
    gout[F_RV] = gq * 2.0 * rv * r * r;
    gout[F_RW] = gq * 2.0 * rw * r * r;
    gout[F_RO] = gq * (-2.0 * q * r) + gs * (-b2 * r);
    gout[F_TT] = gs * ph.gamma;
    if (nf == 8) {
        gout[F_BX] = gs * 2.0 * bx * ph.obeta * r;
        gout[F_BY] = gs * 2.0 * by * ph.obeta * r;
        gout[F_BZ] = gs * 2.0 * bz * ph.obeta * r;
    }
}

}  // namespace r3dk
