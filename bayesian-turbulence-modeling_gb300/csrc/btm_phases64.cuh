// btm_phases64.cuh - the FP64 closure, gradient and assembly phases and the
// FP64 LDU row product and BiCGSTAB, in two forms: the mixed-precision engine's
// FP64 polishing stage (phase_velgrad, phase_grad1, phase_sst, phase_mom_*,
// phase_p_*, phase_turb_*: FP64-accurate) and the FP64 engine's (phase_grads,
// phase_closure, phase_momq_*, phase_pq_*, phase_turbq_*), compiled with
// -fmad=false, whose assembly rounds exactly like the reference.
#pragma once
#include "btm_common.h"
#include "btm_team.cuh"

namespace btm {

// ---------------------------------------------------------------------------
// SST point functions (core/src/SSTModel.cpp:9-96, core/include/SSTModel.hpp:30-39)
// ---------------------------------------------------------------------------
struct Coef {
    double sk1, sw1, b1, al1, sk2, sw2, b2, al2, bstar, a1, kappa;
    int variant;
};
__device__ __forceinline__ Coef load_coef(const DevInst &I) {
    Coef c;
    c.sk1 = I.coeff[0]; c.sw1 = I.coeff[1]; c.b1 = I.coeff[2]; c.al1 = I.coeff[3];
    c.sk2 = I.coeff[4]; c.sw2 = I.coeff[5]; c.b2 = I.coeff[6]; c.al2 = I.coeff[7];
    c.bstar = I.coeff[8]; c.a1 = I.coeff[9]; c.kappa = I.coeff[10];
    c.variant = I.variant;
    return c;
}
__device__ __forceinline__ double blend(double p1, double p2, double F1) { return F1 * p1 + (1.0 - F1) * p2; }

__device__ __forceinline__ double sst_Pw(const Coef &c, double nuT, double S, double k, double omega) {
    double S2 = S * S;
    double lim = 10.0 * c.bstar * smax(k, 0.0) * smax(omega, 1e-20) / smax(nuT, 1e-30);
    return smin(S2, lim);
}

// The closure (core/src/SSTModel.cpp:9-96) with FP64 reciprocals formed once per
// cell (the mixed engine's FP64 polishing stage: FP64-accurate, not
// reference-rounded; phase_closure is the FP64 engine's).
struct SstCell { double F1, F2, nuT, Pk, CDkw; };
__device__ __forceinline__ SstCell sst_cell_fast(const Coef &c, double kc, double wc, double y, double nu, double S,
                                                 double gradDot) {
    SstCell r;
    const double kp = smax(kc, 0.0);
    const double sqrtK = sqrt(kp);
    const double rw = 1.0 / smax(wc, 1e-20);
    const double ySafe = smax(y, 1e-20);
    const double ry = 1.0 / ySafe;
    const double ry2 = ry * ry;
    r.CDkw = 2.0 * c.sw2 * rw * gradDot;
    const double CDpos = smax(r.CDkw, 1e-20);
    const double t1 = sqrtK * rw * ry / c.bstar;
    const double t2 = 500.0 * nu * ry2 * rw;
    if (c.variant == 2) {
        r.F1 = 1.0;
    } else {
        const double t3 = 4.0 * c.sw2 * kp * ry2 / CDpos;
        const double arg1 = smin(smax(t1, t2), t3);
        const double a2 = arg1 * arg1;
        r.F1 = tanh(a2 * a2);
    }
    const double arg2 = smax(2.0 * t1, t2);
    r.F2 = tanh(arg2 * arg2);
    if (c.variant == 1) r.nuT = kp * rw;
    else r.nuT = c.a1 * kp / smax(smax(c.a1 * wc, S * r.F2), 1e-20);
    r.Pk = smin(r.nuT * S * S, 10.0 * c.bstar * kp * smax(wc, 1e-20));
    return r;
}

// ---------------------------------------------------------------------------
// Green-Gauss gradients (core/include/Field.hpp:122-152): per cell, internal
// faces in ascending face order, then boundary faces, then / V.
// ---------------------------------------------------------------------------
template <class T, int NF>
__device__ __forceinline__ void gg_cell(const DevMesh &M, int c, const double *const *phi,
                                        const double *const *phib, double *gx, double *gy, double *gz) {
    double ax[NF], ay[NF], az[NF], pc[NF];
#pragma unroll
    for (int q = 0; q < NF; ++q) { ax[q] = 0.0; ay[q] = 0.0; az[q] = 0.0; pc[q] = LD(phi[q] + c); }
    const int e0 = M.cfOff[c], e1 = M.cfOff[c + 1];
    for (int e = e0; e < e1; ++e) {
        const int f = M.cfFace[e];
        const int oth = M.cfOther[e];
        const double w = M.w[f], sx = M.sfx[f], sy = M.sfy[f], sz = M.sfz[f];
        if (oth >= 0) {
#pragma unroll
            for (int q = 0; q < NF; ++q) {
                double phiF = pc[q] * w + LD(phi[q] + oth) * (1.0 - w);
                ax[q] = ax[q] + sx * phiF;
                ay[q] = ay[q] + sy * phiF;
                az[q] = az[q] + sz * phiF;
            }
        } else {
            const int o = -(oth + 1);
#pragma unroll
            for (int q = 0; q < NF; ++q) {
                double phiF = LD(phi[q] + o) * w + pc[q] * (1.0 - w);
                ax[q] = ax[q] - sx * phiF;
                ay[q] = ay[q] - sy * phiF;
                az[q] = az[q] - sz * phiF;
            }
        }
    }
    const int b0 = M.cbOff[c], b1 = M.cbOff[c + 1];
    for (int e = b0; e < b1; ++e) {
        const int b = M.cbFace[e];
        const double sx = M.bsfx[b], sy = M.bsfy[b], sz = M.bsfz[b];
#pragma unroll
        for (int q = 0; q < NF; ++q) {
            double pb = LD(phib[q] + b);
            ax[q] = ax[q] + sx * pb;
            ay[q] = ay[q] + sy * pb;
            az[q] = az[q] + sz * pb;
        }
    }
    const double V = M.vol[c];
    if (V > 1e-30) {
        const double rv = 1.0 / V;
#pragma unroll
        for (int q = 0; q < NF; ++q) { ax[q] *= rv; ay[q] *= rv; az[q] *= rv; }
    }
#pragma unroll
    for (int q = 0; q < NF; ++q) { gx[q] = ax[q]; gy[q] = ay[q]; gz[q] = az[q]; }
}

// ---------------------------------------------------------------------------
// The FP64 engine's forms of the phases.  An FP64 instruction costs 16 to
// 19 clocks of an SM per warp and 64 of its SMSP, so these do without the ones
// whose result is known: divisions by a known divisor (div_by), 1 - w, the
// reciprocals and relaxation factors of the settings, quotients shared between
// faces or closure functions, sign tests; and with D2 (all normals in the x-y
// plane and no z velocity: DevMesh::is2d and no z-momentum system) the z terms,
// which are zero.  Every remaining operation rounds as in the reference, in the
// same order.  4x128 channel, one instance: closure 124 -> 52 us an outer
// iteration, momentum assembly 70 -> 43, p' assembly 27 -> 16.
// ---------------------------------------------------------------------------
// x / d, correctly rounded, from r = 1 / d correctly rounded: one
// multiplication and two fused multiply-adds (P. Markstein, IBM J. Res. Dev. 34
// (1990) 111; N. Brisebarre, J.-M. Muller, S. K. Raina, IEEE Trans. Comput. 53
// (2004) 1069: exact when nothing over- or underflows on the way).  That is so
// for x within 2^-620 .. 2^620 and d within 2^-300 .. 2^300: the quotient stays
// within 2^-921 .. 2^921, and the remainder is a multiple of 2^-726.  Everything
// else takes the division itself.
template <int E>
__device__ __forceinline__ bool within(double v) {   // |v| in 2^-E .. 2^E
    return ((unsigned int)__double2hiint(v) & 0x7fffffffu) - ((1023u - E) << 20) < (2u * E) << 20;
}
__device__ __forceinline__ double div_by(double x, double d, double r) {
    if (within<620>(x) && within<300>(d)) {
        const double q = x * r;
        return fma(fma(-q, d, x), r, q);
    }
    if (x == 0.0 && within<300>(d)) return x * r;
    return x / d;
}
// smax(v, 0) and smax(-v, 0) without an FP64 comparison (the sign of zero aside)
__device__ __forceinline__ bool is_negative(double v) {   // v < 0: a NaN and -0 are not
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    return u - 0x8000000000000001ull < 0x7ff0000000000000ull;
}
__device__ __forceinline__ double pos_part(double v) { return is_negative(v) ? 0.0 : v; }
__device__ __forceinline__ double flip(double v, bool neg) {
    return __hiloint2double(__double2hiint(v) ^ (neg ? 0x80000000 : 0), __double2loint(v));
}

// The internal faces of cell c in ascending face order: body(face, other cell,
// c is the owner), four list entries fetched at a time.
template <class F>
__device__ __forceinline__ void cell_faces(const DevMesh &M, int c, F body) {
    const int nC = M.nC, nIF = M.nIF, width = M.rowW;
    for (int w0 = 0; w0 < width; w0 += 4) {
        int ent[4], col[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const size_t at = (size_t)(w0 + k < width ? w0 + k : 0) * nC + c;
            col[k] = w0 + k < width ? M.rowCol[at] : -1;
            ent[k] = M.rowEnt[at] - nC;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (col[k] >= 0) body(ent[k] < nIF ? ent[k] : ent[k] - nIF, col[k], ent[k] < nIF);
    }
}

template <class T, int NF, bool D2>
__device__ __forceinline__ void gq_cell(const DevMesh &M, int c, const double *const *phi, const double *const *phib,
                                        double *gx, double *gy, double *gz) {
    double pc[NF];
#pragma unroll
    for (int q = 0; q < NF; ++q) { gx[q] = 0.0; gy[q] = 0.0; gz[q] = 0.0; pc[q] = LD(phi[q] + c); }
    cell_faces(M, c, [&](int f, int oth, bool own) {
        const double w = M.w[f], wn = M.wn[f];
        const double wa = own ? w : wn, wb = own ? wn : w;   // this cell's weight, the other's
        const double sx = flip(M.sfx[f], !own), sy = flip(M.sfy[f], !own), sz = D2 ? 0.0 : flip(M.sfz[f], !own);
#pragma unroll
        for (int q = 0; q < NF; ++q) {
            const double phiF = pc[q] * wa + LD(phi[q] + oth) * wb;
            gx[q] = gx[q] + sx * phiF;
            gy[q] = gy[q] + sy * phiF;
            if (!D2) gz[q] = gz[q] + sz * phiF;
        }
    });
    for (int e = M.cbOff[c]; e < M.cbOff[c + 1]; ++e) {
        const int b = M.cbFace[e];
        const double sx = M.bsfx[b], sy = M.bsfy[b], sz = D2 ? 0.0 : M.bsfz[b];
#pragma unroll
        for (int q = 0; q < NF; ++q) {
            const double pb = LD(phib[q] + b);
            gx[q] = gx[q] + sx * pb;
            gy[q] = gy[q] + sy * pb;
            if (!D2) gz[q] = gz[q] + sz * pb;
        }
    }
    const double V = M.vol[c], r = M.rvol[c];
    if (V > 1e-30) {
#pragma unroll
        for (int q = 0; q < NF; ++q) {
            gx[q] = div_by(gx[q], V, r);
            gy[q] = div_by(gy[q], V, r);
            if (!D2) gz[q] = div_by(gz[q], V, r);
        }
    }
}

// pressure gradient and the velocity gradients of the components in `which`
// (bits 0-2; 8: the pressure) in one pass.  D2: component z and z derivatives
// are left as they are (zeroed once, see phase_grad_init).
template <class T, bool D2>
__device__ __noinline__ void phase_grads(T &tm, const DevMesh &M, DevInst &I, int which) {
    const double *U[3] = {I.ux, I.uy, I.uz};
    const double *UB[3] = {I.ubx, I.uby, I.ubz};
    auto keep = [&](int i, int c, double x, double y, double z) {
        I.g[3 * i][c] = x;
        I.g[3 * i + 1][c] = y;
        if (!D2) I.g[3 * i + 2][c] = z;
    };
    for (int c = tm.spread(); c < M.nC; c += tm.size()) {
        if ((which & 7) == 7) {
            constexpr int NU = D2 ? 2 : 3;
            const double *P[4] = {U[0], U[1], D2 ? I.p : U[2], I.p};
            const double *PB[4] = {UB[0], UB[1], D2 ? I.pb : UB[2], I.pb};
            double gx[NU + 1], gy[NU + 1], gz[NU + 1];
            gq_cell<T, NU + 1, D2>(M, c, P, PB, gx, gy, gz);
#pragma unroll
            for (int i = 0; i < NU; ++i) keep(i, c, gx[i], gy[i], gz[i]);
            I.gpx[c] = gx[NU];
            I.gpy[c] = gy[NU];
            if (!D2) I.gpz[c] = gz[NU];
        } else {
            const int i = which == 1 ? 0 : which == 2 ? 1 : 2;
            const double *P[1] = {U[i]};
            const double *PB[1] = {UB[i]};
            double gx[1], gy[1], gz[1];
            gq_cell<T, 1, D2>(M, c, P, PB, gx, gy, gz);
            keep(i, c, gx[0], gy[0], gz[0]);
        }
    }
}
// the gradients that D2 passes never write
template <class T>
__device__ void phase_grad_init(T &tm, const DevMesh &M, DevInst &I) {
    for (int c = tm.rank(); c < M.nC; c += tm.size()) {
        I.g[2][c] = I.g[5][c] = 0.0;
        I.g[6][c] = I.g[7][c] = I.g[8][c] = 0.0;
        I.gpz[c] = 0.0;
    }
}

// SSTModel::computeFields + frozen |S| + startup floor (SIMPLESolver.cpp:736-768;
// core/src/SSTModel.cpp:9-96), from the gradients in I.g; nutMin < 0 skips the floor
template <class T, bool D2>
__device__ __noinline__ void phase_closure(T &tm, const DevMesh &M, DevInst &I, double nutMin) {
    const Coef cf = load_coef(I);
    const double nu = I.nu;
    const double *P[2] = {I.k, I.om};
    const double *PB[2] = {I.kb, I.omb};
    const double nu500 = 500.0 * nu, sw2x2 = 2.0 * cf.sw2, sw2x4 = 4.0 * cf.sw2, ten = 10.0 * cf.bstar;
    for (int c = tm.spread(); c < M.nC; c += tm.size()) {
        const double S11 = LD(I.g[0] + c), S22 = LD(I.g[4] + c);
        const double S12 = 0.5 * (LD(I.g[1] + c) + LD(I.g[3] + c));
        double Sc;
        if (D2) {
            Sc = sqrt(2.0 * (S11 * S11 + S22 * S22 + 2.0 * (S12 * S12)));
        } else {
            const double S33 = LD(I.g[8] + c);
            const double S13 = 0.5 * (LD(I.g[2] + c) + LD(I.g[6] + c));
            const double S23 = 0.5 * (LD(I.g[5] + c) + LD(I.g[7] + c));
            Sc = sqrt(2.0 * (S11 * S11 + S22 * S22 + S33 * S33 + 2.0 * (S12 * S12 + S13 * S13 + S23 * S23)));
        }
        double gx[2], gy[2], gz[2];
        gq_cell<T, 2, D2>(M, c, P, PB, gx, gy, gz);
        const double kc = pos_part(LD(I.k + c));
        const double wc = smax(LD(I.om + c), 1e-20);
        const double y = smax(M.wd[c], 1e-20), y2 = y * y;
        double dot = gx[0] * gx[1] + gy[0] * gy[1];
        if (!D2) dot = dot + gz[0] * gz[1];
        const double CDkw = sw2x2 / wc * dot;
        // (2 a) / b is twice a / b: F2's first argument is twice F1's, and its
        // second one F1's
        const double term1 = sqrt(kc) / (cf.bstar * wc * y);
        const double term2 = nu500 / (y2 * wc);
        double F1 = 1.0;
        if (cf.variant != 2) {
            const double term3 = sw2x4 * kc / (smax(CDkw, 1e-20) * y2);
            const double arg1 = smin(smax(term1, term2), term3);
            F1 = tanh(arg1 * arg1 * arg1 * arg1);
        }
        const double arg2 = smax(2.0 * term1, term2);
        const double F2 = tanh(arg2 * arg2);
        const double nuT = cf.variant == 1 ? kc / wc : cf.a1 * kc / smax(smax(cf.a1 * wc, Sc * F2), 1e-20);
        I.smag[c] = Sc;
        I.cdkw[c] = CDkw;
        I.f1[c] = F1;
        I.f2[c] = F2;
        I.pk[c] = smin(nuT * Sc * Sc, ten * kc * wc);
        I.nut[c] = (nutMin < 0.0) ? nuT : smax(nuT, nutMin);
    }
}

// momentum assembly (SIMPLESolver.cpp:56-203).  `first`: the diffusion
// coefficient is formed and, where `keepD` is given, kept for the next component
// (viscosity and geometry do not change between components).
template <class T, bool D2>
__device__ __noinline__ void phase_momq_faces(T &tm, const DevMesh &M, DevInst &I, int comp, bool first,
                                              double *keepD) {
    const double nu = I.nu;
    const double *gc0 = I.g[comp], *gc1 = I.g[3 + comp], *gc2 = I.g[6 + comp];
    for (int f = tm.spread(); f < M.nIF; f += tm.size()) {
        const int o = M.own[f], n = M.nbr[f];
        const double Sf = M.area[f], w = M.w[f], wn = M.wn[f];
        const double nuo = LD(I.nut + o), nun = LD(I.nut + n);
        double Df;
        if (first || !keepD) {
            const double nuEff_f = w * (nu + nuo) + wn * (nu + nun);
            Df = div_by(nuEff_f * Sf, M.deltaC[f], M.rdelta[f]);
            if (keepD) keepD[f] = Df;
        } else {
            Df = keepD[f];   // written by this thread
        }
        const double nx = M.nx[f], ny = M.ny[f], nz = D2 ? 0.0 : M.nz[f];
        double m = (LD(I.ux + o) * w + LD(I.ux + n) * wn) * nx + (LD(I.uy + o) * w + LD(I.uy + n) * wn) * ny;
        if (!D2) m = m + (LD(I.uz + o) * w + LD(I.uz + n) * wn) * nz;
        const double mFlux = m * Sf;
        I.upper[f] = -(Df + pos_part(-mFlux));
        I.lower[f] = -(Df + pos_part(mFlux));
        double t = (LD(gc0 + o) * w + LD(gc0 + n) * wn) * nx + (LD(gc1 + o) * w + LD(gc1 + n) * wn) * ny;
        if (!D2) t = t + (LD(gc2 + o) * w + LD(gc2 + n) * wn) * nz;
        I.fflux[f] = (w * nuo + wn * nun) * t * Sf;
    }
}
template <class T>
__device__ __noinline__ void phase_momq_cells(T &tm, const DevMesh &M, DevInst &I, int comp) {
    const double nu = I.nu, fb = I.S.bodyForce[comp];
    const double *Uc = comp == 0 ? I.ux : (comp == 1 ? I.uy : I.uz);
    const double *Ubc = comp == 0 ? I.ubx : (comp == 1 ? I.uby : I.ubz);
    const double *gp = comp == 0 ? I.gpx : (comp == 1 ? I.gpy : I.gpz);
    const double *gc0 = I.g[comp], *gc1 = I.g[3 + comp], *gc2 = I.g[6 + comp];
    const bool wallFn = I.S.useWallFn != 0;
    for (int c = tm.spread(); c < M.nC; c += tm.size()) {
        double diag = 0.0, ts = 0.0, src = 0.0;
        cell_faces(M, c, [&](int f, int, bool own) {
            diag = diag + flip(LD((own ? I.lower : I.upper) + f), true);
            ts = ts + flip(LD(I.fflux + f), !own);
        });
        const double nutc = LD(I.nut + c);
        for (int e = M.cbOff[c]; e < M.cbOff[c + 1]; ++e) {
            const int b = M.cbFace[e];
            const double Sf = M.barea[b];
            const double nuEff = (M.bwall[b] && !wallFn) ? nu : nu + nutc;
            const double Db = div_by(nuEff * Sf, M.bdeltaC[b], M.brdelta[b]);
            const double Ub = LD(Ubc + b);
            const double mFlux = (LD(I.ubx + b) * M.bnx[b] + LD(I.uby + b) * M.bny[b] + LD(I.ubz + b) * M.bnz[b]) * Sf;
            if (mFlux >= 0) {
                diag = diag + (mFlux + Db);
                src = src + Db * Ub;
            } else {
                diag = diag + Db;
                src = src + (Db - mFlux) * Ub;
            }
        }
        // transpose stress, wall-aware boundary treatment in patch order
        if (M.cbpOff[c] < M.cbpOff[c + 1]) {
            const double gcx = LD(gc0 + c), gcy = LD(gc1 + c), gcz = LD(gc2 + c);
            for (int e = M.cbpOff[c]; e < M.cbpOff[c + 1]; ++e) {
                const int b = M.cbpFace[e];
                const double cfac = M.bwall[b] ? 0.0 : nutc;
                ts = ts + cfac * (gcx * M.bnx[b] + gcy * M.bny[b] + gcz * M.bnz[b]) * M.barea[b];
            }
        }
        const double vol = M.vol[c];
        src = src - LD(gp + c) * vol;
        if (fb != 0.0) src = src + fb * vol;
        src = src + ts;
        if (I.inj) src = src + LD(I.inj + (size_t)comp * M.nC + c);
        src = src + I.S.relaxU * diag * LD(Uc + c);
        diag = div_by(diag, I.S.alphaU, I.S.rAlphaU);
        I.diag[c] = diag;
        I.src[c] = src;
        if (comp == 0) I.aPx[c] = diag;
    }
}

// V / aP of every cell (both sides of its faces and the boundary use it) into
// I.ph, which the momentum solves are done with
template <class T>
__device__ __forceinline__ void phase_dp(T &tm, const DevMesh &M, DevInst &I) {
    for (int c = tm.rank(); c < M.nC; c += tm.size()) {
        const double aP = LD(I.aPx + c);
        I.ph[c] = (fabs(aP) > 1e-30) ? M.vol[c] / aP : 0.0;
    }
}
// pressure-correction assembly (SIMPLESolver.cpp:322-450) with that quotient
template <class T, bool D2>
__device__ __noinline__ void phase_pq_faces(T &tm, const DevMesh &M, DevInst &I) {
    const bool rc = M.rhieChow != 0;
    for (int f = tm.spread(); f < M.nIF; f += tm.size()) {
        const int o = M.own[f], n = M.nbr[f];
        const double Sf = M.area[f], delta = M.deltaC[f], rdelta = M.rdelta[f], w = M.w[f], wn = M.wn[f];
        const double dP_f = w * LD(I.ph + o) + wn * LD(I.ph + n);
        const double dPS = dP_f * Sf;
        const double coeff = div_by(dPS, delta, rdelta);
        I.upper[f] = -coeff;
        I.lower[f] = -coeff;
        double m = (LD(I.ux + o) * w + LD(I.ux + n) * wn) * M.nx[f] + (LD(I.uy + o) * w + LD(I.uy + n) * wn) * M.ny[f];
        if (!D2) m = m + (LD(I.uz + o) * w + LD(I.uz + n) * wn) * M.nz[f];
        double massFlux = m * Sf;
        if (rc) {
            double gb = (LD(I.gpx + o) * w + LD(I.gpx + n) * wn) * M.ex[f] + (LD(I.gpy + o) * w + LD(I.gpy + n) * wn) * M.ey[f];
            if (!D2) gb = gb + (LD(I.gpz + o) * w + LD(I.gpz + n) * wn) * M.ez[f];
            massFlux += -dPS * (div_by(LD(I.p + n) - LD(I.p + o), delta, rdelta) - gb);
        }
        I.fflux[f] = massFlux;
    }
}
template <class T>
__device__ __noinline__ void phase_pq_cells(T &tm, const DevMesh &M, DevInst &I) {
    for (int c = tm.spread(); c < M.nC; c += tm.size()) {
        double diag = 0.0, src = 0.0;
        cell_faces(M, c, [&](int f, int, bool own) {
            diag = diag + flip(LD(I.upper + f), true);
            src = src + flip(LD(I.fflux + f), own);
        });
        for (int e = M.cbpOff[c]; e < M.cbpOff[c + 1]; ++e) {
            const int b = M.cbpFace[e];
            const double Sf = M.barea[b];
            const double massFlux = (LD(I.ubx + b) * M.bnx[b] + LD(I.uby + b) * M.bny[b] + LD(I.ubz + b) * M.bnz[b]) * Sf;
            src = src - massFlux;
            if (M.bout[b]) diag = diag + div_by(LD(I.ph + c) * Sf, M.bdeltaC[b], M.brdelta[b]);
        }
        if (!M.hasOutlet && c == 0) diag += fabs(diag) > 1e-30 ? diag : 1.0;
        I.diag[c] = diag;
        I.src[c] = src;
        I.pp[c] = 0.0;
    }
}

// k (which = 0) or omega (which = 1) face pass; without `flux` it takes the face
// mass flux that the last pass left in I.fflux (U does not change from k to omega)
template <class T, bool D2>
__device__ __noinline__ void phase_turbq_faces(T &tm, const DevMesh &M, DevInst &I, int which, bool flux) {
    const Coef cf = load_coef(I);
    const double nu = I.nu;
    const double s1 = which == 0 ? cf.sk1 : cf.sw1, s2 = which == 0 ? cf.sk2 : cf.sw2;
    for (int f = tm.spread(); f < M.nIF; f += tm.size()) {
        const int o = M.own[f], n = M.nbr[f];
        const double Sf = M.area[f], w = M.w[f], wn = M.wn[f];
        const double sg = blend(s1, s2, w * LD(I.f1 + o) + wn * LD(I.f1 + n));
        const double nuEff_f = w * (nu + sg * LD(I.nut + o)) + wn * (nu + sg * LD(I.nut + n));
        const double Df = div_by(nuEff_f * Sf, M.deltaC[f], M.rdelta[f]);
        double mFlux;
        if (flux) {
            double m = (LD(I.ux + o) * w + LD(I.ux + n) * wn) * M.nx[f] + (LD(I.uy + o) * w + LD(I.uy + n) * wn) * M.ny[f];
            if (!D2) m = m + (LD(I.uz + o) * w + LD(I.uz + n) * wn) * M.nz[f];
            mFlux = m * Sf;
            I.fflux[f] = mFlux;
        } else {
            mFlux = I.fflux[f];   // written by this thread
        }
        I.upper[f] = -(Df + pos_part(-mFlux));
        I.lower[f] = -(Df + pos_part(mFlux));
    }
}
template <class T>
__device__ __noinline__ void phase_turbq_cells(T &tm, const DevMesh &M, DevInst &I, int which) {
    const Coef cf = load_coef(I);
    const double nu = I.nu;
    const double s1 = which == 0 ? cf.sk1 : cf.sw1, s2 = which == 0 ? cf.sk2 : cf.sw2;
    const double *phib = which == 0 ? I.kb : I.omb;
    const double *phi = which == 0 ? I.k : I.om;
    const double alpha = which == 0 ? I.S.alphaK : I.S.alphaW;
    const double relax = which == 0 ? I.S.relaxK : I.S.relaxW, rAlpha = which == 0 ? I.S.rAlphaK : I.S.rAlphaW;
    const double ten = 10.0 * cf.bstar;
    for (int c = tm.spread(); c < M.nC; c += tm.size()) {
        double diag = 0.0, src = 0.0;
        cell_faces(M, c, [&](int f, int, bool own) { diag = diag + flip(LD((own ? I.lower : I.upper) + f), true); });
        const double F1c = LD(I.f1 + c), nutc = LD(I.nut + c);
        for (int e = M.cbOff[c]; e < M.cbOff[c + 1]; ++e) {
            const int b = M.cbFace[e];
            const double Sf = M.barea[b];
            const double sg = blend(s1, s2, F1c);
            const double Db = div_by((nu + sg * nutc) * Sf, M.bdeltaC[b], M.brdelta[b]);
            const double vb = LD(phib + b);
            const double mFlux = (LD(I.ubx + b) * M.bnx[b] + LD(I.uby + b) * M.bny[b] + LD(I.ubz + b) * M.bnz[b]) * Sf;
            if (mFlux >= 0) {
                diag = diag + (mFlux + Db);
                src = src + Db * vb;
            } else {
                diag = diag + Db;
                src = src + (Db - mFlux) * vb;
            }
        }
        const double vol = M.vol[c];
        const double omc = LD(I.om + c), omC = smax(omc, 1e-20);
        if (which == 0) {
            src = src + LD(I.pk + c) * vol;
            diag = diag + cf.bstar * omC * vol;
        } else {
            const double S = LD(I.smag + c), F2c = 1.0 - F1c;
            const double lim = ten * pos_part(LD(I.k + c)) * omC / smax(nutc, 1e-30);
            src = src + (F1c * cf.al1 + F2c * cf.al2) * smin(S * S, lim) * vol;
            diag = diag + (F1c * cf.b1 + F2c * cf.b2) * omC * vol;
            src = src + F2c * LD(I.cdkw + c) * vol;
        }
        src = src + relax * diag * LD(phi + c);
        I.diag[c] = div_by(diag, alpha, rAlpha);
        I.src[c] = src;
    }
}

// gradient of one scalar into (gx, gy, gz)
template <class T>
__device__ __noinline__ void phase_grad1(T &tm, const DevMesh &M, const double *phi, const double *phib,
                            double *ox, double *oy, double *oz) {
    const double *P[1] = {phi};
    const double *PB[1] = {phib};
    for (int c = tm.rank(); c < M.nC; c += tm.size()) {
        double gx[1], gy[1], gz[1];
        gg_cell<T, 1>(M, c, P, PB, gx, gy, gz);
        ox[c] = gx[0]; oy[c] = gy[0]; oz[c] = gz[0];
    }
}

// velocity gradients (Field.hpp:232-246): g[3*i+j] = dU_i/dx_j; `which` selects
// components (bit i) so a partially updated U only recomputes what changed
template <class T>
__device__ __noinline__ void phase_velgrad(T &tm, const DevMesh &M, DevInst &I, int which) {
    const double *U[3] = {I.ux, I.uy, I.uz};
    const double *UB[3] = {I.ubx, I.uby, I.ubz};
    for (int c = tm.rank(); c < M.nC; c += tm.size()) {
        if (which == 7) {
            double gx[3], gy[3], gz[3];
            gg_cell<T, 3>(M, c, U, UB, gx, gy, gz);
#pragma unroll
            for (int i = 0; i < 3; ++i) { I.g[3 * i][c] = gx[i]; I.g[3 * i + 1][c] = gy[i]; I.g[3 * i + 2][c] = gz[i]; }
        } else {
            for (int i = 0; i < 3; ++i) {
                if (!(which & (1 << i))) continue;
                const double *P[1] = {U[i]};
                const double *PB[1] = {UB[i]};
                double gx[1], gy[1], gz[1];
                gg_cell<T, 1>(M, c, P, PB, gx, gy, gz);
                I.g[3 * i][c] = gx[0]; I.g[3 * i + 1][c] = gy[0]; I.g[3 * i + 2][c] = gz[0];
            }
        }
    }
}

// SSTModel::computeFields + frozen |S| + startup floor (SIMPLESolver.cpp:736-768).
// Requires velocity gradients in I.g.  nutMin < 0 skips the floor.
template <class T>
__device__ __noinline__ void phase_sst(T &tm, const DevMesh &M, DevInst &I, double nutMin) {
    const Coef cf = load_coef(I);
    const double nu = I.nu;
    const double *P[2] = {I.k, I.om};
    const double *PB[2] = {I.kb, I.omb};
    for (int c = tm.rank(); c < M.nC; c += tm.size()) {
        double S11 = LD(I.g[0] + c), S22 = LD(I.g[4] + c), S33 = LD(I.g[8] + c);
        double S12 = 0.5 * (LD(I.g[1] + c) + LD(I.g[3] + c));
        double S13 = 0.5 * (LD(I.g[2] + c) + LD(I.g[6] + c));
        double S23 = 0.5 * (LD(I.g[5] + c) + LD(I.g[7] + c));
        double Sc = sqrt(2.0 * (S11 * S11 + S22 * S22 + S33 * S33 + 2.0 * (S12 * S12 + S13 * S13 + S23 * S23)));
        double gx[2], gy[2], gz[2];
        gg_cell<T, 2>(M, c, P, PB, gx, gy, gz);
        double kc = smax(LD(I.k + c), 0.0);
        double wc = smax(LD(I.om + c), 1e-20);
        double y = smax(M.wd[c], 1e-20);
        const SstCell r = sst_cell_fast(cf, kc, wc, y, nu, Sc, gx[0] * gx[1] + gy[0] * gy[1] + gz[0] * gz[1]);
        I.smag[c] = Sc;
        I.cdkw[c] = r.CDkw;
        I.f1[c] = r.F1;
        I.f2[c] = r.F2;
        I.pk[c] = r.Pk;
        I.nut[c] = (nutMin < 0.0) ? r.nuT : smax(r.nuT, nutMin);
    }
}

// ---------------------------------------------------------------------------
// assembly (SIMPLESolver.cpp:56-203, 322-450, 483-669)
// ---------------------------------------------------------------------------
// Face pass of the momentum system: upper/lower coefficients and the
// transpose-stress flux of component `comp` (StressOperators.hpp:331-340).
template <class T>
__device__ __noinline__ void phase_mom_faces(T &tm, const DevMesh &M, DevInst &I, int comp) {
    const double nu = I.nu;
    const double *gc0 = I.g[comp], *gc1 = I.g[3 + comp], *gc2 = I.g[6 + comp];
    for (int f = tm.rank(); f < M.nIF; f += tm.size()) {
        const int o = M.own[f], n = M.nbr[f];
        const double Sf = M.area[f], w = M.w[f];
        const double nuo = LD(I.nut + o), nun = LD(I.nut + n);
        double nuEff_o = nu + nuo;
        double nuEff_n = nu + nun;
        double nuEff_f = w * nuEff_o + (1.0 - w) * nuEff_n;
        double Df = nuEff_f * M.aOverD[f];
        double Ufx = LD(I.ux + o) * w + LD(I.ux + n) * (1.0 - w);
        double Ufy = LD(I.uy + o) * w + LD(I.uy + n) * (1.0 - w);
        double Ufz = LD(I.uz + o) * w + LD(I.uz + n) * (1.0 - w);
        const double nx = M.nx[f], ny = M.ny[f], nz = M.nz[f];
        double mFlux = (Ufx * nx + Ufy * ny + Ufz * nz) * Sf;
        double cPos = smax(mFlux, 0.0);
        double cNeg = smax(-mFlux, 0.0);
        I.upper[f] = -(Df + cNeg);
        I.lower[f] = -(Df + cPos);
        double cfac = w * nuo + (1.0 - w) * nun;
        double gx = LD(gc0 + o) * w + LD(gc0 + n) * (1.0 - w);
        double gy = LD(gc1 + o) * w + LD(gc1 + n) * (1.0 - w);
        double gz = LD(gc2 + o) * w + LD(gc2 + n) * (1.0 - w);
        I.fflux[f] = cfac * (gx * nx + gy * ny + gz * nz) * Sf;
    }
}

// Reynolds-stress injection source (SIMPLESolver::addInjectionSource,
// incompressible/src/SIMPLESolver.cpp:224-315), run before the x-momentum
// assembly of every outer iteration.  Per cell the deferred-correction tensor
// D = 2 k b_target + 2 nu_t dev(S) from the velocity gradients `g`
// (g[3*i+j] = dU_i/dx_j) and eddy viscosity `nut` (FP64, or the mixed
// engine's FP32 stage-1 copies); per cell the
// force q = -sum_f (D_f . n_f) A_f gathered over its internal faces in
// ascending face order (D_f distance-weighted, owner side subtracts) and then
// its boundary faces (owner value), the reference's scatter order; then
// blend = q on the first pass of a solve (or alpha >= 1), else
// blend (1 - alpha) + q alpha.  inj[0..3nC) holds the blend, inj[3nC..9nC) D.
template <class T, class G>
__device__ __noinline__ void phase_inj(T &tm, const DevMesh &M, DevInst &I, const G *const *g, const G *nut,
                                       bool first) {
    const int nC = M.nC;
    double *D = I.inj + 3 * (size_t)nC;
    // the mixed engine's stage 1 skips the w gradients of a 2-D instance
    // (identically zero there)
    const bool wGrad = sizeof(G) == 8 || I.solveZ != 0;
    for (int c = tm.rank(); c < nC; c += tm.size()) {
        const double g6 = wGrad ? (double)LD(g[6] + c) : 0.0, g7 = wGrad ? (double)LD(g[7] + c) : 0.0;
        const double S11 = LD(g[0] + c), S22 = LD(g[4] + c), S33 = wGrad ? (double)LD(g[8] + c) : 0.0;
        const double S12 = 0.5 * ((double)LD(g[1] + c) + (double)LD(g[3] + c));
        const double S13 = 0.5 * ((double)LD(g[2] + c) + g6);
        const double S23 = 0.5 * ((double)LD(g[5] + c) + g7);
        const double trS3 = (S11 + S22 + S33) / 3.0;
        const double twoK = 2.0 * LD(I.k + c), twoNu = 2.0 * (double)LD(nut + c);
        const double *bt = M.bTarget + 6 * (size_t)c;
        D[0 * (size_t)nC + c] = twoK * bt[0] + twoNu * (S11 - trS3);
        D[1 * (size_t)nC + c] = twoK * bt[1] + twoNu * (S22 - trS3);
        D[2 * (size_t)nC + c] = twoK * bt[2] + twoNu * (S33 - trS3);
        D[3 * (size_t)nC + c] = twoK * bt[3] + twoNu * S12;
        D[4 * (size_t)nC + c] = twoK * bt[4] + twoNu * S13;
        D[5 * (size_t)nC + c] = twoK * bt[5] + twoNu * S23;
    }
    tm.sync();
    const double r = I.S.alphaInj;
    const bool fresh = first || r >= 1.0;
    for (int c = tm.rank(); c < nC; c += tm.size()) {
        double qx = 0.0, qy = 0.0, qz = 0.0;
        for (int e = M.cfOff[c]; e < M.cfOff[c + 1]; ++e) {
            const int f = M.cfFace[e], oth = M.cfOther[e];
            const int o = oth >= 0 ? c : -(oth + 1), n = oth >= 0 ? oth : c;
            const double w = M.w[f], wn = 1.0 - w;
            double d[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) d[k] = w * LD(D + k * (size_t)nC + o) + wn * LD(D + k * (size_t)nC + n);
            const double nx = M.nx[f], ny = M.ny[f], nz = M.nz[f], A = M.area[f];
            const double fx = (d[0] * nx + d[3] * ny + d[4] * nz) * A;
            const double fy = (d[3] * nx + d[1] * ny + d[5] * nz) * A;
            const double fz = (d[4] * nx + d[5] * ny + d[2] * nz) * A;
            if (oth >= 0) { qx = qx - fx; qy = qy - fy; qz = qz - fz; }
            else { qx = qx + fx; qy = qy + fy; qz = qz + fz; }
        }
        for (int e = M.cbOff[c]; e < M.cbOff[c + 1]; ++e) {
            const int b = M.cbFace[e];
            double d[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) d[k] = LD(D + k * (size_t)nC + c);
            const double nx = M.bnx[b], ny = M.bny[b], nz = M.bnz[b], A = M.barea[b];
            qx = qx - (d[0] * nx + d[3] * ny + d[4] * nz) * A;
            qy = qy - (d[3] * nx + d[1] * ny + d[5] * nz) * A;
            qz = qz - (d[4] * nx + d[5] * ny + d[2] * nz) * A;
        }
        double *bl = I.inj;
        if (fresh) {
            bl[c] = qx;
            bl[nC + c] = qy;
            bl[2 * (size_t)nC + c] = qz;
        } else {
            bl[c] = LD(bl + c) * (1.0 - r) + qx * r;
            bl[nC + c] = LD(bl + nC + c) * (1.0 - r) + qy * r;
            bl[2 * (size_t)nC + c] = LD(bl + 2 * (size_t)nC + c) * (1.0 - r) + qz * r;
        }
    }
    tm.sync();
}

// Cell pass of the momentum system (diag, source, relaxation).
template <class T>
__device__ __noinline__ void phase_mom_cells(T &tm, const DevMesh &M, DevInst &I, int comp) {
    const double nu = I.nu;
    const double alphaU = I.S.alphaU;
    const double relaxDiag = 1.0 / alphaU, relaxSrc = (1.0 - alphaU) / alphaU;
    const double fb = I.S.bodyForce[comp];
    const double *Uc = comp == 0 ? I.ux : (comp == 1 ? I.uy : I.uz);
    const double *Ubc = comp == 0 ? I.ubx : (comp == 1 ? I.uby : I.ubz);
    const double *gp = comp == 0 ? I.gpx : (comp == 1 ? I.gpy : I.gpz);
    const double *gc0 = I.g[comp], *gc1 = I.g[3 + comp], *gc2 = I.g[6 + comp];
    const bool wallFn = I.S.useWallFn != 0;
    for (int c = tm.rank(); c < M.nC; c += tm.size()) {
        double diag = 0.0, ts = 0.0, src = 0.0;
        const int e0 = M.cfOff[c], e1 = M.cfOff[c + 1];
        for (int e = e0; e < e1; ++e) {
            const int f = M.cfFace[e];
            if (M.cfOther[e] >= 0) {
                diag = diag + (-LD(I.lower + f));
                ts = ts + LD(I.fflux + f);
            } else {
                diag = diag + (-LD(I.upper + f));
                ts = ts - LD(I.fflux + f);
            }
        }
        const double nutc = LD(I.nut + c);
        for (int e = M.cbOff[c]; e < M.cbOff[c + 1]; ++e) {
            const int b = M.cbFace[e];
            const double Sf = M.barea[b];
            double nuEff = (M.bwall[b] && !wallFn) ? nu : nu + nutc;
            double Db = nuEff * M.baOverD[b];
            double Ub = LD(Ubc + b);
            double mFlux = (LD(I.ubx + b) * M.bnx[b] + LD(I.uby + b) * M.bny[b] + LD(I.ubz + b) * M.bnz[b]) * Sf;
            if (mFlux >= 0) {
                diag = diag + (mFlux + Db);
                src = src + Db * Ub;
            } else {
                diag = diag + Db;
                src = src + (Db - mFlux) * Ub;
            }
        }
        // transpose stress, wall-aware boundary treatment in patch order
        const double gcx = LD(gc0 + c), gcy = LD(gc1 + c), gcz = LD(gc2 + c);
        for (int e = M.cbpOff[c]; e < M.cbpOff[c + 1]; ++e) {
            const int b = M.cbpFace[e];
            double cfac = M.bwall[b] ? 0.0 : nutc;
            double flux = cfac * (gcx * M.bnx[b] + gcy * M.bny[b] + gcz * M.bnz[b]) * M.barea[b];
            ts = ts + flux;
        }
        const double vol = M.vol[c];
        src = src - LD(gp + c) * vol;
        if (fb != 0.0) src = src + fb * vol;
        src = src + ts;
        if (I.inj) src = src + LD(I.inj + (size_t)comp * M.nC + c);
        const double phi_old = LD(Uc + c);
        src = src + relaxSrc * diag * phi_old;
        diag = diag * relaxDiag;
        I.diag[c] = diag;
        I.src[c] = src;
        if (comp == 0) I.aPx[c] = diag;
    }
}

// Pressure-correction face pass: Laplacian coefficient and (Rhie-Chow) mass flux.
template <class T>
__device__ __noinline__ void phase_p_faces(T &tm, const DevMesh &M, DevInst &I) {
    const bool rc = M.rhieChow != 0;
    for (int f = tm.rank(); f < M.nIF; f += tm.size()) {
        const int o = M.own[f], n = M.nbr[f];
        const double Sf = M.area[f], delta = M.deltaC[f], w = M.w[f];
        const double Vo = M.vol[o], Vn = M.vol[n];
        const double aPo = LD(I.aPx + o), aPn = LD(I.aPx + n);
        double dP_o = (fabs(aPo) > 1e-30) ? Vo / aPo : 0.0;
        double dP_n = (fabs(aPn) > 1e-30) ? Vn / aPn : 0.0;
        double dP_f = w * dP_o + (1.0 - w) * dP_n;
        double coeff = dP_f * Sf / delta;
        I.upper[f] = -coeff;
        I.lower[f] = -coeff;
        double Ufx = LD(I.ux + o) * w + LD(I.ux + n) * (1.0 - w);
        double Ufy = LD(I.uy + o) * w + LD(I.uy + n) * (1.0 - w);
        double Ufz = LD(I.uz + o) * w + LD(I.uz + n) * (1.0 - w);
        double massFlux = (Ufx * M.nx[f] + Ufy * M.ny[f] + Ufz * M.nz[f]) * Sf;
        if (rc) {
            double gbx = LD(I.gpx + o) * w + LD(I.gpx + n) * (1.0 - w);
            double gby = LD(I.gpy + o) * w + LD(I.gpy + n) * (1.0 - w);
            double gbz = LD(I.gpz + o) * w + LD(I.gpz + n) * (1.0 - w);
            massFlux += -dP_f * Sf * ((LD(I.p + n) - LD(I.p + o)) / delta - (gbx * M.ex[f] + gby * M.ey[f] + gbz * M.ez[f]));
        }
        I.fflux[f] = massFlux;
    }
}

template <class T>
__device__ __noinline__ void phase_p_cells(T &tm, const DevMesh &M, DevInst &I) {
    for (int c = tm.rank(); c < M.nC; c += tm.size()) {
        double diag = 0.0, src = 0.0;
        for (int e = M.cfOff[c]; e < M.cfOff[c + 1]; ++e) {
            const int f = M.cfFace[e];
            diag = diag + (-LD(I.upper + f));
            if (M.cfOther[e] >= 0) src = src - LD(I.fflux + f);
            else src = src + LD(I.fflux + f);
        }
        const double aPc = LD(I.aPx + c);
        for (int e = M.cbpOff[c]; e < M.cbpOff[c + 1]; ++e) {
            const int b = M.cbpFace[e];
            const double Sf = M.barea[b];
            double massFlux = (LD(I.ubx + b) * M.bnx[b] + LD(I.uby + b) * M.bny[b] + LD(I.ubz + b) * M.bnz[b]) * Sf;
            src = src - massFlux;
            if (M.bout[b]) {
                double dP_o = (fabs(aPc) > 1e-30) ? M.vol[c] / aPc : 0.0;
                double coeff = dP_o * Sf / M.bdeltaC[b];
                diag = diag + coeff;
            }
        }
        if (!M.hasOutlet && c == 0) diag += fabs(diag) > 1e-30 ? diag : 1.0;
        I.diag[c] = diag;
        I.src[c] = src;
        I.pp[c] = 0.0;
    }
}

// k (which = 0) or omega (which = 1) face pass
template <class T>
__device__ __noinline__ void phase_turb_faces(T &tm, const DevMesh &M, DevInst &I, int which) {
    const Coef cf = load_coef(I);
    const double nu = I.nu;
    const double s1 = which == 0 ? cf.sk1 : cf.sw1, s2 = which == 0 ? cf.sk2 : cf.sw2;
    for (int f = tm.rank(); f < M.nIF; f += tm.size()) {
        const int o = M.own[f], n = M.nbr[f];
        const double Sf = M.area[f], w = M.w[f];
        double F1_f = w * LD(I.f1 + o) + (1.0 - w) * LD(I.f1 + n);
        double sg = blend(s1, s2, F1_f);
        double nuEff_o = nu + sg * LD(I.nut + o);
        double nuEff_n = nu + sg * LD(I.nut + n);
        double nuEff_f = w * nuEff_o + (1.0 - w) * nuEff_n;
        double Df = nuEff_f * M.aOverD[f];
        double Ufx = LD(I.ux + o) * w + LD(I.ux + n) * (1.0 - w);
        double Ufy = LD(I.uy + o) * w + LD(I.uy + n) * (1.0 - w);
        double Ufz = LD(I.uz + o) * w + LD(I.uz + n) * (1.0 - w);
        double mFlux = (Ufx * M.nx[f] + Ufy * M.ny[f] + Ufz * M.nz[f]) * Sf;
        double cPos = smax(mFlux, 0.0);
        double cNeg = smax(-mFlux, 0.0);
        I.upper[f] = -(Df + cNeg);
        I.lower[f] = -(Df + cPos);
    }
}

template <class T>
__device__ __noinline__ void phase_turb_cells(T &tm, const DevMesh &M, DevInst &I, int which) {
    const Coef cf = load_coef(I);
    const double nu = I.nu;
    const double s1 = which == 0 ? cf.sk1 : cf.sw1, s2 = which == 0 ? cf.sk2 : cf.sw2;
    const double *phib = which == 0 ? I.kb : I.omb;
    const double *phi = which == 0 ? I.k : I.om;
    const double alpha = which == 0 ? I.S.alphaK : I.S.alphaW;
    const double relaxDiag = 1.0 / alpha, relaxSrc = (1.0 - alpha) / alpha;
    for (int c = tm.rank(); c < M.nC; c += tm.size()) {
        double diag = 0.0, src = 0.0;
        for (int e = M.cfOff[c]; e < M.cfOff[c + 1]; ++e) {
            const int f = M.cfFace[e];
            if (M.cfOther[e] >= 0) diag = diag + (-LD(I.lower + f));
            else diag = diag + (-LD(I.upper + f));
        }
        const double F1c = LD(I.f1 + c), nutc = LD(I.nut + c);
        for (int e = M.cbOff[c]; e < M.cbOff[c + 1]; ++e) {
            const int b = M.cbFace[e];
            const double Sf = M.barea[b];
            double sg = blend(s1, s2, F1c);
            double nuEff = nu + sg * nutc;
            double Db = nuEff * M.baOverD[b];
            double vb = LD(phib + b);
            double mFlux = (LD(I.ubx + b) * M.bnx[b] + LD(I.uby + b) * M.bny[b] + LD(I.ubz + b) * M.bnz[b]) * Sf;
            if (mFlux >= 0) {
                diag = diag + (mFlux + Db);
                src = src + Db * vb;
            } else {
                diag = diag + Db;
                src = src + (Db - mFlux) * vb;
            }
        }
        const double vol = M.vol[c];
        const double omc = LD(I.om + c);
        if (which == 0) {
            src = src + LD(I.pk + c) * vol;
            double destruction = cf.bstar * smax(omc, 1e-20);
            diag = diag + destruction * vol;
        } else {
            double omC = smax(omc, 1e-20);
            double alphaB = blend(cf.al1, cf.al2, F1c);
            double S = LD(I.smag + c);
            src = src + alphaB * sst_Pw(cf, nutc, S, LD(I.k + c), omc) * vol;
            double betaB = blend(cf.b1, cf.b2, F1c);
            diag = diag + betaB * omC * vol;
            src = src + (1.0 - F1c) * LD(I.cdkw + c) * vol;
        }
        src = src + relaxSrc * diag * LD(phi + c);
        diag = diag * relaxDiag;
        I.diag[c] = diag;
        I.src[c] = src;
    }
}

// ---------------------------------------------------------------------------
// linear algebra on the LDU system (core/include/LinearSolver.hpp)
//
// GB300 executes FP64 at a small fraction of its FP32 rate, so the Krylov and
// multigrid loops avoid FP64 divisions (reciprocal diagonals computed once per
// solve) and use fused multiply-adds.  These solvers already differ from the
// reference in the last bits through their parallel dot products, so nothing
// is lost: the assembly above keeps the reference's exact rounding.
// ---------------------------------------------------------------------------
// y = A x for one cell: diag*x, then face terms in ascending face order
template <class T>
__device__ __forceinline__ double ldu_row(const DevMesh &M, const DevInst &I, const double *x, int c) {
    return ldu_off<T, false>(M, I.diag, x, c, LD(I.diag + c) * LD(x + c));
}

// reciprocal for the Jacobi preconditioner (LinearSolver.hpp:137-140): rows
// with |diag| <= 1e-30 pass the residual through unscaled
__device__ __forceinline__ double jac_rd(double d) { return (fabs(d) > 1e-30) ? 1.0 / d : 1.0; }
// reciprocal for Gauss-Seidel rows: 0 marks a row the sweep leaves unchanged
__device__ __forceinline__ double gs_rd(double d) { return (fabs(d) > 1e-30) ? 1.0 / d : 0.0; }

struct SolveResult {
    int iterations;
    double finalSq, initialRes;   // squared residual norm at the end, norm at the start
    int converged;
};

// The stopping test of the Krylov solvers, sqrt(sq) / r0 < tol on the squared
// residual norm sq, as sq < limit: both operations round monotonically, so
// there is a smallest sq whose rounded quotient reaches tol.  It is found once
// per solve by trying the 32 doubles around the real-valued limit in the lanes
// of one warp, first for the division and then for the square root, which
// takes an FP64 square root and a division (about 17 dependent FP64
// instructions) out of every test with the same outcome.  Where the limit is
// not bracketed (tolerances or norms at the ends of the range) `limit` is NaN
// and the test divides.
__device__ __forceinline__ double bits_step(double x, int ulps) {
    return __longlong_as_double(__double_as_longlong(x) + ulps);
}
inline __device__ __noinline__ double residual_limit(double r0, double tol) {   // by a whole warp
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    if (tol <= 0.0) return 0.0;   // never below
    const double t0 = r0 * tol;
    if (!(t0 > 1e-140 && t0 < 1e140)) return NAN;
    const unsigned reach = __ballot_sync(full, bits_step(t0, lane - 16) / r0 >= tol);
    const int at = __ffs(reach) - 1;
    if (at < 1) return NAN;
    const double t = bits_step(t0, at - 16), s0 = t * t;
    const unsigned reach2 = __ballot_sync(full, sqrt(bits_step(s0, lane - 16)) >= t);
    const int at2 = __ffs(reach2) - 1;
    return at2 < 1 ? (double)NAN : bits_step(s0, at2 - 16);
}
__device__ __forceinline__ bool residual_below(double sq, double limit, double r0, double tol) {
    return isnan(limit) ? sqrt(sq) / r0 < tol : sq < limit;
}
__device__ __forceinline__ double pick(int lane, double a, double b) { return lane == 0 ? a : b; }
__device__ __forceinline__ double pick(int lane, double a, double b, double c) { return lane == 2 ? c : pick(lane, a, b); }
__device__ __forceinline__ double flag64(bool b) { return b ? 1.0 : 0.0; }
// flags travel as 1.0 / 0.0; reading one is no FP64 operation
__device__ __forceinline__ bool is_set(double f) { return __double2hiint(f) != 0; }

// BiCGSTABSolver::solve (LinearSolver.hpp:191-247), right Jacobi preconditioned.
// x is updated in place; A = (I.diag, I.upper, I.lower), b = I.src.  The
// scalars of a step are formed by the warp that folds its dot products.
template <class T>
__device__ __noinline__ SolveResult team_bicgstab(T &tm, const DevMesh &M, DevInst &I, double *x, int maxIter, double tol) {
    SolveResult res = {0, 0.0, 0.0, 0};
    const int nC = M.nC;
    const RowTab rows(M);
    const double *sys = I.diag, *src = I.src;
    double *r = I.r, *rh = I.rh, *pv = I.pv, *v = I.v, *s = I.s, *t = I.t, *ph = I.ph, *sh = I.sh, *rd = I.rd;
    double acc[1] = {0.0};
    for (int c = tm.rank(); c < nC; c += tm.size()) {
        double rc = LD(src + c) - ldu_off<T, false>(rows, sys, (const double *)x, c, LD(sys + c) * LD(x + c));
        r[c] = rc; rh[c] = rc; pv[c] = 0.0; v[c] = 0.0;
        rd[c] = jac_rd(LD(sys + c));
        acc[0] = fma(rc, rc, acc[0]);
    }
    double o[4];
    // |r|^2 is also the first rho; with rho = alpha = omega = 1 before it, the
    // first beta is rho itself
    tm.template sum_then<1, 4>(acc, o, [tol](int lane, double rr, double) {
        const double r0 = sqrt(rr);
        const double limit = residual_limit(r0, tol);
        return lane == 3 ? limit : pick(lane, rr, r0, flag64(r0 < 1e-30));
    });
    double rhoN = o[0];
    const double r0 = o[1], limit = o[3];
    res.initialRes = r0;
    if (is_set(o[2])) { res.converged = 1; return res; }
    double beta = rhoN, omega = 1.0;
    bool small = fabs(rhoN) < 1e-30;
    for (int it = 0; it < maxIter; ++it) {
        if (!tm.ok()) break;
        if (small) break;
        for (int c = tm.rank(); c < nC; c += tm.size()) {
            double p = fma(beta, fma(-omega, LD(v + c), LD(pv + c)), LD(r + c));
            pv[c] = p;
            ph[c] = p * LD(rd + c);
        }
        tm.sync();
        double a1[1] = {0.0};
        for (int c = tm.rank(); c < nC; c += tm.size()) {
            double vc = ldu_off<T, false>(rows, sys, (const double *)ph, c, LD(sys + c) * LD(ph + c));
            v[c] = vc;
            a1[0] = fma(LD(rh + c), vc, a1[0]);
        }
        tm.template sum_then<1, 2>(a1, o, [rhoN](int lane, double rv, double) {
            return pick(lane, flag64(fabs(rv) < 1e-30), rhoN / rv);
        });
        if (is_set(o[0])) break;
        const double alpha = o[1];
        double a2[1] = {0.0};
        for (int c = tm.rank(); c < nC; c += tm.size()) {
            double sc = fma(-alpha, LD(v + c), LD(r + c));
            s[c] = sc;
            sh[c] = sc * LD(rd + c);
            a2[0] = fma(sc, sc, a2[0]);
        }
        tm.template sum_then<1, 2>(a2, o, [=](int lane, double ss, double) {
            return pick(lane, ss, flag64(residual_below(ss, limit, r0, tol)));
        });
        if (is_set(o[1])) {
            for (int c = tm.rank(); c < nC; c += tm.size()) x[c] = fma(alpha, LD(ph + c), LD(x + c));
            res.iterations = it + 1; res.finalSq = o[0]; res.converged = 1;
            tm.sync();
            return res;
        }
        double a3[2] = {0.0, 0.0};
        for (int c = tm.rank(); c < nC; c += tm.size()) {
            double tc = ldu_off<T, false>(rows, sys, (const double *)sh, c, LD(sys + c) * LD(sh + c));
            t[c] = tc;
            a3[0] = fma(tc, tc, a3[0]);
            a3[1] = fma(tc, LD(s + c), a3[1]);
        }
        tm.template sum_then<2, 1>(a3, o, [](int, double tt, double ts) { return (tt > 1e-30) ? ts / tt : 0.0; });
        omega = o[0];
        double a4[2] = {0.0, 0.0};
        for (int c = tm.rank(); c < nC; c += tm.size()) {
            x[c] = LD(x + c) + fma(alpha, LD(ph + c), omega * LD(sh + c));
            double rc = fma(-omega, LD(t + c), LD(s + c));
            r[c] = rc;
            a4[0] = fma(rc, rc, a4[0]);
            a4[1] = fma(LD(rh + c), rc, a4[1]);
        }
        // how the iteration ends (0: on to the next, 1: converged, 2:
        // breakdown), and the next beta = (rho' / rho) (alpha / omega): the two
        // quotients side by side in two lanes
        double e[4];
        tm.template sum_then<2, 4>(a4, e, [=](int lane, double rr, double rho) {
            const double end = residual_below(rr, limit, r0, tol) ? 1.0 : (fabs(omega) < 1e-30 ? 2.0 : 0.0);
            const double q = pick(lane, rho, alpha) / (pick(lane, rhoN, omega) + 1e-30);
            const double b = __shfl_sync(0xffffffffu, q, 0) * __shfl_sync(0xffffffffu, q, 1);
            return lane == 3 ? end : pick(lane, rr, rho, b);
        });
        res.iterations = it + 1;
        res.finalSq = e[0];
        if (is_set(e[3])) { res.converged = e[3] == 1.0; return res; }
        rhoN = e[1];
        beta = e[2];
        small = fabs(rhoN) < 1e-30;
    }
    return res;
}

}  // namespace btm
