// euler_block.cuh -- 3D compressible Euler (HLLC) on blocks of cells, every face of a block once:
// residual, J v and J^T w for Q = K + 1 nodes per direction.
//
// A CTA owns a block of cells (coefficients and result in shared memory):
//   volume  one warp per cell (several cells of low degree): (field, z-slab) lanes contract z and y to
//           node rows, node lanes evaluate the state once and the flux direction by direction,
//           (field, slab) lanes project; only warp barriers;
//   faces   per direction: (face, side, field) threads take the normal trace of the 20 (k = 3)
//           coefficients and expand it to node rows in registers, (face, node) threads evaluate
//           the flux or its adjoint, (face, field) threads project the nodes onto the face modes,
//           (cell, field, pair) threads add both faces of a cell. The cells behind the block's
//           surface are read from global memory; a face between two blocks is evaluated by both.
// The flux functions see the momentum permuted with the normal component first. What bounds the
// kernel: shared-memory wavefronts (two thirds of their peak) and instruction issue (0.55), ahead
// of the FP64 pipe (0.4); the slab tile evaluated every face twice and repeated the normal
// contraction for each of the Q node rows. Measured on B200 (32^3, k = 3, kernel alone): residual
// 0.31 -> 0.18 ms, J^T w 0.60 -> 0.36 ms; residual + J^T w through the evaluator 0.888 -> 0.54 ms;
// J v 24x17x13, k = 2: 62 -> 39 us.
#pragma once
#include "tile_stage.cuh"

namespace bosss {

template <int K, int MODE>
struct EulerCfg {
    static constexpr int NP = np_of(3, K), NPAIR = (K + 1) * (K + 2) / 2, Q = K + 1;
    static constexpr int NG = MODE == MODE_RES ? 1 : 2;
    static constexpr int NT = NG == 1 ? (K == 1 ? 192 : K == 2 ? 128 : 256) : (K == 1 ? 256 : K == 4 ? 192 : 128);
    static constexpr int NW = NT / 32;
    static constexpr int NC = 5 * NP;                       // coefficients of a cell
    static constexpr int S = NC | 1;
    // threads, block capacity (cells, faces of a direction) and CTAs per SM: swept on B200 (32^3, k = 4:
    // 24^3); the configurations with 12-20 warps per SM differ by 10 % at most
    static constexpr int CELLS = NG == 1 ? (K == 1 ? 32 : K == 2 ? 18 : K == 3 ? 16 : 12) : (K == 1 ? 64 : K == 2 ? 18 : 8);
    static constexpr int FACES = NG == 1 ? (K == 1 ? 48 : K == 2 ? 27 : K == 3 ? 24 : 18) : (K == 1 ? 80 : K == 2 ? 27 : 12);
    static constexpr int MINB = NG == 1 ? (K == 2 ? 4 : K == 4 ? 2 : 3) : (K == 2 || K == 3 ? 3 : 2);
    // strides: a warp holds Q nodes of a row by 32 / Q faces (FST), or the faces of several (side,
    // field) rows (RSTR, OSTR = the face count modulo the 16 bank pairs): two accesses per bank pair
    static constexpr int FST = (K == 1 || K == 3) ? FACES : FACES | 1, CST = CELLS | 1;
    static constexpr int to_bank(int x, int r) { return x + ((r - x) % 16 + 16) % 16; }
    static constexpr int RSTR = to_bank((K + 1) * Q * FST, FACES % 16), OSTR = to_bank(Q * Q * FST, FACES % 16);
    // node rows of a face: [group, side, field][p][q2]; the adjoint's second group is the jump of w
    static constexpr int NROW = 10 + (MODE == MODE_RES ? 0 : MODE == MODE_JVP ? 10 : 5);
    static constexpr int NOUT = MODE == MODE_VJP ? 10 : 5;  // face results: fields, or both sides' fields
    // volume: cells per warp, node rounds, scratch of a warp
    static constexpr int CW = K == 1 ? 3 : K == 2 ? 2 : 1;
    static constexpr int NR = (CW * Q * Q * Q + 31) / 32;
    static constexpr int SLV = (Q * Q) | 1;
    static constexpr int W_ROWS = CW * 5 * Q * Q * (K + 1), W_OUT = CW * 5 * Q * SLV, W_PAIR = CW * 5 * Q * ((2 * NPAIR) | 1);
    static constexpr int WS0 = W_ROWS > W_OUT ? W_ROWS : W_OUT;
    static constexpr int WS = WS0 > W_PAIR ? WS0 : W_PAIR;
    static constexpr int FWORK = NROW * RSTR + NOUT * OSTR;
    static constexpr int WORK = FWORK > NW * WS ? FWORK : NW * WS;
    static constexpr int O_TAB = 0, O_COEF = 2 * Q * (K + 1) + Q + 1;
    static constexpr int O_R = O_COEF + NG * CELLS * S, O_WORK = O_R + NC * CST;
    static constexpr size_t SMEM = sizeof(double) * (O_WORK + WORK);
};

__device__ constexpr double kEulE[5] = {0.70710678118654752440, 1.22474487139158904910, 1.58113883008418966600,
                                        1.87082869338697069279, 2.12132034355964257320};

template <int DIR>
__device__ __forceinline__ constexpr int eul_mode(int m, int p, int r) {
    return DIR == 0 ? mode3(m, p, r) : (DIR == 1 ? mode3(p, m, r) : mode3(p, r, m));
}

// HLLC flux through a face normal to the first momentum component (the caller permutes), as
// PhysEuler::inner. The divisions by the two wave-speed differences share one reciprocal of their product;
// the densities have one each: their product leaves the double range where the densities do not,
// and a NaN or zero density of one side would reach the flux of the other
template <class T>
__device__ __forceinline__ void hllc_flux(const PhysParams& p, const T* UA, const T* UB, T* f) {
    const double MS = p.gamma * p.mach * p.mach, G2 = 0.5 * (p.gamma + 1.0) / p.gamma, gm1 = p.gamma - 1.0;
    constexpr int N = 0;
    const T irA = 1.0 / UA[0], irB = 1.0 / UB[0];
    const T unA = UA[1 + N] * irA, unB = UB[1 + N] * irB;
    const T kA = (UA[1] * UA[1] + UA[2] * UA[2] + UA[3] * UA[3]) * irA;
    const T kB = (UB[1] * UB[1] + UB[2] * UB[2] + UB[3] * UB[3]) * irB;
    const T pA = (UA[4] - kA * (MS * 0.5)) * gm1, pB = (UB[4] - kB * (MS * 0.5)) * gm1;
    const T cA = dsqrt(pA * irA) * p.imach, cB = dsqrt(pB * irB) * p.imach;
    T pS = (pA + pB) * 0.5 - (unB - unA) * (cA + cB) * (UA[0] + UB[0]) * (0.125 * MS);
    if (0.0 > pval(pS)) pS = T(0.0);
    T sA = unA - cA, sB = unB + cB;
    if (pval(pS) > pval(pA)) sA = unA - cA * dsqrt(1.0 + (pS / pA - 1.0) * G2);
    if (pval(pS) > pval(pB)) sB = unB + cB * dsqrt(1.0 + (pS / pB - 1.0) * G2);
    const T CA = UA[0] * (sA - unA), CB = UB[0] * (sB - unB);
    const T S = (CB * unB - CA * unA + (pA - pB) * p.ims) / (CB - CA);
    const bool left = pval(S) > 0.0;
    T U[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) U[i] = left ? UA[i] : UB[i];
    const T pp = left ? pA : pB, un = left ? unA : unB, s = left ? sA : sB;
    f[0] = U[1 + N];
#pragma unroll
    for (int c = 0; c < 3; ++c) f[c + 1] = un * U[c + 1];
    f[1 + N] = f[1 + N] + pp * p.ims;
    f[4] = un * (U[4] + pp);
    if (left ? (pval(s) <= 0.0) : (pval(s) >= 0.0)) {
        const T sa = s - un, sS = s - S, t = S - un;
        const T iss = 1.0 / (sa * sS);
        const T ratio = sa * sa * iss;
        f[0] = f[0] + s * (U[0] * ratio - U[0]);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const T m = (c == N) ? U[c + 1] + U[0] * t : U[c + 1];
            f[c + 1] = f[c + 1] + s * (ratio * m - U[c + 1]);
        }
        const T factor = U[0] * S * MS + pp * (sS * iss);
        f[4] = f[4] + s * (ratio * (U[4] + factor * t) - U[4]);
    }
}

// gradient of sum_c f_c(UA, UB) fb[c] with respect to both states, as PhysEuler::inner_adj
__device__ __forceinline__ void hllc_adj(const PhysParams& p, const double* UA, const double* UB, const double* fb,
                                         double* UAb, double* UBb) {
    const double g = p.gamma, gm1 = g - 1.0, MS = g * p.mach * p.mach, iMS = p.ims, G2 = 0.5 * (g + 1.0) / g;
    constexpr int N = 0;
    const double rA = UA[0], rB = UB[0], irA = 1.0 / rA, irB = 1.0 / rB;
    const double unA = UA[1 + N] * irA, unB = UB[1 + N] * irB;
    const double kA = (UA[1] * UA[1] + UA[2] * UA[2] + UA[3] * UA[3]) * irA;
    const double kB = (UB[1] * UB[1] + UB[2] * UB[2] + UB[3] * UB[3]) * irB;
    const double pA = (UA[4] - kA * (MS * 0.5)) * gm1, pB = (UB[4] - kB * (MS * 0.5)) * gm1;
    const double yA = pA * irA, yB = pB * irB;
    const double cA = sqrt(yA) * p.imach, cB = sqrt(yB) * p.imach;
    const double rM = (rA + rB) * 0.5, cM = (cA + cB) * 0.5, vJ = unB - unA;
    const double pSraw = (pA + pB) * 0.5 - vJ * cM * rM * (0.5 * MS);
    const bool clamp = 0.0 > pSraw;
    const double pS = clamp ? 0.0 : pSraw;
    const bool qAact = pS > pA, qBact = pS > pB;
    const double ipA = qAact ? 1.0 / pA : 0.0, ipB = qBact ? 1.0 / pB : 0.0;
    const double qA = qAact ? sqrt(1.0 + (pS * ipA - 1.0) * G2) : 1.0;
    const double qB = qBact ? sqrt(1.0 + (pS * ipB - 1.0) * G2) : 1.0;
    const double sA = unA - cA * qA, sB = unB + cB * qB;
    const double CA = rA * (sA - unA), CB = rB * (sB - unB);
    const double iDd = 1.0 / (CB - CA);
    const double S = (CB * unB - CA * unA + (pA - pB) * iMS) * iDd;
    const bool left = S > 0.0;
    const bool star = left ? (sA <= 0.0) : (sB >= 0.0);
    // reverse: the upwind side's flux
    const double r = left ? rA : rB, E = left ? UA[4] : UB[4], pp = left ? pA : pB, un = left ? unA : unB, s = left ? sA : sB;
    double m[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) m[c] = left ? UA[c + 1] : UB[c + 1];
    double rb = fb[0] * un, unb = fb[0] * r + fb[4] * (E + pp), Eb = fb[4] * un, pb = fb[4] * un + fb[1 + N] * iMS;
    double sb = 0.0, Sb = 0.0, mb[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        unb += fb[c + 1] * m[c];
        mb[c] = fb[c + 1] * un;
    }
    if (star) {
        const double a = s - un, b = s - S, iab = 1.0 / (a * b), ia = b * iab, ib = a * iab, rr = a * ib, t = S - un,
                     r1 = rr - 1.0;
        double rrb = fb[0] * s * r;
        sb += fb[0] * r * r1;
        rb += fb[0] * s * r1;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double w = fb[c + 1], wb = w * s;
            sb += w * r1 * m[c];
            rrb += wb * m[c];
            mb[c] += wb * r1;
        }
        const double wN = fb[1 + N], wbN = wN * s;
        sb += wN * r * rr * t;
        rrb += wbN * r * t;
        rb += wbN * rr * t;
        double tb = wbN * r * rr;
        const double factor = r * S * MS + pp * ia, ef = E + factor * t;
        const double mEb = fb[4] * s;
        sb += fb[4] * (rr * ef - E);
        Eb += mEb * r1;
        rrb += mEb * ef;
        const double fab = mEb * rr * t;
        tb += mEb * rr * factor;
        rb += fab * S * MS;
        Sb += fab * r * MS;
        pb += fab * ia;
        const double ab = -fab * pp * ia * ia + rrb * ib;
        const double bb = -rrb * rr * ib;
        sb += ab + bb;
        unb -= ab + tb;
        Sb += tb - bb;
    }
    double rAb = left ? rb : 0.0, rBb = left ? 0.0 : rb, pAb = left ? pb : 0.0, pBb = left ? 0.0 : pb;
    double unAb = left ? unb : 0.0, unBb = left ? 0.0 : unb, sAb = left ? sb : 0.0, sBb = left ? 0.0 : sb;
    // contact speed S = (CB unB - CA unA + (pA - pB)/MS) / (CB - CA)
    const double Nb = Sb * iDd, Ddb = -Nb * S;
    const double CAb = -Ddb - Nb * unA, CBb = Ddb + Nb * unB;
    unBb += Nb * CB;
    unAb -= Nb * CA;
    pAb += Nb * iMS;
    pBb -= Nb * iMS;
    rAb += CAb * (sA - unA);
    sAb += CAb * rA;
    unAb -= CAb * rA;
    rBb += CBb * (sB - unB);
    sBb += CBb * rB;
    unBb -= CBb * rB;
    // wave speeds
    unAb += sAb;
    unBb += sBb;
    double cAb = -sAb * qA, cBb = sBb * qB, pSb = 0.0;
    if (qAact) {
        const double zb = -sAb * cA * 0.5 / qA * G2 * ipA;
        pSb += zb;
        pAb -= zb * pS * ipA;
    }
    if (qBact) {
        const double zb = sBb * cB * 0.5 / qB * G2 * ipB;
        pSb += zb;
        pBb -= zb * pS * ipB;
    }
    if (!clamp) {
        const double h = 0.5 * MS;
        pAb += 0.5 * pSb;
        pBb += 0.5 * pSb;
        const double ph = pSb * h;
        const double vJb = -ph * cM * rM;
        unBb += vJb;
        unAb -= vJb;
        const double cMb = -ph * vJ * rM;
        cAb += 0.5 * cMb;
        cBb += 0.5 * cMb;
        const double rMb = -ph * vJ * cM;
        rAb += 0.5 * rMb;
        rBb += 0.5 * rMb;
    }
    // primitives of each side: c = sqrt(p / rho) / Ma, p, un
    const double i2M2 = 0.5 * p.imach * p.imach;
    {
        const double yb = cAb * i2M2 / cA;
        pAb += yb * irA;
        const double kb = -pAb * gm1 * (MS * 0.5), mk = 2.0 * kb * irA, ub = unAb * irA;
        UAb[0] = rAb - (yb * yA + kb * kA + unAb * unA) * irA;
#pragma unroll
        for (int d = 0; d < 3; ++d) UAb[d + 1] = (left ? mb[d] : 0.0) + mk * UA[d + 1] + (d == N ? ub : 0.0);
        UAb[4] = (left ? Eb : 0.0) + pAb * gm1;
    }
    {
        const double yb = cBb * i2M2 / cB;
        pBb += yb * irB;
        const double kb = -pBb * gm1 * (MS * 0.5), mk = 2.0 * kb * irB, ub = unBb * irB;
        UBb[0] = rBb - (yb * yB + kb * kB + unBb * unB) * irB;
#pragma unroll
        for (int d = 0; d < 3; ++d) UBb[d + 1] = (left ? 0.0 : mb[d]) + mk * UB[d + 1] + (d == N ? ub : 0.0);
        UBb[4] = (left ? 0.0 : Eb) + pBb * gm1;
    }
}

// ------------------------------------------------------------------ volume
// node rows of one field and slab (contraction over z and y): rows[(a * Q + qy) * NT], NT tasks a warp
template <int K, int NT, int DZ, int DY>
__device__ __forceinline__ void eul_vol_rows(const Tables1D& t, const double* c, const double* tA, const double* tdA, int qz,
                                             double fz, double* rows) {
    constexpr int Q = K + 1, NPAIR = (K + 1) * (K + 2) / 2;
    double T1[NPAIR], z[K + 1];
#pragma unroll
    for (int q = 0; q <= K; ++q) z[q] = (DZ ? tdA : tA)[qz * (K + 1) + q] * fz;
    int pr = 0;
#pragma unroll
    for (int a = 0; a <= K; ++a)
#pragma unroll
        for (int b = 0; b <= K - a; ++b, ++pr) {
            double s = 0.0;
#pragma unroll
            for (int q = 0; q <= K - a - b; ++q) s += c[mode3(a, b, q)] * z[q];
            T1[pr] = s;
        }
#pragma unroll
    for (int qy = 0; qy < Q; ++qy) {
        int i = 0;
#pragma unroll
        for (int a = 0; a <= K; ++a) {
            double s = 0.0;
#pragma unroll
            for (int b = 0; b <= K - a; ++b, ++i) s += T1[i] * (DY ? t.dA[qy][b] : t.A[qy][b]);
            rows[(a * Q + qy) * NT] = s;
        }
    }
}

// project one component of a slab: P2[a, b] += sum_xy g X[qx][a] Y[qy][b]
template <int K, int DX, int DY>
__device__ __forceinline__ void eul_vol_project(const Tables1D& t, const double* o, double* P2) {
    constexpr int Q = K + 1;
#pragma unroll
    for (int qy = 0; qy < Q; ++qy) {
        double P[K + 1];
#pragma unroll
        for (int a = 0; a <= K; ++a) P[a] = 0.0;
#pragma unroll
        for (int qx = 0; qx < Q; ++qx) {
            const double g = o[qy * Q + qx];
#pragma unroll
            for (int a = DX ? 1 : 0; a <= K; ++a) P[a] += g * (DX ? t.dA[qx][a] : t.A[qx][a]);
        }
        int i = 0;
#pragma unroll
        for (int a = 0; a <= K; ++a)
#pragma unroll
            for (int b = 0; b <= K - a; ++b, ++i) P2[i] += P[a] * (DY ? t.dA[qy][b] : t.A[qy][b]);
    }
}

// The node rounds r of a warp are separate code, and with two cells per warp (k = 2) a cell's nodes fall into other
// rounds by its place in the block: every contraction is written out as fma, or the compiler's choice (which of two
// products it fuses) would differ between rounds and a cell's bits would depend on the block it lies in
template <int K, int MODE>
__device__ __forceinline__ void eul_volume(const EvalArgs& a, const double* tA, const double* tdA, const double* tw,
                                           const double* coef, double* work, double* R, int ncell) {
    using C = EulerCfg<K, MODE>;
    constexpr int Q = C::Q, NP = C::NP, NPAIR = C::NPAIR, QV = Q * Q * Q, CW = C::CW, NR = C::NR, SLV = C::SLV;
    constexpr int NTASK = CW * 5 * Q;   // rows: [a][qy][cell, field, qz]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* sw = work + warp * C::WS;
    const PhysParams& ph = a.ph;
    const double gm1 = ph.gamma - 1.0, gMs = ph.gamma * ph.mach * ph.mach;
    for (int c0 = warp * CW; c0 < ncell; c0 += C::NW * CW) {
        const int tc = lane / (5 * Q), tf = (lane / Q) % 5, tz = lane % Q;
        const bool task = lane < NTASK && c0 + tc < ncell;
        const double* cu = coef + (c0 + (task ? tc : 0)) * C::S + tf * NP;
        const double* cv = cu + C::CELLS * C::S;
        double* myrow = sw + (task ? lane : 0);
        const int QQ = Q * Q;
        auto read = [&](double (*st)[5], auto dxc) {   // node values from the rows
            constexpr int DX = decltype(dxc)::value;
            __syncwarp();
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const int n = lane + 32 * r, cc = n / QV, k = n - cc * QV;
                if (n < CW * QV) {
                    const int qx = k % Q, zy = k / Q;
                    const double* x = (DX ? tdA : tA) + qx * (K + 1);
                    const double* rw = sw + (zy % Q) * NTASK + cc * 5 * Q + zy / Q;
#pragma unroll
                    for (int f = 0; f < 5; ++f) {
                        double v = 0.0;
#pragma unroll
                        for (int p = 0; p <= K; ++p) v += rw[p * Q * NTASK + f * Q] * x[p];
                        st[r][f] = v;
                    }
                }
            }
            __syncwarp();
        };
        double P2[NPAIR], P2z[NPAIR];
#pragma unroll
        for (int i = 0; i < NPAIR; ++i) P2[i] = P2z[i] = 0.0;
        double u[NR][5];
        if (task) eul_vol_rows<K, NTASK, 0, 0>(a.tab, cu, tA, tdA, tz, a.g.scaling, myrow);
        read(u, std::integral_constant<int, 0>{});
        if constexpr (MODE == MODE_VJP) {
            // state -> velocities u[0..2], (E + p) / rho in u[3]; adjoint accumulated direction by direction
            double b[NR][5];
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const double ir = 1.0 / u[r][0];
                const double v0 = u[r][1] * ir, v1 = u[r][2] * ir, v2 = u[r][3] * ir;
                const double kin = fma(u[r][3], v2, fma(u[r][2], v1, u[r][1] * v0)), E = u[r][4];
                const double eint = fma(kin, -0.5 * gMs, E);
                u[r][0] = v0;
                u[r][1] = v1;
                u[r][2] = v2;
                u[r][3] = fma(eint, gm1, E) * ir;
                u[r][4] = fma(v2, v2, fma(v1, v1, v0 * v0));
#pragma unroll
                for (int i = 0; i < 5; ++i) b[r][i] = 0.0;
            }
            auto dirn = [&](auto dc) {
                constexpr int DIR = decltype(dc)::value;
                double g[NR][5];
                if (task)
                    eul_vol_rows<K, NTASK, DIR == 2, DIR == 1>(a.tab, cv, tA, tdA, tz, a.g.scaling * a.g.twoh[DIR], myrow);
                read(g, std::integral_constant<int, DIR == 0>{});
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const double ud = u[r][DIR], h = u[r][3], usq = u[r][4];
                    const double q = fma(h, g[r][4], fma(u[r][2], g[r][3], fma(u[r][1], g[r][2], u[r][0] * g[r][1])));
                    const double P = fma(ud, g[r][4], ph.ims * g[r][1 + DIR]);
                    const double kp = gMs * gm1 * P;
                    b[r][0] = fma(ud, q, fma(-0.5 * kp, usq, b[r][0]));
#pragma unroll
                    for (int c = 0; c < 3; ++c) b[r][1 + c] = fma(kp, u[r][c], fma(-ud, g[r][1 + c], b[r][1 + c]));
                    b[r][1 + DIR] -= g[r][0] + q;
                    b[r][4] = fma(-gm1, P, fma(-ud, g[r][4], b[r][4]));
                }
            };
            dirn(std::integral_constant<int, 0>{});
            dirn(std::integral_constant<int, 1>{});
            dirn(std::integral_constant<int, 2>{});
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const int n = lane + 32 * r, cc = n / QV, k = n - cc * QV;
                if (n < CW * QV) {
                    const double f = tw[k % Q] * tw[(k / Q) % Q] * tw[k / QQ] * a.g.detJ * a.g.scaling;
#pragma unroll
                    for (int i = 0; i < 5; ++i) sw[((cc * 5 + i) * Q + k / QQ) * SLV + k % QQ] = b[r][i] * f;
                }
            }
            __syncwarp();
            if (task) eul_vol_project<K, 0, 0>(a.tab, sw + lane * SLV, P2);
        } else {
            // RES: F_d; JVP: dF_d
            double vl[NR][MODE == MODE_JVP ? 5 : 1];
            if constexpr (MODE == MODE_JVP) {
                if (task) eul_vol_rows<K, NTASK, 0, 0>(a.tab, cv, tA, tdA, tz, a.g.scaling, myrow);
                read(vl, std::integral_constant<int, 0>{});
            }
            // u: [ir | u_d ...]: velocities in w, enthalpy E + p in u[0], momenta in u[1..3], p / MS in u[4]
            double w[NR][3], wt[NR][MODE == MODE_JVP ? 3 : 1];
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const double ir = 1.0 / u[r][0];
                double kin = 0.0;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    w[r][c] = u[r][1 + c] * ir;
                    kin = fma(u[r][1 + c], w[r][c], kin);
                }
                const double eint = fma(kin, -0.5 * gMs, u[r][4]);   // p / (gamma - 1)
                if constexpr (MODE == MODE_JVP) {
                    double kt = 0.0;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        wt[r][c] = fma(-w[r][c], vl[r][0], vl[r][1 + c]) * ir;
                        kt = fma(vl[r][1 + c], w[r][c], fma(u[r][1 + c], wt[r][c], kt));
                    }
                    const double et = fma(kt, -0.5 * gMs, vl[r][4]);
                    vl[r][0] = fma(et, gm1, vl[r][4]);
                    vl[r][4] = et * gm1 * ph.ims;
                }
                u[r][0] = fma(eint, gm1, u[r][4]);
                u[r][4] = eint * gm1 * ph.ims;
            }
            auto dirn = [&](auto dc) {
                constexpr int DIR = decltype(dc)::value;
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const int n = lane + 32 * r, cc = n / QV, k = n - cc * QV;
                    if (n < CW * QV) {
                        const double f = -tw[k % Q] * tw[(k / Q) % Q] * tw[k / QQ] * a.g.detJ * a.g.scaling * a.g.twoh[DIR];
                        double* o = sw + (cc * 5 * Q + k / QQ) * SLV + k % QQ;
                        double F[5];
                        if constexpr (MODE == MODE_RES) {
                            F[0] = u[r][1 + DIR];
#pragma unroll
                            for (int c = 0; c < 3; ++c)
                                F[1 + c] = c == DIR ? fma(u[r][1 + c], w[r][DIR], u[r][4]) : u[r][1 + c] * w[r][DIR];
                            F[4] = w[r][DIR] * u[r][0];
                        } else {
                            F[0] = vl[r][1 + DIR];
#pragma unroll
                            for (int c = 0; c < 3; ++c)
                                F[1 + c] = fma(vl[r][1 + c], w[r][DIR],
                                               c == DIR ? fma(u[r][1 + c], wt[r][DIR], vl[r][4]) : u[r][1 + c] * wt[r][DIR]);
                            F[4] = fma(wt[r][DIR], u[r][0], w[r][DIR] * vl[r][0]);
                        }
#pragma unroll
                        for (int i = 0; i < 5; ++i) o[i * Q * SLV] = F[i] * f;
                    }
                }
                __syncwarp();
                if (task) eul_vol_project<K, DIR == 0, DIR == 1>(a.tab, sw + lane * SLV, DIR == 2 ? P2z : P2);
                __syncwarp();
            };
            dirn(std::integral_constant<int, 0>{});
            dirn(std::integral_constant<int, 1>{});
            dirn(std::integral_constant<int, 2>{});
        }
        // contraction over z, (cell, field, pair) lanes
        __syncwarp();
        constexpr int PS = (2 * NPAIR) | 1;
        if (task) {
#pragma unroll
            for (int i = 0; i < NPAIR; ++i) {
                sw[lane * PS + i] = P2[i];
                sw[lane * PS + NPAIR + i] = P2z[i];
            }
        }
        __syncwarp();
        for (int t = lane; t < CW * 5 * NPAIR; t += 32) {
            const int pr = t % NPAIR, cf = t / NPAIR, cc = cf / 5, f = cf % 5;
            if (c0 + cc >= ncell) continue;
            int p = 0, b = pr;
            while (b > K - p) {
                b -= K + 1 - p;
                ++p;
            }
            double acc[K + 1];
#pragma unroll
            for (int q = 0; q <= K; ++q) acc[q] = 0.0;
#pragma unroll
            for (int qz = 0; qz < Q; ++qz) {
                const double s = sw[(cf * Q + qz) * PS + pr], z = sw[(cf * Q + qz) * PS + NPAIR + pr];
#pragma unroll
                for (int q = 0; q <= K; ++q) {
                    acc[q] += s * a.tab.A[qz][q];
                    if (MODE != MODE_VJP && q > 0) acc[q] += z * a.tab.dA[qz][q];
                }
            }
#pragma unroll
            for (int q = 0; q <= K; ++q)
                if (q <= K - p - b) R[(f * NP + mode3(p, b, q)) * C::CST + c0 + cc] = acc[q];
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------ faces
// normal trace (side 0: at +1, side 1: at -1) of NP coefficients, expanded to node rows [p][q2]
template <int K, int DIR>
__device__ __forceinline__ void eul_trace(const double* cf, int side, double sc, double* T) {
    int pr = 0;
#pragma unroll
    for (int p = 0; p <= K; ++p)
#pragma unroll
        for (int r = 0; r <= K - p; ++r, ++pr) {
            double e = 0.0, o = 0.0;
#pragma unroll
            for (int m = 0; m <= K - p - r; ++m) {
                const double v = cf[eul_mode<DIR>(m, p, r)] * kEulE[m];
                if (m & 1) o += v;
                else e += v;
            }
            T[pr] = (side ? e - o : e + o) * sc;
        }
}

template <int K>
__device__ __forceinline__ void eul_expand(const Tables1D& t, const double* T, double* out, int FST) {
    constexpr int Q = K + 1;
#pragma unroll
    for (int q2 = 0; q2 < Q; ++q2) {
        int pr = 0;
#pragma unroll
        for (int p = 0; p <= K; ++p) {
            double v = 0.0;
#pragma unroll
            for (int r = 0; r <= K - p; ++r, ++pr) v += T[pr] * t.A[q2][r];
            out[(p * Q + q2) * FST] = v;
        }
    }
}

struct EulTile {
    int b1, b2, ncell;
};

// coefficients of field f of the cell on side `side` of face (f0, f1, f2); false: no such cell
template <int K, int MODE, int DIR>
__device__ __forceinline__ bool eul_load(const EvalArgs& a, const TileGeom& G, const EulTile& tl, const double* coef,
                                         const double* __restrict__ glob, int f0, int f1, int f2, int side, int f, double* cf) {
    using C = EulerCfg<K, MODE>;
    const int md = G.mem(DIR);
    const int at = (md == 0 ? f0 : md == 1 ? f1 : f2) - 1 + side;
    const int ee = md == 0 ? G.e[0] : md == 1 ? G.e[1] : G.e[2];
    const int oo = md == 0 ? G.o[0] : md == 1 ? G.o[1] : G.o[2];
    const int nn = md == 0 ? G.n[0] : md == 1 ? G.n[1] : G.n[2];
    const int pp = md == 0 ? G.per[0] : md == 1 ? G.per[1] : G.per[2];
    if (at >= 0 && at < ee) {
        const int c = md == 0 ? (at * tl.b1 + f1) * tl.b2 + f2 : md == 1 ? (f0 * tl.b1 + at) * tl.b2 + f2
                                                                         : (f0 * tl.b1 + f1) * tl.b2 + at;
        const double* s = coef + c * C::S + f * C::NP;
#pragma unroll
        for (int n = 0; n < C::NP; ++n) cf[n] = s[n];
        return true;
    }
    int gi = oo + at;
    if (gi < 0 || gi >= nn) {
        if (!pp) return false;
        gi = gi < 0 ? gi + nn : gi - nn;
    }
    const int m0 = md == 0 ? gi : G.o[0] + f0, m1 = md == 1 ? gi : G.o[1] + f1, m2 = md == 2 ? gi : G.o[2] + f2;
    const double* s = glob + (((long long)m0 * G.n[1] + m1) * G.n[2] + m2) * C::NC + f * C::NP;
#pragma unroll
    for (int n = 0; n < C::NP; ++n) cf[n] = __ldg(s + n);
    return true;
}

template <int K, int MODE, int DIR>
__device__ __forceinline__ void eul_face_rows(const EvalArgs& a, const TileGeom& G, const EulTile& tl, const double* coef,
                                              double* rw, int fd1, int fd2, int nf, int t) {
    using C = EulerCfg<K, MODE>;
    const double sc = a.g.scaling;
    {
        const int k = t / nf, fc = t - k * nf;
        const int f2 = fc % fd2, fq = fc / fd2, f1 = fq % fd1, f0 = fq / fd1;
        double cf[C::NP], T[C::NPAIR];
        if (MODE == MODE_VJP && k >= 10) {
            const int f = k - 10;
            double T2[C::NPAIR];
#pragma unroll
            for (int i = 0; i < C::NPAIR; ++i) T[i] = T2[i] = 0.0;
            const double* cv = coef + C::CELLS * C::S;
            const bool hA = eul_load<K, MODE, DIR>(a, G, tl, cv, a.V, f0, f1, f2, 0, f, cf);
            if (hA) eul_trace<K, DIR>(cf, 0, sc, T);
            const bool hB = eul_load<K, MODE, DIR>(a, G, tl, cv, a.V, f0, f1, f2, 1, f, cf);
            if (hB) eul_trace<K, DIR>(cf, 1, sc, T2);
#pragma unroll
            for (int i = 0; i < C::NPAIR; ++i) T[i] -= T2[i];
        } else {
            const int grp = k / 10, ks = k % 10, side = ks / 5, f = ks % 5;
#pragma unroll
            for (int i = 0; i < C::NPAIR; ++i) T[i] = 0.0;
            if (eul_load<K, MODE, DIR>(a, G, tl, coef + grp * C::CELLS * C::S, grp ? a.V : a.U, f0, f1, f2, side, f, cf))
                eul_trace<K, DIR>(cf, side, sc, T);
        }
        eul_expand<K>(a.tab, T, rw + k * C::RSTR + fc, C::FST);
    }
}

// the fluxes at the face nodes; the momentum components are permuted so that the normal one comes
// first, which lets the three directions share this code
template <int K, int MODE>
__device__ __forceinline__ void eul_face_nodes(const EvalArgs& a, const TileGeom& G, const double* tA, const double* tw,
                                               const double* rw, double* ob, int dir, int fd1, int fd2, int nf) {
    using C = EulerCfg<K, MODE>;
    constexpr int Q = C::Q, FST = C::FST;
    const int md = G.mem(dir);
    const double fs = a.g.faceSG[dir] * a.g.scaling;
    const int c1 = 1 + dir, c2 = dir == 0 ? 2 : 1, c3 = dir == 2 ? 2 : 3;   // normal, other components
    auto comp = [&](int i) { return i == 1 ? c1 : i == 2 ? c2 : i == 3 ? c3 : i; };
    for (int t = threadIdx.x; t < Q * Q * nf; t += C::NT) {
        const int q1 = t % Q, rest = t / Q, q2 = rest / nf, fc = rest - q2 * nf;
        const int f2 = fc % fd2, fq = fc / fd2, f1 = fq % fd1, f0 = fq / fd1;
        const int gi = md == 0 ? G.o[0] + f0 : md == 1 ? G.o[1] + f1 : G.o[2] + f2;
        const bool inner = (gi > 0 && gi < a.g.n[dir]) || a.g.periodic[dir];
        double x[K + 1];
#pragma unroll
        for (int p = 0; p <= K; ++p) x[p] = tA[q1 * (K + 1) + p];
        auto val = [&](int k) {
            const double* r = rw + k * C::RSTR + q2 * FST + fc;
            double v = 0.0;
#pragma unroll
            for (int p = 0; p <= K; ++p) v += r[p * Q * FST] * x[p];
            return v;
        };
        const double fac = tw[q1] * tw[q2] * fs;
        double* o = ob + (q2 * Q + q1) * FST + fc;
        constexpr int OS = C::OSTR;
        if (!inner) {   // prescribed-state boundaries run on the generic kernel: no term here
#pragma unroll
            for (int i = 0; i < C::NOUT; ++i) o[i * OS] = 0.0;
            continue;
        }
        if constexpr (MODE == MODE_RES) {
            double UA[5], UB[5], f[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                UA[i] = val(comp(i));
                UB[i] = val(5 + comp(i));
            }
            hllc_flux<double>(a.ph, UA, UB, f);
#pragma unroll
            for (int i = 0; i < 5; ++i) o[comp(i) * OS] = f[i] * fac;
        } else if constexpr (MODE == MODE_JVP) {
            DualN<1> UA[5], UB[5], f[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                UA[i].v = val(comp(i));
                UB[i].v = val(5 + comp(i));
                UA[i].d[0] = val(10 + comp(i));
                UB[i].d[0] = val(15 + comp(i));
            }
            hllc_flux<DualN<1>>(a.ph, UA, UB, f);
#pragma unroll
            for (int i = 0; i < 5; ++i) o[comp(i) * OS] = f[i].d[0] * fac;
        } else {
            double UA[5], UB[5], fb[5], A[5], B[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                UA[i] = val(comp(i));
                UB[i] = val(5 + comp(i));
                fb[i] = val(10 + comp(i)) * fac;
            }
            hllc_adj(a.ph, UA, UB, fb, A, B);
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                o[comp(i) * OS] = A[i];
                o[(5 + comp(i)) * OS] = B[i];
            }
        }
    }
}

// node results of (face, output) onto the face modes, in place
template <int K, int MODE>
__device__ __forceinline__ void eul_face_project(const Tables1D& t1, double* ob, int nf) {
    using C = EulerCfg<K, MODE>;
    constexpr int Q = C::Q, FST = C::FST, NPAIR = C::NPAIR;
    for (int t = threadIdx.x; t < C::NOUT * nf; t += C::NT) {
        const int k = t / nf, fc = t - k * nf;
        double* o = ob + k * C::OSTR + fc;
        double W[NPAIR];
#pragma unroll
        for (int i = 0; i < NPAIR; ++i) W[i] = 0.0;
#pragma unroll
        for (int q2 = 0; q2 < Q; ++q2) {
            double P[K + 1];
#pragma unroll
            for (int p = 0; p <= K; ++p) P[p] = 0.0;
#pragma unroll
            for (int q1 = 0; q1 < Q; ++q1) {
                const double v = o[(q2 * Q + q1) * FST];
#pragma unroll
                for (int p = 0; p <= K; ++p) P[p] += v * t1.A[q1][p];
            }
            int i = 0;
#pragma unroll
            for (int p = 0; p <= K; ++p)
#pragma unroll
                for (int r = 0; r <= K - p; ++r, ++i) W[i] += P[p] * t1.A[q2][r];
        }
#pragma unroll
        for (int i = 0; i < NPAIR; ++i) o[i * FST] = W[i];
    }
}

// both faces of one cell, one field: face modes times the traces of the test functions
template <int K, int MODE, int DIR>
__device__ __forceinline__ void eul_face_add(const TileGeom& G, const EulTile& tl, const double* ob, double* R, int fd1, int fd2,
                                             int t) {
    using C = EulerCfg<K, MODE>;
    const int md = G.mem(DIR);
    const int fstep = md == 0 ? fd1 * fd2 : md == 1 ? fd2 : 1;
    const int f = t / tl.ncell, c = t - f * tl.ncell;
    const int l2 = c % tl.b2, lq = c / tl.b2, l1 = lq % tl.b1, l0 = lq / tl.b1;
    if (l0 >= G.e[0] || l1 >= G.e[1] || l2 >= G.e[2]) return;
    const int fl = (l0 * fd1 + l1) * fd2 + l2;
    // upper face: the cell is the lower side (+f); lower face: the upper side (-f, or its own adjoint)
    const double* ou = ob + f * C::OSTR + fl + fstep;
    const double* ol = ob + (MODE == MODE_VJP ? 5 + f : f) * C::OSTR + fl;
    double* r0 = R + f * C::NP * C::CST + c;
    int pr = 0;
#pragma unroll
    for (int p = 0; p <= K; ++p)
#pragma unroll
        for (int r = 0; r <= K - p; ++r, ++pr) {
            const double gu = ou[pr * C::FST], gl = MODE == MODE_VJP ? ol[pr * C::FST] : -ol[pr * C::FST];
            const double gs = gu + gl, gd = gu - gl;
#pragma unroll
            for (int m = 0; m <= K - p - r; ++m) r0[eul_mode<DIR>(m, p, r) * C::CST] += ((m & 1) ? gd : gs) * kEulE[m];
        }
}

template <int K, int MODE>
__global__ void __launch_bounds__(EulerCfg<K, MODE>::NT, EulerCfg<K, MODE>::MINB)
k_euler_block(const __grid_constant__ EvalArgs a, const __grid_constant__ ModalTile mt) {
    using C = EulerCfg<K, MODE>;
    constexpr int Q = C::Q, NC = C::NC;
    extern __shared__ double sm[];
    double* tA = sm + C::O_TAB;
    double* tdA = tA + Q * (K + 1);
    double* tw = tdA + Q * (K + 1);
    double* coef = sm + C::O_COEF;
    double* R = sm + C::O_R;
    double* rw = sm + C::O_WORK;
    double* ob = rw + C::NROW * C::RSTR;
    const TileGeom G = tile_geom(a.g, mt, blockIdx.x);
    const EulTile tl{mt.b[1], mt.b[2], mt.ncell};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < Q * (K + 1); i += C::NT) {
        tA[i] = a.tab.A[i / (K + 1)][i % (K + 1)];
        tdA[i] = a.tab.dA[i / (K + 1)][i % (K + 1)];
    }
    if (threadIdx.x < Q) tw[threadIdx.x] = a.tab.w[threadIdx.x];
    for (int r = warp; r < G.e[0] * G.e[1]; r += C::NW) {
        const int i0 = r / G.e[1], i1 = r - i0 * G.e[1];
        const long long row = ((long long)(G.o[0] + i0) * G.n[1] + (G.o[1] + i1)) * G.n[2] + G.o[2];
        double* dst = coef + (i0 * tl.b1 + i1) * tl.b2 * C::S;
        for (int e = lane; e < G.e[2] * NC; e += 32) {
            const int c = e / NC;
            tile_cp8(dst + e + c * (C::S - NC), a.U + row * NC + e);
            if constexpr (C::NG > 1) tile_cp8(dst + C::CELLS * C::S + e + c * (C::S - NC), a.V + row * NC + e);
        }
    }
    tile_cp_wait();
    __syncthreads();

    eul_volume<K, MODE>(a, tA, tdA, tw, coef, rw, R, tl.ncell);
    __syncthreads();

    auto dims = [&](int d, int& f0, int& f1, int& f2) {
        const int md = G.mem(d);
        f0 = G.e[0] + (md == 0);
        f1 = G.e[1] + (md == 1);
        f2 = G.e[2] + (md == 2);
    };
    auto rows_add = [&](auto dc) {   // a direction's node rows, and the previous direction's faces into the cells
        constexpr int DIR = decltype(dc)::value;
        int f0, f1, f2, p0 = 0, p1 = 0, p2 = 0;
        dims(DIR, f0, f1, f2);
        if constexpr (DIR > 0) dims(DIR - 1, p0, p1, p2);
        const int nf = f0 * f1 * f2;
        const int nrow = C::NROW * nf, nadd = DIR > 0 ? 5 * tl.ncell : 0;
        for (int t = threadIdx.x; t < nrow + nadd; t += C::NT) {
            if (t < nrow) eul_face_rows<K, MODE, DIR>(a, G, tl, coef, rw, f1, f2, nf, t);
            else if constexpr (DIR > 0) eul_face_add<K, MODE, DIR - 1>(G, tl, ob, R, p1, p2, t - nrow);
        }
    };
#pragma unroll 1
    for (int dir = 0; dir < 3; ++dir) {
        if (dir == 0) rows_add(std::integral_constant<int, 0>{});
        else if (dir == 1) rows_add(std::integral_constant<int, 1>{});
        else rows_add(std::integral_constant<int, 2>{});
        int f0, f1, f2;
        dims(dir, f0, f1, f2);
        const int nf = f0 * f1 * f2;
        __syncthreads();
        eul_face_nodes<K, MODE>(a, G, tA, tw, rw, ob, dir, f1, f2, nf);
        __syncthreads();
        eul_face_project<K, MODE>(a.tab, ob, nf);
        __syncthreads();
    }
    {
        int f0, f1, f2;
        dims(2, f0, f1, f2);
        for (int t = threadIdx.x; t < 5 * tl.ncell; t += C::NT) eul_face_add<K, MODE, 2>(G, tl, ob, R, f1, f2, t);
    }
    __syncthreads();

    for (int r = warp; r < G.e[0] * G.e[1]; r += C::NW) {
        const int i0 = r / G.e[1], i1 = r - i0 * G.e[1];
        const long long row = ((long long)(G.o[0] + i0) * G.n[1] + (G.o[1] + i1)) * G.n[2] + G.o[2];
        const double* src = R + (i0 * tl.b1 + i1) * tl.b2;
        for (int e = lane; e < G.e[2] * NC; e += 32) {
            const int c = e / NC, n = e - c * NC;
            if (row + c < a.cbeg || row + c >= a.cend) continue;
            const double v = src[n * C::CST + c];
            double* q = a.out + row * NC + e;
            if (MODE == MODE_RES) *q = (a.beta == 0.0) ? a.alpha * v : a.beta * *q + a.alpha * v;
            else *q = v;
        }
    }
}

}  // namespace bosss
