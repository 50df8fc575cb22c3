// sip_kernel.cuh -- scalar operators with nonlinear diffusion (SIP with nu(u) = nu0 + nu2 u^2, upwind
// transport, constant source) in three dimensions: residual, J v and J^T w.
//
// A CTA owns a block of cells (tile_stage.cuh) and evaluates every face of the block once:
//   volume   one thread per (cell, z-slab): sum-factorised interpolation row by row, the forms at
//            the nodes of the row and their projection stay in registers; the slabs' partial
//            projections are summed by (cell, x-y pair) threads;
//   faces    per direction: the value and normal-derivative traces as modes of the face (one
//            thread per face side; SIP reads no tangential derivative), one thread per (face, node
//            row) for the forms, then (cell, pencil) threads contract the rows and add both faces
//            of a cell. Faces between two blocks are evaluated by both.
// The quadrature nodes of nu(u) (Q = 2K+1 for order 4K) carry 10-100x the arithmetic of the modes.
// At 48^3 k = 2 the FP64 pipe is 41 % busy and 52 % of the issue slots are used; the rest are the
// latencies between the phases of a block.
//
// Volume nodes: with nu a quadratic of u the volume integrand nu grad u . grad v has total degree
// 4K - 2, so the Gauss rule with 2K nodes per direction (exact to degree 4K - 1) gives the same
// integrals as any larger one; the volume uses min(Q, 2K) nodes (K = 2, Q = 5: 64 instead of 125).
// The faces keep Q: the penalty term reaches degree 4K and takes a maximum of two viscosities.
//
// Measured on B200 against the slab / generic tiles: J v at 48^3 k = 2 (Q = 5) 1.40 -> 0.210 ms,
// residual + J^T w at 21x16x18 k = 4 (Q = 9) 1.14 -> 0.226 ms.
#pragma once
#include "tile_stage.cuh"

namespace bosss {

template <int K, int Q, int MODE>
struct SipCfg {
    static constexpr int NP = np_of(3, K), NPAIR = (K + 1) * (K + 2) / 2;
    static constexpr int QV = Q < 2 * K ? Q : 2 * K, FQ = Q;
    static constexpr int NG = MODE == MODE_RES ? 1 : 2;
    static constexpr int S = NP | 1;
    // threads, largest block, its halo box and its faces per direction (swept on B200; k = 4 residual at
    // 18^3: two CTAs of 192 threads with 16 cells 82 us, one of 256 with 32 cells 92 us)
    static constexpr bool R4 = K == 4 && MODE == MODE_RES;
    static constexpr int NT = R4 ? 192 : 256;
    static constexpr int CELLS = K == 1 ? 128 : K == 2 ? 64 : K == 3 ? 48 : R4 ? 16 : 32;
    static constexpr int SLOTS = K == 1 ? 360 : K == 2 ? 216 : K == 3 ? 180 : R4 ? 96 : 144;
    static constexpr int FACES = K == 1 ? 160 : K == 2 ? 80 : K == 3 ? 64 : R4 ? 24 : 48;
    static constexpr int FST = FACES | 1, CST = CELLS | 1;
    static constexpr int NA = MODE == MODE_VJP ? 4 : 3;      // face results: g, G_A, G_B / g_A, G_A, g_B, G_B
    static constexpr int TR = 4 * NG * NPAIR;                // traces of a face
    static constexpr int ROW = NA * (K + 1) * Q;             // row results of a face
    static constexpr int VP = 2 * NPAIR * QV;                // volume partials of a cell
    static constexpr int O_COEF = 0, O_R = NG * SLOTS * S, O_WORK = O_R + NP * CST;
    static constexpr int WORK = FST * (TR + ROW) > CST * VP ? FST * (TR + ROW) : CST * VP;
    static constexpr size_t SMEM = sizeof(double) * (O_WORK + WORK);
    static constexpr int MINB = SMEM <= 112 * 1024 ? 2 : 1;
};

template <int DIR>
__device__ __forceinline__ constexpr int sip_mode(int m, int p, int r) {
    return DIR == 0 ? mode3(m, p, r) : (DIR == 1 ? mode3(p, m, r) : mode3(p, r, m));
}

// one row of a contraction over y and z: rv[a] = sum_bc c[abc] Ay[b] Az[c], and its y / z derivatives
template <int K>
__device__ __forceinline__ void sip_rows(const double* c, const double* Ay, const double* dAy, const double* Az,
                                         const double* dAz, double* rv, double* ry, double* rz) {
#pragma unroll
    for (int a = 0; a <= K; ++a) {
        double v = 0.0, y = 0.0, z = 0.0;
#pragma unroll
        for (int b = 0; b <= K - a; ++b) {
            double s = 0.0, sz = 0.0;
#pragma unroll
            for (int q = 0; q <= K - a - b; ++q) {
                const double t = c[mode3(a, b, q)];
                s += t * Az[q];
                sz += t * dAz[q];
            }
            v += s * Ay[b];
            y += s * dAy[b];
            z += sz * Ay[b];
        }
        rv[a] = v;
        ry[a] = y;
        rz[a] = z;
    }
}

template <int K, int Q, int MODE, int DIR>
__device__ __forceinline__ void sip_traces(const EvalArgs& a, const TileGeom& G, const double* coef, double* tr, int fd1,
                                           int fd2, int nf, int t) {
    using C = SipCfg<K, Q, MODE>;
    const int md = G.mem(DIR);
    const double sc = a.g.scaling, scn = a.g.scaling * a.g.twoh[DIR];
    {
        const int gs = t / nf, f = t - gs * nf;          // gs = group * 2 + side
        const int side = gs & 1, grp = gs >> 1;
        const int f2 = f % fd2, fq = f / fd2, f1 = fq % fd1, f0 = fq / fd1;
        const int at = (md == 0 ? f0 : md == 1 ? f1 : f2) - 1 + side;   // tile coordinate of the cell
        const int gi = (md == 0 ? G.o[0] : md == 1 ? G.o[1] : G.o[2]) + at;
        const int nn = md == 0 ? G.n[0] : md == 1 ? G.n[1] : G.n[2];
        const int pp = md == 0 ? G.per[0] : md == 1 ? G.per[1] : G.per[2];
        const bool there = (gi >= 0 && gi < nn) || pp;
        const int sl = md == 0 ? G.slot(at, f1, f2) : md == 1 ? G.slot(f0, at, f2) : G.slot(f0, f1, at);
        const double* c = coef + (size_t)grp * C::SLOTS * C::S + sl * C::S;
        double* o = tr + (size_t)gs * 2 * C::NPAIR * C::FST + f;
        int pr = 0;
#pragma unroll
        for (int p = 0; p <= K; ++p)
#pragma unroll
            for (int r = 0; r <= K - p; ++r, ++pr) {
                double ve = 0.0, vo = 0.0, de = 0.0, dq = 0.0;
                if (there) {
#pragma unroll
                    for (int m = 0; m <= K - p - r; ++m) {
                        const double v = c[sip_mode<DIR>(m, p, r)];
                        const double E = a.tab.e[1][m], F = a.tab.de[1][m];   // L_m(1), L_m'(1)
                        if (m & 1) {
                            vo += v * E;
                            dq += v * F;
                        } else {
                            ve += v * E;
                            if (m > 0) de += v * F;
                        }
                    }
                }
                // side 0: the lower cell's trace at +1; side 1: the upper cell's at -1
                o[pr * C::FST] = (side ? ve - vo : ve + vo) * sc;
                o[(C::NPAIR + pr) * C::FST] = (side ? dq - de : de + dq) * scn;
            }
    }
}

// pointwise face terms; s[0..3] = u_A, du_A, u_B, du_B (normal derivatives along +d), s[4..7] the second
// group; results as SipCfg::NA says, without weights
template <int MODE>
__device__ __forceinline__ void sip_face_inner(double vel, double nu0, double nu2, double pnl, const double* s, double* o) {
    const double uA = s[0], dA = s[1], uB = s[2], dB = s[3];
    const double nA = fma(nu2 * uA, uA, nu0), nB = fma(nu2 * uB, uB, nu0);
    const double J = uA - uB;
    const bool mA = fabs(nA) > fabs(nB);
    const double nM = mA ? nA : nB;
    if constexpr (MODE == MODE_RES) {
        double g = 0.5 * (nA * dA + nB * dB) - pnl * nM * J;
        g += vel * (vel > 0.0 ? uA : uB);
        o[0] = g;
        o[1] = 0.5 * nA * J;
        o[2] = 0.5 * nB * J;
    } else if constexpr (MODE == MODE_JVP) {
        const double vA = s[4], eA = s[5], vB = s[6], eB = s[7];
        const double tA = 2.0 * nu2 * uA * vA, tB = 2.0 * nu2 * uB * vB;   // tangents of nu
        const double j = vA - vB, tM = mA ? tA : tB;
        double g = 0.5 * (nA * eA + tA * dA + nB * eB + tB * dB) - pnl * (nM * j + tM * J);
        g += vel * (vel > 0.0 ? vA : vB);
        o[0] = g;
        o[1] = 0.5 * (nA * j + tA * J);
        o[2] = 0.5 * (nB * j + tB * J);
    } else {
        const double wA = s[4], eA = s[5], wB = s[6], eB = s[7];
        const double pA = 2.0 * nu2 * uA, pB = 2.0 * nu2 * uB;             // nu'
        const double jw = wA - wB, sym = 0.5 * (nA * eA + nB * eB) - pnl * nM * jw;
        const double pj = pnl * J * jw;
        double a = sym + pA * (0.5 * (dA * jw + J * eA) - (mA ? pj : 0.0));
        double b = -sym + pB * (0.5 * (dB * jw + J * eB) - (mA ? 0.0 : pj));
        if (vel > 0.0) a += vel * jw;
        else b += vel * jw;
        o[0] = a;
        o[1] = 0.5 * nA * jw;
        o[2] = b;
        o[3] = 0.5 * nB * jw;
    }
}

// boundary face: own traces u, du, second group v, dv; n = +-1 outward along d
template <int MODE>
__device__ __forceinline__ void sip_face_boundary(double vel, bool dir, double nu0, double nu2, double pnl, double n,
                                                  double gD, double u, double du, double v, double dv, double& g, double& Gn) {
    const double an = vel * n, ap = an >= 0.0 ? an : 0.0;
    const double nu = dir ? fma(nu2 * u, u, nu0) : 0.0, df = u - gD;
    if constexpr (MODE == MODE_RES) {
        g = ap * u + nu * (du * n - df * pnl);
        Gn = nu * df * n;
    } else {
        const double nup = dir ? 2.0 * nu2 * u : 0.0;
        if constexpr (MODE == MODE_JVP) {
            const double t = nup * v;
            g = ap * v + t * (du * n - df * pnl) + nu * (dv * n - v * pnl);
            Gn = n * (t * df + nu * v);
        } else {
            g = ap * v + nup * (du * n - df * pnl) * v - nu * pnl * v + n * dv * (nup * df + nu);
            Gn = nu * n * v;
        }
    }
}

template <int K, int Q, int MODE, int DIR>
__device__ __forceinline__ void sip_face_rows(const EvalArgs& a, const TileGeom& G, const double* tr, double* rows, int fd0,
                                              int fd1, int fd2) {
    using C = SipCfg<K, Q, MODE>;
    constexpr int t1 = (DIR == 0) ? 1 : 0, t2 = (DIR == 2) ? 1 : 2;
    const int nf = fd0 * fd1 * fd2;
    const Tables1D& T = a.tab;
    const double vel = a.ph.has_transport ? a.ph.vel[DIR] : 0.0;
    const bool sip = a.ph.has_sip != 0;
    const double nu0 = sip ? a.ph.nu0 : 0.0, nu2 = sip ? a.ph.nu2 : 0.0;
    for (int t = threadIdx.x; t < Q * nf; t += C::NT) {
        const int q2 = t / nf, f = t - q2 * nf;
        const int f2 = f % fd2, fq = f / fd2, f1 = fq % fd1, f0 = fq / fd1;
        const int nn = a.g.n[DIR];
        // physical indices of the upper cell
        int ijk[3];
        {
            const int m0 = G.o[0] + f0, m1 = G.o[1] + f1, m2 = G.o[2] + f2;
            ijk[0] = G.rev ? m2 : m0;
            ijk[1] = m1;
            ijk[2] = G.rev ? m0 : m2;
        }
        const int gi = ijk[DIR];
        const bool per = a.g.periodic[DIR] != 0;
        const bool hasA = gi > 0 || per, hasB = gi < nn || per;
        double Ar[K + 1];
#pragma unroll
        for (int r = 0; r <= K; ++r) Ar[r] = T.A[q2][r];
        // rows of the traces: [group * 2 + side][value, derivative]
        double row[2 * C::NG][2][K + 1];
#pragma unroll
        for (int gs = 0; gs < 2 * C::NG; ++gs)
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                int pr = 0;
#pragma unroll
                for (int p = 0; p <= K; ++p) {
                    double v = 0.0;
#pragma unroll
                    for (int r = 0; r <= K - p; ++r, ++pr) v += tr[((gs * 2 + w) * C::NPAIR + pr) * C::FST + f] * Ar[r];
                    row[gs][w][p] = v;
                }
            }
        double P[C::NA][K + 1];
#pragma unroll
        for (int i = 0; i < C::NA; ++i)
#pragma unroll
            for (int p = 0; p <= K; ++p) P[i][p] = 0.0;
        const double fr = T.w[q2] * a.g.faceSG[DIR] * a.g.scaling, th = a.g.twoh[DIR];
        if (hasA && hasB) {
            double pnl = 0.0;
            if (sip) {
                int iA[3] = {ijk[0], ijk[1], ijk[2]}, iB[3] = {ijk[0], ijk[1], ijk[2]};
                iA[DIR] = gi > 0 ? gi - 1 : nn - 1;
                iB[DIR] = gi < nn ? gi : 0;
                pnl = a.ph.pen * fmax(tile_size<3>(a, iA), tile_size<3>(a, iB));
            }
#pragma unroll
            for (int q1 = 0; q1 < Q; ++q1) {
                double s[8], o[4];
#pragma unroll
                for (int gs = 0; gs < 2 * C::NG; ++gs)
#pragma unroll
                    for (int w = 0; w < 2; ++w) {
                        double v = 0.0;
#pragma unroll
                        for (int p = 0; p <= K; ++p) v += row[gs][w][p] * T.A[q1][p];
                        s[gs * 2 + w] = v;
                    }
                sip_face_inner<MODE>(vel, nu0, nu2, pnl, s, o);
                const double fg = fr * T.w[q1], fG = fg * th;
#pragma unroll
                for (int i = 0; i < C::NA; ++i) {
                    const bool grad = MODE == MODE_VJP ? (i & 1) : i > 0;
                    const double v = o[i] * (grad ? fG : fg);
#pragma unroll
                    for (int p = 0; p <= K; ++p) P[i][p] += v * T.A[q1][p];
                }
            }
        } else {
            const int side = hasA ? 0 : 1;   // the own cell's side
            const double n = hasA ? 1.0 : -1.0;
            const bool dir = sip && a.ph.dirichlet;
            int io[3] = {ijk[0], ijk[1], ijk[2]};
            io[DIR] = hasA ? gi - 1 : gi;
            const double pnl = sip ? 2.0 * a.ph.pen * tile_size<3>(a, io) : 0.0;
            const double xn = a.g.lo[DIR] + (gi + a.g.goff[DIR]) * a.g.h[DIR];
            const double x2 = a.g.lo[t2] + (io[t2] + a.g.goff[t2] + 0.5 + 0.5 * T.xq[q2]) * a.g.h[t2];
            const double gc = a.ph.g0 + (a.ph.g1[DIR] + a.ph.g2[DIR] * xn) * xn + (a.ph.g1[t2] + a.ph.g2[t2] * x2) * x2;
#pragma unroll 1
            for (int q1 = 0; q1 < Q; ++q1) {
                double u[4];
#pragma unroll
                for (int k = 0; k < 2 * C::NG; ++k) {
                    double v = 0.0;
#pragma unroll
                    for (int p = 0; p <= K; ++p)
                        v += (side ? row[(k >> 1) * 2 + 1][k & 1][p] : row[(k >> 1) * 2][k & 1][p]) * T.A[q1][p];
                    u[k] = v;
                }
                const double x1 = a.g.lo[t1] + (io[t1] + a.g.goff[t1] + 0.5 + 0.5 * T.xq[q1]) * a.g.h[t1];
                double g, Gn;
                sip_face_boundary<MODE>(vel, dir, nu0, nu2, pnl, n, gc + (a.ph.g1[t1] + a.ph.g2[t1] * x1) * x1, u[0], u[1],
                                        C::NG > 1 ? u[2] : 0.0, C::NG > 1 ? u[3] : 0.0, g, Gn);
                const double fg = fr * T.w[q1];
                g *= fg;
                Gn *= fg * th;
#pragma unroll
                for (int p = 0; p <= K; ++p) {
                    const double A1 = T.A[q1][p];
                    if (MODE == MODE_VJP) {
                        P[0][p] += side ? 0.0 : g * A1;
                        P[1][p] += side ? 0.0 : Gn * A1;
                        P[2][p] += side ? g * A1 : 0.0;
                        P[C::NA - 1][p] += side ? Gn * A1 : 0.0;
                    } else {
                        P[0][p] += side ? -g * A1 : g * A1;   // the upper cell takes -P[0]
                        P[1][p] += side ? 0.0 : Gn * A1;
                        P[2][p] += side ? Gn * A1 : 0.0;
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < C::NA; ++i)
#pragma unroll
            for (int p = 0; p <= K; ++p) rows[((i * (K + 1) + p) * Q + q2) * C::FST + f] = P[i][p];
    }
}

// one (cell, pencil): rows of the cell's two faces contracted over the second direction and multiplied
// with the traces of the test functions. The pencil is a constant of the branch (the same for a warp
// where the cell count is a multiple of 32)
template <int K, int Q, int MODE, int DIR>
__device__ __forceinline__ void sip_face_add(const EvalArgs& a, const TileGeom& G, const double* rows, double* R, int ncell,
                                             int b1, int b2, int fd1, int fd2, int t) {
    using C = SipCfg<K, Q, MODE>;
    const Tables1D& T = a.tab;
    const int md = G.mem(DIR);
    const int fs = md == 0 ? fd1 * fd2 : md == 1 ? fd2 : 1;   // face stride along DIR
    const int pr = t / ncell, c = t - pr * ncell;
    const int l2 = c % b2, lq = c / b2, l1 = lq % b1, l0 = lq / b1;
    if (l0 >= G.e[0] || l1 >= G.e[1] || l2 >= G.e[2]) return;
    const int fl = (l0 * fd1 + l1) * fd2 + l2, fu = fl + fs;
    constexpr int iB = MODE == MODE_VJP ? 2 : 0, iGB = MODE == MODE_VJP ? 3 : 2;
    int i = 0;
#pragma unroll
    for (int p = 0; p <= K; ++p)
#pragma unroll
        for (int r = 0; r <= K - p; ++r, ++i) {
            if (pr != i) continue;
            double gu = 0.0, Gu = 0.0, gl = 0.0, Gl = 0.0;
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                gu += rows[((0 * (K + 1) + p) * Q + q) * C::FST + fu] * T.A[q][r];
                Gu += rows[((1 * (K + 1) + p) * Q + q) * C::FST + fu] * T.A[q][r];
                gl += rows[((iB * (K + 1) + p) * Q + q) * C::FST + fl] * T.A[q][r];
                Gl += rows[((iGB * (K + 1) + p) * Q + q) * C::FST + fl] * T.A[q][r];
            }
            if (MODE != MODE_VJP) gl = -gl;
            const double gs = gu + gl, gd = gu - gl, Gs = Gu + Gl, Gd = Gu - Gl;
#pragma unroll
            for (int m = 0; m <= K - p - r; ++m) {
                const int n = sip_mode<DIR>(m, p, r);
                double v = ((m & 1) ? gd : gs) * T.e[1][m];
                if (m > 0) v += ((m & 1) ? Gs : Gd) * T.de[1][m];
                R[n * C::CST + c] += v;
            }
        }
}

template <int K, int Q, int MODE>
__device__ __forceinline__ void sip_volume(const EvalArgs& a, const Tables1D& V, const TileGeom& G, const double* coef,
                                           double* part, int ncell, int b1, int b2) {
    using C = SipCfg<K, Q, MODE>;
    constexpr int NP = C::NP, QV = C::QV;
    const double sc = a.g.scaling;
    const double tx = a.g.twoh[0], ty = a.g.twoh[1], tz = a.g.twoh[2];
    const bool tr = a.ph.has_transport != 0, sip = a.ph.has_sip != 0;
    const double vx = tr ? a.ph.vel[0] : 0.0, vy = tr ? a.ph.vel[1] : 0.0, vz = tr ? a.ph.vel[2] : 0.0;
    const double nu0 = sip ? a.ph.nu0 : 0.0, nu2 = sip ? a.ph.nu2 : 0.0;
    for (int t = threadIdx.x; t < QV * ncell; t += C::NT) {
        const int qz = t / ncell, c = t - qz * ncell;
        const int l2 = c % b2, lq = c / b2, l1 = lq % b1, l0 = lq / b1;
        if (l0 >= G.e[0] || l1 >= G.e[1] || l2 >= G.e[2]) continue;
        const double* cu = coef + G.slot(l0, l1, l2) * C::S;
        const double* cv = cu + C::SLOTS * C::S;
        double Az[K + 1], dAz[K + 1];
#pragma unroll
        for (int q = 0; q <= K; ++q) {
            Az[q] = V.A[qz][q] * sc;
            dAz[q] = V.dA[qz][q] * (sc * tz);
        }
        double P2[C::NPAIR], P2z[C::NPAIR];
#pragma unroll
        for (int i = 0; i < C::NPAIR; ++i) P2[i] = P2z[i] = 0.0;
        const double fz = V.w[qz] * a.g.detJ * sc;
#pragma unroll 1
        for (int qy = 0; qy < QV; ++qy) {
            double Ay[K + 1], dAy[K + 1];
#pragma unroll
            for (int b = 0; b <= K; ++b) {
                Ay[b] = V.A[qy][b];
                dAy[b] = V.dA[qy][b] * ty;
            }
            double uv[K + 1], uy[K + 1], uz[K + 1], wv[K + 1], wy[K + 1], wz[K + 1];
            sip_rows<K>(cu, Ay, dAy, Az, dAz, uv, uy, uz);
            if constexpr (C::NG > 1) sip_rows<K>(cv, Ay, dAy, Az, dAz, wv, wy, wz);
            double P[K + 1], Py[K + 1], Pz[K + 1];
#pragma unroll
            for (int b = 0; b <= K; ++b) P[b] = Py[b] = Pz[b] = 0.0;
            const double fy = fz * V.w[qy];
#pragma unroll
            for (int qx = 0; qx < QV; ++qx) {
                double u = 0.0, ux = 0.0, u_y = 0.0, u_z = 0.0, w = 0.0, wx = 0.0, w_y = 0.0, w_z = 0.0;
#pragma unroll
                for (int b = 0; b <= K; ++b) {
                    const double A = V.A[qx][b], dA = V.dA[qx][b];
                    u += uv[b] * A;
                    if (b > 0) ux += uv[b] * dA;
                    u_y += uy[b] * A;
                    u_z += uz[b] * A;
                    if constexpr (C::NG > 1) {
                        if (MODE == MODE_JVP) w += wv[b] * A;
                        if (b > 0) wx += wv[b] * dA;
                        w_y += wy[b] * A;
                        w_z += wz[b] * A;
                    }
                }
                ux *= tx;
                wx *= tx;
                const double f = -fy * V.w[qx], nu = fma(nu2 * u, u, nu0);
                double s = 0.0, gx, gy, gz;
                if constexpr (MODE == MODE_RES) {
                    gx = nu * ux + vx * u;
                    gy = nu * u_y + vy * u;
                    gz = nu * u_z + vz * u;
                } else if constexpr (MODE == MODE_JVP) {
                    const double dn = 2.0 * nu2 * u * w;
                    gx = nu * wx + dn * ux + vx * w;
                    gy = nu * w_y + dn * u_y + vy * w;
                    gz = nu * w_z + dn * u_z + vz * w;
                } else {
                    s = 2.0 * nu2 * u * (ux * wx + u_y * w_y + u_z * w_z) + vx * wx + vy * w_y + vz * w_z;
                    gx = nu * wx;
                    gy = nu * w_y;
                    gz = nu * w_z;
                    s *= f;
                }
                gx *= f * tx;
                gy *= f * ty;
                gz *= f * tz;
#pragma unroll
                for (int b = 0; b <= K; ++b) {
                    const double A = V.A[qx][b], dA = V.dA[qx][b];
                    if (MODE == MODE_VJP) P[b] += s * A;
                    if (b > 0) P[b] += gx * dA;
                    Py[b] += gy * A;
                    Pz[b] += gz * A;
                }
            }
            int pr = 0;
#pragma unroll
            for (int p = 0; p <= K; ++p)
#pragma unroll
                for (int b = 0; b <= K - p; ++b, ++pr) {
                    P2[pr] += P[p] * Ay[b] + Py[p] * V.dA[qy][b];
                    P2z[pr] += Pz[p] * Ay[b];
                }
        }
#pragma unroll
        for (int i = 0; i < C::NPAIR; ++i) {
            part[((2 * i) * QV + qz) * C::CST + c] = P2[i];
            part[((2 * i + 1) * QV + qz) * C::CST + c] = P2z[i];
        }
    }
}

template <int K, int Q, int MODE>
__global__ void __launch_bounds__(SipCfg<K, Q, MODE>::NT, SipCfg<K, Q, MODE>::MINB)
k_sip(const __grid_constant__ EvalArgs a, const __grid_constant__ Tables1D V, const __grid_constant__ ModalTile tl) {
    using C = SipCfg<K, Q, MODE>;
    constexpr int NP = C::NP, QV = C::QV;
    extern __shared__ double sm[];
    double* coef = sm + C::O_COEF;
    double* R = sm + C::O_R;
    double* tr = sm + C::O_WORK;
    double* rows = tr + C::FST * C::TR;
    const TileGeom G = tile_geom(a.g, tl, blockIdx.x);
    const int b1 = tl.b[1], b2 = tl.b[2], ncell = tl.ncell;
    tile_stage<NP, C::S, C::NT>(G, a.U, coef);
    if constexpr (C::NG > 1) tile_stage<NP, C::S, C::NT>(G, a.V, coef + C::SLOTS * C::S);
    tile_cp_wait();
    __syncthreads();

    sip_volume<K, Q, MODE>(a, V, G, coef, tr, ncell, b1, b2);
    __syncthreads();
    for (int t = threadIdx.x; t < C::NPAIR * ncell; t += C::NT) {
        const int pr = t / ncell, c = t - pr * ncell;
        int p = 0, b = pr;
        while (b > K - p) {
            b -= K + 1 - p;
            ++p;
        }
        double acc[K + 1];
#pragma unroll
        for (int q = 0; q <= K; ++q) acc[q] = 0.0;
#pragma unroll
        for (int qz = 0; qz < QV; ++qz) {
            const double s = tr[((2 * pr) * QV + qz) * C::CST + c], z = tr[((2 * pr + 1) * QV + qz) * C::CST + c];
#pragma unroll
            for (int q = 0; q <= K; ++q) acc[q] += s * V.A[qz][q] + z * V.dA[qz][q];
        }
        if (MODE == MODE_RES && pr == 0 && a.ph.has_source) acc[0] += a.ph.src * a.g.detJ * a.g.scaling * 2.82842712474619009760;
#pragma unroll
        for (int q = 0; q <= K; ++q)
            if (q <= K - p - b) R[mode3(p, b, q) * C::CST + c] = acc[q];
    }
    __syncthreads();

    auto dims = [&](int d, int& f0, int& f1, int& f2) {
        const int md = G.mem(d);
        f0 = G.e[0] + (md == 0);
        f1 = G.e[1] + (md == 1);
        f2 = G.e[2] + (md == 2);
    };
    auto direction = [&](auto dirc) {
        constexpr int DIR = decltype(dirc)::value;
        int f0, f1, f2, p0 = 0, p1 = 0, p2 = 0;
        dims(DIR, f0, f1, f2);
        if constexpr (DIR > 0) dims(DIR - 1, p0, p1, p2);
        // this direction's traces, and the previous direction's faces into the cells
        const int nf = f0 * f1 * f2, ntr = 2 * C::NG * nf, nadd = DIR > 0 ? C::NPAIR * ncell : 0;
        for (int t = threadIdx.x; t < ntr + nadd; t += C::NT) {
            if (t < nadd) {
                if constexpr (DIR > 0) sip_face_add<K, Q, MODE, DIR - 1>(a, G, rows, R, ncell, b1, b2, p1, p2, t);
            } else {
                sip_traces<K, Q, MODE, DIR>(a, G, coef, tr, f1, f2, nf, t - nadd);
            }
        }
        __syncthreads();
        sip_face_rows<K, Q, MODE, DIR>(a, G, tr, rows, f0, f1, f2);
        __syncthreads();
    };
    direction(std::integral_constant<int, 0>{});
    direction(std::integral_constant<int, 1>{});
    direction(std::integral_constant<int, 2>{});
    {
        int f0, f1, f2;
        dims(2, f0, f1, f2);
        for (int t = threadIdx.x; t < C::NPAIR * ncell; t += C::NT)
            sip_face_add<K, Q, MODE, 2>(a, G, rows, R, ncell, b1, b2, f1, f2, t);
    }
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int r = warp; r < G.e[0] * G.e[1]; r += C::NT >> 5) {
        const int i0 = r / G.e[1], i1 = r - i0 * G.e[1];
        const long long row = ((long long)(G.o[0] + i0) * G.n[1] + (G.o[1] + i1)) * G.n[2] + G.o[2];
        const double* src = R + (i0 * b1 + i1) * b2;
        for (int e = lane; e < G.e[2] * NP; e += 32) {
            const int c = e / NP, n = e - c * NP;
            if (row + c < a.cbeg || row + c >= a.cend) continue;
            const double v = src[n * C::CST + c];
            double* q = a.out + row * NP + e;
            if (MODE == MODE_RES) *q = (a.beta == 0.0) ? a.alpha * v : a.beta * *q + a.alpha * v;
            else *q = v;
        }
    }
}

}  // namespace bosss
