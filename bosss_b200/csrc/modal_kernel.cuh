// modal_kernel.cuh -- linear constant-coefficient scalar operators (upwind transport, SIP diffusion with
// constant viscosity, constant source) evaluated in the modes, without quadrature nodes.
//
// The basis is a product of 1D normalised Legendre polynomials, so with constant coefficients and
// an exact rule every integral of the form factors into 1D integrals, and orthonormality makes
// those of the directions without a derivative or a trace identities. What is left per
// direction d, on every pencil (p, r) of the other two exponents (modes m = 0 .. K-p-r):
//   volume   R[a] += -vel_d 2/h sum_m D[a][m] u[m]  - nu (2/h)^2 sum_m S[a][m] u[m]
//            D[a][m] = int L_a' L_m (m < a, a-m odd), S[a][m] = int L_a' L_m' (a+m even)
//   faces    value and normal-derivative traces of the pencil on both sides, the linear flux of
//            the pencil, and its product with the traces of the test functions:
//            two rank-2 updates per face instead of Q^2 nodes.
// The adjoint (J^T w) is the same stencil with D transposed and the upwind coefficient of the
// neighbour taken from the other side; the tangent (J v) is the stencil without source and
// boundary data.
//
// Per cell this is about 30 FMA per mode (k = 4: 1020 FMA for 35 modes) against 16 bytes of
// necessary traffic per mode: HBM and FP64 pipe are within a factor of two of each other, where
// the quadrature tiles spend 10-30x the arithmetic on node values.
//
// One thread per cell, both coefficient sets (input and result) in registers; a CTA's block of
// cells and its face halo are staged in shared memory by asynchronous 8-byte copies (vectors
// may start at any double), cells an odd number of doubles apart so that a warp reading the
// same mode of 32 cells covers all banks. Results go back through the same slots, so that
// global stores are runs of consecutive cells.
//
// Measured on B200 against the quadrature tiles: advection-diffusion 20x31x27 k = 3, residual + JVP +
// VJP 495 -> 48 us; 16 instances of 16^3..32^3, k = 1..4, residual + VJP 3.69 -> 0.21 ms; XDG
// Poisson 80^3 k = 2 (both species, cut items and interface) 1.71 -> 0.46 ms.
#pragma once
#include "modal.h"

namespace bosss {


static constexpr int MODAL_NT = 128;

// sqrt((2m+1)/2) = L_m(1) and L_m'(1) = L_m(1) m (m+1) / 2
__device__ constexpr double kE[5] = {0.70710678118654752440, 1.22474487139158904910, 1.58113883008418966600,
                                     1.87082869338697069279, 2.12132034355964257320};
// sqrt(2m+1)
__device__ constexpr double kS[5] = {1.0, 1.73205080756887729353, 2.23606797749978969641, 2.64575131106459059050, 3.0};

template <int D, int K>
struct ModalCfg {
    static constexpr int NP = np_of(D, K);
    static constexpr int S = NP | 1;                       // doubles per cell slot
    // halo box of the largest tile: 4 x 4 x 8 cells in 3D, 8 x 16 in 2D, and one zero slot
    static constexpr int SLOTS = (D == 3 ? 6 * 6 * 10 : 10 * 18) + 1;
    static constexpr size_t SMEM = sizeof(double) * S * SLOTS;
    static constexpr int MINB = SMEM > 75 * 1024 ? 2 : (SMEM > 45 * 1024 ? 3 : 4);
};

template <int D>
__device__ __forceinline__ constexpr int pencil_mode(int dir, int m, int p, int r) {
    return D == 2 ? (dir == 0 ? mode2(m, p) : mode2(p, m))
                  : (dir == 0 ? mode3(m, p, r) : (dir == 1 ? mode3(p, m, r) : mode3(p, r, m)));
}

// coefficients of one face of a cell: with own traces u (value), d (derivative), neighbour traces
// x, dx:  g = cO u + cN x - p (u - x) + sgn (hO d + hN dx) tested with v,  G = k (u - x) with dv/dn;
// the adjoint's upwind term is a jump too: cN = -cO there, folded into p. Jumps are formed before
// they are multiplied with the (large) penalty
struct FaceCoef {
    double cO, cN, p, hO, hN, k;
};

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}

// One tile: cells [o, o + b) in memory order (slow, middle, fast). MODE as the quadrature
// kernels; MASK reads the species masks.
template <int D, int K, bool SIP, int MODE, bool MASK>
__device__ __forceinline__ void modal_tile(const EvalArgs& a, const ModalTile& tl, int tile, const double* __restrict__ in,
                                           double* __restrict__ out, double alpha, double beta, double* sm) {
    using C = ModalCfg<D, K>;
    constexpr int NP = C::NP, S = C::S;
    const GridConst& g = a.g;
    const int tid = threadIdx.x;
    // memory directions: generator order x slow .. z fast; GlobalID order the other way round
    const bool rev = (D == 3) && g.stride[0] == 1 && g.stride[2] != 1;
    const int n0 = rev ? g.n[2] : g.n[0], n1 = (D == 3) ? g.n[1] : 1, n2 = (D == 3) ? (rev ? g.n[0] : g.n[2]) : g.n[1];
    const int per0 = rev ? g.periodic[2] : g.periodic[0], per1 = (D == 3) ? g.periodic[1] : 0;
    const int per2 = (D == 3) ? (rev ? g.periodic[0] : g.periodic[2]) : g.periodic[1];
    const int b0 = tl.b[0], b1 = tl.b[1], b2 = tl.b[2];
    const int t2 = tile % tl.t[2], tq = tile / tl.t[2];
    const int t1 = tq % tl.t[1], t0 = tq / tl.t[1];
    const int o0 = tl.s0 + t0 * b0, o1 = t1 * b1, o2 = t2 * b2;
    const int e0 = min(b0, n0 - o0), e1 = min(b1, n1 - o1), e2 = min(b2, n2 - o2);
    // slots: halo box, fast direction innermost
    const int w2 = b2 + 2, w1 = (D == 3) ? b1 + 2 : 1;
    const int q1 = w2, q0 = w1 * w2;
    auto slot = [&](int i0, int i1, int i2) {   // tile coordinates, -1 .. b
        return ((i0 + 1) * q0 + ((D == 3) ? (i1 + 1) * q1 : 0) + (i2 + 1)) * S;
    };
    double* zero = sm + (C::SLOTS - 1) * S;
    if (tid < NP) zero[tid] = 0.0;

    // ---- stage the tile and its face halo: one warp per run of cells along the fast direction
    {
        const int warp = tid >> 5, lane = tid & 31, nw = MODAL_NT >> 5;
        const int rA = e0 * e1, rB = 2 * e1, rC = (D == 3) ? 2 * e0 : 0;
        for (int r = warp; r < rA + rB + rC; r += nw) {
            int i0, i1, f0 = 0, nf = e2;
            if (r < rA) {
                i0 = r / e1;
                i1 = r - i0 * e1;
                f0 = -1;
                nf = e2 + 2;
            } else if (r < rA + rB) {
                const int q = r - rA;
                i0 = (q & 1) ? e0 : -1;
                i1 = q >> 1;
            } else {
                const int q = r - rA - rB;
                i0 = q >> 1;
                i1 = (q & 1) ? e1 : -1;
            }
            int m0 = o0 + i0, m1 = o1 + i1;
            if (m0 < 0 || m0 >= n0) {
                if (!per0) continue;
                m0 = m0 < 0 ? m0 + n0 : m0 - n0;
            }
            if (D == 3 && (m1 < 0 || m1 >= n1)) {
                if (!per1) continue;
                m1 = m1 < 0 ? m1 + n1 : m1 - n1;
            }
            const long long row = ((long long)m0 * n1 + m1) * n2;
            double* dst = sm + slot(i0, i1, 0);
            for (int e = lane; e < nf * NP; e += 32) {
                const int c = e / NP, n = e - c * NP;
                const int i2 = f0 + c;
                int m2 = o2 + i2;
                if (m2 < 0 || m2 >= n2) {
                    if (!per2) continue;
                    m2 = m2 < 0 ? m2 + n2 : m2 - n2;
                }
                cp_async8(dst + i2 * S + n, in + (row + m2) * NP + n);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }

    // ---- the thread's cell
    const int l0 = tid / (b1 * b2), lr = tid - l0 * b1 * b2;
    const int l1 = lr / b2, l2 = lr - l1 * b2;
    const int c0 = o0 + l0, c1 = o1 + l1, c2 = o2 + l2;
    const long long j = ((long long)c0 * n1 + c1) * n2 + c2;
    const bool active = l0 < e0 && l1 < e1 && l2 < e2 && j >= a.cbeg && j < a.cend;
    int ijk[3] = {rev ? c2 : c0, (D == 3) ? c1 : c2, (D == 3) ? (rev ? c0 : c2) : 0};
    double volm = 1.0;
    unsigned fmask = 0x3fu;
    if constexpr (MASK) {
        if (active) {
            if (a.vol_flag) volm = (a.vol_flag[j] == 1) ? 1.0 : 0.0;
            if (a.face_flag) {
                fmask = 0;
#pragma unroll
                for (int f = 0; f < 2 * D; ++f) fmask |= (a.face_flag[j * 2 * D + f] == 1 ? 1u : 0u) << f;
            }
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();

    double R[NP];
#pragma unroll
    for (int n = 0; n < NP; ++n) R[n] = 0.0;
    if (active) {
        const double* own = sm + slot(l0, l1, l2);
        // a cell without any standard term takes no part (its coefficients may be anything)
        if (MASK && volm == 0.0 && fmask == 0) own = zero;
        double u[NP];
#pragma unroll
        for (int n = 0; n < NP; ++n) u[n] = own[n];
        const bool tr = a.ph.has_transport != 0, sip = SIP && a.ph.has_sip != 0;
        const double nu = sip ? a.ph.nu0 : 0.0;
        double pfo = 0.0;
        if (SIP) pfo = penalty_size(a.cell_pf, g, ijk);

        auto direction = [&](auto dirc) {
            constexpr int DIR = decltype(dirc)::value;
            const double th = g.twoh[DIR], vel = tr ? a.ph.vel[DIR] : 0.0;
            const int sl = (DIR == 0 ? (rev ? 1 : q0) : DIR == 1 ? (D == 3 ? q1 : 1) : (rev ? q0 : 1)) * S;
            FaceCoef fu, fl;
            const double *nbu = own + sl, *nbl = own - sl;
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                FaceCoef& f = s ? fu : fl;
                const double*& nb = s ? nbu : nbl;
                f = FaceCoef{0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
                int i = ijk[DIR] + (s ? 1 : -1);
                bool inner = true;
                if (i < 0 || i >= g.n[DIR]) {
                    inner = g.periodic[DIR] != 0;
                    i = i < 0 ? i + g.n[DIR] : i - g.n[DIR];
                }
                const bool on = !MASK || ((fmask >> (2 * DIR + s)) & 1u);
                if (!inner || !on) nb = zero;
                if (!on) continue;
                if (inner) {
                    // upwind: the lower cell's value where vel > 0, else the upper cell's
                    const double ap = vel > 0.0 ? vel : 0.0, am = vel > 0.0 ? 0.0 : vel;
                    double p = 0.0;
                    if constexpr (SIP) {
                        int ijk2[3] = {ijk[0], ijk[1], ijk[2]};
                        ijk2[DIR] = i;
                        p = sip ? a.ph.pen * fmax(pfo, penalty_size(a.cell_pf, g, ijk2)) * nu : 0.0;
                    }
                    if (MODE == MODE_VJP) {
                        f.p = p - (s ? ap : -am);   // both sides of the upwind flux see the jump of w
                    } else {
                        f.p = p;
                        f.cO = s ? ap : -am;
                        f.cN = s ? am : -ap;
                    }
                    f.hO = f.hN = 0.5 * nu * th;
                    f.k = 0.5 * nu;
                } else {
                    const double an = s ? vel : -vel;
                    if (tr && (D == 2 || an >= 0.0)) f.cO = an;
                    if (sip && a.ph.dirichlet) {
                        const double p = 2.0 * a.ph.pen * pfo * nu;
                        f.p = p;
                        f.hO = nu * th;
                        f.k = nu;
                    }
                }
                f.cO *= th;
                f.cN *= th;
                f.p *= th;
                f.hO *= th;
                f.hN *= th;
                f.k *= th * th;
            }
            const double vT = -vel * th * volm, vS = -nu * th * th * volm;
#pragma unroll
            for (int p = 0; p <= K; ++p)
#pragma unroll
                for (int r = 0; r <= (D == 3 ? K - p : 0); ++r) {
                    constexpr int L1 = K + 1;
                    const int L = K - p - r + 1;
                    // traces: e = even, o = odd modes; L_m(-1) = (-1)^m L_m(1), L_m'(-1) = (-1)^(m+1) L_m'(1)
                    double ue = 0.0, uo = 0.0, de = 0.0, dd = 0.0;
                    double xe = 0.0, xo = 0.0, xde = 0.0, xdo = 0.0, y = 0.0, dy = 0.0;
#pragma unroll
                    for (int m = 0; m < L1; ++m)
                        if (m < L) {
                            const int n = pencil_mode<D>(DIR, m, p, r);
                            const double E = kE[m], F = kE[m] * (0.5 * m * (m + 1));
                            const double v = u[n], vu = nbu[n], vl = nbl[n];
                            if (m & 1) {
                                uo += v * E;
                                xo += vu * E;
                            } else {
                                ue += v * E;
                                xe += vu * E;
                            }
                            y += vl * E;
                            if (SIP && m > 0) {
                                if (m & 1) {
                                    dd += v * F;
                                    xdo += vu * F;
                                } else {
                                    de += v * F;
                                    xde += vu * F;
                                }
                                dy += vl * F;
                            }
                        }
                    const double uP = ue + uo, uM = ue - uo, x = xe - xo;
                    const double Ju = uP - x, Jl = uM - y;
                    double gu = fu.cO * uP - fu.p * Ju, gl = fl.cO * uM - fl.p * Jl, Gu = 0.0, Gl = 0.0;
                    if (MODE != MODE_VJP) {
                        gu += fu.cN * x;
                        gl += fl.cN * y;
                    }
                    if constexpr (SIP) {
                        const double dP = de + dd, dM = dd - de, dx = xdo - xde;
                        gu += fu.hO * dP + fu.hN * dx;
                        gl -= fl.hO * dM + fl.hN * dy;
                        Gu = fu.k * Ju;
                        Gl = -fl.k * Jl;
                    }
                    const double gs = gu + gl, gd = gu - gl, Gs = Gu + Gl, Gd = Gu - Gl;
#pragma unroll
                    for (int m = 0; m < L1; ++m)
                        if (m < L) {
                            const int n = pencil_mode<D>(DIR, m, p, r);
                            const double E = kE[m], F = kE[m] * (0.5 * m * (m + 1));
                            double t = R[n] + ((m & 1) ? gd : gs) * E;
                            if (SIP && m > 0) t += ((m & 1) ? Gs : Gd) * F;
                            // volume
                            double tD = 0.0, tS = 0.0;
#pragma unroll
                            for (int q = 0; q < L1; ++q)
                                if (q < L) {
                                    const int nq = pencil_mode<D>(DIR, q, p, r);
                                    const bool lower = (MODE == MODE_VJP) ? q > m : q < m;
                                    if (lower && ((m - q) & 1)) tD += u[nq] * (kS[m] * kS[q]);
                                    if (SIP && q > 0 && m > 0 && !((m - q) & 1)) {
                                        const int mn = q < m ? q : m;
                                        tS += u[nq] * (kS[m] * kS[q] * (0.5 * mn * (mn + 1)));
                                    }
                                }
                            t += vT * tD;
                            if (SIP && m > 0) t += vS * tS;
                            R[n] = t;
                        }
                }
            // Dirichlet data of boundary faces (residual only): the trace of g_D on the modes of the
            // face; g_D is a sum of one-direction polynomials, so only p = 0 or r = 0 are non-zero
            if constexpr (SIP && MODE == MODE_RES) {
                bool any = a.ph.g0 != 0.0;
#pragma unroll
                for (int d = 0; d < D; ++d) any = any || a.ph.g1[d] != 0.0 || a.ph.g2[d] != 0.0;
                if (any && sip && a.ph.dirichlet && !g.periodic[DIR]) {
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const FaceCoef& f = s ? fu : fl;
                        if (ijk[DIR] != (s ? g.n[DIR] - 1 : 0)) continue;
                        if (MASK && !((fmask >> (2 * DIR + s)) & 1u)) continue;
                        constexpr int d1 = (DIR == 0) ? 1 : 0, d2 = (DIR == 2) ? 1 : 2;
                        const double xn = g.lo[DIR] + (ijk[DIR] + g.goff[DIR] + (s ? 1.0 : 0.0)) * g.h[DIR];
                        const double cst = a.ph.g0 + a.ph.g1[DIR] * xn + a.ph.g2[DIR] * xn * xn;
                        double M1[K + 1], M2[K + 1];
#pragma unroll
                        for (int q = 0; q <= K; ++q) M1[q] = M2[q] = 0.0;
                        for (int q = 0; q < QMAX; ++q) {
                            const double w = a.tab.w[q];
                            if (w == 0.0) break;   // nodes of the rule (the rest of the table is zero)
                            const double x1 = g.lo[d1] + (ijk[d1] + g.goff[d1] + 0.5 + 0.5 * a.tab.xq[q]) * g.h[d1];
                            const double f1 = (a.ph.g1[d1] + a.ph.g2[d1] * x1) * x1 * w;
                            double f2 = 0.0;
                            if (D == 3) {
                                const double x2 = g.lo[d2] + (ijk[d2] + g.goff[d2] + 0.5 + 0.5 * a.tab.xq[q]) * g.h[d2];
                                f2 = (a.ph.g1[d2] + a.ph.g2[d2] * x2) * x2 * w;
                            }
#pragma unroll
                            for (int p = 0; p <= K; ++p) {
                                M1[p] += f1 * a.tab.A[q][p];
                                if (D == 3) M2[p] += f2 * a.tab.A[q][p];
                            }
                        }
                        const double rt2 = 1.41421356237309504880, isc = 1.0 / g.scaling;
#pragma unroll
                        for (int p = 0; p <= K; ++p)
#pragma unroll
                            for (int r = 0; r <= (D == 3 ? K - p : 0); ++r) {
                                if (p > 0 && r > 0) continue;
                                double gD = M1[p] * ((D == 3) ? rt2 : 1.0);
                                if (r > 0) gD = 0.0;
                                if (D == 3 && p == 0) gD += M2[r] * rt2;
                                if (p == 0 && r == 0) gD += cst * ((D == 3) ? 2.0 : rt2);
                                gD *= isc;
                                const double gg = f.p * gD, GG = f.k * gD;
#pragma unroll
                                for (int m = 0; m <= K - p - r; ++m) {
                                    const int n = pencil_mode<D>(DIR, m, p, r);
                                    const double E = kE[m], F = kE[m] * (0.5 * m * (m + 1));
                                    if (s) R[n] += gg * E - GG * F;
                                    else R[n] += ((m & 1) ? -gg : gg) * E + ((m & 1) ? GG : -GG) * F;
                                }
                            }
                    }
                }
            }
        };
        direction(std::integral_constant<int, 0>{});
        direction(std::integral_constant<int, 1>{});
        if constexpr (D == 3) direction(std::integral_constant<int, 2>{});
        if (SIP && MODE == MODE_RES && a.ph.has_source)
            R[0] += volm * a.ph.src * g.detJ * g.scaling * ((D == 3) ? 2.82842712474619009760 : 2.0);
    }
    __syncthreads();
    // ---- results through the cell's own slot, stored in runs of cells
    if (active) {
        double* own = sm + slot(l0, l1, l2);
#pragma unroll
        for (int n = 0; n < NP; ++n) own[n] = R[n];
    }
    __syncthreads();
    {
        const int warp = tid >> 5, lane = tid & 31, nw = MODAL_NT >> 5;
        for (int r = warp; r < e0 * e1; r += nw) {
            const int i0 = r / e1, i1 = r - i0 * e1;
            const long long row = ((long long)(o0 + i0) * n1 + (o1 + i1)) * n2 + o2;
            const double* src = sm + slot(i0, i1, 0);
            for (int e = lane; e < e2 * NP; e += 32) {
                const int c = e / NP;
                if (row + c < a.cbeg || row + c >= a.cend) continue;
                const double v = src[e + c * (S - NP)];
                double* q = out + row * NP + e;
                if (MODE == MODE_RES) *q = (beta == 0.0) ? alpha * v : beta * *q + alpha * v;
                else *q = v;
            }
        }
    }
}

template <class Kern>
inline cudaError_t modal_attr(Kern k, size_t smem, unsigned long long& done) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (done & (1ull << (dev & 63))) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e == cudaSuccess) done |= 1ull << (dev & 63);
    return e;
}

}  // namespace bosss
