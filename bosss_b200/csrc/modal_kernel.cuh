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
// T threads per cell share the pencils of a direction (T by degree: a thread's chain of dependent
// sums is what a small grid waits for, and short chains leave registers for more warps); the
// three directions add to the cell's result in shared memory, each mode once per direction. A
// CTA's block of cells and its face halo are staged by asynchronous 8-byte copies (vectors may
// start at any double), cells an odd number of doubles apart so that a warp reading the same mode
// of 32 cells covers all banks; results leave in runs of consecutive cells.
//
// Measured on B200 against the quadrature tiles: advection-diffusion 20x31x27 k = 3, residual + JVP +
// VJP 496 -> 31 us; 16 instances of 16^3..32^3, k = 1..4, residual + VJP 3.71 -> 0.146 ms; XDG
// Poisson 80^3 k = 2 (both species, cut items and interface) 1.72 -> 0.29 ms, cut items and
// interface (also rewritten) 0.12 ms of it.
#pragma once
#include "tile_stage.cuh"

namespace bosss {

template <int D, int K>
struct ModalCfg {
    static constexpr int NP = np_of(D, K);
    static constexpr int S = NP | 1;                       // doubles per cell slot
    static constexpr int PENCILS = D == 3 ? (K + 1) * (K + 2) / 2 : K + 1;
    // threads per cell: the pencils of a direction are dealt to T threads
    static constexpr int T = D == 2 ? 1 : (K == 4 ? 4 : K == 3 ? 2 : 1);
    static constexpr int MINB = D == 2 ? 4 : (K >= 3 ? 2 : K == 2 ? 4 : 8);
    // cells of the largest tile and its halo box: 4 x 4 x 8 or 4 x 4 x 4 cells in 3D, 8 x 16 in 2D
    static constexpr int CELLS = D == 3 && K == 4 ? 64 : 128;
    static constexpr int BOX = D == 2 ? 10 * 18 : CELLS == 64 ? 6 * 6 * 6 : 6 * 6 * 10;
    static constexpr int NT = CELLS * T;
    // runs a warp copies at a time: few warps have several each (k = 2, 48^3: 29 -> 23 us), sixteen warps
    // one or two (k = 4: four at a time 59 -> 71 us)
    static constexpr int GRP = T == 1 ? 4 : T == 2 ? 2 : 1;
    static constexpr int SLOTS = BOX + 1;   // and one zero slot
    // runs of cells to copy: per row of the tile its cells (with the halo cells that follow on), and
    // halo cells across a periodic wrap; the rows of the slow and middle halos
    static constexpr int ROWS = D == 3 ? 128 : 16, RUNS = 3 * ROWS;
    static constexpr size_t SMEM = sizeof(double) * (S * (SLOTS + CELLS) + 3 * 2 * 6);
};
struct ModalRun {
    long long src;   // first double
    int dst, n;      // slot offset, doubles
};

// thread (0 .. T-1) that evaluates pencil i = (p, r), r fastest: longest pencils first, each to the
// least loaded thread
template <int D, int K>
struct PencilOwner {
    int o[ModalCfg<D, K>::PENCILS] = {};
    constexpr PencilOwner() {
        int load[ModalCfg<D, K>::T] = {};
        for (int L = K + 1; L >= 1; --L) {
            int i = 0;
            for (int p = 0; p <= K; ++p)
                for (int r = 0; r <= (D == 3 ? K - p : 0); ++r, ++i) {
                    if (K - p - r + 1 != L) continue;
                    int best = 0;
                    for (int t = 1; t < ModalCfg<D, K>::T; ++t)
                        if (load[t] < load[best]) best = t;
                    o[i] = best;
                    load[best] += L + 2;
                }
        }
    }
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

// coefficients of face (dir, s) of cell ijk; nb: there is a neighbour whose coefficients enter
template <int D, bool SIP, int MODE>
__device__ __forceinline__ FaceCoef modal_face(const EvalArgs& a, const int* ijk, int dir, int s, bool on, bool& nb) {
    const GridConst& g = a.g;
    FaceCoef f{0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const bool tr = a.ph.has_transport != 0, sip = SIP && a.ph.has_sip != 0;
    const double th = g.twoh[dir], vel = tr ? a.ph.vel[dir] : 0.0, nu = sip ? a.ph.nu0 : 0.0;
    int i = ijk[dir] + (s ? 1 : -1);
    bool inner = true;
    if (i < 0 || i >= g.n[dir]) {
        inner = g.periodic[dir] != 0;
        i = i < 0 ? i + g.n[dir] : i - g.n[dir];
    }
    nb = inner && on;
    if (!on) return f;
    if (inner) {
        // upwind: the lower cell's value where vel > 0, else the upper cell's
        const double ap = vel > 0.0 ? vel : 0.0, am = vel > 0.0 ? 0.0 : vel;
        double p = 0.0;
        if constexpr (SIP) {
            int ijk2[3] = {ijk[0], ijk[1], ijk[2]};
            ijk2[dir] = i;
            p = sip ? a.ph.pen * fmax(tile_size<D>(a, ijk), tile_size<D>(a, ijk2)) * nu : 0.0;
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
            f.p = 2.0 * a.ph.pen * tile_size<D>(a, ijk) * nu;
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
    return f;
}

// the same between two cells that touch no boundary of the global grid
template <int D, bool SIP, int MODE>
__device__ __forceinline__ void modal_plain_face(const EvalArgs& a, int dir, int s, double* o) {
    const bool tr = a.ph.has_transport != 0, sip = SIP && a.ph.has_sip != 0;
    const double th = a.g.twoh[dir], vel = tr ? a.ph.vel[dir] : 0.0, nu = sip ? a.ph.nu0 : 0.0;
    double cj = 0.0;
#pragma unroll
    for (int d = 0; d < D; ++d) cj += 2 * (0.5 * a.g.twoh[d]);
    const double ap = vel > 0.0 ? vel : 0.0, am = vel > 0.0 ? 0.0 : vel;
    const double p = sip ? a.ph.pen * (0.5 * cj) * nu : 0.0;
    o[0] = MODE == MODE_VJP ? 0.0 : (s ? ap : -am) * th;
    o[1] = MODE == MODE_VJP ? 0.0 : (s ? am : -ap) * th;
    o[2] = (MODE == MODE_VJP ? p - (s ? ap : -am) : p) * th;
    o[3] = o[4] = 0.5 * nu * th * th;
    o[5] = 0.5 * nu * (th * th);
}

// the pencils of direction DIR that belong to thread TH of a cell: R (+)= their contributions
template <int D, int K, bool SIP, int MODE, int DIR, int TH>
__device__ __forceinline__ void modal_pencils(const Tables1D& T, const double* own, const double* nbu, const double* nbl,
                                              const FaceCoef& fu, const FaceCoef& fl, double vT, double vS, double* R) {
    constexpr PencilOwner<D, K> owner{};
    constexpr int L1 = K + 1;
    int i = 0;
#pragma unroll
    for (int p = 0; p <= K; ++p)
#pragma unroll
        for (int r = 0; r <= (D == 3 ? K - p : 0); ++r, ++i) {
            if (owner.o[i] != TH) continue;
            const int L = K - p - r + 1;
            // own modes times L_m(1): w; with c_m = m (m+1) / 2 = L_m'(1) / L_m(1) everything on
            // the pencil is sums of w and c w. L_m(-1) = (-1)^m L_m(1), L_m'(-1) = (-1)^(m+1) L_m'(1)
            double w[L1], ue = 0.0, uo = 0.0, de = 0.0, dd = 0.0;
            double x = 0.0, dx = 0.0, y = 0.0, dy = 0.0;
#pragma unroll
            for (int m = 0; m < L1; ++m)
                if (m < L) {
                    const int n = pencil_mode<D>(DIR, m, p, r);
                    const double E = T.e[1][m], F = T.de[1][m], c = 0.5 * m * (m + 1);
                    const double vu = nbu[n], vl = nbl[n];
                    w[m] = own[n] * E;
                    if (m & 1) uo += w[m];
                    else ue += w[m];
                    x += vu * ((m & 1) ? -E : E);
                    y += vl * E;
                    if (SIP && m > 0) {
                        if (m & 1) dd += c * w[m];
                        else de += c * w[m];
                        dx += vu * ((m & 1) ? F : -F);
                        dy += vl * F;
                    }
                }
            const double uP = ue + uo, uM = ue - uo;
            const double Ju = uP - x, Jl = uM - y;
            double gu = fu.cO * uP - fu.p * Ju, gl = fl.cO * uM - fl.p * Jl, Gs = 0.0, Gd = 0.0;
            if (MODE != MODE_VJP) {
                gu += fu.cN * x;
                gl += fl.cN * y;
            }
            if constexpr (SIP) {
                gu += fu.hO * (de + dd) + fu.hN * dx;
                gl -= fl.hO * (dd - de) + fl.hN * dy;
                const double Gu = fu.k * Ju, Gl = fl.k * Jl;
                Gs = Gu - Gl;
                Gd = Gu + Gl;
            }
            const double gs = gu + gl, gd = gu - gl;
            // volume: int L_a' L_m = 2 L_a(1) L_m(1) (m < a, a - m odd), int L_a' L_m' = 2 c_min L_a(1) L_m(1)
            // (a - m even): sums over the modes below / above by parity. above[m]: mode m and those above it of
            // its parity, added directly (what is left of the total after the modes below would carry
            // their rounding: a large mean beside small variations)
            double pre[2] = {0.0, 0.0}, pc[2] = {0.0, 0.0}, above[L1 + 2];
#pragma unroll
            for (int m = L1 + 1; m >= 0; --m) above[m] = 0.0;
#pragma unroll
            for (int m = L1 - 1; m >= 0; --m)
                if (m < L) above[m] = w[m] + above[m + 2];
#pragma unroll
            for (int m = 0; m < L1; ++m)
                if (m < L) {
                    const int n = pencil_mode<D>(DIR, m, p, r);
                    const double c = 0.5 * m * (m + 1);
                    const int e = m & 1;
                    double h = e ? gd : gs;
                    if (MODE == MODE_VJP) h += vT * above[m + 1];
                    else h += vT * pre[1 - e];
                    if (SIP && m > 0) {
                        pc[e] += c * w[m];
                        h += vS * pc[e] + c * ((e ? Gs : Gd) + vS * above[m + 2]);
                    }
                    pre[e] += w[m];
                    if (DIR == 0) R[n] = h * T.e[1][m];
                    else R[n] += h * T.e[1][m];
                }
        }
}

// Dirichlet data of a boundary face (residual only): the trace of g_D on the modes of the face; g_D
// is a sum of one-direction polynomials, so only p = 0 or r = 0 are non-zero
template <int D, int K, int DIR>
__device__ __forceinline__ void modal_boundary_data(const EvalArgs& a, const Tables1D& T, const int* ijk, int s,
                                                    const FaceCoef& f, double* R) {
    const GridConst& g = a.g;
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
                const double E = T.e[1][m], F = T.de[1][m];
                if (s) R[n] += gg * E - GG * F;
                else R[n] += ((m & 1) ? -gg : gg) * E + ((m & 1) ? GG : -GG) * F;
            }
        }
}

// One tile: cells [o, o + b) in memory order (slow, middle, fast). MODE as the quadrature
// kernels; MASK reads the species masks. T: L_m(1) and L_m'(1) in T.e[1], T.de[1], in the
// kernel-parameter bank so that they are operands of the FMAs (as literals they cost two moves
// each: a third of all instructions of the first version).
template <int D, int K, bool SIP, int MODE, bool MASK>
__device__ __forceinline__ void modal_tile(const EvalArgs& a, const Tables1D& T, const ModalTile& tl, int tile,
                                           const double* __restrict__ in, double* __restrict__ out, double alpha, double beta,
                                           double* sm) {
    using C = ModalCfg<D, K>;
    constexpr int NP = C::NP, S = C::S, NT = C::NT;
    const GridConst& g = a.g;
    const int tid = threadIdx.x;
    // memory directions: generator order x slow .. z fast; GlobalID order the other way round
    const TileGeom G = tile_geom<D>(g, tl, tile);
    const bool rev = G.rev;
    const int n0 = G.n[0], n1 = G.n[1], n2 = G.n[2];
    const int per0 = G.per[0], per1 = G.per[1], per2 = G.per[2];
    const int b1 = tl.b[1], b2 = tl.b[2];
    const int o0 = G.o[0], o1 = G.o[1], o2 = G.o[2], e0 = G.e[0], e1 = G.e[1], e2 = G.e[2];
    // slots: halo box, fast direction innermost
    const int w2 = b2 + 2, w1 = (D == 3) ? b1 + 2 : 1;
    const int q1 = w2, q0 = w1 * w2;
    auto slot = [&](int i0, int i1, int i2) {   // tile coordinates, -1 .. b
        return ((i0 + 1) * q0 + ((D == 3) ? (i1 + 1) * q1 : 0) + (i2 + 1)) * S;
    };
    double* zero = sm + (C::SLOTS - 1) * S;
    double* res = sm + C::SLOTS * S;
    double* fct = res + C::CELLS * S;   // [direction][side]: coefficients of a face between plain cells
    if (tid < NP) zero[tid] = 0.0;

    // ---- stage the tile and its face halo: the runs of consecutive cells are found by one thread each
    // (index arithmetic per row and warp took most of the time of the first version), then copied by
    // the warps in turn
    const int warp = tid >> 5, lane = tid & 31;
    constexpr int nw = NT >> 5;
    __shared__ ModalRun runs[C::RUNS];
    const int rA = e0 * e1, rB = 2 * e1, rC = (D == 3) ? 2 * e0 : 0, nrows = rA + rB + rC;
    const int nlo = (o2 == 0 && per2) ? rA : 0, nhi = (o2 + e2 == n2 && per2) ? rA : 0;   // across the wrap
    for (int r = tid; r < nrows; r += NT) {
        int i0, i1;
        if (r < rA) {
            i0 = r / e1;
            i1 = r - i0 * e1;
        } else if (r < rA + rB) {
            i0 = ((r - rA) & 1) ? e0 : -1;
            i1 = (r - rA) >> 1;
        } else {
            i0 = (r - rA - rB) >> 1;
            i1 = ((r - rA - rB) & 1) ? e1 : -1;
        }
        int m0 = o0 + i0, m1 = o1 + i1;
        bool there = true;
        if (m0 < 0 || m0 >= n0) {
            there = per0 != 0;
            m0 = m0 < 0 ? m0 + n0 : m0 - n0;
        }
        if (D == 3 && (m1 < 0 || m1 >= n1)) {
            there = there && per1 != 0;
            m1 = m1 < 0 ? m1 + n1 : m1 - n1;
        }
        const long long row = ((long long)m0 * n1 + m1) * n2;
        ModalRun main{(row + o2) * NP, slot(i0, i1, 0), there ? e2 * NP : 0};
        if (r < rA) {
            if (o2 > 0) {
                main.src -= NP;
                main.dst -= S;
                main.n += NP;
            } else if (nlo) {
                runs[nrows + r] = ModalRun{(row + n2 - 1) * NP, slot(i0, i1, -1), NP};
            }
            if (o2 + e2 < n2) main.n += NP;
            else if (nhi) runs[nrows + nlo + r] = ModalRun{row * NP, slot(i0, i1, e2), NP};
        }
        runs[r] = main;
    }
    __syncthreads();
    const int total = nrows + nlo + nhi;
    for (int r = warp; r < total; r += C::GRP * nw) {   // several runs at a time: their addresses are independent
        const double* src[C::GRP];
        int dst[C::GRP], n[C::GRP], nmax = 0;
#pragma unroll
        for (int k = 0; k < C::GRP; ++k) {
            const int rr = min(r + k * nw, total - 1);
            const ModalRun q = runs[rr];
            src[k] = in + q.src;
            dst[k] = q.dst;
            n[k] = r + k * nw < total ? q.n : 0;
            nmax = max(nmax, n[k]);
        }
        for (int e = lane; e < nmax; e += 32) {
            const int o = e + (S - NP) * (e / NP);
#pragma unroll
            for (int k = 0; k < C::GRP; ++k)
                if (e < n[k]) tile_cp8(sm + dst[k] + o, src[k] + e);
        }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");

    // ---- the thread's cell and share of the pencils
    const int cell = tid % C::CELLS, th = tid / C::CELLS;   // th is warp-uniform
    const int l0 = cell / (b1 * b2), lr = cell - l0 * b1 * b2;
    const int l1 = lr / b2, l2 = lr - l1 * b2;
    const int c0 = o0 + l0, c1 = o1 + l1, c2 = o2 + l2;
    const long long j = ((long long)c0 * n1 + c1) * n2 + c2;
    const bool active = l0 < e0 && l1 < e1 && l2 < e2 && j >= a.cbeg && j < a.cend;
    const int ijk[3] = {rev ? c2 : c0, (D == 3) ? c1 : c2, (D == 3) ? (rev ? c0 : c2) : 0};
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
    const double* own = sm + (active ? slot(l0, l1, l2) : 0);
    // a cell without any standard term takes no part (its coefficients may be anything)
    if (MASK && volm == 0.0 && fmask == 0) own = zero;
    const bool transport = a.ph.has_transport != 0, diffusion = SIP && a.ph.has_sip != 0;
    if (MODE != MODE_VJP && !transport && !diffusion) own = zero;   // a source alone reads no coefficients
    double* R = res + cell * S;
    // a face between two cells away from the boundaries of the global grid has the same
    // coefficients everywhere (unless the caller gives length scales): computed once per CTA
    if (tid < 2 * D) modal_plain_face<D, SIP, MODE>(a, tid >> 1, tid & 1, fct + tid * 6);
    unsigned pl = 0;   // bits 2d, 2d + 1: own cell plain along d, and so is its lower / upper neighbour
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const int gi = ijk[d] + g.goff[d];
        const bool p = g.gper[d] || (gi >= 1 && gi <= g.gn[d] - 2);
        pl |= (p && (g.gper[d] || gi >= 2) ? 1u : 0u) << (2 * d) | (p && (g.gper[d] || gi <= g.gn[d] - 3) ? 2u : 0u) << (2 * d) |
              (p ? 1u : 0u) << (8 + d);
    }
    const bool uniform = !SIP || !a.cell_pf;
    const double nu0 = (SIP && a.ph.has_sip) ? a.ph.nu0 : 0.0;
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();

    auto direction = [&](auto dirc) {
        constexpr int DIR = decltype(dirc)::value;
        if (active) {
            const double thd = g.twoh[DIR], vel = a.ph.has_transport ? a.ph.vel[DIR] : 0.0;
            const int sl = (DIR == 0 ? (rev ? 1 : q0) : DIR == 1 ? (D == 3 ? q1 : 1) : (rev ? q0 : 1)) * S;
            bool h[2];
            FaceCoef fc[2];
            constexpr unsigned others = (D == 3 ? 7u : 3u) & ~(1u << DIR);
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const bool on = !MASK || ((fmask >> (2 * DIR + s)) & 1u);
                const int i = ijk[DIR] + (s ? 1 : -1);
                const bool inner = (i >= 0 && i < g.n[DIR]) || g.periodic[DIR];
                const bool plain = !SIP || (uniform && ((pl >> (2 * DIR + s)) & 1u) && ((pl >> 8) & others) == others);
                h[s] = inner && on;
                if (h[s] && plain) {
                    const double* q = fct + (2 * DIR + s) * 6;
                    fc[s] = FaceCoef{q[0], q[1], q[2], q[3], q[4], q[5]};
                } else {
                    fc[s] = modal_face<D, SIP, MODE>(a, ijk, DIR, s, on, h[s]);
                }
            }
            const FaceCoef &fl = fc[0], &fu = fc[1];
            // a neighbour is read only where the form reads it, with diffusion everywhere, else where the
            // upwind flux takes its value: a zero coefficient times a NaN or Inf would carry it
            // upwind (J^T w takes the jump of w on both sides, as the quadrature kernels do)
            const bool every = MODE == MODE_VJP || diffusion, low = vel > 0.0;   // low: the flux takes the lower cell's value
            const double* nbu = h[1] && (every || (transport && !low)) ? own + sl : zero;
            const double* nbl = h[0] && (every || (transport && low)) ? own - sl : zero;
            const double vT = -2.0 * vel * thd * volm, vS = -2.0 * nu0 * thd * thd * volm;
            if constexpr (C::T == 1) {
                modal_pencils<D, K, SIP, MODE, DIR, 0>(T, own, nbu, nbl, fu, fl, vT, vS, R);
            } else {
                if (th == 0) modal_pencils<D, K, SIP, MODE, DIR, 0>(T, own, nbu, nbl, fu, fl, vT, vS, R);
                else if (th == 1) modal_pencils<D, K, SIP, MODE, DIR, 1>(T, own, nbu, nbl, fu, fl, vT, vS, R);
                if constexpr (C::T > 2) {
                    if (th == 2) modal_pencils<D, K, SIP, MODE, DIR, 2>(T, own, nbu, nbl, fu, fl, vT, vS, R);
                }
                if constexpr (C::T > 3) {
                    if (th == 3) modal_pencils<D, K, SIP, MODE, DIR, 3>(T, own, nbu, nbl, fu, fl, vT, vS, R);
                }
            }
        }
        __syncthreads();
    };
    direction(std::integral_constant<int, 0>{});
    direction(std::integral_constant<int, 1>{});
    if constexpr (D == 3) direction(std::integral_constant<int, 2>{});

    if constexpr (SIP && MODE == MODE_RES) {
        bool any = a.ph.g0 != 0.0;
#pragma unroll
        for (int d = 0; d < D; ++d) any = any || a.ph.g1[d] != 0.0 || a.ph.g2[d] != 0.0;
        const bool data = any && a.ph.has_sip && a.ph.dirichlet;
        if (data || a.ph.has_source) {   // uniform over the CTA
            if (active && th == 0) {
                auto faces = [&](auto dirc) {
                    constexpr int DIR = decltype(dirc)::value;
                    if (!data || g.periodic[DIR]) return;
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        if (ijk[DIR] != (s ? g.n[DIR] - 1 : 0)) continue;
                        if (MASK && !((fmask >> (2 * DIR + s)) & 1u)) continue;
                        bool nb;
                        const FaceCoef f = modal_face<D, SIP, MODE>(a, ijk, DIR, s, true, nb);
                        modal_boundary_data<D, K, DIR>(a, T, ijk, s, f, R);
                    }
                };
                faces(std::integral_constant<int, 0>{});
                faces(std::integral_constant<int, 1>{});
                if constexpr (D == 3) faces(std::integral_constant<int, 2>{});
                if (a.ph.has_source) R[0] += volm * a.ph.src * g.detJ * g.scaling * ((D == 3) ? 2.82842712474619009760 : 2.0);
            }
            __syncthreads();
        }
    }
    // ---- results stored in runs of cells
    for (int r = warp; r < rA; r += C::GRP * nw) {
        const double* src[C::GRP];
        double* dst[C::GRP];
        long long first[C::GRP];
#pragma unroll
        for (int k = 0; k < C::GRP; ++k) {
            const int rr = min(r + k * nw, rA - 1);
            const ModalRun q = runs[rr];
            const long long at = q.src + (o2 > 0 ? NP : 0);   // the row's own cells
            const int i0 = rr / e1, i1 = rr - i0 * e1;
            src[k] = res + ((i0 * b1 + i1) * b2) * S;
            dst[k] = out + at;
            first[k] = at / NP;
        }
        for (int e = lane; e < e2 * NP; e += 32) {
            const int c = e / NP, o = e + c * (S - NP);
#pragma unroll
            for (int k = 0; k < C::GRP; ++k) {
                if (r + k * nw >= rA || first[k] + c < a.cbeg || first[k] + c >= a.cend) continue;
                const double v = src[k][o];
                if (MODE == MODE_RES) dst[k][e] = (beta == 0.0) ? alpha * v : beta * dst[k][e] + alpha * v;
                else dst[k][e] = v;
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
