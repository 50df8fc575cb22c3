// sip.cu -- instances and launches of the nonlinear-diffusion block kernel.
#include "sip.h"

#include <algorithm>

#include "sip_kernel.cuh"

namespace bosss {

namespace {

// block extents: every launch covers the cells [cbeg, cend); cost = waves of resident CTAs times the
// phases of a block (staged cells, faces, volume), the faces between blocks being evaluated twice
template <class C>
ModalTile sip_tiling(const EvalArgs& a) {
    // volume round against a face-row round: QV^2 nodes of a slab against Q of a row
    const double VW = 0.6 * C::QV * C::QV / C::FQ;
    const TileRange r = tile_range(a, 3);
    const int m0 = r.planes, n1 = r.n[1], n2 = r.n[2];
    static thread_local TileMemo memo;
    ModalTile t = memo.get({{0, 0, m0, n1, n2, 0}}, [&] {
        ModalTile best{};
        double bc = 1e300;
        const int ext[] = {1, 2, 3, 4, 5, 6, 8};
        for (int b0 : ext)
            for (int b1 : ext)
                for (int b2 : ext) {
                    const int cells = b0 * b1 * b2;
                    const int fmax = cells + std::max(b1 * b2, std::max(b0 * b2, b0 * b1));
                    if (cells > C::CELLS || (b0 + 2) * (b1 + 2) * (b2 + 2) > C::SLOTS || fmax > C::FACES) continue;
                    const long long t0 = (m0 + b0 - 1) / b0, t1 = (n1 + b1 - 1) / b1, t2 = (n2 + b2 - 1) / b2;
                    const double tiles = (double)t0 * t1 * t2;
                    // a CTA's time from the rounds of its phases (weights: measured shares, k = 2 and 4)
                    auto rounds = [](int tasks) { return (double)((tasks + C::NT - 1) / C::NT); };
                    const int fd[3] = {cells + b1 * b2, cells + b0 * b2, cells + b0 * b1};
                    double cta = 2.0 + VW * rounds(cells * C::QV) + 0.6 * rounds(cells * C::NPAIR);
                    for (int f : fd) cta += 2.0 * rounds(f * C::FQ) + 0.8 * rounds(2 * C::NG * f + C::NPAIR * cells);
                    const double waves = tile_waves(tiles, C::MINB);
                    const double cost = waves * cta;
                    if (cost < bc) {
                        bc = cost;
                        best.b[0] = b0;
                        best.b[1] = b1;
                        best.b[2] = b2;
                        best.t[0] = (int)t0;
                        best.t[1] = (int)t1;
                        best.t[2] = (int)t2;
                    }
                }
        best.ncell = best.b[0] * best.b[1] * best.b[2];
        return best;
    });
    t.s0 = r.s0;
    t.planes = r.planes;
    return t;
}

template <int K, int Q, int MODE>
cudaError_t launch_sip(const EvalArgs& a, cudaStream_t s) {
    using C = SipCfg<K, Q, MODE>;
    if (a.vol_flag || a.face_flag) {   // species masks: the slab tile reads them
        const KernelEntry* slab = registered(PHYS_SIP, 3, K, Q, MODE, VARIANT_SLAB);
        return slab ? slab->launch(a, s) : cudaErrorNotSupported;
    }
    // Products with 7 or 9 nodes on the smallest grids: the generic tile spreads a cell's nodes over 128 or more
    // threads, a block has a thread per z-slab and a chain of phases (24-28 us for k = 3, 41-57 us for k = 4
    // whatever the size). As long as the generic tiles fit one wave -- one CTA per SM for k = 3, two for k = 4 --
    // they are faster (us, generic / block; J v, J^T w within 1 us of it): k = 4, Q = 9, 8 cells 27.3 / 51.8, 216 cells
    // 33.1 / 52.4, 343 cells (second wave) 56.7 / 48.5; Q = 7, 512 cells 38.2 / 41.1, 729 cells 66.1 / 43.8; k = 3, 1 cell
    // 23.2 / 27.3, 216 cells 25.9 / 26.7, 343 cells 30.3 / 26.3
    if constexpr (MODE != MODE_RES && Q >= 7) {
        static const KernelEntry* generic = registered(PHYS_SIP, 3, K, Q, MODE, VARIANT_GENERIC);
        if (generic && whole_grid_ctas(*generic, a.g) <= 148 * (K == 4 ? 2 : 1)) return generic->launch(a, s);
    }
    static const Tables1D V = [] {
        Tables1D t;
        build_tables(K, C::QV, t);
        return t;
    }();
    static unsigned long long done = 0ull;
    int dev = 0;
    cudaGetDevice(&dev);
    if (!(done & (1ull << (dev & 63)))) {
        cudaError_t e = cudaFuncSetAttribute(k_sip<K, Q, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sip<K, Q, MODE>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        if (e != cudaSuccess) return e;
        done |= 1ull << (dev & 63);
    }
    if (a.cend <= a.cbeg) return cudaSuccess;
    const ModalTile tl = sip_tiling<C>(a);
    k_sip<K, Q, MODE><<<tl.t[0] * tl.t[1] * tl.t[2], C::NT, C::SMEM, s>>>(a, V, tl);
    return cudaGetLastError();
}

template <int K, int Q>
KernelEntry entry_of(int mode) {
    KernelEntry e{nullptr, SipCfg<K, Q, MODE_RES>::CELLS, SipCfg<K, Q, MODE_RES>::SMEM};
    e.launch = mode == MODE_RES ? &launch_sip<K, Q, MODE_RES> : mode == MODE_JVP ? &launch_sip<K, Q, MODE_JVP> : &launch_sip<K, Q, MODE_VJP>;
    return e;
}

}  // namespace

KernelEntry sip_entry(int K, int Q, int mode) {
#define BOSSS_SIP_CASE(k, q) \
    if (K == k && Q == q) return entry_of<k, q>(mode);
    BOSSS_SIP_CASE(1, 2)
    BOSSS_SIP_CASE(1, 3)
    BOSSS_SIP_CASE(2, 3)
    BOSSS_SIP_CASE(2, 4)
    BOSSS_SIP_CASE(2, 5)
    BOSSS_SIP_CASE(3, 4)
    BOSSS_SIP_CASE(3, 5)
    BOSSS_SIP_CASE(3, 7)
    BOSSS_SIP_CASE(4, 5)
    BOSSS_SIP_CASE(4, 7)
    BOSSS_SIP_CASE(4, 9)
#undef BOSSS_SIP_CASE
    return KernelEntry{nullptr, 0, 0};
}

}  // namespace bosss
