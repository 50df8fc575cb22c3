// modal.cu -- launches of the modal stencil kernel (modal_kernel.cuh) on one grid, and the tile
// extents of a grid.
#include <algorithm>

#include "modal_kernel.cuh"

namespace bosss {

namespace {

template <int D, int K, bool SIP, int MODE, bool MASK>
__global__ void __launch_bounds__(ModalCfg<D, K>::NT, ModalCfg<D, K>::MINB)
k_modal(const __grid_constant__ EvalArgs a, const __grid_constant__ ModalTile tl) {
    extern __shared__ double smem[];
    modal_tile<D, K, SIP, MODE, MASK>(a, a.tab, tl, blockIdx.x, MODE == MODE_RES ? a.U : a.V, a.out, a.alpha, a.beta, smem);
}

template <int D, int K, bool SIP, int MODE, bool MASK>
cudaError_t launch_masked(const EvalArgs& a, cudaStream_t s) {
    static unsigned long long done = 0ull;
    const size_t smem = ModalCfg<D, K>::SMEM;
    cudaError_t e = modal_attr(k_modal<D, K, SIP, MODE, MASK>, smem, done);
    if (e != cudaSuccess) return e;
    if (a.cend <= a.cbeg) return cudaSuccess;
    const ModalTile tl = modal_tiling(a, D, K);
    k_modal<D, K, SIP, MODE, MASK><<<tl.t[0] * tl.t[1] * tl.t[2], ModalCfg<D, K>::NT, smem, s>>>(a, tl);
    return cudaGetLastError();
}

template <int D, int K, bool SIP, int MODE>
cudaError_t launch_modal(const EvalArgs& a, cudaStream_t s) {
    // species masks (XDG) accompany the SIP residual only in practice; every mode reads them
    if constexpr (SIP && D == 3)
        if (a.vol_flag || a.face_flag) return launch_masked<D, K, SIP, MODE, true>(a, s);
    return launch_masked<D, K, SIP, MODE, false>(a, s);
}

template <int D, int K, bool SIP>
KernelEntry entry_of(int mode) {
    KernelEntry e{nullptr, ModalCfg<D, K>::CELLS, ModalCfg<D, K>::SMEM};
    e.launch = mode == MODE_RES   ? &launch_modal<D, K, SIP, MODE_RES>
               : mode == MODE_JVP ? &launch_modal<D, K, SIP, MODE_JVP>
                                  : &launch_modal<D, K, SIP, MODE_VJP>;
    return e;
}

template <int D>
KernelEntry entry_dim(int phys, int K, int mode) {
    if (phys == PHYS_TRANSPORT) switch (K) {
            case 0: return entry_of<D, 0, false>(mode);
            case 1: return entry_of<D, 1, false>(mode);
            case 2: return entry_of<D, 2, false>(mode);
            case 3: return entry_of<D, 3, false>(mode);
            case 4: return entry_of<D, 4, false>(mode);
        }
    if (phys == PHYS_SIP) switch (K) {
            case 1: return entry_of<D, 1, true>(mode);
            case 2: return entry_of<D, 2, true>(mode);
            case 3: return entry_of<D, 3, true>(mode);
            case 4: return entry_of<D, 4, true>(mode);
        }
    return KernelEntry{nullptr, 0, 0};
}

}  // namespace

KernelEntry modal_entry(int phys, int D, int K, int mode) {
    return D == 2 ? entry_dim<2>(phys, K, mode) : entry_dim<3>(phys, K, mode);
}

ModalTile modal_tiling(const EvalArgs& a, int D, int K, bool shared) {
    const TileRange r = tile_range(a, D);
    const int m0 = r.planes, n1 = r.n[1], n2 = r.n[2];
    int cells = 0, box = 0, per_sm = 1;
    auto cfg = [&](auto c) {
        using C = decltype(c);
        cells = C::CELLS;
        box = C::BOX;
        per_sm = std::min(C::MINB, 4);
    };
    switch (D * 10 + K) {
        case 20: cfg(ModalCfg<2, 0>{}); break;
        case 21: cfg(ModalCfg<2, 1>{}); break;
        case 22: cfg(ModalCfg<2, 2>{}); break;
        case 23: cfg(ModalCfg<2, 3>{}); break;
        case 24: cfg(ModalCfg<2, 4>{}); break;
        case 30: cfg(ModalCfg<3, 0>{}); break;
        case 31: cfg(ModalCfg<3, 1>{}); break;
        case 32: cfg(ModalCfg<3, 2>{}); break;
        case 33: cfg(ModalCfg<3, 3>{}); break;
        default: cfg(ModalCfg<3, 4>{}); break;
    }
    static thread_local TileMemo memo;
    ModalTile t = memo.get({{D, K, m0, n1, n2, (int)shared}}, [&] {
        // extents within the halo box of the slots
        ModalTile best{};
        double bc = 1e300;
        const int c0[] = {1, 2, 3, 4, 5, 6, 8}, c2[] = {2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 16};
        for (int b0 : c0)
            for (int b1 : c0)
                for (int b2 : c2) {
                    if (D == 2 && b1 != 1) continue;
                    if (b0 * b1 * b2 > cells || (b0 + 2) * (D == 3 ? b1 + 2 : 1) * (b2 + 2) > box) continue;
                    const long long t0 = (m0 + b0 - 1) / b0, t1 = (n1 + b1 - 1) / b1, t2 = (n2 + b2 - 1) / b2;
                    const double tiles = (double)t0 * t1 * t2;
                    const double staged = (double)b0 * b1 * b2 + 2.0 * b1 * b2 + 2.0 * b0 * b1 + (D == 3 ? 2.0 * b0 * b2 : 0.0);
                    // a CTA's time: fixed latencies (tile, runs, barriers), its copies and its cells (measured cycles)
                    const double cta = 7.0 + 0.016 * staged + 0.02 * b0 * b1 * b2;
                    const double cost = (shared ? tiles : tile_waves(tiles, per_sm)) * cta;
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

}  // namespace bosss
