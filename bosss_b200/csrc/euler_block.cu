// euler_block.cu -- instances and launches of the Euler block kernel.
#include "euler_block.h"

#include <algorithm>

#include "euler_block.cuh"

namespace bosss {

namespace {

template <class C>
ModalTile euler_tiling(const EvalArgs& a) {
    const TileRange r = tile_range(a, 3);
    const int m0 = r.planes, n1 = r.n[1], n2 = r.n[2];
    static thread_local TileMemo memo;
    ModalTile t = memo.get({{0, 0, m0, n1, n2, 0}}, [&] {
        ModalTile best{};
        double bc = 1e300;
        for (int b0 = 1; b0 <= 8; ++b0)
            for (int b1 = 1; b1 <= 8; ++b1)
                for (int b2 = 1; b2 <= 8; ++b2) {
                    const int cells = b0 * b1 * b2;
                    const int fmax = cells + std::max(b1 * b2, std::max(b0 * b2, b0 * b1));
                    if (cells > C::CELLS || fmax > C::FACES) continue;
                    const long long t0 = (m0 + b0 - 1) / b0, t1 = (n1 + b1 - 1) / b1, t2 = (n2 + b2 - 1) / b2;
                    const double tiles = (double)t0 * t1 * t2;
                    // a CTA's time from the rounds of its phases (weights: measured cycles per round, k = 3)
                    auto rounds = [](int tasks, int per) { return (double)((tasks + per - 1) / per); };
                    const int fd[3] = {cells + b1 * b2, cells + b0 * b2, cells + b0 * b1};
                    double cta = 8.0 + 7.3 * rounds(cells, C::NW * C::CW);
                    for (int f : fd)
                        cta += 3.9 * rounds(f * C::Q * C::Q, C::NT) + 2.5 * rounds(C::NROW * f + 5 * cells, C::NT) +
                               1.0 * rounds(C::NOUT * f, C::NT);
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

template <int K, int MODE>
cudaError_t launch_euler(const EvalArgs& a, cudaStream_t s) {
    using C = EulerCfg<K, MODE>;
    // J^T w for k = 2 on small grids: the slab tiles (4 cells, three CTAs per SM) take 15.6-20.7 us as long as they
    // fit one wave, the blocks' chain of phases 16.6-21.3 us (us, slab / blocks: 8 cells 15.5 / 16.2, 512 cells
    // 16.1 / 16.5, 729 cells 18.4 / 19.2, 1728 cells 20.7 / 21.3, 2744 cells 35.9 / 23.9); the other degrees and modes are
    // faster in blocks at every size
    if constexpr (K == 2 && MODE == MODE_VJP) {
        static const KernelEntry* slab = registered(PHYS_EULER, 3, K, K + 1, MODE, VARIANT_SLAB);
        if (slab && whole_grid_ctas(*slab, a.g) <= 148 * 3) return slab->launch(a, s);
    }
    static unsigned long long done = 0ull;
    int dev = 0;
    cudaGetDevice(&dev);
    if (!(done & (1ull << (dev & 63)))) {
        cudaError_t e = cudaFuncSetAttribute(k_euler_block<K, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k_euler_block<K, MODE>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        if (e != cudaSuccess) return e;
        done |= 1ull << (dev & 63);
    }
    if (a.cend <= a.cbeg) return cudaSuccess;
    const ModalTile tl = euler_tiling<C>(a);
    k_euler_block<K, MODE><<<tl.t[0] * tl.t[1] * tl.t[2], C::NT, C::SMEM, s>>>(a, tl);
    return cudaGetLastError();
}

template <int K>
KernelEntry entry_of(int mode) {
    KernelEntry e{nullptr, EulerCfg<K, MODE_RES>::CELLS, EulerCfg<K, MODE_RES>::SMEM};
    e.launch = mode == MODE_RES ? &launch_euler<K, MODE_RES> : mode == MODE_JVP ? &launch_euler<K, MODE_JVP> : &launch_euler<K, MODE_VJP>;
    return e;
}

}  // namespace

KernelEntry euler_block_entry(int K, int Q, int mode) {
    if (Q == K + 1) switch (K) {
            case 1: return entry_of<1>(mode);
            case 2: return entry_of<2>(mode);
            case 3: return entry_of<3>(mode);
            case 4: return entry_of<4>(mode);
        }
    return KernelEntry{nullptr, 0, 0};
}

}  // namespace bosss
