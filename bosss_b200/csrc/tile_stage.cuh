// tile_stage.cuh -- blocks of cells with a face halo in shared memory (scalar and system tiles).
//
// A CTA owns a block of b[0] x b[1] x b[2] cells in memory order (slow, middle, fast direction of
// the local cell numbering). Every cell of the block and of its six face halos has a slot of S
// doubles in a (b+2)^3 halo box; the corners stay unused. The copies are asynchronous 8-byte
// ones: the caller's vectors may start at any double.
#pragma once
#include <algorithm>

#include "modal.h"

namespace bosss {

__device__ __forceinline__ void tile_cp8(void* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void tile_cp_wait() {
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// 1 / cell length scale of a cell (penalty_size without divisions)
template <int D>
__device__ __forceinline__ double tile_size(const EvalArgs& a, const int* ijk) {
    if (a.cell_pf) return penalty_size(a.cell_pf, a.g, ijk);
    double cj = 0.0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        int nb = 2;
        if (!a.g.gper[d]) {
            const int gi = ijk[d] + a.g.goff[d];
            nb += (gi == 0) + (gi == a.g.gn[d] - 1);
        }
        cj += nb * (0.5 * a.g.twoh[d]);
    }
    return 0.5 * cj;
}

// Time of `tiles` CTAs in units of one CTA's time in a full wave of 148 x per_sm: whole waves, and for
// the rest the pace of an SM that holds fewer CTAs (a CTA alone on its SM runs at about 0.6 of its
// time among three); many waves overlap and count by their share
inline double tile_waves(double tiles, int per_sm) {
    const double slots = 148.0 * per_sm, w = tiles / slots;
    if (w >= 4.0) return w;
    const double full = (double)(long long)w, sm = (tiles - full * slots) / 148.0;
    const double rest = sm <= 0.0 ? 0.0 : sm <= 1.0 ? (per_sm == 1 ? 1.0 : 0.6) : 0.6 + 0.4 * (sm - 1.0) / (per_sm - 1);
    return full + rest;
}

// Extents found for the last grids on one thread: they depend on the sizes alone, and the search over a
// few hundred candidates costs as much as a launch. Several entries, replaced in turn, because callers
// alternate between grids or ranges of one (species B of an XDG operator has up to three ranges); with one
// entry, three small advection-diffusion grids in turn took 9.2 us per residual, with these 6.6
class TileMemo {
public:
    struct Key {
        int v[6];
    };
    template <class Search>
    const ModalTile& get(const Key& k, Search&& search) {
        for (int i = 0; i < used_; ++i)
            if (std::equal(k.v, k.v + 6, key_[i].v)) return tile_[i];
        const int i = next_;
        next_ = (next_ + 1) % SIZE;
        if (used_ < SIZE) ++used_;
        tile_[i] = search();
        key_[i] = k;
        return tile_[i];
    }

    static constexpr int SIZE = 16;

private:
    Key key_[SIZE] = {};
    ModalTile tile_[SIZE] = {};
    int used_ = 0, next_ = 0;
};

// memory-order extents of a grid (slow, middle, fast; 2D: middle = 1), first plane of the slow direction
// and number of planes that hold the cells [cbeg, cend)
struct TileRange {
    int n[3], s0, planes;
};
inline TileRange tile_range(const EvalArgs& a, int D) {
    const GridConst& g = a.g;
    const bool rev = D == 3 && g.stride[0] == 1 && g.stride[2] != 1;
    TileRange r;
    r.n[0] = rev ? g.n[2] : g.n[0];
    r.n[1] = D == 3 ? g.n[1] : 1;
    r.n[2] = D == 3 ? (rev ? g.n[0] : g.n[2]) : g.n[1];
    const long long plane = (long long)r.n[1] * r.n[2];
    r.s0 = (int)(a.cbeg / plane);
    r.planes = (int)std::max<long long>(1, std::min<long long>(r.n[0], (a.cend + plane - 1) / plane) - r.s0);
    return r;
}

// the quadrature kernel that a block kernel leaves some launches to; null: no instance
inline const KernelEntry* registered(int phys, int D, int K, int Q, int mode, int variant) {
    const auto it = kernel_registry().find(KernelKey(phys, D, K, Q, mode, variant));
    return it == kernel_registry().end() ? nullptr : &it->second;
}

// CTAs of the kernel `e` over the whole grid (of a part: the global one, so that parts, cell ranges and the
// whole grid take the same kernel)
inline long long whole_grid_ctas(const KernelEntry& e, const GridConst& g) {
    const long long J = (long long)g.gn[0] * g.gn[1] * g.gn[2];
    return (J + e.cells_per_block - 1) / e.cells_per_block;
}

// memory-order view of a grid and the block of one tile
struct TileGeom {
    bool rev;          // GlobalID order: x fastest
    int n[3], per[3];  // cells and periodicity per memory direction
    int o[3], e[3];    // first cell and (clipped) extent of the block
    int q0, q1;        // slot strides (in slots) of the slow and middle direction
    __device__ __forceinline__ int slot(int i0, int i1, int i2) const { return (i0 + 1) * q0 + (i1 + 1) * q1 + i2 + 1; }
    // memory direction of physical direction d
    __device__ __forceinline__ int mem(int d) const { return rev ? 2 - d : d; }
};

// The block ends with the launch's planes, not with the grid: beyond the range only the face neighbours of
// its cells are read, so that a caller may still be writing the rest (host chunks that are on their way,
// a halo exchange in flight)
template <int D = 3>
__host__ __device__ __forceinline__ TileGeom tile_geom(const GridConst& g, const ModalTile& tl, int tile) {
    TileGeom G;
    G.rev = D == 3 && g.stride[0] == 1 && g.stride[2] != 1;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        G.n[m] = D == 2 ? (m == 1 ? 1 : g.n[m >> 1]) : G.rev ? g.n[2 - m] : g.n[m];
        G.per[m] = D == 2 ? (m == 1 ? 0 : g.periodic[m >> 1]) : G.rev ? g.periodic[2 - m] : g.periodic[m];
    }
    const int t2 = tile % tl.t[2], tq = tile / tl.t[2];
    const int t1 = tq % tl.t[1], t0 = tq / tl.t[1];
    G.o[0] = tl.s0 + t0 * tl.b[0];
    G.o[1] = t1 * tl.b[1];
    G.o[2] = t2 * tl.b[2];
    G.e[0] = min(tl.b[0], tl.planes - t0 * tl.b[0]);   // (from a plane's number: more registers, SIP 2 % slower)
    G.e[1] = min(tl.b[1], G.n[1] - G.o[1]);
    G.e[2] = min(tl.b[2], G.n[2] - G.o[2]);
    G.q1 = tl.b[2] + 2;
    G.q0 = (tl.b[1] + 2) * (tl.b[2] + 2);
    return G;
}

// stage NC consecutive doubles per cell of `in` (cell-major) into slots of S doubles
template <int NC, int S, int NT>
__device__ __forceinline__ void tile_stage(const TileGeom& G, const double* __restrict__ in, double* sm) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int nw = NT >> 5;
    const int rA = G.e[0] * G.e[1], rB = 2 * G.e[1], rC = 2 * G.e[0];
    for (int r = warp; r < rA + rB + rC; r += nw) {
        int i0, i1, f0 = 0, nf = G.e[2];
        if (r < rA) {
            i0 = r / G.e[1];
            i1 = r - i0 * G.e[1];
            f0 = -1;
            nf = G.e[2] + 2;
        } else if (r < rA + rB) {
            const int q = r - rA;
            i0 = (q & 1) ? G.e[0] : -1;
            i1 = q >> 1;
        } else {
            const int q = r - rA - rB;
            i0 = q >> 1;
            i1 = (q & 1) ? G.e[1] : -1;
        }
        int m0 = G.o[0] + i0, m1 = G.o[1] + i1;
        if (m0 < 0 || m0 >= G.n[0]) {
            if (!G.per[0]) continue;
            m0 = m0 < 0 ? m0 + G.n[0] : m0 - G.n[0];
        }
        if (m1 < 0 || m1 >= G.n[1]) {
            if (!G.per[1]) continue;
            m1 = m1 < 0 ? m1 + G.n[1] : m1 - G.n[1];
        }
        const long long row = ((long long)m0 * G.n[1] + m1) * G.n[2];
        double* dst = sm + G.slot(i0, i1, 0) * S;
        for (int e = lane; e < nf * NC; e += 32) {
            const int c = e / NC, k = e - c * NC;
            const int i2 = f0 + c;
            int m2 = G.o[2] + i2;
            if (m2 < 0 || m2 >= G.n[2]) {
                if (!G.per[2]) continue;
                m2 = m2 < 0 ? m2 + G.n[2] : m2 - G.n[2];
            }
            tile_cp8(dst + i2 * S + k, in + (row + m2) * NC + k);
        }
    }
}

}  // namespace bosss
