// Host checks of the tile plans of the block kernels: the memo of the extents found last, and the
// cells that the blocks of a cell range cover and read.
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../bosss_b200/csrc/tile_stage.cuh"

using namespace bosss;

static int failures = 0;
#define CHECK(x) \
    if (!(x)) { \
        ++failures; \
        std::printf("line %d: %s\n", __LINE__, #x); \
    }

// callers that alternate between ranges or grids search once for each
static void check_memo() {
    TileMemo memo;
    int searches = 0;
    auto get = [&](int k) {
        const ModalTile t = memo.get({{3, 2, k, 5, 6, 0}}, [&] {
            ++searches;
            ModalTile s{};
            s.b[0] = k;
            return s;
        });
        CHECK(t.b[0] == k);
    };
    for (int round = 0; round < 10; ++round)
        for (int k = 1; k <= TileMemo::SIZE; ++k) get(k);
    CHECK(searches == TileMemo::SIZE);
    for (int k = 1; k <= 3 * TileMemo::SIZE; ++k) get(k);   // more than it holds: replaced in turn, never mixed up
    CHECK(searches == 3 * TileMemo::SIZE);
    get(3 * TileMemo::SIZE);
    CHECK(searches == 3 * TileMemo::SIZE);
    const ModalTile t = memo.get({{3, 2, 1, 5, 6, 1}}, [&] {   // any part of the key tells grids apart
        ModalTile s{};
        s.b[0] = 77;
        return s;
    });
    CHECK(t.b[0] == 77);
}

// the blocks of a launch cover its cells once and stay within the planes that hold them, whatever the
// extents: beyond, only the face neighbours of those planes (one plane on each side) are read
template <int D>
static void check_range(const int* n, const int* per, bool globalid, long long cbeg, long long cend) {
    EvalArgs a;
    std::memset(&a, 0, sizeof(a));
    a.g.D = D;
    for (int d = 0; d < 3; ++d) {
        a.g.n[d] = d < D ? n[d] : 1;
        a.g.periodic[d] = d < D ? per[d] : 0;
    }
    if (D == 2) {
        a.g.stride[0] = n[1];
        a.g.stride[1] = 1;
    } else if (globalid) {
        a.g.stride[0] = 1;
        a.g.stride[1] = n[0];
        a.g.stride[2] = (long long)n[0] * n[1];
    } else {
        a.g.stride[0] = (long long)n[1] * n[2];
        a.g.stride[1] = n[2];
        a.g.stride[2] = 1;
    }
    a.cbeg = cbeg;
    a.cend = cend;
    const TileRange r = tile_range(a, D);
    const long long plane = (long long)r.n[1] * r.n[2], J = plane * r.n[0];
    const long long first = cbeg / plane * plane, last = (cend + plane - 1) / plane * plane;   // whole planes
    CHECK(r.s0 * plane == first && (r.s0 + r.planes) * plane == last && last <= J);
    for (int b0 = 1; b0 <= 8; ++b0)
        for (int b1 = 1; b1 <= (D == 2 ? 1 : 4); ++b1)
            for (int b2 = 1; b2 <= 5; b2 += 2) {
                ModalTile t{};
                const int b[3] = {b0, b1, b2}, m[3] = {r.planes, r.n[1], r.n[2]};
                for (int d = 0; d < 3; ++d) {
                    t.b[d] = b[d];
                    t.t[d] = (m[d] + b[d] - 1) / b[d];
                }
                t.s0 = r.s0;
                t.planes = r.planes;
                std::vector<int> covered((size_t)J, 0);
                for (int k = 0; k < t.t[0] * t.t[1] * t.t[2]; ++k) {
                    const TileGeom G = tile_geom<D>(a.g, t, k);
                    for (int d = 0; d < 3; ++d) CHECK(G.n[d] == r.n[d] && G.e[d] >= 1 && G.e[d] <= b[d]);
                    CHECK(G.per[0] == (D == 3 && globalid ? per[2] : per[0]));
                    CHECK(G.o[0] + G.e[0] <= r.s0 + r.planes && G.o[1] + G.e[1] <= r.n[1] && G.o[2] + G.e[2] <= r.n[2]);
                    for (int i = 0; i < G.e[0]; ++i)
                        for (int j = 0; j < G.e[1]; ++j)
                            for (int l = 0; l < G.e[2]; ++l)
                                ++covered[(size_t)(((long long)(G.o[0] + i) * r.n[1] + G.o[1] + j) * r.n[2] + G.o[2] + l)];
                }
                for (long long c = 0; c < J; ++c) CHECK(covered[(size_t)c] == (c >= first && c < last));
            }
}

static void check_ranges() {
    const int n3[3] = {9, 4, 5}, n2[2] = {11, 6}, per[3] = {1, 0, 1};
    for (int globalid = 0; globalid < 2; ++globalid) {
        const int p = globalid ? 36 : 20;
        const long long J = 180;
        const long long r[][2] = {{0, J}, {0, 5 * p < J ? 3 * p : p}, {p, 4 * p}, {J - 2 * p, J}, {p, 2 * p}, {7, 8}, {13, 171}};
        for (const auto& c : r) check_range<3>(n3, per, globalid != 0, c[0], c[1]);
    }
    const long long r[][2] = {{0, 66}, {6, 36}, {12, 18}, {60, 66}, {7, 40}};
    for (const auto& c : r) check_range<2>(n2, per, false, c[0], c[1]);
}

int main() {
    check_memo();
    check_ranges();
    return failures != 0;
}
