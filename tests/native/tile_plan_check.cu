// Host checks of the tile plans of the block kernels: the memo of the extents found last.
#include <cstdio>

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

int main() {
    check_memo();
    return failures != 0;
}
