// Test-only: the mixed form's tile arithmetic (mpmg_tiles.h) as C functions.
// Built by tests/test_mixed_tiles.py with g++ into a temporary shared library.
#include "../../mpm-2d_gb300/csrc/mpmg_tiles.h"

// The tiles of members with grids[2 k] x grids[2 k + 1] nodes, as (member, row,
// col) triples in out; the number of tiles is returned.  out may be null.
extern "C" long long batch_tiles(int members, const uint32_t *grids, uint32_t width, uint32_t height, uint32_t *out)
{
    std::vector<MpmgTile> map;
    for (int k = 0; k < members; k++)
        mpmg_append_tiles(map, (uint32_t)k, grids[2 * k], grids[2 * k + 1], width, height);
    for (size_t i = 0; out != nullptr && i < map.size(); i++) {
        out[3 * i] = map[i].member;
        out[3 * i + 1] = map[i].row;
        out[3 * i + 2] = map[i].col;
    }
    return (long long)map.size();
}

// The same for the blocks of a single simulation.
extern "C" void single_tiles(uint32_t Nx, uint32_t width, long long blocks, uint32_t *out)
{
    const uint32_t tiles_x = mpmg_tiles_along(Nx, width);
    for (long long i = 0; i < blocks; i++) {
        const MpmgTile t = mpmg_tile_at(0, (uint32_t)i, tiles_x);
        out[3 * i] = t.member;
        out[3 * i + 1] = t.row;
        out[3 * i + 2] = t.col;
    }
}
