// Tiles of the mixed form's P2G and grid update (mx_p2g_grid_kernel): which
// tile of which simulation a block takes.  Plain C++, so that the index
// arithmetic is checked on the host at grid sizes no test steps.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <vector>

#ifdef __CUDACC__
#define MPMG_HD __host__ __device__ __forceinline__
#else
#define MPMG_HD inline
#endif

// A tile's place: a word each for its row and column, since a grid may have
// more than 2^16 of either (the element count alone is limited, to 2^31).
struct alignas(16) MpmgTile {
    uint32_t member, row, col, unused;
};

// Tiles of `width` elements along a direction with `nodes` nodes: neighbours
// share one element, so each finishes width - 1 nodes.
MPMG_HD uint32_t mpmg_tiles_along(uint32_t nodes, uint32_t width)
{
    return (nodes + width - 2) / (width - 1);
}

// Tile `index` of a simulation with tiles_x tiles a row.
MPMG_HD MpmgTile mpmg_tile_at(uint32_t member, uint32_t index, uint32_t tiles_x)
{
    const uint32_t row = index / tiles_x;
    return MpmgTile{member, row, index - row * tiles_x, 0};
}

// Appends the tiles of a batch's member with Nx x Ny nodes, row by row.
inline void mpmg_append_tiles(std::vector<MpmgTile> &map, uint32_t member, uint32_t Nx, uint32_t Ny, uint32_t width,
                              uint32_t height)
{
    const uint32_t nx = mpmg_tiles_along(Nx, width), ny = mpmg_tiles_along(Ny, height);
    for (uint32_t row = 0; row < ny; row++)
        for (uint32_t col = 0; col < nx; col++) map.push_back(MpmgTile{member, row, col, 0});
}
