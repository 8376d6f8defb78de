// bmg_plan.h -- counts and extents that a launch and the buffer it writes
// have to agree on, as plain integer arithmetic (no CUDA types: the CPU tests
// compile this header by itself).
#pragma once

#include <algorithm>

namespace bmg {

struct Tile {
    int x, y;
};

// block of the one-cell-per-thread kernels: the k extent on lanes; small rows
// give the spare lanes to j
inline Tile cell_tile(int n2) {
    if (n2 >= 64) return {64, 4};
    if (n2 >= 32) return {32, 8};
    if (n2 >= 16) return {16, 16};
    return {8, 32};
}

// what the level-0 reductions need to know of a mesh
struct Level0 {
    int nb;      // bricks
    int max1;    // largest extents along j and k
    int max2;
    int planes;  // planes of all bricks
    bool quads;  // every brick's rows are whole quads (n2 % 4 == 0)
};

inline int blocks_of(int n, int tile) { return (n + tile - 1) / tile; }

// per-block partial sums of the one-cell-per-thread reductions
inline long cell_partials(const Level0& L) {
    const Tile t = cell_tile(L.max2);
    return (long)blocks_of(L.max2, t.x) * blocks_of(L.max1, t.y) * L.planes;
}

// The flexible-CG passes on rows of whole quads: 16 x 16 threads of a quad
// each, and a block for every kQuadPlanes-th plane of the mesh (several
// bricks: four times as many plane groups, since many blocks of a plane lie
// outside their brick).
constexpr int kQuadTile = 16;
constexpr int kQuadPlanes = 64;
inline int quad_planes(const Level0& L) { return std::min(L.planes, L.nb > 1 ? 4 * kQuadPlanes : kQuadPlanes); }
inline long quad_partials(const Level0& L) {
    return (long)blocks_of(L.max2 / 4, kQuadTile) * blocks_of(L.max1, kQuadTile) * quad_planes(L);
}

// partial sums of the flexible-CG steps and of the residual on parity-split rows
inline long step_partials(const Level0& L) { return L.quads ? quad_partials(L) : cell_partials(L); }

// doubles of the context's buffer of partial sums: up to three sums a block
// (rows of 4 or 8 cells have half as many rows of blocks in cell_partials as in
// quad_partials)
inline long partials_capacity(const Level0& L) { return 3 * std::max(cell_partials(L), step_partials(L)); }

}  // namespace bmg
