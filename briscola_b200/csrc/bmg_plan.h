// bmg_plan.h -- counts and extents that a launch and the buffer it writes
// have to agree on, and index ranges of kernels, as plain integer arithmetic
// (no CUDA types: the CPU tests compile this header by itself).
#pragma once

#include <algorithm>

#ifdef __CUDACC__
#define BMG_HD __host__ __device__
#else
#define BMG_HD
#endif

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

// ---- a level spread over a cluster's CTAs (bmg_tail.cu) ----------------------
// i-planes of a CTA, in whole groups of g (the planes that one coarse plane
// covers): rank r owns planes r P .. r P + P - 1 as far as there are any
inline int tail_planes(int n0, int g, int ranks) { return g * ((n0 + g * ranks - 1) / (g * ranks)); }

struct Planes {
    int first, count;
};
BMG_HD inline Planes tail_own(int n0, int P, int rank) {
    const int first = rank * P, left = n0 - first;
    return {first, left < 0 ? 0 : left < P ? left : P};
}

// planes of x that a CTA with `own` reads from memory: its own and the
// neighbours' on either side (-1 and n0 are the level's ghost planes).  The
// cluster is a power of two, so CTAs behind the last plane own none and read
// none.
BMG_HD inline Planes tail_read(Planes own) {
    return {own.first - 1, own.count ? own.count + 2 : 0};
}

}  // namespace bmg
