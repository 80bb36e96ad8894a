// Host-side description of a multigrid level for the fused tile kernels
// (mg_tile.cu): which form the level takes, its row constants, and the tile
// geometry of the two launches.
#pragma once
#include "ow3d_internal.h"

namespace ow3d {

constexpr int kTileMaxNzg = 34;

// Row constants of a level whose interior columns all carry the same
// coefficients (flat bottom, no mixed-derivative terms): row k (index k-1)
// reads lo x_{k-1} + dg x_k + up x_{k+1} + off = b_k, id = 1 / dg, g = lo / dg.
template <typename T>
struct UniTab {
    T id[kTileMaxNzg], g[kTileMaxNzg], lo[kTileMaxNzg], up[kTileMaxNzg];
    T t0, t1, t6;             // bottom row: x_1 = (b_1 - t0 x_2 - t1 x_3) t6
    T wxl, wxr, wyd, wyu;     // neighbour columns' weights
    T gx[2][3], gy[2][3];     // ghost rows (low, high wall): nearest, second, 1 / ghost weight
};

// Row constants of a level with mixed-derivative terms: one minus sigma and
// the 3-point sigma stencils of orders 1 (z) and 2 (y); the column stencils,
// the same at every interior column of a uniform grid.
template <typename T>
struct RowTab {
    T om[kTileMaxNzg], z0[kTileMaxNzg], z1[kTileMaxNzg], z2[kTileMaxNzg];
    T y0[kTileMaxNzg], y1[kTileMaxNzg], y2[kTileMaxNzg];
    T sx1[3], sx2[3], sy1[3], sy2[3];   // centred, orders 1 and 2
    T ex[2][3], ey[2][3];     // order 1 at the ghost columns (low, high wall): the level below the bottom
    T gx[2][3], gy[2][3];     // ghost rows, as in UniTab
};

// One launch's tiles: cores of qx (+ 1 in the first remx) x qy columns, at
// most cx x cy, halo columns around them, HW slots per column parity and row,
// PH rows.
struct TileGeo {
    int cx, cy, ntx, nty, qx, remx, qy, remy, halo, HW, PH, NZP, threads;
    int np;                   // row pairs of a column
    size_t smem;
};

enum TileMode : int { kTileNone = 0, kTileUniform = 1, kTileCross = 2 };

template <typename T>
struct TileLevel {
    int mode = kTileNone;
    UniTab<T> u;
    RowTab<T> r;
    TileGeo down, up;
};

template <typename T>
void tile_geometry(const LevelDev<T>& L, TileLevel<T>& t);

// The right-hand side of both: the level's own (F.bv) when src is null, else
// src * *scale (scale null: 1), rounded to the level's type.
//
// Pre-smoothing from x = 0 (one step), residual and restriction of level F
// into rc (level Cc's right-hand side); the smoothed iterate goes to xs.
// zero: iterate of level Cc to clear, or null.
template <typename T>
void launch_tile_down(const LevelDev<T>& F, const LevelDev<T>& Cc, const TileLevel<T>& t, const double* src,
                      const double* scale, T* xs, T* rc, T* zero, cudaStream_t st);
// Correction xs + P xc and one post-smoothing step, into out (not xs).
template <typename T>
void launch_tile_up(const LevelDev<T>& F, const LevelDev<T>& Cc, const TileLevel<T>& t, const double* src,
                    const double* scale, const T* xs, const T* xc, T* out, cudaStream_t st);

}  // namespace ow3d
