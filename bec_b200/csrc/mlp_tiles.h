// mlp_tiles.h -- how the output of one of the network's GEMMs (m x n, multiples of 64) is cut into tiles, one CTA each. Plain
// C++: the kernel's host side and the tests' compiler read it.
#pragma once

constexpr int kTileRows = 64, kWidestTile = 128;

// columns of a tile in a launch whose tiles are tn wide (16, 32, 64 or 128): a matrix that 128 does not divide stops at 64
constexpr int tile_cols(int n, int tn) { return tn == kWidestTile && n % kWidestTile ? kWidestTile / 2 : tn; }
constexpr int tile_ctas(int m, int n, int tn) { return m / kTileRows * (n / tile_cols(n, tn)); }
