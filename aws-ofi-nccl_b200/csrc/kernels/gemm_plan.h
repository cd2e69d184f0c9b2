// What the products on CTA pairs share on the host: the tiles they run on and their grid.
#pragma once
#include <stdint.h>

#include "gemm_tcgen05.cuh"

namespace b200 {

// Tiles of a product on CTA pairs: their width (a multiple of 32, 128 to 256) and whether those of the last
// wave are halved.
struct PairTiles {
  int width;
  bool halves;
};

// Fills in the tiles of `shape` (M, N and K are set). bn: the kernel's BN; ctas: how many may run. Returns how
// many are launched.
int pair_grid(GemmShape& shape, PairTiles tiles, int bn, int ctas);

// Whether a product runs whole on CTA pairs, neither on single CTAs nor split along K, and then its tiles among the
// widths 128 and 256.
bool runs_on_pairs(int M, int N, int K, int64_t lda, int64_t ldb, bool b_mn, const void* A, const void* B, PairTiles* tiles);

}  // namespace b200
