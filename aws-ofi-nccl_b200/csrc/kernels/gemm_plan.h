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

// Up to this K a tile's stores take longer than its products, and eight epilogue warps are worth the stage that their
// staging area costs, where a pair has several tiles: 4096 x 14336 of K = 128 takes 26.6 us in wide tiles, 29.8 with four warps, of K = 192
// 29.7 and 30.2; at K = 256 four are ahead (32.2, 33.1 with eight), over 40 products of K 200 to 256 by 2.5 %.
constexpr int SHORT_K = 192;

// Whether products may run on CTA pairs at all (B200_GEMM_2CTA).
bool pairs_enabled();

// M tiles of 128 rows per raster group of a kernel of BN `bn` (B200_GEMM_GROUP_M), and of 256 rows on CTA pairs.
int gemm_group_m(int bn);
inline int pair_group_m(int bn) { return (gemm_group_m(bn) + 1) / 2; }

// Order of the tiles of a product on CTA pairs whose group_m, tiles_m and tiles_n are set; elem_bytes: an operand's element.
void plan_walk(GemmShape& shape, int elem_bytes);

// Fills in the tiles of `shape` (M, N and K are set) and their order. bn: the kernel's BN; ctas: how many may run; elem_bytes: an operand's element. Returns how
// many are launched.
int pair_grid(GemmShape& shape, PairTiles tiles, int bn, int ctas, int elem_bytes = 2);

// Whether a product whose epilogue takes the sums in 32 bits (SwiGLU and its gradient) runs whole on CTA pairs, neither on single CTAs nor split
// along K, and then its tiles among the widths 128 and 256. Three rows of single-CTA tiles, which b200_gemm_bf16 has for 257 to 384 rows, don't count: the
// epilogue would be a pass over rounded sums. It would be faster (300 x 5120 x 4096 27.2 us forward, 22.3 in two launches, backward 32.0 and 22.8).
bool runs_on_pairs(int M, int N, int K, int64_t lda, int64_t ldb, bool b_mn, const void* A, const void* B, PairTiles* tiles);

// Clocks of a tile on CTA pairs: its k-blocks, or the stores of the tile before it where those take longer. lines: the
// operands' rows lie on cache lines; warps: epilogue warps.
inline double pair_tile_clocks(int k, int width, bool lines, int warps) {
  const double wide = lines ? 520 : 640;   // a k-block of 256 columns
  const double part = width == 256 ? 1 : width == 192 ? (lines ? .81 : .95) : (lines ? .58 : .72);
  const double blocks = (k + GEMM_BK - 1) / GEMM_BK * wide * part, stores = (width / 64) * 620.0 / (warps / 4) + 250;
  return (blocks > stores ? blocks : stores) + 150;
}
constexpr double LAUNCH_CLOCKS = 10000;   // a launch besides its tiles: ramp, pipeline fill, last stores
// Clocks that moving a product's operands and result takes at least.
inline double memory_clocks(double m, double n, double k) { return 2 * (m * k + n * k + m * n) / 3500; }

// Estimate for a product by itself, on what b200_gemm_bf16 would choose.
double product_clocks(int M, int N, int K, int64_t lda, int64_t ldb, bool b_mn, const void* A, const void* B);

}  // namespace b200
