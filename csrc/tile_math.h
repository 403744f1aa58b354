// Index arithmetic of the persistent tile schedulers, shared by the kernels and by a host-side unit test
// (tests/cpp/test_tile_math.cpp, built with -fsanitize=address,undefined): which tile a linear index names,
// which rows of a ragged expert range a tile covers, and how many tiles a problem has.  Plain integer code that
// compiles for the host and for the device.
#pragma once

#if defined(__CUDACC__)
#define KF_TM_HD __host__ __device__ __forceinline__
#else
#define KF_TM_HD inline
#endif

namespace kf {
namespace tilemath {

KF_TM_HD int imin(int a, int b) { return a < b ? a : b; }
KF_TM_HD int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Grouped rasterisation of an m_blocks x n_blocks tile grid: `group_m` consecutive row blocks share each sweep
// over the column blocks (so the column operand's tiles stay in L2).  Linear index t -> (m, n); a bijection
// onto the grid for 0 <= t < m_blocks * n_blocks, the last group may have fewer rows.
KF_TM_HD void raster(int t, int m_blocks, int n_blocks, int group_m, int& m, int& n) {
  const int per_group = group_m * n_blocks;
  const int g = t / per_group;
  const int first_m = g * group_m;
  const int rows = imin(group_m, m_blocks - first_m);
  const int r = t - g * per_group;
  m = first_m + r % rows;
  n = r / rows;
}

// Smallest and largest document id of a run of positions.  Two runs whose ranges do not meet hold no visible (query, key)
// pair, whatever the order of the ids.
struct IdRange {
  int lo, hi;
};
KF_TM_HD bool ids_meet(IdRange a, IdRange b) { return a.lo <= b.hi && b.lo <= a.hi; }

// Attention backward: whether the walk of a key tile with ids `own` visits query tile j with ids `range`; tiles before `first`
// lie above the causal diagonal.
KF_TM_HD bool query_tile_walked(int j, int first, IdRange range, IdRange own) { return j >= first && ids_meet(range, own); }

// Ragged grouped GEMM.  tile_start[e] = number of row tiles (of `bm` rows) of experts 0..e-1, tile_start[E] the
// total; offsets[e] .. offsets[e+1] are expert e's rows.  Fills tile_start and returns the total.
KF_TM_HD int grouped_tile_starts(const int* offsets, int E, int bm, int* tile_start) {
  int acc = 0;
  for (int e = 0; e < E; ++e) {
    tile_start[e] = acc;
    acc += ceil_div(offsets[e + 1] - offsets[e], bm);
  }
  tile_start[E] = acc;
  return acc;
}

struct GroupedTile {
  int e;      // expert
  int row0;   // first row of the tile in the sorted activation matrix
  int valid;  // rows of the tile that belong to the expert (1 .. bm)
  int nb;     // column block
};

// Linear tile index t (column block fastest) -> the tile; experts without rows own no tile.
KF_TM_HD GroupedTile grouped_decode(int t, int n_blocks, const int* tile_start, const int* offsets, int E, int bm) {
  const int nb = t % n_blocks;
  const int tmi = t / n_blocks;
  int lo = 0, hi = E;  // largest e with tile_start[e] <= tmi (among equal starts the last one owns the tile)
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (tile_start[mid] <= tmi) lo = mid; else hi = mid;
  }
  GroupedTile x;
  x.e = lo;
  const int mb = tmi - tile_start[lo];
  x.row0 = offsets[lo] + mb * bm;
  x.valid = imin(bm, offsets[lo + 1] - x.row0);
  x.nb = nb;
  return x;
}

// Ragged grouped GEMM with tokens as the N side of the MMA: expert e's rows are cut into n = ceil(rows / widest) tiles of
// token_tile_width(rows, n) tokens (the last one may hold fewer, never none), each met by every block of weight rows.
constexpr int NARROWEST_TOKENS = 96;  // below, a tile takes no less time
KF_TM_HD int token_tile_width(int rows, int n) { return n > 0 ? ceil_div(ceil_div(rows, n), 32) * 32 : 0; }

// What a tile takes, in units of one token's share of a k-block on a CTA pair.  Measured, ns per k-block of 64: 96 tokens 210, 128 245, 160
// 285, 192 330, 224 390, 256 430 (products of 4096 and 28 672 rows with 4096 columns, back to back).
KF_TM_HD int token_tile_cost(int width) { return 48 + (width < NARROWEST_TOKENS ? NARROWEST_TOKENS : width); }

// Rounds of `tiles` x `f_blocks` tiles over the pairs, times the average tile.
KF_TM_HD float token_rounds_cost(int tiles, int cost, int f_blocks, int pairs) {
  if (tiles == 0) return 0.f;
  const long long all = (long long)tiles * f_blocks;
  return float((all + pairs - 1) / pairs) * (float(cost) / float(tiles));
}

struct TokenTile {
  int e, fb;       // expert and block of weight rows
  int row0;        // first row of the tile in the sorted activation matrix
  int valid;       // rows of the tile that belong to the expert (1 .. width)
  int width;       // tokens of the tile as computed (a multiple of 32 up to the widest)
};

// Walks the tiles in ascending order of their linear index (experts slowest, token tiles fastest); experts without rows own none.
struct TokenTiles {
  const int* offsets;
  int f_blocks, widest;
  int e, first, n;  // current expert, its first tile, its token tiles
  KF_TM_HD TokenTiles(const int* off, int fb, int w) : offsets(off), f_blocks(fb), widest(w), e(0), first(0) {
    n = ceil_div(off[1] - off[0], w);
  }
  KF_TM_HD TokenTile at(int t) {
    while (t >= first + n * f_blocks) {
      first += n * f_blocks;
      ++e;
      n = ceil_div(offsets[e + 1] - offsets[e], widest);
    }
    const int r = t - first, rows = offsets[e + 1] - offsets[e];
    TokenTile x;
    x.e = e;
    x.fb = r / n;
    x.width = token_tile_width(rows, n);
    const int at = (r - x.fb * n) * x.width;
    x.row0 = offsets[e] + at;
    x.valid = imin(x.width, rows - at);
    return x;
  }
};

struct WgradTile {
  int e, m0, n0;  // expert, first output row / column of the tile
  int row0, rows; // the expert's range of the reduction dimension
};

// Grouped weight gradient: every expert owns m_blocks x n_blocks output tiles, whatever its row count.
KF_TM_HD WgradTile wgrad_decode(int t, int m_blocks, int n_blocks, int bm, int bn, const int* offsets) {
  WgradTile x;
  const int per_e = m_blocks * n_blocks;
  x.e = t / per_e;
  const int r = t - x.e * per_e;
  x.m0 = (r / n_blocks) * bm;
  x.n0 = (r % n_blocks) * bn;
  x.row0 = offsets[x.e];
  x.rows = offsets[x.e + 1] - x.row0;
  return x;
}

// Number of zeroed 16-byte chunks, and the address of chunk i, when the rows `valid .. bk-1` of every
// {64 columns x bk rows} block of a stage (128 bytes per row, `blocks` blocks of `block_bytes`) are cleared.
KF_TM_HD int tail_chunks(int valid, int bk, int blocks) { return (bk - valid) * 8 * blocks; }
KF_TM_HD int tail_chunk_offset(int i, int valid, int bk, int block_bytes) {
  const int per_block = (bk - valid) * 8;
  const int blk = i / per_block, j = i - blk * per_block;
  return blk * block_bytes + valid * 128 + j * 16;
}

}  // namespace tilemath
}  // namespace kf
