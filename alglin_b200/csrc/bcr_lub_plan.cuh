// Host side of the blocked FP64 LU kernel (bcr_lub.cuh): tile constants, the plan of
// a shape and the launch shape of a level.  Included inside namespace bcr.
#pragma once

constexpr int LUB_W = 64;          // panel columns per block (32 where 64 do not fit)
constexpr int LUB_ROWS_MAX = 512;  // one row per thread
constexpr int LUB_SLICES_MAX = 8;  // CTAs of a cluster (the portable limit)
constexpr int LUB_SB = 16;         // columns of a sub-block (registers of a row)
constexpr int LUB_LAST_W = LUB_SB; // columns per block of the last block: one sub-block
constexpr int LUB_UB = LUB_SB + 2; // stride of a column of the sub-block's pivot rows

// column stride of the panel block: 10 mod 16 words of 8 bytes, so that the
// column pairs of an accumulator tile (stride 2 ld) fall into different banks
// and the columns of an A fragment (stride ld) nearly so
__host__ __device__ inline int lub_ld(int rows) { return ((rows + 15) / 16) * 16 + 10; }
// the last block's panel of 16 columns
__host__ __device__ inline size_t lub_last_smem(int rows) { return (size_t)LUB_LAST_W * lub_ld(rows) * sizeof(double); }
// the panel block, the sub-block's operator rows and pivot rows
__host__ __device__ inline size_t lub_smem(int rows, int depth) {
  return ((size_t)(depth + LUB_SB) * lub_ld(rows) + (size_t)depth * LUB_UB) * sizeof(double);
}

// Threads, panel columns per block and their padding for R rows and npiv
// columns: two CTAs of 256 threads per SM where both their panel blocks fit in
// shared memory (their pivot steps and products overlap), else one CTA of 512;
// equal blocks of at most 64 columns (32 where 64 rows-high columns do not
// fit), padded with zero columns to 32, 48 or 64, the depths the products are
// built for.  threads == 0: the kernel does not apply.
struct LubPlan {
  int threads = 0, bw = 0, depth = 0;
  size_t smem = 0;
  int clusters[3] = {0, 0, 0};  // clusters of 2, 4 and 8 CTAs resident at once
};
inline LubPlan lub_plan(int rows, int npiv) {
  LubPlan p;
  if (rows > LUB_ROWS_MAX || npiv < 1) return p;
  for (int most : {LUB_W, 32}) {
    const int blocks = (npiv + most - 1) / most;
    const int bw = ((npiv + blocks - 1) / blocks + 7) / 8 * 8;
    const int depth = bw <= 32 ? 32 : bw <= 48 ? 48 : 64;
    const size_t sm = lub_smem(rows, depth);
    if (rows <= 256 && sm <= 106 * 1024) return {256, bw, depth, sm};
    if (sm <= 210 * 1024) return {512, bw, depth, sm};
  }
  return p;
}

// CTAs per pair (1, 2, 4 or 8: the columns right of its panel are split over a
// cluster) and CTAs of a level with np pairs.  Where the level has few pairs, the
// trailing columns of a pair are split (at least 24 columns each: every CTA
// repeats the panel), as long as all clusters are resident at once: 16 pairs of
// n = 128 in clusters of 8 took two waves, 341 us, and take 212 us in clusters of
// 4.  Every CTA owns one of `slots` slabs, so there are never more CTAs.
struct LubGrid {
  int slices;
  unsigned ctas;
};
inline LubGrid lub_grid(const LubPlan& p, long np, int trail, int slots) {
  int slices = 1;
  for (int i = 0; i < 3 && np <= p.clusters[i] && np * slices * 2 <= slots && trail >= slices * 2 * 24; ++i)
    slices *= 2;
  if (slices > 1) return {slices, (unsigned)(np * slices)};
  const long most = 148L * (512 / p.threads);
  return {1, (unsigned)(np < most ? (np < slots ? np : slots) : (most < slots ? most : slots))};
}
