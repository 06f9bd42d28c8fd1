// common.cuh: device-side layout and integer primitives shared by the decision kernels.
//
// Planes live in HBM with a replicated margin of M samples on every side: a plane of w x h
// samples is stored in (w + 2M) x (h + 2M) bytes, and the margin repeats the nearest edge sample.
// The reference reads every plane through a clamped accessor (src/gpu/intra_common.h:17-25); with
// the margin, clamping a coordinate into [-M, size + M) gives the same sample as clamping it into
// [0, size), so kernels read directly wherever a footprint lies inside the margin and clamp to the
// allocated extent otherwise (which is still exact, and never leaves the allocation).
#pragma once
#include <cstdint>

#include "celv2_decision.h"

namespace celv2cu {

constexpr int kLevels = CELV2_ME_LEVELS;
constexpr int kMaxRefs = CELV2_MAX_REFS;
constexpr int kBlocks = CELV2_SB_BLOCKS;
constexpr int kModes = CELV2_NUM_MODES;
constexpr int kPhases = 16;
// Decision constants (reference src/gpu/inter_common.h:35-55,140, src/gpu/intra_common.h:32-42).
constexpr int kMeRange = 8;
constexpr int kMePenalty = 4;
constexpr int kSubpelPenalty = 16;
constexpr int kInterBits = 3;
constexpr int kIntraInInterBits = 32;
constexpr int kPartBits = 2;

// Margin per pyramid level. The motion search reaches at most 8 * (2^(5-l) - 1) pels from a cell
// at level l (248 at level 0, plus 3/4 pel of refinement), the superblock grid overhangs the padded
// frame by at most 56 samples and intra edges reach 95 samples past a block: 320 >> l (at least
// 32) covers all of it, so the clamping fallback never runs for in-range inputs.
__host__ __device__ constexpr int level_margin(int l) { return (320 >> l) < 32 ? 32 : (320 >> l); }

struct DevPlane {
  const uint8_t* p;   // the sample (0, 0); rows of `stride` bytes; valid rows/cols [-margin, size + margin)
  int stride, w, h, margin;
  long long phase;    // bytes between quarter-pel phase planes (level 0 of a reference), 0: none
};

struct DevPyramid {
  DevPlane lv[kLevels];
};

// A CUtensorMap, as bytes (the host alone knows its type).
struct alignas(128) TensorMap {
  unsigned char bytes[128];
};

// One frame's decision work as the kernels see it (written by the host per launch).
struct FrameJob {
  DevPyramid cur;
  DevPyramid ref[kMaxRefs];
  int nrefs;
  int pw, ph;              // padded luma size (multiple of 8)
  int sb_cols, sb_rows;
  int fcols[kLevels], frows[kLevels];
  int* field[kMaxRefs][kLevels];  // packed MVs: (mvy << 16) | (mvx & 0xffff)
  const int* intra;        // [sb][kModes][kBlocks] SATDs (blocks < 5 unused)
  int2* inter;             // [sb][kMaxRefs][kBlocks]: (best SATD, packed MV)
  celv2_sb_out* out;       // [sb]
  long long lam;           // lambda_q8
  // Work counters for the roofline (null unless stage timing is on): [l] searched centres at
  // level l, [5] inter tile SATDs (tiles x distinct MVs per region), [6] compound 4x4 tiles.
  unsigned long long* stats;
  // Pruning (null: the exhaustive search): per superblock a keep word (include/celv2_decision.h:
  // references, intra, block levels, intra modes; see keep_mask). The kept options are scored
  // exactly as without pruning.
  const uint32_t* keep;
  long long* sb_cost;      // [sb]: the chosen partition's cost (null: not written)
  // Each reference's phase planes as one tensor for TMA (bytes of a stored row, stored rows, phases),
  // and the host's mark of a wait in a kernel that ran out.
  TensorMap map[kMaxRefs];
  int* fault;
};

enum { kStatInterMvs = 5, kStatCompoundTiles = 6, kStats = 8 };

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// The effective keep word of superblock sb: all options without pruning or in a KEY frame;
// otherwise the given references (all of them if none is given), intra if its bit is set, the
// given block levels and intra modes (all of them if none is given).
__device__ __forceinline__ unsigned keep_mask(const FrameJob& job, int sb) {
  const unsigned all = (1u << job.nrefs) - 1u;
  if (!job.keep || job.nrefs == 0) return all | CELV2_KEEP_INTRA | CELV2_KEEP_LEVELS | CELV2_KEEP_MODES;
  const unsigned k = job.keep[sb];
  const unsigned levels = k & CELV2_KEEP_LEVELS, modes = k & CELV2_KEEP_MODES;
  return ((k & all) ? (k & all) : all) | (k & CELV2_KEEP_INTRA) | (levels ? levels : CELV2_KEEP_LEVELS) |
         (modes ? modes : CELV2_KEEP_MODES);
}

// The square level of candidate block b: 0 for 64x64 (and its halves), 1 for 32x32, 2 for 16x16,
// 3 for 8x8.
__host__ __device__ __forceinline__ int block_level(int b) {
  const int sq = b / 5;
  return sq >= 21 ? 3 : sq >= 5 ? 2 : sq >= 1 ? 1 : 0;
}

// Whether level-0 cell (cx, cy) of reference r is read by the inter stage of a superblock that
// keeps r: superblock (sx, sy) reads the cells sx * 8 - 1 .. sx * 8 + 8 (clamped), likewise in y.
__device__ __forceinline__ bool cell_needed(const FrameJob& job, int r, int cx, int cy) {
  if (!job.keep) return true;
  const int x0 = cx >= 8 ? (cx - 1) >> 3 : 0, x1 = min(job.sb_cols - 1, (cx + 1) >> 3);
  const int y0 = cy >= 8 ? (cy - 1) >> 3 : 0, y1 = min(job.sb_rows - 1, (cy + 1) >> 3);
  for (int sy = y0; sy <= y1; sy++)
    for (int sx = x0; sx <= x1; sx++)
      if (keep_mask(job, sy * job.sb_cols + sx) >> r & 1u) return true;
  return false;
}

// The clamped sample (Plane::at, src/gpu/intra_common.h:17-21).
__device__ __forceinline__ int at(const DevPlane& s, int y, int x) {
  y = clampi(y, -s.margin, s.h + s.margin - 1);
  x = clampi(x, -s.margin, s.w + s.margin - 1);
  return s.p[(long long)y * s.stride + x];
}

// Quarter-pel sample (Plane::at_q, src/gpu/intra_common.h:23-25): phase (qy & 3) * 4 + (qx & 3) at
// the whole-pel position (y + (qy >> 2), x + (qx >> 2)).
__device__ __forceinline__ int at_q(const DevPlane& s, int y, int x, int qy, int qx) {
  const uint8_t* base = s.p + (long long)((qy & 3) * 4 + (qx & 3)) * s.phase;
  const int yy = clampi(y + (qy >> 2), -s.margin, s.h + s.margin - 1);
  const int xx = clampi(x + (qx >> 2), -s.margin, s.w + s.margin - 1);
  return base[(long long)yy * s.stride + xx];
}

// Whether the rectangle [x, x + w) x [y, y + h) lies inside the stored plane (margin included).
__device__ __forceinline__ bool inside(const DevPlane& s, int x, int y, int w, int h) {
  return x >= -s.margin && y >= -s.margin && x + w <= s.w + s.margin && y + h <= s.h + s.margin;
}

// Four bytes starting at an arbitrary byte address, from two aligned 32-bit loads.
__device__ __forceinline__ uint32_t load4(const uint8_t* p) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
  const uint32_t sh = (uint32_t)(a & 3) * 8;
  const uint32_t lo = __ldg(w);
  if (sh == 0) return lo;
  return __funnelshift_r(lo, __ldg(w + 1), sh);
}

// The same, both words always loaded (planes have slack behind their last row).
__device__ __forceinline__ uint32_t load4_pair(const uint8_t* p) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
  return __funnelshift_r(__ldg(w), __ldg(w + 1), (uint32_t)(a & 3) * 8);
}

// Columns 0 and 2 (even) or 1 and 3 (odd) of a 4-byte row as two 16-bit lanes.
__device__ __forceinline__ uint32_t bytes_even(uint32_t w) { return __byte_perm(w, 0, 0x4240); }
__device__ __forceinline__ uint32_t bytes_odd(uint32_t w) { return __byte_perm(w, 0, 0x4341); }

// dp4a with unsigned bytes a and signed bytes b: c + sum_k a_k * b_k.
__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// Per 16-bit lane, unsigned.
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t min_u16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// The four 1-D Walsh-Hadamard basis rows of length 4 as signed bytes (column 0 in the low byte):
// (1,1,1,1), (1,-1,1,-1), (1,1,-1,-1), (1,-1,-1,1) -- the rows hadamard4x4's row butterflies form.
__device__ __forceinline__ uint32_t wh_row(int k) {
  return k == 0 ? 0x01010101u : k == 1 ? 0xFF01FF01u : k == 2 ? 0xFFFF0101u : 0x01FFFF01u;
}

// The same rows negated.
__device__ __forceinline__ uint32_t wh_row_neg(int k) {
  return k == 0 ? 0xFFFFFFFFu : k == 1 ? 0x01FF01FFu : k == 2 ? 0x0101FFFFu : 0xFF0101FFu;
}

// Row-transformed cur tile for satd4_rows: C[4k + i] = <row i of the tile, basis row k>.
__device__ __forceinline__ void wh_rows_cur(const uint32_t* c, int* C) {
#pragma unroll
  for (int k = 0; k < 4; k++)
#pragma unroll
    for (int i = 0; i < 4; i++) C[4 * k + i] = dp4a_us(c[i], wh_row(k), 0);
}

// Sum of absolute 4x4 Hadamard coefficients (hadamard4x4, src/gpu/intra_common.h:131-146) of the residual
// cur - pred of a 4x4 tile from the row-transformed cur tile C and the prediction rows p (packed bytes): each residual row coefficient is one dp4a of the prediction
// row with the negated basis row, accumulated onto cur's; the column butterflies follow, the last
// one folded with the absolute values into |x + y| + |x - y| = 2 max(|x|, |y|). The same sum of
// 16 absolute coefficients.
__device__ __forceinline__ int satd4_rows(const int* C, const uint32_t* p) {
  int sum = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t neg = wh_row_neg(k);
    const int r0 = dp4a_us(p[0], neg, C[4 * k]), r1 = dp4a_us(p[1], neg, C[4 * k + 1]);
    const int r2 = dp4a_us(p[2], neg, C[4 * k + 2]), r3 = dp4a_us(p[3], neg, C[4 * k + 3]);
    const int s01 = r0 + r1, d01 = r0 - r1, s23 = r2 + r3, d23 = r2 - r3;
    sum += max(abs(s01), abs(s23)) + max(abs(d01), abs(d23));
  }
  return 2 * sum;
}

// satd4_rows of one cur tile against two predictions p and q: (SATD of p) | (SATD of q) << 16 (each at
// most 16 x 4 x 255). The row coefficients, dp4a as there, meet as two 16-bit lanes of one integer,
// a + b * 65536, so the column butterflies run once for both; a bias of 2048 (their results stay
// within +-2040) makes the lanes clean for the packed maxima: with X = x + 2048, Y = y + 2048,
// max(|x|, |y|) + 2048 = max(max(X, Y), 4096 - min(X, Y)). 50 instructions a tile instead of 71:
// 519 G tile SATDs/s on a B200 in a loop of nothing else, against 402 (and 410 for lanes of one
// prediction's columns, 438 for PTX sad in place of the maxima).
__device__ __forceinline__ uint32_t satd4_pair(const int* C, const uint32_t* p, const uint32_t* q) {
  constexpr uint32_t B = 0x08000800u;
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t neg = wh_row_neg(k);
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; i++) r[i] = (uint32_t)(dp4a_us(q[i], neg, C[4 * k + i]) * 65536 + dp4a_us(p[i], neg, C[4 * k + i]));
    const uint32_t s01 = r[0] + r[1] + B, d01 = r[0] - r[1] + B, s23 = r[2] + r[3] + B, d23 = r[2] - r[3] + B;
    sum += max_u16x2(max_u16x2(s01, s23), 2 * B - min_u16x2(s01, s23)) + max_u16x2(max_u16x2(d01, d23), 2 * B - min_u16x2(d01, d23));
  }
  return 2 * (sum - 8 * B);
}

// The same for two cur tiles, each against its own prediction: P[4k + i] = C[4k + i] of p's tile plus
// 65536 times q's (pack_cur), which the dp4a of p's rows starts from.
__device__ __forceinline__ uint32_t satd4_two(const int* P, const uint32_t* p, const uint32_t* q) {
  constexpr uint32_t B = 0x08000800u;
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t neg = wh_row_neg(k);
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; i++) r[i] = (uint32_t)(dp4a_us(q[i], neg, 0) * 65536 + dp4a_us(p[i], neg, P[4 * k + i]));
    const uint32_t s01 = r[0] + r[1] + B, d01 = r[0] - r[1] + B, s23 = r[2] + r[3] + B, d23 = r[2] - r[3] + B;
    sum += max_u16x2(max_u16x2(s01, s23), 2 * B - min_u16x2(s01, s23)) + max_u16x2(max_u16x2(d01, d23), 2 * B - min_u16x2(d01, d23));
  }
  return 2 * (sum - 8 * B);
}

__device__ __forceinline__ int mv_x(int packed) { return (int)(short)(packed & 0xffff); }
__device__ __forceinline__ int mv_y(int packed) { return packed >> 16; }
__host__ __device__ __forceinline__ int pack_mv(int x, int y) { return (int)(((unsigned)y << 16) | ((unsigned)x & 0xffffu)); }

// ---- Superblock block geometry (src/gpu/sb_blocks.h:12-37) ----
__host__ __device__ __forceinline__ int sb_level_offset(int level) { return ((1 << (2 * level)) - 1) / 3; }

__host__ __device__ __forceinline__ void sb_block_geom(int b, int& x, int& y, int& w, int& h) {
  const int sq = b / 5, kind = b % 5;
  const int level = sq >= 21 ? 3 : sq >= 5 ? 2 : sq >= 1 ? 1 : 0;
  const int idx = sq - sb_level_offset(level), n = 1 << level, size = 64 >> level, half = size / 2;
  const int sx = (idx & (n - 1)) * size, sy = (idx >> level) * size;
  x = sx, y = sy, w = size, h = size;
  if (kind == 1 || kind == 2) h = half, y = sy + (kind == 2 ? half : 0);
  if (kind == 3 || kind == 4) w = half, x = sx + (kind == 4 ? half : 0);
}

__host__ __device__ __forceinline__ int mode_bits(int mode) { return mode == 0 ? 1 : mode < 4 ? 3 : 9; }

__host__ __device__ __forceinline__ bool compound_pair_ok(int a, int b, int nrefs) {
  const int lo = a < b ? a : b, limit = nrefs - 2 < 2 ? nrefs - 2 : 2;
  return a != b && lo <= limit;
}

}  // namespace celv2cu
