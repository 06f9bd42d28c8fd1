// intra.cu: the SATD of every candidate block under each of the 13 intra modes.
//
// Reference rules (src/gpu/intra_common.h): edge_above / edge_left (:47-56), dir_pred (:60-85),
// intra_pred (:89-118), dc_value (:120-128), block_mode_satd (:149-163). Blocks of the 64x64
// square are never intra (kMaxBlockSize 32, :39), so 420 blocks x 13 modes per superblock.
//
// A unit is a superblock, or a third or a ninth of its work where the launch has too few superblocks
// to fill the GPU (launch_intra). Per unit, one CTA:
//  1. stages the source samples around the superblock (rows and columns -1 .. 95 from its origin:
//     above-right and below-left edges reach w + h - 1 past a block) from the margin plane, which
//     already holds the clamped values, twice: by rows (px), where a block's row above is a byte
//     run, and by columns (tr), where its left column is one. The frame-edge rules (edge_above,
//     edge_left: 128 outside the frame) then need no case of their own: px's row -1 is 128 in the
//     frame's top row of superblocks, tr's column -1 in its left column, and the two corner rules
//     (A[-1] at the left edge is the sample right of it, L[-1] at the top edge the one below it)
//     are what the replicated margin holds;
//  2. sums every block's DC;
//  3. spreads the 2304 (block, 4x4 tile) items over the threads, 256 of one class a step; each
//     predicts its tile under the 13 modes and takes the Hadamards; the step's SATDs meet in shared
//     memory as halfwords, where a thread sums eight of one mode with dp2a (a shuffle chain per mode
//     and item was ~130 of an item's instructions).
// The Hadamard of a residual is the cur tile's transform minus the prediction's (linearity), so
// the cur tile is transformed once per item: its rows by dp4a against the Walsh-Hadamard basis.
// DC, V and H predictions change only 1, 4 and 4 of the 16 coefficients (a constant tile only the
// DC; equal rows only the first coefficient of each column transform; constant rows only the
// first row transform), so those three modes cost a few operations on the cur transform; the ten
// others pack their prediction rows into bytes and run the dp4a row transform two at a time (satd4_pair).
// Word-wide predictions: D45's and D135's rows are windows of two words, D67 / D203 blends of two
// 4-byte runs with one weight per row / column, in two 16-bit lanes. D113 and D157 project onto the
// row above or the left column, sample by sample; along a row every sample that lands above shares
// one weight, along a column every sample that lands left does, so a tile is at most four row
// blends and four column blends, one of them transposed and the bytes picked by a mask -- the
// per-sample form of the mixed tiles was 115 of the kernel's 271 us on a 1080p frame, its edge-run
// setup another 33. A 4x4 SATD does not change under transposition (the 2-D Hadamard of the
// transposed residual is the transposed Hadamard), so D157 and D203 come last and by columns, on the
// transform of the cur tile's columns.
// Bound by the integer pipes. 1080p KEY frame (510 superblocks) 271 -> 118 us, ten 720p frames 1,049
// -> 480 us, a 202x122 frame 140 -> 18 us against one CTA per superblock with per-block edge runs,
// per-sample z2 modes and a shuffle reduction per mode and item.
// The output is raw SATDs; the finalize stage adds lambda * bits (which depend on whether the
// frame has references, unknown when prepare() runs this ahead of its launch).
#include <algorithm>
#include <climits>

#include "kernels.h"
#include "tables.h"

namespace celv2cu {

constexpr int kIntraThreads = 256;
// px: rows -1 .. 63 (a block's row above, the cur tiles), columns -4 .. 95, 26 words a row (100 bytes
// used); tr: columns -1 .. 63, rows -4 .. 95, 25 words a column. Sample 0 sits on a word boundary in
// both. The strides keep both stores of a staged 4x4 square free of bank conflicts for a warp of
// 8 x 4 squares (4 * 26 = 8 and 4 * 25 = 4 modulo 32 banks).
constexpr int kPxStride = 104, kTrStride = 100, kStaged = 65;

// ceil(2^24 / (w + h + 2)) of a level's whole squares and of their halves (Smooth's division).
constexpr unsigned inv_den(int den) { return 0xffffffu / (unsigned)den + 1u; }
__constant__ unsigned c_inv_den[3][2] = {{inv_den(66), inv_den(50)}, {inv_den(34), inv_den(26)}, {inv_den(18), inv_den(14)}};

struct IntraSmem {
  alignas(16) uint32_t px[kStaged * kPxStride / 4 + 4];  // + slack of the two-word reads
  alignas(16) uint32_t tr[kStaged * kTrStride / 4 + 4];
  alignas(16) int acc[(kBlocks * kModes + 3) / 4 * 4];
  alignas(16) unsigned short sat[2][kModes][kIntraThreads];  // a step's SATDs (at most 16 x 4 x 255), two steps in turn
  int dc[kBlocks];
};

// Four bytes at byte index i (any alignment) of a word array: two words and a funnel shift.
__device__ __forceinline__ uint32_t lds4(const uint32_t* base, int i) {
  const uint32_t* w = base + (i >> 2);
  return __funnelshift_r(w[0], w[1], (unsigned)(i & 3) * 8);
}

// The 4-byte runs at byte indices i and i + 1 from the same two words.
__device__ __forceinline__ void lds_pair(const uint32_t* base, int i, uint32_t& a, uint32_t& b) {
  const uint32_t* w = base + (i >> 2);
  const uint32_t w0 = w[0], w1 = w[1], sh = (unsigned)(i & 3) * 8;
  a = __funnelshift_r(w0, w1, sh);
  b = __funnelshift_rc(w0, w1, sh + 8);  // a shift of 32 gives w1
}

__device__ __forceinline__ int byte_at(const uint32_t* base, int i) {
  return reinterpret_cast<const uint8_t*>(base)[i];
}

// Bits 15 and 31 of e and o spread over bytes 0, 2 and 1, 3 (prmt with the selectors' sign bits).
__device__ __forceinline__ uint32_t sign_bytes(uint32_t e, uint32_t o) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, 0xfbd9;" : "=r"(d) : "r"(e), "r"(o));
  return d;
}

// The transpose of a 4x4 byte square (rows as words).
__device__ __forceinline__ void transpose4(uint32_t* w) {
  const uint32_t a = __byte_perm(w[0], w[1], 0x5140), b = __byte_perm(w[2], w[3], 0x5140);
  const uint32_t c = __byte_perm(w[0], w[1], 0x7362), d = __byte_perm(w[2], w[3], 0x7362);
  w[0] = __byte_perm(a, b, 0x5410), w[1] = __byte_perm(a, b, 0x7632);
  w[2] = __byte_perm(c, d, 0x5410), w[3] = __byte_perm(c, d, 0x7632);
}

// The low n bytes (n clamped to 0 .. 4) of a word set.
__device__ __forceinline__ uint32_t low_bytes(int n) {
  n = max(0, min(4, n));
  return __funnelshift_rc(0xffffffffu, 0u, 32u - 8u * (unsigned)n);
}

// Byte order reversed (the left column is stored bottom-up).
__device__ __forceinline__ uint32_t rev4(uint32_t v) { return __byte_perm(v, 0, 0x0123); }

// Per byte (p0 * (32 - sh) + p1 * sh + 16) >> 5 -- the directional modes' blend of four samples at
// once: bytes 0 / 2 and 1 / 3 as two 16-bit lanes (at most 255 * 32 + 16 per lane, so no lane
// carries into the next).
__device__ __forceinline__ uint32_t blend4(uint32_t p0, uint32_t p1, int sh) {
  const uint32_t a = (uint32_t)(32 - sh), b = (uint32_t)sh;
  const uint32_t e = ((p0 & 0x00ff00ffu) * a + (p1 & 0x00ff00ffu) * b + 0x00100010u) >> 5;
  const uint32_t o = (((p0 >> 8) & 0x00ff00ffu) * a + ((p1 >> 8) & 0x00ff00ffu) * b + 0x00100010u) >> 5;
  return (e & 0x00ff00ffu) | ((o & 0x00ff00ffu) << 8);
}

// Four predicted samples (0..255) as the bytes of one word, sample 0 in the low byte.
__device__ __forceinline__ uint32_t pack_row(int a, int b, int c, int d) {
  return (uint32_t)a | (uint32_t)b << 8 | (uint32_t)c << 16 | (uint32_t)d << 24;
}

// The z2 modes (dir_pred, intra_common.h): a sample at (ii, jj) of the block projects onto the row
// above at px = 64 jj - (ii + 1) dx quarter-64ths, and is taken there while px >= -64, else from
// the left column at py = 64 ii - (jj + 1) dy (never before L[-1] where it is taken). For a row the
// weight (px & 63) >> 1 is the same at every column and the run moves a sample per column; for a
// column likewise with py. z2_above: row ii's four samples from column c0 on; z2_left: column jj's
// from row r0 on; a, l: the byte index of A[0] in px, of L[0] in tr. Runs that reach before index
// -4 hold no sample that is taken, so the clamp only keeps the reads in range.
__device__ __forceinline__ uint32_t z2_above(const uint32_t* px, int a, int c0, int ii, int dx) {
  const int p = (c0 << 6) - (ii + 1) * dx;
  uint32_t w0, w1;
  lds_pair(px, a + max(p >> 6, -4), w0, w1);
  return blend4(w0, w1, (p & 63) >> 1);
}
__device__ __forceinline__ uint32_t z2_left(const uint32_t* tr, int l, int r0, int jj, int dy) {
  const int p = (r0 << 6) - (jj + 1) * dy;
  uint32_t w0, w1;
  lds_pair(tr, l + max(p >> 6, -4), w0, w1);
  return blend4(w0, w1, (p & 63) >> 1);
}

// parts: units per superblock (1, 3 or 9): part p of 3 is block level 1 + p, part p of 9 a third of
// a level's items (its whole squares, the halves of its first and of its last squares).
__global__ void __launch_bounds__(kIntraThreads, 4) k_intra(const FrameJob* __restrict__ jobs, WorkList w, int parts) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  IntraSmem& S = *reinterpret_cast<IntraSmem*>(smem_raw);
  __shared__ int unit_slot[2];
  const int tid = threadIdx.x;
  int unit, iter = 0;
  while (take_unit(w, unit, iter, unit_slot)) {
  const int jb = part_of(w, unit);
  const FrameJob& job = jobs[w.part[jb].job];
  const int u = unit - w.prefix[jb], usb = u / parts, part = u - usb * parts, sb = w.part[jb].sb0 + usb;
  const int sby = sb / job.sb_cols, sbx = sb - sby * job.sb_cols;
  const unsigned keep = keep_mask(job, sb);
  if (!(keep & CELV2_KEEP_INTRA)) continue;  // intra pruned for this superblock
  const int ox = sbx * 64, oy = sby * 64;
  const DevPlane src = job.cur.lv[0];
  // this unit's items, 256 a step, and its blocks: b0 .. b1 - 1 (of a ninth: some of them)
  const int step0 = part * (9 / parts), step1 = step0 + 9 / parts;
  const int lv0 = 1 + step0 / 3, lv1 = 1 + (step1 - 1) / 3;
  const int b0 = 5 * sb_level_offset(lv0), b1 = 5 * sb_level_offset(lv1 + 1);
  // whether block b is among them
  auto mine = [&](int b) {
    if (parts < 9) return true;
    const int sq = b / 5, sub = part % 3, half = 1 << (2 * lv0 - 1);
    return (b - sq * 5 == 0) ? sub == 0 : sub == (sq - sb_level_offset(lv0) < half ? 1 : 2);
  };

  // 1. staged samples, a 4x4 square per lane, a warp takes 8 x 4 squares: four word loads inside
  //    the margin of a word-aligned plane (the engine's own planes always), else sample by sample
  {
    const int lane = tid & 31;
    const bool top = oy == 0, left = ox == 0;
    const bool words = ((reinterpret_cast<uintptr_t>(src.p) | (uintptr_t)src.stride) & 3) == 0;
    for (int t = tid >> 5; t < 28; t += kIntraThreads / 32) {
      const int xb = (t & 3) * 8 + (lane & 7), yb = (t >> 2) * 4 + (lane >> 3);
      // px needs rows up to 63 (yb <= 16), tr columns up to 63 (xb <= 16)
      if (xb > 24 || yb > 24 || (xb > 16 && yb > 16)) continue;
      const int x = ox + 4 * xb - 4, y = oy + 4 * yb - 4;
      uint32_t q[4];
      if (words && inside(src, x, y, 4, 4)) {
        const uint8_t* g = src.p + (long long)y * src.stride + x;
#pragma unroll
        for (int k = 0; k < 4; k++) q[k] = __ldg(reinterpret_cast<const uint32_t*>(g + (long long)k * src.stride));
      } else {
#pragma unroll
        for (int k = 0; k < 4; k++)
          q[k] = pack_row(at(src, y + k, x), at(src, y + k, x + 1), at(src, y + k, x + 2), at(src, y + k, x + 3));
      }
      if (yb <= 16) {
#pragma unroll
        for (int k = 0; k < 4; k++)  // row 4 yb - 4 + k
          if (yb > 0 || k == 3) S.px[(4 * yb - 3 + k) * (kPxStride / 4) + xb] = top && yb == 0 ? 0x80808080u : q[k];
      }
      if (xb <= 16) {
        transpose4(q);
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (xb > 0 || k == 3) S.tr[(4 * xb - 3 + k) * (kTrStride / 4) + yb] = left && xb == 0 ? 0x80808080u : q[k];
      }
    }
  }
  for (int e = tid; e < (int)(sizeof S.acc / 16); e += kIntraThreads) reinterpret_cast<int4*>(S.acc)[e] = make_int4(0, 0, 0, 0);
  __syncthreads();
  // 2. DC values (dc_value) per block
  for (int b = b0 + tid; b < b1; b += kIntraThreads) {
    if (!mine(b)) continue;
    int x, y, bw, bh;
    sb_block_geom(b, x, y, bw, bh);
    const bool top = oy + y == 0, lft = ox + x == 0;
    const uint32_t* A = S.px + (y * kPxStride + 4 + x) / 4;
    const uint32_t* L = S.tr + (x * kTrStride + 4 + y) / 4;
    int sum = 0, cnt = 0;
    if (!top) {
      for (int j = 0; j < bw / 4; j++) sum = dp4a_us(A[j], 0x01010101u, sum);
      cnt += bw;
    }
    if (!lft) {
      for (int i = 0; i < bh / 4; i++) sum = dp4a_us(L[i], 0x01010101u, sum);
      cnt += bh;
    }
    S.dc[b] = cnt ? (sum + cnt / 2) / cnt : 128;
  }
  __syncthreads();

  // 3. (block, tile) items: 13 predictions + Hadamards per tile, segment sums per block
  int buf = 0;
  for (int st = step0; st < step1; st++) {
    // the items of one CTA-wide step belong to one block level
    if (!(keep & CELV2_KEEP_LEVEL(1 + st / 3))) continue;
    // the step's class of items (uniform): squares of a level, or their halves; 2 ^ lwt tiles a block
    const int level = 1 + st / 3, sub = st - st / 3 * 3;
    const int lwt = 2 * (4 - level) - (sub != 0), lgs = 6 - level;
    const int k = (sub == 2 ? kIntraThreads : 0) + tid, blk = k >> lwt, t = k & ((1 << lwt) - 1);
    const int idx = sub ? blk >> 2 : blk, kind = sub ? 1 + (blk & 3) : 0;
    const int b = (sb_level_offset(level) + idx) * 5 + kind;
    const int lgw = lgs - (kind >= 3), lgh = lgs - (kind == 1 || kind == 2);  // the block's size, log2
    const int bw = 1 << lgw, bh = 1 << lgh;
    const int x = ((idx & ((1 << level) - 1)) << lgs) + (kind == 4 ? bw : 0);
    const int y = ((idx >> level) << lgs) + (kind == 2 ? bh : 0);
    const int c0 = (t & ((bw >> 2) - 1)) * 4, r0 = (t >> (lgw - 2)) * 4;  // the tile's origin inside the block
    const int tx = (x + c0) >> 2, ty = (y + r0) >> 2;
    const int a = y * kPxStride + 4 + x;  // A[k] at byte a + k of px, k >= -1
    const int l = x * kTrStride + 4 + y;  // L[k] at byte l + k of tr, k >= -1
    unsigned short* sat = S.sat[buf][0] + tid;  // mode m's SATD of this item at sat[256 m]
    int C[16];  // the cur tile, row-transformed
    {
      uint32_t cw[4];
#pragma unroll
      for (int i = 0; i < 4; i++) cw[i] = S.px[(ty * 4 + i + 1) * (kPxStride / 4) + tx + 1];
      wh_rows_cur(cw, C);
    }
    const uint32_t a4 = S.px[(a + c0) >> 2], l4 = S.tr[(l + r0) >> 2];  // A[c0 ..], L[r0 ..]
    {
      // DC, V, H: per basis row k the column transform's outputs; T the sum of all 16 absolute
      // coefficients (the cur tile's SATD), Hk0 the first outputs and V0 their absolute sum, U0 the
      // absolute sum of row k = 0's
      int Hk0[4], T = 0, V0 = 0, U0 = 0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int s01 = C[4 * k] + C[4 * k + 1], d01 = C[4 * k] - C[4 * k + 1];
        const int s23 = C[4 * k + 2] + C[4 * k + 3], d23 = C[4 * k + 2] - C[4 * k + 3];
        const int t = abs(s01 + s23) + abs(s01 - s23) + abs(d01 + d23) + abs(d01 - d23);
        T += t, Hk0[k] = s01 + s23, V0 += abs(s01 + s23);
        if (k == 0) U0 = t;
      }
      // DC: only coefficient (0, 0) moves, by 16 v
      const int dc = T - abs(Hk0[0]) + abs(Hk0[0] - 16 * S.dc[b]);
      // V: every row is the above row; the first output of each column transform moves by 4 a_k
      int v = T - V0;
#pragma unroll
      for (int k = 0; k < 4; k++) v += abs(Hk0[k] - 4 * dp4a_us(a4, wh_row(k), 0));
      // H: row i is the constant l_i; row transform k = 0 moves by 4 l_i
      const int r0v = C[0] - 4 * (int)(l4 & 255), r1v = C[1] - 4 * (int)((l4 >> 8) & 255);
      const int r2v = C[2] - 4 * (int)((l4 >> 16) & 255), r3v = C[3] - 4 * (int)(l4 >> 24);
      const int s01 = r0v + r1v, d01 = r0v - r1v, s23 = r2v + r3v, d23 = r2v - r3v;
      const int h = T - U0 + abs(s01 + s23) + abs(s01 - s23) + abs(d01 + d23) + abs(d01 - d23);
      sat[0] = (unsigned short)dc, sat[kIntraThreads] = (unsigned short)v, sat[2 * kIntraThreads] = (unsigned short)h;
    }
    // the ten other modes two at a time (satd4_pair)
    uint32_t pa[4] = {}, pb[4] = {};
    auto both = [&](int m) {
      const uint32_t v = satd4_pair(C, pa, pb);
      sat[m * kIntraThreads] = (unsigned short)v, sat[(m + 1) * kIntraThreads] = (unsigned short)(v >> 16);
    };
    // Smooth: bilinear blend of above, left, top-right and bottom-left, columns 0 / 2 and
    // 1 / 3 as two 16-bit lanes (a sum is at most 255 * 66 + 33)
    if (keep & CELV2_KEEP_MODE(3)) {
      const int den = bw + bh + 2;
      // n / den as the top byte of n * ceil(2^24 / den): exact while n * (den * ceil(2^24 / den) -
      // 2^24) < 2^24 (division by invariant integers using multiplication, Granlund and Montgomery
      // 1994), and the product stays below 2^32; here n <= 255 den + den / 2 and den <= 66
      const unsigned magic = c_inv_den[level - 1][sub != 0];
      const int tr = byte_at(S.px, a + bw - 1), bl = byte_at(S.tr, l + bh - 1);
      const uint32_t ae = a4 & 0x00ff00ffu, ao = (a4 >> 8) & 0x00ff00ffu;
      const uint32_t we = (uint32_t)(bw - c0) | (uint32_t)(bw - 2 - c0) << 16, wo = we - 0x00010001u;
      const uint32_t te = ((uint32_t)(c0 + 1) | (uint32_t)(c0 + 3) << 16) * (uint32_t)tr + (uint32_t)(den / 2) * 0x00010001u;
      const uint32_t to = te + (uint32_t)tr * 0x00010001u;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint32_t ii = (uint32_t)(r0 + i), li = (l4 >> (8 * i)) & 255u, wa = (uint32_t)bh - ii;
        const uint32_t add = (ii + 1) * (uint32_t)bl * 0x00010001u;
        const uint32_t e = ae * wa + we * li + te + add, o = ao * wa + wo * li + to + add;
        const uint32_t q0 = (e & 0xffffu) * magic, q2 = (e >> 16) * magic;
        const uint32_t q1 = (o & 0xffffu) * magic, q3 = (o >> 16) * magic;
        pa[i] = __byte_perm(__byte_perm(q0, q1, 0x0073), __byte_perm(q2, q3, 0x0073), 0x5410);
      }
    }
    // SmoothV (h a power of two, the numerator non-negative): two 16-bit lanes at once
    if (keep & CELV2_KEEP_MODE(4)) {
      const uint32_t ae = a4 & 0x00ff00ffu, ao = (a4 >> 8) & 0x00ff00ffu;
      const int bl = byte_at(S.tr, l + bh - 1);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int ii = r0 + i;
        const uint32_t wa = (uint32_t)(bh - 1 - ii), add = (uint32_t)((ii + 1) * bl + bh / 2) * 0x00010001u;
        const uint32_t e = ((ae * wa + add) >> lgh) & 0x00ff00ffu, o = ((ao * wa + add) >> lgh) & 0x00ff00ffu;
        pb[i] = e | o << 8;
      }
    }
    if (keep & (CELV2_KEEP_MODE(3) | CELV2_KEEP_MODE(4))) both(3);
    // SmoothH: per row the left sample, per column weights (bw - 1 - jj, jj + 1)
    if (keep & CELV2_KEEP_MODE(5)) {
      const int tr = byte_at(S.px, a + bw - 1);
      const uint32_t we = (uint32_t)(bw - 1 - c0) | (uint32_t)(bw - 3 - c0) << 16;
      const uint32_t wo = (uint32_t)(bw - 2 - c0) | (uint32_t)(bw - 4 - c0) << 16;
      const uint32_t te = ((uint32_t)(c0 + 1) | (uint32_t)(c0 + 3) << 16) * (uint32_t)tr + (uint32_t)(bw / 2) * 0x00010001u;
      const uint32_t to = ((uint32_t)(c0 + 2) | (uint32_t)(c0 + 4) << 16) * (uint32_t)tr + (uint32_t)(bw / 2) * 0x00010001u;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint32_t li = (l4 >> (8 * i)) & 255u;
        const uint32_t e = ((li * we + te) >> lgw) & 0x00ff00ffu, o = ((li * wo + to) >> lgw) & 0x00ff00ffu;
        pa[i] = e | o << 8;
      }
    }
    // Paeth, four samples at a time. With u = A - tl and v = L - tl the three distances are pl = |u|,
    // pa = |v| and ptl = |u + v|: where u and v differ in sign that is ||u| - |v||, else it is at
    // least both others (255 in its place). A byte compare x <= y is bit 15 of 0x8000 + y - x in
    // 16-bit lanes, spread over the byte by prmt's sign mode
    if (keep & CELV2_KEEP_MODE(6)) {
      const uint32_t tl4 = (uint32_t)byte_at(S.px, a - 1) * 0x01010101u;
      // bytes 0 / 2 and 1 / 3 of w as lanes; le4: the bytes' mask of x <= y, y's lanes carrying 0x8000
      auto ev = [](uint32_t w) { return w & 0x00ff00ffu; };
      auto od = [](uint32_t w) { return (w >> 8) & 0x00ff00ffu; };
      auto spread = [](uint32_t e, uint32_t o) { return sign_bytes(e, o); };
      const uint32_t te = ev(tl4), h = 0x80008000u;
      const uint32_t su = spread((ev(a4) | h) - te, (od(a4) | h) - te), sv = spread((ev(l4) | h) - te, (od(l4) | h) - te);
      const uint32_t pl = __vabsdiffu4(a4, tl4), pa4 = __vabsdiffu4(l4, tl4), ple = ev(pl), plo = od(pl);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint32_t rep = 0x1111u * (uint32_t)i, li = __byte_perm(l4, 0, rep), pa = __byte_perm(pa4, 0, rep);
        const uint32_t d = __vabsdiffu4(pl, pa) | ~(su ^ __byte_perm(sv, 0, rep));
        const uint32_t pae = ev(pa), de = ev(d) | h, dd = od(d) | h;
        const uint32_t ml = spread(((pae | h) - ple) & (de - ple), ((pae | h) - plo) & (dd - plo));
        const uint32_t ma = spread(de - pae, dd - pae);
        pb[i] = (li & ml) | (~ml & ((a4 & ma) | (tl4 & ~ma)));
      }
    }
    if (keep & (CELV2_KEEP_MODE(5) | CELV2_KEEP_MODE(6))) both(5);
    // D45: derivative 64, no blend: row i is A[r0 + i + 1 + c0 ..] (never past A[w + h - 1])
    if (keep & CELV2_KEEP_MODE(7)) {
      const uint32_t* q = S.px + ((a + r0 + c0) >> 2);
      const uint32_t w0 = q[0], w1 = q[1];
#pragma unroll
      for (int i = 0; i < 3; i++) pa[i] = __funnelshift_r(w0, w1, 8 * (i + 1));
      pa[3] = w1;
    }
    // D67: derivative 27, one weight per row
    if (keep & CELV2_KEEP_MODE(8)) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int pos = (r0 + i + 1) * 27;
        uint32_t w0, w1;
        lds_pair(S.px, a + (pos >> 6) + c0, w0, w1);
        pb[i] = blend4(w0, w1, (pos & 63) >> 1);
      }
    }
    if (keep & (CELV2_KEEP_MODE(7) | CELV2_KEEP_MODE(8))) both(7);
    // D113, by rows: row ii is taken from the left below column ((ii + 1) * 27 - 1) >> 6
    if (keep & CELV2_KEEP_MODE(9)) {
      if (((r0 + 1) * 27 - 1) >> 6 < c0 + 4) {
#pragma unroll
        for (int i = 0; i < 4; i++) pa[i] = z2_above(S.px, a, c0, r0 + i, 27);
      }
      if (((r0 + 4) * 27 - 1) >> 6 > c0) {
        uint32_t q[4];
#pragma unroll
        for (int j = 0; j < 4; j++) q[j] = z2_left(S.tr, l, r0, c0 + j, 151);
        transpose4(q);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const uint32_t k = low_bytes((((r0 + i + 1) * 27 - 1) >> 6) - c0);
          pa[i] = (q[i] & k) | (pa[i] & ~k);
        }
      }
    }
    // D135: derivatives 64 / 64, no blend: row i is the run of L reversed, A[-1], A from
    // A[c0 - r0 - 1 - i] on, so the tile's rows are windows of two words of it
    if (keep & CELV2_KEEP_MODE(10)) {
      const int d = c0 - r0;  // a multiple of 4
      uint32_t q[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int v = d - 4 + 4 * h;  // the run's bytes v .. v + 3
        if (v >= 0) {
          q[h] = S.px[(a + v) >> 2];
        } else {  // L[-v - 2] down to L[-v - 5]; A[-1] where v + 3 is -1
          q[h] = rev4(lds4(S.tr, l - v - 5));
          if (v == -4) q[h] = __byte_perm(q[h], (uint32_t)byte_at(S.px, a - 1), 0x4210);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++) pb[i] = __funnelshift_r(q[0], q[1], 24 - 8 * i);
    }
    if (keep & (CELV2_KEEP_MODE(9) | CELV2_KEEP_MODE(10))) both(9);
    if (keep & (CELV2_KEEP_MODE(11) | CELV2_KEEP_MODE(12))) {
      // D157 and D203 predict columns: from here on C is the transform of the cur tile's columns
      uint32_t col[4];
#pragma unroll
      for (int j = 0; j < 4; j++) col[j] = S.tr[(tx * 4 + j + 1) * (kTrStride / 4) + ty + 1];
      wh_rows_cur(col, C);
    }
    // D157, by columns: column jj is taken from above in rows below 64 (jj + 1) / 151
    if (keep & CELV2_KEEP_MODE(11)) {
      if (64 * (c0 + 1) / 151 < r0 + 4) {
#pragma unroll
        for (int j = 0; j < 4; j++) pa[j] = z2_left(S.tr, l, r0, c0 + j, 27);
      }
      if (64 * (c0 + 4) / 151 > r0) {
        uint32_t q[4];
#pragma unroll
        for (int i = 0; i < 4; i++) q[i] = z2_above(S.px, a, c0, r0 + i, 151);
        transpose4(q);
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const uint32_t k = low_bytes(64 * (c0 + j + 1) / 151 - r0);
          pa[j] = (q[j] & k) | (pa[j] & ~k);
        }
      }
    }
    // z3: D203 (derivative 27), by columns from the column left
    if (keep & CELV2_KEEP_MODE(12)) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int pos = (c0 + j + 1) * 27;
        uint32_t w0, w1;
        lds_pair(S.tr, l + (pos >> 6) + r0, w0, w1);
        pb[j] = blend4(w0, w1, (pos & 63) >> 1);
      }
    }
    if (keep & (CELV2_KEEP_MODE(11) | CELV2_KEEP_MODE(12))) both(11);
    __syncthreads();  // the step's SATDs; the other buffer's readers are past the step before
    // a block's sums: thread (mode, 8 items) adds their halfwords, blocks of more meet in acc
    for (int e = tid; e < kModes * (kIntraThreads / 8); e += kIntraThreads) {
      const int m = e >> 5, g = e & 31;
      if (m >= 3 && !(keep & CELV2_KEEP_MODE(m))) continue;  // nothing written: the sums stay 0
      const uint4 q = *reinterpret_cast<const uint4*>(&S.sat[buf][m][8 * g]);
      const int s0 = (int)__dp2a_lo(q.x, 0x0101u, 0u), s1 = (int)__dp2a_lo(q.y, 0x0101u, 0u);
      const int s2 = (int)__dp2a_lo(q.z, 0x0101u, 0u), s3 = (int)__dp2a_lo(q.w, 0x0101u, 0u);
      const int i0 = (sub == 2 ? kIntraThreads : 0) + 8 * g;
      // item i's block, as above
      auto acc = [&](int i) {
        const int bl = i >> lwt;
        return S.acc + ((sb_level_offset(level) + (sub ? bl >> 2 : bl)) * 5 + (sub ? 1 + (bl & 3) : 0)) * kModes + m;
      };
      if (lwt == 1) {
        *acc(i0) = s0, *acc(i0 + 2) = s1, *acc(i0 + 4) = s2, *acc(i0 + 6) = s3;
      } else if (lwt == 2) {
        *acc(i0) = s0 + s1, *acc(i0 + 4) = s2 + s3;
      } else if (lwt == 3) {
        *acc(i0) = s0 + s1 + s2 + s3;
      } else {
        atomicAdd(acc(i0), s0 + s1 + s2 + s3);
      }
    }
    buf ^= 1;
  }
  __syncthreads();
  int* out = const_cast<int*>(job.intra) + (long long)sb * kBlocks * kModes;
  // mode by mode, as the finalize stage's blocks read them
  for (int bl = b0 + tid; bl < b1; bl += kIntraThreads)
    if (parts < 9 || mine(bl)) {
#pragma unroll
      for (int m = 0; m < kModes; m++) out[m * kBlocks + bl] = S.acc[bl * kModes + m];
    }
  }  // units
}

// Units per superblock. A whole superblock is some 50 us of one CTA's time, so a launch of fewer
// superblocks than the GPU has resident CTAs (592) takes at least that however small it is: thirds
// while there are at most that many, ninths while those still run all at once. Each unit stages the
// samples again, so more parts cost where the GPU is full anyway. us on a B200 with 1 / 3 / 9 parts
// (stage events, ~7 us of them the events): 28 superblocks 48 / 23 / 21, 60: 52 / 35 / 31, 135:
// 52 / 43 / 54, 510: 128 / 119 / 148, 920: 208 / 211 / 281, 2400: 480 / 491 / 632.
static int intra_parts(int sbs, int full) { return sbs * 9 <= full ? 9 : sbs <= full ? 3 : 1; }

void launch_intra(const FrameJob* jobs, const WorkList& w, cudaStream_t st) {
  const int sbs = w.prefix[w.nparts];
  if (sbs <= 0) return;
  const int full = persistent_grid((const void*)k_intra, kIntraThreads, sizeof(IntraSmem), INT_MAX);
  const int parts = intra_parts(sbs, full), units = sbs * parts;
  WorkList wp = w;
  for (int j = 1; j <= w.nparts; j++) wp.prefix[j] = w.prefix[j] * parts;
  k_intra<<<w.queue ? std::min(full, units) : units, kIntraThreads, sizeof(IntraSmem), st>>>(jobs, wp, parts);
}

cudaError_t intra_attributes() {
  const cudaError_t e = cudaFuncSetAttribute(k_intra, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(IntraSmem));
  if (e == cudaSuccess) persistent_grid((const void*)k_intra, kIntraThreads, sizeof(IntraSmem), 1);  // fills the grid cache
  return e;
}

}  // namespace celv2cu
