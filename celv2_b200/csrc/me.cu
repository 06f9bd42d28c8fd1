// me.cu: hierarchical integer motion search, one pyramid level per launch, all references and
// all frames of a batch together.
//
// Reference rules (src/gpu/inter_common.h): sad8 (:96-104), me_search (:108-119), satd8_q
// (:122-133), me_refine (:141-154), me_cell (:162-193); driven level by level, coarsest first,
// as src/gpu/cpu_engine.cpp:68-83 does.
//
// One CTA per 30 (15, 7) consecutive 8x8 cells of one (job, reference):
//  A. the cells' cur blocks are staged in shared memory; one thread per (cell, predictor centre)
//     computes the six centre SADs;
//  B. one thread per cell replays the reference's sequential choice of the two best distinct
//     centres (a best centre of SAD below kMePenalty is the result: nothing else can cost less), and
//     the searches (one or two per cell) get their 24 x 32-byte reference windows staged in shared
//     memory, a warp a search, by aligned 8-byte copies;
//  C. one thread per (search, dx) column slides down the window's 24 rows: each row's 8 bytes at
//     column dx are loaded once (two funnel shifts of three words) and feed, with vabsdiff4, every
//     one of the 17 dy accumulators whose 8x8 block covers that row -- 24 row loads instead of
//     17 x 8 per column. The column's best (cost << 9 | raster index) goes to a shared atomicMin,
//     which yields the reference's first strict minimum in dy-major order;
// Level 0's quarter-pel refinement is its own kernel (k_me_refine).
// Integer ALU bound: 289 x 16 byte-SIMD absolute-difference accumulates per searched centre. Level 0 of
// five 1080p frames of 7 references 1.49 -> 1.25 ms (natural-like) and 0.50 -> 0.43 ms (animation-like,
// 1.50 before the cells that need no search had none) with the windows staged a warp a search instead of
// finding search, cell and place again for every 8 bytes; CTAs of 128 threads and 15 cells 1.62, the
// next unit asked for ahead 1.28, the cells' places found per thread instead of behind a barrier 1.28.
#include <climits>

#include "kernels.h"

namespace celv2cu {

constexpr int kMeThreads = 256;
constexpr int kWinRows = 24, kWinWords = 8;    // a window row: 32 bytes from an 8-byte boundary
constexpr int kWinStride = kWinRows * kWinWords + 8;  // +8 words: neighbouring windows use other banks
// A merged search: the two centres of a cell at most 2 apart in x and y searched as one union
// window of at most 19 x 19 positions (instead of two 17 x 17): 26 rows of 40 bytes, in the space
// of two windows.
constexpr int kMergeMax = 2, kUnion = 17 + kMergeMax, kMWinRows = kUnion + 7, kMWinWords = 10;
static_assert(kMWinRows * kMWinWords <= 2 * kWinStride, "a merged window fits two windows' space");

// Shared state of a CTA of CELLS cells (15 or 30 as configured, the autotuner picking per level; 7 in
// small launches, see me_level_cells). Nearly every cell searches two centres, so a CTA's
// search phase has about 2 x 17 x CELLS (search, column) items: 30 and 15 cells make 1,020 and 510,
// four and two nearly full rounds of 256 threads (32 and 16 cells left a last round 25% and 12%
// full).
template <int CELLS>
struct MeSmem {
  static constexpr int kSearches = 2 * CELLS;  // at most two centres per cell
  alignas(16) uint32_t cur[CELLS][16];
  int bx[CELLS], by[CELLS];  // the cells' blocks (samples)
  int csad[CELLS][6];
  int ccx[CELLS][6], ccy[CELLS][6];
  int scell[kSearches], sx[kSearches], sy[kSearches];
  // the window: its first staged sample (column on an 8-byte boundary, row), the search's first column
  // in it, whether it lies inside the margin
  int wx[kSearches], wy[kSearches], soff[kSearches], wok[kSearches];
  unsigned skey[kSearches];
  // merged searches (entries from the back of the list): the second centre and its key
  int sx2[kSearches], sy2[kSearches];
  unsigned skey2[kSearches];
  int first_search[CELLS], two[CELLS];  // two: 0 one centre, 1 two searches, 2 one merged search
  int need[CELLS];  // the cell is searched (level 0 of a pruned job: some superblock reads it)
  int nsearch, nmerged;
  alignas(16) uint32_t win[kSearches * kWinStride];
};

// An asynchronous 8-byte global -> shared copy (cp.async; both addresses 8-byte aligned).
__device__ __forceinline__ void cp_async8(void* smem_dst, const void* gsrc) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// 4 bytes of a plane at (x .. x + 3, y), clamped like Plane::at where the row leaves the margin.
__device__ __forceinline__ uint32_t row4(const DevPlane& s, int x, int y) {
  if (y >= -s.margin && y < s.h + s.margin && x >= -s.margin && x + 4 <= s.w + s.margin)
    return load4(s.p + (long long)y * s.stride + x);
  uint32_t v = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) v |= (uint32_t)at(s, y, x + k) << (8 * k);
  return v;
}

// acc + the sum of the four byte absolute differences of a and b (PTX vabsdiff4 with its add).
__device__ __forceinline__ unsigned sad4_acc(unsigned a, unsigned b, unsigned acc) {
  unsigned d;
  asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(acc));
  return d;
}

// sad8 of a cur block (shared memory) against the reference at (x, y).
__device__ __forceinline__ int sad8(const uint32_t* c, const DevPlane& ref, int x, int y) {
  unsigned s = 0;
  if (inside(ref, x, y, 8, 8)) {
    const uint8_t* p = ref.p + (long long)y * ref.stride + x;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      s = sad4_acc(c[2 * i], load4(p + (long long)i * ref.stride), s);
      s = sad4_acc(c[2 * i + 1], load4(p + (long long)i * ref.stride + 4), s);
    }
    return (int)s;
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    s = sad4_acc(c[2 * i], row4(ref, x, y + i), s);
    s = sad4_acc(c[2 * i + 1], row4(ref, x + 4, y + i), s);
  }
  return (int)s;
}

// A cell's 16 words from shared memory.
__device__ __forceinline__ void load_cur(const uint32_t* c, uint32_t* cw) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint4 v = reinterpret_cast<const uint4*>(c)[k];
    cw[4 * k] = v.x, cw[4 * k + 1] = v.y, cw[4 * k + 2] = v.z, cw[4 * k + 3] = v.w;
  }
}

// The refinement step's position n (raster 0..8 with the centre, 4, visited first).
__device__ __forceinline__ int refine_pos(int t) { return t == 0 ? 4 : (t <= 4 ? t - 1 : t); }

template <int CELLS>
__global__ void __launch_bounds__(kMeThreads, 1024 / kMeThreads) k_me_level(const FrameJob* __restrict__ jobs, WorkList w, int level) {
  constexpr int kMeCells = CELLS;
  static_assert(CELLS * 6 <= kMeThreads, "a thread per cell and centre");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MeSmem<CELLS>& S = *reinterpret_cast<MeSmem<CELLS>*>(smem_raw);
  __shared__ int unit_slot[2];
  const int tid = threadIdx.x;
  int unit, iter = 0;
  while (take_unit(w, unit, iter, unit_slot)) {
  const int jb = part_of(w, unit);
  const FrameJob& job = jobs[w.part[jb].job];
  const int cols = job.fcols[level], rows = job.frows[level], ncell = cols * rows;
  const int groups = (ncell + kMeCells - 1) / kMeCells;
  const int u = unit - w.prefix[jb];
  const int r = u / groups, cell0 = (u - r * groups) * kMeCells;
  const int ncells = min(kMeCells, ncell - cell0);
  const DevPlane cur = job.cur.lv[level], ref = job.ref[r].lv[level];

  // ---- A. cur blocks, predictor centres and their SADs (me_cell, inter_common.h:164-186) ----
  if (tid < kMeCells) {
    const int cell = cell0 + (tid < ncells ? tid : 0), by = cell / cols, bx = cell - by * cols;
    S.bx[tid] = bx * 8, S.by[tid] = by * 8;
    S.need[tid] = tid < ncells && (level != 0 || cell_needed(job, r, bx, by));
  }
  if (tid == 0) S.nsearch = 0, S.nmerged = 0;
  __syncthreads();
  const bool top = level == kLevels - 1;
  // (a block overhangs the plane by at most 7 samples: inside the margin; rows and margins are multiples
  // of 8 bytes)
  for (int e = tid; e < kMeCells * 8; e += kMeThreads) {
    const int c = e >> 3, i = e & 7;
    const uint2 v = *reinterpret_cast<const uint2*>(cur.p + (long long)(S.by[c] + i) * cur.stride + S.bx[c]);
    S.cur[c][2 * i] = v.x, S.cur[c][2 * i + 1] = v.y;
  }
  int cx = 0, cy = 0;  // this thread's centre, of cell tid / 6 (centre 5: zero)
  if (!top && tid < kMeCells * 6) {
    const int c = tid / 6, k = tid - c * 6;
    if (k < 5 && S.need[c]) {
      const int* pf = job.field[r][level + 1];
      const int pcols = job.fcols[level + 1], prows = job.frows[level + 1];
      const int ox = k == 1 ? -1 : k == 2 ? 1 : 0, oy = k == 3 ? -1 : k == 4 ? 1 : 0;
      const int m = pf[clampi((S.by[c] >> 4) + oy, 0, prows - 1) * pcols + clampi((S.bx[c] >> 4) + ox, 0, pcols - 1)];
      cx = 2 * mv_x(m), cy = 2 * mv_y(m);
    }
  }
  __syncthreads();
  if (!top && tid < kMeCells * 6) {
    const int c = tid / 6, k = tid - c * 6;
    if (S.need[c]) {
      S.ccx[c][k] = cx, S.ccy[c][k] = cy;
      S.csad[c][k] = sad8(S.cur[c], ref, S.bx[c] + cx, S.by[c] + cy);
    }
  }
  __syncthreads();

  // ---- B. the two best distinct centres per cell, the search list ----
  if (tid < ncells && !S.need[tid]) S.first_search[tid] = -1, S.two[tid] = 0;
  if (tid < ncells && S.need[tid]) {
    const int c = tid;
    int px = 0, py = 0, px2 = 0, py2 = 0;
    bool two = false;
    int best = 0x7fffffff;
    if (!top) {
      int second = 0x7fffffff;
      for (int k = 0; k < 6; k++) {
        const int x = S.ccx[c][k], y = S.ccy[c][k], v = S.csad[c][k];
        if ((k > 0 && x == px && y == py) || (two && x == px2 && y == py2)) continue;
        if (v < best) {
          if (k > 0) second = best, px2 = px, py2 = py, two = true;
          best = v, px = x, py = y;
        } else if (v < second) {
          second = v, px2 = x, py2 = y, two = true;
        }
      }
    }
    // search s's window of `bytes` x `rows` around (x, y) - kMeRange
    auto window = [&](int s, int x, int y, int bytes, int rows_) {
      const int x0 = S.bx[c] + x - kMeRange, wx = x0 & ~7, wy = S.by[c] + y - kMeRange;
      S.wx[s] = wx, S.wy[s] = wy, S.soff[s] = x0 - wx, S.wok[s] = inside(ref, wx, wy, bytes, rows_);
    };
    if (best < kMePenalty) {
      // nothing to search: at the best centre the cost is its SAD alone, every other position of its
      // window pays at least kMePenalty, and so does every one of the second centre's but that centre
      // itself, whose SAD is no less -- the usual case on flat content, where a SAD is 0
      S.first_search[c] = -1, S.two[c] = 0;
      S.ccx[c][0] = px, S.ccy[c][0] = py;
    } else if (two && abs(px - px2) <= kMergeMax && abs(py - py2) <= kMergeMax) {
      // one union window for both centres, its entry from the back of the list
      const int s = MeSmem<CELLS>::kSearches - 1 - atomicAdd(&S.nmerged, 1);
      S.first_search[c] = s, S.two[c] = 2;
      S.scell[s] = c, S.sx[s] = px, S.sy[s] = py, S.sx2[s] = px2, S.sy2[s] = py2;
      window(s, min(px, px2), min(py, py2), 4 * kMWinWords, kMWinRows);
      S.skey[s] = S.skey2[s] = 0xffffffffu;
    } else {
      const int s0 = atomicAdd(&S.nsearch, two ? 2 : 1);
      S.first_search[c] = s0, S.two[c] = two;
      for (int k = 0; k < (two ? 2 : 1); k++) {
        const int x = k ? px2 : px, y = k ? py2 : py;
        S.scell[s0 + k] = c, S.sx[s0 + k] = x, S.sy[s0 + k] = y;
        window(s0 + k, x, y, 4 * kWinWords, kWinRows);
        S.skey[s0 + k] = 0xffffffffu;
      }
    }
  }
  __syncthreads();
  const int nsearch = S.nsearch, nmerged = S.nmerged;
  // windows, a warp a search: 24 rows of 32 bytes, a lane an 8-byte column of every eighth row; inside
  // the margin as asynchronous copies (all in flight at once: one memory latency for the whole staging),
  // else word by word with clamping. Plane rows start 8-byte aligned, and so do the window rows in
  // shared memory. (With the search, its cell and its place found again for every 8 bytes this loop was
  // a fifth of the kernel's instructions.)
  const int lane = tid & 31;
  for (int s = tid >> 5; s < nsearch; s += kMeThreads / 32) {
    const int rr = lane >> 2, qd = lane & 3, wx = S.wx[s] + 8 * qd, wy = S.wy[s] + rr;
    uint32_t* dst = S.win + s * kWinStride + rr * kWinWords + 2 * qd;
    if (S.wok[s]) {
      const uint8_t* g = ref.p + (long long)wy * ref.stride + wx;
#pragma unroll
      for (int i = 0; i < kWinRows / 8; i++) cp_async8(dst + 8 * i * kWinWords, g + (long long)(8 * i) * ref.stride);
    } else {
      for (int i = 0; i < kWinRows; i += 8)
        dst[i * kWinWords] = row4(ref, wx, wy + i), dst[i * kWinWords + 1] = row4(ref, wx + 4, wy + i);
    }
  }
  // merged windows: 26 rows of 40 bytes, merged search m (entry kSearches - 1 - m) in the window space of
  // entries kSearches - 2 - 2m, +1; five columns of every sixth row in 30 lanes
  const int mr = lane / 5, mq = lane - mr * 5;
  for (int m = tid >> 5; m < nmerged; m += kMeThreads / 32) {
    const int s = MeSmem<CELLS>::kSearches - 1 - m, wx = S.wx[s] + 8 * mq, wy = S.wy[s];
    uint32_t* dst = S.win + (MeSmem<CELLS>::kSearches - 2 - 2 * m) * kWinStride + 2 * mq;
    const bool ok = S.wok[s];
    if (mr < 6)
      for (int rr = mr; rr < kMWinRows; rr += 6) {
        if (ok)
          cp_async8(dst + rr * kMWinWords, ref.p + (long long)(wy + rr) * ref.stride + wx);
        else
          dst[rr * kMWinWords] = row4(ref, wx, wy + rr), dst[rr * kMWinWords + 1] = row4(ref, wx + 4, wy + rr);
      }
  }
  cp_async_wait_all();
  __syncthreads();

  // ---- C. +-8 search (me_search, inter_common.h:108-119): a thread per (search, dx), then a
  //      thread per (merged search, union column), in one loop so the two kinds share rounds ----
  const int nplain = nsearch * 17, nitems = nplain + nmerged * kUnion;
  for (int item = tid; item < nitems; item += kMeThreads) {
    if (item < nplain) {
    const int s = item / 17, dx = item - s * 17;
    uint32_t cw[16];
    load_cur(S.cur[S.scell[s]], cw);
    const int b = S.soff[s] + dx, wi = b >> 2;
    const unsigned sh = (unsigned)(b & 3) * 8;
    const uint32_t* wr = S.win + s * kWinStride + wi;
    unsigned acc[17];
#pragma unroll
    for (int k = 0; k < 17; k++) acc[k] = 0;
#pragma unroll
    for (int rr = 0; rr < kWinRows; rr++) {
      const uint32_t u0 = wr[rr * kWinWords], u1 = wr[rr * kWinWords + 1], u2 = wr[rr * kWinWords + 2];
      const uint32_t w0 = __funnelshift_r(u0, u1, sh), w1 = __funnelshift_r(u1, u2, sh);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int dy = rr - i;
        if (dy >= 0 && dy <= 16) acc[dy] = sad4_acc(cw[2 * i + 1], w1, sad4_acc(cw[2 * i], w0, acc[dy]));
      }
    }
    // the column's least (cost << 5 | dy): along a column raster order is dy's
    unsigned best = 0xffffffffu;
#pragma unroll
    for (int dy = 0; dy < 17; dy++) best = min(best, (acc[dy] << 5) + (unsigned)(kMePenalty * (dy < kMeRange ? kMeRange - dy : dy - kMeRange) * 32 + dy));
    const unsigned pen_x = kMePenalty * abs(dx - kMeRange);
    atomicMin(&S.skey[s], ((best >> 5) + pen_x) << 9 | ((best & 31) * 17 + dx));
    } else {
    // merged searches: a thread per union column (at most 19); every union position's SAD is the
    // same for both centres, and each centre takes its own penalty and raster index -- the same
    // keys as its own 17 x 17 search, so the same first strict minimum. All 19 union rows are
    // summed (fixed trip counts; rows past the centres' union are never keyed)
    const int m = (item - nplain) / kUnion, du = item - nplain - m * kUnion, s = MeSmem<CELLS>::kSearches - 1 - m;
    const int cx1 = S.sx[s], cy1 = S.sy[s], cx2 = S.sx2[s], cy2 = S.sy2[s];
    const int ux = min(cx1, cx2), uy = min(cy1, cy2);  // union position 0 = centre offset -8
    if (du >= 17 + abs(cx1 - cx2)) continue;
    uint32_t cw[16];
    load_cur(S.cur[S.scell[s]], cw);
    const int b = S.soff[s] + du, wi = b >> 2;
    const unsigned sh = (unsigned)(b & 3) * 8;
    const uint32_t* wr = S.win + (MeSmem<CELLS>::kSearches - 2 - 2 * m) * kWinStride + wi;
    unsigned acc[kUnion];
#pragma unroll
    for (int k = 0; k < kUnion; k++) acc[k] = 0;
#pragma unroll
    for (int rr = 0; rr < kMWinRows; rr++) {
      const uint32_t u0 = wr[rr * kMWinWords], u1 = wr[rr * kMWinWords + 1], u2 = wr[rr * kMWinWords + 2];
      const uint32_t w0 = __funnelshift_r(u0, u1, sh), w1 = __funnelshift_r(u1, u2, sh);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int dy = rr - i;
        if (dy >= 0 && dy < kUnion) acc[dy] = sad4_acc(cw[2 * i + 1], w1, sad4_acc(cw[2 * i], w0, acc[dy]));
      }
    }
#pragma unroll
    for (int t = 0; t < 2; t++) {
      // union column du is the offset ux - 8 + du, column ux + du - c of the window around centre c
      const int dx = ux + du - (t ? cx2 : cx1);  // column in this centre's 17 x 17 window
      const int oy = uy - (t ? cy2 : cy1);       // union row 0's row in its window
      if (dx < 0 || dx > 16) continue;
      unsigned best = 0xffffffffu;
      const unsigned pen_x = kMePenalty * abs(dx - kMeRange);
#pragma unroll
      for (int du_y = 0; du_y < kUnion; du_y++) {
        const int dy = oy + du_y;
        if (dy < 0 || dy > 16) continue;
        const unsigned cost = acc[du_y] + pen_x + kMePenalty * abs(dy - kMeRange);
        const unsigned key = (cost << 9) | (unsigned)(dy * 17 + dx);
        best = key < best ? key : best;
      }
      atomicMin(t ? &S.skey2[s] : &S.skey[s], best);
    }
    }
  }
  __syncthreads();
  if (tid < ncells && S.need[tid]) {
    const int s0 = S.first_search[tid];
    int mx, my;
    if (s0 < 0) {
      mx = S.ccx[tid][0], my = S.ccy[tid][0];
    } else {
    const unsigned k1 = S.skey[s0];
    mx = S.sx[s0] + (int)(k1 & 511) % 17 - kMeRange, my = S.sy[s0] + (int)(k1 & 511) / 17 - kMeRange;
    if (S.two[tid]) {  // the second centre's result only if strictly cheaper (me_cell, :189-192)
      const bool merged = S.two[tid] == 2;
      const unsigned k2 = merged ? S.skey2[s0] : S.skey[s0 + 1];
      const int sx2 = merged ? S.sx2[s0] : S.sx[s0 + 1], sy2 = merged ? S.sy2[s0] : S.sy[s0 + 1];
      if ((k2 >> 9) < (k1 >> 9)) mx = sx2 + (int)(k2 & 511) % 17 - kMeRange, my = sy2 + (int)(k2 & 511) / 17 - kMeRange;
    }
    }
    // level 0 in quarter pels: k_me_refine refines it in place
    job.field[r][level][cell0 + tid] = level == 0 ? pack_mv(mx * 4, my * 4) : pack_mv(mx, my);
  }
  if (job.stats && tid < 32) {  // searched centres, one atomic per unit (the cells sit in warp 0)
    const unsigned n = __reduce_add_sync(0xffffffffu, tid < ncells && S.need[tid] && S.first_search[tid] >= 0 ? (S.two[tid] ? 2u : 1u) : 0u);
    if (tid == 0) atomicAdd(job.stats + level, (unsigned long long)n);
  }
  }  // units
}

// ---- quarter-pel refinement of level 0 (me_refine, inter_common.h:141-154) ----
// One CTA of two warps per 32 consecutive level-0 cells of one (job, reference): a warp holds the halves
// of 16 cells, a lane the upper or the lower two of a cell's four 4x4 tiles side by side, their cur rows
// row-transformed once into registers. In each step a lane scores its tiles at the step's nine positions,
// three words a row and one satd4_two each; the lanes of a load read the same row of 16 neighbouring
// cells, which where their MVs agree -- most of a frame -- is one contiguous run of a phase plane's row
// (a lane per (cell, position, tile) scattered each warp's loads over nine phase planes and was bound by
// the L1's wavefronts). One shuffle adds a cell's halves, two positions at a time, and both its lanes
// replay the centre-first strict choice: no shared memory, no barrier within a unit. The second step's
// centre is the first step's winner, whose SATD the first step has already computed. The centre comes
// first of all: a move has to save more than kSubpelPenalty, so a warp none of whose centres costs more is
// done (five 1080p animation-like frames of 7 references 0.53 -> 0.24 ms).
// Five 1080p frames of 7 references: natural-like 532 -> 438 us, one masked 4K animation-like 114 -> 85,
// against a lane per tile in four warps with the sums through shared memory and a barrier each step. 72
// registers: with 64 it spills (502), with 80 the animation-like one takes 90 (natural-like 434).

// The rows of a half cell's two tiles at (ox, oy) displaced by quarter pels (qx, qy).
__device__ __forceinline__ void rows_at(const DevPlane& ref, int ox, int oy, int qx, int qy, uint32_t* a, uint32_t* b) {
  DevPlane ph = ref;
  ph.p = ref.p + (long long)((qy & 3) * 4 + (qx & 3)) * ref.phase;
  const int x = ox + (qx >> 2), y = oy + (qy >> 2);
  if (inside(ph, x, y, 8, 4)) {
    const uintptr_t p = reinterpret_cast<uintptr_t>(ph.p + (long long)y * ph.stride + x);
    const uint32_t* w = reinterpret_cast<const uint32_t*>(p & ~uintptr_t(3));
    const uint32_t sh = (uint32_t)(p & 3) * 8;
    const int ws = ph.stride >> 2;  // strides are multiples of 64
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t w0 = __ldg(w + i * ws), w1 = __ldg(w + i * ws + 1), w2 = __ldg(w + i * ws + 2);
      a[i] = __funnelshift_r(w0, w1, sh), b[i] = __funnelshift_r(w1, w2, sh);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++) a[i] = row4(ph, x, y + i), b[i] = row4(ph, x + 4, y + i);
  }
}

// The SATD of both tiles.
__device__ __forceinline__ uint32_t satd_half(const int* P, const uint32_t* a, const uint32_t* b) {
  const uint32_t v = satd4_two(P, a, b);
  return (v & 0xffffu) + (v >> 16);  // at most 32,640
}

constexpr int kRefineCells = 32, kRefineThreads = 2 * kRefineCells;

__global__ void __launch_bounds__(kRefineThreads, 14) k_me_refine(const FrameJob* __restrict__ jobs, WorkList w) {
  __shared__ int unit_slot[2];
  const int tid = threadIdx.x, c = (tid >> 5) * 16 + (tid & 15), half = tid >> 4 & 1;
  int unit, iter = 0;
  while (take_unit(w, unit, iter, unit_slot)) {
  const int jb = part_of(w, unit);
  const FrameJob& job = jobs[w.part[jb].job];
  const int cols = job.fcols[0], ncell = cols * job.frows[0];
  const int groups = (ncell + kRefineCells - 1) / kRefineCells;
  const int u = unit - w.prefix[jb];
  const int r = u / groups, cell0 = (u - r * groups) * kRefineCells;
  const int ncells = min(kRefineCells, ncell - cell0);
  const int cell = cell0 + min(c, ncells - 1), by = cell / cols, bx = cell - by * cols;
  const bool need = c < ncells && cell_needed(job, r, bx, by);
  // a warp none of whose cells a kept reference reads (pruned search): nothing to refine
  if (!__any_sync(0xffffffffu, need)) continue;
  const DevPlane cur = job.cur.lv[0], ref = job.ref[r].lv[0];
  int* field = job.field[r][0];
  // this lane's half of its cell: origin, both tiles' cur rows row-transformed
  const int ox = bx * 8, oy = by * 8 + 4 * half;
  int P[16];
  {
    uint32_t cw[4];
    int C[16];
#pragma unroll
    for (int i = 0; i < 4; i++) cw[i] = row4(cur, ox + 4, oy + i);
    wh_rows_cur(cw, C);
#pragma unroll
    for (int i = 0; i < 4; i++) cw[i] = row4(cur, ox, oy + i);
    wh_rows_cur(cw, P);
#pragma unroll
    for (int i = 0; i < 16; i++) P[i] += C[i] * 65536;
  }
  const int m = field[cell];
  int cx = mv_x(m), cy = mv_y(m);  // quarter pels, whole pels so far
  int centre;                      // the centre's SATD (the whole cell)
  {
    uint32_t a[4], b[4];
    rows_at(ref, ox, oy, cx, cy, a, b);
    centre = (int)satd_half(P, a, b);
    centre += __shfl_xor_sync(0xffffffffu, centre, 16);
    // a move must save more than kSubpelPenalty: cells whose centre costs no more stay (flat content: all
    // of a warp's)
    if (!__any_sync(0xffffffffu, need && centre > kSubpelPenalty)) continue;
  }
  // takes a position (dx, dy) of the step around (px, py) if it beats the best so far
  int best, raw, px, py, nx, ny;
  auto choose = [&](int v, int dx, int dy) {
    if (v + kSubpelPenalty < best) best = v + kSubpelPenalty, raw = v, nx = px + dx, ny = py + dy;
  };
#pragma unroll 1
  for (int step = 2; step >= 1; step--) {
    best = raw = centre, px = nx = cx, py = ny = cy;
    // the half-pel step around the whole-pel MV reads four phase planes only (phase 2 one pel left
    // or up of phase 0 at -1/2 pel, at the same pel at +1/2): the rows of the 9 x 5 footprint are
    // loaded once per plane and the positions that share a plane take 8-byte windows of them
    const int X = ox + (cx >> 2), Y = oy + (cy >> 2);
    if (step == 2 && __all_sync(0xffffffffu, inside(ref, X - 1, Y - 1, 9, 5))) {
      const int ws = ref.stride >> 2;
      // n rows from Y + y0 of phase `ph` at column X + x: the windows at it and (x < 0) a column on
      uint32_t a[5], b[5], e[5], f[5];
      auto rows = [&](int ph, int x, int y0, int n) {
        const uintptr_t p = reinterpret_cast<uintptr_t>(ref.p + ph * ref.phase + (long long)(Y + y0) * ref.stride + X + x);
        const uint32_t* q = reinterpret_cast<const uint32_t*>(p & ~uintptr_t(3));
        const uint32_t sh = (uint32_t)(p & 3) * 8;
#pragma unroll
        for (int i = 0; i < 5; i++)
          if (i < n) {
            const uint32_t w0 = __ldg(q + i * ws), w1 = __ldg(q + i * ws + 1), w2 = __ldg(q + i * ws + 2);
            a[i] = __funnelshift_r(w0, w1, sh), b[i] = __funnelshift_r(w1, w2, sh);
            if (x < 0) e[i] = __funnelshift_rc(w0, w1, sh + 8), f[i] = __funnelshift_rc(w1, w2, sh + 8);  // 32: the next word
          }
      };
      // per word two positions' SATDs of the half, then of the cell (at most 65,280 each)
      rows(8, 0, -1, 5);  // phase (2, 0): (0, -1/2) and (0, +1/2)
      uint32_t up = satd_half(P, a, b) << 16, down = satd_half(P, a + 1, b + 1) << 16;
      rows(2, -1, 0, 4);  // phase (0, 2): (-1/2, 0) and (+1/2, 0)
      uint32_t mid = satd_half(P, a, b) | satd_half(P, e, f) << 16;
      rows(10, -1, -1, 5);  // phase (2, 2): the corners
      up |= satd_half(P, a, b), down |= satd_half(P, a + 1, b + 1);
      uint32_t right = satd_half(P, e, f) | satd_half(P, e + 1, f + 1) << 16;
      up += __shfl_xor_sync(0xffffffffu, up, 16), mid += __shfl_xor_sync(0xffffffffu, mid, 16);
      down += __shfl_xor_sync(0xffffffffu, down, 16), right += __shfl_xor_sync(0xffffffffu, right, 16);
      choose(up & 0xffffu, -2, -2), choose(up >> 16, 0, -2), choose(right & 0xffffu, 2, -2);
      choose(mid & 0xffffu, -2, 0), choose(mid >> 16, 2, 0);
      choose(down & 0xffffu, -2, 2), choose(down >> 16, 0, 2), choose(right >> 16, 2, 2);
    } else {
      // the eight positions in order, two at a time
#pragma unroll 1
      for (int k = 1; k < 9; k += 2) {
        uint32_t two = 0;
        int d[2][2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          uint32_t a[4], b[4];
          const int n = refine_pos(k + h), row = n >= 6 ? 1 : n >= 3 ? 0 : -1;
          d[h][0] = (n - 4 - 3 * row) * step, d[h][1] = row * step;
          rows_at(ref, ox, oy, cx + d[h][0], cy + d[h][1], a, b);
          two |= satd_half(P, a, b) << (16 * h);
        }
        two += __shfl_xor_sync(0xffffffffu, two, 16);
        choose(two & 0xffffu, d[0][0], d[0][1]);
        choose(two >> 16, d[1][0], d[1][1]);
      }
    }
    // the next step's centre: its SATD is known
    centre = raw, cx = nx, cy = ny;
  }
  if (!half && need) field[cell] = pack_mv(cx, cy);
  }  // units
}

int refine_units(int nrefs, int cols, int rows) { return nrefs * ((cols * rows + kRefineCells - 1) / kRefineCells); }

void launch_me_refine(const FrameJob* jobs, const WorkList& w, cudaStream_t st) {
  const int units = w.prefix[w.nparts];
  if (units <= 0) return;
  const int grid = w.queue ? persistent_grid((const void*)k_me_refine, kRefineThreads, 0, units) : units;
  k_me_refine<<<grid, kRefineThreads, 0, st>>>(jobs, w);
}

int me_units(int nrefs, int cols, int rows, int cells) { return nrefs * ((cols * rows + cells - 1) / cells); }

// Cells a CTA takes of a level: as configured (15 or 30) where the launch fills the GPU; seven, whose
// searches are one round of 256 threads, while those CTAs are all resident at once: such a launch takes
// one CTA's time, levels 2 and 3 of a 416x240 frame 17 us with 30 cells and 13 with seven (stage events, 7 us of
// them the events), its level 1 16.9 and 14.8.
int me_level_cells(long long cells, int configured) {
  const int full = persistent_grid((const void*)k_me_level<30>, kMeThreads, sizeof(MeSmem<30>), INT_MAX);
  return cells <= 7LL * full ? 7 : configured;
}

template <int CELLS>
static void launch_cells(const FrameJob* jobs, const WorkList& w, int level, cudaStream_t st) {
  const int units = w.prefix[w.nparts];
  const size_t smem = sizeof(MeSmem<CELLS>);
  const int grid = w.queue ? persistent_grid((const void*)k_me_level<CELLS>, kMeThreads, smem, units) : units;
  k_me_level<CELLS><<<grid, kMeThreads, smem, st>>>(jobs, w, level);
}

void launch_me_level(const FrameJob* jobs, const WorkList& w, int level, int cells, cudaStream_t st) {
  if (w.prefix[w.nparts] <= 0) return;
  if (cells == 7)
    launch_cells<7>(jobs, w, level, st);
  else if (cells == 15)
    launch_cells<15>(jobs, w, level, st);
  else
    launch_cells<30>(jobs, w, level, st);
}

template <int CELLS>
static cudaError_t attributes_cells() {
  const size_t smem = sizeof(MeSmem<CELLS>);
  const cudaError_t e = cudaFuncSetAttribute(k_me_level<CELLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) persistent_grid((const void*)k_me_level<CELLS>, kMeThreads, smem, 1);  // fills the grid cache
  return e;
}

cudaError_t me_attributes() {
  cudaError_t e = attributes_cells<7>();
  if (e == cudaSuccess) e = attributes_cells<15>();
  if (e == cudaSuccess) e = attributes_cells<30>();
  if (e == cudaSuccess) persistent_grid((const void*)k_me_refine, kRefineThreads, 0, 1);  // fills the grid cache
  return e;
}

}  // namespace celv2cu
