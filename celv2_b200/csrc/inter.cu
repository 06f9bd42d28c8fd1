// inter.cu: each reference's best single-reference candidate for every candidate block.
//
// Reference rules: mv_cells / candidate_mv_index / repeated_candidate
// (src/gpu/inter_common.h:60-89), block_inter_satd (:223-235) and the per-reference loop of
// best_both (src/gpu/kernels_ref.cpp:54-66): candidates in order, repeats skipped, first strict
// minimum of SATD * 256 + lambda * (3 + r) -- i.e. of the SATD, the bits being constant per
// reference.
//
// Work reuse: a block's SATD at an MV is the sum of its 4x4 tiles' SATDs at that MV (the blocks'
// tiles all sit on the superblock's 4x4 grid), and every candidate MV of a superblock's blocks is
// the level-0 MV of one of the 10 x 10 cells around it. So one CTA per (superblock, reference):
//  1. gathers those 100 MVs (clamped into the field) and their distinct set D through a small hash
//     table (in no particular order: a candidate's rank is its index, not its MV's), and per MV of D
//     the window its prediction takes: 64 rows of 80 bytes from a 16-byte boundary of its phase plane;
//  2. two MVs a step, the windows brought to shared memory by TMA two steps ahead (a ring of three, an
//     mbarrier each way): half the threads an MV, one thread per pair of 4x4 tiles side by side, their
//     cur samples in registers, the pair's rows three words each and its two SATDs the halfwords of
//     one satd4_two; the pair below in the 8x8 cell is eight lanes on, so one shuffle gives the cell's
//     sum and its left half's (its top half's needs none; the other two are differences);
//  3. every so many MVs the 16x16 sums are formed and every candidate in the pass takes its SATD, a
//     block keeping its least (SATD << 7 | candidate index). That is the reference's first strict
//     minimum over the candidates in order: a repeated MV (which the reference skips) has the same
//     SATD as its first occurrence and a larger index, so it never wins. The 8x8 cells' blocks (two
//     thirds of the candidates) go by (cell, candidate), one load for all five blocks, without atomics.
// 256 |D| Hadamards per (superblock, reference) instead of up to 68,352 for the blocks one by one.
// Integer issue bound: five 1080p frames of 7 references 2.04 -> 1.60 ms (17,850 units), 289 -> 227 M
// instructions a frame, against one thread per tile with every row word by word through L1, four
// shuffles an MV, each slot's index listed and every candidate an atomicMin; a 416x240 frame of 3
// references 56 -> 31 us.
// Pruned search: where the superblock keeps no 64-level blocks (no 64x64, 64x32, 32x64), a second
// kernel (k_inter_regions) scores each of its 32x32 regions (16x16 with no 32-level blocks either)
// on its own: a kept block and all its candidates' cells lie inside its region and the ring of
// cells around it, so the region's tiles are scored at the distinct MVs of its 6 x 6 (4 x 4) cells
// only -- exactly the SATDs the whole-superblock pass gives them. The whole-superblock kernel
// (k_inter) keeps its own code and registers: the units of the two kinds go to the two kernels.
// The result per (block, reference) is the winning SATD and MV; the lambda terms are added by the
// finalize stage, which alone needs the costs.
#include <algorithm>
#include <type_traits>

#include "kernels.h"

namespace celv2cu {

constexpr int kInterThreads = 256;  // one per 4x4 tile of the superblock
constexpr int kNb = 100;            // 10 x 10 cells around the superblock
constexpr int kChunk = 64;          // distinct MVs per pass at most
constexpr int kWinRow = 80, kWin = 64 * kWinRow;  // bytes of an MV's window: its row, all of it
constexpr int kRing = 3;
constexpr int kPassG1 = 30;  // MVs whose sums a CTA of four an SM has room for
constexpr int kSlots = 4296;        // candidates of the 425 blocks (cells covered + 8 neighbours)

// Every (block, candidate) slot as b | k << 9 | cell << 16 (its neighbourhood cell), ordered by
// block size, block kind, candidate index, block: a warp's slots then take one path through
// block_satd and name 32 different blocks (no divergence, no colliding shared atomics).
__device__ unsigned g_slot[kSlots];
// Block b's candidate k sits in neighbourhood cell g_cand_cell[c_cand_off[b] + k].
__constant__ short c_cand_off[kBlocks];
__device__ unsigned char g_cand_cell[kSlots];

// An 8x8 cell's candidates as offsets in the neighbourhood, in candidate order (candidate_cell).
__constant__ int c_cell_off[9] = {0, -1, -10, 1, 10, -11, -9, 9, 11};

constexpr int kMaxRegions = 16;  // 16x16 regions of a superblock
constexpr int kRegCells = 256;   // regions x neighbourhood cells at most (16 x 16, 4 x 36, 1 x 100)

// Per candidate slot (in g_slot's order) and per block: level | 32x32 region << 2 | 16x16 region
// << 4. The slots of one level are contiguous in g_slot's order: level l's from c_level_slot[l].
__device__ unsigned char g_slot_aux[kSlots];
__device__ unsigned char g_block_aux[kBlocks];
__constant__ int c_level_slot[5];

// The region pass's shared state.
struct RegionSmem {
  int rnb[kInterThreads];      // per thread (region, local cell): the cell's packed MV
  int D[kRegCells];            // per region r: its distinct MVs at D[r * ncell ..], first occurrence order
  int moff[kRegCells];         // per (region, MV): the superblock's prediction, bytes from the reference's level 0
  unsigned char mfast[kRegCells];  // per (region, MV): the region's prediction lies inside the margin
  unsigned char dmap[kMaxRegions][kNb];  // per region: neighbourhood cell -> its MV's index in the region's D
  unsigned bal[kInterThreads / 32];      // per warp: which lanes hold a first occurrence
  int nd[kMaxRegions];
  int nd_max;
  unsigned key[kBlocks];              // per block: least (SATD << 7 | candidate index) so far
};

// The per-chunk sums follow RegionSmem in shared memory, sized by the launch's chunk (a smaller
// chunk leaves more of the SM's memory to the L1 cache the prediction rows go through).
struct ChunkSums {
  unsigned short (*tile)[256];   // [chunk][256] 4x4 SATDs (at most 16 x 4 x 255 = 16,320)
  unsigned short (*whole8)[64];  // [chunk][64] 8x8 sums (at most 65,280)
  int (*sum16)[16];              // [chunk][16] 16x16 sums
};

__host__ __device__ constexpr size_t inter_smem_bytes(int chunk) {
  return (sizeof(RegionSmem) + 15) / 16 * 16 + (size_t)chunk * (256 * 2 + 64 * 2 + 16 * 4);
}

__device__ __forceinline__ ChunkSums chunk_sums(unsigned char* base, int chunk) {
  unsigned char* p = base + (sizeof(RegionSmem) + 15) / 16 * 16;
  ChunkSums c;
  c.tile = reinterpret_cast<unsigned short (*)[256]>(p);
  c.whole8 = reinterpret_cast<unsigned short (*)[64]>(p + (size_t)chunk * 512);
  c.sum16 = reinterpret_cast<int (*)[16]>(p + (size_t)chunk * 640);
  return c;
}

// The whole-superblock pass (every kept level, the 64-level blocks among them): its shared state, then
// the ring of windows, then the sums of a pass. G groups of 256 threads share a unit's MVs.
constexpr int kNoMv = 0x7fff7fff;  // no motion vector of any field (they stay within +-995 quarter pels)
constexpr int kTab = 256;
constexpr int kUpperSlots = 1416;  // candidates of the blocks above the 8x8 cells' (levels 0-2)

struct WholeSmem {
  unsigned long long full[kRing], empty[kRing];  // mbarriers: a slot's windows are there; every warp is done with them
  int tab[kTab];                // hash table of the cells' MVs
  unsigned char tidx[kTab];     // per table entry: its MV's index in D
  int D[kNb];                   // distinct MVs
  int2 win[kNb];                // per MV of D: its window's first row in the phase plane << 4 | phase; the first
                                // byte of its rows (from the row's start, a multiple of 16) | the prediction's
                                // first byte in them (-1: not all inside the margin, or no MV)
  unsigned char dmap[kNb];      // neighbourhood cell -> its MV's index in D
  unsigned key[kBlocks];        // per block: least (SATD << 7 | candidate index) so far
  int nd;
};

struct PassSums {
  uint2 (*cell)[64];  // [MV][64] per 8x8 cell its four tiles' SATDs: top left | top right << 16, bottom likewise
  int (*sum16)[20];   // [MV][20] 16x16 sums, then the four 32x32 quadrants'
};
constexpr int kPassBytes = 64 * 8 + 20 * 4;  // a pass's sums per MV

constexpr size_t whole_ring_at() { return (sizeof(WholeSmem) + 15) / 16 * 16; }
template <int G>
constexpr size_t whole_smem_bytes(int pass) {
  return whole_ring_at() + 128 + (size_t)kRing * 2 * G * kWin + (size_t)pass * kPassBytes;
}

// The sum of an 8x8 cell's four tiles.
__device__ __forceinline__ uint32_t cell_sum(uint2 q) {
  const uint32_t cols = q.x + q.y;  // (each half at most 32,640)
  return (cols & 0xffffu) + (cols >> 16);
}

// SATD of block b of levels 0-2 at the pass's MV dd.
__device__ __forceinline__ int block_satd(const PassSums& S, int b, int dd) {
  const int sq = b / 5, kind = b - sq * 5;
  const int* s = S.sum16[dd];
  if (sq >= 5) {  // 16x16: children are 8x8 cells
    const int i = sq - 5, c = (i >> 2) * 16 + (i & 3) * 2;
    if (kind == 0) return s[i];
    // the halves' two cells: top, bottom, left, right
    const uint2* W = S.cell[dd] + c + (kind == 2 ? 8 : kind == 4 ? 1 : 0);
    return (int)(cell_sum(W[0]) + cell_sum(W[kind <= 2 ? 1 : 8]));
  }
  if (sq >= 1) {  // 32x32: its four 16x16 squares, or itself
    if (kind == 0) return s[15 + sq];
    const int i = sq - 1, c = (i >> 1) * 8 + (i & 1) * 2 + (kind == 2 ? 4 : kind == 4 ? 1 : 0);
    return s[c] + s[c + (kind <= 2 ? 1 : 4)];
  }
  const int* q = s + 16 + (kind == 2 ? 2 : kind == 4 ? 1 : 0);
  return kind == 0 ? q[0] + q[1] + q[2] + q[3] : q[0] + q[kind <= 2 ? 1 : 2];
}

// SATD of block b at chunk-local MV dd of the region pass.
__device__ __forceinline__ int block_satd(const ChunkSums& S, int b, int dd) {
  const int sq = b / 5, kind = b - sq * 5;
  if (sq >= 21) {  // 8x8 cell c: its tiles t, t + 1, t + 16, t + 17
    const int c = sq - 21, t = (c >> 3) * 32 + (c & 7) * 2;
    const unsigned short* T = S.tile[dd];
    switch (kind) {
      case 0: return S.whole8[dd][c];
      case 1: return T[t] + T[t + 1];
      case 2: return T[t + 16] + T[t + 17];
      case 3: return T[t] + T[t + 16];
      default: return T[t + 1] + T[t + 17];
    }
  }
  if (sq >= 5) {  // 16x16: children are 8x8 cells
    const int i = sq - 5, c = (i >> 2) * 16 + (i & 3) * 2;
    const unsigned short* W = S.whole8[dd];
    switch (kind) {
      case 0: return S.sum16[dd][i];
      case 1: return W[c] + W[c + 1];
      case 2: return W[c + 8] + W[c + 9];
      case 3: return W[c] + W[c + 8];
      default: return W[c + 1] + W[c + 9];
    }
  }
  const int* s = S.sum16[dd];
  if (sq >= 1) {  // 32x32: children are 16x16 squares
    const int i = sq - 1, c0 = (i >> 1) * 8 + (i & 1) * 2;
    const int tl = s[c0], tr = s[c0 + 1], bl = s[c0 + 4], br = s[c0 + 5];
    switch (kind) {
      case 0: return tl + tr + bl + br;
      case 1: return tl + tr;
      case 2: return bl + br;
      case 3: return tl + bl;
      default: return tr + br;
    }
  }
  int q[4];  // the 32x32 quadrants
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int c0 = (i >> 1) * 8 + (i & 1) * 2;
    q[i] = s[c0] + s[c0 + 1] + s[c0 + 4] + s[c0 + 5];
  }
  switch (kind) {
    case 0: return q[0] + q[1] + q[2] + q[3];
    case 1: return q[0] + q[1];
    case 2: return q[2] + q[3];
    case 3: return q[0] + q[2];
    default: return q[1] + q[3];
  }
}

// Neighbourhood index (10 x 10, origin one cell above-left of the superblock) of candidate k of
// the block at superblock-local (bx, by), size bw x bh (candidate_mv_index, inter_common.h:65-78).
__host__ __device__ __forceinline__ int candidate_cell(int bx, int by, int bw, int bh, int k) {
  const int lx = bx >> 3, ly = by >> 3;
  const int cw = ((bx + bw - 1) >> 3) - lx + 1, ch = ((by + bh - 1) >> 3) - ly + 1, cells = cw * ch;
  int cx, cy;
  if (k < cells) {
    const int kr = k / cw;
    cx = lx + (k - kr * cw), cy = ly + kr;
  } else {
    const int n = k - cells;
    const int nl = lx - 1, nr = (bx + bw) >> 3, nt = ly - 1, nbm = (by + bh) >> 3;
    cx = (n == 0 || n == 4 || n == 6) ? nl : (n == 2 || n == 5 || n == 7) ? nr : lx;
    cy = (n == 1 || n == 4 || n == 5) ? nt : (n == 3 || n == 6 || n == 7) ? nbm : ly;
  }
  return (cy + 1) * 10 + cx + 1;
}

__device__ __forceinline__ void mbar_init(unsigned bar, int count) {
  asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Waits for the phase of this parity to end, at most about a second: false then.
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
               : "=r"(done)
               : "r"(bar), "r"(parity)
               : "memory");
  return done != 0;
}
__device__ __forceinline__ unsigned global_ns() {
  unsigned t;
  asm volatile("mov.u32 %0, %globaltimer_lo;" : "=r"(t));
  return t;
}
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
  if (mbar_try(bar, parity)) return true;
  const unsigned t0 = global_ns();
  while (!mbar_try(bar, parity))
    if (global_ns() - t0 > 1000000000u) return false;
  return true;
}
// A box of the tensor at byte x (a multiple of 16), row y, plane z into shared memory, counted by `bar`.
__device__ __forceinline__ void tma_box(unsigned dst, const void* map, int x, int y, int z, unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

// A wait that ran out: none of the launch's jobs counts as decided (with its CTAs gone, units of any of them may
// be left that no CTA takes).
__device__ __forceinline__ void mark_fault(const FrameJob* jobs, const WorkList& w) {
  for (int p = 0; p < w.nparts; p++) *jobs[w.part[p].job].fault = 1;
}

// G groups of 256 threads, 2G halves: half h takes MV h of a step's 2G. pass: MVs whose sums shared
// memory holds, a multiple of 2G.
template <int G>
__global__ void __launch_bounds__(kInterThreads* G, 4 / G) k_inter(const FrameJob* __restrict__ jobs, WorkList w, int pass) {
  constexpr int T = kInterThreads * G, M = 2 * G;  // threads, MVs a step
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WholeSmem& S = *reinterpret_cast<WholeSmem*>(smem_raw);
  // TMA writes to 128-byte boundaries; the dynamic array's own start is only known to be 16-byte aligned
  unsigned char* ring = smem_raw + whole_ring_at();
  ring += (0u - (unsigned)__cvta_generic_to_shared(ring)) & 127u;
  PassSums Q;
  Q.cell = reinterpret_cast<uint2 (*)[64]>(ring + kRing * M * kWin);
  Q.sum16 = reinterpret_cast<int (*)[20]>(ring + kRing * M * kWin + pass * 512);
  __shared__ int unit_slot[2];
  const int tid = threadIdx.x, lane = tid & 31, half = tid >> 7, px = tid & 7, ty = (tid & 127) >> 3;
  const unsigned ring_s = (unsigned)__cvta_generic_to_shared(ring);
  const unsigned full_s = (unsigned)__cvta_generic_to_shared(S.full), empty_s = (unsigned)__cvta_generic_to_shared(S.empty);
  if (tid == 0) {
    for (int i = 0; i < kRing; i++) mbar_init(full_s + 8 * i, 1), mbar_init(empty_s + 8 * i, T / 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  unsigned parity = 0;  // per ring slot: the parity of its next step's round (bit; over all units)
  int unit, iter = 0;
  while (take_unit(w, unit, iter, unit_slot)) {
  const int jb = part_of(w, unit);
  const FrameJob& job = jobs[w.part[jb].job];
  const int nsb = w.part[jb].sbs;
  const int u = unit - w.prefix[jb];
  const int r = u / nsb, sb = w.part[jb].sb0 + u - r * nsb, sby = sb / job.sb_cols, sbx = sb - sby * job.sb_cols;
  const unsigned keep = keep_mask(job, sb);
  // a pruned (superblock, reference) is not scored; without 64-level blocks k_inter_regions scores it
  if (!(keep >> r & 1u) || !(keep & CELV2_KEEP_LEVEL(0))) continue;
  const int ox = sbx * 64, oy = sby * 64;

  // 1. neighbourhood MVs and their distinct set
  int v = 0;
  if (tid < kNb) {
    const int cols = job.fcols[0], rows = job.frows[0];
    const int ny = tid / 10, nx = tid - ny * 10;
    const int cx = clampi(sbx * 8 - 1 + nx, 0, cols - 1), cy = clampi(sby * 8 - 1 + ny, 0, rows - 1);
    v = job.field[r][0][cy * cols + cx];
  }
  for (int e = tid; e < kTab; e += T) S.tab[e] = kNoMv;
  for (int b = tid; b < kBlocks; b += T) S.key[b] = 0xffffffffu;
  if (tid == 0) S.nd = 0;
  // this thread's tiles: their cur rows, row-transformed, in registers (the grid lies inside the margin)
  int P[16];
  {
    const DevPlane& cur = job.cur.lv[0];
    uint32_t c[2][4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint2 q = *reinterpret_cast<const uint2*>(cur.p + (long long)(oy + ty * 4 + i) * cur.stride + ox + px * 8);
      c[0][i] = q.x, c[1][i] = q.y;
    }
    int C[16];
    wh_rows_cur(c[1], C);
    wh_rows_cur(c[0], P);
#pragma unroll
    for (int i = 0; i < 16; i++) P[i] += C[i] * 65536;
  }
  __syncthreads();
  unsigned h = ((unsigned)v * 2654435761u) >> 24;
  if (tid < kNb) {
    for (;; h = (h + 1) & (kTab - 1)) {  // at most 100 of 256 entries are ever taken
      const int old = atomicCAS(&S.tab[h], kNoMv, v);
      if (old == kNoMv) {
        const int i = atomicAdd(&S.nd, 1);
        S.tidx[h] = (unsigned char)i;
        S.D[i] = v;
        // its window; one that is not all inside the margin is read sample by sample
        const DevPlane& ref = job.ref[r].lv[0];
        const int mx = mv_x(v), my = mv_y(v), x = ox + (mx >> 2), y = oy + (my >> 2);
        S.win[i] = make_int2((y + ref.margin) << 4 | (my & 3) * 4 | (mx & 3), inside(ref, x, y, 64, 64) ? x + ref.margin : -1);
      }
      if (old == kNoMv || old == v) break;
    }
  }
  __syncthreads();
  if (tid < kNb) S.dmap[tid] = S.tidx[h];
  const int nd = S.nd, steps = (nd + M - 1) / M;
  if (tid == 0 && job.stats) atomicAdd(job.stats + kStatInterMvs, (unsigned long long)nd * 256);

  __syncthreads();  // dmap complete
  // step s's windows into ring slot `to`, by one thread, once every warp is done with the step that had
  // the slot before; round: the parity of the step's own round (a wait that runs out leaves the
  // step without windows, which ends every thread's own wait for them; the batch is marked there alone: the loop
  // over its jobs in each of these copies was 1.3 of 33 us of a 416x240 frame's stage)
  const void* map = job.map + r;
  auto load_step = [&](int s, unsigned to, unsigned round) {
    if (s >= steps) return;
    const unsigned bar = full_s + 8 * to;
    if (!mbar_wait(empty_s + 8 * to, round ^ 1)) return;
    int2 e[M];
    unsigned bytes = 0;
#pragma unroll
    for (int m = 0; m < M; m++) {
      e[m] = s * M + m < nd ? S.win[s * M + m] : make_int2(0, -1);
      bytes += e[m].y >= 0 ? kWin : 0;
    }
    mbar_expect(bar, bytes);
#pragma unroll
    for (int m = 0; m < M; m++)
      if (e[m].y >= 0) tma_box(ring_s + (to * M + m) * kWin, map, e[m].y & ~15, e[m].x >> 4, e[m].x & 15, bar);
  };
  if (tid == 0) {  // a unit's step s takes slot s % kRing
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
    load_step(0, 0, parity & 1);
    load_step(1, 1, parity >> 1 & 1);
  }

  const unsigned char* win0 = ring + half * kWin + ty * (4 * kWinRow) + px * 8;
  uint32_t* cell0 = &Q.cell[half][(ty >> 1) * 8 + px].x + (ty & 1);
  int p0 = 0;  // the pass's first MV
  bool ok = true;
  int s = 0;
  // 2. tile SATDs at step s's MVs; dst: where this thread's word goes
  auto step = [&](auto slot_c, uint32_t* dst) {
    constexpr unsigned slot = decltype(slot_c)::value, next = (slot + 2) % kRing;
    // (the slot two steps on has had its round of this unit already, or gets its first)
    if (tid == 0) load_step(s + 2, next, parity >> next & 1);
    if (!mbar_wait(full_s + 8 * slot, parity >> slot & 1)) return false;
    const int d = s * M + half;
    if (d < nd) {
      const int wx = S.win[d].y;
      uint32_t a[4], b[4];  // the left and the right tile's rows
      if (wx >= 0) {
        uint32_t w[4][3];
        if (wx & 4) {  // three words a row, two of them an aligned pair
          const unsigned char* g = win0 + (wx & 8) + (slot * M * kWin + 4);
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const uint2 q = *reinterpret_cast<const uint2*>(g + i * kWinRow + 4);
            w[i][0] = *reinterpret_cast<const uint32_t*>(g + i * kWinRow), w[i][1] = q.x, w[i][2] = q.y;
          }
        } else {
          const unsigned char* g = win0 + (wx & 8) + slot * M * kWin;
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const uint2 q = *reinterpret_cast<const uint2*>(g + i * kWinRow);
            w[i][0] = q.x, w[i][1] = q.y, w[i][2] = *reinterpret_cast<const uint32_t*>(g + i * kWinRow + 8);
          }
        }
        const unsigned sh = 8 * (wx & 3);
#pragma unroll
        for (int i = 0; i < 4; i++) a[i] = __funnelshift_r(w[i][0], w[i][1], sh), b[i] = __funnelshift_r(w[i][1], w[i][2], sh);
      } else {  // a window past the margin: sample by sample, clamped
        const int m = S.D[d], mx = mv_x(m), my = mv_y(m);
        DevPlane ph = job.ref[r].lv[0];
        ph.p += (long long)((my & 3) * 4 + (mx & 3)) * ph.phase;
        const int x = ox + px * 8 + (mx >> 2), y = oy + ty * 4 + (my >> 2);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          a[i] = b[i] = 0;
#pragma unroll 1
          for (int q = 3; q >= 0; q--) a[i] = a[i] << 8 | (uint32_t)at(ph, y + i, x + q), b[i] = b[i] << 8 | (uint32_t)at(ph, y + i, x + 4 + q);
        }
      }
      *dst = satd4_two(P, a, b);  // left | right << 16
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty_s + 8 * slot);
    parity ^= 1u << slot;
    s++;
    return true;
  };
  while (p0 < nd) {
    // the pass's steps, three by three (a unit's passes are multiples of three steps long)
    const int end = min(steps, s + pass / M);
    uint32_t* dst = cell0;
    while (ok && s < end) {
      constexpr int kStep = M * 128;  // words of a step's MVs
      ok = step(std::integral_constant<unsigned, 0>{}, dst);
      if (ok && s < end) ok = step(std::integral_constant<unsigned, 1>{}, dst + kStep);
      if (ok && s < end) ok = step(std::integral_constant<unsigned, 2>{}, dst + 2 * kStep);
      dst += 3 * kStep;
    }
    if (!ok) break;  // (all threads at the same step: nothing was loaded)
    const int pn = min(nd, s * M) - p0;  // the pass's MVs
    __syncthreads();
    for (int e = tid; e < pn * 16; e += T) {
      const int dd = e >> 4, i = e & 15;  // 16x16 squares quadrant by quadrant: four lanes hold a 32x32
      const int sy = (i >> 3) * 2 + (i >> 1 & 1), sx = (i >> 2 & 1) * 2 + (i & 1), c = sy * 16 + sx * 2;
      const uint2* W = Q.cell[dd];
      const int v = (int)(cell_sum(W[c]) + cell_sum(W[c + 1]) + cell_sum(W[c + 8]) + cell_sum(W[c + 9]));
      const unsigned four = 0xfu << (tid & 28);
      int q = v + __shfl_xor_sync(four, v, 1);
      q += __shfl_xor_sync(four, q, 2);
      Q.sum16[dd][sy * 4 + sx] = v;
      if ((i & 3) == 0) Q.sum16[dd][16 + (i >> 2)] = q;
    }
    // 3. the blocks of each 8x8 cell: 4G lanes a cell, each every 4G-th of the nine candidates (the cell
    //    itself, then its neighbours left, above, right, below, and the corners). The top half's
    //    candidates below and the left half's to the right are the cell's own row and column again
    //    (repeats, never the first), so those two skip them
    {
      constexpr int L = 4 * G;
      const int cell = tid / L, ci = (cell >> 3) * 10 + (cell & 7) + 11;  // its neighbourhood index
      unsigned m[5] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
      for (int k = tid % L; k < 9; k += L) {
        const int dd = (int)S.dmap[ci + c_cell_off[k]] - p0;
        if (dd < 0 || dd >= pn) continue;
        const uint2 q = Q.cell[dd][cell];
        const unsigned cols = q.x + q.y, left = cols & 0xffffu, all = left + (cols >> 16);
        const unsigned top = (q.x & 0xffffu) + (q.x >> 16);
        m[0] = min(m[0], all << 7 | (unsigned)k);
        if (!(0x190u >> k & 1)) m[1] = min(m[1], top << 7 | (unsigned)k);
        m[2] = min(m[2], (all - top) << 7 | (unsigned)k);
        if (!(0x148u >> k & 1)) m[3] = min(m[3], left << 7 | (unsigned)k);
        m[4] = min(m[4], (all - left) << 7 | (unsigned)k);
      }
#pragma unroll
      for (int i = 0; i < 5; i++)
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) m[i] = min(m[i], __shfl_xor_sync(0xffffffffu, m[i], o));
      if (tid % L == 0) {
        unsigned* key = S.key + (21 + cell) * 5;
#pragma unroll
        for (int i = 0; i < 5; i++) key[i] = min(key[i], m[i]);
      }
    }
    __syncthreads();
    //    every candidate of the other blocks whose MV is in this pass
    for (int e = tid; e < kUpperSlots; e += T) {
      const unsigned bp = __ldg(g_slot + e);
      const int dd = (int)S.dmap[bp >> 16] - p0;
      if (dd < 0 || dd >= pn) continue;
      const int b = bp & 511, k = (bp >> 9) & 127;
      atomicMin(&S.key[b], ((unsigned)block_satd(Q, b, dd) << 7) | (unsigned)k);
    }
    p0 += pn;
    __syncthreads();  // the next pass overwrites the sums
  }
  if (!ok) {  // a wait ran out: the batch is marked, this CTA's steps still in flight are given their time
    if (tid == 0) mark_fault(jobs, w);
    for (int k = s + 1; k < min(s + 3, steps); k++) mbar_wait(full_s + 8 * (k % kRing), parity >> (k % kRing) & 1);
    return;
  }
  int2* out = job.inter + ((long long)sb * kMaxRefs + r) * kBlocks;
  for (int b = tid; b < kBlocks; b += T) {
    const unsigned k = S.key[b];
    out[b] = make_int2((int)(k >> 7), S.D[S.dmap[g_cand_cell[c_cand_off[b] + (k & 127)]]]);
  }
  }  // units
}

// One (superblock, reference) unit of the region pass, regions of R x R samples (32 or 16).
template <int R>
__device__ __forceinline__ void region_unit(RegionSmem& S, const ChunkSums& Q, const FrameJob& job, int r, int sb,
                                            int sbx, int sby, unsigned keep, int chunk) {
  constexpr int nr = 64 / R, nreg = nr * nr, rcells = R / 8, rc = rcells + 2, ncell = rc * rc;
  constexpr int per = kInterThreads / nreg;  // threads per region: 64 (R = 32) or 16 (R = 16)
  static_assert(per >= ncell && (per & (per - 1)) == 0 && nreg * ncell <= kRegCells, "region layout");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ox = sbx * 64, oy = sby * 64;
  const int cols = job.fcols[0], rows = job.frows[0];
  const int* field = job.field[r][0];

  // 1. thread (region reg, local cell lc) reads its neighbourhood cell's MV (clamped into the field)
  const int reg = tid / per, lc = tid % per;
  const bool live = lc < ncell;
  const int c10 = ((reg / nr) * rcells + lc / rc) * 10 + (reg % nr) * rcells + lc % rc;
  int v = 0;
  if (live) {
    const int cx = clampi(sbx * 8 - 1 + c10 % 10, 0, cols - 1), cy = clampi(sby * 8 - 1 + c10 / 10, 0, rows - 1);
    v = __ldg(field + cy * cols + cx);
  }
  S.rnb[tid] = v;
  for (int b = tid; b < kBlocks; b += kInterThreads) S.key[b] = 0xffffffffu;
  if (tid == 0) S.nd_max = 0;
  __syncthreads();
  // the region's first local cell holding this MV; the first occurrences, in local cell order, are
  // the region's distinct MVs: an MV's index is the number of first occurrences before its own
  int firstlc = lc;
  if (live) {
    const int* rn = S.rnb + reg * per;
    for (int k = 0; k < lc; k++)
      if (rn[k] == v) {
        firstlc = k;
        break;
      }
  }
  const bool is_first = live && firstlc == lc;
  const unsigned bal = __ballot_sync(0xffffffffu, is_first);
  if (lane == 0) S.bal[warp] = bal;
  const int nd_sum = __syncthreads_count(is_first);
  int pos, nd;
  if constexpr (per == 16) {  // two regions per warp, a half each
    const unsigned rb = (bal >> ((reg & 1) * 16)) & 0xffffu;
    pos = __popc(rb & ((1u << firstlc) - 1u)), nd = __popc(rb);
  } else {  // a region over two warps: local cells 0-31 and 32-35
    const unsigned ba = S.bal[2 * reg], bb = S.bal[2 * reg + 1];
    pos = firstlc < 32 ? __popc(ba & ((1u << firstlc) - 1u)) : __popc(ba) + __popc(bb & ((1u << (firstlc - 32)) - 1u));
    nd = __popc(ba) + __popc(bb);
  }
  if (live) S.dmap[reg][c10] = (unsigned char)pos;
  const DevPlane cur = job.cur.lv[0], ref = job.ref[r].lv[0];
  if (is_first) {  // per (region, MV): the prediction's offset, inside the margin or not
    const int e = reg * ncell + pos, mx = mv_x(v), my = mv_y(v);
    const int x = ox + (mx >> 2), y = oy + (my >> 2);
    const long long o = (long long)((my & 3) * 4 + (mx & 3)) * ref.phase + (long long)y * ref.stride + x;
    S.D[e] = v;
    S.moff[e] = (int)o;
    S.mfast[e] = inside(ref, x + (reg % nr) * R, y + (reg / nr) * R, R, R) && o == (long long)(int)o;
  }
  if (lc == 0) S.nd[reg] = nd, atomicMax(&S.nd_max, nd);
  if (tid == 0 && job.stats) atomicAdd(job.stats + kStatInterMvs, (unsigned long long)nd_sum * (R / 4) * (R / 4));

  // this thread's tile: its cur rows, row-transformed, in registers (the grid lies inside the margin)
  const int tx = tid & 15, ty = tid >> 4;
  const int treg = (ty / (R / 4)) * nr + tx / (R / 4);  // the tile's region
  int C[16];
  {
    uint32_t c[4];
#pragma unroll
    for (int i = 0; i < 4; i++) c[i] = load4(cur.p + (long long)(oy + ty * 4 + i) * cur.stride + ox + tx * 4);
    wh_rows_cur(c, C);
  }
  // the tile's prediction rows at MV d start at tile_base + moff[d]; words a row apart are ws apart
  const uintptr_t tile_base = reinterpret_cast<uintptr_t>(ref.p) + (uintptr_t)(ty * 4 * ref.stride + tx * 4);
  const int ws = ref.stride >> 2;  // strides are multiples of 64
  __syncthreads();  // MVs, maps, offsets complete
  const int tnd = S.nd[treg], tbase = treg * ncell, nd_max = S.nd_max;
  const int wnd = __reduce_max_sync(0xffffffffu, tnd);  // the most MVs of this warp's regions
  // the candidate slots of the kept levels (contiguous by level in g_slot's order; levels 1-3 here)
  const unsigned lv = (keep & CELV2_KEEP_LEVELS) >> 8;
  const int slot_lo = c_level_slot[__ffs(lv) - 1], slot_hi = c_level_slot[32 - __clz(lv)];
  // chunks of equal size, at most `chunk` MVs each
  const int nchunks = (nd_max + chunk - 1) / chunk, csize = (nd_max + nchunks - 1) / nchunks;

  for (int c0 = 0; c0 < nd_max; c0 += csize) {
    const int nc = min(csize, nd_max - c0);
    const int tnc = min(nc, tnd - c0);  // this tile's region's MVs in the chunk
    const int wnc = min(nc, wnd - c0);  // this warp's
    // 2. tile SATDs at the region's MVs of the chunk (two MVs per step for load parallelism); an
    //    8x8 cell's tiles are lanes l, l + 1, l + 16, l + 17 of one warp (and of one region)
    for (int dd = 0; dd < wnc; dd += 2) {
      int sat[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        // a tile whose region has no MV left scores its region's first MV (always there); those
        // sums are never read: a region's slots name only its own MVs
        const int d = tbase + (tnc > 0 ? c0 + min(dd + h, tnc - 1) : 0);
        uint32_t pr[4];
        if (S.mfast[d]) {  // the usual case: rows from aligned words
          const uintptr_t a = tile_base + (uintptr_t)(intptr_t)S.moff[d];
          const uint32_t* wp = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
          const uint32_t sh = (uint32_t)(a & 3) * 8;
          if (sh == 0) {
#pragma unroll
            for (int i = 0; i < 4; i++) pr[i] = __ldg(wp + i * ws);
          } else {
#pragma unroll
            for (int i = 0; i < 4; i++) pr[i] = __funnelshift_r(__ldg(wp + i * ws), __ldg(wp + i * ws + 1), sh);
          }
        } else {
          const int m = S.D[d], mx = mv_x(m), my = mv_y(m);
          DevPlane ph = ref;
          ph.p = ref.p + (long long)((my & 3) * 4 + (mx & 3)) * ref.phase;
          const int x = ox + tx * 4 + (mx >> 2), y = oy + ty * 4 + (my >> 2);
#pragma unroll
          for (int i = 0; i < 4; i++) {
            pr[i] = 0;
#pragma unroll
            for (int k = 0; k < 4; k++) pr[i] |= (uint32_t)at(ph, y + i, x + k) << (8 * k);
          }
        }
        sat[h] = satd4_rows(C, pr);
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        int v8 = sat[h] + __shfl_xor_sync(0xffffffffu, sat[h], 1);
        v8 += __shfl_xor_sync(0xffffffffu, v8, 16);
        if (dd + h < wnc) {
          Q.tile[dd + h][tid] = (unsigned short)sat[h];
          if (lane < 16 && !(lane & 1)) Q.whole8[dd + h][(tid >> 5) * 8 + (lane >> 1)] = (unsigned short)v8;
        }
      }
    }
    __syncthreads();
    // 16x16 sums (a 16x16 square lies in one region, so its four 8x8 sums exist wherever it is read)
    for (int k = tid; k < nc * 16; k += kInterThreads) {
      const int dd = k >> 4, i = k & 15, c = (i >> 2) * 16 + (i & 3) * 2;
      const unsigned short* W = Q.whole8[dd];
      Q.sum16[dd][i] = W[c] + W[c + 1] + W[c + 8] + W[c + 9];
    }
    __syncthreads();
    // 3. every candidate slot of a kept level whose MV (in its block's region) is in this chunk
    for (int k = slot_lo + tid; k < slot_hi; k += kInterThreads) {
      const unsigned aux = __ldg(g_slot_aux + k);
      if (!(keep & CELV2_KEEP_LEVEL(aux & 3u))) continue;
      const unsigned bp = __ldg(g_slot + k);
      const int d = (int)S.dmap[R == 32 ? (aux >> 2) & 3u : aux >> 4][bp >> 16] - c0;
      if (d < 0 || d >= nc) continue;
      const int b = bp & 511;
      atomicMin(&S.key[b], ((unsigned)block_satd(Q, b, d) << 7) | ((bp >> 9) & 127u));
    }
    __syncthreads();  // the next chunk overwrites the sums
  }
  int2* out = job.inter + ((long long)sb * kMaxRefs + r) * kBlocks;
  for (int b = tid; b < kBlocks; b += kInterThreads) {
    const unsigned aux = __ldg(g_block_aux + b);
    if (!(keep & CELV2_KEEP_LEVEL(aux & 3u))) continue;  // a pruned block: never read
    const int breg = R == 32 ? (aux >> 2) & 3u : aux >> 4;
    const unsigned k = S.key[b];
    out[b] = make_int2((int)(k >> 7), S.D[breg * ncell + S.dmap[breg][g_cand_cell[c_cand_off[b] + (k & 127)]]]);
  }
}

__global__ void __launch_bounds__(kInterThreads, 4) k_inter_regions(const FrameJob* __restrict__ jobs, WorkList w, int chunk) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RegionSmem& S = *reinterpret_cast<RegionSmem*>(smem_raw);
  const ChunkSums Q = chunk_sums(smem_raw, chunk);
  __shared__ int unit_slot[2];
  int unit, iter = 0;
  while (take_unit(w, unit, iter, unit_slot)) {
    const int jb = part_of(w, unit);
    const FrameJob& job = jobs[w.part[jb].job];
    const int nsb = w.part[jb].sbs;
    const int u = unit - w.prefix[jb];
    const int r = u / nsb, sb = w.part[jb].sb0 + u - r * nsb, sby = sb / job.sb_cols, sbx = sb - sby * job.sb_cols;
    const unsigned keep = keep_mask(job, sb);
    // a pruned (superblock, reference) is not scored; with 64-level blocks k_inter scores it
    if (!(keep >> r & 1u) || (keep & CELV2_KEEP_LEVEL(0))) continue;
    // regions: its 32x32 squares, or 16x16 ones where the 32-level blocks are pruned too
    if (keep & CELV2_KEEP_LEVEL(1))
      region_unit<32>(S, Q, job, r, sb, sbx, sby, keep, chunk);
    else
      region_unit<16>(S, Q, job, r, sb, sbx, sby, keep, chunk);
  }
}

void inter_window(unsigned& bytes, unsigned& rows) { bytes = kWinRow, rows = 64; }

// The whole-superblock kernel's groups: one group of 256 threads with 30 MVs' sums fits four CTAs on an
// SM, but a unit is then ~40 us of its CTA's time; with two groups a CTA has half an SM, with four all
// of it. us with one / two / four (stage events, 7 refs 67 MVs a unit): 84 units 43 / 33 / 31, 120 units
// 42 / 31 / 31, 420 units 68 / 63 / 74, 480 units 66 / 56 / 64, 3570 units 307 / 338 / 482 (a barrier
// holds more warps, and a unit's scans and sums leave more of them idle). So four while every unit has an
// SM, two while the units do not fill the GPU at four CTAs an SM.
template <int G>
static void launch_whole(const FrameJob* jobs, const WorkList& w, int chunk, cudaStream_t st) {
  // (a pass is whole rounds of the ring, so a unit's step s always has slot s % kRing)
  const int units = w.prefix[w.nparts], round = kRing * 2 * G, pass = std::max(1, std::min(chunk, G == 1 ? kPassG1 : kChunk) / round) * round;
  const size_t smem = whole_smem_bytes<G>(pass);
  const int grid = w.queue ? persistent_grid((const void*)k_inter<G>, kInterThreads * G, smem, units) : units;
  k_inter<G><<<grid, kInterThreads * G, smem, st>>>(jobs, w, pass);
}

void launch_inter(const FrameJob* jobs, const WorkList& w, int chunk, bool regions, unsigned* region_queue,
                  cudaStream_t st) {
  const int units = w.prefix[w.nparts];
  if (units <= 0) return;
  chunk = chunk < 8 ? 8 : chunk > kChunk ? kChunk : chunk;
  const int sms = persistent_grid((const void*)k_inter<4>, kInterThreads * 4, whole_smem_bytes<4>(kChunk), 1 << 30);
  const int g = units <= sms ? 4 : units <= 4 * sms ? 2 : 1;
  if (g == 4)
    launch_whole<4>(jobs, w, chunk, st);
  else if (g == 2)
    launch_whole<2>(jobs, w, chunk, st);
  else
    launch_whole<1>(jobs, w, chunk, st);
  if (!regions) return;  // no job has keep words: every unit keeps its 64-level blocks
  WorkList wr = w;
  wr.queue = w.queue ? region_queue : nullptr;
  const size_t smem = inter_smem_bytes(chunk);
  const int rgrid = wr.queue ? persistent_grid((const void*)k_inter_regions, kInterThreads, smem, units) : units;
  k_inter_regions<<<rgrid, kInterThreads, smem, st>>>(jobs, wr, chunk);
}

template <int G>
static cudaError_t whole_attributes() {
  const size_t most = whole_smem_bytes<G>(G == 1 ? kPassG1 : kChunk);
  const cudaError_t e = cudaFuncSetAttribute(k_inter<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
  if (e == cudaSuccess) persistent_grid((const void*)k_inter<G>, kInterThreads * G, most, 1);  // fills the grid cache
  return e;
}

cudaError_t inter_attributes() {
  short off[kBlocks];
  static unsigned slot[kSlots];
  static unsigned char cell[kSlots];
  static unsigned long long order[kSlots];  // sort key << 32 | slot
  int o = 0;
  for (int b = 0; b < kBlocks; b++) {
    int x, y, w, h;
    sb_block_geom(b, x, y, w, h);
    const int n = ((x + w - 1) / 8 - x / 8 + 1) * ((y + h - 1) / 8 - y / 8 + 1) + 8;
    const int sq = b / 5, size = sq >= 21 ? 3 : sq >= 5 ? 2 : sq >= 1 ? 1 : 0, kind = b - sq * 5;
    off[b] = (short)o;
    for (int k = 0; k < n && o + k < kSlots; k++) {
      const int c = candidate_cell(x, y, w, h, k);
      cell[o + k] = (unsigned char)c;
      const unsigned desc = (unsigned)b | (unsigned)k << 9 | (unsigned)c << 16;
      order[o + k] = (unsigned long long)(size << 19 | kind << 16 | k << 9 | b) << 32 | desc;
    }
    o += n;
  }
  if (o != kSlots) return cudaErrorInvalidValue;
  std::sort(order, order + kSlots);
  // level | 32x32 region << 2 | 16x16 region << 4 of a block (its region: where its top-left lies)
  auto aux_of = [](int b) {
    int x, y, w, h;
    sb_block_geom(b, x, y, w, h);
    return (unsigned char)(block_level(b) | ((y / 32) * 2 + x / 32) << 2 | ((y / 16) * 4 + x / 16) << 4);
  };
  static unsigned char slot_aux[kSlots];
  unsigned char block_aux[kBlocks];
  int level_slot[5] = {0, 0, 0, 0, kSlots};
  for (int b = 0; b < kBlocks; b++) block_aux[b] = aux_of(b);
  for (int e = 0; e < kSlots; e++) {
    slot[e] = (unsigned)order[e];
    slot_aux[e] = block_aux[slot[e] & 511];
  }
  for (int l = 1; l < 4; l++) {  // the first slot of level l (the slots are ordered by level)
    int e = 0;
    while (e < kSlots && (slot_aux[e] & 3) < l) e++;
    level_slot[l] = e;
  }
  if (level_slot[3] != kUpperSlots) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemcpyToSymbol(c_cand_off, off, sizeof off);
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_slot_aux, slot_aux, sizeof slot_aux);
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_block_aux, block_aux, sizeof block_aux);
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_level_slot, level_slot, sizeof level_slot);
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_cand_cell, cell, sizeof cell);
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_slot, slot, sizeof slot);
  if (e != cudaSuccess) return e;
  e = whole_attributes<1>();
  if (e == cudaSuccess) e = whole_attributes<2>();
  if (e == cudaSuccess) e = whole_attributes<4>();
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_inter_regions, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)inter_smem_bytes(kChunk));
  return e;
}

}  // namespace celv2cu
