// finalize.cu: per superblock, every block's best choice and the partition tree, written as the
// decision record (include/celv2_decision.h).
//
// Reference rules (src/gpu/kernels_ref.cpp): best_both / best_mode (:43-104) -- intra modes in
// order with mode bits (+32 in inter frames), each reference's best (from the inter stage), the
// best of the references and the second best (first strict minimum), the compound of the two
// (src/gpu/inter_common.h:199-220) when the pair is allowed, inter only where strictly cheaper than
// intra; the per-block records (:93-103); decide_square (:125-198) -- bottom-up NONE / HORZ /
// VERT / SPLIT, first strict minimum, the 64x64 square NONE / HORZ / VERT only in inter frames,
// 8x8 squares never split; the preorder tree with its leaves.
//
// One CTA per superblock: a thread per block for the choices, the compound SATDs as (block, tile)
// items reduced per block, then one warp for the partition DP and the preorder tree (bottom-up the
// costs, choices and subtree sizes, top-down the places, a lane a square), then all threads write the
// record with coalesced stores. Bound by the latency of its phases: five 1080p frames of 7 references
// (2,550 superblocks) 0.36 -> 0.24 ms, a 416x240 frame (28) 45 -> 25 us, the latter with 1,024
// threads a superblock (launch_finalize), against per-item plane look-ups, intra SATDs 13 apart, a
// barrier per DP level and one thread's walk of the tree.
#include <climits>
#include <cstddef>

#include "kernels.h"
#include "tables.h"

namespace celv2cu {

constexpr long long kMax = 0x7fffffffffffffffLL;

struct FinSmem {
  long long inter_cost[kBlocks];  // best single-reference cost (kMax: none)
  int inter_mv[kBlocks];
  long long best_cost[kBlocks];
  const uint8_t* comp_p[2][kBlocks];  // the compound's predictions at the block's origin (null: not inside the margins)
  int comp_mv[2][kBlocks];
  int comp_sum[kBlocks];
  int best_mv[kBlocks], best_mv2[kBlocks];
  unsigned char inter_ref[kBlocks], comp_ref[2][kBlocks];  // comp_ref[0] 255: no compound
  unsigned char best_mode[kBlocks], best_ref[kBlocks], best_ref2[kBlocks];
  long long sq_cost[CELV2_SB_SQUARES];
  // per square: its choice, its subtree's tree entries and leaves, and where they begin (-1: not in the tree)
  unsigned char sq_choice[CELV2_SB_SQUARES];
  short sq_nt[CELV2_SB_SQUARES], sq_nl[CELV2_SB_SQUARES], sq_t[CELV2_SB_SQUARES], sq_l[CELV2_SB_SQUARES];
  unsigned char tree[CELV2_SB_OUT_CAP];
  short leaf[CELV2_SB_OUT_CAP];
};

// hadamard4x4 of the byte residuals c - p of a 4x4 tile, rows as packed bytes: columns 0/2 and 1/3 ride as
// two 16-bit lanes through rows and columns, and the last row butterfly folds with the absolute values
// across the lanes (|x + y| + |x - y| = 2 max(|x|, |y|)); two registers' lanes change places so that the
// packed maxima take it for both, on values biased by 2048 as in satd4_pair.
__device__ __forceinline__ int satd4_lanes(const uint32_t* c, const uint32_t* p) {
  constexpr uint32_t B = 0x08000800u;
  uint32_t R[2][4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint32_t e = bytes_even(c[i]) - bytes_even(p[i]), o = bytes_odd(c[i]) - bytes_odd(p[i]);
    R[0][i] = e + o, R[1][i] = e - o;
  }
  uint32_t sum = 0;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const uint32_t* X = R[h];
    const uint32_t s01 = X[0] + X[1], d01 = X[0] - X[1], s23 = X[2] + X[3], d23 = X[2] - X[3];
    const uint32_t v0 = s01 + s23 + B, v1 = s01 - s23 + B, v2 = d01 + d23 + B, v3 = d01 - d23 + B;
    const uint32_t a0 = __byte_perm(v0, v1, 0x5410), b0 = __byte_perm(v0, v1, 0x7632);
    const uint32_t a1 = __byte_perm(v2, v3, 0x5410), b1 = __byte_perm(v2, v3, 0x7632);
    sum += max_u16x2(max_u16x2(a0, b0), 2 * B - min_u16x2(a0, b0)) + max_u16x2(max_u16x2(a1, b1), 2 * B - min_u16x2(a1, b1));
  }
  sum -= 4 * B;
  return 2 * (int)((sum & 0xffffu) + (sum >> 16));
}

template <int T>
__global__ void __launch_bounds__(T, 1024 / T) k_finalize(const FrameJob* __restrict__ jobs, WorkList w) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FinSmem& S = *reinterpret_cast<FinSmem*>(smem_raw);
  __shared__ int unit_slot[2];
  const int tid = threadIdx.x;
  int unit, iter = 0;
  while (take_unit(w, unit, iter, unit_slot)) {
  const int jb = part_of(w, unit);
  const FrameJob& job = jobs[w.part[jb].job];
  const int sb = w.part[jb].sb0 + unit - w.prefix[jb], sby = sb / job.sb_cols, sbx = sb - sby * job.sb_cols;
  const int ox = sbx * 64, oy = sby * 64;
  const int nrefs = job.nrefs;
  const long long lam = job.lam;
  celv2_sb_out* o = job.out + sb;
  const int2* inter = job.inter + (long long)sb * kMaxRefs * kBlocks;
  // pruned references, intra, block levels and intra modes are not candidates
  const unsigned keep = keep_mask(job, sb);

  // 1. each reference's best, the best two references, the records per reference
  unsigned comp_tiles = 0;  // work counter: compound 4x4 tiles
  for (int b = tid; b < kBlocks; b += T) {
    const bool live = keep & CELV2_KEEP_LEVEL(block_level(b));  // a block of a pruned level: no choice
    int2 v[kMaxRefs];
#pragma unroll
    for (int r = 0; r < kMaxRefs; r++)
      if (r < nrefs && live && (keep >> r & 1u)) v[r] = inter[r * kBlocks + b];
    long long ca = kMax, c2 = kMax;
    int a = -1, second = -1, mva = 0, mv2 = 0;
#pragma unroll
    for (int r = 0; r < kMaxRefs; r++) {
      const bool has = r < nrefs && live && (keep >> r & 1u);
      const long long rc = has ? (long long)v[r].x * 256 + lam * (kInterBits + r) : 0;
      const int mv = has ? v[r].y : 0;
      if (has) {  // the first strict minimum, and the first strict minimum of the others
        if (a < 0 || rc < ca) {
          second = a, c2 = ca, mv2 = mva;
          a = r, ca = rc, mva = mv;
        } else if (second < 0 || rc < c2) {
          second = r, c2 = rc, mv2 = mv;
        }
      }
      const long long c8 = rc >> 8;
      o->c_rcost[r][b] = has ? (unsigned)(c8 < 0xfffffffeLL ? c8 : 0xfffffffeLL) : CELV2_NO_REF_COST;
      o->c_rmvx[r][b] = (short)mv_x(mv);
      o->c_rmvy[r][b] = (short)mv_y(mv);
    }
    S.inter_cost[b] = a >= 0 ? ca : kMax;
    S.inter_mv[b] = mva;
    S.inter_ref[b] = (unsigned char)(a >= 0 ? a : 0);
    const bool comp = second >= 0 && compound_pair_ok(a, second, nrefs);
    S.comp_ref[0][b] = (unsigned char)(comp ? a : 255);
    if (comp) {
      int bx, by, bw, bh;
      sb_block_geom(b, bx, by, bw, bh);
      comp_tiles += (unsigned)(bw / 4) * (bh / 4);
      S.comp_ref[1][b] = (unsigned char)second;
      S.comp_mv[0][b] = mva, S.comp_mv[1][b] = mv2;
      S.comp_sum[b] = 0;
      bool in = true;
      const uint8_t* at_block[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const DevPlane& p = job.ref[h ? second : a].lv[0];
        const int m = h ? mv2 : mva, x = ox + bx + (mv_x(m) >> 2), y = oy + by + (mv_y(m) >> 2);
        in &= inside(p, x, y, bw, bh);
        at_block[h] = p.p + (long long)((mv_y(m) & 3) * 4 + (mv_x(m) & 3)) * p.phase + (long long)y * p.stride + x;
      }
      S.comp_p[0][b] = in ? at_block[0] : nullptr, S.comp_p[1][b] = at_block[1];
    }
  }
  if (job.stats) {  // one atomic per warp
    comp_tiles = __reduce_add_sync(0xffffffffu, comp_tiles);
    if ((tid & 31) == 0 && comp_tiles) atomicAdd(job.stats + kStatCompoundTiles, (unsigned long long)comp_tiles);
  }
  __syncthreads();

  // 2. compound SATDs (block_compound_satd): (cur - ((p0 + p1 + 1) >> 1)) per 4x4 tile
  if (nrefs >= 2) {
    const DevPlane& cur = job.cur.lv[0];
    const int stride = cur.stride;  // every plane of the engine's level 0 has it
    for (int item = tid; item < kItems; item += T) {
      int b, x, y, c0, r0, lwt;
      item_place(item, b, x, y, c0, r0, lwt);
      int v = 0;
      const bool comp = S.comp_ref[0][b] != 255;  // uniform over the block's segment
      if (comp) {
        const uint8_t* p0 = S.comp_p[0][b];
        const int cx = ox + x + c0, cy = oy + y + r0;
        if (p0) {
          const long long at_tile = (long long)r0 * stride + c0;
          const uint8_t *q0 = p0 + at_tile, *q1 = S.comp_p[1][b] + at_tile;
          const uint32_t* qc = reinterpret_cast<const uint32_t*>(cur.p + (long long)cy * stride + cx);
          uint32_t c[4], pr[4];
#pragma unroll
          for (int i = 0; i < 4; i++) {
            c[i] = __ldg(qc + i * (stride >> 2));
            pr[i] = __vavgu4(load4_pair(q0 + (long long)i * stride), load4_pair(q1 + (long long)i * stride));  // (a + q + 1) >> 1
          }
          v = satd4_lanes(c, pr);
        } else {
          const DevPlane &f0 = job.ref[S.comp_ref[0][b]].lv[0], &f1 = job.ref[S.comp_ref[1][b]].lv[0];
          const int m0 = S.comp_mv[0][b], m1 = S.comp_mv[1][b];
          uint32_t c[4], pr[4];
#pragma unroll 1
          for (int i = 0; i < 4; i++) {
            c[i] = pr[i] = 0;
#pragma unroll 1
            for (int j = 3; j >= 0; j--) {
              const int p = (at_q(f0, cy + i, cx + j, mv_y(m0), mv_x(m0)) + at_q(f1, cy + i, cx + j, mv_y(m1), mv_x(m1)) + 1) >> 1;
              pr[i] = pr[i] << 8 | (uint32_t)p, c[i] = c[i] << 8 | (uint32_t)at(cur, cy + i, cx + j);
            }
          }
          v = satd4_lanes(c, pr);
        }
      }
      // the block's tiles: 2 ^ lwt lanes, or the whole warp (uniform over it)
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
        if (off < 1 << lwt) v += __shfl_xor_sync(0xffffffffu, v, off);
      if (comp && (tid & ((1 << min(lwt, 5)) - 1)) == 0) {
        if (lwt <= 5) S.comp_sum[b] = v;
        else atomicAdd(&S.comp_sum[b], v);
      }
    }
    __syncthreads();
  }

  // 3. the block's inter choice (compound where strictly cheaper), intra choice, records, best
  const int* intra = job.intra + (long long)sb * kBlocks * kModes;
  for (int b = tid; b < kBlocks; b += T) {
    long long ci = S.inter_cost[b];
    int mv = S.inter_mv[b], ref = S.inter_ref[b], ref2 = CELV2_SINGLE_REF, mv2 = 0;
    const bool live = keep & CELV2_KEEP_LEVEL(block_level(b));
    const bool has_intra = b >= 5 && live && (keep & CELV2_KEEP_INTRA);
    int sat[kModes];
#pragma unroll
    for (int k = 0; k < kModes; k++) sat[k] = has_intra && (keep & CELV2_KEEP_MODE(k)) ? intra[k * kBlocks + b] : 0;
    if (S.comp_ref[0][b] != 255) {
      const int ra = S.comp_ref[0][b], rb = S.comp_ref[1][b];
      const long long cc = (long long)S.comp_sum[b] * 256 + lam * (20 + ra + rb);
      if (cc < ci) ci = cc, ref2 = rb, mv2 = S.comp_mv[1][b];
    }
    long long c = kMax;
    int m = 0;
    if (has_intra) {
#pragma unroll
      for (int k = 0; k < kModes; k++) {
        const long long ck = (long long)sat[k] * 256 + lam * (mode_bits(k) + (nrefs > 0 ? kIntraInInterBits : 0));
        if ((keep & CELV2_KEEP_MODE(k)) && ck < c) c = ck, m = k;
      }
    }
    o->c_inter_cost[b] = ci;
    o->c_intra_cost[b] = c;
    o->c_intra[b] = (unsigned char)m;
    o->c_mvx[b] = (short)mv_x(mv), o->c_mvy[b] = (short)mv_y(mv);
    o->c_ref[b] = (unsigned char)ref, o->c_ref2[b] = (unsigned char)ref2;
    o->c_mv2x[b] = (short)mv_x(mv2), o->c_mv2y[b] = (short)mv_y(mv2);
    const bool take_inter = ci < c;
    S.best_cost[b] = live ? (take_inter ? ci : c) : CELV2_PRUNED_COST;
    S.best_mode[b] = (unsigned char)(take_inter ? kModes : m);
    S.best_mv[b] = take_inter ? mv : 0;
    S.best_ref[b] = (unsigned char)(take_inter ? ref : 0);
    S.best_ref2[b] = (unsigned char)(take_inter ? ref2 : CELV2_SINGLE_REF);
    S.best_mv2[b] = take_inter ? mv2 : 0;
  }
  __syncthreads();

  if (tid < 32) {
    // 4. partition choice bottom-up (decide_square), with the sizes of each square's part of the tree
    const long long part = lam * kPartBits;
#pragma unroll
    for (int level = 3; level >= 0; level--) {
      const int n = 1 << level, size = 64 >> level;
      for (int i = tid; i < n * n; i += 32) {
        const int sq = sb_level_offset(level) + i, b = sq * 5;
        long long c = kMax;
        int ch = 3, nt = 1, nl = 0;
        if (size <= 32 || nrefs > 0) {
          const long long horz = part + S.best_cost[b + 1] + S.best_cost[b + 2];
          const long long vert = part + S.best_cost[b + 3] + S.best_cost[b + 4];
          c = S.best_cost[b], ch = 0;
          if (horz < c) c = horz, ch = 1;
          if (vert < c) c = vert, ch = 2;
        }
        if (level < 3) {
          const int qx = i & (n - 1), qy = i >> level, c0 = sb_level_offset(level + 1) + 2 * qy * (2 * n) + 2 * qx;
          const long long split = part + S.sq_cost[c0] + S.sq_cost[c0 + 1] + S.sq_cost[c0 + 2 * n] + S.sq_cost[c0 + 2 * n + 1];
          if (split < c) c = split, ch = 3;
          if (ch == 3) {
            nt += S.sq_nt[c0] + S.sq_nt[c0 + 1] + S.sq_nt[c0 + 2 * n] + S.sq_nt[c0 + 2 * n + 1];
            nl = S.sq_nl[c0] + S.sq_nl[c0 + 1] + S.sq_nl[c0 + 2 * n] + S.sq_nl[c0 + 2 * n + 1];
          }
        }
        if (ch == 0) nl = 1;
        if (ch == 1 || ch == 2) nt = 3, nl = 2;
        S.sq_cost[sq] = c, S.sq_choice[sq] = (unsigned char)ch;
        S.sq_nt[sq] = (short)nt, S.sq_nl[sq] = (short)nl, S.sq_t[sq] = -1;
      }
      __syncwarp();
    }
    // 5. the preorder tree and its leaves, top-down
    if (tid == 0) {
      if (job.sb_cost) job.sb_cost[sb] = S.sq_cost[0];
      S.sq_t[0] = S.sq_l[0] = 0;
      o->ntree = S.sq_nt[0], o->nblocks = S.sq_nl[0];
      // the record's padding bytes
      reinterpret_cast<unsigned char*>(o)[offsetof(celv2_sb_out, c_rcost) - 1] = 0;
      *reinterpret_cast<unsigned*>(reinterpret_cast<unsigned char*>(o) + sizeof(celv2_sb_out) - 4) = 0;
    }
    __syncwarp();
#pragma unroll
    for (int level = 0; level < 4; level++) {
      const int n = 1 << level;
      for (int i = tid; i < n * n; i += 32) {
        const int sq = sb_level_offset(level) + i, b = sq * 5, ch = S.sq_choice[sq];
        int t = S.sq_t[sq], l = S.sq_l[sq];
        if (t < 0) continue;  // inside a larger leaf
        S.tree[t++] = (unsigned char)ch;
        if (ch == 0) {
          S.leaf[l] = (short)b;
        } else if (ch < 3) {
          const int k = ch == 1 ? 1 : 3;
          S.tree[t] = S.tree[t + 1] = 0;
          S.leaf[l] = (short)(b + k), S.leaf[l + 1] = (short)(b + k + 1);
        } else if (level < 3) {
          const int qx = i & (n - 1), qy = i >> level, c0 = sb_level_offset(level + 1) + 2 * qy * (2 * n) + 2 * qx;
          for (int q = 0; q < 4; q++) {
            const int c = c0 + (q >> 1) * (2 * n) + (q & 1);
            S.sq_t[c] = (short)t, S.sq_l[c] = (short)l;
            t += S.sq_nt[c], l += S.sq_nl[c];
          }
        }
      }
      __syncwarp();
    }
  }
  __syncthreads();
  // 6. tree and leaf fields, zero past the end
  const int ntree = S.sq_nt[0], nblocks = S.sq_nl[0];
  for (int k = tid; k < CELV2_SB_OUT_CAP; k += T) {
    o->tree[k] = k < ntree ? S.tree[k] : 0;
    if (k < nblocks) {
      const int b = S.leaf[k];
      int x, y, bw, bh;
      sb_block_geom(b, x, y, bw, bh);
      const bool in = S.best_mode[b] == kModes;
      const bool two = in && S.best_ref2[b] != CELV2_SINGLE_REF;
      o->w4[k] = (unsigned char)(bw / 4), o->h4[k] = (unsigned char)(bh / 4);
      o->mode[k] = S.best_mode[b];
      o->mvx[k] = (short)(in ? mv_x(S.best_mv[b]) : 0), o->mvy[k] = (short)(in ? mv_y(S.best_mv[b]) : 0);
      o->ref[k] = in ? S.best_ref[b] : 0;
      o->ref2[k] = (unsigned char)(two ? S.best_ref2[b] : CELV2_SINGLE_REF);
      o->mv2x[k] = (short)(two ? mv_x(S.best_mv2[b]) : 0), o->mv2y[k] = (short)(two ? mv_y(S.best_mv2[b]) : 0);
    } else {
      o->w4[k] = o->h4[k] = o->mode[k] = 0;
      o->mvx[k] = o->mvy[k] = 0;
      o->ref[k] = o->ref2[k] = 0;
      o->mv2x[k] = o->mv2y[k] = 0;
    }
  }
  }  // units
}

template <int T>
static void launch_t(const FrameJob* jobs, const WorkList& w, int units, cudaStream_t st) {
  const int grid = w.queue ? persistent_grid((const void*)k_finalize<T>, T, sizeof(FinSmem), units) : units;
  k_finalize<T><<<grid, T, sizeof(FinSmem), st>>>(jobs, w);
}

// A launch of at most one superblock per SM gives each all of its SM.
void launch_finalize(const FrameJob* jobs, const WorkList& w, cudaStream_t st) {
  const int units = w.prefix[w.nparts];
  if (units <= 0) return;
  if (units <= persistent_grid((const void*)k_finalize<1024>, 1024, sizeof(FinSmem), INT_MAX))
    launch_t<1024>(jobs, w, units, st);
  else
    launch_t<256>(jobs, w, units, st);
}

template <int T>
static cudaError_t attributes_t() {
  const cudaError_t e = cudaFuncSetAttribute(k_finalize<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FinSmem));
  if (e == cudaSuccess) persistent_grid((const void*)k_finalize<T>, T, sizeof(FinSmem), 1);  // fills the grid cache
  return e;
}

cudaError_t finalize_attributes() {
  const cudaError_t e = attributes_t<256>();
  return e == cudaSuccess ? attributes_t<1024>() : e;
}

}  // namespace celv2cu
