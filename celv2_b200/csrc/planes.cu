// planes.cu: the engine's input planes in HBM -- 8-bit luma with replicated margins, its 2x2
// pyramid and a reference's quarter-pel phase planes.
//
// Reference rules: round_to_8bit (src/io/y4m.cpp:28-34), build_pyramid_ref
// (src/gpu/kernels_ref.cpp:213-238), downsample_px and subpel_px (src/gpu/inter_common.h:13-33,
// 91-94). Every kernel writes the whole stored extent of its planes, margin included: the value at
// a margin position is the plane's value at the clamped position, which is what the reference's
// clamped reads return (for phase planes: the phase value at the clamped whole-pel position).
// Both take the planes of a launch (blockIdx.z), so a frame's new references go together.
#include <algorithm>

#include "kernels.h"

namespace celv2cu {

// ---- level 0 and the pyramid ----
// One CTA per 64 x 64 tile of stored positions (level 0's margin is five tiles), all five levels: a
// sample of level l is made of the 2^l x 2^l samples below it, so a tile inside the frame needs only
// its own; a margin tile repeats samples of the frame's nearest tile, which it makes again rather
// than wait for. Five launches -- expand and four downsamples, each a pass over the level before,
// a byte a thread -- were 22 us for a 1080p plane and 18 us for a 202x122 one, a launch's latency
// each; this one is 8 and 4.
constexpr int kPyTile = 64, kPyExt = 16, kPySide = kPyTile + kPyExt;

__device__ __forceinline__ int round8(int v, int shift) {
  return min(255, shift > 0 ? (v + (1 << (shift - 1))) >> shift : v);
}

__global__ void __launch_bounds__(256) k_pyramid(PlaneSet set) {
  const PlaneIn& in = set.p[blockIdx.z];
  const DevPlane& l0 = in.pyr.lv[0];
  const int pw = l0.w, ph = l0.h;
  const int X0 = (int)blockIdx.x * kPyTile - l0.margin, Y0 = (int)blockIdx.y * kPyTile - l0.margin;
  if (X0 >= pw + l0.margin || Y0 >= ph + l0.margin) return;  // a smaller plane of the set
  // the frame's tile this one shows, from 16 samples further up or left where the last tile is one
  // 8-sample column (row) wide: level 4's last sample then lies before it
  const int lastx = (pw - 1) & ~(kPyTile - 1), lasty = (ph - 1) & ~(kPyTile - 1);
  const int xs = clampi(X0, 0, lastx), ys = clampi(Y0, 0, lasty);
  const int rx = xs - (xs == lastx && xs > 0 && pw - xs < 16 ? kPyExt : 0);
  const int ry = ys - (ys == lasty && ys > 0 && ph - ys < 16 ? kPyExt : 0);
  __shared__ uint32_t s0[kPySide * kPySide / 4];
  __shared__ uint8_t s1[kPySide / 2][kPySide / 2], s2[kPySide / 4][kPySide / 4], s3[kPySide / 8][kPySide / 8 + 2],
      s4[kPySide / 16][kPySide / 16 + 3];
  const int tid = threadIdx.x;
  // level 0 of the region, four samples a thread (the frame is a multiple of 8 wide: a group of four
  // lies inside it or outside; rows of the packed upload are 8-byte aligned)
  const int nx = min(kPySide, pw - rx) >> 2, ny = min(kPySide, ph - ry);
  for (int e = tid; e < kPySide * kPySide / 4; e += 256) {
    const int r = e / (kPySide / 4), c = e - r * (kPySide / 4);
    if (c >= nx || r >= ny) continue;
    const long long o = (long long)(ry + r) * pw + rx + 4 * c;
    if (in.shift < 0) {  // 8-bit samples
      s0[e] = *reinterpret_cast<const uint32_t*>(static_cast<const uint8_t*>(in.raw) + o);
    } else {
      const ushort4 v = *reinterpret_cast<const ushort4*>(static_cast<const uint16_t*>(in.raw) + o);
      s0[e] = (uint32_t)round8(v.x, in.shift) | (uint32_t)round8(v.y, in.shift) << 8 |
              (uint32_t)round8(v.z, in.shift) << 16 | (uint32_t)round8(v.w, in.shift) << 24;
    }
  }
  __syncthreads();
  // levels 1-4: (a + b + c + d + 2) >> 2 of the 2 x 2 samples below (those past the frame's last whole
  // sample hold nothing and are not shown)
  for (int e = tid; e < kPySide / 2 * (kPySide / 4); e += 256) {  // two samples a thread
    const int r = e / (kPySide / 4), c = e - r * (kPySide / 4);
    const uint32_t a = s0[2 * r * (kPySide / 4) + c], b = s0[(2 * r + 1) * (kPySide / 4) + c];
    const uint32_t v = (a & 0x00ff00ffu) + ((a >> 8) & 0x00ff00ffu) + (b & 0x00ff00ffu) + ((b >> 8) & 0x00ff00ffu) + 0x00020002u;
    s1[r][2 * c] = (uint8_t)(v >> 2), s1[r][2 * c + 1] = (uint8_t)(v >> 18);
  }
  __syncthreads();
  for (int e = tid; e < (kPySide / 4) * (kPySide / 4); e += 256) {
    const int r = e / (kPySide / 4), c = e - r * (kPySide / 4);
    s2[r][c] = (uint8_t)((s1[2 * r][2 * c] + s1[2 * r][2 * c + 1] + s1[2 * r + 1][2 * c] + s1[2 * r + 1][2 * c + 1] + 2) >> 2);
  }
  __syncthreads();
  if (tid < (kPySide / 8) * (kPySide / 8)) {
    const int r = tid / (kPySide / 8), c = tid - r * (kPySide / 8);
    s3[r][c] = (uint8_t)((s2[2 * r][2 * c] + s2[2 * r][2 * c + 1] + s2[2 * r + 1][2 * c] + s2[2 * r + 1][2 * c + 1] + 2) >> 2);
  }
  __syncthreads();
  if (tid < (kPySide / 16) * (kPySide / 16)) {
    const int r = tid / (kPySide / 16), c = tid - r * (kPySide / 16);
    s4[r][c] = (uint8_t)((s3[2 * r][2 * c] + s3[2 * r][2 * c + 1] + s3[2 * r + 1][2 * c] + s3[2 * r + 1][2 * c + 1] + 2) >> 2);
  }
  __syncthreads();
  // the stored positions of this tile at each level, a word a thread (margins, strides and tile
  // origins are multiples of 4 at every level; a row's last word may run into its stride's slack).
  // The outermost tiles show the rest of level 4's margin too, which is wider than theirs / 16.
  const bool fx = blockIdx.x == 0, lx = X0 + kPyTile >= pw + l0.margin;
  const bool fy = blockIdx.y == 0, ly = Y0 + kPyTile >= ph + l0.margin;
#pragma unroll
  for (int l = 0; l < kLevels; l++) {
    const DevPlane& p = in.pyr.lv[l];
    const int x0 = fx ? -p.margin : X0 >> l, x1 = lx ? p.w + p.margin : (X0 + kPyTile) >> l;
    const int y0 = fy ? -p.margin : Y0 >> l, y1 = ly ? p.h + p.margin : (Y0 + kPyTile) >> l;
    const int words = (x1 - x0 + 3) >> 2, n = words * (y1 - y0);
    const int bx = rx >> l, by = ry >> l;
    uint8_t* dst = const_cast<uint8_t*>(p.p);
    for (int e = tid; e < n; e += 256) {
      const int r = e / words, c = e - r * words, x = x0 + 4 * c, y = y0 + r;
      const int sy = clampi(y, 0, max(p.h - 1, 0)) - by;  // (level 4 of an 8-sample frame has no sample)
      uint32_t v;
      if (l == 0) {  // inside or outside the frame as a whole
        const int sx = clampi(x, 0, p.w - 4) - bx;
        v = s0[sy * (kPySide / 4) + (sx >> 2)];
        if (x < 0) v = __byte_perm(v, 0, 0x0000);
        if (x >= p.w) v = __byte_perm(v, 0, 0x3333);
      } else {
        v = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int sx = clampi(x + k, 0, max(p.w - 1, 0)) - bx;
          v |= (uint32_t)(l == 1 ? s1[sy][sx] : l == 2 ? s2[sy][sx] : l == 3 ? s3[sy][sx] : s4[sy][sx]) << (8 * k);
        }
      }
      *reinterpret_cast<uint32_t*>(dst + (long long)y * p.stride + x) = v;
    }
  }
}

// ---- quarter-pel phases ----
// AV2 EIGHTTAP_REGULAR at the quarter phases (src/gpu/inter_common.h:13-19): taps 1-6 as signed bytes
// (taps 0 and 7 are zero at every phase; phase 0 is 128 at tap 3).
__host__ __device__ constexpr int tap(int q, int j) {
  return q == 1 ? (j == 1 ? 2 : j == 2 ? -14 : j == 3 ? 110 : j == 4 ? 38 : j == 5 ? -10 : 2)
         : q == 2 ? (j == 1 || j == 6 ? 2 : j == 2 || j == 5 ? -14 : 76)
                  : (j == 1 ? 2 : j == 2 ? -10 : j == 3 ? 38 : j == 4 ? 110 : j == 5 ? -14 : 2);
}
__device__ constexpr uint32_t tap_bytes(int q, int j, int n) {
  uint32_t v = 0;
  for (int k = 0; k < n; k++) v |= (uint32_t)(uint8_t)(int8_t)tap(q, j + k) << (8 * k);
  return v;
}

__device__ __forceinline__ int dp4a_ss(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp4a.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ int dp2a_ss(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp2a.lo.s32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
// Four values clamped to 0 .. 255 as bytes, the first in the low byte.
__device__ __forceinline__ uint32_t pack_sat(int a, int b, int c, int d) {
  uint32_t lo, v;
  asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, 0;" : "=r"(lo) : "r"(d), "r"(c));
  asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(v) : "r"(b), "r"(a), "r"(lo));
  return v;
}

// The 15 quarter-pel phase planes of level 0 (phase k at lv0.p + k * lv0.phase), separably: one CTA per
// 128 x 32 tile of stored positions, one thread per 4 x 4 of them, so a warp stores 128 bytes of a row
// at a time. The samples minus 128 fit a signed byte and their horizontal sums (taps' absolute sum
// at most 176) a signed halfword, which lets dp4a form the sums and dp2a combine two rows of them a
// step: 576 dp2a for 240 outputs instead of 1,440 multiply-adds. The offsets of 128 come back in the
// last accumulator's start (the taps sum to 128: 128^3 in all). The frame's sides are multiples of 8, so
// a 4 x 4 group lies inside the frame or outside it in x and in y; an outside group makes its nearest
// inside group's and repeats the edge column or row. Writes bound it: a 1080p reference (66 MB of
// planes) 60 -> 20 us against a byte a thread and 32-bit sums.
constexpr int kPhTW = 128, kPhTH = 32, kPhPairs = (kPhTH + 6) / 2, kPhSrcWords = kPhTW / 4 + 2;

__global__ void __launch_bounds__(256) k_subpel_phases(PlaneSet set) {
  const DevPlane& lv0 = set.p[blockIdx.z].pyr.lv[0];
  __shared__ uint32_t src[2 * kPhPairs][kPhSrcWords];  // rows cy0 - 2 .., columns cx0 - 4 .., minus 128
  __shared__ __align__(16) uint32_t hs[4][kPhPairs][kPhTW];  // per phase qx and pair of rows: two horizontal sums
  const int tid = threadIdx.x, W = lv0.w, H = lv0.h, M = lv0.margin;
  const int X0 = (int)blockIdx.x * kPhTW - M, Y0 = (int)blockIdx.y * kPhTH - M;
  if (X0 >= W + M || Y0 >= H + M) return;  // a smaller plane of the set
  const int cx0 = clampi(X0, 0, W - 4), cy0 = clampi(Y0, 0, H - 4);  // the first group shown
  for (int e = tid; e < 2 * kPhPairs * kPhSrcWords; e += 256) {
    const int r = e / kPhSrcWords, c = e - r * kPhSrcWords;
    // every sample a shown group needs lies inside the margin; the rest of the tile's window is clamped
    const int y = min(cy0 - 2 + r, H + M - 1), x = min(cx0 - 4 + 4 * c, W + M - 4);
    src[r][c] = *reinterpret_cast<const uint32_t*>(lv0.p + (long long)y * lv0.stride + x) ^ 0x80808080u;
  }
  __syncthreads();
  for (int e = tid; e < kPhPairs * (kPhTW / 4); e += 256) {
    const int rp = e / (kPhTW / 4), cg = e - rp * (kPhTW / 4);  // a pair of rows, four columns
    uint4 out[4];
    uint32_t* o = reinterpret_cast<uint32_t*>(out);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t* s = &src[2 * rp + h][cg];
      const uint32_t w0 = s[0], w1 = s[1], w2 = s[2];  // columns 4 cg - 4 .. 4 cg + 7 from cx0
#pragma unroll
      for (int k = 0; k < 4; k++) {
        // the six samples c - 2 .. c + 3 of column c = 4 cg + k: bytes k + 2 .. k + 7 of the three words
        const uint32_t a = k < 2 ? __funnelshift_r(w0, w1, 8 * (k + 2)) : k == 2 ? w1 : __funnelshift_r(w1, w2, 8);
        const uint32_t b = k < 2 ? __funnelshift_r(w1, w2, 8 * (k + 2)) : k == 2 ? w2 : w2 >> 8;  // bytes k + 6, k + 7
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int v = q == 0 ? (int)(int8_t)(w1 >> (8 * k)) * 128
                               : dp4a_ss(b, tap_bytes(q, 5, 2), dp4a_ss(a, tap_bytes(q, 1, 4), 0));
          if (h == 0) o[4 * q + k] = (uint32_t)v & 0xffffu;
          else o[4 * q + k] |= (uint32_t)v << 16;
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) *reinterpret_cast<uint4*>(&hs[q][rp][4 * cg]) = out[q];
  }
  __syncthreads();
  const int gx = tid & 31, gy = tid >> 5, x = X0 + 4 * gx, y = Y0 + 4 * gy;
  if (x >= W + M || y >= H + M) return;
  const int cx = clampi(x, 0, W - 4) - cx0, rp0 = (clampi(y, 0, H - 4) - cy0) >> 1;
  uint8_t* base = const_cast<uint8_t*>(lv0.p) + (long long)y * lv0.stride + x;
  constexpr int kStart = (1 << 21) + (1 << 13);  // the offsets' share of a sum, and its rounding
#pragma unroll 1
  for (int qx = 0; qx < 4; qx++) {
    uint4 pr[5];  // rows 2 i, 2 i + 1 of the group's ten, four columns
#pragma unroll
    for (int i = 0; i < 5; i++) pr[i] = *reinterpret_cast<const uint4*>(&hs[qx][rp0 + i][cx]);
#pragma unroll
    for (int qy = 0; qy < 4; qy++) {
      if (qy == 0 && qx == 0) continue;
      uint32_t row[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        int v[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const auto word = [&](int i) { return reinterpret_cast<const uint32_t*>(&pr[i])[c]; };
          if (qy == 0) {  // the centre row alone: 128 times its sum, a row of the third word or the two beside it
            const int r = k + 2;
            const int h = r & 1 ? (int)word(r >> 1) >> 16 : (int)(short)(word(r >> 1) & 0xffffu);
            v[c] = (h * 128 + kStart) >> 14;
          } else {
            int s = kStart;
#pragma unroll
            for (int i = 0; i < 3; i++) {
              const int r = k + 2 * i;  // rows r, r + 1
              const uint32_t w = r & 1 ? __byte_perm(word(r >> 1), word((r >> 1) + 1), 0x5432) : word(r >> 1);
              s = dp2a_ss(w, tap_bytes(qy, 1 + 2 * i, 2), s);
            }
            v[c] = s >> 14;
          }
        }
        row[k] = pack_sat(v[0], v[1], v[2], v[3]);
      }
      if (x < 0 || x >= W) {
        const uint32_t sel = x < 0 ? 0x0000u : 0x3333u;
#pragma unroll
        for (int k = 0; k < 4; k++) row[k] = __byte_perm(row[k], 0, sel);
      }
      if (y < 0) row[1] = row[2] = row[3] = row[0];
      if (y >= H) row[0] = row[1] = row[2] = row[3];
      uint8_t* p = base + (long long)(4 * qy + qx) * lv0.phase;
#pragma unroll
      for (int k = 0; k < 4; k++) *reinterpret_cast<uint32_t*>(p + (long long)k * lv0.stride) = row[k];
    }
  }
}

// The grid over the largest plane of the set, tiles of tw x th stored positions.
static dim3 set_grid(const PlaneSet& s, int tw, int th) {
  int w = 0, h = 0;
  for (int i = 0; i < s.n; i++) {
    const DevPlane& p = s.p[i].pyr.lv[0];
    w = std::max(w, p.w + 2 * p.margin), h = std::max(h, p.h + 2 * p.margin);
  }
  return dim3((w + tw - 1) / tw, (h + th - 1) / th, s.n);
}

void launch_pyramid(const PlaneSet& s, cudaStream_t st) {
  if (s.n > 0) k_pyramid<<<set_grid(s, kPyTile, kPyTile), 256, 0, st>>>(s);
}

void launch_phases(const PlaneSet& s, cudaStream_t st) {
  if (s.n > 0) k_subpel_phases<<<set_grid(s, kPhTW, kPhTH), 256, 0, st>>>(s);
}

}  // namespace celv2cu
