// Device helpers shared by the chain's SAO / ALF / CC-ALF tile kernel
// (sao_alf3.cu) and the encoder's luma ALF trial kernel (sao_alf2.cu).
//
// Packed filters (AlfTablesDev::luma_packed / chroma_packed): two 16-bit clip
// values c a word (2^14 as 2^14 - 1, the same for samples below 2^14), four
// coefficients a word, and the accumulator start -sum(2 c f) of the offset form
// below.  A thread's luma filter is 48 bytes, three 16-byte loads (lanes of a
// warp read different entries, so each load costs its distinct lines; a word
// per clip, coefficient and negated clip cost 24 loads from 144 bytes).
// Expanded for use: c in both 16-bit lanes, and the coefficient as a signed
// byte in bytes 0 and 3, so that dp2a.lo weights the low lane of a packed pair
// of tap sums and dp2a.hi the high lane.
//
// Offset form of the clipped taps: clip(n - cur, -c, c) + c lies in [0, 2c] and
// is max(min(n + (c - cur), 2c), 0), one instruction per pair of samples
// (viaddmin with relu) where the plain form takes two, and two of them add
// without a carry between the lanes, so the sum is an ordinary add and leaves
// the ALU pipe (64 lanes a clock, the pass's bound) to the clips; dp2a runs on
// the FMA pipe.  The 2c that every tap sum carries is in the accumulator
// start.  c - cur is formed lane-wise by one 32-bit add from
// 0x8000 - cur (no borrow), which leaves 0x8000 in each lane; the windows hold
// samples + 0x8000 (kBias) to cancel it.  Samples of 2^14 and above, outside
// any supported depth, would wrap: tiles that hold one take the plain form.
#pragma once

#include <initializer_list>
#include <type_traits>
#include <utility>

#include "internal.h"

namespace h266 {
namespace tile {

__device__ __forceinline__ int clampd(int v, int lo, int hi) { return min(max(v, lo), hi); }
__device__ __forceinline__ int sgn(int v) { return (v > 0) - (v < 0); }

// One component's SAO parameters of one CTB in the form the per-sample step
// needs: band offsets; for edge offset the offset per 2 + sign + sign (the
// edgeIdx remap of eq. 154 folded in), the shared-memory offset of the first
// neighbour (the second is its negation), and the rectangle of samples whose
// two neighbours lie inside the picture and the clip rectangle.  tlo / thi
// hold the same offsets as a signed-byte table (bytes 0..3 of tlo, then thi)
// indexed by the band index 0..3 (4 = no offset) or by 2 - sign - sign.
struct SaoLocal {
  int type, band, bd_shift;
  int off[4];   // band offset per band index 0..3 after the band position
  int eo[5];    // edge offset per 2 + sign(c - a) + sign(c - b)
  int nb;       // smem offset of the first neighbour (row pitch of the component's window)
  int ex0, ey0, ex1, ey1;  // [ex0, ex1) x [ey0, ey1): both neighbours available
  uint32_t tlo, thi;
};

// Fills one SaoLocal from the CTB's SAO parameters (src/sao.rs:504-626):
// hPos / vPos of eq. 152 per class, and the clip rectangle `rect` (component
// samples) intersected with the picture.
__device__ __forceinline__ void sao_local(SaoLocal &s, const SaoCtbDev &p, int pitch, int rx0, int ry0, int rx1,
                                          int ry1, int bd) {
  s.type = p.type;
  s.band = p.band_pos;
  s.bd_shift = bd - 5;
  for (int k = 0; k < 4; ++k) s.off[k] = p.off[k];
  // edgeIdx = 2 + sign + sign, remapped 0 -> 1, 1 -> 2, 2 -> 0 (eq. 154); offset edgeIdx - 1
  s.eo[0] = p.off[0];
  s.eo[1] = p.off[1];
  s.eo[2] = 0;
  s.eo[3] = p.off[2];
  s.eo[4] = p.off[3];
  const int h0 = p.eo_class == 0 ? -1 : (p.eo_class == 1 ? 0 : (p.eo_class == 2 ? -1 : 1));
  const int v0 = p.eo_class == 0 ? 0 : -1;
  s.nb = v0 * pitch + h0;
  const int ah = h0 < 0 ? -h0 : h0, av = v0 < 0 ? -v0 : v0;
  s.ex0 = rx0 + ah;
  s.ex1 = rx1 - ah;
  s.ey0 = ry0 + av;
  s.ey1 = ry1 - av;
  auto b = [](int v) { return (uint32_t)(v & 0xFF); };
  if (p.type == 1) {
    s.tlo = b(p.off[0]) | b(p.off[1]) << 8 | b(p.off[2]) << 16 | b(p.off[3]) << 24;
    s.thi = 0;
  } else {  // indexed by (1 - sign) + (1 - sign): eo[] backwards
    s.tlo = b(s.eo[4]) | b(s.eo[3]) << 8 | b(s.eo[2]) << 16 | b(s.eo[1]) << 24;
    s.thi = b(s.eo[0]);
  }
}

// §8.8.4.2 for one sample at (x, y) whose pre-SAO value is *d (shared memory).
__device__ __forceinline__ int sao_one(const SaoLocal &p, int x, int y, int maxv, const uint16_t *d) {
  const int c = *d;
  if (p.type == 1) {
    const int k = ((c >> p.bd_shift) - p.band) & 31;
    return clampd(k < 4 ? c + p.off[k] : c, 0, maxv);
  }
  if (x < p.ex0 || x >= p.ex1 || y < p.ey0 || y >= p.ey1) return clampd(c, 0, maxv);
  return clampd(c + p.eo[2 + sgn(c - d[p.nb]) + sgn(c - d[-p.nb])], 0, maxv);
}

// Pair of samples (col, col + 1) of a shared-memory row; DC fixes the parity
// of col (col = even base + DC).
template <int DC>
__device__ __forceinline__ uint32_t pair_at(const uint16_t *row, int even_base) {
  const int col = even_base + DC;
  if constexpr ((DC & 1) == 0) {
    return *reinterpret_cast<const uint32_t *>(row + col);
  } else {
    const uint32_t a = *reinterpret_cast<const uint32_t *>(row + col - 1);
    const uint32_t b = *reinterpret_cast<const uint32_t *>(row + col + 1);
    return __byte_perm(a, b, 0x5432);
  }
}

// clip(n - cur, -c, c) for both 16-bit lanes
__device__ __forceinline__ uint32_t clipd(uint32_t n, uint32_t ncur, uint32_t c2, uint32_t nc2) {
  return __viaddmin_s16x2(__viaddmax_s16x2(n, ncur, nc2), 0u, c2);
}
__device__ __forceinline__ uint32_t add2(uint32_t a, uint32_t b) { return __viaddmax_s16x2(a, b, 0x80008000u); }
__device__ __forceinline__ uint32_t neg2(uint32_t a) { return __viaddmax_s16x2(~a, 0x00010001u, 0x80008000u); }

constexpr uint32_t kBias = 0x80008000u;  // the windows' samples are stored with 0x8000 added in each lane

// clip(n - cur, -c, c) + c for both lanes: nb the biased pair, b = c - cur + 0x8000 per lane, c22 = 2c per lane
__device__ __forceinline__ uint32_t clip_off(uint32_t nb, uint32_t b, uint32_t c22) {
  return __viaddmin_s16x2_relu(nb, b, c22);
}
// acc + the low (high) lane of the unsigned pair s times the signed byte 0 (3) of f
__device__ __forceinline__ int dp2a_ulo(uint32_t s, uint32_t f, int acc) {
  int r;
  asm("dp2a.lo.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(s), "r"(f), "r"(acc));
  return r;
}
__device__ __forceinline__ int dp2a_uhi(uint32_t s, uint32_t f, int acc) {
  int r;
  asm("dp2a.hi.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(s), "r"(f), "r"(acc));
  return r;
}
// Clip value k of packed words in both lanes; coefficient k of packed words in bytes 0 and 3.
__device__ __forceinline__ uint32_t clip_of(const uint32_t *w, int k) {
  return __byte_perm(w[k / 2], 0u, (k & 1) ? 0x3232 : 0x1010);
}
__device__ __forceinline__ uint32_t coef_of(const uint32_t *w, int k) {
  return __byte_perm(w[k / 4], 0u, 0x0440u + 0x1001u * (k & 3));
}
// The expanded clips and coefficients of packed luma entry `e`; returns the accumulator start.
__device__ __forceinline__ int luma_filter(const uint32_t *e, uint32_t c2[12], uint32_t f[12]) {
  const uint4 *q = reinterpret_cast<const uint4 *>(e);
  const uint4 a = __ldg(q), b = __ldg(q + 1), d = __ldg(q + 2);
  const uint32_t w[10] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, d.x, d.y};
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    c2[k] = clip_of(w, k);
    f[k] = coef_of(w + 6, k);
  }
  return (int)w[9];
}
// The clip value as the plain form takes it.
__device__ __forceinline__ uint32_t plain_clip(uint32_t c2) { return c2 == 0x3FFF3FFFu ? 0x40004000u : c2; }

template <int DX>
__device__ __forceinline__ void luma_tap(const uint16_t *up, const uint16_t *dn, int c0, const uint32_t ncur[2],
                                         uint32_t c2, uint32_t nc2, uint32_t f, int acc[4]) {
  // tap at (DX, +dy) on row `up`, mirrored tap at (-DX, -dy) on row `dn`
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const uint32_t a = clipd(pair_at<DX>(up, c0 + 2 * q), ncur[q], c2, nc2);
    const uint32_t b = clipd(pair_at<-DX>(dn, c0 + 2 * q), ncur[q], c2, nc2);
    const uint32_t s = add2(a, b);
    acc[2 * q] = __dp2a_lo((int)s, (int)f, acc[2 * q]);
    acc[2 * q + 1] = __dp2a_hi((int)s, (int)f, acc[2 * q + 1]);
  }
}

constexpr uint64_t pack4(std::initializer_list<int> v) {
  uint64_t r = 0;
  int i = 0;
  for (int x : v) r |= (uint64_t)x << (4 * i++);
  return r;
}
constexpr uint32_t pack2(std::initializer_list<int> v) {
  uint32_t r = 0;
  int i = 0;
  for (int x : v) r |= (uint32_t)x << (2 * i++);
  return r;
}

// Class of one block from its four direction sums (eqs. 1463-1482, src/alf.rs:954-1007).
__device__ __forceinline__ void classify(int sh, int sv, int sd0, int sd1, int ac, int bd, uint8_t &f_out,
                                         uint8_t &t_out) {
  int hv1, hv0, dhv, d1, d0, dd;
  if (sv > sh) { hv1 = sv; hv0 = sh; dhv = 1; } else { hv1 = sh; hv0 = sv; dhv = 3; }
  if (sd0 > sd1) { d1 = sd0; d0 = sd1; dd = 0; } else { d1 = sd1; d0 = sd0; dd = 2; }
  const bool pd = (long long)d1 * hv0 > (long long)hv1 * d0;
  const int hvd1 = pd ? d1 : hv1, hvd0 = pd ? d0 : hv0;
  const int dir1 = pd ? dd : dhv, dir2 = pd ? dhv : dd;
  const int dir_s = hvd1 * 2 > 9 * hvd0 ? 2 : (hvd1 > 2 * hvd0 ? 1 : 0);
  const long long act = ((long long)(sh + sv) * ac) >> (bd - 1);
  const int avg = (int)(act > 15 ? 15 : act);
  // varTab (eq. 1480) packed 4 bits per entry, transposeTable 2 bits per entry
  constexpr uint64_t kVarTab = pack4({0, 1, 2, 2, 2, 2, 2, 3, 3, 3, 3, 3, 3, 3, 3, 4});
  constexpr uint32_t kTransposeTable = pack2({0, 1, 0, 2, 2, 3, 1, 3});
  int f = (int)((kVarTab >> (avg * 4)) & 0xF);
  if (dir_s != 0) f += (((dir1 & 1) << 1) + dir_s) * 5;
  f_out = (uint8_t)f;
  t_out = (uint8_t)((kTransposeTable >> ((dir1 * 2 + (dir2 >> 1)) * 2)) & 3);
}

// Laplacian sums per 2x2 cell of the luma window `sL`: cell (cx, cy) covers
// positions (X0 - 2 + 2cx + d, Y0 - 2 + 2cy + d), d = 0, 1.  The horizontal and
// vertical sums share a word, the diagonal ones another: a sum is at most
// 4 * (2^14 - 1) below 2^14 (a tile with larger samples classifies its blocks
// from the window itself).
template <class S, int NT>
__device__ __forceinline__ void luma_cells(const uint16_t *sL, uint2 *cell) {
  for (int i = threadIdx.x; i < S::CH * S::CW; i += NT) {
    const int cy = i / S::CW, cx = i - cy * S::CW;
    uint32_t h = 0, v = 0, d0 = 0, d1 = 0;
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const int r = 2 * cy + d + 1;  // sL row of the position: y = Y0 - 2 + 2cy + d
      const int c = 2 * cx + d + 2;  // sL col: x = X0 - 2 + 2cx + d
      const uint16_t *row = &sL[r * S::SLP + c];
      const int c2 = 2 * row[0];
      h += abs(c2 - row[-1] - row[1]);
      v += abs(c2 - row[-S::SLP] - row[S::SLP]);
      d0 += abs(c2 - row[-S::SLP - 1] - row[S::SLP + 1]);
      d1 += abs(c2 - row[-S::SLP + 1] - row[S::SLP - 1]);
    }
    cell[i] = make_uint2(h + (v << 16), d0 + (d1 << 16));
  }
}

// Class and transposeIdx of every 4x4 block of a W x TH tile (src/alf.rs:750-1008).
// big: a window sample of 2^14 or above (the cells do not hold its sums); wide: one
// of 2^12 or above (four cells do not add within their halves).
template <int W, int TH, class S, int NT>
__device__ __forceinline__ void luma_classes(const uint16_t *sL, const uint2 *cell, uint8_t *cls_f, uint8_t *cls_t,
                                             int Y0, int y_ctb, int ctb, int ph, int bd, bool big, bool wide) {
  const bool bottom = y_ctb + ctb >= ph;
  const bool carve = !bottom || (ph - y_ctb) > ctb - 4;
  const int vb = y_ctb + ctb - 4;
  constexpr int NB = (TH / 4) * (W / 4);
  using Sample = std::conditional_t<S::BIASED, int16_t, uint16_t>;  // biased samples are in order as signed numbers
  const Sample *win = reinterpret_cast<const Sample *>(sL);
  for (int b = threadIdx.x; b < NB; b += NT) {
    const int bx = b % (W / 4), by = b / (W / 4);
    const int y4 = Y0 + 4 * by - y_ctb;
    if (big || y4 == ctb - 8 || y4 == ctb - 4) {  // virtual-boundary rows: windows and padding differ
      int min_y = -2, max_y = 5, ac = 2;
      if (y4 == ctb - 8 && carve) { max_y = 3; ac = 3; }
      else if (y4 == ctb - 4 && carve) { min_y = 0; ac = 3; }
      const bool top_pad = y4 == ctb - 4, bot_pad = y4 == ctb - 8;
      auto pad = [&](int gy) {
        if (top_pad) gy = max(gy, vb);
        if (bot_pad) gy = min(gy, vb - 1);
        return gy - (Y0 - 3);
      };
      int sh = 0, sv = 0, sd0 = 0, sd1 = 0;
      for (int j = min_y; j <= max_y; ++j) {
        const int gy = y_ctb + y4 + j;
        const Sample *rc = &win[pad(gy) * S::SLP], *ru = &win[pad(gy - 1) * S::SLP], *rd = &win[pad(gy + 1) * S::SLP];
        for (int i = (j & 1) ? -1 : -2; i <= 5; i += 2) {
          const int c = 4 * bx + i + 4;
          const int c2 = 2 * rc[c];
          sh += abs(c2 - rc[c - 1] - rc[c + 1]);
          sv += abs(c2 - ru[c] - rd[c]);
          sd0 += abs(c2 - ru[c - 1] - rd[c + 1]);
          sd1 += abs(c2 - ru[c + 1] - rd[c - 1]);
        }
      }
      classify(sh, sv, sd0, sd1, ac, bd, cls_f[b], cls_t[b]);
    } else {
      uint32_t sh = 0, sv = 0, sd0 = 0, sd1 = 0;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint2 *q = &cell[(2 * by + r) * S::CW + 2 * bx];
        uint2 g[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) g[c] = q[c];
        if (!wide) {  // four cells of 4 * 4095 at most add within their halves
          const uint32_t x = g[0].x + g[1].x + g[2].x + g[3].x, y = g[0].y + g[1].y + g[2].y + g[3].y;
          sh += x & 0xFFFF;
          sv += x >> 16;
          sd0 += y & 0xFFFF;
          sd1 += y >> 16;
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            sh += g[c].x & 0xFFFF;
            sv += g[c].x >> 16;
            sd0 += g[c].y & 0xFFFF;
            sd1 += g[c].y >> 16;
          }
        }
      }
      classify((int)sh, (int)sv, (int)sd0, (int)sd1, 2, bd, cls_f[b], cls_t[b]);
    }
  }
}

// Table 45 rows of a luma row `yr` inside its CTB (line-buffer arms always applied,
// src/alf.rs:694, 1117-1130): the filter shift and the row offsets y1..y3.
__device__ __forceinline__ void table45(int yr, int ctb, int &shift, int &y1, int &y2, int &y3) {
  shift = 7;
  y1 = 1;
  y2 = 2;
  y3 = 3;
  if (yr == ctb - 5 || yr == ctb - 4) { shift = 10; y1 = y2 = y3 = 0; }
  else if (yr == ctb - 6 || yr == ctb - 3) { y2 = y3 = 1; }
  else if (yr == ctb - 7 || yr == ctb - 2) { y3 = 2; }
}

// The 7x7 diamond on one run of 4 samples (window row j, block column bx) with
// one block's packed taps; `yr` is the row inside its CTB.  out[] receives the
// filtered samples (src/alf.rs:652-743, Table 45 arms always applied).
template <class S>
__device__ __forceinline__ void luma_run(const S &sm, int j, int bx, int yr, int ctb, const uint32_t c2[12],
                                         const uint32_t nc2[12], const uint32_t f[12], int maxv, int out[4]) {
  int shift, y1, y2, y3;
  table45(yr, ctb, shift, y1, y2, y3);
  const int r = j + 3;
  const int c0 = 4 * bx + 4;
  const uint16_t *R0 = &sm.sL[r * S::SLP];
  const uint16_t *U1 = R0 - y1 * S::SLP, *D1 = R0 + y1 * S::SLP;
  const uint16_t *U2 = R0 - y2 * S::SLP, *D2 = R0 + y2 * S::SLP;
  const uint16_t *U3 = R0 - y3 * S::SLP, *D3 = R0 + y3 * S::SLP;
  const uint32_t cur[2] = {pair_at<0>(R0, c0), pair_at<0>(R0, c0 + 2)};
  const uint32_t ncur[2] = {neg2(cur[0]), neg2(cur[1])};
  int acc[4] = {0, 0, 0, 0};
  luma_tap<0>(D3, U3, c0, ncur, c2[0], nc2[0], f[0], acc);
  luma_tap<1>(D2, U2, c0, ncur, c2[1], nc2[1], f[1], acc);
  luma_tap<0>(D2, U2, c0, ncur, c2[2], nc2[2], f[2], acc);
  luma_tap<-1>(D2, U2, c0, ncur, c2[3], nc2[3], f[3], acc);
  luma_tap<2>(D1, U1, c0, ncur, c2[4], nc2[4], f[4], acc);
  luma_tap<1>(D1, U1, c0, ncur, c2[5], nc2[5], f[5], acc);
  luma_tap<0>(D1, U1, c0, ncur, c2[6], nc2[6], f[6], acc);
  luma_tap<-1>(D1, U1, c0, ncur, c2[7], nc2[7], f[7], acc);
  luma_tap<-2>(D1, U1, c0, ncur, c2[8], nc2[8], f[8], acc);
  luma_tap<3>(R0, R0, c0, ncur, c2[9], nc2[9], f[9], acc);
  luma_tap<2>(R0, R0, c0, ncur, c2[10], nc2[10], f[10], acc);
  luma_tap<1>(R0, R0, c0, ncur, c2[11], nc2[11], f[11], acc);
  const int round = 1 << (shift - 1);
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int cv = (int)((cur[p >> 1] >> ((p & 1) * 16)) & 0xFFFF);
    out[p] = clampd(cv + ((acc[p] + round) >> shift), 0, maxv);
  }
}

// The 12 symmetric tap sums (n+ - cur) + (n- - cur) of one 4-sample run,
// packed per pixel pair, without clipping: the form every filter set whose
// clip values never bind shares (clipIdx 0 gives 2^BitDepth, above any
// |n - cur| of in-range samples).  Same taps and Table 45 rows as luma_run.
template <class S>
__device__ __forceinline__ void luma_sums(const S &sm, int j, int bx, int yr, int ctb, uint32_t sum[2][12],
                                          uint32_t cur[2], int &shift) {
  int y1, y2, y3;
  table45(yr, ctb, shift, y1, y2, y3);
  const int c0 = 4 * bx + 4;
  const uint16_t *R0 = &sm.sL[(j + 3) * S::SLP];
  const uint16_t *U1 = R0 - y1 * S::SLP, *D1 = R0 + y1 * S::SLP;
  const uint16_t *U2 = R0 - y2 * S::SLP, *D2 = R0 + y2 * S::SLP;
  const uint16_t *U3 = R0 - y3 * S::SLP, *D3 = R0 + y3 * S::SLP;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int c = c0 + 2 * q;
    cur[q] = pair_at<0>(R0, c);
    const uint32_t nc = neg2(cur[q]);
    auto tap = [&](uint32_t up, uint32_t dn) {
      return add2(__viaddmax_s16x2(up, nc, 0x80008000u), __viaddmax_s16x2(dn, nc, 0x80008000u));
    };
    sum[q][0] = tap(pair_at<0>(D3, c), pair_at<0>(U3, c));
    sum[q][1] = tap(pair_at<1>(D2, c), pair_at<-1>(U2, c));
    sum[q][2] = tap(pair_at<0>(D2, c), pair_at<0>(U2, c));
    sum[q][3] = tap(pair_at<-1>(D2, c), pair_at<1>(U2, c));
    sum[q][4] = tap(pair_at<2>(D1, c), pair_at<-2>(U1, c));
    sum[q][5] = tap(pair_at<1>(D1, c), pair_at<-1>(U1, c));
    sum[q][6] = tap(pair_at<0>(D1, c), pair_at<0>(U1, c));
    sum[q][7] = tap(pair_at<-1>(D1, c), pair_at<1>(U1, c));
    sum[q][8] = tap(pair_at<-2>(D1, c), pair_at<2>(U1, c));
    sum[q][9] = tap(pair_at<3>(R0, c), pair_at<-3>(R0, c));
    sum[q][10] = tap(pair_at<2>(R0, c), pair_at<-2>(R0, c));
    sum[q][11] = tap(pair_at<1>(R0, c), pair_at<-1>(R0, c));
  }
}

// f(integral_constant<int, 0>) ... f(integral_constant<int, N - 1>): indices as constants
template <class F, int... I>
__device__ __forceinline__ void static_for_impl(F &&f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F &&f) {
  static_for_impl(f, std::make_integer_sequence<int, N>{});
}

__device__ __forceinline__ uint32_t ld32(const uint16_t *p) { return *reinterpret_cast<const uint32_t *>(p); }
__device__ __forceinline__ uint2 ld64(const uint16_t *p) { return *reinterpret_cast<const uint2 *>(p); }
__device__ __forceinline__ void st64(uint16_t *p, uint2 v) { *reinterpret_cast<uint2 *>(p) = v; }

// Rows of packed words around a run of samples: word k covers samples
// (c0 - 2B + 2k, c0 - 2B + 2k + 1) of the row at p = &row[c0].
template <int NW, int B>
struct Words {
  uint32_t w[NW];
  // pair (p[o], p[o + 1])
  template <int O>
  __device__ __forceinline__ uint32_t pair() const {
    static_assert(O + 2 * B >= 0 && O + 2 * B + 1 < 2 * NW, "pair inside the loaded words");
    if constexpr (((O + 2 * B) & 1) == 0) return w[(O + 2 * B) / 2];
    else return __byte_perm(w[(O + 2 * B - 1) / 2], w[(O + 2 * B + 1) / 2], 0x5432);
  }
};

// Loads words [k0, k1) of a Words<NW, B> at p (p - 2B + 2k0 4-byte aligned;
// 64-bit loads where the address is 8-byte aligned by construction: A8).
template <int NW, int B, bool A8>
__device__ __forceinline__ void load_words(Words<NW, B> &r, const uint16_t *p, int k0, int k1) {
  const uint16_t *q = p - 2 * B;
  // word k starts an 8-byte aligned pair of words
  auto lead = [](int k) { return A8 && (((2 * B) % 4 == 0) == (k % 2 == 0)); };
#pragma unroll
  for (int k = 0; k < NW; ++k) {
    if (k < k0 || k >= k1) continue;
    if (k > k0 && lead(k - 1)) continue;  // loaded with word k - 1
    if (lead(k) && k + 1 < k1) {
      const uint2 v = ld64(q + 2 * k);
      r.w[k] = v.x;
      r.w[k + 1 < NW ? k + 1 : k] = v.y;
    } else {
      r.w[k] = ld32(q + 2 * k);
    }
  }
}

// The plain form of the clipped taps for tiles that hold a sample of 2^14 or
// above, sample by sample and tap by tap in 32 bits, as differences take 17 (out
// of line: no picture of a supported depth has any).  w: the packed filter's
// clips, f: its coefficients.
__device__ __forceinline__ int tap_plain(const uint16_t *R, int o, int cur, const uint32_t *w, const uint32_t *f,
                                         int k) {
  int c = (int)(w[k / 2] >> (16 * (k & 1)) & 0xFFFF);
  if (c == 0x3FFF) c = 0x4000;  // as packed (build_packed)
  // the windows' biased samples are in order as signed numbers
  return (clampd((int)(int16_t)R[o] - cur, -c, c) + clampd((int)(int16_t)R[-o] - cur, -c, c)) * (int8_t)(f[k / 4] >> (8 * (k & 3)) & 0xFF);
}
// taps (dx, dy) of the 7x7 and 5x5 diamonds in table order, mirrored taps at (-dx, -dy)
static __constant__ int8_t kLumaTaps[12][2] = {{0, 3}, {1, 2}, {0, 2}, {-1, 2}, {2, 1}, {1, 1},
                                        {0, 1}, {-1, 1}, {-2, 1}, {3, 0}, {2, 0}, {1, 0}};
static __constant__ int8_t kChromaTaps[6][2] = {{0, 2}, {1, 1}, {0, 1}, {-1, 1}, {2, 0}, {1, 0}};

static __device__ __noinline__ void luma_run_plain(const uint16_t *R0, int pitch, int y1, int y2, int y3, int shift,
                                            const uint32_t *tab, int maxv, int out[4]) {
  const int ys[4] = {0, y1, y2, y3};
#pragma unroll 1
  for (int p = 0; p < 4; ++p) {
    const uint16_t *R = R0 + p;
    int acc = 1 << (shift - 1);
#pragma unroll 1
    for (int k = 0; k < 12; ++k)
      acc += tap_plain(R, ys[kLumaTaps[k][1]] * pitch + kLumaTaps[k][0], (int16_t)R[0], tab, tab + 6, k);
    out[p] = clampd((R[0] ^ 0x8000) + (acc >> shift), 0, maxv);
  }
}

template <int SPT>
__device__ __noinline__ void chroma_run_plain(const uint16_t *R0, int pitch, int y1, int y2, int shift,
                                              const uint32_t *ct, int maxv, int v[SPT]) {
  const int ys[3] = {0, y1, y2};
#pragma unroll 1
  for (int p = 0; p < SPT; ++p) {
    const uint16_t *R = R0 + p;
    int acc = 1 << (shift - 1);
#pragma unroll 1
    for (int k = 0; k < 6; ++k)
      acc += tap_plain(R, ys[kChromaTaps[k][1]] * pitch + kChromaTaps[k][0], (int16_t)R[0], ct, ct + 3, k);
    v[p] = clampd((R[0] ^ 0x8000) + (acc >> shift), 0, maxv);
  }
}

// The 5x5 chroma diamond on SPT samples of a row (R0: the first in the biased
// window; jr: the row inside its CTB of ctb_c rows), added to v[] (src/alf.rs:
// 1014-1065, Table 46 line-buffer arms always applied).
template <int SPT>
__device__ __forceinline__ void chroma_alf_run(const uint16_t *R0, int pitch, int jr, int ctb_c, const uint32_t *ct,
                                               int maxv, bool big, int v[SPT]) {
  constexpr int NP = SPT / 2;
  int s2 = 7, y1 = 1, y2 = 2;
  if (jr == ctb_c - 2 || jr == ctb_c - 3) { s2 = 10; y1 = y2 = 0; }
  else if (jr == ctb_c - 1 || jr == ctb_c - 4) { y2 = 1; }
  if (big) {
    chroma_run_plain<SPT>(R0, pitch, y1, y2, s2, ct, maxv, v);
    return;
  }
  uint32_t c2[6], f[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    c2[k] = clip_of(ct, k);
    f[k] = coef_of(ct + 3, k);
  }
  const int start = (int)ct[5] + (1 << (s2 - 1));
  int acc[SPT];
#pragma unroll
  for (int k = 0; k < SPT; ++k) acc[k] = start;
  uint32_t m[NP];  // 0x8000 - cur per lane
  Words<NP + 2, 1> r0, ra, rb;
  load_words<NP + 2, 1, (NP > 1)>(r0, R0, 0, NP + 2);
#pragma unroll
  for (int q = 0; q < NP; ++q) m[q] = kBias - (r0.w[1 + q] ^ kBias);
  auto tap = [&](const Words<NP + 2, 1> &up, const Words<NP + 2, 1> &dn, auto dx, int k) {
    constexpr int DX = decltype(dx)::value;
    const uint32_t c22 = c2[k] + c2[k];
    static_for<NP>([&](auto qc) {
      constexpr int q = decltype(qc)::value;
      const uint32_t b = c2[k] + m[q];
      const uint32_t s = clip_off(up.template pair<DX + 2 * q>(), b, c22) +
                         clip_off(dn.template pair<-DX + 2 * q>(), b, c22);
      acc[2 * q] = dp2a_ulo(s, f[k], acc[2 * q]);
      acc[2 * q + 1] = dp2a_uhi(s, f[k], acc[2 * q + 1]);
    });
  };
  using I0 = std::integral_constant<int, 0>;
  using I1 = std::integral_constant<int, 1>;
  using Im1 = std::integral_constant<int, -1>;
  using I2 = std::integral_constant<int, 2>;
  load_words<NP + 2, 1, (NP > 1)>(ra, R0 + y2 * pitch, 1, NP + 1);
  load_words<NP + 2, 1, (NP > 1)>(rb, R0 - y2 * pitch, 1, NP + 1);
  tap(ra, rb, I0{}, 0);
  load_words<NP + 2, 1, (NP > 1)>(ra, R0 + y1 * pitch, 0, NP + 2);
  load_words<NP + 2, 1, (NP > 1)>(rb, R0 - y1 * pitch, 0, NP + 2);
  tap(ra, rb, I1{}, 1);
  tap(ra, rb, I0{}, 2);
  tap(ra, rb, Im1{}, 3);
  tap(r0, r0, I2{}, 4);
  tap(r0, r0, I1{}, 5);
#pragma unroll
  for (int k = 0; k < SPT; ++k) v[k] = clampd(v[k] + (acc[k] >> s2), 0, maxv);
}

// CC-ALF of SPT chroma samples from the luma window (L0: luma of the first one;
// yline: its luma row inside the CTB; lbb: the line-buffer arms apply), added to
// v[] (Table 47, src/alf.rs:447-523).
template <int SPT>
__device__ __forceinline__ void cc_alf_run(const uint16_t *L0, int pitch, int yline, int ctb, bool lbb,
                                           const int32_t *cc_k, int bd, int maxv, int v[SPT]) {
  auto b8 = [](int x) { return (uint32_t)(x & 0xFF); };
  // taps 0..6 at (0,-yP1), (-1,0), (+1,0), (-1,yP1), (0,yP1), (+1,yP1), (0,yP2) as dp2a byte pairs
  const uint32_t k1 = b8(cc_k[0]) | b8(cc_k[1]) << 24;
  const uint32_t k2 = b8(cc_k[2]) << 8 | b8(cc_k[3]) << 24;
  const uint32_t k3 = b8(cc_k[4]) | b8(cc_k[5]) << 8 | b8(cc_k[6]) << 16;
  const int csum = cc_k[0] + cc_k[1] + cc_k[2] + cc_k[3] + cc_k[4] + cc_k[5] + cc_k[6];
  const int half = 1 << (bd - 1);
  int yp1 = 1, yp2 = 2;
  if (lbb) {
    if (yline == ctb - 5 || yline == ctb - 4) { yp1 = 0; yp2 = 0; }
    else if (yline == ctb - 6 || yline == ctb - 3) { yp2 = 1; }
  }
  // word k of a row: luma samples (2k - 2, 2k - 1) of the run; 8-byte loads for
  // word pairs (k, k + 1), k odd (L0 is 8-byte aligned when SPT > 2)
  constexpr int LW = SPT + 1;
  Words<LW, 1> wt, wm, wb, w2;
  load_words<LW, 1, (SPT > 2)>(wt, L0 - yp1 * pitch, 0, LW);
  load_words<LW, 1, (SPT > 2)>(wm, L0, 0, LW);
  load_words<LW, 1, (SPT > 2)>(wb, L0 + yp1 * pitch, 0, LW);
  load_words<LW, 1, (SPT > 2)>(w2, L0 + yp2 * pitch, 0, LW);
#pragma unroll
  for (int k = 0; k < SPT; ++k) {
    // chroma sample k: luma (2k - 2, 2k - 1) in word k, (2k, 2k + 1) in word k + 1
    int s = __dp2a_lo((int)wt.w[k + 1], (int)k1, 0);
    s = __dp2a_hi((int)wm.w[k], (int)k1, s);
    s = __dp2a_lo((int)wm.w[k + 1], (int)k2, s);
    s = __dp2a_hi((int)wb.w[k], (int)k2, s);
    s = __dp2a_lo((int)wb.w[k + 1], (int)k3, s);
    s = __dp2a_hi((int)w2.w[k + 1], (int)k3, s);
    const int ctr = (int16_t)(wm.w[k + 1] & 0xFFFF);  // biased like the taps: the biases cancel
    s -= ctr * csum;
    v[k] = clampd(v[k] + clampd((s + 64) >> 7, -half, half - 1), 0, maxv);
  }
}

// The same of 4 chroma samples of 4:4:4, whose luma samples are adjacent
// (L0 8-byte aligned): every tap pair is a natural word of a row, with the
// bytes of the coefficients placed for the even or the odd sample of a word.
__device__ __forceinline__ void cc_alf_run_444(const uint16_t *L0, int pitch, int yline, int ctb, bool lbb,
                                               const int32_t *cc_k, int bd, int maxv, int v[4]) {
  uint32_t b[7];
  int csum = 0;
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    b[k] = (uint32_t)(cc_k[k] & 0xFF);
    csum += cc_k[k];
  }
  const uint32_t m_even = b[1] << 8 | b[2] << 24, m_odd = b[1] | b[2] << 16;  // low: the earlier word
  const uint32_t d_even = b[3] << 8 | b[4] << 16 | b[5] << 24, d_odd = b[3] | b[4] << 8 | b[5] << 16;
  const uint32_t t_k = b[0] | b[0] << 24, u_k = b[6] | b[6] << 24;  // low: even sample, high: odd
  const int half = 1 << (bd - 1);
  int yp1 = 1, yp2 = 2;
  if (lbb) {
    if (yline == ctb - 5 || yline == ctb - 4) { yp1 = 0; yp2 = 0; }
    else if (yline == ctb - 6 || yline == ctb - 3) { yp2 = 1; }
  }
  Words<4, 1> m, d;  // word k: samples (2k - 2, 2k - 1)
  load_words<4, 1, true>(m, L0, 0, 4);
  load_words<4, 1, true>(d, L0 + yp1 * pitch, 0, 4);
  const uint2 tw = ld64(L0 - yp1 * pitch), uw = ld64(L0 + yp2 * pitch);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int t = (int)(k ? tw.y : tw.x), u = (int)(k ? uw.y : uw.x), c = (int)m.w[k + 1];
    int e = __dp2a_lo(t, (int)t_k, 0), o = __dp2a_hi(t, (int)t_k, 0);
    e = __dp2a_lo((int)m.w[k], (int)m_even, e);
    e = __dp2a_hi(c, (int)m_even, e);
    o = __dp2a_lo(c, (int)m_odd, o);
    o = __dp2a_hi((int)m.w[k + 2], (int)m_odd, o);
    e = __dp2a_lo((int)d.w[k], (int)d_even, e);
    e = __dp2a_hi((int)d.w[k + 1], (int)d_even, e);
    o = __dp2a_lo((int)d.w[k + 1], (int)d_odd, o);
    o = __dp2a_hi((int)d.w[k + 2], (int)d_odd, o);
    e = __dp2a_lo(u, (int)u_k, e) - (int)(int16_t)c * csum;  // biased like the taps: the biases cancel
    o = __dp2a_hi(u, (int)u_k, o) - (c >> 16) * csum;
    v[2 * k] = clampd(v[2 * k] + clampd((e + 64) >> 7, -half, half - 1), 0, maxv);
    v[2 * k + 1] = clampd(v[2 * k + 1] + clampd((o + 64) >> 7, -half, half - 1), 0, maxv);
  }
}

}  // namespace tile
}  // namespace h266
