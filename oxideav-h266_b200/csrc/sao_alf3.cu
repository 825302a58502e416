// SAO + ALF + CC-ALF tile pass of the chain (src/sao.rs:389-626, src/alf.rs:
// 220-1143), packed-arithmetic form: the default for BitDepth <= 14, ALF
// coefficients in [-128, 127]; other inputs use the scalar pass in sao_alf.cu.
// Chroma of 4:2:2 and 4:4:4 has tiles of its own.  Like the reference, the pass reads the deblocked
// planes and writes the final planes (its snapshot semantics), and post-SAO
// samples are clamped into the CTB's ALF fetch rectangle (the reference's
// clamped sample()).
//
// One CTA per W x TH luma tile (64 x 64 for CTBs of 64 and 128, 32 x 32 for
// CTBs of 32), never straddling a CTB, so the CTB's parameters, clip
// rectangle and virtual boundary are uniform per tile.  Phases, one barrier
// each:
//  1. the deblocked windows of the three planes, staged by the TMA unit (2-D
//     tensor loads of the tile widened by the halo; out-of-picture samples
//     read as 0 and are never used, as every read is clamped into the clip
//     rectangle) while the CTA resolves the SAO parameters of the 3x3 CTB
//     neighbourhood;
//  2. post-SAO windows of all planes, four samples per thread step: inside the
//     tile's own CTB and clip rectangle with one set of parameters, then the
//     quads of neighbouring CTBs with theirs (branch-free, all types), then
//     sample by sample only what is clamped or at the edge of the clip
//     rectangle; signs are one relu clamp per neighbour, offsets come from a
//     signed-byte table by one byte permute;
//  3. luma Laplacian sums per 2x2 cell beside the chroma planes' 5x5 ALF and
//     CC-ALF (a thread per 8 chroma samples of a row, CC-ALF taps as 6 dp2a);
//  4. luma classes, one 4x4 block per thread;
//  5. the 7x7 luma diamond, one block per thread with its 12 taps in
//     registers and each of the 7 rows held as packed words.
// The ALU pipe (64 lanes a clock: half the issue rate) and the waits between
// its instructions bound phases 2, 3 and 5 (issue 0.64 and ALU 0.51 busy over the
// whole launch), so the taps are in the offset form of alf_tile.cuh.  16 1080p 10-bit
// pictures: 364 us (472 with two clamps a tap, pairs instead of quads, border
// samples one by one and word-per-value filter tables; 389 with the plain form's
// branches in every phase).  Tiles with samples outside the packed lanes' range are
// told apart before phase 2 (finish_big).
#include <algorithm>
#include <atomic>
#include <type_traits>
#include <utility>

#include "alf_tile.cuh"
#include "tma.cuh"

namespace h266 {
namespace {

using namespace tile;

constexpr int NT3 = 256;
constexpr uint64_t kWaitNs = 20000000;  // 20 ms: a tile gives up on its window copies after this

// Tiles whose window copies did not complete within the poll limit (they are
// left unfiltered); read and cleared by pass2_wait_timeouts.
__device__ unsigned int g_wait_timeouts;

// Packed SAO parameters of one CTB and component.
struct alignas(16) SaoFast {
  int type;          // 0 copy, 1 band, 2 edge
  int row, shift_x;  // edge: the first neighbour's row offset in the window and column offset (-1, 0, 1)
  uint32_t tlo, thi;  // signed-byte offset table
  uint32_t shift, lane_mask, band_add;  // band: lane index ((c >> shift) - band) & 31
};

template <int W, int TH>
struct Smem3 {
  static constexpr bool BIASED = true;  // the post-SAO windows hold samples + 0x8000
  static constexpr int DLW = W + 16, DLH = TH + 8;          // deblocked luma [X0-8, X1+8) x [Y0-4, Y1+4)
  static constexpr int SLW = W + 8, SLH = TH + 6;           // post-SAO luma [X0-4, X1+4) x [Y0-3, Y1+3)
  static constexpr int CW = W / 2 + 2, CH = TH / 2 + 2;     // 2x2 Laplacian cells
  static constexpr int DCW = W / 2 + 16, DCH = TH / 2 + 6;  // deblocked chroma [x-8, x+8) x [y-3, y+3)
  static constexpr int SCW = W / 2 + 8, SCH = TH / 2 + 4;   // post-SAO chroma [x-4, x+4) x [y-2, y+2)
  // Row pitches of the post-SAO windows: 4 samples past the widths, so that
  // the chroma-phase threads (8 chroma rows of 4 runs per warp) reading luma
  // rows 2 apart, or chroma rows 1 apart, spread over more shared-memory
  // banks; multiples of 4 samples keep the 8-byte row alignment.
  static constexpr int SLP = SLW + 4, SCP = SCW + 4;
  static constexpr int DL_BYTES = DLH * DLW * 2, DC_BYTES = DCH * DCW * 2;
  static constexpr int DC_OFF = (DL_BYTES + 127) & ~127;
  static constexpr int DC_STRIDE = (DC_BYTES + 127) & ~127;
  static constexpr int D_BYTES = DC_OFF + 2 * DC_STRIDE;
  static constexpr int CELL_BYTES = CH * CW * 8;
  static constexpr int U_BYTES = D_BYTES > CELL_BYTES ? D_BYTES : CELL_BYTES;
  // the deblocked windows (TMA destinations); the Laplacian cells reuse the
  // space once the post-SAO windows exist
  alignas(128) uint8_t u[U_BYTES];
  alignas(16) uint16_t sL[SLH * SLP];
  alignas(16) uint16_t sC[2][SCH * SCP];
  uint8_t cls_f[(TH / 4) * (W / 4)], cls_t[(TH / 4) * (W / 4)];
  SaoLocal sao[3][9];
  SaoFast fast[3][9];
  alignas(8) unsigned long long bar;
  unsigned any_sao;  // bit comp * 9 + n: neighbour n of the 3x3 CTB neighbourhood has SAO for comp
  __device__ uint16_t *dL() { return reinterpret_cast<uint16_t *>(u); }
  __device__ uint16_t *dC(int c) { return reinterpret_cast<uint16_t *>(u + DC_OFF + c * DC_STRIDE); }
  __device__ uint2 *cell() { return reinterpret_cast<uint2 *>(u); }
};

// TMA and mbarrier helpers (tma.cuh); waits give up after kWaitNs.
using namespace tile_dev;

// ---------------------------------------------------------------- packed helpers
// Byte permute with sign replication (PTX prmt, default mode: selector bit 3
// copies the sign bit of the selected byte).
__device__ __forceinline__ uint32_t prmt(uint32_t lo, uint32_t hi, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(lo), "r"(hi), "r"(sel));
  return r;
}

// Offsets of two samples from the signed-byte table, idx their indices (0..7
// in each 16-bit lane): the indices in the selector's nibbles 0 and 2, the same
// with the sign-copy bit in nibbles 1 and 3 (the permute reads the low 16 bits).
__device__ __forceinline__ uint32_t lane_bytes(uint32_t tlo, uint32_t thi, uint32_t idx) {
  return prmt(tlo, thi, (idx + (idx >> 8)) * 0x11u + 0x8080u);
}

__device__ __forceinline__ SaoFast sao_fast(const SaoLocal &p, int pitch) {
  SaoFast f;
  f.type = p.type;
  f.row = p.type != 2 || p.nb >= -1 ? 0 : -pitch;
  f.shift_x = p.type != 2 ? 0 : p.nb - f.row;
  f.tlo = p.tlo;
  f.thi = p.thi;
  f.shift = (uint32_t)p.bd_shift;
  const uint32_t m = 0xFFFFu >> p.bd_shift;
  f.lane_mask = m | (m << 16);
  f.band_add = (uint32_t)((32 - p.band) & 31) * 0x00010001u;
  return f;
}

// The same of any CTB and type, without branches, for lanes with parameters of
// their own (the copy type's table is all zero and its row and column offsets
// 0): both indices are formed and the type picks one.
__device__ __forceinline__ uint2 sao_quad_any(const SaoFast &f, const uint16_t *d, uint32_t maxv2) {
  const uint2 c = ld64(d);
  const bool left = f.shift_x < 0, right = f.shift_x > 0;
  const uint32_t sel = f.shift_x ? 0x5432u : 0x3210u;
  // samples x + h .. x + h + 3: each pair from two neighbouring words
  const uint16_t *ra = d + f.row, *rb = d - f.row;
  const uint2 wa = ld64(ra), wb = ld64(rb);
  const uint32_t xa = ld32(left ? ra - 2 : ra + 4), xb = ld32(left ? rb + 4 : rb - 2);
  const uint32_t a0 = __byte_perm(left ? xa : wa.x, left ? wa.x : wa.y, sel);
  const uint32_t a1 = __byte_perm(left ? wa.x : wa.y, left ? wa.y : xa, sel);
  const uint32_t b0 = __byte_perm(right ? xb : wb.x, right ? wb.x : wb.y, sel);
  const uint32_t b1 = __byte_perm(right ? wb.x : wb.y, right ? wb.y : xb, sel);
  const uint32_t n0 = __viaddmax_s16x2(~c.x, 0x00020002u, 0x80008000u);  // 1 - c
  const uint32_t n1 = __viaddmax_s16x2(~c.y, 0x00020002u, 0x80008000u);
  const uint32_t e0 = __viaddmin_s16x2_relu(a0, n0, 0x00020002u) + __viaddmin_s16x2_relu(b0, n0, 0x00020002u);
  const uint32_t e1 = __viaddmin_s16x2_relu(a1, n1, 0x00020002u) + __viaddmin_s16x2_relu(b1, n1, 0x00020002u);
  const uint32_t k0 = __viaddmin_u16x2((((c.x >> f.shift) & f.lane_mask) + f.band_add) & 0x001F001Fu, 0u, 0x00040004u);
  const uint32_t k1 = __viaddmin_u16x2((((c.y >> f.shift) & f.lane_mask) + f.band_add) & 0x001F001Fu, 0u, 0x00040004u);
  const uint32_t v0 = __viaddmin_s16x2_relu(c.x, lane_bytes(f.tlo, f.thi, f.type == 2 ? e0 : k0), maxv2);
  const uint32_t v1 = __viaddmin_s16x2_relu(c.y, lane_bytes(f.tlo, f.thi, f.type == 2 ? e1 : k1), maxv2);
  return f.type ? make_uint2(v0, v1) : c;
}

// Samples (x + h .. x + h + 3) of the row at r = &row[x] (8-byte aligned), h in -1, 0, 1.
__device__ __forceinline__ uint2 quad_shifted(const uint16_t *r, int h) {
  const uint2 w = ld64(r);
  if (h == 0) return w;
  if (h < 0) return make_uint2(__byte_perm(ld32(r - 2), w.x, 0x5432), __byte_perm(w.x, w.y, 0x5432));
  return make_uint2(__byte_perm(w.x, w.y, 0x5432), __byte_perm(w.y, ld32(r + 4), 0x5432));
}

// SAO of the 4 samples at d (8-byte aligned window pointer; all inside one CTB,
// the clip rectangle and the CTB's edge-offset availability rectangle), samples
// below 2^14: the 16-bit lanes wrap between samples 32767 apart and where an
// offset meets a sample near it.
__device__ __forceinline__ uint2 sao_quad(const SaoFast &f, const uint16_t *d, uint32_t maxv2) {
  const uint2 c = ld64(d);
  if (f.type == 0) return c;
  uint32_t o0, o1;
  if (f.type == 2) {
    const uint2 a = quad_shifted(d + f.row, f.shift_x), b = quad_shifted(d - f.row, -f.shift_x);
    // lane-wise 1 - sign(c - n) = clip(n - c + 1, 0, 2); the two add to the table index
    const uint32_t n0 = __viaddmax_s16x2(~c.x, 0x00020002u, 0x80008000u);  // 1 - c
    const uint32_t n1 = __viaddmax_s16x2(~c.y, 0x00020002u, 0x80008000u);
    o0 = __viaddmin_s16x2_relu(a.x, n0, 0x00020002u) + __viaddmin_s16x2_relu(b.x, n0, 0x00020002u);
    o1 = __viaddmin_s16x2_relu(a.y, n1, 0x00020002u) + __viaddmin_s16x2_relu(b.y, n1, 0x00020002u);
  } else {
    const uint32_t k0 = (((c.x >> f.shift) & f.lane_mask) + f.band_add) & 0x001F001Fu;
    const uint32_t k1 = (((c.y >> f.shift) & f.lane_mask) + f.band_add) & 0x001F001Fu;
    o0 = __viaddmin_u16x2(k0, 0u, 0x00040004u);
    o1 = __viaddmin_u16x2(k1, 0u, 0x00040004u);
  }
  return make_uint2(__viaddmin_s16x2_relu(c.x, lane_bytes(f.tlo, f.thi, o0), maxv2),
                    __viaddmin_s16x2_relu(c.y, lane_bytes(f.tlo, f.thi, o1), maxv2));
}

// A rectangle of window quads: columns [x0, x0 + 4 * nq), rows [y0, y0 + ny) of
// component samples, x0 a multiple of 4.
struct FastRect {
  int x0, y0, nq, ny;
  uint32_t magic;  // floor(i / nq) = umulhi(i, magic) for the indices used (nq > 1)
  __device__ int row_of(uint32_t i) const { return nq == 1 ? (int)i : (int)__umulhi(i, magic); }
  __device__ int quads() const { return nq * ny; }
};

__device__ __forceinline__ FastRect fast_rect(int x0, int x1, int y0, int y1) {
  FastRect r;
  x0 = (x0 + 3) & ~3;
  x1 &= ~3;
  r.x0 = x0;
  r.y0 = y0;
  r.nq = x1 > x0 ? (x1 - x0) / 4 : 0;
  r.ny = y1 > y0 ? y1 - y0 : 0;
  if (!r.nq || !r.ny) r.nq = r.ny = 0;
  r.magic = r.nq > 1 ? 0xFFFFFFFFu / (uint32_t)r.nq + 1u : 0u;  // 2^32 / 1 does not fit: row_of
  return r;
}

// The i-th window quad outside the fast rectangle of a window WQ quads wide and
// WH rows high whose origin is (wx0, wy0): rows above, rows below, then the left
// and right parts of the fast rows.
__device__ __forceinline__ void rest_pos(int i, int wx0, int wy0, int WQ, int WH, const FastRect &f, int &x, int &y) {
  const int fy0 = f.ny ? f.y0 : wy0, fy1 = f.ny ? f.y0 + f.ny : wy0;
  const int n_top = WQ * (fy0 - wy0), n_bot = WQ * (wy0 + WH - fy1);
  if (i < n_top + n_bot) {
    const int r = i / WQ;
    x = wx0 + 4 * (i - r * WQ);
    y = i < n_top ? wy0 + r : fy1 + r - (fy0 - wy0);
    return;
  }
  i -= n_top + n_bot;
  const int lq = (f.x0 - wx0) / 4, rq = WQ - lq - f.nq, sq = lq + rq;  // seldom more than one each
  int r, c;
  if (sq == 1) { r = i; c = 0; }
  else if (sq == 2) { r = i >> 1; c = i & 1; }
  else { r = i / sq; c = i - r * sq; }
  y = fy0 + r;
  x = wx0 + 4 * (c < lq ? c : c + f.nq);
}

__device__ __forceinline__ int rest_count(int WQ, int WH, const FastRect &f) { return WQ * WH - f.quads(); }

// ---------------------------------------------------------------- the tile
// Whether the tile with chroma origin (xc0, yc0) has samples of half-height chroma plane c.
__device__ __forceinline__ bool chroma_tile_on(const Pass2Args &a, int c, int xc0, int yc0) {
  const DPlane &P = a.src[c + 1];
  return a.chroma && a.sub_h == 2 && P.w > 0 && P.h > 0 && xc0 < P.w && yc0 < P.h;
}

// Phases 3 to 5 of tile `tile` on its post-SAO windows.  BIG: they may hold samples
// of 2^14 and above; wide: of 2^12 and above.
template <int W, int TH, bool DO_ALF, bool BIG>
__device__ __forceinline__ void finish_tile(const Pass2Args &a, Smem3<W, TH> &sm, int tile, bool wide) {
  using S = Smem3<W, TH>;
  const int tid = threadIdx.x;
  const int X0 = tile % a.tiles_x * W, Y0 = tile / a.tiles_x * TH;
  const int bd = a.bit_depth, maxv = (1 << bd) - 1, log2 = a.ctb_log2, ctb = 1 << log2;
  const int rx = X0 >> log2, ry = Y0 >> log2, y_ctb = ry << log2, ph = a.pic_h;
  const CtbDev *me = rx < a.w_ctbs && ry < a.h_ctbs ? &a.ctbs[ry * a.w_ctbs + rx] : nullptr;
  constexpr int TWC = W / 2, THC = TH / 2;
  const int xc0 = X0 / 2, yc0 = Y0 / 2;


  // ---- (3) luma Laplacian sums per 2x2 cell (into the dead deblocked windows); chroma ALF / CC-ALF
  const bool luma_alf = DO_ALF && me && me->luma_set >= 0;
  if (luma_alf) luma_cells<S, NT3>(sm.sL, sm.cell());
  {
    // thread -> (plane, row, run of SPT samples)
    constexpr int SPT = TWC * THC / (NT3 / 2);  // 8 (64 x 64 tiles) or 2 (32 x 32)
    constexpr int NP = SPT / 2;                 // pairs per thread
    constexpr int RPR = TWC / SPT;              // threads per chroma row
    const int cc = tid / (NT3 / 2), t = tid % (NT3 / 2);
    const int jj = t / RPR, i0 = (t % RPR) * SPT;
    const DPlane &CD = a.dst[cc + 1];
    const int gy = yc0 + jj, gx = xc0 + i0;
    if (chroma_tile_on(a, cc, xc0, yc0) && gy < CD.h && gx < CD.w) {
      const int cf = (DO_ALF && me) ? me->chroma_filt[cc] : -1;
      const int ccf = (DO_ALF && me) ? me->cc_filt[cc] : -1;
      const int ctb_c = ctb / 2, y_ctb_c = y_ctb / 2;
      const uint16_t *R0 = &sm.sC[cc][(jj + 2) * S::SCP + i0 + 4];
      int v[SPT];
      {
        Words<NP + 2, 1> w0;
        load_words<NP + 2, 1, (NP > 1)>(w0, R0, 1, NP + 1);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          const uint32_t cur = w0.w[1 + q] ^ kBias;
          v[2 * q] = (int)(cur & 0xFFFF);
          v[2 * q + 1] = (int)(cur >> 16);
        }
      }
      if (cf >= 0)
        chroma_alf_run<SPT>(R0, S::SCP, gy - y_ctb_c, ctb_c, a.tables.chroma_packed[min(cf, 7)], maxv, BIG, v);
      if (ccf >= 0)  // col 2 i0 + 4 of the luma window = luma x of i0
        cc_alf_run<SPT>(&sm.sL[(2 * jj + 3) * S::SLP + 2 * i0 + 4], S::SLP, (gy - y_ctb_c) * 2, ctb,
                        !(gy * 2 + ctb >= ph && (ph - y_ctb) <= ctb - 4), a.tables.cc_coeff[cc][ccf], bd, maxv, v);
      uint16_t *out = CD.s + (int64_t)gy * CD.stride + gx;
      const bool vec = gx + SPT <= CD.w && ((uintptr_t)out & (2 * SPT - 1)) == 0;
      if (vec && SPT == 8) {
        uint4 o;
        o.x = (uint32_t)v[0] | (uint32_t)v[1] << 16;
        o.y = (uint32_t)v[2] | (uint32_t)v[3] << 16;
        o.z = (uint32_t)v[4] | (uint32_t)v[5] << 16;
        o.w = (uint32_t)v[6 % SPT] | (uint32_t)v[7 % SPT] << 16;
        *reinterpret_cast<uint4 *>(out) = o;
      } else if (vec && SPT == 4) {
        *reinterpret_cast<uint2 *>(out) = make_uint2((uint32_t)v[0] | (uint32_t)v[1 % SPT] << 16,
                                                     (uint32_t)v[2 % SPT] | (uint32_t)v[3 % SPT] << 16);
      } else if (vec && SPT == 2) {
        *reinterpret_cast<uint32_t *>(out) = (uint32_t)v[0] | (uint32_t)v[1 % SPT] << 16;
      } else {
#pragma unroll
        for (int k = 0; k < SPT; ++k)
          if (gx + k < CD.w) out[k] = (uint16_t)v[k];
      }
    }
  }
  const DPlane LD = a.dst[0];
  if (!luma_alf) {
    // the post-SAO tile as it is, 4 samples per store
    for (int p = tid; p < TH * W / 4; p += NT3) {
      const int j = p / (W / 4), i = (p % (W / 4)) * 4;
      const int gx = X0 + i, gy = Y0 + j;
      if (gy >= LD.h || gx >= LD.w) continue;
      uint2 v = ld64(&sm.sL[(j + 3) * S::SLP + i + 4]);
      v.x ^= kBias;
      v.y ^= kBias;
      uint16_t *out = LD.s + (int64_t)gy * LD.stride + gx;
      if (gx + 4 <= LD.w && ((uintptr_t)out & 7) == 0) {
        *reinterpret_cast<uint2 *>(out) = v;
      } else {
        const uint16_t s4[4] = {(uint16_t)(v.x & 0xFFFF), (uint16_t)(v.x >> 16), (uint16_t)(v.y & 0xFFFF),
                                (uint16_t)(v.y >> 16)};
        for (int k = 0; k < 4 && gx + k < LD.w; ++k) out[k] = s4[k];
      }
    }
    return;
  }
  __syncthreads();

  // ---- (4) classes
  luma_classes<W, TH, S, NT3>(sm.sL, sm.cell(), sm.cls_f, sm.cls_t, Y0, y_ctb, ctb, ph, bd, BIG, wide);
  __syncthreads();

  // ---- (5) 7x7 diamond: every thread keeps one block's taps and filters RPT of its 4-sample runs
  constexpr int RUNS = TH * W / 4;
  constexpr int RPT = RUNS / NT3;  // runs per thread: 4 (64 x 64) or 1 (32 x 32)
  constexpr int TPB = 4 / RPT;     // threads per 4x4 block
  const int b = tid / TPB;
  const int bx = b % (W / 4), by = b / (W / 4);
  const uint32_t *tab =
      a.tables.luma_packed + ((size_t)me->luma_set * 100 + sm.cls_f[b] * 4 + sm.cls_t[b]) * kLumaEntry;
  uint32_t c2[12], f[12];  // clip values and coefficients in registers
  const int start = luma_filter(tab, c2, f);
  const int gx = X0 + 4 * bx;
#pragma unroll 1
  for (int rr = 0; rr < RPT; ++rr) {
    const int j = 4 * by + (tid % TPB) * RPT + rr;  // tile row
    const int gy = Y0 + j;
    if (gy >= LD.h || gx >= LD.w) continue;
    int shift, y1, y2, y3;
    table45(gy - y_ctb, ctb, shift, y1, y2, y3);
    const uint16_t *R0 = &sm.sL[(j + 3) * S::SLP + 4 * bx + 4];
    int o[4];
    if (BIG) {
      luma_run_plain(R0, S::SLP, y1, y2, y3, shift, tab, maxv, o);
    } else {
      const int st = start + (1 << (shift - 1));
      int acc[4] = {st, st, st, st};
      // words k of a row: samples (c0 - 4 + 2k, +1), c0 = the run's first sample
      Words<6, 2> ru, rd;
      load_words<6, 2, true>(ru, R0, 0, 6);  // the run's own row
      const uint32_t cur[2] = {ru.w[2] ^ kBias, ru.w[3] ^ kBias};
      const uint32_t m[2] = {kBias - cur[0], kBias - cur[1]};  // 0x8000 - cur per lane
      auto tap = [&](const Words<6, 2> &up, const Words<6, 2> &dn, auto dx, int k) {
        constexpr int DX = decltype(dx)::value;
        const uint32_t c22 = c2[k] + c2[k];
        static_for<2>([&](auto qc) {
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
      using Im2 = std::integral_constant<int, -2>;
      using I3 = std::integral_constant<int, 3>;
      tap(ru, ru, I3{}, 9);
      tap(ru, ru, I2{}, 10);
      tap(ru, ru, I1{}, 11);
      load_words<6, 2, true>(ru, R0 + y3 * S::SLP, 2, 4);
      load_words<6, 2, true>(rd, R0 - y3 * S::SLP, 2, 4);
      tap(ru, rd, I0{}, 0);
      load_words<6, 2, true>(ru, R0 + y2 * S::SLP, 1, 5);
      load_words<6, 2, true>(rd, R0 - y2 * S::SLP, 1, 5);
      tap(ru, rd, I1{}, 1);
      tap(ru, rd, I0{}, 2);
      tap(ru, rd, Im1{}, 3);
      load_words<6, 2, true>(ru, R0 + y1 * S::SLP, 1, 5);
      load_words<6, 2, true>(rd, R0 - y1 * S::SLP, 1, 5);
      tap(ru, rd, I2{}, 4);
      tap(ru, rd, I1{}, 5);
      tap(ru, rd, I0{}, 6);
      tap(ru, rd, Im1{}, 7);
      tap(ru, rd, Im2{}, 8);
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const int cv = (int)((cur[p >> 1] >> ((p & 1) * 16)) & 0xFFFF);
        o[p] = clampd(cv + (acc[p] >> shift), 0, maxv);
      }
    }
    uint16_t *out = LD.s + (int64_t)gy * LD.stride + gx;
    if (gx + 4 <= LD.w && ((uintptr_t)out & 7) == 0) {
      *reinterpret_cast<uint2 *>(out) =
          make_uint2((uint32_t)o[0] | (uint32_t)o[1] << 16, (uint32_t)o[2] | (uint32_t)o[3] << 16);
    } else {
      for (int p = 0; p < 4 && gx + p < LD.w; ++p) out[p] = (uint16_t)o[p];
    }
  }
}

// Phases 2 to 5 of a tile that holds a sample of 2^14 or above, outside every depth
// of the packed lanes, which wrap between samples 32767 apart: its post-SAO windows
// sample by sample, ALF in the plain forms.  Out of line and decided before phase
// 2, so that the other tiles hold none of it (16 1080p pictures from resident
// plans 656 -> 637 us against branches in every phase; the windows formed a second
// time where phase 2 met such a sample: 669, or 684 by a call that returned).
template <int W, int TH, bool DO_ALF>
__device__ __noinline__ void finish_big(const Pass2Args &a, int tile) {
  using S = Smem3<W, TH>;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  S &sm = *reinterpret_cast<S *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
  const int X0 = tile % a.tiles_x * W, Y0 = tile / a.tiles_x * TH, log2 = a.ctb_log2;
  const int rx = X0 >> log2, ry = Y0 >> log2, maxv = (1 << a.bit_depth) - 1;
  int rect[4] = {0, 0, a.pic_w, a.pic_h};
  if (rx < a.w_ctbs && ry < a.h_ctbs)
    for (int k = 0; k < 4; ++k) rect[k] = a.ctbs[ry * a.w_ctbs + rx].rect[k];
#pragma unroll 1
  for (int comp = 0; comp < 3; ++comp) {
    const DPlane &P = a.src[comp];
    const int sh = comp ? 1 : 0, x0 = X0 >> sh, y0 = Y0 >> sh;
    if (comp && !chroma_tile_on(a, comp - 1, x0, y0)) continue;
    const int fx0 = max(rect[0] >> sh, 0), fx1 = min((rect[2] + sh) >> sh, comp ? P.w : a.pic_w);
    const int fy0 = max(rect[1] >> sh, 0), fy1 = min((rect[3] + sh) >> sh, comp ? P.h : a.pic_h);
    const int ww = comp ? S::SCW : S::SLW, wh = comp ? S::SCH : S::SLH, wp = comp ? S::SCP : S::SLP;
    const int ox = x0 - 4, oy = y0 - (comp ? 2 : 3), dx0 = x0 - 8, dy0 = oy - 1, pitch = comp ? S::DCW : S::DLW;
    const uint16_t *D = comp ? sm.dC(comp - 1) : sm.dL();
    uint16_t *out = comp ? sm.sC[comp - 1] : sm.sL;
#pragma unroll 1
    for (int i = threadIdx.x; i < ww * wh; i += NT3) {
      const int r = i / ww, c = i - r * ww;
      const int ax = clampd(ox + c, fx0, fx1 - 1), ay = clampd(oy + r, fy0, fy1 - 1);
      const uint16_t *d = D + (ay - dy0) * pitch + (ax - dx0);
      const SaoLocal &p = sm.sao[comp][((ay >> (log2 - sh)) - ry + 1) * 3 + ((ax >> (log2 - sh)) - rx + 1)];
      out[r * wp + c] = (uint16_t)((p.type ? sao_one(p, ax, ay, maxv, d) : *d) ^ 0x8000);
    }
  }
  __syncthreads();
  finish_tile<W, TH, DO_ALF, true>(a, sm, tile, true);
}

// Tile `tile` of the picture whose parameters are `a` (tensor maps at `maps`).
// PERSIST: the CTA runs many tiles on one barrier, initialised by the caller;
// `phase` is the barrier's next phase and flips with every completed copy.
// Returns false when the window copies did not land in time (the tile is left
// unfiltered and counted; a persistent CTA stops then).
template <int W, int TH, bool DO_SAO, bool DO_ALF, bool GLOBAL_MAPS, bool PERSIST = false>
__device__ __forceinline__ bool sao_alf_tile3(const Pass2Args &a, const Pass2Args *maps, int tile,
                                              uint32_t &phase) {
  using S = Smem3<W, TH>;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  // TMA destinations need 128-byte aligned shared addresses: align the base
  // explicitly (the launch adds 128 bytes)
  S &sm = *reinterpret_cast<S *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
  const int tid = threadIdx.x;
  const int tx = tile % a.tiles_x, ty = tile / a.tiles_x;
  const int X0 = tx * W, Y0 = ty * TH;
  const int bd = a.bit_depth, maxv = (1 << bd) - 1;
  const uint32_t maxv2 = (uint32_t)maxv * 0x00010001u;
  const int log2 = a.ctb_log2, ctb = 1 << log2;
  const int rx = X0 >> log2, ry = Y0 >> log2;
  const int x_ctb = rx << log2, y_ctb = ry << log2;
  const int pw = a.pic_w, ph = a.pic_h;
  const bool in_grid = rx < a.w_ctbs && ry < a.h_ctbs;
  const CtbDev *me = in_grid ? &a.ctbs[ry * a.w_ctbs + rx] : nullptr;
  int rect[4] = {0, 0, pw, ph};
  if (me) {
    rect[0] = me->rect[0];
    rect[1] = me->rect[1];
    rect[2] = me->rect[2];
    rect[3] = me->rect[3];
  }
  const int rx0 = max(rect[0], 0), ry0 = max(rect[1], 0), rx1 = min(rect[2], pw), ry1 = min(rect[3], ph);
  constexpr int TWC = W / 2, THC = TH / 2;
  const int xc0 = X0 / 2, yc0 = Y0 / 2;
  bool chroma_on[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) chroma_on[c] = chroma_tile_on(a, c, xc0, yc0);
  const bool tma = a.tma != 0;

  // ---- (1) deblocked windows (thread 0 starts the copies first, so they
  // overlap the rest of the phase); SAO parameters of the 3x3 CTB neighbourhood
  if (tma && tid == 0) {
    if (!PERSIST) mbar_init(&sm.bar, 1);
    const uint32_t bytes = (a.src[0].w > 0 && a.src[0].h > 0 ? S::DL_BYTES : 0) +
                           (chroma_on[0] ? S::DC_BYTES : 0) + (chroma_on[1] ? S::DC_BYTES : 0);
    if (GLOBAL_MAPS)
      for (int c = 0; c < 3; ++c) tmap_acquire(&maps->tmap[c]);
    // the previous tile's generic accesses of the window space (ordered by the
    // persistent loop's barrier) come before these copies
    if (PERSIST) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(&sm.bar, bytes);
    if (a.src[0].w > 0 && a.src[0].h > 0) tma_load_2d(sm.dL(), &maps->tmap[0], X0 - 8, Y0 - 4, &sm.bar);
#pragma unroll
    for (int c = 0; c < 2; ++c)
      if (chroma_on[c]) tma_load_2d(sm.dC(c), &maps->tmap[1 + c], xc0 - 8, yc0 - 3, &sm.bar);
  }
  int my_type = 0;
  if (tid < 27) {
    const int comp = tid / 9, n = tid % 9;
    const int nx = rx + n % 3 - 1, ny = ry + n / 3 - 1;
    SaoLocal &s = sm.sao[comp][n];
    s.type = 0;
    s.nb = 0;
    s.tlo = s.thi = 0;
    s.bd_shift = bd - 5;
    s.band = 0;
    const bool used = comp == 0 ? a.sao_luma : a.sao_chroma;
    if (DO_SAO && used && nx >= 0 && ny >= 0 && nx < a.w_ctbs && ny < a.h_ctbs) {
      const CtbDev &c = a.ctbs[ny * a.w_ctbs + nx];
      const int sw = comp ? 2 : 1;
      const int cw = comp ? a.src[comp].w : a.src[0].w, ch = comp ? a.src[comp].h : a.src[0].h;
      int q0 = 0, q1 = 0, q2 = cw, q3 = ch;  // clip rectangle in component samples, within the picture
      if (a.has_clip) {
        q0 = max(q0, c.rect[0] / sw);
        q1 = max(q1, c.rect[1] / sw);
        q2 = min(q2, (c.rect[2] + sw - 1) / sw);
        q3 = min(q3, (c.rect[3] + sw - 1) / sw);
      }
      sao_local(s, c.sao[comp], comp ? S::DCW : S::DLW, q0, q1, q2, q3, bd);
      my_type = s.type;
    }
    sm.fast[comp][n] = sao_fast(s, comp ? S::DCW : S::DLW);
  }
  if (tid < 32) {
    const unsigned m = __ballot_sync(0xFFFFFFFFu, my_type != 0);
    if (tid == 0) sm.any_sao = m;
  }
  if (!tma) {
    // windows by 16-byte vector loads (planes whose layout the TMA unit cannot describe)
    auto load = [&](uint16_t *dst, const DPlane &P, int x0, int y0, int WW, int HH) {
      const bool vec = x0 >= 0 && x0 + WW <= P.w && (x0 & 7) == 0 && ((uintptr_t)P.s & 15) == 0 && (P.stride & 7) == 0;
      if (vec) {
        const int NV = WW / 8;
        for (int i = tid; i < HH * NV; i += NT3) {
          const int r = i / NV, c = (i - r * NV) * 8;
          const int gy = clampd(y0 + r, 0, P.h - 1);
          *reinterpret_cast<uint4 *>(dst + r * WW + c) =
              *reinterpret_cast<const uint4 *>(P.s + (int64_t)gy * P.stride + x0 + c);
        }
      } else {
        for (int i = tid; i < HH * WW; i += NT3) {
          const int r = i / WW, c = i - r * WW;
          const int gx = clampd(x0 + c, 0, P.w - 1), gy = clampd(y0 + r, 0, P.h - 1);
          dst[i] = P.s[(int64_t)gy * P.stride + gx];
        }
      }
    };
    if (a.src[0].w > 0 && a.src[0].h > 0) load(sm.dL(), a.src[0], X0 - 8, Y0 - 4, S::DLW, S::DLH);
#pragma unroll
    for (int c = 0; c < 2; ++c)
      if (chroma_on[c]) load(sm.dC(c), a.src[c + 1], xc0 - 8, yc0 - 3, S::DCW, S::DCH);
  }
  __syncthreads();  // SAO parameters, the barrier's initialisation (or the vector-loaded windows)

  // geometry of the packed SAO rectangles while the copies are in flight
  const unsigned any = sm.any_sao;
  const bool sao_on[3] = {DO_SAO && (any & 0x1FFu) != 0, DO_SAO && ((any >> 9) & 0x1FFu) != 0,
                          DO_SAO && ((any >> 18) & 0x1FFu) != 0};
  // packed SAO: offsets as signed bytes, samples below 2^12 (a plain copy has no such limit)
  const bool quads = a.sao_i8 && bd <= 12;
  const bool fast_ok[3] = {!sao_on[0] || quads, !sao_on[1] || quads, !sao_on[2] || quads};
  const int crx0 = rect[0] / 2, cry0 = rect[1] / 2, crx1 = (rect[2] + 1) / 2, cry1 = (rect[3] + 1) / 2;
  FastRect fr[3];
  {
    // luma: inside the own CTB and one sample inside the clip rectangle when any
    // SAO is on (edge offset then sees both neighbours); else the clip rectangle
    const bool s = sao_on[0];
    fr[0] = fast_ok[0] ? fast_rect(max(X0 - 4, s ? max(x_ctb, rx0 + 1) : rx0),
                                min(X0 + W + 4, s ? min(x_ctb + ctb, rx1 - 1) : rx1),
                                max(Y0 - 3, s ? max(y_ctb, ry0 + 1) : ry0),
                                min(Y0 + TH + 3, s ? min(y_ctb + ctb, ry1 - 1) : ry1))
                    : fast_rect(0, 0, 0, 0);
#pragma unroll
    for (int cc = 0; cc < 2; ++cc) {
      const DPlane &CS = a.src[cc + 1];
      const int cx0 = max(crx0, 0), cy0 = max(cry0, 0), cx1 = min(crx1, CS.w), cy1 = min(cry1, CS.h);
      const bool t = sao_on[cc + 1];
      const int cxs = x_ctb / 2, cys = y_ctb / 2, cc_ctb = ctb / 2;
      fr[cc + 1] = (fast_ok[cc + 1] && chroma_on[cc])
                       ? fast_rect(max(xc0 - 4, t ? max(cxs, cx0 + 1) : cx0),
                                   min(xc0 + TWC + 4, t ? min(cxs + cc_ctb, cx1 - 1) : cx1),
                                   max(yc0 - 2, t ? max(cys, cy0 + 1) : cy0),
                                   min(yc0 + THC + 2, t ? min(cys + cc_ctb, cy1 - 1) : cy1))
                       : fast_rect(0, 0, 0, 0);
    }
  }
  bool ok = !tma || mbar_wait_bounded(&sm.bar, phase, kWaitNs);
  // The deblocked samples or'ed together: 2^14 and above is outside every depth of
  // the packed lanes, 2^12 and above (13 and 14 bits, or outside the depth) of the
  // class sums.  The look costs 0.3 % (16 1080p pictures 658.6 -> 660.7 us).
  uint32_t seen = 0;
  if (DO_SAO || DO_ALF) {
    auto look = [&](const uint16_t *w, int n) {
      const uint4 *q = reinterpret_cast<const uint4 *>(w);
      for (int i = tid; i < n / 8; i += NT3) seen |= q[i].x | q[i].y | q[i].z | q[i].w;
    };
    if (a.src[0].w > 0 && a.src[0].h > 0) look(sm.dL(), S::DLH * S::DLW);
    for (int c = 0; c < 2; ++c)
      if (chroma_on[c]) look(sm.dC(c), S::DCH * S::DCW);
  }
  bool wide = false;
  if (__syncthreads_or(!ok || (seen & 0xF000F000u))) {
    ok = __syncthreads_and(ok);
    if (!ok) {  // the copies did not land: count the tile, let them finish (bounded), leave it unfiltered
      if (tid == 0) atomicAdd(&g_wait_timeouts, 1u);
      mbar_wait_bounded(&sm.bar, phase, kWaitNs);
      return false;
    }
    wide = true;
    if (__syncthreads_or((seen & 0xC000C000u) != 0)) {
      finish_big<W, TH, DO_ALF>(a, tile);
      if (tma) phase ^= 1u;
      return true;
    }
  }
  if (tma) phase ^= 1u;

  // ---- (2) post-SAO windows (biased), clamped into the fetch rectangle, 4 samples per step
  {
    constexpr int WQL = S::SLW / 4, WQC = S::SCW / 4;
    const uint16_t *dL = sm.dL();
    auto put = [&](uint16_t *w, uint2 v) { st64(w, make_uint2(v.x ^ kBias, v.y ^ kBias)); };
    {  // the tile's own CTB inside the clip rectangle: one set of parameters
      const SaoFast f = sm.fast[0][4];
      const FastRect q = fr[0];
      for (int i = tid; i < q.quads(); i += NT3) {
        const int r = q.row_of((uint32_t)i), x = q.x0 + 4 * (i - r * q.nq), y = q.y0 + r;
        put(&sm.sL[(y - (Y0 - 3)) * S::SLP + (x - (X0 - 4))],
            sao_quad(f, dL + (y - (Y0 - 4)) * S::DLW + (x - (X0 - 8)), maxv2));
      }
    }
    {
      const int nc0 = chroma_on[0] ? fr[1].quads() : 0, nc1 = chroma_on[1] ? fr[2].quads() : 0;
      for (int i = tid; i < nc0 + nc1; i += NT3) {
        const int cc = i < nc0 ? 0 : 1, j = i - (cc ? nc0 : 0);
        const FastRect &q = fr[1 + cc];
        const SaoFast f = sm.fast[1 + cc][4];
        const int r = q.row_of((uint32_t)j), x = q.x0 + 4 * (j - r * q.nq), y = q.y0 + r;
        put(&sm.sC[cc][(y - (yc0 - 2)) * S::SCP + (x - (xc0 - 4))],
            sao_quad(f, sm.dC(cc) + (y - (yc0 - 3)) * S::DCW + (x - (xc0 - 8)), maxv2));
      }
    }
    // the rest: quads of neighbouring CTBs with their parameters, and sample by
    // sample what is clamped or at the edges of the clip rectangle
    const int ns0 = rest_count(WQL, S::SLH, fr[0]);
    const int ns1 = chroma_on[0] ? rest_count(WQC, S::SCH, fr[1]) : 0;
    const int ns2 = chroma_on[1] ? rest_count(WQC, S::SCH, fr[2]) : 0;
    for (int i = tid; i < ns0 + ns1 + ns2; i += NT3) {
      const int comp = i < ns0 ? 0 : (i < ns0 + ns1 ? 1 : 2), cc = comp ? comp - 1 : 0;
      const int j = i - (comp ? ns0 + (comp == 2 ? ns1 : 0) : 0);
      const int ox = comp ? xc0 - 4 : X0 - 4, oy = comp ? yc0 - 2 : Y0 - 3;  // the window's origin
      int x, y;
      if (comp) rest_pos(j, ox, oy, WQC, S::SCH, fr[comp], x, y);
      else rest_pos(j, ox, oy, WQL, S::SLH, fr[0], x, y);
      // the component's fetch rectangle
      const int fx0 = comp ? max(crx0, 0) : rx0, fy0 = comp ? max(cry0, 0) : ry0;
      const int fx1 = comp ? min(crx1, a.src[comp].w) : rx1, fy1 = comp ? min(cry1, a.src[comp].h) : ry1;
      const int clog = comp ? log2 - 1 : log2;
      const int pitch = comp ? S::DCW : S::DLW;
      const uint16_t *D = comp ? sm.dC(cc) : dL;
      const int dx0 = comp ? xc0 - 8 : X0 - 8, dy0 = comp ? yc0 - 3 : Y0 - 4;
      const bool on = sao_on[comp];
      uint2 v;
      int n = 4;  // of the 3x3 neighbourhood, the CTB that holds the quad
      bool fast = x >= fx0 && x + 4 <= fx1 && y >= fy0 && y < fy1;
      if (fast && on) {
        n = ((y >> clog) - ry + 1) * 3 + ((x >> clog) - rx + 1);
        const SaoLocal &p = sm.sao[comp][n];
        fast = fast_ok[comp] && (p.type != 2 || (x >= p.ex0 && x + 4 <= p.ex1 && y >= p.ey0 && y < p.ey1));
      }
      if (fast) {
        v = sao_quad_any(sm.fast[comp][n], D + (y - dy0) * pitch + (x - dx0), maxv2);
      } else {
        const int ay = clampd(y, fy0, fy1 - 1);
        uint32_t s4[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int ax = clampd(x + k, fx0, fx1 - 1);
          const uint16_t *d = D + (ay - dy0) * pitch + (ax - dx0);
          s4[k] = *d;
          if (on) {
            const SaoLocal &p = sm.sao[comp][((ay >> clog) - ry + 1) * 3 + ((ax >> clog) - rx + 1)];
            if (p.type) s4[k] = (uint16_t)sao_one(p, ax, ay, maxv, d);
          }
        }
        v = make_uint2(s4[0] | s4[1] << 16, s4[2] | s4[3] << 16);
      }
      uint16_t *w = comp ? &sm.sC[cc][(y - oy) * S::SCP + (x - ox)] : &sm.sL[(y - oy) * S::SLP + (x - ox)];
      put(w, v);
    }
  }
  __syncthreads();
  finish_tile<W, TH, DO_ALF, false>(a, sm, tile, wide);
  return true;
}

template <int W, int TH, bool DO_SAO, bool DO_ALF>
__global__ void __launch_bounds__(NT3, 4) k_sao_alf_tiles(const __grid_constant__ Pass2Args a) {
  uint32_t phase = 0;
  sao_alf_tile3<W, TH, DO_SAO, DO_ALF, false>(a, &a, blockIdx.x, phase);
}

// Many pictures in one grid: CTAs [first[i], first[i + 1]) are the tiles of
// picture i, whose parameters (and tensor maps) are args[i].
template <int W, int TH, bool DO_SAO, bool DO_ALF>
__global__ void __launch_bounds__(NT3, 4) k_sao_alf_tiles_batch(const Pass2Args *__restrict__ args,
                                                                const uint32_t *__restrict__ first, int n) {
  __shared__ Pass2Args s_args;  // the picture's parameters, read once per CTA
  const int lo = tile_dev::batch_picture(first, n, blockIdx.x);
  static_assert(sizeof(Pass2Args) % 16 == 0, "vector copy");
  const uint4 *src = reinterpret_cast<const uint4 *>(args + lo);
  uint4 *dst = reinterpret_cast<uint4 *>(&s_args);
  for (int i = threadIdx.x; i < (int)(sizeof(Pass2Args) / 16); i += blockDim.x) dst[i] = src[i];
  __syncthreads();
  uint32_t phase = 0;
  sao_alf_tile3<W, TH, DO_SAO, DO_ALF, true>(s_args, args + lo, (int)(blockIdx.x - first[lo]), phase);
}

// Persistent form of the batched launch: a fixed grid (a chosen number of
// CTAs per SM) drains a device queue of (picture, tile) items -- `queue`
// counts the items handed out (zero at launch) and items [first[i],
// first[i + 1]) are picture i's tiles.  Every CTA keeps one barrier over its
// tiles and reloads the picture's parameters only when the picture changes.
// The queue only ever grows and no CTA waits for another, so the launch ends
// once every item has been taken.
template <int W, int TH, bool DO_SAO, bool DO_ALF>
__global__ void __launch_bounds__(NT3, 4) k_sao_alf_tiles_queue(const Pass2Args *__restrict__ args,
                                                                const uint32_t *__restrict__ first, int n,
                                                                uint32_t total, uint32_t *__restrict__ queue) {
  using S = Smem3<W, TH>;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  S &sm = *reinterpret_cast<S *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
  __shared__ Pass2Args s_args;
  __shared__ uint32_t s_item;
  if (threadIdx.x == 0) mbar_init(&sm.bar, 1);
  uint32_t phase = 0;
  int cur = -1;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(queue, 1u);
    __syncthreads();  // s_item; the previous tile's last reads of s_args and the windows
    const uint32_t t = s_item;
    if (t >= total) break;
    const int lo = tile_dev::batch_picture(first, n, t);
    if (lo != cur) {
      const uint4 *src = reinterpret_cast<const uint4 *>(args + lo);
      uint4 *dst = reinterpret_cast<uint4 *>(&s_args);
      for (int i = threadIdx.x; i < (int)(sizeof(Pass2Args) / 16); i += blockDim.x) dst[i] = src[i];
      cur = lo;
    }
    __syncthreads();
    if (!sao_alf_tile3<W, TH, DO_SAO, DO_ALF, true, true>(s_args, args + lo, (int)(t - first[lo]), phase)) break;
    __syncthreads();  // every thread is done with this tile before thread 0 takes the next item
  }
}

// Tiles of TW chroma samples across the wider of the two chroma planes.
__host__ __device__ inline int chroma_tiles_x(const Pass2Args &a, int tw) {
  const int w = a.src[1].w > a.src[2].w ? a.src[1].w : a.src[2].w;
  return (w + tw - 1) / tw;
}

// ---------------------------------------------------------------- chroma of 4:2:2 and 4:4:4
//
// SAO, 5x5 ALF and CC-ALF of both chroma planes of formats with full-height
// chroma, beside the luma tiles of the packed kernel: one CTA per TW x 32 chroma
// samples of both planes (32 x 32; 16 x 32 for the 16-sample-wide CTBs of 4:2:2 at
// CTB 32, so that a tile never straddles a CTB).  The windows of both planes, and
// of luma where the CTB has a CC filter, are loaded side by side while the SAO
// parameters resolve, then go through the branch-free SAO quads together (each
// window's leftover quads on other warps): three barriers in all.  The diamond
// and CC-ALF run four samples a thread, CC-ALF by dp2a on natural words.  Four
// 1080p 4:4:4 10-bit pictures: 182 -> 149 us against one window after the other,
// eight barriers, scalar CC taps and four CTAs an SM instead of five (160 us).
// The ALU pipe and the waits between its instructions bound it.  The tile's own
// quads in a loop of their own, with one set of parameters, cost more in
// instruction-cache misses than they saved (165 us).
template <int TW, int SW>
struct SmemC {
  static constexpr int NT = TW * 8, TH = 32, LW = TW * SW;
  static constexpr int DW = TW + 16, DH = TH + 6, SCW = TW + 8, SCH = TH + 4, SCP = SCW + 4;  // [x - 8, y - 3), [x - 4, y - 2)
  static constexpr int DLW = LW + 16, DLH = TH + 5, SLW = LW + 8, SLH = TH + 3, SLP = SLW + 4;  // [x - 8, y - 2), [x - 4, y - 1)
  alignas(16) uint16_t dC[2][DW * DH];
  alignas(16) uint16_t dL[DLW * DLH];
  alignas(16) uint16_t sC[2][SCH * SCP];
  alignas(16) uint16_t sL[SLH * SLP];
  SaoLocal sao[3][9];
  SaoFast fast[3][9];
};

template <int TW, int SW>
__device__ __forceinline__ void chroma_tile(const Pass2Args &a, int tile) {
  using S = SmemC<TW, SW>;
  constexpr int NT = S::NT, TH = S::TH;
  __shared__ S sm;
  const int tid = threadIdx.x;
  const int tiles_x = chroma_tiles_x(a, TW);
  const int xc0 = (tile % tiles_x) * TW, yc0 = (tile / tiles_x) * TH;
  const int X0 = xc0 * SW, Y0 = yc0;
  const int bd = a.bit_depth, maxv = (1 << bd) - 1, log2 = a.ctb_log2, ctb = 1 << log2;
  const uint32_t maxv2 = (uint32_t)maxv * 0x00010001u;
  const int rx = X0 >> log2, ry = Y0 >> log2, y_ctb = ry << log2;
  const CtbDev *me = rx < a.w_ctbs && ry < a.h_ctbs ? &a.ctbs[ry * a.w_ctbs + rx] : nullptr;
  const int pw = a.pic_w, ph = a.pic_h;
  int rect[4] = {0, 0, pw, ph};
  if (me)
    for (int k = 0; k < 4; ++k) rect[k] = me->rect[k];
  const bool have_luma = a.src[0].w > 0 && a.src[0].h > 0 && X0 < a.src[0].w && Y0 < a.src[0].h;
  if (tid < 27) {  // SAO parameters of the 3x3 CTB neighbourhood
    const int comp = tid / 9, n = tid % 9, nx = rx + n % 3 - 1, ny = ry + n / 3 - 1;
    SaoLocal &s = sm.sao[comp][n];
    s.type = s.nb = s.band = 0;
    s.tlo = s.thi = 0;
    s.bd_shift = bd - 5;
    const int pitch = comp ? S::DW : S::DLW;
    if (a.do_sao && (comp ? a.sao_chroma : a.sao_luma) && nx >= 0 && ny >= 0 && nx < a.w_ctbs && ny < a.h_ctbs) {
      const CtbDev &c = a.ctbs[ny * a.w_ctbs + nx];
      const int sw = comp ? SW : 1;
      int q0 = 0, q1 = 0, q2 = a.src[comp].w, q3 = a.src[comp].h;
      if (a.has_clip) {
        q0 = max(q0, c.rect[0] / sw);
        q1 = max(q1, (int)c.rect[1]);
        q2 = min(q2, (c.rect[2] + sw - 1) / sw);
        q3 = min(q3, (int)c.rect[3]);
      }
      sao_local(s, c.sao[comp], pitch, q0, q1, q2, q3, bd);
    }
    sm.fast[comp][n] = sao_fast(s, pitch);
  }
  uint32_t far = 0;  // the deblocked samples or'ed together
  const bool cc_any = a.do_alf && me && have_luma && (me->cc_filt[0] >= 0 || me->cc_filt[1] >= 0);
  bool on[2];
  for (int cc = 0; cc < 2; ++cc) on[cc] = xc0 < a.src[1 + cc].w && yc0 < a.src[1 + cc].h;  // uniform per CTA
  // The deblocked window of `src`, dw x dh at (dx0, dy0), clamped into the plane.
  auto load = [&](const DPlane &src, uint16_t *d, int dx0, int dy0, auto dwc, auto dhc) {
    constexpr int dw = decltype(dwc)::value, dh = decltype(dhc)::value, nv = dw / 8;
    if (dx0 >= 0 && dx0 + dw <= src.w && ((uintptr_t)src.s & 15) == 0 && (src.stride & 7) == 0) {
      for (int i = tid; i < dh * nv; i += NT) {
        const int r = i / nv, c = (i - r * nv) * 8, gy = clampd(dy0 + r, 0, src.h - 1);
        const uint4 v = *reinterpret_cast<const uint4 *>(src.s + (int64_t)gy * src.stride + dx0 + c);
        *reinterpret_cast<uint4 *>(&d[r * dw + c]) = v;
        far |= v.x | v.y | v.z | v.w;
      }
    } else {
      for (int i = tid; i < dh * dw; i += NT) {
        const int r = i / dw, c = i - r * dw;
        const uint16_t v =
            src.s[(int64_t)clampd(dy0 + r, 0, src.h - 1) * src.stride + clampd(dx0 + c, 0, src.w - 1)];
        d[r * dw + c] = v;
        far |= v;
      }
    }
  };
  using CDW = std::integral_constant<int, S::DW>;
  using CDH = std::integral_constant<int, S::DH>;
  for (int cc = 0; cc < 2; ++cc)
    if (on[cc]) load(a.src[1 + cc], sm.dC[cc], xc0 - 8, yc0 - 3, CDW{}, CDH{});
  if (cc_any)
    load(a.src[0], sm.dL, X0 - 8, Y0 - 2, std::integral_constant<int, S::DLW>{}, std::integral_constant<int, S::DLH>{});
  // the quads of SAO for samples below 2^14, as in the tile kernel (else sample by sample)
  const bool quads = !__syncthreads_or((far & 0xC000C000u) != 0) && a.sao_i8 && bd <= 12;
  // Post-SAO window of component `comp`: W x H at (wx0, wy0), clamped into
  // [fx0, fx1) x [fy0, fy1); lx: log2 of the CTB's width in the component's
  // samples; `rot`: the thread that takes the first quad.
  uint32_t seen = 0;
  auto window = [&](int comp, const uint16_t *din, uint16_t *out, int wx0, int wy0, int fx0, int fy0, int fx1, int fy1,
                    int lx, int rot, auto wc, auto hc) {
    constexpr int W = decltype(wc)::value, H = decltype(hc)::value, P = W + 4, DP = W + 8, WQ = W / 4;
    const int dx0 = wx0 - 4, dy0 = wy0 - 1;
    for (int i = (tid + NT - rot) % NT; i < WQ * H; i += NT) {
      const int r = i / WQ, x = wx0 + 4 * (i - r * WQ), y = wy0 + r;
      uint2 v;
      bool fast = x >= fx0 && x + 4 <= fx1 && y >= fy0 && y < fy1;
      int n = 4;
      if (fast) {
        n = ((y >> log2) - ry + 1) * 3 + ((x >> lx) - rx + 1);
        const SaoLocal &p = sm.sao[comp][n];
        fast = !p.type || (quads && (p.type != 2 || (x >= p.ex0 && x + 4 <= p.ex1 && y >= p.ey0 && y < p.ey1)));
      }
      if (fast) {
        v = sao_quad_any(sm.fast[comp][n], &din[(y - dy0) * DP + (x - dx0)], maxv2);
      } else {
        const int ay = clampd(y, fy0, fy1 - 1);
        uint32_t s4[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int ax = clampd(x + k, fx0, fx1 - 1);
          const uint16_t *d = &din[(ay - dy0) * DP + (ax - dx0)];
          const SaoLocal &p = sm.sao[comp][((ay >> log2) - ry + 1) * 3 + ((ax >> lx) - rx + 1)];
          s4[k] = p.type ? (uint32_t)(uint16_t)sao_one(p, ax, ay, maxv, d) : *d;
        }
        v = make_uint2(s4[0] | s4[1] << 16, s4[2] | s4[3] << 16);
      }
      if (comp) seen |= v.x | v.y;
      st64(&out[r * P + (x - wx0)], make_uint2(v.x ^ kBias, v.y ^ kBias));
    }
  };
  constexpr int CQ = S::SCW / 4 * S::SCH % NT;  // a chroma window's leftover quads
  if (cc_any)
    window(0, sm.dL, sm.sL, X0 - 4, Y0 - 1, max(rect[0], 0), max(rect[1], 0), min(rect[2], pw), min(rect[3], ph), log2,
           2 * CQ % NT, std::integral_constant<int, S::SLW>{}, std::integral_constant<int, S::SLH>{});
#pragma unroll 1
  for (int cc = 0; cc < 2; ++cc)
    if (on[cc])
      window(1 + cc, sm.dC[cc], sm.sC[cc], xc0 - 4, yc0 - 2, max(rect[0] / SW, 0), max(rect[1], 0),
             min((rect[2] + SW - 1) / SW, a.src[1 + cc].w), min(rect[3], a.src[1 + cc].h), SW == 2 ? log2 - 1 : log2,
             cc * CQ, std::integral_constant<int, S::SCW>{}, std::integral_constant<int, S::SCH>{});
  const bool big = __syncthreads_or((seen & 0xC000C000u) != 0) != 0;
  const int j = tid / (TW / 4), i0 = (tid % (TW / 4)) * 4, gx = xc0 + i0, gy = yc0 + j, jr = gy - y_ctb;
#pragma unroll 1
  for (int cc = 0; cc < 2; ++cc) {
    const DPlane CD = a.dst[1 + cc];
    if (!on[cc] || gx >= CD.w || gy >= CD.h) continue;
    const int cf = a.do_alf && me ? me->chroma_filt[cc] : -1;
    const int ccf = a.do_alf && me && have_luma ? me->cc_filt[cc] : -1;
    const uint16_t *R0 = &sm.sC[cc][(j + 2) * S::SCP + i0 + 4];
    const uint2 w = ld64(R0);
    int v[4] = {(int)((w.x ^ kBias) & 0xFFFF), (int)((w.x ^ kBias) >> 16), (int)((w.y ^ kBias) & 0xFFFF),
                (int)((w.y ^ kBias) >> 16)};
    if (cf >= 0) chroma_alf_run<4>(R0, S::SCP, jr, ctb, a.tables.chroma_packed[min(cf, 7)], maxv, big, v);
    if (ccf >= 0) {  // CC-ALF (apply_cc_alf_ctb, src/alf.rs:447-523)
      const uint16_t *L0 = &sm.sL[(j + 1) * S::SLP + SW * i0 + 4];
      const bool lbb = !(gy + ctb >= ph && (ph - y_ctb) <= ctb - 4);
      const int32_t *k = a.tables.cc_coeff[cc][ccf];
      if (jr == ctb - 3 || jr == ctb - 4) {  // no correction beside the line buffer
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = clampd(v[q], 0, maxv);
      } else if constexpr (SW == 1) {
        cc_alf_run_444(L0, S::SLP, jr, ctb, lbb, k, bd, maxv, v);
      } else {
        cc_alf_run<4>(L0, S::SLP, jr, ctb, lbb, k, bd, maxv, v);
      }
    }
    uint16_t *out = CD.s + (int64_t)gy * CD.stride + gx;
    if (gx + 4 <= CD.w && ((uintptr_t)out & 7) == 0) {
      *reinterpret_cast<uint2 *>(out) =
          make_uint2((uint32_t)v[0] | (uint32_t)v[1] << 16, (uint32_t)v[2] | (uint32_t)v[3] << 16);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (gx + q < CD.w) out[q] = (uint16_t)v[q];
    }
  }
}

template <int TW, int SW>
__global__ void __launch_bounds__(SmemC<TW, SW>::NT, 1280 / SmemC<TW, SW>::NT) k_sao_alf_chroma(const __grid_constant__ Pass2Args a) {
  chroma_tile<TW, SW>(a, blockIdx.x);
}

// Many pictures in one grid, as k_sao_alf_tiles_batch.
template <int TW, int SW>
__global__ void __launch_bounds__(SmemC<TW, SW>::NT, 1280 / SmemC<TW, SW>::NT) k_sao_alf_chroma_batch(const Pass2Args *__restrict__ args,
                                                                            const uint32_t *__restrict__ first, int n) {
  __shared__ Pass2Args s_args;
  const int lo = tile_dev::batch_picture(first, n, blockIdx.x);
  const uint4 *src = reinterpret_cast<const uint4 *>(args + lo);
  uint4 *dst = reinterpret_cast<uint4 *>(&s_args);
  for (int i = threadIdx.x; i < (int)(sizeof(Pass2Args) / 16); i += blockDim.x) dst[i] = src[i];
  __syncthreads();
  chroma_tile<TW, SW>(s_args, (int)(blockIdx.x - first[lo]));
}

template <int W, int TH>
constexpr size_t smem3() {
  return sizeof(Smem3<W, TH>) + 128;
}

// W x TH of a picture's tiles: 64 x 64 (or 64 x 32 by tuning) for CTBs of 64
// and 128, 32 x 32 for 32 and for launches that would leave SMs without a tile.
inline int tile_w(const Pass2Args &a) { return a.ctb_log2 >= 6 && !a.small_tiles ? 64 : 32; }
inline int tile_h(const Pass2Args &a) { return tile_w(a) == 64 && a.tile_h == 32 ? 32 : tile_w(a); }

static_assert(sizeof(Smem3<64, 64>) + 128 + sizeof(Pass2Args) <= 48 * 1024, "default shared-memory limit of a CTA");

// Host-side driver API entry point for the tensor-map encoder (no libcuda link).
using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_fn() {
  static EncodeTiled fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiled>(p);
  }();
  return fn;
}

bool encode_plane(CUtensorMap *m, const DPlane &p, int box_w, int box_h) {
  const EncodeTiled enc = encode_fn();
  if (!enc || !p.s || p.w <= 0 || p.h <= 0) return false;
  if (((uintptr_t)p.s & 15) != 0 || (p.stride * 2) % 16 != 0 || p.stride < p.w) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)p.w, (cuuint64_t)p.h};
  const cuuint64_t strides[1] = {(cuuint64_t)p.stride * 2};
  const cuuint32_t box[2] = {(cuuint32_t)box_w, (cuuint32_t)box_h};
  const cuuint32_t estr[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, p.s, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

bool encode_plane_map(CUtensorMap *m, const DPlane &p, int box_w, int box_h) { return encode_plane(m, p, box_w, box_h); }

namespace {

template <int W, int TH>
void maps_for(Pass2Args &a) {
  using S = Smem3<W, TH>;
  bool ok = encode_plane(&a.tmap[0], a.src[0], S::DLW, S::DLH) || a.src[0].w <= 0 || a.src[0].h <= 0;
  for (int c = 1; c < 3 && ok; ++c)
    if (a.chroma && a.sub_h == 2 && a.src[c].w > 0 && a.src[c].h > 0) ok = encode_plane(&a.tmap[c], a.src[c], S::DCW, S::DCH);
  a.tma = ok ? 1 : 0;
}

template <int W, int TH>
int launch_one(cudaStream_t st, const Pass2Args &in, bool do_sao, bool do_alf) {
  Pass2Args a = in;
  a.tiles_x = (a.ext_w + W - 1) / W;
  a.tiles_y = (a.ext_h + TH - 1) / TH;
  const unsigned n = (unsigned)(a.tiles_x * a.tiles_y);
  const size_t shm = smem3<W, TH>();
  auto go = [&](auto kern) -> int {
    kern<<<n, NT3, shm, st>>>(a);
    H266_CUDA(cudaGetLastError());
    return H266_OK;
  };
  if (do_sao && do_alf) return go(k_sao_alf_tiles<W, TH, true, true>);
  if (do_sao) return go(k_sao_alf_tiles<W, TH, true, false>);
  if (do_alf) return go(k_sao_alf_tiles<W, TH, false, true>);
  return go(k_sao_alf_tiles<W, TH, false, false>);
}

}  // namespace

void pass2_tma_maps(Pass2Args &a) {
  if (tile_w(a) == 32) maps_for<32, 32>(a);
  else if (tile_h(a) == 32) maps_for<64, 32>(a);
  else maps_for<64, 64>(a);
}

int pass2_wait_timeouts(uint32_t *count) {
  unsigned int v = 0, zero = 0;
  H266_CUDA(cudaMemcpyFromSymbol(&v, g_wait_timeouts, sizeof v));
  if (v) H266_CUDA(cudaMemcpyToSymbol(g_wait_timeouts, &zero, sizeof zero));
  *count = v;
  return H266_OK;
}

namespace {
int sm_count() {
  static std::atomic<int> cached{0};
  int v = cached.load();
  if (!v) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      v = 148;
    cached.store(v);
  }
  return v;
}

}  // namespace

uint32_t pass2_large_tiles(const Pass2Args &a) {
  return a.ext_w > 0 && a.ext_h > 0 ? (uint32_t)((a.ext_w + 63) / 64) * (uint32_t)((a.ext_h + 63) / 64) : 0;
}

// One SM works on a 64 x 64 tile for 24 us, on a 32 x 32 one for 13 (a tile
// alone on its SM, bound by its phases' latencies), so launches of at most one
// large tile per SM run in small ones (416 x 240: 24 -> 13.6 us); with more, the
// SMs fill and the small tiles' wider borders cost more than they save.
bool pass2_small_tiles(uint32_t large_tiles) { return large_tiles <= (uint32_t)sm_count(); }

int pass2_packed_variant(Pass2Args &a, bool do_sao, bool do_alf, uint32_t *ctas) {
  const int W = tile_w(a), TH = tile_h(a);
  a.tiles_x = (a.ext_w + W - 1) / W;
  a.tiles_y = (a.ext_h + TH - 1) / TH;
  *ctas = a.ext_w > 0 && a.ext_h > 0 ? (uint32_t)(a.tiles_x * a.tiles_y) : 0;
  return (W == 32 ? 0 : (TH == 64 ? 8 : 4)) + (do_sao ? 2 : 0) + (do_alf ? 1 : 0);
}

namespace {
template <int W, int TH, bool DO_SAO, bool DO_ALF>
int launch_variant(cudaStream_t st, const Pass2Args *d_args, const uint32_t *d_first, int n, uint32_t ctas, int cps,
                   uint32_t *d_queue) {
  const size_t shm = smem3<W, TH>();
  if (cps > 0 && d_queue) {
    auto kern = k_sao_alf_tiles_queue<W, TH, DO_SAO, DO_ALF>;
    const uint32_t grid = std::min<uint32_t>(ctas, (uint32_t)(sm_count() * cps));
    kern<<<grid, NT3, shm, st>>>(d_args, d_first, n, ctas, d_queue);
  } else {
    auto kern = k_sao_alf_tiles_batch<W, TH, DO_SAO, DO_ALF>;
    kern<<<ctas, NT3, shm, st>>>(d_args, d_first, n);
  }
  H266_CUDA(cudaGetLastError());
  return H266_OK;
}
}  // namespace

int launch_pass2_packed_batch(cudaStream_t st, int variant, const Pass2Args *d_args, const uint32_t *d_first, int n,
                              uint32_t ctas, int ctas_per_sm, uint32_t *d_queue, uint64_t *launches) {
  if (!ctas || n <= 0) return H266_OK;
  int rc;
  const int c = ctas_per_sm;
  switch (variant) {
    case 11: rc = launch_variant<64, 64, true, true>(st, d_args, d_first, n, ctas, c, d_queue); break;
    case 10: rc = launch_variant<64, 64, true, false>(st, d_args, d_first, n, ctas, c, d_queue); break;
    case 9: rc = launch_variant<64, 64, false, true>(st, d_args, d_first, n, ctas, c, d_queue); break;
    case 8: rc = launch_variant<64, 64, false, false>(st, d_args, d_first, n, ctas, c, d_queue); break;
    case 7: rc = launch_variant<64, 32, true, true>(st, d_args, d_first, n, ctas, c, d_queue); break;
    case 6: rc = launch_variant<64, 32, true, false>(st, d_args, d_first, n, ctas, c, d_queue); break;
    case 5: rc = launch_variant<64, 32, false, true>(st, d_args, d_first, n, ctas, c, d_queue); break;
    case 4: rc = launch_variant<64, 32, false, false>(st, d_args, d_first, n, ctas, c, d_queue); break;
    case 3: rc = launch_variant<32, 32, true, true>(st, d_args, d_first, n, ctas, c, d_queue); break;
    case 2: rc = launch_variant<32, 32, true, false>(st, d_args, d_first, n, ctas, c, d_queue); break;
    case 1: rc = launch_variant<32, 32, false, true>(st, d_args, d_first, n, ctas, c, d_queue); break;
    default: rc = launch_variant<32, 32, false, false>(st, d_args, d_first, n, ctas, c, d_queue); break;
  }
  if (rc == H266_OK) ++*launches;
  return rc;
}

int pass2_chroma_variant(const Pass2Args &a, uint32_t *ctas) {
  if (!a.chroma || a.sub_h != 1) return -1;
  const int v = a.sub_w == 1 ? 0 : (a.ctb_log2 >= 6 ? 1 : 2), tw = v == 2 ? 16 : 32;
  const int h = std::max(a.src[1].h, a.src[2].h);
  *ctas = (uint32_t)(chroma_tiles_x(a, tw) * ((h + 31) / 32));
  return *ctas ? v : -1;
}

int launch_pass2_chroma_batch(cudaStream_t st, int variant, const Pass2Args *d_args, const uint32_t *d_first, int n,
                              uint32_t ctas, uint64_t *launches) {
  if (!ctas || n <= 0) return H266_OK;
  if (variant == 0) k_sao_alf_chroma_batch<32, 1><<<ctas, 256, 0, st>>>(d_args, d_first, n);
  else if (variant == 1) k_sao_alf_chroma_batch<32, 2><<<ctas, 256, 0, st>>>(d_args, d_first, n);
  else k_sao_alf_chroma_batch<16, 2><<<ctas, 128, 0, st>>>(d_args, d_first, n);
  H266_CUDA(cudaGetLastError());
  ++*launches;
  return H266_OK;
}

namespace {
int launch_pass2_chroma(cudaStream_t st, const Pass2Args &a, uint64_t *launches) {
  uint32_t ctas = 0;
  const int variant = pass2_chroma_variant(a, &ctas);
  if (variant < 0) return H266_OK;
  if (variant == 0) k_sao_alf_chroma<32, 1><<<ctas, 256, 0, st>>>(a);
  else if (variant == 1) k_sao_alf_chroma<32, 2><<<ctas, 256, 0, st>>>(a);
  else k_sao_alf_chroma<16, 2><<<ctas, 128, 0, st>>>(a);
  H266_CUDA(cudaGetLastError());
  ++*launches;
  return H266_OK;
}
}  // namespace

int launch_pass2_packed(cudaStream_t st, const Pass2Args &in, bool do_sao, bool do_alf, uint64_t *launches) {
  if (in.ext_w <= 0 || in.ext_h <= 0) return H266_OK;
  Pass2Args a = in;
  a.do_sao = do_sao;
  a.do_alf = do_alf;
  if (a.sub_h == 1 && a.chroma) {  // full-height chroma: its own tiles
    H266_TRY(launch_pass2_chroma(st, a, launches));
    a.chroma = 0;
  }
  const int rc = tile_w(a) == 64 ? (tile_h(a) == 32 ? launch_one<64, 32>(st, a, do_sao, do_alf)
                                                              : launch_one<64, 64>(st, a, do_sao, do_alf))
                                          : launch_one<32, 32>(st, a, do_sao, do_alf);
  if (rc == H266_OK) ++*launches;
  return rc;
}

}  // namespace h266
