// Encoder SAO decision (src/sao_enc.rs:44-487, sao_decide_picture): per CTB
// and component the band-offset and edge-offset statistics (count and sum of
// src - rec per band / per edge category of each class) gathered on the GPU,
// then the crate's decision arithmetic per CTB on the GPU.
//
// k_sao_stats: one CTA of 128 threads per (CTB, component, slice of about 4096
// samples); a thread takes pairs of samples down a column.  Every thread has
// its own bins in shared memory (bin-major, so a warp's accesses never meet in
// a bank): 32 bands and five edge sums of four classes, count and difference
// sum in one word (count << 24 plus the signed sum of at most 32 differences of
// 17 bits), so a sample costs five read-add-writes and no atomics; the bins are
// added up once per CTA.  The edge sums of a pair come from relu clamps on
// packed lanes.  26 us on a 1080p 10-bit picture (100 with warp matches and
// shared atomics for the bands and 32 predicated adds per sample for the edges).
// k_sao_decide: one warp per CTB, luma, Cb, then Cr within Cb's type
// (src/sao_enc.rs:450-477).
#include <climits>

#include <cstring>

#include "internal.h"

namespace h266 {
namespace {

constexpr int kStatThreads = 128;
constexpr int kSliceSamples = 4096;

struct SaoStats {  // one (CTB, component): sums over at most 128 x 128 samples of 16 bits
  int bo_cnt[32], bo_dif[32];
  int eo_cnt[4][5], eo_dif[4][5];  // category 0 is not gathered (the decision never reads it)
  unsigned vmax, inv_vmin;         // largest sample, and 65536 less the smallest (0: no sample)
};

struct SaoEncArgs {
  DPlane src[3], rec[3];
  int bd, log2, w_ctbs, h_ctbs, luma_on, chroma_on;
};

// The CTB region of component c (src/sao_enc.rs:398-420), clipped to the plane
// as try_band_offset / try_edge_offset_class do (x_end, y_end).
__device__ __forceinline__ bool sao_region(const SaoEncArgs &a, int c, int rx, int ry, int &x0, int &y0, int &x1,
                                           int &y1) {
  const int ctb = 1 << a.log2, pw = a.rec[0].w, ph = a.rec[0].h;
  const int cx = rx * ctb, cy = ry * ctb, cw = min(ctb, pw - cx), ch = min(ctb, ph - cy);
  if (c == 0) {
    x0 = cx;
    y0 = cy;
    x1 = min(cx + cw, a.rec[0].w);
    y1 = min(cy + ch, a.rec[0].h);
    return true;
  }
  if (cw / 2 <= 0 || ch / 2 <= 0) return false;
  x0 = cx / 2;
  y0 = cy / 2;
  x1 = min(x0 + cw / 2, a.rec[c].w);
  y1 = min(y0 + ch / 2, a.rec[c].h);
  return true;
}

// Samples (x, x + 1) of a row, 0 outside [0, w); `even`: the row starts on 4 bytes.
__device__ __forceinline__ uint32_t row_pair(const uint16_t *row, int x, int w, bool even) {
  if (x >= 0 && x + 1 < w && even) return *reinterpret_cast<const uint32_t *>(row + x);
  const uint32_t lo = x >= 0 && x < w ? row[x] : 0u, hi = x + 1 >= 0 && x + 1 < w ? row[x + 1] : 0u;
  return lo | hi << 16;
}

struct RowWin {  // samples x - 2 .. x + 3 of a row
  uint32_t a, b, c;
  __device__ uint32_t left() const { return __byte_perm(a, b, 0x5432); }   // (x - 1, x)
  __device__ uint32_t right() const { return __byte_perm(b, c, 0x5432); }  // (x + 1, x + 2)
};

// 2 - sign(c - n0) - sign(c - n1) of both samples of a pair (0..4 per lane).
// WIDE: samples of more than 14 bits, compared one by one; else every sample of
// the picture is below 2^14 or the call fails, and a larger neighbour (outside
// every CTB's region) compares like 2^15 - 2.
template <bool WIDE>
__device__ __forceinline__ uint32_t edge_sum(uint32_t c, uint32_t one_minus_c, uint32_t n0, uint32_t n1) {
  if (WIDE) {
    uint32_t r = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int v = (c >> (16 * k)) & 0xFFFF, p = (n0 >> (16 * k)) & 0xFFFF, q = (n1 >> (16 * k)) & 0xFFFF;
      r |= (uint32_t)(2 - (v > p) + (v < p) - (v > q) + (v < q)) << (16 * k);
    }
    return r;
  }
  const uint32_t two = 0x00020002u;
  return __viaddmin_s16x2_relu(n0, one_minus_c, two) + __viaddmin_s16x2_relu(n1, one_minus_c, two);
}

// The statistics of rows [y0, y1) x columns [x0, x1) of plane R against S,
// added into the zeroed `o`.  By the whole CTA; y1 - y0 rows of x1 - x0 samples
// are at most kSliceSamples.
template <bool WIDE>
__device__ __forceinline__ void stats_cta(const DPlane &R, const DPlane &S, int x0, int y0, int x1, int y1, int bd,
                                          SaoStats &o, uint32_t *err) {
  constexpr int kBins = 52;
  __shared__ uint32_t bin[kBins][kStatThreads];
  const int tid = threadIdx.x, lane = tid & 31, shift = bd - 5;
#pragma unroll 4
  for (int b = 0; b < kBins; ++b) bin[b][tid] = 0;  // own bins: no barrier until the sums
  int lp = 0;  // log2 of the threads per row
  while ((2 << lp) < x1 - x0) ++lp;
  const int groups = kStatThreads >> lp, rpt = (y1 - y0 + groups - 1) / groups;
  const int x = x0 + 2 * (tid & ((1 << lp) - 1));
  const int ya = y0 + (tid >> lp) * rpt, yb = min(y1, ya + rpt);
  const bool r_even = ((uintptr_t)R.s & 3) == 0 && (R.stride & 1) == 0 && (x & 1) == 0;
  const bool s_even = ((uintptr_t)S.s & 3) == 0 && (S.stride & 1) == 0 && (x & 1) == 0;
  uint32_t hi2 = 0, lo2 = 0xFFFFFFFFu;  // per lane: the largest and smallest counted samples
  bool above = false;
  if (x < x1) {
    // inside: every sample x - 2 .. x + 3 lies in the row, both rows start on 4 bytes, both samples count
    const bool inside = x >= 2 && x + 3 < R.w && r_even && s_even && x + 1 < x1 && x + 1 < S.w;
    const uint16_t *rp = R.s + (int64_t)ya * R.stride + x;
    auto row = [&](int y, const uint16_t *p) {  // p: sample x of row y
      if (y < 0 || y >= R.h) return RowWin{0, 0, 0};
      RowWin w;
      if (inside) {
        const uint32_t *q = reinterpret_cast<const uint32_t *>(p);
        w = RowWin{q[-1], q[0], q[1]};
      } else {
        w = RowWin{row_pair(p - x, x - 2, R.w, r_even), row_pair(p - x, x, R.w, r_even),
                   row_pair(p - x, x + 2, R.w, r_even)};
      }
      if (!WIDE) {
        w.a = __vminu2(w.a, 0x7FFE7FFEu);
        w.c = __vminu2(w.c, 0x7FFE7FFEu);
      }
      return w;
    };
    auto org = [&](int y, const uint16_t *p) {
      if (inside && y < S.h) return *reinterpret_cast<const uint32_t *>(p);
      return y < S.h ? row_pair(p - x, x, S.w, s_even) : 0u;
    };
    const uint16_t *sp = S.s + (int64_t)ya * S.stride + x;
    RowWin up = row(ya - 1, rp - R.stride), cur = row(ya, rp), dn = row(ya + 1, rp + R.stride);
    uint32_t s = org(ya, sp);
    char *own = reinterpret_cast<char *>(&bin[0][tid]);  // bin b of this thread at own + b * kBin
    constexpr int kBin = kStatThreads * 4;
    for (int y = ya; y < yb; ++y) {
      const RowWin next = row(y + 2, rp + 2 * R.stride);  // a row ahead of its use
      const uint32_t s_next = org(y + 1, sp + S.stride);
      const uint32_t c = cur.b, n = WIDE ? 0u : __viaddmax_s16x2(~c, 0x00020002u, 0x80008000u);  // 1 - c
      const uint32_t ub = WIDE ? up.b : __vminu2(up.b, 0x7FFE7FFEu), db = WIDE ? dn.b : __vminu2(dn.b, 0x7FFE7FFEu);
      const RowWin u{up.a, ub, up.c}, d{dn.a, db, dn.c};
      // byte offsets of both samples' bins in their class
      uint32_t e[4] = {edge_sum<WIDE>(c, n, cur.left(), cur.right()) * kBin, edge_sum<WIDE>(c, n, ub, db) * kBin,
                       edge_sum<WIDE>(c, n, u.left(), d.right()) * kBin,
                       edge_sum<WIDE>(c, n, u.right(), d.left()) * kBin};
      constexpr uint32_t kNone = 2u * kBin * 0x00010001u;
      if (y == 0 || y + 1 >= R.h) e[1] = e[2] = e[3] = kNone;  // EO_DIRS, src/sao_enc.rs:166-171: both neighbours inside
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int px = x + k;
        if (!inside) {
          if (px >= x1 || px >= S.w || y >= S.h) continue;
          if (px == 0 || px + 1 >= R.w) {
            const uint32_t m = 0xFFFFu << (16 * k);
            e[0] = (e[0] & ~m) | (kNone & m);
            e[2] = (e[2] & ~m) | (kNone & m);
            e[3] = (e[3] & ~m) | (kNone & m);
          }
        } else if (y >= S.h) {
          continue;
        }
        const uint32_t r = (c >> (16 * k)) & 0xFFFF;
        const uint32_t add = (1u << 24) + ((s >> (16 * k)) & 0xFFFF) - r;
        hi2 = max(hi2, r);
        lo2 = min(lo2, r);
        // the sample's band and its sum in each class: five different bins
        const uint32_t band = r >> shift;
        above |= band > 31;  // a sample above 2^BitDepth - 1: no band in the crate, and the call fails
        uint32_t *at[5];
        at[4] = reinterpret_cast<uint32_t *>(own + min(band, 31u) * kBin);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          at[q] = reinterpret_cast<uint32_t *>(own + ((e[q] >> (16 * k)) & 0xFFFF) + (32 + 5 * q) * kBin);
        uint32_t v[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) v[q] = *at[q];
#pragma unroll
        for (int q = 0; q < 5; ++q) *at[q] = v[q] + add;
      }
      up = cur;
      cur = dn;
      dn = next;
      s = s_next;
      rp += R.stride;
      sp += S.stride;
    }
  }
  uint32_t vmax = hi2, imin = lo2 > 65535u ? 0u : 65536u - lo2;
  if (above) atomicOr(err, 1u);
  vmax = __reduce_max_sync(0xFFFFFFFFu, vmax);
  imin = __reduce_max_sync(0xFFFFFFFFu, imin);
  if (lane == 0) {
    atomicMax(&o.vmax, vmax);
    atomicMax(&o.inv_vmin, imin);
  }
  __syncthreads();
  for (int b = tid >> 5; b < kBins; b += kStatThreads / 32) {
    const int q = (b - 32) / 5, i = (b - 32) % 5;  // edge sums 0, 1, 3, 4 are categories 4, 3, 2, 1 (eo_category)
    if (b >= 32 && i == 2) continue;
    int cnt = 0, dif = 0;
#pragma unroll
    for (int t = lane; t < kStatThreads; t += 32) {
      const uint32_t w = bin[b][t];
      const int d = (int)(w << 8) >> 8;
      dif += d;
      cnt += (int)((w - (uint32_t)d) >> 24);
    }
    cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
    dif = __reduce_add_sync(0xFFFFFFFFu, dif);
    if (lane || !cnt) continue;
    const int cat = i < 2 ? 4 - i : 5 - i;
    atomicAdd(b < 32 ? &o.bo_cnt[b] : &o.eo_cnt[q][cat], cnt);
    atomicAdd(b < 32 ? &o.bo_dif[b] : &o.eo_dif[q][cat], dif);
  }
}

__host__ __device__ inline int slice_rows(int ctb_w) { return ctb_w >= kSliceSamples ? 1 : kSliceSamples / ctb_w; }

// Statistics are added into the zeroed `out`.  blockIdx: CTB, component, slice.
template <bool WIDE>
__global__ void __launch_bounds__(kStatThreads) k_sao_stats(const __grid_constant__ SaoEncArgs a,
                                                            SaoStats *__restrict__ out, uint32_t *__restrict__ err) {
  const int ctb_i = blockIdx.x, c = blockIdx.y;
  const int rx = ctb_i % a.w_ctbs, ry = ctb_i / a.w_ctbs;
  int x0, y0, x1, y1;
  if (!(c == 0 ? a.luma_on : a.chroma_on) || !sao_region(a, c, rx, ry, x0, y0, x1, y1)) return;
  const int rows = slice_rows((1 << a.log2) >> (c ? 1 : 0));
  y0 += blockIdx.z * rows;
  y1 = min(y1, y0 + rows);
  if (x1 <= x0 || y1 <= y0) return;  // uniform per CTA
  stats_cta<WIDE>(a.rec[c], a.src[c], x0, y0, x1, y1, a.bd, out[(size_t)ctb_i * 3 + c], err);
}

__device__ void sao_offsets(h266_sao_ctb &c, const int abs_[4], const uint32_t sign[4], int bd) {
  const int shift = bd - min(bd, 10);  // derive_offset_val, src/sao.rs:356-365
  c.offset_val[0] = 0;
  for (int i = 0; i < 4; ++i) c.offset_val[i + 1] = (1 - 2 * (int)(sign[i] & 1)) * (abs_[i] << shift);
}

// Band and edge candidates of one component from its statistics, one warp
// (every lane returns the same values):
//  * try_band_offset (src/sao_enc.rs:77-171): lane b holds band b's clipped
//    optimum; lane st < 28 the delta of the 4 bands from st; the first
//    minimum wins (the crate's strict < scan from start 0);
//  * try_edge_offset_class (src/sao_enc.rs:211-284): lane 4k + q - 1 holds
//    category q of class k (offset from |diff|, as there).
struct Candidates {
  long long bo_delta;
  int bo_start, bo_off[4];
  long long eo_delta[4];
  int eo_off[4][4];
};

__device__ Candidates candidates(const SaoStats &s, int bd, int lane) {
  Candidates c;
  const long long cmax = (1ll << (min(bd, 10) - 5)) - 1;
  const int n = s.bo_cnt[lane], dif = s.bo_dif[lane];  // at most 2^14 samples of 17-bit differences
  long long opt = 0;
  if (n > 0) {
    opt = (dif + n / 2) / n;
    opt = opt < -cmax ? -cmax : (opt > cmax ? cmax : opt);
  }
  const long long term = n > 0 ? dif * opt : 0;
  long long delta = -(term + __shfl_down_sync(0xffffffffu, term, 1) + __shfl_down_sync(0xffffffffu, term, 2) +
                      __shfl_down_sync(0xffffffffu, term, 3));
  if (lane >= 28) delta = LLONG_MAX;
  int idx = lane;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const long long ov = __shfl_xor_sync(0xffffffffu, delta, o);
    const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (ov < delta || (ov == delta && oi < idx)) {
      delta = ov;
      idx = oi;
    }
  }
  c.bo_delta = delta;
  c.bo_start = idx;
#pragma unroll
  for (int i = 0; i < 4; ++i) c.bo_off[i] = (int)__shfl_sync(0xffffffffu, opt, idx + i);
  const int k = (lane >> 2) & 3, q = (lane & 3) + 1;
  const int en = lane < 16 ? s.eo_cnt[k][q] : 0;
  const int ad = lane < 16 ? abs(s.eo_dif[k][q]) : 0;
  long long eo = 0;
  if (en > 0) {
    eo = (ad + en / 2) / en;
    eo = eo < 0 ? 0 : (eo > 7 ? 7 : eo);
  }
  long long et = ad * eo;
  et += __shfl_xor_sync(0xffffffffu, et, 1);
  et += __shfl_xor_sync(0xffffffffu, et, 2);
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    c.eo_delta[kk] = -__shfl_sync(0xffffffffu, et, 4 * kk);
#pragma unroll
    for (int qq = 0; qq < 4; ++qq) c.eo_off[kk][qq] = (int)__shfl_sync(0xffffffffu, eo, 4 * kk + qq);
  }
  return c;
}

__device__ h266_sao_ctb band_ctb(const Candidates &c, int bd) {  // SaoCtb::band_offset, src/sao.rs:150-167
  h266_sao_ctb out{};
  int ab[4];
  uint32_t sg[4];
  for (int i = 0; i < 4; ++i) {
    ab[i] = c.bo_off[i] < 0 ? -c.bo_off[i] : c.bo_off[i];
    sg[i] = c.bo_off[i] < 0 ? 1u : 0u;
  }
  out.sao_type_idx = 1;
  out.band_position = (uint8_t)(c.bo_start & 31);
  sao_offsets(out, ab, sg, bd);
  return out;
}

__device__ h266_sao_ctb edge_ctb(const Candidates &c, int cls, int bd) {  // SaoCtb::edge_offset, src/sao.rs:169-180
  h266_sao_ctb out{};
  const uint32_t sign[4] = {0, 0, 1, 1};
  out.sao_type_idx = 2;
  out.eo_class = (uint8_t)cls;
  sao_offsets(out, c.eo_off[cls], sign, bd);
  return out;
}

__device__ h266_sao_ctb decide(const Candidates &c, int bd) {  // sao_decide_ctb, src/sao_enc.rs:44-70
  long long best = 0;
  int cls = -1;
  for (int k = 0; k < 4; ++k)  // try_best_edge_offset, src/sao_enc.rs:175-209
    if (c.eo_delta[k] < best) {
      best = c.eo_delta[k];
      cls = k;
    }
  if (cls >= 0) return edge_ctb(c, cls, bd);
  if (c.bo_delta < 0) return band_ctb(c, bd);
  return h266_sao_ctb{};
}

// One warp per CTB.
__global__ void k_sao_decide(const __grid_constant__ SaoEncArgs a, const SaoStats *__restrict__ st,
                             const uint32_t *__restrict__ err, h266_sao_ctb_params *__restrict__ out) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= a.w_ctbs * a.h_ctbs) return;  // uniform per warp
  if (i == 0 && lane == 0) *reinterpret_cast<uint32_t *>(out + a.w_ctbs * a.h_ctbs) = *err;  // read back with the records
  const int rx = i % a.w_ctbs, ry = i / a.w_ctbs;
  h266_sao_ctb_params p{};
  if (a.luma_on) {
    const Candidates c = candidates(st[(size_t)i * 3], a.bd, lane);
    p.luma = decide(c, a.bd);
  }
  int x0, y0, x1, y1;
  if (a.chroma_on && sao_region(a, 1, rx, ry, x0, y0, x1, y1)) {
    const Candidates cb = candidates(st[(size_t)i * 3 + 1], a.bd, lane);
    const Candidates cr = candidates(st[(size_t)i * 3 + 2], a.bd, lane);
    p.cb = decide(cb, a.bd);
    if (p.cb.sao_type_idx == 1) {  // sao_decide_ctb_constrained, src/sao_enc.rs:286-347
      if (cr.bo_delta < 0) {
        p.cr = band_ctb(cr, a.bd);
      } else {
        p.cr.sao_type_idx = 1;
      }
    } else if (p.cb.sao_type_idx == 2) {
      const int cls = p.cb.eo_class;
      if (cr.eo_delta[cls] < 0) {
        p.cr = edge_ctb(cr, cls, a.bd);
      } else {
        p.cr.sao_type_idx = 2;
        p.cr.eo_class = (uint8_t)cls;
      }
    }
  }
  if (lane == 0) out[i] = p;
}

// ---- chroma SAO merge (apply_chroma_sao_merge, src/sao_enc.rs:500-668)
//
// Raster-order dependency: a CTB weighs its own parameters against the
// already merged left and above CTBs, so CTBs run one anti-diagonal per
// launch (both neighbours lie on the previous diagonal).  Per CTB and
// candidate: the SAO of this CTB alone on the pre-SAO planes
// (apply_sao_ctb, src/sao.rs:504-626, no clip rectangle) and the Cb + Cr SSE
// against the original (chroma_ctb_sse_with, src/sao_enc.rs:698-749), then
// the decision by cost SSE + 8 * bits (strict <: independent, left, above).
struct MergeArgs {
  DPlane src[2], pre[2];  // Cb, Cr
  int bd, chr_ctb, w_ctbs;
  const h266_sao_ctb_params *indep;
  h266_sao_ctb_params *merged;
  uint8_t *map;
  unsigned long long *sse;  // [ctb][3]
  unsigned int *count;      // per CTB, zero at the start
  // the wavefront form
  int h_ctbs;
  int max_off;      // largest |offset| of the picture's applied parameters
  SaoStats *stats;  // [ctb][2], zero at the start
  int32_t *from;    // per CTB the CTB whose independent parameters it took
  int32_t *status;  // 1: decided; 0: too many CTBs near the ends of the sample range, left to the diagonals
};

__device__ __forceinline__ int sao_value(const DPlane &P, int x, int y, const h266_sao_ctb &p, int maxv, int bd) {
  const int v = P.s[(int64_t)y * P.stride + x];
  if (p.sao_type_idx == 2) {
    const int c = p.eo_class & 3;
    const int hx = c == 1 ? 0 : (c == 3 ? 1 : -1), vy = c == 0 ? 0 : -1;  // hPos / vPos of neighbour 0
    const int ax = x + hx, ay = y + vy, bx = x - hx, by = y - vy;
    if (ax < 0 || ay < 0 || bx < 0 || by < 0 || ax >= P.w || ay >= P.h || bx >= P.w || by >= P.h)
      return min(max(v, 0), maxv);
    const int n0 = P.s[(int64_t)ay * P.stride + ax], n1 = P.s[(int64_t)by * P.stride + bx];
    int e = 2 + ((v > n0) - (v < n0)) + ((v > n1) - (v < n1));
    if (e <= 2) e = e == 2 ? 0 : e + 1;
    const int off = (e >= 1 && e <= 4) ? p.offset_val[e] : 0;
    return min(max(v + off, 0), maxv);
  }
  if (p.sao_type_idx == 1) {
    const int band = (v >> (bd - 5)) & 31;
    const int k = (band - p.band_position) & 31;
    const int off = k < 4 ? p.offset_val[k + 1] : 0;
    return min(max(v + off, 0), maxv);
  }
  return v;  // not applied: the sample as it is
}

constexpr int kMergeThreads = 512;

// One CTA per (CTB of the diagonal, candidate): the candidate's Cb + Cr SSE,
// stored per CTB; the CTA that completes a CTB's set of candidates (per-CTB
// arrival counter, zeroed by the host; no CTA waits for another) makes the
// decision.
__device__ __forceinline__ void merge_cta(const MergeArgs &a, int ry, int rx, int k) {
  if ((k == 1 && rx == 0) || (k == 2 && ry == 0)) return;  // no such neighbour (uniform per CTA)
  const int i = ry * a.w_ctbs + rx;
  const int tid = threadIdx.x, maxv = (1 << a.bd) - 1;
  const int cx = rx * a.chr_ctb, cy = ry * a.chr_ctb;
  const int cw = max(0, min(a.chr_ctb, a.pre[0].w - cx)), ch = max(0, min(a.chr_ctb, a.pre[0].h - cy));
  const h266_sao_ctb_params &cand = k == 0 ? a.indep[i] : (k == 1 ? a.merged[i - 1] : a.merged[i - a.w_ctbs]);
  const h266_sao_ctb pc[2] = {cand.cb, cand.cr};
  unsigned long long e = 0;
  for (int y = cy + tid / 32; y < cy + ch; y += kMergeThreads / 32)
    for (int x = cx + (tid & 31); x < cx + cw; x += 32)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int d = (int)a.src[c].s[(int64_t)y * a.src[c].stride + x] - sao_value(a.pre[c], x, y, pc[c], maxv, a.bd);
        e += (unsigned long long)((long long)d * d);
      }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
  __shared__ unsigned long long part[kMergeThreads / 32];
  if ((tid & 31) == 0) part[tid / 32] = e;
  __syncthreads();
  if (tid) return;
  unsigned long long t = 0;
  for (int w = 0; w < kMergeThreads / 32; ++w) t += part[w];
  a.sse[(size_t)i * 3 + k] = t;
  __threadfence();
  const unsigned n_cand = 1u + (rx > 0) + (ry > 0);
  if (atomicAdd(&a.count[i], 1u) != n_cand - 1) return;
  __threadfence();
  unsigned long long sse[3];
  for (int q = 0; q < 3; ++q) sse[q] = __ldcg(&a.sse[(size_t)i * 3 + q]);
  auto bits = [](const h266_sao_ctb_params &p) {  // chroma_independent_bit_cost, src/sao_enc.rs:670-696
    long long b = 1;
    b += p.cb.sao_type_idx == 0 ? 1 : (p.cb.sao_type_idx == 1 ? 16 : 10);
    b += p.cr.sao_type_idx == 0 ? 1 : (p.cr.sao_type_idx == 1 ? 16 : 10);
    return b;
  };
  const h266_sao_ctb_params in = a.indep[i];
  long long best = (long long)sse[0] + 8 * bits(in);
  int choice = 0;
  h266_sao_ctb_params out = in;
  if (rx > 0 && (long long)sse[1] + 8 < best) {
    best = (long long)sse[1] + 8;
    choice = 1;
    out.cb = a.merged[i - 1].cb;
    out.cr = a.merged[i - 1].cr;
  }
  if (ry > 0 && (long long)sse[2] + 16 < best) {
    choice = 2;
    out.cb = a.merged[i - a.w_ctbs].cb;
    out.cr = a.merged[i - a.w_ctbs].cr;
  }
  a.merged[i] = out;
  a.map[i] = (uint8_t)choice;
}

// One anti-diagonal `diag` of many pictures: CTAs [first[p], first[p + 1]) of
// the x dimension are picture p's CTBs on it (from its first row up), y the
// candidate.  Pictures without CTBs on the diagonal have none.
__global__ void __launch_bounds__(kMergeThreads) k_sao_merge_diag_batch(const MergeArgs *__restrict__ args,
                                                                         const uint32_t *__restrict__ first, int n,
                                                                         int diag) {
  int lo = 0, hi = n;  // first[lo] <= blockIdx.x < first[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (first[mid] <= blockIdx.x) lo = mid;
    else hi = mid;
  }
  const MergeArgs &a = args[lo];
  const int ry0 = max(0, diag - (a.w_ctbs - 1));
  const int ry = ry0 + (int)(blockIdx.x - first[lo]);
  merge_cta(a, ry, diag - ry, blockIdx.y);
}

// ---- the merge from statistics
//
// SAO adds one offset to every sample of a band or edge category, so a
// candidate changes a CTB's SSE by sum(n off^2 - 2 off sum(src - rec)) over its
// four bands or categories: with the statistics of every CTB (gathered in
// parallel, k_merge_stats) a candidate costs eight terms instead of a pass over
// its samples, and the raster dependency is one CTA walking the anti-diagonals
// with a warp per CTB (k_merge_wave; the SSE without SAO is in every cost and
// drops out).  1080p 10-bit: 23 launches of 17 us become two, of 22 and 31 us.
// That holds where no sample clips.  A candidate that could clip some sample of
// its CTB (the CTB's extremes against the candidate's offsets) is summed from
// the samples by its warp; a picture with more than n / 32 + 4 CTBs within the
// largest offset of the range's ends is left to the diagonal launches, and one of
// more than kSaoWaveRows CTB rows never comes here (its choices would not fit, and
// its statistics take 850 bytes a CTB, more than the CTB where that is small).

// blockIdx: CTB, Cb or Cr, picture.
template <bool WIDE>
__global__ void __launch_bounds__(kStatThreads) k_merge_stats(const MergeArgs *__restrict__ args) {
  const MergeArgs &a = args[blockIdx.z];
  const int i = blockIdx.x, c = blockIdx.y;
  if (i >= a.w_ctbs * a.h_ctbs) return;
  const DPlane R = a.pre[c], S = a.src[c];
  const int x0 = (i % a.w_ctbs) * a.chr_ctb, y0 = (i / a.w_ctbs) * a.chr_ctb;
  const int x1 = min(x0 + a.chr_ctb, R.w), y1 = min(y0 + a.chr_ctb, R.h);
  __shared__ uint32_t err;  // a sample above the depth shows in vmax
  if (x1 <= x0 || y1 <= y0) return;
  stats_cta<WIDE>(R, S, x0, y0, x1, y1, a.bd, a.stats[(size_t)i * 2 + c], &err);
}

// The SSE change of parameters p on component c's region of a CTB, from the
// samples, by one warp.
__device__ long long merge_delta_direct(const MergeArgs &a, int c, int cx, int cy, const h266_sao_ctb &p) {
  const int lane = threadIdx.x & 31, maxv = (1 << a.bd) - 1;
  const int x1 = min(cx + a.chr_ctb, a.pre[c].w), y1 = min(cy + a.chr_ctb, a.pre[c].h);
  long long e = 0;
  for (int y = cy; y < y1; ++y)
    for (int x = cx + lane; x < x1; x += 32) {
      const int s = a.src[c].s[(int64_t)y * a.src[c].stride + x], v = a.pre[c].s[(int64_t)y * a.pre[c].stride + x];
      const long long d1 = s - sao_value(a.pre[c], x, y, p, maxv, a.bd), d0 = s - v;
      e += d1 * d1 - d0 * d0;
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  return e;
}

constexpr int kWaveThreads = 512;

// One CTA per picture.
__global__ void __launch_bounds__(kWaveThreads) k_merge_wave(const MergeArgs *__restrict__ args) {
  const MergeArgs a = args[blockIdx.x];
  const int n = a.w_ctbs * a.h_ctbs, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int maxv = (1 << a.bd) - 1;
  int near = 0;
  for (int i = tid; i < n; i += kWaveThreads)
    for (int c = 0; c < 2; ++c) {
      const SaoStats &s = a.stats[(size_t)i * 2 + c];
      near += s.inv_vmin && ((int)s.vmax > maxv - a.max_off || 65536 - (int)s.inv_vmin < a.max_off);
    }
  __shared__ int s_near;
  if (tid == 0) s_near = 0;
  __syncthreads();
  if (near) atomicAdd(&s_near, near);
  __syncthreads();
  const bool go = s_near <= 2 * (n / 32 + 4);
  if (tid == 0) *a.status = go ? 1 : 0;
  if (!go) return;
  // The last two diagonals' choices by CTB row: what a neighbour's candidate needs.
  struct Choice {
    int type, band, cls, from;
    int off[4];
  };
  __shared__ Choice ring[2][kSaoWaveRows][2];
  // lane 8 k + 4 c + j: offset j of component c of candidate k (own, left, above)
  const int k = lane >> 3, c = (lane >> 2) & 1, j = lane & 3;
  // A CTB's statistics and its own parameters, loaded while the diagonal before
  // it runs: lane l holds band l and edge entry l (class * 5 + category, l < 20)
  // of both components.
  struct Ahead {
    int bc[2], bd[2], ec[2], ed[2], hi[2], lo[2];
    int type, band, cls, off;
  };
  auto load = [&](int d, int ry) {
    Ahead h{};
    const int ry0 = max(0, d - (a.w_ctbs - 1)), ry1 = min(a.h_ctbs - 1, d);
    if (ry < ry0 || ry > ry1 || d > a.w_ctbs + a.h_ctbs - 2) return h;
    const int i = ry * a.w_ctbs + d - ry;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const SaoStats &s = a.stats[(size_t)i * 2 + q];
      h.bc[q] = s.bo_cnt[lane];
      h.bd[q] = s.bo_dif[lane];
      h.ec[q] = (&s.eo_cnt[0][0])[min(lane, 19)];
      h.ed[q] = (&s.eo_dif[0][0])[min(lane, 19)];
      h.hi[q] = s.inv_vmin ? (int)s.vmax : -1;  // no sample: -1
      h.lo[q] = 65536 - (int)s.inv_vmin;
    }
    const h266_sao_ctb &p = c ? a.indep[i].cr : a.indep[i].cb;
    h.type = p.sao_type_idx;
    h.band = p.band_position;
    h.cls = p.eo_class & 3;
    h.off = p.offset_val[j + 1];
    return h;
  };
  Ahead next = load(0, warp);
  for (int d = 0; d <= a.w_ctbs + a.h_ctbs - 2; ++d) {
    const int ry0 = max(0, d - (a.w_ctbs - 1)), ry1 = min(a.h_ctbs - 1, d);
    for (int ry = ry0 + warp; ry <= ry1; ry += kWaveThreads / 32) {
      const int rx = d - ry, i = ry * a.w_ctbs + rx;
      const Ahead h = ry == ry0 + warp ? next : load(d, ry);
      const bool have = k == 0 || (k == 1 && rx > 0) || (k == 2 && ry > 0);
      int type = h.type, band = h.band, cls = h.cls, off32 = h.off, from = i;
      if (k && have && k < 3) {
        const Choice &q = ring[(d - 1) & 1][ry - (k == 2)][c];
        type = q.type;
        band = q.band;
        cls = q.cls;
        off32 = q.off[j];
        from = q.from;
      }
      const int b = (band + j) & 31, en = (cls * 5 + j + 1) & 31;
      // every lane takes part in the exchanges
      const int bc0 = __shfl_sync(0xffffffffu, h.bc[0], b), bc1 = __shfl_sync(0xffffffffu, h.bc[1], b);
      const int bd0 = __shfl_sync(0xffffffffu, h.bd[0], b), bd1 = __shfl_sync(0xffffffffu, h.bd[1], b);
      const int ec0 = __shfl_sync(0xffffffffu, h.ec[0], en), ec1 = __shfl_sync(0xffffffffu, h.ec[1], en);
      const int ed0 = __shfl_sync(0xffffffffu, h.ed[0], en), ed1 = __shfl_sync(0xffffffffu, h.ed[1], en);
      long long e = 0;
      bool clips = false;
      const int hi = c ? h.hi[1] : h.hi[0], lo = c ? h.lo[1] : h.lo[0];
      if (have && k < 3 && (type == 1 || type == 2) && hi >= 0) {
        const long long off = off32;
        const long long cnt = type == 1 ? (c ? bc1 : bc0) : (c ? ec1 : ec0);
        const long long dif = type == 1 ? (c ? bd1 : bd0) : (c ? ed1 : ed0);
        e = cnt * off * off - 2 * off * dif;
        clips = hi + max(off, 0ll) > maxv || lo + min(off, 0ll) < 0;
      }
      // the candidate's sum over its 8 lanes
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
      const unsigned m = __ballot_sync(0xffffffffu, clips);
      long long sum[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) sum[q] = __shfl_sync(0xffffffffu, e, 8 * q);
      if (m) {  // uniform over the warp
        for (int q = 0; q < 3; ++q) {
          if (!(m >> (8 * q) & 0xFFu)) continue;
          const int src = __shfl_sync(0xffffffffu, from, 8 * q);
          sum[q] = merge_delta_direct(a, 0, rx * a.chr_ctb, ry * a.chr_ctb, a.indep[src].cb) +
                   merge_delta_direct(a, 1, rx * a.chr_ctb, ry * a.chr_ctb, a.indep[src].cr);
        }
      }
      auto bits = [](int t) { return t == 0 ? 1 : (t == 1 ? 16 : 10); };
      const int own = 1 + bits(__shfl_sync(0xffffffffu, h.type, 0)) + bits(__shfl_sync(0xffffffffu, h.type, 4));
      long long best = sum[0] + 8 * own;  // chroma_independent_bit_cost
      int choice = 0;
      if (rx > 0 && sum[1] + 8 < best) {
        best = sum[1] + 8;
        choice = 1;
      }
      if (ry > 0 && sum[2] + 16 < best) choice = 2;
      if (k == choice) {  // the chosen candidate's 8 lanes pass it on
        Choice &q = ring[d & 1][ry][c];
        q.off[j] = off32;
        if (j == 0) {
          q.type = type;
          q.band = band;
          q.cls = cls;
          q.from = from;
        }
        if (lane == 8 * k) {
          a.from[i] = from;
          a.map[i] = (uint8_t)choice;
        }
      }
    }
    next = load(d + 1, max(0, d + 1 - (a.w_ctbs - 1)) + warp);
    __syncthreads();  // the next diagonal reads this one's choices
  }
  // the records
  for (int i = tid; i < n; i += kWaveThreads) {
    h266_sao_ctb_params out = a.indep[i];
    const int f = a.from[i];
    if (a.map[i]) {
      out.cb = a.indep[f].cb;
      out.cr = a.indep[f].cr;
    }
    a.merged[i] = out;
  }
}

}  // namespace

size_t sao_merge_args_size() { return sizeof(MergeArgs); }

void fill_sao_merge_args(void *out, const DPlane src[2], const DPlane pre[2], int bd, int chr_ctb, int w_ctbs,
                         int h_ctbs, int max_off, const h266_sao_ctb_params *d_indep, h266_sao_ctb_params *d_merged,
                         uint8_t *d_map, void *d_work, int32_t *d_status) {
  MergeArgs a{};
  for (int c = 0; c < 2; ++c) {
    a.src[c] = src[c];
    a.pre[c] = pre[c];
  }
  a.bd = bd;
  a.chr_ctb = chr_ctb;
  a.w_ctbs = w_ctbs;
  a.h_ctbs = h_ctbs;
  a.indep = d_indep;
  a.merged = d_merged;
  a.map = d_map;
  a.max_off = max_off;
  // the layout of sao_merge_work_bytes, zeroed by the caller
  const size_t n = (size_t)w_ctbs * h_ctbs;
  a.status = d_status;
  a.sse = static_cast<unsigned long long *>(d_work);
  a.count = reinterpret_cast<unsigned int *>(a.sse + n * 3);
  a.from = reinterpret_cast<int32_t *>(a.count + n);
  a.stats = reinterpret_cast<SaoStats *>(a.from + n);
  std::memcpy(out, &a, sizeof a);
}

size_t sao_merge_work_bytes(size_t n, bool wave) { return n * (3 * 8 + 4 + (wave ? 4 + 2 * sizeof(SaoStats) : 0)); }

int launch_sao_merge_wave(cudaStream_t st, const void *d_args, int n, int max_ctbs, bool wide, uint64_t *launches) {
  if (n <= 0 || max_ctbs <= 0) return H266_OK;
  const MergeArgs *args = static_cast<const MergeArgs *>(d_args);
  for (int i0 = 0; i0 < n; i0 += 65535) {  // the z dimension of a grid
    const dim3 grid(max_ctbs, 2, std::min(n - i0, 65535));
    if (wide) k_merge_stats<true><<<grid, kStatThreads, 0, st>>>(args + i0);
    else k_merge_stats<false><<<grid, kStatThreads, 0, st>>>(args + i0);
    H266_CUDA(cudaGetLastError());
    ++*launches;
  }
  k_merge_wave<<<n, kWaveThreads, 0, st>>>(args);
  H266_CUDA(cudaGetLastError());
  ++*launches;
  return H266_OK;
}

int launch_sao_chroma_merge_batch(cudaStream_t st, const void *d_args, const uint32_t *d_first, int n, int n_diags,
                                  const uint32_t *h_totals, uint64_t *launches) {
  const MergeArgs *args = static_cast<const MergeArgs *>(d_args);
  for (int d = 0; d < n_diags; ++d) {
    if (!h_totals[d]) continue;
    k_sao_merge_diag_batch<<<dim3(h_totals[d], 3), kMergeThreads, 0, st>>>(args, d_first + (size_t)d * (n + 1), n, d);
    H266_CUDA(cudaGetLastError());
    ++*launches;
  }
  return H266_OK;
}

size_t sao_stats_bytes(int n_ctbs) { return (size_t)n_ctbs * 3 * sizeof(SaoStats); }

int launch_sao_decide(cudaStream_t st, const DPlane src[3], const DPlane rec[3], int bd, int log2, int w_ctbs,
                      int h_ctbs, bool luma_on, bool chroma_on, void *d_stats, uint32_t *d_err,
                      h266_sao_ctb_params *d_out, uint64_t *launches) {
  const int n = w_ctbs * h_ctbs;
  if (n <= 0) return H266_OK;
  SaoEncArgs a{};
  for (int i = 0; i < 3; ++i) {
    a.src[i] = src[i];
    a.rec[i] = rec[i];
  }
  a.bd = bd;
  a.log2 = log2;
  a.w_ctbs = w_ctbs;
  a.h_ctbs = h_ctbs;
  a.luma_on = luma_on;
  a.chroma_on = chroma_on;
  auto *stats = static_cast<SaoStats *>(d_stats);
  // the error word lies right before the statistics
  H266_CUDA(cudaMemsetAsync(d_err, 0, sizeof(uint32_t) + sao_stats_bytes(n), st));
  const int rows = slice_rows(1 << log2), slices = ((1 << log2) + rows - 1) / rows;
  if (bd > 14) k_sao_stats<true><<<dim3(n, 3, slices), kStatThreads, 0, st>>>(a, stats, d_err);
  else k_sao_stats<false><<<dim3(n, 3, slices), kStatThreads, 0, st>>>(a, stats, d_err);
  H266_CUDA(cudaGetLastError());
  k_sao_decide<<<n, 32, 0, st>>>(a, stats, d_err, d_out);
  H266_CUDA(cudaGetLastError());
  *launches += 2;
  return H266_OK;
}

}  // namespace h266
