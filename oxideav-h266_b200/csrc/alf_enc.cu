// Encoder chroma ALF / CC-ALF trials (src/alf_enc.rs:628-1138): every candidate
// filter of one chroma component evaluated per CTB, the per-CTB choice and its
// commit, in two launches.
//
// k_chroma_trials: one CTA per tile (32x32 chroma samples, 16x16 for CTBs of
// 32, never straddling a CTB) stages the component's window -- and the luma
// window for CC-ALF -- once and runs every candidate on it with the chain's
// packed filters (alf_tile.cuh), four samples a thread; only squared errors
// leave the CTA, added into the (CTB, candidate) table (column 0: the samples
// as they are), plus a copy of the tile for the commit to read its neighbours
// from.  k_chroma_commit: every tile picks its CTB's first minimum of {off,
// candidate 0, ...} (ctb_sse_chroma, src/alf_enc.rs:823-849) and filters once
// more with the winner, into the reconstruction.  18 us of kernels for four
// candidates of a 1080p 10-bit component; a whole chain pass, a candidate plane,
// an upload and an SSE pass per candidate took 20 us for each.
#include "alf_tile.cuh"

namespace h266 {
namespace {

using namespace tile;

template <int TW>
struct ChromaWin {
  static constexpr int NT = TW * TW / 4;              // threads: 4 samples each
  static constexpr int CW = TW + 8, CH = TW + 4;      // chroma [x - 4, x + 4) x [y - 2, y + 2)
  static constexpr int CP = CW + 4;                   // pitches keep 8-byte rows, spread over banks
  static constexpr int LW = 2 * TW + 8, LH = 2 * TW + 4;  // luma [2x - 4, 2x + 4) x [2y - 1, 2y + 3)
  static constexpr int LP = LW + 4;
  alignas(16) uint16_t c[CH * CP];
  alignas(16) uint16_t l[LH * LP];
};

// Rows [y0, y0 + H) x columns [x0, x0 + W) of P, clamped into [rx0, rx1) x
// [ry0, ry1), biased, into `dst`; returns the samples or'ed together.
template <int NT, int W, int H, int PITCH>
__device__ __forceinline__ uint32_t stage_window(uint16_t *dst, const DPlane &P, int x0, int y0, int rx0, int ry0,
                                                 int rx1, int ry1) {
  uint32_t seen = 0;
  for (int i = threadIdx.x; i < W * H; i += NT) {
    const int r = i / W, c = i - r * W;
    const uint16_t v = P.s[(int64_t)clampd(y0 + r, ry0, ry1 - 1) * P.stride + clampd(x0 + c, rx0, rx1 - 1)];
    seen |= v;
    dst[r * PITCH + c] = v ^ 0x8000u;
  }
  return seen;
}

// The tile of this CTA: staged windows, geometry, and the four samples of this thread.
template <int TW>
struct ChromaTile {
  using Win = ChromaWin<TW>;
  int ctb_i, jr, gx, gy, n;  // n: samples of the run inside the plane (<= 0: none)
  int yline;
  bool lbb, big;
  const uint16_t *R0, *L0;
  int cur[4];

  // `from`: the plane the windows are staged from (the reconstruction, or its copy)
  __device__ __forceinline__ bool stage(const ChromaTrialArgs &a, const DPlane &from, Win &w) {
    const int tid = threadIdx.x;
    const int tx = (int)blockIdx.x % a.tiles_x, ty = (int)blockIdx.x / a.tiles_x;
    const int xc0 = tx * TW, yc0 = ty * TW, log2c = a.log2 - 1, ctb = 1 << a.log2;
    const int rx = xc0 >> log2c, ry = yc0 >> log2c;
    ctb_i = -1;
    if (rx >= a.w_ctbs || ry >= a.h_ctbs) return false;
    ctb_i = ry * a.w_ctbs + rx;
    const uint16_t *rect = a.ctbs[ctb_i].rect;
    uint32_t seen = stage_window<Win::NT, Win::CW, Win::CH, Win::CP>(
        w.c, from, xc0 - 4, yc0 - 2, rect[0] / 2, rect[1] / 2, min((rect[2] + 1) / 2, from.w),
        min((rect[3] + 1) / 2, from.h));
    if (a.cc)
      seen |= stage_window<Win::NT, Win::LW, Win::LH, Win::LP>(w.l, a.luma, 2 * xc0 - 4, 2 * yc0 - 1, rect[0], rect[1],
                                                               min((int)rect[2], a.pic_w), min((int)rect[3], a.pic_h));
    big = __syncthreads_or((seen & 0xC000u) != 0) != 0;
    const int j = tid / (TW / 4), i0 = (tid % (TW / 4)) * 4;
    gx = xc0 + i0;
    gy = yc0 + j;
    n = gy < a.rec.h ? min(4, a.rec.w - gx) : 0;
    const int y_ctb = ry << a.log2;
    jr = gy - (y_ctb >> 1);
    yline = 2 * jr;
    lbb = !(gy * 2 + ctb >= a.pic_h && (a.pic_h - y_ctb) <= ctb - 4);
    R0 = &w.c[(j + 2) * Win::CP + i0 + 4];
    L0 = &w.l[(2 * j + 1) * Win::LP + 2 * i0 + 4];
#pragma unroll
    for (int k = 0; k < 4; ++k) cur[k] = R0[k] ^ 0x8000;
    return true;
  }
  // Candidate `f` on the thread's samples.
  __device__ __forceinline__ void filter(const ChromaTrialArgs &a, int f, int v[4]) const {
    const int maxv = (1 << a.bd) - 1;
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = cur[k];
    if (a.cc) cc_alf_run<4>(L0, ChromaWin<TW>::LP, yline, 1 << a.log2, lbb, a.cc_coeff[f], a.bd, maxv, v);
    else chroma_alf_run<4>(R0, ChromaWin<TW>::CP, jr, 1 << (a.log2 - 1), a.packed[f], maxv, big, v);
  }
};

template <int TW>
__global__ void __launch_bounds__(ChromaWin<TW>::NT) k_chroma_trials(const __grid_constant__ ChromaTrialArgs a) {
  __shared__ ChromaWin<TW> w;
  ChromaTile<TW> t;
  if (!t.stage(a, a.rec, w)) return;  // uniform per CTA
  int org[4], n = min(t.n, a.src.w - t.gx);  // the SSE window is the CTB inside both planes
  if (t.gy >= a.src.h) n = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) org[k] = k < n ? (int)a.src.s[(int64_t)t.gy * a.src.stride + t.gx + k] : 0;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (k < t.n) a.copy.s[(int64_t)t.gy * a.copy.stride + t.gx + k] = (uint16_t)t.cur[k];
  unsigned long long *row = a.sse + (size_t)t.ctb_i * (a.n_cand + 1);
  for (int f = -1; f < a.n_cand; ++f) {
    int v[4];
    if (f < 0) {
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = t.cur[k];
    } else {
      t.filter(a, f, v);
    }
    unsigned long long e = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < n) {
        const int d = org[k] - v[k];
        e += (unsigned long long)((long long)d * d);
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
    if ((threadIdx.x & 31) == 0 && e) atomicAdd(row + 1 + f, e);
  }
}

template <int TW>
__global__ void __launch_bounds__(ChromaWin<TW>::NT) k_chroma_commit(const __grid_constant__ ChromaTrialArgs a) {
  __shared__ ChromaWin<TW> w;
  const int log2c = a.log2 - 1;
  const int xc0 = ((int)blockIdx.x % a.tiles_x) * TW, yc0 = ((int)blockIdx.x / a.tiles_x) * TW;
  const int rx = xc0 >> log2c, ry = yc0 >> log2c;
  if (rx >= a.w_ctbs || ry >= a.h_ctbs) return;
  const int i = ry * a.w_ctbs + rx;
  const unsigned long long *row = a.sse + (size_t)i * (a.n_cand + 1);
  unsigned long long best = row[0];
  int p = -1;
  for (int f = 0; f < a.n_cand; ++f)
    if (row[1 + f] < best) {
      best = row[1 + f];
      p = f;
    }
  if (threadIdx.x == 0 && xc0 == rx << log2c && yc0 == ry << log2c) a.pick[i] = (uint8_t)(p + 1);
  if (p < 0) return;  // uniform per CTA
  ChromaTile<TW> t;
  t.stage(a, a.copy, w);
  int v[4];
  t.filter(a, p, v);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (k < t.n) a.rec.s[(int64_t)t.gy * a.rec.stride + t.gx + k] = (uint16_t)v[k];
}

template <int TW>
int launch_tiles(cudaStream_t st, ChromaTrialArgs a, uint64_t *launches) {
  a.tiles_x = (a.rec.w + TW - 1) / TW;
  const unsigned n = (unsigned)(a.tiles_x * ((a.rec.h + TW - 1) / TW));
  k_chroma_trials<TW><<<n, ChromaWin<TW>::NT, 0, st>>>(a);
  H266_CUDA(cudaGetLastError());
  k_chroma_commit<TW><<<n, ChromaWin<TW>::NT, 0, st>>>(a);
  H266_CUDA(cudaGetLastError());
  *launches += 2;
  return H266_OK;
}

}  // namespace

int launch_chroma_trials(cudaStream_t st, const ChromaTrialArgs &a, uint64_t *launches) {
  return a.log2 == 5 ? launch_tiles<16>(st, a, launches) : launch_tiles<32>(st, a, launches);
}

}  // namespace h266
