// k_motion.cu -- block-matching motion estimation (kernel d) and the
// per-pixel vector field / warps / confidence upsampling that turn it into
// neighbour terms.
//
// Reference: EstimateMotion (hvd-core/src/engine/motion.cpp:397-488) with
// BoxBlur (:21-55, 391-395), Decimate (:59-78), BmPass (:105-260),
// RangeFromCentre (:286-298), CostAt (:309-315), MotionConfidence (:321-387);
// VectorsPerPixel / WarpByTiles / UpsampleConfidence[Fast]
// (engine/temporal.cpp:45-254).
//
// Bit-exact to the reference's float arithmetic: this file is compiled with
// FMA contraction off (--fmad=false), every float / double operation is
// issued in the reference's order, and each (pair, tile) visits the
// candidates in the reference's centre-out order with the same
// partial-distortion bail-out and strict-less update (a block per tile forms the
// per-row running sums of all candidates and a warp replays the visit from them;
// searches and tiles past the staged sizes take one thread per tile), so the
// selected vectors, sub-pel fits and confidences equal the reference's bit for
// bit.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "hvdg_common.cuh"
#include "k_motion.h"
#include "per_device.h"

namespace hvdg {

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// BoxBlur (motion.cpp:21-55): prefix sums c_k = c_(k-1) + s_(k-1) of a line in
// double, in order, and out_i = (c_min(i+r+1, n) - c_max(i-r, 0)) * norm. The
// order of the additions is the reference's, so a line is one serial chain of
// double additions (~10 cycles each, 4 us for a 760-sample row) and nothing
// else should be serial: a block takes a band of whole lines into shared
// memory as doubles (all its warps, coalesced), one lane per line runs the
// chain in place, kChain values ahead of their additions, and all warps form
// the window sums from the prefixes. Bands of 8 rows or 16 columns keep many
// blocks in flight. A band is read whole before it is written, so source and
// destination may be the same plane. Against a warp that staged, chained and
// windowed 32 rows in turn (and a thread per column), a PAL pair: rows 86 -> 16
// us, columns 55 -> 10 us.
constexpr int kBoxThreads = 256;
constexpr int kRowBand = 8;
constexpr int kColBand = 16;
constexpr int kChain = 16;

__host__ __device__ constexpr int row_stride(int n) { return (n + 1) | 1; }
constexpr size_t kBoxSmem = 200 << 10;

// c[ss], c[2 ss], ... c[n ss] <- their prefix sums; c[0] <- 0.
__device__ __forceinline__ void chain_line(double* c, int ss, int n) {
  double acc = 0.0;
  c[0] = 0.0;
  int k = 1;
  for (; k + kChain <= n + 1; k += kChain) {
    double v[kChain];
#pragma unroll
    for (int j = 0; j < kChain; ++j) v[j] = c[(k + j) * ss];
#pragma unroll
    for (int j = 0; j < kChain; ++j) {
      acc = acc + v[j];
      c[(k + j) * ss] = acc;
    }
  }
  for (; k <= n; ++k) {
    acc = acc + c[k * ss];
    c[k * ss] = acc;
  }
}

// `rows` (<= kRowBand) rows of n samples.
__device__ __forceinline__ void box_rows(const float* s, float* d, int64_t pitch, int rows,
                                         int n, int r, double norm) {
  extern __shared__ double box_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int stride = row_stride(n);
  double* pre = box_smem + warp * stride;
  if (warp < rows) {
    const float* row = s + (int64_t)warp * pitch;
#pragma unroll 8
    for (int x = lane; x < n; x += 32) pre[x + 1] = (double)row[x];
  }
  __syncthreads();
  if (threadIdx.x < rows) chain_line(box_smem + threadIdx.x * stride, 1, n);
  __syncthreads();
  if (warp < rows) {
    float* row = d + (int64_t)warp * pitch;
#pragma unroll 4
    for (int i = lane; i < n; i += 32) {
      const double hi = pre[i + r + 1 < n ? i + r + 1 : n], lo = pre[i - r > 0 ? i - r : 0];
      row[i] = (float)((hi - lo) * norm);
    }
  }
}

// `cols` (<= kColBand) columns of n samples.
__device__ __forceinline__ void box_cols(const float* s, float* d, int64_t pitch, int band,
                                         int cols, int n, int r, double norm) {
  extern __shared__ double box_smem[];
  const int x = threadIdx.x % band, y0 = threadIdx.x / band, step = kBoxThreads / band;
  if (x < cols) {
#pragma unroll 8
    for (int y = y0; y < n; y += step)
      box_smem[(y + 1) * band + x] = (double)s[(int64_t)y * pitch + x];
  }
  __syncthreads();
  if (threadIdx.x < cols) chain_line(box_smem + threadIdx.x, band, n);
  __syncthreads();
  if (x < cols) {
#pragma unroll 4
    for (int y = y0; y < n; y += step) {
      const double hi = box_smem[(y + r + 1 < n ? y + r + 1 : n) * band + x];
      const double lo = box_smem[(y - r > 0 ? y - r : 0) * band + x];
      d[(int64_t)y * pitch + x] = (float)((hi - lo) * norm);
    }
  }
}

// A line too long for shared memory (more than ~25,000 samples): one thread,
// the last 32 prefixes in a ring (2 r + 1 <= 31). Not in place.
__device__ void box_line_long(const float* s, float* d, int64_t ss, int n, int r, double norm) {
  double ring[32], c = 0.0;
  ring[0] = 0.0;
  for (int k = 1; k <= n + r; ++k) {
    if (k <= n) {
      c = c + (double)s[(int64_t)(k - 1) * ss];
      ring[k & 31] = c;
    }
    const int i = k - r - 1;
    if (i >= 0) d[(int64_t)i * ss] = (float)((c - (i - r > 0 ? ring[(i - r) & 31] : 0.0)) * norm);
  }
}

// Lines of a band: as many as fit, 0 when not even one does.
inline int row_band(int n) {
  return (int)std::min<size_t>(kRowBand, kBoxSmem / (sizeof(double) * row_stride(n)));
}
inline int col_band(int n) {
  const size_t line = sizeof(double) * (n + 1);
  return kBoxSmem / line >= kColBand ? kColBand : kBoxSmem / line >= 4 ? 4 : kBoxSmem / line >= 1;
}

// Vertical pass: one block per (field, 16-column band).
__global__ void __launch_bounds__(kBoxThreads) k_blur_v(const MeField* __restrict__ mf, int nf,
                                                        const float* __restrict__ src, float* dst,
                                                        int r, int src_sel, int band) {
  const int f = blockIdx.y;
  if (f >= nf) return;
  const MeField m = mf[f];
  const double norm = (double)(1.0f / (float)(2 * r + 1));
  const float* s = src + (src_sel == 0 ? m.y_off : m.b_off);
  if (band == 0) {
    const int x = blockIdx.x * kBoxThreads + threadIdx.x;
    if (x < m.w) box_line_long(s + x, dst + m.t_off + x, m.pitch, m.h, r, norm);
    return;
  }
  const int x0 = blockIdx.x * band;
  if (x0 >= m.w) return;
  box_cols(s + x0, dst + m.t_off + x0, m.pitch, band, min(band, m.w - x0), m.h, r, norm);
}

// Horizontal pass: one block per (field, 8-row band).
__global__ void __launch_bounds__(kBoxThreads) k_blur_h(const MeField* __restrict__ mf, int nf,
                                                        const float* __restrict__ src, float* dst,
                                                        int r, int band) {
  const int f = blockIdx.y;
  if (f >= nf) return;
  const MeField m = mf[f];
  const double norm = (double)(1.0f / (float)(2 * r + 1));
  const float* s = src + m.t_off;
  float* d = dst + m.b_off;
  if (band == 0) {
    const int y = blockIdx.x * kBoxThreads + threadIdx.x;
    if (y < m.h)
      box_line_long(s + (int64_t)y * m.pitch, d + (int64_t)y * m.pitch, 1, m.w, r, norm);
    return;
  }
  const int y0 = blockIdx.x * band;
  if (y0 >= m.h) return;
  box_rows(s + (int64_t)y0 * m.pitch, d + (int64_t)y0 * m.pitch, m.pitch, min(band, m.h - y0), m.w,
           r, norm);
}

// ---- Decimate (motion.cpp:59-78): 4 x 4 block mean ---------------------------
__global__ void k_decimate(const MeField* __restrict__ mf, int nf, const float* __restrict__ blur,
                           float* __restrict__ dec) {
  const int f = blockIdx.y;
  if (f >= nf) return;
  const MeField m = mf[f];
  const int hd = m.h / 4, wd = m.w / 4;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= hd * wd) return;
  const int y = i / wd, x = i % wd;
  const float* b = blur + m.b_off;
  float acc = 0.0f;
  for (int dy = 0; dy < 4; ++dy)
    for (int dx = 0; dx < 4; ++dx) acc += b[(int64_t)(y * 4 + dy) * m.pitch + x * 4 + dx];
  dec[m.d_off + (int64_t)y * m.dpitch + x] = acc * (1.0f / 16.0f);
}

// Sum of squared differences over one tile, rows in order, with the
// reference's per-row partial-distortion bail-out (acc >= kill).
__device__ __forceinline__ float tile_ssd(const float* A, const float* B, int pitch, int h, int w,
                                          int ty0, int ty1, int tx0, int tx1, int sy, int sx,
                                          float kill) {
  float acc = 0.0f;
  for (int y = ty0; y < ty1; ++y) {
    const float* arow = A + (int64_t)y * pitch;
    const float* brow = B + (int64_t)clampi(y - sy, 0, h - 1) * pitch;
    for (int x = tx0; x < tx1; ++x) {
      const float diff = arow[x] - brow[clampi(x - sx, 0, w - 1)];
      acc += diff * diff;
    }
    if (acc >= kill) break;
  }
  return acc;
}

// centre-out candidate order (RangeFromCentre, motion.cpp:286-298) for a
// symmetric range [-r, r]: 0, -1, 1, -2, 2, ...
__device__ __forceinline__ int centre_out(int i) { return (i & 1) ? -((i + 1) >> 1) : (i >> 1); }
__device__ __forceinline__ int centre_out_index(int d) {
  return d == 0 ? 0 : (d > 0 ? 2 * d : -2 * d - 1);
}

// ---- coarse absolute pass on the 4x-decimated planes (motion.cpp:406-413) --
__global__ void k_me_coarse(const MeField* __restrict__ mf, const MePair* __restrict__ pairs,
                            int npairs, const float* __restrict__ dec, MeArgs a,
                            float* __restrict__ cdy, float* __restrict__ cdx) {
  const int p = blockIdx.y;
  if (p >= npairs) return;
  const MePair pr = pairs[p];
  const MeField mc = mf[pr.cur], mr = mf[pr.ref];
  const int hd = mc.h / 4, wd = mc.w / 4;
  const int ct = a.tile / 4 > 4 ? a.tile / 4 : 4;
  const int th = (hd + ct - 1) / ct, tw = (wd + ct - 1) / ct;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= th * tw) return;
  const int ty = t / tw, tx = t % tw;
  const int cs = (a.search + 3) / 4 > 1 ? (a.search + 3) / 4 : 1;
  const float* A = dec + mc.d_off;
  const float* B = dec + mr.d_off;
  const int y0 = ty * ct, y1 = min((ty + 1) * ct, hd);
  const int x0 = tx * ct, x1 = min((tx + 1) * ct, wd);
  float best = __int_as_float(0x7f800000);
  float bdy = 0.0f, bdx = 0.0f;
  const int n = 2 * cs + 1;
  for (int i = 0; i < n; ++i) {
    const int dy = centre_out(i);
    for (int j = 0; j < n; ++j) {
      const int dx = centre_out(j);
      const float bias = 1.0f + 0.02f * (float)(abs(dy) + abs(dx));
      const float inv_bias = 1.0f / bias;
      const bool exact = dy == 0 && dx == 0;  // cost0 needs the full sum
      const float kill = exact ? __int_as_float(0x7f800000) : best * inv_bias;
      const float se = tile_ssd(A, B, mc.dpitch, hd, wd, y0, y1, x0, x1, dy, dx, kill);
      const float cost = se * bias;
      if (cost < best) {
        best = cost;
        bdy = (float)dy;
        bdx = (float)dx;
      }
    }
  }
  cdy[a.coarse_off * p + t] = bdy;
  cdx[a.coarse_off * p + t] = bdx;
}

// Candidates, tile rows and reach of k_me_coarse_tile; larger coarse tiles or
// searches keep a thread per tile (k_me_coarse).
constexpr int kCoarseCands = 128;
constexpr int kCoarseRows = 16;
constexpr int kCoarseReach = 5;  // (2 * 5 + 1)^2 <= kCoarseCands

// The coarse search of one tile by a block: the tile and the window its
// candidates reach are staged in shared memory (clamped coordinates resolved
// there), a thread runs one candidate's sum in the reference's order, keeping
// the running sum after every row, and a warp replays the reference's visit
// from those sums: kill = best * (1 / bias), the first row whose running sum
// reaches it (a ballot over the rows) ends the candidate with that sum,
// strict-less update. Every cost and decision is the per-thread kernel's. A
// warp per tile reading global memory took 53 us on a PAL pair (latency of
// three rounds of 64 dependent loads), this takes 22.
__global__ void __launch_bounds__(kCoarseCands) k_me_coarse_tile(
    const MeField* __restrict__ mf, const MePair* __restrict__ pairs, int npairs,
    const float* __restrict__ dec, MeArgs a, float* __restrict__ cdy, float* __restrict__ cdx) {
  constexpr int kWin = kCoarseRows + 2 * kCoarseReach;
  __shared__ float sa[kCoarseRows * kCoarseRows], sb[kWin * (kWin + 1)];
  __shared__ float part[kCoarseCands * (kCoarseRows + 1)];
  const int p = blockIdx.y;
  const MePair pr = pairs[p];
  const MeField mc = mf[pr.cur], mr = mf[pr.ref];
  const int hd = mc.h / 4, wd = mc.w / 4;
  const int ct = a.tile / 4 > 4 ? a.tile / 4 : 4;
  const int th = (hd + ct - 1) / ct, tw = (wd + ct - 1) / ct;
  const int t = blockIdx.x;
  if (t >= th * tw) return;
  const int ty = t / tw, tx = t % tw;
  const int cs = (a.search + 3) / 4 > 1 ? (a.search + 3) / 4 : 1;
  const int n = 2 * cs + 1, ncand = n * n;
  const float* A = dec + mc.d_off;
  const float* B = dec + mr.d_off;
  const int y0 = ty * ct, x0 = tx * ct;
  const int rows = min(ct, hd - y0), cols = min(ct, wd - x0);
  const int ww = cols + 2 * cs;
  for (int i = threadIdx.x; i < rows * cols; i += kCoarseCands)
    sa[i] = A[(int64_t)(y0 + i / cols) * mc.dpitch + x0 + i % cols];
  for (int i = threadIdx.x; i < (rows + 2 * cs) * ww; i += kCoarseCands)
    sb[i] = B[(int64_t)clampi(y0 - cs + i / ww, 0, hd - 1) * mc.dpitch +
              clampi(x0 - cs + i % ww, 0, wd - 1)];
  __syncthreads();
  const int c = threadIdx.x;
  if (c < ncand) {
    const float* b = sb + (cs - centre_out(c / n)) * ww + cs - centre_out(c % n);
    float acc = 0.0f;
    for (int y = 0; y < rows; ++y) {
#pragma unroll 4
      for (int x = 0; x < cols; ++x) {
        const float diff = sa[y * cols + x] - b[y * ww + x];
        acc += diff * diff;
      }
      part[c * (kCoarseRows + 1) + y] = acc;
    }
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  const float inf = __int_as_float(0x7f800000);
  float best = inf, bdy = 0.0f, bdx = 0.0f;
  for (int k = 0; k < ncand; ++k) {
    const int dy = centre_out(k / n), dx = centre_out(k % n);
    const float bias = 1.0f + 0.02f * (float)(abs(dy) + abs(dx));
    const float inv_bias = 1.0f / bias;
    const float kill = dy == 0 && dx == 0 ? inf : best * inv_bias;
    const float* pc = part + k * (kCoarseRows + 1);
    const unsigned hit = __ballot_sync(0xffffffffu, lane < rows && pc[lane] >= kill);
    const float se = pc[hit ? __ffs(hit) - 1 : rows - 1];
    const float cost = se * bias;
    if (cost < best) {
      best = cost;
      bdy = (float)dy;
      bdx = (float)dx;
    }
  }
  if (lane == 0) {
    cdy[a.coarse_off * p + t] = bdy;
    cdx[a.coarse_off * p + t] = bdx;
  }
}

// ---- full-res refinement, sub-pel fit, zero / margin rule (motion.cpp:415-473)
__global__ void k_me_refine(const MeField* __restrict__ mf, const MePair* __restrict__ pairs,
                            int npairs, const float* __restrict__ blur, MeArgs a,
                            const float* __restrict__ cdy, const float* __restrict__ cdx,
                            float* __restrict__ out_mdy, float* __restrict__ out_mdx,
                            float* __restrict__ out_sdy, float* __restrict__ out_sdx,
                            float* __restrict__ out_best) {
  const int p = blockIdx.y;
  if (p >= npairs) return;
  const MePair pr = pairs[p];
  const MeField mc = mf[pr.cur], mr = mf[pr.ref];
  const int h = mc.h, w = mc.w, tile = a.tile;
  const int th = (h + tile - 1) / tile, tw = (w + tile - 1) / tile;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= th * tw) return;
  const int ty = t / tw, tx = t % tw;
  const int hd = h / 4, wd = w / 4;
  const int ct = tile / 4 > 4 ? tile / 4 : 4;
  const int hh = (hd + ct - 1) / ct, ww = (wd + ct - 1) / ct;
  const int gy = min((ty * hh) / th, hh - 1), gx = min((tx * ww) / tw, ww - 1);
  const float base_dy = cdy[a.coarse_off * p + gy * ww + gx] * 4.0f;
  const float base_dx = cdx[a.coarse_off * p + gy * ww + gx] * 4.0f;
  const float* A = blur + mc.b_off;
  const float* B = blur + mr.b_off;
  const int y0 = ty * tile, y1 = min((ty + 1) * tile, h);
  const int x0 = tx * tile, x1 = min((tx + 1) * tile, w);
  const float inf = __int_as_float(0x7f800000);
  // refine: relative candidates RangeFromCentre(-3, 3)^2, no cost0
  const int rby = (int)lroundf(base_dy), rbx = (int)lroundf(base_dx);
  float best = inf, mdy = 0.0f, mdx = 0.0f;
  for (int i = 0; i < 7; ++i) {
    const int dy = centre_out(i);
    for (int j = 0; j < 7; ++j) {
      const int dx = centre_out(j);
      const float bias = 1.0f + 0.02f * (float)(abs(dy) + abs(dx));
      const float inv_bias = 1.0f / bias;
      const float kill = best * inv_bias;
      const float se = tile_ssd(A, B, mc.pitch, h, w, y0, y1, x0, x1, rby + dy, rbx + dx, kill);
      const float cost = se * bias;
      if (cost < best) {
        best = cost;
        mdy = base_dy + (float)dy;
        mdx = base_dx + (float)dx;
      }
    }
  }
  // CostAt at (+-1, 0), (0, +-1): single relative candidate, full sum, bias 1
  const int iy = (int)lroundf(mdy), ix = (int)lroundf(mdx);
  const float cym = tile_ssd(A, B, mc.pitch, h, w, y0, y1, x0, x1,
                             (int)lroundf(mdy + -1.0f), ix, inf) * 1.0f;
  const float cyp = tile_ssd(A, B, mc.pitch, h, w, y0, y1, x0, x1,
                             (int)lroundf(mdy + 1.0f), ix, inf) * 1.0f;
  const float cxm = tile_ssd(A, B, mc.pitch, h, w, y0, y1, x0, x1, iy,
                             (int)lroundf(mdx + -1.0f), inf) * 1.0f;
  const float cxp = tile_ssd(A, B, mc.pitch, h, w, y0, y1, x0, x1, iy,
                             (int)lroundf(mdx + 1.0f), inf) * 1.0f;
  auto parabolic = [](float cm, float c0, float cp) {
    const float den = cm - 2.0f * c0 + cp;
    float sub = 0.0f;
    if (den > 1e-9f) sub = 0.5f * (cm - cp) / fmaxf(den, 1e-9f);
    return fminf(fmaxf(sub, -0.5f), 0.5f);
  };
  float sdy = parabolic(cym, best, cyp);
  float sdx = parabolic(cxm, best, cxp);
  // explicit zero-motion evaluation + "prefer zero" margin rule
  const float cost0 = tile_ssd(A, B, mc.pitch, h, w, y0, y1, x0, x1, 0, 0, inf);
  const float best0 = cost0 * 1.0f;
  if (best0 < best) {
    mdy = 0.0f;
    mdx = 0.0f;
    best = best0;
  }
  if (best > 0.85f * cost0) {
    mdy = 0.0f;
    mdx = 0.0f;
    best = cost0;
    sdy = 0.0f;
    sdx = 0.0f;
  }
  const int o = a.tiles_off * p + t;
  out_mdy[o] = mdy;
  out_mdx[o] = mdx;
  out_sdy[o] = sdy;
  out_sdx[o] = sdx;
  out_best[o] = best;
}

// The full-resolution refinement of one tile by a block of three warps: the
// tile, the reference window that the +-3 candidates and their +-1 neighbours
// reach and the unshifted reference tile are staged in shared memory. Thread
// c runs the sum of one of the 81 shifts within +-4 of the base, thread 81
// the zero-motion one, each in the reference's order; the inner 49 keep their
// running sum after every row. The window's pitch is 9 modulo 32, so the
// shifts of a warp fall into different banks. A warp then replays the
// reference's visit as the coarse search does, and takes the four CostAt sums
// and the zero-motion cost from the full sums -- the same sums in the same
// order, so every cost, decision and vector is the per-thread kernel's. What
// bounds it is one chained addition per pixel of the tile (4 cycles, 2 us for
// 32 x 32); a warp per tile with its operands in global memory and the five
// CostAt sums after the candidates took 186 us on a PAL pair, this takes 31.
constexpr int kRefineCands = 49;  // RangeFromCentre(-3, 3)^2
constexpr int kRefineTile = 64;
constexpr int kRefineThreads = 96;

__host__ __device__ constexpr int refine_pitch(int cols) {
  return (cols + 8 + 31 - 9) / 32 * 32 + 9;  // >= cols + 8, 9 modulo 32
}
inline size_t refine_smem(int tile) {
  return sizeof(float) * (tile * tile + (size_t)(2 * tile + 8) * refine_pitch(tile) +
                          kRefineCands * (tile + 1) + 82);
}

__global__ void __launch_bounds__(kRefineThreads) k_me_refine_tile(
    const MeField* __restrict__ mf, const MePair* __restrict__ pairs, int npairs,
    const float* __restrict__ blur, MeArgs a, const float* __restrict__ cdy,
    const float* __restrict__ cdx, float* __restrict__ out_mdy, float* __restrict__ out_mdx,
    float* __restrict__ out_sdy, float* __restrict__ out_sdx, float* __restrict__ out_best) {
  extern __shared__ float me_part[];
  const int lane = threadIdx.x & 31;
  const int p = blockIdx.y;
  const MePair pr = pairs[p];
  const MeField mc = mf[pr.cur], mr = mf[pr.ref];
  const int h = mc.h, w = mc.w, tile = a.tile;
  const int th = (h + tile - 1) / tile, tw = (w + tile - 1) / tile;
  const int t = blockIdx.x;
  if (t >= th * tw) return;
  const int ty = t / tw, tx = t % tw;
  const int hd = h / 4, wd = w / 4;
  const int ct = tile / 4 > 4 ? tile / 4 : 4;
  const int hh = (hd + ct - 1) / ct, ww = (wd + ct - 1) / ct;
  const int gy = min((ty * hh) / th, hh - 1), gx = min((tx * ww) / tw, ww - 1);
  const float base_dy = cdy[a.coarse_off * p + gy * ww + gx] * 4.0f;
  const float base_dx = cdx[a.coarse_off * p + gy * ww + gx] * 4.0f;
  const float* A = blur + mc.b_off;
  const float* B = blur + mr.b_off;
  const int y0 = ty * tile, y1 = min((ty + 1) * tile, h);
  const int x0 = tx * tile, x1 = min((tx + 1) * tile, w);
  const int rows = y1 - y0, cols = x1 - x0;
  const int pitch = refine_pitch(tile);
  float* sa = me_part;                      // rows x cols
  float* sb = sa + tile * tile;             // (rows + 8) x pitch
  float* s0 = sb + (tile + 8) * pitch;      // rows x pitch, unshifted
  float* part = s0 + tile * pitch;          // kRefineCands x (tile + 1), in visit order
  float* full = part + kRefineCands * (tile + 1);  // 81 shifts, then zero motion
  const float inf = __int_as_float(0x7f800000);
  const int rby = (int)lroundf(base_dy), rbx = (int)lroundf(base_dx);
  for (int i = threadIdx.x; i < rows * cols; i += kRefineThreads) {
    const int y = i / cols, x = i - y * cols;
    sa[i] = A[(int64_t)(y0 + y) * mc.pitch + x0 + x];
    s0[y * pitch + x] = B[(int64_t)(y0 + y) * mc.pitch + x0 + x];
  }
  for (int i = threadIdx.x; i < (rows + 8) * (cols + 8); i += kRefineThreads) {
    const int y = i / (cols + 8), x = i - y * (cols + 8);
    sb[y * pitch + x] = B[(int64_t)clampi(y0 - rby - 4 + y, 0, h - 1) * mc.pitch +
                          clampi(x0 - rbx - 4 + x, 0, w - 1)];
  }
  __syncthreads();
  const int c = threadIdx.x;
  if (c < 82) {
    const int cy = c / 9 - 4, cx = c % 9 - 4;  // shift of thread c < 81
    const float* b = c < 81 ? sb + (4 - cy) * pitch + 4 - cx : s0;
    const bool inner = c < 81 && abs(cy) <= 3 && abs(cx) <= 3;
    float* pc = part + (inner ? centre_out_index(cy) * 7 + centre_out_index(cx) : 0) * (tile + 1);
    float acc = 0.0f;
    for (int y = 0; y < rows; ++y) {
      const float* ar = sa + y * cols;
      const float* br = b + y * pitch;
#pragma unroll 8
      for (int x = 0; x < cols; ++x) {
        const float diff = ar[x] - br[x];
        acc += diff * diff;
      }
      if (inner) pc[y] = acc;
    }
    full[c] = acc;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  float best = inf, mdy = 0.0f, mdx = 0.0f;
  int bdy = 0, bdx = 0;
  for (int k = 0; k < kRefineCands; ++k) {
    const int dy = centre_out(k / 7), dx = centre_out(k % 7);
    const float bias = 1.0f + 0.02f * (float)(abs(dy) + abs(dx));
    const float inv_bias = 1.0f / bias;
    const float kill = best * inv_bias;
    const float* pc = part + k * (tile + 1);
    float se = pc[rows - 1];
    for (int r0 = 0; r0 < rows; r0 += 32) {
      const unsigned hit =
          __ballot_sync(0xffffffffu, r0 + lane < rows && pc[r0 + lane] >= kill);
      if (hit) {
        se = pc[r0 + __ffs(hit) - 1];
        break;
      }
    }
    const float cost = se * bias;
    if (cost < best) {
      best = cost;
      mdy = base_dy + (float)dy;
      mdx = base_dx + (float)dx;
      bdy = dy;
      bdx = dx;
    }
  }
  // CostAt at (+-1, 0), (0, +-1) and the zero-motion cost: full sums. Where no
  // cost is below infinity (non-finite planes) the visit keeps no candidate and
  // CostAt looks around zero motion.
  const float cost0 = full[81] * 1.0f;
  float cym, cyp, cxm, cxp;
  if (best < inf) {
    const float* fc = full + (bdy + 4) * 9 + bdx + 4;
    cym = fc[-9] * 1.0f;
    cyp = fc[9] * 1.0f;
    cxm = fc[-1] * 1.0f;
    cxp = fc[1] * 1.0f;
  } else {
    cym = tile_ssd(A, B, mc.pitch, h, w, y0, y1, x0, x1, -1, 0, inf) * 1.0f;
    cyp = tile_ssd(A, B, mc.pitch, h, w, y0, y1, x0, x1, 1, 0, inf) * 1.0f;
    cxm = tile_ssd(A, B, mc.pitch, h, w, y0, y1, x0, x1, 0, -1, inf) * 1.0f;
    cxp = tile_ssd(A, B, mc.pitch, h, w, y0, y1, x0, x1, 0, 1, inf) * 1.0f;
  }
  if (lane != 0) return;
  auto parabolic = [](float cm, float c0, float cp) {
    const float den = cm - 2.0f * c0 + cp;
    float sub = 0.0f;
    if (den > 1e-9f) sub = 0.5f * (cm - cp) / fmaxf(den, 1e-9f);
    return fminf(fmaxf(sub, -0.5f), 0.5f);
  };
  float sdy = parabolic(cym, best, cyp);
  float sdx = parabolic(cxm, best, cxp);
  const float best0 = cost0 * 1.0f;
  if (best0 < best) {
    mdy = 0.0f;
    mdx = 0.0f;
    best = best0;
  }
  if (best > 0.85f * cost0) {
    mdy = 0.0f;
    mdx = 0.0f;
    best = cost0;
    sdy = 0.0f;
    sdx = 0.0f;
  }
  const int o = a.tiles_off * p + t;
  out_mdy[o] = mdy;
  out_mdx[o] = mdx;
  out_sdy[o] = sdy;
  out_sdx[o] = sdx;
  out_best[o] = best;
}

// ---- MotionConfidence (motion.cpp:321-387) + final vectors ------------------
// (1) A tile's mean, variance and residual ratio: a warp per tile brings the
// tile to shared memory kConfChunk pixels at a time (row by row, coalesced)
// and one lane adds them in the reference's order; conf0 and the ratio go to
// out_conf / out_dy for (2). The two chained additions per pixel bound it (3
// us for 32 x 32); one thread per tile of one block per pair, with the medians
// behind it, took 187 us on a PAL pair, (1) takes 14 and (2) 12.
constexpr int kConfChunk = 1024;
constexpr int kConfWarps = 8;
__global__ void __launch_bounds__(32 * kConfWarps) k_me_tile_stats(
    const MeField* __restrict__ mf, const MePair* __restrict__ pairs,
    const float* __restrict__ blur, MeArgs a, const float* __restrict__ bestv,
    float* __restrict__ out_ratio, float* __restrict__ out_conf0) {
  __shared__ float px[kConfWarps][kConfChunk];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p = blockIdx.y;
  const MeField mc = mf[pairs[p].cur];
  const int h = mc.h, w = mc.w, tile = a.tile;
  const int th = (h + tile - 1) / tile, tw = (w + tile - 1) / tile;
  const int t = blockIdx.x * kConfWarps + warp;
  if (t >= th * tw) return;  // the whole warp; only warp-level sync below
  // rows/cols mapped by min(y / tile, th - 1)
  const int y0 = t / tw * tile, x0 = t % tw * tile;
  const int cols = min(tile, w - x0), n = min(tile, h - y0) * cols;
  const float* A = blur + mc.b_off + (int64_t)y0 * mc.pitch + x0;
  float* v = px[warp];
  float sum = 0.0f, sum2 = 0.0f;
  for (int i0 = 0; i0 < n; i0 += kConfChunk) {
    const int m = min(kConfChunk, n - i0);
#pragma unroll 8
    for (int i = lane; i < m; i += 32)
      v[i] = A[(int64_t)((i0 + i) / cols) * mc.pitch + (i0 + i) % cols];
    __syncwarp();
    if (lane == 0) {
#pragma unroll 16
      for (int i = 0; i < m; ++i) {
        const float x = v[i];
        sum += x;
        sum2 += x * x;
      }
    }
    __syncwarp();
  }
  if (lane != 0) return;
  // the reference counts pixels in float: exact below 2^24, and a tile has fewer
  const float np = (float)n;
  const float norm = 1.0f / fmaxf(1.0f, np);
  const float tmean = sum * norm;
  const float tvar = sum2 * norm - tmean * tmean;
  const int o = a.tiles_off * p + t;
  const float best = bestv[o];
  const float energy = (tvar + 1.0f) * fmaxf(1.0f, np);
  out_conf0[o] = fminf(fmaxf(1.0f - best / energy, 0.0f), 1.0f);
  out_ratio[o] = best / fmaxf(1.0f, np);
}

// (2) The median ratio and the final confidences and vectors, one block per
// pair; the two middle ratios by counting ranks (a few hundred tiles), by
// radix selection past kRankTiles.
constexpr int kRankTiles = 1024;
__global__ void __launch_bounds__(256) k_me_confidence(const MePair* __restrict__ pairs, MeArgs a,
                                                       int nt, const float* __restrict__ mdy,
                                                       const float* __restrict__ mdx,
                                                       const float* __restrict__ sdy,
                                                       const float* __restrict__ sdx,
                                                       float* __restrict__ out_dy,
                                                       float* __restrict__ out_dx,
                                                       float* __restrict__ out_conf) {
  extern __shared__ float ratios[];  // nt
  __shared__ unsigned hist[256];
  __shared__ unsigned bc[2];
  __shared__ float mid[2];
  const int o = a.tiles_off * blockIdx.x;
  for (int t = threadIdx.x; t < nt; t += blockDim.x) ratios[t] = out_dy[o + t];
  __syncthreads();
  // Median (motion.cpp:80-91): nth_element at n/2, averaged with the (n/2-1)-th for even n
  const int k = nt / 2;
  float med, lo;
  if (nt <= kRankTiles) {
    for (int t = threadIdx.x; t < nt; t += blockDim.x) {
      const uint32_t key = float_key(ratios[t]);
      int less = 0, eq = 0;
      for (int u = 0; u < nt; ++u) {
        const uint32_t ku = float_key(ratios[u]);
        less += ku < key;
        eq += ku == key;
      }
      if (less <= k && k < less + eq) mid[0] = ratios[t];
      if (less <= k - 1 && k - 1 < less + eq) mid[1] = ratios[t];
    }
    __syncthreads();
    med = mid[0];
    lo = nt % 2 == 0 ? mid[1] : 0.0f;
  } else {
    med = block_select_kth(ratios, nt, k, hist, bc);
    lo = nt % 2 == 0 ? block_select_kth(ratios, nt, k - 1, hist, bc) : 0.0f;
  }
  if (nt % 2 == 0) med = 0.5f * (med + lo);
  for (int t = threadIdx.x; t < nt; t += blockDim.x) {
    const float excess = fmaxf(0.0f, ratios[t] - med);
    float c = out_conf[o + t];
    c *= (med + 1.0f) / (med + 1.0f + excess);
    c *= 6.0f / (6.0f + med);
    out_conf[o + t] = c;
    out_dy[o + t] = mdy[o + t] + sdy[o + t];
    out_dx[o + t] = mdx[o + t] + sdx[o + t];
  }
}

static void field_blur(const MeField* d_fields, int nf, int max_h, int max_w, const MeBuffers& b,
                       cudaStream_t st);
static PerDeviceOnce refine_once;

void launch_motion_blur(const MeField* d_fields, int nf, int max_h, int max_w, const MeBuffers& b,
                        cudaStream_t st) {
  if (nf <= 0) return;
  field_blur(d_fields, nf, max_h, max_w, b, st);
}

void launch_motion(const MeField* d_fields, int nf, int max_h, int max_w, const MePair* d_pairs,
                   int npairs, const MeArgs& a, const MeBuffers& b, cudaStream_t st) {
  if (nf <= 0 || npairs <= 0) return;
  // blur every field's luma (A = blur(y_cur), B = blur(y_ref) share per field)
  field_blur(d_fields, nf, max_h, max_w, b, st);
  k_decimate<<<dim3(((max_h / 4) * (max_w / 4) + 255) / 256, nf), 256, 0, st>>>(d_fields, nf, b.blur, b.dec);
  const int ct = a.tile / 4 > 4 ? a.tile / 4 : 4;
  const int cth = ((max_h / 4) + ct - 1) / ct, ctw = ((max_w / 4) + ct - 1) / ct;
  const int cn = 2 * ((a.search + 3) / 4 > 1 ? (a.search + 3) / 4 : 1) + 1;
  if (cn * cn <= kCoarseCands && ct <= kCoarseRows) {
    k_me_coarse_tile<<<dim3(cth * ctw, npairs), kCoarseCands, 0, st>>>(
        d_fields, d_pairs, npairs, b.dec, a, b.cdy, b.cdx);
  } else {
    k_me_coarse<<<dim3((cth * ctw + 63) / 64, npairs), 64, 0, st>>>(d_fields, d_pairs, npairs,
                                                                 b.dec, a, b.cdy, b.cdx);
  }
  const int th = (max_h + a.tile - 1) / a.tile, tw = (max_w + a.tile - 1) / a.tile;
  if (a.tile <= kRefineTile) {
    refine_once([] {
      cudaFuncSetAttribute(k_me_refine_tile, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)refine_smem(kRefineTile));
    });
    k_me_refine_tile<<<dim3(th * tw, npairs), kRefineThreads, refine_smem(a.tile), st>>>(
        d_fields, d_pairs, npairs, b.blur, a, b.cdy, b.cdx, b.mdy, b.mdx, b.sdy, b.sdx, b.best);
  } else {
    k_me_refine<<<dim3((th * tw + 63) / 64, npairs), 64, 0, st>>>(
        d_fields, d_pairs, npairs, b.blur, a, b.cdy, b.cdx, b.mdy, b.mdx, b.sdy, b.sdx, b.best);
  }
  launch_me_confidence(d_fields, d_pairs, npairs, max_h, max_w, a, b.blur, b.mdy, b.mdx, b.sdy,
                       b.sdx, b.best, b.dy, b.dx, b.conf, st);
}

// ---------------------------------------------------------------------------
// Integer-SAD motion mode (me_mode 1): exhaustive +-range search of
// block x block tiles on uint16-quantised, integer-box-blurred luma. The
// cost has no reference counterpart (the reference matches float SSD); the
// control structure follows EstimateMotion (motion.cpp:397-488) -- visit
// order RangeFromCentre (:286-298), strict-less update (:244), bias
// 1 + 0.02 (|dy| + |dx|), zero-motion margin 0.85 (:455-473), parabolic
// sub-pel (:437-452), MotionConfidence (:321-387) -- with every decision
// exact in integers: SAD_a (50 + L1_a) < SAD_b (50 + L1_b), and
// 20 best > 17 cost0 for the margin. A parallel argmin over the key
// (biased cost, visit index) selects the same candidate as the reference's
// sequential strict-less scan.
// ---------------------------------------------------------------------------
constexpr float kQuantZero = 16384.0f;   // 0 IRE
constexpr float kQuantScale = 348.16f;   // codes per IRE
constexpr int kSadMaxBlock = 32;
constexpr int kSadMaxRange = 22;         // (2 range + 1)^2 visit indices fit in 11 bits
// block, window and the window's integral image at the largest block and range
constexpr int kSadMaxWin = kSadMaxBlock + 2 * (kSadMaxRange + 1);
// block, window, integral image, then the packed copies (16-bit pairs) of
// the block's rows and of the window's rows at even and odd starts
__host__ __device__ constexpr int sad_smem_ints(int b, int ww) {
  return b * b + ww * ww + (ww + 1) * (ww + 1) + b * (b / 2) + 2 * ww * (ww / 2 + 1);
}
constexpr int kSadMaxSmem = sad_smem_ints(kSadMaxBlock, kSadMaxWin) * (int)sizeof(int);
constexpr int kSadThreads = 224;

int sad_max_block() { return kSadMaxBlock; }
int sad_max_range() { return kSadMaxRange; }

__device__ __forceinline__ int quant_luma(float y) {
  const float t = kQuantZero + kQuantScale * y;  // multiply, then add (no FMA in this unit)
  return (int)fminf(fmaxf(rintf(t), 0.0f), 65535.0f);
}

// The quantised luma's 5 x 5 box (zero outside the field), rounded: integer
// sums, so any order is exact. A block takes a 64 x 16 tile with its border
// into shared memory, sums columns, then rows. One pass over the plane in
// place of a running sum per column and then per row (two 760 x 242 planes:
// 354 -> 7 us).
constexpr int kQbX = 64, kQbY = 16;
__global__ void __launch_bounds__(256) k_sad_blur(const MeField* __restrict__ mf,
                                                  const float* __restrict__ luma,
                                                  int* __restrict__ qblur) {
  __shared__ int q[kQbY + 4][kQbX + 4];
  __shared__ int v[kQbY][kQbX + 4];
  const MeField m = mf[blockIdx.z];
  const int x0 = blockIdx.x * kQbX, y0 = blockIdx.y * kQbY;
  if (x0 >= m.w || y0 >= m.h) return;
  const float* Y = luma + m.y_off;
  for (int i = threadIdx.x; i < (kQbY + 4) * (kQbX + 4); i += 256) {
    const int r = i / (kQbX + 4), c = i % (kQbX + 4), y = y0 + r - 2, x = x0 + c - 2;
    q[r][c] = y >= 0 && y < m.h && x >= 0 && x < m.w ? quant_luma(Y[(int64_t)y * m.pitch + x]) : 0;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kQbY * (kQbX + 4); i += 256) {
    const int r = i / (kQbX + 4), c = i % (kQbX + 4);
    v[r][c] = q[r][c] + q[r + 1][c] + q[r + 2][c] + q[r + 3][c] + q[r + 4][c];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kQbY * kQbX; i += 256) {
    const int r = i / kQbX, c = i % kQbX, y = y0 + r, x = x0 + c;
    if (y < m.h && x < m.w)
      qblur[m.b_off + (int64_t)y * m.pitch + x] =
          (v[r][c] + v[r][c + 1] + v[r][c + 2] + v[r][c + 3] + v[r][c + 4] + 12) / 25;
  }
}


// SAD (or SSD) over the tile of source offset (dy, dx), one warp (lanes over pixels).
__device__ __forceinline__ unsigned long long warp_tile_cost(const int* As, const int* Bs, int b,
                                                             int ww, int S, int bh, int bw,
                                                             int dy, int dx, bool squared,
                                                             int lane) {
  unsigned long long acc = 0;
  for (int i = lane; i < bh * bw; i += 32) {
    const int yy = i / bw, xx = i % bw;
    const int d = As[yy * b + xx] - Bs[(yy - dy + S) * ww + (xx - dx + S)];
    acc += squared ? (unsigned long long)((long long)d * d) : (unsigned long long)abs(d);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}

// The exhaustive scan. For integers |a - b| = 2 max(a, b) - a - b, so a
// candidate's SAD is 2 sum max(A, B) - sum A - sum B over its window, the
// last from the window's integral image: one max and one add per candidate
// pixel, all in exact integers. Each item is one dy and G consecutive dx;
// its rows are split between two adjacent lanes (their sums meet by one
// shuffle), which halves the dependent chain of a candidate's additions.
// Blocks of BW = 16 columns keep a register window of the G + 15 row values
// they read (one new load per pixel). Returns the thread's best key (biased
// cost << 11 | centre-out visit index); the lane holding (0, 0) stores its
// SAD in *sad0.
// Two 16-bit lanes at once (the quantised luma is a uint16 code): the
// per-lane maximum, and the sum of the two lanes added to an accumulator by
// a two-way dot product with (1, 1).
__device__ __forceinline__ unsigned vmax_u16x2(unsigned a, unsigned b) {
  unsigned d;
  asm("max.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// Rows [yb, ye) of one item of a 16-wide block, packed: Ap holds the block's
// rows as 8 pairs (columns 2k, 2k + 1), BpE / BpO each window row's pairs
// starting at even / odd columns. For candidate offset dxg + g the window
// pair under block pair k starts at column e_lo + (G - 1 - g) + 2 k, e_lo =
// S - dxg - (G - 1); a0 = e_lo - Q (even, Q = e_lo & 1) is where this row's
// words are loaded from, so every register index below is a constant.
template <int G, int Q>
__device__ __forceinline__ void sad_rows_packed(const unsigned* __restrict__ Ap,
                                                const unsigned* __restrict__ BpE,
                                                const unsigned* __restrict__ BpO, int hb, int wp,
                                                int yb, int ye, int dy, int S, int a0h,
                                                unsigned (&acc)[G]) {
  constexpr int kWords = (Q + G - 1 + 14) / 2 + 1;
  for (int yy = yb; yy < ye; ++yy) {
    const unsigned* ap = Ap + yy * hb;
    const int row = yy - dy + S;
    const unsigned* be = BpE + row * wp + a0h;
    const unsigned* bo = BpO + row * wp + a0h;
    unsigned wE[kWords], wO[kWords];
#pragma unroll
    for (int j = 0; j < kWords; ++j) {
      wE[j] = be[j];
      wO[j] = bo[j];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const unsigned av = ap[k];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const int off = Q + (G - 1 - g) + 2 * k;
        const unsigned bv = (off & 1) ? wO[off >> 1] : wE[off >> 1];
        acc[g] = __dp2a_lo(vmax_u16x2(av, bv), 0x0101u, acc[g]);
      }
    }
  }
}

template <int G, int BW>
__device__ __forceinline__ unsigned long long sad_scan(const int* As, const int* Bs,
                                                       const int* I, const unsigned* Ap,
                                                       const unsigned* BpE, const unsigned* BpO,
                                                       int b, int ww, int S, int bh, int bw, int s,
                                                       unsigned sum_a, unsigned long long* sad0,
                                                       unsigned one) {
  const int n = 2 * s + 1;
  const int ngroups = (n + G - 1) / G;
  const int items = n * ngroups;
  const int wi = ww + 1;
  const int hsplit = (bh + 1) / 2;
  unsigned long long bestkey = ~0ull;
  // items (dy, group of G offsets) ordered by the parity of their packed
  // window start (odd G alternates it from group to group), so the lanes of a
  // warp take the same packed code path
  const int c0 = (S + s - G + 1) & 1;  // parity of group 0's start
  const int n0 = (G & 1) ? (ngroups - c0 + 1) / 2 : (c0 == 0 ? ngroups : 0);
  for (int base = 0; base < 2 * items; base += blockDim.x) {
    const int it = base + threadIdx.x;
    const bool valid = it < 2 * items;
    const int item = it >> 1, half = it & 1;
    int dyi, grp;
    if (!(G & 1)) {
      dyi = item / ngroups;
      grp = item % ngroups;
    } else if (item < n * n0) {
      dyi = item / n0;
      grp = c0 + 2 * (item % n0);
    } else {
      const int i1 = item - n * n0, n1 = ngroups - n0;
      dyi = i1 / n1;
      grp = (1 - c0) + 2 * (i1 % n1);
    }
    const int dy = dyi - s;
    const int dxg = -s + grp * G;
    unsigned acc[G];
#pragma unroll
    for (int g = 0; g < G; ++g) acc[g] = 0u;
    if (valid) {
      const int yb = half ? hsplit : 0, ye = half ? bh : hsplit;
      if (BW == 16) {
        const int e_lo = S - dxg - (G - 1);
        const int a0h = (e_lo - (e_lo & 1)) >> 1;
        if (e_lo & 1)
          sad_rows_packed<G, 1>(Ap, BpE, BpO, b / 2, ww / 2 + 1, yb, ye, dy, S, a0h, acc);
        else
          sad_rows_packed<G, 0>(Ap, BpE, BpO, b / 2, ww / 2 + 1, yb, ye, dy, S, a0h, acc);
      } else {
        for (int yy = yb; yy < ye; ++yy) {
          const int* ar = As + yy * b;
          // window value under pixel xx at offset dxg + g: br[xx - g]
          const int* br = Bs + (yy - dy + S) * ww + (S - dxg);
          for (int xx = 0; xx < bw; ++xx) {
            const int av = ar[xx];
#pragma unroll
            for (int g = 0; g < G; ++g) acc[g] = (unsigned)max(av, br[xx - g]) * one + acc[g];
          }
        }
      }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) acc[g] += __shfl_xor_sync(0xffffffffu, acc[g], 1);
    if (!valid || half) continue;
    const int r0 = S - dy;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int dx = dxg + g;
      if (dx > s) break;
      const int c0 = S - dx;
      const unsigned sum_b = (unsigned)(I[(r0 + bh) * wi + c0 + bw] - I[r0 * wi + c0 + bw] -
                                        I[(r0 + bh) * wi + c0] + I[r0 * wi + c0]);
      const unsigned sad = 2u * acc[g] - sum_a - sum_b;
      const unsigned long long cost =
          (unsigned long long)sad * (unsigned long long)(50 + abs(dy) + abs(dx));
      const unsigned long long ci =
          (unsigned long long)(centre_out_index(dy) * n + centre_out_index(dx));
      const unsigned long long key = (cost << 11) | ci;
      if (key < bestkey) bestkey = key;
      if (dy == 0 && dx == 0) *sad0 = sad;
    }
  }
  return bestkey;
}

// One CTA per (tile, pair).
__global__ void __launch_bounds__(kSadThreads, 6) k_sad_search(const MeField* __restrict__ mf,
                                                            const MePair* __restrict__ pairs,
                                                            const int* __restrict__ qblur,
                                                            SadArgs a, SadBuffers out) {
  const int p = blockIdx.y, t = blockIdx.x;
  const MePair pr = pairs[p];
  const MeField mc = mf[pr.cur], mr = mf[pr.ref];
  const int h = mc.h, w = mc.w, b = a.block, s = a.range;
  const int th = (h + b - 1) / b, tw = (w + b - 1) / b;
  if (t >= th * tw) return;
  const int ty = t / tw, tx = t % tw;
  const int y0 = ty * b, x0 = tx * b;
  const int bh = min(b, h - y0), bw = min(b, w - x0);
  const int S = s + 1;          // window margin: the search range plus the sub-pel neighbours
  const int ww = b + 2 * S;
  const int wi = ww + 1;
  extern __shared__ int sad_sm[];
  int* As = sad_sm;             // b x b
  int* Bs = sad_sm + b * b;     // ww x ww, B(clamp(y0 - S + wy), clamp(x0 - S + wx))
  int* I = Bs + ww * ww;        // (ww + 1)^2 integral image of Bs
  // packed 16-bit pairs: the block's rows (b / 2 per row), the window's rows
  // from even columns (BpE) and from odd columns (BpO), ww / 2 + 1 per row
  unsigned* Ap = reinterpret_cast<unsigned*>(I + (ww + 1) * (ww + 1));
  unsigned* BpE = Ap + b * (b / 2);
  unsigned* BpO = BpE + ww * (ww / 2 + 1);
  __shared__ unsigned long long red[kSadThreads / 32];
  __shared__ unsigned long long sh_sad0, sh_best, sh_side[4], sh_ssd;
  __shared__ long long sh_s1, sh_s2;
  __shared__ unsigned sh_suma;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int* QA = qblur + mc.b_off;
  const int* QB = qblur + mr.b_off;
  for (int i = tid; i < bh * bw; i += blockDim.x)
    As[(i / bw) * b + i % bw] = QA[(int64_t)(y0 + i / bw) * mc.pitch + x0 + i % bw];
  for (int i = tid; i < ww * ww; i += blockDim.x) {
    const int wy = i / ww, wx = i % ww;
    const int sy = clampi(y0 - S + wy, 0, h - 1), sx = clampi(x0 - S + wx, 0, w - 1);
    Bs[i] = QB[(int64_t)sy * mr.pitch + sx];
  }
  __syncthreads();
  // integral image: row prefix sums, then column prefix sums (exact ints:
  // the whole window sums below 2^31)
  for (int r = tid; r <= ww; r += blockDim.x) {
    int* Ir = I + r * wi;
    Ir[0] = 0;
    int acc = 0;
    if (r == 0) {
      for (int c = 1; c <= ww; ++c) Ir[c] = 0;
    } else {
      const int* br = Bs + (r - 1) * ww;
      for (int c = 1; c <= ww; ++c) {
        acc += br[c - 1];
        Ir[c] = acc;
      }
    }
  }
  {
    // the packed copies (columns past the window's edge pack as 0)
    const int hb = b / 2, wp = ww / 2 + 1;
    for (int i = tid; i < b * hb; i += blockDim.x) {
      const int r = i / hb, k = i % hb;
      Ap[i] = (unsigned)As[r * b + 2 * k] | ((unsigned)As[r * b + 2 * k + 1] << 16);
    }
    for (int i = tid; i < ww * wp; i += blockDim.x) {
      const int r = i / wp, k = i % wp;
      const int* br = Bs + r * ww;
      const unsigned e0 = 2 * k < ww ? (unsigned)br[2 * k] : 0u;
      const unsigned e1 = 2 * k + 1 < ww ? (unsigned)br[2 * k + 1] : 0u;
      const unsigned e2 = 2 * k + 2 < ww ? (unsigned)br[2 * k + 2] : 0u;
      BpE[i] = e0 | (e1 << 16);
      BpO[i] = e1 | (e2 << 16);
    }
  }
  if (warp == 0) {
    unsigned sa = 0;
    for (int i = lane; i < bh * bw; i += 32) sa += (unsigned)As[(i / bw) * b + i % bw];
    for (int o = 16; o > 0; o >>= 1) sa += __shfl_xor_sync(0xffffffffu, sa, o);
    if (lane == 0) sh_suma = sa;
  }
  __syncthreads();
  for (int c = tid; c <= ww; c += blockDim.x)
    for (int r = 1; r <= ww; ++r) I[r * wi + c] += I[(r - 1) * wi + c];
  __syncthreads();
  const int n = 2 * s + 1;
  const unsigned sum_a = sh_suma;
  // 1, in a form the compiler cannot fold: the accumulations are issued as
  // multiply-adds, which run on the FMA pipe beside the max on the integer
  // pipe (a plain add would share the integer pipe with the max)
  const unsigned one = ((unsigned)a.block >> 30) | 1u;
  // G consecutive dx per thread: 11 when it divides the row of candidates
  // (no wasted candidates at +-16), else 8
  unsigned long long bestkey;
  if (n % 11 == 0)
    bestkey = bw == 16 ? sad_scan<11, 16>(As, Bs, I, Ap, BpE, BpO, b, ww, S, bh, bw, s, sum_a, &sh_sad0, one)
                       : sad_scan<11, 0>(As, Bs, I, Ap, BpE, BpO, b, ww, S, bh, bw, s, sum_a, &sh_sad0, one);
  else
    bestkey = bw == 16 ? sad_scan<8, 16>(As, Bs, I, Ap, BpE, BpO, b, ww, S, bh, bw, s, sum_a, &sh_sad0, one)
                       : sad_scan<8, 0>(As, Bs, I, Ap, BpE, BpO, b, ww, S, bh, bw, s, sum_a, &sh_sad0, one);
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, bestkey, o);
    if (v < bestkey) bestkey = v;
  }
  if (lane == 0) red[warp] = bestkey;
  __syncthreads();
  if (tid == 0) {
    unsigned long long m = red[0];
    for (int i = 1; i < (int)(blockDim.x / 32); ++i) m = red[i] < m ? red[i] : m;
    sh_best = m;
  }
  __syncthreads();
  const unsigned long long best = sh_best >> 11;
  const int ci = (int)(sh_best & 2047ull);
  const int mdy = centre_out(ci / n), mdx = centre_out(ci % n);
  // the sub-pel neighbours' unbiased SADs, the zero-margin decision, then the
  // SSD at the final vector and the tile statistics of A (one warp each)
  const unsigned long long cost0 = 50ull * sh_sad0;
  const bool zero = 20ull * best > 17ull * cost0;
  const int fdy = zero ? 0 : mdy, fdx = zero ? 0 : mdx;
  if (warp < 4) {
    const int oy = warp == 0 ? -1 : (warp == 1 ? 1 : 0);
    const int ox = warp == 2 ? -1 : (warp == 3 ? 1 : 0);
    const unsigned long long v =
        warp_tile_cost(As, Bs, b, ww, S, bh, bw, mdy + oy, mdx + ox, false, lane);
    if (lane == 0) sh_side[warp] = v;
  } else if (warp == 4) {
    const unsigned long long v = warp_tile_cost(As, Bs, b, ww, S, bh, bw, fdy, fdx, true, lane);
    if (lane == 0) sh_ssd = v;
  } else if (warp == 5) {
    long long s1 = 0, s2 = 0;
    for (int i = lane; i < bh * bw; i += 32) {
      const long long v = As[(i / bw) * b + i % bw];
      s1 += v;
      s2 += v * v;
    }
    for (int o = 16; o > 0; o >>= 1) {
      s1 += __shfl_xor_sync(0xffffffffu, s1, o);
      s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) {
      sh_s1 = s1;
      sh_s2 = s2;
    }
  }
  __syncthreads();
  if (tid == 0) {
    // parabola through (-1, 50 SAD_m), (0, best), (+1, 50 SAD_p): exact
    // integer numerator and denominator, one division
    auto parabolic = [&](unsigned long long sm, unsigned long long sp) -> double {
      const long long num = 50ll * (long long)sm - 50ll * (long long)sp;
      const long long den = 50ll * (long long)sm - 2ll * (long long)best + 50ll * (long long)sp;
      double sub = den > 0 ? 0.5 * (double)num / (double)den : 0.0;
      return fmin(fmax(sub, -0.5), 0.5);
    };
    double sdy = parabolic(sh_side[0], sh_side[1]);
    double sdx = parabolic(sh_side[2], sh_side[3]);
    if (zero) {
      sdy = 0.0;
      sdx = 0.0;
    }
    const int o = a.tiles_off * p + t;
    out.mdy[o] = (float)fdy;
    out.mdx[o] = (float)fdx;
    out.sdy[o] = (float)sdy;
    out.sdx[o] = (float)sdx;
    const double sc2 = (double)kQuantScale * (double)kQuantScale;
    out.bestv[o] = (double)(sh_ssd * (unsigned long long)(50 + abs(fdy) + abs(fdx))) / (50.0 * sc2);
    out.s1[o] = (double)sh_s1;
    out.s2[o] = (double)sh_s2;
    out.npx[o] = (double)(bh * bw);
    out.dy[o] = (float)((double)fdy + sdy);
    out.dx[o] = (float)((double)fdx + sdx);
  }
}

// MotionConfidence on the IRE scale from the exact integer statistics. A
// cluster of eight CTAs per pair: the rank counts (nt^2 comparisons) bound it,
// so each CTA ranks an eighth of the tiles against all and tells the others of
// the middle ones it finds (750 tiles: 63 us by one CTA in two passes over the
// ranks, 23 by one of 1024 threads in one pass, 14 by the cluster).
constexpr int kSadConfThreads = 256, kSadConfCtas = 8;
__global__ void __cluster_dims__(kSadConfCtas, 1, 1) __launch_bounds__(kSadConfThreads)
    k_sad_confidence(const MeField* __restrict__ mf, const MePair* __restrict__ pairs, SadArgs a,
                     SadBuffers out) {
  extern __shared__ double sadc_sm[];
  __shared__ double mid[2];
  const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int p = blockIdx.x / kSadConfCtas, rank = blockIdx.x % kSadConfCtas;
  const MeField mc = mf[pairs[p].cur];
  const int b = a.block;
  const int th = (mc.h + b - 1) / b, tw = (mc.w + b - 1) / b, nt = th * tw;
  const int t0 = rank * kSadConfThreads + threadIdx.x;
  constexpr int kStep = kSadConfCtas * kSadConfThreads;
  double* ratios = sadc_sm;
  const int o = a.tiles_off * p;
  for (int t = threadIdx.x; t < nt; t += blockDim.x)
    ratios[t] = out.bestv[o + t] / fmax(1.0, out.npx[o + t]);
  __syncthreads();
  cl.sync();  // every CTA of the cluster runs: its shared memory can be written
  // the two middle ratios by counting ranks, both in one pass
  const int k = nt / 2;
  auto tell = [&](int which, double v) {
    for (int r = 0; r < kSadConfCtas; ++r) cl.map_shared_rank(mid, r)[which] = v;
  };
  for (int t = t0; t < nt; t += kStep) {
    const double v = ratios[t];
    int less = 0, eq = 0;
#pragma unroll 8
    for (int u = 0; u < nt; ++u) {
      less += ratios[u] < v;
      eq += ratios[u] == v;
    }
    if (less <= k && k < less + eq) tell(0, v);
    if (less <= k - 1 && k - 1 < less + eq) tell(1, v);
  }
  cl.sync();
  const double med = nt % 2 == 0 ? 0.5 * (mid[0] + mid[1]) : mid[0];
  const double sc2 = (double)kQuantScale * (double)kQuantScale;
  for (int t = t0; t < nt; t += kStep) {
    const double npx = out.npx[o + t];
    const double norm = 1.0 / fmax(1.0, npx);
    const double tmean = out.s1[o + t] * norm;
    const double tvar = (out.s2[o + t] * norm - tmean * tmean) / sc2;
    const double energy = (tvar + 1.0) * fmax(1.0, npx);
    double c = fmin(fmax(1.0 - out.bestv[o + t] / energy, 0.0), 1.0);
    const double excess = fmax(0.0, ratios[t] - med);
    c = c * ((med + 1.0) / (med + 1.0 + excess));
    c = c * (6.0 / (6.0 + med));
    out.conf[o + t] = (float)c;
  }
}

void launch_motion_sad(const MeField* d_fields, int nf, int max_h, int max_w,
                       const MePair* d_pairs, int npairs, const SadArgs& a, const SadBuffers& b,
                       cudaStream_t st) {
  if (nf <= 0 || npairs <= 0) return;
  k_sad_blur<<<dim3((max_w + kQbX - 1) / kQbX, (max_h + kQbY - 1) / kQbY, nf), 256, 0, st>>>(
      d_fields, b.luma, b.qblur);
  const int th = (max_h + a.block - 1) / a.block, tw = (max_w + a.block - 1) / a.block;
  const int ww = a.block + 2 * (a.range + 1);
  const int smem = sad_smem_ints(a.block, ww) * (int)sizeof(int);
  static PerDeviceOnce sad_once;
  sad_once([] {
    cudaFuncSetAttribute(k_sad_search, cudaFuncAttributeMaxDynamicSharedMemorySize, kSadMaxSmem);
  });
  k_sad_search<<<dim3(th * tw, npairs), kSadThreads, smem, st>>>(d_fields, d_pairs, b.qblur, a, b);
  k_sad_confidence<<<npairs * kSadConfCtas, kSadConfThreads, th * tw * (int)sizeof(double), st>>>(
      d_fields, d_pairs, a, b);
}

// ---------------------------------------------------------------------------
// VectorsPerPixel (temporal.cpp:45-112): 3x3 median outlier snap on the tile
// grid, then bilinear interpolation between tile centres.
// ---------------------------------------------------------------------------
__device__ float median9(float* v) {
  // exact middle of 9 values (nth_element(v, v + 4, v + 9))
  for (int i = 0; i < 5; ++i) {
    int mi = i;
    for (int j = i + 1; j < 9; ++j)
      if (v[j] < v[mi]) mi = j;
    const float t = v[i];
    v[i] = v[mi];
    v[mi] = t;
  }
  return v[4];
}

// Snapped tile vectors; one thread per (pair, tile).
__global__ void k_vec_snap(const MeField* __restrict__ mf, const MePair* __restrict__ pairs,
                           int npairs, MeArgs a, const float* __restrict__ dy_in,
                           const float* __restrict__ dx_in, float* __restrict__ dy_out,
                           float* __restrict__ dx_out) {
  const int p = blockIdx.y;
  if (p >= npairs) return;
  const MeField mc = mf[pairs[p].cur];
  const int th = (mc.h + a.tile - 1) / a.tile, tw = (mc.w + a.tile - 1) / a.tile;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= th * tw) return;
  const int o = a.tiles_off * p;
  float vy = dy_in[o + t], vx = dx_in[o + t];
  if (th >= 3 && tw >= 3) {
    const int ty = t / tw, tx = t % tw;
    float ay[9], ax[9];
    int q = 0;
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        const int yy = clampi(ty + dy, 0, th - 1), xx = clampi(tx + dx, 0, tw - 1);
        ay[q] = dy_in[o + yy * tw + xx];
        ax[q] = dx_in[o + yy * tw + xx];
        ++q;
      }
    const float my = median9(ay), mx = median9(ax);
    const float dis = fabsf(vy - my) + fabsf(vx - mx);
    if (dis > 3.0f) {
      vy = my;
      vx = mx;
    }
  }
  dy_out[o + t] = vy;
  dx_out[o + t] = vx;
}

__device__ __forceinline__ void bracket(int coord, int n_tiles, int tile, int* lo, float* frac) {
  if (n_tiles > 1) {
    const float rel = (float)coord / (float)tile - 0.5f;
    *lo = clampi((int)floorf(rel), 0, n_tiles - 2);
    const float centre_lo = ((float)*lo + 0.5f) * (float)tile;
    *frac = fminf(fmaxf(((float)coord - centre_lo) / (float)tile, 0.0f), 1.0f);
  } else {
    *lo = 0;
    *frac = 0.0f;
  }
}

__device__ __forceinline__ float interp_tiles(const float* v, int tw, int iy, int iy1, int ix,
                                              int ix1, float fy, float fx) {
  const float v00 = v[iy * tw + ix], v10 = v[iy1 * tw + ix];
  const float v01 = v[iy * tw + ix1], v11 = v[iy1 * tw + ix1];
  return v00 * (1 - fy) * (1 - fx) + v10 * fy * (1 - fx) + v01 * (1 - fy) * fx + v11 * fy * fx;
}

// Per-pixel vectors for one pair, written as the warp source indices
// (sy, sx) = (clamp(y - lround(vdy)), clamp(x - lround(vdx))) packed in an
// int2, plus (optionally) the interpolated squared confidence (fast mode).
__global__ void k_vec_pixels(const MeField* __restrict__ mf, const MePair* __restrict__ pairs,
                             int npairs, MeArgs a, const float* __restrict__ sdy,
                             const float* __restrict__ sdx, int2* __restrict__ src_idx,
                             const int64_t* __restrict__ pix_off) {
  const int p = blockIdx.z;
  if (p >= npairs) return;
  const MeField mc = mf[pairs[p].cur];
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  if (x >= mc.w || y >= mc.h) return;
  const int th = (mc.h + a.tile - 1) / a.tile, tw = (mc.w + a.tile - 1) / a.tile;
  int iy, ix;
  float fy, fx;
  bracket(y, th, a.tile, &iy, &fy);
  bracket(x, tw, a.tile, &ix, &fx);
  const int iy1 = min(iy + 1, th - 1), ix1 = min(ix + 1, tw - 1);
  const int o = a.tiles_off * p;
  const float vy = interp_tiles(sdy + o, tw, iy, iy1, ix, ix1, fy, fx);
  const float vx = interp_tiles(sdx + o, tw, iy, iy1, ix, ix1, fy, fx);
  const int sy = clampi(y - (int)lroundf(vy), 0, mc.h - 1);
  const int sx = clampi(x - (int)lroundf(vx), 0, mc.w - 1);
  src_idx[pix_off[p] + (int64_t)y * mc.pitch + x] = make_int2(sy, sx);
}

// Squared per-tile confidence -> per pixel.
//   fast: VectorsPerPixel of conf^2 (snap + bilinear), temporal.cpp:245-254
//   slow: nearest tile, squared, then BoxBlur radius 8, temporal.cpp:227-243
__global__ void k_conf_sq(const MeField* __restrict__ mf, const MePair* __restrict__ pairs,
                          int npairs, MeArgs a, const float* __restrict__ conf,
                          float* __restrict__ c2) {
  const int p = blockIdx.y;
  if (p >= npairs) return;
  const MeField mc = mf[pairs[p].cur];
  const int nt = ((mc.h + a.tile - 1) / a.tile) * ((mc.w + a.tile - 1) / a.tile);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const float c = conf[a.tiles_off * p + t];
  c2[a.tiles_off * p + t] = c * c;
}

__global__ void k_conf_pixels_fast(const MeField* __restrict__ mf, const MePair* __restrict__ pairs,
                                   int npairs, MeArgs a, const float* __restrict__ c2s,
                                   float* __restrict__ out, const int64_t* __restrict__ pix_off) {
  const int p = blockIdx.z;
  if (p >= npairs) return;
  const MeField mc = mf[pairs[p].cur];
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  if (x >= mc.w || y >= mc.h) return;
  const int th = (mc.h + a.tile - 1) / a.tile, tw = (mc.w + a.tile - 1) / a.tile;
  int iy, ix;
  float fy, fx;
  bracket(y, th, a.tile, &iy, &fy);
  bracket(x, tw, a.tile, &ix, &fx);
  out[pix_off[p] + (int64_t)y * mc.pitch + x] =
      interp_tiles(c2s + a.tiles_off * p, tw, iy, min(iy + 1, th - 1), ix, min(ix + 1, tw - 1), fy, fx);
}

__global__ void k_conf_pixels_nearest(const MeField* __restrict__ mf, const MePair* __restrict__ pairs,
                                      int npairs, MeArgs a, const float* __restrict__ conf,
                                      float* __restrict__ out, const int64_t* __restrict__ pix_off) {
  const int p = blockIdx.z;
  if (p >= npairs) return;
  const MeField mc = mf[pairs[p].cur];
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  if (x >= mc.w || y >= mc.h) return;
  const int th = (mc.h + a.tile - 1) / a.tile, tw = (mc.w + a.tile - 1) / a.tile;
  const int ty = min(y / a.tile, th - 1), tx = min(x / a.tile, tw - 1);
  const float c = conf[a.tiles_off * p + ty * tw + tx];
  out[pix_off[p] + (int64_t)y * mc.pitch + x] = c * c;
}

// BoxBlur radius r over per-pair planes (the luma blur's arithmetic), and over
// several channels `chan` floats apart: columns, then rows.
__global__ void __launch_bounds__(kBoxThreads) k_pair_blur_v(
    const MeField* __restrict__ mf, const MePair* __restrict__ pairs, int npairs, const float* src,
    float* dst, const int64_t* __restrict__ pix_off, int64_t chan, int r, int band) {
  const int p = blockIdx.y;
  if (p >= npairs) return;
  const MeField m = mf[pairs[p].cur];
  const int x0 = blockIdx.x * band;
  if (x0 >= m.w) return;
  const int64_t o = pix_off[p] + blockIdx.z * chan + x0;
  box_cols(src + o, dst + o, m.pitch, band, min(band, m.w - x0), m.h, r,
           (double)(1.0f / (float)(2 * r + 1)));
}

__global__ void __launch_bounds__(kBoxThreads) k_pair_blur_h(
    const MeField* __restrict__ mf, const MePair* __restrict__ pairs, int npairs, float* plane,
    const int64_t* __restrict__ pix_off, int64_t chan, int r, int band) {
  const int p = blockIdx.y;
  if (p >= npairs) return;
  const MeField m = mf[pairs[p].cur];
  const int y0 = blockIdx.x * band;
  if (y0 >= m.h) return;
  float* d = plane + pix_off[p] + blockIdx.z * chan + (int64_t)y0 * m.pitch;
  box_rows(d, d, m.pitch, min(band, m.h - y0), m.w, r, (double)(1.0f / (float)(2 * r + 1)));
}

static PerDeviceOnce box_once;

static void configure_box() {
  box_once([] {
    cudaFuncSetAttribute(k_blur_v, cudaFuncAttributeMaxDynamicSharedMemorySize, kBoxSmem);
    cudaFuncSetAttribute(k_blur_h, cudaFuncAttributeMaxDynamicSharedMemorySize, kBoxSmem);
    cudaFuncSetAttribute(k_pair_blur_v, cudaFuncAttributeMaxDynamicSharedMemorySize, kBoxSmem);
    cudaFuncSetAttribute(k_pair_blur_h, cudaFuncAttributeMaxDynamicSharedMemorySize, kBoxSmem);
  });
}

// The luma planes' blur (tmp, then blur).
static void field_blur(const MeField* d_fields, int nf, int max_h, int max_w, const MeBuffers& b,
                       cudaStream_t st) {
  configure_box();
  const int cb = col_band(max_h), rb = row_band(max_w);
  const int cl = cb ? cb : kBoxThreads, rl = rb ? rb : kBoxThreads;  // lines per block
  k_blur_v<<<dim3((max_w + cl - 1) / cl, nf), kBoxThreads, sizeof(double) * cb * (max_h + 1), st>>>(
      d_fields, nf, b.luma, b.tmp, 2, 0, cb);
  k_blur_h<<<dim3((max_h + rl - 1) / rl, nf), kBoxThreads,
             sizeof(double) * rb * row_stride(max_w), st>>>(d_fields, nf, b.tmp, b.blur, 2, rb);
}

// `chans` channels of the pairs' planes (fields of a window: every line fits
// shared memory): src -> dst, src and dst may be the same.
static void pair_blur(const MeField* d_fields, const MePair* d_pairs, int npairs, int max_h,
                      int max_w, const float* src, float* dst, const int64_t* pix_off, int chans,
                      int64_t chan, int r, cudaStream_t st) {
  configure_box();
  const int cb = col_band(max_h), rb = row_band(max_w);
  k_pair_blur_v<<<dim3((max_w + cb - 1) / cb, npairs, chans), kBoxThreads,
                  sizeof(double) * cb * (max_h + 1), st>>>(d_fields, d_pairs, npairs, src, dst,
                                                           pix_off, chan, r, cb);
  k_pair_blur_h<<<dim3((max_h + rb - 1) / rb, npairs, chans), kBoxThreads,
                  sizeof(double) * rb * row_stride(max_w), st>>>(d_fields, d_pairs, npairs, dst,
                                                                 pix_off, chan, r, rb);
}

// ---------------------------------------------------------------------------
// Trajectory consensus, fast-mode verification, motion cache, coherence gate
// ---------------------------------------------------------------------------
// numpy.median of up to kTrajMaxPairs values (Median, motion.cpp:80-91 and
// MedianOf, sequence.cpp:29-39: the mean of the two middles for even n)
__device__ float median_small(float* v, int n) {
  for (int i = 1; i < n; ++i) {
    const float x = v[i];
    int j = i - 1;
    while (j >= 0 && v[j] > x) {
      v[j + 1] = v[j];
      --j;
    }
    v[j + 1] = x;
  }
  const int k = n / 2;
  float m = v[k];
  if (n % 2 == 0) m = 0.5f * (m + v[k - 1]);
  return m;
}

// TrajectorySnap (motion.cpp:565-601) with FitTrajectory (:532-563): one
// thread per (field group, tile).
__global__ void k_traj_snap(const MeField* __restrict__ mf, const MePair* __restrict__ pairs,
                            const TrajGroup* __restrict__ groups, int ngroups,
                            const TrajPair* __restrict__ tp, int tile, int tiles_off,
                            float* __restrict__ dy, float* __restrict__ dx,
                            const float* __restrict__ conf) {
  const int g = blockIdx.y;
  if (g >= ngroups) return;
  const TrajGroup G = groups[g];
  if (G.count < 2) return;
  const MeField mc = mf[pairs[G.pair[0]].cur];
  const int th = (mc.h + tile - 1) / tile, tw = (mc.w + tile - 1) / tile;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= th * tw) return;
  float sy[kTrajMaxPairs], sx[kTrajMaxPairs];
  int n = 0;
  for (int i = 0; i < G.count; ++i) {
    const int p = G.pair[i];
    const TrajPair q = tp[p];
    if (q.offset == 0) continue;
    const int o = tiles_off * p + t;
    if (conf[o] <= 0.15f) continue;
    const float of = (float)q.offset;
    sy[n] = (dy[o] - q.parity_shift) / of;
    sx[n] = dx[o] / of;
    ++n;
  }
  float vym = 0.0f, vxm = 0.0f;
  if (n > 0) {
    vym = median_small(sy, n);
    vxm = median_small(sx, n);
  }
  // consensus: the snap applies where >= 3 offsets agree within 1.5 px
  float agree = 0.0f;
  for (int i = 0; i < G.count; ++i) {
    const int p = G.pair[i];
    const TrajPair q = tp[p];
    const int o = tiles_off * p + t;
    const float of = (float)q.offset;
    const float py = of * vym + q.parity_shift;
    const float px = of * vxm;
    const float dev = fabsf(dy[o] - py) + fabsf(dx[o] - px);
    if (dev <= 1.5f) agree += 1.0f;
  }
  if (agree < 3.0f) return;
  for (int i = 0; i < G.count; ++i) {
    const int p = G.pair[i];
    const TrajPair q = tp[p];
    const int o = tiles_off * p + t;
    const float of = (float)q.offset;
    const float py = of * vym + q.parity_shift;
    const float px = of * vxm;
    const float dev = fabsf(dy[o] - py) + fabsf(dx[o] - px);
    if (dev <= 1.5f) {
      dy[o] = py;
      dx[o] = px;
    }
  }
}

// VerifyMotion (motion.cpp:490-530) of pair base + i: one SSD at the rounded
// prediction, one at zero, the prediction kept where it is strictly better.
// The prediction is the trajectory median over the searched pairs of its
// group (sequence.cpp:714-763), or, with pred_dy / pred_dx given, the
// caller's per-tile vectors.
//
// A warp per tile: the squared differences of the prediction and of zero
// motion are formed by all lanes into shared memory, kVerifyChunk pixels at a
// time, and two lanes add them in the reference's order (4 cycles a pixel). A
// thread per sum reading global memory took 96 us for the pairs of a six-frame
// NTSC window, this 20.
constexpr int kVerifyChunk = 1024;
constexpr int kVerifyWarps = 4;
__global__ void __launch_bounds__(32 * kVerifyWarps) k_traj_verify(
    const MeField* __restrict__ mf, const MePair* __restrict__ pairs, int base, int npred,
    const int* __restrict__ grp, const TrajGroup* __restrict__ searched,
    const TrajPair* __restrict__ tp, const float* __restrict__ blur, MeArgs a,
    const float* __restrict__ dy_in, const float* __restrict__ dx_in,
    const float* __restrict__ pred_dy, const float* __restrict__ pred_dx,
    float* __restrict__ out_mdy, float* __restrict__ out_mdx, float* __restrict__ out_sdy,
    float* __restrict__ out_sdx, float* __restrict__ out_best) {
  __shared__ float sq[kVerifyWarps][2][kVerifyChunk];
  const int i = blockIdx.y;
  const int p = base + i;
  const MePair pr = pairs[p];
  const MeField mc = mf[pr.cur], mr = mf[pr.ref];
  const int h = mc.h, w = mc.w, tile = a.tile;
  const int th = (h + tile - 1) / tile, tw = (w + tile - 1) / tile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = blockIdx.x * kVerifyWarps + warp;
  if (t >= th * tw) return;  // the whole warp; only warp-level sync below
  float pdy = 0.0f, pdx = 0.0f;
  if (pred_dy) {
    pdy = pred_dy[a.tiles_off * i + t];
    pdx = pred_dx[a.tiles_off * i + t];
  } else {
    if (lane == 0) {
      const TrajGroup S = searched[grp[i]];
      float sy[kTrajMaxPairs], sx[kTrajMaxPairs];
      for (int k = 0; k < S.count; ++k) {
        const int q = S.pair[k];
        const TrajPair m = tp[q];
        const float of = (float)m.offset;
        sy[k] = (dy_in[a.tiles_off * q + t] - m.parity_shift) / of;
        sx[k] = dx_in[a.tiles_off * q + t] / of;
      }
      const float vym0 = S.count > 0 ? median_small(sy, S.count) : 0.0f;
      const float vxm0 = S.count > 0 ? median_small(sx, S.count) : 0.0f;
      const TrajPair me = tp[p];
      pdy = (float)me.offset * vym0 + me.parity_shift;
      pdx = (float)me.offset * vxm0;
    }
    pdy = __shfl_sync(0xffffffffu, pdy, 0);
    pdx = __shfl_sync(0xffffffffu, pdx, 0);
  }
  const int iy = (int)lroundf(pdy), ix = (int)lroundf(pdx);
  const int y0 = t / tw * tile, x0 = t % tw * tile;
  const int cols = min(tile, w - x0), n = min(tile, h - y0) * cols;
  const float* A = blur + mc.b_off;
  const float* B = blur + mr.b_off;
  float* s0 = sq[warp][0];
  float* s1 = sq[warp][1];
  float acc = 0.0f;
  for (int c0 = 0; c0 < n; c0 += kVerifyChunk) {
    const int m = min(kVerifyChunk, n - c0);
#pragma unroll 4
    for (int k = lane; k < m; k += 32) {
      const int y = y0 + (c0 + k) / cols, x = x0 + (c0 + k) % cols;
      const float v = A[(int64_t)y * mc.pitch + x];
      const float dp = v - B[(int64_t)clampi(y - iy, 0, h - 1) * mc.pitch + clampi(x - ix, 0, w - 1)];
      const float dz = v - B[(int64_t)y * mc.pitch + x];
      s0[k] = dp * dp;
      s1[k] = dz * dz;
    }
    __syncwarp();
    if (lane < 2) {
      const float* v = lane == 0 ? s0 : s1;
#pragma unroll 16
      for (int k = 0; k < m; ++k) acc += v[k];
    }
    __syncwarp();
  }
  const float zero = __shfl_sync(0xffffffffu, acc, 1);
  if (lane != 0) return;
  const float pred = acc;
  const int o = a.tiles_off * p + t;
  if (zero <= pred) {
    out_mdy[o] = 0.0f;
    out_mdx[o] = 0.0f;
    out_best[o] = zero;
  } else {
    // the full float prediction is kept where it won
    out_mdy[o] = pdy;
    out_mdx[o] = pdx;
    out_best[o] = pred;
  }
  out_sdy[o] = 0.0f;
  out_sdx[o] = 0.0f;
}

__global__ void k_motion_cache(const int* __restrict__ gid, int npairs, int nt, int tiles_off,
                               float* __restrict__ dy, float* __restrict__ dx,
                               float* __restrict__ conf, float* __restrict__ cache,
                               int64_t stride, int store) {
  const int i = blockIdx.y;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= npairs || t >= nt) return;
  const int64_t c = (int64_t)gid[i] * nt + t;
  const int o = tiles_off * i + t;
  if (store) {
    cache[c] = dy[o];
    cache[stride + c] = dx[o];
    cache[2 * stride + c] = conf[o];
  } else {
    dy[o] = cache[c];
    dx[o] = cache[stride + c];
    conf[o] = cache[2 * stride + c];
  }
}

// Cross terms of chi_j and chi_k bilinearly warped by the snapped per-pixel
// vectors (WarpBilinearTiles, temporal.cpp:140-168, row offset 0).
__global__ void k_coh_terms(const MeField* __restrict__ mf, const MePair* __restrict__ pairs,
                            int npairs, MeArgs a, CohBuffers b) {
  const int p = blockIdx.z;
  if (p >= npairs) return;
  const MePair pr = pairs[p];
  const MeField mc = mf[pr.cur], mr = mf[pr.ref];
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  if (x >= mc.w || y >= mc.h) return;
  const int th = (mc.h + a.tile - 1) / a.tile, tw = (mc.w + a.tile - 1) / a.tile;
  int iy, ix;
  float fyb, fxb;
  bracket(y, th, a.tile, &iy, &fyb);
  bracket(x, tw, a.tile, &ix, &fxb);
  const int iy1 = min(iy + 1, th - 1), ix1 = min(ix + 1, tw - 1);
  const int o = a.tiles_off * p;
  const float vy = interp_tiles(b.snap_dy + o, tw, iy, iy1, ix, ix1, fyb, fxb);
  const float vx = interp_tiles(b.snap_dx + o, tw, iy, iy1, ix, ix1, fyb, fxb);
  float sy = (float)y - vy + 0.0f;
  float sx = (float)x - vx;
  sy = fminf(fmaxf(sy, 0.0f), (float)mr.h - 1.001f);
  sx = fminf(fmaxf(sx, 0.0f), (float)mr.w - 1.001f);
  const int y0 = (int)sy, x0 = (int)sx;
  const float fy = sy - (float)y0, fx = sx - (float)x0;
  const int y1 = min(y0 + 1, mr.h - 1), x1 = min(x0 + 1, mr.w - 1);
  const float2* K = b.chi + mr.y_off;
  const float2 k00 = K[(int64_t)y0 * mr.pitch + x0], k10 = K[(int64_t)y1 * mr.pitch + x0];
  const float2 k01 = K[(int64_t)y0 * mr.pitch + x1], k11 = K[(int64_t)y1 * mr.pitch + x1];
  const float wre = k00.x * (1 - fy) * (1 - fx) + k10.x * fy * (1 - fx) + k01.x * (1 - fy) * fx +
                    k11.x * fy * fx;
  const float wim = k00.y * (1 - fy) * (1 - fx) + k10.y * fy * (1 - fx) + k01.y * (1 - fy) * fx +
                    k11.y * fy * fx;
  const float2 z1 = b.chi[mc.y_off + (int64_t)y * mc.pitch + x];
  // z1 * conj(cw)
  const float cre = z1.x * wre - z1.y * (-wim);
  const float cim = z1.x * (-wim) + z1.y * wre;
  const int64_t q = b.pix_off[p] + (int64_t)y * mc.pitch + x;
  b.terms[q] = cre;
  b.terms[b.chan_stride + q] = cim;
  b.terms[2 * b.chan_stride + q] = z1.x * z1.x + z1.y * z1.y;
  b.terms[3 * b.chan_stride + q] = wre * wre + wim * wim;
}

__global__ void k_coh_apply(const MeField* __restrict__ mf, const MePair* __restrict__ pairs,
                            int npairs, CohBuffers b, float gate) {
  const int p = blockIdx.z;
  if (p >= npairs) return;
  const MeField mc = mf[pairs[p].cur];
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  if (x >= mc.w || y >= mc.h) return;
  const int64_t q = b.pix_off[p] + (int64_t)y * mc.pitch + x;
  const float re = b.terms[q], im = b.terms[b.chan_stride + q];
  const float m1 = b.terms[2 * b.chan_stride + q], m2 = b.terms[3 * b.chan_stride + q];
  const float num = sqrtf(re * re + im * im);
  const float den = sqrtf(fmaxf(0.0f, m1 * m2)) + 1e-6f;
  const float gamma = fminf(fmaxf(num / den, 0.0f), 1.0f);
  b.conf_px[q] *= (1.0f - gate) + gate * gamma;
}

void launch_vectors(const MeField* d_fields, const MePair* d_pairs, int npairs, int max_h,
                    int max_w, const MeArgs& a, const VecBuffers& v, bool fast_conf,
                    cudaStream_t st) {
  if (npairs <= 0) return;
  const int th = (max_h + a.tile - 1) / a.tile, tw = (max_w + a.tile - 1) / a.tile;
  const int nt = th * tw;
  k_vec_snap<<<dim3((nt + 63) / 64, npairs), 64, 0, st>>>(d_fields, d_pairs, npairs, a, v.dy, v.dx,
                                                          v.snap_dy, v.snap_dx);
  k_vec_pixels<<<dim3((max_w + 127) / 128, max_h, npairs), 128, 0, st>>>(
      d_fields, d_pairs, npairs, a, v.snap_dy, v.snap_dx, v.src_idx, v.pix_off);
  if (fast_conf) {
    k_conf_sq<<<dim3((nt + 63) / 64, npairs), 64, 0, st>>>(d_fields, d_pairs, npairs, a, v.conf, v.c2);
    k_vec_snap<<<dim3((nt + 63) / 64, npairs), 64, 0, st>>>(d_fields, d_pairs, npairs, a, v.c2, v.c2,
                                                            v.c2_snap, v.c2_snap2);
    k_conf_pixels_fast<<<dim3((max_w + 127) / 128, max_h, npairs), 128, 0, st>>>(
        d_fields, d_pairs, npairs, a, v.c2_snap, v.conf_px, v.pix_off);
  } else {
    k_conf_pixels_nearest<<<dim3((max_w + 127) / 128, max_h, npairs), 128, 0, st>>>(
        d_fields, d_pairs, npairs, a, v.conf, v.conf_tmp, v.pix_off);
    pair_blur(d_fields, d_pairs, npairs, max_h, max_w, v.conf_tmp, v.conf_px, v.pix_off, 1, 0, 8, st);
  }
}

void launch_traj_snap(const MeField* d_fields, const MePair* d_pairs, const TrajGroup* d_groups,
                      int ngroups, const TrajPair* d_tp, int max_h, int max_w, int tile,
                      int tiles_off, float* dy, float* dx, const float* conf, cudaStream_t st) {
  if (ngroups <= 0) return;
  const int nt = ((max_h + tile - 1) / tile) * ((max_w + tile - 1) / tile);
  k_traj_snap<<<dim3((nt + 63) / 64, ngroups), 64, 0, st>>>(d_fields, d_pairs, d_groups, ngroups,
                                                           d_tp, tile, tiles_off, dy, dx, conf);
}

void launch_traj_verify(const MeField* d_fields, const MePair* d_pairs, int base, int npred,
                        const int* d_grp, const TrajGroup* d_searched, const TrajPair* d_tp,
                        const float* blur, int max_h, int max_w, const MeArgs& a,
                        const float* dy_in, const float* dx_in, float* mdy, float* mdx,
                        float* sdy, float* sdx, float* best, cudaStream_t st,
                        const float* pred_dy, const float* pred_dx) {
  if (npred <= 0) return;
  const int nt = ((max_h + a.tile - 1) / a.tile) * ((max_w + a.tile - 1) / a.tile);
  k_traj_verify<<<dim3((nt + kVerifyWarps - 1) / kVerifyWarps, npred), 32 * kVerifyWarps, 0, st>>>(
      d_fields, d_pairs, base, npred, d_grp, d_searched, d_tp, blur, a, dy_in, dx_in, pred_dy,
      pred_dx, mdy, mdx, sdy, sdx, best);
}

void launch_me_confidence(const MeField* d_fields, const MePair* d_pairs, int npairs, int max_h,
                          int max_w, const MeArgs& a, const float* blur, const float* mdy,
                          const float* mdx, const float* sdy, const float* sdx, const float* best,
                          float* dy, float* dx, float* conf, cudaStream_t st) {
  if (npairs <= 0) return;
  const int th = (max_h + a.tile - 1) / a.tile, tw = (max_w + a.tile - 1) / a.tile;
  const int nt = th * tw;
  k_me_tile_stats<<<dim3((nt + kConfWarps - 1) / kConfWarps, npairs), 32 * kConfWarps, 0, st>>>(
      d_fields, d_pairs, blur, a, best, dy, conf);
  k_me_confidence<<<npairs, 256, nt * (int)sizeof(float), st>>>(d_pairs, a, nt, mdy, mdx, sdy, sdx,
                                                                dy, dx, conf);
}

void launch_motion_cache(const int* d_gid, int npairs, int nt, int tiles_off, float* dy, float* dx,
                         float* conf, float* cache, int64_t cache_stride, bool store,
                         cudaStream_t st) {
  if (npairs <= 0) return;
  k_motion_cache<<<dim3((nt + 127) / 128, npairs), 128, 0, st>>>(d_gid, npairs, nt, tiles_off, dy,
                                                                dx, conf, cache, cache_stride,
                                                                store ? 1 : 0);
}

void launch_coherence_gate(const MeField* d_fields, const MePair* d_pairs, int npairs, int max_h,
                           int max_w, const MeArgs& a, const CohBuffers& b, float gate,
                           cudaStream_t st) {
  if (npairs <= 0) return;
  const dim3 grid((max_w + 127) / 128, max_h, npairs);
  k_coh_terms<<<grid, 128, 0, st>>>(d_fields, d_pairs, npairs, a, b);
  // ComplexCoherence's four BoxBlur(r = 6) passes (temporal.cpp:186-189)
  pair_blur(d_fields, d_pairs, npairs, max_h, max_w, b.terms, b.terms, b.pix_off, 4, b.chan_stride,
            6, st);
  k_coh_apply<<<grid, 128, 0, st>>>(d_fields, d_pairs, npairs, b, gate);
}

// ---------------------------------------------------------------------------
// DrizzleFrame (sequence.cpp:283-421). Compiled with the rest of this file
// without multiply-add contraction, so every deposit position, weight and
// blend is the reference's float arithmetic; only the order of the float
// accumulations differs (atomics), i.e. the sums agree to rounding.
// ---------------------------------------------------------------------------

// One thread per (pair, source sample): robust agreement weight with the
// target's own decode at the rounded warp, linear split between the two
// fine rows around (2 (y + vy) + p_k) scale.
__global__ void k_drizzle_deposit(const DrizzlePair* __restrict__ pairs, int npairs, DrizzleArgs a) {
  const int pi = blockIdx.z;
  if (pi >= npairs) return;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y;
  if (x >= a.w || y >= a.h) return;
  const DrizzlePair pr = pairs[pi];
  const int L = a.h, W = a.w, HF = 2 * L * a.scale;
  float vy = 0.0f, vx = 0.0f, cpx = 1.0f;
  if (pr.me >= 0) {
    const int th = (L + a.tile - 1) / a.tile, tw = (W + a.tile - 1) / a.tile;
    int iy, ix;
    float fy, fx;
    bracket(y, th, a.tile, &iy, &fy);
    bracket(x, tw, a.tile, &ix, &fx);
    const int iy1 = min(iy + 1, th - 1), ix1 = min(ix + 1, tw - 1);
    const int o = a.tiles_off * pr.me;
    vy = interp_tiles(a.sdy + o, tw, iy, iy1, ix, ix1, fy, fx);
    vx = interp_tiles(a.sdx + o, tw, iy, iy1, ix, ix1, fy, fx);
    cpx = a.conf[o + min(y / a.tile, th - 1) * tw + min(x / a.tile, tw - 1)];
  }
  const int64_t plane = (int64_t)L * a.pitch;
  const float* Yk = a.Y + plane * pr.src;
  const float* Yt = a.Y + plane * pr.tgt;
  const float2* Ck = a.C + plane * pr.src;
  const float2* Ct = a.C + plane * pr.tgt;
  const int syi = clampi((int)lroundf((float)y - vy), 0, L - 1);
  const int sxi = clampi((int)lroundf((float)x - vx), 0, W - 1);
  const float sk = Yk[(int64_t)y * a.pitch + x];
  const float2 ck = Ck[(int64_t)y * a.pitch + x];
  const float dY = sk - Yt[(int64_t)syi * a.pitch + sxi];
  const float2 ct = Ct[(int64_t)syi * a.pitch + sxi];
  const float dr = ck.x - ct.x, di = ck.y - ct.y;
  const float d2 = dY * dY + (dr * dr + di * di);
  const float wgt = cpx * a.eps_b * a.eps_b / (d2 + a.eps_b * a.eps_b);
  const float yf = (2.0f * ((float)y + vy) + (float)a.parity[pr.src]) * (float)a.scale;
  const int xs = clampi((int)lroundf((float)x + vx), 0, W - 1);
  const int y0 = (int)floorf(yf);
  const float fyr = yf - (float)y0;
  const int64_t fp = (int64_t)HF * W;
  for (int off = 0; off < 2; ++off) {
    const int yt = clampi(y0 + off, 0, HF - 1);
    const float ww = wgt * (off == 0 ? (1.0f - fyr) : fyr);
    const int64_t q = (int64_t)yt * W + xs;
    atomicAdd(a.acc + q, ww * sk);
    atomicAdd(a.acc + fp + q, ww * ck.x);
    atomicAdd(a.acc + 2 * fp + q, ww * ck.y);
    atomicAdd(a.acc + 3 * fp + q, ww);
  }
}

// Coverage blend with the linearly interpolated plain weave of fields j0,
// j0 + 1 (sequence.cpp:385-419). One thread per fine sample.
__global__ void k_drizzle_resolve(DrizzleArgs a) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  const int L = a.h, W = a.w, HF = 2 * L * a.scale;
  if (x >= W || r >= HF) return;
  const int64_t plane = (int64_t)L * a.pitch;
  const int p0 = a.parity[a.j0], p1 = a.parity[a.j0 + 1];
  auto woven = [&](int row, float2* c) {
    // row 2 t + p1 from field j0 + 1 (written last), else 2 t + p0 from j0, else 0
    const int t = row >> 1, par = row & 1;
    const int64_t o = (int64_t)t * a.pitch + x;
    if (par == p1) {
      *c = a.C[plane * (a.j0 + 1) + o];
      return a.Y[plane * (a.j0 + 1) + o];
    }
    if (par == p0) {
      *c = a.C[plane * a.j0 + o];
      return a.Y[plane * a.j0 + o];
    }
    *c = make_float2(0.f, 0.f);
    return 0.0f;
  };
  const float fine = (float)r / (float)a.scale;
  const int f0 = clampi((int)floorf(fine), 0, 2 * L - 2);
  const float ff = fine - (float)f0;
  float2 c0, c1;
  const float y0v = woven(f0, &c0), y1v = woven(f0 + 1, &c1);
  const float baseY = y0v * (1.0f - ff) + y1v * ff;
  const float bcr = c0.x * (1.0f - ff) + c1.x * ff;
  const float bci = c0.y * (1.0f - ff) + c1.y * ff;
  const int64_t fp = (int64_t)HF * W, q = (int64_t)r * W + x;
  const float aw = a.acc[3 * fp + q];
  const float mix = aw / (aw + 0.35f);
  const float den = fmaxf(aw, 1e-9f);
  const float dzY = aw > 0.0f ? a.acc[q] / den : 0.0f;
  const float dcr = aw > 0.0f ? a.acc[fp + q] / den : 0.0f;
  const float dci = aw > 0.0f ? a.acc[2 * fp + q] / den : 0.0f;
  a.out_y[q] = mix * dzY + (1.0f - mix) * baseY;
  a.out_c[q] = make_float2(mix * dcr + (1.0f - mix) * bcr, mix * dci + (1.0f - mix) * bci);
}

void launch_drizzle(const DrizzlePair* d_pairs, int npairs, const DrizzleArgs& a, cudaStream_t st) {
  const int HF = 2 * a.h * a.scale;
  if (npairs > 0)
    k_drizzle_deposit<<<dim3((a.w + 127) / 128, a.h, npairs), 128, 0, st>>>(d_pairs, npairs, a);
  k_drizzle_resolve<<<dim3((a.w + 127) / 128, HF), 128, 0, st>>>(a);
}

void launch_vec_snap(const MeField* d_fields, const MePair* d_pairs, int npairs, int max_h,
                     int max_w, const MeArgs& a, const float* dy, const float* dx, float* sdy,
                     float* sdx, cudaStream_t st) {
  if (npairs <= 0) return;
  const int nt = ((max_h + a.tile - 1) / a.tile) * ((max_w + a.tile - 1) / a.tile);
  k_vec_snap<<<dim3((nt + 63) / 64, npairs), 64, 0, st>>>(d_fields, d_pairs, npairs, a, dy, dx,
                                                          sdy, sdx);
}

}  // namespace hvdg
