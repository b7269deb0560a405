// Wyner-Ziv frame kernels other than LDPCA: side-information creation,
// transforms, correlation-noise model, conditional bit probabilities,
// reconstruction, side-information refinement and motion learning.
//
// Every kernel takes the array of per-frame descriptors of a batch and uses
// blockIdx.y (or blockIdx.x for single-block-per-frame kernels) as the frame
// index, so one launch serves every frame of the batch.  Frames whose
// descriptor is not `active` return at once.
//
// Each kernel restates one reference function (paths in DvcDec/src) with the
// same operation order for every float/double result; the module is compiled
// with -fmad=false so no multiply-add is fused.
#include <cuda_runtime.h>

#include <atomic>

#include "dvc_common.cuh"
#include "frame_types.h"
#include "kernels.h"
#include "ldpca_bp.cuh"

namespace dvc {

#define SEARCH_R 32  // defines.h:8
#define LEARN_R 4    // defines.h:11
#define ML_N 81

__constant__ double c_post_scale[16];
__constant__ double c_pre_scale[16];

// updateSI motion-vector weight 1 + 0.05f * |2v| per integer displacement
// (dx, dy) in [-32, 32]^2 (sideInfoCreation.cpp:667-668), indexed
// (dy + 32) * 65 + dx + 32
__device__ double d_si_weight[65 * 65];

cudaError_t upload_transform_scales(const double *post, const double *pre) {
  cudaError_t e = cudaMemcpyToSymbol(c_post_scale, post, sizeof(double) * 16);
  if (e != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_pre_scale, pre, sizeof(double) * 16)) != cudaSuccess) return e;
  // IEEE square root on the host gives the device's bits (no contraction: -ffp-contract=off)
  static double wt[65 * 65];
  for (int dy = -32; dy <= 32; dy++)
    for (int dx = -32; dx <= 32; dx++) {
      const double vx = (double)(dx << 1), vy = (double)(dy << 1);
      wt[(dy + 32) * 65 + dx + 32] = 1.0 + (double)0.05f * sqrt(vx * vx + vy * vy);
    }
  return cudaMemcpyToSymbol(d_si_weight, wt, sizeof wt);
}

// Does the frame take part in step (band, bit)?  band < 0: frame-level steps.
// Bands are decoded in zig-zag order while Qbits > 0 (DVC_Decoder.cpp:161-165,
// 403-407); bitplanes from Qbits down to 1 (:196).
__device__ __forceinline__ bool in_step(const FrameDev &F, int band, int bit) {
  if (band < 0) return true;
  for (int b = 0; b <= band; b++)
    if (F.qbits[c_zigzag[b]] <= 0) return false;
  return bit <= 0 || bit <= F.qbits[c_zigzag[band]];
}

// ROUND, defines.h:23
__device__ __forceinline__ int dround(double x) { return x >= 0.0 ? (int)(x + 0.5) : -(int)(-x + 0.5); }

// x moved by k units in the last place (x positive and finite)
__device__ __forceinline__ double ulp_shift(double x, int k) {
  return __longlong_as_double(__double_as_longlong(x) + (long long)k);
}

// costFunc, sideInfoCreation.cpp:10-12 (K is the float 0.05f, promoted)
__device__ __forceinline__ double cost_func(double mad, double vx, double vy) {
  return mad * (1.0 + (double)0.05f * sqrt(vx * vx + vy * vy));
}

// computeEndPoint, sideInfoCreation.cpp:14-22
__device__ __forceinline__ int end_point(double st, double v, double scale, int lo, int hi) {
  const int e = (int)((st + v * scale) + 0.5);
  return e < lo ? lo : (e > hi ? hi : e);
}

// forward44, transform.cpp:63-104
__device__ __forceinline__ void forward44(int *blk) {
  int t[16];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    t[c] = blk[c] + blk[4 + c] + blk[8 + c] + blk[12 + c];
    t[4 + c] = (blk[c] << 1) + blk[4 + c] - blk[8 + c] - (blk[12 + c] << 1);
    t[8 + c] = blk[c] - blk[4 + c] - blk[8 + c] + blk[12 + c];
    t[12 + c] = blk[c] - (blk[4 + c] << 1) + (blk[8 + c] << 1) - blk[12 + c];
  }
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int *s = t + 4 * r;
    int *o = blk + 4 * r;
    o[0] = s[0] + s[1] + s[2] + s[3];
    o[1] = (s[0] << 1) + s[1] - s[2] - (s[3] << 1);
    o[2] = s[0] - s[1] - s[2] + s[3];
    o[3] = s[0] - (s[1] << 1) + (s[2] << 1) - s[3];
  }
#pragma unroll
  for (int i = 0; i < 16; i++) blk[i] = dround(((double)blk[i]) * c_post_scale[i]);
}

// inverse44, transform.cpp:106-151
__device__ __forceinline__ void inverse44(int *blk) {
  int t[16];
#pragma unroll
  for (int i = 0; i < 16; i++) blk[i] = dround(((double)blk[i]) * c_pre_scale[i]);
#pragma unroll
  for (int c = 0; c < 4; c++) {
    t[c] = blk[c] + blk[4 + c] + blk[8 + c] + (blk[12 + c] >> 1);
    t[4 + c] = blk[c] + (blk[4 + c] >> 1) - blk[8 + c] - blk[12 + c];
    t[8 + c] = blk[c] - (blk[4 + c] >> 1) - blk[8 + c] + blk[12 + c];
    t[12 + c] = blk[c] - blk[4 + c] + blk[8 + c] - (blk[12 + c] >> 1);
  }
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int *s = t + 4 * r;
    int *o = blk + 4 * r;
    o[0] = s[0] + s[1] + s[2] + (s[3] >> 1);
    o[1] = s[0] + (s[1] >> 1) - s[2] - s[3];
    o[2] = s[0] - (s[1] >> 1) - s[2] + s[3];
    o[3] = s[0] - s[1] + s[2] - (s[3] >> 1);
  }
#pragma unroll
  for (int i = 0; i < 16; i++) blk[i] >>= 6;
}

// argmin with the reference's strict-< row-major scan: lowest cost, then lowest scan index
__device__ __forceinline__ void better(double &c, int &i, double c2, int i2) {
  if (c2 < c || (c2 == c && i2 < i)) {
    c = c2;
    i = i2;
  }
}

template <int NT>
__device__ __forceinline__ void block_argmin(double &c, int &i, double *sc, int *si) {
  for (int o = 16; o > 0; o >>= 1) {
    const double c2 = __shfl_xor_sync(0xffffffffu, c, o);
    const int i2 = __shfl_xor_sync(0xffffffffu, i, o);
    better(c, i, c2, i2);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) {
    sc[warp] = c;
    si[warp] = i;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < NT / 32; w++) better(c, i, sc[w], si[w]);
    sc[0] = c;
    si[0] = i;
  }
  __syncthreads();
  c = sc[0];
  i = si[0];
}

// lowest (cost, index) over a full warp for costs >= 0 (never NaN): a
// non-negative double orders like its bit pattern, so three 32-bit warp
// reductions give it (high word, low word among the lanes that hold the
// smallest high word, index among the lanes that hold the smallest cost)
__device__ __forceinline__ void warp_argmin_nonneg(double &c, int &i) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(c);
  const unsigned hw = (unsigned)(b >> 32), lw = (unsigned)b;
  const unsigned mh = __reduce_min_sync(0xffffffffu, hw);
  const unsigned ml = __reduce_min_sync(0xffffffffu, hw == mh ? lw : 0xffffffffu);
  const unsigned mi = __reduce_min_sync(0xffffffffu, (hw == mh && lw == ml) ? (unsigned)i : 0xffffffffu);
  c = __longlong_as_double((long long)(((unsigned long long)mh << 32) | ml));
  i = (int)mi;
}

// ---------------------------------------------------------------- filters

// lowPassFilter, filter.cpp:214-233
__global__ void lowpass_kernel(const uint8_t *__restrict__ in, int w, int h, uint8_t *__restrict__ out) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= w) return;
  double sum = 0;
  for (int m = y - 1; m <= y + 1; m++) {
    if (m < 0 || m >= h) continue;
    for (int n = x - 1; n <= x + 1; n++) {
      if (n < 0 || n >= w) continue;
      sum += (double)in[m * w + n];
    }
  }
  out[y * w + x] = (uint8_t)(sum / 9);
}

// FIR_filter, filter.cpp:55-117, on the output window it keeps.  The taps are
// the separable (1,-5,20,20,-5,1) half-pel filter: /32 horizontally or
// vertically, /1024 at the centre position; zero taps of the reference's 6x6
// tables are skipped (adding +0 to the running sum never changes it).
__global__ void fir_kernel(const uint8_t *__restrict__ in, int w, int h, uint8_t *__restrict__ out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  const int w2 = w << 1;
  if (j >= w2) return;
  const double tap[6] = {1.0, -5.0, 20.0, 20.0, -5.0, 1.0};
  const int sub = (j & 1) + ((i & 1) << 1);
  const int cy = i / 2, cx = j / 2;
  auto px = [&](int yy, int xx) {
    yy = yy < 0 ? 0 : (yy > h - 1 ? h - 1 : yy);
    xx = xx < 0 ? 0 : (xx > w - 1 ? w - 1 : xx);
    return (double)in[yy * w + xx];
  };
  uint8_t v;
  if (sub == 0) {
    v = (uint8_t)px(cy, cx);
  } else {
    double sum = 0.0;
    if (sub == 1) {
      for (int jj = 0; jj < 6; jj++) sum += (tap[jj] / 32.0) * px(cy, cx - 2 + jj);
    } else if (sub == 2) {
      for (int ii = 0; ii < 6; ii++) sum += (tap[ii] / 32.0) * px(cy - 2 + ii, cx);
    } else {
      for (int ii = 0; ii < 6; ii++)
        for (int jj = 0; jj < 6; jj++) sum += ((tap[ii] * tap[jj]) / 1024.0) * px(cy - 2 + ii, cx - 2 + jj);
    }
    int r = (int)(sum + 0.5);
    v = (uint8_t)(r < 0 ? 0 : (r > 255 ? 255 : r));
  }
  out[i * w2 + j] = v;
}

cudaError_t launch_ref_planes(const uint8_t *recon, int w, int h, uint8_t *lp, uint8_t *ip, cudaStream_t s) {
  lowpass_kernel<<<dim3((w + 127) / 128, h), 128, 0, s>>>(recon, w, h, lp);
  fir_kernel<<<dim3((2 * w + 127) / 128, 2 * h), 128, 0, s>>>(recon, w, h, ip);
  return cudaGetLastError();
}

// ----------------------------------------------------- side-info creation

// forwardME, sideInfoCreation.cpp:61-118: per 16x16 block of the future
// low-pass frame, full search of +-32 pixels in the past low-pass frame.
template <int NT>
__global__ void __launch_bounds__(NT) forward_me_kernel(FrameDev *frames) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active) return;
  const int w = F.w, h = F.h, b16w = w / 16;
  const int i = blockIdx.x;
  const int top = (i / b16w) << 4, left = (i % b16w) << 4;
  int st = top - SEARCH_R, sb = top + SEARCH_R, sl = left - SEARCH_R, sr = left + SEARCH_R;
  if (st < 0) st = 0;
  if (sb > h - 16) sb = h - 16;
  if (sl < 0) sl = 0;
  if (sr > w - 16) sr = w - 16;
  const int ww = sr - sl + 16, wh = sb - st + 16;  // staged window (<= 80x80)
  // window rows of 84 bytes in aligned 4-byte words: the window starts at byte
  // `wo` of each row (w is a multiple of 4, so the words of [sl & ~3, sl + ww)
  // stay inside the frame row; ww + 3 <= 84); the block's rows four pixels per
  // word (first pixel lowest)
  constexpr int WS = 84;
  __shared__ __align__(16) uint8_t win[80 * WS];
  __shared__ uint32_t blk4[64];
  __shared__ double sc[NT / 32];
  __shared__ int sidx[NT / 32];
  const int wo = sl & 3, nwd = (wo + ww + 3) >> 2;
  for (int y = threadIdx.x >> 5; y < wh; y += NT / 32) {
    const uint32_t *src = reinterpret_cast<const uint32_t *>(F.past_lp + (size_t)(st + y) * w + (sl - wo));
    uint32_t *dst = reinterpret_cast<uint32_t *>(win + y * WS);
    for (int x = threadIdx.x & 31; x < nwd; x += 32) dst[x] = __ldg(src + x);
  }
  for (int k = threadIdx.x; k < 64; k += NT)
    blk4[k] = __ldg(reinterpret_cast<const uint32_t *>(F.future_lp + (size_t)(top + (k >> 2)) * w + left) + (k & 3));
  __syncthreads();
  const int cw = sr - sl + 1, nc = cw * (sb - st + 1);
  double best = 1e300;
  int bi = 0x7fffffff;
  // candidate c = py * cw + pxo, advanced by NT without a division per candidate
  const int dq = NT / cw, dr = NT - dq * cw;
  int py = threadIdx.x / cw, pxo = threadIdx.x - py * cw;
  for (int c = threadIdx.x; c < nc; c += NT) {
    const int X = pxo + wo, sh = (X & 3) * 8;
    const uint32_t *rb = reinterpret_cast<const uint32_t *>(win) + (X >> 2);
    int sad = 0;
#pragma unroll 4
    for (int m = 0; m < 16; m++) {
      const uint32_t *r = rb + (py + m) * (WS / 4);
      const uint32_t w0 = r[0], w1 = r[1], w2 = r[2], w3 = r[3], w4 = r[4];
      sad += (int)__vsadu4(__funnelshift_r(w0, w1, sh), blk4[4 * m]);
      sad += (int)__vsadu4(__funnelshift_r(w1, w2, sh), blk4[4 * m + 1]);
      sad += (int)__vsadu4(__funnelshift_r(w2, w3, sh), blk4[4 * m + 2]);
      sad += (int)__vsadu4(__funnelshift_r(w3, w4, sh), blk4[4 * m + 3]);
    }
    const double vx = (double)(sl + pxo - left), vy = (double)(st + py - top);
    const double cost = cost_func((double)sad, vx, vy);
    if (cost < 10000000.0) better(best, bi, cost, c);
    pxo += dr;
    py += dq;
    if (pxo >= cw) {
      pxo -= cw;
      py++;
    }
  }
  block_argmin<NT>(best, bi, sc, sidx);
  if (threadIdx.x == 0) {
    MVd v{};
    if (bi != 0x7fffffff) {
      const int py = st + bi / cw, px = sl + bi % cw;
      v.px = (double)px;
      v.py = (double)py;
      v.vx = (double)(px - left);
      v.vy = (double)(py - top);
    }
    F.fmv[i] = v;
    F.holes[2 * i] = (double)left * F.ipc + (double)v.px * F.ifc;
    F.holes[2 * i + 1] = (double)top * F.ipc + (double)v.py * F.ifc;
  }
}

// forwardME, sideInfoCreation.cpp:120-142 (nearest projected hole per
// macroblock) and the half-pel scaling of createSideInfo (:511-521).  A warp
// per macroblock: its lanes share the holes, the first of the nearest wins (a
// thread per macroblock reading all holes took 58 us for a CIF frame, 5 us so).
__global__ void forward_me_post_kernel(FrameDev *frames) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active) return;
  const int w = F.w, h = F.h, b16w = w / 16, b16n = b16w * (h / 16);
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= b16n) return;
  const int top = (i / b16w) << 4, left = (i % b16w) << 4;
  const double maxd = w * w + h * h;
  double mind = maxd;
  int bj = 0x7fffffff;
#pragma unroll 4
  for (int j = lane; j < b16n; j += 32) {
    const double2 hole = reinterpret_cast<const double2 *>(F.holes)[j];
    const double d = (left - hole.x) * (left - hole.x) + (top - hole.y) * (top - hole.y);
    if (d < mind) {
      mind = d;
      bj = j;
    }
  }
  warp_argmin_nonneg(mind, bj);
  if (lane != 0) return;
  MVd b{};
  if (bj != 0x7fffffff) b = F.fmv[bj];
  MVd o;
  o.fx = (double)end_point(left, -b.vx, F.ifc, 0, w - 16);
  o.fy = (double)end_point(top, -b.vy, F.ifc, 0, h - 16);
  o.px = (double)end_point(left, b.vx, F.ipc, 0, w - 16);
  o.py = (double)end_point(top, b.vy, F.ipc, 0, h - 16);
  o.vx = o.px - o.fx;
  o.vy = o.py - o.fy;
  // half-pel units
  o.fx *= 2;
  o.fy *= 2;
  o.px *= 2;
  o.py *= 2;
  o.vx = o.px - o.fx;
  o.vy = o.py - o.fy;
  F.mb_mv[i] = o;
}

// SAD of the BL x BL block (every second half-pel sample of a 2BL x 2BL area)
// at f and p, by LP = 32 or 4 lanes, l the lane's number among them: some rows
// each, or a share of one row.  All lanes of a candidate get the sum.
template <int BL, int LP>
__device__ __forceinline__ int bidirect_sad(const uint8_t *f, const uint8_t *p, int w2, int l) {
  constexpr int SPLIT = LP > BL ? LP / BL : 1;   // lanes per row
  constexpr int ROWS = LP > BL ? 1 : BL / LP;    // rows per lane
  constexpr int PX = BL / SPLIT;                 // samples per lane and row
  const int r0 = LP > BL ? l / SPLIT : l * ROWS, x0 = (l % SPLIT) * PX * 2;
  int sad = 0;
#pragma unroll
  for (int r = 0; r < ROWS; r++) {
    const int o = 2 * (r0 + r) * w2 + x0;
    int a[PX], b[PX];
#pragma unroll
    for (int i = 0; i < PX; i++) {
      a[i] = __ldg(f + o + 2 * i);
      b[i] = __ldg(p + o + 2 * i);
    }
#pragma unroll
    for (int i = 0; i < PX; i++) sad += abs(a[i] - b[i]);
  }
  if constexpr (LP == 32) {
    return __reduce_add_sync(0xffffffffu, sad);
  } else {
    sad += __shfl_xor_sync(0xffffffffu, sad, 1);
    return sad + __shfl_xor_sync(0xffffffffu, sad, 2);
  }
}

// bidirectME, sideInfoCreation.cpp:235-310.  The reference visits blocks in
// raster order and updates the vectors in place; a block's search window uses
// its top and left neighbours' updated and its bottom and right neighbours'
// previous vectors.  Blocks on one anti-diagonal are therefore independent, and
// this kernel (one thread block per frame) walks the anti-diagonals, which is
// equivalent to the raster order.
// What bounds it: the chain of 39 (16x16 blocks) or 79 (8x8) dependent
// diagonals of a CIF frame.  Most windows hold one candidate, which needs no
// search, and a few hold hundreds, so the candidates of all blocks of a diagonal are dealt out to all
// warps: small windows a candidate at a time, its samples over 32 lanes, larger
// ones eight at a time, four lanes each (neighbouring candidates' samples share
// sectors).  One warp per block, a lane per candidate took 592 us a launch for
// either size on a lone CIF frame; now 167 (16x16) and 239 us (cold caches).
template <int BL>
__global__ void __launch_bounds__(1024) bidirect_me_kernel(FrameDev *frames) {
  FrameDev &F = frames[blockIdx.x];
  if (!F.active) return;
  constexpr int BL2 = 2 * BL, NW = 32, SMALL = 4;
  constexpr int MAXD = 288 / BL, MAXB = MAXD * (352 / BL);
  MVd *mv = BL == 16 ? F.mb_mv : F.blk_mv;
  const int w = F.w, h = F.h, bh = h / BL, bw = w / BL, w2 = w << 1;
  const int srb = (h << 1) - BL2, srr = w2 - BL2;
  const double scale = F.ipc / F.ifc;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint8_t *fut = F.future_ip, *pas = F.past_ip;
  __shared__ int16_t px_[MAXB], py_[MAXB];       // future end point of every block
  __shared__ int4 win[MAXD];                     // window of a diagonal's block: top, left, columns, candidates
  __shared__ int first[MAXD + 1];                // first work item of each
  __shared__ double scost[MAXD][NW];             // best cost and candidate by warp
  __shared__ int sidx[MAXD][NW];
  __shared__ int s_d;
  auto past_y = [&](int y2, int fy) { return end_point(y2, (double)(y2 - fy), scale, 0, srb); };
  auto past_x = [&](int x2, int fx) { return end_point(x2, (double)(x2 - fx), scale, 0, srr); };
  auto update = [&](int i, int j, int fy, int fx) {
    const int py = past_y(i * BL2, fy), px = past_x(j * BL2, fx), bi = i * bw + j;
    MVd b;
    b.fx = (double)fx;
    b.fy = (double)fy;
    b.px = (double)px;
    b.py = (double)py;
    b.vx = (double)(px - fx);
    b.vy = (double)(py - fy);
    mv[bi] = b;
    px_[bi] = (int16_t)fx;
    py_[bi] = (int16_t)fy;
  };
  for (int b = threadIdx.x; b < bh * bw; b += 1024) {
    px_[b] = (int16_t)(int)mv[b].fx;
    py_[b] = (int16_t)(int)mv[b].fy;
  }
  __syncthreads();
  for (int d = 0;; d++) {
    if (warp == 0) {
      // the windows of the next diagonal that has a choice to make: a block
      // with one candidate takes it whatever its SAD (the cost is below the
      // limit of 10^7 for any: 256 * 255 * (1 + 0.05 * |(704, 576)|))
      for (; d < bh + bw - 1; d++) {
        const int i0 = d - (bw - 1) > 0 ? d - (bw - 1) : 0;
        const int i1 = d < bh - 1 ? d : bh - 1, nb = i1 - i0 + 1;
        int base = 0;
        for (int q0 = 0; q0 < nb; q0 += 32) {
          const int q = q0 + lane, i = i0 + q, j = d - i, bi = i * bw + j;
          int items = 0;
          if (q < nb) {
            const int st = (i - 1 >= 0) ? py_[bi - bw] + BL2 : py_[bi];
            const int sb = (i + 1 < bh) ? py_[bi + bw] - BL2 : py_[bi];
            const int sl = (j - 1 >= 0) ? px_[bi - 1] + BL2 : px_[bi];
            const int sr = (j + 1 < bw) ? px_[bi + 1] - BL2 : px_[bi];
            const int cw = sr - sl + 1, chh = sb - st + 1;
            const int nc = (cw > 0 && chh > 0) ? cw * chh : 0;
            win[q] = make_int4(st, sl, cw, nc);
            if (nc == 1)
              update(i, j, st, sl);
            else
              items = nc <= SMALL ? nc : (nc + 7) >> 3;
          }
          if (__any_sync(0xffffffffu, items)) {
            int sum = items;
            for (int o = 1; o < 32; o <<= 1) {
              const int v = __shfl_up_sync(0xffffffffu, sum, o);
              if (lane >= o) sum += v;
            }
            if (q < nb) first[q] = base + sum - items;
            base += __shfl_sync(0xffffffffu, sum, 31);
          } else if (q < nb) {
            first[q] = base;
          }
        }
        if (lane == 0) first[nb] = base;
        __syncwarp();
        if (base) break;
      }
      if (lane == 0) s_d = d;
    } else {
      for (int k = threadIdx.x - 32; k < MAXD * NW; k += 1024 - 32) {
        scost[k >> 5][k & 31] = 1e300;
        sidx[k >> 5][k & 31] = 0x7fffffff;
      }
    }
    __syncthreads();
    d = s_d;
    if (d >= bh + bw - 1) break;
    const int i0 = d - (bw - 1) > 0 ? d - (bw - 1) : 0;
    const int i1 = d < bh - 1 ? d : bh - 1, nb = i1 - i0 + 1;
    const int total = first[nb], per = (total + NW - 1) / NW;
    int it = warp * per;
    const int end = min(total, it + per);
    if (it < end) {
      int q = 0;
      while (first[q + 1] <= it) q++;
      while (it < end) {
        const int4 W = win[q];
        const int stop = min(end, first[q + 1]), i = i0 + q, y2 = i * BL2, x2 = (d - i) * BL2;
        const bool small = W.w <= SMALL;
        double best = 1e300;
        int bc = 0x7fffffff;
        for (; it < stop; it++) {
          const int k = it - first[q];
          const int c = small ? k : min(8 * k + (lane >> 2), W.w - 1);  // past the last: the last again
          const int cy = c / W.z, fy = W.x + cy, fx = W.y + c - cy * W.z;
          const int py = past_y(y2, fy), px = past_x(x2, fx);
          const uint8_t *fr = fut + fy * w2 + fx, *pr = pas + py * w2 + px;
          const int mad = small ? bidirect_sad<BL, 32>(fr, pr, w2, lane) : bidirect_sad<BL, 4>(fr, pr, w2, lane & 3);
          // the weight is at least 1: only a SAD not above the best cost can win
          if ((double)mad <= best) {
            const double cost = cost_func((double)mad, (double)(px - fx), (double)(py - fy));
            if (cost < 10000000.0) better(best, bc, cost, c);
          }
        }
        warp_argmin_nonneg(best, bc);
        if (lane == 0) {
          scost[q][warp] = best;
          sidx[q][warp] = bc;
        }
        q++;
        while (q < nb && first[q + 1] <= it) q++;  // blocks with nothing to search
      }
    }
    __syncthreads();
    for (int q = warp; q < nb; q += NW) {
      if (first[q + 1] == first[q]) continue;
      double c = scost[q][lane];
      int bc = sidx[q][lane];
      warp_argmin_nonneg(c, bc);
      if (lane == 0 && bc != 0x7fffffff) update(i0 + q, d - i0 - q, win[q].x + bc / win[q].z, win[q].y + bc % win[q].z);
    }
    __syncthreads();
  }
}

// createSideInfo, sideInfoCreation.cpp:524-545: 8x8 vectors initialised
// from their macroblock's vector
__global__ void init_blk_mv_kernel(FrameDev *frames) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active) return;
  const int w = F.w, h = F.h, b8w = w / 8, b8n = b8w * (h / 8), b16w = w / 16;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= b8n) return;
  const int i = k / b8w, j = k % b8w;
  const int srb = (h - 8) << 1, srr = (w - 8) << 1;
  const int y2 = i << 4, x2 = j << 4;
  const MVd v = F.mb_mv[(i >> 1) * b16w + (j >> 1)];
  MVd o;
  o.fx = (double)end_point(x2, -v.vx, F.ifc, 0, srr);
  o.fy = (double)end_point(y2, -v.vy, F.ifc, 0, srb);
  o.px = (double)end_point(x2, v.vx, F.ipc, 0, srr);
  o.py = (double)end_point(y2, v.vy, F.ipc, 0, srb);
  o.vx = o.px - o.fx;
  o.vy = o.py - o.fy;
  F.blk_mv[k] = o;
}

// motionFilterAndComp, sideInfoCreation.cpp:325-342: mean squared error per 8x8 block
__global__ void mfc_mse_kernel(FrameDev *frames) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active) return;
  const int w = F.w, h = F.h, b8n = (w / 8) * (h / 8), w2 = w << 1;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= b8n) return;
  const MVd v = F.blk_mv[k];
  const int fy = (int)v.fy, fx = (int)v.fx, py = (int)v.py, px = (int)v.px;
  double s = 0.0;
  for (int m = 0; m < 16; m += 2)
    for (int n = 0; n < 16; n += 2) {
      const double d = (double)F.future_ip[(fy + m) * w2 + fx + n] - (double)F.past_ip[(py + m) * w2 + px + n];
      s += d * d;
    }
  F.mse[k] = s / 64;
}

// motionFilterAndComp, sideInfoCreation.cpp:344-405: weighted vector median
// over the 3x3 neighbourhood, then the new end points.  A lane per candidate
// neighbour (16 lanes a block, up to nine of them at work) sums its weighted
// distances in neighbour order; the choice is then the sequential scan's.
// (One thread per block did 72 divisions and roots in a row, 31 us; 9 us so.)
__global__ void mfc_wvmf_kernel(FrameDev *frames) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active) return;
  const int w = F.w, h = F.h, b8w = w / 8, b8h = h / 8, b8n = b8w * b8h;
  const int k = min((int)(blockIdx.x * blockDim.x + threadIdx.x) >> 4, b8n - 1), c = threadIdx.x & 15;
  const int i = k / b8w, j = k % b8w;
  const int srb = (h << 1) - 16, srr = (w << 1) - 16;
  const int y2 = i << 4, x2 = j << 4;
  // neighbours in raster order, those outside the frame left out
  const int r0 = max(i - 1, 0), r1 = min(i + 1, b8h - 1), c0 = max(j - 1, 0), c1 = min(j + 1, b8w - 1);
  const int nw = c1 - c0 + 1, cnt = nw * (r1 - r0 + 1);
  const MVd *mv = F.blk_mv;
  const double *mse = F.mse;
  const int cb = (r0 + min(c, cnt - 1) / nw) * b8w + c0 + min(c, cnt - 1) % nw;
  const double vx = mv[cb].vx, vy = mv[cb].vy, m = mse[cb];
  double wv = 0.0;
  // (both blocks of a warp take all nine turns: the shuffles need every lane)
  for (int q = 0; q < 9; q++) {
    // neighbour q's vector and error from its lane
    const double ox = __shfl_sync(0xffffffffu, vx, q, 16), oy = __shfl_sync(0xffffffffu, vy, q, 16);
    const double om = __shfl_sync(0xffffffffu, m, q, 16);
    if (c == q || q >= cnt) continue;
    const double dx = vx - ox, dy = vy - oy;
    wv += m / om * sqrt(dx * dx + dy * dy);
  }
  double minw = __shfl_sync(0xffffffffu, wv, 0, 16);
  int bc = 0;
  for (int q = 1; q < 9; q++) {
    const double v = __shfl_sync(0xffffffffu, wv, q, 16);
    if (q < cnt && v < minw) {
      minw = v;
      bc = q;
    }
  }
  const double bx = __shfl_sync(0xffffffffu, vx, bc, 16), by = __shfl_sync(0xffffffffu, vy, bc, 16);
  if (c != 0) return;
  MVd o;
  o.fx = (double)end_point(x2, -bx, F.ifc, 0, srr);
  o.fy = (double)end_point(y2, -by, F.ifc, 0, srb);
  o.px = (double)end_point(x2, bx, F.ipc, 0, srr);
  o.py = (double)end_point(y2, by, F.ipc, 0, srb);
  o.vx = o.px - o.fx;
  o.vy = o.py - o.fy;
  F.blk_mv2[k] = o;
}

// motionFilterAndComp, sideInfoCreation.cpp:407-434 (bidirectional motion
// compensation -> side information and residue), then copyIntraBlkToSideInfo
// (intra.cpp:271-288)
__global__ void mfc_comp_kernel(FrameDev *frames) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active) return;
  const int w = F.w, h = F.h, w2 = w << 1;
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.z;
  if (x >= w || y >= h) return;
  const int b8 = (y >> 3) * (w >> 3) + (x >> 3);
  const MVd v = F.blk_mv2[b8];
  const int m = (y & 7) << 1, n = (x & 7) << 1;
  const int fi = ((int)v.fy + m) * w2 + (int)v.fx + n, pi = ((int)v.py + m) * w2 + (int)v.px + n;
  const uint8_t fv = F.future_ip[fi], pv = F.past_ip[pi];
  uint8_t s = (uint8_t)(int)((double)fv * F.ifc + (double)pv * F.ipc);
  if (F.mode[b8] == DVC_INTRA_B) s = F.recon[y * w + x];
  F.si[y * w + x] = s;
  F.residue[y * w + x] = ((int)fv - (int)pv) >> 1;
}

// copySkipBlkToRecons, skipBlock.cpp:3-22: skip blocks take the past frame's pixels
__global__ void skip_copy_kernel(FrameDev *frames) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active || F.skip_mode != 1) return;
  const int w = F.w;
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.z;
  if (x >= w) return;
  if (F.mode[(y >> 3) * (w >> 3) + (x >> 3)] == DVC_SKIP_B) F.recon[y * w + x] = F.past[y * w + x];
}

// ------------------------------------------- transforms and noise parameters

// forwardTransform (transform.cpp:153-190) of the residue, every 4x4 block
__global__ void residue_transform_kernel(FrameDev *frames) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active) return;
  const int w = F.w, b4w = w / 4, b4n = b4w * (F.h / 4);
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= b4n) return;
  const int i = k / b4w, j = k % b4w;
  int b[16];
  for (int m = 0; m < 4; m++)
    for (int n = 0; n < 4; n++) b[4 * m + n] = F.residue[(4 * i + m) * w + 4 * j + n];
  forward44(b);
  for (int m = 0; m < 4; m++)
    for (int n = 0; n < 4; n++) F.side_trans[(4 * i + m) * w + 4 * j + n] = b[4 * m + n];
}

// noiseParameter, noiseModel.cpp:14-45: band mean and variance of |T| over
// every 4x4 block.  The variance accumulates squares past 2^24, so each band's
// sums run sequentially in raster block order, one lane of warp 0 per band.
// What bounds it: that chain, two dependent additions per block side by side
// (6336 blocks at CIF).  The other warps bring the next 4 block rows of
// coefficients into the second half of a double buffer meanwhile, and the
// lanes read eight blocks ahead of their additions: 254 -> 49 us a CIF frame.
// A row is padded by four words so that the 16 lanes (4 x 4 positions of a
// block) read 16 banks.
__global__ void __launch_bounds__(512) noise_band_stats_kernel(FrameDev *frames) {
  FrameDev &F = frames[blockIdx.x];
  if (!F.active) return;
  constexpr int RB = 4, ST = 352 + 4;  // block rows per chunk, words per row
  __shared__ int chunk[2][RB * 4][ST];
  const int band = threadIdx.x;
  const int index = c_zigzag[band & 15];
  // bands are coded while Qbits > 0 in zig-zag order; later ones are unused
  bool active = band < 16;
  for (int b = 0; active && b <= band; b++) active = F.qbits[c_zigzag[b]] > 0;
  const int w = F.w, b4w = w / 4, b4h = F.h / 4, b4n = b4w * b4h;  // b4w is a multiple of 4
  auto load = [&](int i0, int t, int nt) {
    const int rows = min(RB, b4h - i0) * 4, w4 = w >> 2;
    int4(*dst)[ST / 4] = reinterpret_cast<int4(*)[ST / 4]>(chunk[(i0 / RB) & 1]);
    const int4 *src = reinterpret_cast<const int4 *>(F.side_trans + (size_t)4 * i0 * w);
    for (int k = t; k < rows * w4; k += nt) {
      const int r = k / w4;
      dst[r][k - r * w4] = src[k];
    }
  };
  float mean = 0.0f, var = 0.0f;
  load(0, threadIdx.x, blockDim.x);
  for (int i0 = 0; i0 < b4h; i0 += RB) {
    __syncthreads();
    if (threadIdx.x >= 32) {
      if (i0 + RB < b4h) load(i0 + RB, threadIdx.x - 32, blockDim.x - 32);
    } else if (active) {
      for (int i = 0; i < RB && i0 + i < b4h; i++) {
        const int *row = chunk[(i0 / RB) & 1][4 * i + (index >> 2)] + (index & 3);
        int j = 0;
        for (; j + 8 <= b4w; j += 8) {
          float c[8];
#pragma unroll
          for (int q = 0; q < 8; q++) c[q] = fabsf((float)row[4 * (j + q)]);
#pragma unroll
          for (int q = 0; q < 8; q++) {
            mean += c[q];
            var += c[q] * c[q];
          }
        }
        for (; j < b4w; j++) {
          const float c = fabsf((float)row[4 * j]);
          mean += c;
          var += c * c;
        }
      }
    }
  }
  if (!active) return;
  mean /= (float)b4n;
  var = var / (float)b4n - mean * mean;
  F.band_mean[band] = mean;
  F.band_var[band] = var;
}

// noiseParameter, noiseModel.cpp:47-73: alpha per WZ coefficient of coded bands
__global__ void noise_alpha_kernel(FrameDev *frames) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active) return;
  const int w = F.w, b4w = w / 4, b4n = b4w * (F.h / 4);
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= b4n) return;
  const int i = k / b4w, j = k % b4w;
  if (F.mode[(i >> 1) * (w >> 3) + (j >> 1)] != DVC_WZ_B) return;
  int band = 0, index = c_zigzag[0];
  while (band < 16 && F.qbits[index] > 0) {
    const int ci = (4 * i + (index >> 2)) * w + 4 * j + (index & 3);
    const float t = fabsf((float)F.side_trans[ci]);  // the reference stores |T| back first
    const float d = (float)(int)t - F.band_mean[band];
    const float d2 = d * d;
    F.alpha[ci] = d2 > F.band_var[band] ? sqrtf(2 / d2) : sqrtf(2 / F.band_var[band]);
    band++;
    if (band < 16) index = c_zigzag[band];
  }
}

// overCompleteTransform, transform.cpp:275-298: the 4x4 transform of the side
// information at every pixel offset (values fit 16 bits)
__global__ void over_complete_kernel(FrameDev *frames, int band) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active || !in_step(F, band, 0)) return;
  const int w = F.w, srw = w - 3;
  const int left = blockIdx.x * blockDim.x + threadIdx.x, top = blockIdx.z;
  if (left >= srw) return;
  int b[16];
  for (int m = 0; m < 4; m++)
    for (int n = 0; n < 4; n++) b[4 * m + n] = F.si[(top + m) * w + left + n];
  forward44(b);
  int16_t *o = F.oct + ((size_t)top * srw + left) * 16;
#pragma unroll
  for (int c = 0; c < 16; c += 2) {
    const uint32_t pk = (uint32_t)(uint16_t)(int16_t)b[c] | ((uint32_t)(uint16_t)(int16_t)b[c + 1] << 16);
    reinterpret_cast<uint32_t *>(o)[c >> 1] = pk;
  }
}

// init_si_ML, motionLearning.cpp:49-68 (every block), and initSMF (:6-47) for WZ blocks
__global__ void init_ml_kernel(FrameDev *frames) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active) return;
  const int w = F.w, h = F.h, b4w = w / 4, b4n = b4w * (h / 4), srw = w - 3;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= b4n) return;
  const int i = k / b4w, j = k % b4w;
  const int16_t *t = F.oct + ((size_t)(4 * i) * srw + 4 * j) * 16;
  for (int m = 0; m < 4; m++)
    for (int n = 0; n < 4; n++) F.side_trans[(4 * i + m) * w + 4 * j + n] = t[4 * m + n];
  const int s = F.sir_of_blk[k];
  if (s < 0) return;
  const int top = 4 * i, left = 4 * j;
  int st = top - LEARN_R, sb = top + LEARN_R, sl = left - LEARN_R, sr = left + LEARN_R;
  if (st < 0) st = 0;
  if (sb > h - 4) sb = h - 4;
  if (sl < 0) sl = 0;
  if (sr > w - 4) sr = w - 4;
  float *p = F.smf + (size_t)s * ML_N;
  int q = 0;
  for (int m = st; m <= sb; m++)
    for (int n = sl; n <= sr; n++) p[q++] = (m == top && n == left) ? 1.0f : 0.0f;
}

// SMF window of a WZ block (initSMF bounds, motionLearning.cpp:16-27)
struct Win {
  int st, sb, sl, sr;
};
__device__ __forceinline__ Win ml_window(int top, int left, int w, int h) {
  Win r{top - LEARN_R, top + LEARN_R, left - LEARN_R, left + LEARN_R};
  if (r.st < 0) r.st = 0;
  if (r.sb > h - 4) r.sb = h - 4;
  if (r.sl < 0) r.sl = 0;
  if (r.sr > w - 4) r.sr = w - 4;
  return r;
}

// ------------------------------------------------------ correlation noise

// noiseDistribution, noiseModel.cpp:77-132: per WZ block, the (mixture of)
// Laplacian pdf over every coefficient value of the band.  The exponential
// depends only on the integer distance d = |k - range - s_m|, so each block
// first tabulates expf(-alpha*d) (the same float expression) for every d it
// needs, then sums the 81-candidate mixture in the reference's order.
#define NOISE_TAB 2048

// The mixture for up to four values of one lane, k0 + c * 32 * NW (c < NC):
// one table address per candidate serves all of them through immediate
// offsets.  Each value's sum still runs over the candidates in order.
template <int NC, int NW>
__device__ __forceinline__ void noise_mix(const float *e0, const int4 *sc4, const float4 *pr4, int nm4, float *out,
                                          int k0, int rmax) {
  float s[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) s[c] = 0.0f;
  for (int m4 = 0; m4 < nm4; m4++) {
    const int4 v = sc4[m4];
    const float4 p = pr4[m4];
    const float *ax = e0 - v.x, *ay = e0 - v.y, *az = e0 - v.z, *aw = e0 - v.w;
#pragma unroll
    for (int c = 0; c < NC; c++) s[c] += p.x * ax[c * 32 * NW];
#pragma unroll
    for (int c = 0; c < NC; c++) s[c] += p.y * ay[c * 32 * NW];
#pragma unroll
    for (int c = 0; c < NC; c++) s[c] += p.z * az[c * 32 * NW];
#pragma unroll
    for (int c = 0; c < NC; c++) s[c] += p.w * aw[c * 32 * NW];
  }
#pragma unroll
  for (int c = 0; c < NC; c++)
    if (k0 + c * 32 * NW < rmax) out[k0 + c * 32 * NW] = s[c];
}

template <int NT>
__global__ void __launch_bounds__(NT) noise_dist_kernel(FrameDev *frames, XlmDev xt, int band) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active || !in_step(F, band, 0)) return;
  const int s_idx = blockIdx.x;
  if (s_idx >= F.nsir) return;
  const int w = F.w, h = F.h, b4w = w / 4, srw = w - 3;
  const int index = c_zigzag[band];
  const int range = F.crange[index];
  const int blk = F.sir[s_idx];
  const int top = (blk / b4w) << 2, left = (blk % b4w) << 2;
  constexpr int ML_N4 = (ML_N + 3) & ~3;
  __shared__ float etab[NOISE_TAB];
  __shared__ __align__(16) float prob[ML_N4];
  __shared__ __align__(16) int sc[ML_N4];
  __shared__ int s_n, s_dmax;
  const XlSmall xs = xl_small_global(xt);
  float *out = F.pdf + (size_t)s_idx * F.pdf_stride;
  if (index == 0) {
    const float a = F.alpha[top * w + left];
    const int s = F.oct[((size_t)top * srw + left) * 16];
    for (int k = threadIdx.x; k < range; k += NT) out[k] = xl_expf(xt, xs, -a * (float)abs(k - s));
    return;
  }
  const float a = F.alpha[(top + (index >> 2)) * w + left + (index & 3)];
  // the SMF candidates in row-major window order, gathered in parallel
  const Win wn = ml_window(top, left, w, h);
  const int cw = wn.sr - wn.sl + 1, ncand = cw * (wn.sb - wn.st + 1);
  if (threadIdx.x == 0) s_dmax = 0;
  __syncthreads();
  int mx = 0;
  for (int q = threadIdx.x; q < ncand; q += NT) {
    const int m = wn.st + q / cw, n = wn.sl + q % cw;
    const int v = F.oct[((size_t)m * srw + n) * 16 + index];
    sc[q] = v;
    prob[q] = F.smf[(size_t)s_idx * ML_N + q];
    mx = max(mx, abs(v));
  }
  // pad to a multiple of 4 with zero-probability terms: they add +0 to a
  // non-negative sum, which leaves it unchanged
  for (int q = ncand + threadIdx.x; q < ((ncand + 3) & ~3); q += NT) {
    sc[q] = 0;
    prob[q] = 0.0f;
  }
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) atomicMax(&s_dmax, mx);
  if (threadIdx.x == 0) s_n = ncand;
  __syncthreads();
  if (threadIdx.x == 0) s_dmax += range;
  __syncthreads();
  const int nm = s_n, dmax = s_dmax;
  const int rmax = 2 * range + 1;
  if (dmax < NOISE_TAB / 2 - 32) {
    // a symmetric table, etab[ETC + d] = etab[ETC - d] = expf(-a*d), read at
    // pc - v directly: one address per term, no absolute value.  Values are
    // taken in groups of 32 (one per lane); warp w takes groups w, w + NW, ...,
    // up to four per pass.  The last group of a block reads up to 31 entries
    // past dmax for values past rmax, which are not stored: those entries
    // hold 0.
    constexpr int ETC = NOISE_TAB / 2 - 1;
    constexpr int NW = NT / 32;
    for (int d = threadIdx.x; d <= dmax + 31; d += NT) {
      if (d <= dmax) {
        const float e = xl_expf(xt, xs, -a * (float)d);
        etab[ETC + d] = e;
        etab[ETC - d] = e;
      } else {
        etab[ETC + d] = 0.0f;
      }
    }
    __syncthreads();
    const int nm4 = (nm + 3) >> 2;
    const int4 *sc4 = reinterpret_cast<const int4 *>(sc);
    const float4 *pr4 = reinterpret_cast<const float4 *>(prob);
    const int lane = threadIdx.x & 31, groups = (rmax + 31) >> 5;
    for (int g = threadIdx.x >> 5; g < groups; g += 4 * NW) {
      const int k0 = g * 32 + lane, nc = min(4, (groups - g + NW - 1) / NW);
      const float *e0 = etab + ETC + (k0 - range);
      if (nc == 4)
        noise_mix<4, NW>(e0, sc4, pr4, nm4, out, k0, rmax);
      else if (nc == 3)
        noise_mix<3, NW>(e0, sc4, pr4, nm4, out, k0, rmax);
      else if (nc == 2)
        noise_mix<2, NW>(e0, sc4, pr4, nm4, out, k0, rmax);
      else
        noise_mix<1, NW>(e0, sc4, pr4, nm4, out, k0, rmax);
    }
    return;
  }
  const int tab = dmax < NOISE_TAB ? dmax + 1 : NOISE_TAB;
  for (int d = threadIdx.x; d < tab; d += NT) etab[d] = xl_expf(xt, xs, -a * (float)d);
  __syncthreads();
  if (dmax < NOISE_TAB) {
    // every distance is in the table: candidates four at a time, in order
    const int nm4 = (nm + 3) >> 2;
    const int4 *sc4 = reinterpret_cast<const int4 *>(sc);
    const float4 *pr4 = reinterpret_cast<const float4 *>(prob);
    for (int k = threadIdx.x; k < rmax; k += NT) {
      const int pc = k - range;
      float sum = 0.0f;
      for (int m4 = 0; m4 < nm4; m4++) {
        const int4 v = sc4[m4];
        const float4 p = pr4[m4];
        sum += p.x * etab[abs(pc - v.x)];
        sum += p.y * etab[abs(pc - v.y)];
        sum += p.z * etab[abs(pc - v.z)];
        sum += p.w * etab[abs(pc - v.w)];
      }
      out[k] = sum;
    }
    return;
  }
  for (int k = threadIdx.x; k < rmax; k += NT) {
    const int pc = k - range;
    float sum = 0.0f;
    for (int m = 0; m < nm; m++) {
      const int d = abs(pc - sc[m]);
      const float e = d < NOISE_TAB ? etab[d] : xl_expf(xt, xs, -a * (float)d);
      sum += prob[m] * e;
    }
    out[k] = sum;
  }
}

// p[lo..hi) summed in ascending order (a float sum of condBitProb).  Each lane
// walks its own row, so the reads wait on memory: once aligned they are 16 bytes
// each, and up to eight are in flight before their additions.
__device__ __forceinline__ float interval_sum(const float *p, int lo, int hi) {
  float a = 0.0f;
  int q = lo;
  for (; q < hi && (reinterpret_cast<uintptr_t>(p + q) & 15); q++) a += __ldg(p + q);
  constexpr int U = 8;
  for (; q + 4 <= hi; q = min(q + 4 * U, q + ((hi - q) & ~3))) {
    float4 u[U];
    // past the last whole quad +0 is added to a sum that is not negative
#pragma unroll
    for (int i = 0; i < U; i++)
      u[i] = q + 4 * i + 4 <= hi ? __ldg(reinterpret_cast<const float4 *>(p + q) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < U; i++) {
      a += u[i].x;
      a += u[i].y;
      a += u[i].z;
      a += u[i].w;
    }
  }
  for (; q < hi; q++) a += __ldg(p + q);
  return a;
}

// condBitProb, noiseModel.cpp:191-310: LR = p0/p1 from sequential interval
// sums of the pdf.  Non-WZ blocks get the reference's certain-zero ratio when
// the frame has skip or intra blocks.  Beside each ratio go its logarithm and
// its term of the entropy bound, which every speculative block of the ladder
// would otherwise compute again.  The two sums are latency-bound chains, so two
// lanes take a 4x4 block: the even one sums p0 and writes the ratio and its
// logarithm, the odd one sums p1 and writes the entropy term.  Blocks of 64
// threads, so that the rows of one CIF frame (6336) spread over all SMs.
// With a thread for both sums, four quads of each in flight, and blocks of 128
// threads (50 of 148 SMs for a lone CIF frame) 20.7 us a step, now 18.2; sixteen
// CIF frames 26.2 -> 20.5.
__global__ void __launch_bounds__(64) cond_bit_kernel(FrameDev *frames, XlmDev xt, int band, int bit) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active || !in_step(F, band, bit)) return;
  const int w = F.w, b4w = w / 4, b4n = b4w * (F.h / 4);
  const int t = blockIdx.x * blockDim.x + threadIdx.x, k = t >> 1, odd = t & 1;
  const int s_idx = k < b4n ? F.sir_of_blk[k] : -1;
  float sum = 0.0f;
  if (s_idx >= 0) {
    const int index = c_zigzag[band], step = F.step[index], range = F.crange[index];
    const int i = k / b4w, j = k % b4w;
    const int rc = F.recons_trans[(4 * i + (index >> 2)) * w + 4 * j + (index & 3)];
    const float *p = F.pdf + (size_t)s_idx * F.pdf_stride;
    const int iq = (1 << (bit - 1)) - 1;
    // interval ends are clamped to the pdf row; consistent bitstreams never reach the clamp
    if (index == 0) {
      const int bl = odd ? ((rc << 1) + 1) << (bit - 1) : rc << bit, bu = bl + iq;
      sum = interval_sum(p, max(bl * step, 0), min((bu + 1) * step, range));
    } else {
      const int ls = F.level_shift[index];
      const int bl = (odd ? ((rc << 1) + 1) << (bit - 1) : rc << bit) - ls;
      int bu = bl + iq;
      if (odd && bu > ls) bu = ls;
      const int vl = (bl <= 0) ? (bl - 1) * step + 1 : bl * step;
      const int vu = ((bu < 0) ? bu * step + 1 : (bu + 1) * step) + range;
      sum = interval_sum(p, max(vl + range, 0), min(vu, 2 * range + 1));
    }
  }
  const float other = __shfl_xor_sync(0xffffffffu, sum, 1);
  if (k >= b4n) return;
  const XlSmall xs = xl_small_global(xt);
  float lr;
  if (s_idx < 0) {
    lr = F.skip_mode == 1 || F.intra_mode == 1 ? 0.9999f / 0.0001f : F.lr[k];
  } else {
    float p0 = odd ? other : sum, p1 = odd ? sum : other;
    p0 = p0 / (p0 + p1);
    p1 = 1 - p0;
    if (p0 <= 0.0001)
      lr = (float)(0.0001 / 0.9999);
    else if (p0 >= 0.9999)
      lr = (float)(0.9999 / 0.0001);
    else
      lr = p0 / p1;
  }
  if (odd) {
    F.term[k] = ld_entropy_term(lr, xt, xs);
  } else {
    F.lr[k] = lr;
    F.llr[k] = xl_logf(xt, xs, lr);
  }
}

// ------------------------------------------------------- reconstruction

// reconstruction (reconstruction.cpp:184-289) of the band's coefficient, then
// inverseTransform (transform.cpp:234-273) of the block; one thread per WZ block
__global__ void recon_kernel(FrameDev *frames, int band) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active || !in_step(F, band, 0)) return;
  const int s_idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (s_idx >= F.nsir) return;
  const int w = F.w, b4w = w / 4;
  const int blk = F.sir[s_idx];
  const int top = (blk / b4w) << 2, left = (blk % b4w) << 2;
  if (band >= 0) {
    const int index = c_zigzag[band], step = F.step[index];
    const int ci = (top + (index >> 2)) * w + left + (index & 3);
    int lo, hi;
    if (index == 0) {
      const int q = F.recons_trans[ci];
      lo = q * step;
      hi = (q + 1) * step;
    } else {
      const int q = F.recons_trans[ci] - F.level_shift[index];
      if (q == 0) {
        lo = -step + 1;
        hi = step;
      } else if (q > 0) {
        lo = q * step;
        hi = (q + 1) * step;
      } else {
        lo = (q - 1) * step + 1;
        hi = q * step + 1;
      }
    }
    const int sc = F.side_trans[ci];
    const double a = F.alpha[ci];
    int v;
    // The reference rounds with its C library's double exp; this kernel uses
    // the device's.  Both are within an ulp of the true value, and every other
    // operation here is IEEE and identical on both sides, so the rounded result
    // can only differ where moving an exp result by a couple of ulps moves the
    // argument of ROUND across a .5 boundary.  Such steps are counted (every
    // exp result moved by -2 and +2 ulps), so a decode can show that it met none.
    bool tie = false;
    if (a <= 0.0001) {
      v = (lo + hi) / 2;
    } else if (sc < lo || sc >= hi) {
      const double e = exp(a * (double)step);
      const int u = dround(1.0 / a + (double)step / (1.0 - e));
      for (int k = -2; k <= 2 && F.near_ties; k += 4)
        tie |= dround(1.0 / a + (double)step / (1.0 - ulp_shift(e, k))) != u;
      v = sc < lo ? lo + u : hi - u;
    } else {
      const double r = sc - lo, d = hi - sc;
      const double er = exp(-a * r), ed = exp(-a * d);
      const int u = dround(((r + 1.0 / a) * er - (d + 1.0 / a) * ed) / (2.0 - (er + ed)));
      for (int k = 0; k < 4 && F.near_ties; k++) {
        const double er2 = ulp_shift(er, (k & 1) ? 2 : -2), ed2 = ulp_shift(ed, (k & 2) ? 2 : -2);
        tie |= dround(((r + 1.0 / a) * er2 - (d + 1.0 / a) * ed2) / (2.0 - (er2 + ed2))) != u;
      }
      v = sc + u;
    }
    if (tie) atomicAdd(F.near_ties, 1ull);
    F.side_trans[ci] = v;
    F.dbf[ci] = ((v ^ sc) != 0) ? 1 : 0;
  }
  int b[16];
  for (int m = 0; m < 4; m++)
    for (int n = 0; n < 4; n++) b[4 * m + n] = F.side_trans[(top + m) * w + left + n];
  inverse44(b);
  for (int m = 0; m < 4; m++)
    for (int n = 0; n < 4; n++) {
      const int c = b[4 * m + n];
      F.recon[(top + m) * w + left + n] = (uint8_t)(c < 0 ? 0 : (c > 255 ? 255 : c));
    }
}

// -------------------------------------------------- side-info refinement

// sum of the four byte differences |a_i - b_i| plus c
__device__ __forceinline__ uint32_t sad4_acc(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// updateSI + subPelRefine, sideInfoCreation.cpp:598-736: per WZ block, +-32
// integer search against the past and future reconstructions (cost = SAD with
// the motion-vector weight; strict-< row-major argmin), a +-1 half-pel
// refinement in the interpolated frames, and the bidirectional average.
//
// One thread block takes a 16x16 tile of a frame, whose (up to) 16 WZ blocks
// search nearly the same 80x80 pixels of either reference; a warp takes a
// block.  Forming every SAD is bound by instruction issue, so candidates are ruled
// out eight to a lane and step before their SADs are formed: the tile's window holds,
// for every position, the floored means of the four 2x2 quadrants of the 4x4
// block there, one word.  With d the sum of the four mean differences (one
// packed instruction), SAD >= 4 d - 12; the weight of a candidate is at least
// 1 + 0.1 max(|dx|, |dy|); so one whose bound exceeds the best cost so far can
// neither win nor tie.  0.5 to 2% of the candidates are left once the best is
// near its final value, and it starts from the zero-motion candidate and the
// previous band's best.  Those left are queued per warp (by groups of eight
// columns) and weighed 32 at a time; the (cost, index) order makes the result
// independent of the order in which candidates are weighed.
// What bounds it now is shared memory: with many tiles in flight (65 QCIF frames)
// L1 runs at 88% of its peak and 58% of the issue slots are used; a lone CIF
// frame's 396 tiles are 0.9 of a wave and take as long as the last of them.
// All SADs of a block by packed instructions took 93 us for a band of two CIF
// frames (40 M warp instructions a frame) and 70 us for a lone one; so 72 and 43
// us (20 M) with 256 threads, two blocks to a warp and three thread blocks an
// SM, 74 and 50 us with 512 threads (two an SM: a frame's 396 tiles need a
// second wave; held to 40 registers for three, 99 and 61 us).
constexpr int kSiTile = 16;                  // pixels a side
constexpr int kSiRows = kSiTile + 2 * 32;    // pixel rows of the window
constexpr int kSiStride = 96;                // bytes of a pixel row: 80, and the word after any 4-byte group
constexpr int kSiMeanStride = 84;            // bytes of a row of 2x2 means
constexpr int kSiQuadStride = 80;            // words of a row of quadrant means
constexpr int kSiQueue = 36;                 // groups waiting in a warp: fewer than 4, and the 32 of a step

struct SiShared {
  uint32_t quad[2][(kSiRows - 3) * kSiQuadStride];
  uint8_t px[2][kSiRows * kSiStride];
  uint8_t mean[(kSiRows - 1) * kSiMeanStride + 4];
  uint16_t queue[16][kSiQueue];
  uint16_t most[16][SEARCH_R + 4];  // by max(|dx|, |dy|): largest d that is weighed
};

template <int NT>
__global__ void __launch_bounds__(NT, NT == 512 ? 2 : 3) update_si_kernel(FrameDev *frames, int band) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active || !in_step(F, band, 0)) return;
  constexpr int NW = NT / 32, BPW = 16 / NW;  // warps, WZ blocks per warp
  const int w = F.w, h = F.h, b4w = w / 4, w2 = w << 1, h2 = h << 1;
  const int tpr = w / kSiTile, ty = (int)blockIdx.x / tpr * kSiTile, tx = (int)blockIdx.x % tpr * kSiTile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // WZ list positions of the tile's blocks, in the lanes of every warp
  const int mine = lane < 16 ? F.sir_of_blk[((ty >> 2) + (lane >> 2)) * b4w + (tx >> 2) + (lane & 3)] : -1;
  if (__ballot_sync(0xffffffffu, mine >= 0) == 0) return;
  extern __shared__ __align__(16) uint8_t si_smem[];
  SiShared &S = *reinterpret_cast<SiShared *>(si_smem);
  // the window: rows and columns [r0, r1) x [c0, c1) of both references, in
  // 16-byte chunks (the tile, the frame and the planes' bases are multiples of 16)
  const int r0 = max(0, ty - SEARCH_R), r1 = min(h, ty + kSiTile + SEARCH_R);
  const int c0 = max(0, tx - SEARCH_R), c1 = min(w, tx + kSiTile + SEARCH_R);
  const int rows = r1 - r0;
  {
    const int ch = (int)threadIdx.x % 5;
    for (int y = (int)threadIdx.x / 5; y < rows; y += NT / 5) {
      if (16 * ch >= c1 - c0 || (int)threadIdx.x >= NT / 5 * 5) continue;
#pragma unroll
      for (int ref = 0; ref < 2; ref++) {
        const uint8_t *src = (ref ? F.future : F.past) + (size_t)(r0 + y) * w + c0 + 16 * ch;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(S.px[ref] + y * kSiStride + 16 * ch);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  // the thread's column (four pixels) and run of rows when the means are made
  constexpr int RUN = (kSiRows + NT / 20 - 1) / (NT / 20);
  const int by_ = (int)threadIdx.x / 20 * RUN, bx_ = by_ < kSiRows ? (int)threadIdx.x % 20 : 20, mcols = (c1 - c0) >> 2;
  const float inv_w = 1.0001f / (1.0f + 0.1f * (float)lane);  // over the weight of a candidate lane away, rounded up
#pragma unroll
  for (int ref = 0; ref < 2; ref++) {
    __syncthreads();
    // means of 2x2 pixels at every position, four to a word, a run of rows per
    // thread: the pair sums of a row serve the means above and below it
    if (bx_ < mcols) {
      constexpr uint32_t M = 0x00ff00ffu;
      const uint32_t *p = reinterpret_cast<const uint32_t *>(S.px[ref]) + by_ * (kSiStride / 4) + bx_;
      uint32_t *o = reinterpret_cast<uint32_t *>(S.mean) + by_ * (kSiMeanStride / 4) + bx_;
      uint32_t even = 0, odd = 0;
#pragma unroll
      for (int i = 0; i <= RUN; i++) {
        if (by_ + i < rows) {
          const uint32_t v = p[i * (kSiStride / 4)], u = __funnelshift_r(v, p[i * (kSiStride / 4) + 1], 8);
          const uint32_t e = (v & M) + (u & M), d = ((v >> 8) & M) + ((u >> 8) & M);
          if (i > 0) o[(i - 1) * (kSiMeanStride / 4)] = (((even + e) >> 2) & M) | ((((odd + d) >> 2) & M) << 8);
          even = e;
          odd = d;
        }
      }
    }
    __syncthreads();
    // the four quadrants' means of the block at every position, one word each
    if (bx_ < mcols) {
      const uint32_t *m = reinterpret_cast<const uint32_t *>(S.mean) + by_ * (kSiMeanStride / 4) + bx_;
      uint4 *o = reinterpret_cast<uint4 *>(S.quad[ref] + by_ * kSiQuadStride) + bx_;
      uint32_t h0[RUN + 2], h1[RUN + 2];  // left and right means of a row's positions, side by side
#pragma unroll
      for (int i = 0; i < RUN + 2; i++) {
        if (by_ + i < rows - 1) {
          const uint32_t l = m[i * (kSiMeanStride / 4)], r = __funnelshift_r(l, m[i * (kSiMeanStride / 4) + 1], 16);
          h0[i] = __byte_perm(l, r, 0x5140);
          h1[i] = __byte_perm(l, r, 0x7362);
          if (i >= 2)
            o[(i - 2) * (kSiQuadStride / 4)] =
                make_uint4(__byte_perm(h0[i - 2], h0[i], 0x5410), __byte_perm(h0[i - 2], h0[i], 0x7632),
                           __byte_perm(h1[i - 2], h1[i], 0x5410), __byte_perm(h1[i - 2], h1[i], 0x7632));
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int bw = 0; bw < BPW; bw++) {
    const int blk = warp + bw * NW, s_idx = __shfl_sync(0xffffffffu, mine, blk);
    if (s_idx < 0) continue;
    const int top = ty + (blk >> 2) * 4, left = tx + (blk & 3) * 4;
    const int st = max(0, top - SEARCH_R), sb = min(h - 4, top + SEARCH_R);
    const int sl = max(0, left - SEARCH_R), sr = min(w - 4, left + SEARCH_R);
    const int cw = sr - sl + 1, nrow = sb - st + 1;  // cw is one more than a multiple of 4
    const int y0 = top - st, x0 = left - sl;         // zero motion; x0 is a multiple of 4
    const double *wt = d_si_weight + (SEARCH_R - y0) * 65 + SEARCH_R - x0;
    uint16_t *most = S.most[warp], *queue = S.queue[warp];
    uint32_t cur[4], cq = 0;
#pragma unroll
    for (int m = 0; m < 4; m++) cur[m] = *reinterpret_cast<const uint32_t *>(F.recon + (size_t)(top + m) * w + left);
#pragma unroll
    for (int m = 0; m < 2; m++) {
      constexpr uint32_t M = 0x00ff00ffu;
      const uint32_t v = (cur[2 * m] & M) + ((cur[2 * m] >> 8) & M) + (cur[2 * m + 1] & M) + ((cur[2 * m + 1] >> 8) & M);
      cq |= ((v & 0xffffu) >> 2 | (v >> 18) << 8) << (16 * m);
    }
    // a candidate is row << 8 | column of the block's window, in the scan's order
    const int zero = y0 << 8 | x0, last = lane < 2 ? F.si_mv[2 * s_idx + lane] : -1;
    int found[2];
#pragma unroll
    for (int ref = 0; ref < 2; ref++) {
      const uint32_t *px = reinterpret_cast<const uint32_t *>(S.px[ref]) + (st - r0) * (kSiStride / 4) + ((sl - c0) >> 2);
      const uint32_t *quad = S.quad[ref] + (st - r0) * kSiQuadStride + (sl - c0);
      // SAD of the candidate in row r, column x
      auto sad_at = [&](int r, int x) {
        const uint32_t *p = px + r * (kSiStride / 4) + (x >> 2);
        const int sh = (x & 3) * 8;
        uint32_t sad = 0;
#pragma unroll
        for (int m = 0; m < 4; m++, p += kSiStride / 4) sad = sad4_acc(__funnelshift_r(p[0], p[1], sh), cur[m], sad);
        return sad;
      };
      // zero motion (lane 0) and the previous band's best (lane 1; -1 before the first band)
      double best;
      int bi = zero;
      {
        const int prev = __shfl_sync(0xffffffffu, last, ref), at = lane == 1 && prev >= 0 ? prev : zero;
        const int r = at >> 8, x = at & 255;
        const double c = (double)(int)sad_at(r, x) * __ldg(wt + r * 65 + x);
        best = __shfl_sync(0xffffffffu, c, 0);
        const double c1 = __shfl_sync(0xffffffffu, c, 1);
        if (prev >= 0) better(best, bi, c1, prev);
      }
      auto set_most = [&]() {
        __syncwarp();
        const float b = (float)best;
        most[lane] = (uint16_t)(((int)(b * inv_w) + 1 + 12) >> 2);
        if (lane < 2) most[SEARCH_R + lane] = (uint16_t)(((int)(b * (1.0001f / 4.2f)) + 1 + 12) >> 2);
        __syncwarp();
      };
      set_most();
      int cnt = 0;
      // weigh the last n (at most 4) groups of the queue, a lane per candidate
      auto weigh = [&](int n) {
        __syncwarp();
        cnt -= n;
        const int e = queue[cnt + min(lane >> 3, n - 1)], r = e >> 4, x = min(8 * (e & 15) + (lane & 7), cw - 1);
        // d <= most means SAD <= 4 most - 9 for the same distance: most groups end here
        const uint32_t sad = sad_at(r, x);
        const bool near = (int)sad <= 4 * (int)most[max(abs(x - x0), abs(r - y0))] - 9;
        if (__any_sync(0xffffffffu, near)) {
          int i = r << 8 | x;
          double c = near ? (double)(int)sad * __ldg(wt + r * 65 + x) : 1e300;
          const bool win = c < best || (c == best && i < bi);
          if (__any_sync(0xffffffffu, win)) {
            if (!win) {
              c = 1e300;
              i = 0x7fffffff;
            }
            warp_argmin_nonneg(c, i);
            best = c;
            bi = i;
            set_most();
          }
        }
        __syncwarp();
      };
      // queue the groups (row r, group g) of the lanes that hit, weigh when there are 4
      auto add = [&](uint32_t hits, int entry) {
        if (hits >> lane & 1u) queue[cnt + __popc(hits & ((1u << lane) - 1u))] = (uint16_t)entry;
        cnt += __popc(hits);
        while (cnt >= 4) weigh(4);
      };
      // four rows a step, from the block's own row outwards; eight groups of
      // eight columns a row, a group per lane (a group past the window's
      // columns may hit: its candidates count as the last column's)
      const int g = lane & 7, down = (lane >> 3) & 1, odd = lane >> 4;
      const int dx = min(max(max(8 * g - x0, x0 - 8 * g - 7), 0), SEARCH_R);
      const int have = down ? nrow - 1 - y0 : y0 + 1;                 // rows on this lane's side
      const int mine_n = 8 * g < cw - 1 ? (have - odd + 1) >> 1 : 0;  // steps in which it has one
      const int r_0 = down ? y0 + 1 + odd : y0 - odd, r_s = down ? 2 : -2;
      const int steps = (max(y0 + 1, nrow - 1 - y0) + 1) >> 1;
      const uint32_t most_a = (uint32_t)__cvta_generic_to_shared(most) + 2 * (down + odd);
      const int stride = r_s * 4 * kSiQuadStride, dx2 = 2 * (dx - down - odd);
      // a lane without rows stays on the block's own row
      uint32_t qa = (uint32_t)__cvta_generic_to_shared(quad + 8 * g + (mine_n > 0 ? r_0 : y0) * kSiQuadStride);
      for (int s = 0; s < steps; s++) {
        uint32_t q0, q1, q2, q3, q4, q5, q6, q7, far;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(q0), "=r"(q1), "=r"(q2), "=r"(q3) : "r"(qa) : "memory");
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4 + 16];" : "=r"(q4), "=r"(q5), "=r"(q6), "=r"(q7) : "r"(qa) : "memory");
        asm volatile("{\n\t.reg .u16 t;\n\tld.shared.u16 t, [%1];\n\tcvt.u32.u16 %0, t;\n\t}" : "=r"(far) : "r"(most_a + max(dx2, 4 * s)) : "memory");
        const uint32_t a = __vimin3_u32(sad4_acc(q0, cq, 0u), sad4_acc(q1, cq, 0u), sad4_acc(q2, cq, 0u));
        const uint32_t b = __vimin3_u32(sad4_acc(q3, cq, 0u), sad4_acc(q4, cq, 0u), sad4_acc(q5, cq, 0u));
        const uint32_t d = min(__vimin3_u32(sad4_acc(q6, cq, 0u), sad4_acc(q7, cq, 0u), a), b);
        const uint32_t hits = __ballot_sync(0xffffffffu, d <= far && s < mine_n);
        if (hits) add(hits, (r_0 + r_s * s) << 4 | g);
        if (s + 1 < mine_n) qa += stride;
      }
      for (int rr = 0; rr < nrow; rr += 32) {  // the last column
        const int r = min(rr + lane, nrow - 1);
        const uint32_t d = sad4_acc(quad[r * kSiQuadStride + cw - 1], cq, 0u);
        const uint32_t hits = __ballot_sync(0xffffffffu, d <= most[max(cw - 1 - x0, abs(r - y0))] && rr + lane < nrow);
        if (hits) add(hits, r << 4 | (cw - 1) >> 3);
      }
      while (cnt > 0) weigh(min(cnt, 4));
      found[ref] = bi;
    }
    if (lane < 2) F.si_mv[2 * s_idx + lane] = lane ? found[1] : found[0];
    // subPelRefine in the half-pel planes, no vector weight
    // (sideInfoCreation.cpp:598-640): one lane per (reference, offset) SAD,
    // then the strict-< scan over the offsets in the reference's (di, dj) order
    const int which = lane >= 9, k = lane - 9 * which, mv = which ? found[1] : found[0];
    int sad = 0x7fffffff;  // offset outside the half-pel plane: not a candidate
    if (lane < 18) {
      const int tt = ((st + (mv >> 8)) << 1) + k / 3 - 1, ll = ((sl + (mv & 255)) << 1) + k % 3 - 1;
      if (tt >= 0 && tt <= h2 - 8 && ll >= 0 && ll <= w2 - 8) {
        const uint8_t *p = (which ? F.future_ip : F.past_ip) + tt * w2 + ll;
        sad = 0;
#pragma unroll
        for (int m = 0; m < 4; m++)
#pragma unroll
          for (int n = 0; n < 4; n++) sad += abs((int)(cur[m] >> (8 * n) & 255u) - (int)__ldg(p + 2 * m * w2 + 2 * n));
      }
    }
    int off[2];  // first offset with the lowest SAD, or 9: none (the integer position, as the reference leaves it)
#pragma unroll
    for (int ref = 0; ref < 2; ref++) {
      const int v = (lane >= 9 * ref && lane < 9 * ref + 9) ? sad : 0x7fffffff;
      const int least = __reduce_min_sync(0xffffffffu, v);
      off[ref] = least == 0x7fffffff ? 9 : __ffs(__ballot_sync(0xffffffffu, v == least)) - 1 - 9 * ref;
    }
    if (lane < 16) {
      const int m = lane >> 2, n = lane & 3;
      double v[2];
#pragma unroll
      for (int ref = 0; ref < 2; ref++) {
        const int y = st + (found[ref] >> 8), x = sl + (found[ref] & 255), o = off[ref];
        const int yy = o < 9 ? (y << 1) + o / 3 - 1 : y, xx = o < 9 ? (x << 1) + o % 3 - 1 : x;
        v[ref] = (double)(ref ? F.future_ip : F.past_ip)[(yy + 2 * m) * w2 + xx + 2 * n];
      }
      F.si[(top + m) * w + left + n] = (uint8_t)(int)(v[0] * F.ipc + v[1] * F.ifc);
    }
  }
}

// ------------------------------------------------------ motion learning

// bytes a[0..3], the first lowest, from the aligned words that hold them
__device__ __forceinline__ uint32_t load4_u8(const uint8_t *a) {
  const uintptr_t u = reinterpret_cast<uintptr_t>(a);
  const uint32_t *wp = reinterpret_cast<const uint32_t *>(u & ~(uintptr_t)3);
  const uint32_t sh = (uint32_t)(u & 3) * 8;
  const uint32_t lo = wp[0], hi = sh ? wp[1] : 0u;
  return __funnelshift_r(lo, hi, sh);
}

// updateSMF, motionLearning.cpp:70-127, and update_si_ML, :129-160: a block's
// candidate probabilities, and with them the ML side coefficients of the bands
// above `band`.  The block's float sum of squared pixel differences only ever
// holds integers below 2^24 (16 terms of at most 255^2), so every float step of
// it is exact and it equals the integer sum, taken here four pixels at a time
// (vabsdiffu4, dp4a).  Both sums run in candidate order, so a block is a chain
// of 81 adds and then one of 81 multiply-adds per coefficient; what bounds the
// kernel is their latency and the window loads'.  Sixteen lanes take a block: they
// share its candidates, three loads of a window in flight, all walk the (same)
// sum, and each then owns one coefficient, two rows of nine candidates in
// flight; the probabilities stay in shared memory between the two parts.  As two
// kernels of a warp a block and a thread a coefficient, with one load of a chain
// in flight, 16.7 + 18.4 us a band for one CIF frame; now 22.7 (eight lanes a
// block and a coefficient pair each: 28.7).
__global__ void __launch_bounds__(128) update_ml_kernel(FrameDev *frames, XlmDev xt, int band) {
  __shared__ float s_p[8][ML_N];  // ML_N is odd: the two blocks of a warp read two banks
  FrameDev &F = frames[blockIdx.y];
  if (!F.active || !in_step(F, band, 0)) return;
  const int lane = threadIdx.x & 15;
  const int s_idx = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
  const bool live = s_idx < F.nsir;
  const int w = F.w, h = F.h, b4w = w / 4, srw = w - 3;
  const int blk = live ? F.sir[s_idx] : 0;
  const int top = (blk / b4w) << 2, left = (blk % b4w) << 2;
  const Win wn = ml_window(top, left, w, h);
  const int cw = wn.sr - wn.sl + 1, nc = live ? cw * (wn.sb - wn.st + 1) : 0;
  const XlSmall xs = xl_small_global(xt);
  float *pr = s_p[threadIdx.x >> 4];
  if (live) {
    uint32_t cb[4];
#pragma unroll
    for (int ii = 0; ii < 4; ii++) cb[ii] = load4_u8(F.recon + (size_t)(top + ii) * w + left);
    // three rounds of loads in flight; past the last candidate it is read again
    const int inv = 65536 / cw + 1;  // q / cw for q < 81, cw < 10
    for (int q0 = lane; q0 < nc; q0 += 48) {
      uint32_t sse[3] = {0, 0, 0};
#pragma unroll
      for (int r = 0; r < 3; r++) {
        const int q = min(q0 + 16 * r, nc - 1), qm = (q * inv) >> 16;
        const uint8_t *c = F.si + (size_t)(wn.st + qm) * w + wn.sl + q - qm * cw;
#pragma unroll
        for (int ii = 0; ii < 4; ii++) {
          const uint32_t d = __vabsdiffu4(cb[ii], load4_u8(c + (size_t)ii * w));
          sse[r] = __dp4a(d, d, sse[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < 3; r++) {
        const float e = xl_expf(xt, xs, (float)-0.01f * (float)sse[r]);
        if (q0 + 16 * r < nc) pr[q0 + 16 * r] = e;
      }
    }
  }
  __syncwarp();
  float sum = 0.0f;
#pragma unroll 9
  for (int q = 0; q < nc; q++) sum += pr[q];
  __syncwarp();
  if (live) {
    const int center = (top - wn.st) * cw + left - wn.sl;
    float *p = F.smf + (size_t)s_idx * ML_N;
#pragma unroll 3
    for (int q = lane; q < nc; q += 16) {
      const float v = sum > 0.0 ? pr[q] / sum : (q == center ? 1.0f : pr[q]);
      pr[q] = v;
      p[q] = v;
    }
  }
  __syncwarp();
  bool want = false;  // the lane's raster position belongs to a band above `band`
  for (int c = band + 1; c < 16; c++) want |= c_zigzag[c] == lane;
  if (!live || !want) return;
  float acc = 0.0f;
  const int16_t *o = F.oct + lane;
#pragma unroll 2
  for (int m = wn.st; m <= wn.sb; m++, pr += cw) {
    const int16_t *row = o + ((size_t)m * srw + wn.sl) * 16;
    int v[2 * LEARN_R + 1];
#pragma unroll
    for (int j = 0; j <= 2 * LEARN_R; j++) v[j] = j < cw ? row[j * 16] : 0;
#pragma unroll
    for (int j = 0; j <= 2 * LEARN_R; j++)
      if (j < cw) acc += pr[j] * (float)v[j];
  }
  F.side_trans[(top + (lane >> 2)) * w + left + (lane & 3)] = (int)acc;
}

// ------------------------------------------------------------- launchers

// ------------------------------------------------------------ deblocking
//
// The reference's deblocking filter (DvcDec/src/deblock.cpp:346-386): every
// vertical 4x4 block edge in raster order, then every horizontal one, each
// filtered from a decision taken on the frame before filtering
// (deblock_44_decision, :228-344) with the strength and thresholds of the
// H.264 in-loop filter.  Decisions are independent, so one thread takes each
// edge; the filter of an edge touches up to three pixels on each side and
// only its own pixel lines, so one thread walks each pixel row (vertical
// edges) and then each pixel column (horizontal edges) in the reference's
// order.

// alpha, beta and tc0 by QP (H.264 tables 8-16 and 8-17; deblock.cpp:16-37)
__constant__ uint8_t c_db_alpha[52] = {0,  0,  0,  0,  0,  0,  0,  0,  0,   0,   0,   0,   0,   0,   0,   0,   4,   4,
                                       5,  6,  7,  8,  9,  10, 12, 13, 15,  17,  20,  22,  25,  28,  32,  36,  40,  45,
                                       50, 56, 63, 71, 80, 90, 101, 113, 127, 144, 162, 182, 203, 226, 255, 255};
__constant__ uint8_t c_db_beta[52] = {0, 0, 0, 0, 0, 0, 0, 0, 0,  0,  0,  0,  0,  0,  0,  0,  2,  2,
                                      2, 3, 3, 3, 3, 4, 4, 4, 6,  6,  7,  7,  8,  8,  9,  9,  10, 10,
                                      11, 11, 12, 12, 13, 13, 14, 14, 15, 15, 16, 16, 17, 17, 18, 18};
__constant__ uint8_t c_db_tc0[52][3] = {
    {0, 0, 0},   {0, 0, 0},   {0, 0, 0},   {0, 0, 0},    {0, 0, 0},    {0, 0, 0},    {0, 0, 0},    {0, 0, 0},
    {0, 0, 0},   {0, 0, 0},   {0, 0, 0},   {0, 0, 0},    {0, 0, 0},    {0, 0, 0},    {0, 0, 0},    {0, 0, 0},
    {0, 0, 0},   {0, 0, 1},   {0, 0, 1},   {0, 0, 1},    {0, 0, 1},    {0, 1, 1},    {0, 1, 1},    {1, 1, 1},
    {1, 1, 1},   {1, 1, 1},   {1, 1, 1},   {1, 1, 2},    {1, 1, 2},    {1, 1, 2},    {1, 1, 2},    {1, 2, 3},
    {1, 2, 3},   {2, 2, 3},   {2, 2, 4},   {2, 3, 4},    {2, 3, 4},    {3, 3, 5},    {3, 4, 6},    {3, 4, 6},
    {4, 5, 7},   {4, 5, 8},   {4, 6, 9},   {5, 7, 10},   {6, 8, 11},   {6, 8, 13},   {7, 10, 14},  {8, 11, 16},
    {9, 12, 18}, {10, 13, 20}, {11, 15, 23}, {13, 17, 25}};
// quantiser table (reconstruction.cpp:9-43): the WZ-edge weights are Qtable[i] / sum
__constant__ int c_db_qtable[9][16] = {
    {0},
    {16, 8, 0, 0, 8, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {32, 8, 0, 0, 8, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},
    {32, 8, 4, 0, 8, 4, 0, 0, 4, 0, 0, 0, 0, 0, 0, 0},
    {32, 16, 8, 4, 16, 8, 4, 0, 8, 4, 0, 0, 4, 0, 0, 0},
    {32, 16, 8, 4, 16, 8, 4, 4, 8, 4, 4, 0, 4, 4, 0, 0},
    {64, 16, 8, 8, 16, 8, 8, 4, 8, 8, 4, 4, 8, 4, 4, 0},
    {64, 32, 16, 8, 32, 16, 8, 4, 16, 8, 4, 4, 8, 4, 4, 0},
    {128, 64, 32, 16, 64, 32, 16, 8, 32, 16, 8, 4, 16, 8, 4, 0}};

#define DB_NONE 0
#define DB_WZ 1    // both sides WZ blocks: strength from the reconstruction flags and variances
#define DB_ISWZ 2  // an intra or skip side: H.264-style strength 1..4
#define DB_BSMAX 0.14

// weighted count of the coefficients reconstruction changed, and the
// "flat block" indicator, of the 4x4 block at (bx, by) (deblock.cpp:286-327)
__device__ void db_block_stats(const FrameDev &F, int bx, int by, double &phi, double &chi) {
  const int *qt = c_db_qtable[F.qindex];
  int qsum = 0;
  for (int i = 0; i < 16; i++) qsum += qt[i];
  phi = 0.0;
  int sum = 0, sq = 0;
  for (int m = 0; m < 4; m++) {
    const int idx = ((by << 2) + m) * F.w + (bx << 2);
    for (int n = 0; n < 4; n++) {
      if (F.dbf[idx + n]) phi += (double)qt[(m << 2) + n] / (double)qsum;
      const int v = F.recon[idx + n];
      sum += v;
      sq += v * v;
    }
  }
  const double var = (double)sq / 16.0 - ((double)sum / 16.0) * ((double)sum / 16.0);
  chi = var < 50.0 ? 1.0 : 0.0;
}

// deblock_44_decision (deblock.cpp:228-344) for the edge between 4x4 blocks 1 and 2
__device__ int db_decide(const FrameDev &F, int x1, int y1, int x2, int y2, double &bs) {
  const int b8w = F.w >> 3;
  const int p1 = (y1 >> 1) * b8w + (x1 >> 1), p2 = (y2 >> 1) * b8w + (x2 >> 1);
  const int t1 = F.mode[p1], t2 = F.mode[p2];
  if (t1 == DVC_INTRA_B && t2 == DVC_INTRA_B) {
    bs = 3.0;
    return DB_ISWZ;
  }
  if (t1 == DVC_INTRA_B || t2 == DVC_INTRA_B) {
    bs = (t1 == DVC_WZ_B || t2 == DVC_WZ_B) ? 4.0 : 3.0;
    return DB_ISWZ;
  }
  if (t1 == DVC_SKIP_B && t2 == DVC_SKIP_B) {
    bs = 0.0;
    return DB_NONE;
  }
  if (t1 == DVC_SKIP_B || t2 == DVC_SKIP_B) {
    if (F.past_is_wz) {
      const int ps = t1 == DVC_SKIP_B ? p1 : p2;
      bs = F.past_mode[ps] == DVC_INTRA_B ? 2.0 : 1.0;
    } else {
      bs = 2.0;
    }
    return DB_ISWZ;
  }
  double phi1, chi1, phi2, chi2;
  db_block_stats(F, x1, y1, phi1, chi1);
  db_block_stats(F, x2, y2, phi2, chi2);
  const double P = 0.9;
  bs = DB_BSMAX * (P * ((phi1 + phi2) / 2.0) + (1.0 - P) * ((chi1 + chi2) / 2.0));
  return bs > 0.0 ? DB_WZ : DB_NONE;
}

// vertical edges at i*W4 + j (j < W4-1), horizontal edges at n + i*W4 + j (i < H4-1)
__global__ void deblock_decide_kernel(FrameDev *frames) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active || !F.deblock) return;
  const int w4 = F.w >> 2, h4 = F.h >> 2, n = w4 * h4;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 2 * n) return;
  const int dir = e >= n, k = dir ? e - n : e, i = k / w4, j = k - i * w4;
  double bs = 0.0;
  int mode = DB_NONE;
  if (dir == 0 ? j < w4 - 1 : i < h4 - 1) mode = dir == 0 ? db_decide(F, j, i, j + 1, i, bs) : db_decide(F, j, i, j, i + 1, bs);
  F.db_mode[e] = (uint8_t)mode;
  F.db_bs[e] = bs;
}

__device__ __forceinline__ int db_clip3(int lo, int hi, int x) { return x < lo ? lo : x > hi ? hi : x; }

// deblock_filter (deblock.cpp:40-206) on one pixel line across one edge: p[0..7*st]
// holds L3 L2 L1 L0 | R0 R1 R2 R3
__device__ void db_line(uint8_t *p, int st, int mode, double bs, const FrameDev &F) {
  const int alpha = c_db_alpha[F.db_qp], beta = c_db_beta[F.db_qp];
  const int L3 = p[0], L2 = p[st], L1 = p[2 * st], L0 = p[3 * st];
  const int R0 = p[4 * st], R1 = p[5 * st], R2 = p[6 * st], R3 = p[7 * st];
  if (!(abs(R0 - L0) < alpha && abs(R0 - R1) < beta && abs(L0 - L1) < beta)) return;
  const double mu = DB_BSMAX * 0.5;
  const bool strong = mode == DB_ISWZ ? (int)bs == 4 : bs > mu;
  if (strong) {
    const int RL0 = L0 + R0;
    const int small_gap = abs(R0 - L0) < ((alpha >> 2) + 2);
    const int aq = (abs(R0 - R2) < beta) & small_gap, ap = (abs(L0 - L2) < beta) & small_gap;
    if (ap) {
      p[3 * st] = (uint8_t)((R1 + ((L1 + RL0) << 1) + L2 + 4) >> 3);
      p[2 * st] = (uint8_t)((L2 + L1 + RL0 + 2) >> 2);
      p[st] = (uint8_t)((((L3 + L2) << 1) + L2 + L1 + RL0 + 4) >> 3);
    } else {
      p[3 * st] = (uint8_t)(((L1 << 1) + L0 + R1 + 2) >> 2);
    }
    if (aq) {
      p[4 * st] = (uint8_t)((L1 + ((R1 + RL0) << 1) + R2 + 4) >> 3);
      p[5 * st] = (uint8_t)((R2 + R0 + L0 + R1 + 2) >> 2);
      p[6 * st] = (uint8_t)((((R3 + R2) << 1) + R2 + R1 + RL0 + 4) >> 3);
    } else {
      p[4 * st] = (uint8_t)(((R1 << 1) + R0 + L1 + 2) >> 2);
    }
    return;
  }
  if (mode == DB_WZ && !(bs > 0.0)) return;
  const int RL0 = (L0 + R0 + 1) >> 1;
  const int aq = abs(R0 - R2) < beta, ap = abs(L0 - L2) < beta;
  const int C0 = mode == DB_ISWZ ? (int)c_db_tc0[F.db_qp][(int)bs - 1] : (int)(bs * (F.db_pow - 1));
  const int tc0 = C0 + ap + aq;
  const int dif = db_clip3(-tc0, tc0, (((R0 - L0) << 2) + (L1 - R1) + 4) >> 3);
  if (ap) p[2 * st] = (uint8_t)(p[2 * st] + db_clip3(-C0, C0, (L2 + RL0 - (L1 << 1)) >> 1));
  p[3 * st] = (uint8_t)db_clip3(0, 255, L0 + dif);
  p[4 * st] = (uint8_t)db_clip3(0, 255, R0 - dif);
  if (aq) p[5 * st] = (uint8_t)(p[5 * st] + db_clip3(-C0, C0, (R2 + RL0 - (R1 << 1)) >> 1));
}

// pass 0: copy the frame; pass 1: vertical edges along each pixel row; pass 2:
// horizontal edges down each pixel column; pass 3: copy the result back
__global__ void deblock_pass_kernel(FrameDev *frames, int pass) {
  FrameDev &F = frames[blockIdx.y];
  if (!F.active || !F.deblock) return;
  const int w = F.w, h = F.h, w4 = w >> 2, h4 = h >> 2, n = w4 * h4;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (pass == 0) {
    if (t < w * h) F.db_img[t] = F.recon[t];
  } else if (pass == 1) {
    if (t >= h) return;
    const int i = t >> 2;
    for (int j = 0; j < w4 - 1; j++) {
      const int e = i * w4 + j;
      if (F.db_mode[e] != DB_NONE) db_line(F.db_img + (size_t)t * w + (j << 2), 1, F.db_mode[e], F.db_bs[e], F);
    }
  } else if (pass == 2) {
    if (t >= w) return;
    const int j = t >> 2;
    for (int i = 0; i < h4 - 1; i++) {
      const int e = n + i * w4 + j;
      if (F.db_mode[e] != DB_NONE) db_line(F.db_img + (size_t)(i << 2) * w + t, w, F.db_mode[e], F.db_bs[e], F);
    }
  } else {
    if (t < w * h) F.recon[t] = F.db_img[t];
  }
}

cudaError_t launch_deblock(FrameDev *fr, int nf, int w, int h, cudaStream_t s) {
  const int n = (w / 4) * (h / 4);
  deblock_decide_kernel<<<dim3((2 * n + 127) / 128, nf), 128, 0, s>>>(fr);
  deblock_pass_kernel<<<dim3((w * h + 127) / 128, nf), 128, 0, s>>>(fr, 0);
  deblock_pass_kernel<<<dim3((h + 127) / 128, nf), 128, 0, s>>>(fr, 1);
  deblock_pass_kernel<<<dim3((w + 127) / 128, nf), 128, 0, s>>>(fr, 2);
  deblock_pass_kernel<<<dim3((w * h + 127) / 128, nf), 128, 0, s>>>(fr, 3);
  return cudaGetLastError();
}

static inline dim3 g2(int n, int tpb, int frames) { return dim3((n + tpb - 1) / tpb, frames); }

// threads per search block of the two motion searches (the candidate columns
// or positions each thread walks follow from it); process-wide, set when a
// context is created (dvc_b200.autotune picks them; the output never depends on them)
static int g_si_threads = 256, g_fme_threads = 256;

void set_me_shapes(int si_threads, int fme_threads) {
  g_si_threads = si_threads == 512 ? 512 : 256;
  g_fme_threads = (fme_threads == 128 || fme_threads == 512) ? fme_threads : 256;
}

cudaError_t launch_side_info(FrameDev *fr, int nf, int w, int h, cudaStream_t s) {
  const int b16n = (w / 16) * (h / 16), b8n = (w / 8) * (h / 8);
  if (g_fme_threads == 128)
    forward_me_kernel<128><<<dim3(b16n, nf), 128, 0, s>>>(fr);
  else if (g_fme_threads == 512)
    forward_me_kernel<512><<<dim3(b16n, nf), 512, 0, s>>>(fr);
  else
    forward_me_kernel<256><<<dim3(b16n, nf), 256, 0, s>>>(fr);
  forward_me_post_kernel<<<g2(b16n * 32, 128, nf), 128, 0, s>>>(fr);
  bidirect_me_kernel<16><<<nf, 1024, 0, s>>>(fr);
  init_blk_mv_kernel<<<g2(b8n, 128, nf), 128, 0, s>>>(fr);
  bidirect_me_kernel<8><<<nf, 1024, 0, s>>>(fr);
  mfc_mse_kernel<<<g2(b8n, 128, nf), 128, 0, s>>>(fr);
  mfc_wvmf_kernel<<<g2(b8n * 16, 128, nf), 128, 0, s>>>(fr);
  mfc_comp_kernel<<<dim3((w + 127) / 128, nf, h), 128, 0, s>>>(fr);
  return cudaGetLastError();
}

cudaError_t launch_frame_prep(FrameDev *fr, int nf, int w, int h, cudaStream_t s) {
  const int b4n = (w / 4) * (h / 4);
  residue_transform_kernel<<<g2(b4n, 128, nf), 128, 0, s>>>(fr);
  noise_band_stats_kernel<<<nf, 512, 0, s>>>(fr);
  noise_alpha_kernel<<<g2(b4n, 128, nf), 128, 0, s>>>(fr);
  over_complete_kernel<<<dim3((w - 3 + 127) / 128, nf, h - 3), 128, 0, s>>>(fr, -1);
  init_ml_kernel<<<g2(b4n, 128, nf), 128, 0, s>>>(fr);
  skip_copy_kernel<<<dim3((w + 127) / 128, nf, h), 128, 0, s>>>(fr);
  return cudaGetLastError();
}

// A batch whose frames have no WZ block (every block intra or skipped) has
// max_nsir == 0: the per-WZ-block kernels have nothing to do and are not launched.
// The block has about one warp per 128 values of the widest pdf of the band
// (2 * max_range + 1 values), so that each lane sums up to four of them.
cudaError_t launch_noise_dist(FrameDev *fr, int nf, int max_nsir, const XlmDev &xt, int band, int max_range,
                              cudaStream_t s) {
  if (max_nsir <= 0) return cudaSuccess;
  const dim3 grid(max_nsir, nf);
  const int warps = (2 * max_range + 1 + 127) / 128;
  if (warps <= 2)
    noise_dist_kernel<64><<<grid, 64, 0, s>>>(fr, xt, band);
  else if (warps <= 4)
    noise_dist_kernel<128><<<grid, 128, 0, s>>>(fr, xt, band);
  else
    noise_dist_kernel<256><<<grid, 256, 0, s>>>(fr, xt, band);
  return cudaGetLastError();
}

cudaError_t launch_cond_bit(FrameDev *fr, int nf, int w, int h, const XlmDev &xt, int band, int bit, cudaStream_t s) {
  cond_bit_kernel<<<g2((w / 4) * (h / 4) * 2, 64, nf), 64, 0, s>>>(fr, xt, band, bit);
  return cudaGetLastError();
}

template <int NT>
static cudaError_t launch_update_si(FrameDev *fr, dim3 tiles, int band, cudaStream_t s) {
  // the attribute is per device: set it once for each device
  static std::atomic<uint64_t> attr_set{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = 1ull << (dev & 63);
  if (!(attr_set.load() & bit)) {
    e = cudaFuncSetAttribute(update_si_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SiShared));
    if (e != cudaSuccess) return e;
    attr_set.fetch_or(bit);
  }
  update_si_kernel<NT><<<tiles, NT, sizeof(SiShared), s>>>(fr, band);
  return cudaGetLastError();
}

cudaError_t launch_band_end(FrameDev *fr, int nf, int w, int h, int max_nsir, int band, const XlmDev &xt,
                            cudaStream_t s) {
  if (max_nsir <= 0) return cudaSuccess;
  recon_kernel<<<g2(max_nsir, 128, nf), 128, 0, s>>>(fr, band);
  const dim3 tiles((w / kSiTile) * (h / kSiTile), nf);
  const cudaError_t e = g_si_threads == 256 ? launch_update_si<256>(fr, tiles, band, s) : launch_update_si<512>(fr, tiles, band, s);
  if (e != cudaSuccess) return e;
  over_complete_kernel<<<dim3((w - 3 + 127) / 128, nf, h - 3), 128, 0, s>>>(fr, band);
  update_ml_kernel<<<g2(max_nsir * 16, 128, nf), 128, 0, s>>>(fr, xt, band);
  return cudaGetLastError();
}

cudaError_t launch_final_inverse(FrameDev *fr, int nf, int max_nsir, cudaStream_t s) {
  if (max_nsir <= 0) return cudaSuccess;
  recon_kernel<<<g2(max_nsir, 128, nf), 128, 0, s>>>(fr, -1);
  return cudaGetLastError();
}

}  // namespace dvc
