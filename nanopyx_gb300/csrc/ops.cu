// Standalone Liquid-Engine ops of the eSRRF / SRRF path, temporal
// correlations and macro-pixel correction (sm_103a).
//
// These follow the reference's float32 arithmetic per output pixel (they are
// the drop-ins for the individual ops and the general fallback of the fused
// kernel); the fused frame-loop kernel in esrrf_fused.cuh is the hot path.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "internal.h"

namespace nx {

namespace {

constexpr int kBlock = 256;

inline unsigned grid_for(long long n, int block = kBlock) {
  long long g = (n + block - 1) / block;
  if (g > 1048576) g = 1048576;  // grid-stride beyond this
  if (g < 1) g = 1;
  return (unsigned)g;
}

// _c_interpolate (src/include/_c_interpolation_catmull_rom.c:21-52) in float:
// pixel-centre taps, out-of-image taps skipped, 0 outside the image.
__device__ __forceinline__ float cr_interp(const float* __restrict__ img, float r, float c,
                                           int rows, int cols) {
  if (r < 0.f || r >= (float)rows || c < 0.f || c >= (float)cols) return 0.f;
  const int r_int = (int)floorf(r - 0.5f);
  const int c_int = (int)floorf(c - 0.5f);
  float q = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int cn = c_int - 1 + j;
    if (cn < 0 || cn >= cols) continue;
    float p = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rn = r_int - 1 + i;
      if (rn < 0 || rn >= rows) continue;
      p = fmaf(__ldg(img + (size_t)rn * cols + cn), cr_cubic(r - ((float)rn + 0.5f)), p);
    }
    q = fmaf(p, cr_cubic(c - ((float)cn + 0.5f)), q);
  }
  return q;
}

__global__ void cr_shift_magnify_kernel(const float* __restrict__ in, int T, int H, int W,
                                        const float* __restrict__ shift_r,
                                        const float* __restrict__ shift_c, float mag_r,
                                        float mag_c, int rowsM, int colsM,
                                        float* __restrict__ out) {
  const long long plane = (long long)rowsM * colsM;
  const long long n = plane * T;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
       idx += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(idx / plane);
    const long long rem = idx - (long long)t * plane;
    const int i = (int)(rem / colsM);
    const int j = (int)(rem - (long long)i * colsM);
    const float row = __fsub_rn(__fdiv_rn((float)i, mag_r), shift_r[t]);
    const float col = __fsub_rn(__fdiv_rn((float)j, mag_c), shift_c[t]);
    out[idx] = cr_interp(in + (size_t)t * H * W, row, col, H, W);
  }
}

// Tiled form of the same resampling for magnifications >= 1: one CTA per
// (frame, up-to-64-row x 256-column output tile).  The sample coordinates and the
// four Catmull-Rom weights of every output row and column of the tile are
// computed once; the input patch the tile reads (zero outside the image, the
// value the reference's skipped taps contribute) is staged in shared memory;
// a vertical pass forms, for every output row and patch column, the 4-tap
// column sum p the per-pixel kernel forms, and the horizontal pass adds the 4
// column taps in the same order -- the same float operations as
// cr_shift_magnify_kernel, so the same results, with 4 shared loads and one
// coalesced store per output instead of 16 global loads and 20 weight
// evaluations.
constexpr int kCrTileCols = 256;
constexpr int kCrMaxTileRows = 64;

// Patch rows / columns a tile can touch at magnification mag >= 1: the taps of
// n consecutive outputs start within floor((n - 1) / mag) + 1 input pixels of
// each other (the extra 1 covers the float rounding of i / mag - shift), plus
// the 4 taps, plus one spare.
inline int cr_patch_extent(int n_out, float mag) {
  return (int)std::floor((double)(n_out - 1) / (double)mag) + 6;
}

// shared memory of a tile of `rows` output rows
inline size_t cr_tile_smem(int rows, float mag_r, float mag_c) {
  const int PR = cr_patch_extent(rows, mag_r), PC = cr_patch_extent(kCrTileCols, mag_c);
  return (size_t)(PR + rows) * PC * sizeof(float) + rows * (sizeof(float4) + sizeof(int));
}

// Output rows per tile: the most (up to 64) whose staging fits in 72 KB, so
// that the stores of a tile outweigh its weight set-up and patch load (64 rows
// beat 32 and 128 at m = 5: 0.53 ms against 0.60 and 0.55 for 100 frames)
inline int cr_tile_rows(float mag_r, float mag_c) {
  for (int rows = kCrMaxTileRows; rows > 32; rows /= 2)
    if (cr_tile_smem(rows, mag_r, mag_c) <= 72 * 1024) return rows;
  return 32;
}

__global__ void __launch_bounds__(kCrTileCols)
    cr_magnify_tiled_kernel(const float* __restrict__ in, int H, int W,
                            const float* __restrict__ shift_r, const float* __restrict__ shift_c,
                            float mag_r, float mag_c, int rowsM, int colsM, int TR, int PR,
                            int PC, float* __restrict__ out) {
  // the float4 row weights first, at the 16-byte aligned base
  extern __shared__ __align__(16) float crs[];
  float4* wr = reinterpret_cast<float4*>(crs);                  // [TR]
  int* rbase = reinterpret_cast<int*>(wr + TR);                 // [TR]
  float* patch = reinterpret_cast<float*>(rbase + TR);          // [PR][PC]
  float* P = patch + PR * PC;                                   // [TR][PC]
  const int t = blockIdx.z;
  const int i0 = blockIdx.y * TR;
  const int j0 = blockIdx.x * kCrTileCols;
  const float sr = shift_r[t], sc = shift_c[t];
  const int tid = threadIdx.x;
  // first patch row / column: the first tap of the tile's first output row / column
  const float row0 = __fsub_rn(__fdiv_rn((float)i0, mag_r), sr);
  const float col0 = __fsub_rn(__fdiv_rn((float)j0, mag_c), sc);
  const int pr0 = (int)floorf(row0 - 0.5f) - 1;
  const int pc0 = (int)floorf(col0 - 0.5f) - 1;
  // this thread's output column: coordinate, validity, patch offset, weights
  const int j = j0 + tid;
  const float col = __fsub_rn(__fdiv_rn((float)j, mag_c), sc);
  const int c_int = (int)floorf(col - 0.5f);
  const int ci = c_int - 1 - pc0;
  const bool cval = j < colsM && !(col < 0.f || col >= (float)W) && ci >= 0 && ci + 3 < PC;
  float wc[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) wc[k] = cr_cubic(col - ((float)(c_int - 1 + k) + 0.5f));
  for (int il = tid; il < TR; il += kCrTileCols) {
    const int i = i0 + il;
    const float row = __fsub_rn(__fdiv_rn((float)i, mag_r), sr);
    const int r_int = (int)floorf(row - 0.5f);
    const int rb = r_int - 1 - pr0;
    const bool rval = i < rowsM && !(row < 0.f || row >= (float)H) && rb >= 0 && rb + 3 < PR;
    float w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = cr_cubic(row - ((float)(r_int - 1 + k) + 0.5f));
    wr[il] = make_float4(w[0], w[1], w[2], w[3]);
    rbase[il] = rval ? rb : -1;
  }
  // patch and vertical pass in warp rows: lanes across the columns, no
  // division by the runtime patch width
  const int lane = tid & 31, warp = tid >> 5;
  const float* f = in + (size_t)t * H * W;
  for (int pr = warp; pr < PR; pr += kCrTileCols / 32) {
    const int r = pr0 + pr;
    const bool rin = r >= 0 && r < H;
    for (int pc = lane; pc < PC; pc += 32) {
      const int c = pc0 + pc;
      patch[pr * PC + pc] = (rin && c >= 0 && c < W) ? __ldg(f + (size_t)r * W + c) : 0.f;
    }
  }
  __syncthreads();
  // vertical pass: P[i][c] = sum_l w_l(i) patch[rbase(i) + l][c] (fma order of
  // the per-pixel kernel: l = 0..3); a row outside the image is all zero
  for (int il = warp; il < TR; il += kCrTileCols / 32) {
    const int rb = rbase[il];
    const float4 w = wr[il];
    for (int c = lane; c < PC; c += 32) {
      float p = 0.f;
      if (rb >= 0) {
        const float* pc = patch + rb * PC + c;
        p = fmaf(pc[0], w.x, p);
        p = fmaf(pc[PC], w.y, p);
        p = fmaf(pc[2 * PC], w.z, p);
        p = fmaf(pc[3 * PC], w.w, p);
      }
      P[il * PC + c] = p;
    }
  }
  __syncthreads();
  if (j >= colsM) return;
  float* o = out + ((size_t)t * rowsM + i0) * colsM + j;
  const int iend = min(TR, rowsM - i0);
  if (cval) {
    // an all-zero P row gives q = +0, the reference's value for a row
    // outside the image, so the loop needs no per-row test
    const float* pp = P + ci;
#pragma unroll 4
    for (int il = 0; il < iend; ++il, pp += PC, o += colsM) {
      float q = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) q = fmaf(pp[k], wc[k], q);
      *o = q;
    }
  } else {
    for (int il = 0; il < iend; ++il, o += colsM) *o = 0.f;
  }
}

// _c_gradient_roberts_cross (src/include/_c_gradients.c:53-73), same
// evaluation order, so bit-identical to the reference.
__global__ void roberts_cross_kernel(const float* __restrict__ in, int T, int H, int W,
                                     float* __restrict__ gc, float* __restrict__ gr) {
  const long long plane = (long long)H * W;
  const long long n = plane * T;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
       idx += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(idx / plane);
    const long long rem = idx - (long long)t * plane;
    const int r1 = (int)(rem / W);
    const int c1 = (int)(rem - (long long)r1 * W);
    const int r0 = r1 > 0 ? r1 - 1 : 0;
    const int c0 = c1 > 0 ? c1 - 1 : 0;
    const float* f = in + (size_t)t * plane;
    const float a = f[(size_t)r0 * W + c1];
    const float b = f[(size_t)r1 * W + c0];
    const float d = f[(size_t)r0 * W + c0];
    const float e = f[(size_t)r1 * W + c1];
    gc[idx] = __fsub_rn(__fadd_rn(__fsub_rn(a, b), e), d);
    gr[idx] = __fsub_rn(__fadd_rn(__fadd_rn(-a, b), e), d);
  }
}

// _c_calculate_rgc (src/include/_c_sr_radial_gradient_convergence.c:17-90) per
// output pixel, float32 as the reference (the FP64 distance weight is
// evaluated in float), reading the given 2m-magnified gradient images.
__global__ void rgc_kernel(const float* __restrict__ gc, const float* __restrict__ gr,
                           const float* __restrict__ img, int T, int rowsM, int colsM, int M,
                           RgcScalars sc, int iw, float* __restrict__ out) {
  const long long plane = (long long)rowsM * colsM;
  const long long n = plane * T;
  const int grad_w = (int)((float)colsM * 2.0f);
  const long long gplane = (long long)(2 * rowsM) * grad_w;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
       idx += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(idx / plane);
    const long long rem = idx - (long long)t * plane;
    const int yM = (int)(rem / colsM);
    const int xM = (int)(rem - (long long)yM * colsM);
    if (yM < sc.margin || yM >= rowsM - sc.margin || xM < sc.margin ||
        xM >= colsM - sc.margin) {
      out[idx] = 0.f;
      continue;
    }
    const float* Gx = gc + (size_t)t * gplane;
    const float* Gy = gr + (size_t)t * gplane;
    const float xc = __fdiv_rn((float)xM + 0.5f, (float)M);
    const float yc = __fdiv_rn((float)yM + 0.5f, (float)M);
    float rgc = 0.f, wsum = 0.f;
    const int by = (int)(2.0f * yc), bx = (int)(2.0f * xc);
    for (int j = sc.start; j < sc.end; ++j) {
      const float vy = (float)(by + j) / 2.0f;
      if (!(0.f < vy && vy <= (float)(rowsM - 1))) continue;
      for (int i = sc.start; i < sc.end; ++i) {
        const float vx = (float)(bx + i) / 2.0f;
        if (!(0.f < vx && vx <= (float)(colsM - 1))) continue;
        const float dx = vx - xc;
        const float dy = vy - yc;
        const float d = sqrtf(dx * dx + dy * dy);
        if (d != 0.f && d <= sc.tSO) {
          float pos_y = vy * (float)M * 2.0f;
          float pos_x = vx * (float)M * 2.0f;
          if (pos_y >= (float)rowsM * 2.0f) pos_y = (float)rowsM * 2.0f - 1.f;
          if (pos_x >= (float)colsM * 2.0f) pos_x = (float)colsM * 2.0f - 1.f;
          if (pos_y < 0.f) pos_y = 0.f;
          if (pos_x < 0.f) pos_x = 0.f;
          const size_t g = (size_t)(int)pos_y * grad_w + (int)pos_x;
          const float gx = __ldg(Gx + g), gy = __ldg(Gy + g);
          const float tt = d * expf(-(d * d) / sc.tSS);
          const float w = (tt * tt) * (tt * tt);
          wsum += w;
          if (gx * dx + gy * dy < 0.f) {
            float dk = fabsf(gy * dx - gx * dy) / sqrtf(gx * gx + gy * gy);
            if (isnan(dk)) dk = d;
            dk = 1.f - dk / d;
            rgc += dk * w;
          }
        }
      }
    }
    rgc = wsum > 0.f ? rgc / wsum : 0.f;
    rgc = rgc < 0.f ? 0.f : apply_sensitivity(rgc, sc.sens_mode, sc.sens_int, sc.sens);
    out[idx] = iw ? rgc * img[idx] : rgc;
  }
}

// The same RGC with the weights tabulated.  An output's window samples sit at
// fixed offsets of its sub-pixel phase, so unit offset and weight depend on
// (phase, window position) only: every block evaluates that table once in
// shared memory, from exact phase centres (the per-pixel kernel's float32
// centres (x + 0.5) / M move it by up to 2^-24 of the coordinate).  The samples of
// all outputs lie on the half-pixel grid, one gradient in M x M, so a block takes a
// tile of 32 x kRgcTileRows input pixels and stages the grid's unit gradients
// first, each normalised once: a sample costs one 8-byte and one broadcast 16-byte
// shared load and seven arithmetic instructions.  A warp serves one output phase of
// one input row, lanes along x; even and odd grid columns lie apart, so that its
// lanes' gradients are neighbours.
// 8 x 600 x 520, M = 2, R = 1.5: 97 us (128 with the rows of the window not
// unrolled); 283 us with the gradients read and normalised per sample, 409 us in
// the per-pixel kernel.  20 x 640 x 640, M = 5, R = 2: 0.37 ms, 2.06 ms per pixel.
constexpr int kRgcTableBytes = 48 * 1024;
constexpr int kRgcTileRows = 8;
constexpr int kRgcSharedMax = 128 * 1024;  // table and tile: at most 114,484 bytes (M = 1)

// gradient direction; 0 where there is none (or none that counts: infinities)
__device__ __forceinline__ float2 unit_gradient(float gx, float gy) {
  float s2 = fmaf(gy, gy, gx * gx);
  if (!(s2 > 1e-30f && s2 < 1e30f)) {  // the squares may not hold: scale first
    const float mx = fmaxf(fabsf(gx), fabsf(gy));
    if (mx == 0.f || isinf(mx)) return make_float2(0.f, 0.f);
    gx = __fdiv_rn(gx, mx);
    gy = __fdiv_rn(gy, mx);
    s2 = fmaf(gy, gy, gx * gx);
  }
  const float r = rsqrtf(s2);
  return make_float2(gx * r, gy * r);
}

struct RgcTile {
  int cols, rows;  // half-grid cells of a tile and its halo, columns in halves
  size_t bytes;    // of the block's shared memory
};
inline RgcTile rgc_tile(int M, int W2) {
  RgcTile t;
  t.cols = (64 + W2) / 2;
  t.rows = 2 * kRgcTileRows - 1 + W2;
  t.bytes = (size_t)M * M * W2 * W2 * sizeof(float4) + (size_t)t.rows * 2 * t.cols * sizeof(float2) +
            (size_t)M * M * sizeof(float);
  return t;
}

// W: the window's side where its rows unroll (3 to 13, radii from 0.5 to below 3.5), or 0
template <int W>
__global__ void __launch_bounds__(kBlock)
    rgc_table_kernel(const float* __restrict__ gc, const float* __restrict__ gr,
                     const float* __restrict__ img, int T, int rowsM, int colsM, int M,
                     RgcScalars sc, int iw, RgcTile tile, int parts,
                     float* __restrict__ out) {
  // table [py][px][j][i] of (unit offset, weight; 0: does not count, -); the
  // tile [row][column parity][column / 2]; sum of weights per phase
  extern __shared__ __align__(16) float4 rgct[];
  const int W2 = W ? W : sc.end - sc.start, MM = M * M;
  float2* const cell = reinterpret_cast<float2*>(rgct + MM * W2 * W2);
  float* const wtot = reinterpret_cast<float*>(cell + tile.rows * 2 * tile.cols);
  for (int e = threadIdx.x; e < MM * W2 * W2; e += kBlock) {
    const int i = e % W2, j = e / W2 % W2, px = e / (W2 * W2) % M, py = e / (W2 * W2 * M);
    // 2 M d = M (c + offset) - (2 p + 1): exact integers
    const int ax = M * ((2 * px + 1) / M + sc.start + i) - (2 * px + 1);
    const int ay = M * ((2 * py + 1) / M + sc.start + j) - (2 * py + 1);
    const float s2 = (float)(ax * ax + ay * ay);
    const float d = __fdiv_rn(__fsqrt_rn(s2), 2.f * (float)M);
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    if (s2 != 0.f && d <= sc.tSO) {
      const float e1 = d * expf(-(d * d) / sc.tSS);
      const float r = __fdiv_rn(1.f, __fsqrt_rn(s2));
      t = make_float4((float)ax * r, (float)ay * r, (e1 * e1) * (e1 * e1), 0.f);
    }
    rgct[e] = t;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < MM; e += kBlock) {
    float w = 0.f;
    for (int k = 0; k < W2 * W2; ++k) w += rgct[e * W2 * W2 + k].z;
    wtot[e] = w;
  }
  const int grad_w = 2 * colsM, kx_max = 2 * (colsM - 1), ky_max = 2 * (rowsM - 1);
  const long long gplane = 2LL * rowsM * grad_w;
  const int tx_n = ((colsM + M - 1) / M + 31) / 32;
  const int ty_n = ((rowsM + M - 1) / M + kRgcTileRows - 1) / kRgcTileRows;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long units = (long long)T * ty_n * tx_n;
  // a tile's (row, phase) items are dealt to `parts` blocks (grid y)
  const int k0 = blockIdx.y * (kBlock / 32) + warp, kstep = parts * (kBlock / 32);
  for (long long u = blockIdx.x; u < units; u += gridDim.x) {
    const int tx = (int)(u % tx_n), ty = (int)(u / tx_n % ty_n);
    const long long t = u / ((long long)tx_n * ty_n);
    const float* Gx = gc + t * gplane;
    const float* Gy = gr + t * gplane;
    const int ny0 = ty * kRgcTileRows, nx0 = tx * 32;
    const int ky0 = 2 * ny0 + sc.start, kx0 = 2 * nx0 + sc.start;
    __syncthreads();  // wtot; the previous tile has been read
    for (int y = warp; y < tile.rows; y += kBlock / 32) {
      const int ky = ky0 + y;
      const size_t row = (size_t)min(max(ky, 0) * M, 2 * rowsM - 1) * grad_w;
      for (int x = lane; x < 2 * tile.cols; x += 32) {
        const int kx = kx0 + x;
        float2 g = make_float2(0.f, 0.f);  // outside: does not count
        if (ky >= 1 && ky <= ky_max && kx >= 1 && kx <= kx_max) {
          const size_t o = row + min(kx * M, grad_w - 1);
          g = unit_gradient(__ldg(Gx + o), __ldg(Gy + o));
        }
        cell[(y * 2 + (x & 1)) * tile.cols + (x >> 1)] = g;
      }
    }
    __syncthreads();
    for (int k = k0; k < kRgcTileRows * MM; k += kstep) {
      const int p = k % MM, yl = k / MM, py = p / M, px = p - py * M;
      const int yM = (ny0 + yl) * M + py, xM = (nx0 + lane) * M + px;
      if (yM >= rowsM || xM >= colsM) continue;
      const size_t o = ((size_t)t * rowsM + yM) * colsM + xM;
      if (yM < sc.margin || yM >= rowsM - sc.margin || xM < sc.margin ||
          xM >= colsM - sc.margin) {
        out[o] = 0.f;
        continue;
      }
      const int cy = (2 * py + 1) / M, cx = (2 * px + 1) / M;
      const float4* e = rgct + p * W2 * W2;
      float rgc = 0.f;
      for (int j = 0; j < W2; ++j, e += W2) {
        // grid column cx + i: parity and index of even and odd i
        const float2* c = cell + (2 * yl + cy + j) * 2 * tile.cols + lane;
        const float2* c0 = cx ? c + tile.cols : c;
        const float2* c1 = cx ? c + 1 : c + tile.cols;
#pragma unroll(W ? W : 4)
        for (int i = 0; i < W2; ++i) {
          const float2 g = (i & 1) ? c1[i >> 1] : c0[i >> 1];
          const float4 w = e[i];
          const float v = fmaf(-fabsf(fmaf(g.y, w.x, -(g.x * w.y))), w.z, w.z);
          if (fmaf(g.y, w.y, g.x * w.x) < 0.f) rgc += v;
        }
      }
      const int by = ky0 + 2 * yl + cy, bx = kx0 + 2 * lane + cx;  // first sample
      float wsum = wtot[p];
      if (by < 1 || by + W2 - 1 > ky_max || bx < 1 || bx + W2 - 1 > kx_max) {
        wsum = 0.f;
        e = rgct + p * W2 * W2;
        for (int j = 0; j < W2; ++j)
          for (int i = 0; i < W2; ++i)
            if (by + j >= 1 && by + j <= ky_max && bx + i >= 1 && bx + i <= kx_max)
              wsum += e[j * W2 + i].z;
      }
      rgc = wsum > 0.f ? rgc / wsum : 0.f;
      rgc = rgc < 0.f ? 0.f : apply_sensitivity(rgc, sc.sens_mode, sc.sens_int, sc.sens);
      out[o] = iw ? rgc * img[o] : rgc;
    }
  }
}

// _c_gradient_radiality (src/include/_c_gradients.c:3-25)
__global__ void gradient_radiality_kernel(const float* __restrict__ in, int T, int h, int w,
                                          float* __restrict__ gx, float* __restrict__ gy) {
  const long long plane = (long long)h * w;
  const long long n = plane * T;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
       idx += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(idx / plane);
    const long long rem = idx - (long long)t * plane;
    const int j = (int)(rem / w);
    const int i = (int)(rem - (long long)j * w);
    float vx = 0.f, vy = 0.f;
    if (j >= 1 && j < h - 1 && i >= 1 && i < w - 1) {
      const float* f = in + (size_t)t * plane;
      vx = __fadd_rn(-f[(size_t)j * w + i - 1], f[(size_t)j * w + i + 1]);
      vy = __fadd_rn(-f[(size_t)(j - 1) * w + i], f[(size_t)(j + 1) * w + i]);
    }
    gx[idx] = vx;
    gy[idx] = vy;
  }
}

// _c_calculate_radiality_per_subpixel (src/include/_c_sr_radiality.c:15-51)
__global__ void radiality_kernel(const float* __restrict__ gx, const float* __restrict__ gy,
                                 const float* __restrict__ img_interp, int T, int h, int w,
                                 int M, RingCoords rc, int border, int positivity, int iw,
                                 float* __restrict__ out) {
  const int rowsM = h * M, colsM = w * M;
  const long long plane = (long long)rowsM * colsM;
  const long long n = plane * T;
  const int lo_j = (1 + border) * M, hi_j = (h - 1 - border) * M;
  const int lo_i = (1 + border) * M, hi_i = (w - 1 - border) * M;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
       idx += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(idx / plane);
    const long long rem = idx - (long long)t * plane;
    const int j = (int)(rem / colsM);
    const int i = (int)(rem - (long long)j * colsM);
    if (j < lo_j || j >= hi_j || i < lo_i || i >= hi_i) {
      out[idx] = 0.f;
      continue;
    }
    const float* GX = gx + (size_t)t * h * w;
    const float* GY = gy + (size_t)t * h * w;
    const float xc = (float)i + 0.5f;
    const float yc = (float)j + 0.5f;
    float div = 0.f;
#pragma unroll 2
    for (int s = 0; s < 12; ++s) {
      const float xr = rc.x[s], yr = rc.y[s];
      const float x0 = __fadd_rn(xc, xr);
      const float y0 = __fadd_rn(yc, yr);
      const float ry = __fdiv_rn(y0, (float)M);
      const float rx = __fdiv_rn(x0, (float)M);
      const float vgx = cr_interp(GX, ry, rx, h, w);
      const float vgy = cr_interp(GY, ry, rx, h, w);
      const float gmag = sqrtf(vgx * vgx + vgy * vgy);
      float dk = 0.f;
      if (gmag != 0.f) {
        dk = 1.f - (fabsf(vgy * (xc - x0) - vgx * (yc - y0)) / gmag) / rc.radius;
        dk = dk * dk;
      }
      if (vgx * xr + vgy * yr > 0.f) div -= dk;
      else div += dk;
    }
    div /= 12.f;
    const float cgh = positivity ? fmaxf(div, 0.f) : div;
    out[idx] = iw ? cgh * img_interp[idx] : cgh;
  }
}

// ---------------------------------------------------------------------------
// temporal records: planes mean, M2, C, A, B of Moments (common.cuh)
// ---------------------------------------------------------------------------
__global__ void record_push_frame_kernel(const float* __restrict__ frame, long long n,
                                         float* __restrict__ rec, int it) {
  const float inv = __frcp_rn((float)(it + 1));
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float v = frame[i];
    Moments m = moments_start(v);
    if (it > 0) {
      m = Moments{rec[i], rec[n + i], rec[2 * n + i], rec[3 * n + i], rec[4 * n + i]};
      moments_push(m, v, inv);
    }
    rec[i] = m.mean;
    rec[n + i] = m.m2;
    rec[2 * n + i] = m.c;
    rec[3 * n + i] = m.a;
    rec[4 * n + i] = m.b;
  }
}

// a followed by b, the rounding of a's mean carried along: the mean is a.mean + lo
__device__ __forceinline__ void moments_merge_lo(Moments& a, float& lo, const Moments& b, int na,
                                                 int nb, bool full) {
  const float q = __fdiv_rn((float)nb, (float)na + (float)nb);
  const float before = a.mean, dl = b.mean - before;
  moments_merge(a, b, na, nb, full);
  if (na > 0 && nb > 0) lo = fmaf(lo, 1.f - q, fmaf(dl, q, before - a.mean));
}
__device__ __forceinline__ void mean_round(Moments& a, float lo) {
  const float mean = a.mean + lo;
  if (mean == mean) a.mean = mean;  // an infinite mean has no rounding to add
}

__device__ __forceinline__ Moments record(const float* __restrict__ r, long long n, bool full) {
  if (full) return Moments{r[0], r[n], r[2 * n], r[3 * n], r[4 * n]};
  return Moments{r[0], 0.f, 0.f, 0.f, 0.f};
}

// The moments of pixel i over nf frames in `chunks` consecutive records (F fields of n
// pixels; 5, or the mean only).  A merge rounds like a push, and small images split into
// more chunks than one chain is short for: up to kMergeGroup records are one chain, more
// are merged in groups of as many and the groups in order, the rounding of the means
// carried along (mean of 32 frames of 26 x 64 in 16 chunks: 6.2e-8 in one chain, 3.9e-8).
// chain: one chain whatever their number.  GROUPS: built for groups at all -- the kernels
// of the usual few records are built without, whose registers keep them at memory speed
// (20 x 512 x 512, m = 5, VAR: 44 us, 61 to 65 with the groups' code in).
constexpr int kMergeGroup = 8;
template <bool GROUPS>
__device__ __forceinline__ Moments merge_records(const float* __restrict__ rec, int F, int chunks,
                                                 int nf, long long n, bool full, bool chain,
                                                 long long i) {
  auto frames = [&](int c) {
    return (int)((long long)(c + 1) * nf / chunks - (long long)c * nf / chunks);
  };
  Moments a{0.f, 0.f, 0.f, 0.f, 0.f};
  int na = 0;
  if (!GROUPS || chain || chunks <= kMergeGroup) {
    for (int c = 0; c < chunks; ++c) {
      const int nc = frames(c);
      moments_merge(a, record(rec + (size_t)c * F * n + i, n, full), na, nc, full);
      na += nc;
    }
    return a;
  }
  float lo = 0.f;
  for (int g = 0; g < chunks; g += kMergeGroup) {
    Moments s{0.f, 0.f, 0.f, 0.f, 0.f};
    int ns = 0;
    float ls = 0.f;
    for (int c = g; c < min(g + kMergeGroup, chunks); ++c) {
      const int nc = frames(c);
      moments_merge_lo(s, ls, record(rec + (size_t)c * F * n + i, n, full), ns, nc, full);
      ns += nc;
    }
    mean_round(s, ls);
    moments_merge_lo(a, lo, s, na, ns, full);
    na += ns;
  }
  mean_round(a, lo);
  return a;
}

// acc (its moments over na frames; nothing there if 0) followed by a block of nb frames in
// `chunks` records, merged among themselves first, so that acc's chain is one of pushes
// (100 frames of 26 x 64 in pushes of 16, m = 2: mean 4.8e-8, 1.1e-7 in one chain of
// chunks).  One launch whatever the chunks: with one each, the 8 chunks of a 16-frame
// block of 48 x 60, m = 2, took 53 us a push instead of 28.
// KIND 0: one record, 1: one chain of them, 2: groups.
template <int KIND>
__global__ void record_merge_kernel(float* __restrict__ acc, const float* __restrict__ rec,
                                    long long n, int na, int nb, int chunks) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const Moments b = KIND == 0 ? record(rec + i, n, true)
                                : merge_records<KIND == 2>(rec, 5, chunks, nb, n, true, false, i);
    Moments a = b;
    if (na > 0) {
      a = record(acc + i, n, true);
      moments_merge(a, b, na, nb, true);
    }
    acc[i] = a.mean;
    acc[n + i] = a.m2;
    acc[2 * n + i] = a.c;
    acc[3 * n + i] = a.a;
    acc[4 * n + i] = a.b;
  }
}

// Merges the `nchunks` consecutive records of one timepoint in frame order and
// writes the correlations of corr_mask.  full: 5-field records; else one field
// (the mean) per record.
template <bool GROUPS>
__device__ __forceinline__ void finalize_pixel(const float* __restrict__ rec, int F,
                                               int nchunks, int nf, long long n, int corr_mask,
                                               float* __restrict__ out, long long out_stride,
                                               bool full, bool chain, long long i) {
  {
    const Moments a = merge_records<GROUPS>(rec, F, nchunks, nf, n, full, chain, i);
    const float fn = (float)nf;
    int ci = 0;
    if (corr_mask & NX_CORR_AVG) out[(ci++) * out_stride + i] = a.mean;
    if (corr_mask & NX_CORR_VAR) {
      const float v = __fdiv_rn(a.m2, fn);
      out[(ci++) * out_stride + i] = v > 0.f ? v : 0.f;
    }
    if (corr_mask & NX_CORR_TAC2) out[(ci++) * out_stride + i] = __fdiv_rn(a.c, fn - 1.f);
  }
}

// every timepoint of one reconstruction in one launch (blockIdx.y): timepoint
// tp holds nf = min(fpt, T - tp fpt) frames in min(chunks, nf) records
template <bool GROUPS>
__global__ void finalize_kernel(const float* __restrict__ rec, int F, int chunks, int T, int fpt,
                                long long n, int corr_mask, float* __restrict__ out,
                                long long out_stride, bool full) {
  const int tp = blockIdx.y;
  const int nf = min(fpt, T - tp * fpt);
  const float* r = rec + (size_t)tp * chunks * F * n;
  float* o = out + (size_t)tp * n;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    finalize_pixel<GROUPS>(r, F, min(chunks, nf), nf, n, corr_mask, o, out_stride, full, false,
                           i);
}

// a batch's finalisations in one launch: block -> job by binary search on
// the jobs' first blocks, one pixel per thread
template <bool GROUPS>
__global__ void finalize_jobs_kernel(const FinalizeJob* __restrict__ jobs, int njobs) {
  int lo = 0, hi = njobs - 1;
  const int bx = blockIdx.x;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].block0 <= bx) lo = mid;
    else hi = mid - 1;
  }
  const FinalizeJob j = jobs[lo];
  const long long i = (long long)(bx - j.block0) * blockDim.x + threadIdx.x;
  if (i < j.n)
    finalize_pixel<GROUPS>(j.rec, j.F, j.nchunks, j.nf, j.n, j.corr_mask, j.out, j.out_stride,
                           j.full != 0, j.chain != 0, i);
}

// sr_temporal_correlations.py:46-75,205-221 on a resident stack, float32 and
// in numpy's order (sequential over frames, no contraction)
__global__ void temporal_stack_kernel(const float* __restrict__ x, int T, long long n, int corr,
                                      float* __restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float s = 0.f;
    for (int t = 0; t < T; ++t) s = __fadd_rn(s, x[(size_t)t * n + i]);
    const float mean = __fdiv_rn(s, (float)T);
    if (corr == NX_CORR_AVG) {
      out[i] = mean;
    } else if (corr == NX_CORR_VAR) {
      float q = 0.f;
      for (int t = 0; t < T; ++t) {
        const float c = __fsub_rn(x[(size_t)t * n + i], mean);
        q = __fadd_rn(q, __fmul_rn(c, c));
      }
      out[i] = __fdiv_rn(q, (float)T);
    } else {
      float q = 0.f;
      float prev = T > 0 ? __fsub_rn(x[i], mean) : 0.f;
      for (int t = 1; t < T; ++t) {
        const float c = __fsub_rn(x[(size_t)t * n + i], mean);
        q = __fadd_rn(q, __fmul_rn(prev, c));
        prev = c;
      }
      out[i] = __fdiv_rn(q, (float)(T - 1));
    }
  }
}

// VAR and TAC2 with each CTA's 128 pixels x T frames staged in shared memory,
// so the stack is read from HBM once (the two-pass per-pixel kernel reads it
// twice); identical operations and order.
constexpr int kTcPix = 128;
constexpr int kTcMaxFrames = 400;  // 128 x 400 floats = 200 KB of shared memory

__global__ void __launch_bounds__(kTcPix)
    temporal_stack_smem_kernel(const float* __restrict__ x, int T, long long n, int corr,
                               bool vec, float* __restrict__ out) {
  extern __shared__ __align__(16) float ts[];  // [T][kTcPix]
  const long long p0 = (long long)blockIdx.x * kTcPix;
  const int tid = threadIdx.x;
  const long long i = p0 + tid;
  const bool in = i < n;
  if (vec) {
    // every 16-byte piece of the CTA's T x 128 block as one asynchronous copy,
    // all issued before the single wait (enough bytes in flight to fill HBM)
    for (int k = tid; k < T * (kTcPix / 4); k += kTcPix) {
      const int t = k / (kTcPix / 4), c = (k % (kTcPix / 4)) * 4;
      const unsigned dst = smem_addr(ts + t * kTcPix + c);
      const float* src = x + (size_t)t * n + p0 + c;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  } else {
    for (int t = 0; t < T; ++t) ts[t * kTcPix + tid] = in ? __ldg(x + (size_t)t * n + i) : 0.f;
  }
  if (!in) return;  // each thread reads back only its own column
  float s = 0.f;
  for (int t = 0; t < T; ++t) s = __fadd_rn(s, ts[t * kTcPix + tid]);
  const float mean = __fdiv_rn(s, (float)T);
  if (corr == NX_CORR_AVG) {
    out[i] = mean;
  } else if (corr == NX_CORR_VAR) {
    float q = 0.f;
    for (int t = 0; t < T; ++t) {
      const float c = __fsub_rn(ts[t * kTcPix + tid], mean);
      q = __fadd_rn(q, __fmul_rn(c, c));
    }
    out[i] = __fdiv_rn(q, (float)T);
  } else {
    float q = 0.f;
    float prev = __fsub_rn(ts[tid], mean);
    for (int t = 1; t < T; ++t) {
      const float c = __fsub_rn(ts[t * kTcPix + tid], mean);
      q = __fadd_rn(q, __fmul_rn(prev, c));
      prev = c;
    }
    out[i] = __fdiv_rn(q, (float)(T - 1));
  }
}

// sr_temporal_correlations.py:4-43 (orders 0, 1, -1) and :111-157 (ACRF
// orders 2, 3, 4 without lag-time integration), float32 per pixel
__global__ void srrf_temporal_kernel(const float* __restrict__ x, int T, long long n, int order,
                                     float* __restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    if (order == 0) {
      float m = -INFINITY;
      for (int t = 0; t < T; ++t) m = fmaxf(m, x[(size_t)t * n + i]);
      out[i] = m;
      continue;
    }
    if (order == -1) {
      // sum_{t0 <= t1} r+_t0 r+_t1 / (T (T + 1) / 2), r+ = max(r, 0)
      float s1 = 0.f, s2 = 0.f;
      for (int t = 0; t < T; ++t) {
        const float r = fmaxf(x[(size_t)t * n + i], 0.f);
        s1 += r;
        s2 = fmaf(r, r, s2);
      }
      const float cnt = 0.5f * (float)T * (float)(T + 1);
      out[i] = 0.5f * (s1 * s1 + s2) / fmaxf(cnt, 1.f);
      continue;
    }
    float s = 0.f;
    for (int t = 0; t < T; ++t) s = __fadd_rn(s, x[(size_t)t * n + i]);
    const float mean = __fdiv_rn(s, (float)T);
    if (order == 1) {
      out[i] = mean;
      continue;
    }
    float ab = 0.f, abc = 0.f, abcd = 0.f, cd = 0.f, ac = 0.f, bd = 0.f, ad = 0.f, bc = 0.f;
    for (int t = 0; t < T - order; ++t) {
      const float a = __fsub_rn(x[(size_t)t * n + i], mean);
      const float b = __fsub_rn(x[(size_t)(t + 1) * n + i], mean);
      ab = __fadd_rn(ab, __fmul_rn(a, b));
      if (order == 3) {
        const float c = __fsub_rn(x[(size_t)(t + 2) * n + i], mean);
        abc = __fadd_rn(__fadd_rn(abc, __fmul_rn(a, b)), c);
      }
      if (order == 4) {
        const float c = __fsub_rn(x[(size_t)(t + 2) * n + i], mean);
        const float d = __fsub_rn(x[(size_t)(t + 3) * n + i], mean);
        abcd = __fadd_rn(abcd, __fmul_rn(__fmul_rn(__fmul_rn(a, b), c), d));
        cd = __fadd_rn(cd, __fmul_rn(c, d));
        ac = __fadd_rn(ac, __fmul_rn(a, c));
        bd = __fadd_rn(bd, __fmul_rn(b, d));
        ad = __fadd_rn(ad, __fmul_rn(a, d));
        bc = __fadd_rn(bc, __fmul_rn(b, c));
      }
    }
    float v;
    if (order == 3) v = fabsf(abc);
    else if (order == 4) v = fabsf(abcd - ab * cd - ac * bd - ad * bc);
    else v = fabsf(ab);
    out[i] = __fdiv_rn(v, (float)T);
  }
}

// ACRF of order 2, 3, 4 with lag-time integration
// (sr_temporal_correlations.py:111-121,159-200), one pixel per thread, the
// reference's float32 operations in its order (no contraction).  Per level:
// the lag products over t < n_iter (ab restarts, abc and the order-4 sums run
// on across levels), and frame t, once read, is replaced in place by
// sum_{k < order-1} frame[t*order + k] / order for t < n_bin (else 0) --
// zeroed first, so the k = 0 term of t = 0 reads the zero.  The last level's
// correlation over n_binned is the result; 0 when no level runs.
__global__ void srrf_acrf_integrated_kernel(float* __restrict__ im, int T, long long n, int order,
                                            AcrfSchedule sch, float* __restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float* x = im + i;
    float s = 0.f;
    for (int t = 0; t < T; ++t) s = __fadd_rn(s, x[(size_t)t * n]);
    const float mean = __fdiv_rn(s, (float)T);
    const float fo = (float)order;
    float res = 0.f;
    float abc = 0.f, abcd = 0.f, cd = 0.f, ac = 0.f, bd = 0.f, ad = 0.f, bc = 0.f;
    for (int L = 0; L < sch.n_levels; ++L) {
      float ab = 0.f;
      const int n_iter = sch.n_iter[L], n_bin = sch.n_bin[L];
      for (int t = 0; t < n_iter; ++t) {
        const float a = __fsub_rn(x[(size_t)t * n], mean);
        const float b = __fsub_rn(x[(size_t)(t + 1) * n], mean);
        const float pab = __fmul_rn(a, b);
        ab = __fadd_rn(ab, pab);
        if (order == 3) {
          const float c = __fsub_rn(x[(size_t)(t + 2) * n], mean);
          abc = __fadd_rn(__fadd_rn(abc, pab), c);
        } else if (order == 4) {
          const float c = __fsub_rn(x[(size_t)(t + 2) * n], mean);
          const float d = __fsub_rn(x[(size_t)(t + 3) * n], mean);
          abcd = __fadd_rn(abcd, __fmul_rn(__fmul_rn(pab, c), d));
          cd = __fadd_rn(cd, __fmul_rn(c, d));
          ac = __fadd_rn(ac, __fmul_rn(a, c));
          bd = __fadd_rn(bd, __fmul_rn(b, d));
          ad = __fadd_rn(ad, __fmul_rn(a, d));
          bc = __fadd_rn(bc, __fmul_rn(b, c));
        }
        float v = 0.f;
        if (t < n_bin) {
          const int tb = t * order;
          for (int k = 0; k < order - 1; ++k) {
            const float src = (tb + k == t) ? v : x[(size_t)(tb + k) * n];
            v = __fadd_rn(v, __fdiv_rn(src, fo));
          }
        }
        x[(size_t)t * n] = v;
      }
      float num;
      if (order == 3) {
        num = fabsf(abc);
      } else if (order == 4) {
        num = __fsub_rn(__fsub_rn(__fsub_rn(abcd, __fmul_rn(ab, cd)), __fmul_rn(ac, bd)),
                        __fmul_rn(ad, bc));
        num = fabsf(num);
      } else {
        num = fabsf(ab);
      }
      res = __fdiv_rn(num, sch.n_binned[L]);
    }
    out[i] = res;
  }
}

// Camera integers to float32, exact.  HBM-bound: 8 values per thread from one
// vector load (16 bytes of 16-bit, 8 of 8-bit pixels) into two 16-byte stores;
// scalar where the pointers do not allow it and for the rest.
template <typename S>
__global__ void __launch_bounds__(256)
    to_float_kernel(const S* __restrict__ src, long long n, int vec, float* __restrict__ dst) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long n8 = vec ? n / 8 : 0;
  for (long long i = t; i < n8; i += stride) {
    union {
      uint4 q;
      uint2 d;
      S v[8];
    } u;
    if constexpr (sizeof(S) == 2) u.q = __ldg(reinterpret_cast<const uint4*>(src) + i);
    else u.d = __ldg(reinterpret_cast<const uint2*>(src) + i);
    float4* o = reinterpret_cast<float4*>(dst) + 2 * i;
    o[0] = make_float4((float)u.v[0], (float)u.v[1], (float)u.v[2], (float)u.v[3]);
    o[1] = make_float4((float)u.v[4], (float)u.v[5], (float)u.v[6], (float)u.v[7]);
  }
  for (long long i = n8 * 8 + t; i < n; i += stride) dst[i] = (float)src[i];
}

template <typename S>
cudaError_t launch_to_float(const void* src, long long n, float* dst, cudaStream_t s) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(src), b = reinterpret_cast<uintptr_t>(dst);
  const int vec = a % (8 * sizeof(S)) == 0 && b % 16 == 0;
  const long long items = vec ? (n + 7) / 8 : n;
  const unsigned grid = (unsigned)std::max<long long>(1, std::min<long long>((items + 255) / 256,
                                                                             152LL * 32));
  to_float_kernel<S><<<grid, 256, 0, s>>>(static_cast<const S*>(src), n, vec, dst);
  return cudaGetLastError();
}

// macro-pixel map, stage 1: block (s, py, chunk) sums the macro-pixel rows
// [chunk*rpc, (chunk+1)*rpc) of phase row py; thread t owns phase px = t % M
// (blockDim is a multiple of M); Kahan sums, fixed-order block reduction.
// HBM-bound: kMpcAhead loads of a row are in flight before the dependent sum
// chain takes them, in its order.
constexpr int kMpcAhead = 8;
__global__ void mpc_partial_kernel(const float* __restrict__ img, int rowsM, int colsM, int M,
                                   int nch, float* __restrict__ part) {
  extern __shared__ float red[];
  const int s = blockIdx.x;
  const int py = blockIdx.y;
  const int ch = blockIdx.z;
  const int rows = rowsM / M, cols = colsM / M;
  const int rpc = (rows + nch - 1) / nch;
  const int r0 = ch * rpc, r1 = min(rows, r0 + rpc);
  const float* f = img + (size_t)s * rowsM * colsM;
  const int width = cols * M, step = blockDim.x;
  float sum = 0.f, comp = 0.f;
  for (int ry = r0; ry < r1; ++ry) {
    const float* row = f + (size_t)(ry * M + py) * colsM;
    for (int x0 = threadIdx.x; x0 < width; x0 += kMpcAhead * step) {
      float v[kMpcAhead];
#pragma unroll
      for (int k = 0; k < kMpcAhead; ++k) {
        const int x = x0 + k * step;
        v[k] = x < width ? __ldg(row + x) : 0.f;
      }
#pragma unroll
      for (int k = 0; k < kMpcAhead; ++k) {
        if (x0 + k * step < width) {
          const float yk = v[k] - comp;
          const float tk = sum + yk;
          comp = (tk - sum) - yk;
          sum = tk;
        }
      }
    }
  }
  red[threadIdx.x] = sum;
  __syncthreads();
  if ((int)threadIdx.x < M) {
    float tot = 0.f, c2 = 0.f;
    for (int t = threadIdx.x; t < (int)blockDim.x; t += M) {
      const float yk = red[t] - c2;
      const float tk = tot + yk;
      c2 = (tk - tot) - yk;
      tot = tk;
    }
    part[(((size_t)s * M + py) * nch + ch) * M + threadIdx.x] = tot;
  }
}

// stage 2: every block rebuilds its slice's M x M map from the partials (fixed
// order) and divides its pixels by the map value of their phase when non-zero.
// A thread keeps its VEC columns, so their phases cost one modulo per thread
// instead of a division and two modulos per pixel, and walks down its block's
// rows kMpcRows at a time; the partials are staged with all threads' loads in
// flight (staged != 0) before the dependent sums.
constexpr int kMpcRows = 4;
constexpr int kMpcThreads = 128;
constexpr int kMpcStage = 8192;  // partials (floats) staged in shared memory
template <int VEC>
__global__ void __launch_bounds__(kMpcThreads)
    mpc_apply_kernel(float* __restrict__ img, int rowsM, int colsM, int M, int nch, int staged,
                     int rows_per_block, const float* __restrict__ part) {
  extern __shared__ float cmap[];  // [M * M], then the staged partials
  const int s = blockIdx.z;
  const int rows = rowsM / M, cols = colsM / M;
  const float inv_n = 1.f / (float)((long long)rows * cols);
  const float* ps = part + (size_t)s * M * nch * M;
  if (staged) {
    float* st = cmap + M * M;
    for (int k = threadIdx.x; k < M * nch * M; k += kMpcThreads) st[k] = __ldg(ps + k);
    __syncthreads();
    ps = st;
  }
  for (int k = threadIdx.x; k < M * M; k += kMpcThreads) {
    const int py = k / M, px = k % M;
    const float* pp = ps + (size_t)py * nch * M + px;
    float tot = 0.f, c2 = 0.f;
    for (int ch = 0; ch < nch; ++ch) {
      const float yk = pp[(size_t)ch * M] - c2;
      const float tk = tot + yk;
      c2 = (tk - tot) - yk;
      tot = tk;
    }
    cmap[k] = (rows * cols > 0) ? tot * inv_n : 0.f;
  }
  __syncthreads();
  const int x = (blockIdx.x * kMpcThreads + threadIdx.x) * VEC;
  if (x >= colsM) return;
  int ph[VEC];
  ph[0] = x % M;
#pragma unroll
  for (int k = 1; k < VEC; ++k) ph[k] = ph[k - 1] + 1 == M ? 0 : ph[k - 1] + 1;
  const int y1 = min(rowsM, (int)(blockIdx.y + 1) * rows_per_block);
  float* f = img + (size_t)s * rowsM * colsM + x;
  int y = blockIdx.y * rows_per_block;
  const float* crow = cmap + (y % M) * M;
  for (; y < y1; y += kMpcRows) {
    float v[kMpcRows][VEC];
#pragma unroll
    for (int r = 0; r < kMpcRows; ++r) {
      if (y + r >= y1) break;
      const float* q = f + (size_t)(y + r) * colsM;
      if constexpr (VEC == 4) {
        const float4 t = *reinterpret_cast<const float4*>(q);
        v[r][0] = t.x;
        v[r][1] = t.y;
        v[r][2] = t.z;
        v[r][3] = t.w;
      } else {
        v[r][0] = *q;
      }
    }
#pragma unroll
    for (int r = 0; r < kMpcRows; ++r) {
      if (y + r >= y1) break;
#pragma unroll
      for (int k = 0; k < VEC; ++k) {
        const float c = crow[ph[k]];
        if (c != 0.f) v[r][k] = __fdiv_rn(v[r][k], c);
      }
      float* q = f + (size_t)(y + r) * colsM;
      if constexpr (VEC == 4)
        *reinterpret_cast<float4*>(q) = make_float4(v[r][0], v[r][1], v[r][2], v[r][3]);
      else
        *q = v[r][0];
      crow += M;
      if (crow == cmap + M * M) crow = cmap;
    }
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
cudaError_t launch_to_float32(const void* src, int type, long long n, float* dst,
                              cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  switch (type) {
    case NX_TYPE_U8: return launch_to_float<uint8_t>(src, n, dst, s);
    case NX_TYPE_I8: return launch_to_float<int8_t>(src, n, dst, s);
    case NX_TYPE_U16: return launch_to_float<uint16_t>(src, n, dst, s);
    default: return launch_to_float<int16_t>(src, n, dst, s);
  }
}

cudaError_t launch_cr_shift_magnify(const float* in, int T, int H, int W, const float* shift_r,
                                    const float* shift_c, float mag_r, float mag_c, int rowsM,
                                    int colsM, float* out, cudaStream_t s) {
  const long long n = (long long)T * rowsM * colsM;
  if (n == 0) return cudaSuccess;
  if (mag_r >= 1.f && mag_c >= 1.f && T <= 65535 && rowsM / 32 < 65535) {
    // shared memory for the largest tile staging (32 rows at magnification 1,
    // or any tile cr_tile_rows picks: <= 72 KB); each launch uses what its
    // magnifications need
    static const size_t smem_max = std::max<size_t>(cr_tile_smem(32, 1.f, 1.f), 72 * 1024);
    static int attr_dev = -1;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (attr_dev != dev) {
      e = cudaFuncSetAttribute(cr_magnify_tiled_kernel,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max);
      if (e != cudaSuccess) return e;
      attr_dev = dev;
    }
    const int TR = cr_tile_rows(mag_r, mag_c);
    const int PR = cr_patch_extent(TR, mag_r), PC = cr_patch_extent(kCrTileCols, mag_c);
    const size_t smem = cr_tile_smem(TR, mag_r, mag_c);
    const dim3 grid((unsigned)((colsM + kCrTileCols - 1) / kCrTileCols),
                    (unsigned)((rowsM + TR - 1) / TR), (unsigned)T);
    cr_magnify_tiled_kernel<<<grid, kCrTileCols, smem, s>>>(in, H, W, shift_r, shift_c, mag_r,
                                                            mag_c, rowsM, colsM, TR, PR, PC, out);
    return cudaGetLastError();
  }
  cr_shift_magnify_kernel<<<grid_for(n), kBlock, 0, s>>>(in, T, H, W, shift_r, shift_c, mag_r,
                                                         mag_c, rowsM, colsM, out);
  return cudaGetLastError();
}

cudaError_t launch_roberts_cross(const float* in, int T, int H, int W, float* gc, float* gr,
                                 cudaStream_t s) {
  const long long n = (long long)T * H * W;
  if (n == 0) return cudaSuccess;
  roberts_cross_kernel<<<grid_for(n), kBlock, 0, s>>>(in, T, H, W, gc, gr);
  return cudaGetLastError();
}

RgcScalars rgc_scalars(int M, float radius, float sensitivity, int pad_edges) {
  RgcScalars sc{};
  const float sigma = (float)((double)radius / 2.355);
  const float fwhm = radius;
  sc.tSS = 2.0f * sigma * sigma;
  sc.tSO = 2.0f * sigma + 1.0f;
  sc.start = -(int)(2.0f * fwhm);
  sc.end = (int)(2.0f * fwhm + 1.0f);
  sc.margin = pad_edges ? 0 : (int)((double)fwhm * (double)M);
  sc.sens = sensitivity;
  if (!(sensitivity > 1.0f)) {
    sc.sens_mode = 0;
  } else if (sensitivity == std::floor(sensitivity) && sensitivity <= 16.0f) {
    sc.sens_mode = 1;
    sc.sens_int = (int)sensitivity;
  } else if (sensitivity - 0.5f == std::floor(sensitivity) && sensitivity <= 16.0f) {
    sc.sens_mode = 3;
    sc.sens_int = (int)sensitivity;
  } else {
    sc.sens_mode = 2;
  }
  return sc;
}

cudaError_t launch_rgc(const float* gc, const float* gr, const float* img, int T, int rowsM,
                       int colsM, int M, const RgcScalars& sc, int iw, float* out,
                       cudaStream_t s) {
  const long long n = (long long)T * rowsM * colsM;
  if (n == 0) return cudaSuccess;
  // the table form where the table fits (e.g. M = 5 up to R = 2, M = 2 up to 6;
  // 8 x 600 x 520, M = 2, R = 1.5: 97 against 409 us) and 32-bit positions hold
  const int W2 = sc.end - sc.start;
  const size_t table = (size_t)M * M * W2 * W2 * sizeof(float4);
  if (M <= 64 && table <= kRgcTableBytes && rowsM < (1 << 24) && colsM < (1 << 24)) {
    const RgcTile tile = rgc_tile(M, W2);
    const auto launch = [&](auto kernel) {
      if (tile.bytes > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(
            kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRgcSharedMax);
        if (e != cudaSuccess) return e;
      }
      const long long units =
          (long long)T * (((rowsM + M - 1) / M + kRgcTileRows - 1) / kRgcTileRows) *
          (((colsM + M - 1) / M + 31) / 32);
      // small images: several blocks per tile, so that every SM has two
      const int parts = (int)std::min<long long>(M * M, std::max(1LL, 2 * 152 / units));
      const dim3 grid((unsigned)std::min<long long>(units, 152LL * 8), (unsigned)parts);
      kernel<<<grid, kBlock, tile.bytes, s>>>(gc, gr, img, T, rowsM, colsM, M, sc, iw, tile,
                                              parts, out);
      return cudaGetLastError();
    };
    switch (W2) {
      case 3: return launch(rgc_table_kernel<3>);
      case 5: return launch(rgc_table_kernel<5>);
      case 7: return launch(rgc_table_kernel<7>);
      case 9: return launch(rgc_table_kernel<9>);
      case 11: return launch(rgc_table_kernel<11>);
      case 13: return launch(rgc_table_kernel<13>);
      default: return launch(rgc_table_kernel<0>);
    }
  }
  rgc_kernel<<<grid_for(n), kBlock, 0, s>>>(gc, gr, img, T, rowsM, colsM, M, sc, iw, out);
  return cudaGetLastError();
}

cudaError_t launch_gradient_radiality(const float* in, int T, int h, int w, float* gx, float* gy,
                                      cudaStream_t s) {
  const long long n = (long long)T * h * w;
  if (n == 0) return cudaSuccess;
  gradient_radiality_kernel<<<grid_for(n), kBlock, 0, s>>>(in, T, h, w, gx, gy);
  return cudaGetLastError();
}

RingCoords ring_coords(int M, float ring_radius) {
  // _le_radiality.pyx:92-104: float32 ring of 12 points at ringRadius * m
  RingCoords rc{};
  rc.radius = (float)((double)ring_radius * (double)M);
  const float step = (float)((3.14159265358979323846 * 2.0) / 12.0);
  for (int k = 0; k < 12; ++k) {
    const float arg = step * (float)k;
    rc.x[k] = (float)(std::cos((double)arg) * (double)rc.radius);
    rc.y[k] = (float)(std::sin((double)arg) * (double)rc.radius);
  }
  return rc;
}

cudaError_t launch_radiality(const float* gx, const float* gy, const float* img_interp, int T,
                             int h, int w, int M, const RingCoords& rc, int border, int positivity,
                             int iw, float* out, cudaStream_t s) {
  const long long n = (long long)T * h * M * w * M;
  if (n == 0) return cudaSuccess;
  radiality_kernel<<<grid_for(n), kBlock, 0, s>>>(gx, gy, img_interp, T, h, w, M, rc, border,
                                                  positivity, iw, out);
  return cudaGetLastError();
}

cudaError_t launch_record_push_frame(const float* frame, long long n, float* rec, int it,
                                     cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  record_push_frame_kernel<<<grid_for(n), kBlock, 0, s>>>(frame, n, rec, it);
  return cudaGetLastError();
}

cudaError_t launch_record_merge(float* acc, const float* rec, long long n, int n_acc, int n_blk,
                                int chunks, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const auto kernel = chunks == 1             ? record_merge_kernel<0>
                      : chunks <= kMergeGroup ? record_merge_kernel<1>
                                              : record_merge_kernel<2>;
  kernel<<<grid_for(n), kBlock, 0, s>>>(acc, rec, n, n_acc, n_blk, chunks);
  return cudaGetLastError();
}

bool merges_in_groups(const FinalizeJob& j) { return !j.chain && j.nchunks > kMergeGroup; }

cudaError_t launch_finalize_jobs(const FinalizeJob* jobs, int njobs, int total_blocks, bool groups,
                                 cudaStream_t s) {
  if (njobs == 0 || total_blocks == 0) return cudaSuccess;
  const auto kernel = groups ? finalize_jobs_kernel<true> : finalize_jobs_kernel<false>;
  kernel<<<total_blocks, kBlock, 0, s>>>(jobs, njobs);
  return cudaGetLastError();
}

cudaError_t launch_finalize(const float* rec, int F, int chunks, int T, int fpt, int n_tp,
                            long long n, int corr_mask, float* out, long long out_stride,
                            bool full, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const auto kernel = chunks > kMergeGroup ? finalize_kernel<true> : finalize_kernel<false>;
  for (int tp = 0; tp < n_tp; tp += 65535) {  // grid.y limit
    const int cnt = std::min(n_tp - tp, 65535);
    kernel<<<dim3(grid_for(n), (unsigned)cnt), kBlock, 0, s>>>(
        rec + (size_t)tp * chunks * F * n, F, chunks, T - tp * fpt, fpt, n, corr_mask,
        out + (size_t)tp * n, out_stride, full);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_temporal_stack(const float* stack, int T, long long n, int corr, float* out,
                                  cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const long long blocks = (n + kTcPix - 1) / kTcPix;
  // AVG reads the stack once in the per-pixel kernel already; VAR and TAC2
  // re-read it there, so they stage each pixel block in shared memory
  if (corr != NX_CORR_AVG && T >= 1 && T <= kTcMaxFrames && blocks <= 0x7fffffffLL) {
    // 16-byte copies need a 16-byte aligned base, whole 4-pixel pieces in every
    // frame (n % 4 == 0) and a whole last block
    const bool vec = (reinterpret_cast<uintptr_t>(stack) & 15u) == 0 && n % kTcPix == 0;
    static int attr_dev = -1;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (attr_dev != dev) {
      e = cudaFuncSetAttribute(temporal_stack_smem_kernel,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(kTcMaxFrames * kTcPix * sizeof(float)));
      if (e != cudaSuccess) return e;
      attr_dev = dev;
    }
    temporal_stack_smem_kernel<<<(unsigned)blocks, kTcPix, (size_t)T * kTcPix * sizeof(float),
                                 s>>>(stack, T, n, corr, vec, out);
    return cudaGetLastError();
  }
  temporal_stack_kernel<<<grid_for(n), kBlock, 0, s>>>(stack, T, n, corr, out);
  return cudaGetLastError();
}

cudaError_t launch_srrf_temporal(const float* stack, int T, long long n, int order, float* out,
                                 cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  srrf_temporal_kernel<<<grid_for(n), kBlock, 0, s>>>(stack, T, n, order, out);
  return cudaGetLastError();
}

cudaError_t launch_srrf_acrf_integrated(float* im, int T, long long n, int order,
                                        const AcrfSchedule& sch, float* out, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  srrf_acrf_integrated_kernel<<<grid_for(n), kBlock, 0, s>>>(im, T, n, order, sch, out);
  return cudaGetLastError();
}

// partial-sum chunks of the macro-pixel map per (slice, phase row)
static int mpc_chunks(int rowsM, int M) { return std::max(1, std::min(kMpcChunks, rowsM / M)); }

size_t mpc_scratch_bytes(int S, int rowsM, int M) {
  return (size_t)std::max(S, 1) * M * M * mpc_chunks(rowsM, M) * sizeof(float);
}

cudaError_t launch_mpc(float* img, int S, int rowsM, int colsM, int M, float* map,
                       cudaStream_t s) {
  if ((long long)S * rowsM * colsM == 0) return cudaSuccess;
  const int rows = rowsM / M;
  const int nch = mpc_chunks(rowsM, M);
  const int block = M <= 32 ? 32 * M : ((1024 / M) * M);
  if (rows > 0) {
    mpc_partial_kernel<<<dim3((unsigned)S, (unsigned)M, (unsigned)nch), block,
                         block * sizeof(float), s>>>(img, rowsM, colsM, M, nch, map);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  } else {
    cudaError_t e = cudaMemsetAsync(map, 0, (size_t)S * M * M * nch * sizeof(float), s);
    if (e != cudaSuccess) return e;
  }
  // float4 columns where every row starts on a 16-byte boundary
  const bool vec = colsM % 4 == 0 && (reinterpret_cast<uintptr_t>(img) & 15u) == 0;
  const int gx = (colsM + kMpcThreads * (vec ? 4 : 1) - 1) / (kMpcThreads * (vec ? 4 : 1));
  const int npart = M * M * nch;
  // staged only where map and partials fit 48 KB together: from m = 79 on they do not,
  // and the map alone (40 KB at m = 100) still does
  const int staged = npart <= kMpcStage && (M * M + npart) * sizeof(float) <= 48 * 1024;
  const size_t smem = (size_t)(M * M + (staged ? npart : 0)) * sizeof(float);
  // rows per block: enough blocks for the chip (2048), but no more than 64 rows
  // (a longer walk gains nothing once the map is a small part of it); and within
  // the grid.y limit.  100 x 1280 x 1280, m = 5, both kernels: 1361 -> 332 us
  // (5.9 TB/s over the two reads and the write); 10 x 2560 x 2560: 490 -> 150 us;
  // one 500 x 500 image: 18 -> 13 us.
  const long long want = (rowsM * (long long)S * gx + 2047) / 2048;
  const int rpb = (int)std::max<long long>(
      (rowsM + 65534) / 65535, std::max<long long>(kMpcRows, std::min<long long>(64, want)));
  const unsigned gy = (unsigned)((rowsM + rpb - 1) / rpb);
  for (int s0 = 0; s0 < S; s0 += 65535) {  // grid.z limit
    const int cnt = std::min(S - s0, 65535);
    float* im = img + (size_t)s0 * rowsM * colsM;
    const float* pm = map + (size_t)s0 * npart;
    const dim3 grid((unsigned)gx, gy, (unsigned)cnt);
    if (vec)
      mpc_apply_kernel<4><<<grid, kMpcThreads, smem, s>>>(im, rowsM, colsM, M, nch, staged, rpb, pm);
    else
      mpc_apply_kernel<1><<<grid, kMpcThreads, smem, s>>>(im, rowsM, colsM, M, nch, staged, rpb, pm);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace nx
