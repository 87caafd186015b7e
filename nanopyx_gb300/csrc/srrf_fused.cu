// Fused SRRF radiality kernel (sm_103a): one CTA owns a 32 x TY tile of input
// pixels, loops over frames, and per frame
//   1. stages the input tile + halo in shared memory,
//   2. forms the central-difference gradients   (_c_gradients.c:3-25),
//   3. Catmull-Rom-magnifies the intensity      (_c_interpolation_catmull_rom.c:21-52),
//   4. evaluates radiality over the 12-point ring for the thread's M outputs
//      (_c_sr_radiality.c:15-51): two Catmull-Rom interpolations of the gradient
//      per ring point from shared memory.
// The reference's ring positions depend on the output row only through
// y0 = (j + 0.5) + yRing and on the column only through x0 = (i + 0.5) + xRing, so
// the tap rows / columns and Catmull-Rom weights of every (output row, ring
// point) and (output column, ring point) are tabulated once per tile in shared
// memory, in the reference's own float32 arithmetic (x0 rounded, x0 / m IEEE).
//
// What bounds it: shared-memory wavefronts (column weights and row sums, 67 % of
// the pipe) and issue (59 %).  100 x 256 x 256, m = 5, ring 0.5 px: one frame a
// pass, all 12 row passes at once 4.98 ms; frame pairs on packed arithmetic with
// the row passes in groups 2.94; tile rows per magnification and chunks that fill
// the last wave 2.86; the next pass's input loaded behind the ring points 2.71;
// no comparisons in the ring sum 2.65 (2.68 with weak gradients kept exact).
#include <algorithm>
#include <atomic>
#include <cstring>

#include "common.cuh"
#include "internal.h"

namespace nx {

namespace {

constexpr int kRing = 12;
constexpr int kHalo = 5;  // input rows/cols around the tile: ring radius <= 2 px

// FP = 2: two consecutive frames per pass: the interpolation weights, ring tables and
// offsets of a pass serve both, and the arithmetic runs on packed f32x2 (the
// same IEEE operations per frame).  FP = 1: one, for one frame and for launches that leave
// SMs idle (see launch_srrf_m), where a pair is only a longer pass.
// V: a value of the pass's frames; Q: two of them (a gradient's x and y) as they lie
// in shared memory.
template <int FP>
struct Frames;
template <>
struct Frames<1> {
  using V = float;
  using Q = float2;
  __device__ static V all(float a) { return a; }
  __device__ static V fma(V a, V b, V c) { return __fmaf_rn(a, b, c); }
  __device__ static V mul(V a, V b) { return __fmul_rn(a, b); }
  template <class F>
  __device__ static V each(F f, V a) { return f(a); }
  template <class F>
  __device__ static V each(F f, V a, V b) { return f(a, b); }
  template <class F>
  __device__ static V of(F f) { return f(0); }
  __device__ static V x(const Q& q) { return q.x; }
  __device__ static V y(const Q& q) { return q.y; }
  __device__ static Q both(V x, V y) { return make_float2(x, y); }
  __device__ static float frame(V a, int) { return a; }
};
template <>
struct Frames<2> {
  using V = float2;
  using Q = float4;
  __device__ static V all(float a) { return make_float2(a, a); }
  __device__ static V fma(V a, V b, V c) { return __ffma2_rn(a, b, c); }
  __device__ static V mul(V a, V b) { return __fmul2_rn(a, b); }
  template <class F>
  __device__ static V each(F f, V a) { return make_float2(f(a.x), f(a.y)); }
  template <class F>
  __device__ static V each(F f, V a, V b) { return make_float2(f(a.x, b.x), f(a.y, b.y)); }
  template <class F>
  __device__ static V of(F f) { return make_float2(f(0), f(1)); }
  __device__ static V x(const Q& q) { return make_float2(q.x, q.y); }
  __device__ static V y(const Q& q) { return make_float2(q.z, q.w); }
  __device__ static Q both(V x, V y) { return make_float4(x.x, x.y, y.x, y.y); }
  __device__ static float frame(V a, int k) { return k ? a.y : a.x; }
};

template <int M, int FP>
struct SrrfTile {
  // tile rows, measured.  Pairs (100 x 256 x 256; m = 6, 8: 50 frames): m = 2: 4 / 8 / 12
  // rows 0.68 / 0.83 / 0.77 ms; m = 3: 2 / 4 / 8 rows 1.34 / 1.54 / 1.25; m = 4:
  // 2 / 4 / 6 rows 2.06 / 2.13 / 1.96; m = 5: 3 / 4 / 5 / 6 rows 3.13 / 2.86 /
  // 3.15 / 2.94; m = 6: 1 / 2 / 4 rows 2.48 / 2.55 / 1.97; m = 8: 1 / 2 / 3 rows
  // 3.68 / 3.49 / 3.69.  One frame of 30 x 30 and of 400 x 400, us: m = 3: 4 rows 12.5
  // and 66, 8 rows 16 and 71; m = 4: 4 / 5 / 6 rows 15 / 16 / 18 and 114 / 100 / 94;
  // m = 5: 4 / 5 / 6 rows 18 / 21 / 23 and 139 / 133 / 125; m = 6: 2 / 3 / 4 rows 16 /
  // 19 / 21 and 255 / 201 / 175; m = 8: 1 / 2 rows 19 / 20 and 353 / 324
  static constexpr int TY =
      FP == 2 ? (M == 2 ? 4 : M == 3 ? 8 : M == 4 ? 6 : M == 5 ? 4 : M == 6 ? 4 : 2)
              : (M == 4 || M == 5 ? 5 : M == 8 ? 2 : 4);
  static constexpr int TX = 32;
  static constexpr int NT = 32 * TY * M;
  static constexpr int IH = TY + 2 * kHalo;  // input tile rows
  static constexpr int IW = TX + 2 * kHalo;
  static constexpr int OY = TY * M, OX = TX * M;
  static constexpr int RIW = TX + 4;
  // ring points whose row pass is formed at a time: for pairs the buffer of a warp is
  // 1.3 KB instead of 8 for all 12 (100 x 256 x 256, m = 5: 2 / 3 / 4 points 2.71 / 2.78 /
  // 2.89 ms); a single frame's pass is too short to hide the waits between groups (one
  // 400 x 400 frame, 2 / 4 / 12 points 145 / 145 / 140 us)
  static constexpr int RG = FP == 2 ? 2 : 12;
  static constexpr int UR = FP == 2 ? 1 : 2;  // ring points unrolled
  static constexpr int al(int n) { return (n + 31) / 32 * 32; }
  static constexpr int O_IN = 0;                        // input tiles (FP frames)
  static constexpr int S_IN = al(IH * IW);
  static constexpr int O_G = O_IN + FP * S_IN;          // gradients Q (gx, gx', gy, gy')
  static constexpr int O_RI = O_G + al(IH * IW * 2 * FP);   // intensity row pass V (v, v')
  static constexpr int O_RW = O_RI + al(OY * RIW * FP);     // intensity row weights [OY][5]
  static constexpr int O_CW = O_RW + al(OY * 5);        // intensity col weights [OX][5]
  static constexpr int O_RT = O_CW + al(OX * 5);        // ring row taps [OY][12][8]
  // ring column taps of output column (lane, px) as 5 weights on the columns
  // cb .. cb + 4 of the row-pass buffer, cb = the first tap of px = 0 (the taps
  // of px = 1 .. M-1 start at cb or cb + 1): [ring][px][lane] float4 (weights
  // 0..3) and float (weight 4), lane-contiguous
  static constexpr int O_CW4 = O_RT + al(OY * kRing * 8);
  static constexpr int O_CW1 = O_CW4 + al(kRing * M * TX * 4);
  static constexpr int O_CB = O_CW1 + al(kRing * M * TX);  // [ring][lane] int: cb - x_start
  // per-warp row pass of the gradient interpolation: [ring of the group][IW]
  // Q, plus one zeroed Q after the last (read with weight 0)
  static constexpr int RBW = (RG * IW + 1) * 2 * FP;
  static constexpr int O_RB = O_CB + al(kRing * TX);
  static constexpr int FLOATS = O_RB + (NT / 32) * RBW;
  static constexpr size_t SMEM = size_t(FLOATS) * 4;
};

struct SrrfParams {
  const float* in;      // (T, h, w)
  const float* interp;  // (T, h*M, w*M) magnified intensity, or nullptr: computed here
  float* out;           // (T, h*M, w*M)
  int T, h, w;
  int tiles_x, tiles_y;
  int chunks;           // frame chunks (grid y)
  int border, positivity, iw;
  float rr;         // ring radius * M (float, as the reference)
  float inv_rr;     // 1 / rr
  float xr[kRing], yr[kRing];
};

// ring tap entry: [0] first tap index (int bits), [1..4] weights, [5] centre
// minus ring point (yc - y0 or xc - x0), [6] inside flag (1 / 0)
__device__ __forceinline__ void ring_entry(float* e, float c, float ring, int M, int n) {
  const float p0 = __fadd_rn(c, ring);
  const float r = __fdiv_rn(p0, (float)M);
  const int ri = (int)floorf(r - 0.5f);
  e[0] = __int_as_float(ri - 1);
#pragma unroll
  for (int t = 0; t < 4; ++t) e[1 + t] = cr_cubic(r - ((float)(ri - 1 + t) + 0.5f));
  e[5] = __fsub_rn(c, p0);
  e[6] = (r >= 0.f && r < (float)n) ? 1.f : 0.f;
  e[7] = 0.f;
}

// Added to every squared gradient: keeps rsqrt finite without one, and no more
// than a squared gradient's own rounding (an ulp up to 2^-125, half an ulp and
// less above), so that radiality does not depend on a stack's units.
constexpr float kTiny = 1.40129846e-45f;  // 2^-149, the smallest float

// v >= 0 with the sign of s
__device__ __forceinline__ float with_sign(float v, float s) {
  return __int_as_float(__float_as_int(v) | (__float_as_int(s) & 0x80000000));
}

template <int M, int FP>
__global__ void __launch_bounds__(SrrfTile<M, FP>::NT, 1) srrf_fused_kernel(const SrrfParams p) {
  using G = SrrfTile<M, FP>;
  using F = Frames<FP>;
  using V = typename F::V;
  using Q = typename F::Q;
  constexpr int TY = G::TY;
  extern __shared__ __align__(128) float sm[];
  float* tin = sm + G::O_IN;
  Q* grad = reinterpret_cast<Q*>(sm + G::O_G);
  V* ri = reinterpret_cast<V*>(sm + G::O_RI);
  float* rw = sm + G::O_RW;
  float* cw = sm + G::O_CW;
  float* rt = sm + G::O_RT;
  float4* cw4 = reinterpret_cast<float4*>(sm + G::O_CW4);
  float* cw1 = sm + G::O_CW1;
  int* cbt = reinterpret_cast<int*>(sm + G::O_CB);
  Q* rb = reinterpret_cast<Q*>(sm + G::O_RB + (threadIdx.x >> 5) * G::RBW);

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int ty = warp % TY;
  const int py = warp / TY;
  const int tile = blockIdx.x;
  // chunks of whole passes (the last one may hold one frame of two)
  const int passes = (p.T + FP - 1) / FP;
  const int f_begin = FP * (int)((long long)blockIdx.y * passes / p.chunks);
  const int f_end = min(p.T, FP * (int)((long long)(blockIdx.y + 1) * passes / p.chunks));
  const int nx0 = (tile % p.tiles_x) * G::TX;
  const int ny0 = (tile / p.tiles_x) * TY;
  const int h = p.h, w = p.w;
  const int rowsM = h * M, colsM = w * M;
  const int y_start = ny0 - kHalo, x_start = nx0 - kHalo;

  // ---- per-tile tables ------------------------------------------------------
  for (int i = tid; i < G::OY; i += G::NT) {
    const int yM = ny0 * M + i;
    const int nyo = ny0 + i / M;
    const float ry = __fdiv_rn((float)yM, (float)M);
    const int rb = (int)floorf(ry - 0.5f);
    float w5[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int k = rb - 1 + t - (nyo - 2);
      const float wt = cr_cubic(ry - ((float)(rb - 1 + t) + 0.5f));
#pragma unroll
      for (int kk = 0; kk < 5; ++kk) w5[kk] = (k == kk) ? wt : w5[kk];
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) rw[i * 5 + k] = w5[k];
    const float yc = (float)yM + 0.5f;
    for (int s = 0; s < kRing; ++s) ring_entry(rt + (i * kRing + s) * 8, yc, p.yr[s], M, h);
  }
  for (int i = tid; i < G::OX; i += G::NT) {
    const int xM = nx0 * M + i;
    const int nxo = nx0 + i / M;
    const float rx = __fdiv_rn((float)xM, (float)M);
    const int cb = (int)floorf(rx - 0.5f);
    float w5[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int k = cb - 1 + t - (nxo - 2);
      const float wt = cr_cubic(rx - ((float)(cb - 1 + t) + 0.5f));
#pragma unroll
      for (int kk = 0; kk < 5; ++kk) w5[kk] = (k == kk) ? wt : w5[kk];
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) cw[i * 5 + k] = w5[k];
  }
  for (int i = tid; i < kRing * G::TX; i += G::NT) {
    const int s = i / G::TX, ln = i % G::TX;
    int cb = 0;
    for (int px = 0; px < M; ++px) {
      float e[8];
      ring_entry(e, (float)((nx0 + ln) * M + px) + 0.5f, p.xr[s], M, w);
      const int c0 = __float_as_int(e[0]);
      if (px == 0) cb = c0;
      // 0 or 1: the M phases of one lane span less than one input pixel
      const int off = min(max(c0 - cb, 0), 1);
      // a column outside the image contributes nothing (the reference skips
      // it): all its weights are zero
      float w5[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
      if (e[6] != 0.f) {
#pragma unroll
        for (int u = 0; u < 4; ++u) w5[u + off] = e[1 + u];
      }
      cw4[(s * M + px) * G::TX + ln] = make_float4(w5[0], w5[1], w5[2], w5[3]);
      cw1[(s * M + px) * G::TX + ln] = w5[4];
    }
    cbt[s * G::TX + ln] = cb - x_start;
  }
  if ((tid & 31) == 0) rb[G::RG * G::IW] = F::both(F::all(0.f), F::all(0.f));

  const int ny = ny0 + ty, nx = nx0 + lane;
  const int j = ny * M + py;  // output row
  const int lo_j = (1 + p.border) * M, hi_j = (h - 1 - p.border) * M;
  const int lo_i = (1 + p.border) * M, hi_i = (w - 1 - p.border) * M;
  const bool row_ok = j >= lo_j && j < hi_j && ny < h;
  const float* rrow = rt + ((ty * M + py) * kRing) * 8;
  const size_t plane = (size_t)rowsM * colsM;

  const bool own_intensity = p.interp == nullptr;
  // the next pass's input values, loaded while the current pass computes
  constexpr int NPF = (G::IH * G::IW + G::NT - 1) / G::NT;
  V pf[NPF];
  auto fetch = [&](int f) {
    const float* src = p.in + (size_t)f * h * w;
    const float* src1 = f + 1 < f_end ? src + (size_t)h * w : src;  // FP = 2
#pragma unroll
    for (int k = 0; k < NPF; ++k) {
      const int i = tid + k * G::NT;
      const int r = y_start + i / G::IW, c = x_start + i % G::IW;
      const bool in = i < G::IH * G::IW && r >= 0 && r < h && c >= 0 && c < w;
      const size_t o = (size_t)r * w + c;
      pf[k] = in ? F::of([&](int fr) { return __ldg((fr ? src1 : src) + o); }) : F::all(0.f);
    }
  };
  if (f_begin < f_end) fetch(f_begin);
  for (int f = f_begin; f < f_end; f += FP) {
    const bool two = FP == 2 && f + 1 < f_end;  // an odd last frame stands in for its partner
    __syncthreads();  // tables ready / previous pass's shared data consumed
#pragma unroll
    for (int k = 0; k < NPF; ++k) {
      const int i = tid + k * G::NT;
      if (i < G::IH * G::IW) {
#pragma unroll
        for (int fr = 0; fr < FP; ++fr) tin[fr * G::S_IN + i] = F::frame(pf[k], fr);
      }
    }
    if (f + FP < f_end) fetch(f + FP);
    __syncthreads();
    // gradients (zero outside rows/cols 1..n-2) and the intensity row pass
    for (int i = tid; i < G::IH * G::IW; i += G::NT) {
      const int rl = i / G::IW, cl = i % G::IW;
      const int r = y_start + rl, c = x_start + cl;
      Q g = F::both(F::all(0.f), F::all(0.f));
      if (r >= 1 && r < h - 1 && c >= 1 && c < w - 1 && rl >= 1 && rl < G::IH - 1 && cl >= 1 &&
          cl < G::IW - 1) {
        const float* t = tin + i;
        g = F::both(F::of([&](int fr) {
                      return __fadd_rn(-t[fr * G::S_IN - 1], t[fr * G::S_IN + 1]);
                    }),
                    F::of([&](int fr) {
                      return __fadd_rn(-t[fr * G::S_IN - G::IW], t[fr * G::S_IN + G::IW]);
                    }));
      }
      grad[i] = g;
    }
    for (int i = tid; own_intensity && i < G::OY * G::RIW; i += G::NT) {
      const int oy = i / G::RIW, cc = i % G::RIW;
      const int nyo = ny0 + oy / M;
      const float* w5 = rw + oy * 5;
      const float* col = tin + (nyo - 2 - y_start) * G::IW + (nx0 - 2 + cc - x_start);
      V sum = F::all(0.f);
#pragma unroll
      for (int k = 0; k < 5; ++k)
        sum = F::fma(F::all(w5[k]), F::of([&](int fr) { return col[fr * G::S_IN + k * G::IW]; }),
                     sum);
      ri[i] = sum;
    }
    __syncthreads();
    V div[M];
#pragma unroll
    for (int px = 0; px < M; ++px) div[px] = F::all(0.f);
    const float yc = (float)j + 0.5f;
#pragma unroll 1
    for (int sg = 0; sg < kRing; sg += G::RG) {
      // row pass of the ring interpolation: the ring points of this warp's output
      // row share their tap rows and weights, so each (ring point, tile column)
      // sum over the 4 tap rows is formed once per warp (same fma order as the
      // 16-tap form: rows first, then columns)
      __syncwarp();
      for (int idx = lane; idx < G::RG * G::IW; idx += 32) {
        const int s = idx / G::IW, c = idx - s * G::IW;
        const float4 rA = *reinterpret_cast<const float4*>(rrow + (sg + s) * 8);
        const float4 rB = *reinterpret_cast<const float4*>(rrow + (sg + s) * 8 + 4);
        V vx = F::all(0.f), vy = vx;
        if (rB.z != 0.f) {
          const int r0 = __float_as_int(rA.x) - y_start;
          const float wr[4] = {rA.y, rA.z, rA.w, rB.x};
          const Q* gp = grad + r0 * G::IW + c;
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const Q g = gp[t * G::IW];
            const V wt = F::all(wr[t]);
            vx = F::fma(F::x(g), wt, vx);
            vy = F::fma(F::y(g), wt, vy);
          }
        }
        rb[idx] = F::both(vx, vy);
      }
      __syncwarp();
      // radiality of this thread's M outputs, ring point by ring point: the M
      // columns share one window of 5 row-pass columns (cb .. cb + 4), each
      // output weights it with its own 5-vector (its 4 taps and a zero), which
      // is the 4-tap fma sequence of the reference with a + 0 at one end
#pragma unroll G::UR
      for (int s = sg; s < sg + G::RG; ++s) {
        const float dy = __fsub_rn(yc, __fadd_rn(yc, p.yr[s]));  // yc - y0
        const Q* rp = rb + (s - sg) * G::IW + cbt[s * G::TX + lane];
        Q col[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) col[k] = rp[k];
#pragma unroll
        for (int px = 0; px < M; ++px) {
          const float4 wa = cw4[(s * M + px) * G::TX + lane];
          const float we = cw1[(s * M + px) * G::TX + lane];
          const float wv[5] = {wa.x, wa.y, wa.z, wa.w, we};
          const float xc = (float)(nx * M + px) + 0.5f;
          const float dx = __fsub_rn(xc, __fadd_rn(xc, p.xr[s]));  // xc - x0
          V vgx = F::all(0.f), vgy = vgx;
#pragma unroll
          for (int k = 0; k < 5; ++k) {
            const V wk = F::all(wv[k]);
            vgx = F::fma(F::x(col[k]), wk, vgx);
            vgy = F::fma(F::y(col[k]), wk, vgy);
          }
          // dk = (1 - |vGy (xc - x0) - vGx (yc - y0)| / GMag / ringRadius)^2, 0
          // without a gradient; subtracted where the gradient points outwards.
          // No comparisons (the ALU pipe was the busiest): rsqrt is 2^74.5 of
          // kTiny alone and at most 2^74 with a gradient, so a saturating FMA
          // of it turns "any gradient" into 0 or 1, and the sign of the
          // inward component (+0, never -0, where there is none: ring radius 0)
          // is moved onto dk by a logic operation.
          const V g2 = F::fma(vgx, vgx, F::fma(vgy, vgy, F::all(kTiny)));
          const V rs = F::each([](float v) { return rsqrtf(v); }, g2);
          constexpr float kAnySlope = -2.11758237e-22f;  // -2^-72: 2^74.5 -> -5.66, 2^74 -> -4
          const V any =
              F::each([](float v) { return __saturatef(__fmaf_rn(v, kAnySlope, 5.3f)); }, rs);
          const V cr = F::fma(vgy, F::all(dx), F::mul(vgx, F::all(-dy)));
          V dk = F::fma(F::each([](float v) { return fabsf(v); }, cr),
                        F::mul(rs, F::all(-p.inv_rr)), F::all(1.f));
          dk = F::mul(dk, dk);
          const V in = F::fma(vgx, F::all(-p.xr[s]),
                              F::fma(vgy, F::all(-p.yr[s]), F::all(0.f)));
          dk = F::each(with_sign, dk, in);
          div[px] = F::fma(any, dk, div[px]);
        }
      }
    }
#pragma unroll
    for (int px = 0; px < M; ++px) {
      const int i = nx * M + px;  // output column
      V val = F::all(0.f);
      const size_t o = (size_t)f * plane + (size_t)j * colsM + i;
      if (row_ok && nx < w && i >= lo_i && i < hi_i) {
        val = F::each([](float v) { return v / 12.f; }, div[px]);
        if (p.positivity) val = F::each([](float v) { return fmaxf(v, 0.f); }, val);
        if (p.iw) {
          if (own_intensity) {
            // column pass of the intensity magnification (5 taps of the row pass)
            const float* w5 = cw + (lane * M + px) * 5;
            const V* rr = ri + (ty * M + py) * G::RIW + lane;
            V sum = F::all(0.f);
#pragma unroll
            for (int k = 0; k < 5; ++k) sum = F::fma(F::all(w5[k]), rr[k], sum);
            val = F::mul(val, sum);
          } else {
            val = F::of([&](int fr) {
              return fr && !two ? 0.f
                                : F::frame(val, fr) * __ldg(p.interp + o + (fr ? plane : 0));
            });
          }
        }
      }
      if (ny < h && nx < w) {
        p.out[o] = F::frame(val, 0);
        if (two) p.out[o + plane] = F::frame(val, 1);
      }
    }
  }
}

// blocks of a kernel resident on an SM, its shared memory allowed; asked once per device
template <int M, int FP>
cudaError_t srrf_resident(int dev, int* per_sm) {
  using G = SrrfTile<M, FP>;
  static std::atomic<int> known{-1};  // dev << 8 | blocks
  const int k = known.load(std::memory_order_relaxed);
  if (k >= 0 && k >> 8 == dev) {
    *per_sm = k & 255;
    return cudaSuccess;
  }
  cudaError_t e = cudaFuncSetAttribute(srrf_fused_kernel<M, FP>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::SMEM);
  if (e != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, srrf_fused_kernel<M, FP>, G::NT,
                                                    G::SMEM);
  if (e != cudaSuccess) return e;
  *per_sm = std::min(std::max(*per_sm, 1), 255);
  known.store(dev << 8 | *per_sm, std::memory_order_relaxed);
  return cudaSuccess;
}

// frame chunks: the count with the fewest passes on the busiest SM, a block
// costing its passes plus about one pass for its tables
int srrf_chunks(long long tiles, long long passes, long long slots) {
  long long best = -1;
  int chunks = 1;
  for (long long c = 1; c <= std::min<long long>(passes, 64); ++c) {
    const long long cost = (tiles * c + slots - 1) / slots * ((passes + c - 1) / c + 1);
    if (best < 0 || cost < best) {
      best = cost;
      chunks = (int)c;
    }
  }
  return chunks;
}

template <int M, int FP>
cudaError_t launch_srrf_f(const SrrfParams& prm, int dev, int sms, cudaStream_t s) {
  using G = SrrfTile<M, FP>;
  SrrfParams q = prm;
  q.tiles_x = (prm.w + G::TX - 1) / G::TX;
  q.tiles_y = (prm.h + G::TY - 1) / G::TY;
  int per_sm = 1;
  cudaError_t e = srrf_resident<M, FP>(dev, &per_sm);
  if (e != cudaSuccess) return e;
  const long long tiles = (long long)q.tiles_x * q.tiles_y;
  q.chunks = srrf_chunks(tiles, ((long long)prm.T + FP - 1) / FP, (long long)sms * per_sm);
  srrf_fused_kernel<M, FP><<<dim3((unsigned)tiles, (unsigned)q.chunks), G::NT, G::SMEM, s>>>(q);
  return cudaGetLastError();
}

template <int M>
cudaError_t launch_srrf_m(const SrrfParams& prm, cudaStream_t s) {
  using G = SrrfTile<M, 1>;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // one frame a pass where there is one only (400 x 400, m = 5: 133 us, 182 as a pair of
  // its own), or where every frame's tile finds an SM of its own (two frames of 64 x 64:
  // 21 us, 23 as a pair); beyond that pairs (two frames of 200 x 200: 64 us, two single
  // ones 80)
  const long long tiles = (long long)((prm.w + G::TX - 1) / G::TX) * ((prm.h + G::TY - 1) / G::TY);
  if (prm.T == 1 || tiles * prm.T <= sms) return launch_srrf_f<M, 1>(prm, dev, sms, s);
  return launch_srrf_f<M, 2>(prm, dev, sms, s);
}

}  // namespace

// fused radiality for m in {2, 3, 4, 5, 6, 8} and ring radius <= 2 px; returns
// cudaErrorNotSupported otherwise (the caller then uses the per-pixel kernel)
cudaError_t launch_srrf_fused(const float* in, const float* img_interp, int T, int h, int w,
                              int M, const RingCoords& rc, float ring_radius, int border,
                              int positivity, int iw, float* out, cudaStream_t s) {
  if (!(ring_radius >= 0.f && ring_radius <= 2.0f)) return cudaErrorNotSupported;
  SrrfParams p;
  memset(&p, 0, sizeof(p));
  p.in = in;
  p.interp = img_interp;
  p.out = out;
  p.T = T;
  p.h = h;
  p.w = w;
  p.border = border;
  p.positivity = positivity;
  p.iw = iw;
  p.rr = rc.radius;
  // a ring below 2^-26 leaves every centre where it is, (xc + xr) - xc = 0, so its term
  // is 1 for any factor; 0 keeps 2^74.5 / rr finite
  p.inv_rr = rc.radius >= 1.49e-8f ? 1.f / rc.radius : 0.f;
  for (int k = 0; k < kRing; ++k) {
    p.xr[k] = rc.x[k];
    p.yr[k] = rc.y[k];
  }
  if ((long long)T * h * w == 0) return cudaSuccess;
  switch (M) {
    case 2: return launch_srrf_m<2>(p, s);
    case 3: return launch_srrf_m<3>(p, s);
    case 4: return launch_srrf_m<4>(p, s);
    case 5: return launch_srrf_m<5>(p, s);
    case 6: return launch_srrf_m<6>(p, s);
    case 8: return launch_srrf_m<8>(p, s);
    default: return cudaErrorNotSupported;
  }
}

}  // namespace nx
