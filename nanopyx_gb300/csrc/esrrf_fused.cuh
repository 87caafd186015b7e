// Fused eSRRF frame-loop kernel (sm_103a), warp-specialised.
//
// One CTA works through units -- (stack, 32 x TY tile of input pixels = a
// 32M x TY*M tile of output pixels, timepoint, frame chunk) -- two or four
// frames per pass.  Its producer warps, per pass,
//   1. receive the input tiles + halo by TMA (mbarrier), or by plain loads when
//      the row pitch is not 16-byte aligned;
//   2. compute Roberts-Cross gradients          (_c_gradients.c:53-73) and the
//      row pass of the intensity magnification  (_c_interpolation_catmull_rom.c:21-52);
//   3. Catmull-Rom-interpolate the gradients on the half-pixel grid -- the only
//      positions the reference RGC ever reads from its 2m-magnified gradient
//      images (rows/cols k*m, clamped to 2*m*H-1;
//      _c_sr_radial_gradient_convergence.c:45-61) -- walking down columns, and
//      normalise them into a double-buffered slot;
// while its consumer warps, one thread per input pixel and output row phase,
//   4. evaluate RGC for the thread's M output pixels with FP64-derived phase
//      tables of the distance weights      (_c_sr_radial_gradient_convergence.c:17-90),
//      on packed f32x2 arithmetic (two frames in one register pair);
//   5. apply ^sensitivity, the intensity (column pass) and the margin, and
//      either write the per-frame value (eSRRF_ST stack) or fold it into
//      per-pixel streaming temporal moments kept in shared memory (Welford
//      mean and M2, lag-1 co-moment, last and first value as deviations; see
//      Moments).
// Nothing of size (T, 2Hm, 2Wm) or (T, Hm, Wm) is ever materialised for the
// temporal modes.
//
// What bounds it: the register reads and FMA pipe of step 4 (see rgc_sample).
// 100 x 512 x 512, m = 5, R = 1.5, VAR + TAC2, of 5.79 ms: the RGC core 4.9,
// the epilogue 0.5, the producers 0.35 (each found by leaving the others out).
// How that kernel got there from 7.66 ms:
//   saturating half-plane test, mirrored table entries           7.14
//   gradients walked down columns instead of a column pass, its
//   buffer and a row pass; 4 frames a pass in the shared memory
//   that frees; intensity rows 5 outputs at a time               6.31
//   epilogue in whole blocks (power, intensity, then moments):
//   no register spills                                           5.79
#pragma once

#include <cuda.h>

#include <algorithm>

#include "common.cuh"

namespace nx {

enum FusedMode : int { kModeStack = 0, kModeSum = 1, kModeFull = 2 };

__host__ __device__ constexpr int mode_fields(int mode) {
  return mode == kModeFull ? 5 : (mode == kModeSum ? 1 : 0);
}

constexpr int kMaxSens = 4;    // sensitivities sharing one RGC pass (AVG mode)
constexpr int kMaxTmaps = 24;  // TMA descriptors carried in the kernel parameters

struct FusedParams {
  const float* in;     // (T, H, W)
  int T, H, W;
  int rowsM, colsM;
  int tiles_x;
  int fpt;             // frames per timepoint
  int n_tp;            // number of timepoints
  int chunks;          // chunks per timepoint (the last timepoint uses min(chunks, its frames))
  int margin;
  int iw;
  float cy[4], cx[4];  // taps (rows H-2 .. H+1, cols W-2 ..) of the clamped index 2H / 2W
  const float* tbl;      // [M][2J+1][3][NS4*4]  (a = dx*w/d, b = dy*w/d, w) per sample
  const float* inv_wsum; // [M][M]
  const float* wfull;    // [M][M][2J+1][2J+1]
  float* out;            // stack (T, rowsM, colsM) or records [n_tp*chunks][F][rowsM][colsM]
  unsigned* status;
  int tmap;              // index into the kernel's TMA descriptor pack, or -1: plain loads
  int tiles_y;
  int F;                 // record fields: 5 (VAR/TAC2) or n_sens (AVG: the mean per sensitivity)
  int n_sens;            // AVG mode: sensitivities evaluated on the same RGC (others: 1)
  int sens_mode_k[kMaxSens];  // see apply_sensitivity (common.cuh)
  int sens_int_k[kMaxSens];
  float sens_k[kMaxSens];
  unsigned long long wait_ns;  // bound of every producer/consumer wait (0: kWaitLimitNs)
  // failure-detection self-test only (0 in every computation): the producers
  // withhold the `full` arrival of the first pass of each CTA's first unit, so
  // the consumers' bounded wait runs out and the CTA takes its abort path
  int test_withhold_full;
};

struct TmapPack {
  CUtensorMap m[kMaxTmaps];
};

// Work list of one launch: units = (item, tile, timepoint, frame chunk), tiles
// fastest.  One item may be carried by value (`single`); several live in
// device memory with their first unit index in `unit_start`.  With `counter`
// CTAs take units dynamically (persistent launch), else unit = blockIdx.x.
struct UnitTable {
  const FusedParams* items;
  const int* unit_start;  // [n_items + 1]
  int n_items;
  int total_units;
  unsigned* counter;
  int ns_cap;  // largest n_sens among the items (sizes the AVG-mode temporal state)
  FusedParams single;
};

// Warp roles of the eSRRF kernel.  Each CTA runs 32 * TY * M / PYT consumer
// threads (one per input pixel and PYT output row phases: RGC, normalisation,
// temporal update) and producer warps that prepare the gradient and intensity
// tiles of the next frames (TMA, Roberts-Cross, Catmull-Rom passes,
// normalisation) into a double-buffered slot while the consumers work on the
// current one, so the two overlap on the SM.
template <int M, int V = 0>
struct EsrrfTile {
  // rows per tile: as many consumer warps as the registers allow without
  // spilling
  static constexpr int TY = (M <= 2) ? 8 : (M <= 5 ? 4 : (M == 6 ? 2 : 1));
  // output row phases per consumer thread: both at m = 2, where a gradient
  // sample meets only 4 outputs and its loads (shared by the phases of a thread)
  // fill the shared-memory pipe.  100 x 512 x 512, R = 1.5, VAR: 1.32 ms with
  // one phase and 384 producer threads, 1.25 ms with two and 256 (384: 1.28,
  // 512: 1.48).  At m = 3 .. 8 one phase and the threads it gives are better
  // (m = 3: 0.64 against 0.70 ms, m = 6: 1.09 / 1.44, m = 8: 2.06 / 2.00).
  static constexpr int PYT = M == 2 ? 2 : 1;
  // producer threads: the preparation per input pixel is the same for every m
  // while the RGC work grows with m^2, so small m needs more producers
  // (m = 3, 128 / 256 threads: 0.71 / 0.64 ms; m = 4: 0.70 / 0.65 at R = 1 and
  // 2.20 / 2.23 at R = 2.5; m = 5, 96 / 128 / 160: 6.04 / 5.84 / 6.07).
  // Tile variant V = 1 (instantiated for m = 2, 4, 5) has one producer warp
  // group fewer (m = 5: 3 warps), for the tiling autotuner to weigh against
  // the default on a given batch.
  static constexpr int NP_DEFAULT = M == 1 ? 384 : (M <= 4 ? 256 : 128);
  static constexpr int NP_ALT = M == 1 ? 256 : (M <= 4 ? 128 : 96);
  static constexpr int NP = V == 0 ? NP_DEFAULT : NP_ALT;
  // most frames a pass carries (4 where the layout fits shared memory, else 2)
  static constexpr int FP_MAX = 4;
  // one CTA per SM: registers for the consumers (m = 8 with 2 CTAs per SM at
  // 80 registers measured 11 % slower than 1 CTA)
  static constexpr int MIN_BLOCKS = 1;
};

// Frames per pass (FP = 2 or 4): a consumer carries FP / 2 pairs of consecutive
// frames through each pass.  The RGC core runs on packed f32x2 arithmetic (a
// frame pair in one register pair) and every phase-table load serves all the
// pairs; the temporal state is read and written once per pass.
template <int M, int J, int TY, int FP, int NP_ = EsrrfTile<M>::NP, int PYT_ = EsrrfTile<M>::PYT>
struct Geo {
  static constexpr int TX = 32;
  static constexpr int W2 = 2 * J + 1;
  static constexpr int NQ = 2 * J + 2;
  static constexpr int NPR = FP / 2;  // frame pairs per pass
  static constexpr int PYT = PYT_;
  static constexpr int HG_R = 2 * TY + 2 * J;
  static constexpr int HGP = TX + J;
  static constexpr int RLO = (J + 1) / 2 + 2;
  static constexpr int RHI = TY + (J - 1) / 2 + 2;
  static constexpr int NRY = RLO + RHI;
  static constexpr int CLO = (J + 1) / 2 + 2;
  static constexpr int CHI = TX + (J - 1) / 2 + 2;
  static constexpr int NCX = CLO + CHI;
  static constexpr int IY = RLO + 1;
  static constexpr int BH = NRY + 1;
  static constexpr int IX = ((CLO + 1 + 3) / 4) * 4;
  static constexpr int BW = ((IX + CHI + 3) / 4) * 4;
  static constexpr int NS = M * W2;
  static constexpr int NS4 = (NS + 3) / 4;
  static constexpr int OY = TY * M;
  static constexpr int OX = TX * M;
  static constexpr int RIW = TX + 4;
  static constexpr int NTC = 32 * TY * (M / PYT);  // consumer threads
  static constexpr int NP = NP_;                   // producer threads
  static constexpr int NT = NTC + NP;
  // prepared passes in flight between producers and consumers (3 or 4
  // measured no faster: the producers keep up)
  static constexpr int NSLOT = 2;
  // phase-table block per (py, jj): NE float4 entries, one per mirrored couple
  // of samples (see rgc_core), each value broadcast into a frame pair
  static constexpr int NE = (J + 1) * M + (M + 1) / 2;
  // unit gradients of one slot: one plane per frame pair of float4
  // (nx, nx', ny, ny')
  static constexpr int HG_PLANE = HG_R * 2 * HGP;  // samples per plane
  // the gradient walk (see Producer::gradients): steps along an axis that each
  // yield up to two half-grid samples, and rows of steps per walk
  static constexpr int NB = TX + J + (J & 1);
  static constexpr int NA = TY + J + (J & 1);
  static constexpr int SEG = 4;
  static constexpr int NSEG = (NA + SEG - 1) / SEG;
  static constexpr int LEFT = NB - 32;  // columns beyond one warp

  __host__ __device__ static constexpr int al(int n) { return (n + 31) / 32 * 32; }
  // shared-memory layout (in floats, 128-byte aligned blocks)
  static constexpr int O_INB = 0;
  static constexpr int S_INB = al(BH * BW);  // FP input tiles
  static constexpr int O_G = O_INB + FP * S_INB;
  static constexpr int S_G = al(NRY * NCX * 4);  // per frame pair: (gc, gc', gr, gr')
  static constexpr int O_HG = O_G + NPR * S_G;
  static constexpr int S_HG = al(HG_PLANE * 4) * NPR;   // one slot
  static constexpr int O_RI = O_HG + NSLOT * S_HG;      // NSLOT slots
  static constexpr int S_RI = al(OY * RIW * 2);  // intensity row pass per frame pair (v, v')
  static constexpr int O_TB = O_RI + NSLOT * NPR * S_RI;  // NSLOT slots of NPR planes
  static constexpr int S_TB = al(M * W2 * NE * 4);
  static constexpr int O_RW = O_TB + S_TB;
  static constexpr int S_RW = al(OY * 8);      // 5 weights per output row, rows of 8
  static constexpr int O_CW = O_RW + S_RW;
  static constexpr int S_CW = al(OX * 5);
  // per-output temporal state kept out of registers, [output][consumer] planes:
  //   FULL: float4 (mean, M2, C, A) then float B;  SUM: the mean per sensitivity
  static constexpr int NO = PYT * M;           // outputs per consumer
  static constexpr int O_TW = O_CW + S_CW;     // 1 / sum w per output
  static constexpr int O_TK = O_TW + NO * NTC;
  static constexpr int S_TK_FULL = 5 * NO * NTC;
  static constexpr int O_BAR_FULL = O_TK + S_TK_FULL;
  // AVG mode keeps the running mean of ns_cap sensitivities per output
  __host__ __device__ static constexpr int o_bar(int mode, int ns_cap) {
    return mode == 1 ? O_TK + ns_cap * NO * NTC : (mode == 2 ? O_BAR_FULL : O_TK);
  }
  // 2 NSLOT + 2 mbarriers after o_bar
  __host__ __device__ static constexpr size_t smem_bytes(int mode, int ns_cap) {
    return size_t(o_bar(mode, ns_cap) + 32) * 4;
  }
};

constexpr size_t kMaxSmemPerBlock = 227 * 1024;
constexpr size_t kSmemBudget = kMaxSmemPerBlock - sizeof(FusedParams) - 64;

// compile-time configuration of one instantiation
template <int M, int J, int MODE, int V = 0>
struct FusedCfg {
  static constexpr int TY = EsrrfTile<M, V>::TY;
  static constexpr int NP = EsrrfTile<M, V>::NP;
  static constexpr int PYT = EsrrfTile<M, V>::PYT;
  static constexpr int NSC = MODE == kModeSum ? kMaxSens : 1;
  static constexpr int FP =
      EsrrfTile<M, V>::FP_MAX >= 4 &&
              Geo<M, J, TY, 4, NP, PYT>::smem_bytes(MODE, NSC) <= kSmemBudget ? 4 : 2;
  using G = Geo<M, J, TY, FP, NP, PYT>;
};

// Unit gradients of a frame pair are kept scaled by 2^32: the half-plane test
// t < 0 of a sample is then a saturating FMA of the scaled gradients, which
// gives exactly 0 or 1 unless |t| < 2^-32, where the sample's contribution
// w (1 - |sin|) is itself below w 2^-64.  A power of two, so nothing else rounds
// differently.
constexpr float kGradScale = 4294967296.f;

// max(v, 0) that keeps a NaN
__device__ __forceinline__ float clamp0(float v) {
  float r;
  asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(r) : "f"(v));
  return r;
}

// r^1.5 of a frame pair, as power_compensated (common.cuh) forms it
__device__ __forceinline__ float2 power_1p5(const float2& r) {
  const float2 s = make_float2(__fsqrt_rn(r.x), __fsqrt_rn(r.y));
  const float2 q = __fmul2_rn(r, s);
  const float2 d = __ffma2_rn(make_float2(-s.x, -s.y), s, r);
  const float2 e = __ffma2_rn(__fmul2_rn(make_float2(0.5f, 0.5f), d), s,
                              __ffma2_rn(r, s, make_float2(-q.x, -q.y)));
  const float2 v = __fadd2_rn(q, e);
  return make_float2(v.x == v.x ? v.x : q.x, v.y == v.y ? v.y : q.y);
}

// The powers that are not worth their code in every unrolled use, a frame pair a
// call (150 frames of 227 x 333, m = 5, s = 2.5: 3.27 ms, 3.54 with a call per value).
static __device__ __noinline__ float2 apply_sensitivity_pair(float2 r, int mode, int n, float s) {
  if (mode == 2) return make_float2(powf(r.x, s), powf(r.y, s));
  float2 p = r, e = make_float2(0.f, 0.f), below = make_float2(1.f, 1.f);
  if (mode == 1) {
#pragma unroll 1
    for (int k = 1; k < n; ++k) p = __fmul2_rn(p, r);
    return p;
  }
  // power_compensated (common.cuh)
#pragma unroll 1
  for (int k = 1; k < n; ++k) {
    const float2 q = __fmul2_rn(p, r);
    e = __ffma2_rn(e, r, __ffma2_rn(p, r, make_float2(-q.x, -q.y)));
    below = p;
    p = q;
  }
  const float2 t = make_float2(__fsqrt_rn(r.x), __fsqrt_rn(r.y));
  const float2 q = __fmul2_rn(p, t);
  const float2 d = __ffma2_rn(make_float2(-t.x, -t.y), t, r);
  e = __ffma2_rn(e, t, __ffma2_rn(p, t, make_float2(-q.x, -q.y)));
  e = __ffma2_rn(__fmul2_rn(__fmul2_rn(make_float2(0.5f, 0.5f), below), d), t, e);
  const float2 v = __fadd2_rn(q, e);
  return make_float2(v.x == v.x ? v.x : q.x, v.y == v.y ? v.y : q.y);
}

// r ^ sensitivity of a thread's values (mode and n are uniform over the launch):
// squares and cubes, and (HALF) the power 1.5, in place; the others by call --
// with powf and the square root inlined per sensitivity and column, the AVG
// kernels' code outgrew the instruction cache (4 x 4 sweep of 200 x 256 x 256,
// m = 4: 13.46 against 12.39 ms), and the powers 2.5 and 3.5 in place cost every
// kernel registers (m = 5: 30 to 70 bytes more spilled per thread).
template <bool HALF, int A, int B>
__device__ __forceinline__ void apply_sens_all(float2 (&r)[A][B], int mode, int n, float s) {
  if (mode == 0) return;
  if (mode == 1 && n <= 3) {
#pragma unroll
    for (int i = 0; i < A; ++i)
#pragma unroll
      for (int j = 0; j < B; ++j) {
        const float2 q = __fmul2_rn(r[i][j], r[i][j]);
        r[i][j] = n == 3 ? __fmul2_rn(q, r[i][j]) : q;
      }
    return;
  }
  if (HALF && mode == 3 && n == 1) {
#pragma unroll
    for (int i = 0; i < A; ++i)
#pragma unroll
      for (int j = 0; j < B; ++j) r[i][j] = power_1p5(r[i][j]);
    return;
  }
#pragma unroll
  for (int i = 0; i < A; ++i)
#pragma unroll
    for (int j = 0; j < B; ++j) r[i][j] = apply_sensitivity_pair(r[i][j], mode, n, s);
}

// geometry of one unit (tile, timepoint, frame chunk), shared by both roles
struct UnitGeo {
  int nx0, ny0, H, W, f0, f1;
  int RY0, CX0, y_start, x_start, kmax_y, kmax_x;
};

// ---------------------------------------------------------------------------
// producer warps: input tiles -> slot s (unit gradients hg, intensity rows ri)
// ---------------------------------------------------------------------------
template <typename G, int M, int J>
struct Producer {
  float* inb;
  float* gsm;  // Roberts-Cross gradients, one plane of float4 per frame pair
  float* hg0;  // slot 0; slot s at hg0 + s * S_HG
  float* ri0;  // slot s, frame pair pp at ri0 + (s * NPR + pp) * S_RI
  const float* rw;
  int ptid;

  // Roberts-Cross gradients and the intensity row pass of np frame pairs; tin:
  // the input tile of every frame
  __device__ void roberts_and_rows(const FusedParams& p, const UnitGeo& u, int nf, int np,
                                   int s) const {
    for (int pp = 0; pp < np; ++pp) {
      const float* t0 = inb + 2 * pp * G::S_INB;
      // an odd last frame stands in for its missing partner
      const float* t1 = 2 * pp + 1 < nf ? t0 + G::S_INB : t0;
      float4* g4 = reinterpret_cast<float4*>(gsm + pp * G::S_G);
      for (int i = ptid; i < G::NRY * G::NCX; i += G::NP) {
        const int rl = i / G::NCX, cl = i % G::NCX;
        const int r = u.RY0 + rl, c = u.CX0 + cl;
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r >= 0 && r < u.H && c >= 0 && c < u.W) {
          const int ie = (r - u.y_start) * G::BW + (c - u.x_start);  // image[r1][c1]
          const int ia = r > 0 ? ie - G::BW : ie;                    // image[r0][c1]
          const int ib = c > 0 ? ie - 1 : ie;                        // image[r1][c0]
          const int id = c > 0 ? ia - 1 : ia;                        // image[r0][c0]
          const float a0 = t0[ia], b0 = t0[ib], d0 = t0[id], e0 = t0[ie];
          const float a1 = t1[ia], b1 = t1[ib], d1 = t1[id], e1 = t1[ie];
          g.x = __fsub_rn(__fadd_rn(__fsub_rn(a0, b0), e0), d0);
          g.y = __fsub_rn(__fadd_rn(__fsub_rn(a1, b1), e1), d1);
          g.z = __fsub_rn(__fadd_rn(__fadd_rn(-a0, b0), e0), d0);
          g.w = __fsub_rn(__fadd_rn(__fadd_rn(-a1, b1), e1), d1);
        }
        g4[i] = g;
      }
      // intensity row pass: one input row and column at a time, whose 5 taps
      // serve the M output rows
      if (!p.iw) continue;
      float2* ri = reinterpret_cast<float2*>(ri0 + (s * G::NPR + pp) * G::S_RI);
      for (int i = ptid; i < (G::OY / M) * G::RIW; i += G::NP) {
        const int ty = i / G::RIW, cc = i % G::RIW;
        const int off = (u.ny0 + ty - 2 - u.y_start) * G::BW + (u.nx0 - 2 + cc - u.x_start);
        float2 v[5];
#pragma unroll
        for (int k = 0; k < 5; ++k)
          v[k] = make_float2(t0[off + k * G::BW], t1[off + k * G::BW]);
#pragma unroll
        for (int py = 0; py < M; ++py) {
          const float* w = rw + (ty * M + py) * 8;
          const float4 wa = *reinterpret_cast<const float4*>(w);
          const float w5[5] = {wa.x, wa.y, wa.z, wa.w, w[4]};
          float2 sum = make_float2(0.f, 0.f);
#pragma unroll
          for (int k = 0; k < 5; ++k) sum = __ffma2_rn(make_float2(w5[k], w5[k]), v[k], sum);
          ri[(ty * M + py) * G::RIW + cc] = sum;
        }
      }
    }
  }

  // one half-grid sample of a frame pair: normalise and store
  __device__ __forceinline__ static void emit(const float4& v, bool valid, float4* dst) {
    const float2 x = make_float2(v.x, v.y), y = make_float2(v.z, v.w);
    const float2 m2 = __ffma2_rn(x, x, __fmul2_rn(y, y));
    const float i0 = rsqrtf(m2.x) * kGradScale, i1 = rsqrtf(m2.y) * kGradScale;
    const float2 inv = make_float2(i0, i1);
    const float2 nx = __fmul2_rn(x, inv), ny = __fmul2_rn(y, inv);
    const bool k0 = valid && m2.x > 0.f, k1 = valid && m2.y > 0.f;
    *dst = make_float4(k0 ? nx.x : 0.f, k1 ? nx.y : 0.f, k0 ? ny.x : 0.f, k1 ? ny.y : 0.f);
  }

  // w0 q0 + w1 q1 + w2 q2 + w3 q3 of a frame pair's (gx, gx', gy, gy')
  __device__ __forceinline__ static float4 taps(const float4& q0, const float4& q1,
                                                const float4& q2, const float4& q3,
                                                const float (&w)[4]) {
    auto tap = [](float wk, const float4& q, float2& x, float2& y) {
      const float2 w2 = make_float2(wk, wk);
      x = __ffma2_rn(w2, make_float2(q.x, q.y), x);
      y = __ffma2_rn(w2, make_float2(q.z, q.w), y);
    };
    float2 x = __fmul2_rn(make_float2(w[0], w[0]), make_float2(q0.x, q0.y));
    float2 y = __fmul2_rn(make_float2(w[0], w[0]), make_float2(q0.z, q0.w));
    tap(w[1], q1, x, y);
    tap(w[2], q2, x, y);
    tap(w[3], q3, x, y);
    return make_float4(x.x, x.y, y.x, y.y);
  }

  // Gradient Catmull-Rom on the half-grid and its normalisation -> slot s.
  // Half-grid index 2 a takes the taps a-2 .. a+1 of its axis with weights
  // (-1, 9, 9, -1) / 16, index 2 a + 1 is sample a itself; indices from 2 H
  // (2 W) on are all the clamped last position, whose taps H-2 .. H+1 are
  // those of a = H.  A thread takes one half-grid column and walks down the row
  // steps of a segment with the four newest rows of its column in registers:
  // per row 4 shared loads (an even index) or 1 (an odd one), per step two
  // samples, without the buffer between a column and a row pass.  Lanes run
  // along the columns of one parity; the LEFT columns beyond a warp are done
  // one step per thread.
  __device__ void gradients(const FusedParams& p, const UnitGeo& u, int np, int s) const {
    const int a0 = u.ny0 - (J + 1) / 2, b0 = u.nx0 - (J + 1) / 2;
    const int tH = u.H - a0;  // step of a = H
    const int main_jobs = np * G::NSEG * 64;
    const int jobs = main_jobs + np * G::NA * G::LEFT * 2;
    for (int i = ptid; i < jobs; i += G::NP) {
      int pp, c, t0, t1, odd;
      if (i < main_jobs) {
        const int wj = i >> 5;
        odd = wj >= np * G::NSEG;
        const int k = odd ? wj - np * G::NSEG : wj;
        pp = k / G::NSEG;
        t0 = (k - pp * G::NSEG) * G::SEG;
        t1 = min(t0 + G::SEG, G::NA);
        c = i & 31;
      } else {
        const int k = i - main_jobs;
        const int pl = k / (G::NA * G::LEFT);
        const int r = k - pl * (G::NA * G::LEFT);
        odd = pl >= np;
        pp = odd ? pl - np : pl;
        t0 = r / G::LEFT;
        t1 = t0 + 1;
        c = 32 + r - t0 * G::LEFT;
      }
      // an odd J starts its tile at an odd half-grid index: the first even and
      // the last odd index of the steps are outside the slot
      if ((J & 1) && c == (odd ? G::NB - 1 : 0)) continue;
      const int b = b0 + c;
      const int kx = 2 * b + odd;
      const bool vx = kx >= 1 && kx <= u.kmax_x;
      const bool cclamp = b >= u.W;
      const bool four = cclamp || !odd;
      const float4* g4 = reinterpret_cast<const float4*>(gsm + pp * G::S_G) +
                         (cclamp ? u.W - 2 - u.CX0 : (odd ? c + 2 : c));
      // slot column of kx: [parity][index]
      float4* hg = reinterpret_cast<float4*>(hg0 + s * G::S_HG) + pp * G::HG_PLANE +
                   ((J & 1) ? (odd ? c : G::HGP + c - 1) : odd * G::HGP + c);
      float4 win[4];
      auto row = [&](int r) {
        const float4* q = g4 + r * G::NCX;
        float4 v = q[0];
        if (four) {
          float w[4] = {-0.0625f, 0.5625f, 0.5625f, -0.0625f};
          if (cclamp) {
#pragma unroll
            for (int k = 0; k < 4; ++k) w[k] = p.cx[k];
          }
          v = taps(v, q[1], q[2], q[3], w);
        }
        return v;
      };
      const int ts = min(t0, tH);
#pragma unroll
      for (int k = 0; k < 3; ++k) win[k + 1] = row(ts + k);
#pragma unroll
      for (int d = 0; d < G::SEG; ++d) {
        const int t = t0 + d;
        if (t >= t1) break;
        if (d == 0 || t <= tH) {  // past a = H the window stays
#pragma unroll
          for (int k = 0; k < 3; ++k) win[k] = win[k + 1];
          win[3] = row(min(t, tH) + 3);
        }
        const int a = a0 + t;
        const int kyl = 2 * t - (J & 1);  // slot row of 2 a
        const bool rclamp = a >= u.H;
        float w[4] = {-0.0625f, 0.5625f, 0.5625f, -0.0625f};
        if (rclamp) {
#pragma unroll
          for (int k = 0; k < 4; ++k) w[k] = p.cy[k];
        }
        const float4 e = taps(win[0], win[1], win[2], win[3], w);
        if (!(J & 1) || t >= 1)
          emit(e, vx && 2 * a >= 1 && 2 * a <= u.kmax_y, hg + kyl * 2 * G::HGP);
        if (!(J & 1) || t < G::NA - 1)
          emit(rclamp ? e : win[2], vx && a >= 0 && 2 * a + 1 <= u.kmax_y,
               hg + (kyl + 1) * 2 * G::HGP);
      }
    }
  }
};

// Numerator of the horizontal offset of half-grid sample q (of the NQ a window
// row spans) from the centre of output phase px, 2 M dx = M (q - J) - (2 px + 1);
// zero only for the middle phase of an odd M at q = J + 1.
template <int M, int J>
__host__ __device__ constexpr int dx_num(int px, int q) {
  return M * (q - J) - (2 * px + 1);
}

// whether sample q lies in the window of output phase px
template <int M, int J>
__host__ __device__ constexpr bool in_window(int px, int q) {
  const int ii = q - (2 * px + 1) / M;
  return px >= 0 && px < M && ii >= 0 && ii < 2 * J + 1;
}

// One sample of the RGC for a frame pair: acc += [n.(a, b) < 0] (w - |n x (a, b)|).
// With rho = b / a, n.(a, b) = a (gx + gy rho) and |n x (a, b)| = |a| |gy - gx rho|;
// SIGN is the sign of dx (of a), a constant of the unrolled loops.  For dx = 0
// the two are gy b and |b| |gx|, and rho, nab stand for sign b and -|b|.
//
// The test is a saturating scalar FMA per frame (kGradScale): 0 or 1 straight
// from the FMA pipe.  In a loop of samples with their constants in registers
// this form took 10.8 cycles per sample pair and scheduler, the comparison it
// replaces (a packed FMA and two ALU set instructions) 12.1; four packed FMAs
// alone take 10.8, because each reads six register operands.
template <int SIGN>
__device__ __forceinline__ void rgc_sample(const float4& g, float rho, float nrho, float nab,
                                           float w, float2& acc) {
  const float2 gx = make_float2(g.x, g.y), gy = make_float2(g.z, g.w);
  float2 m, t2;
  if (SIGN > 0) {
    m = make_float2(__saturatef(__fmaf_rn(-gy.x, rho, -gx.x)),
                    __saturatef(__fmaf_rn(-gy.y, rho, -gx.y)));
  } else if (SIGN < 0) {
    m = make_float2(__saturatef(__fmaf_rn(gy.x, rho, gx.x)),
                    __saturatef(__fmaf_rn(gy.y, rho, gx.y)));
  } else {
    m = make_float2(__saturatef(__fmul_rn(-gy.x, rho)), __saturatef(__fmul_rn(-gy.y, rho)));
  }
  t2 = SIGN == 0 ? gx : __ffma2_rn(gx, make_float2(nrho, nrho), gy);
  const float2 v = __ffma2_rn(make_float2(nab, nab), make_float2(fabsf(t2.x), fabsf(t2.y)),
                              make_float2(w, w));
  acc = __ffma2_rn(m, v, acc);
}

// RGC of one consumer's PYT * M outputs for NPR frame pairs of the slot at hgf.
// Contribution of sample (phase, offset): (dp < 0) ? w - |u| : 0 with
// dp = n.(a, b) and u = n x (a, b) (n the unit gradient).
//
// Mirror images share a table entry: sample q seen from phase px and sample
// NQ - q seen from phase M - 1 - px lie at opposite dx and the same dy, so they
// have the same weight and |a| and opposite rho.  Walking q from both ends loads
// (J + 1) M + M / 2 entries per window row instead of M (2J + 1) (m = 5,
// R = 1.5: 20 used for 35 samples).
//
// The phases of a thread share every gradient load (LDS.128, four wavefronts a
// warp) of a half-grid row.  Phases of the lower half of a pixel (cpy = 0) use
// row k as window row k, those of the upper half (cpy = 1) as window row k - 1;
// with both in one thread (PYT = M) the first and the last row serve one half.
template <typename G, int M, int J, int NPR>
struct RgcCore {
  static constexpr int PYT = G::PYT;
  const float4* hg;   // this lane's first sample of row 2 ty
  const float4* tb4;  // phase table of row phase py0
  int cpy;            // of every phase of the thread unless PYT = M

  // one row of the slot (at r) for the phases D0 .. D1 - 1; tb: the table of
  // phase 0 at that row, were its cpy that of every phase
  template <int D0, int D1>
  __device__ __forceinline__ static void row(const float4* r, const float4* tb,
                                             float2 (&acc)[NPR][PYT * M]) {
    auto grad = [&](int pp, int q) {
      return r[(q & 1) * G::HGP + pp * G::HG_PLANE + (q >> 1)];
    };
    auto table = [&](int d) {
      return tb + (d * G::W2 - (PYT == M && M > 1 ? (2 * d + 1) / M : 0)) * G::NE;
    };
    auto sample = [&](int px, int q, const float4& g, float rho, float nrho, const float4& T,
                      float2& a) {
      const int dxn = dx_num<M, J>(px, q);
      if (dxn > 0) rgc_sample<1>(g, rho, nrho, T.z, T.w, a);
      else if (dxn < 0) rgc_sample<-1>(g, rho, nrho, T.z, T.w, a);
      else rgc_sample<0>(g, rho, nrho, T.z, T.w, a);
    };
    if constexpr (M <= 2) {
      // gradient-major order: one half-grid sample at a time, applied to every
      // output phase px whose window holds it
#pragma unroll
      for (int q = 0; q < G::NQ; ++q) {
        float4 g[NPR];
#pragma unroll
        for (int pp = 0; pp < NPR; ++pp) g[pp] = grad(pp, q);
#pragma unroll
        for (int d = D0; d < D1; ++d)
#pragma unroll
          for (int px = 0; px < M; ++px) {
            if (!in_window<M, J>(px, q)) continue;
            // entry (rho, -rho, -|a|, w) of this sample, or of its mirror image
            const bool own = q <= J || (q == J + 1 && 2 * px < M);
            const float4 T = table(d)[own ? q * M + px : (G::NQ - q) * M + M - 1 - px];
#pragma unroll
            for (int pp = 0; pp < NPR; ++pp)
              sample(px, q, g[pp], own ? T.x : T.y, own ? T.y : T.x, T, acc[pp][d * M + px]);
          }
      }
    } else {
#pragma unroll
      for (int q = 0; q <= J + 1; ++q) {
        const int qm = G::NQ - q;  // the mirrored sample (none for q = 0)
        float4 ga[NPR], gb[NPR];
#pragma unroll
        for (int pp = 0; pp < NPR; ++pp) {
          ga[pp] = grad(pp, q);
          gb[pp] = (q >= 1 && qm != q) ? grad(pp, qm) : ga[pp];
        }
#pragma unroll
        for (int d = D0; d < D1; ++d)
#pragma unroll
          for (int px = 0; px < (q == J + 1 ? (M + 1) / 2 : M); ++px) {
            const int pm = M - 1 - px;
            const bool use_a = in_window<M, J>(px, q);
            const bool use_b = q >= 1 && (q != qm || px != pm) && in_window<M, J>(pm, qm);
            if (!use_a && !use_b) continue;
            const float4 T = table(d)[q * M + px];  // (rho, -rho, -|a|, w) of (px, q)
#pragma unroll
            for (int pp = 0; pp < NPR; ++pp) {
              if (use_a) sample(px, q, ga[pp], T.x, T.y, T, acc[pp][d * M + px]);
              if (use_b) sample(pm, qm, gb[pp], T.y, T.x, T, acc[pp][d * M + pm]);
            }
          }
      }
    }
  }

  __device__ __forceinline__ void run(float2 (&acc)[NPR][PYT * M]) const {
#pragma unroll
    for (int pp = 0; pp < NPR; ++pp)
#pragma unroll
      for (int o = 0; o < PYT * M; ++o) acc[pp][o] = make_float2(0.f, 0.f);
    // window rows stay a loop: unrolled, the core's code outgrows the
    // instruction cache (measured 2 % slower and with register spills)
    const float4* r = hg + cpy * 2 * G::HGP;
    const float4* t = tb4;
    if constexpr (PYT == M && M > 1) {
      constexpr int DH = M / 2;  // phases d < DH have cpy = 0
      row<0, DH>(r, t, acc);
#pragma unroll 1
      for (int k = 1; k < G::NQ - 1; ++k) {
        r += 2 * G::HGP;
        t += G::NE;
        row<0, M>(r, t, acc);
      }
      row<DH, M>(r + 2 * G::HGP, t + G::NE, acc);
    } else {
#pragma unroll 1
      for (int k = 0; k < G::W2; ++k, r += 2 * G::HGP, t += G::NE) row<0, PYT>(r, t, acc);
    }
  }
};

template <int M, int J, int TY, int FP, int MODE, int NP, int PYT>
__global__ void __launch_bounds__(32 * TY * (M / PYT) + NP, EsrrfTile<M>::MIN_BLOCKS)
    esrrf_fused_kernel(const __grid_constant__ TmapPack maps, const UnitTable ut) {
  using G = Geo<M, J, TY, FP, NP, PYT>;
  extern __shared__ __align__(128) float sm[];
  __shared__ FusedParams sp;
  __shared__ int s_unit;
  __shared__ int s_abort;
  float4* tb4 = reinterpret_cast<float4*>(sm + G::O_TB);
  float* rw = sm + G::O_RW;
  float* cw = sm + G::O_CW;
  float* tw = sm + G::O_TW;  // tw[output * NTC + tid]
  float* tk = sm + G::O_TK;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + G::o_bar(MODE, ut.ns_cap));
  uint64_t* full = bars;                    // [NSLOT] slot prepared (NP arrivals)
  uint64_t* empty = bars + G::NSLOT;        // [NSLOT] slot released (NTC arrivals)
  uint64_t* pbar = bars + 2 * G::NSLOT;     // producer-group barrier (NP arrivals)
  uint64_t* tbar = bars + 2 * G::NSLOT + 1; // TMA input tiles of a pass

  const int tid = threadIdx.x;
  const bool producer = tid >= G::NTC;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int ty = warp % TY;  // consumers
  const int py0 = PYT == M ? 0 : warp / TY * PYT;
  const Producer<G, M, J> prod{sm + G::O_INB, sm + G::O_G, sm + G::O_HG,
                               sm + G::O_RI, rw, tid - G::NTC};

  if (tid == 0) {
    for (int k = 0; k < G::NSLOT; ++k) {
      mbar_init(&full[k], G::NP);
      mbar_init(&empty[k], G::NTC);
    }
    mbar_init(pbar, G::NP);
    mbar_init(tbar, 1);
    fence_mbar_init();
    s_abort = 0;
  }
  __syncthreads();
  unsigned gp = 0;      // frame passes since launch: slot gp % NSLOT, use gp / NSLOT (all threads)
  unsigned tphase = 0;  // producers: parity of the next completion of tbar
  bool tpend = false;   // producers: TMA loads into the input tiles are in flight
  unsigned pphase = 0;  // producers: parity of the next completion of pbar
  int cur_item = -1;

  for (int iter = 0;; ++iter) {
  int unit;
  if (ut.counter) {
    if (tid == 0) s_unit = (int)atomicAdd(ut.counter, 1u);
    __syncthreads();
    unit = s_unit;
  } else {
    unit = blockIdx.x + iter * gridDim.x;
  }
  if (unit >= ut.total_units) break;
  int item = 0;
  if (ut.items) {
    int lo = 0, hi = ut.n_items - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(ut.unit_start + mid) <= unit) lo = mid;
      else hi = mid - 1;
    }
    item = lo;
  }
  if (item != cur_item) {
    if (tid == 0) sp = ut.items ? ut.items[item] : ut.single;
    __syncthreads();
    {
      // plan layout [py][jj]{a, b, w}[NS4 * 4] -> one float4 per mirrored couple
      // (see rgc_core), in the orientation of its sample (px, q):
      //   dx != 0: (rho, -rho, -|a| / scale, w) with rho = b / a;
      //   dx == 0: (sign b, 0, -|b| / scale, w);  outside the radius: zeros
      constexpr int N4 = G::NS4 * 4;
      const float* src = sp.tbl;
      for (int i = tid; i < M * G::W2 * G::NE; i += G::NT) {
        const int blk = i / G::NE, k = i % G::NE;
        const int q = k / M, px = k % M;
        const bool own = in_window<M, J>(px, q);
        const int sp_px = own ? px : M - 1 - px, sq = own ? q : G::NQ - q;
        float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in_window<M, J>(sp_px, sq)) {
          const int s = sp_px * G::W2 + sq - (2 * sp_px + 1) / M;
          const float a = own ? src[(blk * 3 + 0) * N4 + s] : -src[(blk * 3 + 0) * N4 + s];
          const float b = src[(blk * 3 + 1) * N4 + s];
          const float w = src[(blk * 3 + 2) * N4 + s];
          if (w != 0.f) {
            if (dx_num<M, J>(px, q) == 0) {
              e = make_float4(b > 0.f ? 1.f : -1.f, 0.f, -fabsf(b) / kGradScale, w);
            } else if (a != 0.f) {
              const float rho = __fdiv_rn(b, a);
              e = make_float4(rho, -rho, -fabsf(a) / kGradScale, w);
            }
          }
        }
        tb4[blk * G::NE + k] = e;
      }
    }
    cur_item = item;
  }
  const FusedParams& p = sp;
  const unsigned long long lim = p.wait_ns ? p.wait_ns : kWaitLimitNs;
  const int local = unit - (ut.items ? __ldg(ut.unit_start + item) : 0);
  const int tiles = p.tiles_x * p.tiles_y;
  const int tile = local % tiles;
  const int tp = (local / tiles) / p.chunks;
  const int chunk = (local / tiles) % p.chunks;

  // frames of this unit
  const int tp_f0 = tp * p.fpt;
  const int tp_nf = min(p.fpt, p.T - tp_f0);
  const int nch = min(p.chunks, tp_nf);
  int npass = 0;
  if (chunk < nch) {  // uniform across the CTA
  UnitGeo u;
  u.nx0 = (tile % p.tiles_x) * G::TX;
  u.ny0 = (tile / p.tiles_x) * TY;
  u.H = p.H;
  u.W = p.W;
  u.f0 = tp_f0 + (int)((long long)chunk * tp_nf / nch);
  u.f1 = tp_f0 + (int)((long long)(chunk + 1) * tp_nf / nch);
  u.RY0 = u.ny0 - G::RLO;
  u.CX0 = u.nx0 - G::CLO;
  u.y_start = u.ny0 - G::IY;
  u.x_start = u.nx0 - G::IX;
  u.kmax_y = 2 * p.rowsM - 2;
  u.kmax_x = 2 * p.colsM - 2;
  const int f0 = u.f0, f1 = u.f1;
  npass = (f1 - f0 + FP - 1) / FP;

  // ---- per-CTA constants: intensity interpolation weights -----------------
  for (int i = tid; i < G::OY; i += G::NT) {
    const int yM = u.ny0 * M + i;
    const int nyp = u.ny0 + i / M;
    const float ry = __fdiv_rn((float)yM, (float)M);
    const int rb = (int)floorf(ry - 0.5f);
    float w5[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int nb = rb - 1 + t;
      const int k = nb - (nyp - 2);
      const float w = cr_cubic(ry - ((float)nb + 0.5f));
#pragma unroll
      for (int kk = 0; kk < 5; ++kk) w5[kk] = (k == kk) ? w : w5[kk];
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) rw[i * 8 + k] = w5[k];
  }
  for (int i = tid; i < G::OX; i += G::NT) {
    const int xM = u.nx0 * M + i;
    const int nxp = u.nx0 + i / M;
    const float rx = __fdiv_rn((float)xM, (float)M);
    const int cb = (int)floorf(rx - 0.5f);
    float w5[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int nb = cb - 1 + t;
      const int k = nb - (nxp - 2);
      const float w = cr_cubic(rx - ((float)nb + 0.5f));
#pragma unroll
      for (int kk = 0; kk < 5; ++kk) w5[kk] = (k == kk) ? w : w5[kk];
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) cw[i * 5 + k] = w5[k];
  }

  // ---- 1 / sum w of the outputs: several row phases per consumer --------------
  // by all warps, so that the windows of an edge tile are no longer a chain than with one
  // phase (a push of one frame of 64 x 64, m = 2: 24.9 us by the consumers alone, 20.3 so);
  // with one phase the consumers' own loop below is the shorter (256 x 256, m = 5: 130 us
  // a push, 147 by all warps)
  if constexpr (PYT > 1) {
    for (int e = tid; e < G::NO * G::NTC; e += G::NT) {
      const int o = e / G::NTC, c = e % G::NTC;  // output o of consumer c
      const int py = (PYT == M ? 0 : (c >> 5) / TY * PYT) + o / M, px = o % M;
      const int ky_lo = 2 * (u.ny0 + (c >> 5) % TY) + (2 * py + 1) / M - J;
      const int kx_lo = 2 * (u.nx0 + (c & 31)) + (2 * px + 1) / M - J;
      float iw = p.inv_wsum[py * M + px];
      if (ky_lo < 1 || ky_lo + 2 * J > u.kmax_y || kx_lo < 1 || kx_lo + 2 * J > u.kmax_x) {
        const float* wf = p.wfull + (size_t)(py * M + px) * G::W2 * G::W2;
        float s = 0.f;
        for (int jj = 0; jj < G::W2; ++jj) {
          if (ky_lo + jj < 1 || ky_lo + jj > u.kmax_y) continue;
          for (int ii = 0; ii < G::W2; ++ii)
            if (kx_lo + ii >= 1 && kx_lo + ii <= u.kmax_x) s += wf[jj * G::W2 + ii];
        }
        iw = s > 0.f ? 1.f / s : 0.f;
      }
      tw[e] = iw;
    }
  }

  // ---- consumer constants --------------------------------------------------
  const int ny = u.ny0 + ty;
  const int nx = u.nx0 + lane;
  unsigned omask = 0;  // bit per output: forced to 0 / not written; bit 31: outside the image
  if (!producer) {
#pragma unroll
    for (int d = 0; d < PYT; ++d) {
      const int py = py0 + d, yM = ny * M + py;
      const int cpy = (2 * py + 1) / M;
      const int ky_lo = 2 * ny + cpy - J, ky_hi = 2 * ny + cpy + J;
      const bool by = (ky_lo < 1) || (ky_hi > u.kmax_y);
#pragma unroll
      for (int px = 0; px < M; ++px) {
        const int cpx = (2 * px + 1) / M;
        const int xM = nx * M + px;
        const int kx_lo = 2 * nx + cpx - J, kx_hi = 2 * nx + cpx + J;
        if constexpr (PYT == 1) {
          float iw = p.inv_wsum[py * M + px];
          if (by || kx_lo < 1 || kx_hi > u.kmax_x) {
            // window reaches invalid half-grid samples: they count in neither sum
            const float* wf = p.wfull + (size_t)(py * M + px) * G::W2 * G::W2;
            float s = 0.f;
            for (int jj = 0; jj < G::W2; ++jj) {
              const int ky = ky_lo + jj;
              if (ky < 1 || ky > u.kmax_y) continue;
              for (int ii = 0; ii < G::W2; ++ii) {
                const int kx = kx_lo + ii;
                if (kx < 1 || kx > u.kmax_x) continue;
                s += wf[jj * G::W2 + ii];
              }
            }
            iw = s > 0.f ? 1.f / s : 0.f;
          }
          tw[(d * M + px) * G::NTC + tid] = iw;
        }
        const bool outside = (ny >= u.H) || (nx >= u.W);
        const bool in_margin = (yM < p.margin) || (yM >= p.rowsM - p.margin) ||
                               (xM < p.margin) || (xM >= p.colsM - p.margin);
        if (outside) omask |= (1u << (d * M + px)) | (1u << 31);
        else if (in_margin) omask |= (1u << (d * M + px));
      }
    }
  }
  __syncthreads();

  if (producer) {
    // ======================= producer warps =================================
    constexpr unsigned kTileBytes = unsigned(G::BH * G::BW * 4);
    const bool use_tma = p.tmap >= 0;
    const CUtensorMap* tmap = use_tma ? &maps.m[p.tmap] : nullptr;
    const bool leader = prod.ptid == 0;
    // the input tiles of the pass whose first frame is f (leader only)
    auto fetch = [&](int f) {
      const int n = min(FP, f1 - f);
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(tbar, n * kTileBytes);
      for (int k = 0; k < n; ++k)
        tma_load_3d(prod.inb + k * G::S_INB, tmap, tbar, u.x_start, u.y_start, f + k);
      tpend = true;
    };
    auto group_sync = [&]() {  // all producer threads
      mbar_arrive(pbar);
      const bool ok = mbar_wait_or_abort(pbar, pphase & 1u, &s_abort, lim);
      pphase ^= 1u;
      return ok;
    };
    if (use_tma && leader) fetch(f0);
    for (int j = 0; j < npass; ++j) {
      const unsigned g = gp + j;
      const int s = (int)(g % G::NSLOT);
      const unsigned use = g / G::NSLOT;
      const int fa = f0 + j * FP;
      const int nf = min(FP, f1 - fa);
      const int np = (nf + 1) / 2;
      // slot s is free once the consumers released its previous use
      bool ok = use == 0 || mbar_wait_or_abort(&empty[s], (use - 1) & 1u, &s_abort, lim);
      if (ok && use_tma) {
        ok = mbar_wait_or_abort(tbar, tphase, &s_abort, lim);
        if (ok) {
          tphase ^= 1u;
          tpend = false;
        }
      } else if (ok) {
        for (int fr = 0; fr < nf; ++fr) {
          const float* src = p.in + (size_t)(fa + fr) * u.H * u.W;
          float* dst = prod.inb + fr * G::S_INB;
          for (int i = prod.ptid; i < G::BH * G::BW; i += G::NP) {
            const int r = u.y_start + i / G::BW;
            const int c = u.x_start + i % G::BW;
            dst[i] = (r >= 0 && r < u.H && c >= 0 && c < u.W) ? __ldg(src + (size_t)r * u.W + c)
                                                               : 0.f;
          }
        }
        ok = group_sync();
      }
      // (the group_sync at the end of the previous pass freed the gradient planes)
      if (ok) {
        prod.roberts_and_rows(p, u, nf, np, s);
        ok = group_sync();
      }
      if (ok) {
        // the input tiles are free: fetch the next pass's frames
        if (use_tma && leader && fa + FP < f1) fetch(fa + FP);
        prod.gradients(p, u, np, s);
        if (!(p.test_withhold_full && iter == 0 && j == 0)) mbar_arrive(&full[s]);
        ok = group_sync();
      }
      if (!ok) {
        *(volatile int*)&s_abort = 1;
        break;
      }
    }
  } else {
    // ======================= consumers ======================================
    const size_t plane = (size_t)p.rowsM * p.colsM;
    for (int j = 0; j < npass; ++j) {
      const unsigned g = gp + j;
      const int s = (int)(g % G::NSLOT);
      const unsigned use = g / G::NSLOT;
      const int fa = f0 + j * FP;
      const int nf = min(FP, f1 - fa);
      if (!mbar_wait_or_abort(&full[s], use & 1u, &s_abort, lim)) {
        *(volatile int*)&s_abort = 1;
        break;
      }
      const float* hgf = sm + G::O_HG + s * G::S_HG;
      const bool first = (fa == f0);
      // frame fa + fr is frame k = fa - f0 + fr of this unit's series; 1 / (k + 1)
      // by the fast reciprocal (the increment it scales is a deviation-sized term,
      // so its ~1 ulp error does not show; the IEEE reciprocal cost 2 % of the kernel)
      float inv_n[FP];
#pragma unroll
      for (int fr = 0; fr < FP; ++fr) inv_n[fr] = __fdividef(1.0f, (float)(fa - f0 + fr + 1));
      float2 acc[G::NPR][G::NO];
      {
        const int cpy = PYT == M ? (M > 1 ? 0 : 1) : (2 * py0 + 1) / M;
        const float4* g0 = reinterpret_cast<const float4*>(hgf) + 4 * ty * G::HGP + lane;
        const float4* t0 = tb4 + py0 * G::W2 * G::NE;
        if (G::NPR == 1 || nf > 2) {
          RgcCore<G, M, J, G::NPR>{g0, t0, cpy}.run(acc);
        } else {  // the last pass of a chunk may hold one frame pair only
          float2 acc1[1][G::NO];
          RgcCore<G, M, J, 1>{g0, t0, cpy}.run(acc1);
#pragma unroll
          for (int o = 0; o < G::NO; ++o) {
            acc[0][o] = acc1[0][o];
#pragma unroll
            for (int pp = 1; pp < G::NPR; ++pp) acc[pp][o] = make_float2(0.f, 0.f);
          }
        }
      }

      // ---- normalise, ^sensitivity, intensity, margin, temporal ------------
#pragma unroll
      for (int o = 0; o < G::NO; ++o) {
        const float twv = tw[o * G::NTC + tid];
#pragma unroll
        for (int pp = 0; pp < G::NPR; ++pp)
          acc[pp][o] = make_float2(clamp0(acc[pp][o].x * twv), clamp0(acc[pp][o].y * twv));
      }
      if (MODE != kModeSum)
        apply_sens_all<true>(acc, p.sens_mode_k[0], p.sens_int_k[0], p.sens_k[0]);
#pragma unroll
      for (int d = 0; d < PYT; ++d) {
      const int py = py0 + d, yM = ny * M + py;
      // magnified intensity of this thread's outputs: column pass of the
      // Catmull-Rom interpolation from the row-pass values (5 taps per output)
      float2 ival[G::NPR][M];
      if (p.iw) {
        float2 rv[G::NPR][5];
#pragma unroll
        for (int pp = 0; pp < G::NPR; ++pp) {
          const float2* ri = reinterpret_cast<const float2*>(
              sm + G::O_RI + (s * G::NPR + pp) * G::S_RI) + (ty * M + py) * G::RIW + lane;
#pragma unroll
          for (int k = 0; k < 5; ++k) rv[pp][k] = ri[k];
        }
#pragma unroll
        for (int px = 0; px < M; ++px) {
#pragma unroll
          for (int pp = 0; pp < G::NPR; ++pp) ival[pp][px] = make_float2(0.f, 0.f);
#pragma unroll
          for (int k = 0; k < 5; ++k) {
            const float w = cw[(lane * M + px) * 5 + k];
#pragma unroll
            for (int pp = 0; pp < G::NPR; ++pp)
              ival[pp][px] = __ffma2_rn(make_float2(w, w), rv[pp][k], ival[pp][px]);
          }
          if (MODE != kModeSum) {
#pragma unroll
            for (int pp = 0; pp < G::NPR; ++pp)
              acc[pp][d * M + px] = __fmul2_rn(acc[pp][d * M + px], ival[pp][px]);
          }
        }
      } else if (MODE == kModeSum) {
#pragma unroll
        for (int px = 0; px < M; ++px)
#pragma unroll
          for (int pp = 0; pp < G::NPR; ++pp) ival[pp][px] = make_float2(1.f, 1.f);
      }
      if (d == PYT - 1) mbar_arrive(&empty[s]);  // slot s fully read
      // outputs in the margin are 0 whatever their intensity
      const unsigned zmask = omask >> (d * M) & ((1u << M) - 1u);
      if (MODE != kModeSum && zmask != 0) {
#pragma unroll
        for (int px = 0; px < M; ++px)
          if (zmask >> px & 1u)
#pragma unroll
            for (int pp = 0; pp < G::NPR; ++pp) acc[pp][d * M + px] = make_float2(0.f, 0.f);
      }
      if (MODE == kModeStack) {
        if (!(omask >> 31)) {
          float* o = p.out + (size_t)fa * plane + (size_t)yM * p.colsM + (size_t)nx * M;
#pragma unroll
          for (int fr = 0; fr < FP; ++fr) {
            if (fr < nf)
#pragma unroll
              for (int px = 0; px < M; ++px)
                o[fr * plane + px] = (fr & 1) ? acc[fr / 2][d * M + px].y : acc[fr / 2][d * M + px].x;
          }
        }
      } else if (MODE == kModeSum) {
        // running mean per sensitivity; unrolled over the sensitivity slots (a
        // runtime-bounded loop here made the compiler re-materialise addresses
        // in the RGC core: +14 % instructions)
#pragma unroll
        for (int k = 0; k < kMaxSens; ++k) {
          if (k >= p.n_sens) break;
          const int smode = p.sens_mode_k[k], sint = p.sens_int_k[k];
          const float sval = p.sens_k[k];
#pragma unroll
          for (int px = 0; px < M; ++px) {
            float* ks = tk + (k * G::NO + d * M + px) * G::NTC + tid;
            float2 r[G::NPR][1];
#pragma unroll
            for (int pp = 0; pp < G::NPR; ++pp) r[pp][0] = acc[pp][d * M + px];
            apply_sens_all<false>(r, smode, sint, sval);
#pragma unroll
            for (int pp = 0; pp < G::NPR; ++pp) {
              r[pp][0] = __fmul2_rn(r[pp][0], ival[pp][px]);
              if (zmask >> px & 1u) r[pp][0] = make_float2(0.f, 0.f);
            }
            float mu = first ? r[0][0].x : *ks;
#pragma unroll
            for (int fr = 0; fr < FP; ++fr)
              if (fr < nf)
                mu = fmaf(((fr & 1) ? r[fr / 2][0].y : r[fr / 2][0].x) - mu, inv_n[fr], mu);
            *ks = mu;
          }
        }
      } else {
#pragma unroll
        for (int px = 0; px < M; ++px) {
          const int o = d * M + px;
          float4* st = reinterpret_cast<float4*>(tk) + o * G::NTC + tid;
          float* stl = tk + 4 * G::NO * G::NTC + o * G::NTC + tid;
          Moments mo = moments_start(acc[0][o].x);
          if (!first) {
            const float4 t = *st;
            mo = Moments{t.x, t.y, t.z, t.w, *stl};
          }
#pragma unroll
          for (int fr = 0; fr < FP; ++fr)
            if (fr < nf && !(first && fr == 0))
              moments_push(mo, (fr & 1) ? acc[fr / 2][o].y : acc[fr / 2][o].x, inv_n[fr]);
          *st = make_float4(mo.mean, mo.m2, mo.c, mo.a);
          *stl = mo.b;
        }
      }
      }  // output row phases
    }
  }
  if (!producer && s_abort == 0 && MODE != kModeStack && !(omask >> 31)) {
    const size_t plane = (size_t)p.rowsM * p.colsM;
#pragma unroll
    for (int d = 0; d < PYT; ++d) {
      float* rec = p.out + (size_t)(tp * p.chunks + chunk) * p.F * plane +
                   (size_t)(ny * M + py0 + d) * p.colsM + (size_t)nx * M;
      if (MODE == kModeSum) {
        for (int k = 0; k < p.n_sens; ++k) {
#pragma unroll
          for (int px = 0; px < M; ++px)
            rec[k * plane + px] = tk[(k * G::NO + d * M + px) * G::NTC + tid];
        }
      } else {
#pragma unroll
        for (int px = 0; px < M; ++px) {
          const int o = d * M + px;
          const float4 t = reinterpret_cast<const float4*>(tk)[o * G::NTC + tid];
          rec[px] = t.x;
          rec[plane + px] = t.y;
          rec[2 * plane + px] = t.z;
          rec[3 * plane + px] = t.w;
          rec[4 * plane + px] = tk[4 * G::NO * G::NTC + o * G::NTC + tid];
        }
      }
    }
  }
  }  // chunk < nch
  __syncthreads();  // the unit's shared state is free for the next unit
  if (s_abort) {
    // a wait ran out: the producer leader waits (bounded) for its TMA copies
    // still in flight, then every thread leaves without writing more
    if (producer && prod.ptid == 0 && p.status) atomicOr(p.status, kDevTmaTimeout);
    if (producer && prod.ptid == 0) {
      if (tpend) (void)mbar_wait_bounded(tbar, tphase);
    }
    return;
  }
  gp += npass;
  }  // unit loop
}

template <int M, int J, int MODE, int V = 0>
size_t fused_smem_bytes(int ns_cap) {
  return FusedCfg<M, J, MODE, V>::G::smem_bytes(MODE, ns_cap);
}

template <int M, int J, int MODE, int V = 0>
cudaError_t launch_fused(const UnitTable& ut, const TmapPack& maps, int grid,
                         cudaStream_t stream) {
  using C = FusedCfg<M, J, MODE, V>;
  using G = typename C::G;
  auto kern = esrrf_fused_kernel<M, J, C::TY, C::FP, MODE, C::NP, C::PYT>;
  const size_t smem = G::smem_bytes(MODE, MODE == kModeSum ? ut.ns_cap : 1);
  if (smem > kSmemBudget) return cudaErrorInvalidValue;
  static int attr_done = -1;  // device the attributes were last set for
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (attr_done != dev) {
    const size_t cap = std::min(kSmemBudget, G::smem_bytes(MODE, C::NSC));
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    attr_done = dev;
  }
  if (grid < 1) return cudaSuccess;
  kern<<<grid, G::NT, smem, stream>>>(maps, ut);
  return cudaGetLastError();
}

// resident CTAs per SM of one instantiation (for persistent grids)
template <int M, int J, int MODE, int V = 0>
int fused_occupancy(int ns_cap) {
  using C = FusedCfg<M, J, MODE, V>;
  using G = typename C::G;
  auto kern = esrrf_fused_kernel<M, J, C::TY, C::FP, MODE, C::NP, C::PYT>;
  const size_t smem = G::smem_bytes(MODE, MODE == kModeSum ? ns_cap : 1);
  if (smem > kSmemBudget) return 0;
  // cached per device and sensitivity count (queried once; launches ask per call)
  static int cache[16][kMaxSens + 1] = {};
  int dev = 0;
  const bool cacheable = cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 16 &&
                         ns_cap >= 0 && ns_cap <= kMaxSens;
  if (cacheable && cache[dev][ns_cap] > 0) return cache[dev][ns_cap];
  int n = 0;
  const size_t cap = std::min(kSmemBudget, G::smem_bytes(MODE, C::NSC));
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap) !=
      cudaSuccess)
    return 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, G::NT, smem) != cudaSuccess)
    return 1;
  n = n > 0 ? n : 1;
  if (cacheable) cache[dev][ns_cap] = n;
  return n;
}

// geometry the host needs to build the tensor map for a given (M, J); the
// tile shape does not depend on the mode or on FP
struct FusedGeometry {
  int TY, IX, IY, BW, BH;
};

template <int M, int J, int V = 0>
FusedGeometry fused_geometry() {
  using G = Geo<M, J, EsrrfTile<M, V>::TY, 2>;
  return FusedGeometry{EsrrfTile<M, V>::TY, G::IX, G::IY, G::BW, G::BH};
}

}  // namespace nx
