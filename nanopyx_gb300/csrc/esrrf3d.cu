// eSRRF-3D: radial gradient convergence of volumes
// (src/nanopyx/core/transform/_le_esrrf3d.pyx:65-140).
//
// Per pair of consecutive frames of a (T, S, H, W) stack, as the reference:
//   1. gradients at the input resolution: central differences along x and y,
//      the backward difference along z, halved, indices clamped
//      (src/include/_c_gradients.c:75-116);
//   2. the frame and its three gradients magnified by Catmull-Rom x mxy in
//      every slice; the reference's "linear" z step then repeats each slice
//      mz times (its slice coordinate sM / mz is an integer division, so the
//      second weight is 0, _interpolation.pyx:54-88) -- here the repeat is an
//      index mapping, never materialised.  One kernel does both and stores the
//      gradients normalised, the two frames side by side;
//   3. at every output voxel inside the margins the RGC over the window of
//      input-pixel offsets (src/include/_c_sr_radial_gradient_convergence.c:
//      92-204) on packed f32x2 arithmetic (FP64 steps of the reference -- exp,
//      pow, the quotient of square roots -- in float32 or in the host's table),
//      to the power `sensitivity`, times the interpolated intensity;
//   4. the running mean (mode "average") or Welford variance (mode "std",
//      sqrt(M2 / T) at the end) over the frames, in the reference's order.
//
// The window samples of the mz voxels of one input slice are the same gradients
// at the same offsets, so their RGC is evaluated once wherever the same samples
// lie inside the volume for all of them.
//
// Rounding: weights formed in float64 and rounded once, gradients normalised to half
// an ulp, |n x offset| from exact whole-pixel offsets by one square root good to
// 2^-23, sums row by row.  Error against float64 at 20 x 16 x 128 x 128, mxy = mz = 2,
// R = 1.5: 8.8e-8; with float32 unit offsets, q rsqrt(q) and one chain of sums 9.3e-8
// (no magnification, R = 3, without intensity: 1.2e-7 against 5.6e-7).
//
// What bounds it: issue and register reads of step 3 (14 packed operations and two
// square roots per sample and frame pair) and the L1 wavefronts of its two gradient
// loads.  Same call: one frame at a time, three scalar gradients normalised at every
// sample and every voxel by itself 5.9 ms; frame pairs, gradients normalised once,
// shared z voxels 1.5 ms; window columns in registers 1.33 ms; one instruction for
// the square root 1.24 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "internal.h"

namespace nx {
namespace {

struct Rgc3d {
  int S, H, W, mxy, mz, Hm, Wm, Sm;
  int margin, margin_z;
  int s0, s1, z0, z1;  // window offsets, inclusive
  int sens_mode, sens_int;
  float sensitivity;
  int iw, mode;
};

// Steps 1 and 2 for a frame pair: a block covers kPrepCols x kPrepRows output
// pixels of one slice.  The gradients and the value of every input pixel the
// taps reach go to shared memory as (gx, gx', gy, gy') (gz, gz', v, v') -- zero
// outside the image, the reference's skipped taps -- then each thread keeps one
// output column and a run of rows: 8 shared loads give a row's 4-tap column sums
// of all quantities, and the four newest rows stay in registers.
constexpr int kPrepCols = 64, kPrepRows = 16, kPrepThreads = 256;
constexpr int kPrepRun = kPrepRows / (kPrepThreads / kPrepCols);  // rows per thread

__host__ __device__ inline int prep_extent(int n_out, int mag) { return (n_out - 1) / mag + 6; }

struct Quad {  // float4 (gx, gx', gy, gy') and (gz, gz', v, v')
  float4 a, b;
};

__device__ __forceinline__ void quad_fma(Quad& q, float w, const Quad& v) {
  const float2 w2 = make_float2(w, w);
  float2 x = __ffma2_rn(make_float2(v.a.x, v.a.y), w2, make_float2(q.a.x, q.a.y));
  float2 y = __ffma2_rn(make_float2(v.a.z, v.a.w), w2, make_float2(q.a.z, q.a.w));
  q.a = make_float4(x.x, x.y, y.x, y.y);
  x = __ffma2_rn(make_float2(v.b.x, v.b.y), w2, make_float2(q.b.x, q.b.y));
  y = __ffma2_rn(make_float2(v.b.z, v.b.w), w2, make_float2(q.b.z, q.b.w));
  q.b = make_float4(x.x, x.y, y.x, y.y);
}

// (x, y, z) to a unit vector; 0 without a gradient, and for an infinite one, whose
// samples count nothing in the reference either (its quotient is NaN there)
__device__ __forceinline__ void normalise(float& x, float& y, float& z) {
  float d = fmaf(z, z, fmaf(y, y, x * x));
  if (!(d > 1e-30f && d < 1e30f)) {  // the squares may not hold: scale first
    const float m = fmaxf(fmaxf(fabsf(x), fabsf(y)), fabsf(z));
    if (m == 0.f || isinf(m)) {
      x = y = z = 0.f;
      return;
    }
    x = __fdiv_rn(x, m);
    y = __fdiv_rn(y, m);
    z = __fdiv_rn(z, m);
    d = fmaf(z, z, fmaf(y, y, x * x));
  }
  float r = rsqrtf(d);
  r = fmaf(0.5f * r, fmaf(-d * r, r, 1.f), r);  // to half an ulp
  x *= r;
  y *= r;
  z *= r;
}

size_t rup(size_t b) { return (b + 255) / 256 * 256; }

// The magnified volumes between the two kernels: unit gradients (x, y) and z, and the
// frame, of a frame pair side by side -- A (x, x', y, y'), B (z, z'), I (v, v') -- or
// of one frame (A (x, y), B (z), I (v)) at half the memory.
template <bool PAIR>
struct Volumes {
  using TA = typename std::conditional<PAIR, float4, float2>::type;
  using TB = typename std::conditional<PAIR, float2, float>::type;
  TA* __restrict__ A;
  TB* __restrict__ B;
  TB* __restrict__ I;
  static size_t bytes(size_t voxels) {
    return rup(voxels * sizeof(TA)) + 2 * rup(voxels * sizeof(TB));
  }
  explicit Volumes(char* base, size_t voxels)
      : A((TA*)base), B((TB*)(base + rup(voxels * sizeof(TA)))),
        I((TB*)(base + rup(voxels * sizeof(TA)) + rup(voxels * sizeof(TB)))) {}
};
__device__ __forceinline__ float4 both(const float4& a) { return a; }
__device__ __forceinline__ float4 both(const float2& a) { return make_float4(a.x, a.x, a.y, a.y); }
__device__ __forceinline__ float2 two_of(const float2& a) { return a; }
__device__ __forceinline__ float2 two_of(float a) { return make_float2(a, a); }

template <bool PAIR>
__global__ void __launch_bounds__(kPrepThreads)
    prep3d_kernel(const float* __restrict__ v0, const float* __restrict__ v1, int H, int W, int m,
                  int z_first, const Volumes<PAIR> vol) {
  extern __shared__ __align__(16) float4 patch[];  // [PR][PC][2]
  const int Hm = H * m, Wm = W * m;
  const int nbx = (Wm + kPrepCols - 1) / kPrepCols;
  const int z = z_first + blockIdx.y;
  const int x0 = blockIdx.x % nbx * kPrepCols, y0 = blockIdx.x / nbx * kPrepRows;
  const int PR = prep_extent(kPrepRows, m), PC = prep_extent(kPrepCols, m);
  const int r0 = y0 / m - 2, c0 = x0 / m - 2;  // first input row / column of the patch
  const size_t plane = (size_t)H * W;
  const float* f0 = v0 + z * plane;
  const float* f1 = v1 + z * plane;
  const ptrdiff_t back = z > 0 ? -(ptrdiff_t)plane : 0;  // the slice below (clamped)
  for (int i = threadIdx.x; i < PR * PC; i += kPrepThreads) {
    const int y = r0 + i / PC, x = c0 + i % PC;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (y >= 0 && y < H && x >= 0 && x < W) {
      const size_t o = (size_t)y * W + x;
      const int xp = x < W - 1 ? 1 : 0, xm = x > 0 ? 1 : 0;
      const int yp = y < H - 1 ? W : 0, ym = y > 0 ? W : 0;
      auto grad = [&](const float* f, float& gx, float& gy, float& gz, float& val) {
        val = __ldg(f + o);
        gx = __fsub_rn(__ldg(f + o + xp), __ldg(f + o - xm)) / 2;
        gy = __fsub_rn(__ldg(f + o + yp), __ldg(f + o - ym)) / 2;
        gz = __fsub_rn(val, __ldg(f + o + back)) / 2;
      };
      grad(f0, a.x, a.z, b.x, b.z);
      grad(f1, a.y, a.w, b.y, b.w);
    }
    patch[2 * i] = a;
    patch[2 * i + 1] = b;
  }
  __syncthreads();
  const int x = x0 + threadIdx.x % kPrepCols;
  const int yb = y0 + threadIdx.x / kPrepCols * kPrepRun;
  if (x >= Wm) return;
  auto store = [&](int y, Quad q) {
    normalise(q.a.x, q.a.z, q.b.x);
    normalise(q.a.y, q.a.w, q.b.y);
    const size_t o = ((size_t)z * Hm + y) * Wm + x;
    if constexpr (PAIR) {
      vol.A[o] = q.a;
      vol.B[o] = make_float2(q.b.x, q.b.y);
      vol.I[o] = make_float2(q.b.z, q.b.w);
    } else {
      vol.A[o] = make_float2(q.a.x, q.a.z);
      vol.B[o] = q.b.x;
      vol.I[o] = q.b.z;
    }
  };
  if (m == 1) {  // not magnified: the values themselves
    for (int y = yb; y < min(yb + kPrepRun, Hm); ++y) {
      const int i = (y - r0) * PC + x - c0;
      store(y, Quad{patch[2 * i], patch[2 * i + 1]});
    }
    return;
  }
  const float col = __fdiv_rn((float)x, (float)m);
  const int cb = (int)floorf(col - 0.5f) - 1;
  const bool cin = col < (float)W;
  float wc[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) wc[k] = cin ? cr_cubic(col - ((float)(cb + k) + 0.5f)) : 0.f;
  auto across = [&](int r) {  // 4-tap sums of input row r
    Quad q{make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    const float4* p = patch + 2 * ((r - r0) * PC + cb - c0);
#pragma unroll
    for (int k = 0; k < 4; ++k) quad_fma(q, wc[k], Quad{p[2 * k], p[2 * k + 1]});
    return q;
  };
  Quad win[4];
  int top = INT_MIN;  // input row of win[0]
#pragma unroll 1
  for (int y = yb; y < min(yb + kPrepRun, Hm); ++y) {
    const float row = __fdiv_rn((float)y, (float)m);
    const int rb = (int)floorf(row - 0.5f) - 1;
    if (rb == top + 1) {
#pragma unroll
      for (int k = 0; k < 3; ++k) win[k] = win[k + 1];
      win[3] = across(rb + 3);
    } else if (rb != top) {
#pragma unroll
      for (int k = 0; k < 4; ++k) win[k] = across(rb + k);
    }
    top = rb;
    Quad q{make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    if (row < (float)H) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        quad_fma(q, cr_cubic(row - ((float)(rb + k) + 0.5f)), win[k]);
    }
    store(y, q);
  }
}

// square root to 2^-23 of |n x offset|^2, one instruction (a square below 2^-126
// counts as 0: 1e-19 of a pixel)
__device__ __forceinline__ float root(float q) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(q));
  return r;
}

// g ^ sensitivity (modes 1 to 3 of apply_sensitivity), once a voxel and frame: called, so
// that the kernel keeps to 64 registers (inlined 70, and 1.40 ms a call instead of 1.33)
__device__ __noinline__ float power3d(float g, int mode, int n, float s) {
  return mode == 2 ? powf(g, s) : power_compensated(g, n, mode == 3);
}

// Steps 3 and 4 for a frame pair: a block covers 32 x 8 output pixels inside the
// margins and the mz voxels of one input slice.  tab holds, per window offset
// [k][j][i], the weight w (0: does not count) and w over the offset's length;
// sample columns and rows, from the voxel's float32 coordinates as the reference
// forms them, are tabulated per block (-1: outside the image).
// NI: window columns known at compile time (4: radius 1 to below 2; 0: any) --
// the columns' indices stay in registers and a window row's loads are in flight
// together (whole call, 20 x 16 x 128 x 128, R = 1.5: 1.51 ms with the general
// loop, 1.28 with NI = 4; NI = 6 at R = 2 lost, 3.2 against 2.3: a third of its loads
// belong to samples outside the radius).
constexpr int kMaxWin = 64;  // window offsets per axis are at most 2 int(radius) + 2
// up to this workspace nx_esrrf3d_workspace_bytes asks for frame pairs; above it for the
// least, 16 bytes per magnified voxel instead of 32, so that a volume near the limit of
// the memory still fits (one frame at a time: 2.17 ms a call instead of 1.24)
constexpr size_t kPairBytes = 4ull << 30;
constexpr int kMaxTab = 64;  // table entries kept in shared memory (NI > 0)

template <int NI, bool PAIR>
__global__ void __launch_bounds__(256)
    rgc3d_kernel(const __grid_constant__ Rgc3d p, const Volumes<PAIR> vol,
                 const float2* __restrict__ tab, int s_first, int frame, int two,
                 float* __restrict__ out, float* __restrict__ mean) {
  using TA = typename Volumes<PAIR>::TA;
  using TB = typename Volumes<PAIR>::TB;
  __shared__ int cidx[NI > 0 ? NI : kMaxWin][32], ridx[NI > 0 ? NI : kMaxWin][8];
  __shared__ float2 stab[NI > 0 ? kMaxTab : 1];
  const int nI = NI > 0 ? NI : p.s1 - p.s0 + 1;
  if (NI > 0)
    for (int e = threadIdx.x; e < (p.z1 - p.z0 + 1) * nI * nI; e += 256) stab[e] = __ldg(tab + e);
  const int lane = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int nbx = (p.Wm - 2 * p.margin + 31) / 32;
  const int c0 = p.margin + blockIdx.x % nbx * 32, r0 = p.margin + blockIdx.x / nbx * 8;
  for (int e = threadIdx.x; e < nI * 40; e += 256) {
    const int i = e / 40, t = e % 40;
    const bool isrow = t >= 32;
    const int n = isrow ? p.H : p.W, nm = isrow ? p.Hm : p.Wm;
    // threads past the last voxel of a row or column repeat it
    const int M = min(isrow ? r0 + t - 32 : c0 + t, nm - p.margin - 1);
    const float v = __fadd_rn(__fdiv_rn((float)M, (float)p.mxy), (float)(p.s0 + i));
    const int idx =
        0.f < v && v <= (float)(n - 1) ? min((int)__fmul_rn((float)p.mxy, v), nm - 1) : -1;
    if (isrow) ridx[i][t - 32] = idx;
    else cidx[i][t] = idx;
  }
  __syncthreads();
  const int cM = c0 + lane, rM = r0 + ty;
  const bool active = cM < p.Wm - p.margin && rM < p.Hm - p.margin;
  bool all_in = true;
  for (int i = 0; i < nI; ++i) all_in = all_in && cidx[i][lane] >= 0 && ridx[i][ty] >= 0;
  const bool interior = __all_sync(0xffffffffu, all_in);
  int cx[NI > 0 ? NI : 1];
  unsigned cin = 0;  // bit i: column i lies inside the image
  if constexpr (NI > 0) {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      cx[i] = max(cidx[i][lane], 0);
      cin |= (cidx[i][lane] >= 0 ? 1u : 0u) << i;
    }
  }
  const size_t plane = (size_t)p.Hm * p.Wm;
  // voxels sM = s mz + r, r0 <= r < r1, inside the z margins
  const int s = s_first + blockIdx.y;
  const int ra = max(0, p.margin_z - s * p.mz);
  const int rb = min(p.mz, p.Sm - p.margin_z - s * p.mz);
  auto z_in = [&](int r, int k) {
    const float vz = __fadd_rn(__fdiv_rn((float)(s * p.mz + r), (float)p.mz), (float)k);
    return 0.f < vz && vz <= (float)(p.S - 1);
  };
  bool same = true;  // the same samples lie inside the volume for every r
  for (int k = p.z0; k <= p.z1; ++k)
    for (int r = ra + 1; r < rb; ++r) same = same && z_in(r, k) == z_in(ra, k);
  for (int r = ra; r < rb; r = same ? rb : r + 1) {
    // sums over window rows, then over the rows: short chains of roundings where one
    // over all 44 samples (R = 1.5) cost most of the map's error
    float2 acc = make_float2(0.f, 0.f), row = acc;
    float wsum = 0.f, wrow = 0.f;
    // one sample: unit gradients of the pair against the whole-pixel offset (x, y, z)
    auto sample = [&](float x, float y, float z, const float2& t, const float4& a,
                      const float2& nz, bool ok) {
      const float2 nx = make_float2(a.x, a.y), ny = make_float2(a.z, a.w);
      const float2 rx = make_float2(x, x), ry = make_float2(y, y), rz = make_float2(z, z);
      const float2 mx = make_float2(-x, -x), my = make_float2(-y, -y), mz = make_float2(-z, -z);
      const float2 dot = __ffma2_rn(nz, rz, __ffma2_rn(ny, ry, __fmul2_rn(nx, rx)));
      const float2 c1 = __ffma2_rn(ny, rz, __fmul2_rn(nz, my));
      const float2 c2 = __ffma2_rn(nz, rx, __fmul2_rn(nx, mz));
      const float2 c3 = __ffma2_rn(nx, ry, __fmul2_rn(ny, mx));
      const float2 q = __ffma2_rn(c3, c3, __ffma2_rn(c2, c2, __fmul2_rn(c1, c1)));
      const float2 dk = make_float2(root(q.x), root(q.y));
      const float2 v = __ffma2_rn(dk, make_float2(-t.y, -t.y), make_float2(t.x, t.x));
      row = __fadd2_rn(row, make_float2(ok && dot.x < 0.f ? v.x : 0.f,
                                        ok && dot.y < 0.f ? v.y : 0.f));
      wrow += ok ? t.x : 0.f;
    };
    for (int k = p.z0; k <= p.z1; ++k) {
      if (!z_in(r, k)) continue;
      // slice of the magnified volumes: (int)(vz mz) / mz = s + k (vz mz rounds
      // to s mz + k mz + r or, for r > 0, at worst just below it)
      const TA* Ak = vol.A + (size_t)(s + k) * plane;
      const TB* Bk = vol.B + (size_t)(s + k) * plane;
      const float z = (float)k;
      const float2* tk = (NI > 0 ? stab : tab) + (size_t)(k - p.z0) * nI * nI;
      for (int j = 0; j < nI; ++j) {
        const int ry = ridx[j][ty];
        const float y = (float)(p.s0 + j);
        const TA* Aj = Ak + (size_t)max(ry, 0) * p.Wm;
        const TB* Bj = Bk + (size_t)max(ry, 0) * p.Wm;
        if constexpr (NI > 0) {
          float4 a[NI];
          float2 nz[NI];
#pragma unroll
          for (int i = 0; i < NI; ++i) {
            a[i] = both(__ldg(Aj + cx[i]));
            nz[i] = two_of(__ldg(Bj + cx[i]));
          }
#pragma unroll
          for (int i = 0; i < NI; ++i) {
            const float2 t = tk[j * NI + i];
            if (t.x == 0.f) continue;  // does not count
            sample((float)(p.s0 + i), y, z, t, a[i], nz[i],
                   interior || (ry >= 0 && (cin >> i & 1u)));
          }
        } else {
#pragma unroll 4
          for (int i = 0; i < nI; ++i) {
            const float2 t = __ldg(tk + j * nI + i);
            if (t.x == 0.f) continue;
            const int c = cidx[i][lane];
            sample((float)(p.s0 + i), y, z, t, both(__ldg(Aj + max(c, 0))),
                   two_of(__ldg(Bj + max(c, 0))), interior || (ry >= 0 && c >= 0));
          }
        }
        acc = __fadd2_rn(acc, row);
        wsum += wrow;
        row = make_float2(0.f, 0.f);
        wrow = 0.f;
      }
    }
    if (!active) continue;
    float2 val = make_float2(__fdiv_rn(acc.x, wsum), __fdiv_rn(acc.y, wsum));
    auto power = [&](float g) {
      if (!(g >= 0.f)) return g < 0.f ? 0.f : g;
      return p.sens_mode ? power3d(g, p.sens_mode, p.sens_int, p.sensitivity) : g;
    };
    val.x = power(val.x);
    val.y = power(val.y);
    if (p.iw)
      val = __fmul2_rn(val, two_of(__ldg(vol.I + (size_t)s * plane + (size_t)rM * p.Wm + cM)));
    // voxels that share their samples share their whole history
    size_t o = ((size_t)(s * p.mz + r) * p.Hm + rM) * p.Wm + cM;
    float cur = out[o], mu = p.mode ? mean[o] : 0.f;
    for (int f = 0; f <= two; ++f) {
      const float g = f ? val.y : val.x, fr = (float)(frame + f + 1);
      if (p.mode == 0) {
        cur = __fadd_rn(cur, __fdiv_rn(__fsub_rn(g, cur), fr));
      } else {
        const float delta = __fsub_rn(g, mu);
        mu = __fadd_rn(mu, __fdiv_rn(delta, fr));
        cur = __fadd_rn(cur, __fmul_rn(delta, __fsub_rn(g, mu)));
      }
    }
    for (int q = r; q < (same ? rb : r + 1); ++q, o += plane) {
      out[o] = cur;
      if (p.mode) mean[o] = mu;
    }
  }
}

__global__ void std_finish_kernel(float* __restrict__ out, long long n, float frames) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x)
    out[e] = __fsqrt_rn(__fdiv_rn(out[e], frames));
}

unsigned grid_of(long long n) {
  return (unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, 152LL * 32));
}


}  // namespace
}  // namespace nx

using namespace nx;

extern "C" {

void nx_esrrf3d_workspace_range(int S, int H, int W, int magnification_xy, int magnification_z,
                                int mode, size_t* least, size_t* pairs) {
  size_t rest = 0, one = 256, two = 256;
  if (S >= 1 && H >= 1 && W >= 1 && magnification_xy >= 1 && magnification_z >= 1) {
    const size_t volm = (size_t)S * H * magnification_xy * W * magnification_xy;
    rest = 256 + (mode ? rup(volm * magnification_z * sizeof(float)) : 0) +
           rup((size_t)kMaxWin * kMaxWin * kMaxWin * sizeof(float2));
    one = rest + Volumes<false>::bytes(volm);
    two = rest + Volumes<true>::bytes(volm);
  }
  if (least) *least = one;
  if (pairs) *pairs = two;
}

size_t nx_esrrf3d_workspace_bytes(int S, int H, int W, int magnification_xy,
                                  int magnification_z, int mode) {
  size_t least, pairs;
  nx_esrrf3d_workspace_range(S, H, W, magnification_xy, magnification_z, mode, &least, &pairs);
  return pairs <= kPairBytes ? pairs : least;
}

int nx_esrrf3d_st(const float* d_in, int T, int S, int H, int W, int magnification_xy,
                  int magnification_z, double radius, double radius_z, float sensitivity,
                  int mode, int do_intensity_weighting, float* d_out, void* d_ws,
                  size_t ws_bytes, void* stream) {
  if (T < 1 || S < 1 || H < 1 || W < 1) return nx::set_error("bad stack shape"), NX_ERR_INVALID_ARG;
  if (magnification_xy < 1 || magnification_z < 1)
    return nx::set_error("magnifications must be >= 1"), NX_ERR_INVALID_ARG;
  if (!(radius > 0) || !(radius_z > 0))
    return nx::set_error("radius and radius_z must be > 0"), NX_ERR_INVALID_ARG;
  if (mode != 0 && mode != 1) return nx::set_error("mode must be 0 (average) or 1 (std)"), NX_ERR_INVALID_ARG;
  if (!d_in || !d_out) return nx::set_error("NULL input/output"), NX_ERR_INVALID_ARG;
  size_t need, pair_need;
  nx_esrrf3d_workspace_range(S, H, W, magnification_xy, magnification_z, mode, &need, &pair_need);
  if (!d_ws || ws_bytes < need) {
    nx::set_error("workspace too small: need %zu bytes", need);
    return NX_ERR_WORKSPACE;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const int mxy = magnification_xy, mz = magnification_z;
  Rgc3d p{};
  p.S = S;
  p.H = H;
  p.W = W;
  p.mxy = mxy;
  p.mz = mz;
  p.Hm = H * mxy;
  p.Wm = W * mxy;
  p.Sm = S * mz;
  if ((unsigned long long)p.Sm * (unsigned long long)mz >= (1ULL << 32))
    return nx::set_error("S * magnification_z^2 must be below 2^32"), NX_ERR_INVALID_ARG;
  // the reference's scalars (_le_esrrf3d.pyx:73-86): radius and radius_z are
  // Python floats, sigma and the thresholds C floats
  const float sigma = (float)(radius / 2.355);
  const float sigma_z = (float)(radius_z / 2.355);
  p.margin = (int)(radius * mxy);
  p.margin_z = (int)(radius_z * mz);
  const float tSS = 2 * sigma * sigma, tSO = 2 * sigma + 1;
  const float tSS_z = 2 * sigma_z * sigma_z, tSO_z = 2 * sigma_z + 1;
  const float fwhm = (float)radius, fwhm_z = (float)radius_z;
  p.s0 = -(int)fwhm;
  p.s1 = (int)(fwhm + 1);
  p.z0 = -(int)fwhm_z;
  p.z1 = (int)(fwhm_z + 1);
  const RgcScalars power = rgc_scalars(1, 1.f, sensitivity, 0);
  p.sens_mode = power.sens_mode;
  p.sens_int = power.sens_int;
  p.sensitivity = sensitivity;
  p.iw = do_intensity_weighting ? 1 : 0;
  p.mode = mode;
  const int nI = p.s1 - p.s0 + 1, nK = p.z1 - p.z0 + 1;
  if (nI > kMaxWin || nK > kMaxWin)
    return nx::set_error("radius too large for the 3-D window"), NX_ERR_INVALID_ARG;
  // per offset the weight of the reference's _c_calculate_dw3D
  // (src/include/_c_sr_radial_gradient_convergence.c:96-102), 0 where the sample
  // does not count, and the weight over the offset's length; formed in float64 and
  // rounded once (float32 factors to the fourth power are up to 2.4e-7 off)
  std::vector<float2> tab((size_t)nI * nI * nK);
  for (int k = p.z0; k <= p.z1; ++k)
    for (int j = p.s0; j <= p.s1; ++j)
      for (int i = p.s0; i <= p.s1; ++i) {
        const double dxy2 = (double)i * i + (double)j * j;
        const double d = std::sqrt(dxy2 + (double)k * k), dxy = std::sqrt(dxy2);
        float2 t = make_float2(0.f, 0.f);
        if (d != 0 && dxy <= (double)tSO && (double)k <= (double)tSO_z) {
          const double D = d * std::exp(-dxy2 / (double)tSS - (double)k * k / (double)tSS_z);
          const double w = D * D * D * D;
          t.x = (float)w;
          t.y = (float)(w / d);
        }
        tab[((size_t)(k - p.z0) * nI + (j - p.s0)) * nI + (i - p.s0)] = t;
      }
  // slices at the end of the window in which nothing counts
  while (p.z1 > p.z0) {
    bool any = false;
    for (size_t e = (size_t)(p.z1 - p.z0) * nI * nI; e < (size_t)(p.z1 - p.z0 + 1) * nI * nI; ++e)
      any = any || tab[e].x != 0.f;
    if (any) break;
    --p.z1;
  }
  const bool small = (p.z1 - p.z0 + 1) * nI * nI <= kMaxTab;
  const size_t vol = (size_t)S * H * W;
  const size_t volm = (size_t)S * p.Hm * p.Wm;
  const long long nout = (long long)p.Sm * p.Hm * p.Wm;
  char* b = (char*)d_ws + 256;
  const bool pair = ws_bytes >= pair_need;
  char* const volumes = b;
  b += pair ? Volumes<true>::bytes(volm) : Volumes<false>::bytes(volm);
  float* mean = mode ? (float*)b : nullptr;
  if (mode) b += rup((size_t)nout * sizeof(float));
  float2* dtab = (float2*)b;
  NX_CUDA_TRY(cudaMemcpyAsync(dtab, tab.data(), tab.size() * sizeof(float2),
                              cudaMemcpyHostToDevice, s));
  NX_CUDA_TRY(cudaMemsetAsync(d_out, 0, (size_t)nout * sizeof(float), s));
  if (mean) NX_CUDA_TRY(cudaMemsetAsync(mean, 0, (size_t)nout * sizeof(float), s));
  const int ncol = p.Wm - 2 * p.margin, nrow = p.Hm - 2 * p.margin, nz = p.Sm - 2 * p.margin_z;
  const bool inside = ncol > 0 && nrow > 0 && nz > 0;
  // input slices that hold a voxel inside the z margins
  const int sa = p.margin_z / mz, sb = inside ? (p.Sm - p.margin_z - 1) / mz : sa - 1;
  const unsigned prep_blocks = (unsigned)((p.Wm + kPrepCols - 1) / kPrepCols) *
                               (unsigned)((p.Hm + kPrepRows - 1) / kPrepRows);
  const unsigned rgc_blocks =
      inside ? (unsigned)((ncol + 31) / 32) * (unsigned)((nrow + 7) / 8) : 0;
  const size_t smem =
      (size_t)prep_extent(kPrepRows, mxy) * prep_extent(kPrepCols, mxy) * 2 * sizeof(float4);
  const auto frames = [&](auto is_pair) {
    constexpr bool PAIR = decltype(is_pair)::value;
    const Volumes<PAIR> v(volumes, volm);
    const auto rgc = small && nI == 4 ? rgc3d_kernel<4, PAIR> : rgc3d_kernel<0, PAIR>;
    for (int f = 0; f < T && inside; f += PAIR ? 2 : 1) {
      const float* f0 = d_in + (size_t)f * vol;
      const int two = PAIR && f + 1 < T;  // an odd last frame stands in for its partner
      for (int z = 0; z < S; z += 65535) {  // grid.y limit
        prep3d_kernel<PAIR><<<dim3(prep_blocks, (unsigned)std::min(S - z, 65535)), kPrepThreads,
                              smem, s>>>(f0, two ? f0 + vol : f0, H, W, mxy, z, v);
        if (cudaError_t e = cudaGetLastError()) return e;
      }
      for (int z = sa; z <= sb; z += 65535) {
        rgc<<<dim3(rgc_blocks, (unsigned)std::min(sb - z + 1, 65535)), 256, 0, s>>>(
            p, v, dtab, z, f, two, d_out, mean);
        if (cudaError_t e = cudaGetLastError()) return e;
      }
    }
    return cudaSuccess;
  };
  NX_CUDA_TRY(pair ? frames(std::true_type{}) : frames(std::false_type{}));
  if (mode == 1) {
    std_finish_kernel<<<grid_of(nout), 256, 0, s>>>(d_out, nout, (float)T);
    NX_CUDA_TRY(cudaGetLastError());
  }
  return NX_OK;
}

}  // extern "C"
