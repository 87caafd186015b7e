// Fourier ("FHT") interpolation of the use_fht=True eSRRF path
// (src/nanopyx/core/transform/interpolation.py:22-290; used by
// _le_esrrf.pyx:183-188), on the GPU as dense linear algebra.
//
// The reference interpolates a frame (or a 256-pixel tile of it) by
//   1. tiling it with alternating mirror images and cropping the central
//      N x N square, N the power of two covering both sides;
//   2. moving its spectrum (real FFT along x, complex along y) into an
//      L x L zero spectrum, L = N mag (the upper half of the y frequencies to
//      the top end), inverting, and
//   3. rescaling the result onto the frame's [min, max] and cropping the
//      central (mag h) x (mag w) window;
// frames over 256 px a side are done in overlapping 256-pixel tiles blended
// with Hann windows.  Steps 1-2 are linear and separable:
//   Z = A_re X C_re^T - A_im X C_im^T,
//   A[i][n] = (1/L) sum_{f=-(N-N2)}^{N2-1} e^{2 pi i f (i/L - n/N)}, N2 = ceil(N/2)
//   C[j][m] = (1/L) sum_{k=0}^{N/2} c_k e^{2 pi i k (j/L - m/N)}, c_0 = 1, else 2
// (the one unpaired y frequency makes A complex; the half spectrum along x
// gives C).  That frequency alone makes A_im: A_im[i][n] = -(-1)^n sin(pi i / mag)
// / L, so the second term is the outer product of s_i = sin(pi i / mag) / L and
// r = (sum_n (-1)^n X[n]) C_im^T.  The mirror images are linear too: X = P_h T P_w^T
// of the th x tw tile T, so P goes into the operators (A_re P_h, C P_w and the signs,
// folded in float64 on the host) and the products run over the tile's own rows and
// columns instead of N: two batched FP32 GEMMs plus a rank-1 update.  FP32 on the
// CUDA cores, not TF32 on the tensor cores: the reference transforms in float64,
// and a 10-bit mantissa would not hold the 1e-4 parity bar.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "internal.h"

namespace nx {
namespace {

constexpr int kFhtTile = 256;     // tile side of the reference's tiled path
constexpr int kFhtOverlap = 16;
// Frames per GEMM batch: as many as keep their interpolated squares within half of
// the L2 (the finish kernel reads them back), at least 8 and at most 64, so that
// small squares fill the SMs: 100 x 64 x 64 at m = 2 in 69 us, 16 x 256 x 256 at m = 4 in
// 277, 16 x 200 x 200 at m = 4 in 225 (282 in chunks of 8)
constexpr int kFhtChunkMin = 8, kFhtChunkMax = 64;
constexpr size_t kFhtChunkBytes = 64u << 20;

int pow2_ceil(int n) {
  int p = 1;
  while (p < n) p <<= 1;
  return p;
}

// order-preserving int image of a float, for atomicMin / atomicMax
__device__ __forceinline__ int ordered(float f) {
  const int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float unordered(int i) {
  return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff);
}

__device__ __forceinline__ void block_minmax(float lo, float hi, int* slot) {
  __shared__ float slo[32], shi[32];
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    slo[w] = lo;
    shi[w] = hi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < nw; ++k) {
      lo = fminf(lo, slo[k]);
      hi = fmaxf(hi, shi[k]);
    }
    atomicMin(slot, ordered(lo));
    atomicMax(slot + 1, ordered(hi));
  }
}

// ---------------------------------------------------------------------------
// batched FP32 GEMM, row major: C = A B, 64 x 64 tiles, 4 x 4 per thread
// ---------------------------------------------------------------------------
struct GemmBatch {
  int inner;                    // batch index z = outer * inner + inner_index
  long long sa_o, sa_i, sb_o, sb_i, sc_o, sc_i;
};

// The second product's epilogue: z += s_i r_j (s given), and (min, max) of all z
// into mm[4 batch + 2 ..] (mm given).
struct Rank1 {
  const float* s;     // s_i at s[i * lds]
  long long lds;
  const float* r;     // r_j of a batch at r[batch * N + j]
  int* mm;
};

constexpr int kGB = 64, kGK = 16;

__global__ void __launch_bounds__(256) sgemm_kernel(const float* __restrict__ A,
                                                    const float* __restrict__ B,
                                                    float* __restrict__ C, int M, int N, int K,
                                                    int lda, int ldb, int ldc, GemmBatch bt,
                                                    Rank1 u) {
  __shared__ __align__(16) float As[kGK][kGB + 4];
  __shared__ __align__(16) float Bs[kGK][kGB + 4];
  const int zo = blockIdx.z / bt.inner, zi = blockIdx.z % bt.inner;
  A += zo * bt.sa_o + zi * bt.sa_i;
  B += zo * bt.sb_o + zi * bt.sb_i;
  C += zo * bt.sc_o + zi * bt.sc_i;
  const int m0 = blockIdx.y * kGB, n0 = blockIdx.x * kGB;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += kGK) {
    for (int e = threadIdx.x; e < kGB * kGK; e += 256) {
      const int r = e / kGK, c = e % kGK;  // A tile: row r, column c
      const int gm = m0 + r, gk = k0 + c;
      As[c][r] = (gm < M && gk < K) ? __ldg(A + (size_t)gm * lda + gk) : 0.f;
      const int br = e / kGB, bc = e % kGB;  // B tile: row br, column bc
      const int bk = k0 + br, bn = n0 + bc;
      Bs[br][bc] = (bk < K && bn < N) ? __ldg(B + (size_t)bk * ldb + bn) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kGK; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(&As[k][ty * 4]);
      const float4 b = *reinterpret_cast<const float4*>(&Bs[k][tx * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    __syncthreads();
  }
  float lo = INFINITY, hi = -INFINITY;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
    const float si = u.s ? __ldg(u.s + gm * u.lds) : 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx * 4 + j;
      if (gn >= N) continue;
      float v = acc[i][j];
      if (u.s) v = fmaf(si, __ldg(u.r + (size_t)blockIdx.z * N + gn), v);
      lo = fminf(lo, v);
      hi = fmaxf(hi, v);
      C[(size_t)gm * ldc + gn] = v;
    }
  }
  if (u.mm) block_minmax(lo, hi, u.mm + 4 * blockIdx.z + 2);
}


// The same product in 64 HA x 64 HB tiles, 4 HA x 4 HB per thread on packed f32x2
// (two columns per register pair), the next K slice loaded into registers behind
// the current one and stored to the other half of a double buffer.  Needs K a
// multiple of 16, N and the leading dimensions multiples of 4 and 16-byte
// aligned operands; M is guarded per row.  Every output is one chain of fused
// multiply-adds in ascending k, so the tile changes no bit.
constexpr int kBK = 16;
// more blocks than this for a tile to be taken: one for every SM.  The products of
// 8 frames of 300 x 260 at m = 2 (20 to 512 blocks of 128 x 128): 696 us in 128 x 128
// tiles alone, 602 / 579 / 606 us with the line at 76 / 152 / 304 blocks; one
// 512 x 512 frame at m = 2 whole: 623, 427 / 428 / 424 us.
constexpr int kGemmFill = 152;
template <int HA, int HB>
__global__ void __launch_bounds__(256, 2)
    sgemm_big_kernel(const float* __restrict__ A, const float* __restrict__ B,
                     float* __restrict__ C, int M, int N, int K, int lda, int ldb, int ldc,
                     GemmBatch bt, Rank1 u) {
  constexpr int BM = 64 * HA, BN = 64 * HB;
  __shared__ __align__(16) float As[2][kBK][BM + 4];
  __shared__ __align__(16) float Bs[2][kBK][BN];
  const int zo = blockIdx.z / bt.inner, zi = blockIdx.z % bt.inner;
  A += zo * bt.sa_o + zi * bt.sa_i;
  B += zo * bt.sb_o + zi * bt.sb_i;
  C += zo * bt.sc_o + zi * bt.sc_i;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  // staging: thread t loads A rows t / 4 + 64 h, K quad t % 4, and HB quads of the
  // B slice, row by row
  constexpr int QB = BN / 4, RB = 256 / QB;
  const int ar = tid / 4, ak = tid % 4 * 4, br = tid / QB, bc = tid % QB * 4;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 pa[HA], pb[HB];
  auto load = [&](int k0) {
#pragma unroll
    for (int h = 0; h < HA; ++h) {
      const int gm = m0 + ar + 64 * h;
      pa[h] = gm < M ? __ldg(reinterpret_cast<const float4*>(A + (size_t)gm * lda + k0 + ak)) : zero;
    }
#pragma unroll
    for (int h = 0; h < HB; ++h)
      pb[h] = n0 + bc < N ? __ldg(reinterpret_cast<const float4*>(
                                B + (size_t)(k0 + br + RB * h) * ldb + n0 + bc))
                          : zero;
  };
  auto store = [&](int b) {
#pragma unroll
    for (int h = 0; h < HA; ++h) {
      As[b][ak][ar + 64 * h] = pa[h].x;
      As[b][ak + 1][ar + 64 * h] = pa[h].y;
      As[b][ak + 2][ar + 64 * h] = pa[h].z;
      As[b][ak + 3][ar + 64 * h] = pa[h].w;
    }
#pragma unroll
    for (int h = 0; h < HB; ++h) *reinterpret_cast<float4*>(&Bs[b][br + RB * h][bc]) = pb[h];
  };
  // rows ty * 4 + {0..3} + 64 h, columns tx * 4 + {0..3} + 64 h
  float2 acc[4 * HA][2 * HB];
#pragma unroll
  for (int i = 0; i < 4 * HA; ++i)
#pragma unroll
    for (int j = 0; j < 2 * HB; ++j) acc[i][j] = make_float2(0.f, 0.f);
  load(0);
  store(0);
  __syncthreads();
  int b = 0;
  for (int k0 = 0; k0 < K; k0 += kBK, b ^= 1) {
    const bool more = k0 + kBK < K;
    if (more) load(k0 + kBK);
#pragma unroll
    for (int k = 0; k < kBK; ++k) {
      float4 av[HA];
      float2 bv[2 * HB];
#pragma unroll
      for (int h = 0; h < HA; ++h) av[h] = *reinterpret_cast<const float4*>(&As[b][k][64 * h + ty * 4]);
#pragma unroll
      for (int h = 0; h < HB; ++h) {
        const float4 v = *reinterpret_cast<const float4*>(&Bs[b][k][64 * h + tx * 4]);
        bv[2 * h] = make_float2(v.x, v.y);
        bv[2 * h + 1] = make_float2(v.z, v.w);
      }
#pragma unroll
      for (int i = 0; i < 4 * HA; ++i) {
        const float4 q = av[i >> 2];
        const float a = (i & 3) == 0 ? q.x : (i & 3) == 1 ? q.y : (i & 3) == 2 ? q.z : q.w;
#pragma unroll
        for (int j = 0; j < 2 * HB; ++j)
          acc[i][j] = __ffma2_rn(make_float2(a, a), bv[j], acc[i][j]);
      }
    }
    if (more) store(b ^ 1);
    __syncthreads();
  }
  float lo = INFINITY, hi = -INFINITY;
#pragma unroll
  for (int i = 0; i < 4 * HA; ++i) {
    const int gm = m0 + ty * 4 + (i & 3) + (i >> 2) * 64;
    if (gm >= M) continue;
    const float si = u.s ? __ldg(u.s + gm * u.lds) : 0.f;
#pragma unroll
    for (int h = 0; h < HB; ++h) {
      const int gn = n0 + tx * 4 + 64 * h;
      if (gn >= N) continue;
      float4 v = make_float4(acc[i][2 * h].x, acc[i][2 * h].y, acc[i][2 * h + 1].x,
                             acc[i][2 * h + 1].y);
      if (u.s) {
        const float4 r = __ldg(reinterpret_cast<const float4*>(u.r + (size_t)blockIdx.z * N + gn));
        v = make_float4(fmaf(si, r.x, v.x), fmaf(si, r.y, v.y), fmaf(si, r.z, v.z),
                        fmaf(si, r.w, v.w));
      }
      lo = fminf(lo, fminf(fminf(v.x, v.y), fminf(v.z, v.w)));
      hi = fmaxf(hi, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
      *reinterpret_cast<float4*>(C + (size_t)gm * ldc + gn) = v;
    }
  }
  if (u.mm) block_minmax(lo, hi, u.mm + 4 * blockIdx.z + 2);
}

// operands the vector form can take
bool vector_operands(const float* A, const float* B, const float* C, int N, int K, int lda,
                     int ldb, int ldc, const GemmBatch& bt, const Rank1& u) {
  const uintptr_t ptrs = reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) |
                         reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(u.r);
  const long long strides = lda | ldb | ldc | bt.sa_o | bt.sa_i | bt.sb_o | bt.sb_i | bt.sc_o |
                            bt.sc_i;
  return (ptrs & 15u) == 0 && strides % 4 == 0 && K % kBK == 0 && N % 4 == 0;
}

template <int HA, int HB>
cudaError_t gemm_big(const float* A, const float* B, float* C, int M, int N, int K, int lda,
                     int ldb, int ldc, int batches, const GemmBatch& bt, const Rank1& u,
                     cudaStream_t s) {
  const dim3 grid((unsigned)((N + 64 * HB - 1) / (64 * HB)), (unsigned)((M + 64 * HA - 1) / (64 * HA)),
                  (unsigned)batches);
  sgemm_big_kernel<HA, HB><<<grid, 256, 0, s>>>(A, B, C, M, N, K, lda, ldb, ldc, bt, u);
  return cudaGetLastError();
}

cudaError_t gemm(const float* A, const float* B, float* C, int M, int N, int K, int lda, int ldb,
                 int ldc, int batches, const GemmBatch& bt, const Rank1& u, cudaStream_t s) {
  if (vector_operands(A, B, C, N, K, lda, ldb, ldc, bt, u)) {
    // the largest tile that still gives every SM a block, else the smallest
    const auto blocks = [&](int ha, int hb) {
      return (long long)((N + 64 * hb - 1) / (64 * hb)) * ((M + 64 * ha - 1) / (64 * ha)) * batches;
    };
    if (blocks(2, 2) > kGemmFill)
      return gemm_big<2, 2>(A, B, C, M, N, K, lda, ldb, ldc, batches, bt, u, s);
    if (blocks(1, 2) > kGemmFill)
      return gemm_big<1, 2>(A, B, C, M, N, K, lda, ldb, ldc, batches, bt, u, s);
    return gemm_big<1, 1>(A, B, C, M, N, K, lda, ldb, ldc, batches, bt, u, s);
  }
  const dim3 grid((unsigned)((N + kGB - 1) / kGB), (unsigned)((M + kGB - 1) / kGB),
                  (unsigned)batches);
  sgemm_kernel<<<grid, 256, 0, s>>>(A, B, C, M, N, K, lda, ldb, ldc, bt, u);
  return cudaGetLastError();
}

// a[z][c] = sum_n e[n] X[z][n][c] over the nr rows of a tile (nc columns): e holds
// the signs (-1)^n of the square's rows, summed over a tile row's images
__global__ void __launch_bounds__(256) fht_alternate_kernel(const float* __restrict__ X,
                                                            const float* __restrict__ e, int nr,
                                                            int nc, float* __restrict__ a) {
  __shared__ float red[8][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  const float* x = X + (size_t)blockIdx.y * nr * nc;
  float t = 0.f;
  if (c < nc) {
#pragma unroll 4
    for (int n = g; n < nr; n += 8) t = fmaf(__ldg(e + n), __ldg(x + (size_t)n * nc + c), t);
  }
  red[g][lane] = t;
  __syncthreads();
  if (g == 0 && c < nc) {
    t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += red[k][lane];
    a[(size_t)blockIdx.y * nc + c] = t;
  }
}

// r[z][j] = sum_c a[z][c] Cim[c][j].  Up to kAltInline rows and columns a block forms
// a itself from the tile (X given), a launch less; and block 0 clears the
// extremes the next tile will use (next_mm, n of them).
constexpr int kAltInline = 128;
__global__ void __launch_bounds__(256) fht_rank1_kernel(const float* __restrict__ X,
                                                        const float* __restrict__ e,
                                                        const float* __restrict__ a,
                                                        const float* __restrict__ Cim, int nr,
                                                        int nc, int L, float* __restrict__ r,
                                                        int* __restrict__ next_mm, int n) {
  __shared__ float red[8][32];
  __shared__ float as[kAltInline];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + lane;
  if (blockIdx.x == 0 && blockIdx.y == 0)
    for (int k = threadIdx.x; k < 4 * n; k += 256) next_mm[k] = (k & 1) ? INT_MIN : INT_MAX;
  const float* az = a + (size_t)blockIdx.y * nc;
  if (X) {
    const float* x = X + (size_t)blockIdx.y * nr * nc;
    for (int c = threadIdx.x; c < nc; c += 256) {
      float even = 0.f, odd = 0.f;  // nr is a multiple of 16
#pragma unroll 4
      for (int k = 0; k < nr; k += 2) {
        even = fmaf(__ldg(e + k), __ldg(x + (size_t)k * nc + c), even);
        odd = fmaf(__ldg(e + k + 1), __ldg(x + (size_t)(k + 1) * nc + c), odd);
      }
      as[c] = even + odd;
    }
    __syncthreads();
    az = as;
  }
  float t = 0.f;
  if (j < L) {
#pragma unroll 4
    for (int c = g; c < nc; c += 8) t = fmaf(az[c], __ldg(Cim + (size_t)c * L + j), t);
  }
  red[g][lane] = t;
  __syncthreads();
  if (g == 0 && j < L) {
#pragma unroll
    for (int k = 1; k < 8; ++k) t += red[k][lane];
    r[(size_t)blockIdx.y * L + j] = t;
  }
}

// mirror-padded N x N square of tile (r0, c0, th, tw) of every frame of the
// chunk; slot[z] = (min, max) of the tile (every tile pixel is in the square:
// the upright centre copy lies inside the central crop)
__global__ void fht_gather_kernel(const float* __restrict__ in, int H, int W, int r0, int c0,
                                  int th, int tw, int N, int kh, int kw, int y_roi, int x_roi,
                                  float* __restrict__ X, int* __restrict__ mm) {
  const int z = blockIdx.y;
  const float* f = in + (size_t)z * H * W;
  float lo = INFINITY, hi = -INFINITY;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < N * N; e += gridDim.x * blockDim.x) {
    const int y = e / N, x = e % N;
    const int yp = y + y_roi, xp = x + x_roi;
    const int cy = yp / th, yy = yp % th, cx = xp / tw, xx = xp % tw;
    const int row = ((cy - (kh - 1) / 2) & 1) ? th - 1 - yy : yy;
    const int col = ((cx - (kw - 1) / 2) & 1) ? tw - 1 - xx : xx;
    const float v = __ldg(f + (size_t)(r0 + row) * W + (c0 + col));
    X[(size_t)z * N * N + e] = v;
    lo = fminf(lo, v);
    hi = fmaxf(hi, v);
  }
  block_minmax(lo, hi, mm + 4 * z);
}

// tile (r0, c0, th, tw) of every frame of the chunk as nr x nc, zeros past its edges;
// slot[z] = (min, max) of the tile
__global__ void fht_tile_kernel(const float* __restrict__ in, int H, int W, int r0, int c0, int th,
                                int tw, int nr, int nc, float* __restrict__ X,
                                int* __restrict__ mm) {
  const int z = blockIdx.y;
  const float* f = in + (size_t)z * H * W + (size_t)r0 * W + c0;
  float* o = X + (size_t)z * nr * nc;
  float lo = INFINITY, hi = -INFINITY;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nr * nc; e += gridDim.x * blockDim.x) {
    const int y = e / nc, x = e % nc;
    float v = 0.f;
    if (y < th && x < tw) {
      v = __ldg(f + (size_t)y * W + x);
      lo = fminf(lo, v);
      hi = fmaxf(hi, v);
    }
    o[e] = v;
  }
  block_minmax(lo, hi, mm + 4 * z);
}

__global__ void fht_mm_init_kernel(int* __restrict__ mm, int n) {
  for (int k = threadIdx.x; k < 4 * n; k += blockDim.x) mm[k] = (k & 1) ? INT_MIN : INT_MAX;
}

// rescale onto the tile's [min, max] (the reference's float32 steps
// -= out_min, *= scale, += orig_min), crop, and either store (one piece) or
// add the Hann-weighted piece (tiled: output += piece * outer(wr, wc)).  Pixels no
// earlier tile reaches (from row y_new, column x_new on) start from zero, and pixels
// no later tile reaches (before y_last, x_last) are divided by their summed weights,
// so that most outputs are written once and never read: 8 frames of 300 x 260 at
// m = 2, three interpolations: 117 us, against 164 + 44 + 18 us with a pass that
// clears the output first and one that divides it last.
// The scale is a float64 quotient of the float32 extremes rounded once
// (interpolation.py takes the extremes as Python floats), or float32
// arithmetic throughout (f32_scale: _interpolation.pyx keeps them in C floats).
constexpr int kFinishRows = 16;  // rows per thread: no index division, loads in flight
__global__ void fht_finish_kernel(const float* __restrict__ Z, int L, const int* __restrict__ mm,
                                  int oh, int ow, int y_roi, int x_roi,
                                  const float* __restrict__ wr, const float* __restrict__ wc,
                                  const float* __restrict__ wgt, int y_new, int x_new,
                                  int y_last, int x_last, float* __restrict__ out, int outH,
                                  int outW, int R0, int C0, int f32_scale) {
  const int z = blockIdx.z;
  const float lo = unordered(mm[4 * z]), hi = unordered(mm[4 * z + 1]);
  const float zlo = unordered(mm[4 * z + 2]), zhi = unordered(mm[4 * z + 3]);
  const bool resc = zhi != zlo;
  // one float64 division per block: with one per thread the FP64 pipe was busiest
  // (157 us, 8 rows per thread)
  __shared__ float block_scale;
  if (threadIdx.x == 0 && resc)
    block_scale = f32_scale ? __fdiv_rn(__fsub_rn(hi, lo), __fsub_rn(zhi, zlo))
                            : __double2float_rn(__ddiv_rn((double)hi - (double)lo,
                                                          (double)zhi - (double)zlo));
  __syncthreads();
  const float scale = resc ? block_scale : 1.f;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= ow) return;
  const float wx = wr ? wc[x] : 1.f;
  const int y1 = min(oh, (int)(blockIdx.y + 1) * kFinishRows);
  int y = blockIdx.y * kFinishRows;
  const float* zp = Z + (size_t)z * L * L + (size_t)(y_roi + y) * L + x_roi + x;
  const size_t at = (size_t)(R0 + y) * outW + C0 + x;
  float* o = out + (size_t)z * outH * outW + at;
  const float* g = wgt + at;
  // four rows at a time, all loads before the first store
  for (; y < y1; y += 4, zp += 4 * (size_t)L, o += 4 * (size_t)outW, g += 4 * (size_t)outW) {
    float v[4], a[4], w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool in = y + k < y1;
      v[k] = in ? zp[(size_t)k * L] : 0.f;
      a[k] = wr && in && (y + k < y_new || x < x_new) ? o[(size_t)k * outW] : 0.f;
      w[k] = wr && in && y + k < y_last && x < x_last ? __ldg(g + (size_t)k * outW) : 0.f;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (y + k >= y1) break;
      float r = v[k];
      if (resc) r = __fadd_rn(__fmul_rn(__fsub_rn(r, zlo), scale), lo);
      if (wr) {
        r = __fadd_rn(a[k], __fmul_rn(r, __fmul_rn(wr[y + k], wx)));
        if (w[k] > 0.f) r = __fdiv_rn(r, w[k]);
      }
      o[(size_t)k * outW] = r;
    }
  }
}

__global__ void fht_weight_kernel(const float* __restrict__ wr, const float* __restrict__ wc,
                                  int oh, int ow, float* __restrict__ wgt, int outW, int R0,
                                  int C0) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)oh * ow;
       e += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(e / ow), x = (int)(e % ow);
    const size_t oi = (size_t)(R0 + y) * outW + (C0 + x);
    wgt[oi] = __fadd_rn(wgt[oi], __fmul_rn(wr[y], wc[x]));
  }
}

unsigned blocks_for(long long n, int per = 256, long long cap = 4096) {
  return (unsigned)std::max<long long>(1, std::min<long long>((n + per - 1) / per, cap));
}

}  // namespace
}  // namespace nx

// ---------------------------------------------------------------------------
// plan: tile layout, operators per padded size, windows, blending weights
// ---------------------------------------------------------------------------
struct nx_fht_plan {
  struct Ops {    // full-spectrum variant, per padded size
    int N, L;
    float* ct;    // [2][N][L]: C_re^T then C_im^T
    float* acat;  // [L][2N]: A_re | -A_im
  };
  struct RowOps {  // per (padded size, tile height); n = th rounded up to 16
    int N, th, n;
    float* a;  // [L][n]: A_re with the mirror images folded in
    float* s;  // [L]: the rank-1 term's column
    float* e;  // [n]: its row signs
  };
  struct ColOps {  // per (padded size, tile width); n = tw rounded up to 16
    int N, tw, n;
    float* ct;  // [2][n][L]: C_re^T then C_im^T, folded
  };
  struct Tile {
    int r0, c0, th, tw, N, ops, rows, cols, kh, kw, y_roi, x_roi;
    float *wr, *wc;  // Hann windows (tiled path), device
    int y_new, x_new, y_last, x_last;  // magnified: covered by earlier / later tiles
  };
  int H, W, mag, device, variant;
  bool tiled;
  std::vector<Ops> ops;
  std::vector<RowOps> row_ops;
  std::vector<ColOps> col_ops;
  std::vector<Tile> tiles;
  std::vector<float*> bufs;  // every device allocation of the plan
  float* wgt = nullptr;      // (H mag, W mag) blending weights (tiled path)
  size_t frame_floats = 0;   // workspace floats per frame of a chunk
  int chunk = 1;             // frames per chunk
};

namespace nx {
namespace {

std::vector<int> tile_starts(int dim) {
  const int step = std::max(1, kFhtTile - 2 * kFhtOverlap);
  std::vector<int> s;
  for (int v = 0; v < dim; v += step) s.push_back(v);
  if (!s.empty() && s.back() + kFhtTile < dim) s.push_back(std::max(0, dim - kFhtTile));
  return s;
}

// The float64 operators of one padded size.  Both sums are geometric series:
// sum_{f=a}^{b} e^{2 pi i f t} = e^{i pi (a+b) t} sin(pi (b-a+1) t) / sin(pi t),
// and (b - a + 1) at t = 0 -- the only integer phase, since t = (i - n mag) / L
// lies in (-1, 1).  With |t| >= 1 / L the quotient is well conditioned.  An entry
// depends on d = i - n mag only: every operator is read from tables over d.
struct OpTables {
  int N, mag, L;
  std::vector<double> are, aim, cre, cim;  // [d + L]; aim holds -A_im
  OpTables(int N_, int mag_) : N(N_), mag(mag_), L(N_ * mag_) {
    const int N2 = (N + 1) / 2;
    const int fa = -(N - N2), fb = N2 - 1;  // y frequencies kept
    const int K = N / 2;                    // x frequencies kept: 0 .. K
    const double pi = 3.14159265358979323846;
    for (auto* v : {&are, &aim, &cre, &cim}) v->resize((size_t)2 * L);
    for (int d = 1 - L; d < L; ++d) {
      const double t = (double)d / L;  // i / L - n / N
      // A: sum over f = fa .. fb
      const double da = d == 0 ? (double)(fb - fa + 1)
                               : std::sin(pi * (fb - fa + 1) * t) / std::sin(pi * t);
      const double pa = pi * (fa + fb) * t;
      are[d + L] = std::cos(pa) * da / L;
      aim[d + L] = -std::sin(pa) * da / L;
      // C: 2 sum_{k=0}^{K} e^{2 pi i k t} - 1
      const double dc = d == 0 ? (double)(K + 1) : std::sin(pi * (K + 1) * t) / std::sin(pi * t);
      const double pc = pi * K * t;
      cre[d + L] = (2.0 * std::cos(pc) * dc - 1.0) / L;
      cim[d + L] = 2.0 * std::sin(pc) * dc / L;
    }
  }
  size_t at(int i, int n) const { return (size_t)(i - n * mag + L); }
};

// Both axes with the whole complex spectrum f = -N/2 .. N/2-1 (the fft2 /
// centred-block / ifft2 form of _interpolation.pyx:153-200), i.e. C = A, rounded
// once to float.
void build_full_ops(const OpTables& o, std::vector<float>& ct, std::vector<float>& acat) {
  const int N = o.N, L = o.L;
  ct.assign((size_t)2 * N * L, 0.f);
  acat.assign((size_t)L * 2 * N, 0.f);
  for (int i = 0; i < L; ++i)
    for (int n = 0; n < N; ++n) {
      acat[(size_t)i * 2 * N + n] = (float)o.are[o.at(i, n)];
      acat[(size_t)i * 2 * N + N + n] = (float)o.aim[o.at(i, n)];
      ct[(size_t)n * L + i] = (float)o.are[o.at(i, n)];
      ct[(size_t)N * L + (size_t)n * L + i] = (float)-o.aim[o.at(i, n)];
    }
}

// the tile row (or column) that row n of the square shows: k copies of `size`,
// the centre one upright, the square's first row roi rows into them
int mirror_index(int n, int size, int k, int roi) {
  const int copy = (n + roi) / size, in = (n + roi) % size;
  return ((copy - (k - 1) / 2) & 1) ? size - 1 - in : in;
}

int round16(int n) { return (n + 15) / 16 * 16; }

// A_re, s and the signs for tiles of th rows: the columns of a tile row's images
// are added in float64 and rounded once
void build_row_ops(const OpTables& o, int th, int k, int roi, std::vector<float>& a,
                   std::vector<float>& s, std::vector<float>& e) {
  const int N = o.N, L = o.L, nr = round16(th);
  std::vector<double> row(nr), sign(nr, 0.0);
  std::vector<int> of(N);
  for (int n = 0; n < N; ++n) {
    of[n] = mirror_index(n, th, k, roi);
    sign[of[n]] += (n & 1) ? -1.0 : 1.0;
  }
  a.resize((size_t)L * nr);
  s.resize(L);
  for (int i = 0; i < L; ++i) {
    std::fill(row.begin(), row.end(), 0.0);
    for (int n = 0; n < N; ++n) row[of[n]] += o.are[o.at(i, n)];
    for (int n = 0; n < nr; ++n) a[(size_t)i * nr + n] = (float)row[n];
    s[i] = (float)o.aim[o.at(i, 0)];
  }
  e.assign(sign.begin(), sign.end());
}

// C_re^T and C_im^T for tiles of tw columns
void build_col_ops(const OpTables& o, int tw, int k, int roi, std::vector<float>& ct) {
  const int N = o.N, L = o.L, nc = round16(tw);
  std::vector<double> acc((size_t)2 * nc * L, 0.0);
  for (int n = 0; n < N; ++n) {
    const int c = mirror_index(n, tw, k, roi);
    double* re = acc.data() + (size_t)c * L;
    double* im = re + (size_t)nc * L;
    for (int i = 0; i < L; ++i) {
      re[i] += o.cre[o.at(i, n)];
      im[i] += o.cim[o.at(i, n)];
    }
  }
  ct.assign(acc.begin(), acc.end());
}

std::vector<float> hann_inner(int n) {
  // numpy.hanning(n + 2)[1:-1] cast to float32
  std::vector<float> w(n);
  const double pi = 3.14159265358979323846;
  for (int k = 1; k <= n; ++k) w[k - 1] = (float)(0.5 - 0.5 * std::cos(2.0 * pi * k / (n + 1)));
  return w;
}

int fht_upload(nx_fht_plan* p, const std::vector<float>& h, float** out) {
  float* d = nullptr;
  cudaError_t e = cudaMalloc(&d, h.size() * sizeof(float));
  if (e != cudaSuccess) return cuda_status(e, "FHT plan allocation");
  p->bufs.push_back(d);
  e = cudaMemcpy(d, h.data(), h.size() * sizeof(float), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return cuda_status(e, "FHT plan upload");
  *out = d;
  return NX_OK;
}

// the operators of a tile, shared by the tiles of the same sizes
int build_tile_ops(nx_fht_plan* p, nx_fht_plan::Tile& t) {
  t.ops = t.rows = t.cols = -1;
  for (size_t k = 0; k < p->ops.size(); ++k)
    if (p->ops[k].N == t.N) t.ops = (int)k;
  for (size_t k = 0; k < p->row_ops.size(); ++k)
    if (p->row_ops[k].N == t.N && p->row_ops[k].th == t.th) t.rows = (int)k;
  for (size_t k = 0; k < p->col_ops.size(); ++k)
    if (p->col_ops[k].N == t.N && p->col_ops[k].tw == t.tw) t.cols = (int)k;
  const bool full = p->variant == NX_FHT_FULL_SPECTRUM;
  if (full ? t.ops >= 0 : (t.rows >= 0 && t.cols >= 0)) return NX_OK;
  const OpTables tab(t.N, p->mag);
  std::vector<float> v, w, e;
  int rc = NX_OK;
  if (full) {
    nx_fht_plan::Ops o{t.N, tab.L, nullptr, nullptr};
    build_full_ops(tab, v, w);
    rc = fht_upload(p, v, &o.ct);
    if (!rc) rc = fht_upload(p, w, &o.acat);
    p->ops.push_back(o);
    t.ops = (int)p->ops.size() - 1;
    return rc;
  }
  if (t.rows < 0) {
    nx_fht_plan::RowOps o{t.N, t.th, round16(t.th), nullptr, nullptr, nullptr};
    build_row_ops(tab, t.th, t.kh, t.y_roi, v, w, e);
    rc = fht_upload(p, v, &o.a);
    if (!rc) rc = fht_upload(p, w, &o.s);
    if (!rc) rc = fht_upload(p, e, &o.e);
    p->row_ops.push_back(o);
    t.rows = (int)p->row_ops.size() - 1;
  }
  if (!rc && t.cols < 0) {
    nx_fht_plan::ColOps o{t.N, t.tw, round16(t.tw), nullptr};
    build_col_ops(tab, t.tw, t.kw, t.x_roi, v);
    rc = fht_upload(p, v, &o.ct);
    p->col_ops.push_back(o);
    t.cols = (int)p->col_ops.size() - 1;
  }
  return rc;
}

void fht_plan_free(nx_fht_plan* p) {
  for (float* b : p->bufs) cudaFree(b);
  delete p;
}

}  // namespace
}  // namespace nx

using namespace nx;

extern "C" {

int nx_fht_plan_create(nx_fht_plan** out, int H, int W, int magnification) {
  return nx_fht_plan_create_ex(out, H, W, magnification, NX_FHT_TILED);
}

int nx_fht_plan_create_ex(nx_fht_plan** out, int H, int W, int magnification, int variant) {
  if (!out) return nx::set_error("plan out-pointer is NULL"), NX_ERR_INVALID_ARG;
  if (variant != NX_FHT_TILED && variant != NX_FHT_FULL_SPECTRUM)
    return nx::set_error("unknown Fourier interpolation variant %d", variant), NX_ERR_INVALID_ARG;
  *out = nullptr;
  if (H < 1 || W < 1) return nx::set_error("image must have H, W >= 1"), NX_ERR_INVALID_ARG;
  if (magnification < 1 || magnification > 64)
    return nx::set_error("magnification must be in [1, 64]"), NX_ERR_INVALID_ARG;
  if ((long long)H * magnification >= (1LL << 30) || (long long)W * magnification >= (1LL << 30))
    return nx::set_error("magnified image too large"), NX_ERR_INVALID_ARG;
  auto* p = new nx_fht_plan();
  p->H = H;
  p->W = W;
  p->mag = magnification;
  p->variant = variant;
  cudaGetDevice(&p->device);
  p->tiled = variant == NX_FHT_TILED && (H > kFhtTile || W > kFhtTile);
  std::vector<int> rs{0}, cs{0};
  if (p->tiled) {
    rs = tile_starts(H);
    cs = tile_starts(W);
  }
  for (size_t ri = 0; ri < rs.size(); ++ri)
    for (size_t ci = 0; ci < cs.size(); ++ci) {
      const int r0 = rs[ri], c0 = cs[ci];
      nx_fht_plan::Tile t{};
      t.r0 = r0;
      t.c0 = c0;
      // the neighbours' reach into this tile (starts ascend, at most two overlap)
      t.y_new = ri ? std::max(0, rs[ri - 1] + kFhtTile - r0) * magnification : 0;
      t.x_new = ci ? std::max(0, cs[ci - 1] + kFhtTile - c0) * magnification : 0;
      t.y_last = ri + 1 < rs.size() ? (rs[ri + 1] - r0) * magnification : INT_MAX;
      t.x_last = ci + 1 < cs.size() ? (cs[ci + 1] - c0) * magnification : INT_MAX;
      t.th = p->tiled ? std::min(r0 + kFhtTile, H) - r0 : H;
      t.tw = p->tiled ? std::min(c0 + kFhtTile, W) - c0 : W;
      const int N = std::max(pow2_ceil(t.th), pow2_ceil(t.tw));
      t.kh = (N + t.th - 1) / t.th;
      t.kh += 1 - t.kh % 2;  // odd number of copies
      t.kw = (N + t.tw - 1) / t.tw;
      t.kw += 1 - t.kw % 2;
      t.y_roi = (t.kh * t.th - N) / 2;
      t.x_roi = (t.kw * t.tw - N) / 2;
      t.N = N;
      int rc = build_tile_ops(p, t);
      if (rc) {
        fht_plan_free(p);
        return rc;
      }
      if (p->tiled) {
        rc = fht_upload(p, hann_inner(t.th * magnification), &t.wr);
        if (!rc) rc = fht_upload(p, hann_inner(t.tw * magnification), &t.wc);
        if (rc) {
          fht_plan_free(p);
          return rc;
        }
      }
      p->tiles.push_back(t);
    }
  size_t square = 1;
  for (const auto& t : p->tiles) {
    const size_t N = t.N, L = N * magnification;
    square = std::max(square, L * L * sizeof(float));
    if (variant == NX_FHT_FULL_SPECTRUM) {
      p->frame_floats = std::max(p->frame_floats, N * N + 2 * N * L + L * L);
    } else {  // tile, U, Z, r, alternating sums
      const size_t nr = p->row_ops[t.rows].n, nc = p->col_ops[t.cols].n;
      p->frame_floats = std::max(p->frame_floats,
                                 nr * nc + std::min(nr, nc) * L + L * L + L + nc);
    }
  }
  p->chunk = (int)std::min<size_t>(kFhtChunkMax, std::max<size_t>(kFhtChunkMin, kFhtChunkBytes / square));
  if (p->tiled) {
    // blending weights: the windows summed in the reference's tile order
    const size_t plane = (size_t)H * magnification * W * magnification;
    cudaError_t e = cudaMalloc(&p->wgt, plane * sizeof(float));
    if (e == cudaSuccess) p->bufs.push_back(p->wgt);
    if (e == cudaSuccess) e = cudaMemset(p->wgt, 0, plane * sizeof(float));
    for (const auto& t : p->tiles) {
      if (e != cudaSuccess) break;
      const long long n = (long long)t.th * magnification * t.tw * magnification;
      fht_weight_kernel<<<blocks_for(n), 256>>>(t.wr, t.wc, t.th * magnification,
                                                t.tw * magnification, p->wgt,
                                                W * magnification, t.r0 * magnification,
                                                t.c0 * magnification);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
      const int rc = cuda_status(e, "FHT plan weights");
      fht_plan_free(p);
      return rc;
    }
  }
  *out = p;
  return NX_OK;
}

int nx_fht_plan_destroy(nx_fht_plan* p) {
  if (p) fht_plan_free(p);
  return NX_OK;
}

size_t nx_fht_workspace_bytes(const nx_fht_plan* p, int T) {
  if (!p || T < 1) return 256;
  const size_t tc = (size_t)std::min(T, p->chunk);
  return 256 + ((tc * p->frame_floats * sizeof(float) + 255) / 256) * 256 +
         2 * tc * 4 * sizeof(int);
}

int nx_fht_interpolate(const nx_fht_plan* p, const float* d_in, int T, float* d_out, void* d_ws,
                       size_t ws_bytes, void* stream) {
  if (!p) return nx::set_error("plan is NULL"), NX_ERR_INVALID_ARG;
  int dev = -1;
  cudaGetDevice(&dev);
  if (dev != p->device) return nx::set_error("plan made on another device"), NX_ERR_INVALID_ARG;
  if (T < 0) return nx::set_error("T must be >= 0"), NX_ERR_INVALID_ARG;
  if (T == 0) return NX_OK;
  if (!d_in || !d_out) return nx::set_error("NULL input/output"), NX_ERR_INVALID_ARG;
  if (!d_ws || ws_bytes < nx_fht_workspace_bytes(p, T)) {
    nx::set_error("workspace too small: need %zu bytes", nx_fht_workspace_bytes(p, T));
    return NX_ERR_WORKSPACE;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const int mag = p->mag;
  const bool full = p->variant == NX_FHT_FULL_SPECTRUM;
  const int outH = p->H * mag, outW = p->W * mag;
  const long long plane = (long long)outH * outW;
  char* base = (char*)d_ws + 256;
  float* work = (float*)base;
  int* const mm0 = (int*)(base + ((std::min(T, p->chunk) * p->frame_floats * sizeof(float) + 255) /
                                  256) * 256);
  int* const mms[2] = {mm0, mm0 + 4 * std::min(T, p->chunk)};
  int set = 0;
  bool clear = true;
  for (int t0 = 0; t0 < T; t0 += p->chunk) {
    const int tc = std::min(p->chunk, T - t0);
    const float* in = d_in + (size_t)t0 * p->H * p->W;
    float* out = d_out + (size_t)t0 * plane;
    for (const auto& t : p->tiles) {
      const int N = t.N, L = N * mag;
      // (min, max) slots of the tile input and of the interpolated square: two sets
      // in turn, each cleared while the other's tile runs (the first by itself)
      int* mm = mms[set];
      if (clear) {
        fht_mm_init_kernel<<<1, 32, 0, s>>>(mm, tc);
        NX_CUDA_TRY(cudaGetLastError());
        clear = full;
      }
      float* const X = work;
      float* Z;
      if (full) {
        const auto& o = p->ops[t.ops];
        float* U = X + (size_t)tc * N * N;
        Z = U + (size_t)tc * 2 * N * L;
        fht_gather_kernel<<<dim3(blocks_for((long long)N * N, 256, 256), (unsigned)tc), 256, 0,
                            s>>>(in, p->H, p->W, t.r0, t.c0, t.th, t.tw, N, t.kh, t.kw, t.y_roi,
                                 t.x_roi, X, mm);
        NX_CUDA_TRY(cudaGetLastError());
        // U = X [C_re^T | C_im^T] stacked (batch (frame, part)), then
        // Z = [A_re | -A_im] [U_re ; U_im]: one image per sweep, whose scores
        // keep their bits
        const GemmBatch b1{2, (long long)N * N, 0, 0, (long long)N * L, (long long)2 * N * L,
                           (long long)N * L};
        NX_CUDA_TRY(gemm(X, o.ct, U, N, L, N, N, L, L, 2 * tc, b1, Rank1{}, s));
        const GemmBatch b2{1, 0, 0, (long long)2 * N * L, 0, (long long)L * L, 0};
        NX_CUDA_TRY(gemm(o.acat, U, Z, L, L, 2 * N, 2 * N, L, L, tc, b2,
                         Rank1{nullptr, 0, nullptr, mm}, s));
      } else {
        const auto& ro = p->row_ops[t.rows];
        const auto& co = p->col_ops[t.cols];
        const int nr = ro.n, nc = co.n;
        float* U = X + (size_t)tc * nr * nc;
        Z = U + (size_t)tc * std::min(nr, nc) * L;
        float* r = Z + (size_t)tc * L * L;
        float* alt = r + (size_t)tc * L;
        fht_tile_kernel<<<dim3(blocks_for((long long)nr * nc, 256, 256), (unsigned)tc), 256, 0,
                          s>>>(in, p->H, p->W, t.r0, t.c0, t.th, t.tw, nr, nc, X, mm);
        NX_CUDA_TRY(cudaGetLastError());
        // r of the rank-1 term
        const bool own = nr <= kAltInline && nc <= kAltInline;
        if (!own) {
          fht_alternate_kernel<<<dim3((unsigned)((nc + 31) / 32), (unsigned)tc), 256, 0, s>>>(
              X, ro.e, nr, nc, alt);
          NX_CUDA_TRY(cudaGetLastError());
        }
        fht_rank1_kernel<<<dim3((unsigned)((L + 31) / 32), (unsigned)tc), 256, 0, s>>>(
            own ? X : nullptr, ro.e, alt, co.ct + (size_t)nc * L, nr, nc, L, r, mms[set ^ 1], tc);
        NX_CUDA_TRY(cudaGetLastError());
        // the product onto the L x L square, the larger, runs over the tile's
        // shorter side: U = X C_re^T (the frames' tiles stacked), Z = A_re U + s r^T,
        // or U = A_re X, Z = U C_re^T + s r^T.  8 frames of 300 x 260 at m = 2 (three
        // interpolations of tiles of 256 x 256, 256 x 36, 76 x 256 and 76 x 36): the
        // products 1.08 ms over mirrored squares of N x N, 0.72 ms so (0.58 ms now).
        const Rank1 u{ro.s, 1, r, mm};
        if (nr <= nc) {
          NX_CUDA_TRY(gemm(X, co.ct, U, tc * nr, L, nc, nc, L, L, 1,
                           GemmBatch{1, 0, 0, 0, 0, 0, 0}, Rank1{}, s));
          const GemmBatch b2{1, 0, 0, (long long)nr * L, 0, (long long)L * L, 0};
          NX_CUDA_TRY(gemm(ro.a, U, Z, L, L, nr, nr, L, L, tc, b2, u, s));
        } else {
          const GemmBatch b1{1, 0, 0, (long long)nr * nc, 0, (long long)L * nc, 0};
          NX_CUDA_TRY(gemm(ro.a, X, U, L, nc, nr, nr, nc, nc, tc, b1, Rank1{}, s));
          const GemmBatch b2{1, (long long)L * nc, 0, 0, 0, (long long)L * L, 0};
          NX_CUDA_TRY(gemm(U, co.ct, Z, L, L, nc, nc, L, L, tc, b2, u, s));
        }
      }
      const int oh = t.th * mag, ow = t.tw * mag;
      fht_finish_kernel<<<dim3((unsigned)((ow + 127) / 128),
                               (unsigned)((oh + kFinishRows - 1) / kFinishRows), (unsigned)tc),
                          128, 0, s>>>(Z, L, mm, oh, ow, (L - oh) / 2, (L - ow) / 2,
                               p->tiled ? t.wr : nullptr, p->tiled ? t.wc : nullptr, p->wgt,
                               t.y_new, t.x_new, t.y_last, t.x_last, out, outH, outW,
                               t.r0 * mag, t.c0 * mag, full);
      NX_CUDA_TRY(cudaGetLastError());
      set ^= 1;
    }
  }
  return NX_OK;
}

}  // extern "C"
