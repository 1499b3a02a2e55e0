// mlp.cu - the learned control variate: a small MLP mapping a site's local
// stacking disregistry, twist, layer and sublattice to its first 256
// Chebyshev moments, trained and evaluated on the tensor cores.
//
// Network: 64 input features (16 used, zero padded) -> 256 -> 256 -> 256
// (GELU) -> 256 moments. BF16 weights and activations, FP32 accumulation
// (tc_gemm.cu), FP32 master weights, biases and Adam state.
//
// One training step (captured once into a CUDA graph, replayed per step):
//   gather a Philox-sampled minibatch X [B][64], T [B][256] (+ X^T)
//   forward: Z_l = A_l W_l^T + b_l  (A_0 = X, A_{l+1} = gelu(Z_l), Y = Z_3)
//   loss:    L = (1/B) sum_r sum_j w_j (Y - T)^2,  dZ_3 = (2/B) w (Y - T)
//   backward: dW_l = dZ_l^T A_l, db_l = colsum(dZ_l),
//             dZ_{l-1} = (dZ_l W_l) * gelu'(Z_{l-1})
//   Adam update of all parameters, refresh of the BF16 copies
//   (W_l [out][in] for the forward products, W_l^T [in][out] for dA).
// The reference has no learned component; the network only serves as a
// control variate for the stochastic trace (see the estimator in bench.py).
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "csr.cuh"
#include "pair.cuh"
#include "tc_gemm.cuh"

using namespace leo2d;

namespace {

constexpr int kIn = 64, kHid = 256, kOut = 256, kLayers = 4, kFeat = 16;
constexpr int kInDim[kLayers] = {kIn, kHid, kHid, kHid};
constexpr int64_t kChunk = 1 << 20;  // sites per inference pass
constexpr int kDwSplits = 32;        // K-range splits of the weight-gradient products

__device__ __forceinline__ uint32_t mix32(uint64_t a, uint64_t b) {
  // splitmix64 of (a, b): minibatch indices
  uint64_t z = a * 0x9E3779B97F4A7C15ull + b + 0x632BE59BD9B4E019ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return (uint32_t)((z ^ (z >> 31)) >> 32);
}

// cos and sin of p 2^-64 turns. The quarter turn comes off exactly in integers;
// the rest (at most 1/8 turn) goes through the Taylor series of sin and cos, their
// first terms in pairs and the tail (below 1/60) in FP32: errors up to 5e-9, so
// the rounded FP32 value is that of the FP64 function but for 3 in 1000 near ties
// (then its neighbour).
__device__ __forceinline__ void phase_cos_sin(uint64_t p, FPair& c, FPair& s) {
  const uint32_t q = (uint32_t)((p + (1ull << 61)) >> 62);
  const int64_t r = (int64_t)(p - ((uint64_t)q << 62));
  const int32_t a = (int32_t)(r >> 32);
  const float h = __int2float_rn(a);
  const float l = __fmaf_rn(__uint2float_rn((uint32_t)r), 0x1p-32f, __int2float_rn(a - (int32_t)h));
  // x = 2 pi (h + l) 2^-32
  constexpr double kTurn = 6.283185307179586476925 / 4294967296.0;
  constexpr float kTurnH = (float)kTurn, kTurnL = (float)(kTurn - (double)kTurnH);
  const FPair u = fpair_mul({h, l}, {kTurnH, kTurnL});
  const FPair x = fpair_fast_sum(u.h, u.l);
  const FPair z = fpair_mul(x, x);
  constexpr double kSixth = -1.0 / 6.0;
  constexpr float kSixthH = (float)kSixth, kSixthL = (float)(kSixth - (double)kSixthH);
  const FPair t = fpair_mul(fpair_mul(x, z), {kSixthH, kSixthL});
  float ts = __fmaf_rn(z.h, -1.0f / 39916800.0f, 1.0f / 362880.0f);
  ts = __fmaf_rn(z.h, ts, -1.0f / 5040.0f);
  ts = __fmaf_rn(z.h, ts, 1.0f / 120.0f);
  ts = __fmul_rn(ts, __fmul_rn(x.h, __fmul_rn(z.h, z.h)));
  const FPair s0 = fpair_fast_sum(x.h, t.h);
  const FPair sn = fpair_fast_sum(s0.h, __fadd_rn(s0.l, __fadd_rn(__fadd_rn(x.l, t.l), ts)));
  float tc = __fmaf_rn(z.h, -1.0f / 3628800.0f, 1.0f / 40320.0f);
  tc = __fmaf_rn(z.h, tc, -1.0f / 720.0f);
  tc = __fmaf_rn(z.h, tc, 1.0f / 24.0f);
  tc = __fmul_rn(tc, __fmul_rn(z.h, z.h));
  const FPair c0 = fpair_fast_sum(1.0f, -0.5f * z.h);
  const FPair cs = fpair_fast_sum(c0.h, __fadd_rn(c0.l, __fmaf_rn(-0.5f, z.l, tc)));
  c = (q & 1) ? sn : cs;
  s = (q & 1) ? cs : sn;
  if (q == 1 || q == 2) c = fpair_neg(c);
  if (q >= 2) s = fpair_neg(s);
}

// BF16 features [n][16] of the sites first .. first + n - 1: site_features() with
// the disregistry as fixed-point phases (csr_site_phases) and FP32 pairs. This
// GPU's FP64 pipe gives a warp instruction per 16 cycles and SM: the disregistry
// in FP64 (60 instructions a site, 134 us per 1M sites) and twelve FP64 sines and
// cosines with rows padded to 64 columns in memory (680 us) took twice the time
// of the network; like this the pass is bound by its 48 bytes a site.
__global__ void __launch_bounds__(256) k_site_rows(int64_t n, int64_t first, const SitePhase ph0, const SitePhase ph1,
                                                   const int32_t* __restrict__ grid4, float twist_deg,
                                                   __nv_bfloat16* __restrict__ X) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const int4 g = __ldg(reinterpret_cast<const int4*>(grid4) + first + r);  // i, j, orbital, sheet
    const SitePhase& ph = g.w == 0 ? ph0 : ph1;
    FPair c[2], s[2];
#pragma unroll
    for (int d = 0; d < 2; ++d)
      phase_cos_sin(ph.c[d] + ph.mi[d] * (uint64_t)(int64_t)g.x + ph.mj[d] * (uint64_t)(int64_t)g.y, c[d], s[d]);
    const FPair cc = fpair_mul(c[0], c[1]), ss = fpair_mul(s[0], s[1]);
    const FPair sc = fpair_mul(s[0], c[1]), cs = fpair_mul(c[0], s[1]);
    float f[kFeat];
    f[0] = c[0].h;
    f[1] = s[0].h;
    f[2] = c[1].h;
    f[3] = s[1].h;
    f[4] = fpair_sum(cc, fpair_neg(ss));
    f[5] = fpair_sum(sc, cs);
    f[6] = fpair_sum(cc, ss);
    f[7] = fpair_sum(sc, fpair_neg(cs));
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const FPair p = fpair_mul(c[d], s[d]);
      f[8 + 2 * d] = fpair_sum(fpair_mul(c[d], c[d]), fpair_neg(fpair_mul(s[d], s[d])));
      f[9 + 2 * d] = fpair_sum(p, p);
    }
    f[12] = twist_deg / 3.0f;
    f[13] = (float)g.w;
    f[14] = (float)g.z;
    f[15] = 1.0f;
    uint32_t w[kFeat / 2];
#pragma unroll
    for (int k = 0; k < kFeat / 2; ++k) {
      const __nv_bfloat162 b = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
      w[k] = *reinterpret_cast<const uint32_t*>(&b);
    }
    uint4* dst = reinterpret_cast<uint4*>(X + r * kFeat);
    dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
    dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// Site features from the disregistry (Hstruct::getShiftConfigs), twist,
// layer and sublattice; 16 used columns of 64.
__device__ __forceinline__ void site_features(double d0, double d1, float twist_deg, int layer, int sub,
                                              float* f) {
  const double tp = 6.283185307179586;
  f[0] = (float)cos(tp * d0);
  f[1] = (float)sin(tp * d0);
  f[2] = (float)cos(tp * d1);
  f[3] = (float)sin(tp * d1);
  f[4] = (float)cos(tp * (d0 + d1));
  f[5] = (float)sin(tp * (d0 + d1));
  f[6] = (float)cos(tp * (d0 - d1));
  f[7] = (float)sin(tp * (d0 - d1));
  f[8] = (float)cos(2 * tp * d0);
  f[9] = (float)sin(2 * tp * d0);
  f[10] = (float)cos(2 * tp * d1);
  f[11] = (float)sin(2 * tp * d1);
  f[12] = twist_deg / 3.0f;
  f[13] = (float)layer;
  f[14] = (float)sub;
  f[15] = 1.0f;
}

__global__ void k_features(int64_t n, const double* __restrict__ cfg,
                           const int32_t* __restrict__ grid4, float twist_deg, float* __restrict__ Xf) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    float f[kFeat];
    site_features(cfg[2 * r], cfg[2 * r + 1], twist_deg, grid4[4 * r + 3], grid4[4 * r + 2], f);
    for (int c = 0; c < kFeat; ++c) Xf[r * kFeat + c] = f[c];
  }
}

// Features of selected orbitals rows[r] -> BF16 [n][64].
__global__ void k_features_at(int64_t n, const int64_t* __restrict__ rows, const double* __restrict__ cfg,
                              const int32_t* __restrict__ grid4, float twist_deg, __nv_bfloat16* __restrict__ X) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = rows[r];
    float f[kFeat];
    site_features(cfg[2 * k], cfg[2 * k + 1], twist_deg, grid4[4 * k + 3], grid4[4 * k + 2], f);
    for (int c = 0; c < kIn; ++c) X[r * kIn + c] = __float2bfloat16_rn(c < kFeat ? f[c] : 0.0f);
  }
}

// Host feature rows [n][F] (F <= 64, FP32) -> BF16 [n][64] and its transpose [64][ldt].
__global__ void k_pack_x(int64_t n, int F, const float* __restrict__ src, __nv_bfloat16* __restrict__ X,
                         __nv_bfloat16* __restrict__ Xt, int64_t ldt) {
  const int64_t total = n * kIn;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e / kIn;
    const int c = (int)(e % kIn);
    const __nv_bfloat16 v = __float2bfloat16_rn(c < F ? src[r * F + c] : 0.0f);
    X[e] = v;
    if (Xt) Xt[(int64_t)c * ldt + r] = v;
  }
}

// Minibatch: rows sampled (with replacement) by a hash of (seed, step, row).
__global__ void k_gather(int64_t n_train, int B, const __nv_bfloat16* __restrict__ Xall,
                         const float* __restrict__ Tall, const int64_t* __restrict__ step, uint64_t seed,
                         __nv_bfloat16* __restrict__ Xb, __nv_bfloat16* __restrict__ Xbt, float* __restrict__ Tb) {
  const uint64_t s = (uint64_t)*step;
  const int64_t total = (int64_t)B * (kIn + kOut);
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(e / (kIn + kOut));
    const int c = (int)(e % (kIn + kOut));
    const int64_t src = (int64_t)(((uint64_t)mix32(seed ^ (s << 20), (uint64_t)r) * (uint64_t)n_train) >> 32);
    if (c < kIn) {
      const __nv_bfloat16 v = Xall[src * kIn + c];
      Xb[(int64_t)r * kIn + c] = v;
      Xbt[(int64_t)c * B + r] = v;
    } else {
      Tb[(int64_t)r * kOut + (c - kIn)] = Tall[src * kOut + (c - kIn)];
    }
  }
}

// dY = (2/n) w (Y - T) -> BF16 [n][256], its transpose, FP32; per-block loss sums.
// A block takes 32 rows; a thread 4 columns of 8 rows. The transpose goes through
// shared memory: 2-byte stores a row length apart and six FP64 instructions an
// element for the loss took 28 us at 8192 rows (10 now). w d^2 is a product in FP32
// pairs (2^-45 relative), a thread's 16 terms are summed in pairs, then FP64. A thread
// whose sum left the range where pairs hold that (an overflow, or low parts below
// FP32's smallest) takes its terms again in FP64.
constexpr int kLossRows = 32;
__global__ void __launch_bounds__(512) k_loss(int n, const float* __restrict__ Y, const float* __restrict__ T,
                                              const float* __restrict__ w, __nv_bfloat16* __restrict__ dZ,
                                              __nv_bfloat16* __restrict__ dZt, int64_t ldt, float* __restrict__ dZ32,
                                              double* __restrict__ part) {
  __shared__ __nv_bfloat16 tile[kOut][kLossRows + 2];
  __shared__ double red[16];
  const int j = 4 * (threadIdx.x & 63), g8 = threadIdx.x >> 6;
  const int r0 = blockIdx.x * kLossRows;
  const float scale = 2.0f / (float)n;
  const float4 w4 = *reinterpret_cast<const float4*>(w + j);
  const float wj[4] = {w4.x, w4.y, w4.z, w4.w};
  PairSum sum;
#pragma unroll
  for (int i = 0; i < kLossRows / 8; ++i) {
    const int rr = g8 + 8 * i;
    if (r0 + rr >= n) break;
    const size_t e = (size_t)(r0 + rr) * kOut + j;
    const float4 y4 = *reinterpret_cast<const float4*>(Y + e), t4 = *reinterpret_cast<const float4*>(T + e);
    const float d[4] = {y4.x - t4.x, y4.y - t4.y, y4.z - t4.z, y4.w - t4.w};
    float gr[4];
    __nv_bfloat16 b[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      gr[k] = scale * wj[k] * d[k];
      b[k] = __float2bfloat16_rn(gr[k]);
      tile[j + k][rr] = b[k];
      sum.add(fpair_mul({wj[k], 0.f}, fpair_mul({d[k], 0.f}, {d[k], 0.f})));
    }
    *reinterpret_cast<float4*>(dZ32 + e) = make_float4(gr[0], gr[1], gr[2], gr[3]);
    *reinterpret_cast<uint2*>(dZ + e) = *reinterpret_cast<const uint2*>(b);
  }
  double acc = sum.value();
  const float wmax = fmaxf(fmaxf(fabsf(wj[0]), fabsf(wj[1])), fmaxf(fabsf(wj[2]), fabsf(wj[3])));
  if (!(isfinite(sum.h) && fabsf(sum.h) >= 1e-30f * fmaxf(1.0f, wmax))) {
    acc = 0.0;
    for (int i = 0; i < kLossRows / 8 && r0 + g8 + 8 * i < n; ++i)
      for (int k = 0; k < 4; ++k) {
        const size_t e = (size_t)(r0 + g8 + 8 * i) * kOut + j + k;
        const float d = Y[e] - T[e];
        acc += (double)w[j + k] * (double)d * (double)d;
      }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  for (int e = threadIdx.x; e < kOut * kLossRows; e += blockDim.x) {
    const int c = e / kLossRows, r = e % kLossRows;
    if (r0 + r < n) dZt[(size_t)c * ldt + r0 + r] = tile[c][r];
  }
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int k = 0; k < 16; ++k) s += red[k];
    part[blockIdx.x] = s;
  }
}

// The mean of the block sums, 256 strided chains and a tree (one thread's chain of
// 1024 loads took 51 us).
__global__ void __launch_bounds__(256) k_loss_final(const double* __restrict__ part, int nb, int n,
                                                    const int64_t* __restrict__ step, double* __restrict__ hist,
                                                    int64_t hist_cap, double* __restrict__ last) {
  __shared__ double red[256];
  double s = 0.0;
  for (int b = threadIdx.x; b < nb; b += 256) s += part[b];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x != 0) return;
  s = red[0] / (double)n;
  *last = s;
  const int64_t t = step ? *step : 0;
  if (hist && t < hist_cap) hist[t] = s;
}

// Column sums of x [n][256] (FP32) over blocks of rows, in a fixed order.
__global__ void __launch_bounds__(256) k_colsum_part(int n, int rows_per_block, const float* __restrict__ x,
                                                     float* __restrict__ part) {
  const int j = threadIdx.x;
  const int r0 = blockIdx.x * rows_per_block, r1 = min(n, r0 + rows_per_block);
  float s = 0.0f;
  for (int r = r0; r < r1; ++r) s += x[(int64_t)r * kOut + j];
  part[(int64_t)blockIdx.x * kOut + j] = s;
}

// The last additions of every layer in one launch: dW_l = sum of its K-range splits,
// db_l = sum of its column-sum blocks (fixed orders; as two launches a layer these
// took 30 us of a gradient at 8192 rows, together 13).
struct GradParts {
  const float* dw[kLayers];  // [splits][256 in]
  const float* cs[kLayers];  // [blocks][256]
  int64_t w_off[kLayers], b_off[kLayers];
  int splits, blocks;
};
__global__ void __launch_bounds__(256) k_grad_final(const GradParts a, float* __restrict__ g) {
  const int l = blockIdx.y;
  const int64_t nw = (int64_t)kHid * (l == 0 ? kIn : kHid);
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (blockIdx.x == gridDim.x - 1) {
    float s = 0.0f;
#pragma unroll 8
    for (int b = 0; b < a.blocks; ++b) s += a.cs[l][(int64_t)b * kOut + threadIdx.x];
    g[a.b_off[l] + threadIdx.x] = s;
  } else if (e < nw) {
    float s = 0.0f;
#pragma unroll 8
    for (int k = 0; k < a.splits; ++k) s += a.dw[l][(size_t)k * nw + e];
    g[a.w_off[l] + e] = s;
  }
}

__global__ void k_adam(int64_t np, float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, const int64_t* __restrict__ step, float lr, float b1, float b2,
                       float eps) {
  const double t = (double)(*step + 1);
  const float c1 = (float)(1.0 - pow((double)b1, t)), c2 = (float)(1.0 - pow((double)b2, t));
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

__global__ void k_step_inc(int64_t* step) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *step += 1;
}

// W [out][in] FP32 -> BF16 [out][in] and (optionally) BF16 [in][out].
__global__ void k_refresh(int out, int in, const float* __restrict__ W, __nv_bfloat16* __restrict__ wt,
                          __nv_bfloat16* __restrict__ wn) {
  const int64_t total = (int64_t)out * in;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int o = (int)(e / in), i = (int)(e % in);
    const __nv_bfloat16 b = __float2bfloat16_rn(W[e]);
    wt[e] = b;
    if (wn) wn[(int64_t)i * out + o] = b;
  }
}

__global__ void k_sum_partials(const double* __restrict__ part, int nb, double* __restrict__ out, int accumulate) {
  const int j = threadIdx.x;
  double s = 0.0;
  for (int b = 0; b < nb; ++b) s += part[(int64_t)b * kOut + j];
  out[j] = accumulate ? out[j] + s : s;
}

uint64_t splitmix(uint64_t& x) {
  uint64_t z = (x += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

}  // namespace

struct leo2d_mlp {
  leo2d_ctx* ctx = nullptr;
  int device = 0;  // (the network may be destroyed after its context)
  int64_t np = 0;
  int64_t w_off[kLayers], b_off[kLayers];
  DevBuf<float> p, g, m, v, lw;
  DevBuf<__nv_bfloat16> wt[kLayers], wn[kLayers];
  DevBuf<int64_t> step;
  // training workspace (batch B)
  int B = 0;
  DevBuf<__nv_bfloat16> Xb, Xbt, A[kLayers], At[kLayers], dZ[2], dZt[2];
  DevBuf<float> Tb, Z[kLayers], Y, dZ32[2], cs_part[kLayers], dw_split[kLayers];
  DevBuf<double> loss_part, loss_last, loss_hist;
  int64_t hist_cap = 0;
  CUtensorMap tWf[kLayers];  // boxes of 256 rows, for the fused forward
  CUtensorMap tX, tA[kLayers], tWt[kLayers], tWn[kLayers], tXt, tAt[kLayers], tdZ[2], tdZt[2];
  // training set
  int64_t n_train = 0;
  DevBuf<__nv_bfloat16> Xall;
  DevBuf<float> Tall;
  cudaGraphExec_t graph = nullptr;
  uint64_t graph_seed = 0;
  float graph_lr = 0.f;
  ~leo2d_mlp() {
    if (graph) cudaGraphExecDestroy(graph);
  }
};

namespace {

void refresh_bf16(leo2d_mlp* M) {
  leo2d_ctx* ctx = M->ctx;
  for (int l = 0; l < kLayers; ++l) {
    const int in = kInDim[l];
    launch(ctx, "mlp_refresh", [&] {
      k_refresh<<<grid_for((int64_t)kHid * in, 256, ctx->sm_count * 8), 256, 0, ctx->stream>>>(
          kHid, in, M->p.p + M->w_off[l], M->wt[l].p, l > 0 ? M->wn[l].p : nullptr);
    });
  }
}

// K-range splits of the weight-gradient products of n rows
int dw_splits(int n) { return std::max(1, std::min(kDwSplits, n / 256)); }

void ensure_batch(leo2d_mlp* M, int B) {
  if (M->B == B) return;
  LEO_REQUIRE(B >= 64 && B % 64 == 0 && B <= (1 << 20), "batch must be a multiple of 64 in [64, 2^20]");
  if (M->graph) {
    cudaGraphExecDestroy(M->graph);
    M->graph = nullptr;
  }
  M->B = B;
  M->Xb.alloc((size_t)B * kIn);
  M->Xbt.alloc((size_t)kIn * B);
  M->Tb.alloc((size_t)B * kOut);
  M->Y.alloc((size_t)B * kOut);
  for (int l = 0; l < kLayers; ++l) {
    if (l > 0) {
      M->A[l].alloc((size_t)B * kHid);
      M->At[l].alloc((size_t)kHid * B);
    }
    if (l < kLayers - 1) M->Z[l].alloc((size_t)B * kHid);
  }
  for (int i = 0; i < 2; ++i) {
    M->dZ[i].alloc((size_t)B * kHid);
    M->dZt[i].alloc((size_t)kHid * B);
    M->dZ32[i].alloc((size_t)B * kHid);
  }
  for (int l = 0; l < kLayers; ++l) {
    M->dw_split[l].alloc((size_t)dw_splits(B) * kHid * kInDim[l]);
    M->cs_part[l].alloc((size_t)((B + 63) / 64) * kOut);
  }
  M->loss_part.alloc((size_t)(B + kLossRows - 1) / kLossRows);
  M->loss_last.alloc(1);
  make_tmap_bf16(&M->tX, M->Xb.p, B, kIn, kGemmBM);
  make_tmap_bf16(&M->tXt, M->Xbt.p, kIn, B, kGemmBoxB);
  for (int l = 1; l < kLayers; ++l) {
    make_tmap_bf16(&M->tA[l], M->A[l].p, B, kHid, kGemmBM);
    make_tmap_bf16(&M->tAt[l], M->At[l].p, kHid, B, kGemmBoxB);
  }
  for (int i = 0; i < 2; ++i) {
    make_tmap_bf16(&M->tdZ[i], M->dZ[i].p, B, kHid, kGemmBM);
    make_tmap_bf16(&M->tdZt[i], M->dZt[i].p, kHid, B, kGemmBM);
  }
}

// Forward over the first n rows of Xb (n <= B); Y [n][256] FP32.
void forward_train(leo2d_mlp* M, int n) {
  leo2d_ctx* ctx = M->ctx;
  for (int l = 0; l < kLayers; ++l) {
    GemmArgs g{};
    g.M = n;
    g.N = kHid;
    g.K = kInDim[l];
    g.bias = M->p.p + M->b_off[l];
    g.status = ctx->status.p;
    const CUtensorMap& ta = l == 0 ? M->tX : M->tA[l];
    if (l < kLayers - 1) {
      g.zout = M->Z[l].p;
      g.out_bf16 = M->A[l + 1].p;
      g.out_bf16_t = M->At[l + 1].p;
      g.ld_t = M->B;
      tc_gemm(ctx, kEpiBiasGelu, ta, M->tWt[l], g);
    } else {
      g.out_f32 = M->Y.p;
      tc_gemm(ctx, kEpiBias, ta, M->tWt[l], g);
    }
  }
}

// Loss on rows [0, n) against Tb, then gradients of every parameter into g.
void backward_train(leo2d_mlp* M, int n) {
  leo2d_ctx* ctx = M->ctx;
  const int B = M->B;
  const int lb = (n + kLossRows - 1) / kLossRows;
  launch(ctx, "mlp_loss", [&] {
    k_loss<<<lb, 512, 0, ctx->stream>>>(n, M->Y.p, M->Tb.p, M->lw.p, M->dZ[1].p, M->dZt[1].p, B, M->dZ32[1].p,
                                        M->loss_part.p);
  });
  launch(ctx, "mlp_loss", [&] {
    k_loss_final<<<1, 256, 0, ctx->stream>>>(M->loss_part.p, lb, n, M->step.p, M->loss_hist.p, M->hist_cap,
                                             M->loss_last.p);
  });
  const int rpb = 64;
  GradParts gp{};
  gp.splits = dw_splits(n);
  gp.blocks = (n + rpb - 1) / rpb;
  int cur = 1;  // dZ of layer l lives in buffer `cur`
  for (int l = kLayers - 1; l >= 0; --l) {
    gp.dw[l] = M->dw_split[l].p;
    gp.cs[l] = M->cs_part[l].p;
    gp.w_off[l] = M->w_off[l];
    gp.b_off[l] = M->b_off[l];
    // bias gradient
    launch(ctx, "mlp_colsum", [&] {
      k_colsum_part<<<gp.blocks, 256, 0, ctx->stream>>>(n, rpb, M->dZ32[cur].p, M->cs_part[l].p);
    });
    // weight gradient dW_l [out][in] = dZ_l^T A_l
    {
      GemmArgs g{};
      g.M = kHid;
      g.N = kInDim[l];
      g.K = n;
      g.out_f32 = M->dw_split[l].p;  // a single split writes its product here
      g.status = ctx->status.p;
      // K = n rows: split over up to 32 work items per output tile
      g.k_splits = gp.splits;
      g.split_buf = M->dw_split[l].p;
      tc_gemm(ctx, kEpiF32, M->tdZt[cur], l == 0 ? M->tXt : M->tAt[l], g);
    }
    if (l == 0) break;
    // dZ_{l-1} = (dZ_l W_l) * gelu'(Z_{l-1})
    {
      const int nxt = cur ^ 1;
      GemmArgs g{};
      g.M = n;
      g.N = kHid;
      g.K = kHid;
      g.zin = M->Z[l - 1].p;
      g.out_f32 = M->dZ32[nxt].p;
      g.out_bf16 = M->dZ[nxt].p;
      g.out_bf16_t = M->dZt[nxt].p;
      g.ld_t = B;
      g.status = ctx->status.p;
      tc_gemm(ctx, kEpiGeluBwd, M->tdZ[cur], M->tWn[l], g);
      cur = nxt;
    }
  }
  launch(ctx, "mlp_grad_final", [&] {
    k_grad_final<<<dim3(kHid * kHid / 256 + 1, kLayers), 256, 0, ctx->stream>>>(gp, M->g.p);
  });
}

void adam_update(leo2d_mlp* M, float lr) {
  leo2d_ctx* ctx = M->ctx;
  launch(ctx, "mlp_adam", [&] {
    k_adam<<<grid_for(M->np, 256, ctx->sm_count * 4), 256, 0, ctx->stream>>>(M->np, M->p.p, M->g.p, M->m.p, M->v.p,
                                                                             M->step.p, lr, 0.9f, 0.999f, 1e-8f);
  });
  refresh_bf16(M);
  launch(ctx, "mlp_step", [&] { k_step_inc<<<1, 32, 0, ctx->stream>>>(M->step.p); });
}

void train_step_enqueue(leo2d_mlp* M, uint64_t seed, float lr) {
  leo2d_ctx* ctx = M->ctx;
  const int B = M->B;
  launch(ctx, "mlp_gather", [&] {
    k_gather<<<grid_for((int64_t)B * (kIn + kOut), 256, ctx->sm_count * 8), 256, 0, ctx->stream>>>(
        M->n_train, B, M->Xall.p, M->Tall.p, M->step.p, seed, M->Xb.p, M->Xbt.p, M->Tb.p);
  });
  forward_train(M, B);
  backward_train(M, B);
  adam_update(M, lr);
}

void upload_x(leo2d_mlp* M, const float* x, int64_t n, int F) {
  leo2d_ctx* ctx = M->ctx;
  float* src = ctx_scratch<float>(ctx, (size_t)n * F);  // in stream order, free again after the call's next sync
  h2d(ctx, src, x, (size_t)n * F);
  launch(ctx, "mlp_pack", [&] {
    k_pack_x<<<grid_for(n * kIn, 256, ctx->sm_count * 8), 256, 0, ctx->stream>>>(n, F, src, M->Xb.p, M->Xbt.p,
                                                                                 M->B);
  });
}

// Forward of `n` rows whose BF16 features sit in X (row-major [n][ldx], ldx = 64
// or 16: the TMA boxes are 64 columns wide either way and fill the columns beyond
// the tensor with zeros): either Y [n][256] FP32, or the column sums (FP64) with
// `part` as work space (mlp_fused_part, or a grid of tc_gemm blocks x 256). Only enqueues the fused form. By default one fused launch keeps
// every activation on chip (mlp_fused.cu); option mlp_fused = 0 runs one GEMM
// per layer over chunks of kChunk rows, with the activations in HBM.
void infer_rows(leo2d_mlp* M, const __nv_bfloat16* X, int ldx, int64_t n, float* Y, double* sums_dev, double* part,
                bool accumulate) {
  leo2d_ctx* ctx = M->ctx;
  if (ctx->mlp_fused) {
    CUtensorMap tx;
    make_tmap_bf16(&tx, X, n, ldx, kGemmBM);
    const float* bias[kLayers];
    for (int l = 0; l < kLayers; ++l) bias[l] = M->p.p + M->b_off[l];
    mlp_forward_fused(ctx, tx, M->tWf, bias, n, Y, sums_dev, part, accumulate);
    return;
  }
  const int64_t chunk = std::min<int64_t>(kChunk, n);
  DevBuf<__nv_bfloat16> h0((size_t)chunk * kHid), h1((size_t)chunk * kHid);
  bool first = !accumulate;
  for (int64_t r0 = 0; r0 < n; r0 += chunk) {
    const int rows = (int)std::min<int64_t>(chunk, n - r0);
    CUtensorMap tx, th0, th1;
    make_tmap_bf16(&tx, X + r0 * ldx, rows, ldx, kGemmBM);
    make_tmap_bf16(&th0, h0.p, rows, kHid, kGemmBM);
    make_tmap_bf16(&th1, h1.p, rows, kHid, kGemmBM);
    const CUtensorMap* in_map[kLayers] = {&tx, &th0, &th1, &th0};
    __nv_bfloat16* out_buf[kLayers - 1] = {h0.p, h1.p, h0.p};
    for (int l = 0; l < kLayers; ++l) {
      GemmArgs g{};
      g.M = rows;
      g.N = kHid;
      g.K = kInDim[l];
      g.bias = M->p.p + M->b_off[l];
      g.status = ctx->status.p;
      if (l < kLayers - 1) {
        g.out_bf16 = out_buf[l];
        tc_gemm(ctx, kEpiBiasGelu, *in_map[l], M->tWt[l], g);
      } else if (Y) {
        g.out_f32 = Y + r0 * kOut;
        tc_gemm(ctx, kEpiBias, *in_map[l], M->tWt[l], g);
      } else {
        g.colsum = part;
        const int gr = tc_gemm_grid(ctx, rows, kOut);
        tc_gemm(ctx, kEpiBias, *in_map[l], M->tWt[l], g);
        launch(ctx, "mlp_sum", [&] {
          k_sum_partials<<<1, kOut, 0, ctx->stream>>>(part, gr, sums_dev, first ? 0 : 1);
        });
      }
    }
    first = false;
    ctx_sync(ctx);  // the chunk's tensor maps and buffers are reused by the next chunk
  }
}

}  // namespace

// ---------------------------------------------------------------- C ABI

extern "C" {

int64_t leo2d_mlp_param_count(void) {
  return (int64_t)kHid * kIn + kHid + (int64_t)(kLayers - 1) * ((int64_t)kHid * kHid + kHid);
}

leo2d_status leo2d_mlp_create(leo2d_ctx* ctx, uint64_t seed, leo2d_mlp** out) {
  if (!ctx || !out) return LEO2D_ERR_BAD_ARG;
  *out = nullptr;
  return guard(ctx, [&] {
    LEO_CUDA(cudaSetDevice(ctx->device));
    auto M = std::make_unique<leo2d_mlp>();
    M->ctx = ctx;
    M->device = ctx->device;
    int64_t off = 0;
    for (int l = 0; l < kLayers; ++l) {
      M->w_off[l] = off;
      off += (int64_t)kHid * kInDim[l];
      M->b_off[l] = off;
      off += kHid;
    }
    M->np = off;
    // He-uniform weights on the used inputs (layer 0: the 16 feature columns),
    // a narrower output layer, zero biases; splitmix64 stream from `seed`
    std::vector<float> h((size_t)off, 0.0f);
    uint64_t st = seed;
    for (int l = 0; l < kLayers; ++l) {
      const int in_used = l == 0 ? kFeat : kInDim[l];
      const double a = l == kLayers - 1 ? std::sqrt(1.0 / in_used) : std::sqrt(6.0 / in_used);
      for (int o = 0; o < kHid; ++o)
        for (int i = 0; i < kInDim[l]; ++i) {
          const double u = (double)(splitmix(st) >> 11) * (1.0 / 9007199254740992.0);
          h[M->w_off[l] + (size_t)o * kInDim[l] + i] = i < in_used ? (float)((2.0 * u - 1.0) * a) : 0.0f;
        }
    }
    M->p.alloc(off);
    M->g.alloc(off);
    M->m.alloc(off);
    M->v.alloc(off);
    h2d(ctx, M->p.p, h.data(), (size_t)off);
    LEO_CUDA(cudaMemsetAsync(M->m.p, 0, sizeof(float) * off, ctx->stream));
    LEO_CUDA(cudaMemsetAsync(M->v.p, 0, sizeof(float) * off, ctx->stream));
    LEO_CUDA(cudaMemsetAsync(M->g.p, 0, sizeof(float) * off, ctx->stream));
    std::vector<float> ones(kOut, 1.0f);
    M->lw.alloc(kOut);
    h2d(ctx, M->lw.p, ones.data(), kOut);
    M->step.alloc(1);
    LEO_CUDA(cudaMemsetAsync(M->step.p, 0, sizeof(int64_t), ctx->stream));
    for (int l = 0; l < kLayers; ++l) {
      M->wt[l].alloc((size_t)kHid * kInDim[l]);
      make_tmap_bf16(&M->tWf[l], M->wt[l].p, kHid, kInDim[l], 256);
      make_tmap_bf16(&M->tWt[l], M->wt[l].p, kHid, kInDim[l], kGemmBoxB);
      if (l > 0) {
        M->wn[l].alloc((size_t)kInDim[l] * kHid);
        make_tmap_bf16(&M->tWn[l], M->wn[l].p, kInDim[l], kHid, kGemmBoxB);
      }
    }
    refresh_bf16(M.get());
    tc_gemm_prepare(ctx);
    ctx_sync(ctx);
    *out = M.release();
  });
}

leo2d_status leo2d_mlp_destroy(leo2d_mlp* M) {
  if (!M) return LEO2D_OK;
  cudaSetDevice(M->device);
  delete M;
  return LEO2D_OK;
}

leo2d_status leo2d_mlp_get_params(leo2d_mlp* M, float* out) {
  if (!M || !out) return LEO2D_ERR_BAD_ARG;
  return guard(M->ctx, [&] {
    d2h(M->ctx, out, M->p.p, (size_t)M->np);
    ctx_sync(M->ctx);
  });
}

leo2d_status leo2d_mlp_set_params(leo2d_mlp* M, const float* in) {
  if (!M || !in) return LEO2D_ERR_BAD_ARG;
  return guard(M->ctx, [&] {
    for (int64_t i = 0; i < M->np; ++i) LEO_REQUIRE(std::isfinite(in[i]), "parameters must be finite");
    h2d(M->ctx, M->p.p, in, (size_t)M->np);
    refresh_bf16(M);
    ctx_sync(M->ctx);
  });
}

leo2d_status leo2d_mlp_set_loss_weights(leo2d_mlp* M, const float* w) {
  if (!M || !w) return LEO2D_ERR_BAD_ARG;
  return guard(M->ctx, [&] {
    h2d(M->ctx, M->lw.p, w, kOut);
    ctx_sync(M->ctx);
  });
}

leo2d_status leo2d_mlp_grad(leo2d_mlp* M, const float* x, int32_t F, const float* t, int64_t n, double* loss,
                            float* grad) {
  if (!M || !x || !t || !loss || !grad) return LEO2D_ERR_BAD_ARG;
  leo2d_ctx* ctx = M->ctx;
  return guard(ctx, [&] {
    LEO_REQUIRE(F >= 1 && F <= kIn, "feature count must be 1..64");
    LEO_REQUIRE(n >= 64 && n % 64 == 0 && n <= (1 << 16), "n must be a multiple of 64 in [64, 65536]");
    LEO_CUDA(cudaSetDevice(ctx->device));
    ensure_batch(M, (int)n);
    upload_x(M, x, n, F);
    h2d(ctx, M->Tb.p, t, (size_t)n * kOut);
    if (!M->loss_hist.p) M->loss_hist.alloc(1);
    forward_train(M, (int)n);
    backward_train(M, (int)n);
    d2h(ctx, loss, M->loss_last.p, 1);
    d2h(ctx, grad, M->g.p, (size_t)M->np);
    ctx_check_status(ctx, "MLP gradient");
  });
}

leo2d_status leo2d_mlp_train(leo2d_mlp* M, const float* x, int32_t F, const float* t, int64_t n, int32_t steps,
                             int32_t batch, float lr, uint64_t seed, double* loss_hist) {
  if (!M || !x || !t) return LEO2D_ERR_BAD_ARG;
  leo2d_ctx* ctx = M->ctx;
  return guard(ctx, [&] {
    LEO_REQUIRE(F >= 1 && F <= kIn, "feature count must be 1..64");
    LEO_REQUIRE(n >= 1, "empty training set");
    LEO_REQUIRE(steps >= 0, "steps must be >= 0");
    LEO_REQUIRE(lr > 0 && std::isfinite(lr), "learning rate must be positive");
    LEO_CUDA(cudaSetDevice(ctx->device));
    ensure_batch(M, batch);
    // training set: BF16 features [n][64], FP32 targets [n][256]
    {
      DevBuf<float> src((size_t)n * F);
      h2d(ctx, src.p, x, (size_t)n * F);
      M->Xall.alloc((size_t)n * kIn);
      launch(ctx, "mlp_pack", [&] {
        k_pack_x<<<grid_for(n * kIn, 256, ctx->sm_count * 8), 256, 0, ctx->stream>>>(n, F, src.p, M->Xall.p,
                                                                                     nullptr, 0);
      });
      M->Tall.alloc((size_t)n * kOut);
      h2d(ctx, M->Tall.p, t, (size_t)n * kOut);
      M->n_train = n;
      ctx_sync(ctx);
    }
    int64_t t0 = 0;
    d2h(ctx, &t0, M->step.p, 1);
    ctx_sync(ctx);
    M->hist_cap = t0 + steps;
    DevBuf<double> hist((size_t)std::max<int64_t>(M->hist_cap, 1));
    M->loss_hist = std::move(hist);
    // one step captured once (the sampled rows and Adam's bias correction
    // follow the step counter in device memory), replayed `steps` times
    if (M->graph) {
      cudaGraphExecDestroy(M->graph);
      M->graph = nullptr;
    }
    cudaGraph_t gr = nullptr;
    const bool prof = ctx->profiling;
    ctx->profiling = false;
    LEO_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    try {
      train_step_enqueue(M, seed, lr);
    } catch (...) {
      cudaStreamEndCapture(ctx->stream, &gr);
      if (gr) cudaGraphDestroy(gr);
      ctx->profiling = prof;
      throw;
    }
    LEO_CUDA(cudaStreamEndCapture(ctx->stream, &gr));
    ctx->profiling = prof;
    const cudaError_t e = cudaGraphInstantiate(&M->graph, gr, 0);
    cudaGraphDestroy(gr);
    if (e != cudaSuccess) fail(LEO2D_ERR_CUDA, std::string("graph instantiation: ") + cudaGetErrorString(e));
    for (int s = 0; s < steps; ++s) LEO_CUDA(cudaGraphLaunch(M->graph, ctx->stream));
    if (loss_hist && steps > 0) d2h(ctx, loss_hist, M->loss_hist.p + t0, (size_t)steps);
    ctx_check_status(ctx, "MLP training");
  });
}

leo2d_status leo2d_mlp_predict(leo2d_mlp* M, const float* x, int32_t F, int64_t n, float* y) {
  if (!M || !x || !y) return LEO2D_ERR_BAD_ARG;
  leo2d_ctx* ctx = M->ctx;
  return guard(ctx, [&] {
    LEO_REQUIRE(F >= 1 && F <= kIn, "feature count must be 1..64");
    LEO_REQUIRE(n >= 1, "n must be >= 1");
    LEO_CUDA(cudaSetDevice(ctx->device));
    DevBuf<float> src((size_t)n * F);
    DevBuf<__nv_bfloat16> X((size_t)n * kIn);
    DevBuf<float> Y((size_t)n * kOut);
    h2d(ctx, src.p, x, (size_t)n * F);
    launch(ctx, "mlp_pack", [&] {
      k_pack_x<<<grid_for(n * kIn, 256, ctx->sm_count * 8), 256, 0, ctx->stream>>>(n, F, src.p, X.p, nullptr, 0);
    });
    infer_rows(M, X.p, kIn, n, Y.p, nullptr, nullptr, false);
    d2h(ctx, y, Y.p, (size_t)n * kOut);
    ctx_check_status(ctx, "MLP inference");
  });
}

leo2d_status leo2d_mlp_site_features(leo2d_ctx* ctx, const leo2d_csr* csr, double twist_deg, float* x_out) {
  if (!ctx || !csr || !x_out) return LEO2D_ERR_BAD_ARG;
  return guard(ctx, [&] {
    LEO_CUDA(cudaSetDevice(ctx->device));
    const int64_t n = csr->n;
    DevBuf<double> cfg(2 * (size_t)std::max<int64_t>(n, 1));
    csr_shift_configs(ctx, csr, cfg.p);
    DevBuf<float> xf((size_t)std::max<int64_t>(n, 1) * kFeat);
    if (n > 0)
      launch(ctx, "mlp_features", [&] {
        k_features<<<grid_for(n, 256, ctx->sm_count * 8), 256, 0, ctx->stream>>>(n, cfg.p, csr->grid4.p,
                                                                                 (float)twist_deg, xf.p);
      });
    d2h(ctx, x_out, xf.p, (size_t)n * kFeat);
    ctx_sync(ctx);
  });
}

leo2d_status leo2d_mlp_site_sum(leo2d_mlp* M, const leo2d_csr* csr, double twist_deg, double* sum_out) {
  if (!M || !csr || !sum_out) return LEO2D_ERR_BAD_ARG;
  leo2d_ctx* ctx = M->ctx;
  return guard(ctx, [&] {
    LEO_CUDA(cudaSetDevice(ctx->device));
    const int64_t n = csr->n;
    LEO_REQUIRE(n >= 1, "empty matrix");
    SitePhase ph[2];
    csr_site_phases(csr, ph);
    // Work space from the context: features of one chunk of sites (32 bytes each),
    // the kernel's partial sums, the sums. A chunk is a whole number of tile pairs
    // for every SM, at most 2M sites, so that all of it stays within what the
    // context keeps (64 MiB); the 160 MB that 1M sites took before cost 0.36 ms a
    // call in four allocations.
    const int64_t wave = (int64_t)ctx->sm_count * 2 * kGemmBM;
    const int64_t chunk = std::min<int64_t>(n, std::max<int64_t>(1, (2000000 / wave)) * wave);
    const size_t part_n = std::max(mlp_fused_part(ctx, chunk), (size_t)tc_gemm_grid(ctx, (int)chunk, kOut) * kOut);
    const Scratch ws(ctx, {(size_t)chunk * kFeat * sizeof(__nv_bfloat16), part_n * sizeof(double), kOut * sizeof(double)});
    __nv_bfloat16* X = ws.get<__nv_bfloat16>(0);
    double *part = ws.get<double>(1), *sums = ws.get<double>(2);
    for (int64_t r0 = 0; r0 < n; r0 += chunk) {
      const int64_t rows = std::min(chunk, n - r0);
      launch(ctx, "mlp_features", [&] {
        k_site_rows<<<grid_for(rows, 256, ctx->sm_count * 8), 256, 0, ctx->stream>>>(
            rows, r0, ph[0], ph[1], csr->grid4.p, (float)twist_deg, X);
      });
      infer_rows(M, X, kFeat, rows, nullptr, sums, part, r0 > 0);
    }
    d2h(ctx, sum_out, sums, kOut);
    ctx_check_status(ctx, "MLP site sum");
  });
}

// Control-variate trace moments (see leo2d_gpu.h).
leo2d_status leo2d_kpm_dos_cv(leo2d_ctx* ctx, const leo2d_csr* csr, leo2d_mlp* M, const leo2d_kpm_cfg* cfg,
                              double twist_deg, int64_t num_sites, uint64_t site_seed, const double* weights,
                              double* mu_out, double* parts_out) {
  if (!ctx || !csr || !M || !cfg || !mu_out) return LEO2D_ERR_BAD_ARG;
  return guard(ctx, [&] {
    const int P = cfg->poly_order;
    LEO_REQUIRE(P >= 4 && P % 4 == 0, "poly_order must be a positive multiple of 4");
    LEO_REQUIRE(num_sites >= 0, "num_sites must be >= 0");
    LEO_REQUIRE(M->ctx == ctx, "the network belongs to another context");
    LEO_REQUIRE(!csr->complex_h, "the control variate is trained on real Hamiltonians (no magnetic field)");
    auto check = [&](leo2d_status st) {
      if (st != LEO2D_OK) fail(st, ctx->last_error);
    };
    LEO_CUDA(cudaSetDevice(ctx->device));
    const int64_t n = csr->n;
    const int Pc = std::min(P, kOut);  // moments covered by the network (even)
    // (1) random-phase estimate of every moment: mean over the vectors
    std::vector<double> phase(P, 0.0);
    const int R = cfg->num_vectors;
    if (R > 0) {
      std::vector<double> mu((size_t)R * P);
      check(leo2d_kpm_dos(ctx, csr, cfg, nullptr, mu.data()));
      for (int v = 0; v < R; ++v)
        for (int j = 0; j < P; ++j) phase[j] += mu[(size_t)v * P + j];
      for (int j = 0; j < P; ++j) phase[j] /= R;
    }
    // (2) the network's sum over every orbital
    std::vector<double> F(kOut, 0.0);
    check(leo2d_mlp_site_sum(M, csr, twist_deg, F.data()));
    // (3) exact moments at uniformly drawn orbitals minus the network there
    std::vector<double> corr(kOut, 0.0);
    if (num_sites > 0) {
      std::vector<int64_t> sites((size_t)num_sites);
      uint64_t st = site_seed;
      for (auto& x : sites) x = (int64_t)(((unsigned __int128)splitmix(st) * (uint64_t)n) >> 64);
      leo2d_kpm_cfg lc = *cfg;
      lc.poly_order = ((Pc + 3) / 4) * 4;
      lc.num_vectors = 1;
      std::vector<double> ld((size_t)num_sites * lc.poly_order);
      check(leo2d_kpm_ldos(ctx, csr, &lc, sites.data(), num_sites, ld.data()));
      DevBuf<int64_t> drows((size_t)num_sites);
      h2d(ctx, drows.p, sites.data(), (size_t)num_sites);
      DevBuf<double> dcfg(2 * (size_t)n);
      csr_shift_configs(ctx, csr, dcfg.p);
      DevBuf<__nv_bfloat16> X((size_t)num_sites * kIn);
      DevBuf<float> Y((size_t)num_sites * kOut);
      launch(ctx, "mlp_features", [&] {
        k_features_at<<<grid_for(num_sites, 256, ctx->sm_count * 8), 256, 0, ctx->stream>>>(
            num_sites, drows.p, dcfg.p, csr->grid4.p, (float)twist_deg, X.p);
      });
      infer_rows(M, X.p, kIn, num_sites, Y.p, nullptr, nullptr, false);
      std::vector<float> f((size_t)num_sites * kOut);
      d2h(ctx, f.data(), Y.p, f.size());
      ctx_check_status(ctx, "control-variate sites");
      for (int64_t s_ = 0; s_ < num_sites; ++s_)
        for (int j = 0; j < Pc; ++j)
          corr[j] += ld[(size_t)s_ * lc.poly_order + j] - (double)f[(size_t)s_ * kOut + j];
      for (int j = 0; j < Pc; ++j) corr[j] = corr[j] / (double)num_sites * (double)n;
    }
    for (int j = 0; j < P; ++j) {
      if (j < Pc) {
        const double w = weights ? weights[j] : 1.0;
        const double cv = F[j] + corr[j];
        mu_out[j] = w * cv + (1.0 - w) * phase[j];
      } else {
        mu_out[j] = phase[j];
      }
    }
    if (parts_out) {
      for (int j = 0; j < kOut; ++j) {
        parts_out[j] = F[j];
        parts_out[kOut + j] = corr[j];
        parts_out[2 * kOut + j] = j < P ? phase[j] : 0.0;
      }
    }
  });
}

}  // extern "C"
