// transform.cu - FP64 reconstruction of the DOS from Chebyshev moments.
//
// leo2d_dos_transform replaces Param_tools::densityTransform and
// densityTransformTrace (src/params/param_tools.cpp:661-768): Jackson kernel
// g_i = ((P-i) cos(pi i/P) + sin(pi i/P) cot(pi/P)) / P, then FFTW's REDFT01
// (DCT-III, out_k = in_0 + 2 sum_{j>=1} in_j cos(pi j (k+1/2)/P)) evaluated as a
// direct sum. The cosines come from a table of cospi(m / 2P), m = j (2k+1) mod 4P:
// P^2 evaluations of cospi and 64-bit remainders took 1.1 ms at P = 1000, the sum with
// the table is bound by the FP64 pipe (P^2 / 2 multiply-adds: the even and the odd
// terms of node k, added and subtracted, are nodes k and P - 1 - k).
// Whole call at P = 1000: 1.2 ms -> 52 us (the copies, launches and the wait).
// leo2d_dos_reconstruct evaluates the same damped series on any energy grid.
#include <cmath>
#include <vector>

#include "common.cuh"

using namespace leo2d;

namespace {

// (tan(pi / P) from the host)
__device__ __forceinline__ double jackson(int P, int i, double tan_p) {
  const double pi = 3.141592653589793;
  return ((P - i) * cos((pi * i) / P) + sin((pi * i) / P) / tan_p) / (P);
}

__global__ void k_mean_jackson(const double* __restrict__ mu, int P, int sets, double tan_p, double* __restrict__ in) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P; i += gridDim.x * blockDim.x) {
    double m = 0.0;
    if (sets == 1) {
      m = mu[i];
    } else {
      for (int s = 0; s < sets; ++s) m = m + mu[(size_t)s * P + i] / ((double)sets);
    }
    in[i] = jackson(P, i, tan_p) * m;
  }
}

// tab[m] = cos(pi m / (2P)), 0 <= m < 4P.
__global__ void k_cos_table(int P, double* __restrict__ tab) {
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < 4 * P; m += gridDim.x * blockDim.x)
    tab[m] = cospi((double)m / (double)(2 * (int64_t)P));
}

constexpr int kDctWarps = 8;

// A warp per pair of nodes k and P - 1 - k: the even and the odd terms, lanes over
// j; then a thread per node of the block's pairs for the scale. kTable false: each
// cosine by itself (a limit on allocations that the table would pass).
template <bool kTable>
__global__ void __launch_bounds__(kDctWarps * 32) k_dct3_nodes(const double* __restrict__ in,
                                                               const double* __restrict__ tab, int P, double rescale,
                                                               double shift, double scale, double* __restrict__ dos,
                                                               double* __restrict__ energies) {
  const double pi = 3.141592653589793;
  __shared__ double sums[kDctWarps][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int half = (P + 1) / 2, period = 4 * P;
  for (int k0 = blockIdx.x * kDctWarps; k0 < half; k0 += gridDim.x * kDctWarps) {
    const int k = k0 + warp;
    if (k < half) {
      const int64_t q = 2 * (int64_t)k + 1;
      // terms j = 1 + lane, + 32, ...: a lane's terms are all odd or all even
      int m = (int)(((int64_t)(1 + lane) * q) % period);
      const int step = (int)((32 * q) % period);
      double s = 0.0;
      for (int j = 1 + lane; j < P; j += 32) {
        s += in[j] * (kTable ? tab[m] : cospi((double)m / (double)(2 * (int64_t)P)));
        m += step;
        if (m >= period) m -= period;
      }
#pragma unroll
      for (int o = 16; o > 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane < 2) sums[warp][lane] = s;  // lane 0: odd j, lane 1: even j
    }
    __syncthreads();
    if (threadIdx.x < 2 * kDctWarps) {
      const int w = threadIdx.x >> 1, up = threadIdx.x & 1, kk = k0 + w;
      if (kk < half) {
        const int node = up ? P - 1 - kk : kk;
        const double acc = in[0] + 2.0 * (sums[w][1] + (up ? -sums[w][0] : sums[w][0]));
        const double E = shift + rescale * cos((node * 1.0 + 0.5) * pi / P);
        energies[node] = E;
        dos[node] = scale * acc / (pi * sqrt(rescale * rescale - (E - shift) * (E - shift)));
      }
    }
    __syncthreads();
  }
}

__global__ void k_reconstruct(const double* __restrict__ g, int P, const double* __restrict__ E,
                              int64_t nE, double rescale, double center, double scale,
                              double* __restrict__ out) {
  const double pi = 3.141592653589793;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nE;
       e += (int64_t)gridDim.x * blockDim.x) {
    const double x = (E[e] - center) / rescale;
    if (!(x > -1.0 && x < 1.0)) {
      out[e] = 0.0;
      continue;
    }
    double t0 = 1.0, t1 = x, acc = g[0];
    if (P > 1) acc += 2.0 * g[1] * t1;
    for (int n = 2; n < P; ++n) {
      const double t2 = 2.0 * x * t1 - t0;
      acc += 2.0 * g[n] * t2;
      t0 = t1;
      t1 = t2;
    }
    out[e] = scale * acc / (pi * rescale * sqrt(1.0 - x * x));
  }
}

}  // namespace

namespace leo2d {

void cos_table(leo2d_ctx* ctx, int P, double* tab) {
  launch(ctx, "cos_table", [&] { k_cos_table<<<grid_for(4 * (int64_t)P, 32), 32, 0, ctx->stream>>>(P, tab); });
}

}  // namespace leo2d

extern "C" {

leo2d_status leo2d_dos_transform(leo2d_ctx* ctx, const double* mu, int32_t poly_order,
                                 int32_t num_sets, double rescale, double shift, double scale,
                                 double* dos_out, double* energies_out) {
  if (!ctx || !mu || !dos_out) return LEO2D_ERR_BAD_ARG;
  return guard(ctx, [&] {
    LEO_REQUIRE(poly_order >= 2 && num_sets >= 1, "poly_order >= 2 and num_sets >= 1 required");
    LEO_REQUIRE(rescale > 0 && std::isfinite(rescale) && std::isfinite(shift), "bad rescale/shift");
    LEO_CUDA(cudaSetDevice(ctx->device));
    const int P = poly_order;
    LEO_REQUIRE(P < (1 << 29), "poly_order too large");
    const size_t row = (size_t)P * sizeof(double);
    const bool table = !g_alloc_cap || 4 * row <= g_alloc_cap;
    const Scratch ws(ctx, {row * num_sets, row, table ? 4 * row : 0, row, row});
    double *dmu = ws.get<double>(0), *din = ws.get<double>(1), *tab = ws.get<double>(2), *ddos = ws.get<double>(3),
           *dE = ws.get<double>(4);
    h2d(ctx, dmu, mu, (size_t)P * num_sets);
    // (a warp per block: FP64 functions of 1000 terms on one SM took 9 us)
    launch(ctx, "mean_jackson", [&] {
      k_mean_jackson<<<grid_for(P, 32), 32, 0, ctx->stream>>>(dmu, P, num_sets, std::tan(3.141592653589793 / P), din);
    });
    if (table) cos_table(ctx, P, tab);
    auto nodes = table ? k_dct3_nodes<true> : k_dct3_nodes<false>;
    launch(ctx, "dct3_nodes", [&] {
      nodes<<<grid_for((P + 1) / 2, kDctWarps, (int64_t)ctx->sm_count * 8), kDctWarps * 32, 0, ctx->stream>>>(
          din, tab, P, rescale, shift, scale, ddos, dE);
    });
    d2h(ctx, dos_out, ddos, P);
    if (energies_out) d2h(ctx, energies_out, dE, P);
    ctx_sync(ctx);
  });
}

leo2d_status leo2d_dos_reconstruct(leo2d_ctx* ctx, const double* mu, int32_t poly_order,
                                   const double* energies, int64_t num_energies, double rescale,
                                   double center, double scale, double* dos_out) {
  if (!ctx || !mu || !energies || !dos_out) return LEO2D_ERR_BAD_ARG;
  return guard(ctx, [&] {
    LEO_REQUIRE(poly_order >= 2 && num_energies >= 0, "bad sizes");
    LEO_REQUIRE(rescale > 0 && std::isfinite(rescale) && std::isfinite(center), "bad rescale/center");
    LEO_CUDA(cudaSetDevice(ctx->device));
    const int P = poly_order;
    const size_t terms = (size_t)P * sizeof(double), points = (size_t)num_energies * sizeof(double);
    const Scratch ws(ctx, {terms, terms, points, points});
    double *dmu = ws.get<double>(0), *dg = ws.get<double>(1), *dE = ws.get<double>(2), *dout = ws.get<double>(3);
    h2d(ctx, dmu, mu, P);
    h2d(ctx, dE, energies, num_energies);
    launch(ctx, "mean_jackson", [&] {
      k_mean_jackson<<<grid_for(P, 32), 32, 0, ctx->stream>>>(dmu, P, 1, std::tan(3.141592653589793 / P), dg);
    });
    if (num_energies > 0)
      launch(ctx, "reconstruct", [&] {
        k_reconstruct<<<grid_for(num_energies, 32), 32, 0, ctx->stream>>>(dg, P, dE, num_energies, rescale, center,
                                                                         scale, dout);
      });
    d2h(ctx, dos_out, dout, num_energies);
    ctx_sync(ctx);
  });
}

}  // extern "C"
