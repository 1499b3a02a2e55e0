// row_spmm.cu - every Chebyshev step of a vector block in one cooperative launch,
// over the plain rows of the matrix.
//
// Same recursion as the other step kernels (T_{n+1} = 2 H~ T_n - T_{n-1} with the
// two moment dots fused; Locality::computeDosTraceKPM / computeDosKPM,
// src/locality.cpp:6195-6234, 5997-6033, with SpMatrix::vectorMultiply,
// src/matrix/spmatrix.cpp:346-360, as its product). It serves what the
// tensor-core step does not: supercells and k points, whose step is bound by
// latency and launches, blocks of other widths than 32 (a few local targets),
// and the FP64 recursion.
//
// Common to the forms
//   The block's columns go in slices of CS (8, 16 or 32); the CTAs of a slice
//   form a group of g, each with a contiguous range of rows. Slices never meet;
//   the CTAs of a slice meet at a counter in global memory between steps (one
//   CTA: __syncthreads alone). A 16-byte load takes VL columns of a T_n row (4
//   FP32, 2 FP64), so LPE = CS / VL lanes share an entry. A service warp beside the
//   compute warps adds their dot sums in warp order and polls the barrier while
//   they wait; the CTAs' sums are stored per step and added in CTA order by one
//   reduction per launch. Between steps the matrix does not change: a warp asks
//   for its first entries of the next step before the barrier.
// FP32: the T_n rows a CTA needs (its window) are copied into shared memory at the
//   step's start, and the entries stream through a ring: the loop sees shared-memory
//   latency only. Up to 8000 rows k_cheb_win, LPE lanes a row, sums in the tiled
//   step's order; bound by three trips to L2 and back (window, rows out, barrier),
//   6 us. More rows k_cheb_pan, LPE lanes a block of 4 rows; bound by issue and the
//   shared-memory pipe, two thirds busy each between the same trips.
// FP64 small (k_cheb_small): the CTA's entries stay in shared memory for the whole
//   launch, a warp takes one row at a time, GR = 32 / LPE entries at once with up to U
//   groups in flight; a reduce-scatter over the groups ends a row.
// FP64 (k_cheb_sell): rows in slices of 16, the j-th entries of 16 rows next to
//   each other, LPE lanes own a row. Bound by the FP64 pipe (89 % active).
// Measured per step, tiled step before -> now: the 11,908-orbital cell with 128
//   columns 99 -> 16 us, a 2188-orbital cell with 12 targets 49 -> 8.2 us, 8 columns of
//   a 200k-orbital flake 62 -> 23 us, FP64 with 32 columns of 52k orbitals 251 -> 220
//   us. The first and third, LPE lanes a row: 26 and 27 us over the window, 34 and 42
//   with gathers through L1 (some misses in every group, about 1000 cycles each).
//
// Waits: the service warp polls the slice's counter, at most spin_limit polls or
//   two seconds; then the CTA records a timeout, raises the abort flag that every
//   polling CTA reads, and leaves.
#include <algorithm>
#include <type_traits>

#include "kpm.cuh"
#include "umma.cuh"

using namespace leo2d;

#include "step_kernels.cuh"

namespace {

constexpr int kSellRows = 16;  // rows of a slice of the interleaved format

template <typename T>
struct RowArgs {
  int64_t n, nnz;
  const int64_t* __restrict__ rowptr;  // small: row starts
  const int64_t* __restrict__ off;     // sell: [slices + 1] first position (of 16 entries) of each 16-row slice
  const int32_t* __restrict__ col;     // FP64
  const double* __restrict__ val;      // FP64
  T* x0;                               // T_k for even k
  T* x1;                               // T_k for odd k
  T* x2;                               // exact sums: a third buffer, T_k in x(k mod 3)
  int C;                               // columns of a vector row
  int group;                           // CTAs per slice
  int k0, k1;                          // steps of this launch
  // win: chunks of 8 positions, [chunk][16 rows][8] (off counts chunks)
  const float* __restrict__ wval;
  const uint16_t* __restrict__ widx;   // window positions
  const int32_t* __restrict__ slen;    // [slices] positions
  const int32_t* __restrict__ wlist;   // [tiles][win_stride] the window rows of each tile
  const int32_t* __restrict__ wcnt;    // [tiles]
  int64_t tiles, win_stride;
  int tile_slices, win_cap, slice_cap;
  const int32_t* __restrict__ blk;     // panels: [slices][blocks] the 4-row block at each place
  int warps;                           // panels: warps of a CTA that take slices
  int dot_slots, dot_rows;             // exact sums: the tiled step's row slots of a tile and rows per slot
  int ent_cap;                         // small: entries of a CTA that fit its shared memory
  int row_cap;                         // small: rows of a CTA that fit
  double* partials;                    // [k1 - k0][slices][group][2 CS]
  unsigned* bar;                       // [slices] arrivals, zero at launch
  int* abort;
  int* status;
  uint64_t spin_limit;
  int never_arrive;                    // test hook: barriers wait for one arrival too many
};

template <typename T>
struct RowVec;
template <>
struct RowVec<float> {
  static constexpr int VL = 4;
  float v[4];
  __device__ __forceinline__ void load(const float* p) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  }
  __device__ __forceinline__ void store(float* p) const {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
};
template <>
struct RowVec<double> {
  static constexpr int VL = 2;
  double v[2];
  __device__ __forceinline__ void load(const double* p) {
    const double2 x = *reinterpret_cast<const double2*>(p);
    v[0] = x.x; v[1] = x.y;
  }
  __device__ __forceinline__ void store(double* p) const { *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]); }
};

// A running sum: FP64, or for FP32 terms a pair of FP32 (PairSum).
template <typename T>
struct RowSum;
template <>
struct RowSum<double> {
  double h = 0.0;
  __device__ __forceinline__ void add(double x) { h += x; }
  __device__ __forceinline__ void add(const RowSum& o) { h += o.h; }
  __device__ __forceinline__ RowSum shfl_xor(int o) const {
    RowSum r;
    r.h = __shfl_xor_sync(0xffffffffu, h, o);
    return r;
  }
  __device__ __forceinline__ double value() const { return h; }
};
template <>
struct RowSum<float> : PairSum {
  RowSum() = default;
  __device__ __forceinline__ RowSum(const PairSum& p) : PairSum(p) {}
};

template <typename T>
__device__ __forceinline__ void row_fma(T (&acc)[RowVec<T>::VL], const RowVec<T>& x, T w) {
#pragma unroll
  for (int v = 0; v < RowVec<T>::VL; ++v) acc[v] += w * x.v[v];
}

__device__ __forceinline__ unsigned row_ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// First index whose value is at least t (a non-decreasing list of n).
__device__ int64_t row_lower_bound(const int64_t* a, int64_t n, int64_t t) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (a[mid] < t) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Adds the sums s[2 v + d] (column VL sub + v, dot d) over the warp's rows (lanes
// rl = 0 .. 32 / LPE - 1 of each sub) into out[2 column + d]: a reduce-scatter.
template <typename T, int CS>
__device__ __forceinline__ void row_warp_sums(RowSum<T> (&s)[2 * RowVec<T>::VL], RowSum<T>* out, int rl, int sub) {
  constexpr int VL = RowVec<T>::VL, LPE = CS / VL, RW = 32 / LPE;
  int cnt = 2 * VL, base = 0;  // lane rl keeps `cnt` sums from index `base` on
#pragma unroll
  for (int o = RW / 2; o > 0; o >>= 1) {
    const bool up = (rl & o) != 0;
    if (cnt > 1) {
      cnt >>= 1;
      if (up) base += cnt;
#pragma unroll
      for (int i = 0; i < VL; ++i)
        if (i < cnt) {
          const RowSum<T> send = up ? s[i] : s[i + cnt];
          const RowSum<T> got = send.shfl_xor(o * LPE);
          if (up) s[i] = s[i + cnt];
          s[i].add(got);
        }
    } else {
      s[0].add(s[0].shfl_xor(o * LPE));
    }
  }
  if (rl % (RW > 2 * VL ? RW / (2 * VL) : 1) == 0) {
#pragma unroll
    for (int i = 0; i < 2 * VL; ++i)
      if (i < cnt) out[2 * VL * sub + base + i] = s[i];
  }
}

// The service warp's side of a step's end, after the CTA's rows of T_{k+1} are
// written: announce the CTA (lane 0), ...
template <typename T>
__device__ __forceinline__ void row_announce(const RowArgs<T>& a, int slice) {
  __threadfence();  // the CTA's rows, at GPU scope
  atomicAdd(a.bar + slice, 1u);
}
// ... and wait for the group's arrivals of step k.
template <typename T>
__device__ __forceinline__ int row_await(const RowArgs<T>& a, int k, int slice) {
  const unsigned target = (unsigned)(k + 1 - a.k0) * (unsigned)a.group + (a.never_arrive ? 1u : 0u);
  int ok = 1;
  const uint64_t t0 = umma::now_ns();
  for (uint64_t p = 0;; ++p) {
    if (row_ld_acquire(a.bar + slice) >= target) break;
    if (*reinterpret_cast<volatile int*>(a.abort) != 0) {
      ok = 0;
      break;
    }
    if (p >= a.spin_limit || ((p & 255) == 255 && umma::now_ns() - t0 > 2000000000ull)) {
      atomicExch(a.status, leo2d::kStatusTimeout);
      atomicExch(a.abort, 1);
      ok = 0;
      break;
    }
  }
  __threadfence();
  return ok;
}

template <typename T, int CS>
__device__ __forceinline__ double* row_partials_of(const RowArgs<T>& a, int k, int slice, int bid) {
  return a.partials + (((size_t)(k - a.k0) * (gridDim.x / a.group) + slice) * a.group + bid) * 2 * CS;
}

// The end of a step: the warps' sums in wsum are complete and the CTA's rows of
// T_{k+1} written (first barrier). The service warp announces the CTA, adds the
// sums and waits for the group; the compute warps wait for it. False: give up.
template <typename T, int CS, int W>
__device__ __forceinline__ bool row_step_end(const RowArgs<T>& a, const RowSum<T> (*wsum)[2 * CS], int k, int slice,
                                             int bid, int* go) {
  const bool meet = a.group > 1 && k + 1 < a.k1;
  if (a.group == 1) __threadfence();  // (the next step may read the rows past L1)
  __syncthreads();
  if (threadIdx.x >= W * 32) {
    const int lane = threadIdx.x & 31;
    if (meet && lane == 0) row_announce(a, slice);
#pragma unroll
    for (int t0 = 0; t0 < 2 * CS; t0 += 32) {
      const int t = t0 + lane;
      if (t < 2 * CS) {
        // four chains over the warps: a single one is most of an FP64 sum's rounding
        RowSum<T> s[4];
#pragma unroll
        for (int w = 0; w < W; ++w) s[w & 3].add(wsum[w][t]);
        s[0].add(s[1]);
        s[2].add(s[3]);
        s[0].add(s[2]);
        row_partials_of<T, CS>(a, k, slice, bid)[t] = s[0].value();
      }
    }
    if (meet && lane == 0) *go = row_await(a, k, slice);
  }
  if (!meet) return true;
  __syncthreads();
  return *go != 0;
}

// ---------------------------------------------------------------- small matrices

constexpr int kSmallWarps = 23;

template <int CS>
__global__ void __launch_bounds__(kSmallWarps * 32 + 32, 1) k_cheb_small(const __grid_constant__ RowArgs<double> a) {
  using T = double;
  constexpr int W = kSmallWarps;
  constexpr int VL = RowVec<T>::VL, LPE = CS / VL, GR = 32 / LPE;
  constexpr int U = GR >= 16 ? 5 : 8;  // entry groups of a row in flight
  constexpr int REP = GR / VL;         // lanes holding the same element after the reduction (at least 1)
  static_assert(GR >= VL, "slice width of 8, 16 or 32 columns");
  extern __shared__ __align__(128) unsigned char row_smem[];
  __shared__ RowSum<T> wsum[2][W][2 * CS];
  __shared__ int64_t range[2];
  __shared__ int go;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int grp = lane / LPE, sub = lane % LPE;
  const int slice = (int)blockIdx.x / a.group, bid = (int)blockIdx.x % a.group;
  if (threadIdx.x < 2) {
    const int64_t b = bid + (int)threadIdx.x;
    range[threadIdx.x] = b == 0 ? 0 : b == a.group ? a.n : row_lower_bound(a.rowptr, a.n, a.nnz * b / a.group);
  }
  __syncthreads();
  const int64_t r0 = range[0];
  const int nr = (int)(range[1] - r0);
  const int64_t q0 = a.rowptr[r0];
  const int nq = (int)(a.rowptr[range[1]] - q0);
  // the CTA's entries and row starts, for every step of the launch (read from
  // global memory where a share of very uneven rows exceeds the room)
  const bool fits = nr <= a.row_cap && nq <= a.ent_cap;
  int* rp = reinterpret_cast<int*>(row_smem);
  unsigned char* es = row_smem + (((size_t)a.row_cap + 1) * 4 + 15) / 16 * 16;
  if (fits)
    for (int i = threadIdx.x; i <= nr; i += blockDim.x) rp[i] = (int)(a.rowptr[r0 + i] - q0);
  double* sval = reinterpret_cast<double*>(es);
  int32_t* scol = reinterpret_cast<int32_t*>(es + (size_t)a.ent_cap * 8);
  for (int i = threadIdx.x; fits && i < nq; i += blockDim.x) {
    sval[i] = a.val[q0 + i];
    scol[i] = a.col[q0 + i];
  }
  __syncthreads();
  const int C = a.C;
  // the lane's element after the reduction: column my_c of the row, held by REP lanes
  const int my_c = slice * CS + VL * sub + grp / REP;
  const bool owner = grp % REP == 0;

  for (int k = a.k0; k < a.k1; ++k) {
    RowSum<T>(*ws)[2 * CS] = wsum[k & 1];
    if (warp < W) {
      const T* tn = (k & 1) ? a.x1 : a.x0;
      T* tp = (k & 1) ? a.x0 : a.x1;
      const T* tg = tn + slice * CS + VL * sub;
      const T alpha = k == 0 ? T(1) : T(2);
      RowSum<T> s0, s1;
      for (int row = warp; row < nr; row += W) {
        const int beg = fits ? rp[row] : (int)(a.rowptr[r0 + row] - q0);
        const int end = fits ? rp[row + 1] : (int)(a.rowptr[r0 + row + 1] - q0);
        const int64_t at = (r0 + row) * C + my_c;
        T xn = T(0), xp = T(0);
        if (owner) {
          xn = tn[at];
          if (k != 0) xp = tp[at];
        }
        T acc[VL];
#pragma unroll
        for (int v = 0; v < VL; ++v) acc[v] = T(0);
        for (int e = beg; e < end; e += U * GR) {
          // entries past the row's end: its last one again, with a zero value
          RowVec<T> x[U];
          T w[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (u > 0 && e + u * GR >= end) break;  // warp-uniform
            const int i = e + u * GR + grp, p = min(i, end - 1);
            uint32_t c;
            c = (uint32_t)(fits ? scol[p] : a.col[q0 + p]);
            w[u] = i < end ? (fits ? sval[p] : a.val[q0 + p]) : 0.0;
            x[u].load(tg + (int64_t)c * C);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (u > 0 && e + u * GR >= end) break;
            row_fma<T>(acc, x[u], w[u]);
          }
        }
        // reduce-scatter over the GR groups
        int cnt = VL;
#pragma unroll
        for (int o = GR / 2; o > 0; o >>= 1) {
          const bool up = (grp & o) != 0;
          if (cnt > 1) {
            cnt >>= 1;
#pragma unroll
            for (int i = 0; i < VL / 2; ++i)
              if (i < cnt) {
                const T send = up ? acc[i] : acc[i + cnt];
                const T keep = up ? acc[i + cnt] : acc[i];
                acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o * LPE);
              }
          } else {
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o * LPE);
          }
        }
        if (owner) {
          const T y = k == 0 ? alpha * acc[0] : alpha * acc[0] - xp;
          tp[at] = y;
          s0.h += xn * xn;
          s1.h += y * xn;
        }
      }
      if (owner) {
        ws[warp][2 * (VL * sub + grp / REP)] = s0;
        ws[warp][2 * (VL * sub + grp / REP) + 1] = s1;
      }
    }
    if (!row_step_end<T, CS, W>(a, ws, k, slice, bid, &go)) break;
  }
}

// ---------------------------------------------------------------- larger matrices

// Entries are read once a step: they stay out of L1, which holds the T_n rows.
__device__ __forceinline__ uint32_t row_ld_entry(const int32_t* p) {
  uint32_t r;
  asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(r) : "l"(p));
  return r;
}
__device__ __forceinline__ double row_ld_entry(const double* p) {
  double r;
  asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(r) : "l"(p));
  return r;
}

// FP64: bound by the FP64 pipe (one warp multiply-add takes 16 cycles of an SM).
// 16 compute warps feed its four partitions evenly.
constexpr int kSellWarps = 16;

template <int CS>
__global__ void __launch_bounds__(kSellWarps * 32 + 32, 1) k_cheb_sell(const __grid_constant__ RowArgs<double> a) {
  using T = double;
  constexpr int W = kSellWarps;
  constexpr int VL = RowVec<T>::VL, LPE = CS / VL, RW = 32 / LPE;  // rows of a warp
  constexpr int IPS = kSellRows / RW;                              // items (a warp's rows) of a slice
  constexpr int U = 4;
  static_assert(kSellRows % RW == 0, "a warp's rows lie in one slice");
  __shared__ RowSum<T> wsum[2][W][2 * CS];
  __shared__ int64_t range[2];
  __shared__ int go;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rl = lane / LPE, sub = lane % LPE;
  const int slice = (int)blockIdx.x / a.group, bid = (int)blockIdx.x % a.group;
  const int64_t nsl = (a.n + kSellRows - 1) / kSellRows;
  if (threadIdx.x < 2) {
    const int64_t b = bid + (int)threadIdx.x;
    range[threadIdx.x] = b == 0 ? 0 : b == a.group ? nsl : row_lower_bound(a.off, nsl, a.off[nsl] * b / a.group);
  }
  __syncthreads();
  const int64_t items = range[1] * IPS, first = range[0] * IPS + warp;
  const int C = a.C;

  for (int k = a.k0; k < a.k1; ++k) {
    RowSum<T>(*ws)[2 * CS] = wsum[k & 1];
    if (warp < W) {
      const T* tn = (k & 1) ? a.x1 : a.x0;
      T* tp = (k & 1) ? a.x0 : a.x1;
      const T* tg = tn + slice * CS + VL * sub;
      const T alpha = k == 0 ? T(1) : T(2);
      RowSum<T> s[2 * VL];  // [2 v + d]: column VL sub + v, dot d
      for (int64_t item = first; item < items; item += W) {
        const int64_t row = item * RW + rl;
        const int64_t e0 = __ldg(a.off + item / IPS) * kSellRows + (row % kSellRows);
        const bool in = row < a.n;
        const int64_t at = row * C + slice * CS + VL * sub;
        RowVec<T> xn, xp;
#pragma unroll
        for (int v = 0; v < VL; ++v) xn.v[v] = xp.v[v] = T(0);
        if (in) {
          xn.load(tn + at);
          if (k != 0) xp.load(tp + at);
        }
        T part[2][VL];  // two sums of a row's entries: half the rounding of one chain
#pragma unroll
        for (int v = 0; v < VL; ++v) part[0][v] = part[1][v] = T(0);
        // the longest of this warp's rows (multiply-adds on the slice's padding
        // would cost as much as on entries)
        const int len = (int)__reduce_max_sync(
            0xffffffffu, in ? (unsigned)(__ldg(a.rowptr + row + 1) - __ldg(a.rowptr + row)) : 0u);
        uint32_t c[U];
        T w[U];
        auto load = [&](int u, int j) {
          const int64_t e = e0 + (int64_t)j * kSellRows;
          c[u] = row_ld_entry(a.col + e);
          w[u] = row_ld_entry(a.val + e);
        };
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (u < len) load(u, u);
        for (int j = 0; j < len; j += U) {  // the next group's entries asked for before this one's rows are used
          RowVec<T> x[U];
          T w2[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (j + u < len) x[u].load(tg + (int64_t)c[u] * C);
            w2[u] = w[u];
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (j + U + u < len) load(u, j + U + u);
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (j + u < len) row_fma<T>(part[u & 1], x[u], w2[u]);
        }
        T acc[VL];
#pragma unroll
        for (int v = 0; v < VL; ++v) acc[v] = part[0][v] + part[1][v];
        if (in) {
          RowVec<T> y;
#pragma unroll
          for (int v = 0; v < VL; ++v) {
            y.v[v] = k == 0 ? alpha * acc[v] : alpha * acc[v] - xp.v[v];
            s[2 * v].h += xn.v[v] * xn.v[v];
            s[2 * v + 1].h += y.v[v] * xn.v[v];
          }
          y.store(tp + at);
        }
      }
      row_warp_sums<T, CS>(s, ws[warp], rl, sub);
    }
    if (!row_step_end<T, CS, W>(a, ws, k, slice, bid, &go)) break;
  }
}

// FP32: the rows of T_n that a tile of rows needs (its window) are copied into
// shared memory once a step, all copies in flight at once; the entries stream
// through a ring per warp, 6 chunks ahead.
constexpr int kWinWarps = 23;                                 // + the service warp: 24 warps of 80 registers
constexpr int kWinChunk = 8;                                  // positions of a chunk
// chunks of a warp's ring (6 chunks ahead; 3 for 16 rows, whose chunks are as large)
__host__ __device__ constexpr int win_ring(int rw) { return rw == 16 ? 4 : 8; }
__host__ __device__ constexpr int win_ring_bytes(int rw) { return win_ring(rw) * kWinChunk * rw * 6; }
constexpr int kWinMax = 8192;                                 // rows of a window (16-bit positions, build limit)

__device__ __forceinline__ void row_cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void row_cp8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

// EXACT (few rows): the moments follow the tiled step's to the last bit of its FP32
// arithmetic. A row's entries are added in their order, as there, and its dots
// are grouped as there: FP32 sums over the 4 dot_rows rows of one row slot (one
// tile chunk), FP64 beyond. A density near the band edge amplifies the rounding
// of the moments by the order and more, so a local density of a small cell would
// otherwise move by 1e-3 of its norm. The dots of step k - 1 are taken by the service
// warp during step k from T_{k-1} and T_k, which a third vector buffer keeps.
template <int CS>
__global__ void __launch_bounds__(kWinWarps * 32 + 32, 1) k_cheb_win(const __grid_constant__ RowArgs<float> a) {
  using T = float;
  constexpr int W = kWinWarps;
  constexpr int VL = 4, LPE = CS / VL, RW = 32 / LPE, IPS = kSellRows / RW;
  constexpr int kWinRing = win_ring(RW), kWinAhead = RW == 16 ? 3 : 6;
  constexpr int kVal = kWinChunk * RW * 4, kIdx = kWinChunk * RW * 2;  // bytes of a ring chunk's parts
  extern __shared__ __align__(128) unsigned char row_smem[];
  __shared__ int go;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rl = lane / LPE, sub = lane % LPE;
  const int slice = (int)blockIdx.x / a.group, bid = (int)blockIdx.x % a.group;
  const int C = a.C;
  // this CTA's tiles, of tile_slices 16-row slices each
  const int64_t nsl = (a.n + kSellRows - 1) / kSellRows;
  const int64_t t_first = a.tiles * bid / a.group, t_end = a.tiles * (bid + 1) / a.group;
  const int64_t s_first = min(nsl, t_first * a.tile_slices), s_end = min(nsl, t_end * a.tile_slices);
  const int nslice = (int)(s_end - s_first);
  // shared memory: window | rings | chunk offsets of the slices | lengths | window list
  float* win = reinterpret_cast<float*>(row_smem);
  unsigned char* ring = row_smem + (size_t)a.win_cap * CS * 4 + (size_t)warp * win_ring_bytes(RW);
  int* spos = reinterpret_cast<int*>(row_smem + (size_t)a.win_cap * CS * 4 + (size_t)W * win_ring_bytes(RW));
  int* slen = spos + a.slice_cap + 1;
  int* list = slen + a.slice_cap + 1;
  const int64_t c_first = a.off[s_first];
  for (int i = threadIdx.x; i <= nslice; i += blockDim.x) {
    spos[i] = (int)(a.off[s_first + i] - c_first);
    if (i < nslice) slen[i] = a.slen[s_first + i];
  }
  __syncthreads();

  // The copy side of the warp's entry stream: items warp, warp + W, ... of each
  // tile in turn, chunk by chunk. The lane's sources advance by a fixed stride
  // inside an item.
  constexpr int kSlot = kVal + kIdx;
  constexpr int kNV = kVal / 16, kIB = kIdx >= 128 ? 16 : 8, kNI = kIdx / kIB;  // copying lanes, bytes of an index copy
  const int ntile = (int)(t_end - t_first);
  const int TI = a.tile_slices * IPS;  // items of a whole tile
  auto tile_items = [&](int t) { return min(TI, (nslice - t * a.tile_slices) * IPS); };
  const uint32_t ring_u = (uint32_t)__cvta_generic_to_shared(ring);
  const float* pv = nullptr;
  const uint16_t* pi = nullptr;
  int ft = 0, fi = 0, fleft = 0;   // tile, item of the tile, chunks of it still to copy
  uint32_t fslot = 0, cslot = 0;   // byte offsets of the ring chunks to fill and to use next
  auto fetch_item = [&]() {        // item (ft, fi), or the first one after it that exists
    while (ft < ntile && fi >= tile_items(ft)) {
      ++ft;
      fi = warp;
    }
    if (ft < ntile) {
      const int sl = ft * a.tile_slices + (int)((unsigned)fi / IPS);
      const int p0 = spos[sl];
      fleft = spos[sl + 1] - p0;
      const int64_t e = (c_first + p0) * (kWinChunk * kSellRows) + ((unsigned)fi % IPS) * RW * kWinChunk;
      pv = a.wval + e + 4 * lane;
      pi = a.widx + e + kIB / 2 * lane;
    }
  };
  auto fetch = [&]() {  // one chunk (or an empty group past the last one)
    while (fleft == 0 && ft < ntile) {
      fi += W;
      fetch_item();
    }
    if (fleft > 0) {
      const uint32_t d = ring_u + fslot;
      if (lane < kNV) row_cp16(d + 16 * lane, pv);
      if (lane < kNI) {
        if constexpr (kIB == 16) row_cp16(d + kVal + 16 * lane, pi);
        else row_cp8(d + kVal + 8 * lane, pi);
      }
      pv += kWinChunk * kSellRows;
      pi += kWinChunk * kSellRows;
      --fleft;
    }
    fslot = fslot == (kWinRing - 1) * kSlot ? 0u : fslot + kSlot;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto restart = [&]() {  // the first chunks of a step (the matrix does not change: also before the barrier)
    __syncwarp();
    fslot = cslot = 0;
    ft = 0;
    fi = warp;
    fleft = 0;
    fetch_item();
#pragma unroll 1
    for (int i = 0; i < kWinAhead; ++i) fetch();
  };
  if (warp < W) restart();

  auto buf = [&](int i) { return i == 0 ? a.x0 : i == 1 ? a.x1 : a.x2; };
  // the dots of step k from T_k and T_{k+1}, the CTA's share of the groups
  auto exact_dots = [&](int k) {
    const float* t0 = buf(k % 3) + slice * CS;
    const float* t1 = buf((k + 1) % 3) + slice * CS;
    const int span = 4 * a.dot_slots * a.dot_rows;  // rows of a chunk of four tiles
    const int64_t total = (a.n + span - 1) / span * a.dot_slots * LPE;
    double d[2 * VL];
#pragma unroll
    for (int v = 0; v < 2 * VL; ++v) d[v] = 0.0;
    for (int64_t i = (int64_t)bid * 32 + lane; i < total; i += (int64_t)a.group * 32) {
      const int64_t g = i / LPE;  // (chunk, slot); the lane's columns are 4 sub .. 4 sub + 3
      const int64_t row0 = g / a.dot_slots * span + g % a.dot_slots;
      float e[2 * VL];
#pragma unroll
      for (int v = 0; v < 2 * VL; ++v) e[v] = 0.f;
      for (int tile = 0; tile < 4; ++tile) {
        float f[2 * VL];
#pragma unroll
        for (int v = 0; v < 2 * VL; ++v) f[v] = 0.f;
        for (int r = 0; r < a.dot_rows; ++r) {
          const int64_t row = row0 + (int64_t)(tile * a.dot_rows + r) * a.dot_slots;
          if (row < a.n) {
            const float4 x = __ldcg(reinterpret_cast<const float4*>(t0 + row * C + VL * sub));
            const float4 y = __ldcg(reinterpret_cast<const float4*>(t1 + row * C + VL * sub));
            const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
            for (int v = 0; v < VL; ++v) {
              f[2 * v] = __fmaf_rn(xs[v], xs[v], f[2 * v]);
              f[2 * v + 1] = __fmaf_rn(ys[v], xs[v], f[2 * v + 1]);
            }
          }
        }
#pragma unroll
        for (int v = 0; v < 2 * VL; ++v) e[v] = __fadd_rn(e[v], f[v]);
      }
#pragma unroll
      for (int v = 0; v < 2 * VL; ++v) d[v] += (double)e[v];
    }
#pragma unroll
    for (int o = LPE; o < 32; o <<= 1)
#pragma unroll
      for (int v = 0; v < 2 * VL; ++v) d[v] += __shfl_xor_sync(0xffffffffu, d[v], o);
    if (lane < LPE) {
#pragma unroll
      for (int v = 0; v < 2 * VL; ++v) row_partials_of<T, CS>(a, k, slice, bid)[2 * VL * lane + v] = d[v];
    }
  };

  for (int k = a.k0; k < a.k1; ++k) {
    // (T_{k-1} from one buffer, T_{k+1} into the third)
    const T* tn = buf(k % 3);
    T* tp = buf((k + 1) % 3);
    const T* tm = buf((k + 2) % 3);
    const T alpha = k == 0 ? T(1) : T(2);
    for (int t = 0; t < ntile; ++t) {
      // the tile's window
      const int64_t l0 = (t_first + t) * a.win_stride;
      const int nwin = a.wcnt[t_first + t];
      if (ntile > 1 || k == a.k0) {
        for (int i = threadIdx.x; i < nwin; i += blockDim.x) list[i] = __ldg(a.wlist + l0 + i);
        __syncthreads();
      }
      {
        const uint32_t w_u = (uint32_t)__cvta_generic_to_shared(win);
        const T* src = tn + slice * CS;
        for (int i = threadIdx.x; i < nwin * LPE; i += blockDim.x)
          row_cp16(w_u + 16 * i, src + (int64_t)list[i / LPE] * C + 4 * (i % LPE));
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncthreads();
      if (warp < W) {
        const int items = tile_items(t);
        for (int item = warp; item < items; item += W) {
          const int sl = t * a.tile_slices + (int)((unsigned)item / IPS);
          const int64_t row = (s_first + sl) * kSellRows + ((unsigned)item % IPS) * RW + rl;
          const int len = slen[sl];
          const bool in = row < a.n;
          const int64_t at = row * C + slice * CS + VL * sub;
          float4 xp = make_float4(0.f, 0.f, 0.f, 0.f);
          if (in && k != 0) xp = __ldcg(reinterpret_cast<const float4*>(tm + at));
          T acc[VL];
#pragma unroll
          for (int v = 0; v < VL; ++v) acc[v] = T(0);
#pragma unroll 1
          for (int j = 0; j < len; j += kWinChunk) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kWinAhead - 1) : "memory");
            __syncwarp();
            fetch();
            const unsigned char* rc = ring + cslot;
            cslot = cslot == (kWinRing - 1) * kSlot ? 0u : cslot + kSlot;
            const uint4 ix = *reinterpret_cast<const uint4*>(rc + kVal + rl * (kWinChunk * 2));
            const float4 v0 = *reinterpret_cast<const float4*>(rc + rl * (kWinChunk * 4));
            const float4 v1 = *reinterpret_cast<const float4*>(rc + rl * (kWinChunk * 4) + 16);
            const uint32_t ii[4] = {ix.x, ix.y, ix.z, ix.w};
            const float w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
            RowVec<T> x[kWinChunk];
            auto get = [&](int u) {
              const uint32_t c = (u & 1) ? ii[u >> 1] >> 16 : ii[u >> 1] & 0xffffu;
              x[u].load(win + c * CS + VL * sub);
            };
            if (j + kWinChunk <= len) {
#pragma unroll
              for (int u = 0; u < kWinChunk; ++u) get(u);
#pragma unroll
              for (int u = 0; u < kWinChunk; ++u) row_fma<T>(acc, x[u], w[u]);
            } else {
#pragma unroll
              for (int u = 0; u < kWinChunk - 1; ++u)
                if (j + u < len) {
                  get(u);
                  row_fma<T>(acc, x[u], w[u]);
                }
            }
          }
          if (in) {
            RowVec<T> y;
            const T ps[4] = {xp.x, xp.y, xp.z, xp.w};
#pragma unroll
            for (int v = 0; v < VL; ++v) y.v[v] = k == 0 ? alpha * acc[v] : alpha * acc[v] - ps[v];
            y.store(tp + at);
          }
        }
      }
      if (t + 1 < ntile) __syncthreads();  // the window is read
    }
    const bool last = k + 1 == a.k1;
    if (warp < W) {
      if (!last) restart();
    } else if (k > a.k0) {
      exact_dots(k - 1);
    }
    if (a.group == 1) __threadfence();  // (the next step reads the rows past L1)
    __syncthreads();
    if (a.group > 1) {  // (also after the last step: its dots need every CTA's rows)
      if (threadIdx.x == W * 32) {
        row_announce(a, slice);
        go = row_await(a, k, slice);
      }
      __syncthreads();
      if (go == 0) break;
    }
    if (last && warp == W) exact_dots(k);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ---------------------------------------------------------------- panels

// FP32, more rows: blocks of 4 consecutive rows (under the locality ordering, of a
// compact cluster) share the union of their columns. LPE lanes own a block: a
// gathered T_n row and its 4 values make 16 FMAs a lane, so 16 rows of 32 columns
// cost 5 wavefronts of shared memory for each of their 98 or so common positions where
// row by row they cost 5.75 for each of 4 x 67 entries. The values stored for the zeros
// of the union are paid back by a single index per position (427 bytes a row for 402).
// Per step, the 11,908-orbital cell with 128 columns / 8 columns of a 200k flake:
// 26 / 27 us row by row; panels in row order 23 / 35 (slices padded to their longest
// block); blocks by size within a tile 19 / 24; chunks of 8 to 16 positions and warps
// in fours 17.5 / 23; packed FMAs (half the issue slots of the products) 16 / 22; the
// dots of a block's 4 rows summed in pairs, not of 16 in FP32, 16 / 22.5.
// The window and the entry ring are those of k_cheb_win.
constexpr int kPanRows = 4;
constexpr int kPanWarps = 15;  // + the service warp: 16 warps of 128 registers
// blocks of a warp's item (= a slice of the format), positions of a chunk
__host__ __device__ constexpr int pan_blocks(int cs) { return 128 / cs; }
__host__ __device__ constexpr int pan_chunk(int cs) { return cs == 32 ? 16 : 8; }
constexpr int kPanRing = 3;  // chunks of a warp's ring, all but one of them ahead
__host__ __device__ constexpr int pan_ring_bytes(int cs) { return kPanRing * pan_chunk(cs) * pan_blocks(cs) * 18; }

// (a, b) += w (x, y), both lanes of one fma.rn.f32x2
__device__ __forceinline__ void pan_fma2(float& a, float& b, float w, float x, float y) {
  unsigned long long r;
  asm("{\n\t.reg .b64 s, t, u;\n\tmov.b64 s, {%3, %3};\n\tmov.b64 t, {%4, %5};\n\tmov.b64 u, {%1, %2};\n\t"
      "fma.rn.f32x2 %0, s, t, u;\n\t}"
      : "=l"(r)
      : "f"(a), "f"(b), "f"(w), "f"(x), "f"(y));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}

template <int CS>
__global__ void __launch_bounds__(kPanWarps * 32 + 32, 1) k_cheb_pan(const __grid_constant__ RowArgs<float> a) {
  using T = float;
  constexpr int W = kPanWarps;
  constexpr int VL = 4, LPE = CS / VL, RW = pan_blocks(CS), PC = pan_chunk(CS), RB = kPanRows;
  constexpr int kSliceRows = RW * RB;
  constexpr int kVal = PC * RW * 16, kIdx = PC * RW * 2, kSlot = kVal + kIdx;
  extern __shared__ __align__(128) unsigned char row_smem[];
  __shared__ RowSum<T> wsum[2][W][2 * CS];
  __shared__ int go;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rl = lane / LPE, sub = lane % LPE;
  const int slice = (int)blockIdx.x / a.group, bid = (int)blockIdx.x % a.group;
  const int C = a.C;
  // this CTA's tiles, of tile_slices slices each
  const int64_t nsl = (a.n + kSliceRows - 1) / kSliceRows;
  const int64_t t_first = a.tiles * bid / a.group, t_end = a.tiles * (bid + 1) / a.group;
  const int64_t s_first = min(nsl, t_first * a.tile_slices), s_end = min(nsl, t_end * a.tile_slices);
  const int nslice = (int)(s_end - s_first);
  // shared memory: window | rings | chunk offsets of the slices | lengths | window list
  float* win = reinterpret_cast<float*>(row_smem);
  unsigned char* ring = row_smem + (size_t)a.win_cap * CS * 4 + (size_t)warp * pan_ring_bytes(CS);
  int* spos = reinterpret_cast<int*>(row_smem + (size_t)a.win_cap * CS * 4 + (size_t)W * pan_ring_bytes(CS));
  int* slen = spos + a.slice_cap + 1;
  int* list = slen + a.slice_cap + 1;
  const int64_t c_first = a.off[s_first];
  for (int i = threadIdx.x; i <= nslice; i += blockDim.x) {
    spos[i] = (int)(a.off[s_first + i] - c_first);
    if (i < nslice) slen[i] = a.slen[s_first + i];
  }
  __syncthreads();

  // The copy side of the warp's entry stream: slices warp, warp + step, ... of each
  // tile in turn, chunk by chunk (warps from `step` on have none).
  const int first = warp < a.warps ? warp : 1 << 28, step = a.warps;
  const int ntile = (int)(t_end - t_first);
  auto tile_items = [&](int t) { return min(a.tile_slices, nslice - t * a.tile_slices); };
  const uint32_t ring_u = (uint32_t)__cvta_generic_to_shared(ring);
  const float* pv = nullptr;
  const uint16_t* pi = nullptr;
  int ft = 0, fi = 0, fleft = 0;  // tile, item of the tile, chunks of it still to copy
  uint32_t fslot = 0, cslot = 0;  // byte offsets of the ring chunks to fill and to use next
  auto fetch_item = [&]() {       // item (ft, fi), or the first one after it that exists
    while (ft < ntile && fi >= tile_items(ft)) {
      ++ft;
      fi = first;
    }
    if (ft < ntile) {
      const int sl = ft * a.tile_slices + fi;
      fleft = spos[sl + 1] - spos[sl];
      pv = a.wval + (c_first + spos[sl]) * (kVal / 4) + 4 * lane;
      pi = a.widx + (c_first + spos[sl]) * (kIdx / 2) + 8 * lane;
    }
  };
  auto fetch = [&]() {  // one chunk (or an empty group past the last one)
    while (fleft == 0 && ft < ntile) {
      fi += step;
      fetch_item();
    }
    if (fleft > 0) {
      const uint32_t d = ring_u + fslot + 16 * lane;
#pragma unroll
      for (int i = 0; i < kVal / 512; ++i) row_cp16(d + 512 * i, pv + 128 * i);
      if (lane < kIdx / 16) row_cp16(d + kVal, pi);
      pv += kVal / 4;
      pi += kIdx / 2;
      --fleft;
    }
    fslot = fslot == (kPanRing - 1) * kSlot ? 0u : fslot + kSlot;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto restart = [&]() {  // the first chunks of a step (the matrix does not change: also before the barrier)
    __syncwarp();
    fslot = cslot = 0;
    ft = 0;
    fi = first;
    fleft = 0;
    fetch_item();
#pragma unroll 1
    for (int i = 0; i < kPanRing - 1; ++i) fetch();
  };
  if (warp < W) restart();

  for (int k = a.k0; k < a.k1; ++k) {
    RowSum<T>(*ws)[2 * CS] = wsum[k & 1];
    const T* tn = (k & 1) ? a.x1 : a.x0;
    T* tp = (k & 1) ? a.x0 : a.x1;
    const T alpha = k == 0 ? T(1) : T(2);
    RowSum<T> s[2 * VL];  // [2 v + d]: column VL sub + v, dot d
    for (int t = 0; t < ntile; ++t) {
      // the tile's window
      const int64_t l0 = (t_first + t) * a.win_stride;
      const int nwin = a.wcnt[t_first + t];
      if (ntile > 1 || k == a.k0) {
        for (int i = threadIdx.x; i < nwin; i += blockDim.x) list[i] = __ldg(a.wlist + l0 + i);
        __syncthreads();
      }
      {
        const uint32_t w_u = (uint32_t)__cvta_generic_to_shared(win);
        const T* src = tn + slice * CS;
        for (int i = threadIdx.x; i < nwin * LPE; i += blockDim.x)
          row_cp16(w_u + 16 * i, src + (int64_t)list[i / LPE] * C + 4 * (i % LPE));
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncthreads();
      if (warp < W) {
        const int items = tile_items(t);
        for (int item = first; item < items; item += step) {
          const int sl = t * a.tile_slices + item;
          const int64_t row0 = (int64_t)__ldg(a.blk + (s_first + sl) * RW + rl) * RB;
          const int len = slen[sl];
          float acc[RB][VL];
#pragma unroll
          for (int r = 0; r < RB; ++r)
#pragma unroll
            for (int v = 0; v < VL; ++v) acc[r][v] = 0.f;
#pragma unroll 1
          for (int j = 0; j < len; j += PC) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kPanRing - 2) : "memory");
            __syncwarp();
            fetch();
            const unsigned char* rc = ring + cslot;
            cslot = cslot == (kPanRing - 1) * kSlot ? 0u : cslot + kSlot;
            const uint2* pix = reinterpret_cast<const uint2*>(rc + kVal + rl * (PC * 2));
            auto four = [&](int h) {  // positions 4 h .. 4 h + 3 of the chunk
              const uint2 ix = pix[h];
              const uint32_t c[4] = {ix.x & 0xffffu, ix.x >> 16, ix.y & 0xffffu, ix.y >> 16};
              float4 x[4], w[4];
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                x[u] = *reinterpret_cast<const float4*>(win + c[u] * CS + VL * sub);
                w[u] = *reinterpret_cast<const float4*>(rc + ((4 * h + u) * RW + rl) * 16);
              }
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const float ww[4] = {w[u].x, w[u].y, w[u].z, w[u].w};
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                  pan_fma2(acc[r][0], acc[r][1], ww[r], x[u].x, x[u].y);
                  pan_fma2(acc[r][2], acc[r][3], ww[r], x[u].z, x[u].w);
                }
              }
            };
            four(0);
#pragma unroll
            for (int h = 1; h < PC / 4; ++h)
              if (j + 4 * h < len) four(h);
          }
          const int64_t at = row0 * C + slice * CS + VL * sub;
          // dots: FP32 over the item's 4 rows (as the tiled step; over 16 they lose two bits), then pairs
          T f[2 * VL];
#pragma unroll
          for (int v = 0; v < 2 * VL; ++v) f[v] = T(0);
          float4 xn[RB], xp[RB];
#pragma unroll
          for (int r = 0; r < RB; ++r) {
            xn[r] = xp[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row0 + r < a.n) {
              xn[r] = __ldcg(reinterpret_cast<const float4*>(tn + at + (int64_t)r * C));
              if (k != 0) xp[r] = __ldcg(reinterpret_cast<const float4*>(tp + at + (int64_t)r * C));
            }
          }
#pragma unroll
          for (int r = 0; r < RB; ++r) {
            const float xs[4] = {xn[r].x, xn[r].y, xn[r].z, xn[r].w}, ps[4] = {xp[r].x, xp[r].y, xp[r].z, xp[r].w};
            RowVec<T> y;
#pragma unroll
            for (int v = 0; v < VL; ++v) {
              y.v[v] = k == 0 ? alpha * acc[r][v] : alpha * acc[r][v] - ps[v];
              f[2 * v] += xs[v] * xs[v];
              f[2 * v + 1] += y.v[v] * xs[v];
            }
            if (row0 + r < a.n) y.store(tp + at + (int64_t)r * C);
          }
#pragma unroll
          for (int v = 0; v < 2 * VL; ++v) s[v].add(f[v]);
        }
      }
      if (t + 1 < ntile) __syncthreads();  // the window is read
    }
    if (warp < W) {
      if (k + 1 < a.k1) restart();
      row_warp_sums<T, CS>(s, ws[warp], rl, sub);
    }
    if (!row_step_end<T, CS, W>(a, ws, k, slice, bid, &go)) break;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// dots[step][slice columns][2] = the CTAs' partials added in a fixed order: 1024 / w
// chains over the CTAs (w = 16, 32 or 64 values), then a tree. (One chain over 152 CTAs
// made the moments of an FP64 run four times as inexact as the tiled step's, rms 3.3e-16
// of the largest against 8e-17.)
constexpr int kDotThreads = 1024;
__global__ void __launch_bounds__(kDotThreads) k_row_dots(const double* __restrict__ partials, int slices, int group,
                                                             int w, int C2, double* __restrict__ dots) {
  __shared__ double red[kDotThreads];
  const int step = blockIdx.x, slice = blockIdx.y, t = threadIdx.x % w, g = threadIdx.x / w, chains = kDotThreads / w;
  const double* p = partials + ((size_t)step * slices + slice) * group * w;
  double s = 0.0;
  for (int b = g; b < group; b += chains) s += p[(size_t)b * w + t];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = chains / 2; o > 0; o >>= 1) {
    if (g < o) red[threadIdx.x] += red[threadIdx.x + o * w];
    __syncthreads();
  }
  if (g == 0) dots[(size_t)step * C2 + slice * w + t] = red[t];
}

// ---------------------------------------------------------------- the formats

// FP64: positions of each 16-row slice (its longest row). FP32: also the slice's
// chunks of 8 positions. One thread per slice.
__global__ void k_slice_len(int64_t n, int64_t nsl, const int64_t* __restrict__ rowptr, int chunk,
                            int64_t* __restrict__ count, int32_t* __restrict__ slen) {
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < nsl; s += (int64_t)gridDim.x * blockDim.x) {
    int64_t top = 0;
    for (int64_t r = s * kSellRows; r < min(n, (s + 1) * kSellRows); ++r) top = max(top, rowptr[r + 1] - rowptr[r]);
    count[s] = (top + chunk - 1) / chunk;
    if (slen) slen[s] = (int32_t)top;
  }
}

// FP64, one warp per slice: lane (h, r) writes positions h, h + 2, ... of row r.
// Rows shorter than the slice end in zero values at their first column (their
// own index when they are empty).
__global__ void k_sell_fill(int64_t n, int64_t nsl, const int64_t* __restrict__ rowptr, const int64_t* __restrict__ off,
                            const int32_t* __restrict__ col, const double* __restrict__ val,
                            int32_t* __restrict__ scol, double* __restrict__ sval) {
  const int lane = threadIdx.x & 31, r = lane % kSellRows, h = lane / kSellRows;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
  for (int64_t s = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); s < nsl; s += warps) {
    const int64_t row = s * kSellRows + r, p0 = off[s], len = off[s + 1] - p0;
    const int64_t beg = row < n ? rowptr[row] : 0, cnt = row < n ? rowptr[row + 1] - beg : 0;
    for (int64_t j = h; j < len; j += 32 / kSellRows) {
      const int64_t at = (p0 + j) * kSellRows + r, e = beg + (j < cnt ? j : 0);
      scol[at] = cnt > 0 ? col[e] : (int32_t)min(row, n - 1);
      sval[at] = j < cnt ? val[e] : 0.0;
    }
  }
}

constexpr int kWinThreads = 512;
constexpr int kWinSet = 2 * kWinMax;  // hash slots; more than kWinMax distinct columns are refused

// One CTA per tile: the distinct columns of its rows (an empty row counts its own
// index), sorted, into list[tile * stride ..]; cnt[tile] their number; more than
// `stride` raises *over.
__global__ void __launch_bounds__(kWinThreads) k_win_list(int64_t n, int tile_rows, const int64_t* __restrict__ rowptr,
                                                          const int32_t* __restrict__ col, int64_t stride,
                                                          int32_t* __restrict__ list, int32_t* __restrict__ cnt,
                                                          int* __restrict__ over) {
  extern __shared__ __align__(16) uint32_t win_keys[];
  uint32_t* set = win_keys;            // [kWinSet]
  uint32_t* keys = win_keys + kWinSet;  // [kWinMax]
  __shared__ int fresh, out;
  const int64_t r0 = (int64_t)blockIdx.x * tile_rows, r1 = min(n, r0 + tile_rows);
  for (int i = threadIdx.x; i < kWinSet; i += kWinThreads) set[i] = 0xFFFFFFFFu;
  if (threadIdx.x == 0) fresh = out = 0;
  __syncthreads();
  auto insert = [&](uint32_t c) {
    uint32_t h = (c * 2654435761u) >> (32 - 14);
    for (int probe = 0; probe < kWinSet; ++probe) {  // bounded
      const uint32_t prev = atomicCAS(&set[h], 0xFFFFFFFFu, c);
      if (prev == 0xFFFFFFFFu) {
        atomicAdd(&fresh, 1);
        break;
      }
      if (prev == c) break;
      h = (h + 1) & (kWinSet - 1);
    }
  };
  static_assert(kWinSet == 1 << 14, "hash of 14 bits");
  for (int64_t e = rowptr[r0] + threadIdx.x; e < rowptr[r1]; e += kWinThreads) {
    if (*reinterpret_cast<volatile int*>(&fresh) > (int)stride) break;
    insert((uint32_t)col[e]);
  }
  for (int64_t r = r0 + threadIdx.x; r < r1; r += kWinThreads)
    if (rowptr[r + 1] == rowptr[r] && *reinterpret_cast<volatile int*>(&fresh) <= (int)stride) insert((uint32_t)r);
  __syncthreads();
  const int m = fresh;
  if (m > (int)stride) {
    if (threadIdx.x == 0) {
      atomicExch(over, 1);
      cnt[blockIdx.x] = 0;
    }
    return;
  }
  for (int i = threadIdx.x; i < kWinSet; i += kWinThreads)
    if (set[i] != 0xFFFFFFFFu) keys[atomicAdd(&out, 1)] = set[i];
  int p2 = 1;
  while (p2 < m) p2 <<= 1;
  __syncthreads();
  for (int i = m + threadIdx.x; i < p2; i += kWinThreads) keys[i] = 0xFFFFFFFFu;
  __syncthreads();
  for (int k = 2; k <= p2; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < p2; i += kWinThreads) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const bool up = (i & k) == 0;
          const uint32_t x = keys[i], y = keys[ixj];
          if ((x > y) == up) {
            keys[i] = y;
            keys[ixj] = x;
          }
        }
      }
      __syncthreads();
    }
  for (int i = threadIdx.x; i < m; i += kWinThreads) list[blockIdx.x * stride + i] = (int32_t)keys[i];
  if (threadIdx.x == 0) cnt[blockIdx.x] = m;
}

// One CTA per tile, a warp per row: the chunks of its slices, [chunk][16 rows][8],
// the columns as window positions. Rows shorter than the slice end in zero values
// at their first column (their own index when they are empty).
__global__ void __launch_bounds__(kWinThreads) k_win_fill(int64_t n, int64_t nsl, int tile_slices,
                                                          const int64_t* __restrict__ rowptr,
                                                          const int64_t* __restrict__ off,
                                                          const int32_t* __restrict__ col, const float* __restrict__ val,
                                                          int64_t stride, const int32_t* __restrict__ list,
                                                          const int32_t* __restrict__ cnt, float* __restrict__ wval,
                                                          uint16_t* __restrict__ widx) {
  extern __shared__ __align__(16) uint32_t win_keys[];
  const int m = cnt[blockIdx.x];
  for (int i = threadIdx.x; i < m; i += kWinThreads) win_keys[i] = (uint32_t)list[blockIdx.x * stride + i];
  __syncthreads();
  auto find = [&](uint32_t c) {  // (present)
    int lo = 0, hi = m - 1;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (win_keys[mid] < c) lo = mid + 1;
      else hi = mid;
    }
    return lo;
  };
  const int lane = threadIdx.x & 31;
  const int64_t s0 = (int64_t)blockIdx.x * tile_slices, s1 = min(nsl, s0 + tile_slices);
  for (int64_t row = s0 * kSellRows + (threadIdx.x >> 5); row < s1 * kSellRows; row += kWinThreads / 32) {
    const int64_t s = row / kSellRows, p0 = off[s];
    const int r = (int)(row % kSellRows), room = (int)(off[s + 1] - p0) * kWinChunk;
    const int64_t beg = row < n ? rowptr[row] : 0;
    const int len = row < n ? (int)(rowptr[row + 1] - beg) : 0;
    auto place = [&](int j) { return ((p0 + j / kWinChunk) * kSellRows + r) * kWinChunk + j % kWinChunk; };
    for (int j = lane; j < len; j += 32) {
      const int64_t at = place(j);
      widx[at] = (uint16_t)find((uint32_t)col[beg + j]);
      wval[at] = val[beg + j];
    }
    const uint16_t pad = row >= n ? 0 : (uint16_t)find(len > 0 ? (uint32_t)col[beg] : (uint32_t)row);
    for (int j = len + lane; j < room; j += 32) {
      const int64_t at = place(j);
      widx[at] = pad;
      wval[at] = 0.f;
    }
  }
}

// Panels, one CTA per tile, a warp per block of 4 rows. A bit per window position and
// row gives the block's union; `fill` = 0: size[block] = its positions, and *over is
// raised when a row stores a column twice; 1: the chunks of the tile's slices, values
// [chunk][PC][RW][4], positions [chunk][RW][PC] (both zero before, so that places past
// the union read window row 0 with weight 0).
// The order of a block's positions is free, and decides the bank conflicts of the
// gathers: a quarter warp reads `cls` rows of the window at once (4 for slices of 8
// columns, 2 of 16, 1 of 32), without a conflict when their positions differ modulo cls.
// So block b's m-th position of class c (position modulo cls) goes to place
// cls m + (c - b) mod cls, as long as every class has an m-th one; the others follow.
// Within a class the positions whose weights are all at most a quarter of the block's
// largest come first: a row's many small products are then rounded at the size of their
// own sum, not of the few large ones'. LDOS of a 200k flake, 1000 moments, relative error
// against 64 bits over six sets of targets: 1.2e-6 to 1.8e-6 (1.7e-6 to 3.1e-6 in
// position order, 2.1e-6 to 3.8e-6 in the tiled step), at the same time a step.
constexpr int kPanWords = kWinMax / 32;
constexpr size_t kPanFillSmem =
    (size_t)kWinMax * 4 + (size_t)(kWinThreads / 32) * kPanWords * ((kPanRows + 1) * 4 + 16);
__global__ void __launch_bounds__(kWinThreads) k_pan_fill(int64_t n, int64_t nsl, int tile_slices, int RW, int PC, int cls,
                                                          int fill, const int64_t* __restrict__ rowptr,
                                                          const int32_t* __restrict__ col,
                                                          const float* __restrict__ val, int64_t stride,
                                                          const int32_t* __restrict__ list,
                                                          const int32_t* __restrict__ cnt, int32_t* __restrict__ size,
                                                          const int32_t* __restrict__ order,
                                                          const int64_t* __restrict__ off, float* __restrict__ wval,
                                                          uint16_t* __restrict__ widx, int* __restrict__ over) {
  extern __shared__ __align__(16) uint32_t win_keys[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // per word of 32 positions: the places before it of each class, for small and for large weights
  unsigned long long* pre = reinterpret_cast<unsigned long long*>(win_keys + kWinMax) + (size_t)warp * kPanWords * 2;
  // the union by row, then the positions with a large weight
  uint32_t* bits = win_keys + kWinMax + (size_t)(kWinThreads / 32) * kPanWords * 4 + (size_t)warp * (kPanRows + 1) * kPanWords;
  uint32_t* large = bits + kPanRows * kPanWords;
  const int m = cnt[blockIdx.x], words = (m + 31) / 32;
  for (int i = threadIdx.x; i < m; i += kWinThreads) win_keys[i] = (uint32_t)list[blockIdx.x * stride + i];
  __syncthreads();
  auto find = [&](uint32_t c) {  // (present)
    int lo = 0, hi = m - 1;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (win_keys[mid] < c) lo = mid + 1;
      else hi = mid;
    }
    return lo;
  };
  auto mask = [&](int c) { return (cls == 4 ? 0x11111111u : cls == 2 ? 0x55555555u : ~0u) << c; };
  auto united = [&](int i) {
    uint32_t u = 0;
#pragma unroll
    for (int r = 0; r < kPanRows; ++r) u |= bits[r * kPanWords + i];
    return u;
  };
  const int64_t s0 = (int64_t)blockIdx.x * tile_slices, s1 = min(nsl, s0 + tile_slices);
  for (int64_t at = s0 * RW + warp; at < s1 * RW; at += kWinThreads / 32) {
    const int64_t s = at / RW, b = fill ? order[at] : at, row0 = b * kPanRows;
    const int rl = (int)(at % RW);
    for (int i = lane; i < words; i += 32)
#pragma unroll
      for (int r = 0; r <= kPanRows; ++r) bits[r * kPanWords + i] = 0u;
    float top = 0.f;
    if (fill)
      for (int64_t e = rowptr[min(n, row0)] + lane; e < rowptr[min(n, row0 + kPanRows)]; e += 32)
        top = fmaxf(top, fabsf(val[e]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    __syncwarp();
    bool twice = false;
    for (int r = 0; r < kPanRows && row0 + r < n; ++r)
      for (int64_t e = rowptr[row0 + r] + lane; e < rowptr[row0 + r + 1]; e += 32) {
        const int w = find((uint32_t)col[e]);
        const uint32_t bit = 1u << (w & 31);
        if (atomicOr(&bits[r * kPanWords + (w >> 5)], bit) & bit) twice = true;
        if (fill && fabsf(val[e]) > 0.25f * top) atomicOr(&large[w >> 5], bit);
      }
    __syncwarp();
    // the lane's words, 8 at most
    const int per = (words + 31) / 32, i0 = min(words, lane * per), i1 = min(words, i0 + per);
    int own[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // small ones of each class, large ones
    for (int i = i0; i < i1; ++i)
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if ((c & 3) < cls) own[c] += __popc(united(i) & (c < 4 ? ~large[i] : large[i]) & mask(c & 3));
    int first[8], total[4];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      int x = own[c];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      first[c] = x - own[c];
      const int all = __shfl_sync(0xffffffffu, x, 31);
      if (c < 4) {
        total[c] = all;
      } else {
        first[c] += total[c - 4];
        total[c - 4] += all;
      }
    }
    if (fill == 0) {
      if (__any_sync(0xffffffffu, twice) && lane == 0) atomicExch(over, 1);
      if (lane == 0) size[b] = total[0] + total[1] + total[2] + total[3];
      __syncwarp();
      continue;
    }
    int least = total[0];
    for (int c = 1; c < cls; ++c) least = min(least, total[c]);
    for (int i = i0; i < i1; ++i) {
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const uint32_t u = united(i) & (g ? large[i] : ~large[i]);
        unsigned long long p = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          p |= (unsigned long long)first[4 * g + c] << (16 * c);
          if (c < cls) first[4 * g + c] += __popc(u & mask(c));
        }
        pre[2 * i + g] = p;
      }
    }
    __syncwarp();
    for (int r = 0; r < kPanRows && row0 + r < n; ++r)
      for (int64_t e = rowptr[row0 + r] + lane; e < rowptr[row0 + r + 1]; e += 32) {
        const int w = find((uint32_t)col[e]), i = w >> 5, c = w & (cls - 1);
        const uint32_t below = mask(c) & ((1u << (w & 31)) - 1u);
        const int g = (large[i] >> (w & 31)) & 1;
        const int k = (int)((pre[2 * i + g] >> (16 * c)) & 0xffffu) +
                      __popc(united(i) & (g ? large[i] : ~large[i]) & below);
        int before = 0;  // positions of the classes before it that have no partner
        for (int q = 0; q < c; ++q) before += total[q] - least;
        const int j = k < least ? cls * k + ((c - rl) & (cls - 1)) : cls * least + before + (k - least);
        const int64_t chunk = off[s] + j / PC;
        widx[(chunk * RW + rl) * PC + j % PC] = (uint16_t)w;
        wval[((chunk * PC + j % PC) * RW + rl) * 4 + r] = val[e];
      }
    __syncwarp();
  }
}

// One CTA per tile: its blocks by falling size (slices of blocks of equal length: in
// row order a slice of 16 was padded to its longest by half), the length of each
// slice and its chunks of PC positions.
__global__ void __launch_bounds__(kWinThreads) k_pan_order(int64_t nsl, int tile_slices, int RW, int PC,
                                                           const int32_t* __restrict__ size,
                                                           int32_t* __restrict__ order, int32_t* __restrict__ slen,
                                                           int64_t* __restrict__ count) {
  const int64_t s0 = (int64_t)blockIdx.x * tile_slices, s1 = min(nsl, s0 + tile_slices), b0 = s0 * RW;
  const int nb = (int)((s1 - s0) * RW);
  for (int i = threadIdx.x; i < nb; i += kWinThreads) {
    const int mine = size[b0 + i];
    int rank = 0;
    for (int j = 0; j < nb; ++j) {
      const int other = __ldg(size + b0 + j);
      rank += other > mine || (other == mine && j < i) ? 1 : 0;
    }
    order[b0 + rank] = (int32_t)(b0 + i);
    if (rank % RW == 0) {
      slen[s0 + rank / RW] = mine;
      count[s0 + rank / RW] = (mine + PC - 1) / PC;
    }
  }
}

void row_coop_launch(leo2d_ctx* ctx, const void* kern, unsigned grid, int threads, size_t smem, void* args) {
  int occ = 0;
  allow_smem(ctx, kern);
  LEO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads, smem));
  LEO_REQUIRE(occ >= 1 && grid <= (unsigned)ctx->sm_count, "multi-step launch: the CTAs cannot all be resident");
  void* argv[1] = {args};
  // cooperative: every CTA resident at once, as the barriers need
  launch(ctx, "cheb_steps",
         [&] { LEO_CUDA(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(threads), argv, smem, ctx->stream)); });
}

const void* small_kernel(int cs) {
  return cs == 8 ? (const void*)k_cheb_small<8> : cs == 16 ? (const void*)k_cheb_small<16> : (const void*)k_cheb_small<32>;
}
const void* win_kernel(int cs) {
  return cs == 8 ? (const void*)k_cheb_win<8> : cs == 16 ? (const void*)k_cheb_win<16> : (const void*)k_cheb_win<32>;
}
const void* pan_kernel(int cs) {
  return cs == 8 ? (const void*)k_cheb_pan<8> : cs == 16 ? (const void*)k_cheb_pan<16> : (const void*)k_cheb_pan<32>;
}
const void* sell_kernel(int cs) {
  return cs == 8 ? (const void*)k_cheb_sell<8> : cs == 16 ? (const void*)k_cheb_sell<16> : (const void*)k_cheb_sell<32>;
}

// FP32: rows up to which the EXACT form runs; FP64: rows x column slices up to
// which the small form runs
constexpr int64_t kSmallRows = 8000;
constexpr size_t kRowPartialBytes = (size_t)16 << 20;  // CTA partials held between reductions

size_t small_smem(int row_cap, int ent_cap) {
  return (((size_t)row_cap + 1) * 4 + 15) / 16 * 16 + (size_t)ent_cap * 12;
}
// static shared memory of the kernels: the warps' sums of two steps and a little more
size_t row_static_smem(int warps, int cs) { return (size_t)2 * warps * 2 * cs * 8 + 256; }

size_t win_smem(const RowShape& s, int win_cap, int slice_cap) {
  const size_t rings = s.exact ? (size_t)kWinWarps * win_ring_bytes(128 / s.cs) : (size_t)kPanWarps * pan_ring_bytes(s.cs);
  return (size_t)win_cap * (s.cs * 4 + 4) + rings + 2 * ((size_t)slice_cap + 1) * 4;
}
// One shape of the window format, for the list of those that do not fit.
uint64_t win_key(const RowShape& s, bool perm) {
  return (uint64_t)s.group << 32 | (uint64_t)s.cs << 2 | (s.exact ? 2u : 0u) | (perm ? 1u : 0u);
}
int win_slice_rows(const RowShape& s) { return s.exact ? kSellRows : kPanRows * pan_blocks(s.cs); }

// The window format (rows for the EXACT form, else panels) for `group` CTAs a slice;
// false when a slice alone has too wide a window or a row stores a column twice
// (panels).
bool build_win(leo2d_ctx* ctx, leo2d_csr* csr, bool perm, RowShape& s) {
  const int SR = win_slice_rows(s), PC = s.exact ? kWinChunk : pan_chunk(s.cs);
  const int64_t n = csr->n, nsl = (n + SR - 1) / SR;
  const int64_t* rp = perm ? csr->prow.p : csr->rowptr.p;
  const int32_t* col = perm ? csr->pcol.p : csr->col.p;
  const float* val = perm ? csr->pval32.p : csr->val32.p;
  const size_t room = ctx->smem_optin - row_static_smem(s.warps, s.cs);
  const bool current = csr->win_off.p && csr->win_perm == perm && csr->win_cs == s.cs && csr->win_group == s.group &&
                       csr->win_exact == s.exact;
  if (!current) {
    csr_drop_win(csr);
    csr->win_off.alloc(nsl + 1);
    csr->win_slen.alloc(nsl);
    const size_t list_smem = (size_t)(kWinSet + kWinMax) * sizeof(uint32_t);
    allow_smem(ctx, (const void*)k_win_list);
    DevBuf<int> over(1);
    auto refuse = [&]() {  // (the search is not repeated on the next call)
      csr_drop_win(csr);
      csr->win_refused.push_back(win_key(s, perm));
      return false;
    };
    // tiles per CTA: the fewest whose windows fit
    for (int64_t m = 1;; m += std::max<int64_t>(1, m / 2)) {
      const int64_t ts = std::max<int64_t>(1, (nsl + s.group * m - 1) / (s.group * m));
      const int64_t tiles = (nsl + ts - 1) / ts;
      const int64_t per_cta = (tiles + s.group - 1) / s.group;
      const int64_t slice_cap = ts * per_cta;
      const size_t fixed = win_smem(s, 0, (int)slice_cap);
      if (fixed >= room) return refuse();
      const int64_t cap = std::min<int64_t>((int64_t)((room - fixed) / (s.cs * 4 + 4)) / 4 * 4, kWinMax);
      // (a window holds the tile's own rows and, on a bilayer, as many of the other sheet)
      if (ts > 1 && ts * SR > cap) continue;
      csr->win_list.alloc((size_t)(tiles * cap));
      csr->win_cnt.alloc((size_t)tiles);
      LEO_CUDA(cudaMemsetAsync(over.p, 0, sizeof(int), ctx->stream));
      launch(ctx, "win_build", [&] {
        k_win_list<<<(unsigned)tiles, kWinThreads, list_smem, ctx->stream>>>(n, (int)(ts * SR), rp, col, cap,
                                                                         csr->win_list.p, csr->win_cnt.p, over.p);
      });
      int h = 0;
      d2h(ctx, &h, over.p, 1);
      ctx_sync(ctx);
      if (h != 0) {
        if (ts == 1) return refuse();
        continue;
      }
      csr->win_tiles = tiles;
      csr->win_stride = cap;
      csr->win_tile_slices = (int)ts;
      csr->win_slice_cap = (int)slice_cap;
      break;
    }
    DevBuf<int32_t> size(s.exact ? 0 : (size_t)nsl * pan_blocks(s.cs));
    auto panels = [&](int fill) {
      launch(ctx, "win_build", [&] {
        k_pan_fill<<<(unsigned)csr->win_tiles, kWinThreads, kPanFillSmem, ctx->stream>>>(
            n, nsl, csr->win_tile_slices, pan_blocks(s.cs), PC, 32 / s.cs, fill, rp, col, val, csr->win_stride,
            csr->win_list.p, csr->win_cnt.p, size.p, csr->win_blk.p, csr->win_off.p, csr->win_val.p, csr->win_idx.p,
            over.p);
      });
    };
    {
      DevBuf<int64_t> count(nsl);
      if (s.exact) {
        launch(ctx, "win_build", [&] {
          k_slice_len<<<grid_for(nsl, 256, (int64_t)ctx->sm_count * 16), 256, 0, ctx->stream>>>(n, nsl, rp, kWinChunk, count.p, csr->win_slen.p);
        });
      } else {
        allow_smem(ctx, (const void*)k_pan_fill);
        csr->win_blk.alloc((size_t)nsl * pan_blocks(s.cs));
        panels(0);
        launch(ctx, "win_build", [&] {
          k_pan_order<<<(unsigned)csr->win_tiles, kWinThreads, 0, ctx->stream>>>(
              nsl, csr->win_tile_slices, pan_blocks(s.cs), PC, size.p, csr->win_blk.p, csr->win_slen.p, count.p);
        });
      }
      exclusive_scan_i64(ctx, count.p, csr->win_off.p, nsl);
    }
    int64_t chunks = 0;
    int twice = 0;
    d2h(ctx, &chunks, csr->win_off.p + nsl, 1);
    d2h(ctx, &twice, over.p, 1);
    ctx_sync(ctx);
    if (twice != 0) {
      csr_drop_win(csr);
      csr->win_twice = true;
      return false;
    }
    const size_t count = (size_t)std::max<int64_t>(chunks, 1) * SR * PC;  // values
    const size_t positions = s.exact ? count : count / kPanRows;
    csr->win_val.alloc(count);
    csr->win_idx.alloc(positions);
    if (s.exact) {
      launch(ctx, "win_build", [&] {
        k_win_fill<<<(unsigned)csr->win_tiles, kWinThreads, (size_t)kWinMax * sizeof(uint32_t), ctx->stream>>>(
            n, nsl, csr->win_tile_slices, rp, csr->win_off.p, col, val, csr->win_stride, csr->win_list.p, csr->win_cnt.p,
            csr->win_val.p, csr->win_idx.p);
      });
    } else {
      LEO_CUDA(cudaMemsetAsync(csr->win_val.p, 0, count * sizeof(float), ctx->stream));
      LEO_CUDA(cudaMemsetAsync(csr->win_idx.p, 0, positions * sizeof(uint16_t), ctx->stream));
      panels(1);
    }
    csr->win_perm = perm;
    csr->win_cs = s.cs;
    csr->win_group = s.group;
    csr->win_exact = s.exact;
  }
  s.group = (int)std::min<int64_t>(s.group, csr->win_tiles);
  s.smem = win_smem(s, (int)csr->win_stride, csr->win_slice_cap);
  // Warps that take slices: as few as need the same number of rounds over a tile, in
  // fours, one to each scheduler (20 slices: 12 warps and 8, not 15 and 5, whose
  // latency nothing would cover).
  const int rounds = (csr->win_tile_slices + kPanWarps - 1) / kPanWarps;
  s.slice_warps = std::min(kPanWarps, ((csr->win_tile_slices + rounds - 1) / rounds + 3) / 4 * 4);
  return true;
}

// False when the padding to each slice's longest row would take as much again as the
// entries: the matrix's memory is then the caller's to plan with, not this format's.
bool build_sell(leo2d_ctx* ctx, leo2d_csr* csr, bool perm) {
  if (csr->sell_off.p && csr->sell_perm == perm) return true;
  csr_drop_sell(csr);
  const int64_t n = csr->n, nsl = (n + kSellRows - 1) / kSellRows;
  const int64_t* rp = perm ? csr->prow.p : csr->rowptr.p;
  DevBuf<int64_t> len(nsl);
  csr->sell_off.alloc(nsl + 1);
  launch(ctx, "sell_build", [&] {
    k_slice_len<<<grid_for(nsl, 256, (int64_t)ctx->sm_count * 16), 256, 0, ctx->stream>>>(n, nsl, rp, 1, len.p, nullptr);
  });
  exclusive_scan_i64(ctx, len.p, csr->sell_off.p, nsl);
  int64_t total = 0;
  d2h(ctx, &total, csr->sell_off.p + nsl, 1);
  ctx_sync(ctx);
  const size_t count = (size_t)std::max<int64_t>(total, 1) * kSellRows;
  if (count > 2 * (size_t)csr->nnz + 16 * kSellRows) {  // (a few slices of a small matrix: any padding)
    csr_drop_sell(csr);
    csr->sell_uneven[perm] = true;
    return false;
  }
  csr->sell_col.alloc(count);
  csr->sell_val.alloc(count);
  launch(ctx, "sell_build", [&] {
    k_sell_fill<<<grid_for(nsl, 8, (int64_t)ctx->sm_count * 32), 256, 0, ctx->stream>>>(
        n, nsl, rp, csr->sell_off.p, perm ? csr->pcol.p : csr->col.p, perm ? csr->pval64.p : csr->val64.p,
        csr->sell_col.p, csr->sell_val.p);
  });
  csr->sell_perm = perm;
  return true;
}

}  // namespace

namespace leo2d {

void csr_drop_sell(leo2d_csr* csr) {
  csr->sell_off.release();
  csr->sell_col.release();
  csr->sell_val.release();
}

void csr_drop_win(leo2d_csr* csr) {
  csr->win_off.release();
  csr->win_slen.release();
  csr->win_list.release();
  csr->win_cnt.release();
  csr->win_val.release();
  csr->win_idx.release();
  csr->win_blk.release();
  csr->win_cs = csr->win_group = 0;
}

void csr_drop_rows(leo2d_csr* csr) {
  csr_drop_sell(csr);
  csr_drop_win(csr);
  csr->sell_uneven[0] = csr->sell_uneven[1] = false;
  csr->win_refused.clear();
}

void row_release(leo2d_csr* csr, bool fp64) {
  if (fp64) csr_drop_sell(csr);
  else csr_drop_win(csr);
}

static int row_slices(int cols, int cols_used) {
  const int cs = std::min(cols, 32);
  return std::max(1, (std::min(cols_used, cols) + cs - 1) / cs);
}

bool row_wants_order(int64_t n, bool fp64) { return !fp64 && n > kSmallRows; }

bool row_pays(int64_t n, bool fp64, int steps) {
  // Below 8000 rows and in FP64 the format takes a few small launches; the window
  // format of more rows, with the locality ordering, takes 0.4 ms (9k rows) to 1.5 ms
  // (200k) and gains 20 to 90 us a step. From 32 steps on it pays in the first run
  // already: 8 local targets at P = 64, tiled steps / first run with the format built /
  // later runs: 9k orbitals 0.86 / 0.74 / 0.33 ms, 200k 3.3 / 2.4 / 0.84 ms; 16
  // vectors of 60k 3.2 / 1.4 / 0.64 ms. A shorter run takes the tiled step also where
  // the format is there: the same call gives the same bits whatever ran before it.
  return fp64 || n <= kSmallRows || steps >= 32;
}

// The form and its launch, nothing built.
static RowShape row_shape(const leo2d_ctx* ctx, const leo2d_csr* csr, bool perm, bool fp64, int cols, int cols_used) {
  RowShape s{};
  s.cs = std::min(cols, 32);
  s.slices = row_slices(cols, cols_used);
  const int64_t n = csr->n, most = std::max(1, ctx->sm_count / s.slices);
  if (!fp64) {
    s.form = kRowWin;
    s.exact = n <= kSmallRows && !perm;
    s.warps = s.exact ? kWinWarps : kPanWarps;
    // a slice (16 rows; panels: 64 of 8 columns, 16 of 32) per CTA and up: the rows'
    // latency and the shared-memory bandwidth are spread over every SM
    s.group = (int)std::min<int64_t>(most, (n + win_slice_rows(s) - 1) / win_slice_rows(s));
    s.dot_slots = tile_slots(cols, false, tile_default_warps(cols, false));
    s.dot_rows = tile_default_rows(s.dot_slots);
  } else {
    // The small form: one CTA up to 4 rows a warp (a barrier costs more than
    // three more rows), else about two thirds of a row per warp, so that no warp
    // of an uneven share takes two rows while rows are few.
    s.form = kRowSmall;
    s.warps = kSmallWarps;
    s.group = n <= 4 * kSmallWarps ? 1 : (int)std::min<int64_t>(most, (n + 15) / 16);
    // room of a CTA: its share of the entries and rows and some more (a share that
    // exceeds it is read from global memory)
    const int64_t ent = csr->nnz / s.group + 1, rows = n / s.group + 1;
    s.ent_cap = (int)std::min<int64_t>((ent + ent / 8 + 1024 + 3) / 4 * 4, 1 << 20);
    s.row_cap = (int)std::min<int64_t>(rows + rows / 4 + 64, 1 << 20);
    s.smem = small_smem(s.row_cap, s.ent_cap);
    if (n * s.slices > kSmallRows || s.smem + row_static_smem(kSmallWarps, s.cs) > ctx->smem_optin) {
      s.form = kRowSell;
      s.warps = kSellWarps;
      const int rw = 32 / (s.cs / 2);
      s.group = (int)std::max<int64_t>(1, std::min<int64_t>(most, ((n + rw - 1) / rw + s.warps - 1) / s.warps));
      s.smem = 0;
    }
  }
  return s;
}

bool row_refused(const leo2d_ctx* ctx, const leo2d_csr* csr, bool perm, bool fp64, int cols, int cols_used) {
  const RowShape s = row_shape(ctx, csr, perm, fp64, cols, cols_used);
  if (s.form == kRowSell) return csr->sell_uneven[perm];
  if (s.form != kRowWin) return false;
  if (!s.exact && csr->win_twice) return true;
  return std::find(csr->win_refused.begin(), csr->win_refused.end(), win_key(s, perm)) != csr->win_refused.end();
}

bool row_prepare(leo2d_ctx* ctx, leo2d_csr* csr, bool perm, bool fp64, int cols, int cols_used, RowShape& s) {
  if (row_refused(ctx, csr, perm, fp64, cols, cols_used)) return false;
  s = row_shape(ctx, csr, perm, fp64, cols, cols_used);
  if (s.form == kRowWin && !build_win(ctx, csr, perm, s)) return false;
  if (s.form == kRowSell && !build_sell(ctx, csr, perm)) return false;
  const size_t per_step = (size_t)s.slices * s.group * 2 * s.cs * sizeof(double);
  const size_t held = g_alloc_cap ? std::min(kRowPartialBytes, g_alloc_cap) : kRowPartialBytes;
  s.chunk = (int)std::max<size_t>(1, held / per_step);
  return true;
}

size_t row_partials(const RowShape& s, int steps) {
  return (size_t)std::min(s.chunk, steps) * s.slices * s.group * 2 * s.cs;
}

void row_run(leo2d_ctx* ctx, const leo2d_csr* csr, const RowShape& s, bool perm, bool fp64, int cols, int steps,
             void* x0, void* x1, void* x2, double* partials, unsigned* bar, double* dots) {
  auto go = [&](auto* x, const void* kern) {
    using T = std::remove_pointer_t<decltype(x)>;
    RowArgs<T> a{};
    a.n = csr->n;
    a.nnz = csr->nnz;
    a.rowptr = perm ? csr->prow.p : csr->rowptr.p;
    if (s.form == kRowSmall) {
      a.col = perm ? csr->pcol.p : csr->col.p;
      a.val = perm ? csr->pval64.p : csr->val64.p;
      a.ent_cap = s.ent_cap;
      a.row_cap = s.row_cap;
    } else if (s.form == kRowSell) {
      a.off = csr->sell_off.p;
      a.col = csr->sell_col.p;
      a.val = csr->sell_val.p;
    } else {
      a.off = csr->win_off.p;
      a.slen = csr->win_slen.p;
      a.wval = csr->win_val.p;
      a.widx = csr->win_idx.p;
      a.wlist = csr->win_list.p;
      a.wcnt = csr->win_cnt.p;
      a.tiles = csr->win_tiles;
      a.win_stride = csr->win_stride;
      a.tile_slices = csr->win_tile_slices;
      a.win_cap = (int)csr->win_stride;
      a.slice_cap = csr->win_slice_cap;
      a.blk = csr->win_blk.p;
      a.warps = s.slice_warps;
      a.dot_slots = s.dot_slots;
      a.dot_rows = s.dot_rows;
    }
    a.x0 = static_cast<T*>(x0);
    a.x1 = static_cast<T*>(x1);
    a.x2 = static_cast<T*>(x2);
    a.C = cols;
    a.group = s.group;
    a.partials = partials;
    a.bar = bar;
    a.abort = reinterpret_cast<int*>(bar + kRowBarWords - 1);
    a.status = ctx->status.p;
    a.spin_limit = ctx->spin_limit;
    a.never_arrive = ctx->test_unsatisfied_wait;
    for (int k0 = 0; k0 < steps; k0 += s.chunk) {
      a.k0 = k0;
      a.k1 = std::min(steps, k0 + s.chunk);
      LEO_CUDA(cudaMemsetAsync(bar, 0, sizeof(unsigned) * kRowBarWords, ctx->stream));
      row_coop_launch(ctx, kern, (unsigned)(s.slices * s.group), 32 * (1 + s.warps), s.smem, &a);
      launch(ctx, "row_dots", [&] {
        k_row_dots<<<dim3((unsigned)(a.k1 - a.k0), (unsigned)s.slices), kDotThreads, 0, ctx->stream>>>(
            partials, s.slices, s.group, 2 * s.cs, 2 * cols, dots + (size_t)k0 * 2 * cols);
      });
    }
  };
  if (fp64) go((double*)nullptr, s.form == kRowSmall ? small_kernel(s.cs) : sell_kernel(s.cs));
  else go((float*)nullptr, s.exact ? win_kernel(s.cs) : pan_kernel(s.cs));
}

}  // namespace leo2d
