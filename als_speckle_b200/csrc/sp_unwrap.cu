// Polar unwrap of an N x N float map with cubic B-spline interpolation, and
// its row mean: the `prtfq` / `rftfq` outputs of the reference
// (speckle/phasing.py:1454-1458, :1512-1516, :1603-1605, :1701-1705), which
// call wrapping.unwrap(array, (0, N/2, (N/2, N/2))) (wrapping.py:8-67,
// :131-176) and average each radius over its angles.
//
// wrapping.unwrap samples the map on a polar grid with
// scipy.ndimage.map_coordinates(order=3, mode='constant').  That is cubic
// B-spline interpolation: the map is first turned into B-spline coefficients
// by the recursive prefilter of Unser, Aldroubi & Eden ("B-spline signal
// processing: Part II", IEEE Trans. Signal Process. 41, 1993) along each
// axis, with the whole-sample mirror boundary f[-k] = f[k],
// f[N-1+k] = f[N-1-k] and its exact causal initialisation (Thevenaz, Blu &
// Unser, "Interpolation revisited", IEEE Trans. Med. Imaging 19, 2000);
// every sample is then sum_ij c[i][j] b3(y - i) b3(x - j) over its 4 x 4
// neighbours, the coefficient index mirrored the same way beyond the edges.
// Both steps run in FP64 here; each sample is rounded to float32 (the map's
// type, which map_coordinates keeps) before the row mean.
#include <cmath>

#include "sp_common.cuh"

namespace sp {

// The cubic B-spline's pole and the prefilter's gain (1 - z)(1 - 1/z) = 6.
constexpr double kZ3 = -0.267949192431122706472553658494127633;  // sqrt(3) - 2
constexpr double kGain3 = 6.0;

// Prefilter one line of n values: in[k * stride] (float map or FP64
// coefficients) -> out[k * stride] (FP64); in may equal out.  The recursions
// carry their running value in a register, so only the loads of the next
// inputs are on the critical path and they can be issued ahead.
template <class T>
__device__ void bspline3_line(const T* in, double* out, int n, long stride) {
  const double z = kZ3;
  if (n == 1) {
    out[0] = (double)in[0];
    return;
  }
  // causal initialisation: sum_j z^j x~[j] over one period (length 2n - 2)
  // of the mirrored line x~, divided by 1 - z^(2n-2):
  //   x[0] + z^(n-1) x[n-1] + sum_{k=1}^{n-2} (z^k + z^(2n-2-k)) x[k]
  // (powers by repeated products, which underflow to 0 harmlessly)
  const double zn1 = pow(z, (double)(n - 1));
  double head = 0.0, tail = 0.0, zk = z;
#pragma unroll 8
  for (int k = 1; k < n - 1; ++k) {
    head += zk * (double)in[k * stride];
    zk *= z;
  }
  zk = z;  // z^(n-1-k) for k = n-2 down to 1
#pragma unroll 8
  for (int k = n - 2; k >= 1; --k) {
    tail += zk * (double)in[k * stride];
    zk *= z;
  }
  const double x0 = (double)in[0], xl = (double)in[(long)(n - 1) * stride];
  // the gain (1 - z)(1 - 1/z) = 6 is applied to the inputs as they are read
  double prev = kGain3 * (x0 + zn1 * xl + head + zn1 * tail) / (1.0 - zn1 * zn1);
  out[0] = prev;
#pragma unroll 8
  for (int k = 1; k < n; ++k) {
    prev = kGain3 * (double)in[k * stride] + z * prev;
    out[k * stride] = prev;
  }
  // anti-causal initialisation for the mirror boundary, then the recursion
  double next = (z / (z * z - 1.0)) * (prev + z * out[(long)(n - 2) * stride]);
  out[(long)(n - 1) * stride] = next;
#pragma unroll 8
  for (int k = n - 2; k >= 0; --k) {
    next = z * (next - out[k * stride]);
    out[k * stride] = next;
  }
}

// Lines of kSegMin and more are prefiltered in segments of kSeg values, one
// thread each: the recursions forget their past by |z| = 0.268 a step, so a
// thread that starts kWarm = 32 steps before its segment (after it, for the
// anti-causal one) from zero is off by |z|^32 = 5e-19 of the line's scale,
// below FP64's rounding, and the exact boundary sums need 64 terms only.  One
// thread per line (kept for short and very long lines) is a chain of 4 n
// dependent FP64 steps on n threads: at 512 lines of 512 it took 238 us for
// the columns and 247 us for the rows; the segments take 8 and 7 us.
constexpr int kSeg = 16, kWarm = 32, kSegMin = 128;
constexpr int kSegRowMax = 8192;  // longest row staged in shared memory

// the causal recursion's first value of a line of n >= kSegMin samples,
// p[0] = 6 sum_k z^k x[k] (the mirrored terms carry z^(n-1) < 1e-70)
template <class F>
__device__ __forceinline__ double bspline3_first(F&& x) {
  double s = 0.0;
#pragma unroll 16
  for (int k = 63; k >= 0; --k) s = x(k) + kZ3 * s;
  return kGain3 * s;
}

// Columns, thread (column j, segment): p in registers over the segment and
// the warm-up of the way back; the map is only read and c only written, so
// segments are independent.
__global__ void __launch_bounds__(128) spline_cols_seg_kernel(const float* __restrict__ in,
                                                              double* __restrict__ c, int N) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int s0 = blockIdx.y * kSeg;
  if (j >= N) return;
  const float* x = in + j;
  double prev = 0.0;
  int k = s0 - kWarm;
  if (k <= 0) {
    prev = bspline3_first([&](int i) { return (double)x[(size_t)i * N]; });
    k = 1;
  }
#pragma unroll 16
  for (; k < s0; ++k) prev = kGain3 * (double)x[(size_t)k * N] + kZ3 * prev;
  const double before = prev;  // p[s0 - 1]
  double p[kSeg + kWarm];
#pragma unroll
  for (int i = 0; i < kSeg + kWarm; ++i) {
    const int q = s0 + i;
    if (q > 0 && q < N) prev = kGain3 * (double)x[(size_t)q * N] + kZ3 * prev;
    p[i] = prev;  // (q = 0: prev is p[0] already; past the end: p[N-1])
  }
  double next = 0.0;
#pragma unroll
  for (int i = kSeg + kWarm - 1; i >= 0; --i) {
    const int q = s0 + i;
    if (q < N - 1) {
      next = kZ3 * (next - p[i]);
    } else if (q == N - 1) {  // the anti-causal boundary value
      next = (kZ3 / (kZ3 * kZ3 - 1.0)) * (p[i] + kZ3 * (i > 0 ? p[i - 1] : before));
    }
    if (i < kSeg && q < N) c[(size_t)q * N + j] = next;
  }
}

// Rows in place, one warp per row: the row and its causal values in shared
// memory (one spare value per kSeg, so that lanes a segment apart fall on
// different banks), segments dealt to the lanes.  A row with a value that is
// not finite becomes NaN as a whole, as the unsegmented recursions make it
// (unwrap_kernel does the same across rows).
__device__ __forceinline__ int seg_pad(int k) { return k + k / kSeg; }
__global__ void spline_rows_seg_kernel(double* __restrict__ c, int N) {
  extern __shared__ double row_s[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int row = blockIdx.x * (blockDim.x >> 5) + w;
  double* x = row_s + (size_t)w * (N + N / kSeg + 1) * 2;  // inputs, then c
  double* p = x + (N + N / kSeg + 1);
  if (row >= N) return;
  double* g = c + (size_t)row * N;
  bool bad = false;
  for (int k = lane; k < N; k += 32) {
    const double v = g[k];
    bad |= !isfinite(v);
    x[seg_pad(k)] = v;
  }
  if (__any_sync(0xffffffffu, bad)) {
    for (int k = lane; k < N; k += 32) g[k] = nan("");
    return;
  }
  __syncwarp();
  const double first = bspline3_first([&](int i) { return x[seg_pad(i)]; });
  for (int s0 = lane * kSeg; s0 < N; s0 += 32 * kSeg) {
    double prev = 0.0;
    int k = s0 - kWarm;
    if (k <= 0) {
      prev = first;
      k = 1;
    }
#pragma unroll 8
    for (; k < s0; ++k) prev = kGain3 * x[seg_pad(k)] + kZ3 * prev;
    const int e = s0 + kSeg < N ? s0 + kSeg : N;
    if (s0 == 0) p[0] = first;
#pragma unroll 8
    for (; k < e; ++k) {
      prev = kGain3 * x[seg_pad(k)] + kZ3 * prev;
      p[seg_pad(k)] = prev;
    }
  }
  __syncwarp();
  for (int s0 = lane * kSeg; s0 < N; s0 += 32 * kSeg) {
    const int e = s0 + kSeg < N ? s0 + kSeg : N;
    double next = 0.0;
    int k = e + kWarm - 1;
    if (k >= N - 1) {
      next = (kZ3 / (kZ3 * kZ3 - 1.0)) * (p[seg_pad(N - 1)] + kZ3 * p[seg_pad(N - 2)]);
      if (e == N) x[seg_pad(N - 1)] = next;
      k = N - 2;
    }
#pragma unroll 8
    for (; k >= e; --k) next = kZ3 * (next - p[seg_pad(k)]);
#pragma unroll 8
    for (; k >= s0; --k) {
      next = kZ3 * (next - p[seg_pad(k)]);
      x[seg_pad(k)] = next;
    }
  }
  __syncwarp();
  for (int k = lane; k < N; k += 32) g[k] = x[seg_pad(k)];
}

// One thread per line.  Columns first (thread j walks column j: neighbouring
// threads touch neighbouring addresses), from the float map into the FP64
// coefficients.
__global__ void spline_cols_kernel(const float* __restrict__ in, double* __restrict__ c, int N) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  bspline3_line(in + j, c + j, N, N);
}

// Then rows, in place.
__global__ void spline_rows_kernel(double* __restrict__ c, int N) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  bspline3_line(c + (size_t)i * N, c + (size_t)i * N, N, 1);
}

__device__ __forceinline__ int mirror_index(int i, int n) {
  if ((unsigned)i < (unsigned)n) return i;  // (nearly all: the remainder is a division)
  if (n == 1) return 0;
  const int p = 2 * n - 2;
  i %= p;
  if (i < 0) i += p;
  return i >= n ? p - i : i;
}

// Six times the cubic B-spline weights of the taps floor(u) - 1 .. floor(u) + 2
// for t = u - floor(u): the sixths of both axes are one product at the end.
__device__ __forceinline__ void bspline3_weights6(double t, double w[4]) {
  const double s = 1.0 - t;
  w[0] = s * s * s;
  w[1] = (3.0 * t - 6.0) * t * t + 4.0;
  w[2] = ((3.0 - 3.0 * t) * t + 3.0) * t + 1.0;
  w[3] = t * t * t;
}

__device__ __forceinline__ double bspline3_at(const double* __restrict__ c, int N, double y, double x) {
  const double fy = floor(y), fx = floor(x);
  double wy[4], wx[4];
  bspline3_weights6(y - fy, wy);
  bspline3_weights6(x - fx, wx);
  const int iy = (int)fy - 1, ix = (int)fx - 1;
  int cols[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) cols[b] = mirror_index(ix + b, N);
  double acc = 0.0;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const double* row = c + (size_t)mirror_index(iy + a, N) * N;
    double ra = 0.0;
#pragma unroll
    for (int b = 0; b < 4; ++b) ra += wx[b] * row[cols[b]];
    acc += wy[a] * ra;
  }
  return acc * (1.0 / 36.0);
}

// One block per radius r_in + blockIdx.x: the samples at the `cols` angles
// phi_k = 2 pi k / cols (wrapping.py:46-51 order of operations), written to
// `unwrapped` (row-major, radius by angle) if given, and their mean to `mean`.
// A map with a value that is not finite unwraps to NaN everywhere (the
// prefilter's recursions carry it along every line); after the segmented
// prefilter (`rows_poisoned`) such a value shows as a row of NaN, found here
// in the first column.  Bound by FP64 instructions and their latency: the
// weights' divisions are one product a sample, indices inside the map skip the
// mirror's remainder, and 16 warps a radius keep about three samples a thread
// (512^2, 1608 angles: 19 us with those divisions and 8 warps, now 12.5).
__global__ void unwrap_kernel(const double* __restrict__ c, int N, int r_in, int cols, double cy,
                              double cx, float* __restrict__ unwrapped, float* __restrict__ mean,
                              int rows_poisoned) {
  constexpr double kPi = 3.141592653589793238462643383279502884;
  const int row = blockIdx.x;
  const double r = (double)(r_in + row);
  double part = 0.0;
  if (rows_poisoned) {
    bool bad = false;
    for (int k = threadIdx.x; k < N; k += blockDim.x) bad |= !isfinite(c[(size_t)k * N]);
    if (__syncthreads_or(bad)) {
      for (int k = threadIdx.x; k < cols; k += blockDim.x)
        if (unwrapped) unwrapped[(size_t)row * cols + k] = nanf("");
      if (threadIdx.x == 0 && mean) mean[row] = nanf("");
      return;
    }
  }
  for (int k = threadIdx.x; k < cols; k += blockDim.x) {
    const double phi = (double)k * 2.0 * kPi / (double)cols;
    double sn, cs;
    sincos(phi, &sn, &cs);
    const float v = (float)bspline3_at(c, N, r * sn + cy, r * cs + cx);
    if (unwrapped) unwrapped[(size_t)row * cols + k] = v;
    part += (double)v;
  }
  __shared__ double red[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
  __syncthreads();
  if (threadIdx.x < 32) {
    double s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0 && mean) mean[row] = (float)(s / (double)cols);
  }
}

}  // namespace sp

using namespace sp;

extern "C" int sp_unwrap(const float* in_dev, int N, int r_in, int r_out, double cy, double cx,
                         int columns, double* work_dev, float* unwrapped_dev, float* mean_dev,
                         sp_stream_t stream) {
  SP_CHECK(in_dev && work_dev, SP_ERR_INVALID, "sp_unwrap: input and work pointers are required");
  SP_CHECK(unwrapped_dev || mean_dev, SP_ERR_INVALID, "sp_unwrap: no output requested");
  SP_CHECK(N >= 1 && N <= 65536, SP_ERR_SIZE, "sp_unwrap: N=%d", N);
  SP_CHECK(r_in >= 0 && r_out > r_in, SP_ERR_INVALID, "sp_unwrap: radii %d..%d", r_in, r_out);
  if (columns <= 0) columns = (int)(2.0 * 3.141592653589793 * (double)r_out);
  SP_CHECK(columns >= 1, SP_ERR_INVALID, "sp_unwrap: %d columns", columns);
  // every sample must fall inside the map (the prtfq / rftfq grid, centre N/2
  // and radii below N/2, always does); nothing outside is interpolated
  const double rmax = (double)(r_out - 1);
  SP_CHECK(cy - rmax >= 0.0 && cy + rmax <= (double)(N - 1) && cx - rmax >= 0.0 &&
               cx + rmax <= (double)(N - 1),
           SP_ERR_INVALID, "sp_unwrap: radius %d about (%g, %g) leaves the %d x %d map", r_out - 1,
           cy, cx, N, N);
  cudaStream_t st = as_stream(stream);
  const int tb = 128, nb = (N + tb - 1) / tb;
  const bool seg = N >= kSegMin && N <= kSegRowMax;
  if (seg)
    spline_cols_seg_kernel<<<dim3(nb, (N + kSeg - 1) / kSeg), tb, 0, st>>>(in_dev, work_dev, N);
  else
    spline_cols_kernel<<<nb, tb, 0, st>>>(in_dev, work_dev, N);
  SP_CUDA_TRY(cudaGetLastError());
  if (seg) {
    const auto bytes = [](int n) { return (size_t)(n + n / kSeg + 1) * 2 * sizeof(double); };
    const size_t row_bytes = bytes(N);
    const int warps = row_bytes * 4 <= 64 * 1024 ? 4 : 1;  // rows per CTA
    // (the limit is the process's: the largest call's, whatever this one needs, so
    // that threads with other sizes do not lower it before this launch)
    SP_CUDA_TRY(cudaFuncSetAttribute(spline_rows_seg_kernel,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)bytes(kSegRowMax)));
    spline_rows_seg_kernel<<<(N + warps - 1) / warps, 32 * warps, row_bytes * warps, st>>>(work_dev, N);
  } else {
    spline_rows_kernel<<<nb, tb, 0, st>>>(work_dev, N);
  }
  SP_CUDA_TRY(cudaGetLastError());
  unwrap_kernel<<<r_out - r_in, 512, 0, st>>>(work_dev, N, r_in, columns, cy, cx, unwrapped_dev,
                                               mean_dev, seg ? 1 : 0);
  SP_CUDA_TRY(cudaGetLastError());
  return SP_OK;
}
