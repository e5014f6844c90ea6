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
// thread each.  The recursions are linear, so a segment runs from zero first,
// and what comes in from before it (after it, for the anti-causal one) is the
// sum of the other segments' ends, each times z^kSeg per segment between:
// kFar = 12 of them, beyond which z^(kSeg kFar) = 1e-110 of a value is below
// any sample's last place (float32 spans 4e-84), however far apart the map's
// values lie.  A warm-up of 32 steps in place of the carries dropped 5e-19 of
// the line's largest value, which showed next to a value 1e15 times the others.
// One thread per line (kept for short and very long lines) is a chain of 4 n
// dependent FP64 steps on n threads: at 512 lines of 512 it took 238 us for
// the columns and 247 us for the rows; the segments take 6 and 7 us (as the warm-ups did, 7 and 6; 5% more from 4096 on).
constexpr int kSeg = 16, kFar = 12, kSegMin = 128;
constexpr int kSegMax = 8192;  // longest row staged in shared memory

constexpr double zpow(int n) { return n == 0 ? 1.0 : kZ3 * zpow(n - 1); }
constexpr double kZSeg = zpow(kSeg);

// sum_{k = 1}^{kFar} z^(kSeg (k-1)) at(k), as far as there are `n` of them
template <class F>
__device__ __forceinline__ double far_sum(int n, F&& at) {
  double s = 0.0;
  for (int k = n < kFar ? n : kFar; k >= 1; --k) s = at(k) + kZSeg * s;
  return s;
}

// What a line's length fixes: z^(n-1) and z^(length of the last segment).  The
// causal recursion's first value is that of bspline3_line,
//   6 sum_k z^k x[k] + z^(n-1) (p0[n-1] - 6 x[n-1]),
// p0 the recursion from zero (its mirrored terms; 1 - z^(2n-2) is 1 here).
struct SegLine {
  double zn1, zlast;
};

// Columns: a CTA takes C neighbouring columns, thread (column, segment), the
// segment's values in registers throughout.
template <int C>
__global__ void __launch_bounds__(512) spline_cols_seg_kernel(const float* __restrict__ in,
                                                              double* __restrict__ c, int N,
                                                              SegLine line) {
  __shared__ double ends[512], heads[C * kFar];
  const int S = blockDim.x / C, s = threadIdx.x / C, tx = threadIdx.x % C;
  const int j = blockIdx.x * C + tx, col = j < N ? j : N - 1;
  const int s0 = s * kSeg, n = N - s0 < kSeg ? N - s0 : kSeg;
  const float* x = in + (size_t)s0 * N + col;
  float v[kSeg];
#pragma unroll
  for (int i = 0; i < kSeg; ++i) v[i] = i < n ? x[(size_t)i * N] : 0.f;
  double end = 0.0;
#pragma unroll
  for (int i = 0; i < kSeg; ++i)
    if (i < n) end = kGain3 * (double)v[i] + kZ3 * end;
  ends[s * C + tx] = end;
  if (s < kFar) {
    double head = 0.0;
#pragma unroll
    for (int i = kSeg - 1; i >= 0; --i) head = (double)v[i] + kZ3 * head;
    heads[s * C + tx] = head;
  }
  __syncthreads();
  double prev = 0.0;
  if (s == 0) {
    const double head = far_sum(S, [&](int k) { return heads[(k - 1) * C + tx]; });
    const double tail = ends[(S - 1) * C + tx] +
                        line.zlast * far_sum(S - 1, [&](int k) { return ends[(S - 1 - k) * C + tx]; });
    prev = kGain3 * head + line.zn1 * (tail - kGain3 * (double)in[(size_t)(N - 1) * N + col]);
    end = prev;
#pragma unroll
    for (int i = 1; i < kSeg; ++i) end = kGain3 * (double)v[i] + kZ3 * end;
    ends[tx] = end;
  }
  __syncthreads();
  if (s > 0) prev = far_sum(s, [&](int k) { return ends[(s - k) * C + tx]; });
  const double before = prev;  // p[s0 - 1]
  double p[kSeg];
#pragma unroll
  for (int i = 0; i < kSeg; ++i) {
    if (s0 + i > 0 && i < n) prev = kGain3 * (double)v[i] + kZ3 * prev;
    p[i] = prev;  // (s0 + i = 0: the first value itself)
  }
  // from the last segment's boundary value, or from `next` after the segment
  auto back = [&](double next, auto&& put) {
#pragma unroll
    for (int i = kSeg - 1; i >= 0; --i) {
      if (s == S - 1 && i == n - 1)
        next = (kZ3 / (kZ3 * kZ3 - 1.0)) * (p[i] + kZ3 * (i > 0 ? p[i > 0 ? i - 1 : 0] : before));
      else if (i < n)
        next = kZ3 * (next - p[i]);
      put(i, next);
    }
    return next;
  };
  __syncthreads();  // the causal ends are read
  ends[s * C + tx] = back(0.0, [](int, double) {});
  __syncthreads();
  back(far_sum(S - 1 - s, [&](int k) { return ends[(s + k) * C + tx]; }), [&](int i, double next) {
    if (i < n && j < N) c[(size_t)(s0 + i) * N + j] = next;
  });
}

// Rows in place, one warp per row: the row, its causal values and the segments'
// ends in shared memory (one spare value per kSeg, so that lanes a segment
// apart fall on different banks), segments dealt to the lanes.  A row with a
// value that is not finite becomes NaN as a whole, as the unsegmented
// recursions make it (unwrap_kernel does the same across rows).
__host__ __device__ constexpr int seg_pad(int k) { return k + k / kSeg; }
// doubles of shared memory for a row: inputs (then c), causal values, ends
__host__ __device__ constexpr int seg_row_doubles(int n) {
  return 2 * (seg_pad(n) + 1) + (n + kSeg - 1) / kSeg;
}
__global__ void spline_rows_seg_kernel(double* __restrict__ c, int N, SegLine line) {
  extern __shared__ double row_s[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int row = blockIdx.x * (blockDim.x >> 5) + w;
  double* x = row_s + (size_t)w * seg_row_doubles(N);
  double* p = x + seg_pad(N) + 1;
  double* ends = p + seg_pad(N) + 1;
  const int S = (N + kSeg - 1) / kSeg;
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
  for (int s = lane; s < S; s += 32) {
    const int s0 = s * kSeg, e = s0 + kSeg < N ? s0 + kSeg : N;
    double end = 0.0;
#pragma unroll 8
    for (int k = s0; k < e; ++k) end = kGain3 * x[seg_pad(k)] + kZ3 * end;
    ends[s] = end;
  }
  double first = 0.0;  // lane s: segment s's share of the head sum
  if (lane < kFar && lane < S) {
    const int s0 = lane * kSeg, e = s0 + kSeg < N ? s0 + kSeg : N;
#pragma unroll 8
    for (int k = e - 1; k >= s0; --k) first = x[seg_pad(k)] + kZ3 * first;
    for (int k = 0; k < lane; ++k) first *= kZSeg;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) first += __shfl_xor_sync(0xffffffffu, first, o);
  __syncwarp();
  if (lane == 0) {
    const double tail =
        ends[S - 1] + line.zlast * far_sum(S - 1, [&](int k) { return ends[S - 1 - k]; });
    first = kGain3 * first + line.zn1 * (tail - kGain3 * x[seg_pad(N - 1)]);
    double end = first;
#pragma unroll
    for (int k = 1; k < kSeg; ++k) end = kGain3 * x[seg_pad(k)] + kZ3 * end;
    ends[0] = end;
  }
  __syncwarp();
  for (int s = lane; s < S; s += 32) {
    const int s0 = s * kSeg, e = s0 + kSeg < N ? s0 + kSeg : N;
    double prev = s ? far_sum(s, [&](int k) { return ends[s - k]; }) : first;
    if (s == 0) p[0] = first;
#pragma unroll 8
    for (int k = s ? s0 : 1; k < e; ++k) {
      prev = kGain3 * x[seg_pad(k)] + kZ3 * prev;
      p[seg_pad(k)] = prev;
    }
  }
  __syncwarp();  // the causal ends are read, the causal values complete
  for (int s = lane; s < S; s += 32) {
    const int s0 = s * kSeg, e = s0 + kSeg < N ? s0 + kSeg : N;
    double next = 0.0;
    int k = e - 1;
    if (s == S - 1) {
      next = (kZ3 / (kZ3 * kZ3 - 1.0)) * (p[seg_pad(N - 1)] + kZ3 * p[seg_pad(N - 2)]);
      x[seg_pad(k--)] = next;
    }
#pragma unroll 8
    for (; k >= s0; --k) next = kZ3 * (next - p[seg_pad(k)]);
    ends[s] = next;
  }
  __syncwarp();
  for (int s = lane; s < S; s += 32) {
    const int s0 = s * kSeg;
    int k = s0 + kSeg - 1;
    double next;
    if (s == S - 1) {
      k = N - 2;
      next = x[seg_pad(N - 1)];
    } else {
      next = far_sum(S - 1 - s, [&](int i) { return ends[s + i]; });
    }
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
  const bool seg = N >= kSegMin && N <= kSegMax;
  const int S = (N + kSeg - 1) / kSeg;
  const SegLine line{pow(kZ3, N - 1), pow(kZ3, N - (S - 1) * kSeg)};
  if (!seg)
    spline_cols_kernel<<<nb, tb, 0, st>>>(in_dev, work_dev, N);
  else if (4 * S <= 512)
    spline_cols_seg_kernel<4><<<(N + 3) / 4, 4 * S, 0, st>>>(in_dev, work_dev, N, line);
  else if (2 * S <= 512)
    spline_cols_seg_kernel<2><<<(N + 1) / 2, 2 * S, 0, st>>>(in_dev, work_dev, N, line);
  else
    spline_cols_seg_kernel<1><<<N, S, 0, st>>>(in_dev, work_dev, N, line);
  SP_CUDA_TRY(cudaGetLastError());
  if (seg) {
    const size_t row_bytes = seg_row_doubles(N) * sizeof(double);
    const int warps = row_bytes * 4 <= 64 * 1024 ? 4 : 1;  // rows per CTA
    // (the limit is the process's: the largest call's, whatever this one needs, so
    // that threads with other sizes do not lower it before this launch)
    SP_CUDA_TRY(cudaFuncSetAttribute(spline_rows_seg_kernel,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(seg_row_doubles(kSegMax) * sizeof(double))));
    spline_rows_seg_kernel<<<(N + warps - 1) / warps, 32 * warps, row_bytes * warps, st>>>(work_dev, N,
                                                                                           line);
  } else {
    spline_rows_kernel<<<nb, tb, 0, st>>>(work_dev, N);
  }
  SP_CUDA_TRY(cudaGetLastError());
  unwrap_kernel<<<r_out - r_in, 512, 0, st>>>(work_dev, N, r_in, columns, cy, cx, unwrapped_dev,
                                               mean_dev, seg ? 1 : 0);
  SP_CUDA_TRY(cudaGetLastError());
  return SP_OK;
}
