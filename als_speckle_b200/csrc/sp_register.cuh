// Line kernels of the subpixel registration (sp_register.cu): every 2-D
// transform of the path as two lines_kernel launches whose loads and results
// do the elementwise work around it.
#pragma once
#include "sp_fft2.cuh"

namespace sp {

// N x N planes: F and Rf transforms in natural order, X the transposed half of
// a transform in flight.
struct RegArgs {
  const float2* frames;  // (n, rows, cols)
  const float2* ref;     // (rows, cols)
  float2* F;             // n planes
  float2* Rf;            // the reference's
  float2* X;             // n planes
  const float2* W;       // W[k][q], M columns
  unsigned long long* best;
  const int2* num;       // refined shifts times U
  const float2* cs;      // (cos theta, -sin theta)
  float2* out;           // (n, rows, cols)
  int n, rows, cols, U, M;
};

// which: the six line passes, in their order on the stream
enum { kRegEmbed, kRegColsRef, kRegCols, kRegCross, kRegPeak, kRegShift, kRegCrop };
cudaError_t reg_lines(int N, int which, const RegArgs& a, cudaStream_t st);

__device__ __forceinline__ int signed_freq(int k, int N) { return k >= N / 2 ? k - N : k; }

// exp(2 pi i num / N), N a power of two: the residue is a mask (two's
// complement gives the non-negative residue of a negative numerator too)
__device__ __forceinline__ float2 turn_pow2(int num, int N) {
  float s, c;
  sincospif(2.0f * (float)(num & (N - 1)) / (float)N, &s, &c);
  return make_float2(c, s);
}

// Rows of the frames (into X) and of the reference (plane n, into F's first
// plane, free until the columns are transformed), zero-padded, transposed.
struct RegEmbedOp {
  RegArgs a;
  int planes, lines;
  static constexpr int extra(int) { return 0; }
  __device__ void init(float2*) const {}
  __device__ void prepare(int, float2*) const {}
  using Line = const float2*;
  __device__ __forceinline__ Line line(int f, int r) const {
    return (f < a.n ? a.frames + (int64_t)f * a.rows * a.cols : a.ref) + (int64_t)r * a.cols;
  }
  __device__ __forceinline__ float2 load(Line l, int c, const float2*) const {
    return c < a.cols ? l[c] : make_float2(0.f, 0.f);
  }
  template <int N, class Sync>
  __device__ __forceinline__ void done(int f, int l0, int nl, const float2 (&v)[Lines<N>::E],
                                       float2* smem, int lrow, int t, const Sync& sync) const {
    float2* dst = f < a.n ? a.X + (size_t)f * N * N : a.F;
    transposed_store<N>(v, smem, lrow, t, sync, dst + l0, N, nl, N);
  }
};

// Columns (contiguous in `src`, `rows` long) of planes into `dst`, natural order.
struct RegColsOp {
  const float2* src;
  float2* dst;
  int rows, planes, lines;
  static constexpr int extra(int) { return 0; }
  __device__ void init(float2*) const {}
  __device__ void prepare(int, float2*) const {}
  using Line = const float2*;
  __device__ __forceinline__ Line line(int f, int c) const { return src + ((size_t)f * lines + c) * lines; }
  __device__ __forceinline__ float2 load(Line l, int r, const float2*) const {
    return r < rows ? l[r] : make_float2(0.f, 0.f);
  }
  template <int N, class Sync>
  __device__ __forceinline__ void done(int f, int l0, int nl, const float2 (&v)[Lines<N>::E],
                                       float2* smem, int lrow, int t, const Sync& sync) const {
    transposed_store<N>(v, smem, lrow, t, sync, dst + (size_t)f * N * N + l0, N, nl, N);
  }
};

// Rows of the cross-spectrum F conj(R), inverse, transposed into X.
struct RegCrossOp {
  RegArgs a;
  int planes, lines;
  static constexpr int extra(int) { return 0; }
  __device__ void init(float2*) const {}
  __device__ void prepare(int, float2*) const {}
  struct Line {
    const float2 *F, *R;
  };
  __device__ __forceinline__ Line line(int f, int ky) const {
    return {a.F + ((size_t)f * lines + ky) * lines, a.Rf + (size_t)ky * lines};
  }
  __device__ __forceinline__ float2 load(const Line& l, int kx, const float2*) const {
    return cmulc(l.F[kx], l.R[kx]);
  }
  template <int N, class Sync>
  __device__ __forceinline__ void done(int f, int l0, int nl, const float2 (&v)[Lines<N>::E],
                                       float2* smem, int lrow, int t, const Sync& sync) const {
    transposed_store<N>(v, smem, lrow, t, sync, a.X + (size_t)f * N * N + l0, N, nl, N);
  }
};

// Columns of the cross-correlation, inverse: the largest fftshifted |c| of each
// frame, keyed (|c| bits << 32 | ~index) so that ties go to the first index.
struct RegPeakOp {
  RegArgs a;
  int planes, lines;
  static constexpr int extra(int) { return 0; }
  __device__ void init(float2*) const {}
  __device__ void prepare(int, float2*) const {}
  using Line = const float2*;
  __device__ __forceinline__ Line line(int f, int x) const { return a.X + ((size_t)f * lines + x) * lines; }
  __device__ __forceinline__ float2 load(Line l, int ky, const float2*) const { return l[ky]; }
  template <int N, class Sync>
  __device__ __forceinline__ void done(int f, int l0, int nl, const float2 (&v)[Lines<N>::E], float2*,
                                       int lrow, int t, const Sync&) const {
    constexpr float scale = 1.0f / ((float)N * (float)N);
    unsigned long long mine = 0;
    if (lrow < nl) {
      const int sc = (l0 + lrow + N / 2) % N;
#pragma unroll
      for (int i = 0; i < Lines<N>::E; ++i) {
        const uint32_t sidx = (uint32_t)(((t + i * Lines<N>::T + N / 2) % N) * N + sc);
        const float2 c = make_float2(v[i].x * scale, v[i].y * scale);
        const float m = sqrtf(fmaf(c.x, c.x, c.y * c.y));
        const unsigned long long key =
            ((unsigned long long)__float_as_uint(m) << 32) | (0xffffffffu - sidx);
        mine = key > mine ? key : mine;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, mine, o);
      mine = other > mine ? other : mine;
    }
    if ((threadIdx.x & 31) == 0) atomicMax(&a.best[f], mine);
  }
};

// exp(2 pi i num / den) with num reduced modulo den exactly first
__device__ __forceinline__ float2 turn(long long num, long long den) {
  long long r = num % den;
  if (r < 0) r += den;
  float s, c;
  sincospif(2.0f * (float)((double)r / (double)den), &s, &c);
  return make_float2(c, s);
}

// Rows of F exp(2 pi i k.d/N) exp(-i theta), d = num / U, inverse, transposed
// into X.  The ramp is a row factor exp(2 pi i ky dy/N - i theta) times a column
// factor exp(2 pi i kx dx/N), made once per line and once per plane, so an
// element takes two products (106 us for 128 planes of 256^2 as an elementwise
// pass with a sincospi, the shift's divisions and FP64 sin and cos of theta at
// every element, 64 us with the ramp composed of table entries in this kernel,
// now 29 us with the transform).
struct RegShiftOp {
  RegArgs a;
  int planes, lines;
  static constexpr int extra(int N) { return N; }  // column factors
  __device__ void init(float2*) const {}
  __device__ void prepare(int f, float2* ex) const {
    __syncthreads();  // the previous plane's loads are done
    const int nx = a.num[f].y;
    for (int k = threadIdx.x; k < lines; k += kThreads)
      ex[k] = turn((long long)signed_freq(k, lines) * nx, (long long)a.U * lines);
    __syncthreads();
  }
  struct Line {
    const float2* F;
    float2 w;
  };
  __device__ __forceinline__ Line line(int f, int ky) const {
    return {a.F + ((size_t)f * lines + ky) * lines,
            cmul(turn((long long)signed_freq(ky, lines) * a.num[f].x, (long long)a.U * lines), a.cs[f])};
  }
  __device__ __forceinline__ float2 load(const Line& l, int kx, const float2* ex) const {
    return cmul(l.F[kx], cmul(l.w, ex[kx]));
  }
  template <int N, class Sync>
  __device__ __forceinline__ void done(int f, int l0, int nl, const float2 (&v)[Lines<N>::E],
                                       float2* smem, int lrow, int t, const Sync& sync) const {
    transposed_store<N>(v, smem, lrow, t, sync, a.X + (size_t)f * N * N + l0, N, nl, N);
  }
};

// Columns x < cols, inverse, scaled: the frames' own pixels.
struct RegCropOp {
  RegArgs a;
  int N_, planes, lines;  // lines: cols
  static constexpr int extra(int) { return 0; }
  __device__ void init(float2*) const {}
  __device__ void prepare(int, float2*) const {}
  using Line = const float2*;
  __device__ __forceinline__ Line line(int f, int x) const { return a.X + ((size_t)f * N_ + x) * N_; }
  __device__ __forceinline__ float2 load(Line l, int ky, const float2*) const { return l[ky]; }
  template <int N, class Sync>
  __device__ __forceinline__ void done(int f, int l0, int nl, const float2 (&v)[Lines<N>::E],
                                       float2* smem, int lrow, int t, const Sync& sync) const {
    constexpr float scale = 1.0f / ((float)N * (float)N);
    float2 u[Lines<N>::E];
#pragma unroll
    for (int i = 0; i < Lines<N>::E; ++i) u[i] = make_float2(v[i].x * scale, v[i].y * scale);
    transposed_store<N>(u, smem, lrow, t, sync, a.out + (size_t)f * a.rows * a.cols + l0, a.cols, nl,
                        a.rows);
  }
};

template <int N>
cudaError_t reg_lines_t(int which, const RegArgs& a, const float2* tw, int n_sms, cudaStream_t st) {
  switch (which) {
    case kRegEmbed: return launch_lines<N, -1>(RegEmbedOp{a, a.n + 1, a.rows}, tw, n_sms, st);
    case kRegColsRef: return launch_lines<N, -1>(RegColsOp{a.F, a.Rf, a.rows, 1, N}, tw, n_sms, st);
    case kRegCols: return launch_lines<N, -1>(RegColsOp{a.X, a.F, a.rows, a.n, N}, tw, n_sms, st);
    case kRegCross: return launch_lines<N, +1>(RegCrossOp{a, a.n, N}, tw, n_sms, st);
    case kRegPeak: return launch_lines<N, +1>(RegPeakOp{a, a.n, N}, tw, n_sms, st);
    case kRegShift: return launch_lines<N, +1>(RegShiftOp{a, a.n, N}, tw, n_sms, st);
    default: return launch_lines<N, +1>(RegCropOp{a, N, a.n, a.cols}, tw, n_sms, st);
  }
}

#define SP_DECLARE_REG(N)                                                                  \
  cudaError_t reg_lines_n##N(int which, const RegArgs& a, const float2* tw, int n_sms, cudaStream_t st);
SP_DECLARE_REG(8)
SP_DECLARE_REG(16)
SP_DECLARE_REG(32)
SP_DECLARE_REG(64)
SP_DECLARE_REG(128)
SP_DECLARE_REG(256)
SP_DECLARE_REG(512)
SP_DECLARE_REG(1024)
SP_DECLARE_REG(2048)
SP_DECLARE_REG(4096)

#define SP_DEFINE_REG(N)                                                                    \
  cudaError_t reg_lines_n##N(int which, const RegArgs& a, const float2* tw, int n_sms, cudaStream_t st) { \
    return reg_lines_t<N>(which, a, tw, n_sms, st);                                        \
  }

}  // namespace sp
