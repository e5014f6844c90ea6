// Subpixel registration of frames to a reference frame and their alignment:
// the "align global phase and subpixel shift to trial 0, then average" step
// of the batched-trials workload.  The reference aligns frames only by whole
// pixels (conditioning.align_frames, speckle/conditioning.py:316-430, with
// crosscorr.alignment_coordinates, speckle/crosscorr.py:526-568); this keeps
// its cross-correlation convention and answers at integer shifts and refines
// the peak by the single-step upsampled DFT of Guizar-Sicairos, Thurman &
// Fienup ("Efficient subpixel image registration algorithms", Opt. Lett. 33,
// 156-158, 2008):
//   1. F_f = FFT2(frame f embedded at the corner of N x N), R = the reference's
//   2. X_f = F_f conj(R); c_f = IFFT2(X_f); d0 = the argmax of the fftshifted
//      |c_f| (ties to the first index, as numpy's argmax), a signed shift
//   3. the cross-correlation upsampled by U on an M x M grid (M = ceil(1.5 U))
//      centred on d0: c(d0 + (p - h, q - h)/U) for p, q < M, h = M/2, as two
//      matrix products of X_f' = X_f exp(2 pi i k.d0/N) (signed frequencies)
//      with W[k][q] = exp(2 pi i k (q - h)/(U N)) -- rows first, then columns
//   4. d = d0 + (p* - h, q* - h)/U at the largest |c|, theta = arg c there
//   5. aligned_f = IFFT2(F_f exp(2 pi i k.d/N) exp(-i theta)), cropped: the
//      frame moved by d (aligned_f(y) = frame_f(y + d)) and rotated onto the
//      reference's global phase
// Every phase argument is an integer numerator over N or U N, reduced exactly
// in integers before the (float) sincospi.
#include <algorithm>
#include <cmath>

#include "sp_register.cuh"

namespace sp {

static inline int upsampled_points(int U) { return (3 * U + 1) / 2; }  // ceil(1.5 U)

// the signed coarse shift d0 of frame f from its argmax key
__device__ __forceinline__ int2 coarse_shift(unsigned long long key, int N) {
  const uint32_t sidx = 0xffffffffu - (uint32_t)(key & 0xffffffffu);
  return make_int2((int)(sidx / N) - N / 2, (int)(sidx % N) - N / 2);
}

// W[k][q] = exp(2 pi i k_s (q - h) / (U N)), k < N, q < M
__global__ void reg_kernel_table(float2* __restrict__ W, int N, int U, int M) {
  const int h = M / 2;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N * M; i += gridDim.x * blockDim.x) {
    const int k = i / M, q = i - k * M;
    W[i] = turn((long long)signed_freq(k, N) * (q - h), (long long)U * N);
  }
}

// The upsampled DFT is two complex matrix products, C[i][q] = sum_k A[i][k]
// B[k][q], added up over k in order in FP32 (the peak search compares values
// that differ in the last digits, so the order is part of the result):
//   rows: A = X_f' = F_f conj(R) exp(2 pi i k.d0/N)  (i = ky, k = kx), B = W,
//         C = T1_f, stored
//   cols: A = W^T (i = p, k = ky), B = T1_f; C = the correlation on the fine
//         grid, only its largest |c| kept (ties to the first index p M + q)
// Bound by the FMA pipes: four FMAs per term, as two packed FP32x2
// instructions per term on the real or imaginary parts of two rows i,
//   re += (-a.y b.y), then += a.x b.x;   im += a.y b.x, then += a.x b.y
// (each lane in the order of the scalar form).  A CTA takes 4 R rows and all M
// columns, a warp R rows, whose A values are broadcasts of (re, re, im, im) of
// a row pair from shared memory, and a lane the columns lane + 32 m, m < MQ.
// Shared memory is the next limit (pairing re with im instead needs twice the A
// loads and ran at its bandwidth: 245 us), so a warp keeps R as large as the
// registers allow; four 128-thread CTAs per SM.  Staged one chunk ahead of the
// products, since four CTAs alone did not cover the loads.
// 128 frames, N = 256, M = 96: rows 154 us (178 staged between two barriers,
// FMA pipes 62% busy; 557 with scalar FMAs on 4 x 3 tiles), columns 70 us (the
// loads of A are few there: 69, 234).  The whole call at U = 10, 42, 64, 85,
// 100, 170: 210, 266, 342, 441, 546, 919 us; staged between barriers 254, 302,
// 365, 450, 550, 914.
constexpr int kRegK = 16, kRegThreads = 128, kRegWarps = kRegThreads / 32;

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{.reg .b64 ra, rb, rc, rr;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
      "fma.rn.ftz.f32x2 rr, ra, rb, rc;\n\tmov.b64 {%0, %1}, rr;}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}

// row pairs of a warp for MQ column groups, four accumulator registers each: 16 to
// 64 for up to four groups, 40 to 64 for more
__host__ __device__ constexpr int reg_pairs(int MQ) { return MQ <= 4 ? 4 : 2; }
__host__ __device__ constexpr int reg_tile_rows(int MQ) { return kRegWarps * 2 * reg_pairs(MQ); }

// re[j][m], im[j][m]: the two rows of the warp's pair j, column lane + 32 m.
// `as` holds [pair of the tile][k], `bs` [k][M], two chunks of kRegK each: while
// one is multiplied the next one's B is copied and its A values travel through
// the threads' registers (Src::fetch, then Src::make).  Thread i always stages
// position i % kRegK of the chunk, of pairs i / kRegK + 8 u.
template <int MQ, class Src>
__device__ __forceinline__ void reg_product(float2 (&re)[reg_pairs(MQ)][MQ],
                                            float2 (&im)[reg_pairs(MQ)][MQ], const Src& src, int K, int M,
                                            float4* as, float2* bs) {
  constexpr int R = reg_pairs(MQ), PAIRS = kRegWarps * R, STEP = kRegThreads / kRegK;
  constexpr int U = PAIRS / STEP;
  static_assert(U * STEP == PAIRS, "whole pairs per thread");
  const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int kt = threadIdx.x % kRegK, pt = threadIdx.x / kRegK;
#pragma unroll
  for (int j = 0; j < R; ++j)
#pragma unroll
    for (int m = 0; m < MQ; ++m) re[j][m] = im[j][m] = make_float2(0.f, 0.f);
  typename Src::Raw raw[U];
  auto fetch = [&](int k0) {
    // rows of B are contiguous; k0 and the chunk's length are multiples of 8, so
    // they are whole 16-byte pieces
    const int nk = K - k0 < kRegK ? K - k0 : kRegK;
    float2* dst = bs + (k0 / kRegK % 2) * kRegK * M;
    for (int i = threadIdx.x; i < nk * M / 2; i += kRegThreads)
      cp_async<16>(dst + 2 * i, src.b + (size_t)k0 * M + 2 * i);
    if (kt < nk) {
#pragma unroll
      for (int u = 0; u < U; ++u) raw[u] = src.fetch(pt + u * STEP, k0 + kt);
    }
  };
  auto put = [&](int k0) {
    if (k0 + kt < K) src.make(raw, as + (k0 / kRegK % 2) * PAIRS * kRegK + kt, pt, k0 + kt);
    cp_async_wait_all();
    __syncthreads();
  };
  __syncthreads();  // (what the source prepared)
  fetch(0);
  put(0);
  for (int k0 = 0; k0 < K; k0 += kRegK) {
    const bool more = k0 + kRegK < K;
    if (more) fetch(k0 + kRegK);
    const int nk = K - k0 < kRegK ? K - k0 : kRegK;
    const float4* ac = as + (k0 / kRegK % 2) * PAIRS * kRegK;
    const float2* bc = bs + (k0 / kRegK % 2) * kRegK * M;
#pragma unroll(MQ == 4 ? 2 : 4)  // (MQ = 4 spills at 4; the wider ones, with half the pairs, don't)
    for (int kk = 0; kk < nk; ++kk) {
      float4 a[R];
#pragma unroll
      for (int j = 0; j < R; ++j) a[j] = ac[(w * R + j) * kRegK + kk];
#pragma unroll
      for (int m = 0; m < MQ; ++m) {
        const int q = lane + 32 * m;
        const float2 b = bc[kk * M + (q < M ? q : 0)];
        const float2 bx = make_float2(b.x, b.x), by = make_float2(b.y, b.y);
        const float2 ny = make_float2(-b.y, -b.y);
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const float2 ar = make_float2(a[j].x, a[j].y), ai = make_float2(a[j].z, a[j].w);
          re[j][m] = fma2(ar, bx, fma2(ai, ny, re[j][m]));
          im[j][m] = fma2(ar, by, fma2(ai, bx, im[j][m]));
        }
      }
    }
    if (more) put(k0 + kRegK);  // (the other half: its last readers passed the barrier before)
  }
}

// The modulation's products with their contraction spelled out: left to the
// compiler it depends on the code around them, and frames whose two best grid
// points agree to the last bits then move to the other one.
__device__ __forceinline__ float2 reg_cmul(float2 a, float2 w) {
  return make_float2(fmaf(a.x, w.x, -__fmul_rn(a.y, w.y)), fmaf(a.x, w.y, __fmul_rn(a.y, w.x)));
}
__device__ __forceinline__ float2 reg_cmulc(float2 a, float2 w) {  // a conj(w)
  return make_float2(fmaf(a.x, w.x, __fmul_rn(a.y, w.y)), fmaf(a.y, w.x, -__fmul_rn(a.x, w.y)));
}

// A = X_f' of one frame's rows ky0 ..: the modulation is separable, the row
// factors exp(2 pi i ky d0y/N) made once, the column factors once per position.
struct RegRowsSrc {
  const float2 *F, *R, *b;
  const float2* rowf;
  int N, ky0, d0x;
  struct Raw {
    float2 f0, r0, f1, r1;
  };
  __device__ __forceinline__ Raw fetch(int p, int k) const {
    const float2 z = make_float2(0.f, 0.f);
    if (ky0 + 2 * p >= N) return {z, z, z, z};  // (N is even)
    const size_t idx = (size_t)(ky0 + 2 * p) * N + k;
    return {F[idx], R[idx], F[idx + N], R[idx + N]};
  }
  template <int U>
  __device__ __forceinline__ void make(const Raw (&raw)[U], float4* as, int pt, int k) const {
    const float2 col = turn_pow2(signed_freq(k, N) * d0x, N);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int p = pt + u * (kRegThreads / kRegK);
      const float2 x = reg_cmul(reg_cmul(reg_cmulc(raw[u].f0, raw[u].r0), rowf[2 * p]), col);
      const float2 y = reg_cmul(reg_cmul(reg_cmulc(raw[u].f1, raw[u].r1), rowf[2 * p + 1]), col);
      as[p * kRegK] = make_float4(x.x, y.x, x.y, y.y);
    }
  }
};

template <int MQ>
__global__ void __launch_bounds__(kRegThreads, 4) reg_upsample_rows_kernel(
    const float2* __restrict__ F, const float2* __restrict__ Rf, const float2* __restrict__ W,
    const unsigned long long* __restrict__ best, float2* __restrict__ T1, int N, int M) {
  constexpr int R = reg_pairs(MQ), ROWS = reg_tile_rows(MQ);
  extern __shared__ float4 reg_sm[];
  float2* bs = reinterpret_cast<float2*>(reg_sm + ROWS * kRegK);
  __shared__ float2 rowf[ROWS];
  const int f = blockIdx.y, ky0 = blockIdx.x * ROWS;
  const int2 d0 = coarse_shift(best[f], N);
  for (int r = threadIdx.x; r < ROWS; r += kRegThreads)
    rowf[r] = turn_pow2(signed_freq(ky0 + r, N) * d0.x, N);
  float2 re[R][MQ], im[R][MQ];
  const RegRowsSrc src{F + (size_t)f * N * N, Rf, W, rowf, N, ky0, d0.y};
  reg_product<MQ>(re, im, src, N, M, reg_sm, bs);
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const int ky = ky0 + 2 * ((threadIdx.x / 32) * R + j);
#pragma unroll
    for (int m = 0; m < MQ; ++m) {
      const int q = threadIdx.x % 32 + 32 * m;
      float2* t = T1 + ((size_t)f * N + ky) * M + q;
      if (ky < N && q < M) {  // (N is even)
        t[0] = make_float2(re[j][m].x, im[j][m].x);
        t[M] = make_float2(re[j][m].y, im[j][m].y);
      }
    }
  }
}

struct RegColsSrc {
  const float2 *W, *b;
  int M, p0;
  struct Raw {
    float2 w0, w1;
  };
  __device__ __forceinline__ Raw fetch(int p, int k) const {
    const float2 zero = make_float2(0.f, 0.f);
    const float2* w = W + (size_t)k * M + p0 + 2 * p;
    return {p0 + 2 * p < M ? w[0] : zero, p0 + 2 * p + 1 < M ? w[1] : zero};
  }
  template <int U>
  __device__ __forceinline__ void make(const Raw (&raw)[U], float4* as, int pt, int) const {
#pragma unroll
    for (int u = 0; u < U; ++u)
      as[(pt + u * (kRegThreads / kRegK)) * kRegK] =
          make_float4(raw[u].w0.x, raw[u].w1.x, raw[u].w0.y, raw[u].w1.y);
  }
};

template <int MQ>
__global__ void __launch_bounds__(kRegThreads, 4) reg_upsample_cols_kernel(
    const float2* __restrict__ T1, const float2* __restrict__ W, int N, int M,
    unsigned long long* __restrict__ best_up) {
  constexpr int R = reg_pairs(MQ), ROWS = reg_tile_rows(MQ);
  extern __shared__ float4 reg_sm[];
  float2* bs = reinterpret_cast<float2*>(reg_sm + ROWS * kRegK);
  const int f = blockIdx.y, p0 = blockIdx.x * ROWS;
  float2 re[R][MQ], im[R][MQ];
  const RegColsSrc src{W, T1 + (size_t)f * N * M, M, p0};
  reg_product<MQ>(re, im, src, N, M, reg_sm, bs);
  unsigned long long mine = 0;
  auto take = [&](int p, int q, float x, float y) {
    if (p >= M || q >= M) return;
    const float mag = sqrtf(fmaf(x, x, y * y));  // (spelled out: near-ties turn on its last bit)
    const unsigned long long key =
        ((unsigned long long)__float_as_uint(mag) << 32) | (0xffffffffu - (uint32_t)(p * M + q));
    mine = key > mine ? key : mine;
  };
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const int p = p0 + 2 * ((threadIdx.x / 32) * R + j);
#pragma unroll
    for (int m = 0; m < MQ; ++m) {
      const int q = threadIdx.x % 32 + 32 * m;
      take(p, q, re[j][m].x, im[j][m].x);
      take(p + 1, q, re[j][m].y, im[j][m].y);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, mine, o);
    mine = other > mine ? other : mine;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(&best_up[f], mine);
}

template <int MQ>
static cudaError_t reg_upsample(const RegArgs& a, int N, unsigned long long* best_up, cudaStream_t st) {
  constexpr int rows = reg_tile_rows(MQ);
  const auto bytes = [](int M) {
    return (int)(sizeof(float4) * rows * kRegK + sizeof(float2) * 2 * (size_t)kRegK * M);
  };
  // (the limit is the process's: that of the instantiation's largest M, whatever
  // this call's is, so that threads with other sizes do not lower it between this
  // and the launch)
  const int smem = bytes(a.M), most = bytes(32 * MQ);
  cudaError_t e = cudaFuncSetAttribute(reg_upsample_rows_kernel<MQ>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(reg_upsample_cols_kernel<MQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (e != cudaSuccess) return e;
  reg_upsample_rows_kernel<MQ><<<dim3((N + rows - 1) / rows, a.n), kRegThreads, smem, st>>>(
      a.F, a.Rf, a.W, a.best, a.X, N, a.M);
  reg_upsample_cols_kernel<MQ><<<dim3((a.M + rows - 1) / rows, a.n), kRegThreads, smem, st>>>(
      a.X, a.W, N, a.M, best_up);
  return cudaGetLastError();
}

// Per frame (one warp each): the refined shift d = d0 + (p* - h, q* - h)/U
// (as the integer numerators d U), the phase of c at the peak (recomputed in
// FP64 from T1), and the result record shifts[f] = (dy, dx, theta).  `cs`, the
// turn e^(-i theta) that the shift applies, goes where best_up[f] was.
__global__ void reg_finish_kernel(const float2* __restrict__ T1, const float2* __restrict__ W,
                                  const unsigned long long* __restrict__ best,
                                  unsigned long long* best_up, int n, int N, int U, int M,
                                  int2* __restrict__ num, double* __restrict__ shifts) {
  const int f = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  const int lane = threadIdx.x % 32;
  if (f >= n) return;
  const int2 d0 = coarse_shift(best[f], N);
  const uint32_t idx = 0xffffffffu - (uint32_t)(best_up[f] & 0xffffffffu);
  float2* cs = reinterpret_cast<float2*>(best_up);
  const int p = (int)(idx / M), q = (int)(idx % M), h = M / 2;
  const float2* t1 = T1 + (long long)f * N * M;
  double re = 0.0, im = 0.0;
  for (int ky = lane; ky < N; ky += 32) {
    const float2 w = W[(long long)ky * M + p], t = t1[(long long)ky * M + q];
    re += (double)w.x * t.x - (double)w.y * t.y;
    im += (double)w.x * t.y + (double)w.y * t.x;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    re += __shfl_xor_sync(0xffffffffu, re, o);
    im += __shfl_xor_sync(0xffffffffu, im, o);
  }
  if (lane == 0) {
    const int ny = d0.x * U + (p - h), nx = d0.y * U + (q - h);
    num[f] = make_int2(ny, nx);
    shifts[3 * f] = (double)ny / U;
    shifts[3 * f + 1] = (double)nx / U;
    const double th = atan2(im, re);
    shifts[3 * f + 2] = th;
    cs[f] = make_float2((float)cos(th), (float)-sin(th));  // (after the shuffles: best_up[f] is read)
  }
}

cudaError_t reg_lines(int N, int which, const RegArgs& a, cudaStream_t st) {
  const float2* tw = nullptr;
  cudaError_t e = twiddles(&tw);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 148;
  e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  switch (N) {
    case 8: return reg_lines_n8(which, a, tw, sms, st);
    case 16: return reg_lines_n16(which, a, tw, sms, st);
    case 32: return reg_lines_n32(which, a, tw, sms, st);
    case 64: return reg_lines_n64(which, a, tw, sms, st);
    case 128: return reg_lines_n128(which, a, tw, sms, st);
    case 256: return reg_lines_n256(which, a, tw, sms, st);
    case 512: return reg_lines_n512(which, a, tw, sms, st);
    case 1024: return reg_lines_n1024(which, a, tw, sms, st);
    case 2048: return reg_lines_n2048(which, a, tw, sms, st);
    case 4096: return reg_lines_n4096(which, a, tw, sms, st);
    default: return cudaErrorInvalidValue;
  }
}

struct RegLayout {
  size_t F, X, W, best, best_up, num, total;
};
static RegLayout reg_layout(int n, int N, int U) {
  const int M = upsampled_points(U);
  auto al = [](size_t x) { return (x + 255) / 256 * 256; };
  RegLayout L;
  const size_t NN = (size_t)N * N;
  L.F = 0;
  L.X = L.F + al(sizeof(float2) * (n + 1) * NN);  // frames and (last) the reference
  L.W = L.X + al(sizeof(float2) * (size_t)n * N * (size_t)(N > M ? N : M));
  L.best = L.W + al(sizeof(float2) * (size_t)N * M);
  L.best_up = L.best + al(sizeof(unsigned long long) * n);
  L.num = L.best_up + al(sizeof(unsigned long long) * n);
  L.total = L.num + al(sizeof(int2) * n);
  return L;
}

}  // namespace sp

using namespace sp;

extern "C" int sp_register_workspace_size(int n_frames, int N, int upsample, size_t* bytes) {
  SP_CHECK(bytes && n_frames > 0 && upsample >= 1 && upsample <= 170, SP_ERR_INVALID,
           "sp_register_workspace_size: bad argument");
  SP_CHECK(is_pow2(N) && N >= kMinN && N <= kMaxN, SP_ERR_SIZE, "sp_register: N=%d", N);
  *bytes = reg_layout(n_frames, N, upsample).total;
  return SP_OK;
}

extern "C" int sp_register_subpixel(const void* frames_dev, int n_frames, int rows, int cols,
                                    const void* ref_dev, int N, int upsample, void* work_dev,
                                    size_t work_bytes, double* shifts_dev, void* out_dev,
                                    sp_stream_t stream) {
  SP_CHECK(frames_dev && ref_dev && work_dev && shifts_dev && n_frames > 0, SP_ERR_INVALID,
           "sp_register_subpixel: bad argument");
  SP_CHECK(is_pow2(N) && N >= kMinN && N <= kMaxN, SP_ERR_SIZE, "sp_register_subpixel: N=%d", N);
  SP_CHECK(rows > 0 && cols > 0 && rows <= N && cols <= N, SP_ERR_INVALID,
           "sp_register_subpixel: frames of %d x %d do not fit N=%d", rows, cols, N);
  SP_CHECK(upsample >= 1 && upsample <= 170, SP_ERR_INVALID,
           "sp_register_subpixel: upsample=%d not in [1, 170]", upsample);
  SP_CHECK(n_frames <= 65535, SP_ERR_SIZE, "sp_register_subpixel: at most 65535 frames");
  const RegLayout L = reg_layout(n_frames, N, upsample);
  SP_CHECK(work_bytes >= L.total, SP_ERR_WORKSPACE, "sp_register_subpixel: %zu bytes given, %zu needed",
           work_bytes, L.total);
  cudaStream_t st = as_stream(stream);
  char* ws = static_cast<char*>(work_dev);
  const int M = upsampled_points(upsample);
  auto* best_up = reinterpret_cast<unsigned long long*>(ws + L.best_up);
  float2* F = reinterpret_cast<float2*>(ws + L.F);
  float2* W = reinterpret_cast<float2*>(ws + L.W);
  int2* num = reinterpret_cast<int2*>(ws + L.num);
  const RegArgs a{(const float2*)frames_dev, (const float2*)ref_dev, F, F + (size_t)n_frames * N * N,
                  reinterpret_cast<float2*>(ws + L.X), W,
                  reinterpret_cast<unsigned long long*>(ws + L.best), num,
                  reinterpret_cast<const float2*>(best_up), (float2*)out_dev, n_frames, rows, cols,
                  upsample, M};
  SP_CUDA_TRY(cudaMemsetAsync(a.best, 0, sizeof(unsigned long long) * n_frames, st));
  SP_CUDA_TRY(cudaMemsetAsync(best_up, 0, sizeof(unsigned long long) * n_frames, st));
  reg_kernel_table<<<std::min((N * M + 255) / 256, 148 * 16), 256, 0, st>>>(W, N, upsample, M);
  SP_CUDA_TRY(cudaGetLastError());
  for (int which : {kRegEmbed, kRegColsRef, kRegCols, kRegCross, kRegPeak})
    SP_CUDA_TRY(reg_lines(N, which, a, st));
  switch ((M + 31) / 32) {
    case 1: SP_CUDA_TRY(reg_upsample<1>(a, N, best_up, st)); break;
    case 2: SP_CUDA_TRY(reg_upsample<2>(a, N, best_up, st)); break;
    case 3: SP_CUDA_TRY(reg_upsample<3>(a, N, best_up, st)); break;
    case 4: SP_CUDA_TRY(reg_upsample<4>(a, N, best_up, st)); break;
    case 5: SP_CUDA_TRY(reg_upsample<5>(a, N, best_up, st)); break;
    case 6: SP_CUDA_TRY(reg_upsample<6>(a, N, best_up, st)); break;
    case 7: SP_CUDA_TRY(reg_upsample<7>(a, N, best_up, st)); break;
    default: SP_CUDA_TRY(reg_upsample<8>(a, N, best_up, st)); break;
  }
  reg_finish_kernel<<<(n_frames + 3) / 4, 128, 0, st>>>(a.X, W, a.best, best_up, n_frames, N, upsample,
                                                        M, num, shifts_dev);
  SP_CUDA_TRY(cudaGetLastError());
  if (out_dev) {
    SP_CUDA_TRY(reg_lines(N, kRegShift, a, st));
    SP_CUDA_TRY(reg_lines(N, kRegCrop, a, st));
  }
  return SP_OK;
}
