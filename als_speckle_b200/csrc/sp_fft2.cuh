// Standalone batched 2-D FFT (sp_fft2) on the same Stockham line transform as
// the engine: a row kernel and a column kernel per size, E = min(16, N)
// values per thread.  Replaces pyfft's Plan.execute (phasing.py:1074-1075).
#pragma once
#include "sp_common.cuh"
#include "sp_engine_kernels.cuh"

namespace sp {

template <int N, int DIR>
__global__ void __launch_bounds__(kThreads) fft_rows_kernel(const float2* in,
                                                            float2* out, int batch,
                                                            const float2* __restrict__ tw_all) {
  constexpr int E = (N < 16 ? N : 16);
  constexpr int T = N / E;
  constexpr int L = lines_per_item(N, E);
  constexpr int SH = pad_shift(E);
  using Sync = typename std::conditional<(T <= 32), WarpSync, BlockSync>::type;
  extern __shared__ float2 smem[];
  float2* tw = smem + item_smem_elems(N, E);
  build_stage_twiddles<N, E>(tw, tw_all + N);
  __syncthreads();
  const int tid = threadIdx.x;
  const int lrow = tid / T;
  const int t = tid - lrow * T;
  const bool active = lrow < L;
  const RowLayout<SH> lay{smem + (active ? lrow : 0) * padk(N, SH)};
  const int items = batch * (N / L);
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const size_t row = (size_t)it * L + (active ? lrow : 0);  // global row over the batch
    const size_t off = row * N + t;
    float2 v[E];
    if (active) {
#pragma unroll
      for (int i = 0; i < E; ++i) v[i] = in[off + i * T];
    }
    fft_line<N, E, DIR>(v, lay, Sync{}, active, t, tw);
    if (active) {
#pragma unroll
      for (int i = 0; i < E; ++i) out[off + i * T] = v[i];
    }
  }
}

template <int N, int DIR>
__global__ void __launch_bounds__(kThreads) fft_cols_kernel(const float2* in,
                                                            float2* out, int batch,
                                                            float scale,
                                                            const float2* __restrict__ tw_all) {
  constexpr int E = (N < 16 ? N : 16);
  constexpr int T = N / E;
  constexpr int C = lines_per_item(N, E);
  extern __shared__ float2 smem[];
  float2* tw = smem + item_smem_elems(N, E);
  build_stage_twiddles<N, E>(tw, tw_all + N);
  __syncthreads();
  const int tid = threadIdx.x;
  const int c = tid % C;
  const int t = tid / C;
  const bool active = t < T;
  const ColLayout<pad_shift(E), C> lay{smem + c};
  const int per_plane = N / C;
  const int items = batch * per_plane;
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const int plane = it / per_plane;
    const int col = (it - plane * per_plane) * C + c;
    const size_t off = (size_t)plane * N * N + (size_t)(active ? t : 0) * N + col;
    float2 v[E];
    __syncthreads();
    if (active) {
#pragma unroll
      for (int i = 0; i < E; ++i) v[i] = in[off + (size_t)i * T * N];
    }
    fft_line<N, E, DIR>(v, lay, BlockSync{}, active, t, tw);
    if (active) {
#pragma unroll
      for (int i = 0; i < E; ++i) out[off + (size_t)i * T * N] = make_float2(v[i].x * scale, v[i].y * scale);
    }
  }
}

// ---------------------------------------------------------------------------
// 2-D transforms of frames (n, rows, cols) embedded at the corner of zeroed
// N x N planes, reduced over the frames pixel by pixel (PRTF, RFTF), without
// making the zeros or storing the transforms: the row kernel transforms only
// the frames' own rows, straight from the frames, and leaves them transposed,
// so that a column is contiguous; in the column kernel every line of a CTA is
// then a column of its own, loaded, transformed and added up in registers with
// no barrier wider than the line.  128 frames of 180^2 at N = 512: 40 us of rows
// (shared-memory wavefronts, 78% of their rate: two exchanges, the twiddles and
// the strips' transposition; with its stores in contiguous pieces 37), 71 us of
// columns (instruction issue) and 6 us to add the partial sums up, against 435
// us for embedding, two passes over the planes and an accumulation; columns
// interleaved in a CTA, with block barriers, took 128 us.  37 frames of 173 x 181, RFTF: 55 us (rows
// 14, columns 32, sums 6), from 137 us.  Radix 32 (two stages at 512) made the
// columns 65 us but changed the transforms' rounding.
// ---------------------------------------------------------------------------
struct EmbedArgs {
  const float2* src;
  float2* dst;  // n planes of N x N: plane f, row c = column c of frame f's row transforms
  int n, rows, cols;
  const float2* tw;
};

// threads of the column kernel's CTAs: a line of 16 values a thread
__host__ __device__ constexpr int embed_threads(int N) { return N >= 4096 ? 256 : 128; }
// values per thread: those of sp_fft2, so that the transforms are its bit for
// bit (where F is nearly 0 its phasor amplifies any change of rounding)
__host__ __device__ constexpr int embed_e(int N) { return N < 16 ? N : 16; }
// resident CTAs per SM it is compiled for
__host__ __device__ constexpr int embed_ctas(int N) { return embed_threads(N) > 128 ? 2 : 5; }

// ---------------------------------------------------------------------------
// Lines of planes transformed one by one: a CTA takes L lines of one plane, T
// threads each, with no barrier wider than the line around the transform.  The
// Op supplies line values and takes the results; transposed_store writes them
// out with line and position exchanged, so that the other dimension's lines
// are contiguous for the next kernel.  The strips' pitch (as the column
// pass's) makes its reads, L lines of 16 / L positions per half-warp,
// conflict-free.  E = min(16, N) as in sp_fft2: bitwise its transforms.
// ---------------------------------------------------------------------------
template <int N>
struct Lines {
  static constexpr int E = (N < 16 ? N : 16), T = N / E, L = lines_per_item(N, E), SH = pad_shift(E);
  static constexpr int P = L >= 16 ? next_congruent(padk(N, SH), 1, 2)
                                   : next_congruent(padk(N, SH), 16 / L, 16);
  static constexpr int kTw = L * P;
  static constexpr int kExtra = kTw + tw_stage_total(N, E);  // the Op's own, Op::extra(N) entries
};

template <int T>
struct LineGroupSync {
  using type = typename std::conditional<(T <= 32), WarpSync, LineSync<T>>::type;
  __device__ static type make(int line) {
    if constexpr (T <= 32) return type{};
    else return type{1 + line};
  }
};

// dst[pos * pitch + l] = value of line l at `pos`, for l < nl and pos < np.
// Every thread of the block calls it; the strips are free afterwards.
template <int N, class Sync>
__device__ __forceinline__ void transposed_store(const float2 (&v)[Lines<N>::E], float2* smem, int lrow,
                                                 int t, const Sync& sync, float2* dst, size_t pitch,
                                                 int nl, int np) {
  using LN = Lines<N>;
  const RowLayout<LN::SH> lay{smem + (lrow < LN::L ? lrow : 0) * LN::P};
  sync();  // the line's last stage has read its strip
  if (lrow < LN::L) {
#pragma unroll
    for (int i = 0; i < LN::E; ++i) lay.at(t + i * LN::T) = v[i];
  }
  __syncthreads();
  for (int q = threadIdx.x; q < LN::L * np; q += kThreads) {
    const int l = q % LN::L, pos = q / LN::L;
    if (l < nl) dst[(size_t)pos * pitch + l] = smem[l * LN::P + padk(pos, LN::SH)];
  }
  __syncthreads();
}

// Op: planes, lines (of a plane), extra(N) (float2 entries of shared memory of
// its own), init(extra) (once per CTA) and prepare(plane, extra) (at each new
// plane; block-wide, it synchronises if it writes), line(plane, line) -> Line, what the
// line's threads keep of it, load(Line, pos, extra), done(plane, line0, nl, v,
// smem, lrow, t, sync).
template <int N, int DIR, class Op>
__global__ void __launch_bounds__(kThreads, 3) lines_kernel(Op op, const float2* __restrict__ tw_all) {
  using LN = Lines<N>;
  constexpr int E = LN::E, T = LN::T, L = LN::L;
  extern __shared__ float2 smem[];
  float2* tw = smem + LN::kTw;
  float2* extra = smem + LN::kExtra;
  build_stage_twiddles<N, E>(tw, tw_all + N);
  op.init(extra);
  __syncthreads();
  const int lrow = threadIdx.x / T;
  const int t = threadIdx.x - lrow * T;
  const bool line = lrow < L;
  const RowLayout<LN::SH> lay{smem + (line ? lrow : 0) * LN::P};
  const auto sync = LineGroupSync<T>::make(lrow);
  const int blocks = (op.lines + L - 1) / L;  // of one plane
  const int64_t items = (int64_t)op.planes * blocks;
  // each CTA a run of neighbouring items, so that it prepares few planes
  const int64_t run = (items + gridDim.x - 1) / gridDim.x, i0 = blockIdx.x * run;
  int ready = -1;
  for (int64_t it = i0; it < items && it < i0 + run; ++it) {
    const int f = (int)(it / blocks);
    const int l0 = (int)(it - (int64_t)f * blocks) * L;
    const int nl = op.lines - l0 < L ? op.lines - l0 : L;
    if (f != ready) op.prepare(f, extra);
    ready = f;
    const typename Op::Line ln = op.line(f, l0 + (lrow < nl ? lrow : 0));
    float2 v[E];
#pragma unroll
    for (int i = 0; i < E; ++i)
      v[i] = lrow < nl ? op.load(ln, t + i * T, extra) : make_float2(0.f, 0.f);
    fft_line<N, E, DIR>(v, lay, sync, line, t, tw);
    op.template done<N>(f, l0, nl, v, smem, lrow, t, sync);
  }
}

template <int N, int DIR, class Op>
cudaError_t launch_lines(const Op& op, const float2* tw, int n_sms, cudaStream_t st) {
  const int sm = (Lines<N>::kExtra + Op::extra(N)) * (int)sizeof(float2);
  const cudaError_t e =
      cudaFuncSetAttribute(lines_kernel<N, DIR, Op>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  if (e != cudaSuccess) return e;
  const int64_t items = (int64_t)op.planes * ((op.lines + Lines<N>::L - 1) / Lines<N>::L);
  if (items == 0) return cudaSuccess;
  lines_kernel<N, DIR, Op><<<(int)(items < n_sms * 3 ? items : n_sms * 3), kThreads, sm, st>>>(op, tw);
  return cudaGetLastError();
}

// The frames' rows, zero-padded to N, stored transposed into the planes.
struct EmbedRowsOp {
  const float2* src;
  float2* dst;
  int planes, lines, cols;  // lines: rows of a frame
  static constexpr int extra(int) { return 0; }
  __device__ void init(float2*) const {}
  __device__ void prepare(int, float2*) const {}
  using Line = const float2*;
  __device__ __forceinline__ Line line(int f, int r) const { return src + ((int64_t)f * lines + r) * cols; }
  __device__ __forceinline__ float2 load(Line l, int c, const float2*) const {
    return c < cols ? l[c] : make_float2(0.f, 0.f);
  }
  template <int N, class Sync>
  __device__ __forceinline__ void done(int f, int l0, int nl, const float2 (&v)[Lines<N>::E],
                                       float2* smem, int lrow, int t, const Sync& sync) const {
    transposed_store<N>(v, smem, lrow, t, sync, dst + (size_t)f * N * N + l0, N, nl, N);
  }
};

// Columns of the transposed planes, one line of T threads each.  The work is
// the (column group, frame) pairs, groups outermost, dealt to the CTAs in equal
// runs of `run` pairs; a CTA adds up its frames of one group and stores the
// sum over the lines' own rows of the first plane it read for them (each
// thread overwrites only what it alone has read), still transposed.  So the
// sums of group g lie in planes f with f = 0 or (g n + f) % run = 0 (see
// for_each_sum).  `Op` maps (F, pixel) to the summand.
__host__ __device__ constexpr int embed_group_cols(int N) {
  return lines_per_item_t(N, embed_e(N), embed_threads(N));
}
// An Op's goal values of a group's columns are staged row by row (read straight
// by the columns' threads, every value is a sector of its own: 39 us for 37
// frames at 512, 32 staged; kept in shared memory instead of each thread's
// registers 35).  Pitch: the 32 / L rows of a warp's store on different banks.
__host__ __device__ constexpr int embed_goal_pitch(int N) {
  return N + (embed_group_cols(N) < 32 ? 32 / embed_group_cols(N) : 1);
}
template <int N, class Op>
constexpr int embed_goal_floats() {
  return Op::kGoal ? embed_group_cols(N) * embed_goal_pitch(N) : 0;
}
template <int N, class Op>
__global__ void __launch_bounds__(embed_threads(N), embed_ctas(N)) embed_cols_sum_kernel(EmbedArgs a, Op op,
                                                                                  int run) {
  constexpr int E = embed_e(N), T = N / E, L = embed_group_cols(N);
  constexpr int SH = pad_shift(E);
  extern __shared__ float2 smem[];
  float2* tw = smem + L * padk(N, SH);
  build_stage_twiddles<N, E>(tw, a.tw + N);
  __syncthreads();
  const int lc = threadIdx.x / T;
  const int t = threadIdx.x - lc * T;
  const bool active = lc < L;
  const RowLayout<SH> lay{smem + (active ? lc : 0) * padk(N, SH)};
  const auto sync = LineGroupSync<T>::make(lc);
  const int64_t total = (int64_t)(N / L) * a.n;
  int64_t u = (int64_t)blockIdx.x * run;
  const int64_t end = u + run < total ? u + run : total;
  while (u < end) {
    const int g = (int)(u / a.n), f0 = (int)(u - (int64_t)g * a.n);
    const int nf = (int)(end - u < a.n - f0 ? end - u : a.n - f0);
    const int col = g * L + (active ? lc : 0);
    float2* p = a.dst + (size_t)f0 * N * N + (size_t)col * N + t;
    typename Op::Acc acc[E];
    typename Op::Pixel px[E];
    float* goal = reinterpret_cast<float*>(tw + tw_stage_total(N, E));
    constexpr int GP = embed_goal_pitch(N);
    bool odd_px = false;  // a pixel whose summands need add_odd
    if constexpr (Op::kGoal) {
      __syncthreads();  // the previous group's values are read
      for (int k = threadIdx.x; k < N * L; k += embed_threads(N))
        goal[k % L * GP + k / L] = op.goal[(size_t)(k / L) * N + g * L + k % L];
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < E; ++i) {
      acc[i] = typename Op::Acc{};
      if constexpr (Op::kGoal) px[i] = op.pixel(goal[(active ? lc : 0) * GP + t + i * T]);
      odd_px |= Op::odd(px[i]);
    }
    for (int f = 0; f < nf; ++f) {
      const float2* q = p + (size_t)f * N * N;
      float2 v[E];
#pragma unroll
      for (int i = 0; i < E; ++i)
        v[i] = (active && t + i * T < a.rows) ? __ldcg(q + i * T) : make_float2(0.f, 0.f);
      fft_line<N, E, -1>(v, lay, sync, active, t, tw);
      bool odd = false;
      if (odd_px) {
#pragma unroll
        for (int i = 0; i < E; ++i) Op::add_odd(acc[i], v[i], px[i]);
      } else {
#pragma unroll
        for (int i = 0; i < E; ++i) odd |= !op.add(acc[i], v[i], px[i]);
      }
      if (odd) {
#pragma unroll 1
        for (int i = 0; i < E; ++i) {
          // (register arrays take constant indexes only: pick element i)
          float2 x = v[0];
          typename Op::Pixel y = px[0];
          typename Op::Acc z{};
#pragma unroll
          for (int k = 1; k < E; ++k)
            if (k == i) x = v[k], y = px[k];
          Op::add_odd(z, x, y);
#pragma unroll
          for (int k = 0; k < E; ++k)
            if (k == i) Op::plus(acc[k], z);
        }
      }
      if constexpr (T > 32) __syncwarp();  // the next line barrier takes whole warps
    }
    if (active) {
#pragma unroll
      for (int i = 0; i < E; ++i) p[i * T] = Op::store(acc[i]);
    }
    u += nf;
  }
}

// f(plane) for every plane that holds a sum of column c
template <class F>
__device__ __forceinline__ void for_each_sum(int c, int group_cols, int n, int run, F&& f) {
  const int64_t base = (int64_t)(c / group_cols) * n;
  f(0);
#pragma unroll 4
  for (int k = run - (int)(base % run); k < n; k += run) f(k);
}

// F/|F| summed (phasing_prtf_accumulate2.cl:20-23); nothing where F = 0.  The
// reciprocal square root takes one Newton step (to ~1 ulp, as hypotf and a
// division); magnitudes whose square leaves the normal range go through hypotf.
struct PhasorSum {
  struct Pixel {};
  using Acc = float2;
  __device__ static float2 store(float2 x) { return x; }
  __device__ static void plus(float2& a, float2 b) { a.x += b.x, a.y += b.y; }
  static constexpr bool kGoal = false;
  __device__ __forceinline__ static bool odd(Pixel) { return false; }
  __device__ __forceinline__ static bool plain(float p2) { return p2 > 1e-30f && p2 < 1e30f; }
  // adds the summand unless its magnitude needs add_odd; whether it did
  __device__ __forceinline__ bool add(float2& acc, float2 v, Pixel) const {
    const float p2 = v.x * v.x + v.y * v.y;
    const bool ok = plain(p2);
    float r = ok ? rsqrtf(p2) : 0.f;
    r = r * fmaf(-0.5f * p2 * r, r, 1.5f);
    acc.x = ok ? fmaf(v.x, r, acc.x) : acc.x;
    acc.y = ok ? fmaf(v.y, r, acc.y) : acc.y;
    return ok;
  }
  __device__ static void add_odd(float2& acc, float2 v, Pixel) {
    if (plain(v.x * v.x + v.y * v.y)) return;
    const float h = hypotf(v.x, v.y);
    if (h > 0.f) {
      acc.x += v.x / h;
      acc.y += v.y / h;
    }
  }
};

// 1/sqrt(1 + (g - |F|)^2 / g^2) summed (phasing_rftf_accumulate.cl), g the goal
// modulus.  1/sqrt(x) by the reciprocal square root and one Newton step.  At g = 0
// the quotient is infinite, or NaN for F = 0 too, as in the division; a square past
// the range leaves |F| infinite and the summand 0, as a square root would.  From
// g = 9.2e18 on 1/g^2 is below the normal range (and flushed): a thread with such a
// pixel (`odd`) takes the quotient itself.
struct RftfSum {
  const float* goal;
  struct Pixel {
    float g, inv;  // g, 1/g^2
  };
  using Acc = float;
  __device__ static float2 store(float x) { return make_float2(x, 0.f); }
  __device__ static void plus(float& a, float b) { a += b; }
  static constexpr bool kGoal = true;
  __device__ static Pixel pixel(float g) { return {g, 1.f / (g * g)}; }
  __device__ __forceinline__ static bool odd(Pixel p) { return p.inv == 0.f; }
  __device__ __forceinline__ static float misfit(float2 v, Pixel p) {
    const float p2 = v.x * v.x + v.y * v.y;
    return p.g - (p2 > 0.f && p2 < 3e38f ? p2 * rsqrtf(p2) : p2);
  }
  __device__ __forceinline__ bool add(float& acc, float2 v, Pixel p) const {
    const float d1 = misfit(v, p);
    const float x = 1.f + (d1 * d1) * p.inv;
    float r = rsqrtf(x);
    if (x < 1e30f) r = r * fmaf(-0.5f * x * r, r, 1.5f);
    acc += r;
    return true;
  }
  __device__ __forceinline__ static void add_odd(float& acc, float2 v, Pixel p) {
    const float d1 = misfit(v, p);
    acc += 1.f / sqrtf(1.f + (d1 * d1) / (p.g * p.g));
  }
};

// Row and column kernels of embedded frames; *run and *group_cols say where
// the sums lie (for_each_sum).  The column kernel's runs fill the chip once.
template <int N, class Op>
cudaError_t embed_sum_t(const EmbedArgs& a, const Op& op, int* run, int* group_cols, int n_sms,
                        cudaStream_t st) {
  constexpr int E = embed_e(N), LC = embed_group_cols(N);
  const int sc = (LC * padk(N, pad_shift(E)) + tw_stage_total(N, E)) * (int)sizeof(float2) +
                 embed_goal_floats<N, Op>() * (int)sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(embed_cols_sum_kernel<N, Op>, cudaFuncAttributeMaxDynamicSharedMemorySize, sc);
  if (e != cudaSuccess) return e;
  const int64_t total = (int64_t)(N / LC) * a.n, slots = (int64_t)embed_ctas(N) * n_sms;
  *run = (int)((total + slots - 1) / slots);
  *group_cols = LC;
  e = launch_lines<N, -1>(EmbedRowsOp{a.src, a.dst, a.n, a.rows, a.cols}, a.tw, n_sms, st);
  if (e != cudaSuccess) return e;
  embed_cols_sum_kernel<N, Op><<<(int)((total + *run - 1) / *run), embed_threads(N), sc, st>>>(a, op, *run);
  return cudaGetLastError();
}

template <int N>
cudaError_t fft2_t(const float2* in, float2* out, int batch, int inverse, cudaStream_t st,
                   const float2* tw, int n_sms) {
  constexpr int E = (N < 16 ? N : 16);
  const int sm = (item_smem_elems(N, E) + tw_stage_total(N, E)) * (int)sizeof(float2);
  const int rows_items = batch * (N / lines_per_item(N, E));
  const int grid = rows_items < n_sms * 4 ? rows_items : n_sms * 4;
  const float scale = inverse ? 1.0f / ((float)N * (float)N) : 1.0f;
  cudaError_t e;
  if (inverse) {
    e = cudaFuncSetAttribute(fft_rows_kernel<N, +1>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(fft_cols_kernel<N, +1>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e != cudaSuccess) return e;
    fft_rows_kernel<N, +1><<<grid, kThreads, sm, st>>>(in, out, batch, tw);
    fft_cols_kernel<N, +1><<<grid, kThreads, sm, st>>>(out, out, batch, scale, tw);
  } else {
    e = cudaFuncSetAttribute(fft_rows_kernel<N, -1>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(fft_cols_kernel<N, -1>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e != cudaSuccess) return e;
    fft_rows_kernel<N, -1><<<grid, kThreads, sm, st>>>(in, out, batch, tw);
    fft_cols_kernel<N, -1><<<grid, kThreads, sm, st>>>(out, out, batch, scale, tw);
  }
  return cudaGetLastError();
}

cudaError_t fft2_dispatch(const float2* in, float2* out, int N, int batch, int inverse,
                          cudaStream_t st);

// embed_sum_t of F/|F| (goal null) or of the RFTF's summand (`work`: n N x N
// planes)
cudaError_t frame_sums_dispatch(int N, const float2* src, float2* work, int n, int rows, int cols,
                                const float* goal, int* run, int* group_cols, cudaStream_t st);

// The column kernel's partial sums (SumsAt: where they lie), added up and
// transposed back: element (r, c) lies at row c, column r of their planes.  One
// 32 x 32 tile per block, a thread an element, through shared memory; `f` gets
// each sum and its place.  N < 32: partial tiles.  Bound by the latency of each
// element's few loads, so all elements are in flight at once and the loads of
// four planes together (512^2: 128 frames' PRTF sums 12 to 6 us, 37 frames' RTF
// sums 10 to 5 us, against four elements a thread and one load at a time).  Added
// in FP64: at small N a partial sum is a frame or two, and the FP32 sum of tens of
// them was less exact than the running mean that this replaces (40 frames at
// 128^2, RFTF: rms error 8.8e-8 against 8.0e-8, now 3.5e-8; the sums take the same time to 1 us).
struct SumsAt {
  int frames, run, group_cols;
};
inline dim3 frame_sums_grid(int N) { return dim3((N + 31) / 32, (N + 31) / 32); }
constexpr int kFrameSumsThreads = 1024;  // 32 x 32
template <class F>
__device__ __forceinline__ void transposed_sums(const float2* __restrict__ part, SumsAt at, int N, F&& f) {
  __shared__ float2 tile[32][33];
  const int64_t NN = (int64_t)N * N;
  const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
  if (c0 + ty < N && r0 + tx < N) {
    const float2* p = part + (int64_t)(c0 + ty) * N + r0 + tx;
    double x = 0, y = 0;
    for_each_sum(c0 + ty, at.group_cols, at.frames, at.run, [&](int k) {
      const float2 v = p[k * NN];
      x += v.x;
      y += v.y;
    });
    tile[ty][tx] = make_float2((float)x, (float)y);
  }
  __syncthreads();
  if (r0 + ty < N && c0 + tx < N) f(r0 + ty, c0 + tx, tile[tx][ty]);
}

#define SP_DECLARE_FFT2(N) \
  cudaError_t fft2_n##N(const float2* in, float2* out, int batch, int inverse, cudaStream_t st, \
                        const float2* tw, int n_sms); \
  cudaError_t phasor_frames_n##N(const EmbedArgs& a, int* run, int* group_cols, int n_sms, cudaStream_t st); \
  cudaError_t rftf_frames_n##N(const EmbedArgs& a, const float* goal, int* run, int* group_cols, \
                               int n_sms, cudaStream_t st);
SP_DECLARE_FFT2(8)
SP_DECLARE_FFT2(16)
SP_DECLARE_FFT2(32)
SP_DECLARE_FFT2(64)
SP_DECLARE_FFT2(128)
SP_DECLARE_FFT2(256)
SP_DECLARE_FFT2(512)
SP_DECLARE_FFT2(1024)
SP_DECLARE_FFT2(2048)
SP_DECLARE_FFT2(4096)

#define SP_DEFINE_FFT2(N)                                                                     \
  cudaError_t fft2_n##N(const float2* in, float2* out, int batch, int inverse, cudaStream_t st, \
                        const float2* tw, int n_sms) {                                        \
    return fft2_t<N>(in, out, batch, inverse, st, tw, n_sms);                                 \
  }                                                                                           \
  cudaError_t phasor_frames_n##N(const EmbedArgs& a, int* run, int* group_cols, int n_sms, cudaStream_t st) { \
    return embed_sum_t<N>(a, PhasorSum{}, run, group_cols, n_sms, st);                        \
  }                                                                                           \
  cudaError_t rftf_frames_n##N(const EmbedArgs& a, const float* goal, int* run,               \
                               int* group_cols, int n_sms, cudaStream_t st) {                 \
    return embed_sum_t<N>(a, RftfSum{goal}, run, group_cols, n_sms, st);                      \
  }

}  // namespace sp
