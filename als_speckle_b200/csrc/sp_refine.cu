// Shrinkwrap (refine_support, phasing.py:1747-1815): separable circular
// Gaussian blur of |avg| in FP64 (phasing.py:1786-1790:
// ifft2(fft2(fftshift(g)/sum g) * fft2(|avg|)).real is a circular convolution
// with the separable kernel k_r (x) k_c), the connected parts of the support
// (masking.find_all_objects :379-435), and the per-part thresholds.
#include <vector>

#include "sp_common.cuh"

namespace sp {
namespace {

// ---------------------------------------------------------------------------
// blur: out[pos] = sum_j k[j] in[pos - j] (circular) along one axis, taps in
// order.  Bound by FP64 FMAs and shared-memory reads: a block takes 32 lines
// (one per lane) x 32 positions, a thread 4 neighbouring positions whose inputs
// slide by one a tap, so a tap costs one wide and one broadcast read for four
// FMAs; the inputs of kTaps taps at a time are staged, wrapped round.  At 340^2
// the two axes take 29 and 23 us, against 61 and 55 us for one thread per pixel
// reading (and, along the rows, taking the magnitude of) every tap's input.
// ---------------------------------------------------------------------------
constexpr int kTile = 32, kTaps = 64, kSpan = kTile + kTaps - 1;

template <bool ROWS>
__global__ void __launch_bounds__(256) blur_kernel(const void* __restrict__ in,
                                                   const double* __restrict__ k,
                                                   double* __restrict__ out, int rows, int cols) {
  __shared__ double a[kSpan][kTile + 1];
  __shared__ double kk[kTaps];
  const int lines = ROWS ? rows : cols, n = ROWS ? cols : rows;
  const int across = (n - 1) / kTile + 1;  // (one grid dimension: any shape fits it)
  const int l0 = blockIdx.x / across * kTile, p0 = blockIdx.x % across * kTile;
  const int lane = threadIdx.x % 32, u = 4 * (threadIdx.x / 32);  // positions p0 + u .. u + 3
  double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
  for (int j0 = 0; j0 < n; j0 += kTaps) {
    const int nt = n - j0 < kTaps ? n - j0 : kTaps;
    __syncthreads();  // the previous taps' inputs are used
    int base = (p0 - j0 - (kTaps - 1)) % n;  // position of q = 0 (q = position + kTaps - 1 - tap)
    if (base < 0) base += n;
#pragma unroll 6
    for (int i = threadIdx.x; i < kSpan * kTile; i += 256) {
      // neighbouring threads at neighbouring addresses
      const int q = ROWS ? i % kSpan : i / kTile, l = ROWS ? i / kSpan : i % kTile;
      int pos = base + q;
      if (pos >= n) pos -= n;
      if (pos >= n) pos %= n;  // (n < kSpan)
      double v = 0;
      if (l0 + l < lines) {
        if (ROWS) {
          const float2 z = static_cast<const float2*>(in)[(size_t)(l0 + l) * cols + pos];
          v = (double)sqrtf(fmaf(z.x, z.x, z.y * z.y));
        } else {
          v = static_cast<const double*>(in)[(size_t)pos * cols + l0 + l];
        }
      }
      a[q][l] = v;
    }
    for (int j = threadIdx.x; j < nt; j += 256) kk[j] = k[j0 + j];
    __syncthreads();
    // w[d]: the input of position u + d at the tap
    int q = u + kTaps - 1;
    double w1 = a[q + 1][lane], w2 = a[q + 2][lane], w3 = a[q + 3][lane];
#pragma unroll 8
    for (int j = 0; j < nt; ++j, --q) {
      const double w0 = a[q][lane], c = kk[j];
      s0 = fma(c, w0, s0);
      s1 = fma(c, w1, s1);
      s2 = fma(c, w2, s2);
      s3 = fma(c, w3, s3);
      w3 = w2;
      w2 = w1;
      w1 = w0;
    }
  }
  if (l0 + lane >= lines) return;
  const double s[4] = {s0, s1, s2, s3};
#pragma unroll
  for (int d = 0; d < 4; ++d) {
    const int pos = p0 + u + d;
    if (pos < n) out[ROWS ? (size_t)(l0 + lane) * cols + pos : (size_t)pos * cols + l0 + lane] = s[d];
  }
}

// ---------------------------------------------------------------------------
// connected parts of a mask: 8 neighbours, periodic.  Union-find over pixel
// indexes by atomic minima (Playne & Hawick, IEEE Trans. Parallel Distrib. Syst.
// 29, 2018) with path halving (Tarjan & van Leeuwen, J. ACM 31, 1984), always
// towards the smaller index, so a part's root is its first pixel
// in raster order (the order in which the reference finds the parts).  Runs
// inside a warp's 32 pixels start out linked to their first pixel; then every
// pixel joins its neighbours to the left (across warps) and above where the
// pixel to its left does not already do so.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int part_find(int* parent, int x) {
  volatile int* p = parent;
  int y = p[x];
  while (y != x) {  // (indexes only decrease along the chain, so this ends)
    const int z = p[y];
    if (z != y) p[x] = z;  // halve the path; a racing write also points into the part
    x = y;
    y = z;
  }
  return x;
}
__device__ __forceinline__ void part_join(int* parent, int a, int b) {
  a = part_find(parent, a);
  b = part_find(parent, b);
  while (a != b) {  // a or b decreases every time round
    if (a < b) {
      const int t = a;
      a = b;
      b = t;
    }
    const int old = atomicMin(&parent[a], b);
    if (old == a) return;  // a was a root and now hangs below b
    a = part_find(parent, old);
    b = part_find(parent, b);
  }
}

__global__ void __launch_bounds__(256) parts_init_kernel(const unsigned char* __restrict__ mask,
                                                         int* __restrict__ parent, int rows, int cols) {
  const int across = (cols - 1) / 32 + 1;
  const int c = blockIdx.x % across * 32 + threadIdx.x, r = blockIdx.x / across * 8 + threadIdx.y;
  const bool in = r < rows && c < cols;
  const bool m = in && mask[(size_t)r * cols + c];
  const unsigned run = __ballot_sync(0xffffffffu, m);
  if (!in) return;
  const unsigned gaps = ~run & ((1u << threadIdx.x) - 1);  // the last gap before this pixel
  const int first = gaps ? 32 - __clz(gaps) : 0;
  parent[(size_t)r * cols + c] = m ? r * cols + c - ((int)threadIdx.x - first) : -1;
}

__global__ void __launch_bounds__(256) parts_join_kernel(const unsigned char* __restrict__ mask,
                                                         int* parent, int rows, int cols) {
  const int across = (cols - 1) / 32 + 1;
  const int c = blockIdx.x % across * 32 + threadIdx.x, r = blockIdx.x / across * 8 + threadIdx.y;
  if (r >= rows || c >= cols) return;
  const int i = r * cols + c;
  if (!mask[i]) return;
  const int cw = c ? c - 1 : cols - 1, ce = c + 1 < cols ? c + 1 : 0;
  const int up = (r ? r - 1 : rows - 1) * cols;
  const bool w = mask[r * cols + cw], n = mask[up + c], nw = mask[up + cw], ne = mask[up + ce];
  // column 0 leans on no pixel to its left, so a row that is full all round
  // (periodic) still joins the row above; with fewer than 3 columns left and
  // right are the same pixel and nothing is left out
  const bool lean = c > 0 && cols > 2;
  if (threadIdx.x == 0 && w) part_join(parent, i, r * cols + cw);
  if (n) {
    if (!(lean && w && nw)) part_join(parent, i, up + c);
    if (!lean) {
      if (nw) part_join(parent, i, up + cw);
      if (ne) part_join(parent, i, up + ce);
    }
  } else {
    if (nw && !(lean && w)) part_join(parent, i, up + cw);
    if (ne) part_join(parent, i, up + ce);
  }
}

// label = root + 1; 0 outside the mask and for a pixel with no neighbour in it
// (the flood fill never marks its start pixel, so such a part is empty,
// masking.py:357-372)
__global__ void __launch_bounds__(256) parts_label_kernel(const unsigned char* __restrict__ mask,
                                                          int* parent, int* __restrict__ labels, int rows,
                                                          int cols) {
  const int across = (cols - 1) / 32 + 1;
  const int c = blockIdx.x % across * 32 + threadIdx.x, r = blockIdx.x / across * 8 + threadIdx.y;
  if (r >= rows || c >= cols) return;
  const int i = r * cols + c;
  int l = 0;
  if (mask[i]) {
    bool alone = true;
    for (int dr = -1; dr <= 1; ++dr)
      for (int dc = -1; dc <= 1; ++dc) {
        const int rr = (r + dr + rows) % rows, cc = (c + dc + cols) % cols;
        alone &= rr * cols + cc == i || !mask[rr * cols + cc];
      }
    l = alone ? 0 : part_find(parent, i) + 1;
  }
  labels[i] = l;
}

// The part with the smallest sum of |avg|, the first of equals (phasing.py:1811-1813;
// a comparison with NaN keeps the earlier part, as in the reference's scan): its label.
__global__ void __launch_bounds__(1024) parts_weakest_kernel(const unsigned char* __restrict__ mask,
                                                             const int* __restrict__ parent,
                                                             const double* __restrict__ sums, int total,
                                                             int* __restrict__ weakest) {
  __shared__ double sum[32];
  __shared__ int idx[32], first[32];
  double best = 0;
  int at = total, fst = total;  // `total`: none
  auto take = [&](double s, int i) {
    if (i < total && !isnan(s) && (at == total || s < best || (s == best && i < at))) best = s, at = i;
  };
  for (int i = threadIdx.x; i < total; i += 1024)
    if (mask[i] && parent[i] == i) {
      fst = i < fst ? i : fst;
      take(sums[i + 1], i);
    }
  auto reduce = [&](int width) {
    for (int o = width / 2; o > 0; o >>= 1) {
      const double s = __shfl_xor_sync(0xffffffffu, best, o);
      const int i = __shfl_xor_sync(0xffffffffu, at, o), f = __shfl_xor_sync(0xffffffffu, fst, o);
      take(s, i);
      fst = f < fst ? f : fst;
    }
  };
  reduce(32);
  if (threadIdx.x % 32 == 0) sum[threadIdx.x / 32] = best, idx[threadIdx.x / 32] = at, first[threadIdx.x / 32] = fst;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  best = sum[threadIdx.x];
  at = idx[threadIdx.x];
  fst = first[threadIdx.x];
  reduce(32);
  if (threadIdx.x == 0) {
    const bool keep_first = fst < total && isnan(sums[fst + 1]);
    const int k = keep_first ? fst : at;
    *weakest = k < total ? k + 1 : -1;
  }
}

// ---------------------------------------------------------------------------
// per-label maxima of blurred and sums of |avg| (label 0 = global max), as
// order-preserving 64-bit keys for atomicMax.  One atomic per block for the
// global maximum and, where a warp's labelled pixels are of one part (nearly
// always), one per warp for a part: with one per pixel the atomics on a few
// addresses took 85 us at 340^2.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long dkey(double x) {
  unsigned long long u = (unsigned long long)__double_as_longlong(x);
  return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double dkey_inv(unsigned long long k) {
  const unsigned long long u = (k & 0x8000000000000000ull) ? (k & ~0x8000000000000000ull) : ~k;
  return __longlong_as_double((long long)u);
}
__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, v, o);
    v = other > v ? other : v;
  }
  return v;
}
__global__ void __launch_bounds__(256) label_stats_kernel(const double* __restrict__ blurred,
                                                          const float2* __restrict__ avg,
                                                          const int* __restrict__ labels, int64_t total,
                                                          unsigned long long* __restrict__ maxkey,
                                                          double* __restrict__ sums) {
  __shared__ unsigned long long block_max[8];
  unsigned long long gmax = 0;
  // (whole warps in every round, for the shuffles)
  for (int64_t base = blockIdx.x * (int64_t)256; base < total; base += (int64_t)gridDim.x * 256) {
    const int64_t k = base + threadIdx.x;
    const bool in = k < total;
    const unsigned long long key = in ? dkey(blurred[k]) : 0;
    gmax = key > gmax ? key : gmax;
    const int l = in ? labels[k] : 0;
    const unsigned any = __ballot_sync(0xffffffffu, l > 0);
    if (any == 0) continue;  // uniform over the warp
    double m = 0;
    if (l > 0) {
      const float2 v = avg[k];
      m = (double)sqrtf(fmaf(v.x, v.x, v.y * v.y));
    }
    const int first = __shfl_sync(0xffffffffu, l, __ffs(any) - 1);
    if (__all_sync(0xffffffffu, l == 0 || l == first)) {
      const unsigned long long pk = warp_max(l > 0 ? key : 0);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
      if (threadIdx.x % 32 == 0) {
        atomicMax(&maxkey[first], pk);
        atomicAdd(&sums[first], m);
      }
    } else if (l > 0) {
      atomicMax(&maxkey[l], key);
      atomicAdd(&sums[l], m);
    }
  }
  gmax = warp_max(gmax);
  if (threadIdx.x % 32 == 0) block_max[threadIdx.x / 32] = gmax;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) gmax = block_max[w] > gmax ? block_max[w] : gmax;
    atomicMax(&maxkey[0], gmax);
  }
}

// refined = sum over parts of (b*part > max(b*part)*lt) times (b > max(b)*gt);
// the dropped part's label is kill_label, or *kill_dev when that is given
__global__ void threshold_kernel(const double* __restrict__ blurred, const int* __restrict__ labels,
                                 int64_t total, const unsigned long long* __restrict__ maxkey,
                                 double local_t, double global_t, int kill_label,
                                 const int* __restrict__ kill_dev, float* __restrict__ refined) {
  const double gmax = dkey_inv(maxkey[0]);
  const int kill = kill_dev ? *kill_dev : kill_label;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < total;
       k += (int64_t)gridDim.x * blockDim.x) {
    const double b = blurred[k];
    const int l = labels[k];
    float r = 0.f;
    if (l > 0 && l != kill) {
      // current.max() over the whole array includes the zeros outside the part
      const double pmax = fmax(dkey_inv(maxkey[l]), 0.0);
      r = (b > pmax * local_t) ? 1.f : 0.f;
    }
    if (!(b > gmax * global_t)) r = 0.f;
    refined[k] = r;
  }
}

int grid_of(int64_t n) {
  int64_t g = (n + 255) / 256;
  if (g > 148 * 8) g = 148 * 8;
  return (int)(g < 1 ? 1 : g);
}

cudaError_t launch_blur(const void* avg, int rows, int cols, const double* kr, const double* kc,
                        double* tmp, double* blurred, cudaStream_t st) {
  const int64_t tiles = (int64_t)((rows - 1) / kTile + 1) * ((cols - 1) / kTile + 1);
  if (tiles > INT32_MAX) return cudaErrorInvalidValue;
  blur_kernel<true><<<(unsigned)tiles, 256, 0, st>>>(avg, kc, tmp, rows, cols);
  blur_kernel<false><<<(unsigned)tiles, 256, 0, st>>>(tmp, kr, blurred, rows, cols);
  return cudaGetLastError();
}

}  // namespace
}  // namespace sp

using namespace sp;

extern "C" {

int sp_shrinkwrap(const void* avg, int rows, int cols, const double* kr, const double* kc,
                  const int* labels, int n_labels, double local_t, double global_t, int kill_weakest,
                  void* work, double* blurred, float* refined, double* part_sums,
                  sp_stream_t stream) {
  SP_CHECK(avg && kr && kc && labels && work && blurred && refined && part_sums, SP_ERR_INVALID,
           "sp_shrinkwrap: null pointer");
  SP_CHECK(rows > 0 && cols > 0 && n_labels >= 0, SP_ERR_INVALID, "sp_shrinkwrap: bad size");
  cudaStream_t st = as_stream(stream);
  const int64_t total = (int64_t)rows * cols;
  double* tmp = static_cast<double*>(work);
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(tmp + total);
  SP_CUDA_TRY(launch_blur(avg, rows, cols, kr, kc, tmp, blurred, st));
  // keys start at the smallest order-preserving key (0 encodes -NaN, below all)
  SP_CUDA_TRY(cudaMemsetAsync(keys, 0, sizeof(unsigned long long) * (n_labels + 1), st));
  SP_CUDA_TRY(cudaMemsetAsync(part_sums, 0, sizeof(double) * (n_labels + 1), st));
  label_stats_kernel<<<grid_of(total), 256, 0, st>>>(blurred, (const float2*)avg, labels, total, keys,
                                                     part_sums);
  SP_CUDA_TRY(cudaGetLastError());
  int kill = -1;
  if (kill_weakest && n_labels > 0) {
    // the weakest part is chosen on the host from part_sums (phasing.py:1811-1813)
    std::vector<double> h(n_labels + 1);
    SP_CUDA_TRY(cudaMemcpyAsync(h.data(), part_sums, sizeof(double) * (n_labels + 1),
                                cudaMemcpyDeviceToHost, st));
    SP_CUDA_TRY(cudaStreamSynchronize(st));
    kill = 1;
    for (int l = 2; l <= n_labels; ++l)
      if (h[l] < h[kill]) kill = l;
  }
  threshold_kernel<<<grid_of(total), 256, 0, st>>>(blurred, labels, total, keys, local_t, global_t,
                                                   kill, nullptr, refined);
  SP_CUDA_TRY(cudaGetLastError());
  return SP_OK;
}

// scratch: tmp (doubles) | keys and sums, one per pixel and one (8 bytes each) |
// parents, labels (ints) | the weakest part's label
int sp_refine_workspace_size(int rows, int cols, size_t* bytes) {
  SP_CHECK(bytes && rows > 0 && cols > 0 && (int64_t)rows * cols < INT32_MAX, SP_ERR_INVALID,
           "sp_refine_workspace_size: bad argument");
  const size_t total = (size_t)rows * cols;
  *bytes = 8 * total + 2 * 8 * (total + 1) + 2 * 4 * total + 8;
  return SP_OK;
}

int sp_refine_support(const void* avg, int rows, int cols, const double* kr, const double* kc,
                      const unsigned char* mask, double local_t, double global_t, int kill_weakest,
                      void* work, size_t work_bytes, double* blurred, float* refined,
                      sp_stream_t stream) {
  SP_CHECK(avg && work && blurred && refined && !kr == !kc && (kr || mask), SP_ERR_INVALID,
           "sp_refine_support: null pointer");
  size_t need = 0;
  const int rc = sp_refine_workspace_size(rows, cols, &need);
  if (rc != SP_OK) return rc;
  SP_CHECK(work_bytes >= need, SP_ERR_WORKSPACE, "sp_refine_support: %zu bytes given, %zu needed",
           work_bytes, need);
  cudaStream_t st = as_stream(stream);
  const int64_t total = (int64_t)rows * cols;
  double* tmp = static_cast<double*>(work);
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(tmp + total);
  double* sums = reinterpret_cast<double*>(keys + total + 1);
  int* parent = reinterpret_cast<int*>(sums + total + 1);
  int* labels = parent + total;
  int* weakest = labels + total;
  if (kr) SP_CUDA_TRY(launch_blur(avg, rows, cols, kr, kc, tmp, blurred, st));
  if (!mask) return SP_OK;
  const dim3 grid((unsigned)(((int64_t)(cols - 1) / 32 + 1) * ((rows - 1) / 8 + 1))), block(32, 8);
  parts_init_kernel<<<grid, block, 0, st>>>(mask, parent, rows, cols);
  parts_join_kernel<<<grid, block, 0, st>>>(mask, parent, rows, cols);
  parts_label_kernel<<<grid, block, 0, st>>>(mask, parent, labels, rows, cols);
  SP_CUDA_TRY(cudaGetLastError());
  // (the smallest order-preserving key is 0, and so is an empty sum)
  SP_CUDA_TRY(cudaMemsetAsync(keys, 0, 16 * (size_t)(total + 1), st));
  label_stats_kernel<<<grid_of(total), 256, 0, st>>>(blurred, (const float2*)avg, labels, total, keys,
                                                     sums);
  SP_CUDA_TRY(cudaGetLastError());
  if (kill_weakest) {
    parts_weakest_kernel<<<1, 1024, 0, st>>>(mask, parent, sums, (int)total, weakest);
    SP_CUDA_TRY(cudaGetLastError());
  }
  threshold_kernel<<<grid_of(total), 256, 0, st>>>(blurred, labels, total, keys, local_t, global_t, -1,
                                                   kill_weakest ? weakest : nullptr, refined);
  SP_CUDA_TRY(cudaGetLastError());
  return SP_OK;
}

}  // extern "C"
