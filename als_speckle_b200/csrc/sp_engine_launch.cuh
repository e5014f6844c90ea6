// Per-size engine kernels.  Each size N is compiled in its own translation
// unit (sp_engine_n<N>.cu) so register allocation is per (N, E) and the build
// parallelises; the host engine reaches them through launch_pass().
#pragma once
#include "sp_engine_kernels.cuh"

namespace sp {

struct PassArgs {
  const Slot* slots;
  const Item* items;
  int n_items;
  const int* tick_base;  // optional device counter added to tick_off
  int tick_off;
  const float2* tw;
  int reverse;  // walk the item list from its end
  int overlap;  // independent of the previous kernel of the stream (see chain_start)
  int late;     // let the next kernel in only at the last item
  int early;    // ... or at entry, before the wait
};

// The waits of programmatic launches (see pdl_allow_next).  A kernel whose
// planes are the previous kernel's output waits for it before its first item;
// one that only needs earlier kernels (another size's pass ran in between)
// starts at once, on the SMs that the previous kernel's last round leaves idle,
// and waits after its first item.  Either way it lets the next kernel in only
// after its wait, so when a kernel starts everything before its predecessor is
// complete: the planes that an early first item reads are in L2.  What the wait
// would add is that this SM sees them so: the column pass's 8-byte copies go
// through L1, which may still hold the lines that an earlier tick's pass read
// there.  So an early start makes a device-scope fence first, which drops them;
// nothing that runs beside the kernel writes these planes, so what is read from
// then on is what L2 holds.  With `late`, each CTA lets the next kernel in only
// when it begins its last item: CTAs let in earlier hold SMs that a concurrent line
// of launches could use (20 x 512^2 beside 12 x 256^2: 86 against 91 us per
// iteration; alone, earlier is better, 4 x 2048^2 266 against 268).  With `early`
// (lines of one size, which never set `overlap`) it lets it in before its own wait,
// so that two kernels stand by: where several lines leave most SMs idle, launches
// are what they wait for (40 x 64^2 beside 3 x 256^2, 60 iterations: 915 us, 969
// let in after the wait).
// LINE kernels know the flags; the others, for a size alone on the chip, wait
// and let go at their start (the flags' code in the loop costs the 2048^2 passes
// 2%).
template <bool LINE>
__device__ __forceinline__ void chain_start(const PassArgs& a) {
  if (LINE && a.overlap) {
    __threadfence();
    return;
  }
  if (LINE && a.early) pdl_allow_next();
  pdl_wait_prev();
  if (!(LINE && a.late)) pdl_allow_next();
}
template <bool LINE>
__device__ __forceinline__ void chain_top(const PassArgs& a, int k, bool last) {  // before item k
  if constexpr (LINE) {
    if (a.overlap && k == 1) {
      pdl_wait_prev();
      if (!a.late) pdl_allow_next();
    }
    if (a.late && last && (k > 0 || !a.overlap)) pdl_allow_next();
  }
}
template <bool LINE>
__device__ __forceinline__ void chain_end(const PassArgs& a, bool one_item) {
  if constexpr (LINE) {
    if (a.overlap && one_item) {
      pdl_wait_prev();
      pdl_allow_next();
    }
  }
}

// Copy one slot descriptor into shared memory (word by word).
__device__ __forceinline__ void load_slot(Slot* dst, const Slot* __restrict__ src) {
  static_assert(sizeof(Slot) % 4 == 0, "slot size");
  const int* s = reinterpret_cast<const int*>(src);
  int* d = reinterpret_cast<int*>(dst);
  for (int w = threadIdx.x; w < (int)(sizeof(Slot) / 4); w += blockDim.x) d[w] = s[w];
}

// Request one slot descriptor into shared memory (8-byte cp.async by the
// first threads of the block); it lands with the caller's next commit group.
__device__ __forceinline__ void copy_slot(Slot* dst, const Slot* src) {
  static_assert(sizeof(Slot) % 8 == 0, "slot size");
  constexpr int W = sizeof(Slot) / 8;
  if (threadIdx.x < W)
    cp_async<8>(reinterpret_cast<char*>(dst) + 8 * threadIdx.x,
                reinterpret_cast<const char*>(src) + 8 * threadIdx.x);
}

// An item read ahead into registers (slot < 0: none).
__device__ __forceinline__ Item item_at(const PassArgs& a, int it) {
  return it < a.n_items ? a.items[a.reverse ? a.n_items - 1 - it : it] : Item{-1, 0};
}

// Kernels of TH-thread CTAs walk sub-items: an item (kThreads threads' lines)
// is pass_split of them, and sub-item j is part j % SPLIT of item j / SPLIT.
__host__ __device__ constexpr int pass_split(int N, int E, int TH) {
  return lines_per_item(N, E) / lines_per_item_t(N, E, TH);
}
template <int SPLIT>
__device__ __forceinline__ Item sub_item(const PassArgs& a, int j) {
  Item i = item_at(a, j / SPLIT);
  i.block = SPLIT * i.block + j % SPLIT;
  return i;
}

// E = 32 keeps 64 registers of line data per thread plus the prefetched
// psi/support: one 256-thread CTA per SM with up to 255 registers.  E = 16
// halves that and runs two CTAs per SM.
// smallest E instantiated for size N (8, or N/256 when a line needs more threads)
constexpr int kSmallE(int N) { return (N / kThreads > 8) ? N / kThreads : (N >= 8 ? 8 : N); }

// Resident CTAs per SM each kernel is compiled for (registers per thread =
// 64K / (256 * this)): E = 32 needs ~240 registers, E = 16 fits 128 and E = 8
// fits 64 (four CTAs, 32 warps per SM).
constexpr int min_blocks_for(int E, bool row) {
  return E >= 32 ? 1 : (E >= 16 ? 2 : 4);
}

// Build this size's per-stage twiddle tables in shared memory (once per
// persistent CTA); returns their address.
template <int N, int E>
__device__ __forceinline__ const float2* stage_twiddles(float2* tw, const float2* __restrict__ tw_all) {
  build_stage_twiddles<N, E>(tw, tw_all + N);
  __syncthreads();
  return tw;
}

// Row pass: persistent CTAs walk their items; within a CTA each line group
// (RowGroup) walks them on its own, with its own ring of slot descriptors
// (items k, k+1, k+2) and its own rows of every buffer, so no step of the
// loop waits for the whole block.  The group's rows of the next item's G are
// requested as soon as its psi rows of the current item have been consumed,
// together with the descriptor of the item after that; the item list is read
// ahead into registers.
template <int N, int E, int TH, bool LINE>
__global__ void __launch_bounds__(TH, min_blocks_for(E, true) * (kThreads / TH))
    row_pass_kernel(PassArgs a) {
  using SM = RowSmem<N, E, TH>;
  using RG = RowGroup<N, E, TH>;
  constexpr int SPLIT = pass_split(N, E, TH);
  extern __shared__ float2 smem[];
  __shared__ __align__(16) Slot sl[3][RG::NG];
  const int tick = (a.tick_base ? *a.tick_base : 0) + a.tick_off;
  const float2* tw = stage_twiddles<N, E>(smem + SM::kTw, a.tw);  // block barrier
  float* sup_tile = reinterpret_cast<float*>(smem + SM::kSup);
  const int g = threadIdx.x / RG::GT;
  const int gtid = threadIdx.x - g * RG::GT;
  const int n_sub = SPLIT * a.n_items;
  int it = blockIdx.x;
  if (g >= RG::NG || it >= n_sub) return;  // no lines for this group, or no items
  const auto sync = RG::sync(g);
  const int G = gridDim.x;
  Item i0 = sub_item<SPLIT>(a, it), i1 = sub_item<SPLIT>(a, it + G), i2 = sub_item<SPLIT>(a, it + 2 * G);
  load_slot_by<RG::GT>(&sl[0][g], &a.slots[i0.slot], gtid);
  if (i1.slot >= 0) load_slot_by<RG::GT>(&sl[1][g], &a.slots[i1.slot], gtid);
  sync();
  chain_start<LINE>(a);  // the planes are the previous pass's output
  bool ready = false;
  if (row_finishes(sl[0][g], tick)) {
    prefetch_row_tile<N, E, TH>(sl[0][g], i0.block, smem, g, gtid);
    asm volatile("cp.async.commit_group;" ::: "memory");
    ready = true;
  }
  int par = 0;
  const bool one_item = it + G >= n_sub;
  for (int k = 0; it < n_sub; it += G, ++k) {
    const Item i3 = sub_item<SPLIT>(a, it + 3 * G);
    chain_top<LINE>(a, k, it + G >= n_sub);
    sync();  // the group is done with its rows of both buffers and with item k-1's slot entry
    const Slot& s = sl[k % 3][g];
    auto copy_ring = [&]() {  // item k+2's descriptor into item k-1's entry
      if (i2.slot >= 0) copy_slot_by(&sl[(k + 2) % 3][g], &a.slots[i2.slot], gtid);
    };
    const int step = tick - s.start_tick;
    bool next_ready = false;
    if (step >= 0 && step <= s.n_iter) {
      next_ready = row_item<N, E, TH>(s, step, i0.block, smem + par * SM::kB, smem + (par ^ 1) * SM::kB,
                                  ready, sup_tile, i1.slot >= 0 ? &sl[(k + 1) % 3][g] : nullptr,
                                  i1.block, tick, tw, g, gtid, copy_ring);
    }
    if (next_ready) {
      ready = true;
      par ^= 1;
    } else {
      // nothing is in flight for the next item: it keeps its G rows where
      // they are (global memory) and the buffers need not swap
      copy_ring();
      asm volatile("cp.async.commit_group;" ::: "memory");
      cp_async_wait_all();
      ready = false;
    }
    i0 = i1;
    i1 = i2;
    i2 = i3;
  }
  chain_end<LINE>(a, one_item);
  cp_async_wait_all();
}

// Column pass: persistent CTAs walk their items with one block barrier per
// item.  At the top of item k (after waiting for its G tile and the barrier)
// the block reads the inputs of the last stage of item k-1's inverse
// transforms from the other buffer, requests item k+1's G tile into that
// buffer in the same mapping (each column's threads also request item k's
// modulus), then finishes item k-1 straight into global memory; item k's
// columns then run with no block-wide synchronisation.  Slot descriptors go
// round a ring of three (items k, k+1 and k+2, whose copy is requested during
// item k), and the item list is read ahead into registers, so no step of the
// loop waits on a global load.
template <int N, int E, int TH, bool LINE>
__global__ void __launch_bounds__(TH, min_blocks_for(E, false) * (kThreads / TH))
    col_pass_kernel(PassArgs a) {
  using CS = ColSmem<N, E, TH>;
  constexpr int SPLIT = pass_split(N, E, TH);
  extern __shared__ float2 smem[];
  __shared__ __align__(16) Slot sl[3];
  const int tick = (a.tick_base ? *a.tick_base : 0) + a.tick_off;
  const float2* tw = stage_twiddles<N, E>(smem + CS::kTw, a.tw);  // block barrier
  float* mod = reinterpret_cast<float*>(smem + CS::kMod);
  const int n_sub = SPLIT * a.n_items;
  int it = blockIdx.x;
  if (it >= n_sub) return;  // the whole block leaves together
  const int G = gridDim.x;
  // items k, k+1, k+2 held in registers; item k+3 is read during item k
  Item i0 = sub_item<SPLIT>(a, it), i1 = sub_item<SPLIT>(a, it + G), i2 = sub_item<SPLIT>(a, it + 2 * G);
  load_slot(&sl[0], &a.slots[i0.slot]);
  if (i1.slot >= 0) load_slot(&sl[1], &a.slots[i1.slot]);
  __syncthreads();
  chain_start<LINE>(a);  // the planes (and the transposed modulus) are earlier kernels' output
  copy_col_g<N, E, TH>(sl[0], i0.block, tick, smem);
  asm volatile("cp.async.commit_group;" ::: "memory");
  float2* pend = nullptr;  // plane whose last stage is left in the other buffer
  int pend_block = 0;
  int b = 0;
  const bool one_item = it + G >= n_sub;
  for (int k = 0; it < n_sub; it += G, ++k, b ^= 1) {
    const Item i3 = sub_item<SPLIT>(a, it + 3 * G);
    chain_top<LINE>(a, k, it + G >= n_sub);
    cp_async_wait_all();  // this item's G tile and item k+1's slot descriptor
    __syncthreads();      // ... visible to all; the previous item is finished
    float2* other = smem + (b ^ 1) * CS::kB;
    const Slot& s = sl[k % 3];
    auto copies = [&]() {
      copy_col_mod<N, E, TH>(s, i0.block, tick, mod);
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (i1.slot >= 0) copy_col_g<N, E, TH>(sl[(k + 1) % 3], i1.block, tick, other);
      if (i2.slot >= 0) copy_slot(&sl[(k + 2) % 3], &a.slots[i2.slot]);  // item k-1's entry
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (pend)
      col_last_stage<N, E, TH>(pend, pend_block, other, tw, copies);
    else
      copies();
    pend = nullptr;
    if (col_live(s, tick)) {
      pend = col_item<N, E, TH>(s, tick - s.start_tick, i0.block, smem + b * CS::kB, mod, tw);
      pend_block = i0.block;
    }
    i0 = i1;
    i1 = i2;
    i2 = i3;
  }
  chain_end<LINE>(a, one_item);
  __syncthreads();
  if (pend) col_last_stage<N, E, TH>(pend, pend_block, smem + (b ^ 1) * CS::kB, tw, [] {});
  cp_async_wait_all();
}

// Single-buffered column pass: CTAs of kColSbThreads threads, each walking
// half items (C/2 columns; sub-item j is half j & 1 of item j >> 1), with one
// set of column strips (exchanges and the last stage's inputs) and one
// row-major staging buffer for the G tile (96 KB in all), so two CTAs share
// an SM where the pipelined form fits one.  Two per SM (8 warps, up to 255
// registers) run fastest: with the strips alone (55 KB), three per SM at 170
// registers and four at 128 were slower, giving up per-warp parallelism in
// registers for warps that do not make up for it.
// Per half item: wait for the tile and modulus, barrier, forward transform
// (its first stage reading the staging buffer), projection and inverse
// transform up to its last stage (col_item), barrier, then the last stage in
// the row mapping straight to global memory while the next half's modulus
// (into the strips it has finished with) and tile (into the staging buffer,
// 16-byte copies of whole row segments) are requested; the other CTA on the
// SM covers the copies.  Used where it measures faster (512^2 at E = 32; at
// 1024^2 and above its narrower tiles lose more than the extra warps gain).
constexpr int kColSbThreads = 128;
__host__ __device__ constexpr bool col_single_buffered(int N, int E) { return N == 512 && E == 32; }
// column-pass work units per item
__host__ __device__ constexpr int col_split(int N, int E) {
  return col_single_buffered(N, E) ? pass_split(N, E, kColSbThreads) : 1;
}

template <int N, int E, bool LINE>
__global__ void __launch_bounds__(kColSbThreads, 2) col_pass_sb_kernel(PassArgs a) {
  constexpr int TH = kColSbThreads;
  constexpr int SPLIT = col_split(N, E);
  using CS = ColSmem<N, E, TH, 1>;
  static_assert(SPLIT * CS::C == lines_per_item(N, E), "an item is SPLIT whole sub-items");
  extern __shared__ float2 smem[];
  __shared__ __align__(16) Slot sl[3];
  const int tick = (a.tick_base ? *a.tick_base : 0) + a.tick_off;
  const float2* tw = stage_twiddles<N, E>(smem + CS::kTw, a.tw);  // block barrier
  float* mod = reinterpret_cast<float*>(smem + CS::kMod);
  float2* tile = smem + ColTile<N, E, TH>::kOff;
  const int n_sub = SPLIT * a.n_items;
  int it = blockIdx.x;
  if (it >= n_sub) return;  // the whole block leaves together
  const int G = gridDim.x;
  // sub-items k, k+1, k+2 held in registers; sub-item k+3 is read during k
  Item i0 = sub_item<SPLIT>(a, it), i1 = sub_item<SPLIT>(a, it + G), i2 = sub_item<SPLIT>(a, it + 2 * G);
  load_slot(&sl[0], &a.slots[i0.slot]);
  if (i1.slot >= 0) load_slot(&sl[1], &a.slots[i1.slot]);
  __syncthreads();
  chain_start<LINE>(a);  // the planes (and the transposed modulus) are earlier kernels' output
  copy_col_mod<N, E, TH>(sl[0], i0.block, tick, mod);
  asm volatile("cp.async.commit_group;" ::: "memory");
  if (col_projects(sl[0], tick)) copy_col_tile<N, E, TH>(sl[0].g, i0.block, tile);
  asm volatile("cp.async.commit_group;" ::: "memory");
  const bool one_item = it + G >= n_sub;
  for (int k = 0; it < n_sub; it += G, ++k) {
    const Item i3 = sub_item<SPLIT>(a, it + 3 * G);
    chain_top<LINE>(a, k, it + G >= n_sub);
    cp_async_wait_all();  // this sub-item's modulus and tile, sub-item k+1's descriptor
    __syncthreads();      // ... visible to all; the previous sub-item is finished
    const Slot& s = sl[k % 3];
    float2* pend = nullptr;
    if (col_live(s, tick))
      pend = col_item<N, E, TH, true>(s, tick - s.start_tick, i0.block, smem, mod, tw, tile);
    __syncthreads();  // last-stage inputs in the strips; the modulus strips and the tile consumed
    auto copies = [&]() {
      if (i1.slot >= 0) copy_col_mod<N, E, TH>(sl[(k + 1) % 3], i1.block, tick, mod);
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (i1.slot >= 0 && col_projects(sl[(k + 1) % 3], tick))
        copy_col_tile<N, E, TH>(sl[(k + 1) % 3].g, i1.block, tile);
      if (i2.slot >= 0) copy_slot(&sl[(k + 2) % 3], &a.slots[i2.slot]);  // sub-item k-1's entry
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (pend)
      col_last_stage<N, E, TH>(pend, i0.block, smem, tw, copies);
    else
      copies();
    i0 = i1;
    i1 = i2;
    i2 = i3;
  }
  chain_end<LINE>(a, one_item);
  cp_async_wait_all();
}

// Lone trials and small batches: when the items of kThreads-thread CTAs are
// too few for the chip (a 256^2 trial is 16 of them at E = 16, on 16 of 148
// SMs), both passes run in kSmallThreads-thread CTAs on quarter items (half items at
// 64^2 with E = 32) instead (the same kernels, so bitwise the same results): a lone
// pass is bound by its warps' own instruction chains, which run faster with 2 warps
// on an SM than with 8.  Taken up to two small CTAs per SM (one at 512^2, where two of them
// are as slow as a large one); measured, us per iteration in large / small
// CTAs, small CTAs in brackets: 256^2 x 1 8.5 / 6.1 [64], x 2 8.6 / 7.4 [128],
// x 4 8.7 / 8.5 [256], x 8 9.3 / 10.5 [512]; 512^2 x 1 12.8 / 11.2 [128], x 4
// 16.1 / 17.4 [512]; 128^2 x 1 14.7 / 8.4 [8], x 36 15.5 / 12.1 [288]; 64^2 x
// 40 11.9 / 9.4 [80].  Sizes that run side by side keep the large CTAs: small ones
// of one size take the other's SMs (30 x 128^2 beside 512^2, 60 iterations: 1340 us,
// 1306 with large ones; 4 x 256^2 beside 2 x 1024^2 2266 and 2130).  At 1024^2 a
// trial is 128 items already, and at 512^2 with E < 32 one trial is more small CTAs
// than the rule takes.
constexpr int kSmallThreads = 64;
__host__ __device__ constexpr bool has_small_ctas(int N, int E) {
  return N >= 64 && (N < 512 || (N == 512 && E == 32)) && pass_split(N, E, kSmallThreads) > 1;
}

// pass kinds: 0 column, 1 row, the same in small CTAs, and the same (large) for
// lines of several sizes
enum {
  kPassCol = 0,
  kPassRow = 1,
  kPassColSmall = 2,
  kPassRowSmall = 3,
  kPassColLine = 4,
  kPassRowLine = 5,
  kPassKinds = 6
};

template <int N, int E, int TH>
constexpr size_t col_smem_bytes() {
  if constexpr (TH == kColSbThreads)
    return (size_t)ColTile<N, E, TH>::kTotal * sizeof(float2);
  else
    return (size_t)ColSmem<N, E, TH>::kTotal * sizeof(float2);
}
template <int N, int E, int TH>
constexpr size_t row_smem_bytes() { return (size_t)RowSmem<N, E, TH>::kTotal * sizeof(float2); }

// Call f(kernel, threads, dynamic shared memory) for a pass kind of (N, E);
// cudaErrorInvalidValue for one that is not compiled.
template <int N, int E, class F>
cudaError_t with_pass_kernel(int which, F&& f) {
  auto large = [&](auto line, bool col) {
    constexpr bool LINE = decltype(line)::value;
    if (!col)
      return f(row_pass_kernel<N, E, kThreads, LINE>, kThreads, row_smem_bytes<N, E, kThreads>());
    if constexpr (col_single_buffered(N, E))
      return f(col_pass_sb_kernel<N, E, LINE>, kColSbThreads, col_smem_bytes<N, E, kColSbThreads>());
    else
      return f(col_pass_kernel<N, E, kThreads, LINE>, kThreads, col_smem_bytes<N, E, kThreads>());
  };
  if (which == kPassCol || which == kPassRow) return large(std::false_type{}, which == kPassCol);
  if (which == kPassColLine || which == kPassRowLine)
    return large(std::true_type{}, which == kPassColLine);
  if constexpr (has_small_ctas(N, E)) {
    if (which == kPassColSmall)
      return f(col_pass_kernel<N, E, kSmallThreads, false>, kSmallThreads,
               col_smem_bytes<N, E, kSmallThreads>());
    if (which == kPassRowSmall)
      return f(row_pass_kernel<N, E, kSmallThreads, false>, kSmallThreads,
               row_smem_bytes<N, E, kSmallThreads>());
  }
  return cudaErrorInvalidValue;
}

template <int N, int E>
cudaError_t launch_pass_t(int which, int grid, cudaStream_t st, const PassArgs& a) {
  return with_pass_kernel<N, E>(which, [&](void (*k)(PassArgs), int threads, size_t smem) {
    return launch_pdl(k, grid, threads, smem, st, a);
  });
}

// occupancy[kind] = resident CTAs per SM of each pass kind (0: not compiled)
template <int N, int E>
cudaError_t pass_setup_t(int* occupancy) {
  for (int which = 0; which < kPassKinds; ++which) {
    occupancy[which] = 0;
    if ((which == kPassColSmall || which == kPassRowSmall) && !has_small_ctas(N, E)) continue;
    const cudaError_t e =
        with_pass_kernel<N, E>(which, [&](void (*k)(PassArgs), int threads, size_t smem) {
          cudaError_t r = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem);
          if (r != cudaSuccess) return r;
          return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occupancy[which], k, threads, smem);
        });
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Does a segment of `items` items of (N, E) run in small CTAs?
inline bool use_small_ctas(int N, int E, int items, int sms) {
  return has_small_ctas(N, E) && items * pass_split(N, E, kSmallThreads) <= (N <= 256 ? 2 : 1) * sms;
}

// work units of one item in each pass kind
inline int pass_units(int N, int E, int which) {
  if (which == kPassCol || which == kPassColLine) return col_split(N, E);
  if (which == kPassRow || which == kPassRowLine) return 1;
  return pass_split(N, E, kSmallThreads);
}

// Per-size entry points (defined in sp_engine_n<N>.cu).  E is clamped to N.
#define SP_DECLARE_SIZE(N)                                                                  \
  cudaError_t launch_pass_n##N(int E, int which, int grid, cudaStream_t st, const PassArgs& a); \
  cudaError_t pass_setup_n##N(int E, int* occupancy);
SP_DECLARE_SIZE(8)
SP_DECLARE_SIZE(16)
SP_DECLARE_SIZE(32)
SP_DECLARE_SIZE(64)
SP_DECLARE_SIZE(128)
SP_DECLARE_SIZE(256)
SP_DECLARE_SIZE(512)
SP_DECLARE_SIZE(1024)
SP_DECLARE_SIZE(2048)
SP_DECLARE_SIZE(4096)

#define SP_DEFINE_SIZE(N)                                                                    \
  cudaError_t launch_pass_n##N(int E, int which, int grid, cudaStream_t st, const PassArgs& a) { \
    if (E >= 32 && N >= 32) return launch_pass_t<N, (N >= 32 ? 32 : N)>(which, grid, st, a);   \
    if (E >= 16 && N >= 16) return launch_pass_t<N, (N >= 16 ? 16 : N)>(which, grid, st, a);   \
    return launch_pass_t<N, kSmallE(N)>(which, grid, st, a);                                  \
  }                                                                                          \
  cudaError_t pass_setup_n##N(int E, int* occupancy) {                                       \
    if (E >= 32 && N >= 32) return pass_setup_t<N, (N >= 32 ? 32 : N)>(occupancy);            \
    if (E >= 16 && N >= 16) return pass_setup_t<N, (N >= 16 ? 16 : N)>(occupancy);            \
    return pass_setup_t<N, kSmallE(N)>(occupancy);                                            \
  }

// E actually used for a requested E at size N: 32, 16 or 8, at most N, and at
// least N/256 so that a line needs no more than the CTA's 256 threads
inline int effective_e(int N, int E) {
  int e = (E >= 32 && N >= 32) ? 32 : ((E >= 16 && N >= 16) ? 16 : (N >= 8 ? 8 : N));
  while (N / e > kThreads) e *= 2;
  return e;
}

}  // namespace sp
