// Exact magnitude top-k selection (unsorted), fused with the error-feedback write.
//
// The sparsifying reducers of the research harness call torch.topk on |x|, gather the values,
// then copy the tensor and zero the selected entries (paper-code/gradient_reducers.py:226-253,
// 296-324). Here one radix select does all of it in four launches over x:
//   3 x histogram pass over the 31-bit magnitude key (bits 30..20, 19..9, 8..0), each pass
//       restricted to the keys that matched the digits chosen so far (every CTA re-derives the
//       chosen digit from the previous histogram, so no separate "scan" launches are needed);
//   1 x compaction: keys above the threshold key are all taken, keys equal to it fill the rest;
//       writes values[k], positions[k] (int32) and, optionally, memory = x with the taken
//       entries zeroed.
// The magnitude key of a finite float orders like |x|. The output order is unspecified (as with
// torch.topk(sorted=False)); among exact ties at the threshold any subset may be taken.
#include "psgd_common.cuh"

namespace {

constexpr int TK_THREADS = 512;
constexpr int TK_BINS0 = 2048, TK_BINS1 = 2048, TK_BINS2 = 512;

constexpr int TK_FOUND = 1024;   // selected entries a block collects before it hands them out

// workspace layout (ints): hist0[2048] hist1[2048] hist2[512] | cnt_gt, cnt_eq
constexpr int TK_WS_INTS = TK_BINS0 + TK_BINS1 + TK_BINS2 + 8;

struct Pick {
  unsigned prefix;   // digits chosen so far, already shifted into place
  long long remain;  // how many entries still to take inside the chosen bin
};

__device__ __forceinline__ unsigned tk_key(float v) { return __float_as_uint(v) & 0x7FFFFFFFu; }

// Scan a histogram from its top bin down until `remain` entries are covered; returns the bin and
// updates `remain` to the number to take inside it. Executed redundantly by thread 0 of each CTA.
__device__ int tk_choose(const int* hist, int bins, long long& remain) {
  for (int b = bins - 1; b >= 0; --b) {
    const int c = hist[b];
    if (remain <= c) return b;
    remain -= c;
  }
  return 0;
}

__device__ void tk_derive(const int* ws, int upto, long long k, Pick& p) {
  p.prefix = 0u;
  p.remain = k;
  if (upto >= 1) p.prefix |= (unsigned)tk_choose(ws, TK_BINS0, p.remain) << 20;
  if (upto >= 2) p.prefix |= (unsigned)tk_choose(ws + TK_BINS0, TK_BINS1, p.remain) << 9;
  if (upto >= 3) p.prefix |= (unsigned)tk_choose(ws + TK_BINS0 + TK_BINS1, TK_BINS2, p.remain);
}

// pass = 0, 1, 2
__global__ void __launch_bounds__(TK_THREADS) psgd_topk_hist_kernel(const float* __restrict__ x, long long n, long long k,
                                                                     int* __restrict__ ws, int pass) {
  __shared__ int sh[TK_BINS0];
  __shared__ Pick pick;
  const int bins = pass == 2 ? TK_BINS2 : TK_BINS0;
  for (int b = threadIdx.x; b < bins; b += TK_THREADS) sh[b] = 0;
  if (threadIdx.x == 0) tk_derive(ws, pass, k, pick);
  __syncthreads();
  const unsigned prefix = pick.prefix;
  const unsigned mask = pass == 0 ? 0u : (pass == 1 ? 0x7FF00000u : 0x7FFFFE00u);
  const int shift = pass == 0 ? 20 : (pass == 1 ? 9 : 0);
  const unsigned digit_mask = pass == 2 ? 0x1FFu : 0x7FFu;
  const long long stride = (long long)gridDim.x * TK_THREADS;
  for (long long i = (long long)blockIdx.x * TK_THREADS + threadIdx.x; i < n; i += stride) {
    const unsigned key = tk_key(__ldg(x + i));
    if ((key & mask) == prefix) atomicAdd(&sh[(key >> shift) & digit_mask], 1);
  }
  __syncthreads();
  int* hist = ws + (pass == 0 ? 0 : (pass == 1 ? TK_BINS0 : TK_BINS0 + TK_BINS1));
  for (int b = threadIdx.x; b < bins; b += TK_THREADS)
    if (sh[b]) atomicAdd(hist + b, sh[b]);
}

__global__ void __launch_bounds__(TK_THREADS) psgd_topk_compact_kernel(const float* __restrict__ x, long long n, long long k,
                                                                        int* __restrict__ ws, float* __restrict__ values,
                                                                        int* __restrict__ positions,
                                                                        float* __restrict__ memory) {
  __shared__ Pick pick;
  if (threadIdx.x == 0) tk_derive(ws, 3, k, pick);
  __syncthreads();
  const unsigned threshold = pick.prefix;
  const long long take_equal = pick.remain;       // entries with key == threshold to take
  const long long base_equal = k - take_equal;    // entries with key > threshold come first
  int* cnt_gt = ws + TK_BINS0 + TK_BINS1 + TK_BINS2;
  int* cnt_eq = cnt_gt + 1;
  const long long stride = (long long)gridDim.x * TK_THREADS;
  for (long long i = (long long)blockIdx.x * TK_THREADS + threadIdx.x; i < n; i += stride) {
    const float v = __ldg(x + i);
    const unsigned key = tk_key(v);
    long long slot = -1;
    if (key > threshold) slot = atomicAdd(cnt_gt, 1);
    else if (key == threshold) {
      const long long e = atomicAdd(cnt_eq, 1);
      if (e < take_equal) slot = base_equal + e;
    }
    if (slot >= 0) {
      values[slot] = v;
      positions[slot] = (int)i;
    }
    if (memory) memory[i] = slot >= 0 ? 0.f : v;
  }
}

}  // namespace

PSGD_API int psgd_topk_workspace_ints() { return TK_WS_INTS; }

// Top-k of |x| over n float32 entries (k <= n, n < 2^31): values[k], positions[k] (int32), and
// if `memory` is non-null, memory[i] = 0 where taken else x[i] (memory may alias x only if it IS x).
PSGD_API int psgd_topk_abs(const float* x, long long n, long long k, int* workspace, float* values, int* positions,
                           float* memory, cudaStream_t stream) {
  if (n <= 0 || k <= 0) return 0;
  if (k > n || n >= (1ll << 31)) {
    psgd_set_error("psgd_topk_abs: need 0 < k <= n < 2^31 (k = %lld, n = %lld)", k, n);
    return -1;
  }
  PSGD_CUDA_OK(cudaMemsetAsync(workspace, 0, sizeof(int) * TK_WS_INTS, stream));
  long long blocks = (n + TK_THREADS * 8 - 1) / (TK_THREADS * 8);
  if (blocks > 592) blocks = 592;
  for (int pass = 0; pass < 3; ++pass)
    psgd_topk_hist_kernel<<<(int)blocks, TK_THREADS, 0, stream>>>(x, n, k, workspace, pass);
  psgd_topk_compact_kernel<<<(int)blocks, TK_THREADS, 0, stream>>>(x, n, k, workspace, values, positions, memory);
  PSGD_CUDA_OK(cudaGetLastError());
  return 0;
}

// ---------------------------------------------------------------------------------------------
// The same selection for MANY tensors at once, with two passes over them. The per-tensor reducer of the harness calls the
// selection once per parameter (62 times for ResNet-18, paper-code/gradient_reducers.py:226-253),
// which is launch-bound; here a few launches serve the whole list. Every block serves one (tensor, chunk) pair
// from a block table; every tensor has its own histograms and counters in the workspace, and a digit is chosen
// by the whole block with a parallel suffix scan instead of one thread walking the bins:
//   1. histogram of the leading digit (11 of the 31 bits of |x|): one read;
//   2. every entry above the chosen digit is taken, every entry inside it becomes a candidate (a list of up to
//      `cap` per tensor), and `memory` is written: one read and one write;
//   3. one block per tensor finds the threshold among its candidates and takes those above it.
// A tensor with more candidates than its list holds (many entries of nearly equal size, or a large k) goes the long
// way instead: histograms of the second and the third digit over all entries in launches 2 and 3, and a
// compaction pass in launch 4, which has nothing to do for the others. How long a list one block should walk: ops/topk.py.
// Bound by the reads (L2 for a model of this size) and by what a block costs besides them, so as many blocks as run at a
// time, three per SM, serve the whole list. 62 tensors of ResNet-18 (45 MB), k = numel / 488: 68 us by three histogram passes and a
// compaction, 54 us by lists. With one worker launch 2 writes the dense output beside the memory (TopkItem::out), so that nothing
// is left to combine, every launch starts beside the end of the one before, and the workspace is cleared by the call
// before: the pass of the reducer 86 -> 55 us; with three blocks per SM in place of four, 51.5, of which 12 go
// to launch 1 (45 MB from HBM and as many additions in shared memory), 22 to launch 2 (135 MB), 8 to launch 3 and 2 to launch 4.
namespace {

struct TopkItem {
  const float* x;      // tensor, n entries
  float* memory;       // optional: x with the taken entries zeroed
  long long n;
  long long k;         // entries to take (1 <= k <= n)
  long long out_off;   // start of this tensor's k pairs in values / positions
  long long cand_off;  // start of its candidates, and
  long long cap;       // how many there may be
  float* out;          // optional: the taken entries at their places, zeros elsewhere
};

// Counters of a tensor behind its histograms: what launch 2 leaves for the launches behind it, besides what it counts.
enum TopkCounter { TK_TAKEN = 0, TK_EQUAL = 1, TK_LISTED = 2, TK_WAY = 3, TK_PREFIX = 4, TK_REMAIN = 5 };
constexpr int TK_SHORT = 1, TK_LONG = 2;   // TK_WAY: by the list of candidates, or by two more histograms

// Block-wide: walks `bins` (<= 2048, TK_THREADS threads x 4 bins) from the top until `remain` entries are
// covered; returns the bin in *bin_out and the number to take inside it in *remain_io. `scan`: one
// int per warp.
__device__ void tk_choose_block(const int* hist, int bins, long long* remain_io, int* bin_out, int* scan) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  // thread t owns bins [4t, 4t + 4), counted from the TOP: bin index bins - 1 - j
  int c[4], local = 0;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int j = 4 * t + u;
    c[u] = j < bins ? hist[bins - 1 - j] : 0;
    local += c[u];
  }
  // exclusive prefix sum: inside the warp by shuffles, then over the warps before this one
  int upto = local;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, upto, off);
    if (lane >= off) upto += v;
  }
  if (lane == 31) scan[warp] = upto;
  __syncthreads();
  int base = 0;
#pragma unroll
  for (int w = 0; w < TK_THREADS / 32; ++w) base += w < warp ? scan[w] : 0;
  const long long remain = *remain_io;
  const long long before = base + upto - local;   // entries in the bins above this thread's
  __syncthreads();
  if (before < remain && remain <= before + local) {    // exactly one thread
    long long left = remain - before;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (left <= c[u]) {
        *bin_out = bins - 1 - (4 * t + u);
        *remain_io = left;
        break;
      }
      left -= c[u];
    }
  }
  __syncthreads();
}

// Calls f(value, index) for every entry of a block's part of a tensor (parts are interleaved in runs of
// one block's accesses). 16-byte loads, four of a thread in flight, when the tensor allows them: a
// pass is bound by the reads, which the L2 cache or HBM serve at TB/s only with that much under way.
template <class F>
__device__ __forceinline__ void tk_for_each(const float* __restrict__ x, long long n, int part, int parts, F f) {
  const long long stride = (long long)parts * TK_THREADS;
  long long i = (long long)part * TK_THREADS + threadIdx.x;
  if (((uintptr_t)x & 15u) == 0) {
    const float4* x4 = reinterpret_cast<const float4*>(x);
    const long long n4 = n >> 2;
    for (; i < n4; i += 4 * stride) {
      float4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + u * stride < n4) q[u] = __ldg(x4 + i + u * stride);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + u * stride < n4) f(q[u], (i + u * stride) * 4, 4);
    }
    if (part == 0 && (long long)threadIdx.x < n - n4 * 4) {
      const long long e = n4 * 4 + threadIdx.x;
      f(make_float4(__ldg(x + e), 0.f, 0.f, 0.f), e, 1);
    }
  } else {
    for (; i < n; i += stride) f(make_float4(__ldg(x + i), 0.f, 0.f, 0.f), i, 1);
  }
}

// Digits `from` to `upto` - 1 of one tensor's threshold (block-wide; result in shared `pick`, which has those before).
__device__ void tk_derive_block(const int* ws, int from, int upto, long long k, Pick* pick, long long* remain_sh, int* bin_sh, int* scan) {
  if (threadIdx.x == 0) {
    if (from == 0) {
      pick->prefix = 0u;
      *remain_sh = k;
    }
    *bin_sh = 0;
  }
  __syncthreads();
  if (from < 1 && upto >= 1) {
    tk_choose_block(ws, TK_BINS0, remain_sh, bin_sh, scan);
    if (threadIdx.x == 0) pick->prefix |= (unsigned)(*bin_sh) << 20;
    __syncthreads();
  }
  if (from < 2 && upto >= 2) {
    tk_choose_block(ws + TK_BINS0, TK_BINS1, remain_sh, bin_sh, scan);
    if (threadIdx.x == 0) pick->prefix |= (unsigned)(*bin_sh) << 9;
    __syncthreads();
  }
  if (from < 3 && upto >= 3) {
    tk_choose_block(ws + TK_BINS0 + TK_BINS1, TK_BINS2, remain_sh, bin_sh, scan);
    if (threadIdx.x == 0) pick->prefix |= (unsigned)(*bin_sh);
    __syncthreads();
  }
  if (threadIdx.x == 0) pick->remain = *remain_sh;
  __syncthreads();
}

// Four copies of a block's histogram, by lane: the leading digit of a gradient takes a few dozen values, and
// lanes that meet on one address are served one after another. The copies of a bin are added up by one 16-byte
// access, so whatever holds this has to have its alignment.
struct alignas(16) Bins {
  int c[TK_BINS0 * 4];
};

// Histogram of digit `pass` of the entries that agree with the digits chosen so far (block-wide).
__device__ void tk_histogram(const TopkItem& item, int part, int parts, int* ws, int pass, unsigned prefix, Bins& shared) {
  int* sh = shared.c;
  const int bins = pass == 2 ? TK_BINS2 : TK_BINS0;
  for (int b = threadIdx.x; b < bins * 4; b += TK_THREADS) sh[b] = 0;
  __syncthreads();
  const unsigned mask = pass == 0 ? 0u : (pass == 1 ? 0x7FF00000u : 0x7FFFFE00u);
  const int shift = pass == 0 ? 20 : (pass == 1 ? 9 : 0);
  const unsigned digit_mask = pass == 2 ? 0x1FFu : 0x7FFu;
  int* mine = sh + (threadIdx.x & 3);
  tk_for_each(item.x, item.n, part, parts, [&](const float4& q, long long, int count) {
    const float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const unsigned key = tk_key(v[j]);
      if (j < count && (key & mask) == prefix) atomicAdd(mine + 4 * ((key >> shift) & digit_mask), 1);
    }
  });
  __syncthreads();
  int* hist = ws + (pass == 0 ? 0 : (pass == 1 ? TK_BINS0 : TK_BINS0 + TK_BINS1));
  for (int b = threadIdx.x; b < bins; b += TK_THREADS) {
    const int4 c = reinterpret_cast<const int4*>(sh)[b];
    const int total = c.x + c.y + c.z + c.w;
    if (total) atomicAdd(hist + b, total);
  }
}

__global__ void __launch_bounds__(TK_THREADS) psgd_topk_many_hist_kernel(const TopkItem* __restrict__ items, const int* __restrict__ block_item,
                                                                          const int* __restrict__ block_part, const int* __restrict__ item_parts,
                                                                          int* __restrict__ ws_all) {
  __shared__ Bins sh;
  psgd_launch_dependents();
  const int it = block_item[blockIdx.x];
  tk_histogram(items[it], block_part[blockIdx.x], item_parts[it], ws_all + (long long)it * TK_WS_INTS, 0, 0u, sh);
}

// Entries a block has found, handed out with one addition to a counter of the tensor per block: thousands
// of additions to one address would be served one after another.
struct Found {
  float v[TK_FOUND];
  int p[TK_FOUND];
  int count, base;
};
// `room`: entries of val / pos. A tensor has no more than that unless something writes it during the call.
__device__ __forceinline__ void tk_put(Found& f, int* counter, float* val, int* pos, long long room, float v, int p) {
  const int slot = atomicAdd(&f.count, 1);
  if (slot < TK_FOUND) {
    f.v[slot] = v;
    f.p[slot] = p;
  } else {
    const int at = atomicAdd(counter, 1);
    if (at < room) {
      val[at] = v;
      pos[at] = p;
    }
  }
}
__device__ void tk_hand_out(Found& f, int* counter, float* val, int* pos, long long room) {   // block-wide
  __syncthreads();
  const int mine = min(f.count, TK_FOUND);
  if (threadIdx.x == 0 && mine) f.base = atomicAdd(counter, mine);
  __syncthreads();
  for (int e = threadIdx.x; e < mine && f.base + e < room; e += TK_THREADS) {
    val[f.base + e] = f.v[e];
    pos[f.base + e] = f.p[e];
  }
}

union SplitScratch {
  Bins hist;
  struct { Found above, inside; } found;
};
static_assert(alignof(SplitScratch) % alignof(int4) == 0, "tk_histogram reads its bins by 16 bytes");

// Four entries of a tensor, or the first `count` of them.
__device__ __forceinline__ void tk_store(float* dst, bool wide, long long first, int count, const float* v) {
  if (count == 4 && wide) {
    *reinterpret_cast<float4*>(dst + first) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < count) dst[first + j] = v[j];
  }
}
// What a taken entry leaves in `out`: value / 1 added to zero, as the combination of several workers' entries has it.
__device__ __forceinline__ float tk_dense(float v) { return __fadd_rn(0.f, v); }

// Launch 2: what lies above the leading digit is taken, what lies in it is listed; or the second histogram.
// cand_v / cand_p: lists of candidates. ws_next: workspace of the call after this one, cleared here (a clearing of its own costs
// a call 3.5 us), or null.
__global__ void __launch_bounds__(TK_THREADS, 3) psgd_topk_many_split_kernel(const TopkItem* __restrict__ items, const int* __restrict__ block_item,
                                                                           const int* __restrict__ block_part, const int* __restrict__ item_parts,
                                                                           int* ws_all, int* __restrict__ ws_next,
                                                                           float* __restrict__ values, int* __restrict__ positions,
                                                                           float* __restrict__ cand_v, int* __restrict__ cand_p) {
  __shared__ SplitScratch sh;
  __shared__ int scan[TK_THREADS / 32];
  __shared__ Pick pick;
  __shared__ long long remain_sh;
  __shared__ int bin_sh;
  psgd_launch_dependents();
  const int it = block_item[blockIdx.x], part = block_part[blockIdx.x], parts = item_parts[it];
  const TopkItem item = items[it];
  int* ws = ws_all + (long long)it * TK_WS_INTS;
  psgd_wait_for_predecessor();
  if (ws_next)
    for (int e = part * TK_THREADS + threadIdx.x; e < TK_WS_INTS; e += parts * TK_THREADS) ws_next[(long long)it * TK_WS_INTS + e] = 0;
  tk_derive_block(ws, 0, 1, item.k, &pick, &remain_sh, &bin_sh, scan);
  const unsigned prefix = pick.prefix;
  const bool lists = ws[prefix >> 20] <= item.cap;
  int* counters = ws + TK_BINS0 + TK_BINS1 + TK_BINS2;
  if (part == 0 && threadIdx.x == 0) {
    counters[TK_WAY] = lists ? TK_SHORT : TK_LONG;
    counters[TK_PREFIX] = (int)prefix;
    counters[TK_REMAIN] = (int)remain_sh;
  }
  if (!lists) {
    tk_histogram(item, part, parts, ws, 1, prefix, sh.hist);
    return;
  }
  if (threadIdx.x == 0) sh.found.above.count = sh.found.inside.count = 0;
  __syncthreads();
  float* val = values + item.out_off;
  int* pos = positions + item.out_off;
  float* cv = cand_v + item.cand_off;
  int* cp = cand_p + item.cand_off;
  const bool wide_memory = ((uintptr_t)item.memory & 15u) == 0, wide_out = ((uintptr_t)item.out & 15u) == 0;
  tk_for_each(item.x, item.n, part, parts, [&](const float4& q, long long first, int count) {
    const float v[4] = {q.x, q.y, q.z, q.w};
    float rest[4], dense[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      rest[j] = v[j];
      dense[j] = 0.f;
      const unsigned key = tk_key(v[j]);
      if (j < count && key >= prefix) {
        if ((key & 0x7FF00000u) == prefix) {
          tk_put(sh.found.inside, counters + TK_LISTED, cv, cp, item.cap, v[j], (int)(first + j));
        } else {
          tk_put(sh.found.above, counters + TK_TAKEN, val, pos, item.k, v[j], (int)(first + j));
          rest[j] = 0.f;
          dense[j] = tk_dense(v[j]);
        }
      }
    }
    if (item.memory) tk_store(item.memory, wide_memory, first, count, rest);
    if (item.out) tk_store(item.out, wide_out, first, count, dense);
  });
  tk_hand_out(sh.found.above, counters + TK_TAKEN, val, pos, item.k);
  tk_hand_out(sh.found.inside, counters + TK_LISTED, cv, cp, item.cap);
}

// f(value, index) for every entry of a list from `from` on (block-wide), eight loads of a thread under way.
template <class F>
__device__ __forceinline__ void tk_walk(const float* list, int from, int n, F f) {
  for (int first = from + threadIdx.x; first < n; first += 8 * TK_THREADS) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (first + u * TK_THREADS < n) v[u] = __ldcg(list + first + u * TK_THREADS);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (first + u * TK_THREADS < n) f(v[u], first + u * TK_THREADS);
  }
}

// Launch 3: the threshold among a tensor's candidates, by its first block; or the third histogram. The launch may start while the one
// before still writes the list and the workspace: no read-only loads of them, here or in launch 4. One block walks a list alone,
// three times over, so nothing but the loads under way hides a latency: the first 4096 entries stay in registers.
__global__ void __launch_bounds__(TK_THREADS) psgd_topk_many_refine_kernel(const TopkItem* __restrict__ items, const int* __restrict__ block_item,
                                                                            const int* __restrict__ block_part, const int* __restrict__ item_parts,
                                                                            int* ws_all, float* __restrict__ values,
                                                                            int* __restrict__ positions, const float* cand_v,
                                                                            const int* cand_p) {
  __shared__ Bins bins_sh;
  __shared__ int scan[TK_THREADS / 32];
  __shared__ Pick pick;
  __shared__ long long remain_sh;
  __shared__ int bin_sh, above_sh, equal_sh;
  psgd_launch_dependents();
  const int it = block_item[blockIdx.x];
  const TopkItem item = items[it];
  int* ws = ws_all + (long long)it * TK_WS_INTS;
  const int* counters = ws + TK_BINS0 + TK_BINS1 + TK_BINS2;
  int* sh = bins_sh.c;
  if (block_part[blockIdx.x] == 0)
    for (int b = threadIdx.x; b < TK_BINS1 + TK_BINS2; b += TK_THREADS) sh[b] = 0;
  psgd_wait_for_predecessor();
  if (threadIdx.x == 0) {
    pick.prefix = (unsigned)counters[TK_PREFIX];
    remain_sh = counters[TK_REMAIN];
    above_sh = counters[TK_TAKEN];   // (nobody else takes entries of this tensor any more)
    equal_sh = 0;
  }
  const bool lists = counters[TK_WAY] == TK_SHORT;
  __syncthreads();
  if (!lists) {
    tk_derive_block(ws, 1, 2, item.k, &pick, &remain_sh, &bin_sh, scan);
    tk_histogram(item, block_part[blockIdx.x], item_parts[it], ws, 2, pick.prefix, bins_sh);
    return;
  }
  if (block_part[blockIdx.x] != 0) return;
  const int n = (int)min((long long)counters[TK_LISTED], item.cap);   // what launch 2 has listed
  const float* cv = cand_v + item.cand_off;
  const int* cp = cand_p + item.cand_off;
  constexpr int OWN = 8;
  float own[OWN];
#pragma unroll
  for (int u = 0; u < OWN; ++u) own[u] = (int)threadIdx.x + u * TK_THREADS < n ? __ldcg(cv + threadIdx.x + u * TK_THREADS) : 0.f;
  auto walk = [&](auto f) {
#pragma unroll
    for (int u = 0; u < OWN; ++u)
      if ((int)threadIdx.x + u * TK_THREADS < n) f(own[u], (int)threadIdx.x + u * TK_THREADS);
    tk_walk(cv, OWN * TK_THREADS, n, f);
  };
#pragma unroll 1
  for (int digit = 1; digit <= 2; ++digit) {
    const int bins = digit == 2 ? TK_BINS2 : TK_BINS1, shift = digit == 2 ? 0 : 9;
    const unsigned mask = digit == 2 ? 0x7FFFFE00u : 0x7FF00000u, prefix = pick.prefix;
    int* hist = sh + (digit == 2 ? TK_BINS1 : 0);
    walk([&](float v, int) {
      const unsigned key = tk_key(v);
      if ((key & mask) == prefix) atomicAdd(hist + ((key >> shift) & (unsigned)(bins - 1)), 1);
    });
    __syncthreads();
    tk_choose_block(hist, bins, &remain_sh, &bin_sh, scan);
    if (threadIdx.x == 0) pick.prefix = prefix | ((unsigned)bin_sh << shift);
    __syncthreads();
  }
  const unsigned threshold = pick.prefix;
  const long long take_equal = remain_sh, base_equal = item.k - take_equal;
  float* val = values + item.out_off;
  int* pos = positions + item.out_off;
  walk([&](float v, int e) {
    const unsigned key = tk_key(v);
    if (key < threshold) return;
    long long slot;
    if (key > threshold) {
      slot = atomicAdd(&above_sh, 1);
    } else {
      const long long eq = atomicAdd(&equal_sh, 1);
      if (eq >= take_equal) return;
      slot = base_equal + eq;
    }
    if (slot >= item.k) return;
    const int p = __ldcg(cp + e);
    val[slot] = v;
    pos[slot] = p;
    if (item.memory) item.memory[p] = 0.f;
    if (item.out) item.out[p] = tk_dense(v);
  });
}

// Launch 4: takes the k entries of a tensor with too many candidates.
__global__ void __launch_bounds__(TK_THREADS) psgd_topk_many_compact_kernel(const TopkItem* __restrict__ items, const int* __restrict__ block_item,
                                                                             const int* __restrict__ block_part, const int* __restrict__ item_parts,
                                                                             int* ws_all, float* __restrict__ values,
                                                                             int* __restrict__ positions) {
  __shared__ int scan[TK_THREADS / 32];
  __shared__ Pick pick;
  __shared__ long long remain_sh;
  __shared__ int bin_sh;
  __shared__ Found found;
  psgd_launch_dependents();
  const int it = block_item[blockIdx.x];
  const TopkItem item = items[it];
  int* ws = ws_all + (long long)it * TK_WS_INTS;
  int* counters = ws + TK_BINS0 + TK_BINS1 + TK_BINS2;
  psgd_wait_for_predecessor();
  if (counters[TK_WAY] == TK_SHORT) return;   // launch 3 took the rest
  if (threadIdx.x == 0) {
    pick.prefix = (unsigned)counters[TK_PREFIX];
    remain_sh = counters[TK_REMAIN];
    found.count = 0;
  }
  __syncthreads();
  tk_derive_block(ws, 1, 3, item.k, &pick, &remain_sh, &bin_sh, scan);
  const unsigned threshold = pick.prefix;
  const long long take_equal = pick.remain;
  const long long base_equal = item.k - take_equal;
  float* val = values + item.out_off;
  int* pos = positions + item.out_off;
  const bool wide_memory = ((uintptr_t)item.memory & 15u) == 0, wide_out = ((uintptr_t)item.out & 15u) == 0;
  tk_for_each(item.x, item.n, block_part[blockIdx.x], item_parts[it], [&](const float4& q, long long first, int count) {
    const float v[4] = {q.x, q.y, q.z, q.w};
    float rest[4], dense[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const unsigned key = tk_key(v[j]);
      bool taken = false;
      if (j < count && key >= threshold) {
        const int i = (int)(first + j);
        if (key > threshold) {
          tk_put(found, counters + TK_TAKEN, val, pos, item.k, v[j], i);
          taken = true;
        } else {
          const long long e = atomicAdd(counters + TK_EQUAL, 1);
          if (e < take_equal) {
            val[base_equal + e] = v[j];
            pos[base_equal + e] = i;
            taken = true;
          }
        }
      }
      rest[j] = taken ? 0.f : v[j];
      dense[j] = taken ? tk_dense(v[j]) : 0.f;
    }
    if (item.memory) tk_store(item.memory, wide_memory, first, count, rest);
    if (item.out) tk_store(item.out, wide_out, first, count, dense);
  });
  tk_hand_out(found, counters + TK_TAKEN, val, pos, item.k);
}

}  // namespace

PSGD_API int psgd_topk_item_bytes() { return (int)sizeof(TopkItem); }

// Top-k of |x| for `nitems` tensors in four launches. items: device array of TopkItem; block_item /
// block_part: device tables of `nblocks` entries (which tensor a block serves and which of that
// tensor's `item_parts[item]` interleaved parts); workspace: nitems * psgd_topk_workspace_ints() ints; next_workspace: null, or as
// many ints again that this call clears for the one after it, whose `workspace` they have to be (as `workspace` was cleared by the call before);
// cand_v / cand_p: room for the candidates of all tensors (`cand_off`, `cap` of the items). values / positions receive every
// tensor's k pairs at its `out_off`.
PSGD_API int psgd_topk_abs_many(const void* items, int nitems, const int* block_item, const int* block_part, const int* item_parts,
                                int nblocks, int* workspace, int* next_workspace, float* cand_v, int* cand_p, float* values, int* positions,
                                cudaStream_t stream) {
  if (nitems <= 0 || nblocks <= 0) return 0;
  const TopkItem* it = (const TopkItem*)items;
  if (next_workspace == nullptr) PSGD_CUDA_OK(cudaMemsetAsync(workspace, 0, sizeof(int) * (size_t)TK_WS_INTS * nitems, stream));
  int code = psgd_launch(psgd_topk_many_hist_kernel, nblocks, TK_THREADS, 0, stream, 0, it, block_item, block_part, item_parts, workspace);
  // the others start beside the end of the one before and wait for it
  if (code == 0)
    code = psgd_launch(psgd_topk_many_split_kernel, nblocks, TK_THREADS, 0, stream, 1, it, block_item, block_part, item_parts, workspace,
                       next_workspace, values, positions, cand_v, cand_p);
  if (code == 0)
    code = psgd_launch(psgd_topk_many_refine_kernel, nblocks, TK_THREADS, 0, stream, 1, it, block_item, block_part, item_parts, workspace,
                       values, positions, cand_v, cand_p);
  if (code == 0)
    code = psgd_launch(psgd_topk_many_compact_kernel, nblocks, TK_THREADS, 0, stream, 1, it, block_item, block_part, item_parts, workspace,
                       values, positions);
  return code;
}

// ---------------------------------------------------------------------------------------------
// Combine step of the top-k reducers: after the all-gather every worker holds W lists of
// (value, position) pairs and adds value / W into dense, zeroed outputs
// (paper-code/gradient_reducers.py:262-271 and 333-339 do it with one index_add_ per worker).
// One cooperative launch does the zero fill and the W scatter passes. Positions are unique
// within a worker's list, so a pass is race-free with plain read-modify-writes; a grid barrier
// separates the passes, which keeps the summation order (worker 0, 1, ...) fixed and the result
// bit-identical on every replica and in every run, unlike floating-point atomics.
namespace {

constexpr int SC_THREADS = 256;
constexpr int SC_MAX_SEGMENTS = 1024;

struct SparseSeg {
  float* out;        // dense output of this segment
  long long numel;   // its length
  long long end;     // end of this segment's pairs inside a worker's list (exclusive)
};

// Barrier over all CTAs of a cooperative launch on a counter that only grows (barrier b is passed
// once it reaches b * gridDim.x). Bounded: a CTA that waits longer than ~2 s gives up (all CTAs of a
// cooperative launch are resident, so this only guards against a broken launch).
__device__ bool sc_grid_barrier(unsigned* counter, unsigned& target) {
  __syncthreads();
  bool ok = true;
  if (threadIdx.x == 0) {
    target += gridDim.x;
    __threadfence();
    atomicAdd(counter, 1u);
    const unsigned long long t0 = psgd_globaltimer_ns();
    while (*(volatile unsigned*)counter < target) {
      if (psgd_globaltimer_ns() - t0 > 2000000000ull) { ok = false; break; }
    }
    __threadfence();
  }
  return __syncthreads_and(ok ? 1 : 0) != 0;
}

__global__ void __launch_bounds__(SC_THREADS) psgd_sparse_combine_kernel(const float* __restrict__ values,
                                                                          const int* __restrict__ positions, int workers,
                                                                          long long per_worker, const SparseSeg* __restrict__ segs,
                                                                          int nsegs, float divisor, unsigned* barrier, int* status) {
  // the table travels to shared memory in one go: walked in global memory it costs the zero fill one
  // dependent round trip per segment
  __shared__ SparseSeg seg[SC_MAX_SEGMENTS];
  for (int s = threadIdx.x; s < nsegs; s += SC_THREADS) seg[s] = segs[s];
  __syncthreads();
  const long long tid = (long long)blockIdx.x * SC_THREADS + threadIdx.x;
  const long long stride = (long long)gridDim.x * SC_THREADS;
  for (int s = 0; s < nsegs; ++s) {
    float* out = seg[s].out;
    const long long n = seg[s].numel;
    const long long n4 = ((uintptr_t)out & 15u) == 0 ? n >> 2 : 0;
    for (long long i = tid; i < n4; i += stride) reinterpret_cast<float4*>(out)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (long long i = n4 * 4 + tid; i < n; i += stride) out[i] = 0.f;
  }
  // value * (1 / W) rounded, then added: what torch's division by a scalar followed by index_add_
  // computes on the GPU (no fused multiply-add), so the result matches that sequence bit for bit
  const float inv = 1.0f / divisor;
  unsigned target = 0;
  for (int w = 0; w < workers; ++w) {
    if (!sc_grid_barrier(barrier, target)) {
      if (threadIdx.x == 0) atomicExch(status, 1);
      return;
    }
    const float* val = values + (long long)w * per_worker;
    const int* pos = positions + (long long)w * per_worker;
    for (long long j = tid; j < per_worker; j += stride) {
      int lo = 0, hi = nsegs - 1;   // first segment whose end is above j
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (seg[mid].end > j) hi = mid; else lo = mid + 1;
      }
      const long long p = pos[j];
      if (p >= 0 && p < seg[lo].numel) seg[lo].out[p] = __fadd_rn(seg[lo].out[p], __fmul_rn(val[j], inv));
    }
  }
}

}  // namespace

PSGD_API int psgd_sparse_combine_max_segments() { return SC_MAX_SEGMENTS; }

// values / positions: [workers][per_worker] as gathered; segs: device array of `nsegs` SparseSeg
// (segment s covers pairs [segs[s-1].end, segs[s].end) of every worker's list; positions are local
// to the segment's output); barrier: one zeroed unsigned per launch; status: set to 1 if the grid
// barrier gave up. Writes out_s = sum over workers (in rank order) of the scattered value / divisor.
PSGD_API int psgd_sparse_combine_launch(const float* values, const int* positions, int workers, long long per_worker,
                                        const void* segs, int nsegs, float divisor, unsigned* barrier, int* status,
                                        cudaStream_t stream) {
  if (nsegs <= 0 || workers <= 0) return 0;
  if (nsegs > SC_MAX_SEGMENTS) {
    psgd_set_error("psgd_sparse_combine_launch: %d segments exceed the maximum %d", nsegs, SC_MAX_SEGMENTS);
    return -1;
  }
  static int blocks_cached = 0;
  if (!blocks_cached) {
    int dev = 0, sms = 0, per_sm = 0;
    PSGD_CUDA_OK(cudaGetDevice(&dev));
    PSGD_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    PSGD_CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, psgd_sparse_combine_kernel, SC_THREADS, 0));
    blocks_cached = sms * (per_sm > 4 ? 4 : (per_sm < 1 ? 1 : per_sm));
  }
  PSGD_CUDA_OK(cudaMemsetAsync(barrier, 0, sizeof(unsigned), stream));
  const SparseSeg* segs_t = (const SparseSeg*)segs;
  void* params[] = {(void*)&values, (void*)&positions, (void*)&workers, (void*)&per_worker, (void*)&segs_t,
                    (void*)&nsegs, (void*)&divisor, (void*)&barrier, (void*)&status};
  PSGD_CUDA_OK(cudaLaunchCooperativeKernel((const void*)psgd_sparse_combine_kernel, dim3(blocks_cached), dim3(SC_THREADS), params, 0, stream));
  return 0;
}
