// The last product of a step and the decompression in one pass over the gradient.
//
// When the last half-iteration multiplies with the Q side (P = M Q_hat), a row of the residual needs
// nothing but the same row of P:
//     P[i]   = M[i] Q_hat - sum_h L_h[i] C_h                    (the product, csrc/lowrank_ffma.cu NN)
//     A[i]   = sum_h L_h[i] R_h^T + P[i] Q_hat^T                (the update)
//     M[i]  <- M[i] - A[i],   out[i] <- A[i]                    (csrc/finalize.cu)
// (powersgd/powersgd.py:185-230 in the reference). So a CTA that holds whole rows does both with one read of
// M: 12 bytes per element instead of 16. One worker only: with several, P is summed over the workers before
// the decompression.
//
// One persistent CTA of 512 threads per SM. It is divided into groups of 64 to 512 threads, wide enough for
// the matrix's columns: a thread owns up to C columns, and the values of all factors Q_hat and R_h in these
// columns stay in its registers (up to 64 of them: the register file holds 128 KiB of factors, which shared
// memory then need not) for as long as the matrix lasts. A group works on panels of 4 to 16 whole
// rows, which are contiguous in memory whatever the row pitch: one thread brings them in by bulk copies, a
// ring of three to six panels per group, so loads run ahead while a group multiplies, adds up its warps' sums
// and finishes its rows, and rows of 650 or 27 floats are loaded as fast as any. Other groups fill the SM
// while one waits. Multiplications are packed in pairs of columns (fma.rn.f32x2: two IEEE operations).
// Bound by HBM and by what four warps per scheduler find to do between two barriers: 4 x 4096^2 at rank 4 x 2 takes
// 151 us (805 MB, 5.3 TB/s) where the product (tensor cores) and the decompression took 60 + 146; the pass 421 -> 377.
// Above eight factor columns a thread owns four or two matrix columns only, and the sums over the lanes cost as much as
// the products (50257 x 1024 at rank 16 x 2: 75 + 186 -> 380 us); with the optimizer step, parameters and momentum would come
// through registers between the barriers (GPT-2 medium: 284 + 1315 -> 1661 us). Both stay with the launches apart.
#include "psgd_async.cuh"
#include "psgd_bounds.cuh"

constexpr int PN_THREADS = 512;
constexpr int PN_MIN_GROUP = 64;
constexpr int PN_MAX_GROUPS = PN_THREADS / PN_MIN_GROUP;
constexpr int PN_QUAD = 4;          // panels are whole quads of rows: 16 bytes times the columns, so every copy is aligned
constexpr int PN_MAX_STAGES = 6;
constexpr int PN_MAX_PREV = 3;      // earlier half-iterations of a step
constexpr int PN_MAX_COLUMNS = 8;   // template rank x half-iterations
constexpr int PN_ROW_VALUES = 128;  // most rows x factor columns of a panel
constexpr int PN_RINGS = 200 * 1024;          // of shared memory for the rings of all groups, at least
constexpr int PN_SMEM = 227 * 1024 - 512;     // dynamic; the rest is static

struct PanelArgs {
  const PsgdMat* mats;
  const PsgdTile* tiles;    // segments: rows [row0, row0 + rows) of a matrix, `split` rows per panel
  const int* starts;        // CTA b has the segments starts[b] .. starts[b + 1]
  const float* in;          // Q_hat
  float* out;               // fresh P, and
  float* out2;              // a second copy (the warm-start buffer) or null
  const float* lprev[PN_MAX_PREV];   // earlier factor pairs and cross products
  const float* rprev[PN_MAX_PREV];
  const float* cmat[PN_MAX_PREV];
  int* status;
};

// Columns of a thread: what 64 registers of factor values allow (a few less where a second bound,
// the panels in shared memory, is reached first).
__host__ __device__ constexpr int pn_cols(int kt) { return kt <= 4 ? 12 : 8; }
__host__ __device__ constexpr int pn_even(int k) { return (k + 1) / 2 * 2; }
// Threads of a group for m columns: enough for the columns, and few enough groups for three quads of rows each.
__host__ __device__ inline int pn_group(int m, int cols) {
  int g = PN_MIN_GROUP;
  while (g < PN_THREADS && (g * cols < m || 3 * PN_QUAD * m * 4 * (PN_THREADS / g) > PN_RINGS)) g *= 2;
  return g;
}
// Shared memory in front of the rings, in bytes: barriers; 16 bytes of zeros; row values [group][3][rows][KE] of two equal
// floats; the warps' sums [2][warp][rows][RT]; cross products. For panels of `rows` rows of `groups` groups.
__host__ __device__ constexpr int pn_zero_off() { return PN_MAX_GROUPS * PN_MAX_STAGES * 8; }
__host__ __device__ constexpr int pn_rows_off() { return pn_zero_off() + 16; }
__host__ __device__ constexpr int pn_part_off(int kt, int rows, int groups) { return pn_rows_off() + groups * 3 * rows * pn_even(kt) * 8; }
__host__ __device__ constexpr int pn_cmat_off(int kt, int rt, int rows, int groups) { return pn_part_off(kt, rows, groups) + 2 * (PN_THREADS / 32) * rows * rt * 4; }
__host__ __device__ constexpr int pn_ring_off(int kt, int rt, int rows, int groups) {
  return (pn_cmat_off(kt, rt, rows, groups) + (kt - rt) * rt * 4 + 127) / 128 * 128;
}
// Bytes of one group's ring.
__host__ __device__ constexpr int pn_ring_bytes(int kt, int rt, int rows, int groups) {
  return (PN_SMEM - pn_ring_off(kt, rt, rows, groups)) / groups / 128 * 128;
}

typedef unsigned long long pair2;   // two floats, the first in the low half
__device__ __forceinline__ pair2 pn_pack(float x, float y) {
  pair2 p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(x), "f"(y));
  return p;
}
__device__ __forceinline__ void pn_unpack(pair2 p, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(p)); }
__device__ __forceinline__ pair2 pn_fma(pair2 a, pair2 b, pair2 c) {
  pair2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ pair2 pn_mul(pair2 a, pair2 b) {
  pair2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Sums of N values over the 32 lanes: value i ends up (complete) in the lanes whose top log2(N) bits spell i.
// Every exchange halves what a lane still carries. A lane holds its values in an order of its own (value
// j ^ pn_order(lane) at place j): an upper lane of the first SWAPPED exchanges then has what it keeps where the
// lower one has it, and nothing needs to be selected.
template <int N, int SWAPPED>
__device__ __forceinline__ int pn_order(int lane) {
  int order = 0;
#pragma unroll
  for (int s = 0; s < SWAPPED; ++s)
    if (lane & (16 >> s)) order |= N >> (s + 1);
  return order;
}
template <int N, int SWAPPED>
__device__ __forceinline__ float pn_warp_sums(float (&v)[N], int lane) {
  int off = 16, step = 0;
#pragma unroll
  for (int n = N; n > 1; n >>= 1, off >>= 1, ++step) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      if (i < n / 2) {
        const bool swap = step >= SWAPPED && upper;
        const float keep = swap ? v[i + n / 2] : v[i], send = swap ? v[i] : v[i + n / 2];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
      }
    }
  }
  float s = v[0];
#pragma unroll
  for (; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  return s;
}

// Barrier of a group; true when every thread's `ok` is.
__device__ __forceinline__ bool pn_barrier_and(int id, int threads, bool ok) {
  uint32_t all;
  __syncwarp();   // it counts whole warps: their lanes have to arrive together
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %3, 0;\n\t"
      "bar.red.and.pred p, %1, %2, q;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(all)
      : "r"(id), "r"(threads), "r"((uint32_t)ok)
      : "memory");
  return all != 0;
}
template <int VEC>
__device__ __forceinline__ void pn_load(const float* p, float* v) {
  if (VEC == 4) { const float4 q = *reinterpret_cast<const float4*>(p); v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w; }
  else if (VEC == 2) { const float2 q = *reinterpret_cast<const float2*>(p); v[0] = q.x; v[1] = q.y; }
  else v[0] = *p;
}
template <int VEC>
__device__ __forceinline__ void pn_store(float* p, const float* v) {
  if (VEC == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else if (VEC == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  else *p = v[0];
}

struct PanelSegment {   // in shared memory: registers are for factors
  PsgdMat mat;
  PsgdTile tile;
  uint32_t phases[PN_MAX_GROUPS];   // bit s: the parity that the barrier of place s of a group's ring is in
  int abort;
};

// One segment of a CTA. `first`: the launch's first segment of this CTA, whose panels are asked for before the
// wait for the launch that makes Q_hat. Returns when this group has no panel left or a wait ran out.
//
// Turn i of a group: product of panel i; barrier; P of panel i (sums over the warps), and update and stores of
// panel i - 1, whose P everybody can see since that barrier. So a panel stays in the ring for two turns, and
// the place of panel i - 2 is free after the barrier of turn i. FULL: the matrix has as many columns as the group.
template <int RT, int NH, int VEC, bool FULL>
__device__ __forceinline__ void panel_segment(const PanelArgs& a, PanelSegment& sg, uint8_t* smem, bool first) {
  constexpr int KT = RT * (1 + NH), KE = pn_even(KT), HT = RT * NH, HD = HT > 0 ? HT : 1;
  constexpr int C = pn_cols(KT), NC = C / VEC, NP = C / 2;
  constexpr int BR = RT == 8 ? 2 : 4;                         // rows whose sums are reduced together
  constexpr int LB = BR == 4 ? 2 : 1;                         // log2 of it
  constexpr int SW = LB + (RT == 8 ? 2 : RT == 4 ? 1 : 0);    // exchanges by order: rows, then all but the last bit of the factor column
  int r = sg.mat.r, m = sg.mat.m, tid = threadIdx.x;
  asm volatile("" : "+r"(r), "+r"(m), "+r"(tid));   // the access widths in one kernel share nothing ahead of their branch:
                                                    // what they would keep in registers across it, factors need
  const int lane = tid & 31;
  const int TG = pn_group(m, C), lt = 31 - __clz(TG), G = PN_THREADS >> lt;   // powers of two
  const int g = tid >> lt, tg = tid & (TG - 1), wg = tg >> 5, W = TG >> 5, lw = lt - 5;
  const int PR = sg.tile.split;
  const int panels = (sg.tile.rows + PR - 1) / PR;
  const int count = g < panels ? (panels - g + G - 1) >> (9 - lt) : 0;   // of this group: panels g, g + G, ...
  const int stage_floats = PR * m;
  const int ring = pn_ring_bytes(KT, RT, PR, G) / 4;
  const int S = min(PN_MAX_STAGES, ring / stage_floats);
  const float* zeros = reinterpret_cast<const float*>(smem + pn_zero_off());   // what a column beyond the matrix reads
  uint64_t* full = reinterpret_cast<uint64_t*>(smem) + g * PN_MAX_STAGES;
  pair2* rowv = reinterpret_cast<pair2*>(smem + pn_rows_off()) + g * 3 * PR * KE;
  float* part = reinterpret_cast<float*>(smem + pn_part_off(KT, PR, G)) + g * W * 2 * PR * RT;
  float* cm = reinterpret_cast<float*>(smem + pn_cmat_off(KT, RT, PR, G));
  float* stages = reinterpret_cast<float*>(smem + pn_ring_off(KT, RT, PR, G)) + (size_t)g * ring;

  auto panel_row = [&](int i) { return sg.tile.row0 + (g + i * G) * PR; };
  auto panel_rows = [&](int i) { return min(PR, sg.tile.row0 + sg.tile.rows - panel_row(i)); };
  auto issue = [&](int i, int place) {   // one thread
    const int floats = panel_rows(i) * m, whole = floats & ~3;
    const float* src = sg.mat.grad + (long long)panel_row(i) * m;
    float* dst = stages + place * stage_floats;
    for (int e = whole; e < floats; ++e) dst[e] = src[e];
    psgd_mbar_expect_tx(full + place, (uint32_t)whole * 4u);
    if (whole) psgd_bulk_load(dst, src, (uint32_t)whole * 4u, full + place);
  };
  if (tg == 0)
    for (int i = 0; i < min(S, count); ++i) issue(i, i);
  uint32_t phases = sg.phases[g];
  if (first) psgd_wait_for_predecessor();

  // cross products of the matrix, for all groups
  if (NH > 0) {
    for (int e = tid; e < HT * RT; e += PN_THREADS) {
      const int h = e / (RT * RT), l = e / RT % RT, k = e % RT;
      cm[e] = (l < r && k < r) ? a.cmat[h][(long long)sg.mat.index * PSGD_CMAT_STRIDE + l * r + k] : 0.f;
    }
  }
  // factor values of this thread's columns; zero beyond the matrix and beyond its rank
  pair2 f[NP][KT];
  const int order = pn_order<BR * RT, SW>(lane), order_row = order / RT, order_k = order % RT;
  auto column = [&](int e) { return VEC * (tg + TG * (e / VEC)) + e % VEC; };
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    const int c0 = column(2 * p), c1 = column(2 * p + 1);
#pragma unroll
    for (int k = 0; k < KT; ++k) {
      const int l = k < HT ? k % RT : (k - HT) ^ order_k;
      const float* src = (k < HT ? a.rprev[k / RT < PN_MAX_PREV ? k / RT : 0] : a.in) + sg.mat.q_off + l;
      const bool in = l < r;
      f[p][k] = pn_pack(in && c0 < m ? src[(long long)c0 * r] : 0.f, in && c1 < m ? src[(long long)c1 * r] : 0.f);
    }
  }
  // values of the earlier left factors for this group's next panel, fetched one panel ahead
  constexpr int HV = NH > 0 ? (PN_ROW_VALUES + PN_MIN_GROUP - 1) / PN_MIN_GROUP : 1;
  float ahead[HV];
  auto fetch = [&](int i) {
#pragma unroll
    for (int x = 0; x < HV; ++x) {
      const int e = tg + (x << lt), row = e / HD, k = e % HD;
      ahead[x] = 0.f;
      if (i < count && row < panel_rows(i) && k % RT < r)
        ahead[x] = a.lprev[k / RT < PN_MAX_PREV ? k / RT : 0][sg.mat.p_off + (panel_row(i) + row) * r + k % RT];
    }
  };
  if (NH > 0) fetch(0);
  __syncwarp();
  __syncthreads();   // the cross products are there, and every thread has its group's phases

  int st = 0, before = S - 1, free_place = S - 2;      // ring places of panels i, i - 1 and i - 2
  pair2 *rv = rowv, *rv_before = rowv + 2 * PR * KE;   // row values of panels i and i - 1
  for (int i = 0; i <= count && count > 0; ++i) {
    bool landed = true;
    if (i < count) {
      if (NH > 0) {
#pragma unroll
        for (int x = 0; x < HV; ++x) {
          const int e = tg + (x << lt), row = e / HD, k = e % HD;
          if (row < PR) rv[row * KE + k] = pn_pack(ahead[x], ahead[x]);
        }
      }
      landed = psgd_mbar_wait(full + st, phases >> st & 1, &sg.abort, a.status);
      phases ^= 1u << st;

      // ---- product: this thread's columns, then the lanes of the warp ----
      const float* rowp = stages + st * stage_floats + order_row * m;
      const int step1 = order_row & 1 ? -m : m, step2 = order_row & 2 ? -2 * m : 2 * m;
      float* mine = part + ((i & 1) * W + wg) * PR * RT;
#pragma unroll 1
      for (int b = 0; b < PR; b += BR) {   // (rows that a last panel lacks: whatever lies there, never used)
        float v[BR * RT];
#pragma unroll
        for (int u = 0; u < BR; ++u) {
          const float* here = rowp + (u & 1 ? step1 : 0) + (u & 2 ? step2 : 0);
          pair2 acc[RT];
#pragma unroll
          for (int p0 = 0; p0 < NP; p0 += (VEC == 4 ? 2 : 1)) {
            float x[4];
            if (VEC == 1) {
              x[0] = *(FULL || column(2 * p0) < m ? here + column(2 * p0) : zeros);
              x[1] = *(FULL || column(2 * p0 + 1) < m ? here + column(2 * p0 + 1) : zeros);
            } else {
              pn_load<VEC>(FULL || column(2 * p0) < m ? here + column(2 * p0) : zeros, x);
            }
#pragma unroll
            for (int q = 0; q < (VEC == 4 ? 2 : 1); ++q) {
              const pair2 xx = pn_pack(x[2 * q], x[2 * q + 1]);
#pragma unroll
              for (int k = 0; k < RT; ++k) acc[k] = p0 + q == 0 ? pn_mul(xx, f[0][HT + k]) : pn_fma(xx, f[p0 + q][HT + k], acc[k]);
            }
          }
#pragma unroll
          for (int k = 0; k < RT; ++k) {
            float lo, hi;
            pn_unpack(acc[k], lo, hi);
            v[u * RT + k] = lo + hi;
          }
        }
        rowp += BR * m;
        const float s = pn_warp_sums<BR * RT, SW>(v, lane);
        constexpr int SPAN = 32 / (BR * RT);   // lanes that hold the same sum
        if (lane % SPAN == 0) mine[b * RT + lane / SPAN] = s;
      }
    }
    if (!pn_barrier_and(1 + g, TG, landed)) return;
    if (tg == 0 && i >= 2 && i - 2 + S < count) issue(i - 2 + S, free_place);

    if (i < count) {
      if (NH > 0) fetch(i + 1);
      // ---- P: the warps' sums, W lanes for each, corrected for what earlier half-iterations took out ----
      const int row0 = panel_row(i), values = panel_rows(i) * RT;
      const float* sums = part + (((i & 1) << lw) + (lane & (W - 1))) * PR * RT;
      for (int e0 = wg << (5 - lw); e0 < values; e0 += 32) {
        const int e = e0 + (lane >> lw);
        float s = 0.f;
        if (e < values) {
          const float* lefts = reinterpret_cast<const float*>(rv + e / RT * KE);
          s = sums[e];
          if (NH > 0)
            for (int l = lane & (W - 1); l < HT; l += W) s = fmaf(-lefts[2 * l], cm[l * RT + e % RT], s);
        }
        for (int off = W >> 1; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if ((lane & (W - 1)) == 0 && e < values) {
          const int row = e / RT, k = e % RT;
          if (k >= r) s = 0.f;
          rv[row * KE + HT + k] = pn_pack(s, s);
          if (KE > KT && k == 0) rv[row * KE + KT] = 0ull;
          if (k < r) {
            const int at = sg.mat.p_off + (row0 + row) * r + k;
            a.out[at] = s;
            if (a.out2) a.out2[at] = s;
          }
        }
      }
    }

    // ---- update and residual of the panel before ----
    const int rows = i > 0 ? panel_rows(i - 1) : 0;
    const float* rowp = stages + before * stage_floats;
    const ulonglong2* lv = reinterpret_cast<const ulonglong2*>(rv_before);
    long long off = (long long)panel_row(i - 1) * m;
#pragma unroll 1
    for (int row = 0; row < rows; ++row, off += m, rowp += m, lv += KE / 2) {
      pair2 acc[NP];
#pragma unroll
      for (int k = 0; k < KT; k += 2) {
        const ulonglong2 l = lv[RT >= 4 && k >= HT ? HT / 2 + (((k - HT) ^ order_k) >> 1) : k / 2];
#pragma unroll
        for (int p = 0; p < NP; ++p) acc[p] = k == 0 ? pn_mul(l.x, f[p][0]) : pn_fma(l.x, f[p][k], acc[p]);
        if (k + 1 < KT) {
#pragma unroll
          for (int p = 0; p < NP; ++p) acc[p] = pn_fma(l.y, f[p][k + 1 < KT ? k + 1 : k], acc[p]);
        }
      }
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const int c = VEC * (tg + TG * j);
        if (FULL || c < m) {
          float gv[VEC], av[VEC];
          pn_load<VEC>(rowp + c, gv);
#pragma unroll
          for (int x = 0; x < VEC; ++x) {
            const int e = j * VEC + x;
            float lo, hi;
            pn_unpack(acc[e / 2], lo, hi);
            av[x] = e % 2 ? hi : lo;
            gv[x] -= av[x];
          }
          pn_store<VEC>(sg.mat.grad + off + c, gv);
          pn_store<VEC>(sg.mat.out + off + c, av);
        }
      }
    }
    free_place = before;
    before = st;
    if (++st == S) st = 0;
    rv_before = rv;
    rv = rv == rowv + 2 * PR * KE ? rowv : rv + PR * KE;
  }
  if (tg == 0) sg.phases[g] = phases;
}

template <int RT, int NH>
__global__ void __launch_bounds__(PN_THREADS, 1) psgd_panel_kernel(const __grid_constant__ PanelArgs a) {
  constexpr int C = pn_cols(RT * (1 + NH));
  extern __shared__ __align__(128) uint8_t pn_smem[];
  __shared__ PanelSegment sg;
  const int first = a.starts[blockIdx.x], end = a.starts[blockIdx.x + 1];
  psgd_launch_dependents();
  if (threadIdx.x == 0) {
    sg.abort = 0;
    for (int b = 0; b < PN_MAX_GROUPS * PN_MAX_STAGES; ++b) psgd_mbar_init(reinterpret_cast<uint64_t*>(pn_smem) + b, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < PN_MAX_GROUPS) sg.phases[threadIdx.x] = 0;
  if (threadIdx.x < 4) reinterpret_cast<float*>(pn_smem + pn_zero_off())[threadIdx.x] = 0.f;
  for (int s = first; s < end; ++s) {
    // panels of another height or groups of another width move the rings onto bytes that the segment before wrote
    // by ordinary stores: row values, sums, cross products
    psgd_fence_async_shared();
    __syncwarp();
    __syncthreads();   // every group has left the segment before
    if (*(volatile int*)&sg.abort) break;
    if (threadIdx.x == 0) {
      sg.tile = a.tiles[s];
      sg.mat = a.mats[sg.tile.mat];
    }
    __syncwarp();
    __syncthreads();
#ifdef PSGD_BOUNDS_CHECK
    {
      const PsgdMat& mt = sg.mat;
      const PsgdTile& t = sg.tile;
      constexpr int KT = RT * (1 + NH);
      bool ok = true;
      const unsigned long long addr = (unsigned long long)mt.grad | (unsigned long long)mt.out;
      ok &= PSGD_BC(mt.r >= 1 && mt.r <= RT, 6, PSGD_BC_RANK, mt.r, RT);
      ok &= PSGD_BC(t.row0 >= 0 && t.rows > 0 && t.row0 + t.rows <= mt.n && t.row0 % PN_QUAD == 0, 6, PSGD_BC_TILE_ROWS, t.row0 + t.rows, mt.n);
      ok &= PSGD_BC(mt.m >= 1 && mt.m <= PN_THREADS * C, 6, PSGD_BC_TILE_COLS, mt.m, PN_THREADS * C);
      ok &= PSGD_BC(t.split > 0 && t.split % PN_QUAD == 0 && t.split * KT <= PN_ROW_VALUES, 6, PSGD_BC_SMEM, t.split, PN_ROW_VALUES);
      const long long need = 3ll * t.split * mt.m * 4;
      const int have = pn_ring_bytes(KT, RT, t.split, PN_THREADS / pn_group(mt.m, C));
      ok &= PSGD_BC(need <= have, 6, PSGD_BC_SMEM, need, have);
      ok &= PSGD_BC((unsigned long long)mt.grad % 16 == 0, 6, PSGD_BC_ALIGNMENT, (unsigned long long)mt.grad % 16, 16);
      ok &= PSGD_BC(t.vec == 1 || (t.vec == 2 && addr % 8 == 0 && mt.m % 2 == 0) || (t.vec == 4 && addr % 16 == 0 && mt.m % 4 == 0),
                    6, PSGD_BC_ALIGNMENT, addr % 16, t.vec);
      ok &= PSGD_BC(mt.out != nullptr, 6, PSGD_BC_ELEMENT, 0, 0);
      if (!ok) break;
    }
#endif
    const int vec = sg.tile.vec;
    if (vec == 4 && pn_group(sg.mat.m, C) * C == sg.mat.m) panel_segment<RT, NH, 4, true>(a, sg, pn_smem, s == first);
    else if (vec == 4) panel_segment<RT, NH, 4, false>(a, sg, pn_smem, s == first);
    else if (vec == 2) panel_segment<RT, NH, 2, false>(a, sg, pn_smem, s == first);
    else panel_segment<RT, NH, 1, false>(a, sg, pn_smem, s == first);
  }
  __syncwarp();
  __syncthreads();
  if (*(volatile int*)&sg.abort) psgd_let_copies_land();
}

template <int RT, int NH>
static int panel_launch(const PanelArgs& a, int ctas, int early, cudaStream_t stream) {
  static unsigned long long devices = 0;   // per instantiation
  if (const int code = psgd_allow_shared((const void*)psgd_panel_kernel<RT, NH>, PN_SMEM, devices)) return code;
  return psgd_launch(psgd_panel_kernel<RT, NH>, ctas, PN_THREADS, PN_SMEM, stream, early, a);
}

static int pn_template_rank(int max_r) { return max_r <= 1 ? 1 : max_r <= 2 ? 2 : max_r <= 4 ? 4 : 8; }
static bool pn_takes(int max_r, int nhist) {
  return max_r >= 1 && max_r <= 8 && nhist >= 1 && nhist <= 1 + PN_MAX_PREV && pn_template_rank(max_r) * nhist <= PN_MAX_COLUMNS;
}
// Rows per panel (a multiple of four) for a segment of `rows` rows of a matrix of m columns; 0: the kernel does not take such
// a matrix. A panel of more rows spreads its barrier and its sums over more of them, as long as four panels of
// every group fit the ring (three where four rows are all that fits) and every group has two.
PSGD_API int psgd_panel_rows(int max_r, int nhist, int m, int rows) {
  if (!pn_takes(max_r, nhist) || m < 1) return 0;
  const int rt = pn_template_rank(max_r), kt = rt * nhist, cols = pn_cols(kt);
  if (m > PN_THREADS * cols) return 0;
  const int groups = PN_THREADS / pn_group(m, cols);
  const auto fits = [&](int n, int panels) { return (long long)panels * n * m * 4 <= pn_ring_bytes(kt, rt, n, groups); };
  if (!fits(PN_QUAD, 3)) return 0;
  int n = PN_QUAD;
  while (4 * n * groups <= rows && 2 * n * kt <= PN_ROW_VALUES && fits(2 * n, 4)) n *= 2;
  return n;
}

// Shares of the CTAs, in quads of rows and in the order of the matrices: matrix i has quads[i] of them, each of
// which costs quad_cost[i], and a CTA that goes on to another matrix pays `start`. bounds[c] .. bounds[c + 1] (counted
// over all matrices) is what CTA c gets. The dearest CTA is as cheap as it can be, up to a quad: shares are found in
// fractions and rounded, so that neighbours differ by a quad here and there. Whole quads to the same limit are some per cent
// slower from HBM (4 x 4096^2 377 -> 384 us, 4 x 2048^2 at rank 4 x 2 116 -> 124): all CTAs then read at one stride. Host code.
PSGD_API void psgd_panel_shares(const long long* quads, const long long* quad_cost, int nmats, long long start, int ctas, long long* bounds) {
  const auto fill = [&](double limit) {   // does it all fit when no CTA costs more?
    int mat = 0;
    double taken = 0;      // of this matrix
    long long before = 0;  // quads of the matrices before
    for (int c = 0; c < ctas; ++c) {
      bounds[c] = before + (long long)(taken + 0.5);
      double left = limit;
      for (bool first = true; mat < nmats; first = false) {
        if (!first) left -= (double)start;
        const double fits = left / (double)quad_cost[mat], rest = (double)quads[mat] - taken;
        if (fits < rest) {
          if (first || fits >= 1) taken += fits;   // less of another matrix is not worth its start
          break;
        }
        left -= rest * (double)quad_cost[mat];
        before += quads[mat++];
        taken = 0;
      }
    }
    bounds[ctas] = before;
    return mat == nmats;
  };
  double low = 0, high = 1;   // too little, enough
  for (int i = 0; i < nmats; ++i) high += (double)start + (double)quads[i] * (double)quad_cost[i];
  for (int step = 0; step < 60 && high - low > 1; ++step) {
    const double limit = 0.5 * (low + high);
    (fill(limit) ? high : low) = limit;
  }
  fill(high);
}

// The last half-iteration of a step (basis `in` on the Q side) with the decompression; one worker, no optimizer step. nhist:
// half-iterations of the step; lprev / rprev / cmat: the nhist - 1 earlier factor pairs and their cross products with `in`. tiles:
// segments with `split` = psgd_panel_rows(...) rows per panel, row0 a multiple of four, matrices on a 16-byte
// boundary; starts: ctas + 1 entries. early: see psgd_launch.
PSGD_API int psgd_panel_launch(const void* mats, const void* tiles, const int* starts, int ctas, int max_r, int nhist, const float* in,
                               float* out, float* out2, const float* const* lprev, const float* const* rprev,
                               const float* const* cmat, int* status, int early, cudaStream_t stream) {
  if (ctas <= 0) return 0;
  if (!pn_takes(max_r, nhist)) {
    psgd_set_error("psgd_panel_launch: rank %d with %d half-iterations is not compiled", max_r, nhist);
    return -1;
  }
  PanelArgs a;
  a.mats = (const PsgdMat*)mats;
  a.tiles = (const PsgdTile*)tiles;
  a.starts = starts;
  a.in = in;
  a.out = out;
  a.out2 = out2;
  for (int i = 0; i < PN_MAX_PREV; ++i) {
    a.lprev[i] = i < nhist - 1 ? lprev[i] : nullptr;
    a.rprev[i] = i < nhist - 1 ? rprev[i] : nullptr;
    a.cmat[i] = i < nhist - 1 ? cmat[i] : nullptr;
  }
  a.status = status;
#define PN_CASE(RT, N) \
  if (pn_template_rank(max_r) == RT && nhist == N) return panel_launch<RT, N - 1>(a, ctas, early, stream);
  PN_CASE(1, 1) PN_CASE(1, 2) PN_CASE(1, 3) PN_CASE(1, 4)
  PN_CASE(2, 1) PN_CASE(2, 2) PN_CASE(2, 3) PN_CASE(2, 4)
  PN_CASE(4, 1) PN_CASE(4, 2) PN_CASE(8, 1)
#undef PN_CASE
  return -1;
}

#ifdef PSGD_BOUNDS_CHECK
PSGD_BOUNDS_EXPORT(psgd_bounds_read_panel)
#endif
