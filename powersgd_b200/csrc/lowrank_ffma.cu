// Grouped tall-skinny products on the CUDA cores (exact float32 FMA path).
//
//   NT:  Q[m, r] = M^T[m, n] * Phat[n, r]  -  sum_i R_i[m, r] * C_i[r, r]
//   NN:  P[n, r] = M  [n, m] * Qhat[m, r]  -  sum_i L_i[n, r] * C_i[r, r]
//
// One launch covers EVERY compressed matrix of EVERY shape group: the grid walks a tile list
// built once by the host planner. This replaces the reference's per-group `torch.bmm` and the
// first `baddbmm_` (powersgd/powersgd.py:185-202): the deflation M <- M - P Q^T is never
// materialised between half-iterations; the small terms C_i (from the orthonormalisation
// launch) correct the product instead.
//
// At rank r the product does 2r flops per 4 bytes of M, so for r <= 8 float32 FMAs keep up
// with HBM and this path is bandwidth-bound; it is also the path for matrices whose row
// pitch is not a multiple of 16 bytes (27, 650 floats), which TMA cannot address. Every tile
// names the widest global access its matrix allows (16, 8 or 4 bytes: `PsgdTile::vec`), so one
// launch serves all of them.
//
// Tiles that cover the same output rows (NT: row blocks of one column block; NN: column
// blocks of one row block) write partial sums to a scratch arena; the tile that arrives last
// (arrival counter) adds them in a fixed order, so the result does not depend on scheduling.
#include "psgd_async.cuh"
#include "psgd_bounds.cuh"
#include "psgd_comm.cuh"

constexpr int GEMM_THREADS = 256;
constexpr int GEMM_WARPS = GEMM_THREADS / 32;
constexpr int NT_TILE_COLS = 128;   // columns of M per NT tile
constexpr int NT_MAX_ROWS = 256;    // rows of P-hat staged in smem at a time (128 at RT = 32); a tile may span several such chunks
constexpr int NN_CHUNK_COLS = 128;  // columns consumed per inner iteration of an NN tile
// Most columns of an NN tile: as many rows of Q-hat as fit 32 KiB of shared memory.
template <int RT>
__host__ __device__ constexpr int nn_max_cols() { return RT <= 8 ? 1024 : 8192 / RT; }

struct GemmArgs {
  const PsgdMat* mats;
  const PsgdTile* tiles;
  const float* in;    // orthonormal factor: P-shaped for NT, Q-shaped for NN
  float* out;         // fresh local factor: Q-shaped for NT, P-shaped for NN
  float* out2;        // optional second copy of it (single worker: the warm-start buffer) or null
  int ncorr;
  const float* corr_fac[PSGD_MAX_HIST];  // earlier local factors on the OUTPUT side
  const float* corr_c[PSGD_MAX_HIST];    // [mat][r*r] cross products
  float* partial;     // scratch for split tiles
  int* tickets;       // arrival counters (all zero between launches)
  // Multi-GPU: the epilogue also pushes every finished factor element, tagged with the next
  // epoch, into slot[rank] of every peer's arena. Null for a single worker.
  const PsgdCommDev* comm;
};

#ifdef PSGD_BOUNDS_CHECK
// Capacities of the buffers behind the raw pointers (floats / counters), set by the host through
// psgd_debug_limits_products() before a checked run; 0 = unknown, not checked.
static __device__ long long g_lim_partial, g_lim_tickets, g_lim_p, g_lim_q;

// Validates one product tile against its matrix, the template rank, the access width it claims and
// the scratch capacities. All threads compute the same verdict; a CTA with a bad tile returns
// before it touches memory.
template <int RT>
__device__ __forceinline__ bool product_tile_ok(const PsgdTile& t, const PsgdMat& mt, int kernel_id, int max_rows,
                                                int max_cols, int tile_elems) {
  bool ok = true;
  ok &= PSGD_BC(t.row0 >= 0 && t.rows > 0 && t.row0 + t.rows <= mt.n && t.rows <= max_rows, kernel_id, PSGD_BC_TILE_ROWS, t.row0 + t.rows, mt.n);
  ok &= PSGD_BC(t.col0 >= 0 && t.cols > 0 && t.col0 + t.cols <= mt.m && t.cols <= max_cols, kernel_id, PSGD_BC_TILE_COLS, t.col0 + t.cols, mt.m);
  ok &= PSGD_BC(mt.r >= 1 && mt.r <= RT, kernel_id, PSGD_BC_RANK, mt.r, RT);
  const unsigned long long addr = (unsigned long long)mt.grad;
  ok &= PSGD_BC(t.vec == 1 || (t.vec == 2 && addr % 8 == 0 && mt.m % 2 == 0) || (t.vec == 4 && addr % 16 == 0 && mt.m % 4 == 0),
                kernel_id, PSGD_BC_ALIGNMENT, addr % 16, t.vec);
  ok &= PSGD_BC(t.nsplit >= 1 && t.split >= 0 && t.split < t.nsplit, kernel_id, PSGD_BC_SCRATCH_SLOT, t.split, t.nsplit);
  if (t.nsplit > 1 && g_lim_partial > 0)
    ok &= PSGD_BC((long long)(t.slot0 + t.nsplit) * tile_elems <= g_lim_partial, kernel_id, PSGD_BC_SCRATCH_SLOT,
                  (long long)(t.slot0 + t.nsplit) * tile_elems, g_lim_partial);
  if (t.nsplit > 1 && g_lim_tickets > 0) ok &= PSGD_BC(t.ticket >= 0 && t.ticket < g_lim_tickets, kernel_id, PSGD_BC_TICKET, t.ticket, g_lim_tickets);
  if (g_lim_p > 0) ok &= PSGD_BC((long long)mt.p_off + (long long)mt.n * mt.r <= g_lim_p, kernel_id, PSGD_BC_FACTOR_INDEX, (long long)mt.p_off + (long long)mt.n * mt.r, g_lim_p);
  if (g_lim_q > 0) ok &= PSGD_BC((long long)mt.q_off + (long long)mt.m * mt.r <= g_lim_q, kernel_id, PSGD_BC_FACTOR_INDEX, (long long)mt.q_off + (long long)mt.m * mt.r, g_lim_q);
  return ok;
}
#endif

template <int RT>
__host__ __device__ constexpr int nt_max_rows() { return RT <= 16 ? NT_MAX_ROWS : NT_MAX_ROWS / 2; }
// Staging buffer of an NT tile: rows of P-hat, later the sums of the warps, [warp][column of a lane x RT][32 lanes, padded], all eight
// warps' up to rank 8, four above.
template <int RT>
__host__ __device__ constexpr int nt_sum_warps() { return RT <= 8 ? GEMM_WARPS : GEMM_WARPS / 2; }
// Words from one value of the lanes to the next. 32 results in a row, [column][RT], belong to 32 / (VEC x RT) lanes, one behind the
// other, and to VEC x RT values of theirs: so far apart, they all lie in banks of their own.
template <int RT, int VEC>
__host__ __device__ constexpr int nt_sum_pitch() { return 32 + (VEC * RT >= 32 ? 1 : 32 / (VEC * RT) % 32); }
template <int RT>
__host__ __device__ constexpr int nt_stage_floats() {
  const int sums = nt_sum_warps<RT>() * 4 * RT * nt_sum_pitch<RT, RT == 1 ? 2 : 1>(), rows = nt_max_rows<RT>() * RT;
  return sums > rows ? sums : rows;
}

// A lane owns 4 of the 128 columns of a column block; which ones depends on the access width:
// 4 adjacent (one 16-byte load), 2 + 2 adjacent (two 8-byte loads, 64 columns apart) or 4
// columns 32 apart (scalar loads). Every variant keeps a warp's accesses contiguous.
template <int VEC>
__device__ __forceinline__ int lane_col(int lane, int c) {
  if (VEC == 4) return 4 * lane + c;
  if (VEC == 2) return (c < 2) ? 2 * lane + c : 64 + 2 * lane + (c - 2);
  return lane + 32 * c;
}

// The lane that owns column lc, and which of its columns that is.
template <int VEC>
__host__ __device__ constexpr int col_lane(int lc) { return VEC == 4 ? lc >> 2 : VEC == 2 ? (lc & 63) >> 1 : lc & 31; }
template <int VEC>
__host__ __device__ constexpr int col_of_lane(int lc) { return VEC == 4 ? lc & 3 : VEC == 2 ? (lc & 1) + 2 * (lc >> 6) : lc >> 5; }

// Where value k of column lc lies among a warp's sums.
template <int RT, int VEC>
__host__ __device__ constexpr int nt_sum_at(int lc, int k) { return (col_of_lane<VEC>(lc) * RT + k) * nt_sum_pitch<RT, VEC>() + col_lane<VEC>(lc); }
template <int RT, int VEC>
__host__ __device__ constexpr bool nt_sums_in_banks_of_their_own() {
  for (int first = 0; first < NT_TILE_COLS * RT; first += 32) {
    unsigned banks = 0;
    for (int e = first; e < first + 32; ++e) banks |= 1u << (nt_sum_at<RT, VEC>(e / RT, e % RT) & 31);
    if (banks != ~0u) return false;
  }
  return true;
}

// v[0..3] = the lane's four columns of the row at `rowp` (column block starting at c0, valid up
// to cend); zero where the row or the column does not exist.
template <int VEC>
__device__ __forceinline__ void load_lane_cols(const float* __restrict__ rowp, int c0, int cend, int lane, bool rok,
                                               float* v) {
  if (VEC == 4) {
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
    if (rok && c0 + 4 * lane < cend) q = __ldg(reinterpret_cast<const float4*>(rowp + c0 + 4 * lane));
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else if (VEC == 2) {
    float2 q0 = make_float2(0.f, 0.f), q1 = make_float2(0.f, 0.f);
    if (rok && c0 + 2 * lane < cend) q0 = __ldg(reinterpret_cast<const float2*>(rowp + c0 + 2 * lane));
    if (rok && c0 + 64 + 2 * lane < cend) q1 = __ldg(reinterpret_cast<const float2*>(rowp + c0 + 64 + 2 * lane));
    v[0] = q0.x; v[1] = q0.y; v[2] = q1.x; v[3] = q1.y;
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = (rok && c0 + lane + 32 * c < cend) ? __ldg(rowp + c0 + lane + 32 * c) : 0.f;
  }
}

// ------------------------------------------------------------------------------------------
// NT: each lane owns 4 columns, each warp strides over the tile's rows. Bound by the latency of a tile's
// chain (staging, loads, the sum over the warps, the hand-over) on small models, by how many loads are
// under way on larger ones: ResNet-18 at rank 2 (45 MB) 17.1 -> 12.2 us, the LSTM model at rank 4 (127 MB)
// 55.9 -> 47 us with what follows (loads ahead of the wait, two batches under way, longer tiles).
// ------------------------------------------------------------------------------------------
template <int RT, int VEC>
__device__ __forceinline__ void gemm_nt_tile(const GemmArgs& a, const PsgdTile& t, const PsgdMat& mt, float* smem) {
  const int r = mt.r, m = mt.m;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  float* sP = smem;                        // [rows][RT], then the warps' sums [GEMM_WARPS][128][RT] (RT <= 8)
  float* sSum = smem + nt_stage_floats<RT>();   // [128][RT]
  __shared__ int sLast;
#ifdef PSGD_BOUNDS_CHECK
  if (!product_tile_ok<RT>(t, mt, 1, 1 << 30, NT_TILE_COLS, NT_TILE_COLS * RT)) return;
#endif

  float acc[4][RT];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int k = 0; k < RT; ++k) acc[c][k] = 0.f;

  const float* __restrict__ M = mt.grad;
  const int cend = t.col0 + t.cols;
  constexpr int MAXR = nt_max_rows<RT>();
  constexpr int UR = 4;                       // rows of a warp in flight
  constexpr int STEP = GEMM_WARPS * UR;

  // The gradient does not depend on the launches before this one: the tile's first rows are loaded
  // and the rest is asked into L2 while the basis is still being orthonormalised.
  // Two batches of rows are under way at any time: one alone (16 KiB per CTA) leaves the memory system
  // idle for most of its latency.
  float v0[UR][4], v1[UR][4];
  auto load = [&](float (&v)[UR][4], int row0, int rows, int i0) {
#pragma unroll
    for (int u = 0; u < UR; ++u) {
      const int i = i0 + u * GEMM_WARPS;
      const bool rok = i < rows;
      load_lane_cols<VEC>(M + (long long)(row0 + (rok ? i : 0)) * m, t.col0, cend, lane, rok, v[u]);
    }
  };
  load(v0, t.row0, min(MAXR, t.rows), warp);
  load(v1, t.row0, min(MAXR, t.rows), warp + STEP);
  for (int e = tid + 8 * STEP; e < 4 * min(MAXR, t.rows); e += GEMM_THREADS)   // four lines of 128 bytes per row
    if ((e & 3) * 32 < t.cols) psgd_prefetch_l2(M + (long long)(t.row0 + (e >> 2)) * m + t.col0 + (e & 3) * 32);
  psgd_wait_for_predecessor();

  // a tall tile is walked in chunks of MAXR rows (what fits the staging buffer of P-hat); the
  // accumulators live across chunks, so a matrix with tens of thousands of rows needs tens of
  // partial tiles per column block, not hundreds
  for (int rb = 0; rb < t.rows; rb += MAXR) {
    const int rows = min(MAXR, t.rows - rb);
    if (rb) {
      load(v0, t.row0 + rb, rows, warp);
      load(v1, t.row0 + rb, rows, warp + STEP);
      __syncthreads();  // the previous chunk's rows of P-hat are no longer read
    }
    // stage the chunk's rows of P-hat (zero padded to RT columns)
    const float* pin = a.in + mt.p_off + (long long)(t.row0 + rb) * r;
    if (RT >= 4 && r == RT && ((uintptr_t)pin & 15u) == 0) {
      for (int e = 4 * tid; e < rows * RT; e += 4 * GEMM_THREADS) psgd_copy16(sP + e, pin + e);
    } else {
      for (int e = tid; e < rows * RT; e += GEMM_THREADS) {
        const int row = e / RT, k = e % RT;
        if (k < r) psgd_copy4(sP + e, pin + row * r + k);
        else sP[e] = 0.f;
      }
    }
    psgd_copies_wait();
    __syncthreads();

    auto use = [&](const float (&v)[UR][4], int i0) {
#pragma unroll
      for (int u = 0; u < UR; ++u) {
        const int i = i0 + u * GEMM_WARPS;
        if (i < rows) {
          const float* pr = sP + i * RT;
#pragma unroll
          for (int k = 0; k < RT; ++k) {
            const float pk = pr[k];
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[c][k] = fmaf(v[u][c], pk, acc[c][k]);
          }
        }
      }
    };
    for (int i0 = warp; i0 < rows; i0 += 2 * STEP) {
      use(v0, i0);
      if (i0 + 2 * STEP < rows) load(v0, t.row0 + rb, rows, i0 + 2 * STEP);
      use(v1, i0 + STEP);
      if (i0 + 3 * STEP < rows) load(v1, t.row0 + rb, rows, i0 + 3 * STEP);
    }
  }
  __syncthreads();

  // Sum over the warps, in a fixed order. A warp's values lie lane by lane, so that neither their stores nor the loads of a thread that
  // adds up one (column, k) meet in one bank: written in the order of the result, [column][k], 16 or 32 lanes did, and above rank 8, where
  // one warp after another added to it, the sum was three quarters of a tile: 39 500 of 52 000 cycles on 4 x 1024x1001 at rank 16, 75 000
  // of 134 000 on 3 x 9000x650 at rank 11, 4700 of 13 000 on 4 x 1001x1024 at rank 5; then 2900, 3000 and 1100.
  // The launches: 34.8 -> 12.6 us, 137 -> 60, 9.7 -> 7.7. With one pitch of 33 words for all, the loads still met, two to four to a bank
  // where VEC * RT < 32: launches alone, in the order of the result / 33 words / now, 4 x 1024x1001 at rank 8 9.8 / 10.4 / 9.6, 3 x 1001x777 +
  // 2 x 515x2049 at rank 8 12.3 / 12.4 / 11.9, rank 3 9.3 / 9.9 / 9.5, 4 x 1024x1002 at rank 5 10.0 / 9.2 / 9.0.
  constexpr int SUMS = nt_sum_warps<RT>(), PITCH = nt_sum_pitch<RT, VEC>(), PER_WARP = 4 * RT * PITCH;
  static_assert(SUMS * PER_WARP <= nt_stage_floats<RT>(), "the widest pitch has room");
  static_assert(nt_sums_in_banks_of_their_own<RT, VEC>(), "32 results in a row are added up by a warp");
  auto slot = [&](int w, int c, int k) { return sP + w * PER_WARP + (c * RT + k) * PITCH; };
  if (SUMS < GEMM_WARPS) {
    if (warp >= SUMS) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int k = 0; k < RT; ++k) slot(warp - SUMS, c, k)[lane] = acc[c][k];
    }
    __syncthreads();
    if (warp < SUMS) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int k = 0; k < RT; ++k) slot(warp, c, k)[lane] += acc[c][k];   // (its own places: nobody else reads them yet)
    }
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int k = 0; k < RT; ++k) slot(warp, c, k)[lane] = acc[c][k];
  }
  __syncthreads();
#pragma unroll 1
  for (int e = tid; e < NT_TILE_COLS * RT; e += GEMM_THREADS) {
    const float* of = sP + nt_sum_at<RT, VEC>(e / RT, e % RT);
    float s = of[0];
#pragma unroll
    for (int w = 1; w < SUMS; ++w) s += of[w * PER_WARP];
    sSum[e] = s;
  }
  __syncthreads();

  constexpr int tile_elems = NT_TILE_COLS * RT;
  bool owner = true;  // does this CTA write the output rows?
  if (t.nsplit > 1) {
    float* mine = a.partial + (long long)(t.slot0 + t.split) * tile_elems;
    for (int e = tid; e < tile_elems; e += GEMM_THREADS) __stcg(mine + e, sSum[e]);
    __threadfence();
    __syncthreads();
    if (tid == 0) sLast = (psgd_atom_add_acqrel_gpu(a.tickets + t.ticket, 1) == t.nsplit - 1);
    __syncthreads();
    owner = sLast != 0;
    if (owner) {
      __threadfence();
      psgd_sum_partials<tile_elems, GEMM_THREADS>(a.partial + (long long)t.slot0 * tile_elems, t.nsplit, sSum);
      if (tid == 0) a.tickets[t.ticket] = 0;  // ready for the next launch
      __syncthreads();
    }
  }

  // epilogue: subtract the deflation terms, store Q rows locally and push them to the peers
  float* __restrict__ qout = a.out + mt.q_off;
  uint2* push[PSGD_MAX_WORLD];
  int e1 = 0;
  int npush = 0;
  if (a.comm != nullptr && owner) {
    const PsgdCommDev c = *a.comm;
    e1 = *c.epoch + 1;
    npush = c.world;
    for (int p = 0; p < PSGD_MAX_WORLD; ++p) push[p] = p < c.world ? psgd_comm_slot(c, p, e1, c.rank) + mt.q_off : nullptr;
  }
  for (int e = tid; owner && e < t.cols * r; e += GEMM_THREADS) {
    const int lc = e / r, k = e % r;
    const int col = t.col0 + lc;
    float s = sSum[lc * RT + k];
    for (int i = 0; i < a.ncorr; ++i) {
      const float* f = a.corr_fac[i] + mt.q_off + (long long)col * r;
      const float* cm = a.corr_c[i] + (long long)mt.index * PSGD_CMAT_STRIDE;
      float d = 0.f;
      for (int l = 0; l < r; ++l) d = fmaf(f[l], cm[l * r + k], d);
      s -= d;
    }
    qout[(long long)col * r + k] = s;
    if (a.out2) a.out2[mt.q_off + (long long)col * r + k] = s;
    for (int p = 0; p < npush; ++p) psgd_comm_store(push[p] + (long long)col * r + k, s, e1);
  }
}

template <int RT>
__global__ void __launch_bounds__(GEMM_THREADS, RT <= 4 ? 3 : (RT <= 16 ? 2 : 1)) psgd_gemm_nt_kernel(GemmArgs a) {
  extern __shared__ __align__(16) float smem[];
  psgd_launch_dependents();
  const PsgdTile t = a.tiles[blockIdx.x];
  const PsgdMat mt = a.mats[t.mat];
  if (t.vec == 4) gemm_nt_tile<RT, 4>(a, t, mt, smem);
  else if (t.vec == 2) gemm_nt_tile<RT, 2>(a, t, mt, smem);
  else gemm_nt_tile<RT, 1>(a, t, mt, smem);
}

// ------------------------------------------------------------------------------------------
// NN: each warp owns RPW rows; lanes stride across the columns and reduce at the end.
// ------------------------------------------------------------------------------------------
// Sums of N values over the 32 lanes: value i ends up (complete) in the lanes whose top log2(N) bits
// spell i. Every step halves what a lane still carries, so N values cost N - 1 + 5 - log2(N) shuffles
// instead of 5 N; lanes are paired as in a butterfly (16, 8, 4, 2, 1), so the bits are the same.
template <int N>
__device__ __forceinline__ float warp_sums(float (&v)[N], int lane) {
  static_assert(N >= 1 && N <= 32 && (N & (N - 1)) == 0, "a power of two");
  int off = 16;
#pragma unroll
  for (int n = N; n > 1; n >>= 1, off >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      if (i < n / 2) {
        const float keep = upper ? v[i + n / 2] : v[i], send = upper ? v[i] : v[i + n / 2];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
      }
    }
  }
  float s = v[0];
  for (; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  return s;
}

// A tile is 8 * RPW rows by up to nn_max_cols columns. What bounds it: with few columns per tile the
// chain load - multiply - reduce - hand over; with many, the loads of the gradient. So the rows of
// Q-hat that the tile needs are staged in shared memory once, in the order the lanes read them (a lane
// reads its 4 columns x RT values as RT 16-byte words: read straight from global memory they cost more
// load instructions than the gradient itself), and the loop over 128-column chunks keeps two chunks
// of the gradient under way. ResNet-18 at rank 2 (45 MB) 18.8 -> 16.1 us, 3 x 1001x777 + 2 x 515x2049 at rank 3
// 15.2 -> 12.1 us; tiles of 512 / 256 columns instead: 19.1 / 21.3 us on ResNet-18. The staging itself, as a loop of loads and
// stores with a division for each value, took 2600 of a tile's some 10 000 cycles on ResNet-18, 4100 of 13 500 at rank 3 and, with
// five CTAs per SM at it, 8200 of 17 000 on the LSTM model; by asynchronous copies column by column 1550, 1700 and 4700.
// All CTAs of a column part copy the same rows of Q-hat at the same time. Up to rank 8 they do it by way of L1: launches alone, loads
// and stores / copies by L2 / by L1, 4 x 8192x512 at rank 4 11.7 / 16.3 / 11.3 us, 16000x1000 13.2 / 18.0 / 11.2, 4 x 1024^2 5.4 / 5.6 / 4.6; at rank 8
// 4 x 8192x512 20.1 / 23.4 / 21.3, 10000x1001 24.1 / 19.7 / 13.5, 64 x 512^2 20.4 / 20.3 / 20.7. At rank 16 and 32 by L2: 64 x 512^2
// 43.7 / 30.6 / 32.7 and 173 / 108 / 111, 4 x 8192x512 43.5 / 34.3 / 31.5 and 170 / 110 / 112.
template <int RT, int VEC, int RPW>
__device__ __forceinline__ void gemm_nn_tile(const GemmArgs& a, const PsgdTile& t, const PsgdMat& mt, float* sQ, float* sSum) {
  const int r = mt.r, m = mt.m;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int TILE_ROWS = GEMM_WARPS * RPW;
  __shared__ int sLast;
#ifdef PSGD_BOUNDS_CHECK
  if (!product_tile_ok<RT>(t, mt, 2, TILE_ROWS, nn_max_cols<RT>(), TILE_ROWS * RT)) return;
#endif

  const float* __restrict__ M = mt.grad;

  float acc[RPW * RT];
#pragma unroll
  for (int e = 0; e < RPW * RT; ++e) acc[e] = 0.f;

  const int rbase = warp * RPW;
  const float* rowp[RPW];
  bool rok[RPW];
#pragma unroll
  for (int u = 0; u < RPW; ++u) {
    rok[u] = rbase + u < t.rows;
    rowp[u] = M + (long long)(t.row0 + (rok[u] ? rbase + u : 0)) * m;
  }

  const int cend = t.col0 + t.cols;
  // as in the NT tile, the first loads go out ahead of the wait
  float v0[RPW][4], v1[RPW][4];
  auto load = [&](float (&v)[RPW][4], int c0) {
#pragma unroll
    for (int u = 0; u < RPW; ++u) load_lane_cols<VEC>(rowp[u], c0, cend, lane, rok[u], v[u]);
  };
  load(v0, t.col0);
  load(v1, t.col0 + NN_CHUNK_COLS);   // (zeros where the tile has no such chunk)
  psgd_wait_for_predecessor();

  // element (column lc of the tile, k): chunk of 128 columns, then word of 4 floats, then lane
  const float* qin = a.in + mt.q_off + (long long)t.col0 * r;   // written by the launch before: plain loads
  auto place = [&](int lc, int k) {   // in sQ
    const int b = lc & 127;
    const int ln = col_lane<VEC>(b), c = col_of_lane<VEC>(b);
    const int f = c * RT + k;
    return sQ + (((lc >> 7) * RT + (f >> 2)) * 32 + ln) * 4 + (f & 3);
  };
  // the values of a column lie together in both: copies of up to 16 bytes where the alignment allows them. Zeros for what the loop
  // reads besides: columns beyond the tile in its last chunk, values beyond the rank
  constexpr int W = RT >= 4 ? 4 : RT;
  const bool wide = RT > 1 && r == RT && ((uintptr_t)qin & (4 * W - 1)) == 0;
  if (wide) {
    for (int e = tid; e < t.cols * (RT / W); e += GEMM_THREADS) {
      const int lc = e / (RT / W), k = e % (RT / W) * W;
      if (W == 4 && RT <= 8) psgd_copy16_shared(place(lc, k), qin + e * W);
      else if (W == 4) psgd_copy16(place(lc, k), qin + e * W);
      else psgd_copy8(place(lc, k), qin + e * W);
    }
  }
  for (int lc = (wide ? t.cols : 0) + tid; lc < ((t.cols + 127) & ~127); lc += GEMM_THREADS) {
#pragma unroll
    for (int k = 0; k < RT; ++k) {
      if (lc < t.cols && k < r) psgd_copy4(place(lc, k), qin + lc * r + k);
      else *place(lc, k) = 0.f;
    }
  }
  psgd_copies_wait();
  __syncthreads();

  const float4* q4 = reinterpret_cast<const float4*>(sQ) + lane;
  auto use = [&](const float (&v)[RPW][4]) {
#pragma unroll
    for (int w = 0; w < RT; ++w) {
      const float4 q = q4[w * 32];
      const float qv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = (w * 4 + i) / RT, k = (w * 4 + i) % RT;
#pragma unroll
        for (int u = 0; u < RPW; ++u) acc[u * RT + k] = fmaf(v[u][c], qv[i], acc[u * RT + k]);
      }
    }
    q4 += RT * 32;
  };
  for (int c0 = t.col0; c0 < cend; c0 += 2 * NN_CHUNK_COLS) {
    use(v0);
    if (c0 + 2 * NN_CHUNK_COLS < cend) load(v0, c0 + 2 * NN_CHUNK_COLS);
    if (c0 + NN_CHUNK_COLS < cend) {
      use(v1);
      if (c0 + 3 * NN_CHUNK_COLS < cend) load(v1, c0 + 3 * NN_CHUNK_COLS);
    }
  }

  constexpr int N = RPW * RT < 32 ? RPW * RT : 32;   // values added up at a time
#pragma unroll
  for (int first = 0; first < RPW * RT; first += N) {
    float part[N];
#pragma unroll
    for (int i = 0; i < N; ++i) part[i] = acc[first + i];
    const float s = warp_sums<N>(part, lane);
    constexpr int SPAN = 32 / N;   // lanes that hold the same sum
    if (lane % SPAN == 0) sSum[rbase * RT + first + lane / SPAN] = s;
  }
  __syncthreads();

  constexpr int tile_elems = TILE_ROWS * RT;
  bool owner = true;
  if (t.nsplit > 1) {
    float* mine = a.partial + (long long)(t.slot0 + t.split) * tile_elems;
    for (int e = tid; e < tile_elems; e += GEMM_THREADS) __stcg(mine + e, sSum[e]);
    __threadfence();
    __syncthreads();
    if (tid == 0) sLast = (psgd_atom_add_acqrel_gpu(a.tickets + t.ticket, 1) == t.nsplit - 1);
    __syncthreads();
    owner = sLast != 0;
    if (owner) {
      __threadfence();
      psgd_sum_partials<tile_elems, GEMM_THREADS>(a.partial + (long long)t.slot0 * tile_elems, t.nsplit, sSum);
      if (tid == 0) a.tickets[t.ticket] = 0;
      __syncthreads();
    }
  }

  float* __restrict__ pout = a.out + mt.p_off;
  uint2* push[PSGD_MAX_WORLD];
  int e1 = 0;
  int npush = 0;
  if (a.comm != nullptr && owner) {
    const PsgdCommDev c = *a.comm;
    e1 = *c.epoch + 1;
    npush = c.world;
    for (int p = 0; p < PSGD_MAX_WORLD; ++p) push[p] = p < c.world ? psgd_comm_slot(c, p, e1, c.rank) + mt.p_off : nullptr;
  }
  for (int e = tid; owner && e < t.rows * r; e += GEMM_THREADS) {
    const int lr = e / r, k = e % r;
    const int row = t.row0 + lr;
    float s = sSum[lr * RT + k];
    for (int i = 0; i < a.ncorr; ++i) {
      const float* f = a.corr_fac[i] + mt.p_off + (long long)row * r;
      const float* cm = a.corr_c[i] + (long long)mt.index * PSGD_CMAT_STRIDE;
      float d = 0.f;
      for (int l = 0; l < r; ++l) d = fmaf(f[l], cm[l * r + k], d);
      s -= d;
    }
    pout[(long long)row * r + k] = s;
    if (a.out2) a.out2[mt.p_off + (long long)row * r + k] = s;
    for (int p = 0; p < npush; ++p) psgd_comm_store(push[p] + (long long)row * r + k, s, e1);
  }
}

// Rows of a warp: 64 sums at most in registers. Every row more spreads the rows of Q-hat that a tile stages, as many bytes as 32 rows
// of its part of the matrix at rank 16, over more of them: 4 x 1024x1001 at rank 16, two rows / four 19.1 / 13.9 us, 3 x 9000x650 at rank
// 11 69.8 / 62.2.
template <int RT>
__host__ __device__ constexpr int nn_rows_per_warp() { return RT <= 16 ? 4 : 2; }
// PER_SM: CTAs of an SM that registers have to allow. More registers let more of a tile's loads run ahead, which is what a launch of at most
// two tiles per SM needs; with more tiles a third CTA does more: us per pass, two / three, 3 x 1001x777 + 2 x 515x2049 at rank
// 3 x 3 (198 tiles) 89.4 / 94.1, ResNet-18's recorded step (443) 105.6 / 102.2, LSTM step (1532) 212.7 / 212.0. At rank 1 a fourth one, where
// that saves a round; launches alone, three / four, 6 x 512x4608 (480 tiles) 10.5 / 9.2, 16000x1000 (500) 7.5 / 6.8, 4 x 4000x650 (500) 6.6 / 6.9, 2 x
// 16000x1000 (1000) 23.2 / 21.9; where it saves none, 10000x1001 (313) 6.0 / 9.2, 40 x 512^2 (640) 5.9 / 6.3.
template <int RT, int RPW, int PER_SM>
__global__ void __launch_bounds__(GEMM_THREADS, PER_SM) psgd_gemm_nn_kernel(GemmArgs a) {
  extern __shared__ __align__(16) float smem[];   // staged rows of Q-hat
  __shared__ float sSum[GEMM_WARPS * RPW * RT];
  psgd_launch_dependents();
  const PsgdTile t = a.tiles[blockIdx.x];
  const PsgdMat mt = a.mats[t.mat];
  if (t.vec == 4) gemm_nn_tile<RT, 4, RPW>(a, t, mt, smem, sSum);
  else if (t.vec == 2) gemm_nn_tile<RT, 2, RPW>(a, t, mt, smem, sSum);
  else gemm_nn_tile<RT, 1, RPW>(a, t, mt, smem, sSum);
}

// ------------------------------------------------------------------------------------------
// Host launchers
// ------------------------------------------------------------------------------------------
static void fill_args(GemmArgs& a, const void* mats, const void* tiles, const float* in, float* out, float* out2,
                      int ncorr, const float* const* corr_fac, const float* const* corr_c, float* partial,
                      int* tickets, const void* comm) {
  a.mats = (const PsgdMat*)mats;
  a.tiles = (const PsgdTile*)tiles;
  a.in = in;
  a.out = out;
  a.out2 = out2;
  a.ncorr = ncorr;
  for (int i = 0; i < PSGD_MAX_HIST; ++i) {
    a.corr_fac[i] = i < ncorr ? corr_fac[i] : nullptr;
    a.corr_c[i] = i < ncorr ? corr_c[i] : nullptr;
  }
  a.partial = partial;
  a.tickets = tickets;
  a.comm = (const PsgdCommDev*)comm;
}

template <int RT>
static int launch_nt(const GemmArgs& a, int ntiles, int early, cudaStream_t stream) {
  const size_t smem = (size_t)(nt_stage_floats<RT>() + NT_TILE_COLS * RT) * sizeof(float);
  if (smem > 48 * 1024) {
    static unsigned long long devices = 0;   // per instantiation
    if (const int code = psgd_allow_shared((const void*)psgd_gemm_nt_kernel<RT>, smem, devices)) return code;
  }
  return psgd_launch(psgd_gemm_nt_kernel<RT>, ntiles, GEMM_THREADS, smem, stream, early, a);
}

template <int RT>
static int launch_nn(const GemmArgs& a, int ntiles, int early, cudaStream_t stream) {
  constexpr int RPW = nn_rows_per_warp<RT>();
  const size_t smem = (size_t)nn_max_cols<RT>() * RT * sizeof(float);
  if (RT >= 8 || ntiles <= 2 * 148) return psgd_launch(psgd_gemm_nn_kernel<RT, RPW, 2>, ntiles, GEMM_THREADS, smem, stream, early, a);
  if (RT == 1 && psgd_ceil_div(ntiles, 4 * 148) < psgd_ceil_div(ntiles, 3 * 148)) return psgd_launch(psgd_gemm_nn_kernel<RT, RPW, RT == 1 ? 4 : 2>, ntiles, GEMM_THREADS, smem, stream, early, a);
  return psgd_launch(psgd_gemm_nn_kernel<RT, RPW, RT >= 8 ? 2 : 3>, ntiles, GEMM_THREADS, smem, stream, early, a);
}

#define PSGD_DISPATCH_RT(FN)                                   \
  if (max_r <= 1) return FN<1>(a, ntiles, early, stream);             \
  if (max_r <= 2) return FN<2>(a, ntiles, early, stream);             \
  if (max_r <= 4) return FN<4>(a, ntiles, early, stream);             \
  if (max_r <= 8) return FN<8>(a, ntiles, early, stream);             \
  if (max_r <= 16) return FN<16>(a, ntiles, early, stream);           \
  return FN<32>(a, ntiles, early, stream);

// Rows handled by one NN tile for the template rank that `max_r` selects (the planner needs it).
PSGD_API int psgd_gemm_nn_tile_rows(int max_r) {
  const int rt = max_r <= 1 ? 1 : max_r <= 2 ? 2 : max_r <= 4 ? 4 : max_r <= 8 ? 8 : max_r <= 16 ? 16 : 32;
  return GEMM_WARPS * (rt <= 16 ? nn_rows_per_warp<16>() : nn_rows_per_warp<32>());
}
// Most columns of an NN tile (a multiple of 128).
PSGD_API int psgd_gemm_nn_max_cols(int max_r) { return max_r <= 8 ? 1024 : max_r <= 16 ? nn_max_cols<16>() : nn_max_cols<32>(); }
PSGD_API int psgd_gemm_nt_max_rows(int max_r) { return max_r <= 16 ? NT_MAX_ROWS : NT_MAX_ROWS / 2; }
PSGD_API int psgd_gemm_template_rank(int max_r) {
  return max_r <= 1 ? 1 : max_r <= 2 ? 2 : max_r <= 4 ? 4 : max_r <= 8 ? 8 : max_r <= 16 ? 16 : 32;
}

// `transposed` bit 0: NT (Q = M^T P), else NN (P = M Q); bit 1: the launch directly before this one in
// `stream` is one of this library's that leaves the gradients alone (see psgd_launch). Every tile carries the access width of
// its matrix (`vec`: 4 needs a 16-byte aligned base and m % 4 == 0; 2 an 8-byte aligned base and
// an even m). `out2`, when not null, receives a second copy of the fresh factor.
PSGD_API int psgd_gemm_ffma_launch(int transposed, int max_r, const void* mats, const void* tiles, int ntiles,
                                   const float* in, float* out, float* out2, int ncorr,
                                   const float* const* corr_fac, const float* const* corr_c, float* partial,
                                   int* tickets, const void* comm, cudaStream_t stream) {
  if (ntiles <= 0) return 0;
  if (max_r > PSGD_MAX_RANK || ncorr > PSGD_MAX_HIST) {
    psgd_set_error("psgd_gemm_ffma_launch: rank %d or history %d beyond the compiled maximum", max_r, ncorr);
    return -1;
  }
  GemmArgs a;
  fill_args(a, mats, tiles, in, out, out2, ncorr, corr_fac, corr_c, partial, tickets, comm);
  const int early = (transposed >> 1) & 1;
  if (transposed & 1) { PSGD_DISPATCH_RT(launch_nt) }
  PSGD_DISPATCH_RT(launch_nn)
}

#ifdef PSGD_BOUNDS_CHECK
PSGD_BOUNDS_EXPORT(psgd_bounds_read_products)
// Capacities (floats / counters) of the partial-sum arena, the ticket table and the P- and Q-shaped
// factor buffers of the launches that follow; 0 leaves a capacity unchecked.
PSGD_API int psgd_debug_limits_products(long long partial_floats, long long tickets, long long p_floats, long long q_floats) {
  PSGD_CUDA_OK(cudaMemcpyToSymbol(g_lim_partial, &partial_floats, sizeof(long long)));
  PSGD_CUDA_OK(cudaMemcpyToSymbol(g_lim_tickets, &tickets, sizeof(long long)));
  PSGD_CUDA_OK(cudaMemcpyToSymbol(g_lim_p, &p_floats, sizeof(long long)));
  PSGD_CUDA_OK(cudaMemcpyToSymbol(g_lim_q, &q_floats, sizeof(long long)));
  return 0;
}
#endif
