// Batched orthonormalisation of tall factor matrices, spread over the whole GPU.
//
// Replaces the reference's per-group `torch.linalg.qr` / joint-norm division
// (powersgd/orthogonalization.py:4-8) and the research harness' column-serial Gram-Schmidt
// (paper-code/gradient_reducers.py:945-956) with a Gram-matrix formulation that walks the
// tall matrix twice, whatever the rank (in a cluster, the second time from registers or L2):
//
//   G = X^T X        accumulated in float64, fixed summation order (bit-reproducible)
//   G = R^T R        Cholesky in float64, by one warp up to rank 4, by the whole block above
//   X <- X R^-1      by forward substitution in float64, rounded to float32 once
//
// With a float64 Gram matrix one pass is as orthonormal as float32 can express for any X
// that float32 can represent (error ~ 1e-16 * cond(X)^2 + 6e-8). A pivot below 1e-12 of its
// column's squared norm means the column is noise at float32 input precision; it is replaced
// by a canonical basis vector (what Householder QR yields for a zero column), so a factor
// that collapsed to zero (an all-zero gradient) recovers on the next step.
//
// Rank-1 units keep the reference's quirk: ONE Frobenius norm over the whole shape group
// (all B matrices jointly), floored at 1e-16, divides every entry.
//
// One launch with a cluster of CTAs per unit (psgd_orth_cluster_kernel), or, for long units, small models and
// several workers, two with one CTA per row chunk of a unit in both. The first writes the chunk's partial Gram
// matrix (and partial cross products F_i^T X against earlier factors of the same side). In the
// second EVERY chunk adds the partials of its unit in chunk order, factorises the sum and solves
// its own rows; one chunk per earlier factor also publishes the cross products
// C_i = (F_i^T X) R^-1 = F_i^T X_hat that the product kernels use to deflate algebraically.
// Both launches are bound by latency (a factor is tens of kilobytes), so what counts is the length
// of the dependent chain: factorising redundantly takes the place of an arrival counter, a memory
// fence, a lone last CTA and a second round trip through memory, and the second launch is
// released early (programmatic dependent launch) so that only its wait remains. Both launches
// together, before and after: 21 factors of ResNet-18 at rank 2 12.3 / 9.3 us, 50257 x 16 43 / 24 us; with the factorisation as
// a loop, loads in batches and rows by way of shared memory 50257 x 1024 at rank 16 445 -> 433 us per pass, 4 x 1024^2 at rank 8
// 57.8 -> 55.3.
//
// Multi-GPU: the factor to orthonormalise is the SUM over workers of what the previous product
// launch pushed into this rank's slot arena. The first launch is then also the consumer of that
// in-kernel all-reduce (powersgd/powersgd.py:205-209 in the reference is a blocking library
// call): every CTA polls the tagged words of its rows in the W slots, adds them in rank order, and
// writes the sum to the factor buffer and to the copy the decompression reads.
#include "psgd_bounds.cuh"
#include "psgd_comm.cuh"

typedef struct {
  int32_t x_off;      // float offset of the unit inside the factor buffer
  int32_t sub_len;    // rows of one sub-matrix
  int32_t nsub;       // sub-matrices in the unit (> 1 only for rank-1 groups)
  int32_t r;          // columns
  int32_t first_mat;  // descriptor index of sub-matrix 0 (sub-matrices are consecutive)
  int32_t chunk0;     // index of the unit's first chunk (chunks of a unit are consecutive)
  int32_t nchunks;
  int32_t pad;
} PsgdOrthUnit;  // 32 bytes

typedef struct {
  int32_t unit;
  int32_t sub;    // sub-matrix the chunk lies in (chunks never straddle sub-matrices)
  int32_t row0;   // first row, counted from the start of the unit
  int32_t rows;
} PsgdOrthChunk;  // 16 bytes

struct OrthArgs {
  const PsgdOrthUnit* units;
  const PsgdOrthChunk* chunks;
  float* x;                          // factor buffer, orthonormalised in place
  float* copy_to;                    // optional second destination (same layout) or null
  int nprev;                         // earlier same-side factor buffers
  const float* prev[PSGD_MAX_HIST];  // each laid out like x
  float* cmat[PSGD_MAX_HIST];        // out: [mat][r*r] blocks with stride PSGD_CMAT_STRIDE
  double* part;                      // scratch: [chunk][1 + nprev][RT*RT] partial sums
  float* head;                       // scratch: [unit][2*RT*RT] the unit's first 2r rows as they came in: what
                                     // replacing a column needs of X while other chunks overwrite it in place
  const PsgdCommDev* comm;           // not null: x is first gathered from the channel's slots (see above)
  float* sum_out;                    // with comm: second destination of the gathered sum (laid out like x)
};

constexpr int ORTH_THREADS = 256;
constexpr int ORTH_WARPS = ORTH_THREADS / 32;
constexpr int ORTH_STAGE_ROWS_X_RT = 2048;  // staged rows per pass at RT >= 8 = 2048 / RT, as float64: conversions
                                            // issue at a fraction of the FMA rate, so each value is converted
                                            // once and not once per pair it takes part in

// Rows of a chunk when the unit is short: two rows per thread of the second launch at RT <= 4, one
// staging pass of the first launch above that.
template <int RT>
__host__ __device__ constexpr int orth_base_rows() { return RT <= 4 ? 512 : ORTH_STAGE_ROWS_X_RT / RT; }

template <int RT>
__device__ __forceinline__ void orth_load_row(const float* p, int r, double* v) {
  if (RT == 4 && r == 4 && ((uintptr_t)p & 15u) == 0) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x; v[1 % RT] = q.y; v[2 % RT] = q.z; v[3 % RT] = q.w;
  } else if (RT == 2 && r == 2 && ((uintptr_t)p & 7u) == 0) {
    const float2 q = *reinterpret_cast<const float2*>(p);
    v[0] = q.x; v[1 % RT] = q.y;
  } else {
#pragma unroll
    for (int c = 0; c < RT; ++c) v[c] = c < r ? (double)p[c] : 0.0;
  }
}

// out[j * RT + k] = sum over the chunk's rows of a[row][j] * b[row][k], in float64 and in a fixed
// order. a, b: first row of the chunk, r floats per row. `stage`: 2 * ORTH_STAGE_ROWS_X_RT doubles.
template <int RT>
__device__ __forceinline__ void chunk_pairs(const float* a, const float* b, int r, int rows, double* stage, double* out, int tid) {
  constexpr int NP = RT * RT;
  if (RT <= 4) {
    // one row per thread, every pair in registers; lanes by shuffles, warps in index order
    double acc[NP];
#pragma unroll
    for (int e = 0; e < NP; ++e) acc[e] = 0.0;
#pragma unroll 2
    for (int row = tid; row < rows; row += ORTH_THREADS) {
      double va[RT], vb[RT];
      orth_load_row<RT>(a + (long long)row * r, r, va);
      orth_load_row<RT>(b + (long long)row * r, r, vb);
#pragma unroll
      for (int e = 0; e < NP; ++e) acc[e] = fma(va[e / RT], vb[e % RT], acc[e]);
    }
#pragma unroll
    for (int e = 0; e < NP; ++e) {
      const double s = psgd_warp_sum(acc[e]);
      if ((tid & 31) == 0) stage[(tid >> 5) * NP + e] = s;
    }
    __syncthreads();
    if (tid < NP) {
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < ORTH_WARPS; ++w) s += stage[w * NP + tid];
      out[tid] = s;
    }
    __syncthreads();
  } else {
    // rows staged as float64; every thread owns a 4 x 4 block of pairs and every NG-th row, so 8
    // values read feed 16 multiply-adds; at the end the row groups of a warp are added in pairs, the warps in index order
    constexpr int SR = ORTH_STAGE_ROWS_X_RT / RT;
    constexpr int NB = RT / 4 < 1 ? 1 : RT / 4;
    constexpr int NG = ORTH_THREADS / (NB * NB);
    constexpr int PER = SR * RT / ORTH_THREADS;   // staged values per thread
    double* sa = stage;
    double* sb = stage + ORTH_STAGE_ROWS_X_RT;
    const bool same = a == b;
    const int blk = tid % (NB * NB), g = tid / (NB * NB);
    const int j0 = blk / NB * 4, k0 = blk % NB * 4;
    double acc[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) acc[e] = 0.0;
    float na[PER], nb[PER];
    auto fetch = [&](int first) {
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int e = tid + i * ORTH_THREADS, row = first + e / RT, c = e % RT;
        const bool in = row < rows && c < r;
        na[i] = in ? a[(long long)row * r + c] : 0.f;
        nb[i] = (in && !same) ? b[(long long)row * r + c] : 0.f;
      }
    };
    fetch(0);
    const double* rb = same ? sa : sb;
    for (int first = 0; first < rows; first += SR) {
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        sa[tid + i * ORTH_THREADS] = (double)na[i];
        if (!same) sb[tid + i * ORTH_THREADS] = (double)nb[i];
      }
      __syncthreads();
      if (first + SR < rows) fetch(first + SR);  // lands while this pass is multiplied
      const int n = min(SR, rows - first);
#pragma unroll 2
      for (int row = g; row < n; row += NG) {
        const double2 a0 = *reinterpret_cast<const double2*>(sa + row * RT + j0), a1 = *reinterpret_cast<const double2*>(sa + row * RT + j0 + 2);
        const double2 b0 = *reinterpret_cast<const double2*>(rb + row * RT + k0), b1 = *reinterpret_cast<const double2*>(rb + row * RT + k0 + 2);
        const double va[4] = {a0.x, a0.y, a1.x, a1.y}, vb[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[e] = fma(va[e >> 2], vb[e & 3], acc[e]);
      }
      __syncthreads();
    }
    // sums over the row groups of a warp (its lanes GW apart hold the same pairs), then over the warps
    constexpr int GW = NB * NB < 32 ? NB * NB : 32;
    constexpr int LEFT = 16 * GW / 32 < 1 ? 1 : 16 * GW / 32;   // values a lane ends up with
    int off = 16;
#pragma unroll
    for (int n = 16; n > LEFT; n >>= 1, off >>= 1) {
      const bool upper = (tid & off) != 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i < n / 2) {
          const double keep = upper ? acc[i + n / 2] : acc[i], send = upper ? acc[i] : acc[i + n / 2];
          acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
      }
    }
    const int e0 = GW < 32 ? (tid & 31) / GW * LEFT : 0;   // the first of them
    constexpr int SETS = GW < 32 ? ORTH_WARPS : NG;        // (RT = 32: the groups are whole warps apart)
    const int set = GW < 32 ? tid >> 5 : g;
    static_assert(SETS * NP <= 2 * ORTH_STAGE_ROWS_X_RT, "the sums of the warps fit where the rows were staged");
#pragma unroll
    for (int i = 0; i < LEFT; ++i) {
      const int e = e0 + i;
      stage[set * NP + (j0 + (e >> 2)) * RT + k0 + (e & 3)] = acc[i];
    }
    __syncthreads();
    for (int p = tid; p < NP; p += ORTH_THREADS) {
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < SETS; ++w) s += stage[w * NP + p];
      out[p] = s;
    }
    __syncthreads();
  }
}

template <int RT>
__global__ void __launch_bounds__(ORTH_THREADS) psgd_orth_gram_kernel(OrthArgs a) {
  constexpr int NP = RT * RT;
  const PsgdOrthChunk ch = a.chunks[blockIdx.x];
  const PsgdOrthUnit u = a.units[ch.unit];
  const int r = u.r;
  const int tid = threadIdx.x;
  __shared__ __align__(16) double stage[RT <= 4 ? ORTH_WARPS * NP : 2 * ORTH_STAGE_ROWS_X_RT];
  psgd_launch_dependents();
  psgd_wait_for_predecessor();
#ifdef PSGD_BOUNDS_CHECK
  {
    bool ok = true;
    ok &= PSGD_BC(r >= 1 && r <= RT, 5, PSGD_BC_RANK, r, RT);
    ok &= PSGD_BC(ch.row0 >= 0 && ch.rows > 0 && (long long)ch.row0 + ch.rows <= (long long)u.sub_len * u.nsub,
                  5, PSGD_BC_CHUNK, (long long)ch.row0 + ch.rows, (long long)u.sub_len * u.nsub);
    ok &= PSGD_BC((int)blockIdx.x >= u.chunk0 && (int)blockIdx.x < u.chunk0 + u.nchunks, 5, PSGD_BC_CHUNK, blockIdx.x, u.chunk0 + u.nchunks);
    if (!ok) return;
  }
#endif
  const long long base = (long long)u.x_off + (long long)ch.row0 * r;
  float* x = a.x + base;
  if (a.comm != nullptr) {
    // gather: this chunk is a contiguous run of rows * r words in every slot
    const PsgdCommDev& c = *a.comm;
    const int e1 = *c.epoch + 1;
    float* sw = a.sum_out + base;
    const int n = ch.rows * r;
    bool ok = true;
    constexpr int NB = 4;
    for (int i0 = tid; i0 < n; i0 += NB * ORTH_THREADS) {
      int64_t idx[NB];
      float v[NB];
#pragma unroll
      for (int j = 0; j < NB; ++j) idx[j] = (i0 + j * ORTH_THREADS < n) ? base + i0 + j * ORTH_THREADS : -1;
      psgd_comm_reduce_batch<NB>(c, e1, idx, NB, v, ok);
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const int i = i0 + j * ORTH_THREADS;
        if (i < n) {
          x[i] = v[j];
          sw[i] = v[j];
        }
      }
    }
    psgd_comm_close_epoch(c, e1);  // (CTA barrier inside) every word of this chunk has been read
    __syncthreads();               // and every element of x written
  }
  const int stride = 1 + a.nprev;
  double* my_part = a.part + (long long)blockIdx.x * stride * NP;
  chunk_pairs<RT>(x, x, r, ch.rows, stage, my_part, tid);
  for (int p = 0; p < a.nprev; ++p) chunk_pairs<RT>(a.prev[p] + base, x, r, ch.rows, stage, my_part + (long long)(1 + p) * NP, tid);
  const int head_rows = min(2 * r - ch.row0, ch.rows);
  float* head = a.head + (long long)ch.unit * 2 * NP + (long long)ch.row0 * r;
  for (int e = tid; e < head_rows * r; e += ORTH_THREADS) head[e] = x[e];
}

// ---- factorisation ---------------------------------------------------------------------------
// R upper triangular with R^T R = G (row-major in sR, zero below the diagonal) and sDiagInv = 1 / R[c][c]; by one warp up to
// RT = 4, by the whole block above. A thread has one entry of the trailing matrix (four at RT = 32); a step hands the
// row just finished round through shared memory, and the rows are scaled by their pivots' square roots together at the end.
// What bounds it is not the chain of r pivots but fetching its code, which runs once per launch: with a column per lane
// in registers the r steps have to be unrolled, some 1250 cycles for each of 16 columns, nearly all of them
// instruction misses. As a loop: 5800 -> 1600 cycles at RT = 4, 12200 -> 2600 at 8, 24700 -> 4100 at 16.
// False (in all threads that take part) when a pivot is not above the rounding noise of its column (or is not a number).
template <int RT>
__device__ __forceinline__ bool orth_cholesky(const double* sG, double* sR, double* sDiagInv, int r, int tid) {
  constexpr int NP = RT * RT, PER = NP > ORTH_THREADS ? NP / ORTH_THREADS : 1;
  auto sync = [] {
    if (RT <= 4) __syncwarp();
    else __syncthreads();
  };
  double v[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) v[k] = tid + k * ORTH_THREADS < NP ? sG[tid + k * ORTH_THREADS] : 0.0;
#pragma unroll 1
  for (int c = 0; c < r; ++c) {
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int e = tid + k * ORTH_THREADS;
      if (e / RT == c) sR[e] = v[k];
    }
    sync();
    const double ref = sG[c * RT + c], piv = sR[c * RT + c];
    if (!((ref > 0.0) && (piv > 1e-12 * ref))) return false;
    const double inv = 1.0 / piv;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int e = tid + k * ORTH_THREADS;
      if (e < NP) v[k] = fma(-(sR[c * RT + e / RT] * inv), sR[c * RT + e % RT], v[k]);   // (rows up to c: of no use any more)
    }
  }
  sync();
  double scale[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int e = tid + k * ORTH_THREADS, row = e / RT;
    scale[k] = e < NP && row < r ? rsqrt(sR[row * RT + row]) : 0.0;
    v[k] = e < NP && row < r && e % RT >= row ? sR[e] * scale[k] : 0.0;
  }
  sync();
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int e = tid + k * ORTH_THREADS;
    if (e < NP) sR[e] = v[k];
    if (e < NP && e / RT == e % RT && e / RT < r) sDiagInv[e / RT] = scale[k];
  }
  return true;
}

// The same with canonical vectors in the place of columns that are noise: sDead[c] = -1 for a column
// that stays, the row of the basis vector that replaces it, or -2 for one that could not be
// completed (its output is zero). Rare (a factor that collapsed), so it is written for clarity.
template <int RT>
__device__ __noinline__ void orth_cholesky_substituting(double* sG, double* sR, double* sDiagInv, int* sDead, int r,
                                                        const float* head, long long len, int lane) {
  for (int e = lane; e < RT * RT; e += 32) sR[e] = 0.0;
  __syncwarp();
  for (int c = 0; c < r; ++c) {
    int attempt = 0;
    double piv = 0.0, inv_piv = 0.0;
    while (true) {
      double s = sG[c * RT + c];
      for (int i = 0; i < c; ++i) s -= sR[i * RT + c] * sR[i * RT + c];
      const double ref = sG[c * RT + c];
      const bool ok = (ref > 0.0) && (s > 1e-12 * ref);
      if (ok) { inv_piv = rsqrt(s); piv = s * inv_piv; break; }
      if (attempt == 2) { piv = 0.0; break; }
      // substitute column c by the basis vector e_row; its Gram entries are matrix entries
      const long long row = (attempt == 0 ? c : c + r) % len;
      ++attempt;
      __syncwarp();
      if (lane < r) {
        double g;
        if (lane == c) g = 1.0;
        else if (sDead[lane] >= 0) g = (sDead[lane] == (int)row) ? 1.0 : 0.0;
        else if (sDead[lane] == -2) g = 0.0;
        else g = (double)head[row * r + lane];
        sG[c * RT + lane] = g;
        sG[lane * RT + c] = g;
      }
      if (lane == 0) sDead[c] = (int)row;
      __syncwarp();
      // entries above the diagonal of column c were built from the old column: redo them
      if (lane == 0) {
        for (int i = 0; i < c; ++i) {
          if (sDead[i] == -2) { sR[i * RT + c] = 0.0; continue; }
          double t = sG[i * RT + c];
          for (int l = 0; l < i; ++l) t -= sR[l * RT + i] * sR[l * RT + c];
          sR[i * RT + c] = t * sDiagInv[i];
        }
      }
      __syncwarp();
    }
    __syncwarp();
    if (piv == 0.0) {
      // could not be completed: drop the column (its output is zero)
      if (lane == 0) {
        sDead[c] = -2;
        sR[c * RT + c] = 1.0;
        sDiagInv[c] = 1.0;
        for (int i = 0; i < c; ++i) sR[i * RT + c] = 0.0;
      }
      __syncwarp();
      continue;  // row c of R stays zero right of the diagonal
    }
    if (lane == 0) {
      sR[c * RT + c] = piv;
      sDiagInv[c] = inv_piv;
    }
    // row c of R, right of the diagonal: one lane per column
    for (int k = c + 1 + lane; k < r; k += 32) {
      double t = sG[c * RT + k];
      for (int i = 0; i < c; ++i) t -= sR[i * RT + c] * sR[i * RT + k];
      sR[c * RT + k] = t * inv_piv;
    }
    __syncwarp();
  }
}

// The two together, block-wide; sDead is set. Ends with a barrier.
template <int RT>
__device__ __forceinline__ void orth_factorise(double* sG, double* sR, double* sDiagInv, int* sDead, int r, const float* head, long long len, int tid) {
  if (tid < RT) sDead[tid] = -1;
  bool ok = true;
  if (RT > 4 || tid < 32) ok = orth_cholesky<RT>(sG, sR, sDiagInv, r, tid);
  if (!ok) {
    if (RT > 4) __syncthreads();   // everybody has read the pivot that failed
    __syncwarp();
    if (tid < 32) orth_cholesky_substituting<RT>(sG, sR, sDiagInv, sDead, r, head, len, tid);
  }
  __syncthreads();
}

// v <- v R^-1 for one row of RT values (columns beyond r are zero and stay so).
template <int RT>
__device__ __forceinline__ void orth_solve_row(double* v, const double* sR, const double* sDiagInv, int r) {
#pragma unroll
  for (int k = 0; k < RT; ++k) {
    if (k < r) {
      v[k] *= sDiagInv[k];
#pragma unroll
      for (int c = k + 1; c < RT; ++c) v[c] = fma(-v[k], sR[k * RT + c], v[c]);
    }
  }
}

// Sum over the unit's chunks, in a fixed order, of the partial matrix at `first` (one every `stride`
// doubles) into sOut[RT*RT]. Up to eight threads share one entry, each adding every eighth chunk.
template <int RT>
__device__ __forceinline__ void orth_sum_chunks(const double* first, long long stride, int nchunks, double* red, double* sOut, int tid) {
  constexpr int NP = RT * RT;
  constexpr int PARTS = NP * 8 <= ORTH_THREADS ? 8 : (NP < ORTH_THREADS ? ORTH_THREADS / NP : 1);
  for (int p = tid; p < NP * PARTS; p += ORTH_THREADS) {
    const int e = p % NP, part = p / NP;
    double s = 0.0;
    constexpr int B = RT <= 4 ? 8 : 16;   // loads under way
    // A short unit has one partial per thread and no use for the code below, which costs 5 to 14 % of both launches (0.3 us) to be run through.
    if (nchunks <= PARTS) s = part < nchunks ? __ldcg(first + part * stride + e) : 0.0;
    for (int c = nchunks <= PARTS ? nchunks : part; c < nchunks; c += B * PARTS) {
      double q[B];
#pragma unroll
      for (int j = 0; j < B; ++j) q[j] = c + j * PARTS < nchunks ? __ldcg(first + (c + j * PARTS) * stride + e) : 0.0;
#pragma unroll
      for (int j = 0; j < B; ++j) s += q[j];
    }
    if (PARTS == 1) sOut[e] = s;
    else red[p] = s;
  }
  __syncthreads();
  if (PARTS > 1) {
    if (tid < NP) {
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < PARTS; ++i) s += red[i * NP + tid];
      sOut[tid] = s;
    }
    __syncthreads();
  }
}

// X <- X' R^-1 on the rows of a CTA at RT >= 8, one row per thread. The rows pass through shared memory (`tile`, orth_tile_rows
// of them), so that global memory sees whole lines: a thread that reads and writes its own row of 16 floats by single
// accesses touches a line with each (50257 x 16: 20 000 -> 13 400 cycles for the 640 rows of a chunk). As everywhere in these launches code that runs once or twice costs some 5 cycles per
// instruction to be fetched: what is not the usual case (a rank below RT) is left to loops.
template <int RT>
__host__ __device__ constexpr int orth_tile_pitch() { return RT + 1; }   // odd: no two rows of a warp in one bank
template <int RT>
__host__ __device__ constexpr int orth_tile_rows() { return RT <= 16 ? ORTH_THREADS : ORTH_THREADS / 2; }
template <int RT>
__host__ __device__ constexpr int orth_tile_floats() { return orth_tile_rows<RT>() * orth_tile_pitch<RT>(); }
// Values of a tile per thread; at r = RT they are fetched into registers, a tile ahead.
template <int RT>
__host__ __device__ constexpr int orth_tile_values() { return orth_tile_rows<RT>() * RT / ORTH_THREADS; }
template <int RT>
__device__ __forceinline__ void orth_tile_fetch(const float* x, int rows, int r, float* q, int tid) {
  if (r != RT) return;
#pragma unroll
  for (int j = 0; j < orth_tile_values<RT>(); ++j) q[j] = tid + j * ORTH_THREADS < rows * RT ? x[tid + j * ORTH_THREADS] : 0.f;
}
template <int RT>
__device__ __forceinline__ void orth_solve_rows(float* x, float* x2, int row0, int rows, int r, const double* sR, const double* sDiagInv,
                                                const int* sDead, float* ahead, float* tile, int tid) {
  constexpr int T = orth_tile_rows<RT>(), TP = orth_tile_pitch<RT>(), STEP = ORTH_THREADS / RT * TP;
  float* mine = tile + tid / RT * TP + tid % RT;   // of the values that this thread moves at r = RT
#pragma unroll 1
  for (int first = 0; first < rows; first += T) {
    const int n = min(T, rows - first);
    float* to = x + (long long)first * r;
    float* to2 = x2 ? x2 + (long long)first * r : nullptr;
    if (r == RT) {
#pragma unroll
      for (int j = 0; j < orth_tile_values<RT>(); ++j) mine[j * STEP] = ahead[j];   // (zeros beyond the last row)
      if (first + T < rows) orth_tile_fetch<RT>(to + T * RT, min(T, rows - first - T), r, ahead, tid);
    } else {
#pragma unroll 4
      for (int e = tid; e < n * r; e += ORTH_THREADS) tile[e / r * TP + e % r] = to[e];
    }
    __syncthreads();
    if (tid < n) {
      float* row = tile + tid * TP;
      double v[RT];
#pragma unroll
      for (int k = 0; k < RT; ++k) {
        v[k] = k < r ? (double)row[k] : 0.0;
        if (k < r && sDead[k] != -1) v[k] = sDead[k] == row0 + first + tid ? 1.0 : 0.0;
      }
      orth_solve_row<RT>(v, sR, sDiagInv, r);
#pragma unroll
      for (int k = 0; k < RT; ++k)
        if (k < r) row[k] = (float)v[k];
    }
    __syncthreads();
    if (r == RT) {
#pragma unroll
      for (int j = 0; j < orth_tile_values<RT>(); ++j) {
        const int e = tid + j * ORTH_THREADS;
        if (e < n * RT) {
          const float q = mine[j * STEP];
          to[e] = q;
          if (to2) to2[e] = q;
        }
      }
    } else {
#pragma unroll 1
      for (int e = tid; e < n * r; e += ORTH_THREADS) {
        const float q = tile[e / r * TP + e % r];
        to[e] = q;
        if (to2) to2[e] = q;
      }
    }
    __syncthreads();
  }
}

// The same at RT <= 4: a row that a thread holds already.
template <int RT>
__device__ __forceinline__ void orth_row_solve(double* v, float* xr, float* xr2, int row, int r, const double* sR, const double* sDiagInv,
                                               const int* sDead) {
#pragma unroll
  for (int k = 0; k < RT; ++k)
    if (k < r && sDead[k] != -1) v[k] = sDead[k] == row ? 1.0 : 0.0;
  orth_solve_row<RT>(v, sR, sDiagInv, r);
  if (RT == 4 && r == 4 && (((uintptr_t)xr | (uintptr_t)xr2) & 15u) == 0) {
    const float4 q = make_float4((float)v[0], (float)v[1 % RT], (float)v[2 % RT], (float)v[3 % RT]);
    *reinterpret_cast<float4*>(xr) = q;
    if (xr2) *reinterpret_cast<float4*>(xr2) = q;
  } else if (RT == 2 && r == 2 && (((uintptr_t)xr | (uintptr_t)xr2) & 7u) == 0) {
    const float2 q = make_float2((float)v[0], (float)v[1 % RT]);
    *reinterpret_cast<float2*>(xr) = q;
    if (xr2) *reinterpret_cast<float2*>(xr2) = q;
  } else {
#pragma unroll
    for (int c = 0; c < RT; ++c)
      if (c < r) {
        xr[c] = (float)v[c];
        if (xr2) xr2[c] = (float)v[c];
      }
  }
}

// C = (F^T X') R^-1 from sG = F^T X, X' = X with the substituted columns; f: the unit's part of F.
template <int RT>
__device__ __forceinline__ void orth_publish(const double* sG, const float* f, float* cmat, int first_mat, int r, const double* sR,
                                             const double* sDiagInv, const int* sDead, int tid) {
  if (tid >= r) return;
  const double* v = sG + tid * RT;
  const auto value = [&](int k) {   // (column k of X' may be the basis vector e_d)
    const int d = sDead[k];
    return d == -1 ? v[k] : d >= 0 ? (double)f[(long long)d * r + tid] : 0.0;
  };
  double w[RT];
#pragma unroll
  for (int k = 0; k < RT; ++k) w[k] = k < r ? value(k) : 0.0;
  orth_solve_row<RT>(w, sR, sDiagInv, r);
  float* cm = cmat + (long long)first_mat * PSGD_CMAT_STRIDE + tid * r;
#pragma unroll
  for (int k = 0; k < RT; ++k)
    if (k < r) cm[k] = (float)w[k];
}

// Second launch: X <- X' R^-1 (rank 1: X / d) on every row chunk, optionally mirrored to copy_to.
// RT = 4: five CTAs per SM, as many as before the loads of the sums came in batches, or 100 units of 64 rows take 5.9 us in place of 5.0.
template <int RT>
__global__ void __launch_bounds__(ORTH_THREADS, RT == 4 ? 5 : 1) psgd_orth_apply_kernel(OrthArgs a) {
  constexpr int NP = RT * RT;
  const PsgdOrthChunk ch = a.chunks[blockIdx.x];
  const PsgdOrthUnit u = a.units[ch.unit];
  const int r = u.r;
  const int tid = threadIdx.x;
  __shared__ __align__(16) double sG[NP], sR[NP], sDiagInv[RT], red[ORTH_THREADS];
  __shared__ int sDead[RT];
  float* x = a.x + u.x_off;
  float* x2 = a.copy_to ? a.copy_to + u.x_off : nullptr;
  const long long stride = (long long)(1 + a.nprev) * NP;
  const double* unit_part = a.part + u.chunk0 * stride;
  const int ci = (int)blockIdx.x - u.chunk0;   // this chunk's number inside its unit
  psgd_launch_dependents();
  psgd_wait_for_predecessor();

  orth_sum_chunks<RT>(unit_part, stride, u.nchunks, red, sG, tid);
  if (RT == 1 || r == 1) {
    // joint Frobenius norm of the whole unit, float32 semantics of the division
    const float d = fmaxf((float)sqrt(sG[0]), 1e-16f);
    for (int i = tid; i < ch.rows; i += ORTH_THREADS) {
      const float v = x[ch.row0 + i] / d;
      x[ch.row0 + i] = v;
      if (x2) x2[ch.row0 + i] = v;
    }
    // cross products per sub-matrix: (sum of f * x over the sub-matrix) / d; every chunk has its share
    for (int e = ci * ORTH_THREADS + tid; e < a.nprev * u.nsub; e += u.nchunks * ORTH_THREADS) {
      const int p = e / u.nsub, s = e % u.nsub;
      const int per = u.nchunks / u.nsub;   // every sub-matrix has the same number of chunks
      double t = 0.0;
#pragma unroll 4
      for (int c = s * per; c < (s + 1) * per; ++c) t += __ldcg(unit_part + c * stride + (1 + p) * NP);
      a.cmat[p][(long long)(u.first_mat + s) * PSGD_CMAT_STRIDE] = (float)(t / (double)d);
    }
    return;
  }

  // the first rows travel while the sum is factorised
  double v[RT <= 4 ? RT : 1];
  __shared__ float tile[RT <= 4 ? 1 : orth_tile_floats<RT>()];
  float ahead[RT <= 4 ? 1 : orth_tile_values<RT>()];
  float* xc = x + (long long)ch.row0 * r;
  float* xc2 = x2 ? x2 + (long long)ch.row0 * r : nullptr;
  if constexpr (RT <= 4) {
    if (tid < ch.rows) orth_load_row<RT>(xc + (long long)tid * r, r, v);
  } else {
    orth_tile_fetch<RT>(xc, min(orth_tile_rows<RT>(), ch.rows), r, ahead, tid);
  }
  orth_factorise<RT>(sG, sR, sDiagInv, sDead, r, a.head + (long long)ch.unit * 2 * NP, (long long)u.sub_len * u.nsub, tid);
  if constexpr (RT <= 4) {
    for (int lr = tid; lr < ch.rows; lr += ORTH_THREADS) {
      float* xr = xc + (long long)lr * r;
      if (lr != tid) orth_load_row<RT>(xr, r, v);
      orth_row_solve<RT>(v, xr, xc2 ? xc2 + (long long)lr * r : nullptr, ch.row0 + lr, r, sR, sDiagInv, sDead);
    }
  } else {
    orth_solve_rows<RT>(xc, xc2, ch.row0, ch.rows, r, sR, sDiagInv, sDead, ahead, tile, tid);
  }
  // ---- cross products: chunk p of the unit (modulo their number) has factor p ----
  for (int p = ci; p < a.nprev; p += u.nchunks) {
    __syncthreads();
    orth_sum_chunks<RT>(unit_part + (long long)(1 + p) * NP, stride, u.nchunks, red, sG, tid);
    orth_publish<RT>(sG, a.prev[p] + u.x_off, a.cmat[p], u.first_mat, r, sR, sDiagInv, sDead, tid);
  }
}

// ---- one launch for both: a cluster of CTAs per unit -------------------------------------------
// What the two launches above spend on a short factor is mostly not theirs: the second one's start, the way of
// the partial sums through memory, and a second read of the rows. Here a cluster of ORTH_CLUSTER CTAs holds
// a unit: every CTA multiplies its rows, puts its partial matrices into the shared memory of all (of the one that publishes,
// for cross products), and after one cluster barrier everybody adds them in the order of the CTAs, factorises and
// solves the rows that it still has in registers (RT <= 4) or in L2. One worker only; units as psgd_orth_takes_clusters
// allows. Of the some 3 us that are left at RT = 4 a quarter each goes to the products, the exchange, the factorisation and the
// solution. us per pass, two launches / one: 3 x 1001x777 + 2 x 515x2049 at rank 3 x 3 114.7 / 99.6, ResNet-18's recorded step
// 112.5 / 108.4, 4 x 4096^2 at 4 x 2 378 / 369, 4 x 1024^2 at 8 x 1 55.3 / 54.2.
// `same`: the last earlier factor holds what x holds on entry, so its cross products are the Gram matrix.
constexpr int ORTH_CLUSTER = 8;

__device__ __forceinline__ uint32_t orth_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void orth_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void orth_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// *p = v in the shared memory of CTA `rank` of the cluster, where `p` is this CTA's address of it.
__device__ __forceinline__ void orth_put(double* p, uint32_t rank, double v) {
  uint32_t at;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}

// Sums of N doubles over the lanes, as warp_sums in lowrank_ffma.cu: value i ends up in the lanes whose top log2(N) bits spell i.
template <int N>
__device__ __forceinline__ double orth_warp_sums(double (&v)[N], int lane) {
  int off = 16;
#pragma unroll
  for (int n = N; n > 1; n >>= 1, off >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      if (i < n / 2) {
        const double keep = upper ? v[i + n / 2] : v[i], send = upper ? v[i] : v[i + n / 2];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
      }
    }
  }
  double s = v[0];
#pragma unroll
  for (; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  return s;
}

template <int RT>
__host__ __device__ constexpr int orth_kept_rows() { return RT == 1 ? 8 : 4; }   // per thread, RT <= 4
constexpr int ORTH_CLUSTER_SUBS = 64;   // cross products of whole sub-matrices that a CTA can have
// Shared memory in doubles: stage of the products; partial matrices of this CTA's rows; slots of the cluster for the
// Gram matrix and for the cross products that this CTA publishes; R and what belongs to it.
template <int RT>
__host__ __device__ constexpr int orth_stage_doubles() { return RT <= 4 ? ORTH_WARPS * RT * RT * PSGD_MAX_HIST : 2 * ORTH_STAGE_ROWS_X_RT; }
template <int RT>
__host__ __device__ constexpr int orth_cluster_doubles() {
  return orth_stage_doubles<RT>() + (RT <= 4 ? 0 : PSGD_MAX_HIST * RT * RT) + 2 * ORTH_CLUSTER * RT * RT + 2 * RT * RT + RT + ORTH_CLUSTER_SUBS;
}

template <int RT>
__global__ void __launch_bounds__(ORTH_THREADS) psgd_orth_cluster_kernel(OrthArgs a, int same) {
  constexpr int NP = RT * RT, CL = ORTH_CLUSTER;
  static_assert(RT <= 4 || orth_tile_floats<RT>() * sizeof(float) <= orth_stage_doubles<RT>() * sizeof(double), "the tile of rows takes the place of the stage");
  extern __shared__ __align__(16) double orth_smem[];
  double* stage = orth_smem;                                           // products; later the tile of rows (RT >= 8)
  double* mine = stage + orth_stage_doubles<RT>();                     // [1 + nprev][NP] (RT >= 8)
  double* slots = mine + (RT <= 4 ? 0 : PSGD_MAX_HIST * NP);           // [CL][NP]
  double* cross = slots + CL * NP;                                     // [CL][NP]
  double* sG = cross + CL * NP;
  double* sR = sG + NP;
  double* sDiagInv = sR + NP;
  double* subs = sDiagInv + RT;                                        // [ORTH_CLUSTER_SUBS]
  __shared__ int sDead[RT];
  const int ui = (int)blockIdx.x / CL;
  const PsgdOrthUnit u = a.units[ui];
  const uint32_t rank = orth_cluster_rank();
  const int r = u.r, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // rows of this CTA: a share of the unit; whole sub-matrices where there are several
  const int len = u.sub_len * u.nsub;
  const int per = u.nsub > 1 ? (u.nsub + CL - 1) / CL * u.sub_len : ((len + CL - 1) / CL + 3) / 4 * 4;
  const int row0 = min((int)rank * per, len), rows = min(per, len - row0);
  psgd_launch_dependents();
#ifdef PSGD_BOUNDS_CHECK
  {
    bool ok = true;   // the same verdict in all CTAs of a cluster
    ok &= PSGD_BC(r >= 1 && r <= RT, 5, PSGD_BC_RANK, r, RT);
    ok &= PSGD_BC(u.sub_len > 0 && u.nsub > 0 && (u.nsub == 1 || (r == 1 && (u.nsub + CL - 1) / CL * a.nprev <= ORTH_CLUSTER_SUBS)), 5, PSGD_BC_CHUNK, u.nsub, CL);
    ok &= PSGD_BC(a.nprev < CL, 5, PSGD_BC_CHUNK, a.nprev, CL);
    if (!ok) return;
  }
#endif
  orth_cluster_arrive();   // all CTAs run: their shared memory may be written
  psgd_wait_for_predecessor();
  float* x = a.x + u.x_off + (long long)row0 * r;
  float* x2 = a.copy_to ? a.copy_to + u.x_off + (long long)row0 * r : nullptr;
  const int crosses = a.nprev - same;   // products of their own
  {
    const int head_rows = min(2 * r - row0, rows);
    float* head = a.head + (long long)ui * 2 * NP + (long long)row0 * r;
    for (int e = tid; e < head_rows * r; e += ORTH_THREADS) head[e] = x[e];
  }

  if (u.nsub > 1) {
    // cross products of whole sub-matrices (r = 1): one warp for each of them and each factor
    for (int e = warp; e < rows / u.sub_len * a.nprev; e += ORTH_WARPS) {
      const int s = e / a.nprev, p = e % a.nprev;
      const float* f = a.prev[p] + u.x_off + row0 + s * u.sub_len;
      const float* g = x + s * u.sub_len;
      double t = 0.0;
#pragma unroll 8
      for (int i = lane; i < u.sub_len; i += 32) t = fma((double)f[i], (double)g[i], t);
      t = psgd_warp_sum(t);
      if (lane == 0) subs[e] = t;
    }
  }
  constexpr int KEPT = RT <= 4 ? orth_kept_rows<RT>() : 1;
  float kept[KEPT][RT <= 4 ? RT : 1];   // this thread's first rows of x
  if constexpr (RT <= 4) {
    const bool wide = (RT == 4 && r == 4 && ((uintptr_t)x & 15u) == 0) || (RT == 2 && r == 2 && ((uintptr_t)x & 7u) == 0);
    auto row_of = [&](const float* base, bool aligned, int row, float* v) {
      if (RT == 4 && aligned) {
        const float4 q = *reinterpret_cast<const float4*>(base + (long long)row * 4);
        v[0] = q.x; v[1 % RT] = q.y; v[2 % RT] = q.z; v[3 % RT] = q.w;
      } else if (RT == 2 && aligned) {
        const float2 q = *reinterpret_cast<const float2*>(base + (long long)row * 2);
        v[0] = q.x; v[1 % RT] = q.y;
      } else {
#pragma unroll
        for (int c = 0; c < RT; ++c) v[c] = c < r ? base[(long long)row * r + c] : 0.f;
      }
    };
    double acc[NP];
    auto add = [&](const float* f, const float* g) {
#pragma unroll
      for (int e = 0; e < NP; ++e) acc[e] = fma((double)f[e / RT], (double)g[e % RT], acc[e]);
    };
    auto close = [&](int p) {
      const double s = orth_warp_sums<NP>(acc, lane);
      if (lane % (32 / NP) == 0) stage[(p * ORTH_WARPS + warp) * NP + lane / (32 / NP)] = s;
#pragma unroll
      for (int e = 0; e < NP; ++e) acc[e] = 0.0;
    };
#pragma unroll
    for (int e = 0; e < NP; ++e) acc[e] = 0.0;
#pragma unroll
    for (int i = 0; i < KEPT; ++i) {
#pragma unroll
      for (int c = 0; c < RT; ++c) kept[i][c] = 0.f;
      if (tid + i * ORTH_THREADS < rows) row_of(x, wide, tid + i * ORTH_THREADS, kept[i]);
    }
    float first[KEPT][RT];   // the same rows of the first earlier factor travel beside them
    if (crosses > 0 && u.nsub == 1) {
      const float* f = a.prev[0] + u.x_off + (long long)row0 * r;
#pragma unroll
      for (int i = 0; i < KEPT; ++i) {
#pragma unroll
        for (int c = 0; c < RT; ++c) first[i][c] = 0.f;
        if (tid + i * ORTH_THREADS < rows) row_of(f, false, tid + i * ORTH_THREADS, first[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < KEPT; ++i) add(kept[i], kept[i]);
    for (int row = tid + KEPT * ORTH_THREADS; row < rows; row += ORTH_THREADS) {
      float v[RT];
      row_of(x, wide, row, v);
      add(v, v);
    }
    close(0);
    if (u.nsub == 1) {
      for (int p = 0; p < crosses; ++p) {
        const float* f = a.prev[p] + u.x_off + (long long)row0 * r;
        if (p == 0) {
#pragma unroll
          for (int i = 0; i < KEPT; ++i) add(first[i], kept[i]);
        }
        for (int row = tid + (p == 0 ? KEPT * ORTH_THREADS : 0); row < rows; row += ORTH_THREADS) {
          float v[RT], w[RT];
          row_of(f, false, row, w);
          row_of(x, wide, row, v);
          add(w, v);
        }
        close(1 + p);
      }
    }
    __syncthreads();
    orth_cluster_wait();
    if (tid < NP * CL) {
      const int e = tid % NP;
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < ORTH_WARPS; ++w) s += stage[w * NP + e];
      orth_put(slots + rank * NP + e, tid / NP, s);
    }
    if (u.nsub == 1) {
      for (int e = tid; e < crosses * NP; e += ORTH_THREADS) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < ORTH_WARPS; ++w) s += stage[((1 + e / NP) * ORTH_WARPS + w) * NP + e % NP];
        orth_put(cross + rank * NP + e % NP, e / NP, s);
      }
    }
  } else {
    chunk_pairs<RT>(x, x, r, max(rows, 0), stage, mine, tid);
    for (int p = 0; p < crosses && u.nsub == 1; ++p)
      chunk_pairs<RT>(a.prev[p] + u.x_off + (long long)row0 * r, x, r, max(rows, 0), stage, mine + (1 + p) * NP, tid);
    orth_cluster_wait();
    for (int e = tid; e < NP * CL; e += ORTH_THREADS) orth_put(slots + rank * NP + e % NP, e / NP, mine[e % NP]);
    for (int e = tid; e < crosses * NP && u.nsub == 1; e += ORTH_THREADS) orth_put(cross + rank * NP + e % NP, e / NP, mine[NP + e]);
  }
  orth_cluster_arrive();
  float ahead[RT <= 4 ? 1 : orth_tile_values<RT>()];
  if constexpr (RT > 4) orth_tile_fetch<RT>(x, min(orth_tile_rows<RT>(), rows), r, ahead, tid);
  orth_cluster_wait();   // every partial matrix is there, and every CTA has copied its rows of `head`
  for (int e = tid; e < NP; e += ORTH_THREADS) {
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < CL; ++c) s += slots[c * NP + e];
    sG[e] = s;
  }
  __syncthreads();

  if (RT == 1 || r == 1) {
    const float d = fmaxf((float)sqrt(sG[0]), 1e-16f);   // joint Frobenius norm, float32 semantics of the division
    auto put = [&](int i, float q) {
      q = q / d;
      x[i] = q;
      if (x2) x2[i] = q;
    };
    if constexpr (RT <= 4) {
#pragma unroll
      for (int i = 0; i < KEPT; ++i)
        if (tid + i * ORTH_THREADS < rows) put(tid + i * ORTH_THREADS, kept[i][0]);
    }
    for (int i = tid + (RT <= 4 ? KEPT * ORTH_THREADS : 0); i < rows; i += ORTH_THREADS) put(i, x[i]);
    if (u.nsub > 1) {
      for (int e = tid; e < rows / u.sub_len * a.nprev; e += ORTH_THREADS)
        a.cmat[e % a.nprev][(long long)(u.first_mat + row0 / u.sub_len + e / a.nprev) * PSGD_CMAT_STRIDE] = (float)(subs[e] / (double)d);
    } else if ((int)rank < a.nprev && tid == 0) {
      double t = 0.0;
      for (int c = 0; c < CL; ++c) t += ((int)rank < crosses ? cross : slots)[c * NP];
      a.cmat[rank][(long long)u.first_mat * PSGD_CMAT_STRIDE] = (float)(t / (double)d);
    }
    return;
  }

  orth_factorise<RT>(sG, sR, sDiagInv, sDead, r, a.head + (long long)ui * 2 * NP, len, tid);
  if constexpr (RT <= 4) {
    auto solve = [&](int lr, const float* q) {
      double v[RT];
#pragma unroll
      for (int c = 0; c < RT; ++c) v[c] = (double)q[c];
      orth_row_solve<RT>(v, x + (long long)lr * r, x2 ? x2 + (long long)lr * r : nullptr, row0 + lr, r, sR, sDiagInv, sDead);
    };
#pragma unroll
    for (int i = 0; i < KEPT; ++i)
      if (tid + i * ORTH_THREADS < rows) solve(tid + i * ORTH_THREADS, kept[i]);
    for (int lr = tid + KEPT * ORTH_THREADS; lr < rows; lr += ORTH_THREADS) {
      float q[RT];
#pragma unroll
      for (int c = 0; c < RT; ++c) q[c] = c < r ? x[(long long)lr * r + c] : 0.f;
      solve(lr, q);
    }
  } else {
    orth_solve_rows<RT>(x, x2, row0, rows, r, sR, sDiagInv, sDead, ahead, reinterpret_cast<float*>(stage), tid);
  }
  if ((int)rank < a.nprev) {
    __syncthreads();   // nobody reads the Gram matrix any more
    for (int e = tid; e < NP; e += ORTH_THREADS) {
      double s = 0.0;
#pragma unroll
      for (int c = 0; c < CL; ++c) s += ((int)rank < crosses ? cross : slots)[c * NP + e];
      sG[e] = s;
    }
    __syncthreads();
    orth_publish<RT>(sG, a.prev[rank] + u.x_off, a.cmat[rank], u.first_mat, r, sR, sDiagInv, sDead, tid);
  }
}

template <int RT>
static int orth_cluster_smem(size_t& smem) {
  smem = (size_t)orth_cluster_doubles<RT>() * sizeof(double);
  static unsigned long long devices = 0;   // per instantiation
  return smem > 48 * 1024 ? psgd_allow_shared((const void*)psgd_orth_cluster_kernel<RT>, smem, devices) : 0;
}

// Clusters that run at a time on the current device; 0 if it does not say.
template <int RT>
static int orth_clusters_at_a_time() {
  static int known[64] = {};   // by device, one more than that
  int device = 0, n = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return 0;
  int* at = known + device;
  const int before = __atomic_load_n(at, __ATOMIC_RELAXED);
  if (before > 0) return before - 1;
  size_t smem;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attrs[2];
  if (orth_cluster_smem<RT>(smem) != 0) return 0;
  psgd_launch_config(cfg, attrs, 1024 * ORTH_CLUSTER, ORTH_THREADS, smem, nullptr, 0, ORTH_CLUSTER);
  if (cudaOccupancyMaxActiveClusters(&n, psgd_orth_cluster_kernel<RT>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  __atomic_store_n(at, n + 1, __ATOMIC_RELAXED);
  return n;
}

template <int RT>
static int orth_cluster_launch(const OrthArgs& a, int nunits, int same, int early, cudaStream_t stream) {
  size_t smem;
  if (const int code = orth_cluster_smem<RT>(smem)) return code;
  return psgd_launch_clusters(psgd_orth_cluster_kernel<RT>, nunits * ORTH_CLUSTER, ORTH_THREADS, smem, stream, early, ORTH_CLUSTER, a, same);
}

template <int RT>
static int orth_launch_rt(const OrthArgs& a, int nchunks, int early, cudaStream_t stream) {
  const int rc = psgd_launch(psgd_orth_gram_kernel<RT>, nchunks, ORTH_THREADS, 0, stream, early & 1, a);
  if (rc != 0) return rc;
  return psgd_launch(psgd_orth_apply_kernel<RT>, nchunks, ORTH_THREADS, 0, stream, (early >> 1) & 1, a);
}

// Template rank used for factors of rank max_r, and the rows of one chunk at that rank.
PSGD_API int psgd_orth_template_rank(int max_r) {
  return max_r <= 1 ? 1 : max_r <= 2 ? 2 : max_r <= 4 ? 4 : max_r <= 8 ? 8 : max_r <= 16 ? 16 : 32;
}
// Rows of a chunk when the longest unit has `longest` rows. A short unit takes the base size. Every
// chunk of the second launch reads the partial matrices of ALL chunks of its unit, so their number is
// bounded for a long factor: at the bound the partial Gram matrices of a unit are 2, 8, 32, 64, 160 and
// 384 KiB at template ranks 1 to 32 (as much again per earlier factor for the chunk that publishes its
// cross products), read in as long as the chunk's own rows take. (An embedding of 50257 rows at rank 16: 79
// chunks instead of 393.) Chunks do not straddle the members of a rank-1 group, so a group of many
// matrices has at least one chunk per member, and their reads grow with the square of the members: 8 bytes
// per pair of members, 8 MB out of L2 for a thousand.
template <int RT>
static int orth_chunk_rows(long long longest) {
  const int base = orth_base_rows<RT>(), most = RT <= 4 ? 256 : RT == 8 ? 128 : RT == 16 ? 80 : 48;
  const long long rows = (longest + most - 1) / most;
  return (int)((rows + base - 1) / base > 1 ? (rows + base - 1) / base * base : base);
}
PSGD_API int psgd_orth_chunk_rows(int max_r, long long longest) {
  switch (psgd_orth_template_rank(max_r)) {
    case 1: return orth_chunk_rows<1>(longest);
    case 2: return orth_chunk_rows<2>(longest);
    case 4: return orth_chunk_rows<4>(longest);
    case 8: return orth_chunk_rows<8>(longest);
    case 16: return orth_chunk_rows<16>(longest);
    default: return orth_chunk_rows<32>(longest);
  }
}
// Whether one launch with a cluster per unit is the faster one for a list of `units` units, `rows` rows in all, whose longest unit has
// `longest` rows in at most `subs` sub-matrices, with `nprev` earlier factors. A cluster has eight SMs for a unit however long it
// is, the two launches have one per chunk. us, two launches / one, 1 and 24 units: rank 1, 4096 rows 3.9 / 2.4 and 4.8 / 2.8, 16384 4.3 / 2.7 and
// 5.9 / 3.2, 24000 4.3 / 4.9; rank 2, 4096 4.7 / 3.0 and 5.9 / 3.4, 12288 5.0 / 4.4 and 6.3 / 5.5, 24000 5.1 / 7.1; rank 4, 1024 5.7 / 3.3 and 6.7 /
// 3.6, 12288 6.3 / 5.5 and 10.4 / 6.9, 16384 6.4 / 6.8; rank 8, 1024 6.5 / 5.0 and 8.3 / 5.8, 2048 6.7 / 5.5 and 7.9 / 6.7, 4096 6.9 / 7.6 and 11.4 /
// 9.4; rank 16, 1024 8.5 / 7.7 and 10.2 / 9.5, 2048 9.0 / 9.5 and 15.1 / 12.4.
// Some 46 clusters run at a time up to rank 2 and 30 above; what is beyond them waits for a round of its own, while the two launches
// spread over all SMs. 64 rows, rank 2, 46, 60 and 400 units 4.0 / 3.2, 4.2 / 5.9, 4.8 / 27; rank 4, 30, 34 and 400 units 4.7 / 3.7, 4.8 / 6.6,
// 6.6 / 46; rank 16, 30, 34 and 400 units 9.0 / 7.9, 8.5 / 13.7, 13 / 99. Only where the rows bound both do more rounds pay: 60 units of 8192 rows at rank 1
// 7.7 / 5.7, 2 10.4 / 7.9, 4 16.6 / 10.2; of 4096 5.0 / 5.4, 6.6 / 6.7 and 10.2 / 8.6 (74 units 10.5 / 12.3).
PSGD_API int psgd_orth_takes_clusters(int max_r, long long longest, int subs, int nprev, int units, long long rows) {
  const int rt = psgd_orth_template_rank(max_r);
  if (rt > 16 || nprev >= ORTH_CLUSTER || (subs > 1 && (subs + ORTH_CLUSTER - 1) / ORTH_CLUSTER * nprev > ORTH_CLUSTER_SUBS)) return 0;
  if (longest > (rt == 1 ? 16384 : rt <= 4 ? 12288 : rt == 8 ? 3072 : 1536)) return 0;
  if (rt <= 4 && rows >= 8192ll * units) return 1;
  switch (rt) {
    case 1: return units <= orth_clusters_at_a_time<1>();
    case 2: return units <= orth_clusters_at_a_time<2>();
    case 4: return units <= orth_clusters_at_a_time<4>();
    case 8: return units <= orth_clusters_at_a_time<8>();
    default: return units <= orth_clusters_at_a_time<16>();
  }
}
// Scratch per chunk (doubles) for `nprev` earlier factors; per unit: 2 * RT*RT floats (`head`).
PSGD_API int psgd_orth_part_doubles(int max_r, int nprev) {
  const int rt = psgd_orth_template_rank(max_r);
  return (1 + nprev) * rt * rt;
}

// units / chunks: device tables; all units of one call share the template rank RT >= max r.
// part: nchunks * psgd_orth_part_doubles(max_r, nprev) doubles; head: nunits * 2 * RT*RT floats.
// comm / sum_out: see OrthArgs (null for a single worker or when x already holds the factor).
// early: see psgd_launch; bit 0 for the first launch, bit 1 for the second, which follows it; bit 2: one launch for both, a cluster per
// unit (lists for which psgd_orth_takes_clusters says so, no channel); bit 3, with bit 2: the last earlier factor holds the values of x.
// Bits 0 and 1 are off with
// several workers: the first launch then waits for peers, and the CTAs of an early successor would hold
// their places on the SMs meanwhile.
PSGD_API int psgd_orth_launch(const void* units, int nunits, const void* chunks, int nchunks, int max_r, float* x,
                              float* copy_to, int nprev, const float* const* prev, float* const* cmat,
                              double* part, float* head, const void* comm,
                              float* sum_out, int early, cudaStream_t stream) {
  if (nunits <= 0 || nchunks <= 0) return 0;
  if (max_r > PSGD_MAX_RANK || nprev > PSGD_MAX_HIST) {
    psgd_set_error("psgd_orth_launch: rank %d or history %d beyond the compiled maximum", max_r, nprev);
    return -1;
  }
  OrthArgs a;
  a.units = (const PsgdOrthUnit*)units;
  a.chunks = (const PsgdOrthChunk*)chunks;
  a.x = x;
  a.copy_to = copy_to;
  a.nprev = nprev;
  for (int i = 0; i < PSGD_MAX_HIST; ++i) {
    a.prev[i] = i < nprev ? prev[i] : nullptr;
    a.cmat[i] = i < nprev ? cmat[i] : nullptr;
  }
  a.part = part;
  a.head = head;
  a.comm = (const PsgdCommDev*)comm;
  a.sum_out = sum_out;
  if ((early & 4) != 0) {
    const int same = (early >> 3) & 1;
    if (comm != nullptr || nprev >= ORTH_CLUSTER || (same && nprev == 0)) {
      psgd_set_error("psgd_orth_launch: no cluster form for a channel, %d earlier factors (same: %d)", nprev, same);
      return -1;
    }
    switch (psgd_orth_template_rank(max_r)) {
      case 1: return orth_cluster_launch<1>(a, nunits, same, early & 1, stream);
      case 2: return orth_cluster_launch<2>(a, nunits, same, early & 1, stream);
      case 4: return orth_cluster_launch<4>(a, nunits, same, early & 1, stream);
      case 8: return orth_cluster_launch<8>(a, nunits, same, early & 1, stream);
      case 16: return orth_cluster_launch<16>(a, nunits, same, early & 1, stream);
      default:
        psgd_set_error("psgd_orth_launch: no cluster form at rank %d", max_r);
        return -1;
    }
  }
  if (comm != nullptr && sum_out == nullptr) {
    psgd_set_error("psgd_orth_launch: a channel was given without a destination for the gathered sum");
    return -1;
  }
  switch (psgd_orth_template_rank(max_r)) {
    case 1: return orth_launch_rt<1>(a, nchunks, early, stream);
    case 2: return orth_launch_rt<2>(a, nchunks, early, stream);
    case 4: return orth_launch_rt<4>(a, nchunks, early, stream);
    case 8: return orth_launch_rt<8>(a, nchunks, early, stream);
    case 16: return orth_launch_rt<16>(a, nchunks, early, stream);
    default: return orth_launch_rt<32>(a, nchunks, early, stream);
  }
}

#ifdef PSGD_BOUNDS_CHECK
PSGD_BOUNDS_EXPORT(psgd_bounds_read_orth)
#endif
