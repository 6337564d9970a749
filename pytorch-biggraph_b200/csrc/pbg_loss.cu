// Loss, its gradient, masks and batch statistics, one warp per positive edge and problem.
// Fuses, for a whole wave:
//   the ignore masks (-1e9)             torchbiggraph/model.py:566-580, 836-844
//   logistic / ranking / softmax        torchbiggraph/losses.py:53-161
//   relation weight, sum of both sides  torchbiggraph/batching.py:139-150
//   violator counts                     torchbiggraph/train_cpu.py:98-99
//   d(loss)/d(score)                    (autograd of the above)
// and rewrites the score matrix S_p in place as the coefficient matrix T_p whose two products
// with the operand tiles are the backward pass of the comparator:
//   dot / cos :  T_ij = dS_ij,            T_ii = d(loss)/d(pos score_i)
//   l2        :  T_ij = -dS_ij / S_ij     (= -2 dLoss/d(squared distance)), same on the diagonal
//   squared_l2:  T_ij = 2 dS_ij
// The diagonal of S is always masked, which is what frees it to carry the positive pair.
#include "pbg_rows.cuh"

#define LOSS_WARPS 8

template <int NV>
__global__ void __launch_bounds__(32 * LOSS_WARPS) loss_kernel(WaveDims d, WaveBatches wb, WaveBufs w) {
  pdl_begin();
  const int item = (int)blockIdx.x * LOSS_WARPS + (int)(threadIdx.x >> 5);
  const int per_prob = d.nblk * d.Pm;
  if (item >= 2 * per_prob) return;
  const int p = item >= per_prob ? 1 : 0, rem = item - p * per_prob;
  const int lb = d.byPm.div(rem);
  loss_row<NV>(d, wb, w, p, d.blk0 + lb, rem - lb * d.Pm, threadIdx.x & 31);
}

// l2 family: column sums of T_p over the chunk's positives (coefficient of the negative row's own |b|^2 term).  A CTA takes
// 32 columns: its eight warps bring up to 128 rows of them into shared memory at once, one warp adds them up in row order.
// (The sum of a column is one chain, and a thread that read its own column sixteen rows at a time waited for memory seven times
// over a chunk of 100 rows: 26 us for 60 chunks of 200 columns, 16 so.)
#define COLSUM_ROWS 128
__global__ void __launch_bounds__(256) colsum_kernel(WaveDims d, WaveBatches wb, WaveBufs w) {
  pdl_begin();
  __shared__ float rows[COLSUM_ROWS][32];
  const int p = blockIdx.z, blk = d.blk0 + blockIdx.y, lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + lane;
  const BlockInfo bi = block_info(d, wb, blk);
  const float *T = w.S[p] + (size_t)blk * d.Pm * d.Ms + j;
  float s = 0.f;
  for (int i0 = 0; i0 < bi.n; i0 += COLSUM_ROWS) {
    const int n = bi.n - i0 < COLSUM_ROWS ? bi.n - i0 : COLSUM_ROWS;
    float v[COLSUM_ROWS / 8];
#pragma unroll
    for (int u = 0; u < COLSUM_ROWS / 8; ++u) v[u] = j < d.Mm && wl + 8 * u < n ? T[(size_t)(i0 + wl + 8 * u) * d.Ms] : 0.f;
#pragma unroll
    for (int u = 0; u < COLSUM_ROWS / 8; ++u) rows[wl + 8 * u][lane] = v[u];
    __syncthreads();
    if (wl == 0) {
#pragma unroll 16
      for (int i = 0; i < n; ++i) s += rows[i][lane];
    }
    __syncthreads();
  }
  if (wl == 0 && j < d.Mm) w.coef[p][(size_t)blk * d.Mm + j] = s;
}

// Standard relations: a chunk row is scored in both problems (as a negative of one, as the
// scored side of the other), and both gradients land on the same prepared row.  One warp per
// (side, block, row m) merges them into the combined coefficient matrix A[side] (see WaveBufs), so
// that the backward pass is ONE product per side with K = Mm, and keeps the row sum of A for the
// l2 family (coefficient of the row's own |y|^2 term).
template <int NV>
__global__ void __launch_bounds__(32 * LOSS_WARPS) coef_kernel(WaveDims d, WaveBatches wb, WaveBufs w) {
  pdl_begin();
  int lane = threadIdx.x & 31;
  const int item = (int)blockIdx.x * LOSS_WARPS + (int)(threadIdx.x >> 5);
  const int per_side = d.nblk * d.Mm;
  if (item >= 2 * per_side) return;
  const int side = item >= per_side ? 1 : 0, rem = item - side * per_side;
  const int lb = d.byMm.div(rem), m = rem - lb * d.Mm;
  const int blk = d.blk0 + lb;
  BlockInfo bi = block_info(d, wb, blk);
  if (bi.n == 0) return;
  // side 0 (lhs rows): negatives of problem 0 (columns of T0), scored side of problem 1 (rows of T1)
  const float *Tcol = w.S[side] + (size_t)blk * d.Pm * d.Ms;        // T_side[j][m], j < Pm
  const float *Trow = w.S[1 - side] + ((size_t)blk * d.Pm + m) * d.Ms;   // T_other[m][j], m < Pm
  size_t arow = ((size_t)blk * d.Mm + m) * w.Ma;
  float *A = w.A[side] + arow;
  float rowsum = 0.f;
  // bf16-plane tier: the planes of the row beside it
  unsigned short *ABr = w.AB[side] ? w.AB[side] + ((size_t)blk * w.npl * d.Mm + m) * w.Kb : nullptr;
  // NV columns per lane at a time, read before the first of them is written (see loss_kernel)
  for (int j0 = lane; j0 < w.Ma; j0 += 32 * NV) {
    float a[NV];
#pragma unroll
    for (int u = 0; u < NV; ++u) {
      const int j = j0 + 32 * u;
      a[u] = 0.f;
      if (j < d.Mm) {
        if (j < bi.n) a[u] += Tcol[(size_t)j * d.Ms + m];
        if (m < bi.n) a[u] += Trow[j];
      }
    }
#pragma unroll
    for (int u = 0; u < NV; ++u) {
      const int j = j0 + 32 * u;
      if (j >= w.Ma) break;
      rowsum += a[u];
      A[j] = a[u];
      if (ABr) put_planes1(ABr + j, (size_t)d.Mm * w.Kb, a[u], w.npl);
    }
  }
  if (d.cmp >= PBG_CMP_L2) {
    rowsum = warp_sum(rowsum);
    if (lane == 0) w.coef[side][(size_t)blk * d.Mm + m] = rowsum;
  }
}

template <int NV>
__global__ void __launch_bounds__(32 * LOSS_WARPS) loss_softmax_kernel(WaveDims d, WaveBatches wb, WaveBufs w) {
  pdl_begin();
  const int item = (int)blockIdx.x * LOSS_WARPS + (int)(threadIdx.x >> 5);
  const int per_prob = d.nblk * d.Pm;
  if (item >= 2 * per_prob) return;
  const int p = item >= per_prob ? 1 : 0, rem = item - p * per_prob;
  const int lb = d.byPm.div(rem);
  loss_softmax_row<NV>(d, wb, w, p, d.blk0 + lb, rem - lb * d.Pm, threadIdx.x & 31);
}

// Combined coefficient matrices under the dot / cos comparators, one warp per 32 x 32 tile of
// A[side]: lane l reads 32 consecutive values of row j0 + l of T_side (whole 128-byte lines, eight
// 16-byte loads) and keeps them; value r of every lane is then column j0 + l of output row m0 + r,
// so that both the transposed term and the direct term T_other[m][j] are read and A is written in
// whole lines without a shuffle or shared memory.
template <bool PL>
__global__ void __launch_bounds__(32 * LOSS_WARPS) coef_tile_kernel(WaveDims d, WaveBatches wb, WaveBufs w) {
  pdl_begin();
  int lane = threadIdx.x & 31;
  const int item = (int)blockIdx.x * LOSS_WARPS + (int)(threadIdx.x >> 5);
  const int tiles = (d.Mm + 31) / 32;
  const long long per_side = (long long)d.nblk * tiles * tiles;
  if (item >= 2 * per_side) return;
  const int side = item >= per_side ? 1 : 0;
  const unsigned rem = (unsigned)(item - side * per_side);
  int lb = (int)(rem / (unsigned)(tiles * tiles)), tt = (int)(rem - (unsigned)lb * tiles * tiles);
  int m0 = (tt / tiles) * 32, j0 = (tt % tiles) * 32;
  const int blk = d.blk0 + lb;
  BlockInfo bi = block_info(d, wb, blk);
  if (bi.n == 0) return;
  const int j = j0 + lane;
  float t[32];
  const float *src = w.S[side] + ((size_t)blk * d.Pm + j) * d.Ms + m0;       // T_side[j][m0 ..]
  const bool has = j < bi.n;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    float4 v = (has && m0 + 4 * q < d.Ms) ? ld4(src + 4 * q) : f4zero();
    t[4 * q] = v.x; t[4 * q + 1] = v.y; t[4 * q + 2] = v.z; t[4 * q + 3] = v.w;
  }
  const float *orow = w.S[1 - side] + (size_t)blk * d.Pm * d.Ms;              // T_other[m][j]
  // All 32 values of the direct term are requested before the first is used: added as they came, each read waited for the
  // one before it (12 us for 20 blocks of 100 rows, 20 us for 70 blocks of 200).
  float o[32];
#pragma unroll
  for (int r = 0; r < 32; ++r) o[r] = m0 + r < bi.n && j < d.Mm ? orow[(size_t)(m0 + r) * d.Ms + j] : 0.f;
#pragma unroll
  for (int r = 0; r < 32; ++r) {
    const float a = t[r] + o[r];
    t[r] = m0 + r >= bi.n ? t[r] : a;                   // (the sum is left alone where there is no second term)
    if (j >= d.Mm || m0 + r >= d.Mm) t[r] = 0.f;
  }
  float *A = w.A[side] + (size_t)blk * d.Mm * w.Ma;
  if (!PL) {
#pragma unroll
    for (int r = 0; r < 32; ++r) {
      int m = m0 + r;
      if (m < d.Mm && j < w.Ma) A[(size_t)m * w.Ma + j] = t[r];
    }
    return;
  }
  // bf16-plane tier: the three planes instead of the fp32 matrix.  Two rows at a time: neighbouring
  // lanes swap one row's planes, so that every lane stores two columns of one row (4-byte stores):
  // even lanes the columns (j, j + 1) of row m, odd lanes (j - 1, j) of row m + 1.
  unsigned short *AB = w.AB[side] + (size_t)blk * w.npl * d.Mm * w.Kb;
  const size_t aplane = (size_t)d.Mm * w.Kb;
  const int npl = w.npl;
  const bool odd = lane & 1;
#pragma unroll
  for (int r = 0; r < 32; r += 2) {
    unsigned pl[2][3];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      bf16_planes(t[r + h], pl[h][0], pl[h][1], pl[h][2]);
    }
    // what the neighbour stores: its row is m for an even neighbour, m + 1 for an odd one
    unsigned give[3], keep[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) { give[q] = odd ? pl[0][q] : pl[1][q]; keep[q] = odd ? pl[1][q] : pl[0][q]; }
    unsigned g01 = __shfl_xor_sync(0xffffffffu, give[0] | (give[1] << 16), 1);
    unsigned g2 = __shfl_xor_sync(0xffffffffu, give[2], 1);
    unsigned got[3] = {g01 & 0xffffu, g01 >> 16, g2};
    const int m = m0 + r + (odd ? 1 : 0), col = j & ~1;
    if (m < d.Mm && col < w.Kb) {
      unsigned short *dst = AB + (size_t)m * w.Kb + col;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        unsigned lo = odd ? got[q] : keep[q], hi = odd ? keep[q] : got[q];
        if (q < npl) *(unsigned *)(dst + q * aplane) = lo | (hi << 16);
      }
    }
  }
}

int launch_loss(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st) {
  long long items = 2ll * d.nblk * d.Pm;
  const int loss_ctas = (int)((items + LOSS_WARPS - 1) / LOSS_WARPS);
  const bool dotlike = d.cmp < PBG_CMP_L2;
  if (dotlike && d.loss == PBG_LOSS_SOFTMAX && d.Ms <= 128) pbg_launch(loss_softmax_kernel<4>, loss_ctas, 32 * LOSS_WARPS, 0, st, d, wb, w);
  else if (dotlike && d.loss == PBG_LOSS_SOFTMAX && d.Ms <= 256) pbg_launch(loss_softmax_kernel<8>, loss_ctas, 32 * LOSS_WARPS, 0, st, d, wb, w);
  else if (dotlike && d.loss == PBG_LOSS_SOFTMAX && d.Ms <= 512) pbg_launch(loss_softmax_kernel<16>, loss_ctas, 32 * LOSS_WARPS, 0, st, d, wb, w);
  else if (dotlike && d.loss == PBG_LOSS_SOFTMAX && d.Ms <= 1024) pbg_launch(loss_softmax_kernel<32>, loss_ctas, 32 * LOSS_WARPS, 0, st, d, wb, w);
  else if (d.Ms <= 128) pbg_launch(loss_kernel<4>, loss_ctas, 32 * LOSS_WARPS, 0, st, d, wb, w);
  else if (d.Ms <= 256) pbg_launch(loss_kernel<8>, loss_ctas, 32 * LOSS_WARPS, 0, st, d, wb, w);
  else if (d.Ms <= 512) pbg_launch(loss_kernel<16>, loss_ctas, 32 * LOSS_WARPS, 0, st, d, wb, w);
  else if (d.Ms <= 1024) pbg_launch(loss_kernel<32>, loss_ctas, 32 * LOSS_WARPS, 0, st, d, wb, w);
  else pbg_launch(loss_kernel<0>, loss_ctas, 32 * LOSS_WARPS, 0, st, d, wb, w);
  if (!d.dynamic) {
    if (dotlike) {
      const int tiles = (d.Mm + 31) / 32;
      long long warps = 2ll * d.nblk * tiles * tiles;
      if (w.AB[0]) pbg_launch(coef_tile_kernel<true>, (int)((warps + LOSS_WARPS - 1) / LOSS_WARPS), 32 * LOSS_WARPS, 0, st, d, wb, w);
      else pbg_launch(coef_tile_kernel<false>, (int)((warps + LOSS_WARPS - 1) / LOSS_WARPS), 32 * LOSS_WARPS, 0, st, d, wb, w);
    } else {
      long long rows = 2ll * d.nblk * d.Mm;
      pbg_launch(coef_kernel<8>, (int)((rows + LOSS_WARPS - 1) / LOSS_WARPS), 32 * LOSS_WARPS, 0, st, d, wb, w);
    }
    return 2;
  }
  if (d.cmp >= PBG_CMP_L2) {
    dim3 g((d.Mm + 31) / 32, d.nblk, 2);
    pbg_launch(colsum_kernel, g, 256, 0, st, d, wb, w);
    return 2;
  }
  return 1;
}

// N3 regularizer value (torchbiggraph/regularizers.py:51-97), one warp per positive row of a chunk
// block: coef * sum m^3 over the adjusted rows of the edge -- standard relations: the prepared lhs
// row and the prepared op(rhs) row; dynamic relations: those of both passes (N0, Q0, N1, Q1) -- plus
// the operator parameters: per edge with dynamic relations; once per CHUNK with standard relations
// (sum(params^3) * len(src_pos) where src_pos is the [chunks, P, D] view, regularizers.py:88-92),
// which row 0 of the block carries.  Runs after the gather, on the snapshot the wave reads.
__global__ void __launch_bounds__(32 * LOSS_WARPS) reg_value_kernel(WaveDims d, WaveBatches wb, WaveBufs w) {
  pdl_begin();
  int lane = threadIdx.x & 31;
  const int item = (int)blockIdx.x * LOSS_WARPS + (int)(threadIdx.x >> 5);
  if (item >= d.nblk * d.Pm) return;
  const int lb = d.byPm.div(item), i = item - lb * d.Pm;
  const int blk = d.blk0 + lb;
  BlockInfo bi = block_info(d, wb, blk);
  if (bi.n == 0) return;
  size_t prow = (size_t)blk * d.Pm + i;
  float tot = 0.f;
  if (i < bi.n) {
    const bool cplx = d.op == PBG_OP_COMPLEX_DIAGONAL;
    const int D = d.D;
    const float *rows[6];
    int nr = 0;
    rows[nr++] = w.X[ARR_N0] + ((size_t)blk * w.xrows[ARR_N0] + i) * d.Dp;
    rows[nr++] = w.X[ARR_N1] + ((size_t)blk * w.xrows[ARR_N1] + i) * d.Dp;
    if (d.dynamic) {
      rows[nr++] = w.X[ARR_Q0] + ((size_t)blk * w.xrows[ARR_Q0] + i) * d.Dp;
      rows[nr++] = w.X[ARR_Q1] + ((size_t)blk * w.xrows[ARR_Q1] + i) * d.Dp;
    }
    if (d.op != PBG_OP_NONE) {
      if (d.dynamic) {
        long long rl = w.rel[bi.e0 + i];
        if (rl >= 0 && rl < d.num_rels) {
          if (w.theta[0]) rows[nr++] = w.theta[0] + (size_t)rl * D;
          if (w.theta[1]) rows[nr++] = w.theta[1] + (size_t)rl * D;
        }
      } else if (i == 0 && w.theta[0]) {
        rows[nr++] = w.theta[0] + (size_t)wb.rel[bi.b] * D;
      }
    }
    for (int q = 0; q < nr; ++q)
      for (int dd = lane * 4; dd < D; dd += 128) tot += n3_val4(rows[q], dd, D, cplx);
    tot = warp_sum(tot) * d.reg_coef;
  }
  if (lane == 0) w.regrow[prow] = tot;
}

int launch_reg_value(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st) {
  long long items = (long long)d.nblk * d.Pm;
  pbg_launch(reg_value_kernel, (int)((items + LOSS_WARPS - 1) / LOSS_WARPS), 32 * LOSS_WARPS, 0, st, d, wb, w);
  return 1;
}

// Scores as the reference returns them (model.py:842-844): [count] positives and
// [count, Pl + U] negatives per side with ignored entries set to -1e9; single batch (wave of 1).
__global__ void export_scores_kernel(WaveDims d, WaveBatches wb, WaveBufs w, float *lhs_pos, float *rhs_pos,
                                     float *lhs_neg, float *rhs_neg) {
  pdl_begin();
  int e = blockIdx.x;                       // edge of the batch
  int p = blockIdx.y;
  BlockInfo b0 = block_info(d, wb, 0);
  int Pl = b0.Pl;
  if (Pl == 0) return;
  int c = e / Pl, i = e - c * Pl;
  BlockInfo bi = block_info(d, wb, c);
  float *pos = p == 0 ? lhs_pos : rhs_pos;
  float *neg = p == 0 ? lhs_neg : rhs_neg;
  size_t prow = (size_t)c * d.Pm + i;
  if (threadIdx.x == 0) pos[e] = w.spos[p][prow];
  if (!d.neg_enabled[p]) return;
  int cols = d.batch_negs ? Pl + d.U : d.U;
  const float *S = w.S[p] + prow * d.Ms;
  for (int j = threadIdx.x; j < cols; j += blockDim.x) {
    int src = d.batch_negs ? (j < Pl ? j : d.Pm + (j - Pl)) : d.Pm + j;
    neg[(size_t)e * cols + j] = col_masked(d, bi, 1, i, src) ? PBG_MASKED : S[src];
  }
}

int launch_export_scores(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, float *lhs_pos,
                         float *rhs_pos, float *lhs_neg, float *rhs_neg, cudaStream_t st) {
  if (wb.n[0] <= 0) return 0;
  dim3 g(wb.n[0], 2);
  pbg_launch(export_scores_kernel, g, 128, 0, st, d, wb, w, lhs_pos, rhs_pos, lhs_neg, rhs_neg);
  return 1;
}

// ---- evaluation (RankingEvaluator, torchbiggraph/eval.py:43-81), one batch at a time -------------
// One warp per positive row and problem, one pass over its scores (four 16-byte loads in flight per lane): rank among the
// negatives and the loss (softmax with a running maximum).  The score matrix is read once and not written.  The samples of
// the randomized AUC (torchbiggraph/util.py:415-428: `count` random (positive, negative) pairs per side) are drawn by
// threads of their own, one sample each, in the first CTAs of the grid.  A CTA's eight warps are summed and the last CTA
// adds up the CTAs' sums.  (Rank, AUC, loss and sum as kernels of their own, the loss with the coefficient matrix it
// writes for training, took 107 us on 5000 edges against 1000 negatives a side; this kernel with one load in flight, the
// row's sample drawn by its warp's first lane and the last sum one dependent read after the other left 32 us behind
// the score kernel, now 22.)
struct EvalRow {
  float s, m = -INFINITY, acc = 0.f;
  int ge = 0;
  // four scores; `live`: bit u is set where column u counts, `exists`: where the reference's matrix has the column
  template <bool ALL>
  __device__ __forceinline__ void take(const float4 &q, int loss, float margin, unsigned live, unsigned exists) {
    float x[4] = {q.x, q.y, q.z, q.w};
    float mx = -INFINITY;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool on = ALL || (live >> u & 1u);
      ge += (ALL || (exists >> u & 1u)) && (on ? x[u] : PBG_MASKED) >= s;
      x[u] = on ? x[u] : -INFINITY;
      mx = fmaxf(mx, x[u]);
    }
    if (loss == PBG_LOSS_SOFTMAX) {
      if (mx > m) { acc *= expf(m - mx); m = mx; }              // (the first time: 0 x exp(-inf) = 0)
      if (m > -INFINITY)
#pragma unroll
        for (int u = 0; u < 4; ++u) acc += expf(x[u] - m);
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (x[u] > -INFINITY) acc += loss == PBG_LOSS_RANKING ? fmaxf(0.f, (x[u] - s) + margin) : softplusf(x[u]);
    }
  }
};

__global__ void __launch_bounds__(32 * LOSS_WARPS) eval_rows_kernel(WaveDims d, WaveBatches wb, WaveBufs w, int auc_ctas, double *part, unsigned *done, double *out8) {
  pdl_begin();
  __shared__ double sm[LOSS_WARPS][8];
  __shared__ float row_loss[LOSS_WARPS];
  __shared__ int row_ge[LOSS_WARPS], row_hits[LOSS_WARPS];     // negatives at or above the positive (-1: no row); AUC hits, 16 bits a side
  __shared__ bool closing;
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int count = wb.n[0], per_prob = d.nblk * d.Pm;
  float lossv = 0.f;
  int ge = -1, hits = 0;
  if ((int)blockIdx.x < auc_ctas) {
    const int id = (int)blockIdx.x * 32 * LOSS_WARPS + threadIdx.x, p = id >= count ? 1 : 0, smp = id - p * count;
    bool hit = false;
    if (smp < count && d.neg_enabled[p]) {
      const BlockInfo bi = block_info(d, wb, 0);
      const int Mlog = d.batch_negs ? bi.Pl + d.U : d.U;
      if (Mlog > 0) {
        unsigned long long h = pbg_mix64(w.seed ^ pbg_mix64(0xA0C0FFEEull + (unsigned long long)p * 0x10001ull + smp));
        const int ei = (int)(h % (unsigned long long)count);
        h = pbg_mix64(h);
        const long long flat = (long long)(h % ((unsigned long long)count * Mlog));
        const int er = (int)(flat / Mlog), j = (int)(flat - (long long)er * Mlog);
        const int src = d.batch_negs ? (j < bi.Pl ? j : d.Pm + (j - bi.Pl)) : d.Pm + j;
        const int c = er / bi.Pl, ii = er - c * bi.Pl;
        const BlockInfo b2 = block_info(d, wb, c);
        const float neg = col_masked(d, b2, 1, ii, src) ? PBG_MASKED : w.S[p][((size_t)c * d.Pm + ii) * d.Ms + src];
        hit = w.spos[p][(size_t)(ei / bi.Pl) * d.Pm + (ei % bi.Pl)] > neg;
      }
    }
    const unsigned h0 = __ballot_sync(0xffffffffu, hit && p == 0), h1 = __ballot_sync(0xffffffffu, hit && p == 1);
    hits = __popc(h0) | __popc(h1) << 16;
  }
  const int item = ((int)blockIdx.x - auc_ctas) * LOSS_WARPS + wl;
  if (item >= 0 && item < 2 * per_prob) {
    const int p = item >= per_prob ? 1 : 0, rem = item - p * per_prob;
    const int blk = d.byPm.div(rem), i = rem - blk * d.Pm;
    const BlockInfo bi = block_info(d, wb, blk);
    if (i < bi.n) {
      const size_t prow = (size_t)blk * d.Pm + i;
      const float *S = w.S[p] + prow * d.Ms;
      const float s = w.spos[p][prow];
      const float wr = wb.wrel[bi.b] * (w.ew ? w.ew[bi.e0 + i] : 1.0f);
      const bool enabled = d.neg_enabled[p] != 0;
      const int Mlog = !enabled ? 0 : (d.batch_negs ? bi.Pl + d.U : d.U);
      EvalRow r;
      r.s = s;
      if (enabled) {
        for (int j0 = lane * 4; j0 < d.Mm; j0 += 512) {
          float4 q[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) if (j0 + 128 * k < d.Mm) q[k] = ld4(S + j0 + 128 * k);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int j = j0 + 128 * k;
            if (j >= d.Mm) break;
            if (j >= d.Pm ? j + 3 < d.Mm : (d.batch_negs && j + 3 < bi.n && (unsigned)(i - j) >= 4u)) r.take<true>(q[k], d.loss, d.margin, 15u, 15u);
            else {
              unsigned live = 0u, exists = 0u;
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const int c = j + u;
                const bool e = c < d.Pm ? (d.batch_negs && c < bi.Pl) : c < d.Mm;       // a column of the reference's matrix
                exists |= (unsigned)e << u;
                live |= (unsigned)(e && (c >= d.Pm || (c != i && c < bi.n))) << u;
              }
              r.take<false>(q[k], d.loss, d.margin, live, exists);
            }
          }
        }
      }
      if (enabled) ge = warp_sum_int(r.ge);
      if (d.loss == PBG_LOSS_SOFTMAX) {
        const float mw = warp_max(r.m);
        const float z = warp_sum(r.m > -INFINITY ? r.acc * expf(r.m - mw) : 0.f);
        float mm = fmaxf(mw, s);
        if (mw == -INFINITY) mm = fmaxf(s, PBG_MASKED);               // every column masked
        if (Mlog > 0) lossv = -s + mm + logf((mw > -INFINITY ? z * expf(mw - mm) : 0.f) + expf(s - mm));
      } else {
        const float acc = warp_sum(r.acc);
        lossv = d.loss == PBG_LOSS_RANKING ? (Mlog > 0 ? acc : 0.f) : (Mlog > 0 ? acc / (float)Mlog : 0.f) + softplusf(-s);
      }
      lossv *= wr;
    }
  }
  if (lane == 0) { row_loss[wl] = lossv; row_ge[wl] = ge; row_hits[wl] = hits; }
  __syncthreads();
  if (threadIdx.x < 8) {                                       // the sums' doubles: eight rows at once, then a sum each
    const int rk = row_ge[threadIdx.x] + 1;
    const bool on = rk > 0;
    const double v[8] = {(double)row_loss[threadIdx.x], (double)rk, on ? 1.0 / rk : 0.0, (double)(on && rk <= 1), (double)(on && rk <= 10), (double)(on && rk <= 50),
                         (double)(row_hits[threadIdx.x] & 0xffff), (double)(row_hits[threadIdx.x] >> 16)};
#pragma unroll
    for (int k = 0; k < 8; ++k) sm[threadIdx.x][k] = v[k];
    __syncwarp(0xffu);
    double s = 0.0;
    for (int u = 0; u < LOSS_WARPS; ++u) s += sm[u][threadIdx.x];
    part[(size_t)blockIdx.x * 8 + threadIdx.x] = s;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) closing = atomicAdd(done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (closing) close_eval(part, gridDim.x, done, out8);
}

int launch_eval(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, double *part, unsigned *done, double *out8, cudaStream_t st) {
  pbg_launch(eval_rows_kernel, pbg_eval_ctas(d.nblk, d.Pm), 32 * LOSS_WARPS, 0, st, d, wb, w, pbg_eval_auc_ctas(d.nblk, d.Pm), part, done, out8);
  return 1;
}
