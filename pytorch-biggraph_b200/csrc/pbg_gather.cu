// Row gather fused with the relation operator and comparator.prepare: builds the operand tiles
// of one wave (see pbg_common.cuh for the layout) straight from the embedding tables, one warp
// per row slot, 16-byte loads and stores.  Replaces, for a whole wave at once,
//   F.embedding gathers                 torchbiggraph/model.py:57-61, 645-646
//   sample_entities                     torchbiggraph/model.py:70-75
//   adjust_embs (operator + prepare)    torchbiggraph/model.py:478-506, operators.py:49-157, 197-338
//   zero padding of the last chunk      torchbiggraph/model.py:787-800
//   the positive scores                 torchbiggraph/model.py:177, 267-274
// and emits the sort keys that group gradient slots by table row.
#include "pbg_rows.cuh"

#define GATHER_WARPS 8

// Resident CTAs per SM, by the float4 a lane holds of a row.  A warp waits for one row after the other, so what counts is warps, also
// where registers spill to memory for them (general kernel: 12 to 400 bytes of stores a thread up to 512 floats, 280 to 672 at 1024,
// 2,056 to 2,664 at 2048; a CTA less spills only at 2048, 380 to 948).  Gather class of a wave of 14 batches (1000 edges, 100 + 100
// negatives, one after the other), us, with a CTA less / this / a CTA more:
//   general kernel             128 floats           256              512                1024              2048
//     translation, cos         34.4 / 33.7 / 32.0   44.0/40.4/41.6   68.1/58.5/59.3     136 /104 /109     216 / 206
//       three planes           31.1 / 29.2 / 29.3   43.6/41.1/44.8   84.5/77.9/82.6     203 /164 /178     363 / 394
//     dynamic, complex, dot    37.3 / 36.8 / 36.1   55.6/49.7/53.1   104 /93.0/91.6     270 /199 /202     532 / 479
//       three planes           46.8 / 45.7 / 47.6   72.7/71.9/81.4   151 /149 /160      386 /315 /328     825 / 779
//   plain kernel, three planes, two CTAs less up to 256 floats, one more from 513: 64 floats 21.1 / 19.4, 128 23.4 / 21.8, 256 30.0 /
//   29.5, 768 83.7 / 79.1, 1024 108 / 99.7 (there the third spilled); without planes the same within 2 %.
// (One row in which a CTA less would do better: standard relations with planes at 2048 floats.)
template <int VEC> struct GatherCtas {
  enum { GENERAL = VEC >= 8 ? 2 : VEC == 4 ? 3 : VEC == 2 ? 4 : 5, PLAIN = VEC >= 16 ? 1 : VEC == 8 ? 2 : VEC == 4 ? 4 : 6 };
};

template <int VEC, bool PL>
__global__ void __launch_bounds__(32 * GATHER_WARPS, GatherCtas<VEC>::GENERAL) gather_kernel(WaveDims d, WaveBatches wb, WaveBufs w) {
  pdl_begin();
  const int item = (int)blockIdx.x * GATHER_WARPS + (int)(threadIdx.x >> 5);
  if (item >= d.nblk * d.Mm) return;
  const int lb = d.byMm.div(item);
  gather_slot<VEC, PL>(d, wb, w, d.blk0 + lb, item - lb * d.Mm, threadIdx.x & 31);
}

// The same work when nothing has to be computed on the way -- standard relations, no operator, dot
// comparator: the operand rows are plain copies of the table rows, and the positive score is their
// dot product.  Both rows of a slot (lhs side, rhs side) are loaded at once, which doubles the bytes
// a warp keeps in flight, and the kernel carries none of the operator / prepare code of the general
// one.
template <int VEC, bool PL>
__global__ void __launch_bounds__(32 * GATHER_WARPS, GatherCtas<VEC>::PLAIN) gather_plain_kernel(WaveDims d, WaveBatches wb, WaveBufs w) {
  pdl_begin();
  int lane = threadIdx.x & 31;
  const int item = (int)blockIdx.x * GATHER_WARPS + (int)(threadIdx.x >> 5);
  if (item >= d.nblk * d.Mm) return;
  const int lb = d.byMm.div(item), r = item - lb * d.Mm;
  const int blk = d.blk0 + lb;
  BlockInfo bi = block_info(d, wb, blk);
  const int D = d.D;
  size_t nrow = (size_t)blk * d.Mm + r;
  const size_t noff = nrow * d.Dp;
  float *n0 = w.X[ARR_N0] + noff, *n1 = w.X[ARR_N1] + noff;
  long long i0, i1;
  const bool edge = r < d.Pm;
  if (edge) {
    bool ok = r < bi.n;
    i0 = ok ? w.lhs[bi.e0 + r] : -1;
    i1 = ok ? w.rhs[bi.e0 + r] : -1;
    if (ok && (i0 < 0 || i0 >= d.n_rows[0] || i1 < 0 || i1 >= d.n_rows[1])) {
      if (lane == 0) atomicOr(w.errflag, 1);
      ok = false;
    }
    if (!ok) i0 = i1 = -1;                                  // padding row: exact zeros on both sides
  } else {
    i0 = slot_row(d, wb, w, bi, 0, r);
    i1 = slot_row(d, wb, w, bi, 1, r);
    if (i0 >= d.n_rows[0]) { if (lane == 0) atomicOr(w.errflag, 1); i0 = -1; }
    if (i1 >= d.n_rows[1]) { if (lane == 0) atomicOr(w.errflag, 1); i1 = -1; }
  }
  float4 a[VEC], b[VEC];
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    int dd = c * 128 + lane * 4;
    a[c] = (i0 >= 0 && dd < D) ? ld4(w.W[0] + (size_t)i0 * D + dd) : f4zero();
  }
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    int dd = c * 128 + lane * 4;
    b[c] = (i1 >= 0 && dd < D) ? ld4(w.W[1] + (size_t)i1 * D + dd) : f4zero();
  }
  if (i0 >= 0) add_global<VEC>(a, w.glob[0], D, lane);       // padding rows stay exact zeros
  if (i1 >= 0) add_global<VEC>(b, w.glob[1], D, lane);
  if (PL) {
    // bf16-plane tier: the contractions read the planes, nothing reads the fp32 operand rows
    const size_t plane = (size_t)d.Mm * w.Dpb;
    unsigned short *x0 = w.XB[0] + ((size_t)blk * w.npl * d.Mm + r) * w.Dpb, *x1 = w.XB[1] + ((size_t)blk * w.npl * d.Mm + r) * w.Dpb;
    const bool three = w.npl > 2;
#pragma unroll
    for (int c = 0; c < VEC; ++c) {
      int dd = c * 128 + lane * 4;
      if (dd < D) {
        uint2 p0, p1, p2;
        bf16_planes4(a[c], p0, p1, p2);
        *(uint2 *)(x0 + dd) = p0; *(uint2 *)(x0 + plane + dd) = p1;
        if (three) *(uint2 *)(x0 + 2 * plane + dd) = p2;
        bf16_planes4(b[c], p0, p1, p2);
        *(uint2 *)(x1 + dd) = p0; *(uint2 *)(x1 + plane + dd) = p1;
        if (three) *(uint2 *)(x1 + 2 * plane + dd) = p2;
      }
    }
  } else {
    store_row<VEC>(n0, a, D, lane);
    store_row<VEC>(n1, b, D, lane);
  }
  float s = 0.f;
  if (edge) {
#pragma unroll
    for (int c = 0; c < VEC; ++c) s += f4dot(a[c], b[c]);
    s = warp_sum(s);
  }
  if (lane == 0) {
    w.aux[ARR_N0][nrow] = 0.f; w.aux[ARR_N1][nrow] = 0.f;
    if (edge) { size_t q = (size_t)blk * d.Pm + r; w.spos[0][q] = s; w.spos[1][q] = s; }
  }
}

// linear / affine operators: R2 holds A.x for every rhs row of the chunk blocks; this kernel adds
// the translation (affine), applies comparator.prepare, writes the operand row to N1 and, for the
// chunk's edges, the positive score against the lhs row already in N0.
template <int VEC>
__global__ void __launch_bounds__(32 * GATHER_WARPS) postop_kernel(WaveDims d, WaveBatches wb, WaveBufs w) {
  pdl_begin();
  int lane = threadIdx.x & 31;
  const int item = (int)blockIdx.x * GATHER_WARPS + (int)(threadIdx.x >> 5);
  if (item >= d.nblk * d.Mm) return;
  const int lb = d.byMm.div(item), r = item - lb * d.Mm;
  const int blk = d.blk0 + lb;
  BlockInfo bi = block_info(d, wb, blk);
  const int D = d.D;
  size_t nrow = (size_t)blk * d.Mm + r, noff = nrow * d.Dp;
  long long id = slot_row(d, wb, w, bi, 1, r);
  bool ok = id >= 0 && id < d.n_rows[1];
  if (ok && r < d.Pm) {                         // the edge's lhs id must be valid too (gather zeroed the rows otherwise)
    long long il = w.lhs[bi.e0 + r];
    ok = il >= 0 && il < d.n_rows[0];
  }
  float4 z[VEC], y0[VEC];
  if (!ok) {
    zero_row<VEC>(w.X[ARR_N1] + noff, D, lane);
    if (lane == 0) {
      w.aux[ARR_N1][nrow] = 0.f;
      if (r < d.Pm) { size_t q = (size_t)blk * d.Pm + r; w.spos[0][q] = 0.f; w.spos[1][q] = 0.f; }
    }
    return;
  }
  load_row<VEC>(z, w.R2 + noff, D, lane);
  if (d.op == PBG_OP_AFFINE) {
    const float *t = w.theta[0] + (size_t)wb.rel[bi.b] * d.opw + (size_t)D * D;
#pragma unroll
    for (int c = 0; c < VEC; ++c) {
      int dd = c * 128 + lane * 4;
      if (dd < D) z[c] = z[c] + ld4(t + dd);
    }
  }
  float a1 = prepare_row<VEC>(z, d.cmp);
  store_row<VEC>(w.X[ARR_N1] + noff, z, D, lane);
  if (lane == 0) w.aux[ARR_N1][nrow] = a1;
  if (r < d.Pm) {
    load_row<VEC>(y0, w.X[ARR_N0] + noff, D, lane);
    float s = positive_score<VEC>(y0, z, d.cmp);
    size_t q = (size_t)blk * d.Pm + r;
    if (lane == 0) { w.spos[0][q] = s; w.spos[1][q] = s; }
  }
}

int launch_postop(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st) {
  long long items = (long long)d.nblk * d.Mm;
  int ctas = (int)((items + GATHER_WARPS - 1) / GATHER_WARPS);
  int vec = (d.D + 127) / 128;
  if (vec <= 1) pbg_launch(postop_kernel<1>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
  else if (vec <= 2) pbg_launch(postop_kernel<2>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
  else if (vec <= 4) pbg_launch(postop_kernel<4>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
  else if (vec <= 8) pbg_launch(postop_kernel<8>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
  else pbg_launch(postop_kernel<16>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
  return 1;
}

int launch_gather(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st) {
  long long items = (long long)d.nblk * d.Mm;
  int ctas = (int)((items + GATHER_WARPS - 1) / GATHER_WARPS);
  int vec = (d.D + 127) / 128;
  const bool plain = !d.dynamic && !d.matrix_op && d.max_norm <= 0.f && d.cmp == PBG_CMP_DOT && (d.op == PBG_OP_NONE || w.theta[0] == nullptr);
  if (plain && w.XB[0] && d.reg_coef == 0.f) {      // planes only: nothing reads the fp32 operand rows then
    if (vec <= 1) pbg_launch(gather_plain_kernel<1, true>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    else if (vec <= 2) pbg_launch(gather_plain_kernel<2, true>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    else if (vec <= 4) pbg_launch(gather_plain_kernel<4, true>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    else if (vec <= 8) pbg_launch(gather_plain_kernel<8, true>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    else pbg_launch(gather_plain_kernel<16, true>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    return 1;
  }
  if (plain && !w.XB[0]) {
    if (vec <= 1) pbg_launch(gather_plain_kernel<1, false>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    else if (vec <= 2) pbg_launch(gather_plain_kernel<2, false>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    else if (vec <= 4) pbg_launch(gather_plain_kernel<4, false>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    else if (vec <= 8) pbg_launch(gather_plain_kernel<8, false>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    else pbg_launch(gather_plain_kernel<16, false>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    return 1;
  }
  if (w.XB[0]) {
    if (vec <= 1) pbg_launch(gather_kernel<1, true>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    else if (vec <= 2) pbg_launch(gather_kernel<2, true>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    else if (vec <= 4) pbg_launch(gather_kernel<4, true>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    else if (vec <= 8) pbg_launch(gather_kernel<8, true>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    else pbg_launch(gather_kernel<16, true>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
    return 1;
  }
  if (vec <= 1) pbg_launch(gather_kernel<1, false>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
  else if (vec <= 2) pbg_launch(gather_kernel<2, false>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
  else if (vec <= 4) pbg_launch(gather_kernel<4, false>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
  else if (vec <= 8) pbg_launch(gather_kernel<8, false>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
  else pbg_launch(gather_kernel<16, false>, ctas, 32 * GATHER_WARPS, 0, st, d, wb, w);
  return 1;
}

// One thread per occurrence slot (waves too large for the one-kernel sort, which builds its keys itself).
__global__ void build_keys_kernel(WaveDims d, WaveBatches wb, WaveBufs w, unsigned long long *keys, unsigned int *vals) {
  pdl_begin();
  int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= d.nocc) return;
  keys[o] = slot_key(d, wb, w, o);
  vals[o] = (unsigned int)o;
}

int launch_build_keys(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w,
                      unsigned long long *keys, unsigned int *vals, cudaStream_t st) {
  pbg_launch(build_keys_kernel, (d.nocc + 255) / 256, 256, 0, st, d, wb, w, keys, vals);
  return 1;
}

// ------------------------------------------------------------------------------------------------
// Ranking against ALL entities of a side's table (relations with all_negs=True, torchbiggraph/model.py:582-617;
// what RankingEvaluator needs for full-ranking MRR, torchbiggraph/eval.py:43-81).  One chunk holds the whole
// batch, the negatives of a side are every row of its table, and an edge's own true entity is ignored.
//   allnegs_rows_kernel     per edge: the two scored rows (prepared, operator applied where the mode says so)
//                           and the positive score(s)
//   allnegs_slab_kernel     a slab of both tables' rows as candidates: global embedding, operator (standard relations,
//                           rhs side), prepare -> rows of Y (planes of YB) and the row's |y|^2; with the first slab
//                           also the samples of the randomized AUC
//   scores, never stored: per (tile of candidates, edge) the count scoring >= the positive and the loss partials --
//                           allnegs_tc_kernel (pbg_rank_tc.cu), or in the fp32 tier allnegs_score_kernel's 64 x 64 tiles
//   allnegs_merge_kernel    one warp per edge and side folds the slab's tiles into the running state; after the last
//                           slab ranks, loss and the evaluator's sums
// Both sides go through every launch together: a table that fits one slab takes four launches in all.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ int allnegs_rows_of(const WaveDims &d, const AllNegs &a, int side, long long row0) {
  if (!d.neg_enabled[side]) return 0;
  const long long left = d.n_rows[side] - row0;
  return left < 0 ? 0 : left < a.slab ? (int)left : a.slab;
}
template <int VEC>
__device__ __forceinline__ void store_planes(unsigned short *x, size_t plane, const float4 (&v)[VEC], int D, int lane) {
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    const int dd = c * 128 + lane * 4;
    if (dd < D) {
      uint2 p0, p1, p2;
      bf16_planes4(v[c], p0, p1, p2);
      *(uint2 *)(x + dd) = p0; *(uint2 *)(x + plane + dd) = p1; *(uint2 *)(x + 2 * plane + dd) = p2;
    }
  }
}
template <int VEC>
__device__ __forceinline__ void allnegs_q_planes(const AllNegs &a, int side, int e, const float4 (&v)[VEC], int D, int lane) {
  const size_t plane = (size_t)a.qrows * a.Dpb;
  store_planes<VEC>(a.QB + (size_t)side * 3 * plane + (size_t)e * a.Dpb, plane, v, D, lane);
}

template <int VEC>
__global__ void __launch_bounds__(32 * GATHER_WARPS) allnegs_rows_kernel(WaveDims d, WaveBufs w, AllNegs a, int rel_std) {
  pdl_begin_open(a.seam);
  int lane = threadIdx.x & 31;
  int e = blockIdx.x * GATHER_WARPS + (threadIdx.x >> 5);
  if (e >= a.B) return;
  const int D = d.D;
  long long il = w.lhs[e], ir = w.rhs[e], rl = d.dynamic ? 0 : rel_std;
  if (d.dynamic && d.op != PBG_OP_NONE) rl = w.rel[e];
  bool ok = il >= 0 && il < d.n_rows[0] && ir >= 0 && ir < d.n_rows[1] && (d.op == PBG_OP_NONE || (rl >= 0 && rl < d.num_rels));
  float *q0 = a.Q[0] + (size_t)e * d.Dp, *q1 = a.Q[1] + (size_t)e * d.Dp;
  if (!ok) {
    if (lane == 0) { atomicOr(w.errflag, 1); a.pos[0][e] = 0.f; a.pos[1][e] = 0.f; a.qn[0][e] = 0.f; a.qn[1][e] = 0.f; }
    zero_row<VEC>(q0, D, lane); zero_row<VEC>(q1, D, lane);
    if (a.QB) {
      float4 z[VEC];
#pragma unroll
      for (int c = 0; c < VEC; ++c) z[c] = f4zero();
      allnegs_q_planes<VEC>(a, 0, e, z, D, lane); allnegs_q_planes<VEC>(a, 1, e, z, D, lane);
    }
    return;
  }
  const float *xl = w.W[0] + (size_t)il * D, *xr = w.W[1] + (size_t)ir * D;
  float4 x[VEC], yl[VEC], yr[VEC], z[VEC];
  // lhs row, prepared (no operator)
  load_row<VEC>(x, xl, D, lane);
  const float scl = renorm_row<VEC>(x, d.max_norm);
  add_global<VEC>(x, w.glob[0], D, lane);
#pragma unroll
  for (int c = 0; c < VEC; ++c) yl[c] = x[c];
  float al = prepare_row<VEC>(yl, d.cmp);
  float s1 = 0.f, a1 = al;
  if (d.dynamic) {
    // problem 1 scores op_lhs(lhs) against the rhs candidates
    const float *th1 = (d.op != PBG_OP_NONE && w.theta[1]) ? w.theta[1] + (size_t)rl * D : nullptr;
    apply_operator<VEC>(z, x, xl, th1, d.op, D, lane, nullptr, scl);
    a1 = prepare_row<VEC>(z, d.cmp);
    store_row<VEC>(q1, z, D, lane);
    if (a.QB) allnegs_q_planes<VEC>(a, 1, e, z, D, lane);
  } else {
    store_row<VEC>(q1, yl, D, lane);
    if (a.QB) allnegs_q_planes<VEC>(a, 1, e, yl, D, lane);
  }
  // rhs row through the rhs operator, prepared
  load_row<VEC>(x, xr, D, lane);
  const float scr = renorm_row<VEC>(x, d.max_norm);
  add_global<VEC>(x, w.glob[1], D, lane);
  const float *th0 = (d.op != PBG_OP_NONE && w.theta[0]) ? w.theta[0] + (size_t)rl * D : nullptr;
  apply_operator<VEC>(yr, x, xr, th0, d.op, D, lane, w.glob[1], scr);
  float a0 = prepare_row<VEC>(yr, d.cmp);
  store_row<VEC>(q0, yr, D, lane);
  if (a.QB) allnegs_q_planes<VEC>(a, 0, e, yr, D, lane);
  float s0 = positive_score<VEC>(yl, yr, d.cmp);          // problem 0: c(lhs, op_rhs(rhs))
  if (d.dynamic) {
    // problem 1: c(prepared rhs without operator, op_lhs(lhs))
#pragma unroll
    for (int c = 0; c < VEC; ++c) yr[c] = x[c];
    prepare_row<VEC>(yr, d.cmp);
    s1 = positive_score<VEC>(yr, z, d.cmp);
  } else {
    s1 = s0;
  }
  if (lane == 0) {
    a.pos[0][e] = s0; a.pos[1][e] = s1;
    a.qn[0][e] = d.cmp >= PBG_CMP_L2 ? a0 : 0.f;
    a.qn[1][e] = d.cmp >= PBG_CMP_L2 ? a1 : 0.f;
  }
}

// one candidate: row `row` of the table of `side` through global embedding, operator and prepare; returns its |y|^2
template <int VEC>
__device__ __forceinline__ float allnegs_candidate(float4 (&z)[VEC], const WaveDims &d, const WaveBufs &w, int side, long long row, int rel_std, int lane) {
  const int D = d.D;
  const float *xrow = w.W[side] + (size_t)row * D;
  float4 x[VEC];
  load_row<VEC>(x, xrow, D, lane);
  const float sc = renorm_row<VEC>(x, d.max_norm);
  add_global<VEC>(x, w.glob[side], D, lane);
  // standard relations apply the operator to every rhs row, negatives included; with dynamic relations negatives get none
  const float *th = (side == 1 && !d.dynamic && d.op != PBG_OP_NONE && w.theta[0]) ? w.theta[0] + (size_t)rel_std * D : nullptr;
  apply_operator<VEC>(z, x, xrow, th, d.op, D, lane, w.glob[side], sc);
  return prepare_row<VEC>(z, d.cmp);
}

// grid (row groups, sides): candidates row0 .. of both tables; `auc_ctas` CTAs of each side take the AUC's samples (B of
// them), torchbiggraph/util.py:415-428: `count` random (positive, (edge, candidate)) pairs per side, hits left in auc[side].
// The candidates need nothing from the edges' rows, so the first slab starts as a sibling of allnegs_rows_kernel; the samples
// wait for it, in the middle of the grid's order (last of side 0, first of side 1), where neither the wait nor their chain of
// reads is the end of the kernel.  (One batch of 1000 edges against 14,951 rows of 400 floats a side: 185.2 us behind the rows and with the samples last, 184.3 so.)
template <int VEC>
__global__ void __launch_bounds__(32 * GATHER_WARPS) allnegs_slab_kernel(WaveDims d, WaveBufs w, AllNegs a, long long row0, int rel_std, int slab_ctas, int auc_ctas) {
  const int lane = threadIdx.x & 31, side = blockIdx.y, D = d.D;
  const int cta = (int)blockIdx.x - (side == 1 ? auc_ctas : 0);            // candidates: 0 .. slab_ctas - 1
  const bool samples = cta < 0 || cta >= slab_ctas;
  float4 z[VEC];
  if (!samples) {
    const bool sibling = row0 == 0;                                      // (a later slab follows the merge of the one before)
    if (!sibling) pdl_begin();
    else { pdl_release(); seam_enter(a.seam); }
    const int r = cta * GATHER_WARPS + (threadIdx.x >> 5);
    if (r < allnegs_rows_of(d, a, side, row0)) {
      const float aux = allnegs_candidate<VEC>(z, d, w, side, row0 + r, rel_std, lane);
      if (a.YB) {
        const size_t plane = (size_t)a.slab * a.Dpb;
        store_planes<VEC>(a.YB + (size_t)side * 3 * plane + (size_t)r * a.Dpb, plane, z, D, lane);
      } else {
        store_row<VEC>(a.Y[side] + (size_t)r * d.Dp, z, D, lane);
      }
      if (lane == 0) a.yn[side][r] = d.cmp >= PBG_CMP_L2 ? aux : 0.f;
    }
    return;                                                // (the samples' CTAs wait for the rows' end)
  }
  pdl_begin();
  const int smp = (cta < 0 ? (int)blockIdx.x : cta - slab_ctas) * GATHER_WARPS + (threadIdx.x >> 5);
  if (smp == 0 && side == 0) seam_close(a.seam);
  if (smp >= a.B || !d.neg_enabled[side]) return;
  unsigned long long h = pbg_mix64(w.seed ^ pbg_mix64(0xA11CE5ull + (unsigned long long)side * 0x10001ull + smp));
  const int ei = (int)(h % (unsigned long long)a.B);
  h = pbg_mix64(h);
  const int er = (int)(h % (unsigned long long)a.B);
  h = pbg_mix64(h);
  const long long cand = (long long)(h % (unsigned long long)d.n_rows[side]);
  float neg = PBG_MASKED;
  if (cand != (side == 0 ? w.lhs : w.rhs)[er]) {
    const float yn = allnegs_candidate<VEC>(z, d, w, side, cand, rel_std, lane);
    const float *qr = a.Q[side] + (size_t)er * d.Dp;
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < VEC; ++c) { const int dd = c * 128 + lane * 4; if (dd < D) s += f4dot(ld4(qr + dd), z[c]); }
    s = warp_sum(s);
    if (d.cmp >= PBG_CMP_L2) {
      const float qv = (yn - 2.0f * s) + a.qn[side][er];
      s = d.cmp == PBG_CMP_L2 ? -sqrtf(fmaxf(qv, 1e-30f)) : -qv;
    }
    neg = s;
  }
  if (lane == 0) a.auc[side][smp] = a.pos[side][ei] > neg ? 1 : 0;
}

#define AN_TILE 64
// grid (edge tiles, candidate tiles of the slab, sides); 256 threads, each a 4 x 4 block of the 64 x 64 score tile
__global__ void __launch_bounds__(256) allnegs_score_kernel(WaveDims d, WaveBufs w, AllNegs a, long long row0) {
  pdl_begin();
  __shared__ float sq[16][AN_TILE + 1], sy[16][AN_TILE + 1];
  __shared__ int scnt[16][AN_TILE];
  __shared__ float sa[16][AN_TILE], sb[16][AN_TILE];
  const int te = blockIdx.x, tc = blockIdx.y, side = blockIdx.z, t = threadIdx.x;
  const int n = allnegs_rows_of(d, a, side, row0);
  if (tc * AN_TILE >= n) return;
  const int ty = t >> 4, tx = t & 15;                        // rows 4 ty .. 4 ty + 3 (edges), cols 4 tx .. (candidates)
  const float *Q = a.Q[side];
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  const int e0 = te * AN_TILE, c0 = tc * AN_TILE;
  for (int k0 = 0; k0 < d.D; k0 += 16) {
    // 64 rows x 16 k of each operand: thread t loads row t / 4, k (t % 4) * 4 .. + 3
    int lr = t >> 2, lk = (t & 3) * 4;
    float4 vq = f4zero(), vy = f4zero();
    if (e0 + lr < a.B && k0 + lk < d.D) vq = ld4(Q + (size_t)(e0 + lr) * d.Dp + k0 + lk);
    if (c0 + lr < n && k0 + lk < d.D) vy = ld4(a.Y[side] + (size_t)(c0 + lr) * d.Dp + k0 + lk);
    __syncthreads();
    sq[lk][lr] = vq.x; sq[lk + 1][lr] = vq.y; sq[lk + 2][lr] = vq.z; sq[lk + 3][lr] = vq.w;
    sy[lk][lr] = vy.x; sy[lk + 1][lr] = vy.y; sy[lk + 2][lr] = vy.z; sy[lk + 3][lr] = vy.w;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      float qv[4], yv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { qv[i] = sq[k][ty * 4 + i]; yv[i] = sy[k][tx * 4 + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(qv[i], yv[j], acc[i][j]);
    }
  }
  // comparator, the ignored true entity, count and loss partials of this thread's 4 candidates per edge
  const long long *truth = side == 0 ? w.lhs : w.rhs;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int e = e0 + ty * 4 + i;
    int cnt = 0;
    float pa = 0.f, pb = d.loss == PBG_LOSS_SOFTMAX ? -INFINITY : 0.f;
    if (e < a.B) {
      const float pos = a.pos[side][e];
      const long long tid = truth[e];
      float sv[4];
      bool live[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = c0 + tx * 4 + j;
        live[j] = c < n && row0 + c != tid;
        float s = acc[i][j];
        if (d.cmp >= PBG_CMP_L2) {
          float qv = (a.yn[side][c < n ? c : 0] - 2.0f * s) + a.qn[side][e];       // model.py:226-246
          s = d.cmp == PBG_CMP_L2 ? -sqrtf(fmaxf(qv, 1e-30f)) : -qv;
        }
        sv[j] = s;
        if (live[j]) {
          cnt += s >= pos;
          if (d.loss == PBG_LOSS_RANKING) pa += fmaxf(0.f, (s - pos) + d.margin);
          else if (d.loss == PBG_LOSS_LOGISTIC) pa += fmaxf(s, 0.f) + log1pf(expf(-fabsf(s)));
          else pb = fmaxf(pb, s);
        }
      }
      if (d.loss == PBG_LOSS_SOFTMAX && pb > -INFINITY)
#pragma unroll
        for (int j = 0; j < 4; ++j) if (live[j]) pa += expf(sv[j] - pb);
    }
    scnt[tx][ty * 4 + i] = cnt; sa[tx][ty * 4 + i] = pa; sb[tx][ty * 4 + i] = pb;
  }
  __syncthreads();
  if (t < AN_TILE) {
    const int e = e0 + t;
    if (e < a.B) {
      int cnt = 0;
      float pa = 0.f, pb = d.loss == PBG_LOSS_SOFTMAX ? -INFINITY : 0.f;
      for (int x = 0; x < 16; ++x) {                       // the 16 column groups in a fixed order
        cnt += scnt[x][t];
        if (d.loss == PBG_LOSS_SOFTMAX) {
          float m2 = sb[x][t];
          if (m2 > -INFINITY) {
            float m = fmaxf(pb, m2);
            pa = (pb > -INFINITY ? pa * expf(pb - m) : 0.f) + sa[x][t] * expf(m2 - m);
            pb = m;
          }
        } else pa += sa[x][t];
      }
      size_t o = (size_t)tc * a.B + e;
      a.pcnt[side][o] = cnt; a.pa[side][o] = pa; a.pb[side][o] = pb;
    }
  }
}

// One warp per (side, edge).  The partials of the slab's tiles are folded across the lanes and into the running state;
// with the last slab every warp turns its state into rank and loss, the CTA's eight are summed, and the last CTA to
// finish adds up the CTAs' sums in CTA order.
// out8: loss, pos_rank, mrr, r1, r10, r50 sums over both sides' ranks, AUC hits per side.
__global__ void __launch_bounds__(32 * GATHER_WARPS) allnegs_merge_kernel(WaveDims d, WaveBufs w, AllNegs a, long long row0, int first, int last, float wrel, double *out8) {
  pdl_begin();
  __shared__ double sm[GATHER_WARPS][8];
  __shared__ bool closing;
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int item = blockIdx.x * GATHER_WARPS + wl;
  const int side = item >= a.B ? 1 : 0, e = item - side * a.B;
  const bool live = item < 2 * a.B && d.neg_enabled[side];
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (live) {
    const int n = allnegs_rows_of(d, a, side, row0);
    const int per = a.slab / a.tiles, ntiles = (n + per - 1) / per;       // candidates per partial; partials that hold any
    int cnt = 0;
    float ra = 0.f, rb = -INFINITY;
    for (int t0 = lane; t0 < ntiles; t0 += 128) {                          // four partials in flight
      int pc[4];
      float fa[4], fb[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const size_t o = (size_t)(t0 + 32 * u) * a.B + e;
        const bool on = t0 + 32 * u < ntiles;
        pc[u] = on ? a.pcnt[side][o] : 0;
        fa[u] = on ? a.pa[side][o] : 0.f;
        fb[u] = on && d.loss == PBG_LOSS_SOFTMAX ? a.pb[side][o] : -INFINITY;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        cnt += pc[u];
        if (d.loss == PBG_LOSS_SOFTMAX) {
          const float m2 = fb[u], m = fmaxf(rb, m2);
          if (m2 > -INFINITY) { ra = (rb > -INFINITY ? ra * expf(rb - m) : 0.f) + fa[u] * expf(m2 - m); rb = m; }
        } else ra += fa[u];
      }
    }
    cnt = warp_sum_int(cnt);
    if (d.loss == PBG_LOSS_SOFTMAX) {
      const float m = warp_max(rb);
      ra = warp_sum(rb > -INFINITY ? ra * expf(rb - m) : 0.f);
      rb = m;
    } else ra = warp_sum(ra);
    if (lane == 0) {
      if (!first) {
        cnt += a.cnt[side][e];
        if (d.loss == PBG_LOSS_SOFTMAX) {
          const float pb = a.rb[side][e], m = fmaxf(rb, pb);
          if (m > -INFINITY) ra = (pb > -INFINITY ? a.ra[side][e] * expf(pb - m) : 0.f) + (rb > -INFINITY ? ra * expf(rb - m) : 0.f);
          rb = m;
        } else ra += a.ra[side][e];
      }
      if (!last) { a.cnt[side][e] = cnt; a.ra[side][e] = ra; a.rb[side][e] = rb; }
      else {
        const float wgt = wrel * (w.ew ? w.ew[e] : 1.0f), pos = a.pos[side][e];
        float lossv;
        if (d.loss == PBG_LOSS_RANKING) lossv = ra;
        else if (d.loss == PBG_LOSS_LOGISTIC) lossv = ra / (float)d.n_rows[side] + (fmaxf(-pos, 0.f) + log1pf(expf(-fabsf(pos))));   // M counts the ignored column
        else {
          const float m = fmaxf(rb, pos);
          lossv = -pos + m + logf((rb > -INFINITY ? ra * expf(rb - m) : 0.f) + expf(pos - m));
        }
        const int rk = cnt + 1;
        v[0] = (double)(wgt * lossv); v[1] = rk; v[2] = 1.0 / rk; v[3] = rk <= 1; v[4] = rk <= 10; v[5] = rk <= 50;
        v[6 + side] = a.auc[side][e];
      }
    }
  }
  if (!last) return;
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < 8; ++k) sm[wl][k] = v[k];
  __syncthreads();
  if (threadIdx.x < 8) {
    double s = 0.0;
    for (int u = 0; u < GATHER_WARPS; ++u) s += sm[u][threadIdx.x];
    a.part[(size_t)blockIdx.x * 8 + threadIdx.x] = s;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) closing = atomicAdd(a.done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (closing) close_eval(a.part, gridDim.x, a.done, out8);
}

// scratch of the evaluation; `slab`: candidates per side prepared at a time
static void allnegs_layout(AllNegs &a, char *mem, int maxB, int Dp, int Dpb, int slab, bool planes, size_t &bytes) {
  size_t off = 0;
  auto take = [&](size_t n) { char *r = mem ? mem + off : nullptr; off += (n + 255) / 256 * 256; return r; };
  const int tiles = planes ? slab / 128 : slab / AN_TILE;
  const size_t ctas = (2 * (size_t)maxB + GATHER_WARPS - 1) / GATHER_WARPS;
  for (int s = 0; s < 2; ++s) {
    a.Q[s] = (float *)take((size_t)maxB * Dp * 4);
    a.qn[s] = (float *)take((size_t)maxB * 4); a.pos[s] = (float *)take((size_t)maxB * 4); a.auc[s] = (int *)take((size_t)maxB * 4);
    a.Y[s] = planes ? nullptr : (float *)take((size_t)slab * Dp * 4);
    a.yn[s] = (float *)take((size_t)slab * 4);
    a.pcnt[s] = (int *)take((size_t)tiles * maxB * 4); a.pa[s] = (float *)take((size_t)tiles * maxB * 4); a.pb[s] = (float *)take((size_t)tiles * maxB * 4);
    a.cnt[s] = (int *)take((size_t)maxB * 4); a.ra[s] = (float *)take((size_t)maxB * 4); a.rb[s] = (float *)take((size_t)maxB * 4);
  }
  a.QB = planes ? (unsigned short *)take(6 * (size_t)maxB * Dpb * 2) : nullptr;
  a.YB = planes ? (unsigned short *)take(6 * (size_t)slab * Dpb * 2) : nullptr;
  a.part = (double *)take(ctas * 8 * 8);
  a.slab = slab; a.qrows = maxB; a.Dpb = Dpb; a.tiles = tiles;
  bytes = off;
}

// Slabs of 8192 candidates, or with planes as many as keep both sides inside about 96 MB (they are read from L2): a
// slab's launches have a last round of tiles that leaves SMs idle, so fewer and larger ones are better; never more than
// the largest table has.
size_t pbg_allnegs_bytes(int maxB, int D, bool planes, long long table_rows, int &slab) {
  const int Dp = (D + 31) / 32 * 32, Dpb = (D + 7) / 8 * 8;
  long long rows = 8192;
  if (planes) {
    rows = 96ll * 1024 * 1024 / (12ll * Dpb);
    if (rows < 8192) rows = 8192;
    if (rows > 65536) rows = 65536;
  }
  if (rows > table_rows) rows = table_rows;
  slab = (int)((rows + 255) / 256 * 256);
  AllNegs a;
  size_t bytes;
  allnegs_layout(a, nullptr, maxB, Dp, Dpb, slab, planes, bytes);
  return bytes;
}

// Runs the whole evaluation of one batch against all rows of both tables; `mem` holds pbg_allnegs_bytes bytes.
int launch_allnegs_eval(const WaveDims &d, const WaveBufs &w, char *mem, int maxB, int B, int slab, bool planes, int rel_std, float wrel,
                        unsigned *done, unsigned *seam, double *out8, cudaStream_t st) {
  AllNegs a;
  size_t bytes;
  allnegs_layout(a, mem, maxB, d.Dp, (d.D + 7) / 8 * 8, slab, planes, bytes);
  a.B = B; a.done = done; a.seam = nullptr;
  int launches = 0;
  const int vec = (d.D + 127) / 128;
  const int ectas = (B + GATHER_WARPS - 1) / GATHER_WARPS;
#define AN_V(K, ...) do { if (vec <= 1) pbg_launch(K<1>, __VA_ARGS__); else if (vec <= 2) pbg_launch(K<2>, __VA_ARGS__); else if (vec <= 4) pbg_launch(K<4>, __VA_ARGS__); \
                            else if (vec <= 8) pbg_launch(K<8>, __VA_ARGS__); else pbg_launch(K<16>, __VA_ARGS__); } while (0)
  long long most = 0;
  for (int s = 0; s < 2; ++s) if (d.neg_enabled[s] && d.n_rows[s] > most) most = d.n_rows[s];
  if (most > 0) a.seam = seam;                                // (with no candidates there is no second sibling to clear it)
  AN_V(allnegs_rows_kernel, ectas, 32 * GATHER_WARPS, 0, st, d, w, a, rel_std);
  ++launches;
  for (long long row0 = 0; row0 == 0 || row0 < most; row0 += slab) {
    const int n = (int)(most - row0 < slab ? most - row0 : slab);
    const int sctas = (n + GATHER_WARPS - 1) / GATHER_WARPS, first = row0 == 0, last = row0 + slab >= most;
    if (n > 0) {                                              // (neither side has negatives: no candidates, and zeros from the merge)
      AN_V(allnegs_slab_kernel, dim3(sctas + (first ? ectas : 0), 2), 32 * GATHER_WARPS, 0, st, d, w, a, row0, rel_std, sctas, first ? ectas : 0);
      if (planes) launch_allnegs_score_tc(d, w, a, row0, st);
      else pbg_launch(allnegs_score_kernel, dim3((B + AN_TILE - 1) / AN_TILE, (n + AN_TILE - 1) / AN_TILE, 2), 256, 0, st, d, w, a, row0);
      launches += 2;
    }
    pbg_launch(allnegs_merge_kernel, (2 * B + GATHER_WARPS - 1) / GATHER_WARPS, 32 * GATHER_WARPS, 0, st, d, w, a, row0, first, last, wrel, out8);
    ++launches;
  }
#undef AN_V
  pbg_note_launch();
  return launches;
}
