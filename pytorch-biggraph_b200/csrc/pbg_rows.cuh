// What one warp does to one row in the passes of a wave -- gather, loss, pull-back -- as functions: the kernels of
// pbg_gather.cu, pbg_loss.cu and pbg_update.cu run one pass each over every row of a wave, chunk_kernel (pbg_chunk.cu)
// runs them one after the other over the rows of one chunk block.
#pragma once
#include "pbg_common.cuh"

// ---- gather ----------------------------------------------------------------------------------------
template <int VEC>
__device__ __forceinline__ void load_row(float4 (&v)[VEC], const float *row, int D, int lane) {
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    int d = c * 128 + lane * 4;
    v[c] = d < D ? ld4(row + d) : f4zero();
  }
}
// F.embedding(max_norm=...) (torchbiggraph/model.py:57-61): a looked-up row whose 2-norm exceeds
// max_norm is used scaled by max_norm / (norm + 1e-7).  Here the scale is applied in registers and
// returned; the table itself is rewritten by the update kernel, which owns each touched row alone
// (RowState::load applies the same scale before the optimizer steps) -- rewriting it from the gather
// would let the duplicates of a row read it half-scaled.
template <int VEC>
__device__ __forceinline__ float renorm_row(float4 (&v)[VEC], float max_norm) {
  if (max_norm <= 0.f) return 1.0f;
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < VEC; ++c) ss += f4dot(v[c], v[c]);
  float norm = sqrtf(warp_sum(ss));
  if (!(norm > max_norm)) return 1.0f;
  float sc = max_norm / (norm + 1e-7f);
#pragma unroll
  for (int c = 0; c < VEC; ++c) v[c] = v[c] * sc;
  return sc;
}
// row += the global embedding of the row's entity type (config.global_emb; model.py:486-492), if any
template <int VEC>
__device__ __forceinline__ void add_global(float4 (&v)[VEC], const float *glob, int D, int lane) {
  if (!glob) return;
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    int d = c * 128 + lane * 4;
    if (d < D) v[c] = v[c] + ld4(glob + d);
  }
}
template <int VEC>
__device__ __forceinline__ void store_row(float *row, const float4 (&v)[VEC], int D, int lane) {
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    int d = c * 128 + lane * 4;
    if (d < D) st4(row + d, v[c]);
  }
}
template <int VEC>
__device__ __forceinline__ void put_row(float *base, size_t off, const float4 (&v)[VEC], int D, int lane) {
  store_row<VEC>(base + off, v, D, lane);
}
// bf16-plane tier: the three planes of operand row r of block blk in array a
template <int VEC>
__device__ __forceinline__ void put_row_planes(const WaveBufs &w, int a, int blk, int r, const float4 (&v)[VEC], int D, int lane) {
  const size_t plane = (size_t)w.xrows[a] * w.Dpb;
  unsigned short *x = w.XB[a] + ((size_t)blk * w.npl * w.xrows[a] + r) * w.Dpb;
  const bool three = w.npl > 2;
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    int dd = c * 128 + lane * 4;
    if (dd < D) {
      uint2 p0, p1, p2;
      bf16_planes4(v[c], p0, p1, p2);
      *(uint2 *)(x + dd) = p0; *(uint2 *)(x + plane + dd) = p1;
      if (three) *(uint2 *)(x + 2 * plane + dd) = p2;
    }
  }
}
template <int VEC>
__device__ __forceinline__ void zero_row_planes(const WaveBufs &w, int a, int blk, int r, int D, int lane) {
  const size_t plane = (size_t)w.xrows[a] * w.Dpb;
  unsigned short *x = w.XB[a] + ((size_t)blk * w.npl * w.xrows[a] + r) * w.Dpb;
  const bool three = w.npl > 2;
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    int dd = c * 128 + lane * 4;
    if (dd < D) {
      *(uint2 *)(x + dd) = make_uint2(0, 0); *(uint2 *)(x + plane + dd) = make_uint2(0, 0);
      if (three) *(uint2 *)(x + 2 * plane + dd) = make_uint2(0, 0);
    }
  }
}
template <int VEC>
__device__ __forceinline__ void zero_row(float *row, int D, int lane) {
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    int d = c * 128 + lane * 4;
    if (d < D) st4(row + d, f4zero());
  }
}

// z = op(x; theta).  complex_diagonal pairs element d with d +- D/2, which lives in another
// lane: the partner chunk is re-read from memory (an L1 hit).
template <int VEC>
__device__ __forceinline__ void apply_operator(float4 (&z)[VEC], const float4 (&x)[VEC], const float *xrow,
                                               const float *theta, int op, int D, int lane, const float *glob = nullptr, float rsc = 1.0f) {
  int h = D >> 1;
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    int d = c * 128 + lane * 4;
    if (d >= D) { z[c] = f4zero(); continue; }
    if (op == PBG_OP_NONE || theta == nullptr) { z[c] = x[c]; continue; }
    float4 t = ld4(theta + d);
    if (op == PBG_OP_DIAGONAL) z[c] = x[c] * t;
    else if (op == PBG_OP_TRANSLATION) z[c] = x[c] + t;
    else {  // complex_diagonal: theta = [real | imag]
      int dp = d < h ? d + h : d - h;
      float4 xp = ld4(xrow + dp) * rsc, tp = ld4(theta + dp);
      if (glob) xp = xp + ld4(glob + dp);
      z[c] = d < h ? x[c] * t - xp * tp      // re = a_re p_re - a_im p_im
                   : xp * t + x[c] * tp;     // im = a_re p_im + a_im p_re
    }
  }
}

// comparator.prepare in place; returns the per-row auxiliary value kept for the later kernels
// (cos: 1/|z|, l2 family: |y|^2, dot: 0).
template <int VEC>
__device__ __forceinline__ float prepare_row(float4 (&z)[VEC], int cmp) {
  if (cmp == PBG_CMP_DOT) return 0.f;
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < VEC; ++c) ss += f4dot(z[c], z[c]);
  ss = warp_sum(ss);
  if (cmp != PBG_CMP_COS) return ss;
  float inv = 1.0f / sqrtf(ss);          // no epsilon: a zero row gives inf/NaN as in model.py:191-192
#pragma unroll
  for (int c = 0; c < VEC; ++c) z[c] = z[c] * inv;
  return inv;
}

template <int VEC>
__device__ __forceinline__ float positive_score(const float4 (&a)[VEC], const float4 (&b)[VEC], int cmp) {
  float s = 0.f;
  if (cmp == PBG_CMP_DOT || cmp == PBG_CMP_COS) {
#pragma unroll
    for (int c = 0; c < VEC; ++c) s += f4dot(a[c], b[c]);
    return warp_sum(s);
  }
#pragma unroll
  for (int c = 0; c < VEC; ++c) { float4 df = a[c] - b[c]; s += f4dot(df, df); }
  s = warp_sum(s);
  return cmp == PBG_CMP_L2 ? -sqrtf(fmaxf(s, 1e-30f)) : -s;
}

// One slot of a chunk block -- an edge's two rows, or the two uniform negatives of a column -- from the tables to the operand
// arrays, by one warp.
template <int VEC, bool PL>
__device__ __forceinline__ void gather_slot(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, int blk, int r, int lane) {
  BlockInfo bi = block_info(d, wb, blk);
  const int D = d.D;
  size_t nrow = (size_t)blk * d.Mm + r;
  const size_t noff = nrow * d.Dp;
  float *n0 = w.X[ARR_N0] + noff, *n1 = w.X[ARR_N1] + noff;
  float4 x[VEC], z[VEC], y0[VEC], y1[VEC];

  if (r < d.Pm) {                                           // ---- an edge of the chunk ----------
    size_t qrow = (size_t)blk * d.Pm + r;
    const size_t qoff = qrow * d.Dp;
    float *q0 = d.dynamic ? w.X[ARR_Q0] + qoff : nullptr;
    float *q1 = d.dynamic ? w.X[ARR_Q1] + qoff : nullptr;
    long long il = -1, ir = -1, rl = d.dynamic ? 0 : wb.rel[bi.b];
    bool ok = r < bi.n;
    if (ok) {
      il = w.lhs[bi.e0 + r];
      ir = w.rhs[bi.e0 + r];
      if (d.dynamic && d.op != PBG_OP_NONE) rl = w.rel[bi.e0 + r];
      if (il < 0 || il >= d.n_rows[0] || ir < 0 || ir >= d.n_rows[1] ||
          (d.op != PBG_OP_NONE && (rl < 0 || rl >= d.num_rels))) {
        if (lane == 0) atomicOr(w.errflag, 1);
        ok = false;
      }
    }
    if (!ok) {                                              // padding row: exact zeros
      zero_row<VEC>(n0, D, lane);
      zero_row<VEC>(n1, D, lane);
      if (d.matrix_op) zero_row<VEC>(w.R1 + noff, D, lane);
      if (d.dynamic) { zero_row<VEC>(q0, D, lane); zero_row<VEC>(q1, D, lane); }
      if (PL) {
        zero_row_planes<VEC>(w, ARR_N0, blk, r, D, lane); zero_row_planes<VEC>(w, ARR_N1, blk, r, D, lane);
        if (d.dynamic) { zero_row_planes<VEC>(w, ARR_Q0, blk, r, D, lane); zero_row_planes<VEC>(w, ARR_Q1, blk, r, D, lane); }
      }
      if (lane == 0) {
        w.aux[ARR_N0][nrow] = 0.f; w.aux[ARR_N1][nrow] = 0.f;
        if (d.dynamic) { w.aux[ARR_Q0][qrow] = 0.f; w.aux[ARR_Q1][qrow] = 0.f; }
        w.spos[0][qrow] = 0.f; w.spos[1][qrow] = 0.f;
      }
      return;
    }
    const float *xl = w.W[0] + (size_t)il * D, *xr = w.W[1] + (size_t)ir * D;
    const float *th0 = (d.op != PBG_OP_NONE && w.theta[0]) ? w.theta[0] + (size_t)rl * D : nullptr;
    // Up to 256 floats the rhs row is requested with the lhs row, before anything is written (behind the writes of the lhs
    // row it waited for them); wider rows leave no registers for it.
    constexpr bool EARLY = VEC <= 2;
    float4 xe[EARLY ? VEC : 1];
    if constexpr (EARLY) load_row<VEC>(xe, xr, D, lane);
    auto rhs_row = [&] {
      if constexpr (EARLY) {
#pragma unroll
        for (int c = 0; c < VEC; ++c) x[c] = xe[c];
      } else load_row<VEC>(x, xr, D, lane);
    };
    // lhs row without operator -> N0
    load_row<VEC>(x, xl, D, lane);
    const float scl = renorm_row<VEC>(x, d.max_norm);
    add_global<VEC>(x, w.glob[0], D, lane);
#pragma unroll
    for (int c = 0; c < VEC; ++c) y0[c] = x[c];
    float a0 = prepare_row<VEC>(y0, d.cmp);
    put_row<VEC>(w.X[ARR_N0], noff, y0, D, lane);
    if (PL) put_row_planes<VEC>(w, ARR_N0, blk, r, y0, D, lane);
    if (d.matrix_op) {
      // linear / affine: the raw rhs row goes to R1; operator, prepare and the positive score
      // follow in the contraction and postop_kernel
      rhs_row();
      renorm_row<VEC>(x, d.max_norm);
      add_global<VEC>(x, w.glob[1], D, lane);
      store_row<VEC>(w.R1 + noff, x, D, lane);
      if (lane == 0) w.aux[ARR_N0][nrow] = a0;
    } else if (!d.dynamic) {
      // rhs row through the operator -> N1; one positive score shared by both problems
      rhs_row();
      const float scr = renorm_row<VEC>(x, d.max_norm);
      if (d.max_norm > 0.f && lane == 0) w.rscale[nrow] = scr;
      add_global<VEC>(x, w.glob[1], D, lane);
      apply_operator<VEC>(y1, x, xr, th0, d.op, D, lane, w.glob[1], scr);
      float a1 = prepare_row<VEC>(y1, d.cmp);
      put_row<VEC>(w.X[ARR_N1], noff, y1, D, lane);
      if (PL) put_row_planes<VEC>(w, ARR_N1, blk, r, y1, D, lane);
      float s = positive_score<VEC>(y0, y1, d.cmp);
      if (lane == 0) {
        w.aux[ARR_N0][nrow] = a0; w.aux[ARR_N1][nrow] = a1;
        w.spos[0][qrow] = s; w.spos[1][qrow] = s;
      }
    } else {
      const float *th1 = (d.op != PBG_OP_NONE && w.theta[1]) ? w.theta[1] + (size_t)rl * D : nullptr;
      // op_lhs(lhs row) -> Q1 (x still holds the lhs row)
      apply_operator<VEC>(z, x, xl, th1, d.op, D, lane, nullptr, scl);
      float aq1 = prepare_row<VEC>(z, d.cmp);
      put_row<VEC>(w.X[ARR_Q1], qoff, z, D, lane);
      if (PL) put_row_planes<VEC>(w, ARR_Q1, blk, r, z, D, lane);
      // rhs row without operator -> N1
      rhs_row();
      const float scr = renorm_row<VEC>(x, d.max_norm);
#pragma unroll
      for (int c = 0; c < VEC; ++c) y1[c] = x[c];
      float a1 = prepare_row<VEC>(y1, d.cmp);
      put_row<VEC>(w.X[ARR_N1], noff, y1, D, lane);
      if (PL) put_row_planes<VEC>(w, ARR_N1, blk, r, y1, D, lane);
      float s1 = positive_score<VEC>(y1, z, d.cmp);         // problem 1: c(rhs, op_lhs(lhs))
      // op_rhs(rhs row) -> Q0
      apply_operator<VEC>(z, x, xr, th0, d.op, D, lane, nullptr, scr);
      float aq0 = prepare_row<VEC>(z, d.cmp);
      put_row<VEC>(w.X[ARR_Q0], qoff, z, D, lane);
      if (PL) put_row_planes<VEC>(w, ARR_Q0, blk, r, z, D, lane);
      float s0 = positive_score<VEC>(y0, z, d.cmp);         // problem 0: c(lhs, op_rhs(rhs))
      if (lane == 0) {
        w.aux[ARR_N0][nrow] = a0; w.aux[ARR_N1][nrow] = a1;
        w.aux[ARR_Q0][qrow] = aq0; w.aux[ARR_Q1][qrow] = aq1;
        w.spos[0][qrow] = s0; w.spos[1][qrow] = s1;
      }
    }
    return;
  }
  // ---- a uniformly drawn negative row, one per side ------------------------------------------
  // (both rows are requested before the first is written, as above)
  constexpr bool BOTH = VEC <= 2;
  const long long ids[2] = {slot_row(d, wb, w, bi, 0, r), slot_row(d, wb, w, bi, 1, r)};
  float4 xb[BOTH ? VEC : 1];
  if constexpr (BOTH)
    if (ids[1] >= 0 && ids[1] < d.n_rows[1]) load_row<VEC>(xb, w.W[1] + (size_t)ids[1] * D, D, lane);
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    float *dst = side == 0 ? n0 : n1;
    long long id = ids[side];
    if (id >= d.n_rows[side]) { if (lane == 0) atomicOr(w.errflag, 1); id = -1; }
    if (id < 0) {
      zero_row<VEC>(dst, D, lane);
      if (PL) zero_row_planes<VEC>(w, side, blk, r, D, lane);
      if (side == 1 && d.matrix_op) zero_row<VEC>(w.R1 + noff, D, lane);
      if (lane == 0) w.aux[side][nrow] = 0.f;
      continue;
    }
    const float *xrow = w.W[side] + (size_t)id * D;
    if (BOTH && side == 1) {
#pragma unroll
      for (int c = 0; c < VEC; ++c) x[c] = xb[BOTH ? c : 0];
    } else load_row<VEC>(x, xrow, D, lane);
    const float scu = renorm_row<VEC>(x, d.max_norm);
    if (side == 1 && d.max_norm > 0.f && lane == 0) w.rscale[nrow] = scu;
    add_global<VEC>(x, w.glob[side], D, lane);
    if (side == 1 && d.matrix_op) { store_row<VEC>(w.R1 + noff, x, D, lane); continue; }
    const float *th = nullptr;
    if (side == 1 && !d.dynamic && d.op != PBG_OP_NONE && w.theta[0]) {
      int rl = wb.rel[bi.b];
      if (rl >= 0 && rl < d.num_rels) th = w.theta[0] + (size_t)rl * D;
    }
    apply_operator<VEC>(z, x, xrow, th, d.op, D, lane, w.glob[side], scu);
    float a = prepare_row<VEC>(z, d.cmp);
    put_row<VEC>(w.X[side], noff, z, D, lane);
    if (PL) put_row_planes<VEC>(w, side, blk, r, z, D, lane);
    if (lane == 0) w.aux[side][nrow] = a;
  }
}

// ---- loss ------------------------------------------------------------------------------------------
__device__ __forceinline__ float softplusf(float x) {           // log(1 + e^x), stable
  return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x)));
}
__device__ __forceinline__ float sigmoidf(float x) { return 1.0f / (1.0f + expf(-x)); }

// column j of the negatives of a chunk: is it ignored, and does it exist at all?
__device__ __forceinline__ bool col_masked(const WaveDims &d, const BlockInfo &bi, int enabled, int i, int j) {
  if (!enabled) return true;
  if (j >= d.Pm) return false;                       // uniform negatives are never masked
  if (!d.batch_negs) return true;                    // uniform-only mode: no batch negatives
  return j == i || j >= bi.n;                        // own positive; padding of the last chunk
}

__device__ __forceinline__ float coef_from_dscore(int cmp, float dS, float S) {
  if (cmp == PBG_CMP_L2) return (-S > 1e-15f) ? -dS / S : 0.f;   // clamp at 1e-30 kills the gradient
  if (cmp == PBG_CMP_SQUARED_L2) return 2.0f * dS;
  return dS;
}

// NV > 0: the row (at most 32 NV columns) is read into registers before the first coefficient is written.  Written column
// by column behind the reads, every read waited for the write before it (the compiler cannot tell the rows apart): 24 to
// 31 us for 2 x 70 blocks of 100 rows x 200 columns where the bytes take 4.  NV == 0: rows of any length, column by column.
// The row's scores are where the coefficients go to, or (FROM) somewhere else.
template <int NV, bool FROM = false>
__device__ __forceinline__ void loss_row(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, int p, int blk, int i, int lane, const float *from = nullptr) {
  BlockInfo bi = block_info(d, wb, blk);
  if (bi.n == 0) return;
  float *S = w.S[p] + ((size_t)blk * d.Pm + i) * d.Ms;
  const float *Sr = FROM ? from : S;
  // bf16-plane tier with dynamic relations: T is an MMA operand, its planes go beside it
  unsigned short *TBr = w.TB[p] ? w.TB[p] + ((size_t)blk * w.npl * d.Pm + i) * w.Kb : nullptr;
  const size_t tplane = (size_t)d.Pm * w.Kb;
  auto put = [&](int j, float t) {
    S[j] = t;
    if (TBr) put_planes1(TBr + j, tplane, t, w.npl);
  };
  size_t prow = (size_t)blk * d.Pm + i;
  const int Mm = d.Mm;
  if (i >= bi.n) {                                   // padded positive: contributes nothing
    for (int j = lane; j < d.Ms; j += 32) put(j, 0.f);
    if (lane == 0) {
      w.lossrow[p][prow] = 0.f; w.violrow[p][prow] = 0;
      if (d.cmp >= PBG_CMP_L2) w.coef[2 + p][prow] = 0.f;
    }
    return;
  }
  const int enabled = d.neg_enabled[p];
  const float s = w.spos[p][prow];
  const float wr = wb.wrel[bi.b] * (w.ew ? w.ew[bi.e0 + i] : 1.0f);   // relation weight x edge weight
  // number of negative columns the reference's score matrix has for this row (masked included)
  const int Mlog = !enabled ? 0 : (d.batch_negs ? bi.Pl + d.U : d.U);
  float lossv = 0.f, ds = 0.f, rowsum = 0.f;
  int viol = 0;
  constexpr int NR = NV > 0 ? NV : 1;
  float sv[NR];
  unsigned live = 0u;                                 // bit u: column lane + 32 u counts
  if (NV > 0) {
#pragma unroll
    for (int u = 0; u < NR; ++u) {
      const int j = lane + 32 * u;
      const bool c = j < Mm && !col_masked(d, bi, enabled, i, j);
      sv[u] = c ? Sr[j] : 0.f;
      live |= c ? 1u << u : 0u;
    }
  }
  // every live column j with its score, in the order j = lane, lane + 32, ...
  auto each = [&](auto &&f) {
    if (NV > 0) {
#pragma unroll
      for (int u = 0; u < NR; ++u) if (live >> u & 1u) f(lane + 32 * u, sv[u]);
    } else {
      for (int j = lane; j < Mm; j += 32) if (!col_masked(d, bi, enabled, i, j)) f(j, Sr[j]);
    }
  };
  // writes the row: f(score) in the live columns, zeros elsewhere (the diagonal is filled below)
  auto fill = [&](auto &&f) {
    if (NV > 0) {
#pragma unroll
      for (int u = 0; u < NR; ++u) {
        const int j = lane + 32 * u;
        const float t = live >> u & 1u ? f(sv[u]) : 0.f;
        rowsum += t;
        if (j < d.Ms) put(j, t);
      }
    } else {
      for (int j = lane; j < d.Ms; j += 32) {
        const float t = j < Mm && !col_masked(d, bi, enabled, i, j) ? f(Sr[j]) : 0.f;
        rowsum += t;
        put(j, t);
      }
    }
  };

  if (d.loss == PBG_LOSS_SOFTMAX) {
    // -s + log(e^s + sum_j e^S_ij); masked entries are e^-1e9 = 0 (losses.py:143-159)
    if (Mlog > 0) {
      float mx = -INFINITY;
      each([&](int, float x) { mx = fmaxf(mx, x); });
      mx = warp_max(mx);
      float m = fmaxf(mx, s);
      if (mx == -INFINITY) m = fmaxf(s, PBG_MASKED);      // every column masked
      float z = 0.f;
      each([&](int, float x) { z += expf(x - m); viol += x > s; });
      z = warp_sum(z);
      float es = expf(s - m);
      float Z = z + es;
      lossv = -s + m + logf(Z);
      ds = es / Z - 1.0f;
      float invZ = 1.0f / Z;
      fill([&](float x) { return coef_from_dscore(d.cmp, wr * expf(x - m) * invZ, x); });
    } else {
      fill([&](float) { return 0.f; });                    // losses.py:139-140: loss 0, no gradient
    }
  } else if (d.loss == PBG_LOSS_RANKING) {
    // sum_j max(0, margin - s + S_ij) (losses.py:116-122)
    if (Mlog > 0) {
      each([&](int, float x) {
        const float v = (x - s) + d.margin;
        viol += x > s;
        if (v > 0.f) { lossv += v; ds -= 1.0f; }
      });
      fill([&](float x) { return (x - s) + d.margin > 0.f ? coef_from_dscore(d.cmp, wr, x) : 0.f; });
      lossv = warp_sum(lossv);
      ds = warp_sum(ds);
    } else {
      fill([&](float) { return 0.f; });
    }
  } else {
    // softplus(-s) + (1/M) sum_j softplus(S_ij), M counts masked columns (losses.py:61-80)
    float nw = Mlog > 0 ? 1.0f / (float)Mlog : 0.f;
    each([&](int, float x) { viol += x > s; lossv += softplusf(x); });
    fill([&](float x) { return coef_from_dscore(d.cmp, wr * nw * sigmoidf(x), x); });
    lossv = warp_sum(lossv) * nw + softplusf(-s);
    ds = -sigmoidf(-s);
  }
  viol = warp_sum_int(viol);
  rowsum = warp_sum(rowsum);
  // positive pair folded into the diagonal; the positive score of the l2 family is the direct
  // form -sqrt(max(sum (a-b)^2, 1e-30)) (model.py:267-274)
  float tdiag = coef_from_dscore(d.cmp, wr * ds, s);
  __syncwarp();
  if (lane == 0) {
    put(i, tdiag);
    w.lossrow[p][prow] = wr * lossv;
    w.violrow[p][prow] = viol;
    if (d.cmp >= PBG_CMP_L2) w.coef[2 + p][prow] = rowsum + tdiag;
  }
}

// Softmax under the dot / cos comparators with at most 32 NV negative columns: the warp keeps the
// row in registers, so the scores are read once, the masks evaluated once and every exponential
// taken once (the general kernel makes three passes).  Same arithmetic, same summation order.
template <int NV, bool FROM = false>
__device__ __forceinline__ void loss_softmax_row(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, int p, int blk, int i, int lane, const float *from = nullptr) {
  BlockInfo bi = block_info(d, wb, blk);
  if (bi.n == 0) return;
  float *S = w.S[p] + ((size_t)blk * d.Pm + i) * d.Ms;
  const float *Sr = FROM ? from : S;
  // bf16-plane tier with dynamic relations: T is an MMA operand, its planes go beside it
  unsigned short *TBr = w.TB[p] ? w.TB[p] + ((size_t)blk * w.npl * d.Pm + i) * w.Kb : nullptr;
  const size_t tplane = (size_t)d.Pm * w.Kb;
  const int npl = w.npl;
  size_t prow = (size_t)blk * d.Pm + i;
  const int Mm = d.Mm;
  const int enabled = d.neg_enabled[p];
  const int Mlog = !enabled ? 0 : (d.batch_negs ? bi.Pl + d.U : d.U);
  if (i >= bi.n || Mlog == 0) {                      // padded positive, or no negatives at all: no loss, no gradient
#pragma unroll
    for (int u = 0; u < NV; ++u) { int j = lane + 32 * u; if (j < d.Ms) S[j] = 0.f; }
    if (TBr)
      for (int j = 2 * lane; j < d.Ms; j += 64) { *(unsigned *)(TBr + j) = 0u; *(unsigned *)(TBr + tplane + j) = 0u; if (npl > 2) *(unsigned *)(TBr + 2 * tplane + j) = 0u; }
    if (lane == 0) { w.lossrow[p][prow] = 0.f; w.violrow[p][prow] = 0; }
    return;
  }
  const float s = w.spos[p][prow];
  const float wr = wb.wrel[bi.b] * (w.ew ? w.ew[bi.e0 + i] : 1.0f);   // relation weight x edge weight
  float sv[NV];
  float mx = -INFINITY;
#pragma unroll
  for (int u = 0; u < NV; ++u) {
    int j = lane + 32 * u;
    bool valid = j < Mm && !col_masked(d, bi, enabled, i, j);
    sv[u] = valid ? Sr[j] : -INFINITY;
    mx = fmaxf(mx, sv[u]);
  }
  mx = warp_max(mx);
  float m = fmaxf(mx, s);
  if (mx == -INFINITY) m = fmaxf(s, PBG_MASKED);      // every column masked
  float z = 0.f;
  int viol = 0;
#pragma unroll
  for (int u = 0; u < NV; ++u) {
    bool valid = sv[u] != -INFINITY;
    viol += valid && sv[u] > s;
    sv[u] = valid ? expf(sv[u] - m) : 0.f;
    z += sv[u];
  }
  z = warp_sum(z);
  viol = warp_sum_int(viol);
  float es = expf(s - m);
  float Z = z + es;
  float lossv = -s + m + logf(Z);
  float invZ = 1.0f / Z;
  float tdiag = wr * (es / Z - 1.0f);
#pragma unroll
  for (int u = 0; u < NV; ++u) {
    int j = lane + 32 * u;
    if (j < d.Ms) S[j] = j == i ? tdiag : wr * sv[u] * invZ;
  }
  if (TBr) {
    // two column groups at a time: neighbouring lanes swap one group's planes, so that every lane stores
    // two columns of one group (4-byte stores): even lanes (j, j + 1) of group u, odd lanes (j - 1, j) of u + 1
    const bool odd = lane & 1;
#pragma unroll
    for (int u = 0; u < NV; u += 2) {
      const int j0 = lane + 32 * u, j1 = j0 + 32;
      unsigned a[3], b[3], give[3], keep[3];
      bf16_planes(j0 == i ? tdiag : wr * sv[u] * invZ, a[0], a[1], a[2]);
      bf16_planes(j1 == i ? tdiag : wr * sv[u + 1] * invZ, b[0], b[1], b[2]);
#pragma unroll
      for (int q = 0; q < 3; ++q) { give[q] = odd ? a[q] : b[q]; keep[q] = odd ? b[q] : a[q]; }
      unsigned g01 = __shfl_xor_sync(0xffffffffu, give[0] | (give[1] << 16), 1);
      unsigned g2 = __shfl_xor_sync(0xffffffffu, give[2], 1);
      unsigned got[3] = {g01 & 0xffffu, g01 >> 16, g2};
      const int col = (odd ? j1 : j0) & ~1;
      if (col < d.Ms) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          unsigned lo = odd ? got[q] : keep[q], hi = odd ? keep[q] : got[q];
          if (q < npl) *(unsigned *)(TBr + q * tplane + col) = lo | (hi << 16);
        }
      }
    }
  }
  if (lane == 0) { w.lossrow[p][prow] = wr * lossv; w.violrow[p][prow] = viol; }
}

// ---- pull-back -------------------------------------------------------------------------------------
enum { CK_DOT = 0, CK_COS = 1, CK_L2 = 2 };      // comparator kinds of the pull-back

// v = gradient of the operator output behind slot (a, blk, r): the contraction's row, plus the regularizer's own
// gradient on the rows it covers (reg), back through comparator.prepare -- cos: (g - y <g, y>) / |z|; l2 family: the
// row's own |y|^2 term (dynamic: ga = T.N - rowsum(T) a, gb = T^T.Q - colsum(T) b; standard: g = A.N' - rowsum(A) y).
// yv: the operand row (y: where it lies); cf: what the l2 family takes of it; inv: 1 / |z| under cos.
template <int VEC, int CK>
__device__ __forceinline__ void gz_math(float4 (&v)[VEC], const float4 (&yv)[VEC], const float *y, float cf, float inv, const WaveDims &d, int lane, bool reg) {
  const int D = d.D;
  if (reg) {
#pragma unroll
    for (int c = 0; c < VEC; ++c) {
      const int dd = c * 128 + lane * 4;
      if (dd < D) v[c] = v[c] + n3_grad4(y, dd, D, d.op == PBG_OP_COMPLEX_DIAGONAL) * d.reg_coef;
    }
  }
  if (CK == CK_COS) {
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < VEC; ++c) s += f4dot_yx(v[c], yv[c]);
    s = warp_sum(s);
#pragma unroll
    for (int c = 0; c < VEC; ++c) v[c] = (v[c] - yv[c] * s) * inv;
  } else if (CK == CK_L2) {
#pragma unroll
    for (int c = 0; c < VEC; ++c) v[c] = v[c] - yv[c] * cf;
  }
}
template <int VEC, int CK>
__device__ __forceinline__ void gz_row(float4 (&v)[VEC], const WaveDims &d, const WaveBufs &w, int a, int blk, int r, int lane, bool reg) {
  const int D = d.D;
  const size_t xr = (size_t)blk * w.xrows[a] + r, gr = (size_t)blk * w.grows[a] + r;
  const float *y = w.X[a] + xr * d.Dp, *g = w.GX[a] + gr * d.Dp;
  float4 yv[VEC];
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    const int dd = c * 128 + lane * 4;
    v[c] = dd < D ? ld4(g + dd) : f4zero();
    yv[c] = CK != CK_DOT && dd < D ? ld4(y + dd) : f4zero();
  }
  gz_math<VEC, CK>(v, yv, y, CK == CK_L2 ? w.coef[a][gr] : 0.f, CK == CK_COS ? w.aux[a][xr] : 1.f, d, lane, reg);
}

// Back through the operator: v (gradient of its output) becomes the gradient of the raw row, pg the contribution to
// the operator row.  x: the raw row, used as x * xs (+ xadd).  complex_diagonal pairs element d with d +- D/2, which
// another lane holds: v goes through `part` (D floats of the warp's own shared memory), the partners of x and theta are
// read again (L1 / L2).
template <int VEC>
__device__ __forceinline__ void operator_back(float4 (&v)[VEC], float4 (&pg)[VEC], const WaveDims &d, const float *theta, const float *x,
                                              float xs, const float *xadd, float *part, int lane) {
  const int D = d.D;
  auto raw = [&](int e) {
    float4 q = ld4(x + e) * xs;
    if (xadd) q = q + ld4(xadd + e);
    return q;
  };
  if (d.op == PBG_OP_TRANSLATION) {
#pragma unroll
    for (int c = 0; c < VEC; ++c) pg[c] = v[c];
    return;
  }
  if (d.op == PBG_OP_DIAGONAL) {
#pragma unroll
    for (int c = 0; c < VEC; ++c) {
      const int dd = c * 128 + lane * 4;
      if (dd < D) { pg[c] = v[c] * raw(dd); v[c] = v[c] * ld4(theta + dd); }
    }
    return;
  }
  const int h = D >> 1;
  __syncwarp();                                              // the previous row's partners have been read
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    const int dd = c * 128 + lane * 4;
    if (dd < D) st4(part + dd, v[c]);
  }
  __syncwarp();
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    const int dd = c * 128 + lane * 4;
    if (dd < D) {
      const int dp = dd < h ? dd + h : dd - h;
      const float4 vp = ld4(part + dp), xv = raw(dd), xp = raw(dp), t = ld4(theta + dd), tp = ld4(theta + dp);
      // d real = g_re a_re + g_im a_im ;  d imag = -g_re a_im + g_im a_re
      pg[c] = dd < h ? v[c] * xv + vp * xp : v[c] * xp - vp * xv;
      // gx_re = g_re p_re + g_im p_im ;  gx_im = -g_re p_im + g_im p_re
      v[c] = dd < h ? v[c] * t + vp * tp : v[c] * tp - vp * t;
    }
  }
}

// Standard relations: what is left of the pull-back of a gradient slot (std_pullback_kernel) behind gz_row -- the operator, with
// the row's contribution to the operator row into PG, and out.  row: the slot's entity; part: D floats of the warp's own
// shared memory.
template <int VEC>
__device__ __forceinline__ void std_pullback_finish(float4 (&v)[VEC], const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, int side, const BlockInfo &bi, int blk, int r,
                                                    long long row, int lane, float *part) {
  const int a = side ? ARR_N1 : ARR_N0, D = d.D;
  if (side == 1 && w.PG) {
    float4 pg[VEC];
    const float xs = d.max_norm > 0.f ? w.rscale[(size_t)blk * d.Mm + r] : 1.0f;   // the raw row entered the operator scaled
    operator_back<VEC>(v, pg, d, w.theta[0] + (size_t)wb.rel[bi.b] * D, w.W[1] + (size_t)row * D, xs, w.glob[1], part, lane);
    store_row<VEC>(w.PG + ((size_t)blk * d.Mm + r) * d.Dp, pg, D, lane);
  }
  __syncwarp();
  store_row<VEC>(w.GX[a] + ((size_t)blk * w.grows[a] + r) * d.Dp, v, D, lane);
}
template <int VEC>
__device__ __forceinline__ void std_pullback_empty(const WaveDims &d, const WaveBufs &w, int side, int blk, int r, int lane) {   // no row behind the slot: nothing for param_sums to add
  const int a = side ? ARR_N1 : ARR_N0;
  zero_row<VEC>(w.GX[a] + ((size_t)blk * w.grows[a] + r) * d.Dp, d.D, lane);
  if (side == 1 && w.PG) zero_row<VEC>(w.PG + ((size_t)blk * d.Mm + r) * d.Dp, d.D, lane);
}

// Dynamic relations: the same for slot r of operand array a (dyn_pullback_kernel).  entity: the slot's is inside its table.
template <int VEC, int CK>
__device__ __forceinline__ void dyn_pullback_finish(float4 (&v)[VEC], const WaveDims &d, const WaveBufs &w, int a, const BlockInfo &bi, int blk, int r, int lane, float *part) {
  const int D = d.D;
  const bool q = a >= ARR_Q0;
  float *prow = q && w.GR[a - ARR_Q0] ? w.GR[a - ARR_Q0] + ((size_t)blk * d.Pm + r) * d.Dp : nullptr;
  const float *theta = nullptr;
  if (prow) {
    const long long rl = w.rel[bi.e0 + r];
    const float *tab = w.theta[a - ARR_Q0];
    if (tab && rl >= 0 && rl < d.num_rels) theta = tab + (size_t)rl * D;
  }
  if (theta) {
    float4 pg[VEC];
    const int na = a == ARR_Q0 ? ARR_N1 : ARR_N0;              // the slot's operator-free copy (prepared raw row)
    const size_t nrow = (size_t)blk * w.xrows[na] + r;
    const float xs = CK == CK_COS ? 1.0f / w.aux[na][nrow] : 1.0f;
    operator_back<VEC>(v, pg, d, theta, w.X[na] + nrow * d.Dp, xs, nullptr, part, lane);
#pragma unroll
    for (int c = 0; c < VEC; ++c) {
      const int dd = c * 128 + lane * 4;
      // N3 regularizer on the edge's own parameter row (still as the wave found it)
      if (dd < D && d.reg_coef != 0.f) pg[c] = pg[c] + n3_grad4(theta, dd, D, d.op == PBG_OP_COMPLEX_DIAGONAL) * d.reg_coef;
    }
    store_row<VEC>(prow, pg, D, lane);
  }
  __syncwarp();
  store_row<VEC>(w.GX[a] + ((size_t)blk * w.grows[a] + r) * d.Dp, v, D, lane);
}
// an entity id outside its table (the call reports it): the edge's operator-row slot may still be a valid one (its key depends
// on the relation id only), so it gets a zero gradient rather than whatever the row held
template <int VEC>
__device__ __forceinline__ void dyn_pullback_empty(const WaveDims &d, const WaveBufs &w, int a, int blk, int r, int lane) {
  if (a >= ARR_Q0 && w.GR[a - ARR_Q0]) zero_row<VEC>(w.GR[a - ARR_Q0] + ((size_t)blk * d.Pm + r) * d.Dp, d.D, lane);
}
// the table a slot's entity belongs to: N arrays hold lhs / rhs rows (chunk, then uniform), Q0 = op_rhs(rhs), Q1 = op_lhs(lhs)
__device__ __forceinline__ int slot_side(int a) { return a == ARR_N0 || a == ARR_Q1 ? 0 : 1; }
