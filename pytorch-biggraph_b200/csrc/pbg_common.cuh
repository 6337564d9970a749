// Shared declarations of the sm_100a training-step library: wave layout in HBM, decoding of
// row slots, and the small device helpers every kernel uses.
//
// Vocabulary (PyTorch-BigGraph's): a *bucket* is a (lhs partition, rhs partition) pair; a
// *batch* is batch_size edges; a batch is cut into *chunks* of P = num_batch_negs edges which
// serve as each other's negatives, plus U uniformly drawn negative rows per chunk
// (torchbiggraph/model.py:508-622).  A *wave* is the k batches this library keeps in flight.
//
// Layout of one wave in the workspace (all float32, row stride Dp = dim rounded up to 32):
//   block blk = b * Cm + c        (b-th batch of the wave, c-th chunk, Cm chunks per batch)
//   N0[blk][Mm][Dp]  prepared lhs rows: Pm chunk rows then U uniform rows   (Mm = Pm + U)
//   N1[blk][Mm][Dp]  prepared rhs rows: Pm chunk rows then U uniform rows
//   Q0[blk][Pm][Dp]  rows scored against N0 (the "lhs corrupted" problem 0)
//   Q1[blk][Pm][Dp]  rows scored against N1 (the "rhs corrupted" problem 1)
// Standard relations (operator on the rhs only): Q0 is the first Pm rows of N1 and Q1 the first
// Pm rows of N0 (aliases).  Dynamic relations: N0/N1 hold rows WITHOUT operator, Q0 holds
// op_rhs[rel](rhs rows), Q1 holds op_lhs[rel](lhs rows) (model.py:705-758).
//   S_p[blk][Pm][Ms]   scores of problem p, later overwritten by the coefficient matrix T_p
//   dynamic relations:  GN_p[blk][Mm][Dp] = T_p^T . Q_p      GQ_p[blk][Pm][Dp] = T_p . N_p
//   standard relations: GN0 = A[0] . N1,  GN1 = A[1] . N0  with the combined matrices A (WaveBufs)
// T_p holds d(loss)/d(score) with the gradient of the positive score folded into its (masked,
// otherwise unused) diagonal, so the two products above are the whole backward of the
// comparator.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <mutex>
#include <map>
#include <utility>
#include "../../include/pbg_b200.h"

#define PBG_KMAX 32                 // most batches in one wave
#define PBG_MASKED (-1e9f)          // torchbiggraph/model.py:836-839
#define PBG_ADAGRAD_EPS 1e-10f      // row_adagrad.py:94, async_adagrad.py:84

enum { ARR_N0 = 0, ARR_N1 = 1, ARR_Q0 = 2, ARR_Q1 = 3, ARR_R0 = 4, ARR_R1 = 5 };

// Division of slot and block numbers (below 2^31) by a size that is fixed for the launch: one high multiply and a shift
// instead of the twenty-odd instructions of an integer division (Granlund and Montgomery, division by invariant integers
// using multiplication).  With l = ceil(log2 d) and m = ceil(2^(31 + l) / d),
// n / d = floor(n m / 2^(31 + l)): m exceeds the exact quotient by less than 1, so the product exceeds n / d by less
// than n / 2^(31 + l) < 1 / d.  Kernels of a few hundred instructions per row of 100 floats spend a quarter of them on five
// such divisions.
struct FastDiv {
  unsigned m;
  int s;                // l - 1; -1: division by 1
  FastDiv() = default;
  explicit FastDiv(int d) {
    int l = 0;
    while ((1ll << l) < d) ++l;
    s = l - 1;
    m = l == 0 ? 0u : (unsigned)(((1ull << (31 + l)) + (unsigned)d - 1) / (unsigned)d);
  }
  __device__ __forceinline__ int div(int n) const { return s < 0 ? n : (int)(__umulhi((unsigned)n, m) >> s); }
};

struct WaveDims {
  int D, Dp;            // dim, workspace row stride (floats)
  int Pm, U, Mm, Ms;    // chunk slots, uniform negatives, Pm+U, score row stride
  int Cm;               // chunks per batch (max)
  FastDiv byMm, byPm, byCm, bySpb;
  int k, nblk;          // batches in this wave; chunk blocks THIS LAUNCH covers (k*Cm for a whole wave)
  int blk0;             // first chunk block of this launch (a wave may be launched in two parts)
  int op, cmp, loss, dynamic;
  int batch_negs;       // 1: batch_uniform mode, 0: uniform-only mode (num_batch_negs == 0)
  int neg_enabled[2];   // problem 0 = lhs negatives, problem 1 = rhs negatives
  int num_batch_negs;
  int spb;              // occurrence slots per batch (see occ_decode)
  int nocc;             // k * spb
  float margin;
  float reg_coef;       // N3 regularizer weight, 0 = off
  float max_norm;       // > 0: looked-up rows longer than this are used (and kept) scaled to it
  long long n_rows[2];  // rows of the lhs / rhs table
  int shared_table;     // lhs and rhs read the same table
  int num_rels;
  int matrix_op;        // operator is linear / affine (standard relations): applied by contractions, not in the gather
  int opw;              // floats per operator-table row: D, or D*D (+ D) for linear (affine)
  int pulled_back;      // the gradient slots have been through the pull-back already (chunk_kernel)
  unsigned long long key_rel_base;   // first sort key of operator-table rows
  unsigned long long key_invalid;    // sort key of slots that carry no gradient
};

struct WaveBatches {
  long long off[PBG_KMAX];    // first edge of the batch in the edge arrays
  long long gidx[PBG_KMAX];   // index of the batch in the call (uniform-id array, stats, RNG)
  int n[PBG_KMAX];            // edges in the batch
  int rel[PBG_KMAX];          // relation of the batch (standard mode)
  float wrel[PBG_KMAX];       // relation weight of the batch
};

struct WaveBufs {
  float *X[4];       int xrows[4];   // operand arrays N0,N1,Q0,Q1 (rows per block; aliases allowed)
  float *aux[4];                     // per operand row: cos -> 1/|z|, l2 -> |y|^2 (indexed like X)
  float *GX[4];      int grows[4];   // gradient arrays GN0,GN1,GQ0,GQ1
  float *GR[2];                      // dynamic relations with an operator: per edge the gradient of its operator row,
                                     // [0] rhs table (slots ARR_R0), [1] lhs table (ARR_R1), rows like GQ; null: not kept
  float *PG;                         // standard relations, diagonal / complex_diagonal: per N1 row its contribution to the operator row's gradient; else null
  float *S[2];                       // scores / coefficient matrices
  // Standard relations: combined coefficient matrices, one per side, [nblk][Mm][Ma]:
  //   A[0][m][j] = (j < Pm ? T0[j][m] : 0) + (m < Pm ? T1[m][j] : 0)   gradient of the lhs rows  = A[0] . N1
  //   A[1][m][j] = (j < Pm ? T1[j][m] : 0) + (m < Pm ? T0[m][j] : 0)   gradient of the rhs rows  = A[1] . N0
  float *A[2];
  int Ma;                            // row stride of A (Mm rounded up to 4)
  // bf16-plane tier: every fp32 operand value as three bf16 planes b0 + b1 + b2 (b0 = bf16(x), b1 =
  // bf16(x - b0), b2 = bf16(x - b0 - b1)); the contractions read these instead of X / A
  //   XB[a]     [nblk][3][xrows[a]][Dpb]   planes of the operand rows N0, N1, Q0, Q1 (aliased like X)
  //   AB[side]  [nblk][3][Mm][Kb]          planes of the merged coefficient matrices (standard relations)
  //   TB[p]     [nblk][3][Pm][Kb]          planes of the coefficient matrices T_p (dynamic relations)
  //                                          (also standard relations with the fused score / loss kernel; AB is then unused)
  unsigned short *XB[4], *AB[2], *TB[2];     // null outside that tier
  int Dpb, Kb;                       // row strides in elements (D and Mm rounded up to 8: 16-byte rows)
  int npl;                           // planes per value: 3 (bf16x6: all six products of order <= 2) or 2 (bf16x3: b0.b0 + b0.b1 + b1.b0)
  float *spos[2];                    // positive scores [nblk][Pm]
  float *coef[4];                    // l2: colsum(T0), colsum(T1), rowsum(T0), rowsum(T1)
  float *lossrow[2];                 // per positive row: weighted loss term
  float *rscale;                     // max_norm: scale applied to the raw row of every N1 slot [blk][Mm] (1 = none)
  float *regrow;                     // per positive row: its share of the N3 regularizer (reg_coef != 0)
  int *violrow[2];                   // per positive row: #(neg > pos)
  const long long *lhs, *rhs, *rel;  // edge arrays
  const float *ew;                  // per-edge weights parallel to the edge arrays, or null
  const long long *ul, *ur;          // uniform ids [batches][Cm][U] or null
  unsigned long long seed;
  float *W[2], *G[2];                // embedding tables / RowAdagrad state (lhs, rhs)
  float *theta[2], *acc[2];          // operator tables: [0] applied to rhs rows, [1] to lhs rows
  // linear / affine operators: R1 = raw rhs rows, R2 = A.x (forward) then g.A (backward), both laid
  // out like N1; dA = per-batch gradient of the operator row [k][opw]
  float *R1, *R2, *dA;
  float *relpart;                    // standard mode: [blk][D] partial operator gradients
  float *glob[2], *gacc[2];          // global embedding of the lhs / rhs entity type + AsyncAdagrad accumulator, or null
  int glob_shared;                   // both sides are of one entity type: glob[0] == glob[1], one step per batch
  float *globpart;                   // [side][blk][D] partial sums of the row gradients (global-embedding gradient)
  int *errflag;                      // device error word (bit 0: id out of range)
};

struct BlockInfo { int b, c, Pl, n; long long e0; };

// Which batch/chunk a block is, its logical chunk size Pl = min(num_batch_negs or U, batch
// edges) (model.py:648-656) and how many of its Pm slots hold real edges.
__device__ __forceinline__ BlockInfo block_info(const WaveDims &d, const WaveBatches &wb, int blk) {
  BlockInfo bi;
  bi.b = d.byCm.div(blk);
  bi.c = blk - bi.b * d.Cm;
  int nb = wb.n[bi.b];
  int lim = d.batch_negs ? d.num_batch_negs : d.U;
  bi.Pl = nb < lim ? nb : lim;
  int first = bi.c * bi.Pl;
  int n = nb - first;
  bi.n = bi.Pl > 0 ? (n < 0 ? 0 : (n > bi.Pl ? bi.Pl : n)) : 0;
  bi.e0 = wb.off[bi.b] + first;
  return bi;
}

// Counter-based generator for device-drawn uniform negatives (stands where the reference
// calls torch.randint, model.py:70-75): splitmix64 of (seed, batch, side, chunk, j).
__device__ __forceinline__ unsigned long long pbg_mix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ long long pbg_uniform_id(unsigned long long seed, long long gidx, int side,
                                                    int c, int j, long long nrows) {
  unsigned long long h = pbg_mix64(seed ^ pbg_mix64((unsigned long long)gidx * 2ull + (unsigned)side));
  h = pbg_mix64(h + ((unsigned long long)(unsigned)c << 32) + (unsigned)j);
  return (long long)__umul64hi(h, (unsigned long long)nrows);
}

// Table row behind slot r of block (b, c) on `side` (0 lhs, 1 rhs); -1 when the slot is empty.
__device__ __forceinline__ long long slot_row(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w,
                                              const BlockInfo &bi, int side, int r) {
  if (r < d.Pm) {
    if (r >= bi.n) return -1;
    return side == 0 ? w.lhs[bi.e0 + r] : w.rhs[bi.e0 + r];
  }
  if (bi.n == 0 || !d.neg_enabled[side]) return -1;
  int j = r - d.Pm;
  const long long *u = side == 0 ? w.ul : w.ur;
  if (u) return u[(wb.gidx[bi.b] * d.Cm + bi.c) * (long long)d.U + j];
  return pbg_uniform_id(w.seed, wb.gidx[bi.b], side, bi.c, j, d.n_rows[side]);
}

// Occurrence index o -> (batch b, array a, block, row).  Per batch the slots are enumerated
// [N0: Cm*Mm | N1: Cm*Mm | Q0: Cm*Pm | Q1: Cm*Pm | R0: Cm*Pm | R1: Cm*Pm]; the Q slots and R0/R1
// (operator-table rows touched through Q0/Q1) exist only with dynamic relations -- with standard
// relations a chunk row has ONE gradient slot, in GN0 / GN1.  Enumeration is batch-major so that
// a stable sort by row keeps a row's occurrences in batch order.
struct Occ { int b, a, blk, r; };
__device__ __forceinline__ Occ occ_decode(const WaveDims &d, int o) {
  Occ q;
  q.b = d.bySpb.div(o);
  int w = o - q.b * d.spb;
  int nN = d.Cm * d.Mm, nQ = d.dynamic ? d.Cm * d.Pm : 0;   // standard relations: N slots only
  bool whole = false;                                      // rows of Mm slots (N arrays) or of Pm
  if (w < nN) { q.a = ARR_N0; whole = true; }
  else if ((w -= nN) < nN) { q.a = ARR_N1; whole = true; }
  else if ((w -= nN) < nQ) q.a = ARR_Q0;
  else if ((w -= nQ) < nQ) q.a = ARR_Q1;
  else if ((w -= nQ) < nQ) q.a = ARR_R0;
  else { w -= nQ; q.a = ARR_R1; }
  int c = whole ? d.byMm.div(w) : d.byPm.div(w);
  q.r = w - c * (whole ? d.Mm : d.Pm);
  q.blk = q.b * d.Cm + c;
  return q;
}

// Sort key of occurrence slot o: the table row its gradient belongs to.
//   lhs-table rows            key = row
//   rhs-table rows            key = row (+ lhs rows when the tables differ)
//   operator-table rows       key = key_rel_base + table * num_rels + rel   (dynamic relations)
//   slots without gradient    key = key_invalid (sorts to the end)
__device__ __forceinline__ unsigned long long slot_key(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, int o) {
  Occ q = occ_decode(d, o);
  BlockInfo bi = block_info(d, wb, q.blk);
  unsigned long long key = d.key_invalid;
  unsigned long long rbase = d.shared_table ? 0ull : (unsigned long long)d.n_rows[0];
  if (q.a == ARR_N0 || q.a == ARR_N1) {
    int side = q.a == ARR_N0 ? 0 : 1;
    long long row = slot_row(d, wb, w, bi, side, q.r);
    if (row >= 0 && row < d.n_rows[side]) key = (side ? rbase : 0ull) + (unsigned long long)row;
  } else if (q.r < bi.n) {
    long long e = bi.e0 + q.r;
    if (q.a == ARR_Q0) {
      long long row = w.rhs[e];
      if (row >= 0 && row < d.n_rows[1]) key = rbase + (unsigned long long)row;
    } else if (q.a == ARR_Q1) {
      long long row = w.lhs[e];
      if (row >= 0 && row < d.n_rows[0]) key = (unsigned long long)row;
    } else if (d.dynamic && d.op != PBG_OP_NONE) {
      long long rl = w.rel[e];
      int t = q.a == ARR_R0 ? 0 : 1;
      if (rl >= 0 && rl < d.num_rels) key = d.key_rel_base + (unsigned long long)t * d.num_rels + (unsigned long long)rl;
    }
  }
  return key;
}

// Programmatic dependent launch: every kernel of the step is launched while the kernel before it in the stream still
// runs (pbg_launch) and begins with this -- it waits until that one is complete and its writes are visible, then lets
// the next one be scheduled.  What overlaps is the launch itself, one to two microseconds per kernel of a step of ten.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() { pdl_wait(); pdl_release(); }

// Siblings: two launches in a row that read the same inputs and write different places.  The second starts as the first
// one's CTAs leave (their last round is half empty) and is complete only after it (what comes next counts on both).  What it
// reads has been waited for by the first, but the memory model gives that to the first alone, so the first hands it on: one
// thread, behind the wait, releases a word, and the second acquires it before it reads anything -- by causality it then sees
// what the first saw.  Where the word is not there yet, or not any more, it waits like every other kernel.  The
// second clears the word behind its wait for the first's end, so each pair starts from zero.
//   first:   pdl_begin_open(word)         (all threads; a null word: no sibling follows)
//   second:  pdl_release(), then seam_enter(word) by every thread that reads, each for itself, and by whole warps;
//            pdl_wait() and seam_close(word) before it ends.  Inputs through plain or __ldcg loads and bulk copies only:
//            the read-only path (const __restrict__ pointers) is outside of the memory model's order.
__device__ __forceinline__ void pdl_begin_open(unsigned *seam) {
  int opens = seam != nullptr && blockIdx.x == 0;
  asm volatile("" : "+r"(opens));                            // (the parameter is fetched in front of the wait, not behind it)
  pdl_wait();
  if (opens) {
    if (threadIdx.x == 0) asm volatile("st.release.gpu.global.u32 [%0], %1;" :: "l"(seam), "r"(1u) : "memory");
    __syncthreads();                                         // (the dependents are let go by the first thread that gets there)
  }
  pdl_release();
}
__device__ __forceinline__ void seam_enter(const unsigned *seam) {
  unsigned open;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(open) : "l"(seam) : "memory");
  if (open == 0u) pdl_wait();
  __syncwarp();
  asm volatile("fence.proxy.async.global;" ::: "memory");    // bulk copies read behind it too
}
__device__ __forceinline__ void seam_close(unsigned *seam) {
  if (threadIdx.x == 0) *seam = 0u;
}

// N3 regularizer pieces at elements [dd, dd + 4) of a row y: the term is sum m^3 with m = |y_d|, or for
// complex_diagonal the modulus of the pair (y_d, y_{d +- D/2}) counted once per pair
// (torchbiggraph/operators.py:42-43, 151-157).  n3_grad4: d(sum m^3)/dy = 3 m y.
__device__ __forceinline__ float4 n3_grad4(const float *y, int dd, int D, bool cplx) {
  float4 v = *reinterpret_cast<const float4 *>(y + dd);
  if (!cplx) return make_float4(3.f * fabsf(v.x) * v.x, 3.f * fabsf(v.y) * v.y, 3.f * fabsf(v.z) * v.z, 3.f * fabsf(v.w) * v.w);
  int h = D >> 1;
  float4 p = *reinterpret_cast<const float4 *>(y + (dd < h ? dd + h : dd - h));
  return make_float4(3.f * sqrtf(v.x * v.x + p.x * p.x) * v.x, 3.f * sqrtf(v.y * v.y + p.y * p.y) * v.y,
                     3.f * sqrtf(v.z * v.z + p.z * p.z) * v.z, 3.f * sqrtf(v.w * v.w + p.w * p.w) * v.w);
}
__device__ __forceinline__ float n3_val4(const float *y, int dd, int D, bool cplx) {
  float4 v = *reinterpret_cast<const float4 *>(y + dd);
  if (!cplx) { float a = fabsf(v.x), b = fabsf(v.y), c = fabsf(v.z), e = fabsf(v.w); return a * a * a + b * b * b + c * c * c + e * e * e; }
  int h = D >> 1;
  if (dd >= h) return 0.f;                                  // the pair is counted at its real part
  float4 p = *reinterpret_cast<const float4 *>(y + dd + h);
  float a = sqrtf(v.x * v.x + p.x * p.x), b = sqrtf(v.y * v.y + p.y * p.y), c = sqrtf(v.z * v.z + p.z * p.z), e = sqrtf(v.w * v.w + p.w * p.w);
  return a * a * a + b * b * b + c * c * c + e * e * e;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ int warp_sum_int(int v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }
__device__ __forceinline__ float4 f4zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ float4 operator+(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 operator-(float4 a, float4 b) { return make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w); }
__device__ __forceinline__ float4 operator*(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float4 operator*(float4 a, float s) { return make_float4(a.x * s, a.y * s, a.z * s, a.w * s); }
// (Rounding orders spelled out: which products the compiler contracts would otherwise depend on the code around the call.
// Two are in use, so that sums stay bit for bit what they were when their kernels were written.)
__device__ __forceinline__ float f4dot(float4 a, float4 b) { return __fmaf_rn(a.w, b.w, __fmaf_rn(a.z, b.z, __fmaf_rn(a.y, b.y, __fmul_rn(a.x, b.x)))); }
__device__ __forceinline__ float f4dot_yx(float4 a, float4 b) { return __fmaf_rn(a.w, b.w, __fmaf_rn(a.z, b.z, __fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)))); }
__device__ __forceinline__ float f4sum(float4 a) { return a.x + a.y + a.z + a.w; }
// The three bf16 planes of x (round to nearest each time; the remainders are exact in fp32):
// float(b0) + float(b1) + float(b2) == x to 24 mantissa bits.
__device__ __forceinline__ void bf16_planes(float x, unsigned &b0, unsigned &b1, unsigned &b2) {
  __nv_bfloat16 h0 = __float2bfloat16_rn(x);
  float r = x - __bfloat162float(h0);
  __nv_bfloat16 h1 = __float2bfloat16_rn(r);
  r -= __bfloat162float(h1);
  b0 = __bfloat16_as_ushort(h0); b1 = __bfloat16_as_ushort(h1); b2 = __bfloat16_as_ushort(__float2bfloat16_rn(r));
}
// planes of four consecutive values, packed for one 8-byte store per plane
__device__ __forceinline__ void bf16_planes4(float4 v, uint2 &p0, uint2 &p1, uint2 &p2) {
  unsigned a0, a1, a2, b0, b1, b2, c0, c1, c2, d0, d1, d2;
  bf16_planes(v.x, a0, a1, a2); bf16_planes(v.y, b0, b1, b2); bf16_planes(v.z, c0, c1, c2); bf16_planes(v.w, d0, d1, d2);
  p0 = make_uint2(a0 | (b0 << 16), c0 | (d0 << 16));
  p1 = make_uint2(a1 | (b1 << 16), c1 | (d1 << 16));
  p2 = make_uint2(a2 | (b2 << 16), c2 | (d2 << 16));
}
// one value's planes into a plane array: p0 at dst, the others one / two plane strides further
__device__ __forceinline__ void put_planes1(unsigned short *dst, size_t plane, float v, int npl) {
  unsigned b0, b1, b2;
  bf16_planes(v, b0, b1, b2);
  dst[0] = (unsigned short)b0; dst[plane] = (unsigned short)b1;
  if (npl > 2) dst[2 * plane] = (unsigned short)b2;
}
// tf32(x), the part of x a kind::tf32 MMA sees exactly: round to nearest, 10 mantissa bits kept, by two integer instructions
// (add half an ulp of the 10-bit mantissa, clear the low 13 bits): cvt.rna.tf32 runs at a fraction of the ALU rate, which is
// what bounds a kernel that splits whole operand tiles.  Differs from cvt only on NaN payloads and when rounding carries
// into Inf.
__device__ __forceinline__ float tf32_round(float x) { return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u); }
__device__ __forceinline__ float4 tf32_round4(float4 v) { return make_float4(tf32_round(v.x), tf32_round(v.y), tf32_round(v.z), tf32_round(v.w)); }

// 16 bytes from global to shared memory, asynchronously; zeros without `real`.
__device__ __forceinline__ void cp_async16(float *dst, const float *src, bool real) {
  const int bytes = real ? 16 : 0;                    // nothing read, zeros written
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

// ---- host-side helpers ---------------------------------------------------------------------------
// Opt-in to more than 48 KB of dynamic shared memory.  The attribute belongs to the (kernel, device)
// pair, so a process that drives several GPUs has to set it on each of them: the pairs already done
// are remembered under a mutex, with the device that is current at the call.
// A launch that fails because of its configuration leaves an error that a later successful call can hide
// from a cudaGetLastError made at the end of an entry point: the launchers note it at once in this
// per-thread latch, which the entry points read (and clear) before they report success.
inline cudaError_t &pbg_launch_error() {
  static thread_local cudaError_t e = cudaSuccess;
  return e;
}
inline void pbg_note_launch(cudaError_t e = cudaGetLastError()) {
  if (e != cudaSuccess && pbg_launch_error() == cudaSuccess) pbg_launch_error() = e;
}
// Nothing is launched behind a launch that failed: the kernels of a call take what the ones before them left (sorted keys,
// counts, sums) for places in memory, and would find another call's there.
inline bool pbg_launch_failed() { return pbg_launch_error() != cudaSuccess; }
inline cudaError_t pbg_take_launch_error() {
  const cudaError_t e = pbg_launch_error(), last = cudaGetLastError();      // (the runtime keeps the same error: taken with it)
  pbg_launch_error() = cudaSuccess;
  return e != cudaSuccess ? e : last;
}
inline cudaError_t pbg_opt_in_smem(const void *kernel, int bytes) {
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, int> done;       // (kernel, device) -> bytes opted in so far
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) { pbg_note_launch(e); return e; }
  std::lock_guard<std::mutex> lock(mu);
  auto it = done.find({kernel, dev});
  if (it != done.end() && it->second >= bytes) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done[{kernel, dev}] = bytes;
  else pbg_note_launch(e);
  return e;
}
// Opt-in to clusters of sixteen CTAs (eight is the portable limit), per (kernel, device) like the above.
inline cudaError_t pbg_opt_in_cluster16(const void *kernel) {
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, bool> done;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) { pbg_note_launch(e); return e; }
  std::lock_guard<std::mutex> lock(mu);
  bool &d = done[{kernel, dev}];
  if (d) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) d = true;
  else pbg_note_launch(e);
  return e;
}
inline int pbg_sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 1;
  return sms > 0 ? sms : 1;
}

// Launches a kernel that begins with pdl_begin().
template <class... P, class... A>
inline void pbg_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
  if (pbg_launch_failed()) return;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at; cfg.numAttrs = 1;
  pbg_note_launch(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

// A kernel that waits for the whole launch before it, as CUDA's stream order has it.
template <class... P, class... A>
inline void pbg_launch_in_order(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
  if (pbg_launch_failed()) return;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
  pbg_note_launch(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

// The same as pbg_launch for a kernel of clusters of `ctas` CTAs.
template <class... P, class... A>
inline void pbg_launch_clusters(void (*kernel)(P...), int clusters, int ctas, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
  if (pbg_launch_failed()) return;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * ctas)); cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = ctas; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 2;
  pbg_note_launch(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

// ---- host-side launchers (one per translation unit) ------------------------------------------
struct SortPlan {
  unsigned long long *keys[2];
  unsigned int *vals[2];
  unsigned int *hist;     // pbg_sort_hist_entries(max_n) counters
  int max_n;              // capacity
  int result;             // which of keys[]/vals[] holds the sorted output after pbg_sort
};
int pbg_sort_warps(int n);
size_t pbg_sort_hist_entries(int n);   // digit counters (unsigned int) a sort of n pairs needs
// Stable LSD radix sort of n (key, value) pairs on `bits` low key bits; returns launches made.
int pbg_sort(SortPlan &sp, int n, int bits, cudaStream_t st);

// Stable sort in one kernel, a thread-block cluster per list: lists of at most PBG_CLUSTER_SORT_MAX pairs, keys below 2^32.
#define PBG_CLUSTER_SORT_MAX (16 * 1024 * 16)
inline bool pbg_cluster_sort_fits(long long n, int bits) { return n <= PBG_CLUSTER_SORT_MAX && bits <= 32; }
bool pbg_cluster_sort_available(long long n);   // on the current device, for lists of up to n pairs
#define PBG_SORT_WAVES 4            // most waves of one launch
struct SortWave { WaveBatches wb; int k; unsigned long long *keys; unsigned int *vals; };
struct SortWaves { SortWave w[PBG_SORT_WAVES]; int count; };
// keys of the slots of `waves` (built on the fly) sorted into each wave's keys / vals
int launch_sort_waves(const WaveDims &d, const WaveBufs &w, const SortWaves &waves, int bits, cudaStream_t st);
// rows[i] -> (row, i) pairs sorted by row; rows outside [0, num_rows) are flagged and sort to the end as num_rows
int launch_sort_rows(const long long *rows, long long num_rows, int n, int bits, unsigned long long *keys, unsigned int *vals,
                     int *errflag, cudaStream_t st);

int launch_build_keys(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w,
                      unsigned long long *keys, unsigned int *vals, cudaStream_t st);
int launch_gather(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st);
// seams: words 0 and 8 are those of the gradients' sibling launches (a wave's first and second part); zero between calls
void *pbg_tc_plan_create(const WaveDims &d, const WaveBufs &w, int nblk_max, int precision, unsigned *seams);
void pbg_tc_plan_destroy(void *plan);
// standard relations, plane tiers: score contraction of both problems + loss + coefficient planes in one kernel
void *pbg_pair_plan_create(const WaveDims &d, const WaveBufs &w, int nblk_max);
void pbg_pair_plan_destroy(void *plan);
int launch_pair_score(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, void *plan, cudaStream_t st);
int launch_grad_dual_tc(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, void *plan, cudaStream_t st);
int launch_score_tc(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, void *plan, cudaStream_t st);
int launch_grad_tc(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, void *plan, cudaStream_t st);
int launch_matrix_forward(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st);
int launch_matrix_backward(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st);
int launch_matrix_update(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, float lr, cudaStream_t st);
int launch_postop(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st);
int launch_gz_rows(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st);
int launch_score_simt(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st);
int launch_grad_simt(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st);
// Gather, scores, loss, gradients and pull-back of the chunk blocks of a small wave in one kernel, a cluster of CTAs to a block.
// pbg_chunk_fits: shapes it takes; pbg_chunk_available: the current device can hold its clusters.
bool pbg_chunk_fits(int Pm, int Mm, int D);
bool pbg_chunk_available();
int launch_chunk_step(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st);
// the forward half of it for one batch, straight into the caller's score arrays (see launch_export_scores)
int launch_chunk_scores(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, float *lhs_pos, float *rhs_pos, float *lhs_neg, float *rhs_neg, cudaStream_t st);
int launch_loss(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st);
int launch_export_scores(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w,
                         float *lhs_pos, float *rhs_pos, float *lhs_neg, float *rhs_neg, cudaStream_t st);
// What the optimizer kernels of a wave work with.  hubcnt: two sets of counters, HUB_SET ints apart, used in turn
// (*turn): while one set counts, the kernel behind it clears the other for the next user; a set holds the words of the
// sibling launches too (HUB_SEAM_*).  per_batch (may be null) / sum: where
// the Stats of the wave's batches go.
struct UpdateScratch {
  float *psum; long long *hublist; int *hubcnt; unsigned *turn; long long *bigtab;
  pbg_batch_stats *per_batch; double *sum;
};
int launch_update(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, const unsigned long long *keys, const unsigned int *vals,
                  float lr, float rel_lr, const UpdateScratch &us, cudaStream_t st);
// hublist and bigtab: a part for the embedding rows and one for the operator rows (as are hubcnt[0..1] and hubcnt[HUB_REL ..] of a set).
// Places in a set of hubcnt, a line each: the operator rows' counters, the words (pdl_begin_open) of the two tile and the two
// hub kernels.
enum { HUB_REL = 32, HUB_SEAM_TILE = 64, HUB_SEAM_HUB = 96, HUB_SET = 128 };
inline long long pbg_hublist_entries(long long nocc) { return nocc / 8 + 64; }
// bigtab: a line for each row with 256 and more slots: where its batches start, and (last) a counter (zero between waves)
enum { BIGTAB_LINE = PBG_KMAX + 1 };
inline size_t pbg_bigtab_bytes(long long nocc) { return (size_t)(nocc / 256 + 2) * BIGTAB_LINE * sizeof(long long); }
// Evaluation of one batch after its scores.  out8 (host or device memory): loss, then pos_rank, mrr, r1, r10, r50 summed over
// both sides, then the AUC hits per side.  part: 8 doubles for each of the kernel's CTAs; done: a counter, zero at first.
inline int pbg_eval_auc_ctas(int nblk, int Pm) { return (int)((2ll * nblk * Pm + 255) / 256); }
inline int pbg_eval_ctas(int nblk, int Pm) { return pbg_eval_auc_ctas(nblk, Pm) + (int)((2ll * nblk * Pm + 7) / 8); }
int launch_eval(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, double *part, unsigned *done, double *out8, cudaStream_t st);
// The evaluator's last step, by the last CTA of a kernel (256 threads): the CTAs' partial sums [ctas][8] added up in a
// fixed order (32 runs, then the runs), the counter cleared for the next call.
__device__ __forceinline__ void close_eval(const double *part, int ctas, unsigned *done, double *out8) {
  __shared__ double run[32][8];
  const int k = threadIdx.x & 7, y = threadIdx.x >> 3;
  double s = 0.0;
  __threadfence();
  for (int c0 = y; c0 < ctas; c0 += 32 * 8) {                // eight reads in flight, past the L1
    double x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = c0 + 32 * u < ctas ? __ldcg(part + (size_t)(c0 + 32 * u) * 8 + k) : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) s += x[u];
  }
  run[y][k] = s;
  __syncthreads();
  if (threadIdx.x < 8) {
    double t = 0.0;
    for (int u = 0; u < 32; ++u) t += run[u][k];
    out8[k] = t;
    if (k == 0) *done = 0u;
    __threadfence_system();
  }
}

// Ranking against all entities (pbg_gather.cu, pbg_rank_tc.cu): one chunk holds the batch of B edges, the candidates of a
// side come in slabs of its table.
struct AllNegs {
  float *Q[2];            // [B][Dp]  Q[0]: scored against lhs candidates (op_rhs(rhs) rows), Q[1]: against rhs candidates
  float *qn[2], *pos[2];  // [B] |q|^2 (l2 family); positive score of problem 0 / 1
  float *Y[2], *yn[2];    // candidate slab [slab][Dp] (fp32 tier), |y|^2
  unsigned short *QB, *YB;              // other tiers: bf16 planes [2][3][qrows][Dpb], [2][3][slab][Dpb]
  int *pcnt[2]; float *pa[2], *pb[2];   // per (tile of the slab, edge): count, loss partials
  int *cnt[2]; float *ra[2], *rb[2];    // per-edge state over the slabs so far
  int *auc[2];                          // per edge: did its sample of the randomized AUC hit
  unsigned *seam;                       // word of the first two kernels, siblings (pdl_begin_open)
  double *part; unsigned *done;         // per-CTA sums of the last kernel, and how many CTAs have left theirs
  int B, slab, qrows, Dpb, tiles;       // tiles: partials per edge and slab
};
size_t pbg_allnegs_bytes(int maxB, int D, bool planes, long long table_rows, int &slab);
// out8: what the evaluator returns (see launch_eval), in host or device memory
int launch_allnegs_eval(const WaveDims &d, const WaveBufs &w, char *mem, int maxB, int B, int slab, bool planes, int rel_std, float wrel,
                        unsigned *done, unsigned *seam, double *out8, cudaStream_t st);
int launch_allnegs_score_tc(const WaveDims &d, const WaveBufs &w, const AllNegs &a, long long row0, cudaStream_t st);
int launch_reg_value(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st);
int launch_row_adagrad_sorted(float *emb, float *state, int dim, const unsigned long long *keys,
                              const unsigned int *vals, const float *grads, int n, float lr,
                              unsigned long long key_invalid, cudaStream_t st);
int launch_reverse_permutation(const long long *perm, long long n, long long *out, int *errflag, cudaStream_t st);
int launch_shuffle_rows(const void *in, void *out, long long rows, long long row_bytes, const long long *perm, int *errflag, cudaStream_t st);
int launch_randperm(SortPlan &sp, long long n, unsigned long long seed, long long *out, cudaStream_t st);
size_t pbg_randperm_bytes(long long n);
size_t pbg_randperm_counter_bytes();     // of it, at its start: the counters
int launch_randperm_dealt(char *mem, unsigned turn, long long n, unsigned long long seed, long long *out, int *errflag, cudaStream_t st);
bool pbg_sub_bucket_inline(int R);
int launch_sub_bucket(SortPlan &sp, const long long *lhs, const long long *rhs, const long long *rel, long long n, int R, const long long *tables,
                      const long long *tables_dev, int nl, int nr, int dynamic, long long *lhs_out, long long *rhs_out, long long *rel_out,
                      long long *counts, int *errflag, cudaStream_t st);
int launch_iota_keys(const long long *rows, long long num_rows, int n, unsigned long long *keys,
                     unsigned int *vals, int *errflag, cudaStream_t st);
