// A small wave in one kernel: what gather, score, loss, gradient and pull-back kernels do, for one chunk block per cluster.
//
// Up to the optimizer a chunk block needs nothing of another block.  A wave of one batch is some twenty blocks of 50 edges, and
// its kernels -- six or seven of them, each behind the whole grid of the one before -- take 3 to 13 us for work of one or two:
// start-up, tensor memory, the way through L2 of every intermediate.  Here a cluster of eight CTAs keeps a block from its ids
// to its gradient rows, with two cluster barriers on the way (2,000 cycles each, the write and the read through L2 that they
// order included):
//
//   gather     a warp per slot                             gather_slot -> X, aux, spos
//   scores     a CTA has up to 16 rows of one problem with all their columns: scores to shared memory, then a warp per row
//              takes the loss and writes the coefficients  loss_row    -> T, loss, violators
//   gradients  a CTA has 32 gradient rows of one side, a warp four of them with all columns in its lanes: the pull-back
//              follows in registers                        -> GX.  Standard relations: the merged coefficients
//              A[side] = T_side^T + T_other are added up on their way into shared memory, no array of them exists
//
// The products run on the CUDA cores in every precision tier: fp32 products summed in fp32, k ascending, which is what the
// fp32 tier's gemm_tile_kernel computes bit for bit, and closer to the exact sum than the split operands of the others.
//
// What bounds it: the chain.  Cycles of a block of 50 edges and 100 columns, dimension 100, cos: gather 7,600, barrier 2,200,
// scores and loss 17,000, barrier 3,200, gradients and pull-back 15,000 to 21,000 -- a quarter of it waiting for instructions
// that every launch fetches anew, shared-memory reads in the products most of the rest (a 16-byte read is four wavefronts, also
// where the warp reads one address).  27 us where the kernels it replaces took 47 of a fp32 batch of 1000 edges: the whole call
// 91.0 -> 71.2 us.  Passes of their own for scores, loss, gradients and pull-back (four barriers) took 31 us; one CTA per
// block and problem on the tensor cores, everything in shared memory, 25 to 28 (16 warps an SM are too few for per-row work).
#include <cooperative_groups.h>

#include "pbg_rows.cuh"

namespace cg = cooperative_groups;

#define CHUNK_CTAS 8
#define CHUNK_WARPS 8
#define CHUNK_THREADS (32 * CHUNK_WARPS)
#define CHUNK_K 128                 // k-values of a staged tile, and columns of a score tile
#define CHUNK_LD (CHUNK_K + 4)      // row stride of a k-contiguous tile: rows 4 banks apart, 16-byte reads without conflicts
#define CHUNK_BM 16                 // rows of a score tile
#define CHUNK_BG 32                 // rows of a gradient tile: four for each warp
#define CHUNK_MM 256                // most columns

struct ChunkOut { float *pos[2], *neg[2]; };          // scores only: [count], [count, columns] per problem

// The scores of this CTA's share of the rows of problem p, 16 rows at a time with all their columns, and what becomes of
// them: the loss and the coefficients (TRAIN), or the caller's score arrays.
template <int NV, bool TRAIN>
__device__ __forceinline__ void chunk_scores(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, const BlockInfo &bi, int blk, int p, int part, int parts, float *sm, const ChunkOut &out) {
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5, lane = tx;
  const int c_lo = d.batch_negs ? 0 : d.Pm;           // without batch negatives the chunk's own columns are all masked
  const int nk = (d.D + CHUNK_K - 1) / CHUNK_K;
  float *Ss = sm, *As = Ss + CHUNK_BM * (CHUNK_MM + 4), *Bs = As + CHUNK_BM * CHUNK_LD;
  const float *A = w.X[ARR_Q0 + p] + (size_t)blk * w.xrows[ARR_Q0 + p] * d.Dp, *B = w.X[ARR_N0 + p] + (size_t)blk * d.Mm * d.Dp;
  const int rows = TRAIN ? d.Pm : bi.n, share = (rows + parts - 1) / parts, m_end = min(rows, (part + 1) * share);
  for (int m0 = part * share; m0 < m_end; m0 += CHUNK_BM) {
    const int mrows = min(CHUNK_BM, min(m_end, bi.n) - m0);         // (edges; rows behind them only get their zeros)
    for (int n0 = c_lo; n0 < d.Mm && mrows > 0 && d.neg_enabled[p]; n0 += CHUNK_K) {
      const int ncols = min(CHUNK_K, d.Mm - n0);
      float acc[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
      for (int kc = 0; kc < nk; ++kc) {
        const int k0 = kc * CHUNK_K, k4s = (min(CHUNK_K, d.D - k0) + 3) / 4;
        __syncthreads();                              // the last readers of the buffers
        for (int i = tid; i < (CHUNK_BM + CHUNK_K) * (CHUNK_K / 4); i += CHUNK_THREADS) {
          const int row = i / (CHUNK_K / 4), k4 = i % (CHUNK_K / 4);
          const bool a = row < CHUNK_BM;
          const int r = a ? row : row - CHUNK_BM;
          const bool real = a ? r < mrows : r < ncols;
          if (k4 < k4s && (a || r < (ncols + 31) / 32 * 32))
            cp_async16((a ? As : Bs) + r * CHUNK_LD + k4 * 4, (a ? A + (size_t)(real ? m0 + r : 0) * d.Dp : B + (size_t)(real ? n0 + r : 0) * d.Dp) + k0 + k4 * 4, real);
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        // a warp has two rows, a lane every 32nd column
        const float *a0 = As + ty * 2 * CHUNK_LD, *b0 = Bs + tx * CHUNK_LD;
        if (ty * 2 < mrows)
#pragma unroll 2
          for (int k4 = 0; k4 < k4s; ++k4) {
            float4 a[2], b[4];
#pragma unroll
            for (int i = 0; i < 2; ++i) a[i] = ld4(a0 + i * CHUNK_LD + k4 * 4);
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = j * 32 < ncols ? ld4(b0 + j * 32 * CHUNK_LD + k4 * 4) : f4zero();
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
                acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
                acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
                acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
              }
          }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int m = ty * 2 + i;
        if (m >= mrows) continue;
        const float an = d.cmp >= PBG_CMP_L2 ? w.aux[ARR_Q0 + p][(size_t)blk * w.xrows[ARR_Q0 + p] + m0 + m] : 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int n = n0 + tx + 32 * j;
          if (n >= d.Mm) continue;
          float v = acc[i][j];
          if (d.cmp >= PBG_CMP_L2) {                  // model.py:226-246, as in gemm_tile_kernel
            const float q = (w.aux[ARR_N0 + p][(size_t)blk * d.Mm + n] - 2.0f * v) + an;
            v = d.cmp == PBG_CMP_L2 ? -sqrtf(fmaxf(q, 1e-30f)) : -q;
          }
          if (TRAIN) Ss[m * (CHUNK_MM + 4) + n] = v;
          else if (n >= d.Pm || n < bi.Pl) {          // (columns between a short chunk's edges and the uniform ones do not exist)
            const int cols = d.batch_negs ? bi.Pl + d.U : d.U, col = n >= d.Pm ? cols - d.U + n - d.Pm : n;
            out.neg[p][(size_t)(bi.c * bi.Pl + m0 + m) * cols + col] = col_masked(d, bi, 1, m0 + m, n) ? PBG_MASKED : v;
          }
        }
      }
    }
    if (!TRAIN) {
      if (tid < mrows) out.pos[p][bi.c * bi.Pl + m0 + tid] = w.spos[p][(size_t)blk * d.Pm + m0 + tid];
      continue;
    }
    __syncwarp();                                     // a warp's two rows are its own
    for (int m = ty * 2; m < ty * 2 + 2 && m0 + m < m_end; ++m) {
      const float *Sr = Ss + m * (CHUNK_MM + 4);
      if (d.loss == PBG_LOSS_SOFTMAX && d.cmp < PBG_CMP_L2) loss_softmax_row<NV, true>(d, wb, w, p, blk, m0 + m, lane, Sr);
      else loss_row<NV, true>(d, wb, w, p, blk, m0 + m, lane, Sr);
    }
  }
}

// Gradient rows, C (M x D) = A (M x K) . B (K x D, rows of an operand array), where
//   A[m][k] = (At, k < kt ? At[k][m] : 0) + (Ad, m < md ? Ad[m][k] : 0)
// At and Ad are coefficient matrices of the block (row stride Ms); either may be null.
struct ChunkProduct { const float *At, *Ad, *B; int a, M, K, kt, md; };

// 32 rows of it, four to a warp with all their columns in its lanes, and their pull-back.
template <int VEC, int CK>
__device__ __forceinline__ void chunk_gradient_rows(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, const BlockInfo &bi, int blk, const ChunkProduct &g, int m0, bool pull, float *sm) {
  constexpr int KC = CHUNK_K / VEC, W = VEC * 128;    // rows of B at a time, and their width
  const int tid = threadIdx.x, lane = tid & 31, wl = tid >> 5, D = d.D;
  float *As = sm, *Bs = sm + CHUNK_BG * CHUNK_LD;
  const int a = g.a, side = slot_side(a), mw = m0 + wl * 4;
  // entities of the warp's rows: asked for here, needed behind the product
  const long long id_l = pull && lane < 4 && mw + lane < g.M ? slot_row(d, wb, w, bi, side, mw + lane) : -1;
  float4 acc[4][VEC];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int c = 0; c < VEC; ++c) acc[i][c] = f4zero();
  float rs[4] = {0.f, 0.f, 0.f, 0.f};                 // l2 family: row sums of A
  const int mt = tid & 31, m = m0 + mt, kq = tid >> 5;
  for (int ka = 0; ka < g.K; ka += CHUNK_K) {         // k-values of A in shared memory
    const int kas = min(CHUNK_K, g.K - ka), k4s = (kas + 3) / 4;
    __syncthreads();
    // a thread brings four k-values of a row at a time; all of its requests go out before the first is used
    float4 t[4], o[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k4 = kq + 8 * u, k = ka + 4 * k4;
      const bool in = k4 < k4s;
      auto at = [&](int q) { return in && g.At && m < d.Mm && k + q < g.kt ? g.At[(size_t)(k + q) * d.Ms + m] : 0.f; };
      t[u] = make_float4(at(0), at(1), at(2), at(3));
      o[u] = in && g.Ad && m < g.md ? ld4(g.Ad + (size_t)m * d.Ms + k) : f4zero();
    }
    for (int kb = 0; kb < kas; kb += KC) {            // rows of B beside it
      const int kbs = min(KC, kas - kb);
      if (kb > 0) __syncthreads();
      for (int i = tid; i < (kbs + 3) / 4 * 4 * (W / 4); i += CHUNK_THREADS) {
        const int k = i / (W / 4), c4 = i % (W / 4) * 4;
        const bool real = k < kbs && c4 < D;
        if (c4 < D) cp_async16(Bs + k * W + c4, real ? g.B + (size_t)(ka + kb + k) * d.Dp + c4 : g.B, real);
      }
      cp_async_commit();
      if (kb == 0) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int k4 = kq + 8 * u;
          if (k4 < k4s) st4(As + mt * CHUNK_LD + k4 * 4, t[u] + o[u]);
        }
      }
      cp_async_wait<0>();
      __syncthreads();
      const float *aw = As + wl * 4 * CHUNK_LD + kb, *bl = Bs + lane * 4;
      if (mw < g.M)
#pragma unroll 1
        for (int k4 = 0; k4 < (kbs + 3) / 4; ++k4) {
          float4 av[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) av[i] = ld4(aw + i * CHUNK_LD + k4 * 4);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float4 b[VEC];
#pragma unroll
            for (int c = 0; c < VEC; ++c) b[c] = ld4(bl + (k4 * 4 + q) * W + c * 128);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float x = q == 0 ? av[i].x : q == 1 ? av[i].y : q == 2 ? av[i].z : av[i].w;
#pragma unroll
              for (int c = 0; c < VEC; ++c) {
                acc[i][c].x = fmaf(x, b[c].x, acc[i][c].x);
                acc[i][c].y = fmaf(x, b[c].y, acc[i][c].y);
                acc[i][c].z = fmaf(x, b[c].z, acc[i][c].z);
                acc[i][c].w = fmaf(x, b[c].w, acc[i][c].w);
              }
            }
          }
        }
    }
    if (CK == CK_L2) {
      // lane by lane as coef_kernel takes them (columns lane, lane + 32, ...)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        for (int k = lane; k < kas; k += 32) rs[i] += As[(wl * 4 + i) * CHUNK_LD + k];
    }
  }
  float4 yv[4][VEC];
  float cf[4], inv[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const size_t xr = (size_t)blk * w.xrows[a] + mw + i, gr = (size_t)blk * w.grows[a] + mw + i;
    const bool in = mw + i < g.M;
    // (l2: the rows of GQ take the row sums of T, which the loss has left; the others those of A)
    cf[i] = CK == CK_L2 && in ? (a >= ARR_Q0 && d.dynamic ? w.coef[a][gr] : 0.f) : 0.f;
    inv[i] = CK == CK_COS && in ? w.aux[a][xr] : 1.f;
#pragma unroll
    for (int c = 0; c < VEC; ++c) {
      const int dd = c * 128 + lane * 4;
      yv[i][c] = CK != CK_DOT && in && dd < D ? ld4(w.X[a] + xr * d.Dp + dd) : f4zero();
      if (dd >= D) acc[i][c] = f4zero();              // (columns of B behind the rows' end were never staged)
    }
  }
  float *part = As + wl * 4 * CHUNK_LD;               // the warp's own rows of A: read for the last time by it
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = mw + i;
    if (r >= g.M) break;
    const long long id = __shfl_sync(0xffffffffu, id_l, i);
    if (!pull) { store_row<VEC>(w.GX[a] + ((size_t)blk * w.grows[a] + r) * d.Dp, acc[i], D, lane); continue; }
    if (id < 0 || id >= d.n_rows[side]) {
      if (d.dynamic) dyn_pullback_empty<VEC>(d, w, a, blk, r, lane); else std_pullback_empty<VEC>(d, w, side, blk, r, lane);
      continue;
    }
    if (CK == CK_L2 && !(a >= ARR_Q0 && d.dynamic)) cf[i] = warp_sum(rs[i]);
    const float *y = w.X[a] + ((size_t)blk * w.xrows[a] + r) * d.Dp;
    gz_math<VEC, CK>(acc[i], yv[i], y, cf[i], inv[i], d, lane, d.reg_coef != 0.f && r < bi.n && r < d.Pm);
    if (d.dynamic) dyn_pullback_finish<VEC, CK>(acc[i], d, w, a, bi, blk, r, lane, part);
    else std_pullback_finish<VEC>(acc[i], d, wb, w, side, bi, blk, r, id, lane, part);
  }
}

// Standard relations: GN_side = A[side] . N_other, two products.  Dynamic ones: GN_p = T_p^T . Q_p, GQ_p = T_p . N_p.
template <int VEC, int CK>
__device__ __forceinline__ void chunk_gradients(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, const BlockInfo &bi, int blk, int side, int part, int parts, float *sm) {
  const int tm = (d.Mm + CHUNK_BG - 1) / CHUNK_BG, tq = d.dynamic ? (bi.n + CHUNK_BG - 1) / CHUNK_BG : 0;
  const size_t tblk = (size_t)blk * d.Pm * d.Ms;
  const bool has_op = d.op != PBG_OP_NONE && w.theta[0] != nullptr;
  const bool rows_change = CK != CK_DOT || d.reg_coef != 0.f;
  const float *T = w.S[side] + tblk;
  for (int mt = part; mt < tm + tq; mt += parts) {
    ChunkProduct g;
    int m0 = mt * CHUNK_BG;
    bool pull = rows_change;
    if (mt >= tm) {                                   // GQ
      m0 = (mt - tm) * CHUNK_BG;
      g.At = nullptr; g.Ad = T; g.B = w.X[ARR_N0 + side] + (size_t)blk * d.Mm * d.Dp;
      g.a = ARR_Q0 + side; g.M = bi.n; g.K = d.Mm; g.kt = 0; g.md = bi.n;
      pull = pull || has_op;
    } else {
      const int from = d.dynamic ? ARR_Q0 + side : ARR_N0 + (1 - side);
      g.At = T; g.B = w.X[from] + (size_t)blk * w.xrows[from] * d.Dp;
      g.a = ARR_N0 + side; g.M = d.Mm; g.kt = bi.n;
      // rows behind the chunk's edges are scored in one problem only: nothing is added to their part of T^T
      const bool both = !d.dynamic && m0 < bi.n;
      g.Ad = both ? w.S[1 - side] + tblk : nullptr; g.md = bi.n; g.K = both ? d.Mm : bi.n;
      pull = pull || (!d.dynamic && side == 1 && w.PG);
    }
    chunk_gradient_rows<VEC, CK>(d, wb, w, bi, blk, g, m0, pull, sm);
  }
}

template <int VEC, int NV, bool TRAIN>
__global__ void __launch_bounds__(CHUNK_THREADS, 2)
chunk_kernel(const __grid_constant__ WaveDims d, const __grid_constant__ WaveBatches wb, const __grid_constant__ WaveBufs w, const __grid_constant__ ChunkOut out) {
  extern __shared__ __align__(16) float chunk_sm[];
  cg::cluster_group cluster = cg::this_cluster();
  const int nct = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), blk = d.blk0 + (int)blockIdx.x / nct;
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5, warp = wl * nct + rank, warps = CHUNK_WARPS * nct;
  pdl_begin();
  const BlockInfo bi = block_info(d, wb, blk);
  if (bi.n == 0) return;                              // (the whole cluster)
#pragma unroll 1
  for (int r = warp; r < d.Mm; r += warps) gather_slot<VEC, false>(d, wb, w, blk, r, lane);
  cluster.sync();
  chunk_scores<NV, TRAIN>(d, wb, w, bi, blk, rank & 1, rank >> 1, nct >> 1, chunk_sm, out);
  if (!TRAIN) return;
  cluster.sync();
  if (d.cmp >= PBG_CMP_L2) chunk_gradients<VEC, CK_L2>(d, wb, w, bi, blk, rank & 1, rank >> 1, nct >> 1, chunk_sm);
  else if (d.cmp == PBG_CMP_COS) chunk_gradients<VEC, CK_COS>(d, wb, w, bi, blk, rank & 1, rank >> 1, nct >> 1, chunk_sm);
  else chunk_gradients<VEC, CK_DOT>(d, wb, w, bi, blk, rank & 1, rank >> 1, nct >> 1, chunk_sm);
}

// ---- host side -----------------------------------------------------------------------------------
static size_t chunk_smem() {
  const size_t scores = CHUNK_BM * (CHUNK_MM + 4) + (CHUNK_BM + CHUNK_K) * CHUNK_LD, grads = CHUNK_BG * CHUNK_LD + CHUNK_K * CHUNK_K;
  return (scores > grads ? scores : grads) * sizeof(float);
}
bool pbg_chunk_fits(int Pm, int Mm, int D) { return Pm <= CHUNK_MM && Mm <= CHUNK_MM && D <= 256; }

template <int VEC, int NV, bool TRAIN>
static cudaError_t chunk_opt_in() { return pbg_opt_in_smem((const void *)chunk_kernel<VEC, NV, TRAIN>, (int)chunk_smem()); }

bool pbg_chunk_available() {
  const void *kernel = (const void *)chunk_kernel<2, 8, true>;                     // the one that takes the most registers
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CHUNK_CTAS); cfg.blockDim = dim3(CHUNK_THREADS); cfg.dynamicSmemBytes = chunk_smem();
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = CHUNK_CTAS; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
  cfg.attrs = &at; cfg.numAttrs = 1;
  int n = 0;
  const bool ok = chunk_opt_in<2, 8, true>() == cudaSuccess && cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n >= 1;
  if (!ok) pbg_take_launch_error();                   // (an answer, not a failure of the call that asked)
  return ok;
}

template <int VEC, int NV, bool TRAIN>
static void launch_chunk(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, const ChunkOut &out, cudaStream_t st) {
  chunk_opt_in<VEC, NV, TRAIN>();
  pbg_launch_clusters(chunk_kernel<VEC, NV, TRAIN>, d.nblk, CHUNK_CTAS, CHUNK_THREADS, chunk_smem(), st, d, wb, w, out);
}

int launch_chunk_step(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st) {
  WaveBufs v = w;
  for (int p = 0; p < 2; ++p) v.TB[p] = nullptr;      // (coefficients as fp32 only: the tensor cores have no part in this)
  const ChunkOut none = {};
  const int vec = (d.D + 127) / 128;
  const bool wide = d.Ms > 128;                       // (only where PBG_CHUNK=1 asks for it: by itself the rule stops at 128 columns)
#define CHUNK(V) (wide ? launch_chunk<V, 8, true>(d, wb, v, none, st) : launch_chunk<V, 4, true>(d, wb, v, none, st))
  if (vec <= 1) CHUNK(1); else CHUNK(2);
#undef CHUNK
  return 1;
}

int launch_chunk_scores(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, float *lhs_pos, float *rhs_pos, float *lhs_neg, float *rhs_neg, cudaStream_t st) {
  const ChunkOut out = {{lhs_pos, rhs_pos}, {lhs_neg, rhs_neg}};
  const int vec = (d.D + 127) / 128;
  if (vec <= 1) launch_chunk<1, 4, false>(d, wb, w, out, st);
  else launch_chunk<2, 4, false>(d, wb, w, out, st);
  return 1;
}
