// Optimizer steps of one wave.
//
// First the pull-back: what a gradient slot contributes depends on nothing but the slot's own rows, so one pass over
// the slots (std_pullback_kernel, dyn_pullback_kernel) takes every gradient row back through comparator.prepare and
// the relation operator in place, and sums or stores what the operator rows and global vectors get.
//
// The sorted occurrence list (pbg_sort.cu) puts all gradient slots of a table row next to each
// other, in batch order.  A warp keeps a row in registers, and for every batch of the wave that
// touched it sums the slots' gradient rows and applies one optimizer step:
//   embedding rows  RowAdagrad   G += mean(g^2); w -= lr g / (sqrt(G) + 1e-10)
//                                (torchbiggraph/row_adagrad.py:84-96; duplicates are summed first,
//                                 the `coalesce` of line 83)
//   operator rows   AsyncAdagrad G += g^2 elementwise; theta -= lr_rel g / (sqrt(G) + 1e-10)
//                                (torchbiggraph/async_adagrad.py:75-85)
// A row is read once and written once per wave however many batches touched it, and the
// optimizer state never leaves HBM.  Everything is summed in a fixed order: results are
// reproducible run to run.
#include "pbg_rows.cuh"

#define UPD_WARPS 8

// Standard relations: the pull-back of a wave's gradient slots, one warp per row of a chunk block and side -- the
// gradient of the raw row written over the slot's own gradient row.  Under diagonal and complex_diagonal the row's
// contribution to the relation's operator row goes to PG beside it (under a translation it IS the gradient row).
// first_side / sides: what is left out needs no change.  (One warp per row and no sums in here: a kernel that also
// summed per chunk block ran 20 CTAs on a single batch.)
template <int VEC, int CK>
__global__ void __launch_bounds__(32 * UPD_WARPS) std_pullback_kernel(WaveDims d, WaveBatches wb, WaveBufs w, int side0) {
  pdl_begin();
  extern __shared__ __align__(16) float wpart[];             // [UPD_WARPS][VEC * 128]
  const int wl = threadIdx.x >> 5, item = (int)blockIdx.x * UPD_WARPS + wl;
  if (item >= d.nblk * d.Mm) return;
  const int lb = d.byMm.div(item);
  const int side = side0 + blockIdx.y, a = side ? ARR_N1 : ARR_N0, blk = d.blk0 + lb, r = item - lb * d.Mm, lane = threadIdx.x & 31;
  if (side == 1 && d.matrix_op) return;                      // linear / affine: R2 holds the gradient of the raw row already
  const BlockInfo bi = block_info(d, wb, blk);
  if (bi.n <= 0) return;
  const long long row = slot_row(d, wb, w, bi, side, r);
  if (row < 0 || row >= d.n_rows[side]) { std_pullback_empty<VEC>(d, w, side, blk, r, lane); return; }
  float4 v[VEC];
  gz_row<VEC, CK>(v, d, w, a, blk, r, lane, d.reg_coef != 0.f && r < bi.n && r < d.Pm);
  std_pullback_finish<VEC>(v, d, wb, w, side, bi, blk, r, row, lane, wpart + (size_t)wl * VEC * 128);
}

// The vectors that every row of a batch shares in standard relations: the relation's operator row, and the vector of
// each entity type (config.global_emb: added to every row of the type before the operator, so its gradient is the sum of
// the raw rows' gradients).  Both steps ride on launches that are there anyway, as CTAs beside the embedding rows' work
// -- what they step is read by nothing before the next wave -- where they were four kernels of 14 to 27 us on a batch
// of 1000 edges at dimension 128, two of them a single CTA:
//   param_sums   beside the tiles: CTA (vector, chunk block, 128 columns) adds up the block's rows, warp u rows u, u + 8, ...
//                (two such sequences per warp here), the eight sums in order, into one partial row per block
//   param_step   beside the big hub rows: adds up a batch's partial rows and takes the dense AsyncAdagrad steps batch
//                after batch (torchbiggraph/async_adagrad.py:75-85, train_cpu.py:215-230)
// kinds: 0 operator row, 1 / 2 vector of the lhs / rhs entity type (one vector for both sides: two sums, one step)
// cleared0 / cleared1: the pull-back has been over every row of that side
struct ParamJob { int sums, sum_kind[3], steps, step_kind[3], cleared0, cleared1; float lr; };
static inline int param_sum_ctas(const WaveDims &d, const ParamJob &job) { return job.sums * d.nblk * ((d.D + 127) / 128); }
static inline int param_step_ctas(const WaveDims &d, const ParamJob &job) { return job.steps * ((d.D + 31) / 32); }

// (128 threads)
__device__ __forceinline__ void param_sums(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, const ParamJob &job, int cta, float *sm) {
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int cols = (d.D + 127) / 128;
  const int dd = (cta % cols) * 128 + lane * 4;
  const int blk = cta / cols % d.nblk, kind = job.sum_kind[cta / cols / d.nblk];
  const int side = kind == 1 ? 0 : 1;
  const BlockInfo bi = block_info(d, wb, blk);
  const float *src = kind == 0 ? (w.PG ? w.PG : w.GX[ARR_N1]) : kind == 1 ? w.GX[ARR_N0] : d.matrix_op ? w.R2 : w.GX[ARR_N1];
  src += (size_t)blk * d.Mm * d.Dp + dd;
  // the rows of both sequences of this warp, four each in flight; rows without an entity behind them hold zeros where the
  // pull-back has been over them, else (checked) their ids are looked at
  const bool checked = kind == 0 ? !job.cleared1 : kind == 1 ? !job.cleared0 : !job.cleared1 || d.matrix_op;
  float4 s[2] = {f4zero(), f4zero()};
  if (bi.n > 0 && dd < d.D) {
    for (int r0 = wl; r0 < d.Mm; r0 += 32) {
      float4 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int r = r0 + 4 * u;
        bool real = r < d.Mm;
        if (checked && real) { const long long row = slot_row(d, wb, w, bi, side, r); real = row >= 0 && row < d.n_rows[side]; }
        v[u] = real ? ld4(src + (size_t)r * d.Dp) : f4zero();
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) s[u & 1] = s[u & 1] + v[u];
    }
    if (kind == 0 && wl == 0 && d.reg_coef != 0.f)
      // N3 regularizer on the relation's parameters: sum(params^3) * number of chunks
      // (regularizers.py:88-92), i.e. once per chunk block; theta is still the wave's snapshot here
      s[0] = s[0] + n3_grad4(w.theta[0] + (size_t)wb.rel[bi.b] * d.D, dd, d.D, d.op == PBG_OP_COMPLEX_DIAGONAL) * d.reg_coef;
  }
  st4(sm + wl * 128 + lane * 4, s[0]);
  st4(sm + (wl + 4) * 128 + lane * 4, s[1]);
  __syncthreads();
  if (wl == 0 && dd < d.D) {
    float4 t = ld4(sm + lane * 4);
#pragma unroll
    for (int u = 1; u < 8; ++u) t = t + ld4(sm + u * 128 + lane * 4);
    float *out = kind == 0 ? w.relpart : w.globpart + (kind == 2 ? (size_t)d.nblk * d.D : 0);
    st4(out + (size_t)blk * d.D + dd, t);
  }
}

// (256 threads; sm: PBG_KMAX * 32 floats)
__device__ __forceinline__ void param_step(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, const ParamJob &job, int cta, float *sm) {
  const int colctas = (d.D + 31) / 32;
  const int kind = job.step_kind[cta / colctas];
  const int col = threadIdx.x & 31, y = threadIdx.x >> 5, dd = (cta % colctas) * 32 + col;
  const float *part = (kind == 0 ? w.relpart : w.globpart + (kind == 2 ? (size_t)d.nblk * d.D : 0)) + dd;
  const float *part2 = kind == 1 && w.glob_shared ? w.globpart + (size_t)d.nblk * d.D + dd : nullptr;   // one vector: both sides' gradients add up
  if (dd < d.D) {
    for (int b = y; b < d.k; b += UPD_WARPS) {
      float s = 0.f, s2 = 0.f;
#pragma unroll 10
      for (int c = 0; c < d.Cm; ++c) s += part[((size_t)b * d.Cm + c) * d.D];
      if (part2) {
#pragma unroll 10
        for (int c = 0; c < d.Cm; ++c) s2 += part2[((size_t)b * d.Cm + c) * d.D];
        s += s2;
      }
      sm[b * 32 + col] = s;
    }
  }
  __syncthreads();
  if (y != 0 || dd >= d.D) return;
  float *acc = kind == 0 ? w.acc[0] : w.gacc[kind - 1], *val = kind == 0 ? w.theta[0] : w.glob[kind - 1];
  // the row of the relation in hand stays in registers (a global vector is one row)
  int cur = -1;
  float a = 0.f, v = 0.f;
  for (int b = 0; b < d.k; ++b) {
    if (wb.n[b] <= 0) continue;
    const int row = kind == 0 ? wb.rel[b] : 0;
    if (kind == 0 && (row < 0 || row >= d.num_rels)) continue;
    const float g = sm[b * 32 + col];
    if (row != cur) {
      if (cur >= 0) { acc[(size_t)cur * d.D + dd] = a; val[(size_t)cur * d.D + dd] = v; }
      cur = row;
      a = acc[(size_t)row * d.D + dd]; v = val[(size_t)row * d.D + dd];
    }
    a += g * g;
    v -= job.lr * g / (sqrtf(a) + PBG_ADAGRAD_EPS);
  }
  if (cur >= 0) { acc[(size_t)cur * d.D + dd] = a; val[(size_t)cur * d.D + dd] = v; }
}

// ------------------------------------------------------------------------------------------------
// Segmented optimizer step over the sorted slot list.
//
// The list is cut into tiles of TILE slots, one warp per tile (after issuing L2 prefetches for the
// gradient and table rows of its slots); the warp reads the keys of slots
// [t0-32, t0+32) and the values of [t0, t0+32) in two coalesced loads and finds segment (= table
// row) boundaries with ballots.
//   * a row with at most SHORT_MAX slots is handled entirely by the warp whose tile holds its first
//     slot: row and state in registers, one optimizer step per batch that touched it;
//   * a longer row (a hub of the graph) is summed tile by tile: every warp writes, for each
//     (batch, tile) run of its slots, one partial gradient row to psum[first slot of the run]; the
//     warp that holds the head registers the row in hublist, and hub_kernel finishes it
//     with one CTA per row (eight warps add the partial rows of a batch in a fixed order).
// RULE selects the table and its optimizer: embedding rows / RowAdagrad, or (dynamic relations)
// operator rows / AsyncAdagrad.
// ------------------------------------------------------------------------------------------------
#define TILE 4
#define SHORT_MAX 24
#define HUB_BIG 256     // rows with at least this many slots in a wave get their batches summed by separate CTAs
// hublist holds nocc / 8 + 64 entries; a hub row has more than SHORT_MAX slots, so the rows themselves need fewer than
// nocc / 16 + 32 of them and the list of big rows (at most nocc / HUB_BIG) lives in the rest.  hubcnt[0] counts hub
// rows, hubcnt[1] big rows.
__device__ __forceinline__ long long *hub_biglist(long long *hublist, int nocc) { return hublist + nocc / 16 + 32; }
__device__ __forceinline__ const long long *hub_biglist(const long long *hublist, int nocc) { return hublist + nocc / 16 + 32; }
enum { RULE_EMB = 0, RULE_REL = 1 };

// The kernels of the operator rows (dynamic relations) work beside those of the embedding rows launched just before them, as
// their siblings (pdl_begin_open): other rows, other places in psum, lists and counters of their own.  Each of the four is
// bound by the chain of one row, so in turn they took as long as all their chains together (dimension 400, 1,345 relations,
// every row a hub: the update 172 us a wave, 157 so; dimension 200, 14,824 relations: 169 and 164).  The last CTA of such a
// kernel has no other work than to wait for the end of the one before.
__host__ __device__ __forceinline__ bool has_operator_rows(const WaveDims &d) { return d.dynamic && d.op != PBG_OP_NONE; }
__device__ __forceinline__ bool sibling_begin(unsigned *seam) {
  pdl_release();
  if (blockIdx.x == gridDim.x - 1) {
    pdl_wait();
    seam_close(seam);
    return false;
  }
  seam_enter(seam);
  return true;
}
// The sorted list, the hub lists and their counters: written before the launch, so the operator rows' kernels, which do not
// wait for the launch before them, read past the read-only path.
template <int RULE, class T>
__device__ __forceinline__ T ld_list(const T *p) { return RULE == RULE_REL ? __ldcg(p) : *p; }

template <int VEC, int RULE>
struct RowState {
  float4 v[VEC], a[VEC];     // row; per-element accumulator (RULE_REL only)
  float G;                   // per-row accumulator (RULE_EMB only)
  float *prow, *pacc;

  // where the row and its optimizer state live
  __device__ __forceinline__ void locate(const WaveDims &d, const WaveBufs &w, unsigned long long key) {
    const int D = d.D;
    if (RULE == RULE_EMB) {
      int side = (!d.shared_table && key >= (unsigned long long)d.n_rows[0]) ? 1 : 0;
      long long row = (long long)(side ? key - (unsigned long long)d.n_rows[0] : key);
      prow = w.W[side] + (size_t)row * D;
      pacc = w.G[side] + row;
    } else {
      unsigned long long rk = key - d.key_rel_base;
      int t = rk >= (unsigned long long)d.num_rels ? 1 : 0;
      long long rl = (long long)(rk - (unsigned long long)t * d.num_rels);
      prow = w.theta[t] + (size_t)rl * D;
      pacc = w.acc[t] + (size_t)rl * D;
    }
  }
  __device__ __forceinline__ void load(const WaveDims &d, const WaveBufs &w, unsigned long long key, int lane) {
    const int D = d.D;
    locate(d, w, key);
    if (RULE == RULE_EMB) G = *pacc;
#pragma unroll
    for (int c = 0; c < VEC; ++c) {
      int dd = c * 128 + lane * 4;
      v[c] = dd < D ? ld4(prow + dd) : f4zero();
      if (RULE == RULE_REL) a[c] = dd < D ? ld4(pacc + dd) : f4zero();
    }
    if (RULE == RULE_EMB && d.max_norm > 0.f) {
      // the lookup of this wave used the row scaled to max_norm (F.embedding(max_norm=...), model.py:57-61;
      // same arithmetic as the gather): the table keeps the scaled row, the optimizer steps start from it
      float ss = 0.f;
#pragma unroll
      for (int c = 0; c < VEC; ++c) ss += f4dot(v[c], v[c]);
      float norm = sqrtf(warp_sum(ss));
      if (norm > d.max_norm) {
        float sc = d.max_norm / (norm + 1e-7f);
#pragma unroll
        for (int c = 0; c < VEC; ++c) v[c] = v[c] * sc;
      }
    }
  }
  // one optimizer step with the summed gradient g of one batch
  __device__ __forceinline__ void step(const float4 (&g)[VEC], float lr, float invD) {
    if (RULE == RULE_EMB) {
      float ss = 0.f;
#pragma unroll
      for (int c = 0; c < VEC; ++c) ss += f4dot(g[c], g[c]);
      ss = warp_sum(ss);
      G += ss * invD;
      float stepv = lr / (sqrtf(G) + PBG_ADAGRAD_EPS);
#pragma unroll
      for (int c = 0; c < VEC; ++c) v[c] = v[c] - g[c] * stepv;
    } else {
#pragma unroll
      for (int c = 0; c < VEC; ++c) {
        a[c] = a[c] + g[c] * g[c];
        v[c].x -= lr * g[c].x / (sqrtf(a[c].x) + PBG_ADAGRAD_EPS);
        v[c].y -= lr * g[c].y / (sqrtf(a[c].y) + PBG_ADAGRAD_EPS);
        v[c].z -= lr * g[c].z / (sqrtf(a[c].z) + PBG_ADAGRAD_EPS);
        v[c].w -= lr * g[c].w / (sqrtf(a[c].w) + PBG_ADAGRAD_EPS);
      }
    }
  }
  // RowAdagrad step of an embedding row whose batch's mean squared gradient is known already
  __device__ __forceinline__ void step_with_norm(const float4 (&g)[VEC], float lr, float mean_sq) {
    G += mean_sq;
    float stepv = lr / (sqrtf(G) + PBG_ADAGRAD_EPS);
#pragma unroll
    for (int c = 0; c < VEC; ++c) v[c] = v[c] - g[c] * stepv;
  }
  __device__ __forceinline__ void store(int D, int lane) {
#pragma unroll
    for (int c = 0; c < VEC; ++c) {
      int dd = c * 128 + lane * 4;
      if (dd < D) { st4(prow + dd, v[c]); if (RULE == RULE_REL) st4(pacc + dd, a[c]); }
    }
    if (RULE == RULE_EMB && lane == 0) *pacc = G;
  }
};

// Embedding rows: 4 warps per CTA, each with row buffers in shared memory that it fills with
// bulk asynchronous copies (cp.async.bulk, completion on the warp's mbarrier): the gradient rows
// of a whole tile are in flight at once instead of one dependent 16-byte-per-lane load at a time.
#define TILE_WARPS_EMB 4
#define UPD_WAIT_LIMIT 4000000

// (Embedding rows of up to 256 floats have a kernel of their own, narrow_tile_kernel.)
// The operator rows' slots are staged from GR (dyn_pullback_kernel), eight warps per CTA, four above 1024 floats.
// Resident CTAs per SM: operator rows of up to 256 floats are bound by the latency of a slot's chain of loads, not by bytes,
// and gain from twice the warps (dimension 200, when both kinds of rows had it: update 55.8 -> 52.5 ms per 2.16 M edges); the
// wide rows stay at the register count that keeps them all but free of spills.
template <int VEC, int RULE>
struct TileWarps { enum { N = RULE == RULE_EMB ? TILE_WARPS_EMB : VEC > 8 ? UPD_WARPS / 2 : UPD_WARPS }; };

template <int VEC, int RULE>
__global__ void __launch_bounds__(32 * TileWarps<VEC, RULE>::N, RULE == RULE_EMB ? 3 : VEC == 2 ? 4 : 2)
tile_update_kernel(WaveDims d, WaveBatches wb, WaveBufs w, const unsigned long long *__restrict__ keys,
                   const unsigned int *__restrict__ vals, float lr, float *__restrict__ psum,
                   long long *__restrict__ hublist, int *__restrict__ hubcnt, ParamJob job, int aside) {
  if (RULE == RULE_EMB) pdl_begin_open(has_operator_rows(d) ? (unsigned *)hubcnt + HUB_SEAM_TILE : nullptr);
  else if (!sibling_begin((unsigned *)hubcnt - HUB_REL + HUB_SEAM_TILE)) return;
  constexpr int WARPS = TileWarps<VEC, RULE>::N, STAGE = TILE;
  extern __shared__ __align__(128) float stage_all[];        // [WARPS][STAGE][Dp]
  __shared__ __align__(8) unsigned long long sbar[WARPS];
  const unsigned FULL = 0xffffffffu;
  const unsigned long long SENT = ~0ull;
  int lane = threadIdx.x & 31;
  const int wl = threadIdx.x >> 5;
  if (RULE == RULE_EMB && blockIdx.x < aside) { param_sums(d, wb, w, job, blockIdx.x, stage_all); return; }
  long long t0 = ((long long)(blockIdx.x - aside) * WARPS + wl) * TILE;
  if (t0 >= d.nocc) return;
  float *stage = stage_all + (size_t)wl * STAGE * d.Dp;
  const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&sbar[wl]);
  uint32_t phase = 0;
  int staged_lo = 0, staged_hi = 0;                           // window slots whose rows are in `stage`
  if (lane == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  const int D = d.D;
  const float invD = 1.0f / (float)D;
  const unsigned long long lo = RULE == RULE_EMB ? 0ull : d.key_rel_base;
  const unsigned long long hi = RULE == RULE_EMB ? d.key_rel_base : d.key_invalid;
  long long pa = t0 - 32 + lane, pb = t0 + lane;
  unsigned long long kA = pa >= 0 ? ld_list<RULE>(keys + pa) : SENT;
  unsigned long long kB = pb < d.nocc ? ld_list<RULE>(keys + pb) : SENT;
  unsigned int vB = pb < d.nocc ? ld_list<RULE>(vals + pb) : 0u;
  const int bB = d.bySpb.div((int)vB);              // batch of this lane's slot
  if (__shfl_sync(FULL, kB, TILE - 1) < lo) return;          // tile holds only the other rule's rows
  // Copies the gradient rows of window slots j0 .. j0+cnt-1 (cnt <= STAGE) into the stage buffers and
  // waits for them; the wait is bounded (bit 1 of the error word when it runs out).
  auto stage_rows = [&](int j0, int cnt) {
    __syncwarp();                                            // everyone is done with the old rows
    unsigned int v = __shfl_sync(FULL, vB, j0 + (lane < cnt ? lane : 0));
    if (lane == 0) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"((uint32_t)(cnt * d.D * 4)) : "memory");
    }
    __syncwarp();
    if (lane < cnt) {
      const Occ oc = occ_decode(d, (int)v);
      const float *g;
      if (RULE == RULE_REL) g = w.GR[oc.a == ARR_R1 ? 1 : 0] + ((size_t)oc.blk * d.Pm + oc.r) * d.Dp;
      else {
        const float *gbase = (d.matrix_op && oc.a == ARR_N1) ? w.R2 : w.GX[oc.a];
        g = gbase + ((size_t)oc.blk * w.grows[oc.a] + oc.r) * d.Dp;
      }
      uint32_t dst = (uint32_t)__cvta_generic_to_shared(stage + (size_t)lane * d.Dp);
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   :: "r"(dst), "l"(g), "r"((uint32_t)(d.D * 4)), "r"(bar) : "memory");
    }
    bool done = false;
    for (int it = 0; it < UPD_WAIT_LIMIT && !done; ++it) {
      uint32_t ok;
      asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                   : "=r"(ok) : "r"(bar), "r"(phase) : "memory");
      done = ok != 0;
    }
    if (!done && lane == 0) atomicOr(w.errflag, 2);
    phase ^= 1u;
    staged_lo = j0; staged_hi = j0 + cnt;
  };
  // What the tile's row segments are, from ballots alone: [first, last) are the window slots whose rows this warp reads --
  // without a leading short row that belongs to an earlier tile, and with the rest of a trailing short row that begins here.
  auto segment = [&](int i, unsigned long long key, int &run, bool &hub, bool &head_here) {
    unsigned fm = __ballot_sync(FULL, kB == key);
    unsigned rest = ~(fm >> i);
    run = rest ? __ffs(rest) - 1 : 32 - i;                   // slots i .. i+run-1 of the window share the key
    int back = 0;
    if (i == 0) back = __clz(~__ballot_sync(FULL, kA == key)); // slots of this row just before the tile
    head_here = back == 0;
    hub = i + run >= 32 || back == 32 || back + run > SHORT_MAX;
  };
  int first = __popc(__ballot_sync(FULL, lane < TILE && kB < lo)), last = __popc(__ballot_sync(FULL, lane < TILE && kB < hi));
  if (first >= last) return;
  {
    int run;
    bool hub, head_here;
    if (first == 0) {
      segment(0, __shfl_sync(FULL, kB, 0), run, hub, head_here);
      if (!hub && !head_here) first = run < TILE ? run : TILE;
    }
    if (first >= last) return;
    if (last == TILE) {
      const unsigned long long key = __shfl_sync(FULL, kB, TILE - 1);
      const int start = __ffs(__ballot_sync(FULL, kB == key)) - 1;
      segment(start, key, run, hub, head_here);
      if (!hub && head_here) last = start + run;
    }
  }
  if (RULE == RULE_EMB) {
    // get the rows this tile will need moving towards L2 before the dependent loads start
#pragma unroll
    for (int i = 0; i < TILE; ++i) {
      if (i < first || i >= last) continue;
      unsigned long long key = __shfl_sync(FULL, kB, i);
      int side = (!d.shared_table && key >= (unsigned long long)d.n_rows[0]) ? 1 : 0;
      const float *wr = w.W[side] + (size_t)(side ? key - (unsigned long long)d.n_rows[0] : key) * D;
      for (int f = lane * 32; f < D; f += 1024) asm volatile("prefetch.global.L2 [%0];" :: "l"(wr + f));
    }
  }
  stage_rows(first, last - first < STAGE ? last - first : STAGE);
  int i = first;
  while (i < TILE) {
    unsigned long long key = __shfl_sync(FULL, kB, i);
    if (key >= hi) return;                                   // sorted: nothing of this rule follows
    int run;
    bool hub, head_here;
    segment(i, key, run, hub, head_here);
    int nproc = hub ? (run < TILE - i ? run : TILE - i) : run;
    RowState<VEC, RULE> rs;
    if (!hub) rs.load(d, w, key, lane);
    float4 acc[VEC];
#pragma unroll
    for (int c = 0; c < VEC; ++c) acc[c] = f4zero();
    int cur_b = -1, run_start = 0;
    for (int j = i; j <= i + nproc; ++j) {
      bool in = j < i + nproc;
      const int b = in ? __shfl_sync(FULL, bB, j) : -1;
      if (cur_b >= 0 && b != cur_b) {                                     // a batch of this row is complete
        if (hub) {
          float *dst = psum + (size_t)(t0 + run_start) * d.Dp;
#pragma unroll
          for (int c = 0; c < VEC; ++c) {
            int dd = c * 128 + lane * 4;
            if (dd < D) st4(dst + dd, acc[c]);
          }
        } else {
          rs.step(acc, lr, invD);
        }
#pragma unroll
        for (int c = 0; c < VEC; ++c) acc[c] = f4zero();
      }
      if (!in) break;
      if (b != cur_b) { cur_b = b; run_start = j; }
      if (j >= staged_hi) stage_rows(j, last - j < STAGE ? last - j : STAGE);       // more slots than buffers
      const float *gs = stage + (size_t)(j - staged_lo) * d.Dp;
#pragma unroll
      for (int c = 0; c < VEC; ++c) {
        int dd = c * 128 + lane * 4;
        if (dd < D) acc[c] = acc[c] + ld4(gs + dd);
      }
    }
    if (!hub) rs.store(D, lane);
    else if (head_here && lane == 0) {
      const long long head = t0 + i;
      hublist[atomicAdd(hubcnt, 1)] = head;
      // a row's slots are contiguous in the sorted list: it has HUB_BIG or more of them exactly when the slot
      // HUB_BIG - 1 places after its head still carries its key; those few rows go on a second list
      if (head + HUB_BIG - 1 < (long long)d.nocc && ld_list<RULE>(keys + head + HUB_BIG - 1) == key)
        hub_biglist(hublist, d.nocc)[atomicAdd(hubcnt + 1, 1)] = head;
    }
    i += nproc;
  }
}

// The same for embedding rows of up to 256 floats, two tiles and two rows at a time.  A row of 100 floats is 25 of a warp's 32
// 16-byte lanes, and what the tile kernel executes is mostly not its arithmetic: segment ballots, slot decoding, pointer and
// loop bookkeeping, the sum over the warp, a square root and a division, some 400 instructions for each slot's 100 additions
// (issue slots 58 % busy at 2 % of the DRAM bandwidth, 30 us for 48,000 slots).  Here a half-warp holds a row as NP
// pieces of 64 floats, and the two halves work on two row segments with the same instructions; slots are decoded and segments
// found one per lane, once for both tiles.  Tiles and hubs of such a wave together: 54 us before, 49 so.  Sums keep their
// order: lane l of a half has what lanes l and l + 16 have there.
//
// A segment is what one of the tile kernel's loops handles: a short row that begins in one of the two tiles, with all its
// slots, or the part of a hub row inside one tile.
#define NARROW_WARPS 4
template <int NP> struct NarrowStage { enum { N = NP == 2 ? 16 : 8 }; };
template <int NP>
__global__ void __launch_bounds__(32 * NARROW_WARPS, NP == 2 ? 6 : 4)
narrow_tile_kernel(WaveDims d, WaveBatches wb, WaveBufs w, const unsigned long long *__restrict__ keys, const unsigned int *__restrict__ vals,
                   float lr, float *__restrict__ psum, long long *__restrict__ hublist, int *__restrict__ hubcnt, ParamJob job, int aside) {
  pdl_begin_open(has_operator_rows(d) ? (unsigned *)hubcnt + HUB_SEAM_TILE : nullptr);
  constexpr int NARROW_STAGE = NarrowStage<NP>::N;
  extern __shared__ __align__(128) float stage_all[];        // [NARROW_WARPS][NARROW_STAGE][Dp]
  __shared__ __align__(8) unsigned long long sbar[NARROW_WARPS];
  if (blockIdx.x < aside) { param_sums(d, wb, w, job, blockIdx.x, stage_all); return; }
  const unsigned FULL = 0xffffffffu;
  const unsigned long long SENT = ~0ull;
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5, half = lane >> 4, l16 = lane & 15;
  const int t0 = ((int)(blockIdx.x - aside) * NARROW_WARPS + wl) * 2 * TILE;
  if (t0 >= d.nocc) return;
  float *stage = stage_all + (size_t)wl * NARROW_STAGE * d.Dp;
  const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&sbar[wl]);
  if (lane == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  const int D = d.D;
  const float invD = 1.0f / (float)D;
  // a lane per slot: the window [t0, t0 + 32), and the 32 keys before it
  const unsigned long long kA = t0 - 32 + lane >= 0 ? keys[t0 - 32 + lane] : SENT;
  const unsigned long long kB = t0 + lane < d.nocc ? keys[t0 + lane] : SENT;
  const unsigned int vB = t0 + lane < d.nocc ? vals[t0 + lane] : 0u;
  const unsigned same = __match_any_sync(FULL, kB);          // equal keys are neighbours
  const int row0 = __ffs(same) - 1, row_end = 32 - __clz(same);
  const int back = __clz(~__ballot_sync(FULL, kA == __shfl_sync(FULL, kB, 0)));      // slots of the window's first row before it
  const bool begins = row0 == lane && (lane > 0 || back == 0);
  const bool hub = row_end - row0 + (row0 == 0 ? back : 0) > SHORT_MAX;              // (a row that leaves the window has 25 and more slots in it)
  const bool starts = lane < 2 * TILE && kB < d.key_rel_base && (begins || (hub && (lane & (TILE - 1)) == 0));
  int count = row_end - lane;                                // slots of the segment that starts here
  if (hub && count > TILE - (lane & (TILE - 1))) count = TILE - (lane & (TILE - 1));
  unsigned rest = __ballot_sync(FULL, starts);
  if (rest == 0) return;
  const int first = __ffs(rest) - 1;
  const int last = __reduce_max_sync(FULL, starts ? lane + count : 0);
  const int staged = last - first < NARROW_STAGE ? last - first : NARROW_STAGE;
  const int attr = count | (hub ? 64 : 0) | (begins ? 128 : 0);
  // gradient rows: into shared memory by bulk copies, all in flight together; what finds no room is read where it lies
  const float *src = nullptr;
  int bB = 0;
  if (lane >= first && lane < last) {
    const Occ oc = occ_decode(d, (int)vB);
    const float *gbase = (d.matrix_op && oc.a == ARR_N1) ? w.R2 : w.GX[oc.a];
    src = gbase + ((size_t)oc.blk * w.grows[oc.a] + oc.r) * d.Dp;
    bB = d.bySpb.div((int)vB);
  }
  if (lane == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"((uint32_t)(staged * D * 4)) : "memory");
  __syncwarp();
  if (lane >= first && lane < first + staged) {
    float *to = stage + (size_t)(lane - first) * d.Dp;
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"((uint32_t)__cvta_generic_to_shared(to)), "l"(src), "r"((uint32_t)(D * 4)), "r"(bar) : "memory");
    src = to;
  }
  // where the rows of the short segments are; each lane of a segment's half, a few of a slot's for the prefetch
  auto place = [&](unsigned long long key, float *&prow, float *&pacc) {
    const int side = (!d.shared_table && key >= (unsigned long long)d.n_rows[0]) ? 1 : 0;
    const size_t row = (size_t)(side ? key - (unsigned long long)d.n_rows[0] : key);
    prow = w.W[side] + row * D;
    pacc = w.G[side] + row;
  };
  {
    const int slot = lane >> 2;                              // 2 * TILE slots x four 128-byte lines at a time
    const unsigned long long key = __shfl_sync(FULL, kB, slot);
    const int a = __shfl_sync(FULL, starts ? attr : 64, slot);
    if (!(a & 64)) {
      float *prow, *pacc;
      place(key, prow, pacc);
      for (int f = (lane & 3) * 32; f < D; f += 128) asm volatile("prefetch.global.L2 [%0];" :: "l"(prow + f));
    }
  }
  bool ok[NP];
#pragma unroll
  for (int c = 0; c < NP; ++c) ok[c] = c * 64 + l16 * 4 < D;
  // |x|^2 of a half's row, summed as the tile kernel's warp does
  auto square = [&](const float4 (&x)[NP]) {
    float even = f4dot(x[0], x[0]), odd = f4dot(x[1], x[1]);
#pragma unroll
    for (int c = 2; c < NP; c += 2) { even += f4dot(x[c], x[c]); odd += f4dot(x[c + 1], x[c + 1]); }
    float ss = even + odd;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(FULL, ss, o);
    return ss;
  };
  float4 nv[NP];
  float nG;
  float *nrow, *nacc;
  int nstart, nattr;
  auto next = [&]() {                                        // the next two segments, one a half; their rows requested
    const int a = __ffs(rest) - 1;
    rest &= rest - 1;
    const int b = __ffs(rest) - 1;
    rest &= rest - 1;
    nstart = half ? b : a;                                   // -1: none
    const int at = nstart < 0 ? 0 : nstart;
    const unsigned long long key = __shfl_sync(FULL, kB, at);
    nattr = __shfl_sync(FULL, attr, at);
    if (nstart < 0) nattr = 64;
    nG = 0.f;
    nrow = nacc = nullptr;
#pragma unroll
    for (int c = 0; c < NP; ++c) nv[c] = f4zero();
    if (!(nattr & 64)) {
      place(key, nrow, nacc);
#pragma unroll
      for (int c = 0; c < NP; ++c) if (ok[c]) nv[c] = ld4(nrow + c * 64 + l16 * 4);
      nG = *nacc;
    }
  };
  next();
  {
    bool done = false;
    for (int it = 0; it < UPD_WAIT_LIMIT && !done; ++it) {
      uint32_t ok;
      asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(bar), "r"(0u) : "memory");
      done = ok != 0;
    }
    if (!done && lane == 0) atomicOr(w.errflag, 2);
  }
  __syncwarp();
  for (bool more = true; more;) {
    float4 v[NP], acc[NP];
#pragma unroll
    for (int c = 0; c < NP; ++c) { v[c] = nv[c]; acc[c] = f4zero(); }
    float G = nG;
    float *prow = nrow, *pacc = nacc;
    const int start = nstart, n = nattr & 63;
    const bool is_hub = nattr & 64, head = nattr & 128;
    more = rest != 0;
    if (more) next();
    if (d.max_norm > 0.f) {                                  // as RowState::load
      const float ss = square(v);
      const float norm = sqrtf(ss);
      if (norm > d.max_norm) {
        const float sc = d.max_norm / (norm + 1e-7f);
#pragma unroll
        for (int c = 0; c < NP; ++c) v[c] = v[c] * sc;
      }
    }
    // A slot each, as for most rows of a wave: no loop over batches (update class of the plumbing bucket 3.55 -> 3.48 ms).
    if (__all_sync(FULL, n == 1 && !is_hub)) {
      const float *g = (const float *)__shfl_sync(FULL, (unsigned long long)src, start);
#pragma unroll
      for (int c = 0; c < NP; ++c) if (ok[c]) acc[c] = acc[c] + ld4(g + c * 64 + l16 * 4);
      G += square(acc) * invD;
      const float stepv = lr / (sqrtf(G) + PBG_ADAGRAD_EPS);
#pragma unroll
      for (int c = 0; c < NP; ++c) if (ok[c]) st4(prow + c * 64 + l16 * 4, v[c] - acc[c] * stepv);
      if (l16 == 0) *pacc = G;
      continue;
    }
    const int other = __shfl_xor_sync(FULL, n, 16), most = n > other ? n : other;
    int cur = -1, run_start = 0;
    for (int j = 0; j <= most; ++j) {
      const int at = (start + j) & 31;
      const int bs = __shfl_sync(FULL, bB, at);
      const float *g = (const float *)__shfl_sync(FULL, (unsigned long long)src, at);
      const int b = j < n ? bs : -1;
      const bool flush = j <= n && cur >= 0 && b != cur;     // a batch of this row is complete
      if (__any_sync(FULL, flush && !is_hub)) {
        const float ss = square(acc);
        if (flush && !is_hub) {
          G += ss * invD;
          const float stepv = lr / (sqrtf(G) + PBG_ADAGRAD_EPS);
#pragma unroll
          for (int c = 0; c < NP; ++c) v[c] = v[c] - acc[c] * stepv;
        }
      }
      if (flush && is_hub) {
        float *dst = psum + (size_t)(t0 + run_start) * d.Dp;
#pragma unroll
        for (int c = 0; c < NP; ++c) if (ok[c]) st4(dst + c * 64 + l16 * 4, acc[c]);
      }
      if (flush) {
#pragma unroll
        for (int c = 0; c < NP; ++c) acc[c] = f4zero();
      }
      if (j < n) {
        if (b != cur) { cur = b; run_start = start + j; }
#pragma unroll
        for (int c = 0; c < NP; ++c) if (ok[c]) acc[c] = acc[c] + ld4(g + c * 64 + l16 * 4);
      }
    }
    if (start >= 0 && !is_hub) {
#pragma unroll
      for (int c = 0; c < NP; ++c) if (ok[c]) st4(prow + c * 64 + l16 * 4, v[c]);
      if (l16 == 0) *pacc = G;
    } else if (start >= 0 && head && l16 == 0) {
      const long long at = t0 + start;
      hublist[atomicAdd(hubcnt, 1)] = at;
      // (big rows: see the tile kernel)
      if (at + HUB_BIG - 1 < (long long)d.nocc && keys[at + HUB_BIG - 1] == keys[at]) hub_biglist(hublist, d.nocc)[atomicAdd(hubcnt + 1, 1)] = at;
    }
  }
}

// First slot of batch b, and first of a later batch, among the slots of the row `key` that starts at head: two such searches in
// the same rounds.  Row and batch are ascending along the list, so "still in the row and below b" and "still in the row and
// not above b" hold on prefixes; the first round probes the same positions for both.  (Three searches one after the other -- the
// row's end, then the batch in it -- were six rounds of a load and a barrier, of about 1,000 cycles each: hub kernel and all of a
// plumbing wave 115.3 -> 114.5 us.)
template <class Key, class Batch>
__device__ __forceinline__ void coop_batch_range(const unsigned long long *keys, const unsigned int *vals, long long head, long long end, unsigned long long key, int b,
                                                 Key &&key_at, Batch &&batch_at, long long &q, long long &eb) {
  long long lo[2] = {head, head}, hi[2] = {end, end};
  bool same = true;                                          // both ranges are the same so far: one probe serves both
  while (lo[0] < hi[0] || lo[1] < hi[1]) {
    long long stride[2];
    int in[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      stride[u] = (hi[u] - lo[u] + blockDim.x - 1) / blockDim.x;
      const long long pos = lo[u] + (long long)threadIdx.x * stride[u];
      if (u == 0 || !same) {
        in[u] = -1;
        if (pos < hi[u] && key_at(keys + pos) == key) in[u] = batch_at(vals + pos);
        else if (pos < hi[u]) in[u] = PBG_KMAX;              // behind the row
      } else in[1] = in[0];
    }
    const int cnt[2] = {__syncthreads_count(in[0] >= 0 && in[0] < b), __syncthreads_count(in[1] >= 0 && in[1] <= b)};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (lo[u] >= hi[u]) continue;
      if (cnt[u] == 0) { hi[u] = lo[u]; continue; }
      const long long nhi = lo[u] + (long long)cnt[u] * stride[u];
      lo[u] += (long long)(cnt[u] - 1) * stride[u] + 1;
      if (nhi < hi[u]) hi[u] = nhi;
      if (stride[u] == 1) lo[u] = hi[u];
    }
    same = same && lo[0] == lo[1] && hi[0] == hi[1];
  }
  q = hi[0];
  eb = hi[1];
}

// Per-batch Stats (train_cpu.py:95-101) of batch b of the wave, summed by one CTA in a fixed order; the running totals
// live in `sum` (loss, violators_lhs, violators_rhs, count, reg).  The first k CTAs of the embedding rows'
// hub_kernel do this: as a kernel of its own it was 5 to 29 us per wave of one CTA per batch, and a launch.
__device__ __forceinline__ void batch_stats(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, int b, pbg_batch_stats *per_batch, double *sum) {
  __shared__ double sl[UPD_WARPS], sr[UPD_WARPS];
  __shared__ long long sv0[UPD_WARPS], sv1[UPD_WARPS];
  const int t = threadIdx.x, lane = t & 31;
  double l = 0.0, rg = 0.0;
  long long v0 = 0, v1 = 0;
  const int rows = d.Cm * d.Pm;
  const int lim = d.batch_negs ? d.num_batch_negs : d.U, nb = wb.n[b], Pl = nb < lim ? nb : lim;
#pragma unroll 4
  for (int r = t; r < rows; r += blockDim.x) {
    const int c = d.byPm.div(r), i = r - c * d.Pm;
    if (i >= Pl || c * Pl + i >= nb) continue;
    const size_t prow = (size_t)b * rows + r;
    l += (double)w.lossrow[0][prow] + (double)w.lossrow[1][prow];
    if (d.reg_coef != 0.f) rg += (double)w.regrow[prow];
    v0 += w.violrow[0][prow];
    v1 += w.violrow[1][prow];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, o); rg += __shfl_xor_sync(0xffffffffu, rg, o);
    v0 += __shfl_xor_sync(0xffffffffu, v0, o); v1 += __shfl_xor_sync(0xffffffffu, v1, o);
  }
  if (lane == 0) { sl[t >> 5] = l; sr[t >> 5] = rg; sv0[t >> 5] = v0; sv1[t >> 5] = v1; }
  __syncthreads();
  if (t == 0) {
    for (int u = 1; u < UPD_WARPS; ++u) { l += sl[u]; rg += sr[u]; v0 += sv0[u]; v1 += sv1[u]; }
    pbg_batch_stats s;
    s.loss = (float)l; s.reg = (float)rg; s.violators_lhs = v0; s.violators_rhs = v1; s.count = nb;
    if (per_batch) per_batch[wb.gidx[b]] = s;
    atomicAdd(&sum[0], l);
    atomicAdd(&sum[1], (double)v0);
    atomicAdd(&sum[2], (double)v1);
    atomicAdd(&sum[3], (double)nb);
    atomicAdd(&sum[4], rg);
  }
}

// What is left after the tiles: the hub rows, and (aside) the work that rides along.
//
// A hub row's slots [head, end) are in batch order; the tile warps have summed them in runs that start at a batch's first
// slot q and at every multiple of TILE inside the batch.  One CTA finishes a row: a probe per thread over its first 256
// slots gives, in a single round of loads, the row's end and where each of its batches starts; warp w adds up the
// partial rows of batches w, w + 8, ... into tot[batch][] and, for embedding rows, takes the batch's squared norm while it
// has the sum in registers; then the optimizer steps are taken in batch order.
//
// The few rows that collect 256 and more slots per wave (the top nodes of a power-law partition) would keep one CTA busy
// long after every other row is done.  For them one CTA per (row, batch) adds that batch's partial rows up first -- warp w
// takes runs w, w + 8, ..., the eight sums are added in warp order -- leaves the total in the batch's first partial row and
// the batch's start in the row's line of bigtab, and the CTA that finds itself the last of the row's batches finishes the
// row.  (A kernel for the sums and one for the rows cost a launch and 9 us more per wave of 56,000 slots at dimension
// 100: the second waited for the longest search of the first.)  All sums run in a fixed order.
template <int VEC, int RULE>
__global__ void __launch_bounds__(32 * UPD_WARPS)
hub_kernel(WaveDims d, WaveBatches wb, WaveBufs w, const unsigned long long *__restrict__ keys, const unsigned int *__restrict__ vals, float lr,
           float *psum, const long long *__restrict__ hublist, const int *__restrict__ hubcnt, int *__restrict__ hubcnt_next,
           long long *bigtab, int aside, ParamJob job, pbg_batch_stats *per_batch, double *sum) {
  if (RULE == RULE_EMB) pdl_begin_open(has_operator_rows(d) ? (unsigned *)hubcnt + HUB_SEAM_HUB : nullptr);
  else if (!sibling_begin((unsigned *)hubcnt - HUB_REL + HUB_SEAM_HUB)) return;
  static_assert(32 * UPD_WARPS == HUB_BIG, "one probe per thread covers exactly the rows that are not big");
  extern __shared__ __align__(16) float tot[];               // [k][VEC * 128]; sums of a big row's batch: [UPD_WARPS][VEC * 128]
  __shared__ long long bstart[PBG_KMAX + 1];
  __shared__ float bnorm[PBG_KMAX];                           // mean squared gradient of a batch (embedding rows)
  __shared__ int sbatch[32 * UPD_WARPS];
  __shared__ unsigned long long skey;
  __shared__ bool closing;
  if (blockIdx.x == 0 && threadIdx.x < 2) hubcnt_next[threadIdx.x] = 0;      // its last reader is behind us in the stream
  // the first CTAs of the embedding rows' launch (aside) have other work
  int cta0 = 0;
  if (RULE == RULE_EMB && aside) {
    cta0 = d.k + job.steps * ((d.D + 31) / 32);               // param_step_ctas
    if (blockIdx.x < d.k) { batch_stats(d, wb, w, blockIdx.x, per_batch, sum); return; }
    if (blockIdx.x < cta0) { param_step(d, wb, w, job, blockIdx.x - d.k, tot); return; }
  }
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int D = d.D;
  const float invD = 1.0f / (float)D;
  const int nh = ld_list<RULE>(hubcnt), nbig = ld_list<RULE>(hubcnt + 1);                 // the tile kernel listed the rows
  const long long *biglist = hub_biglist(hublist, d.nocc);
  // the batches of the big rows first, then the list of all hub rows, big ones skipped
  const int ctas = (int)gridDim.x - (RULE == RULE_REL) - cta0, items = nbig * d.k + nh;
  for (int item = blockIdx.x - cta0; item < items; item += ctas) {
    const bool from_big = item < nbig * d.k;
    const int h = item / d.k;
    const long long head = ld_list<RULE>(from_big ? biglist + h : hublist + (item - nbig * d.k));
    long long *line = bigtab + (size_t)h * BIGTAB_LINE;       // [b] first slot of batch b or -1; last: a counter
    if (from_big) {
      const int b = item - h * d.k;
      const unsigned long long key = ld_list<RULE>(keys + head);
      // where batch b starts and ends inside the row (both right behind it where it has no slot there)
      long long q, eb;
      coop_batch_range(keys, vals, head, (long long)d.nocc, key, b, [&](const unsigned long long *p) { return ld_list<RULE>(p); },
                       [&](const unsigned int *p) { return d.bySpb.div((int)ld_list<RULE>(p)); }, q, eb);
      const long long ftb = (q / TILE + 1) * TILE;
      const long long nruns = q < eb ? 1 + (eb > ftb ? (eb - 1 - ftb) / TILE + 1 : 0) : 0;
      if (nruns > 1) {
        float4 acc[VEC];
#pragma unroll
        for (int c = 0; c < VEC; ++c) acc[c] = f4zero();
        // four of the warp's partial rows in flight at a time, added in run order
        for (long long r0 = wl; r0 < nruns; r0 += 4 * UPD_WARPS) {
          const float *src[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            long long r = r0 + (long long)u * UPD_WARPS;
            src[u] = r < nruns ? psum + (size_t)(r == 0 ? q : ftb + (r - 1) * TILE) * d.Dp : nullptr;
          }
#pragma unroll
          for (int c = 0; c < VEC; ++c) {
            int dd = c * 128 + lane * 4;
            if (dd < D) {
              float4 v[4];
#pragma unroll
              for (int u = 0; u < 4; ++u) v[u] = src[u] ? ld4(src[u] + dd) : f4zero();
#pragma unroll
              for (int u = 0; u < 4; ++u) acc[c] = acc[c] + v[u];
            }
          }
        }
#pragma unroll
        for (int c = 0; c < VEC; ++c) st4(&tot[(size_t)wl * VEC * 128 + c * 128 + lane * 4], acc[c]);
        __syncthreads();
        float *dst = psum + (size_t)q * d.Dp;
        for (int dd = threadIdx.x * 4; dd < D; dd += 4 * blockDim.x) {
          float4 t = ld4(&tot[dd]);
#pragma unroll
          for (int u = 1; u < UPD_WARPS; ++u) t = t + ld4(&tot[(size_t)u * VEC * 128 + dd]);
          st4(dst + dd, t);
        }
      }
      if (threadIdx.x == 0) line[b] = q < eb ? q : -1;
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) closing = atomicAdd((unsigned long long *)&line[PBG_KMAX], 1ull) == (unsigned long long)(d.k - 1);
      __syncthreads();
      if (!closing) continue;                                 // another batch of the row is still being summed
      __threadfence();
      if (threadIdx.x == 0) line[PBG_KMAX] = 0;           // for the next wave
    }
    const long long p = head + threadIdx.x;
    const unsigned long long kp = p < (long long)d.nocc ? ld_list<RULE>(keys + p) : ~0ull;
    const int bp = p < (long long)d.nocc ? d.bySpb.div((int)ld_list<RULE>(vals + p)) : -1;
    // what the CTAs of a big row's batches left (past L1: this CTA may have read the lines before)
    const long long tabv = from_big && threadIdx.x < PBG_KMAX ? __ldcg(line + threadIdx.x) : -1;
    if (threadIdx.x == 0) skey = kp;
    for (int i = threadIdx.x; i <= PBG_KMAX; i += blockDim.x) bstart[i] = -1;
    __syncthreads();
    const unsigned long long key = skey;
    const bool in = kp == key;
    sbatch[threadIdx.x] = in ? bp : -1;
    if (wl == 0) {
      // the row these steps start from: on its way to L2 while the sums are made
      RowState<VEC, RULE> where;
      where.locate(d, w, key);
      for (int f = lane * 32; f < D; f += 1024) {
        asm volatile("prefetch.global.L2 [%0];" :: "l"(where.prow + f));
        if (RULE == RULE_REL) asm volatile("prefetch.global.L2 [%0];" :: "l"(where.pacc + f));
      }
    }
    const int cnt = __syncthreads_count(in);                  // slots of the row among the first 256 (they are contiguous)
    const bool big = cnt == (int)blockDim.x;                  // one row per batch is left of it
    if (big && !from_big) continue;                           // taken from the list of big rows
    const long long end = head + cnt;                         // (not of a big row: it has one partial row per batch)
    if (!big) {
      if (in && (threadIdx.x == 0 || sbatch[threadIdx.x - 1] != bp)) bstart[bp] = p;     // first slot of batch bp
    } else {
      if (threadIdx.x < d.k) bstart[threadIdx.x] = tabv;
    }
    __syncthreads();
    // ---- per-batch totals ----
    for (int bq = wl; bq < d.k; bq += UPD_WARPS) {
      long long q = bstart[bq];
      if (q < 0) continue;
      long long eb = end;
      for (int nb = bq + 1; nb < d.k; ++nb) if (bstart[nb] >= 0) { eb = bstart[nb]; break; }
      long long ftb = (q / TILE + 1) * TILE;
      long long nruns = big ? 1 : 1 + (eb > ftb ? (eb - 1 - ftb) / TILE + 1 : 0);
      float4 acc[VEC];
#pragma unroll
      for (int c = 0; c < VEC; ++c) acc[c] = f4zero();
      // four partial rows in flight at a time; they are still added in run order
      for (long long r0 = 0; r0 < nruns; r0 += 4) {
        const float *src[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          long long r = r0 + u;
          long long start = r == 0 ? q : ftb + (r - 1) * TILE;
          src[u] = r < nruns ? psum + (size_t)start * d.Dp : nullptr;
        }
#pragma unroll
        for (int c = 0; c < VEC; ++c) {
          int dd = c * 128 + lane * 4;
          if (dd < D) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = src[u] ? (big ? __ldcg((const float4 *)(src[u] + dd)) : ld4(src[u] + dd)) : f4zero();
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[c] = acc[c] + v[u];
          }
        }
      }
#pragma unroll
      for (int c = 0; c < VEC; ++c) st4(&tot[(size_t)bq * VEC * 128 + c * 128 + lane * 4], acc[c]);
      if (RULE == RULE_EMB) {
        // the same expression, on the same values, as RowState::step evaluates
        float ss = 0.f;
#pragma unroll
        for (int c = 0; c < VEC; ++c) ss += f4dot_yx(acc[c], acc[c]);
        ss = warp_sum(ss);
        if (lane == 0) bnorm[bq] = __fmul_rn(ss, invD);
      }
    }
    __syncthreads();
    // ---- optimizer steps in batch order ----
    // Every thread steps four columns of the row through all batches (the batch norms are known, so nothing in a
    // step crosses columns): the same arithmetic per element, in the same order, as one warp stepping whole rows --
    // which took eight times as long, one dependent instruction stream of a lone warp.  (A row that max_norm has to
    // rescale first needs its norm: that case keeps the one-warp form.)
    // With more hub rows than CTAs (a small graph, where every row is one) the kernel is bound by the instructions it
    // executes, not by one row's chain, and the one-warp form executes fewer.
    if ((RULE == RULE_EMB && d.max_norm > 0.f) || items > ctas) {
      if (wl == 0) {
        RowState<VEC, RULE> rs;
        rs.load(d, w, key, lane);
        for (int bq = 0; bq < d.k; ++bq) {
          if (bstart[bq] < 0) continue;
          float4 g[VEC];
#pragma unroll
          for (int c = 0; c < VEC; ++c) g[c] = ld4(&tot[(size_t)bq * VEC * 128 + c * 128 + lane * 4]);
          if (RULE == RULE_EMB) rs.step_with_norm(g, lr, bnorm[bq]);
          else rs.step(g, lr, invD);
        }
        rs.store(D, lane);
      }
    } else {
      RowState<VEC, RULE> where;
      where.locate(d, w, key);
      const float G0 = RULE == RULE_EMB ? *where.pacc : 0.f;
      float Gl = G0;
      for (int dd = threadIdx.x * 4; dd < D; dd += 4 * blockDim.x) {
        float4 v = ld4(where.prow + dd), a = f4zero();
        if (RULE == RULE_REL) a = ld4(where.pacc + dd);
        Gl = G0;
        for (int bq = 0; bq < d.k; ++bq) {
          if (bstart[bq] < 0) continue;
          const float4 g = ld4(&tot[(size_t)bq * VEC * 128 + dd]);
          if (RULE == RULE_EMB) {
            Gl += bnorm[bq];
            const float stepv = lr / (sqrtf(Gl) + PBG_ADAGRAD_EPS);
            v = v - g * stepv;
          } else {
            a = a + g * g;
            v.x -= lr * g.x / (sqrtf(a.x) + PBG_ADAGRAD_EPS);
            v.y -= lr * g.y / (sqrtf(a.y) + PBG_ADAGRAD_EPS);
            v.z -= lr * g.z / (sqrtf(a.z) + PBG_ADAGRAD_EPS);
            v.w -= lr * g.w / (sqrtf(a.w) + PBG_ADAGRAD_EPS);
          }
        }
        st4(where.prow + dd, v);
        if (RULE == RULE_REL) st4(where.pacc + dd, a);
      }
      if (RULE == RULE_EMB && threadIdx.x == 0) {
        // (thread 0 owns columns 0..3 of every row, so its Gl went through all batches)
        *where.pacc = Gl;
      }
    }
    __syncthreads();
  }
}

// linear / affine operators: turns GN1 rows (gradient w.r.t. the prepared operand) into the
// gradient w.r.t. the operator output, in place; slots without a row get zeros.  The two
// contractions of launch_matrix_backward read the result.
template <int VEC, int CK>
__global__ void __launch_bounds__(32 * UPD_WARPS) gz_rows_kernel(WaveDims d, WaveBatches wb, WaveBufs w) {
  pdl_begin();
  int lane = threadIdx.x & 31;
  const int item = (int)blockIdx.x * UPD_WARPS + (int)(threadIdx.x >> 5);
  if (item >= d.nblk * d.Mm) return;
  const int lb = d.byMm.div(item), r = item - lb * d.Mm;
  const int blk = d.blk0 + lb;
  BlockInfo bi = block_info(d, wb, blk);
  const int D = d.D;
  float *row = w.GX[ARR_N1] + ((size_t)blk * d.Mm + r) * d.Dp;
  long long id = slot_row(d, wb, w, bi, 1, r);
  float4 v[VEC];
  if (id < 0 || id >= d.n_rows[1]) {
#pragma unroll
    for (int c = 0; c < VEC; ++c) v[c] = f4zero();
  } else {
    gz_row<VEC, CK>(v, d, w, ARR_N1, blk, r, lane, false);
  }
  __syncwarp();
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    int dd = c * 128 + lane * 4;
    if (dd < D) st4(row + dd, v[c]);
  }
}

static inline int comparator_kind(const WaveDims &d) { return d.cmp >= PBG_CMP_L2 ? CK_L2 : d.cmp == PBG_CMP_COS ? CK_COS : CK_DOT; }
// KERNEL<VEC, CK> with the row width and comparator of the wave
#define PBG_ROWS_CK(VEC, KERNEL, ...)                                        \
  do {                                                                       \
    const int ck_ = comparator_kind(d);                                      \
    if (ck_ == CK_DOT) pbg_launch(KERNEL<VEC, CK_DOT>, __VA_ARGS__);         \
    else if (ck_ == CK_COS) pbg_launch(KERNEL<VEC, CK_COS>, __VA_ARGS__);    \
    else pbg_launch(KERNEL<VEC, CK_L2>, __VA_ARGS__);                        \
  } while (0)

int launch_gz_rows(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, cudaStream_t st) {
  long long items = (long long)d.nblk * d.Mm;
  int ctas = (int)((items + UPD_WARPS - 1) / UPD_WARPS);
  int vec = (d.D + 127) / 128;
#define GZ(V) PBG_ROWS_CK(V, gz_rows_kernel, ctas, 32 * UPD_WARPS, 0, st, d, wb, w)
  if (vec <= 1) GZ(1); else if (vec <= 2) GZ(2); else if (vec <= 4) GZ(4); else if (vec <= 8) GZ(8); else GZ(16);
#undef GZ
  return 1;
}

// AsyncAdagrad on the matrix (and translation) of the batch's relation, batch by batch
// (async_adagrad.py:75-85).  dA[b] comes from launch_matrix_backward; the gradient of an affine
// translation is the column sum of the batch's GN1 rows.
__global__ void relupdate_matrix_kernel(WaveDims d, WaveBatches wb, WaveBufs w, float lr) {
  pdl_begin();
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.opw) return;
  const long long DD = (long long)d.D * d.D;
  for (int b = 0; b < d.k; ++b) {
    if (wb.n[b] <= 0) continue;
    int rl = wb.rel[b];
    if (rl < 0 || rl >= d.num_rels) continue;
    float g;
    if (e < DD) g = w.dA[(size_t)b * d.opw + e];
    else {
      int dd = (int)(e - DD);
      g = 0.f;
      const float *rows = w.GX[ARR_N1] + (size_t)b * d.Cm * d.Mm * d.Dp + dd;
      for (int r = 0; r < d.Cm * d.Mm; ++r) g += rows[(size_t)r * d.Dp];
    }
    size_t idx = (size_t)rl * d.opw + e;
    float a = w.acc[0][idx] + g * g;
    w.acc[0][idx] = a;
    w.theta[0][idx] -= lr * g / (sqrtf(a) + PBG_ADAGRAD_EPS);
  }
}

int launch_matrix_update(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, float lr, cudaStream_t st) {
  pbg_launch(relupdate_matrix_kernel, (d.opw + 255) / 256, 256, 0, st, d, wb, w, lr);
  return 1;
}

// Dynamic relations: the pull-back, one warp per slot -- the gradient of the table row written over the slot's own
// gradient row, and for the slots that went through an operator the gradient of the edge's operator row into GR -- so
// that both sorted, row-by-row update kernels only add rows.  first_q: the slots of N0 and N1 are left out (dot
// comparator, no regularizer: what they hold is the row's gradient already; on a dimension-400 graph of 1000-row chunks
// they are half of the slots).
template <int VEC, int CK>
__global__ void __launch_bounds__(32 * UPD_WARPS, VEC <= 4 ? 4 : 1) dyn_pullback_kernel(WaveDims d, WaveBatches wb, WaveBufs w, int first_q) {
  pdl_begin();
  extern __shared__ __align__(16) float wpart[];             // [UPD_WARPS][VEC * 128]
  const int wl = threadIdx.x >> 5;
  const int nN = d.nblk * d.Mm, nQ = d.nblk * d.Pm;
  int item = (int)blockIdx.x * UPD_WARPS + wl + (first_q ? 2 * nN : 0);
  if (item >= 2 * nN + 2 * nQ) return;
  int a;
  if (item < nN) a = ARR_N0;
  else if ((item -= nN) < nN) a = ARR_N1;
  else if ((item -= nN) < nQ) a = ARR_Q0;
  else { item -= nQ; a = ARR_Q1; }
  const int rows = a <= ARR_N1 ? d.Mm : d.Pm, lb = a <= ARR_N1 ? d.byMm.div(item) : d.byPm.div(item);
  const int blk = d.blk0 + lb, r = item - lb * rows, lane = threadIdx.x & 31, side = slot_side(a);
  const BlockInfo bi = block_info(d, wb, blk);
  if (bi.n <= 0 || (a >= ARR_Q0 && r >= bi.n)) return;
  const long long id = slot_row(d, wb, w, bi, side, r);
  if (id < 0 || id >= d.n_rows[side]) { dyn_pullback_empty<VEC>(d, w, a, blk, r, lane); return; }
  float4 v[VEC];
  gz_row<VEC, CK>(v, d, w, a, blk, r, lane, d.reg_coef != 0.f && r < bi.n && r < d.Pm);    // (regularized: the chunk's edges in every operand array)
  dyn_pullback_finish<VEC, CK>(v, d, w, a, bi, blk, r, lane, wpart + (size_t)wl * VEC * 128);
}

// The pull-back of a wave (what is left to do depends on the comparator, the operator and the options) and the job it
// leaves for param_step.
template <int VEC>
static int launch_pullback(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, float rel_lr, ParamJob &job, cudaStream_t st) {
  const size_t smem = (size_t)UPD_WARPS * VEC * 128 * sizeof(float);
  const bool has_op = d.op != PBG_OP_NONE && w.theta[0] != nullptr;
  const bool rows_change = d.cmp != PBG_CMP_DOT || d.reg_coef != 0.f;
  pbg_opt_in_smem((const void *)std_pullback_kernel<VEC, CK_DOT>, (int)smem);
  pbg_opt_in_smem((const void *)std_pullback_kernel<VEC, CK_COS>, (int)smem);
  pbg_opt_in_smem((const void *)std_pullback_kernel<VEC, CK_L2>, (int)smem);
  pbg_opt_in_smem((const void *)dyn_pullback_kernel<VEC, CK_DOT>, (int)smem);
  pbg_opt_in_smem((const void *)dyn_pullback_kernel<VEC, CK_COS>, (int)smem);
  pbg_opt_in_smem((const void *)dyn_pullback_kernel<VEC, CK_L2>, (int)smem);
  job.sums = job.steps = job.cleared0 = job.cleared1 = 0; job.lr = rel_lr;
  if (d.dynamic) {
    if (d.pulled_back || (!rows_change && !has_op)) return 0;
    const int first_q = rows_change ? 0 : 1;
    const long long rows = 2ll * d.nblk * d.Pm + (first_q ? 0 : 2ll * d.nblk * d.Mm);
    PBG_ROWS_CK(VEC, dyn_pullback_kernel, (unsigned)((rows + UPD_WARPS - 1) / UPD_WARPS), 32 * UPD_WARPS, smem, st, d, wb, w, first_q);
    return 1;
  }
  const bool row_op = has_op && !d.matrix_op;
  if (row_op) { job.sum_kind[job.sums++] = 0; job.step_kind[job.steps++] = 0; }
  if (w.glob[0]) { job.sum_kind[job.sums++] = 1; job.step_kind[job.steps++] = 1; }
  if (w.glob[1]) {
    job.sum_kind[job.sums++] = 2;
    if (!w.glob_shared) job.step_kind[job.steps++] = 2;
  }
  if (!rows_change && !(row_op && w.PG)) return 0;
  job.cleared0 = rows_change; job.cleared1 = 1;
  if (d.pulled_back) return 0;
  const dim3 grid((unsigned)(((long long)d.nblk * d.Mm + UPD_WARPS - 1) / UPD_WARPS), rows_change ? 2 : 1);
  PBG_ROWS_CK(VEC, std_pullback_kernel, grid, 32 * UPD_WARPS, smem, st, d, wb, w, rows_change ? 0 : 1);
  return 1;
}

template <int VEC>
static int launch_update_vec(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w,
                             const unsigned long long *keys, const unsigned int *vals, float lr, float rel_lr,
                             const UpdateScratch &us, cudaStream_t st) {
  constexpr int REL_WARPS = TileWarps<VEC, RULE_REL>::N;
  const long long tiles = ((long long)d.nocc + TILE - 1) / TILE;
  const int hub_ctas = 592;     // (half and twice as many measured the same: the kernel takes as long as its longest row)
  // per-batch totals of one hub row, or eight partial sums of one batch of a big row
  const size_t hub_smem = (size_t)(d.k > UPD_WARPS ? d.k : UPD_WARPS) * VEC * 128 * sizeof(float);
  static_assert(PBG_KMAX * 32 <= UPD_WARPS * 128, "param_step works in the same shared memory");
  // the attribute is set once for the largest wave this row width allows in 227 KB
  size_t hub_smem_max = (size_t)PBG_KMAX * VEC * 128 * sizeof(float);
  if (hub_smem_max > 222 * 1024) hub_smem_max = 222 * 1024;    // of 227 KB: the kernel has up to 5 KB of static shared memory
  // per device (a process may hold contexts on several GPUs); a failed opt-in makes the launch fail,
  // which the caller's cudaGetLastError reports
  pbg_opt_in_smem((const void *)hub_kernel<VEC, RULE_EMB>, (int)hub_smem_max);
  ParamJob job;
  int launches = launch_pullback<VEC>(d, wb, w, rel_lr, job, st);
  int *hubcnt = us.hubcnt + HUB_SET * (*us.turn & 1), *hubcnt_next = us.hubcnt + HUB_SET * ((*us.turn + 1) & 1);
  ++*us.turn;
  const int sum_ctas = param_sum_ctas(d, job);
  if (VEC <= 2) {
    constexpr int NP = VEC == 1 ? 2 : 4, STAGE = NarrowStage<NP>::N;
    const size_t smem = (size_t)NARROW_WARPS * STAGE * d.Dp * 4;                 // (also enough for param_sums, from a Dp of 32 up)
    const long long units = ((long long)d.nocc + 2 * TILE - 1) / (2 * TILE);
    pbg_opt_in_smem((const void *)narrow_tile_kernel<NP>, NARROW_WARPS * STAGE * VEC * 512);
    pbg_launch(narrow_tile_kernel<NP>, sum_ctas + (unsigned)((units + NARROW_WARPS - 1) / NARROW_WARPS), 32 * NARROW_WARPS, smem, st, d, wb, w, keys, vals, lr, us.psum, us.hublist, hubcnt, job, sum_ctas);
  } else {
    constexpr int V = VEC <= 2 ? 4 : VEC;
    constexpr int EMB_WARPS = TileWarps<V, RULE_EMB>::N;
    pbg_opt_in_smem((const void *)tile_update_kernel<V, RULE_EMB>, EMB_WARPS * TILE * V * 512);
    pbg_launch(tile_update_kernel<V, RULE_EMB>, sum_ctas + (unsigned)((tiles + EMB_WARPS - 1) / EMB_WARPS), 32 * EMB_WARPS, (size_t)EMB_WARPS * TILE * d.Dp * 4, st, d, wb, w, keys, vals, lr, us.psum, us.hublist, hubcnt, job, sum_ctas);
  }
  const bool rel_rows = has_operator_rows(d);
  long long *rel_hublist = us.hublist + pbg_hublist_entries(d.nocc), *rel_bigtab = us.bigtab + pbg_bigtab_bytes(d.nocc) / sizeof(long long);
  if (rel_rows) {
    pbg_opt_in_smem((const void *)tile_update_kernel<VEC, RULE_REL>, REL_WARPS * TILE * VEC * 512);
    pbg_launch(tile_update_kernel<VEC, RULE_REL>, (unsigned)((tiles + REL_WARPS - 1) / REL_WARPS) + 1, 32 * REL_WARPS, (size_t)REL_WARPS * TILE * d.Dp * 4, st, d, wb, w, keys, vals, rel_lr, us.psum, rel_hublist, hubcnt + HUB_REL, job, 0);
  }
  pbg_launch(hub_kernel<VEC, RULE_EMB>, d.k + param_step_ctas(d, job) + hub_ctas, 32 * UPD_WARPS, hub_smem, st,
             d, wb, w, keys, vals, lr, us.psum, us.hublist, hubcnt, hubcnt_next, us.bigtab, 1, job, us.per_batch, us.sum);
  launches += 2;
  if (rel_rows) {
    pbg_opt_in_smem((const void *)hub_kernel<VEC, RULE_REL>, (int)hub_smem_max);
    pbg_launch(hub_kernel<VEC, RULE_REL>, hub_ctas + 1, 32 * UPD_WARPS, hub_smem, st,
               d, wb, w, keys, vals, rel_lr, us.psum, rel_hublist, hubcnt + HUB_REL, hubcnt_next + HUB_REL, rel_bigtab, 0, job, (pbg_batch_stats *)nullptr, (double *)nullptr);
    launches += 2;
  }
  if (d.op != PBG_OP_NONE && w.theta[0] != nullptr) {
    if (d.matrix_op) {
      launches += launch_matrix_update(d, wb, w, rel_lr, st);
    }
  }
  pbg_note_launch();
  return launches;
}

int launch_update(const WaveDims &d, const WaveBatches &wb, const WaveBufs &w, const unsigned long long *keys, const unsigned int *vals,
                  float lr, float rel_lr, const UpdateScratch &us, cudaStream_t st) {
  int vec = (d.D + 127) / 128;
  if (vec <= 1) return launch_update_vec<1>(d, wb, w, keys, vals, lr, rel_lr, us, st);
  if (vec <= 2) return launch_update_vec<2>(d, wb, w, keys, vals, lr, rel_lr, us, st);
  if (vec <= 4) return launch_update_vec<4>(d, wb, w, keys, vals, lr, rel_lr, us, st);
  if (vec <= 8) return launch_update_vec<8>(d, wb, w, keys, vals, lr, rel_lr, us, st);
  return launch_update_vec<16>(d, wb, w, keys, vals, lr, rel_lr, us, st);
}

// Stand-alone sparse RowAdagrad step (row_adagrad.py:80-96): rows sorted with duplicates adjacent,
// vals[q] = index of the gradient row.
template <int VEC>
__global__ void __launch_bounds__(32 * UPD_WARPS)
row_adagrad_sorted_kernel(float *emb, float *state, int D, const unsigned long long *__restrict__ keys,
                          const unsigned int *__restrict__ vals, const float *__restrict__ grads, int n,
                          float lr, unsigned long long key_invalid) {
  pdl_begin();
  int lane = threadIdx.x & 31;
  long long pos = (long long)blockIdx.x * UPD_WARPS + (threadIdx.x >> 5);
  if (pos >= n) return;
  unsigned long long key = keys[pos];
  if (key >= key_invalid) return;
  if (pos > 0 && keys[pos - 1] == key) return;
  float4 acc[VEC];
#pragma unroll
  for (int c = 0; c < VEC; ++c) acc[c] = f4zero();
  for (long long q = pos; q < n && keys[q] == key; ++q) {
    const float *g = grads + (size_t)vals[q] * D;
#pragma unroll
    for (int c = 0; c < VEC; ++c) {
      int dd = c * 128 + lane * 4;
      if (dd < D) acc[c] = acc[c] + ld4(g + dd);
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < VEC; ++c) ss += f4dot(acc[c], acc[c]);
  ss = warp_sum(ss);
  float G = state[key] + ss / (float)D;
  float stepv = lr / (sqrtf(G) + PBG_ADAGRAD_EPS);
  float *wrow = emb + (size_t)key * D;
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    int dd = c * 128 + lane * 4;
    if (dd < D) st4(wrow + dd, ld4(wrow + dd) - acc[c] * stepv);
  }
  if (lane == 0) state[key] = G;
}

int launch_row_adagrad_sorted(float *emb, float *state, int dim, const unsigned long long *keys,
                              const unsigned int *vals, const float *grads, int n, float lr,
                              unsigned long long key_invalid, cudaStream_t st) {
  int ctas = (n + UPD_WARPS - 1) / UPD_WARPS;
  int vec = (dim + 127) / 128;
#define RA(V) pbg_launch(row_adagrad_sorted_kernel<V>, ctas, 32 * UPD_WARPS, 0, st, emb, state, dim, keys, vals, grads, n, lr, key_invalid)
  if (vec <= 1) RA(1); else if (vec <= 2) RA(2); else if (vec <= 4) RA(4); else if (vec <= 8) RA(8); else RA(16);
#undef RA
  return 1;
}
