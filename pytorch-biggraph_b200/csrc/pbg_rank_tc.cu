// Ranking against all entities on the tensor cores: the score tiles of pbg_eval_batch_all_negs in every precision tier
// but fp32.  128 edges x 256 candidates per tile, operands as three bf16 planes per value and the six plane products of
// order <= 2 (fp32-level accuracy whatever the training tier), accumulators in tensor memory; a tile's scores are
// counted and summed where they lie and never stored.
//
// The CUDA-core tiles this replaces ran at 18 TFLOP/s of useful work (1000 edges against 14,951 entities a side,
// dimension 400: 1.0 ms of a 1.33 ms call; this one takes 123 us of 186).  Not at a limit: 32 k-values of a tile take 2,500 to
// 2,800 cycles, where the products take 1,540 and shared memory is busy for 1,690 (72 KB loaded, 144 KB read).
//
// Persistent CTAs walk the tiles of both sides, the row blocks of the same candidates one after the other: CTAs that run at the
// same time then ask L2 for the same candidates (188.0 us a call, 189.7 with the candidate blocks first).
//   warp 0     TMA producer, one box (all planes) per operand
//   warp 1     tensor memory and MMA issue; two accumulators alternate
//   warps 2-9  epilogue: thread = edge, two warps per 32 tensor-memory lanes, each one half of the columns
// Every mbarrier wait is bounded (bit 1 of the error word); every TMA load is CTA-local.
#include "pbg_tc.cuh"

#define RK_THREADS 320
#define RK_STAGES 3
#define RK_BN 256
#define RK_PLANE_A (128u * 64u)
#define RK_PLANE_B ((unsigned)RK_BN * 64u)
#define RK_STAGE (3u * (RK_PLANE_A + RK_PLANE_B))

struct RankMaps { CUtensorMap q, y; };     // planes of the scored rows / of the candidate slab: 4-D (k, row, plane, side)

__global__ void __launch_bounds__(RK_THREADS, 1)
allnegs_tc_kernel(const __grid_constant__ RankMaps maps, WaveDims d, WaveBufs w, AllNegs a, long long row0) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) unsigned long long bars[2 * RK_STAGES + 4];
  __shared__ uint32_t tmem_base_s;
  __shared__ volatile int failed;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t bar0 = smem_u32(&bars[0]);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (RK_STAGES + s); };
  auto accf_bar = [&](int b) { return bar0 + 8u * (2 * RK_STAGES + b); };
  auto acce_bar = [&](int b) { return bar0 + 8u * (2 * RK_STAGES + 2 + b); };
  int *errflag = w.errflag;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * RK_STAGES + 2; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar0 + 8u * i));
    for (int b = 0; b < 2; ++b) asm volatile("mbarrier.init.shared::cta.b64 [%0], 256;" :: "r"(acce_bar(b)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    failed = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" :: "r"(smem_u32(&tmem_base_s)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_s;
  pdl_begin();                                               // barriers and tensor memory are set up beside the kernel before this one
  const int nkb = (d.D + 31) / 32;
  const int tiles_m = (a.B + 127) / 128, tiles_n = a.slab / RK_BN;
  const int ntiles = 2 * tiles_m * tiles_n;
  // tile t -> side, edges [m0, m0 + 128), candidates [n0, n0 + 256) of the slab; every role walks the same list
  auto tile_live = [&](int t, int &side, int &m0, int &n0, int &n) {
    m0 = (t % tiles_m) * 128;
    n0 = (t / tiles_m % tiles_n) * RK_BN;
    side = t / tiles_m / tiles_n;
    const long long left = d.n_rows[side] - row0;
    n = left < a.slab ? (int)left : a.slab;                              // candidates of the slab on this side
    return d.neg_enabled[side] && n0 < n;
  };
  int side, m0, n0, n;
  if (warp == 0) {
    int git = 0;
    bool stop = false;
    for (int t = blockIdx.x; t < ntiles && !stop; t += gridDim.x) {
      if (__any_sync(0xffffffffu, failed != 0)) break;
      if (!tile_live(t, side, m0, n0, n)) continue;
      for (int kb = 0; kb < nkb; ++kb, ++git) {
        const int s = git % RK_STAGES;
        bool ok = true;
        if (git >= RK_STAGES && lane == 0) ok = mbar_wait(empty_bar(s), (uint32_t)((git / RK_STAGES) - 1) & 1, errflag);
        if (!__all_sync(0xffffffffu, ok)) { failed = 1; stop = true; break; }
        const uint32_t fb = full_bar(s), st = smem_u32(smem + (size_t)s * RK_STAGE);
        if (lane == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(fb), "r"(RK_STAGE) : "memory");
        __syncwarp();
        if (lane == 0) tma_load_4d(st, &maps.q, kb * 32, m0, 0, side, fb);
        else if (lane == 1) tma_load_4d(st + 3 * RK_PLANE_A, &maps.y, kb * 32, n0, 0, side, fb);
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(RK_BN >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    const int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};   // smallest contributions first
    const bool leader = elect_one();
    StageRing at;
    int j = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
      if (__any_sync(0xffffffffu, failed != 0)) break;
      if (!tile_live(t, side, m0, n0, n)) continue;
      const int ab = j & 1;
      if (j >= 2 && !__all_sync(0xffffffffu, mbar_wait(acce_bar(ab), (uint32_t)((j >> 1) - 1) & 1, errflag))) { failed = 1; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      bool ok = true;
      for (int kb = 0; kb < nkb; ++kb, at.next(RK_STAGES)) {
        const int s = at.s;
        if (!__all_sync(0xffffffffu, mbar_wait(full_bar(s), at.parity, errflag))) { failed = 1; ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t sa = smem_u32(smem) + (uint32_t)s * RK_STAGE;
        const uint64_t da = smem_desc(sa, 0, 512, 4), db = smem_desc(sa + 3 * RK_PLANE_A, 0, 512, 4);
#pragma unroll
        for (int k16 = 0; k16 < 2; ++k16) {
          if (k16 * 16 >= d.D - kb * 32) break;                          // the tail of K is zero fill
#pragma unroll
          for (int tt = 0; tt < 6; ++tt)
            if (leader) mma_f16(tmem + (uint32_t)ab * 256u, desc_at(da, pa[tt] * RK_PLANE_A + k16 * 32), desc_at(db, pb[tt] * RK_PLANE_B + k16 * 32), idesc, kb > 0 || k16 > 0 || tt > 0);
        }
        if (leader) mma_commit(empty_bar(s));
      }
      if (!ok) break;
      if (leader) mma_commit(accf_bar(ab));
      ++j;
    }
  } else if (warp >= 2) {
    const int q = warp & 3, half = (warp - 2) >> 2;
    int j = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
      if (__any_sync(0xffffffffu, failed != 0)) break;                   // warp-uniform exit (tcgen05.ld is warp-wide)
      if (!tile_live(t, side, m0, n0, n)) continue;
      const int ab = j & 1;
      bool okw = true;
      if (lane == 0) okw = mbar_wait(accf_bar(ab), (uint32_t)(j >> 1) & 1, errflag);
      if (!__all_sync(0xffffffffu, okw)) { failed = 1; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int e = m0 + q * 32 + lane;
      const bool real = e < a.B;
      const float pos = real ? a.pos[side][e] : 0.f, qn = real ? a.qn[side][e] : 0.f;
      const long long own = real ? (side == 0 ? w.lhs : w.rhs)[e] - row0 : -1;     // the edge's own entity, as a row of the slab
      const float *yn = a.yn[side];
      int cnt = 0;
      float ra = 0.f, rb = d.loss == PBG_LOSS_SOFTMAX ? -INFINITY : 0.f;
#pragma unroll 1
      for (int c0 = half * 128; c0 < half * 128 + 128 && n0 + c0 < n; c0 += 32) {
        uint32_t r[32];
        tmem_ld32(tmem + (uint32_t)ab * 256u + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, r);
        float sv[32], mx = -INFINITY;
        unsigned live = 0u;
#pragma unroll
        for (int jj = 0; jj < 32; ++jj) {
          const int c = n0 + c0 + jj;
          float s = __uint_as_float(r[jj]);
          if (d.cmp >= PBG_CMP_L2) {
            const float qv = (yn[c < n ? c : 0] - 2.0f * s) + qn;        // model.py:226-246
            s = d.cmp == PBG_CMP_L2 ? -sqrtf(fmaxf(qv, 1e-30f)) : -qv;
          }
          sv[jj] = s;
          if (c < n && c != own) {
            live |= 1u << jj;
            cnt += s >= pos;
            mx = fmaxf(mx, s);
          }
        }
        if (d.loss == PBG_LOSS_RANKING) {
#pragma unroll
          for (int jj = 0; jj < 32; ++jj) if (live >> jj & 1u) ra += fmaxf(0.f, (sv[jj] - pos) + d.margin);
        } else if (d.loss == PBG_LOSS_LOGISTIC) {
#pragma unroll
          for (int jj = 0; jj < 32; ++jj) if (live >> jj & 1u) ra += fmaxf(sv[jj], 0.f) + log1pf(expf(-fabsf(sv[jj])));
        } else if (live) {
          if (mx > rb) { ra *= expf(rb - mx); rb = mx; }                  // (the first time: 0 x exp(-inf) = 0)
#pragma unroll
          for (int jj = 0; jj < 32; ++jj) if (live >> jj & 1u) ra += expf(sv[jj] - rb);
        }
      }
      if (real) {
        const size_t o = (size_t)(2 * (n0 / RK_BN) + half) * a.B + e;
        a.pcnt[side][o] = cnt; a.pa[side][o] = ra; a.pb[side][o] = rb;
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(acce_bar(ab)) : "memory");
      ++j;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    // if a wait ran out, copies / MMAs may still be in flight: a bounded grace period before the tensor memory goes back
    if (failed) for (int it = 0; it < 200000; ++it) __nanosleep(20);
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem) : "memory");
  }
}

int launch_allnegs_score_tc(const WaveDims &d, const WaveBufs &w, const AllNegs &a, long long row0, cudaStream_t st) {
  // (encoding two maps is a microsecond of host time beside a call of a hundred)
  RankMaps maps;
  if (!encode4_planes(&maps.q, a.QB, 3, d.D, a.B, a.qrows, 2, a.Dpb, 128) ||
      !encode4_planes(&maps.y, a.YB, 3, d.D, a.slab, a.slab, 2, a.Dpb, RK_BN)) {
    pbg_note_launch(cudaErrorUnknown);
    return 0;
  }
  const size_t smem = RK_STAGES * RK_STAGE + 1024;
  pbg_opt_in_smem((const void *)allnegs_tc_kernel, (int)smem);
  const int tiles = 2 * ((a.B + 127) / 128) * (a.slab / RK_BN), sms = pbg_sm_count();
  pbg_launch(allnegs_tc_kernel, tiles < sms ? tiles : sms, RK_THREADS, smem, st, maps, d, w, a, row0);
  pbg_note_launch();
  return 1;
}
