// Stable LSD radix sort of (row key, occurrence) pairs: groups the gradient slots of one wave by
// the embedding row they belong to, in batch order, so that the update kernel can sum duplicate
// rows before the (non-linear) RowAdagrad step -- the device counterpart of `grad.coalesce()` in
// torchbiggraph/row_adagrad.py:83.
//
// One pass sorts `db` key bits (up to 11, 2048 bins; the passes split the key bits evenly) with
// three launches:
//   radix_hist     every warp owns a run of RUN consecutive pairs and counts its digits into
//                  hist[digit][warp]
//   radix_scan     one CTA per digit: exclusive scan of that digit's row of warp counts, row total
//                  to totals[digit]
//   radix_scatter  every CTA turns totals[] into digit bases (a block scan of <= 2048 values), then
//                  every warp walks its run in order and writes each pair to
//                  base[digit] + scanned[digit][warp] + (earlier pairs of the run with that digit)
// Ranking inside a run uses __match_any_sync, so equal digits keep their input order (stable).
//
// That is the form for long lists.  A list that fits in the shared memory of one thread-block cluster -- every wave
// up to 262,144 slots -- is sorted by ONE kernel (sort_waves_kernel, at the end of this file).
#include <cooperative_groups.h>

#include "pbg_common.cuh"

namespace cg = cooperative_groups;

#define RUN_ITEMS 8                      // pairs per lane per run
#define RUN (32 * RUN_ITEMS)             // pairs per warp
#define SORT_WARPS_PER_CTA 4
#define MAX_BINS 2048

int pbg_sort_warps(int n) { return (n + RUN - 1) / RUN; }
// counters a sort of n pairs needs: [MAX_BINS][warps] + [MAX_BINS] totals
size_t pbg_sort_hist_entries(int n) { return (size_t)MAX_BINS * pbg_sort_warps(n) + MAX_BINS; }

__global__ void __launch_bounds__(32 * SORT_WARPS_PER_CTA)
radix_hist(const unsigned long long *__restrict__ keys, int n, int shift, int nbins, unsigned int *__restrict__ hist,
           int nwarps) {
  __shared__ unsigned int cnt[SORT_WARPS_PER_CTA][MAX_BINS];
  int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int wg = blockIdx.x * SORT_WARPS_PER_CTA + wl;
  const unsigned long long mask = (unsigned long long)(nbins - 1);
  for (int i = lane; i < nbins; i += 32) cnt[wl][i] = 0;
  __syncwarp();
  if (wg < nwarps) {
    int base = wg * RUN;
    for (int it = 0; it < RUN_ITEMS; ++it) {
      int i = base + it * 32 + lane;
      bool ok = i < n;
      unsigned int dg = ok ? (unsigned int)((keys[i] >> shift) & mask) : 0u;
      unsigned int act = __ballot_sync(0xffffffffu, ok);
      if (ok) {
        unsigned int peers = __match_any_sync(act, dg);
        if ((peers & ((1u << lane) - 1u)) == 0u) cnt[wl][dg] += __popc(peers);   // lowest peer adds
      }
      __syncwarp();
    }
    for (int i = lane; i < nbins; i += 32) hist[(size_t)i * nwarps + wg] = cnt[wl][i];
  }
}

// grid = nbins CTAs of 128 threads: exclusive scan of hist[digit][0..nwarps) in place.
__global__ void __launch_bounds__(128) radix_scan(unsigned int *__restrict__ hist, int nwarps,
                                                  unsigned int *__restrict__ totals) {
  __shared__ unsigned int part[128];
  unsigned int *row = hist + (size_t)blockIdx.x * nwarps;
  int t = threadIdx.x;
  int per = (nwarps + 127) / 128;
  int lo = t * per, hi = lo + per < nwarps ? lo + per : nwarps;
  unsigned int s = 0;
  for (int i = lo; i < hi; ++i) s += row[i];
  part[t] = s;
  __syncthreads();
  for (int off = 1; off < 128; off <<= 1) {
    unsigned int v = t >= off ? part[t - off] : 0u;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  unsigned int run = part[t] - s;
  for (int i = lo; i < hi; ++i) { unsigned int v = row[i]; row[i] = run; run += v; }
  if (t == 127) totals[blockIdx.x] = part[127];
}

__global__ void __launch_bounds__(32 * SORT_WARPS_PER_CTA)
radix_scatter(const unsigned long long *__restrict__ keys, const unsigned int *__restrict__ vals, int n,
              int shift, int nbins, const unsigned int *__restrict__ hist, const unsigned int *__restrict__ totals,
              int nwarps, unsigned long long *__restrict__ keys_out, unsigned int *__restrict__ vals_out) {
  __shared__ unsigned int pos[SORT_WARPS_PER_CTA][MAX_BINS];
  __shared__ unsigned int base[MAX_BINS];
  __shared__ unsigned int wsum[SORT_WARPS_PER_CTA];
  int wl = threadIdx.x >> 5, lane = threadIdx.x & 31, t = threadIdx.x;
  const unsigned long long mask = (unsigned long long)(nbins - 1);
  // digit bases: exclusive scan of totals[0..nbins) by the whole CTA (each thread a contiguous chunk)
  {
    constexpr int T = 32 * SORT_WARPS_PER_CTA;
    int per = (nbins + T - 1) / T;
    int lo = t * per, hi = lo + per < nbins ? lo + per : nbins;
    unsigned int s = 0;
    for (int i = lo; i < hi; ++i) s += totals[i];
    unsigned int incl = s;                                   // inclusive scan inside the warp
    for (int off = 1; off < 32; off <<= 1) {
      unsigned int v = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += v;
    }
    if (lane == 31) wsum[wl] = incl;
    __syncthreads();
    unsigned int before = 0;
    for (int k = 0; k < wl; ++k) before += wsum[k];
    unsigned int run = before + incl - s;
    for (int i = lo; i < hi; ++i) { base[i] = run; run += totals[i]; }
    __syncthreads();
  }
  int wg = blockIdx.x * SORT_WARPS_PER_CTA + wl;
  if (wg >= nwarps) return;
  for (int i = lane; i < nbins; i += 32) pos[wl][i] = base[i] + hist[(size_t)i * nwarps + wg];
  __syncwarp();
  int b0 = wg * RUN;
  for (int it = 0; it < RUN_ITEMS; ++it) {
    int i = b0 + it * 32 + lane;
    bool ok = i < n;
    unsigned long long key = ok ? keys[i] : 0ull;
    unsigned int dg = (unsigned int)((key >> shift) & mask);
    unsigned int act = __ballot_sync(0xffffffffu, ok);
    unsigned int peers = 0u;
    if (ok) {
      peers = __match_any_sync(act, dg);
      unsigned int before = __popc(peers & ((1u << lane) - 1u));
      unsigned int dst = pos[wl][dg] + before;
      keys_out[dst] = key;
      vals_out[dst] = vals[i];
    }
    __syncwarp();                                          // every peer has read pos[] by now
    if (ok && (peers & ((1u << lane) - 1u)) == 0u) pos[wl][dg] += __popc(peers);
    __syncwarp();
  }
}

int pbg_sort(SortPlan &sp, int n, int bits, cudaStream_t st) {
  int launches = 0;
  int src = 0;
  sp.result = 0;
  if (n <= 0) return 0;
  int nwarps = pbg_sort_warps(n);
  int ctas = (nwarps + SORT_WARPS_PER_CTA - 1) / SORT_WARPS_PER_CTA;
  int passes = (bits + 10) / 11;
  int db = (bits + passes - 1) / passes;                   // digit bits of every pass (<= 11)
  int nbins = 1 << db;
  unsigned int *totals = sp.hist + (size_t)MAX_BINS * nwarps;
  for (int pass = 0, shift = 0; pass < passes; ++pass, shift += db) {
    pbg_launch_in_order(radix_hist, ctas, 32 * SORT_WARPS_PER_CTA, 0, st, sp.keys[src], n, shift, nbins, sp.hist, nwarps);
    pbg_launch_in_order(radix_scan, nbins, 128, 0, st, sp.hist, nwarps, totals);
    pbg_launch_in_order(radix_scatter, ctas, 32 * SORT_WARPS_PER_CTA, 0, st, sp.keys[src], sp.vals[src], n, shift, nbins, sp.hist, totals,
                        nwarps, sp.keys[src ^ 1], sp.vals[src ^ 1]);
    launches += 3;
    src ^= 1;
  }
  sp.result = src;
  return launches;
}

// keys[i] = rows[i] (invalid rows flagged and sent to the end), vals[i] = i: the set-up of the
// stand-alone sparse RowAdagrad entry point.
__global__ void iota_keys(const long long *__restrict__ rows, long long num_rows, int n,
                          unsigned long long *__restrict__ keys, unsigned int *__restrict__ vals,
                          int *errflag) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  long long r = rows[i];
  bool bad = r < 0 || r >= num_rows;
  if (bad) atomicOr(errflag, 1);
  keys[i] = bad ? (unsigned long long)num_rows : (unsigned long long)r;
  vals[i] = (unsigned int)i;
}

int launch_iota_keys(const long long *rows, long long num_rows, int n, unsigned long long *keys,
                     unsigned int *vals, int *errflag, cudaStream_t st) {
  pbg_launch_in_order(iota_keys, (n + 255) / 256, 256, 0, st, rows, num_rows, n, keys, vals, errflag);
  return 1;
}

// ------------------------------------------------------------------------------------------------
// One kernel, one cluster per list.  The three-launch passes above are latency: seven launches for the two passes of a
// wave of 4,000 slots (keys included), each a few microseconds of which hardly any is work.  Here the list never leaves
// the cluster: every thread holds IPT pairs in registers, a pass ranks them inside the warp (ballots), scans the warps'
// digit counts inside the CTA, exchanges the CTAs' digit totals through distributed shared memory (one cluster
// barrier) and writes every pair to its place in the shared memory of the CTA that owns it (a second barrier); the last
// pass writes to global memory.  Digits of at most 8 bits: the warps' counters of a CTA are 32 KB, and the exchange of
// 16 x 256 totals is one coalesced round.
// ------------------------------------------------------------------------------------------------
#define CS_THREADS 1024
#define CS_WARPS 32
#define CS_BINS 256

struct SortRows { const long long *rows; long long num_rows; int n; unsigned long long *keys; unsigned int *vals; int *errflag; };

// Another CTA's shared memory may be written only once that CTA is known to run.  The kernels therefore arrive at the
// cluster's barrier first thing, and the wait that belongs to it stands in front of the first remote store; the key build
// and the first ranking lie between the two.
template <int IPT>
__device__ __forceinline__ void cluster_sort_body(uint2 (&item)[IPT], int n, int bits, unsigned long long *keys_out, unsigned int *vals_out,
                                                  unsigned char *smem) {
  uint2 *buf = (uint2 *)smem;                                           // [CS_THREADS * IPT] pairs of this CTA
  unsigned int *cnt = (unsigned int *)(smem + (size_t)CS_THREADS * IPT * 8);   // [CS_WARPS][bins]
  unsigned int *all = cnt + CS_WARPS * CS_BINS;                         // [CTAs][bins] digit totals of every CTA
  unsigned int *base = all + 16 * CS_BINS;                              // [bins]
  unsigned int *wsum = base + CS_BINS;                                  // [8]
  cg::cluster_group cluster = cg::this_cluster();
  const int nct = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int t = threadIdx.x, lane = t & 31, wl = t >> 5;
  const int passes = (bits + 7) / 8, db = (bits + passes - 1) / passes, bins = 1 << db;
  const unsigned int mask = (unsigned int)bins - 1u, lt = (1u << lane) - 1u;
  unsigned int *wc = cnt + wl * bins;
  unsigned int off[IPT];
  for (int pass = 0, shift = 0; pass < passes; ++pass, shift += db) {
    for (int i = lane; i < bins; i += 32) wc[i] = 0u;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      const unsigned int dg = (item[i].x >> shift) & mask;
      unsigned int peers = 0xffffffffu;
      for (int b = 0; b < db; ++b) {
        const unsigned int m = __ballot_sync(0xffffffffu, (dg >> b) & 1u);
        peers &= ((dg >> b) & 1u) ? m : ~m;
      }
      const unsigned int before = wc[dg];
      __syncwarp();
      if ((peers & lt) == 0u) wc[dg] = before + __popc(peers);
      __syncwarp();
      off[i] = before + __popc(peers & lt);
    }
    __syncthreads();
    if (pass == 0) cluster.barrier_wait();                              // every CTA of the cluster runs: its shared memory may be written
    if (t < bins) {
      unsigned int run = 0u, c[CS_WARPS];
#pragma unroll
      for (int w = 0; w < CS_WARPS; ++w) c[w] = cnt[w * bins + t];
#pragma unroll
      for (int w = 0; w < CS_WARPS; ++w) { cnt[w * bins + t] = run; run += c[w]; }
      for (int c = 0; c < nct; ++c) cluster.map_shared_rank(all, c)[rank * CS_BINS + t] = run;
    }
    cluster.sync();                                                     // totals are everywhere; every pair is in registers
    unsigned int tot = 0u, lower = 0u;
    if (t < bins) {
      for (int c = 0; c < nct; ++c) { const unsigned int v = all[c * CS_BINS + t]; tot += v; if (c < rank) lower += v; }
    }
    if (t < CS_BINS) {
      unsigned int incl = tot;
      for (int o = 1; o < 32; o <<= 1) { const unsigned int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
      if (lane == 31) wsum[wl] = incl;
      base[t] = incl - tot + lower;
    }
    __syncthreads();
    if (t < CS_BINS && wl > 0) {
      unsigned int before = 0u;
      for (int w = 0; w < wl; ++w) before += wsum[w];
      base[t] += before;
    }
    __syncthreads();
    const bool last = pass == passes - 1;
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      const unsigned int dg = (item[i].x >> shift) & mask;
      const unsigned int pos = base[dg] + wc[dg] + off[i];
      if (last) {
        if (pos < (unsigned int)n) { keys_out[pos] = item[i].x; vals_out[pos] = item[i].y; }
      } else {
        cluster.map_shared_rank(buf, pos / (CS_THREADS * IPT))[pos % (CS_THREADS * IPT)] = item[i];
      }
    }
    if (!last) {
      cluster.sync();
#pragma unroll
      for (int i = 0; i < IPT; ++i) item[i] = buf[(wl * IPT + i) * 32 + lane];
    }
  }
}

template <int IPT>
static size_t cluster_sort_smem() { return (size_t)CS_THREADS * IPT * 8 + (CS_WARPS * CS_BINS + 16 * CS_BINS + CS_BINS + 8) * 4; }

// Pairs beyond the list's end carry the largest key; they come last in every pass and are not written out.
template <int IPT>
__global__ void __launch_bounds__(CS_THREADS, 1)
sort_waves_kernel(WaveDims d, WaveBufs w, const __grid_constant__ SortWaves waves, int bits) {
  extern __shared__ __align__(16) unsigned char cs_smem[];
  cg::this_cluster().barrier_arrive();
  const int nct = (int)cg::this_cluster().num_blocks(), rank = (int)cg::this_cluster().block_rank();
  const SortWave &sw = waves.w[blockIdx.x / nct];
  const int n = sw.k * d.spb;
  const int first = rank * CS_THREADS * IPT + (threadIdx.x >> 5) * 32 * IPT + (threadIdx.x & 31);
  uint2 item[IPT];
#pragma unroll
  for (int i = 0; i < IPT; ++i) {
    const int o = first + i * 32;
    item[i] = make_uint2(o < n ? (unsigned int)slot_key(d, sw.wb, w, o) : 0xffffffffu, (unsigned int)o);
  }
  cluster_sort_body<IPT>(item, n, bits, sw.keys, sw.vals, cs_smem);
}

template <int IPT>
__global__ void __launch_bounds__(CS_THREADS, 1) sort_rows_kernel(SortRows a, int bits) {
  extern __shared__ __align__(16) unsigned char cs_smem[];
  cg::this_cluster().barrier_arrive();
  const int first = (int)cg::this_cluster().block_rank() * CS_THREADS * IPT + (threadIdx.x >> 5) * 32 * IPT + (threadIdx.x & 31);
  uint2 item[IPT];
#pragma unroll
  for (int i = 0; i < IPT; ++i) {
    const int o = first + i * 32;
    unsigned int key = 0xffffffffu;
    if (o < a.n) {
      const long long r = a.rows[o];
      const bool bad = r < 0 || r >= a.num_rows;
      if (bad) atomicOr(a.errflag, 1);
      key = (unsigned int)(bad ? a.num_rows : r);
    }
    item[i] = make_uint2(key, (unsigned int)o);
  }
  cluster_sort_body<IPT>(item, a.n, bits, a.keys, a.vals, cs_smem);
}

// CTAs and pairs per thread for a list of n: one pair per thread as long as the cluster can grow, then up to sixteen on
// sixteen CTAs.  A barrier of a large cluster costs less than building and ranking more pairs per thread: a list of
// 4,000 slots took 21 us on one CTA with four pairs per thread.
static void cluster_shape(int n, int &ctas, int &ipt) {
  ipt = 1;
  for (ctas = 1; ctas < 16 && ctas * CS_THREADS < n; ctas *= 2) {}
  while (ctas * CS_THREADS * ipt < n) ipt *= 2;
}

// KERNEL<pairs per thread>(args) on `lists` clusters
#define CS_LAUNCH(KERNEL, LISTS, ...)                                                                       \
  do {                                                                                                      \
    if (ipt == 1) launch_cluster(KERNEL<1>, LISTS, ctas, cluster_sort_smem<1>(), st, __VA_ARGS__);          \
    else if (ipt == 2) launch_cluster(KERNEL<2>, LISTS, ctas, cluster_sort_smem<2>(), st, __VA_ARGS__);     \
    else if (ipt == 4) launch_cluster(KERNEL<4>, LISTS, ctas, cluster_sort_smem<4>(), st, __VA_ARGS__);     \
    else if (ipt == 8) launch_cluster(KERNEL<8>, LISTS, ctas, cluster_sort_smem<8>(), st, __VA_ARGS__);     \
    else launch_cluster(KERNEL<16>, LISTS, ctas, cluster_sort_smem<16>(), st, __VA_ARGS__);                 \
  } while (0)

template <class... Args>
static void launch_cluster(void (*kernel)(Args...), int lists, int ctas, size_t smem, cudaStream_t st, Args... args) {
  if (pbg_launch_failed()) return;
  pbg_opt_in_smem((const void *)kernel, (int)smem);
  if (ctas > 8) pbg_opt_in_cluster16((const void *)kernel);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(lists * ctas); cfg.blockDim = dim3(CS_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = ctas; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
  cfg.attrs = &at; cfg.numAttrs = 1;
  pbg_note_launch(cudaLaunchKernelEx(&cfg, kernel, args...));
}

// Whether clusters of this shape can be resident on the device at all: with part of its SMs (MPS, MIG, green contexts) there may
// be no sixteen of them close enough together that each have the shared memory free.
template <int IPT>
static bool cluster_resident(int ctas) {
  for (const void *kernel : {(const void *)sort_waves_kernel<IPT>, (const void *)sort_rows_kernel<IPT>}) {
    if (pbg_opt_in_smem(kernel, (int)cluster_sort_smem<IPT>()) != cudaSuccess) return false;
    if (ctas > 8 && pbg_opt_in_cluster16(kernel) != cudaSuccess) return false;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas); cfg.blockDim = dim3(CS_THREADS); cfg.dynamicSmemBytes = cluster_sort_smem<IPT>();
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = ctas; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) return false;
  }
  return true;
}

// The largest list takes the most CTAs and shared memory; where its clusters fit, those of shorter lists do.
bool pbg_cluster_sort_available(long long n) {
  int ctas, ipt;
  cluster_shape((int)(n < PBG_CLUSTER_SORT_MAX ? n : PBG_CLUSTER_SORT_MAX), ctas, ipt);
  const bool ok = ipt == 1 ? cluster_resident<1>(ctas) : ipt == 2 ? cluster_resident<2>(ctas) : ipt == 4 ? cluster_resident<4>(ctas) : ipt == 8 ? cluster_resident<8>(ctas) : cluster_resident<16>(ctas);
  if (!ok) pbg_take_launch_error();                          // (an answer, not a failure of the call that asked)
  return ok;
}

int launch_sort_waves(const WaveDims &d, const WaveBufs &w, const SortWaves &waves, int bits, cudaStream_t st) {
  int most = 0, ctas, ipt;
  for (int i = 0; i < waves.count; ++i) if (waves.w[i].k > most) most = waves.w[i].k;
  cluster_shape(most * d.spb, ctas, ipt);
  CS_LAUNCH(sort_waves_kernel, waves.count, d, w, waves, bits);
  return 1;
}

int launch_sort_rows(const long long *rows, long long num_rows, int n, int bits, unsigned long long *keys, unsigned int *vals,
                     int *errflag, cudaStream_t st) {
  SortRows a{rows, num_rows, n, keys, vals, errflag};
  int ctas, ipt;
  cluster_shape(n, ctas, ipt);
  CS_LAUNCH(sort_rows_kernel, 1, a, bits);
  return 1;
}
