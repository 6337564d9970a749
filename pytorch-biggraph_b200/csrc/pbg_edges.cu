// The edge-list utilities either side of the training step, on the device: what the reference's native
// module torchbiggraph._C does on host threads (torchbiggraph/util.cpp) --
//   reverse_permutation   util.cpp:103-125   out[perm[i]] = i
//   shuffle               util.cpp:127-220   row i of a table moves to row perm[i]
//   sub_bucket            util.cpp:260-423   stable split of a bucket's edges into N x M sub-buckets
//   randperm              util.cpp:14-101    a seeded random permutation (also stands where the trainers call
//                                            torch.randperm for the per-bucket edge shuffle, train_cpu.py:857-859,
//                                            train_gpu.py:245)
// All of it is integer / byte work bound by HBM: coalesced 8- and 16-byte accesses, one stable LSD radix sort
// (pbg_sort.cu) where an order is needed.  Range violations are reported through the context's error word and the
// offending elements skipped; nothing faults.
#include "pbg_common.cuh"

// res[perm[i]] = i
__global__ void reverse_permutation_kernel(const long long *__restrict__ perm, long long n, long long *__restrict__ out, int *errflag) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  long long p = perm[i];
  if (p < 0 || p >= n) { atomicOr(errflag, 1); return; }
  out[p] = i;
}

// out row perm[r] = in row r.  A group of G threads moves a row of `units` elements of type T, four elements per thread in
// flight; G is the power of two that covers a row in at most four steps.  (One thread per element divided a 64-bit index
// by the row length for every 16 bytes: 4.4 TB/s on 303,000 rows of 400 bytes.)
template <class T>
__global__ void __launch_bounds__(256) shuffle_rows_kernel(const T *__restrict__ in, T *__restrict__ out, long long rows, int units, int G,
                                                           const long long *__restrict__ perm, int *errflag) {
  const int per = 256 / G, sub = threadIdx.x % G;
  const long long r = (long long)blockIdx.x * per + threadIdx.x / G;
  if (r >= rows) return;
  const long long p = perm[r];
  if (p < 0 || p >= rows) { if (sub == 0) atomicOr(errflag, 1); return; }
  const T *src = in + r * units;
  T *dst = out + p * units;
  for (int u0 = sub; u0 < units; u0 += 4 * G) {
    T v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) if (u0 + k * G < units) v[k] = src[u0 + k * G];
#pragma unroll
    for (int k = 0; k < 4; ++k) if (u0 + k * G < units) dst[u0 + k * G] = v[k];
  }
}

// A random permutation is the indices in the order of (44 hashed bits, index); ties, vanishingly rare, keep index order.
__device__ __forceinline__ unsigned long long randperm_hash(unsigned long long seed, long long i) {
  return pbg_mix64(seed ^ pbg_mix64((unsigned long long)i + 0x51ED270B0F1ull)) >> 20;
}

// Up to RP_MAX indices in two kernels: the hash is uniform, so its top bits deal the indices to buckets of 350 to 700 (of up
// to 2,048 beyond 1.4 million indices), which a CTA sorts in shared memory.  A bucket has room for RP_CAP; one that overflows (a thousand standard
// deviations away) raises the error word's bit 8 and the caller takes the general sort.  Keys in a bucket: the remaining
// hash bits above the index (55 bits together), one comparison for both.  (Four radix passes of three launches took 260 us for
// 269,507 indices.)
#define RP_CAP 4096
#define RP_MAX (1ll << 22)
#define RP_MAX_BUCKETS 2048
static int rp_index_bits(long long n) { int b = 1; while ((n - 1) >> b) ++b; return b; }
static int rp_bits(long long n) { int b = 0; while ((n >> b) > 700 && (1 << b) < RP_MAX_BUCKETS) ++b; return b; }

__global__ void __launch_bounds__(256) randperm_deal_kernel(long long n, unsigned long long seed, int bits, int index_bits, unsigned long long *buckets, unsigned int *count,
                                                            unsigned int *count_next, int *errflag) {
  __shared__ unsigned int cnt[RP_MAX_BUCKETS];
  const int nb = 1 << bits, t = threadIdx.x;
  if (blockIdx.x == 0) for (int i = t; i < RP_MAX_BUCKETS; i += 256) count_next[i] = 0u;      // last read by the call before this one
  for (int i = t; i < nb; i += 256) cnt[i] = 0u;
  __syncthreads();
  unsigned long long h[8];
  unsigned int at[8];
  const long long i0 = (long long)blockIdx.x * 2048 + t;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const long long i = i0 + u * 256;
    if (i < n) { h[u] = randperm_hash(seed, i); at[u] = atomicAdd(&cnt[h[u] >> (44 - bits)], 1u); }
  }
  __syncthreads();
  for (int i = t; i < nb; i += 256) cnt[i] = cnt[i] ? atomicAdd(&count[i], cnt[i]) : 0u;   // where this CTA's part of the bucket begins
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const long long i = i0 + u * 256;
    if (i >= n) continue;
    const unsigned int b = (unsigned int)(h[u] >> (44 - bits)), pos = cnt[b] + at[u];
    if (pos < RP_CAP) buckets[(size_t)b * RP_CAP + pos] = (h[u] & ((1ull << (44 - bits)) - 1ull)) << index_bits | (unsigned long long)i;
    else atomicOr(errflag, 256);
  }
}

// One CTA per bucket orders its keys by counting: a thousand bins of the hash's next bits, at most a few keys in each, then
// every key counts the smaller ones of its own bin.  Five barriers whatever the size; the bitonic sort of the keys before it
// was 55 steps in a row, 27 us for 269,507 indices (7.3 us now).  The indices leave behind the smaller buckets'.
#define RP_SORT_THREADS 512
#define RP_BIN_BITS 10
__global__ void __launch_bounds__(RP_SORT_THREADS) randperm_sort_kernel(const unsigned long long *__restrict__ buckets, const unsigned int *__restrict__ count,
                                                                        int key_bits, int index_bits, long long *__restrict__ out) {
  constexpr int PER = RP_CAP / RP_SORT_THREADS, WARPS = RP_SORT_THREADS / 32;
  __shared__ unsigned long long key[RP_CAP];
  __shared__ unsigned int start[(1 << RP_BIN_BITS) + 1];      // the bins' counts, then where each begins
  __shared__ unsigned int below[WARPS], bins[WARPS];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5, b = blockIdx.x, shift = key_bits - RP_BIN_BITS;
  const int n = count[b] < RP_CAP ? (int)count[b] : RP_CAP;
  start[t] = start[t + RP_SORT_THREADS] = 0u;
  unsigned int s = 0u;
  for (int i = t; i < b; i += RP_SORT_THREADS) s += count[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) below[w] = s;
  unsigned long long k[PER];
  unsigned int at[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u)
    if (t + u * RP_SORT_THREADS < n) k[u] = buckets[(size_t)b * RP_CAP + t + u * RP_SORT_THREADS];
  __syncthreads();
#pragma unroll
  for (int u = 0; u < PER; ++u)
    if (t + u * RP_SORT_THREADS < n) at[u] = atomicAdd(&start[k[u] >> shift], 1u);
  __syncthreads();
  const unsigned int c0 = start[2 * t], c1 = start[2 * t + 1];
  unsigned int incl = c0 + c1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const unsigned int x = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += x; }
  if (lane == 31) bins[w] = incl;
  __syncthreads();
  unsigned int base = 0u, first = incl - c0 - c1;
#pragma unroll
  for (int u = 0; u < WARPS; ++u) { base += below[u]; first += u < w ? bins[u] : 0u; }
  start[2 * t] = first;
  start[2 * t + 1] = first + c0;
  if (t == 0) start[1 << RP_BIN_BITS] = (unsigned int)n;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < PER; ++u)
    if (t + u * RP_SORT_THREADS < n) key[start[k[u] >> shift] + at[u]] = k[u];
  __syncthreads();
  for (int i = t; i < n; i += RP_SORT_THREADS) {
    const unsigned long long x = key[i];
    unsigned int pos = start[x >> shift];
    for (unsigned int j = pos, end = start[(x >> shift) + 1]; j < end; ++j) pos += key[j] < x;
    out[base + pos] = (long long)(x & ((1ull << index_bits) - 1ull));
  }
}

// the general form, any length: keys for the radix sort
__global__ void randperm_keys_kernel(long long n, unsigned long long seed, unsigned long long *keys, unsigned int *vals) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  keys[i] = randperm_hash(seed, i);
  vals[i] = (unsigned int)i;
}
__global__ void widen_kernel(const unsigned int *__restrict__ vals, long long n, long long *__restrict__ out) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (long long)vals[i];
}

// Per-relation tables of a sub_bucket call, in device memory: [R] lhs permutation pointers, [R] rhs permutation
// pointers, [R] lhs entity counts, [R] rhs entity counts, [R] lhs sub-partition sizes, [R] rhs sub-partition sizes.
struct SubBucketArgs {
  const long long *lhs, *rhs, *rel;
  long long n;
  const long long *const *lperm, *const *rperm;
  const long long *lcount, *rcount, *lsize, *rsize;
  int R, nl, nr, dynamic;
};
// The same tables inside the kernel's parameters, for up to SB_INLINE relations (no upload, no wait for it).
#define SB_INLINE 16
struct SubBucketTables { long long v[6 * SB_INLINE]; };

// the argument structure with its table pointers aimed at the tables in the parameters (in_dev null) or in device memory
__device__ __forceinline__ SubBucketArgs sub_bucket_bind(SubBucketArgs a, const SubBucketTables &in, const long long *in_dev) {
  const long long *t = in_dev ? in_dev : in.v;
  a.lperm = (const long long *const *)t;
  a.rperm = (const long long *const *)(t + a.R);
  a.lcount = t + 2 * a.R; a.rcount = t + 3 * a.R; a.lsize = t + 4 * a.R; a.rsize = t + 5 * a.R;
  return a;
}

// permuted offsets of edge e; false (and the error word set) when an id is outside its table
__device__ __forceinline__ bool sub_bucket_offsets(const SubBucketArgs &a, long long e, long long &lo, long long &ro, long long &relid, int *errflag) {
  relid = a.dynamic ? 0 : a.rel[e];
  if (relid < 0 || relid >= a.R) { atomicOr(errflag, 4); return false; }          // "rel > numRelations" (util.cpp:320-322)
  long long l = a.lhs[e], r = a.rhs[e];
  if (l < 0 || l >= a.lcount[relid] || r < 0 || r >= a.rcount[relid]) { atomicOr(errflag, 1); return false; }
  lo = a.lperm[relid][l];
  ro = a.rperm[relid][r];
  if (lo < 0 || lo >= a.lcount[relid] || ro < 0 || ro >= a.rcount[relid]) { atomicOr(errflag, 1); return false; }
  return true;
}

// Up to SB_BINS - 1 sub-buckets (127 x 127 need more): stable counting sort in three launches that carry the edges along --
//   sub_bucket_hist     every warp owns a run of consecutive edges, keeps their keys and counts them into hist[key][warp]
//   sub_bucket_scan     one CTA per key: exclusive scan of its row of warp counts; the row's total is the sub-bucket's size
//   sub_bucket_scatter  every warp walks its run in order and writes each edge's offsets to its place
// (Keys, a radix pass over (key, index) pairs, a gather and binary searches for the sizes were six launches.)
// Runs are 64 edges up to 255 sub-buckets (an edge is a chain of three dependent reads, and a run walks its 32-edge rows
// one after the other), 256 above (the table of counts grows with both).
static inline int sb_run(int nb) { return nb < 256 ? 64 : 256; }
#define SB_WARPS 4
#define SB_BINS 1024
__global__ void __launch_bounds__(32 * SB_WARPS) sub_bucket_hist(SubBucketArgs args, const __grid_constant__ SubBucketTables in, const long long *in_dev, unsigned short *keys,
                                                                 unsigned int *hist, int nwarps, int run, int *errflag) {
  __shared__ unsigned int cnt[SB_WARPS][SB_BINS];
  const SubBucketArgs a = sub_bucket_bind(args, in, in_dev);
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31, wg = blockIdx.x * SB_WARPS + wl, nb = a.nl * a.nr;
  if (wg >= nwarps) return;
  for (int i = lane; i <= nb; i += 32) cnt[wl][i] = 0u;
  __syncwarp();
  for (int it = 0; it < run / 32; ++it) {
    const long long e = (long long)wg * run + it * 32 + lane;
    int key = nb;                                            // edges that cannot be placed come last
    if (e < a.n) {
      long long lo, ro, relid;
      if (sub_bucket_offsets(a, e, lo, ro, relid, errflag)) key = (int)(lo / a.lsize[relid]) * a.nr + (int)(ro / a.rsize[relid]);
      keys[e] = (unsigned short)key;
      atomicAdd(&cnt[wl][key], 1u);
    }
  }
  __syncwarp();
  for (int i = lane; i <= nb; i += 32) hist[(size_t)i * nwarps + wg] = cnt[wl][i];
}

// Eight counts per thread and round, all in flight together: the rounds are a chain of load, scan and barrier, and one count
// per thread took five of them for 269,507 edges (9.3 us, 6.1 us now).
__global__ void __launch_bounds__(1024) sub_bucket_scan(unsigned int *hist, int nwarps, int nb, unsigned int *totals, long long *counts) {
  constexpr int PER = 8;
  __shared__ unsigned int part[32];
  unsigned int *row = hist + (size_t)blockIdx.x * nwarps;
  const int t = threadIdx.x, lane = t & 31, wl = t >> 5;
  unsigned int carry = 0u;
  for (int i0 = 0; i0 < nwarps; i0 += 1024 * PER) {
    const int i = i0 + t * PER;
    unsigned int v[PER], sum = 0u;
#pragma unroll
    for (int u = 0; u < PER; ++u) v[u] = i + u < nwarps ? row[i + u] : 0u;
#pragma unroll
    for (int u = 0; u < PER; ++u) sum += v[u];
    unsigned int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const unsigned int x = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += x; }
    if (lane == 31) part[wl] = incl;
    __syncthreads();
    unsigned int upto = part[lane];                           // every warp scans the 32 parts for itself
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const unsigned int x = __shfl_up_sync(0xffffffffu, upto, o); if (lane >= o) upto += x; }
    const unsigned int lower = __shfl_sync(0xffffffffu, upto, wl > 0 ? wl - 1 : 0);
    unsigned int at = carry + (wl > 0 ? lower : 0u) + incl - sum;
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      if (i + u < nwarps) row[i + u] = at;
      at += v[u];
    }
    carry += __shfl_sync(0xffffffffu, upto, 31);
    __syncthreads();
  }
  if (t == 0) {
    totals[blockIdx.x] = carry;
    if (blockIdx.x < nb) counts[blockIdx.x] = carry;
  }
}

__global__ void __launch_bounds__(32 * SB_WARPS) sub_bucket_scatter(SubBucketArgs args, const __grid_constant__ SubBucketTables in, const long long *in_dev,
                                                                    const unsigned short *__restrict__ keys, const unsigned int *__restrict__ hist,
                                                                    const unsigned int *__restrict__ totals, int nwarps, int run, long long *lhs_out, long long *rhs_out,
                                                                    long long *rel_out, int *errflag) {
  __shared__ unsigned int base[SB_BINS], pos[SB_WARPS][SB_BINS];
  __shared__ unsigned int wsum[SB_WARPS];
  const SubBucketArgs a = sub_bucket_bind(args, in, in_dev);
  const int t = threadIdx.x, wl = t >> 5, lane = t & 31, wg = blockIdx.x * SB_WARPS + wl, nb = a.nl * a.nr;
  // where each sub-bucket begins: exclusive scan of the totals, a contiguous part per thread
  {
    const int per = (nb + 32 * SB_WARPS - 1) / (32 * SB_WARPS), lo = t * per < nb ? t * per : nb, hi = lo + per < nb ? lo + per : nb;
    unsigned int s = 0u;
    for (int i = lo; i < hi; ++i) s += totals[i];
    unsigned int incl = s;
    for (int o = 1; o < 32; o <<= 1) { const unsigned int x = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += x; }
    if (lane == 31) wsum[wl] = incl;
    __syncthreads();
    unsigned int at = incl - s;
    for (int u = 0; u < wl; ++u) at += wsum[u];
    for (int i = lo; i < hi; ++i) { base[i] = at; at += totals[i]; }
    __syncthreads();
  }
  if (wg >= nwarps) return;
  for (int i = lane; i < nb; i += 32) pos[wl][i] = base[i] + hist[(size_t)i * nwarps + wg];
  __syncwarp();
  for (int it = 0; it < run / 32; ++it) {
    const long long e = (long long)wg * run + it * 32 + lane;
    const int key = e < a.n ? (int)keys[e] : nb;
    const unsigned int peers = __match_any_sync(0xffffffffu, key), before = __popc(peers & ((1u << lane) - 1u));
    unsigned int dst = 0u;
    if (key < nb) dst = pos[wl][key] + before;
    __syncwarp();                                            // every peer has read pos[] by now
    if (key < nb && before == 0u) pos[wl][key] += __popc(peers);
    __syncwarp();
    long long lo, ro, relid;
    if (key < nb && sub_bucket_offsets(a, e, lo, ro, relid, errflag)) {
      lhs_out[dst] = lo % a.lsize[relid];
      rhs_out[dst] = ro % a.rsize[relid];
      rel_out[dst] = a.rel[e];
    }
  }
}

// The general form: keys and edge numbers through the radix sort.
__global__ void sub_bucket_keys_kernel(SubBucketArgs a, unsigned long long *keys, unsigned int *vals, int *errflag) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.n) return;
  long long lo, ro, relid;
  unsigned long long key = (unsigned long long)a.nl * a.nr;            // edges that cannot be placed sort to the end
  if (sub_bucket_offsets(a, e, lo, ro, relid, errflag))
    key = (unsigned long long)(lo / a.lsize[relid]) * a.nr + (unsigned long long)(ro / a.rsize[relid]);
  keys[e] = key;
  vals[e] = (unsigned int)e;
}

__global__ void sub_bucket_emit_kernel(SubBucketArgs a, const unsigned long long *__restrict__ keys, const unsigned int *__restrict__ vals,
                                       long long *lhs_out, long long *rhs_out, long long *rel_out, int *errflag) {
  long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= a.n) return;
  if (keys[q] >= (unsigned long long)a.nl * a.nr) return;
  long long e = vals[q], lo, ro, relid;
  if (!sub_bucket_offsets(a, e, lo, ro, relid, errflag)) return;
  lhs_out[q] = lo % a.lsize[relid];
  rhs_out[q] = ro % a.rsize[relid];
  rel_out[q] = a.rel[e];
}

// counts[b] = number of sorted keys equal to b (one thread per sub-bucket, two binary searches)
__global__ void sub_bucket_counts_kernel(const unsigned long long *__restrict__ keys, long long n, int nb, long long *counts) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nb) return;
  auto lower = [&](unsigned long long v) {
    long long lo = 0, hi = n;
    while (lo < hi) { long long mid = (lo + hi) >> 1; if (keys[mid] < v) lo = mid + 1; else hi = mid; }
    return lo;
  };
  counts[b] = lower((unsigned long long)b + 1) - lower((unsigned long long)b);
}

static inline int grid_for(long long n, int threads) { return (int)((n + threads - 1) / threads); }

int launch_reverse_permutation(const long long *perm, long long n, long long *out, int *errflag, cudaStream_t st) {
  if (n > 0) pbg_launch_in_order(reverse_permutation_kernel, grid_for(n, 256), 256, 0, st, perm, n, out, errflag);
  return n > 0;
}

template <class T>
static void shuffle_as(const void *in, void *out, long long rows, long long row_bytes, const long long *perm, int *errflag, cudaStream_t st) {
  const int units = (int)(row_bytes / (long long)sizeof(T));
  int G = 1;
  while (G < 256 && 4 * G < units) G *= 2;
  pbg_launch_in_order(shuffle_rows_kernel<T>, grid_for(rows, 256 / G), 256, 0, st, (const T *)in, (T *)out, rows, units, G, perm, errflag);
}

int launch_shuffle_rows(const void *in, void *out, long long rows, long long row_bytes, const long long *perm, int *errflag, cudaStream_t st) {
  if (rows <= 0 || row_bytes <= 0) return 0;
  const uintptr_t al = (uintptr_t)in | (uintptr_t)out | (uintptr_t)row_bytes;
  if (al % 16 == 0) shuffle_as<uint4>(in, out, rows, row_bytes, perm, errflag, st);
  else if (al % 8 == 0) shuffle_as<unsigned long long>(in, out, rows, row_bytes, perm, errflag, st);
  else if (al % 4 == 0) shuffle_as<unsigned int>(in, out, rows, row_bytes, perm, errflag, st);
  else shuffle_as<unsigned char>(in, out, rows, row_bytes, perm, errflag, st);
  return 1;
}

// scratch of the two-kernel randperm (0: n is too large for it): counters, which start at zero, then the buckets
size_t pbg_randperm_bytes(long long n) {
  if (n > RP_MAX) return 0;
  return pbg_randperm_counter_bytes() + ((size_t)RP_CAP * 8 << rp_bits(n));
}
size_t pbg_randperm_counter_bytes() { return 2 * RP_MAX_BUCKETS * sizeof(unsigned int); }
int launch_randperm_dealt(char *mem, unsigned turn, long long n, unsigned long long seed, long long *out, int *errflag, cudaStream_t st) {
  const int bits = rp_bits(n), index_bits = rp_index_bits(n);
  unsigned int *counts = (unsigned int *)mem;
  unsigned int *cur = counts + (turn & 1) * RP_MAX_BUCKETS, *next = counts + ((turn + 1) & 1) * RP_MAX_BUCKETS;
  unsigned long long *buckets = (unsigned long long *)(mem + pbg_randperm_counter_bytes());
  pbg_launch_in_order(randperm_deal_kernel, grid_for(n, 2048), 256, 0, st, n, seed, bits, index_bits, buckets, cur, next, errflag);
  pbg_launch_in_order(randperm_sort_kernel, 1 << bits, RP_SORT_THREADS, 0, st, buckets, cur, 44 - bits + index_bits, index_bits, out);
  return 2;
}

int launch_randperm(SortPlan &sp, long long n, unsigned long long seed, long long *out, cudaStream_t st) {
  if (n <= 0) return 0;
  pbg_launch_in_order(randperm_keys_kernel, grid_for(n, 256), 256, 0, st, n, seed, sp.keys[0], sp.vals[0]);
  int launches = 1 + pbg_sort(sp, (int)n, 44, st);
  pbg_launch_in_order(widen_kernel, grid_for(n, 256), 256, 0, st, sp.vals[sp.result], n, out);
  return launches + 1;
}

// tables: [6 R] in host memory; tables_dev: where they lie on the device when R is above SB_INLINE (pbg_sub_bucket_inline)
bool pbg_sub_bucket_inline(int R) { return R <= SB_INLINE; }
int launch_sub_bucket(SortPlan &sp, const long long *lhs, const long long *rhs, const long long *rel, long long n, int R, const long long *tables,
                      const long long *tables_dev, int nl, int nr, int dynamic, long long *lhs_out, long long *rhs_out, long long *rel_out,
                      long long *counts, int *errflag, cudaStream_t st) {
  SubBucketArgs a;
  a.lhs = lhs; a.rhs = rhs; a.rel = rel; a.n = n; a.R = R; a.nl = nl; a.nr = nr; a.dynamic = dynamic;
  a.lperm = (const long long *const *)tables_dev;
  a.rperm = (const long long *const *)(tables_dev + R);
  a.lcount = tables_dev + 2 * R; a.rcount = tables_dev + 3 * R; a.lsize = tables_dev + 4 * R; a.rsize = tables_dev + 5 * R;
  const int nb = nl * nr;
  if (n <= 0) return 0;
  if (nb < SB_BINS) {
    SubBucketTables in;
    const bool inl = pbg_sub_bucket_inline(R);
    for (int i = 0; i < 6 * SB_INLINE; ++i) in.v[i] = inl && i < 6 * R ? tables[i] : 0;
    const int run = sb_run(nb), nwarps = (int)((n + run - 1) / run), ctas = (nwarps + SB_WARPS - 1) / SB_WARPS;
    unsigned short *keys = (unsigned short *)sp.keys[0];
    unsigned int *totals = sp.hist + (size_t)(nb + 1) * nwarps;
    pbg_launch_in_order(sub_bucket_hist, ctas, 32 * SB_WARPS, 0, st, a, in, inl ? nullptr : tables_dev, keys, sp.hist, nwarps, run, errflag);
    pbg_launch_in_order(sub_bucket_scan, nb + 1, 1024, 0, st, sp.hist, nwarps, nb, totals, counts);
    pbg_launch_in_order(sub_bucket_scatter, ctas, 32 * SB_WARPS, 0, st, a, in, inl ? nullptr : tables_dev, keys, sp.hist, totals, nwarps, run, lhs_out, rhs_out, rel_out, errflag);
    return 3;
  }
  pbg_launch_in_order(sub_bucket_keys_kernel, grid_for(n, 256), 256, 0, st, a, sp.keys[0], sp.vals[0], errflag);
  int bits = 1;
  while ((1ll << bits) <= nb) ++bits;                                   // keys run up to nb (the "cannot be placed" key)
  int launches = 1 + pbg_sort(sp, (int)n, bits, st);
  pbg_launch_in_order(sub_bucket_emit_kernel, grid_for(n, 256), 256, 0, st, a, sp.keys[sp.result], sp.vals[sp.result], lhs_out, rhs_out, rel_out, errflag);
  pbg_launch_in_order(sub_bucket_counts_kernel, grid_for(nb, 128), 128, 0, st, sp.keys[sp.result], n, nb, counts);
  return launches + 2;
}
