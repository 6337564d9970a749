// Device helpers shared by the tcgen05 kernels: bounded mbarrier waits, TMA tile loads, shared-memory
// matrix descriptors, and the host-side tensor-map encoders.
#pragma once
#include <cuda.h>

#include "pbg_common.cuh"

#define TC_WAIT_LIMIT 4000000

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int *errflag) {
  for (int it = 0; it < TC_WAIT_LIMIT; ++it) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
  }
  atomicOr(errflag, 2);
  return false;
}

// Place in a ring of stages: which one, and the parity of the pass over the ring.  The consumer of a stage waits for `parity`,
// its producer for the other one (a fresh barrier lets it through).  Counted, not divided out of a running number: in the plane
// tiers, whose number of stages is known at run time, a 64-bit division by it stood in front of every wait of the producer and
// of the thread that issues the products (two planes, 1000-row chunks at dimension 400: gradients 7.83 ms with it, 6.80 without;
// dual gradient of 20-chunk waves at dimension 100, three planes: 28.8 and 26.1 us).
struct StageRing {
  int s = 0;
  uint32_t parity = 0;
  __device__ __forceinline__ void next(int stages) { if (++s == stages) { s = 0; parity ^= 1u; } }
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
               :: "r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, int c3, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
               :: "r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar) : "memory");
}

__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, int c3, int c4, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
               :: "r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar) : "memory");
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t layout) {
  return ((uint64_t)((addr >> 4) & 0x3FFF)) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46) | ((uint64_t)layout << 61);
}

// One lane of a converged warp.  The warp that issues products runs its loop as a whole -- waits, counters and descriptors are
// the same in every lane, so that they live in uniform registers, which is where the instruction takes them from -- and one
// lane issues.
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(one));
  return one != 0;
}
// D (+)= A . B on shared-memory descriptors
__device__ __forceinline__ void mma_f16(uint32_t acc, uint64_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" :: "r"(acc), "l"(a), "l"(b), "r"(idesc), "r"(add ? 1u : 0u) : "memory");
}
__device__ __forceinline__ void mma_tf32(uint32_t acc, uint64_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}" :: "r"(acc), "l"(a), "l"(b), "r"(idesc), "r"(add ? 1u : 0u) : "memory");
}
// arrives on the barrier when the products issued so far are done
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}
// The descriptor of an operand `bytes` (a multiple of 16) further on: shared-memory addresses fit the field without a carry.
__device__ __forceinline__ uint64_t desc_at(uint64_t desc, uint32_t bytes) { return desc + (bytes >> 4); }

// 32 columns of this thread's tensor-memory lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                 "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
                 "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
                 "=r"(r[30]), "=r"(r[31]) : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- host side: tensor maps ---------------------------------------------------------------------
typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                             const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeFn get_encode() {
  static EncodeFn fn = nullptr;
  if (!fn) {
    cudaDriverEntryPointQueryResult q;
    void *p = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess) fn = (EncodeFn)p;
  }
  return fn;
}

// Every operand tile of a stage is ONE box, whatever it holds: a bulk tensor copy costs its issue and its own walk
// through the copy engine, a few hundred cycles each, and a stage of 32 k-values used to be up to fifteen of them (a box
// per plane, and per 32 or 64 columns of an MN-major operand).  An array is therefore described with its planes and its
// column blocks as dimensions of their own.
inline bool encode_map(CUtensorMap *tm, CUtensorMapDataType type, const void *base, int rank, const cuuint64_t *dims, const cuuint64_t *strides,
                       const cuuint32_t *box, CUtensorMapSwizzle swizzle) {
  EncodeFn enc = get_encode();
  if (!enc) return false;
  cuuint32_t es[5] = {1, 1, 1, 1, 1};
  return enc(tm, type, (cuuint32_t)rank, (void *)base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// fp32 arrays [nblk][rows][ld].  K-major operands and outputs: boxes of box_inner floats x box_rows rows (128-byte swizzle;
// 64 bytes wide: 64-byte swizzle), coordinates (column, row, block).
inline bool encode3(CUtensorMap *tm, const float *base, int inner, int rows, int nblk, int ld, long long blk_stride, int box_inner, int box_rows) {
  const cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)rows, (cuuint64_t)nblk};
  const cuuint64_t strides[2] = {(cuuint64_t)ld * 4, (cuuint64_t)blk_stride * 4};
  const cuuint32_t box[3] = {(cuuint32_t)box_inner, (cuuint32_t)box_rows, 1};
  return encode_map(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, base, 3, dims, strides, box, box_inner * 4 == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B);
}
// MN-major operands: `atoms` blocks of 32 columns x box_k rows, coordinates (0, k row, column block, block).  The last block
// of columns may reach past the row's end: what it brings belongs to output columns that are clipped.
inline bool encode3_mn(CUtensorMap *tm, const float *base, int inner, int rows, int nblk, int ld, long long blk_stride, int box_k, int atoms) {
  const cuuint64_t dims[4] = {32, (cuuint64_t)rows, (cuuint64_t)((inner + 31) / 32), (cuuint64_t)nblk};
  const cuuint64_t strides[3] = {(cuuint64_t)ld * 4, 128, (cuuint64_t)blk_stride * 4};
  const cuuint32_t box[4] = {32, (cuuint32_t)box_k, (cuuint32_t)atoms, 1};
  return encode_map(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, base, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B);
}

// bf16 plane arrays [nblk][npl][rows][ld].  K-major: all planes of 32 k-values x box_rows rows (64-byte swizzle), coordinates
// (k, row, 0, block).
inline bool encode4_planes(CUtensorMap *tm, const unsigned short *base, int npl, int inner, int rows, int rows_alloc, int nblk, int ld, int box_rows) {
  const cuuint64_t dims[4] = {(cuuint64_t)inner, (cuuint64_t)rows, (cuuint64_t)npl, (cuuint64_t)nblk};
  const cuuint64_t strides[3] = {(cuuint64_t)ld * 2, (cuuint64_t)rows_alloc * ld * 2, (cuuint64_t)npl * rows_alloc * ld * 2};
  const cuuint32_t box[4] = {32, (cuuint32_t)box_rows, (cuuint32_t)npl, 1};
  return encode_map(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B);
}
// MN-major: `atoms` blocks of 64 columns, each all planes of 32 rows (128-byte swizzle), coordinates (0, k row, 0, column
// block, block)
inline bool encode4_planes_mn(CUtensorMap *tm, const unsigned short *base, int npl, int inner, int rows, int rows_alloc, int nblk, int ld, int atoms) {
  const cuuint64_t dims[5] = {64, (cuuint64_t)rows, (cuuint64_t)npl, (cuuint64_t)((inner + 63) / 64), (cuuint64_t)nblk};
  const cuuint64_t strides[4] = {(cuuint64_t)ld * 2, (cuuint64_t)rows_alloc * ld * 2, 128, (cuuint64_t)npl * rows_alloc * ld * 2};
  const cuuint32_t box[5] = {64, 32, (cuuint32_t)npl, (cuuint32_t)atoms, 1};
  return encode_map(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, 5, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}
