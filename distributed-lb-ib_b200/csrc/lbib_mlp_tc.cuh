/*
 * The surrogate MLP's GEMM on the 5th-generation tensor cores (sm_100a):
 * tcgen05.mma kind::f16 with BF16 operands in shared memory and the FP32
 * accumulator in tensor memory (TMEM), read back with tcgen05.ld for the
 * bias / GELU epilogue.
 *
 * C[M][N] = sum_k A(m,k) B(k,n).  One CTA computes a 128 x BN tile: TMEM
 * lane i holds row m0 + i, BN FP32 columns.
 *
 * Every BF16 matrix of the network (activations, dZ, weights) lies in global
 * memory as 16-byte chunks of 8 consecutive columns, in blocks of `blk`
 * rows: chunk (c, r) of columns 8c..8c+7 of row r at chunk index
 * ((r / blk) * C + c) * blk + r % blk, with C the chunks of a row.  Eight
 * consecutive chunks are one 8 x 16-byte "core matrix" of the tensor cores'
 * no-swizzle layout, whichever way the matrix is used -- rows as M or N and
 * columns as K (K-major), or columns as M or N and rows as K (MN-major) --
 * so that with blk = 128 (activations, dZ) or 32 (weights, each also kept
 * transposed) a K slice of an operand is ONE contiguous run of global
 * memory, as it lies in the operand buffer.  An epilogue thread, which holds
 * 8 columns of one row, writes one chunk, a warp's 32 rows contiguous.
 *
 * These products are small (K is a layer's width or a share of the batch)
 * and bound by latency.  For the 80 KB of a tile with K = 256: the threads'
 * own 16-byte cp.async from row-major matrices took ~6000 cycles to issue;
 * bulk copies of 0.5 to 2 KB runs ~65 cycles each, 48 or more of them; one
 * copy per operand and slice of 128 (four in all) is what remains.
 *
 * Operands are staged in K slices of 128 (eight MMAs of K = 16), kStages
 * slices deep: a K of 256 is in flight whole.  One thread issues the copies
 * of a slice to its mbarrier, another its MMAs when that mbarrier completes,
 * and commits them to a second one, on which a refill of the buffer waits.
 * Every wait is bounded: on a timeout the CTA records an error, skips the
 * rest and still frees its TMEM.
 */
#ifndef LBIB_MLP_TC_CUH
#define LBIB_MLP_TC_CUH

#include <stdint.h>

#include <cuda_bf16.h>

namespace lbib_tc {

constexpr int BM = 128;   /* rows per CTA = TMEM lanes                 */
constexpr int BK = 128;   /* K per stage: up to eight MMAs of K = 16   */
constexpr int NT = 512;   /* threads per CTA: four warps per TMEM quadrant */
constexpr int kStages = 2;   /* K slices staged at once                  */
constexpr long kSpin = 1L << 24;   /* try_wait polls before giving up  */

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

/* Shared-memory matrix descriptor: canonical layout, no swizzle. */
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);           /* start address        [0,14)  */
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;         /* leading byte offset  [16,30) */
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;         /* stride byte offset   [32,46) */
  d |= (uint64_t)1 << 46;                              /* descriptor version 1 [46,48) */
  return d;                                            /* base offset 0, no swizzle    */
}

/* Instruction descriptor: BF16 x BF16 -> FP32, M x N; a_mn / b_mn: the
 * operand's shared-memory tile is MN-major (core-matrix rows run along K,
 * each holding 8 consecutive M or N elements) instead of K-major. */
__host__ __device__ constexpr uint32_t instr_desc_bf16(int M, int N, bool a_mn = false, bool b_mn = false) {
  return (1u << 4)                      /* D format F32   [4,6)   */
         | (1u << 7)                    /* A format BF16  [7,10)  */
         | (1u << 10)                   /* B format BF16  [10,13) */
         | ((a_mn ? 1u : 0u) << 15)     /* A major        [15]    */
         | ((b_mn ? 1u : 0u) << 16)     /* B major        [16]    */
         | ((uint32_t)(N >> 3) << 17)   /* N / 8          [17,23) */
         | ((uint32_t)(M >> 4) << 24);  /* M / 16         [24,29) */
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

/* Wait for completion `parity` of the barrier; false after kSpin polls. */
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t a = smem_u32(bar);
  for (long i = 0; i < kSpin; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

template <int NCOL>
__device__ __forceinline__ void tmem_alloc(uint32_t* slot) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
               "r"((uint32_t)NCOL)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

template <int NCOL>
__device__ __forceinline__ void tmem_free(uint32_t taddr) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"((uint32_t)NCOL) : "memory");
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
      :
      : "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

/* 8 consecutive FP32 columns of this thread's TMEM lane. */
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

/* `bytes` (a multiple of 16) global -> shared by the bulk copy engine;
 * the barrier counts them. */
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

/* Programmatic dependent launch: let the next kernel of the stream start
 * its set-up; wait until the kernels before this one are done and their
 * writes visible (nothing global is read or written before that). */
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

/* An operand X(r, k) in the chunk layout above: the matrix's rows are the
 * tile's rows and its columns K (mn = 0), or the other way round (mn = 1,
 * blk = 128 = BK only). */
struct Operand {
  const __nv_bfloat16* p;
  int C, blk, mn;
};

/* All CTAs of the cluster; shared-memory writes before it are visible to
 * their readers after it. */
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
/* A float at the same shared-memory place of CTA `rank` of the cluster. */
__device__ __forceinline__ float ld_cluster(const float* p, uint32_t rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

/* The operand's rows [r0, r0 + R) (r0 a multiple of R; R = blk when K-major)
 * at K elements [k0, k0 + kn), k0 a multiple of BK and kn <= BK of 16: its
 * bytes, and their copy to shared memory at s.  MN-major copies the whole
 * block of BK matrix rows, of the columns that exist: what lies in the buffer
 * for the others only reaches rows or columns of the tile that are not
 * written. */
template <int R>
__device__ __forceinline__ uint32_t slice_bytes(const Operand& X, int r0, int kn) {
  return X.mn ? min(R / 8, X.C - r0 / 8) * BK * 16 : R * kn * 2;
}
template <int R>
__device__ __forceinline__ void fetch_slice(uint32_t s, const Operand& X, int r0, int k0, int kn, uint64_t* bar) {
  const long chunk = X.mn ? ((long)(k0 / BK) * X.C + r0 / 8) * BK : ((long)(r0 / R) * X.C + k0 / 8) * R;
  bulk_copy(s, X.p + chunk * 8, slice_bytes<R>(X, r0, kn), bar);
}

/* The descriptor of a staged operand's K = 16 step j: core matrices along K
 * are 16 R bytes apart and along the rows 128 (K-major), or 128 and 16 BK
 * (MN-major); the leading byte offset is the one along K. */
template <int R>
__device__ __forceinline__ uint64_t operand_desc(uint32_t s, int mn, int j) {
  return mn ? smem_desc(s + j * 2 * 128, 128, BK * 16) : smem_desc(s + j * 2 * R * 16, R * 16, 128);
}

}  // namespace lbib_tc

#endif
