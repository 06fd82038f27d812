// The 5th-generation tensor core of sm_100a as the kernels here use it: tensor memory (allocation, loads and stores of
// a thread's lane), the matrix instruction issued by one thread with its operands described in shared memory, the
// commit that signals an mbarrier when the instructions issued so far are done, and the descriptors. One CTA per tile
// (cta_group::1) and two CTAs on one tile (cta_group::2, `_pair`).
#pragma once
#include "pipeline.cuh"

namespace nibt {

using nibp::smem_u32;

// ---- one thread of a converged warp. The tensor core and the copy engine take their operands from the warp's uniform
// registers. A role that a whole warp runs, in loops whose bounds, waits and addresses are the warp's and not a thread's, with
// only the instructions themselves behind elect_one(), keeps them there; a role that lane 0 runs alone has every operand of
// every instruction moved over first (about 150 cycles for one tcgen05.mma: more than the instruction takes).
__device__ __forceinline__ bool elect_one() {
    unsigned is;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(is));
    return is != 0;
}
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
// a wait of the whole warp, with one answer
__device__ __forceinline__ bool warp_wait(unsigned long long* bar, unsigned parity) { return __all_sync(0xffffffffu, nibp::mbar_wait(bar, parity)); }

// ---- who may share an SM. With dependent launches a CTA of the next kernel can be resident beside CTAs of this one, and an allocation
// of tensor memory waits until columns are free: a CTA that held columns which a CTA of an earlier kernel still has to allocate
// would wait for that kernel's end for good. So CTAs that fit an SM's shared memory together fit its 512 columns together: two of the
// prompt attention's, or one of any product's and as many of the prompt attention's as fit beside it, and no two products'.
constexpr int SM_SHARED = 228 * 1024, CTA_RESERVED = 1024, SM_TMEM_COLS = 512;       // bytes, bytes, columns
constexpr int PROMPT_SMEM = 5 * 16384 + 1280, PROMPT_COLS = 256;                      // the prompt attention's smallest CTA
constexpr bool product_fits_tmem(int smem, int cols) {
    return 2 * (smem + CTA_RESERVED) > SM_SHARED &&
           cols + (SM_SHARED - smem - CTA_RESERVED) / (PROMPT_SMEM + CTA_RESERVED) * PROMPT_COLS <= SM_TMEM_COLS;
}
constexpr bool prompt_fits_tmem(int smem, int cols) { return smem >= PROMPT_SMEM && cols == PROMPT_COLS && 3 * (PROMPT_SMEM + CTA_RESERVED) > SM_SHARED; }

// ---- tensor memory: allocated and freed by one whole warp; the address arrives in shared memory
__device__ __forceinline__ void tmem_alloc(unsigned* dst_smem, unsigned cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(dst_smem)), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(unsigned addr, unsigned cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(unsigned* dst_smem, unsigned cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(dst_smem)), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc_pair(unsigned addr, unsigned cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(addr), "r"(cols) : "memory");
}
constexpr int tmem_cols(int n) { return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : n <= 256 ? 256 : 512; }

// ---- ordering of tensor-core work against the barriers and __syncthreads of the other threads
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// ---- the barrier gets one arrival when the instructions this thread has issued so far are done
__device__ __forceinline__ void tc_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
// ... the barrier at this offset in BOTH CTAs of the pair (a signal, not a copy: no data is multicast)
__device__ __forceinline__ void tc_commit_pair(unsigned long long* bar) {
    const unsigned short mask = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
                 ::"r"(smem_u32(bar)), "h"(mask) : "memory");
}

// ---- D[tmem] (+)= A[smem] . B[smem]^T, bfloat16 operands, 32-bit accumulation
__device__ __forceinline__ void tc_mma(unsigned d_tmem, unsigned long long a_desc, unsigned long long b_desc,
                                       unsigned idesc, bool accumulate) {
    const unsigned acc = accumulate ? 1u : 0u;
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tc_mma_pair(unsigned d_tmem, unsigned long long a_desc, unsigned long long b_desc,
                                            unsigned idesc, bool accumulate) {
    const unsigned acc = accumulate ? 1u : 0u;
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}

// ---- D[tmem] (+)= A[tmem] . B[smem]^T: A has a row per lane, two bfloat16 of K to a column (the even one below)
__device__ __forceinline__ void tc_mma_ts(unsigned d_tmem, unsigned a_tmem, unsigned long long b_desc, unsigned idesc, bool accumulate) {
    const unsigned acc = accumulate ? 1u : 0u;
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}

// ---- a thread's TMEM lane to and from registers. The values of a load may be used only after tmem_wait_ld();
// issue every load of a batch first and wait once: a load's latency is hundreds of cycles.
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16_async(unsigned addr, unsigned (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_ld16(unsigned addr, float (&v)[16]) {
    unsigned r[16];
    tmem_ld16_async(addr, r);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld32_async(unsigned addr, unsigned (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_st16(unsigned addr, const unsigned (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}

// ---- shared-memory matrix descriptors, 128-byte swizzle (cute/arch/mma_sm100_desc.hpp: SmemDescriptor)
// K-major operand tile: rows of 128 bytes (64 bfloat16 of K), groups of 8 rows 1024 bytes apart.
__device__ __forceinline__ unsigned long long desc_kmajor(unsigned smem_addr) {
    unsigned long long d = 0;
    d |= (unsigned long long)((smem_addr & 0x3FFFFu) >> 4);       // start address, bits [0,14)
    d |= (unsigned long long)1 << 16;                             // leading byte offset (unused with swizzle), encoded 1
    d |= (unsigned long long)(1024 >> 4) << 32;                   // stride byte offset: 8 rows * 128 bytes
    d |= (unsigned long long)1 << 46;                             // descriptor version of sm_100
    d |= (unsigned long long)2 << 61;                             // layout type: SWIZZLE_128B
    return d;
}
// MN-major operand (cute/atom/mma_traits_sm100.hpp, canonical layout ((8,n),(8,k)):((1,LBO),(8,SBO)) in 16-byte
// units): 64 elements of MN are contiguous in a 128-byte row, 8 rows of K form a 1024-byte group (SBO), the next 64
// elements of MN start `lbo_bytes` further on.
__device__ __forceinline__ unsigned long long desc_mnmajor(unsigned smem_addr, unsigned lbo_bytes) {
    unsigned long long d = 0;
    d |= (unsigned long long)((smem_addr & 0x3FFFFu) >> 4);
    d |= (unsigned long long)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (unsigned long long)(1024 >> 4) << 32;
    d |= (unsigned long long)1 << 46;
    d |= (unsigned long long)2 << 61;
    return d;
}
// Instruction descriptor (cute/arch/mma_sm100_desc.hpp: InstrDescriptor): D float, A and B bfloat16, A K-major,
// the instruction's M (128, or 256 for a pair) and N; b_mn: the B operand is MN-major.
__host__ __device__ constexpr unsigned instr_desc(int m, int n, bool b_mn = false) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn ? 1u : 0u) << 16) | ((unsigned)(n >> 3) << 17) | ((unsigned)(m >> 4) << 24);
}

}  // namespace nibt
