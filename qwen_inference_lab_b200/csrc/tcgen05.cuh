// What the kernels that issue tcgen05.mma share: barriers, TMA loads, descriptors, the MMA itself, reads of tensor memory.
//
// One thread issues copies, MMAs and commits, but its whole warp walks the loop around them, and the instructions are
// predicated (`leader`) instead of branched around.  Their operands live in uniform registers.  Where the warp is known to
// run as one (its number from uniform_warp(), no `if (lane == 0)`) they are computed there; in a branch of one lane each
// of them is computed per thread and moved: 65 cycles of an MMA's issue and 140 of a copy's, so that a stage of 64 k took the
// issuing threads of the two-block tile product 640 cycles whatever there was to multiply (now 190).
#pragma once
#include "common.cuh"
#include <cuda.h>

__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
__device__ __forceinline__ unsigned uniform(unsigned v) { return __shfl_sync(0xffffffffu, v, 0); }
// Is this lane the one that issues?  The same lane every time; the warp is whole.
__device__ __forceinline__ bool elect_one() {
    unsigned p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes, bool leader) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t"
                 "@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}\n"
                 ::"r"(smem_u32(bar)), "r"(bytes), "r"((unsigned)leader) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned done;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return done != 0;
}
// Bounded wait: false when the barrier did not complete in about a second.
#define TC_WAIT_CYCLES 2000000000ll
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long start = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - start > TC_WAIT_CYCLES) return false;
    }
    return true;
}

// The same for a whole warp, which goes on or gives up together: lanes that left by themselves would be missing from the
// warp-wide instructions that follow.
__device__ __forceinline__ bool warp_mbar_wait(unsigned long long* bar, unsigned parity) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity)) != 0;
}

// Shared-memory matrix descriptor: K-major operand, rows of 128 bytes, 128-byte swizzle, groups of 8
// rows 1024 bytes apart (the layout a TMA load with CU_TENSOR_MAP_SWIZZLE_128B writes).
__device__ __forceinline__ unsigned long long umma_desc(unsigned smem_addr) {
    unsigned long long d = 0;
    d |= (unsigned long long)((smem_addr & 0x3FFFF) >> 4);          // start address, 16-byte units
    d |= (unsigned long long)1 << 16;                                // leading byte offset (unused with swizzle)
    d |= (unsigned long long)(1024 >> 4) << 32;                      // stride byte offset: 8 rows
    d |= (unsigned long long)1 << 46;                                // descriptor version of sm_100
    d |= (unsigned long long)2 << 61;                                // 128-byte swizzle
    return d;
}
// Instruction descriptor: bfloat16 x bfloat16 -> float32, both operands K-major.
__device__ __forceinline__ unsigned umma_idesc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(m >> 4) << 24);
}
__device__ __forceinline__ void umma_bf16(unsigned tmem_d, unsigned long long desc_a, unsigned long long desc_b,
                                          unsigned idesc, unsigned accumulate, bool leader) {
    asm volatile("{\n\t.reg .pred p, q;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "setp.ne.b32 q, %5, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                 ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"((unsigned)leader) : "memory");
}
// Arrives on the barrier once the MMAs that this thread issued so far are done.
__device__ __forceinline__ void umma_commit(unsigned long long* bar, bool leader) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %1, 0;\n\t"
                 "@p tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n"
                 ::"r"(smem_u32(bar)), "r"((unsigned)leader) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* smem, const CUtensorMap* map, unsigned long long* bar, int x, int y, bool leader) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
                 "@p cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}\n"
                 ::"r"(smem_u32(smem)), "l"((unsigned long long)map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"((unsigned)leader) : "memory");
}
// The same with the hint that these bytes are the first to leave L2: a weight tile that only one tile of tokens reads
// (a product of at most 128 rows) is read once a step.
__device__ __forceinline__ unsigned long long stream_policy() {
    unsigned long long policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(policy));
    return policy;
}
__device__ __forceinline__ void tma_load_2d_stream(void* smem, const CUtensorMap* map, unsigned long long* bar, int x, int y,
                                                   unsigned long long policy, bool leader) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
                 "@p cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;\n\t}\n"
                 ::"r"(smem_u32(smem)), "l"((unsigned long long)map), "r"(smem_u32(bar)), "r"(x), "r"(y), "l"(policy), "r"((unsigned)leader) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// 32 columns of this lane of tensor memory; a warp-wide instruction.
__device__ __forceinline__ void tmem_load_32(unsigned taddr, float (&v)[32]) {
    unsigned r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
