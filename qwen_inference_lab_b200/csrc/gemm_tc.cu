// C[M,N] = A[M,K] * W[N,K]^T (+ bias) (+ residual) in bfloat16 with float32
// accumulation on the fifth-generation tensor cores: the projections of prompt
// portions (M from a few dozen to thousands of tokens).
//
// Blackwell-native structure, one persistent block per SM, 320 threads:
//   warp 0      walks the stages of a 4-stage ring; its elected lane arms a stage's mbarrier with the
//               byte count and issues the TMA loads (cp.async.bulk.tensor, 128-byte swizzle) of a
//               128 x 64 tile of A and a 256 x 64 tile of W;
//   warp 1      walks them behind it; its elected lane issues tcgen05.mma (128 x 256 x 16, operands from
//               shared memory through matrix descriptors, accumulator in tensor memory) four times per
//               stage, then tcgen05.commit, which frees the stage when the MMAs have read it; the warp
//               also allocates and frees the 512 columns of tensor memory (why the warps walk along: tcgen05.cuh);
//   warps 2-9   read the finished accumulator with tcgen05.ld (each warp its quarter of the 128
//               lanes and one half of the columns), apply the epilogue and store bfloat16; meanwhile warp 1 already fills
//               the other half of tensor memory with the next tile.
// Tiles go round-robin over the blocks: tile = blockIdx.x + i * gridDim.x, tokens fastest, so
// blocks that run together share the same weight columns in L2.
//
// Epilogues: bias, residual (may alias out), or `silu_pairs`: W's rows are stored as groups of
// [8 gate rows, 8 up rows] and the kernel writes silu(gate) * up, N/2 values per token
// (qil/model.py:71), so the [M, 2I] intermediate never exists in memory.
//
// Every wait on an mbarrier is bounded (and begins once the kernel before this one has ended: launched chained, a block may
// be there long before).  A wait that runs out records its place in the error
// word, the role stops issuing, every role runs out in turn, the producer drains its copies in
// flight (again bounded), the tensor memory is freed and the kernel returns; the host reads the
// error word.  No multicast loads are used.
#include "tcgen05.cuh"
#include <stdlib.h>

QIL_ERROR_STORAGE

#define TC_BM 128
#define TC_BN 256
#define TC_BK 64
#define TC_STAGES 4
#define TC_EPILOGUE_WARPS 8              // two a quarter of the lanes: half the time from the last MMA to the last store
#define TC_THREADS (64 + 32 * TC_EPILOGUE_WARPS)
#define TC_A_BYTES (TC_BM * TC_BK * 2)
#define TC_B_BYTES (TC_BN * TC_BK * 2)
#define TC_STAGE_BYTES (TC_A_BYTES + TC_B_BYTES)

// The query/key/value projection can end in what otherwise is a kernel of its own: per-head RMSNorm of
// queries and keys, the rotation of both by the token's position, queries to their buffer and keys and
// values into the token's page of the cache (qil/model.py:52-57, qil/cache.py:93-94).  Heads are 128 wide,
// so every 128-column half of an output tile is one whole head and one thread holds a token's head in
// registers.  The arithmetic and its rounding points are those of rope_kv.cu's bfloat16 kernel: the
// product rounded to bfloat16 first, sums of squares and the normalising factor in float32, the normed
// value rounded before the weight multiplies it, every product and sum of the rotation rounded by itself.
struct TcQkvTail {
    bf16* q_out;                 // [tokens, n_q_heads, 128]; null: the ordinary epilogue
    bf16* pages;                 // one layer's cache: [page][2][n_kv_heads][page_size][128]
    const float* rope;           // [rope_rows][128]: 64 cosines then 64 sines per position; null: no rotation
    const bf16* q_norm;          // [128] or null
    const bf16* k_norm;
    const int* positions;        // [tokens]
    const int* token_row;        // [tokens] block-table row
    const int* block_table;
    float eps;
    int table_stride, rope_rows, n_q_heads, n_kv_heads, page_size, num_pages;
};

__device__ __forceinline__ void tc_store_qkv_head(unsigned taddr, int m, int M, int head, const TcQkvTail& t,
                                                  const bf16* __restrict__ bias) {
    typedef __nv_bfloat162 bf2;
    // The head as 64 packed pairs (elements 2i, 2i + 1), rounded to bfloat16 as the product's output is.
    // Packed arithmetic from here on: one instruction per two values, and half the registers; the single
    // epilogue warp of a scheduler runs one dependent instruction after the other, so their number is
    // what the epilogue costs.
    bf2 pk[64];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        float part[32];
        __syncwarp();                              // the load is a warp-wide instruction: every lane takes part
        tmem_load_32(taddr + c * 32, part);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float x = part[2 * i], y = part[2 * i + 1];
            if (bias != nullptr) {
                const float2 b = __bfloat1622float2(*reinterpret_cast<const bf2*>(bias + head * 128 + c * 32 + 2 * i));
                x += b.x; y += b.y;
            }
            pk[c * 16 + i] = __floats2bfloat162_rn(x, y);
        }
    }
    if (m >= M) return;
    const bool is_q = head < t.n_q_heads;
    const bool is_k = !is_q && head < t.n_q_heads + t.n_kv_heads;
    const bf16* norm_w = is_q ? t.q_norm : (is_k ? t.k_norm : nullptr);
    if (norm_w != nullptr) {
        float sq = 0.f;
#pragma unroll
        for (int i = 0; i < 64; ++i) {
            const float2 f = __bfloat1622float2(pk[i]);
            sq = fmaf(f.x, f.x, sq);
            sq = fmaf(f.y, f.y, sq);
        }
        const float scale = rsqrtf(sq / 128.0f + t.eps);
        const bf2* w2 = reinterpret_cast<const bf2*>(norm_w);
#pragma unroll
        for (int i = 0; i < 64; ++i) {
            const float2 f = __bfloat1622float2(pk[i]);
            pk[i] = __hmul2_rn(__floats2bfloat162_rn(f.x * scale, f.y * scale), w2[i]);
        }
    }
    const int pos = t.positions[m];
    if ((is_q || is_k) && t.rope != nullptr) {
        const int row = (pos >= t.rope_rows && t.rope_rows > 0) ? t.rope_rows - 1 : pos;
        const float4* cs = reinterpret_cast<const float4*>(t.rope + (size_t)row * 128);
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
            // the table holds values already rounded to bfloat16: the conversion is exact
            const float4 cf = cs[i / 2], sf = cs[16 + i / 2];
            const bf2 c0 = __floats2bfloat162_rn(cf.x, cf.y), c1 = __floats2bfloat162_rn(cf.z, cf.w);
            const bf2 s0 = __floats2bfloat162_rn(sf.x, sf.y), s1 = __floats2bfloat162_rn(sf.z, sf.w);
            const bf2 lo0 = pk[i], lo1 = pk[i + 1], hi0 = pk[32 + i], hi1 = pk[32 + i + 1];
            // every product and sum rounds by itself (the _rn forms are never contracted into fused multiply-adds)
            pk[i] = __hsub2_rn(__hmul2_rn(lo0, c0), __hmul2_rn(hi0, s0));
            pk[i + 1] = __hsub2_rn(__hmul2_rn(lo1, c1), __hmul2_rn(hi1, s1));
            pk[32 + i] = __hadd2_rn(__hmul2_rn(lo0, s0), __hmul2_rn(hi0, c0));
            pk[32 + i + 1] = __hadd2_rn(__hmul2_rn(lo1, s1), __hmul2_rn(hi1, c1));
        }
    }
    bf16* dst;
    if (is_q) {
        dst = t.q_out + ((size_t)m * t.n_q_heads + head) * 128;
    } else {
        const int kv_head = is_k ? head - t.n_q_heads : head - t.n_q_heads - t.n_kv_heads;
        const int index = pos / t.page_size;                 // a position the table has no entry for writes nothing
        const int page = (pos >= 0 && index < t.table_stride) ? t.block_table[(size_t)t.token_row[m] * t.table_stride + index] : -1;
        if (page < 0 || page >= t.num_pages) return;        // never write outside the pool
        dst = t.pages + ((((size_t)page * 2 + (is_k ? 0 : 1)) * t.n_kv_heads + kv_head) * t.page_size + pos % t.page_size) * 128;
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        uint4 packed;
        packed.x = *reinterpret_cast<const unsigned*>(&pk[4 * q]);
        packed.y = *reinterpret_cast<const unsigned*>(&pk[4 * q + 1]);
        packed.z = *reinterpret_cast<const unsigned*>(&pk[4 * q + 2]);
        packed.w = *reinterpret_cast<const unsigned*>(&pk[4 * q + 3]);
        *reinterpret_cast<uint4*>(dst + q * 8) = packed;
    }
}

// One warp's quarter (32 rows) and half (128 columns) of a finished 128 x 256 accumulator: tcgen05.ld 32 columns at a time,
// epilogue, bfloat16 stores.  m is this lane's output row, n0 its first output column.
__device__ __forceinline__ void tc_store_accumulator(unsigned taddr, int m, int n0, int M, int N, int silu_pairs,
                                                     const bf16* __restrict__ bias, const bf16* residual, bf16* out) {
#pragma unroll 1
    for (int c = 0; c < TC_BN / 64; ++c) {
        float v[32];
        __syncwarp();                              // the load below is a warp-wide instruction
        tmem_load_32(taddr + c * 32, v);
        const int n = n0 + c * 32;
        if (m >= M || n >= N) {
            // nothing to store for this lane
        } else if (silu_pairs) {
            // columns come as [8 gate, 8 up] groups: 32 columns give 16 outputs
            const int out_width = N / 2;
            bf16* dst = out + (size_t)m * out_width + n / 2;
#pragma unroll
            for (int grp = 0; grp < 2; ++grp) {
                uint4 packed;
                bf16* o = reinterpret_cast<bf16*>(&packed);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float gate = round_to<bf16>(v[grp * 16 + i]);
                    const float up = round_to<bf16>(v[grp * 16 + 8 + i]);
                    const float act = round_to<bf16>(__fdividef(gate, 1.0f + __expf(-gate)));
                    o[i] = __float2bfloat16_rn(act * up);
                }
                if (n + grp * 16 < N) *reinterpret_cast<uint4*>(dst + grp * 8) = packed;
            }
        } else {
            bf16* dst = out + (size_t)m * N + n;
            const bf16* res = residual ? residual + (size_t)m * N + n : nullptr;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (n + q * 8 >= N) break;
                uint4 packed, rv = make_uint4(0u, 0u, 0u, 0u);
                if (res) rv = *reinterpret_cast<const uint4*>(res + q * 8);
                const bf16* r8 = reinterpret_cast<const bf16*>(&rv);
                bf16* o = reinterpret_cast<bf16*>(&packed);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float x = v[q * 8 + i];
                    if (bias) x += __bfloat162float(bias[n + q * 8 + i]);
                    if (res) x = __bfloat162float(r8[i]) + x;
                    o[i] = __float2bfloat16_rn(x);
                }
                *reinterpret_cast<uint4*>(dst + q * 8) = packed;
            }
        }
    }
}

struct TcShared {
    unsigned long long full[TC_STAGES];
    unsigned long long empty[TC_STAGES];
    unsigned long long acc_full[2];
    unsigned long long acc_empty[2];
    unsigned tmem_base;
    unsigned pad;
};

__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
               const bf16* __restrict__ bias, const bf16* residual, bf16* out,
               int M, int N, int K, int silu_pairs, int* error_word, const TcQkvTail tail) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    TcShared* sh = reinterpret_cast<TcShared*>(tiles + TC_STAGES * TC_STAGE_BYTES);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int tiles_m = (M + TC_BM - 1) / TC_BM, tiles_n = (N + TC_BN - 1) / TC_BN;
    const int n_tiles = tiles_m * tiles_n;
    const int k_blocks = (K + TC_BK - 1) / TC_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < TC_STAGES; ++s) { mbar_init(&sh->full[s], 1); mbar_init(&sh->empty[s], 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(&sh->acc_full[a], 1); mbar_init(&sh->acc_empty[a], TC_EPILOGUE_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     ::"r"(smem_u32(&sh->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = uniform(sh->tmem_base);

    if (warp == 0) {
        const bool leader = elect_one();
        if (leader) {
            asm volatile("prefetch.tensormap [%0];\n" ::"l"((unsigned long long)&map_a) : "memory");
            asm volatile("prefetch.tensormap [%0];\n" ::"l"((unsigned long long)&map_w) : "memory");
        }
        __syncwarp();
        const unsigned long long policy = stream_policy();
        qil_wait_for_producer();
        qil_release_consumer();      // the block holds its tensor memory
        int stage = 0;
        unsigned phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            const int m0 = (tile % tiles_m) * TC_BM, n0 = (tile / tiles_m) * TC_BN;
            for (int kb = 0; kb < k_blocks; ++kb) {
                if (!warp_mbar_wait(&sh->empty[stage], phase ^ 1)) { if (leader) atomicExch(error_word, 1); ok = false; break; }
                mbar_arrive_expect_tx(&sh->full[stage], TC_STAGE_BYTES, leader);
                unsigned char* a_dst = tiles + stage * TC_STAGE_BYTES;
                tma_load_2d(a_dst, &map_a, &sh->full[stage], kb * TC_BK, m0, leader);
                if (tiles_m == 1) tma_load_2d_stream(a_dst + TC_A_BYTES, &map_w, &sh->full[stage], kb * TC_BK, n0, policy, leader);
                else tma_load_2d(a_dst + TC_A_BYTES, &map_w, &sh->full[stage], kb * TC_BK, n0, leader);
                if (++stage == TC_STAGES) { stage = 0; phase ^= 1; }
            }
        }
        // copies still in flight land in this block's shared memory: wait for them (bounded)
        // before the block may leave, whether or not anyone consumes them
        for (int i = 0; i < TC_STAGES; ++i) {
            if (!warp_mbar_wait(&sh->empty[stage], phase ^ 1)) { if (leader) atomicExch(error_word, 2); break; }
            if (++stage == TC_STAGES) { stage = 0; phase ^= 1; }
        }
    } else if (warp == 1) {
        const bool leader = elect_one();
        const unsigned idesc = umma_idesc(TC_BM, TC_BN);
        qil_wait_for_producer();       // the bounded waits below count this kernel's own time
        int stage = 0, acc = 0;
        unsigned phase = 0, acc_phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            if (!warp_mbar_wait(&sh->acc_empty[acc], acc_phase ^ 1)) { if (leader) atomicExch(error_word, 3); ok = false; break; }
            tc_fence_after();
            const unsigned tmem_d = tmem_base + (unsigned)acc * TC_BN;
            for (int kb = 0; kb < k_blocks; ++kb) {
                if (!warp_mbar_wait(&sh->full[stage], phase)) { if (leader) atomicExch(error_word, 4); ok = false; break; }
                tc_fence_after();
                const unsigned a_addr = smem_u32(tiles + stage * TC_STAGE_BYTES);
                const unsigned b_addr = a_addr + TC_A_BYTES;
#pragma unroll
                for (int k = 0; k < TC_BK / 16; ++k) {
                    // 16 k-values are 32 bytes: advance the start address inside the swizzled row
                    umma_bf16(tmem_d, umma_desc(a_addr + k * 32), umma_desc(b_addr + k * 32), idesc,
                              (kb | k) ? 1u : 0u, leader);
                }
                umma_commit(&sh->empty[stage], leader);      // the stage is free once these MMAs have read it
                if (++stage == TC_STAGES) { stage = 0; phase ^= 1; }
            }
            if (!ok) break;
            umma_commit(&sh->acc_full[acc], leader);          // the accumulator is complete once all MMAs are done
            acc ^= 1;
            if (acc == 0) acc_phase ^= 1;
        }
    } else {
        const int quarter = warp & 3;                      // the TMEM lanes this warp may read
        const int half = warp < 6 ? 0 : 128;               // and the columns it takes
        qil_wait_for_producer();                           // outputs may still be read, the residual written, before this
        int acc = 0;
        unsigned acc_phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            const int m0 = (tile % tiles_m) * TC_BM, n0 = (tile / tiles_m) * TC_BN;
            if (!warp_mbar_wait(&sh->acc_full[acc], acc_phase)) { if (lane == 0) atomicExch(error_word, 5); ok = false; break; }
            tc_fence_after();
            const int m = m0 + quarter * 32 + lane;
            const unsigned taddr = tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)acc * TC_BN + half;
            if (tail.q_out != nullptr) {
                if (n0 + half < N) tc_store_qkv_head(taddr, m, M, (n0 + half) / 128, tail, bias);
            } else {
                tc_store_accumulator(taddr, m, n0 + half, M, N, silu_pairs, bias, residual, out);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->acc_empty[acc]);
            acc ^= 1;
            if (acc == 0) acc_phase ^= 1;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// ------------------------------------------------------------------ two SMs on one tile
// The same product with pairs of blocks (a cluster of two, on neighbouring SMs) working on one
// 256 x 256 output tile with tcgen05.mma.cta_group::2.  Each block of a pair loads its own 128 rows of A
// and its own half (128 output features) of the W tile; one thread of the pair's first block issues the
// MMAs, which read A and W from both blocks' shared memory and write each block's 128 x 256 half of the
// accumulator into that block's tensor memory.  Against the one-block kernel every MMA reads half as
// many bytes of shared memory per block (8 KB instead of 12 KB per 128 x 256 x 16 step), which is what
// keeps the tensor pipe fed, and a stage is 32 KB instead of 48 KB, so six stages fit instead of four.
//
// Barriers.  full[s] lives in the first block: its producer arms it with the bytes of both blocks and
// the second block's copies complete on it too (the barrier operand of a cta_group::2 copy may be the
// peer's).  empty[s] and acc_full[a] exist in both blocks and are signalled by one tcgen05.commit with a
// multicast mask of both.  acc_empty[a] lives in the first block and collects the arrivals of the sixteen
// epilogue warps of the pair, the second block's through shared::cluster addresses.  Every wait is
// local to the waiting block and bounded as in the kernel above; the pair meets at a cluster barrier
// before either block frees its tensor memory and leaves.  None of the loads is a multicast load.
#define T2_STAGES 6
#define T2_A_BYTES (128 * TC_BK * 2)
#define T2_B_BYTES (128 * TC_BK * 2)
#define T2_STAGE_BYTES (T2_A_BYTES + T2_B_BYTES)

struct Tc2Shared {
    unsigned long long full[T2_STAGES];
    unsigned long long empty[T2_STAGES];
    unsigned long long acc_full[2];
    unsigned long long acc_empty[2];
    unsigned tmem_base;
    unsigned pad;
};

__device__ __forceinline__ void mbar_arrive_cluster(unsigned cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(cluster_addr) : "memory");
}
// A tile copy of a block of a pair; `bar_cluster` may be a barrier of the pair's other block.
__device__ __forceinline__ void tma_load_2d_pair(void* smem, const CUtensorMap* map, unsigned bar_cluster, int x, int y, bool leader) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
                 "@p cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}\n"
                 ::"r"(smem_u32(smem)), "l"((unsigned long long)map), "r"(bar_cluster), "r"(x), "r"(y), "r"((unsigned)leader) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(unsigned tmem_d, unsigned long long desc_a, unsigned long long desc_b,
                                               unsigned idesc, unsigned accumulate, bool leader) {
    const unsigned zero = 0u;
    asm volatile("{\n\t.reg .pred p, q;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "setp.ne.b32 q, %6, 0;\n\t"
                 "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}\n"
                 ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(zero), "r"((unsigned)leader) : "memory");
}
// Arrives, once the pair's MMAs so far are done, on the barrier at this offset in both blocks.
__device__ __forceinline__ void umma_commit_pair(unsigned long long* bar, bool leader) {
    const unsigned short both = 3;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t"
                 "@p tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}\n"
                 ::"r"(smem_u32(bar)), "h"(both), "r"((unsigned)leader) : "memory");
}
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                    const bf16* __restrict__ bias, const bf16* residual, bf16* out,
                    int M, int N, int K, int silu_pairs, int* error_word, const TcQkvTail tail) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    Tc2Shared* sh = reinterpret_cast<Tc2Shared*>(tiles + T2_STAGES * T2_STAGE_BYTES);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int tiles_m = (M + 255) / 256, tiles_n = (N + TC_BN - 1) / TC_BN;
    const int n_tiles = tiles_m * tiles_n;
    const int k_blocks = (K + TC_BK - 1) / TC_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < T2_STAGES; ++s) { mbar_init(&sh->full[s], 1); mbar_init(&sh->empty[s], 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(&sh->acc_full[a], 1); mbar_init(&sh->acc_empty[a], 2 * TC_EPILOGUE_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {     // the same warp of both blocks, the same address: the pair's allocation
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     ::"r"(smem_u32(&sh->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // the other block's barriers are initialised before anything arrives on them
    tc_fence_after();
    const unsigned tmem_base = uniform(sh->tmem_base);

    if (warp == 0) {
        const bool leader = elect_one();
        if (leader) {
            asm volatile("prefetch.tensormap [%0];\n" ::"l"((unsigned long long)&map_a) : "memory");
            asm volatile("prefetch.tensormap [%0];\n" ::"l"((unsigned long long)&map_w) : "memory");
        }
        __syncwarp();
        const unsigned full_of_first = uniform(map_to_rank(smem_u32(sh->full), 0));
        qil_wait_for_producer();
        qil_release_consumer();      // the block holds its tensor memory
        int stage = 0;
        unsigned phase = 0;
        bool ok = true;
        for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
            const int m0 = (tile % tiles_m) * 256 + (int)rank * 128, n0 = (tile / tiles_m) * TC_BN + (int)rank * 128;
            for (int kb = 0; kb < k_blocks; ++kb) {
                if (!warp_mbar_wait(&sh->empty[stage], phase ^ 1)) { if (leader) atomicExch(error_word, 1); ok = false; break; }
                mbar_arrive_expect_tx(&sh->full[stage], 2 * T2_STAGE_BYTES, leader && rank == 0);
                unsigned char* a_dst = tiles + stage * T2_STAGE_BYTES;
                tma_load_2d_pair(a_dst, &map_a, full_of_first + stage * 8, kb * TC_BK, m0, leader);
                tma_load_2d_pair(a_dst + T2_A_BYTES, &map_w, full_of_first + stage * 8, kb * TC_BK, n0, leader);
                if (++stage == T2_STAGES) { stage = 0; phase ^= 1; }
            }
        }
        for (int i = 0; i < T2_STAGES; ++i) {      // this block's copies in flight land before it leaves
            if (!warp_mbar_wait(&sh->empty[stage], phase ^ 1)) { if (leader) atomicExch(error_word, 2); break; }
            if (++stage == T2_STAGES) { stage = 0; phase ^= 1; }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const bool leader = elect_one();
            const unsigned idesc = umma_idesc(256, TC_BN);
            qil_wait_for_producer();
            int stage = 0, acc = 0;
            unsigned phase = 0, acc_phase = 0;
            bool ok = true;
            for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
                if (!warp_mbar_wait(&sh->acc_empty[acc], acc_phase ^ 1)) { if (leader) atomicExch(error_word, 3); ok = false; break; }
                tc_fence_after();
                const unsigned tmem_d = tmem_base + (unsigned)acc * TC_BN;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!warp_mbar_wait(&sh->full[stage], phase)) { if (leader) atomicExch(error_word, 4); ok = false; break; }
                    tc_fence_after();
                    const unsigned a_addr = smem_u32(tiles + stage * T2_STAGE_BYTES);
                    const unsigned b_addr = a_addr + T2_A_BYTES;
#pragma unroll
                    for (int k = 0; k < TC_BK / 16; ++k)
                        umma_bf16_pair(tmem_d, umma_desc(a_addr + k * 32), umma_desc(b_addr + k * 32), idesc,
                                       (kb | k) ? 1u : 0u, leader);
                    umma_commit_pair(&sh->empty[stage], leader);
                    if (++stage == T2_STAGES) { stage = 0; phase ^= 1; }
                }
                if (!ok) break;
                umma_commit_pair(&sh->acc_full[acc], leader);
                acc ^= 1;
                if (acc == 0) acc_phase ^= 1;
            }
        }
    } else {
        const int quarter = warp & 3, half = warp < 6 ? 0 : 128;
        qil_wait_for_producer();
        int acc = 0;
        unsigned acc_phase = 0;
        bool ok = true;
        for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
            const int m0 = (tile % tiles_m) * 256 + (int)rank * 128, n0 = (tile / tiles_m) * TC_BN;
            if (!warp_mbar_wait(&sh->acc_full[acc], acc_phase)) { if (lane == 0) atomicExch(error_word, 5); ok = false; break; }
            tc_fence_after();
            const int m = m0 + quarter * 32 + lane;
            const unsigned taddr = tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)acc * TC_BN + half;
            if (tail.q_out != nullptr) {
                if (n0 + half < N) tc_store_qkv_head(taddr, m, M, (n0 + half) / 128, tail, bias);
            } else {
                tc_store_accumulator(taddr, m, n0 + half, M, N, silu_pairs, bias, residual, out);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(&sh->acc_empty[acc]), 0));
            acc ^= 1;
            if (acc == 0) acc_phase ^= 1;
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // neither block leaves while the other may still read its tiles or signal it
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// ------------------------------------------------------------------ two SMs on one tile, the tokens cut evenly
// The kernel above with the operands' places changed: features lie on the accumulator's lanes (W is the MMA's A operand) and
// tokens on its columns, because a tile may have any multiple of 16 columns.  The launch cuts the tokens into even tiles
// (521 are three of 176 where tiles of 256 compute 768), as `tokens_a_tile` says.
//
// Epilogue: a lane holds a feature, memory wants a token's features side by side.  Two groups of four warps take 32 columns
// in turn: the warps leave their lanes' float32 sums in the group's staging buffer, then take its rows (a token's 128
// features; of the q/k/v projection a whole head), four features a lane.  Tensor memory is free for the next tile once
// it is staged.  Barriers and bounded waits are those of the kernel above; a group's four warps meet at a barrier of their own,
// which has no limit, so behind each bounded wait they go on together or leave together.
#define TE_STAGES 6
#define TE_W_BYTES (128 * TC_BK * 2)
#define TE_STAGE_BYTES (2 * TE_W_BYTES)          // and up to 128 tokens
#define TE_CHUNK 32                              // tokens a group stages at a time
#define TE_ROW 132                               // floats a staged token: eight rows side by side are in eight different groups of banks
#define TE_STAGING_BYTES (TE_CHUNK * TE_ROW * 4)

struct TcEvenShared {
    unsigned long long full[TE_STAGES];
    unsigned long long empty[TE_STAGES];
    unsigned long long acc_full[2];
    unsigned long long acc_empty[2];
    unsigned tmem_base;
    unsigned pad;
};

// The factors that norm the heads of eight staged tokens, lane & 7 of them this lane's: the squares of the product's bfloat16
// values one after the other, as tc_store_qkv_head adds them, so that a token's bits do not depend on the kernel that its
// step's size picks.  Lanes of one token square a quarter of the features each; the sum goes through them in their order.
__device__ __forceinline__ float te_norm_scale(const float* row, const bf16* __restrict__ bias, float eps, int lane) {
    const int first = lane >> 3 << 5;
    float v[32];
#pragma unroll
    for (int c = 0; c < 32; c += 4) {
        float4 f = *reinterpret_cast<const float4*>(row + first + c);
        if (bias != nullptr) {
            const uint2 raw = *reinterpret_cast<const uint2*>(bias + first + c);
            const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
            f.x += x.x; f.y += x.y; f.z += y.x; f.w += y.y;
        }
        const float2 a = __bfloat1622float2(__floats2bfloat162_rn(f.x, f.y)), b = __bfloat1622float2(__floats2bfloat162_rn(f.z, f.w));
        v[c] = a.x; v[c + 1] = a.y; v[c + 2] = b.x; v[c + 3] = b.y;
    }
    float sq = 0.f;
#pragma unroll
    for (int turn = 0; turn < 4; ++turn) {
#pragma unroll
        for (int c = 0; c < 32; ++c) sq = fmaf(v[c], v[c], sq);
        sq = __shfl_sync(0xffffffffu, sq, turn * 8 + (lane & 7));          // those whose turn it was
    }
    return rsqrtf(sq / 128.0f + eps);
}

// One token's head of the q/k/v projection, four values a lane (`f`: the product, with its bias): the arithmetic and the
// rounding points of tc_store_qkv_head.  cf, sf: the lane's cosines and sines.
__device__ __forceinline__ uint2 te_qkv_values(const float4& f, const bf16* norm_w, float scale, bool rotate, const float4& cf, const float4& sf,
                                               int lane) {
    typedef __nv_bfloat162 bf2;
    bf2 lo = __floats2bfloat162_rn(f.x, f.y), hi = __floats2bfloat162_rn(f.z, f.w);
    if (norm_w != nullptr) {
        const float2 a = __bfloat1622float2(lo), b = __bfloat1622float2(hi);
        const uint2 w = *reinterpret_cast<const uint2*>(norm_w + lane * 4);
        lo = __hmul2_rn(__floats2bfloat162_rn(a.x * scale, a.y * scale), *reinterpret_cast<const bf2*>(&w.x));
        hi = __hmul2_rn(__floats2bfloat162_rn(b.x * scale, b.y * scale), *reinterpret_cast<const bf2*>(&w.y));
    }
    if (rotate) {
        // the table holds values already rounded to bfloat16: the conversion is exact
        const bf2 c0 = __floats2bfloat162_rn(cf.x, cf.y), c1 = __floats2bfloat162_rn(cf.z, cf.w);
        const bf2 s0 = __floats2bfloat162_rn(sf.x, sf.y), s1 = __floats2bfloat162_rn(sf.z, sf.w);
        // lanes 0..15 hold the first half of the head, lane + 16 the partners of a lane's values
        const unsigned other_lo = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<const unsigned*>(&lo), 16);
        const unsigned other_hi = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<const unsigned*>(&hi), 16);
        const bf2 p0 = *reinterpret_cast<const bf2*>(&other_lo), p1 = *reinterpret_cast<const bf2*>(&other_hi);
        // every product and sum rounds by itself (the _rn forms are never contracted into fused multiply-adds)
        if (lane < 16) {
            lo = __hsub2_rn(__hmul2_rn(lo, c0), __hmul2_rn(p0, s0));
            hi = __hsub2_rn(__hmul2_rn(hi, c1), __hmul2_rn(p1, s1));
        } else {
            lo = __hadd2_rn(__hmul2_rn(p0, s0), __hmul2_rn(lo, c0));
            hi = __hadd2_rn(__hmul2_rn(p1, s1), __hmul2_rn(hi, c1));
        }
    }
    uint2 packed;
    packed.x = *reinterpret_cast<const unsigned*>(&lo);
    packed.y = *reinterpret_cast<const unsigned*>(&hi);
    return packed;
}

// The four warps of an epilogue group meet.
__device__ __forceinline__ void te_group_sync(int group) { asm volatile("bar.sync %0, 128;\n" ::"r"(group + 1) : "memory"); }
// The same, and true if all of them come with `ok`: one whose wait ran out takes the other three along, who would otherwise
// meet without it for good.
__device__ __forceinline__ bool te_group_agrees(int group, bool ok) {
    unsigned all;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
                 "bar.red.and.pred p, %1, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(all) : "r"(group + 1), "r"((unsigned)ok) : "memory");
    return all != 0;
}

// The rows of a staged chunk that one of the group's four warps takes: tokens m0 + i of i = part, part + 4, ... < rows (of the q/k/v
// projection eight side by side), the 128 features from n0 on.
__device__ __forceinline__ void te_store_rows(const float* staged, int part, int rows, int m0, int n0, int N, int silu_pairs,
                                              const bf16* __restrict__ bias, const bf16* residual, bf16* out, const TcQkvTail& tail, int lane) {
    constexpr int R = TE_CHUNK / 4;
    if (n0 >= N) return;
    if (silu_pairs) {
        // columns come as [8 gate, 8 up] groups: half a warp a token, four outputs a lane
        const int col = ((lane & 15) >> 1) * 16 + (lane & 1) * 4;
#pragma unroll
        for (int r = 0; r < R; r += 2) {
            const int i = part + 4 * (r + (lane >> 4));
            const float4 g = *reinterpret_cast<const float4*>(staged + i * TE_ROW + col);
            const float4 u = *reinterpret_cast<const float4*>(staged + i * TE_ROW + col + 8);
            if (i >= rows || n0 + col >= N) continue;
            const float gate[4] = {g.x, g.y, g.z, g.w}, up[4] = {u.x, u.y, u.z, u.w};
            uint2 packed;
            bf16* o = reinterpret_cast<bf16*>(&packed);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float x = round_to<bf16>(gate[e]);
                const float act = round_to<bf16>(__fdividef(x, 1.0f + __expf(-x)));
                o[e] = __float2bfloat16_rn(act * round_to<bf16>(up[e]));
            }
            *reinterpret_cast<uint2*>(out + (size_t)(m0 + i) * (N / 2) + n0 / 2 + (lane & 15) * 4) = packed;
        }
        return;
    }
    const int n = n0 + lane * 4;
    const bool inside = n < N;
    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
    if (bias != nullptr && inside) {
        const uint2 raw = *reinterpret_cast<const uint2*>(bias + n);
        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        b = make_float4(x.x, x.y, y.x, y.y);
    }
    if (tail.q_out != nullptr) {
        // The 128 features are one whole head.  A row's place is asked for by a lane of its own, and all rows' rotations before the
        // sums of squares, whose chain is as long as those trips to L2.
        const int head = n0 / 128;
        const bool is_q = head < tail.n_q_heads, is_k = !is_q && head < tail.n_q_heads + tail.n_kv_heads;
        const bf16* norm_w = is_q ? tail.q_norm : (is_k ? tail.k_norm : nullptr);
        const bool rotate = (is_q || is_k) && tail.rope != nullptr;
        const int mine = part * R + (lane & (R - 1));
        int pos_of_lane = 0, page_of_lane = -1;
        if (mine < rows) {
            pos_of_lane = tail.positions[m0 + mine];
            const int index = pos_of_lane / tail.page_size;          // a position the table has no entry for writes nothing
            if (!is_q && pos_of_lane >= 0 && index < tail.table_stride)
                page_of_lane = tail.block_table[(size_t)tail.token_row[m0 + mine] * tail.table_stride + index];
        }
        float4 cf[R], sf[R];
        int pos[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            pos[r] = __shfl_sync(0xffffffffu, pos_of_lane, r);
            const int row = (pos[r] >= tail.rope_rows && tail.rope_rows > 0) ? tail.rope_rows - 1 : pos[r];
            cf[r] = sf[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (rotate && part * R + r < rows) {
                const float* cs = tail.rope + (size_t)row * 128 + (lane & 15) * 4;
                cf[r] = *reinterpret_cast<const float4*>(cs);
                sf[r] = *reinterpret_cast<const float4*>(cs + 64);
            }
        }
        const float scale_of_lane = norm_w != nullptr ? te_norm_scale(staged + mine * TE_ROW, bias ? bias + n0 : nullptr, tail.eps, lane) : 1.f;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = part * R + r, page = __shfl_sync(0xffffffffu, page_of_lane, r);
            const float scale = __shfl_sync(0xffffffffu, scale_of_lane, r);
            float4 f = *reinterpret_cast<const float4*>(staged + i * TE_ROW + lane * 4);
            f.x += b.x; f.y += b.y; f.z += b.z; f.w += b.w;
            const uint2 values = te_qkv_values(f, norm_w, scale, rotate, cf[r], sf[r], lane);
            if (i >= rows) continue;
            bf16* dst;
            if (is_q) {
                dst = tail.q_out + ((size_t)(m0 + i) * tail.n_q_heads + head) * 128;
            } else {
                if (page < 0 || page >= tail.num_pages) continue;        // never write outside the pool
                const int kv_head = is_k ? head - tail.n_q_heads : head - tail.n_q_heads - tail.n_kv_heads;
                dst = tail.pages + ((((size_t)page * 2 + (is_k ? 0 : 1)) * tail.n_kv_heads + kv_head) * tail.page_size + pos[r] % tail.page_size) * 128;
            }
            *reinterpret_cast<uint2*>(dst + lane * 4) = values;
        }
        return;
    }
    if (!inside) return;
    uint2 held[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        held[r] = make_uint2(0u, 0u);
        if (residual != nullptr && part + 4 * r < rows) held[r] = *reinterpret_cast<const uint2*>(residual + (size_t)(m0 + part + 4 * r) * N + n);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = part + 4 * r;
        if (i >= rows) break;
        float4 f = *reinterpret_cast<const float4*>(staged + i * TE_ROW + lane * 4);
        f.x += b.x; f.y += b.y; f.z += b.z; f.w += b.w;
        if (residual != nullptr) {
            const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&held[r].x)), y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&held[r].y));
            f.x = x.x + f.x; f.y = x.y + f.y; f.z = y.x + f.z; f.w = y.y + f.w;
        }
        const __nv_bfloat162 lo = __floats2bfloat162_rn(f.x, f.y), hi = __floats2bfloat162_rn(f.z, f.w);
        uint2 packed;
        packed.x = *reinterpret_cast<const unsigned*>(&lo);
        packed.y = *reinterpret_cast<const unsigned*>(&hi);
        *reinterpret_cast<uint2*>(out + (size_t)(m0 + i) * N + n) = packed;
    }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1)
gemm_tc_even_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                    const bf16* __restrict__ bias, const bf16* residual, bf16* out,
                    int M, int N, int K, int nt, int silu_pairs, int* error_word, const TcQkvTail tail) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* staging = tiles + TE_STAGES * TE_STAGE_BYTES;
    TcEvenShared* sh = reinterpret_cast<TcEvenShared*>(staging + 2 * TE_STAGING_BYTES);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int tiles_m = (M + nt - 1) / nt, tiles_n = (N + 255) / 256;
    const int n_tiles = tiles_m * tiles_n;
    const int k_blocks = (K + TC_BK - 1) / TC_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < TE_STAGES; ++s) { mbar_init(&sh->full[s], 1); mbar_init(&sh->empty[s], 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(&sh->acc_full[a], 1); mbar_init(&sh->acc_empty[a], 2 * TC_EPILOGUE_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {     // the same warp of both blocks, the same address: the pair's allocation
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     ::"r"(smem_u32(&sh->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // the other block's barriers are initialised before anything arrives on them
    tc_fence_after();
    const unsigned tmem_base = uniform(sh->tmem_base);

    if (warp == 0) {
        const bool leader = elect_one();
        if (leader) {
            asm volatile("prefetch.tensormap [%0];\n" ::"l"((unsigned long long)&map_x) : "memory");
            asm volatile("prefetch.tensormap [%0];\n" ::"l"((unsigned long long)&map_w) : "memory");
        }
        __syncwarp();
        const unsigned full_of_first = uniform(map_to_rank(smem_u32(sh->full), 0));
        const unsigned stage_bytes = 2 * (TE_W_BYTES + nt * TC_BK);            // both blocks' weights and tokens
        qil_wait_for_producer();     // the weights too: a caller's weight may be what the kernel before wrote
        qil_release_consumer();      // the block holds its tensor memory
        int stage = 0;
        unsigned phase = 0;
        bool ok = true;
        for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
            const int m0 = tile % tiles_m * nt + (int)rank * (nt / 2), n0 = tile / tiles_m * 256 + (int)rank * 128;
            for (int kb = 0; kb < k_blocks; ++kb) {
                if (!warp_mbar_wait(&sh->empty[stage], phase ^ 1)) { if (leader) atomicExch(error_word, 1); ok = false; break; }
                mbar_arrive_expect_tx(&sh->full[stage], stage_bytes, leader && rank == 0);
                unsigned char* to = tiles + stage * TE_STAGE_BYTES;
                tma_load_2d_pair(to, &map_w, full_of_first + stage * 8, kb * TC_BK, n0, leader);
                tma_load_2d_pair(to + TE_W_BYTES, &map_x, full_of_first + stage * 8, kb * TC_BK, m0, leader);
                if (++stage == TE_STAGES) { stage = 0; phase ^= 1; }
            }
        }
        for (int i = 0; i < TE_STAGES; ++i) {      // this block's copies in flight land before it leaves
            if (!warp_mbar_wait(&sh->empty[stage], phase ^ 1)) { if (leader) atomicExch(error_word, 2); break; }
            if (++stage == TE_STAGES) { stage = 0; phase ^= 1; }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const bool leader = elect_one();
            const unsigned idesc = umma_idesc(256, nt);
            qil_wait_for_producer();
            int stage = 0, acc = 0;
            unsigned phase = 0, acc_phase = 0;
            bool ok = true;
            for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
                if (!warp_mbar_wait(&sh->acc_empty[acc], acc_phase ^ 1)) { if (leader) atomicExch(error_word, 3); ok = false; break; }
                tc_fence_after();
                const unsigned tmem_d = tmem_base + (unsigned)acc * 256;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!warp_mbar_wait(&sh->full[stage], phase)) { if (leader) atomicExch(error_word, 4); ok = false; break; }
                    tc_fence_after();
                    const unsigned w_addr = smem_u32(tiles + stage * TE_STAGE_BYTES), x_addr = w_addr + TE_W_BYTES;
#pragma unroll
                    for (int k = 0; k < TC_BK / 16; ++k)
                        umma_bf16_pair(tmem_d, umma_desc(w_addr + k * 32), umma_desc(x_addr + k * 32), idesc, (kb | k) ? 1u : 0u, leader);
                    umma_commit_pair(&sh->empty[stage], leader);
                    if (++stage == TE_STAGES) { stage = 0; phase ^= 1; }
                }
                if (!ok) break;
                umma_commit_pair(&sh->acc_full[acc], leader);
                acc ^= 1;
                if (acc == 0) acc_phase ^= 1;
            }
        }
    } else {
        const int quarter = warp & 3, group = warp < 6 ? 0 : 1;
        float* staged = reinterpret_cast<float*>(staging + group * TE_STAGING_BYTES);
        qil_wait_for_producer();
        int acc = 0;
        unsigned acc_phase = 0;
        for (int tile = pair; tile < n_tiles; tile += n_pairs) {
            const int m0 = (tile % tiles_m) * nt, n0 = (tile / tiles_m) * 256 + (int)rank * 128;
            const bool ok = warp_mbar_wait(&sh->acc_full[acc], acc_phase);
            if (!ok && lane == 0) atomicExch(error_word, 5);
            if (!te_group_agrees(group, ok)) break;      // nothing of this tile is stored
            tc_fence_after();
            const unsigned taddr = tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)acc * 256;
            for (int c0 = group * TE_CHUNK; c0 < nt; c0 += 2 * TE_CHUNK) {
                float v[32];
                tmem_load_32(taddr + c0, v);
                if (c0 + 2 * TE_CHUNK >= nt) {          // this warp's last columns: the accumulator's next tile may begin
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(&sh->acc_empty[acc]), 0));
                }
                if (c0 >= 2 * TE_CHUNK) te_group_sync(group);      // the rows of the chunk before have been read
#pragma unroll
                for (int i = 0; i < 32; ++i) staged[i * TE_ROW + quarter * 32 + lane] = v[i];
                te_group_sync(group);
                const int rows = min(min(TE_CHUNK, nt - c0), M - m0 - c0);
                te_store_rows(staged, quarter, rows, m0 + c0, n0, N, silu_pairs, bias, residual, out, tail, lane);
                __syncwarp();
            }
            if (group * TE_CHUNK >= nt) {                // a tile of one chunk: nothing for the second group
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(&sh->acc_empty[acc]), 0));
            }
            acc ^= 1;
            if (acc == 0) acc_phase ^= 1;
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // neither block leaves while the other may still read its tiles or signal it
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// ------------------------------------------------------------------ a few dozen rows
// The product for the rows between a decode step's and a prompt portion's (17 to 128): its time is that of reading W
// once, as for the decode product, but there are too many rows for mma.sync to keep up.  128 output features sit on the
// 128 lanes of the accumulator and the rows on its columns (W is the MMA's A operand), so a block's MMAs cost what the
// rows need and a stage is nearly all weights.  One tile a block and nothing persistent: what counts is that every SM
// streams from the first to the last microsecond.  So
//   - a cluster of up to eight blocks cuts a tile's K; every block leaves its float32 sums in its shared memory and adds
//     up, in block order, its share of the rows out of all of them (the same bits on every launch);
//   - two blocks fit an SM, and a launch chained to the kernel before it has its barriers and tensor memory set up and its
//     ring full of weights when that kernel ends.  (Dependents are released only when the block holds its tensor
//     memory: blocks of a later launch never hold what blocks of an earlier one wait for.)
// Waits are bounded as above.  Measured beside the rule that cuts K, in qil_gemm_tc_rows.
#define TR_BM 128
#define TR_W_BYTES (TR_BM * TC_BK * 2)
#define TR_MOST_STAGES 6
#define TR_MOST_BLOCKS 8

struct TrShared {
    unsigned long long full[TR_MOST_STAGES];
    unsigned long long empty[TR_MOST_STAGES];
    unsigned long long acc_full;
    unsigned tmem_base;
    unsigned pad;
};

// ROWS columns of accumulator: M <= ROWS
template <int ROWS>
struct TrShape {
    static constexpr int X_BYTES = ROWS * TC_BK * 2;
    static constexpr int STAGE_BYTES = TR_W_BYTES + X_BYTES;
    static constexpr int STAGES = ROWS <= 32 ? 5 : ROWS <= 64 ? 4 : 3;         // two blocks an SM
    static constexpr int SMEM = STAGES * STAGE_BYTES + (int)sizeof(TrShared) + 1024;
};

__device__ __forceinline__ float4 cluster_read4(const float* at, unsigned rank) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(map_to_rank(smem_u32(at), rank)) : "memory");
    return v;
}

template <int ROWS, bool PAIRS>
__global__ void __launch_bounds__(192, 2)
gemm_tc_rows_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                    const bf16* __restrict__ bias, const bf16* residual, bf16* out,
                    int M, int N, int K, int* error_word) {
    typedef TrShape<ROWS> Shape;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    TrShared* sh = reinterpret_cast<TrShared*>(ring + Shape::STAGES * Shape::STAGE_BYTES);
    float* sums = reinterpret_cast<float*>(ring);          // [ROWS][128] once the ring is read out
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank(), blocks = cluster_blocks();
    const int n0 = blockIdx.x / blocks * TR_BM;
    const int k_blocks = (K + TC_BK - 1) / TC_BK;
    const int kb0 = (int)((long long)k_blocks * rank / blocks), kb1 = (int)((long long)k_blocks * (rank + 1) / blocks);

    if (threadIdx.x == 0) {
        for (int s = 0; s < Shape::STAGES; ++s) { mbar_init(&sh->full[s], 1); mbar_init(&sh->empty[s], 1); }
        mbar_init(&sh->acc_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     ::"r"(smem_u32(&sh->tmem_base)), "r"((unsigned)ROWS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = uniform(sh->tmem_base);

    if (warp == 0) {
        const bool leader = elect_one();
        const unsigned long long policy = stream_policy();
        // the ring's first round: weights, which no kernel writes, before the kernel before this one has ended
        const int first = kb1 - kb0 < Shape::STAGES ? kb1 - kb0 : Shape::STAGES;
        for (int s = 0; s < first; ++s) {
            mbar_arrive_expect_tx(&sh->full[s], Shape::STAGE_BYTES, leader);
            tma_load_2d_stream(ring + s * Shape::STAGE_BYTES, &map_w, &sh->full[s], (kb0 + s) * TC_BK, n0, policy, leader);
        }
        qil_wait_for_producer();
        qil_release_consumer();
        for (int s = 0; s < first; ++s)
            tma_load_2d(ring + s * Shape::STAGE_BYTES + TR_W_BYTES, &map_x, &sh->full[s], (kb0 + s) * TC_BK, 0, leader);
        int stage = first == Shape::STAGES ? 0 : first;
        unsigned phase = first == Shape::STAGES ? 1 : 0;
        for (int kb = kb0 + first; kb < kb1; ++kb) {
            if (!warp_mbar_wait(&sh->empty[stage], phase ^ 1)) { if (leader) atomicExch(error_word, 1); break; }
            mbar_arrive_expect_tx(&sh->full[stage], Shape::STAGE_BYTES, leader);
            unsigned char* to = ring + stage * Shape::STAGE_BYTES;
            tma_load_2d_stream(to, &map_w, &sh->full[stage], kb * TC_BK, n0, policy, leader);
            tma_load_2d(to + TR_W_BYTES, &map_x, &sh->full[stage], kb * TC_BK, 0, leader);
            if (++stage == Shape::STAGES) { stage = 0; phase ^= 1; }
        }
        for (int i = 0; i < first; ++i) {      // copies in flight land before the block may leave
            const int back = (stage + Shape::STAGES - first + i) % Shape::STAGES;
            const unsigned round = (unsigned)((kb1 - kb0 - first + i) / Shape::STAGES) & 1;
            if (!warp_mbar_wait(&sh->empty[back], round)) { if (leader) atomicExch(error_word, 2); break; }
        }
    } else if (warp == 1) {
        const bool leader = elect_one();
        const unsigned idesc = umma_idesc(TR_BM, ROWS);
        qil_wait_for_producer();       // the rows come after it; the bounded waits count this kernel's own time
        int stage = 0;
        unsigned phase = 0;
        bool ok = true;
        for (int kb = kb0; kb < kb1; ++kb) {
            if (!warp_mbar_wait(&sh->full[stage], phase)) { if (leader) atomicExch(error_word, 4); ok = false; break; }
            tc_fence_after();
            const unsigned w_addr = smem_u32(ring + stage * Shape::STAGE_BYTES), x_addr = w_addr + TR_W_BYTES;
#pragma unroll
            for (int k = 0; k < TC_BK / 16; ++k)
                umma_bf16(tmem_base, umma_desc(w_addr + k * 32), umma_desc(x_addr + k * 32), idesc, (kb > kb0 || k) ? 1u : 0u, leader);
            umma_commit(&sh->empty[stage], leader);
            if (++stage == Shape::STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit(&sh->acc_full, leader);
    } else {
        const int quarter = warp & 3;
        qil_wait_for_producer();
        if (warp_mbar_wait(&sh->acc_full, 0)) {          // every stage has been read: the ring is free
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < ROWS / 32; ++c) {
                float v[32];
                __syncwarp();
                tmem_load_32(tmem_base + ((unsigned)(quarter * 32) << 16) + c * 32, v);
#pragma unroll
                for (int i = 0; i < 32; ++i) sums[(c * 32 + i) * TR_BM + quarter * 32 + lane] = v[i];
            }
            tc_fence_before();
        } else if (lane == 0) {
            atomicExch(error_word, 5);
        }
    }
    __syncwarp();
    qil_wait_for_producer();       // outputs are written below: what still reads them has ended
    cluster_sync_all();
    // 4 outputs of a row a thread, out of 4 sums, or of 4 of a gate and 4 of the matching up features (columns come as
    // [8 gate, 8 up] groups); the cluster's blocks take rows in turn.  Everything an item needs is asked for before any of it
    // is used, for U items at a time: what this costs is trips to other blocks' shared memory and to L2.
    constexpr int GROUPS = PAIRS ? TR_BM / 8 : TR_BM / 4, PARTS = PAIRS ? 2 : 1, U = 4 / PARTS;
    const int items = (M - (int)rank + (int)blocks - 1) / (int)blocks * GROUPS;
    for (int item0 = threadIdx.x; item0 < items; item0 += 192 * U) {
        float v[U][4 * PARTS];
        uint2 rv[U];
        int row[U], col[U];                    // the row, and the tile's column of the first sum
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int item = min(item0 + u * 192, items - 1), group = item % GROUPS;
            row[u] = item / GROUPS * (int)blocks + (int)rank;
            col[u] = PAIRS ? (group >> 1) * 16 + (group & 1) * 4 : group * 4;
            rv[u] = make_uint2(0u, 0u);
            if (!PAIRS && residual != nullptr && n0 + col[u] < N)
                rv[u] = *reinterpret_cast<const uint2*>(residual + (size_t)row[u] * N + n0 + col[u]);
#pragma unroll
            for (int i = 0; i < 4 * PARTS; ++i) v[u][i] = 0.f;
        }
        for (unsigned b0 = 0; b0 < blocks; b0 += 4) {
            float4 part[U][4][PARTS];
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int q = 0; q < PARTS; ++q)
                        if (b0 + b < blocks) part[u][b][q] = cluster_read4(sums + row[u] * TR_BM + col[u] + q * 8, b0 + b);
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int q = 0; q < PARTS; ++q)
                        if (b0 + b < blocks) {
                            v[u][4 * q] += part[u][b][q].x; v[u][4 * q + 1] += part[u][b][q].y;
                            v[u][4 * q + 2] += part[u][b][q].z; v[u][4 * q + 3] += part[u][b][q].w;
                        }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int n = n0 + col[u];
            if (item0 + u * 192 >= items || n >= N) continue;
            uint2 packed;
            bf16* o = reinterpret_cast<bf16*>(&packed);
            if (PAIRS) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float gate = round_to<bf16>(v[u][i]), up = round_to<bf16>(v[u][4 * (PARTS - 1) + i]);
                    const float act = round_to<bf16>(__fdividef(gate, 1.0f + __expf(-gate)));
                    o[i] = __float2bfloat16_rn(act * up);
                }
                *reinterpret_cast<uint2*>(out + (size_t)row[u] * (N / 2) + n0 / 2 + (col[u] >> 4) * 8 + (col[u] & 4)) = packed;
            } else {
                const bf16* r4 = reinterpret_cast<const bf16*>(&rv[u]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float x = v[u][i];
                    if (bias) x += __bfloat162float(bias[n + i]);
                    if (residual) x = __bfloat162float(r4[i]) + x;
                    o[i] = __float2bfloat16_rn(x);
                }
                *reinterpret_cast<uint2*>(out + (size_t)row[u] * N + n) = packed;
            }
        }
    }
    __syncwarp();
    cluster_sync_all();            // no block leaves while another reads its sums
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"((unsigned)ROWS) : "memory");
    }
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult status;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &status) == cudaSuccess &&
            status == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)ptr;
    }
    return fn;
}

// A row-major bfloat16 matrix [rows, cols] seen through boxes of [box_rows, 64] with 128-byte swizzle.
static int make_map(CUtensorMap* map, const void* base, int rows, int cols, int box_rows) {
    EncodeTiledFn encode = encode_tiled();
    if (encode == nullptr) QIL_REFUSE("gemm_tc: the driver does not offer cuTensorMapEncodeTiled");
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    const cuuint32_t box[2] = {TC_BK, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) QIL_REFUSE("gemm_tc: cuTensorMapEncodeTiled failed with %d for a [%d, %d] matrix", (int)r, rows, cols);
    return 0;
}

extern "C" int qil_gemm_tc_min_rows() { return 17; }

// How many pairs of blocks of a kernel run at a time on the current device, asked once (`known`, by device: the limit of shared memory
// that it raises belongs to the function on a device); 0: refused.
#define TC_MOST_DEVICES 64
template <typename Kernel>
static int pairs_at_a_time(Kernel kernel, int smem, int sm_count, int* known) {
    int device = -1;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess || device < 0 || device >= TC_MOST_DEVICES) {
        snprintf(qil_error_text, sizeof(qil_error_text), "gemm_tc: device %d is out of range", device);
        return 0;
    }
    if (known[device] > 0) return known[device];
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) {
        snprintf(qil_error_text, sizeof(qil_error_text), "gemm_tc: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
        return 0;
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(sm_count & ~1);
    config.blockDim = dim3(TC_THREADS);
    config.dynamicSmemBytes = smem;
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &config);
    if (e != cudaSuccess || clusters <= 0) { (void)cudaGetLastError(); clusters = sm_count / 2; }
    return known[device] = clusters < sm_count / 2 ? clusters : sm_count / 2;
}

// What a 16-wide step of K costs a tile of the even kernel, in cycles: nt / 2 of MMA, or those that bring its 128 features and
// nt / 2 tokens to each block.  A tile of the other two costs 128.
static int even_step(int nt) { return nt / 2 > 64 + nt / 4 ? nt / 2 : 64 + nt / 4; }

// How many tokens a tile of the even kernel takes: as many as make the fewest and cheapest waves of `pairs` tiles.  `cost`: of
// those waves, a step of K.
static int tokens_a_tile(int M, int tiles_n, int pairs, long long* cost) {
    int best = 256;
    *cost = -1;
    for (int count = (M + 255) / 256; count <= (M + 15) / 16; ++count) {
        const int nt = ((M + count - 1) / count + 15) / 16 * 16;
        const long long tiles = (long long)((M + nt - 1) / nt) * tiles_n, waves = (tiles + pairs - 1) / pairs;
        if (*cost < 0 || waves * even_step(nt) < *cost) { best = nt; *cost = waves * even_step(nt); }
        if (tiles > 8ll * pairs) break;
    }
    return best;
}

// Does the even kernel take the product?  Where even tiles make its waves a tenth cheaper than those of 256 (from 256
// tokens on, pairs of blocks) or 128 tokens (one block), and K is long enough to hide an epilogue that goes through shared
// memory and grows with a tile's tokens.  A single wave of tiles has it once, that of q/k/v (`tail`) is the longer one.  The lines
// lie where every product measured on the even side is at least as fast.
// Measured, us (the other kernels / this one at the tokens a tile in brackets, weights from memory):
//   gate/up of 24576 x 4096: 129 tokens 64 / 48, 300 73 / 58, 521 102 / 79, 2048 256 / 256 (waves no cheaper: not taken)
//   gate/up in two waves:    12288 x 2048 at 300 tokens 25.6 / 19.5, 521 28.2 / 23.8; K below 2048 not taken (9216 x 1536 at 521 20.9 / 17.7,
//                            but 9216 x 1024 at 700 17.1 / 18.1)
//   gate/up in one wave:     6144 x 1024 at 129 11.1 / 8.3, 300 12.0 / 9.9, 521 [176] 12.4 / 12.1, 560 [192] 12.4 / 12.5 (not taken);
//                            4608 x 768 at 480 [128] 10.2 / 9.3, 700 [176] 10.8 / 11.2 (not taken); 4608 x 256 at 300 [80] 7.2 / 6.4, 480 [128]
//                            7.3 / 7.4 (not taken); 6144 x 96 at 128 [48] 6.1 / 5.5, 255 [96] 6.2 / 6.5 (not taken)
//   q/k/v in one wave:       6144 x 4096 at 521 33.2 / 31.3; 4096 x 2048 at 512 [128] 21.9 / 18.1, 600 [160] 22.3 / 22.0, 700 [176]
//                            22.8 / 23.0 (not taken); 6144 x 2560 at 512 [176] 25.7 / 25.1, 560 [192] 25.4 / 25.9 (not taken)
//   q/k/v in more:           6144 x 4096 at 776 [144] 50 / 41, 1021 [176] 51 / 46; 5120 x 3072 at 850 [128] 35.7 / 31.2, 1021 [160] 36.1 / 36.7
//                            (not taken); 4096 x 3584 at 1350 [160] 40.2 / 39.1, 1500 [176] 40.5 / 41.7 (not taken); 4096 x 2048 at 1200 [144]
//                            28.1 / 31.9 (not taken)
static int even_tokens(int M, int N, int K, bool tail, int pairs, int sm_count) {
    const int tiles_n = (N + 255) / 256;
    long long cost;
    const int nt = tokens_a_tile(M, tiles_n, pairs, &cost);
    const long long tiles = (long long)((M + nt - 1) / nt) * tiles_n;
    const long long others = M >= 256 ? (long long)((M + 255) / 256) * tiles_n : (long long)((M + TC_BM - 1) / TC_BM) * tiles_n;
    const int at_a_time = M >= 256 ? pairs : sm_count;
    const long long other_cost = (others + at_a_time - 1) / at_a_time * 128;
    const bool one_wave = tiles <= pairs;
    const bool hidden = !tail ? K >= 2048 || (one_wave && nt <= 48 + K / 8)
                              : one_wave ? K >= 2048 && nt <= 96 + K / 32 : nt <= K / 16 - 64;
    return hidden && 10 * cost <= 9 * other_cost ? nt : 0;
}

// The rule by itself: the tokens a tile, 0 for another kernel.
extern "C" int qil_gemm_tc_even_tokens(int M, int N, int K, int tail, int pairs, int sm_count) {
    return even_tokens(M, N, K, tail != 0, pairs, sm_count);
}

// nt: tokens a tile of the even kernel (0: as even_tokens says, which may be another kernel).
static int launch_gemm_tc(const void* a, const void* w, const void* bias, const void* residual, void* out,
                          int M, int N, int K, int silu_pairs, int nt, int sm_count, int* error_word, const TcQkvTail& tail,
                          cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 8) QIL_REFUSE("gemm_tc: K %d must be a positive multiple of 8 (16-byte rows for TMA)", K);
    if (N % 8) QIL_REFUSE("gemm_tc: N %d must be a multiple of 8", N);
    if (((uintptr_t)a | (uintptr_t)w | (uintptr_t)out | (uintptr_t)residual) & 15)
        QIL_REFUSE("gemm_tc: operands must be 16-byte aligned");
    if (silu_pairs && (N % 16 || bias != nullptr || residual != nullptr))
        QIL_REFUSE("gemm_tc: silu_pairs needs N %% 16 == 0 and neither bias nor residual");
    if (error_word == nullptr || sm_count <= 0) QIL_REFUSE("gemm_tc: needs an error word and the SM count");
    CUtensorMap map_a, map_w;
    static int pair_env = -1;
    if (pair_env < 0) {
        const char* e = getenv("QIL_GEMM_TC_PAIRS");
        pair_env = (e != nullptr && e[0] == '0') ? 0 : 1;
    }
    if (nt != 0 && (nt < 16 || nt > 256 || nt % 16)) QIL_REFUSE("gemm_tc: tiles of %d tokens; a multiple of 16 up to 256", nt);
    const bool even_fits = ((uintptr_t)bias & 7) == 0;                     // its epilogue reads four values of the bias at once
    if (nt > 0 && !even_fits) QIL_REFUSE("gemm_tc: tiles of a number of tokens want an 8-byte aligned bias");
    static int even_known[TC_MOST_DEVICES];
    const int smem_even = TE_STAGES * TE_STAGE_BYTES + 2 * TE_STAGING_BYTES + (int)sizeof(TcEvenShared) + 1024;
    int even_pairs = 0;
    if (nt > 0 || (pair_env == 1 && even_fits)) {
        even_pairs = pairs_at_a_time(gemm_tc_even_kernel, smem_even, sm_count, even_known);
        if (even_pairs == 0) return -1;
        if (nt == 0) nt = even_tokens(M, N, K, tail.q_out != nullptr, even_pairs, sm_count);
    }
    if (nt > 0) {
        if (make_map(&map_a, a, M, K, nt / 2)) return -1;
        if (make_map(&map_w, w, N, K, 128)) return -1;
        const long long tiles = (long long)((M + nt - 1) / nt) * ((N + 255) / 256);
        if (tiles > 0x7fffffffll) QIL_REFUSE("gemm_tc: [%d, %d] x [%d, %d] is too large for one launch", M, K, N, K);
        qil_launch_chained(gemm_tc_even_kernel, dim3(2 * (tiles < even_pairs ? (int)tiles : even_pairs)), dim3(TC_THREADS), smem_even,
                           stream, map_a, map_w, (const bf16*)bias, (const bf16*)residual, (bf16*)out, M, N, K, nt, silu_pairs, error_word, tail);
        QIL_CHECK_LAUNCH();
    }
    if (make_map(&map_a, a, M, K, TC_BM)) return -1;
    if (make_map(&map_w, w, N, K, TC_BN)) return -1;
    const int smem = TC_STAGES * TC_STAGE_BYTES + (int)sizeof(TcShared) + 1024;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) QIL_REFUSE("gemm_tc: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
        configured = true;
    }
    if (M >= 256 && pair_env == 1) {
        // two SMs per 256 x 256 tile; the W map's box is the 128 output features one block loads
        if (make_map(&map_w, w, N, K, 128)) return -1;
        const int smem_pair = T2_STAGES * T2_STAGE_BYTES + (int)sizeof(Tc2Shared) + 1024;
        static int pair_known[TC_MOST_DEVICES];
        const int pairs_resident = pairs_at_a_time(gemm_tc_pair_kernel, smem_pair, sm_count, pair_known);
        if (pairs_resident == 0) return -1;
        const int pair_tiles = ((M + 255) / 256) * ((N + TC_BN - 1) / TC_BN);
        const int pairs = pair_tiles < pairs_resident ? pair_tiles : pairs_resident;
        qil_launch_chained(gemm_tc_pair_kernel, dim3(2 * pairs), dim3(TC_THREADS), smem_pair, stream, map_a, map_w, (const bf16*)bias,
                           (const bf16*)residual, (bf16*)out, M, N, K, silu_pairs, error_word, tail);
        QIL_CHECK_LAUNCH();
    }
    const int n_tiles = ((M + TC_BM - 1) / TC_BM) * ((N + TC_BN - 1) / TC_BN);
    const int blocks = n_tiles < sm_count ? n_tiles : sm_count;
    qil_launch_chained(gemm_tc_kernel, dim3(blocks), dim3(TC_THREADS), smem, stream, map_a, map_w, (const bf16*)bias,
                       (const bf16*)residual, (bf16*)out, M, N, K, silu_pairs, error_word, tail);
    QIL_CHECK_LAUNCH();
}

// error_word: a device int the caller zeroes once and reads after synchronising; non-zero means a
// bounded wait inside the kernel ran out (1-2 producer, 3-4 MMA issuer, 5 epilogue).
extern "C" int qil_gemm_tc(const void* a, const void* w, const void* bias, const void* residual, void* out,
                           int M, int N, int K, int silu_pairs, int nt, int sm_count, int* error_word, cudaStream_t stream) {
    TcQkvTail none = {};
    return launch_gemm_tc(a, w, bias, residual, out, M, N, K, silu_pairs, nt, sm_count, error_word, none, stream);
}

// The stacked query/key/value projection of heads of 128 with its tail fused (see TcQkvTail): w is
// [(n_q_heads + 2 n_kv_heads) * 128, K] (queries, then keys, then values; n_kv_heads may be 0 for a layer
// that reads another layer's cache), q_out [M, n_q_heads * 128], pages one layer of the cache.  rope
// float32 [rope_rows, 128] (cosines then sines, values representable in bfloat16) or null; q_norm, k_norm
// bfloat16 [128] or null; positions, token_row int32 [M]; block_table int32 rows of table_stride.
extern "C" int qil_gemm_tc_qkv(const void* a, const void* w, const void* bias, void* q_out, void* pages,
                               const float* rope, int rope_rows, const void* q_norm, const void* k_norm, float eps,
                               const int* positions, const int* token_row, const int* block_table, int table_stride,
                               int n_q_heads, int n_kv_heads, int page_size, int num_pages,
                               int M, int K, int nt, int sm_count, int* error_word, cudaStream_t stream) {
    if (n_q_heads <= 0 || n_kv_heads < 0) QIL_REFUSE("gemm_tc_qkv: %d query heads, %d kv heads", n_q_heads, n_kv_heads);
    if (q_out == nullptr || positions == nullptr) QIL_REFUSE("gemm_tc_qkv: needs the query buffer and the positions");
    if (n_kv_heads > 0 && (pages == nullptr || token_row == nullptr || block_table == nullptr || page_size <= 0 || num_pages <= 0))
        QIL_REFUSE("gemm_tc_qkv: keys and values need the cache, the block table and the tokens' rows");
    if (((uintptr_t)q_out | (uintptr_t)pages | (uintptr_t)rope | (uintptr_t)q_norm | (uintptr_t)k_norm) & 15)
        QIL_REFUSE("gemm_tc_qkv: buffers must be 16-byte aligned");
    TcQkvTail tail = {};
    tail.q_out = (bf16*)q_out; tail.pages = (bf16*)pages; tail.rope = rope; tail.rope_rows = rope_rows;
    tail.q_norm = (const bf16*)q_norm; tail.k_norm = (const bf16*)k_norm; tail.eps = eps;
    tail.positions = positions; tail.token_row = token_row; tail.block_table = block_table;
    tail.table_stride = table_stride; tail.n_q_heads = n_q_heads; tail.n_kv_heads = n_kv_heads;
    tail.page_size = page_size > 0 ? page_size : 1; tail.num_pages = num_pages;
    const int N = (n_q_heads + 2 * n_kv_heads) * 128;
    return launch_gemm_tc(a, w, bias, nullptr, q_out, M, N, K, 0, nt, sm_count, error_word, tail, stream);
}

// ------------------------------------------------------------------ a few dozen rows: launch
template <int ROWS, bool PAIRS>
static int launch_rows(const CUtensorMap& map_x, const CUtensorMap& map_w, const bf16* bias, const bf16* residual, bf16* out,
                       int M, int N, int K, int blocks, int* error_word, cudaStream_t stream) {
    const int smem = TrShape<ROWS>::SMEM;
    static bool configured[64];                            // by device: the limit belongs to the function on a device
    int device = -1;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess || device < 0 || device >= 64) QIL_REFUSE("gemm_tc_rows: device %d is out of range", device);
    if (!configured[device]) {
        e = cudaFuncSetAttribute(gemm_tc_rows_kernel<ROWS, PAIRS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) QIL_REFUSE("gemm_tc_rows: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
        configured[device] = true;
    }
    e = qil_launch_clusters(gemm_tc_rows_kernel<ROWS, PAIRS>, dim3((N + TR_BM - 1) / TR_BM * blocks), dim3(192), smem, blocks, stream,
                            map_x, map_w, bias, residual, out, M, N, K, error_word);
    if (e != cudaSuccess) {
        cudaGetLastError();
        snprintf(qil_error_text, sizeof(qil_error_text), "%s", cudaGetErrorString(e));
        return (int)e;
    }
    QIL_CHECK_LAUNCH();
}

// M <= 128 rows; the rest as qil_gemm_tc.  (The rows that come without silu_pairs end at a line of the caller's.)  w must be written
// before the kernel before this one begins: it is read while that one may still run.  Measured, us for a tile's K cut into
// 1 / 2 / 4 / 8 at 32 rows, weights from memory: 6144 x 1024 7.2 / 5.8 / 5.8 / 11.4, 4096 x 4096 16.4 / 10.9 / 9.8 / 9.6, 6144 x 4096
// 17.2 / 12.4 / 11.7 / 16.2, 1024 x 3072 12.4 / 7.6 / 5.7 / 5.7, 24576 x 4096 35.2 / 37.5 / 40.6 / 51.7; at 64 rows 6144 x 1024
// 8.9 / 6.3 / 7.3 / 14.9, 4096 x 4096 20.7 / 12.9 / 10.4 / 11.7, 24576 x 4096 37.4 / 41.6 / 46.5 / 65.9: what a block adds up grows with the
// rows and the cluster, so K is cut while a block keeps six stages and the blocks are at most four thirds of the SMs.
extern "C" int qil_gemm_tc_rows(const void* a, const void* w, const void* bias, const void* residual, void* out,
                                int M, int N, int K, int silu_pairs, int sm_count, int* error_word, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (M > 128) QIL_REFUSE("gemm_tc_rows: %d rows, 128 at most", M);
    if (K <= 0 || K % 8) QIL_REFUSE("gemm_tc_rows: K %d must be a positive multiple of 8 (16-byte rows for TMA)", K);
    if (N % 8) QIL_REFUSE("gemm_tc_rows: N %d must be a multiple of 8", N);
    if (((uintptr_t)a | (uintptr_t)w | (uintptr_t)out | (uintptr_t)residual) & 15)
        QIL_REFUSE("gemm_tc_rows: operands must be 16-byte aligned");
    if (silu_pairs && (N % 16 || bias != nullptr || residual != nullptr))
        QIL_REFUSE("gemm_tc_rows: silu_pairs needs N %% 16 == 0 and neither bias nor residual");
    if (error_word == nullptr || sm_count <= 0) QIL_REFUSE("gemm_tc_rows: needs an error word and the SM count");
    const int rows = M <= 32 ? 32 : M <= 64 ? 64 : 128, tiles = (N + TR_BM - 1) / TR_BM, k_blocks = (K + TC_BK - 1) / TC_BK;
    int blocks = 1;
    while (2 * blocks <= TR_MOST_BLOCKS && 6 * 2 * blocks <= k_blocks && tiles * 2 * blocks * 3 <= 4 * sm_count) blocks *= 2;
    CUtensorMap map_x, map_w;
    if (make_map(&map_x, a, M, K, rows)) return -1;
    if (make_map(&map_w, w, N, K, TR_BM)) return -1;
#define ROWS_ARGS map_x, map_w, (const bf16*)bias, (const bf16*)residual, (bf16*)out, M, N, K, blocks, error_word, stream
    if (rows == 32) return silu_pairs ? launch_rows<32, true>(ROWS_ARGS) : launch_rows<32, false>(ROWS_ARGS);
    if (rows == 64) return silu_pairs ? launch_rows<64, true>(ROWS_ARGS) : launch_rows<64, false>(ROWS_ARGS);
    return silu_pairs ? launch_rows<128, true>(ROWS_ARGS) : launch_rows<128, false>(ROWS_ARGS);
#undef ROWS_ARGS
}
