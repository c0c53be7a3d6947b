// C[M,N] = (A[M,K] * W[N,K]^T (+ bias[N])) (* col_scale[N]) (+ residual[M,N]) with float32 FMA on the
// CUDA cores: the matrix product of the true 32-bit path (no TF32, no tensor
// cores), also used when a weight is stored in float32 inside a bfloat16 model.
//
// A row's result does not depend on which other rows share the launch: which kernel takes a product's rows depends on
// how many they are, but all of them sum an element's products in one order.  float32 operands whose rows are whole
// 16-byte vectors and longer than CHAIN_K: K is cut into runs of `run_length(K)` (at most GEMM_RUNS of them), a run is two
// chains of FMA in ascending k, one over its even and one over its odd k (a packed FMA works on both), whose sums are
// added; the runs' sums are added in ascending order.  All others: one chain over K in ascending k.
//
// Weights are row-major [out_features, in_features] as in the checkpoint
// (qil/model.py:32-40: nn.Linear).
#include "common.cuh"

// ---------------------------------------------------------------- float32 operands in whole vectors
#define GEMM_RUNS 8
#define RUN_STEP 32     // runs are multiples of this
// Up to here a product is one run and one chain in ascending k, as in the kernel below that took all of them once.  That
// order is neither faster nor closer to the exact sum than runs are (a step of five rows of a 96-wide model: 71 us with
// runs of 32, 76 with 64, 85 with 128, 96 with the chain).  It is kept for float32 models that are held to an oracle in
// float32: a replayed row of a small Virulix model is compared at 1e-5 (1 + |x|) with an oracle that is itself 1.01e-5 from
// 64 bits there, and left that tolerance (1.17e-5) with runs of 32, 64 and 128 and with the chain up to a K of 80 only.
#define CHAIN_K 256

static __host__ __device__ __forceinline__ int run_length(int K) {
    if (K <= CHAIN_K) return CHAIN_K;
    return (((K + RUN_STEP - 1) / RUN_STEP + GEMM_RUNS - 1) / GEMM_RUNS) * RUN_STEP;
}

// acc += the products of four k's: as two chains, or (CHAIN) as one, whose sum is the lower half of acc
template <bool CHAIN>
__device__ __forceinline__ void fma_quad(unsigned long long& acc, const ulonglong2& a, const ulonglong2& b) {
    if (!CHAIN) {
        fma_pair(acc, a.x, b.x);
        fma_pair(acc, a.y, b.y);
        return;
    }
    const float4 p = *reinterpret_cast<const float4*>(&a), q = *reinterpret_cast<const float4*>(&b);
    float sum = __uint_as_float((unsigned)acc);
    sum = fmaf(p.x, q.x, sum);
    sum = fmaf(p.y, q.y, sum);
    sum = fmaf(p.z, q.z, sum);
    sum = fmaf(p.w, q.w, sum);
    acc = __float_as_uint(sum);
}

__device__ __forceinline__ float pair_sum(unsigned long long v) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    return lo + hi;
}

// Blocks of a cluster share a tile's runs: block r of c takes runs r * GEMM_RUNS / c on.
__device__ __forceinline__ float cluster_read(const float* at, int rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(map_to_rank((unsigned)__cvta_generic_to_shared(at), rank)) : "memory");
    return v;
}

struct GemmArgs {
    const float* A; const float* W; const float* bias; const float* residual; float* C; const float* col_scale;
    int M, N, K, lda;
};

__device__ __forceinline__ void gemm_store(const GemmArgs& g, int m, int n, float v) {
    // every operation rounds by itself, in whichever kernel this is inlined
    if (g.bias != nullptr) v = __fadd_rn(v, g.bias[n]);
    if (g.col_scale != nullptr) v = __fmul_rn(v, g.col_scale[n]);
    if (g.residual != nullptr) v = __fadd_rn(g.residual[(size_t)m * g.N + n], v);
    g.C[(size_t)m * g.N + n] = v;
}

// Up to 16 rows (a decode step): the weights are read once and everything else has to stay out of their way.  A block
// streams 64 weight rows through a ring of stages of 32 k (one 128-byte line a row and stage); a thread holds F
// features and RM rows, MG groups of 64 / F threads share a stage.  Bound by memory at one row (151936 x 1024: 105 us,
// 5.9 TB/s), from eight on by the shared-memory reads of the activations, which broadcast to a warp (143 us; a thread of
// twice the rows or features has too few warps beside it).  The 64 x 64 tiles this replaced took 8 rows like 64: a decode
// step of 8 rows of the 1024-wide model 68.3 ms, 36.9 with this alone.
#define STREAM_BN 64
#define STREAM_BK 32
#define STREAM_LD (STREAM_BK + 4)      // a quarter warp's 16-byte reads of 8 rows meet every bank once

template <int RM, int MG, int F, bool CHAIN>
__global__ void __launch_bounds__(STREAM_BN / F * MG)
gemm_f32_stream_kernel(const GemmArgs g, int stages) {      // stages: 4 or 8
    constexpr int MT = RM * MG, FT = STREAM_BN / F, THREADS = FT * MG;
    constexpr int STAGE = STREAM_BN * STREAM_LD + MT * STREAM_BK;
    extern __shared__ __align__(16) float smem[];
    float* sums = smem + stages * STAGE;                 // [runs of this block][MT][STREAM_BN]
    const unsigned blocks = cluster_blocks(), rank = cluster_rank();
    const int tid = threadIdx.x, f = tid % FT, mg = tid / FT;
    const int n0 = blockIdx.x / blocks * STREAM_BN;
    const int run = run_length(g.K), runs = (g.K + run - 1) / run, per = GEMM_RUNS / blocks;
    const int k_begin = min(g.K, (int)rank * per * run), k_end = min(g.K, ((int)rank + 1) * per * run);
    const int n_stages = (k_end - k_begin + STREAM_BK - 1) / STREAM_BK, run_stages = run / STREAM_BK;

    // the first stages' weight lines are asked of L2 while the kernel before this one ends
    for (int i = tid; i < min(stages, n_stages) * STREAM_BN; i += THREADS) {
        const int row = n0 + i % STREAM_BN, k = k_begin + i / STREAM_BN * STREAM_BK;
        if (row < g.N) asm volatile("prefetch.global.L2 [%0];" ::"l"(g.W + (size_t)row * g.K + k));
    }
    qil_wait_for_producer();
    qil_release_consumer();

    auto load = [&](int stage) {
        if (stage < n_stages) {
            float* ws = smem + stage % stages * STAGE;
            float* as = ws + STREAM_BN * STREAM_LD;
            const int k0 = k_begin + stage * STREAM_BK;
#pragma unroll
            for (int i = tid; i < STREAM_BN * 8; i += THREADS) {
                const int row = i >> 3, k = k0 + (i & 7) * 4;
                const bool inside = n0 + row < g.N && k < k_end;
                copy16(ws + row * STREAM_LD + (i & 7) * 4, inside ? g.W + (size_t)(n0 + row) * g.K + k : g.W, inside);
            }
            for (int i = tid; i < MT * 8; i += THREADS) {
                const int row = i >> 3, k = k0 + (i & 7) * 4;
                const bool inside = row < g.M && k < k_end;
                copy16(as + row * STREAM_BK + (i & 7) * 4, inside ? g.A + (size_t)row * g.lda + k : g.A, inside);
            }
        }
        copies_commit();
    };
    for (int s = 0; s < stages - 1; ++s) load(s);

    unsigned long long acc[F][RM];
    float total[F][RM];
#pragma unroll
    for (int j = 0; j < F; ++j)
#pragma unroll
        for (int r = 0; r < RM; ++r) { acc[j][r] = 0ull; total[j][r] = 0.f; }
    for (int s = 0; s < n_stages; ++s) {
        // the oldest of the groups in flight is this stage
        if (stages == 4) copies_wait<2>(); else copies_wait<6>();
        __syncthreads();
        load(s + stages - 1);
        const float* ws = smem + s % stages * STAGE + f * STREAM_LD;
        const float* as = smem + s % stages * STAGE + STREAM_BN * STREAM_LD + mg * RM * STREAM_BK;
#pragma unroll
        for (int q = 0; q < STREAM_BK / 4; ++q) {
            ulonglong2 w[F];
#pragma unroll
            for (int j = 0; j < F; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(ws + j * FT * STREAM_LD + q * 4);
#pragma unroll
            for (int r = 0; r < RM; ++r) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(as + r * STREAM_BK + q * 4);
#pragma unroll
                for (int j = 0; j < F; ++j) fma_quad<CHAIN>(acc[j][r], a, w[j]);
            }
        }
        if ((s + 1) % run_stages == 0 || s + 1 == n_stages) {
#pragma unroll
            for (int j = 0; j < F; ++j)
#pragma unroll
                for (int r = 0; r < RM; ++r) {
                    const float v = pair_sum(acc[j][r]);
                    acc[j][r] = 0ull;
                    total[j][r] += v;
                    if (blocks > 1) sums[(s / run_stages * MT + mg * RM + r) * STREAM_BN + j * FT + f] = v;
                }
        }
    }
    if (blocks == 1) {
#pragma unroll
        for (int j = 0; j < F; ++j)
#pragma unroll
            for (int r = 0; r < RM; ++r) {
                const int m = mg * RM + r, n = n0 + j * FT + f;
                if (m < g.M && n < g.N) gemm_store(g, m, n, total[j][r]);
            }
        return;
    }
    cluster_sync_all();
    for (int e = rank * THREADS + tid; e < g.M * STREAM_BN; e += blocks * THREADS) {
        if (n0 + e % STREAM_BN >= g.N) continue;
        float v = 0.f;
        for (int r = 0; r < runs; ++r) v += cluster_read(sums + r % per * MT * STREAM_BN + e, r / per);
        gemm_store(g, e / STREAM_BN, n0 + e % STREAM_BN, v);
    }
    cluster_sync_all();      // no block leaves while another reads its sums
}

// More rows: 8 x 4 outputs a thread, tiles of BM x 64, both operands through a ring of stages of 32 k as they lie in
// memory (k innermost, so that a 16-byte read is two packed FMA operands and nothing is transposed or duplicated).
// Without a cluster a block adds its runs' sums up in shared memory; a cluster of GEMM_RUNS takes one run a block.
// Bound by the 16-byte reads of shared memory, each of which returns 512 bytes to a warp whether its lanes share them or
// not: scalar FMA, packed FMA and 8 x 8 outputs a thread all end within 5 %.  So the reads run ahead of the FMA by four k
// and a stage holds 32 k (a barrier half as often): 512 x 6144 x 1024 237 -> 196 us (33 TFLOP/s), 512 x 1024 x 3072 124 ->
// 100; unpipelined 64 x 64 x 16 tiles with scalar FMA ran at 9 TFLOP/s.
#define TILE_BN 64
#define TILE_BK 32
#define TILE_LD (TILE_BK + 4)
#define TILE_STAGES 2

template <int BM, bool CHAIN>
__global__ void __launch_bounds__(BM * 2, BM == 64 ? 3 : 6)
gemm_f32_tile_kernel(const GemmArgs g) {
    constexpr int J = TILE_BN / 16, THREADS = BM * 2, TY = BM / 8, STAGE = (BM + TILE_BN) * TILE_LD;
    extern __shared__ __align__(16) float smem[];
    const unsigned blocks = cluster_blocks(), rank = cluster_rank();
    // one block: its running sums beside the ring; a cluster: the run's sums in the ring's place
    float* sums = blocks > 1 ? smem : smem + TILE_STAGES * STAGE;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // a warp holds 4 x 8 threads; two warps side by side cover the 16 columns of threads
    const int ty = (warp >> 1) * 4 + (lane >> 3), tx = (warp & 1) * 8 + (lane & 7);
    const int n0 = blockIdx.x / blocks * TILE_BN, m0 = blockIdx.y * BM;
    const int run = run_length(g.K), runs = (g.K + run - 1) / run;
    const int k_begin = blocks > 1 ? min(g.K, (int)rank * run) : 0, k_end = blocks > 1 ? min(g.K, k_begin + run) : g.K;
    const int n_stages = (k_end - k_begin + TILE_BK - 1) / TILE_BK, run_stages = run / TILE_BK;
    qil_wait_for_producer();
    qil_release_consumer();

    auto load = [&](int stage) {
        if (stage < n_stages) {
            float* to = smem + stage % TILE_STAGES * STAGE;
            const int k0 = k_begin + stage * TILE_BK;
#pragma unroll
            for (int i = 0; i < (BM + TILE_BN) * 8 / THREADS; ++i) {
                const int idx = tid + i * THREADS, row = idx >> 3, k = k0 + (idx & 7) * 4;
                const float* from;
                bool inside = k < k_end;
                if (row < BM) {
                    inside = inside && m0 + row < g.M;
                    from = g.A + (size_t)(m0 + row) * g.lda + k;
                } else {
                    inside = inside && n0 + row - BM < g.N;
                    from = g.W + (size_t)(n0 + row - BM) * g.K + k;
                }
                copy16(to + row * TILE_LD + (idx & 7) * 4, inside ? from : g.W, inside);
            }
        }
        copies_commit();
    };
    for (int s = 0; s < TILE_STAGES - 1; ++s) load(s);

    unsigned long long acc[8][J];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < J; ++j) acc[i][j] = 0ull;
    for (int s = 0; s < n_stages; ++s) {
        copies_wait<TILE_STAGES - 2>();
        __syncthreads();
        load(s + TILE_STAGES - 1);
        const float* as = smem + s % TILE_STAGES * STAGE + ty * TILE_LD;
        const float* ws = smem + s % TILE_STAGES * STAGE + (BM + tx) * TILE_LD;
        // the next four k's operands are read while these four multiply
        ulonglong2 w[2][J], a[2][8];
        auto read = [&](int q) {
#pragma unroll
            for (int j = 0; j < J; ++j) w[q & 1][j] = *reinterpret_cast<const ulonglong2*>(ws + j * 16 * TILE_LD + q * 4);
#pragma unroll
            for (int i = 0; i < 8; ++i) a[q & 1][i] = *reinterpret_cast<const ulonglong2*>(as + i * TY * TILE_LD + q * 4);
        };
        read(0);
#pragma unroll
        for (int q = 0; q < TILE_BK / 4; ++q) {
            if (q + 1 < TILE_BK / 4) read(q + 1);
            if constexpr (CHAIN) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < J; ++j) fma_quad<true>(acc[i][j], a[q & 1][i], w[q & 1][j]);
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < J; ++j) fma_pair(acc[i][j], a[q & 1][i].x, w[q & 1][j].x);
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < J; ++j) fma_pair(acc[i][j], a[q & 1][i].y, w[q & 1][j].y);
            }
        }
        if (blocks == 1 && ((s + 1) % run_stages == 0 || s + 1 == n_stages)) {
            const bool first = s < run_stages, last = s + 1 == n_stages;
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    float* at = sums + (i * J + j) * THREADS + tid;
                    const float v = pair_sum(acc[i][j]);
                    acc[i][j] = 0ull;
                    const float so_far = first ? v : *at + v;
                    if (!last) {
                        *at = so_far;
                    } else {
                        const int m = m0 + ty + i * TY, n = n0 + tx + j * 16;
                        if (m < g.M && n < g.N) gemm_store(g, m, n, so_far);
                    }
                }
        }
    }
    if (blocks == 1) return;
    copies_wait<0>();
    __syncthreads();            // the ring is read out
    if (n_stages > 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < J; ++j) sums[(ty + i * TY) * TILE_BN + tx + j * 16] = pair_sum(acc[i][j]);
    }
    cluster_sync_all();
    for (int e = rank * THREADS + tid; e < BM * TILE_BN; e += blocks * THREADS) {
        const int m = m0 + e / TILE_BN, n = n0 + e % TILE_BN;
        if (m >= g.M || n >= g.N) continue;
        float v = 0.f;
        for (int r = 0; r < runs; ++r) v += cluster_read(sums + e, r);
        gemm_store(g, m, n, v);
    }
    cluster_sync_all();
}

// ---------------------------------------------------------------- any types, any K
#define BM 64
#define BN 64
#define BK 16

template <typename TA, typename TW>
__global__ void __launch_bounds__(256)
gemm_f32_kernel(const TA* __restrict__ A, const TW* __restrict__ Wt, const TW* __restrict__ bias,
                const TA* residual, TA* C, int M, int N, int K, int lda,
                const float* __restrict__ col_scale) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;      // 16 x 16 threads, 4 x 4 outputs each
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        // 64 rows x 16 k = 1024 elements per operand, 4 per thread
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int idx = tid + e * 256;
            const int r = idx >> 4, kk = idx & 15;
            const int k = k0 + kk;
            float a = 0.f, w = 0.f;
            if (k < K) {
                if (m0 + r < M) a = to_f32<TA>(A[(size_t)(m0 + r) * lda + k]);
                if (n0 + r < N) w = to_f32<TW>(Wt[(size_t)(n0 + r) * K + k]);
            }
            As[kk][r] = a;
            Ws[kk][r] = w;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (bias != nullptr) v += to_f32<TW>(bias[n]);
            if (col_scale != nullptr) v *= col_scale[n];
            if (residual != nullptr) v = to_f32<TA>(residual[(size_t)m * N + n]) + v;
            C[(size_t)m * N + n] = from_f32<TA>(v);
        }
    }
}


// ---------------------------------------------------------------- launches
template <typename... KArgs, typename... Args>
static cudaError_t launch_clusters(void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, int blocks,
                                   cudaStream_t stream, Args... args) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return qil_launch_clusters(kernel, grid, dim3(threads), smem, blocks, stream, args...);
}

template <int RM, int MG, int F>
static cudaError_t launch_stream(const GemmArgs& g, int blocks, int stages, cudaStream_t stream) {
    const int tiles = (g.N + STREAM_BN - 1) / STREAM_BN;
    size_t smem = (size_t)stages * (STREAM_BN * STREAM_LD + RM * MG * STREAM_BK) * sizeof(float);
    if (blocks > 1) smem += (size_t)(GEMM_RUNS / blocks) * RM * MG * STREAM_BN * sizeof(float);
    return launch_clusters(g.K > CHAIN_K ? gemm_f32_stream_kernel<RM, MG, F, false> : gemm_f32_stream_kernel<RM, MG, F, true>,
                           dim3(tiles * blocks), STREAM_BN / F * MG, smem, blocks, stream, g, stages);
}

template <int BM_>
static cudaError_t launch_tile(const GemmArgs& g, int blocks, cudaStream_t stream) {
    const size_t ring = (size_t)TILE_STAGES * (BM_ + TILE_BN) * TILE_LD * sizeof(float);
    const size_t sums = (size_t)BM_ * TILE_BN * sizeof(float);
    const dim3 grid((g.N + TILE_BN - 1) / TILE_BN * blocks, (g.M + BM_ - 1) / BM_);
    return launch_clusters(g.K > CHAIN_K ? gemm_f32_tile_kernel<BM_, false> : gemm_f32_tile_kernel<BM_, true>, grid, BM_ * 2, blocks > 1 ? (ring > sums ? ring : sums) : ring + sums,
                           blocks, stream, g);
}

// What `count` blocks of the 64-row tile kernel take, in waves of three blocks an SM.  An SM works through one block in
// half the time it takes for three.
static double tile_waves(long long count) {
    const long long rest = count % (3 * 148);
    return (double)(count / (3 * 148)) + (rest == 0 ? 0. : rest <= 148 ? 0.52 : rest <= 222 ? 0.75 : 1.);
}

// Which kernel, and how many blocks share a tile's runs.  Measured with weights streamed from memory, us:
//   stream kernel, cluster of 1 / 2 / 4 / 8: 8 rows 4096 x 1024 19.3 / 12.2 / 9.4 / 10.0, 1024 x 3072 55.7 / 30.1 /
//   16.0 / 11.6; 1 row 151936 x 1024 105 / 138 / 109 / 144.  So a cluster as large as fills five blocks an SM.
//   16 rows with the stream kernel 10.5 and 14.7 (4096 x 1024, 1024 x 3072), 24 with 32-row tiles 18.1 and 22.3.
//   32-row tiles against 64-row tiles: 64 rows 28.4 / 31.3 and 27.6 / 34.3; 128 rows the wider ones halve the weight reads.
//   64-row tiles (with stages of 16 k) alone and in clusters of eight: 128 x 4096 x 1024 64.5 / 49.7, 512 x 1024 x 3072 173 / 123, 512 x 6144 x
//   1024 237 / 253: a cluster costs a quarter on top and pays where its finer blocks fill the SMs better than that.
static cudaError_t gemm_f32_vectors(const GemmArgs& g, cudaStream_t stream) {
    const long long columns = (g.N + 63) / 64;             // STREAM_BN and TILE_BN
    const bool chain = g.K <= CHAIN_K;                     // one run: nothing for a cluster to share
    if (g.M <= 16) {
        int blocks = 1;
        while (!chain && blocks < GEMM_RUNS && columns * blocks < 5 * 148) blocks *= 2;
        const int stages = columns * blocks <= 2 * 148 ? 8 : 4;        // few blocks: a deeper ring in each
        if (g.M <= 1) return launch_stream<1, 1, 1>(g, blocks, stages, stream);
        if (g.M <= 2) return launch_stream<2, 1, 1>(g, blocks, stages, stream);
        if (g.M <= 4) return launch_stream<2, 2, 1>(g, blocks, stages, stream);
        if (g.M <= 8) return launch_stream<4, 2, 1>(g, blocks, stages, stream);
        return launch_stream<4, 4, 2>(g, blocks, stages, stream);
    }
    if (g.M <= 64) return launch_tile<32>(g, !chain && columns * ((g.M + 31) / 32) < 6 * 148 ? GEMM_RUNS : 1, stream);
    const long long tiles = columns * ((g.M + 63) / 64);
    return launch_tile<64>(g, !chain && tile_waves(tiles) * GEMM_RUNS > 1.25 * tile_waves(tiles * GEMM_RUNS) ? GEMM_RUNS : 1, stream);
}

// residual may alias C (each element is read and written by the same thread).
extern "C" int qil_gemm_f32(const void* A, int lda, const void* Wt, const void* bias, const void* residual,
                            void* C, int M, int N, int K, int act_dtype, int weight_dtype,
                            const float* col_scale, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || lda < K) QIL_REFUSE("gemm_f32: K %d lda %d", K, lda);
    if ((M + BM - 1) / BM > 65535) QIL_REFUSE("gemm_f32: M %d is too large for one launch", M);
    if (act_dtype == QIL_F32 && weight_dtype == QIL_F32 && K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)Wt) & 15) == 0) {
        const GemmArgs g = {(const float*)A, (const float*)Wt, (const float*)bias, (const float*)residual, (float*)C, col_scale, M, N, K, lda};
        const cudaError_t e = gemm_f32_vectors(g, stream);
        if (e != cudaSuccess) {
            cudaGetLastError();             // reported here: the next launch does not answer for it
            snprintf(qil_error_text, sizeof(qil_error_text), "%s", cudaGetErrorString(e));
            return (int)e;
        }
        QIL_CHECK_LAUNCH();
    }
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    QIL_DISPATCH_2(act_dtype, weight_dtype,
        (gemm_f32_kernel<T, W><<<grid, 256, 0, stream>>>((const T*)A, (const W*)Wt, (const W*)bias,
                                                        (const T*)residual, (T*)C, M, N, K, lda, col_scale)));
    QIL_CHECK_LAUNCH();
}
