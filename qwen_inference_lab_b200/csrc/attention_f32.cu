// Causal grouped-query attention over paged float32 keys and values for heads of 32, 64 and 128: the attention of the
// true 32-bit path, float32 FMA on the CUDA cores (csrc/attention_generic.cu takes every other head size, type and
// option).
//
// A token's result is the same bits however a step was cut and whatever else is in it.  Both kernels below do the same
// arithmetic per query: keys are cut at absolute positions into spans of SPAN; a score is two chains of FMA over the
// even and the odd elements of the head (one packed FMA does both); within a span the softmax takes the span's own
// maximum, lane l of a warp sums the weights of keys l, l + 32, ... and a fixed tree sums the lanes; values are added
// by one chain of FMA in ascending key order; spans join in ascending order (`join`).
#include "common.cuh"

#define SPAN 256

__device__ __forceinline__ float2 pair_of(unsigned long long v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ unsigned long long twice(float v) {
    unsigned long long p;
    asm("mov.b64 %0, {%1, %1};" : "=l"(p) : "f"(v));
    return p;
}
struct Pages {
    const float* cache;
    const int* block_table;
    int table_stride, n_kv_heads, page_size, num_pages;
};

// element offset of a key's row for a kv head, -1 where there is none (its value row lies n_kv_heads * page_size rows on)
template <int D>
__device__ __forceinline__ long long row_offset(const Pages& p, const int* table, int kv_head, int key) {
    const int index = key / p.page_size;
    const int page = index < p.table_stride ? table[index] : -1;
    if (page < 0 || page >= p.num_pages) return -1;
    return ((long long)page * 2 * p.n_kv_heads * p.page_size + (long long)kv_head * p.page_size + key % p.page_size) * D;
}

// one query's scores over a span -> weights in place; (maximum, sum) to every lane
__device__ __forceinline__ float2 span_softmax(float* scores, int lane) {
    float s[SPAN / 32], m = -INFINITY, l = 0.f;
#pragma unroll
    for (int j = 0; j < SPAN / 32; ++j) {
        s[j] = scores[j * 32 + lane];
        m = fmaxf(m, s[j]);
    }
    m = warp_max(m);
#pragma unroll
    for (int j = 0; j < SPAN / 32; ++j) {
        const float p = s[j] == -INFINITY ? 0.f : expf(s[j] - m);
        scores[j * 32 + lane] = p;
        l += p;
    }
    return make_float2(m, warp_sum(l));
}

// what a span changes about the running (maximum, sum): the factors of what was there and of what it brings
__device__ __forceinline__ float2 join(float& m_run, float& l_run, float m, float l) {
    const float m_new = fmaxf(m_run, m), keep = expf(m_run - m_new), bring = expf(m - m_new);
    l_run = fmaf(l_run, keep, __fmul_rn(l, bring));
    m_run = m_new;
    return make_float2(keep, bring);
}

// ---------------------------------------------------------------- single tokens
// A block takes one span of one (token, kv head) and all its query heads, so that keys and values are read once.  They
// come through a ring of SINGLE_SLOTS stages of 16 KB: first the keys, 32 elements of 128 of them a stage (a key a
// thread, whose sums stay in registers over the stages of a head), then the values, 4096 / D whole rows a stage (a value
// element a thread).  Spans of a token are joined by the block that draws its last ticket.  A span that does not hold the
// token itself asks for its first stages before the kernel before this one, which writes the token's own key and value,
// has ended.  Bound by memory and a block's chain of stages: 8 tokens of 16 heads at contexts up to 2000 read 85 MB a
// layer.  (Keys by whole rows, 32 of them a stage and a warp a query head, left two of four warps idle with two heads a
// kv head: 34 us a layer; the step with this form and the chained launches around it 2.80 -> 2.35 ms.)
#define SINGLE_THREADS 128
#define SINGLE_STAGE 4096       // floats
#define SINGLE_SLOTS 4

template <int D, int G>     // G: query heads per kv head, rounded up
__global__ void __launch_bounds__(SINGLE_THREADS)
attention_f32_single_kernel(const float* __restrict__ q, const Pages pages, float* __restrict__ out,
                            const int* __restrict__ info, float* part_o, float* part_ml, int* tickets,
                            int n_q_heads, int window, float scale) {
    constexpr int PARTS = SINGLE_THREADS / D, PER = (G + PARTS - 1) / PARTS, CHUNKS = D / 32, VALUES = SINGLE_STAGE / D;
    extern __shared__ __align__(16) float smem[];
    long long* offsets = reinterpret_cast<long long*>(smem);               // [SPAN]
    float* ring = smem + 2 * SPAN;                                         // [SLOTS][STAGE]
    float* qs = ring + SINGLE_SLOTS * SINGLE_STAGE;                        // [G][D]
    float* ps = qs + G * D;                                                // [G][SPAN]
    float* ml = ps + G * SPAN;                                             // [G][2]
    __shared__ int drawn;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i = blockIdx.x / pages.n_kv_heads, kv_head = blockIdx.x % pages.n_kv_heads, span = blockIdx.y;
    const int group = n_q_heads / pages.n_kv_heads;
    const int token = info[4 * i], pos = info[4 * i + 1];
    const int lo = window > 0 && pos - window + 1 > 0 ? pos - window + 1 : 0;
    const int first_span = lo / SPAN, n_spans = pos / SPAN - first_span + 1;
    if (span < first_span || span >= first_span + n_spans) { qil_wait_for_producer(); return; }
    const int* table = pages.block_table + (size_t)info[4 * i + 2] * pages.table_stride;
    const int key0 = span * SPAN, from_key = max(lo - key0, 0), last_key = min(pos - key0, SPAN - 1);
    for (int k = tid; k < SPAN; k += SINGLE_THREADS)
        offsets[k] = k >= from_key && k <= last_key ? row_offset<D>(pages, table, kv_head, key0 + k) : -1;
    for (int k = tid; k < G * SPAN; k += SINGLE_THREADS) ps[k] = -INFINITY;
    __syncthreads();

    const int k_begin = from_key / SINGLE_THREADS, k_stages = (last_key / SINGLE_THREADS + 1 - k_begin) * CHUNKS;
    const int v_begin = from_key / VALUES, n_stages = k_stages + last_key / VALUES + 1 - v_begin;
    const long long plane = (long long)pages.n_kv_heads * pages.page_size * D;
    auto load = [&](int stage) {
        if (stage < n_stages) {
            float* to = ring + stage % SINGLE_SLOTS * SINGLE_STAGE;
            if (stage < k_stages) {
                // a key's 8 pieces of 16 bytes lie in an order of its own: 8 threads that read one piece of 8 keys each
                // then meet every bank once
                const int row0 = (k_begin + stage / CHUNKS) * SINGLE_THREADS;
                const float* from = pages.cache + stage % CHUNKS * 32;
#pragma unroll
                for (int n = 0; n < SINGLE_STAGE / 4 / SINGLE_THREADS; ++n) {
                    const int row = n * 16 + (tid >> 3), piece = tid & 7;
                    const long long at = offsets[row0 + row];
                    copy16(to + row * 32 + (piece ^ (row & 7)) * 4, at >= 0 ? from + at + piece * 4 : pages.cache, at >= 0);
                }
            } else {
                const int row0 = (v_begin + stage - k_stages) * VALUES;
#pragma unroll
                for (int n = 0; n < SINGLE_STAGE / 4 / SINGLE_THREADS; ++n) {
                    const int idx = n * SINGLE_THREADS + tid, row = idx / (D / 4), col = idx % (D / 4) * 4;
                    const long long at = offsets[row0 + row];
                    copy16(to + row * D + col, at >= 0 ? pages.cache + plane + at + col : pages.cache, at >= 0);
                }
            }
        }
        copies_commit();
    };
    const bool early = pos - key0 >= SPAN;
    if (early)
        for (int s = 0; s < SINGLE_SLOTS - 1; ++s) load(s);
    qil_wait_for_producer();
    qil_release_consumer();
    if (!early)
        for (int s = 0; s < SINGLE_SLOTS - 1; ++s) load(s);
    const float* q_rows = q + ((size_t)token * n_q_heads + kv_head * group) * D;
    for (int k = tid; k < G * D; k += SINGLE_THREADS) qs[k] = k < group * D ? q_rows[k] : 0.f;

    unsigned long long dot[G];
#pragma unroll
    for (int r = 0; r < G; ++r) dot[r] = 0ull;
    for (int s = 0; s < k_stages; ++s) {
        copies_wait<SINGLE_SLOTS - 2>();
        __syncthreads();
        load(s + SINGLE_SLOTS - 1);
        const float* row = ring + s % SINGLE_SLOTS * SINGLE_STAGE + tid * 32;
        const float* qc = qs + s % CHUNKS * 32;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const ulonglong2 k4 = *reinterpret_cast<const ulonglong2*>(row + (c ^ (tid & 7)) * 4);
#pragma unroll
            for (int r = 0; r < G; ++r) {
                const ulonglong2 q4 = *reinterpret_cast<const ulonglong2*>(qc + r * D + c * 4);
                fma_pair(dot[r], q4.x, k4.x);
                fma_pair(dot[r], q4.y, k4.y);
            }
        }
        if (s % CHUNKS == CHUNKS - 1) {
            const int k = (k_begin + s / CHUNKS) * SINGLE_THREADS + tid;
            const bool there = offsets[k] >= 0;
#pragma unroll
            for (int r = 0; r < G; ++r) {
                const float2 halves = pair_of(dot[r]);
                if (there) ps[r * SPAN + k] = (halves.x + halves.y) * scale;
                dot[r] = 0ull;
            }
        }
    }
    __syncthreads();
    for (int r = warp; r < group; r += SINGLE_THREADS / 32) {
        const float2 v = span_softmax(ps + r * SPAN, lane);
        if (lane == 0) { ml[2 * r] = v.x; ml[2 * r + 1] = v.y; }
    }
    float acc[PER];
#pragma unroll
    for (int r = 0; r < PER; ++r) acc[r] = 0.f;
    const int d = tid % D, part = tid / D;      // a thread sums one value element of every PARTS-th query head
    for (int s = k_stages; s < n_stages; ++s) {
        copies_wait<SINGLE_SLOTS - 2>();
        __syncthreads();
        load(s + SINGLE_SLOTS - 1);
        const float* rows = ring + s % SINGLE_SLOTS * SINGLE_STAGE + d;
        const int k0 = (v_begin + s - k_stages) * VALUES;
        const int last = min(VALUES, last_key - k0 + 1);
#pragma unroll 4
        for (int k = 0; k < last; k += 4) {     // rows past the last key are zeros with weight zero
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = rows[(k + e) * D];
#pragma unroll
            for (int r = 0; r < PER; ++r) {
                if (part + r * PARTS >= G) continue;
                const float4 p = *reinterpret_cast<const float4*>(ps + (part + r * PARTS) * SPAN + k0 + k);
                acc[r] = fmaf(p.x, v[0], acc[r]);
                acc[r] = fmaf(p.y, v[1], acc[r]);
                acc[r] = fmaf(p.z, v[2], acc[r]);
                acc[r] = fmaf(p.w, v[3], acc[r]);
            }
        }
    }
    float* out_rows = out + ((size_t)token * n_q_heads + kv_head * group) * D;
    if (n_spans == 1) {
#pragma unroll
        for (int r = 0; r < PER; ++r) {
            const int h = part + r * PARTS;
            if (h < group) out_rows[h * D + d] = ml[2 * h + 1] > 0.f ? acc[r] / ml[2 * h + 1] : 0.f;
        }
        return;
    }
    const size_t slot0 = ((size_t)i * n_q_heads + kv_head * group) * gridDim.y;    // [query head of the group][span]
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        const int h = part + r * PARTS;
        if (h >= group) continue;
        const size_t slot = slot0 + (size_t)h * gridDim.y + span;
        part_o[slot * D + d] = acc[r];
        if (d == 0) { part_ml[2 * slot] = ml[2 * h]; part_ml[2 * slot + 1] = ml[2 * h + 1]; }
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) drawn = atomicAdd(tickets + blockIdx.x, 1);
    __syncthreads();
    if (drawn != n_spans - 1) return;
    if (tid == 0) tickets[blockIdx.x] = 0;
    __threadfence();
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        const int h = part + r * PARTS;
        if (h >= group) continue;
        float m_run = -INFINITY, l_run = 0.f, o_run = 0.f;
        const size_t slot = slot0 + (size_t)h * gridDim.y + first_span;
#pragma unroll 8
        for (int s = 0; s < n_spans; ++s) {
            const float2 v = __ldcg(reinterpret_cast<const float2*>(part_ml) + slot + s);
            const float o = __ldcg(part_o + (slot + s) * D + d);
            if (v.y == 0.f) continue;           // no key was seen (weights that are not a number do count)
            const float2 f = join(m_run, l_run, v.x, v.y);
            o_run = fmaf(o_run, f.x, __fmul_rn(o, f.y));
        }
        out_rows[h * D + d] = l_run > 0.f ? o_run / l_run : 0.f;
    }
}

// ---------------------------------------------------------------- prompt portions
// A block takes 64 query rows (the query heads of a kv head for as many consecutive tokens) and walks the spans.  A span's
// keys come 32 elements at a time, all 256 of them a stage of 32 KB, and a thread holds 8 x 8 scores over the stages of a
// head; its values come 8192 / D rows a stage, and a thread holds 4 elements of 64 * D / 1024 rows.  Bound by the 16-byte
// reads of shared memory, each of which returns 512 bytes to a warp whether its lanes share them or not.
#define TILE_THREADS 256
#define TILE_ROWS 64
#define TILE_STAGE 8192         // floats
#define TILE_SLOTS 3
#define SCORE_LD (SPAN + 4)

template <int D>
__global__ void __launch_bounds__(TILE_THREADS)
attention_f32_tile_kernel(const float* __restrict__ q, const Pages pages, float* __restrict__ out,
                          const int* __restrict__ info, int n_subtiles, int singles, int n_q_heads, int window, float scale) {
    constexpr int LD = D + 4, GROUPS = TILE_THREADS / (D / 4), PER = TILE_ROWS / GROUPS, CHUNKS = D / 32, VALUES = TILE_STAGE / D;
    extern __shared__ __align__(16) float smem[];
    long long* offsets = reinterpret_cast<long long*>(smem);               // [SPAN]
    float* ring = smem + 2 * SPAN;                                         // [SLOTS][STAGE]
    float* qs = ring + TILE_SLOTS * TILE_STAGE;                            // [64][LD]
    float* ps = qs + TILE_ROWS * LD;                                       // [64][SCORE_LD]
    float* ml = ps + TILE_ROWS * SCORE_LD;                                 // [64][2]
    qil_wait_for_producer();
    qil_release_consumer();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kv_head = blockIdx.y, group = n_q_heads / pages.n_kv_heads, per_tile = TILE_ROWS / group;
    const int* mine = info + 4 * (blockIdx.x / n_subtiles);
    const int skip = blockIdx.x % n_subtiles * per_tile;
    const int tokens = min(per_tile, (singles ? 1 : mine[2]) - skip);
    if (tokens <= 0) return;
    const int token0 = mine[0] + skip, pos0 = mine[1] + skip, rows = tokens * group;
    const int* table = pages.block_table + (size_t)mine[singles ? 2 : 3] * pages.table_stride;
    auto low = [&](int pos) { return window > 0 && pos - window + 1 > 0 ? pos - window + 1 : 0; };
    const int lo = low(pos0), hi = pos0 + tokens - 1;
    for (int idx = tid; idx < TILE_ROWS * (D / 4); idx += TILE_THREADS) {
        const int row = idx / (D / 4), col = idx % (D / 4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < rows)
            v = *reinterpret_cast<const float4*>(q + ((size_t)(token0 + row / group) * n_q_heads + kv_head * group + row % group) * D + col);
        *reinterpret_cast<float4*>(qs + row * LD + col) = v;
    }
    // scores: rows ry + 8 i, keys kx + 32 j of a span (a warp holds 4 x 8 threads); values: columns d .. d + 3 of
    // rows row0 .. row0 + PER - 1
    const int ry = (warp >> 2) * 4 + (lane >> 3), kx = (warp & 3) * 8 + (lane & 7);
    const int d = tid % (D / 4) * 4, row0 = tid / (D / 4) * PER;
    const long long plane = (long long)pages.n_kv_heads * pages.page_size * D;
    float m_run[PER], l_run[PER], o_run[PER][4];
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        m_run[r] = -INFINITY; l_run[r] = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) o_run[r][e] = 0.f;
    }

    for (int span = lo / SPAN; span <= hi / SPAN; ++span) {
        const int key0 = span * SPAN, from_key = max(lo - key0, 0), last_key = min(hi - key0, SPAN - 1);
        const int v_begin = from_key / VALUES, n_stages = CHUNKS + last_key / VALUES + 1 - v_begin;
        __syncthreads();                        // the span before is read out
        for (int k = tid; k < SPAN; k += TILE_THREADS)
            offsets[k] = k >= from_key && k <= last_key ? row_offset<D>(pages, table, kv_head, key0 + k) : -1;
        for (int idx = tid; idx < TILE_ROWS * (SCORE_LD / 4); idx += TILE_THREADS)
            reinterpret_cast<float4*>(ps)[idx] = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        __syncthreads();
        auto load = [&](int stage) {            // the first CHUNKS stages are the keys, the rest the values
            if (stage < n_stages) {
                float* to = ring + stage % TILE_SLOTS * TILE_STAGE;
                if (stage < CHUNKS) {
                    // a key's 8 pieces of 16 bytes lie in an order of its own, as in the kernel above
#pragma unroll
                    for (int n = 0; n < SPAN * 8 / TILE_THREADS; ++n) {
                        const int row = n * (TILE_THREADS / 8) + (tid >> 3), piece = tid & 7;
                        const long long at = offsets[row];
                        copy16(to + row * 32 + (piece ^ (row & 7)) * 4, at >= 0 ? pages.cache + at + stage * 32 + piece * 4 : pages.cache, at >= 0);
                    }
                } else {
                    const int rows0 = (v_begin + stage - CHUNKS) * VALUES;
#pragma unroll
                    for (int n = 0; n < TILE_STAGE / 4 / TILE_THREADS; ++n) {
                        const int idx = n * TILE_THREADS + tid, row = idx / (D / 4), col = idx % (D / 4) * 4;
                        const long long at = offsets[rows0 + row];
                        copy16(to + row * D + col, at >= 0 ? pages.cache + plane + at + col : pages.cache, at >= 0);
                    }
                }
            }
            copies_commit();
        };
        for (int s = 0; s < TILE_SLOTS - 1; ++s) load(s);
        {
            const int j_begin = from_key / 32, j_end = last_key / 32 + 1;       // 32 keys that hold none are left out
            unsigned long long dot[8][8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) dot[i][j] = 0ull;
            for (int s = 0; s < CHUNKS; ++s) {
                copies_wait<TILE_SLOTS - 2>();
                __syncthreads();
                load(s + TILE_SLOTS - 1);
                const float* stage = ring + s % TILE_SLOTS * TILE_STAGE + kx * 32;
                const float* qc = qs + ry * LD + s * 32;
#pragma unroll 2
                for (int c = 0; c < 8; ++c) {
                    ulonglong2 q4[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) q4[i] = *reinterpret_cast<const ulonglong2*>(qc + i * 8 * LD + c * 4);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (j < j_begin || j >= j_end) continue;
                        const ulonglong2 k4 = *reinterpret_cast<const ulonglong2*>(stage + j * 32 * 32 + (c ^ (kx & 7)) * 4);
#pragma unroll
                        for (int i = 0; i < 8; ++i) fma_pair(dot[i][j], q4[i].x, k4.x);
#pragma unroll
                        for (int i = 0; i < 8; ++i) fma_pair(dot[i][j], q4[i].y, k4.y);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int k = kx + 32 * j, key = key0 + k;
                const bool there = offsets[k] >= 0;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int row = ry + 8 * i, pos = pos0 + row / group;
                    const float2 halves = pair_of(dot[i][j]);
                    if (there && row < rows && key <= pos && key >= low(pos)) ps[row * SCORE_LD + k] = (halves.x + halves.y) * scale;
                }
            }
        }
        __syncthreads();
        for (int r = warp; r < rows; r += TILE_THREADS / 32) {
            const float2 v = span_softmax(ps + r * SCORE_LD, lane);
            if (lane == 0) { ml[2 * r] = v.x; ml[2 * r + 1] = v.y; }
        }
        unsigned long long acc[PER][2];
#pragma unroll
        for (int r = 0; r < PER; ++r) acc[r][0] = acc[r][1] = 0ull;
        for (int s = CHUNKS; s < n_stages; ++s) {
            copies_wait<TILE_SLOTS - 2>();
            __syncthreads();
            load(s + TILE_SLOTS - 1);
            const float* stage = ring + s % TILE_SLOTS * TILE_STAGE + d;
            const int k0 = (v_begin + s - CHUNKS) * VALUES;
            // where every key of the stage is seen by every row no key is skipped; elsewhere a key that a row does not see
            // must not reach its sum even with weight zero (its value may be an infinity)
            if (key0 + k0 + VALUES - 1 <= pos0 && key0 + k0 >= low(hi)) {
#pragma unroll 2
                for (int k = 0; k < VALUES; k += 4) {
                    ulonglong2 v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[e] = *reinterpret_cast<const ulonglong2*>(stage + (k + e) * D);
#pragma unroll
                    for (int r = 0; r < PER; ++r) {
                        const float4 p = *reinterpret_cast<const float4*>(ps + (row0 + r) * SCORE_LD + k0 + k);
                        fma_pair(acc[r][0], twice(p.x), v[0].x); fma_pair(acc[r][1], twice(p.x), v[0].y);
                        fma_pair(acc[r][0], twice(p.y), v[1].x); fma_pair(acc[r][1], twice(p.y), v[1].y);
                        fma_pair(acc[r][0], twice(p.z), v[2].x); fma_pair(acc[r][1], twice(p.z), v[2].y);
                        fma_pair(acc[r][0], twice(p.w), v[3].x); fma_pair(acc[r][1], twice(p.w), v[3].y);
                    }
                }
            } else {
                // four rows at a time over the keys that any of them sees
                constexpr int Q = PER < 4 ? PER : 4;
#pragma unroll
                for (int r0 = 0; r0 < PER; r0 += Q) {
                    int from[Q], to[Q], first = VALUES, end = 0;
#pragma unroll
                    for (int r = 0; r < Q; ++r) {
                        const int pos = pos0 + (row0 + r0 + r) / group;
                        from[r] = max(0, low(pos) - key0 - k0);
                        to[r] = row0 + r0 + r < rows ? min(VALUES, pos - key0 - k0 + 1) : 0;
                        first = min(first, from[r]);
                        end = max(end, to[r]);
                    }
                    for (int k = first; k < end; ++k) {
                        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(stage + k * D);
#pragma unroll
                        for (int r = 0; r < Q; ++r)
                            if (k >= from[r] && k < to[r]) {
                                const unsigned long long p = twice(ps[(row0 + r0 + r) * SCORE_LD + k0 + k]);
                                fma_pair(acc[r0 + r][0], p, v.x); fma_pair(acc[r0 + r][1], p, v.y);
                            }
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < PER; ++r) {
            if (row0 + r >= rows) continue;
            const float m = ml[2 * (row0 + r)], l = ml[2 * (row0 + r) + 1];
            if (l == 0.f) continue;             // no key was seen (weights that are not a number do count)
            const float2 f = join(m_run[r], l_run[r], m, l), a = pair_of(acc[r][0]), b = pair_of(acc[r][1]);
            o_run[r][0] = fmaf(o_run[r][0], f.x, __fmul_rn(a.x, f.y));
            o_run[r][1] = fmaf(o_run[r][1], f.x, __fmul_rn(a.y, f.y));
            o_run[r][2] = fmaf(o_run[r][2], f.x, __fmul_rn(b.x, f.y));
            o_run[r][3] = fmaf(o_run[r][3], f.x, __fmul_rn(b.y, f.y));
        }
    }
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        const int row = row0 + r;
        if (row >= rows) continue;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (l_run[r] > 0.f)
            v = make_float4(o_run[r][0] / l_run[r], o_run[r][1] / l_run[r], o_run[r][2] / l_run[r], o_run[r][3] / l_run[r]);
        *reinterpret_cast<float4*>(out + ((size_t)(token0 + row / group) * n_q_heads + kv_head * group + row % group) * D + d) = v;
    }
}

// ---------------------------------------------------------------- launches
template <typename Kernel, typename... Args>
static int launch(Kernel kernel, dim3 grid, int threads, size_t smem, cudaStream_t stream, Args... args) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = qil_launch_chained(kernel, grid, dim3(threads), smem, stream, args...);
    if (e != cudaSuccess) {
        cudaGetLastError();
        snprintf(qil_error_text, sizeof(qil_error_text), "%s", cudaGetErrorString(e));
        return (int)e;
    }
    QIL_CHECK_LAUNCH();
}

template <int D, int G>
static int launch_single(const float* q, const Pages& pages, float* out, const int* info, int n, int n_spans, float* part_o,
                         float* part_ml, int* tickets, int n_q_heads, int window, float scale, cudaStream_t stream) {
    const size_t smem = (size_t)(2 * SPAN + SINGLE_SLOTS * SINGLE_STAGE + G * (D + SPAN + 2)) * sizeof(float);
    return launch(attention_f32_single_kernel<D, G>, dim3(n * pages.n_kv_heads, n_spans), SINGLE_THREADS, smem, stream, q, pages,
                  out, info, part_o, part_ml, tickets, n_q_heads, window, scale);
}

template <int D>
static int launch_tile(const float* q, const Pages& pages, float* out, const int* info, int n, int singles, int tile_tokens,
                       int n_q_heads, int window, float scale, cudaStream_t stream) {
    const size_t smem = (size_t)(2 * SPAN + TILE_SLOTS * TILE_STAGE + TILE_ROWS * (D + 4) + TILE_ROWS * (SCORE_LD + 2)) * sizeof(float);
    const int per_tile = TILE_ROWS / (n_q_heads / pages.n_kv_heads), subtiles = singles ? 1 : (tile_tokens + per_tile - 1) / per_tile;
    return launch(attention_f32_tile_kernel<D>, dim3(n * subtiles, pages.n_kv_heads), TILE_THREADS, smem, stream, q, pages, out, info,
                  subtiles, singles, n_q_heads, window, scale);
}

static int check(const void* q, const void* cache, const void* out, int n_q_heads, const Pages& p, int head_dim, int window) {
    if (p.n_kv_heads <= 0 || n_q_heads <= 0 || n_q_heads % p.n_kv_heads || n_q_heads / p.n_kv_heads > TILE_ROWS || p.n_kv_heads > 65535)
        QIL_REFUSE("attention_f32: %d query heads over %d kv heads", n_q_heads, p.n_kv_heads);
    if (head_dim != 32 && head_dim != 64 && head_dim != 128) QIL_REFUSE("attention_f32: heads of %d", head_dim);
    if (p.page_size <= 0 || window < 0) QIL_REFUSE("attention_f32: page_size %d window %d", p.page_size, window);
    if ((((uintptr_t)q | (uintptr_t)cache | (uintptr_t)out) & 15) != 0) QIL_REFUSE("attention_f32: operands must start on 16 bytes");
    return 0;
}

// info int32 [n][4]: (first token, its position, tokens up to tile_tokens, block-table row) a tile of consecutive
// tokens; with `singles` (token, its position, block-table row, unused) a token
extern "C" int qil_attention_f32_tiles(const void* q, const void* cache, void* out, const int* info, int n, int singles, int tile_tokens,
                                       const int* block_table, int table_stride, int n_q_heads, int n_kv_heads, int head_dim,
                                       int page_size, int num_pages, int window, float scale, cudaStream_t stream) {
    if (n <= 0) return 0;
    const Pages pages = {(const float*)cache, block_table, table_stride, n_kv_heads, page_size, num_pages};
    const int refused = check(q, cache, out, n_q_heads, pages, head_dim, window);
    if (refused) return refused;
    if (!singles && tile_tokens <= 0) QIL_REFUSE("attention_f32: tiles of %d tokens", tile_tokens);
#define ARGS (const float*)q, pages, (float*)out, info, n, singles, tile_tokens, n_q_heads, window, scale, stream
    if (head_dim == 32) return launch_tile<32>(ARGS);
    if (head_dim == 64) return launch_tile<64>(ARGS);
    return launch_tile<128>(ARGS);
#undef ARGS
}

// info as with `singles` above; every position lies below n_spans * SPAN; part_o [n][n_q_heads][n_spans][head_dim] and
// part_ml [n][n_q_heads][n_spans][2] float32 scratch; tickets int32 [n * n_kv_heads], zero before and after
extern "C" int qil_attention_f32_singles(const void* q, const void* cache, void* out, const int* info, int n, int n_spans,
                                         float* part_o, float* part_ml, int* tickets, const int* block_table, int table_stride,
                                         int n_q_heads, int n_kv_heads, int head_dim, int page_size, int num_pages, int window,
                                         float scale, cudaStream_t stream) {
    if (n <= 0) return 0;
    const Pages pages = {(const float*)cache, block_table, table_stride, n_kv_heads, page_size, num_pages};
    const int refused = check(q, cache, out, n_q_heads, pages, head_dim, window);
    if (refused) return refused;
    const int group = n_q_heads / n_kv_heads;
    if (group > 8) QIL_REFUSE("attention_f32: %d query heads a kv head for single tokens", group);
    if (n_spans <= 0 || n_spans > 65535) QIL_REFUSE("attention_f32: %d spans", n_spans);
#define ARGS (const float*)q, pages, (float*)out, info, n, n_spans, part_o, part_ml, tickets, n_q_heads, window, scale, stream
#define BY_GROUP(D) return group == 1 ? launch_single<D, 1>(ARGS) : group == 2 ? launch_single<D, 2>(ARGS) \
                         : group <= 4 ? launch_single<D, 4>(ARGS) : launch_single<D, 8>(ARGS)
    if (head_dim == 32) BY_GROUP(32);
    if (head_dim == 64) BY_GROUP(64);
    BY_GROUP(128);
#undef BY_GROUP
#undef ARGS
}

extern "C" int qil_attention_f32_span() { return SPAN; }
