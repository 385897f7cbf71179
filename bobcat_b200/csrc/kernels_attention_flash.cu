// Prefill attention for heads of 64, 128 or 256 elements over an f16 cache: 64-key tiles, online softmax, the two
// products on tensor cores. Counterpart of attention_flash (crates/bobcat-metal/src/attention.metal:290-480), which
// the reference uses for head_dim == 64 and at least 32 queries (backend.rs:2185-2225); the wider heads (Qwen3.5's
// attention layers have 256 elements) take the same path here instead of the chunk kernels.
//
// Arithmetic. Keys and values are the cache's fp16 values, exactly. The scaled query and the
// probabilities are each split into two fp16 halves (value = hi + lo, about 22 bits), so neither
// is rounded to fp16: every product is fp16 x fp16 accumulated in f32, and the result differs from
// an f32 evaluation only by summation order. The row maximum, exponentials (expf) and row sums are
// f32, as in the chunk kernels.
//
// Work. A CTA of eight warps takes 128 rows of one KV head (four warps and 64 rows for heads of 64), a row being a query of one of the heads that share it (the
// heads of a query are neighbouring rows), so a tile of keys is fetched once for all of them. The keys are
// also cut, into `splits` neighbouring parts of a CTA's tiles, where that fills the device: 64 queries of eight heads are four CTAs
// otherwise. Each part leaves its unnormalised sums with its maximum and sum of exponentials, and a second launch joins them.
//
// A warp owns 16 rows. Scores S = Q K^T come from mma.m16n8k16 with the query fragments held in
// registers (heads of 64; wider heads re-read them from the staged queries at every step, their
// registers hold the output instead) and key fragments read with ldmatrix from the staged tile; the accumulator layout of S
// is the A-fragment layout of the second product, so probabilities go from registers straight into
// P V, whose value fragments are ldmatrix.trans reads of the staged tile. Keys and values have a buffer each: the values of a
// tile arrive under its scores, the next keys under its P V. Bound by the multiplies (one per 8 cycles and
// scheduler) for wide heads, by the exponentials' instructions for heads of 64.
//
// Measured: 64 queries of 8 heads of 256 behind 0 to 2000 positions 110 us before (four warps, loads and multiplies in
// turn, a CTA per head), 22 with the join; 512 queries of 16 heads behind 4500 positions 500 us, 267; 512 queries
// of 32 heads of 64 from position 0 33 us, 27.

#include "async_utils.cuh"
#include "device_utils.cuh"
#include "kernels.h"

namespace bc {
namespace k {

namespace {

constexpr int kKeys = 64;      // keys per tile
// Rows per CTA, 16 to a warp. Heads of 64 take small CTAs, four to an SM (their registers allow it): more, finer work.
template <int HD>
constexpr int flash_rows() { return HD == 64 ? 64 : 128; }
template <int HD>
constexpr int flash_threads() { return 2 * flash_rows<HD>(); }
constexpr uint32_t kMaxSplits = 32;
// Halves per staged row: 16 bytes more than the head, so the 8 rows of an ldmatrix fall in distinct banks.
template <int HD>
constexpr int flash_pitch() { return HD + 8; }
template <int HD>
constexpr size_t flash_smem_bytes() { return (size_t)(2 * flash_rows<HD>() + 2 * kKeys) * flash_pitch<HD>() * 2; }

struct FlashParams {
    const float* q;
    const __half* k_cache;
    const __half* v_cache;
    float* out;
    uint32_t n_heads, n_kv_heads, first_pos, n_queries, q_stride, q_head_stride;
    uint32_t splits;
    float* parts;      // splits > 1: [split][query][head][HD] unnormalised sums, then [split][query][head] (maximum, sum)
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// (x, y) as half2 bits of the high parts, and of what the high parts left over.
__device__ __forceinline__ void split_half2(float x, float y, uint32_t& hi, uint32_t& lo) {
    __half2 h = __floats2half2_rn(x, y);
    float2 back = __half22float2(h);
    __half2 l = __floats2half2_rn(x - back.x, y - back.y);
    hi = *reinterpret_cast<uint32_t*>(&h);
    lo = *reinterpret_cast<uint32_t*>(&l);
}

template <int HD>
__global__ void __launch_bounds__(flash_threads<HD>(), HD == 64 ? 4 : 1) attention_flash_kernel(const __grid_constant__ FlashParams p) {
    constexpr int kRows = flash_rows<HD>(), kFlashThreads = flash_threads<HD>(), kHead = HD, kPitch = flash_pitch<HD>();
    constexpr bool kQueriesInRegisters = HD == 64;
    extern __shared__ __align__(16) uint8_t flash_smem[];
    __half (*q_hi)[kPitch] = reinterpret_cast<__half (*)[kPitch]>(flash_smem);
    __half (*q_lo)[kPitch] = q_hi + kRows;
    __half (*k_tile)[kPitch] = q_lo + kRows;
    __half (*v_tile)[kPitch] = k_tile + kKeys;
    __shared__ uint64_t row_at[kRows];

    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const uint32_t group = p.n_heads / p.n_kv_heads, n_rows = p.n_queries * group;
    const uint32_t row0 = (gridDim.x - 1 - blockIdx.x) * kRows, kv_head = blockIdx.y;  // the last queries see most keys: first
    const uint32_t kv_dim = p.n_kv_heads * kHead;
    const uint32_t kv_len = p.first_pos + p.n_queries;  // cache rows that exist
    const float scale = 1.0f / sqrtf((float)kHead);

    // Key tiles up to the position of the CTA's last query, and this CTA's part of them.
    const uint32_t last_query = (min(row0 + kRows, n_rows) - 1) / group;
    const uint32_t all_tiles = (p.first_pos + last_query) / kKeys + 1, per_split = (all_tiles + p.splits - 1) / p.splits;
    const uint32_t first_tile = blockIdx.z * per_split, end_tile = min(first_tile + per_split, all_tiles);

    const __half* kc = p.k_cache + (uint64_t)kv_head * kHead;
    const __half* vc = p.v_cache + (uint64_t)kv_head * kHead;
    // Rows past the cache's end repeat its last one: their scores are masked.
    auto bring = [&](const __half* from, __half (*to)[kPitch], uint32_t tile) {
#pragma unroll
        for (int n = 0; n < kKeys * (kHead / 8) / kFlashThreads; ++n) {
            const int i = tid + n * kFlashThreads, row = i / (kHead / 8), piece = i % (kHead / 8);
            const uint32_t key = min(tile * kKeys + row, kv_len - 1);
            async::cp_async_16((uint32_t)__cvta_generic_to_shared(&to[row][8 * piece]), from + (uint64_t)key * kv_dim + 8 * piece);
        }
        async::cp_async_commit();
    };
    if (first_tile < end_tile) bring(kc, k_tile, first_tile);

    // Stage the scaled queries as hi + lo halves; rows past the batch are zero. Where a row lies is worked out once per row (the
    // divisions, for every pair of elements, took 18 us of a CTA with 128 rows of 256).
    if (tid < kRows) {
        const uint32_t row = row0 + tid;
        row_at[tid] = row < n_rows ? (uint64_t)(row / group) * p.q_stride + (uint64_t)(kv_head * group + row % group) * p.q_head_stride : ~0ull;
    }
    __syncthreads();
    {
        constexpr int kPairs = kHead / 2, kRowStep = kFlashThreads / kPairs > 0 ? kFlashThreads / kPairs : 1, kAtOnce = 8;
        static_assert(kFlashThreads % kPairs == 0 && kRows % (kRowStep * kAtOnce) == 0, "whole rounds");
        const int pair = tid % kPairs;
        for (int first = tid / kPairs; first < kRows; first += kRowStep * kAtOnce) {
            float2 v[kAtOnce];
#pragma unroll
            for (int n = 0; n < kAtOnce; ++n) {
                const uint64_t at = row_at[first + n * kRowStep];
                v[n] = at != ~0ull ? *reinterpret_cast<const float2*>(p.q + at + 2 * pair) : make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int n = 0; n < kAtOnce; ++n) {
                uint32_t hi, lo;
                split_half2(v[n].x * scale, v[n].y * scale, hi, lo);
                *reinterpret_cast<uint32_t*>(&q_hi[first + n * kRowStep][2 * pair]) = hi;
                *reinterpret_cast<uint32_t*>(&q_lo[first + n * kRowStep][2 * pair]) = lo;
            }
        }
    }

    // Query fragments: k-steps of 16 elements, hi and lo.
    constexpr int kHeld = kQueriesInRegisters ? kHead / 16 : 1;
    uint32_t qa_hi[kHeld][4], qa_lo[kHeld][4];
    const int m = lane >> 3, r = lane & 7;
    auto query_fragments = [&](int ks, uint32_t (&hi)[4], uint32_t (&lo)[4]) {
        const int row = warp * 16 + (m & 1) * 8 + r, col = ks * 16 + (m >> 1) * 8;
        ldmatrix_x4(hi, (uint32_t)__cvta_generic_to_shared(&q_hi[row][col]));
        ldmatrix_x4(lo, (uint32_t)__cvta_generic_to_shared(&q_lo[row][col]));
    };
    if (kQueriesInRegisters) {
        __syncthreads();
#pragma unroll
        for (int ks = 0; ks < kHeld; ++ks) query_fragments(ks, qa_hi[ks], qa_lo[ks]);
    }

    float o[kHead / 8][4];
#pragma unroll
    for (int n = 0; n < kHead / 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[n][i] = 0.f;
    float row_max[2] = {-INFINITY, -INFINITY}, row_sum[2] = {0.f, 0.f};

    // This thread's two rows, g and g + 8 of the warp's 16, and their positions.
    const uint32_t row_a = row0 + warp * 16 + g, row_b = row_a + 8;
    const uint32_t pos_a = p.first_pos + row_a / group, pos_b = p.first_pos + row_b / group;
    // A warp whose queries all lie before a tile has nothing to add from it.
    const uint32_t warp_first_pos = p.first_pos + (row0 + warp * 16) / group, warp_last_pos = p.first_pos + (row0 + warp * 16 + 15) / group;

    for (uint32_t tile = first_tile; tile < end_tile; ++tile) {
        const uint32_t key0 = tile * kKeys;
        const bool skip = key0 > warp_last_pos;  // warp-uniform
        async::cp_async_wait<0>();
        __syncthreads();  // the keys are there, the previous values have been read
        bring(vc, v_tile, tile);

        // S = Q K^T: 8 tiles of 8 keys. Four accumulators take their hi products, then their lo ones: a product does not wait
        // for the one before it.
        float s[8][4];
        if (!skip) {
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) s[n][i] = 0.f;
#pragma unroll
            for (int ks = 0; ks < kHead / 16; ++ks) {
                if (!kQueriesInRegisters) query_fragments(ks, qa_hi[0], qa_lo[0]);
                const uint32_t (&a_hi)[4] = qa_hi[kQueriesInRegisters ? ks : 0];
                const uint32_t (&a_lo)[4] = qa_lo[kQueriesInRegisters ? ks : 0];
#pragma unroll
                for (int np = 0; np < 4; np += 2) {  // two pairs of key tiles
                    uint32_t b[2][4];
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        ldmatrix_x4(b[h], (uint32_t)__cvta_generic_to_shared(&k_tile[(np + h) * 16 + (m >> 1) * 8 + r][ks * 16 + (m & 1) * 8]));
#pragma unroll
                    for (int n = 0; n < 4; ++n) mma_f16(s[2 * np + n], a_hi, b[n >> 1][(n & 1) * 2], b[n >> 1][(n & 1) * 2 + 1]);
#pragma unroll
                    for (int n = 0; n < 4; ++n) mma_f16(s[2 * np + n], a_lo, b[n >> 1][(n & 1) * 2], b[n >> 1][(n & 1) * 2 + 1]);
                }
            }
            // Causal mask (only tiles that reach past a query's position need it).
            if (key0 + kKeys - 1 > warp_first_pos) {
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    const uint32_t key = key0 + n * 8 + 2 * t;
                    if (key > pos_a) s[n][0] = -INFINITY;
                    if (key + 1 > pos_a) s[n][1] = -INFINITY;
                    if (key > pos_b) s[n][2] = -INFINITY;
                    if (key + 1 > pos_b) s[n][3] = -INFINITY;
                }
            }
            // Online softmax. A row that has seen no key yet (a part of the keys may lie past it) keeps a maximum of
            // minus infinity and sums of zero.
            float tile_max[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                tile_max[0] = fmaxf(tile_max[0], fmaxf(s[n][0], s[n][1]));
                tile_max[1] = fmaxf(tile_max[1], fmaxf(s[n][2], s[n][3]));
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                tile_max[h] = fmaxf(tile_max[h], __shfl_xor_sync(0xffffffffu, tile_max[h], 1));
                tile_max[h] = fmaxf(tile_max[h], __shfl_xor_sync(0xffffffffu, tile_max[h], 2));
            }
            float correction[2], top[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float m_new = fmaxf(row_max[h], tile_max[h]);
                top[h] = m_new == -INFINITY ? 0.f : m_new;
                correction[h] = expf(row_max[h] - top[h]);  // exp(-inf) = 0 on the first keys
                row_max[h] = m_new;
            }
            float tile_sum[2] = {0.f, 0.f};
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                s[n][0] = expf(s[n][0] - top[0]);
                s[n][1] = expf(s[n][1] - top[0]);
                s[n][2] = expf(s[n][2] - top[1]);
                s[n][3] = expf(s[n][3] - top[1]);
                tile_sum[0] += s[n][0] + s[n][1];
                tile_sum[1] += s[n][2] + s[n][3];
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                tile_sum[h] += __shfl_xor_sync(0xffffffffu, tile_sum[h], 1);
                tile_sum[h] += __shfl_xor_sync(0xffffffffu, tile_sum[h], 2);
                row_sum[h] = row_sum[h] * correction[h] + tile_sum[h];
            }
#pragma unroll
            for (int n = 0; n < kHead / 8; ++n) {
                o[n][0] *= correction[0];
                o[n][1] *= correction[0];
                o[n][2] *= correction[1];
                o[n][3] *= correction[1];
            }
        }
        async::cp_async_wait<0>();
        __syncthreads();  // the values are there, the keys have been read
        if (tile + 1 < end_tile) bring(kc, k_tile, tile + 1);
        if (skip) continue;

        // O += P V: 4 k-steps of 16 keys; the scores' accumulator layout is the A-fragment layout.
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            uint32_t pa_hi[4], pa_lo[4];
            split_half2(s[2 * kk][0], s[2 * kk][1], pa_hi[0], pa_lo[0]);
            split_half2(s[2 * kk][2], s[2 * kk][3], pa_hi[1], pa_lo[1]);
            split_half2(s[2 * kk + 1][0], s[2 * kk + 1][1], pa_hi[2], pa_lo[2]);
            split_half2(s[2 * kk + 1][2], s[2 * kk + 1][3], pa_hi[3], pa_lo[3]);
#pragma unroll
            for (int np = 0; np < kHead / 16; np += 2) {  // two pairs of 8-element output tiles
                uint32_t b[2][4];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    ldmatrix_x4_trans(b[h], (uint32_t)__cvta_generic_to_shared(&v_tile[kk * 16 + (m & 1) * 8 + r][(np + h) * 16 + (m >> 1) * 8]));
#pragma unroll
                for (int n = 0; n < 4; ++n) mma_f16(o[2 * np + n], pa_hi, b[n >> 1][(n & 1) * 2], b[n >> 1][(n & 1) * 2 + 1]);
#pragma unroll
                for (int n = 0; n < 4; ++n) mma_f16(o[2 * np + n], pa_lo, b[n >> 1][(n & 1) * 2], b[n >> 1][(n & 1) * 2 + 1]);
            }
        }
    }
    async::cp_async_wait<0>();

    // Normalise and store: row g holds columns 2t, 2t + 1 of each 8-element tile. A part of the keys leaves its sums as they are.
    const bool whole = p.splits == 1;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t row = h ? row_b : row_a;
        if (row >= n_rows) continue;
        const uint64_t at = (uint64_t)(row / group) * p.n_heads + kv_head * group + row % group, total = (uint64_t)p.n_queries * p.n_heads;
        if (!whole) {
            if (t == 0)
                *reinterpret_cast<float2*>(p.parts + p.splits * total * kHead + (blockIdx.z * total + at) * 2) = make_float2(row_max[h], row_sum[h]);
            if (row_max[h] == -INFINITY) continue;  // joins with a weight of zero, unread
        }
        const float factor = whole ? 1.f / row_sum[h] : 1.f;
        float* out = (whole ? p.out + at * kHead : p.parts + (blockIdx.z * total + at) * kHead) + 2 * t;
#pragma unroll
        for (int n = 0; n < kHead / 8; ++n) *reinterpret_cast<float2*>(out + n * 8) = make_float2(o[n][2 * h] * factor, o[n][2 * h + 1] * factor);
    }
}

// Joins the parts of the keys, a warp per (query, head).
template <int HD>
__global__ void __launch_bounds__(256) attention_join_kernel(const float* __restrict__ parts, float* __restrict__ out, uint32_t splits, uint32_t total) {
    constexpr int kQuads = HD / 64;  // pairs of elements a lane holds
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31, at = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (at >= total) return;
    float2 ms = make_float2(-INFINITY, 0.f);
    if (lane < splits) ms = __ldcg(reinterpret_cast<const float2*>(parts + (uint64_t)splits * total * HD + ((uint64_t)lane * total + at) * 2));
    const float top = warp_max(ms.x), weight = ms.x == -INFINITY ? 0.f : expf(ms.x - top);
    const float inverse = 1.f / warp_sum(weight * ms.y);
    float2 sum[kQuads];
#pragma unroll
    for (int i = 0; i < kQuads; ++i) sum[i] = make_float2(0.f, 0.f);
    for (uint32_t z0 = 0; z0 < splits; z0 += 8) {
        float2 v[8][kQuads];
        float w[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            const uint32_t z = z0 + k;
            w[k] = z < splits ? __shfl_sync(0xffffffffu, weight, z & 31) : 0.f;
            const float2* from = reinterpret_cast<const float2*>(parts + ((uint64_t)z * total + at) * HD) + lane;
#pragma unroll
            for (int i = 0; i < kQuads; ++i) v[k][i] = w[k] != 0.f ? __ldcg(from + i * 32) : make_float2(0.f, 0.f);  // unwritten where it weighs nothing
        }
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k)
#pragma unroll
            for (int i = 0; i < kQuads; ++i) {
                sum[i].x += w[k] * v[k][i].x;
                sum[i].y += w[k] * v[k][i].y;
            }
    }
#pragma unroll
    for (int i = 0; i < kQuads; ++i) reinterpret_cast<float2*>(out + (uint64_t)at * HD)[lane + i * 32] = make_float2(sum[i].x * inverse, sum[i].y * inverse);
}

// Parts of the keys: the fewest modelled time. A tile takes 3.6 us (heads of 64, up to four CTAs to an SM) to 7.1 (heads of 256), a CTA 6 us around them, a
// part's sums are written and read once at L2 rates, the joining launch costs 4 us. The sums must fit the scratch the caller
// has (attention_scratch_floats), and a head's rows of (maximum, sum) a warp.
uint32_t choose_splits(const AttentionShape& s) {
    const uint32_t rows = s.head_dim == 64 ? flash_rows<64>() : flash_rows<256>(), units = (s.n_queries * (s.n_heads / s.n_kv_heads) + rows - 1) / rows * s.n_kv_heads;
    const uint32_t tiles = (s.first_pos + s.n_queries - 1) / kKeys + 1, slots = (uint32_t)sm_count() * (s.head_dim == 64 ? 4 : 1);
    const uint64_t floats = s.scratch_floats ? s.scratch_floats : attention_scratch_floats(s.n_heads, s.head_dim, s.n_ctx, s.n_queries);
    const uint64_t room = floats / ((uint64_t)s.n_queries * s.n_heads * (s.head_dim + 2));
    uint32_t most = tiles < kMaxSplits ? tiles : kMaxSplits, best = 1;
    if (room < most) most = room > 0 ? (uint32_t)room : 1;
    float least = 0.f;
    const float tile_us = 2.5f + s.head_dim * 0.018f, part_us = (float)s.n_queries * s.n_heads * s.head_dim * 8e-6f / 8.f;
    for (uint32_t splits = 1; splits <= most; ++splits) {
        const uint32_t waves = (units * splits + slots - 1) / slots, per = (tiles + splits - 1) / splits;
        const float us = waves * (per * tile_us + 6.f) + (splits > 1 ? 4.f + splits * part_us : 0.f);
        if (splits == 1 || us < least) {
            best = splits;
            least = us;
        }
    }
    return best;
}

// The parts are stored 8 bytes at a time.
uint32_t splits_for(const float* scratch, const AttentionShape& s) { return (uintptr_t)scratch % 8 == 0 ? choose_splits(s) : 1; }

template <int HD>
cudaError_t launch_flash(cudaStream_t stream, const FlashParams& p) {
    const uint32_t group = p.n_heads / p.n_kv_heads, total = p.n_queries * p.n_heads;
    cudaError_t e = ensure_dynamic_smem((const void*)attention_flash_kernel<HD>, flash_smem_bytes<HD>());
    if (e != cudaSuccess) return e;
    e = launch_dependent(attention_flash_kernel<HD>, dim3((p.n_queries * group + flash_rows<HD>() - 1) / flash_rows<HD>(), p.n_kv_heads, p.splits), dim3(flash_threads<HD>()),
                         flash_smem_bytes<HD>(), stream, p);
    if (e != cudaSuccess || p.splits == 1) return e;
    return launch_dependent(attention_join_kernel<HD>, dim3((total + 7) / 8), dim3(256), 0, stream, static_cast<const float*>(p.parts), p.out, p.splits, total);
}

}  // namespace

bool attention_flash_supported(bool kv_half, const AttentionShape& s) {
    return kv_half && (s.head_dim == 64 || s.head_dim == 128 || s.head_dim == 256) && s.n_queries >= 32 && s.pos_ptr == nullptr &&
           s.n_kv_heads > 0 && s.n_heads % s.n_kv_heads == 0 && s.q_stride % 2 == 0 && s.q_head_stride % 2 == 0;
}

int attention_flash_launches(const float* scratch, const AttentionShape& s) { return splits_for(scratch, s) > 1 ? 2 : 1; }

cudaError_t attention_flash(cudaStream_t stream, const float* q, const void* k_cache, const void* v_cache, float* scratch, float* out,
                            const AttentionShape& s) {
    const uint32_t splits = splits_for(scratch, s);
    const FlashParams p{q, static_cast<const __half*>(k_cache), static_cast<const __half*>(v_cache), out, s.n_heads, s.n_kv_heads,
                        s.first_pos, s.n_queries, s.q_stride, s.q_head_stride, splits, scratch};
    switch (s.head_dim) {
        case 64: return launch_flash<64>(stream, p);
        case 128: return launch_flash<128>(stream, p);
        default: return launch_flash<256>(stream, p);
    }
}

}  // namespace k
}  // namespace bc
