// The prefill contraction for more than a few tokens: Y[t][r] (store) sum_c W[r][c] X[t][c] on tcgen05
// from weights that were expanded to fp16 once, when the model was uploaded.
//
// Arithmetic: that of kernels_matmul_umma.cu, operand for operand. Weights are (q - 8) * d rounded to fp16
// once (dequant_word, at upload instead of on every launch), inputs are rounded to fp16, products
// accumulate in f32 (the reference's Q4_0 prefill kernel, crates/bobcat-metal/src/matmul.metal:249-470).
//
// Why expanded weights. The kernel that dequantises on the way into shared memory is bound by that
// conversion: its tensor cores wait for operands half of the time (2.6B shape, 512 tokens: 410 TFLOP/s). A
// weight takes 2 bytes here instead of 18/32, which a device with 180 GB has room for (4.9 GB at 2.6B), and
// reading them costs 0.75 ms per pass at the HBM rate, less than the multiply of 100 tokens and more. When
// the expanded copy does not fit the device, Mat::half_tiles is null and the dequantising kernel serves.
//
// Shape. Persistent CTAs of ten warps, one per SM: a loader thread, an MMA thread, eight epilogue warps.
// A tile is 128 weight rows x up to 256 tokens (of a SwiGLU 64 rows of either matrix, or 128 of both x up to 128 tokens).
// K advances 64 columns per stage through a ring of 192 KB, four to eight stages; both operands
// arrive by bulk copies of contiguous memory (the weight tile is stored as the 16 KB image the MMA reads,
// the tokens come packed, kernels_matmul_umma.cu's pack kernels), so no thread touches an operand. Tensor
// memory holds two accumulators of 256 columns: a tile's epilogue runs under the next tile's main
// loop. Measured apart on this device: one tcgen05.mma M128 N256 K16 per 128 cycles (2.19 PFLOP/s), full rate
// down to N = 128, with or without swizzle; bulk copies out of L2 above 15 TB/s.
//
// Matrices with few tiles split K; the partial products go to scratch and are added in index order by
// the next normalisation or by reduce_kernel. Every wait is bounded, as in kernels_matmul_umma.cu.

#include <cstdlib>

#include "async_utils.cuh"
#include "device_utils.cuh"
#include "kernels.h"
#include "../../include/bobcat_cuda.h"

namespace bc {
namespace k {

namespace {

using namespace async;

constexpr uint32_t kRows = 128, kChunkK = 64, kCores = kChunkK / 8;
constexpr uint32_t kATile = kRows * kChunkK * 2;       // 16 KB: [8-row group][core along K][row][16 bytes]
constexpr uint32_t kGroupBytes = 8 * kChunkK * 2, kCoreBytes = 128;
constexpr uint32_t kMaxStages = 8, kRingBytes = 192 * 1024;  // a stage: a tile's weights and its tokens
constexpr uint32_t kEpilogueWarps = 8, kThreads = (2 + kEpilogueWarps) * 32;
constexpr uint32_t kTmemColumns = 512, kAccColumns = 256;
constexpr uint32_t kSpinLimit = 1u << 22;
constexpr uint32_t kTurnBytes = 640;                   // per epilogue warp: a 32 x 8 block turned into operand layout
constexpr uint32_t kSwapBytes = 2 * 2 * 8 * 32 * 4;    // per pair of epilogue warps: 8 columns of 32 rows each way, twice
constexpr size_t kSmemBytes = kRingBytes + kEpilogueWarps * kTurnBytes + kEpilogueWarps / 2 * kSwapBytes + 1024;
constexpr uint32_t kMaxSplit = 8;

__device__ int* g_wait_word;  // where a wait that ran out leaves its code (kernels.h), null until set

// What a tile of 128 accumulator rows is: rows of one matrix; 128 rows of both matrices of a SwiGLU (two accumulators, up to
// 128 tokens); or 64 rows of either (one accumulator, up to 256 tokens: more, finer tiles from the same bytes).
enum Kind { kPlain = 1, kWhole = 2, kHalves = 3 };
constexpr uint32_t a_bytes(int kind) { return kind == kWhole ? 2 * kATile : kATile; }

struct HalfParams {
    // Up to four matrices that read the same inputs: row tiles [first_tile[i], first_tile[i + 1]) are
    // matrix i's. Dual: tiles[0] = gate, tiles[1] = up, one matrix of outputs.
    const __half* tiles[4];
    float* y[4];
    uint32_t first_tile[5], rows[4], stride[4];
    int n_matrices;
    const __half* packed;      // [n_chunks][token_groups][8 cores][8 tokens][8 halves]
    uint32_t n_chunks, n_tokens, token_groups;
    uint32_t stages, stage_bytes;
    uint32_t tile_tokens, token_tiles, split, n_tiles;  // n_tiles = row tiles x split x token tiles
    int store;
    __half* packed_out;        // dual: the result as the packed operand of the product that consumes it
};

struct Tile {
    uint32_t row_tile, part, tok0, n;      // n: the MMA's N, a multiple of 16
    uint32_t chunk0, chunks;
};

__device__ __forceinline__ Tile tile_at(const HalfParams& p, uint32_t i) {
    Tile t;
    const uint32_t token_tile = i % p.token_tiles, rest = i / p.token_tiles;
    t.part = rest % p.split;
    t.row_tile = rest / p.split;
    t.tok0 = token_tile * p.tile_tokens;
    const uint32_t left = p.n_tokens - t.tok0;
    t.n = left >= p.tile_tokens ? p.tile_tokens : (left + 15u) & ~15u;
    const uint32_t per = (p.n_chunks + p.split - 1) / p.split;
    t.chunk0 = min(t.part * per, p.n_chunks);
    t.chunks = min(per, p.n_chunks - t.chunk0);
    return t;
}

__device__ __forceinline__ void give_up(volatile int* dead, int code) {
    *dead = 1;
    if (g_wait_word) *reinterpret_cast<volatile int*>(g_wait_word) = code;
}

// The epilogue of a plain product: a warp's 32 rows, every other unit of 16 tokens, two units in flight. Bound by
// instructions while it asked for every value what to do with it: 8 us for 128 rows x 256 tokens, which nothing
// hides when a CTA has one tile; 512 tokens of 6144 x 2048 19.0 us with it, 14.1 now (with the MMA warp's change).
__device__ __forceinline__ void store_tile(uint32_t from, uint32_t half, uint32_t units, const Tile& t, float* out, uint32_t stride, uint32_t out_row,
                                           uint32_t rows, uint32_t n_tokens, int store) {
    const bool stores = out_row < rows;
    auto put = [&](uint32_t u, float (&v)[16]) {
        const uint32_t tok = t.tok0 + u * 16;
        if (!stores || tok >= n_tokens) return;
        if (t.chunks == 0) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = 0.f;
        }
        const uint32_t live = n_tokens - tok;
        float* to = out + (uint64_t)tok * stride + out_row;
        if (store == BC_STORE_OVERWRITE && live >= 16) {
#pragma unroll
            for (int j = 0; j < 16; ++j, to += stride) *to = v[j];
            return;
        }
        if (store == BC_STORE_OVERWRITE) {
#pragma unroll
            for (int j = 0; j < 16; ++j, to += stride)
                if ((uint32_t)j < live) *to = v[j];
            return;
        }
        float old[16];
        float* at = to;
#pragma unroll
        for (int j = 0; j < 16; ++j, at += stride) old[j] = (uint32_t)j < live ? __ldcg(at) : 0.f;
        if (store == BC_STORE_ACCUMULATE) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] += old[j];
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = old[j] / (1.f + expf(-old[j])) * v[j];
        }
#pragma unroll
        for (int j = 0; j < 16; ++j, to += stride)
            if ((uint32_t)j < live) *to = v[j];
    };
    for (uint32_t u = half; u < units; u += 4) {
        float v[16], w[16];
        const bool second = u + 2 < units;  // the same for the whole warp
        __syncwarp();
        tmem_load_16_start(from + u * 16, v);
        if (second) tmem_load_16_start(from + (u + 2) * 16, w);
        tmem_load_wait(v, w);
        put(u, v);
        if (second) put(u + 2, w);
    }
}

// A warp's 32 rows x 8 tokens as fp16 operand of the consuming product, of which the rows are a block of 32 columns and the tokens a
// group. The values turn through shared memory into 16-byte core-matrix rows (9 rows of 16 bytes per core matrix
// keep both sides free of bank conflicts); a lane stores one, 8 lanes to a 128-byte line.
__device__ __forceinline__ void put_group(const float* v, uint8_t* turn_bytes, const HalfParams& p, uint32_t row0, uint32_t block, uint32_t tok, uint32_t lane) {
    __half* turn = reinterpret_cast<__half*>(turn_bytes);
    const uint32_t core = (lane & 15) >> 2, e = lane & 3;
    const uint32_t at = (lane >> 4) * 4 + (e & 1) * 2 + (e >> 1);
#pragma unroll
    for (int j = 0; j < 8; ++j) turn[(core * 9 + j) * 8 + at] = __float2half_rn(v[j]);
    __syncwarp();
    const uint32_t tr = lane & 7, mm = lane >> 3;
    const uint4 row16 = *reinterpret_cast<const uint4*>(turn + (mm * 9 + tr) * 8);
    const uint32_t chunk = (row0 >> 6) + (block >> 1), jj = (block & 1) * 4 + mm;
    reinterpret_cast<uint4*>(p.packed_out)[(((uint64_t)chunk * p.token_groups + (tok >> 3)) * kCores + jj) * 8 + tr] = row16;
}

template <int KIND>
__global__ void __launch_bounds__(kThreads, 1) matmul_half_kernel(const __grid_constant__ HalfParams p) {
    constexpr bool kDual = KIND != kPlain;
    constexpr uint32_t kABytes = a_bytes(KIND);
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* turns = smem + kRingBytes;
    const uint32_t n_stages = p.stages, stage_bytes = p.stage_bytes;
    __shared__ __align__(8) uint64_t bars[2 * kMaxStages + 4];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int dead_flag;
    volatile int* dead = &dead_flag;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + kMaxStages * 8, acc_full0 = empty0 + kMaxStages * 8, acc_empty0 = acc_full0 + 16;
    const uint32_t ring = smem_u32(smem);
    // The next launch may set itself up; it waits for this one before it touches its outputs.
    pdl_launch_dependents();
    if (tid == 0) {
        for (uint32_t s = 0; s < n_stages; ++s) {
            mbar_init(full0 + 8 * s, 1);   // the loader's arrive.expect_tx
            mbar_init(empty0 + 8 * s, 1);  // the MMA thread's commit
        }
        for (uint32_t a = 0; a < 2; ++a) {
            mbar_init(acc_full0 + 8 * a, 1);
            mbar_init(acc_empty0 + 8 * a, kEpilogueWarps);
        }
        dead_flag = 0;
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), kTmemColumns);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        // ---- loader. The weights are nobody's output: the first tile's weight copies go out before the
        // wait for the preceding launch, the tokens' follow it.
        if (lane == 0) {
            uint32_t stage = 0, phase = 1;
            bool waited = false;
            for (uint32_t i = blockIdx.x; i < p.n_tiles; i += gridDim.x) {
                const Tile t = tile_at(p, i);
                int m = 0;
                if (!kDual)
                    while (m + 1 < p.n_matrices && t.row_tile >= p.first_tile[m + 1]) ++m;
                const uint64_t at = KIND == kHalves ? ((uint64_t)(t.row_tile / 2) * p.n_chunks * 2 + (t.row_tile & 1)) * (kATile / 4)  // half of a 128-row tile
                                                    : ((uint64_t)(t.row_tile - (kDual ? 0 : p.first_tile[m])) * p.n_chunks + t.chunk0) * (kATile / 2);
                const __half* a = p.tiles[m] + at;
                const __half* a2 = kDual ? p.tiles[1] + at : nullptr;
                const __half* b = p.packed + ((uint64_t)t.chunk0 * p.token_groups + t.tok0 / 8) * (8 * kChunkK);
                const uint32_t b_bytes = t.n * kChunkK * 2;
                auto weights = [&](uint32_t c, uint32_t s) {
                    constexpr uint32_t kEach = kDual ? kABytes / 2 : kABytes;
                    mbar_arrive_expect(full0 + 8 * s, kABytes + b_bytes);
                    bulk_load(ring + s * stage_bytes, a + (uint64_t)c * (kATile / 2), kEach, full0 + 8 * s);
                    if (kDual) bulk_load(ring + s * stage_bytes + kEach, a2 + (uint64_t)c * (kATile / 2), kEach, full0 + 8 * s);
                };
                auto tokens = [&](uint32_t c, uint32_t s) {
                    bulk_load(ring + s * stage_bytes + kABytes, b + (uint64_t)c * p.token_groups * (8 * kChunkK), b_bytes, full0 + 8 * s);
                };
                uint32_t c = 0;
                if (!waited) {
                    const uint32_t first = t.chunks < n_stages ? t.chunks : n_stages;  // free stages: nothing to wait for
                    for (; c < first; ++c) weights(c, c);
                    pdl_wait();
                    waited = true;
                    for (uint32_t s = 0; s < first; ++s) tokens(s, s);
                    stage = first % n_stages;
                    phase = first == n_stages ? 0 : 1;
                }
                for (; c < t.chunks; ++c) {
                    if (!mbar_wait(empty0 + 8 * stage, phase, kSpinLimit, dead)) {
                        give_up(dead, 3);
                        break;
                    }
                    weights(c, stage);
                    tokens(c, stage);
                    if (++stage == n_stages) stage = 0, phase ^= 1;
                }
                if (*dead) break;
            }
        }
    } else if (warp == 1) {
        // ---- the tensor core. The whole warp walks the chunks and one lane issues: values the warp shares stay in uniform
        // registers, where the instruction wants its descriptors (a loop inside one lane moved them there for every
        // multiply: 510 cycles per chunk whatever its width, the multiplies of 256 tokens).
        uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 1;
        const uint64_t desc0 = umma_desc(ring, kCoreBytes, kGroupBytes);
        bool alive = true;
        for (uint32_t i = blockIdx.x; i < p.n_tiles && alive; i += gridDim.x) {
            const Tile t = tile_at(p, i);
            const uint32_t idesc = umma_idesc_f16(kRows, t.n);
            if (!__all_sync(0xffffffffu, mbar_wait(acc_empty0 + 8 * acc, acc_phase, kSpinLimit, dead))) {
                if (lane == 0) give_up(dead, 1);
                break;
            }
            tc_fence_after_sync();
            for (uint32_t c = 0; c < t.chunks; ++c) {
                if (!__all_sync(0xffffffffu, mbar_wait(full0 + 8 * stage, phase, kSpinLimit, dead))) {
                    if (lane == 0) give_up(dead, 4);
                    alive = false;
                    break;
                }
                tc_fence_after_sync();
                const uint64_t a_desc = desc0 + ((stage * stage_bytes) >> 4), b_desc = a_desc + (kABytes >> 4);
                if (elect_one()) {
#pragma unroll
                    for (uint32_t m = 0; m < (KIND == kWhole ? 2u : 1u); ++m)
#pragma unroll
                        for (uint32_t j = 0; j < kChunkK / 16; ++j)
                            umma_f16(tmem + acc * kAccColumns + m * (kAccColumns / 2), a_desc + ((m * kATile + j * 2 * kCoreBytes) >> 4),
                                     b_desc + ((j * 2 * kCoreBytes) >> 4), idesc, (c | j) != 0);
                    umma_commit(empty0 + 8 * stage);
                }
                if (++stage == n_stages) stage = 0, phase ^= 1;
            }
            if (alive && elect_one()) umma_commit(acc_full0 + 8 * acc);
            if (++acc == 2) acc = 0, acc_phase ^= 1;
        }
    } else {
        // ---- epilogue: a warp reads lanes 32 * (warp % 4).. of tensor memory and every other 16 columns
        const uint32_t ew = warp - 2, quarter = warp & 3, half = ew >> 2;
        uint32_t acc = 0, acc_phase = 0;
        pdl_wait();  // y, the partial products and the packed output are other launches' to read or write until now
        for (uint32_t i = blockIdx.x; i < p.n_tiles; i += gridDim.x) {
            const Tile t = tile_at(p, i);
            int m = 0;
            if (!kDual)
                while (m + 1 < p.n_matrices && t.row_tile >= p.first_tile[m + 1]) ++m;
            const uint32_t rows = p.rows[m], stride = p.stride[m];
            const uint32_t row0 = KIND == kHalves ? t.row_tile * (kRows / 2) : (t.row_tile - (kDual ? 0 : p.first_tile[m])) * kRows;
            const uint32_t block = KIND == kHalves ? quarter & 1 : quarter, out_row = row0 + block * 32 + lane;  // the warp's 32 rows of the tile
            float* out = p.y[m] + (p.split > 1 ? (uint64_t)t.part * p.n_tokens * stride : 0);
            const bool ok = lane != 0 || mbar_wait(acc_full0 + 8 * acc, acc_phase, kSpinLimit, dead);
            // A wait that ran out voids the results; the warp walks on (further waits end at once), because others meet it below.
            if (!__all_sync(0xffffffffu, ok) && lane == 0) give_up(dead, 2);
            tc_fence_after_sync();
            const uint32_t from = tmem + ((quarter * 32) << 16) + acc * kAccColumns, units = t.n / 16;
            if (KIND == kPlain) {
                store_tile(from, half, units, t, out, stride, out_row, rows, p.n_tokens, p.store);
            } else if (KIND == kWhole) {
                for (uint32_t u = half; u < units; u += 2) {
                    float v[16], up[16];
                    __syncwarp();
                    tmem_load_16_start(from + u * 16, v);
                    tmem_load_16_start(from + kAccColumns / 2 + u * 16, up);
                    tmem_load_wait(v, up);
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = v[j] / (1.f + expf(-v[j])) * up[j];
                    const uint32_t tok = t.tok0 + u * 16;
                    if (p.packed_out) {
                        if (row0 + block * 32 < rows) {
                            put_group(v, turns + ew * kTurnBytes, p, row0, block, tok, lane);
                            __syncwarp();
                            put_group(v + 8, turns + ew * kTurnBytes, p, row0, block, tok + 8, lane);
                        }
                    } else if (out_row < rows) {
                        float* to = out + (uint64_t)tok * stride + out_row;
#pragma unroll
                        for (int j = 0; j < 16; ++j, to += stride)
                            if (tok + j < p.n_tokens) *to = v[j];
                    }
                }
            } else {
                // Lanes 0 to 63 of the accumulator are rows of gate, the other 64 the same rows of up. Of 16 tokens the warp
                // that reads the gates takes the first 8 and the warp that reads the same rows of up the others; they
                // swap what the other one needs. Two buffers in turn: whoever is at the next barrier has read this one.
                const bool has_gate = quarter < 2;
                const uint32_t pair = half * 2 + (quarter & 1);
                float* swap = reinterpret_cast<float*>(turns + kEpilogueWarps * kTurnBytes + pair * kSwapBytes);
                for (uint32_t u = half; u < units; u += 2) {
                    float v[16];
                    __syncwarp();
                    tmem_load_16(from + u * 16, v);
                    float* buffer = swap + ((u >> 1) & 1) * (2 * 8 * 32);
                    float mine[8], other[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        mine[j] = has_gate ? v[j] : v[8 + j];
                        buffer[(has_gate ? 8 + j : j) * 32 + lane] = has_gate ? v[8 + j] : v[j];
                    }
                    asm volatile("bar.sync %0, 64;" ::"r"(1 + pair) : "memory");
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        other[j] = buffer[(has_gate ? j : 8 + j) * 32 + lane];
                        const float g = has_gate ? mine[j] : other[j], up = has_gate ? other[j] : mine[j];
                        mine[j] = g / (1.f + expf(-g)) * up;
                    }
                    const uint32_t tok = t.tok0 + u * 16 + (has_gate ? 0 : 8);
                    if (p.packed_out) {
                        if (row0 + block * 32 < rows) put_group(mine, turns + ew * kTurnBytes, p, row0, block, tok, lane);
                    } else if (out_row < rows) {
                        float* to = out + (uint64_t)tok * stride + out_row;
#pragma unroll
                        for (int j = 0; j < 8; ++j, to += stride)
                            if (tok + j < p.n_tokens) *to = mine[j];
                    }
                }
            }
            // The accumulator is read: the MMA thread may overwrite it.
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty0 + 8 * acc);
            if (++acc == 2) acc = 0, acc_phase ^= 1;
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (*dead) __nanosleep(100000);  // let copies and instructions still in flight land before the CTA goes
    if (warp == 1) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem, kTmemColumns);
    }
}

// Split layout -> expanded operand tiles: one thread per 16 bytes (eight weights of one row).
__global__ void expand_tiles_kernel(const uint4* __restrict__ quants, const __half* __restrict__ scales, uint32_t n_rows, uint32_t n_blocks,
                                    uint4* __restrict__ tiles, uint64_t total) {
    const uint64_t o = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= total) return;
    const uint32_t in_tile = o % (kATile / 16), row_in_group = in_tile & 7, core = (in_tile >> 3) & (kCores - 1), group = in_tile >> 6;
    const uint64_t tile = o / (kATile / 16);
    const uint32_t n_chunks = n_blocks / 2, chunk = tile % n_chunks, row = (uint32_t)(tile / n_chunks) * kRows + group * 8 + row_in_group;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (row < n_rows) {
        const uint64_t block = (uint64_t)row * n_blocks + chunk * 2 + (core >> 2);
        const uint4 q = quants[block];
        const uint32_t w = (core & 3) == 0 ? q.x : (core & 3) == 1 ? q.y : (core & 3) == 2 ? q.z : q.w;
        v = dequant_word(w, __half2half2(scales[block]));
    }
    tiles[o] = v;
}

struct Tiling {
    uint32_t tile_tokens, split;
    int kind;
};

// The tiling with the smallest modelled time, in us, fitted to 16 to 512 tokens of matrices of 2048 to 10752 rows and columns:
// waves of tiles over the SMs, each chunk of 64 columns bound by the MMA (2 cycles per token and matrix at 1.4 GHz),
// by the SM's share of L2 or by the ring's round trip; a start and a last epilogue that nothing hides; a split's partial
// products, written and read once; the weights' time from HBM, of which a quarter shows beside the rest. Against the quickest of all tilings, matrices of the
// 350M shape, which the fit left out, us with the packing and sums' launches for 33, 128 and 512 tokens: 1024 x 4608 10.2, 10.9, 16.3 (quickest 10.0,
// 10.9, 16.1); gate and up 4608 x 1024 11.3, 11.3, 18.1 (11.1, 11.3, 17.5); 3072 x 1024 14.3, 14.5, 10.6 (11.6, 8.4, 10.6: K in one part, without the
// sums' launch, which the model takes for cheaper than it is there).
Tiling choose_tiling(uint32_t rows, uint32_t n_chunks, uint32_t n_tokens, bool dual, bool may_split) {
    const uint32_t sms = (uint32_t)sm_count();
    Tiling best{};
    double best_us = 1e30;
    for (int kind = dual ? kWhole : kPlain; kind <= (dual ? kHalves : kPlain); ++kind) {
        const uint32_t row_tiles = kind == kHalves ? (rows + kRows / 2 - 1) / (kRows / 2) : (rows + kRows - 1) / kRows;
        const uint32_t widest = kind == kWhole ? 128 : 256, fewest = (n_tokens + widest - 1) / widest;
        for (uint32_t token_tiles = fewest; token_tiles <= fewest + 6; ++token_tiles) {
            const uint32_t width = ((n_tokens + token_tiles - 1) / token_tiles + 15u) & ~15u;
            if (width < 48 && token_tiles > fewest) break;
            const uint32_t needed = (n_tokens + width - 1) / width;
            const double mma = 2.0 * width * (kind == kWhole ? 2 : 1) / 1400.0, load = (a_bytes(kind) + 128.0 * width) / (kind == kPlain ? 125e3 : kind == kHalves ? 115e3 : 105e3);
            const double trip = kind == kHalves ? 0.285 : 0.25, bound = mma > load ? mma : load, chunk = bound > trip ? bound : trip;
            for (uint32_t split = 1; split <= (may_split && !dual ? kMaxSplit : 1u); ++split) {
                if (split > 1 && n_chunks / split < 4) break;
                const uint32_t tiles = row_tiles * needed * split, waves = (tiles + sms - 1) / sms;
                double us = waves * ((n_chunks + split - 1) / split) * chunk;
                const double hbm = (double)row_tiles * n_chunks * a_bytes(kind) / 6.2e6;
                us = (us > hbm ? us + 0.25 * hbm : hbm + 0.25 * us) + 2.8 + 0.0095 * width * (dual ? 2 : 1) + (kind == kWhole ? 2.0 : 0.0);
                if (split > 1) us += 1.0 + 0.15 * split + (double)split * n_tokens * rows * 4 / 8e6;
                if (us < best_us) best_us = us, best = Tiling{width, split, kind};
            }
        }
    }
    return best;
}

bool half_disabled() {
    static const bool off = [] {
        const char* v = std::getenv("BOBCAT_NO_HALF_MATMUL");
        return v && v[0] == '1';
    }();
    return off;
}

template <int KIND>
cudaError_t launch_kind(cudaStream_t stream, HalfParams& p) {
    p.stage_bytes = a_bytes(KIND) + p.tile_tokens * kChunkK * 2;
    p.stages = kRingBytes / p.stage_bytes < kMaxStages ? kRingBytes / p.stage_bytes : kMaxStages;
    const void* kernel = (const void*)matmul_half_kernel<KIND>;
    cudaError_t e = ensure_dynamic_smem(kernel, kSmemBytes);
    if (e != cudaSuccess) return e;
    const uint32_t sms = (uint32_t)sm_count();
    void* args[] = {&p};
    return launch_kernel(kernel, dim3(p.n_tiles < sms ? p.n_tiles : sms), dim3(kThreads), kSmemBytes, stream, args);
}

cudaError_t launch_half(cudaStream_t stream, HalfParams& p, Tiling tiling) {
    p.tile_tokens = tiling.tile_tokens;
    p.token_tiles = (p.n_tokens + tiling.tile_tokens - 1) / tiling.tile_tokens;
    p.split = tiling.split;
    p.n_tiles = p.first_tile[p.n_matrices] * p.split * p.token_tiles;
    if (p.n_tiles == 0) return cudaSuccess;
    switch (tiling.kind) {
        case kPlain: return launch_kind<kPlain>(stream, p);
        case kWhole: return launch_kind<kWhole>(stream, p);
        default: return launch_kind<kHalves>(stream, p);
    }
}

uint32_t row_tiles_of(const Mat& w) { return (w.n_rows + kRows - 1) / kRows; }

void common(HalfParams& p, const Mat& w, const void* packed, uint32_t n_tokens, int store) {
    p.packed = static_cast<const __half*>(packed);
    p.n_chunks = w.n_cols / kChunkK;
    p.n_tokens = n_tokens;
    p.token_groups = ((n_tokens + 15u) & ~15u) / 8;
    p.store = store;
}

}  // namespace

cudaError_t matmul_half_wait_word(int* word) { return cudaMemcpyToSymbol(g_wait_word, &word, sizeof word); }

uint64_t half_tiles_bytes(uint32_t n_rows, uint32_t n_cols) { return (uint64_t)((n_rows + kRows - 1) / kRows) * (n_cols / kChunkK) * kATile; }

bool half_tiles_supported(uint32_t n_cols) { return !half_disabled() && n_cols % kChunkK == 0 && n_cols > 0; }

bool half_tiles_fit(uint64_t bytes) {
    size_t free_bytes = 0, total_bytes = 0;
    return cudaMemGetInfo(&free_bytes, &total_bytes) == cudaSuccess && bytes <= free_bytes / 2;
}

cudaError_t expand_half_tiles(cudaStream_t stream, const void* quants, const __half* scales, uint32_t n_rows, uint32_t n_cols, void* tiles) {
    const uint64_t total = half_tiles_bytes(n_rows, n_cols) / 16;
    if (total == 0) return cudaSuccess;
    expand_tiles_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(static_cast<const uint4*>(quants), scales, n_rows, n_cols / 32,
                                                                          static_cast<uint4*>(tiles), total);
    return cudaGetLastError();
}

bool matmul_half_supported(const Mat& w, uint32_t n_tokens) { return w.half_tiles != nullptr && n_tokens >= kMinHalfTokens && !half_disabled(); }

uint32_t matmul_half_split(const Mat& w, uint32_t n_tokens) {
    return choose_tiling(w.n_rows, w.n_cols / kChunkK, n_tokens, false, w.n_rows % 4 == 0).split;
}

cudaError_t matmul_half(cudaStream_t stream, const Mat* const* ws, float* const* ys, int n, const void* packed, uint32_t n_tokens, uint32_t y_stride,
                        int32_t store, uint32_t split) {
    if (n < 1 || n > 4) return cudaErrorInvalidValue;
    HalfParams p{};
    common(p, *ws[0], packed, n_tokens, store);
    p.n_matrices = n;
    for (int i = 0; i < n; ++i) {
        if (ws[i]->n_cols != ws[0]->n_cols || !ws[i]->half_tiles) return cudaErrorInvalidValue;
        p.tiles[i] = static_cast<const __half*>(ws[i]->half_tiles);
        p.y[i] = ys[i];
        p.rows[i] = ws[i]->n_rows;
        p.stride[i] = n == 1 ? y_stride : ws[i]->n_rows;
        p.first_tile[i + 1] = p.first_tile[i] + row_tiles_of(*ws[i]);
    }
    Tiling tiling = choose_tiling(n == 1 ? ws[0]->n_rows : p.first_tile[n] * kRows, p.n_chunks, n_tokens, false, split > 1);
    if (split > 1 && tiling.split != split) return cudaErrorInvalidValue;  // the caller sized the partial products by matmul_half_split
    return launch_half(stream, p, tiling);
}

bool matmul_half_swiglu_whole(const Mat& gate, uint32_t n_tokens) {
    return choose_tiling(gate.n_rows, gate.n_cols / kChunkK, n_tokens, true, false).kind == kWhole;
}

cudaError_t matmul_half_swiglu(cudaStream_t stream, const Mat& gate, const Mat& up, const void* packed, float* y, uint32_t n_tokens, uint32_t y_stride,
                               void* packed_out) {
    if (gate.n_rows != up.n_rows || gate.n_cols != up.n_cols || !gate.half_tiles || !up.half_tiles || (packed_out && gate.n_rows % kChunkK != 0))
        return cudaErrorInvalidValue;
    HalfParams p{};
    common(p, gate, packed, n_tokens, BC_STORE_OVERWRITE);
    p.n_matrices = 1;
    p.tiles[0] = static_cast<const __half*>(gate.half_tiles);
    p.tiles[1] = static_cast<const __half*>(up.half_tiles);
    p.y[0] = y;
    p.rows[0] = gate.n_rows;
    p.stride[0] = y_stride;
    const Tiling tiling = choose_tiling(gate.n_rows, p.n_chunks, n_tokens, true, false);
    p.first_tile[1] = tiling.kind == kHalves ? (gate.n_rows + kRows / 2 - 1) / (kRows / 2) : row_tiles_of(gate);
    p.packed_out = static_cast<__half*>(packed_out);
    return launch_half(stream, p, tiling);
}

}  // namespace k
}  // namespace bc
