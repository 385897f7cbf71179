// Products of a batch over Q4_0 experts of a few rows each (mixture-of-experts prefill): tcgen05 with the weights as an
// operand in tensor memory.
//
// Arithmetic: that of the other half-precision products (kernels_matmul_umma.cu): weights (q - 8) * d rounded to
// fp16 once, inputs rounded to fp16, products accumulated in f32 (crates/bobcat-metal/src/matmul.metal:473-506).
//
// Sums. An instruction cuts its sum off instead of rounding it, so what one accumulator loses grows with its K: against float64 of the same
// rounded operands (2-norm), 1.1e-7 for 64 columns, 1.8e-7 for 128, 6.4e-7 for 512, 2.1e-6 for 1792. Up to 64 rows an expert on the average, tensor
// memory therefore sums 128 columns (of up to 1024 columns, 64), and the storing warps add the parts up in registers, rounding: 2.0e-7 for 1792 and more (stretches
// of 2048 columns are added up by themselves), what sums on mma.sync over 16 warps have. Experts of more rows sum all of K in tensor memory, as
// matmul_umma_kernel does.
//
// What bounds it. Every expert's weights are read and unpacked once for a few dozen rows, so unpacking is the work: a stage (128 rows x
// 256 columns) is 32 pairs of blocks, each 104 packed-half and logic instructions of a warp, which issue every second cycle: 512 cycles on four
// schedulers. On mma.sync (matmul_few_kernel) the multiplies took the same issue slots (8 cycles each, 32 rows in four groups),
// and every 16-row tile's sums met over 16 warps: 1.9 us per tile of 2048 columns, 0.8 of them multiplies. Here one instruction multiplies
// 128 rows by all of an expert's. The unpacked
// weights go to tensor memory, not to shared memory, whose 128 bytes per cycle writing and reading them back (1024 cycles a stage) would
// take instead: tcgen05.st 16x128b takes the registers as they are unpacked, because the decode tiles
// are in mma fragment order (lane (g, t): rows g and g + 8, word t of a block), so a row's columns lie in the order (pair of halves j,
// word t); the rows' operand is packed in the same order. What a stage takes beyond that is the hand-over between warps:
// with stages of 64 columns (and one accumulator) gate and up of the block below took 82 us, of 128 67, of 256 52.
//
// Shape. Persistent CTAs, one per SM, equal runs of the jobs (128 weight rows, of a SwiGLU 64 of either matrix) of all experts' groups of
// up to `tile_tokens` rows. 16 unpacking warps: a warp owns 16 of the tile's rows (its lanes of tensor memory) in every other stage.
// One warp brings the weights' bytes (a lane per tile, eight pairs of blocks at a time), one the rows' operand, one issues the
// multiplies, eight (two a quarter of the lanes, half of the rows each) sum and store, from one of two sets of accumulators while the other fills. A set is
// two parts, a stage's: handed over one by one, with the wait for a free accumulator behind the stage's, parts cost 24 us more than the 9 they cost. Eight warps, since
// four would need 64 registers a thread for the sums and 27 warps leave 72. Every wait is bounded.
//
// Measured with the packing of the rows, 4 of 32 experts, gate and up 1792 x 2048 and down 2048 x 1792, us: 203 tokens 68.6 and 39.2 (one accumulator 60.0 and
// 37.5, matmul_few_kernel 102 and 65.5; HBM time 20 and 10); 16 tokens 55.9 and 35.9 (46.6 and 29.7; 57.0 and 35.3); 512 tokens 101 and 57.6 (81.8
// and 47.6 with groups of 128 rows, whose sums do not fit the registers; 220 and 137).

#include "async_utils.cuh"
#include "device_utils.cuh"
#include "kernels.h"
#include "../../include/bobcat_cuda.h"

namespace bc {
namespace k {

namespace {

using namespace async;

constexpr uint32_t kMaxStages = 3, kStageColumns = 128, kStagePairs = 4;  // columns of tensor memory: 256 fp16 weights
constexpr uint32_t kTmemColumns = 512;                                    // the accumulators, then the stages' weights: 3 beside up to 32 rows, else 2
constexpr uint32_t kUnpackWarps = 16, kStoreWarps = 8, kMmaWarp = 24, kRowsWarp = 25, kTilesWarp = 26, kThreads = 27 * 32;
constexpr uint32_t kSegmentRows = 64;                                     // rows whose parts of K are added up in registers: half of them per storing warp
constexpr uint32_t kChunkPairs = 16, kPairQuants = 512, kPairScales = 64, kChunkBytes = kChunkPairs * (kPairQuants + kPairScales);  // decode tiles
constexpr uint32_t kTiles = 8, kMaxRawSlots = 3, kRawPairs = 8, kRawSlot = kRawPairs * (kPairQuants + kPairScales);  // of a tile of 16 rows: quants, then scales
constexpr uint32_t kRawStages = kRawPairs / kStagePairs;
constexpr uint32_t kGroupBytes = 1024;                                  // 8 rows x 64 columns of the rows' operand
constexpr uint32_t kSwapFloats = 2 * 16 * 32;                           // per pair of storing warps: 16 rows x 32 outputs, two in turn
constexpr uint32_t kKeepPairs = 32;                                     // pairs of blocks summed in one go
constexpr uint32_t kSpinLimit = 1u << 22;

__device__ int* g_wait_word;  // where a wait that ran out leaves its code (kernels.h), null until set

__device__ __forceinline__ void give_up(volatile int* dead, int code) {
    *dead = 1;
    if (g_wait_word) *reinterpret_cast<volatile int*>(g_wait_word) = code;
}

// A whole warp's wait; false, with the code left behind, when it runs out. What follows a first poll that failed is out of the way
// of the code that passes.
__device__ __noinline__ bool wait_on(uint32_t bar, uint32_t parity, volatile int* dead, int code) {
    if (__all_sync(0xffffffffu, mbar_wait(bar, parity, kSpinLimit, dead))) return true;
    if ((threadIdx.x & 31) == 0) give_up(dead, code);
    return false;
}
__device__ __forceinline__ bool await(uint32_t bar, uint32_t parity, volatile int* dead, int code) {
    return __all_sync(0xffffffffu, mbar_test(bar, parity)) || wait_on(bar, parity, dead, code);
}

struct ExpertsUmmaParams {
    const uint8_t* tiles[2];  // gate (or the matrix), up: decode tiles of the stacked experts
    float* y;                 // [entry][n_rows]
    const __half* packed;     // [pair][expert * cap_groups + group][8 cores][8 rows][8 halves]
    const uint32_t* offsets;
    const uint32_t* entries;
    uint32_t n_experts, n_rows, n_pairs, n_jobs, cap_groups, tile_tokens, stages, raw_slots;
};

// The expert and the place among its groups (of up to `rows` entries) of group number `group` of all experts; false, with
// the number of groups in `place`, if there are fewer. The whole warp calls it.
__device__ __forceinline__ bool find_group(const ExpertsUmmaParams& p, uint32_t group, uint32_t& expert, uint32_t& place) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t before = 0;
    for (uint32_t base = 0; base < p.n_experts; base += 32) {
        const uint32_t count = base + lane < p.n_experts ? (p.offsets[base + lane + 1] - p.offsets[base + lane] + p.tile_tokens - 1) / p.tile_tokens : 0;
        uint32_t sum = count;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const uint32_t lower = __shfl_up_sync(0xffffffffu, sum, d);
            if (lane >= (uint32_t)d) sum += lower;
        }
        const uint32_t holds = __ballot_sync(0xffffffffu, before + sum > group);
        if (holds) {
            const int at = __ffs(holds) - 1;
            expert = base + at;
            place = group - before - __shfl_sync(0xffffffffu, sum - count, at);
            return true;
        }
        before += __shfl_sync(0xffffffffu, sum, 31);
    }
    place = before;
    return false;
}

// A CTA's run of jobs through all groups; each role walks it by itself.
struct Run {
    uint32_t left, group, job, expert, place;
    // The CTA's share of the jobs of n_groups groups.
    __device__ __forceinline__ void start(const ExpertsUmmaParams& p, uint32_t n_groups) {
        const uint64_t jobs = (uint64_t)n_groups * p.n_jobs, at = jobs * blockIdx.x / gridDim.x;
        left = (uint32_t)(jobs * (blockIdx.x + 1) / gridDim.x - at);
        group = (uint32_t)(at / p.n_jobs) - 1;  // the first step goes on to its group
        job = p.n_jobs - 1;
        first = (uint32_t)(at % p.n_jobs);
    }
    __device__ __forceinline__ bool next(const ExpertsUmmaParams& p) {
        if (left == 0) return false;
        --left;
        if (++job == p.n_jobs) {
            job = first;
            first = 0;
            find_group(p, ++group, expert, place);
        }
        return true;
    }
    uint32_t first;
};

// One thread: D[tmem] (+)= A[tmem] * B^T over K = 16.
__device__ __forceinline__ void umma_f16_a_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Whole warp: 16 lanes x 32 columns of tensor memory; register 2 j of lane (g, t) goes to lane g, column 4 j + t, register 2 j + 1
// to lane g + 8.
__device__ __forceinline__ void tmem_store_16x32(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]),
                 "r"(v[14]), "r"(v[15])
                 : "memory");
}

// a += b, both pairs of lanes rounded to nearest.
__device__ __forceinline__ void add_two(float& a0, float& a1, float b0, float b1) {
    asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %3};\n\tadd.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}" : "+f"(a0), "+f"(a1) : "f"(b0), "f"(b1));
}

// Whole warp: 8 accumulator columns of its 32 lanes (tmem_load_16).
__device__ __forceinline__ void tmem_load_8(uint32_t taddr, float (&v)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "r"(taddr)
        : "memory");
}

// SEGMENT: pairs of blocks (64 columns each) that tensor memory sums, the sums being added up in registers, two at a time; 0: it sums all of K.
template <bool DUAL, uint32_t SEGMENT>
__global__ void __launch_bounds__(kThreads, 1) experts_umma_kernel(const __grid_constant__ ExpertsUmmaParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];  // the rows' stages, the raw slots, the swap buffers
    __shared__ __align__(8) uint64_t bars[2 * kMaxStages + 4], raw_bars[2 * kTiles * kMaxRawSlots];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int dead_flag;
    volatile int* dead = &dead_flag;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full = smem_u32(bars), free = full + kMaxStages * 8, acc_full = free + kMaxStages * 8, acc_empty = acc_full + 16;
    const uint32_t pair_bytes = p.tile_tokens / 8 * kGroupBytes, stage_bytes = kStagePairs * pair_bytes, job_stages = (p.n_pairs + kStagePairs - 1) / kStagePairs;
    const uint32_t set_columns = (SEGMENT ? 2 : 1) * p.tile_tokens, n_stages = p.stages, a_at = 2 * set_columns, raw_slots = p.raw_slots;
    const uint32_t raw_full = smem_u32(raw_bars), raw_free = raw_full + kTiles * kMaxRawSlots * 8, raw = smem_u32(smem) + n_stages * stage_bytes;
    pdl_launch_dependents();
    if (tid == 0) {
        for (uint32_t s = 0; s < n_stages; ++s) {
            mbar_init(full + 8 * s, kUnpackWarps / 2 + 1);  // the weights, and the copy of the rows
            mbar_init(free + 8 * s, 1);                     // the MMA thread's commit
        }
        for (uint32_t a = 0; a < 2; ++a) {
            mbar_init(acc_full + 8 * a, 1);
            mbar_init(acc_empty + 8 * a, kStoreWarps);
        }
        for (uint32_t i = 0; i < kTiles * kMaxRawSlots; ++i) {
            mbar_init(raw_full + 8 * i, 1);
            mbar_init(raw_free + 8 * i, 2);  // the two warps of the tile
        }
        dead_flag = 0;
        mbar_init_fence();
    }
    if (warp == kMmaWarp) tmem_alloc(smem_u32(&tmem_slot), kTmemColumns);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_slot;
    pdl_wait();  // the grouping decides the CTA's work
    Run run;
    {
        uint32_t expert, n_groups;
        find_group(p, ~0u, expert, n_groups);
        run.start(p, n_groups);
    }

    if (warp < kUnpackWarps) {
        // ---- the weights: every second stage of the CTA. Tensor memory: lanes 16 * tile, in the warp's quarter.
        const uint32_t tile = 2 * (warp & 3) + (warp >> 2 & 1), g = lane >> 2, weights_at = tmem + ((tile * 16) << 16) + a_at;
        uint32_t slot = 0, slot_phase = 0, stage = 0, phase = 1, turn = warp >> 3;  // turn 0: the warp's stage
        bool alive = true;
        for (uint32_t jobs = run.left; jobs > 0 && alive; --jobs) {
            for (uint32_t first = 0; first < job_stages && alive; first += kRawStages) {
                const uint32_t bar = (tile * kMaxRawSlots + slot) * 8, from = raw + (tile * raw_slots + slot) * kRawSlot, here = min(kRawStages, job_stages - first);
                alive = await(raw_full + bar, slot_phase, dead, 6);
                for (uint32_t s = 0; s < here && alive; ++s, turn ^= 1) {
                    if (turn == 0) {
                        // Two pairs at a time; the first two are unpacked before the wait for the stage's columns.
#pragma unroll
                        for (uint32_t h = 0; h < kStagePairs; h += 2) {
                            uint32_t v[2][16];
#pragma unroll
                            for (uint32_t i = 0; i < 2; ++i) {
                                const uint32_t pair = s * kStagePairs + h + i;
                                uint4 q;
                                uint2 d;
                                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w) : "r"(from + pair * kPairQuants + lane * 16) : "memory");
                                asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(d.x), "=r"(d.y) : "r"(from + kRawPairs * kPairQuants + pair * kPairScales + g * 8) : "memory");
                                const __half2 s0 = *reinterpret_cast<const __half2*>(&d.x), s1 = *reinterpret_cast<const __half2*>(&d.y);  // of rows g and g + 8
                                const uint4 lo0 = dequant_word(q.x, __low2half2(s0)), hi0 = dequant_word(q.y, __high2half2(s0));
                                const uint4 lo1 = dequant_word(q.z, __low2half2(s1)), hi1 = dequant_word(q.w, __high2half2(s1));
                                v[i][0] = lo0.x, v[i][1] = hi0.x, v[i][2] = lo0.y, v[i][3] = hi0.y, v[i][4] = lo0.z, v[i][5] = hi0.z, v[i][6] = lo0.w, v[i][7] = hi0.w;
                                v[i][8] = lo1.x, v[i][9] = hi1.x, v[i][10] = lo1.y, v[i][11] = hi1.y, v[i][12] = lo1.z, v[i][13] = hi1.z, v[i][14] = lo1.w, v[i][15] = hi1.w;
                            }
                            if (h == 0) {
                                alive = await(free + 8 * stage, phase, dead, 1);
                                if (!alive) break;
                                tc_fence_after_sync();
                            }
#pragma unroll
                            for (uint32_t i = 0; i < 2; ++i) tmem_store_16x32(weights_at + stage * kStageColumns + (h + i) * 32, v[i]);
                        }
                        if (!alive) break;
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(full + 8 * stage);
                    }
                    if (++stage == n_stages) stage = 0, phase ^= 1;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(raw_free + bar);
                if (++slot == raw_slots) slot = 0, slot_phase ^= 1;
            }
        }
    } else if (warp == kTilesWarp) {
        // ---- the weights' bytes: a lane per tile, eight pairs of blocks at a time by two copies. (Copies of a warp's two pairs, 16 a stage,
        // kept the copy engine busy for 0.5 us a stage.)
        const uint32_t tiles_per_expert = p.n_rows / 16, tile = lane & (kTiles - 1);
        const uint64_t tile_bytes = (uint64_t)p.n_pairs * (kPairQuants + kPairScales);
        uint32_t slot = 0, phase = 1;
        bool alive = true;
        while (alive && run.next(p)) {
            const uint32_t in_expert = DUAL ? run.job * 4 + (tile & 3) : run.job * 8 + tile;
            const bool there = in_expert < tiles_per_expert;  // past the expert's rows: whatever lies in the slot
            const uint8_t* base = p.tiles[DUAL ? tile >> 2 : 0] + ((uint64_t)run.expert * tiles_per_expert + (there ? in_expert : 0)) * tile_bytes;
            for (uint32_t pair = 0; pair < p.n_pairs; pair += kRawPairs) {
                const uint32_t bar = (tile * kMaxRawSlots + slot) * 8;
                alive = __all_sync(0xffffffffu, mbar_wait(raw_free + bar, phase, kSpinLimit, dead));
                if (!alive) {
                    if (lane == 0) give_up(dead, 7);
                    break;
                }
                if (lane < kTiles) {
                    const uint32_t chunk = pair / kChunkPairs, in_chunk = pair % kChunkPairs, pairs = min(kRawPairs, p.n_pairs - pair);
                    const uint32_t to = raw + (tile * raw_slots + slot) * kRawSlot;
                    const uint8_t* at = base + chunk * kChunkBytes;
                    if (there) {
                        mbar_arrive_expect(raw_full + bar, pairs * (kPairQuants + kPairScales));
                        bulk_load(to, at + in_chunk * kPairQuants, pairs * kPairQuants, raw_full + bar);
                        bulk_load(to + kRawPairs * kPairQuants, at + min(kChunkPairs, p.n_pairs - chunk * kChunkPairs) * kPairQuants + in_chunk * kPairScales, pairs * kPairScales,
                                  raw_full + bar);
                    } else {
                        mbar_arrive(raw_full + bar);
                    }
                }
                __syncwarp();
                if (++slot == raw_slots) slot = 0, phase ^= 1;
            }
        }
    } else if (warp == kRowsWarp) {
        // ---- the rows' operand: the groups of eight rows that the expert's region has from this place on.
        uint32_t stage = 0, phase = 1;
        const uint32_t groups = p.tile_tokens / 8, all_groups = p.n_experts * p.cap_groups;
        while (run.next(p)) {
            const uint32_t group0 = run.place * groups, here = min(groups, p.cap_groups - group0);
            const __half* from = p.packed + ((uint64_t)run.expert * p.cap_groups + group0) * (kGroupBytes / 2);
            bool alive = true;
            for (uint32_t c = 0; c < p.n_pairs; c += kStagePairs) {
                alive = await(free + 8 * stage, phase, dead, 2);
                if (!alive) break;
                if (lane == 0) {
                    const uint32_t pairs = min(kStagePairs, p.n_pairs - c);
                    mbar_arrive_expect(full + 8 * stage, pairs * here * kGroupBytes);
                    for (uint32_t i = 0; i < pairs; ++i)
                        bulk_load(smem_u32(smem) + stage * stage_bytes + i * pair_bytes, from + (uint64_t)(c + i) * all_groups * (kGroupBytes / 2), here * kGroupBytes, full + 8 * stage);
                }
                __syncwarp();
                if (++stage == n_stages) stage = 0, phase ^= 1;
            }
            if (!alive) break;
        }
    } else if (warp == kMmaWarp) {
        // ---- the tensor core. The whole warp walks the stages and one lane issues.
        uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 1;
        const uint64_t desc0 = umma_desc(smem_u32(smem), 128, kGroupBytes);
        const uint32_t idesc = umma_idesc_f16(128, p.tile_tokens);
        // Every loop ends by a vote: the compiler then keeps the descriptors in uniform registers, where the instruction wants them.
        const uint32_t jobs = run.left;
        bool alive = true;
        // A set of accumulators (of two segments, or of all of K): free, filled, handed to the storing warps.
        auto begin = [&]() {
            alive = await(acc_empty + 8 * acc, acc_phase, dead, 3);
            tc_fence_after_sync();
            return __all_sync(0xffffffffu, alive);
        };
        auto finish = [&]() {
            if (elect_one()) umma_commit(acc_full + 8 * acc);
            __syncwarp();
            if (++acc == 2) acc = 0, acc_phase ^= 1;
        };
        constexpr uint32_t kPart = SEGMENT ? 2 * SEGMENT : kStagePairs;
        for (uint32_t job = 0; __all_sync(0xffffffffu, job < jobs && alive); ++job) {
            if (SEGMENT == 0 && !begin()) break;
            for (uint32_t c = 0; c < job_stages; ++c) {
                if (SEGMENT && !begin()) break;  // ahead of the stage, which takes longer
                alive = await(full + 8 * stage, phase, dead, 4);
                if (__any_sync(0xffffffffu, !alive)) break;
                tc_fence_after_sync();
                const uint64_t b_desc = desc0 + ((stage * stage_bytes) >> 4);
                const uint32_t pairs = min(kStagePairs, p.n_pairs - c * kStagePairs);
#pragma unroll
                for (uint32_t part = 0; part < kStagePairs; part += kPart) {
                    if (part >= pairs || (part > 0 && !begin())) break;
                    if (elect_one()) {
#pragma unroll
                        for (uint32_t i = part; i < part + kPart; ++i) {
                            if (i >= pairs) break;
                            const uint32_t segment = SEGMENT ? (i - part) / SEGMENT : 0, first = SEGMENT ? (i - part) % SEGMENT : c | i;
#pragma unroll
                            for (uint32_t j = 0; j < 4; ++j)
                                umma_f16_a_tmem(tmem + acc * set_columns + segment * p.tile_tokens, tmem + a_at + stage * kStageColumns + i * 32 + j * 8,
                                                b_desc + ((i * pair_bytes + j * 256) >> 4), idesc, (first | j) != 0);
                        }
                    }
                    __syncwarp();
                    if (SEGMENT) finish();
                }
                if (__any_sync(0xffffffffu, !alive)) break;
                if (elect_one()) umma_commit(free + 8 * stage);
                __syncwarp();
                if (++stage == n_stages) stage = 0, phase ^= 1;
            }
            if (SEGMENT == 0 && alive) finish();
        }
    } else {
        // ---- the sums and stores: a warp reads lanes 32 * (warp % 4).. of tensor memory and has one half of the rows of x, 16 at a time. Of a
        // SwiGLU lanes 0 to 63 are rows of gate, the other 64 the same rows of up: of 16 rows of x either warp takes eight, and
        // they swap what the other one needs.
        const uint32_t quarter = warp & 3, half = (warp - kUnpackWarps) >> 2, block = DUAL ? quarter & 1 : quarter;
        const bool has_gate = quarter < 2;
        const uint32_t couple = half * 2 + (quarter & 1);
        float* swap = reinterpret_cast<float*>(smem + n_stages * stage_bytes + kTiles * raw_slots * kRawSlot) + couple * kSwapFloats;
        uint32_t acc = 0, acc_phase = 0, turn = 0;
        while (run.next(p)) {
            auto begin = [&]() {
                const bool ok = lane != 0 || mbar_wait(acc_full + 8 * acc, acc_phase, kSpinLimit, dead);
                // A wait that ran out voids the results; the warp walks on (further waits end at once), because another meets it below.
                if (!__all_sync(0xffffffffu, ok) && lane == 0) give_up(dead, 5);
                tc_fence_after_sync();
                return tmem + ((quarter * 32) << 16) + acc * set_columns;
            };
            auto finish = [&]() {  // the accumulator is read: the MMA thread may overwrite it
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty + 8 * acc);
                if (++acc == 2) acc = 0, acc_phase ^= 1;
            };
            // The warp's share of the rows.
            const uint32_t first = p.offsets[run.expert] + run.place * p.tile_tokens, rows = min(p.tile_tokens, p.offsets[run.expert + 1] - first);
            const uint32_t each = (rows + 31) / 32 * 16, row0 = half * each, row_end = min(rows, row0 + each);
            auto entry_of = [&](uint32_t r) { return r + (lane & 15) < row_end ? p.entries[first + r + (lane & 15)] : 0; };
            auto store = [&](uint32_t r, uint32_t entry, const float (&v)[16]) {  // rows r .. r + 15
                const uint32_t out = run.job * (DUAL ? 64 : 128) + block * 32 + lane;
                __syncwarp();
                if constexpr (DUAL) {
                    float* buffer = swap + (turn++ & 1) * (16 * 32);
#pragma unroll
                    for (int j = 0; j < 8; ++j) buffer[(has_gate ? 8 + j : j) * 32 + lane] = has_gate ? v[8 + j] : v[j];
                    asm volatile("bar.sync %0, 64;" ::"r"(1 + couple) : "memory");
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float other = buffer[(has_gate ? j : 8 + j) * 32 + lane], mine = has_gate ? v[j] : v[8 + j];
                        const float gate = has_gate ? mine : other, up = has_gate ? other : mine;
                        const uint32_t at = (has_gate ? 0 : 8) + j, row = __shfl_sync(0xffffffffu, entry, at);
                        if (r + at < row_end && out < p.n_rows) p.y[(uint64_t)row * p.n_rows + out] = gate / (1.f + expf(-gate)) * up;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const uint32_t row = __shfl_sync(0xffffffffu, entry, j);
                        if (r + j < row_end && out < p.n_rows) p.y[(uint64_t)row * p.n_rows + out] = v[j];
                    }
                }
            };
            if constexpr (SEGMENT != 0) {
                // Looked up here: behind the sums, the trips to memory would keep the accumulators of the next job waiting.
                const uint32_t entry0 = entry_of(row0), entry1 = entry_of(row0 + 16);
                const uint32_t blocks = row_end <= row0 ? 0 : row_end <= row0 + 16 ? 2 : 4;  // of eight rows
                float sum[32], *kept = reinterpret_cast<float*>(smem + n_stages * stage_bytes + kTiles * raw_slots * kRawSlot) + kStoreWarps / 2 * kSwapFloats + (warp - kUnpackWarps) * (32 * 32) + lane;
#pragma unroll
                for (int i = 0; i < 32; ++i) sum[i] = -0.f;  // leaves the first part as it is
                for (uint32_t pair = 0; pair < p.n_pairs; pair += 2 * SEGMENT) {
                    const uint32_t from = begin() + row0;
#pragma unroll
                    for (uint32_t g = 0; g < 2; ++g) {
                        if (g > 0 && pair + SEGMENT >= p.n_pairs) break;
#pragma unroll
                        for (uint32_t b = 0; b < 4; ++b) {
                            if (b >= blocks) break;
                            float v[8];
                            tmem_load_8(from + g * p.tile_tokens + 8 * b, v);
#pragma unroll
                            for (int i = 0; i < 8; i += 2) add_two(sum[8 * b + i], sum[8 * b + i + 1], v[i], v[i + 1]);
                        }
                    }
                    finish();
                    const uint32_t done = pair + 2 * SEGMENT;
                    if (done % kKeepPairs == 0 && done < p.n_pairs) {  // a long sum would lose more: its stretches are added up by themselves
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            kept[i * 32] = done == kKeepPairs ? sum[i] : kept[i * 32] + sum[i];
                            sum[i] = -0.f;
                        }
                    }
                }
                if (p.n_pairs > kKeepPairs)
#pragma unroll
                    for (int i = 0; i < 32; ++i) sum[i] += kept[i * 32];
                if (blocks > 0) store(row0, entry0, *reinterpret_cast<const float(*)[16]>(sum));
                if (blocks > 2) store(row0 + 16, entry1, *reinterpret_cast<const float(*)[16]>(sum + 16));
            } else {
                const uint32_t from = begin();
                for (uint32_t r = row0; r < row_end; r += 16) {
                    float v[16];
                    const uint32_t entry = entry_of(r);
                    tmem_load_16(from + r, v);
                    store(r, entry, v);
                }
                finish();
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (*dead) __nanosleep(100000);  // let copies and instructions still in flight land before the CTA goes
    if (warp == kMmaWarp) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem, kTmemColumns);
    }
}

// Sorted entry i of expert e (offsets[e] <= i < offsets[e + 1]) becomes row i - offsets[e] of the expert's region, which starts at
// group e * cap_groups; its row of x is the entry's token (gather: entry / n_used) or the entry itself. One thread
// per 16 bytes: core b * 4 + j of a chunk of 64 columns holds, for t = 0 .. 3, pair j of word t of block b (columns 4 t + (j & 1) and
// two on, of the low half of the block or, j >= 2, the high one). Rows past an expert's last stay unwritten: they only reach
// accumulator columns nobody stores.
__global__ void __launch_bounds__(256) pack_experts_kernel(const float* __restrict__ x, uint4* __restrict__ packed, const uint32_t* __restrict__ offsets,
                                                           const uint32_t* __restrict__ entries, uint32_t n_experts, uint32_t n_used, int gather,
                                                           uint32_t n_cols, uint32_t cap_groups, uint32_t total_entries) {
    pdl_launch_dependents();
    pdl_wait();
    const uint64_t o = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t n_chunks = n_cols / 64;
    if (o >= (uint64_t)total_entries * n_chunks * 8) return;
    const uint32_t core = o % 8, chunk = (uint32_t)(o / 8 % n_chunks), i = (uint32_t)(o / 8 / n_chunks);
    if (i >= offsets[n_experts]) return;  // a grouping over a range of experts keeps fewer entries than tokens x slots
    uint32_t lo = 0, hi = n_experts;  // the expert of sorted entry i: the last e with offsets[e] <= i
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (offsets[mid] <= i) lo = mid;
        else hi = mid;
    }
    const uint32_t local = i - offsets[lo], entry = entries[i], row = gather ? entry / n_used : entry, j = core & 3;
    const float4* src = reinterpret_cast<const float4*>(x + (uint64_t)row * n_cols + chunk * 64 + (core >> 2) * 32 + (j >> 1) * 16);
    uint32_t out[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const float4 f = src[t];
        const __half2 h = j & 1 ? __floats2half2_rn(f.y, f.w) : __floats2half2_rn(f.x, f.z);
        out[t] = *reinterpret_cast<const uint32_t*>(&h);
    }
    const uint64_t group = (uint64_t)lo * cap_groups + local / 8, groups = (uint64_t)n_experts * cap_groups;
    packed[((chunk * groups + group) * 8 + core) * 8 + (local & 7)] = make_uint4(out[0], out[1], out[2], out[3]);
}

}  // namespace

cudaError_t matmul_experts_wait_word(int* word) { return cudaMemcpyToSymbol(g_wait_word, &word, sizeof word); }

// Where the matrices have decode tiles and the jobs fill the device. Up to 64 rows an expert on the average, fewer than three jobs an SM of
// which an SM's have fewer than 16 rows together leave a batch to matmul_few_kernel, whose jobs are tiles of 16 rows: us, this kernel and that one, both with
// their packing: 4 experts of 512 x 512, 40 tokens of 2 14 and 8, of 256 x 4096, 64 tokens of 1 25 and 13; 8 of 1792 x 2048 with up (224 jobs), 40 tokens of
// 2 28 and 25, 64 tokens 28 and 32; 8 of 2048 x 1792 (128 jobs), 40 tokens 18.9 and 18.4, 96 tokens 20 and 26; 16 of 1408 x 2048 with up (352 jobs), 16 tokens of 4 35 and 32;
// 32 of 1792 x 2048 with up (896 jobs), 16 tokens of 4 50 and 53, 203 tokens 72 and 106. With more rows, narrow matrices
// of few jobs go to matmul_umma_kernel's grouped mode, whose start is shorter: 8 of 128 x 128, 300 tokens of 2 14 and 10, 4 of 512 x 512 16.5 and 15 (700 tokens 16.9 and
// 17.5), with up 8 of 96 x 128 16 and 14 (700 tokens 17 and 20); wider ones 2 of 1024 x 2816, 300 tokens of 1 25 and 31, 32 of 1792 x 2048 with up, 2048 tokens of
// 4 203 and 292. (2 of 1024 x 2816 with 2048 rows each, where this kernel's 256 jobs are a second round on some SMs: 63 and 52.)
bool matmul_experts_tiles_supported(const Mat& w, const Mat* up, uint32_t n_rows, uint32_t n_experts, uint32_t n_tokens, uint32_t n_used) {
    if (w.format != BC_Q4_0 || w.tiles == nullptr || w.n_cols % 64 != 0 || w.n_cols == 0 || (up && up->tiles == nullptr) || n_rows % 16 != 0) return false;
    const uint64_t share = ((uint64_t)n_tokens * n_used + n_experts - 1) / n_experts, jobs = (uint64_t)n_experts * ((n_rows + (up ? 63 : 127)) / (up ? 64 : 128)), sms = (uint64_t)sm_count();
    if (matmul_few_experts_supported(w, up, n_rows, n_experts, n_tokens, n_used)) return jobs >= 3 * sms || jobs * share >= 16 * sms;
    return w.n_cols > 512 || jobs * ((share + 127) / 128) >= (up ? 20u : 40u);
}

cudaError_t matmul_experts_tiles(cudaStream_t stream, const Mat& w, const Mat* up, uint32_t n_rows, uint32_t n_experts, const float* x, bool gather,
                                 const uint32_t* offsets, const uint32_t* entries, uint32_t n_used, float* y, uint32_t n_tokens, void* scratch) {
    if (n_rows == 0 || n_experts == 0 || n_tokens == 0) return cudaSuccess;
    const uint32_t total = n_tokens * n_used, cap_groups = ((n_tokens + 15u) & ~15u) / 8;
    const uint64_t outputs = (uint64_t)total * (w.n_cols / 64) * 8;
    cudaError_t e = launch_dependent(pack_experts_kernel, dim3((unsigned)((outputs + 255) / 256)), dim3(256), 0, stream, x, static_cast<uint4*>(scratch), offsets, entries,
                                     n_experts, n_used, gather ? 1 : 0, w.n_cols, cap_groups, total);
    if (e != cudaSuccess) return e;
    // Groups of rows as wide as an expert's likely share with room for the busier ones: a second group costs a second pass over the expert's
    // weights, wider groups only a larger operand (64 rows: 8 KB a stage).
    const uint32_t share = (total + n_experts - 1) / n_experts;
    uint32_t likely = share + 2;
    while ((likely - share) * (likely - share) < 6 * share) ++likely;
    likely = likely < n_tokens ? likely : n_tokens;
    ExpertsUmmaParams p{};
    p.tiles[0] = static_cast<const uint8_t*>(w.tiles);
    p.tiles[1] = up ? static_cast<const uint8_t*>(up->tiles) : nullptr;
    p.y = y;
    p.packed = static_cast<const __half*>(scratch);
    p.offsets = offsets;
    p.entries = entries;
    p.n_experts = n_experts;
    p.n_rows = n_rows;
    p.n_pairs = w.n_cols / 64;
    p.n_jobs = (n_rows + (up ? 63 : 127)) / (up ? 64 : 128);
    p.cap_groups = cap_groups;
    const uint32_t segment = share > kSegmentRows ? 0 : p.n_pairs <= 16 ? 1 : 2;
    p.tile_tokens = segment == 0 ? 128 : likely <= 32 ? 32 : 64;
    p.stages = p.tile_tokens == 32 ? kMaxStages : 2;
    p.raw_slots = segment == 0 ? 2 : kMaxRawSlots;
    const size_t smem = (size_t)p.stages * kStagePairs * (p.tile_tokens / 8) * kGroupBytes + kTiles * p.raw_slots * kRawSlot + kStoreWarps / 2 * kSwapFloats * sizeof(float) +
                        (segment != 0 && p.n_pairs > kKeepPairs ? kStoreWarps * 32 * 32 * sizeof(float) : 0);
    const void* kernel = segment == 0   ? up ? (const void*)experts_umma_kernel<true, 0> : (const void*)experts_umma_kernel<false, 0>
                         : segment == 1 ? up ? (const void*)experts_umma_kernel<true, 1> : (const void*)experts_umma_kernel<false, 1>
                                        : up ? (const void*)experts_umma_kernel<true, 2> : (const void*)experts_umma_kernel<false, 2>;
    if ((e = ensure_dynamic_smem(kernel, smem)) != cudaSuccess) return e;
    void* args[] = {&p};
    return launch_kernel(kernel, dim3((unsigned)sm_count()), dim3(kThreads), smem, stream, args);
}

}  // namespace k
}  // namespace bc
