// Q4_0 products against few rows (at most 64): passes over several sequences, prompts and prefill chunks of
// some tokens, the experts of a batch. Two arithmetics, one weight stream.
//
// Exact (the rows stay f32). An f32 input is exactly the sum of three bf16 values (8 significant bits
// each, and bf16 has the range of f32), a quant minus 8 is exact in bf16, so the products of mma.m16n8k16 are
// exact and its f32 accumulator holds a block's sum of 32 products; the block's fp16 scale multiplies that sum in f32, as
// the decode kernel does (lfm2.rs computes the same sums row by row in f64, crates/bobcat/src/scalar.rs:292-304).
// Half. fp16 weights (q - 8) * d rounded once, fp16 inputs, f32 sums: the arithmetic of the prefill kernels
// (crates/bobcat-metal/src/matmul.metal:519-521), from the operand their packing kernels write.
//
// What bounds it. The weights are the decode kernel's tiles (kernels_matvec_mma.cu), unpacked in registers straight into
// A fragments. A pair of blocks of a 16-row tile is 1024 weights, 576 bytes, 100 cycles per scheduler at the HBM rate. Exact
// with 8 rows it costs about 75 issue slots and 12 MMAs (one per 8 cycles and scheduler: 96 cycles); half with 32
// rows about 60 slots and 16 MMAs. Logic, shifts and the packed half and bf16 arithmetic issue every second cycle, so the loop alone, from
// shared memory and without any waiting, takes 1520 cycles per tile of 2048 columns (0.8 us; its MMAs 768, everything but its MMAs
// 870), and doubling the warps changes nothing. That is why the inputs live in registers: a warp owns a fixed range
// of K (one to three pairs of blocks) for the whole launch, loads its inputs' B fragments once, and then walks
// over the CTA's row tiles, whose weights are all it loads. (The kernels that served these shapes before: f32 tiles
// through shared memory, 240 us per product whatever its size; a group of warps per tile that read the tokens'
// fragments from shared memory for every tile, 30 us for gate and up of the 2.6B shape with 32 rows, at 36 % of its issue slots.)
//
// Work. A CTA of 16 warps covers a range of K of up to 48 pairs (3072 columns), the warps next to each
// other along K, and takes row tiles c, c + n, ... A warp leaves a tile's partial sums in shared memory, and while
// the next tile is multiplied some of the warps add them up in warp order and store. Wider matrices
// take a cluster of CTAs, one per range, which meet through distributed shared memory, again in rank order: no partial
// products in global memory, no second launch, results independent of timing. Rows beyond a launch's group of 8 (exact)
// or 32 (half) are further groups in blockIdx.y, working at the same time on the same weights out of L2; those of experts
// are cut into equal runs (at the kernel).
//
// The weights come through a ring of shared memory, a tile by one bulk copy (a slice of a tile by some more) several steps ahead, which
// one warp asks for; a step's slot is refilled once every warp has arrived with its sums. The first
// steps are requested before the wait for the preceding launch. (With per-lane cp.async into slots of a lane's own, 24 requests and their
// addresses in every warp took 2 us of a launch before its first multiply: 11 rows of the 350M shape's prompt 632 us, now 606, six
// sequences of the 2.6B shape 12.43 -> 12.16 ms; 24 rows with half operands 11.47 -> 11.52 ms a
// scoring request.)

#include <cstdlib>

#include "async_utils.cuh"
#include "device_facts.h"
#include "device_utils.cuh"
#include "kernels.h"
#include "../../include/bobcat_cuda.h"

namespace bc {
namespace k {

namespace {

constexpr uint32_t kWarps = 16, kThreads = kWarps * 32;
constexpr uint32_t kChunkPairs = 16;             // pairs of blocks per chunk of the tile layout
constexpr uint32_t kPairQuants = 512, kPairScales = 64;
constexpr uint32_t kChunkBytes = kChunkPairs * (kPairQuants + kPairScales);
constexpr uint32_t kMaxPairsPerWarp = 3;
constexpr uint32_t kMaxSlices = 8;               // CTAs per cluster
constexpr uint32_t kMaxExactTokens = 64, kHalfGroup = 32;
constexpr uint32_t kMaxFewTokens = kHalfGroup;   // half: beyond, the tcgen05 kernel on expanded weights is quicker (64 rows of gate and up at 2.6B: 20 us against 33)
constexpr uint32_t kPairBytes = kPairQuants + kPairScales;
constexpr uint32_t kSpinLimit = 1u << 22;
// Tiles per step: two where the registers allow, because what a step costs besides its multiplies (requests, hand-over, sums) is
// as many instructions as a tile's multiplies.
constexpr int tiles_per_step(int nt) { return nt <= 2 ? 2 : 1; }
constexpr uint32_t partial_bytes(int nt) { return 2 * (uint32_t)tiles_per_step(nt) * kWarps * (uint32_t)nt * 512; }

__device__ int* g_wait_word;  // where a wait that ran out leaves its code (kernels.h), null until set

// The rest of a wait whose first poll failed. One that runs out leaves a code and the warp carries on, because the others and the
// cluster's barriers need it. A function of its own, out of the way of the steps' code: 11 rows of the 350M shape's prompt take 627 us (626
// without the report), with the loop and the report inline 629 to 648.
__device__ __noinline__ void wait_on(uint32_t bar, uint32_t parity, int code) {
    for (uint32_t spin = 1; spin < kSpinLimit; ++spin)
        if (async::mbar_test(bar, parity)) return;
    if (g_wait_word) *reinterpret_cast<volatile int*>(g_wait_word) = code;
}

struct FewParams {
    // Plain: up to four matrices that share the inputs, a job per tile of their concatenation.
    // Dual: tiles[0] = gate, tiles[1] = up, a job per tile pair.
    const uint8_t* tiles[4];
    float* y[4];
    uint32_t seg_tiles[4], seg_rows[4], seg_stride[4];
    int n_segments, dual, store;
    uint32_t n_jobs;               // with experts: tiles per expert
    uint32_t n_pairs, slice_pairs; // pairs of blocks per row, and per CTA of a cluster
    uint32_t slices;               // CTAs per cluster
    uint32_t n_tokens;
    const float* x;                // exact: [n_tokens][n_pairs * 64]
    const float* norm_weight;      // constant: read ahead of the wait
    float eps;
    const uint4* packed;           // half: the packed fp16 operand, [pair][token group][8 cores][8 tokens] of 16 bytes
    uint32_t token_groups;
    __half* packed_out;            // half, dual: the result as the packed operand of the product that consumes it
    // Experts: expert z has n_jobs tiles of the stacked matrices, its rows are the
    // entries offsets[z] .. offsets[z + 1]; entry e reads x row e / n_used (gather) or e and writes y row e.
    const uint32_t* offsets;
    const uint32_t* entries;
    uint32_t n_experts;
    uint32_t n_used;
    int gather;
    uint32_t cap_groups;           // half: an expert's rows are packed from token group z * cap_groups on
};

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma_bf16_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// What is left of a pair of values after its rounded bf16 pair: exact in f32.
__device__ __forceinline__ void take_off(float& lo, float& hi, uint32_t pair) {
    lo -= __uint_as_float(pair << 16);
    hi -= __uint_as_float(pair & 0xffff0000u);
}

// The eight quants of a word minus 8, as bf16, in the order of dequant_word: (e = 0, 2), (1, 3) of the
// low nibbles, then of the high ones. 0x4300 is 128.0 with a unit in the last place of one.
__device__ __forceinline__ uint4 quants_bf16(uint32_t w) {
    const uint32_t magic = 0x43004300u, bias = 0xc308c308u;  // 128, -136
    const uint32_t one = 0x3f803f80u;
    uint32_t v[4] = {(w & 0x000f000fu) | magic, ((w >> 8) & 0x000f000fu) | magic, ((w >> 4) & 0x000f000fu) | magic, ((w >> 12) & 0x000f000fu) | magic};
#pragma unroll
    for (int i = 0; i < 4; ++i) asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(v[i]) : "r"(v[i]), "r"(one), "r"(bias));
    return make_uint4(v[0], v[1], v[2], v[3]);
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
// A float at the same shared-memory address of CTA `rank` of the cluster.
__device__ __forceinline__ float remote_float(const float* p, uint32_t rank) {
    uint32_t at;
    float v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(async::smem_u32(p)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}

// The expert and the place among its groups (of up to `rows` entries) of group number `group` of all experts; false, with
// the number of groups in `place`, if there are fewer. The whole warp calls it.
__device__ __forceinline__ bool find_group(const uint32_t* offsets, uint32_t n_experts, uint32_t rows, uint32_t group, uint32_t& expert, uint32_t& place) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t before = 0;
    for (uint32_t base = 0; base < n_experts; base += 32) {
        const uint32_t count = base + lane < n_experts ? (offsets[base + lane + 1] - offsets[base + lane] + rows - 1) / rows : 0;
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

// NT groups of 8 rows (exact: one), W pairs of blocks per warp, DEPTH steps of weights in flight.
//
// Experts: how many rows each has is known on the device alone, so the launch is as wide as the device and every CTA (cluster)
// takes an equal run of the jobs of all groups of rows, which may end in the next group, whose inputs it then loads. (A share of the CTAs
// per expert and group, for the likely number of groups, left SMs idle or began a second wave. An expert block of 32 experts of 1792
// x 2048, us with all its launches: 2 tokens 103 -> 91; passes of 15 sequences of such a model 15.6 -> 12.6 ms.)
// Built on the same loop and taken back: four more warps for the sums and stores, so that the others only multiply (12.08 ms
// against 11.95, and four more sums per tile in flight); with them a tile's loads and its first unpacking ahead of the tile before (13.1 ms: spills).
template <bool EXACT, bool EXPERTS, int NT, int W, int DEPTH>
__global__ void __launch_bounds__(kThreads, 1) matmul_few_kernel(const __grid_constant__ FewParams p) {
    static_assert(!EXACT || NT == 1, "the pieces of more rows do not fit the registers");
    constexpr uint32_t kTileSums = 128 * NT, kPieces = EXACT ? 3 : NT, T = tiles_per_step(NT), kTileSlot = W * kWarps * kPairBytes, kStepBytes = T * kTileSlot;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float sums[2][T * kTileSums];        // clusters: this CTA's sums of a step
    __shared__ __align__(8) uint64_t arrived[2];    // the warps' sums of a step are there
    __shared__ __align__(8) uint64_t full[DEPTH];   // the weights of a step are there
    __shared__ float squares[kWarps][8];            // a warp's share of the rows' sums of squares
    float4* partial = reinterpret_cast<float4*>(smem);  // [step % 2][tile][warp][row group][lane]
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t bars = async::smem_u32(arrived), full_bars = async::smem_u32(full);
    if (tid < 2) async::mbar_init(bars + tid * 8, kWarps);
    else if (tid < 2 + DEPTH) async::mbar_init(full_bars + (tid - 2) * 8, 1);
    async::mbar_init_fence();
    __syncthreads();
    pdl_launch_dependents();
    const uint32_t slices = p.slices, slice = blockIdx.x % slices, cta = blockIdx.x / slices, n_ctas = gridDim.x / slices;
    uint64_t run_at = 0, run_end = 0;  // experts: the jobs of this CTA, counted through all groups
    if constexpr (EXPERTS) {
        pdl_wait();  // the grouping decides the CTA's work
        uint32_t expert, n_groups;
        find_group(p.offsets, p.n_experts, 8 * NT, ~0u, expert, n_groups);
        run_at = (uint64_t)n_groups * p.n_jobs * cta / n_ctas;
        run_end = (uint64_t)n_groups * p.n_jobs * (cta + 1) / n_ctas;
    }
    // This CTA's pairs, and of these this warp's: [pair0, pair0 + live).
    const uint32_t slice_pair0 = slice * p.slice_pairs, slice_pairs = min(p.n_pairs - slice_pair0, p.slice_pairs), pair0 = slice_pair0 + warp * W;
    const uint32_t live = warp * W < slice_pairs ? min((uint32_t)W, slice_pairs - warp * W) : 0;
    const uint64_t tile_bytes = (uint64_t)p.n_pairs * kPairBytes;

    // Where the lane's share of each pair lies in a slot: a whole tile as it lies in memory, a slice's quants ahead of its scales.
    uint32_t quant_at[W], scale_at[W];
#pragma unroll
    for (int i = 0; i < W; ++i) {
        const uint32_t pair = warp * W + i, chunk = pair / kChunkPairs, in_chunk = pair % kChunkPairs;
        const uint32_t chunk_pairs = min(kChunkPairs, slice_pairs - min(slice_pairs, chunk * kChunkPairs));
        quant_at[i] = (slices == 1 ? chunk * kChunkBytes + in_chunk * kPairQuants : pair * kPairQuants) + lane * 16;
        scale_at[i] = (slices == 1 ? chunk * kChunkBytes + chunk_pairs * kPairQuants + in_chunk * kPairScales : kWarps * W * kPairQuants + pair * kPairScales) + g * 8;
    }

    // The stream of weights, in the order in which the steps are multiplied, through all groups. The warps ask for steps in turn (always the
    // same one made 24 rows of the 2.6B shape 1 % slower); with experts the last one does, which keeps the place. One lane
    // copies a whole tile; of a slice, each lane the quants or the scales of one chunk. (A lane's copy starts copy_src into the
    // tile; lanes 16 and up serve the step's second tile.)
    uint32_t copy_bytes = (lane & 15) == 0 ? (uint32_t)tile_bytes : 0, copy_src = 0, copy_dst = 0;
    if (slices > 1) {
        const uint32_t chunk = slice_pair0 / kChunkPairs + (lane >> 1 & 7), unit = lane & 1 ? kPairScales : kPairQuants;
        const uint32_t from = max(chunk * kChunkPairs, slice_pair0), to = min((chunk + 1) * kChunkPairs, slice_pair0 + slice_pairs);
        copy_bytes = from < to ? (to - from) * unit : 0;
        copy_src = chunk * kChunkBytes + (lane & 1 ? min(kChunkPairs, p.n_pairs - min(chunk * kChunkPairs, p.n_pairs)) * kPairQuants : 0) + (from - chunk * kChunkPairs) * unit;
        copy_dst = (from - slice_pair0) * unit + (lane & 1 ? kWarps * W * kPairQuants : 0);
    }
    const uint32_t ring = async::smem_u32(smem) + partial_bytes(NT);
    uint64_t ask_at = run_at;
    uint32_t ask_first = cta, ask_step = n_ctas, ask_tile = 0;
    uint32_t ask_tiles = EXPERTS ? 0 : (p.n_jobs > cta ? (p.n_jobs - cta + n_ctas - 1) / n_ctas : 0) << p.dual;
    auto tile_of = [&](uint32_t tile) {
        uint32_t job = ask_first + ask_step * (tile >> p.dual);
        int seg = p.dual ? tile & 1 : 0;
        if (!EXPERTS && !p.dual) {
            while (seg + 1 < p.n_segments && job >= p.seg_tiles[seg]) {
                job -= p.seg_tiles[seg];
                ++seg;
            }
        }
        return p.tiles[seg] + (uint64_t)job * tile_bytes;
    };
    auto request = [&](uint32_t into) {
        if (ask_tile >= ask_tiles) {
            if (!EXPERTS || ask_at >= run_end) return;
            uint32_t expert = 0, place = 0;
            if (!find_group(p.offsets, p.n_experts, 8 * NT, (uint32_t)(ask_at / p.n_jobs), expert, place)) return;
            const uint32_t in_expert = (uint32_t)(ask_at % p.n_jobs), jobs = (uint32_t)min((uint64_t)(p.n_jobs - in_expert), run_end - ask_at);
            ask_first = expert * p.n_jobs + in_expert;
            ask_step = 1;
            ask_tiles = jobs << p.dual;
            ask_tile = 0;
            ask_at += jobs;
        }
        const uint32_t bar = full_bars + into * 8, tile = ask_tile + (lane >> 4);
        if (lane == 0) async::mbar_arrive_expect(bar, min(T, ask_tiles - ask_tile) * slice_pairs * kPairBytes);
        __syncwarp();
        if (copy_bytes && (lane >> 4) < T && tile < ask_tiles)
            async::bulk_load(ring + into * kStepBytes + (lane >> 4) * kTileSlot + copy_dst, tile_of(tile) + copy_src, copy_bytes, bar);
    };
    for (int d = 0; d < DEPTH; ++d, ask_tile += T)
        if (warp == kWarps - 1) request(d);

    uint32_t steps_before = 0;  // steps of the groups before this one
    uint32_t slot = 0, slot_parity = 0;
    do {  // plain: once; a whole cluster goes round or leaves together
    uint32_t n_tokens = p.n_tokens, first_entry = 0, expert = 0, group = blockIdx.y;
    uint32_t first_job = cta, job_step = n_ctas, my_jobs = p.n_jobs > cta ? (p.n_jobs - cta + n_ctas - 1) / n_ctas : 0;
    if constexpr (EXPERTS) {
        if (run_at >= run_end || !find_group(p.offsets, p.n_experts, 8 * NT, (uint32_t)(run_at / p.n_jobs), expert, group)) break;
        first_entry = p.offsets[expert];
        n_tokens = p.offsets[expert + 1] - first_entry;
        first_job = (uint32_t)(run_at % p.n_jobs);
        job_step = 1;
        my_jobs = (uint32_t)min((uint64_t)(p.n_jobs - first_job), run_end - run_at);
        run_at += my_jobs;
    }
    const uint32_t token0 = group * (8 * NT);
    const uint32_t n_tiles = p.dual ? 2 * my_jobs : my_jobs, n_steps = (n_tiles + T - 1) / T;  // of a pair of matrices the tiles alternate

    // The warp's inputs: for row g of a group, the eight columns of every block that meet this lane's quants, in
    // the order the unpacking emits; exact: as three bf16 pieces of one group, half: one piece per group.
    uint4 piece[W][2][kPieces];
    if constexpr (EXACT) {
        const uint32_t token = token0 + g;
        const bool has_row = token < n_tokens;
        float4 weight[W][2][2];
    #pragma unroll
        for (int i = 0; i < W; ++i)
    #pragma unroll
            for (int b = 0; b < 2; ++b)
    #pragma unroll
                for (int h = 0; h < 2; ++h) {
                    weight[i][b][h] = make_float4(1.f, 1.f, 1.f, 1.f);
                    if (p.norm_weight && (uint32_t)i < live)
                        weight[i][b][h] = __ldg(reinterpret_cast<const float4*>(p.norm_weight + (pair0 + i) * 64 + b * 32 + h * 16 + 4 * t));
                }
        if (!EXPERTS) pdl_wait();
        uint32_t in_row = token;
        if (EXPERTS && has_row) {
            const uint32_t entry = p.entries[first_entry + token];
            in_row = p.gather ? entry / p.n_used : entry;
        }
        float square = 0.f;
        {
            const float* row = p.x + (uint64_t)(has_row ? in_row : 0) * p.n_pairs * 64;
            float4 v[W][2][2];
    #pragma unroll
            for (int i = 0; i < W; ++i)
    #pragma unroll
                for (int b = 0; b < 2; ++b)
    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        v[i][b][h] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (has_row && (uint32_t)i < live) v[i][b][h] = *reinterpret_cast<const float4*>(row + (pair0 + i) * 64 + b * 32 + h * 16 + 4 * t);
                    }
    #pragma unroll
            for (int i = 0; i < W; ++i)
    #pragma unroll
                for (int b = 0; b < 2; ++b) {
                    float e[8];  // (0, 2), (1, 3) of the low half block, then of the high one
    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float4 x = v[i][b][h], w = weight[i][b][h];
                        square += x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
                        e[4 * h] = x.x * w.x, e[4 * h + 1] = x.z * w.z, e[4 * h + 2] = x.y * w.y, e[4 * h + 3] = x.w * w.w;
                    }
    #pragma unroll
                    for (int s = 0; s < 3; ++s) {
                        uint32_t r[4];
    #pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            r[q] = bf16_pair(e[2 * q], e[2 * q + 1]);
                            take_off(e[2 * q], e[2 * q + 1], r[q]);
                        }
                        piece[i][b][s] = make_uint4(r[0], r[1], r[2], r[3]);
                    }
                }
        }
        if (p.norm_weight) {
            square += __shfl_xor_sync(0xffffffffu, square, 1);
            square += __shfl_xor_sync(0xffffffffu, square, 2);
            if (t == 0) squares[warp][g] = square;
        }
    } else {
        if (!EXPERTS) pdl_wait();
        const uint32_t group0 = (EXPERTS ? expert * p.cap_groups : 0) + group * NT;
        const uint32_t groups = (n_tokens - token0 + 7) / 8;  // groups past the rows stay zero
#pragma unroll
        for (int i = 0; i < W; ++i)
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    piece[i][b][j] = make_uint4(0, 0, 0, 0);
                    if ((uint32_t)i < live && (uint32_t)j < groups)
                        piece[i][b][j] = __ldcg(p.packed + (((uint64_t)(pair0 + i) * p.token_groups + group0 + j) * 8 + b * 4 + t) * 8 + g);  // not __ldg: it may move ahead of the wait
                }
    }

    if (live == 0) {  // a warp without a range of K: its sums are zero, once for all steps
#pragma unroll
        for (uint32_t i = 0; i < 2 * T; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) partial[((i * kWarps + warp) * NT + j) * 32 + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
    }

    // ---- The steps. A warp multiplies the tiles of step u into registers; then, once every warp has left its
    // sums of step u - 1 in shared memory, the warps whose turn it is add those up; then it leaves its own. So a warp meets the
    // others one step late and none stands at a barrier while the rest still multiply, and two buffers do:
    // whoever has arrived with step u - 1 is through with the sums of step u - 2.
    // Sums: a warp takes four rows of the tile x one group of eight of x; lane (tk, e) = (lane / 4, lane % 4).
    const uint32_t turn = NT == 1 ? warp & 3 : NT == 2 ? warp & 7 : warp;  // which four rows and which group
    const uint32_t e = lane & 3, tk = lane >> 2, row_in_tile = (turn & 3) * 4 + e, tok = token0 + (turn >> 2) * 8 + tk;
    // In the accumulator layout [group][lane][4], with the halves of a lane's four values swapped for every other pair of rows, so
    // that the 32 values a warp reads at once lie in different banks.
    const uint32_t at = ((((turn >> 2) * 32 + (row_in_tile & 7) * 4 + (tk >> 1)) * 4) + (row_in_tile >> 3) * 2 + (tk & 1)) ^ (row_in_tile & 2);
    const uint32_t out_row = EXPERTS && tok < n_tokens ? p.entries[first_entry + tok] : tok;
    auto my_turn = [&](uint32_t step) { return NT == 1 ? (step & 3) == warp >> 2 : NT == 2 ? (step & 1) == warp >> 3 : warp < 4 * NT; };
    auto over_warps = [&](uint32_t step, uint32_t h) {
        const float* base = reinterpret_cast<const float*>(partial) + (((steps_before + step) & 1) * T + h) * (kWarps * kTileSums) + at;
        float sum = 0.f;
#pragma unroll
        for (uint32_t w = 0; w < kWarps; ++w) sum += base[w * kTileSums];
        return sum;
    };
    float scale = 1.f, gate = 0.f;
    bool scaled = !EXACT || p.norm_weight == nullptr;
    auto output = [&](uint32_t tile, float*& out) {  // where this thread's output of a tile goes; false: nowhere
        uint32_t job = first_job + job_step * (tile >> p.dual);
        int seg = 0;
        if (!EXPERTS && !p.dual)
            while (seg + 1 < p.n_segments && job >= p.seg_tiles[seg]) {
                job -= p.seg_tiles[seg];
                ++seg;
            }
        const uint32_t row = job * 16 + row_in_tile;
        out = p.y[seg] + (uint64_t)out_row * p.seg_stride[seg] + row;
        return tok < n_tokens && row < p.seg_rows[seg];
    };
    // The outputs' old values of the step that is finished next, read before the multiplies that come in between.
    float old[T];
    auto fetch_old = [&](uint32_t step) {
        if (p.dual || p.store == BC_STORE_OVERWRITE || !my_turn(step) || turn % slices != slice) return;
#pragma unroll
        for (uint32_t h = 0; h < T; ++h) {
            float* out;
            if (step * T + h < n_tiles && output(step * T + h, out)) old[h] = *out;
        }
    };
    // Stores a finished step: `total(h)` gives the sum of this thread's output of its tile h.
    auto finish = [&](uint32_t step, auto&& total) {
        if constexpr (EXACT) {
            if (!scaled) {
                float squared = 0.f;  // warps without a range of K have left zeros
                for (uint32_t s = 0; s < slices; ++s) {
                    float part[kWarps];
#pragma unroll
                    for (uint32_t w = 0; w < kWarps; ++w) part[w] = slices == 1 ? squares[w][tk] : remote_float(&squares[w][tk], s);
#pragma unroll
                    for (uint32_t w = 0; w < kWarps; ++w) squared += part[w];
                }
                scale = rsqrtf(squared / (float)(p.n_pairs * 64) + p.eps);
                scaled = true;
            }
        }
#pragma unroll
        for (uint32_t h = 0; h < T; ++h) {
            const uint32_t tile = step * T + h;
            if (tile >= n_tiles) break;
            if (p.dual && !(tile & 1)) {
                gate = total(h) * scale;
                continue;
            }
            if (!EXACT && p.packed_out) {
                // The rows are columns of the next product, whose operand wants columns (0, 2), (1, 3) of a group of four
                // as pairs of halves: the lane of the first row stores the four rows' 8 bytes.
                const uint32_t row = (first_job + job_step * (tile >> 1)) * 16 + row_in_tile;
                const float v = gate / (1.f + expf(-gate)) * total(h);
                const float v1 = __shfl_down_sync(0xffffffffu, v, 1), v2 = __shfl_down_sync(0xffffffffu, v, 2), v3 = __shfl_down_sync(0xffffffffu, v, 3);
                const __half2 even = __floats2half2_rn(v, v2), odd = __floats2half2_rn(v1, v3);
                if (e == 0 && tok < p.token_groups * 8 && row < p.seg_rows[0])
                    *reinterpret_cast<uint2*>(p.packed_out + packed_operand_index(tok, row, p.token_groups)) =
                        make_uint2(*reinterpret_cast<const uint32_t*>(&even), *reinterpret_cast<const uint32_t*>(&odd));
                continue;
            }
            float* out;
            const bool stores = output(tile, out);
            float sum = total(h) * scale;
            if (p.dual) sum = gate / (1.f + expf(-gate)) * sum;
            else if (p.store == BC_STORE_ACCUMULATE) sum += old[h];
            else if (p.store == BC_STORE_SWIGLU) sum = old[h] / (1.f + expf(-old[h])) * sum;
            if (stores) *out = sum;
        }
    };
    // Clusters: this CTA's sums go to `sums`, and a step is finished one step later still, by the CTA whose rank the
    // warp's turn falls to.
    auto finish_cluster = [&](uint32_t step) {
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
        if (my_turn(step) && turn % slices == slice) {
            float part[T][kMaxSlices], total[T];  // all on their way before the first is added
#pragma unroll
            for (uint32_t h = 0; h < T; ++h)
#pragma unroll
                for (uint32_t s = 0; s < kMaxSlices; ++s) part[h][s] = s < slices ? remote_float(&sums[step & 1][h * kTileSums + turn * 32 + lane], s) : 0.f;
#pragma unroll
            for (uint32_t h = 0; h < T; ++h) {
                total[h] = 0.f;
#pragma unroll
                for (uint32_t s = 0; s < kMaxSlices; ++s) total[h] += part[h][s];
            }
            finish(step, [&](uint32_t h) { return total[h]; });
        }
    };

    for (uint32_t u = 0; u <= n_steps; ++u) {
        float acc[T][NT][4];
        const uint32_t behind = slices == 1 ? 1 : 2;
        if (u >= behind) fetch_old(u - behind);
        if (u < n_steps && live) {
            if (!async::mbar_test(full_bars + slot * 8, slot_parity)) wait_on(full_bars + slot * 8, slot_parity, 2);
            uint4 q[T][W];
            uint2 d[T][W];
#pragma unroll
            for (uint32_t h = 0; h < T; ++h)
#pragma unroll
                for (int i = 0; i < W; ++i) {
                    const uint32_t from = ring + slot * kStepBytes + h * kTileSlot;
                    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(q[h][i].x), "=r"(q[h][i].y), "=r"(q[h][i].z), "=r"(q[h][i].w) : "r"(from + quant_at[i]) : "memory");
                    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(d[h][i].x), "=r"(d[h][i].y) : "r"(from + scale_at[i]) : "memory");
                }
#pragma unroll
            for (uint32_t h = 0; h < T; ++h) {
#pragma unroll
                for (int j = 0; j < NT; ++j) acc[h][j][0] = acc[h][j][1] = acc[h][j][2] = acc[h][j][3] = 0.f;
                if (h > 0 && u * T + h >= n_tiles) continue;
#pragma unroll
                for (int i = 0; i < W; ++i) {
                    if (i > 0 && (uint32_t)i >= live) break;
                    const uint32_t rows[2][2] = {{q[h][i].x, q[h][i].y}, {q[h][i].z, q[h][i].w}};
                    const uint32_t scales[2] = {d[h][i].x, d[h][i].y};
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        const __half2 both = *reinterpret_cast<const __half2*>(&scales[b]);  // of rows g and g + 8
                        if constexpr (EXACT) {
                            const uint4 lo = quants_bf16(rows[b][0]), hi = quants_bf16(rows[b][1]);
                            const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
                            float c[4];
                            mma_bf16_first(c, a0, piece[i][b][2].x, piece[i][b][2].y);  // the smallest pieces first
                            mma_bf16(c, a1, piece[i][b][2].z, piece[i][b][2].w);
#pragma unroll
                            for (int s = 1; s >= 0; --s) {
                                mma_bf16(c, a0, piece[i][b][s].x, piece[i][b][s].y);
                                mma_bf16(c, a1, piece[i][b][s].z, piece[i][b][s].w);
                            }
                            const float2 ds = __half22float2(both);
                            acc[h][0][0] = fmaf(c[0], ds.x, acc[h][0][0]);
                            acc[h][0][1] = fmaf(c[1], ds.x, acc[h][0][1]);
                            acc[h][0][2] = fmaf(c[2], ds.y, acc[h][0][2]);
                            acc[h][0][3] = fmaf(c[3], ds.y, acc[h][0][3]);
                        } else {
                            const uint4 lo = dequant_word(rows[b][0], __low2half2(both)), hi = dequant_word(rows[b][1], __high2half2(both));
                            const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
                            for (int j = 0; j < NT; ++j) mma_f16(acc[h][j], a0, piece[i][b][j].x, piece[i][b][j].y);
#pragma unroll
                            for (int j = 0; j < NT; ++j) mma_f16(acc[h][j], a1, piece[i][b][j].z, piece[i][b][j].w);
                        }
                    }
                }
            }
        }
        if (u > 0) {
            const uint32_t before = u - 1, turns = steps_before + before;  // buffers and barriers alternate through all groups
            // Every warp arrives for every step whatever happens, so the wait ends; it is bounded like all waits.
            if (!async::mbar_test(bars + (turns & 1) * 8, (turns >> 1) & 1)) wait_on(bars + (turns & 1) * 8, (turns >> 1) & 1, 1);
            if (warp == (EXPERTS ? kWarps - 1 : before % kWarps)) request(slot == 0 ? DEPTH - 1 : slot - 1);  // every warp has its weights of that step in registers
            ask_tile += T;
            if (slices == 1) {
                if (my_turn(before)) finish(before, [&](uint32_t h) { return over_warps(before, h); });
            } else {
                if (before > 0) finish_cluster(before - 1);
                if (my_turn(before)) {
#pragma unroll
                    for (uint32_t h = 0; h < T; ++h) sums[before & 1][h * kTileSums + turn * 32 + lane] = over_warps(before, h);
                }
                asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
            }
        }
        if (u < n_steps) {
            if (live) {
#pragma unroll
                for (uint32_t h = 0; h < T; ++h)
#pragma unroll
                    for (int j = 0; j < NT; ++j)
                        partial[(((((steps_before + u) & 1) * T + h) * kWarps + warp) * NT + j) * 32 + lane] =
                            g & 2 ? make_float4(acc[h][j][2], acc[h][j][3], acc[h][j][0], acc[h][j][1]) : make_float4(acc[h][j][0], acc[h][j][1], acc[h][j][2], acc[h][j][3]);
            }
            __syncwarp();
            if (lane == 0) async::mbar_arrive(bars + ((steps_before + u) & 1) * 8);
            slot = slot == DEPTH - 1 ? 0 : slot + 1;
            slot_parity ^= slot == 0;
        }
    }
    if (slices > 1) {
        if (n_steps) {
            fetch_old(n_steps - 1);
            finish_cluster(n_steps - 1);
        }
        cluster_sync();  // no CTA leaves, or goes on, while another reads its sums
    }
    steps_before += n_steps;
    } while (EXPERTS);
}

bool switched_off(const char* name) {
    const char* v = std::getenv(name);
    return v && v[0] == '1';
}
bool exact_disabled() {
    static const bool off = switched_off("BOBCAT_NO_EXACT_MATMUL");
    return off;
}
bool few_disabled() {
    static const bool off = switched_off("BOBCAT_NO_FEW_MATMUL");
    return off;
}

template <bool EXACT, bool EXPERTS, int NT, int W, int DEPTH>
cudaError_t launch_as(cudaStream_t stream, FewParams& p, uint32_t groups) {
    const void* kernel = (const void*)matmul_few_kernel<EXACT, EXPERTS, NT, W, DEPTH>;
    const size_t smem = partial_bytes(NT) + (size_t)kWarps * DEPTH * tiles_per_step(NT) * W * kPairBytes;
    cudaError_t e = ensure_dynamic_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t config = {};
    config.blockDim = dim3(kThreads);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    int n = 0;
    if (p.slices > 1) {
        attributes[n].id = cudaLaunchAttributeClusterDimension;
        attributes[n].val.clusterDim.x = p.slices;
        attributes[n].val.clusterDim.y = attributes[n].val.clusterDim.z = 1;
        ++n;
    }
    // Clusters that fit on the device at once: a cluster lives inside one GPC, so a few SMs stay over.
    static DeviceFacts<kMaxSlices + 1> fit;
    int resident = sm_count();
    if (p.slices > 1) {
        int device = 0;
        cudaGetDevice(&device);
        const bool known = fit.get(device, (int)p.slices, [&](int* clusters) {
            config.gridDim = dim3(p.slices * (unsigned)sm_count());
            config.attrs = attributes;
            config.numAttrs = n;
            e = cudaOccupancyMaxActiveClusters(clusters, kernel, &config);
            if (e == cudaSuccess && *clusters < 1) *clusters = 1;
            return e == cudaSuccess;
        }, &resident);
        if (!known) return e;
    }
    if (EXPERTS) {
        config.gridDim = dim3(p.slices * (unsigned)resident);
    } else {
        const uint32_t share = (uint32_t)resident / groups, most = share > 0 ? share : 1;
        config.gridDim = dim3(p.slices * (p.n_jobs < most ? p.n_jobs : most), groups);
    }
    if (pdl_enabled()) {
        attributes[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attributes[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    config.attrs = attributes;
    config.numAttrs = n;
    return cudaLaunchKernelEx(&config, matmul_few_kernel<EXACT, EXPERTS, NT, W, DEPTH>, (const FewParams)p);
}
template <bool EXACT, int NT, int W, int DEPTH>
cudaError_t launch(cudaStream_t stream, FewParams& p, uint32_t groups) {
    return p.offsets ? launch_as<EXACT, true, NT, W, DEPTH>(stream, p, groups) : launch_as<EXACT, false, NT, W, DEPTH>(stream, p, groups);
}

// Cut K: as few CTAs per cluster as hold the inputs at `most` pairs per warp, evenly.
uint32_t cut(FewParams& p, uint32_t most) {
    p.slices = (p.n_pairs + kWarps * most - 1) / (kWarps * most);
    p.slice_pairs = (p.n_pairs + p.slices - 1) / p.slices;
    p.slices = (p.n_pairs + p.slice_pairs - 1) / p.slice_pairs;
    return (p.slice_pairs + kWarps - 1) / kWarps;  // pairs per warp
}

cudaError_t launch_exact(cudaStream_t stream, FewParams& p) {
    const uint32_t groups = (p.n_tokens + 7) / 8;
    switch (cut(p, kMaxPairsPerWarp)) {
        case 1: return launch<true, 1, 1, 6>(stream, p, groups);
        case 2: return launch<true, 1, 2, 4>(stream, p, groups);
        default: return launch<true, 1, 3, 3>(stream, p, groups);
    }
}

// Row groups of 8 a launch's CTA holds: the fewest that cover the rows in as few groups of 32 as possible
// (33 rows: two groups of 24). `rows`: those of the largest (expert: likely) batch.
cudaError_t launch_half(cudaStream_t stream, FewParams& p, uint32_t rows) {
    const uint32_t parts = (rows + kHalfGroup - 1) / kHalfGroup, nt = ((rows + parts - 1) / parts + 7) / 8;
    const uint32_t w = cut(p, nt <= 2 ? 3 : 2), groups = (p.n_tokens + 8 * (nt < 2 ? 2 : nt) - 1) / (8 * (nt < 2 ? 2 : nt));
    if (nt <= 2) {
        switch (w) {
            case 1: return launch<false, 2, 1, 6>(stream, p, groups);
            case 2: return launch<false, 2, 2, 4>(stream, p, groups);
            default: return launch<false, 2, 3, 2>(stream, p, groups);
        }
    }
    if (nt == 3) return w == 1 ? launch<false, 3, 1, 8>(stream, p, groups) : launch<false, 3, 2, 6>(stream, p, groups);
    return w == 1 ? launch<false, 4, 1, 8>(stream, p, groups) : launch<false, 4, 2, 6>(stream, p, groups);
}

}  // namespace

cudaError_t matmul_few_wait_word(int* word) { return cudaMemcpyToSymbol(g_wait_word, &word, sizeof word); }

// Up to 64 rows: every group of 8 rows repeats the weights' unpacking, which stays ahead of the tile
// kernel at any of these counts. The inputs of a row must fit a cluster's registers (24 576 columns).
bool matmul_exact_supported(const Mat& w, uint32_t n_tokens) {
    return !exact_disabled() && w.format == BC_Q4_0 && w.tiles != nullptr && n_tokens > 0 && n_tokens <= kMaxExactTokens && w.n_cols % 64 == 0 && w.n_cols > 0 &&
           w.n_cols / 64 <= kWarps * kMaxPairsPerWarp * kMaxSlices;
}

cudaError_t matmul_exact(cudaStream_t stream, const Mat* const* ws, float* const* ys, const uint32_t* strides, int n, const float* x, Norm norm,
                         uint32_t n_tokens, int32_t store) {
    if (n < 1 || n > 4 || !matmul_exact_supported(*ws[0], n_tokens) || (norm.weight && !norm.constant)) return cudaErrorInvalidValue;
    FewParams p{};
    p.n_segments = n;
    for (int i = 0; i < n; ++i) {
        if (ws[i]->n_cols != ws[0]->n_cols || !ws[i]->tiles) return cudaErrorInvalidValue;
        p.tiles[i] = static_cast<const uint8_t*>(ws[i]->tiles);
        p.y[i] = ys[i];
        p.seg_tiles[i] = (ws[i]->n_rows + 15) / 16;
        p.seg_rows[i] = ws[i]->n_rows;
        p.seg_stride[i] = strides[i];
        p.n_jobs += p.seg_tiles[i];
    }
    if (p.n_jobs == 0) return cudaSuccess;
    p.n_pairs = ws[0]->n_cols / 64;
    p.n_tokens = n_tokens;
    p.x = x;
    p.norm_weight = norm.weight;
    p.eps = norm.eps;
    p.store = store;
    return launch_exact(stream, p);
}

cudaError_t matmul_exact_swiglu(cudaStream_t stream, const Mat& gate, const Mat& up, const float* x, Norm norm, float* y, uint32_t n_tokens) {
    if (gate.n_rows != up.n_rows || gate.n_cols != up.n_cols || !matmul_exact_supported(gate, n_tokens) || !up.tiles || (norm.weight && !norm.constant)) return cudaErrorInvalidValue;
    FewParams p{};
    p.n_segments = 1;
    p.dual = 1;
    p.tiles[0] = static_cast<const uint8_t*>(gate.tiles);
    p.tiles[1] = static_cast<const uint8_t*>(up.tiles);
    p.y[0] = y;
    p.seg_rows[0] = p.seg_stride[0] = gate.n_rows;
    p.n_jobs = p.seg_tiles[0] = (gate.n_rows + 15) / 16;
    if (p.n_jobs == 0) return cudaSuccess;
    p.n_pairs = gate.n_cols / 64;
    p.n_tokens = n_tokens;
    p.x = x;
    p.norm_weight = norm.weight;
    p.eps = norm.eps;
    p.store = BC_STORE_OVERWRITE;
    return launch_exact(stream, p);
}

bool matmul_exact_experts_supported(const Mat& w, const Mat* up, uint32_t n_rows, uint32_t n_tokens) {
    return matmul_exact_supported(w, n_tokens) && n_rows % 16 == 0 && (!up || (up->format == BC_Q4_0 && up->tiles && up->n_cols == w.n_cols));
}

cudaError_t matmul_exact_experts(cudaStream_t stream, const Mat& w, const Mat* up, uint32_t n_rows, uint32_t n_experts, const float* x, bool gather,
                                 const uint32_t* offsets, const uint32_t* entries, uint32_t n_used, float* y, uint32_t n_tokens) {
    if (!matmul_exact_experts_supported(w, up, n_rows, n_tokens)) return cudaErrorInvalidValue;
    if (n_rows == 0 || n_experts == 0) return cudaSuccess;
    FewParams p{};
    p.n_segments = 1;
    p.tiles[0] = static_cast<const uint8_t*>(w.tiles);
    if (up) p.tiles[1] = static_cast<const uint8_t*>(up->tiles), p.dual = 1;
    p.y[0] = y;
    p.seg_rows[0] = p.seg_stride[0] = n_rows;
    p.n_jobs = n_rows / 16;
    p.n_pairs = w.n_cols / 64;
    p.n_tokens = n_tokens;  // an expert gets at most all of them
    p.x = x;
    p.store = BC_STORE_OVERWRITE;
    p.offsets = offsets;
    p.entries = entries;
    p.n_experts = n_experts;
    p.n_used = n_used;
    p.gather = gather;
    return launch_exact(stream, p);
}

// ---- half-precision operands

bool matmul_few_supported(const Mat& w, uint32_t n_tokens) {
    return !few_disabled() && w.format == BC_Q4_0 && w.tiles != nullptr && n_tokens > 0 && n_tokens <= kMaxFewTokens && w.n_cols % 64 == 0 && w.n_cols > 0 &&
           w.n_cols / 64 <= kWarps * 2 * kMaxSlices;
}

cudaError_t matmul_few(cudaStream_t stream, const Mat* const* ws, float* const* ys, const uint32_t* strides, int n, const void* packed,
                       uint32_t n_tokens, int32_t store) {
    if (n < 1 || n > 4) return cudaErrorInvalidValue;
    FewParams p{};
    p.n_segments = n;
    for (int i = 0; i < n; ++i) {
        if (ws[i]->n_cols != ws[0]->n_cols || !ws[i]->tiles) return cudaErrorInvalidValue;
        p.tiles[i] = static_cast<const uint8_t*>(ws[i]->tiles);
        p.y[i] = ys[i];
        p.seg_tiles[i] = (ws[i]->n_rows + 15) / 16;
        p.seg_rows[i] = ws[i]->n_rows;
        p.seg_stride[i] = strides[i];
        p.n_jobs += p.seg_tiles[i];
    }
    if (p.n_jobs == 0) return cudaSuccess;
    p.n_pairs = ws[0]->n_cols / 64;
    p.packed = static_cast<const uint4*>(packed);
    p.token_groups = ((n_tokens + 15u) & ~15u) / 8;
    p.n_tokens = n_tokens;
    p.store = store;
    return launch_half(stream, p, n_tokens);
}

cudaError_t matmul_few_swiglu(cudaStream_t stream, const Mat& gate, const Mat& up, const void* packed, float* y, uint32_t n_tokens, uint32_t y_stride,
                              void* packed_out) {
    if (gate.n_rows != up.n_rows || gate.n_cols != up.n_cols || !gate.tiles || !up.tiles || (packed_out && gate.n_rows % 64 != 0)) return cudaErrorInvalidValue;
    FewParams p{};
    p.n_segments = 1;
    p.dual = 1;
    p.tiles[0] = static_cast<const uint8_t*>(gate.tiles);
    p.tiles[1] = static_cast<const uint8_t*>(up.tiles);
    p.y[0] = y;
    p.seg_rows[0] = gate.n_rows;
    p.seg_stride[0] = y_stride;
    p.n_jobs = p.seg_tiles[0] = (gate.n_rows + 15) / 16;
    if (p.n_jobs == 0) return cudaSuccess;
    p.n_pairs = gate.n_cols / 64;
    p.packed = static_cast<const uint4*>(packed);
    p.token_groups = ((n_tokens + 15u) & ~15u) / 8;
    p.n_tokens = n_tokens;
    p.store = BC_STORE_OVERWRITE;
    p.packed_out = static_cast<__half*>(packed_out);
    return launch_half(stream, p, n_tokens);
}

// Experts: any number of tokens, as long as an expert gets a few of them on average (at most 64). Batches whose jobs fill the device
// go to kernels_matmul_experts.cu first.
bool matmul_few_experts_supported(const Mat& w, const Mat* up, uint32_t n_rows, uint32_t n_experts, uint32_t n_tokens, uint32_t n_used) {
    return !few_disabled() && w.format == BC_Q4_0 && w.tiles != nullptr && n_tokens > 0 && w.n_cols % 64 == 0 && w.n_cols > 0 &&
           w.n_cols / 64 <= kWarps * 2 * kMaxSlices && (!up || up->tiles != nullptr) && n_rows % 16 == 0 &&
           (uint64_t)n_tokens * n_used <= (uint64_t)64 * n_experts;
}

cudaError_t matmul_few_experts(cudaStream_t stream, const Mat& w, const Mat* up, uint32_t n_rows, uint32_t n_experts, const void* packed,
                               const uint32_t* offsets, const uint32_t* entries, float* y, uint32_t n_tokens, uint32_t n_entries) {
    if (n_rows == 0 || n_experts == 0) return cudaSuccess;
    FewParams p{};
    p.n_segments = 1;
    p.tiles[0] = static_cast<const uint8_t*>(w.tiles);
    if (up) p.tiles[1] = static_cast<const uint8_t*>(up->tiles), p.dual = 1;
    p.y[0] = y;
    p.seg_rows[0] = p.seg_stride[0] = n_rows;
    p.n_jobs = p.seg_tiles[0] = n_rows / 16;
    p.n_pairs = w.n_cols / 64;
    p.packed = static_cast<const uint4*>(packed);
    p.cap_groups = ((n_tokens + 15u) & ~15u) / 8;
    p.token_groups = n_experts * p.cap_groups;
    p.n_tokens = n_tokens;  // an expert gets at most all of them
    p.store = BC_STORE_OVERWRITE;
    p.offsets = offsets;
    p.entries = entries;
    p.n_experts = n_experts;
    p.n_used = 1;
    // Groups of rows as wide as an expert's likely share, with room for the busier ones.
    const uint32_t share = (n_entries + n_experts - 1) / n_experts;
    uint32_t rows = share + 1;
    while ((rows - share) * (rows - share) < share) ++rows;
    rows = rows < n_tokens ? rows : n_tokens;
    return launch_half(stream, p, rows < kHalfGroup ? rows : kHalfGroup);
}

}  // namespace k
}  // namespace bc
