// Q4_0 products against a few rows with f32 operands: passes over a handful of sequences, prompts of
// a few tokens, the experts of such batches, and larger batches that ask for f32 operands.
//
// Arithmetic. No operand is rounded. An f32 input is exactly the sum of three bf16 values (8
// significant bits each, and bf16 has the range of f32), a quant minus 8 is exact in bf16, so the
// products of mma.m16n8k16 are exact and its f32 accumulator holds a block's sum of 32 products; the
// block's fp16 scale multiplies that sum in f32, as the decode kernel does (lfm2.rs computes the same
// sums row by row in f64, crates/bobcat/src/scalar.rs:292-304).
//
// What bounds it. With up to 8 rows a pair of blocks of a 16-row tile (1024 weights, 576 bytes) costs
// about 75 issue slots and 12 MMAs (one per 8 cycles and scheduler), against 100 cycles per
// scheduler for its bytes at the HBM rate: the three are balanced, so the kernel is a weight stream
// like the decode kernel as long as nothing else is in the loop. That is why the inputs live in
// registers: a warp owns a fixed range of K (one to three pairs of blocks) for the whole launch, reads its
// inputs once, splits them into their bf16 pieces (24 registers per pair), and then walks over the CTA's row
// tiles, whose weights are all it loads. The tile kernel that served these shapes before dequantised
// into shared memory one element at a time: 240 us per product whatever its size.
//
// Work. A CTA of 16 warps covers a range of K of up to 48 pairs (3072 columns), the warps next to each
// other along K, and takes row tiles c, c + n, ... in batches of four tiles (two tile pairs for gate and
// up). A warp leaves a tile's 16 x 8 partial sums in shared memory; after the batch's barrier 512
// threads add the warps' sums in warp order and store. Wider matrices take a cluster of CTAs, one per
// range, which meet through distributed shared memory, again in rank order: no partial products in
// global memory, no second launch, results independent of timing. Rows beyond 8 are further groups
// of 8 in blockIdx.y, working at the same time on the same weights out of L2.
//
// The weights (decode tiles, kernels_matvec_mma.cu) come through per-lane slots of shared memory filled by
// cp.async several tiles ahead; a lane reads back only what it copied itself, so the ring needs no
// barrier. The first tiles are requested before the wait for the preceding launch.

#include <cstdlib>

#include "async_utils.cuh"
#include "device_utils.cuh"
#include "kernels.h"
#include "../../include/bobcat_cuda.h"

namespace bc {
namespace k {

namespace {

constexpr uint32_t kWarps = 16, kThreads = kWarps * 32;
constexpr uint32_t kChunkPairs = 16;             // pairs of blocks per chunk of the tile layout
constexpr uint32_t kPairQuants = 512, kPairScales = 64, kBlockBytes = 288;
constexpr uint32_t kChunkBytes = kChunkPairs * (kPairQuants + kPairScales);
constexpr uint32_t kUnits = 4;                   // tiles per batch: a thread per output of a batch
constexpr uint32_t kMaxPairsPerWarp = 3;
constexpr uint32_t kMaxSlices = 8;               // CTAs per cluster
constexpr uint32_t kMaxExactTokens = 64;
constexpr uint32_t kSlotPair = 768;              // a lane's 16 bytes of quants and 8 of scales, for 32 lanes
constexpr uint32_t kPartialBytes = 2 * kUnits * kWarps * 512;

struct ExactParams {
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
    const float* x;                // [n_tokens][n_pairs * 64]
    const float* norm_weight;
    float eps;
    // Experts: blockIdx.z is an expert of the stacked matrices (n_jobs tiles each), its rows are the
    // entries offsets[z] .. offsets[z + 1]; entry e reads x row e / n_used (gather) or e and writes y row e.
    const uint32_t* offsets;
    const uint32_t* entries;
    uint32_t n_used;
    int gather;
};

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
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

__device__ __forceinline__ void cp_async_8(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
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

// W pairs of blocks per warp, DEPTH tiles of weights in flight.
template <int W, int DEPTH>
__global__ void __launch_bounds__(kThreads, 1) matmul_exact_kernel(const ExactParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float sums[2][kUnits * 128];         // clusters: this CTA's sums of a batch
    __shared__ float squares[kWarps][8];            // a warp's share of the rows' sums of squares
    float4* partial = reinterpret_cast<float4*>(smem);  // [batch parity][unit][warp][lane]
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    pdl_launch_dependents();
    uint32_t n_tokens = p.n_tokens, first_entry = 0;
    const uint32_t slices = p.slices, slice = blockIdx.x % slices, cta = blockIdx.x / slices, n_ctas = gridDim.x / slices;
    uint64_t expert_tile = 0;
    if (p.offsets) {
        pdl_wait();  // the grouping decides the CTA's work
        first_entry = p.offsets[blockIdx.z];
        n_tokens = p.offsets[blockIdx.z + 1] - first_entry;
        expert_tile = (uint64_t)blockIdx.z * p.n_jobs;
    }
    const uint32_t token0 = blockIdx.y * 8;
    if (token0 >= n_tokens) return;  // a whole cluster leaves together
    const uint32_t my_jobs = p.n_jobs > cta ? (p.n_jobs - cta + n_ctas - 1) / n_ctas : 0;
    const uint32_t n_units = p.dual ? 2 * my_jobs : my_jobs;
    // This warp's pairs: [pair0, pair0 + live).
    const uint32_t slice_end = min(p.n_pairs, (slice + 1) * p.slice_pairs), pair0 = slice * p.slice_pairs + warp * W;
    const uint32_t live = pair0 < slice_end ? min((uint32_t)W, slice_end - pair0) : 0;
    const uint32_t used_warps = (slice_end - slice * p.slice_pairs + W - 1) / W;  // of this CTA
    const uint64_t tile_bytes = (uint64_t)p.n_pairs * (2 * kBlockBytes);

    // Where the lane's share of each pair lies inside a tile.
    uint32_t quant_at[W], scale_at[W];
#pragma unroll
    for (int i = 0; i < W; ++i) {
        const uint32_t pair = pair0 + i, chunk = pair / kChunkPairs, in_chunk = pair % kChunkPairs;
        const uint32_t chunk_pairs = min(kChunkPairs, p.n_pairs - chunk * kChunkPairs);
        quant_at[i] = chunk * kChunkBytes + in_chunk * kPairQuants + lane * 16;
        scale_at[i] = chunk * kChunkBytes + chunk_pairs * kPairQuants + in_chunk * kPairScales + g * 8;
    }
    const uint32_t ring = async::smem_u32(smem) + kPartialBytes + warp * (DEPTH * W * kSlotPair);
    auto tile_of = [&](uint32_t unit) {
        uint32_t job = cta + n_ctas * (p.dual ? unit >> 1 : unit);
        if (p.offsets || p.dual) return p.tiles[p.dual ? unit & 1 : 0] + (expert_tile + job) * tile_bytes;
        int seg = 0;
        while (seg + 1 < p.n_segments && job >= p.seg_tiles[seg]) {
            job -= p.seg_tiles[seg];
            ++seg;
        }
        return p.tiles[seg] + (uint64_t)job * tile_bytes;
    };
    uint32_t requested = 0;  // units requested; unit u lies in slot u % DEPTH
    auto request = [&]() {
        if (requested < n_units) {
            const uint8_t* tile = tile_of(requested);
            const uint32_t slot = ring + (requested % DEPTH) * (W * kSlotPair);
#pragma unroll
            for (int i = 0; i < W; ++i) {
                if ((uint32_t)i < live) {
                    async::cp_async_16(slot + i * kSlotPair + lane * 16, tile + quant_at[i]);
                    cp_async_8(slot + i * kSlotPair + kPairQuants + lane * 8, tile + scale_at[i]);
                }
            }
        }
        async::cp_async_commit();
        ++requested;
    };
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) request();

    // The warp's inputs: row g of the group, the eight columns of every block that meet this lane's
    // quants, as three bf16 pieces in the order quants_bf16 emits.
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
    if (!p.offsets) pdl_wait();
    uint32_t in_row = token;
    if (p.offsets && has_row) {
        const uint32_t entry = p.entries[first_entry + token];
        in_row = p.gather ? entry / p.n_used : entry;
    }
    uint4 piece[W][2][3];
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

    // The output of a batch that a thread finishes: with two matrices, of both.
    const uint32_t my_unit = p.dual ? 2 * (tid >> 7) : tid >> 7, within = tid & 127, from_lane = within >> 2, from_reg = within & 3;
    const uint32_t out_row = (from_lane >> 2) + 8 * (from_reg >> 1), out_token = token0 + 2 * (from_lane & 3) + (from_reg & 1);
    const bool finishes = (!p.dual || tid < kThreads / 2) && out_token < n_tokens;
    float scale = 1.f;
    bool scaled = p.norm_weight == nullptr;
    uint32_t dest_row = out_token;
    if (p.offsets && finishes) dest_row = p.entries[first_entry + out_token];

    uint32_t parity = 0;
    for (uint32_t first = 0; first < n_units; first += kUnits, parity ^= 1) {
        const uint32_t batch = min(kUnits, n_units - first);
        for (uint32_t u = 0; u < batch; ++u) {
            const uint32_t slot = ring + ((first + u) % DEPTH) * (W * kSlotPair);
            async::cp_async_wait<DEPTH - 1>();
            uint4 q[W];
            uint2 d[W];
#pragma unroll
            for (int i = 0; i < W; ++i) {
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(q[i].x), "=r"(q[i].y), "=r"(q[i].z), "=r"(q[i].w) : "r"(slot + i * kSlotPair + lane * 16));
                asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(d[i].x), "=r"(d[i].y) : "r"(slot + i * kSlotPair + kPairQuants + lane * 8));
            }
            request();  // refills this slot: the lane has its share in registers
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < W; ++i) {
                if ((uint32_t)i >= live) break;
                const uint32_t rows[2][2] = {{q[i].x, q[i].y}, {q[i].z, q[i].w}};
                const uint32_t scales[2] = {d[i].x, d[i].y};
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const uint4 lo = quants_bf16(rows[b][0]), hi = quants_bf16(rows[b][1]);
                    const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
                    float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int s = 2; s >= 0; --s) {  // the smallest pieces first
                        mma_bf16(c, a0, piece[i][b][s].x, piece[i][b][s].y);
                        mma_bf16(c, a1, piece[i][b][s].z, piece[i][b][s].w);
                    }
                    const float2 ds = __half22float2(*reinterpret_cast<const __half2*>(&scales[b]));
                    acc[0] = fmaf(c[0], ds.x, acc[0]);
                    acc[1] = fmaf(c[1], ds.x, acc[1]);
                    acc[2] = fmaf(c[2], ds.y, acc[2]);
                    acc[3] = fmaf(c[3], ds.y, acc[3]);
                }
            }
            if (live) partial[((parity * kUnits + u) * kWarps + warp) * 32 + lane] = make_float4(acc[0], acc[1], acc[2], acc[3]);
        }
        // Where this thread's output goes, and its old value on the way.
        float* out = nullptr;
        float old = 0.f;
        const bool mine = finishes && my_unit < batch && (slices == 1 || tid % slices == slice);
        if (mine) {
            uint32_t job = cta + n_ctas * ((first + my_unit) >> p.dual);
            int seg = 0;
            if (!p.offsets && !p.dual)
                while (seg + 1 < p.n_segments && job >= p.seg_tiles[seg]) {
                    job -= p.seg_tiles[seg];
                    ++seg;
                }
            if (job * 16 + out_row < p.seg_rows[seg]) {
                out = p.y[seg] + (uint64_t)dest_row * p.seg_stride[seg] + job * 16 + out_row;
                if (!p.dual && p.store != BC_STORE_OVERWRITE) old = *out;
            }
        }
        __syncthreads();
        const float* base = reinterpret_cast<const float*>(partial + parity * (kUnits * kWarps * 32)) + within;
        float sum = 0.f, second = 0.f;
        if (slices == 1) {
            if (out) {
                for (uint32_t w = 0; w < used_warps; ++w) sum += base[(my_unit * kWarps + w) * 128];
                if (p.dual)
                    for (uint32_t w = 0; w < used_warps; ++w) second += base[((my_unit + 1) * kWarps + w) * 128];
                if (!scaled) {
                    float total = 0.f;
                    for (uint32_t w = 0; w < used_warps; ++w) total += squares[w][out_token - token0];
                    scale = rsqrtf(total / (float)(p.n_pairs * 64) + p.eps);
                    scaled = true;
                }
            }
        } else {
            // A thread sums unit tid / 128 over this CTA's warps; the cluster's CTAs share the outputs among them.
            float own = 0.f;
            if ((tid >> 7) < batch)
                for (uint32_t w = 0; w < used_warps; ++w) own += base[((tid >> 7) * kWarps + w) * 128];
            sums[parity][tid] = own;
            cluster_sync();
            if (out) {
                for (uint32_t s = 0; s < slices; ++s) sum += remote_float(&sums[parity][my_unit * 128 + within], s);
                if (p.dual)
                    for (uint32_t s = 0; s < slices; ++s) second += remote_float(&sums[parity][(my_unit + 1) * 128 + within], s);
                if (!scaled) {
                    float total = 0.f;
                    for (uint32_t s = 0; s < slices; ++s) {
                        const uint32_t pairs = min(p.n_pairs, (s + 1) * p.slice_pairs) - s * p.slice_pairs;
                        for (uint32_t w = 0; w * W < pairs; ++w) total += remote_float(&squares[w][out_token - token0], s);
                    }
                    scale = rsqrtf(total / (float)(p.n_pairs * 64) + p.eps);
                    scaled = true;
                }
            }
        }
        if (out) {
            sum *= scale;
            if (p.dual) sum = sum / (1.f + expf(-sum)) * (second * scale);
            else if (p.store == BC_STORE_ACCUMULATE) sum += old;
            else if (p.store == BC_STORE_SWIGLU) sum = old / (1.f + expf(-old)) * sum;
            *out = sum;
        }
    }
    async::cp_async_wait<0>();
    if (slices > 1) cluster_sync();  // no CTA leaves while another reads its sums
}

bool exact_disabled() {
    static const bool off = [] { const char* v = std::getenv("BOBCAT_NO_EXACT_MATMUL"); return v && v[0] == '1'; }();
    return off;
}

template <int W, int DEPTH>
cudaError_t launch(cudaStream_t stream, ExactParams& p, uint32_t groups, uint32_t experts, uint32_t busy_experts) {
    const void* kernel = (const void*)matmul_exact_kernel<W, DEPTH>;
    const size_t smem = kPartialBytes + (size_t)kWarps * DEPTH * W * kSlotPair;
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
    static int fit[kMaxSlices + 1] = {};
    int resident = sm_count();
    if (p.slices > 1) {
        if (fit[p.slices] == 0) {
            config.gridDim = dim3(p.slices * (unsigned)sm_count());
            config.attrs = attributes;
            config.numAttrs = n;
            int clusters = 0;
            e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &config);
            if (e != cudaSuccess) return e;
            fit[p.slices] = clusters > 0 ? clusters : 1;
        }
        resident = fit[p.slices];
    }
    // (Few experts get more than 8 entries: their further groups do not count.)
    const uint32_t share = (uint32_t)resident / (p.offsets ? busy_experts : groups), most = share > 0 ? share : 1;
    config.gridDim = dim3(p.slices * (p.n_jobs < most ? p.n_jobs : most), groups, experts);
    if (pdl_enabled()) {
        attributes[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attributes[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    config.attrs = attributes;
    config.numAttrs = n;
    return cudaLaunchKernelEx(&config, matmul_exact_kernel<W, DEPTH>, (const ExactParams)p);
}

// Cut K: as few CTAs per cluster as hold the inputs, then as few pairs per warp as fill the CTA.
cudaError_t launch_exact(cudaStream_t stream, ExactParams& p, uint32_t experts, uint32_t busy_experts) {
    p.slices = (p.n_pairs + kWarps * kMaxPairsPerWarp - 1) / (kWarps * kMaxPairsPerWarp);
    p.slice_pairs = (p.n_pairs + p.slices - 1) / p.slices;
    p.slices = (p.n_pairs + p.slice_pairs - 1) / p.slice_pairs;
    const uint32_t groups = (p.n_tokens + 7) / 8;
    switch ((p.slice_pairs + kWarps - 1) / kWarps) {
        case 1: return launch<1, 8>(stream, p, groups, experts, busy_experts);
        case 2: return launch<2, 5>(stream, p, groups, experts, busy_experts);
        default: return launch<3, 4>(stream, p, groups, experts, busy_experts);
    }
}

}  // namespace

// Up to 64 rows: every group of 8 rows repeats the weights' unpacking, which stays ahead of the tile
// kernel at any of these counts. The inputs of a row must fit a cluster's registers (24 576 columns).
bool matmul_exact_supported(const Mat& w, uint32_t n_tokens) {
    return !exact_disabled() && w.format == BC_Q4_0 && w.tiles != nullptr && n_tokens > 0 && n_tokens <= kMaxExactTokens && w.n_cols % 64 == 0 && w.n_cols > 0 &&
           w.n_cols / 64 <= kWarps * kMaxPairsPerWarp * kMaxSlices;
}

cudaError_t matmul_exact(cudaStream_t stream, const Mat* const* ws, float* const* ys, const uint32_t* strides, int n, const float* x, Norm norm,
                         uint32_t n_tokens, int32_t store) {
    if (n < 1 || n > 4 || !matmul_exact_supported(*ws[0], n_tokens)) return cudaErrorInvalidValue;
    ExactParams p{};
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
    return launch_exact(stream, p, 1, 1);
}

cudaError_t matmul_exact_swiglu(cudaStream_t stream, const Mat& gate, const Mat& up, const float* x, Norm norm, float* y, uint32_t n_tokens) {
    if (gate.n_rows != up.n_rows || gate.n_cols != up.n_cols || !matmul_exact_supported(gate, n_tokens) || !up.tiles) return cudaErrorInvalidValue;
    ExactParams p{};
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
    return launch_exact(stream, p, 1, 1);
}

bool matmul_exact_experts_supported(const Mat& w, const Mat* up, uint32_t n_rows, uint32_t n_tokens) {
    return matmul_exact_supported(w, n_tokens) && n_rows % 16 == 0 && (!up || (up->format == BC_Q4_0 && up->tiles && up->n_cols == w.n_cols));
}

cudaError_t matmul_exact_experts(cudaStream_t stream, const Mat& w, const Mat* up, uint32_t n_rows, uint32_t n_experts, const float* x, bool gather,
                                 const uint32_t* offsets, const uint32_t* entries, uint32_t n_used, float* y, uint32_t n_tokens) {
    if (!matmul_exact_experts_supported(w, up, n_rows, n_tokens)) return cudaErrorInvalidValue;
    if (n_rows == 0 || n_experts == 0) return cudaSuccess;
    ExactParams p{};
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
    p.n_used = n_used;
    p.gather = gather;
    // Experts that probably have entries, if the router spreads its picks: each of the others costs CTAs that leave at once.
    const uint32_t entries_in_all = n_tokens * n_used;
    uint32_t busy = (uint32_t)((uint64_t)n_experts * entries_in_all / (n_experts + entries_in_all));
    return launch_exact(stream, p, n_experts, busy > 0 ? busy : 1);
}

}  // namespace k
}  // namespace bc
