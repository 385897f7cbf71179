// Products of a large f32 matrix with one to sixteen f32 rows: the logits of a step, of a prompt's last token
// and of a pass over several sequences (the output matrix is the model's largest and is kept in f32).
//
// Bound by HBM: the matrix is read once and nothing else is large. A persistent CTA per SM of eight warps; a warp
// takes R neighbouring rows at a time and streams them through a ring of its own in shared memory with cp.async,
// across the ends of its rows, so that 96 KB are in flight on every SM from before the dependency wait to the last
// row; loads into registers stop at each row's end, where the warp adds its lanes, and leave a last wave that is
// a half empty on the average. A lane copies exactly the 16 bytes it will multiply, so no thread waits for
// another. The inputs lie in shared memory for the launch. With several rows of X a warp holds 8 x T sums and
// one read of a row's weights serves them all; the lanes' sums are added by halving (N - 1 + log N exchanges
// instead of 5 N).
//
// Every sum is the one of kernels_matvec.cu's warp per row (lane l adds the products of quads l, l + 32, ...,
// then the lanes in butterfly order), so a row's result does not depend on how many are computed together.
//
// Measured, 65536 x 2048 (537 MB): one row 114 us before, 84 now (6.4 TB/s); six rows 242 us (a warp per 64 matrix rows, bound by
// instruction issue), 85 now. 151936 x 2048 with one row: 276 us, 192 now.

#include "async_utils.cuh"
#include "device_utils.cuh"
#include "kernels.h"
#include "../../include/bobcat_cuda.h"

namespace bc {
namespace k {

namespace {

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kRingBytes = 96 * 1024;
constexpr size_t kMaxSmem = 227 * 1024 - 1024;

struct StreamParams {
    const float* w;
    const float* x;  // [n_tokens][n_cols]
    const float* norm_weight;  // one token: RMSNorm of x first
    float* y;        // [n_tokens][y_stride]
    uint32_t n_rows, n_cols, n_tokens, y_stride;
    float eps;
    bool constant;   // w: its first rows are on their way before the wait
};

template <int R, int T>
__global__ void __launch_bounds__(kThreads, 1) stream_f32_kernel(const __grid_constant__ StreamParams p) {
    constexpr int kStageBytes = R * 512, kStages = kRingBytes / (kWarps * kStageBytes), N = R * T;
    static_assert(T == 1 || (N % 32 == 0), "the sums are added by halving");
    extern __shared__ __align__(16) float4 stream_smem[];
    __shared__ float scratch[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float4* ring = stream_smem + (size_t)warp * (kStages * R * 32) + lane;
    float4* xs = stream_smem + kRingBytes / 16;
    const uint32_t quads = p.n_cols / 4, steps = (quads + 31) / 32, units = (p.n_rows + R - 1) / R, stride = gridDim.x * kWarps;
    const uint32_t first = warp * gridDim.x + blockIdx.x;  // neighbouring CTAs read neighbouring rows
    pdl_launch_dependents();

    // The stream: step `ahead_step` of unit `ahead_unit` is copied next.
    uint32_t ahead_unit = first, ahead_step = 0, ahead_slot = 0;
    const float4* w4 = reinterpret_cast<const float4*>(p.w);
    auto copy_next = [&]() {
        asm volatile("" ::: "memory");  // the slot has been read
        if (ahead_unit < units) {
            const uint32_t quad = ahead_step * 32 + lane;
            if (quad < quads) {
                const uint32_t to = async::smem_u32(ring + ahead_slot * (R * 32));
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const uint32_t row = min(ahead_unit * R + r, p.n_rows - 1);
                    async::cp_async_16(to + r * 512, w4 + (uint64_t)row * quads + quad);
                }
            }
            if (++ahead_step == steps) {
                ahead_step = 0;
                ahead_unit += stride;
            }
        }
        ahead_slot = ahead_slot + 1 == kStages ? 0 : ahead_slot + 1;
        async::cp_async_commit();  // a group per step, empty past the end
    };
    if (!p.constant) pdl_wait();
#pragma unroll
    for (int i = 0; i < kStages - 1; ++i) copy_next();
    pdl_wait();

    float scale = 1.f, sumsq = 0.f;
    const float4* x4 = reinterpret_cast<const float4*>(p.x);
    for (uint32_t i = threadIdx.x; i < T * quads; i += kThreads) {
        float4 v = T == 1 || i < p.n_tokens * quads ? x4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        if (T == 1 && p.norm_weight) {
            sumsq += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
            const float4 w = reinterpret_cast<const float4*>(p.norm_weight)[i];
            v.x *= w.x; v.y *= w.y; v.z *= w.z; v.w *= w.w;
        }
        xs[i] = v;
    }
    if (T == 1 && p.norm_weight) scale = rsqrtf(block_sum(sumsq, scratch) / (float)p.n_cols + p.eps);
    else __syncthreads();

    uint32_t slot = 0;
    for (uint32_t unit = first; unit < units; unit += stride) {
        float acc[N];
#pragma unroll
        for (int i = 0; i < N; ++i) acc[i] = 0.f;
        for (uint32_t step = 0; step < steps; ++step) {
            copy_next();  // into the slot that the previous step left
            async::cp_async_wait<kStages - 1>();
            const uint32_t quad = step * 32 + lane;
            if (quad < quads) {
                const float4* from = ring + slot * (R * 32);
                float4 w[R];
#pragma unroll
                for (int r = 0; r < R; ++r) w[r] = from[r * 32];
#pragma unroll
                for (int t = 0; t < T; ++t) {
                    const float4 xv = xs[t * quads + quad];
#pragma unroll
                    for (int r = 0; r < R; ++r) acc[r * T + t] += w[r].x * xv.x + w[r].y * xv.y + w[r].z * xv.z + w[r].w * xv.w;
                }
            }
            slot = slot + 1 == kStages ? 0 : slot + 1;
        }
        if (T == 1) {
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = warp_sum(acc[r]) * scale;
            if (lane == 0) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (unit * R + r < p.n_rows) p.y[unit * R + r] = acc[r];
            }
        } else {
            // Halving: a lane keeps half of its sums and gives the other half to its partner. Lane l ends with sums
            // l * (N / 32) + i.
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const bool upper = lane & o;
#pragma unroll
                for (int i = 0; i < N * o / 32; ++i) {
                    const float keep = upper ? acc[i + N * o / 32] : acc[i], give = upper ? acc[i] : acc[i + N * o / 32];
                    acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            }
#pragma unroll
            for (int i = 0; i < N / 32; ++i) {
                const uint32_t at = lane * (N / 32) + i, row = unit * R + at / T, token = at % T;
                if (row < p.n_rows && token < p.n_tokens) p.y[(uint64_t)token * p.y_stride + row] = acc[i];
            }
        }
    }
    async::cp_async_wait<0>();
}

template <int R, int T>
cudaError_t launch_stream(cudaStream_t stream, const StreamParams& p) {
    const size_t smem = kRingBytes + (size_t)T * p.n_cols * 4;
    cudaError_t e = ensure_dynamic_smem((const void*)stream_f32_kernel<R, T>, smem);
    if (e != cudaSuccess) return e;
    const uint32_t units = (p.n_rows + R - 1) / R, ctas = (units + kWarps - 1) / kWarps, sms = (uint32_t)sm_count();
    return launch_dependent(stream_f32_kernel<R, T>, dim3(ctas < sms ? ctas : sms), dim3(kThreads), smem, stream, p);
}

// Rows of X that fit beside the ring.
uint32_t rows_that_fit(uint32_t n_cols) { return (uint32_t)((kMaxSmem - kRingBytes) / ((size_t)n_cols * 4)); }

bool streamable(const Mat& w, const float* x) {
    return w.format == BC_F32 && w.n_cols > 0 && w.n_cols % 4 == 0 && ((reinterpret_cast<uintptr_t>(w.data) | reinterpret_cast<uintptr_t>(x)) & 15) == 0;
}

}  // namespace

// From four rows a warp and SM on the stream is worth its start; below that kernels_matvec.cu splits rows over warps.
bool stream_f32_supported(const Mat& w, const float* x) {
    return streamable(w, x) && w.n_rows >= (uint32_t)sm_count() * kWarps * 4 && rows_that_fit(w.n_cols) >= 1;
}

cudaError_t stream_f32(cudaStream_t stream, const Mat& w, const float* x, Norm norm, float* y) {
    return launch_stream<4, 1>(stream, StreamParams{static_cast<const float*>(w.data), x, norm.weight, y, w.n_rows, w.n_cols, 1, w.n_rows, norm.eps, w.constant});
}

// Several rows: as many as sixteen, when they fit beside the ring at once (a second pass would read the matrix again).
bool stream_f32_rows_supported(const Mat& w, const float* x, uint32_t n_tokens) {
    const uint32_t tile = n_tokens <= 4 ? 4 : n_tokens <= 8 ? 8 : 16;
    return streamable(w, x) && n_tokens >= 1 && n_tokens <= 16 && rows_that_fit(w.n_cols) >= tile;
}

cudaError_t stream_f32_rows(cudaStream_t stream, const Mat& w, const float* x, float* y, uint32_t n_tokens, uint32_t y_stride) {
    const StreamParams p{static_cast<const float*>(w.data), x, nullptr, y, w.n_rows, w.n_cols, n_tokens, y_stride, 0.f, w.constant};
    if (n_tokens <= 4) return launch_stream<8, 4>(stream, p);
    if (n_tokens <= 8) return launch_stream<8, 8>(stream, p);
    return launch_stream<8, 16>(stream, p);
}

}  // namespace k
}  // namespace bc
