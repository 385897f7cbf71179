// The small kernels of the decode and prefill graphs: weight repack and expansion, embedding
// gather, RMSNorm, per-head norm + rotary embedding + cache store, conversions, the batched short
// convolution, and argmax. Counterparts: crates/bobcat-metal/src/norm.metal, conv.metal,
// quant.metal:279-330 (expand).

#include "device_utils.cuh"
#include "kernels.h"
#include "../../include/bobcat_cuda.h"

namespace bc {
namespace k {

namespace {

constexpr int kThreads = 256;

inline int blocks_for(uint64_t n, int per_block = kThreads) {
    uint64_t b = (n + per_block - 1) / per_block;
    return (int)(b < 1 ? 1 : b);
}

// GGUF Q4_0 block = 2 bytes of fp16 scale + 16 bytes of quants, 18 bytes, so blocks are only
// 2-byte aligned. One thread moves one block.
__global__ void repack_q4_0_kernel(const uint8_t* __restrict__ raw, uint64_t n_blocks, uint4* __restrict__ quants,
                                   __half* __restrict__ scales) {
    uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n_blocks) return;
    const uint16_t* p = reinterpret_cast<const uint16_t*>(raw + 18 * b);
    uint16_t h[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) h[i] = p[i];
    scales[b] = __ushort_as_half(h[0]);
    uint4 q;
    q.x = h[1] | ((uint32_t)h[2] << 16);
    q.y = h[3] | ((uint32_t)h[4] << 16);
    q.z = h[5] | ((uint32_t)h[6] << 16);
    q.w = h[7] | ((uint32_t)h[8] << 16);
    quants[b] = q;
}

// One thread per Q4_0 block: value = f32(q - 8) * f32(d), the single multiply of
// scalar::dequantize_q4_0 (crates/bobcat/src/scalar.rs:98-105), so the f32 output is bit-identical.
template <typename Out>
__global__ void expand_q4_0_kernel(const uint4* __restrict__ quants, const __half* __restrict__ scales,
                                   uint64_t n_blocks, Out* __restrict__ out) {
    uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n_blocks) return;
    uint4 q = quants[b];
    float d = __half2float(scales[b]);
    uint32_t words[4] = {q.x, q.y, q.z, q.w};
    Out* o = out + 32 * b;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t byte = (words[w] >> (8 * i)) & 0xffu;
            float lo = (float)((int)(byte & 0xfu) - 8) * d;
            float hi = (float)((int)(byte >> 4) - 8) * d;
            o[4 * w + i] = (Out)lo;
            o[16 + 4 * w + i] = (Out)hi;
        }
    }
}

template <typename In, typename Out>
__global__ void convert_kernel(const In* __restrict__ src, Out* __restrict__ dst, uint64_t n) {
    pdl_launch_dependents();
    pdl_wait();
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = (Out)(float)src[i];
}

__global__ void silu_mul_kernel(float* __restrict__ x, const float* __restrict__ gate, uint64_t n) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        float g = gate[i];
        x[i] = g / (1.f + expf(-g)) * x[i];
    }
}

// Dequantise a matrix kept in its GGUF byte layout (Q8_0, Q6_K), one thread per element.
template <typename Out>
__global__ void expand_bytes_kernel(Mat w, Out* __restrict__ out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (uint64_t)w.n_rows * w.n_cols) return;
    const uint32_t row = (uint32_t)(i / w.n_cols), col = (uint32_t)(i % w.n_cols);
    float v;
    if (w.format == BC_Q8_0) v = q8_0_at(static_cast<const uint8_t*>(w.data) + (uint64_t)row * (w.n_cols >> 5) * kQ8_0BlockBytes, col);
    else v = q6k_at(static_cast<const uint8_t*>(w.data) + (uint64_t)row * (w.n_cols >> 8) * kQ6KBlockBytes, col);
    out[i] = (Out)v;
}

// grid (ceil(n_embd / threads), n_tokens)
__global__ void embed_kernel(Mat w, const uint32_t* __restrict__ tokens, Pos pos, float* __restrict__ out) {
    pdl_launch_dependents();
    pdl_wait();
    uint32_t token = tokens[(pos.ptr ? *pos.ptr : 0u) + pos.value + blockIdx.y];
    uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= w.n_cols) return;
    float v;
    if (w.format == BC_Q4_0) {
        uint64_t block = (uint64_t)token * (w.n_cols >> 5) + (c >> 5);
        const uint8_t* q = reinterpret_cast<const uint8_t*>(static_cast<const uint4*>(w.data) + block);
        uint32_t i = c & 31;
        uint8_t byte = q[i & 15];
        int n = i < 16 ? (byte & 0xf) : (byte >> 4);
        v = (float)(n - 8) * __half2float(w.scales[block]);
    } else if (w.format == BC_F16) {
        v = __half2float(static_cast<const __half*>(w.data)[(uint64_t)token * w.n_cols + c]);
    } else if (w.format == BC_Q8_0) {
        v = q8_0_at(static_cast<const uint8_t*>(w.data) + (uint64_t)token * (w.n_cols >> 5) * kQ8_0BlockBytes, c);
    } else if (w.format == BC_Q6_K) {
        v = q6k_at(static_cast<const uint8_t*>(w.data) + (uint64_t)token * (w.n_cols >> 8) * kQ6KBlockBytes, c);
    } else {
        v = static_cast<const float*>(w.data)[(uint64_t)token * w.n_cols + c];
    }
    out[(uint64_t)blockIdx.y * w.n_cols + c] = v;
}

// One CTA per row: out = w * (x * rsqrt(mean(x^2) + eps)), the order of scalar::rms_norm
// (crates/bobcat/src/scalar.rs:224-229).
__global__ void __launch_bounds__(kThreads) rms_norm_kernel(const float* __restrict__ x, const float* __restrict__ weight,
                                                             float* __restrict__ out, uint32_t n_cols, float eps) {
    __shared__ float scratch[32];
    pdl_launch_dependents();
    pdl_wait();
    const float* row = x + (uint64_t)blockIdx.x * n_cols;
    float* o = out + (uint64_t)blockIdx.x * n_cols;
    float sumsq = 0.f;
    for (uint32_t c = threadIdx.x; c < n_cols; c += blockDim.x) sumsq += row[c] * row[c];
    float total = block_sum(sumsq, scratch);
    float scale = rsqrtf(total / (float)n_cols + eps);
    for (uint32_t c = threadIdx.x; c < n_cols; c += blockDim.x) o[c] = weight[c] * (row[c] * scale);
}

struct NormRopeParams {
    const float* src;
    void* dst;
    const float* weight;
    uint32_t n_heads, head_dim, head_stride, n_rot, first_pos, src_stride, dst_stride;
    float theta, eps;
    int dst_half;
};

// One warp per (head, token): RMSNorm over head_dim with the shared weight, then the NeoX rotation
// of the first n_rot elements (pairs i, i + n_rot / 2; inverse frequency 1 / theta^(2i / n_rot)
// and angle in f32, as scalar::rope_neox does, crates/bobcat/src/scalar.rs:253-266), then the
// store as f32 or half. grid (n_heads, n_tokens), 32 threads.
__global__ void norm_rope_kernel(NormRopeParams p) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x;
    const uint32_t head = blockIdx.x, token = blockIdx.y;
    const float* src = p.src + (uint64_t)token * p.src_stride + (uint64_t)head * p.head_stride;
    const uint64_t dst_index = (uint64_t)token * p.dst_stride + (uint64_t)head * p.head_dim;
    // head_dim <= 256: each lane holds up to 8 elements, element e = lane + 32 j.
    float v[8];
    float sumsq = 0.f;
    const int per_lane = p.head_dim / 32;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        v[j] = 0.f;
        if (j < per_lane) {
            v[j] = src[lane + 32 * j];
            sumsq += v[j] * v[j];
        }
    }
    sumsq = warp_sum(sumsq);
    float scale = rsqrtf(sumsq / (float)p.head_dim + p.eps);
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (j < per_lane) v[j] = p.weight[lane + 32 * j] * (v[j] * scale);
    // Rotation: element e < n_rot / 2 pairs with e + n_rot / 2. n_rot / 2 is a multiple of 16 here
    // only when n_rot is a multiple of 32; handle any even n_rot through shared memory.
    __shared__ float head_values[256];
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (j < per_lane) head_values[lane + 32 * j] = v[j];
    __syncwarp();
    const uint32_t half_rot = p.n_rot / 2;
    const float pos = (float)(p.first_pos + token);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (j >= per_lane) continue;
        uint32_t e = lane + 32 * j;
        float result = v[j];
        if (e < p.n_rot) {
            uint32_t i = e < half_rot ? e : e - half_rot;
            float inv_freq = 1.0f / powf(p.theta, (float)(2 * i) / (float)p.n_rot);
            float angle = pos * inv_freq;
            float s, c;
            sincosf(angle, &s, &c);
            float a = head_values[i], b = head_values[i + half_rot];
            result = e < half_rot ? a * c - b * s : b * c + a * s;
        }
        if (p.dst_half) static_cast<__half*>(p.dst)[dst_index + e] = __float2half_rn(result);
        else static_cast<float*>(p.dst)[dst_index + e] = result;
    }
}

// The gated short convolution over a batch (crates/bobcat/src/lfm2.rs:456-475): bx = B * X, the
// taps over bx of this token and the kernel - 1 before it (from the batch, or from the history for
// the first tokens), times C. bcx is [n_tokens][3 n_embd], out is [n_tokens][n_embd], history is
// [kernel - 1][n_embd], oldest first. kernel <= K. The sum runs in the order of the token-by-token
// recurrence, so batches of any split give the same bits. With `packed`, the results go out as the fp16 operand
// of the product that consumes them (rows up to the next multiple of 16 tokens zero) instead of as f32 rows.
//
// Bound by L2 traffic. A thread takes V neighbouring channels (four when they can be loaded at once) of R tokens and
// keeps the window of products in registers, so B and X are read 1 + (K - 1) / R times; one thread per element, which
// reads them K times, took 9.1 us at 512 tokens of 2048 channels and 1.9 more for the history in a second launch, now
// 5.2 together. Only the first run of tokens reads the history (R >= K - 1), and the same threads rewrite it.
template <int K, int V>
__global__ void __launch_bounds__(128) short_conv_kernel(const float* __restrict__ bcx, const float* taps, float* history,
                                                         float* __restrict__ out, __half* __restrict__ packed, uint32_t n_embd, uint32_t kernel,
                                                         uint32_t n_tokens, bool constant_taps) {
    constexpr int R = K <= 4 ? 4 : 8;
    static_assert(R >= K - 1, "only the first run may read the history");
    pdl_launch_dependents();  // the output projection that reads the packed results may set itself up meanwhile
    const uint32_t ch = (blockIdx.x * blockDim.x + threadIdx.x) * V, skip = K - kernel;  // taps and window are aligned to the newest
    if (ch >= n_embd) return;
    if (!constant_taps) pdl_wait();  // the recording may have written them
    float tap[K][V];
#pragma unroll
    for (int kk = 0; kk < K; ++kk)
#pragma unroll
        for (int v = 0; v < V; ++v) tap[kk][v] = kk >= (int)skip ? taps[(uint64_t)(ch + v) * kernel + kk - skip] : 0.f;
    pdl_wait();
    auto load = [&](const float* at, float (&to)[V]) {
        if (V == 4) {
            const float4 f = *reinterpret_cast<const float4*>(at);
            to[0] = f.x, to[1 % V] = f.y, to[2 % V] = f.z, to[3 % V] = f.w;
        } else {
            to[0] = *at;
        }
    };
    auto products = [&](uint32_t t, float (&to)[V]) {
        float b[V], x[V];
        load(bcx + (uint64_t)t * 3 * n_embd + ch, b);
        load(bcx + (uint64_t)t * 3 * n_embd + 2 * n_embd + ch, x);
#pragma unroll
        for (int v = 0; v < V; ++v) to[v] = b[v] * x[v];
    };
    const uint32_t rows = packed ? (n_tokens + 15u) & ~15u : n_tokens;
    for (uint32_t run = blockIdx.y; (uint64_t)run * R < rows; run += gridDim.y) {
        const uint32_t t0 = run * R;
        float window[K - 1][V], bx[R][V], c[R][V];
#pragma unroll
        for (int kk = 0; kk < K - 1; ++kk) {
#pragma unroll
            for (int v = 0; v < V; ++v) window[kk][v] = 0.f;
            if (kk < (int)skip) continue;
            const int64_t src = (int64_t)t0 - (K - 1) + kk;
            if (t0 == 0) load(history + (uint64_t)(kk - skip) * n_embd + ch, window[kk]);
            else if (src < (int64_t)n_tokens) products((uint32_t)src, window[kk]);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int v = 0; v < V; ++v) bx[r][v] = c[r][v] = 0.f;
            if (t0 + r < n_tokens) {
                products(t0 + r, bx[r]);
                load(bcx + (uint64_t)(t0 + r) * 3 * n_embd + n_embd + ch, c[r]);
            }
        }
        // The history after the batch: slot kk holds the product of token n_tokens - (kernel - 1) + kk, or an older slot when the batch is
        // shorter than the history. Read beside the rest, written at the end: one after the other behind the outputs they were two trips to L2.
        float kept[K - 1][V];
        if (t0 == 0) {
#pragma unroll
            for (int kk = 0; kk < K - 1; ++kk) {
                if (kk < (int)skip) continue;
                const int64_t src = (int64_t)n_tokens - (K - 1) + kk;
                if (src >= 0) products((uint32_t)src, kept[kk]);
                else load(history + (uint64_t)(src + K - 1 - skip) * n_embd + ch, kept[kk]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            float y[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                float sum = tap[K - 1][v] * bx[r][v];
#pragma unroll
                for (int kk = 0; kk < K - 1; ++kk)
                    if (kk >= (int)skip) sum += tap[kk][v] * (r + kk < K - 1 ? window[r + kk < K - 1 ? r + kk : 0][v] : bx[r + kk >= K - 1 ? r + kk - (K - 1) : 0][v]);
                y[v] = c[r][v] * sum;
            }
            if (t0 + r >= rows) break;
            if (packed) {  // four neighbouring columns are 8 bytes in the order 0, 2, 1, 3
                const __half2 p0 = __floats2half2_rn(y[0], y[2 % V]), p1 = __floats2half2_rn(y[1 % V], y[3 % V]);
                *reinterpret_cast<uint2*>(packed + packed_operand_index(t0 + r, ch, rows / 8)) =
                    make_uint2(*reinterpret_cast<const uint32_t*>(&p0), *reinterpret_cast<const uint32_t*>(&p1));
            } else if (V == 4) {
                *reinterpret_cast<float4*>(out + (uint64_t)(t0 + r) * n_embd + ch) = make_float4(y[0], y[1 % V], y[2 % V], y[3 % V]);
            } else {
                out[(uint64_t)(t0 + r) * n_embd + ch] = y[0];
            }
        }
        if (t0 != 0) continue;
#pragma unroll
        for (int kk = 0; kk < K - 1; ++kk) {
            if (kk < (int)skip) continue;
#pragma unroll
            for (int v = 0; v < V; ++v) history[(uint64_t)(kk - skip) * n_embd + ch + v] = kept[kk][v];
        }
    }
}

// One cluster (or a CTA) scans the vocabulary; ties go to the lowest index.
struct ArgmaxOut {
    uint32_t* out;       // direct mode: the word to write
    uint32_t* readback;  // direct mode: optional host-mapped copy
    uint32_t* counter;   // step mode (non-null): position counter
    int advance;
    uint32_t* tokens;
    uint32_t offset;
    uint32_t* ring;
    uint32_t ring_slots;
};

template <unsigned CTAS>
__global__ void __launch_bounds__(kArgmaxThreads) argmax_kernel(const float* __restrict__ x, uint32_t n, ArgmaxOut o) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t index = argmax_cluster<CTAS>(x, n);
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    if (o.counter) {
        uint32_t pos = *o.counter;
        if (o.advance) {
            pos += 1;
            *o.counter = pos;
        }
        o.tokens[pos + o.offset] = index;
        if (o.ring) o.ring[pos % o.ring_slots] = index;
    } else {
        *o.out = index;
        if (o.readback) *o.readback = index;
    }
}

// One warp per head. Blocks [0, n_heads) treat q, [n_heads, n_heads + n_kv) treat k, the rest copy v.
__global__ void rope_store_kernel(RopeStore p, Pos pos_ref) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x;
    const uint32_t pos = (pos_ref.ptr ? *pos_ref.ptr : 0u) + pos_ref.value;
    const uint32_t hd = p.head_dim, kv_dim = p.n_kv_heads * hd;
    uint32_t block = blockIdx.x;
    if (block >= p.n_heads + p.n_kv_heads) {
        uint32_t head = block - p.n_heads - p.n_kv_heads;
        const float* src = p.v + (uint64_t)head * hd;
        uint64_t at = (uint64_t)pos * kv_dim + (uint64_t)head * hd;
        for (uint32_t e = lane; e < hd; e += 32) {
            if (p.kv_half) static_cast<__half*>(p.v_cache)[at + e] = __float2half_rn(src[e]);
            else static_cast<float*>(p.v_cache)[at + e] = src[e];
        }
        return;
    }
    const bool is_q = block < p.n_heads;
    const uint32_t head = is_q ? block : block - p.n_heads;
    const float* src = is_q ? p.q + (uint64_t)head * p.q_head_stride : p.k + (uint64_t)head * hd;
    const float* weight = is_q ? p.q_norm : p.k_norm;
    __shared__ float values[256];
    float sumsq = 0.f;
    for (uint32_t e = lane; e < hd; e += 32) {
        float v = src[e];
        values[e] = v;
        sumsq += v * v;
    }
    sumsq = warp_sum(sumsq);
    const float scale = rsqrtf(sumsq / (float)hd + p.eps);
    __syncwarp();
    for (uint32_t e = lane; e < hd; e += 32) values[e] = weight[e] * (values[e] * scale);
    __syncwarp();
    const uint32_t half_rot = p.n_rot / 2;
    for (uint32_t e = lane; e < hd; e += 32) {
        float result = values[e];
        if (e < p.n_rot) {
            uint32_t i = e < half_rot ? e : e - half_rot;
            float inv_freq = 1.0f / powf(p.theta, (float)(2 * i) / (float)p.n_rot);
            float angle = (float)pos * inv_freq;
            float s, c;
            sincosf(angle, &s, &c);
            float a = values[i], b = values[i + half_rot];
            result = e < half_rot ? a * c - b * s : b * c + a * s;
        }
        if (is_q) {
            p.q[(uint64_t)head * p.q_head_stride + e] = result;
        } else {
            uint64_t at = (uint64_t)pos * kv_dim + (uint64_t)head * hd + e;
            if (p.kv_half) static_cast<__half*>(p.k_cache)[at] = __float2half_rn(result);
            else static_cast<float*>(p.k_cache)[at] = result;
        }
    }
}

// The batch form: norm and rotation of q and k, and the K and V rows into the caches. A CTA serves a token (with gridDim.y
// CTAs to a token when there are few), a warp a head at a time; the token's cosines and sines, the costly part, are
// computed once per CTA (or read from the table), where a launch each for q, k and v with a warp per head computed them
// per element: 24.5 us together at 512 tokens of 32 + 8 + 8 heads of 64, now 8.7. Same arithmetic as norm_rope_kernel.
constexpr int kRopeWarps = 8;

__global__ void __launch_bounds__(32 * kRopeWarps) rope_store_batch_kernel(RopeBatch p) {
    __shared__ float head_values[kRopeWarps][256];
    __shared__ float2 rot[128];
    pdl_launch_dependents();
    const uint32_t token = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t half_rot = p.n_rot / 2, pos = p.first_pos + token;
    if (tid < half_rot) {
        if (p.rope_table) {
            rot[tid] = p.rope_table[(uint64_t)pos * half_rot + tid];
        } else {
            const float inv_freq = 1.0f / powf(p.theta, (float)(2 * tid) / (float)p.n_rot);
            float sn, cs;
            sincosf((float)pos * inv_freq, &sn, &cs);
            rot[tid] = make_float2(cs, sn);
        }
    }
    __syncthreads();
    pdl_wait();
    const uint32_t hd = p.head_dim, kv_dim = p.n_kv_heads * hd, heads = p.n_heads + p.n_kv_heads + (p.v_dst ? p.n_kv_heads : 0);
    float* values = head_values[warp];
    const int per_lane = hd / 32;
    for (uint32_t item = blockIdx.y * kRopeWarps + warp; item < heads; item += gridDim.y * kRopeWarps) {
        const bool is_q = item < p.n_heads, is_v = item >= p.n_heads + p.n_kv_heads;
        const uint32_t head = is_q ? item : is_v ? item - p.n_heads - p.n_kv_heads : item - p.n_heads;
        const float* src = is_q ? p.q + (uint64_t)token * p.q_stride + (uint64_t)head * p.q_head_stride
                                : (is_v ? p.v : p.k) + (uint64_t)token * kv_dim + (uint64_t)head * hd;
        const uint64_t at = (uint64_t)token * kv_dim + (uint64_t)head * hd;
        float v[8];
        float sumsq = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            v[j] = 0.f;
            if (j < per_lane) {
                v[j] = src[lane + 32 * j];
                sumsq += v[j] * v[j];
            }
        }
        if (is_v) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (j < per_lane) p.v_dst[at + lane + 32 * j] = __float2half_rn(v[j]);
            continue;
        }
        sumsq = warp_sum(sumsq);
        const float scale = rsqrtf(sumsq / (float)hd + p.eps);
        const float* weight = is_q ? p.q_norm : p.k_norm;
        __syncwarp();  // the previous head's values are read
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j < per_lane) {
                v[j] = weight[lane + 32 * j] * (v[j] * scale);
                values[lane + 32 * j] = v[j];
            }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j >= per_lane) continue;
            const uint32_t e = lane + 32 * j;
            float result = v[j];
            if (e < p.n_rot) {
                const uint32_t i = e < half_rot ? e : e - half_rot;
                const float a = values[i], b = values[i + half_rot];
                const float2 cs = rot[i];
                result = e < half_rot ? a * cs.x - b * cs.y : b * cs.x + a * cs.y;
            }
            if (is_q) p.q_dst[(uint64_t)token * p.q_dst_stride + (uint64_t)head * p.q_dst_head_stride + e] = result;
            else if (p.kv_half) static_cast<__half*>(p.k_dst)[at + e] = __float2half_rn(result);
            else static_cast<float*>(p.k_dst)[at + e] = result;
        }
    }
}

__global__ void rope_table_kernel(float2* table, uint32_t n_positions, uint32_t n_rot, float theta) {
    const uint32_t half_rot = n_rot / 2;
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (uint64_t)n_positions * half_rot) return;
    const uint32_t pos = (uint32_t)(i / half_rot), pair = (uint32_t)(i % half_rot);
    const float inv_freq = 1.0f / powf(theta, (float)(2 * pair) / (float)n_rot);
    float s, c;
    sincosf((float)pos * inv_freq, &s, &c);
    table[i] = make_float2(c, s);
}

// y[i] += x[i].
__global__ void add_floats_kernel(float* __restrict__ y, const float* __restrict__ x, uint64_t n) {
    pdl_launch_dependents();
    pdl_wait();
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] += x[i];
}

__global__ void advance_kernel(uint32_t* counter) {
    pdl_launch_dependents();
    pdl_wait();
    *counter += 1;
}

__global__ void seed_step_kernel(const volatile uint32_t* seed, uint32_t* counter, uint32_t* tokens) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t pos = seed[0];
    *counter = pos;
    tokens[pos] = seed[1];
}

}  // namespace

cudaError_t repack_q4_0(cudaStream_t stream, const uint8_t* raw, uint64_t n_blocks, void* quants, __half* scales) {
    if (n_blocks == 0) return cudaSuccess;
    repack_q4_0_kernel<<<blocks_for(n_blocks), kThreads, 0, stream>>>(raw, n_blocks, static_cast<uint4*>(quants), scales);
    return cudaGetLastError();
}

cudaError_t expand(cudaStream_t stream, const Mat& w, void* out, bool out_half) {
    uint64_t n = (uint64_t)w.n_rows * w.n_cols;
    if (n == 0) return cudaSuccess;
    if (w.format == BC_Q4_0) {
        uint64_t nb = n / 32;
        if (out_half)
            expand_q4_0_kernel<__half><<<blocks_for(nb), kThreads, 0, stream>>>(static_cast<const uint4*>(w.data), w.scales, nb, static_cast<__half*>(out));
        else
            expand_q4_0_kernel<float><<<blocks_for(nb), kThreads, 0, stream>>>(static_cast<const uint4*>(w.data), w.scales, nb, static_cast<float*>(out));
    } else if (w.format == BC_Q8_0 || w.format == BC_Q6_K) {
        if (out_half) expand_bytes_kernel<__half><<<blocks_for(n), kThreads, 0, stream>>>(w, static_cast<__half*>(out));
        else expand_bytes_kernel<float><<<blocks_for(n), kThreads, 0, stream>>>(w, static_cast<float*>(out));
    } else if (w.format == BC_F16) {
        if (out_half) convert_kernel<__half, __half><<<blocks_for(n), kThreads, 0, stream>>>(static_cast<const __half*>(w.data), static_cast<__half*>(out), n);
        else convert_kernel<__half, float><<<blocks_for(n), kThreads, 0, stream>>>(static_cast<const __half*>(w.data), static_cast<float*>(out), n);
    } else {
        if (out_half) convert_kernel<float, __half><<<blocks_for(n), kThreads, 0, stream>>>(static_cast<const float*>(w.data), static_cast<__half*>(out), n);
        else convert_kernel<float, float><<<blocks_for(n), kThreads, 0, stream>>>(static_cast<const float*>(w.data), static_cast<float*>(out), n);
    }
    return cudaGetLastError();
}

cudaError_t embed(cudaStream_t stream, const Mat& w, const uint32_t* tokens, Pos pos, float* out, uint32_t n_tokens) {
    if (n_tokens == 0) return cudaSuccess;
    dim3 grid(blocks_for(w.n_cols), n_tokens);
    Mat wm = w;
    void* args[] = {&wm, &tokens, &pos, &out};
    return launch_kernel((const void*)embed_kernel, grid, dim3(kThreads), 0, stream, args);
}

cudaError_t rms_norm(cudaStream_t stream, const float* x, const float* weight, float* out, uint32_t n_cols, uint32_t n_rows,
                     float eps) {
    if (n_rows == 0) return cudaSuccess;
    {
        cudaError_t launched = launch_dependent(rms_norm_kernel, dim3(n_rows), dim3(kThreads), 0, stream, x, weight, out, n_cols, eps);
        if (launched != cudaSuccess) return launched;
    }
    return cudaGetLastError();
}

cudaError_t norm_rope(cudaStream_t stream, const float* src, void* dst, bool dst_half, const float* weight, uint32_t n_heads,
                      uint32_t head_dim, uint32_t head_stride, uint32_t n_rot, uint32_t first_pos, uint32_t n_tokens,
                      uint32_t src_stride, uint32_t dst_stride, float theta, float eps) {
    if (n_tokens == 0 || n_heads == 0) return cudaSuccess;
    NormRopeParams p{src, dst, weight, n_heads, head_dim, head_stride, n_rot, first_pos, src_stride, dst_stride, theta, eps, dst_half ? 1 : 0};
    dim3 grid(n_heads, n_tokens);
    {
        cudaError_t launched = launch_dependent(norm_rope_kernel, grid, dim3(32), 0, stream, p);
        if (launched != cudaSuccess) return launched;
    }
    return cudaGetLastError();
}

cudaError_t convert_half(cudaStream_t stream, const float* src, __half* dst, uint64_t n) {
    if (n == 0) return cudaSuccess;
    {
        cudaError_t launched = launch_dependent(convert_kernel<float, __half>, dim3(blocks_for(n)), dim3(kThreads), 0, stream, src, dst, n);
        if (launched != cudaSuccess) return launched;
    }
    return cudaGetLastError();
}

cudaError_t copy_floats(cudaStream_t stream, const float* src, float* dst, uint64_t n) {
    if (n == 0) return cudaSuccess;
    return cudaMemcpyAsync(dst, src, n * sizeof(float), cudaMemcpyDeviceToDevice, stream);
}

cudaError_t silu_mul(cudaStream_t stream, float* x, const float* gate, uint64_t n) {
    if (n == 0) return cudaSuccess;
    silu_mul_kernel<<<blocks_for(n), kThreads, 0, stream>>>(x, gate, n);
    return cudaGetLastError();
}

cudaError_t short_conv(cudaStream_t stream, const float* bcx, const float* taps, float* history, float* out, uint32_t n_embd,
                       uint32_t kernel, uint32_t n_tokens, bool constant_taps, void* packed) {
    if (n_tokens == 0) return cudaSuccess;
    if (packed && n_embd % 64 != 0) return cudaErrorInvalidValue;
    if (kernel < 2 || kernel > 9) return cudaErrorInvalidValue;
    const uint32_t rows = packed ? ((n_tokens + 15u) & ~15u) : n_tokens;
    const bool wide = n_embd % 4 == 0 && ((uintptr_t)bcx | (uintptr_t)history | (uintptr_t)out) % 16 == 0;
    if (packed && !wide) return cudaErrorInvalidValue;
    auto launch = [&](auto conv, uint32_t per_thread, uint32_t run) {
        const uint32_t runs = (rows + run - 1) / run;
        return launch_dependent(conv, dim3((n_embd / per_thread + 127) / 128, runs < 65535u ? runs : 65535u), dim3(128), 0, stream, bcx, taps, history, out,
                                static_cast<__half*>(packed), n_embd, kernel, n_tokens, constant_taps);
    };
    if (kernel <= 4) return wide ? launch(short_conv_kernel<4, 4>, 4, 4) : launch(short_conv_kernel<4, 1>, 1, 4);
    return wide ? launch(short_conv_kernel<9, 4>, 4, 8) : launch(short_conv_kernel<9, 1>, 1, 8);
}

namespace {
cudaError_t launch_argmax(cudaStream_t stream, const float* x, uint32_t n, const ArgmaxOut& o) {
    if (n <= kArgmaxAlone) return launch_dependent(argmax_kernel<1>, dim3(1), dim3(kArgmaxThreads), 0, stream, x, n, o);
    return launch_clusters(argmax_kernel<kArgmaxCluster>, dim3(kArgmaxCluster), dim3(kArgmaxThreads), kArgmaxCluster, stream, x, n, o);
}
}  // namespace

cudaError_t argmax(cudaStream_t stream, const float* x, uint32_t n, uint32_t* out, uint32_t* readback) {
    const ArgmaxOut o{out, readback, nullptr, 0, nullptr, 0, nullptr, 1};
    return launch_argmax(stream, x, n, o);
}

cudaError_t argmax_step(cudaStream_t stream, const float* x, uint32_t n, uint32_t* counter, bool advance, uint32_t* tokens,
                        uint32_t offset, uint32_t* ring, uint32_t ring_slots) {
    const ArgmaxOut o{nullptr, nullptr, counter, advance ? 1 : 0, tokens, offset, ring, ring_slots ? ring_slots : 1};
    return launch_argmax(stream, x, n, o);
}

cudaError_t add_floats(cudaStream_t stream, float* y, const float* x, uint64_t n) {
    if (n == 0) return cudaSuccess;
    void* args[] = {&y, &x, &n};
    return launch_kernel((const void*)add_floats_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, args);
}

cudaError_t advance(cudaStream_t stream, uint32_t* counter) {
    void* args[] = {&counter};
    return launch_kernel((const void*)advance_kernel, dim3(1), dim3(1), 0, stream, args);
}

cudaError_t seed_step(cudaStream_t stream, const uint32_t* seed, uint32_t* counter, uint32_t* tokens) {
    return launch_dependent(seed_step_kernel, dim3(1), dim3(1), 0, stream, static_cast<const volatile uint32_t*>(seed), counter, tokens);
}

cudaError_t rope_table(cudaStream_t stream, float2* table, uint32_t n_positions, uint32_t n_rot, float theta) {
    const uint64_t items = (uint64_t)n_positions * (n_rot / 2);
    if (items == 0) return cudaSuccess;
    rope_table_kernel<<<(unsigned)((items + 255) / 256), 256, 0, stream>>>(table, n_positions, n_rot, theta);
    return cudaGetLastError();
}

cudaError_t rope_store_batch(cudaStream_t stream, const RopeBatch& p) {
    if (p.n_tokens == 0) return cudaSuccess;
    const uint32_t heads = p.n_heads + p.n_kv_heads + (p.v_dst ? p.n_kv_heads : 0);
    uint32_t parts = (uint32_t)(2 * sm_count()) / p.n_tokens, most = (heads + kRopeWarps - 1) / kRopeWarps;
    parts = parts < 1 ? 1 : parts > most ? most : parts;  // about two CTAs per SM at least, no CTA without a head per warp
    RopeBatch params = p;
    void* args[] = {&params};
    return launch_kernel((const void*)rope_store_batch_kernel, dim3(p.n_tokens, parts), dim3(32 * kRopeWarps), 0, stream, args);
}

cudaError_t rope_store(cudaStream_t stream, const RopeStore& p, Pos pos) {
    RopeStore params = p;
    void* args[] = {&params, &pos};
    return launch_kernel((const void*)rope_store_kernel, dim3(p.n_heads + 2 * p.n_kv_heads), dim3(32), 0, stream, args);
}

}  // namespace k
}  // namespace bc
