// Qwen3.5 kernels: the Gated DeltaNet layer (causal convolution, gates, the delta-rule recurrence,
// the gated output norm) and the sigmoid output gate of Qwen's attention layers.
// Counterparts: crates/bobcat-metal/src/gdn.metal (gdn_conv :14, gdn_gated_norm :106, gdn_gates :132,
// gdn_qk_norm :181, gdn_recurrence :222, attention_gate :307); the arithmetic they must reproduce is
// crates/bobcat/src/qwen35.rs:430-516 and :754-778, f32 throughout and in the reference's order.

#include <cstdlib>

#include "async_utils.cuh"
#include "device_utils.cuh"
#include "kernels.h"

namespace bc {
namespace k {

namespace {

// beta = sigmoid(beta); decay = exp(a * softplus(alpha + dt_bias)), softplus(x) = x above 20
// (qwen35.rs:479-481, :776-778). In place over [n_tokens][n_v_heads]; alpha receives the decay.
__device__ __forceinline__ void gate_pair(float* __restrict__ beta, float* __restrict__ alpha, const float* __restrict__ a,
                                          const float* __restrict__ dt_bias, uint32_t n_v_heads, uint32_t i) {
    const uint32_t head = i % n_v_heads;
    beta[i] = 1.f / (1.f + expf(-beta[i]));
    const float v = alpha[i] + dt_bias[head];
    const float sp = v > 20.f ? v : log1pf(expf(v));
    alpha[i] = expf(a[head] * sp);
}

__global__ void gdn_gates_kernel(float* __restrict__ beta, float* __restrict__ alpha, const float* __restrict__ a,
                                 const float* __restrict__ dt_bias, uint32_t n_v_heads, uint32_t n) {
    pdl_launch_dependents();
    pdl_wait();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) gate_pair(beta, alpha, a, dt_bias, n_v_heads, i);
}

struct RecurrenceParams {
    const float* qkv;    // [n_tokens][2 * key_dim + value_dim]: q heads, k heads, v heads (after the conv)
    const float* beta;   // [n_tokens][n_v_heads]
    const float* decay;  // [n_tokens][n_v_heads]
    float* state;        // [n_v_heads][k_dim][v_dim]
    float* out;          // [n_tokens][n_v_heads * v_dim]
    uint32_t n_k_heads, n_v_heads, k_dim, v_dim, n_tokens;
    int normalize;       // L2-normalise q (times 1/sqrt(k_dim)) and k here, as decode does
};

// l2_normalize of one head's q or k (qwen35.rs:762-768), element e * 32 + lane in `x[e]`: the sum of
// squares is taken per run of 32 elements across the warp and the runs are added in order, which
// is the order gdn_step_kernel takes (there a warp holds one run), so a batch and single steps
// normalise to the same bits. Returns the factor 1 / sqrt(sum + 1e-6).
template <int PER>
__device__ __forceinline__ float l2_factor(const float (&x)[PER]) {
    float sum = 0.f;
#pragma unroll
    for (int e = 0; e < PER; ++e) sum += warp_sum(x[e] * x[e]);
    return 1.0f / sqrtf(sum + 1e-6f);
}

// The causal convolution with SiLU over a batch. x and out are [n_tokens][conv_dim]; taps are [conv_dim][kernel],
// oldest first; history is [conv_dim][kernel - 1] raw inputs, oldest first. The sum starts from the newest tap's term
// and adds the earlier inputs oldest first (qwen35.rs:449-461), from the batch or, for its first tokens, from the
// history, so any split into batches gives the same bits. kernel <= K.
//
// A warp takes 32 * PER neighbouring channels of R tokens, a lane channels e * 32 + lane, with the window of inputs in
// registers. With `n_norm` the first n_norm groups of channels are q heads, then k heads: their outputs are also
// L2-normalised here (q scaled by 1 / sqrt(head size)), which is why a warp holds a whole head. CTAs past the
// convolution's compute the gates. Only the first run of tokens reads the history (R >= K - 1); its threads
// rewrite it. Bound by L2 traffic and latency: 512 tokens of 8192 channels took 44 us for the convolution (a thread per
// element that read its inputs `kernel` times), 4.1 for the norms, 2.4 for the history and 2.0 for the gates in four
// launches, now 14.9 in one; 64 tokens of 6144 channels 13.7, now 8.4.
struct ConvParams {
    const float *x, *taps;
    float *history, *out;
    uint32_t conv_dim, kernel, n_tokens, n_norm, conv_ctas;
    float *beta, *alpha;  // gates: with n_gates
    const float *a, *dt_bias;
    uint32_t n_v_heads, n_gates;
    bool constant_taps;  // a model's: read ahead of the wait. An op call's are read after it: its recording may write them
};

template <int PER, int K, int R>
__global__ void __launch_bounds__(256) gdn_conv_kernel(const __grid_constant__ ConvParams p) {
    static_assert(R >= K - 1, "only the first run may read the history");
    pdl_launch_dependents();
    if (blockIdx.x >= p.conv_ctas) {
        pdl_wait();
        const uint32_t i = (blockIdx.x - p.conv_ctas) * blockDim.x + threadIdx.x;
        if (i < p.n_gates) gate_pair(p.beta, p.alpha, p.a, p.dt_bias, p.n_v_heads, i);
        return;
    }
    const uint32_t lane = threadIdx.x & 31, n_groups = (p.conv_dim + 32 * PER - 1) / (32 * PER), skip = K - p.kernel;
    const uint64_t item = (uint64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const uint32_t group = (uint32_t)(item % n_groups), t0 = (uint32_t)(item / n_groups) * R;
    if (t0 >= p.n_tokens) return;
    const uint32_t c0 = group * 32 * PER + lane;
    if (!p.constant_taps) pdl_wait();
    float tap[PER][K], window[PER][K - 1 + R];  // inputs of tokens t0 - (K - 1) .. t0 + R - 1
#pragma unroll
    for (int e = 0; e < PER; ++e) {
        const uint32_t c = c0 + e * 32;
#pragma unroll
        for (int i = 0; i < K; ++i) tap[e][i] = i >= (int)skip && c < p.conv_dim ? p.taps[(uint64_t)c * p.kernel + i - skip] : 0.f;
    }
    pdl_wait();
#pragma unroll
    for (int i = 0; i < K - 1 + R; ++i) {
        const int64_t src = (int64_t)t0 - (K - 1) + i;
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const uint32_t c = c0 + e * 32;
            window[e][i] = 0.f;
            if (c >= p.conv_dim || i < (int)skip) continue;
            if (src < 0) window[e][i] = p.history[(uint64_t)c * (p.kernel - 1) + i - skip];
            else if (src < (int64_t)p.n_tokens) window[e][i] = p.x[(uint64_t)src * p.conv_dim + c];
        }
    }
    // The history after the batch: slot i holds the input of token n_tokens - (kernel - 1) + i, or an older slot when the
    // batch is shorter than the history. Read here, beside the window, and written at the end by the first run's threads.
    float kept[PER][K - 1];
    if (t0 == 0) {
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const uint32_t c = c0 + e * 32;
#pragma unroll
            for (int i = 0; i < K - 1; ++i) {
                if (c >= p.conv_dim || i < (int)skip) continue;
                const int64_t src = (int64_t)p.n_tokens - (K - 1) + i;
                kept[e][i] = src >= 0 ? p.x[(uint64_t)src * p.conv_dim + c] : p.history[(uint64_t)c * (p.kernel - 1) + src + (K - 1) - skip];
            }
        }
    }
    // All tokens of the run at once: their sums over the warp are independent. (Rows past the batch are zeros and not stored.)
    float v[R][PER];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            float sum = tap[e][K - 1] * window[e][K - 1 + r];
#pragma unroll
            for (int i = 0; i < K - 1; ++i)
                if (i >= (int)skip) sum += tap[e][i] * window[e][i + r];
            v[r][e] = sum / (1.f + expf(-sum));
        }
    if (group < p.n_norm) {
        float squares[R][PER];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int e = 0; e < PER; ++e) squares[r][e] = v[r][e] * v[r][e];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int e = 0; e < PER; ++e) squares[r][e] += __shfl_xor_sync(0xffffffffu, squares[r][e], o);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            float sum = 0.f;  // l2_factor's sum
#pragma unroll
            for (int e = 0; e < PER; ++e) sum += squares[r][e];
            float factor = 1.0f / sqrtf(sum + 1e-6f);
            if (group < p.n_norm / 2) factor = (1.0f / sqrtf((float)(32 * PER))) * factor;
#pragma unroll
            for (int e = 0; e < PER; ++e) v[r][e] *= factor;
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (t0 + r >= p.n_tokens) break;
#pragma unroll
        for (int e = 0; e < PER; ++e)
            if (c0 + e * 32 < p.conv_dim) p.out[(uint64_t)(t0 + r) * p.conv_dim + c0 + e * 32] = v[r][e];
    }
    if (t0 != 0) return;
#pragma unroll
    for (int e = 0; e < PER; ++e)
#pragma unroll
        for (int i = 0; i < K - 1; ++i)
            if (c0 + e * 32 < p.conv_dim && i >= (int)skip) p.history[(uint64_t)(c0 + e * 32) * (p.kernel - 1) + i - skip] = kept[e][i];
}

// The delta rule over a run of tokens. One warp (a CTA of its own) per 8 state columns of a value
// head; four neighbouring lanes share a column, each holding a quarter of its k_dim state values in
// registers for the whole run. Per token (qwen35.rs:483-506): S *= decay; r = sum_i S[i] k_i;
// delta = (v - r) beta; S[i] += k_i delta; o = sum_i S[i] q_i. A lane sums its quarter as two
// interleaved partial sums and the quarters are added in order - the arithmetic of
// gdn_step_kernel, so a batch and single steps walk the same values. Value head h reads key head
// h % n_k_heads. A column's recurrence needs nothing of the other columns, so the warps share no
// state and meet at no barrier: each stages (and, when asked, normalises) the token's q and k for
// itself. A head spreads over v_dim / 8 warps, and a token is a chain of k_dim / 4 multiply-adds;
// the earlier form (a CTA per head, a thread per column with all k_dim values, two block barriers
// per token) took 1.45 us per token.
constexpr uint32_t kRecurrenceWarps = 4;  // independent warps per CTA, one per SM partition

template <int KDIM>
__global__ void __launch_bounds__(32 * kRecurrenceWarps) gdn_recurrence_kernel(RecurrenceParams p) {
    constexpr int PER = KDIM / 32;   // elements of q and of k a lane brings in
    constexpr int MINE = KDIM / 4;   // state values of its column a lane holds
    static_assert(KDIM % 32 == 0 && MINE % 4 == 0, "k_dim");
    // A token's inputs come through a ring of kAhead + 1 slots of shared memory, copied
    // (cp.async) kAhead tokens ahead: a token that loaded its successor's inputs into registers
    // and handed them on lasted one trip to memory, however little it computed.
    constexpr int kAhead = 7, kSlots = kAhead + 1;
    // A quarter of q (of k) is followed by four floats of padding, so the four quarters that a
    // warp's lanes read at once lie in different banks.
    struct Slot {
        float q[KDIM + 16], k[KDIM + 16], v[8], beta, decay, pad[2];
    };
    auto at = [](uint32_t e) { return e + 4 * (e / MINE); };
    __shared__ __align__(16) Slot rings[kRecurrenceWarps][kSlots];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t vd = p.v_dim, groups = (vd + 7) / 8;
    const uint32_t unit = blockIdx.x * kRecurrenceWarps + (threadIdx.x >> 5);  // (head, group of 8 columns)
    if (unit >= p.n_v_heads * groups) return;  // whole warps; the warps of a CTA never meet
    Slot* ring = rings[threadIdx.x >> 5];
    const uint32_t head = unit / groups, lane = threadIdx.x & 31, part = lane & 3, first_lane = lane & ~3u;
    const uint32_t column = lane >> 2, j = (unit % groups) * 8 + column;
    const uint32_t key_head = head % p.n_k_heads;
    const uint32_t key_dim = p.n_k_heads * KDIM, conv_dim = 2 * key_dim + p.n_v_heads * vd;
    float* state = p.state + (uint64_t)head * KDIM * vd + (uint64_t)part * MINE * vd;
    float S[MINE];
    if (j < vd) {
#pragma unroll
        for (int i = 0; i < MINE; ++i) S[i] = state[(uint64_t)i * vd + j];
    }
    // Lane l brings elements e * 32 + l of q and of k; the first lane of a column its v; lanes 1 and 2 the gates.
    auto bring = [&](uint32_t t) {
        if (t < p.n_tokens) {
            Slot& slot = ring[t % kSlots];
            const float* row = p.qkv + (uint64_t)t * conv_dim;
#pragma unroll
            for (int e = 0; e < PER; ++e) {
                async::cp_async_4(async::smem_u32(&slot.q[at(e * 32 + lane)]), row + key_head * KDIM + e * 32 + lane);
                async::cp_async_4(async::smem_u32(&slot.k[at(e * 32 + lane)]), row + key_dim + key_head * KDIM + e * 32 + lane);
            }
            if (part == 0 && j < vd) async::cp_async_4(async::smem_u32(&slot.v[column]), row + 2 * key_dim + head * vd + j);
            if (lane == 1) async::cp_async_4(async::smem_u32(&slot.beta), p.beta + (uint64_t)t * p.n_v_heads + head);
            if (lane == 2) async::cp_async_4(async::smem_u32(&slot.decay), p.decay + (uint64_t)t * p.n_v_heads + head);
        }
        async::cp_async_commit();
    };
#pragma unroll
    for (int t = 0; t < kAhead; ++t) bring((uint32_t)t);
    for (uint32_t t = 0; t < p.n_tokens; ++t) {
        __syncwarp();  // every lane is through with the slot the next copy overwrites (the previous token's)
        bring(t + kAhead);
        async::cp_async_wait<kAhead>();  // all but the newest kAhead groups: this token's bytes are in
        __syncwarp();
        Slot& slot = ring[t % kSlots];
        if (p.normalize) {
            float q[PER], k[PER];
#pragma unroll
            for (int e = 0; e < PER; ++e) {
                q[e] = slot.q[at(e * 32 + lane)];
                k[e] = slot.k[at(e * 32 + lane)];
            }
            const float q_scale = (1.0f / sqrtf((float)KDIM)) * l2_factor<PER>(q), k_scale = l2_factor<PER>(k);
#pragma unroll
            for (int e = 0; e < PER; ++e) {
                slot.q[at(e * 32 + lane)] = q[e] * q_scale;
                slot.k[at(e * 32 + lane)] = k[e] * k_scale;
            }
            __syncwarp();
        }
        const float decay = slot.decay, beta = slot.beta, v = j < vd ? slot.v[column] : 0.f;
        // Every lane takes part in the shuffles; lanes past the last column carry zeros.
        const float4* k4 = reinterpret_cast<const float4*>(slot.k + part * (MINE + 4));
        const float4* q4 = reinterpret_cast<const float4*>(slot.q + part * (MINE + 4));
        float r0 = 0.f, r1 = 0.f;
        if (j < vd) {
#pragma unroll
            for (int i = 0; i < MINE / 4; ++i) {
                const float4 kk = k4[i];
                S[4 * i] *= decay;
                S[4 * i + 1] *= decay;
                S[4 * i + 2] *= decay;
                S[4 * i + 3] *= decay;
                r0 += S[4 * i] * kk.x + S[4 * i + 2] * kk.z;
                r1 += S[4 * i + 1] * kk.y + S[4 * i + 3] * kk.w;
            }
        }
        const float r_part = r0 + r1;
        float r = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) r += __shfl_sync(0xffffffffu, r_part, first_lane + q);  // the quarters in order
        const float delta = (v - r) * beta;
        float o0 = 0.f, o1 = 0.f;
        if (j < vd) {
#pragma unroll
            for (int i = 0; i < MINE / 4; ++i) {
                const float4 kk = k4[i], qq = q4[i];
                S[4 * i] += kk.x * delta;
                S[4 * i + 1] += kk.y * delta;
                S[4 * i + 2] += kk.z * delta;
                S[4 * i + 3] += kk.w * delta;
                o0 += S[4 * i] * qq.x + S[4 * i + 2] * qq.z;
                o1 += S[4 * i + 1] * qq.y + S[4 * i + 3] * qq.w;
            }
        }
        const float o_part = o0 + o1;
        float out = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) out += __shfl_sync(0xffffffffu, o_part, first_lane + q);
        if (j < vd && part == 0) p.out[(uint64_t)t * p.n_v_heads * vd + head * vd + j] = out;
    }
    async::cp_async_wait<0>();
    if (j < vd) {
#pragma unroll
        for (int i = 0; i < MINE; ++i) state[(uint64_t)i * vd + j] = S[i];
    }
}

// One warp per (token, value head): x = RMSNorm(x) * weight * silu(z) (qwen35.rs:508-513).
__global__ void __launch_bounds__(256) gdn_gated_norm_kernel(float* __restrict__ x, const float* __restrict__ z, const float* __restrict__ weight,
                                                             uint32_t v_dim, uint32_t n_rows, float eps) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31, index = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (index >= n_rows) return;
    float* row = x + (uint64_t)index * v_dim;
    const float* gate = z + (uint64_t)index * v_dim;
    float sumsq = 0.f;
    for (uint32_t d = lane; d < v_dim; d += 32) sumsq += row[d] * row[d];
    sumsq = warp_sum(sumsq);
    const float scale = rsqrtf(sumsq / (float)v_dim + eps);
    for (uint32_t d = lane; d < v_dim; d += 32) {
        float g = gate[d];
        row[d] = weight[d] * (row[d] * scale) * (g / (1.f + expf(-g)));
    }
}

// The same with the result as the fp16 operand of the product that follows (kernels_matmul_umma.cu's pack_kernel), rows up to
// the next multiple of 16 tokens zero. LANES = v_dim / 8 lanes share a row, each with one 16-byte output. Bound by L2
// traffic: 512 tokens of 32 heads of 128 took 17.0 us with one warp per CTA and 3.8 for the packing, now 5.9; 64
// tokens of 16 heads 4.2 + 2.1, now 4.2.
template <int LANES>
__global__ void __launch_bounds__(256) gdn_gated_norm_pack_kernel(const float* __restrict__ x, const float* __restrict__ z, const float* __restrict__ weight,
                                                                  __half* __restrict__ packed, uint32_t n_heads, uint32_t n_tokens, uint32_t token_groups,
                                                                  float eps) {
    constexpr uint32_t kDim = LANES * 8;
    pdl_launch_dependents();
    const uint32_t i = threadIdx.x % LANES, index = blockIdx.x * (256 / LANES) + threadIdx.x / LANES;
    const uint32_t token = index / n_heads, head = index % n_heads;
    const uint32_t d = (i >> 3) * 64 + ((i >> 2) & 1) * 32 + 4 * (i & 3);  // elements d .. d + 3 and d + 16 .. d + 19 of the head
    const float4 wl = __ldg(reinterpret_cast<const float4*>(weight + d)), wh = __ldg(reinterpret_cast<const float4*>(weight + d + 16));
    pdl_wait();
    float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo, gl = lo, gh = lo;
    if (token < n_tokens) {
        const uint64_t at = ((uint64_t)token * n_heads + head) * kDim + d;
        lo = *reinterpret_cast<const float4*>(x + at), hi = *reinterpret_cast<const float4*>(x + at + 16);
        gl = *reinterpret_cast<const float4*>(z + at), gh = *reinterpret_cast<const float4*>(z + at + 16);
    }
    float sumsq = (lo.x * lo.x + lo.y * lo.y + lo.z * lo.z + lo.w * lo.w) + (hi.x * hi.x + hi.y * hi.y + hi.z * hi.z + hi.w * hi.w);
#pragma unroll
    for (int o = 1; o < LANES; o <<= 1) sumsq += __shfl_xor_sync(0xffffffffu, sumsq, o);
    const float scale = rsqrtf(sumsq / (float)kDim + eps);
    auto value = [&](float v, float w, float g) { return w * (v * scale) * (g / (1.f + expf(-g))); };
    const __half2 p0 = __floats2half2_rn(value(lo.x, wl.x, gl.x), value(lo.z, wl.z, gl.z)), p1 = __floats2half2_rn(value(lo.y, wl.y, gl.y), value(lo.w, wl.w, gl.w));
    const __half2 p2 = __floats2half2_rn(value(hi.x, wh.x, gh.x), value(hi.z, wh.z, gh.z)), p3 = __floats2half2_rn(value(hi.y, wh.y, gh.y), value(hi.w, wh.w, gh.w));
    if (token < token_groups * 8)
        *reinterpret_cast<uint4*>(packed + packed_operand_index(token, head * kDim + d, token_groups)) =
            make_uint4(*reinterpret_cast<const uint32_t*>(&p0), *reinterpret_cast<const uint32_t*>(&p1), *reinterpret_cast<const uint32_t*>(&p2),
                       *reinterpret_cast<const uint32_t*>(&p3));
}

// ---- One token through a whole DeltaNet mixer in one launch (decode): the causal convolution
// with SiLU and its history shift, the gates, the L2 norms of q and k, the delta rule on the state
// and the gated RMSNorm of the output, i.e. gdn_conv + gdn_gates + gdn_recurrence + gdn_gated_norm
// for n_tokens == 1 (qwen35.rs:430-516). One CTA per key head; it serves the value heads that read
// that key head (h = key_head + m * n_k_heads), one thread per state column of each, so the
// convolution of q and k happens once and nothing races on its history.
struct StepParams {
    const float* qkv;      // [conv_dim] projections before the convolution: q heads, k heads, v heads
    const float* taps;     // [conv_dim][kernel]
    float* history;        // [conv_dim][kernel - 1]
    const float* beta;     // [n_v_heads] before the sigmoid
    const float* alpha;    // [n_v_heads] before the softplus
    const float* a;        // [n_v_heads]
    const float* dt_bias;  // [n_v_heads]
    float* state;          // [n_v_heads][k_dim][v_dim]
    const float* z;        // [n_v_heads * v_dim]
    const float* norm_weight;  // [v_dim]
    float* out;            // [n_v_heads * v_dim]
    uint32_t n_k_heads, n_v_heads, k_dim, v_dim, kernel;
    float eps;
};

constexpr int kStepParts = 4;   // threads that share a state column, each holding a quarter of its rows, when a CTA serves a key head
constexpr uint32_t kStepRanks = 4;  // CTAs that share a key head where its columns allow it

// The convolution of one channel for one token (same order of additions as gdn_conv) and the shifted history, which the
// caller stores when nobody reads the old one any more.
struct ConvStep {
    float value, next[7];
};
__device__ __forceinline__ ConvStep conv_step(const StepParams& p, uint32_t channel) {
    const uint32_t H = p.kernel - 1;
    const float* tap = p.taps + (uint64_t)channel * p.kernel;
    const float* hist = p.history + (uint64_t)channel * H;
    const float input = p.qkv[channel];
    float past[7], taps[8];
#pragma unroll
    for (uint32_t i = 0; i < 7; ++i) {
        past[i] = i < H ? hist[i] : 0.f;
        taps[i] = i < H ? tap[i] : 0.f;
    }
    float sum = tap[H] * input;
    ConvStep c;
#pragma unroll
    for (uint32_t i = 0; i < 7; ++i) {
        if (i < H) sum += taps[i] * past[i];
        c.next[i] = i + 1 < H && i < 6 ? past[i < 6 ? i + 1 : 6] : input;
    }
    c.value = sum / (1.f + expf(-sum));
    return c;
}
__device__ __forceinline__ void keep_history(const StepParams& p, uint32_t channel, const ConvStep& c) {
    const uint32_t H = p.kernel - 1;
    float* hist = p.history + (uint64_t)channel * H;
#pragma unroll
    for (uint32_t i = 0; i < 7; ++i)
        if (i < H) hist[i] = c.next[i];
}

// ROWS rows of a state column to a thread, up to COLUMNS columns to a CTA. `ranks` CTAs (a cluster) share the columns of a key head's value heads: the state
// is 4 MB of traffic, which one CTA per key head (16 of them) moved in 11.6 us; with four it is on 64 SMs, is asked for
// in L2 before the wait for the preceding launch, and takes 7.4 us. Every CTA convolves q and k for itself; the first
// one stores their history when all have read it. A value head's sum of squares meets through distributed shared memory.
template <int KDIM, int ROWS, int COLUMNS>
__global__ void __launch_bounds__(1024) gdn_step_kernel(const __grid_constant__ StepParams p, uint32_t ranks) {
    // Thread (part, column): rows [part * ROWS, (part + 1) * ROWS) of a column of the state of value head
    // key_head + m * n_k_heads. The rows are loaded into registers first of all, so that read overlaps the convolution;
    // the parts' partial dot products meet in shared memory.
    constexpr int kParts = KDIM / ROWS;
    __shared__ __align__(16) float qs[KDIM], ks[KDIM];
    __shared__ float scratch[96];
    __shared__ float r_part[kParts][COLUMNS], o_part[kParts][COLUMNS], v_full[COLUMNS];
    __shared__ float head_squares;  // of this CTA's columns, where a value head spans several CTAs
    pdl_launch_dependents();
    const uint32_t rank = blockIdx.x % ranks, key_head = blockIdx.x / ranks, tid = threadIdx.x, vd = p.v_dim;
    const uint32_t lane = tid & 31, warp = tid >> 5;
    const uint32_t key_dim = p.n_k_heads * KDIM, columns = p.n_v_heads / p.n_k_heads * vd / ranks;
    const uint32_t column_id = tid % columns, part = tid / columns;  // blockDim.x == kParts * columns
    const uint32_t m = (rank * columns + column_id) / vd, j = (rank * columns + column_id) % vd, head = key_head + m * p.n_k_heads;
    float* column = p.state + (uint64_t)head * KDIM * vd + (uint64_t)(part * ROWS) * vd + j;
    if (lane == 0) {  // a warp's 32 columns of a row are a line (a hint: what is in flight is still seen)
#pragma unroll
        for (int i = 0; i < ROWS; ++i) asm volatile("prefetch.global.L2 [%0];" ::"l"(column + (uint64_t)i * vd));
    }
    pdl_wait();
    float S[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) S[i] = column[(uint64_t)i * vd];
    // q and k of this key head: threads below KDIM convolve one channel of each. The column's element of v: part 0.
    ConvStep qc{}, kc{}, vc{};
    if (tid < KDIM) {
        qc = conv_step(p, key_head * KDIM + tid);
        kc = conv_step(p, key_dim + key_head * KDIM + tid);
    }
    if (part == 0) {
        vc = conv_step(p, 2 * key_dim + head * vd + j);
        keep_history(p, 2 * key_dim + head * vd + j, vc);
        v_full[column_id] = vc.value;  // where every part can read it
    }
    const float qv = qc.value, kv = kc.value;
    // l2_normalize (qwen35.rs:762-768): f32 sum of squares, x *= scale / sqrt(sum + 1e-6).
    const float q2 = warp_sum(qv * qv), k2 = warp_sum(kv * kv);
    if (lane == 0) {
        scratch[warp] = q2;
        scratch[32 + warp] = k2;
    }
    // beta = sigmoid(beta); decay = exp(a * softplus(alpha + dt_bias)), softplus(x) = x above 20.
    const float braw = p.beta[head], araw = p.alpha[head] + p.dt_bias[head];
    const float beta = 1.f / (1.f + expf(-braw));
    const float decay = expf(p.a[head] * (araw > 20.f ? araw : log1pf(expf(araw))));
    const float gate = part == 0 ? p.z[head * vd + j] : 0.f, norm_weight = part == 0 ? p.norm_weight[j] : 0.f;
    __syncthreads();
    if (tid < KDIM) {
        float qsum = 0.f, ksum = 0.f;
        for (uint32_t w = 0; w < (KDIM + 31) / 32; ++w) {
            qsum += scratch[w];
            ksum += scratch[32 + w];
        }
        qs[tid] = qv * ((1.0f / sqrtf((float)KDIM)) / sqrtf(qsum + 1e-6f));
        ks[tid] = kv * (1.0f / sqrtf(ksum + 1e-6f));
    }
    __syncthreads();
    const float4* k4 = reinterpret_cast<const float4*>(ks + part * ROWS);
    const float4* q4 = reinterpret_cast<const float4*>(qs + part * ROWS);
    float r0 = 0.f, r1 = 0.f;
#pragma unroll
    for (int i = 0; i < ROWS / 4; ++i) {
        const float4 kk = k4[i];
        S[4 * i] *= decay;
        S[4 * i + 1] *= decay;
        S[4 * i + 2] *= decay;
        S[4 * i + 3] *= decay;
        r0 += S[4 * i] * kk.x + S[4 * i + 2] * kk.z;
        r1 += S[4 * i + 1] * kk.y + S[4 * i + 3] * kk.w;
    }
    r_part[part][column_id] = r0 + r1;
    __syncthreads();
    float r = 0.f;
#pragma unroll
    for (int q = 0; q < kParts; ++q) r += r_part[q][column_id];  // every part adds them in the same order
    const float delta = (v_full[column_id] - r) * beta;
    float o0 = 0.f, o1 = 0.f;
#pragma unroll
    for (int i = 0; i < ROWS / 4; ++i) {
        const float4 kk = k4[i], qq = q4[i];
        S[4 * i] += kk.x * delta;
        S[4 * i + 1] += kk.y * delta;
        S[4 * i + 2] += kk.z * delta;
        S[4 * i + 3] += kk.w * delta;
        o0 += S[4 * i] * qq.x + S[4 * i + 2] * qq.z;
        o1 += S[4 * i + 1] * qq.y + S[4 * i + 3] * qq.w;
    }
    o_part[part][column_id] = o0 + o1;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ROWS; ++i) column[(uint64_t)i * vd] = S[i];
    // Gated RMSNorm over each value head's v_dim outputs, by the part-0 threads (v_dim is a multiple
    // of 32, so a warp belongs to one head): out = weight * (o * scale) * silu(z).
    float o = 0.f;
    if (part == 0) {
#pragma unroll
        for (int q = 0; q < kParts; ++q) o += o_part[q][column_id];
    }
    const float sq = warp_sum(o * o);
    if (lane == 0) scratch[64 + warp] = sq;
    __syncthreads();
    const bool spans = vd > columns;  // a value head's columns lie in vd / columns CTAs
    float sumsq = 0.f;
    {
        const uint32_t warps_here = (spans ? columns : vd) / 32, first = spans ? 0 : (column_id / vd) * warps_here;
        for (uint32_t w = 0; w < warps_here; ++w) sumsq += scratch[64 + first + w];
    }
    if (ranks > 1) {
        if (tid == 0) head_squares = sumsq;
        asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
        if (spans) {
            const uint32_t per_head = vd / columns, first = rank / per_head * per_head;
            sumsq = 0.f;
            for (uint32_t c = 0; c < per_head; ++c) {
                uint32_t at;
                float other;
                asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(&head_squares)), "r"(first + c));
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(other) : "r"(at) : "memory");
                sumsq += other;
            }
        }
    }
    if (rank == 0 && tid < KDIM) {  // every CTA of the cluster has read the old history
        keep_history(p, key_head * KDIM + tid, qc);
        keep_history(p, key_dim + key_head * KDIM + tid, kc);
    }
    if (part == 0) {
        const float scale = rsqrtf(sumsq / (float)vd + p.eps);
        p.out[head * vd + j] = norm_weight * (o * scale) * (gate / (1.f + expf(-gate)));
    }
    if (ranks > 1) asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");  // its sums may still be read
}

// out[t][h][d] *= sigmoid(gate) with the gate read from the interleaved q projection:
// q_gate[t][h][head_dim + d] of [n_tokens][n_heads][2 * head_dim] (qwen35.rs:383-390, :422-424).
__global__ void attention_gate_kernel(float* __restrict__ out, const float* __restrict__ q_gate, uint32_t n_heads, uint32_t head_dim,
                                      uint64_t n) {
    pdl_launch_dependents();
    pdl_wait();
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t d = i % head_dim;
    uint64_t th = i / head_dim;  // token * n_heads + head
    float g = q_gate[th * 2 * head_dim + head_dim + d];
    out[i] *= 1.f / (1.f + expf(-g));
}

}  // namespace

template <int PER>
cudaError_t launch_conv(cudaStream_t stream, ConvParams& p) {
    // Runs of 8 tokens read 1.4 times what they must, runs of 4 1.75 times: the short ones while the long ones would leave
    // fewer than 16 warps to an SM.
    const uint32_t groups = (p.conv_dim + 32 * PER - 1) / (32 * PER);
    const bool brief = p.kernel <= 4 && (uint64_t)groups * ((p.n_tokens + 7) / 8) < (uint64_t)sm_count() * 16;
    const uint32_t run = brief ? 4 : 8;
    p.conv_ctas = (uint32_t)(((uint64_t)groups * ((p.n_tokens + run - 1) / run) + 7) / 8);
    void* args[] = {&p};
    const void* kernel = p.kernel > 4 ? (const void*)gdn_conv_kernel<PER, 8, 8> : brief ? (const void*)gdn_conv_kernel<PER, 4, 4> : (const void*)gdn_conv_kernel<PER, 4, 8>;
    return launch_kernel(kernel, dim3(p.conv_ctas + (p.n_gates + 255) / 256), dim3(256), 0, stream, args);
}

cudaError_t gdn_conv(cudaStream_t stream, const float* x, const float* taps, float* history, float* out, uint32_t conv_dim,
                     uint32_t kernel, uint32_t n_tokens) {
    if (n_tokens == 0) return cudaSuccess;
    ConvParams p{x, taps, history, out, conv_dim, kernel, n_tokens, 0, 0, nullptr, nullptr, nullptr, nullptr, 1, 0, false};
    return launch_conv<4>(stream, p);
}

cudaError_t gdn_conv_gates(cudaStream_t stream, const float* x, const float* taps, float* history, float* out, float* beta, float* alpha, const float* a,
                           const float* dt_bias, uint32_t n_k_heads, uint32_t n_v_heads, uint32_t k_dim, uint32_t v_dim, uint32_t kernel, uint32_t n_tokens) {
    if (n_tokens == 0) return cudaSuccess;
    ConvParams p{x, taps, history, out, 2 * n_k_heads * k_dim + n_v_heads * v_dim, kernel, n_tokens, 2 * n_k_heads, 0, beta, alpha, a, dt_bias, n_v_heads,
                 n_v_heads * n_tokens, true};
    switch (k_dim) {
        case 32: return launch_conv<1>(stream, p);
        case 64: return launch_conv<2>(stream, p);
        case 96: return launch_conv<3>(stream, p);
        default: return launch_conv<4>(stream, p);
    }
}

cudaError_t gdn_gates(cudaStream_t stream, float* beta, float* alpha, const float* a, const float* dt_bias, uint32_t n_v_heads,
                      uint32_t n_tokens) {
    uint32_t n = n_v_heads * n_tokens;
    if (n == 0) return cudaSuccess;
    void* args[] = {&beta, &alpha, &a, &dt_bias, &n_v_heads, &n};
    return launch_kernel((const void*)gdn_gates_kernel, dim3((n + 127) / 128), dim3(128), 0, stream, args);
}

cudaError_t gdn_recurrence(cudaStream_t stream, const float* qkv, const float* beta, const float* decay, float* state, float* out,
                           uint32_t n_k_heads, uint32_t n_v_heads, uint32_t k_dim, uint32_t v_dim, uint32_t n_tokens, bool normalize) {
    if (n_tokens == 0) return cudaSuccess;
    RecurrenceParams p{qkv, beta, decay, state, out, n_k_heads, n_v_heads, k_dim, v_dim, n_tokens, normalize ? 1 : 0};
    void* args[] = {&p};
    // A warp per 8 state columns of a head.
    const void* kernel = k_dim == 32 ? (const void*)gdn_recurrence_kernel<32> : k_dim == 64 ? (const void*)gdn_recurrence_kernel<64>
                       : k_dim == 96 ? (const void*)gdn_recurrence_kernel<96> : (const void*)gdn_recurrence_kernel<128>;
    const uint32_t units = n_v_heads * ((v_dim + 7) / 8);
    return launch_kernel(kernel, dim3((units + kRecurrenceWarps - 1) / kRecurrenceWarps), dim3(32 * kRecurrenceWarps), 0, stream, args);
}

bool gdn_step_supported(uint32_t n_k_heads, uint32_t n_v_heads, uint32_t k_dim, uint32_t v_dim, uint32_t kernel) {
    if (n_k_heads == 0 || n_v_heads % n_k_heads != 0 || kernel < 2 || kernel > 8) return false;
    if (k_dim != 32 && k_dim != 64 && k_dim != 96 && k_dim != 128) return false;
    const uint32_t columns = (n_v_heads / n_k_heads) * v_dim;  // state columns a CTA serves
    return v_dim % 32 == 0 && columns <= 256 && kStepParts * columns >= k_dim;
}

cudaError_t gdn_step(cudaStream_t stream, const float* qkv, const float* taps, float* history, const float* beta, const float* alpha,
                     const float* a, const float* dt_bias, float* state, const float* z, const float* norm_weight, float* out,
                     uint32_t n_k_heads, uint32_t n_v_heads, uint32_t k_dim, uint32_t v_dim, uint32_t kernel, float eps) {
    StepParams p{qkv, taps, history, beta, alpha, a, dt_bias, state, z, norm_weight, out, n_k_heads, n_v_heads, k_dim, v_dim, kernel, eps};
    const uint32_t columns = n_v_heads / n_k_heads * v_dim, share = columns / kStepRanks;
    // Four CTAs to a key head: whole warps of columns, at most 64 of them, and a value head's either in one CTA or over whole ones.
    if (columns % (32 * kStepRanks) == 0 && share <= 64 && (share % v_dim == 0 || v_dim % share == 0)) {
        auto launch = [&](auto kernel) {
            cudaLaunchConfig_t config = {};
            config.gridDim = dim3(n_k_heads * kStepRanks);
            config.blockDim = dim3(share * (k_dim / 8));
            config.stream = stream;
            cudaLaunchAttribute attributes[2];
            attributes[0].id = cudaLaunchAttributeClusterDimension;
            attributes[0].val.clusterDim.x = kStepRanks;
            attributes[0].val.clusterDim.y = attributes[0].val.clusterDim.z = 1;
            attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attributes[1].val.programmaticStreamSerializationAllowed = 1;
            config.attrs = attributes;
            config.numAttrs = pdl_enabled() ? 2 : 1;
            return cudaLaunchKernelEx(&config, kernel, (const StepParams)p, (uint32_t)kStepRanks);
        };
        switch (k_dim) {
            case 32: return launch(gdn_step_kernel<32, 8, 64>);
            case 64: return launch(gdn_step_kernel<64, 8, 64>);
            case 96: return launch(gdn_step_kernel<96, 8, 64>);
            default: return launch(gdn_step_kernel<128, 8, 64>);
        }
    }
    uint32_t ranks = 1;
    void* args[] = {&p, &ranks};
    const uint32_t threads = kStepParts * columns;
    const void* kernel_fn = k_dim == 32 ? (const void*)gdn_step_kernel<32, 32 / kStepParts, 256> : k_dim == 64 ? (const void*)gdn_step_kernel<64, 64 / kStepParts, 256>
                          : k_dim == 96 ? (const void*)gdn_step_kernel<96, 96 / kStepParts, 256> : (const void*)gdn_step_kernel<128, 128 / kStepParts, 256>;
    return launch_kernel(kernel_fn, dim3(n_k_heads), dim3(threads), 0, stream, args);
}

cudaError_t gdn_gated_norm(cudaStream_t stream, float* x, const float* z, const float* weight, uint32_t v_dim, uint32_t n_rows,
                           float eps) {
    if (n_rows == 0) return cudaSuccess;
    void* args[] = {&x, &z, &weight, &v_dim, &n_rows, &eps};
    return launch_kernel((const void*)gdn_gated_norm_kernel, dim3((n_rows + 7) / 8), dim3(256), 0, stream, args);
}

bool gdn_gated_norm_pack_supported(uint32_t v_dim) { return v_dim == 64 || v_dim == 128 || v_dim == 256; }

cudaError_t gdn_gated_norm_pack(cudaStream_t stream, const float* x, const float* z, const float* weight, uint32_t v_dim, uint32_t n_heads, uint32_t n_tokens,
                                float eps, void* packed) {
    if (n_tokens == 0) return cudaSuccess;
    if (!gdn_gated_norm_pack_supported(v_dim)) return cudaErrorInvalidValue;
    uint32_t token_groups = ((n_tokens + 15u) & ~15u) / 8;
    const uint32_t lanes = v_dim / 8, rows = token_groups * 8 * n_heads, per_cta = 256 / lanes;
    void* args[] = {&x, &z, &weight, &packed, &n_heads, &n_tokens, &token_groups, &eps};
    const void* kernel = lanes == 8 ? (const void*)gdn_gated_norm_pack_kernel<8> : lanes == 16 ? (const void*)gdn_gated_norm_pack_kernel<16>
                                                                                              : (const void*)gdn_gated_norm_pack_kernel<32>;
    return launch_kernel(kernel, dim3((rows + per_cta - 1) / per_cta), dim3(256), 0, stream, args);
}

cudaError_t attention_gate(cudaStream_t stream, float* out, const float* q_gate, uint32_t n_heads, uint32_t head_dim, uint32_t n_tokens) {
    uint64_t n = (uint64_t)n_tokens * n_heads * head_dim;
    if (n == 0) return cudaSuccess;
    void* args[] = {&out, &q_gate, &n_heads, &head_dim, &n};
    return launch_kernel((const void*)attention_gate_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, args);
}

}  // namespace k
}  // namespace bc
