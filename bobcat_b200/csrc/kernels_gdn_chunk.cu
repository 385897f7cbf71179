// The gated delta rule over a batch in chunks of 64 tokens, f32 throughout.
//
// The rule (crates/bobcat/src/qwen35.rs:483-506), per value head with state S [k_dim][v_dim]:
// S *= a_t; delta_t = beta_t (v_t - S^T k_t); S += k_t delta_t^T; o_t = S^T q_t. Token by token that is a chain
// of dot products, 1.1 us per token (kernels_gdn.cu): 40 of the 73 ms of a 1501-token suffix on the 9B
// shape. Over a chunk it is linear algebra (the WY form of the delta rule: Yang, Kautz, Hatamizadeh, "Gated
// Delta Networks", 2024). With D(t, s) the product of the decays of tokens s + 1 .. t, g_t that of tokens 0 .. t and
// S the state before the chunk:
//   (I + L) delta = X,   L(t, s) = beta_t D(t, s) k_t.k_s for s < t,   x_t = beta_t (v_t - g_t S^T k_t)
//   o_t = g_t S^T q_t + sum over s <= t of A(t, s) delta_s,            A(t, s) = D(t, s) q_t.k_s
//   S   = g_63 S + sum over s of D(63, s) k_s delta_s^T
// so a chunk costs a handful of small matrix products. D is built by multiplication, never by dividing
// products, so decays of any size (zero included) are safe.
//
// gdn_chunk_prepare_kernel computes what does not depend on the state, for all chunks at once: a CTA per
// (16 rows of L and A, value head, chunk), which also inverts its 16 x 16 diagonal block of I + L (forward
// substitution; the triangular solve then needs four steps instead of 64). gdn_chunk_kernel carries
// the state: a CTA per (32 state columns, value head) with its slab of S in shared memory walks over the chunks; columns
// are independent, so nothing is exchanged. Its multiply-adds, 0.95 M per chunk and CTA against 128 per cycle, are 4 us; the reads of their
// operands from shared memory (128 bytes per cycle into registers, whether lanes share them or not) bound it: register tiles of 4 x 4, from
// rows padded to keep the reads free of bank conflicts, take as long as the reads. The next chunk arrives by cp.async while this one is
// computed. One chunk of 64 tokens takes 21.5 us of both launches in a chain of them, 512 tokens 111 (26.4 and 117 before the outputs' rows went to warps that lie in
// one block, the loops were unrolled further and the preparation below got its copies and straight-line decays). By the device's timer after the wait this
// kernel's part is 12.3 us, with a lane per column for the other products too 16.2; with cold caches under ncu a launch of it is no quicker than before (17.5 and 18.0).

#include <type_traits>

#include "async_utils.cuh"
#include "device_utils.cuh"
#include "kernels.h"

namespace bc {
namespace k {

namespace {

constexpr uint32_t kChunk = 64, kBlock = 16, kBlocks = kChunk / kBlock;
// Per (chunk, value head) in the scratch: L, A, the inverted diagonal blocks, g, D(63, .).
constexpr uint32_t kLAt = 0, kAAt = kChunk * kChunk, kInvAt = 2 * kChunk * kChunk, kGAt = kInvAt + kBlocks * kBlock * kBlock, kLastAt = kGAt + kChunk;
constexpr uint32_t kUnitFloats = kLastAt + kChunk;

struct ChunkParams {
    const float* qkv;    // [n_tokens][2 * key_dim + value_dim], q and k normalised
    const float* beta;   // [n_tokens][n_v_heads]
    const float* decay;  // [n_tokens][n_v_heads]
    float* state;        // [n_v_heads][k_dim][v_dim]
    float* out;          // [n_tokens][n_v_heads * v_dim]
    float* scratch;      // [n_chunks][n_v_heads][kUnitFloats]
    uint32_t n_k_heads, n_v_heads, v_dim, n_tokens;
};

__device__ int* g_wait_word;  // where a wait that ran out leaves its code (kernels.h), null until set

// The rows' copies; a wait that runs out leaves a code and the CTA carries on, its results void.
__device__ __forceinline__ void wait_rows(uint32_t bar) {
    for (uint32_t spin = 0; spin < 1u << 22; ++spin)
        if (async::mbar_test(bar, 0)) return;
    if (g_wait_word) *reinterpret_cast<volatile int*>(g_wait_word) = 1;
}

// 16 bytes, or zeros.
__device__ __forceinline__ void cp_async_16_or_zero(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void fma4(float (&acc)[4], float a, const float4& b) {
    acc[0] = fmaf(a, b.x, acc[0]);
    acc[1] = fmaf(a, b.y, acc[1]);
    acc[2] = fmaf(a, b.z, acc[2]);
    acc[3] = fmaf(a, b.w, acc[3]);
}
__device__ __forceinline__ float along4(const float4& a, const float (&b)[4], float acc) { return fmaf(a.w, b[3], fmaf(a.z, b[2], fmaf(a.y, b[1], fmaf(a.x, b[0], acc)))); }
__device__ __forceinline__ float dot4(const float4& a, const float4& b, float acc) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}

// grid (row block, value head, chunk), 256 threads. Bound by latency while there are few chunks: with a loop that looked up each decay on
// the way down to D(t, s) and the rows in pieces of 16 bytes a launch took 10.8 us after its wait (2.8, 1.8, and 5.5 for the products). Now
// the way down is straight-line code and a row is one copy: 7.3 us.
constexpr uint32_t kPrepareThreads = 256;

template <int KDIM>
__global__ void __launch_bounds__(kPrepareThreads) gdn_chunk_prepare_kernel(ChunkParams p) {
    constexpr uint32_t kPitch = KDIM + 4;  // 16-byte aligned rows, neighbouring rows four banks apart
    extern __shared__ __align__(16) float smem[];
    float* ks = smem;                       // [64][kPitch]
    float* qs = ks + kChunk * kPitch;       // [16][kPitch]
    __shared__ __align__(16) float decays[kChunk];
    __shared__ float betas[kBlock], ratio[kBlock][kChunk + 1], low[kBlock][kBlock + 1];
    __shared__ __align__(8) uint64_t arrived;
    const uint32_t block = blockIdx.x, head = blockIdx.y, chunk = blockIdx.z, tid = threadIdx.x, bar = async::smem_u32(&arrived);
    const uint32_t first = chunk * kChunk, live = min(kChunk, p.n_tokens - first), row0 = block * kBlock, n_cols = row0 + kBlock;
    const uint32_t key_dim = p.n_k_heads * KDIM, conv_dim = 2 * key_dim + p.n_v_heads * p.v_dim, key_head = head % p.n_k_heads;
    float* unit = p.scratch + ((uint64_t)chunk * p.n_v_heads + head) * kUnitFloats;
    const bool products = row0 < live;  // a block past the batch only passes the decays on
    pdl_launch_dependents();
    if (tid == 0) {
        async::mbar_init(bar, 1);
        async::mbar_init_fence();
    }
    __syncthreads();
    pdl_wait();
    // A row of K or of Q per thread; rows past the batch are zero.
    if (products && tid < n_cols + kBlock) {
        const bool is_q = tid >= n_cols;
        const uint32_t t = is_q ? row0 + tid - n_cols : tid;
        float* to = is_q ? qs + (tid - n_cols) * kPitch : ks + tid * kPitch;
        if (tid == 0) async::mbar_arrive_expect(bar, (min(live, n_cols) + min(live - row0, kBlock)) * KDIM * 4);
        if (t < live) {
            async::bulk_load(async::smem_u32(to), p.qkv + (uint64_t)(first + t) * conv_dim + (is_q ? 0 : key_dim) + key_head * KDIM, KDIM * 4, bar);
        } else {
#pragma unroll 4
            for (uint32_t c = 0; c < KDIM / 4; ++c) reinterpret_cast<float4*>(to)[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    if (tid >= 3 * kChunk) {
        const uint32_t t = tid - 3 * kChunk;
        decays[t] = t < live ? p.decay[(uint64_t)(first + t) * p.n_v_heads + head] : 1.f;
    } else if (tid >= 2 * kChunk && tid < 2 * kChunk + kBlock) {
        const uint32_t t = row0 + tid - 2 * kChunk;
        betas[tid - 2 * kChunk] = t < live ? p.beta[(uint64_t)(first + t) * p.n_v_heads + head] : 0.f;
    }
    __syncthreads();
    // D(t, s) for the block's rows: a thread per s multiplies its way down.
    if (tid < n_cols) {
        float d = 1.f;
        for (uint32_t b = 0; b < block; ++b) {
            float a[kBlock];
#pragma unroll
            for (uint32_t i = 0; i < kBlock; ++i) a[i] = decays[b * kBlock + i];
#pragma unroll
            for (uint32_t i = 0; i < kBlock; ++i)
                if (b * kBlock + i > tid) d *= a[i];
        }
        float a[kBlock];
#pragma unroll
        for (uint32_t i = 0; i < kBlock; ++i) a[i] = decays[row0 + i];
#pragma unroll
        for (uint32_t i = 0; i < kBlock; ++i) {
            if (row0 + i > tid) d *= a[i];
            if (row0 + i >= tid) ratio[i][tid] = d;
        }
    }
    if (products) wait_rows(bar);
    __syncthreads();
    if (tid < kBlock) unit[kGAt + row0 + tid] = decays[0] * ratio[tid][0];
    if (block == kBlocks - 1 && tid < kChunk) unit[kLastAt + tid] = ratio[kBlock - 1][tid];
    if (!products) return;
    // Two rows of K and of Q against up to four interleaved columns per thread of the first half. (One half K, the other Q: 9 us instead of
    // 5.5, the columns' reads from shared memory twice.)
    auto multiply = [&](auto columns) {
        constexpr uint32_t kColumns = decltype(columns)::value;  // per thread: the blocks up to this one
        const uint32_t rg = tid >> 4, cg = tid & 15;
        float kk[2][kColumns] = {}, qk[2][kColumns] = {};
        const float4* k_rows[2] = {reinterpret_cast<const float4*>(ks + (row0 + rg) * kPitch), reinterpret_cast<const float4*>(ks + (row0 + rg + 8) * kPitch)};
        const float4* q_rows[2] = {reinterpret_cast<const float4*>(qs + rg * kPitch), reinterpret_cast<const float4*>(qs + (rg + 8) * kPitch)};
#pragma unroll 4
        for (int c = 0; c < KDIM / 4; ++c) {
            const float4 a0 = k_rows[0][c], a1 = k_rows[1][c], b0 = q_rows[0][c], b1 = q_rows[1][c];
#pragma unroll
            for (uint32_t j = 0; j < kColumns; ++j) {
                const float4 col = *reinterpret_cast<const float4*>(ks + (cg + kBlock * j) * kPitch + 4 * c);
                kk[0][j] = dot4(a0, col, kk[0][j]);
                kk[1][j] = dot4(a1, col, kk[1][j]);
                qk[0][j] = dot4(b0, col, qk[0][j]);
                qk[1][j] = dot4(b1, col, qk[1][j]);
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i)
#pragma unroll
            for (uint32_t j = 0; j < kColumns; ++j) {
                const uint32_t r = rg + 8 * i, t = row0 + r, s = cg + kBlock * j;
                const float d = s <= t ? ratio[r][s] : 0.f;
                const float l = s < t ? betas[r] * d * kk[i][j] : 0.f;
                unit[kLAt + t * kChunk + s] = l;
                unit[kAAt + t * kChunk + s] = s <= t ? d * qk[i][j] : 0.f;
                if (j + 1 == kColumns) low[r][cg] = l;
            }
    };
    if (tid < 128) {
        static_assert(kBlocks == 4, "a chunk is four blocks");
        switch (block) {
            case 0: multiply(std::integral_constant<uint32_t, 1>()); break;
            case 1: multiply(std::integral_constant<uint32_t, 2>()); break;
            case 2: multiply(std::integral_constant<uint32_t, 3>()); break;
            default: multiply(std::integral_constant<uint32_t, 4>()); break;
        }
    }
    __syncthreads();
    // The inverse of the diagonal block: a thread per column of the identity.
    if (tid < kBlock) {
        float x[kBlock];
#pragma unroll
        for (uint32_t i = 0; i < kBlock; ++i) {
            float v = i == tid ? 1.f : 0.f;
#pragma unroll
            for (uint32_t j = 0; j < i; ++j) v = fmaf(-low[i][j], x[j], v);
            x[i] = v;
        }
#pragma unroll
        for (uint32_t i = 0; i < kBlock; ++i) unit[kInvAt + (block * kBlock + i) * kBlock + tid] = x[i];
    }
}

constexpr uint32_t kSlab = 32, kThreads = 256, kWarps = kThreads / 32;

template <int KDIM>
struct Slots {
    static constexpr uint32_t kPitch = KDIM + 4, kSlabPitch = kSlab + 4, kTriPitch = kChunk + 4, kInvPitch = kBlock + 4;
    // What arrives per chunk, in two slots; the queries have one, refilled as soon as they are used.
    float k[2][kChunk * kPitch];
    float l[2][kChunk * kTriPitch], a[2][kChunk * kTriPitch];
    float v[2][kChunk * kSlabPitch];        // v, then X, then delta
    float inv[2][kChunk * kInvPitch];
    float g[2][kChunk], last[2][kChunk], beta[2][kChunk];
    float q[kChunk * kPitch];
    float state[KDIM * kSlabPitch];
    float past[kChunk * kSlabPitch];        // g_t S^T q_t
    float right[kBlock * kSlabPitch];       // a block's right-hand side
};

// grid (slab of 32 columns, value head), 256 threads.
template <int KDIM>
__global__ void __launch_bounds__(kThreads, 1) gdn_chunk_kernel(ChunkParams p) {
    using S = Slots<KDIM>;
    constexpr uint32_t kRowVec = KDIM / 4;
    extern __shared__ __align__(16) float smem[];
    S& sh = *reinterpret_cast<S*>(smem);
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t tid = threadIdx.x, head = blockIdx.y, col0 = blockIdx.x * kSlab, vd = p.v_dim;
    const uint32_t key_dim = p.n_k_heads * KDIM, conv_dim = 2 * key_dim + p.n_v_heads * vd, key_head = head % p.n_k_heads;
    const uint32_t n_chunks = (p.n_tokens + kChunk - 1) / kChunk;
    float* state = p.state + (uint64_t)head * KDIM * vd + col0;

    auto bring_q = [&](uint32_t chunk) {
        const uint32_t first = chunk * kChunk;
        for (uint32_t i = tid; i < kChunk * kRowVec; i += kThreads) {
            const uint32_t t = i / kRowVec, c = i % kRowVec;
            const bool ok = first + t < p.n_tokens;
            cp_async_16_or_zero(async::smem_u32(sh.q + t * S::kPitch + 4 * c), p.qkv + (uint64_t)(ok ? first + t : 0) * conv_dim + key_head * KDIM + 4 * c, ok);
        }
    };
    auto bring = [&](uint32_t chunk, uint32_t slot) {
        const uint32_t first = chunk * kChunk;
        for (uint32_t i = tid; i < kChunk * kRowVec; i += kThreads) {
            const uint32_t t = i / kRowVec, c = i % kRowVec;
            const bool ok = first + t < p.n_tokens;
            cp_async_16_or_zero(async::smem_u32(sh.k[slot] + t * S::kPitch + 4 * c),
                                p.qkv + (uint64_t)(ok ? first + t : 0) * conv_dim + key_dim + key_head * KDIM + 4 * c, ok);
        }
        for (uint32_t i = tid; i < kChunk * (kSlab / 4); i += kThreads) {
            const uint32_t t = i / (kSlab / 4), c = i % (kSlab / 4);
            const bool ok = first + t < p.n_tokens;
            cp_async_16_or_zero(async::smem_u32(sh.v[slot] + t * S::kSlabPitch + 4 * c),
                                p.qkv + (uint64_t)(ok ? first + t : 0) * conv_dim + 2 * key_dim + head * vd + col0 + 4 * c, ok);
        }
        const float* unit = p.scratch + ((uint64_t)chunk * p.n_v_heads + head) * kUnitFloats;
        for (uint32_t i = tid; i < kChunk * (kChunk / 4); i += kThreads) {
            const uint32_t t = i / (kChunk / 4), c = i % (kChunk / 4);
            if (c / 4 > t / kBlock || first + (t & ~(kBlock - 1)) >= p.n_tokens) continue;  // above the diagonal blocks, past the batch: never read
            async::cp_async_16(async::smem_u32(sh.l[slot] + t * S::kTriPitch + 4 * c), unit + kLAt + t * kChunk + 4 * c);
            async::cp_async_16(async::smem_u32(sh.a[slot] + t * S::kTriPitch + 4 * c), unit + kAAt + t * kChunk + 4 * c);
        }
        if (tid < kChunk * (kBlock / 4) && first + (tid >> 2 & ~(kBlock - 1)) < p.n_tokens)
            async::cp_async_16(async::smem_u32(sh.inv[slot] + (tid >> 2) * S::kInvPitch + 4 * (tid & 3)), unit + kInvAt + (tid >> 2) * kBlock + 4 * (tid & 3));
        if (tid < kChunk / 4) async::cp_async_16(async::smem_u32(sh.g[slot] + 4 * tid), unit + kGAt + 4 * tid);
        else if (tid < kChunk / 2) async::cp_async_16(async::smem_u32(sh.last[slot] + 4 * (tid - kChunk / 4)), unit + kLastAt + 4 * (tid - kChunk / 4));
        if (tid >= kChunk && tid < 2 * kChunk) {
            const uint32_t t = tid - kChunk;
            const bool ok = first + t < p.n_tokens;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(async::smem_u32(sh.beta[slot] + t)),
                         "l"(p.beta + (uint64_t)(ok ? first + t : 0) * p.n_v_heads + head), "r"(ok ? 4 : 0)
                         : "memory");
        }
    };
    for (uint32_t i = tid; i < KDIM * (kSlab / 4); i += kThreads)
        async::cp_async_16(async::smem_u32(sh.state + (i / (kSlab / 4)) * S::kSlabPitch + 4 * (i % (kSlab / 4))), state + (uint64_t)(i / (kSlab / 4)) * vd + 4 * (i % (kSlab / 4)));
    bring(0, 0);
    bring_q(0);
    async::cp_async_commit();

    const uint32_t rg = tid >> 3, cg = tid & 7;  // 32 row groups x 8 groups of 4 columns
    const uint32_t lane = tid & 31, t0 = (tid >> 5) * (kChunk / kWarps);  // the outputs: a lane owns a column, a warp eight tokens
    constexpr uint32_t kTokens = kChunk / kWarps;
    for (uint32_t chunk = 0; chunk < n_chunks; ++chunk) {
        const uint32_t slot = chunk & 1, live = min(kChunk, p.n_tokens - chunk * kChunk), blocks = (live + kBlock - 1) / kBlock;
        async::cp_async_wait<0>();
        __syncthreads();  // this chunk is here, and everyone is through with the slot the next one takes
        if (chunk + 1 < n_chunks) bring(chunk + 1, slot ^ 1);
        float* x = sh.v[slot];
        // ---- S^T k and S^T q: rows rg and rg + 32 of both.
        {
            float acc[4][4] = {};
            const float4* rows[4] = {reinterpret_cast<const float4*>(sh.k[slot] + rg * S::kPitch), reinterpret_cast<const float4*>(sh.q + rg * S::kPitch),
                                     reinterpret_cast<const float4*>(sh.k[slot] + (rg + 32) * S::kPitch), reinterpret_cast<const float4*>(sh.q + (rg + 32) * S::kPitch)};
            const int n_rows = live > 32 ? 4 : 2;
#pragma unroll 4
            for (uint32_t c = 0; c < kRowVec; ++c) {
                float4 s[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) s[e] = *reinterpret_cast<const float4*>(sh.state + (4 * c + e) * S::kSlabPitch + 4 * cg);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (i >= n_rows) break;
                    const float4 r = rows[i][c];
                    fma4(acc[i], r.x, s[0]);
                    fma4(acc[i], r.y, s[1]);
                    fma4(acc[i], r.z, s[2]);
                    fma4(acc[i], r.w, s[3]);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t t = rg + 32 * h;
                const float g = sh.g[slot][t], b = sh.beta[slot][t];
                float4* xv = reinterpret_cast<float4*>(x + t * S::kSlabPitch + 4 * cg);
                const float4 v = *xv;
                const float* kr = acc[2 * h];
                const float* qr = acc[2 * h + 1];
                *xv = make_float4(b * (v.x - g * kr[0]), b * (v.y - g * kr[1]), b * (v.z - g * kr[2]), b * (v.w - g * kr[3]));
                *reinterpret_cast<float4*>(sh.past + t * S::kSlabPitch + 4 * cg) = make_float4(g * qr[0], g * qr[1], g * qr[2], g * qr[3]);
            }
        }
        __syncthreads();
        if (chunk + 1 < n_chunks) bring_q(chunk + 1);
        async::cp_async_commit();
        // ---- (I + L) delta = X, a block of 16 rows at a time: a thread finishes one row's two columns.
        {
            const uint32_t r = tid >> 4, c2 = (tid & 15) * 2;
            for (uint32_t b = 0; b < blocks; ++b) {
                const uint32_t t = b * kBlock + r;
                float2 y = *reinterpret_cast<const float2*>(x + t * S::kSlabPitch + c2);
                const float4* l = reinterpret_cast<const float4*>(sh.l[slot] + t * S::kTriPitch);
#pragma unroll 4
                for (uint32_t s4 = 0; s4 < b * (kBlock / 4); ++s4) {
                    const float4 w = l[s4];
                    const float* d = x + 4 * s4 * S::kSlabPitch + c2;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 delta = *reinterpret_cast<const float2*>(d + e * S::kSlabPitch);
                        const float we = e == 0 ? w.x : e == 1 ? w.y : e == 2 ? w.z : w.w;
                        y.x = fmaf(-we, delta.x, y.x);
                        y.y = fmaf(-we, delta.y, y.y);
                    }
                }
                *reinterpret_cast<float2*>(sh.right + r * S::kSlabPitch + c2) = y;
                __syncthreads();
                float2 z = make_float2(0.f, 0.f);
                const float4* inv = reinterpret_cast<const float4*>(sh.inv[slot] + t * S::kInvPitch);
#pragma unroll
                for (int s4 = 0; s4 < (int)kBlock / 4; ++s4) {
                    const float4 w = inv[s4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 right = *reinterpret_cast<const float2*>(sh.right + (4 * s4 + e) * S::kSlabPitch + c2);
                        const float we = e == 0 ? w.x : e == 1 ? w.y : e == 2 ? w.z : w.w;
                        z.x = fmaf(we, right.x, z.x);
                        z.y = fmaf(we, right.y, z.y);
                    }
                }
                *reinterpret_cast<float2*>(x + t * S::kSlabPitch + c2) = z;
                __syncthreads();
            }
        }
        // ---- the outputs of the warp's tokens, A delta on top of the state's share.
        if (t0 < live) {
            float acc[kTokens];
#pragma unroll
            for (uint32_t i = 0; i < kTokens; ++i) acc[i] = sh.past[(t0 + i) * S::kSlabPitch + lane];
            const float4* a4 = reinterpret_cast<const float4*>(sh.a[slot] + t0 * S::kTriPitch);
            const uint32_t vectors = (t0 / kBlock + 1) * (kBlock / 4);  // the tokens lie in one block
#pragma unroll 2
            for (uint32_t s4 = 0; s4 < vectors; ++s4) {
                float delta[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) delta[e] = x[(4 * s4 + e) * S::kSlabPitch + lane];
#pragma unroll
                for (uint32_t i = 0; i < kTokens; ++i) acc[i] = along4(a4[i * (S::kTriPitch / 4) + s4], delta, acc[i]);
            }
#pragma unroll
            for (uint32_t i = 0; i < kTokens; ++i)
                if (t0 + i < live) p.out[(uint64_t)(chunk * kChunk + t0 + i) * p.n_v_heads * vd + head * vd + col0 + lane] = acc[i];
        }
        // ---- the state: a thread owns KDIM / 32 rows of S x 4 columns.
        {
            constexpr int kOwn = KDIM / 32;  // rows rg * kOwn ..
            float acc[kOwn][4] = {};
            const float* kr = sh.k[slot] + rg * kOwn;
#pragma unroll 8
            for (uint32_t s = 0; s < blocks * kBlock; ++s) {
                const float w = sh.last[slot][s];
                float4 d = *reinterpret_cast<const float4*>(x + s * S::kSlabPitch + 4 * cg);
                d.x *= w, d.y *= w, d.z *= w, d.w *= w;
                float kv[kOwn];
                if (kOwn == 4) {
                    const float4 k4 = *reinterpret_cast<const float4*>(kr + s * S::kPitch);
                    kv[0] = k4.x, kv[1 % kOwn] = k4.y, kv[2 % kOwn] = k4.z, kv[3 % kOwn] = k4.w;
                } else {
#pragma unroll
                    for (int e = 0; e < kOwn; ++e) kv[e] = kr[s * S::kPitch + e];
                }
#pragma unroll
                for (int e = 0; e < kOwn; ++e) fma4(acc[e], kv[e], d);
            }
            const float g = sh.g[slot][kChunk - 1];
#pragma unroll
            for (int e = 0; e < kOwn; ++e) {
                float4* s = reinterpret_cast<float4*>(sh.state + (rg * kOwn + e) * S::kSlabPitch + 4 * cg);
                float4 v = *s;
                v.x = fmaf(g, v.x, acc[e][0]);
                v.y = fmaf(g, v.y, acc[e][1]);
                v.z = fmaf(g, v.z, acc[e][2]);
                v.w = fmaf(g, v.w, acc[e][3]);
                *s = v;
                if (chunk + 1 == n_chunks) *reinterpret_cast<float4*>(state + (uint64_t)(rg * kOwn + e) * vd + 4 * cg) = v;
            }
        }
    }
    async::cp_async_wait<0>();
}

template <int KDIM>
cudaError_t launch_chunks(cudaStream_t stream, const ChunkParams& p) {
    const uint32_t n_chunks = (p.n_tokens + kChunk - 1) / kChunk;
    constexpr size_t prepare_smem = (size_t)(kChunk + kBlock) * (KDIM + 4) * sizeof(float);
    cudaError_t e = ensure_dynamic_smem((const void*)gdn_chunk_prepare_kernel<KDIM>, prepare_smem);
    if (e == cudaSuccess) e = ensure_dynamic_smem((const void*)gdn_chunk_kernel<KDIM>, sizeof(Slots<KDIM>));
    if (e != cudaSuccess) return e;
    e = launch_dependent(gdn_chunk_prepare_kernel<KDIM>, dim3(kBlocks, p.n_v_heads, n_chunks), dim3(kPrepareThreads), prepare_smem, stream, p);
    if (e != cudaSuccess) return e;
    return launch_dependent(gdn_chunk_kernel<KDIM>, dim3(p.v_dim / kSlab, p.n_v_heads), dim3(kThreads), sizeof(Slots<KDIM>), stream, p);
}

}  // namespace

cudaError_t gdn_chunk_wait_word(int* word) { return cudaMemcpyToSymbol(g_wait_word, &word, sizeof word); }

uint64_t gdn_chunk_scratch_bytes(uint32_t n_v_heads, uint32_t n_tokens) {
    return (uint64_t)((n_tokens + kChunk - 1) / kChunk) * n_v_heads * kUnitFloats * sizeof(float);
}

// From 12 tokens on: a chunk, however few of its tokens are live, takes about as long as the chain takes for ten.
bool gdn_chunk_supported(uint32_t n_v_heads, uint32_t k_dim, uint32_t v_dim, uint32_t n_tokens) {
    return n_tokens >= 12 && n_tokens <= 65535u * kChunk && n_v_heads <= 65535u && v_dim % kSlab == 0 && (k_dim == 32 || k_dim == 64 || k_dim == 96 || k_dim == 128);
}

cudaError_t gdn_chunk(cudaStream_t stream, const float* qkv, const float* beta, const float* decay, float* state, float* out, void* scratch,
                      uint32_t n_k_heads, uint32_t n_v_heads, uint32_t k_dim, uint32_t v_dim, uint32_t n_tokens) {
    ChunkParams p{qkv, beta, decay, state, out, static_cast<float*>(scratch), n_k_heads, n_v_heads, v_dim, n_tokens};
    switch (k_dim) {
        case 32: return launch_chunks<32>(stream, p);
        case 64: return launch_chunks<64>(stream, p);
        case 96: return launch_chunks<96>(stream, p);
        default: return launch_chunks<128>(stream, p);
    }
}

}  // namespace k
}  // namespace bc
