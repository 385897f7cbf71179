// Token sampling on the device: the steps of the reference's Sampler::sample
// (crates/bobcat-cli/src/sampler.rs:45-112, llama.cpp's order) without sorting the vocabulary and
// without bringing the logits to the host: repetition penalty, top-k, top-p, min-p, temperature,
// then the draw.
//
// The reference sorts the candidates by logit and walks them in that order three times (the
// top-p cut, the min-p floor, the draw). Walking a sorted list until a running sum crosses a
// target is a selection problem: it needs the key at which the sum crosses, not the order of
// everything else. Logits map to 32-bit keys that sort the same way (descending logit = ascending
// key), and a key is found four bits at a time: the summed weight per value of the next four bits
// (over the candidates that match the bits decided so far), a walk over the 16 sums to the one
// where the running sum crosses, eight rounds:
//   top-k   - the key of the k-th largest logit (weights 1),
//   top-p   - the key where the softmax at temperature one, summed from the largest logit down,
//             reaches top_p,
//   min-p   - a plain threshold, logit >= largest + ln(min_p),
//   draw    - the key where the softmax of the survivors at the temperature, summed from the
//             largest logit down, passes the uniform draw; equal logits are told apart by index.
// Where the reference's unstable sort breaks ties between equal logits arbitrarily at a cut, every
// logit equal to the cut value is kept here. The uniform draw comes from the caller (the
// reference draws it from fastrand, whose stream is the host's business), so the kernel is a
// function of its inputs. All sums are taken in a fixed order.
//
// What bounds it: the chain of rounds. A cluster of eight CTAs holds the logits in its shared memory (8 192
// or 18 992 per CTA at the vocabularies in use), so a round reads nothing from global memory; a thread keeps its 16 sums in
// registers (selects and adds, no atomics: most logits share the first bits of their keys, and a
// histogram by shared-memory float atomics spent its time on that contention, in one CTA 587 us per draw at 65 536
// logits with top-k and top-p); the CTAs exchange 16 floats each through distributed shared memory. Top-k needs the rounds only
// until at most 1024 logits can be among the k largest, three or four of the eight: those go to the first CTA, which
// sorts them and finds the cuts and the draw by prefix sums (65 536 logits, k 40, top-p: 71 us with 24 rounds, 24 us now).

#include <cfloat>

#include "device_utils.cuh"
#include "kernels.h"

namespace bc {
namespace k {

namespace {

constexpr int kSampleThreads = 1024;
constexpr uint32_t kRepeatLastN = 64;  // REPEAT_LAST_N, sampler.rs:9-10

// Ascending key = descending logit. NaNs sort last.
__device__ __forceinline__ uint32_t descending_key(float v) {
    uint32_t bits = __float_as_uint(v);
    uint32_t ascending = (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);
    return ~ascending;
}

struct SampleParams {
    float* logits;
    uint32_t n;
    const uint32_t* recent;
    uint32_t n_recent;
    Sampling settings;
    float uniform;
    uint32_t* out;
    uint32_t* readback;
};

constexpr uint32_t kCtas = 8, kWarps = kSampleThreads / 32;
constexpr int kDigits = 16;

struct Shared {
    float warps[kWarps][kDigits];     // the warps' sums of a round
    float mine[2][kDigits];           // this CTA's, read by the cluster; the parity alternates between exchanges
    float all[kCtas][kDigits];        // every CTA's
    uint32_t counts[kWarps];
};

__device__ __forceinline__ void cluster_sync() { asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory"); }
__device__ __forceinline__ float remote_float(const float* p, uint32_t rank) {
    uint32_t at;
    float v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}

// The CTA's share of the logits and the exchange with the other CTAs.
struct Slice {
    const float* v;     // shared memory, or the logits themselves when a share does not fit there
    uint32_t count;     // logits of this CTA
    uint32_t parity;    // of the next exchange
    Shared& sh;

    // sh.mine[parity] of every CTA into sh.all. Whoever writes sh.mine again does so with the
    // other parity, and the exchange after that orders it behind this one's reads.
    __device__ void exchange(int n) {
        cluster_sync();
        for (int i = threadIdx.x; i < (int)kCtas * n; i += kSampleThreads) sh.all[i / n][i % n] = remote_float(&sh.mine[parity][i % n], i / n);
        __syncthreads();
        parity ^= 1;
    }
    // The sums over the CTAs, in rank order, into sh.all[0].
    __device__ void exchange_sums() {
        cluster_sync();
        if (threadIdx.x < kDigits) {
            float x = 0.f;
#pragma unroll
            for (uint32_t r = 0; r < kCtas; ++r) x += remote_float(&sh.mine[parity][threadIdx.x], r);
            sh.all[0][threadIdx.x] = x;
        }
        __syncthreads();
        parity ^= 1;
    }
    __device__ float total(float x, bool largest) {
        x = largest ? warp_max(x) : warp_sum(x);
        __syncthreads();
        if ((threadIdx.x & 31) == 0) sh.warps[threadIdx.x >> 5][0] = x;
        __syncthreads();
        if (threadIdx.x < 32) {
            x = sh.warps[threadIdx.x][0];
            x = largest ? warp_max(x) : warp_sum(x);
            if (threadIdx.x == 0) sh.mine[parity][0] = x;
        }
        exchange(1);
        float t = sh.all[0][0];
        for (uint32_t r = 1; r < kCtas; ++r) t = largest ? fmaxf(t, sh.all[r][0]) : t + sh.all[r][0];
        return t;
    }
};

// The smallest key K among the candidates (keys <= limit) at which the weight summed over keys
// <= K passes `target` (exceeds it, or reaches it when `inclusive`). `weight(logit)` gives a
// candidate's weight. Returns K; `below` then holds the weight of the candidates with smaller keys.
// When the target lies beyond the total (rounding), the largest candidate key is returned. With `enough`, it stops as soon as the
// candidates that share K's bits so far, and those before them, weigh no more: `stopped` is set and the largest key
// they may have is returned.
template <typename W>
__device__ uint32_t select_key(Slice& slice, uint32_t limit, float target, bool inclusive, W weight, float& below, float enough = 0.f, bool* stopped = nullptr) {
    Shared& sh = slice.sh;
    uint32_t prefix = 0;
    below = 0.f;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int shift = 28; shift >= 0; shift -= 4) {
        float sums[kDigits];
#pragma unroll
        for (int d = 0; d < kDigits; ++d) sums[d] = 0.f;
        for (uint32_t i = threadIdx.x; i < slice.count; i += kSampleThreads) {
            const float v = slice.v[i];
            const uint32_t key = descending_key(v);
            if (key > limit || (shift < 28 && (key >> (shift + 4)) != prefix)) continue;
            const uint32_t digit = (key >> shift) & 15u;
            const float w = weight(v);
#pragma unroll
            for (int d = 0; d < kDigits; ++d) sums[d] += digit == (uint32_t)d ? w : 0.f;
        }
        // A warp's 16 sums by halving: after the step of `half`, a lane keeps half as many digits.
        // Lanes 2 d and 2 d + 1 end up with digit d.
#pragma unroll
        for (int half = 8, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
#pragma unroll
            for (int d = 0; d < half; ++d) {
                const bool high = lane & bit;
                const float give = high ? sums[d] : sums[d + half];
                const float got = __shfl_xor_sync(0xffffffffu, give, bit);
                sums[d] = (high ? sums[d + half] : sums[d]) + got;
            }
        }
        sums[0] += __shfl_xor_sync(0xffffffffu, sums[0], 1);
        __syncthreads();
        if ((lane & 1) == 0) sh.warps[warp][lane >> 1] = sums[0];
        __syncthreads();
        if (threadIdx.x < kDigits) {
            float x = 0.f;
            for (uint32_t w = 0; w < kWarps; ++w) x += sh.warps[w][threadIdx.x];
            sh.mine[slice.parity][threadIdx.x] = x;
        }
        slice.exchange_sums();
        // Every thread walks the same 16 sums.
        float running = below, before_last = below;
        int chosen = -1, last_filled = 0;
#pragma unroll 1
        for (int d = 0; d < kDigits; ++d) {
            const float h = sh.all[0][d];
            if (h <= 0.f) continue;
            last_filled = d;
            before_last = running;
            const float with = running + h;
            if (inclusive ? with >= target : with > target) {
                chosen = d;
                break;
            }
            running = with;
        }
        if (chosen < 0) {
            // Past the end: settle on the last filled digit, with everything before it below.
            chosen = last_filled;
            running = before_last;
        }
        below = running;
        prefix = (prefix << 4) | (uint32_t)chosen;
        if (stopped && running + sh.all[0][chosen] <= enough) {
            *stopped = true;
            return prefix << shift | ((1u << shift) - 1u);
        }
    }
    return prefix;
}

constexpr uint32_t kSorted = kSampleThreads;  // candidates that the first CTA can sort, one to a thread

struct Sorted {
    unsigned long long items[kSorted];  // key, index: neighbours may change places in any order on the way here
    uint32_t count;
    float warps[kWarps];
    uint32_t found[kWarps];
};

__device__ __forceinline__ float logit_of(uint32_t key) {
    const uint32_t ascending = ~key;
    return __uint_as_float((ascending & 0x80000000u) ? ascending & 0x7fffffffu : ~ascending);
}

// Inclusive prefix sum over the CTA's threads.
__device__ float scan(float x, Sorted& st) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float other = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += other;
    }
    __syncthreads();
    if (lane == 31) st.warps[warp] = x;
    __syncthreads();
    float before = 0.f;
    for (uint32_t w = 0; w < warp; ++w) before += st.warps[w];
    return before + x;
}
// The first thread for which `yes` holds, or `otherwise`.
__device__ uint32_t first_of(bool yes, uint32_t otherwise, Sorted& st) {
    const uint32_t votes = __ballot_sync(0xffffffffu, yes);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) st.found[threadIdx.x >> 5] = votes ? (threadIdx.x & ~31u) + __ffs(votes) - 1 : 0xffffffffu;
    __syncthreads();
    const uint32_t first = __reduce_min_sync(0xffffffffu, st.found[threadIdx.x & 31]);
    return first == 0xffffffffu ? otherwise : first;
}

// The rest of the draw on one CTA, over the candidates in st.items (at least top_k of them).
__device__ void draw_sorted(const SampleParams& p, Sorted& st, float top) {
    const Sampling& s = p.settings;
    const uint32_t tid = threadIdx.x, count = st.count;
    unsigned long long item = tid < count ? st.items[tid] : ~0ull;
    // Bitonic sort; strides within a warp by shuffles.
    uint32_t size = 32;
    while (size < count) size *= 2;
    for (uint32_t run = 2; run <= size; run *= 2) {
        for (uint32_t step = run / 2; step > 0; step /= 2) {
            unsigned long long other;
            if (step < 32) {
                other = __shfl_xor_sync(0xffffffffu, item, step);
            } else {
                __syncthreads();
                st.items[tid] = item;
                __syncthreads();
                other = st.items[tid ^ step];
            }
            const bool ascending = (tid & run) == 0, lower = (tid & step) == 0;
            if (tid < size && (ascending == lower ? other < item : other > item)) item = other;
        }
    }
    __syncthreads();
    st.items[tid] = item;
    __syncthreads();
    const uint32_t key = (uint32_t)(item >> 32);
    const float v = logit_of(key);
    // Candidates: keys up to the k-th, then up to where the softmax reaches top_p, then above the floor.
    uint32_t limit = (uint32_t)(st.items[min((uint32_t)s.top_k, count) - 1] >> 32);
    bool in = tid < count && key <= limit;
    if (s.top_p < 1.0f) {
        const uint32_t last = first_of(!in, kSorted, st) - 1;
        const float sum = scan(in ? expf(v - top) : 0.f, st);
        __syncthreads();
        if (tid == last) st.warps[0] = sum;
        __syncthreads();
        const float total = st.warps[0];
        const uint32_t at = first_of(in && sum >= s.top_p * total, last, st);
        limit = (uint32_t)(st.items[at] >> 32);
    }
    if (s.min_p > 0.f) limit = min(limit, descending_key(top + logf(s.min_p)));
    in = tid < count && key <= limit;
    const uint32_t last = first_of(!in, kSorted, st) - 1;
    const float inv_t = 1.0f / s.temperature, w = in ? expf((v - top) * inv_t) : 0.f, sum = scan(w, st);
    __syncthreads();
    if (tid == last) st.warps[0] = sum;
    __syncthreads();
    const float target = p.uniform * st.warps[0];
    const uint32_t at = first_of(in && sum > target, last, st);
    const uint32_t picked = (uint32_t)(st.items[at] >> 32);
    // Equal logits: the remainder picks among them by index, which is their order here.
    const uint32_t start = first_of(in && key == picked, at, st), end = first_of(tid > start && !(in && key == picked), kSorted, st);
    if (tid == start) {
        uint32_t wanted = 0;
        if (w > 0.f && end - start > 1) wanted = min((uint32_t)(fmaxf(target - (sum - w), 0.f) / w), end - start - 1);
        const uint32_t index = (uint32_t)st.items[start + wanted];
        *p.out = index;
        if (p.readback) *p.readback = index;
    }
}

__global__ void __launch_bounds__(kSampleThreads) sample_kernel(SampleParams p, uint32_t share, int in_shared) {
    extern __shared__ float held[];
    __shared__ Shared sh;
    __shared__ Sorted sorted;
    if (threadIdx.x == 0) sorted.count = 0;  // before the first exchange, after which other CTAs add to it
    pdl_launch_dependents();
    pdl_wait();
    const Sampling s = p.settings;
    const uint32_t tid = threadIdx.x, rank = blockIdx.x;
    const uint32_t begin = min(p.n, rank * share), count = min(p.n - begin, share);
    float* logits = p.logits + begin;

    // Repetition penalty: each distinct token among the last 64 takes it once (sampler.rs:47-63), from the CTA that holds its logit.
    if (fabsf(s.repeat_penalty - 1.0f) > FLT_EPSILON && p.n_recent) {
        const uint32_t window = min(p.n_recent, kRepeatLastN);
        const uint32_t* recent = p.recent + (p.n_recent - window);
        if (tid < window) {
            const uint32_t token = recent[tid];
            bool first = token >= begin && token < begin + count;
            for (uint32_t j = 0; j < tid && first; ++j) first = recent[j] != token;
            if (first) {
                const float logit = p.logits[token];
                p.logits[token] = logit > 0.f ? logit / s.repeat_penalty : logit * s.repeat_penalty;
            }
        }
        __syncthreads();
    }
    Slice slice{in_shared ? held : logits, count, 0, sh};

    // The largest logit and its lowest index.
    float best = -INFINITY;
    uint32_t best_index = 0xffffffffu;
    for (uint32_t i = tid; i < count; i += kSampleThreads) {
        const float v = logits[i];
        if (in_shared) held[i] = v;  // read back by the same thread, and by others after the barriers below
        if (v > best || best_index == 0xffffffffu) {
            best = v;
            best_index = begin + i;
        }
    }
    const float top = slice.total(best, true);
    if (s.temperature <= 0.f) {
        // Greedy: the first maximum (sampler.rs:70-76).
        uint32_t candidate = best == top ? best_index : 0xffffffffu;
        candidate = __reduce_min_sync(0xffffffffu, candidate);
        if ((tid & 31) == 0) sh.counts[tid >> 5] = candidate;
        __syncthreads();
        if (tid < 32) {
            candidate = __reduce_min_sync(0xffffffffu, sh.counts[tid]);
            if (tid == 0) sh.mine[slice.parity][0] = __uint_as_float(candidate);
        }
        slice.exchange(1);
        if (rank == 0 && tid == 0) {
            uint32_t index = 0xffffffffu;
            for (uint32_t r = 0; r < kCtas; ++r) index = min(index, __float_as_uint(sh.all[r][0]));
            *p.out = index;
            if (p.readback) *p.readback = index;
        }
        cluster_sync();  // no CTA leaves while another reads its sums
        return;
    }

    uint32_t limit = 0xffffffffu;  // candidates are the logits whose key is <= limit
    float below;
    if (s.top_k > 0 && s.top_k < p.n) {
        bool few = false;
        limit = select_key(slice, limit, (float)s.top_k - 0.5f, false, [](float) { return 1.0f; }, below, (float)kSorted, &few);
        if (few) {
            for (uint32_t i = tid; i < count; i += kSampleThreads) {
                const uint32_t key = descending_key(slice.v[i]);
                if (key > limit) continue;
                uint32_t at, slot;
                asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(&sorted.count)));
                asm volatile("atom.shared::cluster.add.u32 %0, [%1], 1;" : "=r"(slot) : "r"(at) : "memory");
                if (slot >= kSorted) continue;  // cannot be: there are no more
                asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(&sorted.items[slot])));
                asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(at), "l"((unsigned long long)key << 32 | (begin + i)) : "memory");
            }
            cluster_sync();
            if (rank == 0) draw_sorted(p, sorted, top);
            return;
        }
    }
    auto unit_softmax = [top](float v) { return expf(v - top); };
    if (s.top_p < 1.0f) {
        float mine = 0.f;
        for (uint32_t i = tid; i < count; i += kSampleThreads) {
            const float v = slice.v[i];
            if (descending_key(v) <= limit) mine += unit_softmax(v);
        }
        const float total = slice.total(mine, false);
        limit = select_key(slice, limit, s.top_p * total, true, unit_softmax, below);
    }
    if (s.min_p > 0.f) {
        // p >= p_first * min_p, with p proportional to exp(logit - top) (sampler.rs:98-99).
        const uint32_t floor_key = descending_key(top + logf(s.min_p));
        limit = min(limit, floor_key);
    }

    // The draw over the survivors at the temperature (sampler.rs:101-111).
    const float inv_t = 1.0f / s.temperature;
    auto tempered = [top, inv_t](float v) { return expf((v - top) * inv_t); };
    float mine = 0.f;
    for (uint32_t i = tid; i < count; i += kSampleThreads) {
        const float v = slice.v[i];
        if (descending_key(v) <= limit) mine += tempered(v);
    }
    const float total = slice.total(mine, false);
    const float target = p.uniform * total;
    const uint32_t picked_key = select_key(slice, limit, target, false, tempered, below);

    // Equal logits share the key: the draw's remainder picks among them by index. A thread looks at
    // neighbouring logits, so ties are counted in the order of their indexes.
    const uint32_t per_thread = (count + kSampleThreads - 1) / kSampleThreads;
    const uint32_t first = min(count, tid * per_thread), last = min(count, first + per_thread);
    uint32_t ties = 0;
    float tie_weight = 0.f;
    for (uint32_t i = first; i < last; ++i) {
        const float v = slice.v[i];
        if (descending_key(v) == picked_key) {
            ++ties;
            tie_weight = tempered(v);
        }
    }
    uint32_t inclusive_scan = ties;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t other = __shfl_up_sync(0xffffffffu, inclusive_scan, o);
        if ((tid & 31) >= o) inclusive_scan += other;
    }
    if ((tid & 31) == 31) sh.counts[tid >> 5] = inclusive_scan;
    tie_weight = warp_max(tie_weight);  // the same value from every thread that has one
    if ((tid & 31) == 0) sh.warps[tid >> 5][0] = tie_weight;
    __syncthreads();
    uint32_t before = inclusive_scan - ties, in_cta = 0;
    for (uint32_t w = 0; w < (tid >> 5); ++w) before += sh.counts[w];
    if (tid == 0) {
        float w = 0.f;
        for (uint32_t i = 0; i < kWarps; ++i) in_cta += sh.counts[i], w = fmaxf(w, sh.warps[i][0]);
        sh.mine[slice.parity][0] = __uint_as_float(in_cta);
        sh.mine[slice.parity][1] = w;
    }
    slice.exchange(2);
    uint32_t all_ties = 0;
    float w = 0.f;
    for (uint32_t r = 0; r < kCtas; ++r) {
        const uint32_t there = __float_as_uint(sh.all[r][0]);
        if (r < rank) before += there;
        all_ties += there;
        w = fmaxf(w, sh.all[r][1]);
    }
    uint32_t wanted = 0;
    if (w > 0.f && all_ties > 1) {
        const float remainder = fmaxf(target - below, 0.f);
        wanted = min((uint32_t)(remainder / w), all_ties - 1);
    }
    if (ties && wanted >= before && wanted < before + ties) {
        uint32_t seen = before;
        for (uint32_t i = first; i < last; ++i) {
            if (descending_key(slice.v[i]) != picked_key) continue;
            if (seen == wanted) {
                *p.out = begin + i;
                if (p.readback) *p.readback = begin + i;
                break;
            }
            ++seen;
        }
    }
    cluster_sync();
}

// ---- log-probabilities of label tokens: log-softmax in f64 (engine.rs:425-433)

constexpr uint32_t kLogSumLogits = 512;  // of a CTA

// A CTA's share: its largest logit and the f64 sum of the exponentials relative to it. Bound by f64 arithmetic, about six operations
// per cycle and SM, so the logits are spread over all of them: 65 536 in 6 us with the kernel below, where reading
// them back and summing on one host core took 0.4 ms a prompt.
__global__ void __launch_bounds__(256) log_sum_kernel(const float* __restrict__ logits, uint32_t n, double* __restrict__ partial) {
    __shared__ float tops[8];
    __shared__ double sums[8];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t tid = threadIdx.x, first = blockIdx.x * kLogSumLogits, last = min(n, first + kLogSumLogits);
    float top = -INFINITY;
    for (uint32_t i = first + tid; i < last; i += 256) top = fmaxf(top, __ldcg(logits + i));
    top = warp_max(top);
    if ((tid & 31) == 0) tops[tid >> 5] = top;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) top = fmaxf(top, tops[w]);
    double sum = 0.0;
    for (uint32_t i = first + tid; i < last; i += 256) sum += exp((double)__ldcg(logits + i) - (double)top);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((tid & 31) == 0) sums[tid >> 5] = sum;
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < 8; ++w) sum += sums[w];
        partial[2 * blockIdx.x] = (double)top;
        partial[2 * blockIdx.x + 1] = sum;
    }
}

__global__ void __launch_bounds__(256) label_log_probs_kernel(const float* __restrict__ logits, const double* __restrict__ partial, uint32_t n_partial,
                                                              const uint32_t* __restrict__ labels, uint32_t n_labels, double* __restrict__ out) {
    __shared__ double tops[8], sums[8];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t tid = threadIdx.x;
    double top = -INFINITY, sum = 0.0;
    for (uint32_t i = tid; i < n_partial; i += 256) top = fmax(top, __ldcg(partial + 2 * i));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    if ((tid & 31) == 0) tops[tid >> 5] = top;
    __syncthreads();
    for (int w = 0; w < 8; ++w) top = fmax(top, tops[w]);
    for (uint32_t i = tid; i < n_partial; i += 256) sum += __ldcg(partial + 2 * i + 1) * exp(__ldcg(partial + 2 * i) - top);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((tid & 31) == 0) sums[tid >> 5] = sum;
    __syncthreads();
    sum = 0.0;
    for (int w = 0; w < 8; ++w) sum += sums[w];
    const double log_sum = top + log(sum);
    for (uint32_t i = tid; i < n_labels; i += 256) out[i] = (double)__ldcg(logits + labels[i]) - log_sum;
}

}  // namespace

uint64_t label_log_probs_scratch(uint32_t n) { return (uint64_t)((n + kLogSumLogits - 1) / kLogSumLogits) * 2; }

cudaError_t label_log_probs(cudaStream_t stream, const float* logits, uint32_t n, const uint32_t* labels, uint32_t n_labels, double* scratch, double* out) {
    if (n == 0 || n_labels == 0) return cudaSuccess;
    const uint32_t parts = (n + kLogSumLogits - 1) / kLogSumLogits;
    cudaError_t e = launch_dependent(log_sum_kernel, dim3(parts), dim3(256), 0, stream, logits, n, scratch);
    if (e != cudaSuccess) return e;
    return launch_dependent(label_log_probs_kernel, dim3(1), dim3(256), 0, stream, logits, static_cast<const double*>(scratch), parts, labels, n_labels, out);
}

cudaError_t sample(cudaStream_t stream, float* logits, uint32_t n, const uint32_t* recent, uint32_t n_recent, const Sampling& settings,
                   float uniform, uint32_t* out, uint32_t* readback) {
    SampleParams p{logits, n, recent, n_recent, settings, uniform, out, readback};
    const uint32_t share = (n + kCtas - 1) / kCtas;
    constexpr size_t most = 200 * 1024;  // beside the kernel's static shared memory
    const size_t bytes = (size_t)share * 4 <= most ? (size_t)share * 4 : 0;
    cudaError_t e = ensure_dynamic_smem((const void*)sample_kernel, bytes);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(kCtas);
    config.blockDim = dim3(kSampleThreads);
    config.dynamicSmemBytes = bytes;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = kCtas;
    attributes[0].val.clusterDim.y = attributes[0].val.clusterDim.z = 1;
    attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attributes;
    config.numAttrs = pdl_enabled() ? 2 : 1;
    return cudaLaunchKernelEx(&config, sample_kernel, p, share, bytes ? 1 : 0);
}

}  // namespace k
}  // namespace bc
