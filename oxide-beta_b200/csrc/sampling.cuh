// Step bookkeeping and top-k selection kernels.
//
// step_begin / step_end replace the reference's one-thread decode_state_update / mark_seen
// launches (crates/oxide-torch-cuda/src/kernel_module.rs:1287-1317,1981-1986): the token ids and
// positions of every sequence live on the device so that a captured step can be replayed for any
// position. topk_stage1 / topk_stage2 produce the same list as the reference's two-stage top-k
// (kernel_module.rs:1988-2075): descending score, lowest index first among equal scores,
// repetition penalty applied to seen tokens, NaN never selected, unused slots (-inf, 0).
#pragma once
#include "common.cuh"

namespace oxg4 {

struct StepCtl {              // device-resident control words, written by the host before a step
    int32_t mark_seen;        // 1: seen[b][token[b]] = 1 at step begin
    int32_t feed_back;        // 1: next token[b] = arg-max of this step (device-resident greedy loop)
    int32_t step;             // steps run since the loop started (index into `history`)
    int32_t history_cap;      // capacity of `history` in steps
    int32_t sample;           // 1: the token fed back is drawn from the step's top-k list (sample_candidates_kernel)
    float temperature, top_p;
};

__global__ void step_begin_kernel(int B, int V, const uint32_t* tokens, uint8_t* seen, const StepCtl* ctl) {
    pdl_wait();
    pdl_launch();
    if (!ctl->mark_seen) return;
    for (int b = threadIdx.x; b < B; b += blockDim.x) {       // launched as a single block
        const uint32_t t = tokens[b];
        if (t != kInactiveToken && t < (uint32_t)V) seen[(size_t)b * V + t] = 1;
    }
}

__global__ void step_end_kernel(int B, uint32_t* tokens, int32_t* pos, const uint32_t* best_ids,
                                uint32_t* history, StepCtl* ctl) {
    pdl_wait();
    pdl_launch();
    const int fb = ctl->feed_back;
    const int step = ctl->step;
    const int hist_cap = ctl->history_cap;
    for (int b = threadIdx.x; b < B; b += blockDim.x) {       // launched as a single block
        if (tokens[b] == kInactiveToken) continue;
        pos[b] += 1;
        if (fb) {
            const uint32_t nxt = best_ids[b];
            if (step < hist_cap) history[(size_t)step * B + b] = nxt;
            tokens[b] = nxt;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && fb) ctl->step = step + 1;
}

// f32::total_cmp key (the reference sorts candidates with it, sampling.rs:88-158)
DEVINL int32_t total_order_key_dev(float f) {
    int32_t b = __float_as_int(f);
    b ^= (int32_t)(((uint32_t)(b >> 31)) >> 1);
    return b;
}

// The reference's sample_topk_candidates (crates/oxide-torch-models/src/models/gemma4/sampling.rs:88-158) on
// the device, one thread per sequence over the step's (<= 64) top-k candidates: temperature, stable
// descending sort, softmax, top-p cut, xorshift64 (13, 7, 17), 24-bit uniform, cumulative pick. The same
// f32 operations in the same order as the host version (oxg4_sample_topk_candidates); the generator state
// lives on the device so that a sampled generation loop needs no per-token host round trip. The chosen
// token replaces best_ids[b], which step_end feeds back. `softcap` > 0 applies tanh(x / cap) * cap first.
__global__ void sample_candidates_kernel(int B, int k, float softcap, const uint32_t* tokens, const uint32_t* cand_ids,
                                         const float* cand_scores, const StepCtl* ctl, unsigned long long* rng,
                                         uint32_t* best_ids, float* best_scores) {
    pdl_wait();
    pdl_launch();
    if (!ctl->sample) return;
    const float temperature = ctl->temperature, top_p = ctl->top_p;
    for (int b = threadIdx.x; b < B; b += blockDim.x) {       // launched as a single block
        if (tokens[b] == kInactiveToken) continue;
        uint32_t id[64];
        float v[64];
        int n = 0;
        for (int i = 0; i < k; ++i) {
            float s = cand_scores[(size_t)b * k + i];
            // final_logit_softcapping is applied to the candidate scores before they are sampled
            // (gemma4_cuda/mod.rs:573-579, decode.rs:644,746), as the host path does
            if (softcap > 0.0f) s = tanhf(s / softcap) * softcap;
            if (isfinite(s)) { id[n] = cand_ids[(size_t)b * k + i]; v[n] = s / temperature; ++n; }
        }
        if (n == 0) continue;                                  // keep the arg-max
        for (int i = 1; i < n; ++i) {                          // stable insertion sort, descending total order
            const float vi = v[i];
            const uint32_t ii = id[i];
            int j = i - 1;
            while (j >= 0 && total_order_key_dev(v[j]) < total_order_key_dev(vi)) { v[j + 1] = v[j]; id[j + 1] = id[j]; --j; }
            v[j + 1] = vi;
            id[j + 1] = ii;
        }
        const float maximum = v[0];
        float total = 0.0f;
        for (int i = 0; i < n; ++i) { v[i] = expf(v[i] - maximum); total += v[i]; }
        if (total == 0.0f || !isfinite(total)) continue;
        for (int i = 0; i < n; ++i) v[i] /= total;
        if (top_p < 1.0f) {
            float cumulative = 0.0f;
            int keep = 0;
            for (int i = 0; i < n; ++i) {
                cumulative += v[i];
                ++keep;
                if (cumulative >= top_p) break;
            }
            n = max(keep, 1);
            total = 0.0f;
            for (int i = 0; i < n; ++i) total += v[i];
        } else {
            total = 1.0f;
        }
        unsigned long long r = rng[b];
        if (r == 0) r = 0x4d595df4d0f33173ull;
        r ^= r << 13;
        r ^= r >> 7;
        r ^= r << 17;
        rng[b] = r;
        const float unit = __fdiv_rn((float)((uint32_t)(r >> 40)), 16777216.0f);
        float threshold = __fmul_rn(unit, total);
        int pick = n - 1;
        for (int i = 0; i < n; ++i) {
            if (threshold <= v[i]) { pick = i; break; }
            threshold = __fsub_rn(threshold, v[i]);
        }
        best_ids[b] = id[pick];
        best_scores[b] = v[pick];
    }
}

// Tensor parallelism: every rank holds the arg-max of its vocabulary slice; after an all-gather this
// picks the global winner (same tie-break as everywhere: higher score, then lower id).
__global__ void tp_pick_kernel(int B, int ranks, const float* all_scores, const uint32_t* all_ids,
                               uint32_t* ids, float* scores) {
    pdl_wait();
    pdl_launch();
    for (int b = threadIdx.x; b < B; b += blockDim.x) {
        Cand best{all_scores[b], all_ids[b]};
        for (int r = 1; r < ranks; ++r) {
            const Cand c{all_scores[(size_t)r * B + b], all_ids[(size_t)r * B + b]};
            if (cand_better(c, best)) best = c;
        }
        ids[b] = best.i;
        scores[b] = best.s;
    }
}

constexpr int kTopkThreads = 256;
constexpr int kTopkChunk = 2048;

// Top-k lists hold the best candidates in order: higher score first, lower id among equal scores. A candidate is compared as
// one 64-bit key; 0 stands for none (a score of minus infinity or NaN is never selected, a negative zero equals zero).
//
// Rounds of arg-max with removal over all candidates of a block cost two barriers and a scan each. Instead a warp
// picks the best of its 256 scores by itself (every lane keeps eight in order, a round is two warp reductions), and one warp
// merges sorted lists by their heads (1B model, 40 candidates of 262144 with a repetition penalty: a step with its list 1.50 ms, now
// 1.33; a step without one takes 1.24).
DEVINL uint64_t cand_key(float s, uint32_t id) {
    if (!(s > -INFINITY)) return 0;
    const uint32_t b = s == 0.0f ? 0u : __float_as_uint(s);
    return ((uint64_t)(b ^ ((b >> 31) ? 0xffffffffu : 0x80000000u)) << 32) | (uint32_t)~id;
}
DEVINL uint64_t warp_max_key(uint64_t k) {
    const uint32_t hi = __reduce_max_sync(0xffffffffu, (uint32_t)(k >> 32));
    const uint32_t lo = __reduce_max_sync(0xffffffffu, (uint32_t)(k >> 32) == hi ? (uint32_t)k : 0u);
    return ((uint64_t)hi << 32) | lo;
}

// The best top_k of `lists` sorted lists of `len` candidates each (at most 64), by one warp; out(r, where) receives the place of the r-th
// one in `c`, or -1 where there are no more. What is taken leaves its list, so that a list's best candidate is always its first: the
// merge needs no memory beside the lists, and takes as many of them as shared memory holds.
template <typename F>
DEVINL void merge_lists(Cand* c, int lists, int len, int top_k, F&& out) {
    const int lane = threadIdx.x & 31;
    uint64_t best = 0;
    int from = 0;
    auto look = [&]() {                                        // the best head of the lane's lists
        best = 0;
        for (int l = lane; l < lists; l += 32) {
            const Cand o = c[l * len];
            const uint64_t k = cand_key(o.s, o.i);
            if (k > best) { best = k; from = l; }
        }
    };
    look();
    for (int r = 0; r < top_k; ++r) {
        const uint64_t m = warp_max_key(best);
        if (m == 0) {
            if (lane == 0) out(r, -1);
            continue;
        }
        const bool mine = m == best;                           // ids are unique: one lane
        if (mine) out(r, from * len);
        Cand* list = c + __shfl_sync(0xffffffffu, from, __ffs(__ballot_sync(0xffffffffu, mine)) - 1) * len;
        Cand next[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int i = lane + 32 * q;
            if (i < len) next[q] = i + 1 < len ? list[i + 1] : Cand{-INFINITY, 0u};
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (lane + 32 * q < len) list[lane + 32 * q] = next[q];
        __syncwarp();
        if (mine) look();
    }
}

// grid (chunks, B): per-chunk sorted top-k over columns [col0, col0 + n_cols) of the [B, ld] logits (a
// tensor-parallel rank scans its own vocabulary slice); candidate ids are vocabulary ids
__global__ void __launch_bounds__(kTopkThreads)
topk_stage1_kernel(const float* logits, int ld, int col0, int n_cols, const uint8_t* seen, float penalty, int top_k,
                   Cand* stage) {
    constexpr int W = kTopkThreads / 32, E = kTopkChunk / kTopkThreads;
    __shared__ Cand list[W * 64];
    pdl_wait();
    pdl_launch();
    const int b = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int start = blockIdx.x * kTopkChunk;
    const int n = min(kTopkChunk, n_cols - start);
    const size_t base = (size_t)b * ld + col0 + start;
    // a lane's scores and keys, best first
    uint64_t key[E];
    float sc[E];
#pragma unroll
    for (int j = 0; j < E; ++j) {
        const int i = warp * 32 * E + j * 32 + lane;
        float s = -INFINITY;
        if (i < n) {
            s = logits[base + i];
            if (seen != nullptr && penalty > 1.0f && seen[base + i] != 0) s = s >= 0.0f ? s / penalty : s * penalty;
        }
        sc[j] = s;
    }
    if (top_k == 1) {                                          // arg-max: nothing to keep in order
        Cand c{-INFINITY, 0xffffffffu};
#pragma unroll
        for (int j = 0; j < E; ++j)
            if (sc[j] > c.s) c = Cand{sc[j], (uint32_t)(col0 + start + warp * 32 * E + j * 32 + lane)};
        c = warp_best(c);
        if (lane == 0) list[warp] = c;
        __syncthreads();
        if (warp != 0) return;
        c = warp_best(lane < W ? list[lane] : Cand{-INFINITY, 0xffffffffu});
        if (lane == 0) stage[(size_t)b * gridDim.x + blockIdx.x] = Cand{c.s, c.i == 0xffffffffu ? 0u : c.i};
        return;
    }
#pragma unroll
    for (int j = 0; j < E; ++j) key[j] = cand_key(sc[j], (uint32_t)(col0 + start + warp * 32 * E + j * 32 + lane));
#pragma unroll
    for (int p = 0; p < E; ++p)                                // odd-even transposition
#pragma unroll
        for (int j = p & 1; j + 1 < E; j += 2)
            if (key[j + 1] > key[j]) {
                const uint64_t k = key[j]; key[j] = key[j + 1]; key[j + 1] = k;
                const float t = sc[j]; sc[j] = sc[j + 1]; sc[j + 1] = t;
            }
    for (int r = 0; r < top_k; ++r) {
        const uint64_t m = warp_max_key(key[0]);
        if (m == 0) {
            if (lane == 0) list[warp * top_k + r] = Cand{-INFINITY, 0u};
        } else if (m == key[0]) {
            list[warp * top_k + r] = Cand{sc[0], ~(uint32_t)m};
#pragma unroll
            for (int j = 0; j + 1 < E; ++j) { key[j] = key[j + 1]; sc[j] = sc[j + 1]; }
            key[E - 1] = 0;
        }
    }
    __syncthreads();
    if (warp != 0) return;
    Cand* dst = stage + ((size_t)b * gridDim.x + blockIdx.x) * top_k;
    merge_lists(list, W, top_k, top_k, [&](int r, int where) { dst[r] = where < 0 ? Cand{-INFINITY, 0u} : list[where]; });
}

// Tensor parallelism: every rank holds the sorted top-k of its vocabulary slice; after an all-gather
// ([ranks][B][k] scores and ids) one block per sequence merges the ranks * k candidates into the global
// top-k (descending score, lower id first among equal scores, as everywhere).
__global__ void __launch_bounds__(kTopkThreads)
tp_topk_merge_kernel(int B, int ranks, int k, const float* all_scores, const uint32_t* all_ids, uint32_t* ids,
                     float* scores) {
    __shared__ Cand all[8 * 64];
    pdl_wait();
    pdl_launch();
    const int b = blockIdx.x, n = ranks * k;
    for (int i = threadIdx.x; i < n; i += kTopkThreads) {
        const size_t from = ((size_t)(i / k) * B + b) * k + i % k;
        all[i] = Cand{all_scores[from], all_ids[from]};
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    merge_lists(all, ranks, k, k, [&](int r, int where) {
        ids[(size_t)b * k + r] = where < 0 ? 0u : all[where].i;
        scores[(size_t)b * k + r] = where < 0 ? -INFINITY : all[where].s;
    });
}

// grid (1, B): merge of n / top_k sorted lists of top_k candidates; dynamic shared memory topk_merge_smem(n)
inline size_t topk_merge_smem(int n) { return (size_t)n * sizeof(Cand); }
__global__ void __launch_bounds__(kTopkThreads)
topk_stage2_kernel(const Cand* stage, int n, int top_k, uint32_t* ids, float* scores) {
    extern __shared__ __align__(16) unsigned char sm2[];
    Cand* all = reinterpret_cast<Cand*>(sm2);
    pdl_wait();
    pdl_launch();
    const int b = blockIdx.y;
    for (int i = threadIdx.x; i < n; i += kTopkThreads) all[i] = stage[(size_t)b * n + i];
    __syncthreads();
    if (threadIdx.x >= 32) return;
    merge_lists(all, n / top_k, top_k, top_k, [&](int r, int where) {
        ids[(size_t)b * top_k + r] = where < 0 ? 0u : all[where].i;
        scores[(size_t)b * top_k + r] = where < 0 ? -INFINITY : all[where].s;
    });
}

}  // namespace oxg4
