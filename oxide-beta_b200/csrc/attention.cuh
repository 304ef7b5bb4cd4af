// Decode attention over a paged KV cache: one launch per layer does what the reference spreads
// over slice_rows x3, rms_norm (q), rope_state (q), rms_norm (k), rope_state (k), rms_norm_unit
// (v), cache_write_f32_state x2 and gqa_decode_block_state
// (crates/oxide-torch-models/src/gemma4_cuda/decode.rs:82-157; device math in
// crates/oxide-torch-cuda/src/kernel_module.rs:1133-1246,1423-1439,1510-1550,1790-1894).
//
// attn_step_kernel, attn_decode_kernel: decode steps. attn_rows_kernel: rows whose K/V are in the cache already (prompt chunks, KV-shared layers). The
// visible positions of a sequence are partitioned into up to `n_splits` contiguous ranges, a CTA each (split-KV "flash decoding" with
// an online softmax per warp). Partial sums are added in a fixed order, so the result does not depend on scheduling. Attention
// scale is 1.0 as in the reference (no 1/sqrt(d)).
//
// Cache layout: pool[page][kv_head][token_in_page][head_dim]; a sequence's slot -> page mapping
// comes from its page table. Ring semantics follow the reference: slot = position % capacity,
// capacity = min(window, max_seq) on sliding layers (kernel_module.rs:1811-1831), so the ring
// itself implements the window.
//
// HBM-bound: bytes per launch = 2 * visible_positions * kv_heads * head_dim * sizeof(KV element).
#pragma once
#include <cooperative_groups.h>
#include <type_traits>

#include "common.cuh"

namespace oxg4 {

constexpr int kAttnThreads = 512;
constexpr int kAttnStepThreads = 256;     // attn_step_kernel: shares an SM with the projections around it
constexpr int kAttnWarps = kAttnThreads / 32;

struct AttnArgs {
    const float* qkv;        // [qkv_splits, split_rows, qkv_n] QKV projection output (K-split partials), columns q | k | v
    int qkv_n;
    int qkv_splits;          // partials to add (1 for the small-batch kernels)
    int split_rows;          // rows between two partials
    uint16_t* out_bf16;      // optional BF16 copy of the output, [B, Nq * D] (input of the tcgen05 O projection)
    int B, Nq, Nkv;
    const float* q_norm;     // [D]
    const float* k_norm;     // [D]
    const float* inv_freq;   // [D/2]: theta^(-2i/D) / factor
    int rotary_half;         // rotary_dim / 2; frequency lanes at or above it pass through
    float eps;
    const int32_t* pos;      // [B] absolute position of the token being processed
    const uint32_t* tokens;  // [B] (kInactiveToken rows are skipped)
    void* kpool;
    void* vpool;
    const int32_t* page_table;   // [B, pages_per_seq]
    int pages_per_seq, page_tokens;
    const int32_t* cap;      // [B] ring capacity of this layer kind for each sequence
    int window;              // a token sees the last `window` positions up to its own (sliding layers), INT_MAX otherwise
    int group;               // attn_step_kernel: query heads per kv head
    int early;               // attn_step_kernel: the dependent launch may start before this kernel waits for its predecessor
    const int32_t* row_seq;  // [B] sequence (page table, ring) of every row, or null: row b is sequence b
    int n_splits, min_split;
    float* part;             // [B, Nkv, n_splits, G, D + 2]
    unsigned int* ticket;    // [B, Nkv]
    float* out;              // [B, Nq * D]
    unsigned long long* ts;  // optional timeline slots of this launch (4 entries) or null
    unsigned long long* ts_mid;  // optional: further stamps inside the kernel (attn_step_kernel three, attn_decode_kernel one to four)
};

template <typename KT, int EPT> struct KVec;
template <> struct KVec<uint16_t, 8> {
    static DEVINL void load(const uint16_t* p, float (&o)[8]) {
        uint4 v = ldg_stream16(p);
        o[0] = bf16lo(v.x); o[1] = bf16hi(v.x); o[2] = bf16lo(v.y); o[3] = bf16hi(v.y);
        o[4] = bf16lo(v.z); o[5] = bf16hi(v.z); o[6] = bf16lo(v.w); o[7] = bf16hi(v.w);
    }
};
template <> struct KVec<uint16_t, 4> {
    static DEVINL void load(const uint16_t* p, float (&o)[4]) {
        uint2 v = ldg_stream8(p);
        o[0] = bf16lo(v.x); o[1] = bf16hi(v.x); o[2] = bf16lo(v.y); o[3] = bf16hi(v.y);
    }
};
template <> struct KVec<uint16_t, 2> {
    static DEVINL void load(const uint16_t* p, float (&o)[2]) {
        uint32_t v = ldg_stream4(p);
        o[0] = bf16lo(v); o[1] = bf16hi(v);
    }
};
template <> struct KVec<float, 8> {
    static DEVINL void load(const float* p, float (&o)[8]) {
        uint4 a = ldg_stream16(p), b = ldg_stream16(p + 4);
        o[0] = __uint_as_float(a.x); o[1] = __uint_as_float(a.y); o[2] = __uint_as_float(a.z);
        o[3] = __uint_as_float(a.w); o[4] = __uint_as_float(b.x); o[5] = __uint_as_float(b.y);
        o[6] = __uint_as_float(b.z); o[7] = __uint_as_float(b.w);
    }
};
template <> struct KVec<float, 4> {
    static DEVINL void load(const float* p, float (&o)[4]) {
        uint4 a = ldg_stream16(p);
        o[0] = __uint_as_float(a.x); o[1] = __uint_as_float(a.y); o[2] = __uint_as_float(a.z);
        o[3] = __uint_as_float(a.w);
    }
};
template <> struct KVec<float, 2> {
    static DEVINL void load(const float* p, float (&o)[2]) {
        uint2 a = ldg_stream8(p);
        o[0] = __uint_as_float(a.x); o[1] = __uint_as_float(a.y);
    }
};

// A lane's slice of one K or V row as loaded (packed), converted only when it is consumed, so that
// the next positions' loads can be in flight in few registers.
template <typename KT, int EPT> struct KRaw {
    static constexpr int NWORDS = EPT * (int)sizeof(KT) / 4;
    uint32_t w[NWORDS];
};
template <typename KT, int EPT> DEVINL void kraw_load(const KT* p, KRaw<KT, EPT>& r) {
    constexpr int NWD = KRaw<KT, EPT>::NWORDS;
    if constexpr (NWD == 8) {
        const uint4 x = ldg_stream16(p), y = ldg_stream16((const char*)p + 16);
        r.w[0] = x.x; r.w[1] = x.y; r.w[2] = x.z; r.w[3] = x.w; r.w[4] = y.x; r.w[5] = y.y; r.w[6] = y.z; r.w[7] = y.w;
    } else if constexpr (NWD == 4) {
        const uint4 x = ldg_stream16(p);
        r.w[0] = x.x; r.w[1] = x.y; r.w[2] = x.z; r.w[3] = x.w;
    } else if constexpr (NWD == 2) {
        const uint2 x = ldg_stream8(p);
        r.w[0] = x.x; r.w[1] = x.y;
    } else {
        r.w[0] = ldg_stream4(p);
    }
}
template <typename KT, int EPT> DEVINL void kraw_cvt(const KRaw<KT, EPT>& r, float (&o)[EPT]) {
    if constexpr (sizeof(KT) == 2) {
#pragma unroll
        for (int i = 0; i < EPT / 2; ++i) { o[2 * i] = bf16lo(r.w[i]); o[2 * i + 1] = bf16hi(r.w[i]); }
    } else {
#pragma unroll
        for (int i = 0; i < EPT; ++i) o[i] = __uint_as_float(r.w[i]);
    }
}

template <typename KT> DEVINL KT kv_store_cvt(float v);
template <> DEVINL float kv_store_cvt<float>(float v) { return v; }
template <> DEVINL uint16_t kv_store_cvt<uint16_t>(float v) { return (uint16_t)f32_to_bf16_bits(v); }
template <typename KT> DEVINL float kv_widen(KT v);
template <> DEVINL float kv_widen<float>(float v) { return v; }
template <> DEVINL float kv_widen<uint16_t>(uint16_t v) { return __uint_as_float((uint32_t)v << 16); }

struct BarCta {
    DEVINL void operator()() const { __syncthreads(); }
};

// Norm of one head (times w) and, with `rotate`, its rotation: channel d rotates with d + D / 2, sixteen lanes away; cs(e) and sn(e) are
// the factors of this lane's channels (sn negated in the first half), 1 and 0 past the rotated ones. The result is rounded once. Element by
// element, as the K/V rows of the first round occupy most registers meanwhile.
template <typename NT, int EPT, typename C, typename S>
DEVINL void norm_rotate(float (&t)[EPT], const float (&w)[EPT], const C& cs, const S& sn, float eps, bool rotate) {
    NT ss = 0;
#pragma unroll
    for (int e = 0; e < EPT; ++e) ss += (NT)t[e] * (NT)t[e];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const NT r = (NT)1 / sqrt(ss / (NT)(32 * EPT) + (NT)eps);
    if (rotate) {                                      // one branch around the shuffles, not one for each of them
#pragma unroll
        for (int e = 0; e < EPT; ++e) {
            const NT v = (NT)t[e] * r * (NT)w[e];
            t[e] = (float)(v * (NT)cs(e) + __shfl_xor_sync(0xffffffffu, v, 16) * (NT)sn(e));
        }
    } else {
#pragma unroll
        for (int e = 0; e < EPT; ++e) t[e] = (float)((NT)t[e] * r * (NT)w[e]);
    }
}
// With an f32 cache norm and rotation of a step's token are done in doubles: their roundings in q and k were most of the error of
// the scores, and with it of an f32 model.
template <typename KT> using NormT = typename std::conditional<sizeof(KT) == 4, double, float>::type;

// One CTA's share of a launch: split `s` of kv head `kvh` of sequence `b`, computed by the `nthreads`
// threads that call it (tid = threadIdx.x < nthreads). `sm` is attn_cta_floats() floats of shared memory.
template <typename KT, int D, int G, bool CL, bool DEEP, typename BAR>
DEVINL void attn_cta(const AttnArgs& a, float* sm, const int s, const int kvh, const int b, const int nthreads,
                     const BAR bar) {
    constexpr int EPT = D / 32;
    const int NW = nthreads >> 5;            // 16 warps when few CTAs exist (latency), 4 when many (occupancy)
    float* qs = sm;                          // [G][D]
    float* kcur = qs + G * D;                // [D]
    float* vcur = kcur + D;                  // [D]
    float* wm = qs + G * D + (CL ? 2 * D : 0);   // [NW][G]
    float* wl = wm + NW * G;                 // [NW][G]
    float* wacc = wl + NW * G;               // [NW][G][D]
    float* cpart = wacc + NW * G * D;        // [G][D + 2] this CTA's partial (cluster variant)
    float* rope = cpart + (CL ? G * (D + 2) : 0);   // [D] cos (first half) and sin (second half) of pos * inv_freq
    __shared__ unsigned int s_last;
    __shared__ float s_scale[16 * 8], s_l[16 * 8], s_M[8];   // merge scratch: up to 16 warps or cluster splits x 8 heads

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int half = D / 2;

    // The variant that merges through global memory (CL = false) serves the rows of a prompt chunk: K and V of
    // every row, the current position included, are already in the cache (qkv_post_kernel appended the whole
    // chunk first), so the CTA only norms its queries.
    constexpr bool ext = !CL;
    // model constants for this lane's slice of a head: fetched before the dependency wait
    float w[EPT];                            // CL: of this warp's first task, see below
    auto load_w = [&](int task) {
#pragma unroll
        for (int e = 0; e < EPT; ++e) w[e] = task < G || ext ? a.q_norm[lane * EPT + e] : task == G ? a.k_norm[lane * EPT + e] : 1.0f;
    };
    load_w(warp);
    // Step state (token, position, ring capacity, page table) and the K/V rows of earlier positions were complete before the step's
    // first kernel (which waits before it lets its successor start), a chunk's row data before the chunk: they may be read, and the
    // rotation factors computed, ahead of the dependency wait.
    const bool active = a.tokens[b] != kInactiveToken;
    const int pos = a.pos[b];
    const int sb = a.row_seq ? a.row_seq[b] : b;
    const int cap = a.cap[sb];
    const int lo = max(0, pos + 1 - min(cap, a.window));
    const int n = pos - lo + 1;
    const int n_eff = min(a.n_splits, (n + a.min_split - 1) / a.min_split);
    const bool has_work = active && s < n_eff;
    float* part = a.part + (((size_t)b * a.Nkv + kvh) * a.n_splits) * (size_t)(G * (D + 2));
    size_t cur_off = 0;
    // this CTA's range of positions, and the loads of its first step: K/V rows of earlier positions were
    // written by earlier steps, so they can be in flight while the QKV projection finishes and while the
    // prologue below runs
    const int begin = has_work ? lo + (int)(((long long)n * s) / n_eff) : 0;
    const int end = has_work ? lo + (int)(((long long)n * (s + 1)) / n_eff) : 0;
    constexpr int PD = DEEP ? 4 : 2;
    typedef KRaw<KT, EPT> Raw;
    const KT* kpool = (const KT*)a.kpool;
    const KT* vpool = (const KT*)a.vpool;
    const int32_t* pt = a.page_table + (size_t)sb * a.pages_per_seq;
    auto row_offset = [&](int p) -> size_t {
        const int slot = p % cap;
        return (((size_t)pt[slot / a.page_tokens] * a.Nkv + kvh) * a.page_tokens +
                (slot % a.page_tokens)) * (size_t)D + lane * EPT;
    };
    auto issue = [&](int p, Raw& kr, Raw& vr) {            // loads only; the current token comes from shared memory
        if (p < end && (p != pos || ext)) {
            const size_t off = row_offset(p);
            kraw_load<KT, EPT>(kpool + off, kr);
            kraw_load<KT, EPT>(vpool + off, vr);
        }
    };
    Raw kr[PD], vr[PD];
    if (has_work && !ext) {
#pragma unroll
        for (int q = 0; q < PD; ++q) issue(begin + warp + q * NW, kr[q], vr[q]);
    }
    if (has_work) {
        const int slot_cur = pos % cap;
        cur_off = (((size_t)pt[slot_cur / a.page_tokens] * a.Nkv + kvh) *
                       a.page_tokens + (slot_cur % a.page_tokens)) * (size_t)D;
        // rotation factors of this position, one cosf or sinf per thread instead of 2 * D / 32 per lane
        for (int i = tid; i < D; i += nthreads) {
            const int fi = i % half;
            if (fi < a.rotary_half) {
                const float angle = (float)pos * a.inv_freq[fi];
                rope[i] = i < half ? cosf(angle) : sinf(angle);
            }
        }
    }
    stamp(a.ts, 0);
    pdl_wait();
    pdl_launch();
    stamp(a.ts, 1);
    if (has_work && ext) {
        // rows of a prompt chunk: the K/V rows of this very chunk were appended by the preceding kernel, so
        // nothing may be read from the cache before the dependency wait
#pragma unroll
        for (int q = 0; q < PD; ++q) issue(begin + warp + q * NW, kr[q], vr[q]);
    }

    if (has_work) {
        const bool owner = (s == n_eff - 1);        // the range that contains `pos`
        bar();                                      // the rotation factors are in shared memory
        // tasks 0..G-1: query heads (norm + rope); task G: key (norm + rope + append);
        // task G+1: value (unit norm + append). One warp per task.
        const int n_tasks = (owner && !ext) ? G + 2 : G;
        for (int task = warp; task < n_tasks; task += NW) {
            int col;
            if (task < G) col = (kvh * G + task) * D;
            else if (task == G) col = a.Nq * D + kvh * D;
            else col = (a.Nq + a.Nkv) * D + kvh * D;
            float t[EPT];
            float ss = 0.0f;
#pragma unroll
            for (int e = 0; e < EPT; ++e) {
                float v = 0.0f;
                for (int sp = 0; sp < a.qkv_splits; ++sp)
                    v += __ldcg(a.qkv + ((size_t)sp * a.split_rows + b) * a.qkv_n + col + lane * EPT + e);
                t[e] = v;
                ss += v * v;
            }
            float* dst = task < G ? qs + task * D : (task == G ? kcur : vcur);
            if constexpr (CL) {
                if (task != warp) load_w(task);
                const float* f = rope + (lane & 15) * EPT;
                norm_rotate<NormT<KT>>(t, w, [&](int e) { return f[e]; }, [&](int e) { return lane < 16 ? -f[half + e] : f[half + e]; }, a.eps, task <= G);
#pragma unroll
                for (int e = 0; e < EPT; ++e) dst[lane * EPT + e] = t[e];
            } else {
                ss = warp_sum(ss);
                const float r = 1.0f / sqrtf(ss / (float)D + a.eps);
#pragma unroll
                for (int e = 0; e < EPT; ++e) dst[lane * EPT + e] = t[e] * r * w[e];
                __syncwarp();
                float o[EPT];
#pragma unroll
                for (int e = 0; e < EPT; ++e) {
                    const int d = lane * EPT + e;
                    const int fi = d % half;
                    float v = dst[d];
                    if (fi < a.rotary_half) {
                        const float pv = dst[d < half ? d + half : d - half];
                        const float rotated = d < half ? -pv : pv;
                        v = v * rope[fi] + rotated * rope[half + fi];
                    }
                    o[e] = v;
                }
                __syncwarp();
#pragma unroll
                for (int e = 0; e < EPT; ++e) dst[lane * EPT + e] = o[e];
            }
            if (task >= G) {
                // append to the cache; keep the stored (possibly BF16-rounded) value for this step
                KT* pool = (KT*)(task == G ? a.kpool : a.vpool);
                __syncwarp();
#pragma unroll
                for (int e = 0; e < EPT; ++e) {
                    const int d = lane * EPT + e;
                    const KT stored = kv_store_cvt<KT>(dst[d]);
                    pool[cur_off + d] = stored;
                    dst[d] = kv_widen<KT>(stored);
                }
            }
        }
        bar();
        stamp(a.ts, 2);

        float q_[G][EPT];
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int e = 0; e < EPT; ++e) q_[g][e] = qs[g * D + lane * EPT + e];
        float m[G], l[G], acc[G][EPT];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            m[g] = -INFINITY;
            l[g] = 0.0f;
#pragma unroll
            for (int e = 0; e < EPT; ++e) acc[g][e] = 0.0f;
        }
        // The PD positions of a step: all PD * G dot products first, their butterfly reductions interleaved
        // (PD * G independent shuffles per level instead of one dependent chain per score), then the
        // updates in position order.
        auto use_step = [&](int p0, const Raw* kr, const Raw* vr, auto pd_tag) {
            constexpr int NP = decltype(pd_tag)::value;
            float sc[NP][G];
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                const int pq = p0 + q * NW;
                float kf[EPT];
                if (pq == pos && !ext) {
#pragma unroll
                    for (int e = 0; e < EPT; ++e) kf[e] = kcur[lane * EPT + e];
                } else {
                    kraw_cvt<KT, EPT>(kr[q], kf);          // rows past `end` were never loaded: their scores are not used
                }
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    float t = 0.0f;
#pragma unroll
                    for (int e = 0; e < EPT; ++e) t = fmaf(q_[g][e], kf[e], t);
                    sc[q][g] = t;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int q = 0; q < NP; ++q)
#pragma unroll
                    for (int g = 0; g < G; ++g) sc[q][g] += __shfl_xor_sync(0xffffffffu, sc[q][g], o);
            // one online-softmax step for the NP positions together: a single rescale of the running sums
            float pe[NP][G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float mn = m[g];
#pragma unroll
                for (int q = 0; q < NP; ++q)
                    if (p0 + q * NW < end) mn = fmaxf(mn, sc[q][g]);
                const float corr = expf(m[g] - mn);       // exp(-inf) = 0 on the first step
                float ls = l[g] * corr;
#pragma unroll
                for (int q = 0; q < NP; ++q) {
                    pe[q][g] = (p0 + q * NW < end) ? expf(sc[q][g] - mn) : 0.0f;
                    ls += pe[q][g];
                }
                l[g] = ls;
                m[g] = mn;
#pragma unroll
                for (int e = 0; e < EPT; ++e) acc[g][e] *= corr;
            }
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                const int pq = p0 + q * NW;
                if (pq >= end) break;
                float vf[EPT];
                if (pq == pos && !ext) {
#pragma unroll
                    for (int e = 0; e < EPT; ++e) vf[e] = vcur[lane * EPT + e];
                } else {
                    kraw_cvt<KT, EPT>(vr[q], vf);
                }
#pragma unroll
                for (int g = 0; g < G; ++g)
#pragma unroll
                    for (int e = 0; e < EPT; ++e) acc[g][e] = fmaf(pe[q][g], vf[e], acc[g][e]);
            }
        };
        // PD positions per step, the next step's loads issued before this step's arithmetic: 2 * PD rows of
        // K and of V in flight per warp (PD = 4 when one sequence has the whole GPU and latency is all that counts)
        for (int p = begin + warp; p < end; p += PD * NW) {
            Raw nk[PD], nv[PD];
#pragma unroll
            for (int q = 0; q < PD; ++q) issue(p + (PD + q) * NW, nk[q], nv[q]);
            use_step(p, kr, vr, std::integral_constant<int, PD>{});
#pragma unroll
            for (int q = 0; q < PD; ++q) { kr[q] = nk[q]; vr[q] = nv[q]; }
        }

        stamp(a.ts_mid, 1);
        // merge the warps of this CTA (fixed warp order)
#pragma unroll
        for (int g = 0; g < G; ++g) {
            if (lane == 0) { wm[warp * G + g] = m[g]; wl[warp * G + g] = l[g]; }
#pragma unroll
            for (int e = 0; e < EPT; ++e) wacc[((size_t)warp * G + g) * D + lane * EPT + e] = acc[g][e];
        }
        bar();
        // one scale factor exp(m_w - M) per (warp, head), computed once instead of once per output element
        if (tid < NW * G) {
            const int g = tid % G;
            float M = -INFINITY;
            for (int w = 0; w < NW; ++w) M = fmaxf(M, wm[w * G + g]);
            const float mw = wm[tid];
            s_scale[tid] = (mw == -INFINITY) ? 0.0f : expf(mw - M);
            if (tid < G) s_M[g] = M;
        }
        bar();
        float* my = CL ? cpart : part + (size_t)s * (G * (D + 2));
        for (int idx = tid; idx < G * D; idx += nthreads) {
            const int g = idx / D, d = idx % D;
            float A = 0.0f, L = 0.0f;
            for (int w = 0; w < NW; ++w) {
                const float e = s_scale[w * G + g];
                A += e * wacc[((size_t)w * G + g) * D + d];
                L += e * wl[w * G + g];
            }
            my[g * (D + 2) + d] = A;
            if (d == 0) { my[g * (D + 2) + D] = s_M[g]; my[g * (D + 2) + D + 1] = L; }
        }
    }

    if constexpr (CL) {
        // ---- cluster merge: every CTA finishes a slice of the outputs from its peers' shared memory ----
        namespace cg = cooperative_groups;
        cg::cluster_group cluster = cg::this_cluster();
        stamp(a.ts_mid, 2);
        cluster.sync();                                    // every CTA of the cluster arrives, with or without work
        stamp(a.ts_mid, 3);
        if (active) {
            // (m, l) of every split -> this CTA's shared memory in one round of remote loads, then one scale
            // factor per (split, head); the weighted sums below are independent remote loads
            if (tid < n_eff * G) {
                const int sp = tid / G, g = tid % G;
                const float* ps = cluster.map_shared_rank(cpart, sp) + g * (D + 2);
                s_scale[tid] = ps[D];
                s_l[tid] = ps[D + 1];
            }
            bar();
            if (tid < G) {
                const int g = tid;
                float M = -INFINITY;
                for (int sp = 0; sp < n_eff; ++sp) M = fmaxf(M, s_scale[sp * G + g]);
                float L = 0.0f;
                for (int sp = 0; sp < n_eff; ++sp) {
                    const float ms = s_scale[sp * G + g];
                    const float e = (ms == -INFINITY) ? 0.0f : expf(ms - M);
                    s_scale[sp * G + g] = e;
                    L += e * s_l[sp * G + g];
                }
                s_M[g] = L;
            }
            bar();
            const int cs = (int)gridDim.x;
            const int per = (G * D + cs - 1) / cs;
            const int hi = min(G * D, (s + 1) * per);
            for (int idx = s * per + tid; idx < hi; idx += nthreads) {
                const int g = idx / D, d = idx % D;
                float A = 0.0f;
                for (int sp = 0; sp < n_eff; ++sp)
                    A += s_scale[sp * G + g] * cluster.map_shared_rank(cpart, sp)[g * (D + 2) + d];
                {
                    const size_t oi = (size_t)b * a.Nq * D + (size_t)(kvh * G + g) * D + d;
                    const float ov = A / s_M[g];
                    a.out[oi] = ov;
                    if (a.out_bf16) a.out_bf16[oi] = (uint16_t)f32_to_bf16_bits(ov);
                }
            }
        }
        cluster.sync();                                    // no CTA leaves while a peer may still read its partial
        stamp(a.ts, 3);
        return;
    }
    // ---- last CTA of this (sequence, kv head) merges the split partials in split order ----
    stamp(a.ts_mid, 0);
    __threadfence();
    bar();
    if (tid == 0)
        s_last = (atomicAdd(&a.ticket[b * a.Nkv + kvh], 1u) == (unsigned)a.n_splits - 1u) ? 1u : 0u;
    bar();
    if (s_last) {
        __threadfence();
        if (active) {
            // (m, l) of every split -> shared memory, one scale factor per (split, head), then the
            // weighted sum over splits with independent loads (fixed split order)
            constexpr int PS = G * (D + 2);
            float* sf = wacc;                         // [n_eff][G] m, then exp(m - M)
            float* sl = wacc + a.n_splits * G;        // [n_eff][G] l
            float* sL = sl + a.n_splits * G;          // [G]
            for (int idx = tid; idx < n_eff * G; idx += nthreads) {
                const int sp = idx / G, g = idx % G;
                sf[idx] = __ldcg(part + (size_t)sp * PS + g * (D + 2) + D);
                sl[idx] = __ldcg(part + (size_t)sp * PS + g * (D + 2) + D + 1);
            }
            bar();
            for (int g = warp; g < G; g += NW) {               // a CTA of many has four warps, a group up to eight heads
                float M = -INFINITY;
                for (int sp = lane; sp < n_eff; sp += 32) M = fmaxf(M, sf[sp * G + g]);
                M = warp_max(M);
                float L = 0.0f;
                for (int sp = lane; sp < n_eff; sp += 32) {
                    const float ms = sf[sp * G + g];
                    const float e = (ms == -INFINITY) ? 0.0f : expf(ms - M);
                    sf[sp * G + g] = e;
                    L += e * sl[sp * G + g];
                }
                L = warp_sum(L);
                if (lane == 0) sL[g] = L;
            }
            bar();
            for (int idx = tid; idx < G * D; idx += nthreads) {
                const int g = idx / D, d = idx % D;
                const float* ps = part + g * (D + 2) + d;
                float A = 0.0f;
                // sixteen independent loads in flight per round trip to L2
                for (int s0 = 0; s0 < n_eff; s0 += 16) {
                    float v[16];
#pragma unroll
                    for (int q = 0; q < 16; ++q) v[q] = (s0 + q < n_eff) ? __ldcg(ps + (size_t)(s0 + q) * PS) : 0.0f;
#pragma unroll
                    for (int q = 0; q < 16; ++q)
                        if (s0 + q < n_eff) A += sf[(s0 + q) * G + g] * v[q];
                }
                {
                    const size_t oi = (size_t)b * a.Nq * D + (size_t)(kvh * G + g) * D + d;
                    const float ov = A / sL[g];
                    a.out[oi] = ov;
                    if (a.out_bf16) a.out_bf16[oi] = (uint16_t)f32_to_bf16_bits(ov);
                }
            }
        }
        if (tid == 0) a.ticket[b * a.Nkv + kvh] = 0u;
    }
    stamp(a.ts, 3);
}

// Decode steps of many units over many positions (attn_step_kernel takes the others). CL: the splits of one (sequence, kv head) form a
// thread-block cluster (gridDim.x <= 16 CTAs); partials stay in shared memory and are merged through distributed shared memory after one
// cluster barrier; the CTA that owns the current position also norms, rotates and appends its K and V.
// CTAs per SM that the registers are cut for. Head size 256 with rows ahead: one, its own choice of 64 registers spilled 800 bytes. 128 with a
// BF16 cache: two, so that a launch behind one that fills its SMs starts on the first half of them that are free (5 us a layer of the ~27B widths).
template <typename KT, int D, bool DEEP> constexpr int decode_ctas() { return !DEEP ? 0 : D == 256 ? 1 : D == 128 && sizeof(KT) == 2 ? 2 : 0; }
template <typename KT, int D, int G, bool DEEP>
__global__ void __launch_bounds__(kAttnThreads, decode_ctas<KT, D, DEEP>()) attn_decode_kernel(const AttnArgs a) {
    extern __shared__ __align__(16) float attn_sm[];
    attn_cta<KT, D, G, true, DEEP>(a, attn_sm, blockIdx.x, blockIdx.y, blockIdx.z, blockDim.x, BarCta{});
}

// Rows whose K/V are in the cache already (a prompt chunk, a KV-shared layer): partials go through global memory and the
// last CTA to arrive (atomic ticket) merges them.
template <typename KT, int D, int G>
__global__ void __launch_bounds__(kAttnThreads) attn_rows_kernel(const AttnArgs a) {
    extern __shared__ __align__(16) float attn_sm[];
    attn_cta<KT, D, G, false, false>(a, attn_sm, blockIdx.x, blockIdx.y, blockIdx.z, blockDim.x, BarCta{});
}

// Floats of shared memory of the two with NW warps per CTA
template <bool CL> inline size_t attn_cta_floats(int D, int G, int NW) {
    return (size_t)G * D + (CL ? 2 * D + G * (D + 2) : 0) + 2 * NW * G + (size_t)NW * G * D + D;
}

// ---- decode steps ----------------------------------------------------------------------------------------------------
DEVINL uint32_t map_cluster(const void* p, uint32_t rank) {      // shared-memory address of the same place in CTA `rank` of the cluster
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
template <int N> DEVINL void st_cluster(uint32_t addr, const float* v) {
    if constexpr (N >= 4) {
#pragma unroll
        for (int i = 0; i < N; i += 4)
            asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr + 4 * i), "f"(v[i]), "f"(v[i + 1]), "f"(v[i + 2]), "f"(v[i + 3]) : "memory");
    } else {
        asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v[0]), "f"(v[1]) : "memory");
    }
}
template <int N> DEVINL void load_row_piece(const float* p, float (&v)[N]) {
    if constexpr (N >= 4) {
#pragma unroll
        for (int i = 0; i < N; i += 4) {
            const float4 x = __ldcg(reinterpret_cast<const float4*>(p + i));
            v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
        }
    } else {
        const float2 x = __ldcg(reinterpret_cast<const float2*>(p));
        v[0] = x.x; v[1] = x.y;
    }
}

// Floats of shared memory of attn_step_kernel with NW warps per CTA and clusters of `splits` CTAs
template <int D, int G> inline size_t attn_step_floats(int NW, int splits) {
    return (size_t)(G + 3) * D + (size_t)NW * G * D + (size_t)2 * splits * NW * G + 64 * NW;
}

// One token per sequence. Grid (split, unit, sequence), the splits of a unit form a thread-block cluster. A unit is G of the
// query heads of one kv head: all of them, or, with few sequences, fewer, as long as the CTAs still have an SM each
// (a CTA's time is a chain of latencies and not the K/V bytes, which the other units of the kv head find in L2).
//
// The CTA norms and rotates its queries; the CTA whose range holds the current position also makes k and v, uses the stored
// values, and (first unit of the kv head) appends them. Each warp runs an online softmax over its positions and then pushes its
// un-normalised sums to the CTAs of the cluster that own them (every CTA finishes a slice of the outputs): no merge inside the
// CTA, and one cluster barrier instead of a round of remote loads between two. At 272 positions of the ~4B model (8 units of 16
// CTAs where there were 4 with two heads each) the launch went from 12.6 to 7.0 us of the step; one sequence of the ~1B model with an
// f32 cache, 512 positions: 15.9 to 7.4 us.
// Ahead of the dependency wait: step state, rotation factors and the K/V rows of earlier positions. All of it was complete before
// the step's first kernel let its successor start.
template <typename KT, int D, int G>
__global__ void __launch_bounds__(kAttnStepThreads, 2) attn_step_kernel(const AttnArgs a) {
    constexpr int EPT = D / 32, HALF = D / 2;
    constexpr int PD = G <= 2 ? 4 : 2;                 // positions of a warp per round
    constexpr bool DB = sizeof(KT) == 2 || G > 2;      // the next round's rows are loaded ahead of this round's arithmetic
    extern __shared__ __align__(16) float attn_sm[];
    const int NW = blockDim.x >> 5, ns = gridDim.x;
    float* qs = attn_sm;                               // [G][D]
    float* kcur = qs + G * D;                          // [D]
    float* vcur = kcur + D;                            // [D]
    float* rope = vcur + D;                            // [D]: cos (first half) and sin (second half) of pos * inv_freq
    float* in_acc = rope + D;                          // [ns * NW][per] sums pushed by the cluster's warps for this CTA's outputs
    float* in_ml = in_acc + NW * G * D;                // [ns * NW][G][2]
    float* red = in_ml + 2 * ns * NW * G;              // [2][threads]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int s = blockIdx.x, b = blockIdx.z;
    const int hsplit = a.group / G, kvh = blockIdx.y / hsplit, head0 = kvh * a.group + (blockIdx.y % hsplit) * G;
    const int per = G * D / ns;                        // outputs that this CTA finishes (powers of two)
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // waited for ahead of the first remote store

    // ---- ahead of the dependency wait ----
    const bool active = a.tokens[b] != kInactiveToken;
    const int pos = a.pos[b], cap = a.cap[b];
    const int lo = max(0, pos + 1 - min(cap, a.window));
    const int n = pos - lo + 1;
    const int n_eff = min(ns, (n + a.min_split - 1) / a.min_split);
    const bool has_work = active && s < n_eff;
    const int begin = has_work ? lo + (int)(((long long)n * s) / n_eff) : 0;
    const int end = has_work ? lo + (int)(((long long)n * (s + 1)) / n_eff) : 0;
    typedef KRaw<KT, EPT> Raw;
    const KT* kpool = (const KT*)a.kpool;
    const KT* vpool = (const KT*)a.vpool;
    const int32_t* pt = a.page_table + (size_t)b * a.pages_per_seq;
    auto row_offset = [&](int p) -> size_t {
        const int slot = p % cap;
        return (((size_t)pt[slot / a.page_tokens] * a.Nkv + kvh) * a.page_tokens + (slot % a.page_tokens)) * (size_t)D + lane * EPT;
    };
    auto issue = [&](int p, Raw& kr, Raw& vr) {        // loads only; the current token comes from shared memory
        if (p < end && p != pos) {
            const size_t off = row_offset(p);
            kraw_load<KT, EPT>(kpool + off, kr);
            kraw_load<KT, EPT>(vpool + off, vr);
        }
    };
    Raw kr[PD], vr[PD];
    if (has_work) {
#pragma unroll
        for (int q = 0; q < PD; ++q) issue(begin + warp + q * NW, kr[q], vr[q]);
        // rotation factors of this position, one cosf or sinf per thread
        for (int i = tid; i < D; i += blockDim.x) {
            const int fi = i % HALF;
            float f = i < HALF ? 1.0f : 0.0f;
            if (fi < a.rotary_half) {
                const float angle = (float)pos * a.inv_freq[fi];
                f = i < HALF ? cosf(angle) : sinf(angle);
            }
            rope[i] = f;
        }
    }
    __syncthreads();
    // tasks 0 .. G-1: query heads (norm + rotation), G: key (norm + rotation + append), G+1: value (unit norm + append); one warp each
    const bool owner = s == n_eff - 1;                 // its range contains `pos`
    const int n_tasks = has_work ? (owner ? G + 2 : G) : 0;
    float cs[EPT], sn[EPT], w[EPT];
    const size_t cur = has_work ? row_offset(pos) : 0;
    if (warp < n_tasks) {
#pragma unroll
        for (int e = 0; e < EPT; ++e) {
            const int fi = (lane & 15) * EPT + e;
            cs[e] = rope[fi];
            sn[e] = lane < 16 ? -rope[HALF + fi] : rope[HALF + fi];
            w[e] = warp <= G ? (warp < G ? a.q_norm : a.k_norm)[lane * EPT + e] : 1.0f;
        }
    }
    stamp(a.ts, 0);
    if (a.early) pdl_launch();
    pdl_wait();
    if (!a.early) pdl_launch();
    stamp(a.ts, 1);

    for (int task = warp; task < n_tasks; task += NW) {
        const int col = (task < G ? head0 + task : task == G ? a.Nq + kvh : a.Nq + a.Nkv + kvh) * D + lane * EPT;
        float t[EPT];
        load_row_piece<EPT>(a.qkv + (size_t)b * a.qkv_n + col, t);
        for (int sp = 1; sp < a.qkv_splits; ++sp) {
            float u[EPT];
            load_row_piece<EPT>(a.qkv + ((size_t)sp * a.split_rows + b) * a.qkv_n + col, u);
#pragma unroll
            for (int e = 0; e < EPT; ++e) t[e] += u[e];
        }
        if (task != warp) {                            // a second task of the warp
#pragma unroll
            for (int e = 0; e < EPT; ++e) {
                const int fi = (lane & 15) * EPT + e;
                cs[e] = rope[fi];
                sn[e] = lane < 16 ? -rope[HALF + fi] : rope[HALF + fi];
                w[e] = task <= G ? (task < G ? a.q_norm : a.k_norm)[lane * EPT + e] : 1.0f;
            }
        }
        norm_rotate<NormT<KT>>(t, w, [&](int e) { return cs[e]; }, [&](int e) { return sn[e]; }, a.eps, task <= G);
        float* dst = (task < G ? qs + task * D : task == G ? kcur : vcur) + lane * EPT;
        if (task >= G) {
            // the stored (possibly BF16-rounded) value is what this step uses too
            KT* pool = (KT*)(task == G ? a.kpool : a.vpool);
#pragma unroll
            for (int e = 0; e < EPT; ++e) {
                const KT stored = kv_store_cvt<KT>(t[e]);
                if (blockIdx.y % hsplit == 0) pool[cur + e] = stored;
                t[e] = kv_widen<KT>(stored);
            }
        }
#pragma unroll
        for (int e = 0; e < EPT; ++e) dst[e] = t[e];
    }
    __syncthreads();
    stamp(a.ts, 2);

    if (has_work) {
        float q_[G][EPT], m[G], l[G], acc[G][EPT];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            m[g] = -INFINITY;
            l[g] = 0.0f;
#pragma unroll
            for (int e = 0; e < EPT; ++e) {
                q_[g][e] = qs[g * D + lane * EPT + e];
                acc[g][e] = 0.0f;
            }
        }
        // One round: all PD * G dot products, their butterfly reductions interleaved, one online-softmax step for the PD positions
        auto use_round = [&](int p0) {
            float sc[PD][G];
#pragma unroll
            for (int q = 0; q < PD; ++q) {
                float kf[EPT];
                if (p0 + q * NW == pos) {
#pragma unroll
                    for (int e = 0; e < EPT; ++e) kf[e] = kcur[lane * EPT + e];
                } else {
                    kraw_cvt<KT, EPT>(kr[q], kf);      // rows past `end` were never loaded: their scores are not used
                }
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    float t = 0.0f;
#pragma unroll
                    for (int e = 0; e < EPT; ++e) t = fmaf(q_[g][e], kf[e], t);
                    sc[q][g] = t;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int q = 0; q < PD; ++q)
#pragma unroll
                    for (int g = 0; g < G; ++g) sc[q][g] += __shfl_xor_sync(0xffffffffu, sc[q][g], o);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float mn = m[g];
#pragma unroll
                for (int q = 0; q < PD; ++q)
                    if (p0 + q * NW < end) mn = fmaxf(mn, sc[q][g]);
                const float corr = expf(m[g] - mn);    // exp(-inf) = 0 in the first round
                float ls = l[g] * corr;
#pragma unroll
                for (int q = 0; q < PD; ++q) {
                    sc[q][g] = (p0 + q * NW < end) ? expf(sc[q][g] - mn) : 0.0f;
                    ls += sc[q][g];
                }
                l[g] = ls;
                m[g] = mn;
#pragma unroll
                for (int e = 0; e < EPT; ++e) acc[g][e] *= corr;
            }
#pragma unroll
            for (int q = 0; q < PD; ++q) {
                const int pq = p0 + q * NW;
                if (pq >= end) break;
                float vf[EPT];
                if (pq == pos) {
#pragma unroll
                    for (int e = 0; e < EPT; ++e) vf[e] = vcur[lane * EPT + e];
                } else {
                    kraw_cvt<KT, EPT>(vr[q], vf);
                }
#pragma unroll
                for (int g = 0; g < G; ++g)
#pragma unroll
                    for (int e = 0; e < EPT; ++e) acc[g][e] = fmaf(sc[q][g], vf[e], acc[g][e]);
            }
        };
        for (int p = begin + warp; p < end; p += PD * NW) {
            if constexpr (DB) {
                Raw nk[PD], nv[PD];
#pragma unroll
                for (int q = 0; q < PD; ++q) issue(p + (PD + q) * NW, nk[q], nv[q]);
                use_round(p);
#pragma unroll
                for (int q = 0; q < PD; ++q) { kr[q] = nk[q]; vr[q] = nv[q]; }
            } else {
                use_round(p);
#pragma unroll
                for (int q = 0; q < PD; ++q) issue(p + (PD + q) * NW, kr[q], vr[q]);
            }
        }
        stamp(a.ts_mid, 1);
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");    // every CTA of the cluster runs
        // output (g, d) is number g * D + d; CTA (number / per) finishes it. A lane's EPT channels lie in one slice
        const int src = s * NW + warp;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int o = g * D + lane * EPT, rank = o / per, at = o - rank * per;
            st_cluster<EPT>(map_cluster(in_acc + (size_t)src * per + at, rank), acc[g]);
            if (at == 0 || (lane == 0 && per > D)) {
                const float ml[2] = {m[g], l[g]};
                st_cluster<2>(map_cluster(in_ml + ((size_t)src * G + g) * 2, rank), ml);
            }
        }
    } else {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    stamp(a.ts_mid, 2);
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    stamp(a.ts_mid, 3);
    if (!active) return;                               // the same for the whole cluster
    // ---- this CTA's outputs: `parts` threads each, adding the sources in a fixed order ----
    const int T = blockDim.x, S = n_eff * NW, parts = per < T ? T / per : 1;
    for (int o0 = 0; o0 < per; o0 += T) {
        const int o = o0 + (per < T ? tid % per : tid), part = per < T ? tid / per : 0;
        const int g = (s * per + o) / D;               // one head per warp: slices and heads are powers of two, and a warp's outputs lie side by side
        float M = -INFINITY;
        for (int i = lane; i < S; i += 32) M = fmaxf(M, in_ml[((size_t)i * G + g) * 2]);
        M = warp_max(M);
        float A = 0.0f, L = 0.0f;
#pragma unroll 4
        for (int i = part; i < S; i += parts) {
            const float2 ml = *reinterpret_cast<const float2*>(in_ml + ((size_t)i * G + g) * 2);
            const float e = ml.x == -INFINITY ? 0.0f : expf(ml.x - M);
            A += e * in_acc[(size_t)i * per + o];
            L += e * ml.y;
        }
        if (parts > 1) {
            red[tid] = A;
            red[T + tid] = L;
            __syncthreads();
            if (tid < per) {
                A = L = 0.0f;
                for (int i = 0; i < parts; ++i) { A += red[i * per + tid]; L += red[T + i * per + tid]; }
            }
        }
        if (part == 0) {
            const size_t oi = ((size_t)b * a.Nq + head0) * D + (size_t)s * per + o;
            const float ov = A / L;
            a.out[oi] = ov;
            if (a.out_bf16) a.out_bf16[oi] = (uint16_t)f32_to_bf16_bits(ov);
        }
    }
    stamp(a.ts, 3);
}

}  // namespace oxg4
