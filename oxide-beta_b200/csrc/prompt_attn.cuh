// Causal / sliding attention of prompt passes on the tensor cores: the rows of a pass are hundreds of tokens of a few
// sequences, BF16 keys and values. Replaces gqa_prefill_block (crates/oxide-torch-cuda/src/kernel_module.rs:1896-1974); the
// attention scale is 1.0 as in the reference.
//
// The kernel of attention_mma.cuh gives eight (token, head) rows to a warp, which is what a decode step has; in a prompt
// that makes 64 groups of every 256 tokens read the same keys and values. Here a CTA owns 128 (token, head) rows of one kv
// head (128 / G tokens), 16 per warp, and every tile of 64 positions is read once for all of them.
//
// Keys and values come from two places: positions before the pass from the cache pages, positions of the pass from the
// buffers that qkv_post_kernel left (kc, vc). A sliding ring is therefore not touched before all rows have attended
// (kv_append_kernel copies the rows that stay afterwards), and a pass may carry more tokens than the ring has spare rows.
//
// Data path. A ring of three slots in shared memory takes the K and V tiles in turn (K0 V0 K1 V1 ...), filled by cp.async; the
// two barriers of a tile (before the scores, before the value product) also hand the freed slot to the next copy, so two
// tiles are always in flight. Rows are stored in 16-byte pieces xor-ed with the row number (conflict-free ldmatrix).
//
// Arithmetic. mma.sync.m16n8k16 BF16, f32 accumulation. Queries are BF16 high and low parts (q = hi + lo to 2^-17) and enter
// the scores as two products into one accumulator; the softmax weights are split the same way for the value product. K and
// V are BF16, so nothing that f32 would keep is lost. Bound by the tensor pipe: 8 * D operations per (token, head, position),
// twice the plain count because of the split. Measured (B200, one launch for 2047 tokens of one prompt, 8 / 4 heads of 256,
// window 1024): 137 us mean of both layer kinds; eight launches of attention_mma.cuh's kernels with their merges 8 x 70 us.
// 2048 tokens of unequal prompts: ~12B widths 120 us (8 x 100), ~27B widths 110 us (8 x 97).
#pragma once
#include "attention_mma.cuh"
#include "latent_mma.cuh"

namespace oxg4 {

constexpr int kPaRows = 128;             // (token, head) rows per CTA
constexpr int kPaTile = 64;              // positions per tile
constexpr int kPaThreads = 256;
constexpr int kPaSlots = 3;

struct PromptAttnArgs {
    const uint16_t* q_hl;                // [R][Nq][2][D] BF16: high part, then low part
    const uint16_t *kc, *vc;             // [Nkv][kv_rows][D] this pass's keys and values
    int kv_rows;
    int Nq, Nkv, lg_group;               // query heads per kv head: 2^lg_group
    // row tiles, the longest first: first row, tokens, first row of the run
    const int32_t *tile_row0, *tile_n, *tile_run0;
    const int32_t *row_pos, *row_seq;    // [R]
    const uint16_t *kpool, *vpool;
    const int32_t* page_table;
    int pages_per_seq, page_tokens;
    const int32_t* cap;
    int window;
    int splits;                          // the positions of a tile are dealt to this many CTAs
    float* part;                         // splits > 1: [splits][R * Nq][D + 2] un-normalised sums, maximum, sum of weights
    int R;
    uint16_t* out;                       // [R, Nq * D] BF16
};

template <int D> constexpr size_t prompt_attn_smem() { return (size_t)kPaRows * D * 4 + (size_t)kPaSlots * kPaTile * D * 2; }

template <int D>
__global__ void __launch_bounds__(kPaThreads, 1) prompt_attn_kernel(const PromptAttnArgs a) {
    const int G = 1 << a.lg_group;
    constexpr int ROWB = D * 2;                                // bytes of a row
    constexpr int CH = D / 8;                                  // 16-byte pieces of a row
    constexpr uint32_t SLOT = kPaTile * ROWB;
    extern __shared__ __align__(128) unsigned char pa_smem[];
    unsigned char* sq = pa_smem;                               // [2][128][D]: high parts, low parts
    const uint32_t q_addr = smem_u32(sq), ring = q_addr + 2u * kPaRows * ROWB;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int split = blockIdx.x % a.splits, kvh = blockIdx.x / a.splits % a.Nkv, tile = blockIdx.x / a.splits / a.Nkv;
    const int row0 = a.tile_row0[tile], ntok = a.tile_n[tile], run0 = a.tile_run0[tile];
    const int pos0 = a.row_pos[row0], pstart = a.row_pos[run0];           // first token of the tile, of the run
    const int seq = a.row_seq[row0], cap = a.cap[seq];
    const int32_t* pt = a.page_table + (size_t)seq * a.pages_per_seq;
    const int lo = max(0, pos0 + 1 - a.window), hi = pos0 + ntok;         // positions [lo, hi) are visible to someone
    // tiles: those of the cache part [lo, pstart), then those of this pass [max(lo, pstart), hi)
    const int n_old = lo < pstart ? (pstart - lo + kPaTile - 1) / kPaTile : 0;
    const int new0 = max(lo, pstart), n_all = n_old + (hi - new0 + kPaTile - 1) / kPaTile;
    const int per = (n_all + a.splits - 1) / a.splits, j0 = split * per, j1 = min(n_all, j0 + per);
    auto tile_range = [&](int j, int& base, int& end) {
        if (j < n_old) {
            base = lo + j * kPaTile;
            end = min(base + kPaTile, pstart);
        } else {
            base = new0 + (j - n_old) * kPaTile;
            end = min(base + kPaTile, hi);
        }
    };
    pdl_wait();
    pdl_launch();

    // copies item 2j (keys of tile j) or 2j + 1 (values) into its slot: a warp moves eight rows, D / 8 lanes per row
    auto load = [&](int item) {
        const int j = j0 + (item >> 1);
        if (j < j1) {
            int base, end;
            tile_range(j, base, end);
            const bool is_v = item & 1, old = j < n_old;
            const uint16_t* src0 = old ? (is_v ? a.vpool : a.kpool) : (is_v ? a.vc : a.kc);
            size_t off = 0;
            const int my = base + warp * 8 + (lane & 7);
            const bool ok = my < end;
            if (ok) {
                if (old) {
                    const int slot = my % cap;
                    off = ((size_t)pt[slot / a.page_tokens] * a.Nkv + kvh) * a.page_tokens + slot % a.page_tokens;
                } else {
                    off = (size_t)kvh * a.kv_rows + run0 + (my - pstart);
                }
                off *= D;
            }
            const unsigned valid = __ballot_sync(0xffffffffu, ok);
            const uint32_t dst = ring + (uint32_t)(item % kPaSlots) * SLOT;
            constexpr int RPI = 32 / (CH < 32 ? CH : 32);      // rows a warp moves at a time
#pragma unroll
            for (int i = 0; i < 8; i += RPI) {
                const int r = i + lane / (CH < 32 ? CH : 32), c = lane % (CH < 32 ? CH : 32), row = warp * 8 + r;
                const size_t o = __shfl_sync(0xffffffffu, off, r);
                cp_async16(dst + row * ROWB + ((c ^ (row & 7)) << 4), src0 + o + c * 8, (valid >> r) & 1);
            }
        }
        cp_async_commit();                                     // one group per item, empty past the end
    };

    // queries: row r = (token r / G, head r % G); rows past the tile's tokens are zero
    for (int i = tid; i < 2 * kPaRows * CH; i += kPaThreads) {
        const int part = i / (kPaRows * CH), r = i / CH % kPaRows, c = i % CH;
        const bool ok = (r >> a.lg_group) < ntok;
        const uint16_t* src = a.q_hl + (((size_t)(row0 + (ok ? r >> a.lg_group : 0)) * a.Nq + kvh * G + (r & (G - 1))) * 2 + part) * D + c * 8;
        cp_async16(q_addr + (uint32_t)part * kPaRows * ROWB + r * ROWB + ((c ^ (r & 7)) << 4), src, ok);
    }
    load(0);                                                   // the queries belong to the first group
    load(1);

    const int lm_i = lane >> 3, lm_r = lane & 7;
    const int wrow = warp * 16, g = lane >> 2, cc = (lane & 3) * 2;
    // the two rows of this lane: positions of their tokens
    const int tokA = (wrow + g) >> a.lg_group, tokB = (wrow + g + 8) >> a.lg_group;
    const int posA = pos0 + tokA, posB = pos0 + tokB;
    const int loA = posA + 1 - a.window, loB = posB + 1 - a.window;
    const int wpos_min = pos0 + (wrow >> a.lg_group), wlo_max = pos0 + ((wrow + 15) >> a.lg_group) + 1 - a.window;     // all rows of the warp see [wlo_max, wpos_min]
    const uint32_t qrow = wrow + (lm_i & 1) * 8 + lm_r;
    const uint32_t qbase = q_addr + qrow * ROWB, qx = qrow & 7, qc = lm_i >> 1;

    float o[D / 8][4];
#pragma unroll
    for (int i = 0; i < D / 8; ++i) { o[i][0] = 0.0f; o[i][1] = 0.0f; o[i][2] = 0.0f; o[i][3] = 0.0f; }
    float mA = -INFINITY, mB = -INFINITY, lA = 0.0f, lB = 0.0f;

    for (int j = j0, it = 0; j < j1; ++j, ++it) {
        int base, end;
        tile_range(j, base, end);
        cp_async_wait<1>();                                    // keys of tile j
        __syncthreads();                                       // ... for everybody; and everybody is done with values j - 1
        load(2 * it + 2);
        const uint32_t kb = ring + (uint32_t)((2 * it) % kPaSlots) * SLOT;
        float s[8][4];
#pragma unroll
        for (int n = 0; n < 8; ++n) { s[n][0] = 0.0f; s[n][1] = 0.0f; s[n][2] = 0.0f; s[n][3] = 0.0f; }
#pragma unroll 2
        for (int kp = 0; kp < D / 32; ++kp) {                  // pairs of 16-wide k-steps
            uint32_t ha[4], hb[4], la[4], lb[4];
            const uint32_t ca = ((kp * 4 + qc) ^ qx) << 4, cb = ((kp * 4 + 2 + qc) ^ qx) << 4;
            ldmatrix_x4(ha, qbase + ca);
            ldmatrix_x4(hb, qbase + cb);
            ldmatrix_x4(la, qbase + kPaRows * ROWB + ca);
            ldmatrix_x4(lb, qbase + kPaRows * ROWB + cb);
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                uint32_t kf[4];
                const int prow = n * 8 + lm_r;
                ldmatrix_x4(kf, kb + prow * ROWB + (((kp * 4 + lm_i) ^ (prow & 7)) << 4));
                mma_bf16_16816(s[n], ha, kf[0], kf[1]);
                mma_bf16_16816(s[n], hb, kf[2], kf[3]);
                mma_bf16_16816(s[n], la, kf[0], kf[1]);
                mma_bf16_16816(s[n], lb, kf[2], kf[3]);
            }
        }
        // ---- online softmax ----
        if (!(base >= wlo_max && base + kPaTile - 1 <= wpos_min && end - base == kPaTile)) {
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int p = base + n * 8 + cc + e;
                    if (p >= end || p > posA || p < loA) s[n][e] = -INFINITY;
                    if (p >= end || p > posB || p < loB) s[n][2 + e] = -INFINITY;
                }
        }
        float nA = mA, nB = mB;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            nA = fmaxf(nA, fmaxf(s[n][0], s[n][1]));
            nB = fmaxf(nB, fmaxf(s[n][2], s[n][3]));
        }
        nA = fmaxf(nA, __shfl_xor_sync(0xffffffffu, nA, 1));
        nA = fmaxf(nA, __shfl_xor_sync(0xffffffffu, nA, 2));
        nB = fmaxf(nB, __shfl_xor_sync(0xffffffffu, nB, 1));
        nB = fmaxf(nB, __shfl_xor_sync(0xffffffffu, nB, 2));
        const bool moved = nA > mA || nB > mB;
        // a row that has seen nothing yet keeps weights and factor at zero and one
        const float cA = nA > -INFINITY ? expf(mA - nA) : 1.0f, cB = nB > -INFINITY ? expf(mB - nB) : 1.0f;
        const float sA = nA > -INFINITY ? nA : 0.0f, sB = nB > -INFINITY ? nB : 0.0f;
        lA *= cA;
        lB *= cB;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            s[n][0] = expf(s[n][0] - sA);
            s[n][1] = expf(s[n][1] - sA);
            s[n][2] = expf(s[n][2] - sB);
            s[n][3] = expf(s[n][3] - sB);
            lA += s[n][0] + s[n][1];
            lB += s[n][2] + s[n][3];
        }
        mA = nA;
        mB = nB;
        if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
            for (int i = 0; i < D / 8; ++i) { o[i][0] *= cA; o[i][1] *= cA; o[i][2] *= cB; o[i][3] *= cB; }
        }
        cp_async_wait<1>();                                    // values of tile j
        __syncthreads();                                       // ... for everybody; and everybody is done with keys j
        load(2 * it + 3);
        const uint32_t vb = ring + (uint32_t)((2 * it + 1) % kPaSlots) * SLOT;
        // ---- O += P V ----
#pragma unroll
        for (int ks = 0; ks < kPaTile / 16; ++ks) {
            uint32_t ph[4], pl[4];
            split_pack(s[2 * ks][0], s[2 * ks][1], ph[0], pl[0]);
            split_pack(s[2 * ks][2], s[2 * ks][3], ph[1], pl[1]);
            split_pack(s[2 * ks + 1][0], s[2 * ks + 1][1], ph[2], pl[2]);
            split_pack(s[2 * ks + 1][2], s[2 * ks + 1][3], ph[3], pl[3]);
            const int prow = ks * 16 + (lm_i & 1) * 8 + lm_r;
#pragma unroll
            for (int np = 0; np < D / 16; ++np) {
                uint32_t vf[4];
                ldmatrix_x4_trans(vf, vb + prow * ROWB + (((np * 2 + (lm_i >> 1)) ^ (prow & 7)) << 4));
                mma_bf16_16816(o[2 * np], ph, vf[0], vf[1]);
                mma_bf16_16816(o[2 * np + 1], ph, vf[2], vf[3]);
                mma_bf16_16816(o[2 * np], pl, vf[0], vf[1]);
                mma_bf16_16816(o[2 * np + 1], pl, vf[2], vf[3]);
            }
        }
    }
    cp_async_wait<0>();
    lA += __shfl_xor_sync(0xffffffffu, lA, 1);
    lA += __shfl_xor_sync(0xffffffffu, lA, 2);
    lB += __shfl_xor_sync(0xffffffffu, lB, 1);
    lB += __shfl_xor_sync(0xffffffffu, lB, 2);
    if (a.splits > 1) {
        auto put = [&](int r, int tok, int e, float m, float l) {
            if (tok >= ntok) return;
            float* dst = a.part + (((size_t)split * a.R + row0 + tok) * a.Nq + kvh * G + (r & (G - 1))) * (D + 2);
#pragma unroll
            for (int i = 0; i < D / 8; ++i) *reinterpret_cast<float2*>(dst + i * 8 + cc) = make_float2(o[i][e], o[i][e + 1]);
            if ((lane & 3) == 0) *reinterpret_cast<float2*>(dst + D) = make_float2(m, l);
        };
        put(wrow + g, tokA, 0, mA, lA);
        put(wrow + g + 8, tokB, 2, mB, lB);
        return;
    }
    // normalised rows as BF16 through the warp's own query rows, then 16-byte stores
    const float iA = 1.0f / lA, iB = 1.0f / lB;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
        const uint32_t rA = wrow + g, rB = rA + 8;
        const uint32_t vA = f32_to_bf16_bits(o[i][0] * iA) | (f32_to_bf16_bits(o[i][1] * iA) << 16);
        const uint32_t vB = f32_to_bf16_bits(o[i][2] * iB) | (f32_to_bf16_bits(o[i][3] * iB) << 16);
        *reinterpret_cast<uint32_t*>(sq + rA * ROWB + ((i ^ (rA & 7)) << 4) + cc * 2) = vA;
        *reinterpret_cast<uint32_t*>(sq + rB * ROWB + ((i ^ (rB & 7)) << 4) + cc * 2) = vB;
    }
    __syncwarp();
    for (int i = lane; i < 16 * CH; i += 32) {
        const int r = wrow + i / CH, c = i % CH, tok = r >> a.lg_group;
        if (tok < ntok)
            *reinterpret_cast<uint4*>(a.out + ((size_t)(row0 + tok) * a.Nq + kvh * G + (r & (G - 1))) * D + c * 8) =
                *reinterpret_cast<const uint4*>(sq + r * ROWB + ((c ^ (r & 7)) << 4));
    }
}

// One warp per (row, head): adds the splits' partials in order and writes the normalised BF16 output.
template <int D>
__global__ void __launch_bounds__(128) prompt_merge_kernel(const PromptAttnArgs a) {
    constexpr int EPT = D / 32;
    pdl_wait();
    pdl_launch();
    const int job = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (job >= a.R * a.Nq) return;
    const size_t stride = (size_t)a.R * a.Nq * (D + 2);
    const float* p = a.part + (size_t)job * (D + 2);
    float M = -INFINITY;
    for (int s = 0; s < a.splits; ++s) M = fmaxf(M, p[s * stride + D]);
    float L = 0.0f, acc[EPT];
#pragma unroll
    for (int e = 0; e < EPT; ++e) acc[e] = 0.0f;
    for (int s = 0; s < a.splits; ++s) {
        const float* q = p + s * stride;
        const float f = q[D] == -INFINITY ? 0.0f : expf(q[D] - M);
        L += f * q[D + 1];
#pragma unroll
        for (int e = 0; e < EPT; e += 2) {
            const float2 v = *reinterpret_cast<const float2*>(q + lane * EPT + e);
            acc[e] += f * v.x;
            acc[e + 1] += f * v.y;
        }
    }
    uint32_t bits[EPT];
#pragma unroll
    for (int e = 0; e < EPT; ++e) bits[e] = f32_to_bf16_bits(acc[e] / L);
    st_u16_vec<EPT>(a.out + (size_t)job * D + lane * EPT, bits);
}

// Copies the keys and values of a pass that stay in the ring (the last `cap` positions of every sequence) to the cache pages;
// one warp per (row, kv head).
struct KvAppendArgs {
    const uint16_t *kc, *vc;             // [Nkv][kv_rows][D]
    int kv_rows, R, Nkv;
    const int32_t *row_pos, *row_seq, *row_end;      // row_end: position behind the sequence's last token of the pass
    uint16_t *kpool, *vpool;
    const int32_t* page_table;
    int pages_per_seq, page_tokens;
    const int32_t* cap;
};
template <int D>
__global__ void __launch_bounds__(128) kv_append_kernel(const KvAppendArgs a) {
    constexpr int EPT = D / 32;          // BF16 values per lane
    pdl_wait();
    pdl_launch();
    const int job = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (job >= a.R * a.Nkv) return;
    const int row = job / a.Nkv, kvh = job % a.Nkv, seq = a.row_seq[row], pos = a.row_pos[row], cap = a.cap[seq];
    if (pos < a.row_end[row] - cap) return;
    const int slot = pos % cap;
    const size_t dst = (((size_t)a.page_table[(size_t)seq * a.pages_per_seq + slot / a.page_tokens] * a.Nkv + kvh) * a.page_tokens +
                        slot % a.page_tokens) * (size_t)D + lane * EPT;
    const size_t src = ((size_t)kvh * a.kv_rows + row) * D + lane * EPT;
    if constexpr (EPT == 8) {
        *reinterpret_cast<uint4*>(a.kpool + dst) = *reinterpret_cast<const uint4*>(a.kc + src);
        *reinterpret_cast<uint4*>(a.vpool + dst) = *reinterpret_cast<const uint4*>(a.vc + src);
    } else if constexpr (EPT == 4) {
        *reinterpret_cast<uint2*>(a.kpool + dst) = *reinterpret_cast<const uint2*>(a.kc + src);
        *reinterpret_cast<uint2*>(a.vpool + dst) = *reinterpret_cast<const uint2*>(a.vc + src);
    } else {
        *reinterpret_cast<uint32_t*>(a.kpool + dst) = *reinterpret_cast<const uint32_t*>(a.kc + src);
        *reinterpret_cast<uint32_t*>(a.vpool + dst) = *reinterpret_cast<const uint32_t*>(a.vc + src);
    }
}

}  // namespace oxg4
