// Weight-streaming projection kernel for BF16 weights, 1..8 activation rows (more: gemv_rows.cuh).
//
// Prologues and epilogues are those of gemv.cuh (see there for the reference launches it replaces). The weights go through shared
// memory and meet the activations on the tensor cores, so that a CTA can use them up several times faster than HBM delivers
// them: what arrived while the kernel waited for its predecessor, or made its activations, is then gone in no time.
//
// Data path. Every CTA owns a contiguous block of output rows and cuts it into boxes of up to 32 rows x 64 columns (with gate and
// up 16 rows of each), which its eight warps take in turn; a warp has its own ring of boxes, filled by TMA (128-byte swizzle,
// so that ldmatrix meets no bank conflict) at the request of its first lane, and waits for nobody else. Weights depend on no
// other kernel: the ring is filled ahead of the dependency wait. A launch of a decode step lets its successor start at once (`early`), and two CTAs of successive launches
// share an SM: the successor's ring fills while this kernel still runs. (They share it one by one only while no kernel that
// fills an SM by itself lets its successor start early: CTAs of the successor would then gather on the SMs that are left.)
// The copies carry an evict-first L2 policy: a step reads every weight once, and with the default policy they pushed K/V rows,
// activations and the kernels' own code out of L2 (attention launch of the ~4B model, 272 positions: 20.0 us, 13.4 with it).
//
// Arithmetic. mma.sync.m16n8k16 (BF16 x BF16 -> f32): the activations are the 16-row A operand (batch rows, or the inputs of
// the row segments; unused rows are zero registers), eight weight rows the B operand, read by ldmatrix, 32 columns at a
// time: three instructions per 512 bytes of weights, where multiply-adds on widened values take about thirty. The partial sums that
// the warps have of a row meet in shared memory and are added in warp order.
// Products of BF16 values are exact in f32; accumulation is f32.
//
// HBM-bound: bytes per launch = N * K * 2.
#pragma once
#include "gemv.cuh"

namespace oxg4 {

constexpr int kGmWarps = 8;
constexpr int kGmThreads = kGmWarps * 32;
constexpr int kGmMaxSlots = 6;
constexpr int kGmBoxRows = 32;                         // weight rows of a box, at most (with gate and up: 16 of each)
constexpr int kGmMaxRows = 8;                          // activation rows of a launch's pass

// Row stride (elements) of the activations in shared memory: whole units of 32, rows 64 bytes apart modulo 128, so that the
// eight lanes of an LDS.128 phase (two batch rows x four column groups) hit eight different 16-byte bank groups.
__host__ __device__ inline int mma_x_stride(int K) {
    const int units = (K + 31) / 32;
    return (units | 1) * 32;
}

DEVINL void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                           uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Sum over the `warps` warps of a team (a power of two, teams of neighbouring warps) of the CTA; every thread calls it.
DEVINL float team_sum(float v, int warps, float* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_sum(v);
    if (warps == 1) return v;
    __syncthreads();                                // protect `red` against the previous use
    if (lane == 0) red[warp] = v;
    __syncthreads();
    const int w0 = warp & ~(warps - 1);
    float t = 0.0f;
    for (int w = 0; w < warps; ++w) t += red[w0 + w];
    return t;
}

// Activations in shared memory: inside a unit of 32 columns the pairs (c, c + 1) are stored in the order in which a lane of
// the A operand wants them, those of column group t = c % 8 / 2 one after the other.
DEVINL int x_place(int c) { return (c & ~31) + ((c & 7) >> 1) * 8 + ((c >> 3) & 3) * 2; }
DEVINL void x_put4(uint16_t* row, int c, float4 v) {   // c a multiple of 4
    uint16_t* p = row + x_place(c);
    *reinterpret_cast<uint32_t*>(p) = f32_to_bf16_bits(v.x) | (f32_to_bf16_bits(v.y) << 16);
    *reinterpret_cast<uint32_t*>(p + 8) = f32_to_bf16_bits(v.z) | (f32_to_bf16_bits(v.w) << 16);
}
DEVINL void x_put(uint16_t* row, int c, float v) { row[x_place(c) + (c & 1)] = (uint16_t)f32_to_bf16_bits(v); }

// MAXJ: groups of four values of a residual row per thread in the norms of one row (hidden <= MAXJ * 1024); with 3 the norm
// weights wait in registers too
template <int PRO, int EPI, int MAXJ>
__global__ void __launch_bounds__(kGmThreads, 2)
gemv_mma_kernel(const __grid_constant__ CUtensorMap map0, const __grid_constant__ CUtensorMap map1, const GemvArgs a) {
    constexpr bool NORM = PRO == PRO_NORM || PRO == PRO_SHIFT;
    constexpr bool TWO = EPI == EPI_GATEUP;            // gate and up rows come from two matrices
    constexpr bool SEGS = (PRO == PRO_SHIFT || PRO == PRO_PLAIN) && EPI == EPI_STORE;   // may have several inputs
    constexpr bool AHEAD = NORM && MAXJ <= 3;
    constexpr int GROUPS = kGmBoxRows / 8;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* rings = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[kGmWarps][kGmMaxSlots];
    __shared__ float red[32];
    __shared__ unsigned int s_last;
    __shared__ volatile int failed;
    const int K = a.K, NS = a.places, SB = a.place_bytes, R = a.box_rows;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b0 = blockIdx.y * a.bpp;
    const int nb = min(a.bpp, a.B - b0);               // rows of this pass
    const int nseg = SEGS ? max(1, a.nseg) : 1;
    const int nx = SEGS && nseg > 1 ? nseg : nb;       // rows of the A operand (several inputs: one row each)
    const int nxp = SEGS && nseg > 1 ? nseg : a.bpp;
    const int XS = mma_x_stride(K);
    const int PB = a.pass_boxes;                       // boxes whose partial sums meet in one combine
    uint16_t* xs = reinterpret_cast<uint16_t*>(rings + (size_t)kGmWarps * NS * SB);              // [nx][XS]
    float* pieces = reinterpret_cast<float*>(xs + (size_t)nxp * XS);                             // [2, or 1][PB boxes][32 rows][warps][nx]

    // this CTA's rows: (virtual) rows, or with two matrices rows of each of them
    int row_first = 0, rows_cta = 0;
    if constexpr (EPI == EPI_STORE_GLU) {              // a gate row and its up row stay together
        block_range(a.N / 2, gridDim.x, blockIdx.x, row_first, rows_cta);
        row_first *= 2;
        rows_cta *= 2;
    } else {
        block_range(TWO ? a.N / 2 : a.N, gridDim.x, blockIdx.x, row_first, rows_cta);
    }
    const int n_boxes = (rows_cta + R - 1) / R, ncb = (K + 63) >> 6;

    // ---- ahead of the dependency wait nothing reads what the previous kernel wrote ----
    // This warp's items: number i is column block cb of box rb, all (rb, cb) in order dealt to the warps in turn.
    auto next_item = [&](int& rb, int& cb) {
        cb += kGmWarps;
        while (cb >= ncb) { cb -= ncb; ++rb; }
    };
    int rb = 0, cb = warp;
    while (cb >= ncb) { cb -= ncb; ++rb; }
    unsigned char* ring = rings + (size_t)warp * NS * SB;
    uint64_t* bar = bars[warp];
    const bool once = gridDim.y == 1;                  // rows that take several passes read the weights again
    const uint64_t policy = evict_first_policy();
    auto load_box = [&](unsigned char* dst, const CUtensorMap* map, int x, int y, uint64_t* b) {
        if (once) tma_load_2d_hint(dst, map, x, y, b, policy);
        else tma_load_2d(dst, map, x, y, b);
    };
    const uint32_t box_bytes = (uint32_t)(R * 128 * (TWO ? 2 : 1));
    int irb = rb, icb = cb;                            // next item to request (lane 0)
    auto request = [&](int slot) {
        mbar_expect_tx(&bar[slot], box_bytes);
        load_box(ring + (size_t)slot * SB, &map0, icb * 64, row_first + irb * R, &bar[slot]);
        if constexpr (TWO) load_box(ring + (size_t)slot * SB + SB / 2, &map1, icb * 64, row_first + irb * R, &bar[slot]);
        next_item(irb, icb);
    };
    if (tid == 0) failed = 0;
    if (lane == 0) {
        for (int s = 0; s < NS; ++s) mbar_init(&bar[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int s = 0; s < NS && irb < n_boxes; ++s) request(s);
    }
    __syncwarp();
    if (a.early) pdl_launch();
    const int k4 = K >> 2;
    float4 wpost[AHEAD ? MAXJ : 1], wnorm[AHEAD ? MAXJ : 1];
    if constexpr (NORM) {
        if (AHEAD && nb == 1) {
#pragma unroll
            for (int j = 0; j < (AHEAD ? MAXJ : 1); ++j) {
                const int i4 = tid + j * kGmThreads;
                wnorm[j] = wpost[j] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
                if (i4 < k4) {
                    wnorm[j] = *reinterpret_cast<const float4*>(a.w_norm + 4 * i4);
                    if (a.w_post) wpost[j] = *reinterpret_cast<const float4*>(a.w_post + 4 * i4);
                }
            }
        } else {
            for (int i = tid * 32; i < K; i += kGmThreads * 32) {
                prefetch_l2(a.w_norm + i);
                if (a.w_post) prefetch_l2(a.w_post + i);
            }
        }
    }
    for (int i = tid; i < nx * (XS - K); i += kGmThreads) {               // columns past K
        const int b = i / (XS - K), c = K + i - b * (XS - K);
        xs[(size_t)b * XS + x_place(c) + (c & 1)] = 0;
    }
    stamp(a.ts, 0);
    pdl_wait();
    stamp(a.ts, 1);
    const int dead = *(const volatile int*)a.err;      // an earlier launch failed: this one uses none of its data (looked at behind the prologue)

    // ---- prologue: x[nx][K] (BF16) in shared memory ----
    if constexpr (PRO == PRO_PLAIN) {
        if (a.in_x != nullptr) {                       // already BF16 in the operand's order
            const int k8 = ((K + 31) & ~31) >> 3;
            for (int x = 0; x < nx; ++x) {
                const uint4* src = reinterpret_cast<const uint4*>(a.in_x + (size_t)(b0 + x) * (8 * k8));
#pragma unroll 8
                for (int i = tid; i < k8; i += kGmThreads) reinterpret_cast<uint4*>(xs + (size_t)x * XS)[i] = src[i];
            }
        } else for (int x = 0; x < nx; ++x) {
            const float* src = a.in + (nseg > 1 ? (size_t)x * a.B : (size_t)(b0 + x)) * K;
#pragma unroll 4
            for (int i4 = tid; i4 < k4; i4 += kGmThreads) x_put4(xs + (size_t)x * XS, 4 * i4, *reinterpret_cast<const float4*>(src + 4 * i4));
        }
    } else if constexpr (PRO == PRO_GNORM) {
        const int group = a.gn_group ? a.gn_group : a.gn_n;
        const bool aligned = (((uintptr_t)a.in | (uintptr_t)a.gn_w | (uintptr_t)a.gn_gate | (uintptr_t)a.gn_tail) & 15) == 0 &&
                             ((a.gn_n | a.gn_tail_at | a.gn_tail_n | group) & 3) == 0;
        auto gate = [&](float z) { return a.act == ACT_SILU ? silu(z) : sigmoid(z); };
        const int gl = group >> 2;                     // lanes of a group of four values each
        const bool lanes = gl <= 32 && (gl & (gl - 1)) == 0;
        if (aligned && (group == a.gn_n || lanes)) {
            const int n4 = a.gn_n >> 2, n4w = (n4 + 31) & ~31;
            float r = 1.0f;
            const bool whole = a.gn_group == a.gn_n && !lanes;
            if (whole) {
                float ss = 0.0f;
#pragma unroll 4
                for (int i4 = tid; i4 < n4; i4 += kGmThreads) ss += sum_sq4(*reinterpret_cast<const float4*>(a.in + 4 * i4));
                r = 1.0f / sqrtf(team_sum(ss, kGmWarps, red) / (float)a.gn_n + a.eps);
            }
            constexpr int U = 4;                       // groups of four values in flight
            for (int base = tid; base < n4w; base += U * kGmThreads) {
                float4 v[U], z[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i4 = base + u * kGmThreads;
                    v[u] = z[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (i4 < n4) {
                        v[u] = *reinterpret_cast<const float4*>(a.in + 4 * i4);
                        if (a.gn_gate) z[u] = *reinterpret_cast<const float4*>(a.gn_gate + 4 * i4);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i4 = base + u * kGmThreads;
                    if (i4 >= n4w) break;              // the same for a whole warp
                    float s = r;
                    if (a.gn_group && !whole) {
                        float ss = sum_sq4(v[u]);
                        for (int o = gl >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                        s = 1.0f / sqrtf(ss / (float)group + a.eps);
                    }
                    if (i4 >= n4) continue;
                    float4 o = make_float4(v[u].x * s, v[u].y * s, v[u].z * s, v[u].w * s);
                    if (a.gn_w) {
                        const float4 w = *reinterpret_cast<const float4*>(a.gn_w + 4 * i4);
                        o.x *= w.x; o.y *= w.y; o.z *= w.z; o.w *= w.w;
                    }
                    if (a.gn_gate) { o.x *= gate(z[u].x); o.y *= gate(z[u].y); o.z *= gate(z[u].z); o.w *= gate(z[u].w); }
                    x_put4(xs, 4 * i4, o);
                }
            }
        } else {
            auto put = [&](int i, float v) {
                if (a.gn_w) v *= a.gn_w[i];
                if (a.gn_gate) v *= gate(a.gn_gate[i]);
                x_put(xs, i, v);
            };
            if (a.gn_group == 0 || a.gn_group == a.gn_n) {
                float r = 1.0f;
                if (a.gn_group) {
                    float ss = 0.0f;
                    for (int i = tid; i < a.gn_n; i += kGmThreads) ss += a.in[i] * a.in[i];
                    r = 1.0f / sqrtf(team_sum(ss, kGmWarps, red) / (float)a.gn_n + a.eps);
                }
                for (int i = tid; i < a.gn_n; i += kGmThreads) put(i, a.in[i] * r);
            } else {
                for (int g = warp; g < a.gn_n / a.gn_group; g += kGmWarps) {
                    const float* src = a.in + (size_t)g * a.gn_group;
                    float s = 0.0f;
                    for (int i = lane; i < a.gn_group; i += 32) s += src[i] * src[i];
                    s = 1.0f / sqrtf(warp_sum(s) / (float)a.gn_group + a.eps);
                    for (int i = lane; i < a.gn_group; i += 32) put(g * a.gn_group + i, src[i] * s);
                }
            }
        }
        if (a.gn_tail != nullptr) {
            for (int i = a.gn_n + tid; i < a.gn_tail_at; i += kGmThreads) x_put(xs, i, 0.0f);
            if (aligned) {
                const int n4 = a.gn_tail_n >> 2;
#pragma unroll 4
                for (int i4 = tid; i4 < n4; i4 += kGmThreads)
                    x_put4(xs, a.gn_tail_at + 4 * i4, *reinterpret_cast<const float4*>(a.gn_tail + 4 * i4));
                for (int i = a.gn_tail_at + a.gn_tail_n + tid; i < K; i += kGmThreads) x_put(xs, i, 0.0f);
            } else {
                for (int i = a.gn_tail_at + tid; i < K; i += kGmThreads)
                    x_put(xs, i, i < a.gn_tail_at + a.gn_tail_n ? a.gn_tail[i - a.gn_tail_at] : 0.0f);
            }
        } else {
            for (int i = a.gn_n + tid; i < K; i += kGmThreads) x_put(xs, i, 0.0f);
        }
    } else {
        const bool writer = (blockIdx.x == 0);
        const float norm_n = (float)(a.norm_n ? a.norm_n : K);
        const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f), one = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        auto update = [&](float4 h, float4 t, float r, float4 w) {
            return make_float4((h.x + t.x * r * w.x) * a.scalar, (h.y + t.y * r * w.y) * a.scalar, (h.z + t.z * r * w.z) * a.scalar,
                               (h.w + t.w * r * w.w) * a.scalar);
        };
        auto load4 = [&](const float* p) { return *reinterpret_cast<const float4*>(p); };
        if (nb == 1) {
            // one row: the residual row stays in registers between the two sums
            const size_t ro = (size_t)b0 * K;
            float4 h[MAXJ];
            if (a.embed != nullptr) {
                // kernel_module.rs:1272-1285: embedding row widened to f32, times sqrt(hidden)
                uint32_t tok = a.tokens[b0];
                if (tok == kInactiveToken) tok = 0;
#pragma unroll
                for (int j = 0; j < MAXJ; ++j) {
                    const int i4 = tid + j * kGmThreads;
                    h[j] = i4 < k4 ? embed4<uint16_t>(a.embed, (size_t)tok * K + 4 * i4, a.embed_scale) : zero;
                }
            } else {
                float4 t[MAXJ];
#pragma unroll
                for (int j = 0; j < MAXJ; ++j) {
                    const int i4 = tid + j * kGmThreads;
                    t[j] = i4 < k4 && a.raw != nullptr ? load4(a.raw + ro + 4 * i4) : zero;
                    h[j] = i4 < k4 ? load4(a.h_in + ro + 4 * i4) : zero;
                }
                if (a.raw != nullptr) {                // null: h_in already is the layer's input (layer-wise tracing)
                    float r = 1.0f;
                    if (a.w_post != nullptr) {
                        float ss = 0.0f;
#pragma unroll
                        for (int j = 0; j < MAXJ; ++j) ss += sum_sq4(t[j]);
                        r = 1.0f / sqrtf(team_sum(ss, kGmWarps, red) / norm_n + a.eps);
                    }
#pragma unroll
                    for (int j = 0; j < MAXJ; ++j) {
                        const int i4 = tid + j * kGmThreads;
                        float4 w = one;
                        if constexpr (AHEAD) w = wpost[j];
                        else if (a.w_post != nullptr && i4 < k4) w = load4(a.w_post + 4 * i4);
                        h[j] = update(h[j], t[j], r, w);
                    }
                }
            }
            float ss = 0.0f;
#pragma unroll
            for (int j = 0; j < MAXJ; ++j) {
                const int i4 = tid + j * kGmThreads;
                if (writer && i4 < k4) *reinterpret_cast<float4*>(a.h_out + ro + 4 * i4) = h[j];
                ss += sum_sq4(h[j]);
            }
            const float r2 = 1.0f / sqrtf(team_sum(ss, kGmWarps, red) / norm_n + a.eps);
            const bool first = PRO == PRO_SHIFT && a.pos[0] == 0;
#pragma unroll
            for (int j = 0; j < MAXJ; ++j) {
                const int i4 = tid + j * kGmThreads;
                if (i4 >= k4) continue;
                float4 w;
                if constexpr (AHEAD) w = wnorm[j];
                else w = load4(a.w_norm + 4 * i4);
                const float4 c = make_float4(h[j].x * r2 * w.x, h[j].y * r2 * w.y, h[j].z * r2 * w.z, h[j].w * r2 * w.w);
                if constexpr (PRO == PRO_SHIFT) {
                    const float4 p = first ? zero : load4(a.shift_state + 4 * i4);
                    if (writer) *reinterpret_cast<float4*>(a.x_f32 + 4 * i4) = c;
                    for (int sg = 0; sg < nseg; ++sg) {
                        const float4 mu = load4(a.mu + (size_t)sg * K + 4 * i4);
                        x_put4(xs + (size_t)sg * XS, 4 * i4, make_float4(c.x + (p.x - c.x) * mu.x, c.y + (p.y - c.y) * mu.y,
                                                                        c.z + (p.z - c.z) * mu.z, c.w + (p.w - c.w) * mu.w));
                    }
                } else {
                    x_put4(xs, 4 * i4, c);
                }
            }
        } else if constexpr (PRO == PRO_NORM) {
            // several rows side by side, a team of warps each (more rows than warps: in turns); the rows come from L2 three times
            const int teams = nb <= 2 ? 2 : nb <= 4 ? 4 : 8, tw = kGmWarps / teams, tl = tid & (32 * tw - 1), step = 32 * tw;
            for (int bt = 0; bt < nb; bt += teams) {
                const int b = bt + warp / tw;
                const bool mine = b < nb;
                const size_t ro = (size_t)(b0 + (mine ? b : 0)) * K;
                const int n4 = mine ? k4 : 0;
                uint32_t tok = 0;
                if (a.embed != nullptr && mine) {
                    tok = a.tokens[b0 + b];
                    if (tok == kInactiveToken) tok = 0;
                }
                const bool pending = a.embed == nullptr && a.raw != nullptr;
                float r = 1.0f;
                if (pending && a.w_post != nullptr) {
                    float ss = 0.0f;
#pragma unroll 10
                    for (int i4 = tl; i4 < n4; i4 += step) ss += sum_sq4(load4(a.raw + ro + 4 * i4));
                    r = 1.0f / sqrtf(team_sum(ss, tw, red) / norm_n + a.eps);
                }
                auto hidden = [&](int i4) -> float4 {
                    if (a.embed != nullptr) return embed4<uint16_t>(a.embed, (size_t)tok * K + 4 * i4, a.embed_scale);
                    const float4 h = load4(a.h_in + ro + 4 * i4);
                    if (!pending) return h;
                    return update(h, load4(a.raw + ro + 4 * i4), r, a.w_post != nullptr ? load4(a.w_post + 4 * i4) : one);
                };
                float ss = 0.0f;
#pragma unroll 5
                for (int i4 = tl; i4 < n4; i4 += step) {
                    const float4 h = hidden(i4);
                    if (writer) *reinterpret_cast<float4*>(a.h_out + ro + 4 * i4) = h;
                    ss += sum_sq4(h);
                }
                const float r2 = 1.0f / sqrtf(team_sum(ss, tw, red) / norm_n + a.eps);
#pragma unroll 5
                for (int i4 = tl; i4 < n4; i4 += step) {
                    const float4 h = hidden(i4), w = load4(a.w_norm + 4 * i4);
                    x_put4(xs + (size_t)b * XS, 4 * i4, make_float4(h.x * r2 * w.x, h.y * r2 * w.y, h.z * r2 * w.z, h.w * r2 * w.w));
                }
            }
        }
    }
    __syncthreads();
    if (!a.early && tid == 0) pdl_launch();
    stamp(a.ts, 2);

    // ---- body ----
    const int g8 = lane >> 2, t4 = lane & 3;
    auto g_of = [](int g) { return 8 * (TWO ? g % (GROUPS / 2) : g); };      // first row of a group in its box
    const uint32_t frag = (uint32_t)((lane & 7) * 128);                // ldmatrix: row lane % 8, 16-byte chunk 4 * unit + lane / 8, swizzled
    const int c16 = lane >> 3, x7 = lane & 7;
    const uint16_t* xa = xs + (size_t)g8 * XS + t4 * 8;
    const bool has_a = g8 < nx;
    Cand best{-INFINITY, 0xffffffffu};
    int slot = 0, pass = 0;
    uint32_t phase = 0;
    // a failed wait, here or in a launch before: the warp goes on without data, so that it meets the others at every barrier
    bool ok = !__any_sync(0xffffffffu, dead != 0);
    for (int p0 = 0; p0 < n_boxes; p0 += PB, ++pass) {
        float* pc = pieces + (size_t)(pass & 1) * PB * kGmBoxRows * kGmWarps * nx;
        const int r0 = p0 * R, rows_here = min(PB * R, rows_cta - r0);
        for (int box = p0; box < min(n_boxes, p0 + PB); ++box) {
            float acc[GROUPS][4];
#pragma unroll
            for (int g = 0; g < GROUPS; ++g) acc[g][0] = acc[g][1] = acc[g][2] = acc[g][3] = 0.0f;
            while (rb == box && ok) {
                if (!mbar_wait_warp(&bar[slot], phase, &failed)) {
                    if (lane == 0) wait_failed(a.err, 7, &failed);
                    ok = false;
                    break;
                }
                const uint32_t base = smem_u32(ring + (size_t)slot * SB) + frag;
                uint4 x[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {          // the row of the A operand ends with whole units: a unit past K is not read
                    x[u] = make_uint4(0u, 0u, 0u, 0u);
                    const int at = (cb * 2 + u) * 32;
                    if (has_a && at < K) x[u] = *reinterpret_cast<const uint4*>(xa + at);
                }
                uint32_t w[2][GROUPS][4];
#pragma unroll
                for (int g = 0; g < GROUPS; ++g)
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        if (g_of(g) < R) asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                                     : "=r"(w[u][g][0]), "=r"(w[u][g][1]), "=r"(w[u][g][2]), "=r"(w[u][g][3])
                                     : "r"(base + (uint32_t)((TWO && g >= GROUPS / 2 ? SB / 2 + (g - GROUPS / 2) * 1024 : g * 1024) + (((u * 4 + c16) ^ x7) << 4))));
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int g = 0; g < GROUPS; ++g)
                        if (g_of(g) < R) mma_bf16_16816(acc[g], x[u].x, 0u, x[u].y, 0u, w[u][g][0], w[u][g][1]);
                __syncwarp();                          // all lanes have read the slot (every ldmatrix has delivered)
                if (lane == 0 && irb < n_boxes) request(slot);
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int g = 0; g < GROUPS; ++g)
                        if (g_of(g) < R) mma_bf16_16816(acc[g], x[u].z, 0u, x[u].w, 0u, w[u][g][2], w[u][g][3]);
                next_item(rb, cb);
                if (++slot == NS) { slot = 0; phase ^= 1; }
            }
            // lane (g8, t4) holds batch row g8 of weight rows 2 * t4 and 2 * t4 + 1 of every group
#pragma unroll
            for (int g = 0; g < GROUPS; ++g) {
                float* q0 = pc + ((size_t)((box - p0) * kGmBoxRows + g * 8 + 2 * t4) * kGmWarps + warp) * nx;
                float* q1 = q0 + (size_t)kGmWarps * nx;
                if (has_a) { q0[g8] = acc[g][0]; q1[g8] = acc[g][1]; }
            }
        }
        __syncthreads();
        // add the pieces in warp order and apply the epilogue; the next pass writes the other half of `pieces`
        auto total = [&](int rl, int b, int half = 0) -> float {
            const int box = rl / R;
            const float* q = pc + ((size_t)(box * kGmBoxRows + half * (kGmBoxRows / 2) + rl - box * R) * kGmWarps) * nx + b;
            float v = 0.0f;
#pragma unroll
            for (int w = 0; w < kGmWarps; ++w) v += q[(size_t)w * nx];
            return v;
        };
        if constexpr (EPI == EPI_STORE) {
            for (int idx = tid; idx < rows_here * nb; idx += kGmThreads) {
                const int b = idx / rows_here, rl = idx - b * rows_here, row = row_first + r0 + rl;
                a.out[(size_t)(b0 + b) * a.N + row] = total(rl, SEGS && nseg > 1 ? row / a.seg_rows : b);
            }
        } else if constexpr (EPI == EPI_STORE_GLU) {
            const int ld = (a.glu_from + a.N) / 2;
            for (int idx = tid; idx < rows_here * nb; idx += kGmThreads) {
                const int b = idx / rows_here, rl = idx - b * rows_here, row = row_first + r0 + rl;
                float* o = a.out + (size_t)(b0 + b) * ld;
                if (row < a.glu_from) o[row] = total(rl, b);
                else if (!(row & 1)) o[a.glu_from + (row - a.glu_from) / 2] = glu_mul(a.act, total(rl, b), total(rl + 1, b));
            }
        } else if constexpr (EPI == EPI_GATEUP) {
            for (int idx = tid; idx < rows_here * nb; idx += kGmThreads) {
                const int b = idx / rows_here, rl = idx - b * rows_here;
                const float v = glu_mul(a.act, total(rl, b), total(rl, b, 1));
                const int row = row_first + r0 + rl, n = a.N / 2;
                if (a.out_x != nullptr) x_put(a.out_x + (size_t)(b0 + b) * ((n + 31) & ~31), row, v);
                else a.out[(size_t)(b0 + b) * n + row] = v;
            }
        } else {
            // thread -> (row tid % RP, batch row tid / RP); RP a power of two, at most 256 / nb
            const int RP = PB * kGmBoxRows, rl = tid & (RP - 1), b = tid / RP;
            if (rl < rows_here && b < nb) {
                const float v = total(rl, b);
                const int vid = a.row_offset + row_first + r0 + rl;
                const size_t gb = (size_t)(b0 + b) * a.n_total;
                if (a.out) a.out[gb + vid] = v;
                float sc = v;          // kernel_module.rs:2008-2016: penalty on seen tokens, NaN skipped, strict '>'
                if (a.seen && a.penalty > 1.0f && a.seen[gb + vid]) sc = sc >= 0.0f ? sc / a.penalty : sc * a.penalty;
                const Cand cnd{sc, (uint32_t)vid};
                if (sc == sc && sc > -INFINITY && cand_better(cnd, best)) best = cnd;
            }
        }
    }

    if constexpr (EPI == EPI_LOGITS) {
        __syncthreads();
        Cand* wc = reinterpret_cast<Cand*>(pieces);        // [nb][RP]
        const int RP = PB * kGmBoxRows;
        if (tid / RP < nb) wc[tid] = best;
        __syncthreads();
        for (int b = warp; b < nb; b += kGmWarps) {
            Cand c = wc[b * RP + lane];
            for (int i = lane + 32; i < RP; i += 32)
                if (cand_better(wc[b * RP + i], c)) c = wc[b * RP + i];
            c = warp_best(c);
            if (lane == 0) a.blk_best[(size_t)(b0 + b) * gridDim.x + blockIdx.x] = c;
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = (atomicAdd(&a.ticket[blockIdx.y], 1u) == gridDim.x - 1) ? 1u : 0u;
        __syncthreads();
        if (s_last) {
            __threadfence();
            for (int b = warp; b < nb; b += kGmWarps) {
                Cand c{-INFINITY, 0xffffffffu};
                for (int gi = lane; gi < (int)gridDim.x; gi += 32) {
                    const Cand* src = &a.blk_best[(size_t)(b0 + b) * gridDim.x + gi];
                    Cand o;
                    o.s = __ldcg(&src->s);
                    o.i = __ldcg(&src->i);
                    if (cand_better(o, c)) c = o;
                }
                c = warp_best(c);
                if (lane == 0) {
                    a.best_ids[b0 + b] = (c.i == 0xffffffffu) ? 0u : c.i;
                    a.best_scores[b0 + b] = c.s;
                }
            }
            if (tid == 0) a.ticket[blockIdx.y] = 0u;       // ready for the next launch / replay
        }
    }
    if (!ok && lane == 0) {                            // no copy may be in flight when the CTA ends
        for (int i = 0; i < NS && (rb < irb || (rb == irb && cb < icb)); ++i) {
            if (!mbar_wait(&bar[slot], phase)) break;
            next_item(rb, cb);
            if (++slot == NS) { slot = 0; phase ^= 1; }
        }
    }
    stamp(a.ts, 3);
}

}  // namespace oxg4
