// Projection of many activation rows (prompt passes) on pairs of SMs: tcgen05 with cta_group::2, fed by TMA.
//
// out[r, n] = sum_k x[r, k] * W[n, k]   (the reference's cuBLAS contract, crates/oxide-torch-cuda/src/cublas.rs:101-153:
// BF16 operands, f32 accumulation), or x_i[r, i] = bf16(act(gate_i . x_r) * (up_i . x_r)) with the gate and up
// projections in one launch (kernel_module.rs:1441-1458, 1338-1348).
//
// With hundreds of rows a projection is bound by the tensor cores, and what feeds them is shared memory: a 128 x 256 tile
// per SM reads and refills 192 bytes per clock and SM. A pair of CTAs forms one 256 x BN tile instead: each CTA holds 128
// activation rows (the M operand) and half of the BN weight rows (the N operand), which its partner reads as well, so the
// refill is half of that. The tile is activations x weights and not weights x activations as in tc_gemm.cuh: a TMEM lane
// is then an activation row, an epilogue thread owns consecutive output columns (32-byte stores), and gate and up rows of
// one launch meet in one thread (CTA 0 of the pair loads the gate rows, CTA 1 the up rows).
//
//   warp 0, one lane : TMA producer of the CTA's own operands; the pair's bytes are counted on CTA 0's barrier
//   warp 1, one lane : MMA issuer, CTA 0 only (tcgen05.mma.cta_group::2, M = 256); its commits reach both CTAs
//   warps 2..9       : epilogue of the CTA's 128 rows, two warps per TMEM lane quadrant, each half of the columns; two
//                      accumulators of up to 256 TMEM columns, so that the MMAs of the next tile run while this one is stored
//
// Work. Tiles are numbered row tiles fastest. Either the pairs take whole tiles in turn (many tiles: the weight tile crosses
// HBM once and the activations, a few MB, stay in L2), or all k-blocks of all tiles are dealt to the pairs as equal
// contiguous ranges (few tiles: whole ones would leave pairs idle in the last round). A tile that is cut gives one partial
// output per piece, slot = number of the piece inside the tile; the consumers add S slots in order, and the pair with a
// tile's last piece clears the slots that the tile does not use. No multicast loads.
//
// Failures are those of tc_gemm.cuh (bounded waits, `*err`, launches that find it set), for both CTAs together: a CTA that stops
// tells its partner, both meet at a cluster barrier, then CTA 0 waits (bounded) for all copies of the pair in flight, both for the
// MMAs' commits, and they meet again before their shared memory and TMEM go away.
//
// Measured (B200, back-to-back launches): gate/up of the ~4B widths, 2048 rows, 163 us = 1.31 PFLOP/s of 1.40 sustained by
// cuBLAS (weight-streaming kernel, eight blocks of 256 rows: 8 x 64 us + 8 x 15 us for the activation kernel); ~27B widths
// 682 us = 1.39 PFLOP/s; down projection of the ~4B widths 94 us = 1.14 PFLOP/s (8 x 41 us). Eight epilogue warps and not
// four: with 1152 columns a tile's activations took longer than its products (181 -> 74 us).
#pragma once
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "tc_gemm.cuh"

namespace oxg4 {

constexpr int kPgThreads = 320;
constexpr int kPgTileM = 256;        // activation rows of a pair's tile
constexpr int kPgStages = 6;         // 6 x 32 KiB per CTA
constexpr uint32_t kPgHalf = 128 * kTcTileK * 2;          // 16 KiB: 128 rows of 64 BF16 values
constexpr uint32_t kPgStage = 2 * kPgHalf;

enum { PG_STORE = 0, PG_GLU = 1 };

struct PairGemmArgs {
    int M, N, K;             // activation rows, rows of ONE weight matrix, columns
    int bn;                  // weight rows of a tile, both halves together: a multiple of 32, at most 256
    int cut;                 // 1: k-blocks dealt as ranges (PG_STORE only), 0: whole tiles in turn
    int S;                   // most pieces of a tile (1 unless cut)
    float* out;              // PG_STORE: [S, M, ld]
    uint16_t* out_bf16;      // PG_GLU: [M, ld]
    int ld;
    int act;                 // PG_GLU: activation of the gate
    int* err;
};

DEVINL uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}
DEVINL void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the pair's CTA 0 keeps the barriers that both CTAs' copies and epilogues signal: the CTA's own shared address with the
// rank bit of the cluster window cleared
constexpr uint32_t kPairLeadMask = 0xFEFFFFFFu;
// the same shared variable in the other CTA of the pair
DEVINL uint32_t partner_addr(const volatile void* p) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32((const void*)p)), "r"(cluster_rank() ^ 1u));
    return a;
}
DEVINL uint32_t ld_partner(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(partner_addr(p)) : "memory");
    return v;
}
DEVINL void pair_stop(volatile int* stop) {
    *stop = 1;
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(partner_addr(stop)), "r"(1) : "memory");
}
DEVINL void pair_failed(int* err, int code, volatile int* stop) {
    atomicCAS(err, 0, code);
    pair_stop(stop);
}
// Between the two closing cluster barriers of a failed pair, one thread per CTA. CTA 0's barriers count both CTAs' bytes, which may have
// stopped at different stages: `mine` / `theirs` stages filled, `half` bytes each.
DEVINL void pair_drain(uint64_t* full, uint64_t* empty, uint64_t* acc_full, uint32_t rank, uint32_t mine, uint32_t theirs, uint32_t half,
                       uint32_t committed, uint32_t accs) {
    if (rank == 0) {
        for (uint32_t i = mine; i < theirs; ++i) mbar_expect_tx(&full[i % kPgStages], half);
        for (uint32_t i = theirs; i < mine; ++i)                // bytes that the partner did not send
            asm volatile("mbarrier.complete_tx.relaxed.cluster.shared::cta.b64 [%0], %1;"
                         ::"r"(smem_u32(&full[i % kPgStages])), "r"(half) : "memory");
    }
    ring_drain(full, empty, kPgStages, rank == 0 ? max(mine, theirs) : 0u, committed);
    if (accs > 0) mbar_wait(&acc_full[(accs - 1) & 1], ((accs - 1) >> 1) & 1);
}

DEVINL void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar) & kPairLeadMask)
        : "memory");
}
DEVINL void mbar_arrive_lead(uint64_t* bar) {
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, 0;\n\t"
                 "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [a];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
// completion of this thread's MMAs so far, signalled to the barrier at the same address in both CTAs
DEVINL void mma_commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
DEVINL void tmem_ld16(uint32_t (&v)[16], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(addr));
}
DEVINL void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
DEVINL void st_global_32b(void* p, const uint32_t* v) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

// The pieces of tiles that a pair works on, in order; every role of the pair walks the same sequence.
struct PairWalk {
    int tile, kb0, kb1, piece;           // k-blocks [kb0, kb1) of `tile`, the tile's piece number `piece`
    int pos, end, step, KB, cut, q, rem; // pos: next tile (whole tiles) or next k-block over all tiles (ranges)
    DEVINL PairWalk(int pair, int pairs, int n_tiles, int KB_, int cut_) : KB(KB_), cut(cut_) {
        if (cut) {
            const int W = n_tiles * KB;
            q = W / pairs;
            rem = W % pairs;
            pos = pair * q + min(pair, rem);
            end = pos + q + (pair < rem ? 1 : 0);
            step = pair;                 // ranges: this pair's number
        } else {
            pos = pair;
            end = n_tiles;
            step = pairs;
            q = rem = 0;
        }
    }
    DEVINL bool next() {
        if (pos >= end) return false;
        if (!cut) {
            tile = pos;
            kb0 = 0;
            kb1 = KB;
            piece = 0;
            pos += step;
            return true;
        }
        tile = pos / KB;
        kb0 = pos - tile * KB;
        kb1 = min(KB, kb0 + end - pos);
        const int first = tile * KB, bound = rem * (q + 1);       // the pair that starts the tile
        piece = step - (first < bound ? first / (q + 1) : rem + (first - bound) / q);
        pos += kb1 - kb0;
        return true;
    }
};

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPgThreads, 1)
pair_gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                 const __grid_constant__ CUtensorMap map_w1, const PairGemmArgs a) {
    extern __shared__ unsigned char pg_dyn[];
    unsigned char* tiles = (unsigned char*)(((uintptr_t)pg_dyn + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full[kPgStages], empty[kPgStages], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int failed;
    __shared__ uint32_t issued, committed, accs;               // ring stages filled, stages and accumulators whose MMAs were committed

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();
    const int pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
    const int cols = EPI == PG_GLU ? a.bn / 2 : a.bn;          // output columns of a tile
    const int tiles_m = (a.M + kPgTileM - 1) / kPgTileM, tiles_n = (a.N + cols - 1) / cols;
    const int kblocks = (a.K + kTcTileK - 1) / kTcTileK;
    const PairWalk start(pair, pairs, tiles_m * tiles_n, kblocks, a.cut);
    const uint32_t half_bytes = (uint32_t)(a.bn / 2) * kTcTileK * 2;
    if (tid == 0) {
        for (int s = 0; s < kPgStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 16); }
        failed = 0;
        committed = accs = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();                                          // lane 0 comes from the barriers
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    __syncwarp();
    cluster_sync_all();                                        // both CTAs' barriers exist before anyone signals them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;

    if (warp == 0 && lane == 0) {
        // ---- TMA producer: the CTA's 128 activation rows and its half of the weight rows ----
        PairWalk w = start;
        int kb = 0, xrow = 0, wrow = 0;
        const CUtensorMap* wm = (EPI == PG_GLU && rank == 1) ? &map_w1 : &map_w;
        auto enter = [&]() {
            if (!w.next()) return false;
            const int n0 = w.tile / tiles_m * cols;
            kb = w.kb0;
            xrow = w.tile % tiles_m * kPgTileM + (int)rank * 128;
            wrow = EPI == PG_GLU ? n0 : n0 + (int)rank * (a.bn / 2);
            return true;
        };
        bool more = enter();
        auto advance = [&]() {
            if (++kb == w.kb1) more = enter();
        };
        // the first ring of weight tiles depends on nothing the preceding kernel writes
        int pre_k[kPgStages], pre_x[kPgStages], n_pre = 0;
        while (n_pre < kPgStages && more) {
            if (rank == 0) mbar_expect_tx(&full[n_pre], 2 * (kPgHalf + half_bytes));
            tma_load_2d_pair(tiles + (size_t)n_pre * kPgStage + kPgHalf, wm, kb * kTcTileK, wrow, &full[n_pre]);
            pre_k[n_pre] = kb * kTcTileK;
            pre_x[n_pre] = xrow;
            ++n_pre;
            advance();
        }
        pdl_wait();
        pdl_launch();
        for (int i = 0; i < n_pre; ++i) tma_load_2d_pair(tiles + (size_t)i * kPgStage, &map_x, pre_k[i], pre_x[i], &full[i]);
        uint32_t it = (uint32_t)n_pre;
        for (; more && !failed; ++it) {
            const int s = it % kPgStages;
            if (!mbar_wait(&empty[s], ((it / kPgStages) & 1) ^ 1, &failed)) { pair_failed(a.err, 1, &failed); break; }
            if (rank == 0) mbar_expect_tx(&full[s], 2 * (kPgHalf + half_bytes));
            tma_load_2d_pair(tiles + (size_t)s * kPgStage, &map_x, kb * kTcTileK, xrow, &full[s]);
            tma_load_2d_pair(tiles + (size_t)s * kPgStage + kPgHalf, wm, kb * kTcTileK, wrow, &full[s]);
            advance();
        }
        // every stage has been read, so every copy has landed and every commit has been signalled, before the CTA ends
        const uint32_t tail = min(it, (uint32_t)kPgStages);
        for (uint32_t i = it - tail; i < it; ++i)
            if (!mbar_wait(&empty[i % kPgStages], (i / kPgStages) & 1, &failed)) { pair_failed(a.err, 5, &failed); break; }
        issued = it;
    } else {
        pdl_wait();
        pdl_launch();
    }
    if (warp == 1 && lane == 0 && rank == 0) {
        // ---- MMA issuer of the pair ----
        const uint32_t idesc = umma_idesc_bf16(kPgTileM, a.bn);
        uint32_t it = 0, tile_i = 0;
        PairWalk w = start;
        for (; !failed && w.next(); ++tile_i) {
            const uint32_t ab = tile_i & 1, use = tile_i >> 1;
            if (use > 0 && !mbar_wait(&acc_empty[ab], (use - 1) & 1, &failed)) { pair_failed(a.err, 2, &failed); break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem + ab * 256;
            const int nk = w.kb1 - w.kb0;
            for (int j = 0; j < nk; ++j, ++it) {
                const int s = it % kPgStages;
                if (!mbar_wait(&full[s], (it / kPgStages) & 1, &failed)) { pair_failed(a.err, 3, &failed); break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned char* sa = tiles + (size_t)s * kPgStage;
                const uint64_t da = umma_smem_desc(sa), db = umma_smem_desc(sa + kPgHalf);
#pragma unroll
                for (int k = 0; k < kTcTileK / 16; ++k) {
                    const uint32_t accumulate = (j > 0 || k > 0) ? 1u : 0u;
                    asm volatile(
                        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                        ::"r"(acc), "l"(da + (uint64_t)(2 * k)), "l"(db + (uint64_t)(2 * k)), "r"(idesc), "r"(accumulate)
                        : "memory");
                }
                mma_commit_pair(&empty[s]);
            }
            committed = it;
            if (failed) break;
            mma_commit_pair(&acc_full[ab]);
            accs = tile_i + 1;
        }
    }
    __syncwarp();

    // ---- epilogue: warps 2..9; thread = TMEM lane = activation row ----
    if (warp >= 2) {
        const int quad = warp & 3, part = (warp - 2) >> 2;
        uint32_t tile_i = 0;
        PairWalk w = start;
        const bool dead = failed_before(a.err);
        if (dead && lane == 0) pair_stop(&failed);
        for (; !dead && w.next(); ++tile_i) {
            const uint32_t ab = tile_i & 1, use = tile_i >> 1;
            if (!mbar_wait_warp(&acc_full[ab], use & 1, &failed)) { if (lane == 0) pair_failed(a.err, 4, &failed); break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int n0 = w.tile / tiles_m * cols;
            const int row = w.tile % tiles_m * kPgTileM + (int)rank * 128 + quad * 32 + lane;
            const bool row_ok = row < a.M;
            const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + ab * 256;
            if constexpr (EPI == PG_STORE) {
                float* dst = a.out + ((size_t)w.piece * a.M + row) * a.ld + n0;
                const bool vec = (a.ld & 7) == 0;
                for (int c0 = part * 32; c0 < a.bn; c0 += 64) {
                    uint32_t v[2][16];
                    __syncwarp();                              // rows past M skip the stores: all lanes meet before the aligned loads
                    tmem_ld16(v[0], taddr + (uint32_t)c0);
                    tmem_ld16(v[1], taddr + (uint32_t)c0 + 16);
                    tmem_ld_wait();
                    if (!row_ok) continue;
                    if (vec && n0 + c0 + 32 <= a.N) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) st_global_32b(dst + c0 + q * 8, &v[q >> 1][(q & 1) * 8]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (n0 + c0 + j < a.N) dst[c0 + j] = __uint_as_float(v[j >> 4][j & 15]);
                    }
                }
                if (w.kb1 == kblocks && w.piece + 1 < a.S && row_ok) {      // slots that this tile does not use
                    const uint32_t zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                    for (int sl = w.piece + 1; sl < a.S; ++sl) {
                        float* z = a.out + ((size_t)sl * a.M + row) * a.ld + n0;
                        for (int c0 = part * 8; c0 < a.bn; c0 += 16) {
                            if (vec && n0 + c0 + 8 <= a.N) st_global_32b(z + c0, zero);
                            else
                                for (int j = 0; j < 8; ++j)
                                    if (n0 + c0 + j < a.N) z[c0 + j] = 0.0f;
                        }
                    }
                }
            } else {
                uint16_t* dst = a.out_bf16 + (size_t)row * a.ld + n0;
                const bool vec = (a.ld & 15) == 0;
                for (int c0 = part * 16; c0 < cols; c0 += 32) {
                    uint32_t g[16], up[16], o[8];
                    __syncwarp();
                    tmem_ld16(g, taddr + (uint32_t)c0);
                    tmem_ld16(up, taddr + (uint32_t)(cols + c0));
                    tmem_ld_wait();
                    if (!row_ok) continue;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float x0 = glu_mul(a.act, __uint_as_float(g[2 * j]), __uint_as_float(up[2 * j]));
                        const float x1 = glu_mul(a.act, __uint_as_float(g[2 * j + 1]), __uint_as_float(up[2 * j + 1]));
                        o[j] = f32_to_bf16_bits(x0) | (f32_to_bf16_bits(x1) << 16);
                    }
                    if (vec && n0 + c0 + 16 <= a.N) {
                        st_global_32b(dst + c0, o);
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (n0 + c0 + j < a.N) dst[c0 + j] = (uint16_t)(o[j >> 1] >> ((j & 1) * 16));
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_lead(&acc_empty[ab]);
        }
    }

    // ---- teardown: always reached, also after a failed wait ----
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    __syncwarp();
    cluster_sync_all();
    if (failed) {                                              // the same in all threads of the pair: nobody sets it behind the barrier
        if (tid == 0)
            pair_drain(full, empty, acc_full, rank, issued, ld_partner(&issued), kPgHalf + half_bytes, rank == 0 ? committed : ld_partner(&committed),
                       rank == 0 ? accs : ld_partner(&accs));
        __syncthreads();
        __syncwarp();
        cluster_sync_all();
    }
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
}

inline size_t pair_gemm_smem_bytes() { return (size_t)kPgStage * kPgStages + 1024; }

// How a projection is cut for M rows: tile width, pairs, ranges or whole tiles, slots of partial outputs.
struct PairPlan {
    int bn = 256, pairs = 1, cut = 0, S = 1;
};

// most pieces of a tile when n_tiles tiles of KB k-blocks are dealt to `pairs` equal ranges
inline int pair_pieces(int n_tiles, int KB, int pairs) {
    const long long W = (long long)n_tiles * KB, q = W / pairs, rem = W % pairs;
    auto owner = [&](long long w) { return w < rem * (q + 1) ? w / (q + 1) : rem + (w - rem * (q + 1)) / q; };
    int most = 1;
    for (int t = 0; t < n_tiles; ++t) most = std::max(most, (int)(owner((long long)(t + 1) * KB - 1) - owner((long long)t * KB)) + 1);
    return most;
}

// The cheapest plan by the times measured for single launches (B200, 64-column blocks): a pair takes 0.42 us per k-block of a
// 256-wide tile and hardly less for a narrower one (0.37 us at 128: the refill of shared memory and not the tensor cores
// sets the pace), about 3 us to start and drain; every slot of partial outputs is written and read once (~4.5 TB/s).
// max_rows: rows of `ld` floats that the output buffer holds (slots * M must fit). glu: gate and up in one launch.
inline PairPlan pair_plan(int M, int N, int K, bool glu, size_t max_rows, int num_sms) {
    const int P = num_sms / 2, KB = (K + kTcTileK - 1) / kTcTileK, tiles_m = (M + kPgTileM - 1) / kPgTileM;
    PairPlan best;
    double best_us = 1e30;
    for (int bn : {256, 224, 192, 160, 128}) {
        const int cols = glu ? bn / 2 : bn, T = tiles_m * ((N + cols - 1) / cols);
        const double kb_us = bn == 128 ? 0.37 : bn == 160 ? 0.41 : 0.42;
        auto consider = [&](int pairs, int cut) {
            const int S = cut ? pair_pieces(T, KB, pairs) : 1;
            if ((size_t)S * M > max_rows && S > 1) return;
            const long long blocks = cut ? ((long long)T * KB + pairs - 1) / pairs : (long long)((T + pairs - 1) / pairs) * KB;
            const double us = blocks * kb_us + 3.0 + (S > 1 ? S * 8.0 * M * N / 4.5e6 : 0.0);
            if (us < best_us - 1e-6) {
                best_us = us;
                best.bn = bn; best.pairs = pairs; best.cut = cut; best.S = S;
            }
        };
        consider(std::min(T, P), 0);
        if (glu || T >= 4 * P) continue;                      // ranges of whole weight matrices would defeat L2
        if ((long long)T * KB >= P) consider(P, 1);
        for (int s = 2; s * T <= P && s <= KB; ++s) consider(s * T, 1);
    }
    return best;
}

}  // namespace oxg4
