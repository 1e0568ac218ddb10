// The GEMM of calls with many activation rows: D[M, N] = (hi + lo)[M, K] . W[N, K]^T with the epilogues of gemm_tc_kernel, on pairs of SMs.
//
// Two CTAs of a cluster work on one 256 x 256 tile (tcgen05.mma.cta_group::2): each holds its 128 rows of the activations (hi and lo) and half of
// the weight tile, 48 KB per k block where a single CTA with a 128 x 256 tile fetches 64.  What bounds it: the tensor cores under the power limit
// (1.65 to 1.69 PFLOP/s of issued products in bursts, 1.4 to 1.55 inside a long call; singles 1.64 to 1.66 where their waves are full).
// Tiles that do not fill a wave are cut along K, evenly over all pairs (as gemm_dec_kernel cuts all of its work): a part of a tile goes to the
// workspace, the last of its parts to arrive adds them up in k order and runs the epilogue (nobody waits for anybody).  448 tiles of a 4096 x 3584
// output took four waves of 148 for 3.03 waves of work.  In turn with the single CTAs, single -> pairs: 4096 x 3584 x 18944 805 -> 672 us,
// 4096 x 3584 x 3584 155 -> 139, 4096 x 37888 x 3584 1341 -> 1315, 2048 x 14336 (gated) x 4096 587 -> 578, 2048 x 16448 x 4096 357 -> 339.
#pragma once
#include "gemm_tc.cuh"

namespace fl {

constexpr int kPairStages = 4, kPairEpiWarps = 16, kPairThreads = 64 + 32 * kPairEpiWarps;
constexpr uint32_t kPairABytes = 128 * 64 * 2, kPairStage = 3 * kPairABytes;      // hi | lo rows of this CTA, its half of the weight tile
constexpr size_t kPairSmem = (size_t)kPairStages * kPairStage + 1024;
constexpr int kPairMaxSlices = 8;
constexpr int kPairMaxClusters = kNumSMs / 2;
constexpr size_t kPairWsFloats = (size_t)kPairMaxClusters * 2 * 2 * 128 * 256;    // [cluster][first | second tile of its range][CTA][column][row]

struct PairArgs {
    GemmArgs g;                 // M, N, K, bias, out, ldo, out2, act, act_limit as gemm_tc_kernel takes them
    int nk, mp, nt;             // k blocks; pair rows (256 rows each) and column tiles
    int full, L;                // whole tiles per cluster, then k blocks per cluster of the tiles that are left
    float* ws;                  // parts of shared tiles
    int* tickets;               // [2 tiles left]: zero between launches
    int* failed;                // set when a wait ran out
};
struct PairPlan { int nk, mp, nt, clusters, full, L; };
// glu: a tile is 128 gate and the 128 matching up rows
inline PairPlan pair_plan(int M, int N, int K, bool glu, int max_clusters) {
    PairPlan p;
    p.nk = (K + kGemmBK - 1) / kGemmBK;
    p.mp = (M + 255) / 256;
    p.nt = glu ? (N + 127) / 128 : (N + 255) / 256;
    const int T = p.mp * p.nt;
    p.clusters = max_clusters;
    p.full = T / p.clusters;
    const int left = T % p.clusters;
    p.L = left == 0 ? 1 : std::max((left * p.nk + p.clusters - 1) / p.clusters, (p.nk + kPairMaxSlices - 2) / (kPairMaxSlices - 1));
    if (p.full == 0) p.clusters = (left * p.nk + p.L - 1) / p.L;
    return p;
}
// Whether pairs are the faster way, counted in k blocks of a tile: a single CTA's tiles fill whole waves of 148, pairs pay about 20 k blocks for
// the parts of shared tiles (their way through the workspace) and 12 for the rest.  Single -> pairs, us, by the pairs (of 74) that a last wave would
// fill: 10 (1536 x 3584 x 18944) 400 -> 275, 12 (2560 x 4096 x 14336) 482 -> 379, 22 (1536 x 4096 x 14336) 295 -> 228, 38 (2048 x 3584 x 18944)
// 410 -> 375, 48 (3584 x 3584 x 18944) 636 -> 602, 54 (2048 x 4096 x 14336) 314 -> 316, 66 (2560 x 3584 x 18944) 440 -> 454: a last wave that is nearly full
// runs at a higher clock than the whole chip does under the power limit.  The line lies at a quarter of a wave and not at the two thirds up to which
// single shapes gain, because cut tiles are sums in another order, and a whole prompt of 2048 rows and width 4096 with the line there took 6.43 ms instead of
// 6.44 at a distance from 64 bits of 5.5e-4 instead of 5.4e-4.  K = 2048 is too short for any of it: 3072 x 11264 x 2048, 10: 193 -> 215.
constexpr int kPairMinRows = 1024;
inline bool pair_wins(const PairPlan& p, int M, int max_clusters) {
    const int T = p.mp * p.nt, left = T - p.full * max_clusters, single = ((M + 127) / 128 * p.nt + kNumSMs - 1) / kNumSMs * p.nk;
    if (M < kPairMinRows || p.full == 0 || 4 * left > max_clusters) return false;
    return left == 0 ? p.full >= 4 && p.full * p.nk <= single : p.full * p.nk + p.L + 20 + 12 <= single;
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// completes on a barrier of the pair's first CTA (mbar: its shared::cluster address)
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* tmap, int c0, int c1, uint32_t mbar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(tmap),
                 "r"(c0), "r"(c1), "r"(mbar)
                 : "memory");
}
// a whole warp: one elected lane issues
__device__ __forceinline__ void umma_bf16_pair_warp(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p, e;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "elect.sync _|e, 0xFFFFFFFF;\n"
        "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on the barrier of both CTAs when all products issued so far have completed
__device__ __forceinline__ void umma_commit_pair_warp(uint64_t* bar) {
    asm volatile(
        "{\n"
        ".reg .pred e;\n"
        "elect.sync _|e, 0xFFFFFFFF;\n"
        "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
        "}\n" ::"r"(smem_u32(bar)),
        "h"((uint16_t)3)
        : "memory");
}
// Release at cluster scope: the waits of the pair acquire there, and the default scope, the CTA, would order nothing for the other CTA.  In
// bert_block_kernel these arrives are what stands between the second CTA's operand stores and the products that the first one issues over them.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// orders nothing but itself: for what is no memory
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// false when the wait ran out (seconds): the caller leaves its loop
__device__ __forceinline__ bool pair_wait(uint64_t* bar, uint32_t parity) {
    for (int i = 0; i < (1 << 20); ++i) {
        uint32_t done;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmH, const __grid_constant__ CUtensorMap tmL, const __grid_constant__ CUtensorMap tmW, const PairArgs p) {
    static_assert(EPI == GEPI_F32 || EPI == GEPI_SILU_HL || EPI == GEPI_GLU_HL, "epilogues of the many-row GEMMs");
    constexpr bool kGlu = EPI == GEPI_GLU_HL;
    const GemmArgs& g = p.g;
    extern __shared__ uint8_t gsm_raw[];
    uint8_t* gsm = gsm_raw + ((1024u - (smem_u32(gsm_raw) & 1023u)) & 1023u);      // (the same offset in both CTAs)
    __shared__ __align__(8) uint64_t full[kPairStages], empty[kPairStages], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ int s_last;
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int cl = blockIdx.x >> 1, G = gridDim.x >> 1, nk = p.nk, T = p.mp * p.nt;
    const int left0 = p.full * G, units = (T - left0) * nk;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kPairStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 2 * kPairEpiWarps); }
        mbar_fence_init();
        tma_prefetch_desc(&tmH);
        tma_prefetch_desc(&tmL);
        tma_prefetch_desc(&tmW);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;

    // This cluster's work in order: whole tiles cl, cl + G, ..., then its run of k blocks of the tiles that are left.
    // -> false at the end; tile, [kb0, kb1)
    struct Walk { int seg = 0, u = 0; };
    const int u1 = min((cl + 1) * p.L, units);
    auto next = [&](Walk& w, int& tile, int& kb0, int& kb1) {
        if (w.seg < p.full) {
            tile = cl + w.seg * G; kb0 = 0; kb1 = nk;
        } else {
            if (w.seg == p.full) w.u = cl * p.L;
            if (w.u >= u1) return false;
            tile = left0 + w.u / nk; kb0 = w.u % nk; kb1 = min(nk, kb0 + u1 - w.u);
            w.u += kb1 - kb0;
        }
        ++w.seg;
        return true;
    };
    // 8 pair rows share a weight tile before the walk moves on (see kGemmRasterRows)
    auto place = [&](int tile, int& m, int& n) {
        constexpr int RM = kGemmRasterRows / 2;
        const int per = RM * p.nt, first = tile / per * RM, local = tile % per, cnt = min(RM, p.mp - first);
        m = (first + local % cnt) * 256 + (int)rank * 128;
        n = local / cnt * (kGlu ? 128 : 256);
    };
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {
            pdl_wait();
            asm volatile("fence.proxy.async;" ::: "memory");      // the previous kernel's generic-proxy stores -> TMA reads
            Walk w;
            int tile, kb0, kb1, st = 0;
            uint32_t ph = 1;
            while (ok && next(w, tile, kb0, kb1)) {
                int m0, n0;
                place(tile, m0, n0);
                const int wrow = kGlu ? n0 + (int)rank * g.N : n0 + (int)rank * 128;      // the gate rows in the first CTA, the up rows in the second
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!(ok = pair_wait(&empty[st], ph))) break;
                    if (rank == 0) mbar_expect_tx(&full[st], 2 * kPairStage);      // both CTAs' loads complete on the first one's barrier
                    const uint32_t bar = mapa_u32(smem_u32(&full[st]), 0), sa = smem_u32(gsm) + st * kPairStage;
                    tma_load_2d_pair(sa, &tmH, kb * kGemmBK, m0, bar);
                    tma_load_2d_pair(sa + kPairABytes, &tmL, kb * kGemmBK, m0, bar);
                    tma_load_2d_pair(sa + 2 * kPairABytes, &tmW, kb * kGemmBK, wrow, bar);
                    if (++st == kPairStages) { st = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {             // the whole warp, one elected lane issues (see uniform_warp); a wait that ran out ends the waiting, not the walk
            constexpr uint32_t idesc = umma_idesc_bf16(256, 256);
            const uint64_t base = umma_smem_desc_sw128(gsm);
            Walk w;
            int tile, kb0, kb1, st = 0;
            uint32_t ph = 0, seg = 0;
            auto wait = [&](uint64_t* bar, uint32_t parity) {
                if (ok) ok = pair_wait(bar, parity);
                __syncwarp();
                tc_fence_after();
            };
            while (next(w, tile, kb0, kb1)) {
                const uint32_t as = seg & 1, tacc = tmem_base + as * 256;
                wait(&acc_empty[as], ((seg >> 1) & 1) ^ 1);
                for (int kb = kb0; kb < kb1; ++kb) {
                    wait(&full[st], ph);
                    const uint64_t ah = base + (uint64_t)(st * (kPairStage >> 4)), al = ah + (kPairABytes >> 4), b = al + (kPairABytes >> 4);
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_bf16_pair_warp(tacc, ah + 2 * k, b + 2 * k, idesc, ((kb - kb0) | k) ? 1u : 0u);
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_bf16_pair_warp(tacc, al + 2 * k, b + 2 * k, idesc, 1u);
                    umma_commit_pair_warp(&empty[st]);
                    if (++st == kPairStages) { st = 0; ph ^= 1; }
                }
                umma_commit_pair_warp(&acc_full[as]);
                ++seg;
            }
        }
    } else {
        const int q = warp & 3, cs = (warp - 2) >> 2;         // TMEM lane quarter (hardware rule); columns [64 cs, 64 cs + 64) (gated: [32 cs, ..) of both halves)
        const int lrow = q * 32 + lane;
        Walk w;
        int tile, kb0, kb1;
        uint32_t seg = 0;
        while (next(w, tile, kb0, kb1)) {                     // (to the end even behind a wait that ran out: the warps meet at barriers)
            int m0, n0;
            place(tile, m0, n0);
            const uint32_t as = seg & 1;
            if (ok) ok = __all_sync(0xFFFFFFFFu, pair_wait(&acc_full[as], (seg >> 1) & 1));
            ++seg;
            tc_fence_after();
            const uint32_t at = tmem_base + as * 256 + ((uint32_t)(q * 32) << 16);
            const int row = m0 + lrow;
            const bool whole = kb0 == 0 && kb1 == nk;
            const int r = tile - left0;                       // (of a tile that is left)
            bool store = whole;
            int c0 = 0, c1 = 0;
            if (!whole) {
                // this part's columns to the workspace, 32 consecutive rows per store; the last part of the tile to arrive reads all of them back
                c0 = r * nk / p.L; c1 = ((r + 1) * nk - 1) / p.L;
                float* part = p.ws + ((size_t)((cl * 2 + r - cl * p.L / nk) * 2 + (int)rank) * 256) * 128 + lrow;
#pragma unroll 1
                for (int c = cs * 64; ok && c < cs * 64 + 64; c += 32) {
                    uint32_t v[32];
                    tmem_ld32(at + (uint32_t)c, v);
#pragma unroll
                    for (int j = 0; j < 32; ++j) part[(size_t)(c + j) * 128] = __uint_as_float(v[j]);
                }
                asm volatile("bar.sync 1, %0;" ::"n"(32 * kPairEpiWarps) : "memory");
                if (threadIdx.x == 64 && ok) {
                    __threadfence();
                    int* t = p.tickets + 2 * r + (int)rank;
                    s_last = atomicAdd(t, 1) == c1 - c0;
                    if (s_last) *t = 0;
                    __threadfence();
                }
                asm volatile("bar.sync 1, %0;" ::"n"(32 * kPairEpiWarps) : "memory");
                store = s_last != 0;
            }
            // 16 columns from column c on: of the accumulator, or of the tile's parts in k order
            auto get = [&](int c, float (&o)[16]) {
                if (whole) {
                    uint32_t v[16];
                    tmem_ld16(at + (uint32_t)c, v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) o[j] = __uint_as_float(v[j]);
                    return;
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) o[j] = 0.f;
                for (int s0 = c0; s0 <= c1; s0 += 2) {
                    float v[2][16];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int s = min(s0 + u, c1);
                        const float* part = p.ws + ((size_t)((s * 2 + r - s * p.L / nk) * 2 + (int)rank) * 256 + c) * 128 + lrow;
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[u][j] = __ldcg(part + (size_t)j * 128);
                    }
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        if (s0 + u <= c1) {
#pragma unroll
                            for (int j = 0; j < 16; ++j) o[j] += v[u][j];
                        }
                }
            };
            if (store && ok) {
#pragma unroll 1
                for (int i = 0; i < (kGlu ? 2 : 4); ++i) {
                    const int c = kGlu ? cs * 32 + i * 16 : cs * 64 + i * 16;      // column of the tile's output
                    float a[16];
                    get(c, a);
                    if constexpr (kGlu) {
                        float b[16];
                        get(c + 128, b);
                        if (row < g.M && n0 + c < g.N) glu_store16(g, row, n0 + c, a, b);
                    } else if constexpr (EPI == GEPI_SILU_HL) {
                        if (row < g.M && n0 + c < g.N) silu_store16(g, row, n0 + c, a);
                    } else {
                        if (row < g.M) f32_store16(g, row, n0 + c, a);
                    }
                    __syncwarp();
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&acc_empty[as]), 0));
        }
    }
    if (!ok) {                   // a wait ran out: report it, leave the copies in flight time to land, go on to the end
        if (lane == 0 && p.failed != nullptr) *p.failed = 1;
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // the other CTA's products read this one's shared memory, its epilogue arrives on this one's barriers
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

}  // namespace fl
