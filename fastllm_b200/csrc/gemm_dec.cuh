// The GEMM of calls with few activation rows: out[slice][row][n] = (hi + lo)[R, K] . W[N, K]^T for R <= 128, sm_100a only.
//
// The weights are read once and are nearly all the traffic; they are the 128-row MMA operand, the activations a tile of BN rows whose hi
// and lo halves lie back to back in a stage and are multiplied by one MMA of N = 2 BN.  What bounds it: HBM, behind 4 to 5 us per launch from the
// wait to the first product and from the last weight to the next kernel's start.  The work is cut evenly: the (weight tile, k) stages of
// the whole matrix lie in a row and every block takes L of them, across tile borders.  A tile that several blocks share leaves a slice per
// block, in k order; whoever has the tile's end writes zeros into the slices that the tile does not need, so the consumer adds the same number
// everywhere (a fixed order: deterministic, no atomics).  gemm_tc_kernel, which did this before, cut every tile alike until the items filled
// whole waves: 28672 x 4096 became 13 slices, 20 items of 5 k blocks per block, and the walk from item to item cost as much as a k block.
// One launch behind another with a small kernel between them, cold weights, 8 rows: 6144 x 4096 12.9 -> 11.4 us, 4096 x 4096 9.9 -> 9.0,
// 28672 x 4096 41.1 -> 38.3 (2 slices instead of 13), 4096 x 14336 23.1 -> 21.3; 64 rows: 13.2 -> 12.8, 10.7 -> 10.0, 45.6 -> 42.6, 25.4 -> 24.3.
#pragma once
#include "gemm_tc.cuh"

namespace fl {

// How a matrix of few-row products is cut: stages of KS k blocks (64 columns) of a 128-row weight tile, L stages per block.
struct DecPlan { int nks = 0, L = 0, ctas = 0, slices = 0; };
constexpr int kDecMaxSlices = 16;
// k blocks that the tensor core adds up before the epilogue's registers take over: its adder truncates, so sums of a whole tile (64 k blocks, and
// 224 at K = 14336) were further from 64 bits than the slices of 5 to 25 k blocks that the consumer used to add (logits of a 4096-wide
// layered model: 1.1e-5, whole tiles 1.3e-5, chains of 8: see the tests' bounds and the measured calls).
constexpr int kDecChain = 8;
__host__ __device__ constexpr int dec_ks(int BN) { return BN <= 32 ? 2 : 1; }
inline int dec_bn(int R) { return R <= 16 ? 16 : (R <= 32 ? 32 : (R <= 64 ? 64 : 128)); }
inline DecPlan dec_plan(int N, int K, int R) {
    const int cols = kGemmBK * dec_ks(dec_bn(R)), tiles = (N + kGemmBM - 1) / kGemmBM;
    auto cut = [&](int nks, int L) {
        DecPlan p{nks, L, (tiles * nks + L - 1) / L, 0};
        for (int m = 0; m < tiles; ++m) p.slices = std::max(p.slices, ((m + 1) * nks - 1) / L - m * nks / L + 1);
        return p;
    };
    const int nks = (K + cols - 1) / cols;
    const DecPlan even = cut(nks, std::max((tiles * nks + kNumSMs - 1) / kNumSMs, (nks + kDecMaxSlices - 2) / (kDecMaxSlices - 1)));
    // Cuts at the same places in every tile leave fewer slices to their consumers.  Up to a fifth fewer blocks still keep HBM as busy
    // (4096 x 4096 and 4096 x 14336, 8 rows: 147 blocks, 6 slices 8.8 and 21.5 us; 128 blocks, 4 slices 9.0 and 21.3); one slice less is not worth
    // it (32000 x 4096: 2 slices 42.1 us, 125 blocks of one slice 43.7).  Whole steps of three layers and a vocabulary of 32000, even -> aligned, us,
    // 8, 32, 64 and 128 rows: Mistral-7B's sizes 327 -> 322, 369 -> 363, 414 -> 408, 537 -> 523, TinyLlama's 151 -> 152, 174 -> 174, 205 -> 200, 254 -> 248,
    // Qwen2.5-7B's 331 -> 333, 372 -> 367, 414 -> 414, 520 -> 524.
    for (int L = even.L; 5 * L <= 6 * even.L; ++L)
        if (nks % L == 0 && nks / L + 2 <= even.slices) return cut(nks, L);
    return even;
}

// floats that the slices of R rows and up to N columns take: L >= tiles nks / 148, so a tile has at most 148 / tiles + 2 of them
inline size_t dec_scratch(size_t R, size_t N) { return R * (2 * N + (kNumSMs + 2) * kGemmBM); }

struct DecArgs {
    int N, R, K;
    float* out;                 // [slices][R][N]
    long long split_stride;
    int nks, L, slices;         // as the plan says
};

template <int BN> struct DecShape {
    static constexpr int KS = dec_ks(BN);
    static constexpr uint32_t kW = kGemmBM * kGemmBK * 2, kX = BN * kGemmBK * 2;      // one weight box, one half of the activations
    static constexpr uint32_t kStage = KS * (kW + 2 * kX);
    static constexpr int kStages = 204800 / kStage < 6 ? 204800 / kStage : 6;
    // a warp per 32 lanes and 32-column chunk of the accumulator: warps without a chunk would only hold registers that the blocks of the
    // neighbouring kernels need to be set up beside this one
    static constexpr int kEpi = 4 * (BN <= 32 ? 1 : BN / 32), kThreads = 64 + 32 * kEpi;
    static constexpr uint32_t kAcc = 2 * BN, kTmem = 2 * kAcc;                         // W . hi | W . lo, two stages
    static constexpr size_t kSmem = (size_t)kStages * kStage + 1024;
};

template <int BN>
__global__ void __launch_bounds__(DecShape<BN>::kThreads, 1)
gemm_dec_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmH, const __grid_constant__ CUtensorMap tmL, const DecArgs g) {
    using S = DecShape<BN>;
    constexpr int KS = S::KS, kStages = S::kStages;
    extern __shared__ uint8_t gsm_raw[];
    uint8_t* gsm = gsm_raw + ((1024u - (smem_u32(gsm_raw) & 1023u)) & 1023u);
    __shared__ __align__(8) uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_s;
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int nks = g.nks;
    const int tiles = (g.N + kGemmBM - 1) / kGemmBM;
    const int u0 = blockIdx.x * g.L, u1 = min(u0 + g.L, tiles * nks);       // this block's stages of the flattened (tile, k) walk

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], S::kEpi); }
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(&tmem_base_s, S::kTmem);
    if (threadIdx.x == 32 * 2) { tma_prefetch_desc(&tmH); tma_prefetch_desc(&tmL); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;

    if (warp == 0) {
        if (lane == 0) {
            auto weights = [&](int u, int st) {
                const int m0 = u / nks * kGemmBM, k0 = u % nks * (KS * kGemmBK);
                uint8_t* sa = gsm + (size_t)st * S::kStage;
                mbar_expect_tx(&full[st], S::kStage);
#pragma unroll
                for (int k = 0; k < KS; ++k) tma_load_2d(sa + k * S::kW, &tmW, k0 + k * kGemmBK, m0, &full[st]);
            };
            auto rows = [&](int u, int st) {
                const int k0 = u % nks * (KS * kGemmBK);
                uint8_t* sx = gsm + (size_t)st * S::kStage + KS * S::kW;
#pragma unroll
                for (int k = 0; k < KS; ++k) {
                    tma_load_2d(sx + 2 * k * S::kX, &tmH, k0 + k * kGemmBK, 0, &full[st]);
                    tma_load_2d(sx + (2 * k + 1) * S::kX, &tmL, k0 + k * kGemmBK, 0, &full[st]);
                }
            };
            // the weights do not depend on the kernels before this one: the first ring-full is requested ahead of the wait
            const int pre = min(u1, u0 + kStages);
            for (int u = u0; u < pre; ++u) weights(u, u - u0);
            pdl_wait();
            asm volatile("fence.proxy.async;" ::: "memory");      // the previous kernel's generic-proxy stores -> TMA reads
            for (int u = u0; u < pre; ++u) rows(u, u - u0);
            int st = 0;
            uint32_t ph = 0;
            for (int u = pre; u < u1; ++u) {
                mbar_wait(&empty[st], ph);
                weights(u, st);
                rows(u, st);
                if (++st == kStages) { st = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        {                                                         // the whole warp, one elected lane issues (see uniform_warp)
            constexpr uint32_t idesc = umma_idesc_bf16(kGemmBM, 2 * BN);
            const uint64_t base = umma_smem_desc_sw128(gsm);
            int st = 0;
            uint32_t ph = 0, seg = 0;
            for (int u = u0; u < u1; ++seg) {                     // one chain after the other
                const int end = min(min(u1, (u / nks + 1) * nks), u + kDecChain / KS);
                const uint32_t as = seg & 1, tacc = tmem_base + as * S::kAcc;
                mbar_wait(&acc_empty[as], ((seg >> 1) & 1) ^ 1);
                tc_fence_after();
                uint32_t acc = 0;
                for (; u < end; ++u) {
                    const uint64_t sd = base + (uint64_t)(st * (S::kStage >> 4));
                    mbar_wait(&full[st], ph);
                    tc_fence_after();
#pragma unroll
                    for (int k = 0; k < KS; ++k) {
                        const uint64_t a = sd + (uint64_t)((k * S::kW) >> 4), b = sd + (uint64_t)((KS * S::kW + 2 * k * S::kX) >> 4);
#pragma unroll
                        for (int q = 0; q < kGemmBK / 16; ++q) umma_bf16_warp(tacc, a + 2 * q, b + 2 * q, idesc, (k | q) ? 1u : acc);
                    }
                    acc = 1;
                    umma_commit_warp(&empty[st]);
                    if (++st == kStages) { st = 0; ph ^= 1; }
                }
                umma_commit_warp(&acc_full[as]);
            }
        }
    } else {
        const int q = warp & 3, c0 = ((warp - 2) >> 2) * 32;      // TMEM lane quarter (hardware rule), column chunk
        constexpr int kCols = BN < 32 ? BN : 32;
        uint32_t seg = 0;
        for (int u = u0; u < u1;) {
            const int tile = u / nks, end = min(u1, (tile + 1) * nks);
            const int row = tile * kGemmBM + q * 32 + lane;
            const int slice = (int)blockIdx.x - tile * nks / g.L;
            const bool last = end == (tile + 1) * nks;            // the tile's end: the slices behind this one stay zero
            float* o = g.out + (size_t)slice * (size_t)g.split_stride + (size_t)c0 * g.N + row;
            float v[32];
            for (int c = u; c < end; c += kDecChain / KS, ++seg) {
                const uint32_t as = seg & 1, at = tmem_base + as * S::kAcc + ((uint32_t)(q * 32) << 16) + (uint32_t)c0;
                uint32_t r[32];
                mbar_wait(&acc_full[as], (seg >> 1) & 1);
                tc_fence_after();
                tmem_ld32(at, r);
                if (BN >= 32) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t r2[16];
                        tmem_ld16(at + (uint32_t)(BN + 16 * h), r2);
#pragma unroll
                        for (int j = 0; j < 16; ++j) r[16 * h + j] = __float_as_uint(__uint_as_float(r[16 * h + j]) + __uint_as_float(r2[j]));
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(r[j + 16]));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[as]);
#pragma unroll
                for (int j = 0; j < kCols; ++j) v[j] = c == u ? __uint_as_float(r[j]) : v[j] + __uint_as_float(r[j]);
            }
            if (row < g.N) {                                      // for a fixed column the 32 lanes write 32 consecutive floats
#pragma unroll
                for (int j = 0; j < kCols; ++j)
                    if (c0 + j < g.R) o[(size_t)j * g.N] = v[j];
                if (last)
                    for (int s = slice + 1; s < g.slices; ++s) {
                        o += g.split_stride;
                        for (int j = 0; j < kCols && c0 + j < g.R; ++j) o[(size_t)j * g.N] = 0.f;
                    }
            }
            u = end;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, S::kTmem);
    }
}

}  // namespace fl
