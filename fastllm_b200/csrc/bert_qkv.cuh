// The front of an encoder layer in one kernel: q|k|v = x Wqkv^T + b and, per sentence and head, softmax(q k^T / sqrt(d)) v, for sentences of up to 128
// tokens, hidden 384 and 12 heads of 32 (all-MiniLM-L6-v2), sm_100a only.  Restates models/embeddings.rs:130-166 as the GEMM and bert_attn_kernel do: same
// operands, same order of products, q, k, v and the probabilities in bf16 where theirs are.
//
// Two CTAs of a cluster take two groups of whole sentences of up to 128 rows each (tcgen05.mma.cta_group::2, see gemm_pair.cuh: a single CTA would read
// every weight from L2 for 128 tokens, 18 TB/s at the tensor cores' rate).  A unit of work is up to three heads of such a pair: 288 columns of q|k|v in TMEM,
// rounded into shared memory by twelve warps, which then are the attention's (mma.sync, a sentence's 16 query rows of a head at a time) while the tensor
// core makes the next unit's columns.  The clusters take equal runs of heads (up to four heads a run none crosses from one pair of groups to the next: 60 x 43
// tokens 366 -> 354 us, 36 x 65 354 -> 345); x stays in shared memory over the units of a pair.
// q, k and v never leave the SM: the GEMM and the attention moved 75 MB each way between them at 256 x 128 tokens.
// Whole encoder, GEMM and attention -> this kernel, us (with the block kernel as it is): 256 x 128 tokens 1280 -> 1107, 76 x 128 552 -> 517, 400 x 43 788 ->
// 645, 1500 x 20 1690 -> 1177, 60 x 43 377 -> 354; a layer of 256 x 128: 87 -> 66.  (Runs of whole units of three heads: 76 x 128 567.)
// A unit of 128-token sentences takes about 14500 clocks: 2200 to bring q|k|v into shared memory, 12000 of attention in which the tensor core's 3700 for
// the next unit run -- the warps' products (3300), ex2 (3100) and shared memory (3300 and the operands of the other products) would overlap better with
// more warps than the registers allow (eight warps of 168 registers: 17800; two row tiles a warp and an online softmax: no gain).
#pragma once
#include "bert.cuh"
#include "bert_block.cuh"

namespace fl {

constexpr int kBqAllHeads = 12, kBqHeads = 3, kBqCols = kBqHeads * kBertD;                       // heads, heads per unit at most, columns of q (k, v) per unit
constexpr int kBqStages = 4, kBqWarps = 12, kBqThreads = 64 + 32 * kBqWarps;
constexpr uint32_t kBqPart = kBqCols / 2 * 128, kBqStage = 2 * kBqPart;                          // per CTA: 2 x [48 rows][64 columns] of Wqkv
constexpr int kBqLd = 3 * kBqCols + 8;                                                           // a row of q|k|v in shared memory: 37 x 16 bytes, conflict-free ldmatrix
constexpr size_t kBqSmem = (size_t)kBbX + kBqStages * kBqStage + (size_t)128 * kBqLd * 2 + 3 * kBbH * 4 + 1024;
static_assert(kBqAllHeads * kBertD == kBbH && kBqSmem <= 232448, "");

struct BertQkvArgs {
    int b, t, spc;              // sentences, tokens of each, sentences per CTA: 128 / t
    const float* bias;          // [1152]
    float inv_scale;            // 1 / sqrt(d)
    uint16_t* ctx;              // [b t, 384]
    int* failed;                // set when a wait ran out
};

// two f32 at a time: x * y, x + y
__device__ __forceinline__ float2 mul_f32x2(float2 x, float2 y) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<const uint64_t&>(x)), "l"(reinterpret_cast<const uint64_t&>(y)));
    return d;
}
__device__ __forceinline__ float2 add_f32x2(float2 x, float2 y) {
    float2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<const uint64_t&>(x)), "l"(reinterpret_cast<const uint64_t&>(y)));
    return d;
}
// 16 query rows (m0 on) of a sentence's head: sq, sk, sv at the sentence's first row.  The rows of o take the place of the q rows that this warp alone reads.
// Every operation on a score is bert_attn_kernel's, in its order, so that a sentence's embedding is the same to the bit whichever kernel takes it: score /
// sqrt(d), minus the row's largest, e to that as 2^(x log2 e) (weights below 2^-126 are zero), a lane's sum a pair of neighbouring keys at a time.  (One fma
// in front of ex2 and the sums two columns at a time: 256 x 128 tokens 1080 us instead of 1107, but weights on other sides of bf16 roundings, 1.2e-3 in an embedding.  The products with 1 / sqrt(d) are
// __fmul_rn: a packed product in front of the packed sum comes out of the assembler as one fma.)
// LD: elements of a row.  KT: 16-key steps of the sentence's t tokens; rows behind it read as its last one, as queries nobody uses what they give, as keys their weight is zero.
template <int KT, int LD>
__device__ __forceinline__ void bq_attention(uint16_t* sq, const uint16_t* sk, const uint16_t* sv, int t, int m0, float inv_scale, uint16_t* ctx, int lane) {
    const int g = lane >> 2, tq = lane & 3;
    const float2 log2e = make_float2(1.4426950408889634f, 1.4426950408889634f);
    uint32_t qa[2][4];
    float2 s[2 * KT][2];
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) ldmatrix_x4(qa[ks], sq + min(m0 + (lane & 15), t - 1) * LD + ks * 16 + (lane >> 4) * 8);
    // two key tiles a step, the next step's keys requested before this one's products
    uint32_t kb[2][2][4];
    auto keys = [&](int i) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int r = (2 * i + u) * 8 + (lane & 7);
            ldmatrix_x4(kb[i & 1][u], sk + (i + 1 < KT ? r : min(r, t - 1)) * LD + (lane >> 3) * 8);
        }
    };
    keys(0);
#pragma unroll
    for (int i = 0; i < KT; ++i) {
        if (i + 1 < KT) keys(i + 1);
        float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int ks = 0; ks < 2; ++ks)
#pragma unroll
            for (int u = 0; u < 2; ++u) mma_bf16_16816(c[u], qa[ks], kb[i & 1][u][2 * ks], kb[i & 1][u][2 * ks + 1]);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int nt = 2 * i + u;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                s[nt][h] = make_float2(__fmul_rn(c[u][2 * h], inv_scale), __fmul_rn(c[u][2 * h + 1], inv_scale));
                if (i + 1 == KT) {
                    if (nt * 8 + tq * 2 >= t) s[nt][h].x = -INFINITY;
                    if (nt * 8 + tq * 2 + 1 >= t) s[nt][h].y = -INFINITY;
                }
            }
        }
    }
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int nt = 0; nt < 2 * KT; ++nt)
#pragma unroll
        for (int h = 0; h < 2; ++h) mx[h] = fmaxf(fmaxf(mx[h], s[nt][h].x), s[nt][h].y);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xFFFFFFFFu, mx[h], 1));
        mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xFFFFFFFFu, mx[h], 2));
    }
    const float2 b0 = make_float2(-mx[0], -mx[0]), b1 = make_float2(-mx[1], -mx[1]);
    float sum[2] = {0.f, 0.f};
    float o[4][4];
#pragma unroll
    for (int dt = 0; dt < 4; ++dt) o[dt][0] = o[dt][1] = o[dt][2] = o[dt][3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < KT; ++ks) {
        uint32_t pa[4], vb[2][4];
        const int vr = ks * 16 + (lane & 15);
#pragma unroll
        for (int d = 0; d < 2; ++d) ldmatrix_x4_trans(vb[d], sv + (ks + 1 < KT ? vr : min(vr, t - 1)) * LD + d * 16 + (lane >> 4) * 8);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float2 x = mul_f32x2(add_f32x2(s[2 * ks + h][0], b0), log2e), y = mul_f32x2(add_f32x2(s[2 * ks + h][1], b1), log2e);
            x.x = ex2_approx(x.x); x.y = ex2_approx(x.y);
            y.x = ex2_approx(y.x); y.y = ex2_approx(y.y);
            sum[0] += x.x + x.y;
            sum[1] += y.x + y.y;
            pa[2 * h] = pack_bf16(x.x, x.y);
            pa[2 * h + 1] = pack_bf16(y.x, y.y);
        }
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            mma_bf16_16816(o[2 * d], pa, vb[d][0], vb[d][1]);
            mma_bf16_16816(o[2 * d + 1], pa, vb[d][2], vb[d][3]);
        }
    }
    float inv[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float l = sum[h];
        l += __shfl_xor_sync(0xFFFFFFFFu, l, 1);
        l += __shfl_xor_sync(0xFFFFFFFFu, l, 2);
        inv[h] = 1.f / l;
    }
    __syncwarp();
#pragma unroll
    for (int dt = 0; dt < 4; ++dt) {
        if (m0 + g < t) *reinterpret_cast<uint32_t*>(sq + (m0 + g) * LD + dt * 8 + tq * 2) = pack_bf16(o[dt][0] * inv[0], o[dt][1] * inv[0]);
        if (m0 + g + 8 < t) *reinterpret_cast<uint32_t*>(sq + (m0 + g + 8) * LD + dt * 8 + tq * 2) = pack_bf16(o[dt][2] * inv[1], o[dt][3] * inv[1]);
    }
    __syncwarp();
#pragma unroll
    for (int r = m0 + g; r < m0 + 16; r += 8)           // whole 64-byte pieces of the rows
        if (r < t) *reinterpret_cast<uint4*>(ctx + (size_t)r * kBbH + tq * 8) = *reinterpret_cast<const uint4*>(sq + r * LD + tq * 8);
}
// 32 columns on their way; tmem_arrived32: all that were requested are there
__device__ __forceinline__ void tmem_request32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_arrived32(uint32_t (&r)[32]) {
#pragma unroll
    for (int i = 0; i < 32; i += 16)
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]), "+r"(r[i + 4]), "+r"(r[i + 5]), "+r"(r[i + 6]), "+r"(r[i + 7]), "+r"(r[i + 8]),
                       "+r"(r[i + 9]), "+r"(r[i + 10]), "+r"(r[i + 11]), "+r"(r[i + 12]), "+r"(r[i + 13]), "+r"(r[i + 14]), "+r"(r[i + 15])
                     :
                     : "memory");
}

// Four heads, of `pieces` 16-row tiles each, as two units of two instead of three and one: the warps go round a unit's pieces in whole rounds.
// (37 / 46 x 65 tokens 373 -> 368, 381 -> 378 us; units of two throughout, three rounds instead of four for twelve heads: 300 x 67 1034 -> 1055.)
__host__ __device__ constexpr bool bq_halves(int pieces) {
    auto rounds = [](int n) { return (n + kBqWarps - 1) / kBqWarps; };
    return 2 * rounds(2 * pieces) < rounds(3 * pieces) + rounds(pieces);
}
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kBqThreads, 1)
bert_qkv_attn_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const BertQkvArgs g) {
    extern __shared__ uint8_t gsm_raw[];
    uint8_t* sX = gsm_raw + ((1024u - (smem_u32(gsm_raw) & 1023u)) & 1023u);
    uint8_t* sW = sX + kBbX;
    uint16_t* sQ = reinterpret_cast<uint16_t*>(sW + kBqStages * kBqStage);          // [128][kBqLd]: q | k | v of three heads
    float* sB = reinterpret_cast<float*>(sQ + 128 * kBqLd);                          // the biases (a few KB of L1 are left beside all this)
    __shared__ __align__(8) uint64_t w_full[kBqStages], w_empty[kBqStages], x_full[3], x_free, acc_full, acc_free;
    __shared__ uint32_t tmem_base_s;
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int cl = blockIdx.x >> 1, G = gridDim.x >> 1;
    const int groups = (g.b + g.spc - 1) / g.spc, heads = (groups + 1) / 2 * kBqAllHeads;      // of all pairs, in a row
    const int h0 = (int)((long long)heads * cl / G), h1 = (int)((long long)heads * (cl + 1) / G);
    // the unit that begins at a head: how many heads
    const bool halves = bq_halves(g.spc * ((g.t + 15) / 16));
    auto unit = [&](int h) {
        const int left = min(h1 - h, kBqAllHeads - h % kBqAllHeads);
        return left == 4 && halves ? 2 : min(kBqHeads, left);
    };

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kBqStages; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_empty[s], 1); }
        for (int k = 0; k < 3; ++k) mbar_init(&x_full[k], 1);
        mbar_init(&x_free, 1);
        mbar_init(&acc_full, 1);
        mbar_init(&acc_free, 2 * kBqWarps);
        mbar_fence_init();
        tma_prefetch_desc(&tmX); tma_prefetch_desc(&tmW);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {
            int st = 0;
            uint32_t ph = 1;
            // stage i of a unit: two k blocks of its heads' rows of q (i < 3), k, v (48 rows whatever the heads: the box's; what lies behind is not used)
            auto stage = [&](int h, int n, int i) {
                if (!ok || !(ok = pair_wait(&w_empty[st], ph))) return;
                if (rank == 0) mbar_expect_tx(&w_full[st], 2 * kBqStage);
                const uint32_t bar = mapa_u32(smem_u32(&w_full[st]), 0), sa = smem_u32(sW) + st * kBqStage;
                const int row = i / 3 * kBbH + h % kBqAllHeads * kBertD + (int)rank * n * (kBertD / 2);
#pragma unroll
                for (int k = 0; k < 2; ++k) tma_load_2d_pair(sa + k * kBqPart, &tmW, (i % 3 * 2 + k) * 64, row, bar);
                if (++st == kBqStages) { st = 0; ph ^= 1; }
            };
            int tiles = 0;
            for (int h = h0, n; ok && h < h1; h += n) {
                n = unit(h);
                int first = 0;
                if (h == h0) {                      // the first ring of weights does not wait for the kernels before
                    for (; first < kBqStages; ++first) stage(h, n, first);
                    pdl_wait();
                    asm volatile("fence.proxy.async;" ::: "memory");
                }
                if (h == h0 || h % kBqAllHeads == 0) {
                    if (tiles > 0 && !(ok = pair_wait(&x_free, (tiles - 1) & 1))) break;
                    const int row = (h / kBqAllHeads * 2 + (int)rank) * g.spc * g.t;
                    for (int k = 0; k < kBbKb; ++k) {       // (the products start with the first two blocks)
                        if (rank == 0 && k % 2 == 0) mbar_expect_tx(&x_full[k / 2], 4 * 16384);
                        tma_load_2d_pair(smem_u32(sX) + k * 16384, &tmX, k * 64, row, mapa_u32(smem_u32(&x_full[k / 2]), 0));
                    }
                    ++tiles;
                }
                for (; first < 9; ++first) stage(h, n, first);
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {             // (the whole warp, see uniform_warp; a wait that ran out ends the waiting, not the walk)
            const uint64_t dX = umma_smem_desc_sw128(sX), dW = umma_smem_desc_sw128(sW);
            uint32_t c = 0;                         // stages so far
            int tiles = 0, units = 0;
            auto wait = [&](uint64_t* bar, uint32_t parity) {
                if (ok) ok = pair_wait(bar, parity);
                __syncwarp();
                tc_fence_after();
            };
            for (int h = h0, n; h < h1; h += n, ++units) {
                n = unit(h);
                const uint32_t idesc = umma_idesc_bf16(256, n * kBertD);
                wait(&acc_free, (units & 1) ^ 1);
                const bool fresh = h == h0 || h % kBqAllHeads == 0;
#pragma unroll 1
                for (int i = 0; i < 9; ++i, ++c) {
                    if (fresh && i < 3) wait(&x_full[i], tiles & 1);
                    const uint32_t st = c % kBqStages, col = i / 3 * kBqCols;
                    const uint64_t a = dX + (uint64_t)(i % 3 * 2048), b = dW + (uint64_t)(st * (kBqStage >> 4));
                    wait(&w_full[st], (c / kBqStages) & 1);
#pragma unroll
                    for (int k = 0; k < 2; ++k)
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            umma_bf16_pair_warp(tmem + col, a + (uint64_t)(k * 1024 + 2 * q), b + (uint64_t)(k * (kBqPart >> 4) + 2 * q), idesc, (k | q) ? 1u : (uint32_t)(i % 3 != 0));
                    umma_commit_pair_warp(&w_empty[st]);
                }
                umma_commit_pair_warp(&acc_full);
                tiles += fresh;
                if (h + n < h1 && (h + n) % kBqAllHeads == 0) umma_commit_pair_warp(&x_free);
            }
        }
    } else {
        const int q = warp & 3, aw = warp - 2, part = aw >> 2, lrow = q * 32 + lane;         // row of the CTA; q, k or v
        static_assert(kBqWarps == 12, "a warp per 32 rows of q, k and v");
        const uint32_t lane_at = (uint32_t)(q * 32) << 16;
        const int mts = (g.t + 15) / 16;
        auto esync = [] { asm volatile("bar.sync 1, %0;" ::"n"(32 * kBqWarps) : "memory"); };
        for (int i = threadIdx.x - 64; i < 3 * kBbH; i += 32 * kBqWarps) sB[i] = g.bias[i];
        esync();
        pdl_wait();
        for (int hd = h0, n, units = 0; hd < h1; hd += n, ++units) {             // (to the end even behind a wait that ran out: the warps meet at barriers)
            n = unit(hd);
            if (ok) ok = __all_sync(0xFFFFFFFFu, pair_wait(&acc_full, units & 1));
            tc_fence_after();
            const int head0 = hd % kBqAllHeads;
            uint8_t* dst = reinterpret_cast<uint8_t*>(sQ + lrow * kBqLd + part * kBqCols);
            const float* bias = sB + part * kBbH + head0 * kBertD;
            uint32_t v[kBqHeads][32];
#pragma unroll
            for (int c = 0; c < kBqHeads; ++c) tmem_request32(tmem + lane_at + (uint32_t)(part * kBqCols + c * 32), v[c]);
#pragma unroll
            for (int c = 0; c < kBqHeads; ++c) tmem_arrived32(v[c]);
#pragma unroll
            for (int c = 0; c < kBqHeads; ++c) {
                if (c >= n) continue;           // (a unit of fewer heads)
#pragma unroll
                for (int j = 0; j < 32; j += 8) {
                    const float4 x = *reinterpret_cast<const float4*>(bias + c * 32 + j), y = *reinterpret_cast<const float4*>(bias + c * 32 + j + 4);
                    const uint32_t* z = v[c] + j;
                    *reinterpret_cast<uint4*>(dst + (c * 32 + j) * 2) =
                        make_uint4(pack_bf16x2(__uint_as_float(z[0]) + x.x, __uint_as_float(z[1]) + x.y), pack_bf16x2(__uint_as_float(z[2]) + x.z, __uint_as_float(z[3]) + x.w),
                                   pack_bf16x2(__uint_as_float(z[4]) + y.x, __uint_as_float(z[5]) + y.y), pack_bf16x2(__uint_as_float(z[6]) + y.z, __uint_as_float(z[7]) + y.w));
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster_relaxed(mapa_u32(smem_u32(&acc_free), 0));      // (loaded into registers: no memory changes hands)
            esync();                                // q, k, v of three heads are there
            const int grp = hd / kBqAllHeads * 2 + (int)rank, ns = min(g.spc, g.b - grp * g.spc);
            uint16_t* ctx = g.ctx + (size_t)grp * g.spc * g.t * kBbH + head0 * kBertD;
            // (a rejected wait leaves nothing to store)
            for (int it = aw; ok && it < ns * mts * n; it += kBqWarps) {
                const int h = it % n, s = it / n / mts, m0 = it / n % mts * 16;
                uint16_t *row = sQ + s * g.t * kBqLd + h * kBertD, *to = ctx + (size_t)s * g.t * kBbH + h * kBertD;
                auto go = [&](auto kt) { bq_attention<decltype(kt)::value, kBqLd>(row, row + kBqCols, row + 2 * kBqCols, g.t, m0, g.inv_scale, to, lane); };
                switch (mts) {
                    case 1: go(std::integral_constant<int, 1>{}); break;
                    case 2: go(std::integral_constant<int, 2>{}); break;
                    case 3: go(std::integral_constant<int, 3>{}); break;
                    case 4: go(std::integral_constant<int, 4>{}); break;
                    case 5: go(std::integral_constant<int, 5>{}); break;
                    case 6: go(std::integral_constant<int, 6>{}); break;
                    case 7: go(std::integral_constant<int, 7>{}); break;
                    default: go(std::integral_constant<int, 8>{});
                }
            }
            esync();                                // the next unit's take their place
        }
    }
    if (!ok) {                   // a wait ran out: report it, leave the copies in flight time to land, go on to the end
        if (lane == 0 && g.failed != nullptr) *g.failed = 1;
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // the first CTA's products read the other one's shared memory, the other one's warps arrive on the first one's barriers
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

}  // namespace fl
