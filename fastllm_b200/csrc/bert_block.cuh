// What follows the attention in an encoder layer, in one kernel: x1 = LN(ctx Wo^T + bo + x), x' = LN(gelu(x1 W1^T + b1) W2^T + b2 + x1),
// for hidden 384 and intermediate 1536 (all-MiniLM-L6-v2), sm_100a only.  Restates models/embeddings.rs:185-190, 229-241 as the launch chain does
// (fl_bert.cu: same operands, same order of products, bf16 where the chain's tensors are bf16).
//
// Two CTAs of a cluster take 256 tokens (tcgen05.mma.cta_group::2, see gemm_pair.cuh): each holds its 128 rows of ctx, then x1, in shared memory
// and half of every weight tile.  The 1536-wide activations exist 128 columns at a time: S (128 TMEM columns) -> GELU -> shared memory -> O (384
// columns).  The tensor core alternates between the next columns' S and the last columns' O while the epilogue warps turn S into operands.
// As five launches every layer moved 100 to 200 MB of activations between kernels that each waited for HBM and for their epilogues' stores.  256 tokens
// take 51 us, of which the products are 22 (1.6 us per 128 intermediate columns, measured by themselves, 2.4 for the output projection).  The rest is the
// chain from S to the next operand that the products wait for (2.3 us per 128 columns instead of 1.6: load, GELU (1.0 us, the tanh unit), store, fence,
// release (0.25)), the two norms, and the first loads.  Beside 225 KB of shared memory an SM has a few KB of L1: the norms' parameters are brought into the
// operand's place, which is free while they run, and the residual comes 128 bytes of a row per eight lanes; read through L1 by every thread for its own
// row both took 9 us more (256 x 128 tokens: 112 -> 102 us a layer).  8 epilogue warps: 16 were no faster.
#pragma once
#include "gemm_pair.cuh"

namespace fl {

constexpr int kBbH = 384, kBbI = 1536, kBbKb = kBbH / 64, kBbChunks = kBbI / 128;
constexpr int kBbStages = 4;
// epilogue warps: kBbSlices per TMEM lane quarter, a slice of the columns each
constexpr int kBbSlices = 2, kBbEpiWarps = 4 * kBbSlices, kBbThreads = 64 + 32 * kBbEpiWarps;
constexpr uint32_t kBbStage = 24576;        // per CTA: 2 x [96 rows][64 columns] of Wo / W2, or 3 x [64 rows][64 columns] of W1
constexpr uint32_t kBbX = kBbKb * 16384, kBbHid = 2 * 16384;
constexpr size_t kBbSmem = (size_t)kBbX + kBbHid + kBbStages * kBbStage + 1024;

// [128 rows][64 columns] of shared memory to the tile at (c0, c1); rows past the tensor are left out
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* tmap, const void* src, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(tmap), "r"(c0), "r"(c1), "r"(smem_u32(src)) : "memory");
}

struct BertBlockArgs {
    int T;                      // tokens
    const uint16_t* x;          // [T, 384] the layer's input, replaced by its output (through tmX)
    const float *bo, *b1, *b2, *ln1w, *ln1b, *ln2w, *ln2b;
    float eps;
    int* failed;                // set when a wait ran out
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kBbThreads, 1)
bert_block_kernel(const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tm1,
                  const __grid_constant__ CUtensorMap tm2, const __grid_constant__ CUtensorMap tmX, const BertBlockArgs g) {
    extern __shared__ uint8_t gsm_raw[];
    uint8_t* sX = gsm_raw + ((1024u - (smem_u32(gsm_raw) & 1023u)) & 1023u);
    uint8_t* sH = sX + kBbX;
    uint8_t* sW = sH + kBbHid;
    __shared__ __align__(8) uint64_t w_full[kBbStages], w_empty[kBbStages], a_full[kBbKb / 2], x_ready, x_free, s_full, s_free, h_ready, h_free, o_full;
    __shared__ uint32_t tmem_base_s;
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int cl = blockIdx.x >> 1, G = gridDim.x >> 1, tiles = (g.T + 255) / 256;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kBbStages; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_empty[s], 1); }
        for (int k = 0; k < kBbKb / 2; ++k) mbar_init(&a_full[k], 1);
        mbar_init(&x_ready, 2 * kBbEpiWarps);
        mbar_init(&x_free, 1);
        mbar_init(&s_full, 1);
        mbar_init(&s_free, 2 * kBbEpiWarps);
        mbar_init(&h_ready, 2 * kBbEpiWarps);
        mbar_init(&h_free, 1);
        mbar_init(&o_full, 1);
        mbar_fence_init();
        tma_prefetch_desc(&tmC); tma_prefetch_desc(&tmO); tma_prefetch_desc(&tm1); tma_prefetch_desc(&tm2);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s, tS = tmem + kBbH;
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {
            int st = 0;
            uint32_t ph = 1;
            // one stage of weights: kind 0 Wo, 1 W1, 2 W2
            auto stage = [&](int kind, int chunk, int part) {
                if (!ok || !(ok = pair_wait(&w_empty[st], ph))) return;
                if (rank == 0) mbar_expect_tx(&w_full[st], 2 * kBbStage);
                const uint32_t bar = mapa_u32(smem_u32(&w_full[st]), 0), sa = smem_u32(sW) + st * kBbStage;
                if (kind == 1) {
#pragma unroll
                    for (int k = 0; k < 3; ++k) tma_load_2d_pair(sa + k * 8192, &tm1, (part * 3 + k) * 64, chunk * 128 + (int)rank * 64, bar);
                } else {
                    const CUtensorMap* tm = kind == 0 ? &tmO : &tm2;
                    const int c = kind == 0 ? part * 64 : chunk * 128 + part * 64;
#pragma unroll
                    for (int n = 0; n < 2; ++n) tma_load_2d_pair(sa + n * 12288, tm, c, n * 192 + (int)rank * 96, bar);
                }
                if (++st == kBbStages) { st = 0; ph ^= 1; }
            };
            int it = 0;
            for (int tile = cl; ok && tile < tiles; tile += G, ++it) {
                int first = 0;
                if (it == 0) {                      // the first ring of weights does not wait for the kernels before
                    for (; first < kBbStages; ++first) stage(0, 0, first);
                    pdl_wait();
                    asm volatile("fence.proxy.async;" ::: "memory");
                }
                if (it > 0 && !(ok = pair_wait(&x_free, (it - 1) & 1))) break;
                for (int k = 0; k < kBbKb; ++k) {       // (the products start with the first two blocks)
                    if (rank == 0 && k % 2 == 0) mbar_expect_tx(&a_full[k / 2], 4 * 16384);
                    tma_load_2d_pair(smem_u32(sX) + k * 16384, &tmC, k * 64, tile * 256 + (int)rank * 128, mapa_u32(smem_u32(&a_full[k / 2]), 0));
                }
                for (; first < kBbKb; ++first) stage(0, 0, first);
                for (int j = 0; j <= kBbChunks; ++j) {
                    if (j < kBbChunks) { stage(1, j, 0); stage(1, j, 1); }
                    if (j > 0) { stage(2, j - 1, 0); stage(2, j - 1, 1); }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {             // (the whole warp, see uniform_warp; a wait that ran out ends the waiting, not the walk)
            constexpr uint32_t id1 = umma_idesc_bf16(256, 128), id2 = umma_idesc_bf16(256, 192);
            const uint64_t dX = umma_smem_desc_sw128(sX), dH = umma_smem_desc_sw128(sH), dW = umma_smem_desc_sw128(sW);
            uint32_t n = 0;                         // stages so far
            auto wait = [&](uint64_t* bar, uint32_t parity) {
                if (ok) ok = pair_wait(bar, parity);
                __syncwarp();
                tc_fence_after();
            };
            // O (two halves of 192 columns) += A (one k block) . the next stage
            auto out = [&](uint64_t a, uint32_t acc) {
                const uint32_t st = n % kBbStages;
                const uint64_t b = dW + (uint64_t)(st * (kBbStage >> 4));
                wait(&w_full[st], (n / kBbStages) & 1);
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int q = 0; q < 4; ++q) umma_bf16_pair_warp(tmem + h * 192, a + 2 * q, b + (uint64_t)(h * (12288 >> 4) + 2 * q), id2, q ? 1u : acc);
                umma_commit_pair_warp(&w_empty[st]);
                ++n;
            };
            uint32_t chunk = 0;                     // over all tiles
            int it = 0;
            for (int tile = cl; tile < tiles; tile += G, ++it) {
                for (int k = 0; k < kBbKb; ++k) {
                    if (k % 2 == 0) wait(&a_full[k / 2], it & 1);
                    out(dX + (uint64_t)(k * 1024), k ? 1u : 0u);
                }
                umma_commit_pair_warp(&o_full);
                wait(&x_ready, it & 1);
                for (int j = 0; j <= kBbChunks; ++j) {
                    if (j < kBbChunks) {
                        wait(&s_free, ((chunk + j) & 1) ^ 1);
                        for (int p = 0; p < 2; ++p) {
                            const uint32_t st = n % kBbStages;
                            const uint64_t b = dW + (uint64_t)(st * (kBbStage >> 4)), a = dX + (uint64_t)(p * 3 * 1024);
                            wait(&w_full[st], (n / kBbStages) & 1);
#pragma unroll
                            for (int k = 0; k < 3; ++k)
#pragma unroll
                                for (int q = 0; q < 4; ++q)
                                    umma_bf16_pair_warp(tS, a + (uint64_t)(k * 1024 + 2 * q), b + (uint64_t)(k * (8192 >> 4) + 2 * q), id1, (k | q) ? 1u : (uint32_t)p);
                            umma_commit_pair_warp(&w_empty[st]);
                            ++n;
                        }
                        umma_commit_pair_warp(&s_full);
                    }
                    if (j > 0) {
                        wait(&h_ready, (chunk + j - 1) & 1);
                        for (int k = 0; k < 2; ++k) out(dH + (uint64_t)(k * 1024), (j > 1 || k) ? 1u : 0u);
                        umma_commit_pair_warp(&h_free);
                    }
                }
                umma_commit_pair_warp(&o_full);
                chunk += kBbChunks;
            }
        }
    } else {
        const int q = warp & 3, cs = (warp - 2) >> 2, lrow = q * 32 + lane;      // row of the CTA; slice of the columns
        constexpr int kOC = kBbH / kBbSlices, kSC = 128 / kBbSlices;              // columns of O and of S per warp
        const uint32_t lane_at = (uint32_t)(q * 32) << 16;
        // while the norms run the operand is not there yet, or done with: [slice][128] row sums; bias | weight | bias of the norm
        float2* part = reinterpret_cast<float2*>(sH);
        float* par = reinterpret_cast<float*>(sH + kBbSlices * 128 * 8);
        auto esync = [] { asm volatile("bar.sync 1, %0;" ::"n"(32 * kBbEpiWarps) : "memory"); };
        auto wait = [&](uint64_t* bar, uint32_t parity) { if (ok) ok = __all_sync(0xFFFFFFFFu, pair_wait(bar, parity)); tc_fence_after(); };
        // Arrives on the first CTA's barriers.  Operands in shared memory are released at the scope that the first CTA's products need: its own warps
        // within the CTA, the second one's warps at cluster scope, which takes 0.25 us that the products wait for.  s_free hands over no
        // memory -- what was loaded from S is in registers -- and needs no release (256 x 128 tokens, us: everything released at cluster scope by
        // both CTAs 1405, by the second one alone 1381, this 1348; one release behind a barrier of the eight warps 1355).
        auto arrive = [&](uint64_t* bar) {
            __syncwarp();
            if (lane != 0) return;
            if (rank == 0) mbar_arrive(bar); else mbar_arrive_cluster(mapa_u32(smem_u32(bar), 0));
        };
        auto free_s = [&] { __syncwarp(); if (lane == 0) mbar_arrive_cluster_relaxed(mapa_u32(smem_u32(&s_free), 0)); };
        // 16-byte chunk c of the row inside a tile of 64-column blocks
        auto at = [&](int c) { return (uint32_t)(c >> 3) * 16384u + (uint32_t)lrow * 128u + (uint32_t)(((c & 7) ^ (lrow & 7)) << 4); };
        // a norm's parameters, 288 pieces of 16 bytes: on their way, and into shared memory once the operand's place is free
        const int pi = threadIdx.x - 64;
        auto request = [&](const float* b, const float* w, const float* lb, float4 (&v)[2]) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int i = pi + k * 32 * kBbEpiWarps;
                if (i < 3 * (kBbH / 4)) v[k] = __ldg(reinterpret_cast<const float4*>(i < kBbH / 4 ? b : i < kBbH / 2 ? w : lb) + i % (kBbH / 4));
            }
        };
        auto put = [&](const float4 (&v)[2]) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int i = pi + k * 32 * kBbEpiWarps;
                if (i < 3 * (kBbH / 4)) reinterpret_cast<float4*>(par)[i] = v[k];
            }
        };
        // this thread's columns of O: + bias + the row of sX, kept in TMEM; -> mean and 1 / deviation of the row
        auto row_sums = [&](float& mean, float& inv) {
            float s = 0.f, s2 = 0.f;
#pragma unroll
            for (int i = 0; i < kOC / 32; ++i) {
                const int c = cs * kOC + 32 * i;
                uint32_t v[32], r[16];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint4 z = *reinterpret_cast<const uint4*>(sX + at(c / 8 + k));
                    r[4 * k] = z.x; r[4 * k + 1] = z.y; r[4 * k + 2] = z.z; r[4 * k + 3] = z.w;
                }
                tmem_ld32(tmem + lane_at + (uint32_t)c, v);
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    const float4 b = *reinterpret_cast<const float4*>(par + c + j);
                    const float y[4] = {__uint_as_float(v[j]) + b.x + bf16lo(r[j >> 1]), __uint_as_float(v[j + 1]) + b.y + bf16hi(r[j >> 1]),
                                        __uint_as_float(v[j + 2]) + b.z + bf16lo(r[(j >> 1) + 1]), __uint_as_float(v[j + 3]) + b.w + bf16hi(r[(j >> 1) + 1])};
#pragma unroll
                    for (int e = 0; e < 4; ++e) { v[j + e] = __float_as_uint(y[e]); s += y[e]; s2 = fmaf(y[e], y[e], s2); }
                }
                tmem_st32(tmem + lane_at + (uint32_t)c, v);
            }
            part[cs * 128 + lrow] = make_float2(s, s2);
            esync();
            s = s2 = 0.f;
#pragma unroll
            for (int k = 0; k < kBbSlices; ++k) { const float2 p = part[k * 128 + lrow]; s += p.x; s2 += p.y; }
            mean = s / (float)kBbH;
            inv = 1.f / sqrtf(s2 / (float)kBbH - mean * mean + g.eps);
        };
        // 32 normalised columns as bf16 pairs
        auto normed = [&](int c, float mean, float inv, uint32_t (&o)[16]) {
            uint32_t v[32];
            tmem_ld32(tmem + lane_at + (uint32_t)c, v);
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                const float4 w = *reinterpret_cast<const float4*>(par + kBbH + c + j), b = *reinterpret_cast<const float4*>(par + 2 * kBbH + c + j);
                o[j >> 1] = pack_bf16x2((__uint_as_float(v[j]) - mean) * inv * w.x + b.x, (__uint_as_float(v[j + 1]) - mean) * inv * w.y + b.y);
                o[(j >> 1) + 1] = pack_bf16x2((__uint_as_float(v[j + 2]) - mean) * inv * w.z + b.z, (__uint_as_float(v[j + 3]) - mean) * inv * w.w + b.w);
            }
        };
        if (pi < kBbI / 32) asm volatile("prefetch.global.L1 [%0];" ::"l"(g.b1 + 32 * pi));
        float4 p1[2], p2[2];
        request(g.bo, g.ln1w, g.ln1b, p1);
        pdl_wait();
        uint32_t chunk = 0, of = 0;
        for (int tile = cl; tile < tiles; tile += G) {            // (to the end even behind a wait that ran out: the warps meet at barriers)
            // The residual, on its way while the first products run: this warp's 32 rows and half of the columns, 128 bytes of a row per eight lanes (thread ==
            // row would take 32 lines a load), into the places of sX that the warp itself fills with x1.
            const int row0 = tile * 256 + (int)rank * 128;
            float mean, inv;
            uint4 res[kOC / 8];
            auto place = [&](int k, int& r) { r = q * 32 + k % 8 * 4 + (lane >> 3); return (uint32_t)(cs * (kOC / 64) + k / 8) * 16384u + (uint32_t)r * 128u + (uint32_t)(((lane & 7) ^ (r & 7)) << 4); };
#pragma unroll
            for (int k = 0; k < kOC / 8; ++k) {
                int r;
                place(k, r);
                res[k] = row0 + r < g.T ? *reinterpret_cast<const uint4*>(g.x + (size_t)(row0 + r) * kBbH + cs * kOC + k / 8 * 64 + (lane & 7) * 8) : make_uint4(0u, 0u, 0u, 0u);
            }
            put(p1);
            request(g.b2, g.ln2w, g.ln2b, p2);
            wait(&o_full, of++ & 1);
#pragma unroll
            for (int k = 0; k < kOC / 8; ++k) {
                int r;
                const uint32_t to = place(k, r);
                *reinterpret_cast<uint4*>(sX + to) = res[k];
            }
            esync();
            row_sums(mean, inv);
#pragma unroll 1
            for (int c = cs * kOC; c < cs * kOC + kOC; c += 32) {
                uint32_t o[16];
                normed(c, mean, inv, o);                          // (over the residual's values that this thread alone reads)
#pragma unroll
                for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(sX + at(c / 8 + k)) = make_uint4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_fence_before();
            arrive(&x_ready);
            for (int j = 0; j < kBbChunks; ++j, ++chunk) {
                uint32_t v[kSC], o[kSC / 2];
                wait(&s_full, chunk & 1);
#pragma unroll
                for (int h = 0; h < kSC; h += 32) tmem_ld32(tS + lane_at + (uint32_t)(cs * kSC + h), reinterpret_cast<uint32_t(&)[32]>(v[h]));
                tc_fence_before();
                free_s();
#pragma unroll
                for (int i = 0; i < kSC; i += 4) {
                    const float4 b = __ldg(reinterpret_cast<const float4*>(g.b1 + j * 128 + cs * kSC + i));
                    o[i >> 1] = pack_bf16x2(gelu_tanh_f(__uint_as_float(v[i]) + b.x), gelu_tanh_f(__uint_as_float(v[i + 1]) + b.y));
                    o[(i >> 1) + 1] = pack_bf16x2(gelu_tanh_f(__uint_as_float(v[i + 2]) + b.z), gelu_tanh_f(__uint_as_float(v[i + 3]) + b.w));
                }
                wait(&h_free, (chunk & 1) ^ 1);                   // the products with the columns before have read the buffer
#pragma unroll
                for (int k = 0; k < kSC / 8; ++k) *reinterpret_cast<uint4*>(sH + at(cs * (kSC / 8) + k)) = make_uint4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                arrive(&h_ready);
            }
            wait(&o_full, of++ & 1);
            put(p2);
            request(g.bo, g.ln1w, g.ln1b, p1);
            esync();
            row_sums(mean, inv);
#pragma unroll 1
            for (int c = cs * kOC; c < cs * kOC + kOC; c += 32) {
                uint32_t o[16];
                normed(c, mean, inv, o);          // (over the x1 values that this thread alone reads)
#pragma unroll
                for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(sX + at(c / 8 + k)) = make_uint4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_fence_before();
            esync();
            if (threadIdx.x == 64) {
                for (int k = 0; ok && row0 < g.T && k < kBbKb; ++k) tma_store_2d(&tmX, sX + k * 16384, k * 64, row0);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                mbar_arrive(&x_free);
            }
        }
        if (threadIdx.x == 64) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    if (!ok) {                   // a wait ran out: report it, leave the copies in flight time to land, go on to the end
        if (lane == 0 && g.failed != nullptr) *g.failed = 1;
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // the other CTA's products read this one's shared memory, its epilogue arrives on this one's barriers
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

}  // namespace fl
