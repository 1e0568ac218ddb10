// Grouped-query attention of a layered decoder over a portion of a prompt, on the 5th-gen tensor cores in one kernel.
//
// One block owns 128 query rows of one head and walks the 64-key pages its rows can see; the structure is attn_prefill_tc_kernel's:
//   warp 0, 10   producers: K pages and pages of V^T by 2-D TMA (128-byte swizzle), gathered from the cache by ly_gqa_pages_kernel
//   warp 1       allocates TMEM and issues S = Q K^T (q = hi + lo) ahead of, and O += P V (P = hi + lo) behind the softmax
//   warps 2 - 9  softmax: thread == query row x half a page; score cap, masks, running maximum that moves only by more than 2^tau
// What this design adds: any position the portion starts at, windows with kept first keys, chunk masks, the score cap, sinks in the
// denominator, the output gate, and heads of up to 128 channels that need not be 64 or 128 (padded with zeros).
// Before, each group of heads took five launches per 1024 rows (gather, queries, scores GEMM, softmax, values GEMM) and the scores and
// probabilities of every row travelled through HBM: 8 bytes per score written and read once.
// Bound: the softmax warps (one exponential, and with a cap one tanh, per score) beside 2 x 2 MMA passes.
// Measured: 2048 tokens, 32 query heads of 128 on 8 key heads, score cap and sink: 82 launches of 1410 us -> 2 launches of 244 us; 333 tokens,
// 16 on 4 heads, two layers: 380 -> 75 us.
#pragma once
#include "gemm_tc.cuh"
#include "layered_ops.cuh"

namespace fl {

constexpr int kGtQ = 128, kGtThreads = 352, kGtKStages = 3, kGtSBufs = 4;
__host__ __device__ constexpr int gqa_tc_vstages(int dv) { return dv == 128 ? 2 : 3; }
__host__ __device__ constexpr size_t gqa_tc_smem(int dk, int dv) {
    return (size_t)2 * (dk / 64) * 16384 + 65536 + (size_t)kGtKStages * dk * 128 + (size_t)gqa_tc_vstages(dv) * dv * 128 + 1024;
}

// mbar_wait that gives up after about two seconds.  A block whose wait ran out stops at one page for all its softmax threads, lets its own copies
// and products land, frees its TMEM and leaves a mark that the host reads behind the step (GqaTcArgs.failed): the call then returns an error.
__device__ __forceinline__ bool gt_try(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ bool gt_wait(uint64_t* bar, uint32_t parity) {
    if (gt_try(bar, parity)) return true;
    const long long t0 = clock64();
    do {
        if (gt_try(bar, parity)) return true;
    } while (clock64() - t0 < (1ll << 32));
    return false;
}

// Where the gathered pages lie: buffer page b holds the cache's page b for b < first, else page base + (b - first).
struct GqaPages {
    int first, base, pages;         // kept first pages in front / first page of the contiguous part / pages in all
    __host__ __device__ int at(int page) const { return page < base ? page : first + page - base; }
    __host__ __device__ int page(int b) const { return b < first ? b : base + b - first; }
};
struct GqaTcArgs {
    const float* proj; int ldp, off_q;      // prepared queries
    int row0, Ts, pos0;                     // the portion: first row of the step, rows, position of the first
    int H, G, D, Dv;
    GqaPages pg;
    int window, keep_first, chunk;
    float scale, softcap;
    int sink; const float* sinkv;
    uint16_t *ohi, *olo; int ldo;
    OutGate gate;
    float tau;
    int* failed;                            // pinned host memory: set by a block that gave up
};

// kc [G][64 pages][DK] and vt [G][DV][64 pages] of the pages a portion reads; keys at or behind `end` and channels behind D / Dv are zero.
// grid (pages, G)
template <int DK, int DV>
static __global__ void __launch_bounds__(256) ly_gqa_pages_kernel(const uint16_t* __restrict__ pool, const int* __restrict__ page_row, GqaPages pg, int end, KvLayout kv, int D,
                                                                  int Dv, uint16_t* __restrict__ kc, uint16_t* __restrict__ vt) {
    pdl_chain();
    __shared__ uint16_t tile[DV][kKvPage + 2];
    const int b = blockIdx.x, g = blockIdx.y, page = pg.page(b), nkp = pg.pages * kKvPage, tid = threadIdx.x;
    const int keys = min(kKvPage, end - page * kKvPage);
    const uint16_t* src = pool + (size_t)page_row[page] * kKvPage * kv.E;
    uint16_t* k = kc + ((size_t)g * nkp + (size_t)b * kKvPage) * DK;
    const int ko = g * kv.ks, vo = kv.vo + g * kv.vs;
    if (((kv.E | ko | D) & 7) == 0) {
        for (int i = tid; i < kKvPage * (DK / 8); i += 256) {
            const int t = i / (DK / 8), c = i % (DK / 8) * 8;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (t < keys && c < D) v = *reinterpret_cast<const uint4*>(src + (size_t)t * kv.E + ko + c);
            *reinterpret_cast<uint4*>(k + (size_t)t * DK + c) = v;
        }
    } else {
        for (int i = tid; i < kKvPage * DK; i += 256) {
            const int t = i / DK, c = i % DK;
            k[i] = (t < keys && c < D) ? src[(size_t)t * kv.E + ko + c] : (uint16_t)0;
        }
    }
    for (int i = tid; i < kKvPage * DV; i += 256) {
        const int t = i / DV, c = i % DV;
        const int ch = c < Dv ? (c + kv.roll < Dv ? c + kv.roll : c + kv.roll - Dv) : c;
        tile[ch][t] = (t < keys && c < Dv) ? src[(size_t)t * kv.E + vo + c] : (uint16_t)0;
    }
    __syncthreads();
    uint16_t* v = vt + (size_t)g * DV * nkp + (size_t)b * kKvPage;
    for (int i = tid; i < DV * (kKvPage / 2); i += 256) {
        const int c = i / (kKvPage / 2), t = i % (kKvPage / 2) * 2;
        *reinterpret_cast<uint32_t*>(v + (size_t)c * nkp + t) = (uint32_t)tile[c][t] | (uint32_t)tile[c][t + 1] << 16;
    }
}

template <int DK, int DV>
static __global__ void __launch_bounds__(kGtThreads, 1) ly_gqa_tc_kernel(const __grid_constant__ CUtensorMap tmk, const __grid_constant__ CUtensorMap tmv, const GqaTcArgs a) {
    constexpr int HALF = DK / 64, NK = kGtKStages, NV = gqa_tc_vstages(DV), NS = kGtSBufs;
    constexpr uint32_t kQBytes = HALF * 16384, kPOff = 2 * kQBytes, kKTile = DK * 128, kVTile = DV * 128, kKOff = kPOff + 65536, kVOff = kKOff + NK * kKTile;
    extern __shared__ __align__(1024) uint8_t gtsm_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gtsm_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t k_full[NK], k_empty[NK], v_full[NV], v_empty[NV], s_full[NS], s_free[NS], p_ready[2], p_free[2], q_ready, drained;
    __shared__ int gave_up[2];
    __shared__ uint32_t s_tmem;
    __shared__ float xmax[2][2][kGtQ], xsum[2][kGtQ];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int qt = gridDim.x - 1 - blockIdx.x, head = blockIdx.y, grp = head / (a.H / a.G);       // latest (heaviest) query tiles first
    const int q0 = qt * kGtQ, p_lo = a.pos0 + q0, p_hi = a.pos0 + min(a.Ts, q0 + kGtQ) - 1;       // positions of the tile's rows
    // pages: the kept first ones in front of the contiguous range that the rows' windows and chunks reach
    const int lo = max(a.window > 0 ? max(p_lo - a.window + 1, 0) : 0, a.chunk > 0 ? p_lo / a.chunk * a.chunk : 0);
    const int t0 = lo / kKvPage, nf = (a.window > 0 && a.keep_first > 0) ? min((a.keep_first + kKvPage - 1) / kKvPage, t0) : 0;
    const int np = nf + p_hi / kKvPage - t0 + 1;
    auto page_of = [&](int j) { return j < nf ? j : t0 + j - nf; };

    if (tid == 0) {
        for (int i = 0; i < NK; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
        for (int i = 0; i < NV; ++i) { mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
        for (int i = 0; i < NS; ++i) { mbar_init(&s_full[i], 1); mbar_init(&s_free[i], 8); }
        for (int i = 0; i < 2; ++i) { mbar_init(&p_ready[i], 8); mbar_init(&p_free[i], 1); }
        mbar_init(&q_ready, 8);
        mbar_init(&drained, 1);
        gave_up[0] = gave_up[1] = 0;
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(&s_tmem, 512);
    pdl_launch_dependents();
    pdl_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem, sm_s = smem_u32(sm), tO = tmem + NS * 64;
    const int nkp = a.pg.pages * kKvPage;

    if (warp == 0) {
        if (lane == 0) {
            asm volatile("fence.proxy.async;" ::: "memory");
            int j = 0;
            for (; j < np; ++j) {
                const int st = j % NK, row = grp * nkp + a.pg.at(page_of(j)) * kKvPage;
                if (!gt_wait(&k_empty[st], ((j / NK) & 1) ^ 1)) break;
                mbar_expect_tx(&k_full[st], kKTile);
#pragma unroll
                for (int hf = 0; hf < HALF; ++hf) tma_load_2d(sm + kKOff + st * kKTile + hf * 8192, &tmk, hf * 64, row, &k_full[st]);
            }
            if (j < np) {
                for (int i = j > NK ? j - NK : 0; i < j; ++i) gt_wait(&k_full[i % NK], (i / NK) & 1);
                *a.failed = 1;
            }
        }
    } else if (warp == 10) {
        if (lane == 0) {
            asm volatile("fence.proxy.async;" ::: "memory");
            int j = 0;
            for (; j < np; ++j) {
                const int st = j % NV;
                if (!gt_wait(&v_empty[st], ((j / NV) & 1) ^ 1)) break;
                mbar_expect_tx(&v_full[st], kVTile);
                tma_load_2d(sm + kVOff + st * kVTile, &tmv, a.pg.at(page_of(j)) * kKvPage, grp * DV, &v_full[st]);
            }
            if (j < np) {
                for (int i = j > NV ? j - NV : 0; i < j; ++i) gt_wait(&v_full[i % NV], (i / NV) & 1);
                *a.failed = 1;
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc_s = umma_idesc_bf16(128, 64), idesc_o = umma_idesc_bf16(128, DV);
            int qi = 0, pi = 0;
            const bool q_ok = gt_wait(&q_ready, 0);
            tc_fence_after();
            // whichever is ready next: neither product waits for the other
            for (uint32_t spin = 0; q_ok && pi < np && spin < (1u << 26); ++spin) {
                if (pi < qi && mbar_test(&p_ready[pi & 1], (pi >> 1) & 1) && mbar_test(&v_full[pi % NV], (pi / NV) & 1)) {
                    const int b = pi & 1;
                    tc_fence_after();
                    const uint64_t vdesc = umma_smem_desc_sw128(sm + kVOff + (pi % NV) * kVTile);
#pragma unroll
                    for (int hl = 0; hl < 2; ++hl) {
                        const uint64_t pdesc = umma_smem_desc_sw128(sm + kPOff + (b * 2 + hl) * 16384);
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) umma_bf16(tO, pdesc + 2 * kk, vdesc + 2 * kk, idesc_o, (pi > 0 || hl > 0 || kk > 0) ? 1u : 0u);
                    }
                    umma_commit(&v_empty[pi % NV]);
                    umma_commit(&p_free[b]);
                    ++pi;
                    spin = 0;
                } else if (qi < np && mbar_test(&k_full[qi % NK], (qi / NK) & 1) && mbar_test(&s_free[qi % NS], ((qi / NS) & 1) ^ 1)) {
                    const int st = qi % NK, sb = qi % NS;
                    tc_fence_after();
                    const uint32_t tS = tmem + sb * 64;
#pragma unroll
                    for (int hl = 0; hl < 2; ++hl)
#pragma unroll
                        for (int hf = 0; hf < HALF; ++hf) {
                            const uint64_t qdesc = umma_smem_desc_sw128(sm + hl * kQBytes + hf * 16384);
                            const uint64_t kdesc = umma_smem_desc_sw128(sm + kKOff + st * kKTile + hf * 8192);
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk) umma_bf16(tS, qdesc + 2 * kk, kdesc + 2 * kk, idesc_s, (hl > 0 || hf > 0 || kk > 0) ? 1u : 0u);
                        }
                    umma_commit(&s_full[sb]);
                    umma_commit(&k_empty[st]);
                    ++qi;
                    spin = 0;
                }
            }
            if (pi < np) {
                umma_commit(&drained);
                gt_wait(&drained, 0);
                *a.failed = 1;
            }
        }
    } else {
        const int half = (warp - 2) >> 2, quarter = warp & 3, r = quarter * 32 + lane;
        const int lrow = min(q0 + r, a.Ts - 1), irow = a.pos0 + lrow;          // rows past the portion are clamped: computed, never stored
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        auto gsync = [] { asm volatile("bar.sync 2, 256;" ::: "memory"); };
        {   // q row times the score scale -> hi | lo halves, swizzled operand layout.  (Scaled here and not with the scores: a masked score is
            // -inf, which a scale of zero or below would turn into NaN or +inf, and the maximum would be that of the unscaled scores.)
            const float* qsrc = a.proj + (size_t)(a.row0 + lrow) * a.ldp + a.off_q + (size_t)head * a.D;
#pragma unroll
            for (int cc = 0; cc < DK / 16; ++cc) {
                const int c = half * (DK / 16) + cc;
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
                if (c * 8 < a.D) { x = *reinterpret_cast<const float4*>(qsrc + c * 8); y = *reinterpret_cast<const float4*>(qsrc + c * 8 + 4); }
                x.x *= a.scale; x.y *= a.scale; x.z *= a.scale; x.w *= a.scale;
                y.x *= a.scale; y.y *= a.scale; y.z *= a.scale; y.w *= a.scale;
                uint4 h, l;
                h.x = pack_bf16x2(x.x, x.y); h.y = pack_bf16x2(x.z, x.w); h.z = pack_bf16x2(y.x, y.y); h.w = pack_bf16x2(y.z, y.w);
                l.x = pack_bf16x2(x.x - bf16lo(h.x), x.y - bf16hi(h.x)); l.y = pack_bf16x2(x.z - bf16lo(h.y), x.w - bf16hi(h.y));
                l.z = pack_bf16x2(y.x - bf16lo(h.z), y.y - bf16hi(h.z)); l.w = pack_bf16x2(y.z - bf16lo(h.w), y.w - bf16hi(h.w));
                const uint32_t off = (uint32_t)(c >> 3) * 16384u + (uint32_t)r * 128u + (uint32_t)(((c & 7) ^ (r & 7)) << 4);
                sts128(sm_s + off, h);
                sts128(sm_s + kQBytes + off, l);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&q_ready);
        }
        constexpr float kLog2e = 1.4426950408889634f;
        const bool cap = a.softcap > 0.f;
        const float in_cap = cap ? 1.f / a.softcap : 0.f;
        const int w_lo = a.window > 0 ? irow - a.window + 1 : 0, c_lo = a.chunk > 0 ? irow / a.chunk * a.chunk : 0;
        float m = -INFINITY, l = 0.f;
        bool ok = true;
        for (int j = 0; j < np; ++j) {
            const int b = j & 1, sb = j % NS, key0 = page_of(j) * kKvPage + half * 32;
            ok &= gt_wait(&s_full[sb], (j / NS) & 1);
            tc_fence_after();
            float sc[32];
            {
                uint32_t r0[32];
                tmem_ld32(tmem + lane_addr + sb * 64 + half * 32, r0);
#pragma unroll
                for (int e = 0; e < 32; ++e) sc[e] = __uint_as_float(r0[e]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_free[sb]);
            if (cap) {
#pragma unroll
                for (int e = 0; e < 32; ++e) sc[e] = a.softcap * tanhf(sc[e] * in_cap);
            }
            float mx = -INFINITY;
            if (key0 + 31 <= p_lo && (a.window <= 0 || key0 > p_hi - a.window) && (a.chunk <= 0 || key0 >= p_hi / a.chunk * a.chunk)) {      // all keys visible to all rows
#pragma unroll
                for (int e = 0; e < 32; ++e) mx = fmaxf(mx, sc[e]);
            } else {
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    const int key = key0 + e;
                    sc[e] = (key <= irow && key >= c_lo && (key >= w_lo || key < a.keep_first)) ? sc[e] : -INFINITY;
                    mx = fmaxf(mx, sc[e]);
                }
            }
            xmax[b][half][r] = mx;
            if (!ok) gave_up[b] = 1;
            gsync();
            if (gave_up[b]) { ok = false; break; }       // one decision for the 256 threads (this page's word is next written behind the next page's barrier)
            mx = fmaxf(mx, xmax[b][half ^ 1][r]) * kLog2e;           // offsets and exponents in the exp2 domain
            // the offset m follows the maximum lazily (see attn_prefill_tc_kernel)
            const bool bump = mx > m + a.tau;
            const float mn = bump ? mx : m;
            const float mu = mn == -INFINITY ? 0.f : mn;
            const float alpha = bump ? ex2_approx(m - mu) : 1.f;
            m = mn;
            float ps = 0.f;
#pragma unroll
            for (int e = 0; e < 32; ++e) {
                sc[e] = ex2_approx(fmaf(sc[e], kLog2e, -mu));
                ps += sc[e];
            }
            l = l * alpha + ps;
            if (j > 0 && __any_sync(0xFFFFFFFFu, bump)) {
                ok &= gt_wait(&p_free[b ^ 1], ((j - 1) >> 1) & 1);      // the P.V before has completed (which barrier: see attn_prefill_tc_kernel)
                tc_fence_after();
#pragma unroll 1
                for (int c4 = 0; c4 < DV / 64; ++c4) {
                    uint32_t o[32];
                    tmem_ld32(tO + lane_addr + half * (DV / 2) + c4 * 32, o);
#pragma unroll
                    for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
                    tmem_st32(tO + lane_addr + half * (DV / 2) + c4 * 32, o);
                }
            }
            ok &= gt_wait(&p_free[b], ((j >> 1) & 1) ^ 1);
            const uint32_t ph = sm_s + kPOff + (b * 2) * 16384 + (uint32_t)r * 128u;
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                uint4 h, lo4;
                h.x = pack_bf16x2(sc[8 * cc], sc[8 * cc + 1]); h.y = pack_bf16x2(sc[8 * cc + 2], sc[8 * cc + 3]);
                h.z = pack_bf16x2(sc[8 * cc + 4], sc[8 * cc + 5]); h.w = pack_bf16x2(sc[8 * cc + 6], sc[8 * cc + 7]);
                lo4.x = pack_bf16x2(sc[8 * cc] - bf16lo(h.x), sc[8 * cc + 1] - bf16hi(h.x));
                lo4.y = pack_bf16x2(sc[8 * cc + 2] - bf16lo(h.y), sc[8 * cc + 3] - bf16hi(h.y));
                lo4.z = pack_bf16x2(sc[8 * cc + 4] - bf16lo(h.z), sc[8 * cc + 5] - bf16hi(h.z));
                lo4.w = pack_bf16x2(sc[8 * cc + 6] - bf16lo(h.w), sc[8 * cc + 7] - bf16hi(h.w));
                const uint32_t off = (uint32_t)(((half * 4 + cc) ^ (r & 7)) << 4);
                sts128(ph + off, h);
                sts128(ph + 16384 + off, lo4);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[b]);
        }
        xsum[half][r] = l;
        gsync();
        float sum = l + xsum[half ^ 1][r];
        if (a.sink) sum += ex2_approx(fmaf(a.sinkv ? a.sinkv[head] : 0.f, kLog2e, -m));
        ok = ok && gt_wait(&p_free[(np - 1) & 1], ((np - 1) >> 1) & 1);      // the last P.V, and with it all before
        if (!ok) *a.failed = 1;
        tc_fence_after();
        const float inv = ok ? 1.f / sum : __int_as_float(0x7FC00000);
        const int row = a.row0 + lrow;
        const size_t obase = (size_t)row * a.ldo + (size_t)head * a.Dv;
#pragma unroll 1
        for (int c4 = 0; c4 < DV / 64; ++c4) {
            uint32_t o[32];
            const int col = half * (DV / 2) + c4 * 32;
            tmem_ld32(tO + lane_addr + col, o);
            if (q0 + r < a.Ts) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (col + c * 8 >= a.Dv) continue;
                    float v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        v[e] = __uint_as_float(o[8 * c + e]) * inv;
                        if (a.gate.g != nullptr) v[e] *= a.gate.at(row, head, col + c * 8 + e);
                    }
                    uint4 h, lo4;
                    h.x = pack_bf16x2(v[0], v[1]); h.y = pack_bf16x2(v[2], v[3]); h.z = pack_bf16x2(v[4], v[5]); h.w = pack_bf16x2(v[6], v[7]);
                    lo4.x = pack_bf16x2(v[0] - bf16lo(h.x), v[1] - bf16hi(h.x)); lo4.y = pack_bf16x2(v[2] - bf16lo(h.y), v[3] - bf16hi(h.y));
                    lo4.z = pack_bf16x2(v[4] - bf16lo(h.z), v[5] - bf16hi(h.z)); lo4.w = pack_bf16x2(v[6] - bf16lo(h.w), v[7] - bf16hi(h.w));
                    *reinterpret_cast<uint4*>(a.ohi + obase + col + c * 8) = h;
                    *reinterpret_cast<uint4*>(a.olo + obase + col + c * 8) = lo4;
                }
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

}  // namespace fl
