// The encoder on few short sentences in ONE launch: a cluster of blocks per up to 64 tokens (whole sentences).
//
// A query of a dozen tokens through the launch chain is 44 kernels, each of them a few microseconds of latency around almost no work (the
// 24 GEMMs fill 2 to 8 of 148 SMs and walk K one 64-column block after the other).  Here the blocks of a cluster split every projection's
// output columns; phases are separated by the cluster's hardware barrier instead of a kernel boundary, and the weights of a phase -- which
// depend on nothing -- travel into shared memory while the cluster waits for the phase before.
//   per layer: a head's q, k, v and its attention in one block (12 of the 16) | x + W_o ctx | LayerNorm (every block for itself) ->
//   gelu(W_i x1) | x1 + W_o2 h | LayerNorm
// The results are the chain's, bit for bit: an output's products go into its f32 accumulator 16 columns of K at a time in ascending order, as
// tcgen05.mma takes them (mma.sync m16n8k16 sums the same 16 products to the same bits, in whatever order they stand inside the 16), so K is
// not split over warps; the attention is bert_qkv.cuh's, roundings and the order of every other sum are those of bert.cuh.
// Bound: latency -- 4 phases x 6 layers (cluster barrier, L2 round trips of activations, a chain of 24 to 96 MMAs of 35 clocks each).
// One sentence of 4 / 19 / 48 / 64 tokens, whole call: 243 / 254 / 268 / 277 us as 44 launches, 97 / 122 / 171 / 196 us here (121 / 161 / 224 / 270 with q, k, v
// by columns, a phase more, weights in 8-byte copies and a tile's rows loaded for every column tile).  A layer of 19 tokens: 31000 clocks, of which q, k, v
// 2500, attention 1300, the two halves of the feed-forward 2800 and 4700, the two norms 2300 each, barriers and round trips 1000 to 1500 a phase.
// (K in quarters over the warps is no faster, and its sums are not the chain's: 16-bit activations carry that to 3e-3 in the embedding.)
#pragma once
#include "bert_qkv.cuh"

namespace fl {

constexpr int kBsTokens = 64, kBsThreads = 256, kBsH = 384, kBsI = 1536, kBsHeads = 12;     // all-MiniLM-L6-v2's sizes
__host__ __device__ constexpr int bs_ld(int k) { return k + 8; }        // elements of an operand row in shared memory: an odd number of 16-byte pieces, for ldmatrix

// A layer's matrices once more, block by block as they lie in shared memory: a block's rows of W_qkv (its head's; zero without one), W_o, W_i, W_o2,
// each of one copy.  (A bulk copy per row of the matrices themselves: 216 copies a layer, 127 instead of 122 us for 19 tokens.)
constexpr int kBsCluster = 16;
constexpr int kBsQkvRows = 3 * kBertD, kBsORows = kBsH / kBsCluster, kBsIRows = kBsI / kBsCluster;
constexpr int kBsAtO = kBsQkvRows * bs_ld(kBsH), kBsAtI = kBsAtO + kBsORows * bs_ld(kBsH), kBsAtO2 = kBsAtI + kBsIRows * bs_ld(kBsH),
              kBsPack = kBsAtO2 + kBsORows * bs_ld(kBsI);                     // elements of a block
static_assert(kBsAtO % 8 == 0 && kBsAtI % 8 == 0 && kBsAtO2 % 8 == 0 && kBsPack % 8 == 0 && kBsH % 8 == 0 && kBsI % 8 == 0, "16-byte pieces");
// grid (pieces / 256, blocks of a cluster, layers); the layers' matrices lie `stride` elements apart.  16 bytes a thread: rows and their ends are whole pieces.
static __global__ void __launch_bounds__(256) bert_small_pack_kernel(const uint16_t* __restrict__ wqkv, const uint16_t* __restrict__ wo, const uint16_t* __restrict__ wi,
                                                                     const uint16_t* __restrict__ wo2, size_t stride, uint16_t* __restrict__ out) {
    const int rank = blockIdx.y, i = (blockIdx.x * 256 + threadIdx.x) * 8;
    if (i >= kBsPack) return;
    const int ld = i < kBsAtO2 ? bs_ld(kBsH) : bs_ld(kBsI), k = i < kBsAtO2 ? kBsH : kBsI;
    const int at = i < kBsAtO ? 0 : i < kBsAtI ? kBsAtO : i < kBsAtO2 ? kBsAtI : kBsAtO2, r = (i - at) / ld, c = (i - at) % ld;
    const uint16_t* src = nullptr;
    if (c < k) {
        if (i >= kBsAtO2) src = wo2 + (size_t)(rank * kBsORows + r) * kBsI;
        else if (i >= kBsAtI) src = wi + (size_t)(rank * kBsIRows + r) * kBsH;
        else if (i >= kBsAtO) src = wo + (size_t)(rank * kBsORows + r) * kBsH;
        else if (rank < kBsHeads) src = wqkv + (size_t)(r / kBertD * kBsH + rank * kBertD + r % kBertD) * kBsH;
    }
    const uint4 v = src != nullptr ? *reinterpret_cast<const uint4*>(src + blockIdx.z * stride + c) : make_uint4(0u, 0u, 0u, 0u);
    *reinterpret_cast<uint4*>(out + ((size_t)blockIdx.z * kBsCluster + rank) * kBsPack + i) = v;
}

struct BertSmallLayer {
    const uint16_t* pack;                   // [kBsCluster][kBsPack]
    const float *bqkv, *bo, *bi, *bo2, *ln1w, *ln1b, *ln2w, *ln2b;
};
struct BertSmallArgs {
    const BertSmallLayer* layers;           // device
    const uint16_t *wemb, *pemb; const float *lnw, *lnb;
    const uint32_t *ids, *mask;             // [b t]; mask may be null
    int L, b, t, V, maxpos, spc;            // spc: sentences per cluster
    float eps, inv_scale;                   // inv_scale: 1 / sqrt(d)
    uint16_t *ctx, *h; float* pre;          // workspace rows as the launch chain has them
    int* failed;                            // set when a wait ran out
    float* out;
};
// Shared memory of a block, in bytes: a layer's vectors twice | x | W_o and the head's q, k, v, or W_o2 | W_qkv, W_i or the gathered rows of ctx or h
template <int MT, int CL>
struct BsSmem {
    static constexpr int NQ = 3 * kBertD / 8, NO = kBsH / 8 / CL, NI = kBsI / 8 / CL;        // column tiles per block: a head's q, k, v; of the two other widths
    static_assert(CL == kBsCluster && kBsHeads <= CL && NO * CL * 8 == kBsH && NI * CL * 8 == kBsI, "a head per block, whole tiles per block");
    static constexpr int NV = 4 * kBsH + (NQ + 2 * NO + NI) * 8;
    // h arrives in pieces of its columns, one multiplied while the next are on their way: all at once, or (rows that would not fit) two
    static constexpr int kHPiece = MT <= 3 ? kBsI / 4 : kBsI / 6, kPieces = kBsI / kHPiece, kHBufs = MT <= 2 ? kPieces : 2;
    static constexpr int kHBuf = MT * 16 * bs_ld(kHPiece), kQkvLd = bs_ld(3 * kBertD);          // elements
    static constexpr size_t max2(size_t a, size_t b) { return a > b ? a : b; }
    static constexpr size_t kX = (size_t)2 * NV * 4, kWo = kX + (size_t)MT * 16 * bs_ld(kBsH) * 2, kQkv = kWo + (size_t)NO * 8 * bs_ld(kBsH) * 2,
                            kR = kWo + (size_t)NO * 8 * bs_ld(kBsI) * 2;
    static constexpr size_t kBytes = kR + max2((size_t)(NQ > NI ? NQ : NI) * 8 * bs_ld(kBsH) * 2, max2((size_t)MT * 16 * bs_ld(kBsH) * 2, (size_t)kHBufs * kHBuf * 2));
    static_assert(kHPiece % 32 == 0 && kX % 16 == 0 && kQkv + (size_t)MT * 16 * kQkvLd * 2 <= kR && kBytes <= 232448 - 256, "");
};

__device__ __forceinline__ void bs_arrive() { __syncwarp(); asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void bs_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// columns [k0, k0 + KP) of the cluster's rows of an activation that the cluster wrote
template <int KP>
__device__ __forceinline__ void bs_bring_rows(uint16_t* dst, const uint16_t* src, int ld, int k0, int rows) {
    for (int i = threadIdx.x; i < rows * (KP / 8); i += kBsThreads) {
        const int r = i / (KP / 8), c = i % (KP / 8) * 8;
        cp_async16(dst + r * bs_ld(KP) + c, src + (size_t)r * ld + k0 + c);
    }
}
// One projection's NT x MT tiles of 8 columns x 16 rows: a warp has one row tile and every WR-th column tile, so that its rows are loaded once for all
// of them (a tile at a time shared memory was the bound: 9 loads of 512 bytes for 6 products).
template <int MT, int NT>
struct BsTiles {
    static constexpr int WR = 8 / (MT == 3 ? 4 : MT), IT = (NT + WR - 1) / WR;
    float acc[IT][4];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < IT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    }
    // += A [.., KP] . columns [k0, k0 + KP) of W
    template <int KP>
    __device__ __forceinline__ void add(const uint16_t* A, const uint16_t* W, int ldw, int k0, int warp, int lane) {
        const int rt = warp / WR, ct = warp % WR;
        if (rt >= MT || ct >= NT) return;
        const uint16_t* a = A + (rt * 16 + (lane & 15)) * bs_ld(KP) + (lane >> 4) * 8;
        const uint16_t* w = W + (ct * 8 + (lane & 7)) * ldw + k0 + (lane >> 3) * 8;
#pragma unroll 6
        for (int s = 0; s < KP / 32; ++s) {
            uint32_t x[2][4];
            ldmatrix_x4(x[0], a + s * 32);
            ldmatrix_x4(x[1], a + s * 32 + 16);
            uint32_t b[IT][4];
#pragma unroll
            for (int i = 0; i < IT; ++i)
                if (ct + WR * i < NT) ldmatrix_x4(b[i], w + i * WR * 8 * ldw + s * 32);
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < IT; ++i)
                    if (ct + WR * i < NT) mma_bf16_16816(acc[i], x[h], b[i][2 * h], b[i][2 * h + 1]);
        }
    }
    // out(row, column pair inside the block, sums)
    template <typename Fn>
    __device__ __forceinline__ void store(int rows, int warp, int lane, Fn&& out) const {
        const int rt = warp / WR, ct = warp % WR, r = rt * 16 + (lane >> 2);
#pragma unroll
        for (int i = 0; i < IT; ++i)
            if (rt < MT && ct + WR * i < NT) {
                const int c = (ct + WR * i) * 8 + (lane & 3) * 2;
                if (r < rows) out(r, c, make_float2(acc[i][0], acc[i][1]));
                if (r + 8 < rows) out(r + 8, c, make_float2(acc[i][2], acc[i][3]));
            }
    }
};

// LayerNorm of the rows of pre (f32, global, written by the whole cluster) into the x tile; a warp has four rows on their way at a time
// (w, b: shared memory)
__device__ __forceinline__ void bs_layernorm(const float* pre, int rows, const float* w, const float* b, float eps, uint16_t* sx, int warp, int lane) {
    constexpr int NW = kBsThreads / 32, U = 4;
    for (int r0 = warp; r0 < rows; r0 += NW * U) {
        float4 v[U][3];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int j = 0; j < 3; ++j)
                v[u][j] = r0 + u * NW < rows ? __ldcg(reinterpret_cast<const float4*>(pre + (size_t)(r0 + u * NW) * kBsH) + lane + 32 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
        float s[U], s2[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            s[u] = s2[u] = 0.f;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const float4 x = v[u][j];
                s[u] += (x.x + x.y) + (x.z + x.w);
                s2[u] = fmaf(x.x, x.x, s2[u]); s2[u] = fmaf(x.y, x.y, s2[u]); s2[u] = fmaf(x.z, x.z, s2[u]); s2[u] = fmaf(x.w, x.w, s2[u]);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)        // (warp_sum, the rows side by side)
#pragma unroll
            for (int u = 0; u < U; ++u) {
                s[u] += __shfl_xor_sync(0xFFFFFFFFu, s[u], o);
                s2[u] += __shfl_xor_sync(0xFFFFFFFFu, s2[u], o);
            }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int r = r0 + u * NW;
            if (r >= rows) break;
            const float mean = s[u] / (float)kBsH, inv = 1.f / sqrtf(s2[u] / (float)kBsH - mean * mean + eps);
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int c = lane + 32 * j;
                const float4 x = v[u][j], w4 = reinterpret_cast<const float4*>(w)[c], b4 = reinterpret_cast<const float4*>(b)[c];
                *reinterpret_cast<uint2*>(sx + r * bs_ld(kBsH) + 4 * c) =
                    make_uint2(pack_bf16x2((x.x - mean) * inv * w4.x + b4.x, (x.y - mean) * inv * w4.y + b4.y),
                               pack_bf16x2((x.z - mean) * inv * w4.z + b4.z, (x.w - mean) * inv * w4.w + b4.w));
            }
        }
    }
}

// MT: row tiles of 16 (the cluster's tokens, rounded up); CL: blocks per cluster.  grid clusters * CL.
template <int MT, int CL>
static __global__ void __launch_bounds__(kBsThreads, 1) bert_small_kernel(const BertSmallArgs a) {
    using M = BsSmem<MT, CL>;
    constexpr int NQ = M::NQ, NO = M::NO, NI = M::NI, LDX = bs_ld(kBsH);
    extern __shared__ __align__(16) uint8_t bs_smem[];
    float* sv = reinterpret_cast<float*>(bs_smem);                          // a layer's vectors, two layers
    uint16_t* sx = reinterpret_cast<uint16_t*>(bs_smem + M::kX);            // x
    uint16_t* swo = reinterpret_cast<uint16_t*>(bs_smem + M::kWo);          // W_o, W_o2
    uint16_t* sqkv = reinterpret_cast<uint16_t*>(bs_smem + M::kQkv);        // the head's q | k | v (behind W_o)
    uint16_t* sr = reinterpret_cast<uint16_t*>(bs_smem + M::kR);            // W_qkv | ctx | W_i | h, one after the other
    __shared__ __align__(8) uint64_t front, wi, wo2;                        // a layer's vectors, W_qkv and W_o; its W_i; its W_o2 are there
    const int rank = blockIdx.x % CL, cl = blockIdx.x / CL, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int s0 = cl * a.spc, ns = min(a.spc, a.b - s0), rows = ns * a.t;
    const size_t row0 = (size_t)s0 * a.t;
    uint16_t *ctx = a.ctx + row0 * kBsH, *hb = a.h + row0 * kBsI;
    float* pre = a.pre + row0 * kBsH;
    const bool has_head = rank < kBsHeads;
    bool ok = true;

    if (tid == 0) {
        mbar_init(&front, 1); mbar_init(&wi, 1); mbar_init(&wo2, 1);
        mbar_fence_init();
    }
    __syncthreads();
    // the block's biases and the LayerNorm vectors of a layer: [2][ln1w | ln1b | ln2w | ln2b | bqkv | bo | bi | bo2]; its rows of W_qkv and W_o
    auto bring_layer = [&](int l) {
        const BertSmallLayer& w = a.layers[l];
        float* d = sv + (l & 1) * M::NV;
        if (tid == 0) mbar_expect_tx(&front, (uint32_t)((M::NV - (has_head ? 0 : NQ * 8)) * 4 + (has_head ? kBsAtO * 2 : 0) + (kBsAtI - kBsAtO) * 2));
        const uint16_t* pack = w.pack + (size_t)rank * kBsPack;
        // (a copy per warp: the lanes of a warp issue theirs one after the other)
        const int v = lane == 0 ? warp : lane == 1 ? 8 + warp : -1;
        if (has_head && v == 0) bulk_g2s(sr, pack, kBsAtO * 2, &front);
        if (v == 1) bulk_g2s(swo, pack + kBsAtO, (kBsAtI - kBsAtO) * 2, &front);
        const float* const ln[4] = {w.ln1w, w.ln1b, w.ln2w, w.ln2b};
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (v == 2 + i) bulk_g2s(d + i * kBsH, ln[i], kBsH * 4, &front);
        d += 4 * kBsH;
#pragma unroll
        for (int p = 0; p < 3; ++p)
            if (has_head && v == 6 + p) bulk_g2s(d + p * kBertD, w.bqkv + p * kBsH + rank * kBertD, kBertD * 4, &front);
        if (v == 9) bulk_g2s(d + NQ * 8, w.bo + rank * NO * 8, NO * 8 * 4, &front);
        if (v == 10) bulk_g2s(d + (NQ + NO) * 8, w.bi + rank * NI * 8, NI * 8 * 4, &front);
        if (v == 11) bulk_g2s(d + (NQ + NO + NI) * 8, w.bo2 + rank * NO * 8, NO * 8 * 4, &front);
    };
    bring_layer(0);

    // word + position embedding, LayerNorm (eps 1e-12): every block for itself; rows behind the sentences are zero
    for (int i = tid; i < (MT * 16 - rows) * LDX; i += kBsThreads) sx[(size_t)rows * LDX + i] = 0;
    for (int r = warp; r < rows; r += kBsThreads / 32) {
        const uint32_t id = min(a.ids[row0 + r], (uint32_t)(a.V - 1));
        const int pos = min(r % a.t, a.maxpos - 1);
        const uint16_t *w = a.wemb + (size_t)id * kBsH, *p = a.pemb + (size_t)pos * kBsH;
        float v[12];
        float s = 0.f, s2 = 0.f;
#pragma unroll
        for (int j = 0; j < 12; ++j) {
            const int c = lane + 32 * j;
            v[j] = __uint_as_float((uint32_t)w[c] << 16) + __uint_as_float((uint32_t)p[c] << 16);
            s += v[j];
            s2 = fmaf(v[j], v[j], s2);
        }
        s = warp_sum(s);
        s2 = warp_sum(s2);
        const float mean = s / (float)kBsH, inv = 1.f / sqrtf(s2 / (float)kBsH - mean * mean + 1e-12f);
#pragma unroll
        for (int j = 0; j < 12; ++j) {
            const int c = lane + 32 * j;
            sx[r * LDX + c] = f32_to_bf16_rne((v[j] - mean) * inv * a.lnw[c] + a.lnb[c]);
        }
    }

#pragma unroll 1
    for (int l = 0; l < a.L; ++l) {
        const BertSmallLayer& w = a.layers[l];
        ok = ok && pair_wait(&front, l & 1);
        __syncthreads();                    // the x tile, the layer's vectors, W_qkv and W_o are complete
        const float *ln1w = sv + (l & 1) * M::NV, *ln1b = ln1w + kBsH, *ln2w = ln1b + kBsH, *ln2b = ln2w + kBsH, *bqkv = ln2b + kBsH, *bo = bqkv + NQ * 8, *bi = bo + NO * 8,
                    *bo2 = bi + NI * 8;
        if (has_head) {
            BsTiles<MT, NQ> y;
            y.zero();
            y.template add<kBsH>(sx, sr, bs_ld(kBsH), 0, warp, lane);
            y.store(rows, warp, lane, [&](int r, int c, float2 s) {
                *reinterpret_cast<uint32_t*>(sqkv + r * M::kQkvLd + c) = pack_bf16x2(s.x + bqkv[c], s.y + bqkv[c + 1]);
            });
        }
        __syncthreads();
        if (has_head) {     // the block's warps share the head's (sentence, 16 query rows)
            const int pairs = ns, per = 16, split = (a.t + per - 1) / per;
            for (int it = warp; it < pairs * split; it += kBsThreads / 32) {
                const int sent = it % pairs, m0 = it / pairs * per;
                uint16_t *q = sqkv + sent * a.t * M::kQkvLd, *to = ctx + (size_t)sent * a.t * kBsH + rank * kBertD;
                auto go = [&](auto kt) { bq_attention<decltype(kt)::value, M::kQkvLd>(q, q + kBertD, q + 2 * kBertD, a.t, m0, a.inv_scale, to, lane); };
                switch (split) {
                    case 1: go(std::integral_constant<int, 1>{}); break;
                    case 2: go(std::integral_constant<int, 2>{}); break;
                    case 3: go(std::integral_constant<int, 3>{}); break;
                    default: go(std::integral_constant<int, 4>{});
                }
            }
        }
        bs_arrive();
        bs_wait();
        auto residual = [&](const float* bias) {
            return [&, bias](int r, int c, float2 s) {
                const int col = rank * NO * 8 + c;
                const uint32_t x = *reinterpret_cast<const uint32_t*>(sx + r * LDX + col);
                *reinterpret_cast<float2*>(pre + (size_t)r * kBsH + col) = make_float2(s.x + bias[c] + bf16lo(x), s.y + bias[c + 1] + bf16hi(x));
            };
        };
        bs_bring_rows<kBsH>(sr, ctx, kBsH, 0, rows);
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        {
            BsTiles<MT, NO> y;
            y.zero();
            y.template add<kBsH>(sr, swo, bs_ld(kBsH), 0, warp, lane);
            y.store(rows, warp, lane, residual(bo));
        }
        bs_arrive();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();                    // ctx and W_o have been read
        if (tid == 0) {
            mbar_expect_tx(&wi, (kBsAtO2 - kBsAtI) * 2);
            bulk_g2s(sr, w.pack + (size_t)rank * kBsPack + kBsAtI, (kBsAtO2 - kBsAtI) * 2, &wi);
            mbar_expect_tx(&wo2, (kBsPack - kBsAtO2) * 2);
            bulk_g2s(swo, w.pack + (size_t)rank * kBsPack + kBsAtO2, (kBsPack - kBsAtO2) * 2, &wo2);
        }
        bs_wait();
        bs_layernorm(pre, rows, ln1w, ln1b, a.eps, sx, warp, lane);
        ok = ok && pair_wait(&wi, l & 1);
        __syncthreads();
        {
            BsTiles<MT, NI> y;
            y.zero();
            y.template add<kBsH>(sx, sr, bs_ld(kBsH), 0, warp, lane);
            y.store(rows, warp, lane, [&](int r, int c, float2 s) {
                *reinterpret_cast<uint32_t*>(hb + (size_t)r * kBsI + rank * NI * 8 + c) = pack_bf16x2(gelu_tanh_f(s.x + bi[c]), gelu_tanh_f(s.y + bi[c + 1]));
            });
        }
        bs_arrive();
        bs_wait();
        {
            BsTiles<MT, NO> y;
            y.zero();
            constexpr int AHEAD = M::kHBufs == M::kPieces ? M::kPieces : 1;
#pragma unroll
            for (int p = 0; p < AHEAD; ++p) {
                bs_bring_rows<M::kHPiece>(sr + p * M::kHBuf, hb, kBsI, p * M::kHPiece, rows);
                cp_async_commit();
            }
            ok = ok && pair_wait(&wo2, l & 1);
            if constexpr (AHEAD == M::kPieces) {
                auto piece = [&](auto at) {
                    constexpr int P = decltype(at)::value;
                    cp_async_wait<AHEAD - 1 - P>();
                    __syncthreads();
                    y.template add<M::kHPiece>(sr + P * M::kHBuf, swo, bs_ld(kBsI), P * M::kHPiece, warp, lane);
                };
                static_assert(AHEAD != M::kPieces || M::kPieces == 4, "");
                piece(std::integral_constant<int, 0>{});
                piece(std::integral_constant<int, 1>{});
                piece(std::integral_constant<int, 2>{});
                piece(std::integral_constant<int, 3>{});
            } else {
#pragma unroll 1
                for (int p = 0; p < M::kPieces; ++p) {
                    if (p > 0) __syncthreads();                 // the piece before has been read
                    if (p + 1 < M::kPieces) bs_bring_rows<M::kHPiece>(sr + ((p + 1) & 1) * M::kHBuf, hb, kBsI, (p + 1) * M::kHPiece, rows);
                    cp_async_commit();
                    cp_async_wait<1>();
                    __syncthreads();
                    y.template add<M::kHPiece>(sr + (p & 1) * M::kHBuf, swo, bs_ld(kBsI), p * M::kHPiece, warp, lane);
                }
            }
            y.store(rows, warp, lane, residual(bo2));
        }
        bs_arrive();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();                    // h and W_o2 have been read
        if (l + 1 < a.L) bring_layer(l + 1);
        bs_wait();
        bs_layernorm(pre, rows, ln2w, ln2b, a.eps, sx, warp, lane);
    }
    if (!ok) {          // a wait ran out: report it, leave the copies in flight time to land, go on to the end
        if (lane == 0 && a.failed != nullptr) *a.failed = 1;
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    __syncthreads();
    // masked mean pooling and L2 norm: a block takes every CL-th sentence, a thread up to two columns; tot[w]: squares of columns 32 w ..
    __shared__ float tot[kBsH / 32];
    for (int s = rank; s < ns; s += CL) {
        float acc[2] = {0.f, 0.f}, cnt = 0.f;
        for (int r = 0; r < a.t; ++r) {
            const float m = a.mask ? (float)a.mask[row0 + (size_t)s * a.t + r] : 1.f;
            cnt += m;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int c = tid + u * kBsThreads;
                if (c < kBsH) acc[u] = fmaf(__uint_as_float((uint32_t)sx[(s * a.t + r) * LDX + c] << 16), m, acc[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            acc[u] /= cnt * (float)kBsH;
            const float sq = warp_sum(acc[u] * acc[u]);
            if (lane == 0 && warp + 8 * u < kBsH / 32) tot[warp + 8 * u] = sq;
        }
        __syncthreads();
        float sum = 0.f;
        for (int k = 0; k < kBsH / 32; ++k) sum += tot[k];
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int c = tid + u * kBsThreads;
            if (c < kBsH) a.out[(size_t)(s0 + s) * kBsH + c] = acc[u] / sqrtf(sum);
        }
    }
}
template <int MT, int CL>
constexpr size_t bert_small_smem() { return BsSmem<MT, CL>::kBytes; }

}  // namespace fl
