// The encoder on few short sentences in ONE launch: a cluster of blocks per up to 64 tokens (whole sentences).
//
// A query of a dozen tokens through the launch chain is 44 kernels, each of them a few microseconds of latency around almost no work (the
// 24 GEMMs fill 2 to 8 of 148 SMs and walk K one 64-column block after the other).  Here the blocks of a cluster split every projection's
// output columns; phases are separated by the cluster's hardware barrier instead of a kernel boundary, and the weights of a phase -- which
// depend on nothing -- travel into shared memory while the cluster waits for the phase before.
//   per layer: x -> q|k|v | attention, one warp per (sentence, head, 16 query rows) | x + W_o ctx | LayerNorm (every block for itself) ->
//   gelu(W_i x1) | x1 + W_o2 h | LayerNorm
// The results are the chain's, bit for bit: an output's products go into its f32 accumulator 16 columns of K at a time in ascending order, as
// tcgen05.mma takes them (mma.sync m16n8k16 sums the same 16 products to the same bits, in whatever order they stand inside the 16), so K is
// not split over warps; attention, roundings and the order of every other sum are those of bert.cuh.
// Bound: latency -- 5 phases x 6 layers of about 5 us (cluster barrier, L2 round trips of activations and weights, a chain of 24 to 96 MMAs).
// One sentence of 4 / 19 / 48 / 64 tokens, whole call: 243 / 254 / 268 / 277 us as 44 launches, 120 / 160 / 224 / 269 us here.  (K in quarters over
// the warps is no faster, and its sums are not the chain's: 16-bit activations carry that to 3e-3 in the embedding.)
#pragma once
#include "bert.cuh"
#include "gemm_tc.cuh"

namespace fl {

constexpr int kBsTokens = 64, kBsThreads = 256, kBsH = 384, kBsI = 1536, kBsHeads = 12;     // all-MiniLM-L6-v2's sizes
// Operand rows in shared memory: bf16, 32 columns as four 16-byte pieces, piece q = columns 4 q .. 4 q + 3 of the first 16 and of the second 16.
// One 16-byte load is then a lane's share of two MMAs, both inside their own 16 columns of K.  h and ctx lie in global memory the same way.
__host__ __device__ constexpr int bs_at(int c) { return (c & ~31) | ((c >> 2 & 3) << 3) | ((c >> 4 & 1) << 2) | (c & 3); }
__host__ __device__ constexpr int bs_ld(int k) { return k + 32; }       // the eight lanes of a quarter-warp's 16-byte load on different banks

struct BertSmallLayer {
    const uint16_t *wqkv, *wo, *wi, *wo2;
    const float *bqkv, *bo, *bi, *bo2, *ln1w, *ln1b, *ln2w, *ln2b;
};
struct BertSmallArgs {
    const BertSmallLayer* layers;           // device
    const uint16_t *wemb, *pemb; const float *lnw, *lnb;
    const uint32_t *ids, *mask;             // [b t]; mask may be null
    int L, b, t, V, maxpos, spc;            // spc: sentences per cluster
    float eps, inv_scale;
    uint16_t *qkv, *ctx, *h; float* pre;    // workspace rows as the launch chain has them
    float* out;
};
// Shared memory of a block, in bytes: a layer's vectors twice | x | W_o or W_o2 | W_qkv, W_i or the gathered rows of ctx or h
template <int MT, int CL>
struct BsSmem {
    static constexpr int NQ = 3 * kBsH / 8 / CL, NO = kBsH / 8 / CL, NI = kBsI / 8 / CL;        // column tiles per block of the three widths
    static_assert(NQ * CL * 8 == 3 * kBsH && NO * CL * 8 == kBsH && NI * CL * 8 == kBsI, "whole tiles per block");
    static constexpr int NV = 4 * kBsH + (NQ + 2 * NO + NI) * 8;
    // h arrives whole, or (rows that would not fit) in pieces of its columns, one multiplied while the next is on its way
    static constexpr int kHPiece = MT <= 2 ? kBsI : (MT == 3 ? kBsI / 4 : kBsI / 6), kPieces = kBsI / kHPiece, kHBufs = kPieces > 1 ? 2 : 1;
    static constexpr int kHBuf = MT * 16 * bs_ld(kHPiece);                                       // elements
    static constexpr size_t max2(size_t a, size_t b) { return a > b ? a : b; }
    static constexpr size_t kX = (size_t)2 * NV * 4, kWo = kX + (size_t)MT * 16 * bs_ld(kBsH) * 2, kR = kWo + (size_t)NO * 8 * bs_ld(kBsI) * 2;
    static constexpr size_t kBytes = kR + max2((size_t)(NQ > NI ? NQ : NI) * 8 * bs_ld(kBsH) * 2, max2((size_t)MT * 16 * bs_ld(kBsH) * 2, (size_t)kHBufs * kHBuf * 2));
    static_assert(kHPiece % 32 == 0 && kX % 16 == 0 && kBytes <= 232448, "");
};

__device__ __forceinline__ void bs_arrive() { __syncwarp(); asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void bs_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// rows [0, ROWS) of a weight matrix [.., K], on their way
template <int ROWS, int K>
__device__ __forceinline__ void bs_bring_weights(uint16_t* dst, const uint16_t* W) {
    for (int i = threadIdx.x; i < ROWS * (K / 4); i += kBsThreads) {
        const int r = i / (K / 4), c = i % (K / 4) * 4;
        cp_async8(dst + r * bs_ld(K) + bs_at(c), W + (size_t)r * K + c);
    }
}
// columns [k0, k0 + KP) of the cluster's rows of an activation that the cluster wrote
template <int KP>
__device__ __forceinline__ void bs_bring_rows(uint16_t* dst, const uint16_t* src, int ld, int k0, int rows) {
    for (int i = threadIdx.x; i < rows * (KP / 8); i += kBsThreads) {
        const int r = i / (KP / 8), c = i % (KP / 8) * 8;
        cp_async16(dst + r * bs_ld(KP) + c, src + (size_t)r * ld + k0 + c);
    }
}
// One projection's NT x MT tiles of 8 columns x 16 rows, dealt to the warps: warp w has tiles w, w + 8, ... (column tiles first).
template <int MT, int NT>
struct BsTiles {
    static constexpr int IT = (NT * MT + 7) / 8;
    float acc[IT][4];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < IT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    }
    // += A [.., KP] . columns [k0, k0 + KP) of W
    template <int KP>
    __device__ __forceinline__ void add(const uint16_t* A, const uint16_t* W, int ldw, int k0, int warp, int lane) {
        const int g = lane >> 2, q = lane & 3;
#pragma unroll 12
        for (int s = 0; s < KP / 32; ++s)
#pragma unroll
            for (int i = 0; i < IT; ++i) {
                const int tile = warp + 8 * i;
                if (tile < NT * MT) {
                    const uint16_t* a = A + (tile / NT * 16 + g) * bs_ld(KP) + s * 32 + q * 8;
                    const uint4 x0 = *reinterpret_cast<const uint4*>(a), x1 = *reinterpret_cast<const uint4*>(a + 8 * bs_ld(KP));
                    const uint4 w = *reinterpret_cast<const uint4*>(W + (tile % NT * 8 + g) * ldw + k0 + s * 32 + q * 8);
                    const uint32_t a0[4] = {x0.x, x1.x, x0.y, x1.y}, a1[4] = {x0.z, x1.z, x0.w, x1.w};
                    mma_bf16_16816(acc[i], a0, w.x, w.y);
                    mma_bf16_16816(acc[i], a1, w.z, w.w);
                }
            }
    }
    // out(row, column pair inside the block, sums)
    template <typename Fn>
    __device__ __forceinline__ void store(int rows, int warp, int lane, Fn&& out) const {
#pragma unroll
        for (int i = 0; i < IT; ++i) {
            const int tile = warp + 8 * i;
            if (tile < NT * MT) {
                const int r = tile / NT * 16 + (lane >> 2), c = tile % NT * 8 + (lane & 3) * 2;
                if (r < rows) out(r, c, make_float2(acc[i][0], acc[i][1]));
                if (r + 8 < rows) out(r + 8, c, make_float2(acc[i][2], acc[i][3]));
            }
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
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int r = r0 + u * NW;
            if (r >= rows) break;
            float s = 0.f, s2 = 0.f;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const float4 x = v[u][j];
                s += (x.x + x.y) + (x.z + x.w);
                s2 = fmaf(x.x, x.x, s2); s2 = fmaf(x.y, x.y, s2); s2 = fmaf(x.z, x.z, s2); s2 = fmaf(x.w, x.w, s2);
            }
            s = warp_sum(s);
            s2 = warp_sum(s2);
            const float mean = s / (float)kBsH, inv = 1.f / sqrtf(s2 / (float)kBsH - mean * mean + eps);
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int c = lane + 32 * j;
                const float4 x = v[u][j], w4 = reinterpret_cast<const float4*>(w)[c], b4 = reinterpret_cast<const float4*>(b)[c];
                *reinterpret_cast<uint2*>(sx + r * bs_ld(kBsH) + bs_at(4 * c)) =
                    make_uint2(pack_bf16x2((x.x - mean) * inv * w4.x + b4.x, (x.y - mean) * inv * w4.y + b4.y),
                               pack_bf16x2((x.z - mean) * inv * w4.z + b4.z, (x.w - mean) * inv * w4.w + b4.w));
            }
        }
    }
}

// bert_attn_kernel for 16 query rows of a head, operands straight from global memory (its key tiles behind the sentence add zeros; here there
// are KT tiles of eight keys).  base: q columns of the head in the sentence's first row of q|k|v; ctx: the sentence's first row, permuted.
template <int KT>
__device__ __forceinline__ void bs_attention(const uint16_t* base, int t, int m0, float inv_scale, uint16_t* ctx, int lane) {
    constexpr int LD = 3 * kBsH;
    const int g = lane >> 2, q = lane & 3;
    const uint2 zero2 = make_uint2(0u, 0u);
    auto ld8 = [&](const uint16_t* p, int row) { return row < t ? __ldcg(reinterpret_cast<const uint2*>(p + (size_t)row * LD)) : zero2; };
    uint32_t qa[2][4], vv[KT][4];
    uint2 kk[KT][2];
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
        const uint2 x0 = ld8(base + ks * 16 + q * 4, m0 + g), x1 = ld8(base + ks * 16 + q * 4, m0 + g + 8);
        qa[ks][0] = x0.x; qa[ks][1] = x1.x; qa[ks][2] = x0.y; qa[ks][3] = x1.y;
    }
#pragma unroll
    for (int nt = 0; nt < KT; ++nt) {
        const int key = nt * 8 + g;
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) kk[nt][ks] = ld8(base + kBsH + ks * 16 + q * 4, key);
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (key < t) v = __ldcg(reinterpret_cast<const uint4*>(base + 2 * kBsH + (size_t)key * LD + q * 8));
        vv[nt][0] = v.x; vv[nt][1] = v.y; vv[nt][2] = v.z; vv[nt][3] = v.w;
    }
    float s[KT][4];
#pragma unroll
    for (int nt = 0; nt < KT; ++nt) {
        s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) mma_bf16_16816(s[nt], qa[ks], kk[nt][ks].x, kk[nt][ks].y);
    }
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int nt = 0; nt < KT; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) s[nt][e] = nt * 8 + q * 2 + (e & 1) < t ? s[nt][e] * inv_scale : -INFINITY;
        mx0 = fmaxf(mx0, fmaxf(s[nt][0], s[nt][1]));
        mx1 = fmaxf(mx1, fmaxf(s[nt][2], s[nt][3]));
    }
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xFFFFFFFFu, mx0, 1)); mx0 = fmaxf(mx0, __shfl_xor_sync(0xFFFFFFFFu, mx0, 2));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xFFFFFFFFu, mx1, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xFFFFFFFFu, mx1, 2));
    float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
    for (int nt = 0; nt < KT; ++nt) {
        s[nt][0] = __expf(s[nt][0] - mx0); s[nt][1] = __expf(s[nt][1] - mx0);
        s[nt][2] = __expf(s[nt][2] - mx1); s[nt][3] = __expf(s[nt][3] - mx1);
        sum0 += s[nt][0] + s[nt][1];
        sum1 += s[nt][2] + s[nt][3];
    }
    sum0 += __shfl_xor_sync(0xFFFFFFFFu, sum0, 1); sum0 += __shfl_xor_sync(0xFFFFFFFFu, sum0, 2);
    sum1 += __shfl_xor_sync(0xFFFFFFFFu, sum1, 1); sum1 += __shfl_xor_sync(0xFFFFFFFFu, sum1, 2);
    // A lane's 16 bytes of a key are channels 8 q .. 8 q + 7; transposing register j of eight keys gives the operand of the channels
    // {8 q' + 2 j, 8 q' + 2 j + 1: q' < 4}, and the sums o[j] of this lane are those of its own q: eight neighbouring channels per row.
    float o[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < KT / 2; ++ks) {
        const uint32_t pa[4] = {pack_bf16(s[2 * ks][0], s[2 * ks][1]), pack_bf16(s[2 * ks][2], s[2 * ks][3]), pack_bf16(s[2 * ks + 1][0], s[2 * ks + 1][1]),
                                pack_bf16(s[2 * ks + 1][2], s[2 * ks + 1][3])};
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_bf16_16816(o[j], pa, movmatrix_trans(vv[2 * ks][j]), movmatrix_trans(vv[2 * ks + 1][j]));
    }
    const float i0 = 1.f / sum0, i1 = 1.f / sum1;
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {        // channels 8 q + 4 hf ..
        uint16_t* p = ctx + bs_at(q * 8 + hf * 4);
        const float *a = o[2 * hf], *b = o[2 * hf + 1];
        if (m0 + g < t) *reinterpret_cast<uint2*>(p + (size_t)(m0 + g) * kBsH) = make_uint2(pack_bf16(a[0] * i0, a[1] * i0), pack_bf16(b[0] * i0, b[1] * i0));
        if (m0 + g + 8 < t) *reinterpret_cast<uint2*>(p + (size_t)(m0 + g + 8) * kBsH) = make_uint2(pack_bf16(a[2] * i1, a[3] * i1), pack_bf16(b[2] * i1, b[3] * i1));
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
    uint16_t* sr = reinterpret_cast<uint16_t*>(bs_smem + M::kR);            // W_qkv | ctx | W_i | h, one after the other
    const int rank = blockIdx.x % CL, cl = blockIdx.x / CL, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int s0 = cl * a.spc, ns = min(a.spc, a.b - s0), rows = ns * a.t;
    const size_t row0 = (size_t)s0 * a.t;
    uint16_t *qkv = a.qkv + row0 * 3 * kBsH, *ctx = a.ctx + row0 * kBsH, *hb = a.h + row0 * kBsI;
    float* pre = a.pre + row0 * kBsH;

    // the block's biases and the LayerNorm vectors of a layer: [2][ln1w | ln1b | ln2w | ln2b | bqkv | bo | bi | bo2]; its rows of W_qkv
    auto bring_layer = [&](int l) {
        const BertSmallLayer& w = a.layers[l];
        float* d = sv + (l & 1) * M::NV;
        for (int i = tid; i < kBsH; i += kBsThreads) {
            cp_async_f32(d + i, w.ln1w + i); cp_async_f32(d + kBsH + i, w.ln1b + i);
            cp_async_f32(d + 2 * kBsH + i, w.ln2w + i); cp_async_f32(d + 3 * kBsH + i, w.ln2b + i);
        }
        d += 4 * kBsH;
        if (tid < NQ * 8) cp_async_f32(d + tid, w.bqkv + rank * NQ * 8 + tid);
        if (tid < NO * 8) { cp_async_f32(d + NQ * 8 + tid, w.bo + rank * NO * 8 + tid); cp_async_f32(d + (NQ + NO + NI) * 8 + tid, w.bo2 + rank * NO * 8 + tid); }
        if (tid < NI * 8) cp_async_f32(d + (NQ + NO) * 8 + tid, w.bi + rank * NI * 8 + tid);
        bs_bring_weights<NQ * 8, kBsH>(sr, w.wqkv + (size_t)rank * NQ * 8 * kBsH);
        bs_bring_weights<NO * 8, kBsH>(swo, w.wo + (size_t)rank * NO * 8 * kBsH);
        cp_async_commit();
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
            sx[r * LDX + bs_at(c)] = f32_to_bf16_rne((v[j] - mean) * inv * a.lnw[c] + a.lnb[c]);
        }
    }

#pragma unroll 1
    for (int l = 0; l < a.L; ++l) {
        const BertSmallLayer& w = a.layers[l];
        cp_async_wait<0>();
        __syncthreads();                    // the x tile, the layer's vectors, W_qkv and W_o are complete
        const float *ln1w = sv + (l & 1) * M::NV, *ln1b = ln1w + kBsH, *ln2w = ln1b + kBsH, *ln2b = ln2w + kBsH, *bqkv = ln2b + kBsH, *bo = bqkv + NQ * 8, *bi = bo + NO * 8,
                    *bo2 = bi + NI * 8;
        {
            BsTiles<MT, NQ> y;
            y.zero();
            y.template add<kBsH>(sx, sr, bs_ld(kBsH), 0, warp, lane);
            y.store(rows, warp, lane, [&](int r, int c, float2 s) {
                *reinterpret_cast<uint32_t*>(qkv + (size_t)r * 3 * kBsH + rank * NQ * 8 + c) = pack_bf16x2(s.x + bqkv[c], s.y + bqkv[c + 1]);
            });
        }
        bs_arrive();
        bs_wait();
        {   // attention: the cluster's warps share the (sentence, head, 16 query rows)
            const int pairs = ns * kBsHeads, per = 16, split = (a.t + per - 1) / per;
            for (int it = warp * CL + rank; it < pairs * split; it += CL * (kBsThreads / 32)) {
                const int pr = it % pairs, sent = pr / kBsHeads, head = pr % kBsHeads;
                bs_attention<2 * MT>(qkv + (size_t)sent * a.t * 3 * kBsH + head * kBertD, a.t, it / pairs * per, a.inv_scale, ctx + (size_t)sent * a.t * kBsH + head * kBertD, lane);
            }
        }
        bs_arrive();
        bs_wait();
        auto residual = [&](const float* bias) {
            return [&, bias](int r, int c, float2 s) {
                const int col = rank * NO * 8 + c;
                const uint32_t x = *reinterpret_cast<const uint32_t*>(sx + r * LDX + bs_at(col));
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
        __syncthreads();                    // ctx and W_o have been read
        bs_bring_weights<NI * 8, kBsH>(sr, w.wi + (size_t)rank * NI * 8 * kBsH);
        cp_async_commit();
        bs_bring_weights<NO * 8, kBsI>(swo, w.wo2 + (size_t)rank * NO * 8 * kBsI);
        cp_async_commit();
        bs_wait();
        bs_layernorm(pre, rows, ln1w, ln1b, a.eps, sx, warp, lane);
        cp_async_wait<1>();
        __syncthreads();
        {
            BsTiles<MT, NI> y;
            y.zero();
            y.template add<kBsH>(sx, sr, bs_ld(kBsH), 0, warp, lane);
            y.store(rows, warp, lane, [&](int r, int c, float2 s) {
                *reinterpret_cast<uint32_t*>(hb + (size_t)r * kBsI + bs_at(rank * NI * 8 + c)) = pack_bf16x2(gelu_tanh_f(s.x + bi[c]), gelu_tanh_f(s.y + bi[c + 1]));
            });
        }
        bs_arrive();
        bs_wait();
        {
            BsTiles<MT, NO> y;
            y.zero();
            bs_bring_rows<M::kHPiece>(sr, hb, kBsI, 0, rows);
            cp_async_commit();
#pragma unroll 1
            for (int p = 0; p < M::kPieces; ++p) {
                if (p > 0) __syncthreads();                 // the piece before has been read
                if (p + 1 < M::kPieces) bs_bring_rows<M::kHPiece>(sr + ((p + 1) & 1) * M::kHBuf, hb, kBsI, (p + 1) * M::kHPiece, rows);
                cp_async_commit();
                cp_async_wait<1>();
                __syncthreads();
                y.template add<M::kHPiece>(sr + (p & 1) * M::kHBuf, swo, bs_ld(kBsI), p * M::kHPiece, warp, lane);
            }
            y.store(rows, warp, lane, residual(bo2));
        }
        bs_arrive();
        __syncthreads();                    // h and W_o2 have been read
        if (l + 1 < a.L) bring_layer(l + 1);
        bs_wait();
        bs_layernorm(pre, rows, ln2w, ln2b, a.eps, sx, warp, lane);
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
                if (c < kBsH) acc[u] = fmaf(__uint_as_float((uint32_t)sx[(s * a.t + r) * LDX + bs_at(c)] << 16), m, acc[u]);
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
