// The encoder on few short sentences in ONE launch: a cluster of blocks per up to 64 tokens (whole sentences).
//
// A query of a dozen tokens through the launch chain is 44 kernels, each of them a few microseconds of latency around almost no work (the
// 24 GEMMs fill 2 to 8 of 148 SMs and walk K one 64-column block after the other).  Here the blocks of a cluster split every projection's
// output columns; phases are separated by the cluster's hardware barrier instead of a kernel boundary, and the weights of a phase -- which
// depend on nothing -- travel into registers while the cluster waits for the phase before.
//   per layer: x -> q|k|v | attention, one warp per (sentence, head, rows) | x + W_o ctx | LayerNorm (every block for itself) -> gelu(W_i x1) |
//   x1 + W_o2 h | LayerNorm
// A warp multiplies a quarter of K (mma.sync m16n8k16, f32 accumulation) for half of the block's columns; the four quarters meet in shared
// memory in a fixed order.  Roundings are the chain's: q|k|v, ctx, x, h in bf16, sums, residuals and LayerNorm in f32 (and the
// probabilities, which the chain rounds).
// Bound: latency -- 5 phases x 6 layers of about 4 us (cluster barrier, L2 round trips of activations and weights, a few MMAs).
// One sentence of 19 tokens, whole call: 257 -> 161 us.
#pragma once
#include "bert.cuh"
#include "gemm_tc.cuh"

namespace fl {

constexpr int kBsTokens = 64, kBsThreads = 256, kBsH = 384, kBsI = 1536, kBsHeads = 12;     // all-MiniLM-L6-v2's sizes
constexpr int kBsLdX = kBsH + 8;            // bf16 row of the x tile: neighbouring rows start four banks apart

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

__device__ __forceinline__ void bs_arrive() { __syncwarp(); asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void bs_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// One projection.  Output columns of the cluster: NT tiles of eight per block, block `rank` has columns [rank NT 8, ...); warp = (K quarter ks,
// column half tg).  Within 32 columns of K a lane holds eight neighbouring ones of its row (16-byte loads); weights and activations are
// permuted alike, so the sum does not change.
template <int NT, int K>
struct BsWeights {
    static constexpr int HT = (NT + 1) / 2, STEPS = K / 4 / 32;
    uint4 w[HT][STEPS];
    __device__ __forceinline__ void load(const uint16_t* W, int rank, int warp, int lane) {
        const int ks = warp & 3, tg = warp >> 2;
#pragma unroll
        for (int i = 0; i < HT; ++i) {
            const int tile = tg * HT + i;
            if (tile < NT) {
                const uint16_t* p = W + (size_t)((rank * NT + tile) * 8 + (lane >> 2)) * K + ks * (K / 4) + (lane & 3) * 8;
#pragma unroll
                for (int s = 0; s < STEPS; ++s) w[i][s] = *reinterpret_cast<const uint4*>(p + s * 32);
            }
        }
    }
};
// red [4 quarters][MT 16 rows][NT 8 + 4] += A . W^T; row(r): pointer to row r's K activations (shared or global), r < MT 16
template <int MT, int NT, int K, typename RowFn>
__device__ __forceinline__ void bs_gemm(const BsWeights<NT, K>& bw, RowFn&& rows16, float* red, int warp, int lane) {
    constexpr int LDR = NT * 8 + 4;
    const int ks = warp & 3, tg = warp >> 2, g = lane >> 2, q = lane & 3;
    using W = BsWeights<NT, K>;
    float acc[MT][W::HT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int i = 0; i < W::HT; ++i) acc[m][i][0] = acc[m][i][1] = acc[m][i][2] = acc[m][i][3] = 0.f;
#pragma unroll
    for (int s = 0; s < W::STEPS; ++s) {
        const int k = ks * (K / 4) + s * 32 + q * 8;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const uint4 x0 = rows16(m * 16 + g, k), x1 = rows16(m * 16 + g + 8, k);
            const uint32_t a0[4] = {x0.x, x1.x, x0.y, x1.y}, a1[4] = {x0.z, x1.z, x0.w, x1.w};
#pragma unroll
            for (int i = 0; i < W::HT; ++i)
                if (tg * W::HT + i < NT) {
                    const uint32_t b0[2] = {bw.w[i][s].x, bw.w[i][s].y}, b1[2] = {bw.w[i][s].z, bw.w[i][s].w};
                    mma_bf16_16816(acc[m][i], a0, b0);
                    mma_bf16_16816(acc[m][i], a1, b1);
                }
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int i = 0; i < W::HT; ++i)
            if (tg * W::HT + i < NT) {
                float* r = red + (size_t)(ks * MT * 16 + m * 16 + g) * LDR + (tg * W::HT + i) * 8 + q * 2;
                r[0] = acc[m][i][0]; r[1] = acc[m][i][1];
                r[8 * LDR] = acc[m][i][2]; r[8 * LDR + 1] = acc[m][i][3];
            }
}
// columns of the block, two at a time: out(row, column pair inside the block, sums of the four quarters)
template <int MT, int NT, typename Fn>
__device__ __forceinline__ void bs_fold(const float* red, int rows, Fn&& out) {
    constexpr int LDR = NT * 8 + 4, HALF = NT * 4, Q = MT * 16 * LDR;
    for (int i = threadIdx.x; i < rows * HALF; i += kBsThreads) {
        const int r = i / HALF, c = i % HALF * 2;
        const float* p = red + r * LDR + c;
        float2 s = *reinterpret_cast<const float2*>(p);
#pragma unroll
        for (int k = 1; k < 4; ++k) {
            const float2 v = *reinterpret_cast<const float2*>(p + k * Q);
            s.x += v.x; s.y += v.y;
        }
        out(r, c, s);
    }
}

__device__ __forceinline__ uint32_t bs_word(const uint4& v, int e) { return e == 0 ? v.x : (e == 1 ? v.y : (e == 2 ? v.z : v.w)); }

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
                *reinterpret_cast<uint2*>(sx + r * kBsLdX + 4 * c) = make_uint2(pack_bf16x2((x.x - mean) * inv * w4.x + b4.x, (x.y - mean) * inv * w4.y + b4.y),
                                                                                pack_bf16x2((x.z - mean) * inv * w4.z + b4.z, (x.w - mean) * inv * w4.w + b4.w));
            }
        }
    }
}

// MT: row tiles of 16 (the cluster's tokens, rounded up); CL: blocks per cluster.  grid clusters * CL.
template <int MT, int CL>
static __global__ void __launch_bounds__(kBsThreads, 1) bert_small_kernel(const BertSmallArgs a) {
    constexpr int NQ = 3 * kBsH / 8 / CL, NO = kBsH / 8 / CL, NI = kBsI / 8 / CL;        // column tiles per block of the three widths
    static_assert(NQ * CL * 8 == 3 * kBsH && NO * CL * 8 == kBsH && NI * CL * 8 == kBsI, "whole tiles per block");
    extern __shared__ __align__(16) uint8_t bs_smem[];
    uint16_t* sx = reinterpret_cast<uint16_t*>(bs_smem);                                // [MT 16][kBsLdX]
    float* red = reinterpret_cast<float*>(bs_smem + (size_t)MT * 16 * kBsLdX * 2);      // [4][MT 16][NI 8 + 4]
    const int rank = blockIdx.x % CL, cl = blockIdx.x / CL, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int s0 = cl * a.spc, ns = min(a.spc, a.b - s0), rows = ns * a.t;
    const size_t row0 = (size_t)s0 * a.t;
    uint16_t *qkv = a.qkv + row0 * 3 * kBsH, *ctx = a.ctx + row0 * kBsH, *hb = a.h + row0 * kBsI;
    float* pre = a.pre + row0 * kBsH;

    // word + position embedding, LayerNorm (eps 1e-12): every block for itself; rows behind the sentences are zero
    for (int i = tid; i < (MT * 16 - rows) * kBsLdX; i += kBsThreads) sx[(size_t)rows * kBsLdX + i] = 0;
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
            sx[r * kBsLdX + c] = f32_to_bf16_rne((v[j] - mean) * inv * a.lnw[c] + a.lnb[c]);
        }
    }
    auto from_x = [&](int r, int k) { return *reinterpret_cast<const uint4*>(sx + r * kBsLdX + k); };
    const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
    // the block's biases and the LayerNorm vectors of a layer, on their way a layer ahead: [2][ln1w | ln1b | ln2w | ln2b | bqkv | bo | bi | bo2]
    constexpr int NB = (NQ + 2 * NO + NI) * 8, NV = 4 * kBsH + NB;
    float* sv = red + (size_t)4 * MT * 16 * (NI * 8 + 4);
    auto bring_vectors = [&](int l) {
        const BertSmallLayer& w = a.layers[l];
        float* d = sv + (l & 1) * NV;
        for (int i = tid; i < kBsH; i += kBsThreads) {
            cp_async_f32(d + i, w.ln1w + i); cp_async_f32(d + kBsH + i, w.ln1b + i);
            cp_async_f32(d + 2 * kBsH + i, w.ln2w + i); cp_async_f32(d + 3 * kBsH + i, w.ln2b + i);
        }
        d += 4 * kBsH;
        if (tid < NQ * 8) cp_async_f32(d + tid, w.bqkv + rank * NQ * 8 + tid);
        if (tid < NO * 8) { cp_async_f32(d + NQ * 8 + tid, w.bo + rank * NO * 8 + tid); cp_async_f32(d + (NQ + NO + NI) * 8 + tid, w.bo2 + rank * NO * 8 + tid); }
        if (tid < NI * 8) cp_async_f32(d + (NQ + NO) * 8 + tid, w.bi + rank * NI * 8 + tid);
        cp_async_commit();
    };
    bring_vectors(0);

    BsWeights<NQ, kBsH> wq;
    wq.load(a.layers[0].wqkv, rank, warp, lane);
#pragma unroll 1
    for (int l = 0; l < a.L; ++l) {
        const BertSmallLayer& w = a.layers[l];
        cp_async_wait<0>();
        __syncthreads();                    // the x tile and the layer's vectors are complete
        const float *ln1w = sv + (l & 1) * NV, *ln1b = ln1w + kBsH, *ln2w = ln1b + kBsH, *ln2b = ln2w + kBsH, *bqkv = ln2b + kBsH, *bo = bqkv + NQ * 8, *bi = bo + NO * 8,
                    *bo2 = bi + NI * 8;
        bs_gemm<MT, NQ, kBsH>(wq, from_x, red, warp, lane);
        __syncthreads();
        bs_fold<MT, NQ>(red, rows, [&](int r, int c, float2 s) {
            const int col = rank * NQ * 8 + c;
            *reinterpret_cast<uint32_t*>(qkv + (size_t)r * 3 * kBsH + col) = pack_bf16x2(s.x + bqkv[c], s.y + bqkv[c + 1]);
        });
        BsWeights<NO, kBsH> wo;
        bs_arrive();
        wo.load(w.wo, rank, warp, lane);
        bs_wait();
        {   // attention: the cluster's warps share the (sentence, head) pairs, several warps of a pair its query rows
            // (whole stretches of `per` rows only: the first row of every item is one of the sentence)
            const int pairs = ns * kBsHeads, warps = CL * (kBsThreads / 32), most = max(1, min(a.t, warps / pairs)), per = (a.t + most - 1) / most, split = (a.t + per - 1) / per;
            for (int it = warp * CL + rank; it < pairs * split; it += warps) {
                const int pr = it % pairs, sent = pr / kBsHeads, head = pr % kBsHeads, first = it / pairs * per, last = min(a.t, first + per);
                const uint16_t* base = qkv + (size_t)sent * a.t * 3 * kBsH + head * kBertD;
                uint4 kk[2][4], vv[2][4];   // this lane's keys and values: lane, lane + 32
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint4* p = reinterpret_cast<const uint4*>(base + (size_t)(lane + 32 * u) * 3 * kBsH + kBsH) + c;
                        kk[u][c] = lane + 32 * u < a.t ? __ldcg(p) : zero4;
                        vv[u][c] = lane + 32 * u < a.t ? __ldcg(p + kBsH / 8) : zero4;
                    }
                uint16_t qn = __ldcg(base + (size_t)first * 3 * kBsH + lane);
                for (int i = first; i < last; ++i) {
                    const float qv = __uint_as_float((uint32_t)qn << 16) * a.inv_scale;
                    if (i + 1 < last) qn = __ldcg(base + (size_t)(i + 1) * 3 * kBsH + lane);
                    float sc[2] = {0.f, 0.f};
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float q0 = __shfl_sync(0xFFFFFFFFu, qv, c * 8 + e * 2), q1 = __shfl_sync(0xFFFFFFFFu, qv, c * 8 + e * 2 + 1);
#pragma unroll
                            for (int u = 0; u < 2; ++u) {
                                const uint32_t kv = bs_word(kk[u][c], e);
                                sc[u] = fmaf(q0, bf16lo(kv), fmaf(q1, bf16hi(kv), sc[u]));
                            }
                        }
                    if (lane >= a.t) sc[0] = -INFINITY;
                    if (lane + 32 >= a.t) sc[1] = -INFINITY;
                    const float m = warp_max(fmaxf(sc[0], sc[1]));
                    sc[0] = __expf(sc[0] - m);
                    sc[1] = __expf(sc[1] - m);
                    const float inv = 1.f / warp_sum(sc[0] + sc[1]);
                    // 32 sums over the lanes: halves of them are exchanged, lane c ends with channel c's
                    float o[32];
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const uint32_t v0 = bs_word(vv[0][c], e), v1 = bs_word(vv[1][c], e);
                            o[c * 8 + e * 2] = fmaf(sc[0], bf16lo(v0), sc[1] * bf16lo(v1));
                            o[c * 8 + e * 2 + 1] = fmaf(sc[0], bf16hi(v0), sc[1] * bf16hi(v1));
                        }
#pragma unroll
                    for (int n = 16; n >= 1; n >>= 1) {
                        const bool up = lane & n;
#pragma unroll
                        for (int j = 0; j < n; ++j) {
                            const float give = up ? o[j] : o[j + n], keep = up ? o[j + n] : o[j];
                            o[j] = keep + __shfl_xor_sync(0xFFFFFFFFu, give, n);
                        }
                    }
                    ctx[(size_t)(sent * a.t + i) * kBsH + head * kBertD + lane] = f32_to_bf16_rne(o[0] * inv);
                }
            }
        }
        bs_arrive();
        bs_wait();
        auto from_ctx = [&](int r, int k) { return r < rows ? __ldcg(reinterpret_cast<const uint4*>(ctx + (size_t)r * kBsH + k)) : zero4; };
        bs_gemm<MT, NO, kBsH>(wo, from_ctx, red, warp, lane);
        __syncthreads();
        auto residual = [&](const float* bias) {
            return [&, bias](int r, int c, float2 s) {
                const int col = rank * NO * 8 + c;
                const uint32_t x = *reinterpret_cast<const uint32_t*>(sx + r * kBsLdX + col);
                *reinterpret_cast<float2*>(pre + (size_t)r * kBsH + col) = make_float2(s.x + bias[c] + bf16lo(x), s.y + bias[c + 1] + bf16hi(x));
            };
        };
        bs_fold<MT, NO>(red, rows, residual(bo));
        BsWeights<NI, kBsH> wi;
        bs_arrive();
        wi.load(w.wi, rank, warp, lane);
        bs_wait();
        bs_layernorm(pre, rows, ln1w, ln1b, a.eps, sx, warp, lane);
        __syncthreads();
        bs_gemm<MT, NI, kBsH>(wi, from_x, red, warp, lane);
        __syncthreads();
        bs_fold<MT, NI>(red, rows, [&](int r, int c, float2 s) {
            const int col = rank * NI * 8 + c;
            *reinterpret_cast<uint32_t*>(hb + (size_t)r * kBsI + col) = pack_bf16x2(gelu_tanh_f(s.x + bi[c]), gelu_tanh_f(s.y + bi[c + 1]));
        });
        BsWeights<NO, kBsI> wd;
        bs_arrive();
        wd.load(w.wo2, rank, warp, lane);
        if (l + 1 < a.L) bring_vectors(l + 1);
        bs_wait();
        auto from_h = [&](int r, int k) { return r < rows ? __ldcg(reinterpret_cast<const uint4*>(hb + (size_t)r * kBsI + k)) : zero4; };
        bs_gemm<MT, NO, kBsI>(wd, from_h, red, warp, lane);
        __syncthreads();
        bs_fold<MT, NO>(red, rows, residual(bo2));
        bs_arrive();
        if (l + 1 < a.L) wq.load(a.layers[l + 1].wqkv, rank, warp, lane);
        bs_wait();
        bs_layernorm(pre, rows, ln2w, ln2b, a.eps, sx, warp, lane);
    }
    __syncthreads();
    // masked mean pooling and L2 norm: a block takes every CL-th sentence, a thread up to two columns
    __shared__ float tot[kBsThreads / 32];
    for (int s = rank; s < ns; s += CL) {
        float acc[2] = {0.f, 0.f}, cnt = 0.f;
        for (int r = 0; r < a.t; ++r) {
            const float m = a.mask ? (float)a.mask[row0 + (size_t)s * a.t + r] : 1.f;
            cnt += m;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int c = tid + u * kBsThreads;
                if (c < kBsH) acc[u] = fmaf(__uint_as_float((uint32_t)sx[(s * a.t + r) * kBsLdX + c] << 16), m, acc[u]);
            }
        }
        acc[0] /= cnt * (float)kBsH;
        acc[1] /= cnt * (float)kBsH;
        const float sq = warp_sum(acc[0] * acc[0] + acc[1] * acc[1]);
        if (lane == 0) tot[warp] = sq;
        __syncthreads();
        float sum = 0.f;
        for (int k = 0; k < kBsThreads / 32; ++k) sum += tot[k];
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int c = tid + u * kBsThreads;
            if (c < kBsH) a.out[(size_t)(s0 + s) * kBsH + c] = acc[u] / sqrtf(sum);
        }
    }
}
template <int MT, int CL>
constexpr size_t bert_small_smem() { return (size_t)MT * 16 * kBsLdX * 2 + (size_t)4 * MT * 16 * (kBsI / CL + 4) * 4 + (size_t)2 * (4 * kBsH + (5 * kBsH + kBsI) / CL) * 4; }

}  // namespace fl
