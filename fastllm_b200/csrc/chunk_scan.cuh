// The recurrences of the layered decoders over long portions of a prompt (serving precision), 64 tokens at a time.
//
// Token by token a state S of [D, Dv] floats per head is read and written once per token and nothing of token t + 1 can start before
// token t: ly_rec_scan_kernel takes 0.25 to 0.3 us per token and ly_gla_scan_kernel 1 us, however much of the chip is free.  Within a chunk of C = 64 tokens the same sums are products of small matrices, and only the state
// at the chunks' borders is serial:
//   o_i = q_i^T (decay to i) S_0 + sum_{j <= i} (q_i . k_j decayed from j to i) u_j,     S_C = (decay to C) S_0 + sum_j (k_j decayed to C) u_j^T
//   (Yang et al., "Gated linear attention transformers with hardware-efficient training", 2024; the delta rule's u by the WY form of
//   Yang et al., "Parallelizing linear transformers with the delta rule over sequence length", 2024)
// Every product is an f32 FMA chain on f32 operands, as in the token-serial kernels, and every decay is a running product of the tokens'
// own factors (each <= 1: nothing is divided and nothing can overflow).
//   1. ly_chunk_in_kernel / ly_chunk_gla_kernel / ly_chunk_delta_kernel   one block per (chunk, head): everything that needs no state
//   2. ly_chunk_state_kernel / ly_chunk_delta_state_kernel                 the states at the chunks' starts, chunk by chunk
//   3. ly_chunk_out_kernel / ly_chunk_out_heads_kernel                     one block per (chunk, head): what the starting state adds
// Bound: 1 and 3 by latency -- operands in shared memory, 4 x 4 results per thread (64 FMA per 8 16-byte loads), 16 warps per SM:
// at 1024 tokens ncu has the FMA pipe at 24 to 47 %, issue slots at 42 to 60 %, shared memory at 37 to 52 %.  2: HBM.
// Measured per layer, token by token -> chunks, kernel by kernel: gated linear attention, 1531 tokens, 16 heads of 128 x 128: 1575 -> 192 us; Mamba-2, 2048
// tokens, 128 heads of 128 x 64: 772 -> 470 us (four heads per block: their scores are multiplied once); delta rule, 2048 tokens, 32 heads of 128 x 128: 596 -> 576 us,
// 1024 tokens, 16 heads: 304 -> 204; lightning attention, 333 tokens, 16 heads: 89 -> 57 us.  Same model, same tokens: the logits agree to 1e-5 .. 4e-5, their
// error against 64 bits is unchanged.
#pragma once
#include "layered_ops.cuh"

namespace fl {

constexpr int kCsC = 64;                // tokens per chunk
constexpr int kCsSlab = 64;             // value columns at a time
constexpr int kCsPad = 4;               // floats behind a row in shared memory: neighbouring rows start four banks apart
constexpr int kCsLdA = kCsC + kCsPad;   // row stride of a [64][64] operand
constexpr int kCsChunks = 32;           // chunks whose states are held at a time (32 heads of 128 x 128: 67 MB), over all sequences of a step
// Portions from this length on (at least a chunk).  Two layers of the kind alone, whole prefill, us, token by token -> in chunks:
// gated linear attention, one / four portions of 64 and 127 tokens: width 1024 240 -> 231, 366 -> 245 / 322 -> 308, 443 -> 306; 2048 274 -> 268, 402 -> 290 / 382 ->
// 345, 523 -> 367.
// Mamba-2, 160 / 192 / 224 / 255 tokens: one portion of width 1024 301 -> 308, 261 -> 282, 327 -> 293, 410 -> 347; 2048 352 -> 380, 362 -> 361, 411 -> 381, 457 -> 402;
// 4096 499 -> 538, 540 -> 532, 582 -> 562; four portions of 1024 370 -> 410, 410 -> 426, 455 -> 436, 429 -> 448; 2048 572 -> 578, 629 -> 590, 681 -> 603, 729 -> 605;
// 4096 1068 -> 1076, 1163 -> 1109, 1330 -> 1279, 1436 -> 1324.  Lightning (beside attention): 2048 396 -> 418, 421 -> 426, 437 -> 431, 452 -> 437; four 720 -> 738,
// 760 -> 756, 847 -> 820, 901 -> 854.
// Delta rule, 192 / 224 / 255 / 320 tokens: one portion of 1024 364 -> 341, 292 -> 340, 304 -> 333, 389 -> 370; 2048 380 -> 409, 363 -> 403, 445 -> 442, 480 -> 453;
// 4096 467 -> 492, 498 -> 539, 601 -> 556, 622 -> 594; four of 1024 407 -> 422, 446 -> 439, 497 -> 451, 501 -> 479; 2048 523 -> 582, 569 -> 610, 606 -> 618, 709 -> 772;
// 4096 837 -> 1001, 976 -> 1186, 1036 -> 1200, 1377 -> 1632: where serial blocks fill the SMs more than once they stay ahead for longer.
constexpr int kCsMinTokensGla = 64, kCsMinTokensOne = 192, kCsMinTokensDelta = 256;      // (One: one decay per head, no delta rule)

struct ChunkArgs {
    const float* src; int ld, off_q, off_k, off_v;      // q, k [G][D], v [H][Dv] per row
    const float* ab;                // [T, H, 2]: decay, strength (unused by the gated linear attention)
    const float* dskip;             // [H] or nullptr
    const float *z, *zb; float inv_tau, qscale;         // gated linear attention: decay pre-activation [T, H * D], its bias; query scale
    float* o;                       // [T, H * Dv]
    float* state;                   // [slots][H][D][Dv]
    const int *seq_row0, *seq_slot, *seq_pos0;
    int n, H, G, D, Dv;
    int min_tokens;                 // of a portion that goes in chunks
    int span0, span;                // chunks [span0, span0 + span) of every sequence are handled by this round of launches
    float* us;                      // [chunk][H][D][Dv]: what a chunk adds to the state, then the state at its start
    float* dec;                     // [chunk][H]: decay over a chunk ([chunk][H][D] for the gated linear attention)
    float* qd;                      // [T][H * D]: queries decayed from their chunk's start (gated linear attention)
    float* aq;                      // delta: [chunk][H][64][64] (q_i . k_j) decayed
    float* wk;                      // delta: [chunk][H][64][D], what multiplies the starting state in u
};
// chunks of a sequence of `len` tokens in this span
__device__ __forceinline__ int cs_count(const ChunkArgs& a, int len) {
    return len < a.min_tokens ? 0 : max(0, min(a.span, (len + kCsC - 1) / kCsC - a.span0));
}
// chunk number of the launch -> sequence, first row, tokens; false: none
__device__ __forceinline__ bool cs_find(const ChunkArgs& a, int chunk, int& row, int& len) {
    int r0 = a.seq_row0[0];
    for (int s = 0; s < a.n; ++s) {
        const int r1 = a.seq_row0[s + 1], c = cs_count(a, r1 - r0);
        if (chunk < c) {
            row = r0 + (a.span0 + chunk) * kCsC;
            len = min(kCsC, r1 - row);
            return true;
        }
        chunk -= c;
        r0 = r1;
    }
    return false;
}

// ---- products of operands in shared memory, 256 threads, a 64 x 64 result: thread (ty, tx) holds rows ty + 16 r, r < 4 ------------------
__device__ __forceinline__ void cs_thread(int& ty, int& tx) {         // (of 256 threads; a block of 512 makes two results at a time)
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5 & 7;
    ty = (w & 1) * 8 + (lane >> 2);
    tx = (w >> 1) * 4 + (lane & 3);
}
__device__ __forceinline__ void cs_fma4(float (&acc)[4], float x, const float4& y) {
    acc[0] = fmaf(x, y.x, acc[0]); acc[1] = fmaf(x, y.y, acc[1]); acc[2] = fmaf(x, y.z, acc[2]); acc[3] = fmaf(x, y.w, acc[3]);
}
// acc[r][c] += sum_k A[ty + 16 r][k] B[tx + 16 c][k]
template <int K>
__device__ __forceinline__ void cs_mm_nt(float (&acc)[4][4], const float* A, int lda, const float* B, int ldb, int ty, int tx) {
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        float4 x[4], y[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) x[r] = *reinterpret_cast<const float4*>(A + (ty + 16 * r) * lda + k);
#pragma unroll
        for (int c = 0; c < 4; ++c) y[c] = *reinterpret_cast<const float4*>(B + (tx + 16 * c) * ldb + k);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(x[r].x, y[c].x, fmaf(x[r].y, y[c].y, fmaf(x[r].z, y[c].z, fmaf(x[r].w, y[c].w, acc[r][c]))));
    }
}
// acc[r][c] += sum_k A[ty + 16 r][k] B[k][4 tx + c]
template <int K>
__device__ __forceinline__ void cs_mm_nn(float (&acc)[4][4], const float* A, int lda, const float* B, int ldb, int ty, int tx) {
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        float4 x[4], y[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) x[r] = *reinterpret_cast<const float4*>(A + (ty + 16 * r) * lda + k);
#pragma unroll
        for (int i = 0; i < 4; ++i) y[i] = *reinterpret_cast<const float4*>(B + (k + i) * ldb + 4 * tx);
#pragma unroll
        for (int r = 0; r < 4; ++r) { cs_fma4(acc[r], x[r].x, y[0]); cs_fma4(acc[r], x[r].y, y[1]); cs_fma4(acc[r], x[r].z, y[2]); cs_fma4(acc[r], x[r].w, y[3]); }
    }
}
// acc[r][c] += sum_k A[k][m0 + 4 ty + r] B[k][4 tx + c]
template <int K>
__device__ __forceinline__ void cs_mm_tn(float (&acc)[4][4], const float* A, int lda, const float* B, int ldb, int ty, int tx) {
#pragma unroll 4
    for (int k = 0; k < K; ++k) {
        const float4 x = *reinterpret_cast<const float4*>(A + k * lda + 4 * ty), y = *reinterpret_cast<const float4*>(B + k * ldb + 4 * tx);
        cs_fma4(acc[0], x.x, y); cs_fma4(acc[1], x.y, y); cs_fma4(acc[2], x.z, y); cs_fma4(acc[3], x.w, y);
    }
}
__device__ __forceinline__ void cs_zero(float (&acc)[4][4]) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
}
// rows [0, len) x columns [0, D) of src (row stride ld) into dst [64][ldd], times scale; what lies outside is zero
template <int DP, int NT = 256>
__device__ __forceinline__ void cs_load(float* dst, int ldd, const float* src, int ld, int len, int D, float scale) {
    for (int i = threadIdx.x; i < kCsC * (DP / 4); i += NT) {
        const int r = i / (DP / 4), c = i % (DP / 4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < len && c < D) v = *reinterpret_cast<const float4*>(src + (size_t)r * ld + c);
        v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale;
        *reinterpret_cast<float4*>(dst + r * ldd + c) = v;
    }
}
// value columns [v0, v0 + 64), row j times rows[j] (nullptr: 1)
__device__ __forceinline__ void cs_load_slab(float* dst, const float* src, int ld, int len, int v0, int Dv, const float* rows) {
    for (int i = threadIdx.x & 255; i < kCsC * (kCsSlab / 4); i += 256) {
        const int r = i / (kCsSlab / 4), c = i % (kCsSlab / 4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < len && v0 + c < Dv) v = *reinterpret_cast<const float4*>(src + (size_t)r * ld + v0 + c);
        if (rows != nullptr) { const float s = rows[r]; v.x *= s; v.y *= s; v.z *= s; v.w *= s; }
        *reinterpret_cast<float4*>(dst + r * kCsLdA + c) = v;
    }
}
// o (rows [0, len) of the head, columns [v0, v0 + 64)) = A V;  us [D][Dv] = K^T V
template <int DP>
__device__ __forceinline__ void cs_slab_products(const ChunkArgs& a, const float* sA, const float* sK, int ldk, const float* sV, int row, int len, int hd, int v0, float* us, int ty, int tx) {
    float acc[4][4];
    cs_zero(acc);
    cs_mm_nn<kCsC>(acc, sA, kCsLdA, sV, kCsLdA, ty, tx);
    const int col = v0 + 4 * tx;
    if (col < a.Dv) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = ty + 16 * r;
            if (i < len) *reinterpret_cast<float4*>(a.o + (size_t)(row + i) * a.H * a.Dv + hd * a.Dv + col) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        }
    }
#pragma unroll 1
    for (int m0 = 0; m0 < DP; m0 += 64) {
        cs_zero(acc);
        cs_mm_tn<kCsC>(acc, sK + m0, ldk, sV, kCsLdA, ty, tx);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int d = m0 + 4 * ty + r;
            if (d < a.D && col < a.Dv) *reinterpret_cast<float4*>(us + (size_t)d * a.Dv + col) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        }
    }
}
// One decay per head and token: sa[t] = decay of token t (1 behind the portion).  The decay from token j to token i of a thread's results
// (i = ty + 16 r, j = tx + 16 c: block row r, block column c) is (start of i's 16-token block to i) x (the blocks between) x (j to its block's
// end), inside a block the product itself: every factor is <= 1, and no thread multiplies more than 15 of them one after the other.
struct CsDecay {
    float sa[kCsC], pre[kCsC], suf[kCsC], end[kCsC];    // end: j to the chunk's end
    float whole;
};
// between two barriers of the caller: sa is there before, the tables are there behind the next one
__device__ __forceinline__ void cs_decay_tables(CsDecay& d, int t) {       // t: token of the thread
    const int b0 = t & ~15;
    float p = 1.f, q = 1.f, e = 1.f;
    for (int i = b0; i <= t; ++i) p *= d.sa[i];
    for (int i = t + 1; i < b0 + 16; ++i) q *= d.sa[i];
    for (int i = b0 + 16; i < kCsC; ++i) e *= d.sa[i];
    d.pre[t] = p;
    d.suf[t] = q;
    d.end[t] = q * e;
    if (t == 0) d.whole = p * q * e;
}
// factors of the thread's results: zero above the diagonal
__device__ __forceinline__ void cs_decay_factors(float (&f)[4][4], const CsDecay& d, int ty, int tx) {
    float in = 1.f, blk[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) blk[b] = d.pre[16 * b + 15];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (c > r) { f[r][c] = 0.f; continue; }
            if (c == r) {
                in = 1.f;
                for (int i = tx + 1; i <= ty; ++i) in *= d.sa[16 * r + i];
                f[r][c] = tx <= ty ? in : 0.f;
                continue;
            }
            float x = d.pre[16 * r + ty] * d.suf[16 * c + tx];
#pragma unroll
            for (int b = 1; b < 3; ++b)
                if (b > c && b < r) x *= blk[b];
            f[r][c] = x;
        }
}

// ---- lightning attention, Mamba-2: one decay per head and token ---------------------------------------------------------------------
// HB neighbouring heads that read the same q and k (Mamba-2's groups) share a block: their scores differ by the decays alone.  The decays' products of all
// of them are made at the start; a head's values (a slab of 64 columns at a time) are on their way while the slab before is multiplied.
// (Heads one after the other, each with its tables, its loads and two passes over its values: 338 -> 233 us for 2048 tokens of 128 heads of 128 x 64,
// four heads a block; 34 -> 26 for 333 tokens of 16 heads of 128 x 128.)
template <int DP>
constexpr size_t cs_in_smem() { return ((size_t)(kCsC * (DP + kCsPad) > 2 * kCsC * kCsLdA ? kCsC * (DP + kCsPad) : 2 * kCsC * kCsLdA) + kCsC * (DP + kCsPad) + kCsC * kCsLdA) * 4; }
template <int DP, int HB>
static __global__ void __launch_bounds__(256, 2) ly_chunk_in_kernel(ChunkArgs a) {
    pdl_chain();
    extern __shared__ __align__(16) float sm[];
    constexpr int LD = DP + kCsPad, FREE = kCsC * LD > 2 * kCsC * kCsLdA ? kCsC * LD : 2 * kCsC * kCsLdA, B = 16;
    float *sQ = sm, *sK = sQ + FREE, *sA = sK + kCsC * LD;             // two value slabs take the queries' place once they are used
    __shared__ CsDecay dec[HB];
    __shared__ float sb[HB][kCsC], sw[HB][kCsC], sin[HB][kCsC][B];       // strength, strength x decay to the chunk's end, decays inside a 16-token block: [to][from]
    const int h0 = blockIdx.y * HB, g = h0 / (a.H / a.G), tid = threadIdx.x;
    int row, len, ty, tx;
    if (!cs_find(a, blockIdx.x, row, len)) return;
    cs_thread(ty, tx);
    const float* src = a.src + (size_t)row * a.ld;
    cs_load<DP>(sQ, LD, src + a.off_q + g * a.D, a.ld, len, a.D, 1.f);
    cs_load<DP>(sK, LD, src + a.off_k + g * a.D, a.ld, len, a.D, 1.f);
    const int th = tid / kCsC, tt = tid % kCsC;         // the tables: a head per 64 threads
    if (th < HB) {
        const float2 v = tt < len ? *reinterpret_cast<const float2*>(a.ab + ((size_t)(row + tt) * a.H + h0 + th) * 2) : make_float2(1.f, 0.f);
        dec[th].sa[tt] = v.x;
        sb[th][tt] = v.y;
    }
    __syncthreads();
    if (th < HB) {
        cs_decay_tables(dec[th], tt);
        sw[th][tt] = sb[th][tt] * dec[th].end[tt];
        if (tt == 0) a.dec[(size_t)blockIdx.x * a.H + h0 + th] = dec[th].whole;
        float f[B], p = 1.f;
#pragma unroll
        for (int j = 0; j < B; ++j) f[j] = dec[th].sa[(tt & ~15) + j];
#pragma unroll
        for (int j = B - 1; j >= 0; --j) {
            sin[th][tt][j] = j <= (tt & 15) ? p : 0.f;
            if (j <= (tt & 15)) p *= f[j];
        }
    }
    float qk[4][4];
    cs_zero(qk);
    cs_mm_nt<DP>(qk, sQ, LD, sK, LD, ty, tx);
    __syncthreads();                    // the queries are done with, the tables are there
    const int slabs = (a.Dv + kCsSlab - 1) / kCsSlab, items = HB * slabs;
    auto bring = [&](int item) {        // values of rows behind the portion and of columns behind the head are zero
        float* dst = sQ + (item & 1) * kCsC * kCsLdA;
        const float* v = src + a.off_v + (h0 + item / slabs) * a.Dv;
        const int v0 = item % slabs * kCsSlab;
        for (int i = tid; i < kCsC * (kCsSlab / 4); i += 256) {
            const int r = i / (kCsSlab / 4), c = i % (kCsSlab / 4) * 4;
            if (r < len && v0 + c < a.Dv) cp_async16(dst + r * kCsLdA + c, v + (size_t)r * a.ld + v0 + c);
            else *reinterpret_cast<float4*>(dst + r * kCsLdA + c) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        cp_async_commit();
    };
    bring(0);
#pragma unroll 1
    for (int item = 0; item < items; ++item) {
        const int hh = item / slabs, hd = h0 + hh, v0 = item % slabs * kCsSlab;
        if (item + 1 < items) bring(item + 1);
        else cp_async_commit();
        if (v0 == 0) {                  // scores of the head: decayed, times the keys' strengths
            const CsDecay& d = dec[hh];
            float blk[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) blk[k] = d.pre[16 * k + 15];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float f = 0.f;
                    if (c == r) f = sin[hh][16 * r + ty][tx];
                    if (c < r) {
                        f = d.pre[16 * r + ty] * d.suf[16 * c + tx];
#pragma unroll
                        for (int k = 1; k < 3; ++k)
                            if (k > c && k < r) f *= blk[k];
                    }
                    sA[(ty + 16 * r) * kCsLdA + tx + 16 * c] = qk[r][c] * f * sb[hh][tx + 16 * c];
                }
        }
        cp_async_wait<1>();
        __syncthreads();
        const float* sV = sQ + (item & 1) * kCsC * kCsLdA;
        const float dsk = a.dskip ? a.dskip[hd] : 0.f;
        float* us = a.us + ((size_t)blockIdx.x * a.H + hd) * a.D * a.Dv;
        const int col = v0 + 4 * tx;
        {
            float acc[4][4];
            cs_zero(acc);
            cs_mm_nn<kCsC>(acc, sA, kCsLdA, sV, kCsLdA, ty, tx);
            if (col < a.Dv) {
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int i = ty + 16 * r;
                    if (i >= len) continue;
                    const float4 x = *reinterpret_cast<const float4*>(sV + i * kCsLdA + 4 * tx);
                    *reinterpret_cast<float4*>(a.o + (size_t)(row + i) * a.H * a.Dv + hd * a.Dv + col) =
                        dsk != 0.f ? make_float4(fmaf(dsk, x.x, acc[r][0]), fmaf(dsk, x.y, acc[r][1]), fmaf(dsk, x.z, acc[r][2]), fmaf(dsk, x.w, acc[r][3]))
                                   : make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
                }
            }
        }
        {   // what the chunk adds to the state: K^T (strength x decay x V), all key channels in one walk over the tokens
            constexpr int MB = DP / 64;
            float acc[MB][4][4];
#pragma unroll
            for (int m = 0; m < MB; ++m) cs_zero(acc[m]);
#pragma unroll 4
            for (int k = 0; k < kCsC; ++k) {
                const float s = sw[hh][k];
                float4 y = *reinterpret_cast<const float4*>(sV + k * kCsLdA + 4 * tx);
                y.x *= s; y.y *= s; y.z *= s; y.w *= s;
#pragma unroll
                for (int m = 0; m < MB; ++m) {
                    const float4 x = *reinterpret_cast<const float4*>(sK + k * LD + 64 * m + 4 * ty);
                    cs_fma4(acc[m][0], x.x, y); cs_fma4(acc[m][1], x.y, y); cs_fma4(acc[m][2], x.z, y); cs_fma4(acc[m][3], x.w, y);
                }
            }
#pragma unroll
            for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int d = 64 * m + 4 * ty + r;
                    if (d < a.D && col < a.Dv) *reinterpret_cast<float4*>(us + (size_t)d * a.Dv + col) = make_float4(acc[m][r][0], acc[m][r][1], acc[m][r][2], acc[m][r][3]);
                }
        }
        __syncthreads();                // the slab and the scores have been read
    }
}

// ---- gated linear attention: one decay per head, token and key channel ---------------------------------------------------------------
// The chunk's score matrix in 16 x 16 blocks: on the diagonal each pair's decay is the running product itself; below it the query is
// decayed from its block's start, the key to the end of the block before that, so every factor stays <= 1.
// One block fits an SM: sixteen warps, each half of the block with a slab of values of its own.  (Eight warps, and a reduction over the warp per pair of
// the diagonal blocks: 209 -> 125 us for 1531 tokens of 16 heads of 128 x 128.)
constexpr int kCsGlaThreads = 512;
template <int DP>
constexpr size_t cs_gla_smem() { return ((size_t)2 * kCsC * (DP + kCsPad) + (kCsC * (DP + kCsPad) > 2 * kCsC * kCsLdA ? kCsC * (DP + kCsPad) : 2 * kCsC * kCsLdA) + kCsC * kCsLdA + kCsC / 16 * DP) * 4; }
template <int DP>
static __global__ void __launch_bounds__(kCsGlaThreads, 1) ly_chunk_gla_kernel(ChunkArgs a) {
    pdl_chain();
    extern __shared__ __align__(16) float sm[];
    constexpr int LD = DP + kCsPad, B = 16, NB = kCsC / B, NT = kCsGlaThreads, FREE = kCsC * LD > 2 * kCsC * kCsLdA ? kCsC * LD : 2 * kCsC * kCsLdA;
    float *sQ = sm, *sK = sQ + kCsC * LD, *sF = sK + kCsC * LD, *sA = sF + FREE, *sB = sA + kCsC * kCsLdA;    // sF: the tokens' decays, then two value slabs
    const int hd = blockIdx.y, tid = threadIdx.x, lane = tid & 31, w = tid >> 5, D = a.D;
    int row, len, ty, tx;
    if (!cs_find(a, blockIdx.x, row, len)) return;
    cs_thread(ty, tx);
    const float* src = a.src + (size_t)row * a.ld;
    cs_load<DP, NT>(sQ, LD, src + a.off_q + hd * D, a.ld, len, D, a.qscale);
    cs_load<DP, NT>(sK, LD, src + a.off_k + hd * D, a.ld, len, D, 1.f);
    for (int i = tid; i < kCsC * DP; i += NT) {
        const int t = i / DP, d = i % DP;
        float f = 1.f;
        if (t < len && d < D) {         // alpha = sigmoid(z)^(1/tau), as the token-serial kernel evaluates it
            const float z = a.z[(size_t)(row + t) * a.H * D + hd * D + d] + a.zb[hd * D + d];
            f = expf(-(fmaxf(-z, 0.f) + log1pf(expf(-fabsf(z)))) * a.inv_tau);
        }
        sF[t * LD + d] = f;
    }
    for (int i = tid; i < kCsC * kCsLdA; i += NT) sA[i] = 0.f;
    __syncthreads();
    // diagonal blocks: a warp takes a key, its lanes four channels each; the sums over the lanes for all of the block's queries at once
    for (int j = w; j < kCsC; j += NT / 32) {
        const bool on = lane * 4 < DP;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 p = on ? *reinterpret_cast<const float4*>(sK + j * LD + lane * 4) : zero;
        const int b0 = j / B * B;
        float s[B];
#pragma unroll
        for (int e = 0; e < B; ++e) {
            const int i = b0 + e;
            s[e] = 0.f;
            if (i >= j && on) {
                if (i > j) {
                    const float4 f = *reinterpret_cast<const float4*>(sF + i * LD + lane * 4);
                    p.x *= f.x; p.y *= f.y; p.z *= f.z; p.w *= f.w;
                }
                const float4 q = *reinterpret_cast<const float4*>(sQ + i * LD + lane * 4);
                s[e] = fmaf(q.x, p.x, fmaf(q.y, p.y, fmaf(q.z, p.z, q.w * p.w)));
            }
        }
#pragma unroll
        for (int o = 16, n = B / 2; n > 0; o >>= 1, n >>= 1)        // a lane keeps half of its sums, sends the other half: sum lane / 2 is left
#pragma unroll
            for (int e = 0; e < n; ++e) {
                const bool up = lane & o;
                const float keep = up ? s[e + n] : s[e], send = up ? s[e] : s[e + n];
                s[e] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, o);
            }
        const float t = s[0] + __shfl_xor_sync(0xFFFFFFFFu, s[0], 1);
        if ((lane & 1) == 0 && b0 + lane / 2 >= j) sA[(b0 + lane / 2) * kCsLdA + j] = t;
    }
    __syncthreads();
    // queries decayed from their block's start, keys to their block's end, the blocks' whole decays
    for (int r = tid; r < 2 * NB * DP; r += NT) {
        const int d = r % DP, b = r / DP % NB;
        float f[B], x[B];
        float* v = (r < NB * DP ? sQ : sK) + b * B * LD + d;
#pragma unroll
        for (int i = 0; i < B; ++i) { f[i] = sF[(b * B + i) * LD + d]; x[i] = v[i * LD]; }
        float run = 1.f;
        if (r < NB * DP) {
#pragma unroll
            for (int i = 0; i < B; ++i) { run *= f[i]; v[i * LD] = x[i] * run; }
            sB[b * DP + d] = run;
        } else {
#pragma unroll
            for (int i = B - 1; i >= 0; --i) { v[i * LD] = x[i] * run; run *= f[i]; }
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int b = 1; b <= NB; ++b) {     // keys of the blocks before b, decayed to the end of block b - 1
        for (int i = tid; i < (b - 1) * B * DP; i += NT) sK[i / DP * LD + i % DP] *= sB[(b - 1) * DP + i % DP];
        __syncthreads();
        if (b == NB) break;
        for (int p = tid; p < B * b * B; p += NT) {        // 16 queries x 16 b keys; a warp: 8 keys x 4 queries
            const int i = b * B + (p / 32 % 4) * 4 + (p & 3), j = p / 128 * 8 + (p >> 2 & 7);
            float s = 0.f;
#pragma unroll 4
            for (int k = 0; k < DP; k += 4) {
                const float4 x = *reinterpret_cast<const float4*>(sQ + i * LD + k), y = *reinterpret_cast<const float4*>(sK + j * LD + k);
                s = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, s))));
            }
            sA[i * kCsLdA + j] = s;
        }
        __syncthreads();
    }
    // queries decayed from the chunk's start, for the part that the starting state adds
    for (int i = tid; i < kCsC * DP; i += NT) {
        const int t = i / DP, d = i % DP;
        if (t >= len || d >= D) continue;
        float q = sQ[t * LD + d];
        for (int b = 0; b < t / B; ++b) q *= sB[b * DP + d];
        a.qd[(size_t)(row + t) * a.H * D + hd * D + d] = q;
    }
    for (int d = tid; d < D; d += NT) {
        float p = 1.f;
        for (int b = 0; b < NB; ++b) p *= sB[b * DP + d];
        a.dec[((size_t)blockIdx.x * a.H + hd) * D + d] = p;
    }
    float* us = a.us + ((size_t)blockIdx.x * a.H + hd) * D * a.Dv;
    const int half = tid >> 8;
    float* sV = sF + half * kCsC * kCsLdA;
    for (int vb = 0; vb < a.Dv; vb += 2 * kCsSlab) {
        const int v0 = vb + half * kCsSlab;
        if (v0 < a.Dv) cs_load_slab(sV, src + a.off_v + hd * a.Dv, a.ld, len, v0, a.Dv, nullptr);
        __syncthreads();
        if (v0 < a.Dv) cs_slab_products<DP>(a, sA, sK, LD, sV, row, len, hd, v0, us, ty, tx);
        __syncthreads();
    }
}

// ---- the states at the chunks' starts -------------------------------------------------------------------------------------------------
// us[chunk] <- S at the chunk's start; S <- dec[chunk] S + (what us[chunk] held).  Four state elements per thread, the next chunk's
// addition on its way.  grid (H D Dv / 1024, sequences)
static __global__ void __launch_bounds__(256) ly_chunk_state_kernel(ChunkArgs a, int dec_rows) {
    pdl_chain();
    const int seq = blockIdx.y;
    int r0 = a.seq_row0[0], c0 = 0, cnt = 0, tokens = 0;
    for (int s = 0; s <= seq; ++s) {
        const int r1 = a.seq_row0[s + 1];
        c0 += cnt;
        tokens = r1 - r0;
        cnt = cs_count(a, tokens);
        r0 = r1;
    }
    const size_t per = (size_t)a.H * a.D * a.Dv, e = ((size_t)blockIdx.x * 256 + threadIdx.x) * 4;
    if (cnt == 0 || e >= per) return;
    const int dd = (int)(e / a.Dv);                 // head * D + state row
    const size_t ds = dec_rows ? (size_t)a.H * a.D : (size_t)a.H, di = dec_rows ? dd : dd / a.D;
    float* st = a.state + (size_t)a.seq_slot[seq] * per + e;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.span0 > 0 || a.seq_pos0[seq] != 0) s = *reinterpret_cast<const float4*>(st);
    float* u = a.us + (size_t)c0 * per + e;
    const float* dec = a.dec + (size_t)c0 * ds + di;
    float4 next = *reinterpret_cast<const float4*>(u);
    float fnext = dec[0];
    for (int c = 0; c < cnt; ++c, u += per) {
        const float4 add = next;
        const float f = fnext;
        if (c + 1 < cnt) { next = *reinterpret_cast<const float4*>(u + per); fnext = dec[(size_t)(c + 1) * ds]; }
        *reinterpret_cast<float4*>(u) = s;
        s.x = fmaf(s.x, f, add.x); s.y = fmaf(s.y, f, add.y); s.z = fmaf(s.z, f, add.z); s.w = fmaf(s.w, f, add.w);
    }
    *reinterpret_cast<float4*>(st) = s;
}

// ---- what the starting state adds: o += (decayed q) S ----------------------------------------------------------------------------------
// One decay per head, HB heads of a block that read the same q: their states (64 columns at a time) and what o holds are on their way while the ones
// before are multiplied: 206 -> 152 us for 2048 tokens of 128 heads of
// 128 x 64, four heads a block.
template <int DP>
constexpr size_t cs_out_smem() { return ((size_t)kCsC * (DP + kCsPad) + 2 * DP * kCsLdA) * 4; }
template <int DP, int HB>
static __global__ void __launch_bounds__(256, 2) ly_chunk_out_heads_kernel(ChunkArgs a) {
    pdl_chain();
    extern __shared__ __align__(16) float sm[];
    constexpr int LD = DP + kCsPad;
    float *sQ = sm, *sS = sQ + kCsC * LD;               // two state slabs
    __shared__ float sa[HB][kCsC], pre[HB][kCsC], sp[HB][kCsC];          // decays; their products from the start of 16 tokens, of the chunk
    const int h0 = blockIdx.y * HB, g = h0 / (a.H / a.G), tid = threadIdx.x;
    int row, len, ty, tx;
    if (!cs_find(a, blockIdx.x, row, len)) return;
    cs_thread(ty, tx);
    const int slabs = (a.Dv + kCsSlab - 1) / kCsSlab, items = HB * slabs;
    auto bring = [&](int item) {
        float* dst = sS + (item & 1) * DP * kCsLdA;
        const float* S = a.us + ((size_t)blockIdx.x * a.H + h0 + item / slabs) * a.D * a.Dv;
        const int v0 = item % slabs * kCsSlab;
        for (int i = tid; i < DP * (kCsSlab / 4); i += 256) {
            const int d = i / (kCsSlab / 4), c = i % (kCsSlab / 4) * 4;
            if (d < a.D && v0 + c < a.Dv) cp_async16(dst + d * kCsLdA + c, S + (size_t)d * a.Dv + v0 + c);
            else *reinterpret_cast<float4*>(dst + d * kCsLdA + c) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        cp_async_commit();
    };
    bring(0);
    cs_load<DP>(sQ, LD, a.src + (size_t)row * a.ld + a.off_q + g * a.D, a.ld, len, a.D, 1.f);
    const int th = tid / kCsC, tt = tid % kCsC;
    if (th < HB) sa[th][tt] = tt < len ? a.ab[((size_t)(row + tt) * a.H + h0 + th) * 2] : 1.f;
    __syncthreads();
    if (th < HB) {
        float p = 1.f;
        for (int i = tt & ~15; i <= tt; ++i) p *= sa[th][i];
        pre[th][tt] = p;
    }
    __syncthreads();
    if (th < HB) {
        float p = pre[th][tt];
        for (int k = 0; k < tt / 16; ++k) p *= pre[th][16 * k + 15];
        sp[th][tt] = p;
    }
#pragma unroll 1
    for (int item = 0; item < items; ++item) {
        const int hh = item / slabs, col = item % slabs * kCsSlab + 4 * tx;
        float* op = a.o + (size_t)row * a.H * a.Dv + (h0 + hh) * a.Dv + col;
        if (item + 1 < items) bring(item + 1);
        else cp_async_commit();
        float4 x[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) x[r] = col < a.Dv && ty + 16 * r < len ? *reinterpret_cast<const float4*>(op + (size_t)(ty + 16 * r) * a.H * a.Dv) : make_float4(0.f, 0.f, 0.f, 0.f);
        cp_async_wait<1>();
        __syncthreads();
        float acc[4][4];
        cs_zero(acc);
        cs_mm_nn<DP>(acc, sQ, LD, sS + (item & 1) * DP * kCsLdA, kCsLdA, ty, tx);
        if (col < a.Dv) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int i = ty + 16 * r;
                const float p = sp[hh][i];
                if (i < len) *reinterpret_cast<float4*>(op + (size_t)i * a.H * a.Dv) = make_float4(acc[r][0] * p + x[r].x, acc[r][1] * p + x[r].y, acc[r][2] * p + x[r].z, acc[r][3] * p + x[r].w);
            }
        }
        __syncthreads();                // the slab has been read
    }
}
// MODE 1: gated linear attention (q from qd); 2: delta rule (q from src, decayed here) -- o holds u on entry, o = A u + (decayed q) S with A from aq.
template <int DP, int MODE>
static __global__ void __launch_bounds__(256, 2) ly_chunk_out_kernel(ChunkArgs a) {
    pdl_chain();
    extern __shared__ __align__(16) float sm[];
    constexpr int LD = DP + kCsPad;
    float *sQ = sm, *sS = sQ + kCsC * LD, *sA = sS + DP * kCsLdA, *sU = sA + kCsC * kCsLdA;      // sA, sU: MODE 2 alone
    __shared__ float sa[kCsC], sp[kCsC];
    const int hd = blockIdx.y, g = hd / (a.H / a.G), tid = threadIdx.x;
    int row, len, ty, tx;
    if (!cs_find(a, blockIdx.x, row, len)) return;
    cs_thread(ty, tx);
    if (MODE == 1) {
        cs_load<DP>(sQ, LD, a.qd + (size_t)row * a.H * a.D + hd * a.D, a.H * a.D, len, a.D, 1.f);
    } else {
        cs_load<DP>(sQ, LD, a.src + (size_t)row * a.ld + a.off_q + g * a.D, a.ld, len, a.D, 1.f);
        if (tid < kCsC) sa[tid] = tid < len ? a.ab[((size_t)(row + tid) * a.H + hd) * 2] : 1.f;
        __syncthreads();
        if (tid < kCsC) {
            float p = 1.f;
            for (int i = 0; i <= tid; ++i) p *= sa[i];
            sp[tid] = p;
        }
    }
    if (MODE == 2) {
        const float* aq = a.aq + ((size_t)blockIdx.x * a.H + hd) * kCsC * kCsC;
        for (int i = tid; i < kCsC * kCsC / 4; i += 256)
            *reinterpret_cast<float4*>(sA + i / (kCsC / 4) * kCsLdA + i % (kCsC / 4) * 4) = *reinterpret_cast<const float4*>(aq + i * 4);
    }
    const float* S = a.us + ((size_t)blockIdx.x * a.H + hd) * a.D * a.Dv;
    for (int v0 = 0; v0 < a.Dv; v0 += kCsSlab) {
        __syncthreads();
        for (int i = tid; i < DP * (kCsSlab / 4); i += 256) {
            const int d = i / (kCsSlab / 4), c = i % (kCsSlab / 4) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (d < a.D && v0 + c < a.Dv) v = *reinterpret_cast<const float4*>(S + (size_t)d * a.Dv + v0 + c);
            *reinterpret_cast<float4*>(sS + d * kCsLdA + c) = v;
        }
        if (MODE == 2) cs_load_slab(sU, a.o + (size_t)row * a.H * a.Dv + hd * a.Dv, a.H * a.Dv, len, v0, a.Dv, nullptr);
        __syncthreads();
        float acc[4][4];
        cs_zero(acc);
        cs_mm_nn<DP>(acc, sQ, LD, sS, kCsLdA, ty, tx);
        if (MODE == 2) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float p = sp[ty + 16 * r];
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[r][c] *= p;
            }
        }
        if (MODE == 2) cs_mm_nn<kCsC>(acc, sA, kCsLdA, sU, kCsLdA, ty, tx);
        const int col = v0 + 4 * tx;
        if (col < a.Dv) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int i = ty + 16 * r;
                if (i >= len) continue;
                float4* op = reinterpret_cast<float4*>(a.o + (size_t)(row + i) * a.H * a.Dv + hd * a.Dv + col);
                float4 v = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
                if (MODE == 1) { const float4 x = *op; v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w; }
                *op = v;
            }
        }
    }
}

// ---- gated delta rule -------------------------------------------------------------------------------------------------------------------
// u_i = b_i (v_i - (decay to i) S_0^T k_i - sum_{j < i} (decay from j to i) (k_i . k_j) u_j): with M the strictly lower matrix
// b_i (k_i . k_j) (decay from j to i) and T = (I + M)^-1, u = T (b v) - T (b (decay to i) k) S_0.  This kernel leaves T (b v) in o and the
// matrix in front of S_0 in wk, and the decayed (q_i . k_j) in aq.  T is built from its 16 x 16 diagonal blocks, by substitution.
template <int DP>
static __global__ void __launch_bounds__(256) ly_chunk_delta_kernel(ChunkArgs a) {
    pdl_chain();
    extern __shared__ __align__(16) float sm[];
    constexpr int LD = DP + kCsPad, B = 16, NB = kCsC / B;
    float *sQ = sm, *sK = sQ + kCsC * LD, *sM = sK + kCsC * LD, *sT = sM + kCsC * kCsLdA;       // the value slab takes the queries' place
    __shared__ CsDecay dec;
    __shared__ float sb[kCsC], sp[kCsC];
    const int hd = blockIdx.y, g = hd / (a.H / a.G), tid = threadIdx.x;
    int row, len, ty, tx;
    if (!cs_find(a, blockIdx.x, row, len)) return;
    cs_thread(ty, tx);
    const float* src = a.src + (size_t)row * a.ld;
    cs_load<DP>(sQ, LD, src + a.off_q + g * a.D, a.ld, len, a.D, 1.f);
    cs_load<DP>(sK, LD, src + a.off_k + g * a.D, a.ld, len, a.D, 1.f);
    if (tid < kCsC) {
        dec.sa[tid] = tid < len ? a.ab[((size_t)(row + tid) * a.H + hd) * 2] : 1.f;
        sb[tid] = tid < len ? a.ab[((size_t)(row + tid) * a.H + hd) * 2 + 1] : 0.f;
    }
    __syncthreads();
    if (tid < kCsC) cs_decay_tables(dec, tid);
    for (int i = tid; i < kCsC * kCsLdA; i += 256) sT[i] = 0.f;
    float acc[4][4], kk[4][4], f[4][4];
    cs_zero(acc);
    cs_mm_nt<DP>(acc, sQ, LD, sK, LD, ty, tx);
    cs_zero(kk);
    cs_mm_nt<DP>(kk, sK, LD, sK, LD, ty, tx);
    __syncthreads();
    if (tid < kCsC) {                   // decay from the chunk's start
        float p = dec.pre[tid];
        for (int b = 0; b < tid / 16; ++b) p *= dec.pre[16 * b + 15];
        sp[tid] = p;
    }
    cs_decay_factors(f, dec, ty, tx);
    float* aq = a.aq + ((size_t)blockIdx.x * a.H + hd) * kCsC * kCsC;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int i = ty + 16 * r, j = tx + 16 * c;
            aq[i * kCsC + j] = acc[r][c] * f[r][c];
            sM[i * kCsLdA + j] = i > j ? kk[r][c] * sb[i] * f[r][c] : 0.f;
        }
    __syncthreads();
    // diagonal blocks of T: one thread per column, x_i = [i == c] - sum_{j < i} M_ij x_j
    if (tid < kCsC) {
        const int b0 = tid / B * B, c = tid % B;
        float x[B];
#pragma unroll
        for (int i = 0; i < B; ++i) {
            float s = i == c ? 1.f : 0.f;
#pragma unroll
            for (int j = 0; j < i; ++j) s = fmaf(-sM[(b0 + i) * kCsLdA + b0 + j], x[j], s);
            x[i] = s;
            sT[(b0 + i) * kCsLdA + b0 + c] = s;
        }
    }
    __syncthreads();
    // below the diagonal, one block diagonal after the other: T_IJ = -T_II sum_{J <= L < I} M_IL T_LJ (the inner sum parked above the diagonal)
    const int br = tid / B, bc = tid % B;
#pragma unroll 1
    for (int off = 1; off < NB; ++off) {
        for (int J = 0; J + off < NB; ++J) {
            const int I = J + off;
            float s = 0.f;
            for (int l = J * B; l < I * B; ++l) s = fmaf(sM[(I * B + br) * kCsLdA + l], sT[l * kCsLdA + J * B + bc], s);
            sT[(J * B + br) * kCsLdA + I * B + bc] = s;
        }
        __syncthreads();
        for (int J = 0; J + off < NB; ++J) {
            const int I = J + off;
            float s = 0.f;
#pragma unroll
            for (int l = 0; l < B; ++l) s = fmaf(sT[(I * B + br) * kCsLdA + I * B + l], sT[(J * B + l) * kCsLdA + I * B + bc], s);
            sT[(I * B + br) * kCsLdA + J * B + bc] = -s;
        }
        __syncthreads();
    }
    for (int i = tid; i < kCsC * kCsC; i += 256) {
        const int r = i / kCsC, c = i % kCsC;
        if (c / B > r / B) sT[r * kCsLdA + c] = 0.f;
    }
    // T (b v), slab by slab
    for (int v0 = 0; v0 < a.Dv; v0 += kCsSlab) {
        __syncthreads();
        cs_load_slab(sQ, src + a.off_v + hd * a.Dv, a.ld, len, v0, a.Dv, sb);
        __syncthreads();
        cs_zero(acc);
        cs_mm_nn<kCsC>(acc, sT, kCsLdA, sQ, kCsLdA, ty, tx);
        const int col = v0 + 4 * tx;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = ty + 16 * r;
            if (i < len && col < a.Dv)
                *reinterpret_cast<float4*>(a.o + (size_t)(row + i) * a.H * a.Dv + hd * a.Dv + col) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        }
    }
    // T (b (decay to i) k)
    for (int i = tid; i < kCsC * DP; i += 256) sK[i / DP * LD + i % DP] *= sb[i / DP] * sp[i / DP];
    __syncthreads();
    float* wk = a.wk + ((size_t)blockIdx.x * a.H + hd) * kCsC * a.D;
#pragma unroll 1
    for (int m0 = 0; m0 < DP; m0 += 64) {
        cs_zero(acc);
        cs_mm_nn<kCsC>(acc, sT, kCsLdA, sK + m0, LD, ty, tx);
        const int d = m0 + 4 * tx;
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (d < a.D) *reinterpret_cast<float4*>(wk + (ty + 16 * r) * a.D + d) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
    }
}
// The delta rule's states, chunk by chunk: u -= wk S (in o), us[chunk] = S, S <- (decay over the chunk) S + sum_j (k_j decayed to the end) u_j^T.
// One block per (32 value columns, head, sequence) with its columns of S in shared memory; the next chunk's operands arrive while this one is
// multiplied.
constexpr int kCsCols = 32;
template <int DP>
static __global__ void __launch_bounds__(256) ly_chunk_delta_state_kernel(ChunkArgs a) {
    pdl_chain();
    extern __shared__ __align__(16) float sm[];
    constexpr int LD = DP + kCsPad, LC = kCsCols + kCsPad, STAGE = 2 * kCsC * LD + kCsC * LC + kCsC;
    float* sS = sm;                                 // [DP][LC]
    float* stage = sS + DP * LC;                    // two of [wk 64 x LD | k 64 x LD | u 64 x LC | decay 64]
    const int seq = blockIdx.z, hd = blockIdx.y, g = hd / (a.H / a.G), v0 = blockIdx.x * kCsCols, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int r0 = a.seq_row0[0], r1 = r0, c0 = 0, cnt = 0;
    for (int s = 0; s <= seq; ++s) {
        r0 = r1;
        r1 = a.seq_row0[s + 1];
        c0 += cnt;
        cnt = cs_count(a, r1 - r0);
    }
    if (cnt == 0) return;
    const int D = a.D, Dv = a.Dv;
    float* st = a.state + ((size_t)a.seq_slot[seq] * a.H + hd) * D * Dv + v0;
    const bool fresh = a.span0 == 0 && a.seq_pos0[seq] == 0;
    for (int i = tid; i < DP * kCsCols; i += 256) {
        const int d = i / kCsCols, c = i % kCsCols;
        sS[d * LC + c] = (!fresh && d < D && v0 + c < Dv) ? st[(size_t)d * Dv + c] : 0.f;
    }
    for (int i = tid; i < 2 * STAGE; i += 256) stage[i] = 0.f;          // what no copy writes reads as zero
    __syncthreads();
    auto issue = [&](int c) {
        float *sw = stage + (c & 1) * STAGE, *sk = sw + kCsC * LD, *su = sk + kCsC * LD, *sd = su + kCsC * LC;
        const int row = r0 + (a.span0 + c) * kCsC, len = min(kCsC, r1 - row);
        const float* wk = a.wk + ((size_t)(c0 + c) * a.H + hd) * kCsC * D;
        for (int i = tid; i < kCsC * (DP / 4); i += 256) {
            const int r = i / (DP / 4), d = i % (DP / 4) * 4;
            if (d >= D) continue;
            cp_async16(sw + r * LD + d, wk + r * D + d);
            if (r < len) cp_async16(sk + r * LD + d, a.src + (size_t)(row + r) * a.ld + a.off_k + g * D + d);
            else *reinterpret_cast<float4*>(sk + r * LD + d) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        for (int i = tid; i < kCsC * (kCsCols / 4); i += 256) {
            const int r = i / (kCsCols / 4), x = i % (kCsCols / 4) * 4;
            if (r < len && v0 + x < Dv) cp_async16(su + r * LC + x, a.o + (size_t)(row + r) * a.H * Dv + hd * Dv + v0 + x);
            else *reinterpret_cast<float4*>(su + r * LC + x) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (tid < kCsC) {
            if (tid < len) cp_async_f32(sd + tid, a.ab + ((size_t)(row + tid) * a.H + hd) * 2);
            else sd[tid] = 1.f;
        }
    };
    issue(0);
    cp_async_commit();
    __shared__ float se[kCsC + 1];
    for (int c = 0; c < cnt; ++c) {
        if (c + 1 < cnt) issue(c + 1);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        float *sw = stage + (c & 1) * STAGE, *sk = sw + kCsC * LD, *su = sk + kCsC * LD, *sd = su + kCsC * LC;
        const int row = r0 + (a.span0 + c) * kCsC, len = min(kCsC, r1 - row);
        if (tid <= kCsC) {              // decay from token tid - 1 to the chunk's end; [0]: over the whole chunk
            float p = 1.f;
            for (int i = tid; i < kCsC; ++i) p *= sd[i];
            se[tid] = p;
        }
        // u = T(b v) - wk S: thread = two rows x four columns
        const int ur = (w * 4 + (lane >> 3)) * 2, uc = (lane & 7) * 4;
        float x[2][4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float4 v = *reinterpret_cast<const float4*>(su + (ur + r) * LC + uc);
            x[r][0] = -v.x; x[r][1] = -v.y; x[r][2] = -v.z; x[r][3] = -v.w;
        }
#pragma unroll 4
        for (int k = 0; k < DP; k += 4) {
            float4 y[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) y[i] = *reinterpret_cast<const float4*>(sS + (k + i) * LC + uc);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float4 m = *reinterpret_cast<const float4*>(sw + (ur + r) * LD + k);
                cs_fma4(x[r], m.x, y[0]); cs_fma4(x[r], m.y, y[1]); cs_fma4(x[r], m.z, y[2]); cs_fma4(x[r], m.w, y[3]);
            }
        }
        __syncthreads();                // se is there; nobody reads the old u any more
        float* us = a.us + ((size_t)(c0 + c) * a.H + hd) * D * Dv + v0;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float4 v = make_float4(-x[r][0], -x[r][1], -x[r][2], -x[r][3]);
            if (ur + r < len && v0 + uc < Dv) *reinterpret_cast<float4*>(a.o + (size_t)(row + ur + r) * a.H * Dv + hd * Dv + v0 + uc) = v;
            const float f = se[ur + r + 1];         // the state takes u decayed to the chunk's end
            *reinterpret_cast<float4*>(su + (ur + r) * LC + uc) = make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
        }
        __syncthreads();
        // S <- decay S + K^T u: thread = DP / 32 rows x four columns
        constexpr int RPT = DP / 32;
        const int sr = (w * 4 + (lane >> 3)) * RPT;
        const float all = se[0];
        float s[RPT][4];
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            const float4 v = *reinterpret_cast<const float4*>(sS + (sr + r) * LC + uc);
            if (sr + r < D && v0 + uc < Dv) *reinterpret_cast<float4*>(us + (size_t)(sr + r) * Dv + uc) = v;
            s[r][0] = v.x * all; s[r][1] = v.y * all; s[r][2] = v.z * all; s[r][3] = v.w * all;
        }
#pragma unroll 4
        for (int j = 0; j < kCsC; ++j) {
            const float4 u = *reinterpret_cast<const float4*>(su + j * LC + uc);
            float k[RPT];
            if (RPT == 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(sk + j * LD + sr);
                k[0] = k4.x; k[1] = k4.y; k[RPT - 2] = k4.z; k[RPT - 1] = k4.w;
            } else {
                const float2 k2 = *reinterpret_cast<const float2*>(sk + j * LD + sr);
                k[0] = k2.x; k[1] = k2.y;
            }
#pragma unroll
            for (int r = 0; r < RPT; ++r) cs_fma4(s[r], k[r], u);
        }
#pragma unroll
        for (int r = 0; r < RPT; ++r) *reinterpret_cast<float4*>(sS + (sr + r) * LC + uc) = make_float4(s[r][0], s[r][1], s[r][2], s[r][3]);
        __syncthreads();
    }
    for (int i = tid; i < DP * kCsCols; i += 256) {
        const int d = i / kCsCols, c = i % kCsCols;
        if (d < D && v0 + c < Dv) st[(size_t)d * Dv + c] = sS[d * LC + c];
    }
}

}  // namespace fl
