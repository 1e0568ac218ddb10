// The exact mode's GEMM (sm_100a): Y[p, n] = sum_k A[row(p), k] * W[n, k], A f32, W bf16 bit patterns, f64 sums, every output the rounded f32 of its
// dot product, whatever K.  Arguments as LyGemm's (layered_ops.cuh).
//
// The f64 tensor pipe (mma.m8n8k4, 64 FMA per clock and SM) bounds it.  K is dealt in chunks of 16 columns to eight sums, chunk c to sum c % 8; the
// eight are added in order at the end.  That order depends on K alone, so a row's result is bitwise the same whatever rows stand beside it and
// whichever form was taken.  A warp holds one of the sums of all BM x 32 outputs of a tile, and nothing of what it reads is read by another
// warp: it has a ring of its own (cp.async, no barrier of the block before the end), operands lie there as they come -- f32 and bf16 -- and are
// widened in registers.  A lane's 16 bytes of a row are its columns of four products (product s takes columns {4 q + s}), so rows of 64 and
// 32 bytes need no padding against bank conflicts.
//
// Measured alone (us, 8 or 16 rows a tile as f64_rows_per_tile has it; before: blocks of 32 x 32 outputs whose operands went through shared memory as
// doubles behind a barrier per 64 columns, 8 x 64 for few rows; the pipe's rate): 203 x 1024 x 2816 66 -> 45 (32), 203 x 5632 x 1024 124 -> 87 (64),
// 17 x 1024 x 2816 56 -> 13, 8 x 32000 x 1024 93 -> 29 (14), 1 x 512 x 512 13 -> 5.  What is left: tiles per SM in whole numbers (0.7 to 0.9), rows of
// padding, the first chunk's way from HBM, the last addition.  Tiles of 32 rows: 1.3 to 2.5 times as long.  The eight sums dealt to 2 or 4 blocks of a
// cluster: 12 to 15 us instead of 13 at 32 x 1024 x 2816, otherwise slower.
#pragma once
#include "layered_ops.cuh"

namespace fl {

constexpr int kF64BN = 32, kF64Chunk = 16, kF64Sums = 8, kF64Ring = 4;
template <int BM>
struct F64Form {
    static constexpr int kStage = BM * kF64Chunk * 4 + kF64BN * kF64Chunk * 2;       // bytes of a warp's stage
    static constexpr int kSmem = kF64Sums * kF64Ring * kStage, kPerSM = BM == 16 ? 3 : 4;
    static_assert(kSmem >= kF64Sums * BM * kF64BN * 8, "the sums take the rings' place");
};
// Rows of a tile: tiles of 8 rows take 1.06 times as long per row as tiles of 16 (every 32 x 16 weights are widened for fewer products), but are
// twice as many where the chip has SMs to spare and leave fewer rows of padding.  An SM's tiles come in whole numbers.  rows: of a group, on average.
inline int f64_rows_per_tile(double rows, int cols, int groups, bool known) {
    auto tiles = [&](int bm) { return groups * ((cols + kF64BN - 1) / kF64BN) * (known ? std::ceil(rows / bm) : rows / bm + 0.5); };
    return 2 * std::ceil(tiles(16) / kNumSMs) <= 1.06 * std::ceil(tiles(8) / kNumSMs) ? 16 : 8;
}
__device__ __forceinline__ void mma_f64_884(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b));
}
// 16 bytes as copies of UNIT bytes (16, 8 or 4, which both addresses are multiples of): the first `bytes` are read, the others are zero
template <int UNIT>
__device__ __forceinline__ void cp_async_piece(uint32_t smem_dst, const void* gsrc, const void* any, int bytes) {
#pragma unroll
    for (int at = 0; at < 16; at += UNIT) {
        const int n = UNIT == 16 ? bytes : max(0, min(UNIT, bytes - at));
        const void* p = n > 0 ? static_cast<const char*>(gsrc) + at : any;
        if (UNIT == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_dst), "l"(p), "r"(n) : "memory");
        else if (UNIT == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_dst + at), "l"(p), "r"(n) : "memory");
        else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_dst + at), "l"(p), "r"(n) : "memory");
    }
}
// Bytes that a copy of W takes at a time: what the rows' addresses are multiples of.  A's go twice as many at a time, up to 16.
// Rows of 2-byte pieces alone (odd K) are read an element at a time, a chunk ahead of its place in the ring.  Prompts of 203 / 600 tokens, delta rule and
// dense feed-forward, us, every row that is no multiple of 16 bytes an element at a time as it was needed -> this: width 1028 1000 -> 650, 2230 -> 1480; 1026
// 1003 -> 720, 2240 -> 1620; 1023 1030 -> 905, 2340 -> 2060 (1024, by 16 bytes: 610, 1405).
inline int f64_unit(const LyGemm& g) {
    auto fits = [](const void* p, long long gs, long long row, int unit) { return ((reinterpret_cast<uintptr_t>(p) | (uintptr_t)gs | (uintptr_t)row) & (unit - 1)) == 0; };
    for (int u = 16; u > 2; u /= 2)
        if (fits(g.W, g.w_gs * 2, (long long)g.K * 2, u) && fits(g.A, g.a_gs * 4, (long long)g.lda * 4, std::min(16, 2 * u))) return u;
    return 2;
}

template <int BM, int UNIT>
static __global__ void __launch_bounds__(32 * kF64Sums, F64Form<BM>::kPerSM) ly_gemm64_kernel(LyGemm g) {
    pdl_chain();
    using F = F64Form<BM>;
    constexpr int MT = BM / 8, NT = kF64BN / 8, NA = BM / 8, NB = kF64BN * 2 / 32;
    extern __shared__ __align__(16) uint8_t sm64[];          // the warps' rings, then their sums
    const int grp = blockIdx.z;
    int p_lo = 0, p_hi = g.R;
    if (g.grp_off != nullptr) { p_lo = g.grp_off[grp]; p_hi = g.grp_off[grp + 1]; }
    const int p0 = p_lo + blockIdx.y * BM;
    if (p0 >= p_hi) return;
    const int n0 = blockIdx.x * kF64BN, tid = threadIdx.x, sum = tid >> 5, lane = tid & 31;
    const float* A = g.A + (size_t)grp * g.a_gs;
    const uint16_t* Wm = g.W + (size_t)grp * g.w_gs;
    float* Y = g.Y + (size_t)grp * g.y_gs;
    // 16-byte pieces of a stage: piece i of A is row i / 4, columns 4 (i % 4) ..; piece i of W is row i / 2, columns 8 (i % 2) ..
    const float* arow[NA];
    const uint16_t* wrow[NB];
#pragma unroll
    for (int t = 0; t < NA; ++t) {
        const int ap = p0 + (lane + 32 * t) / 4;
        arow[t] = ap < p_hi ? A + (size_t)(g.a_idx ? g.a_idx[ap] : ap) * g.lda : nullptr;
    }
#pragma unroll
    for (int t = 0; t < NB; ++t) {
        const int n = n0 + (lane + 32 * t) / 2;
        wrow[t] = n < g.N ? Wm + (size_t)n * g.K : nullptr;
    }
    uint8_t* ring = sm64 + (size_t)sum * kF64Ring * F::kStage;
    const int chunks = (g.K + kF64Chunk - 1) / kF64Chunk, mine = chunks > sum ? (chunks - sum + kF64Sums - 1) / kF64Sums : 0;
    auto fetch = [&](int j) {
        if (j < mine) {
            uint8_t* s = ring + (j % kF64Ring) * F::kStage;
            const int ka = (sum + kF64Sums * j) * kF64Chunk + lane % 4 * 4, kw = (sum + kF64Sums * j) * kF64Chunk + lane % 2 * 8;
            const int ba = ka < g.K ? (UNIT >= 8 ? 16 : 4 * min(4, g.K - ka)) : 0, bw = kw < g.K ? (UNIT == 16 ? 16 : 2 * min(8, g.K - kw)) : 0;     // (K is a multiple of UNIT / 2)
#pragma unroll
            for (int t = 0; t < NA; ++t) cp_async_piece<UNIT >= 8 ? 16 : 2 * UNIT>(smem_u32(s + (lane + 32 * t) * 16), arow[t] + ka, A, arow[t] != nullptr ? ba : 0);
            if (UNIT > 2) {
#pragma unroll
                for (int t = 0; t < NB; ++t) cp_async_piece<UNIT>(smem_u32(s + BM * kF64Chunk * 4 + (lane + 32 * t) * 16), wrow[t] + kw, Wm, wrow[t] != nullptr ? bw : 0);
            }
        }
        cp_async_commit();
    };
    // odd K: chunk j of W through registers
    uint32_t held[NB][4];
    auto load = [&](int j) {
        if (UNIT > 2 || j >= mine) return;
        const int kw = (sum + kF64Sums * j) * kF64Chunk + lane % 2 * 8;
#pragma unroll
        for (int t = 0; t < NB; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const uint32_t lo = wrow[t] != nullptr && kw + 2 * e < g.K ? wrow[t][kw + 2 * e] : 0u, hi = wrow[t] != nullptr && kw + 2 * e + 1 < g.K ? wrow[t][kw + 2 * e + 1] : 0u;
                held[t][e] = lo | hi << 16;
            }
    };
    auto put = [&](int j) {
        if (UNIT > 2 || j >= mine) return;
        uint8_t* s = ring + (j % kF64Ring) * F::kStage + BM * kF64Chunk * 4;
#pragma unroll
        for (int t = 0; t < NB; ++t) *reinterpret_cast<uint4*>(s + (lane + 32 * t) * 16) = make_uint4(held[t][0], held[t][1], held[t][2], held[t][3]);
    };
    auto wide = [](uint32_t b) { return (double)__uint_as_float(b); };
    double acc[MT][NT][2] = {};
#pragma unroll
    for (int j = 0; j < kF64Ring - 1; ++j) { fetch(j); load(j); put(j); }
    for (int j = 0; j < mine; ++j) {
        cp_async_wait<kF64Ring - 2>();
        __syncwarp();                   // chunk j is there; every lane has read chunk j - 1, whose place the next one takes
        fetch(j + kF64Ring - 1);
        load(j + kF64Ring - 1);
        const uint8_t* s = ring + (j % kF64Ring) * F::kStage;
        float4 a[MT];
        uint2 b[NT];
#pragma unroll
        for (int i = 0; i < MT; ++i) a[i] = *reinterpret_cast<const float4*>(s + i * 512 + lane * 16);
#pragma unroll
        for (int n = 0; n < NT; ++n) b[n] = *reinterpret_cast<const uint2*>(s + BM * kF64Chunk * 4 + n * 256 + lane * 8);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            double av[MT], bv[NT];
#pragma unroll
            for (int i = 0; i < MT; ++i) av[i] = (double)(e == 0 ? a[i].x : e == 1 ? a[i].y : e == 2 ? a[i].z : a[i].w);
#pragma unroll
            for (int n = 0; n < NT; ++n) bv[n] = wide(e == 0 ? b[n].x << 16 : e == 1 ? b[n].x & 0xFFFF0000u : e == 2 ? b[n].y << 16 : b[n].y & 0xFFFF0000u);
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int n = 0; n < NT; ++n) mma_f64_884(acc[i][n], av[i], bv[n]);
        }
        put(j + kF64Ring - 1);
    }
    cp_async_wait<0>();
    __syncthreads();
    double* sums = reinterpret_cast<double*>(sm64);          // [sum][BM][32]
    {
        double* d = sums + (size_t)sum * BM * kF64BN + (lane >> 2) * kF64BN + (lane & 3) * 2;
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int n = 0; n < NT; ++n) *reinterpret_cast<double2*>(d + i * 8 * kF64BN + n * 8) = make_double2(acc[i][n][0], acc[i][n][1]);
    }
    __syncthreads();
    for (int o = tid; o < BM * kF64BN; o += 32 * kF64Sums) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < kF64Sums; ++q) t += sums[(size_t)q * BM * kF64BN + o];
        const int p = p0 + o / kF64BN, n = n0 + o % kF64BN;
        if (p < p_hi && n < g.N) Y[(size_t)p * g.ldy + n] = (float)t;
    }
}

}  // namespace fl
