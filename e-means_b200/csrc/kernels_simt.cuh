// FP32 SIMT fused assign: x . c^T contraction in registers with a running
// top-2 per row in the epilogue, so no m x k score matrix ever reaches HBM.
// This is the plain FP32 form of the search (src/cpu.rs:108-167 computes the
// same scores on the CPU); its result is certified and re-scored exactly by
// kernels_exact.cuh.
#pragma once
#include "common.cuh"

namespace emb {

// What bounds it: the FP32 pipe (74 TF/s) and the shared-memory port beside it.
// A scalar FFMA takes its scheduler's whole issue rate, so every load and address
// instruction costs FMA time, and 8 x 8 values per thread need four 16-byte shared
// loads per 64 FMAs, the port's limit. Hence paired FMAs (fma.rn.f32x2: two IEEE
// FMAs, half the issue slots) over neighbouring columns and 8 x 16 values per thread
// (six loads per 128 FMAs); the running top-2 of a thread's rows lives in shared
// memory, touched once per tile. 200,000 x 96 rows, k = 1024: 1488 -> 951 us (26 ->
// 41 TF/s; FMA pipe 59% busy, the rest mostly shared-load latency that two warps per
// scheduler do not cover). Storing each row value twice, so that its pair is one
// load, or 8 x 8 values with two CTAs per SM measured 32 TF/s.
// Few rows (100 x 96, k = 1024: 30 -> 13 us) take 64 x 64 tiles, 4 x 4 values per
// thread.
constexpr int kSimtBK = 16, kSimtThreads = 256;

// Tile of the form with 4 RG rows and 4 CG columns per thread: a warp's lanes stand
// 4 x 8, the eight warps 4 x 2.
template <int RG, int CG>
struct SimtTile {
    static constexpr int BM = 64 * RG, BN = 64 * CG;
    // two stages of rows and of centroids, and the threads' top-2 lists
    static constexpr size_t smem = (size_t)2 * kSimtBK * (BM + BN) * sizeof(float) +
                                   (size_t)4 * RG * kSimtThreads * sizeof(float4);
};
using SimtLarge = SimtTile<2, 4>;
using SimtSmall = SimtTile<1, 1>;

// Loads a 16 E x kSimtBK slab of rows (or centroids) into registers: thread t takes
// E consecutive elements of row t / (16 / E). Out-of-range entries are zero.
template <typename T, int E>
EMB_DEV void simt_load(float (&r)[E], const T* __restrict__ base, const uint32_t* __restrict__ gather, int row0,
                       int nrows, int d, int k0, bool vec4) {
    const int t = threadIdx.x;
    const int row = row0 + t / (16 / E);
    const int col = k0 + (t % (16 / E)) * E;
#pragma unroll
    for (int i = 0; i < E; i++) r[i] = 0.0f;
    if (row >= nrows) return;
    const size_t src = gather ? gather[row] : (size_t)row;
    const T* p = base + src * (size_t)d + col;
    if (sizeof(T) == 4 && vec4 && col + E <= d) {
#pragma unroll
        for (int i = 0; i < E; i += 4) {
            const float4 a = *reinterpret_cast<const float4*>(p + i);
            r[i] = a.x; r[i + 1] = a.y; r[i + 2] = a.z; r[i + 3] = a.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < E; i++)
            if (col + i < d) r[i] = to_f32(p[i]);
    }
}

// Grid: (ceil(m / BM), nsplit). CTA (bx, by) searches rows [BM bx, + BM) against
// centroid tiles by, by + nsplit, ... and writes its top-2 per row to
// part_s/part_i[by][row][0..1]. norms are padded to whole 256-centroid tiles.
template <typename T, int RG, int CG>
__global__ void __launch_bounds__(kSimtThreads, RG * CG > 4 ? 1 : 2)
k_assign_simt(const T* __restrict__ x, const uint32_t* __restrict__ gather, int m, int d,
              const float* __restrict__ c, const float* __restrict__ norms, int k,
              float* __restrict__ part_s, uint32_t* __restrict__ part_i, int vec4) {
    constexpr int BM = SimtTile<RG, CG>::BM, BN = SimtTile<RG, CG>::BN, TM = 4 * RG, TN = 4 * CG;
    extern __shared__ __align__(16) float simt_sm[];
    float* As = simt_sm;                                              // [2][kSimtBK][BM]
    float* Bs = As + 2 * kSimtBK * BM;                                // [2][kSimtBK][BN]
    float4* tops = reinterpret_cast<float4*>(Bs + 2 * kSimtBK * BN);  // [TM][threads]: s1, i1, s2, i2
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rbase = (warp >> 1) * 16 * RG + (lane >> 3) * 4;  // + 16 g: this thread's row groups
    const int cbase = (warp & 1) * 32 * CG + (lane & 7) * 4;    // + 32 g: its column groups
    const int row0 = blockIdx.x * BM;
    const int nsplit = gridDim.y;
    const int ntiles = (k + BN - 1) / BN;
    const int nk = (d + kSimtBK - 1) / kSimtBK;
    const float inf = __int_as_float(0x7f800000), none = __uint_as_float(0xffffffffu);
#pragma unroll
    for (int i = 0; i < TM; i++) tops[i * kSimtThreads + tid] = make_float4(inf, none, inf, none);
    auto store = [&](int buf, const float (&ra)[TM], const float (&rb)[TN]) {
        float* a = As + (buf * kSimtBK + (tid % (16 / TM)) * TM) * BM + tid / (16 / TM);
        float* b = Bs + (buf * kSimtBK + (tid % (16 / TN)) * TN) * BN + tid / (16 / TN);
#pragma unroll
        for (int i = 0; i < TM; i++) a[i * BM] = ra[i];
#pragma unroll
        for (int i = 0; i < TN; i++) b[i * BN] = rb[i];
    };

    // One stream of (tile, K step) slabs through the two buffers: the slab after this
    // one is loaded into registers while this one is multiplied, also across tiles.
    float ra[TM], rb[TN];
    simt_load(ra, x, gather, row0, m, d, 0, vec4);
    simt_load(rb, c, (const uint32_t*)nullptr, (int)blockIdx.y * BN, k, d, 0, vec4);
    store(0, ra, rb);
    __syncthreads();
    int buf = 0;
    for (int tile = blockIdx.y; tile < ntiles; tile += nsplit) {
        const int col0 = tile * BN;
        float2 acc[TM][TN / 2];
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN / 2; j++) acc[i][j] = make_float2(0.0f, 0.0f);
        for (int kt = 0; kt < nk; kt++, buf ^= 1) {
            const bool last = kt + 1 == nk;
            const bool more = !last || tile + nsplit < ntiles;
            if (more) {
                const int k1 = last ? 0 : (kt + 1) * kSimtBK;
                simt_load(ra, x, gather, row0, m, d, k1, vec4);
                simt_load(rb, c, (const uint32_t*)nullptr, last ? col0 + nsplit * BN : col0, k, d, k1, vec4);
            }
            const float* at = As + buf * kSimtBK * BM + rbase;
            const float* bt = Bs + buf * kSimtBK * BN + cbase;
#pragma unroll
            for (int kk = 0; kk < kSimtBK; kk++) {
                float2 b[TN / 2];
#pragma unroll
                for (int g = 0; g < CG; g++) {
                    const float4 v = *reinterpret_cast<const float4*>(bt + kk * BN + 32 * g);
                    b[2 * g] = make_float2(v.x, v.y);
                    b[2 * g + 1] = make_float2(v.z, v.w);
                }
#pragma unroll
                for (int g = 0; g < RG; g++) {
                    const float4 v = *reinterpret_cast<const float4*>(at + kk * BM + 16 * g);
                    const float a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int j = 0; j < TN / 2; j++)
                            acc[4 * g + i][j] = __ffma2_rn(make_float2(a[i], a[i]), b[j], acc[4 * g + i][j]);
                }
            }
            if (more) store(buf ^ 1, ra, rb);
            __syncthreads();
        }
        // Epilogue: score = norms_j - 2 acc (one rounding), running top-2 per row.
        float n[TN];
#pragma unroll
        for (int g = 0; g < CG; g++) {
            const float4 v = *reinterpret_cast<const float4*>(norms + col0 + cbase + 32 * g);
            n[4 * g] = v.x; n[4 * g + 1] = v.y; n[4 * g + 2] = v.z; n[4 * g + 3] = v.w;
        }
#pragma unroll
        for (int j = 0; j < TN; j++)  // columns past k never enter
            if (col0 + cbase + (j >> 2) * 32 + (j & 3) >= k) n[j] = inf;
#pragma unroll
        for (int i = 0; i < TM; i++) {
            float sc[TN], mn = inf;
#pragma unroll
            for (int j = 0; j < TN / 2; j++) {
                const float2 s2 = __ffma2_rn(make_float2(-2.0f, -2.0f), acc[i][j], make_float2(n[2 * j], n[2 * j + 1]));
                sc[2 * j] = s2.x;
                sc[2 * j + 1] = s2.y;
                mn = fminf(mn, fminf(s2.x, s2.y));
            }
            // A thread's columns ascend, so only a strictly smaller score can enter.
            const float4 t4 = tops[i * kSimtThreads + tid];
            if (mn < t4.z) {
                Top2 t;
                t.s1 = t4.x; t.i1 = __float_as_uint(t4.y); t.s2 = t4.z; t.i2 = __float_as_uint(t4.w);
#pragma unroll
                for (int j = 0; j < TN; j++)
                    t.push_fast(sc[j], (uint32_t)(col0 + cbase + (j >> 2) * 32 + (j & 3)));
                tops[i * kSimtThreads + tid] = make_float4(t.s1, __uint_as_float(t.i1), t.s2, __uint_as_float(t.i2));
            }
        }
    }
    // One thread per row merges the 16 threads that share it (8 lanes of two warps).
    __syncthreads();
    if (tid < BM && row0 + tid < m) {
        const int wr = tid / (16 * RG), g = tid % (16 * RG) / 16, ly = (tid & 15) >> 2, i = 4 * g + (tid & 3);
        Top2 t;
        t.init();
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const float4 e = tops[i * kSimtThreads + (wr * 2 + (q >> 3)) * 32 + ly * 8 + (q & 7)];
            t.push(e.x, __float_as_uint(e.y));
            t.push(e.z, __float_as_uint(e.w));
        }
        const size_t o = ((size_t)blockIdx.y * m + row0 + tid) * 2;
        part_s[o] = t.s1;
        part_i[o] = t.i1;
        part_s[o + 1] = t.s2;
        part_i[o + 1] = t.i2;
    }
}

}  // namespace emb
