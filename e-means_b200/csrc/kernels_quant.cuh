// Int8 quantizer on the device: the fit (per-dimension mean shift and the
// peak of the centred magnitudes) and the encode / clipped count / decode of
// Int8Quantizer (src/quantize.rs:45-96), bit-exact with the reference.
//
// Exactness notes, per step of Int8Quantizer::fit (src/quantize.rs:45-62):
//  * mean: the reference adds the rows in order into one f64 accumulator per
//    dimension (`:48-51`). f64 addition is not associative, so a tree reduction
//    could differ in the last bit; k_quant_colpart / k_quant_colscan add whole
//    blocks of rows where that provably rounds nowhere and replay the rest in
//    row order.
//  * peak: `select_nth_unstable_by(idx, f32::total_cmp)` over |x - shift|
//    (`:53-56`). Every magnitude has a clear sign bit, so total_cmp is the
//    unsigned order of the bit patterns (NaNs above +inf); the select is a
//    three-pass radix select on those bit patterns (11 + 10 + 10 bits), or one
//    max / min reduction when idx is the last / first rank.
//  * encode: `((v - s) * scale).round().clamp(-128, 127) as i8` (`:65-73`):
//    two separately rounded f32 operations, round half away from zero, and the
//    saturating cast that sends NaN to 0.
#pragma once
#include <cstdint>

#include "common.cuh"

namespace emb {

constexpr int kQThreads = 512;     // element-wise passes
constexpr int kQBins0 = 2048;      // bits 30..20 of a magnitude (bit 31 is always clear)
constexpr int kQBins = 1024;       // bits 19..10, then bits 9..0

struct QuantSelect {
    unsigned long long rank;  // rank still to find inside the current prefix
    unsigned int prefix;      // bit pattern chosen so far (the peak after the last pass)
    unsigned int pad;
    unsigned long long hist[kQBins0];
};

__device__ __forceinline__ void qs_cp_async16(float* smem, const float* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void qs_cp_async4(float* smem, const float* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void qs_cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void qs_cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Per-dimension f64 sums in row order, then shift = (f32)(sum / n)
// (src/quantize.rs:48-52), without walking the n dependent adds one by one.
//
// A chain acc <- RN(acc + x_i) rounds only where a partial sum needs more than 53
// bits: with every x_i and acc multiples of 2^q, all partial sums of magnitude at
// most 2^(53 + q) are exact, and then any order of adding gives the chain's bits.
//   k_quant_colpart  per block of kQsubRows rows and dimension: the sum, the
//                    range of its prefix sums and its smallest non-zero magnitude
//                    (which bounds q). One pass over the rows: HBM bounds it.
//                    A block is added as four parts that start at zero: a part's sums
//                    lie within the range's width, hi - lo, so they are exact where
//                    that is at most 2^(53 + q).
//   k_quant_colscan  one warp per dimension walks the blocks 32 at a time: a lane's
//                    block is accepted as a whole when the range above shows that
//                    no partial sum inside it (nor inside its parts) rounds; the first
//                    block that is not is replayed from its rows (quant_replay64), which
//                    finds the adds that do round by their exact error and redoes the
//                    rest from there.
// On 500,000 x 512 unit-norm rows: 0.175 ms (5.9 TB/s of rows, 0.90 of the copy
// bandwidth) and 0.068 ms, against 4.25 ms for the chain itself (16.7 cycles an
// add). Blocks of 256 rows: with 64 the scan of four times the entries took
// 0.20 ms, and the rows it replays are few (none for most dimensions here).
constexpr int kQsubRows = 256;
constexpr int kQpartRows = 64;  // rows per thread of k_quant_colpart
constexpr int kQscanDepth = 7;  // batches of 32 blocks in flight per warp (cp.async)
constexpr int kQscanWarps = 8;  // neighbouring dimensions per CTA: they share the entries' sectors
constexpr size_t kQsubBytes = (size_t)24 << 20;  // entries held at once; longer samples go in slabs of rows

struct __align__(16) QuantSub {
    double sum;
    float lo, hi;  // range of the prefix sums, rounded outwards
};

// Smallest non-zero magnitude in a form that one unsigned minimum keeps: the bits
// without the sign, doubled, less one (zero wraps to the largest value).
__device__ __forceinline__ uint32_t quant_tiny(float v) { return (__float_as_uint(v) << 1) - 1u; }
// The exponent of the lowest bit a value of at least that magnitude can have.
__device__ __forceinline__ int quant_tiny_lsb(uint32_t tiny) {
    if (tiny == 0xffffffffu) return 900;  // nothing but zeros
    return max((int)(((tiny + 1u) >> 1) >> 23), 1) - 150;
}
__device__ __forceinline__ double quant_pow2(int e) { return __hiloint2double((min(e, 1000) + 1023) << 20, 0); }
// The exponent of the lowest set bit of a finite double.
__device__ __forceinline__ int quant_lsb(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    if (b == 0) return 900;
    const int e = (int)(b >> 52);
    const unsigned long long m = (b & 0xfffffffffffffull) | (e ? 1ull << 52 : 0ull);
    return max(e, 1) - 1075 + (__ffsll((long long)m) - 1);
}

// V consecutive dimensions per thread (V = 4: d % 4 == 0, 16-byte loads). 64 threads
// side by side take the (block, dimensions) pairs, the four groups of 64 a quarter
// of the block's rows each; their results are joined in row order through shared
// memory.
template <int V>
__global__ void __launch_bounds__(256) k_quant_colpart(const float* __restrict__ x, size_t n, size_t d, size_t nsub,
                                                       QuantSub* __restrict__ sub, uint32_t* __restrict__ tiny) {
    constexpr int kParts = kQsubRows / kQpartRows;
    static_assert(kParts == 4, "256 threads: four parts of 64");
    __shared__ double sum_s[kParts - 1][V][64];
    __shared__ float rng_s[kParts - 1][4][V][64];
    __shared__ uint32_t tiny_s[kParts - 1][V][64];
    const size_t dq = d / V;
    const int lt = threadIdx.x & 63, part = threadIdx.x >> 6;
    const size_t e = (size_t)blockIdx.x * 64 + lt;
    const bool live = e < nsub * dq;
    const size_t s = live ? e / dq : 0, q = live ? e - s * dq : 0;
    const size_t r0 = s * kQsubRows + (size_t)part * kQpartRows;
    const float* p = x + r0 * d + q * V;
    const int rows = live && r0 < n ? (int)min((size_t)kQpartRows, n - r0) : 0;
    // The prefix sums' range comes from two f32 chains rounded up and down: the f64
    // conversions it would take otherwise cost more issue time than the loads.
    double acc[V];
    float up[V], dn[V], lo[V], hi[V];
    uint32_t tn[V];
#pragma unroll
    for (int i = 0; i < V; i++) {
        acc[i] = 0.0;
        up[i] = dn[i] = lo[i] = hi[i] = 0.0f;
        tn[i] = 0xffffffffu;
    }
    auto take = [&](const float (&v)[V]) {
#pragma unroll
        for (int i = 0; i < V; i++) {
            acc[i] = __dadd_rn(acc[i], (double)v[i]);
            dn[i] = __fadd_rd(dn[i], v[i]);
            up[i] = __fadd_ru(up[i], v[i]);
            lo[i] = fminf(lo[i], dn[i]);
            hi[i] = fmaxf(hi[i], up[i]);
            tn[i] = min(tn[i], quant_tiny(v[i]));
        }
    };
    auto load = [&](int r, float (&v)[V]) {
        if constexpr (V == 4) {
            const float4 f = __ldg(reinterpret_cast<const float4*>(p + (size_t)r * d));
            v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
        } else {
            v[0] = __ldg(p + (size_t)r * d);
        }
    };
    int r = 0;
    for (; r + 8 <= rows; r += 8) {
        float v[8][V];
#pragma unroll
        for (int u = 0; u < 8; u++) load(r + u, v[u]);
#pragma unroll
        for (int u = 0; u < 8; u++) take(v[u]);
    }
    for (; r < rows; r++) {
        float v[V];
        load(r, v);
        take(v);
    }
    if (part > 0) {
#pragma unroll
        for (int i = 0; i < V; i++) {
            sum_s[part - 1][i][lt] = acc[i];
            rng_s[part - 1][0][i][lt] = dn[i];
            rng_s[part - 1][1][i][lt] = up[i];
            rng_s[part - 1][2][i][lt] = lo[i];
            rng_s[part - 1][3][i][lt] = hi[i];
            tiny_s[part - 1][i][lt] = tn[i];
        }
    }
    __syncthreads();
    if (part > 0 || !live) return;
#pragma unroll
    for (int i = 0; i < V; i++) {
#pragma unroll
        for (int o = 0; o < kParts - 1; o++) {
            lo[i] = fminf(lo[i], __fadd_rd(dn[i], rng_s[o][2][i][lt]));
            hi[i] = fmaxf(hi[i], __fadd_ru(up[i], rng_s[o][3][i][lt]));
            dn[i] = __fadd_rd(dn[i], rng_s[o][0][i][lt]);
            up[i] = __fadd_ru(up[i], rng_s[o][1][i][lt]);
            acc[i] = __dadd_rn(acc[i], sum_s[o][i][lt]);
            tn[i] = min(tn[i], tiny_s[o][i][lt]);
        }
        QuantSub o;
        o.sum = acc[i];
        o.lo = lo[i];
        o.hi = hi[i];
        sub[s * d + q * V + i] = o;
        tiny[s * d + q * V + i] = tn[i];
    }
}

__device__ __forceinline__ double quant_scan32(double v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v = __dadd_rn(v, u);
    }
    return v;
}

__device__ __forceinline__ double quant_two_sum_err(double a, double b, double s) {
    const double bb = __dsub_rn(s, a);
    return __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb));
}

// acc after 64 rows (lane i holds rows i and 32 + i), every rounding of the chain
// kept. Mostly no add rounds after all: one look at all 64 partial sums shows that
// (acc + the values' prefix sum is the chain's partial sum up to and including the
// first add that rounds, and its two-sum error shows which that is). The rest is
// then added one by one, from the warp's shared memory. The look needs the prefix
// sums to be exact: 64 times the largest value within 53 bits of the lowest bit.
// rough counts the groups that needed most of the adds.
__device__ __forceinline__ double quant_replay64(double acc, float x0, float x1, int lane, double* buf, int& rough) {
    int s0 = 0;
    const uint32_t tn = __reduce_min_sync(0xffffffffu, min(quant_tiny(x0), quant_tiny(x1)));
    if (tn == 0xffffffffu) return acc;  // zeros change nothing
    const uint32_t mx =
        __reduce_max_sync(0xffffffffu, max(__float_as_uint(x0) & 0x7fffffffu, __float_as_uint(x1) & 0x7fffffffu));
    if (mx < 0x7f800000u && isfinite(acc) &&
        64.0 * (double)__uint_as_float(mx) <= quant_pow2(53 + quant_tiny_lsb(tn))) {
        const double i0 = quant_scan32((double)x0, lane), i1r = quant_scan32((double)x1, lane);
        const double i1 = __dadd_rn(__shfl_sync(0xffffffffu, i0, 31), i1r);
        const double p0 = __dadd_rn(acc, i0), p1 = __dadd_rn(acc, i1);
        const unsigned b0 = __ballot_sync(0xffffffffu, quant_two_sum_err(acc, i0, p0) != 0.0);
        const unsigned b1 = __ballot_sync(0xffffffffu, quant_two_sum_err(acc, i1, p1) != 0.0);
        if (!(b0 | b1)) return __shfl_sync(0xffffffffu, p1, 31);
        const int f = b0 ? __ffs((int)b0) - 1 : __ffs((int)b1) - 1;
        acc = __shfl_sync(0xffffffffu, b0 ? p0 : p1, f);
        s0 = f + (b0 ? 1 : 33);
    }
    rough += s0 < 33;
    buf[lane] = (double)x0;
    buf[32 + lane] = (double)x1;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 64; i += 16) {
        if (i + 16 > s0) {
            double u[16];
#pragma unroll
            for (int j = 0; j < 16; j++) u[j] = buf[i + j];
#pragma unroll
            for (int j = 0; j < 16; j++)
                if (i + j >= s0) acc = __dadd_rn(acc, u[j]);
        }
    }
    __syncwarp();
    return acc;
}

// acc after 256 rows (doubles in shared memory), added one by one, 16 at a time with the
// next 16 on their way.
__device__ __forceinline__ double quant_chain256(double acc, const double* rows) {
    double a[16], b[16];
#pragma unroll
    for (int j = 0; j < 16; j++) a[j] = rows[j];
#pragma unroll 1
    for (int r = 0; r < kQsubRows; r += 32) {
#pragma unroll
        for (int j = 0; j < 16; j++) b[j] = rows[r + 16 + j];
#pragma unroll
        for (int j = 0; j < 16; j++) acc = __dadd_rn(acc, a[j]);
        const double* next = rows + (r + 32) % kQsubRows;  // (the first again at the end: not used)
#pragma unroll
        for (int j = 0; j < 16; j++) a[j] = next[j];
#pragma unroll
        for (int j = 0; j < 16; j++) acc = __dadd_rn(acc, b[j]);
    }
    return acc;
}

// One warp per dimension; first / last: the sample's first / last slab of rows
// (carry holds the sums in between). sub = nullptr: no entries, every block is
// replayed (short samples: n <= kQscanShort, where the entries' launch costs more
// than they save).
// Where the adds round often (magnitudes spread over many binades), looking first is
// slower than the chain: a warp that has met kRoughFirst groups of 64 rows that needed
// most of their adds, in one block after another, leaves the next blocks to its whole CTA:
// kQscanJoint of them, and twice as many, up to kQscanJointMost, each time that this
// happens again (then at the first such group) within as many as the last time. There one
// warp adds, a lane a dimension, and the others bring the rows: each row's 32 bytes are
// read once, where a warp alone touches 32 lines for 32 values of its column, which bounds
// it (9.6 ns a row, 17 with two CTAs on an SM), and no FP64 cycles go into 32 equal
// results. Whole fits, each dimension's warp replaying by itself / so / every dimension as
// one chain from the start: magnitudes over 60 binades, 200,000 x 64 1986 / 1250 / 1784 us,
// 50,000 x 2048 1097 / 618 / 575; squares of normals 200,000 x 64 1873 / 1359 / 1781,
// 50,000 x 2048 967 / 790 / 576, 50,000 x 64 508 / 499 / 497; normals, 200,000 x 64, 126 /
// 129 / 1781; unit-norm embeddings, 500,000 x 512, six samples, 472 .. 520 / 474 .. 492 /
// 4515 .. 4520. Two groups to begin with: such samples up to 548; two of them afterwards as
// well, or joint runs of 16 blocks at first: the squares, 50,000 x 64, 1.05 and 1.33 times
// as long.
constexpr size_t kQscanShort = 2048;
constexpr int kRoughFirst = 3, kQscanJoint = 32, kQscanJointMost = 256;
constexpr int kQscanPitch = kQsubRows + 4;  // of a dimension's converted rows: no bank conflicts across dimensions
struct QuantRing {
    QuantSub sub[kQscanWarps][kQscanDepth][32];
    uint32_t tiny[kQscanWarps][kQscanDepth][32];
};
union QuantScanSmem {
    QuantRing ring;                                // a warp's entries
    double joint[2][kQscanWarps][kQscanPitch];     // two blocks of all its dimensions' rows
};
__global__ void __launch_bounds__(32 * kQscanWarps) k_quant_colscan(const float* __restrict__ x, size_t n, size_t d,
                                                                    size_t nsub, const QuantSub* __restrict__ sub,
                                                                    const uint32_t* __restrict__ tiny,
                                                                    double* __restrict__ carry, bool first, bool last,
                                                                    size_t n_all, float* __restrict__ shift) {
    __shared__ __align__(16) uint8_t smem_raw[sizeof(QuantScanSmem)];
    __shared__ __align__(16) double chain_s[kQscanWarps][64];
    __shared__ size_t pos_s[kQscanWarps];
    __shared__ double acc_s[kQscanWarps];
    QuantScanSmem& sm = *reinterpret_cast<QuantScanSmem*>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t t = (size_t)blockIdx.x * kQscanWarps + warp;
    const size_t nb = (nsub + 31) / 32;
    auto issue = [&](size_t b) {  // each lane copies, and later reads, its own entries only
        const size_t s = b * 32 + lane;
        if (s < nsub) {
            qs_cp_async16(reinterpret_cast<float*>(&sm.ring.sub[warp][b % kQscanDepth][lane]),
                          reinterpret_cast<const float*>(sub + s * d + t));
            qs_cp_async4(reinterpret_cast<float*>(&sm.ring.tiny[warp][b % kQscanDepth][lane]),
                         reinterpret_cast<const float*>(tiny + s * d + t));
        }
        qs_cp_commit();
    };
    double acc = first || t >= d ? 0.0 : carry[t];
    size_t pos = t < d ? 0 : nsub;  // blocks before it are in acc
    constexpr int kPer = kQsubRows / 32;
    float ahead[kPer];  // rows of block ahead_s, loaded before they are needed
    size_t ahead_s = ~(size_t)0;
    int rough = 0;  // groups of the latest replayed blocks that needed most of their adds
    size_t joint = kQscanJoint, joint_end = 0;  // blocks of the CTA's last joint run, and its end
    bool leave = false;
    auto rows_of = [&](size_t s, float (&v)[kPer]) {
#pragma unroll
        for (int u = 0; u < kPer; u++) {
            const size_t r = s * kQsubRows + u * 32 + lane;
            v[u] = r < n ? __ldg(x + r * d + t) : 0.0f;
        }
    };
    auto replay = [&](size_t s) {
        float v[kPer];
        if (s == ahead_s) {
#pragma unroll
            for (int u = 0; u < kPer; u++) v[u] = ahead[u];
        } else {
            rows_of(s, v);
        }
        if (!sub) {
            ahead_s = s + 1;
            rows_of(ahead_s, ahead);
        }
#pragma unroll
        for (int u = 0; u < kPer; u += 2) acc = quant_replay64(acc, v[u], v[u + 1], lane, chain_s[warp], rough);
        leave = rough >= (joint_end && s <= joint_end + joint ? 1 : kRoughFirst);
        pos = s + 1;
    };
    // The blocks from pos on, until the end or until the warp leaves some to all of them.
    auto scan = [&]() {
        leave = false;
        rough = 0;
        if (!sub) {
            while (pos < nsub && !leave) replay(pos);
            return;
        }
        const size_t b0 = pos / 32;
        for (size_t b = b0; b < b0 + kQscanDepth - 1; b++) issue(b);
        for (size_t b = b0; b < nb && !leave; b++) {
            issue(b + kQscanDepth - 1);
            qs_cp_wait<kQscanDepth - 1>();
            QuantSub e{0.0, 0.0f, 0.0f};
            uint32_t tn = 0xffffffffu;
            if (b * 32 + lane < nsub) {
                e = sm.ring.sub[warp][b % kQscanDepth][lane];
                tn = sm.ring.tiny[warp][b % kQscanDepth][lane];
            }
            const size_t end = min(nsub, b * 32 + 32);
            const int qx = quant_tiny_lsb(tn);
            const int qmin = __reduce_min_sync(0xffffffffu, qx);
            if (qmin == 900) {  // nothing but zeros
                pos = end;
                continue;
            }
            const float mag = fmaxf(fabsf(e.lo), fabsf(e.hi));
            const float magmax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mag)));
            // Sums of any of these blocks are exact; otherwise one block at a time.
            const bool wide = 32.0 * (double)magmax < quant_pow2(53 + qmin);
            const bool fin = isfinite(e.sum);
            while (pos < end && !leave) {
                const int s0 = (int)(pos - b * 32), lim = wide ? 32 : s0 + 1;
                double before = 0.0;  // of the blocks s0 .. lane - 1
                if (wide) {
                    before = __shfl_up_sync(0xffffffffu, quant_scan32(lane >= s0 ? e.sum : 0.0, lane), 1);
                    if (lane == 0) before = 0.0;
                }
                const double p = __dadd_rn(acc, before);
                bool ok = tn == 0xffffffffu || isnan(p) || (isinf(p) && fin);
                if (!ok) {
                    const double top = quant_pow2(53 + min(qx, quant_lsb(p)));
                    ok = fin && __dsub_ru((double)e.hi, (double)e.lo) <= quant_pow2(53 + qx) &&
                         __dadd_ru(p, (double)e.hi) <= top && __dadd_rd(p, (double)e.lo) >= -top;
                }
                const unsigned bad = __ballot_sync(0xffffffffu, lane >= s0 && lane < lim && !ok);
                const int f = bad ? __ffs((int)bad) - 1 : lim;  // the blocks before it are taken whole
                acc = __shfl_sync(0xffffffffu, bad ? p : __dadd_rn(p, e.sum), bad ? f : lim - 1);
                if (f > s0) rough = 0;
                pos = min(end, b * 32 + f);
                if (bad) replay(pos);
            }
        }
        qs_cp_wait<0>();
    };
    for (;;) {
        if (pos < nsub) scan();
        if (lane == 0) {
            pos_s[warp] = pos;
            acc_s[warp] = acc;
        }
        __syncthreads();  // the ring is free as well
        size_t s = nsub;
        for (int w = 0; w < kQscanWarps; w++) s = min(s, pos_s[w]);
        if (s == nsub) break;  // the same for all
        joint = joint_end && s <= joint_end + joint ? min(2 * joint, (size_t)kQscanJointMost) : kQscanJoint;
        const size_t end = min(nsub, s + joint);
        joint_end = end;
        // Warp 0 adds, lane l dimension l % 8 (a warp for each would take the FP64 pipe's
        // time for 32 equal results); the others bring the next block.
        constexpr int kLoaders = 32 * (kQscanWarps - 1), kValues = kQsubRows * kQscanWarps;
        auto bring = [&](size_t blk, int buf) {
            float v[(kValues + kLoaders - 1) / kLoaders];
            const int e0 = (int)threadIdx.x - 32;
#pragma unroll
            for (int i = 0; e0 + i * kLoaders < kValues && i < (kValues + kLoaders - 1) / kLoaders; i++) {
                const int e = e0 + i * kLoaders;
                const size_t r = blk * kQsubRows + e / kQscanWarps;
                const size_t c = (size_t)blockIdx.x * kQscanWarps + e % kQscanWarps;
                v[i] = r < n && c < d ? __ldg(x + r * d + c) : 0.0f;
            }
#pragma unroll
            for (int i = 0; e0 + i * kLoaders < kValues && i < (kValues + kLoaders - 1) / kLoaders; i++) {
                const int e = e0 + i * kLoaders;
                sm.joint[buf][e % kQscanWarps][e / kQscanWarps] = (double)v[i];
            }
        };
        const int mine = lane % kQscanWarps;
        acc = acc_s[mine];
        pos = pos_s[mine];
        if (warp > 0) bring(s, 0);
        __syncthreads();
        for (int buf = 0; s < end; s++, buf ^= 1) {
            if (warp == 0) {
                const double sum = quant_chain256(acc, sm.joint[buf][mine]);
                if (pos == s) {  // (a dimension further on joins in when the blocks get there)
                    acc = sum;
                    pos = s + 1;
                }
            } else if (s + 1 < end) {
                bring(s + 1, buf ^ 1);
            }
            __syncthreads();
        }
        if (threadIdx.x < kQscanWarps) {
            acc_s[threadIdx.x] = acc;
            pos_s[threadIdx.x] = pos;
        }
        __syncthreads();
        acc = acc_s[warp];
        pos = pos_s[warp];
        __syncwarp();
    }
    if (lane == 0 && t < d) {
        if (last) shift[t] = __double2float_rn(__ddiv_rn(acc, (double)n_all));
        else carry[t] = acc;
    }
}

// The element-wise passes visit elements e = 4 * t + j * S (t the global thread
// index, S = 4 x threads in the grid). The host sizes the grid so that S is a
// multiple of d: a thread's four dimensions, and so its four shifts, never change.
__device__ __forceinline__ unsigned int quant_mag_bits(float v, float s) {
    return __float_as_uint(fabsf(__fsub_rn(v, s)));
}

// pass 0: histogram of bits 30..20; pass 1: of bits 19..10 among magnitudes whose
// bits 30..20 are sel->prefix; pass 2: of bits 9..0 among those matching bits 30..10.
template <int PASS>
__global__ void __launch_bounds__(kQThreads) k_quant_hist(const float* __restrict__ x, size_t N, size_t d,
                                                          const float* __restrict__ shift, QuantSelect* sel) {
    constexpr int NB = PASS == 0 ? kQBins0 : kQBins;
    __shared__ unsigned int h[NB];
    for (int i = threadIdx.x; i < NB; i += blockDim.x) h[i] = 0;
    const unsigned int prefix = PASS == 0 ? 0u : sel->prefix;
    __syncthreads();
    auto count = [&](unsigned int bits) {
        if (PASS == 0) {
            atomicAdd(&h[bits >> 20], 1u);
        } else if (PASS == 1) {
            if ((bits >> 20) == prefix) atomicAdd(&h[(bits >> 10) & 1023u], 1u);
        } else {
            if ((bits >> 10) == prefix) atomicAdd(&h[bits & 1023u], 1u);
        }
    };
    const size_t nthr = (size_t)gridDim.x * blockDim.x;
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t N4 = N / 4, S4 = nthr;
    if (t < N4) {
        float s[4];
#pragma unroll
        for (int i = 0; i < 4; i++) s[i] = shift[(4 * t + i) % d];
        const float4* x4 = reinterpret_cast<const float4*>(x);
        for (size_t g = t; g < N4; g += S4) {
            const float4 v = __ldg(x4 + g);
            count(quant_mag_bits(v.x, s[0]));
            count(quant_mag_bits(v.y, s[1]));
            count(quant_mag_bits(v.z, s[2]));
            count(quant_mag_bits(v.w, s[3]));
        }
    }
    if (t < N - 4 * N4) {  // the last N % 4 elements
        const size_t e = 4 * N4 + t;
        count(quant_mag_bits(x[e], shift[e % d]));
    }
    __syncthreads();
    for (int i = threadIdx.x; i < NB; i += blockDim.x)
        if (h[i]) atomicAdd(&sel->hist[i], (unsigned long long)h[i]);
}

// One warp: find the bin holding rank `rank` (pass 0: the rank passed in; later
// passes: sel->rank), extend the prefix by it, keep the rank within that bin and
// clear the histogram for the next pass.
__global__ void k_quant_pick(QuantSelect* sel, int pass, unsigned long long rank0) {
    const int lane = threadIdx.x;
    const int nb = pass == 0 ? kQBins0 : kQBins, per = nb / 32;
    unsigned long long rank = pass == 0 ? rank0 : sel->rank;
    unsigned long long mine = 0;
    for (int i = 0; i < per; i++) mine += sel->hist[lane * per + i];
    unsigned long long incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const unsigned long long excl = incl - mine;
    const unsigned int hit = __ballot_sync(0xffffffffu, incl > rank);
    const int owner = hit ? __ffs(hit) - 1 : 31;
    int bin = nb - 1;
    unsigned long long below = 0;
    if (lane == owner) {
        unsigned long long cum = excl;
        bin = lane * per + per - 1;
        for (int i = 0; i < per; i++) {
            const unsigned long long c = sel->hist[lane * per + i];
            if (cum + c > rank) {
                bin = lane * per + i;
                break;
            }
            cum += c;
        }
        below = cum;
    }
    bin = __shfl_sync(0xffffffffu, bin, owner);
    below = __shfl_sync(0xffffffffu, below, owner);
    __syncwarp();
    for (int i = lane; i < nb; i += 32) sel->hist[i] = 0;
    if (lane == 0) {
        sel->prefix = pass == 0 ? (unsigned int)bin : (sel->prefix << 10) | (unsigned int)bin;
        sel->rank = rank - below;
    }
}

// The largest (MAX) or smallest magnitude's bit pattern into sel->prefix, which
// the host initialises to 0 (MAX) or 0xffffffff (MIN).
template <bool MAX>
__global__ void __launch_bounds__(kQThreads) k_quant_extreme(const float* __restrict__ x, size_t N, size_t d,
                                                             const float* __restrict__ shift, QuantSelect* sel) {
    unsigned int best = MAX ? 0u : 0xffffffffu;
    auto take = [&](unsigned int b) { best = MAX ? max(best, b) : min(best, b); };
    const size_t nthr = (size_t)gridDim.x * blockDim.x;
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t N4 = N / 4;
    if (t < N4) {
        float s[4];
#pragma unroll
        for (int i = 0; i < 4; i++) s[i] = shift[(4 * t + i) % d];
        const float4* x4 = reinterpret_cast<const float4*>(x);
        auto take4 = [&](const float4& v) {
            take(quant_mag_bits(v.x, s[0]));
            take(quant_mag_bits(v.y, s[1]));
            take(quant_mag_bits(v.z, s[2]));
            take(quant_mag_bits(v.w, s[3]));
        };
        size_t g = t;
        for (; g + 3 * nthr < N4; g += 4 * nthr) {  // four loads in flight
            const float4 a = __ldg(x4 + g), b = __ldg(x4 + g + nthr), c = __ldg(x4 + g + 2 * nthr),
                         e = __ldg(x4 + g + 3 * nthr);
            take4(a);
            take4(b);
            take4(c);
            take4(e);
        }
        for (; g < N4; g += nthr) take4(__ldg(x4 + g));
    }
    if (t < N - 4 * N4) {
        const size_t e = 4 * N4 + t;
        take(quant_mag_bits(x[e], shift[e % d]));
    }
    for (int o = 16; o; o >>= 1) {
        const unsigned int v = __shfl_xor_sync(0xffffffffu, best, o);
        best = MAX ? max(best, v) : min(best, v);
    }
    if ((threadIdx.x & 31) == 0) {
        if (MAX) atomicMax(&sel->prefix, best);
        else atomicMin(&sel->prefix, best);
    }
}

// One code, and whether the value clips: src/quantize.rs:69 and :91.
__device__ __forceinline__ int quant_code(float v, float s, float scale, unsigned int& clipped) {
    const float y = __fmul_rn(__fsub_rn(v, s), scale);
    clipped += !(y >= -128.5f && y < 127.5f);
    if (y != y) return 0;  // NaN: the saturating cast gives 0
    return (int)fminf(fmaxf(roundf(y), -128.f), 127.f);
}

// Encode 16 elements per thread and step (four float4 loads, one 16-byte store);
// the host sizes the grid so that 16 x threads in the grid is a multiple of d.
// codes may be null (count only); clipped may be null (codes only).
__global__ void __launch_bounds__(kQThreads) k_quant_encode(const float* __restrict__ x, size_t N, size_t d,
                                                            const float* __restrict__ shift, float scale,
                                                            int8_t* __restrict__ codes,
                                                            unsigned long long* __restrict__ clipped) {
    const size_t nthr = (size_t)gridDim.x * blockDim.x;
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t N16 = N / 16;
    unsigned int clip = 0;
    if (t < N16) {
        float s[16];
#pragma unroll
        for (int i = 0; i < 16; i++) s[i] = shift[(16 * t + i) % d];
        const float4* x4 = reinterpret_cast<const float4*>(x);
        for (size_t g = t; g < N16; g += nthr) {
            float v[16];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float4 f = __ldcs(x4 + 4 * g + q);
                v[4 * q] = f.x;
                v[4 * q + 1] = f.y;
                v[4 * q + 2] = f.z;
                v[4 * q + 3] = f.w;
            }
            uint32_t w[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                uint32_t packed = 0;
#pragma unroll
                for (int i = 0; i < 4; i++)
                    packed |= (uint32_t)(quant_code(v[4 * q + i], s[4 * q + i], scale, clip) & 0xff) << (8 * i);
                w[q] = packed;
            }
            if (codes) __stcs(reinterpret_cast<uint4*>(codes) + g, make_uint4(w[0], w[1], w[2], w[3]));
        }
    }
    if (t < N - 16 * N16) {
        const size_t e = 16 * N16 + t;
        const int c = quant_code(x[e], shift[e % d], scale, clip);
        if (codes) codes[e] = (int8_t)c;
    }
    if (clipped) {
        for (int o = 16; o; o >>= 1) clip += __shfl_xor_sync(0xffffffffu, clip, o);
        if ((threadIdx.x & 31) == 0 && clip) atomicAdd(clipped, (unsigned long long)clip);
    }
}

// Int8Quantizer::decode, src/quantize.rs:76-79: v * (1 / scale) + s, two
// separately rounded operations (inv is the host's correctly rounded 1 / scale).
__global__ void k_quant_decode(const float* __restrict__ codes, size_t N, size_t d, const float* __restrict__ shift,
                               float inv, float* __restrict__ out) {
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < N; e += (size_t)gridDim.x * blockDim.x)
        out[e] = __fadd_rn(__fmul_rn(codes[e], inv), shift[e % d]);
}

}  // namespace emb
