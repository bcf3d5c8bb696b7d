// Attention of a LLaMA prompt step (many query rows at once) over the un-rotated f16 cache: mhsa.comp, softmax.comp and
// kqv_matching.comp of the reference as matrix products in one launch.
//
// attention_fused_kernel (attention.cu) gives every query row CTAs of its own, which read and rotate the whole cache once per
// row: at 64 rows and 1024 positions 1.07 GB of cache rows pass through L2 and half a billion key values are rotated per layer.
// Here a cluster holds one head and up to 64 query rows; a CTA takes 128 keys, rotates each once and multiplies it with all rows:
//
//   S = Q K^T     A = queries, B = keys, both as f16 pairs hi + lo (22 bits): q_hi k_hi + q_lo k_hi + q_hi k_lo
//   O = P V       A = probabilities as f16 pairs, B = values, f16 as they are in the cache
//
// with f32 sums.  The lo halves keep their bits because queries and keys are scaled by a power of two per row and the probabilities by 2^15,
// and the sums of 16 values that a tensor-core instruction forms (it truncates) are added by ordinary f32 additions.  Relative error of the
// outputs against 64 bits, scores of rms 1, 32 heads, attention_fused_kernel / here (one long chain of sums, keys as they are):
//   positions      0 .. 63              192 .. 255           900 .. 963           1900 .. 1963
//                  1.4e-7 / 2.0e-7      5.9e-7 / 5.8e-7      2.57e-6 / 2.48e-6    6.1e-6 / 5.9e-6      for keys of any size from 2^-14 to 2^12
//                  (4.7e-7)             (8.5e-7)             (2.8e-6)                                  (and 4e-4 for keys of size 2^-14)
// The operands are 64 rows high and a CTA has one pass over 128 keys: nothing to pipeline, and half a tcgen05 tile, so these are mma.sync.
//
// Rotation: the score of query z (position P + z) and key p turns by the distance P + z - p.  Both are turned from one position, queries forwards and
// keys backwards, so no row of the table is needed per pair.
// A warp owns 16 keys: a thread reads its part of two key rows from shared memory (raw rows, brought by bulk copies) -- the order of the head's
// 128 values is free as long as Q uses the same one --, turns pairs in f32 and splits them in registers.
//
// The softmax of a CTA's keys needs the maximum over its eight warps (one exchange), the CTAs of the cluster meet once at the end
// through distributed shared memory, each finishing its share of the rows.  No scratch, no counters.
//
// Bound by latency.  Between the launches of a 7B session (32 heads, 64 rows, 1024 positions) a launch takes 20 to 24 us, 38 where a CTA has a second chunk
// of keys: 5 to the queries in fragments, 7 for the scores, 2.5 softmax, 3 values, 4 the meeting of the cluster.  It took 40 to 48: of 32 clusters of 8 CTAs two ran
// after the others (see launch_attention_prompt), the queries took 7 (unrolled code, rows of the table from HBM).  Two CTAs per SM hide some of it behind each other.
#include <math.h>

#include <algorithm>

#include "attention_gqa.cuh"
#include "common.cuh"
#include "ctx.h"

namespace lv {

constexpr int kApQ = 64, kApKeys = 128, kApHead = 128, kApThreads = 256, kApWarps = kApThreads / 32;
constexpr uint32_t kApMaxCluster = 8;
constexpr uint32_t kApStride = kApHead * 2 + 16;                        // bytes of a key or value row: eight rows of an ldmatrix fall into different banks
constexpr uint32_t kApPlane = (kApQ / 16) * (kApHead / 16) * 32 * 16;   // one f16 plane of 64 x 128 values in fragment order: 16384
constexpr uint32_t kApQBytes = 2 * kApPlane, kApRowBytes = kApKeys * kApStride;
static_assert(2 * kApPlane <= kApRowBytes, "the probabilities of a chunk take the place of its keys");
constexpr uint32_t kApOStride = kApHead + 8;                            // floats
constexpr uint32_t kApRedBytes = (2 * kApWarps + 5) * kApQ * 4;
constexpr size_t kApSmemBytes = kApQBytes + 2 * kApRowBytes + kApRedBytes;      // two CTAs per SM
static_assert(size_t(kApQ) * kApOStride * 4 <= kApRowBytes, "the outputs of a CTA take the place of its values");
constexpr float kApLog2e = 1.4426950408889634f;
constexpr float kApPScale = 15.f;                                       // log2: probabilities as f16 pairs keep 22 bits down to 2^-17, 11 down to 2^-29

__device__ __forceinline__ void ap_mma(float (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// (x, y) -> f16 pairs hi, lo with hi + lo = (x, y) to 22 bits
__device__ __forceinline__ void ap_split(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// the two halves of w, 0 in place of one that is not finite
__device__ __forceinline__ uint32_t ap_finite(uint32_t w) {
    if ((w & 0x7c00u) == 0x7c00u) w &= 0xffff0000u;
    if ((w & 0x7c000000u) == 0x7c000000u) w &= 0x0000ffffu;
    return w;
}

// (cos, sin) of two pairs at the distance d (sin turns its sign with it), from the table
__device__ __forceinline__ float4 ap_table_row(const float* table, int d, uint32_t dim) {
    float4 w = *reinterpret_cast<const float4*>(table + size_t(abs(d)) * kApHead + dim);
    if (d < 0) { w.y = -w.y; w.w = -w.w; }
    return w;
}
__device__ __forceinline__ float4 ap_add_angles(const float4& a, const float4& b) {
    return make_float4(fmaf(a.x, b.x, -(a.y * b.y)), fmaf(a.y, b.x, a.x * b.y), fmaf(a.z, b.z, -(a.w * b.w)), fmaf(a.w, b.z, a.z * b.w));
}

// The order of the head's values in the fragments: step ks of thread t holds the four from ap_first_dim(ks, t) on; eight lanes (two key
// rows, four threads) that read 16 bytes of their rows hit different banks.
__device__ __forceinline__ uint32_t ap_first_dim(uint32_t ks, uint32_t t) { return 64 * (ks >> 2) + 16 * t + 8 * ((ks >> 1) & 1) + 4 * (ks & 1); }

// xh: the outputs go there as split activations of zpad rows (lv_act_split_f16) instead of to out
// grid (heads, C, ceil(batch / 64)), clusters of (1, C, 1): CTA `rank` takes the 128-key chunks rank, rank + C, ...; ONE_PASS: C chunks at most
template <bool ONE_PASS>
__global__ void __launch_bounds__(kApThreads, 2) attention_prompt_kernel(float* __restrict__ out, const float* __restrict__ q,
                                                                         const __half* __restrict__ kc, const __half* __restrict__ vc,
                                                                         const uint32_t* __restrict__ pos, const float* __restrict__ table,
                                                                         uint32_t heads, uint32_t batch, uint32_t max_ctx, float scale, uint32_t* err,
                                                                         __half* __restrict__ xh, uint32_t zpad) {
    pdl_launch_dependents();
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* s_q = smem;                                            // [plane][m tile][k step][lane][16 bytes]
    uint8_t* s_v = s_q + kApQBytes;
    uint8_t* s_k = s_v + kApRowBytes;                               // keys, then probabilities [plane][m tile][warp][lane][16 bytes]
    float* s_max = reinterpret_cast<float*>(s_k + kApRowBytes);     // [warp][row]
    float* s_sum = s_max + kApWarps * kApQ;                         // [warp][row]
    float* s_m = s_sum + kApWarps * kApQ;                           // row maximum (read by the cluster)
    float* s_l = s_m + kApQ;                                        // row sum (read by the cluster)
    float* s_f = s_l + kApQ;                                        // factor of the old outputs
    float* s_qf = s_f + kApQ;                                       // scores -> log2 units
    float* s_o = reinterpret_cast<float*>(s_v);                     // [row][kApOStride], after the last product
    __shared__ __align__(8) uint64_t s_bar[2];                      // keys, values

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t h = blockIdx.x, rank = blockIdx.y, C = gridDim.y, dim = heads * kApHead;
    const uint32_t z0 = blockIdx.z * kApQ;
    if (threadIdx.x < 2) {
        mbar_init(&s_bar[threadIdx.x], 1);
        fence_mbar_init();
    }
    if (threadIdx.x < kApQ) {
        s_m[threadIdx.x] = -INFINITY;
        s_l[threadIdx.x] = 0.f;
    }
    const uint32_t c_max = (max_ctx - 1) >> 5;
    {
        // Table rows, keys and values are in HBM more often than not (a layer's weights pass through L2 between two of its steps): what this CTA will
        // read is on its way to L2 before the previous kernel has ended.  A hint: the position may be that of an earlier step.
        const uint32_t guess = min(__ldcg(pos), max_ctx - 1) + z0, p0 = rank * kApKeys, i = threadIdx.x & (kApKeys - 1);
        if (p0 + i <= guess && p0 + i < max_ctx) l2_prefetch((threadIdx.x < kApKeys ? kc : vc) + size_t(p0 + i) * dim + h * kApHead, kApHead * sizeof(__half));
        if (threadIdx.x == 0) l2_prefetch(table, min(17u, max_ctx) * kApHead * 4);
        const uint32_t c0 = guess >> 5, c = (p0 + 16 * warp + 16) >> 5;
        if (lane == 0) l2_prefetch(table + size_t(32 * min(c0 > c ? c0 - c : c - c0, c_max)) * kApHead, kApHead * 4);
        if (lane == 1 && warp < 3) l2_prefetch(table + size_t(32 * min(uint32_t(warp), c_max)) * kApHead, kApHead * 4);
    }
    __syncthreads();
    pdl_wait();
    const uint32_t P = *pos + z0;                                   // position of this tile's first row
    const uint32_t want = min(uint32_t(kApQ), batch - z0);
    // rows whose position lies outside the caches and the rotation table are reported and left out
    const uint32_t nq = P >= max_ctx ? 0u : min(want, max_ctx - P);
    if (nq < want && threadIdx.x == 0 && h == 0 && rank == 0) atomicOr(err, ERR_BAD_INDEX);
    if (nq == 0) return;                                            // (the same for the whole cluster)
    const uint32_t last = P + nq - 1, n_chunks = last / kApKeys + 1, n_mt = (nq + 31) / 32 * 2;      // tiles of 16 rows, in pairs
    const uint32_t active = min(C, n_chunks);                       // CTAs of the cluster that have keys
    bool ok = true;

    auto load_rows = [&](uint32_t p0) {                             // rows beyond the last position: any finite row, their weights are 0
        if (threadIdx.x < 2) mbar_expect_tx(&s_bar[threadIdx.x], kApKeys * kApHead * uint32_t(sizeof(__half)));
        const uint32_t i = threadIdx.x & (kApKeys - 1);
        const size_t row = size_t(min(p0 + i, last)) * dim + h * kApHead;
        if (threadIdx.x < kApKeys) bulk_g2s(s_k + i * kApStride, kc + row, kApHead * sizeof(__half), &s_bar[0]);
        else bulk_g2s(s_v + i * kApStride, vc + row, kApHead * sizeof(__half), &s_bar[1]);
    };
    static_assert(kApThreads == 2 * kApKeys, "one key and one value row per pair of threads");
    // Angles: position 32 c + d, |d| <= 16 where the table has the rows, is turned from 32 c0 by the table rows of 32 (c - c0) and of d, queries forwards
    // and keys backwards.  (The table's angles are rounded products of distance and frequency: rows of few distances, mostly small or powers
    // of two times 32, keep that error below that of a row of any distance.)
    const uint32_t c0 = P >> 5;
    float4 far[4];                                                  // of this warp's 32 positions, four steps ahead
    auto load_far = [&](uint32_t p0, uint32_t ks, int i) {
        far[i] = ap_table_row(table, int(32 * c0) - int(32 * min((p0 + 16 * warp + 16) >> 5, c_max)), ap_first_dim(ks, t));
    };
    auto load_first_far = [&](uint32_t p0) {
        if (p0 + 16 * warp > last) return;
#pragma unroll
        for (int i = 0; i < 4; ++i) load_far(p0, i, i);
    };
    if (rank < n_chunks) {
        load_rows(rank * kApKeys);
        // ---- queries: turned by their row, scaled by a power of two so that the largest value of a row is in [1024, 2048) --------
        // Two rows of a warp at a time, the next two on their way: all rows at once are unrolled code that runs once (6 us, most of it instruction fetches).
        constexpr int kRows = 2;
        float4 x[kRows], near[kRows], far[kRows];
        auto fetch = [&](uint32_t r0) {
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const uint32_t r = r0 + i * kApWarps;
                x[i] = near[i] = far[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r >= nq) continue;
                const uint32_t c = min((P + r + 16) >> 5, c_max);
                x[i] = *reinterpret_cast<const float4*>(q + size_t(z0 + r) * dim + h * kApHead + 4 * lane);
                near[i] = ap_table_row(table, int(P + r) - int(32 * c), 4 * lane);
                far[i] = ap_table_row(table, int(32 * (c - c0)), 4 * lane);
            }
        };
        fetch(warp);
#pragma unroll 1
        for (uint32_t r0 = warp; r0 < 16 * n_mt; r0 += kRows * kApWarps) {
            float4 v[kRows];
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const float4 w = ap_add_angles(far[i], near[i]);
                v[i] = make_float4(w.x * x[i].x - w.y * x[i].y, w.y * x[i].x + w.x * x[i].y, w.z * x[i].z - w.w * x[i].w, w.w * x[i].z + w.z * x[i].w);
            }
            fetch(r0 + kRows * kApWarps);
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const uint32_t r = r0 + i * kApWarps;
                const float top = warp_max(fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w))));
                const uint32_t e = max(__float_as_uint(top) >> 23, 11u);
                const float up = __uint_as_float((264u - e) << 23), down = __uint_as_float((e - 10u) << 23);      // 2^(137 - e), 2^(e - 137)
                if (lane == 0) s_qf[r] = down * scale * kApLog2e;
                uint32_t hi0, lo0, hi1, lo1;
                ap_split(v[i].x * up, v[i].y * up, hi0, lo0);
                ap_split(v[i].z * up, v[i].w * up, hi1, lo1);
                // ap_first_dim(ks, t4) == 4 lane; rows 8 .. 15 of a tile are words 1 and 3 of a fragment
                const uint32_t ks = 4 * (lane >> 4) + 2 * ((lane >> 1) & 1) + (lane & 1), t4 = (lane >> 2) & 3;
                uint32_t* at = reinterpret_cast<uint32_t*>(s_q + (((r >> 4) * 8 + ks) * 32 + (r & 7) * 4 + t4) * 16) + ((r >> 3) & 1);
                at[0] = hi0;
                at[2] = hi1;
                at[kApPlane / 4] = lo0;
                at[kApPlane / 4 + 2] = lo1;
            }
        }
        load_first_far(rank * kApKeys);
    }
    __syncthreads();

    float o[4][2][4];                                               // rows 16 i + g, + 8; dims 16 warp + 8 j + 2 t, + 1
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) o[i][j][c] = 0.f;

    uint32_t phase = 0;
    for (uint32_t chunk = rank; chunk < n_chunks; chunk += C) {
        const uint32_t p0 = chunk * kApKeys, my0 = p0 + 16 * warp;  // this warp's 16 keys
        float s[4][2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int c = 0; c < 4; ++c) s[i][j][c] = 0.f;
        ok = mbar_wait_warp(&s_bar[0], phase, err) && ok;
        float key_unit[2][2] = {{1.f, 1.f}, {1.f, 1.f}};            // of the keys 8 j + 2 t + c
        if (my0 <= last) {
            // a key is scaled by a power of two so that its largest value is in [2048, 4096): turned it stays inside f16, and its lo half
            // keeps its bits
            const uint8_t* key[2];
            float up[2];
            int near[2];                                                            // from the keys to the table row of their 32 positions
            const uint32_t c = min((my0 + 16) >> 5, c_max);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                key[j] = s_k + (16 * warp + 8 * j + g) * kApStride;
                __half2 top = __half2{};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 w = *reinterpret_cast<const uint4*>(key[j] + 128 * (i >> 1) + 32 * t + 16 * (i & 1));
                    const __half2* h2 = reinterpret_cast<const __half2*>(&w);
                    top = __hmax2(top, __hmax2(__hmax2(__habs2(h2[0]), __habs2(h2[1])), __hmax2(__habs2(h2[2]), __habs2(h2[3]))));
                }
                float m = fmaxf(__low2float(top), __high2float(top));
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
                near[j] = int(32 * c) - int(min(my0 + 8 * j + g, last));
                const uint32_t e = max(__float_as_uint(m) >> 23, 103u);            // (2^-24 is the smallest f16)
                up[j] = __uint_as_float((265u - e) << 23);                          // 2^(138 - e)
                const float down = __uint_as_float((e - 11u) << 23);                // 2^(e - 138)
#pragma unroll
                for (int c = 0; c < 2; ++c) key_unit[j][c] = __shfl_sync(0xffffffffu, down, 4 * (2 * t + c));
            }
#pragma unroll 1
            for (uint32_t half = 0; half < 2; ++half) {
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4) {
                    const uint32_t ks = 4 * half + k4;
                    uint32_t bh[2][2], bl[2][2];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint2 w = *reinterpret_cast<const uint2*>(key[j] + 2 * ap_first_dim(ks, t));
                        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
                        const float4 f = ap_add_angles(far[k4], ap_table_row(table, near[j], ap_first_dim(ks, t)));      // mhsa.comp:50-54
                        const float cos0 = up[j] * f.x, sin0 = up[j] * f.y, cos1 = up[j] * f.z, sin1 = up[j] * f.w;
                        ap_split(cos0 * a.x + sin0 * a.y, cos0 * a.y - sin0 * a.x, bh[j][0], bl[j][0]);
                        ap_split(cos1 * b.x + sin1 * b.y, cos1 * b.y - sin1 * b.x, bh[j][1], bl[j][1]);
                    }
                    if (half == 0) load_far(p0, 4 + k4, k4);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (uint32_t(i) >= n_mt) break;
                        const uint8_t* at = s_q + ((i * 8 + ks) * 32 + lane) * 16;
                        const uint4 ah = *reinterpret_cast<const uint4*>(at), al = *reinterpret_cast<const uint4*>(at + kApPlane);
                        // the tensor core's sums truncate: those of 16 values each are added here
                        float d[2][4] = {};
#pragma unroll
                        for (int j = 0; j < 2; ++j) ap_mma(d[j], al, bh[j][0], bh[j][1]);
#pragma unroll
                        for (int j = 0; j < 2; ++j) ap_mma(d[j], ah, bl[j][0], bl[j][1]);
#pragma unroll
                        for (int j = 0; j < 2; ++j) ap_mma(d[j], ah, bh[j][0], bh[j][1]);
#pragma unroll
                        for (int j = 0; j < 2; ++j)
#pragma unroll
                            for (int c = 0; c < 4; ++c) s[i][j][c] += d[j][c];
                    }
                }
            }
        }
        // ---- softmax: scores in log2 units, masked; the maximum of a row over the chunk ------------------------------
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (uint32_t(i) >= n_mt) break;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t r = 16 * i + g + 8 * u;
                const float f = s_qf[r];
                float top = -INFINITY;
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        float& x = s[i][j][2 * u + c];
                        x = my0 + 8 * j + 2 * t + c <= P + r ? x * (f * key_unit[j][c]) : -INFINITY;
                        top = fmaxf(top, x);
                    }
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
                if (t == 0) s_max[warp * kApQ + r] = top;
            }
        }
        __syncthreads();
        if (threadIdx.x < 16 * n_mt) {
            const uint32_t r = threadIdx.x;
            const float old = s_m[r];
            float m = old;
#pragma unroll
            for (int w = 0; w < kApWarps; ++w) m = fmaxf(m, s_max[w * kApQ + r]);
            s_m[r] = m;
            s_f[r] = old == -INFINITY ? 0.f : exp2f(old - m);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (uint32_t(i) >= n_mt) break;
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t r = 16 * i + g + 8 * u;
                const float m = s_m[r], base = m == -INFINITY ? 0.f : m - kApPScale, f = s_f[r];
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float e0 = exp2f(s[i][j][2 * u] - base), e1 = exp2f(s[i][j][2 * u + 1] - base);
                    sum += e0 + e1;
                    ap_split(e0, e1, hi[2 * j + u], lo[2 * j + u]);       // a0: rows g, keys 2t; a1: rows g + 8; a2, a3: keys + 8
                    o[i][j][2 * u] *= f;
                    o[i][j][2 * u + 1] *= f;
                }
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                if (t == 0) s_sum[warp * kApQ + r] = sum;
            }
            uint8_t* at = s_k + ((i * 8 + warp) * 32 + lane) * 16;
            *reinterpret_cast<uint4*>(at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(at + kApPlane) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
        ok = mbar_wait_warp(&s_bar[1], phase, err) && ok;
        phase ^= 1u;
        __syncthreads();
        if (threadIdx.x < 16 * n_mt) {
            const uint32_t r = threadIdx.x;
            float l = s_l[r] * s_f[r];
#pragma unroll
            for (int w = 0; w < kApWarps; ++w) l += s_sum[w * kApQ + r];
            s_l[r] = l;
        }
        // ---- values: warp w owns dims 16 w ..; a step is the 16 keys of one warp ---------------------------------------
        const uint32_t steps = min(uint32_t(kApWarps), (last - p0) / 16 + 1);
        auto load_values = [&](uint32_t (&b)[4], uint32_t ks) {
            const uint32_t vrow = smem_u32(s_v + (16 * ks + (lane & 15)) * kApStride + (16 * warp + (lane >> 4) * 8) * 2);
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(vrow) : "memory");
        };
        // A row must not depend on keys behind it, and a probability of 0 does not take a value out of a product that is not finite (an entry
        // of the cache that left the range of f16).  So a warp looks for such values in chunks with keys that some row does not see, leaves
        // them out of the products and adds them below to the rows that see them.  0 x value is NaN for them and stays so in a sum.
        const bool look = p0 + kApKeys - 1 > P;
        bool odd = false;
        auto look_at = [](__half2& seen, const uint32_t (&b)[4]) {
#pragma unroll
            for (int i = 0; i < 4; ++i) seen = __hfma2(*reinterpret_cast<const __half2*>(&b[i]), __half2{}, seen);
        };
        auto is_odd = [](__half2 seen) { return __any_sync(0xffffffffu, __hisnan(__low2half(seen)) || __hisnan(__high2half(seen))) != 0; };
        if (!ONE_PASS && look) {
            __half2 seen = {};
            for (uint32_t ks = 0; ks < steps; ++ks) {
                uint32_t b[4];
                load_values(b, ks);
                look_at(seen, b);
            }
            odd = is_odd(seen);
        }
        while (true) {
            __half2 seen = {};
#pragma unroll 1
            for (uint32_t ks = 0; ks < steps; ++ks) {
                uint32_t b[4];
                load_values(b, ks);
                if (ONE_PASS) look_at(seen, b);
                if (odd) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) b[i] = ap_finite(b[i]);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (uint32_t(i) >= n_mt) break;
                    const uint8_t* at = s_k + ((i * 8 + ks) * 32 + lane) * 16;
                    const uint4 ah = *reinterpret_cast<const uint4*>(at), al = *reinterpret_cast<const uint4*>(at + kApPlane);
                    float d[2][4] = {};
#pragma unroll
                    for (int j = 0; j < 2; ++j) ap_mma(d[j], al, b[2 * j], b[2 * j + 1]);
#pragma unroll
                    for (int j = 0; j < 2; ++j) ap_mma(d[j], ah, b[2 * j], b[2 * j + 1]);
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int c = 0; c < 4; ++c) o[i][j][c] += d[j][c];
                }
            }
            if (!ONE_PASS || !look || odd || !is_odd(seen)) break;
            odd = true;                                             // once more, without them
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int c = 0; c < 4; ++c) o[i][j][c] = 0.f;
        }
        if (odd) {
            for (uint32_t k = 0; k < 16 * steps; ++k) {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const uint32_t v = *reinterpret_cast<const uint32_t*>(s_v + k * kApStride + 2 * (16 * warp + 8 * j + 2 * t));
                    const uint32_t f = v ^ ap_finite(v);            // what was left out
                    if (f == 0) continue;
                    const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&f));
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            if (uint32_t(i) >= n_mt || p0 + k > P + 16 * i + g + 8 * u) continue;
                            // the probability of row 16 i + g + 8 u and key k in the fragments
                            const uint8_t* at = s_k + ((i * 8 + (k >> 4)) * 32 + 4 * g + ((k & 7) >> 1)) * 16 + (2 * ((k >> 3) & 1) + u) * 4 + 2 * (k & 1);
                            const float e = __half2float(*reinterpret_cast<const __half*>(at)) + __half2float(*reinterpret_cast<const __half*>(at + kApPlane));
                            if ((f & 0xffffu) != 0) o[i][j][2 * u] = fmaf(e, x.x, o[i][j][2 * u]);
                            if ((f >> 16) != 0) o[i][j][2 * u + 1] = fmaf(e, x.y, o[i][j][2 * u + 1]);
                        }
                }
            }
        }
        if (!ONE_PASS) fence_proxy_async();                         // the next keys come by bulk copies into bytes that were written by stores
        __syncthreads();                                            // values and probabilities are used up
        if (ONE_PASS) break;
        if (chunk + C < n_chunks) {
            load_rows((chunk + C) * kApKeys);
            load_first_far((chunk + C) * kApKeys);
        }
    }

    if (C == 1) {                                                   // no other CTA has keys of these rows
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t r = 16 * i + g + 8 * u;
                if (r >= nq || !ok) continue;
                const float f = 1.f / s_l[r];
                float* to = out + size_t(z0 + r) * dim + h * kApHead + 16 * warp + 2 * t;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float v[2] = {o[i][j][2 * u] * f, o[i][j][2 * u + 1] * f};
                    if (xh != nullptr) split_store_n<2>(xh, zpad, z0 + r, h * kApHead + 16 * warp + 2 * t + 8 * j, v);
                    else *reinterpret_cast<float2*>(to + 8 * j) = make_float2(v[0], v[1]);
                }
            }
        return;
    }
    // ---- the CTAs of the cluster meet -------------------------------------------------------------------------
    if (rank < active) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (uint32_t(i) >= n_mt) break;
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    *reinterpret_cast<float2*>(s_o + (16 * i + g + 8 * u) * kApOStride + 16 * warp + 8 * j + 2 * t) = make_float2(o[i][j][2 * u], o[i][j][2 * u + 1]);
        }
    }
    cluster_sync();
    for (uint32_t r = rank + C * warp; r < nq && ok; r += C * kApWarps) {          // a warp finishes a row: four values per lane
        float m = -INFINITY, l = 0.f;
        if (uint32_t(lane) < active) {
            m = cluster_load(s_m + r, lane);
            l = cluster_load(s_l + r, lane);
        }
        const float top = warp_max(m), w = m == -INFINITY ? 0.f : exp2f(m - top);
        const float den = warp_sum(l * w);
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f), part[kApMaxCluster];
        const float* mine = s_o + r * kApOStride + 4 * lane;
#pragma unroll
        for (uint32_t c = 0; c < kApMaxCluster; ++c) part[c] = c < active ? cluster_load4(mine, c) : sum;
#pragma unroll
        for (uint32_t c = 0; c < kApMaxCluster; ++c) {
            const float f = __shfl_sync(0xffffffffu, w, c);
            sum.x = fmaf(part[c].x, f, sum.x);
            sum.y = fmaf(part[c].y, f, sum.y);
            sum.z = fmaf(part[c].z, f, sum.z);
            sum.w = fmaf(part[c].w, f, sum.w);
        }
        const float v[4] = {sum.x / den, sum.y / den, sum.z / den, sum.w / den};
        if (xh != nullptr) split_store_n<4>(xh, zpad, z0 + r, h * kApHead + 4 * lane, v);
        else *reinterpret_cast<float4*>(out + size_t(z0 + r) * dim + h * kApHead + 4 * lane) = make_float4(v[0], v[1], v[2], v[3]);
    }
    cluster_sync();                                      // no CTA leaves while another reads its shared memory
}

int attention_prompt_configure(lv_ctx* ctx) {
    LV_REQUIRE(size_t(ctx->max_smem_optin) >= kApSmemBytes + 1024, "device has too little shared memory for the prompt attention kernel");
    LV_CUDA(cudaFuncSetAttribute(attention_prompt_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kApSmemBytes)));
    LV_CUDA(cudaFuncSetAttribute(attention_prompt_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kApSmemBytes)));
    for (uint32_t c = 1; c <= kApMaxCluster; ++c) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(1, c);
        cfg.blockDim = dim3(kApThreads);
        cfg.dynamicSmemBytes = kApSmemBytes;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1;
        attr[0].val.clusterDim.y = c;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        LV_CUDA(cudaOccupancyMaxActiveClusters(&n, attention_prompt_kernel<false>, &cfg));
        ctx->ap_clusters[c] = uint32_t(n);
    }
    return LV_OK;
}

int launch_attention_prompt(lv_ctx* ctx, float* out, const float* q, const void* k_cache, const void* v_cache, const uint32_t* pos,
                            const float* rope_table, uint32_t heads, uint32_t max_ctx, uint32_t batch, void* xh) {
    const uint32_t chunks = (max_ctx + kApKeys - 1) / kApKeys, tiles = (batch + kApQ - 1) / kApQ;
    // Clusters so small that all of them run at a time, where that is possible: between the launches of a session two of 32 clusters of 8 had to wait for the others
    // to end (40 us where 24 were needed), and in clusters of 7 only the last of 1024 positions take a second pass (10 us).  Next to other kernels a tenth
    // fewer find room than the device holds on its own (there 32 clusters of 8 do run at a time: 27 us at 960 positions, 40 in clusters of 7).
    // ms of a prompt of six layers, clusters of 8 / 7 / 6 / 5 / 4: 32 heads, 1984 tokens in steps of 64 28.3 / 25.0 / 25.5 / 25.9 / 27.0; 40 heads, 1024 tokens 16.5 /
    // 16.6 / 15.2 / 15.2 / 15.5, 1984 tokens 34.8 / 35.0 / 30.8 / 31.3 / 32.2; 16 heads, 1984 tokens 17.0 / 17.5 / 17.9 / 18.6 / 19.5.  A launch of 52 heads on its
    // own, 64 rows at 960 of 1024 / 1900 of 2048 positions: 48.8 / 79.2 us in clusters of 8, 40.4 / 68.2 in clusters of 4.
    uint32_t C = std::min(kApMaxCluster, chunks);
    for (uint32_t c = C; c >= 4; --c)
        if (10 * heads * tiles <= 9 * ctx->ap_clusters[c]) {
            C = c;
            break;
        }
    auto* kernel = chunks <= C ? attention_prompt_kernel<true> : attention_prompt_kernel<false>;
    LV_CUDA(launch_pdl_cluster(ctx, kernel, dim3(heads, C, tiles), dim3(kApThreads), dim3(1, C), kApSmemBytes, out, q,
                               static_cast<const __half*>(k_cache), static_cast<const __half*>(v_cache), pos, rope_table, heads, batch, max_ctx,
                               1.0f / sqrtf(float(kApHead)), ctx->d_err, static_cast<__half*>(xh), (batch + 15u) & ~15u));
    return LV_OK;
}

}  // namespace lv
