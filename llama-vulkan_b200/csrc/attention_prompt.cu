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
// with f32 sums, so scores and probabilities are as exact as the f32 arithmetic of attention_fused_kernel.  The operands are 64
// rows high and a CTA has one pass over 128 keys: nothing to pipeline, and half a tcgen05 tile, so these are mma.sync.
//
// Rotation: the score of query z (position P + z) and key p turns by the distance P + z - p.  Keys are turned by P - p, with the
// table row of that distance (the sign of sin is flipped for p > P), and queries by z, so no row of the table is needed per pair.
// A warp owns 16 keys: a thread reads its part of two key rows from shared memory (raw rows, brought by bulk copies) in 16-byte loads
// -- the order of the head's 128 values is free as long as Q uses the same one --, turns pairs in f32 and splits them in registers.
//
// The softmax of a CTA's keys needs the maximum over its eight warps (one exchange), the CTAs of the cluster meet once at the end
// through distributed shared memory, each finishing its share of the rows.  No scratch, no counters.
//
// Bound by latency: 64 rows at 1000 positions take 24.5 us (237 before), of which the matrix products are 5; 2 are the query preparation,
// 3 the softmax's exchanges, 4 the meeting of the cluster.  Two CTAs per SM hide some of it behind each other.
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
constexpr float kApPScale = 12.f;                                       // log2: probabilities as f16 pairs keep 22 bits down to 2^-26

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

// four floats in the shared memory of another CTA of the cluster
__device__ __forceinline__ float4 ap_cluster_load4(const float* local, uint32_t rank) {
    uint32_t at;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at));
    return v;
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
    float4 cs[2][2][4];                                             // table rows of this thread's two keys: [half][key][step]
    float turn[2];
    auto load_table = [&](uint32_t p0, int half) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint32_t p = min(p0 + 16 * warp + 8 * j + g, last);
            const float* row = table + size_t(p > P ? p - P : P - p) * kApHead;
            turn[j] = p > P ? -0.5f : 0.5f;
#pragma unroll
            for (int i = 0; i < 4; ++i) cs[half][j][i] = *reinterpret_cast<const float4*>(row + ap_first_dim(4 * half + i, t));
        }
    };
    if (rank < n_chunks) {
        load_rows(rank * kApKeys);
        // ---- queries: turned by their row, scaled by a power of two so that the largest value of a row is in [1024, 2048) --------
        constexpr int kRows = 4;                                    // rows of a warp at a time, all loads before the first use
        for (uint32_t r0 = warp; r0 < 16 * n_mt; r0 += kRows * kApWarps) {
            float4 x[kRows], w[kRows];
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const uint32_t r = r0 + i * kApWarps;
                x[i] = r < nq ? *reinterpret_cast<const float4*>(q + size_t(z0 + r) * dim + h * kApHead + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
                w[i] = r < nq ? *reinterpret_cast<const float4*>(table + size_t(r) * kApHead + 4 * lane) : x[i];
            }
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const uint32_t r = r0 + i * kApWarps;
                if (r >= 16 * n_mt) break;
                const float4 v = make_float4(w[i].x * x[i].x - w[i].y * x[i].y, w[i].y * x[i].x + w[i].x * x[i].y,
                                             w[i].z * x[i].z - w[i].w * x[i].w, w[i].w * x[i].z + w[i].z * x[i].w);
                const float top = warp_max(fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
                const uint32_t e = max(__float_as_uint(top) >> 23, 11u);
                const float up = __uint_as_float((264u - e) << 23), down = __uint_as_float((e - 10u) << 23);      // 2^(137 - e), 2^(e - 137)
                if (lane == 0) s_qf[r] = 2.f * down * scale * kApLog2e;       // (keys enter halved, see below)
                uint32_t hi0, lo0, hi1, lo1;
                ap_split(v.x * up, v.y * up, hi0, lo0);
                ap_split(v.z * up, v.w * up, hi1, lo1);
                // ap_first_dim(ks, t4) == 4 lane; rows 8 .. 15 of a tile are words 1 and 3 of a fragment
                const uint32_t ks = 4 * (lane >> 4) + 2 * ((lane >> 1) & 1) + (lane & 1), t4 = (lane >> 2) & 3;
                uint32_t* at = reinterpret_cast<uint32_t*>(s_q + (((r >> 4) * 8 + ks) * 32 + (r & 7) * 4 + t4) * 16) + ((r >> 3) & 1);
                at[0] = hi0;
                at[2] = hi1;
                at[kApPlane / 4] = lo0;
                at[kApPlane / 4 + 2] = lo1;
            }
        }
        load_table(rank * kApKeys, 0);
        if (ONE_PASS) load_table(rank * kApKeys, 1);                // (with several passes the outputs take the registers)
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
        if (my0 <= last) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                if (!ONE_PASS && half != 0) load_table(p0, 1);
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4) {
                    const int ks = 4 * half + k4;
                    uint32_t bh[2][2], bl[2][2];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint2 w = *reinterpret_cast<const uint2*>(s_k + (16 * warp + 8 * j + g) * kApStride + 2 * ap_first_dim(ks, t));
                        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
                        // mhsa.comp:50-54 with half the key, so that a turned value never leaves the range of f16
                        const float4 f = cs[half][j][k4];
                        const float c0 = 0.5f * f.x, s0 = turn[j] * f.y, c1 = 0.5f * f.z, s1 = turn[j] * f.w;
                        ap_split(c0 * a.x + s0 * a.y, c0 * a.y - s0 * a.x, bh[j][0], bl[j][0]);
                        ap_split(c1 * b.x + s1 * b.y, c1 * b.y - s1 * b.x, bh[j][1], bl[j][1]);
                    }
#pragma unroll
                    for (int i = 0; i < 4; i += 2) {                // two tiles of rows: four sums in turn, so that none waits for its last product
                        if (uint32_t(i) >= n_mt) break;
                        const uint8_t* at = s_q + ((i * 8 + ks) * 32 + lane) * 16;
                        const uint4 ah0 = *reinterpret_cast<const uint4*>(at), al0 = *reinterpret_cast<const uint4*>(at + kApPlane);
                        const uint4 ah1 = *reinterpret_cast<const uint4*>(at + 4096), al1 = *reinterpret_cast<const uint4*>(at + kApPlane + 4096);
#pragma unroll
                        for (int j = 0; j < 2; ++j) { ap_mma(s[i][j], al0, bh[j][0], bh[j][1]); ap_mma(s[i + 1][j], al1, bh[j][0], bh[j][1]); }
#pragma unroll
                        for (int j = 0; j < 2; ++j) { ap_mma(s[i][j], ah0, bl[j][0], bl[j][1]); ap_mma(s[i + 1][j], ah1, bl[j][0], bl[j][1]); }
#pragma unroll
                        for (int j = 0; j < 2; ++j) { ap_mma(s[i][j], ah0, bh[j][0], bh[j][1]); ap_mma(s[i + 1][j], ah1, bh[j][0], bh[j][1]); }
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
                        x = my0 + 8 * j + 2 * t + c <= P + r ? x * f : -INFINITY;
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
        // them out of the products and adds them below to the rows that see them.
        bool odd = false;
        if (p0 + kApKeys - 1 > P) {
            __half2 nan = __float2half2_rn(0.f);
            for (uint32_t ks = 0; ks < steps; ++ks) {
                uint32_t b[4];
                load_values(b, ks);
#pragma unroll
                for (int i = 0; i < 4; ++i) nan = __hfma2(*reinterpret_cast<const __half2*>(&b[i]), __float2half2_rn(0.f), nan);
            }
            odd = __any_sync(0xffffffffu, __hisnan(__low2half(nan)) || __hisnan(__high2half(nan)));
        }
#pragma unroll
        for (uint32_t ks = 0; ks < uint32_t(kApWarps); ++ks) {
            if (ks >= steps) break;
            uint32_t b[4];
            load_values(b, ks);
            if (odd) {
#pragma unroll
                for (int i = 0; i < 4; ++i) b[i] = ap_finite(b[i]);
            }
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
                if (uint32_t(i) >= n_mt) break;
                const uint8_t* at = s_k + ((i * 8 + ks) * 32 + lane) * 16;
                const uint4 ah0 = *reinterpret_cast<const uint4*>(at), al0 = *reinterpret_cast<const uint4*>(at + kApPlane);
                const uint4 ah1 = *reinterpret_cast<const uint4*>(at + 4096), al1 = *reinterpret_cast<const uint4*>(at + kApPlane + 4096);
#pragma unroll
                for (int j = 0; j < 2; ++j) { ap_mma(o[i][j], al0, b[2 * j], b[2 * j + 1]); ap_mma(o[i + 1][j], al1, b[2 * j], b[2 * j + 1]); }
#pragma unroll
                for (int j = 0; j < 2; ++j) { ap_mma(o[i][j], ah0, b[2 * j], b[2 * j + 1]); ap_mma(o[i + 1][j], ah1, b[2 * j], b[2 * j + 1]); }
            }
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
            load_table((chunk + C) * kApKeys, 0);
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
        for (uint32_t c = 0; c < kApMaxCluster; ++c) part[c] = c < active ? ap_cluster_load4(mine, c) : sum;
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
    return LV_OK;
}

int launch_attention_prompt(lv_ctx* ctx, float* out, const float* q, const void* k_cache, const void* v_cache, const uint32_t* pos,
                            const float* rope_table, uint32_t heads, uint32_t max_ctx, uint32_t batch, void* xh) {
    const uint32_t chunks = (max_ctx + kApKeys - 1) / kApKeys, C = std::min(kApMaxCluster, chunks);
    auto* kernel = chunks <= C ? attention_prompt_kernel<true> : attention_prompt_kernel<false>;
    LV_CUDA(launch_pdl_cluster(ctx, kernel, dim3(heads, C, (batch + kApQ - 1) / kApQ), dim3(kApThreads), dim3(1, C), kApSmemBytes, out, q,
                               static_cast<const __half*>(k_cache), static_cast<const __half*>(v_cache), pos, rope_table, heads, batch, max_ctx,
                               1.0f / sqrtf(float(kApHead)), ctx->d_err, static_cast<__half*>(xh), (batch + 15u) & ~15u));
    return LV_OK;
}

}  // namespace lv
