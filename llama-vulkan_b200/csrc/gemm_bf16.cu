// Products of several tokens with bfloat16 matrices on the tcgen05 tensor cores, dense and per expert.
//
//   out[t][r] = act(factor * sum_k W[r][k] x[t][k])        W and x bfloat16, sums f32
//
// A CTA covers 128 rows of W (the M of the MMA) and NT tokens (its N).  Both operands are K-major and come by TMA in boxes of
// 64 columns with the 128-byte swizzle; one lane issues the loads, one lane the MMAs, four warps read the
// accumulator from tensor memory (lane = row, column = token, so a warp stores 32 consecutive features of a token).  The
// first weight tiles are requested before the previous kernel has finished.
//
// Two CTAs may share a tile of 256 rows (TWO): each brings its own rows of W and half of the tokens, and one lane of the first issues products
// that read both shared memories (cta_group::2), so 64 columns of 256 x 256 cost an SM 32 KB instead of 48.
//
// What bounds it: the operands' way from L2.  An SM takes in about 46 bytes per clock (measured), so 64 columns of a tile cost
// (128 + NT) * 128 / 46 clocks against 2 NT of the tensor pipe: 534 / 128 at NT = 64, 712 / 256 at 128, 1070 / 512 at 256.  So wide tiles
// come first, and a matrix whose wide tiles are too few is split along K over a cluster of up to eight CTAs: each leaves its
// partial sums in its own shared memory, where the stages were, and they are added in split order (deterministic) through
// distributed shared memory, every CTA finishing its share of the tokens.  A launch of more tiles than SMs without a split runs two CTAs
// per SM, so that the set-up and the stores of one run beside the products of the other.
// us, before (tiles of 64 or 128 tokens, one CTA per SM, partial sums through global memory) -> wide tiles -> pairs of CTAs and eight epilogue
// warps.  512 tokens: 16512 x 4096 107.8 -> 57.1 -> 45.8 (1.51 PFLOP/s), 4096 x 16512 79.6 -> 55.1 -> 47.0, 8448 x 2048 30.1 -> 19.7 -> 17.2,
// 2048 x 8448 41.6 -> 21.0 -> 22; 2048 tokens: 16512 x 4096 389 -> 224 -> 181, 4096 x 16512 317 -> 189 -> 153 (1.82 PFLOP/s).
// Sums of split products are nearer to 64 bits than before (2048 x 8448, 512 tokens: 9.4e-6 -> 2.2e-6 relative), the others the same.
//
// Experts: lv_expert_route sorts the (token, choice) pairs of a step by expert and lists tiles of NT rows; the input rows lie
// in that order (lv_norm_conv scatters them there), a tile multiplies them with its expert's rows of the stacked matrix.
// The gated pair keeps two accumulators, so gate and up of a feature meet in one thread.
//
// Windows (lv_gemm_bf16_window): x is a cache, and the rows to multiply are those that the step's tokens see; where they begin is
// only known on the device, so a tile finds its rows from the position word, and tiles behind the last row leave at once.
//
// Every wait is bounded (common.cuh); a lost wait sets the error word, the CTA drains and frees its tensor memory.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "attention_gqa.cuh"
#include "common.cuh"
#include "ctx.h"
#include "tcgen05.cuh"
#include "tmap.h"

namespace lv {

// TMA warp, MMA warp, eight epilogue warps; four where the parts of a split meet (512 tokens of 8448 x 2048: 19.7 us with four, 17.2 with
// eight; 60 tokens of 2048 x 2048, split: 9.1 and 11.4)
constexpr int kBgThreads = 320, kBgThreadsSplit = 192;
constexpr int kBgRows = 128, kBgK = 64;
constexpr uint32_t kBgTile = kBgRows * kBgK * 2;
constexpr size_t kBgSmemBudget = 200 * 1024, kBgSmemHalf = 108 * 1024;      // one / two CTAs per SM
constexpr uint32_t kBgMaxStages = 8;
constexpr uint32_t kBgMaxSplits = 8;         // portable cluster size

struct GemmBf16Params {
    uint32_t rows, tokens, K, splits, stages;
    void* out;
    uint32_t out_ld, out_bf16;
    float factor;
    int act;
    const lv_expert_tile* tiles;
    const uint32_t* pos;        // windows: the position word, null otherwise
    uint32_t window, batch;
    uint32_t* err;
};

struct GemmBf16Maps {
    CUtensorMap w, w2, x;
};

__host__ __device__ constexpr uint32_t bg_stage_bytes(int NT, bool pair, bool two) { return (pair ? 2 : 1) * kBgTile + (two ? NT / 2 : NT) * kBgK * 2; }
// Accumulators that chunks of K take in turn.  The tensor core's sums truncate, an error that grows with the number of additions that follow one
// another; narrow tiles, whose K is cut over at most eight CTAs, have the tensor memory for two chains of half the length.  (1024 x 3072, 60
// tokens: relative error 3.5e-7 -> 1.9e-7; 2048 x 512, 16 tokens: 4.8e-7 -> 2.4e-7.)
__host__ __device__ constexpr uint32_t bg_banks(int NT) { return NT <= 64 ? 2u : 1u; }
__host__ __device__ constexpr uint32_t bg_tmem_cols(int NT, bool pair) {
    const int need = NT * (pair ? 2 : 1) * int(bg_banks(NT));
    return need <= 32 ? 32 : need <= 64 ? 64 : need <= 128 ? 128 : need <= 256 ? 256 : 512;
}

// grid (row tiles, token tiles, splits), clusters of (TWO ? 2 : 1, 1, splits)
template <int NT, bool PAIR, bool GROUPED, bool TWO>
__global__ void __launch_bounds__(kBgThreads, 2) gemm_bf16_kernel(const GemmBf16Params p, const __grid_constant__ GemmBf16Maps maps) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023));
    constexpr uint32_t kStage = bg_stage_bytes(NT, PAIR, TWO), kCols = bg_tmem_cols(NT, PAIR), kXAt = (PAIR ? 2 : 1) * kBgTile;
    constexpr uint32_t kBanks = bg_banks(NT), kBankCols = NT * (PAIR ? 2 : 1);
    __shared__ uint64_t full[kBgMaxStages], empty[kBgMaxStages], acc_full;
    __shared__ uint32_t s_tmem;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    uint32_t row0 = blockIdx.x * kBgRows, tok0 = blockIdx.y * NT, n_tok;
    uint32_t w_row0 = row0, x_row0 = tok0;
    const bool wait_first = GROUPED || p.pos != nullptr;
    if (!GROUPED && p.pos != nullptr) {
        pdl_wait();
        const uint32_t P = *p.pos, first = p.window != 0 && P + 1 > p.window ? P + 1 - p.window : 0, n = min(p.tokens, P + p.batch - first);
        if (tok0 >= n) return;
        n_tok = min(uint32_t(NT), n - tok0);
        x_row0 = first + tok0;
    } else if constexpr (GROUPED) {
        pdl_wait();
        const lv_expert_tile t = p.tiles[blockIdx.y];
        if (t.rows == 0) return;
        tok0 = x_row0 = t.row0;
        n_tok = t.rows;
        w_row0 += t.expert * p.rows;
    } else {
        n_tok = min(uint32_t(NT), p.tokens - tok0);
    }
    const uint32_t chunks_all = (p.K + kBgK - 1) / kBgK;
    const uint32_t c0 = chunks_all * blockIdx.z / p.splits, n_chunks = chunks_all * (blockIdx.z + 1) / p.splits - c0;

    if (threadIdx.x < 2 * kBgMaxStages + 1) {
        const uint32_t i = threadIdx.x;
        mbar_init(i < kBgMaxStages ? &full[i] : i < 2 * kBgMaxStages ? &empty[i - kBgMaxStages] : &acc_full, 1);
        fence_mbar_init();
    }
    const uint32_t half = TWO ? blockIdx.x & 1u : 0u;         // which CTA of a pair this is; the first one issues the products of both
    if (warp == 1) {
        if constexpr (TWO) tc_alloc_pair(&s_tmem, kCols);
        else tc_alloc(&s_tmem, kCols);
    }
    tc_fence_before_sync();
    __syncthreads();
    if constexpr (TWO) cluster_sync();                        // the barriers of the pair exist before either signals the other's
    tc_fence_after_sync();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&s_tmem);
    // not before every CTA of this launch has its tensor memory: a CTA of the next one beside it could take what is missing, and wait for
    // this launch with it
    pdl_launch_dependents();
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {
            // TWO: both CTAs' copies complete on the first one's barrier, which counts the bytes of both
            uint32_t bar0 = smem_u32(&full[0]);
            if constexpr (TWO) {
                const uint32_t local = bar0;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar0) : "r"(local), "r"(2u * blockIdx.z));
            }
            auto load = [&](void* dst, const CUtensorMap* map, uint32_t c, uint32_t y, uint32_t s) {
                if constexpr (TWO) tma_load_2d_pair(dst, map, int((c0 + c) * kBgK), int(y), bar0 + 8u * s);
                else tma_load_2d_plain(dst, map, int((c0 + c) * kBgK), int(y), &full[s]);
            };
            auto load_w = [&](uint32_t c, uint32_t s) {
                if (half == 0) mbar_expect_tx(&full[s], (TWO ? 2 : 1) * kStage);
                load(smem + s * kStage, &maps.w, c, w_row0, s);
                if constexpr (PAIR) load(smem + s * kStage + kBgTile, &maps.w2, c, w_row0, s);
            };
            auto load_x = [&](uint32_t c, uint32_t s) { load(smem + s * kStage + kXAt, &maps.x, c, x_row0 + half * (NT / 2), s); };
            const uint32_t first = min(p.stages, n_chunks);
            for (uint32_t c = 0; c < first; ++c) load_w(c, c);
            if (!wait_first) pdl_wait();
            for (uint32_t c = 0; c < first; ++c) load_x(c, c);
            uint32_t s = 0, phase = 0;
            for (uint32_t c = first; c < n_chunks; ++c) {
                if (!mbar_wait(&empty[s], phase, p.err)) break;
                load_w(c, s);
                load_x(c, s);
                if (++s == p.stages) { s = 0; phase ^= 1u; }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && half == 0) {
            // f32 accumulator, bfloat16 operands, both K-major
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(NT >> 3) << 17) | (uint32_t((TWO ? 2 * kBgRows : kBgRows) >> 4) << 24);
            const uint32_t mask = 3u << (2u * blockIdx.z);            // TWO: the cluster's CTAs that a commit reports to
            const uint64_t base = tc_smem_desc(smem_u32(smem));
            uint32_t s = 0, phase = 0;
            for (uint32_t c = 0; c < n_chunks && ok; ++c) {
                ok = mbar_wait(&full[s], phase, p.err);
                if (!ok) break;
                tc_fence_after_sync();
                const uint64_t a = base + ((s * kStage) >> 4), b = a + (kXAt >> 4);
#pragma unroll
                for (int k = 0; k < kBgK / 16; ++k) {
                    const uint32_t acc = (c >= kBanks || k != 0) ? 1u : 0u, to = tmem + c % kBanks * kBankCols;
                    tc_mma_16bit<TWO>(to, a + 2u * k, b + 2u * k, idesc, acc);
                    if constexpr (PAIR) tc_mma_16bit<TWO>(to + NT, a + (kBgTile >> 4) + 2u * k, b + 2u * k, idesc, acc);
                }
                if constexpr (TWO) tc_commit_pair(&empty[s], mask);
                else tc_commit(&empty[s]);
                if (++s == p.stages) { s = 0; phase ^= 1u; }
            }
            if (ok) {
                if constexpr (TWO) tc_commit_pair(&acc_full, mask);
                else tc_commit(&acc_full);
            }
        }
    } else {
        // ---- epilogue: warp w reads lanes 32 (w mod 4) .. + 31 of the accumulator, half of its columns -----------
        const uint32_t quarter = uint32_t(warp) & 3u, tr = quarter * 32u + uint32_t(lane);
        const uint32_t row = row0 + tr, taddr = tmem + (quarter * 32u << 16);
        ok = mbar_wait_warp(&acc_full, 0, p.err);
        tc_fence_after_sync();
        constexpr int kAcc = PAIR ? 2 : 1;
        float* partial = reinterpret_cast<float*>(smem);         // [accumulator][token][128 rows]: all stages have been used up
        auto finish = [&](const float (&v)[16], const float (&g)[16], uint32_t z0) {
            if (row >= p.rows) return;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                if (z0 + i >= n_tok) break;
                const float r = PAIR ? silu_f32(v[i]) * g[i] : product_act(v[i] * p.factor, p.act);
                const size_t at = size_t(tok0 + z0 + i) * p.out_ld + row;
                if (p.out_bf16) static_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(r);
                else static_cast<float*>(p.out)[at] = r;
            }
        };
        if (ok) {
            // (NT = 16: the first four warps have all columns)
            const uint32_t share = blockDim.x == kBgThreads ? (NT / 2 + 15) / 16 * 16 : NT, z_first = uint32_t(warp - 2) / 4 * share;
            for (uint32_t z0 = z_first; z0 < min(z_first + share, uint32_t(NT)); z0 += 16) {
                uint32_t u[kAcc][16];
#pragma unroll
                for (int a = 0; a < kAcc; ++a) tc_load16(u[a], taddr + a * NT + z0);
                tc_wait_load();
                float v[16], g[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) { v[i] = __uint_as_float(u[0][i]); g[i] = __uint_as_float(u[kAcc - 1][i]); }
                if (kBanks == 2 && n_chunks > 1) {
#pragma unroll
                    for (int a = 0; a < kAcc; ++a) tc_load16(u[a], taddr + kBankCols + a * NT + z0);
                    tc_wait_load();
#pragma unroll
                    for (int i = 0; i < 16; ++i) { v[i] += __uint_as_float(u[0][i]); g[i] += __uint_as_float(u[kAcc - 1][i]); }
                }
                if (p.splits == 1) {
                    finish(v, g, z0);
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        partial[(z0 + i) * kBgRows + tr] = v[i];
                        if constexpr (PAIR) partial[(NT + z0 + i) * kBgRows + tr] = g[i];
                    }
                }
            }
        }
        tc_fence_before_sync();
    }
    __syncthreads();
    // Of a pair, either CTA's release may ask for both: not before both have read their accumulators.  Nor does a CTA leave while the other
    // one's products or signals may reach it; of a split, the partial sums of all CTAs are in place.
    if (TWO || p.splits > 1) {
        __syncwarp();
        cluster_sync();
    }
    if (warp == 1) {
        tc_fence_after_sync();
        if constexpr (TWO) tc_free_pair(tmem, kCols);
        else tc_free(tmem, kCols);
    }
    if (p.splits > 1) {
        // a warp has whole tokens, a lane four rows of them; kTok tokens are on their way together
        constexpr int kTok = PAIR ? 2 : 4, kWarps = kBgThreadsSplit / 32;
        const float* mine = reinterpret_cast<const float*>(smem) + 4 * lane;
        const uint32_t row = row0 + 4 * uint32_t(lane), z_end = n_tok * (blockIdx.z + 1) / p.splits;
        const bool vec = row + 4 <= p.rows && p.out_ld % 4 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0;
        pdl_wait();                                       // (of the warps only the loading one has waited for the previous kernel)
        for (uint32_t z0 = n_tok * blockIdx.z / p.splits + warp; z0 < z_end; z0 += kTok * kWarps) {
            float4 v[kTok] = {}, g[kTok] = {};
#pragma unroll 2
            for (uint32_t c = 0; c < p.splits; ++c) {
#pragma unroll
                for (int i = 0; i < kTok; ++i) {
                    const uint32_t z = min(z0 + uint32_t(i) * kWarps, n_tok - 1);
                    const float4 a = cluster_load4(mine + z * kBgRows, TWO ? 2 * c + half : c);
                    v[i] = make_float4(v[i].x + a.x, v[i].y + a.y, v[i].z + a.z, v[i].w + a.w);
                    if constexpr (PAIR) {
                        const float4 b = cluster_load4(mine + (NT + z) * kBgRows, TWO ? 2 * c + half : c);
                        g[i] = make_float4(g[i].x + b.x, g[i].y + b.y, g[i].z + b.z, g[i].w + b.w);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < kTok; ++i) {
                const uint32_t z = z0 + uint32_t(i) * kWarps;
                if (z >= z_end) break;
                const float x[4] = {v[i].x, v[i].y, v[i].z, v[i].w}, y[4] = {g[i].x, g[i].y, g[i].z, g[i].w};
                float o[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) o[j] = PAIR ? silu_f32(x[j]) * y[j] : product_act(x[j] * p.factor, p.act);
                const size_t at = size_t(tok0 + z) * p.out_ld + row;
                if (p.out_bf16) {
                    auto* to = static_cast<__nv_bfloat16*>(p.out) + at;
                    if (vec) {
                        const __nv_bfloat162 lo = __floats2bfloat162_rn(o[0], o[1]), hi = __floats2bfloat162_rn(o[2], o[3]);
                        *reinterpret_cast<uint2*>(to) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
                    } else {
                        for (int j = 0; j < 4; ++j) if (row + j < p.rows) to[j] = __float2bfloat16_rn(o[j]);
                    }
                } else {
                    float* to = static_cast<float*>(p.out) + at;
                    if (vec) *reinterpret_cast<float4*>(to) = make_float4(o[0], o[1], o[2], o[3]);
                    else for (int j = 0; j < 4; ++j) if (row + j < p.rows) to[j] = o[j];
                }
            }
        }
        __syncwarp();
        cluster_sync();                                   // no CTA leaves while another reads its shared memory
    }
}

// rows of an expert tile: by the rows an expert gets when the ids spread evenly
__host__ __device__ inline uint32_t bg_expert_tile(uint32_t batch, uint32_t top, uint32_t experts) {
    const uint32_t mean = (batch * top + experts - 1) / experts;
    return mean <= 12 ? 16 : mean <= 24 ? 32 : mean <= 56 ? 64 : 128;
}

// Sorts the (token, choice) pairs of a step by expert, one CTA per layer.
__global__ void __launch_bounds__(1024) expert_route_kernel(const lv_route_job* __restrict__ jobs, const uint32_t* __restrict__ token_log,
                                                            const uint32_t* __restrict__ pos, uint32_t vocab, uint32_t batch, uint32_t* err) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ uint32_t s_cursor[];               // [experts]: count, then next free row
    const lv_route_job job = jobs[blockIdx.x];
    const uint32_t pairs = batch * job.top, first = *pos, tile_rows = bg_expert_tile(batch, job.top, job.experts);
    for (uint32_t e = threadIdx.x; e < job.experts; e += blockDim.x) s_cursor[e] = 0;
    __syncthreads();
    auto expert = [&](uint32_t i) {
        const uint32_t id = token_log[first + i / job.top];
        const uint32_t e = id < vocab ? job.table[size_t(id) * job.top + i % job.top] : job.experts;
        if (e < job.experts) return e;
        atomicOr(err, ERR_BAD_INDEX);
        return 0u;
    };
    for (uint32_t i = threadIdx.x; i < pairs; i += blockDim.x) atomicAdd(&s_cursor[expert(i)], 1u);
    __syncthreads();
    if (threadIdx.x < 32) {
        // a lane sums the rows and tiles of consecutive experts, the warp forms the prefix, the lane hands them out
        const uint32_t per = (job.experts + 31) / 32, e0 = min(job.experts, threadIdx.x * per), e1 = min(job.experts, e0 + per);
        uint32_t rows = 0, tiles = 0;
        for (uint32_t e = e0; e < e1; ++e) {
            rows += s_cursor[e];
            tiles += (s_cursor[e] + tile_rows - 1) / tile_rows;
        }
        uint32_t row_at = rows, tile_at = tiles;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t r = __shfl_up_sync(0xffffffffu, row_at, o), t = __shfl_up_sync(0xffffffffu, tile_at, o);
            if (threadIdx.x >= uint32_t(o)) { row_at += r; tile_at += t; }
        }
        const uint32_t all_tiles = __shfl_sync(0xffffffffu, tile_at, 31);
        row_at -= rows;
        tile_at -= tiles;
        for (uint32_t e = e0; e < e1; ++e) {
            const uint32_t n = s_cursor[e];
            for (uint32_t r = 0; r < n; r += tile_rows, ++tile_at)
                if (tile_at < job.max_tiles) job.tiles[tile_at] = {e, row_at + r, min(tile_rows, n - r)};
            s_cursor[e] = row_at;
            row_at += n;
        }
        for (uint32_t t = all_tiles + threadIdx.x; t < job.max_tiles; t += 32) job.tiles[t] = {0u, 0u, 0u};
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < pairs; i += blockDim.x) job.index[i] = atomicAdd(&s_cursor[expert(i)], 1u);
}

// How a product is cut: tokens of a tile, pairs of CTAs, splits along K.
struct BgPlan {
    uint32_t nt = 0, splits = 1;
    bool two = false;
    float clocks = 0.f;
};

// Fills in the splits and the clocks of a plan: 64 columns of a tile take the time of the tensor pipe or that of the operands' way.  A launch
// costs 6000 clocks beside them (measured on products of one wave), the meeting of a split's cluster 2000 more and 4 per token of the tile;
// as many splits as the device holds at once, each with at least four chunks.
static void bg_cut(const lv_ctx* ctx, BgPlan* plan, uint32_t rows, uint32_t cols, uint32_t token_tiles, bool pair) {
    const uint32_t sms = uint32_t(ctx->sm_count), chunks = (cols + kBgK - 1) / kBgK, cluster = plan->two ? 2 : 1;
    const uint32_t ctas = ((rows + kBgRows - 1) / kBgRows + cluster - 1) / cluster * cluster * token_tiles;
    const float c = std::max(2.f * plan->nt * (pair ? 2 : 1), bg_stage_bytes(int(plan->nt), pair, plan->two) / 46.f);
    // without a split: two CTAs share an SM, so a last wave that is not full costs its part only
    plan->clocks = (ctas > sms ? float(ctas) / sms + 0.25f : 1.f) * chunks * c + 6000.f;
    plan->splits = 1;
    for (uint32_t s = 2; s * cluster <= kBgMaxSplits && chunks / s >= 4; ++s) {
        if (ctas / cluster > ctx->bg_clusters[s * cluster]) continue;
        const float t = (chunks + s - 1) / s * c + 8000.f + 4.f * plan->nt;
        if (t < plan->clocks) { plan->clocks = t; plan->splits = s; }
    }
}

// Shared memory of a launch, from a budget for its stages; the parts of a split take the stages' place.
template <int NT, bool PAIR, bool TWO>
constexpr uint32_t bg_stages(size_t budget) { return std::min<uint32_t>(kBgMaxStages, uint32_t(budget / bg_stage_bytes(NT, PAIR, TWO))); }
template <int NT, bool PAIR, bool TWO>
constexpr size_t bg_smem(uint32_t stages, bool split) {
    return std::max(size_t(stages) * bg_stage_bytes(NT, PAIR, TWO), split ? size_t(PAIR ? 2 : 1) * NT * kBgRows * sizeof(float) : 0) + 1024;
}

// The largest size is set once: the attribute belongs to the kernel, and contexts launch from threads of their own.
template <int NT, bool PAIR, bool GROUPED, bool TWO>
static int bg_configure(lv_ctx* ctx) {
    constexpr size_t smem = bg_smem<NT, PAIR, TWO>(bg_stages<NT, PAIR, TWO>(kBgSmemBudget), true);
    LV_REQUIRE(size_t(ctx->max_smem_optin) >= smem, "device has too little shared memory for the bfloat16 product");
    LV_CUDA(cudaFuncSetAttribute(gemm_bf16_kernel<NT, PAIR, GROUPED, TWO>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    return LV_OK;
}

// How many clusters of each size the device holds at a time, one CTA per SM: the SMs of a cluster are neighbours, so of 148 SMs clusters of
// eight fill fewer than clusters of two.  (Two waves of clusters made a product of 2048 x 2048 with 60 tokens 18 us instead of 9.)
int gemm_bf16_configure(lv_ctx* ctx) {
    auto* kernel = gemm_bf16_kernel<128, false, false, false>;
    int (*const configure[])(lv_ctx*) = {
        bg_configure<16, false, false, false>, bg_configure<32, false, false, false>, bg_configure<64, false, false, false>, bg_configure<128, false, false, false>,
        bg_configure<128, false, false, true>, bg_configure<256, false, false, false>, bg_configure<256, false, false, true>,
        bg_configure<16, false, true, false>, bg_configure<32, false, true, false>, bg_configure<64, false, true, false>, bg_configure<128, false, true, false>,
        bg_configure<16, true, true, false>, bg_configure<32, true, true, false>, bg_configure<64, true, true, false>, bg_configure<128, true, true, false>};
    for (auto* f : configure)
        if (int rc = f(ctx)) return rc;
    for (uint32_t s = 2; s <= kBgMaxSplits; ++s) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(1, 1, s);
        cfg.blockDim = dim3(kBgThreads);
        cfg.dynamicSmemBytes = bg_smem<128, false, false>(bg_stages<128, false, false>(kBgSmemBudget), true);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = s;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        LV_CUDA(cudaOccupancyMaxActiveClusters(&n, kernel, &cfg));
        ctx->bg_clusters[s] = uint32_t(n);
    }
    return LV_OK;
}

template <int NT, bool PAIR, bool GROUPED, bool TWO>
static int gemm_bf16_launch(lv_ctx* ctx, GemmBf16Params p, const GemmBf16Maps& maps, const BgPlan& plan, uint32_t token_tiles) {
    constexpr uint32_t kCluster = TWO ? 2 : 1;
    const uint32_t row_tiles = ((p.rows + kBgRows - 1) / kBgRows + kCluster - 1) / kCluster * kCluster, ctas = row_tiles * token_tiles;
    p.splits = plan.splits;
    p.stages = bg_stages<NT, PAIR, TWO>(p.splits == 1 && ctas > uint32_t(ctx->sm_count) ? kBgSmemHalf : kBgSmemBudget);
    p.err = ctx->d_err;
    const size_t smem = bg_smem<NT, PAIR, TWO>(p.stages, p.splits > 1);
    auto* kernel = gemm_bf16_kernel<NT, PAIR, GROUPED, TWO>;
    LV_REQUIRE(token_tiles <= 65535, "gemm_bf16: too many token tiles");
    const dim3 grid(row_tiles, token_tiles, p.splits);
    if (kCluster * p.splits == 1) LV_CUDA(launch_pdl(ctx, kernel, grid, dim3(kBgThreads), smem, p, maps));
    else LV_CUDA(launch_pdl_cluster(ctx, kernel, grid, dim3(p.splits > 1 ? kBgThreadsSplit : kBgThreads), dim3(kCluster, 1, p.splits), smem, p, maps));
    return LV_OK;
}

// The plan that takes least by the model above, for a product of `tokens` rows.
static BgPlan bg_plan(const lv_ctx* ctx, uint32_t rows, uint32_t cols, uint32_t tokens) {
    BgPlan best;
    for (uint32_t n : {16u, 32u, 64u, 128u, 256u}) {
        if (n > 32 && n / 2 >= tokens) break;                    // (half of it would do)
        if (n == 16 && tokens > 16) continue;
        for (bool two : {false, true}) {
            if (two && (n < 128 || rows <= kBgRows)) continue;
            BgPlan plan;
            plan.nt = n;
            plan.two = two;
            bg_cut(ctx, &plan, rows, cols, (tokens + n - 1) / n, false);
            if (best.nt == 0 || plan.clocks < best.clocks) best = plan;
        }
    }
    return best;
}

template <bool PAIR, bool GROUPED>
static int gemm_bf16_pick(lv_ctx* ctx, const GemmBf16Params& p, const GemmBf16Maps& maps, const BgPlan& plan, uint32_t token_tiles) {
    switch (plan.nt) {
        case 16: return gemm_bf16_launch<16, PAIR, GROUPED, false>(ctx, p, maps, plan, token_tiles);
        case 32: return gemm_bf16_launch<32, PAIR, GROUPED, false>(ctx, p, maps, plan, token_tiles);
        case 64: return gemm_bf16_launch<64, PAIR, GROUPED, false>(ctx, p, maps, plan, token_tiles);
        case 128:
            if constexpr (!GROUPED)
                if (plan.two) return gemm_bf16_launch<128, PAIR, GROUPED, true>(ctx, p, maps, plan, token_tiles);
            return gemm_bf16_launch<128, PAIR, GROUPED, false>(ctx, p, maps, plan, token_tiles);
        default:
            if constexpr (!GROUPED) {
                if (plan.two) return gemm_bf16_launch<256, PAIR, GROUPED, true>(ctx, p, maps, plan, token_tiles);
                return gemm_bf16_launch<256, PAIR, GROUPED, false>(ctx, p, maps, plan, token_tiles);
            }
            return fail(LV_ERR_BAD_ARGUMENTS, "gemm_bf16: tile of an expert");
    }
}

static bool bg_aligned(const void* p) { return p != nullptr && (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace lv

using namespace lv;

extern "C" int lv_gemm_bf16(lv_ctx* ctx, void* out, int out_type, uint32_t out_ld, const void* w, uint32_t rows, uint32_t ld, uint32_t cols,
                            const void* x, uint32_t x_ld, uint32_t batch, float factor, int act) {
    LV_ENTER(ctx);
    LV_REQUIRE(out && bg_aligned(w) && bg_aligned(x) && rows && cols && batch && out_ld >= rows, "bad gemm_bf16 arguments");
    LV_REQUIRE(ld % 8 == 0 && ld >= cols && x_ld % 8 == 0 && x_ld >= cols && (out_type == LV_TYPE_F32 || out_type == LV_TYPE_BF16), "gemm_bf16: bad strides");
    LV_REQUIRE(act == LV_ACT_NONE || act == LV_ACT_RELU2, "gemm_bf16: unknown activation");
    GemmBf16Params p{};
    p.rows = rows; p.tokens = batch; p.K = cols; p.out = out; p.out_ld = out_ld; p.out_bf16 = out_type == LV_TYPE_BF16; p.factor = factor; p.act = act;
    const BgPlan plan = bg_plan(ctx, rows, cols, batch);
    const uint32_t nt = plan.nt;
    GemmBf16Maps maps{};
    if (int rc = make_bf16_map(&maps.w, w, rows, cols, ld, kBgRows)) return rc;
    if (int rc = make_bf16_map(&maps.x, x, batch, cols, x_ld, plan.two ? nt / 2 : nt)) return rc;
    maps.w2 = maps.w;
    return gemm_bf16_pick<false, false>(ctx, p, maps, plan, (batch + nt - 1) / nt);
}

extern "C" int lv_gemm_bf16_plan(lv_ctx* ctx, uint32_t rows, uint32_t cols, uint32_t tokens, uint32_t* plan) {
    LV_ENTER(ctx);
    LV_REQUIRE(rows && cols && tokens && plan, "bad gemm_bf16_plan arguments");
    const BgPlan p = bg_plan(ctx, rows, cols, tokens);
    plan[0] = p.nt;
    plan[1] = p.two ? 2 : 1;
    plan[2] = p.splits;
    return LV_OK;
}

extern "C" int lv_gemm_bf16_window(lv_ctx* ctx, void* out, int out_type, uint32_t out_ld, const void* w, uint32_t rows, uint32_t ld, uint32_t cols,
                                   const void* x, uint32_t x_ld, uint32_t x_rows, const uint32_t* pos, uint32_t batch, uint32_t window, uint32_t max_rows) {
    LV_ENTER(ctx);
    LV_REQUIRE(out && bg_aligned(w) && bg_aligned(x) && rows && cols && batch && pos && max_rows && x_rows && out_ld >= rows, "bad gemm_bf16 arguments");
    LV_REQUIRE(ld % 8 == 0 && ld >= cols && x_ld % 8 == 0 && x_ld >= cols && (out_type == LV_TYPE_F32 || out_type == LV_TYPE_BF16), "gemm_bf16: bad strides");
    GemmBf16Params p{};
    p.rows = rows; p.tokens = max_rows; p.K = cols; p.out = out; p.out_ld = out_ld; p.out_bf16 = out_type == LV_TYPE_BF16; p.factor = 1.0f;
    p.pos = pos; p.window = window; p.batch = batch;
    const BgPlan plan = bg_plan(ctx, rows, cols, max_rows);
    const uint32_t nt = plan.nt;
    GemmBf16Maps maps{};
    if (int rc = make_bf16_map(&maps.w, w, rows, cols, ld, kBgRows)) return rc;
    if (int rc = make_bf16_map(&maps.x, x, x_rows, cols, x_ld, plan.two ? nt / 2 : nt)) return rc;
    maps.w2 = maps.w;
    return gemm_bf16_pick<false, false>(ctx, p, maps, plan, (max_rows + nt - 1) / nt);
}

extern "C" uint32_t lv_expert_tile_rows(uint32_t batch, uint32_t top, uint32_t experts) {
    return experts ? bg_expert_tile(batch, top, experts) : 0;
}

extern "C" uint32_t lv_expert_max_tiles(uint32_t batch, uint32_t top, uint32_t experts) {
    if (!experts) return 0;
    const uint32_t nt = bg_expert_tile(batch, top, experts), pairs = batch * top;
    return pairs / nt + std::min(experts, pairs);
}

extern "C" int lv_expert_route(lv_ctx* ctx, const lv_route_job* jobs, uint32_t n_jobs, uint32_t max_experts, const uint32_t* token_log,
                               const uint32_t* pos, uint32_t vocab, uint32_t batch) {
    LV_ENTER(ctx);
    LV_REQUIRE(jobs && n_jobs && token_log && pos && vocab && batch, "bad expert_route arguments");
    LV_REQUIRE(max_experts && max_experts <= 8192, "expert_route: more than 8192 experts");
    LV_CUDA(launch_pdl(ctx, expert_route_kernel, dim3(n_jobs), dim3(1024), max_experts * 4, jobs, token_log, pos, vocab, batch, ctx->d_err));
    return LV_OK;
}

static int expert_gemm(lv_ctx* ctx, bool pair, void* out, int out_type, uint32_t out_ld, const lv_expert_args* a, const lv_expert_tile* tiles, const void* x,
                       uint32_t x_ld, uint32_t batch) {
    LV_ENTER(ctx);
    LV_REQUIRE(out && a && tiles && bg_aligned(x) && batch && bg_aligned(a->w0) && (!pair || bg_aligned(a->w1)), "bad expert product arguments");
    LV_REQUIRE(a->ld % 8 == 0 && a->ld >= a->cols && x_ld % 8 == 0 && x_ld >= a->cols && a->rows && a->cols && a->experts && a->top && out_ld >= a->rows &&
               (out_type == LV_TYPE_F32 || out_type == LV_TYPE_BF16), "expert product: bad strides");
    GemmBf16Params p{};
    p.rows = a->rows; p.tokens = batch * a->top; p.K = a->cols; p.out = out; p.out_ld = out_ld; p.out_bf16 = out_type == LV_TYPE_BF16; p.factor = 1.0f;
    p.tiles = tiles;
    const uint32_t nt = lv_expert_tile_rows(batch, a->top, a->experts), n_tiles = lv_expert_max_tiles(batch, a->top, a->experts);
    // tiles have as many tokens as the router made them; pairs of CTAs gain nothing on them (a prompt of Sonuzen 2048: 5.78 ms without, 6.04 with)
    BgPlan plan;
    plan.nt = nt;
    bg_cut(ctx, &plan, a->rows, a->cols, n_tiles, pair);
    GemmBf16Maps maps{};
    if (int rc = make_bf16_map(&maps.w, a->w0, uint64_t(a->experts) * a->rows, a->cols, a->ld, kBgRows)) return rc;
    maps.w2 = maps.w;
    if (pair)
        if (int rc = make_bf16_map(&maps.w2, a->w1, uint64_t(a->experts) * a->rows, a->cols, a->ld, kBgRows)) return rc;
    if (int rc = make_bf16_map(&maps.x, x, uint64_t(batch) * a->top, a->cols, x_ld, nt)) return rc;
    return pair ? gemm_bf16_pick<true, true>(ctx, p, maps, plan, n_tiles) : gemm_bf16_pick<false, true>(ctx, p, maps, plan, n_tiles);
}

extern "C" int lv_gemm_bf16_expert_gate_up(lv_ctx* ctx, void* out, uint32_t out_ld, const lv_expert_args* a, const lv_expert_tile* tiles, const void* x,
                                           uint32_t x_ld, uint32_t batch) {
    return expert_gemm(ctx, true, out, LV_TYPE_BF16, out_ld, a, tiles, x, x_ld, batch);
}

extern "C" int lv_gemm_bf16_expert_down(lv_ctx* ctx, float* out, uint32_t out_ld, const lv_expert_args* a, const lv_expert_tile* tiles, const void* x,
                                        uint32_t x_ld, uint32_t batch) {
    return expert_gemm(ctx, false, out, LV_TYPE_F32, out_ld, a, tiles, x, x_ld, batch);
}
