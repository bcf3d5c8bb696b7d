// Batched products over quantised weights with the weight tiles in tensor memory (the default form of lv_gemm_tc*).
//
//   out[z][r] = sum_k W[r][k] * x[z][k]        z < Z <= 64
//
// The work is a list of units: tiles of 128 rows (64 + 64 of a SiLU pair) times groups of 256 columns, tile by tile.  A persistent
// launch of at most one CTA per SM gives every CTA an equal run of consecutive units, wherever tiles begin and end in it (or an equal share of
// one tile, see launch_typed): a run is cut into segments, one per tile that it touches.  A segment that covers a whole tile is finished by its CTA.  Of the others
// the partial accumulators go to scratch, each reported as soon as it lies there, and whoever comes last adds the parts in the order of K
// (deterministic) and applies the epilogue: mostly the CTA whose run ends inside the tile, which then takes its own part from its registers.  The
// four warps that hold sixteen tokens of a tile do this by themselves.
//
// What bounds it: one CTA per row tile and share of K ran in waves that were filled to 60-80 %, and paid set-up, ring filling and the
// pass over the parts in every wave; within a wave two raw stages and one barrier hand-over per 64 columns made a group take 1.2 us
// where the tensor pipe needs 0.5 us (Z = 64) and HBM 0.4 us.  Here those costs are paid once per launch, the weights arrive through three
// (q8_0) or four and more raw stages, and activations are handed over 128 columns at a time.
//
// Roles (20 warps):
//   0..15  producers.  A warp reaches only its own quarter of the tensor memory's lanes (= tile rows), so warp w dequantises rows
//          32 (w % 4) .. + 31 of tile w / 4 of each group: two blocks of a row per thread into 32 registers (fp16 pairs of hi = fp16(w),
//          11 significant bits), stored with tcgen05.st.  Two such buffers of four 64-column tiles.  The same warps read finished
//          accumulators back, one unit after the segment's end, so that the last products run while the next unit is prepared.
//   16     raw ring: 2-D tensor-map loads of q4_0 / q8_0 rows.
//   17, 18 one lane each issues tcgen05.mma: tiles 0 and 1 of a group into accumulator bank 0, tiles 2 and 3 into bank 1 (two fp32
//          chains of half the length); N = 2 zpad columns: the activations' hi and lo planes.
//   19     activation ring: one bulk copy per two tiles of K (q8_0, whose raw stages are larger: one).  The number of stages is even, so that
//          a stage always belongs to one issuing lane (a parity wait cannot tell a phase from the one two uses later).
//
// us per launch back to back, 16 / 64 tokens of q4_0: 11008 x 4096 pair 27.3 / 30.5, 4096 x 11008 17.2 / 19.7, 4096 x 4096 9.5 / 11.8 (q8_0 28.6 / 33.7,
// 18.5 / 20.7, 10.5 / 12.4).  When every CTA reported its parts at its end, the last one read all of them back, and the epilogues were unrolled code that
// runs once (instruction fetches: 12 us of a whole pair tile), these took 35.8 / 43.5, 17.4 / 20.2, 10.7 / 12.5 (38.0 / 46.5, 18.9 / 22.9, 12.0 / 13.7).
// 1.7 % (0 to 4) of the present times is the price of giving a wait up in order: a producer's two votes per unit 1.1, the last barrier that collects them 0.6.
// A unit takes about 1700 clocks: 700 of dequantisation, 450 of waiting for and fetching raw words, 90 of tcgen05.st, the rest loop, barriers
// and drains; the tensor pipe needs 1024 of them at 64 tokens.
//
// An accumulator takes a whole segment, up to 16 units of 4096 columns: the error beside the rounding of the weights is 3.7e-6 of a gated pair (2.4e-6
// with two shares of K), 1.4e-6 of the three attention products (8.5e-7), against 2.1e-4 and 1.8e-4 that the weights leave.
//
// Every wait is bounded (common.cuh); a lost wait sets the context's error word, the CTA drains and frees its tensor memory.
#include <cstdlib>

#include "gemm_tc.cuh"
#include "tcgen05.cuh"
#include "tmap.h"

namespace lv {

constexpr int kTsProducers = 16;
constexpr int kTsThreads = (kTsProducers + 4) * 32;
constexpr int kTsMaxRaw = 8, kTsMaxB = 16;
constexpr uint32_t kTsABase = 256, kTsTileCols = kTcChunkK / 2;      // tensor memory: accumulators in columns 0..255, weights from 256 on
constexpr uint32_t kTsGateBytes = kTcMaxZ * 64 * sizeof(float);      // the epilogue's gate exchange
constexpr uint32_t kTsBarBytes = 640;
constexpr uint32_t kTsSmemBytes = 227 * 1024;
// Tiles of K per activation stage: two, where the raw stages leave room for four stages of 64 tokens (32 KB each).
template <int QT> __host__ __device__ constexpr uint32_t ts_b_tiles() { return QT == T_Q4_0 ? 2u : 1u; }

struct TsPlan {
    uint32_t units, per;       // units of the launch and of a CTA
    uint32_t groups;           // units of a tile
    uint32_t shares;           // 0: runs of `per` units; otherwise CTAs of a tile, each with an equal part of its units
    uint32_t n_raw, n_b;       // stages of the two rings
};

__device__ __forceinline__ float ts_silu(float up, float gate) { return up * gate / (expf(-gate) + 1.0f); }      // matmul_silu_ff.comp:95

// Where row 0 of token z goes in the f16 cache of matrix mi, or null (reported) beyond its end.
__device__ __forceinline__ __half* ts_cache_row(const GemmTcParams& p, const GemvMatrix& M, int mi, uint32_t z) {
    __half* cache = static_cast<__half*>(M.out);
    uint32_t at;
    if (p.group != nullptr) {                // matrix 0 is wk, matrix 2 is wv (lv_gemm_tc_qkv_kvappend_group)
        const lv_group_member& m = p.group[z];
        cache = static_cast<__half*>(mi == 0 ? m.k_cache : m.v_cache);
        at = *m.pos;
    } else {
        at = *p.pos + z;
    }
    if (at < p.ctx_rows) return cache + size_t(at) * M.rows;
    atomicOr(p.err, ERR_BAD_INDEX);
    return nullptr;
}

// A thread's 16 finished tokens of one row, tokens z0 .. of which the last is below Z.  All residuals of a thread, or the cache rows of a warp's tokens
// (lane i looks up token z0 + i), are on their way together: one trip to L2.  Called by whole warps; `live` is false for rows beyond the matrix.
__device__ __forceinline__ void ts_store16(const GemmTcParams& p, const GemvMatrix& M, int mi, uint32_t row, uint32_t z0, bool live, const float (&v)[16]) {
    if (M.epilogue == EPI_STORE_F16_AT_POS) {
        const uint32_t lane = threadIdx.x & 31u;
        const __half* at = lane < 16 && z0 + lane < p.Z ? ts_cache_row(p, M, mi, z0 + lane) : nullptr;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            __half* to = reinterpret_cast<__half*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(at), i));
            if (live && to != nullptr) to[row] = __float2half_rn(v[i]);
        }
        return;
    }
    if (!live) return;
    float* o = static_cast<float*>(M.out) + size_t(z0) * M.rows + row;
    if (M.epilogue == EPI_ADD) {                                                       // matmul.glsl:68-72
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (z0 + i < p.Z) x[i] = o[size_t(i) * M.rows];
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (z0 + i < p.Z) o[size_t(i) * M.rows] = x[i] + v[i];
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (z0 + i < p.Z) o[size_t(i) * M.rows] = v[i];
    }
}

// The words of a raw row that tile TT of its group needs, in 16-byte loads: the tile's two blocks (36 / 68 bytes) start at byte 36 TT /
// 68 TT, in chunk 2 TT / 4 TT and TT words into it.
template <int QT> __host__ __device__ constexpr int ts_tile_words() { return tc_raw_row_bytes<QT>() / 16; }          // 9 / 17
template <int QT> __host__ __device__ constexpr int ts_load_chunks() { return (ts_tile_words<QT>() + 3 + 3) / 4; }    // 3 / 5

// Two blocks of a row -> 32 registers in element order (column j = elements 2j, 2j + 1), each fp16(w) with w = (q - 8) d or q d: the
// quants are widened by placing them in the mantissa of a power of two whose last place is their unit (1024 for the low nibble, 64 for
// the high one, which so needs no shift), the offset is subtracted exactly and the product rounded once.
// Block 0: scale in the low half of word 0, payload shifted by two bytes; block 1: scale in the high half of the middle word, payload
// word-aligned.
template <int QT, int TT>
__device__ __forceinline__ void ts_dequant(const uint32_t (&L)[4 * ts_load_chunks<QT>()], uint32_t (&cols)[32]) {
    constexpr int kQW = (ts_tile_words<QT>() - 1) / 2;                    // payload words of a block: 4 / 8
    auto product = [](uint32_t bits, __half2 off, __half2 d2) {
        const __half2 v = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&bits), off), d2);
        return *reinterpret_cast<const uint32_t*>(&v);
    };
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        const uint32_t dbits = b == 0 ? __byte_perm(L[TT], 0u, 0x1010) : __byte_perm(L[TT + kQW], 0u, 0x3232);
        const __half2 d2 = *reinterpret_cast<const __half2*>(&dbits);
#pragma unroll
        for (int k = 0; k < kQW; ++k) {
            // bytes 0, 1 and 2, 3 of payload word k
            const uint32_t lo = b == 0 ? L[TT + k] : L[TT + kQW + 1 + k], hi = b == 0 ? L[TT + k + 1] : lo;
            if constexpr (QT == T_Q4_0) {
                // low nibbles = elements 4k .. 4k+3, high nibbles = 16 + 4k .. 19 + 4k
                const uint32_t v01 = __byte_perm(lo, 0u, b == 0 ? 0x4342 : 0x4140), v23 = __byte_perm(hi, 0u, b == 0 ? 0x4140 : 0x4342);
                const __half2 off_lo = __floats2half2_rn(1032.0f, 1032.0f), off_hi = __floats2half2_rn(72.0f, 72.0f);
                cols[16 * b + 2 * k] = product((v01 & 0x000f000fu) | 0x64006400u, off_lo, d2);
                cols[16 * b + 2 * k + 1] = product((v23 & 0x000f000fu) | 0x64006400u, off_lo, d2);
                cols[16 * b + 8 + 2 * k] = product((v01 & 0x00f000f0u) | 0x54005400u, off_hi, d2);
                cols[16 * b + 8 + 2 * k + 1] = product((v23 & 0x00f000f0u) | 0x54005400u, off_hi, d2);
            } else {
                // int8 in element order; the sign bit is flipped (q + 128) on the way into the mantissa of 1024
                const uint32_t u01 = __byte_perm(lo, 0x64646464u, b == 0 ? 0x4342 : 0x4140), u23 = __byte_perm(hi, 0x64646464u, b == 0 ? 0x4140 : 0x4342);
                const __half2 off = __floats2half2_rn(1152.0f, 1152.0f);
                cols[16 * b + 2 * k] = product(u01 ^ 0x00800080u, off, d2);
                cols[16 * b + 2 * k + 1] = product(u23 ^ 0x00800080u, off, d2);
            }
        }
    }
}

template <int QT>
__global__ void __launch_bounds__(kTsThreads, 1) gemm_tc_stream_kernel(const GemmTcParams p, const TsPlan plan, const __grid_constant__ GemmTcMaps maps) {
    pdl_launch_dependents();
    extern __shared__ uint8_t smem_raw[];
    // swizzled tiles need 1024-byte alignment
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023));
    constexpr int kRawRowBytes = tc_raw_row_bytes<QT>(), kRawStage = tc_raw_stage<QT>();
    const uint32_t b_tile = 2u * p.zpad * kTcChunkK * 2u;        // bytes of 64 columns of both planes
    constexpr uint32_t kBT = ts_b_tiles<QT>();
    const uint32_t b_stage = kBT * b_tile;
    uint8_t* bring = smem;
    uint8_t* rawring = bring + plan.n_b * b_stage;
    float* gate_s = reinterpret_cast<float*>(rawring + plan.n_raw * kRawStage);          // [64 tokens][64 rows]
    uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(gate_s) + kTsGateBytes);
    uint64_t* raw_full = bars;                              // [8]
    uint64_t* raw_empty = raw_full + kTsMaxRaw;             // [8]
    uint64_t* b_full = raw_empty + kTsMaxRaw;               // [16]
    uint64_t* b_empty = b_full + kTsMaxB;                   // [16]
    uint64_t* a_full = b_empty + kTsMaxB;                   // [buffer][half]
    uint64_t* a_empty = a_full + 4;                         // [buffer][half]
    uint64_t* acc_full = a_empty + 4;
    uint64_t* acc_empty = acc_full + 1;
    uint64_t* group_bar = acc_empty + 1;                    // [4] the four warps of a token group
    constexpr int kBars = 2 * kTsMaxRaw + 2 * kTsMaxB + 14;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kBars);
    volatile uint32_t* s_seen = tmem_slot + 1;              // [4] arrivals at the last tile as the four warps of a token group go by
    volatile uint32_t* s_late = s_seen + 4;                 // [2][4] this CTA's warps were the last to arrive at the first / last tile
    static_assert(kBars * 8 + 13 * 4 <= int(kTsBarBytes), "barrier area");

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool pair = p.m[0].w_gate != nullptr;
    const uint32_t rows_per_tile = pair ? kTcRows / 2 : kTcRows;
    const uint32_t t0 = (p.m[0].rows + rows_per_tile - 1) / rows_per_tile;
    const uint32_t t1 = t0 + (p.n_mat > 1 ? (p.m[1].rows + rows_per_tile - 1) / rows_per_tile : 0);
    // which matrix a tile belongs to, and its first row there (a last tile may reach past the matrix: the tensor map fills the
    // missing rows with zero blocks and the epilogue leaves them out)
    auto matrix_of = [&](uint32_t tile, uint32_t& row0) {
        const int mi = (p.n_mat > 1 && tile >= t1) ? 2 : (tile >= t0 ? 1 : 0);
        row0 = (tile - (mi == 2 ? t1 : (mi == 1 ? t0 : 0))) * rows_per_tile;
        return mi;
    };
    const uint32_t G = plan.groups, shares = plan.shares, share = shares != 0 ? blockIdx.x % shares : 0u;
    const uint32_t u0 = shares != 0 ? blockIdx.x / shares * G + G * share / shares : blockIdx.x * plan.per;
    const uint32_t n_units = (shares != 0 ? u0 - G * share / shares + G * (share + 1) / shares : min(plan.units, u0 + plan.per)) - u0;
    const uint32_t tile0 = u0 / G, g0 = u0 - tile0 * G;     // where this CTA's run begins
    // the CTAs that work on tile t
    auto first_of = [&](uint32_t t) { return shares != 0 ? t * shares : t * G / plan.per; };
    auto last_of = [&](uint32_t t) { return shares != 0 ? t * shares + shares - 1 : ((t + 1) * G - 1) / plan.per; };
    const uint32_t bank_cols = 2u * p.zpad;

    // one barrier per thread (a single thread takes about a microsecond for all of them)
    if (threadIdx.x < kBars) {
        const int i = int(threadIdx.x);
        uint32_t count = 1;                                                            // raw_full, b_full, b_empty, a_empty
        if (i >= kTsMaxRaw && i < 2 * kTsMaxRaw) count = kTsProducers;                  // raw_empty
        else if (i >= 2 * kTsMaxRaw + 2 * kTsMaxB) {
            const int j = i - 2 * kTsMaxRaw - 2 * kTsMaxB;
            if (j < 4) count = kTsProducers / 2;                                        // a_full: the eight warps of a half
            else if (j == 8) count = 2;                                                 // acc_full: both issuing lanes
            else if (j == 9) count = kTsProducers;                                      // acc_empty
            else if (j >= 10) count = 4;                                                // group_bar
        }
        mbar_init(&bars[i], count);
        fence_mbar_init();
    }
    if (threadIdx.x >= kTsThreads - 8) s_late[threadIdx.x - (kTsThreads - 8)] = 0;
    if (warp == kTsProducers + 1) tc_alloc(tmem_slot, 512);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    constexpr uint32_t tmem_base = 0;                       // the allocation is all of the tensor memory

    bool ok = true;
    uint32_t issued = 0;                                    // stages that a ring or issuing warp has asked for

    if (warp == kTsProducers) {
        // ---------------- raw ring: weights do not depend on the previous kernel ----------------
        if (lane == 0) {
            uint32_t tile = tile0, g = g0, row0, rs = 0, phase = 1;
            int mi = matrix_of(tile, row0);
            for (uint32_t i = 0; i < n_units && ok; ++i) {
                if (i >= plan.n_raw) ok = mbar_wait(&raw_empty[rs], phase, p.err);
                if (!ok) break;
                uint8_t* dst = rawring + rs * kRawStage;
                const int x = int(g * (kRawRowBytes / 8));
                mbar_expect_tx(&raw_full[rs], kRawStage);
                if (pair) {
                    tma_load_2d_plain(dst, &maps.w[0], x, int(row0), &raw_full[rs]);                                      // w3 rows -> tile rows 0..63
                    tma_load_2d_plain(dst + (kTcRows / 2) * kRawRowBytes, &maps.gate, x, int(row0), &raw_full[rs]);      // w1 rows -> 64..127
                } else {
                    tma_load_2d_plain(dst, mi == 0 ? &maps.w[0] : (mi == 1 ? &maps.w[1] : &maps.w[2]), x, int(row0), &raw_full[rs]);
                }
                ++issued;
                if (++rs == plan.n_raw) { rs = 0; phase ^= 1u; }
                if (++g == G) { g = 0; mi = matrix_of(++tile, row0); }
            }
        }
    } else if (warp == kTsProducers + 3) {
        // ---------------- activation ring -------------------------------------------------------
        if (lane == 0) {
            pdl_wait();                                        // the activations come from the previous kernel
            const uint8_t* xh = reinterpret_cast<const uint8_t*>(p.xh);
            uint32_t g = g0, bs = 0, phase = 1;
            constexpr uint32_t kStages = 4 / kBT;              // stages of a unit; consecutive ones belong to the two MMA lanes in turn
            for (uint32_t i = 0; i < kStages * n_units && ok; ++i) {
                if (i >= plan.n_b) ok = mbar_wait(&b_empty[bs], phase, p.err);
                if (!ok) break;
                const uint32_t j = i % kStages, t = kBT == 2 ? 2 * j : 2 * (j & 1u) + (j >> 1);       // first tile of the stage
                mbar_expect_tx(&b_full[bs], b_stage);
                bulk_g2s(bring + bs * b_stage, xh + size_t(4 * g + t) * b_tile, b_stage, &b_full[bs]);
                ++issued;
                if (++bs == plan.n_b) { bs = 0; phase ^= 1u; }
                if (j + 1 == kStages && ++g == G) g = 0;
            }
        }
    } else if (warp > kTsProducers) {
        // ---------------- MMA lanes ---------------------------------------------------------------
        // (the whole warp runs the loop and one elected lane issues: operands that the compiler knows to be the same for the warp
        // go to the tensor core without a detour through the lanes)
        const uint32_t h = uint32_t(__shfl_sync(0xffffffffu, warp, 0)) - (kTsProducers + 1);
        // fp32 accumulator, fp16 A and B, both K-major, M = 128, N = 2 zpad
        const uint32_t idesc = (1u << 4) | ((uint32_t(kTcRows) >> 4) << 24) | (((2u * p.zpad) >> 3) << 17);
        const uint64_t b_desc0 = tc_smem_desc(smem_u32(bring));
        const uint32_t bank = tmem_base + h * bank_cols;
        uint32_t g = g0, bs = h, b_phase = 0, seg = 0;
        bool first = true;
        for (uint32_t i = 0; i < n_units && ok; ++i) {
            const uint32_t ab = i & 1u;
            // the accumulators of the previous segment have been read
            if (first && seg > 0) ok = mbar_wait_all(acc_empty, (seg - 1) & 1u, p.err);
            ok = ok && mbar_wait_all(&a_full[2 * ab + h], (i >> 1) & 1u, p.err);
            const uint32_t a_tmem = tmem_base + kTsABase + (4u * ab + 2u * h) * kTsTileCols;
#pragma unroll
            for (uint32_t st = 0; st < 2 / kBT; ++st) {
                ok = ok && mbar_wait_all(&b_full[bs], b_phase, p.err);
                if (!ok) break;
                tc_fence_after_sync();
                const uint64_t b_desc = b_desc0 + ((bs * b_stage) >> 4);
                if (tc_elect()) {
#pragma unroll
                    for (uint32_t t = 0; t < kBT; ++t)
#pragma unroll
                        for (int k = 0; k < kTcChunkK / 16; ++k)          // 16 fp16 along K = 2 address units of B = 8 TMEM columns of A
                            tc_mma_f16_ta(bank, a_tmem + (st + t) * kTsTileCols + 8u * k, b_desc + t * (b_tile >> 4) + 2u * k, idesc,
                                          (!first || st + t != 0 || k != 0) ? 1u : 0u);
                    tc_commit(&b_empty[bs]);
                }
                __syncwarp();
                ++issued;
                bs += 2;
                if (bs >= plan.n_b) { bs -= plan.n_b; b_phase ^= 1u; }
            }
            if (!ok) break;
            first = ++g == G || i + 1 == n_units;
            if (tc_elect()) {
                tc_commit(&a_empty[2 * ab + h]);
                if (first) tc_commit(acc_full);
            }
            __syncwarp();
            if (first) {
                g = 0;
                ++seg;
            }
        }
    } else {
        // ---------------- producers ---------------------------------------------------------------
        const uint32_t quarter = uint32_t(warp) & 3u, tt = uint32_t(warp) >> 2, half = tt >> 1;
        const uint32_t tr = quarter * 32u + uint32_t(lane);             // tile row
        const uint32_t lanes_at = (quarter * 32u) << 16;

        // Sixteen tokens of a tile belong to the four warps of one `tt`, a thread has one row of them.  These four warps finish a tile whose
        // parts come from several CTAs on their own: the counter of (tile, tt) counts warps.
        const uint32_t z0 = 16u * tt;
        const bool active = z0 < p.zpad;
        uint32_t met = 0;
        auto group_sync = [&]() {                                        // (a bounded wait: a warp may have given up elsewhere)
            __syncwarp();
            if (lane == 0) mbar_arrive(&group_bar[tt]);
            ok = ok && mbar_wait_all(&group_bar[tt], met & 1u, p.err);
            ++met;
            return ok;
        };
        auto part_of = [&](uint32_t c, uint32_t t) {                     // CTA c's part of tile t: its first segment, or its last
            const uint32_t slot = shares != 0 || c * plan.per >= t * G ? 0u : 1u;
            return p.scratch + (size_t(2 * c + slot) * p.zpad + z0) * kTcRows + tr;
        };
        // This warp's share of a part is in memory.  One lane orders what the warp has stored before the addition and, where it is the last, the addition
        // before the flag that sends the group to the other parts.
        auto arrive = [&](uint32_t t, uint32_t which) {
            __syncwarp();
            if (lane == 0 && atom_add_release_gpu(&p.counters[4 * t + tt], 1u) + 1 == 4 * (last_of(t) - first_of(t) + 1)) {
                __threadfence();
                s_late[4 * which + tt] = 1;
            }
        };
        // adds the parts of tile t in the order of K (`own` of them from v, none when it is no CTA) and leaves the counter ready for the next launch
        auto add_parts = [&](uint32_t t, uint32_t own, float (&v)[16]) {
            const uint32_t c_last = last_of(t);
            float sum[16] = {};
#pragma unroll 1
            for (uint32_t c = first_of(t); c <= c_last; ++c) {
                float x[16];
                const float* q = part_of(c, t);
#pragma unroll
                for (int i = 0; i < 16; ++i) x[i] = c == own ? v[i] : __ldcg(q + size_t(i) * kTcRows);
#pragma unroll
                for (int i = 0; i < 16; ++i) sum[i] += x[i];
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = sum[i];
            if (quarter == 0 && lane == 0) p.counters[4 * t + tt] = 0;
        };
        auto store = [&](uint32_t t, float (&v)[16]) {
            uint32_t row0;
            const int mi = matrix_of(t, row0);
            const GemvMatrix& M = p.m[mi];
            if (!pair) {
                ts_store16(p, M, mi, row0 + tr, z0, row0 + tr < M.rows, v);
                return;
            }
            // Tile rows 64..127 carry the gate (w1) of rows 0..63.  The two warps of a row hand each other eight tokens of what they have and finish
            // eight each, four at a time in a loop that stays one: this code runs once or twice per launch, and unrolled it took 12 us (11008 x 4096, 16
            // tokens), nearly all of it instruction fetches.
            const bool gate = quarter >= 2;
            float* swap = gate_s + z0 * 64 + (tr & 63u);
#pragma unroll
            for (int i = 0; i < 8; ++i) swap[(gate ? i : i + 8) * 64] = gate ? v[i] : v[i + 8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = gate ? v[i + 8] : v[i];
            if (!group_sync()) return;
            const uint32_t row = row0 + (tr & 63u), from = gate ? 8 : 0;
            if (row < M.rows) {
#pragma unroll 1
                for (uint32_t at = from; at < from + 8 && z0 + at < p.Z; at += 4) {
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) {
                        const float other = swap[(at + i) * 64], y = ts_silu(gate ? other : v[i], gate ? v[i] : other);
                        const uint32_t z = z0 + at + i;
                        if (z >= p.Z) break;
                        if (p.split_out != nullptr) split_store(p.split_out, p.zpad, z, row, y);
                        else static_cast<float*>(M.out)[size_t(z) * M.rows + row] = y;
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[i] = v[i + 4];
                }
            }
            group_sync();
        };

        // Reads the accumulators of segment `seg` and stores them, or parks them as a part.  The CTA whose last segment completes a tile (the parts
        // of the others having arrived long ago, as first segments do) adds them to the values that it holds and leaves nothing behind.  Returns whether a
        // part was parked whose arrival has still to be reported.
        auto drain = [&](uint32_t seg, uint32_t tile, bool whole, uint32_t slot, bool final) {
            pdl_wait();                                        // (outputs, parts and counters may still be in use by the previous kernel)
            uint32_t seen = 0;
            const uint32_t parts = last_of(tile) - first_of(tile) + 1;
            if (!whole && final && active && quarter == 0 && lane == 0) seen = ld_acquire_gpu(&p.counters[4 * tile + tt]);
            ok = mbar_wait_warp_tc(acc_full, seg & 1u, p.err);
            if (!ok) return false;
            tc_fence_after_sync();
            float v[16];
            if (active) {
                uint32_t a[16], b[16];
                tc_load16(a, tmem_base + lanes_at + z0);
                tc_load16(b, tmem_base + lanes_at + p.zpad + z0);
                tc_wait_load();
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(b[i]) + __uint_as_float(a[i]);      // the small terms first
                tc_load16(a, tmem_base + lanes_at + bank_cols + z0);
                tc_load16(b, tmem_base + lanes_at + bank_cols + p.zpad + z0);
                tc_wait_load();
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] += __uint_as_float(b[i]) + __uint_as_float(a[i]);
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty);
            if (!active) return false;
            if (!whole) {
                bool last = false;
                if (final) {
                    if (quarter == 0 && lane == 0) s_seen[tt] = seen;
                    if (!group_sync()) return false;
                    last = s_seen[tt] == 4 * (parts - 1);
                }
                if (!last) {
                    float* part = p.scratch + (size_t(2 * blockIdx.x + slot) * p.zpad + z0) * kTcRows + tr;
#pragma unroll
                    for (int i = 0; i < 16; ++i) __stcg(part + size_t(i) * kTcRows, v[i]);
                    if (!final) return true;
                    arrive(tile, 1);
                    if (!group_sync() || s_late[4 + tt] == 0) return false;
                }
                add_parts(tile, blockIdx.x, v);
            }
            store(tile, v);
            return false;
        };

        uint32_t tile = tile0, g = g0, seg = 0, seg_begin = g0, rs = 0, raw_phase = 0;
        bool pending = false, pend_whole = false, parked = false;
        uint32_t pend_tile = 0, pend_slot = 0, pend_seg = 0;
        // the raw words of a unit are fetched while the one before it is dequantised (rows are 9 / 17 chunks of 16 bytes apart, so a
        // quarter warp's loads fall into different banks)
        uint32_t L[4 * ts_load_chunks<QT>()];
        auto fetch = [&]() {
            ok = mbar_wait_all(&raw_full[rs], raw_phase, p.err);
            if (!ok) return;
            const uint4* src = reinterpret_cast<const uint4*>(rawring + rs * kRawStage + tr * kRawRowBytes) + (QT == T_Q4_0 ? 2u : 4u) * tt;
#pragma unroll
            for (int c = 0; c < ts_load_chunks<QT>(); ++c) {
                const uint4 v = src[c];
                L[4 * c] = v.x; L[4 * c + 1] = v.y; L[4 * c + 2] = v.z; L[4 * c + 3] = v.w;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&raw_empty[rs]);
            if (++rs == plan.n_raw) { rs = 0; raw_phase ^= 1u; }
        };
        fetch();
        for (uint32_t i = 0; i < n_units && ok; ++i) {
            uint32_t cols[32];
            switch (tt) {                      // (the same for the whole warp)
                case 0: ts_dequant<QT, 0>(L, cols); break;
                case 1: ts_dequant<QT, 1>(L, cols); break;
                case 2: ts_dequant<QT, 2>(L, cols); break;
                default: ts_dequant<QT, 3>(L, cols); break;
            }
            if (i + 1 < n_units) fetch();
            if (!ok) break;
            const uint32_t ab = i & 1u;
            if (i >= 2) {
                ok = mbar_wait_all(&a_empty[2 * ab + half], ((i >> 1) - 1) & 1u, p.err);
                if (!ok) break;
                tc_fence_after_sync();
            }
            const uint32_t taddr = tmem_base + lanes_at + kTsABase + (4u * ab + tt) * kTsTileCols;
            asm volatile(
                "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
                "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
                ::"r"(taddr), "r"(cols[0]), "r"(cols[1]), "r"(cols[2]), "r"(cols[3]), "r"(cols[4]), "r"(cols[5]), "r"(cols[6]), "r"(cols[7]),
                  "r"(cols[8]), "r"(cols[9]), "r"(cols[10]), "r"(cols[11]), "r"(cols[12]), "r"(cols[13]), "r"(cols[14]), "r"(cols[15]),
                  "r"(cols[16]), "r"(cols[17]), "r"(cols[18]), "r"(cols[19]), "r"(cols[20]), "r"(cols[21]), "r"(cols[22]), "r"(cols[23]),
                  "r"(cols[24]), "r"(cols[25]), "r"(cols[26]), "r"(cols[27]), "r"(cols[28]), "r"(cols[29]), "r"(cols[30]), "r"(cols[31])
                : "memory");
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[2 * ab + half]);
            if (parked) {                      // one unit after its stores
                arrive(tile0, 0);
                parked = false;
            }
            if (pending) {
                parked = drain(pend_seg, pend_tile, pend_whole, pend_slot, false);
                pending = false;
            }
            if (++g == G || i + 1 == n_units) {
                pending = true;
                pend_whole = seg_begin == 0 && g == G;
                pend_tile = tile;
                pend_slot = (seg == 0) ? 0u : 1u;
                pend_seg = seg;
                ++seg;
                ++tile;
                g = seg_begin = 0;
            }
        }
        // (After a lost wait, whose error word ends every later one, arrivals stay out and the warps of a CTA may disagree about `ok`: every wait of theirs for one
        // another is bounded, and gemm_tc_reset takes the counters back to 0 when the error is reported.)
        if (ok && parked) arrive(tile0, 0);
        if (ok && pending) drain(pend_seg, pend_tile, pend_whole, pend_slot, true);
        // the part of the first tile was the last one after all
        if (ok && active && group_sync() && s_late[tt] != 0) {
            float v[16];
            add_parts(tile0, 0xffffffffu, v);
            store(tile0, v);
        }
    }
    tc_fence_before_sync();
    if (__syncthreads_or(!ok)) {
        // a wait was lost: copies and products that are on their way end before shared and tensor memory are given back
        auto drain_ring = [&](uint64_t* full, uint32_t n) {
            for (uint32_t s = 0; s < min(issued, n); ++s) mbar_drain(&full[s], ((issued - 1 - s) / n) & 1u);
        };
        if (lane == 0 && warp == kTsProducers) drain_ring(raw_full, plan.n_raw);
        else if (lane == 0 && warp == kTsProducers + 3) drain_ring(b_full, plan.n_b);
        else if (lane == 0 && warp > kTsProducers && issued != 0) {
            const uint32_t own = plan.n_b / 2, last = issued - 1;          // the last stage of this issuing lane's half of the ring
            mbar_drain(&b_empty[2 * (last % own) + uint32_t(warp) - (kTsProducers + 1)], (last / own) & 1u);
        }
        __syncthreads();
    }
    if (warp == kTsProducers + 1) {
        tc_fence_after_sync();
        tc_free(tmem_base, 512);
    }
}

int gemm_tc_stream_configure(lv_ctx* ctx) {
    LV_REQUIRE(size_t(ctx->max_smem_optin) >= size_t(kTsSmemBytes), "device has too little shared memory for the batched product");
    LV_CUDA((cudaFuncSetAttribute(gemm_tc_stream_kernel<T_Q4_0>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTsSmemBytes))));
    LV_CUDA((cudaFuncSetAttribute(gemm_tc_stream_kernel<T_Q8_0>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTsSmemBytes))));
    return LV_OK;
}

template <int QT>
static int launch_typed(lv_ctx* ctx, const GemmTcParams& p, const GemmTcMaps& maps, uint32_t tiles) {
    TsPlan plan{};
    plan.groups = p.K / (4 * kTcChunkK);
    plan.units = tiles * plan.groups;
    const uint32_t sms = uint32_t(ctx->sm_count);
    // Equal runs; at least two units each (one instead of two: 2048 x 2048 6.7 -> 8.4 us, 512 x 5632 9.9 -> 13.3).
    plan.per = max((plan.units + sms - 1) / sms, min(2u, plan.groups));
    // Runs that begin and end inside tiles have two segments, and tiles up to eight parts: about two units more for the CTA that ends last.  Where
    // equal shares of every tile fit the SMs with no more units than that, each CTA has one segment.  us per launch back to back, q4_0, runs -> shares:
    //   tokens   2048 x 5632    3 x 2048 x 2048   5120 x 5120    4096 x 11008    1408 x 4096 pair   8192 x 4096     (three units more:) 5120 x 13824   6656 x 6656
    //     16     10.4 ->  9.7    9.2 ->  8.9      12.3 -> 12.1   17.6 -> 17.3    10.2 ->  9.9       13.9 -> 13.6                        22.9 -> 24.2    16.6 -> 18.1
    //     64     13.6 -> 12.6   11.5 -> 10.8      14.8 -> 14.3   20.9 -> 19.8    13.1 -> 12.5       16.7 -> 15.6                        26.3 -> 26.8    19.7 -> 20.2
    // and the same in q8_0.
    const uint32_t most = sms / tiles, n_shares = most == 0 ? 0 : max((plan.groups + most - 1) / most, min(2u, plan.groups));      // units of a CTA
    if (most > 1 && plan.groups % plan.per != 0 && n_shares <= plan.per + 2) plan.shares = (plan.groups + n_shares - 1) / n_shares;
    // whole tiles only, where the arrival counters or the scratch (two parts per CTA) would not do
    static const char* no_split = getenv("LV_GEMM_TC_NO_SPLIT");
    if (tiles > kTcMaxTiles || size_t(sms) * 2 * p.zpad * kTcRows * sizeof(float) > kTcScratchBytes || (no_split != nullptr && no_split[0] == '1'))
        plan.per = (tiles + sms - 1) / sms * plan.groups, plan.shares = 0;
    // shared memory: up to 128 KB of activations (96 KB beside the larger q8_0 stages) in an even number of stages, the rest raw stages
    const uint32_t b_stage = ts_b_tiles<QT>() * 4u * p.zpad * kTcChunkK;
    plan.n_b = min(uint32_t(kTsMaxB), (QT == T_Q4_0 ? 131072u : 98304u) / b_stage) & ~1u;
    plan.n_raw = min(uint32_t(kTsMaxRaw), (kTsSmemBytes - 1024 - kTsGateBytes - kTsBarBytes - plan.n_b * b_stage) / uint32_t(tc_raw_stage<QT>()));
    LV_CUDA((launch_pdl(ctx, gemm_tc_stream_kernel<QT>, dim3(plan.shares != 0 ? tiles * plan.shares : (plan.units + plan.per - 1) / plan.per), dim3(kTsThreads), kTsSmemBytes, p, plan, maps)));
    return LV_OK;
}

int launch_gemm_tc_stream(lv_ctx* ctx, const GemmTcParams& p, const GemmTcMaps& maps, int wtype, uint32_t tiles) {
    return wtype == T_Q4_0 ? launch_typed<T_Q4_0>(ctx, p, maps, tiles) : launch_typed<T_Q8_0>(ctx, p, maps, tiles);
}

}  // namespace lv
