// What the batched products over quantised weights share: gemm_tc.cu (weight tiles in shared memory) and
// gemm_tc_stream.cu (weight tiles in tensor memory, the default).
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "ctx.h"
#include "gemv_stream.cuh"

namespace lv {

constexpr int kTcRows = 128;                   // rows of W per CTA = M of the MMA
constexpr int kTcMaxZ = 64;                    // tokens per launch = N of the MMA (padded to 16)
constexpr int kTcChunkK = 64;                  // K per A/B tile: 64 fp16 = one 128-byte swizzle row
constexpr int kTcRawBlocks = 8;                // q-blocks of a row per raw stage (4 tiles of K)

template <int QT> struct TcTraits;
template <> struct TcTraits<T_Q4_0> { static constexpr int kBlockBytes = kQ4BlockBytes; };
template <> struct TcTraits<T_Q8_0> { static constexpr int kBlockBytes = kQ8BlockBytes; };
template <int QT> __host__ __device__ constexpr int tc_raw_row_bytes() { return kTcRawBlocks * TcTraits<QT>::kBlockBytes; }       // 144 / 272
template <int QT> __host__ __device__ constexpr int tc_raw_stage() { return kTcRows * tc_raw_row_bytes<QT>(); }                   // 18432 / 34816

constexpr size_t kTcScratchBytes = size_t(32) << 20;
constexpr uint32_t kTcMaxTiles = 1024;
constexpr size_t kTcCounterBytes = 4 * kTcMaxTiles * sizeof(uint32_t);

struct GemmTcParams {
    GemvMatrix m[3];         // same meaning as in the GEMV; w_gate set = SiLU pair (64 + 64 rows per CTA)
    int n_mat;
    const uint32_t* pos;     // device word for EPI_STORE_F16_AT_POS
    uint32_t K;
    uint32_t Z;              // tokens (columns actually written)
    uint32_t zpad;           // Z rounded up to 16 = N of the MMA
    uint32_t ctx_rows;
    const __half* xh;        // split activations, one contiguous pre-swizzled B tile per 64 columns of K (act_split_kernel)
    uint32_t splits;         // CTAs that share one tile of rows, each taking a contiguous range of K
    float* scratch;          // splits > 1: partial accumulators [tile][split][zpad][128]; gemm_tc_stream.cu: [CTA][first, last tile][zpad][128]
    uint32_t* counters;      // arrivals per tile; gemm_tc_stream.cu: per tile and sixteen tokens (zero between launches; after an error gemm_tc_reset sees to it)
    uint32_t* err;
    __half* split_out;       // SiLU pairs, gemm_tc_stream.cu: finished rows go there as the split activations of the next product, not to m[0].out
    const lv_group_member* group;   // non-null: token z is member z of a group step; cache rows go to its own caches at its own position
};

struct GemmTcMaps {
    CUtensorMap w[3];
    CUtensorMap gate;
};

// Eight nibbles of one word -> fp16((q - 8) * d), same output order as dequant_word.
__device__ __forceinline__ void dequant_word_hi(uint32_t w, __half2 d2, uint32_t (&hi)[4]) {
    const uint32_t v01 = __byte_perm(w, 0u, 0x4140), v23 = __byte_perm(w, 0u, 0x4342);
    const uint32_t raw[4] = {(v01 & 0x000f000fu) | 0x64006400u, (v23 & 0x000f000fu) | 0x64006400u,
                             ((v01 >> 4) & 0x000f000fu) | 0x64006400u, ((v23 >> 4) & 0x000f000fu) | 0x64006400u};
    const __half2 off = __floats2half2_rn(1032.0f, 1032.0f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __half2 h = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&raw[i]), off), d2);
        hi[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
}

// Four int8 of one word -> fp16(q * d): out[0] = elements (4k, 4k+1), out[1] = (4k+2, 4k+3).
__device__ __forceinline__ void dequant_word_q8_hi(uint32_t w, __half2 d2, uint32_t (&out)[2]) {
    const uint32_t u = w ^ 0x80808080u;                                       // q + 128 as unsigned bytes
    const uint32_t raw[2] = {__byte_perm(u, 0x64646464u, 0x4140), __byte_perm(u, 0x64646464u, 0x4342)};   // 1024 + 128 + q
    const __half2 off = __floats2half2_rn(1152.0f, 1152.0f);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const __half2 h = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&raw[i]), off), d2);
        out[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
}

int gemm_tc_stream_configure(lv_ctx* ctx);
int launch_gemm_tc_stream(lv_ctx* ctx, const GemmTcParams& p, const GemmTcMaps& maps, int wtype, uint32_t tiles);      // gemm_tc_stream.cu

}  // namespace lv
