// Matrix-vector products with bfloat16 weights: the decode-side products of models whose weights are not quantised.
//
//   lv_gemv_bf16                 one matrix (stacked projections that share an input); optional factor and activation
//   lv_gemv_bf16_mingru          three products per channel and the gated recurrence on them in the epilogue
//   lv_gemv_bf16_expert_gate_up  silu(gate x) * (up x) of the experts that a table gives a token
//   lv_gemv_bf16_expert_down     the mean of those experts' down products
//
// Weights are bfloat16 [rows][ld] (ld a multiple of 8, the tail of a row zero), inputs and results f32 and the arithmetic
// f32 throughout: a bfloat16 weight is exact in f32, so the same kernels serve a 32-bit evaluation.  The bound is HBM: two
// bytes per multiply-add, each weight read once.  A warp computes two or three rows, lanes taking 16 bytes of every row per
// step with four steps in flight (up to 6 KB per warp); the first weights are requested before the previous kernel has
// finished.  Lanes are combined by shuffles in a fixed order, so a result does not depend on the launch.  Matrices with few rows
// are cut along K over the warps of a CTA, so that enough loads are in flight.
//
// gridDim.y = tokens: every token has its own pass over the weights.  Prompts use gemm_bf16.cu instead.
#include <cuda_bf16.h>

#include "common.cuh"
#include "ctx.h"

namespace lv {

constexpr int kGbWarps = 8, kGbThreads = kGbWarps * 32;
constexpr int kGbUnroll = 4;

// (Not ld.global.nc, which says that nobody writes these bytes: the assembler then moves requests behind the wait for the previous kernel.  us in a chain of launches,
// nc / this: 1024 x 1024 2.45 / 1.94, 2048 x 2048 3.40 / 2.61, 3072 x 2048 4.93 / 4.17, 9280 x 2048 8.36 / 7.55.)
__device__ __forceinline__ uint4 gb_load_w(const __nv_bfloat16* p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

// eight consecutive inputs; those at or beyond K are zero
__device__ __forceinline__ void gb_load_x(float (&x)[8], const float* src, uint32_t k, uint32_t K) {
    if (k + 8 <= K) {
        const float4 a = *reinterpret_cast<const float4*>(src + k), b = *reinterpret_cast<const float4*>(src + k + 4);
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = k + i < K ? src[k + i] : 0.f;
    }
}

__device__ __forceinline__ void gb_fma(float& acc, uint4 w, const float (&x)[8]) {
    const uint32_t q[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        acc = fmaf(__uint_as_float(q[i] << 16), x[2 * i], acc);
        acc = fmaf(__uint_as_float(q[i] & 0xffff0000u), x[2 * i + 1], acc);
    }
}

struct GbSettled {
    __device__ __forceinline__ bool operator()() const { return false; }
};

// Partial dot products of NR rows with x over this lane's share of K.  WAIT: the rows are known before the previous kernel
// has finished and their first elements are requested before waiting for it.  settle: called after the wait; true: it has changed the rows
// (which were only a guess) and their first elements are requested again.
template <int NR, bool WAIT, typename Settle = GbSettled>
__device__ __forceinline__ void gb_dot(float (&acc)[NR], const __nv_bfloat16* const (&row)[NR], const float* x, uint32_t K, Settle settle = Settle()) {
    const uint32_t lane8 = (threadIdx.x & 31u) * 8u;
    uint4 w[kGbUnroll][NR];
    auto fetch = [&](uint32_t k0) {
#pragma unroll
        for (int u = 0; u < kGbUnroll; ++u) {
            const uint32_t k = k0 + u * 256u + lane8;
#pragma unroll
            for (int r = 0; r < NR; ++r) w[u][r] = k < K ? gb_load_w(row[r] + k) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    fetch(0);
    if constexpr (WAIT) pdl_wait();
    if (settle()) fetch(0);
    for (uint32_t k0 = 0; k0 < K; k0 += 256u * kGbUnroll) {
#pragma unroll
        for (int u = 0; u < kGbUnroll; ++u) {
            const uint32_t k = k0 + u * 256u + lane8;
            if (k < K) {
                float xv[8];
                gb_load_x(xv, x, k, K);
#pragma unroll
                for (int r = 0; r < NR; ++r) gb_fma(acc[r], w[u][r], xv);
            }
        }
        if (k0 + 256u * kGbUnroll < K) fetch(k0 + 256u * kGbUnroll);
    }
}

struct GemvBf16Params {
    const __nv_bfloat16* w[3];
    uint32_t rows;
    uint32_t ld, K;
    const float* x;
    uint32_t x_ld;
    float* out;
    uint32_t out_ld;
    float factor;
    int act;
};

// SPLIT: warps that share two rows
template <int SPLIT>
__global__ void __launch_bounds__(kGbThreads) gemv_bf16_kernel(const GemvBf16Params p) {
    pdl_launch_dependents();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t u = 2u * (blockIdx.x * (kGbWarps / SPLIT) + warp / SPLIT);
    float acc[2] = {0.f, 0.f};
    if constexpr (SPLIT == 1) {
        if (u >= p.rows) return;
        const __nv_bfloat16* row[2] = {p.w[0] + size_t(u) * p.ld, p.w[0] + size_t(min(u + 1, p.rows - 1)) * p.ld};
        gb_dot<2, true>(acc, row, p.x + size_t(blockIdx.y) * p.x_ld, p.K);
    } else {
        const uint32_t per = (p.K + SPLIT * 256 - 1) / (SPLIT * 256) * 256, first = warp % SPLIT * per, count = u < p.rows && first < p.K ? min(per, p.K - first) : 0;
        const __nv_bfloat16* row[2] = {p.w[0] + size_t(min(u, p.rows - 1)) * p.ld + first, p.w[0] + size_t(min(u + 1, p.rows - 1)) * p.ld + first};
        gb_dot<2, true>(acc, row, p.x + size_t(blockIdx.y) * p.x_ld + first, count);
    }
    float a0 = warp_sum(acc[0]), a1 = warp_sum(acc[1]);
    if constexpr (SPLIT > 1) {
        __shared__ float s_part[kGbWarps][2];
        if (lane == 0) { s_part[warp][0] = a0; s_part[warp][1] = a1; }
        __syncthreads();
        if (warp % SPLIT != 0) return;
        a0 = a1 = 0.f;
#pragma unroll
        for (int k = 0; k < SPLIT; ++k) { a0 += s_part[warp + k][0]; a1 += s_part[warp + k][1]; }
    }
    if (lane < 2 && u + lane < p.rows) p.out[size_t(blockIdx.y) * p.out_ld + u + lane] = product_act((lane ? a1 : a0) * p.factor, p.act);
}

__global__ void __launch_bounds__(kGbThreads) gemv_bf16_mingru_kernel(const GemvBf16Params p, const float* __restrict__ bz, const float* __restrict__ bx,
                                                                      float* __restrict__ state, const uint32_t* __restrict__ pos) {
    pdl_launch_dependents();
    const uint32_t c = blockIdx.x * kGbWarps + (threadIdx.x >> 5);
    if (c >= p.rows) return;
    const __nv_bfloat16* row[3] = {p.w[0] + size_t(c) * p.ld, p.w[1] + size_t(c) * p.ld, p.w[2] + size_t(c) * p.ld};
    float acc[3] = {0.f, 0.f, 0.f};
    gb_dot<3, true>(acc, row, p.x, p.K);
    const float az = warp_sum(acc[0]), ax = warp_sum(acc[1]), ag = warp_sum(acc[2]);
    if ((threadIdx.x & 31u) == 0) p.out[c] = mingru_step(az + bz[c], ax + bx[c], ag, *pos == 0 ? 0.f : state[c], &state[c]);
}

struct ExpertGemvParams {
    const __nv_bfloat16* gate;      // [experts * ff][ld]; the down matrix [experts * width][ld] in lv_gemv_bf16_expert_down
    const __nv_bfloat16* up;
    uint32_t ld, K, rows, experts, top, vocab;
    const uint32_t* table;          // [vocab][top]
    const uint32_t* token_log;
    const uint32_t* pos;
    uint32_t log_places;            // one token: places of token_log, 0 where its experts may not be looked up early
    const float* x;
    uint32_t x_ld;
    float* out;
    uint32_t out_ld;
    uint32_t* err;
};

__device__ __forceinline__ uint32_t gb_expert(const ExpertGemvParams& p, uint32_t t, uint32_t slot) {
    const uint32_t id = p.token_log[*p.pos + t];
    const uint32_t e = id < p.vocab ? p.table[size_t(id) * p.top + slot] : p.experts;
    if (e < p.experts) return e;
    if ((threadIdx.x & 31u) == 0) atomicOr(p.err, ERR_BAD_INDEX);      // (each warp looks up its own choices)
    return 0;
}

// The same before the previous kernel has finished: a guess.  The position and the token are those of the step unless an earlier launch
// that is still running writes them; whoever uses the guess asks again after the wait.
__device__ __forceinline__ uint32_t gb_expert_guess(const ExpertGemvParams& p, uint32_t slot) {
    const uint32_t at = *reinterpret_cast<const volatile uint32_t*>(p.pos);
    const uint32_t id = at < p.log_places ? *reinterpret_cast<const volatile uint32_t*>(p.token_log + at) : p.vocab;
    const uint32_t e = id < p.vocab ? p.table[size_t(id) * p.top + slot] : 0;
    return e < p.experts ? e : 0;
}

// A token's experts are known when the step begins, so one token's weights are on their way while the norm before it runs (a single CTA):
// half of a row of 2048 columns.
__global__ void __launch_bounds__(kGbThreads) gemv_bf16_expert_gate_up_kernel(const ExpertGemvParams p) {
    pdl_launch_dependents();
    const uint32_t t = blockIdx.y, slot = blockIdx.z;
    const uint32_t i = blockIdx.x * kGbWarps + (threadIdx.x >> 5);
    const __nv_bfloat16* row[2];
    auto rows_of = [&](uint32_t e) {
        const size_t at = (size_t(e) * p.rows + min(i, p.rows - 1)) * p.ld;
        row[0] = p.gate + at;
        row[1] = p.up + at;
    };
    float acc[2] = {0.f, 0.f};
    if (p.log_places != 0) {
        const uint32_t guess = gb_expert_guess(p, slot);
        rows_of(guess);
        gb_dot<2, true>(acc, row, p.x, p.K, [&]() {
            const uint32_t e = gb_expert(p, 0, slot);
            if (e == guess) return false;
            rows_of(e);
            return true;
        });
    } else {
        pdl_wait();
        rows_of(gb_expert(p, t, slot));
        gb_dot<2, false>(acc, row, p.x + size_t(t) * p.x_ld, p.K);
    }
    const float g = warp_sum(acc[0]), u = warp_sum(acc[1]);
    if (i < p.rows && (threadIdx.x & 31u) == 0) p.out[(size_t(t) * p.top + slot) * p.out_ld + i] = silu_f32(g) * u;
}

// SHARE warps share two rows, each taking every SHARE-th expert of the token, and their sums are added in that order.  One warp for all
// experts had their rows in flight one after the other: four experts of 2048 x 1408 took 17 us where HBM needs 3.5.
template <int SHARE>
__global__ void __launch_bounds__(kGbThreads) gemv_bf16_expert_down_kernel(const ExpertGemvParams p) {
    pdl_launch_dependents();
    __shared__ float s_part[kGbWarps][2];
    const uint32_t t = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, mine = warp % SHARE;
    const uint32_t r = 2u * (blockIdx.x * (kGbWarps / SHARE) + warp / SHARE);
    const __nv_bfloat16* row[2];
    auto rows_of = [&](uint32_t e) {
        const size_t first = size_t(e) * p.rows;
        row[0] = p.gate + (first + min(r, p.rows - 1)) * p.ld;
        row[1] = p.gate + (first + min(r + 1, p.rows - 1)) * p.ld;
    };
    const float* x = p.x + size_t(t) * p.top * p.x_ld;
    float acc[2] = {0.f, 0.f};
    uint32_t s = mine;                                       // (SHARE <= top)
    if (p.log_places != 0) {
        const uint32_t guess = gb_expert_guess(p, s);
        rows_of(guess);
        gb_dot<2, true>(acc, row, x + size_t(s) * p.x_ld, p.K, [&]() {
            const uint32_t e = gb_expert(p, 0, s);
            if (e == guess) return false;
            rows_of(e);
            return true;
        });
        s += SHARE;
    } else {
        pdl_wait();
    }
    for (; s < p.top; s += SHARE) {
        rows_of(gb_expert(p, t, s));
        gb_dot<2, false>(acc, row, x + size_t(s) * p.x_ld, p.K);
    }
    float a0 = warp_sum(acc[0]), a1 = warp_sum(acc[1]);
    if constexpr (SHARE > 1) {
        if (lane == 0) { s_part[warp][0] = a0; s_part[warp][1] = a1; }
        __syncthreads();
        if (mine != 0) return;
        a0 = a1 = 0.f;
#pragma unroll
        for (int k = 0; k < SHARE; ++k) { a0 += s_part[warp + k][0]; a1 += s_part[warp + k][1]; }
    }
    if (lane < 2 && r + lane < p.rows) p.out[size_t(t) * p.out_ld + r + lane] = (lane ? a1 : a0) / float(p.top);
}

static bool gb_aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace lv

using namespace lv;

extern "C" int lv_gemv_bf16(lv_ctx* ctx, float* out, uint32_t out_ld, const void* w, uint32_t rows, uint32_t ld, uint32_t cols, const float* x,
                            uint32_t x_ld, uint32_t batch, float factor, int act) {
    LV_ENTER(ctx);
    LV_REQUIRE(out && w && rows && x && cols && batch && batch <= 65535 && out_ld >= rows, "bad gemv_bf16 arguments");
    LV_REQUIRE(ld % 8 == 0 && ld >= cols && x_ld >= cols && (batch == 1 || x_ld % 4 == 0) && gb_aligned(x) && gb_aligned(w), "gemv_bf16: bad strides");
    LV_REQUIRE(act == LV_ACT_NONE || act == LV_ACT_RELU2, "gemv_bf16: unknown activation");
    GemvBf16Params p{};
    p.w[0] = static_cast<const __nv_bfloat16*>(w);
    p.rows = rows;
    p.ld = ld; p.K = cols; p.x = x; p.x_ld = x_ld; p.out = out; p.out_ld = out_ld; p.factor = factor; p.act = act;
    // three or more CTAs per SM, at least 512 columns per warp
    uint32_t split = 1;
    while (split < 8 && uint64_t(rows) * batch * split < uint64_t(48) * uint32_t(ctx->sm_count) && cols >= 512 * 2 * split) split *= 2;
    const uint32_t per_cta = 2 * kGbWarps / split;
    auto* kernel = split == 1 ? gemv_bf16_kernel<1> : split == 2 ? gemv_bf16_kernel<2> : split == 4 ? gemv_bf16_kernel<4> : gemv_bf16_kernel<8>;
    LV_CUDA(launch_pdl(ctx, kernel, dim3((rows + per_cta - 1) / per_cta, batch), dim3(kGbThreads), 0, p));
    return LV_OK;
}

extern "C" int lv_gemv_bf16_mingru(lv_ctx* ctx, float* out, const void* wz, const void* wx, const void* wg, uint32_t ld, uint32_t channels, uint32_t cols,
                                   const float* bz, const float* bx, const float* x, float* state, const uint32_t* pos) {
    LV_ENTER(ctx);
    LV_REQUIRE(out && wz && wx && wg && bz && bx && x && state && pos && channels && cols, "bad mingru arguments");
    LV_REQUIRE(ld % 8 == 0 && ld >= cols && gb_aligned(x) && gb_aligned(wz) && gb_aligned(wx) && gb_aligned(wg), "mingru: bad strides");
    GemvBf16Params p{};
    p.w[0] = static_cast<const __nv_bfloat16*>(wz);
    p.w[1] = static_cast<const __nv_bfloat16*>(wx);
    p.w[2] = static_cast<const __nv_bfloat16*>(wg);
    p.rows = channels;
    p.ld = ld; p.K = cols; p.x = x; p.out = out;
    LV_CUDA(launch_pdl(ctx, gemv_bf16_mingru_kernel, dim3((channels + kGbWarps - 1) / kGbWarps), dim3(kGbThreads), 0, p, bz, bx, state, pos));
    return LV_OK;
}

static int expert_params(const lv_expert_args* a, ExpertGemvParams* p, uint32_t batch) {
    LV_REQUIRE(a && a->table && a->token_log && a->pos && a->experts && a->top && a->vocab && a->rows && a->cols, "bad expert arguments");
    LV_REQUIRE(a->ld % 8 == 0 && a->ld >= a->cols && a->w0 && gb_aligned(a->w0) && (!a->w1 || gb_aligned(a->w1)), "experts: bad matrices");
    p->gate = static_cast<const __nv_bfloat16*>(a->w0);
    p->up = static_cast<const __nv_bfloat16*>(a->w1);
    p->ld = a->ld; p->K = a->cols; p->rows = a->rows; p->experts = a->experts; p->top = a->top; p->vocab = a->vocab;
    p->table = a->table; p->token_log = a->token_log; p->pos = a->pos;
    p->log_places = batch == 1 ? a->log_places : 0;
    return LV_OK;
}

extern "C" int lv_gemv_bf16_expert_gate_up(lv_ctx* ctx, float* out, uint32_t out_ld, const lv_expert_args* a, const float* x, uint32_t x_ld, uint32_t batch) {
    LV_ENTER(ctx);
    ExpertGemvParams p{};
    if (const int rc = expert_params(a, &p, batch)) return rc;
    LV_REQUIRE(out && x && gb_aligned(x) && batch && batch <= 65535 && a->top <= 65535 && p.up && out_ld >= p.rows && x_ld >= p.K && (batch == 1 || x_ld % 4 == 0), "bad expert_gate_up arguments");
    p.x = x; p.x_ld = x_ld; p.out = out; p.out_ld = out_ld; p.err = ctx->d_err;
    LV_CUDA(launch_pdl(ctx, gemv_bf16_expert_gate_up_kernel, dim3((p.rows + kGbWarps - 1) / kGbWarps, batch, p.top), dim3(kGbThreads), 0, p));
    return LV_OK;
}

extern "C" int lv_gemv_bf16_expert_down(lv_ctx* ctx, float* out, uint32_t out_ld, const lv_expert_args* a, const float* x, uint32_t x_ld, uint32_t batch) {
    LV_ENTER(ctx);
    ExpertGemvParams p{};
    if (const int rc = expert_params(a, &p, batch)) return rc;
    LV_REQUIRE(out && x && gb_aligned(x) && batch && batch <= 65535 && out_ld >= p.rows && x_ld >= p.K && x_ld % 4 == 0, "bad expert_down arguments");
    p.x = x; p.x_ld = x_ld; p.out = out; p.out_ld = out_ld; p.err = ctx->d_err;
    // warps per pair of rows: as many as there are experts, a power of two up to four
    const uint32_t share = p.top >= 4 ? 4 : p.top >= 2 ? 2 : 1, per_cta = 2 * kGbWarps / share;
    auto* kernel = share == 4 ? gemv_bf16_expert_down_kernel<4> : share == 2 ? gemv_bf16_expert_down_kernel<2> : gemv_bf16_expert_down_kernel<1>;
    LV_CUDA(launch_pdl(ctx, kernel, dim3((p.rows + per_cta - 1) / per_cta, batch), dim3(kGbThreads), 0, p));
    return LV_OK;
}
