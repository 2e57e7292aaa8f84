// Prefill palettized GEMM: Y[t][:] = lut_gemv(X[t][:]) for every activation row
// (prefill_cpu, src/lut/engine_impl.rs:1046-1053; kernel counterpart
// templates/palettized_gemm.metal:16-117).
#include "common.cuh"

namespace prism {

// X, or a copy of it in scratch where Y's rows lie over X's: the kernels read X while they store Y.
static int gemm_input(prism_cuda_ctx *ctx, const LutTensor &t, const uint16_t **X, uint32_t m_tok, const uint16_t *Y) {
    const size_t xn = (size_t)m_tok * t.k, yn = (size_t)m_tok * t.m;
    if (*X >= Y + yn || Y >= *X + xn) return PRISM_OK;
    if (reinterpret_cast<uintptr_t>(*X) & 15) return fail(ctx, PRISM_E_ARG, "gemm: X must be 16-byte aligned");
    PRISM_TRY(ensure_tmp(ctx, xn));
    PRISM_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->tmp_scratch, *X, xn * 2, cudaMemcpyDeviceToDevice, ctx->stream));
    *X = ctx->tmp_scratch;
    return PRISM_OK;
}

int launch_gemm(prism_cuda_ctx *ctx, const LutTensor &t, const uint16_t *X, uint32_t m_tok, uint16_t *Y) {
    if (t.k % 8) return fail(ctx, PRISM_E_ARG, "gemm: dim_n must be a multiple of 8");
    PRISM_TRY(gemm_input(ctx, t, &X, m_tok, Y));
    bool few = false;
    if (m_tok >= 2) PRISM_TRY(gemm_few_tokens(ctx, GEMV_PLAIN, t, nullptr, X, t.k, Y, t.m, nullptr, m_tok, -1.0f, &few));
    if (few) return PRISM_OK;
    if (ctx->gemm_variant == 1 && gemm_tc5_eligible(ctx, t, m_tok)) return launch_gemm_tc5(ctx, t, X, m_tok, Y, nullptr);
    // activation rows as the batch dimension of the GEMV kernel, 32768 rows per launch
    for (uint32_t t0 = 0; t0 < m_tok; t0 += 32768) {
        const uint32_t nb = m_tok - t0 < 32768 ? m_tok - t0 : 32768;
        PRISM_TRY(launch_gemv(ctx, GEMV_PLAIN, t, nullptr, X + (size_t)t0 * t.k, t.k, Y + (size_t)t0 * t.m, t.m,
                              nullptr, nb));
    }
    return PRISM_OK;
}

int launch_gemm_add(prism_cuda_ctx *ctx, const LutTensor &t, const uint16_t *X, uint32_t m_tok, uint16_t *h, uint16_t *tmp) {
    bool few = false;
    if (m_tok >= 2) PRISM_TRY(gemm_few_tokens(ctx, GEMV_RESID, t, nullptr, X, t.k, h, t.m, h, m_tok, -1.0f, &few));
    if (few) return PRISM_OK;
    if (ctx->gemm_variant == 1 && gemm_tc5_eligible(ctx, t, m_tok) && gemm_tc5_wide(t, h)) return launch_gemm_tc5(ctx, t, X, m_tok, h, h);
    PRISM_TRY(launch_gemm(ctx, t, X, m_tok, tmp));
    return launch_vec_add(ctx, h, tmp, m_tok * t.m);
}

int gemm_swiglu_fused(prism_cuda_ctx *ctx, const LutTensor &tg, const LutTensor &tu, uint32_t m_tok, const uint16_t *act, bool *fused) {
    *fused = false;
    if (ctx->gemm_variant != 1 || !gemm_tc5_eligible(ctx, tg, m_tok) || !gemm_tc5_eligible(ctx, tu, m_tok) || tg.bits != tu.bits || !gemm_tc5_wide(tg, act)) return PRISM_OK;
    return swiglu_tc5_pays(ctx, tg, m_tok, fused);
}
int launch_gemm_swiglu(prism_cuda_ctx *ctx, const LutTensor &tg, const LutTensor &tu, const uint16_t *X, uint32_t m_tok, uint16_t *act, uint16_t *u) {
    bool few = false, fused = false;
    if (m_tok >= 2 && tg.bits == tu.bits && tg.k == tu.k && tg.m == tu.m)
        PRISM_TRY(gemm_few_tokens(ctx, GEMV_SWIGLU, tg, &tu, X, tg.k, act, tg.m, nullptr, m_tok, -1.0f, &few));
    if (few) return PRISM_OK;
    PRISM_TRY(gemm_swiglu_fused(ctx, tg, tu, m_tok, act, &fused));
    if (fused) return launch_swiglu_tc5(ctx, tg, tu, X, m_tok, act);
    PRISM_TRY(launch_gemm(ctx, tg, X, m_tok, act));
    PRISM_TRY(launch_gemm(ctx, tu, X, m_tok, u));
    return launch_silu_mul(ctx, act, act, u, m_tok * tg.m);
}

}  // namespace prism
