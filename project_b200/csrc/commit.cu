// Column commitment as the reference performs it (trapdoor KZG): the tau-evaluation
// of every column by packed evaluation against w(tau), then one fixed-base
// multiplication [p_k(tau)] G per column; and the honest-prover alternative, a
// Lagrange-basis SRS [L_i(tau)] G against which a column is committed by an MSM
// (same group element, because sum_i f_i [L_i(tau)] G = [sum_i f_i L_i(tau)] G).
#include <cstring>

#include "common.cuh"

namespace gzk
{
    int eval_batch_enqueue(gzk_ctx* ctx, gzk_buf* const* cols, size_t k_count, size_t len, unsigned log2n, const gzk_buf* weights, Fr* dest);
    int eval_status_error(gzk_ctx* ctx, int status);
    int g1_same_base_enqueue(gzk_ctx* ctx, const uint8_t base[96], const Fr* scalars, int kind, size_t count, uint8_t* out_pinned);
}

using namespace gzk;

extern "C"
{
    int gzk_commit_batch(gzk_ctx* ctx, gzk_buf* const* cols, size_t k_count, size_t len, unsigned log2n, const gzk_buf* weights_tau,
                         const uint8_t base[96], uint8_t* tau_evals_out, uint8_t* points_out)
    {
        if (ctx == nullptr) return GZK_E_INVALID;
        if (k_count == 0) return GZK_OK;
        if (tau_evals_out == nullptr || points_out == nullptr || base == nullptr) return fail(ctx, GZK_E_INVALID, "commit_batch: null argument");
        // one wait for both steps: the evaluations stay on the device between them
        void* d_evals = nullptr;
        void* h_out = nullptr;
        int rc = ensure_scratch(ctx, 3, k_count * sizeof(Fr), &d_evals);
        if (rc != GZK_OK) return rc;
        if ((rc = eval_batch_enqueue(ctx, cols, k_count, len, log2n, weights_tau, static_cast<Fr*>(d_evals))) != GZK_OK) return rc;
        if ((rc = ensure_pinned(ctx, k_count * (96 + sizeof(Fr)) + 64, &h_out)) != GZK_OK) return rc;
        if ((rc = g1_same_base_enqueue(ctx, base, static_cast<const Fr*>(d_evals), GZK_KIND_FR, k_count, static_cast<uint8_t*>(h_out))) != GZK_OK) return rc;
        uint8_t* h_evals = static_cast<uint8_t*>(h_out) + k_count * 96;
        GZK_CUDA_TRY(ctx, cudaMemcpyAsync(h_evals, d_evals, k_count * sizeof(Fr), cudaMemcpyDeviceToHost, ctx->stream));
        GZK_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_status, ctx->d_status, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
        GZK_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        if ((rc = eval_status_error(ctx, *ctx->h_status)) != GZK_OK) return rc;
        std::memcpy(points_out, h_out, k_count * 96);
        std::memcpy(tau_evals_out, h_evals, k_count * sizeof(Fr));
        return GZK_OK;
    }

    int gzk_srs_lagrange(gzk_ctx* ctx, unsigned log2n, const uint8_t base[96], const uint8_t tau[32], gzk_buf* out_points)
    {
        if (ctx == nullptr) return GZK_E_INVALID;
        if (log2n > 28) return fail(ctx, GZK_E_INVALID, "srs_lagrange: domain too large");
        const size_t n = static_cast<size_t>(1) << log2n;
        if (out_points == nullptr || out_points->kind != GZK_KIND_G1 || out_points->count < n)
            return fail(ctx, GZK_E_INVALID, "srs_lagrange: output must be a G1 buffer of the domain size");
        gzk_buf* weights = nullptr;
        int rc = gzk_buf_alloc(ctx, GZK_KIND_FR_MONT, n, &weights);
        if (rc != GZK_OK) return rc;
        rc = gzk_bary_weights(ctx, log2n, tau, weights);
        if (rc == GZK_OK) rc = gzk_g1_fixed_base_mul(ctx, base, weights, n, out_points);
        const std::string message = ctx->last_error;
        gzk_buf_free(ctx, weights);
        if (rc != GZK_OK) ctx->last_error = message;
        return rc;
    }
}
