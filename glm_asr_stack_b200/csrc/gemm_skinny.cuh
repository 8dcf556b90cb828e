// Few-row FP4 linear (gemm_skinny.cu): out[M, sum N_s] = epilogue(x[M, K] * concat_s(W_s[N_s, K])^T) for M <= 16,
// reading the packed e2m1 weights and their e4m3 scales as stored.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace glmasr {

static constexpr int kSkinnyMaxRows = 16;

struct SkinnyParams {
    const __nv_bfloat16 *x;             // [M, K], row pitch ldx (multiple of 8 elements, 16-byte aligned)
    int ldx, M, K;
    const __nv_bfloat16 *norm_w;        // not NULL: x is RMS-normalised with this weight first (eps below)
    float eps;
    const uint8_t *w[3];                // packed e2m1 [N_s, K/2]
    const uint8_t *ws[3];               // e4m3 [N_s, K/16]
    float alpha[3];                     // per-tensor factor of segment s
    int seg_rows[3];                    // N_s, multiples of 16
    int num_segs;
    int epi;                            // EPI_STORE (+ bias), EPI_RESIDUAL, EPI_SILU_GATE (segments 0 / 1 = gate / up)
    __nv_bfloat16 *out;
    const __nv_bfloat16 *residual;      // row pitch ldo; may be out
    const __nv_bfloat16 *bias;
    int ldo;
    int early_weights;                  // 1: nothing still running writes the weights, load them before the dependency wait
    int late_trigger;                   // 1: signal the dependents after the dependency wait
    int *status;
    // filled by the launcher
    int units, units_per_cta, units_per_group, groups, pass_tiles;
};

// cudaErrorInvalidValue when the shape is not covered (nothing launched).
bool skinny_covers(int M, int K, const int *seg_rows, int num_segs, int epi);
// Whether the kernel is the faster route for a shape that it covers (the other one: bf16 copies of the weights).
bool skinny_pays(int M, int K, const int *seg_rows, int num_segs, int epi, int num_sms);
// *rounds: rounds in which a CTA reads its weights.
cudaError_t launch_skinny_linear(SkinnyParams p, int num_sms, cudaStream_t st, int *rounds);

}  // namespace glmasr
