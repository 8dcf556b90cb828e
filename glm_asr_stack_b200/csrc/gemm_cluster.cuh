// bf16 GEMM for up to a few hundred rows, K cut over a thread-block cluster (gemm_cluster.cu).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace glmasr {

static constexpr int kClusterMaxRows = 512;

struct alignas(64) ClusterGemmParams {
    CUtensorMap tm_x;                   // tokens [M, K] bf16, boxes of n_tok rows x 64 elements, 128B swizzle
    CUtensorMap tm_w[3];                // weights [N_s, K] bf16, boxes of 128 rows (64 for EPI_SILU_GATE) x 64 elements
    int seg_rows[3], seg_tiles[3];      // N_s, ceil(N_s / 128)
    int num_segs;
    int M, k_blocks;                    // K / 64
    int epi;                            // EPI_STORE (+ bias), EPI_SILU_GATE, EPI_RESIDUAL (+ bias), EPI_GELU
    __nv_bfloat16 *out;
    const __nv_bfloat16 *residual, *bias;
    int ldo;
    int early_weights;                  // 1: nothing still running writes the weights, load them before the dependency wait
    int late_trigger;                   // 1: signal the dependents after the dependency wait
    int *status;
    // filled by choose_cluster_gemm
    int n_tok, token_tiles, splits, stages, w_tiles;
};

// Tile shape for `w_tiles` 128-row weight tiles, M tokens and K = 64 * k_blocks.  Returns the time expected of it in ns, 0 when
// the shape is not covered.
double choose_cluster_gemm(ClusterGemmParams &p, int w_tiles, int num_sms);
cudaError_t launch_cluster_gemm(const ClusterGemmParams &p, cudaStream_t st);

}  // namespace glmasr
