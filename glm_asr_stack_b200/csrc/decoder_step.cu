// Batched single-token decode step of the 28-layer decoder behind the engine's own entry point
// (reference: decoder_decode_step_batched, Infer-engine/cuda/decoder.cu:1849-2173), plus the
// reference-named glue entry points it is built from.
//
// Same inputs, outputs and side effects as the reference driver: gathers query_ptrs[i] rows,
// runs every layer (RMSNorm eps 1e-5, q|k|v, rotate-half RoPE at position = cached length, KV
// write to the paged pool, paged GQA attention over cached+1 tokens, o + residual, RMSNorm,
// gate|up + SiLU-gate, down + residual), final RMSNorm, writes the rows back to query_ptrs[i],
// bumps h_seq_lens / d_seq_lens.  Differences in HOW:
//   * tensor names are resolved once per WeightStore into a per-layer pointer table (the reference
//     does ~37 linear string scans per layer per step);
//   * q|k|v and gate|up are single fused GEMMs with SiLU-gate / residual in the epilogue, RoPE,
//     cache write and attention read q/k/v in place from the fused output;
//   * the per-sequence block-table rows are gathered by one kernel (the reference issues one
//     cudaMemcpy per sequence);
//   * no per-layer residual copies: the norm writes to a second buffer.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <vector>

#include "../../include/glmasr_engine_types.h"
#include "../../include/glmasr_fp4.h"
#include "decode_tail.cuh"
#include "decoder_ops.cuh"
#include "runtime.cuh"
#include "step_pages.h"

namespace glmasr {
int fp4_linear_w4a4_prequantized(uint16_t *out, int ldo, const uint8_t *xq, const uint8_t *xq_sf,
                                 const glmasr_fp4_weight *weights, int num_weights, float input_scale, int epilogue,
                                 const uint16_t *residual, int M, int K, uint8_t *q_out = nullptr,
                                 uint8_t *q_out_sf = nullptr, float q_out_input_scale = 0.0f);   // api.cu
int fp4_linear_w4a16_normed(uint16_t *out, int ldo, const uint16_t *x, const uint16_t *norm_w, float eps,
                            const glmasr_fp4_weight *weights, int num_weights, int epilogue, int M, int K);   // api.cu
int fp4_linear_w4a16_silu_quantized(uint8_t *q_out, uint8_t *q_out_sf, float q_out_input_scale, const uint16_t *x, int ldx,
                                    const glmasr_fp4_weight *gate_up, int M, int K);             // api.cu

struct ProjRef {
    int dtype = -1;                     // GLMASR_DTYPE_UINT8 (FP4) or GLMASR_DTYPE_BF16
    const void *w = nullptr;
    const uint8_t *scales = nullptr;
    float global_scale = 1.0f;
    float input_scale = 1.0f;
    const uint16_t *pre = nullptr;
    int N = 0, K = 0;
};

struct LayerRef {
    const uint16_t *norm1 = nullptr, *norm2 = nullptr;
    ProjRef q, k, v, o, gate, up, down;
};

struct ModelRefs {
    const glmasr_WeightStore *ws = nullptr;
    int count = -1;
    uint64_t fingerprint = 0;
    std::vector<LayerRef> layers;
    const uint16_t *final_norm = nullptr;
};

static ModelRefs g_refs;
// cached environment switches (-1 = not read yet), see prefer_w4a4() / pairs_w4a4()
static int g_native_switch = -1, g_pairs_switch = -1;

static const glmasr_Tensor *find_tensor(const glmasr_WeightStore *ws, const char *name) {
    for (int i = 0; i < ws->count; ++i)
        if (ws->names[i] != nullptr && strcmp(ws->names[i], name) == 0) return &ws->tensors[i];
    return nullptr;
}

static const glmasr_Tensor *require_tensor(const glmasr_WeightStore *ws, const char *name) {
    const glmasr_Tensor *t = find_tensor(ws, name);
    if (t == nullptr) {   // reference: wget(), Infer-engine/cuda/decoder.cu:849-854
        fprintf(stderr, "Weight not found: %s\n", name);
        exit(1);
    }
    return t;
}

static float read_scalar(const glmasr_Tensor *t, float fallback) {
    // reference: decoder_scalar_read_cached (Infer-engine/cuda/decoder.cu:165-187); read once here
    if (t == nullptr || t->data == nullptr) return fallback;
    float v = fallback;
    GLMASR_CUDA_CHECK(cudaMemcpy(&v, t->data, sizeof(float), cudaMemcpyDeviceToHost));
    return v;
}

static ProjRef resolve_proj(const glmasr_WeightStore *ws, int layer, const char *block, const char *proj) {
    char name[256];
    ProjRef r;
    snprintf(name, sizeof(name), "language_model.model.layers.%d.%s.%s.weight", layer, block, proj);
    const glmasr_Tensor *tw = require_tensor(ws, name);
    r.dtype = tw->dtype;
    r.w = tw->data;
    r.N = (int)tw->shape[0];
    r.K = tw->dtype == GLMASR_DTYPE_UINT8 ? (int)tw->shape[1] * 2 : (int)tw->shape[1];
    GLMASR_CHECK(tw->dtype == GLMASR_DTYPE_UINT8 || tw->dtype == GLMASR_DTYPE_BF16,
                 "Unsupported decoder weight dtype %d for %s", tw->dtype, name);
    snprintf(name, sizeof(name), "language_model.model.layers.%d.%s.%s.weight_scale", layer, block, proj);
    const glmasr_Tensor *ts = find_tensor(ws, name);
    r.scales = ts ? (const uint8_t *)ts->data : nullptr;
    snprintf(name, sizeof(name), "language_model.model.layers.%d.%s.%s.weight_scale_2", layer, block, proj);
    r.global_scale = read_scalar(find_tensor(ws, name), 1.0f);
    snprintf(name, sizeof(name), "language_model.model.layers.%d.%s.%s.input_scale", layer, block, proj);
    r.input_scale = read_scalar(find_tensor(ws, name), 1.0f);
    snprintf(name, sizeof(name), "language_model.model.layers.%d.%s.%s.pre_quant_scale", layer, block, proj);
    const glmasr_Tensor *tp = find_tensor(ws, name);
    r.pre = tp ? (const uint16_t *)tp->data : nullptr;
    return r;
}

// The table is cached per weight store.  The store's address alone is not an identity (a freed store's
// address is reused by the next one), so the key also folds in every tensor's data pointer and size:
// ~300 loads per call, nothing against a step's 200 launches.
static uint64_t store_fingerprint(const glmasr_WeightStore *ws) {
    uint64_t h = 1469598103934665603ull;
    for (int i = 0; i < ws->count; ++i) {
        h = (h ^ (uint64_t)(uintptr_t)ws->tensors[i].data) * 1099511628211ull;
        h = (h ^ (uint64_t)ws->tensors[i].nbytes) * 1099511628211ull;
    }
    return h;
}

static const ModelRefs &model_refs(const glmasr_WeightStore *ws, int num_layers) {
    const uint64_t fp = store_fingerprint(ws);
    if (g_refs.ws == ws && g_refs.count == ws->count && g_refs.fingerprint == fp && (int)g_refs.layers.size() == num_layers)
        return g_refs;
    g_refs = ModelRefs();
    g_refs.ws = ws;
    g_refs.count = ws->count;
    g_refs.fingerprint = fp;
    g_refs.layers.resize(num_layers);
    char name[256];
    for (int l = 0; l < num_layers; ++l) {
        LayerRef &L = g_refs.layers[l];
        snprintf(name, sizeof(name), "language_model.model.layers.%d.input_layernorm.weight", l);
        L.norm1 = (const uint16_t *)require_tensor(ws, name)->data;
        snprintf(name, sizeof(name), "language_model.model.layers.%d.post_attention_layernorm.weight", l);
        L.norm2 = (const uint16_t *)require_tensor(ws, name)->data;
        L.q = resolve_proj(ws, l, "self_attn", "q_proj");
        L.k = resolve_proj(ws, l, "self_attn", "k_proj");
        L.v = resolve_proj(ws, l, "self_attn", "v_proj");
        L.o = resolve_proj(ws, l, "self_attn", "o_proj");
        L.gate = resolve_proj(ws, l, "mlp", "gate_proj");
        L.up = resolve_proj(ws, l, "mlp", "up_proj");
        L.down = resolve_proj(ws, l, "mlp", "down_proj");
    }
    g_refs.final_norm = (const uint16_t *)require_tensor(ws, "language_model.model.norm.weight")->data;
    return g_refs;
}

void forget_model_refs() {
    g_refs = ModelRefs();
    g_native_switch = g_pairs_switch = -1;
}

// The two arithmetic switches are read from the environment on first use and kept (the reference reads its
// switch once per process); glmasr_decoder_forget_weights() drops them together with the pointer table, so a
// host that changes the environment between two models gets the new values.
static bool prefer_w4a4() {
    // reference: prefer_nvfp4_cutlass, Infer-engine/cuda/decoder.cu:142-151
    if (g_native_switch < 0) {
        const char *e = getenv("GLMASR_USE_CUTLASS_NVFP4");
        g_native_switch = (e && e[0] && strcmp(e, "0") != 0) ? 1 : 0;
    }
    return g_native_switch == 1;
}

// Which arithmetic the same-input PAIRS (k|v, gate|up) use when GLMASR_USE_CUTLASS_NVFP4 selects the native
// path.  The reference never runs a fused pair natively: linear_proj_pair_same_input
// (Infer-engine/cuda/decoder.cu:923-978) always dequantises both weights and runs a bf16 GEMM, so with the
// switch on its q, o and down projections are W4A4 and its k|v and gate|up are W4A16 (pairs that carry a
// pre_quant_scale are not fused and go through nvfp4_linear one by one, :957-963).  That mix is the default
// here.  GLMASR_NVFP4_PAIRS=1 opts in to running the pairs in W4A4 as well (q|k|v and gate|up each one
// block-scaled FP4 GEMM on a shared quantised input): faster, but not the reference's arithmetic.
static bool pairs_w4a4() {
    if (g_pairs_switch < 0) {
        const char *e = getenv("GLMASR_NVFP4_PAIRS");
        g_pairs_switch = (e && e[0] && strcmp(e, "0") != 0) ? 1 : 0;
    }
    return g_pairs_switch == 1 && prefer_w4a4();
}

static glmasr_fp4_weight as_weight(const ProjRef &p) {
    glmasr_fp4_weight w;
    w.w_packed = (const uint8_t *)p.w;
    w.w_scales = p.scales;
    w.w_global_scale = p.global_scale;
    w.N = p.N;
    return w;
}

// One projection on its own: the reference's linear_proj (Infer-engine/cuda/decoder.cu:861-921)
// with an optional fused residual.
static void single_proj(uint16_t *out, int ldo, const uint16_t *x, int ldx, const ProjRef &p, int M,
                        const uint16_t *residual, uint16_t *scratch) {
    if (p.dtype == GLMASR_DTYPE_BF16) {
        // bf16_linear keeps the reference's dense signature: go through the scratch buffer when the
        // destination is a column slice of a wider buffer, or when it is also the residual (the drivers
        // update the hidden state in place, and the GEMM must not overwrite what is still to be added)
        GLMASR_CHECK(ldx == p.K, "bf16 projection needs a dense input");
        uint16_t *dst = (ldo == p.N && out != residual) ? out : scratch;
        bf16_linear(nullptr, dst, x, (const uint16_t *)p.w, nullptr, M, p.N, p.K);
        if (residual) {
            GLMASR_CHECK(ldo == p.N, "bf16 projection with residual needs a dense output");
            residual_add(out, dst, residual, M * p.N);
        } else if (dst != out) {
            GLMASR_CUDA_CHECK(cudaMemcpy2DAsync(out, (size_t)ldo * 2, dst, (size_t)p.N * 2, (size_t)p.N * 2, M,
                                                cudaMemcpyDeviceToDevice, current_stream()));
        }
        return;
    }
    const glmasr_fp4_weight w = as_weight(p);
    const int epi = residual ? GLMASR_EPI_RESIDUAL : GLMASR_EPI_STORE;
    int rc = -1;
    if (prefer_w4a4() && p.scales != nullptr && p.input_scale > 0.0f)
        rc = glmasr_fp4_linear_fused(GLMASR_MODE_W4A4, out, ldo, x, ldx, &w, 1, p.input_scale, p.pre, nullptr, epi,
                                     residual, M, p.K);
    if (rc != 0)
        rc = glmasr_fp4_linear_fused(GLMASR_MODE_W4A16, out, ldo, x, ldx, &w, 1, 1.0f, p.pre, scratch, epi, residual, M,
                                     p.K);
    GLMASR_CHECK(rc == 0, "decoder projection failed (N=%d K=%d M=%d)", p.N, p.K, M);
}

// Several same-input FP4 projections as one GEMM when the reference's own fusion rule allows it
// (all FP4, none with a pre_quant_scale: Infer-engine/cuda/decoder.cu:957-963): W4A16 like the reference's
// fused pair, or W4A4 when the pairs were opted in to the native path and share their input_scale.
// Returns false when the caller has to run them one by one.
static bool fusable(const ProjRef *const *ps, int n) {
    for (int i = 0; i < n; ++i)
        if (ps[i]->dtype != GLMASR_DTYPE_UINT8 || ps[i]->pre != nullptr || ps[i]->K != ps[0]->K) return false;
    return true;
}

static bool fused_proj(uint16_t *out, int ldo, const uint16_t *x, int ldx, const ProjRef *const *ps, int n, int epi,
                       int M) {
    if (!fusable(ps, n)) return false;
    glmasr_fp4_weight w[3];
    for (int i = 0; i < n; ++i) w[i] = as_weight(*ps[i]);
    bool w4a4 = pairs_w4a4();
    for (int i = 0; i < n && w4a4; ++i)
        if (ps[i]->scales == nullptr || !(ps[i]->input_scale > 0.0f) || ps[i]->input_scale != ps[0]->input_scale) w4a4 = false;
    const int rc = glmasr_fp4_linear_fused(w4a4 ? GLMASR_MODE_W4A4 : GLMASR_MODE_W4A16, out, ldo, x, ldx, w, n,
                                           w4a4 ? ps[0]->input_scale : 1.0f, nullptr, nullptr, epi, nullptr, M, ps[0]->K);
    return rc == 0;
}

// RMSNorm feeding several same-input FP4 projections in W4A4: the norm kernel quantises its own
// result (same bytes as norm, then the stand-alone quantiser) and the GEMM takes it as it is.
// Returns false when the projections cannot share one quantised input; the caller then runs the
// norm and the projections separately.
static bool norm_then_fused_proj_w4a4(uint16_t *out, int ldo, const uint16_t *x, const uint16_t *norm_w, float eps,
                                      const ProjRef *const *ps, int n, int epi, int M, int H, uint8_t *xq, uint8_t *xsf,
                                      cudaStream_t st, uint8_t *q_out = nullptr, uint8_t *q_out_sf = nullptr,
                                      float q_out_scale = 0.0f) {
    if (!pairs_w4a4() || (H % 256) != 0) return false;
    glmasr_fp4_weight w[3];
    for (int i = 0; i < n; ++i) {
        const ProjRef &p = *ps[i];
        if (p.dtype != GLMASR_DTYPE_UINT8 || p.pre != nullptr || p.K != H || p.scales == nullptr ||
            !(p.input_scale > 0.0f) || p.input_scale != ps[0]->input_scale)
            return false;
        w[i] = as_weight(p);
    }
    if (!launch_rmsnorm_quant(xq, xsf, (const __nv_bfloat16 *)x, (const __nv_bfloat16 *)norm_w, eps, ps[0]->input_scale,
                              M, H, st))
        return false;
    note_launches(1);
    const int rc = fp4_linear_w4a4_prequantized(out, ldo, xq, xsf, w, n, ps[0]->input_scale, epi, nullptr, M, H, q_out,
                                                q_out_sf, q_out_scale);
    GLMASR_CHECK(rc == 0, "decoder projection on a quantised norm output failed (M=%d H=%d)", M, H);
    return true;
}

static bool attn_scalar_forced() {
    static int v = -1;
    if (v < 0) {
        const char *e = getenv("GLMASR_ATTN_SCALAR");
        v = (e && e[0] == '1') ? 1 : 0;
    }
    return v == 1;
}

// A projection that can take an activation quantised by its producer kernel (W4A4, plain FP4 weight).
static bool takes_quantised_input(const ProjRef &p) {
    return prefer_w4a4() && p.dtype == GLMASR_DTYPE_UINT8 && p.pre == nullptr && p.scales != nullptr && p.input_scale > 0.0f &&
           (p.K % 256) == 0;
}

static void single_proj_prequantized(uint16_t *out, int ldo, const uint8_t *xq, const uint8_t *xsf, const ProjRef &p, int M,
                                     const uint16_t *residual) {
    const glmasr_fp4_weight w = as_weight(p);
    const int rc = fp4_linear_w4a4_prequantized(out, ldo, xq, xsf, &w, 1, p.input_scale,
                                                residual ? GLMASR_EPI_RESIDUAL : GLMASR_EPI_STORE, residual, M, p.K);
    GLMASR_CHECK(rc == 0, "decoder projection on a quantised input failed (N=%d K=%d M=%d)", p.N, p.K, M);
}

// RMSNorm and same-input W4A16 projections of a few rows as one launch; false when that route does not cover them.
static bool normed_proj_w4a16(uint16_t *out, int ldo, const uint16_t *x, const uint16_t *norm_w, float eps, const ProjRef *const *ps,
                              int n, int epi, int M, int H) {
    if (prefer_w4a4() || !fusable(ps, n) || ps[0]->K != H) return false;
    glmasr_fp4_weight w[3];
    for (int i = 0; i < n; ++i) {
        if (ps[i]->scales == nullptr) return false;
        w[i] = as_weight(*ps[i]);
    }
    return fp4_linear_w4a16_normed(out, ldo, x, norm_w, eps, w, n, epi, M, H) == 0;
}

// Scratch of one driver call (private workspace slots), shared by the per-layer stages below.
struct StepBuffers {
    uint16_t *nrm;       // [M, H] bf16: normed hidden state, for consumers that take bf16
    uint16_t *qkv;       // [M, H + 2 KV]
    uint16_t *act;       // [M, 2 F]: SiLU-gate output (first F columns when fused) or gate | up
    uint16_t *scratch;   // [M, max(H, F)]
    uint8_t *nq, *nsf;   // quantised normed hidden state (K = H)
    uint8_t *aq, *asf;   // quantised attention output (K = H) / SiLU-gate output (K = F)
};

// q | k | v of one layer from the pre-norm hidden state into B.qkv [M, H + 2 KV].  Returns the number of
// glue launches (norms) the caller has to account for.
static int project_qkv(const LayerRef &R, const uint16_t *hid, const StepBuffers &B, int M, int H, int KV, cudaStream_t st) {
    const int NQKV = H + 2 * KV;
    const ProjRef *qkv_p[3] = {&R.q, &R.k, &R.v};
    const ProjRef *kv_p[2] = {&R.k, &R.v};
    // (1) pairs opted in to W4A4: norm + quantiser in one launch, one q|k|v GEMM on the quantised rows
    if (norm_then_fused_proj_w4a4(B.qkv, NQKV, hid, R.norm1, 1e-5f, qkv_p, 3, GLMASR_EPI_STORE, M, H, B.nq, B.nsf, st)) return 0;
    // (2) the reference's mix: q through the native path, k|v as one W4A16 GEMM
    //     (Infer-engine/cuda/decoder.cu:1995-2035); the norm writes its result in both forms
    if (prefer_w4a4() && takes_quantised_input(R.q) && R.q.K == H && fusable(kv_p, 2) && R.k.K == H &&
        launch_rmsnorm_quant(B.nq, B.nsf, (const __nv_bfloat16 *)hid, (const __nv_bfloat16 *)R.norm1, 1e-5f, R.q.input_scale, M, H,
                             st, (__nv_bfloat16 *)B.nrm)) {
        single_proj_prequantized(B.qkv, NQKV, B.nq, B.nsf, R.q, M, nullptr);
        const bool ok = fused_proj(B.qkv + H, NQKV, B.nrm, H, kv_p, 2, GLMASR_EPI_STORE, M);
        GLMASR_CHECK(ok, "decoder k|v projection failed (M=%d H=%d)", M, H);
        return 1;
    }
    // (3) W4A16 throughout, few rows: norm and projection in one launch
    if (normed_proj_w4a16(B.qkv, NQKV, hid, R.norm1, 1e-5f, qkv_p, 3, GLMASR_EPI_STORE, M, H)) return 0;
    // (4) everything else: bf16 norm, then whatever can be fused
    launch_rmsnorm((__nv_bfloat16 *)B.nrm, (const __nv_bfloat16 *)hid, (const __nv_bfloat16 *)R.norm1, 1e-5f, M, H, st);
    // W4A16 throughout: one q|k|v GEMM gives the values of fp4_linear(q) + the fused k|v pair
    if (!prefer_w4a4() && fused_proj(B.qkv, NQKV, B.nrm, H, qkv_p, 3, GLMASR_EPI_STORE, M)) return 1;
    single_proj(B.qkv, NQKV, B.nrm, H, R.q, M, nullptr, B.scratch);
    if (!fused_proj(B.qkv + H, NQKV, B.nrm, H, kv_p, 2, GLMASR_EPI_STORE, M)) {
        single_proj(B.qkv + H, NQKV, B.nrm, H, R.k, M, nullptr, B.scratch);
        single_proj(B.qkv + H + KV, NQKV, B.nrm, H, R.v, M, nullptr, B.scratch);
    }
    return 1;
}

// post-attention norm -> gate|up -> SiLU-gate -> down + residual, in place on hid [M, H].  Returns the glue
// launches the caller has to account for.
static int project_mlp(const LayerRef &R, uint16_t *hid, const StepBuffers &B, int M, int H, int F, cudaStream_t st) {
    const ProjRef *gu_p[2] = {&R.gate, &R.up};
    // the producer of down's input quantises for it when down runs natively
    const bool down_q = takes_quantised_input(R.down) && R.down.K == F && (F % 64) == 0;
    // (1) pairs opted in to W4A4
    if (down_q && norm_then_fused_proj_w4a4(B.act, F, hid, R.norm2, 1e-5f, gu_p, 2, GLMASR_EPI_SILU_GATE, M, H, B.nq, B.nsf, st,
                                            B.aq, B.asf, R.down.input_scale)) {
        single_proj_prequantized(hid, H, B.aq, B.asf, R.down, M, hid);
        return 0;
    }
    if (norm_then_fused_proj_w4a4(B.act, F, hid, R.norm2, 1e-5f, gu_p, 2, GLMASR_EPI_SILU_GATE, M, H, B.nq, B.nsf, st)) {
        single_proj(hid, H, B.act, F, R.down, M, hid, B.scratch);
        return 0;
    }
    // (2) W4A16 throughout, few rows: norm, gate|up and SiLU-gate in one launch
    if (R.gate.N == F && R.up.N == F && normed_proj_w4a16(B.act, F, hid, R.norm2, 1e-5f, gu_p, 2, GLMASR_EPI_SILU_GATE, M, H)) {
        single_proj(hid, H, B.act, F, R.down, M, hid, B.scratch);
        return 0;
    }
    launch_rmsnorm((__nv_bfloat16 *)B.nrm, (const __nv_bfloat16 *)hid, (const __nv_bfloat16 *)R.norm2, 1e-5f, M, H, st);
    // (3) the reference's mix: gate|up as one W4A16 GEMM (Infer-engine/cuda/decoder.cu:2107-2112) whose SiLU-gate
    //     epilogue writes the native down projection's quantised operand
    if (prefer_w4a4() && !pairs_w4a4() && down_q && fusable(gu_p, 2) && R.gate.K == H && R.gate.N == F && R.up.N == F) {
        const glmasr_fp4_weight gu[2] = {as_weight(R.gate), as_weight(R.up)};
        if (fp4_linear_w4a16_silu_quantized(B.aq, B.asf, R.down.input_scale, B.nrm, H, gu, M, H) == 0) {
            single_proj_prequantized(hid, H, B.aq, B.asf, R.down, M, hid);
            return 1;
        }
    }
    // (4) everything else
    if (!fused_proj(B.act, F, B.nrm, H, gu_p, 2, GLMASR_EPI_SILU_GATE, M)) {
        single_proj(B.act, F, B.nrm, H, R.gate, M, nullptr, B.scratch);
        single_proj(B.act + (size_t)M * F, F, B.nrm, H, R.up, M, nullptr, B.scratch);
        silu_elementwise_mul(B.act, B.act + (size_t)M * F, M * F);
    }
    single_proj(hid, H, B.act, F, R.down, M, hid, B.scratch);
    return 1;
}

// ---- the layer tail as one co-resident kernel (decode_tail.cu) -----------------------------------------------
// Taken when every projection of the step runs in W4A4 (GLMASR_USE_CUTLASS_NVFP4=1 GLMASR_NVFP4_PAIRS=1), the batch
// is at most 256 rows and every shape divides into the kernel's units; GLMASR_DECODE_TAIL=0 keeps the step on one
// launch per operation.
static constexpr int kTailDebugSlot = 51;   // workspace slot of the layer tail's cycle counters (experiment builds)
static bool g_tail_refused = false;     // a launch was refused by the runtime: do not try again in this process
static bool tail_enabled() {
    static int v = -1;
    if (v < 0) {
        const char *e = getenv("GLMASR_DECODE_TAIL");
        v = (e && e[0] == '0') ? 0 : 1;
    }
    return v == 1 && !g_tail_refused && pairs_w4a4();
}

// GLMASR_TAIL_CPM="o,gate_up,down,qkv": CTAs per row tile for the four GEMM phases of the layer tail (0 or
// missing: the library's own choice, tail_choose_cpm).  For measurements.
static int tail_cpm_override(int which) {
    static int v[4] = {-1, 0, 0, 0};
    if (v[0] < 0) {
        v[0] = 0;
        const char *e = getenv("GLMASR_TAIL_CPM");
        if (e != nullptr) sscanf(e, "%d,%d,%d,%d", &v[0], &v[1], &v[2], &v[3]);
    }
    return which >= 0 && which < 4 ? v[which] : 0;
}

static bool tail_fill_gemm(TailGemm &g, const uint8_t *xq, const uint8_t *xsf, int M, int num_m_tiles, int grid,
                           const ProjRef *const *ps, int n, int epi, uint16_t *out, int ldo, uint8_t *q_out, uint8_t *q_out_sf,
                           float q_out_scale, int which = -1) {
    memset(&g, 0, sizeof(g));
    const int K = ps[0]->K;
    if (n < 1 || n > kTailMaxSegs || (K % 256) != 0) return false;
    int units = 0;
    for (int i = 0; i < n; ++i) {
        const ProjRef &p = *ps[i];
        if (p.dtype != GLMASR_DTYPE_UINT8 || p.pre != nullptr || p.scales == nullptr || p.K != K || !(p.input_scale > 0.0f) ||
            p.input_scale != ps[0]->input_scale || (p.N % 32) != 0 || p.N < 32 * kTailMaxRunUnits)
            return false;
        g.seg_units[i] = p.N / 32;
        g.alpha[i] = p.input_scale * p.global_scale;
        units += g.seg_units[i];
        if (!make_u8_tmap_sw128(&g.tm_w[i], p.w, (uint64_t)K / 2, (uint64_t)p.N, (uint64_t)K / 2, 128, 32)) return false;
    }
    if (epi == TAIL_EPI_SILU_QUANT && n == 2) units = g.seg_units[0];
    int cpm = tail_choose_cpm(units, K, epi == TAIL_EPI_SILU_QUANT, grid, num_m_tiles);
    const int forced = tail_cpm_override(which);
    if (forced > 0 && forced <= grid / num_m_tiles && (units + forced - 1) / forced <= kTailMaxRunUnits) cpm = forced;
    if (cpm <= 0) return false;
    g.cpm = cpm;
    for (int i = 0, first = 0; i < n; ++i) {
        const bool silu = epi == TAIL_EPI_SILU_QUANT;
        g.sfb[i] = tail_tiled_scales(ps[i]->scales, ps[i]->N, K, cpm, silu ? g.seg_units[0] : units, silu ? 0 : first, current_stream());
        if (g.sfb[i] == nullptr) return false;
        first += g.seg_units[i];
    }
    if (epi == TAIL_EPI_SILU_QUANT) {
        if (n != 2 || ps[0]->N != ps[1]->N || (ps[0]->N % 64) != 0 || q_out == nullptr || q_out_sf == nullptr || !(q_out_scale > 0.0f))
            return false;
        units = g.seg_units[0];
        g.q_packed = q_out;
        g.q_sf = q_out_sf;
        g.q_inv_in = 1.0f / q_out_scale;
        g.q_ld = ps[0]->N / 2;
        g.q_sf_chunks = ps[0]->N / 64;
    }
    if (!make_u8_tmap_sw128(&g.tm_a, xq, (uint64_t)K / 2, (uint64_t)M, (uint64_t)K / 2, 128, 128)) return false;
    g.sfa = xsf;
    g.num_segs = n;
    g.K = K;
    g.epi = epi;
    g.out = (__nv_bfloat16 *)out;
    g.ldo = ldo;
    return true;
}

// o + residual, norm + quantiser, gate|up + SiLU-gate + quantiser, down + residual of layer R and, when `next`
// is given, that layer's input norm + quantiser and its q|k|v projection, in one launch.  aq / asf: the quantised
// attention output (K = H).  False (nothing launched) when a shape or weight kind is not covered.
static bool launch_layer_tail(const LayerRef &R, const LayerRef *next, uint16_t *hid, const StepBuffers &B, uint8_t *gq,
                              uint8_t *gsf, unsigned int *counter, unsigned int &base, int M, int H, int KV, int F,
                              cudaStream_t st, int max_phases = 0) {
    const int grid = tail_grid_size();
    if (grid <= 0 || M > 256 || (H % 64) != 0 || H > 4096) return false;
    const int num_m_tiles = (M + 127) / 128;
    static TailParams P;       // 3 KB: not on the stack of every call
    P.num_phases = 0;
    auto add = [&](int kind, int index) {
        P.kind[P.num_phases] = kind;
        P.index[P.num_phases] = index;
        ++P.num_phases;
    };
    auto fill_norm = [&](TailNorm &nm, const uint16_t *w, float input_scale) {
        nm.x = (const __nv_bfloat16 *)hid;
        nm.weight = (const __nv_bfloat16 *)w;
        nm.q_packed = B.nq;
        nm.q_sf = B.nsf;
        nm.eps = 1e-5f;
        nm.inv_in = 1.0f / input_scale;
        nm.dim = H;
    };
    const ProjRef *o_p[1] = {&R.o}, *gu_p[2] = {&R.gate, &R.up}, *down_p[1] = {&R.down};
    if (R.o.K != H || R.o.N != H || R.gate.K != H || R.gate.N != F || R.down.K != F || R.down.N != H) return false;
    if (!tail_fill_gemm(P.g[0], B.aq, B.asf, M, num_m_tiles, grid, o_p, 1, TAIL_EPI_RESIDUAL, hid, H, nullptr, nullptr, 0.0f, 0)) return false;
    if (!tail_fill_gemm(P.g[1], B.nq, B.nsf, M, num_m_tiles, grid, gu_p, 2, TAIL_EPI_SILU_QUANT, nullptr, 0, gq, gsf, R.down.input_scale, 1))
        return false;
    if (!tail_fill_gemm(P.g[2], gq, gsf, M, num_m_tiles, grid, down_p, 1, TAIL_EPI_RESIDUAL, hid, H, nullptr, nullptr, 0.0f, 2)) return false;
    // o and down write the same columns of the hidden state; with the same split every thread of the down phase
    // adds to what it wrote itself in the o phase
    P.g[0].res_local = 1;
    P.g[2].res_local = (P.g[0].cpm == P.g[2].cpm && R.o.N == R.down.N) ? 1 : 0;
    fill_norm(P.n[0], R.norm2, R.gate.input_scale);
    add(TAIL_GEMM, 0);
    add(TAIL_NORM, 0);
    add(TAIL_GEMM, 1);
    add(TAIL_GEMM, 2);
    double flops = 2.0 * M * ((double)H * H + 2.0 * F * H + (double)H * F);
    double wbytes = 0.5625 * ((double)H * H + 2.0 * F * H + (double)H * F);
    if (next != nullptr) {
        const ProjRef *qkv_p[3] = {&next->q, &next->k, &next->v};
        if (next->q.K != H || next->q.N != H || next->k.N != KV || next->v.N != KV) return false;
        if (!tail_fill_gemm(P.g[3], B.nq, B.nsf, M, num_m_tiles, grid, qkv_p, 3, TAIL_EPI_STORE, B.qkv, H + 2 * KV, nullptr, nullptr, 0.0f, 3))
            return false;
        fill_norm(P.n[1], next->norm1, next->q.input_scale);
        add(TAIL_NORM, 1);
        add(TAIL_GEMM, 3);
        flops += 2.0 * M * (double)(H + 2 * KV) * H;
        wbytes += 0.5625 * (double)(H + 2 * KV) * H;
    }
    if (max_phases > 0 && max_phases < P.num_phases) P.num_phases = max_phases;
    P.M = M;
    P.num_m_tiles = num_m_tiles;
    P.counter = counter;
    P.base = base;
    P.status = device_status_word();
#ifdef GLMASR_EXPERIMENTS
    {
        const char *e = getenv("GLMASR_TAIL_DEBUG");
        P.debug = e ? atoi(e) : 0;
        P.dbg = (unsigned long long *)workspace_slot(kTailDebugSlot, (size_t)grid * kTailMaxPhases * 16 * 8);
    }
#endif
    profile_bracket_begin(flops, wbytes);
    const cudaError_t e = launch_decode_tail(P, st);
    profile_bracket_end();
    if (e != cudaSuccess) {
        // e.g. a device that cannot keep the whole grid co-resident: nothing ran, the caller takes the
        // one-launch-per-operation path from here on
        (void)cudaGetLastError();
        g_tail_refused = true;
        return false;
    }
    base += (unsigned int)grid;
    note_launches(1);
    return true;
}

}  // namespace glmasr

using namespace glmasr;

enum DecodeSlot : int {   // workspace slots 13.. (api.cu owns 0..12)
    WS_D_HID = 13, WS_D_NORM = 14, WS_D_QKV = 15, WS_D_ATTN = 16, WS_D_ACT = 17, WS_D_SLOT = 18, WS_D_LENS = 19,
    WS_D_BT = 20, WS_D_ROWS = 21, WS_D_PTRS = 22, WS_D_SCRATCH = 23, WS_D_XQ = 26, WS_D_XSF = 27,
    WS_D_POS = 28, WS_D_OFFS = 29,
    // 30, 31: api.cu (split-K).  Quantised hand-overs of the decode step share the layer path's slots 24, 25
    // (both are temporaries of one call).
    WS_D_AQ = 24, WS_D_ASF = 25,
    WS_D_GQ = 48, WS_D_GSF = 49, WS_D_COUNTER = 50,   // layer tail: quantised SiLU-gate output, grid counter
    // 51: the layer tail's cycle counters (experiment builds)
    WS_D_ANGLES = 52,                                 // cos / sin of every row's position
};

// ============================================================================================
// reference-named glue entry points
// ============================================================================================
extern "C" void rmsnorm(uint16_t *out, const uint16_t *x, const uint16_t *weight, float eps, int rows, int dim) {
    launch_rmsnorm((__nv_bfloat16 *)out, (const __nv_bfloat16 *)x, (const __nv_bfloat16 *)weight, eps, rows, dim,
                   current_stream());
    note_launches(1);
    GLMASR_CUDA_CHECK(cudaGetLastError());
}

extern "C" void embedding_lookup(uint16_t *out, const uint16_t *table, const int *ids, int n, int dim) {
    launch_embedding_lookup((__nv_bfloat16 *)out, (const __nv_bfloat16 *)table, ids, n, dim, current_stream());
    note_launches(1);
    GLMASR_CUDA_CHECK(cudaGetLastError());
}

extern "C" void reshape_and_cache(uint16_t *key_cache, uint16_t *value_cache, const uint16_t *key, const uint16_t *value,
                                  const int64_t *slot_mapping, int num_tokens, int num_kv_heads, int head_dim,
                                  int block_size) {
    const int row = num_kv_heads * head_dim;
    launch_reshape_and_cache((__nv_bfloat16 *)key_cache, (__nv_bfloat16 *)value_cache, (const __nv_bfloat16 *)key, row,
                             (const __nv_bfloat16 *)value, row, slot_mapping, num_tokens, num_kv_heads, head_dim,
                             block_size, current_stream());
    GLMASR_CUDA_CHECK(cudaGetLastError());
}

extern "C" void paged_decode_attention(uint16_t *out, const uint16_t *query, const uint16_t *key_cache,
                                       const uint16_t *value_cache, const int *block_tables, const int *seq_lens,
                                       int num_seqs, int num_q_heads, int num_kv_heads, int head_dim, int block_size,
                                       int max_blocks_per_seq) {
    const int ld = num_q_heads * head_dim;
    const bool ok = launch_paged_decode_attention((__nv_bfloat16 *)out, ld, (const __nv_bfloat16 *)query, ld,
                                                  (const __nv_bfloat16 *)key_cache, (const __nv_bfloat16 *)value_cache,
                                                  block_tables, seq_lens, num_seqs, num_q_heads, num_kv_heads, head_dim,
                                                  block_size, max_blocks_per_seq, current_stream());
    GLMASR_CHECK(ok, "paged_decode_attention: unsupported shape (head_dim %d, %d q / %d kv heads)", head_dim,
                 num_q_heads, num_kv_heads);
    GLMASR_CUDA_CHECK(cudaGetLastError());
}

extern "C" void glmasr_rope_single_token(uint16_t *tensor, const int *positions, int num_seqs, int n_heads,
                                         int head_dim) {
    launch_rope_single_token((__nv_bfloat16 *)tensor, n_heads * head_dim, 0, positions, num_seqs, n_heads, head_dim,
                             current_stream());
    GLMASR_CUDA_CHECK(cudaGetLastError());
}

extern "C" int glmasr_rope_qk_cache(uint16_t *qkv, int ld, int k_col, int v_col, const int *positions,
                                    const int64_t *slot_mapping, uint16_t *key_cache, uint16_t *value_cache, int num_seqs,
                                    int q_heads, int kv_heads, int head_dim) {
    if (qkv == nullptr || positions == nullptr || slot_mapping == nullptr || key_cache == nullptr || value_cache == nullptr)
        return -1;
    if (!launch_rope_qk_cache((__nv_bfloat16 *)qkv, ld, k_col, v_col, positions, slot_mapping, (__nv_bfloat16 *)key_cache,
                              (__nv_bfloat16 *)value_cache, num_seqs, q_heads, kv_heads, head_dim, current_stream()))
        return -1;
    note_launches(1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

extern "C" int glmasr_rmsnorm_quant(uint8_t *packed_out, uint8_t *tiled_scale_out, const uint16_t *x, const uint16_t *weight,
                                    float eps, float input_scale, int rows, int dim) {
    if (packed_out == nullptr || tiled_scale_out == nullptr || x == nullptr || weight == nullptr) return -1;
    if (!launch_rmsnorm_quant(packed_out, tiled_scale_out, (const __nv_bfloat16 *)x, (const __nv_bfloat16 *)weight, eps,
                              input_scale, rows, dim, current_stream()))
        return -1;
    note_launches(1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// W4A4 linear on an activation that is already quantised (e2m1 bytes [M, K/2] + 128x4-tiled scales, as
// glmasr_rmsnorm_quant or a quantising epilogue writes them).  resident = 0: the library's regular GEMM kernels;
// resident = 1: one GEMM phase of the co-resident layer-tail kernel (M <= 256; GLMASR_EPI_RESIDUAL adds in place,
// residual == out; GLMASR_EPI_SILU_GATE writes only the quantised product q_out / q_out_sf).  Both give the same bytes.
extern "C" int glmasr_fp4_linear_quantized(int resident, uint16_t *out, int ldo, const uint8_t *xq, const uint8_t *xq_sf,
                                           const glmasr_fp4_weight *weights, int num_weights, float input_scale, int epilogue,
                                           const uint16_t *residual, int M, int K, uint8_t *q_out, uint8_t *q_out_sf,
                                           float q_out_input_scale) {
    if (xq == nullptr || xq_sf == nullptr || weights == nullptr || num_weights < 1 || num_weights > 3 || M <= 0) return -1;
    if (!resident)
        return fp4_linear_w4a4_prequantized(out, ldo, xq, xq_sf, weights, num_weights, input_scale, epilogue, residual, M, K, q_out,
                                            q_out_sf, q_out_input_scale);
    const int grid = tail_grid_size();
    if (grid <= 0 || M > 256) return -1;
    ProjRef refs[3];
    const ProjRef *ps[3];
    for (int i = 0; i < num_weights; ++i) {
        refs[i].dtype = GLMASR_DTYPE_UINT8;
        refs[i].w = weights[i].w_packed;
        refs[i].scales = weights[i].w_scales;
        refs[i].global_scale = weights[i].w_global_scale;
        refs[i].input_scale = input_scale;
        refs[i].N = weights[i].N;
        refs[i].K = K;
        ps[i] = &refs[i];
    }
    int epi = TAIL_EPI_STORE;
    if (epilogue == GLMASR_EPI_RESIDUAL) {
        if (residual != out || out == nullptr) return -1;
        epi = TAIL_EPI_RESIDUAL;
    } else if (epilogue == GLMASR_EPI_SILU_GATE) {
        if (q_out == nullptr || q_out_sf == nullptr) return -1;
        epi = TAIL_EPI_SILU_QUANT;
    } else if (out == nullptr) {
        return -1;
    }
    static TailParams P;
    const int num_m_tiles = (M + 127) / 128;
    if (!tail_fill_gemm(P.g[0], xq, xq_sf, M, num_m_tiles, grid, ps, num_weights, epi, out, ldo, q_out, q_out_sf, q_out_input_scale))
        return -1;
    unsigned int *counter = (unsigned int *)workspace_slot(WS_D_COUNTER, kTailCounterBytes);
    if (cudaMemsetAsync(counter, 0, kTailCounterBytes, current_stream()) != cudaSuccess) return -1;
    P.kind[0] = TAIL_GEMM;
    P.index[0] = 0;
    P.num_phases = 1;
    P.M = M;
    P.num_m_tiles = num_m_tiles;
    P.counter = counter;
    P.base = 0;
    P.status = device_status_word();
    if (launch_decode_tail(P, current_stream()) != cudaSuccess) {
        (void)cudaGetLastError();
        return -1;
    }
    note_launches(1);
    return 0;
}

static ProjRef proj_of(const glmasr_fp4_weight &w, float input_scale, int K) {
    ProjRef r;
    r.dtype = GLMASR_DTYPE_UINT8;
    r.w = w.w_packed;
    r.scales = w.w_scales;
    r.global_scale = w.w_global_scale;
    r.input_scale = input_scale;
    r.N = w.N;
    r.K = K;
    return r;
}

// One launch of the co-resident layer-tail kernel on the caller's buffers (the decode driver above does the same
// on its private workspace): o + residual | norm + quantiser | gate|up + SiLU-gate + quantiser | down + residual
// and, with `next`, | norm + quantiser | q|k|v of the following layer.
extern "C" int glmasr_decode_layer_tail(uint16_t *hidden, int M, const uint8_t *attn_q, const uint8_t *attn_sf,
                                        const glmasr_layer_weights *lw, const uint16_t *post_attention_norm,
                                        const glmasr_layer_weights *next, const uint16_t *next_input_norm, uint16_t *next_qkv,
                                        uint8_t *norm_q, uint8_t *norm_sf, uint8_t *act_q, uint8_t *act_sf, int max_phases) {
    if (hidden == nullptr || attn_q == nullptr || attn_sf == nullptr || lw == nullptr || post_attention_norm == nullptr ||
        norm_q == nullptr || norm_sf == nullptr || act_q == nullptr || act_sf == nullptr || M <= 0 || M > 256)
        return -1;
    if (next != nullptr && (next_input_norm == nullptr || next_qkv == nullptr)) return -1;
    const int H = lw->hidden, F = lw->ffn;
    LayerRef R, N;
    R.norm2 = post_attention_norm;
    R.o = proj_of(lw->o, lw->in_o, H);
    R.gate = proj_of(lw->gate, lw->in_gate_up, H);
    R.up = proj_of(lw->up, lw->in_gate_up, H);
    R.down = proj_of(lw->down, lw->in_down, F);
    int KV = 0;
    if (next != nullptr) {
        N.norm1 = next_input_norm;
        N.q = proj_of(next->q, next->in_qkv, H);
        N.k = proj_of(next->k, next->in_qkv, H);
        N.v = proj_of(next->v, next->in_qkv, H);
        KV = next->k.N;
    }
    StepBuffers B = {nullptr, next_qkv, nullptr, nullptr, norm_q, norm_sf, const_cast<uint8_t *>(attn_q), const_cast<uint8_t *>(attn_sf)};
    unsigned int *counter = (unsigned int *)workspace_slot(WS_D_COUNTER, kTailCounterBytes);
    if (cudaMemsetAsync(counter, 0, kTailCounterBytes, current_stream()) != cudaSuccess) return -1;
    unsigned int base = 0;
    return launch_layer_tail(R, next != nullptr ? &N : nullptr, hidden, B, act_q, act_sf, counter, base, M, H, KV, F,
                             current_stream(), max_phases)
               ? 0
               : -1;
}

#ifdef GLMASR_EXPERIMENTS
// experiment builds only: read (and clear) the layer-tail kernel's cycle counters [CTAs][phases][16]
extern "C" int glmasr_tail_debug_read(unsigned long long *host_out, int clear) {
    const int grid = tail_grid_size();
    const size_t bytes = (size_t)grid * kTailMaxPhases * 16 * 8;
    unsigned long long *d = (unsigned long long *)workspace_slot(kTailDebugSlot, bytes);
    cudaStreamSynchronize(current_stream());
    if (host_out != nullptr && cudaMemcpy(host_out, d, bytes, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    if (clear) cudaMemset(d, 0, bytes);
    return grid;
}
#endif

// ============================================================================================
// decoder_decode_step_batched
// ============================================================================================
extern "C" void decoder_decode_step_batched(void *handle, const void *ws_v, uint16_t **query_ptrs, void *pool_v,
                                            void *bts_v, int *d_seq_lens, int *h_seq_lens, int num_seqs,
                                            int *seq_indices, uint16_t *dequant_buf, const void *cfg_v) {
    (void)handle;
    (void)dequant_buf;
    const glmasr_WeightStore *ws = (const glmasr_WeightStore *)ws_v;
    const glmasr_ModelConfig *cfg = (const glmasr_ModelConfig *)cfg_v;
    glmasr_KVPool *pool = (glmasr_KVPool *)pool_v;
    glmasr_BlockTable *bts = (glmasr_BlockTable *)bts_v;
    if (num_seqs <= 0) return;
    GLMASR_CHECK(query_ptrs != nullptr, "decoder_decode_step_batched: query_ptrs is NULL");
    GLMASR_CHECK(pool != nullptr, "decoder_decode_step_batched: pool is NULL");
    GLMASR_CHECK(bts != nullptr, "decoder_decode_step_batched: bts is NULL");
    GLMASR_CHECK(d_seq_lens != nullptr, "decoder_decode_step_batched: d_seq_lens is NULL");
    GLMASR_CHECK(h_seq_lens != nullptr, "decoder_decode_step_batched: h_seq_lens is NULL");

    const int H = cfg->dec_hidden, L = cfg->dec_layers, QH = cfg->dec_heads, KVH = cfg->dec_kv_heads;
    const int HD = cfg->dec_head_dim, F = cfg->dec_ffn;
    const int KV = KVH * HD, NQKV = H + 2 * KV, M = num_seqs;
    GLMASR_CHECK(QH * HD == H, "decoder_decode_step_batched: heads * head_dim != hidden");
    const ModelRefs &refs = model_refs(ws, L);
    cudaStream_t st = current_stream();

    // ---- host-side step set-up (reference: decoder.cu:1911-1938) ----
    std::vector<int64_t> h_slot(M);
    std::vector<int> h_total(M), h_rows(M);
    bool contiguous = true;
    int max_total = 0;
    for (int s = 0; s < M; ++s) {
        const int cached = h_seq_lens[s];
        GLMASR_CHECK(query_ptrs[s] != nullptr, "decoder_decode_step_batched: query_ptrs[%d] is NULL", s);
        GLMASR_CHECK(bts[s].h_table != nullptr, "decoder_decode_step_batched: bts[%d].h_table is NULL", s);
        GLMASR_CHECK(cached >= 0, "decoder_decode_step_batched: negative seq len for seq %d", s);
        const int logical = cached / pool->block_size;
        GLMASR_CHECK(logical < bts[s].num_blocks, "decoder_decode_step_batched: seq %d length %d exceeds %d allocated blocks",
                     s, cached, bts[s].num_blocks);
        h_slot[s] = (int64_t)bts[s].h_table[logical] * (int64_t)pool->block_size + (int64_t)(cached % pool->block_size);
        h_total[s] = cached + 1;
        if (cached + 1 > max_total) max_total = cached + 1;
        h_rows[s] = seq_indices ? seq_indices[s] : bts[s].seq_idx;
        GLMASR_CHECK(h_rows[s] >= 0 && h_rows[s] < pool->max_seqs,
                     "decoder_decode_step_batched: invalid seq index %d for batch row %d", h_rows[s], s);
        if (query_ptrs[s] != query_ptrs[0] + (size_t)s * H) contiguous = false;
    }
    const bool rows_independent = !rows_share_new_pages(bts, h_seq_lens, M, pool->block_size);

    uint16_t *hid = (uint16_t *)workspace_slot(WS_D_HID, (size_t)M * H * 2);
    uint16_t *nrm = (uint16_t *)workspace_slot(WS_D_NORM, (size_t)M * H * 2);
    uint16_t *qkv = (uint16_t *)workspace_slot(WS_D_QKV, (size_t)M * NQKV * 2);
    uint16_t *att = (uint16_t *)workspace_slot(WS_D_ATTN, (size_t)M * H * 2);
    uint16_t *act = (uint16_t *)workspace_slot(WS_D_ACT, (size_t)M * 2 * F * 2);
    int64_t *d_slot = (int64_t *)workspace_slot(WS_D_SLOT, (size_t)M * sizeof(int64_t));
    int *d_total = (int *)workspace_slot(WS_D_LENS, (size_t)M * sizeof(int));
    int *d_bt = (int *)workspace_slot(WS_D_BT, (size_t)M * pool->max_blocks_per_seq * sizeof(int));
    int *d_rows = (int *)workspace_slot(WS_D_ROWS, (size_t)M * sizeof(int));
    uint16_t **d_ptrs = (uint16_t **)workspace_slot(WS_D_PTRS, (size_t)M * sizeof(void *));
    uint16_t *scratch = (uint16_t *)workspace_slot(WS_D_SCRATCH, (size_t)M * (F > H ? F : H) * 2);
    uint8_t *nq = (uint8_t *)workspace_slot(WS_D_XQ, (size_t)M * H / 2);
    uint8_t *nsf = (uint8_t *)workspace_slot(WS_D_XSF, tiled_scale_bytes(M, H));
    // quantised attention output (K = H) and SiLU-gate output (K = F) handed to the o / down projections
    const int KQ = F > H ? F : H;
    uint8_t *aq = (uint8_t *)workspace_slot(WS_D_AQ, (size_t)M * KQ / 2);
    uint8_t *asf = (uint8_t *)workspace_slot(WS_D_ASF, tiled_scale_bytes(M, KQ));

    const StepBuffers B = {nrm, qkv, act, scratch, nq, nsf, aq, asf};

    // the rotary angles depend on the positions only: one evaluation for all layers
    float *rope_angles = (float *)workspace_slot(WS_D_ANGLES, (size_t)M * HD * sizeof(float));
    {
        PlainLaunch plain(true);        // the kernels behind it fetch weights and cached rows early
        if (launch_step_setup((__nv_bfloat16 *)hid, query_ptrs, M, H, h_slot.data(), d_slot, h_total.data(), d_total, h_rows.data(),
                              pool->d_block_tables, d_bt, pool->max_blocks_per_seq, d_seq_lens, rope_angles, HD, st)) {
            note_launches(1);
            if (!contiguous) GLMASR_CUDA_CHECK(cudaMemcpyAsync(d_ptrs, query_ptrs, (size_t)M * sizeof(void *), cudaMemcpyHostToDevice, st));
        } else {
            GLMASR_CUDA_CHECK(cudaMemcpyAsync(d_slot, h_slot.data(), (size_t)M * sizeof(int64_t), cudaMemcpyHostToDevice, st));
            GLMASR_CUDA_CHECK(cudaMemcpyAsync(d_total, h_total.data(), (size_t)M * sizeof(int), cudaMemcpyHostToDevice, st));
            GLMASR_CUDA_CHECK(cudaMemcpyAsync(d_rows, h_rows.data(), (size_t)M * sizeof(int), cudaMemcpyHostToDevice, st));
            if (contiguous) {
                GLMASR_CUDA_CHECK(cudaMemcpyAsync(hid, query_ptrs[0], (size_t)M * H * 2, cudaMemcpyDeviceToDevice, st));
            } else {
                GLMASR_CUDA_CHECK(cudaMemcpyAsync(d_ptrs, query_ptrs, (size_t)M * sizeof(void *), cudaMemcpyHostToDevice, st));
                launch_gather_rows((__nv_bfloat16 *)hid, (const __nv_bfloat16 *const *)d_ptrs, M, H, st);
            }
            launch_gather_block_tables(d_bt, pool->d_block_tables, d_rows, M, pool->max_blocks_per_seq, st);
            // the vectors above are pageable host memory: the async copies have completed staging on return
            if (launch_rope_angles(rope_angles, d_seq_lens, M, HD, st)) note_launches(1);
            else rope_angles = nullptr;
        }
    }
    SettledWeights settled(true);

    // the layer tail (o .. next layer's q|k|v) as one co-resident launch where it applies
    const bool tail = tail_enabled() && M <= 256;
    uint8_t *gq = nullptr, *gsf = nullptr;
    unsigned int *tail_counter = nullptr, tail_base = 0;
    if (tail) {
        gq = (uint8_t *)workspace_slot(WS_D_GQ, (size_t)M * F / 2);
        gsf = (uint8_t *)workspace_slot(WS_D_GSF, tiled_scale_bytes(M, F));
        tail_counter = (unsigned int *)workspace_slot(WS_D_COUNTER, kTailCounterBytes);
        GLMASR_CUDA_CHECK(cudaMemsetAsync(tail_counter, 0, kTailCounterBytes, st));
    }
    bool have_qkv = false;      // the previous layer's tail already projected this layer's q | k | v

    for (int l = 0; l < L; ++l) {
        const LayerRef &R = refs.layers[l];
        __nv_bfloat16 *k_base = (__nv_bfloat16 *)pool->k_cache + (size_t)l * pool->layer_stride;
        __nv_bfloat16 *v_base = (__nv_bfloat16 *)pool->v_cache + (size_t)l * pool->layer_stride;

        // q | k | v into one [M, H + 2 KV] buffer
        int glue = 0;
        bool early_cache = false;       // attention may read the cache and the step's tables ahead of its dependency wait
        if (!have_qkv) {
            LateTrigger late;
            glue = project_qkv(R, hid, B, M, H, KV, st);
            early_cache = late_trigger_taken();
        }
        have_qkv = false;
        // attention writes the o projection's quantised operand itself when that projection runs in W4A4
        const bool o_q = takes_quantised_input(R.o) && R.o.K == H && !attn_scalar_forced();
        // RoPE on q and k (position = cached length), KV write and attention over cached + 1 tokens: one launch ...
        bool ok = rows_independent && !attn_scalar_forced() &&
                  launch_paged_decode_split((__nv_bfloat16 *)att, H, (const __nv_bfloat16 *)qkv, NQKV, H, H + KV, rope_angles, d_slot,
                                            k_base, v_base, d_bt, d_total, M, QH, KVH, HD, pool->block_size,
                                            pool->max_blocks_per_seq, max_total, st, early_cache, o_q ? aq : nullptr,
                                            o_q ? asf : nullptr, R.o.input_scale);
        if (ok && !o_q) {
            single_proj(hid, H, att, H, R.o, M, hid, scratch);
            glue += project_mlp(R, hid, B, M, H, F, st);
            note_launches(glue + 1);
            continue;
        }
        // ... or, in layouts that one does not take and where rows read what others of the step write, one each
        if (!ok) {
            if (launch_rope_qk_cache((__nv_bfloat16 *)qkv, NQKV, H, H + KV, d_seq_lens, d_slot, k_base, v_base, M, QH, KVH, HD, st, rope_angles)) {
                glue += 1;
            } else {
                launch_rope_single_token((__nv_bfloat16 *)qkv, NQKV, 0, d_seq_lens, M, QH, HD, st);
                launch_rope_single_token((__nv_bfloat16 *)qkv, NQKV, H, d_seq_lens, M, KVH, HD, st);
                launch_reshape_and_cache(k_base, v_base, (const __nv_bfloat16 *)qkv + H, NQKV,
                                         (const __nv_bfloat16 *)qkv + H + KV, NQKV, d_slot, M, KVH, HD, pool->block_size, st);
                glue += 3;
            }
            if (o_q)
                ok = launch_paged_decode_attention_mma((__nv_bfloat16 *)att, H, (const __nv_bfloat16 *)qkv, NQKV, k_base, v_base,
                                                       d_bt, d_total, M, QH, KVH, HD, pool->block_size, pool->max_blocks_per_seq,
                                                       st, aq, asf, R.o.input_scale);
        }
        if (ok && tail &&
            launch_layer_tail(R, l + 1 < L ? &refs.layers[l + 1] : nullptr, hid, B, gq, gsf, tail_counter, tail_base, M, H, KV, F, st)) {
            have_qkv = l + 1 < L;
            note_launches(glue + 1);
            continue;
        }
        if (ok) {
            single_proj_prequantized(hid, H, aq, asf, R.o, M, hid);
        } else {
            ok = launch_paged_decode_attention((__nv_bfloat16 *)att, H, (const __nv_bfloat16 *)qkv, NQKV, k_base, v_base, d_bt,
                                               d_total, M, QH, KVH, HD, pool->block_size, pool->max_blocks_per_seq, st);
            GLMASR_CHECK(ok, "decoder_decode_step_batched: unsupported attention shape");
            // o + residual -> hid (residual is the pre-norm hidden state)
            single_proj(hid, H, att, H, R.o, M, hid, scratch);
        }

        glue += project_mlp(R, hid, B, M, H, F, st);
        note_launches(glue + 1);   // norms, RoPE / cache write, attention (the projections count themselves)
    }

    // final norm straight into the caller's rows, advanced lengths with it
    if (contiguous) {
        launch_rmsnorm_lens((__nv_bfloat16 *)query_ptrs[0], (const __nv_bfloat16 *)hid, (const __nv_bfloat16 *)refs.final_norm, 1e-5f,
                            M, H, d_seq_lens, d_total, st);
        note_launches(1);
    } else {
        launch_rmsnorm_lens((__nv_bfloat16 *)hid, (const __nv_bfloat16 *)hid, (const __nv_bfloat16 *)refs.final_norm, 1e-5f, M, H,
                            d_seq_lens, d_total, st);
        launch_scatter_rows((__nv_bfloat16 *const *)d_ptrs, (const __nv_bfloat16 *)hid, M, H, st);
        note_launches(2);
    }
    for (int s = 0; s < M; ++s) h_seq_lens[s] = h_total[s];
    GLMASR_CUDA_CHECK(cudaGetLastError());
}

// The reference's attention plug-in entry points (Infer-engine/cuda/flash_fwd_vllm.h:21-30), served
// by this library's own kernel: q / k / v rows of sequence s are [cu_seqlens[s], cu_seqlens[s+1]),
// row strides in elements, out dense [total, q_heads * head_dim].  Returns 1 on success like the plug-in.
extern "C" int flash_fwd_vllm_gqa_available(void) { return 1; }

extern "C" int flash_fwd_vllm_gqa_launch(void *q, void *k, void *v, void *out, int total_seqlen, int max_seqlen, int q_heads,
                                         int kv_heads, int head_dim, int q_row_stride, int k_row_stride, int v_row_stride,
                                         int num_seqs, int *d_cu_seqlens, int is_causal) {
    if (q == nullptr || k == nullptr || v == nullptr || out == nullptr || d_cu_seqlens == nullptr) return 0;
    if (total_seqlen <= 0 || num_seqs <= 0) return 1;
    if (!launch_prefill_attention((__nv_bfloat16 *)out, q_heads * head_dim, (const __nv_bfloat16 *)q, q_row_stride,
                                  (const __nv_bfloat16 *)k, k_row_stride, (const __nv_bfloat16 *)v, v_row_stride,
                                  d_cu_seqlens, nullptr, num_seqs, max_seqlen, total_seqlen, q_heads, kv_heads, head_dim,
                                  is_causal != 0,
                                  current_stream()))
        return 0;
    note_launches(1);
    return cudaGetLastError() == cudaSuccess ? 1 : 0;
}

// ============================================================================================
// decoder_prefill_paged_batched (reference: Infer-engine/cuda/decoder.cu:1219-1557)
// ============================================================================================
// Batched variable-length prefill, in place on hidden [total_tokens, H]: sequence s owns rows
// [seq_offsets[s], seq_offsets[s] + seq_lens[s]) and the blocks of bts[s]; positions start at 0.
// Per layer: RMSNorm -> q|k|v (one GEMM) -> RoPE(q, k) + K / V rows into the paged cache (one
// launch) -> causal attention over the sequence's own tokens -> o + residual -> RMSNorm ->
// gate|up with SiLU-gate -> down + residual; final RMSNorm.  seq_lens / seq_offsets are host arrays
// as in the reference.
extern "C" void decoder_prefill_paged_batched(void *handle, const void *ws_v, uint16_t *hidden, int total_tokens,
                                              int num_seqs, const int *seq_lens, const int *seq_offsets, void *pool_v,
                                              void *bts_v, uint16_t *dequant_buf, const void *cfg_v) {
    (void)handle;
    (void)dequant_buf;
    const glmasr_WeightStore *ws = (const glmasr_WeightStore *)ws_v;
    const glmasr_ModelConfig *cfg = (const glmasr_ModelConfig *)cfg_v;
    glmasr_KVPool *pool = (glmasr_KVPool *)pool_v;
    glmasr_BlockTable *bts = (glmasr_BlockTable *)bts_v;
    GLMASR_CHECK(total_tokens > 0, "decoder_prefill_paged_batched requires tokens");
    GLMASR_CHECK(num_seqs > 0, "decoder_prefill_paged_batched requires sequences");
    GLMASR_CHECK(hidden != nullptr && seq_lens != nullptr && seq_offsets != nullptr && pool != nullptr && bts != nullptr,
                 "decoder_prefill_paged_batched received null metadata");

    const int H = cfg->dec_hidden, L = cfg->dec_layers, QH = cfg->dec_heads, KVH = cfg->dec_kv_heads;
    const int HD = cfg->dec_head_dim, F = cfg->dec_ffn;
    const int KV = KVH * HD, NQKV = H + 2 * KV, M = total_tokens;
    GLMASR_CHECK(QH * HD == H, "decoder_prefill_paged_batched: heads * head_dim != hidden");
    const ModelRefs &refs = model_refs(ws, L);
    cudaStream_t st = current_stream();

    // ---- host-side set-up: slot of every token, its position, the sequence table ----
    std::vector<int64_t> h_slot((size_t)M, -1);
    std::vector<int> h_pos((size_t)M, 0), h_meta((size_t)2 * num_seqs);
    int max_len = 0;
    for (int s = 0; s < num_seqs; ++s) {
        const int len = seq_lens[s], off = seq_offsets[s];
        GLMASR_CHECK(len >= 0 && off >= 0 && off + len <= M, "decoder_prefill_paged_batched: sequence %d outside the batch", s);
        GLMASR_CHECK(bts[s].h_table != nullptr, "decoder_prefill_paged_batched: bts[%d].h_table is NULL", s);
        for (int t = 0; t < len; ++t) {
            const int blk = t / pool->block_size;
            GLMASR_CHECK(blk < bts[s].num_blocks, "Prefill block table too small for seq=%d tok=%d", s, t);
            h_slot[(size_t)off + t] = (int64_t)bts[s].h_table[blk] * (int64_t)pool->block_size + (int64_t)(t % pool->block_size);
            h_pos[(size_t)off + t] = t;
        }
        h_meta[s] = off;
        h_meta[num_seqs + s] = len;
        if (len > max_len) max_len = len;
    }
    GLMASR_CHECK(max_len > 0, "decoder_prefill_paged_batched max_seq_len invalid");
    for (int t = 0; t < M; ++t)
        GLMASR_CHECK(h_slot[t] >= 0, "decoder_prefill_paged_batched: token row %d belongs to no sequence", t);

    uint16_t *nrm = (uint16_t *)workspace_slot(WS_D_NORM, (size_t)M * H * 2);
    uint16_t *qkv = (uint16_t *)workspace_slot(WS_D_QKV, (size_t)M * NQKV * 2);
    uint16_t *att = (uint16_t *)workspace_slot(WS_D_ATTN, (size_t)M * H * 2);
    uint16_t *act = (uint16_t *)workspace_slot(WS_D_ACT, (size_t)M * 2 * F * 2);
    uint16_t *scratch = (uint16_t *)workspace_slot(WS_D_SCRATCH, (size_t)M * (F > H ? F : H) * 2);
    uint8_t *nq = (uint8_t *)workspace_slot(WS_D_XQ, (size_t)M * H / 2);
    uint8_t *nsf = (uint8_t *)workspace_slot(WS_D_XSF, tiled_scale_bytes(M, H));
    // quantised SiLU-gate output (K = F) handed to the down projection
    const int KQ = F > H ? F : H;
    uint8_t *aq = (uint8_t *)workspace_slot(WS_D_AQ, (size_t)M * KQ / 2);
    uint8_t *asf = (uint8_t *)workspace_slot(WS_D_ASF, tiled_scale_bytes(M, KQ));
    int64_t *d_slot = (int64_t *)workspace_slot(WS_D_SLOT, (size_t)M * sizeof(int64_t));
    int *d_pos = (int *)workspace_slot(WS_D_POS, (size_t)M * sizeof(int));
    int *d_meta = (int *)workspace_slot(WS_D_OFFS, (size_t)2 * num_seqs * sizeof(int));
    const StepBuffers B = {nrm, qkv, act, scratch, nq, nsf, aq, asf};
    // pageable host vectors: the copies have been staged when these calls return
    GLMASR_CUDA_CHECK(cudaMemcpyAsync(d_slot, h_slot.data(), (size_t)M * sizeof(int64_t), cudaMemcpyHostToDevice, st));
    GLMASR_CUDA_CHECK(cudaMemcpyAsync(d_pos, h_pos.data(), (size_t)M * sizeof(int), cudaMemcpyHostToDevice, st));
    GLMASR_CUDA_CHECK(cudaMemcpyAsync(d_meta, h_meta.data(), (size_t)2 * num_seqs * sizeof(int), cudaMemcpyHostToDevice, st));
    float *rope_angles = (float *)workspace_slot(WS_D_ANGLES, (size_t)M * HD * sizeof(float));
    {
        PlainLaunch plain(true);
        if (launch_rope_angles(rope_angles, d_pos, M, HD, st)) note_launches(1);
        else rope_angles = nullptr;
    }
    SettledWeights settled(rope_angles != nullptr);

    uint16_t *hid = hidden;
    for (int l = 0; l < L; ++l) {
        const LayerRef &R = refs.layers[l];
        __nv_bfloat16 *k_base = (__nv_bfloat16 *)pool->k_cache + (size_t)l * pool->layer_stride;
        __nv_bfloat16 *v_base = (__nv_bfloat16 *)pool->v_cache + (size_t)l * pool->layer_stride;
        int glue = 0;

        glue += project_qkv(R, hid, B, M, H, KV, st);
        if (launch_rope_qk_cache((__nv_bfloat16 *)qkv, NQKV, H, H + KV, d_pos, d_slot, k_base, v_base, M, QH, KVH, HD, st, rope_angles)) {
            glue += 1;
        } else {
            launch_rope_single_token((__nv_bfloat16 *)qkv, NQKV, 0, d_pos, M, QH, HD, st);
            launch_rope_single_token((__nv_bfloat16 *)qkv, NQKV, H, d_pos, M, KVH, HD, st);
            launch_reshape_and_cache(k_base, v_base, (const __nv_bfloat16 *)qkv + H, NQKV,
                                     (const __nv_bfloat16 *)qkv + H + KV, NQKV, d_slot, M, KVH, HD, pool->block_size, st);
            glue += 3;
        }
        // attention; where the o projection takes a quantised operand the kernel writes that instead of bf16
        const bool o_q = takes_quantised_input(R.o) && R.o.K == H && QH * HD == H;
        if (o_q && launch_prefill_attention((__nv_bfloat16 *)att, H, (const __nv_bfloat16 *)qkv, NQKV,
                                            (const __nv_bfloat16 *)qkv + H, NQKV, (const __nv_bfloat16 *)qkv + H + KV, NQKV,
                                            d_meta, d_meta + num_seqs, num_seqs, max_len, M, QH, KVH, HD, true, st, aq, asf,
                                            R.o.input_scale)) {
            single_proj_prequantized(hid, H, aq, asf, R.o, M, hid);
        } else {
            const bool ok = launch_prefill_attention((__nv_bfloat16 *)att, H, (const __nv_bfloat16 *)qkv, NQKV,
                                                     (const __nv_bfloat16 *)qkv + H, NQKV,
                                                     (const __nv_bfloat16 *)qkv + H + KV, NQKV, d_meta, d_meta + num_seqs,
                                                     num_seqs, max_len, M, QH, KVH, HD, true, st);
            GLMASR_CHECK(ok, "decoder_prefill_paged_batched: unsupported attention shape");
            single_proj(hid, H, att, H, R.o, M, hid, scratch);
        }
        glue += 1;

        glue += project_mlp(R, hid, B, M, H, F, st);
        note_launches(glue);
    }
    launch_rmsnorm((__nv_bfloat16 *)hid, (const __nv_bfloat16 *)hid, (const __nv_bfloat16 *)refs.final_norm, 1e-5f, M, H, st);
    note_launches(1);
    GLMASR_CUDA_CHECK(cudaGetLastError());
}

extern "C" void glmasr_decoder_forget_weights(void) { forget_model_refs(); }
