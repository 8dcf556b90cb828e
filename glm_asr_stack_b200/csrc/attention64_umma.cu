// Self-attention with head_dim 64 (the audio encoder: 20 heads, 1500 keys, no mask; the plug-in entry may also ask for a
// causal mask) on the tcgen05 tensor cores: per sequence softmax(Q K^T / 8 [+ causal mask]) V, the arithmetic of
// prefill_attention_umma.cu.
//
// Sixteen sequences of 1500 rows, 20 heads: 382 -> 302 us (the head_dim 128 kernel run at 64, with its launch that transposed V,
// before).  With 64 dims a score costs 256 multiply-adds of tensor work and one exponential, so the special-function unit (16 per
// clock and SM) is the bound: 0.75 G exponentials per layer of 16 full windows are 319 k cycles of it.  The head_dim 128
// kernel run at 64 (64 keys a step) took 616 k: about 950 cycles of every soft-max step are not exponentials -- tensor-memory
// load, maximum, hand-overs -- and two warps per scheduler cannot hide them behind each other's 512.  Four CTAs per SM with a
// serial chain each (one score buffer shared with P) were no better (3400 cycles a step, the two round trips to the MMA
// warp in it).  So here
//   * a step is 128 keys: the fixed part is paid once per 1024 exponential cycles;
//   * a thread takes its row's 128 scores into registers at once and frees the score buffer: the next Q K^T runs under
//     the exponentials;
//   * P goes to its own 64 columns of tensor memory, from where it is the second product's A operand: no shared-memory
//     stores, no proxy fence.  Scores [0, 128), P [128, 192), output [192, 256): two CTAs per SM;
//   * V is read as it lies in memory (MN-major B operand).
//   warp 0 TMA producer, warp 1 MMA issuer, warps 2-5 soft-max (thread = query row = TMEM lane).
#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>

#include "decoder_ops.cuh"
#include "ptx.cuh"
#include "runtime.cuh"

namespace glmasr {

namespace {

constexpr int QT = 128, KT = 128, HD = 64, THREADS64 = 192, CTAS_PER_SM = 2;
constexpr int Q_BYTES = QT * 128, KV_BYTES = KT * 128;
constexpr int OFF_Q = 0, OFF_K = Q_BYTES, OFF_V = OFF_K + 2 * KV_BYTES, OFF_BAR = OFF_V + 2 * KV_BYTES;
constexpr int SMEM64 = OFF_BAR + 256;
constexpr int TMEM_COLS64 = 256, COL_P = 128, COL_O = 192;
constexpr float kRescale = 8.0f;              // log2 units: P may grow to 2^8 of the value the accumulator is expressed against

enum : int { B_QFULL = 0, B_QEMPTY = 1, B_KFULL = 2, B_KEMPTY = 4, B_VFULL = 6, B_VEMPTY = 8, B_SFULL = 10, B_SFREE = 11, B_PFULL = 12, B_PVDONE = 13 };

struct Attn64Params {
    CUtensorMap tm_q, tm_k, tm_v;
    __nv_bfloat16 *out;
    const int *seq_offsets, *seq_lens;        // seq_lens NULL: seq_offsets is cumulative (num_seqs + 1 entries)
    int *status;
    int ldo, num_q_heads, num_seqs, group, q_tiles, total_items, causal;
    float scale_log2;                         // log2(e) / sqrt(head_dim)
};

struct Item64 {
    int head, seq, q0, off, len, n;
};
// Items that run side by side share K and V: all query tiles of a (sequence, head) in a row, so that 16 full windows' 123 MB
// of K and V pass through L2 once (query-tile-major order read them from DRAM twelve times over: 350 us a layer whatever
// the soft-max did).  Under a causal mask the tiles differ in length, longest first.
__device__ __forceinline__ bool decode_item64(const Attn64Params &p, int item, Item64 &it) {
    const int pairs = p.num_q_heads * p.num_seqs;
    const int x = p.causal ? item % pairs : item / p.q_tiles;
    const int tile = p.causal ? p.q_tiles - 1 - item / pairs : item % p.q_tiles;
    it.q0 = tile * QT;
    it.head = x % p.num_q_heads;
    it.seq = x / p.num_q_heads;
    it.off = p.seq_offsets[it.seq];
    it.len = p.seq_lens != nullptr ? p.seq_lens[it.seq] : p.seq_offsets[it.seq + 1] - it.off;
    if (it.q0 >= it.len) return false;
    const int kv_end = p.causal ? min(it.len, it.q0 + QT) : it.len;
    it.n = (kv_end + KT - 1) / KT;
    return true;
}

__device__ __forceinline__ float ex2_sfu(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&b);
}
__global__ void __launch_bounds__(THREADS64, CTAS_PER_SM) attention64_umma_kernel(const __grid_constant__ Attn64Params p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if ((sbase & 1023u) != 0) {                 // the swizzled tiles need a 1024-byte aligned base
        if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, ST_BAD_LAYOUT);
        return;
    }
    auto bar = [&](int i) { return sbase + OFF_BAR + 8u * (uint32_t)i; };
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + OFF_BAR + 192);
    volatile int *abort_word = reinterpret_cast<volatile int *>(smem + OFF_BAR + 200);
    if (threadIdx.x == 0) {
        for (int i = 0; i <= B_PVDONE; ++i) mbar_init(bar(i), i == B_PFULL || i == B_SFREE ? 128 : 1);
        *abort_word = 0;
        fence_mbar_init();
        tma_prefetch_desc(&p.tm_q);
        tma_prefetch_desc(&p.tm_k);
        tma_prefetch_desc(&p.tm_v);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32((const void *)tmem_slot), TMEM_COLS64);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();                                 // nothing above touched global memory

    if (warp == 0) {
        // ---- TMA producer ----
        const bool leader = elect_one();
        uint32_t kv = 0, qi = 0;
        bool ok = true;
        for (int item = blockIdx.x; ok && item < p.total_items; item += gridDim.x) {
            Item64 it;
            if (!decode_item64(p, item, it)) continue;
            const int kv_col = it.head / p.group * HD;
            if (!mbar_wait_warp(bar(B_QEMPTY), (qi & 1u) ^ 1u, abort_word, ST_TIMEOUT_ATTENTION)) break;
            if (leader) {
                mbar_expect_tx(bar(B_QFULL), Q_BYTES);
                tma_load_2d(sbase + OFF_Q, &p.tm_q, bar(B_QFULL), it.head * HD, it.off + it.q0);
            }
            ++qi;
            for (int j = 0; j < it.n; ++j, ++kv) {
                const uint32_t s = kv & 1u, ph = ((kv >> 1) & 1u) ^ 1u;
                if (!mbar_wait_warp(bar(B_KEMPTY + s), ph, abort_word, ST_TIMEOUT_ATTENTION)) { ok = false; break; }
                if (leader) {
                    mbar_expect_tx(bar(B_KFULL + s), KV_BYTES);
                    tma_load_2d(sbase + OFF_K + s * KV_BYTES, &p.tm_k, bar(B_KFULL + s), kv_col, it.off + j * KT);
                }
                if (!mbar_wait_warp(bar(B_VEMPTY + s), ph, abort_word, ST_TIMEOUT_ATTENTION)) { ok = false; break; }
                if (leader) {
                    mbar_expect_tx(bar(B_VFULL + s), KV_BYTES);
                    tma_load_2d(sbase + OFF_V + s * KV_BYTES, &p.tm_v, bar(B_VFULL + s), kv_col, it.off + j * KT);
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer ----
        const bool leader = elect_one();
        constexpr uint32_t idesc_s = idesc_bf16(128, KT), idesc_o = idesc_bf16(128, HD) | kIdescBMnMajor;
        uint32_t ks = 0, kp = 0, qi = 0;        // S products issued, P V products issued, items started
        bool ok = true;
        for (int item = blockIdx.x; ok && item < p.total_items; item += gridDim.x) {
            Item64 it;
            if (!decode_item64(p, item, it)) continue;
            if (!mbar_wait_warp(bar(B_QFULL), qi & 1u, abort_word, ST_TIMEOUT_ATTENTION)) break;
            ++qi;
            for (int j = 0; j <= it.n; ++j) {
                if (j < it.n) {
                    const uint32_t s = ks & 1u;
                    if (!mbar_wait_warp(bar(B_KFULL + s), (ks >> 1) & 1u, abort_word, ST_TIMEOUT_ATTENTION)) { ok = false; break; }
                    // the score buffer is free once the soft-max has taken the step before into registers
                    if (!mbar_wait_warp(bar(B_SFREE), (ks & 1u) ^ 1u, abort_word, ST_TIMEOUT_ATTENTION)) { ok = false; break; }
                    tc_fence_after();
                    if (leader) {
                        const uint64_t ad = smem_desc_sw128(sbase + OFF_Q), bd = smem_desc_sw128(sbase + OFF_K + s * KV_BYTES);
#pragma unroll
                        for (int k = 0; k < HD / 16; ++k) umma_bf16(tmem_base, ad + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), idesc_s, k > 0 ? 1u : 0u);
                        umma_commit(bar(B_SFULL));
                        umma_commit(bar(B_KEMPTY + s));
                        if (j == it.n - 1) umma_commit(bar(B_QEMPTY));      // last product that reads this Q tile
                    }
                    ++ks;
                }
                if (j >= 1) {
                    const uint32_t s = kp & 1u;
                    if (!mbar_wait_warp(bar(B_VFULL + s), (kp >> 1) & 1u, abort_word, ST_TIMEOUT_ATTENTION)) { ok = false; break; }
                    if (!mbar_wait_warp(bar(B_PFULL), kp & 1u, abort_word, ST_TIMEOUT_ATTENTION)) { ok = false; break; }
                    tc_fence_after();
                    if (leader) {
                        const uint64_t bd = smem_desc_sw128_mn(sbase + OFF_V + s * KV_BYTES, KV_BYTES);
                        const int k_steps = (min(KT, it.len - (j - 1) * KT) + 15) >> 4;
#pragma unroll
                        for (int k = 0; k < KT / 16; ++k)
                            if (k < k_steps)
                                umma_bf16_ts(tmem_base + COL_O, tmem_base + COL_P + 8u * (uint32_t)k, bd + (uint64_t)((2048 * k) >> 4),
                                             idesc_o, (j > 1 || k > 0) ? 1u : 0u);
                        umma_commit(bar(B_PVDONE));
                        umma_commit(bar(B_VEMPTY + s));
                    }
                    ++kp;
                }
            }
        }
    } else {
        // ---- soft-max ----
        const int quad = warp & 3;                      // TMEM lane quadrant of this warp
        const int row = quad * 32 + lane;
        const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16);
        const float scale = p.scale_log2;
        const unsigned long long scale2 = pack_f32x2(scale, scale);
        uint32_t sc = 0;
        bool ok = true;
        for (int item = blockIdx.x; ok && item < p.total_items; item += gridDim.x) {
            Item64 it;
            if (!decode_item64(p, item, it)) continue;
            const int row_g = it.q0 + row;
            const int visible = p.causal ? min(it.len, row_g + 1) : it.len;
            float m = -INFINITY, l = 0.0f;
            for (int j = 0; j < it.n; ++j, ++sc) {
                if (!mbar_wait_warp(bar(B_SFULL), sc & 1u, abort_word, ST_TIMEOUT_ATTENTION)) { ok = false; break; }
                tc_fence_after();
                const int lim = visible - j * KT;       // columns [0, lim) of this step count for this row
                // keys of this step that exist: whole blocks of 32 columns behind them cost nothing, nor does the second product
                // walk past them (20 heads, 100 sequences of 60 rows 32.2 -> 25.6 us, one of 400 rows 11.6 -> 10.4)
                const int v_rows = it.len - j * KT, blocks = (min(v_rows, KT) + 31) >> 5;
                uint32_t sr[4][32];
#pragma unroll
                for (int h = 0; h < 4; ++h)
                    if (h < blocks) tmem_ld_x32(t_row + 32u * h, sr[h]);
                tmem_ld_wait();
                tc_fence_before();
                mbar_arrive(bar(B_SFREE));
                if (lim < KT) {
#pragma unroll
                    for (int c = 0; c < KT; ++c)
                        if (c >= lim) sr[c >> 5][c & 31] = 0xFF800000u;      // -inf
                }
                float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    mx0 = max3(mx0, __uint_as_float(sr[0][c]), __uint_as_float(sr[0][c + 1]));
                    mx1 = max3(mx1, __uint_as_float(sr[1][c]), __uint_as_float(sr[1][c + 1]));
                    mx2 = max3(mx2, __uint_as_float(sr[2][c]), __uint_as_float(sr[2][c + 1]));
                    mx3 = max3(mx3, __uint_as_float(sr[3][c]), __uint_as_float(sr[3][c + 1]));
                }
                const float m_new = fmaxf(m, max3(mx0, mx1, fmaxf(mx2, mx3)) * scale);
                float alpha = 1.0f;
                if (j == 0) {
                    m = m_new;
                } else if (m_new - m > kRescale) {
                    alpha = ex2_sfu(m - m_new);
                    m = m_new;
                }
                const bool rescale = __any_sync(0xFFFFFFFFu, alpha != 1.0f);
                // the product of the step before reads P and adds to the accumulator: it has to be complete
                if (sc > 0) {
                    if (!mbar_wait_warp(bar(B_PVDONE), (sc - 1u) & 1u, abort_word, ST_TIMEOUT_ATTENTION)) { ok = false; break; }
                    tc_fence_after();
                }
                if (rescale) {
#pragma unroll 1
                    for (int h = 0; h < 4; ++h) {
                        uint32_t o[16];
                        tmem_ld_x16(t_row + COL_O + 16u * h, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
                        tmem_st_x16(t_row + COL_O + 16u * h, o);
                    }
                    l *= alpha;
                }
                const unsigned long long neg_m2 = pack_f32x2(-m, -m);
                unsigned long long sum2 = pack_f32x2(0.0f, 0.0f);
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    if (h >= blocks) break;
                    uint32_t pk[16];
#pragma unroll
                    for (int c = 0; c < 32; c += 2) {
                        float t0, t1;
                        unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sr[h][c]), __uint_as_float(sr[h][c + 1])), scale2, neg_m2), t0, t1);
                        t0 = ex2_sfu(t0);
                        t1 = ex2_sfu(t1);
                        sum2 = add_f32x2(sum2, pack_f32x2(t0, t1));
                        pk[c >> 1] = pack_bf16(t0, t1);
                    }
                    tmem_st_x16(t_row + COL_P + 16u * h, pk);
                }
                float sum_lo, sum_hi;
                unpack_f32x2(sum2, sum_lo, sum_hi);
                l += sum_lo + sum_hi;
                // keys past the sequence's end weigh nothing, but the rows behind it may hold anything (another sequence, or
                // memory nobody wrote): 0 * NaN must not reach the sum
                if (v_rows < KT) {
                    const uint32_t s = sc & 1u;
                    if (!mbar_wait_warp(bar(B_VFULL + s), (sc >> 1) & 1u, abort_word, ST_TIMEOUT_ATTENTION)) { ok = false; break; }
                    for (int c = v_rows * 8 + row; c < blocks * 256; c += 128)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(sbase + OFF_V + s * KV_BYTES + (uint32_t)c * 16u), "r"(0) : "memory");
                    fence_proxy_async_smem();
                }
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(bar(B_PFULL));
            }
            if (!ok) break;
            if (!mbar_wait_warp(bar(B_PVDONE), (sc - 1u) & 1u, abort_word, ST_TIMEOUT_ATTENTION)) { ok = false; break; }
            tc_fence_after();
            // a row's 64 results are 128 contiguous bytes: four 32-byte stores, whole sectors each
            const float inv = l > 0.0f ? 1.0f / l : 0.0f;
            __nv_bfloat16 *dst = p.out + (size_t)(it.off + row_g) * p.ldo + (size_t)it.head * HD;
#pragma unroll 1
            for (int h = 0; h < 4; ++h) {
                uint32_t o[16], w[8];
                tmem_ld_x16(t_row + COL_O + 16u * h, o);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 8; ++e) w[e] = pack_bf16(__uint_as_float(o[2 * e]) * inv, __uint_as_float(o[2 * e + 1]) * inv);
                if (row_g < it.len) {
                    if ((((uintptr_t)p.out | (uintptr_t)(p.ldo * 2)) & 31) == 0) {
                        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + 16 * h), "r"(w[0]), "r"(w[1]),
                                     "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                                     : "memory");
                    } else {
                        reinterpret_cast<uint4 *>(dst + 16 * h)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                        reinterpret_cast<uint4 *>(dst + 16 * h)[1] = make_uint4(w[4], w[5], w[6], w[7]);
                    }
                }
            }
            tc_fence_before();      // ordered before this warp's next P hand-over, after which the accumulator is overwritten
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_word != 0) {
        for (int i = 0; i < 64; ++i) __nanosleep(1000);      // let copies in flight land
        if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, *abort_word);
    }
    if (warp == 1) {
        __syncwarp();
        tmem_dealloc(tmem_base, TMEM_COLS64);
    }
}

}  // namespace

// The layout has been checked by launch_prefill_attention_umma (16-byte aligned rows, row pitches multiples of 8).
bool launch_attention64_umma(__nv_bfloat16 *out, int ldo, const __nv_bfloat16 *q, int ldq, const __nv_bfloat16 *k, int ldk,
                             const __nv_bfloat16 *v, int ldv, const int *seq_offsets, const int *seq_lens, int num_seqs,
                             int max_seq_len, int total_tokens, int num_q_heads, int num_kv_heads, bool causal, cudaStream_t st) {
    static PerDevice<bool> configured;
    if (once_per_device(configured, [] { return cudaFuncSetAttribute(attention64_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM64); }) != cudaSuccess)
        return false;
    GLMASR_PREFER_MAX_SMEM(attention64_umma_kernel);
    Attn64Params p;
    memset(&p, 0, sizeof(p));
    if (!make_bf16_tmap_sw128(&p.tm_q, q, (uint64_t)num_q_heads * HD, (uint64_t)total_tokens, (uint64_t)ldq * 2, 64, QT)) return false;
    if (!make_bf16_tmap_sw128(&p.tm_k, k, (uint64_t)num_kv_heads * HD, (uint64_t)total_tokens, (uint64_t)ldk * 2, 64, KT)) return false;
    if (!make_bf16_tmap_sw128(&p.tm_v, v, (uint64_t)num_kv_heads * HD, (uint64_t)total_tokens, (uint64_t)ldv * 2, 64, KT)) return false;
    p.out = out;
    p.seq_offsets = seq_offsets;
    p.seq_lens = seq_lens;
    p.status = device_status_word();
    p.ldo = ldo;
    p.num_q_heads = num_q_heads;
    p.num_seqs = num_seqs;
    p.group = num_q_heads / num_kv_heads;
    p.q_tiles = (max_seq_len + QT - 1) / QT;
    p.total_items = p.q_tiles * num_q_heads * num_seqs;
    p.causal = causal ? 1 : 0;
    p.scale_log2 = 1.4426950408889634f / 8.0f;
    const int grid = p.total_items < CTAS_PER_SM * num_sms() ? p.total_items : CTAS_PER_SM * num_sms();
    const cudaError_t e = launch_chained(attention64_umma_kernel, dim3(grid), dim3(THREADS64), (size_t)SMEM64, st, p);
    if (e != cudaSuccess) (void)cudaGetLastError();         // refused: the caller goes on to the warp-level kernel
    return e == cudaSuccess;
}

}  // namespace glmasr
