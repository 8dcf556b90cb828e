// W4A16 linear for a handful of rows (decode of a few sequences).
//
// With M <= 16 rows the tcgen05 kernels leave most of the chip idle: a 2048-column projection has sixteen 128-wide
// tiles, and each of those CTAs pulls its whole K range through one ring at the ~100 GB/s one SM gets (down projection,
// K = 6144: 27 us; a decode step of one sequence took 2.56 ms, 0.06 of the rate of the bytes it has to read).  Here the
// weights are the MMA's 16-row operand and the tokens its 8-column operand (mma.sync m16n8k16: 128 token lanes of a
// tcgen05 tile would be empty), so the work cuts into 16-row units that spread over every SM:
//   * a CTA takes `units_per_cta` consecutive 16-row units (gate and up rows together for the SiLU epilogue) and asks for
//     ALL their bytes -- packed nibbles and block scales, as stored -- with bulk copies before it waits for the preceding
//     kernel.  The copies run under the predecessor's tail, so the weight stream does not wait for the chain of
//     activations; the small footprint (two of these kernels share an SM) is what makes that overlap possible.
//     Weights too tall for that (an output head) go through two groups of slots;
//   * eight warps split K in chunks of 128: lane (g, t) owns the 32 consecutive elements 32 t .. 32 t + 31 of a chunk for
//     rows g and g + 8, two whole scale blocks, so that its weights are one 16-byte shared load per row.  The MMA's
//     k order is a permutation of that (the same one for both operands): pairs (i, i + 4) of every 8-nibble word;
//   * e2m1 -> bf16 without a table: sign to bit 15, exponent and mantissa to bits 8..6 read as bf16 of value * 2^-126
//     (subnormals included), one packed multiply by scale * 2^112 gives value * scale * 2^-14 exactly, and 2^14 goes into
//     the per-tensor factor;
//   * RMSNorm of the input is folded in: x * w is rounded to bf16 as the operand, 1 / rms (from the same registers)
//     multiplies the fp32 sums;
//   * the eight partial sums meet in shared memory, fixed order.
// Asking for a warp's activations of several K chunks at once (two or three, 124 - 128 registers) made a decode step of one
// sequence slower, 1106 against 1029 us, and so did three of these CTAs per SM at 80 registers (1076 against 999).
// W4A4 stays on the block-scaled MMA: with the quantiser folded in here too (every CTA rounds the rows for itself) one row of
// [2048, 2048] took 8.5 us on the device against 7.2 for quantiser and MMA.
// From 17 rows the tokens' operand no longer fits the registers beside the accumulators and the bf16 copies on the cluster
// GEMM are faster (19 sequences: 1.96 against 2.33 ms a step).
// Bound: instruction issue of the dequantisation (five instructions per two weights; 1.8 us for gate|up) and the fixed
// latencies of a launch in a dependent chain, with the 28 MB of a layer's weights streamed underneath.
#include "gemm_skinny.cuh"

#include <cuda_bf16.h>

#include "gemm_umma.cuh"
#include "ptx.cuh"
#include "runtime.cuh"

namespace glmasr {

static constexpr int kWarpsSk = 8;
static constexpr int kThreadsSk = kWarpsSk * 32;
static constexpr int kSmemHeader = 1280;            // barriers, abort word, sums of squares [8][16]
static constexpr int kSmemWeights = 150 * 1024;     // most that weight slots may take

__host__ __device__ constexpr int sk_tiles_per_pass(int nt) { return nt == 1 ? 6 : 4; }
__host__ __device__ inline int sk_slot_bytes(int K) { return 16 * (K / 2 + 16) + 16 * (K / 16 + 16); }

__device__ __forceinline__ uint32_t lds16_sk(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint4 lds128_sk(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
// scale byte -> bf16x2 of (scale * 2^112) twice; decoded as the reference does (no NaN pattern, sign honoured)
__device__ __forceinline__ uint32_t scale_x2(uint32_t b) {
    const float f = __uint_as_float(((b & 0x7Fu) << 20) | ((b & 0x80u) << 24));      // scale * 2^-120
    const float s = f * 8.307674973655724e34f * 8.307674973655724e34f;               // 2^116 twice
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %1;" : "=r"(d) : "f"(s));
    return d;
}
// nibbles I and I + 4 of w as a bf16 pair of value * 2^-126
template <int I>
__device__ __forceinline__ uint32_t nib_pair(uint32_t w) {
    constexpr int up = 12 - 4 * I;                       // brings nibble I to bits 15..12 (and I + 4 to 31..28)
    uint32_t mag;
    if constexpr (up > 6) mag = w << (up - 6);
    else mag = w >> (6 - up);
    return ((w << up) & 0x80008000u) | (mag & 0x01C001C0u);
}
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

enum SkinnySource : int { SK_PLAIN = 0, SK_NORM = 1 };

// One 8-element word pair order: elements 0..7 of `v` (four bf16x2 words) as the pairs (0,4) (1,5) (2,6) (3,7).
__device__ __forceinline__ void permute8(const uint4 &v, uint32_t (&o)[4]) {
    o[0] = __byte_perm(v.x, v.z, 0x5410);
    o[1] = __byte_perm(v.x, v.z, 0x7632);
    o[2] = __byte_perm(v.y, v.w, 0x5410);
    o[3] = __byte_perm(v.y, v.w, 0x7632);
}

template <int NT, int SRC>
__global__ void __launch_bounds__(kThreadsSk, 2) skinny_linear_kernel(const __grid_constant__ SkinnyParams p) {
    constexpr int R = sk_tiles_per_pass(NT);            // 16-row tiles accumulated at a time
    extern __shared__ __align__(128) uint8_t sk_smem[];
    volatile int *abort_word = reinterpret_cast<volatile int *>(sk_smem + 32);
    float *ssum = reinterpret_cast<float *>(sk_smem + 64);                    // [8 warps][NT * 8]
    const int slot_bytes = sk_slot_bytes(p.K);
    const int w_pitch = p.K / 2 + 16, s_pitch = p.K / 16 + 16;
    const bool silu = p.epi == EPI_SILU_GATE;
    const int mt = silu ? 2 : 1;                        // 16-row tiles per unit
    const uint32_t bars = smem_u32(sk_smem);
    const uint32_t slots = bars + kSmemHeader;
    float *part = reinterpret_cast<float *>(sk_smem + kSmemHeader + (size_t)p.groups * p.units_per_group * mt * slot_bytes);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    const int u0 = blockIdx.x * p.units_per_cta;
    const int u_end = min(p.units, u0 + p.units_per_cta);
    const int rounds = (u_end - u0 + p.units_per_group - 1) / p.units_per_group;

    if (!p.late_trigger) pdl_launch_dependents();
    if (threadIdx.x == 0) {
        mbar_init(bars, 1);
        mbar_init(bars + 8, 1);
        *abort_word = 0;
        fence_mbar_init();
        fence_proxy_async_smem();
    }
    __syncthreads();

    // every byte of round r's weights: a warp per 16-row tile, a lane per row of nibbles or scales
    auto issue_round = [&](int r) {
        const int first = u0 + r * p.units_per_group;
        const int tiles = (min(u_end, first + p.units_per_group) - first) * mt;
        const int grp = r % p.groups;
        const uint32_t bar = bars + 8 * grp;
        if (threadIdx.x == 0) mbar_expect_tx(bar, (uint32_t)tiles * 16u * (uint32_t)(p.K / 2 + p.K / 16));
        for (int t = warp; t < tiles; t += kWarpsSk) {
            int seg, row;
            if (silu) {
                seg = t & 1;
                row = (first + (t >> 1)) * 16;
            } else {
                row = (first + t) * 16;
                seg = 0;
                while (seg < p.num_segs - 1 && row >= p.seg_rows[seg]) row -= p.seg_rows[seg++];
            }
            const uint32_t dst = slots + (uint32_t)((grp * p.units_per_group * mt + t) * slot_bytes);
            const int rr = lane & 15;
            if (lane < 16)
                bulk_load_1d(dst + rr * w_pitch, p.w[seg] + (size_t)(row + rr) * (p.K / 2), p.K / 2, bar);
            else
                bulk_load_1d(dst + 16 * w_pitch + rr * s_pitch, p.ws[seg] + (size_t)(row + rr) * (p.K / 16), p.K / 16, bar);
        }
    };
    if (!p.early_weights) pdl_wait();
    for (int r = 0; r < p.groups && r < rounds; ++r) issue_round(r);
    if (p.early_weights) pdl_wait();
    if (p.late_trigger) pdl_launch_dependents();

    const int chunks = p.K >> 7;
    float ss[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) ss[n] = 0.0f;

    for (int r = 0; r < rounds; ++r) {
        const int first = u0 + r * p.units_per_group;
        const int tiles = (min(u_end, first + p.units_per_group) - first) * mt;
        const int grp = r % p.groups;
        bool landed = false;
        for (int t0 = 0; t0 < tiles; t0 += R) {
            float acc[R][NT][4];
#pragma unroll
            for (int t = 0; t < R; ++t)
#pragma unroll
                for (int n = 0; n < NT; ++n) acc[t][n][0] = acc[t][n][1] = acc[t][n][2] = acc[t][n][3] = 0.0f;
            for (int c = warp; c < chunks; c += kWarpsSk) {
                // tokens' operand: 32 consecutive elements of this chunk for token 8 n + g
                uint32_t b[NT][16];
                const int k0 = c * 128 + tq * 32;
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    uint4 v[4];
                    const int tok = n * 8 + g;
                    const uint4 *src = reinterpret_cast<const uint4 *>(p.x + (size_t)tok * p.ldx + k0);
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[j] = tok < p.M ? src[j] : make_uint4(0u, 0u, 0u, 0u);
                    if (SRC == SK_NORM) {
                        const uint4 *nw = reinterpret_cast<const uint4 *>(p.norm_w + k0);
                        const bool count = r == 0 && t0 == 0;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const uint4 w4 = nw[j];
                            if (count) {
                                const uint32_t xs[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    const float lo = __uint_as_float(xs[e] << 16), hi = __uint_as_float(xs[e] & 0xFFFF0000u);
                                    ss[n] = fmaf(lo, lo, ss[n]);
                                    ss[n] = fmaf(hi, hi, ss[n]);
                                }
                            }
                            v[j] = make_uint4(mul_bf16x2(v[j].x, w4.x), mul_bf16x2(v[j].y, w4.y), mul_bf16x2(v[j].z, w4.z),
                                              mul_bf16x2(v[j].w, w4.w));
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t o[4];
                        permute8(v[j], o);
#pragma unroll
                        for (int e = 0; e < 4; ++e) b[n][4 * j + e] = o[e];
                    }
                }
                if (!landed) {
                    if (!mbar_wait(bars + 8 * grp, (uint32_t)((r / p.groups) & 1), abort_word, ST_TIMEOUT_PRODUCER)) atomicExch(p.status, ST_TIMEOUT_PRODUCER);
                    landed = true;
                }
#pragma unroll
                for (int t = 0; t < R; ++t) {
                    if (t0 + t < tiles) {
                        const uint32_t base = slots + (uint32_t)((grp * p.units_per_group * mt + t0 + t) * slot_bytes);
                        const uint32_t wa = base + g * w_pitch + c * 64 + tq * 16;
                        const uint32_t sa = base + 16 * w_pitch + g * s_pitch + c * 8 + tq * 2;
                        const uint4 w0 = lds128_sk(wa), w1 = lds128_sk(wa + 8 * w_pitch);
                        const uint32_t sb0 = lds16_sk(sa), sb1 = lds16_sk(sa + 8 * s_pitch);
                        const uint32_t s0[2] = {scale_x2(sb0 & 0xFFu), scale_x2(sb0 >> 8)};
                        const uint32_t s1[2] = {scale_x2(sb1 & 0xFFu), scale_x2(sb1 >> 8)};
                        const uint32_t q0[4] = {w0.x, w0.y, w0.z, w0.w}, q1[4] = {w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const uint32_t m0 = s0[j >> 1], m1 = s1[j >> 1];
                            uint32_t a0 = mul_bf16x2(nib_pair<0>(q0[j]), m0), a1 = mul_bf16x2(nib_pair<0>(q1[j]), m1);
                            uint32_t a2 = mul_bf16x2(nib_pair<1>(q0[j]), m0), a3 = mul_bf16x2(nib_pair<1>(q1[j]), m1);
#pragma unroll
                            for (int n = 0; n < NT; ++n) mma_16816(acc[t][n], a0, a1, a2, a3, b[n][4 * j], b[n][4 * j + 1]);
                            a0 = mul_bf16x2(nib_pair<2>(q0[j]), m0), a1 = mul_bf16x2(nib_pair<2>(q1[j]), m1);
                            a2 = mul_bf16x2(nib_pair<3>(q0[j]), m0), a3 = mul_bf16x2(nib_pair<3>(q1[j]), m1);
#pragma unroll
                            for (int n = 0; n < NT; ++n) mma_16816(acc[t][n], a0, a1, a2, a3, b[n][4 * j + 2], b[n][4 * j + 3]);
                        }
                    }
                }
            }
            // partial sums of this warp: [tile][row 0..15][token], tokens contiguous
#pragma unroll
            for (int t = 0; t < R; ++t)
                if (t0 + t < tiles) {
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        float *dst = part + ((size_t)(warp * p.pass_tiles + t) * 16 + g) * (NT * 8) + n * 8 + tq * 2;
                        *reinterpret_cast<float2 *>(dst) = make_float2(acc[t][n][0], acc[t][n][1]);
                        *reinterpret_cast<float2 *>(dst + 8 * (NT * 8)) = make_float2(acc[t][n][2], acc[t][n][3]);
                    }
                }
            if (SRC == SK_NORM && r == 0 && t0 == 0) {
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    ss[n] += __shfl_xor_sync(0xFFFFFFFFu, ss[n], 1);
                    ss[n] += __shfl_xor_sync(0xFFFFFFFFu, ss[n], 2);
                    if (tq == 0) ssum[warp * (NT * 8) + n * 8 + g] = ss[n];
                }
            }
            __syncthreads();
            if (*abort_word != 0) {
                for (int i = 0; i < 64; ++i) __nanosleep(1000);     // let copies in flight land
                return;
            }
            // sum over the warps, epilogue: a thread per (unit, token, row), rows fastest
            const int units = (min(tiles, t0 + R) - t0) / mt;
            for (int i = threadIdx.x; i < units * 16 * p.M; i += kThreadsSk) {
                const int row = i & 15, um = i >> 4, tok = um % p.M, u = um / p.M;
                float v[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    v[h] = 0.0f;
                    if (h < mt) {
                        const float *src = part + ((size_t)(u * mt + h) * 16 + row) * (NT * 8) + tok;
#pragma unroll
                        for (int w = 0; w < kWarpsSk; ++w) v[h] += src[(size_t)w * p.pass_tiles * 16 * NT * 8];
                    }
                }
                if (SRC == SK_NORM) {
                    float s = 0.0f;
#pragma unroll
                    for (int w = 0; w < kWarpsSk; ++w) s += ssum[w * (NT * 8) + tok];
                    const float inv = 1.0f / sqrtf(s / p.K + p.eps);
                    v[0] *= inv;
                    v[1] *= inv;
                }
                const int unit = first + t0 / mt + u;
                const int col = unit * 16 + row;
                if (silu) {
                    const float gt = __bfloat162float(__float2bfloat16(v[0] * (p.alpha[0] * 16384.0f)));
                    const float up = __bfloat162float(__float2bfloat16(v[1] * (p.alpha[1] * 16384.0f)));
                    const float e = __expf(-gt);
                    p.out[(size_t)tok * p.ldo + col] = __float2bfloat16(gt / (1.0f + e) * up);
                } else {
                    int seg = 0, c0 = col;
                    while (seg < p.num_segs - 1 && c0 >= p.seg_rows[seg]) c0 -= p.seg_rows[seg++];
                    float o = v[0] * (p.alpha[seg] * 16384.0f);
                    const size_t at = (size_t)tok * p.ldo + col;
                    if (p.bias != nullptr) o += __bfloat162float(p.bias[col]);
                    if (p.epi == EPI_RESIDUAL) o = __bfloat162float(__float2bfloat16(o)) + __bfloat162float(p.residual[at]);
                    p.out[at] = __float2bfloat16(o);
                }
            }
            __syncthreads();
        }
        if (r + p.groups < rounds) issue_round(r + p.groups);
    }
}

bool skinny_covers(int M, int K, const int *seg_rows, int num_segs, int epi) {
    if (M < 1 || M > kSkinnyMaxRows || K < 256 || (K % 256) != 0 || K > 8192 || num_segs < 1 || num_segs > 3) return false;
    if (epi != EPI_STORE && epi != EPI_RESIDUAL && epi != EPI_SILU_GATE) return false;
    if (epi == EPI_SILU_GATE && (num_segs != 2 || seg_rows[0] != seg_rows[1])) return false;
    for (int i = 0; i < num_segs; ++i)
        if (seg_rows[i] <= 0 || (seg_rows[i] % 16) != 0) return false;
    return true;
}

// The other route reads bf16 copies, 3.6 times the bytes; this one pays for dequantising and, per CTA, for the rows' operand in
// every pass.  Both sides in us, weights not in L2, this kernel / the other:
//   * weights of a CTA all requested up front (they fit the slots), K >= 1536: 2048 x 6144 8.9 / 24.8 (1 row), 12.4 / 24.8 (16);
//     12288 x 2048 9.3 / 20.6, 15.2 / 19.8; 8192 x 4096 11.9 / 30, 14.8 / 19.6; 4096 x 8192 13.3 / 41, 16.5 / 32: always;
//   * taller ones go through the ring.  Below 128 KB of rows the other route is slow as well: 24576 x 2048 16.4 / 32 (1), 24.5 / 30
//     (16); 59264 x 2048 34.6 / 58, 50.9 / 53 (12) but 55 / 52 (16); 24576 x 6144 59 / 85, 81 / 88 (9).  From 128 KB of rows on it
//     is not: 16384 x 8192 58 / 49 (8), 66 / 49 (16); 8192 x 6144 32 / 27 (12); 12288 x 4096 26 / 23 (16);
//   * K below 1536 leaves warps without a chunk and units too short: 9472 x 1024 5.4 / 9.6 (1), 7.3 / 9.3 (16), 16384 x 1024 10.8 / 11.9
//     (8), 14.6 / 11.6 (16); 9472 x 512 5.5 / 6.3 (8), 7.0 / 6.3 (16), 16384 x 512 8.6 / 7.7 (8); 16384 x 256 7.0 / 5.9 (1).
bool skinny_pays(int M, int K, const int *seg_rows, int num_segs, int epi, int num_sms) {
    const int mt = epi == EPI_SILU_GATE ? 2 : 1;
    int rows = 0;
    for (int i = 0; i < (mt == 2 ? 1 : num_segs); ++i) rows += seg_rows[i];
    const int tiles = (rows / 16 + num_sms - 1) / num_sms * mt;         // 16-row tiles of a CTA
    if (K < 512) return M <= 8 && tiles <= 1;
    if (K < 1024) return tiles <= (M <= 8 ? 4 : 1);
    if (K < 1536) return M <= 8 || tiles <= 4;
    if (tiles * sk_slot_bytes(K) <= kSmemWeights) return true;
    return M * K < 65536 && !(M > 12 && tiles > 20);
}

template <int NT>
static cudaError_t launch_nt(const SkinnyParams &p, int grid, size_t smem, cudaStream_t st) {
    void (*kernel)(SkinnyParams) = p.norm_w != nullptr ? skinny_linear_kernel<NT, SK_NORM> : skinny_linear_kernel<NT, SK_PLAIN>;
    static PerDevice<bool> ready[2];
    const cudaError_t e = once_per_device(ready[p.norm_w != nullptr ? SK_NORM : SK_PLAIN], [&] {
        const cudaError_t e1 = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
        if (e1 != cudaSuccess) return e1;
        return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    });
    if (e != cudaSuccess) return e;
    return launch_chained(kernel, dim3(grid), dim3(kThreadsSk), smem, st, p);
}

cudaError_t launch_skinny_linear(SkinnyParams p, int num_sms, cudaStream_t st, int *rounds) {
    if (!skinny_covers(p.M, p.K, p.seg_rows, p.num_segs, p.epi)) return cudaErrorInvalidValue;
    const int mt = p.epi == EPI_SILU_GATE ? 2 : 1;
    int rows = 0;
    for (int i = 0; i < (mt == 2 ? 1 : p.num_segs); ++i) rows += p.seg_rows[i];
    p.units = rows / 16;
    p.units_per_cta = (p.units + num_sms - 1) / num_sms;
    const int unit_bytes = mt * sk_slot_bytes(p.K);
    const int nt = p.M <= 8 ? 1 : 2;
    const int per_pass = sk_tiles_per_pass(nt) / mt;         // units accumulated at a time
    if (p.units_per_cta * unit_bytes <= kSmemWeights) {
        p.groups = 1;
        p.units_per_group = p.units_per_cta;
    } else {
        p.groups = 2;
        p.units_per_group = kSmemWeights / 2 / unit_bytes;
        if (p.units_per_group > per_pass) p.units_per_group = p.units_per_group / per_pass * per_pass;
        if (p.units_per_group < 1) p.groups = 1, p.units_per_group = 1;
    }
    const int grid = (p.units + p.units_per_cta - 1) / p.units_per_cta;
    *rounds = (p.units_per_cta + p.units_per_group - 1) / p.units_per_group;
    p.pass_tiles = sk_tiles_per_pass(nt) < p.units_per_group * mt ? sk_tiles_per_pass(nt) : p.units_per_group * mt;
    const size_t smem = kSmemHeader + (size_t)p.groups * p.units_per_group * unit_bytes +
                        (size_t)kWarpsSk * p.pass_tiles * 16 * nt * 8 * sizeof(float);
    return nt == 1 ? launch_nt<1>(p, grid, smem, st) : launch_nt<2>(p, grid, smem, st);
}

}  // namespace glmasr
