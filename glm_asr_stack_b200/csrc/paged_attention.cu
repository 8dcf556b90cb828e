// Paged GQA decode attention, head_dim 128, as a flash-decoding kernel (reference semantics:
// paged_decode_attention, Infer-engine/cuda/paged_kv.cu:321-422, 440-519).
//
// The batched decode step reads ~170 MB of K and V per layer (4.8 GB per step) and only ~1 k
// flops per 512 bytes, so the kernel has to be HBM-bound; a scalar warp-per-head loop (the
// reference's design) is instruction-bound at ~1/10 of the bandwidth.  Here:
//   * one CTA per (kv head, sequence), four warps; warp w takes the 16-token tiles w, w+4, ... of the
//     context and keeps its own online-softmax state; the four partial results are merged through
//     shared memory at the end;
//   * each tile's K and V rows (16 x 256 B each) are brought to shared memory with 16-byte cp.async
//     into a 2-deep per-warp ring (64 KB per CTA, so three CTAs share an SM: measured faster than a deeper ring with two) (rows past the sequence or in masked pages are zero-filled), with
//     the 16-byte chunks XOR-swizzled by row so that ldmatrix is bank-conflict free;
//   * S = Q K^T and O += P V run on mma.sync m16n8k16 (bf16 in, fp32 accumulate): the G <= 8 query
//     heads of the group are rows 0..G-1 of the 16-row A operand.  Four query rows are far below the
//     64/128-row minimum of tcgen05, so the warp-level MMA is the right tool here.
// Result differences to the reference (token-serial fp32 loop): P is rounded to bf16 before the
// PV product and the summation order differs; both are far inside the bf16 output tolerance.
#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>

#include "decoder_ops.cuh"
#include "fp4_format.cuh"
#include "runtime.cuh"

namespace glmasr {

static constexpr int kTile = 16;                       // tokens per tile
static constexpr int kRowBytes = 256;                  // one K or V row of one kv head (128 bf16)
static constexpr int kTileBytes = kTile * kRowBytes;   // 4 KB
static constexpr int kStages = 2;
static constexpr int kWarps = 4;
static constexpr int kWarpSmem = kStages * 2 * kTileBytes;          // K and V rings of one warp: 16 KB
static constexpr int kAttnSmem = kWarps * kWarpSmem;                // 64 KB


__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// D(16x8, fp32) += A(16x16, bf16, row) * B(16x8, bf16, col)
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&b);
}

// swizzled byte offset of 16-byte chunk c (0..15) of row r (0..15) inside a 4 KB tile
__device__ __forceinline__ uint32_t tile_off(int r, int c) { return (uint32_t)(r * kRowBytes + ((c ^ (r & 7)) << 4)); }

// PAGE_ALIGNED: block_size is a multiple of the 16-token tile, so a tile lies in one page: one block-table
// lookup and one division per tile instead of one per row, and row addresses by pointer increments.
template <bool PAGE_ALIGNED>
__global__ void __launch_bounds__(kWarps * 32) paged_decode_attention_mma_kernel(
    __nv_bfloat16 *__restrict__ out, int ldo, const __nv_bfloat16 *__restrict__ query, int ldq,
    const __nv_bfloat16 *__restrict__ key_cache, const __nv_bfloat16 *__restrict__ value_cache,
    const int *__restrict__ block_tables, const int *__restrict__ seq_lens, int num_kv_heads, int group,
    int block_size, int max_blocks_per_seq, float scale, uint8_t *__restrict__ q_packed, uint8_t *__restrict__ q_sf,
    int q_sf_chunks, float q_inv_in) {
    extern __shared__ __align__(1024) uint8_t smem[];
    pdl_launch_dependents();
    pdl_wait();
    const int kv_head = blockIdx.x;
    const int seq = blockIdx.y;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2;            // MMA row / column group of this lane (query head when < group)
    const int tq = lane & 3;
    const int seq_len = seq_lens[seq];
    const int q_head0 = kv_head * group;

    if (seq_len <= 0) {                 // reference: zeros
        if (q_packed != nullptr) {      // zeros quantise to zero codes and zero scales
            const int hidden = num_kv_heads * group * 128;
            for (int i = threadIdx.x; i < group * 64; i += blockDim.x)
                q_packed[(size_t)seq * (hidden / 2) + (size_t)q_head0 * 64 + i] = 0;
            for (int b = threadIdx.x; b < group * 8; b += blockDim.x) {
                const int kb = q_head0 * 8 + b, rem = seq & 127;
                q_sf[((((size_t)(seq >> 7) * q_sf_chunks + (kb >> 2)) * 32 + (rem & 31)) * 4 + (rem >> 5)) * 4 + (kb & 3)] = 0;
            }
            return;
        }
        for (int i = threadIdx.x; i < group * 128; i += blockDim.x)
            out[(size_t)seq * ldo + (size_t)q_head0 * 128 + i] = __float2bfloat16(0.0f);
        return;
    }

    const uint32_t smem_base = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t ring = smem_base + (uint32_t)warp * kWarpSmem;
    const int *bt = block_tables + (size_t)seq * max_blocks_per_seq;
    const size_t row_elems = (size_t)num_kv_heads * 128;
    const size_t head_off = (size_t)kv_head * 128;
    const int num_tiles = (seq_len + kTile - 1) / kTile;
    const int my_tiles = num_tiles > warp ? (num_tiles - warp + kWarps - 1) / kWarps : 0;

    // ---- producer: this warp's tile i (global tile index warp + 4 i) into ring slot i % kStages ----
    auto load_tile = [&](int i) {
        const int tile = warp + kWarps * i;
        const uint32_t kdst = ring + (uint32_t)(i % kStages) * (2 * kTileBytes);
        const uint32_t vdst = kdst + kTileBytes;
        const int c = lane & 15;                        // 16-byte chunk of the row
        if (PAGE_ALIGNED) {
            const int t0 = tile * kTile;
            const int page = t0 / block_size;
            const int blk = bt[page];
            const bool page_ok = blk >= 0;
            const int r0 = lane >> 4;
            size_t off = page_ok ? ((size_t)blk * block_size + (size_t)(t0 - page * block_size) + r0) * row_elems + head_off + c * 8 : 0;
            const int rows_left = seq_len - t0;         // rows r < rows_left exist
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int r = j * 2 + r0;
                const bool valid = page_ok && r < rows_left;
                const size_t o = valid ? off : 0;
                cp_async16_zfill(kdst + tile_off(r, c), key_cache + o, valid);
                cp_async16_zfill(vdst + tile_off(r, c), value_cache + o, valid);
                off += 2 * row_elems;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int r = j * 2 + (lane >> 4);          // row of the tile
                const int t = tile * kTile + r;
                int blk = -1;
                if (t < seq_len) blk = bt[t / block_size];
                const bool valid = blk >= 0;
                const size_t base = valid ? ((size_t)blk * block_size + (size_t)(t % block_size)) * row_elems + head_off + c * 8 : 0;
                cp_async16_zfill(kdst + tile_off(r, c), key_cache + base, valid);
                cp_async16_zfill(vdst + tile_off(r, c), value_cache + base, valid);
            }
        }
    };

    float acc[16][4];                   // O accumulators: 16 dim-tiles of 8; [.][0..1] are rows g (valid), [2..3] rows g+8 (unused)
#pragma unroll
    for (int n = 0; n < 16; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
    float run_max = -INFINITY, run_sum = 0.0f;

#pragma unroll
    for (int i = 0; i < kStages - 1; ++i) {
        if (i < my_tiles) load_tile(i);
        cp_async_commit();
    }

    // ---- Q fragments (loaded while the first K / V tiles are on their way): rows = query heads of the group (lanes with g >= group hold zeros) ----
    uint32_t qa[8][2];
    {
        const __nv_bfloat16 *qp = query + (size_t)seq * ldq + (size_t)(q_head0 + g) * 128;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            qa[ks][0] = 0u;
            qa[ks][1] = 0u;
            if (g < group) {
                qa[ks][0] = *reinterpret_cast<const uint32_t *>(qp + ks * 16 + tq * 2);
                qa[ks][1] = *reinterpret_cast<const uint32_t *>(qp + ks * 16 + 8 + tq * 2);
            }
        }
    }


    for (int i = 0; i < my_tiles; ++i) {
        if (i + kStages - 1 < my_tiles) load_tile(i + kStages - 1);
        cp_async_commit();
        cp_async_wait<kStages - 1>();        // this warp's tile i has landed (groups complete in order)
        __syncwarp();

        const int t0 = (warp + kWarps * i) * kTile;
        const uint32_t kbase = ring + (uint32_t)(i % kStages) * (2 * kTileBytes);
        const uint32_t vbase = kbase + kTileBytes;

        // ---- S = Q K^T for 16 tokens: two 8-token column tiles ----
        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            uint32_t kb[4];
            ldmatrix_x4(kbase + tile_off((lane & 7) + 8 * (lane >> 4), 2 * ks + ((lane >> 3) & 1)), kb);
            mma_bf16_16816(s0, qa[ks][0], 0u, qa[ks][1], 0u, kb[0], kb[1]);
            mma_bf16_16816(s1, qa[ks][0], 0u, qa[ks][1], 0u, kb[2], kb[3]);
        }
        // this lane holds, for query head g, the scores of tokens t0 + {2tq, 2tq+1, 8+2tq, 9+2tq}
        float sc[4] = {s0[0], s0[1], s1[0], s1[1]};
        float tmax = -INFINITY;
        const bool tile_page_ok = PAGE_ALIGNED ? bt[t0 / block_size] >= 0 : true;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int t = t0 + (e >> 1) * 8 + tq * 2 + (e & 1);
            const bool ok = PAGE_ALIGNED ? (tile_page_ok && t < seq_len) : (t < seq_len && bt[t / block_size] >= 0);
            sc[e] = ok ? sc[e] * scale : -INFINITY;
            tmax = fmaxf(tmax, sc[e]);
        }
        tmax = fmaxf(tmax, __shfl_xor_sync(0xFFFFFFFFu, tmax, 1));
        tmax = fmaxf(tmax, __shfl_xor_sync(0xFFFFFFFFu, tmax, 2));
        const float m_new = fmaxf(run_max, tmax);
        const float corr = (run_max == -INFINITY) ? 0.0f : __expf(run_max - m_new);
        float p[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) p[e] = (sc[e] == -INFINITY) ? 0.0f : __expf(sc[e] - m_new);
        run_sum = run_sum * corr + ((p[0] + p[1]) + (p[2] + p[3]));
        run_max = m_new;
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            acc[n][0] *= corr;
            acc[n][1] *= corr;
        }
        // ---- O += P V ----
        const uint32_t pa0 = pack_bf16x2(p[0], p[1]);
        const uint32_t pa2 = pack_bf16x2(p[2], p[3]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            uint32_t vb[4];
            ldmatrix_x4_trans(vbase + tile_off((lane & 7) + 8 * ((lane >> 3) & 1), 2 * j + (lane >> 4)), vb);
            mma_bf16_16816(acc[2 * j], pa0, 0u, pa2, 0u, vb[0], vb[1]);
            mma_bf16_16816(acc[2 * j + 1], pa0, 0u, pa2, 0u, vb[2], vb[3]);
        }
        __syncwarp();                        // every lane is done with this slot before it is refilled
    }
    cp_async_wait<0>();

    // ---- merge the four warps' partial results ----
    run_sum += __shfl_xor_sync(0xFFFFFFFFu, run_sum, 1);
    run_sum += __shfl_xor_sync(0xFFFFFFFFu, run_sum, 2);
    __syncthreads();                         // rings are dead: reuse shared memory for the partials
    float *part = reinterpret_cast<float *>(smem);              // [warp][head][130]: max, sum, 128 accumulators
    constexpr int kPart = 130;
    if (g < group) {
        float *mine = part + ((size_t)warp * 8 + g) * kPart;
        if (tq == 0) {
            mine[0] = run_max;
            mine[1] = run_sum;
        }
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            mine[2 + n * 8 + tq * 2] = acc[n][0];
            mine[2 + n * 8 + tq * 2 + 1] = acc[n][1];
        }
    }
    __syncthreads();
    if (q_packed != nullptr) {
        // the o projection's operand directly: 16-element blocks of the bf16-rounded result through the
        // activation quantiser (same bytes as the bf16 output followed by the stand-alone quantiser)
        const int hidden = num_kv_heads * group * 128;
        for (int task = threadIdx.x; task < group * 8; task += blockDim.x) {
            const int h = task >> 3, b = task & 7;
            float m = -INFINITY;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) m = fmaxf(m, part[((size_t)w * 8 + h) * kPart]);
            float e[kWarps], den = 0.0f;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const float *pw = part + ((size_t)w * 8 + h) * kPart;
                e[w] = (pw[0] == -INFINITY) ? 0.0f : __expf(pw[0] - m);
                den += e[w] * pw[1];
            }
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                float num = 0.0f;
#pragma unroll
                for (int w = 0; w < kWarps; ++w) num += e[w] * part[((size_t)w * 8 + h) * kPart + 2 + b * 16 + j];
                v[j] = __bfloat162float(__float2bfloat16(num / (den + 1e-9f)));
            }
            uint32_t lo, hi;
            const uint32_t sf = quantize_block16(v, q_inv_in, lo, hi);
            const int col = (q_head0 + h) * 128 + b * 16;
            *reinterpret_cast<uint2 *>(q_packed + (size_t)seq * (hidden / 2) + (col >> 1)) = make_uint2(lo, hi);
            const int kb = col >> 4, rem = seq & 127;
            q_sf[((((size_t)(seq >> 7) * q_sf_chunks + (kb >> 2)) * 32 + (rem & 31)) * 4 + (rem >> 5)) * 4 + (kb & 3)] = (uint8_t)sf;
        }
        return;
    }
    for (int idx = threadIdx.x; idx < group * 128; idx += blockDim.x) {
        const int h = idx >> 7, d = idx & 127;
        float m = -INFINITY;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) m = fmaxf(m, part[((size_t)w * 8 + h) * kPart]);
        float num = 0.0f, den = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const float *pw = part + ((size_t)w * 8 + h) * kPart;
            const float e = (pw[0] == -INFINITY) ? 0.0f : __expf(pw[0] - m);
            num += e * pw[2 + d];
            den += e * pw[1];
        }
        out[(size_t)seq * ldo + (size_t)(q_head0 + h) * 128 + d] = __float2bfloat16(num / (den + 1e-9f));
    }
}

bool launch_paged_decode_attention_mma(__nv_bfloat16 *out, int ldo, const __nv_bfloat16 *query, int ldq,
                                       const __nv_bfloat16 *key_cache, const __nv_bfloat16 *value_cache,
                                       const int *block_tables, const int *seq_lens, int num_seqs, int num_q_heads,
                                       int num_kv_heads, int head_dim, int block_size, int max_blocks_per_seq,
                                       cudaStream_t st, uint8_t *q_packed, uint8_t *q_sf, float q_input_scale) {
    if (head_dim != 128 || num_kv_heads <= 0 || num_q_heads % num_kv_heads != 0) return false;
    const int group = num_q_heads / num_kv_heads;
    if (group > 8 || (ldq % 2) != 0) return false;
    if ((((uintptr_t)key_cache | (uintptr_t)value_cache) & 15) != 0 || (((uintptr_t)query) & 3) != 0) return false;
    if (num_seqs <= 0) return true;
    if (q_packed != nullptr && (q_sf == nullptr || !(q_input_scale > 0.0f) || (((uintptr_t)q_packed) & 7) != 0)) return false;
    const int q_sf_chunks = num_q_heads * head_dim / 64;
    const float q_inv_in = q_packed != nullptr ? 1.0f / q_input_scale : 0.0f;
    static PerDevice<bool> configured;
    const cudaError_t ready = once_per_device(configured, [] {
        const cudaError_t e = cudaFuncSetAttribute(paged_decode_attention_mma_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnSmem);
        if (e != cudaSuccess) return e;
        return cudaFuncSetAttribute(paged_decode_attention_mma_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnSmem);
    });
    if (ready != cudaSuccess) return false;
    GLMASR_PREFER_MAX_SMEM(paged_decode_attention_mma_kernel<true>);
    GLMASR_PREFER_MAX_SMEM(paged_decode_attention_mma_kernel<false>);
    const float scale = 1.0f / sqrtf((float)head_dim);
    dim3 grid(num_kv_heads, num_seqs);
    if (block_size % kTile == 0)
        launch_chained(paged_decode_attention_mma_kernel<true>, grid, dim3(kWarps * 32), (size_t)kAttnSmem, st, out, ldo, query,
                       ldq, key_cache, value_cache, block_tables, seq_lens, num_kv_heads, group, block_size,
                       max_blocks_per_seq, scale, q_packed, q_sf, q_sf_chunks, q_inv_in);
    else
        launch_chained(paged_decode_attention_mma_kernel<false>, grid, dim3(kWarps * 32), (size_t)kAttnSmem, st, out, ldo, query,
                       ldq, key_cache, value_cache, block_tables, seq_lens, num_kv_heads, group, block_size,
                       max_blocks_per_seq, scale, q_packed, q_sf, q_sf_chunks, q_inv_in);
    return true;
}

// --------------------------------------------------------------------------------------------
// The same attention with what precedes it in a decode step folded in: RoPE on the new token's q and
// k heads, its K / V rows into the cache, attention over cached + 1 tokens.  A batch of a few sequences has kv_heads x
// num_seqs blocks of work -- four CTAs for one sequence -- each a serial walk over the context, so the context of a
// (sequence, kv head) is cut into `gridDim.x` contiguous shares, one CTA each, and the CTAs of a cluster merge their
// partial results through distributed shared memory.  One sequence, 300 tokens: rope + cache and attention were two
// launches of 3 + 9 us in the chain.  The new token's K / V row is put into the staged tile from the q|k|v buffer, so
// the cache write is off the critical path; lengths, block table and cached rows are asked for while the projection still
// runs (19 sequences: 13.3 -> 7.5 us).  A large batch takes it unsplit, one launch less (256 sequences: 2606 -> 2588 us a step).
// 16-token tiles inside one page (block_size % 16 == 0), head_dim 128.
// --------------------------------------------------------------------------------------------
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

__global__ void __launch_bounds__(kWarps * 32) paged_decode_split_kernel(
    __nv_bfloat16 *__restrict__ out, int ldo, const __nv_bfloat16 *__restrict__ qkv, int ld, int k_col, int v_col,
    const float *__restrict__ angles, const int64_t *__restrict__ slot_mapping, __nv_bfloat16 *key_cache,
    __nv_bfloat16 *value_cache, const int *__restrict__ block_tables, const int *__restrict__ seq_lens, int num_kv_heads,
    int group, int block_size, int max_blocks_per_seq, float scale, int early_cache, uint8_t *__restrict__ q_packed,
    uint8_t *__restrict__ q_sf, int q_sf_chunks, float q_inv_in) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ float merged[8 * 130];           // this CTA's result per head: max, sum, 128 accumulators
    pdl_launch_dependents();
    if (!early_cache) pdl_wait();
    const int split = blockIdx.x, splits = gridDim.x, kv_head = blockIdx.y, seq = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    const int seq_len = seq_lens[seq];
    const int q_head0 = kv_head * group;
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem) + (uint32_t)warp * kWarpSmem;
    const int *bt = block_tables + (size_t)seq * max_blocks_per_seq;
    const size_t row_elems = (size_t)num_kv_heads * 128;
    const size_t head_off = (size_t)kv_head * 128;
    const int num_tiles = (seq_len + kTile - 1) / kTile;
    const int per = (num_tiles + splits - 1) / splits;
    const int tile0 = split * per;
    const int tile_end = min(num_tiles, tile0 + per);
    const int mine = tile_end - tile0 - warp;
    const int my_tiles = mine > 0 ? (mine + kWarps - 1) / kWarps : 0;

    auto load_tile = [&](int i) {
        const int t0 = (tile0 + warp + kWarps * i) * kTile;
        const uint32_t kdst = ring + (uint32_t)(i % kStages) * (2 * kTileBytes);
        const uint32_t vdst = kdst + kTileBytes;
        const int c = lane & 15, r0 = lane >> 4;
        const int page = t0 / block_size;
        const int blk = bt[page];
        const bool page_ok = blk >= 0;
        size_t off = page_ok ? ((size_t)blk * block_size + (size_t)(t0 - page * block_size) + r0) * row_elems + head_off + c * 8 : 0;
        const int rows_left = seq_len - t0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int r = j * 2 + r0;
            const bool valid = page_ok && r < rows_left;
            const size_t o = valid ? off : 0;
            cp_async16_zfill(kdst + tile_off(r, c), key_cache + o, valid);
            cp_async16_zfill(vdst + tile_off(r, c), value_cache + o, valid);
            off += 2 * row_elems;
        }
    };
    float acc[16][4];
#pragma unroll
    for (int n = 0; n < 16; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
    float run_max = -INFINITY, run_sum = 0.0f;
#pragma unroll
    for (int i = 0; i < kStages - 1; ++i) {
        if (i < my_tiles) load_tile(i);
        cp_async_commit();
    }
    if (early_cache) pdl_wait();        // up to here: lengths, block table and cached rows, none of them the q|k|v projection's

    // q fragments, rotated in registers: a lane holds dims d and d + 64 of its head (k steps ks and ks + 4)
    uint32_t qa[8][2];
    const float *cs = angles + (size_t)seq * 128;
    {
        const __nv_bfloat16 *qp = qkv + (size_t)seq * ld + (size_t)(q_head0 + g) * 128;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int d = ks * 16 + h * 8 + tq * 2;
                qa[ks][h] = 0u;
                qa[ks + 4][h] = 0u;
                if (g < group) {
                    const uint32_t lo = *reinterpret_cast<const uint32_t *>(qp + d), hi = *reinterpret_cast<const uint32_t *>(qp + 64 + d);
                    const float2 c2 = *reinterpret_cast<const float2 *>(cs + d), s2 = *reinterpret_cast<const float2 *>(cs + 64 + d);
                    const float a0 = __uint_as_float(lo << 16), a1 = __uint_as_float(lo & 0xFFFF0000u);
                    const float b0 = __uint_as_float(hi << 16), b1 = __uint_as_float(hi & 0xFFFF0000u);
                    qa[ks][h] = pack_bf16x2(a0 * c2.x - b0 * s2.x, a1 * c2.y - b1 * s2.y);
                    qa[ks + 4][h] = pack_bf16x2(a0 * s2.x + b0 * c2.x, a1 * s2.y + b1 * c2.y);
                }
            }
    }
    // the new token's rows: the warp that owns the last tile rotates k and keeps both rows for that tile
    const int last_tile = num_tiles - 1;
    const bool own_new = my_tiles > 0 && last_tile == tile0 + warp + kWarps * (my_tiles - 1);
    uint32_t new_k[2] = {0u, 0u};
    uint2 new_v = make_uint2(0u, 0u);
    if (own_new) {
        const __nv_bfloat16 *row = qkv + (size_t)seq * ld;
        const __nv_bfloat16 *kp = row + k_col + head_off;
        const uint32_t lo = *reinterpret_cast<const uint32_t *>(kp + 2 * lane), hi = *reinterpret_cast<const uint32_t *>(kp + 64 + 2 * lane);
        new_v = *reinterpret_cast<const uint2 *>(row + v_col + head_off + 4 * lane);
        const float2 c2 = *reinterpret_cast<const float2 *>(cs + 2 * lane), s2 = *reinterpret_cast<const float2 *>(cs + 64 + 2 * lane);
        const float a0 = __uint_as_float(lo << 16), a1 = __uint_as_float(lo & 0xFFFF0000u);
        const float b0 = __uint_as_float(hi << 16), b1 = __uint_as_float(hi & 0xFFFF0000u);
        new_k[0] = pack_bf16x2(a0 * c2.x - b0 * s2.x, a1 * c2.y - b1 * s2.y);
        new_k[1] = pack_bf16x2(a0 * s2.x + b0 * c2.x, a1 * s2.y + b1 * c2.y);
        const size_t slot = (size_t)slot_mapping[seq] * row_elems + head_off;
        *reinterpret_cast<uint32_t *>(key_cache + slot + 2 * lane) = new_k[0];
        *reinterpret_cast<uint32_t *>(key_cache + slot + 64 + 2 * lane) = new_k[1];
        *reinterpret_cast<uint2 *>(value_cache + slot + 4 * lane) = new_v;
    }

    for (int i = 0; i < my_tiles; ++i) {
        if (i + kStages - 1 < my_tiles) load_tile(i + kStages - 1);
        cp_async_commit();
        cp_async_wait<kStages - 1>();
        __syncwarp();
        const int t0 = (tile0 + warp + kWarps * i) * kTile;
        const uint32_t kbase = ring + (uint32_t)(i % kStages) * (2 * kTileBytes);
        const uint32_t vbase = kbase + kTileBytes;
        if (own_new && i == my_tiles - 1) {
            const int r = (seq_len - 1) & (kTile - 1);
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(kbase + tile_off(r, lane >> 2) + (lane & 3) * 4), "r"(new_k[0]) : "memory");
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(kbase + tile_off(r, 8 + (lane >> 2)) + (lane & 3) * 4), "r"(new_k[1]) : "memory");
            asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(vbase + tile_off(r, lane >> 1) + (lane & 1) * 8), "r"(new_v.x), "r"(new_v.y) : "memory");
            __syncwarp();
        }
        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            uint32_t kb[4];
            ldmatrix_x4(kbase + tile_off((lane & 7) + 8 * (lane >> 4), 2 * ks + ((lane >> 3) & 1)), kb);
            mma_bf16_16816(s0, qa[ks][0], 0u, qa[ks][1], 0u, kb[0], kb[1]);
            mma_bf16_16816(s1, qa[ks][0], 0u, qa[ks][1], 0u, kb[2], kb[3]);
        }
        float sc[4] = {s0[0], s0[1], s1[0], s1[1]};
        float tmax = -INFINITY;
        const bool tile_page_ok = bt[t0 / block_size] >= 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int t = t0 + (e >> 1) * 8 + tq * 2 + (e & 1);
            sc[e] = tile_page_ok && t < seq_len ? sc[e] * scale : -INFINITY;
            tmax = fmaxf(tmax, sc[e]);
        }
        tmax = fmaxf(tmax, __shfl_xor_sync(0xFFFFFFFFu, tmax, 1));
        tmax = fmaxf(tmax, __shfl_xor_sync(0xFFFFFFFFu, tmax, 2));
        const float m_new = fmaxf(run_max, tmax);
        const float corr = (run_max == -INFINITY) ? 0.0f : __expf(run_max - m_new);
        float p[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) p[e] = (sc[e] == -INFINITY) ? 0.0f : __expf(sc[e] - m_new);
        run_sum = run_sum * corr + ((p[0] + p[1]) + (p[2] + p[3]));
        run_max = m_new;
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            acc[n][0] *= corr;
            acc[n][1] *= corr;
        }
        const uint32_t pa0 = pack_bf16x2(p[0], p[1]);
        const uint32_t pa2 = pack_bf16x2(p[2], p[3]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            uint32_t vb[4];
            ldmatrix_x4_trans(vbase + tile_off((lane & 7) + 8 * ((lane >> 3) & 1), 2 * j + (lane >> 4)), vb);
            mma_bf16_16816(acc[2 * j], pa0, 0u, pa2, 0u, vb[0], vb[1]);
            mma_bf16_16816(acc[2 * j + 1], pa0, 0u, pa2, 0u, vb[2], vb[3]);
        }
        __syncwarp();
    }
    cp_async_wait<0>();

    run_sum += __shfl_xor_sync(0xFFFFFFFFu, run_sum, 1);
    run_sum += __shfl_xor_sync(0xFFFFFFFFu, run_sum, 2);
    __syncthreads();
    float *part = reinterpret_cast<float *>(smem);              // [warp][head][130]
    constexpr int kPart = 130;
    if (g < group) {
        float *dst = part + ((size_t)warp * 8 + g) * kPart;
        if (tq == 0) {
            dst[0] = run_max;
            dst[1] = run_sum;
        }
#pragma unroll
        for (int n = 0; n < 16; ++n) *reinterpret_cast<float2 *>(dst + 2 + n * 8 + tq * 2) = make_float2(acc[n][0], acc[n][1]);
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < group * 128; idx += blockDim.x) {
        const int h = idx >> 7, d = idx & 127;
        float m = -INFINITY;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) m = fmaxf(m, part[((size_t)w * 8 + h) * kPart]);
        float num = 0.0f, den = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const float *pw = part + ((size_t)w * 8 + h) * kPart;
            const float e = (pw[0] == -INFINITY) ? 0.0f : __expf(pw[0] - m);
            num += e * pw[2 + d];
            den += e * pw[1];
        }
        if (splits == 1) {
            const __nv_bfloat16 v = __float2bfloat16(num / (den + 1e-9f));
            if (q_packed != nullptr) merged[h * 128 + d] = __bfloat162float(v);
            else out[(size_t)seq * ldo + (size_t)(q_head0 + h) * 128 + d] = v;
        } else {
            merged[h * kPart + 2 + d] = num;
            if (d == 0) {
                merged[h * kPart] = m;
                merged[h * kPart + 1] = den;
            }
        }
    }
    if (splits == 1) {
        if (q_packed == nullptr) return;
        // finished heads through the activation quantiser
        __syncthreads();
        const int hidden = num_kv_heads * group * 128;
        for (int task = threadIdx.x; task < group * 8; task += blockDim.x) {
            const int h = task >> 3, b = task & 7;
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = merged[h * 128 + b * 16 + j];
            uint32_t lo, hi;
            const uint32_t sf = quantize_block16(v, q_inv_in, lo, hi);
            const int col = (q_head0 + h) * 128 + b * 16;
            *reinterpret_cast<uint2 *>(q_packed + (size_t)seq * (hidden / 2) + (col >> 1)) = make_uint2(lo, hi);
            const int kb = col >> 4, rem = seq & 127;
            q_sf[((((size_t)(seq >> 7) * q_sf_chunks + (kb >> 2)) * 32 + (rem & 31)) * 4 + (rem >> 5)) * 4 + (kb & 3)] = (uint8_t)sf;
        }
        return;
    }
    cluster_sync_all();
    const uint32_t base = smem_u32(merged);
    for (int idx = split * (int)blockDim.x + threadIdx.x; idx < group * 128; idx += splits * (int)blockDim.x) {
        const int h = idx >> 7, d = idx & 127;
        float m = -INFINITY, num = 0.0f, den = 0.0f;
        float ms[8], ls[8], vs[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            ms[r] = -INFINITY, ls[r] = 0.0f, vs[r] = 0.0f;
            if (r < splits) {
                const uint32_t a = mapa_shared(base, (uint32_t)r) + (uint32_t)(h * kPart) * 4u;
                ms[r] = ld_cluster_f32(a);
                ls[r] = ld_cluster_f32(a + 4);
                vs[r] = ld_cluster_f32(a + 8 + 4 * d);
            }
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) m = fmaxf(m, ms[r]);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float e = ms[r] == -INFINITY ? 0.0f : __expf(ms[r] - m);
            num += e * vs[r];
            den += e * ls[r];
        }
        out[(size_t)seq * ldo + (size_t)(q_head0 + h) * 128 + d] = __float2bfloat16(num / (den + 1e-9f));
    }
    cluster_sync_all();          // nobody leaves while its results are being read
}

bool launch_paged_decode_split(__nv_bfloat16 *out, int ldo, const __nv_bfloat16 *qkv, int ld, int k_col, int v_col,
                               const float *angles, const int64_t *slot_mapping, __nv_bfloat16 *key_cache,
                               __nv_bfloat16 *value_cache, const int *block_tables, const int *seq_lens, int num_seqs,
                               int num_q_heads, int num_kv_heads, int head_dim, int block_size, int max_blocks_per_seq,
                               int max_len, cudaStream_t st, bool early_cache, uint8_t *q_packed, uint8_t *q_sf, float q_input_scale) {
    if (head_dim != 128 || num_kv_heads <= 0 || num_q_heads % num_kv_heads != 0 || num_seqs <= 0 || angles == nullptr) return false;
    const int group = num_q_heads / num_kv_heads;
    if (group > 8 || (ld % 8) != 0 || (k_col % 8) != 0 || (v_col % 8) != 0 || (block_size % kTile) != 0) return false;
    if ((((uintptr_t)key_cache | (uintptr_t)value_cache | (uintptr_t)qkv) & 15) != 0) return false;
    if (q_packed != nullptr && (q_sf == nullptr || !(q_input_scale > 0.0f) || (((uintptr_t)q_packed) & 7) != 0)) return false;
    // unsplit on a chip that it leaves half empty, the serial walk with RoPE in front of it is the longer way round: a W4A4
    // step of 1 / 9 sequences, 16 query and 4 kv heads, takes 1745 / 1823 us with it and 1710 / 1788 us with two launches,
    // of 19 sequences 1813 and 1817 us, of 40 / 100 sequences 1807 / 1896 and 1857 / 1963 us
    if (q_packed != nullptr && num_seqs * num_kv_heads <= num_sms() / 2) return false;
    // three 64 KB CTAs fit an SM: up to three per SM in one wave, at least two tiles for every CTA.  A result that is quantised is not
    // split: another order of its sums moves values across e2m1 rounding boundaries, and a chain of such layers amplifies it.
    const int tiles = (max_len + kTile - 1) / kTile;
    int splits = 1;
    while (q_packed == nullptr && splits < 8 && num_seqs * num_kv_heads * splits * 2 <= 3 * num_sms() && tiles >= splits * 4) splits *= 2;
    static PerDevice<bool> configured;
    if (once_per_device(configured, [] { return cudaFuncSetAttribute(paged_decode_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnSmem); }) != cudaSuccess)
        return false;
    GLMASR_PREFER_MAX_SMEM(paged_decode_split_kernel);
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(splits, num_kv_heads, num_seqs);
    cfg.blockDim = dim3(kWarps * 32);
    cfg.dynamicSmemBytes = kAttnSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    const cudaError_t launched =
        cudaLaunchKernelEx(&cfg, paged_decode_split_kernel, out, ldo, qkv, ld, k_col, v_col, angles, slot_mapping, key_cache,
                           value_cache, block_tables, seq_lens, num_kv_heads, group, block_size, max_blocks_per_seq,
                           1.0f / sqrtf((float)head_dim), early_cache && pdl_enabled() ? 1 : 0, q_packed, q_sf,
                           num_q_heads * head_dim / 64, q_packed != nullptr ? 1.0f / q_input_scale : 0.0f);
    if (launched != cudaSuccess) (void)cudaGetLastError();       // refused: the caller goes on to the separate launches
    return launched == cudaSuccess;
}

}  // namespace glmasr
