// out[M, sum N_s] = epilogue(x[M, K] * concat_s(W_s[N_s, K])^T), bf16 operands, for M up to a few hundred rows: the
// prompt of one clip, the encoder on one short clip, the W4A16 decode of a batch.
//
// These shapes have few output tiles (173 rows x 2048 columns: thirty-two 128 x 128 ones) and a long K, and one SM pulls
// operands at about 60 bytes a clock whatever the rest of the chip does, so a GEMM that gives a tile to a CTA takes
// as long as one CTA's walk over K: 25 us for K = 6144, most of the chip idle.  Here
//   * the weight rows are the 128 accumulator lanes and the tokens (up to 256) the accumulator columns: a decode batch of
//     20 pays for 32 token columns instead of 128 token rows;
//   * K is cut over a cluster of up to eight CTAs, each with its own ring of TMA stages and fp32 accumulator; the partial
//     tiles meet in distributed shared memory, every CTA of the cluster adding (in rank order) and finishing every
//     splits-th token.  Two CTAs can share an SM;
//   * weights that no running kernel writes are requested before the wait for the preceding kernel.
// Split and tile are chosen by expected time (choose_cluster_gemm).  Bound: the L2 -> SM rate for the operands, the round
// trips of the ring (1.3 us each with all SMs loading), then the fixed latency of a launch.
#include "gemm_cluster.cuh"

#include <cuda_bf16.h>

#include "gemm_device.cuh"
#include "gemm_umma.cuh"
#include "ptx.cuh"
#include "runtime.cuh"

namespace glmasr {

static constexpr int kCgThreads = 256;
static constexpr int kCgHeader = 1024;              // barriers, flags; keeps the stages 1024-byte aligned
static constexpr int kCgWBytes = 128 * 128;         // 128 weight rows x 64 elements

__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// A wait ran out: loads and MMAs in flight end before their memory is reused or given up.  The MMA warp alone calls it, ahead of
// the barrier that holds all others: a test of the flag by every thread further down made each launch 0.25 us longer.
__device__ __forceinline__ void let_copies_land() {
#pragma unroll 1
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
}

// CMAX: largest cluster this instance serves; 16 / CMAX items are in flight per thread in the reduction.
template <int CMAX>
__global__ void __launch_bounds__(kCgThreads, 2) cluster_gemm_kernel(const __grid_constant__ ClusterGemmParams p) {
    extern __shared__ uint8_t cg_raw[];
    // header at the first 1024-byte boundary: [0,64) full, [64,128) empty, [128] done, [136] tmem, [140] abort
    const uint32_t raw = smem_u32(cg_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *hdr = cg_raw + (base - raw);
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(hdr + 136);
    volatile int *abort_word = reinterpret_cast<volatile int *>(hdr + 140);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x;                    // K share = position in the cluster
    const int w_tile = blockIdx.y, tok0 = blockIdx.z * p.n_tok;
    const int S = p.stages;
    const uint32_t stage_bytes = kCgWBytes + (uint32_t)p.n_tok * 128u;
    const uint32_t ring = base + kCgHeader;
    auto full = [&](int s) { return base + 8u * s; };
    auto empty = [&](int s) { return base + 64u + 8u * s; };
    const uint32_t done = base + 128;
    uint32_t cols = 32;
    while ((int)cols < p.n_tok) cols <<= 1;
    const bool silu = p.epi == EPI_SILU_GATE;
    // this CTA's k blocks
    const int kb_lo = (int)((long long)p.k_blocks * rank / p.splits), kb_hi = (int)((long long)p.k_blocks * (rank + 1) / p.splits);
    const int n_kb = kb_hi - kb_lo;
    // weight tile -> tensor, row, output column
    int seg = 0, wt = w_tile, col0 = 0;
    if (!silu)
        while (seg < p.num_segs - 1 && wt >= p.seg_tiles[seg]) {
            wt -= p.seg_tiles[seg];
            col0 += p.seg_rows[seg];
            ++seg;
        }
    const int row0 = silu ? wt * 64 : wt * 128;
    col0 += row0;

    if (!p.late_trigger) pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        mbar_init(done, 1);
        *abort_word = 0;
        fence_mbar_init();
        fence_proxy_async_smem();
    }
    if (warp == 1) {
        tmem_alloc(base + 136, cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // Both roles run warp-uniform with one elected lane issuing: in a divergent single-lane loop the operand addresses leave
    // the uniform registers and a stage takes 0.1 us longer.
    if (warp == 0) {
        // ---- producer ----
        const bool leader = elect_one();
        const CUtensorMap *tw = &p.tm_w[seg];
        auto load_w = [&](int kb, int s) {
            const uint32_t dst = ring + (uint32_t)s * stage_bytes;
            const int x = (kb_lo + kb) * 64;
            mbar_expect_tx(full(s), stage_bytes);
            tma_load_2d(dst, tw, full(s), x, row0);
            if (silu) tma_load_2d(dst + kCgWBytes / 2, &p.tm_w[1], full(s), x, row0);
        };
        const int pre = p.early_weights ? min(n_kb, S) : 0;
        for (int kb = 0; kb < pre; ++kb)
            if (leader) load_w(kb, kb);
        pdl_wait();
        if (p.late_trigger) pdl_launch_dependents();
        int s = 0;
        uint32_t ph = 1;
        for (int kb = 0; kb < n_kb; ++kb) {
            if (!mbar_wait_warp(empty(s), ph, abort_word, ST_TIMEOUT_PRODUCER)) break;      // the MMA warp fails with it
            if (leader) {
                if (kb >= pre) load_w(kb, s);
                tma_load_2d(ring + (uint32_t)s * stage_bytes + kCgWBytes, &p.tm_x, full(s), (kb_lo + kb) * 64, tok0);
            }
            if (++s == S) s = 0, ph ^= 1u;
        }
    } else if (warp == 1) {
        // ---- MMA issuer ----
        const bool leader = elect_one();
        const uint32_t idesc = idesc_bf16(128, p.n_tok);
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int kb = 0; kb < n_kb; ++kb) {
            ok = mbar_wait_warp(full(s), ph, abort_word, ST_TIMEOUT_MMA);
            if (!ok) break;
            tc_fence_after();
            const uint32_t a = ring + (uint32_t)s * stage_bytes;
            const uint64_t ad = smem_desc_sw128(a), bd = smem_desc_sw128(a + kCgWBytes);
            if (leader) {
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_bf16(tmem, ad + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                umma_commit(empty(s));
            }
            if (++s == S) s = 0, ph ^= 1u;
        }
        if (leader) umma_commit(done);
        // this warp polls, the others sleep at the barrier below
        const bool fin = mbar_wait_warp(done, 0, abort_word, ST_TIMEOUT_EPILOGUE);
        if (__builtin_expect(!(fin && ok), 0)) let_copies_land();
    }
    pdl_wait();                         // residual, bias and out belong to the preceding kernels until here
    __syncthreads();                    // the ring is dead: every load of it has been consumed by a completed MMA
    tc_fence_after();
    // accumulator -> shared memory as [token][128 weight rows] fp32 (a warp stores 32 consecutive rows of a token)
    float *part = reinterpret_cast<float *>(cg_raw + (ring - raw));
    {
        const int quad = warp & 3;
        const uint32_t t_row = tmem + ((uint32_t)(quad * 32) << 16);
        for (int c = (warp >> 2) * 16; c < p.n_tok; c += 32) {
            uint32_t r[16];
            tmem_ld_x16(t_row + (uint32_t)c, r);
            tmem_ld_wait();
            float *dst = part + (size_t)c * 128 + quad * 32 + lane;
#pragma unroll
            for (int i = 0; i < 16; ++i) dst[i * 128] = __uint_as_float(r[i]);
        }
    }
    tc_fence_before();
    if (p.splits > 1) cluster_sync_all();
    else __syncthreads();

    // every splits-th token is this CTA's: add the shares in rank order, finish four columns per thread.  The remote loads
    // are what this phase waits for, so a thread has 16 of them (256 bytes) in flight.
    const int n_here = min(p.n_tok, p.M - tok0);
    const int mine = n_here > rank ? (n_here - rank + p.splits - 1) / p.splits : 0;
    const uint32_t part_addr = smem_u32(part);
    const int quads = silu ? 16 : 32;
    const int n_cols = min(silu ? 64 : 128, p.seg_rows[seg] - row0);
    const int items = mine * quads;
    constexpr int U = CMAX == 1 ? 8 : 16 / CMAX;
    const bool vec_out = (p.ldo & 3) == 0 && (col0 & 3) == 0 && (((uintptr_t)p.out | (uintptr_t)p.residual) & 7) == 0;
    for (int i0 = threadIdx.x; i0 < items; i0 += kCgThreads * U) {
        float4 pv[U][CMAX];
#pragma unroll
        for (int h = 0; h < (silu ? 2 : 1); ++h) {
            float4 sum[U];
#pragma unroll
            for (int e = 0; e < U; ++e) {
                const int i = i0 + e * kCgThreads;
                const int tok = rank + p.splits * (i / quads);
                const uint32_t off = part_addr + (uint32_t)(tok * 128 + 4 * (i % quads)) * 4u + (uint32_t)h * 256u;
#pragma unroll
                for (int r = 0; r < CMAX; ++r)
                    pv[e][r] = (i < items && r < p.splits) ? ld_cluster_f32x4(CMAX == 1 ? off : mapa_shared(off, (uint32_t)r))
                                                           : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (int e = 0; e < U; ++e) {
                sum[e] = pv[e][0];
#pragma unroll
                for (int r = 1; r < CMAX; ++r) {
                    sum[e].x += pv[e][r].x;
                    sum[e].y += pv[e][r].y;
                    sum[e].z += pv[e][r].z;
                    sum[e].w += pv[e][r].w;
                }
            }
            if (silu && h == 0) {       // gate: kept in this CTA's own tile (nobody else reads these tokens)
#pragma unroll
                for (int e = 0; e < U; ++e) {
                    const int i = i0 + e * kCgThreads;
                    if (i < items) reinterpret_cast<float4 *>(part)[(rank + p.splits * (i / quads)) * 32 + i % quads] = sum[e];
                }
                continue;
            }
#pragma unroll
            for (int e = 0; e < U; ++e) {
                const int i = i0 + e * kCgThreads;
                if (i >= items) continue;
                const int tok = rank + p.splits * (i / quads), c = 4 * (i % quads);
                if (c >= n_cols) continue;
                const size_t at = (size_t)(tok0 + tok) * p.ldo + col0 + c;
                float v[4] = {sum[e].x, sum[e].y, sum[e].z, sum[e].w};
                const int n = min(4, n_cols - c);
                if (silu) {
                    const float4 g4 = reinterpret_cast<float4 *>(part)[tok * 32 + i % quads];
                    const float g[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[j] = silu_gate(bf16_round(g[j]), bf16_round(v[j]));
                } else {
                    float bias[4] = {0.0f, 0.0f, 0.0f, 0.0f}, res[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                    if (p.bias != nullptr) {
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (j < n) bias[j] = __bfloat162float(p.bias[col0 + c + j]);
                    }
                    if (p.epi == EPI_RESIDUAL) {
                        if (vec_out && n == 4) {
                            const uint2 w = *reinterpret_cast<const uint2 *>(p.residual + at);
                            res[0] = __uint_as_float(w.x << 16), res[1] = __uint_as_float(w.x & 0xFFFF0000u);
                            res[2] = __uint_as_float(w.y << 16), res[3] = __uint_as_float(w.y & 0xFFFF0000u);
                        } else {
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (j < n) res[j] = __bfloat162float(p.residual[at + j]);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (p.epi == EPI_RESIDUAL) {
                            // bf16(bf16(bf16(acc) + bias) + residual), the middle step only with a bias
                            v[j] = bf16_round(v[j]);
                            if (p.bias != nullptr) v[j] = bf16_round(v[j] + bias[j]);
                            v[j] += res[j];
                        } else {
                            v[j] += bias[j];
                            if (p.epi == EPI_GELU) v[j] = gelu_tanh(v[j]);
                        }
                    }
                }
                if (vec_out && n == 4) {
                    const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
                    *reinterpret_cast<uint2 *>(p.out + at) =
                        make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (j < n) p.out[at + j] = __float2bfloat16(v[j]);
                }
            }
        }
    }
    if (p.splits > 1) cluster_sync_all();       // nobody leaves while its shares are being read
    else __syncthreads();
    if (threadIdx.x == 0 && *abort_word != 0 && p.status != nullptr) atomicCAS(p.status, 0, *abort_word);
    if (warp == 1) tmem_dealloc(tmem, cols);
}

static size_t cg_smem_bytes(int n_tok, int stages) {
    int body = stages * (kCgWBytes + n_tok * 128);
    if (body < n_tok * 512) body = n_tok * 512;             // the partial tile takes the ring's place
    return 1024 + kCgHeader + (size_t)body;
}

static void fill_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *attr, dim3 grid, size_t smem, cudaStream_t st) {
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kCgThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = grid.x;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
}

typedef void (*ClusterGemmKernel)(ClusterGemmParams);
static ClusterGemmKernel cg_kernel(int splits) {
    return splits == 1 ? cluster_gemm_kernel<1> : (splits <= 4 ? cluster_gemm_kernel<4> : cluster_gemm_kernel<8>);
}

static cudaError_t cg_ready() {
    static PerDevice<bool> ready;
    return once_per_device(ready, [] {
        for (int c : {1, 4, 8}) {
            cudaError_t e = cudaFuncSetAttribute(cg_kernel(c), cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(cg_kernel(c), cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    });
}

// Clusters of `splits` CTAs that the device holds at once at this shared-memory size (graphics processing clusters have
// 16 to 20 SMs here, so it is less than 148 * 2 / splits), 0 when it holds none; asked once per pair and device.
struct ClustersKnown {
    int n[9][16];                   // 0: not asked yet, -1: none
};
static int cg_max_clusters(ClustersKnown &known, int splits, size_t smem) {
    const int slot = (int)(smem >> 14) & 15;
    int &v = known.n[splits][slot];
    if (v == 0) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[2];
        fill_config(cfg, attr, dim3(splits, 64, 1), (size_t)(slot + 1) << 14, nullptr);
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, cg_kernel(splits), &cfg) != cudaSuccess || n < 1) {
            (void)cudaGetLastError();
            n = -1;
        }
        v = n;
    }
    return v > 0 ? v : 0;
}

// Times in ns, fitted to 471 launches of this kernel on a B200 (sixteen shapes of K 384 to 6144 and 512 to 8192 columns, 1 to 512
// rows, chains of launches, weights not in L2; standard deviation 7 %, the short K = 384 up to 26 % too high): a fixed 2.9 us,
// then the slower of the operand stream -- 190 bytes per ns and SM -- and the ring's round trips of 1.2 us, then the shares'
// way through distributed shared memory, 2.7 TB/s for the whole chip, or the one accumulator's through the CTA's own.
double choose_cluster_gemm(ClusterGemmParams &p, int w_tiles, int num_sms) {
    if (p.M < 1 || p.M > kClusterMaxRows || p.k_blocks < 1 || w_tiles < 1) return 0.0;
    if (cg_ready() != cudaSuccess) return 0.0;
    static PerDevice<ClustersKnown> per_device;
    ClustersKnown *known = per_device.here();
    if (known == nullptr) return 0.0;
    p.w_tiles = w_tiles;
    double best = 1e30;
    for (int tt = (p.M + 255) / 256; tt <= (p.M + 63) / 64; ++tt) {
        const int n_tok = ((p.M + tt - 1) / tt + 15) / 16 * 16;
        if ((p.M + n_tok - 1) / n_tok != tt) continue;
        const int stage = kCgWBytes + n_tok * 128;
        // a ring of about 100 KB: two CTAs share an SM, or this kernel's first loads the predecessor's last ones
        int stages = (100 * 1024) / stage;
        stages = stages > 8 ? 8 : (stages < 2 ? 2 : stages);
        const size_t smem = cg_smem_bytes(n_tok, stages);
        for (int c = 1; c <= 8 && (c == 1 || c * 2 <= p.k_blocks); ++c) {
            const int clusters = w_tiles * tt;
            const int room = cg_max_clusters(*known, c, smem);
            if (room == 0) continue;
            const double waves = (clusters + room - 1) / room;
            const int per_sm = smem <= 113 * 1024 ? 2 : 1;
            const double share = clusters * c > num_sms && per_sm == 2 ? 2.0 : 1.0;
            const int resident = clusters * c < num_sms * per_sm ? clusters * c : num_sms * per_sm;
            const int kb = (p.k_blocks + c - 1) / c;
            const double stream = kb * stage * share / 190.0, trips = (kb + stages - 1) / stages * 1200.0;
            double ns = waves * (stream > trips ? stream : trips) + 2900.0;
            ns += waves * (c > 1 ? 1630.0 + n_tok * 512.0 * resident / 2700.0 : n_tok * 22.0 * share);
            if (ns < best) best = ns, p.splits = c, p.n_tok = n_tok, p.token_tiles = tt, p.stages = stages;
        }
    }
    return best < 1e29 ? best : 0.0;
}

cudaError_t launch_cluster_gemm(const ClusterGemmParams &p, cudaStream_t st) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    fill_config(cfg, attr, dim3(p.splits, p.w_tiles, p.token_tiles), cg_smem_bytes(p.n_tok, p.stages), st);
    return cudaLaunchKernelEx(&cfg, cg_kernel(p.splits), p);
}

}  // namespace glmasr
