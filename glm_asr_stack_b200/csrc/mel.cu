// Log-mel front end (reference: mel_spectrogram, Infer-engine/cuda/mel.cu:111-294), batched over windows.
//
// Per 16 kHz window: n_frames = clamp(ceil(samples / 160), 1, 3000) frames of 400 samples centred on
// f * 160 (zero outside the signal), periodic Hann window, 400-point real DFT (bins 0..200), power, the
// 201 x 128 mel filterbank (given transposed, as the engine loads it), log10(p + 1e-10), clamp to
// (window maximum - 8), (v + 4) / 4, bf16.
//
// The reference runs five launches and a cuFFT call per window, one window at a time.  Here a whole batch
// of windows is two launches:
//   mel_power_kernel      grid (frame tiles, windows): a CTA stages the tile's samples in shared memory,
//                         applies the window and evaluates the DFT directly against a 400-entry twiddle table, folded
//                         twice: x[t] +- x[400 - t] (cosine and sine have that symmetry) leaves taps 0..200, and the
//                         sums over even and odd taps give bin k as their sum and bin 200 - k as their difference, a
//                         quarter of the multiply-adds and shorter sums.  A thread has two bins (and their mirror
//                         images) of 8 frames.  Then the power spectrum times the filterbank in the reference's
//                         summation order (16 frames per filter value read), log10, the fp32 result to scratch and the
//                         tile's maximum to the window's maximum (atomic).  Bound: shared-memory reads and
//                         multiply-adds of the DFT in balance, little else.  Unfolded, a bin a thread and 32 frames a
//                         CTA it took 1750 us for sixteen 30 s windows and 196 us for one of 3.7 s, now 383 and 40;
//   mel_normalize_kernel  clamp, affine map, bf16, written mel-major [128, n_frames] like the reference or
//                         time-major [n_frames, 128] (what the encoder's convolution-as-GEMM reads).
// The window maximum is the maximum over the WHOLE window.  The reference's second reduction pass
// (final_max_kernel, mel.cu:195-206) reduces inside each warp but lets thread 0 alone write, so it returns
// the maximum of one eighth of the block maxima; that is a defect, not a definition, and is not reproduced.
// fp32 throughout, like the reference; results agree with it to the rounding of a different DFT
// factorisation (compared within one bf16 unit in the tests).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include <type_traits>

#include "../../include/glmasr_fp4.h"
#include "runtime.cuh"

namespace glmasr {

constexpr int kFft = 400, kHop = 160, kMels = 128, kBins = 201, kMaxFrames = 3000;
constexpr int kTileFrames = 16;                                    // frames per CTA
constexpr int kTileSamples = (kTileFrames - 1) * kHop + kFft;      // 2800
constexpr int kMelThreads = 128;
constexpr int kSlots = 51;                                         // threads per 8 frames: bins i and i + 51 of 0..100
constexpr int kRow = kTileFrames + 4;                              // floats per tap or bin: 16-byte rows, spread over the banks

enum : int { WS_MEL_LOG = 35, WS_MEL_MAX = 36 };                   // private workspace slots of this file

struct MelSmem {
    float sum[kBins][kRow], dif[kBins][kRow];     // windowed x[t] + x[400 - t], x[t] - x[400 - t]
    float power[kBins][kRow];                     // first the tile's raw samples (kTileSamples floats), then the power spectrum
    float2 tw[kFft];                              // (cos, sin)(2 pi j / 400)
    float hann[kFft];
    float red[kMelThreads / 32];
};
static_assert(kTileSamples <= kBins * kRow, "the raw samples of a tile are staged in the power array");
static_assert(kMelThreads == 64 * (kTileFrames / 8) && kMelThreads == kMels, "thread = (slot, 8 frames), then thread = mel bin");

__device__ __forceinline__ void atomic_max_float(float *addr, float v) {
    // the cell starts as 0xFFFFFFFF: below every float in both orders used here
    if (v >= 0.0f) atomicMax(reinterpret_cast<int *>(addr), __float_as_int(v));
    else atomicMin(reinterpret_cast<unsigned int *>(addr), __float_as_uint(v));
}

__global__ void __launch_bounds__(kMelThreads) mel_power_kernel(const float *__restrict__ pcm, long long pcm_stride,
                                                                const int *__restrict__ num_samples,
                                                                const float *__restrict__ filters_t,
                                                                float *__restrict__ logmel, float *__restrict__ win_max) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    MelSmem &s = *reinterpret_cast<MelSmem *>(smem_raw);
    pdl_launch_dependents();
    pdl_wait();
    const int w = blockIdx.y, tid = threadIdx.x;
    const int ns = num_samples[w];
    int n_frames = (ns + kHop - 1) / kHop;
    n_frames = n_frames < 1 ? 1 : (n_frames > kMaxFrames ? kMaxFrames : n_frames);
    const int f0 = blockIdx.x * kTileFrames;
    if (f0 >= n_frames) return;
    const float *x = pcm + (size_t)w * (size_t)pcm_stride;

    // twiddles, the window, and the tile's samples (coalesced; zero outside the signal)
    float *raw = &s.power[0][0];
    const int s0 = f0 * kHop - kFft / 2;                 // first sample of the tile
    for (int j = tid; j < kFft; j += kMelThreads) {
        float sn, cs;
        sincospif((float)j * (2.0f / kFft), &sn, &cs);
        s.tw[j] = make_float2(cs, sn);
        // periodic Hann window as the reference evaluates it (mel.cu:118: the argument in double, cosf of its float)
        s.hann[j] = 0.5f * (1.0f - cosf((float)(2.0 * 3.14159265358979323846 * j / kFft)));
    }
    for (int i = tid; i < kTileSamples; i += kMelThreads) {
        const int idx = s0 + i;
        raw[i] = (idx >= 0 && idx < ns) ? x[idx] : 0.0f;
    }
    __syncthreads();
    for (int f = 0; f < kTileFrames; ++f) {              // lanes over t: the frames overlap, 160 samples apart
        const bool live = f0 + f < n_frames;
        for (int t = tid; t < kBins; t += kMelThreads) {
            const float a = live ? raw[f * kHop + t] * s.hann[t] : 0.0f;
            const bool paired = t != 0 && t != kFft / 2;
            const float b = live && paired ? raw[f * kHop + kFft - t] * s.hann[kFft - t] : 0.0f;
            s.sum[t][f] = a + b;
            s.dif[t][f] = paired ? a - b : 0.0f;         // the sine is zero at the unpaired taps
        }
    }
    __syncthreads();

    const int slot = tid & 63, fg = (tid >> 6) * 8;
    if (slot < kSlots) {
        // [bin][even / odd taps][frame]
        float re[2][2][8], im[2][2][8];
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int i = 0; i < 8; ++i) re[b][0][i] = re[b][1][i] = im[b][0][i] = im[b][1][i] = 0.0f;
        const int k0 = slot, k1 = slot + kSlots;         // k1 = 101 (a mirror image of 99) is computed and not stored
        int j0 = 0, j1 = 0;                              // (k * t) mod 400
        auto tap = [&](int t, auto odd) {
            constexpr int o = decltype(odd)::value;
            const float2 c0 = s.tw[j0], c1 = s.tw[j1];
            const float4 sa = *reinterpret_cast<const float4 *>(&s.sum[t][fg]), sb = *reinterpret_cast<const float4 *>(&s.sum[t][fg + 4]);
            const float4 da = *reinterpret_cast<const float4 *>(&s.dif[t][fg]), db = *reinterpret_cast<const float4 *>(&s.dif[t][fg + 4]);
            const float sv[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
            const float dv[8] = {da.x, da.y, da.z, da.w, db.x, db.y, db.z, db.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                re[0][o][i] = fmaf(sv[i], c0.x, re[0][o][i]);
                im[0][o][i] = fmaf(dv[i], c0.y, im[0][o][i]);     // its sign does not matter for the power
                re[1][o][i] = fmaf(sv[i], c1.x, re[1][o][i]);
                im[1][o][i] = fmaf(dv[i], c1.y, im[1][o][i]);
            }
            j0 += k0;
            if (j0 >= kFft) j0 -= kFft;
            j1 += k1;
            if (j1 >= kFft) j1 -= kFft;
        };
#pragma unroll 2
        for (int t = 0; t < kFft / 2; t += 2) {
            tap(t, std::integral_constant<int, 0>());
            tap(t + 1, std::integral_constant<int, 1>());
        }
        tap(kFft / 2, std::integral_constant<int, 0>());
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const int k = b == 0 ? k0 : k1;
            if (k > kFft / 4) break;
            float p[8], q[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float r1 = re[b][0][i] + re[b][1][i], i1 = im[b][0][i] + im[b][1][i];
                const float r2 = re[b][0][i] - re[b][1][i], i2 = im[b][0][i] - im[b][1][i];
                p[i] = r1 * r1 + i1 * i1;
                q[i] = r2 * r2 + i2 * i2;
            }
            *reinterpret_cast<float4 *>(&s.power[k][fg]) = make_float4(p[0], p[1], p[2], p[3]);
            *reinterpret_cast<float4 *>(&s.power[k][fg + 4]) = make_float4(p[4], p[5], p[6], p[7]);
            if (k != kFft / 4) {
                *reinterpret_cast<float4 *>(&s.power[kFft / 2 - k][fg]) = make_float4(q[0], q[1], q[2], q[3]);
                *reinterpret_cast<float4 *>(&s.power[kFft / 2 - k][fg + 4]) = make_float4(q[4], q[5], q[6], q[7]);
            }
        }
    }
    __syncthreads();

    // filterbank, log10, tile maximum: thread = mel bin, all frames of the tile
    const int m = tid;
    float p[kTileFrames];
#pragma unroll
    for (int f = 0; f < kTileFrames; ++f) p[f] = 0.0f;
#pragma unroll 4
    for (int k = 0; k < kBins; ++k) {                    // mel.cu:141-149
        const float fw = filters_t[k * kMels + m];
#pragma unroll
        for (int f = 0; f < kTileFrames; f += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(&s.power[k][f]);
            p[f] += v.x * fw;
            p[f + 1] += v.y * fw;
            p[f + 2] += v.z * fw;
            p[f + 3] += v.w * fw;
        }
    }
    float tmax = -FLT_MAX;
#pragma unroll
    for (int f = 0; f < kTileFrames; ++f)
        if (f0 + f < n_frames) {
            const float v = log10f(p[f] + 1e-10f);
            logmel[((size_t)w * kMaxFrames + (size_t)(f0 + f)) * kMels + m] = v;
            tmax = fmaxf(tmax, v);
        }
    for (int off = 16; off > 0; off >>= 1) tmax = fmaxf(tmax, __shfl_xor_sync(0xFFFFFFFFu, tmax, off));
    if ((tid & 31) == 0) s.red[tid >> 5] = tmax;
    __syncthreads();
    if (tid == 0) {
        float v = s.red[0];
        for (int i = 1; i < kMelThreads / 32; ++i) v = fmaxf(v, s.red[i]);
        if (v > -FLT_MAX) atomic_max_float(win_max + w, v);
    }
}

// out = bf16((max(v, vmax - 8) + 4) / 4)   (mel.cu:217-233).  grid (frame tiles of 32, windows), block (32, 8).
__global__ void mel_normalize_kernel(const float *__restrict__ logmel, const float *__restrict__ win_max,
                                     const int *__restrict__ num_samples, __nv_bfloat16 *__restrict__ out,
                                     long long out_stride, int time_major) {
    __shared__ float tile[32][kMels + 1];
    pdl_launch_dependents();
    pdl_wait();
    const int w = blockIdx.y;
    const int ns = num_samples[w];
    int n_frames = (ns + kHop - 1) / kHop;
    n_frames = n_frames < 1 ? 1 : (n_frames > kMaxFrames ? kMaxFrames : n_frames);
    const int f0 = blockIdx.x * 32;
    if (f0 >= n_frames) return;
    const float floor_v = win_max[w] - 8.0f;
    __nv_bfloat16 *o = out + (size_t)w * (size_t)out_stride;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int f = ty; f < 32; f += 8) {
        if (f0 + f >= n_frames) break;
        const float *src = logmel + ((size_t)w * kMaxFrames + (size_t)(f0 + f)) * kMels;
        for (int m = tx; m < kMels; m += 32) {
            const float v = (fmaxf(src[m], floor_v) + 4.0f) / 4.0f;
            if (time_major) o[(size_t)(f0 + f) * kMels + m] = __float2bfloat16(v);
            else tile[f][m] = v;
        }
    }
    if (time_major) return;
    __syncthreads();
    // mel-major [128, n_frames]: consecutive threads write consecutive frames of one mel row
    for (int m = ty; m < kMels; m += 8)
        if (f0 + tx < n_frames) o[(size_t)m * n_frames + f0 + tx] = __float2bfloat16(tile[tx][m]);
}

static PerDevice<bool> g_mel_smem_ready;

// d_num_samples: device array [num_windows].  Returns false on a bad argument.
bool launch_mel_batched(const float *pcm, long long pcm_stride, const int *d_num_samples, int num_windows, int max_frames,
                        const float *filters_t, __nv_bfloat16 *out, long long out_stride, int time_major, cudaStream_t st) {
    if (num_windows <= 0) return true;
    if (pcm == nullptr || d_num_samples == nullptr || filters_t == nullptr || out == nullptr) return false;
    const cudaError_t ready = once_per_device(g_mel_smem_ready, [] {
        return cudaFuncSetAttribute(mel_power_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MelSmem));
    });
    if (ready != cudaSuccess) return false;
    float *logmel = (float *)workspace_slot(WS_MEL_LOG, (size_t)num_windows * kMaxFrames * kMels * sizeof(float));
    float *win_max = (float *)workspace_slot(WS_MEL_MAX, (size_t)num_windows * sizeof(float));
    if (cudaMemsetAsync(win_max, 0xFF, (size_t)num_windows * sizeof(float), st) != cudaSuccess) return false;
    const int tiles = (max_frames + kTileFrames - 1) / kTileFrames;
    // only the two launches' own results decide: an error some earlier call of the process left behind is not ours
    const cudaError_t e1 = launch_chained(mel_power_kernel, dim3(tiles, num_windows), dim3(kMelThreads), sizeof(MelSmem), st, pcm,
                                          pcm_stride, d_num_samples, filters_t, logmel, win_max);
    const cudaError_t e2 = launch_chained(mel_normalize_kernel, dim3((max_frames + 31) / 32, num_windows), dim3(32, 8), (size_t)0, st,
                                          (const float *)logmel, (const float *)win_max, d_num_samples, out, out_stride, time_major);
    note_launches(2);
    return e1 == cudaSuccess && e2 == cudaSuccess;
}

static int frames_for(int ns) {
    int n = (ns + kHop - 1) / kHop;
    return n < 1 ? 1 : (n > kMaxFrames ? kMaxFrames : n);
}

}  // namespace glmasr

using namespace glmasr;

enum : int { WS_MEL_NS = 37 };

// Infer-engine/include/cuda_kernels.h:12-14, Infer-engine/cuda/mel.cu:253-294: one window, output mel-major
// [128, n_frames] bf16, *out_frames (host) = n_frames.
extern "C" void mel_spectrogram(const float *pcm, int num_samples, const float *mel_filters_transposed, uint16_t *mel_out,
                                int *out_frames) {
    cudaStream_t st = current_stream();
    int *d_ns = (int *)workspace_slot(WS_MEL_NS, 4096 * sizeof(int));
    GLMASR_CUDA_CHECK(cudaMemcpyAsync(d_ns, &num_samples, sizeof(int), cudaMemcpyHostToDevice, st));
    const int n = frames_for(num_samples);
    if (out_frames != nullptr) *out_frames = n;
    // an empty clip has no samples to point at: nothing is read from pcm then, any valid pointer will do
    if (pcm == nullptr && num_samples <= 0) pcm = mel_filters_transposed;
    GLMASR_CHECK(launch_mel_batched(pcm, 0, d_ns, 1, n, mel_filters_transposed, (__nv_bfloat16 *)mel_out, 0, 0, st),
                 "mel_spectrogram: bad arguments (pcm %p, %d samples, filters %p, out %p)", (const void *)pcm, num_samples,
                 (const void *)mel_filters_transposed, (void *)mel_out);
}

// Infer-engine/cuda/mel.cu:86-109: the reference frees its FFT plan and buffers; here the buffers are private
// workspace slots released by glmasr_fp4_cleanup, so there is nothing to do.
extern "C" void mel_cleanup(void) {}

extern "C" int glmasr_mel_spectrogram_batched(const float *pcm, long long pcm_stride, const int *num_samples_host,
                                              int num_windows, const float *mel_filters_transposed, uint16_t *mel_out,
                                              long long out_stride, int time_major, int *out_frames_host) {
    if (num_windows <= 0) return 0;
    if (num_windows > 4096 || pcm == nullptr || num_samples_host == nullptr || mel_filters_transposed == nullptr || mel_out == nullptr)
        return -1;
    cudaStream_t st = current_stream();
    int *d_ns = (int *)workspace_slot(WS_MEL_NS, 4096 * sizeof(int));
    int max_frames = 1;
    for (int i = 0; i < num_windows; ++i) {
        if (num_samples_host[i] < 0) return -1;
        const int n = frames_for(num_samples_host[i]);
        if (out_frames_host != nullptr) out_frames_host[i] = n;
        if (n > max_frames) max_frames = n;
    }
    if (cudaMemcpyAsync(d_ns, num_samples_host, (size_t)num_windows * sizeof(int), cudaMemcpyHostToDevice, st) != cudaSuccess) return -1;
    // the copy above reads pageable host memory: it has been staged when the call returns
    return launch_mel_batched(pcm, pcm_stride, d_ns, num_windows, max_frames, mel_filters_transposed, (__nv_bfloat16 *)mel_out,
                              out_stride, time_major, st)
               ? 0
               : -1;
}
