// Log-mel frontend: PCM -> normalised log-mel features [utterance, frame, 128] fp32, the input
// of the subsampling stage.  Replaces run_frontend (src/cuda/frontend.rs:230-316) and its kernels
// pk_sm89_frame_window / cuFFT R2C / pk_sm89_mel_log_sparse / pk_sm89_normalize_mel
// (kernels/sm89/frontend.cu:11-115); CPU definition: CpuMelFrontend::compute
// (src/frontend.rs:114-215).
//
// mel_frames_kernel takes a tile of consecutive frames per CTA from the PCM to the log-mel rows, so the
// framed signal and the spectrum never travel through HBM (the reference stores both); a
// second kernel normalises every mel row over the valid frames in double precision.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "pk100_internal.h"
#include "ptx_sm100.cuh"

namespace pk100 {

constexpr int kFft = 512;
constexpr int kFftBins = kFft / 2 + 1;
constexpr int kHop = 160;
constexpr int kMels = 128;
constexpr int kMelThreads = 256;
constexpr int kMelWarps = kMelThreads / 32;
constexpr int kKeptTaps = 1024;                     // a bank with more non-zeros is read from global memory
constexpr int kExchange = 320;                      // complex values of one warp's exchange buffer, padding included

template <int Tile>                                 // frames per CTA
struct MelSmem {
    static constexpr int kPcm = (Tile - 1) * kHop + kFft + 2;   // from two samples before the first frame
    static constexpr int kPowerPitch = Tile + 4;    // 16-byte reads of 8 neighbouring bins hit 8 different bank groups
    alignas(16) float pcm[kPcm];                    // raw samples of the tile, zero outside the utterance
    alignas(16) float2 exchange[kMelWarps][kExchange];
    float2 twiddle[kFft];                           // e^{-2 pi i k / 512}
    alignas(16) float power[kFftBins * kPowerPitch];   // [bin][frame]
    float2 taps[kKeptTaps];                         // {filter value, offset of its bin in `power` as int bits}
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul_neg_i(float2 a) { return make_float2(a.y, -a.x); }

__device__ __forceinline__ void dft4(float2 (&v)[4]) {
    const float2 s02 = cadd(v[0], v[2]), d02 = csub(v[0], v[2]);
    const float2 s13 = cadd(v[1], v[3]), d13 = cmul_neg_i(csub(v[1], v[3]));
    v[0] = cadd(s02, s13); v[1] = cadd(d02, d13); v[2] = csub(s02, s13); v[3] = csub(d02, d13);
}

// 8-point DFT in natural order: the two 4-point DFTs of even and odd elements, then radix 2
__device__ __forceinline__ void dft8(float2 (&v)[8]) {
    constexpr float kHalfSqrt = 0.70710678118654752f;
    float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft4(e);
    dft4(o);
    o[1] = make_float2(kHalfSqrt * (o[1].x + o[1].y), kHalfSqrt * (o[1].y - o[1].x));
    o[2] = cmul_neg_i(o[2]);
    o[3] = make_float2(kHalfSqrt * (o[3].y - o[3].x), -kHalfSqrt * (o[3].x + o[3].y));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[i] = cadd(e[i], o[i]);
        v[i + 4] = csub(e[i], o[i]);
    }
}

// One CTA = `Tile` consecutive frames of one utterance.  The tile's samples are staged once
// (neighbouring frames share 352 of their 512 samples) and pre-emphasised where they are read.  A warp transforms one frame
// at a time: the 512 real samples as 256 complex ones, 8 per lane, 256 = 8 x 8 x 4 with the first two
// factors in registers and the warp's own exchange buffer in between (no CTA barrier inside a
// transform, a lane's twiddles stay in registers), then the split into the 257 bins of the real
// transform.  The mel filters run after all spectra with one thread per (mel bin, Tile / 2 frames),
// so a filter tap is fetched once per Tile / 2 frames.
// Tile: 32 for large batches (staging and twiddles shared by four frames per warp), 8 where 32 would
// leave SMs without a CTA.  The radix-2 form with one CTA per frame spent its time on 9 barriers and
// shared-memory round trips per frame and on one tap fetch per frame and mel bin.
// 8 x 60 s (48 008 frames): 410 us before, 68 us now.
template <int Tile>
__global__ void __launch_bounds__(kMelThreads, 2)
mel_frames_kernel(const float* __restrict__ samples, long long sample_stride, const int* __restrict__ sample_counts,
                  const float* __restrict__ window, const int* __restrict__ filter_offsets,
                  const int* __restrict__ filter_bins, const float* __restrict__ filter_values,
                  float* __restrict__ mel, int frame_cap, float preemphasis, float log_zero_guard) {
    extern __shared__ __align__(16) uint8_t mel_smem[];
    MelSmem<Tile>& sm = *reinterpret_cast<MelSmem<Tile>*>(mel_smem);
    constexpr int kPowerPitch = MelSmem<Tile>::kPowerPitch, kPerThread = Tile / 2;
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    const int frame0 = blockIdx.x * Tile, utt = blockIdx.y;
    const int count = sample_counts[utt];
    const int frames = count > 0 ? count / kHop + 1 : 0;
    const int mel_bin = tid % kMels, frame_half = tid / kMels;      // mel phase: kPerThread frames per thread
    float* out = mel + (static_cast<size_t>(utt) * frame_cap + frame0 + frame_half * kPerThread) * kMels + mel_bin;
    const int rows_left = frame_cap - frame0 - frame_half * kPerThread;      // rows of the output block from `out` on
    if (frame0 >= frames) {                        // beyond this utterance: zero rows
#pragma unroll
        for (int i = 0; i < kPerThread; ++i)
            if (i < rows_left) out[static_cast<size_t>(i) * kMels] = 0.0f;
        return;
    }
    const float* pcm = samples + static_cast<size_t>(utt) * sample_stride;
    const int sample0 = frame0 * kHop - kFft / 2 - 2;
    const int tap_count = __ldg(filter_offsets + kMels);
    const bool kept_taps = tap_count <= kKeptTaps;
    if (kept_taps)
        for (int t = tid; t < tap_count; t += kMelThreads)
            sm.taps[t] = make_float2(__ldg(filter_values + t), __int_as_float(__ldg(filter_bins + t) * kPowerPitch));
    // asynchronous copies: all of a thread's samples are in flight at once
    for (int i = tid; i < MelSmem<Tile>::kPcm; i += kMelThreads) {
        const int sample = sample0 + i;
        const bool inside = sample >= 0 && sample < count;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(&sm.pcm[i])),
                     "l"(pcm + (inside ? sample : 0)), "r"(inside ? 4 : 0) : "memory");
    }
    {
        float s, c;
        sincospif(-2.0f * static_cast<float>(tid) / static_cast<float>(kFft), &s, &c);
        sm.twiddle[tid] = make_float2(c, s);
        sm.twiddle[tid + kFft / 2] = make_float2(-c, -s);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    const int k8 = lane / 4, s4 = lane % 4;
    float2* ex = sm.exchange[warp];
    const float2* tw = sm.twiddle;
    float2 tw_a[7], tw_b[7];                         // W_256^(lane k) and W_32^(s4 q)
#pragma unroll
    for (int k = 1; k < 8; ++k) {
        tw_a[k - 1] = tw[2 * lane * k];
        tw_b[k - 1] = tw[16 * s4 * k];
    }
    float2 win[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int n = 2 * (lane + 32 * j);
        win[j] = make_float2(__ldg(window + n), __ldg(window + n + 1));
    }
    for (int f = warp; f < Tile; f += kMelWarps) {
        if (frame0 + f >= frames) break;
        const float* src = sm.pcm + f * kHop + 2;
        const int left = count - ((frame0 + f) * kHop - kFft / 2);   // samples of this frame before the utterance's end
        float2 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {               // complex sample n = lane + 32 j
            const int n = 2 * (lane + 32 * j);
            const float2 x = *reinterpret_cast<const float2*>(src + n);
            v[j] = make_float2((x.x - preemphasis * src[n - 1]) * win[j].x, (x.y - preemphasis * x.x) * win[j].y);
            if (n + 2 > left) {                     // past the end the pre-emphasised signal is zero, too
                if (n >= left) v[j].x = 0.0f;
                if (n + 1 >= left) v[j].y = 0.0f;
            }
        }
        dft8(v);                                     // over j -> output digit k (low)
#pragma unroll
        for (int k = 1; k < 8; ++k) v[k] = cmul(v[k], tw_a[k - 1]);
        // [k][lane] with 36 complex per row: both sides of the exchange are free of bank conflicts
#pragma unroll
        for (int k = 0; k < 8; ++k) ex[k * 36 + lane] = v[k];
        __syncwarp();
#pragma unroll
        for (int m = 0; m < 8; ++m) v[m] = ex[k8 * 36 + s4 + 4 * m];
        dft8(v);                                     // over m -> middle digit q
#pragma unroll
        for (int q = 1; q < 8; ++q) v[q] = cmul(v[q], tw_b[q - 1]);
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 8; ++q) ex[k8 * 38 + s4 + 4 * q] = v[q];
        __syncwarp();
        float2 w[2][4];                              // digits q = s4 and s4 + 4, the four elements of the last factor
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float4* pair = reinterpret_cast<const float4*>(ex + k8 * 38 + 4 * (s4 + 4 * e));
            const float4 a = pair[0], b = pair[1];
            w[e][0] = make_float2(a.x, a.y); w[e][1] = make_float2(a.z, a.w);
            w[e][2] = make_float2(b.x, b.y); w[e][3] = make_float2(b.z, b.w);
            dft4(w[e]);
        }
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int bin = k8 + 8 * (s4 + 4 * e) + 64 * r;
                ex[bin + 4 * (bin >> 4)] = w[e][r];
            }
        __syncwarp();
        // X[k] = (Z[k] + conj Z[256 - k]) / 2 + W^k (Z[k] - conj Z[256 - k]) / 2i, and its mirror
        float* power = sm.power + f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = lane + 32 * i, mirror = (kFft / 2 - k) % (kFft / 2);
            const float2 a = ex[k + 4 * (k >> 4)], b = ex[mirror + 4 * (mirror >> 4)];
            const float er = 0.5f * (a.x + b.x), ei = 0.5f * (a.y - b.y);
            const float2 odd = make_float2(0.5f * (a.y + b.y), 0.5f * (b.x - a.x));
            const float2 t = cmul(odd, tw[k]);
            const float xr = er + t.x, xi = ei + t.y, yr = er - t.x, yi = ei - t.y;
            power[k * kPowerPitch] = xr * xr + xi * xi;
            power[(kFft / 2 - k) * kPowerPitch] = yr * yr + yi * yi;
        }
        if (lane == 0) {
            const float2 a = ex[128 + 4 * (128 >> 4)];
            power[128 * kPowerPitch] = a.x * a.x + a.y * a.y;
        }
        __syncwarp();
    }
    __syncthreads();
    float sum[kPerThread];
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) sum[i] = 0.0f;
    auto add_tap = [&](float tap, int offset) {
        const float4* p = reinterpret_cast<const float4*>(sm.power + offset + frame_half * kPerThread);
#pragma unroll
        for (int i = 0; i < kPerThread / 4; ++i) {
            const float4 a = p[i];
            sum[4 * i] = fmaf(tap, a.x, sum[4 * i]); sum[4 * i + 1] = fmaf(tap, a.y, sum[4 * i + 1]);
            sum[4 * i + 2] = fmaf(tap, a.z, sum[4 * i + 2]); sum[4 * i + 3] = fmaf(tap, a.w, sum[4 * i + 3]);
        }
    };
    const int tap_begin = __ldg(filter_offsets + mel_bin), tap_end = __ldg(filter_offsets + mel_bin + 1);
    if (kept_taps) {
#pragma unroll 4
        for (int t = tap_begin; t < tap_end; ++t) add_tap(sm.taps[t].x, __float_as_int(sm.taps[t].y));
    } else {
        for (int t = tap_begin; t < tap_end; ++t) add_tap(__ldg(filter_values + t), __ldg(filter_bins + t) * kPowerPitch);
    }
#pragma unroll
    for (int i = 0; i < kPerThread; ++i)
        if (i < rows_left)
            out[static_cast<size_t>(i) * kMels] = frame0 + frame_half * kPerThread + i < frames ? logf(sum[i] + log_zero_guard) : 0.0f;
}

// Mean and unbiased variance of every mel bin over the valid frames in double precision, rows at or
// beyond the valid count become zero (frontend.cu:64-115).  A cluster of 8 CTAs owns 32 mel bins of
// one utterance: each CTA takes an eighth of the frames (128-byte row pieces, lane = bin), keeps them in
// shared memory between the passes where they fit (6144 frames), and the partial sums meet
// through distributed shared memory.  With one CTA per bin and strided columns: 243 us for 8 x 60 s,
// 22 us now.
constexpr int kNormCluster = 8;
constexpr int kNormBins = 32;
constexpr int kNormThreads = 512;
constexpr int kNormWarps = kNormThreads / 32;
constexpr int kNormRows = 768;                      // rows a CTA keeps in shared memory
constexpr int kNormSmem = kNormRows * kNormBins * 4;

__global__ void __cluster_dims__(kNormCluster, 1, 1) __launch_bounds__(kNormThreads, 2)
mel_normalize_kernel(float* __restrict__ mel, const int* __restrict__ sample_counts, int frame_cap, float epsilon,
                     int* __restrict__ valid_out) {
    extern __shared__ __align__(16) float norm_rows[];
    __shared__ double part[kNormWarps][kNormBins];
    __shared__ double total[2][kNormBins];
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    const int rank = static_cast<int>(cluster.block_rank());
    const int bin0 = blockIdx.y * kNormBins, utt = blockIdx.z;
    const int count = sample_counts[utt];
    const int valid = count > 0 ? count / kHop : 0;
    const int frames = count > 0 ? valid + 1 : 0;
    if (rank == 0 && blockIdx.y == 0 && tid == 0 && valid_out != nullptr) valid_out[utt] = valid;
    const int per = (frames + kNormCluster - 1) / kNormCluster;
    const int first = min(rank * per, frames), last = min(first + per, frames);
    const bool kept = per <= kNormRows;
    float* rows = mel + (static_cast<size_t>(utt) * frame_cap) * kMels + bin0 + lane;
    // sum over this CTA's warps, then over the cluster; every thread gets its bin's total
    auto cluster_sum = [&](double v, int slot) {
        part[warp][lane] = v;
        __syncthreads();
        if (warp == 0) {
            double s = part[0][lane];
#pragma unroll
            for (int w = 1; w < kNormWarps; ++w) s += part[w][lane];
            total[slot][lane] = s;
        }
        cluster.sync();
        double s = 0.0;
#pragma unroll
        for (int c = 0; c < kNormCluster; ++c) s += *cluster.map_shared_rank(&total[slot][lane], c);
        return s;
    };
    double s = 0.0;
#pragma unroll 4
    for (int f = first + warp; f < last; f += kNormWarps) {
        const float v = rows[static_cast<size_t>(f) * kMels];
        if (kept) norm_rows[(f - first) * kNormBins + lane] = v;
        if (f < valid) s += static_cast<double>(v);
    }
    const double sum = cluster_sum(s, 0);
    const double mean = valid > 0 ? sum / valid : 0.0;
    double q = 0.0;
#pragma unroll 4
    for (int f = first + warp; f < min(last, valid); f += kNormWarps) {
        const double d = static_cast<double>(kept ? norm_rows[(f - first) * kNormBins + lane] : rows[static_cast<size_t>(f) * kMels]) - mean;
        q += d * d;
    }
    const double sq = cluster_sum(q, 1);
    const double variance = valid > 1 ? sq / static_cast<double>(valid - 1) : 0.0;
    const double inverse = 1.0 / (sqrt(variance) + static_cast<double>(epsilon));
#pragma unroll 4
    for (int f = first + warp; f < last; f += kNormWarps) {
        const float v = kept ? norm_rows[(f - first) * kNormBins + lane] : rows[static_cast<size_t>(f) * kMels];
        rows[static_cast<size_t>(f) * kMels] = f < valid ? static_cast<float>((static_cast<double>(v) - mean) * inverse) : 0.0f;
    }
    cluster.sync();          // no CTA leaves while a peer may still read its totals
}

}  // namespace pk100

using namespace pk100;

extern "C" int pk100_mel_frames_for(int samples) { return samples > 0 ? samples / kHop + 1 : 0; }

template <int Tile>
static int launch_mel_frames(cudaStream_t stream, const pk100_frontend_weights* w, const float* samples, int utterances,
                             long long sample_stride, const int* sample_counts, float* mel, int frame_cap) {
    const cudaError_t err = cudaFuncSetAttribute(mel_frames_kernel<Tile>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 sizeof(MelSmem<Tile>));
    if (err != cudaSuccess) return static_cast<int>(err);
    mel_frames_kernel<Tile><<<dim3((frame_cap + Tile - 1) / Tile, utterances), kMelThreads, sizeof(MelSmem<Tile>), stream>>>(
        samples, sample_stride, sample_counts, w->window, w->filter_offsets, w->filter_bins, w->filter_values, mel,
        frame_cap, w->preemphasis, w->log_zero_guard);
    return pk100_launch_status();
}

extern "C" int pk100_mel_frontend(void* stream_v, const pk100_frontend_weights* w, const float* samples,
                                  int utterances, long long sample_stride, const int* sample_counts, float* mel,
                                  int frame_cap, int* valid_frames) {
    if (!w || !w->window || !w->filter_offsets || !w->filter_bins || !w->filter_values || !samples ||
        !sample_counts || !mel)
        return PK100_ERR_NULL;
    if (utterances == 0) return PK100_OK;
    if (utterances < 0 || frame_cap <= 0 || sample_stride <= 0) return PK100_ERR_SHAPE;
    // every frame a utterance of sample_stride samples can have must fit the output block
    if (sample_stride / kHop + 1 > frame_cap) return PK100_ERR_SHAPE;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    // 8-frame tiles while 32-frame ones would not give every SM two CTAs
    const long long frames = static_cast<long long>(frame_cap) * utterances;
    const int frc = frames >= 32LL * 2 * pk100_cta_budget()
        ? launch_mel_frames<32>(stream, w, samples, utterances, sample_stride, sample_counts, mel, frame_cap)
        : launch_mel_frames<8>(stream, w, samples, utterances, sample_stride, sample_counts, mel, frame_cap);
    if (frc != PK100_OK) return frc;
    // (an attribute of the function, kept per device by the runtime; setting it again costs little)
    const cudaError_t err = cudaFuncSetAttribute(mel_normalize_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kNormSmem);
    if (err != cudaSuccess) return static_cast<int>(err);
    mel_normalize_kernel<<<dim3(kNormCluster, kMels / kNormBins, utterances), kNormThreads, kNormSmem, stream>>>(
        mel, sample_counts, frame_cap, w->normalize_epsilon, valid_frames);
    return pk100_launch_status();
}
