// 8x depthwise-striding convolution subsampling (mel [frames,128] -> [frames/8, 1024])
// for a batch of utterances.  The convolutions are channel-parallel kernels (thread =
// channel, coalesced over the 256 channels), the first two fused so that the largest
// intermediate never reaches HBM; the two pointwise layers and
// the 4096 -> 1024 projection are tcgen05 GEMMs (pk100_gemm).  Semantics follow
// kernels/sm89/subsampling.cu:11-226 and the host tiling of
// src/cuda/subsampling.rs:436-804 (without its 256-frame tiles: the whole batch is
// processed at once).
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>

#include "pk100_internal.h"
#include "ptx_sm100.cuh"
#include "row_quant.cuh"

namespace pk100 {

constexpr int kChannels = 256;
constexpr int kMelBins = 128;

__device__ __forceinline__ int frames_of(const int* per_utt, int utt, int uniform) {
    return per_utt != nullptr ? per_utt[utt] : uniform;
}

// both halves rounded to fp16 and through ReLU; a NaN becomes 0 (max.f16x2 returns the operand that is a number,
// the .relu form of the conversion would keep it)
__device__ __forceinline__ __half2 relu_half2(Pair v) {
    const float2 f = halves_of(v);
    return __hmax2(__floats2half2_rn(f.x, f.y), __half2half2(__ushort_as_half(0)));
}

// E4M3 codes of one row, absmax / 448 per row: the arithmetic of pk100_pack_weight_rows
__device__ __forceinline__ float e4m3_row_scale(float absmax) { return absmax > 0.0f ? __fdiv_rn(absmax, 448.0f) : 1.0f; }

// First two stages in one kernel: conv 3x3 s2 (1 -> 256 channels) + bias + ReLU, rounded to fp16,
// feeding the depthwise conv 3x3 s2 + bias.  The intermediate [frames/2, 64, 256] tensor (98 KB per
// output frame, 786 MB for 8 x 60 s) stays in registers instead of making a round trip through HBM.
// One CTA = a run of consecutive output frames (as many as fill the device evenly, at most 8: the
// weights are fetched once per run) x half of the output features; thread = two neighbouring channels x kFirstOuts
// output features.  The mel rows are staged in
// shared memory with every value stored twice, so that one load feeds the packed multiply-adds of
// both channels.  Intermediate rows are walked in order; the row shared by two output frames
// (2*f2 + 1) is computed once and scattered into both, so a frame costs two rows of the first
// convolution, not three.  The accumulation order of both convolutions (bias, then taps row by row)
// is the reference's (kernels/sm89/subsampling.cu:11-179); the out-of-range taps it skips are zero
// taps on zero values here.
// Bound by its fp32 multiply-adds (about 6000 packed warp instructions per output frame).  8 x 60 s: 405 us
// with one frame per CTA, one channel per thread and three rows per frame, 330 us now (E4M3 372 us, where
// a quantising pass of 270 us followed before).
// Fp8: the result leaves as E4M3 with one scale per (frame, feature) row of 256 channels; each row
// is first rounded to fp16, as when a separate kernel quantises the fp16 tensor.
// in [utt][in_stride frames][128] fp32 -> out [utt][out_cap][32][256]
constexpr int kFirstOuts = 8;                              // output features per thread
constexpr int kFirstMaxFrames = 8;
constexpr int first_rows(int frames) { return 4 * frames + 3; }   // mel rows 4*f2_first - 3 .. 4*f2_last + 3
constexpr int kFirstThreads = 256;                         // 128 channel pairs x 2 parts
constexpr int kFirstPitch = kMelBins + 2;                  // column t at index t + 1, one zero column on each side

template <bool Fp8>
__global__ void __launch_bounds__(kFirstThreads, 2)
subsample_first_fused_kernel(const float* __restrict__ in, const __half* __restrict__ w0,
                             const __half* __restrict__ b0, const __half* __restrict__ w1,
                             const __half* __restrict__ b1, void* __restrict__ out, float* __restrict__ out_scales,
                             int in_stride, int in_frames_uniform, const int* __restrict__ in_frames_per_utt,
                             int out_cap, int run) {
    extern __shared__ __align__(16) uint8_t first_smem[];
    auto mel = reinterpret_cast<float2 (*)[kFirstPitch]>(first_smem);      // [first_rows(run)]
    constexpr int kRows = 2 * kFirstOuts;                  // output features of this CTA
    __shared__ float row_max[2][4][kRows];                 // [frame parity][warp of a part][feature]
    __shared__ float2 row_div[2][kRows];                   // [frame parity][feature]: divisor and reciprocal
    __shared__ Pair taps[2][9][kChannels / 2];             // both convolutions' taps as channel pairs
    const int tid = threadIdx.x;
    const int ch = (tid % 128) * 2;                        // channels ch, ch + 1
    const int part = blockIdx.z * 2 + tid / 128;           // outputs kFirstOuts * part .. + kFirstOuts - 1
    const int first = blockIdx.x * run, utt = blockIdx.y;
    const int in_frames = frames_of(in_frames_per_utt, utt, in_frames_uniform);
    const int f1_frames = (in_frames + 1) / 2;
    const int f2_frames = (f1_frames + 1) / 2;
    if (first >= f2_frames) return;
    const float* src = in + static_cast<size_t>(utt) * in_stride * kMelBins;
    for (int i = tid; i < first_rows(run) * kFirstPitch; i += kFirstThreads) {
        const int row = i / kFirstPitch, t = i % kFirstPitch - 1;
        const int f = 4 * first - 3 + row;
        const float v = (f >= 0 && f < in_frames && t >= 0 && t < kMelBins) ? src[static_cast<size_t>(f) * kMelBins + t] : 0.0f;
        (&mel[0][0])[i] = make_float2(v, v);
    }
    for (int i = tid; i < kChannels / 2 * 9; i += kFirstThreads) {
        const int pair = i / 9, tap = i % 9;
        taps[0][tap][pair] = pair_of(__half2float(w0[pair * 18 + tap]), __half2float(w0[pair * 18 + 9 + tap]));
        taps[1][tap][pair] = pair_of(__half2float(w1[pair * 18 + tap]), __half2float(w1[pair * 18 + 9 + tap]));
    }
    const Pair bias0 = pair_of(__half2float(b0[ch]), __half2float(b0[ch + 1]));
    const Pair bias1 = pair_of(__half2float(b1[ch]), __half2float(b1[ch + 1]));
    __syncthreads();
    // Nine taps as registers.  Reloaded per intermediate row and convolution (`volatile` keeps the
    // compiler from holding all 18 pairs across the loop, which spills the sums).
    const uint32_t taps_addr = smem_u32(&taps[0][0][ch / 2]);
    auto load_taps = [&](Pair (&w)[9], int conv) {
#pragma unroll
        for (int i = 0; i < 9; ++i)
            asm volatile("ld.shared.b64 %0, [%1];" : "=l"(w[i]) : "r"(taps_addr + (conv * 9 + i) * (kChannels / 2 * 8)));
    };
    // one intermediate row (staged mel rows 2*k .. 2*k + 2), rounded to fp16: v[m + 1] = feature
    // 2 * kFirstOuts * part + m, m = -1 .. 2 * kFirstOuts - 1 (the first quarter has no feature -1)
    auto walk_row = [&](int k, __half2 (&v)[2 * kFirstOuts + 1]) {
        Pair w[9];
        load_taps(w, 0);
        // taps on rows in front of the first or behind the last frame
        const int f1 = 2 * first - 1 + k;                  // its mel rows: 2*f1 - 1 .. 2*f1 + 1
        if (f1 == 0 || 2 * f1 + 1 >= in_frames) [[unlikely]] {
            const bool head = f1 == 0, tail = 2 * f1 + 1 >= in_frames;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                w[i] = head ? 0ull : w[i];
                w[6 + i] = tail ? 0ull : w[6 + i];
            }
        }
        const float2* base[3];
        Pair c0[3], c1[3];                                 // columns 2*m1 - 1, 2*m1 of the sliding window
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            base[a] = &mel[2 * k + a][4 * kFirstOuts * part];          // index of column 4*kFirstOuts*part - 1
            c0[a] = *reinterpret_cast<const Pair*>(base[a]);
            c1[a] = *reinterpret_cast<const Pair*>(base[a] + 1);
        }
        v[0] = __half2half2(__ushort_as_half(0));
        if (part > 0) {                                    // the odd feature left of the first output
            Pair acc = bias0;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                acc = pair_fma(*reinterpret_cast<const Pair*>(base[a] - 2), w[a * 3 + 0], acc);
                acc = pair_fma(*reinterpret_cast<const Pair*>(base[a] - 1), w[a * 3 + 1], acc);
                acc = pair_fma(c0[a], w[a * 3 + 2], acc);
            }
            v[0] = relu_half2(acc);
        }
#pragma unroll
        for (int m = 0; m < 2 * kFirstOuts; ++m) {
            Pair acc = bias0;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                // columns 2*m1 + 1 and 2*m1 + 2: 16-byte aligned, because an even column sits at an odd index
                const ulonglong2 nx = *reinterpret_cast<const ulonglong2*>(base[a] + 2 * m + 2);
                // (column -1 is outside)
                acc = pair_fma(c0[a], m == 0 && part == 0 ? 0ull : w[a * 3 + 0], acc);
                acc = pair_fma(c1[a], w[a * 3 + 1], acc);
                acc = pair_fma(nx.x, w[a * 3 + 2], acc);
                c0[a] = nx.x;
                c1[a] = nx.y;
            }
            v[m + 1] = relu_half2(acc);
        }
    };
    // output m2 takes features 2*m2 - 1, 2*m2, 2*m2 + 1 as taps 0, 1, 2
    auto scatter = [&](Pair (&sums)[kFirstOuts], const Pair (&w)[9], int kf, const __half2 (&v)[2 * kFirstOuts + 1]) {
        Pair left = pair_of(v[0]);
#pragma unroll
        for (int m = 0; m < kFirstOuts; ++m) {
            if (m > 0 || part > 0) sums[m] = pair_fma(left, w[kf * 3 + 0], sums[m]);
            sums[m] = pair_fma(pair_of(v[2 * m + 1]), w[kf * 3 + 1], sums[m]);
            left = pair_of(v[2 * m + 2]);
            sums[m] = pair_fma(left, w[kf * 3 + 2], sums[m]);
        }
    };

    Pair cur[kFirstOuts], next[kFirstOuts];
#pragma unroll
    for (int m = 0; m < kFirstOuts; ++m) cur[m] = bias1;
    if (first > 0) {
        __half2 v[2 * kFirstOuts + 1];
        walk_row(0, v);
        Pair w[9];
        load_taps(w, 1);
        scatter(cur, w, 0, v);
    }
#pragma unroll 1
    for (int i = 0; i < run; ++i) {
        const int f2 = first + i;
        if (f2 >= f2_frames) break;
#pragma unroll
        for (int m = 0; m < kFirstOuts; ++m) next[m] = bias1;
#pragma unroll 1
        for (int kf = 1; kf < 3; ++kf) {
            if (kf == 2 && 2 * f2 + 1 >= f1_frames) break;
            __half2 v[2 * kFirstOuts + 1];
            walk_row(2 * i + kf, v);
            Pair w[9];
            load_taps(w, 1);
            if (kf == 1) {
                scatter(cur, w, 1, v);
            } else {
                scatter(cur, w, 2, v);
                scatter(next, w, 0, v);
            }
        }
        const size_t row0 = (static_cast<size_t>(utt) * out_cap + f2) * 32 + part * kFirstOuts;
        if constexpr (Fp8) {
            const int warp = tid / 32, lane = tid % 32, local = (tid / 128) * kFirstOuts, par = i & 1;
            __half2 h[kFirstOuts];
#pragma unroll
            for (int m = 0; m < kFirstOuts; ++m) {
                const float2 f = halves_of(cur[m]);
                h[m] = __floats2half2_rn(f.x, f.y);
                const float2 r = __half22float2(__habs2(h[m]));
                // non-negative floats order like their bits
                const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(r.x, r.y)));
                if (lane == 0) row_max[par][warp % 4][local + m] = __uint_as_float(top);
            }
            __syncthreads();
            if (tid < kRows) {                             // one division and one reciprocal per row
                const float scale = e4m3_row_scale(fmaxf(fmaxf(row_max[par][0][tid], row_max[par][1][tid]),
                                                         fmaxf(row_max[par][2][tid], row_max[par][3][tid])));
                const RowDivisor div(scale);
                row_div[par][tid] = make_float2(div.s, div.y);
                out_scales[(static_cast<size_t>(utt) * out_cap + f2) * 32 + blockIdx.z * kRows + tid] = scale;
            }
            __syncthreads();
            uint8_t* dst = static_cast<uint8_t*>(out) + row0 * kChannels + ch;
#pragma unroll
            for (int m = 0; m < kFirstOuts; ++m) {
                const float2 d = row_div[par][local + m];
                const RowDivisor div(d.x, d.y);
                const float2 f = __half22float2(h[m]);
                *reinterpret_cast<uint16_t*>(dst + static_cast<size_t>(m) * kChannels) =
                    static_cast<uint16_t>(__nv_cvt_float2_to_fp8x2(make_float2(div(f.x), div(f.y)), __NV_SATFINITE, __NV_E4M3));
            }
        } else {
            __half* dst = static_cast<__half*>(out) + row0 * kChannels + ch;
#pragma unroll
            for (int m = 0; m < kFirstOuts; ++m) {
                const float2 f = halves_of(cur[m]);
                *reinterpret_cast<__half2*>(dst + static_cast<size_t>(m) * kChannels) = __floats2half2_rn(f.x, f.y);
            }
        }
#pragma unroll
        for (int m = 0; m < kFirstOuts; ++m) cur[m] = next[m];
    }
}

// N halves (a multiple of 8), 16 bytes at a time where the caller's pointer allows it
template <int N>
__device__ __forceinline__ void load_halves(__half (&dst)[N], const __half* src) {
    if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
#pragma unroll
        for (int i = 0; i < N / 8; ++i) reinterpret_cast<uint4*>(dst)[i] = __ldg(reinterpret_cast<const uint4*>(src) + i);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) dst[i] = src[i];
    }
}

// depthwise conv 3x3, stride 2, pad 1, + bias (no activation), HBM-bound: a thread owns 8 channels
// (16-byte loads and stores) of one output frame and walks kDepthwiseRun output features, each input
// feature loaded once per input row.  Tap order (frame taps outer, feature taps inner, out-of-range
// taps skipped) as in the reference.
// in [utt][in_cap][in_feats][256] -> out [utt][out_cap][in_feats/2][256]
constexpr int kDepthwiseRun = 4;

__global__ void __launch_bounds__(128)
subsample_depthwise_kernel(const __half* __restrict__ in, const __half* __restrict__ w,
                           const __half* __restrict__ b, __half* __restrict__ out, int in_cap,
                           int in_feats, int out_cap, int mel_frames_uniform,
                           const int* __restrict__ mel_frames_per_utt, int in_level) {
    const int ch = (threadIdx.x % 32) * 8;
    const int out_feats = in_feats / 2;
    const int feat0 = (blockIdx.x * 4 + threadIdx.x / 32) * kDepthwiseRun;
    const int of = blockIdx.y;
    const int utt = blockIdx.z;
    int in_frames = frames_of(mel_frames_per_utt, utt, mel_frames_uniform);
    for (int l = 0; l < in_level; ++l) in_frames = (in_frames + 1) / 2;
    const int out_frames = (in_frames + 1) / 2;
    if (of >= out_frames || feat0 >= out_feats) return;
    Pair sums[kDepthwiseRun][4];
    // 8 channels x 9 taps: 144 contiguous bytes
    alignas(16) __half taps[72];
    alignas(16) __half bias[8];
    load_halves<8>(bias, b + ch);
    load_halves<72>(taps, w + static_cast<size_t>(ch) * 9);
#pragma unroll
    for (int g = 0; g < kDepthwiseRun; ++g)
#pragma unroll
        for (int c = 0; c < 4; ++c) sums[g][c] = pair_of(reinterpret_cast<const __half2*>(bias)[c]);
    const __half* src = in + static_cast<size_t>(utt) * in_cap * in_feats * kChannels + ch;
    constexpr int kCols = 2 * kDepthwiseRun + 1;
#pragma unroll
    for (int kf = 0; kf < 3; ++kf) {
        const int f = of * 2 + kf - 1;
        if (f < 0 || f >= in_frames) continue;
        uint4 col[kCols];
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
            const int t = feat0 * 2 + j - 1;
            col[j] = (t >= 0 && t < in_feats)
                ? __ldg(reinterpret_cast<const uint4*>(src + (static_cast<size_t>(f) * in_feats + t) * kChannels))
                : make_uint4(0, 0, 0, 0);
        }
        Pair tap[3][4];
#pragma unroll
        for (int kt = 0; kt < 3; ++kt)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                tap[kt][c] = pair_of(__half2float(taps[(2 * c) * 9 + kf * 3 + kt]), __half2float(taps[(2 * c + 1) * 9 + kf * 3 + kt]));
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
            const __half2* h = reinterpret_cast<const __half2*>(&col[j]);
            const int t = feat0 * 2 + j - 1;
            if (t < 0 || t >= in_feats) continue;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const Pair v = pair_of(h[c]);
                // column j is tap j - 2 g of output g
#pragma unroll
                for (int g = 0; g < kDepthwiseRun; ++g)
                    if (j - 2 * g >= 0 && j - 2 * g < 3) sums[g][c] = pair_fma(v, tap[j - 2 * g][c], sums[g][c]);
            }
        }
    }
    __half* dst = out + ((static_cast<size_t>(utt) * out_cap + of) * out_feats + feat0) * kChannels + ch;
#pragma unroll
    for (int g = 0; g < kDepthwiseRun; ++g) {
        if (feat0 + g >= out_feats) break;
        uint4 raw;
        __half2* h = reinterpret_cast<__half2*>(&raw);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float2 f = halves_of(sums[g][c]);
            h[c] = __floats2half2_rn(f.x, f.y);
        }
        *reinterpret_cast<uint4*>(dst + static_cast<size_t>(g) * kChannels) = raw;
    }
}

// [utt][cap][16][256] -> rows [utt*seg_stride + frame][channel*16 + feature]; rows at or
// beyond the utterance's output length are zero (kernels/sm89/subsampling.cu:202-226).
// row_base != nullptr (packed batch): utterance utt starts at row row_base[utt] and has whole 128-row tiles.
// 128 threads per row, thread = two neighbouring channels: their 32 features are contiguous in the row.
// Fp8: the row leaves as E4M3 codes with one scale (absmax / 448).
template <bool Fp8>
__global__ void __launch_bounds__(128)
subsample_flatten_kernel(const __half* __restrict__ in, void* __restrict__ out, float* __restrict__ out_scales,
                         int in_cap, int seg_stride, int mel_frames_uniform,
                         const int* __restrict__ mel_frames_per_utt, const int* __restrict__ row_base) {
    __shared__ float warp_max[4];
    const int frame = blockIdx.x, utt = blockIdx.y, tid = threadIdx.x;
    int valid = frames_of(mel_frames_per_utt, utt, mel_frames_uniform);
    for (int l = 0; l < 3; ++l) valid = (valid + 1) / 2;
    if (row_base != nullptr && frame >= (valid + 127) / 128 * 128) return;
    const size_t row = (row_base != nullptr ? static_cast<size_t>(row_base[utt]) : static_cast<size_t>(utt) * seg_stride) + frame;
    const __half2* src = reinterpret_cast<const __half2*>(in + (static_cast<size_t>(utt) * in_cap + frame) * 16 * kChannels) + tid;
    __half2 v[16];
#pragma unroll
    for (int f = 0; f < 16; ++f) v[f] = frame < valid ? src[f * (kChannels / 2)] : __half2half2(__ushort_as_half(0));
    if constexpr (Fp8) {
        float mx = 0.0f;
#pragma unroll
        for (int f = 0; f < 16; ++f) {
            const float2 m = __half22float2(__habs2(v[f]));
            mx = fmaxf(mx, fmaxf(m.x, m.y));
        }
        mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
        if (tid % 32 == 0) warp_max[tid / 32] = mx;
        __syncthreads();
        const float scale = e4m3_row_scale(fmaxf(fmaxf(warp_max[0], warp_max[1]), fmaxf(warp_max[2], warp_max[3])));
        const RowDivisor div(scale);
        if (tid == 0) out_scales[row] = scale;
        uint4* dst = reinterpret_cast<uint4*>(static_cast<uint8_t*>(out) + row * 4096 + tid * 32);
        uint32_t q[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            q[0][i] = q[1][i] = 0;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float2 a = __half22float2(v[4 * i + 2 * j]), b = __half22float2(v[4 * i + 2 * j + 1]);
                q[0][i] |= static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(div(a.x), div(b.x)), __NV_SATFINITE, __NV_E4M3)) << (16 * j);
                q[1][i] |= static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(div(a.y), div(b.y)), __NV_SATFINITE, __NV_E4M3)) << (16 * j);
            }
        }
        dst[0] = make_uint4(q[0][0], q[0][1], q[0][2], q[0][3]);
        dst[1] = make_uint4(q[1][0], q[1][1], q[1][2], q[1][3]);
    } else {
        uint4* dst = reinterpret_cast<uint4*>(static_cast<__half*>(out) + row * 4096 + tid * 32);
        uint32_t lo[8], hi[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t a = *reinterpret_cast<const uint32_t*>(&v[2 * i]), b = *reinterpret_cast<const uint32_t*>(&v[2 * i + 1]);
            lo[i] = __byte_perm(a, b, 0x5410);
            hi[i] = __byte_perm(a, b, 0x7632);
        }
        dst[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        dst[1] = make_uint4(lo[4], lo[5], lo[6], lo[7]);
        dst[2] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        dst[3] = make_uint4(hi[4], hi[5], hi[6], hi[7]);
    }
}

}  // namespace pk100

using namespace pk100;

namespace {
long long up256(long long v) { return (v + 255) / 256 * 256; }
struct Caps { int f1, f2, f3; };
Caps caps(int frames) {
    Caps c;
    c.f1 = (frames + 1) / 2;
    c.f2 = (c.f1 + 1) / 2;
    c.f3 = (c.f2 + 1) / 2;
    return c;
}
}  // namespace

extern "C" long long pk100_subsampling_workspace_bytes(int utterances, int frames, int seg_stride) {
    if (utterances <= 0 || frames <= 0 || seg_stride <= 0) return 0;
    const Caps c = caps(frames);
    const long long u = utterances;
    return 2 * up256(u * c.f2 * 32 * 256 * 2) +
           2 * up256(u * c.f3 * 16 * 256 * 2) + up256(u * seg_stride * 4096LL * 2) + 256;
}

extern "C" long long pk100_subsampling_fp8_workspace_bytes(int utterances, int frames, int seg_stride) {
    if (utterances <= 0 || frames <= 0 || seg_stride <= 0) return 0;
    const Caps c = caps(frames);
    const long long u = utterances;
    return pk100_subsampling_workspace_bytes(utterances, frames, seg_stride) +
           up256(u * c.f2 * 32 * 256) + up256(u * c.f2 * 32 * 4) + up256(u * seg_stride * 4096LL) + up256(u * seg_stride * 4);
}

static int run_subsampling(void* stream_v, const pk100_subsampling_weights* w, const pk100_subsampling_fp8* q,
                           const float* mel, int mel_stride, int utterances, int frames, const int* mel_frames,
                           void* workspace, void* output, int seg_stride, const int* row_base, int rows, int* status);

extern "C" int pk100_run_subsampling(void* stream_v, const pk100_subsampling_weights* w,
                                     const float* mel, int utterances, int frames,
                                     const int* mel_frames, void* workspace, void* output,
                                     int seg_stride, int* status) {
    return run_subsampling(stream_v, w, nullptr, mel, frames, utterances, frames, mel_frames, workspace, output, seg_stride,
                           nullptr, utterances * seg_stride, status);
}

extern "C" int pk100_run_subsampling_rows(void* stream_v, const pk100_subsampling_weights* w, const pk100_subsampling_fp8* q,
                                          const float* mel, int mel_stride, int utterances, int frames, const int* mel_frames,
                                          void* workspace, void* output, int seg_stride, const int* row_base, int rows,
                                          int* status) {
    if (q != nullptr && (!q->pw1_q || !q->pw1_scales || !q->proj_q || !q->proj_scales)) return PK100_ERR_NULL;
    if (utterances < 0 || mel_stride < frames) return PK100_ERR_SHAPE;
    if (row_base == nullptr ? rows != utterances * seg_stride : (rows <= 0 || rows % 128 != 0 || rows > utterances * seg_stride))
        return PK100_ERR_SHAPE;
    return run_subsampling(stream_v, w, q, mel, mel_stride, utterances, frames, mel_frames, workspace, output, seg_stride,
                           row_base, rows, status);
}

extern "C" int pk100_run_subsampling_fp8(void* stream_v, const pk100_subsampling_weights* w,
                                         const pk100_subsampling_fp8* q, const float* mel, int utterances,
                                         int frames, const int* mel_frames, void* workspace, void* output,
                                         int seg_stride, int* status) {
    if (!q || !q->pw1_q || !q->pw1_scales || !q->proj_q || !q->proj_scales) return PK100_ERR_NULL;
    return run_subsampling(stream_v, w, q, mel, frames, utterances, frames, mel_frames, workspace, output, seg_stride,
                           nullptr, utterances * seg_stride, status);
}

static int run_subsampling(void* stream_v, const pk100_subsampling_weights* w, const pk100_subsampling_fp8* q,
                           const float* mel, int mel_stride, int utterances, int frames, const int* mel_frames,
                           void* workspace, void* output, int seg_stride, const int* row_base, int rows, int* status) {
    if (!w || !mel || !workspace || !output) return PK100_ERR_NULL;
    if (!w->conv0_w || !w->conv0_b || !w->dw1_w || !w->dw1_b || !w->pw1_w || !w->pw1_b || !w->dw2_w ||
        !w->dw2_b || !w->pw2_w || !w->pw2_b || !w->proj_w || !w->proj_b)
        return PK100_ERR_NULL;
    if (utterances == 0) return PK100_OK;
    if (utterances < 0 || frames <= 0) return PK100_ERR_SHAPE;
    const Caps c = caps(frames);
    if (seg_stride < c.f3) return PK100_ERR_SHAPE;
    if (reinterpret_cast<uintptr_t>(workspace) & 255u) return PK100_ERR_ALIGN;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    const long long u = utterances;
    char* p = static_cast<char*>(workspace);
    auto take = [&p](long long bytes) { char* cur = p; p += up256(bytes); return cur; };
    __half* s2 = reinterpret_cast<__half*>(take(u * c.f2 * 32 * 256 * 2));
    __half* s3 = reinterpret_cast<__half*>(take(u * c.f2 * 32 * 256 * 2));
    __half* s4 = reinterpret_cast<__half*>(take(u * c.f3 * 16 * 256 * 2));
    __half* s5 = reinterpret_cast<__half*>(take(u * c.f3 * 16 * 256 * 2));
    __half* flat = reinterpret_cast<__half*>(take(u * seg_stride * 4096LL * 2));
    take(256);                                              // (slack counted by the fp16 size function)
    // E4M3 variant: quantised rows of the first depthwise output and of the flattened features
    uint8_t* q2 = q ? reinterpret_cast<uint8_t*>(take(u * c.f2 * 32 * 256)) : nullptr;
    float* q2_scales = q ? reinterpret_cast<float*>(take(u * c.f2 * 32 * 4)) : nullptr;
    uint8_t* qflat = q ? reinterpret_cast<uint8_t*>(take(u * seg_stride * 4096LL)) : nullptr;
    float* qflat_scales = q ? reinterpret_cast<float*>(take(u * seg_stride * 4)) : nullptr;

    const auto *w0 = static_cast<const __half*>(w->conv0_w), *b0 = static_cast<const __half*>(w->conv0_b);
    const auto *w1 = static_cast<const __half*>(w->dw1_w), *b1 = static_cast<const __half*>(w->dw1_b);
    // frames per CTA: whole waves over the 2 resident CTAs of every SM (a frame range takes two CTAs, one per
    // half of the features), each CTA with at most kFirstMaxFrames frames
    const long long sms = pk100_cta_budget(), total = u * c.f2, waves = (total + sms * kFirstMaxFrames - 1) / (sms * kFirstMaxFrames);
    const int run = static_cast<int>((total + sms * waves - 1) / (sms * waves));
    const dim3 first_grid((c.f2 + run - 1) / run, utterances, 32 / (2 * kFirstOuts));
    const size_t first_bytes = sizeof(float2) * kFirstPitch * first_rows(run);
    auto first_kernel = q != nullptr ? subsample_first_fused_kernel<true> : subsample_first_fused_kernel<false>;
    const cudaError_t err = cudaFuncSetAttribute(first_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 sizeof(float2) * kFirstPitch * first_rows(kFirstMaxFrames));
    if (err != cudaSuccess) return static_cast<int>(err);
    first_kernel<<<first_grid, kFirstThreads, first_bytes, stream>>>(mel, w0, b0, w1, b1, q != nullptr ? static_cast<void*>(q2) : s2,
                                                                     q2_scales, mel_stride, frames, mel_frames, c.f2, run);
    int rc = pk100_launch_status();
    if (rc != PK100_OK) return rc;

    pk100_gemm_args a{};
    a.kind = PK100_KIND_F16; a.epilogue = PK100_EPI_LINEAR;
    a.m = static_cast<int>(u * c.f2 * 32); a.n = 256; a.k = 256;
    a.a = s2; a.lda = 256; a.b = w->pw1_w; a.ldb = 256;
    a.row_scale = 1.0f; a.alpha = 1.0f; a.bias = w->pw1_b; a.act = PK100_ACT_RELU;
    a.out = s3; a.ld_out = 256; a.out_type = PK100_OUT_F16; a.out_scale = 1.0f; a.status = status;
    pk100_gemm_args first = a;
    if (q != nullptr) {
        first.kind = PK100_KIND_E4M3; first.a = q2; first.b = q->pw1_q; first.row_scales = q2_scales;
        first.col_scales = q->pw1_scales;
    }
    if ((rc = pk100_gemm_chained(stream, &first, true)) != PK100_OK) return rc;

    subsample_depthwise_kernel<<<dim3(16 / (4 * kDepthwiseRun), c.f3, utterances), 128, 0, stream>>>(
        s3, static_cast<const __half*>(w->dw2_w), static_cast<const __half*>(w->dw2_b), s4, c.f2, 32,
        c.f3, frames, mel_frames, 2);
    if ((rc = pk100_launch_status()) != PK100_OK) return rc;

    a.m = static_cast<int>(u * c.f3 * 16);
    a.a = s4; a.b = w->pw2_w; a.bias = w->pw2_b; a.out = s5;
    if ((rc = pk100_gemm_chained(stream, &a, true)) != PK100_OK) return rc;

    if (q != nullptr)
        subsample_flatten_kernel<true><<<dim3(seg_stride, utterances), 128, 0, stream>>>(s5, qflat, qflat_scales, c.f3, seg_stride,
                                                                                         frames, mel_frames, row_base);
    else
        subsample_flatten_kernel<false><<<dim3(seg_stride, utterances), 128, 0, stream>>>(s5, flat, nullptr, c.f3, seg_stride,
                                                                                          frames, mel_frames, row_base);
    if ((rc = pk100_launch_status()) != PK100_OK) return rc;

    a.m = rows; a.n = 1024; a.k = 4096;
    a.a = flat; a.lda = 4096; a.b = w->proj_w; a.ldb = 4096; a.bias = w->proj_b; a.act = PK100_ACT_NONE;
    a.out = output; a.ld_out = 1024;
    if (q != nullptr) {
        a.kind = PK100_KIND_E4M3; a.a = qflat; a.b = q->proj_q; a.row_scales = qflat_scales;
        a.col_scales = q->proj_scales;
    }
    return pk100_gemm_chained(stream, &a, true);
}
