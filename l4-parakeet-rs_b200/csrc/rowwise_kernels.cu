// Memory-bound row-wise operators of the FastConformer block for sm_100a:
// LayerNorm (+ fused quantisers), activation / weight quantisers, masked GLU,
// depthwise conv + BatchNorm + SiLU (+ fused per-row E4M3 packing).
// One warp owns one 1024-wide row: 16-byte vector loads, the row stays in
// registers between the statistics passes, reductions are warp shuffles.
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>

#include <atomic>

#include "pk100_internal.h"
#include "ptx_sm100.cuh"
#include "row_quant.cuh"

namespace pk100 {

constexpr int kWidth = 1024;

__device__ __forceinline__ float warp_sum_all(float v) {
#pragma unroll
    for (int off = 16; off > 0; off /= 2) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

__device__ __forceinline__ float warp_max_all(float v) {
#pragma unroll
    for (int off = 16; off > 0; off /= 2) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}

__device__ __forceinline__ void unpack8(const uint4& raw, float (&f)[8]) {
    const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 p = __half22float2(h[i]);
        f[2 * i] = p.x;
        f[2 * i + 1] = p.y;
    }
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    uint4 raw;
    __half2* h = reinterpret_cast<__half2*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
    return raw;
}

__device__ __forceinline__ uint2 e4m3x8(const float (&f)[8]) {
    uint2 out;
    out.x = __nv_cvt_float2_to_fp8x2(make_float2(f[0], f[1]), __NV_SATFINITE, __NV_E4M3) |
            (static_cast<uint32_t>(
                 __nv_cvt_float2_to_fp8x2(make_float2(f[2], f[3]), __NV_SATFINITE, __NV_E4M3)) << 16);
    out.y = __nv_cvt_float2_to_fp8x2(make_float2(f[4], f[5]), __NV_SATFINITE, __NV_E4M3) |
            (static_cast<uint32_t>(
                 __nv_cvt_float2_to_fp8x2(make_float2(f[6], f[7]), __NV_SATFINITE, __NV_E4M3)) << 16);
    return out;
}

__device__ __forceinline__ int clamp_s8(float v) { return max(-127, min(127, __float2int_rn(v))); }

__device__ __forceinline__ uint2 s8x8(const float (&f)[8]) {
    uint2 out;
    out.x = (clamp_s8(f[0]) & 255) | ((clamp_s8(f[1]) & 255) << 8) | ((clamp_s8(f[2]) & 255) << 16) |
            ((clamp_s8(f[3]) & 255) << 24);
    out.y = (clamp_s8(f[4]) & 255) | ((clamp_s8(f[5]) & 255) << 8) | ((clamp_s8(f[6]) & 255) << 16) |
            ((clamp_s8(f[7]) & 255) << 24);
    return out;
}

// Row geometry of a batch of utterances concatenated along the row axis:
// segment s owns rows [s*seg_stride, (s+1)*seg_stride); its first `valid` rows
// carry data (seg_valid[s] when given, else the uniform `valid_rows`).
__device__ __forceinline__ int segment_valid(const int* seg_valid, int seg, int valid_rows) {
    return seg_valid != nullptr ? seg_valid[seg] : valid_rows;
}

// Where a row lies in its utterance.  Uniform batches: segment s owns rows [s*seg_stride, (s+1)*seg_stride),
// its first seg_valid[s] (or the uniform valid_rows) rows carry data.  Packed batches: `tiles` gives per
// 128-row tile the first row of the utterance it belongs to and that utterance's row count.
__device__ __forceinline__ bool row_live(const pk100_rows& g, int row) {
    if (g.tiles != nullptr) {
        const int2 t = __ldg(g.tiles + row / 128);
        return row - t.x < t.y;
    }
    const int seg = row / g.seg_stride;
    return row - seg * g.seg_stride < segment_valid(g.seg_valid, seg, g.valid_rows);
}

// ------------------------------------------------------------- LayerNorm
// gamma and beta of this lane's 32 columns (column i * 256 + lane * 8 + j), packed
struct NormVectors {
    uint4 g[4], b[4];
    // `volatile`: stays where it is written, so that the second norm's vectors are fetched per row (from L1)
    // and not held across the row loop beside the first norm's.  (The pair form spills 112 to 128 bytes a
    // thread at its 128 registers all the same.)
    static __device__ __forceinline__ uint4 fetch(const __half* p) {
        uint4 v;
        asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
        return v;
    }
    __device__ __forceinline__ void load(const __half* gamma, const __half* beta, int lane) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            g[i] = fetch(gamma + i * 256 + lane * 8);
            b[i] = fetch(beta + i * 256 + lane * 8);
        }
    }
};

// Normalise one row held as 4 x 8 values per lane; the results are rounded to fp16 (`h`, packed) and
// left in x.  The order of the sums (a lane's 32 values in column order, then the butterfly) is fixed.
__device__ __forceinline__ void normalise_row(float (&x)[4][8], uint4 (&h)[4], const NormVectors& v, float eps) {
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) sum += x[i][j];
    const float mean = warp_sum_all(sum) * (1.0f / kWidth);
    float sq = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            x[i][j] -= mean;
            sq = fmaf(x[i][j], x[i][j], sq);
        }
    const float rstd = rsqrtf(warp_sum_all(sq) * (1.0f / kWidth) + eps);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float g[8], b[8];
        unpack8(v.g[i], g);
        unpack8(v.b[i], b);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[i][j] = fmaf(x[i][j] * rstd, g[j], b[j]);
        h[i] = pack8(x[i]);
        unpack8(h[i], x[i]);
    }
}

// bits of the row's largest |value| from the packed fp16 values, those of a NaN where the row has one
__device__ __forceinline__ unsigned row_absmax_bits(const uint4 (&h)[4]) {
    __half2 mx = __habs2(*reinterpret_cast<const __half2*>(&h[0].x));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t w[4] = {h[i].x, h[i].y, h[i].z, h[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) mx = __hmax2_nan(mx, __habs2(*reinterpret_cast<const __half2*>(&w[j])));
    }
    // non-negative floats order like their bits, infinity and then NaN last
    const float2 m = __half22float2(mx);
    return __reduce_max_sync(0xffffffffu, max(__float_as_uint(m.x), __float_as_uint(m.y)));
}

// four INT8 codes rne(q) of |q| <= 127 (no NaN) in one word: adding 1.5 * 2^23 leaves the integer in the low mantissa bits
__device__ __forceinline__ uint32_t codes_s8x4(float a, float b, float c, float d) {
    constexpr float kMagic = 12582912.0f;
    const uint32_t lo = __byte_perm(__float_as_uint(a + kMagic), __float_as_uint(b + kMagic), 0x0040);
    const uint32_t hi = __byte_perm(__float_as_uint(c + kMagic), __float_as_uint(d + kMagic), 0x0040);
    return __byte_perm(lo, hi, 0x5410);
}

// Write one normalised row in the requested encoding (x is used up).
template <int Mode>
__device__ __forceinline__ void emit_row(float (&x)[4][8], const uint4 (&h)[4], float inv_scale,
                                         void* out, float* scales, size_t row, int lane) {
    if constexpr (Mode == PK100_LN_F16) {
        __half* o = reinterpret_cast<__half*>(out) + row * kWidth;
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(o + i * 256 + lane * 8) = h[i];
        return;
    }
    uint8_t* o = reinterpret_cast<uint8_t*>(out) + row * kWidth;
    if constexpr (Mode == PK100_LN_S4_ROW) {
        // every signed 4-bit code is used: the scale is the larger of max/7 and -min/8
        float mx = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) mx = fmaxf(mx, fmaxf(__fdiv_rn(x[i][j], 7.0f), __fdiv_rn(-x[i][j], 8.0f)));
        mx = warp_max_all(mx);
        const float scale = mx > 0.0f ? mx : 1.0f;
        if (lane == 0) scales[row] = scale;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t w[2] = {0u, 0u};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int q = max(-8, min(7, __float2int_rn(__fdiv_rn(x[i][j], scale))));
                w[j / 4] |= static_cast<uint32_t>(q & 255) << (8 * (j % 4));
            }
            *reinterpret_cast<uint2*>(o + i * 256 + lane * 8) = make_uint2(w[0], w[1]);
        }
    } else if constexpr (Mode == PK100_LN_E4M3_FIXED) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float q[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) q[j] = x[i][j] * inv_scale;
            *reinterpret_cast<uint2*>(o + i * 256 + lane * 8) = e4m3x8(q);
        }
    } else {
        float mx = __uint_as_float(row_absmax_bits(h));
        if (!isfinite(mx)) {                               // (the whole warp or none of it)
            // the maximum is taken over what is a number; INT8 codes of NaN and of infinity / infinity are 0
            float top = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    top = fmaxf(top, fabsf(x[i][j]));
                    if (Mode == PK100_LN_S8_ROW && !isfinite(x[i][j])) x[i][j] = 0.0f;
                }
            mx = warp_max_all(top);
        }
        const float scale = mx > 0.0f ? __fdiv_rn(mx, Mode == PK100_LN_E4M3_ROW ? 448.0f : 127.0f) : 1.0f;
        if (lane == 0) scales[row] = scale;
        const RowDivisor div(scale);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float q[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) q[j] = div(x[i][j]);
            *reinterpret_cast<uint2*>(o + i * 256 + lane * 8) = Mode == PK100_LN_S8_ROW
                ? make_uint2(codes_s8x4(q[0], q[1], q[2], q[3]), codes_s8x4(q[4], q[5], q[6], q[7])) : e4m3x8(q);
        }
    }
}

template <int Mode>
__device__ __forceinline__ void emit_zero_row(void* out, float* scales, size_t row, int lane) {
    if constexpr (Mode == PK100_LN_F16) {
        __half* o = reinterpret_cast<__half*>(out) + row * kWidth;
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(o + i * 256 + lane * 8) = make_uint4(0, 0, 0, 0);
    } else {
        // (8 bytes at a time like the codes of a live row: the output need not be aligned to more)
        uint8_t* o = reinterpret_cast<uint8_t*>(out) + row * kWidth;
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<uint2*>(o + i * 256 + lane * 8) = make_uint2(0, 0);
        if (scales != nullptr && lane == 0) scales[row] = 1.0f;      // (fixed scale: only where the caller gives an array)
    }
}

// One warp per row, walking the rows of the grid; the next row is requested before the current one is
// reduced.  Mode / Mode2: PK100_LN_*.  Mode2 >= 0: a second LayerNorm is applied to the f16-rounded
// first result and written to out2 (the "pair" form: block-output norm + next block's first norm in
// one pass over the row).  Bound by HBM for large row counts (45 056 rows, 138 MB: INT8 57 -> 38 us, E4M3 43 -> 31 us, pair 69 -> 54 us against one row per
// warp with full divisions and gamma / beta fetched per row) and by the latency of
// load, two reductions and store for a few hundred rows.
template <int Mode, int Mode2>
__global__ void __launch_bounds__(256, 2)
layer_norm_kernel(const __half* __restrict__ in, const __half* __restrict__ gamma,
                  const __half* __restrict__ beta, void* __restrict__ out, float* scales, float inv_scale,
                  const __half* __restrict__ gamma2, const __half* __restrict__ beta2, void* __restrict__ out2,
                  float* scales2, float inv_scale2, int total_rows, const pk100_rows geometry, float eps) {
    const int lane = threadIdx.x % 32;
    const int first = blockIdx.x * 8 + threadIdx.x / 32, step = gridDim.x * 8;
    grid_dependents_launch();
    grid_dependency_wait();
    NormVectors v;
    v.load(gamma, beta, lane);
    uint4 raw[4];
    auto request = [&](int row) {
        const uint4* src = reinterpret_cast<const uint4*>(in + static_cast<size_t>(row) * kWidth) + lane;
#pragma unroll
        for (int i = 0; i < 4; ++i) raw[i] = src[i * 32];
    };
    if (first < total_rows) request(first);
    for (int row = first; row < total_rows; row += step) {
        float x[4][8];
#pragma unroll
        for (int i = 0; i < 4; ++i) unpack8(raw[i], x[i]);
        if (row + step < total_rows) request(row + step);
        if (!row_live(geometry, row)) {
            emit_zero_row<Mode>(out, scales, row, lane);
            if constexpr (Mode2 >= 0) emit_zero_row<Mode2>(out2, scales2, row, lane);
            continue;
        }
        uint4 h[4];
        normalise_row(x, h, v, eps);
        emit_row<Mode>(x, h, inv_scale, out, scales, row, lane);
        if constexpr (Mode2 >= 0) {
            NormVectors v2;
            v2.load(gamma2, beta2, lane);
            normalise_row(x, h, v2, eps);
            emit_row<Mode2>(x, h, inv_scale2, out2, scales2, row, lane);
        }
    }
}

// ------------------------------------------------- 2:4 structured sparsity of E4M3 activations
// The reference's FF2 input format (kernels/sm89/encoder.cu:685-704, :1037-1054): per four
// consecutive bytes the two largest 7-bit magnitudes are kept, ties to the lower index.
// Returns the two kept bytes (low 16 bits, index order) and their 2-bit indices (bits 16-19).
__device__ __forceinline__ uint32_t compress_quartet(uint32_t packed) {
    uint32_t data = 0, meta = 0;
    int count = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t mag = (packed >> (8 * i)) & 127u;
        int rank = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t other = (packed >> (8 * j)) & 127u;
            rank += (other > mag || (other == mag && j < i)) ? 1 : 0;
        }
        if (rank < 2) {
            data |= ((packed >> (8 * i)) & 255u) << (8 * count);
            meta |= static_cast<uint32_t>(i) << (2 * count);
            ++count;
        }
    }
    return data | (meta << 16);
}

__device__ __forceinline__ uint32_t expand_quartet(uint32_t two_bytes, uint32_t meta4) {
    return ((two_bytes & 255u) << (8 * (meta4 & 3u))) | (((two_bytes >> 8) & 255u) << (8 * ((meta4 >> 2) & 3u)));
}

// mode 0: dense -> dense with the dropped bytes zeroed; 1: dense -> data [rows, cols/2] + metadata
// [rows, cols/8] behind it; 2: that layout -> dense.  One thread per 16 dense bytes (4 quartets).
__global__ void sparse24_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, int rows, int cols,
                                int mode) {
    const size_t chunk = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t chunks_per_row = static_cast<size_t>(cols) / 16;
    if (chunk >= chunks_per_row * rows) return;
    const size_t row = chunk / chunks_per_row, c16 = chunk % chunks_per_row;
    const size_t data_bytes = static_cast<size_t>(rows) * (cols / 2);
    if (mode == 2) {
        const uint2 data = *reinterpret_cast<const uint2*>(in + row * (cols / 2) + c16 * 8);
        const uint32_t meta = *reinterpret_cast<const uint16_t*>(in + data_bytes + row * (cols / 8) + c16 * 2);
        uint4 dense;
        dense.x = expand_quartet(data.x & 0xFFFFu, meta & 15u);
        dense.y = expand_quartet(data.x >> 16, (meta >> 4) & 15u);
        dense.z = expand_quartet(data.y & 0xFFFFu, (meta >> 8) & 15u);
        dense.w = expand_quartet(data.y >> 16, (meta >> 12) & 15u);
        *reinterpret_cast<uint4*>(out + row * cols + c16 * 16) = dense;
        return;
    }
    const uint4 v = *reinterpret_cast<const uint4*>(in + row * cols + c16 * 16);
    const uint32_t words[4] = {v.x, v.y, v.z, v.w};
    uint32_t packed[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) packed[i] = compress_quartet(words[i]);
    if (mode == 0) {
        uint4 dense;
        dense.x = expand_quartet(packed[0] & 0xFFFFu, packed[0] >> 16);
        dense.y = expand_quartet(packed[1] & 0xFFFFu, packed[1] >> 16);
        dense.z = expand_quartet(packed[2] & 0xFFFFu, packed[2] >> 16);
        dense.w = expand_quartet(packed[3] & 0xFFFFu, packed[3] >> 16);
        *reinterpret_cast<uint4*>(out + row * cols + c16 * 16) = dense;
    } else {
        uint2 data;
        data.x = (packed[0] & 0xFFFFu) | (packed[1] << 16);
        data.y = (packed[2] & 0xFFFFu) | (packed[3] << 16);
        *reinterpret_cast<uint2*>(out + row * (cols / 2) + c16 * 8) = data;
        const uint32_t meta = (packed[0] >> 16) | ((packed[1] >> 16) << 4) | ((packed[2] >> 16) << 8) |
                              ((packed[3] >> 16) << 12);
        *reinterpret_cast<uint16_t*>(out + data_bytes + row * (cols / 8) + c16 * 2) = static_cast<uint16_t>(meta);
    }
}

// Packed INT4 codes (low nibble = even index, two's complement) -> one INT8 byte per code.
__global__ void unpack_s4_kernel(const uint8_t* __restrict__ packed, int8_t* __restrict__ out, size_t bytes) {
    const size_t i = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) * 4;
    if (i + 4 <= bytes) {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(packed + i);
        uint32_t lo = 0, hi = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int byte = (w >> (8 * b)) & 255;
            const int even = (byte & 15) >= 8 ? (byte & 15) - 16 : (byte & 15);
            const int odd = (byte >> 4) >= 8 ? (byte >> 4) - 16 : (byte >> 4);
            const uint32_t pair = static_cast<uint32_t>(even & 255) | (static_cast<uint32_t>(odd & 255) << 8);
            if (b < 2) lo |= pair << (16 * b); else hi |= pair << (16 * (b - 2));
        }
        *reinterpret_cast<uint2*>(out + 2 * i) = make_uint2(lo, hi);
    } else {
        for (size_t j = i; j < bytes; ++j) {
            const int byte = packed[j];
            out[2 * j] = static_cast<int8_t>((byte & 15) >= 8 ? (byte & 15) - 16 : (byte & 15));
            out[2 * j + 1] = static_cast<int8_t>((byte >> 4) >= 8 ? (byte >> 4) - 16 : (byte >> 4));
        }
    }
}

// ------------------------------------------------------------ quantisers
__global__ void quantize_fixed_kernel(const __half* __restrict__ in, uint8_t* __restrict__ out,
                                      size_t elements, float inv_scale, int to_s8) {
    const size_t i = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) * 8;
    if (i + 8 <= elements) {
        float f[8];
        unpack8(*reinterpret_cast<const uint4*>(in + i), f);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] *= inv_scale;
        *reinterpret_cast<uint2*>(out + i) = to_s8 ? s8x8(f) : e4m3x8(f);
    } else {
        for (size_t j = i; j < elements; ++j) {
            const float v = __half2float(in[j]) * inv_scale;
            out[j] = to_s8 ? static_cast<uint8_t>(clamp_s8(v) & 255)
                           : static_cast<uint8_t>(__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3));
        }
    }
}

// Per-row weight packers, run once at load.  One CTA per output row.
// format: 0 E4M3 (absmax/448), 1 S8 (absmax/127), 2 S4 per row (max(v/7,-v/8), -8..7),
//         3 S4 with one fp16 scale per 128 K (absmax/7, -7..7; scales [K/128, N]).
__global__ void __launch_bounds__(256)
pack_weight_rows_kernel(const __half* __restrict__ w, int n, int k, int ldw, int format,
                        uint8_t* __restrict__ out, float* __restrict__ scales,
                        __half* __restrict__ group_scales) {
    __shared__ float s_part[8];
    __shared__ float s_scale;
    const int row = blockIdx.x;
    const int tid = threadIdx.x;
    const __half* src = w + static_cast<size_t>(row) * ldw;
    if (format == 3) {
        // one warp per group of 128
        const int warp = tid / 32, lane = tid % 32;
        for (int g = warp; g < k / 128; g += 8) {
            float v[4];
            float mx = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[j] = __half2float(src[g * 128 + lane * 4 + j]);
                mx = fmaxf(mx, fabsf(v[j]));
            }
            mx = warp_max_all(mx);
            __half s16 = __float2half_rn(mx > 0.0f ? __fdiv_rn(mx, 7.0f) : 1.0f);
            float s = __half2float(s16);
            if (!(s > 0.0f)) { s = 1.0f; s16 = __float2half_rn(1.0f); }
            if (lane == 0) group_scales[static_cast<size_t>(g) * n + row] = s16;
            int q[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) q[j] = max(-7, min(7, __float2int_rn(__fdiv_rn(v[j], s))));
            const uint16_t packed = static_cast<uint16_t>((q[0] & 15) | ((q[1] & 15) << 4) |
                                                          ((q[2] & 15) << 8) | ((q[3] & 15) << 12));
            *reinterpret_cast<uint16_t*>(out + static_cast<size_t>(row) * (k / 2) + g * 64 + lane * 2) =
                packed;
        }
        return;
    }
    float mx = 0.0f;
    for (int c = tid; c < k; c += 256) {
        const float v = __half2float(src[c]);
        mx = fmaxf(mx, format == 2 ? fmaxf(__fdiv_rn(v, 7.0f), __fdiv_rn(-v, 8.0f)) : fabsf(v));
    }
    mx = warp_max_all(mx);
    if (tid % 32 == 0) s_part[tid / 32] = mx;
    __syncthreads();
    if (tid == 0) {
        float m = 0.0f;
        for (int i = 0; i < 8; ++i) m = fmaxf(m, s_part[i]);
        float s;
        if (format == 0) s = m > 0.0f ? __fdiv_rn(m, 448.0f) : 1.0f;
        else if (format == 1) s = m > 0.0f ? __fdiv_rn(m, 127.0f) : 1.0f;
        else s = m > 0.0f ? m : 1.0f;
        s_scale = s;
        scales[row] = s;
    }
    __syncthreads();
    const float s = s_scale;
    if (format == 2) {
        for (int c = tid * 2; c < k; c += 512) {
            const int a = max(-8, min(7, __float2int_rn(__fdiv_rn(__half2float(src[c]), s))));
            const int b = max(-8, min(7, __float2int_rn(__fdiv_rn(__half2float(src[c + 1]), s))));
            out[static_cast<size_t>(row) * (k / 2) + c / 2] =
                static_cast<uint8_t>((a & 15) | ((b & 15) << 4));
        }
    } else {
        for (int c = tid; c < k; c += 256) {
            const float v = __fdiv_rn(__half2float(src[c]), s);
            out[static_cast<size_t>(row) * k + c] = format == 1
                ? static_cast<uint8_t>(clamp_s8(v) & 255)
                : static_cast<uint8_t>(__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3));
        }
    }
}

// INT4 group-128 codes -> fp16 weights W[n,k] = f16(code * scale[k/128, n]).
__global__ void dequant_w4g128_kernel(const uint8_t* __restrict__ codes,
                                      const __half* __restrict__ group_scales, int n, int k,
                                      __half* __restrict__ out) {
    const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;   // byte index
    const size_t total = static_cast<size_t>(n) * (k / 2);
    if (idx >= total) return;
    const int row = static_cast<int>(idx / (k / 2));
    const int kk = static_cast<int>(idx % (k / 2)) * 2;
    const float s = __half2float(group_scales[static_cast<size_t>(kk / 128) * n + row]);
    const uint8_t b = codes[idx];
    int lo = b & 15, hi = b >> 4;
    lo = lo >= 8 ? lo - 16 : lo;
    hi = hi >= 8 ? hi - 16 : hi;
    *reinterpret_cast<__half2*>(out + static_cast<size_t>(row) * k + kk) =
        __floats2half2_rn(static_cast<float>(lo) * s, static_cast<float>(hi) * s);
}

// ------------------------------------------------------------------- GLU
__global__ void glu_masked_kernel(const __half* __restrict__ in, __half* __restrict__ out,
                                  int total_rows, int seg_stride, int valid_rows,
                                  const int* __restrict__ seg_valid) {
    const size_t idx = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) * 8;
    if (idx >= static_cast<size_t>(total_rows) * kWidth) return;
    const int row = static_cast<int>(idx / kWidth);
    const int col = static_cast<int>(idx % kWidth);
    const int seg = row / seg_stride;
    uint4 result = make_uint4(0, 0, 0, 0);
    if (row - seg * seg_stride < segment_valid(seg_valid, seg, valid_rows)) {
        float a[8], g[8], r[8];
        unpack8(*reinterpret_cast<const uint4*>(in + static_cast<size_t>(row) * 2 * kWidth + col), a);
        unpack8(*reinterpret_cast<const uint4*>(in + static_cast<size_t>(row) * 2 * kWidth + kWidth + col), g);
#pragma unroll
        for (int j = 0; j < 8; ++j) r[j] = __fdividef(a[j], 1.0f + __expf(-g[j]));
        result = pack8(r);
    }
    *reinterpret_cast<uint4*>(out + idx) = result;
}

// ------------------------------------------------- depthwise + BN + SiLU
// One CTA = 256 threads x 4 channels = all 1024 channels of a strip of kStrip rows; the 8 halo rows come
// from L2.  Two neighbouring channels share every packed fp32 instruction (fma.rn.f32x2 and friends,
// each half rounds like the scalar one).  A window of 9 rows slides down the strip in registers;
// the row's E4M3 scale takes one warp reduction and one exchange through shared memory; scale and divisor of eight
// rows are formed once per warp, a row per lane, and handed round by shuffles (every thread
// formed them for every row before).  Long strips read
// fewer halo rows, short ones keep every SM busy: 16 rows where that gives the device two CTAs per SM,
// else 8 (strips of 32 rows: 77 -> 75 us at 45 056 rows, 42.7 -> 44.7 at 24 576).  Bound by issue slots
// (convolution, BatchNorm, SiLU and E4M3 rounding of every element).  us, divisors per thread / per lane: 94.4 / 77.2
// at 45 056 rows, 16.6 / 13.7 at 6144, 5.8 / 5.0 at 768, 4.7 / 4.0 at 128 (155 at 45 056 with scalar instructions and
// full divisions).
template <bool Quantize, int kStrip>
__global__ void __launch_bounds__(256, 2)
depthwise_bn_silu_kernel(const __half* __restrict__ in, const __half* __restrict__ wdw,
                         const float* __restrict__ bn_gamma, const float* __restrict__ bn_beta,
                         const float* __restrict__ bn_mean, const float* __restrict__ bn_var,
                         void* __restrict__ out, float* __restrict__ row_scales, const pk100_rows geometry, float eps) {
    __shared__ float s_max[kStrip / 8][8][8];
    grid_dependents_launch();
    grid_dependency_wait();
    const int tid = threadIdx.x;
    const int lane = tid % 32, warp = tid / 32;
    const int c0 = tid * 4;
    size_t base;                                       // first row of the utterance
    int r0, rows, stride;                              // this strip's first row in it, its valid rows, its block
    if (geometry.tiles != nullptr) {
        const int2 t = __ldg(geometry.tiles + blockIdx.x / (128 / kStrip));
        base = t.x;
        r0 = blockIdx.x * kStrip - t.x;
        rows = t.y;
        stride = r0 + kStrip;                          // tiles are whole
    } else {
        const int strips = (geometry.seg_stride + kStrip - 1) / kStrip, seg = blockIdx.x / strips;
        base = static_cast<size_t>(seg) * geometry.seg_stride;
        r0 = (blockIdx.x % strips) * kStrip;
        rows = segment_valid(geometry.seg_valid, seg, geometry.valid_rows);
        stride = geometry.seg_stride;
    }

    // this thread's 4 x 9 taps are 72 contiguous bytes (8-byte aligned): 9 vector loads
    Pair w[9][2], rstd[2], gam[2], add[2], neg_mean[2];
    {
        alignas(8) __half taps[36];
        const uint2* src = reinterpret_cast<const uint2*>(wdw + static_cast<size_t>(c0) * 9);
#pragma unroll
        for (int i = 0; i < 9; ++i) reinterpret_cast<uint2*>(taps)[i] = __ldg(src + i);
#pragma unroll
        for (int t = 0; t < 9; ++t)
#pragma unroll
            for (int c = 0; c < 2; ++c) w[t][c] = pair_of(__half2float(taps[(2 * c) * 9 + t]), __half2float(taps[(2 * c + 1) * 9 + t]));
        const float4 var = __ldg(reinterpret_cast<const float4*>(bn_var + c0));
        const float4 g4 = __ldg(reinterpret_cast<const float4*>(bn_gamma + c0));
        const float4 b4 = __ldg(reinterpret_cast<const float4*>(bn_beta + c0));
        const float4 m4 = __ldg(reinterpret_cast<const float4*>(bn_mean + c0));
        rstd[0] = pair_of(rsqrtf(var.x + eps), rsqrtf(var.y + eps)); rstd[1] = pair_of(rsqrtf(var.z + eps), rsqrtf(var.w + eps));
        gam[0] = pair_of(g4.x, g4.y); gam[1] = pair_of(g4.z, g4.w);
        add[0] = pair_of(b4.x, b4.y); add[1] = pair_of(b4.z, b4.w);
        neg_mean[0] = pair_of(-m4.x, -m4.y); neg_mean[1] = pair_of(-m4.z, -m4.w);
    }

    // rows r0 - 4 .. of the window arrive as packed halves; the strip's loads are issued 8 rows at a time
    auto load_row = [&](int r) {
        return r >= 0 && r < rows ? *reinterpret_cast<const uint2*>(in + (base + r) * kWidth + c0) : make_uint2(0, 0);
    };
    auto widen = [&](uint2 raw, Pair (&dst)[2]) {
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
        dst[0] = pair_of(a.x, a.y);
        dst[1] = pair_of(b.x, b.y);
    };
    Pair win[9][2];
    uint2 ahead[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) ahead[t] = load_row(r0 - 4 + t);
#pragma unroll
    for (int t = 0; t < 8; ++t) widen(ahead[t], win[t + 1]);            // slots 1..8 = rows r0-4..r0+3
#pragma unroll
    for (int t = 0; t < 8; ++t) ahead[t] = load_row(r0 + 4 + t);

#pragma unroll 1
    for (int blk = 0; blk < kStrip / 8; ++blk) {
        __half2 y[8][2];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = r0 + blk * 8 + i;
            // slide: drop the oldest row, take row r + 4
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                win[t][0] = win[t + 1][0];
                win[t][1] = win[t + 1][1];
            }
            widen(ahead[i], win[8]);
            if (blk + 1 < kStrip / 8) ahead[i] = load_row(r + 12);
            __half2 top = __half2half2(__ushort_as_half(0));
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                Pair acc = 0ull;
#pragma unroll
                for (int t = 0; t < 9; ++t) acc = pair_fma(win[t][c], w[t][c], acc);
                acc = pair_fma(pair_mul(pair_add(acc, neg_mean[c]), rstd[c]), gam[c], add[c]);
                const float2 v = halves_of(acc);
                y[i][c] = __floats2half2_rn(__fdividef(v.x, 1.0f + __expf(-v.x)), __fdividef(v.y, 1.0f + __expf(-v.y)));
                if (r >= rows) y[i][c] = __half2half2(__ushort_as_half(0));
                top = __hmax2(top, __habs2(y[i][c]));
            }
            if constexpr (Quantize) {
                const float2 m = __half22float2(top);
                // non-negative floats order like their bits
                const unsigned mx = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(m.x, m.y)));
                if (lane == 0) s_max[blk][i][warp] = __uint_as_float(mx);
            }
        }
        RowDivisor mine(1.0f, 1.0f);                   // lane j: that of row j mod 8 of the block
        if constexpr (Quantize) {
            __syncthreads();
            const int row = lane % 8;
            const float4 a = *reinterpret_cast<const float4*>(&s_max[blk][row][0]), b = *reinterpret_cast<const float4*>(&s_max[blk][row][4]);
            const float mx = fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)), fmaxf(fmaxf(b.x, b.y), fmaxf(b.z, b.w)));
            const float scale = mx > 0.0f ? __fdiv_rn(mx, 448.0f) : 1.0f;
            mine = RowDivisor(scale);
            if (tid < 8 && r0 + blk * 8 + tid < stride) row_scales[base + r0 + blk * 8 + tid] = scale;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = r0 + blk * 8 + i;
            if (r >= stride) continue;                 // the same for the whole CTA
            const size_t grow = base + r;
            if constexpr (Quantize) {
                const RowDivisor div(__shfl_sync(0xffffffffu, mine.s, i), __shfl_sync(0xffffffffu, mine.y, i));
                const float2 p = __half22float2(y[i][0]), q = __half22float2(y[i][1]);
                const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(div(p.x), div(p.y)), __NV_SATFINITE, __NV_E4M3);
                const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(div(q.x), div(q.y)), __NV_SATFINITE, __NV_E4M3);
                *reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(out) + grow * kWidth + c0) = lo | (hi << 16);
            } else {
                uint2 raw;
                raw.x = *reinterpret_cast<const uint32_t*>(&y[i][0]);
                raw.y = *reinterpret_cast<const uint32_t*>(&y[i][1]);
                *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(out) + grow * kWidth + c0) = raw;
            }
        }
    }
}

}  // namespace pk100

// ------------------------------------------------------------ C-ABI entry
using namespace pk100;

// Rows per launch beyond one per resident warp are walked by the same warps.
template <int Mode, int Mode2>
static int launch_layer_norm(void* stream, const void* input, const void* gamma, const void* beta, void* output, float* scales,
                             float inv_scale, const void* gamma2, const void* beta2, void* output2, float* scales2,
                             float inv_scale2, int total_rows, const pk100_rows& geometry, float eps, bool dependent = true) {
    auto kernel = layer_norm_kernel<Mode, Mode2>;
    static std::atomic<int> resident{0};                   // CTAs per SM
    if (resident.load(std::memory_order_relaxed) == 0) {
        int per_sm = 0;
        const cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, 0);
        if (err != cudaSuccess) return static_cast<int>(err);
        resident.store(per_sm > 0 ? per_sm : 1, std::memory_order_relaxed);
    }
    const int blocks = (total_rows + 7) / 8, cap = pk100_cta_budget() * resident.load(std::memory_order_relaxed);
    pk100_launch(dependent, kernel, dim3(blocks < cap ? blocks : cap), dim3(256), 0, static_cast<cudaStream_t>(stream),
        static_cast<const __half*>(input), static_cast<const __half*>(gamma), static_cast<const __half*>(beta), output, scales,
        inv_scale, static_cast<const __half*>(gamma2), static_cast<const __half*>(beta2), output2, scales2, inv_scale2,
        total_rows, geometry, eps);
    return pk100_launch_status();
}

int pk100_layer_norm_rows(void* stream, const void* input, const void* gamma, const void* beta, void* output, float* scales,
                          int mode, float inv_scale, int total_rows, const pk100_rows& geometry, float eps, bool dependent) {
#define PK_LN(M) case M: return launch_layer_norm<M, -1>(stream, input, gamma, beta, output, scales, inv_scale, nullptr, \
                                                         nullptr, nullptr, nullptr, 0.0f, total_rows, geometry, eps, dependent)
    switch (mode) {
    PK_LN(PK100_LN_F16); PK_LN(PK100_LN_E4M3_FIXED); PK_LN(PK100_LN_E4M3_ROW); PK_LN(PK100_LN_S8_ROW); PK_LN(PK100_LN_S4_ROW);
    default: return PK100_ERR_SHAPE;
    }
#undef PK_LN
}

int pk100_layer_norm_pair_rows(void* stream, const void* input, const void* gamma, const void* beta, void* output,
                               const void* next_gamma, const void* next_beta, void* next_output, float* next_scales,
                               int next_mode, float next_inv_scale, int total_rows, const pk100_rows& geometry, float eps) {
#define PK_LN(M) case M: return launch_layer_norm<PK100_LN_F16, M>(stream, input, gamma, beta, output, nullptr, 0.0f, next_gamma, \
                                                                   next_beta, next_output, next_scales, next_inv_scale, total_rows, geometry, eps)
    switch (next_mode) {
    PK_LN(PK100_LN_F16); PK_LN(PK100_LN_E4M3_FIXED); PK_LN(PK100_LN_E4M3_ROW); PK_LN(PK100_LN_S8_ROW); PK_LN(PK100_LN_S4_ROW);
    default: return PK100_ERR_SHAPE;
    }
#undef PK_LN
}

extern "C" int pk100_layer_norm(void* stream, const void* input, const void* gamma,
                                const void* beta, void* output, float* scales, int mode,
                                float inv_scale, int total_rows, int seg_stride, int valid_rows,
                                const int* seg_valid, float eps) {
    if (!input || !gamma || !beta || !output) return PK100_ERR_NULL;
    if (total_rows <= 0) return total_rows == 0 ? PK100_OK : PK100_ERR_SHAPE;
    if (seg_stride <= 0 || mode < 0 || mode > PK100_LN_S4_ROW) return PK100_ERR_SHAPE;
    if (mode >= PK100_LN_E4M3_ROW && !scales) return PK100_ERR_NULL;
    return pk100_layer_norm_rows(stream, input, gamma, beta, output, scales, mode, inv_scale, total_rows,
                                 pk100_rows{nullptr, seg_stride, valid_rows, seg_valid}, eps);
}

extern "C" int pk100_layer_norm_pair(void* stream, const void* input, const void* gamma,
                                     const void* beta, void* output, const void* next_gamma,
                                     const void* next_beta, void* next_output, float* next_scales,
                                     int next_mode, float next_inv_scale, int total_rows,
                                     int seg_stride, int valid_rows, const int* seg_valid,
                                     float eps) {
    if (!input || !gamma || !beta || !output || !next_gamma || !next_beta || !next_output)
        return PK100_ERR_NULL;
    if (total_rows <= 0) return total_rows == 0 ? PK100_OK : PK100_ERR_SHAPE;
    if (seg_stride <= 0 || next_mode < 0 || next_mode > PK100_LN_S4_ROW) return PK100_ERR_SHAPE;
    if (next_mode >= PK100_LN_E4M3_ROW && !next_scales)
        return PK100_ERR_NULL;
    return pk100_layer_norm_pair_rows(stream, input, gamma, beta, output, next_gamma, next_beta, next_output, next_scales,
                                      next_mode, next_inv_scale, total_rows,
                                      pk100_rows{nullptr, seg_stride, valid_rows, seg_valid}, eps);
}

extern "C" int pk100_quantize_fp8_fixed(void* stream, const void* input, void* output,
                                        long long elements, float inverse_scale) {
    if (!input || !output) return PK100_ERR_NULL;
    if (elements <= 0) return elements == 0 ? PK100_OK : PK100_ERR_SHAPE;
    const long long threads = (elements + 7) / 8;
    quantize_fixed_kernel<<<static_cast<unsigned>((threads + 255) / 256), 256, 0,
                            static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half*>(input), static_cast<uint8_t*>(output),
        static_cast<size_t>(elements), inverse_scale, 0);
    return pk100_launch_status();
}

extern "C" int pk100_quantize_int8(void* stream, const void* input, void* output,
                                   float inverse_scale, long long elements) {
    if (!input || !output) return PK100_ERR_NULL;
    if (elements <= 0) return elements == 0 ? PK100_OK : PK100_ERR_SHAPE;
    const long long threads = (elements + 7) / 8;
    quantize_fixed_kernel<<<static_cast<unsigned>((threads + 255) / 256), 256, 0,
                            static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half*>(input), static_cast<uint8_t*>(output),
        static_cast<size_t>(elements), inverse_scale, 1);
    return pk100_launch_status();
}

extern "C" int pk100_pack_weight_rows(void* stream, const void* weight, int n, int k, int ldw,
                                      int format, void* packed, float* scales,
                                      void* group_scales) {
    if (!weight || !packed) return PK100_ERR_NULL;
    if (n <= 0 || k <= 0 || ldw < k || format < 0 || format > 3) return PK100_ERR_SHAPE;
    if (format == 3 && group_scales == nullptr) return PK100_ERR_NULL;
    if (format != 3 && scales == nullptr) return PK100_ERR_NULL;
    if (format == 3 && k % 128 != 0) return PK100_ERR_SHAPE;
    if (format == 2 && k % 2 != 0) return PK100_ERR_SHAPE;
    pack_weight_rows_kernel<<<n, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half*>(weight), n, k, ldw, format, static_cast<uint8_t*>(packed),
        scales, static_cast<__half*>(group_scales));
    return pk100_launch_status();
}

extern "C" int pk100_dequant_w4g128(void* stream, const void* codes, const void* group_scales,
                                    int n, int k, void* weight_f16) {
    if (!codes || !group_scales || !weight_f16) return PK100_ERR_NULL;
    if (n <= 0 || k <= 0 || k % 128 != 0) return PK100_ERR_SHAPE;
    const size_t total = static_cast<size_t>(n) * (k / 2);
    dequant_w4g128_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0,
                            static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint8_t*>(codes), static_cast<const __half*>(group_scales), n, k,
        static_cast<__half*>(weight_f16));
    return pk100_launch_status();
}

extern "C" int pk100_unpack_s4(void* stream, const void* packed, void* codes, long long packed_bytes) {
    if (!packed || !codes) return PK100_ERR_NULL;
    if (packed_bytes < 0) return PK100_ERR_SHAPE;
    if (packed_bytes == 0) return PK100_OK;
    if ((reinterpret_cast<uintptr_t>(packed) & 3u) || (reinterpret_cast<uintptr_t>(codes) & 7u)) return PK100_ERR_ALIGN;
    const size_t threads = (static_cast<size_t>(packed_bytes) + 3) / 4;
    unpack_s4_kernel<<<static_cast<unsigned>((threads + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint8_t*>(packed), static_cast<int8_t*>(codes), static_cast<size_t>(packed_bytes));
    return pk100_launch_status();
}

static int sparse24_launch(void* stream, const void* input, void* output, int rows, int cols, int mode) {
    if (!input || !output) return PK100_ERR_NULL;
    if (rows < 0 || cols <= 0 || cols % 16 != 0) return PK100_ERR_SHAPE;
    if (rows == 0) return PK100_OK;
    if ((reinterpret_cast<uintptr_t>(input) | reinterpret_cast<uintptr_t>(output)) & 15u) return PK100_ERR_ALIGN;
    const size_t chunks = static_cast<size_t>(rows) * (cols / 16);
    sparse24_kernel<<<static_cast<unsigned>((chunks + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint8_t*>(input), static_cast<uint8_t*>(output), rows, cols, mode);
    return pk100_launch_status();
}

extern "C" int pk100_prune_2of4_e4m3(void* stream, const void* dense, void* pruned, int rows, int cols) {
    return sparse24_launch(stream, dense, pruned, rows, cols, 0);
}
extern "C" int pk100_compress_2of4_e4m3(void* stream, const void* dense, void* compressed, int rows, int cols) {
    return sparse24_launch(stream, dense, compressed, rows, cols, 1);
}
extern "C" int pk100_decompress_2of4_e4m3(void* stream, const void* compressed, void* dense, int rows, int cols) {
    return sparse24_launch(stream, compressed, dense, rows, cols, 2);
}

extern "C" int pk100_glu_masked(void* stream, const void* input, void* output, int total_rows,
                                int seg_stride, int valid_rows, const int* seg_valid) {
    if (!input || !output) return PK100_ERR_NULL;
    if (total_rows <= 0) return total_rows == 0 ? PK100_OK : PK100_ERR_SHAPE;
    if (seg_stride <= 0) return PK100_ERR_SHAPE;
    const size_t threads = static_cast<size_t>(total_rows) * kWidth / 8;
    glu_masked_kernel<<<static_cast<unsigned>((threads + 255) / 256), 256, 0,
                        static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half*>(input), static_cast<__half*>(output), total_rows, seg_stride,
        valid_rows, seg_valid);
    return pk100_launch_status();
}

int pk100_depthwise_bn_silu_rows(void* stream, const void* input, const void* dw_weight, const float* bn_gamma, const float* bn_beta,
                                 const float* bn_mean, const float* bn_var, void* output, float* row_scales, int quantize,
                                 int total_rows, int segments, const pk100_rows& geometry, float eps) {
    if (!input || !dw_weight || !bn_gamma || !bn_beta || !bn_mean || !bn_var || !output || (quantize && !row_scales))
        return PK100_ERR_NULL;
    auto misaligned = [](const void* ptr, uintptr_t mask) { return (reinterpret_cast<uintptr_t>(ptr) & mask) != 0; };
    if (misaligned(dw_weight, 7) || misaligned(bn_gamma, 15) || misaligned(bn_beta, 15) ||
        misaligned(bn_mean, 15) || misaligned(bn_var, 15) || misaligned(input, 7))
        return PK100_ERR_ALIGN;      // the kernel reads taps 8 bytes and BatchNorm vectors 16 bytes at a time
    auto launch = [&](auto kernel, int strip) {
        const int per_segment = geometry.tiles != nullptr ? 0 : (geometry.seg_stride + strip - 1) / strip;
        const int blocks = geometry.tiles != nullptr ? total_rows / strip : segments * per_segment;
        pk100_launch_chained(kernel, dim3(blocks), dim3(256), 0, static_cast<cudaStream_t>(stream),
            static_cast<const __half*>(input), static_cast<const __half*>(dw_weight), bn_gamma, bn_beta, bn_mean, bn_var, output,
            row_scales, geometry, eps);
        return pk100_launch_status();
    };
    const bool wide = total_rows >= 2 * pk100_cta_budget() * 16;
    if (quantize) return wide ? launch(depthwise_bn_silu_kernel<true, 16>, 16) : launch(depthwise_bn_silu_kernel<true, 8>, 8);
    return wide ? launch(depthwise_bn_silu_kernel<false, 16>, 16) : launch(depthwise_bn_silu_kernel<false, 8>, 8);
}

extern "C" int pk100_depthwise_bn_silu(void* stream, const void* input, const void* dw_weight,
                                       const float* bn_gamma, const float* bn_beta,
                                       const float* bn_mean, const float* bn_var, void* output,
                                       float* row_scales, int quantize, int segments,
                                       int seg_stride, int valid_rows, const int* seg_valid,
                                       float eps) {
    if (!input || !dw_weight || !bn_gamma || !bn_beta || !bn_mean || !bn_var || !output || (quantize && !row_scales))
        return PK100_ERR_NULL;
    if (segments <= 0) return segments == 0 ? PK100_OK : PK100_ERR_SHAPE;
    if (seg_stride <= 0) return PK100_ERR_SHAPE;
    return pk100_depthwise_bn_silu_rows(stream, input, dw_weight, bn_gamma, bn_beta, bn_mean, bn_var, output, row_scales, quantize,
                                        segments * seg_stride, segments, pk100_rows{nullptr, seg_stride, valid_rows, seg_valid}, eps);
}
