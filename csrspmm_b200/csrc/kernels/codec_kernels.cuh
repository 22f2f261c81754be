// e2m1 value codec on the device: the same format, scale rule and rounding as the host codec
// (csrspmm_b200_e2m1_scale / _encode / _decode), for values that already live on the GPU.
// No counterpart in the reference, whose "Fp4" kernels take fp32 values
// (src/device/csrspmm_warp_per_row_fp4.cu:9-19).
#pragma once

#include "common.cuh"

namespace csrspmm_b200 {

// One CTA takes chunks of kCodecThreads * kCodecPer elements, every thread 16 of them, four 16-byte loads in
// flight (arrays that do not start on 16 bytes: plain loads).
constexpr int kCodecThreads = 256;
constexpr int kCodecPer = 16;
constexpr int kCodecMaxCtas = kSms * 4;

// 16 values from position i0 on (0 beyond n)
__device__ __forceinline__ void load_codec(long long n, const float* __restrict__ values, long long i0, float (&v)[kCodecPer])
{
    if (i0 + kCodecPer <= n && (reinterpret_cast<uintptr_t>(values) & 15u) == 0) {
#pragma unroll
        for (int q = 0; q < kCodecPer / 4; ++q) {
            const float4 x = __ldg(reinterpret_cast<const float4*>(values + i0) + q);
            v[4 * q] = x.x, v[4 * q + 1] = x.y, v[4 * q + 2] = x.z, v[4 * q + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int q = 0; q < kCodecPer; ++q) v[q] = i0 + q < n ? __ldg(values + i0 + q) : 0.0f;
    }
}

__device__ __forceinline__ float codec_block_max(float mx)
{
    __shared__ float warp_max[kCodecThreads / 32];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = mx;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kCodecThreads / 32; ++w) mx = fmaxf(mx, warp_max[w]);
    return mx;
}

// max |v| of each CTA's share, NaNs ignored
__global__ void __launch_bounds__(kCodecThreads) e2m1_absmax_kernel(long long n, const float* __restrict__ values,
                                                                    float* __restrict__ cta_max)
{
    wait_for_previous_grid();
    release_next_grid();
    float mx = 0.0f;
    const long long stride = (long long)gridDim.x * (kCodecThreads * kCodecPer);
    for (long long i = ((long long)blockIdx.x * kCodecThreads + threadIdx.x) * kCodecPer; i < n; i += stride) {
        float v[kCodecPer];
        load_codec(n, values, i, v);
#pragma unroll
        for (int q = 0; q < kCodecPer; ++q) {
            const float a = fabsf(v[q]);
            if (a > mx) mx = a;  // false for NaN
        }
    }
    mx = codec_block_max(mx);
    if (threadIdx.x == 0) cta_max[blockIdx.x] = mx;
}

// nearest code point, ties to the even code, saturating at 6, sign kept, NaN -> +0
__device__ __forceinline__ unsigned e2m1_encode_one(float v, float scale)
{
    if (v != v) return 0u;
    const float q = __fdiv_rn(v, scale);
    const unsigned s = (__float_as_uint(q) >> 31) ? 8u : 0u;
    const float a = fabsf(q);
    // midpoints between the magnitudes 0, .5, 1, 1.5, 2, 3, 4, 6; a tie goes down when the lower code is even
    unsigned code = 7u;
    if (a < 0.25f || a == 0.25f) code = 0u;
    else if (a < 0.75f) code = 1u;
    else if (a < 1.25f || a == 1.25f) code = 2u;
    else if (a < 1.75f) code = 3u;
    else if (a < 2.5f || a == 2.5f) code = 4u;
    else if (a < 3.5f) code = 5u;
    else if (a < 5.0f || a == 5.0f) code = 6u;
    return s | code;
}

// Largest magnitude whose code is k or less, k = 0 .. 6: the same answer as a division per value, which is monotone, for a dozen
// instructions less (16 M values with the search for the scale: 71 -> 51 us).  The magnitude between codes k and k + 1 times the scale is a unit in the last
// place or two away from it.  Scales that the product would leave the range with (kCodecScaleMin .. Max): division.
constexpr float kCodecScaleMin = 1.17549435e-38f, kCodecScaleMax = 4.0e37f;

__device__ __forceinline__ float e2m1_last_of_code(int k, float scale)
{
    const float middle = k < 2 ? 0.25f + 0.5f * k : k < 4 ? 1.25f + 0.5f * (k - 2) : k < 6 ? 2.5f + (k - 4) : 5.0f;
    int bits = __float_as_int(__fmul_rn(middle, scale));
    while (bits > 0 && e2m1_encode_one(__int_as_float(bits), scale) > (unsigned)k) --bits;
    while (e2m1_encode_one(__int_as_float(bits + 1), scale) <= (unsigned)k) ++bits;
    return __int_as_float(bits);
}

// The codes of 16 elements per thread and step, 8 bytes at a time.  The scale is the argument, or
// (cta_max given) follows from the maxima a previous kernel left, in which case CTA 0 reports its bits.
__global__ void __launch_bounds__(kCodecThreads) e2m1_encode_kernel(long long n, const float* __restrict__ values, float scale,
                                                                    const float* __restrict__ cta_max, int num_max,
                                                                    unsigned char* __restrict__ packed, long long* scale_bits)
{
    wait_for_previous_grid();
    release_next_grid();
    if (cta_max != nullptr) {
        float mx = 0.0f;
        for (int k = threadIdx.x; k < num_max; k += kCodecThreads) mx = fmaxf(mx, cta_max[k]);
        mx = codec_block_max(mx);
        scale = mx > 0.0f ? __fdiv_rn(mx, 6.0f) : 1.0f;
        if (blockIdx.x == 0 && threadIdx.x == 0) *scale_bits = (long long)__float_as_uint(scale);
    }
    __shared__ float last_of_code[7];
    const bool by_limits = scale >= kCodecScaleMin && scale <= kCodecScaleMax;
    if (by_limits && threadIdx.x < 7) last_of_code[threadIdx.x] = e2m1_last_of_code(threadIdx.x, scale);
    __syncthreads();
    float last[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) last[k] = last_of_code[k];
    auto code_of = [&](float v) {
        if (!by_limits) return e2m1_encode_one(v, scale);
        unsigned code = (__float_as_uint(v) >> 28) & 8u;
#pragma unroll
        for (int k = 0; k < 7; ++k) code += fabsf(v) > last[k];
        return v == v ? code : 0u;
    };
    const long long stride = (long long)gridDim.x * (kCodecThreads * kCodecPer);
    const bool wide = (reinterpret_cast<uintptr_t>(packed) & 7u) == 0;
    for (long long i = ((long long)blockIdx.x * kCodecThreads + threadIdx.x) * kCodecPer; i < n; i += stride) {
        float v[kCodecPer];
        load_codec(n, values, i, v);
        unsigned word[2] = {0u, 0u};  // elements beyond n are 0: code 0
#pragma unroll
        for (int q = 0; q < kCodecPer; ++q) word[q >> 3] |= (i + q < n ? code_of(v[q]) : 0u) << (4 * (q & 7));
        if (wide && i + kCodecPer <= n) {
            *reinterpret_cast<uint2*>(packed + (i >> 1)) = make_uint2(word[0], word[1]);
        } else {
#pragma unroll
            for (int q = 0; q < kCodecPer; q += 2)
                if (i + q < n) packed[(i + q) >> 1] = (unsigned char)(word[q >> 3] >> (4 * (q & 7)));
        }
    }
}

__global__ void __launch_bounds__(256) e2m1_decode_kernel(long long n, const unsigned char* __restrict__ packed,
                                                          float scale, float* __restrict__ values)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const unsigned byte = __ldg(packed + (i >> 1));
        values[i] = decode_e2m1((i & 1) ? (byte >> 4) : (byte & 15u), scale);
    }
}

}  // namespace csrspmm_b200
