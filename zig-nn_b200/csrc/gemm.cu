// f32 rows -> fp16 rows with a power-of-two scale per row: the operand preparation of the transposed
// quantised product (gemm_trans.cu: grad_out rows; nn_training_kernels.metal:1149-1242 is the reference's
// statement of that product).
#include "gemm_common.cuh"

namespace zq {
namespace {

// x16[m][k] = fp16(x[m][k] * 2^-e_m), post[m] = 2^e_m, with e_m chosen so that the row's largest magnitude
// lands just under 2^14 (full fp16 precision for the large elements, no overflow). A row whose largest
// magnitude is below 2^-100 (vanishing gradients) is not scaled: 2^(13 - e) would overflow, and the row's
// products are zero at f32 accuracy anyway.
// VEC: 16-byte aligned rows of a multiple of four elements; the first 8 K elements of a row stay in registers between
// the two passes (512 rows of 6912, an element at a time and twice from memory: 10.5 us for 21 MB).
template <bool VEC>
__global__ void __launch_bounds__(256)
convert_rows_f16_kernel(const float* __restrict__ x, __half* __restrict__ x16, float* __restrict__ post,
                        uint32_t K) {
    __shared__ float red[8];
    constexpr uint32_t kHeld = VEC ? 8 : 1;
    const float* row = x + (size_t)blockIdx.x * K;
    __half* out = x16 + (size_t)blockIdx.x * K;
    const float4* row4 = reinterpret_cast<const float4*>(row);
    float4 held[kHeld];
    float amax = 0.0f;
    auto take = [&](const float4& v) {
        amax = fmaxf(fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
    };
    if (VEC) {
#pragma unroll
        for (uint32_t u = 0; u < kHeld; ++u) {
            const uint32_t i = threadIdx.x + u * 256;
            held[u] = i < K / 4 ? row4[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (uint32_t u = 0; u < kHeld; ++u) take(held[u]);
        for (uint32_t i = threadIdx.x + kHeld * 256; i < K / 4; i += 256) take(row4[i]);
    } else {
        for (uint32_t i = threadIdx.x; i < K; i += blockDim.x) amax = fmaxf(amax, fabsf(row[i]));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, off));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    float a = red[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) a = fmaxf(a, red[w]);
    const int e = row_scale_exponent(a);
    const float pre = ldexpf(1.0f, -e);
    if (threadIdx.x == 0) post[blockIdx.x] = ldexpf(1.0f, e);
    if (VEC) {
        auto put = [&](uint32_t i, const float4& v) {
            const __half2 lo = __floats2half2_rn(v.x * pre, v.y * pre), hi = __floats2half2_rn(v.z * pre, v.w * pre);
            reinterpret_cast<uint2*>(out)[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        };
#pragma unroll
        for (uint32_t u = 0; u < kHeld; ++u) {
            const uint32_t i = threadIdx.x + u * 256;
            if (i < K / 4) put(i, held[u]);
        }
        for (uint32_t i = threadIdx.x + kHeld * 256; i < K / 4; i += 256) put(i, row4[i]);
    } else {
        for (uint32_t i = threadIdx.x; i < K; i += blockDim.x) out[i] = __float2half_rn(row[i] * pre);
    }
}

}  // namespace

int launch_convert_rows_f16(const float* x, __half* x16, float* post, uint32_t m_rows, uint32_t in_dim,
                            cudaStream_t st) {
    // Rows that give every thread a 16-byte access; narrower ones leave threads idle whose registers keep other rows off the
    // SM (transposed product of 4200 gradients, element by element and so: 256 columns 14.1 and 18.0 us, 768 columns 23.8
    // and 25.5, 1024 and more level or faster).
    if (((uintptr_t)x & 15) == 0 && ((uintptr_t)x16 & 7) == 0 && in_dim % 4 == 0 && in_dim >= 1024)
        convert_rows_f16_kernel<true><<<m_rows, 256, 0, st>>>(x, x16, post, in_dim);
    else
        convert_rows_f16_kernel<false><<<m_rows, 256, 0, st>>>(x, x16, post, in_dim);
    ZQ_LAUNCH_CHECK();
    return ZQ_OK;
}

}  // namespace zq
