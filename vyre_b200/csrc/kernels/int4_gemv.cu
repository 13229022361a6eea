// Decode linear for group-quantized int4 weights (batch <= 8 per pass): which kernel takes a shape, and the generic kernel.
//
//   y[m, n] = cast( sum_k x[m, k] * (q[n, k] - 8) * s[n, k / group] )
//
// Replaces the generated scalar kernel of vyre-libs/src/nn/linear/inner/linear_4bit.rs:399-775 (one warp per
// output, 4-byte loads, scalar f32 FMA) for the row-major layout of
// vyre-primitives/src/math/quantized/programs.rs:186-300.
#include <cuda_bf16.h>

#include "dependent_launch.cuh"
#include "kernels.h"

namespace vybk {
namespace {

// ---- fallback: any group size dividing k, any batch; warp per output row, plain 32-bit loads -------------------
__global__ void __launch_bounds__(256) int4_linear_generic_kernel(const uint16_t* x,
                                                                 const uint32_t* w,
                                                                 const uint16_t* scales, void* y,
                                                                 uint32_t m, uint32_t n, uint32_t k, uint32_t group,
                                                                 uint32_t out_f32) {
    dependent_start();
    const uint32_t row = blockIdx.x * 8 + (threadIdx.x >> 5);
    const uint32_t lane = threadIdx.x & 31;
    if (row >= n) return;
    const uint32_t words = k / 8, groups = k / group;
    for (uint32_t b0 = 0; b0 < m; b0 += 4) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (uint32_t wi = lane; wi < words; wi += 32) {
            const uint32_t word = w[size_t(row) * words + wi];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t kk = wi * 8 + i;
                const float s = __uint_as_float(uint32_t(scales[size_t(row) * groups + kk / group]) << 16);
                const float wv = float(int((word >> (4 * i)) & 0xF) - 8) * s;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (b0 + j < m) acc[j] = fmaf(__uint_as_float(uint32_t(x[size_t(b0 + j) * k + kk]) << 16), wv, acc[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float v = acc[j];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0 && b0 + j < m) {
                if (out_f32)
                    static_cast<float*>(y)[size_t(b0 + j) * n + row] = v;
                else
                    static_cast<__nv_bfloat16*>(y)[size_t(b0 + j) * n + row] = __float2bfloat16_rn(v);
            }
        }
    }
}

}  // namespace

bool int4_gemv_supported(uint32_t m, uint32_t n, uint32_t k, uint32_t group) {
    return m >= 1 && m <= 8 && n >= 1 && group == 128 && k >= 1024 && k % 1024 == 0;
}

cudaError_t launch_int4_gemv(const void* x_bf16, const void* w_packed, const void* scale_bf16, void* y, uint32_t m,
                             uint32_t n, uint32_t k, uint32_t out_f32, int sm_count, cudaStream_t stream,
                             uint32_t* status, bool constant_weights) {
    const size_t out_elem = out_f32 ? 4 : 2;
    const uint32_t step = out_f32 ? 1 : 4;  // rows per launch of the half-SM kernel: f32 outputs get the single-row precision
    // Rows of 6144, 8192, ... (multiples of 2048 beyond 4096): the half-SM kernel per k block, sums carried in f32. More bf16 rows
    // than one launch of it takes: one launch on the tensor cores with the weights in tensor memory, which reads them once (4096 x
    // 14336 at 8 rows: 13.7 us against 26.6 us). f32 outputs stay: the integer sums of a group are exact, the tensor cores' are
    // not (activations of widely different size, relative error against 64-bit sums: 0.8e-7 against 1.4 to 2.0e-7).
    if (int4_gemv_kblocks_supported(1, n, k, 128)) {
        if (!out_f32 && m > 4 && int4_skinny_supported(x_bf16, w_packed, scale_bf16, m, n, k, 128))
            return launch_int4_skinny(x_bf16, w_packed, scale_bf16, y, m, n, k, 0, sm_count, stream, status, constant_weights);
        for (uint32_t b0 = 0; b0 < m; b0 += step) {
            const uint32_t mb = m - b0 < step ? m - b0 : step;
            cudaError_t e = launch_int4_gemv_kblocks(static_cast<const uint16_t*>(x_bf16) + size_t(b0) * k, w_packed, scale_bf16,
                                                     static_cast<uint8_t*>(y) + size_t(b0) * n * out_elem, mb, n, k, out_f32,
                                                     sm_count, stream, constant_weights);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    // Whole rows of 2048 or 4096 k. Three to eight batch rows (f32 outputs: from two rows): one launch on the f16 tensor path, eight
    // batch rows per MMA
    if (m >= (out_f32 ? 2u : 3u) && int4_gemv_batch8_supported(m, n, k, 128))
        return launch_int4_gemv_batch8(x_bf16, w_packed, scale_bf16, y, m, n, k, out_f32, sm_count, stream, constant_weights);
    // ... fewer: the half-SM kernel, whose launches overlap on every SM (26-bit block-floating activations, 57-bit for a single row)
    if (int4_gemv_halfsm_supported(1, n, k, 128)) {
        for (uint32_t b0 = 0; b0 < m; b0 += step) {
            const uint32_t mb = m - b0 < step ? m - b0 : step;
            cudaError_t e = launch_int4_gemv_halfsm(static_cast<const uint16_t*>(x_bf16) + size_t(b0) * k, w_packed, scale_bf16,
                                                    static_cast<uint8_t*>(y) + size_t(b0) * n * out_elem, mb, n, k, out_f32,
                                                    sm_count, stream, status, constant_weights);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    // Other k (odd multiples of 1024). bf16 outputs: the tensor-memory kernel (14336 x 5120 at 8 rows: 16.5 us against 47.5 us of the
    // bulk-copy kernel, 4096 x 11264 at one row: 11.9 against 22.7 us), except where a row is one k block of the bulk-copy kernel and every SM has
    // one 16-row tile of it at most: there it needs no cluster reduction (2048 x 1024 at one row 6.4 against 8.3 us, at eight 7.3 against
    // 7.9; 2048 x 3072 at one row 6.4 against 8.5, but 8.3 against 7.6 at 128 x 3072 and four). f32 outputs: the bulk-copy kernel, for its exact
    // group sums (activations of widely different size: error 0.6 to 1.0e-7 against 1.1 to 2.9e-7).
    const bool small = n <= 16 * uint32_t(sm_count) && (k == 1024 || (k == 3072 && m <= 2));
    if (!out_f32 && !small && int4_skinny_supported(x_bf16, w_packed, scale_bf16, m, n, k, 128))
        return launch_int4_skinny(x_bf16, w_packed, scale_bf16, y, m, n, k, 0, sm_count, stream, status, constant_weights);
    return launch_int4_gemv_bulk(x_bf16, w_packed, scale_bf16, y, m, n, k, out_f32, sm_count, stream, status, constant_weights);
}

cudaError_t launch_int4_linear_generic(const void* x_bf16, const void* w_packed, const void* scale_bf16, void* y,
                                       uint32_t m, uint32_t n, uint32_t k, uint32_t group, uint32_t out_f32,
                                       cudaStream_t stream) {
    return launch_dependent(int4_linear_generic_kernel, dim3((n + 7) / 8), dim3(256), 0, stream, static_cast<const uint16_t*>(x_bf16),
                            static_cast<const uint32_t*>(w_packed), static_cast<const uint16_t*>(scale_bf16), y, m, n, k, group, out_f32);
}

}  // namespace vybk

