// Activations as block fixed point, in the order the int8 tensor-core kernels' B fragments want (see qmv_imma.cuh for the
// arithmetic): made once per row where several blocks of a kernel use the same rows.
#pragma once

#include "common.cuh"
#include "qmv_imma.cuh"

namespace iq {

// Row r of an activation matrix as block fixed point: per group of 64 inputs 128 bytes, the high digits' fragments of the
// four lanes of a quad (16 bytes each: two MMAs) and the low digits', and {2^(e-15), sum}.
struct FixedRows {
    unsigned char* digits;  // [rows][groups][2][4][16]
    float2* scale;          // [rows][groups]
};

// Eight consecutive inputs (word w8 of the group's eight) of a row's group: the eight threads of a group are eight
// neighbouring lanes. See qmv_imma.cuh for the arithmetic.
__device__ __forceinline__ void fixed_point_unit(const float (&v)[8], int w8, unsigned char* digits, float2* scale) {
    float amax = 0.f, sum = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        amax = fmaxf(amax, fabsf(v[k]));
        sum += v[k];
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
    }
    float sc, inv;
    qi_group_scale<8>(amax, sum, sc, inv);
    if (digits == nullptr) return;
    if (w8 == 0) *scale = make_float2(sc, sum);
    uint32_t hi_w[2], lo_w[2];
    qi_digits8<false, 8>(v, inv, hi_w, lo_w);
    unsigned char* f = digits + (w8 >> 1) * 16 + (w8 & 1) * 8;
    *reinterpret_cast<uint2*>(f) = make_uint2(hi_w[0], hi_w[1]);
    *reinterpret_cast<uint2*>(f + 64) = make_uint2(lo_w[0], lo_w[1]);
}

// One row of D inputs (starting at element `start` of x) by `threads` threads, a multiple of 32.
__device__ __forceinline__ void fixed_point_row(const void* x, int32_t x_dtype, size_t start, int D, const FixedRows& fx, int row, int tid, int threads) {
    const int units = D / 8, upad = (units + 31) / 32 * 32;
    for (int u = tid; u < upad; u += threads) {
        const bool live = u < units;
        float v[8];
        load_x8(x, x_dtype, start + (live ? u : 0) * 8, v);
        const size_t g = (size_t)row * (D / 64) + (live ? u : 0) / 8;
        fixed_point_unit(v, u & 7, live ? fx.digits + g * 128 : nullptr, fx.scale + g);
    }
}

}  // namespace iq
