// Activations as block fixed point, in the order the int8 tensor-core kernels' B fragments want (see qmv_imma.cuh for the
// arithmetic): made once per row where several blocks of a kernel use the same rows.
#pragma once

#include "common.cuh"
#include "qmv_imma.cuh"

namespace iq {

// Row r of an activation matrix as block fixed point: per group of 64 inputs 128 bytes, the high digits' fragments of the
// four lanes of a quad (16 bytes each: two MMAs) and the low digits', and {2^(e-15), sum}. The wide form has a third digit (23 bits,
// see qi_digits23) and 192 bytes.
struct FixedRows {
    unsigned char* digits;  // [rows][groups][2 or 3][4][16]
    float2* scale;          // [rows][groups]
};

// Eight consecutive inputs (word w8 of the group's eight) of a row's group: the eight threads of a group are eight
// neighbouring lanes. See qmv_imma.cuh for the arithmetic.
template <bool WIDE>
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
    uint32_t d[3][2];
    if (WIDE) qi_digits23<false>(v, inv, d);
    else qi_digits8<false, 8>(v, inv, d[0], d[1]);
    unsigned char* f = digits + (w8 >> 1) * 16 + (w8 & 1) * 8;
#pragma unroll
    for (int i = 0; i < (WIDE ? 3 : 2); i++) *reinterpret_cast<uint2*>(f + 64 * i) = make_uint2(d[i][0], d[i][1]);
}

// One row of D inputs (starting at element `start` of x) by `threads` threads, a multiple of 32.
template <bool WIDE>
__device__ __forceinline__ void fixed_point_row(const void* x, int32_t x_dtype, size_t start, int D, const FixedRows& fx, int row, int tid, int threads) {
    const int units = D / 8, upad = (units + 31) / 32 * 32;
    for (int u = tid; u < upad; u += threads) {
        const bool live = u < units;
        float v[8];
        load_x8(x, x_dtype, start + (live ? u : 0) * 8, v);
        const size_t g = (size_t)row * (D / 64) + (live ? u : 0) / 8;
        fixed_point_unit<WIDE>(v, u & 7, live ? fx.digits + g * (WIDE ? 192 : 128) : nullptr, fx.scale + g);
    }
}

}  // namespace iq
