// One LayerNorm row by one warp with the row held in registers (d = NV * 128): the body of ln_reg_kernel
// (elementwise.cu), shared with the kernels that normalise rows they have just completed (gemm_skinny.cu).
// Mean and variance are accumulated in double like the reference's layer_norm_f (src/encoder.c:25-37):
// y = ((x - mu) * inv) * w + b. L2: read the row past the L1 (it was written by other CTAs of the same launch).
#pragma once
#include "common.cuh"
#include "gemm.h"

namespace mb {

// int8 row by the reference's activation rule (quantize_act_int8, src/qmat.c:186-202)
__device__ __forceinline__ int8_t act_q8(float y, float inv) {
    const float v = __fmul_rn(y, inv);
    int q = (int)(v >= 0.0f ? __fadd_rn(v, 0.5f) : __fsub_rn(v, 0.5f));
    q = q > 127 ? 127 : (q < -127 ? -127 : q);
    return (int8_t)q;
}

// Mean and 1 / sqrt(variance + eps) of a row of K values from a lane's part of it (column of four lane + 32 j is v[j]), in double
// like the reference. One pass over differences from the row's first value: a large mean costs nothing, and since that value
// is one of the row's, its own distance is at most sqrt(K) deviations, so the subtraction of s^2 / K loses at most log2 K of
// the 53 bits. Both sums go through one exchange and there is one rsqrt: the dependent double operations, the divisions and
// the square root of the two-pass form took 4000 cycles of a warp (a LayerNorm launch of one row 6.6 us).
template <int NV>
__device__ __forceinline__ void ln_stats(const float4 (&v)[NV], int K, float &muf, float &inv) {
    const double x0 = (double)__shfl_sync(0xffffffffu, v[0].x, 0), rk = 1.0 / (double)K;
    double s0 = 0.0, s1 = 0.0, q0 = 0.0, q1 = 0.0;
#pragma unroll
    for (int j = 0; j < NV; j++) {
        const double a = (double)v[j].x - x0, b = (double)v[j].y - x0, c = (double)v[j].z - x0, d = (double)v[j].w - x0;
        s0 += a + b; s1 += c + d;
        q0 = fma(a, a, q0); q1 = fma(b, b, q1); q0 = fma(c, c, q0); q1 = fma(d, d, q1);
    }
    double s = s0 + s1, q = q0 + q1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { s += __shfl_xor_sync(0xffffffffu, s, o); q += __shfl_xor_sync(0xffffffffu, q, o); }
    const double m = s * rk, ve = fma(-s, m, q) * rk + 1e-5;
    muf = (float)(x0 + m);
    inv = (float)rsqrt(ve);
}

// weight and bias of a lane's columns
template <int NV>
struct LnVectors {
    float4 w[NV], b[NV];
    __device__ __forceinline__ void load(const float *__restrict__ pw, const float *__restrict__ pb, int lane) {
#pragma unroll
        for (int j = 0; j < NV; j++) { w[j] = reinterpret_cast<const float4 *>(pw)[lane + 32 * j]; b[j] = reinterpret_cast<const float4 *>(pb)[lane + 32 * j]; }
    }
};

// Every step over the whole row before the next one, the choice of outputs outside of the loops, neighbours converted in pairs,
// and (ln_reg_kernel) weight and bias on their way before the kernels in front have ended: with the outputs chosen value by
// value a voice command took 1.940 ms instead of 1.837 (85 of its 267 launches are LayerNorms), 15 s on 24 layers 6.09 instead
// of 5.74, eight utterances with int8 activations 5.80 instead of 5.40.
template <int NV, bool L2>
__device__ __forceinline__ void ln_row(const float *__restrict__ x, const LnVectors<NV> &p, float *__restrict__ out, __half *__restrict__ hi,
                                       __half *__restrict__ lo, int8_t *__restrict__ q8, float *__restrict__ sx8, int row, int act, int lane) {
    constexpr int d = NV * 128;
    const float4 *xr = reinterpret_cast<const float4 *>(x + (size_t)row * d) + lane;
    float4 v[NV];
#pragma unroll
    for (int j = 0; j < NV; j++) v[j] = L2 ? __ldcg(xr + 32 * j) : xr[32 * j];
    float muf, inv;
    ln_stats<NV>(v, d, muf, inv);
#pragma unroll
    for (int j = 0; j < NV; j++)            // the finished values replace the inputs in the registers
        v[j] = make_float4(((v[j].x - muf) * inv) * p.w[j].x + p.b[j].x, ((v[j].y - muf) * inv) * p.w[j].y + p.b[j].y,
                           ((v[j].z - muf) * inv) * p.w[j].z + p.b[j].z, ((v[j].w - muf) * inv) * p.w[j].w + p.b[j].w);
    if (act == ACT_SILU)
#pragma unroll
        for (int j = 0; j < NV; j++) v[j] = make_float4(silu_f(v[j].x), silu_f(v[j].y), silu_f(v[j].z), silu_f(v[j].w));
    if (q8) {
        float amax = 0.0f;
#pragma unroll
        for (int j = 0; j < NV; j++) amax = fmaxf(fmaxf(amax, fmaxf(fabsf(v[j].x), fabsf(v[j].y))), fmaxf(fabsf(v[j].z), fabsf(v[j].w)));
        amax = warp_max(amax);
        const float qinv = amax > 0.0f ? 127.0f / amax : 0.0f;
        if (lane == 0) sx8[row] = amax > 0.0f ? amax / 127.0f : 0.0f;
        char4 *o = reinterpret_cast<char4 *>(q8 + (size_t)row * d) + lane;
#pragma unroll
        for (int j = 0; j < NV; j++) o[32 * j] = make_char4(act_q8(v[j].x, qinv), act_q8(v[j].y, qinv), act_q8(v[j].z, qinv), act_q8(v[j].w, qinv));
    }
    if (out) {
        float4 *o = reinterpret_cast<float4 *>(out + (size_t)row * d) + lane;
#pragma unroll
        for (int j = 0; j < NV; j++) o[32 * j] = v[j];
    }
    if (!hi) return;
    uint2 *ph = reinterpret_cast<uint2 *>(hi + (size_t)row * d) + lane, *pl = reinterpret_cast<uint2 *>(lo + (size_t)row * d) + lane;
    uint2 h[NV], l[NV];
#pragma unroll
    for (int j = 0; j < NV; j++) split_h16x4(v[j], h[j], l[j]);
#pragma unroll
    for (int j = 0; j < NV; j++) ph[32 * j] = h[j];
    if (lo)
#pragma unroll
        for (int j = 0; j < NV; j++) pl[32 * j] = l[j];
}
template <int NV, bool L2>
__device__ __forceinline__ void ln_row(const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ b,
                                       float *__restrict__ out, __half *__restrict__ hi, __half *__restrict__ lo, int8_t *__restrict__ q8,
                                       float *__restrict__ sx8, int row, int act, int lane) {
    LnVectors<NV> p;
    p.load(w, b, lane);
    ln_row<NV, L2>(x, p, out, hi, lo, q8, sx8, row, act, lane);
}

}  // namespace mb
