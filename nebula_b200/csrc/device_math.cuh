// Scalar device helpers shared by every kernel: the reference's activation
// functions and TF32 rounding.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/nebula_b200.h"

namespace nb {

// Programmatic dependent launch.  The first call of every kernel lets the next one on the stream become resident while
// this one runs (its set-up, its first weight tiles); grid_dependency_wait returns when every earlier kernel is
// complete and its writes are visible.  A kernel waits before its first access to anything an earlier kernel
// writes or reads, its own stores included; every thread block passes the wait, so completion is transitive.
__device__ __forceinline__ void grid_dependents_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_begin() {
    grid_dependents_start();
    grid_dependency_wait();
}

// Round-to-nearest conversion of an fp32 value to TF32 (10-bit mantissa), kept
// in fp32 storage with the low 13 mantissa bits cleared.  The tensor core reads
// only the upper 19 bits of each operand, so pre-rounded data makes its result
// independent of how it treats the dropped bits.
__device__ __forceinline__ float round_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// exp in double without branches, so that several of them overlap: the argument is reduced by Cody and Waite's split of ln 2
// to |r| <= 0.35, the exponential of r is its Taylor polynomial of degree 12 (the rest is at most 2.1 * 2^-53 of it), and the power of
// two is added to the exponent.  Arguments are cut to +-708, where the result is still a normal number: the callers add it to 1,
// or compare against where exp overflows themselves.  NaN stays NaN.
// The library's exp and division branch on their special cases, which puts the chains of a thread's values one behind the
// other: the tanh layer of 512 x 256 x 256 took 17.4 us with them, 15.2 with these; 2^24 values by themselves 45 and 39.
__device__ __forceinline__ double exp_for_activation(double z) {
    z = z > 708.0 ? 708.0 : z;
    z = z < -708.0 ? -708.0 : z;
    const double big = 6755399441055744.0;              // 1.5 * 2^52: adding it leaves the nearest integer in the low bits
    const double kb = fma(z, 1.4426950408889634, big), k = kb - big;
    double r = fma(k, -0.6931471805598903, z);     // ln 2 to 42 bits: k times it is exact
    r = fma(k, -5.497923018708371e-14, r);             // and the rest
    double p = 1.0 / 479001600.0;
    p = fma(p, r, 1.0 / 39916800.0);
    p = fma(p, r, 1.0 / 3628800.0);
    p = fma(p, r, 1.0 / 362880.0);
    p = fma(p, r, 1.0 / 40320.0);
    p = fma(p, r, 1.0 / 5040.0);
    p = fma(p, r, 1.0 / 720.0);
    p = fma(p, r, 1.0 / 120.0);
    p = fma(p, r, 1.0 / 24.0);
    p = fma(p, r, 1.0 / 6.0);
    p = fma(p, r, 0.5);
    p = fma(p, r, 1.0);
    p = fma(p, r, 1.0);
    return __hiloint2double(__double2hiint(p) + (__double2loint(kb) << 20), __double2loint(p));
}
// n / d for d in [1, 1e308): the hardware's approximation of 1 / d, one step of Newton's iteration, and one correction of the
// quotient by its remainder.
__device__ __forceinline__ double divide_for_activation(double n, double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    y = fma(y, fma(-d, y, 1.0), y);
    const double q = n * y;
    return fma(fma(-d, q, n), y, q);
}
__device__ __forceinline__ float logistic_double(float x) { return (float)divide_for_activation(1.0, 1.0 + exp_for_activation(-(double)x)); }
__device__ __forceinline__ float loggy_double(float x) { return (float)(divide_for_activation(2.0, 1.0 + exp_for_activation(-(double)x)) - 1.0); }
__device__ __forceinline__ float tanh_double(float x) {
    const double z = 2.0 * (double)x, e = exp_for_activation(z);
    const double t = divide_for_activation(e - 1.0, e + 1.0);
    return z > 709.782712893384 ? __int_as_float(0x7fffffff) : (float)t;        // (inf - 1) / (inf + 1)
}

// The reference's CPU activations (common/activations.cc:6-91).  Its constants
// are doubles, so each formula is evaluated in double and stored back as float,
// which reproduces the CPU results including tanh's NaN for large inputs
// ((inf-1)/(inf+1)) and the non-textbook elu/hardtan/lhtan definitions.
__device__ __forceinline__ float apply_activation(float x, int act) {
    switch (act) {
        case NB_ACT_LINEAR: return x;
        case NB_ACT_RELU: return x > 0.0f ? x : 0.0f;
        case NB_ACT_LEAKY: return x > 0.0f ? x : (float)(0.1 * (double)x);
        case NB_ACT_RELIE: return x > 0.0f ? x : (float)(0.01 * (double)x);
        case NB_ACT_LOGISTIC: return logistic_double(x);
        case NB_ACT_LOGGY: return loggy_double(x);
        case NB_ACT_TANH: return tanh_double(x);
        case NB_ACT_ELU: return x > 0.0f ? x * x : (float)((double)x * (exp((double)x) - 1.0));
        case NB_ACT_HARDTAN: return (x < 1.0f && x > -1.0f) ? 1.0f : 0.0f;
        case NB_ACT_LHTAN: return (x > 0.0f && x < 1.0f) ? 1.0f : 0.0f;
        case NB_ACT_PLSE:
            if (x < -4.0f) return (float)(0.01 * ((double)x + 4.0));
            if (x > 4.0f) return (float)(0.01 * ((double)x - 4.0) + 1.0);
            return (float)(0.125 * (double)x + 0.5);
        case NB_ACT_RAMP: return x > 0.0f ? (float)((double)x * ((double)x + 0.01)) : (float)(0.01 * (double)x);
        case NB_ACT_STAIR: {
            const int n = (int)x;
            if (n % 2) return x - (float)n + (float)(int)((double)x / 2.0);
            return (float)(int)((double)x / 2.0);
        }
        default: return x;
    }
}

// Out-of-line copy for unrolled epilogues: keeps the (large) switch out of the
// instruction stream of loops that almost always run relu / leaky / linear.
static __device__ __noinline__ float apply_activation_call(float x, int act) { return apply_activation(x, act); }

// Four values at once: a double exponential is a long chain, and the four chains overlap.
__device__ __forceinline__ float4 apply_activation4(float4 x, int act) {
    if (act == NB_ACT_LOGISTIC) return make_float4(logistic_double(x.x), logistic_double(x.y), logistic_double(x.z), logistic_double(x.w));
    if (act == NB_ACT_LOGGY) return make_float4(loggy_double(x.x), loggy_double(x.y), loggy_double(x.z), loggy_double(x.w));
    if (act == NB_ACT_TANH) return make_float4(tanh_double(x.x), tanh_double(x.y), tanh_double(x.z), tanh_double(x.w));
    return make_float4(apply_activation(x.x, act), apply_activation(x.y, act), apply_activation(x.z, act), apply_activation(x.w, act));
}

static __device__ __noinline__ float4 apply_activation4_call(float4 x, int act) { return apply_activation4(x, act); }

// One LSTM cell update (lstm_layer.cc:286-311) from the four gate pre-activations of a hidden unit: out of line to
// keep the GEMM epilogue small, with the four gate activations inline so that their exp chains overlap. The
// products and the sum round to fp32 separately, as the CPU path's loops do.
static __device__ __noinline__ float2 lstm_cell_unit(float zi, float zf, float zg, float zo, float c_prev) {
    const float ig = apply_activation(zi, NB_ACT_LOGISTIC);
    const float fg = apply_activation(zf, NB_ACT_LOGISTIC);
    const float gg = apply_activation(zg, NB_ACT_TANH);
    const float og = apply_activation(zo, NB_ACT_LOGISTIC);
    const float c = __fadd_rn(__fmul_rn(c_prev, fg), __fmul_rn(ig, gg));
    return make_float2(c, __fmul_rn(apply_activation(c, NB_ACT_TANH), og));
}

// The same update with the gate activations evaluated in fp32 (expf/tanhf, a few ulp from the double formulas):
// used by the TF32 GEMM epilogue, where the pre-activations already carry ~1e-3 of operand rounding and the few
// epilogue threads of a small-batch step cannot hide double-precision latency.
__device__ __forceinline__ float2 lstm_cell_unit_f32_inline(float zi, float zf, float zg, float zo, float c_prev) {
    const float ig = 1.0f / (1.0f + expf(-zi));
    const float fg = 1.0f / (1.0f + expf(-zf));
    const float gg = tanhf(zg);
    const float og = 1.0f / (1.0f + expf(-zo));
    const float c = __fadd_rn(__fmul_rn(c_prev, fg), __fmul_rn(ig, gg));
    return make_float2(c, __fmul_rn(tanhf(c), og));
}
// (out of line for the GEMM epilogue, which has no registers to spare; the same operations in the same order)
static __device__ __noinline__ float2 lstm_cell_unit_f32(float zi, float zf, float zg, float zo, float c_prev) {
    const float ig = 1.0f / (1.0f + expf(-zi));
    const float fg = 1.0f / (1.0f + expf(-zf));
    const float gg = tanhf(zg);
    const float og = 1.0f / (1.0f + expf(-zo));
    const float c = __fadd_rn(__fmul_rn(c_prev, fg), __fmul_rn(ig, gg));
    return make_float2(c, __fmul_rn(tanhf(c), og));
}

// relu, leaky and linear inline; everything else through the out-of-line copy
__device__ __forceinline__ float apply_activation_fast(float x, int act) {
    if (act == NB_ACT_RELU) return x > 0.0f ? x : 0.0f;
    if (act == NB_ACT_LINEAR) return x;
    if (act == NB_ACT_LEAKY) return x > 0.0f ? x : (float)(0.1 * (double)x);
    return apply_activation_call(x, act);
}

// relu, leaky and linear only
__device__ __forceinline__ float4 apply_activation4_cheap(float4 x, int act) {
    if (act == NB_ACT_LINEAR) return x;
    if (act == NB_ACT_RELU) return make_float4(x.x > 0.0f ? x.x : 0.0f, x.y > 0.0f ? x.y : 0.0f, x.z > 0.0f ? x.z : 0.0f, x.w > 0.0f ? x.w : 0.0f);
    auto leaky = [](float v) { return v > 0.0f ? v : (float)(0.1 * (double)v); };
    return make_float4(leaky(x.x), leaky(x.y), leaky(x.z), leaky(x.w));
}

__device__ __forceinline__ float4 apply_activation4_fast(float4 x, int act) {
    if (act == NB_ACT_RELU || act == NB_ACT_LINEAR || act == NB_ACT_LEAKY)
        return make_float4(apply_activation_fast(x.x, act), apply_activation_fast(x.y, act), apply_activation_fast(x.z, act),
                           apply_activation_fast(x.w, act));
    return apply_activation4_call(x, act);
}

}  // namespace nb
