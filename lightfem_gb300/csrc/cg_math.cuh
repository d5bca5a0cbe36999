// Arithmetic the PCG kernel files share: FP32 pairs for the mixed loop's sums and
// scalars, and the pointwise preconditioners.
#pragma once

#include "common.cuh"

namespace lfgpu {
namespace {

// An unevaluated FP32 pair (hi + lo) for the dot products of the FP32 loop: each
// addition is Knuth's two-sum, so the pair carries about 48 bits.  This keeps
// the dot products near FP64 accuracy with FP32 arithmetic only -- FP64 shuffles
// and adds in every thread would keep GB300's narrow FP64 pipe busy for several
// microseconds per reduction.
struct FloatPair {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float s = __fadd_rn(hi, x);
        const float bp = __fsub_rn(s, hi);
        const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(x, bp));
        lo = __fadd_rn(lo, e);
        hi = s;
    }
    __device__ __forceinline__ void add(const FloatPair& o) {
        add(o.hi);
        lo = __fadd_rn(lo, o.lo);
    }
};

// FP32-pair per-thread values summed over the CTA (the mixed inner loop): warp
// sums as pairs, then the warps' pairs in warp 0, whose threads all get the CTA's
// totals as pairs in w (the other threads' w is zero).  FP32 arithmetic only: on
// GB300 a dependent FP64 add takes about as long as a dozen FP32 ones.
// NT > 0: only the CTA's first NT threads take part, synchronised on named barrier 1.
template <int NT>
__device__ __forceinline__ void pair_reduce_sync() {
    if constexpr (NT == 0)
        __syncthreads();
    else
        asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
}

template <int K, int NT = 0>
__device__ __forceinline__ void block_pair_reduce(FloatPair (&v)[K], FloatPair (&w)[K]) {
    __shared__ float2 s_warp[32 * kMaxReduce];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            FloatPair other;
            other.hi = __shfl_xor_sync(0xffffffffu, v[k].hi, o);
            other.lo = __shfl_xor_sync(0xffffffffu, v[k].lo, o);
            v[k].add(other);
        }
    }
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) s_warp[warp * K + k] = make_float2(v[k].hi, v[k].lo);
    }
    pair_reduce_sync<NT>();
#pragma unroll
    for (int k = 0; k < K; ++k) w[k] = FloatPair{};
    if (warp == 0) {
        const int nw = (NT == 0 ? static_cast<int>(blockDim.x) : NT) >> 5;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (lane < nw) {
                const float2 t = s_warp[lane * K + k];
                w[k].hi = t.x;
                w[k].lo = t.y;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                FloatPair other;
                other.hi = __shfl_xor_sync(0xffffffffu, w[k].hi, o);
                other.lo = __shfl_xor_sync(0xffffffffu, w[k].lo, o);
                w[k].add(other);
            }
        }
    }
    pair_reduce_sync<NT>();  // s_warp is free again
}

__device__ __forceinline__ double2 block2_apply(const double* __restrict__ blk, int i, double r0, double r1) {
    const double f0 = blk[3 * i], f1 = blk[3 * i + 1], f2 = blk[3 * i + 2];
    double s0 = __dmul_rn(r0, f0);
    double s1 = __dmul_rn(__dsub_rn(r1, __dmul_rn(f1, s0)), f2);
    s1 = __dmul_rn(s1, f2);
    s0 = __dmul_rn(__dsub_rn(s0, __dmul_rn(f1, s1)), f0);
    return make_double2(s0, s1);
}

__device__ __forceinline__ float2 block2_apply32(const float* __restrict__ blk, int i, float r0, float r1) {
    const float f0 = blk[3 * i], f1 = blk[3 * i + 1], f2 = blk[3 * i + 2];
    float s0 = r0 * f0;
    float s1 = (r1 - f1 * s0) * f2;
    s1 = s1 * f2;
    s0 = (s0 - f1 * s1) * f0;
    return make_float2(s0, s1);
}

// z of node i from the preconditioner's values pc (Jacobi: the inverse diagonal,
// two floats a node; 2x2 blocks: the factor, three floats a node), wherever they are.
template <int PRECOND>
__device__ __forceinline__ float2 precond32_at(const float* pc, int i, float2 rv) {
    if (PRECOND == LFGPU_PRECOND_JACOBI) {
        const float2 d = reinterpret_cast<const float2*>(pc)[i];
        return make_float2(d.x * rv.x, d.y * rv.y);
    }
    return block2_apply32(pc, i, rv.x, rv.y);
}

__device__ __forceinline__ float pnew(float z, float p, float beta) { return __fmaf_rn(beta, p, z); }
__device__ __forceinline__ float with_diag(float off, float hi, float lo, float x) { return fmaf(hi, x, off) + lo * x; }

// (hi, lo) += (ah + al) * p with error-free transformations (Knuth's two-sum,
// the fma two-product), then renormalised so |lo| <= ulp(hi) / 2.  The _rn
// intrinsics keep the compiler from fusing the steps the error terms rely on.
__device__ __forceinline__ void pair_axpy(float& hi, float& lo, float ah, float al, float p) {
    const float prod = __fmul_rn(ah, p);
    const float perr = __fmaf_rn(al, p, __fmaf_rn(ah, p, -prod));
    const float s = __fadd_rn(hi, prod);
    const float bp = __fsub_rn(s, hi);
    const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(prod, bp));
    const float l = __fadd_rn(lo, __fadd_rn(err, perr));
    hi = __fadd_rn(s, l);
    lo = __fsub_rn(l, __fsub_rn(hi, s));
}

// num / den as an unevaluated FP32 pair (hi + lo, about 44 bits; Dekker's
// division): one FP32 quotient, its remainder from an error-free product, and a
// correction.  The loop's scalars (alpha, beta) come from this instead of an FP64
// division, whose dependent steps take a large part of a microsecond on GB300
// and hold up every CTA waiting for them.
__device__ __forceinline__ void pair_quotient(float nh, float nl, float dh, float dl, float& hi, float& lo) {
    const float q1 = __fdiv_rn(nh, dh);
    const float p = __fmul_rn(q1, dh);
    const float pe = __fmaf_rn(q1, dh, -p);  // q1 * dh = p + pe exactly
    const float r = __fadd_rn(__fsub_rn(__fsub_rn(nh, p), pe), __fsub_rn(nl, __fmul_rn(q1, dl)));
    const float q2 = __fdiv_rn(r, dh);
    hi = __fadd_rn(q1, q2);
    lo = __fsub_rn(q2, __fsub_rn(hi, q1));
}
__device__ __forceinline__ void pair_quotient(double num, double den, float& hi, float& lo) {
    const float nh = static_cast<float>(num), nl = static_cast<float>(num - static_cast<double>(nh));
    const float dh = static_cast<float>(den), dl = static_cast<float>(den - static_cast<double>(dh));
    pair_quotient(nh, nl, dh, dl, hi, lo);
}

}  // namespace
}  // namespace lfgpu
