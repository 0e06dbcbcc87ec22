// wd_hop_f64.cuh -- operand access and epilogue of the FP64 hopping kernels
// (the policies of wd_hop.cuh), shared by the FP64-pipe kernels
// (wd_dslash_f64.cu) and the fixed-point kernels (wd_dslash_fix.cu).
#pragma once
#include <cmath>
#include <cstdint>
#include "wd_hop.cuh"

// Output scaling without the FP64 pipe when alpha is 1 or a power of two
// (DslashoffdNew's -1/2, the Schur operator's first hop's 1): a power-of-two
// factor only moves the exponent, so integer arithmetic on the bits gives
// the FP64 product exactly; zeros, subnormal results and non-finite values
// take the FP64 multiply.  24 fewer FP64 operations per site (of ~890).
struct F64Scale {
    double alpha;
    int mode;       // 0: multiply, 1: identity, 2: exponent shift
    int shift;      // mode 2: alpha = sign * 2^shift
    uint64_t sign;  // mode 2: sign bit of alpha

    static F64Scale make(double a)
    {
        F64Scale f{a, 0, 0, 0};
        int e = 0;
        const double m = std::frexp(a, &e);  // a = m * 2^e, |m| in [0.5, 1)
        if (a == 1.0) f.mode = 1;
        else if (std::fabs(m) == 0.5 && e - 1 > -1000 && e - 1 < 1000) {
            f.mode = 2;
            f.shift = e - 1;
            f.sign = a < 0 ? 0x8000000000000000ull : 0ull;
        }
        return f;
    }
    __device__ __forceinline__ double apply(double v) const
    {
        if (mode == 1) return v;
        if (mode == 2) {
            const uint64_t b = (uint64_t)__double_as_longlong(v);
            const int ex = (int)((b >> 52) & 0x7ff);
            if (ex > 0 && ex < 0x7ff && ex + shift > 0 && ex + shift < 0x7ff)
                return __longlong_as_double((long long)((b + ((uint64_t)(int64_t)shift << 52)) ^ sign));
        }
        return v * alpha;
    }
    __device__ __forceinline__ double2 apply(double2 v) const { return make_double2(apply(v.x), apply(v.y)); }
};

template <int THREADS>
struct HopF64 {
    using C = double2;
    static constexpr int kThreads = THREADS;
    static constexpr bool kPairDirs = true;  // FP64-pipe bound: fewest operations wins
    WdGeom g;
    int cb;
    const double2 *in;                  // parity 1-cb block [12][Vh] (kernels that start early read it too)
    const double2 *__restrict__ gauge;  // [4][2][9][Vh]
    const double2 *__restrict__ x;      // parity cb block or null
    double2 *__restrict__ out;          // parity cb block
    double alpha, beta;
    F64Scale scale;                     // alpha, applied when there is no x
    const int *stop = nullptr;          // device gate (wd_gate_closed)

    __device__ __forceinline__ void load_in(int s, C *v) const
    {
#pragma unroll
        for (int c = 0; c < 12; ++c) v[c] = in[(size_t)c * g.Vh + s];
    }
    __device__ __forceinline__ void load_link(int mu, int par, int s, C *U) const
    {
        const double2 *b = gauge + (size_t)((mu * 2 + par) * 9) * g.Vh + s;
#pragma unroll
        for (int k = 0; k < 9; ++k) U[k] = b[(size_t)k * g.Vh];
    }
    __device__ __forceinline__ void epilogue(int s, const C *acc) const
    {
        if (x) {
#pragma unroll
            for (int c = 0; c < 12; ++c)
                out[(size_t)c * g.Vh + s] = c_axpby(alpha, acc[c], beta, x[(size_t)c * g.Vh + s]);
        } else {
#pragma unroll
            for (int c = 0; c < 12; ++c) out[(size_t)c * g.Vh + s] = scale.apply(acc[c]);
        }
    }
};

// The same kernel on the reference's own site-major layout (AoS: the 12
// complex components of a site contiguous, [site][spin*3+colour]) for the
// input and output parity blocks; the links stay in the SoA planes.  A warp's
// 32 neighbour sites are 6 KB of consecutive bytes, so every fetched line is
// used, and the FP64 pipe (not the access pattern) still bounds the kernel.
// The host-buffer path runs it on the staging buffers directly, with no
// layout conversion between the copies and the arithmetic, where the
// fixed-point hop (which reads both layouts) does not take the links.
template <int THREADS>
struct HopF64AoS : HopF64<THREADS> {
    __device__ __forceinline__ void load_in(int s, double2 *v) const
    {
        const double2 *b = this->in + (size_t)s * 12;
#pragma unroll
        for (int c = 0; c < 12; ++c) v[c] = b[c];
    }
    __device__ __forceinline__ void epilogue(int s, const double2 *acc) const
    {
        double2 *o = this->out + (size_t)s * 12;
        if (this->x) {  // site-major x block of the output parity
            const double2 *xv = this->x + (size_t)s * 12;
#pragma unroll
            for (int c = 0; c < 12; ++c) o[c] = c_axpby(this->alpha, acc[c], this->beta, xv[c]);
        } else {
#pragma unroll
            for (int c = 0; c < 12; ++c) o[c] = this->scale.apply(acc[c]);
        }
    }
};
