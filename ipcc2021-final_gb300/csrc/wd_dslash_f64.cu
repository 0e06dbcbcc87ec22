// wd_dslash_f64.cu -- native FP64 hopping kernel (the plain drop-in arithmetic),
// for lattices whose links the fixed-point hop (wd_dslash_fix.cu) does not hold
// and launches that may not use its copy of them.
//
// Storage: double2 planes, spinor [12][Vh] per parity, links [mu][parity][9][Vh].
// Algorithmic traffic per output site: 8 links x 144 B + 1 spinor in x 192 B
// + 1 spinor out x 192 B = 1536 B (+192 B when the epilogue reads x).
// Arithmetic: 1320 flop per site.  On GB300 the FP64 pipe (~1.2 TFLOP/s
// measured) rather than HBM bounds this kernel, so it is written for the
// fewest FP64 operations (~790 per site): direction pairs combined
// (wd_hop_mu), the first direction assigned, and a power-of-two output scale
// applied on the exponent bits (F64Scale).  wd_dslash_df.cu holds the
// double-float variant that moves the arithmetic onto the FP32 pipe.
#include "wd_hop_f64.cuh"
#include "wd_kernels.h"
#include "wd_reduce.cuh"
#include <type_traits>
#include "wd_tune.h"

namespace {

// The reliable update's second Schur hop fused with the true residual:
// s = bhat - (alpha acc + beta x), rounded to FP32 into s32 (FP32 site
// layout: plane j holds components 2j, 2j+1), |s32|^2 reduced over the grid.
template <bool DAG, class P>
__global__ void __launch_bounds__(P::kThreads) k_hop_f64_res(const P p, const WdResSink r)
{
    const int s = blockIdx.x * P::kThreads + threadIdx.x;
    float n = 0.f;
    if (s < p.g.Vh) {
        double2 acc[12];
        wd_hop_site<DAG>(p, s, acc);
        const size_t Vh = p.g.Vh;
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            float v[4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const size_t i = (size_t)(2 * j + h) * Vh + s;
                const double2 o = c_axpby(p.alpha, acc[2 * j + h], p.beta, p.x[i]);
                const double2 b = r.bhat[i];
                v[2 * h] = (float)(b.x - o.x);
                v[2 * h + 1] = (float)(b.y - o.y);
                n = fmaf(v[2 * h], v[2 * h], fmaf(v[2 * h + 1], v[2 * h + 1], n));
            }
            r.s32[(size_t)j * Vh + s] = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
    double tot;
    if (wd_grid_sum<P::kThreads>((double)n, r.red, &tot)) *r.result = tot;
}

}  // namespace

wd_status wd_hop_df_residual(wd_context *ctx, const wd_lattice *lat, const float4 *in_block, const float4 *x_block,
                             const float4 *bhat, float4 *s32, double mass, WdRed red,
                             double *result);

wd_status wd_hop_hi_residual(wd_context *ctx, const wd_lattice *lat, WdVec in, WdVec x, WdVec bhat, WdVec s32,
                             double mass, WdRed red, double *result)
{
    if (in.prec != x.prec || in.prec != bhat.prec || s32.prec != WD_PREC_F32)
        return wd_fail(ctx, WD_ERR_BAD_ARG, "residual hop: in, x, bhat of one storage, s32 FP32");
    const double a = 4.0 + mass;
    if (in.prec == WD_PREC_DF64)
        return wd_hop_df_residual(ctx, lat, (const float4 *)in.p, (const float4 *)x.p, (const float4 *)bhat.p,
                                  (float4 *)s32.p, mass, red, result);
    if (in.prec != WD_PREC_F64) return wd_fail(ctx, WD_ERR_BAD_ARG, "residual hop: FP64 or double-float storage");
    const WdResSink r{(const double2 *)bhat.p, (float4 *)s32.p, red, result};
    if (const WdTried t = wd_hop_fix_residual(ctx, lat, (const double2 *)in.p, (const double2 *)x.p, -0.25 / a, a, r))
        return *t;
    auto run = [&](auto tag) -> wd_status {
        using P = HopF64<decltype(tag)::value>;
        P p;
        p.g = lat->g;
        p.cb = 0;
        p.in = (const double2 *)in.p;
        p.gauge = lat->gauge;
        p.x = (const double2 *)x.p;
        p.out = nullptr;
        p.alpha = -0.25 / a;
        p.beta = a;
        p.scale = F64Scale::make(p.alpha);
        const int blocks = (lat->g.Vh + P::kThreads - 1) / P::kThreads;
        k_hop_f64_res<false><<<blocks, P::kThreads, 0, ctx->stream>>>(p, r);
        WD_LAUNCHED(ctx);
        return WD_OK;
    };
    // the plain FP64 hop's tuned shape: 128, 64 or 256 threads per block
    const int v = wd_tune_choice(ctx, "hop_f64", lat->g.Vh);
    if (v == 1) return run(std::integral_constant<int, 64>());
    if (v == 2) return run(std::integral_constant<int, 256>());
    return run(std::integral_constant<int, 128>());
}

wd_status wd_hop_f64_aos_range(wd_context *ctx, cudaStream_t stream, const wd_lattice *lat, const double2 *in_aos,
                               double2 *out_aos, const double2 *x_aos, int cb, int dag, double alpha, double beta,
                               int s_lo, int s_hi)
{
    if (s_hi <= s_lo) return WD_OK;
    if (const WdTried t = wd_hop_fix_aos_range(ctx, stream, lat, in_aos, out_aos, x_aos, cb, dag, alpha, beta, s_lo, s_hi))
        return *t;
    using P = HopF64AoS<64>;
    P p;
    p.g = lat->g;
    p.cb = cb;
    p.in = in_aos;
    p.gauge = lat->gauge;
    p.x = x_aos;
    p.out = out_aos;
    p.alpha = alpha;
    p.beta = beta;
    p.scale = F64Scale::make(alpha);
    const int n = s_hi - s_lo;
    const int blocks = (n + P::kThreads - 1) / P::kThreads;
    if (dag) wd_hop_kernel_range<true><<<blocks, P::kThreads, 0, stream>>>(p, s_lo, s_hi);
    else wd_hop_kernel_range<false><<<blocks, P::kThreads, 0, stream>>>(p, s_lo, s_hi);
    WD_LAUNCHED(ctx);
    return WD_OK;
}

wd_status wd_hop_f64(wd_context *ctx, const wd_lattice *lat, const double2 *in_block,
                     double2 *out_block, const double2 *x_block, int cb, int dag, double alpha,
                     double beta, const int *stop)
{
    if (const WdTried t = wd_hop_fix(ctx, lat, in_block, out_block, x_block, cb, dag, alpha, beta, stop)) return *t;
    auto run = [&](auto tag) -> wd_status {
        using P = HopF64<decltype(tag)::value>;
        P p;
        p.g = lat->g;
        p.cb = cb;
        p.in = in_block;
        p.gauge = lat->gauge;
        p.x = x_block;
        p.out = out_block;
        p.alpha = alpha;
        p.beta = beta;
        p.scale = F64Scale::make(alpha);
        p.stop = stop;
        const int blocks = (lat->g.Vh + P::kThreads - 1) / P::kThreads;
        if (dag) wd_hop_kernel<true><<<blocks, P::kThreads, 0, ctx->stream>>>(p);
        else wd_hop_kernel<false><<<blocks, P::kThreads, 0, ctx->stream>>>(p);
        WD_LAUNCHED(ctx);
        return WD_OK;
    };
    // variants: 128, 64, 256 threads per block
    return wd_tune_launch(ctx, "hop_f64", lat->g.Vh, kHopF64Variants, [&](int v) -> wd_status {
        if (v == 1) return run(std::integral_constant<int, 64>());
        if (v == 2) return run(std::integral_constant<int, 256>());
        return run(std::integral_constant<int, 128>());
    });
}
