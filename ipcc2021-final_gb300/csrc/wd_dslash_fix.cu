// wd_dslash_fix.cu -- the FP64 hopping term computed in 64-bit fixed point.
#include <type_traits>
#include "wd_fix.cuh"
#include "wd_kernels.h"
#include "wd_reduce.cuh"

namespace {

// One direction's links: reference AoS -> FP64 planes and fixed-point planes
// (a tile of 64 sites through shared memory, each link read once).  *bad is
// set when a link is outside what the fixed-point kernels are written for:
// the integer ranges need |u| <= 1 and absolute row and column sums (columns:
// the backward terms) of at most sqrt(6), and links much smaller than a
// unitary matrix's would lose digits below the fixed 2^-60.
__global__ void __launch_bounds__(256) k_gauge_in(const double2 *__restrict__ aos, double2 *__restrict__ soa,
                                                  int4 *__restrict__ fix, int Vh, int *bad)
{
    constexpr int kTile = 64;
    __shared__ double2 tile[kTile * 9];
    const int b = blockIdx.y, s0 = blockIdx.x * kTile, ns = min(kTile, Vh - s0);
    const double2 *src = aos + ((size_t)b * Vh + s0) * 9;
    soa += (size_t)b * 9 * Vh + s0;
    fix += (size_t)b * 9 * Vh + s0;
    for (int i = threadIdx.x; i < ns * 9; i += blockDim.x) tile[i] = src[i];
    __syncthreads();
    for (int i = threadIdx.x; i < ns * 9; i += blockDim.x) {
        const int c = i / ns, s = i - c * ns;
        const double2 v = tile[s * 9 + c];
        soa[(size_t)c * Vh + s] = v;
        const long long re = __double2ll_rn(v.x * 0x1p60), im = __double2ll_rn(v.y * 0x1p60);
        const long long r1 = (re + (1ll << 29)) >> 30, i1 = (im + (1ll << 29)) >> 30;
        fix[(size_t)c * Vh + s] = make_int4((int)r1, (int)(re - (r1 << 30)), (int)i1, (int)(im - (i1 << 30)));
    }
    for (int s = threadIdx.x; s < ns; s += blockDim.x) {
        double row[3] = {0, 0, 0}, col[3] = {0, 0, 0};
        bool ok = true;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const double ax = fabs(tile[s * 9 + k].x), ay = fabs(tile[s * 9 + k].y);
            ok = ok && ax <= 1.0 + 0x1p-20 && ay <= 1.0 + 0x1p-20 && ax + ay <= 1.5;  // false for NaN too
            row[k / 3] += ax + ay;
            col[k % 3] += ax + ay;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
            ok = ok && row[k] >= 0.99 && row[k] <= 2.46 && col[k] >= 0.99 && col[k] <= 2.46;
        if (!ok) *bad = 1;
    }
}

template <class Base>
struct HopFix : Base {
    const int4 *__restrict__ links;
};

// The FP64-pipe arithmetic for a site whose values do not fit a block scale
template <bool DAG, class P>
__device__ __noinline__ void f64_route(const P &p, int s)
{
    double2 acc[12];
    wd_hop_site<DAG>(p, s, acc);
    p.epilogue(s, acc);
}

// Output sites [s_lo, s_hi), two threads a site
template <bool DAG, class P, int T>
__global__ void __launch_bounds__(T, 512 / T) k_hop_fix(const __grid_constant__ P p, int s_lo, int s_hi)
{
    extern __shared__ __align__(16) char smem[];
    const int id = blockIdx.x * T + threadIdx.x, half = id & 1;
    const int s0 = s_lo + (id >> 1), s = s0 < s_hi ? s0 : s_hi - 1;
    double2 up[3], low[3];
    const bool ok = wd_fix::site<DAG>(p, *reinterpret_cast<wd_fix::Stage<T> *>(smem), s, half, up, low);
    if (s0 >= s_hi) return;
    if (ok) {
        p.store_spin(s, half, up);
        p.store_spin(s, 3 - half, low);
    } else if (half == 0) {
        f64_route<DAG>(p, s);
    }
}

template <class P>
__device__ __noinline__ void f64_route_acc(const P &p, int s, double2 *acc)
{
    wd_hop_site<false>(p, s, acc);
}

// The reliable update's second Schur hop fused with the true residual (as
// k_hop_f64_res): s = bhat - (alpha acc + beta x) in FP64, rounded to FP32
// into s32 (plane c/2, half c&1 of the float4 for component c), |s32|^2
// reduced over the grid.
template <class P, int T>
__global__ void __launch_bounds__(T, 512 / T) k_hop_fix_res(const __grid_constant__ P p, const WdResSink r)
{
    extern __shared__ __align__(16) char smem[];
    const int id = blockIdx.x * T + threadIdx.x, half = id & 1;
    const int s0 = id >> 1, Vh = p.g.Vh, s = s0 < Vh ? s0 : Vh - 1;
    double2 v[6];
    const bool ok = wd_fix::site<false>(p, *reinterpret_cast<wd_fix::Stage<T> *>(smem), s, half, v, v + 3);
    float n = 0.f;
    if (s0 < Vh) {
        if (!ok) {
            double2 acc[12];
            f64_route_acc(p, s, acc);
            for (int k = 0; k < 3; ++k) {
                v[k] = acc[half * 3 + k];
                v[3 + k] = acc[(3 - half) * 3 + k];
            }
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const int c = (k < 3 ? half : 3 - half) * 3 + k % 3;
            const size_t i = (size_t)c * Vh + s;
            const double2 o = c_axpby(p.alpha, v[k], p.beta, p.x[i]), b = r.bhat[i];
            const float2 f = make_float2((float)(b.x - o.x), (float)(b.y - o.y));
            reinterpret_cast<float2 *>(r.s32 + (size_t)(c >> 1) * Vh + s)[c & 1] = f;
            n = fmaf(f.x, f.x, fmaf(f.y, f.y, n));
        }
    }
    double tot;
    if (wd_grid_sum<T>((double)n, r.partial, r.counter, &tot)) *r.result = tot;
}

// launch shapes of the plain and the residual hop: threads per block
template <class Run>
wd_status with_threads(int variant, Run run)
{
    if (variant == 1) return run(std::integral_constant<int, 64>());
    if (variant == 2) return run(std::integral_constant<int, 32>());
    return run(std::integral_constant<int, 128>());
}

}  // namespace

wd_status wd_gauge_ref_to_soa_fix(wd_context *ctx, const WdGeom &g, int mu, const double2 *ref, double2 *soa, void *fix,
                                  int *bad)
{
    const size_t off = (size_t)mu * 2 * 9 * g.Vh;
    k_gauge_in<<<dim3((g.Vh + 63) / 64, 2), 256, 0, ctx->stream>>>(ref, soa + off, (int4 *)fix + off, g.Vh, bad);
    WD_LAUNCHED(ctx);
    return WD_OK;
}

template <class Base>
static HopFix<Base> make_fix(const wd_lattice *lat, const double2 *in, double2 *out, const double2 *x,
                             int cb, double alpha, double beta)
{
    HopFix<Base> p;
    p.g = lat->g;
    p.cb = cb;
    p.in = in;
    p.gauge = lat->gauge;
    p.x = x;
    p.out = out;
    p.alpha = alpha;
    p.beta = beta;
    p.scale = F64Scale::make(alpha);
    p.links = (const int4 *)lat->gauge_fix;
    return p;
}

wd_status wd_hop_fix(wd_context *ctx, const wd_lattice *lat, const double2 *in, double2 *out,
                     const double2 *x, int cb, int dag, double alpha, double beta, int variant)
{
    const auto p = make_fix<HopF64<128>>(lat, in, out, x, cb, alpha, beta);
    using P = std::decay_t<decltype(p)>;
    return with_threads(variant, [&](auto t) -> wd_status {
        constexpr int T = decltype(t)::value;
        constexpr size_t sm = sizeof(wd_fix::Stage<T>);
        const int blocks = (int)(((int64_t)lat->g.Vh * 2 + T - 1) / T);
        if (dag) k_hop_fix<true, P, T><<<blocks, T, sm, ctx->stream>>>(p, 0, lat->g.Vh);
        else k_hop_fix<false, P, T><<<blocks, T, sm, ctx->stream>>>(p, 0, lat->g.Vh);
        WD_LAUNCHED(ctx);
        return WD_OK;
    });
}

wd_status wd_hop_fix_residual(wd_context *ctx, const wd_lattice *lat, const double2 *in,
                              const double2 *x, double alpha, double beta, const WdResSink &r, int variant)
{
    const auto p = make_fix<HopF64<128>>(lat, in, nullptr, x, 0, alpha, beta);
    using P = std::decay_t<decltype(p)>;
    return with_threads(variant, [&](auto t) -> wd_status {
        constexpr int T = decltype(t)::value;
        const int blocks = (int)(((int64_t)lat->g.Vh * 2 + T - 1) / T);
        k_hop_fix_res<P, T><<<blocks, T, sizeof(wd_fix::Stage<T>), ctx->stream>>>(p, r);
        WD_LAUNCHED(ctx);
        return WD_OK;
    });
}

wd_status wd_hop_fix_aos_range(wd_context *ctx, cudaStream_t stream, const wd_lattice *lat, const double2 *in_aos,
                               double2 *out_aos, const double2 *x_aos, int cb, int dag,
                               double alpha, double beta, int s_lo, int s_hi)
{
    constexpr int T = 64;
    constexpr size_t sm = sizeof(wd_fix::Stage<T>);
    const auto p = make_fix<HopF64AoS<T>>(lat, in_aos, out_aos, x_aos, cb, alpha, beta);
    using P = std::decay_t<decltype(p)>;
    const int blocks = (int)(((int64_t)(s_hi - s_lo) * 2 + T - 1) / T);
    if (dag) k_hop_fix<true, P, T><<<blocks, T, sm, stream>>>(p, s_lo, s_hi);
    else k_hop_fix<false, P, T><<<blocks, T, sm, stream>>>(p, s_lo, s_hi);
    WD_LAUNCHED(ctx);
    return WD_OK;
}
