// wd_cg.cu -- one CG iteration's vector work on device-side scalars (WdCgDev),
// on FP64 or double-float vectors.  HBM-bound passes (FP64's complex update:
// FP64 pipe); what they save over host scalars is the two host waits an
// iteration (about 30 us of an 8^3x16 iteration's 146).  Reductions: fixed
// grid, fixed fold order.
#include <type_traits>
#include "wd_async.cuh"
#include "wd_df.cuh"
#include "wd_reduce.cuh"
#include "wd_solver.h"

namespace {

#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

// vector entries of one storage in registers: FP64 complex, or double-float complex
struct VF64 {
    using E = double2;
    using C = double2;  // complex scalar
    using R = double;   // real scalar and sums
    static __device__ __forceinline__ C load(E e) { return e; }
    static __device__ __forceinline__ E store(C c) { return c; }
    static __device__ __forceinline__ R real(double a) { return a; }
    static __device__ __forceinline__ R zero() { return 0.0; }
    static __device__ __forceinline__ double value(R r) { return r; }
    static __device__ __forceinline__ R madd(R s, R a, R b) { return fma(a, b, s); }
    // v + a u: real a, and complex a as separate products and sums (src/invert.cpp:89-107)
    static __device__ __forceinline__ C axpy(R a, C u, C v) { return make_double2(fma(a, u.x, v.x), fma(a, u.y, v.y)); }
    static __device__ __forceinline__ C caxpy(R re, R im, C u, C v)
    {
        return make_double2(v.x + fma(re, u.x, -im * u.y), v.y + fma(re, u.y, im * u.x));
    }
    static __device__ __forceinline__ R re(C c) { return c.x; }
    static __device__ __forceinline__ R im(C c) { return c.y; }
    static __device__ __forceinline__ R neg(R a) { return -a; }
};
struct VDF {
    using E = float4;
    using C = dfc;
    using R = dfr;
    static __device__ __forceinline__ C load(E e) { return df_from_f4(e); }
    static __device__ __forceinline__ E store(C c) { return df_to_f4(c); }
    static __device__ __forceinline__ R real(double a) { return df_split(a); }
    static __device__ __forceinline__ R zero() { return dfr{0.f, 0.f}; }
    static __device__ __forceinline__ double value(R r) { return df_value(r); }
    static __device__ __forceinline__ R madd(R s, R a, R b) { return df_madd(s, a, b); }
    static __device__ __forceinline__ C axpy(R a, C u, C v) { return dfc{df_madd(v.re, a, u.re), df_madd(v.im, a, u.im)}; }
    static __device__ __forceinline__ C caxpy(R re, R im, C u, C v) { return c_madd(v, dfc{re, im}, u); }
    static __device__ __forceinline__ R re(C c) { return c.re; }
    static __device__ __forceinline__ R im(C c) { return c.im; }
    static __device__ __forceinline__ R neg(R a) { return dfr{-a.h, -a.l}; }
};

template <class V>
__device__ __forceinline__ typename V::R norm_acc(typename V::R s, typename V::C c)
{
    return V::madd(V::madd(s, V::re(c), V::re(c)), V::im(c), V::im(c));
}

template <class V>
__global__ void __launch_bounds__(WD_RED_THREADS) k_cgd_norm(const typename V::E *t, int64_t n, WdCgDev *dev,
                                                             WdRed red)
{
    wd_pdl_wait(gridDim.x > 152);
    if (dev->stop) return;
    typename V::R s = V::zero();
    GRID_STRIDE(i, n) s = norm_acc<V>(s, V::load(t[i]));
    double tot;
    if (wd_grid_sum<WD_RED_THREADS>(V::value(s), red, &tot)) wd_cg_set_alpha(dev, tot, 0.0, false);
}

template <class V>
__global__ void __launch_bounds__(WD_RED_THREADS) k_cgd_dot(const typename V::E *p,
                                                            const typename V::E *q, int64_t n, WdCgDev *dev,
                                                            WdRed red)
{
    wd_pdl_wait(gridDim.x > 152);
    if (dev->stop) return;
    typename V::R re = V::zero(), im = V::zero();
    GRID_STRIDE(i, n)
    {
        const typename V::C u = V::load(p[i]), v = V::load(q[i]);
        re = V::madd(V::madd(re, V::re(u), V::re(v)), V::im(u), V::im(v));
        im = V::madd(V::madd(im, V::re(u), V::im(v)), V::neg(V::im(u)), V::re(v));
    }
    double t[2];
    if (wd_grid_sum_n<WD_RED_THREADS, 2>({V::value(re), V::value(im)}, red, t))
        wd_cg_set_alpha(dev, t[0], t[1], true);
}

template <class V, bool CPLX>
__global__ void __launch_bounds__(WD_RED_THREADS) k_cgd_update(const typename V::E *p,
                                                               const typename V::E *q,
                                                               typename V::E *x,
                                                               typename V::E *r, int64_t n, WdCgDev *dev,
                                                               WdRed red)
{
    wd_pdl_wait(gridDim.x > 152);
    if (dev->stop) return;
    const typename V::R re = V::real(dev->are), im = V::real(dev->aim), mre = V::neg(re), mim = V::neg(im);
    typename V::R s = V::zero();
    GRID_STRIDE(i, n)
    {
        const typename V::C pv = V::load(p[i]), qv = V::load(q[i]);
        typename V::C xv = V::load(x[i]), rv = V::load(r[i]);
        xv = CPLX ? V::caxpy(re, im, pv, xv) : V::axpy(re, pv, xv);
        rv = CPLX ? V::caxpy(mre, mim, qv, rv) : V::axpy(mre, qv, rv);
        x[i] = V::store(xv);
        r[i] = V::store(rv);
        s = norm_acc<V>(s, rv);
    }
    double tot;
    if (wd_grid_sum<WD_RED_THREADS>(V::value(s), red, &tot)) wd_cg_set_beta(dev, tot);
}

template <class V>
__global__ void k_cgd_xpby(const typename V::E *r, typename V::E *p, int64_t n,
                           const WdCgDev *dev)
{
    wd_pdl_wait(gridDim.x > 152);
    if (dev->stop) return;
    const typename V::R b = V::real(dev->beta);
    GRID_STRIDE(i, n) p[i] = V::store(V::axpy(b, V::load(p[i]), V::load(r[i])));
}

// blocks of the reducing passes: about two entries a thread, so that small
// vectors do not pay 608 block sums (8^3x16 update: 12.4 us with them)
inline int red_blocks(int64_t n)
{
    const int64_t b = (n + 2 * WD_RED_THREADS - 1) / (2 * WD_RED_THREADS);
    return (int)(b < WD_RED_BLOCKS ? b : WD_RED_BLOCKS);
}

// An early launch leaves a one-wave grid unevenly spread over the SMs, which
// the FP64 passes pay for (FP64 pipe: 17.7 against 16.6 ms a reference CG at
// 16^3x32) and the double-float passes where their threads loop (59.8 against
// 57.7 ms a CG at 32^3x64).  Up to a block per SM the former gain (2.02 against
// 2.28 ms at 4^4), and up to the full grid the latter (1.88 against 2.03 at
// 8^3x32)
template <class V>
bool early_reduce(int64_t n)
{
    return red_blocks(n) <= (std::is_same_v<V, VDF> ? WD_RED_BLOCKS - 1 : 152);
}

// runs f(V()) for the vectors' storage
template <class F>
wd_status typed(wd_context *ctx, WdVec v, F f)
{
    if (v.prec == WD_PREC_F64) f(VF64());
    else if (v.prec == WD_PREC_DF64) f(VDF());
    else return wd_fail(ctx, WD_ERR_BAD_ARG, "CG vectors are FP64 or double-float");
    WD_LAUNCHED(ctx);
    return WD_OK;
}

}  // namespace

wd_status wd_cgd_norm(wd_context *ctx, WdVec t, int64_t n, WdCgDev *dev, WdRed red)
{
    return typed(ctx, t, [&](auto v) {
        using V = decltype(v);
        wd_launch_pdl(early_reduce<V>(n), k_cgd_norm<V>, red_blocks(n), WD_RED_THREADS, 0, ctx->stream, (const typename V::E *)t.p, n, dev, red);
    });
}

wd_status wd_cgd_dot(wd_context *ctx, WdVec p, WdVec q, int64_t n, WdCgDev *dev, WdRed red)
{
    return typed(ctx, p, [&](auto v) {
        using V = decltype(v);
        using E = typename V::E;
        wd_launch_pdl(early_reduce<V>(n), k_cgd_dot<V>, red_blocks(n), WD_RED_THREADS, 0, ctx->stream, (const E *)p.p, (const E *)q.p, n, dev, red);
    });
}

wd_status wd_cgd_update(wd_context *ctx, bool cplx, WdVec p, WdVec q, WdVec x, WdVec r, int64_t n, WdCgDev *dev,
                        WdRed red)
{
    return typed(ctx, p, [&](auto v) {
        using V = decltype(v);
        using E = typename V::E;
        const E *pp = (const E *)p.p, *qq = (const E *)q.p;
        E *xx = (E *)x.p, *rr = (E *)r.p;
        if (cplx) wd_launch_pdl(early_reduce<V>(n), k_cgd_update<V, true>, red_blocks(n), WD_RED_THREADS, 0, ctx->stream, pp, qq, xx, rr, n, dev, red);
        else wd_launch_pdl(early_reduce<V>(n), k_cgd_update<V, false>, red_blocks(n), WD_RED_THREADS, 0, ctx->stream, pp, qq, xx, rr, n, dev, red);
    });
}

wd_status wd_cgd_xpby(wd_context *ctx, WdVec r, WdVec p, int64_t n, const WdCgDev *dev)
{
    const int64_t b = (n + 255) / 256;
    return typed(ctx, p, [&](auto v) {
        using V = decltype(v);
        using E = typename V::E;
        wd_launch_pdl(std::is_same_v<V, VF64> || b <= 152 * 16, k_cgd_xpby<V>, (int)(b < 152 * 16 ? b : 152 * 16), 256, 0, ctx->stream, (const E *)r.p, (E *)p.p, n, dev);
    });
}
