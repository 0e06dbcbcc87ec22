// wd_dslash_fix.cu -- the FP64 hopping term computed in 64-bit fixed point.
#include <type_traits>
#include "wd_fix.cuh"
#include "wd_fix_links.h"
#include "wd_kernels.h"
#include "wd_reduce.cuh"
#include "wd_solver.h"
#include "wd_tune.h"

namespace {

// FP64 planes -> fixed-point planes (if fix is given).  *bad is set when a link
// is outside what the fixed-point kernels are written for: the integer ranges
// need |u| <= 1 and absolute row and column sums (columns: the backward terms)
// of at most sqrt(6), the look at a component's terms needs such sums of 0.99,
// and links much smaller than a unitary matrix's would lose digits below the
// fixed 2^-60.  On integers and FP32, so that HBM bounds it (once for a set of
// links), not the FP64 pipe.
struct Fixed {
    int hi, lo;   // round(x 2^60) in two limbs
    float size;   // |x|
};
__device__ __forceinline__ Fixed fixed(double x)
{
    const uint32_t hw = (uint32_t)__double2hiint(x), e = hw >> 20 & 0x7ff;
    // |x| 2^60 = m 2^(e - 1015), m of 53 bits; e <= 1023 where the link fits
    const uint64_t m = (uint64_t)(hw & 0xfffffu | (e ? 0x100000u : 0)) << 32 | (uint32_t)__double2loint(x);
    const int n = min(1015 - (int)e, 62);
    const uint64_t q = n > 0 ? (m + (1ull << (n - 1))) >> n : m << min(-n, 8);
    const long long t = (int)hw < 0 ? -(long long)q : (long long)q, t1 = (t + (1ll << 29)) >> 30;
    Fixed f{(int)t1, (int)(t - (t1 << 30)), 0.f};
    if (e > 1100) f.size = __int_as_float(0x7f800000);  // too large, infinite, NaN
    else if (e > 900) f.size = __uint_as_float((e - 896) << 23 | (uint32_t)(m >> 29 & 0x7fffffu));
    return f;
}

__global__ void __launch_bounds__(128) k_gauge_fix(const double2 *__restrict__ gauge, int4 *__restrict__ fix, int Vh,
                                                   int *bad)
{
    const int s = blockIdx.x * 128 + threadIdx.x;
    if (s >= Vh) return;
    const size_t i0 = (size_t)blockIdx.y * 9 * Vh + s;  // direction and parity
    float row[3] = {0, 0, 0}, col[3] = {0, 0, 0};
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const double2 v = gauge[i0 + (size_t)k * Vh];
        const Fixed x = fixed(v.x), y = fixed(v.y);
        if (fix) fix[i0 + (size_t)k * Vh] = make_int4(x.hi, x.lo, y.hi, y.lo);
        ok = ok && x.size <= 1.f + 0x1p-20f && y.size <= 1.f + 0x1p-20f && x.size + y.size <= 1.5f;
        row[k / 3] += x.size + y.size;
        col[k % 3] += x.size + y.size;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) ok = ok && row[k] >= 0.99f && row[k] <= 2.46f && col[k] >= 0.99f && col[k] <= 2.46f;
    if (!ok) *bad = 1;
}

struct FixArgs {
    WdGeom g;
    int cb;                // output parity (of the first blocks when both parities run)
    const double2 *in;     // source parity block; whole field when both parities run, as x and out
    const double2 *gauge;  // FP64 links, for the sites that need them
    const double2 *x;
    double2 *out;
    const int4 *links;
    double alpha, beta;    // alpha = pre * post: what the integer sums take on their exponent, and the rest
    wd_fix::Pow2 pre;
    double post;           // 1, or alpha where that is no power of two (scaled = 1)
    int scaled;
    const int *stop;
    double2 *zero;         // a parity block to clear beside out, or null
};
// One block's parity: its operand pointers
struct FixView {
    int cb;
    const double2 *in, *x;
    double2 *out;
};

// |v| 2^(1023 - E) as FP32, cut, but not to zero (v's exponent is at most E).
// On integers: as a product, a comparison and a conversion on the FP64 pipe
// these bound a hop over nothing but sites in doubt (32^4, unit links, one
// colour: 1.39 ms, now 0.51; a propagator at 16^3x32 30.7 -> 30.0).
__device__ __forceinline__ float size_of(double v, uint32_t E)
{
    const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
    const int e = (int)(hi >> 20 & 0x7ff) - (int)E + 127;
    const uint32_t b = e >= 77 ? (uint32_t)e << 23 | (hi << 3 & 0x7fffffu) | lo >> 29 : 77u << 23;
    return (hi << 1 | lo) == 0 ? 0.f : __uint_as_float(b);
}

// A closer look at a thread's components of a site in doubt: the sums S of
// the sizes of the products that make up each real, from the FP64 operands.
// Returns the reals whose S is zero as a bit mask (2k + {0: re, 1: im} for
// component k of wd_fix::site's v): the fixed-point sum may be off zero by a unit.
// Returns -1 if another S is below the share of the block scale that the
// fixed-point sum is used for: the FP64 route.
template <bool DAG, bool AOS>
__device__ __forceinline__ int small_sums(const FixArgs &a, const double2 *in, int cb, int s, int half, uint32_t E)
{
    const wd_fix::Operands<AOS> p{a.g, cb, in, nullptr};
    const WdSite c = wd_site(a.g, s, cb);
    const float least = 2.f / (1 << wd_fix::kLeastExp);  // (the block scale is 2 here)
    float sum[12] = {};  // own spin re, im per colour; spin 3 - half likewise
#pragma unroll 1
    for (int d = 0; d < 8; ++d) {
        const int mu = d >> 1;
        const bool fwd = !(d & 1), turn = mu == 0 || mu == 2;
        const int nb = wd_neighbour(a.g, s, c, mu, fwd);
        const double sg = (fwd ? -1.0 : 1.0) * (DAG ? -1.0 : 1.0);
        float ur[9], ui[9];
        const double2 *u = a.gauge + (size_t)((mu * 2 + (fwd ? cb : 1 - cb)) * 9) * a.g.Vh + (fwd ? s : nb);
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const double2 e = u[(size_t)k * a.g.Vh];
            ur[k] = size_of(e.x, 1023);
            ui[k] = size_of(e.y, 1023);
        }
        // the lower spin's terms come from the same half for mu = 0, 1, from the other for mu = 2, 3
#pragma unroll 1
        for (int which = 0; which < (mu < 2 ? 1 : 2); ++which) {
            const int h = half ^ which;
            const double sigma = h ? -1.0 : 1.0, f = mu == 1 ? -sg * sigma : mu == 2 ? sg * sigma : sg;
            const double2 *so = p.spin(nb, h), *sp = p.spin(nb, mu < 2 ? 3 - h : 2 + h);
            float hr[3], hi[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double2 x = so[k * p.colour_stride()], y = sp[k * p.colour_stride()];
                hr[k] = size_of(turn ? fma(-f, y.y, x.x) : fma(f, y.x, x.x), E);
                hi[k] = size_of(turn ? fma(f, y.x, x.y) : fma(f, y.y, x.y), E);
            }
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                float re = 0.f, im = 0.f;
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const float ar = fwd ? ur[r * 3 + b] : ur[b * 3 + r], ai = fwd ? ui[r * 3 + b] : ui[b * 3 + r];
                    re += ar * hr[b] + ai * hi[b];
                    im += ar * hi[b] + ai * hr[b];
                }
                if (which == 0) {
                    sum[2 * r] += re;
                    sum[2 * r + 1] += im;
                }
                if (mu < 2 || which == 1) {
                    sum[6 + 2 * r] += turn ? im : re;
                    sum[7 + 2 * r] += turn ? re : im;
                }
            }
        }
        float m = sum[0];
#pragma unroll
        for (int k = 1; k < 12; ++k) m = fminf(m, sum[k]);
        if (m >= least) return 0;
    }
    int zero = 0;
#pragma unroll
    for (int k = 0; k < 12; ++k) {
        if (sum[k] == 0.f) zero |= 1 << k;
        else if (sum[k] < least) return -1;
    }
    return zero;
}

// Sets right, where they need it, a thread's components t of a site that is in
// doubt or out of range.  Out of line and on memory, so that the common path
// keeps its registers (with the values alive across the call a hop took 11 %
// longer).  A hop whose sites all take the FP64 pipe here (32^4, unit links, one
// colour 1e10 of the others) takes 1.87 ms, against 0.75 in the FP64-pipe
// kernel, one thread a site.
template <bool DAG, bool AOS>
__device__ __noinline__ void rare_site(const FixArgs &a, const double2 *in, int cb, int s, int half, uint32_t E,
                                       wd_fix::Judged state, double2 *t)
{
    if (state == wd_fix::kDoubt) {
        const int zero = small_sums<DAG, AOS>(a, in, cb, s, half, E);
        if (zero >= 0) {
            for (int k = 0; k < 6; ++k) {
                if (zero >> 2 * k & 1) t[k].x = 0.0;
                if (zero >> 2 * k & 2) t[k].y = 0.0;
            }
            return;
        }
    }
    std::conditional_t<AOS, HopF64AoS<128>, HopF64<128>> p;
    p.g = a.g;
    p.cb = cb;
    p.in = in;
    p.gauge = a.gauge;
    double2 acc[12];
    wd_hop_site<DAG>(p, s, acc);
    const double pre = a.scaled ? 1.0 : a.alpha;
#pragma unroll
    for (int k = 0; k < 6; ++k) t[k] = c_scale(k < 3 ? acc[half * 3 + k] : acc[(3 - half) * 3 + k - 3], pre);
}

template <bool AOS>
__device__ __forceinline__ size_t entry(const FixArgs &a, int c, int s)
{
    return AOS ? (size_t)s * 12 + c : (size_t)c * a.g.Vh + s;
}
__device__ __noinline__ double2 scale_rare(double2 v, double f) { return c_scale(v, f); }

// alpha acc + beta x from v = pre acc.  The forms are separate kernels: FP64
// operations that a condition turns off still hold the FP64 pipe for their
// 16 cycles (with one kernel for all, D_eo at 32^3x64 took 0.391 ms, not 0.370).
enum Form {
    kPlain,   // no x (a factor that is no power of two is met by no solver)
    kPow2X,   // x, alpha a power of two: one operation per real, one rounding
    kScaledX  // x, any alpha
};
template <Form F>
__device__ __forceinline__ double2 hop_value(const FixArgs &a, const FixView &w, size_t i, double2 v)
{
    if constexpr (F == kPlain) {
        if (a.scaled) v = scale_rare(v, a.post);
        return v;
    } else {
        const double2 x = w.x[i];
        if constexpr (F == kScaledX) v = c_scale(v, a.post);
        return make_double2(fma(a.beta, x.x, v.x), fma(a.beta, x.y, v.y));
    }
}

// ---- epilogues: put() takes each component's hopping sum v, finish() the
// grid's sums of what put() added up in n.  The FP64 pipe has little room
// beside the hop's own 132 operations per site, so products are merged
// (r - al (alpha v + beta x) in two multiply-adds).
template <bool AOS_, Form F>
struct EpiStore {
    static constexpr bool AOS = AOS_;
    static constexpr int N = 0;
    using Num = double;
    __device__ __forceinline__ void put(const FixArgs &a, const FixView &w, int c, int s, double2 v, double *) const
    {
        const size_t i = entry<AOS>(a, c, s);
        w.out[i] = hop_value<F>(a, w, i, v);
        if (F == kPlain && a.zero) a.zero[i] = make_double2(0.0, 0.0);
    }
};
// t stored, |t|^2 -> alpha
struct EpiNorm {
    static constexpr bool AOS = false;
    static constexpr int N = 1;
    using Num = double;
    WdCgDev *dev;
    WdRed red;
    __device__ __forceinline__ void put(const FixArgs &a, const FixView &w, int c, int s, double2 v, double *n) const
    {
        const size_t i = entry<false>(a, c, s);
        const double2 o = hop_value<kScaledX>(a, w, i, v);
        w.out[i] = o;
        n[0] = fma(o.x, o.x, fma(o.y, o.y, n[0]));
    }
    __device__ __forceinline__ void finish(const double *t) const { wd_cg_set_alpha(dev, t[0], 0.0, false); }
};
// q not stored: r -= alpha q, y += alpha p, |r|^2 -> beta or the gate
struct EpiUpdate {
    static constexpr bool AOS = false;
    static constexpr int N = 1;
    using Num = double;
    WdCgDev *dev;
    WdRed red;
    const double2 *p;
    double2 *r, *y;
    __device__ __forceinline__ void put(const FixArgs &a, const FixView &w, int c, int s, double2 v, double *n) const
    {
        const size_t i = entry<false>(a, c, s);
        const double al = dev->are, av = -al * a.post, ax = -al * a.beta;
        const double2 x = w.x[i], pv = p[i];
        double2 rv = r[i], yv = y[i];
        rv = make_double2(fma(av, v.x, fma(ax, x.x, rv.x)), fma(av, v.y, fma(ax, x.y, rv.y)));
        yv = make_double2(fma(al, pv.x, yv.x), fma(al, pv.y, yv.y));
        r[i] = rv;
        y[i] = yv;
        n[0] = fma(rv.x, rv.x, fma(rv.y, rv.y, n[0]));
    }
    __device__ __forceinline__ void finish(const double *t) const { wd_cg_set_beta(dev, t[0]); }
};
// q stored, (p, q) -> alpha; p is a whole field
struct EpiDot {
    static constexpr bool AOS = false;
    static constexpr int N = 2;
    using Num = double;
    WdCgDev *dev;
    WdRed red;
    const double2 *p;
    __device__ __forceinline__ void put(const FixArgs &a, const FixView &w, int c, int s, double2 v, double *n) const
    {
        const size_t i = entry<false>(a, c, s);
        const double2 q = hop_value<kPow2X>(a, w, i, v), u = p[(size_t)w.cb * 12 * a.g.Vh + i];
        w.out[i] = q;
        n[0] = fma(u.x, q.x, fma(u.y, q.y, n[0]));
        n[1] = fma(u.x, q.y, fma(-u.y, q.x, n[1]));
    }
    __device__ __forceinline__ void finish(const double *t) const { wd_cg_set_alpha(dev, t[0], t[1], true); }
};
// The reliable update's second Schur hop fused with the true residual (as
// k_hop_f64_res): s = bhat - (alpha acc + beta x) in FP64, rounded to FP32
// into s32 (plane c/2, half c&1 of the float4 for component c), |s32|^2.
struct EpiRes {
    static constexpr bool AOS = false;
    static constexpr int N = 1;
    using Num = float;
    WdRed red;
    WdResSink r;
    __device__ __forceinline__ void put(const FixArgs &a, const FixView &w, int c, int s, double2 v, float *n) const
    {
        const size_t i = entry<false>(a, c, s);
        const double2 x = w.x[i], b = r.bhat[i];
        const float2 f = make_float2((float)fma(-a.post, v.x, fma(-a.beta, x.x, b.x)),
                                     (float)fma(-a.post, v.y, fma(-a.beta, x.y, b.y)));
        reinterpret_cast<float2 *>(r.s32 + (size_t)(c >> 1) * a.g.Vh + s)[c & 1] = f;
        n[0] = fmaf(f.x, f.x, fmaf(f.y, f.y, n[0]));
    }
    __device__ __forceinline__ void finish(const double *t) const { *r.result = t[0]; }
};

// |b - M x|^2 and |b|^2 -> result[0], result[1]; nothing stored
struct EpiTrueRes {
    static constexpr bool AOS = false;
    static constexpr int N = 2;
    using Num = double;
    WdRed red;
    const double2 *b;
    double *result;
    __device__ __forceinline__ void put(const FixArgs &a, const FixView &w, int c, int s, double2 v, double *n) const
    {
        const size_t i = entry<false>(a, c, s);
        const double2 x = w.x[i], bv = b[(size_t)w.cb * 12 * a.g.Vh + i];
        const double2 d = make_double2(bv.x - fma(a.beta, x.x, v.x), bv.y - fma(a.beta, x.y, v.y));
        n[0] = fma(d.x, d.x, fma(d.y, d.y, n[0]));
        n[1] = fma(bv.x, bv.x, fma(bv.y, bv.y, n[1]));
    }
    __device__ __forceinline__ void finish(const double *t) const
    {
        result[0] = t[0];
        result[1] = t[1];
    }
};

// 512 threads per SM (128 registers each).  Output sites [s_lo, s_hi).  T > 0: T threads a block, two a site; T = 0: the
// form with a direction pair per warp, 16 sites a block.  gridDim.y = 2 runs
// both parities (s_lo = 0, s_hi = Vh).
constexpr int block_threads(int T) { return T ? T : 128; }
template <bool DAG, int T, class Epi>
__global__ void __launch_bounds__(block_threads(T), 512 / block_threads(T))
    k_hop_fix(const __grid_constant__ FixArgs a, const __grid_constant__ Epi epi, int s_lo, int s_hi)
{
    wd_pdl_wait(T > 0);
    if (a.stop && *a.stop) return;
    constexpr bool AOS = Epi::AOS;
    constexpr int B = block_threads(T);
    extern __shared__ __align__(16) char smem[];
    FixView w{a.cb, a.in, a.x, a.out};
    if (gridDim.y == 2) {
        const size_t half_field = (size_t)12 * a.g.Vh;
        w.cb = a.cb ^ blockIdx.y;
        w.in += (1 - w.cb) * half_field;
        w.x += w.cb * half_field;
        w.out += w.cb * half_field;
    }
    const wd_fix::Operands<AOS> p{a.g, w.cb, w.in, a.links};
    const int l = threadIdx.x & 31, half = l & 1;
    const int s0 = s_lo + (T ? (int)(blockIdx.x * B + threadIdx.x) >> 1 : (int)blockIdx.x * 16 + (l >> 1));
    const int s = s0 < s_hi ? s0 : s_hi - 1;
    double2 v[6];
    uint32_t E;
    wd_fix::Judged state;
    if constexpr (T > 0) state = wd_fix::site<DAG>(p, *reinterpret_cast<wd_fix::Stage<B> *>(smem), s, half, a.pre, v, E);
    else state = wd_fix::site_split<DAG>(p, *reinterpret_cast<wd_fix::Split *>(smem), s, half, a.pre, v, E);
    typename Epi::Num n[Epi::N ? Epi::N : 1] = {};
    const int warp = threadIdx.x >> 5;  // split form: warps 0-2 hold colour `warp` of the two spins
    if (state != wd_fix::kGood && (T > 0 || warp < 3)) {
        double2 t[6];
#pragma unroll
        for (int k = 0; k < (T ? 6 : 2); ++k) t[T ? k : 3 * k + warp] = v[k];
        rare_site<DAG, AOS>(a, w.in, w.cb, s, half, E, state, t);
#pragma unroll
        for (int k = 0; k < (T ? 6 : 2); ++k) v[k] = t[T ? k : 3 * k + warp];
    }
    if (s0 < s_hi && (T > 0 || warp < 3)) {
#pragma unroll
        for (int k = 0; k < (T ? 6 : 2); ++k) {
            const int spin = k < (T ? 3 : 1) ? half : 3 - half;
            epi.put(a, w, spin * 3 + (T ? k % 3 : warp), s, v[k], n);
        }
    }
    if constexpr (Epi::N > 0) {
        double d[Epi::N], t[Epi::N];
#pragma unroll
        for (int k = 0; k < Epi::N; ++k) d[k] = (double)n[k];
        if (wd_grid_sum_n<B, Epi::N>(d, epi.red, t)) epi.finish(t);
    }
}

// A launch over up to this many output sites takes the form with a direction
// pair per warp: there the chip has warps to spare and the time is one
// thread's chain (us per hop, split / not: 6.7 / 9.1 at 4096 sites, 6.9 / 10.3
// at 8192, 11.8 / 12.3 at 13824, 12.8 / 14.3 at 16384, 16.6 / 14.4 at 20736).
constexpr int kSplitSites = 16384;

template <bool DAG, int T, class Epi>
void launch_fix(cudaStream_t stream, const FixArgs &a, const Epi &epi, bool both, int s_lo, int s_hi)
{
    constexpr int B = T ? T / 2 : 16;  // sites a block
    constexpr size_t sm = T ? sizeof(wd_fix::Stage<T ? T : 128>) : sizeof(wd_fix::Split);
    const dim3 grid((unsigned)((s_hi - s_lo + B - 1) / B), both ? 2 : 1);
    // blocks that wait for the predecessor take the SMs it leaves idle first: with
    // fewer than three blocks per SM the early launch leaves them unevenly spread
    // (15.5 against 12.3 us at 13824 sites; 15.5 against 18.4 at 32768, 512 blocks)
    const bool early = T == 0 || grid.x * grid.y >= 3 * 152;
    wd_launch_pdl(early, k_hop_fix<DAG, T, Epi>, grid, T ? T : 128, sm, stream, a, epi, s_lo, s_hi);
}

template <bool DAG, class Epi>
wd_status run_fix(wd_context *ctx, cudaStream_t stream, const FixArgs &a, const Epi &epi, bool both, int s_lo, int s_hi)
{
    if ((both ? 2 : 1) * (s_hi - s_lo) <= kSplitSites) launch_fix<DAG, 0>(stream, a, epi, both, s_lo, s_hi);
    else launch_fix<DAG, 128>(stream, a, epi, both, s_lo, s_hi);
    WD_LAUNCHED(ctx);
    return WD_OK;
}
template <bool DAG, class Epi>
wd_status run_fix(wd_context *ctx, const FixArgs &a, const Epi &epi, bool both = false)
{
    return run_fix<DAG>(ctx, ctx->stream, a, epi, both, 0, a.g.Vh);
}

// stored hops, in the form their x and alpha ask for
template <bool AOS>
wd_status store_fix(wd_context *ctx, cudaStream_t stream, const FixArgs &a, int dag, bool both, int s_lo, int s_hi)
{
    auto run = [&](auto epi) {
        return dag ? run_fix<true>(ctx, stream, a, epi, both, s_lo, s_hi) : run_fix<false>(ctx, stream, a, epi, both, s_lo, s_hi);
    };
    if (!a.x) return run(EpiStore<AOS, kPlain>());
    if (!a.scaled) return run(EpiStore<AOS, kPow2X>());
    return run(EpiStore<AOS, kScaledX>());
}

FixArgs fix_args(const wd_lattice *lat, const void *in, void *out, const void *x, int cb, double alpha, double beta,
                 const int *stop = nullptr)
{
    const F64Scale f = F64Scale::make(alpha);
    const bool pow2 = f.mode == 1 || (f.mode == 2 && f.shift >= -60 && f.shift <= 60);
    const wd_fix::Pow2 pre{pow2 ? f.shift : 0, pow2 && alpha < 0 ? 0x80000000u : 0u};
    return FixArgs{lat->g, cb, (const double2 *)in, lat->gauge, (const double2 *)x, (double2 *)out,
                   (const int4 *)lat->gauge_fix, alpha, beta, pre, pow2 ? 1.0 : alpha, !pow2, stop, nullptr};
}

// A launch's hold on the lattice's fixed-point links: the lock shared, if they
// are there or can be built.  A stream that is being captured may not use them:
// the graph would keep their address past the moment they are freed or replaced,
// while the FP64 links stay where they are as long as the lattice.  Nor may a
// lattice size whose FP64-pipe shape the caller has pinned: that kernel runs.
struct Links {
    WdFixShared lock;
    Links(wd_context *ctx, const wd_lattice *lat, cudaStream_t stream)
    {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return;
        if (wd_tune_pinned(ctx, "hop_f64", lat->g.Vh)) return;
        lock = WdFixShared(wd_fix_mutex());
        if (lat->fix_state == wd_lattice::kFixReady) return;
        lock.unlock();
        if (!wd_fix_ensure(ctx, lat)) return;
        lock.lock();
        if (lat->fix_state != wd_lattice::kFixReady) lock.unlock();  // taken back in between
    }
    explicit operator bool() const { return lock.owns_lock(); }
};

}  // namespace

wd_status wd_gauge_to_fix(wd_context *ctx, const wd_lattice *lat, void *fix, int *bad)
{
    const int Vh = lat->g.Vh;
    WD_CUDA(ctx, cudaMemsetAsync(bad, 0, sizeof(int), ctx->stream));
    k_gauge_fix<<<dim3((Vh + 127) / 128, 8), 128, 0, ctx->stream>>>(lat->gauge, (int4 *)fix, Vh, bad);
    WD_LAUNCHED(ctx);
    return WD_OK;
}

WdTried wd_hop_fix(wd_context *ctx, const wd_lattice *lat, const double2 *in, double2 *out, const double2 *x, int cb,
                   int dag, double alpha, double beta, const int *stop, double2 *zero)
{
    const Links links(ctx, lat, ctx->stream);
    if (!links) return {};
    FixArgs a = fix_args(lat, in, out, x, cb, alpha, beta, stop);
    a.zero = zero;
    // (one shape: 64 and 32 threads a block run within 0.3 % of 128)
    return store_fix<false>(ctx, ctx->stream, a, dag, false, 0, lat->g.Vh);
}

WdTried wd_hop_fix_M(wd_context *ctx, const wd_lattice *lat, const double2 *in, double2 *out, double mass, int dag,
                     const int *stop)
{
    const Links links(ctx, lat, ctx->stream);
    if (!links) return {};
    return store_fix<false>(ctx, ctx->stream, fix_args(lat, in, out, in, 0, -0.5, 4.0 + mass, stop), dag, true, 0,
                            lat->g.Vh);
}

WdTried wd_hop_fix_residual(wd_context *ctx, const wd_lattice *lat, const double2 *in, const double2 *x, double alpha,
                            double beta, const WdResSink &r)
{
    const Links links(ctx, lat, ctx->stream);
    if (!links) return {};
    return run_fix<false>(ctx, fix_args(lat, in, nullptr, x, 0, alpha, beta), EpiRes{r.red, r});
}

WdTried wd_hop_fix_norm(wd_context *ctx, const wd_lattice *lat, WdVec in, WdVec t, WdVec p, double mass, WdCgDev *dev,
                        WdRed red)
{
    const Links links(ctx, lat, ctx->stream);
    if (!links) return {};
    const double a = 4.0 + mass;
    return run_fix<false>(ctx, fix_args(lat, in.p, t.p, p.p, 0, -0.25 / a, a, &dev->stop), EpiNorm{dev, red});
}

WdTried wd_hop_fix_update(wd_context *ctx, const wd_lattice *lat, WdVec in, WdVec t, WdVec p, WdVec r, WdVec x,
                          double mass, WdCgDev *dev, WdRed red)
{
    const Links links(ctx, lat, ctx->stream);
    if (!links) return {};
    const double a = 4.0 + mass;
    return run_fix<true>(ctx, fix_args(lat, in.p, nullptr, t.p, 0, -0.25 / a, a, &dev->stop),
                         EpiUpdate{dev, red, (const double2 *)p.p, (double2 *)r.p, (double2 *)x.p});
}

WdTried wd_hop_fix_M_dot(wd_context *ctx, const wd_lattice *lat, WdVec in, WdVec q, WdVec p, double mass, WdCgDev *dev,
                         WdRed red)
{
    const Links links(ctx, lat, ctx->stream);
    if (!links) return {};
    return run_fix<true>(ctx, fix_args(lat, in.p, q.p, in.p, 0, -0.5, 4.0 + mass, &dev->stop),
                         EpiDot{dev, red, (const double2 *)p.p}, true);
}

WdTried wd_hop_fix_M_residual(wd_context *ctx, const wd_lattice *lat, const double2 *b, const double2 *x, double mass,
                              WdRed red, double *result)
{
    const Links links(ctx, lat, ctx->stream);
    if (!links) return {};
    return run_fix<false>(ctx, fix_args(lat, x, nullptr, x, 0, -0.5, 4.0 + mass),
                          EpiTrueRes{red, b, result}, true);
}

WdTried wd_hop_fix_aos_range(wd_context *ctx, cudaStream_t stream, const wd_lattice *lat, const double2 *in_aos,
                             double2 *out_aos, const double2 *x_aos, int cb, int dag, double alpha, double beta,
                             int s_lo, int s_hi)
{
    const Links links(ctx, lat, stream);
    if (!links) return {};
    return store_fix<true>(ctx, stream, fix_args(lat, in_aos, out_aos, x_aos, cb, alpha, beta), dag, false, s_lo, s_hi);
}
