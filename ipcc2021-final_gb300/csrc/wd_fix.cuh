// wd_fix.cuh -- the FP64 hopping term in 64-bit fixed point, on the integer
// pipes.
//
// GB300 issues 2 FP64 operations per clock and SM; the FP64 form of the hop
// (wd_hop.cuh) needs 792 of them per site, which bounds it at 1.45 ms at
// 32^3x64 however its 0.24 ms of memory traffic is arranged.  The integer
// pipes take 24-28 wide multiply-adds (32 x 32 + 64 bits) per clock and SM, and
// SU(3) links have entries within [-1, 1], so the matrix products are done on
// integers: a link entry is round(u 2^60) in two 30-bit limbs (laid out
// once, by the first hop on a set of links), a projected half-spinor is brought to one exponent per output
// site (a block scale) in limbs of 28 and 30 bits, and a product costs three
// wide multiply-adds (the low x low one is below the last place).  The sums
// over colours and over the eight directions are exact integers and are
// rounded to FP64 once.  The FP64 pipe keeps the projections (one addition
// per real, as in the FP64 form) and the final conversion.
//
// Precision.  With all |h| < 2^E', a half-spinor value is cut at 2^(E'-58),
// a link at 2^-61, and a direction's term errs by about one unit of 2^(E'-58);
// the FP64 form rounds each of its ~25 operations per component at
// 2^-53 of the running sum.  Measured relative L2 error of one hop, Gaussian
// fields: 1.4e-16 here, 2.0e-16 in FP64 (both against torch's own FP64 sums).
// The unit is one for all colours, spins and neighbours of a site.  So that no
// component loses digits beside larger ones, the sums stand only where every
// component's own terms are large enough for it (kLeastExp below); other
// sites, and those whose exponents do not fit (block exponents beyond 2^877,
// nonzero values below 2^-894, NaN, infinity), are recomputed on the FP64 pipe
// by the calling kernel.  The look at the terms is 48 of a thread's 3000
// instructions (0.354 -> 0.371 ms at 32^3x64, 0.118 -> 0.120 at 24^3x48).
//
// Two threads share a site: each carries one of the two half-spinor
// components through the eight link products and accumulates its own upper
// spin and its shares of the two lower spins, exchanged once at the end.
// That halves the accumulators (36 registers), needs no spinor twice, and
// fills the chip at half the volume.  Each pair's operands for the next
// direction are copied to shared memory by cp.async while the current ones
// are multiplied (0.472 -> 0.386 ms at 32^3x64); a row's links are read
// from there when the row is due (0.377).  Complex products take three real
// ones (Gauss): additions are cheaper than wide multiply-adds here.
// Measured at 32^3x64: 0.371 ms (FP64 form 1.453 ms), 4.34 TB/s of
// compulsory bytes, 65 % of measured HBM.  What bounds it now is issue and
// the integer pipes together (at 24^3x48 fma-heavy pipe 58 %, FP64 54 %, ALU
// 37 %, issue slots 45 % busy with 15 warps an SM); with every load served by
// L1 it is no faster.  Dropped: converting with F2I.S64.F64 (0.67 ms: it
// occupies the FP64 pipe), projecting after conversion on
// integers (0.458 ms before staging), 20 warps per SM at 96 registers (0.395
// ms against 0.372), the next direction's projection ahead of the current
// product (0.381 ms).
#pragma once
#include "wd_async.cuh"
#include "wd_hop_f64.cuh"

// Block scale of a site: E is the largest biased FP64 exponent among the
// projected half-spinors met so far; a value x is held as the integer
// x 2^(1080-E), |.| < 2^58.  Links are integers round(u 2^60) = hi 2^30 + lo.
namespace wd_fix {

constexpr int kUnit = 1080;        // x = T 2^(E - kUnit)
constexpr int kExpTiny = 128;      // nonzero values with exponents up to this need the FP64 route ...
constexpr int kExpLow = 200;       // ... when the block exponent is below this
constexpr int kExpHigh = 1900;     // block exponents above this (and NaN, infinity) take the FP64 route

// What is known of a thread's components at a site
enum Judged {
    kGood,   // as good as FP64 arithmetic gives them
    kDoubt,  // one may be too small beside the block scale
    kFp64    // values that the block scale does not hold
};
// A component may be small because its terms cancel, or because they are all
// small beside the block's largest value (one colour, spin or link entry beside
// another); then the fixed unit, 2^-58 of the block scale, may be large beside it.
// Let S be the sum of |U| |h| over the products behind a real of the result.
// A row of a link's |re| and |im| adds up to at least 0.99 (checked when the
// fixed-point links are made), so one direction whose half-spinor has its six
// reals at 2^-7 of the block scale or more gives all reals that it enters S
// >= 0.99 x 2^-7 of the scale: the unit is below 2^-50.9 S.  In a dense field the
// eight directions miss that for two half-sites in ten million.
constexpr int kLeastExp = 7;

__device__ __forceinline__ float absmax3(float a, float b, float c)
{
    float d;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// The FP64 number with words (hi, lo) as limbs l1 2^30 + l0 of trunc(x
// 2^(1080-E)) (off by less than one unit below zero); ekey = E<<21 | 0x1fffff.
// sh: E less its exponent
__device__ __forceinline__ void limbs(uint32_t hi, uint32_t lo, uint32_t ekey, int &l1, int &l0, uint32_t &sh)
{
    sh = (ekey - (hi << 1)) >> 21;  // E - exponent (the sign bit shifts out)
    const uint32_t h7 = (__funnelshift_l(lo, hi, 7) & 0x07ffffffu) | 0x08000000u;
    unsigned long long w = ((unsigned long long)h7 << 32) | (lo << 7);
    asm("shr.u64 %0, %0, %1;" : "+l"(w) : "r"(sh));
    const uint32_t neg = (uint32_t)((int)hi >> 31);  // one's complement: the missing unit is 2^-60 of the block scale
    l1 = (int)((uint32_t)(w >> 32) ^ neg);
    l0 = (int)(((uint32_t)w ^ neg) >> 2);
}

// c + a b.  Written as the carry pair: ptxas makes one wide multiply-add of
// it, where mad.wide.s32 costs an extra ALU operation (measured).
__device__ __forceinline__ long long macw(long long c, int a, int b)
{
    long long d;
    asm("{\n\t.reg .u32 l, h;\n\tmov.b64 {l, h}, %1;\n\tmad.lo.cc.s32 l, %2, %3, l;\n\tmadc.hi.s32 h, %2, %3, h;\n\t"
        "mov.b64 %0, {l, h};\n\t}"
        : "=l"(d)
        : "l"(c), "r"(a), "r"(b));
    return d;
}

// (re, im) of sum_b U[a][b] h_b (forward) or sum_b conj(U[b][a]) h_b
// (backward) by three products per complex one: with u = c + i d and
// h = x + i y, k = x (c + d): re = k - d (x + y), im = k + c (y - x)
// (backward d -> -d).  x, q = -(x + y) (backward x + y), v = y - x: limbs.
template <bool FWD, int T>
__device__ __forceinline__ void su3_row(const int4 (*link)[T / 2], const int *x1, const int *x0, const int *q1,
                                        const int *q0, const int *v1, const int *v0, int a, long long &re, long long &im)
{
    long long k, m;
    int4 u[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        u[b] = link[FWD ? a * 3 + b : b * 3 + a][threadIdx.x >> 1];
        const int s1 = FWD ? u[b].x + u[b].z : u[b].x - u[b].z, s0 = FWD ? u[b].y + u[b].w : u[b].y - u[b].w;
        k = b == 0 ? (long long)s1 * x1[b] : macw(k, s1, x1[b]);
        m = macw(b == 0 ? 1ll << 29 : m, s1, x0[b]);
        m = macw(m, s0, x1[b]);
    }
    long long rk = k, rm = m, ik = k, im_ = m;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        rk = macw(rk, u[b].z, q1[b]);
        rm = macw(rm, u[b].z, q0[b]);
        rm = macw(rm, u[b].w, q1[b]);
        ik = macw(ik, u[b].x, v1[b]);
        im_ = macw(im_, u[b].x, v0[b]);
        im_ = macw(im_, u[b].y, v1[b]);
    }
    re = rk + (rm >> 30);
    im = ik + (im_ >> 30);
}

// Accumulators of one thread: its own spin (o), and its shares of the two
// lower spins reached through mu = 0, 1 (P) and mu = 2, 3 (Q); re, im per colour.
struct Acc {
    long long o[6], P[6], Q[6];
    uint32_t E;
    uint32_t tiny;  // OR of nonzero bits of values too small for the block scale
    // of the half-spinors reached through mu = 0, 1 and through mu = 2, 3: the largest of the
    // exponents of their smallest reals; at least 1 if one of them is not zero
    uint32_t least[2];
};

// Two slots of one direction's operands for a block of T threads (T / 2 sites)
template <int T>
struct Stage {
    double2 spin[2][6][T];   // each thread's own spin and partner spin, 3 colours each
    int4 link[2][9][T / 2];  // one link matrix per site
};

// What a hop reads: the source parity block (SoA planes, or the reference's
// site-major layout) and the fixed-point links
template <bool AOS>
struct Operands {
    WdGeom g;
    int cb;             // output parity
    const double2 *in;  // parity 1 - cb
    const int4 *links;
    __device__ __forceinline__ const double2 *spin(int s, int k) const
    {
        return AOS ? in + (size_t)s * 12 + k * 3 : in + (size_t)(k * 3) * g.Vh + s;
    }
    __device__ __forceinline__ size_t colour_stride() const { return AOS ? 1 : (size_t)g.Vh; }
};

template <int MU, bool FWD, int T, bool AOS>
__device__ __forceinline__ void stage(const Operands<AOS> &p, Stage<T> &sm, int slot, int s, const WdSite &c, int half)
{
    const int nb = wd_neighbour(p.g, s, c, MU, FWD), i = threadIdx.x;
    const double2 *a = p.spin(nb, half), *b = p.spin(nb, MU < 2 ? 3 - half : 2 + half);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        wd_cp_async_ca<16>(&sm.spin[slot][k][i], a + k * p.colour_stride());
        wd_cp_async_ca<16>(&sm.spin[slot][3 + k][i], b + k * p.colour_stride());
    }
    // the pair's two threads copy alternate elements of its link
    const int4 *l = p.links + (size_t)((MU * 2 + (FWD ? p.cb : 1 - p.cb)) * 9 + half) * p.g.Vh + (FWD ? s : nb);
#pragma unroll
    for (int k = 0; k < 4; ++k) wd_cp_async_cg16(&sm.link[slot][2 * k + half][i >> 1], l + (size_t)(2 * k) * p.g.Vh);
    if (half == 0) wd_cp_async_cg16(&sm.link[slot][8][i >> 1], l + (size_t)8 * p.g.Vh);
    wd_cp_async_commit();
}

template <int MU, bool FWD, bool DAG, bool FIRST, int T>
__device__ __forceinline__ void dir(const Stage<T> &sm, int slot, int half, double sigma, Acc &A)
{
    constexpr int SG = (FWD ? -1 : 1) * (DAG ? -1 : 1);
    double2 so[3], sp[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        so[k] = sm.spin[slot][k][threadIdx.x];
        sp[k] = sm.spin[slot][3 + k][threadIdx.x];
    }
    // partner term: mu 0: sg i b, mu 1: -sg sigma b, mu 2: sg sigma i b, mu 3: sg b
    constexpr int C0 = MU == 1 ? -SG : SG;
    const double cb_ = (MU == 1 || MU == 2) ? C0 * sigma : (double)C0;
    double2 h[3];
    float m = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if constexpr (MU == 0 || MU == 2) h[k] = make_double2(fma(-cb_, sp[k].y, so[k].x), fma(cb_, sp[k].x, so[k].y));
        else h[k] = make_double2(fma(cb_, sp[k].x, so[k].x), fma(cb_, sp[k].y, so[k].y));
        m = absmax3(m, __int_as_float(__double2hiint(h[k].x)), __int_as_float(__double2hiint(h[k].y)));
    }
    const uint32_t some = min(__float_as_uint(m), 1u);
    m = absmax3(m, __shfl_xor_sync(0xffffffffu, m, 1), m);
    const uint32_t mb = __float_as_uint(m) & 0x7fffffffu;
    const uint32_t e = mb >> 20;
    if (mb < ((uint32_t)(kExpTiny + 1) << 20)) {
#pragma unroll
        for (int k = 0; k < 3; ++k)
            A.tiny |= (uint32_t)(__double2hiint(h[k].x) << 1) | (uint32_t)__double2loint(h[k].x) |
                      (uint32_t)(__double2hiint(h[k].y) << 1) | (uint32_t)__double2loint(h[k].y);
    }
    if constexpr (FIRST) {
        A.E = e > (uint32_t)kExpTiny ? e : kExpTiny;
    } else if (__any_sync(0xffffffffu, e > A.E)) {
        const uint32_t d = e > A.E ? (e - A.E > 63 ? 63 : e - A.E) : 0;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            A.o[k] >>= d;
            A.P[k] >>= d;
            if (MU >= 2 && !(MU == 2 && FWD)) A.Q[k] >>= d;
        }
        A.E = e > A.E ? e : A.E;
    }
    const uint32_t ekey = (A.E << 21) | 0x1fffffu;
    int x1[3], x0[3], q1[3], q0[3], v1[3], v0[3];
    uint32_t sh = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        int y1, y0;
        uint32_t sx, sy;
        limbs(__double2hiint(h[k].x), __double2loint(h[k].x), ekey, x1[k], x0[k], sx);
        limbs(__double2hiint(h[k].y), __double2loint(h[k].y), ekey, y1, y0, sy);
        sh = k ? __vimax3_u32(sh, sx, sy) : max(sx, sy);
        q1[k] = FWD ? -(x1[k] + y1) : x1[k] + y1;
        q0[k] = FWD ? -(x0[k] + y0) : x0[k] + y0;
        v1[k] = y1 - x1[k];
        v0[k] = y0 - x0[k];
    }
    A.least[MU / 2] = __vimax3_u32(A.least[MU / 2], A.E - sh, some);
    const long long hm64 = -(long long)half;  // sigma: all ones on the second half-spinor
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        long long tr, ti;
        su3_row<FWD, T>(sm.link[slot], x1, x0, q1, q0, v1, v0, a, tr, ti);
        if constexpr (FIRST) {
            A.o[2 * a] = tr;
            A.o[2 * a + 1] = ti;
        } else {
            A.o[2 * a] += tr;
            A.o[2 * a + 1] += ti;
        }
        // lower spins: mu 0: P -= sg i t;  1: P -= sg sigma t;  2: Q -= sg sigma i t;  3: Q += sg t
        // (sigma = -1 by one's complement: the forward and backward terms'
        // missing units cancel, or leave one unit of 2^-57 of the block scale)
        if constexpr (MU == 1 || MU == 2) {
            tr ^= hm64;
            ti ^= hm64;
        }
        long long *d = MU < 2 ? A.P : A.Q;
        if constexpr (FIRST) {  // MU == 0
            d[2 * a] = SG > 0 ? ti : -ti;
            d[2 * a + 1] = SG > 0 ? -tr : tr;
        } else if constexpr (MU == 0 || MU == 2) {  // -sg i t = sg (ti, -tr)
            if constexpr (SG > 0) {
                d[2 * a] += ti;
                d[2 * a + 1] -= tr;
            } else {
                d[2 * a] -= ti;
                d[2 * a + 1] += tr;
            }
        } else {
            constexpr int K = MU == 1 ? -SG : SG;
            if constexpr (K > 0) {
                d[2 * a] += tr;
                d[2 * a + 1] += ti;
            } else {
                d[2 * a] -= tr;
                d[2 * a + 1] -= ti;
            }
        }
    }
}

// sign * T 2^(E - kUnit + shift) as FP64, T rounded once; kexp = (E - kUnit +
// shift) << 20, sign = 0 or the sign bit (exponents here are far from FP64's
// limits: see the ranges above)
__device__ __forceinline__ double value(long long T, int kexp, uint32_t sign)
{
    const double v = (double)T;
    const int hi = __double2hiint(v);
    return hi ? __hiloint2double((int)((uint32_t)(hi + kexp) ^ sign), __double2loint(v)) : 0.0;
}

// a power-of-two factor of the result, applied on the exponent: sign 2^shift
struct Pow2 {
    int shift;      // |shift| <= 60
    uint32_t sign;
};

__device__ __forceinline__ bool in_range(uint32_t E, uint32_t tiny)
{
    return E <= (uint32_t)kExpHigh && !(tiny && E < (uint32_t)kExpLow);
}

__device__ __forceinline__ Judged judged(uint32_t E, uint32_t tiny, bool good)
{
    return !in_range(E, tiny) ? kFp64 : good ? kGood : kDoubt;
}
// least reaches 2^-kLeastExp of the block scale 2^(E + 1), or nothing is there
__device__ __forceinline__ bool good(uint32_t least, uint32_t E) { return least > E - kLeastExp || !least; }

__device__ __forceinline__ void clear(Acc &A)
{
    A.least[0] = A.least[1] = 0;

#pragma unroll
    for (int k = 0; k < 6; ++k) A.o[k] = A.P[k] = A.Q[k] = 0;
    A.tiny = 0;
    A.E = kExpTiny;
}

// f times the hopping term at site s for the thread pair (half = 0, 1):
// v[0..2] is spin `half`, v[3..5] spin 3 - half, E the block exponent.
template <bool DAG, int T, bool AOS>
__device__ __forceinline__ Judged site(const Operands<AOS> &p, Stage<T> &sm, int s, int half, Pow2 f, double2 *v,
                                       uint32_t &E)
{
    const WdSite c = wd_site(p.g, s, p.cb);
    const double sigma = half ? -1.0 : 1.0;
    Acc A;
    clear(A);
    stage<0, true, T>(p, sm, 0, s, c, half);
    // the copies of this direction have landed, and every lane has read the
    // other slot, before the next direction's copies go into it
    auto step = [&](auto mu, auto fwd) {
        constexpr int MU = decltype(mu)::value;
        constexpr bool FWD = decltype(fwd)::value;
        constexpr int S = FWD ? 0 : 1;
        wd_cp_async_wait<0>();
        __syncwarp();
        if constexpr (FWD) stage<MU, false, T>(p, sm, 1, s, c, half);
        else if constexpr (MU < 3) stage<(MU + 1) & 3, true, T>(p, sm, 0, s, c, half);
        dir<MU, FWD, DAG, MU == 0 && FWD, T>(sm, S, half, sigma, A);
    };
    auto both = [&](auto mu) {
        step(mu, std::true_type());
        step(mu, std::false_type());
    };
    both(std::integral_constant<int, 0>());
    both(std::integral_constant<int, 1>());
    both(std::integral_constant<int, 2>());
    both(std::integral_constant<int, 3>());
    const uint32_t tiny = A.tiny | __shfl_xor_sync(0xffffffffu, A.tiny, 1);
    const int kexp = ((int)A.E - kUnit + f.shift) << 20;
    E = A.E;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const long long lr = A.P[2 * k] + __shfl_xor_sync(0xffffffffu, A.Q[2 * k], 1);
        const long long li = A.P[2 * k + 1] + __shfl_xor_sync(0xffffffffu, A.Q[2 * k + 1], 1);
        v[k] = make_double2(value(A.o[2 * k], kexp, f.sign), value(A.o[2 * k + 1], kexp, f.sign));
        v[3 + k] = make_double2(value(lr, kexp, f.sign), value(li, kexp, f.sign));
    }
    // (the lower spin's terms of mu = 2, 3 come from the partner's half)
    const uint32_t own = max(A.least[0], A.least[1]), low = max(A.least[0], __shfl_xor_sync(0xffffffffu, A.least[1], 1));
    // sums without terms are exactly zero, but for the missing units of negative zeros
    if (__any_sync(0xffffffffu, !own || !low)) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (!own) v[k] = make_double2(0.0, 0.0);
            if (!low) v[3 + k] = make_double2(0.0, 0.0);
        }
    }
    return judged(E, tiny, good(own, E) && good(low, E));
}

// The same with a direction pair per warp, for lattices too small to fill the
// chip with two threads a site: the block's four warps take mu = 0..3 of its
// 16 sites, leave their integer sums in shared memory, and warps 0-2 add up
// colour 0-2 of the two spins: v[0] of spin `half`, v[1] of spin 3 - half.
struct Split {
    Stage<128> st;
    uint32_t E[4][32], tiny[4][32], least[4][32];
    // a thread's sums (re, im): of its own spin's colour c (k = c) and lower share (k = 3 + c), in
    // the place of its spinor copies once it has read them
    __device__ __forceinline__ longlong2 &sum(int warp, int k, int lane)
    {
        return reinterpret_cast<longlong2 &>(st.spin[0][k][warp * 32 + lane]);
    }
};

template <bool DAG, bool AOS>
__device__ __forceinline__ Judged site_split(const Operands<AOS> &p, Split &sm, int s, int half, Pow2 f, double2 *v,
                                             uint32_t &E)
{
    const WdSite c = wd_site(p.g, s, p.cb);
    const double sigma = half ? -1.0 : 1.0;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    auto pair = [&](auto mu) {
        constexpr int MU = decltype(mu)::value;
        Acc A;
        clear(A);
        stage<MU, true, 128>(p, sm.st, 0, s, c, half);
        stage<MU, false, 128>(p, sm.st, 1, s, c, half);
        wd_cp_async_wait<0>();
        __syncwarp();
        dir<MU, true, DAG, false, 128>(sm.st, 0, half, sigma, A);
        dir<MU, false, DAG, false, 128>(sm.st, 1, half, sigma, A);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const long long *d = MU < 2 ? A.P : A.Q;
            sm.sum(MU, k, l) = make_longlong2(A.o[2 * k], A.o[2 * k + 1]);
            sm.sum(MU, 3 + k, l) = make_longlong2(d[2 * k], d[2 * k + 1]);
        }
        sm.E[MU][l] = A.E;
        sm.tiny[MU][l] = A.tiny;
        sm.least[MU][l] = A.least[MU / 2];
    };
    if (w == 0) pair(std::integral_constant<int, 0>());
    else if (w == 1) pair(std::integral_constant<int, 1>());
    else if (w == 2) pair(std::integral_constant<int, 2>());
    else pair(std::integral_constant<int, 3>());
    __syncthreads();
    uint32_t tiny = 0, own = 0, low = 0;
    E = 0;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int j = m < 2 ? l : l ^ 1;  // the lower share of mu = 2, 3 is the partner's
        own = max(own, sm.least[m][l]);
        low = max(low, sm.least[m][j]);
        E = max(E, sm.E[m][l]);  // the pair's two lanes hold the same exponent
        tiny |= sm.tiny[m][l] | sm.tiny[m][l ^ 1];
    }
    if (w < 3) {
        long long t[4] = {0, 0, 0, 0};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const uint32_t d = min(E - sm.E[m][l], 63u);
            const int j = m < 2 ? l : l ^ 1;
            const longlong2 a = sm.sum(m, w, l), b = sm.sum(m, 3 + w, j);
            t[0] += a.x >> d;
            t[1] += a.y >> d;
            t[2] += b.x >> d;
            t[3] += b.y >> d;
        }
        const int kexp = ((int)E - kUnit + f.shift) << 20;
        v[0] = make_double2(value(t[0], kexp, f.sign), value(t[1], kexp, f.sign));
        v[1] = make_double2(value(t[2], kexp, f.sign), value(t[3], kexp, f.sign));
        if (!own) v[0] = make_double2(0.0, 0.0);
        if (!low) v[1] = make_double2(0.0, 0.0);
    }
    return judged(E, tiny, good(own, E) && good(low, E));
}

}  // namespace wd_fix
