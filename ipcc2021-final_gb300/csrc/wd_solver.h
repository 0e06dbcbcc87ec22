// wd_solver.h -- operator compositions and work buffers shared by the solvers (internal).
#pragma once
#include "wd_internal.cuh"

// A device vector owned by a solver (freed on scope exit).
struct WdVecBuf {
    WdVec v;
    wd_context *ctx = nullptr;  // owner of the cached block
    WdVecBuf() = default;
    WdVecBuf(const WdVecBuf &) = delete;
    WdVecBuf &operator=(const WdVecBuf &) = delete;
    ~WdVecBuf() { release(); }
    void release();
};
wd_status wd_vec_alloc(wd_context *ctx, WdVecBuf &b, wd_precision prec, int64_t n_complex);

// M (dag=0) or M^dag on full-lattice vectors of one storage
wd_status wd_apply_M_v(wd_context *ctx, const wd_lattice *lat, WdVec in, WdVec out, double mass, int dag,
                       const int *stop = nullptr);
// Schur operator a - D_eo D_oe/(4a) (or its adjoint) on even blocks; tmp_o is an odd block
wd_status wd_apply_Mhat_v(wd_context *ctx, const wd_lattice *lat, WdVec v, WdVec out, WdVec tmp_o, double mass,
                          int dag);
// |b - M x| / |b| in FP64
wd_status wd_true_residual(wd_context *ctx, const wd_lattice *lat, const double2 *b, const double2 *x, double mass,
                           double *rel);
// mixed-precision (FP32 / FP16 inner) even-odd CG with reliable updates
wd_status wd_solve_cg_eo_mixed(wd_context *ctx, const wd_lattice *lat, const double2 *src, double2 *x,
                               const wd_solver_params *prm, wd_solver_stats *stats);
// reliable-update pieces shared by the mixed solvers (wd_mixed.cu):
// xh (FP64 or double-float) += xs (FP32), xs = 0
wd_status wd_mx_accum(wd_context *ctx, int Vh, wd_precision H, WdVec xs, WdVec xh);
// one system's buffers for a reliable update (even-parity half-lattice blocks)
struct WdMxReliable {
    WdVec xs;         // FP32 solution increment (zeroed)
    WdVec x_e;        // high-precision solution
    WdVec bhat;       // high-precision Schur source
    WdVec tmp_oh;     // high-precision odd-parity work
    WdVec scratch_h;  // high-precision work, used as two FP32 blocks
    WdVec rs;         // FP32 iterated residual, receives Mhat^dag s
    bool x_zero = false;  // x_e and xs are zero: s is bhat
};
// x_e += xs; s = bhat - Mhat x_e (high precision, kept only as FP32);
// rs = Mhat^dag s (FP32); rr = |rs|^2, ss = |s|^2; p_restart (storage L) <- rs
// when given
wd_status wd_mx_reliable(wd_context *ctx, const wd_lattice *lat, double mass, wd_precision L, wd_precision H,
                         const WdMxReliable &v, const WdVec *p_restart, double *rr, double *ss);
// the same with no host wait: |rs|^2 and |s|^2 land in the device doubles
// rr_dev and ss_dev, for the caller to fetch (several systems per fetch).
// Its kernels go to ctx->stream.  scratch (device, optional): the
// reductions' work space of wd_red_doubles(wd_red_blocks(Vh), 1) doubles,
// owned by the caller -- needed when updates of several systems run on
// different streams at once; without it a block from the context's
// work-buffer cache (stream-ordered on ctx->stream) is used.
wd_status wd_mx_reliable_enqueue(wd_context *ctx, const wd_lattice *lat, double mass, wd_precision L, wd_precision H,
                                 const WdMxReliable &v, const WdVec *p_restart, double *rr_dev, double *ss_dev,
                                 double *scratch = nullptr);
// p (storage L) = rs (FP32) + beta p
wd_status wd_mx_xpay(wd_context *ctx, int Vh, wd_precision L, WdVec rs, double beta, WdVec p);

// Device-side scalars of one mixed-precision solve.  The iteration kernels
// read and write them, so iterations run back to back with no host wait: the
// hop that forms t = Mhat p also reduces |t|^2 and sets alpha, the hop that
// forms q = Mhat^dag t applies the CG update and reduces |r_s|^2, and the
// last block of that reduction decides on the device whether a reliable
// update is due (stop = 1) -- after which every later iteration kernel in the
// queue returns at once until the host has run the update and cleared stop.
struct WdMxDev {
    double rr;        // |r_s|^2 of the current iterate
    double rr_max;    // |r_s|^2 right after the last reliable update
    double target2;   // an update is due once |r_s|^2 <= target2 (squared normal-residual target)
    double delta2;    // ... or once |r_s|^2 < delta2 * rr_max
    double tt;        // |t|^2 = |Mhat p|^2 of the running iteration
    double rr_new;    // |r_s|^2 after the running iteration's update
    float alpha, beta;
    int stop;         // 0 iterate; 1 reliable update due; 2 non-finite scalar
    int iters;        // iterations completed on the device
};

// Device-side scalars of the FP64 / double-float CG solvers (wd_solver.cu):
// the reductions' last blocks set alpha and beta and close the stop gate, so
// iterations run back to back with no host wait.
struct WdCgDev {
    double rr;        // |r|^2 of the current iterate (the previous one once stop is set)
    double rr_new;    // |r|^2 after the running iteration's update
    double target2;   // stop once |r|^2 <= target2 (strict: < target2)
    double are, aim;  // alpha
    double beta;
    int strict;
    int stop;         // 0 iterate; 1 target reached; 2 non-finite |r|^2
    int iters;        // iterations completed
};

#ifdef __CUDACC__
// alpha = |r|^2 / d, d complex (src/invert.cpp:79-83); real d for the even-odd CG
__device__ __forceinline__ void wd_cg_set_alpha(WdCgDev *d, double re, double im, bool cplx)
{
    if (cplx) {
        const double n = re * re + im * im;
        d->are = (d->rr * re) / n;
        d->aim = (0.0 - d->rr * im) / n;
    } else {
        d->are = d->rr / re;
        d->aim = 0.0;
    }
}
// after the update of r: beta, or the stop gate
__device__ __forceinline__ void wd_cg_set_beta(WdCgDev *d, double rr_new)
{
    d->iters++;
    d->rr_new = rr_new;
    if (!isfinite(rr_new)) d->stop = 2;
    else if (d->strict ? rr_new < d->target2 : rr_new <= d->target2) d->stop = 1;
    else {
        d->beta = rr_new / d->rr;
        d->rr = rr_new;
    }
}
#endif

// One iteration's pieces on n complex entries of one storage (FP64 or
// double-float), all no-ops while dev->stop != 0 (wd_cg.cu).  red: for
// wd_red_blocks(Vh) blocks of two sums.
// alpha from |t|^2, or from the complex (p, q)
wd_status wd_cgd_norm(wd_context *ctx, WdVec t, int64_t n, WdCgDev *dev, WdRed red);
wd_status wd_cgd_dot(wd_context *ctx, WdVec p, WdVec q, int64_t n, WdCgDev *dev, WdRed red);
// x += alpha p, r -= alpha q, |r|^2 -> beta or the gate
wd_status wd_cgd_update(wd_context *ctx, bool cplx, WdVec p, WdVec q, WdVec x, WdVec r, int64_t n, WdCgDev *dev,
                        WdRed red);
// p = r + beta p
wd_status wd_cgd_xpby(wd_context *ctx, WdVec r, WdVec p, int64_t n, const WdCgDev *dev);

// The same fused into the fixed-point FP64 hops (wd_dslash_fix.cu).
//   t = -D_eo in / (4a) + a p on even blocks (a = 4 + mass), |t|^2 -> alpha
WdTried wd_hop_fix_norm(wd_context *ctx, const wd_lattice *lat, WdVec in, WdVec t, WdVec p, double mass, WdCgDev *dev,
                        WdRed red);
//   q = -D_eo^dag in / (4a) + a t, not stored: r -= alpha q, x += alpha p, |r|^2 -> beta or the gate
WdTried wd_hop_fix_update(wd_context *ctx, const wd_lattice *lat, WdVec in, WdVec t, WdVec p, WdVec r, WdVec x,
                          double mass, WdCgDev *dev, WdRed red);
//   |b - M x|^2 and |b|^2 -> result[0], result[1] (device)
WdTried wd_hop_fix_M_residual(wd_context *ctx, const wd_lattice *lat, const double2 *b, const double2 *x, double mass,
                              WdRed red, double *result);
//   q = M^dag in on the whole lattice, (p, q) -> alpha
WdTried wd_hop_fix_M_dot(wd_context *ctx, const wd_lattice *lat, WdVec in, WdVec q, WdVec p, double mass, WdCgDev *dev,
                         WdRed red);
