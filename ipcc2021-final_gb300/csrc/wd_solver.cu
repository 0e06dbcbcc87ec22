// wd_solver.cu -- conjugate-gradient solvers on resident fields.
//
// WD_SOLVER_CGNR_REF follows the reference CGinvert (src/invert.cpp:25-121)
// step for step: CG on M^dag M x = M^dag b over the whole lattice, complex
// alpha = (r,r)/(p,q), beta = (r,r)_new/(r,r)_old, stop on the absolute
// normal residual |r| < tol.  WD_SOLVER_CG_EO solves the same system through
// the even-odd Schur complement Mhat = a - D_eo D_oe/(4a) (a = 4+m), which
// needs half the hopping applications per iteration and converges in fewer
// iterations; it stops on the relative true residual |b - M x|/|b|.
//
// Both run in FP64 or in double-float (prec = WD_PREC_DF64: the same
// recurrences on float-pair vectors; on links that the fixed-point hop does
// not hold, where FP64 runs on GB300's narrow FP64 pipe, about 4x faster).
// Mixed precision (FP32 / FP16 inner) lives in wd_mixed.cu.
#include <chrono>
#include <cmath>
#include <limits>
#include "wd_fix_links.h"
#include "wd_kernels.h"
#include "wd_solver.h"

// ---------------------------------------------------------------- buffers
wd_status wd_vec_alloc(wd_context *ctx, WdVecBuf &b, wd_precision prec, int64_t n_complex)
{
    b.release();
    size_t bytes = (size_t)n_complex * wd_entry_bytes(prec);
    if (prec == WD_PREC_F16) bytes += (size_t)(n_complex / 12) * sizeof(float);
    wd_status st = wd_dev_alloc(ctx, &b.v.p, bytes);
    if (st != WD_OK) return st;
    b.ctx = ctx;
    b.v.prec = prec;
    b.v.scale = prec == WD_PREC_F16 ? (float *)((char *)b.v.p + (size_t)n_complex * wd_entry_bytes(prec)) : nullptr;
    return WD_OK;
}

void WdVecBuf::release()
{
    if (ctx) wd_dev_free(ctx, v.p);
    v = WdVec{};
    ctx = nullptr;
}

// half of a full-lattice vector (parity 0 or 1)
static inline WdVec par_half(WdVec v, int par, int Vh) { return wd_offset(v, (int64_t)par * 12 * Vh, (int64_t)par * Vh); }

// ---------------------------------------------------------------- operators
wd_status wd_apply_M_v(wd_context *ctx, const wd_lattice *lat, WdVec in, WdVec out, double mass, int dag,
                       const int *stop)
{
    if (in.prec == WD_PREC_F64)
        if (const WdTried r = wd_hop_fix_M(ctx, lat, (const double2 *)in.p, (double2 *)out.p, mass, dag, stop)) return *r;
    const int Vh = lat->g.Vh;
    for (int cb = 0; cb < 2; ++cb) {
        const WdVec x = par_half(in, cb, Vh);
        wd_status st = wd_hop_v(ctx, lat, par_half(in, 1 - cb, Vh), par_half(out, cb, Vh), &x, cb, dag, -0.5, 4.0 + mass,
                                stop);
        if (st != WD_OK) return st;
    }
    return WD_OK;
}

// Schur operator on even blocks: out = a v - D_eo D_oe v / (4a) (dag: with D^dag = Mhat^dag).
wd_status wd_apply_Mhat_v(wd_context *ctx, const wd_lattice *lat, WdVec v, WdVec out, WdVec tmp_o, double mass,
                          int dag)
{
    const double a = 4.0 + mass;
    wd_status st = wd_hop_v(ctx, lat, v, tmp_o, nullptr, 1, dag, 1.0, 0.0);
    if (st != WD_OK) return st;
    return wd_hop_v(ctx, lat, tmp_o, out, &v, 0, dag, -0.25 / a, a);
}

// |b - M x| / |b| recomputed in FP64 (full-lattice arrays): one launch that
// stores nothing on fixed-point links (48^3x96: 12 -> 5 ms of a solve's
// closing check), else M x, the difference and two norms.
wd_status wd_true_residual(wd_context *ctx, const wd_lattice *lat, const double2 *b, const double2 *x, double mass,
                           double *rel)
{
    const int64_t n = lat->volume * 12;
    double2 r[2];
    wd_status st;
    const int64_t rb = wd_red_blocks(lat->g.Vh);
    WdVecBuf buf;
    WdTried one;
    if (wd_fix_ensure(ctx, lat)) {  // (the allocation may give the links back)
        if ((st = wd_vec_alloc(ctx, buf, WD_PREC_F64, (int64_t)wd_red_doubles(rb, 2) / 2 + 1)) != WD_OK) return st;
        const WdRed red = wd_red_view(buf.v.p, rb);
        double2 *res = (double2 *)ctx->red_partial + WD_RED_BLOCKS;
        WD_CUDA(ctx, cudaMemsetAsync(red.counters, 0, wd_red_counters(rb) * sizeof(unsigned), ctx->stream));
        one = wd_hop_fix_M_residual(ctx, lat, b, x, mass, red, &res[0].x);
    }
    if (one) {
        if (*one != WD_OK) return *one;
        if ((st = wd_red_fetch(ctx, 1, r)) != WD_OK) return st;
        r[1].x = r[0].y;
    } else {
        WdVecBuf tmp;
        if ((st = wd_vec_alloc(ctx, tmp, WD_PREC_F64, n)) != WD_OK) return st;
        double2 *t = (double2 *)tmp.v.p;
        if ((st = wd_apply_M_v(ctx, lat, WdVec{(void *)x}, tmp.v, mass, 0)) != WD_OK) return st;
        if ((st = wd_blas_xpayz(ctx, b, make_double2(-1.0, 0.0), t, t, n)) != WD_OK) return st;
        if ((st = wd_red_norm2(ctx, t, n, 0)) != WD_OK) return st;
        if ((st = wd_red_norm2(ctx, b, n, 1)) != WD_OK) return st;
        if ((st = wd_red_fetch(ctx, 2, r)) != WD_OK) return st;
    }
    *rel = r[1].x > 0 ? std::sqrt(r[0].x / r[1].x) : std::sqrt(r[0].x);
    return WD_OK;
}

namespace {

// CG iterations on device scalars, queued ahead of the host.  The host
// enqueues a few iterations, asks for a copy of the scalars, and looks at the
// copy before last while the device works on; iterations queued past the one
// that closed the gate are no-ops.
struct CgLoop {
    wd_context *ctx;
    WdCgDev *dev = nullptr;  // device
    WdCgDev *host;           // three pinned copies: two in flight, one for uploads
    WdRed red;
    void *blk = nullptr;
    int chunk = 1;           // iterations per look

    CgLoop(wd_context *c) : ctx(c), host((WdCgDev *)c->state_host) {}
    ~CgLoop() { wd_dev_free(ctx, blk); }
    wd_status alloc(int Vh)
    {
        chunk = Vh <= 32768 ? 4 : Vh <= 524288 ? 2 : 1;
        const int64_t rb = wd_red_blocks(Vh);
        wd_status st = wd_dev_alloc(ctx, &blk, 256 + wd_red_doubles(rb, 2) * sizeof(double));
        if (st != WD_OK) return st;
        dev = (WdCgDev *)blk;
        red = wd_red_view((char *)blk + 256, rb);
        WD_CUDA(ctx, cudaMemsetAsync(red.counters, 0, wd_red_counters(rb) * sizeof(unsigned), ctx->stream));
        return WD_OK;
    }
    wd_status start(double rr, double target, bool strict, int iters)
    {
        static_assert(sizeof(WdCgDev) <= 256 && 3 * sizeof(WdCgDev) <= WD_STATE_HOST_BYTES, "device scalars");
        host[2] = WdCgDev{};
        host[2].rr = rr;
        // (a square that underflows is still met by a residual of zero)
        host[2].target2 = std::fmax(target * target, std::numeric_limits<double>::denorm_min());
        host[2].strict = strict;
        host[2].iters = iters;
        WD_CUDA(ctx, cudaMemcpyAsync(dev, &host[2], sizeof(WdCgDev), cudaMemcpyHostToDevice, ctx->stream));
        return WD_OK;
    }
    // up to `left` iterations; on return every queued one is done and *end holds the scalars
    template <class Iteration>
    wd_status run(int left, Iteration iteration, WdCgDev *end)
    {
        int looks = 0, seen = 0;  // copies asked for, and looked at
        bool stop = false;
        wd_status st = WD_OK;
        while (!stop && left > 0 && st == WD_OK) {
            const int k = chunk < left ? chunk : left;
            for (int i = 0; i < k && st == WD_OK; ++i) st = iteration();
            if (st != WD_OK) break;
            left -= k;
            WD_CUDA(ctx, cudaMemcpyAsync(&host[looks & 1], dev, sizeof(WdCgDev), cudaMemcpyDeviceToHost, ctx->stream));
            WD_CUDA(ctx, cudaEventRecord(ctx->chunk_done[looks & 1], ctx->stream));
            ++looks;
            if (looks - seen == 2) {
                WD_CUDA(ctx, cudaEventSynchronize(ctx->chunk_done[seen & 1]));
                stop = host[seen & 1].stop != 0;
                ++seen;
            }
        }
        WD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (st == WD_OK && looks > 0) *end = host[(looks - 1) & 1];
        return st;
    }
};

wd_status fetch1(wd_context *ctx, double2 *v) { return wd_red_fetch(ctx, 1, v); }

}  // namespace

// ------------------------------------------------------- reference CGNR
// src/invert.cpp:25-121 on full-lattice vectors of one storage (FP64 or df).
static wd_status cgnr_ref_core(wd_context *ctx, const wd_lattice *lat, WdVec src, WdVec x,
                               const wd_solver_params *prm, wd_solver_stats *stats)
{
    const int64_t n = lat->volume * 12;
    const double m = prm->mass;
    const bool f64 = src.prec == WD_PREC_F64;
    WdVecBuf b[5];
    for (auto &v : b) {
        wd_status s = wd_vec_alloc(ctx, v, src.prec, n);
        if (s != WD_OK) return s;
    }
    WdVec r0 = b[0].v, q = b[1].v, qq = b[2].v, p = b[3].v, Mdb = b[4].v;
    CgLoop loop(ctx);
    wd_status st = loop.alloc(lat->g.Vh);
    if (st != WD_OK) return st;
    WdCgDev *dev = loop.dev;
    // Mdb = M^dag src; r0 = Mdb - M^dag M x   (src/invert.cpp:41-58)
    if ((st = wd_apply_M_v(ctx, lat, src, Mdb, m, 1)) != WD_OK) return st;
    if ((st = wd_apply_M_v(ctx, lat, x, qq, m, 0)) != WD_OK) return st;
    if ((st = wd_apply_M_v(ctx, lat, qq, r0, m, 1)) != WD_OK) return st;
    if ((st = wd_v_xpayz(ctx, Mdb, make_double2(-1.0, 0.0), r0, r0, n)) != WD_OK) return st;
    if ((st = wd_v_norm2(ctx, r0, n, 0)) != WD_OK) return st;
    double2 red;
    if ((st = fetch1(ctx, &red)) != WD_OK) return st;
    if ((st = wd_v_copy(ctx, p, r0, n)) != WD_OK) return st;
    if ((st = loop.start(red.x, prm->tol, true, 0)) != WD_OK) return st;
    // qq = M p, q = M^dag qq, alpha = (r,r) / (p,q); dest += alpha p; r0 -= alpha q; |r0|^2
    // (src/invert.cpp:77-107); beta = (r,r)_new / (r,r), p = r + beta p (:67-76)
    auto iteration = [&]() -> wd_status {
        wd_status e;
        if ((e = wd_apply_M_v(ctx, lat, p, qq, m, 0, &dev->stop)) != WD_OK) return e;
        WdTried fused;
        if (f64) fused = wd_hop_fix_M_dot(ctx, lat, qq, q, p, m, dev, loop.red);
        if (fused) {
            if (*fused != WD_OK) return *fused;
        } else {
            if ((e = wd_apply_M_v(ctx, lat, qq, q, m, 1, &dev->stop)) != WD_OK) return e;
            if ((e = wd_cgd_dot(ctx, p, q, n, dev, loop.red)) != WD_OK) return e;
        }
        if ((e = wd_cgd_update(ctx, true, p, q, x, r0, n, dev, loop.red)) != WD_OK) return e;
        return wd_cgd_xpby(ctx, r0, p, n, dev);
    };
    WdCgDev end{};
    end.rr = end.rr_new = red.x;
    if ((st = loop.run(prm->max_iter - 1, iteration, &end)) != WD_OK) return st;
    stats->iterations = end.iters;
    if (end.stop == 2) return wd_fail(ctx, WD_ERR_NAN, "CG residual is not finite");
    stats->residual = std::sqrt(end.rr_new);
    stats->converged = end.stop == 1;
    return WD_OK;
}

// ----------------------------------------------------- even-odd Schur CG
static wd_status cg_eo_core(wd_context *ctx, const wd_lattice *lat, WdVec src, WdVec x, const wd_solver_params *prm,
                            wd_solver_stats *stats)
{
    const int Vh = lat->g.Vh;
    const int64_t nh = (int64_t)12 * Vh;
    const double m = prm->mass, a = 4.0 + m;
    const bool f64 = src.prec == WD_PREC_F64;
    WdVecBuf b[7];
    for (auto &v : b) {
        wd_status s = wd_vec_alloc(ctx, v, src.prec, nh);
        if (s != WD_OK) return s;
    }
    WdVec bhat = b[0].v, r = b[1].v, p = b[2].v, t = b[3].v, q = b[4].v, tmp_o = b[5].v, s_e = b[6].v;
    const WdVec b_e = par_half(src, 0, Vh), b_o = par_half(src, 1, Vh);
    WdVec x_e = par_half(x, 0, Vh), x_o = par_half(x, 1, Vh);
    CgLoop loop(ctx);
    wd_status st = loop.alloc(Vh);
    if (st != WD_OK) return st;
    WdCgDev *dev = loop.dev;

    // bhat_e = b_e + D_eo b_o / (2a)
    if ((st = wd_hop_v(ctx, lat, b_o, bhat, &b_e, 0, 0, 0.5 / a, 1.0)) != WD_OK) return st;
    if (!prm->use_initial_guess && (st = wd_v_zero(ctx, x_e, nh)) != WD_OK) return st;
    double2 red[2];
    if ((st = wd_v_norm2(ctx, src, 2 * nh, 1)) != WD_OK) return st;
    if ((st = wd_red_fetch(ctx, 2, red)) != WD_OK) return st;
    const double norm_b = std::sqrt(red[1].x) > 0 ? std::sqrt(red[1].x) : 1.0;

    // s = bhat - Mhat x (its norm is the full-system true residual |b - M x|
    // once x_o = (b_o + D_oe x_e / 2)/a), r = Mhat^dag s
    double ss = 0.0;
    auto residuals = [&](double *rr, bool x_zero) -> wd_status {
        wd_status e;
        const WdVec s = x_zero ? bhat : s_e;
        if (!x_zero) {
            if ((e = wd_apply_Mhat_v(ctx, lat, x_e, t, tmp_o, m, 0)) != WD_OK) return e;
            if ((e = wd_v_xpayz(ctx, bhat, make_double2(-1.0, 0.0), t, s, nh)) != WD_OK) return e;
        }
        if ((e = wd_apply_Mhat_v(ctx, lat, s, r, tmp_o, m, 1)) != WD_OK) return e;
        if ((e = wd_v_norm2(ctx, r, nh, 0)) != WD_OK) return e;
        if ((e = wd_v_norm2(ctx, s, nh, 1)) != WD_OK) return e;
        double2 v[2];
        if ((e = wd_red_fetch(ctx, 2, v)) != WD_OK) return e;
        *rr = v[0].x;
        ss = v[1].x;
        return WD_OK;
    };
    // t = Mhat p, alpha = rr / |t|^2, q = Mhat^dag t, the update with |r|^2, p = r + beta p
    auto iteration = [&]() -> wd_status {
        wd_status e;
        if ((e = wd_hop_v(ctx, lat, p, tmp_o, nullptr, 1, 0, 1.0, 0.0, &dev->stop)) != WD_OK) return e;
        WdTried fused;
        if (f64) fused = wd_hop_fix_norm(ctx, lat, tmp_o, t, p, m, dev, loop.red);
        if (fused) {
            if (*fused != WD_OK) return *fused;
        } else {
            if ((e = wd_hop_v(ctx, lat, tmp_o, t, &p, 0, 0, -0.25 / a, a, &dev->stop)) != WD_OK) return e;
            if ((e = wd_cgd_norm(ctx, t, nh, dev, loop.red)) != WD_OK) return e;
        }
        if ((e = wd_hop_v(ctx, lat, t, tmp_o, nullptr, 1, 1, 1.0, 0.0, &dev->stop)) != WD_OK) return e;
        fused.reset();
        if (f64) fused = wd_hop_fix_update(ctx, lat, tmp_o, t, p, r, x_e, m, dev, loop.red);
        if (fused) {
            if (*fused != WD_OK) return *fused;
        } else {
            if ((e = wd_hop_v(ctx, lat, tmp_o, q, &t, 0, 1, -0.25 / a, a, &dev->stop)) != WD_OK) return e;
            if ((e = wd_cgd_update(ctx, false, p, q, x_e, r, nh, dev, loop.red)) != WD_OK) return e;
        }
        return wd_cgd_xpby(ctx, r, p, nh, dev);
    };

    double rr;
    if ((st = residuals(&rr, !prm->use_initial_guess)) != WD_OK) return st;
    if ((st = wd_v_copy(ctx, p, r, nh)) != WD_OK) return st;
    // normal-residual target from the observed ratio |r| / |s|
    double ratio = ss > 0 ? std::sqrt(rr / ss) : 1.0;
    double target = prm->tol * norm_b * ratio * 0.5;
    double true_res = std::sqrt(ss) / norm_b;
    int iters = 0;
    bool converged = true_res <= prm->tol;
    while (!converged && iters < prm->max_iter) {
        WdCgDev end{};
        if ((st = loop.start(rr, target, false, iters)) != WD_OK) return st;
        if ((st = loop.run(prm->max_iter - iters, iteration, &end)) != WD_OK) return st;
        iters = end.iters;
        if (end.stop == 2) {
            stats->iterations = iters;
            return wd_fail(ctx, WD_ERR_NAN, "CG residual is not finite");
        }
        if (end.stop != 1) break;  // out of iterations
        // check the true residual; replace r by the recomputed one
        double rr_new;
        if ((st = residuals(&rr_new, false)) != WD_OK) return st;
        stats->reliable_updates++;
        true_res = std::sqrt(ss) / norm_b;
        if (true_res <= prm->tol) {
            converged = true;
            break;
        }
        ratio = ss > 0 ? std::sqrt(rr_new / ss) : ratio;
        target = std::fmin(target * 0.5, prm->tol * norm_b * ratio * 0.5);
        if ((st = wd_v_xpby(ctx, r, rr_new / end.rr, p, nh)) != WD_OK) return st;
        rr = rr_new;
    }
    // x_o = (b_o + D_oe x_e / 2) / a
    if ((st = wd_hop_v(ctx, lat, x_e, x_o, &b_o, 1, 0, 0.5 / a, 1.0 / a)) != WD_OK) return st;
    stats->iterations = iters;
    stats->residual = true_res;
    stats->converged = converged;
    return WD_OK;
}

// Runs a solver core in the requested arithmetic on FP64 fields.
template <class Core>
static wd_status run_in(wd_context *ctx, const wd_lattice *lat, const double2 *src, double2 *x, wd_precision prec,
                        Core core)
{
    WdVec vs{(void *)src}, vx{(void *)x};
    if (prec == WD_PREC_F64) return core(vs, vx);
    const int64_t n = lat->volume * 12;
    WdVecBuf ds, dx;
    wd_status st = wd_vec_alloc(ctx, ds, WD_PREC_DF64, n);
    if (st == WD_OK) st = wd_vec_alloc(ctx, dx, WD_PREC_DF64, n);
    if (st == WD_OK) st = wd_convert_f64_to_df(ctx, src, (float4 *)ds.v.p, n);
    if (st == WD_OK) st = wd_convert_f64_to_df(ctx, x, (float4 *)dx.v.p, n);
    if (st == WD_OK) st = core(ds.v, dx.v);
    if (st == WD_OK) st = wd_convert_df_to_f64(ctx, (const float4 *)dx.v.p, x, n);
    return st;
}

extern "C" void wd_solver_params_default(wd_solver_params *p)
{
    if (!p) return;
    p->kind = WD_SOLVER_CG_EO;
    p->mass = 0.1;
    p->tol = 1e-10;
    p->max_iter = 1000;
    p->prec = WD_PREC_F64;
    p->delta = 0.1;
    p->use_initial_guess = 0;
    p->prec_reliable = WD_PREC_F64;
}

extern "C" wd_status wd_solve(wd_context *ctx, const wd_lattice *lat, const wd_field *src, wd_field *dest,
                              const wd_solver_params *params, wd_solver_stats *stats)
{
    if (!ctx || !lat || !src || !dest || !params) return wd_fail(ctx, WD_ERR_BAD_ARG, "null argument");
    if (src == dest) return wd_fail(ctx, WD_ERR_BAD_ARG, "source and solution must be different fields");
    if (src->lat->volume != lat->volume || dest->lat->volume != lat->volume)
        return wd_fail(ctx, WD_ERR_BAD_ARG, "field does not belong to this lattice size");
    if (src->storage != WD_PREC_F64 || dest->storage != WD_PREC_F64)
        return wd_fail(ctx, WD_ERR_BAD_ARG, "solver fields must be FP64 (prec selects the arithmetic)");
    if (params->max_iter < 1 || !(params->tol > 0)) return wd_fail(ctx, WD_ERR_BAD_ARG, "bad tolerance or max_iter");
    if (params->prec < WD_PREC_F64 || params->prec > WD_PREC_F16)
        return wd_fail(ctx, WD_ERR_BAD_ARG, "unknown precision");
    wd_solver_stats local;
    if (!stats) stats = &local;
    *stats = wd_solver_stats{};
    wd_memory_freed();  // a program may have freed memory of its own since the links were last refused theirs
    const auto t0 = std::chrono::steady_clock::now();
    wd_status st;
    const bool mixed = params->prec == WD_PREC_F32 || params->prec == WD_PREC_F16;
    switch (params->kind) {
    case WD_SOLVER_CGNR_REF:
        if (mixed) return wd_fail(ctx, WD_ERR_BAD_ARG, "the reference CG runs in FP64 or double-float only");
        st = run_in(ctx, lat, src->d, dest->d, params->prec,
                    [&](WdVec s, WdVec x) { return cgnr_ref_core(ctx, lat, s, x, params, stats); });
        break;
    case WD_SOLVER_CG_EO:
        if (mixed)
            st = wd_solve_cg_eo_mixed(ctx, lat, src->d, dest->d, params, stats);
        else
            st = run_in(ctx, lat, src->d, dest->d, params->prec,
                        [&](WdVec s, WdVec x) { return cg_eo_core(ctx, lat, s, x, params, stats); });
        break;
    default: return wd_fail(ctx, WD_ERR_BAD_ARG, "unknown solver kind");
    }
    if (st != WD_OK) return st;
    WD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    stats->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    // the FP64 true residual |b - M x|/|b| of whatever the solver returned
    // (a check of the result, after the timed solve)
    st = wd_true_residual(ctx, lat, src->d, dest->d, params->mass, &stats->true_residual);
    if (st != WD_OK) return st;
    return stats->converged ? WD_OK : WD_ERR_NOT_CONVERGED;
}

extern "C" wd_status wd_check(wd_context *ctx, const wd_lattice *lat, const wd_field *b, const wd_field *x,
                              double mass, double out[12])
{
    if (!ctx || !lat || !b || !x || !out) return wd_fail(ctx, WD_ERR_BAD_ARG, "null argument");
    if (b->storage != WD_PREC_F64 || x->storage != WD_PREC_F64)
        return wd_fail(ctx, WD_ERR_BAD_ARG, "check needs FP64 fields");
    const int64_t n = lat->volume * 12;
    WdVecBuf bufs[6];
    for (auto &v : bufs) {
        wd_status s = wd_vec_alloc(ctx, v, WD_PREC_F64, n);
        if (s != WD_OK) return s;
    }
    const WdVec vb = wd_whole(b), vx = wd_whole(x);
    const WdVec Mb = bufs[0].v, Mdb = bufs[1].v, MMb = bufs[2].v, Mx = bufs[3].v, MMx = bufs[4].v, tmp = bufs[5].v;
    auto d2 = [](WdVec v) { return (double2 *)v.p; };
    wd_status st;
    // the sequence of src/check.cpp:37-60
    if ((st = wd_apply_M_v(ctx, lat, vb, Mb, mass, 0)) != WD_OK) return st;
    if ((st = wd_apply_M_v(ctx, lat, vb, Mdb, mass, 1)) != WD_OK) return st;
    if ((st = wd_apply_M_v(ctx, lat, Mb, MMb, mass, 1)) != WD_OK) return st;
    if ((st = wd_apply_M_v(ctx, lat, vx, Mx, mass, 0)) != WD_OK) return st;
    if ((st = wd_apply_M_v(ctx, lat, Mx, MMx, mass, 1)) != WD_OK) return st;
    if ((st = wd_red_norm2(ctx, b->d, n, 0)) != WD_OK) return st;
    if ((st = wd_red_norm2(ctx, x->d, n, 1)) != WD_OK) return st;
    if ((st = wd_red_dot(ctx, d2(Mb), d2(Mb), n, 2)) != WD_OK) return st;
    if ((st = wd_red_dot(ctx, b->d, d2(MMb), n, 3)) != WD_OK) return st;
    if ((st = wd_red_dot(ctx, d2(Mx), d2(Mx), n, 4)) != WD_OK) return st;
    if ((st = wd_red_dot(ctx, x->d, d2(MMx), n, 5)) != WD_OK) return st;
    if ((st = wd_blas_xpayz(ctx, d2(Mx), make_double2(-1.0, 0.0), b->d, d2(tmp), n)) != WD_OK) return st;
    if ((st = wd_red_norm2(ctx, d2(tmp), n, 6)) != WD_OK) return st;
    if ((st = wd_blas_xpayz(ctx, d2(MMx), make_double2(-1.0, 0.0), d2(Mdb), d2(tmp), n)) != WD_OK) return st;
    if ((st = wd_red_norm2(ctx, d2(tmp), n, 7)) != WD_OK) return st;
    double2 r[8];
    if ((st = wd_red_fetch(ctx, 8, r)) != WD_OK) return st;
    out[0] = std::sqrt(r[0].x);
    out[1] = std::sqrt(r[1].x);
    out[2] = r[2].x, out[3] = r[2].y;
    out[4] = r[3].x, out[5] = r[3].y;
    out[6] = r[4].x, out[7] = r[4].y;
    out[8] = r[5].x, out[9] = r[5].y;
    out[10] = std::sqrt(r[6].x);
    out[11] = std::sqrt(r[7].x);
    return WD_OK;
}
