// wd_blas.cu -- layout conversion and BLAS-1 with deterministic reductions.
//
// Reductions (norm_2 / vector_p of include/operator_mpi.h:15-79) use a fixed
// grid of WD_RED_BLOCKS blocks: each block folds its grid-stride share with
// warp shuffles into one FP64 partial, and a single-block pass adds the
// partials in a fixed tree order.  The result is bitwise reproducible for a
// given length and lands in a device slot, so solvers can keep it on the
// device.  Double-float vectors accumulate per thread in double-float on the
// FP32 pipe and convert to FP64 once per thread.
#include "wd_kernels.h"
#include "wd_df.cuh"
#include "wd_reduce.cuh"

namespace {

constexpr int kTile = 64;  // sites per transpose tile

// ------------------------------------------------ storage converters
struct StF64 {
    __device__ static void store(void *out, int c, int s, int Vh, double2 v) { ((double2 *)out)[(size_t)c * Vh + s] = v; }
    __device__ static double2 load(const void *in, int c, int s, int Vh) { return ((const double2 *)in)[(size_t)c * Vh + s]; }
};
struct StDF {
    __device__ static void store(void *out, int c, int s, int Vh, double2 v) { ((float4 *)out)[(size_t)c * Vh + s] = df_pack(v); }
    __device__ static double2 load(const void *in, int c, int s, int Vh) { return df_unpack(((const float4 *)in)[(size_t)c * Vh + s]); }
};
// FP32: components in pairs, plane j = comps (2j, 2j+1) as float4 {re0, im0, re1, im1}
struct StF32 {
    __device__ static void store(void *out, int c, int s, int Vh, double2 v)
    {
        ((float2 *)out)[((size_t)(c >> 1) * Vh + s) * 2 + (c & 1)] = make_float2((float)v.x, (float)v.y);
    }
    __device__ static double2 load(const void *in, int c, int s, int Vh)
    {
        const float2 f = ((const float2 *)in)[((size_t)(c >> 1) * Vh + s) * 2 + (c & 1)];
        return make_double2(f.x, f.y);
    }
};

template <int NC, class St>
__global__ void __launch_bounds__(256) k_aos_to_soa(const double2 *__restrict__ aos, void *__restrict__ soa,
                                                    int Vh, size_t block_bytes)
{
    __shared__ double2 tile[kTile * NC];
    const int b = blockIdx.y;
    const int s0 = blockIdx.x * kTile;
    const int ns = min(kTile, Vh - s0);
    const double2 *src = aos + ((size_t)b * Vh + s0) * NC;
    void *dst = (char *)soa + b * block_bytes;
    for (int i = threadIdx.x; i < ns * NC; i += blockDim.x) tile[i] = src[i];
    __syncthreads();
    for (int i = threadIdx.x; i < ns * NC; i += blockDim.x) {
        const int c = i / ns, s = i - c * ns;
        St::store(dst, c, s0 + s, Vh, tile[s * NC + c]);
    }
}

template <int NC, class St>
__global__ void __launch_bounds__(256) k_soa_to_aos(const void *__restrict__ soa, double2 *__restrict__ aos,
                                                    int Vh, size_t block_bytes)
{
    __shared__ double2 tile[kTile * NC];
    const int b = blockIdx.y;
    const int s0 = blockIdx.x * kTile;
    const int ns = min(kTile, Vh - s0);
    const void *src = (const char *)soa + b * block_bytes;
    for (int i = threadIdx.x; i < ns * NC; i += blockDim.x) {
        const int c = i / ns, s = i - c * ns;
        tile[s * NC + c] = St::load(src, c, s0 + s, Vh);
    }
    __syncthreads();
    double2 *dst = aos + ((size_t)b * Vh + s0) * NC;
    for (int i = threadIdx.x; i < ns * NC; i += blockDim.x) dst[i] = tile[i];
}

// ------------------------------------------------------- reductions
#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

__global__ void __launch_bounds__(WD_RED_THREADS) k_norm2(const double2 *__restrict__ a, int64_t n, double2 *partial)
{
    double s = 0.0;
    GRID_STRIDE(i, n)
    {
        const double2 v = a[i];
        s = fma(v.x, v.x, s);
        s = fma(v.y, v.y, s);
    }
    wd_block_partial(s, partial);
}

__global__ void __launch_bounds__(WD_RED_THREADS) k_dot(const double2 *__restrict__ a, const double2 *__restrict__ b,
                                                        int64_t n, double2 *partial)
{
    double re = 0.0, im = 0.0;
    GRID_STRIDE(i, n)
    {
        const double2 u = a[i], v = b[i];
        re = fma(u.x, v.x, re);
        re = fma(u.y, v.y, re);
        im = fma(u.x, v.y, im);
        im = fma(-u.y, v.x, im);
    }
    wd_block_partial(re, im, partial);
}

__global__ void __launch_bounds__(WD_RED_THREADS) k_norm2_df(const float4 *__restrict__ a, int64_t n, double2 *partial)
{
    dfr s{0.f, 0.f};
    GRID_STRIDE(i, n)
    {
        const dfc v = df_from_f4(a[i]);
        s = df_madd(df_madd(s, v.re, v.re), v.im, v.im);
    }
    wd_block_partial(df_value(s), partial);
}

__global__ void __launch_bounds__(WD_RED_THREADS) k_dot_df(const float4 *__restrict__ a, const float4 *__restrict__ b,
                                                           int64_t n, double2 *partial)
{
    dfc s = c_zero(dfc());
    GRID_STRIDE(i, n) { s = c_maddc(s, df_from_f4(a[i]), df_from_f4(b[i])); }
    wd_block_partial(df_value(s.re), df_value(s.im), partial);
}

// One block of 1024 threads folds WD_RED_BLOCKS partials into *result.
__global__ void __launch_bounds__(1024) k_red_finish(const double2 *__restrict__ partial, int nparts, double2 *result)
{
    __shared__ double sa[32], sb[32];
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        a += partial[i].x;
        b += partial[i].y;
    }
    a = wd_warp_sum(a);
    b = wd_warp_sum(b);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) {
        sa[w] = a;
        sb[w] = b;
    }
    __syncthreads();
    if (w == 0) {
        a = l < (int)(blockDim.x >> 5) ? sa[l] : 0.0;
        b = l < (int)(blockDim.x >> 5) ? sb[l] : 0.0;
        a = wd_warp_sum(a);
        b = wd_warp_sum(b);
        if (l == 0) *result = make_double2(a, b);
    }
}

// ------------------------------------------------------------ FP64 BLAS
__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}

__global__ void k_axpby(double2 a, const double2 *__restrict__ x, double2 b, double2 *__restrict__ y, int64_t n)
{
    GRID_STRIDE(i, n)
    {
        const double2 u = cmul(a, x[i]), v = cmul(b, y[i]);
        y[i] = make_double2(u.x + v.x, u.y + v.y);
    }
}

// z may alias y (element-wise read before write)
__global__ void k_xpayz(const double2 *__restrict__ x, double2 a, const double2 *y, double2 *z, int64_t n)
{
    GRID_STRIDE(i, n)
    {
        const double2 u = x[i], v = y[i];
        z[i] = make_double2(u.x + fma(a.x, v.x, -a.y * v.y), u.y + fma(a.x, v.y, a.y * v.x));
    }
}

__global__ void k_scale(double a, const double2 *__restrict__ x, double2 *__restrict__ y, int64_t n)
{
    GRID_STRIDE(i, n)
    {
        const double2 u = x[i];
        y[i] = make_double2(a * u.x, a * u.y);
    }
}

// x /= |x| with the sum |x|^2 on the device, where it was just left; one
// thread's square root and quotient a block (FP64 pipe)
__global__ void k_unit(double2 *__restrict__ x, int64_t n, const double2 *norm2)
{
    __shared__ double f;
    if (threadIdx.x == 0) f = norm2->x > 0 ? 1.0 / sqrt(norm2->x) : 1.0;
    __syncthreads();
    const double a = f;
    GRID_STRIDE(i, n)
    {
        const double2 u = x[i];
        x[i] = make_double2(a * u.x, a * u.y);
    }
}

// y = x + b y, b real
__global__ void k_xpby_real(const double2 *__restrict__ x, double b, double2 *__restrict__ y, int64_t n)
{
    GRID_STRIDE(i, n)
    {
        const double2 u = x[i], v = y[i];
        y[i] = make_double2(fma(b, v.x, u.x), fma(b, v.y, u.y));
    }
}

// ----------------------------------------------------- double-float BLAS
__host__ __device__ __forceinline__ dfc dfc_split(double2 a) { return dfc{df_split(a.x), df_split(a.y)}; }

__global__ void k_axpby_df(dfc a, const float4 *__restrict__ x, dfc b, float4 *__restrict__ y, int64_t n)
{
    GRID_STRIDE(i, n) { y[i] = df_to_f4(c_madd(c_mul(a, df_from_f4(x[i])), b, df_from_f4(y[i]))); }
}

__global__ void k_xpayz_df(const float4 *__restrict__ x, dfc a, const float4 *y, float4 *z, int64_t n)
{
    GRID_STRIDE(i, n) { z[i] = df_to_f4(c_madd(df_from_f4(x[i]), a, df_from_f4(y[i]))); }
}

__global__ void k_xpby_real_df(const float4 *__restrict__ x, dfr b, float4 *__restrict__ y, int64_t n)
{
    GRID_STRIDE(i, n)
    {
        const dfc u = df_from_f4(x[i]), v = df_from_f4(y[i]);
        y[i] = df_to_f4(dfc{df_madd(u.re, b, v.re), df_madd(u.im, b, v.im)});
    }
}

inline int blas_blocks(int64_t n)
{
    int64_t b = (n + 255) / 256;
    return (int)(b < 152 * 16 ? (b < 1 ? 1 : b) : 152 * 16);
}

}  // namespace

// ------------------------------------------------------------- layout
template <int NC>
static wd_status to_soa(wd_context *ctx, const WdGeom &g, const double2 *ref, void *soa, wd_precision prec)
{
    dim3 grid((g.Vh + kTile - 1) / kTile, 2);
    const size_t bb = (size_t)NC * g.Vh * wd_entry_bytes(prec);
    switch (prec) {
    case WD_PREC_F64: k_aos_to_soa<NC, StF64><<<grid, 256, 0, ctx->stream>>>(ref, soa, g.Vh, bb); break;
    case WD_PREC_DF64: k_aos_to_soa<NC, StDF><<<grid, 256, 0, ctx->stream>>>(ref, soa, g.Vh, bb); break;
    case WD_PREC_F32: k_aos_to_soa<NC, StF32><<<grid, 256, 0, ctx->stream>>>(ref, soa, g.Vh, bb); break;
    default: return wd_fail(ctx, WD_ERR_BAD_ARG, "no direct layout conversion for this storage");
    }
    WD_LAUNCHED(ctx);
    return WD_OK;
}

wd_status wd_spinor_ref_to_soa(wd_context *ctx, const WdGeom &g, const double2 *ref, WdVec soa)
{
    return to_soa<12>(ctx, g, ref, soa.p, soa.prec);
}

wd_status wd_spinor_soa_to_ref(wd_context *ctx, const WdGeom &g, WdVec soa, double2 *ref)
{
    dim3 grid((g.Vh + kTile - 1) / kTile, 2);
    const size_t bb = (size_t)12 * g.Vh * wd_entry_bytes(soa.prec);
    switch (soa.prec) {
    case WD_PREC_F64: k_soa_to_aos<12, StF64><<<grid, 256, 0, ctx->stream>>>(soa.p, ref, g.Vh, bb); break;
    case WD_PREC_DF64: k_soa_to_aos<12, StDF><<<grid, 256, 0, ctx->stream>>>(soa.p, ref, g.Vh, bb); break;
    case WD_PREC_F32: k_soa_to_aos<12, StF32><<<grid, 256, 0, ctx->stream>>>(soa.p, ref, g.Vh, bb); break;
    default: return wd_fail(ctx, WD_ERR_BAD_ARG, "no direct layout conversion for this storage");
    }
    WD_LAUNCHED(ctx);
    return WD_OK;
}

wd_status wd_gauge_ref_to_soa(wd_context *ctx, const WdGeom &g, int mu, const double2 *ref, double2 *soa)
{
    return to_soa<9>(ctx, g, ref, soa + (size_t)mu * 2 * 9 * g.Vh, WD_PREC_F64);
}

// n 16-byte entries from src to dst on `stream`, either side possibly host
// memory the device addresses directly.  76 blocks (half the SMs) keep the
// CPU-GPU link busy and leave the SMs to the concurrent arithmetic: the
// pageable host-buffer DslashoffdNew at 32^3x64 ran 2.72-2.80 ms per call
// with 19-114 blocks and 3.1-3.2 ms with 304-1216.
__global__ void k_copy16(const double2 *__restrict__ src, double2 *__restrict__ dst, int64_t n)
{
    GRID_STRIDE(i, n) { dst[i] = src[i]; }
}

wd_status wd_copy_kernel(wd_context *ctx, cudaStream_t stream, const double2 *src, double2 *dst, int64_t n)
{
    if (n <= 0) return WD_OK;
    const int64_t b = (n + 255) / 256;
    k_copy16<<<(int)(b < 76 ? b : 76), 256, 0, stream>>>(src, dst, n);
    WD_LAUNCHED(ctx);
    return WD_OK;
}

// ---------------------------------------------------------- reductions
wd_status wd_red_finish(wd_context *ctx, int slot)
{
    double2 *part = (double2 *)ctx->red_partial;
    k_red_finish<<<1, 1024, 0, ctx->stream>>>(part, WD_RED_BLOCKS, part + WD_RED_BLOCKS + slot);
    WD_LAUNCHED(ctx);
    return WD_OK;
}

wd_status wd_red_norm2(wd_context *ctx, const double2 *a, int64_t n, int slot)
{
    k_norm2<<<WD_RED_BLOCKS, WD_RED_THREADS, 0, ctx->stream>>>(a, n, (double2 *)ctx->red_partial);
    WD_LAUNCHED(ctx);
    return wd_red_finish(ctx, slot);
}

wd_status wd_red_dot(wd_context *ctx, const double2 *a, const double2 *b, int64_t n, int slot)
{
    k_dot<<<WD_RED_BLOCKS, WD_RED_THREADS, 0, ctx->stream>>>(a, b, n, (double2 *)ctx->red_partial);
    WD_LAUNCHED(ctx);
    return wd_red_finish(ctx, slot);
}

wd_status wd_red_fetch(wd_context *ctx, int nslots, double2 *host)
{
    double2 *part = (double2 *)ctx->red_partial;
    WD_CUDA(ctx, cudaMemcpyAsync(ctx->red_result, part + WD_RED_BLOCKS, sizeof(double2) * nslots,
                                 cudaMemcpyDeviceToHost, ctx->stream));
    WD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    memcpy(host, ctx->red_result, sizeof(double2) * nslots);
    return WD_OK;
}

wd_status wd_blas_axpby(wd_context *ctx, double2 a, const double2 *x, double2 b, double2 *y, int64_t n)
{
    k_axpby<<<blas_blocks(n), 256, 0, ctx->stream>>>(a, x, b, y, n);
    WD_LAUNCHED(ctx);
    return WD_OK;
}

wd_status wd_blas_xpayz(wd_context *ctx, const double2 *x, double2 a, const double2 *y, double2 *z, int64_t n)
{
    k_xpayz<<<blas_blocks(n), 256, 0, ctx->stream>>>(x, a, y, z, n);
    WD_LAUNCHED(ctx);
    return WD_OK;
}

wd_status wd_blas_scale(wd_context *ctx, double a, const double2 *x, double2 *y, int64_t n)
{
    k_scale<<<blas_blocks(n), 256, 0, ctx->stream>>>(a, x, y, n);
    WD_LAUNCHED(ctx);
    return WD_OK;
}

wd_status wd_blas_unit(wd_context *ctx, double2 *x, int64_t n, int slot)
{
    k_unit<<<blas_blocks(n), 256, 0, ctx->stream>>>(x, n, (const double2 *)ctx->red_partial + WD_RED_BLOCKS + slot);
    WD_LAUNCHED(ctx);
    return WD_OK;
}

// ------------------------------------------- precision-dispatched BLAS
static wd_status same_prec(wd_context *ctx, std::initializer_list<WdVec> v)
{
    const wd_precision p = v.begin()->prec;
    for (const WdVec &x : v)
        if (x.prec != p) return wd_fail(ctx, WD_ERR_BAD_ARG, "mixed storage precisions in one BLAS call");
    if (p != WD_PREC_F64 && p != WD_PREC_DF64)
        return wd_fail(ctx, WD_ERR_BAD_ARG, "BLAS-1 on this storage is not available");
    return WD_OK;
}

wd_status wd_v_norm2(wd_context *ctx, WdVec a, int64_t n, int slot)
{
    wd_status st = same_prec(ctx, {a});
    if (st != WD_OK) return st;
    if (a.prec == WD_PREC_F64) return wd_red_norm2(ctx, (const double2 *)a.p, n, slot);
    k_norm2_df<<<WD_RED_BLOCKS, WD_RED_THREADS, 0, ctx->stream>>>((const float4 *)a.p, n, (double2 *)ctx->red_partial);
    WD_LAUNCHED(ctx);
    return wd_red_finish(ctx, slot);
}

wd_status wd_v_dot(wd_context *ctx, WdVec a, WdVec b, int64_t n, int slot)
{
    wd_status st = same_prec(ctx, {a, b});
    if (st != WD_OK) return st;
    if (a.prec == WD_PREC_F64) return wd_red_dot(ctx, (const double2 *)a.p, (const double2 *)b.p, n, slot);
    k_dot_df<<<WD_RED_BLOCKS, WD_RED_THREADS, 0, ctx->stream>>>((const float4 *)a.p, (const float4 *)b.p, n,
                                                                (double2 *)ctx->red_partial);
    WD_LAUNCHED(ctx);
    return wd_red_finish(ctx, slot);
}

wd_status wd_v_axpby(wd_context *ctx, double2 a, WdVec x, double2 b, WdVec y, int64_t n)
{
    wd_status st = same_prec(ctx, {x, y});
    if (st != WD_OK) return st;
    if (x.prec == WD_PREC_F64) return wd_blas_axpby(ctx, a, (const double2 *)x.p, b, (double2 *)y.p, n);
    k_axpby_df<<<blas_blocks(n), 256, 0, ctx->stream>>>(dfc_split(a), (const float4 *)x.p, dfc_split(b),
                                                        (float4 *)y.p, n);
    WD_LAUNCHED(ctx);
    return WD_OK;
}

wd_status wd_v_xpayz(wd_context *ctx, WdVec x, double2 a, WdVec y, WdVec z, int64_t n)
{
    wd_status st = same_prec(ctx, {x, y, z});
    if (st != WD_OK) return st;
    if (x.prec == WD_PREC_F64) return wd_blas_xpayz(ctx, (const double2 *)x.p, a, (const double2 *)y.p, (double2 *)z.p, n);
    k_xpayz_df<<<blas_blocks(n), 256, 0, ctx->stream>>>((const float4 *)x.p, dfc_split(a), (const float4 *)y.p,
                                                        (float4 *)z.p, n);
    WD_LAUNCHED(ctx);
    return WD_OK;
}

wd_status wd_v_xpby(wd_context *ctx, WdVec x, double b, WdVec y, int64_t n)
{
    wd_status st = same_prec(ctx, {x, y});
    if (st != WD_OK) return st;
    if (x.prec == WD_PREC_F64)
        k_xpby_real<<<blas_blocks(n), 256, 0, ctx->stream>>>((const double2 *)x.p, b, (double2 *)y.p, n);
    else
        k_xpby_real_df<<<blas_blocks(n), 256, 0, ctx->stream>>>((const float4 *)x.p, df_split(b), (float4 *)y.p, n);
    WD_LAUNCHED(ctx);
    return WD_OK;
}

wd_status wd_v_copy(wd_context *ctx, WdVec dst, WdVec src, int64_t n)
{
    if (dst.prec != src.prec) return wd_fail(ctx, WD_ERR_BAD_ARG, "copy between different storages");
    WD_CUDA(ctx, cudaMemcpyAsync(dst.p, src.p, n * wd_entry_bytes(src.prec), cudaMemcpyDeviceToDevice, ctx->stream));
    if (src.scale && dst.scale)
        WD_CUDA(ctx, cudaMemcpyAsync(dst.scale, src.scale, n / 12 * sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
    return WD_OK;
}

wd_status wd_v_zero(wd_context *ctx, WdVec v, int64_t n)
{
    WD_CUDA(ctx, cudaMemsetAsync(v.p, 0, n * wd_entry_bytes(v.prec), ctx->stream));
    if (v.scale) WD_CUDA(ctx, cudaMemsetAsync(v.scale, 0, n / 12 * sizeof(float), ctx->stream));
    return WD_OK;
}
