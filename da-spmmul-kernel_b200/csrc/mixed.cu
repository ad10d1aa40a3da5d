// mixed.cu -- mixed-precision SpMM (BF16 / FP16 storage, FP8 E4M3 B with
// per-column scales, FP32 accumulation, optional Kahan rows) and the device
// quantizers that produce its inputs.  No counterpart in the reference, whose
// kernels are FP32 only (spmm.h:17-18); this extends that value/B type.
#include "gather_win.cuh"
#include "internal.h"
#include "kernels.cuh"

#include <cuda_runtime.h>

#include <algorithm>

namespace daspmm {

template <typename TV, typename TB>
static void launch_mixed(const Resolved &r, const KArgs &a, bool kahan, cudaStream_t st)
{
#define DASPMM_MW(w)                                                                        \
    if (r.W == w) {                                                                         \
        if (kahan) launch_walk<w, TV, TB>(r, a, st);                                        \
        else launch_win<w, TV, TB>(r, a, st);                                               \
        return;                                                                             \
    }
    DASPMM_MW(128) DASPMM_MW(64) DASPMM_MW(32)
#undef DASPMM_MW
}

static size_t fmt_bytes(int f)
{
    return f == DASPMM_F32 ? 4 : (f == DASPMM_E4M3 ? 1 : 2);
}

template <typename TQ>
__device__ __forceinline__ TQ quant(float x);
template <> __device__ __forceinline__ bf16 quant<bf16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ fp16 quant<fp16>(float x) { return __float2half_rn(x); }
template <> __device__ __forceinline__ fp8 quant<fp8>(float x)
{
    fp8 q;
    q.__x = __nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3);
    return q;
}

// q[i] = round(x[i] / scale[i % ncols]) (scale may be null: 1): any count, any
// alignment.
template <typename TQ>
static __global__ void k_quantize(const float *__restrict__ x, TQ *q, size_t n,
                                  const float *__restrict__ scale, int ncols)
{
    pdl_wait();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        float v = x[i];
        if (scale) v = v / scale[i % (size_t)ncols];
        q[i] = quant<TQ>(v);
    }
}

// Eight values rounded and packed (E4M3: 8 bytes, BF16 / FP16: 16 bytes).
template <typename TQ>
__device__ __forceinline__ void store8(TQ *q, const float (&v)[8])
{
    uint32_t w[2 * sizeof(TQ)];
    if constexpr (sizeof(TQ) == 1) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * i], v[4 * i + 1]),
                                                         __NV_SATFINITE, __NV_E4M3);
            const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * i + 2], v[4 * i + 3]),
                                                         __NV_SATFINITE, __NV_E4M3);
            w[i] = lo | (hi << 16);
        }
        *reinterpret_cast<uint2 *>(q) = make_uint2(w[0], w[1]);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            TQ p[2] = {quant<TQ>(v[2 * i]), quant<TQ>(v[2 * i + 1])};
            w[i] = *reinterpret_cast<const uint32_t *>(p);
        }
        *reinterpret_cast<uint4 *>(q) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// The same in vectors of eight (x 16-byte, q 8- or 16-byte aligned; n and,
// with scales, ncols multiples of 8).  Bound by memory: 4 bytes read and 1 or 2
// written per element.  A thread keeps its column (the active threads are a
// multiple of the vectors in a row), so its scales are loaded once and no
// index is divided; two vectors are in flight.  It walks from the end of x
// towards its start: column maxima taken just before (daspmm_e4m3_scales)
// left the end in L2.  262,144 x 256 to E4M3: 142 us one by one (a 64-bit
// remainder per element), 55 us here (6.1 TB/s).
template <typename TQ, bool SCALED>
static __global__ void __launch_bounds__(256)
    k_quantize8(const float *__restrict__ x, TQ *q, long long nvec,
                const float *__restrict__ scale, int cvec)
{
    pdl_wait();
    long long active = (long long)gridDim.x * blockDim.x;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float sc[8];
    if constexpr (SCALED) {
        active = active / cvec * cvec;  // cvec <= threads (checked by the launch)
        if (t >= active) return;
        const int c = (int)(t % cvec) * 8;
#pragma unroll
        for (int e = 0; e < 8; ++e) sc[e] = __ldg(scale + c + e);
    }
    auto one = [&](long long v, const float4 &a, const float4 &b) {
        float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        if constexpr (SCALED) {
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = f[e] / sc[e];
        }
        store8<TQ>(q + v * 8, f);
    };
    const long long turns = t < nvec ? (nvec - t + active - 1) / active : 0;
    const float4 *xv = reinterpret_cast<const float4 *>(x);
    long long v = t + (turns - 1) * active;
    for (long long k = turns; k > 0;) {
        const float4 a0 = __ldg(xv + 2 * v), b0 = __ldg(xv + 2 * v + 1);
        if (k > 1) {
            const long long v1 = v - active;
            const float4 a1 = __ldg(xv + 2 * v1), b1 = __ldg(xv + 2 * v1 + 1);
            one(v, a0, b0);
            one(v1, a1, b1);
            v = v1 - active;
            k -= 2;
        } else {
            one(v, a0, b0);
            k = 0;
        }
    }
}

// amax[k] = max_i |B[i, k]| as float bits (non-negative floats order as
// unsigned integers, so an integer max is exact and order-independent).
// V columns per lane (4: 16-byte loads, ncols % 4 == 0 and B 16-byte aligned),
// X lanes (a power of two) across the columns of a tile, 32 / X rows per warp
// and step, four steps in flight; the eight warps of a CTA meet in shared
// memory, one atomic per column and CTA.  Bound by reading B: 262,144 x 256 90 us with one
// 4-byte load in flight per lane, 49 us here (5.5 TB/s).
template <int V>
static __global__ void __launch_bounds__(256)
    k_colmax(const float *__restrict__ B, int nrows, int ncols, int X, unsigned *amax)
{
    __shared__ unsigned part[8][32 * V];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cl = lane % X, rl = lane / X, R = 32 / X;
    const int col = (blockIdx.x * X + cl) * V;
    const bool on = col < ncols;
    unsigned m[V];
#pragma unroll
    for (int e = 0; e < V; ++e) m[e] = 0;
    const long long step = (long long)gridDim.y * 8 * R;
    pdl_wait();
    auto take = [&](const float (&f)[V]) {
#pragma unroll
        for (int e = 0; e < V; ++e) m[e] = max(m[e], __float_as_uint(fabsf(f[e])));
    };
    long long i = ((long long)blockIdx.y * 8 + warp) * R + rl;
    for (; on && i + 3 * step < nrows; i += 4 * step) {
        float f[4][V];
#pragma unroll
        for (int u = 0; u < 4; ++u) ld_nc<V>(f[u], B + (size_t)(i + u * step) * ncols + col);
#pragma unroll
        for (int u = 0; u < 4; ++u) take(f[u]);
    }
    for (; on && i < nrows; i += step) {
        float f[V];
        ld_nc<V>(f, B + (size_t)i * ncols + col);
        take(f);
    }
#pragma unroll
    for (int e = 0; e < V; ++e) {
        for (int d = X; d < 32; d <<= 1) m[e] = max(m[e], __shfl_xor_sync(kFull, m[e], d));
        if (rl == 0) part[warp][cl * V + e] = m[e];
    }
    __syncthreads();
    for (int k = threadIdx.x; k < X * V; k += 256) {
        const int c = blockIdx.x * X * V + k;
        if (c >= ncols) break;
        unsigned a = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) a = max(a, part[w][k]);
        atomicMax(amax + c, a);
    }
}

static __global__ void k_zero_u32(unsigned *p, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    if (i < n) p[i] = 0;
}

// scale[k] = amax[k] / 448 (the largest finite E4M3), 1 for an all-zero column
static __global__ void k_scale_finish(unsigned *amax_bits, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    if (i >= n) return;
    const float m = __uint_as_float(amax_bits[i]);
    reinterpret_cast<float *>(amax_bits)[i] = m > 0.0f ? m / 448.0f : 1.0f;
}

// A launch that may be scheduled while the stream's previous kernel drains
// (every kernel launched with it waits for that kernel before it touches
// memory).
template <typename... P, typename... A>
static void launch_after(void (*kernel)(P...), dim3 grid, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Vectors of eight where sizes and addresses allow it, else one by one.
template <typename TQ>
static void launch_quantize(const float *x, void *q, size_t n, const float *scale, int ncols,
                            cudaStream_t st)
{
    const unsigned most = (unsigned)device_sms() * 8;  // the CTAs that fit at once
    const unsigned g8 = (unsigned)std::max<size_t>(1, std::min<size_t>((n / 8 + 255) / 256, most));
    const bool vec = n % 8 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)q % (8 * sizeof(TQ)) == 0;
    if (vec && !scale) {
        launch_after(k_quantize8<TQ, false>, dim3(g8), st, x, (TQ *)q, (long long)(n / 8), scale, 1);
    } else if (vec && ncols % 8 == 0 && (long long)g8 * 256 >= ncols / 8) {
        // (after the kernel that makes the scales, not beside it: they are read through
        // the read-only path, 57 us against 88 with plain loads)
        k_quantize8<TQ, true><<<g8, 256, 0, st>>>(x, (TQ *)q, (long long)(n / 8), scale, ncols / 8);
    } else {
        const unsigned g = (unsigned)std::min<size_t>((n + 255) / 256, 148 * 64);
        launch_after(k_quantize<TQ>, dim3(g), st, x, (TQ *)q, n, scale, ncols);
    }
}

template <int V>
static void launch_colmax(const float *B, int nrows, int ncols, unsigned *bits, cudaStream_t st)
{
    const int vecs = ncols / V;
    int X = 1;
    while (X < 32 && X < vecs) X <<= 1;
    const unsigned gx = (unsigned)((vecs + X - 1) / X);
    // about eight CTAs per SM over all column tiles, each with whole steps of work
    const long long rows = 8 * (32 / X);
    const long long gy = std::max<long long>(1, (long long)device_sms() * 8 / gx);
    const long long need = ((long long)nrows + rows * 4 - 1) / (rows * 4);
    launch_after(k_colmax<V>, dim3(gx, (unsigned)std::max<long long>(1, std::min(gy, need))), st, B,
                 nrows, ncols, X, bits);
}

}  // namespace daspmm

using namespace daspmm;

extern "C" {

daspmm_status daspmm_spmm_mixed(const daspmm_config *cfg_in, int layout, int nr, int nc, int nnz,
                                int nv, const int *rowPtr, const int *colIdx,
                                const void *values, int val_fmt, const void *B, int b_fmt,
                                const float *b_scales, float *C, float beta, int kahan_min,
                                void *workspace, size_t ws_bytes, void *stream)
{
    if (layout != DASPMM_ROW_MAJOR) return DASPMM_ERR_UNSUPPORTED;
    if (val_fmt < DASPMM_F32 || val_fmt > DASPMM_F16) return DASPMM_ERR_UNSUPPORTED;
    if (b_fmt < DASPMM_F32 || b_fmt > DASPMM_E4M3) return DASPMM_ERR_INVALID;
    if (b_fmt == DASPMM_E4M3 && !b_scales) return DASPMM_ERR_INVALID;
    const bool combo = (val_fmt == DASPMM_F32 && b_fmt == DASPMM_F32) ||
                       (val_fmt == DASPMM_BF16 && b_fmt == DASPMM_BF16) ||
                       (val_fmt == DASPMM_F16 && b_fmt == DASPMM_F16) ||
                       (val_fmt == DASPMM_F32 && b_fmt == DASPMM_E4M3) ||
                       (val_fmt == DASPMM_BF16 && b_fmt == DASPMM_E4M3);
    if (!combo) return DASPMM_ERR_UNSUPPORTED;
    daspmm_config cfg = cfg_in ? *cfg_in : daspmm_config{};
    cfg.alg = DASPMM_ALG_CSR_BALANCED;
    if (cfg.pipe && cfg.pipe != 4) return DASPMM_ERR_UNSUPPORTED;
    cfg.pipe = 4;
    // measured: reduced-precision B (the 16-lane group kernel) runs best, like
    // FP32, at 96 nonzeros per chunk for one 128-column tile and at 128 for
    // wider products (BF16 N = 128: 71.3 against 74.2 us; E4M3 64.6 against
    // 65.4).  Never more chunks than the FP32 default, so a workspace sized
    // for it still suffices.
    if (!cfg.chunk && nv > 0 && nnz >= 0) {
        const int L = cfg.lanes_col;  // the tile's width as resolve() has it
        const int W = L == 8 || L == 16 || L == 32 ? 4 * L
                                                   : (nv % 128 == 0 ? 128 : (nv % 64 == 0 ? 64 : 32));
        const int most = nv == 128 ? 96 : 128;
        // (compensated rows are cut no more often than that: their pieces are added plainly)
        cfg.chunk = kahan_min > 0 ? most : window_chunk(nv, W, nr, nnz, most);
        if (!cfg.snap && kahan_min <= 0) cfg.snap = window_snap(cfg.chunk);
    }
    Resolved r;
    daspmm_status s = resolve(&cfg, layout, nr, nc, nnz, nv, nullptr, C, &r);
    if (s != DASPMM_OK) return s;
    if (r.pipe != 4) return DASPMM_ERR_UNSUPPORTED;  // needs nv % 32 == 0
    const int VL = r.W / 32;
    if (B && ((uintptr_t)B % (VL * fmt_bytes(b_fmt)))) return DASPMM_ERR_INVALID;
    if (nr == 0) return DASPMM_OK;
    if (!B || !C || !rowPtr || (nnz > 0 && (!colIdx || !values))) return DASPMM_ERR_INVALID;
    cudaStream_t st = (cudaStream_t)stream;
    WorkspaceLock hold;
    if (!workspace) {
        hold = hold_workspace(st);
        const size_t need = workspace_bytes(r, nv);
        s = cached_workspace(need, st, &workspace);
        if (s != DASPMM_OK) return s;
        ws_bytes = need;
    }
    if (workspace_least(r, nv) > ws_bytes) return DASPMM_ERR_WORKSPACE;

    KArgs a{};
    a.nr = nr; a.nc = nc; a.nnz = nnz; a.nv = nv;
    a.ldb = nv; a.ldc = nv;
    a.rowPtr = rowPtr; a.colIdx = colIdx;
    a.vals = reinterpret_cast<const float *>(values);
    a.B = reinterpret_cast<const float *>(B);
    a.C = C; a.beta = beta;
    a.L = r.L; a.S = 1; a.chunk = r.chunk; a.nchunks = r.nchunks;
    a.bscale = b_scales;
    a.kahan_min = kahan_min > 0 ? kahan_min : 0x7fffffff;
    a.l2_window = r.l2_window;
    a.b_bytes = (size_t)fmt_bytes(b_fmt) * nc * nv;
    carve_balanced(r, workspace, ws_bytes, &a);
    const bool kahan = kahan_min > 0;
    launch_partition(r, nr, nnz, rowPtr, a, !kahan, st);
    timer_before(st);  // the optional timer brackets the main kernel
    if (val_fmt == DASPMM_F32 && b_fmt == DASPMM_F32) launch_mixed<float, float>(r, a, kahan, st);
    else if (val_fmt == DASPMM_BF16 && b_fmt == DASPMM_BF16) launch_mixed<bf16, bf16>(r, a, kahan, st);
    else if (val_fmt == DASPMM_F16) launch_mixed<fp16, fp16>(r, a, kahan, st);
    else if (val_fmt == DASPMM_F32) launch_mixed<float, fp8>(r, a, kahan, st);
    else launch_mixed<bf16, fp8>(r, a, kahan, st);
    timer_after(st);
    count_launches(1);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? DASPMM_OK : cuda_fail(e);
}

daspmm_status daspmm_quantize(int fmt, size_t n, const float *x, void *q, const float *col_scales,
                              int ncols, void *stream)
{
    if (n == 0) return DASPMM_OK;
    if (!x || !q || (col_scales && ncols <= 0)) return DASPMM_ERR_INVALID;
    cudaStream_t st = (cudaStream_t)stream;
    switch (fmt) {
    case DASPMM_BF16: launch_quantize<bf16>(x, q, n, col_scales, ncols, st); break;
    case DASPMM_F16: launch_quantize<fp16>(x, q, n, col_scales, ncols, st); break;
    case DASPMM_E4M3: launch_quantize<fp8>(x, q, n, col_scales, ncols, st); break;
    default: return DASPMM_ERR_UNSUPPORTED;
    }
    count_launches(1);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? DASPMM_OK : cuda_fail(e);
}

daspmm_status daspmm_e4m3_scales(int nrows, int ncols, const float *B, float *scales, void *stream)
{
    if (nrows < 0 || ncols <= 0 || !scales || (nrows > 0 && !B)) return DASPMM_ERR_INVALID;
    cudaStream_t st = (cudaStream_t)stream;
    unsigned *bits = reinterpret_cast<unsigned *>(scales);
    const dim3 gc((ncols + 255) / 256);
    launch_after(k_zero_u32, gc, st, bits, ncols);
    if (nrows > 0) {
        if (ncols % 4 == 0 && (uintptr_t)B % 16 == 0) launch_colmax<4>(B, nrows, ncols, bits, st);
        else launch_colmax<1>(B, nrows, ncols, bits, st);
    }
    launch_after(k_scale_finish, gc, st, bits, ncols);
    count_launches(nrows > 0 ? 3 : 2);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? DASPMM_OK : cuda_fail(e);
}

}  // extern "C"
