// gather_lean.cuh -- k_bal_lean, the per-nonzero walk of the balanced row-major
// product for rows summed with Kahan compensation, and the loads, stores and element
// conversions that it shares with the window kernel (gather_win.cuh), which takes every
// other such product.
//
// It takes the chunks of the balanced split (k_partition).  A row split across
// chunks is finished inside the kernel: its last piece to arrive adds all
// pieces in chunk order, so no fix-up launch is needed and a result does not
// depend on scheduling.
//
// Storage types (mixed precision): values TV in {float, bf16, fp16}, B in
// TB in {float, bf16, fp16, fp8 e4m3}; products and sums are FP32.  For FP8
// B, column k carries an FP32 scale (B = q * scale[k]); sums are taken over
// the unscaled q and each output column is scaled once, when its row is
// stored.  Rows of at least kahan_min nonzeros are summed with Kahan compensation (each
// piece of a split row included).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "internal.h"
#include "kernels.cuh"
#include "tma.cuh"

namespace daspmm {

using bf16 = __nv_bfloat16;
using fp16 = __half;
using fp8 = __nv_fp8_e4m3;

// 8 consecutive floats (32 bytes, 32-byte aligned).
__device__ __forceinline__ void ld8_nc(float (&r)[8], const float *p)
{
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]),
          "=f"(r[7])
        : "l"(p));
}
__device__ __forceinline__ void ld8_plain(float (&r)[8], const float *p)
{
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]),
                   "=f"(r[6]), "=f"(r[7])
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void ld8_cg(float (&r)[8], const float *p)
{
    asm volatile("ld.global.cg.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]),
                   "=f"(r[6]), "=f"(r[7])
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void st8(float *p, const float (&r)[8])
{
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(r[0]),
                 "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7])
                 : "memory");
}
__device__ __forceinline__ void st8_hint(float *p, const float (&r)[8], uint64_t pol)
{
    asm volatile("st.global.L2::cache_hint.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8}, %9;" ::
                     "l"(p), "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]),
                 "f"(r[6]), "f"(r[7]), "l"(pol)
                 : "memory");
}

// N consecutive elements of B (storage type T) as floats, one vector load.
template <typename T, int N>
__device__ __forceinline__ void ld_b(float (&r)[N], const T *p)
{
    if constexpr (std::is_same<T, float>::value) {
        if constexpr (N == 8) ld8_nc(r, reinterpret_cast<const float *>(p));
        else ld_nc<N>(r, reinterpret_cast<const float *>(p));
    } else if constexpr (sizeof(T) == 2) {
        // 2-byte types: N = 8 -> 16 bytes, 4 -> 8 bytes, 2 -> 4 bytes, 1 -> 2 bytes
        uint32_t w[(N + 1) / 2];
        if constexpr (N == 8) {
            const uint4 t = __ldg(reinterpret_cast<const uint4 *>(p));
            w[0] = t.x; w[1] = t.y; w[2] = t.z; w[3] = t.w;
        } else if constexpr (N == 4) {
            const uint2 t = __ldg(reinterpret_cast<const uint2 *>(p));
            w[0] = t.x; w[1] = t.y;
        } else if constexpr (N == 2) {
            w[0] = __ldg(reinterpret_cast<const unsigned int *>(p));
        } else {
            w[0] = __ldg(reinterpret_cast<const unsigned short *>(p));
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const unsigned short h = (unsigned short)(w[i / 2] >> (16 * (i & 1)));
            if constexpr (std::is_same<T, bf16>::value) r[i] = __uint_as_float((uint32_t)h << 16);
            else r[i] = __half2float(__ushort_as_half(h));
        }
    } else {  // fp8 e4m3: N bytes
        uint32_t w[(N + 3) / 4];
        if constexpr (N == 8) {
            const uint2 t = __ldg(reinterpret_cast<const uint2 *>(p));
            w[0] = t.x; w[1] = t.y;
        } else if constexpr (N == 4) {
            w[0] = __ldg(reinterpret_cast<const unsigned int *>(p));
        } else if constexpr (N == 2) {
            w[0] = __ldg(reinterpret_cast<const unsigned short *>(p));
        } else {
            w[0] = __ldg(reinterpret_cast<const unsigned char *>(p));
        }
#pragma unroll
        for (int i = 0; i < N; i += 2) {
            const __half2_raw h2 = __nv_cvt_fp8x2_to_halfraw2(
                (__nv_fp8x2_storage_t)(w[i / 4] >> (8 * (i % 4))), __NV_E4M3);
            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&h2));
            r[i] = f.x;
            if (i + 1 < N) r[i + 1] = f.y;
        }
    }
}

// One value of A (storage type T) as float, L2 hint.
template <typename T>
__device__ __forceinline__ float ld_val(const T *p, uint64_t pol)
{
    if constexpr (std::is_same<T, float>::value) {
        return ld_hint_f32(reinterpret_cast<const float *>(p), pol);
    } else {
        unsigned short h;
        asm("ld.global.nc.L2::cache_hint.u16 %0, [%1], %2;" : "=h"(h) : "l"(p), "l"(pol));
        if constexpr (std::is_same<T, bf16>::value) return __uint_as_float((uint32_t)h << 16);
        else return __half2float(__ushort_as_half(h));
    }
}

#ifndef DASPMM_LEAN_MINB
#define DASPMM_LEAN_MINB 5  // CTAs of 256 threads per SM: 40 warps, <= 48 registers
#endif
#ifndef DASPMM_LEAN_U
#define DASPMM_LEAN_U 4     // nonzeros (B rows) in flight per warp step
#endif

// One chunk of the balanced split, column tile `tile` of `tiles`, summed by
// the whole warp with the per-nonzero walk: every nonzero is compared with
// the end of the current row (row ends from a 32-entry lane cache), so empty
// rows, beta != 0 and Kahan rows are all handled.  A row split across chunks
// leaves its pieces in carry slots; the last piece to arrive adds them all
// in chunk order (piece_arrive).  W / 32 elements of the B row per lane.
template <int W, int U, typename TV, typename TB>
__device__ __forceinline__ void lean_chunk(const KArgs &a, int c, int tile, int tiles,
                                           uint64_t pol_once)
{
    constexpr int VL = W / 32;  // elements of the B row per lane
    constexpr bool SCALED = std::is_same<TB, fp8>::value;
    const int lane = threadIdx.x & 31;
    const int tb = tile * W + lane * VL;
    const TB *Bl = reinterpret_cast<const TB *>(a.B) + tb;
    const TV *Av = reinterpret_cast<const TV *>(a.vals);
    float sc[VL];
#pragma unroll
    for (int e = 0; e < VL; ++e) sc[e] = SCALED ? __ldg(a.bscale + tb + e) : 1.0f;
    const int2 m0 = a.meta[c], m1 = a.meta[c + 1];
    const int k0 = m0.x, k1 = m1.x, s1 = m1.y;
    int r = m0.y;
    bool cont = k0 > __ldg(a.rowPtr + r);
    // row-end cache: lane l holds rowPtr[rb + 1 + l]; the next 32 are prefetched
    int rb = r;
    int rc = __ldg(a.rowPtr + min(rb + 1 + lane, a.nr));
    int rn = __ldg(a.rowPtr + min(rb + 33 + lane, a.nr));
    int re = __shfl_sync(kFull, rc, 0);
    float acc[VL], comp[VL];
#pragma unroll
    for (int e = 0; e < VL; ++e) acc[e] = comp[e] = 0.0f;
    // Kahan rows: length of the current row (its start is the previous end)
    int rs = __ldg(a.rowPtr + r);
    bool kh = re - rs >= a.kahan_min;

    const bool head_piece = cont;  // row m0.y continues from an earlier chunk
    auto emit = [&](int row, bool ends) {
        if constexpr (SCALED) {
#pragma unroll
            for (int e = 0; e < VL; ++e) acc[e] *= sc[e];
        }
        if (ends && !cont) {
            float *dst = a.C + (size_t)row * a.ldc + tb;
            if (a.beta != 0.0f) {
                float old[VL];
                ld_plain<VL>(old, dst);
#pragma unroll
                for (int e = 0; e < VL; ++e) acc[e] = fmaf(a.beta, old[e], acc[e]);
            }
            st_hint<VL>(dst, acc, pol_once);
        } else {  // a piece of a row split across chunks: park it in its carry slot
            st_v<VL>(slot_ptr(a, c, cont ? 0 : 1, tb), acc);
        }
#pragma unroll
        for (int e = 0; e < VL; ++e) acc[e] = comp[e] = 0.0f;
        cont = false;
    };
    auto step = [&](int p, float v, const float (&b)[VL]) {
        while (p >= re) {
            emit(r, true);
            ++r;
            if (r - rb >= 32) {
                rb += 32;
                rc = rn;
                rn = __ldg(a.rowPtr + min(rb + 33 + lane, a.nr));
            }
            rs = re;
            re = __shfl_sync(kFull, rc, r - rb);
            kh = re - rs >= a.kahan_min;
        }
        if (kh) {
#pragma unroll
            for (int e = 0; e < VL; ++e) {  // Kahan: carry the rounding error along
                const float y = fmaf(v, b[e], -comp[e]);
                const float t = acc[e] + y;
                comp[e] = (t - acc[e]) - y;
                acc[e] = t;
            }
        } else {
#pragma unroll
            for (int e = 0; e < VL; ++e) acc[e] = fmaf(v, b[e], acc[e]);
        }
    };
    // Windows of 32 nonzeros: lane l holds the column/value of nonzero
    // wb + l; the next window's are loaded while this one is gathered.
    auto load_win = [&](int wb, int &col, float &val) {
        const bool ok = wb + lane < k1;
        col = ok ? ld_hint_s32(a.colIdx + wb + lane, pol_once) : 0;
        val = ok ? ld_val<TV>(Av + wb + lane, pol_once) : 0.0f;
    };
    int ccur, cnext;
    float vcur, vnext;
    load_win(k0, ccur, vcur);
    for (int wb = k0; wb < k1; wb += 32) {
        load_win(wb + 32, cnext, vnext);
        const int cnt = min(32, k1 - wb);
        int t = 0;
        for (; t + U <= cnt; t += U) {  // U rows in flight
            int cc[U];
            float vv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                cc[u] = __shfl_sync(kFull, ccur, t + u);
                vv[u] = __shfl_sync(kFull, vcur, t + u);
            }
            float b[U][VL];
#pragma unroll
            for (int u = 0; u < U; ++u) ld_b<TB, VL>(b[u], Bl + (size_t)cc[u] * a.ldb);
#pragma unroll
            for (int u = 0; u < U; ++u) step(wb + t + u, vv[u], b[u]);
        }
        for (; t < cnt; ++t) {
            float b[VL];
            ld_b<TB, VL>(b, Bl + (size_t)__shfl_sync(kFull, ccur, t) * a.ldb);
            step(wb + t, __shfl_sync(kFull, vcur, t), b);
        }
        ccur = cnext;
        vcur = vnext;
    }
    while (r < s1) {
        emit(r, true);
        ++r;
    }
    const int head_row = m0.y;
    bool tail_piece = false;
    if (r < a.nr && r == s1 && __ldg(a.rowPtr + r) < k1) {
        tail_piece = !cont;  // a continuing row here is the head piece itself
        emit(r, false);
    }
    // the pieces this chunk parked arrive (at most two; fence + count, and
    // the last piece of a row adds them all)
    if (head_piece) piece_arrive<VL>(a, head_row, tb, tiles, tile);
    if (tail_piece) piece_arrive<VL>(a, s1, tb, tiles, tile);
}

template <int W, int U, typename TV, typename TB>
__global__ void __launch_bounds__(256, DASPMM_LEAN_MINB) k_bal_lean(const KArgs a)
{
    const int lane = threadIdx.x & 31;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    const uint64_t pol_once = policy_evict_first();
    pdl_wait();  // the boundaries (k_partition) are complete
    // Chunks are handed out dynamically -- each warp starts with chunk = its
    // index, then takes the next unclaimed one from the column tile's queue
    // head (zeroed by k_partition), so warps that draw short chunks take more
    // and no wave of chunks is left half-used.
    long long cl = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    while (cl < a.nchunks) {
        lean_chunk<W, U, TV, TB>(a, (int)cl, blockIdx.y, gridDim.y, pol_once);
        unsigned int nx = 0;
        if (lane == 0) nx = atomicAdd(a.head + blockIdx.y, 1u);
        cl = nwarps + (long long)__shfl_sync(kFull, nx, 0);
    }
}

// ---------------------------------------------------------------- worker groups
// VL floats: plain / L2-hinted stores, plain and L2-coherent loads (VL = 8: one
// 32-byte access, 16: two).
template <int VL>
__device__ __forceinline__ void st_n(float *p, const float (&r)[VL])
{
    if constexpr (VL == 16) {
        st8(p, *reinterpret_cast<const float(*)[8]>(&r[0]));
        st8(p + 8, *reinterpret_cast<const float(*)[8]>(&r[8]));
    } else if constexpr (VL == 8) {
        st8(p, r);
    } else {
        st_v<VL>(p, r);
    }
}
template <int VL>
__device__ __forceinline__ void st_hint_n(float *p, const float (&r)[VL], uint64_t pol)
{
    if constexpr (VL == 16) {
        st8_hint(p, *reinterpret_cast<const float(*)[8]>(&r[0]), pol);
        st8_hint(p + 8, *reinterpret_cast<const float(*)[8]>(&r[8]), pol);
    } else if constexpr (VL == 8) {
        st8_hint(p, r, pol);
    } else {
        st_hint<VL>(p, r, pol);
    }
}
template <int VL>
__device__ __forceinline__ void ld_plain_n(float (&r)[VL], const float *p)
{
    if constexpr (VL == 16) {
        ld8_plain(*reinterpret_cast<float(*)[8]>(&r[0]), p);
        ld8_plain(*reinterpret_cast<float(*)[8]>(&r[8]), p + 8);
    } else if constexpr (VL == 8) {
        ld8_plain(r, p);
    } else {
        ld_plain<VL>(r, p);
    }
}
template <int VL>
__device__ __forceinline__ void ld_cg_n(float (&r)[VL], const float *p)
{
    if constexpr (VL == 16) {
        ld8_cg(*reinterpret_cast<float(*)[8]>(&r[0]), p);
        ld8_cg(*reinterpret_cast<float(*)[8]>(&r[8]), p + 8);
    } else if constexpr (VL == 8) {
        ld8_cg(r, p);
    } else {
        ld_cg<VL>(r, p);
    }
}

// NW 32-bit words (NW = 8: one 32-byte load, 4: 16 bytes, 2: 8 bytes) of B,
// read-only path, left packed; elem<TB>() unpacks element i as a float.
template <int NW>
__device__ __forceinline__ void ld_raw(uint32_t (&w)[NW], const void *p)
{
    if constexpr (NW == 8) {
        float f[8];
        ld8_nc(f, reinterpret_cast<const float *>(p));
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = __float_as_uint(f[i]);
    } else if constexpr (NW == 4) {
        const uint4 t = __ldg(reinterpret_cast<const uint4 *>(p));
        w[0] = t.x; w[1] = t.y; w[2] = t.z; w[3] = t.w;
    } else if constexpr (NW == 2) {
        const uint2 t = __ldg(reinterpret_cast<const uint2 *>(p));
        w[0] = t.x; w[1] = t.y;
    } else {
        static_assert(NW == 1, "4-, 8-, 16- or 32-byte lane loads");
        w[0] = __ldg(reinterpret_cast<const unsigned int *>(p));
    }
}
// acc[0] += a * lo(w), acc[1] += a * hi(w) for two packed 16-bit B elements
// and a 16-bit value a of the same type (BF16 or FP16), FP32 accumulate in one
// instruction each (fma.rn.f32.bf16 / .f16, sm_100): the product of two 16-bit
// values is exact in FP32, so each result is the single rounding of
// a*b + acc -- bit-identical to fmaf on the widened operands.
template <typename T>
__device__ __forceinline__ void fma2_16(float &acc0, float &acc1, unsigned short a, uint32_t w)
{
    unsigned short lo, hi;
    asm("mov.b32 {%0, %1}, %2;" : "=h"(lo), "=h"(hi) : "r"(w));
    if constexpr (std::is_same<T, bf16>::value) {
        asm("fma.rn.f32.bf16 %0, %1, %2, %0;" : "+f"(acc0) : "h"(a), "h"(lo));
        asm("fma.rn.f32.bf16 %0, %1, %2, %0;" : "+f"(acc1) : "h"(a), "h"(hi));
    } else {
        asm("fma.rn.f32.f16 %0, %1, %2, %0;" : "+f"(acc0) : "h"(a), "h"(lo));
        asm("fma.rn.f32.f16 %0, %1, %2, %0;" : "+f"(acc1) : "h"(a), "h"(hi));
    }
}

template <typename TB, int NW>
__device__ __forceinline__ float elem(const uint32_t (&w)[NW], int i)
{
    if constexpr (std::is_same<TB, float>::value) {
        return __uint_as_float(w[i]);
    } else if constexpr (std::is_same<TB, bf16>::value) {
        const uint32_t x = w[i >> 1];
        return __uint_as_float((i & 1) ? (x & 0xFFFF0000u) : (x << 16));
    } else if constexpr (std::is_same<TB, fp16>::value) {
        return __half2float(__ushort_as_half((unsigned short)(w[i >> 1] >> (16 * (i & 1)))));
    } else {  // fp8 e4m3 (element pairs share one conversion; see elem2)
        const __half2_raw h2 = __nv_cvt_fp8x2_to_halfraw2(
            (__nv_fp8x2_storage_t)(w[i >> 2] >> (8 * (i & 2))), __NV_E4M3);
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&h2));
        return (i & 1) ? f.y : f.x;
    }
}


}  // namespace daspmm
