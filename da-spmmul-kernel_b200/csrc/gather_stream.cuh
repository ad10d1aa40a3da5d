// gather_stream.cuh -- k_stream: balanced-CSR products of few dense columns (nv <=
// 8, SpMV among them) through shared memory.
//
// With a B row of a few bytes a product is bound by its index and value stream
// and by latency, not by B.  So the work is split by nonzeros alone: a CTA takes
// a chunk of consecutive nonzeros, loads their columns, values and B rows with
// all threads at once (coalesced, several independent loads per thread, no
// carried state), and only then do threads take rows: one per (row, column) sums
// its row's products from shared memory in nonzero order, long rows a warp.
// Rows without nonzeros fall out of the row loop; a chunk with more than kStreamRows rows
// is left to k_stream_fix, whose warps share out the rows (a million rows of 8, the lower
// half empty, N = 1 / 8 670 / 2043 us when one CTA walked them, 37 / 65 so; column-major
// N = 8 6027 and 128).  A chunk's boundary moves down to the start of a row shorter than
// kStreamSnap; longer rows are cut there, each piece leaves its sum in a slot and
// k_stream_fix adds the slots in chunk order.
// No partition pass: two warps of the CTA find the chunk's rows by a 32-way search
// while the others load (so the chunk's load starts kStreamSnap - 1 nonzeros
// early, where its boundary can be).
//
// The chunk makes one wave of eight CTAs per SM where shared memory allows.  SpMV of
// 262k x 262k with 8 random nonzeros per row: 35 us (a thread per 32 nonzeros, a
// partition and a fix-up pass) -> 15 us.
#pragma once

#include "internal.h"
#include "kernels.cuh"
#include "tma.cuh"

namespace daspmm {

// Up to here k_stream, above the window kernel.  us of either on the 262k power-law
// matrix / a uniform-random one of 8 per row when the line was drawn: 8 columns 29 / 33
// and 33 / 33, 12 columns 47 / 47 and 39 / 34, 16 columns 40 / 51 and 37 / 34 (k_stream at 8 now
// 26 / 26; the gather before both 97 / 54 at 8, 106 / 82 at 16).
constexpr int kStreamMaxNv = 8;
constexpr int kStreamSnap = 64;
constexpr int kStreamLong = 96;  // nonzeros from which on a warp sums a row
constexpr int kStreamPlain = 0, kStreamOne = 1, kStreamBased = 2;  // see k_stream
constexpr int kStreamRows = 4096;  // a chunk of more rows is left to k_stream_fix (a CTA
                                   // walks so many in 16 turns at one column)

// Shared memory of a chunk: values, and the rows of B (see pitch in k_stream).
inline size_t stream_smem(int chunk, int nv, bool cmc)
{
    return sizeof(float) * (size_t)(chunk + kStreamSnap) * ((cmc ? nv | 1 : nv) + 1);
}

// The last row r in [0, nr) with rowPtr[r] <= k (the one that holds nonzero k, 0 <= k <
// nnz), by the whole warp.
__device__ __forceinline__ int row_of(const int *__restrict__ rowPtr, int nr, int k)
{
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = nr;  // rowPtr[lo] <= k < rowPtr[hi]
    while (hi - lo > 1) {
        const int step = (hi - lo + 31) / 32, x = lo + (lane + 1) * step;
        const bool le = x < hi && __ldg(rowPtr + x) <= k;
        const int n = __popc(__ballot_sync(kFull, le));
        lo += n * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// NV: nv where it is known at compile time, else 0.  V floats per load of B (nv % V
// == 0, B aligned to them).  CMB / CMC: B / C column-major (B only with V == 1).  KIND, of
// which each is a form of its own because the checks in one for all cost 1 to 10 % at one
// and eight columns: kStreamOne, beta is 1, so a row without nonzeros is C's already and not
// touched; kStreamBased, the rows are some of a larger matrix's, whose row pointer does not
// start at 0 and whose nnz may be the matrix's.
template <int NV, int V, bool CMB, bool CMC, int KIND>
__global__ void __launch_bounds__(256) k_stream(const KArgs a)
{
    extern __shared__ __align__(16) float stream_mem[];
    __shared__ int2 bound[2];  // the chunk's first nonzero and row, and the next chunk's
    __shared__ bool cut[2];    // does a row go on across them?
    __shared__ int longs[64], nlong;
    const int nv = NV ? NV : a.nv, nvec = nv / V;
    // B rows in shared memory: for column-major C the lanes of a warp take the rows of
    // one column, so their pitch is odd (and they are stored float by float)
    const int pitch = CMC ? (nv | 1) : nv;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int c = blockIdx.x;
    const uint64_t pol_once = policy_evict_first();
    pdl_trigger();
    pdl_wait();
    constexpr bool BASED = KIND == kStreamBased;
    const int base = BASED ? __ldg(a.rowPtr) : 0, stop = BASED ? __ldg(a.rowPtr + a.nr) : a.nnz;
    long long kn0 = (long long)c * a.chunk;
    if (BASED) kn0 = min((long long)stop, base + kn0);
    const int kn1 = (int)min((long long)stop, kn0 + a.chunk);
    const int klo = BASED ? max(base, (int)kn0 - (kStreamSnap - 1))
                          : c == 0 ? 0 : (int)kn0 - (kStreamSnap - 1);  // chunk >= kStreamSnap
    const int n = kn1 - klo;
    float *sb = stream_mem, *sv = stream_mem + (a.chunk + kStreamSnap) * pitch;
    if (t == 0) nlong = 0;
    if (warp < 2) {  // these find the chunk's rows, the others load
        const int k = warp == 0 ? (int)kn0 : kn1;
        int2 m = make_int2(k, warp == 0 && (!BASED || c == 0) ? 0 : a.nr);
        bool across = false;
        if (BASED ? k < stop && (warp == 1 || c > 0) : warp == 0 ? c > 0 : k < a.nnz) {
            const int r = row_of(a.rowPtr, a.nr, k);
            const int rs = __ldg(a.rowPtr + r), re = __ldg(a.rowPtr + r + 1);
            // (never before the chunk's load begins, whatever the row pointer says)
            m = make_int2(re - rs < kStreamSnap ? max(rs, k - (kStreamSnap - 1)) : k, r);
            across = m.x > rs;
        }
        if (lane == 0) {
            bound[warp] = m;
            cut[warp] = across;
            if (warp == 0) const_cast<int2 *>(a.meta)[c] = m;
        }
    } else {
        // The loads: thread (j, v) takes vector v of nonzero j's row of B.
        const unsigned inv = NV || nvec == 1 ? 0u : 0xFFFFFFFFu / (unsigned)nvec + 1u;
        auto split = [&](int i, int &j, int &v) {
            if (NV) {
                j = i / (NV ? NV / V : 1);
                v = i % (NV ? NV / V : 1);
            } else {
                j = nvec == 1 ? i : (int)__umulhi((unsigned)i, inv);  // exact: i < 2^20
                v = i - j * nvec;
            }
        };
        const int items = n * nvec;
        constexpr int U = V == 1 && NV != 1 ? 4 : 8, T = 192;
        for (int i0 = t - 64; i0 < items; i0 += T * U) {
            int j[U], v[U], col[U];
            float b[U][V];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                split(min(i0 + u * T, items - 1), j[u], v[u]);
                col[u] = ld_hint_s32(a.colIdx + klo + j[u], pol_once);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (v[u] == 0) sv[j[u]] = ld_hint_f32(a.vals + klo + j[u], pol_once);
                if constexpr (CMB) b[u][0] = __ldg(a.B + (size_t)v[u] * a.ldb + col[u]);
                else ld_nc<V>(b[u], a.B + (size_t)col[u] * a.ldb + v[u] * V);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                float *s = sb + j[u] * pitch + v[u] * V;
                if constexpr (CMC) {
#pragma unroll
                    for (int e = 0; e < V; ++e) s[e] = b[u][e];
                } else {
                    st_v<V>(s, b[u]);
                }
            }
        }
    }
    __syncthreads();
    // The rows: [r0, s1), and row s1 if it begins here and goes on.
    const int k0 = bound[0].x, r0 = bound[0].y, k1 = bound[1].x, s1 = bound[1].y;
    const bool head = cut[0], tail = cut[1];
    const int rows = s1 - r0 + (tail ? 1 : 0);
    if (s1 - r0 > kStreamRows) {  // more than one CTA should walk: k_stream_fix's
        if (t == 0) const_cast<int2 *>(a.meta)[a.nchunks].x = (int)a.head_base;
        return;
    }
    auto dest = [&](int row, int k) -> float * {
        if (row == r0 && head) return a.slots + ((size_t)c * 2) * nv + k;
        if (row == s1) return a.slots + ((size_t)c * 2 + 1) * nv + k;
        return CMC ? a.C + (size_t)k * a.ldc + row : a.C + (size_t)row * a.ldc + k;
    };
    auto beta_of = [&](int row) { return (row == r0 && head) || row == s1 ? 0.0f : a.beta; };
    // (row, VC columns) of thread t, then every 256 further: row-major, columns next to
    // each other, so a warp stores whole lines; column-major, rows.
    constexpr int VC = CMC ? 1 : V;
    constexpr int least = KIND == kStreamOne ? 1 : 0;  // nonzeros of the rows that are written
    const int fast = CMC ? max(rows, 1) : nv / VC;
    int lo = t % fast, hi = t / fast;
    const int dlo = 256 % fast, dhi = 256 / fast;
    for (; hi < (CMC ? nv : rows);
         lo += dlo, hi += dhi + (lo >= fast), lo -= lo >= fast ? fast : 0) {
        const int row = r0 + (CMC ? lo : hi), k = CMC ? hi : lo * VC;
        if (CMC && lo >= rows) continue;
        const int p0 = max(__ldg(a.rowPtr + row), k0), p1 = min(__ldg(a.rowPtr + row + 1), k1);
        const int len = p1 - p0;
        if ((unsigned)(len - least) >= (unsigned)(kStreamLong - least)) {  // long, or not written
            if (k == 0 && len > 0) {
                const int q = atomicAdd(&nlong, 1);
                if (q < 64) longs[q] = row;  // (a chunk holds fewer)
            }
            continue;
        }
        float x[VC];
#pragma unroll
        for (int e = 0; e < VC; ++e) x[e] = 0.0f;
#pragma unroll 4
        for (int p = p0 - klo; p < p1 - klo; ++p) {
            float b[VC];
            ld_plain<VC>(b, sb + p * pitch + k);
            const float v = sv[p];
#pragma unroll
            for (int e = 0; e < VC; ++e) x[e] = fmaf(v, b[e], x[e]);
        }
        float *d = dest(row, k);
        const float beta = beta_of(row);
        if (beta != 0.0f) {
            float old[VC];
            ld_plain<VC>(old, d);
#pragma unroll
            for (int e = 0; e < VC; ++e) x[e] = fmaf(beta, old[e], x[e]);
        }
        st_v<VC>(d, x);
    }
    __syncthreads();
    // Long rows: (32 / kp) lanes per column, each every so many nonzeros, then a tree.
    int kp = 1;
    while (kp < nv) kp <<= 1;
    const int k = lane & (kp - 1), step = 32 / kp;
    for (int i = warp; i < min(nlong, 64); i += 8) {
        const int row = longs[i];
        const int p0 = max(__ldg(a.rowPtr + row), k0), p1 = min(__ldg(a.rowPtr + row + 1), k1);
        float x = 0.0f;
        if (k < nv)
            for (int p = p0 - klo + lane / kp; p < p1 - klo; p += step)
                x = fmaf(sv[p], sb[p * pitch + k], x);
        for (int d = kp; d < 32; d <<= 1) x += __shfl_xor_sync(kFull, x, d);
        if (lane < kp && k < nv) {
            float *d = dest(row, k);
            const float beta = beta_of(row);
            *d = beta == 0.0f ? x : fmaf(beta, *d, x);
        }
    }
}

// Rows that chunk c begins, up to the next chunk's first: more than kStreamRows?
__device__ __forceinline__ bool many_rows(const KArgs &a, int c)
{
    return (c + 1 < a.nchunks ? a.meta[c + 1].y : a.nr) - a.meta[c].y > kStreamRows;
}

// What k_stream leaves.
//
// Rows cut at chunk boundaries: the warp of the boundary after a row's first piece
// adds that piece's tail slot and the head slots of the chunks the row reaches.
//
// The chunks of more than kStreamRows rows, most of them without nonzeros, which one CTA
// would walk alone (it says that there are some with the call's number behind the
// boundaries; an old number there that happens to be this one's costs a look at the
// boundaries): 32 rows per warp and turn, a lane per row, rows of more than 16 nonzeros by
// the warp.  Their pieces of cut rows are summed with the slots of the others.
//
// cmb: B is column-major.
template <bool CMC>
static __global__ void __launch_bounds__(256) k_stream_fix(const KArgs a, bool cmb)
{
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, nv = a.nv;
    const bool left = a.meta[a.nchunks].x == (int)a.head_base;
    const long long c = 1 + (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    int2 m = make_int2(0, 0), before = m;
    int rs = 0, re = 0;
    if (c < a.nchunks) {
        m = a.meta[c];
        before = a.meta[c - 1];
        if (m.y < a.nr) {  // (behind the last nonzero otherwise)
            rs = __ldg(a.rowPtr + m.y);
            re = __ldg(a.rowPtr + m.y + 1);
        } else {
            rs = m.x;
        }
    }
    const bool here = m.x > rs && before.x <= rs;  // a row is cut here for the first time
    if (!here && !left) return;
    const int base = a.based ? __ldg(a.rowPtr) : 0;
    const size_t col_step = cmb ? 1 : a.ldb, k_step = cmb ? a.ldb : 1;
    int kp = 1;
    while (kp < nv) kp <<= 1;
    const int k = lane & (kp - 1), sub = lane / kp, subs = 32 / kp;
    // nonzeros [p0, p1) of a row, this lane's share of them in its column
    auto piece = [&](float x, int p0, int p1) {
        for (int p = p0 + sub; p < p1; p += subs)
            x = fmaf(__ldg(a.vals + p),
                     __ldg(a.B + __ldg(a.colIdx + p) * col_step + k * k_step), x);
        return x;
    };
    auto store = [&](int row, int col, float x, bool holds) {
        float *d = CMC ? a.C + (size_t)col * a.ldc + row : a.C + (size_t)row * a.ldc + col;
        if (a.beta == 0.0f) *d = x;
        else if (a.beta != 1.0f || holds) *d = fmaf(a.beta, *d, x);
    };
    if (here) {
        const int last = min((re - 1 - base) / a.chunk, a.nchunks - 1);  // of its last piece
        const bool first_left = m.y - before.y > kStreamRows, last_left = many_rows(a, last);
        float x = 0.0f;
        if (k < nv) {
            if (last_left) x = piece(x, base + last * a.chunk, re);
            if (first_left) x = piece(x, rs, m.x);
            for (long long q = c + sub; q <= last - last_left; q += subs)
                x += __ldcg(a.slots + (q * 2) * nv + k);
        }
        for (int d = kp; d < 32; d <<= 1) x += __shfl_xor_sync(kFull, x, d);
        if (lane < kp && k < nv) {
            if (!first_left) x += __ldcg(a.slots + ((c - 1) * 2 + 1) * nv + k);
            store(m.y, k, x, true);
        }
    }
    if (!left) return;
    const int nwarps = (int)gridDim.x * 8, w = (int)blockIdx.x * 8 + (threadIdx.x >> 5);
    constexpr int T = 4;  // groups of 32 rows in flight, nwarps apart: those that hold
                          // something lie next to each other, and so on different warps
    for (long long b = 32LL * w; b < a.nr; b += 32LL * T * nwarps) {
        int p0[T], len[T];
        int2 m[T];
        int next[T];
#pragma unroll
        for (int g = 0; g < T; ++g) {
            const long long row = b + 32LL * g * nwarps + lane;
            p0[g] = row < a.nr ? __ldg(a.rowPtr + row) : 0;
            len[g] = row < a.nr ? __ldg(a.rowPtr + row + 1) - p0[g] : -1;
        }
        // Chunk c begins in the row of nonzero c * chunk, so a row lies in the chunk of the
        // last nonzero of the rows up to it.
#pragma unroll
        for (int g = 0; g < T; ++g) {
            const int h = min(max(p0[g] + max(len[g], 0) - 1 - base, 0) / a.chunk, a.nchunks - 1);
            m[g] = a.meta[h];
            next[g] = h + 1 < a.nchunks ? a.meta[h + 1].y : a.nr;
        }
#pragma unroll
        for (int g = 0; g < T; ++g) {
            const long long r0 = b + 32LL * g * nwarps;
            const int row = (int)(r0 + lane);
            // of a chunk with too many rows; the chunk's first may be the last piece of a cut one
            if (next[g] - m[g].y <= kStreamRows || (row == m[g].y && m[g].x > p0[g])) len[g] = -1;
            const bool none = __all_sync(kFull, len[g] == 0);
            if (none && a.beta == 1.0f) continue;
            if (!CMC && none) {  // nothing in 32 rows: whole lines of beta*C
                float *d = a.C + (size_t)r0 * a.ldc;
                for (int i = lane; i < 32 * nv; i += 32)
                    d[i] = a.beta == 0.0f ? 0.0f : fmaf(a.beta, d[i], 0.0f);
                continue;
            }
            if (len[g] >= 0 && len[g] <= 16) {
                float x[kStreamMaxNv];
#pragma unroll
                for (int e = 0; e < kStreamMaxNv; ++e) x[e] = 0.0f;
                for (int p = p0[g]; p < p0[g] + len[g]; ++p) {
                    const float v = __ldg(a.vals + p);
                    const float *bp = a.B + __ldg(a.colIdx + p) * col_step;
#pragma unroll
                    for (int e = 0; e < kStreamMaxNv; ++e)
                        if (e < nv) x[e] = fmaf(v, __ldg(bp + e * k_step), x[e]);
                }
#pragma unroll
                for (int e = 0; e < kStreamMaxNv; ++e)
                    if (e < nv) store(row, e, x[e], len[g] > 0);
            }
            for (unsigned more = __ballot_sync(kFull, len[g] > 16); more; more &= more - 1) {
                const int l = __ffs(more) - 1;
                const int q0 = __shfl_sync(kFull, p0[g], l), q1 = q0 + __shfl_sync(kFull, len[g], l);
                float x = k < nv ? piece(0.0f, q0, q1) : 0.0f;
                for (int d = kp; d < 32; d <<= 1) x += __shfl_xor_sync(kFull, x, d);
                if (lane < kp && k < nv) store((int)r0 + l, k, x, true);
            }
        }
    }
}

// The CTAs of k_stream_fix: eight boundaries each, and enough for the rows that may be
// left (no chunk of fewer rows has more than kStreamRows).
inline int stream_fix_ctas(int nchunks, int nr)
{
    const int cuts = (nchunks - 1 + 7) / 8;
    if (nr <= kStreamRows) return cuts;
    return std::max(cuts, std::min(nr / 2048 + 1, device_sms() * 4));
}

// Nonzeros per chunk: one wave of eight CTAs per SM, in steps of 128, at most what
// eight CTAs' shared memory holds and 1280 (beyond, a thread's loads take a second
// round: SpMV on the power-law matrix 15.9 us at 1280, 19.4 at 1792, 17.5 at 512; four
// columns 20 at 1024, 23 at 512, 31 at 256).
inline int stream_chunk_most(int nv)
{
    return std::max(256, std::min(1280, (6880 / (nv + 1) - kStreamSnap) / 128 * 128));
}
inline int stream_chunk(int nnz, int nv)
{
    const long long per = ((long long)nnz + device_sms() * 8 - 1) / (device_sms() * 8);
    return (int)std::max<long long>(128, std::min<long long>((per + 127) / 128 * 128,
                                                             stream_chunk_most(nv)));
}

template <int NV, int V, bool CMB, bool CMC>
inline void launch_stream_as(const KArgs &a, cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)a.nchunks);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = stream_smem(a.chunk, a.nv, CMC);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg,
                       a.based          ? k_stream<NV, V, CMB, CMC, kStreamBased>
                       : a.beta == 1.0f ? k_stream<NV, V, CMB, CMC, kStreamOne>
                                        : k_stream<NV, V, CMB, CMC, kStreamPlain>,
                       a);
    const int fix = stream_fix_ctas(a.nchunks, a.nr);
    if (fix > 0) {
        cfg.gridDim = dim3((unsigned)fix);
        cfg.dynamicSmemBytes = 0;
        cudaLaunchKernelEx(&cfg, k_stream_fix<CMC>, a, CMB);
    }
}

// V: floats per load of a row-major B; cmb: B is column-major.
template <bool CMC>
inline void launch_stream(int V, bool cmb, const KArgs &a, cudaStream_t st)
{
    if (a.nv == 1) launch_stream_as<1, 1, false, CMC>(a, st);
    else if (cmb) launch_stream_as<0, 1, true, CMC>(a, st);
    else if (V == 4 && a.nv == 4) launch_stream_as<4, 4, false, CMC>(a, st);
    else if (V == 4 && a.nv == 8) launch_stream_as<8, 4, false, CMC>(a, st);
    else if (V == 2) launch_stream_as<0, 2, false, CMC>(a, st);
    else launch_stream_as<0, 1, false, CMC>(a, st);
}

}  // namespace daspmm
