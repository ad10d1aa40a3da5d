// gather_win.cuh -- k_win: balanced-CSR row-major SpMM by worker groups, and the
// rules that choose its shape.
//
// Bound: on graphs whose B rows mostly hit in L2, the gather's latency under
// load and the instructions around it (64 KB to 128 KB of B rows in flight per
// SM); with B rows at random from HBM, HBM itself.
#pragma once

#include "gather_lean.cuh"

namespace daspmm {

// NB bytes (32, 16, 8, 4, 2 or 1) of B in the read-only path, left packed.
template <int NB>
__device__ __forceinline__ void ld_bytes(uint32_t (&w)[NB >= 4 ? NB / 4 : 1], const void *p)
{
    if constexpr (NB >= 4) ld_raw<NB / 4>(w, p);
    else if constexpr (NB == 2) w[0] = __ldg(reinterpret_cast<const unsigned short *>(p));
    else w[0] = __ldg(reinterpret_cast<const unsigned char *>(p));
}

// Two choices that give the same bits and differ in what the compiler makes of the
// window loop; each shape has the one that measures best (see launch_win).
constexpr int kFormLate = 1;  // a nonzero's value is fetched from its lane with its sum, not
                              // with its load
constexpr int kFormLim = 2;   // a window's end is kept, not its length

// The columns of a worker's lane: J vectors of V, vector j at tb + j*G*V.
template <int G, int V, int J, bool MASK>
struct WinCols {
    int tb, nv;
    __device__ __forceinline__ bool on(int j) const { return !MASK || tb + j * G * V < nv; }
};

// A piece of split row `row`, already stored in its carry slot by this worker,
// arrives: piece_arrive for G lanes (`gmask`) and J vectors of V columns per
// lane, in chunks counted from nonzero `base`.  Templated on the kernel's types so that
// every kernel has its own copy: ptxas 12.9 crashes (at build time) on one copy shared by
// two kernels.
template <int G, int V, int J, int U, typename TV, typename TB, int MINB, bool BETA, bool MASK,
          int FORM>
static __device__ __noinline__ void piece_arrive_win(const int *__restrict__ rowPtr, int *cnt,
                                                     const float *slots, float *C, int ldc,
                                                     int nv, int chunk, float beta, int row,
                                                     int tb, int tiles, int tile, unsigned gmask,
                                                     int base)
{
    const WinCols<G, V, J, MASK> cs{tb, nv};
    const int rs = __ldg(rowPtr + row) - base, re = __ldg(rowPtr + row + 1) - base;
    const int c0 = first_chunk(rs, chunk), c1 = last_chunk(re, chunk);
    __threadfence();
    __syncwarp(gmask);
    int last = 0;
    if ((threadIdx.x & (G - 1)) == 0)
        last = atomicAdd(cnt + (size_t)c0 * tiles + tile, 1) == c1 - c0;
    last = __shfl_sync(gmask, last, 0, G);
    if (!last) return;
    // every piece has arrived: the counter goes back to zero for the next call
    if ((threadIdx.x & (G - 1)) == 0) cnt[(size_t)c0 * tiles + tile] = 0;
    __threadfence();
#pragma unroll
    for (int j = 0; j < J; ++j) {
        if (!cs.on(j)) continue;
        const int col = tb + j * G * V;
        float tot[V];
        ld_cg_n<V>(tot, slots + ((size_t)c0 * 2 + 1) * nv + col);
        constexpr int P = 2;  // independent carry loads in flight
        for (int cb = c0 + 1; cb <= c1; cb += P) {
            float hp[P][V];
#pragma unroll
            for (int u = 0; u < P; ++u)
                if (cb + u <= c1) ld_cg_n<V>(hp[u], slots + ((size_t)(cb + u) * 2) * nv + col);
#pragma unroll
            for (int u = 0; u < P; ++u)
                if (cb + u <= c1)
#pragma unroll
                    for (int e = 0; e < V; ++e) tot[e] += hp[u][e];
        }
        float *dst = C + (size_t)row * ldc + col;
        if constexpr (BETA) {
            float old[V];
            ld_plain_n<V>(old, dst);
#pragma unroll
            for (int e = 0; e < V; ++e) tot[e] = fmaf(beta, old[e], tot[e]);
        }
        st_n<V>(dst, tot);
    }
}

// The worker-group window kernel.  Each G-lane group of a warp is a worker: it
// takes one chunk of a group of 32 / G consecutive chunks and covers its
// column tile of a B row with G lanes x J loads of V elements, so one warp
// instruction gathers 32 / G nonzeros.  A window is at most G nonzeros; the
// ends of the rows that finish in it come as one bitmask (lane l looks at the
// end of row r + l), so the window is summed straight through, min(U, G) B
// rows in flight, and a row is stored at its bit.
//
// Rows without nonzeros are k_partition's (it stores beta*C there, and leaves a
// bitmap of them).  A window's rows follow one another: in a group of chunks
// that has empty rows (or whose workspace had no room for the bitmap) a window
// also ends at the first of them, and the next one starts at the row of the next
// nonzero, found among the G rows in sight or, where those are all empty, by a
// G-way search.  The other groups do not ask: a loop that asked at each window
// kept it waiting for the answer before its first load (BF16 N = 256 on the
// power-law matrix 152 us, without 117), and a second loop for the groups with
// gaps cost the first one registers (138).
//
// A worker short of nonzeros in a step pads with column 0 and value 0.  If row 0 of
// B holds an Inf or NaN that is no zero, but it is added after the worker's last
// row end, so it can reach only a piece of a row that goes on in the next chunk,
// and that is then summed again.
//
// BETA: C = sum + beta*C; a row's old values are loaded when the row before it
// is stored, the first one's with the window, so no store waits for its load
// (and all of a window's are prefetched to L2 when the ends are found).  MASK:
// columns at or past nv are neither loaded (the loads are clamped to the last
// vector) nor stored.  FORM: see kFormLate.
template <int G, int V, int J, int U, typename TV, typename TB, int MINB, bool BETA, bool MASK,
          int FORM>
__global__ void __launch_bounds__(256, MINB) k_win(const KArgs a)
{
    constexpr int NW = 32 / G;                     // workers per warp
    constexpr int W = G * V * J;                   // columns of a tile
    constexpr int NB = V * (int)sizeof(TB);        // bytes of a lane's load
    constexpr int RAW = NB >= 4 ? NB / 4 : 1;
    constexpr int UU = U < G ? U : G;              // rows in flight per step
    constexpr unsigned GM = G == 32 ? 0xFFFFFFFFu : ((1u << G) - 1u);
    constexpr bool SCALED = std::is_same<TB, fp8>::value;
    // FP16 values and B: one mixed-precision FMA per element (measured 2-3%
    // faster at N = 256 / 512; the BF16 form of that instruction measured
    // slower than unpacking to FP32, so BF16 unpacks)
    constexpr bool PAIR16 =
        std::is_same<TV, fp16>::value && std::is_same<TB, fp16>::value && V >= 2;
    constexpr bool LATE = (FORM & kFormLate) != 0, LIM = (FORM & kFormLim) != 0;
    const int lane = threadIdx.x & 31, w = lane / G, gl = lane % G;
    const unsigned gmask = GM << (G * w);
    const int tile = blockIdx.y, tiles = gridDim.y;
    const WinCols<G, V, J, MASK> cs{tile * W + gl * V, a.nv};
    const TB *Bl[J];  // this lane's vectors of row 0
#pragma unroll
    for (int j = 0; j < J; ++j)
        Bl[j] = reinterpret_cast<const TB *>(a.B) +
                (MASK ? min(cs.tb + j * G * V, a.nv - V) : cs.tb + j * G * V);
    const TV *Av = reinterpret_cast<const TV *>(a.vals);
    const uint64_t pol_once = policy_evict_first();
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;

    pdl_trigger();
    pdl_wait();  // the boundaries (or the list) are complete
    float sc[SCALED ? J : 1][SCALED ? V : 1];  // read after the wait, like every input
    if constexpr (SCALED) {
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
            for (int e = 0; e < V; ++e) sc[j][e] = __ldg(a.bscale + cs.tb + j * G * V + e);
    }
    const long long ngroups = ((long long)a.nchunks + NW - 1) / NW;
    // (without nonzeros nothing is padded, and B may have no rows)
    bool pad_ok = true;
    if (a.nnz > 0) {
#pragma unroll
        for (int j = 0; j < J; ++j) {
            uint32_t b[RAW];
            ld_bytes<NB>(b, Bl[j]);
#pragma unroll
            for (int e = 0; e < V; ++e) pad_ok &= isfinite(elem<TB, RAW>(b, e));
        }
    }
    pad_ok = __all_sync(kFull, pad_ok);
    long long gi = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    while (gi < ngroups) {
        const int c = (int)(NW * gi) + w;
        const bool have = c < a.nchunks;
        int wb = 0, ke = 0, s1 = 0, r = 0;  // the next nonzero, the chunk's end, rows
        if (have) {
            const int2 m0 = a.meta[c], m1 = a.meta[c + 1];
            wb = m0.x;
            ke = m1.x;
            s1 = m1.y;
            r = m0.y;
        }
        int E = __ldg(a.rowPtr + min(r + 1 + gl, a.nr));  // lane l: the end of row r + l
        const int rstart = __ldg(a.rowPtr + r);
        // Empty rows among [r, s1)?  More rows than nonzeros say so at once; else the
        // bitmap, G words of 32 rows at a time.
        bool gaps = have && (!a.emap || s1 - r > ke - wb);
        if (have && !gaps) {
            for (int q = (r >> 5) + gl; q <= (s1 - 1) >> 5; q += G) {
                unsigned m = __ldcg(a.emap + q);
                if (q == r >> 5) m &= 0xFFFFFFFFu << (r & 31);
                if (q == (s1 - 1) >> 5) m &= 0xFFFFFFFFu >> (31 - ((s1 - 1) & 31));
                gaps |= m != 0;
            }
        }
        const bool any_gaps = __any_sync(kFull, gaps);
        auto load_win = [&](int p, int &col, float &val) {
            const bool ok = p + gl < ke;
            col = ok ? ld_hint_s32(a.colIdx + p + gl, pol_once) : 0;
            val = ok ? ld_val<TV>(Av + p + gl, pol_once) : 0.0f;
        };
        int ccur, cnext;
        float vcur, vnext;
        load_win(wb, ccur, vcur);
        const int r0 = r, k0 = wb;
        bool cont = have && wb > rstart;  // row r began in an earlier chunk
        const bool head_piece = cont;
        int nwin = (ke - wb + G - 1) / G;  // windows to go, of the worker with most
#pragma unroll
        for (int o = G; o < 32; o <<= 1) nwin = max(nwin, __shfl_xor_sync(kFull, nwin, o));
        float acc[J][V];
        auto clear = [&] {
#pragma unroll
            for (int j = 0; j < J; ++j)
#pragma unroll
                for (int e = 0; e < V; ++e) acc[j][e] = 0.0f;
        };
        clear();
        // One nonzero's share of the sums, and the store where a row ends.
        float *cdst;
        float old[BETA ? J : 1][BETA ? V : 1];  // BETA: the current row's old values
        auto c_row = [&](int row) { return a.C + (size_t)row * a.ldc + cs.tb; };
        auto fetch_old = [&](const float *p, bool any) {
#pragma unroll
            for (int j = 0; j < (BETA ? J : 0); ++j)
                if (any && cs.on(j)) ld_plain_n<BETA ? V : 1>(old[j], p + j * G * V);
        };
        auto prefetch_old = [&](bool in) {
            if (BETA && in) {
                const float *p = a.C + (size_t)(r + gl) * a.ldc + tile * W;
#pragma unroll
                for (int k = 0; k < W; k += 32)
                    if (!MASK || tile * W + k < a.nv)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(p + k));
            }
        };
        auto add = [&](float v, const uint32_t (&b)[J][RAW]) {
            if constexpr (PAIR16) {
                // v holds the FP16 value widened exactly: narrowing is exact
                const unsigned short a16 = __half_as_ushort(__float2half_rn(v));
#pragma unroll
                for (int j = 0; j < J; ++j)
#pragma unroll
                    for (int i = 0; i < RAW; ++i)
                        fma2_16<TB>(acc[j][2 * i], acc[j][2 * i + 1], a16, b[j][i]);
            } else {
#pragma unroll
                for (int j = 0; j < J; ++j)
#pragma unroll
                    for (int e = 0; e < V; ++e)
                        acc[j][e] = fmaf(v, elem<TB, RAW>(b[j], e), acc[j][e]);
            }
        };
        auto flush = [&]() {
#pragma unroll
            for (int j = 0; j < J; ++j) {
                if constexpr (SCALED) {
#pragma unroll
                    for (int e = 0; e < V; ++e) acc[j][e] *= sc[j][e];
                }
                if constexpr (BETA) {
                    if (!cont) {
#pragma unroll
                        for (int e = 0; e < V; ++e)
                            acc[j][e] = fmaf(a.beta, old[j][e], acc[j][e]);
                    }
                }
                if (cs.on(j)) st_hint_n<V>(cdst + j * G * V, acc[j], pol_once);
            }
            clear();
            cont = false;
        };
        bool sought = false;
        int lim = ke;  // where this window ends at the latest
        for (; nwin > 0; --nwin) {
            int wlen = G;  // (without gaps; a worker's last window may hold fewer)
            int skip = 0;  // empty rows between this window's and the next one's
            if (any_gaps) {
                const int left = ke - wb;  // <= 0: this worker is done
                // the first row in sight that is empty, and the window up to it
                int prev = __shfl_up_sync(kFull, E, 1, G);
                if (gl == 0) prev = wb;
                const bool holds = left > 0 && E > prev;
                const unsigned live = (__ballot_sync(kFull, holds) >> (G * w)) & GM;
                const int f = __ffs(~live | (1u << (G - 1) << 1)) - 1;  // rows r .. r + f - 1
                const int Ef = __shfl_sync(kFull, E, max(0, f - 1), G);
                wlen = f > 0 ? max(0, min(min(G, left), Ef - wb)) : 0;
                // (a row pointer that does not ascend must not hold the loop up)
                if (sought && wlen == 0) wlen = min(1, max(0, left));
                if (gl >= wlen) {  // not this window's
                    ccur = 0;
                    vcur = 0.0f;
                }
                bool seek = wlen == 0 && left > 0;  // row r is empty: where is nonzero wb?
                sought = seek;
                if (__any_sync(kFull, seek)) {
                    const int near = __ffs(live) - 1;  // in sight
                    int lo = near >= 0 ? r + near : min(r + G, a.nr), hi = s1;
                    bool far = seek && near < 0 && lo < hi;  // rowPtr[lo] <= wb
                    while (__any_sync(kFull, far)) {
                        const int step = (hi - lo + G) / G, x = lo + gl * step;
                        const bool le = far && x <= hi && __ldg(a.rowPtr + x) <= wb;
                        const int m = max(1, __popc(__ballot_sync(kFull, le) & gmask));
                        if (far) {
                            lo += (m - 1) * step;
                            hi = min(hi, lo + step - 1);
                            far = lo < hi;
                        }
                    }
                    if (seek) r = lo;
                }
                if (f > 0 && wlen > 0 && wlen == Ef - wb) skip = max(0, __ffs(live >> f) - 1);
                lim = wb + wlen;
                nwin = 1 + (max(0, left - wlen) + G - 1) / G;
#pragma unroll
                for (int o = G; o < 32; o <<= 1)
                    nwin = max(nwin, __shfl_xor_sync(kFull, nwin, o));
            }
            const int wn = LIM ? min(wb + G, lim) : wb + wlen;
            load_win(wn, cnext, vnext);
            const int pos = E - 1 - wb;
            const bool in = r + gl < a.nr && pos >= 0 &&
                            (LIM ? E <= wn : pos < min(ke - wb, wlen));
            const unsigned ends =
                (__reduce_or_sync(kFull, in ? (1u << (pos + G * w)) : 0u) >> (G * w)) & GM;
            prefetch_old(in);
            // the next window's row ends load while this one is summed
            E = __ldg(a.rowPtr + min(r + __popc(ends) + skip + 1 + gl, a.nr));
            fetch_old(c_row(r), ends != 0);
            cdst = cont ? slot_ptr(a, c, 0, cs.tb) : c_row(r);
#pragma unroll
            for (int g = 0; g < G / UU; ++g) {
                int cc[UU];
                float vv[UU];
#pragma unroll
                for (int u = 0; u < UU; ++u) {
                    cc[u] = __shfl_sync(kFull, ccur, g * UU + u, G);
                    if (!LATE) vv[u] = __shfl_sync(kFull, vcur, g * UU + u, G);
                }
                uint32_t b[UU][J][RAW];
#pragma unroll
                for (int u = 0; u < UU; ++u)
#pragma unroll
                    for (int j = 0; j < J; ++j)
                        ld_bytes<NB>(b[u][j], Bl[j] + (size_t)cc[u] * a.ldb);
#pragma unroll
                for (int u = 0; u < UU; ++u) {
                    if (LATE) vv[u] = __shfl_sync(kFull, vcur, g * UU + u, G);
                    add(vv[u], b[u]);
                    if ((ends >> (g * UU + u)) & 1u) {
                        flush();
                        ++r;
                        cdst = c_row(r);
                        fetch_old(cdst, (ends >> (g * UU + u)) > 1u);
                    }
                }
                asm volatile("" ::: "memory");
            }
            if (any_gaps) {
                r += skip;
                if (wn - wb < G && wn < ke) clear();  // it ended with a row: only padding is left
            }
            wb = wn;
            ccur = cnext;
            vcur = vnext;
        }
        // row s1 holds nonzeros of this chunk and goes on in the next one: a piece of it
        // (the head piece again if the row fills the chunk)
        bool tail = false;
        if (have && s1 < a.nr) {
            const int t0 = __ldg(a.rowPtr + s1);
            if (t0 < ke) {
                if (!pad_ok) {  // the sum went on into the padding: once more, without
                    clear();
                    for (int q = max(t0, k0); q < ke; ++q) {
                        uint32_t b[J][RAW];
                        const int col = __ldg(a.colIdx + q);
#pragma unroll
                        for (int j = 0; j < J; ++j)
                            ld_bytes<NB>(b[j], Bl[j] + (size_t)col * a.ldb);
                        add(ld_val<TV>(Av + q, pol_once), b);
                    }
                }
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    if constexpr (SCALED) {
#pragma unroll
                        for (int e = 0; e < V; ++e) acc[j][e] *= sc[j][e];
                    }
                    if (cs.on(j)) st_n<V>(slot_ptr(a, c, cont ? 0 : 1, cs.tb) + j * G * V, acc[j]);
                }
                tail = !cont;
            }
        }
        // (a row is cut where chunks begin by count, so its chunk says where they are
        // counted from: 0, or the first of a larger matrix's rows)
        if (head_piece)
            piece_arrive_win<G, V, J, U, TV, TB, MINB, BETA, MASK, FORM>(
                a.rowPtr, a.cnt, a.slots, a.C, a.ldc, a.nv, a.chunk, a.beta, r0, cs.tb, tiles, tile,
                gmask, k0 - c * a.chunk);
        if (tail)
            piece_arrive_win<G, V, J, U, TV, TB, MINB, BETA, MASK, FORM>(
                a.rowPtr, a.cnt, a.slots, a.C, a.ldc, a.nv, a.chunk, a.beta, s1, cs.tb, tiles, tile,
                gmask, ke - (c + 1) * a.chunk);
        __syncwarp();
        // the next group from the tile's queue; a call makes exactly ngroups
        // claims, so a planned product counts on from where the last one ended
        unsigned int nx = 0;
        if (lane == 0) nx = atomicAdd(a.head + tile, 1u) - a.head_base;
        gi = nwarps + (long long)__shfl_sync(kFull, nx, 0);
    }
}

// A launch that may overlap the previous kernel of the stream (programmatic
// dependent launch); the kernel calls pdl_wait() before reading its inputs.
// With a.l2_window > 0 the launch also carries an L2 access-policy window
// over B (that many thousandths of its lines persisting, the rest streaming).
// A failure is left in the runtime's last error for the caller's check.
inline void launch_pdl(void (*kernel)(KArgs), dim3 grid, cudaStream_t st, const KArgs &a)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 1;
    if (a.l2_window > 0 && a.b_bytes > 0) {
        int dev = 0, maxw = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&maxw, cudaDevAttrMaxAccessPolicyWindowSize, dev);
        at[1].id = cudaLaunchAttributeAccessPolicyWindow;
        at[1].val.accessPolicyWindow.base_ptr = const_cast<float *>(a.B);
        at[1].val.accessPolicyWindow.num_bytes = std::min<size_t>(a.b_bytes, (size_t)maxw);
        at[1].val.accessPolicyWindow.hitRatio = std::min(1.0f, a.l2_window / 1000.0f);
        at[1].val.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
        at[1].val.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
        cfg.numAttrs = maxw > 0 ? 2 : 1;
    }
    cfg.attrs = at;
    cudaLaunchKernelEx(&cfg, kernel, a);
}

template <int G, int V, int J, int U, typename TV, typename TB, int MINB, bool MASK,
          int FORM = 0>
inline void launch_win_as(const Resolved &r, const KArgs &a, cudaStream_t st)
{
    constexpr int NW = 32 / G;
    const long long groups = ((long long)a.nchunks + NW - 1) / NW;
    const unsigned gg = (unsigned)std::max<long long>(
        1, std::min<long long>((groups + 7) / 8, (long long)device_sms() * MINB));
    const dim3 grid(gg, r.tiles);
    if (a.beta == 0.0f)
        launch_pdl(k_win<G, V, J, U, TV, TB, MINB, false, MASK, FORM>, grid, st, a);
    else
        launch_pdl(k_win<G, V, J, U, TV, TB, MINB, true, MASK,
                         std::is_same<TB, float>::value ? kFormLim : kFormLate>, grid, st, a);
}

// B and C aligned for lane loads of V elements (and 32-byte stores from eight
// columns per lane on).
template <typename TB>
inline bool win_aligned(const KArgs &a, int V)
{
    const uintptr_t cs = V >= 8 ? 32 : 4 * V;
    return reinterpret_cast<uintptr_t>(a.B) % (V * sizeof(TB)) == 0 &&
           (reinterpret_cast<uintptr_t>(a.C) | reinterpret_cast<uintptr_t>(a.slots)) % cs == 0;
}

// The shape for a tile of W = 128, 64 or 32 columns that divides nv: a wide form,
// and one for B or C off its alignment.  Measured (us per product) on the 262k
// power-law matrix / a 262k uniform-random one of 8 per row, some rows empty; in
// brackets the kernel before it, which left every chunk with an empty row to a
// walk in a second launch:
//   FP32, N = 32 / 64 / 128 / 256 / 512: 34.4 / 52.3 / 83.5 / 161 / 302 [33.9 / 53.3 /
//     83.8 / 162 / 307], random 39.5 / 60.7 / 122 / 247 / 492 [58.2 / 80.3 / 150 / 281 / 522]
//   BF16, N = 32 .. 256: 35.2 / 46.4 / 67.5 / 127 [35.4 / 45.1 / 71.2 / 136], random
//     38.1 / 52.3 / 84.4 / 169 [54.5 / 70.1 / 112 / 215]
//   FP16: 34.1 / 42.6 / 62.0 / 116 [35.0 / 43.1 / 62.9 / 118], random 35.1 / 47.5 / 74.2 /
//     148 [53.4 / 67.7 / 97.9 / 184]
//   BF16 values, E4M3 B: 36.5 / 46.4 / 65.4 / 130 [45.1 / 45.4 / 64.6 / 131], random
//     41.2 / 51.6 / 81.9 / 143 [51.5 / 65.9 / 98.4 / 181]
// FP32 rows of 128 columns take 16-lane workers with 32-byte loads; 2-byte B 16
// rows in flight (their registers are those of 8 FP32 rows; a worker's lanes are the
// most: 8 rows with 8 lanes); the narrower tiles
// of 2- and 1-byte B 8-byte loads in 24 warps per SM, E4M3 in 32 columns 4-byte
// ones (8-lane workers: windows of 8 nonzeros, against 4 with 8-byte loads,
// 54.7 and 46.0 us); E4M3 in 128 columns 8-byte loads in 16-lane workers for one
// tile, 16-byte loads in 8-lane ones for wider products.
// The loop's form (kFormLate, kFormLim), us on the power-law matrix / the uniform-random one
// with none, late, lim, both; what is taken stands first:
//   FP32     N = 32 none 34.6 / 39.4, 36.0 / 42.7, 34.9 / 39.9, 38.1 / 48.1; N = 64 none 56 / 57,
//            58 / 59, 63 / 66, 58 / 59; N = 128 none 84.6 / 121, 92 / 132, 83.9 / 121, 85.7 / 123
//   BF16     N = 32 late 36.3 / 39.3, none 36.9 / 39.1, lim 35.9 / 38.5, both 36.3 / 39.6; N = 64
//            none 45.1 / 49.7, 46.1 / 52.0, 46.3 / 52.3, 46.4 / 53.1; N = 128 both 66.6 / 84.7,
//            none 69.9 / 87.9, late 68.4 / 85.7, lim 68.3 / 85.6
//   FP16     N = 32 none 34.8 / 37.5, 37.1 / 43.1, 34.7 / 37.3, 35.4 / 39.8; N = 64 lim 43.5 /
//            47.9, none 45.0 / 50.8, late 45.3 / 50.9, both 45.6 / 52.6; N = 128 both 64.4 / 80.0,
//            none 70.3 / 89.3, late 69.6 / 87.7, lim 65.7 / 80.8 (uniform rows of 20 lose: 73.6,
//            lim 71.4)
//   E4M3 B   N = 32 both 35.8 / 37.6, none 36.0 / 38.5, late 36.6 / 41.6, lim 36.0 / 38.4; N = 64
//            none 46.3 / 50.3, 46.8 / 52.7, 47.8 / 54.2, 46.2 / 52.0; N = 128 lim 61.3 / 72.1, none
//            61.9 / 73.0, late 63.1 / 75.6, both 62.5 / 74.2; N = 256 late 128.5 / 142.6, none 133 /
//            151, lim 133 / 150, both 128.9 / 143.5
//   masked   none: N = 41 57.5 / 59.1, 58.9 / 61.3, 57.2 / 59.2, 59.0 / 61.7
template <int W, typename TV, typename TB>
inline void launch_win(const Resolved &r, const KArgs &a, cudaStream_t st)
{
    constexpr bool f32 = std::is_same<TB, float>::value;
    constexpr bool f16 = std::is_same<TB, fp16>::value;
    constexpr bool b2 = sizeof(TB) == 2;
    if constexpr (W == 128) {
        if constexpr (f32) {
            if (win_aligned<TB>(a, 8))
                return launch_win_as<16, 8, 1, 8, TV, TB, 2, false>(r, a, st);
        } else if constexpr (b2) {
            if (win_aligned<TB>(a, 8))
                return launch_win_as<16, 8, 1, 16, TV, TB, 2, false, kFormLate | kFormLim>(r, a, st);
        } else {
            if (r.tiles == 1 && win_aligned<TB>(a, 8))
                return launch_win_as<16, 8, 1, 16, TV, TB, 2, false, kFormLim>(r, a, st);
            if (r.tiles > 1 && win_aligned<TB>(a, 16))
                return launch_win_as<8, 16, 1, 8, TV, TB, 2, false, kFormLate>(r, a, st);
        }
        launch_win_as<16, 4, 2, 8, TV, TB, 2, false>(r, a, st);
    } else if constexpr (W == 64) {
        constexpr int V = b2 ? 4 : 8;
        if (win_aligned<TB>(a, V))
            return launch_win_as<64 / V, V, 1, 64 / V, TV, TB, f32 ? 2 : 3, false,
                                 f16 ? kFormLim : 0>(r, a, st);
        launch_win_as<16, 2, 2, 8, TV, TB, 3, false>(r, a, st);
    } else {
        if (win_aligned<TB>(a, 4))
            return launch_win_as<8, 4, 1, 8, TV, TB, 3, false,
                                 f32 || f16 ? 0 : b2 ? kFormLate : kFormLate | kFormLim>(r, a, st);
        launch_win_as<16, 1, 2, 8, TV, TB, 3, false>(r, a, st);
    }
}

// The walk for products with Kahan rows.
template <int W, typename TV, typename TB>
inline void launch_walk(const Resolved &r, const KArgs &a, cudaStream_t st)
{
    const unsigned gx = (unsigned)std::max<long long>(
        1, std::min<long long>(((long long)a.nchunks + 7) / 8,
                               (long long)device_sms() * DASPMM_LEAN_MINB));
    launch_pdl(k_bal_lean<W, DASPMM_LEAN_U, TV, TB>, dim3(gx, r.tiles), st, a);
}

}  // namespace daspmm
