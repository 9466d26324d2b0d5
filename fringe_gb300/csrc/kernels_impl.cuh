// kernels_impl.cuh -- pixel kernels and their launchers (included by
// kernels_f32.cu and kernels_f64.cu so the two precisions compile in parallel).
//
// k_solve, k_rest      : eigen-solves from the tensor-core Gamma records.
// k_pixels<float, NP>  : plain FP32 kernel over a contiguous pixel range (windows
//                        the Gamma kernel does not take, and runs without scratch).
// k_pixels<double, NP> : the work list written by the FP32 pass (pixels whose
//                        discrete decisions fall inside the FP32 rounding band)
//                        in float-float, then FP64 (settle_pixel), or FP64 over
//                        every pixel when no list is given (used to check the
//                        other forms).
// All are persistent: the grid is sized to the resident capacity of the
// GPU; warps stride over a pixel range, or draw work-list entries from a
// cursor.
#pragma once
#include <type_traits>
#include "kernels.h"
#include "pixel.cuh"
#include "solve_tile.cuh"

namespace fpl {

template <typename T, int NP>
__global__ void k_pixels(KParams P)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int warps = blockDim.x >> 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char *sm = smem + (size_t)warp * KPixWarp<T, NP>::bytes;
    const long long gw = (long long)blockIdx.x * warps + warp;
    const long long nw = (long long)gridDim.x * warps;
    // C in tensor memory: FP64 at 64 dates (one lane quadrant per warp) and
    // FP32 at <= 32 dates (2*NP columns of the warp's quadrant per warp)
    __shared__ uint32_t tslot;
    uint32_t tbase = 0, taddr = 0;
    int tcols = 0;
    if constexpr (CInTmem<T, NP>::value) {
        tcols = 512;
        tbase = tmem_alloc_cta(&tslot, warp, tcols);
        taddr = tbase + ((uint32_t)(32 * (warp & 3)) << 16);
    } else if constexpr (CRowsTmemF<T, NP>::value) {
        tcols = tmem_cols_for(warps, NP);
        tbase = tmem_alloc_cta(&tslot, warp, (uint32_t)tcols);
        taddr = tbase + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(warp >> 2) * CRowsTmem<NP>::kColsPerWarp;
    }
    if (sizeof(T) == 4 || P.fb_list == nullptr) {
        for (long long q = gw; q < P.npix; q += nw) {
            if constexpr (sizeof(T) == 4) process_pixel<T, NP>(P, P.pix_begin + q, sm, lane, taddr);
            else fp64_pixel<NP>(P, P.pix_begin + q, sm, lane, taddr);
        }
    } else {
        int cnt = *((volatile int *)P.fb_count);
        cnt = cnt < P.fb_cap ? cnt : P.fb_cap;
        for (long long q = list_first(); q < cnt; q = fb_next(P, lane))
            settle_pixel<NP>(P, P.fb_list[q], sm, lane, taddr);
    }
    if constexpr (CInTmem<T, NP>::value || CRowsTmemF<T, NP>::value) tmem_free_cta(tbase, warp, (uint32_t)tcols);
}

// ---- eigen-solves from the Gamma records ---------------------------------
// Pixels are solved in registers by k_solve, G lanes per pixel
// (solve_tile.cuh); those it hands back, phase_link's with a bandwidth (MLE with
// STBAS's temporal coherence) and those of bandwidth 1 by k_rest, a warp per pixel with its coherence
// rows in tensor memory (pixel_solve).  Neither issues an MMA.
enum { TK_REST = 0, TK_MLE = 1, TK_EVD = 2 };
__host__ __device__ __forceinline__ int tile_kind(const KParams &P)
{
    if (P.semantics == SEM_PL) return P.method == M_STBAS ? TK_REST : TK_MLE;
    // a bandwidth of 1 makes C tridiagonal: pixel_solve's reduction is exact
    // there and keeps the phases of components that the eigenvector hardly has
    if (P.method == M_STBAS && P.bw == 1) return TK_REST;
    return P.method == M_MLE ? TK_MLE : TK_EVD;
}

template <int G, int NL> struct SolveShape {
    using M = Tile<G, NL>;
    static constexpr int PX = 32 / G;                       // pixels per warp
    static constexpr size_t bytes = PX * M::bytes;          // shared memory per warp
    static constexpr int cols = 8 * M::NB;                  // tensor-memory columns per warp
    // warps per CTA (one CTA per SM) that the registers allow: NB 8-register blocks and the working set
    static constexpr int max_warps = M::NB >= 20 ? 8 : (M::NB >= 12 ? 12 : (M::NB >= 10 ? 16 : (M::NB >= 6 ? 20 : 24)));
    static __host__ __device__ long long items(long long px) { return (px + PX - 1) / PX; }
};

// Solve kernel over a pixel source: SRC(q) gives (launch, pixel) of item q
// of [0, total); pixels of launches of another kind are left alone.
template <int G, int NL, int KIND, typename SRC>
__device__ __forceinline__ void solve_loop(long long total, const SRC &src)
{
    using SH = SolveShape<G, NL>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int warps = blockDim.x >> 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long nw = (long long)gridDim.x * warps;
    __shared__ uint32_t tslot;
    uint32_t tcols = 32;
    while ((int)tcols < (warps + 3) / 4 * SH::cols) tcols <<= 1;
    const uint32_t tbase = tmem_alloc_cta(&tslot, warp, tcols);
    const uint32_t taddr = tbase + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(warp >> 2) * (uint32_t)SH::cols;
    const int g = lane & (G - 1), h = lane / G;
    const TileLane L{g, g >> 2, g & 3,
                     (uint32_t)__cvta_generic_to_shared(smem) + (uint32_t)(warp * SH::bytes + h * Tile<G, NL>::bytes)};
    const long long items = SH::items(total);
    for (long long k0 = (long long)blockIdx.x * warps; k0 < items; k0 += nw) {
        const long long k = k0 + warp;
        // A CTA's 8 or 12 warps start their pixels together, so that they share the
        // instruction fetches of code larger than the cache (384 x 320, N = 64,
        // 12.2 -> 9.9 ms; 300 x 400, N = 45, 6.15 -> 5.30 ms).  With 16 lanes per pixel the
        // code is smaller and the wait costs more than it gives (N = 23: 1.40 -> 1.47 ms).
        if constexpr (G == 32) __syncthreads();
        if (k >= items) continue;
        const long long q0 = SH::PX * k;
        const bool in = q0 + h < total;
        long long pp;
        const KParams &P = src(in ? q0 + h : q0, pp);
        const bool valid = in && tile_kind(P) == KIND;
        if (k + nw < items && q0 + SH::PX * nw + h < total) {
            long long pn;
            const KParams &Pn = src(q0 + SH::PX * nw + h, pn);
            tile_prefetch<G>(Pn, pn, g);
        }
        if (!__any_sync(0xffffffffu, valid)) continue;
        int state;
        if constexpr (KIND == TK_MLE) state = tile_mle<G, NL>(P, pp, L, taddr, valid);
        else state = tile_evd<G, NL>(P, pp, L, taddr, valid);
        if (valid && state == TILE_GENERAL && g == 0) rest_put(P, pp);
        __syncwarp();
    }
    tmem_free_cta(tbase, warp, tcols);
}

template <int G, int NL, int KIND>
__global__ void __launch_bounds__(32 * SolveShape<G, NL>::max_warps, 1) k_solve(const __grid_constant__ KParams P)
{
    const KParams *p = &P;
    solve_loop<G, NL, KIND>(P.npix, [p](long long q, long long &pp) -> const KParams & {
        pp = p->pix_begin + q;
        return *p;
    });
}

// over many launches of one padded depth
template <int G, int NL, int KIND>
__global__ void __launch_bounds__(32 * SolveShape<G, NL>::max_warps, 1) k_solve_batch(const BatchEntry *__restrict__ ents,
                                                                                     int nent, long long total)
{
    solve_loop<G, NL, KIND>(total, [&](long long q, long long &pp) -> const KParams & {
        int lo = 0, hi = nent - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (ents[mid].px_offset <= q) lo = mid; else hi = mid - 1;
        }
        pp = ents[lo].P.pix_begin + (q - ents[lo].px_offset);
        return ents[lo].P;
    });
}

// coherence of a pixel from its samples, in FP32 (out of line: few pixels have
// samples that the records cannot hold)
template <int NP>
__device__ __noinline__ int rest_coherence(const KParams &P, long long pp, unsigned char *sm, int lane)
{
    return pixel_coherence<float, NP, RestLay<NP>, RestLay<NP>::cm>(P, pp, sm, lane);
}

// the pixels of entry P that k_solve left: every one, or those of its rest
// list.  FP32 form: a pixel with a finite sample outside the range of the bf16 parts
// has no record; its coherence is formed from the samples as the plain kernel forms it.  (1024^2,
// N = 30, every 64th row at 1e-17 of the others' amplitude: 437 ms by the FP64 list, 26.5 ms.)
template <int NP>
__device__ __forceinline__ void rest_loop(const KParams &P, unsigned char *sm, int lane, const CRowsTmem<NP> &cp)
{
    C2<float> *A = reinterpret_cast<C2<float> *>(sm + Lay<float, NP>::wm);
    const bool listed = tile_kind(P) != TK_REST;
    const long long cnt = listed ? *((volatile int *)(P.fb_count + 1)) : P.npix;
    for (long long q = list_first(); q < cnt; q = rest_next(P, lane)) {
        long long loc = q;
        bool plain;
        if (listed) {
            const int e = P.rest[q];
            plain = e < 0;
            loc = plain ? ~e : e;
        } else {
            plain = P.parts == 3 && P.cinfo[q] == CI_DEFER;
        }
        const long long pp = P.cbase + loc;
        int npix;
        float cfro = -1.f;
        bool go;
        if (plain) {
            npix = rest_coherence<NP>(P, pp, sm, lane);
            go = npix >= 0;
            if (go) rows_from_smem<NP>(cp, A, lane);
        } else if constexpr (NP <= 32) {
            npix = pixel_load_gamma<NP, false>(P, pp, sm, lane, A);
            go = npix >= 0 && rows_coherence<NP>(P, pp, A, sm, cp, lane, &cfro);
        } else {
            // two rows per lane: normalise in the slab, then copy the rows over
            npix = pixel_load_gamma<NP>(P, pp, sm, lane, A);
            go = npix >= 0;
            if (go) rows_from_smem<NP>(cp, A, lane);
        }
        if (go) pixel_solve<float, NP>(P, pp, sm, lane, npix, cp, cfro);
        __syncwarp();
    }
}

template <int NP> constexpr int rest_max_warps() { return NP <= 32 ? 20 : 5; }

template <int NP>
__global__ void __launch_bounds__(32 * rest_max_warps<NP>(), 1) k_rest(const __grid_constant__ KParams P)
{
    if (tile_kind(P) != TK_REST && *((volatile int *)(P.fb_count + 1)) == 0) return;
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ uint32_t tslot;
    const int tcols = tmem_cols_for(blockDim.x >> 5, NP);
    const uint32_t tbase = tmem_alloc_cta(&tslot, warp, tcols);
    const CRowsTmem<NP> cp{tbase + ((uint32_t)(32 * (warp & 3)) << 16) +
                           (uint32_t)(warp >> 2) * CRowsTmem<NP>::kColsPerWarp};
    rest_loop<NP>(P, smem + (size_t)warp * RestLay<NP>::bytes_noc, lane, cp);
    tmem_free_cta(tbase, warp, tcols);
}

template <int NP>
__global__ void __launch_bounds__(32 * rest_max_warps<NP>(), 1) k_rest_batch(const BatchEntry *__restrict__ ents, int nent)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ uint32_t tslot;
    const int tcols = tmem_cols_for(blockDim.x >> 5, NP);
    const uint32_t tbase = tmem_alloc_cta(&tslot, warp, tcols);
    const CRowsTmem<NP> cp{tbase + ((uint32_t)(32 * (warp & 3)) << 16) +
                           (uint32_t)(warp >> 2) * CRowsTmem<NP>::kColsPerWarp};
    for (int e = 0; e < nent; ++e) rest_loop<NP>(ents[e].P, smem + (size_t)warp * RestLay<NP>::bytes_noc, lane, cp);
    tmem_free_cta(tbase, warp, tcols);
}

// One CTA per SM for the kernels above: at least half the shared memory, so
// that a second CTA never waits on a tensor-memory allocation
constexpr size_t kSolveSmem = 224 * 1024;
template <int G, int NL> static int solve_warps()
{
    using SH = SolveShape<G, NL>;
    const int by_smem = int(kSolveSmem / SH::bytes), by_tmem = 4 * (512 / SH::cols);
    const int w = by_smem < by_tmem ? by_smem : by_tmem;
    return w < SH::max_warps ? w : SH::max_warps;
}
static size_t solve_smem(size_t per_warp, int warps) { return cmax(per_warp * warps, kSolveSmem / 2 + 1024); }

template <typename K>
static cudaError_t solve_configure(K kern, bool *configured)
{
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && configured[dev]) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSolveSmem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e != cudaSuccess) return e;
    if (dev < 64) configured[dev] = true;
    return cudaSuccess;
}

// Grid and warps per CTA for `items` warp items: a full CTA per SM, or, when
// there are fewer items than warps, as many SMs with fewer warps each
static long long solve_grid(long long items, int num_sms, int *warps)
{
    const long long per = (items + num_sms - 1) / num_sms;
    if (per < *warps) *warps = per < 1 ? 1 : (int)per;
    const long long need = (items + *warps - 1) / *warps;
    return need < num_sms ? (need > 0 ? need : 1) : num_sms;
}

template <int NP>
static cudaError_t configure_rest()
{
    static bool configured[64] = {false};
    return solve_configure(k_rest<NP>, configured);
}
template <int G, int NL, int KIND>
static cudaError_t configure_solve_kind()
{
    static bool configured[64] = {false};
    return solve_configure(k_solve<G, NL, KIND>, configured);
}

template <int NP>
static cudaError_t launch_rest_t(const KParams &P, int num_sms, cudaStream_t st)
{
    cudaError_t e = configure_rest<NP>();
    if (e != cudaSuccess) return e;
    int warps = rest_max_warps<NP>();
    const long long blocks = solve_grid(P.npix, num_sms, &warps);
    k_rest<NP><<<(unsigned)blocks, warps * 32, solve_smem(RestLay<NP>::bytes_noc, warps), st>>>(P);
    return cudaGetLastError();
}

template <int G, int NL, int KIND>
static cudaError_t launch_solve_kind(const KParams &P, int num_sms, cudaStream_t st)
{
    cudaError_t e = configure_solve_kind<G, NL, KIND>();
    if (e != cudaSuccess) return e;
    int warps = solve_warps<G, NL>();
    const long long blocks = solve_grid(SolveShape<G, NL>::items(P.npix), num_sms, &warps);
    k_solve<G, NL, KIND><<<(unsigned)blocks, warps * 32, solve_smem(SolveShape<G, NL>::bytes, warps), st>>>(P);
    return cudaGetLastError();
}

template <int G, int NL>
static cudaError_t launch_solve_t(const KParams &P, int num_sms, cudaStream_t st)
{
    constexpr int NP = G == 32 ? 64 : (NL == 2 ? 16 : 32);
    cudaError_t e = cudaSuccess;
    if (tile_kind(P) == TK_MLE) e = launch_solve_kind<G, NL, TK_MLE>(P, num_sms, st);
    else if (tile_kind(P) == TK_EVD) e = launch_solve_kind<G, NL, TK_EVD>(P, num_sms, st);
    return e != cudaSuccess ? e : launch_rest_t<NP>(P, num_sms, st);
}

template <int G, int NL>
static cudaError_t prepare_solve_t()
{
    constexpr int NP = G == 32 ? 64 : (NL == 2 ? 16 : 32);
    cudaError_t e = configure_solve_kind<G, NL, TK_MLE>();
    if (e == cudaSuccess) e = configure_solve_kind<G, NL, TK_EVD>();
    return e != cudaSuccess ? e : configure_rest<NP>();
}

// attributes of the batch kernels, set once per device
template <int G, int NL>
static cudaError_t configure_solve_batch()
{
    constexpr int NP = G == 32 ? 64 : (NL == 2 ? 16 : 32);
    static bool mle[64] = {false}, evd[64] = {false}, rest[64] = {false};
    cudaError_t e = solve_configure(k_solve_batch<G, NL, TK_MLE>, mle);
    if (e == cudaSuccess) e = solve_configure(k_solve_batch<G, NL, TK_EVD>, evd);
    return e != cudaSuccess ? e : solve_configure(k_rest_batch<NP>, rest);
}

// kinds: which kinds of pixels the entries hold (bit KIND); warps_req > 0: at
// most that many warps per CTA (the batch autotuner's candidates); 0: as many
// as fit
template <int G, int NL>
static cudaError_t launch_solve_batch_t(const BatchEntry *ents, int nent, long long total, int kinds, int num_sms,
                                       cudaStream_t st, int warps_req)
{
    constexpr int NP = G == 32 ? 64 : (NL == 2 ? 16 : 32);
    cudaError_t e = configure_solve_batch<G, NL>();
    if (e != cudaSuccess) return e;
    int warps = solve_warps<G, NL>();
    if (warps_req > 0 && warps > warps_req) warps = warps_req;
    const unsigned blocks = (unsigned)solve_grid(SolveShape<G, NL>::items(total), num_sms, &warps);
    const size_t smem = solve_smem(SolveShape<G, NL>::bytes, warps);
    if (kinds & (1 << TK_MLE)) k_solve_batch<G, NL, TK_MLE><<<blocks, warps * 32, smem, st>>>(ents, nent, total);
    if (kinds & (1 << TK_EVD)) k_solve_batch<G, NL, TK_EVD><<<blocks, warps * 32, smem, st>>>(ents, nent, total);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    int rw = rest_max_warps<NP>();
    const long long rb = solve_grid(total, num_sms, &rw);
    k_rest_batch<NP><<<(unsigned)rb, rw * 32, solve_smem(RestLay<NP>::bytes_noc, rw), st>>>(ents, nent);
    return cudaGetLastError();
}

template <typename T, int NP>
static cudaError_t launch_t(const KParams &P, int num_sms, cudaStream_t st)
{
    static bool configured[64] = {false};
    const size_t per_warp = KPixWarp<T, NP>::bytes;
    const size_t budget = 224 * 1024;   // of the 227 KB a block may opt into
    int warps = int(budget / per_warp);
    if (warps > 16) warps = 16;
    if (CInTmem<T, NP>::value && warps > 4) warps = 4;   // one tensor-memory lane quadrant per warp
    // and no more threads than the kernel's registers allow in one CTA
    static int max_threads[64] = {0};
    {
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev < 64 && !max_threads[dev]) {
            cudaFuncAttributes fa;
            cudaError_t e = cudaFuncGetAttributes(&fa, k_pixels<T, NP>);
            if (e != cudaSuccess) return e;
            max_threads[dev] = fa.maxThreadsPerBlock;
        }
        const int lim = (dev < 64 ? max_threads[dev] : 1024) / 32;
        if (warps > lim) warps = lim;
    }
    if (warps < 1) warps = 1;
    size_t smem = per_warp * warps;
    // tensor-memory rows: one CTA per SM (at least half the shared memory),
    // so a second CTA never waits on a tensor-memory allocation
    constexpr bool one_cta = CInTmem<T, NP>::value || CRowsTmemF<T, NP>::value;
    if (one_cta && smem < budget / 2 + 1024) smem = budget / 2 + 1024;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_pixels<T, NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        e = cudaFuncSetAttribute(k_pixels<T, NP>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pixels<T, NP>, warps * 32, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1 || one_cta) per_sm = 1;
    long long work = P.npix;
    long long blocks = (long long)num_sms * per_sm;
    long long need = (work + warps - 1) / warps;
    if (sizeof(T) == 4 && need < blocks) blocks = need > 0 ? need : 1;
    k_pixels<T, NP><<<(unsigned)blocks, warps * 32, smem, st>>>(P);
    return cudaGetLastError();
}

}  // namespace fpl
