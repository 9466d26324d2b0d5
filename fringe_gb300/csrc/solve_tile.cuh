// solve_tile.cuh -- MLE eigen-solve with the matrices in registers (FP32):
// two pixels per warp up to 32 dates, one up to 64.
//
// The solver is three factorisations per pixel -- the Cholesky test of C, the
// inverse of |C|, the factorisation of M - sigma I -- and three or four pairs of
// triangular solves.  With a row per lane and the matrix in shared memory
// (pixel_solve) every matrix entry costs a shared load and a store per
// elimination step, the lanes of finished rows idle, and shared memory holds
// few warps (18.9 k warp instructions per pixel at 30 dates; 5 warps per SM at 64).
// Here G = 16 (32) lanes own a pixel's matrix as a G/4 x 4 block-cyclic grid of 2 x 2
// blocks: dates are paired, and lane (lr, lc) of the grid holds the blocks of row
// pairs m = (G/4) mi + lr and column pairs l = 4 li + lc that the lower triangle
// needs, li < RT (mi + 1) with RT = G/16.  Blocks with li < RT mi lie below the
// diagonal for every lane; the others (diagonal-level) also hold entries above it.
// An elimination step publishes one column through shared memory (the lanes
// that hold it), and every lane reads the entries of its rows and columns: a
// few 16-byte loads for up to 80 (160) packed multiply-adds (fma.rn.f32x2,
// which issue once for two).  Finished rows and columns drop out of the unrolled code
// four pairs at a time.  With G = 16 two pixels share every instruction, so the
// fixed cost of a step (pivot, reciprocal, addresses, barrier) is paid half as often.
//
// A 2 x 2 block (rows i, i'; columns j, j') is held as two diagonal pairs,
// D = (a_ij, a_i'j') and E = (a_i'j, a_ij'), real and imaginary parts apart, so
// that a rank-1 update multiplies the row pair, straight or swapped, with the
// column pair entry by entry.
//
// This path takes the common case to its end (phases, compressed SLC,
// temporal coherence).  Where a decision is not settled on first sight -- C
// within the band of the 1e-6 test, |C| not positive definite, a shift above
// lambda_1, slow convergence -- the pixel goes on a list for pixel_solve, which decides
// as it always did.  Solve kernels on GB300: 2048^2, N = 30, 11 x 21, 91.9 ->
// 47.2 ms; 384 x 320, N = 64, ill-conditioned, 37.7 -> 9.0 ms; 333 x 517, N = 23,
// 2.77 -> 1.21 ms; 1023 x 777, N = 15, 4.29 -> 2.95 ms.  The FMA pipe bounds it (a
// packed multiply-add holds it for 2.3 clocks), then instruction fetch: swaps and signs
// are therefore moves and bit operations, not products (1024^2, N = 30, 13.75 -> 12.7 ms).
// Tried and slower: one copy of an elimination or sweep step's code for both columns of a
// pair, or of the sweep for all pivots (its branches cost more than the fetches: 8 to 15%).
#pragma once
#include "f32x2.cuh"
#include "pixel.cuh"

namespace fpl {
// internal linkage: the header is compiled into more than one unit
namespace {

__device__ __forceinline__ float rcp_fast(float a)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

// rsqrtf of a normal number (the same result without its steps for subnormal ones)
__device__ __forceinline__ float rsqrt_fast(float a)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

// shared memory by 32-bit address (volatile: ordered with the barriers)
__device__ __forceinline__ float lds1(uint32_t a)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ f32x2 lds2(uint32_t a)
{
    f32x2 v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void lds4(uint32_t a, f32x2 &x, f32x2 &y)
{
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(a));
}
__device__ __forceinline__ void sts1(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" :: "r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void sts2(uint32_t a, float x, float y)
{
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" :: "r"(a), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void sts4(uint32_t a, float x, float y, float z, float w)
{
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" :: "r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

// 8 consecutive 32-bit TMEM columns of each lane
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

// one 2 x 2 complex block (see the file comment) and one real one
struct CBlk { f32x2 dr, di, er, ei; };
struct RBlk { f32x2 d, e; };

// The grid of G lanes with NL row blocks (2 G NL / 4 dates at most)
template <int G, int NL> struct Tile {
    static constexpr int LRN = G / 4, RT = LRN / 4;        // grid rows; column blocks per row block
    static constexpr int T = LRN * NL;                     // date pairs
    static constexpr int NLC = RT * NL;                    // column blocks
    static constexpr int NB = RT * NL * (NL + 1) / 2;      // blocks per lane
    static __host__ __device__ constexpr int blk(int mi, int li) { return RT * mi * (mi + 1) / 2 + li; }
    // Shared memory of one pixel.  W: the published columns of a factorisation,
    // 16 bytes (re_i, re_i', im_i, im_i') per row pair.  Column 2 t + par keeps row
    // pairs m >= t; columns t and TW - 1 - t share a slot of TW + 1 entries (t < TW / 2:
    // entry m; else entry TW - 1 - m, its pair's own at TW).  The odd slot length
    // lets the forward solve (one column, consecutive rows) and the backward
    // solve (one row, consecutive columns) both read without bank conflicts.
    static constexpr int TW = NL == 3 ? 4 * LRN : T;       // slots are split at a whole segment
    static constexpr uint32_t PAR = 16u * (TW / 2) * (TW + 1);
    static constexpr uint32_t dg = 2 * PAR;                // per pair: 1/d_0, 1/d_1, l_10 d_0 (re, im)
    static constexpr uint32_t z = dg + 16 * T;             // vector, 16 bytes per pair as in W
    static constexpr uint32_t v = z + 16 * T;              // sweep columns (two), pivots; 1/sqrt(P)
    static constexpr uint32_t bytes = v + 2 * 8 * T + 16;
    static_assert(bytes % 16 == 0, "16-byte vectors");
};

// lane's place in the grid
struct TileLane {
    int g, lr, lc;     // lane of the group, grid row and column
    uint32_t mem;      // the pixel's shared memory
};

template <int G> __device__ __forceinline__ float gsum(float v)
{
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <int G> __device__ __forceinline__ float gmax(float v)
{
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ f32x2 shflx2(f32x2 a, int o)
{
    return pk(__shfl_xor_sync(0xffffffffu, lo2(a), o), __shfl_xor_sync(0xffffffffu, hi2(a), o));
}

// One elimination step of the LDL^H factorisation: pivot k = 2 t + PAR, t =
// 4 S + tl.  Publishes column k, then a_ij -= v_i conj(v_j) / p for the
// trailing blocks.  ok &= (p > 0): the LDL^H pivots are the Cholesky ones squared.
template <int G, int NL, int S, int PAR>
__device__ __forceinline__ void tile_ldl_step(CBlk (&A)[Tile<G, NL>::NB], const TileLane &L, int tl, bool &ok)
{
    using M = Tile<G, NL>;
    constexpr int TW = M::TW, RT = M::RT, LRN = M::LRN, NLC = M::NLC;
    constexpr int MS = S / RT;                             // row block of the pivot pair
    constexpr bool LOW = 4 * S < TW / 2;
    const int t = 4 * S + tl, tr = t - LRN * MS;           // pivot pair; its grid row
    const uint32_t sb = L.mem + PAR * M::PAR + 16u * (uint32_t)((LOW ? t : TW - 1 - t) * (TW + 1));
    const uint32_t diag = sb + 16u * (LOW ? t : TW);
    auto at = [&](int pair) { return sb + 16u * (uint32_t)(LOW ? pair : TW - 1 - pair); };
    if (L.lc == tl) {
#pragma unroll
        for (int mi = MS; mi < NL; ++mi) {
            const CBlk &b = A[M::blk(mi, S)];
            const uint32_t a = (!LOW && mi == MS && L.lr == tr) ? diag : at(LRN * mi + L.lr);
            if (mi > MS || L.lr >= tr) {
                if (PAR == 0) sts4(a, lo2(b.dr), lo2(b.er), lo2(b.di), lo2(b.ei));
                else sts4(a, hi2(b.er), hi2(b.dr), hi2(b.ei), hi2(b.di));
            }
        }
    }
    __syncwarp();
    const float p = lds1(diag + 4 * PAR);
    ok = ok && p > 0.f;
    const float r = rcp_fast(p), nr = -r;
    if (L.lr == tr && L.lc == tl) {
        const uint32_t d = L.mem + M::dg + 16u * (uint32_t)t;
        sts1(d + 4 * PAR, r);
        if (PAR == 0) sts2(d + 8, lo2(A[M::blk(MS, S)].er), lo2(A[M::blk(MS, S)].ei));
    }
    f32x2 cr[NLC - S], ci[NLC - S];
#pragma unroll
    for (int li = S; li < NLC; ++li)
        lds4((!LOW && li == S && L.lc == tl) ? diag : at(4 * li + L.lc), cr[li - S], ci[li - S]);
    const f32x2 nr2 = pk(nr, nr);
    f32x2 nci[NLC - S];
#pragma unroll
    for (int li = S; li < NLC; ++li) nci[li - S] = ci[li - S] ^ 0x8000000080000000ull;
#pragma unroll
    for (int mi = MS; mi < NL; ++mi) {
        f32x2 vr, vi;
        lds4((!LOW && mi == MS && L.lr == tr) ? diag : at(LRN * mi + L.lr), vr, vi);
        const f32x2 sr = mul2(vr, nr2), si = mul2(vi, nr2);
        const f32x2 srs = swap2(sr), sis = swap2(si);
#pragma unroll
        for (int li = S; li < RT * (mi + 1); ++li) {
            CBlk &b = A[M::blk(mi, li)];
            b.dr = fma2(si, ci[li - S], fma2(sr, cr[li - S], b.dr));
            b.di = fma2(sr, nci[li - S], fma2(si, cr[li - S], b.di));
            b.er = fma2(sis, ci[li - S], fma2(srs, cr[li - S], b.er));
            b.ei = fma2(srs, nci[li - S], fma2(sis, cr[li - S], b.ei));
        }
    }
}

template <int G, int NL, int S>
__device__ __forceinline__ void tile_ldl_seg(CBlk (&A)[Tile<G, NL>::NB], const TileLane &L, int tp, bool &ok)
{
    if constexpr (S < Tile<G, NL>::NLC) {
#pragma unroll 1
        for (int tl = 0; tl < 4; ++tl) {
            if (4 * S + tl >= tp) break;
            tile_ldl_step<G, NL, S, 0>(A, L, tl, ok);
            tile_ldl_step<G, NL, S, 1>(A, L, tl, ok);
        }
        tile_ldl_seg<G, NL, S + 1>(A, L, tp, ok);
    }
}

// One step of the symmetric sweep (Gauss-Jordan) of the real matrix in K,
// pivot k = 2 t + PAR: a_ij -= v_i v_j / p for all i, j with v_k replaced by p - 1,
// which turns row and column k into a_ik / p and a_kk into 2 - 1/p (the 2 is taken
// off at the end).  v comes from column k (pairs of the pivot's row block and
// below) and from row k (pairs before it).
template <int G, int NL, int S, int PAR>
__device__ __forceinline__ void tile_sweep_step(RBlk (&K)[Tile<G, NL>::NB], const TileLane &L, int tl, bool &ok)
{
    using M = Tile<G, NL>;
    constexpr int T = M::T, RT = M::RT, LRN = M::LRN, NLC = M::NLC, MS = S / RT;
    const int tr = 4 * S + tl - LRN * MS;
    const uint32_t vb = L.mem + M::v + 8u * T * PAR, pslot = L.mem + M::v + 16u * T + 4u * PAR;
    if (L.lc == tl) {
        const bool own = L.lr == tr;
#pragma unroll
        for (int mi = MS; mi < NL; ++mi) {
            const RBlk &b = K[M::blk(mi, S)];
            float x = PAR == 0 ? lo2(b.d) : hi2(b.e), y = PAR == 0 ? lo2(b.e) : hi2(b.d);
            if (mi == MS && own) {
                sts1(pslot, PAR == 0 ? x : y);
                if (PAR == 0) x -= 1.f;
                else y -= 1.f;
            }
            sts2(vb + 8u * (uint32_t)(LRN * mi + L.lr), x, y);
        }
    }
    if (MS > 0 && L.lr == tr) {
#pragma unroll
        for (int li = 0; li < RT * MS; ++li) {
            const RBlk &b = K[M::blk(MS, li)];
            sts2(vb + 8u * (uint32_t)(4 * li + L.lc), PAR == 0 ? lo2(b.d) : lo2(b.e), PAR == 0 ? hi2(b.e) : hi2(b.d));
        }
    }
    __syncwarp();
    const float p = lds1(pslot);
    ok = ok && p > 0.f;
    const float nr = -rcp_fast(p);
    f32x2 c[NLC];
#pragma unroll
    for (int li = 0; li < NLC; ++li) c[li] = lds2(vb + 8u * (uint32_t)(4 * li + L.lc));
#pragma unroll
    for (int mi = 0; mi < NL; ++mi) {
        const f32x2 v = lds2(vb + 8u * (uint32_t)(LRN * mi + L.lr));
        const f32x2 s = mul2(v, pk(nr, nr)), ss = swap2(s);
#pragma unroll
        for (int li = 0; li < RT * (mi + 1); ++li) {
            RBlk &b = K[M::blk(mi, li)];
            b.d = fma2(s, c[li], b.d);
            b.e = fma2(ss, c[li], b.e);
        }
    }
}

template <int G, int NL, int S>
__device__ __forceinline__ void tile_sweep_seg(RBlk (&K)[Tile<G, NL>::NB], const TileLane &L, int tp, bool &ok)
{
    if constexpr (S < Tile<G, NL>::NLC) {
#pragma unroll 1
        for (int tl = 0; tl < 4; ++tl) {
            if (4 * S + tl >= tp) break;
            tile_sweep_step<G, NL, S, 0>(K, L, tl, ok);
            tile_sweep_step<G, NL, S, 1>(K, L, tl, ok);
        }
        tile_sweep_seg<G, NL, S + 1>(K, L, tp, ok);
    }
}

// Sums over matrix rows: rows[x] holds the lane's sums over its blocks of row
// pair LRN x + lr, cols[x] those over the columns of its below-diagonal blocks of
// column pair 4 x + lc, which are the mirrored blocks' rows.  On return the diagonal
// lanes (lc = lr mod 4) hold the full sums of row pair LRN x + lr in rows[x].
template <int G, int NL>
__device__ __forceinline__ void tile_row_sums(f32x2 (&rows)[NL], f32x2 (&cols)[Tile<G, NL>::NLC], const TileLane &L)
{
    constexpr int RT = Tile<G, NL>::RT;
#pragma unroll
    for (int x = 0; x < NL; ++x) {
        rows[x] = add2(rows[x], shflx2(rows[x], 1));
        rows[x] = add2(rows[x], shflx2(rows[x], 2));
        if (x + 1 < NL) {
#pragma unroll
            for (int h = 0; h < RT; ++h) {
#pragma unroll
                for (int o = 4; o < G; o <<= 1) cols[RT * x + h] = add2(cols[RT * x + h], shflx2(cols[RT * x + h], o));
            }
            rows[x] = add2(rows[x], (RT == 2 && L.lr >= 4) ? cols[RT * x + RT - 1] : cols[RT * x]);
        }
    }
}

// inf-norm of the symmetric matrix in K (absolute row sums)
template <int G, int NL>
__device__ __forceinline__ float tile_inf_norm(const RBlk (&K)[Tile<G, NL>::NB], const TileLane &L)
{
    using M = Tile<G, NL>;
    f32x2 rows[NL], cols[M::NLC];
    auto abs2 = [](f32x2 a) { return a & 0x7fffffff7fffffffull; };
#pragma unroll
    for (int x = 0; x < NL; ++x) rows[x] = 0ull;
#pragma unroll
    for (int x = 0; x < M::NLC; ++x) cols[x] = 0ull;
#pragma unroll
    for (int mi = 0; mi < NL; ++mi)
#pragma unroll
        for (int li = 0; li < M::RT * (mi + 1); ++li) {
            // D = (ij, i'j'), E = (i'j, ij'): rows (ij + ij', i'j + i'j'), columns (ij + i'j, ij' + i'j')
            const RBlk &b = K[M::blk(mi, li)];
            const f32x2 d = abs2(b.d), e = abs2(b.e);
            rows[mi] = add2(rows[mi], add2(d, swap2(e)));
            if (li < M::RT * mi) cols[li] = add2(cols[li], add2(d, e));
        }
    tile_row_sums<G, NL>(rows, cols, L);
    float mx = 0.f;
    if ((L.lr & 3) == L.lc) {
#pragma unroll
        for (int x = 0; x < NL; ++x) mx = fmaxf(mx, fmaxf(lo2(rows[x]), hi2(rows[x])));
    }
    return gmax<G>(mx);
}

// (L D L^H) x = b with the factor of tile_ldl (columns v = l d in W): lane g of the
// group holds the pair b = rows 2 g, 2 g + 1 in (re, re', im, im').  Every lane takes
// its own pair's 2 x 2 step each time, which is the step's result on lane t, and the
// others take that by shuffle: the pair's factor stays in registers and no lane
// has to keep its result from later steps.  1023 x 777, N = 15: 3.18 -> 2.99 ms;
// N = 64: 9.7 -> 9.1 ms; STBAS 256 x 384, N = 45: 4.90 -> 4.47 ms.
template <int G, int NL>
__device__ __forceinline__ void tile_solve(const TileLane &L, int tp, float &b0r, float &b1r, float &b0i, float &b1i)
{
    using M = Tile<G, NL>;
    constexpr int TW = M::TW;
    const int m = L.g;
    f32x2 rm, vm;
    lds4(L.mem + M::dg + 16u * (uint32_t)(m < tp ? m : 0), rm, vm);
    const float r0 = lo2(rm), r1 = hi2(rm), vr = lo2(vm), vi = hi2(vm);
    float s0r, s0i, s1r, s1i, y1r, y1i;
    auto pair_fwd = [&]() {
        s0r = r0 * b0r;
        s0i = r0 * b0i;
        y1r = fmaf(vi, s0i, fmaf(-vr, s0r, b1r));
        y1i = fmaf(-vi, s0r, fmaf(-vr, s0i, b1i));
        s1r = r1 * y1r;
        s1i = r1 * y1i;
    };
    // forward: y_i -= v_ik y_k / d_k
    auto fwd = [&](int t, uint32_t a) {
        pair_fwd();
        const float p0r = __shfl_sync(0xffffffffu, s0r, t, G), p0i = __shfl_sync(0xffffffffu, s0i, t, G);
        const float p1r = __shfl_sync(0xffffffffu, s1r, t, G), p1i = __shfl_sync(0xffffffffu, s1i, t, G);
        if (m > t && (M::T == G || m < M::T)) {
            f32x2 ar, ai, cr, ci;
            lds4(a, ar, ai);
            lds4(a + M::PAR, cr, ci);
            b0r = fmaf(lo2(ai), p0i, fmaf(-lo2(ar), p0r, b0r));
            b1r = fmaf(hi2(ai), p0i, fmaf(-hi2(ar), p0r, b1r));
            b0i = fmaf(-lo2(ai), p0r, fmaf(-lo2(ar), p0i, b0i));
            b1i = fmaf(-hi2(ai), p0r, fmaf(-hi2(ar), p0i, b1i));
            b0r = fmaf(lo2(ci), p1i, fmaf(-lo2(cr), p1r, b0r));
            b1r = fmaf(hi2(ci), p1i, fmaf(-hi2(cr), p1r, b1r));
            b0i = fmaf(-lo2(ci), p1r, fmaf(-lo2(cr), p1i, b0i));
            b1i = fmaf(-hi2(ci), p1r, fmaf(-hi2(cr), p1i, b1i));
        }
    };
    int t = 0;
    uint32_t a = L.mem + 16u * (uint32_t)m;
#pragma unroll 1
    for (; t < min(tp, TW / 2); ++t, a += 16u * (TW + 1)) fwd(t, a);
    a = L.mem + 16u * (uint32_t)((TW / 2 - 1) * (TW + 1) + TW - 1 - m);
#pragma unroll 1
    for (; t < tp; ++t, a -= 16u * (TW + 1)) fwd(t, a);
    pair_fwd();
    b1r = y1r;
    b1i = y1i;
    // backward: x_k = (y_k - sum_{j > k} conj(v_jk) x_j) / d_k, y kept undivided
    float x0r, x0i, x1r, x1i;
    auto pair_bwd = [&]() {
        x1r = r1 * b1r;
        x1i = r1 * b1i;
        x0r = r0 * fmaf(-vi, x1i, fmaf(-vr, x1r, b0r));      // - conj(v10) x1
        x0i = r0 * fmaf(vi, x1r, fmaf(-vr, x1i, b0i));
    };
    const bool mlow = m < TW / 2;
    const uint32_t step = mlow ? 16u : (uint32_t)-16;
    a = L.mem + 16u * (uint32_t)((mlow ? m : TW - 1 - m) * (TW + 1) + (mlow ? 0 : TW - 1)) + step * (uint32_t)(tp - 1);
#pragma unroll 1
    for (t = tp - 1; t >= 0; --t, a -= step) {
        pair_bwd();
        const float p0r = __shfl_sync(0xffffffffu, x0r, t, G), p0i = __shfl_sync(0xffffffffu, x0i, t, G);
        const float p1r = __shfl_sync(0xffffffffu, x1r, t, G), p1i = __shfl_sync(0xffffffffu, x1i, t, G);
        if (m < t) {
            // columns 2 m and 2 m + 1 at row pair t
            f32x2 ar, ai, cr, ci;
            lds4(a, ar, ai);
            lds4(a + M::PAR, cr, ci);
            b0r = fmaf(-lo2(ai), p0i, fmaf(-lo2(ar), p0r, b0r));
            b0i = fmaf(lo2(ai), p0r, fmaf(-lo2(ar), p0i, b0i));
            b0r = fmaf(-hi2(ai), p1i, fmaf(-hi2(ar), p1r, b0r));
            b0i = fmaf(hi2(ai), p1r, fmaf(-hi2(ar), p1i, b0i));
            b1r = fmaf(-lo2(ci), p0i, fmaf(-lo2(cr), p0r, b1r));
            b1i = fmaf(lo2(ci), p0r, fmaf(-lo2(cr), p0i, b1i));
            b1r = fmaf(-hi2(ci), p1i, fmaf(-hi2(cr), p1r, b1r));
            b1i = fmaf(hi2(ci), p1r, fmaf(-hi2(cr), p1i, b1i));
        }
    }
    pair_bwd();
    const bool in = m < tp;
    b0r = in ? x0r : 0.f;
    b0i = in ? x0i : 0.f;
    b1r = in ? x1r : 0.f;
    b1i = in ? x1i : 0.f;
}

// outcome of a group's pixel
enum { TILE_RUN = 0, TILE_DONE = 1, TILE_GENERAL = 2 };

// zero outputs of a pixel that gets no phases
template <int G> __device__ __forceinline__ void tile_zero(const KParams &P, long long pp, int g)
{
    for (int b = g; b < P.nb; b += G) P.phase[b * P.plane + pp] = make_float2(0.f, 0.f);
    if (g == 0) {
        P.tcorr[pp] = 0.f;
        P.comp[pp] = make_float2(0.f, 0.f);
    }
}

// f(x, block index) on the lanes that hold diagonal blocks: (x, RT x + lr / 4)
template <int G, int NL, typename F> __device__ __forceinline__ void tile_on_diag(const TileLane &L, F &&f)
{
    using M = Tile<G, NL>;
#pragma unroll
    for (int x = 0; x < NL; ++x)
#pragma unroll
        for (int h = 0; h < M::RT; ++h)
            if ((L.lr & 3) == L.lc && (L.lr >> 2) == h) f(x, M::blk(x, M::RT * x + h));
}

// Record to coherence (in A and in tensor memory at taddr) and the start
// vector, C 1 normalised (in z).  MLE: the pixel's method is; else EVD or STBAS
// (whose C is banded).  Returns the outcome so far; cfro = |C|_F.
template <int G, int NL, bool MLE>
__device__ __forceinline__ int tile_begin(const KParams &P, long long pp, const TileLane &L, uint32_t taddr, bool valid,
                                          CBlk (&A)[Tile<G, NL>::NB], float &cfro)
{
    using M = Tile<G, NL>;
    constexpr int RT = M::RT, LRN = M::LRN, NLC = M::NLC;
    const int n = P.nb, dp = (n + 1) >> 1;
    const bool plink = P.semantics == SEM_PL;
    const bool dlane = (L.lr & 3) == L.lc;
    const int dh = L.lr >> 2;
    int state = valid ? TILE_RUN : TILE_DONE;
    int npix = 0;

    // ---- record --------------------------------------------------------------
    if (valid) {
        const long long loc = pp - P.cbase;
        const int info = P.cinfo[loc];
        if (info < 0) {
            tile_zero<G>(P, pp, L.g);
            if (info == CI_DEFER) {
                if (P.parts == 2) defer_fp64(P, pp, L.g, true);
                else if (L.g == 0) rest_put(P, pp, true);
            }
            else if (info == CI_BAD) put_code(P, pp, L.g, MLE ? -1 : -6);
            else if (P.status && L.g == 0) P.status[pp] = (info == CI_CENTRE) ? 1 : 2;
            state = TILE_DONE;
        }
        npix = info;
    }
    {
        const float4 *rec =
            reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(P.cbuf) + (valid ? pp - P.cbase : 0) * (long long)P.cstride);
        const bool rd = state == TILE_RUN;
#pragma unroll
        for (int mi = 0; mi < NL; ++mi)
#pragma unroll
            for (int li = 0; li < RT * (mi + 1); ++li) {
                const int m = LRN * mi + L.lr, l = 4 * li + L.lc;
                const bool low = li < RT * mi || m > l;
                const int a = low ? l : m, b = low ? m : l;
                float4 u = make_float4(0.f, 0.f, 0.f, 0.f), w = u;
                if (rd && b < dp) {
                    const int t = a * dp - a * (a - 1) / 2 + b - a;
                    u = __ldg(rec + 2 * t);
                    w = __ldg(rec + 2 * t + 1);
                }
                // record: (a0,b0) u.xy, (a0,b1) u.zw, (a1,b0) w.xy, (a1,b1) w.zw; lower blocks are its conjugate transpose
                CBlk &k = A[M::blk(mi, li)];
                k.dr = pk(u.x, w.z);
                k.di = low ? pk(-u.y, -w.w) : pk(u.y, w.w);
                k.er = low ? pk(u.z, w.x) : pk(w.x, u.z);
                k.ei = low ? pk(-u.w, -w.y) : pk(w.y, u.w);
            }
    }
    // ---- coherence (evd.cpp:566-582) --------------------------------------------
    bool bad = false;
    const uint32_t yv = L.mem + M::v;
    tile_on_diag<G, NL>(L, [&](int x, int b) {
        sts2(yv + 8u * (uint32_t)(LRN * x + L.lr), lo2(A[b].dr), hi2(A[b].dr));
    });
    __syncwarp();
    // 1/sqrt(P), a pair per lane: on the diagonal lanes it is NL times the code and the
    // work (N = 15: 3.00 -> 2.95 ms with rsqrt_fast in |C|, N = 23: 1.25 -> 1.21 ms)
    if (L.g < M::T) {
        const int i = 2 * L.g;
        const f32x2 p = lds2(yv + 8u * (uint32_t)L.g);
        const float p0 = lo2(p), p1 = hi2(p);
        bad |= i < n && (!(p0 > 0.f) || !isfinite(p0));
        bad |= i + 1 < n && (!(p1 > 0.f) || !isfinite(p1));
        sts2(yv + 8u * (uint32_t)L.g, i < n ? 1.f / sqrtf(p0) : 0.f, i + 1 < n ? 1.f / sqrtf(p1) : 0.f);
    }
    __syncwarp();
    float fs = 0.f;
    {
        f32x2 yc[NLC];
#pragma unroll
        for (int li = 0; li < NLC; ++li) yc[li] = lds2(yv + 8u * (uint32_t)(4 * li + L.lc));
        f32x2 f2 = 0ull, f1 = 0ull;
#pragma unroll
        for (int mi = 0; mi < NL; ++mi) {
            const f32x2 yr = lds2(yv + 8u * (uint32_t)(LRN * mi + L.lr)), ys = swap2(yr);
#pragma unroll
            for (int li = 0; li < RT * (mi + 1); ++li) {
                CBlk &k = A[M::blk(mi, li)];
                const f32x2 d = mul2(yr, yc[li]), e = mul2(ys, yc[li]);
                k.dr = mul2(k.dr, d);
                k.di = mul2(k.di, d);
                k.er = mul2(k.er, e);
                k.ei = mul2(k.ei, e);
                if (!MLE && P.method == M_STBAS) {               // evd.cpp:695-706
                    const int d = 2 * (LRN * mi + L.lr - 4 * li - L.lc), bw = P.bw;     // i - j
                    if (abs(d) > bw) k.dr = k.di = 0ull;
                    const f32x2 m = pk(abs(d + 1) > bw ? 0.f : 1.f, abs(d - 1) > bw ? 0.f : 1.f);
                    k.er = mul2(k.er, m);
                    k.ei = mul2(k.ei, m);
                }
                const bool dg = li >= RT * mi && dlane && dh == li - RT * mi;
                if (dg) {                                        // unit diagonal
                    const int i = 2 * (LRN * mi + L.lr);
                    k.dr = pk(i < n ? 1.f : 0.f, i + 1 < n ? 1.f : 0.f);
                    k.di = 0ull;
                }
                const f32x2 q = fma2(k.dr, k.dr, fma2(k.di, k.di, fma2(k.er, k.er, mul2(k.ei, k.ei))));
                if (li < RT * mi) f2 = add2(f2, q);
                else f1 = add2(f1, q);
                if (dg) k.dr = pk(1.f, 1.f);                     // the padding's too
            }
        }
        fs = gsum<G>(2.f * (lo2(f2) + hi2(f2)) + (lo2(f1) + hi2(f1)));
    }
    // any non-finite entry makes the sum non-finite: the first eigen call is reported as failed
    bad = bad || !isfinite(fs);
    {
        const unsigned any = __ballot_sync(0xffffffffu, bad);
        bad = (G == 16 ? (any >> (threadIdx.x & 16)) & 0xffffu : any) != 0;
    }
    if (state == TILE_RUN && bad) {
        tile_zero<G>(P, pp, L.g);
        put_code(P, pp, L.g, MLE ? -1 : -6);
        state = TILE_DONE;
    }
    if (MLE && state == TILE_RUN && !plink && npix < n) {
        // fewer SHPs than dates: rank-deficient (see pixel_solve)
        tile_zero<G>(P, pp, L.g);
        put_code(P, pp, L.g, -2);
        state = TILE_DONE;
    }
    if (!__any_sync(0xffffffffu, state == TILE_RUN)) return state;
    cfro = sqrtf(fs);

    // ---- C to tensor memory; start vector C 1, normalised (rows of C) -------------
    {
        f32x2 rr[NL], ri[NL], cr[NLC], ci[NLC];
#pragma unroll
        for (int x = 0; x < NL; ++x) rr[x] = ri[x] = 0ull;
#pragma unroll
        for (int x = 0; x < NLC; ++x) cr[x] = ci[x] = 0ull;
        const f32x2 minus = pk(-1.f, -1.f);
#pragma unroll
        for (int mi = 0; mi < NL; ++mi)
#pragma unroll
            for (int li = 0; li < RT * (mi + 1); ++li) {
                const CBlk &k = A[M::blk(mi, li)];
                const uint32_t w[8] = {__float_as_uint(lo2(k.dr)), __float_as_uint(hi2(k.dr)), __float_as_uint(lo2(k.di)),
                                       __float_as_uint(hi2(k.di)), __float_as_uint(lo2(k.er)), __float_as_uint(hi2(k.er)),
                                       __float_as_uint(lo2(k.ei)), __float_as_uint(hi2(k.ei))};
                tmem_st8(taddr + 8u * (uint32_t)M::blk(mi, li), w);
                rr[mi] = add2(rr[mi], add2(k.dr, swap2(k.er)));
                ri[mi] = add2(ri[mi], add2(k.di, swap2(k.ei)));
                if (li < RT * mi) {                              // the mirrored block: conjugate
                    cr[li] = add2(cr[li], add2(k.dr, k.er));
                    ci[li] = fma2(add2(k.di, k.ei), minus, ci[li]);
                }
            }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tile_row_sums<G, NL>(rr, cr, L);
        tile_row_sums<G, NL>(ri, ci, L);
        float un = 0.f;
        if (dlane) {
#pragma unroll
            for (int x = 0; x < NL; ++x) {
                const int i = 2 * (LRN * x + L.lr);
                // the padding's rows hold its unit diagonal alone
                const f32x2 on = pk(i < n ? 1.f : 0.f, i + 1 < n ? 1.f : 0.f);
                rr[x] = mul2(rr[x], on);
                ri[x] = mul2(ri[x], on);
                const f32x2 q = fma2(rr[x], rr[x], mul2(ri[x], ri[x]));
                un += lo2(q) + hi2(q);
            }
        }
        const float inv = rsqrtf(gsum<G>(un));
        if (dlane) {
#pragma unroll
            for (int x = 0; x < NL; ++x)
                sts4(L.mem + M::z + 16u * (uint32_t)(LRN * x + L.lr), inv * lo2(rr[x]), inv * hi2(rr[x]), inv * lo2(ri[x]),
                     inv * hi2(ri[x]));
        }
    }
    __syncwarp();
    return state;
}

// the pixel's own samples of dates 2 g, 2 g + 1 (from the reference date on),
// loaded ahead of the iteration that they are needed after
__device__ __forceinline__ void tile_own(const KParams &P, long long pp, const TileLane &L, bool go, float2 (&own)[2])
{
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = 2 * L.g + h;
        own[h] = make_float2(0.f, 0.f);
        if (go && i < P.nb && i >= P.mini - 1) own[h] = __ldg(P.stack + i * P.plane + pp);
    }
}

// Phases, compressed SLC and temporal coherence of the eigenvector z (pair
// 2 g, 2 g + 1 on lane g) where fin; stbas: only pairs within the bandwidth
// count in the temporal coherence.  Every lane calls it.
template <int G, int NL>
__device__ __forceinline__ void tile_finish(const KParams &P, long long pp, const TileLane &L, uint32_t taddr, bool fin,
                                            bool stbas, float z0r, float z1r, float z0i, float z1i, const float2 (&own)[2])
{
    using M = Tile<G, NL>;
    constexpr int RT = M::RT, LRN = M::LRN;
    const int n = P.nb;
    // ---- phase referencing (evd.cpp:738-749) -----------------------------------------
    const int mref = P.mini - 1;
    float ur, ui;
    {
        const float er = (mref & 1) ? z1r : z0r, ei = (mref & 1) ? z1i : z0i;
        const float wr = __shfl_sync(0xffffffffu, er, mref >> 1, G), wi = __shfl_sync(0xffffffffu, ei, mref >> 1, G);
        const float w2 = fmaf(wr, wr, wi * wi), k = rsqrtf(w2);
        ur = w2 > 0.f ? wr * k : 1.f;
        ui = w2 > 0.f ? wi * k : 0.f;
    }
    float2 o[2];
    float cr = 0.f, ci = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = 2 * L.g + h;
        const float a = h ? z1r : z0r, b = h ? z1i : z0i;
        const float w2 = fmaf(a, a, b * b), k = rsqrtf(w2);
        const float er = w2 > 0.f ? a * k : 1.f, ei = w2 > 0.f ? b * k : 0.f;
        o[h] = (i == mref) ? make_float2(1.f, 0.f) : make_float2(er * ur + ei * ui, ei * ur - er * ui);
        if (fin && i < n) {
            P.phase[i * P.plane + pp] = o[h];
            if (i >= mref) {                           // compressed SLC (evd.cpp:752-762)
                const float2 x = own[h];
                cr += __fadd_rn(__fmul_rn(x.x, o[h].x), __fmul_rn(x.y, o[h].y));
                ci += __fsub_rn(__fmul_rn(x.y, o[h].x), __fmul_rn(x.x, o[h].y));
            }
        }
    }
    if (L.g < M::T) sts4(L.mem + M::z + 16u * (uint32_t)L.g, o[0].x, o[1].x, o[0].y, o[1].y);
    __syncwarp();
    cr = gsum<G>(cr);
    ci = gsum<G>(ci);
    // ---- temporal coherence (evd.cpp:768-786) over the lower triangle: the
    // conjugate of the reference's sum over the upper one -----------------------------
    float tr = 0.f, ti = 0.f;
    {
        // rolled: one block's code for all (1024^2, N = 30: 13.1 -> 12.2 ms by instruction fetch)
        uint32_t ta = taddr;
#pragma unroll 1
        for (int mi = 0; mi < NL; ++mi) {
            // w_i = sum_j exp(i arg C_ij) ph_j over j < i, rows i (lo) and i' (hi)
            float w0r = 0.f, w0i = 0.f, w1r = 0.f, w1i = 0.f;
#pragma unroll 1
            for (int li = 0; li < RT * (mi + 1); ++li, ta += 8u) {
                uint32_t w[8];
                tmem_ld8(ta, w);
                f32x2 pr, pi;
                lds4(L.mem + M::z + 16u * (uint32_t)(4 * li + L.lc), pr, pi);
                const int m = LRN * mi + L.lr, l = 4 * li + L.lc;
                const bool all = li < RT * mi || m > l, some = all || m == l;
                auto term = [&](int e, float pjr, float pji, bool on, float &ar, float &ai) {
                    const float x = __uint_as_float(w[e]), y = __uint_as_float(w[e + 2]);
                    const float m2 = fmaf(x, x, y * y), k = rsqrtf(m2);
                    const float vr = m2 > 0.f ? x * k : 1.f, vi = m2 > 0.f ? y * k : 0.f;
                    if (on) {
                        ar = fmaf(vr, pjr, fmaf(-vi, pji, ar));
                        ai = fmaf(vr, pji, fmaf(vi, pjr, ai));
                    }
                };
                const float jr = lo2(pr), ji = lo2(pi), kr = hi2(pr), ki = hi2(pi);
                const int d = stbas ? P.bw - 2 * (m - l) : 1;        // pairs at most the bandwidth apart
                term(0, jr, ji, all && d >= 0, w0r, w0i);            // (i, j)
                term(1, kr, ki, all && d >= 0, w1r, w1i);            // (i', j')
                term(4, jr, ji, some && d >= 1, w1r, w1i);           // (i', j)
                term(5, kr, ki, all && d >= -1, w0r, w0i);           // (i, j')
            }
            f32x2 ar, ai;
            lds4(L.mem + M::z + 16u * (uint32_t)(LRN * mi + L.lr), ar, ai);
            const int i = 2 * (LRN * mi + L.lr);
            if (i < n) {                                 // times conj(ph_i)
                tr += fmaf(w0r, lo2(ar), w0i * lo2(ai));
                ti += fmaf(w0i, lo2(ar), -(w0r * lo2(ai)));
            }
            if (i + 1 < n) {
                tr += fmaf(w1r, hi2(ar), w1i * hi2(ai));
                ti += fmaf(w1i, hi2(ar), -(w1r * hi2(ai)));
            }
        }
    }
    tr = gsum<G>(tr);
    ti = gsum<G>(ti);
    if (fin && L.g == 0) {
        const float den = (float)(n - mref);
        P.comp[pp] = make_float2(cr / den, ci / den);
        const int pairs = stbas ? (n - P.bw) * P.bw + P.bw * (P.bw - 1) / 2 : n * (n - 1) / 2;
        P.tcorr[pp] = sqrtf(tr * tr + ti * ti) / (float)pairs;   // 0/0 = NaN for one date, as the reference
        if (P.status) P.status[pp] = 0;
    }
}

// MLE: a pixel per G lanes from its Gamma record (every lane of the warp calls
// it; valid: this group has a pixel).  taddr: NB x 8 tensor-memory columns of the
// warp, where C waits between its uses.  Returns TILE_GENERAL where
// pixel_solve has to take the pixel over (its outputs untouched).
template <int G, int NL>
__device__ __forceinline__ int tile_mle(const KParams &P, long long pp, const TileLane &L, uint32_t taddr, bool valid)
{
    using M = Tile<G, NL>;
    constexpr int NB = M::NB, RT = M::RT, LRN = M::LRN, NLC = M::NLC;
    const int n = P.nb, dp = (n + 1) >> 1;
    const bool plink = P.semantics == SEM_PL;
    CBlk A[NB];
    float cfro = 0.f;
    int state = tile_begin<G, NL, true>(P, pp, L, taddr, valid, A, cfro);
    if (!__any_sync(0xffffffffu, state == TILE_RUN)) return state;
    // the groups' steps run together: the padding's pivots are 1
    const int tp = G == 32 ? dp : max(__shfl_sync(0xffffffffu, dp, 0), __shfl_sync(0xffffffffu, dp, 16));
    const float amb = P.amb * (float)n * Eps<float>::v, thr = 1.0e-6f;
    float sigma = 0.f;
    // pass 0: lambda_min(C) > 1e-6 by the factorisation of C - (1e-6 + band) I,
    // the inverse of |C|, M; pass 1: the factor of M - sigma I.  One loop, so that the unrolled
    // factorisation is in the code once.
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        if (pass == 1) {
            // |C| and its inverse (evd.cpp:586-664)
            RBlk K[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                uint32_t w[8];
                tmem_ld8(taddr + 8u * (uint32_t)b, w);
                float a[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    // entries: D lo, D hi, E lo, E hi
                    const float x = __uint_as_float(w[(e & 1) + 4 * (e >> 1)]), y = __uint_as_float(w[(e & 1) + 4 * (e >> 1) + 2]);
                    const float m2 = fmaf(x, x, y * y);
                    a[e] = m2 * rsqrt_fast(fmaxf(m2, 1e-37f));
                }
                K[b].d = pk(a[0], a[1]);
                K[b].e = pk(a[2], a[3]);
            }
            tile_on_diag<G, NL>(L, [&](int, int b) { K[b].d = pk(1.f, 1.f); });
            bool ok = true;
            // norms of |C| and inv|C|; at 25 to 32 dates with one copy of the code, which
            // the instruction cache just does not hold otherwise (1024^2, N = 30: 12.3 ->
            // 11.95 ms; N = 15, where it fits: 3.00 -> 3.05 ms)
            float anorm = 0.f, xnorm = 0.f;
#pragma unroll(NL == 4 ? 1 : 2)
            for (int rep = 0; rep < 2; ++rep) {
                if (rep == 1) {
                    tile_sweep_seg<G, NL, 0>(K, L, tp, ok);
                    // inv|C| = -K, its diagonal 2 - K
#pragma unroll
                    for (int b = 0; b < NB; ++b) {
                        K[b].d ^= 0x8000000080000000ull;
                        K[b].e ^= 0x8000000080000000ull;
                    }
                    tile_on_diag<G, NL>(L, [&](int, int b) { K[b].d = add2(K[b].d, pk(2.f, 2.f)); });
                }
                anorm = xnorm;
                xnorm = tile_inf_norm<G, NL>(K, L);
            }
            if (state == TILE_RUN && !ok) state = TILE_GENERAL;
            if (state == TILE_RUN && (!(anorm * xnorm <= P.cond_max) || (!plink && !(1.f / xnorm > thr + amb * (float)n)))) {
                // condition too large for an FP32 inverse, or 1/||inv|C||| within the band of 1e-6
                tile_zero<G>(P, pp, L.g);
                defer_fp64(P, pp, L.g);
                state = TILE_DONE;
            }
            if (!__any_sync(0xffffffffu, state == TILE_RUN)) return state;
            // M = inv|C| o C and the Rayleigh quotient of the start vector
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                uint32_t w[8];
                tmem_ld8(taddr + 8u * (uint32_t)b, w);
                A[b].dr = mul2(pk(__uint_as_float(w[0]), __uint_as_float(w[1])), K[b].d);
                A[b].di = mul2(pk(__uint_as_float(w[2]), __uint_as_float(w[3])), K[b].d);
                A[b].er = mul2(pk(__uint_as_float(w[4]), __uint_as_float(w[5])), K[b].e);
                A[b].ei = mul2(pk(__uint_as_float(w[6]), __uint_as_float(w[7])), K[b].e);
            }
            f32x2 zr[NLC], zi[NLC], q2 = 0ull;
#pragma unroll
            for (int li = 0; li < NLC; ++li) lds4(L.mem + M::z + 16u * (uint32_t)(4 * li + L.lc), zr[li], zi[li]);
            const f32x2 two = pk(2.f, 2.f), minus = pk(-1.f, -1.f);
#pragma unroll
            for (int mi = 0; mi < NL; ++mi) {
                // y = sum_li weight M z, in the rows' order (D) and swapped (E)
                f32x2 yr = 0ull, yi = 0ull, sr = 0ull, si = 0ull;
#pragma unroll
                for (int li = 0; li < RT * (mi + 1); ++li) {
                    const CBlk &b = A[M::blk(mi, li)];
                    const f32x2 nzi = mul2(zi[li], minus);
                    if (li == RT * mi) {               // the blocks below the diagonal count twice
                        yr = mul2(yr, two); yi = mul2(yi, two); sr = mul2(sr, two); si = mul2(si, two);
                    }
                    yr = fma2(b.di, nzi, fma2(b.dr, zr[li], yr));
                    yi = fma2(b.di, zr[li], fma2(b.dr, zi[li], yi));
                    sr = fma2(b.ei, nzi, fma2(b.er, zr[li], sr));
                    si = fma2(b.ei, zr[li], fma2(b.er, zi[li], si));
                }
                f32x2 xr, xi;
                lds4(L.mem + M::z + 16u * (uint32_t)(LRN * mi + L.lr), xr, xi);
                q2 = fma2(xr, yr, fma2(xi, yi, q2));
                q2 = fma2(swap2(xr), sr, fma2(swap2(xi), si, q2));
            }
            const float rho = gsum<G>(lo2(q2) + hi2(q2));
            sigma = P.shift * fminf(rho, 1.f);
            // lambda_1 > sigma > 1e-6 + band settles the -7 test; the band by
            // |M|_F <= sqrt(n) ||inv|C|||_inf (see pixel_solve)
            const float dM = plink ? 0.f : amb * sqrtf((float)n) * xnorm;
            if (state == TILE_RUN && !(sigma > thr + dM)) state = TILE_GENERAL;
            // the padding keeps a unit pivot
            tile_on_diag<G, NL>(L, [&](int x, int b) {
                const int i = 2 * (LRN * x + L.lr);
                A[b].dr = pk(i < n ? lo2(A[b].dr) - sigma : 1.f, i + 1 < n ? hi2(A[b].dr) - sigma : 1.f);
            });
        } else {
            if (__all_sync(0xffffffffu, plink || state != TILE_RUN)) continue;   // phase_link has no such test
            const float sh = thr + amb * cfro;
            tile_on_diag<G, NL>(L, [&](int, int b) { A[b].dr = add2(A[b].dr, pk(-sh, -sh)); });
        }
        bool ok = true;
        tile_ldl_seg<G, NL, 0>(A, L, tp, ok);
        if (state == TILE_RUN && !ok && (pass == 1 || !plink)) state = TILE_GENERAL;
        if (!__any_sync(0xffffffffu, state == TILE_RUN)) return state;
        __syncwarp();
    }

    // ---- inverse iteration (warp_inverse_iteration's rule, pair per lane) -----------
    f32x2 zr, zi;
    lds4(L.mem + M::z + 16u * (uint32_t)(L.g < M::T ? L.g : 0), zr, zi);
    float z0r = lo2(zr), z1r = hi2(zr), z0i = lo2(zi), z1i = hi2(zi);
    if (L.g >= dp) z0r = z1r = z0i = z1i = 0.f;
    float2 own[2];
    tile_own(P, pp, L, state == TILE_RUN, own);
    const float tol = 1e-5f;
    float rprev = -1.f, cprev = 1.f, gap_good = 0.f;
    bool run = state == TILE_RUN;
    if (run) state = TILE_GENERAL;                    // unless it converges
#pragma unroll 1
    for (int it = 0; it < 10 && __any_sync(0xffffffffu, run); ++it) {
        float x0r = z0r, x1r = z1r, x0i = z0i, x1i = z1i;
        tile_solve<G, NL>(L, tp, x0r, x1r, x0i, x1i);
        const float xx = gsum<G>(fmaf(x0r, x0r, x0i * x0i) + fmaf(x1r, x1r, x1i * x1i));
        const float xv = gsum<G>(fmaf(x0r, z0r, x0i * z0i) + fmaf(x1r, z1r, x1i * z1i));
        const float dl = xv / xx;                     // rho - sigma
        const float a0r = fmaf(-dl, x0r, z0r), a0i = fmaf(-dl, x0i, z0i), a1r = fmaf(-dl, x1r, z1r), a1i = fmaf(-dl, x1i, z1i);
        const float inv = rsqrtf(xx);
        const float rn = sqrtf(gsum<G>(fmaf(a0r, a0r, a0i * a0i) + fmaf(a1r, a1r, a1i * a1i))) * inv;
        if (run) {
            z0r = x0r * inv;
            z1r = x1r * inv;
            z0i = x0i * inv;
            z1i = x1i * inv;
            if (rprev > 0.f) {
                const float c = rn / rprev, crate = fmaxf(c, cprev);
                if (crate < 0.9f) {
                    const float gap = dl * (1.f / crate - 1.f);
                    gap_good = gap;
                    if (rn <= tol * gap) { state = TILE_RUN; run = false; }
                }
                if (run && it >= 3 && c > 0.9f) {
                    if (rn <= 20.f * tol * gap_good) state = TILE_RUN;
                    run = false;
                }
                cprev = c;
            }
            rprev = rn;
        }
    }
    if (!__any_sync(0xffffffffu, state == TILE_RUN)) return state;

    tile_finish<G, NL>(P, pp, L, taddr, state == TILE_RUN, false, z0r, z1r, z0i, z1i, own);
    return state == TILE_RUN ? (int)TILE_DONE : state;
}

// y = C z for the coherence in A and the vector in shared memory: the row
// sums of pair LRN x + lr in (yr, yi)[x] on the diagonal lanes
template <int G, int NL>
__device__ __forceinline__ void tile_matvec(const CBlk (&A)[Tile<G, NL>::NB], const TileLane &L, f32x2 (&yr)[NL],
                                            f32x2 (&yi)[NL])
{
    using M = Tile<G, NL>;
    constexpr int RT = M::RT, LRN = M::LRN, NLC = M::NLC;
    const f32x2 minus = pk(-1.f, -1.f);
    f32x2 cr[NLC], ci[NLC];
#pragma unroll
    for (int x = 0; x < NLC; ++x) cr[x] = ci[x] = 0ull;
#pragma unroll
    for (int mi = 0; mi < NL; ++mi) {
        f32x2 xr, xi, dr = 0ull, di = 0ull, er = 0ull, ei = 0ull;
        lds4(L.mem + M::z + 16u * (uint32_t)(LRN * mi + L.lr), xr, xi);
        const f32x2 sr = swap2(xr), si = swap2(xi), nxr = mul2(xr, minus), nsr = swap2(nxr);
#pragma unroll
        for (int li = 0; li < RT * (mi + 1); ++li) {
            const CBlk &b = A[M::blk(mi, li)];
            f32x2 zr, zi;
            lds4(L.mem + M::z + 16u * (uint32_t)(4 * li + L.lc), zr, zi);
            const f32x2 nzi = mul2(zi, minus);
            dr = fma2(b.di, nzi, fma2(b.dr, zr, dr));
            di = fma2(b.di, zr, fma2(b.dr, zi, di));
            er = fma2(b.ei, nzi, fma2(b.er, zr, er));
            ei = fma2(b.ei, zr, fma2(b.er, zi, ei));
            if (li < RT * mi) {                          // the mirrored block: conj(C_ij) z_i
                cr[li] = fma2(b.di, xi, fma2(b.dr, xr, cr[li]));
                ci[li] = fma2(b.di, nxr, fma2(b.dr, xi, ci[li]));
                cr[li] = fma2(b.ei, si, fma2(b.er, sr, cr[li]));
                ci[li] = fma2(b.ei, nsr, fma2(b.er, si, ci[li]));
            }
        }
        yr[mi] = add2(dr, swap2(er));
        yi[mi] = add2(di, swap2(ei));
    }
    tile_row_sums<G, NL>(yr, cr, L);
    tile_row_sums<G, NL>(yi, ci, L);
}

// EVD and STBAS (evd.cpp:689-732): the eigenvector of the largest eigenvalue
// of C.  Power iteration with warp_power's stopping rule; where it contracts
// slowly (banded coherences do, their eigenvalues cluster), inverse iteration
// with mu I - C, mu just above the Rayleigh quotient: the factorisation
// certifies mu > lambda_max, so the iteration converges to that eigenvector, and
// a shift by the residual converges in a few steps.  Before, such pixels took the
// Householder reduction: 22.8 -> 5.2 ms at 256 x 384, N = 45, bandwidth 10.
template <int G, int NL>
__device__ __forceinline__ int tile_evd(const KParams &P, long long pp, const TileLane &L, uint32_t taddr, bool valid)
{
    using M = Tile<G, NL>;
    constexpr int NB = M::NB, LRN = M::LRN;
    const int n = P.nb, dp = (n + 1) >> 1;
    const bool dlane = (L.lr & 3) == L.lc;
    CBlk A[NB];
    float cfro = 0.f;
    int state = tile_begin<G, NL, false>(P, pp, L, taddr, valid, A, cfro);
    if (!__any_sync(0xffffffffu, state == TILE_RUN)) return state;
    float2 own[2];
    tile_own(P, pp, L, state == TILE_RUN, own);

    float rho = 1.f, rn = 0.f, rprev = -1.f, pratio = 1.f;
    bool run = state == TILE_RUN, slow = false;
#pragma unroll 1
    for (int it = 1; it < 96 && __any_sync(0xffffffffu, run); ++it) {
        f32x2 yr[NL], yi[NL];
        tile_matvec<G, NL>(A, L, yr, yi);
        float zy = 0.f, yy = 0.f, rr = 0.f;
        if (dlane) {
#pragma unroll
            for (int x = 0; x < NL; ++x) {
                f32x2 zr, zi;
                lds4(L.mem + M::z + 16u * (uint32_t)(LRN * x + L.lr), zr, zi);
                const f32x2 a = fma2(zr, yr[x], mul2(zi, yi[x])), b = fma2(yr[x], yr[x], mul2(yi[x], yi[x]));
                zy += lo2(a) + hi2(a);
                yy += lo2(b) + hi2(b);
            }
        }
        const float q = gsum<G>(zy);                        // z is normalised
        yy = gsum<G>(yy);
        if (dlane) {
#pragma unroll
            for (int x = 0; x < NL; ++x) {
                f32x2 zr, zi;
                lds4(L.mem + M::z + 16u * (uint32_t)(LRN * x + L.lr), zr, zi);
                const f32x2 nq = pk(-q, -q), a = fma2(zr, nq, yr[x]), b = fma2(zi, nq, yi[x]), c = fma2(a, a, mul2(b, b));
                rr += lo2(c) + hi2(c);
            }
        }
        const float r = sqrtf(gsum<G>(rr)), inv = rsqrtf(yy);
        __syncwarp();
        if (run) {
            if (dlane) {
#pragma unroll
                for (int x = 0; x < NL; ++x)
                    sts4(L.mem + M::z + 16u * (uint32_t)(LRN * x + L.lr), inv * lo2(yr[x]), inv * hi2(yr[x]),
                         inv * lo2(yi[x]), inv * hi2(yi[x]));
            }
            // eigenvector error ~ rn / gap, the gap about rho (1 - contraction)
            const float ratio = rprev > 0.f ? fminf(r / rprev, 1.f) : 1.f;
            rho = q;
            rn = r;
            rprev = r;
            pratio = ratio;
            if (it >= 2 && r <= 4e-6f * q * fmaxf(1.f - ratio, 0.05f)) run = false;
            else if (it >= 6 && ratio > 0.8f) { run = false; slow = true; }
        }
        __syncwarp();
    }
    slow = slow || run;
    f32x2 vr, vi;
    lds4(L.mem + M::z + 16u * (uint32_t)(L.g < M::T ? L.g : 0), vr, vi);
    float z0r = lo2(vr), z1r = hi2(vr), z0i = lo2(vi), z1i = hi2(vi);
    if (L.g >= dp) z0r = z1r = z0i = z1i = 0.f;
    if (__any_sync(0xffffffffu, slow)) {
        const bool left = slow;
        const int tp = G == 32 ? dp : max(__shfl_sync(0xffffffffu, dp, 0), __shfl_sync(0xffffffffu, dp, 16));
        // mu above rho by three times the estimate r^2 / gap of lambda_max - rho,
        // at most by the residual; the gap from the contraction, dl (1 / c - 1)
        const float tol = 1e-7f;
        // (a gap below 0.2% of rho: the reduction to tridiagonal form tells the
        // eigenvalues apart better)
        bool hard = false;
        float gap = -1.f, up = fminf(rn, 3.f * rn * rn / (rho * fmaxf(1.f - pratio, 0.02f)));
#pragma unroll 1
        for (int att = 0; att < 6 && __any_sync(0xffffffffu, slow && !hard); ++att) {
            up = fmaxf(up, 2e-5f * rho);
            const float mu = rho + up;
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                uint32_t w[8];
                tmem_ld8(taddr + 8u * (uint32_t)b, w);
                A[b].dr = pk(-__uint_as_float(w[0]), -__uint_as_float(w[1]));
                A[b].di = pk(-__uint_as_float(w[2]), -__uint_as_float(w[3]));
                A[b].er = pk(-__uint_as_float(w[4]), -__uint_as_float(w[5]));
                A[b].ei = pk(-__uint_as_float(w[6]), -__uint_as_float(w[7]));
            }
            tile_on_diag<G, NL>(L, [&](int x, int b) {
                const int i = 2 * (LRN * x + L.lr);
                A[b].dr = pk(i < n ? mu - 1.f : 1.f, i + 1 < n ? mu - 1.f : 1.f);
            });
            bool ok = true;
            tile_ldl_seg<G, NL, 0>(A, L, tp, ok);
            __syncwarp();
            if (!ok) up *= 8.f;                             // mu was below lambda_max
            bool act = slow && ok && !hard;
            float rp = -1.f;
#pragma unroll 1
            for (int it = 0; it < 6 && __any_sync(0xffffffffu, act); ++it) {
                float x0r = z0r, x1r = z1r, x0i = z0i, x1i = z1i;
                tile_solve<G, NL>(L, tp, x0r, x1r, x0i, x1i);
                const float xx = gsum<G>(fmaf(x0r, x0r, x0i * x0i) + fmaf(x1r, x1r, x1i * x1i));
                const float xv = gsum<G>(fmaf(x0r, z0r, x0i * z0i) + fmaf(x1r, z1r, x1i * z1i));
                const float dl = xv / xx;                   // mu - rho
                const float a0r = fmaf(-dl, x0r, z0r), a0i = fmaf(-dl, x0i, z0i), a1r = fmaf(-dl, x1r, z1r),
                            a1i = fmaf(-dl, x1i, z1i);
                const float inv = rsqrtf(xx);
                const float r = sqrtf(gsum<G>(fmaf(a0r, a0r, a0i * a0i) + fmaf(a1r, a1r, a1i * a1i))) * inv;
                if (act) {
                    z0r = x0r * inv;
                    z1r = x1r * inv;
                    z0i = x0i * inv;
                    z1i = x1i * inv;
                    rho = mu - dl;
                    if (rp > 0.f) {
                        // the gap by this contraction, unless rounding ended it; the
                        // smallest one seen counts, early contractions being the faster ones
                        const float c = r / rp;
                        const bool floor_ = r <= 1e-6f * dl;
                        if (c < 0.95f && !floor_) {
                            const float gn = dl * (1.f / c - 1.f);
                            gap = gap > 0.f ? fminf(gap, gn) : gn;
                        }
                        if (it >= (att > 0 ? 1 : 2) && (r <= tol * gap || (floor_ && !(gap < dl && gap > 0.f)))) { slow = false; act = false; }
                        else if (c > 0.25f) act = false;    // a closer shift
                        if (gap > 0.f && gap < 2e-3f * rho) hard = true;
                    }
                    rp = r;
                    up = gap > 0.f ? fminf(r, 3.f * r * r / gap) : r;
                }
            }
        }
        if (state == TILE_RUN && (slow || hard)) state = TILE_GENERAL;
        // (pixel_solve counts those that it takes over)
        if (left && state == TILE_RUN && L.g == 0) atomicAdd(P.slow, 1);
    }
    tile_finish<G, NL>(P, pp, L, taddr, state == TILE_RUN, P.method == M_STBAS, z0r, z1r, z0i, z1i, own);
    return state == TILE_RUN ? (int)TILE_DONE : state;
}
// L2 prefetch of a pixel's Gamma record by the lanes of its group
template <int G> __device__ __forceinline__ void tile_prefetch(const KParams &P, long long pp, int g)
{
    const long long loc = pp - P.cbase;
    const char *rec = reinterpret_cast<const char *>(P.cbuf) + loc * (long long)P.cstride * 4;
    const uintptr_t lo = reinterpret_cast<uintptr_t>(rec) & ~uintptr_t(127);
    const uintptr_t hi = reinterpret_cast<uintptr_t>(rec) + (size_t)P.cstride * 4;
    for (uintptr_t a = lo + 128u * (unsigned)g; a < hi; a += G * 128u) asm volatile("prefetch.L2 [%0];" :: "l"(a));
    if (g == G - 1) asm volatile("prefetch.L2 [%0];" :: "l"(P.cinfo + loc));
}

}  // namespace
}  // namespace fpl
