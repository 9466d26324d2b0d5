// gram_box.cu -- coherence matrices on the 5th-generation tensor cores, one
// tile of 128 pixels per GEMM.
//
// The SHP gather + Gamma accumulation
// (src/evd/evd.cpp:516-564, src/phase_link/phase_link.cpp:482-522).  For a
// pixel p the reference sums x_q x_q^H over its SHPs q.  Written for a tile
// of pixels at once this is a masked box filter of the per-sample outer
// products,
//     Gamma_p = sum_q m_pq x_q x_q^H,   m_pq = 1 iff q is an SHP of p,
// which is a dense GEMM over the samples q of the union of the tile's windows:
//     D[p][c] = sum_q A[p][q] B[c][q]
//   A = the 0/1 SHP mask (exact in bf16), rows = the 128 pixels of an
//       8 x 16 pixel tile, columns = the (8+Wy-1) x (16+Wx-1) union samples;
//   B = the outer-product entries Re / Im x_qi conj(x_qj), formed in FP32
//       (the reference's complex<float> products) and split into bf16 parts,
//       so D = A B_1 + A B_2 (+ A B_3) is accumulated in FP32 in tensor memory:
//       two parts (16 significant bits) in the mixed form, three in the FP32
//       form, which hold all 24 bits of the product.  The error of the FP32
//       form's results against 64 bits is that of the plain FP32 kernel or
//       less (STBAS, N = 48: phases 2.9e-7 rad RMS from the oracle, plain kernel
//       2.8e-7; EVD 9.3e-7 against 1.0e-6), and at 1024^2, N = 30, 11 x 21 its Gamma
//       takes 5.8 ms (two parts: 4.3) of an 18.7 ms call; the plain kernel, 20 of
//       whose 32 lanes hold sums, took 52 of 54 ms.
// Each outer product is formed once per tile instead of once for every pixel
// that uses it.  One thread issues tcgen05.mma (M = 128 pixels, N <= 256
// Gamma entries, K = 16 samples) into one of two tensor-memory accumulators;
// the Gamma entries are processed in passes of 512 columns, each pass over
// the tile's samples in chunks of 32, which two warp groups build in turn, each
// into its own operand stage.
//
// Column order (the Gamma record read by the eigen kernel): dates padded to an
// even count and grouped in pairs; block (a, b), a <= b, row-major over the
// upper triangle of pairs, holds 8 floats: Re, Im of Gamma_ij for
// (i, j) = (2a,2b), (2a,2b+1), (2a+1,2b), (2a+1,2b+1).
//
// Operand layout (no swizzle, K-major): core matrices of 8 rows x 16 bytes;
// K-adjacent core matrices 128 B apart, 8-row groups KC*16+16 B apart (the
// 16-byte pad keeps the staging stores free of bank conflicts).
//
// Samples whose value is non-finite, or whose components lie outside
// [2^-50, 2^50] in magnitude (other than 0), are outside the range of the
// split and zeroed in the tile.  A pixel with a non-finite one among its SHPs has
// a non-finite power at that date, so its outcome is known: the failure code
// of the first eigen call (CI_BAD).  A pixel with a finite one is marked CI_DEFER: the
// mixed form settles it in FP64, the FP32 form from its samples in k_rest.  Every wait on the tensor
// core is bounded; on timeout the CTA
// records an error flag, stops, and frees its tensor memory after a second
// bounded wait.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "f32x2.cuh"
#include "kernels.h"
#include "pixel.cuh"

namespace fpl {
namespace {

// 16 warps in two groups of 8 that take alternate chunks: their loads,
// arithmetic and stores overlap (in step on one chunk, the phases followed one
// another)
constexpr int BX_THREADS = 512, BX_GRP = 256;
constexpr int BX_TR = 8, BX_TC = 16, BX_M = 128;   // pixel tile (MMA M)
constexpr int BX_NCOL = 256;                       // Gamma columns per accumulator (MMA N)
// samples per chunk (MMA K of one stage): 32, so that two accumulators (512
// Gamma columns per pass with two parts, 352 with three) fit beside two
// operand stages and two sample buffers
constexpr int BX_KC = 32;
constexpr int BX_MAXK = 2048;                      // union samples per tile
constexpr int BX_MAXW = BX_MAXK / 32;              // union mask words per pixel
constexpr int BX_MAXWX = 63;                       // window width (64-bit row extraction)
constexpr int BX_MISC = 4096;
constexpr int CI_SKIP = -100;                      // pixel outside this launch's rows
constexpr unsigned ERR_TC_TIMEOUT = 2u;
constexpr long long BX_SPIN_LIMIT = 1ll << 26;     // ~ seconds of polling

// shared memory of a CTA; NS: bf16 parts of a product.  Barriers, tables and
// sample buffers come first, at the same place for both NS.
template <int KC, int NS> struct BoxLay {
    // tensor-memory accumulators of BX_NCOL columns each: a pass covers PCOL
    // Gamma columns, and a chunk's samples and mask are loaded and built once for
    // all of them
    static constexpr int NACC = (KC == 32) ? 2 : 1;
    static constexpr int PCOL = NS == 3 ? 352 : NACC * BX_NCOL;
    static constexpr int TCOL = NACC * BX_NCOL;              // tensor-memory columns held
    static constexpr int SBO = KC * 16 + 16;                 // bytes between 8-row groups
    static constexpr int A_BYTES = (BX_M / 8) * SBO;
    static constexpr int B_BYTES = (PCOL / 8) * SBO;         // one part
    static constexpr int STAGE = A_BYTES + NS * B_BYTES;
    static constexpr int MAXPAIR = 32;                       // date pairs: 64 dates
    static constexpr int XRS = KC * 16 + 16;                 // bytes per date pair of X (see put)
    static constexpr int X_BYTES = MAXPAIR * XRS;            // one of two sample buffers
    static constexpr size_t OFF_MISC = 0;
    static constexpr size_t OFF_LUT = OFF_MISC + BX_MISC;          // 256 x 8 bf16 mask patterns
    static constexpr size_t OFF_X = OFF_LUT + 256 * 16;
    static constexpr size_t OFF_ST = OFF_X + 2 * (size_t)X_BYTES;  // two operand stages
    static constexpr size_t OFF_U = OFF_ST + 2 * (size_t)STAGE;
    static constexpr size_t MAX_SMEM = OFF_U + (size_t)BX_M * BX_MAXW * 4;
    static_assert(MAX_SMEM <= 227 * 1024, "shared memory of one CTA");
    static_assert(OFF_ST % 16 == 0 && STAGE % 16 == 0 && PCOL % 16 == 0, "operand alignment");
};

// union samples of a tile: (8 + 2 ny) rows of (16 + 2 nx) samples, packed
// row after row (no padding: every sample slot is a GEMM K index)
__host__ __device__ __forceinline__ int box_union_cols(int nx) { return BX_TC + 2 * nx; }

__device__ __forceinline__ uint32_t smem_addr(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// shared-memory matrix descriptor: start, leading (K) and stride (M/N) byte
// offsets, descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// instruction descriptor, kind::f16: FP32 accumulate, bf16 A and B, both
// K-major, M = 128, N = n
__device__ __forceinline__ uint32_t make_idesc(int n)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        :: "r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accum));
}

__device__ __forceinline__ void tc_commit(uint64_t *mbar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(smem_addr(mbar)) : "memory");
}

__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint64_t *mbar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_addr(mbar)), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *mbar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok) : "r"(smem_addr(mbar)), "r"(parity) : "memory");
    return ok != 0;
}

// 32 consecutive 32-bit TMEM columns of this thread's lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t *r)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// len (<= 63) bits of a little-endian word array starting at bit pos
__device__ __forceinline__ uint64_t extract_bits(const uint32_t *w, int nul, int pos, int len)
{
    const int w0 = pos >> 5, sh = pos & 31;
    uint64_t v = w[w0];
    if (w0 + 1 < nul) v |= (uint64_t)w[w0 + 1] << 32;
    v >>= sh;
    if (sh && w0 + 2 < nul) v |= (uint64_t)w[w0 + 2] << (64 - sh);
    return v & ((1ull << len) - 1ull);
}

// 0 or a normal magnitude in [2^-50, 2^50]: the bf16 split of every product
// of two such components stays normal and the window sums stay finite
__device__ __forceinline__ bool split_range(float v)
{
    const float a = fabsf(v);
    return v == 0.f || (a >= 8.8817842e-16f && a <= 1.1258999e15f);
}

// 8 values of one Gamma column (as pairs) into NS bf16 rows (16 bytes each,
// pstride apart): each part rounds what the parts before it left (exact
// differences)
template <int NS>
__device__ __forceinline__ void store_split(unsigned char *dst, uint32_t pstride, const f32x2 (&v)[4])
{
    uint32_t p[NS][4];
    const f32x2 minus = pk(-1.f, -1.f);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        f32x2 a = v[q];
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const __nv_bfloat162 t = __floats2bfloat162_rn(lo2(a), hi2(a));
            const uint32_t u = *reinterpret_cast<const uint32_t *>(&t);
            p[s][q] = u;
            if (s + 1 < NS) a = fma2(pk(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)), minus, a);
        }
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) *reinterpret_cast<uint4 *>(dst + s * pstride) = make_uint4(p[s][0], p[s][1], p[s][2], p[s][3]);
}

// pipeline state of a CTA, carried from tile to tile (and job to job).  Step n
// (a chunk) uses operand stage n & 1 and is built by group n & 1; its k-th use
// of the stage (k = n >> 1) completes phase k of the stage's two barriers: full
// (built, an arrival per thread of the group) and empty (its MMAs are done).
struct BoxPipe {
    unsigned base;      // steps before this tile
    unsigned issued;    // one past the last step whose MMAs this thread issued
    bool timed_out;
    int blk_dp;         // date pairs the block table was built for
};
struct BoxBars {
    uint64_t full[2], empty[2];
    uint32_t tmem_slot;
    int dead;           // a wait gave up: the others stop waiting
};

// bounded wait for step n on a pair of barriers; true if it gave up (or
// another wait had)
__device__ __forceinline__ bool box_wait(uint64_t *pair, unsigned n, volatile int *dead)
{
    long long spins = 0;
    while (!mbar_try_wait(&pair[n & 1], (n >> 1) & 1u)) {
        if (*dead || ++spins > BX_SPIN_LIMIT) {
            *dead = 1;
            return true;
        }
    }
    return false;
}

// barrier of a group's threads; true if any of them passes true
__device__ __forceinline__ bool group_or(int grp, bool v)
{
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbarrier.cta.red.or.pred p, %2, %3, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(r) : "r"((uint32_t)v), "r"(1 + grp), "n"(BX_GRP) : "memory");
    return r != 0;
}
__device__ __forceinline__ void group_sync(int grp)
{
    asm volatile("barrier.cta.sync %0, %1;" :: "r"(1 + grp), "n"(BX_GRP) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *mbar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_addr(mbar)) : "memory");
}

// tiles of the rows [ra, rb) of a launch: 8-row tiles on the absolute grid
// (rows 8t .. 8t+7 of the scene, whose first row is row -grid0 of the array) so that a pixel's
// Gamma, and its order of accumulation, do not depend on how the rows were split into
// launches or the scene into arrays
__host__ __device__ __forceinline__ int box_first_row(const KParams &P)
{
    return (int(P.pix_begin / P.cols) + P.grid0) / BX_TR * BX_TR - P.grid0;
}
__host__ __device__ __forceinline__ long long box_tiles(const KParams &P)
{
    const int ra = int(P.pix_begin / P.cols), rb = ra + int(P.npix / P.cols);
    if (rb <= ra) return 0;
    return (long long)((P.cols + BX_TC - 1) / BX_TC) * ((rb - box_first_row(P) + BX_TR - 1) / BX_TR);
}

// passes over a tile's samples that n dates take
template <int KC, int NS> __host__ __device__ __forceinline__ int box_passes(int n)
{
    const int dp = (n + 1) >> 1;
    return (4 * dp * (dp + 1) + BoxLay<KC, NS>::PCOL - 1) / BoxLay<KC, NS>::PCOL;
}

// Gamma records of tile t of the launch described by P, its passes from pass0 up to pass1
// (all threads of the CTA call it together)
template <int KC, int NS>
__device__ __forceinline__ void box_tile(const KParams &P, long long t, int pass0, int pass1, unsigned char *smem,
                                         uint32_t tbase, BoxPipe &st)
{
    using L = BoxLay<KC, NS>;
    unsigned char *stages = smem + L::OFF_ST;
    unsigned char *Xb = smem + L::OFF_X;
    unsigned char *misc = smem + L::OFF_MISC;
    BoxBars *bars = reinterpret_cast<BoxBars *>(misc);
    volatile int *dead = &bars->dead;
    int *pinfo = reinterpret_cast<int *>(misc + 64);                     // 128
    int *pdefer = reinterpret_cast<int *>(misc + 64 + 512);              // 128: 0, CI_DEFER or CI_BAD (tiles that are not clean)
    short2 *blk = reinterpret_cast<short2 *>(misc + 64 + 1024);          // <= 528 blocks
    uint32_t *tbad = reinterpret_cast<uint32_t *>(misc + 3200);          // [W] out-of-range samples
    uint32_t *tinf = tbad + BX_MAXW;                                     // [W] non-finite ones
    uint32_t *umask = reinterpret_cast<uint32_t *>(smem + L::OFF_U);     // [128][W]
    const uint4 *lut = reinterpret_cast<const uint4 *>(smem + L::OFF_LUT);
    uint32_t *nm = reinterpret_cast<uint32_t *>(stages + L::STAGE);      // nmap words (stage 1, mask build only)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n = P.nb, dp = (n + 1) >> 1, nblk = dp * (dp + 1) / 2, ncolt = 8 * nblk;
    const int cols = P.cols, rows = P.rows, nul = P.nulong;
    const int wy = 2 * P.ny + 1, wx = P.wx;
    const int uh = BX_TR + wy - 1, uwp = box_union_cols(P.nx);   // union rows, columns
    const int kp = (uh * uwp + KC - 1) / KC * KC, nchunk = kp / KC;
    const int W = kp >> 5;
    const int ra = int(P.pix_begin / cols), rb = ra + int(P.npix / cols);
    const int ntc = (cols + BX_TC - 1) / BX_TC;
    const int min_neigh = (P.semantics == SEM_PL) ? P.min_neigh : 2;   // evd.cpp:566
    const long long plane = P.plane;
    const int R0 = box_first_row(P) + int(t / ntc) * BX_TR, C0 = int(t % ntc) * BX_TC;
    const int grp = (tid / BX_GRP) & 1, gt = tid % BX_GRP;      // group and thread of it

    // samples of a chunk: each thread of the group that builds it loads one
    // sample for up to BX_XPT dates into registers (64 dates over the group), a
    // whole step of the other group ahead; put() stores them in the group's sample buffer and
    // flags samples outside the split range in tbad
    constexpr int BX_XPT = 2 * L::MAXPAIR * KC / BX_GRP;
    static_assert(BX_XPT >= 1 && BX_XPT * (BX_GRP / KC) == 2 * L::MAXPAIR, "date coverage");
    const int sidx = gt % KC, d0 = gt / KC;
    const int gtot = (pass1 - pass0) * nchunk;
    const int g0 = (grp - (int)(st.base & 1)) & 1;              // the group's first step of the tile
    float2 xv[BX_XPT];
    // a group's chunks advance by two, cyclically over the tile: the union row
    // and column of this thread's next sample advance by 2 KC, with a division
    // only at the start (of chunks 0 and 1)
    int us[2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        us[h][0] = (h * KC + sidx) / uwp;
        us[h][1] = h * KC + sidx - us[h][0] * uwp;
    }
    int fch = (nchunk > 1) ? g0 : 0, fur = fch ? us[1][0] : us[0][0], fuc = fch ? us[1][1] : us[0][1];
    const float2 *sbase = P.stack + (long long)d0 * plane;
    auto fetch = [&]() {
        const int r = R0 - P.ny + fur, c = C0 - P.nx + fuc;
        const bool valid = fur < uh && r >= 0 && r < rows && c >= 0 && c < cols;
        const float2 *src = sbase + (valid ? (long long)r * cols + c : 0ll);
#pragma unroll
        for (int q = 0; q < BX_XPT; ++q) {
            const int d = d0 + q * (BX_GRP / KC);
            float2 x = make_float2(0.f, 0.f);
            if (valid && d < n) x = __ldg(src + (long long)(q * (BX_GRP / KC)) * plane);
            xv[q] = x;
        }
        fch += 2;
        if (fch >= nchunk) {
            fch -= nchunk;
            if (fch >= nchunk) fch -= nchunk;
            fur = fch ? us[1][0] : us[0][0];
            fuc = fch ? us[1][1] : us[0][1];
        } else {
            fuc += 2 * KC;
            while (fuc >= uwp) { fuc -= uwp; ++fur; }
        }
    };
    if (g0 < gtot) fetch();

    // Gamma column blocks (a, b), a <= b, of this stack depth
    if (st.blk_dp != dp) {
        __syncthreads();
        for (int b = tid; b < nblk; b += BX_THREADS) {
            int a = 0, rem = b;
            while (rem >= dp - a) { rem -= dp - a; ++a; }
            blk[b] = make_short2((short)a, (short)(a + rem));
        }
        st.blk_dp = dp;
    }
    // the chunk's rest list starts empty (the solve kernels run after this one)
    if (t == 0 && pass0 == 0 && tid == 0) {
        P.fb_count[1] = 0;
        P.fb_count[13] = 0;
    }
    // ---- per-pixel SHP masks over the union samples ----------------
    for (int e = tid; e < BX_M * W; e += BX_THREADS) umask[e] = 0;
    for (int e = tid; e < W; e += BX_THREADS) tbad[e] = tinf[e] = 0;
    for (int e = tid; e < BX_M * nul; e += BX_THREADS) {
        const int m = e / nul, w = e - m * nul;
        const int r = R0 + m / BX_TC, c = C0 + m % BX_TC;
        nm[e] = (r >= ra && r < rb && c < cols) ? __ldg(P.nmap + ((long long)r * cols + c) * nul + w) : 0u;
    }
    __syncthreads();
    for (int e = tid; e < BX_M * wy; e += BX_THREADS) {
        const int m = e / wy, a = e - m * wy;
        const int tr = m / BX_TC, tc = m % BX_TC;
        const int r = R0 + tr, c = C0 + tc;
        const int sr = r - P.ny + a;                    // image row of window row a
        if (r < ra || r >= rb || c >= cols || sr < 0 || sr >= rows) continue;
        uint64_t bits = extract_bits(nm + m * nul, nul, a * wx, wx);
        // window column b is image column c - nx + b (evd.cpp:530-534)
        const int blo = max(0, P.nx - c), bhi = min(wx, cols - c + P.nx);
        if (bhi <= blo) continue;
        bits &= ((1ull << (bhi - blo)) - 1ull) << blo;
        if (!bits) continue;
        const int pos = (tr + a) * uwp + tc;            // union sample of window (a, 0)
        const int w0 = pos >> 5, sh = pos & 31;
        const uint64_t lo = bits << sh;
        const uint32_t hi = sh ? (uint32_t)(bits >> (64 - sh)) : 0u;
        uint32_t *um = umask + m * W;
        if ((uint32_t)lo) atomicOr(um + w0, (uint32_t)lo);
        if ((uint32_t)(lo >> 32)) atomicOr(um + w0 + 1, (uint32_t)(lo >> 32));
        if (hi) atomicOr(um + w0 + 2, hi);
    }
    __syncthreads();
    if (tid < BX_M) {
        const int m = tid, r = R0 + m / BX_TC, c = C0 + m % BX_TC;
        int info = CI_SKIP;                                 // outside rows [ra, rb) of this launch
        if (r >= ra && r < rb && c < cols) {
            const int cflat = P.ny * wx + P.nx;
            if (!((nm[m * nul + (cflat >> 5)] >> (cflat & 31)) & 1u)) {
                info = CI_CENTRE;                       // evd.cpp:517
            } else {
                int cnt = 0;
                for (int w = 0; w < W; ++w) cnt += __popc(umask[m * W + w]);
                info = (cnt < min_neigh) ? CI_FEW : cnt;
            }
        }
        pinfo[m] = info;
    }
    // range checks: always in the first pass; in later passes only if the
    // first found an out-of-range sample in the tile (clean: it found none)
    bool clean = false;
    auto put = [&](unsigned char *xd, int k0) {
        bool xbad = false, xinf = false;
#pragma unroll
        for (int q = 0; q < BX_XPT; ++q) {
            const int d = d0 + q * (BX_GRP / KC);
            if (d >= 2 * dp) break;
            float2 x = xv[q];
            if (!clean && (!split_range(x.x) || !split_range(x.y))) {
                xbad = true;
                xinf = xinf || !isfinite(x.x) || !isfinite(x.y);
                x = make_float2(0.f, 0.f);
            }
            // per date pair: Re and Im of the first date, then of the second,
            // KC samples each (the build reads runs of samples)
            float *xp = reinterpret_cast<float *>(xd + (d >> 1) * L::XRS + (d & 1) * (8 * KC)) + sidx;
            xp[0] = x.x;
            xp[KC] = x.y;
        }
        if (xbad) atomicOr(tbad + ((k0 + sidx) >> 5), 1u << ((k0 + sidx) & 31));
        if (xinf) atomicOr(tinf + ((k0 + sidx) >> 5), 1u << ((k0 + sidx) & 31));
    };
    __syncthreads();

    for (int pass = 0; pass < pass1 - pass0 && !st.timed_out; ++pass) {
        const int cb = (pass0 + pass) * L::PCOL;
        const int ncol = min(L::PCOL, ncolt - cb);
        // accumulator j holds the pass's columns [256 j, 256 j + 256)
        int nmma[L::NACC];
        uint32_t idesc[L::NACC];
#pragma unroll
        for (int j = 0; j < L::NACC; ++j) {
            const int nc = min(BX_NCOL, ncol - j * BX_NCOL);
            nmma[j] = nc > 0 ? (nc + 15) & ~15 : 0;
            idesc[j] = make_idesc(nmma[j] > 0 ? nmma[j] : 16);
        }
        bool late = false;
        {
            // this thread's share of the B build, the same in every chunk of the pass:
            // block bl's rows 4 ia .. 4 ia + 3 (entries (2a + ia, 2b), (2a + ia, 2b + 1), Re
            // and Im) over the 8 samples of K group k8; off < 0: none; zero: columns
            // that pad the last MMA to 16
            constexpr int K8 = KC / 8, NIT = 2;
            static_assert(2 * (L::PCOL / 8) * K8 <= NIT * BX_GRP, "items of a chunk");
            const int nb8 = (ncol + 15) / 16 * 2;
            int it_off[NIT], it_a[NIT], it_b[NIT];
            bool it_zero[NIT];
#pragma unroll
            for (int i = 0; i < NIT; ++i) {
                const int e = gt + i * BX_GRP;
                it_off[i] = -1;
                it_a[i] = it_b[i] = 0;
                it_zero[i] = false;
                if (e < 2 * nb8 * K8) {
                    const int r8 = e / nb8, bl = e - r8 * nb8, ia = r8 & 1, k8 = r8 >> 1;
                    it_off[i] = bl * L::SBO + k8 * 128 + ia * 64;
                    it_zero[i] = bl * 8 >= ncol;
                    const short2 ab = blk[cb / 8 + (it_zero[i] ? 0 : bl)];
                    it_a[i] = ab.x * L::XRS + ia * (8 * KC) + k8 * 32;
                    it_b[i] = ab.y * L::XRS + k8 * 32;
                }
            }
            unsigned char *As = stages + grp * L::STAGE, *Bs = As + L::A_BYTES;
            unsigned char *X = Xb + grp * L::X_BYTES;
            int ch = (g0 - pass * nchunk) & 1;                  // the group's first chunk of the pass
            for (int g = pass * nchunk + ch; ch < nchunk; g += 2, ch += 2) {
                const unsigned step = st.base + (unsigned)g;
                const int k0 = ch * KC;
                // the MMAs that read the stage two steps ago must be done, and the
                // group's last build have read the sample buffer
                late = late || (step >= 2 && box_wait(bars->empty, step - 2, dead));
                if (group_or(grp, late)) { late = true; break; }
                put(X, k0);
                group_sync(grp);
                if (g + 2 < gtot) fetch();
                // ---- A: SHP mask rows ----
#pragma unroll
                for (int e = gt; e < BX_M * K8; e += BX_GRP) {
                    const int m = e & (BX_M - 1), k8 = e >> 7;
                    const int b0 = k0 + k8 * 8;
                    const uint32_t bits = (umask[m * W + (b0 >> 5)] >> (b0 & 31)) & 0xffu;
                    *reinterpret_cast<uint4 *>(As + (m >> 3) * L::SBO + k8 * 128 + (m & 7) * 16) = lut[bits];
                }
                // ---- B: outer-product entries, NS parts ----
                // two samples per packed operation; the products round as
                // fma(xr, yr, xi yi) and fma(xi, yr, -(xr yi))
#pragma unroll
                for (int i = 0; i < NIT; ++i) {
                    if (it_off[i] < 0) continue;
                    unsigned char *db = Bs + it_off[i];
                    if (it_zero[i]) {
                        const uint4 z = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                        for (int c = 0; c < 4; ++c)
#pragma unroll
                            for (int p = 0; p < NS; ++p) *reinterpret_cast<uint4 *>(db + p * L::B_BYTES + c * 16) = z;
                        continue;
                    }
                    auto run8 = [](const unsigned char *src, f32x2 (&v)[4]) {
                        const ulonglong2 u = *reinterpret_cast<const ulonglong2 *>(src);
                        const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(src + 16);
                        v[0] = u.x; v[1] = u.y; v[2] = w.x; v[3] = w.y;
                    };
                    f32x2 xr[4], xi[4], nxr[4];
                    run8(X + it_a[i], xr);
                    run8(X + it_a[i] + 4 * KC, xi);
#pragma unroll
                    for (int q = 0; q < 4; ++q) nxr[q] = xr[q] ^ 0x8000000080000000ull;
#pragma unroll
                    for (int jb = 0; jb < 2; ++jb) {           // i = 2a + ia, j = 2b + jb
                        f32x2 yr[4], yi[4], v[4];
                        run8(X + it_b[i] + jb * (8 * KC), yr);
                        run8(X + it_b[i] + jb * (8 * KC) + 4 * KC, yi);
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[q] = fma2(xr[q], yr[q], mul2(xi[q], yi[q]));       // Re x_i conj(x_j)
                        store_split<NS>(db + (2 * jb) * 16, L::B_BYTES, v);
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[q] = fma2(xi[q], yr[q], mul2(nxr[q], yi[q]));      // Im x_i conj(x_j)
                        store_split<NS>(db + (2 * jb + 1) * 16, L::B_BYTES, v);
                    }
                }
                fence_async_smem();
                mbar_arrive(&bars->full[grp]);
                // one thread of the group, another warp's each time, issues the
                // step's MMAs once all have arrived and the previous step's (another
                // thread's, into the same accumulators) are done
                if (warp == 8 * grp + (int)((step >> 1) & 7u)) {
                    if (lane == 0) {
                        late = box_wait(bars->full, step, dead) || (step >= 1 && box_wait(bars->empty, step - 1, dead));
                        if (!late) {
                            fence_after_sync();
                            const uint32_t a0 = smem_addr(As), b0 = smem_addr(Bs);
#pragma unroll
                            for (int kk = 0; kk < KC / 16; ++kk) {
                                const uint64_t da = make_smem_desc(a0 + kk * 256, 128, L::SBO);
#pragma unroll
                                for (int j = 0; j < L::NACC; ++j) {
                                    if (nmma[j] == 0) continue;
                                    const uint32_t boff = (uint32_t)(j * (BX_NCOL / 8) * L::SBO + kk * 256);
                                    const uint32_t dt = tbase + (uint32_t)(j * BX_NCOL);
#pragma unroll
                                    for (int p = 0; p < NS; ++p)
                                        tc_mma(dt, da, make_smem_desc(b0 + p * L::B_BYTES + boff, 128, L::SBO), idesc[j],
                                               (ch > 0 || kk > 0 || p > 0) ? 1u : 0u);
                                }
                            }
                            tc_commit(&bars->empty[step & 1]);
                            st.issued = step + 1;
                        }
                    }
                    __syncwarp();
                }
            }
        }
        __syncwarp();
        // The pass's MMAs: its last step but one, then the last.  A parity wait for step
        // n tells phases n / 2 and n / 2 - 1 of its barrier apart only where step n - 2 is
        // known to be done.  For step last - 1 both groups know that (one waited for
        // last - 3 itself, the other for last - 2, which is issued after last - 3 is
        // done); for step last it follows from last - 1, which is issued after
        // last - 2 is done.
        {
            const unsigned last = st.base + (unsigned)((pass + 1) * nchunk - 1);
            if (!late && last >= 1) late = box_wait(bars->empty, last - 1, dead);
            if (!late) late = box_wait(bars->empty, last, dead);
        }
        if (__syncthreads_or(late)) { st.timed_out = true; break; }
        fence_after_sync();
        if (pass == 0) {
            // every sample of the tile has been checked and stored: both groups
            // have passed the barrier above
            uint32_t any = 0;
            for (int w = 0; w < W; ++w) any |= tbad[w];
            clean = any == 0;
            if (!clean) {
                if (tid < BX_M) {
                    const int m = tid;
                    uint32_t hit = 0, inf = 0;
                    for (int w = 0; w < W; ++w) {
                        hit |= umask[m * W + w] & tbad[w];
                        inf |= umask[m * W + w] & tinf[w];
                    }
                    pdefer[m] = inf ? CI_BAD : hit ? CI_DEFER : 0;
                }
                __syncthreads();
            }
        }
        // ---- epilogue: warp w reads TMEM lanes 32(w%4).., every fourth 32 columns ----
        // A lane holds its own pixel's columns; they are written out through
        // a 32 x 32 staging tile per warp (in the operand stages, which no
        // MMA reads any more: both stages were waited for above) so that
        // each store instruction writes four pixels' 128 contiguous bytes
        // instead of 32 pixels' 16.
        {
            constexpr int SROW = 36;                        // staging row stride (floats)
            static_assert((BX_THREADS / 32) * 32 * SROW * 4 <= 2 * L::STAGE, "staging fits the stages");
            float *stg = reinterpret_cast<float *>(stages) + warp * (32 * SROW);
            float *rec = reinterpret_cast<float *>(P.cbuf);
            const int q = warp & 3, h = warp >> 2;
            for (int c32 = h; c32 < L::PCOL / 32; c32 += BX_THREADS / 128) {
                const int col0 = 32 * c32;
                if (col0 >= ncol) break;
                uint32_t v[32];
                tmem_ld32(tbase + ((uint32_t)(32 * q) << 16) + (uint32_t)col0, v);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    *reinterpret_cast<float4 *>(stg + lane * SROW + j) =
                        make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                    __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                __syncwarp();
                const int lim = min(32, ncol - col0);
                const int j = 4 * (lane & 7);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int pl = 4 * i + (lane >> 3);          // pixel of the warp's 32
                    const int m = 32 * q + pl;
                    if (j < lim && pinfo[m] >= 0 && (clean || !pdefer[m])) {
                        const long long loc = (long long)(R0 + m / BX_TC) * cols + (C0 + m % BX_TC) - P.cbase;
                        *reinterpret_cast<float4 *>(rec + loc * P.cstride + cb + col0 + j) =
                            *reinterpret_cast<const float4 *>(stg + pl * SROW + j);
                    }
                }
                __syncwarp();
            }
        }
        fence_before_sync();
        __syncthreads();
    }
    if (st.timed_out) return;
    st.base += (unsigned)gtot;
    if (pass0 == 0 && tid < BX_M) {
        const int m = tid, info = pinfo[m];
        if (info != CI_SKIP) {
            const long long loc = (long long)(R0 + m / BX_TC) * cols + (C0 + m % BX_TC) - P.cbase;
            P.cinfo[loc] = (info >= 0 && !clean && pdefer[m]) ? pdefer[m] : info;
        }
    }
    __syncthreads();

}

// barriers, tables and tensor memory, the same for both NS
template <int KC>
__device__ __forceinline__ uint32_t box_setup(unsigned char *smem, BoxPipe &st)
{
    using L = BoxLay<KC, 2>;
    BoxBars *bars = reinterpret_cast<BoxBars *>(smem + L::OFF_MISC);
    const int tid = threadIdx.x, warp = tid >> 5;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_addr(&bars->tmem_slot)), "r"(L::TCOL) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&bars->full[s], BX_GRP);
            mbar_init(&bars->empty[s], 1);
        }
        bars->dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // mask patterns: entry b holds 8 bf16 values, 1 where bit q of b is set
    uint4 *lut = reinterpret_cast<uint4 *>(smem + L::OFF_LUT);
    for (int b = tid; b < 256; b += BX_THREADS) {
        uint32_t v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            v[q] = ((b >> (2 * q)) & 1 ? 0x3F80u : 0u) | ((b >> (2 * q + 1)) & 1 ? 0x3F800000u : 0u);
        lut[b] = make_uint4(v[0], v[1], v[2], v[3]);
    }
    st.base = 0;
    st.issued = 0;
    st.timed_out = false;
    st.blk_dp = -1;
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    return bars->tmem_slot;
}

// on a timeout: record the error, give the MMAs in flight a second bounded
// wait; then release the tensor memory
template <int KC>
__device__ __forceinline__ void box_teardown(unsigned char *smem, uint32_t tbase, BoxPipe &st, unsigned *err)
{
    using L = BoxLay<KC, 2>;
    BoxBars *bars = reinterpret_cast<BoxBars *>(smem + L::OFF_MISC);
    const int tid = threadIdx.x, warp = tid >> 5;
    if (st.timed_out) {
        if (tid == 0) atomicOr(err, ERR_TC_TIMEOUT);
        // threads that issued MMAs wait for their last ones
        if (st.issued > 0) {
            const unsigned n = st.issued - 1;
            long long spins = 0;
            while (!mbar_try_wait(&bars->empty[n & 1], (n >> 1) & 1u) && ++spins < BX_SPIN_LIMIT) {
            }
        }
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tbase), "r"(L::TCOL) : "memory");
    }
}

// nsplit: CTAs that share a tile's passes (launch_box_t)
template <int KC, int NS>
__global__ void __launch_bounds__(BX_THREADS, 1) k_gram_box(const __grid_constant__ KParams P, int nsplit)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    BoxPipe st;
    const uint32_t tbase = box_setup<KC>(smem, st);
    const long long nitems = box_tiles(P) * nsplit;
    const int npass = box_passes<KC, NS>(P.nb);
    for (long long k = blockIdx.x; k < nitems && !st.timed_out; k += gridDim.x) {
        const long long t = k / nsplit;
        const int j = (int)(k - t * nsplit);
        box_tile<KC, NS>(P, t, j * npass / nsplit, (j + 1) * npass / nsplit, smem, tbase, st);
    }
    box_teardown<KC>(smem, tbase, st, P.err);
}

// Many launches' tiles in one persistent launch: segment s covers tiles
// [segs[s].tile_offset, segs[s+1].tile_offset) of the concatenation.
template <int KC>
__global__ void __launch_bounds__(BX_THREADS, 1) k_gram_batch(const BoxSeg *__restrict__ segs, int nseg,
                                                              long long total)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    BoxPipe st;
    const uint32_t tbase = box_setup<KC>(smem, st);
    for (long long t = blockIdx.x; t < total && !st.timed_out; t += gridDim.x) {
        int lo = 0, hi = nseg - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (segs[mid].tile_offset <= t) lo = mid; else hi = mid - 1;
        }
        const KParams &P = segs[lo].P;
        if (P.parts == 3) box_tile<KC, 3>(P, t - segs[lo].tile_offset, 0, box_passes<KC, 3>(P.nb), smem, tbase, st);
        else box_tile<KC, 2>(P, t - segs[lo].tile_offset, 0, box_passes<KC, 2>(P.nb), smem, tbase, st);
    }
    box_teardown<KC>(smem, tbase, st, segs[0].P.err);
}

template <int KC>
size_t box_smem(int ny, int nx, int parts)
{
    const int uh = BX_TR + 2 * ny, uwp = box_union_cols(nx);
    const int kp = (uh * uwp + KC - 1) / KC * KC;
    return (parts == 3 ? BoxLay<KC, 3>::OFF_U : BoxLay<KC, 2>::OFF_U) + (size_t)BX_M * (kp / 32) * 4;
}

template <typename K>
cudaError_t box_configure(K kern, size_t smem_max, bool *configured)
{
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && configured[dev]) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max);
    if (e == cudaSuccess && dev < 64) configured[dev] = true;
    return e;
}

template <int KC, int NS>
cudaError_t launch_box_t(const KParams &P, int num_sms, cudaStream_t st)
{
    static bool configured[64] = {false};
    cudaError_t e = box_configure(k_gram_box<KC, NS>, BoxLay<KC, NS>::MAX_SMEM, configured);
    if (e != cudaSuccess) return e;
    // Where the tiles leave SMs idle, several CTAs share a tile's passes, which are
    // independent columns: as many as run in one wave (more would repeat the tile's mask build
    // without a gain).  32 x 32, FP32 form: 143 -> 50 us at 32 dates (11 x 21), 358 -> 43 us
    // at 64 (11 x 11); with whole tiles such calls took longer than the plain kernel's
    // 105 and 248 us.
    const long long ntiles = std::max<long long>(1, box_tiles(P));
    const int nsplit = (int)std::max<long long>(1, std::min<long long>(box_passes<KC, NS>(P.nb), num_sms / ntiles));
    const long long blocks = std::min<long long>(num_sms, ntiles * nsplit);
    k_gram_box<KC, NS><<<(unsigned)blocks, BX_THREADS, box_smem<KC>(P.ny, P.nx, NS), st>>>(P, nsplit);
    return cudaGetLastError();
}

template <int KC>
cudaError_t configure_box_batch()
{
    static bool configured[64] = {false};
    constexpr size_t m2 = BoxLay<KC, 2>::MAX_SMEM, m3 = BoxLay<KC, 3>::MAX_SMEM;
    return box_configure(k_gram_batch<KC>, m2 > m3 ? m2 : m3, configured);
}

template <int KC>
cudaError_t launch_box_batch_t(const BoxSeg *segs, int nseg, long long total, size_t smem, int num_sms,
                               cudaStream_t st)
{
    cudaError_t e = configure_box_batch<KC>();
    if (e != cudaSuccess) return e;
    long long blocks = num_sms;
    if (total < blocks) blocks = total > 0 ? total : 1;
    k_gram_batch<KC><<<(unsigned)blocks, BX_THREADS, smem, st>>>(segs, nseg, total);
    return cudaGetLastError();
}

}  // namespace

bool gram_box_supported(int nb, int ny, int nx)
{
    const int wx = 2 * nx + 1;
    if (nb < 1 || nb > 64 || wx > BX_MAXWX) return false;
    const int uh = BX_TR + 2 * ny, uwp = box_union_cols(nx);
    return (long long)uh * uwp <= BX_MAXK;
}

int gram_box_record(int nb)
{
    const int dp = (nb + 1) >> 1;
    return 8 * (dp * (dp + 1) / 2);
}

long long gram_box_tiles(const KParams &P) { return box_tiles(P); }

size_t gram_box_smem(const KParams &P) { return box_smem<BX_KC>(P.ny, P.nx, P.parts); }

cudaError_t prepare_gram_batch()
{
    return configure_box_batch<BX_KC>();
}

cudaError_t launch_gram_batch(const BoxSeg *segs, int nseg, long long total, size_t smem, int num_sms,
                              cudaStream_t st)
{
    if (nseg <= 0 || total <= 0) return cudaSuccess;
    return launch_box_batch_t<BX_KC>(segs, nseg, total, smem, num_sms, st);
}

cudaError_t launch_gram_box(const KParams &P, int num_sms, cudaStream_t st)
{
    if (!gram_box_supported(P.nb, P.ny, P.nx) || P.cols <= 0 || P.pix_begin % P.cols || P.npix % P.cols)
        return cudaErrorInvalidValue;
    if (P.npix == 0) return cudaSuccess;
    return P.parts == 3 ? launch_box_t<BX_KC, 3>(P, num_sms, st) : launch_box_t<BX_KC, 2>(P, num_sms, st);
}

}  // namespace fpl
