// nmap.cu -- statistically homogeneous pixels (the nmap bitmask) on the GPU.
//
// Replaces the in-memory core of FRInGE's nmap module
// (src/nmap/nmap.cpp:345-473) and its GPU sketch (src/nmap/nmap_cuda.cu:
// 243-334, one thread per pixel with a bubble sort, not built by the
// reference).  For every pixel the amplitudes of its N dates are compared
// with those of each window neighbour by the two-sample Kolmogorov-Smirnov
// test (src/nmap/KS2sample.hpp:96-144); the neighbour's bit is set in the
// Ulongmask layout (include/fringe/ulongmask.hpp:55-74) when the test's
// probability is at least the threshold.
//
//   k_nmap_sort  (thread per pixel): amplitudes |x_b| / alpha_b exactly as
//                the reference forms them (the float modulus is
//                sqrt(x^2 + y^2) in FP64 rounded to float, the division by
//                the calibration constant in FP64), the validity mask
//                (nonzero, not NaN, optional input mask), and an ascending
//                bitonic sort in registers; sorted amplitudes are written
//                date-planar [N][pixel].
//   k_nmap_ks    (CTA per 32-column tile, a warp per two rows): the KS test of
//                each pixel against the neighbours of the forward half window
//                (the offsets of the reference's loop, src/nmap/nmap.cpp:
//                399-416: rows 0..Ny below, and on its own row the columns right
//                of it).  The probability depends on the statistic D alone (in
//                steps of 1/N; a run of equal values in both samples is one
//                step, as in the reference) and falls with it, so the test asks
//                only whether D reaches the smallest failing value, which the
//                host finds with the reference's Kolmogorov series.  The
//                results go to bit words of 32 columns.
//   k_nmap_ad    (CTA per 32-column tile, a warp per row): the same forward
//                tests with the two-sample Anderson-Darling
//                test (src/nmap/AD2unique.hpp:270-347).  The statistic is a
//                sum over the merged walk, (2n m_j - n(j+1))^2 /
//                ((j+1)(2n-j-1)) for the j+1 first values of which m_j come
//                from the first sample, and the p-value decreases with it:
//                the host finds the largest sum S* whose p-value, computed as
//                the reference computes it, passes the threshold.  Each
//                thread sums in FP32 and decides when it is clear of S* by
//                a margin above its rounding; otherwise it repeats the
//                reference's own FP64 sum, operation for operation, and
//                compares that with S*.  Ties are merged second sample
//                first, so the test is not symmetric: like the reference,
//                each pair is tested with the pixel whose forward half
//                window reaches the other as the first sample.
//   k_nmap_map   (warp per row and 32 columns): the map as the reference sets
//                it (nmap.cpp:447-462): a pixel's forward bits are its own
//                tests, its backward bits those of the neighbour whose
//                forward offset reaches it; the count is their sum.  Each
//                pair is tested once.
//
// 2048^2, N = 30, 11 x 21 (GB300): KS2 30.3 -> 3.66 ms (sort 0.47, tests 3.0,
// map 0.16; before: merge walks of about sixty dependent steps per pair, FP64
// moduli, bits gathered one at a time); AD2 at 701 x 1023, N = 17, 11 x 11:
// 2.07 -> 0.70 ms (sort 0.06, tests 0.56, map 0.02; 0.29 of the 1.37 ms is the host's
// table of p-values, which the context keeps: 0.98 ms where thresholds alternate).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "ctx.h"
#include "fringe_gb300.h"
#include "guard.h"

namespace fpl {
namespace {

constexpr int NM_TC = 32;            // tile columns (one warp per tile row)
constexpr int NM_MAX_TR = 16;        // AD2: tile rows at most (512 threads)
constexpr int NM_SORT_THREADS = 128;
constexpr int NM_AD_SM_WARPS = 48;   // AD2: warps per SM worth having
constexpr int KS_MAX_WARPS = 12;     // KS2: warps per CTA at most (168 registers per thread)

struct NmapParams {
    const float2 *stack;             // [nb][rows][cols]
    const uint8_t *mask;             // optional [rows][cols]
    float *sorted;                   // [nb][rows*cols]
    uint8_t *valid;                  // [rows*cols]
    uint32_t *nmap;                  // [rows*cols][nulong]
    uint32_t *fwd;                   // [rows][column groups][ntap]: forward half-window results (FwdWords)
    int32_t *count;                  // optional [rows*cols]
    double alpha[FPL_MAX_BANDS];     // normalised calibration constants
    float alpha_hi[FPL_MAX_BANDS], alpha_lo[FPL_MAX_BANDS];   // alpha = hi + lo to 2^-48
    int ks_fail;                     // KS2: smallest D that fails the threshold (n + 1: none)
    double ad_star;                  // AD2: largest walk sum whose p-value passes
    float ad_lo, ad_hi;              // AD2: FP32 sums below ad_lo pass, above ad_hi fail
    int ad_mode;                     // AD2: 0 compare, 1 every pair passes, 2 none does
    float ad_w[2 * FPL_MAX_BANDS];   // AD2: n^2 / ((j+1)(2n-j-1)), j < 2n - 1
    long long plane;
    int rows, cols, nb, ny, nx, nulong, tr, ntap, sp;   // sp: stride of the tile's samples (NmTile)
    int unit_alpha;                  // all constants 1: no division
};

// RN24(RN53(v)) for v = a + delta, where delta is known to within a * 2^-44:
// a + (delta -+ a 2^-43) round to the same float unless v lies within that
// distance of a midpoint (about one sample in 2^18), and rounding is
// monotone, so equal roundings settle the value without FP64.
__device__ __forceinline__ bool settled_sum(float a, float delta, float *out)
{
    const float m = a * 1.13686838e-13f;              // 2^-43
    const float lo = __fadd_rn(a, delta - m), hi = __fadd_rn(a, delta + m);
    *out = lo;
    return lo == hi;
}

// float modulus as the reference's std::abs(complex<float>): sqrt(x^2 + y^2)
// in FP64, rounded to float.  FP64 issues two operations per SM and clock
// here and took most of this kernel's time (5 of 6 ms at 2048^2, N = 30), so
// the value is formed in float-float (x^2 + y^2 to 2^-45, one Newton step from the
// FP32 root) and the FP64 chain runs only where that does not settle the rounding.
__device__ __forceinline__ float modulus_f64(float x, float y)
{
    float p = x * x, q = y * y;
    const float pe = fmaf(x, x, -p), qe = fmaf(y, y, -q);
    const float big = fmaxf(p, q), small = fminf(p, q);
    const float s = big + small;
    if (s >= 8.2718061e-25f && s <= 1.2676506e30f) {      // 2^-80 .. 2^100: no part under- or overflows
        const float lo = ((big - s) + small) + (pe + qe);
        const float a = __fsqrt_rn(s);
        const float r = fmaf(-a, a, s) + lo;              // (x^2 + y^2) - a^2
        float out;
        if (settled_sum(a, r * __fdividef(0.5f, a), &out)) return out;
    } else if (x == 0.f && y == 0.f) {
        return 0.f;
    }
    const double m2 = __dadd_rn(__dmul_rn((double)x, (double)x), __dmul_rn((double)y, (double)y));
    return __double2float_rn(__dsqrt_rn(m2));
}

// (float)((double)a / alpha), the reference's calibrated amplitude
// (nmap.cpp:374), alpha = ah + al to 2^-48: the quotient by ah and its
// remainder in FP32, FP64 where the rounding is not settled
__device__ __forceinline__ float calibrated(float a, double alpha, float ah, float al)
{
    if (a >= 1e-10f && a <= 1e10f && ah >= 1e-6f && ah <= 1e6f) {
        const float q = __fdiv_rn(a, ah);
        const float r = fmaf(-q, ah, a) - q * al;         // a - q alpha
        float out;
        if (settled_sum(q, __fdividef(r, ah), &out)) return out;
    }
    return __double2float_rn(__ddiv_rn((double)a, alpha));
}

template <int NPAD>
__global__ void __launch_bounds__(NM_SORT_THREADS) k_nmap_sort(NmapParams P)
{
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= P.plane) return;
    // the moduli go through shared memory (a column per thread), so that the
    // loop over dates stays rolled: unrolled, its code and the sort's outgrew the
    // instruction cache
    __shared__ float stage[NPAD][NM_SORT_THREADS];
    float *mine = &stage[0][threadIdx.x];
    bool ok = P.mask ? P.mask[q] != 0 : true;
    const float2 *src = P.stack + q;
#pragma unroll 1
    for (int b0 = 0; b0 < P.nb; b0 += 8) {
        float2 x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            x[u] = make_float2(1.f, 0.f);
            if (b0 + u < P.nb) x[u] = __ldg(src + (b0 + u) * P.plane);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (b0 + u >= P.nb) break;
            float a = modulus_f64(x[u].x, x[u].y);
            if (!P.unit_alpha) a = calibrated(a, P.alpha[b0 + u], P.alpha_hi[b0 + u], P.alpha_lo[b0 + u]);
            ok = ok && a != 0.f && !isnan(a);
            mine[(b0 + u) * NM_SORT_THREADS] = a;
        }
    }
    float v[NPAD];
#pragma unroll
    for (int b = 0; b < NPAD; ++b) v[b] = b < P.nb ? mine[b * NM_SORT_THREADS] : INFINITY;
    P.valid[q] = ok ? 1 : 0;
    if (!ok) return;
    // ascending bitonic sort (padding +inf stays at the end)
#pragma unroll
    for (int k = 2; k <= NPAD; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll
            for (int i = 0; i < NPAD; ++i) {
                const int l = i ^ j;
                if (l > i) {
                    const float a = v[i], c = v[l];
                    if ((i & k) == 0) {
                        v[i] = fminf(a, c);
                        v[l] = fmaxf(a, c);
                    } else {
                        v[i] = fmaxf(a, c);
                        v[l] = fminf(a, c);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int b = 0; b < NPAD; ++b)
        if (b < P.nb) P.sorted[b * P.plane + q] = v[b];
}

// Sorted amplitudes and validity of a tile (rows R0 .. R0 + HH - 1, columns
// C0 - nx .. C0 + 31 + nx) in shared memory: date b of tile pixel h at
// S[b * db + h * dh], V[HH * HW].  Each warp copies whole (date, row) runs,
// asynchronously: loads through registers left one in flight per warp, and
// the tile's load took as long as its tests (k_nmap_ks 1.14 -> 0.79 ms at
// 1024^2, N = 30).
__device__ __forceinline__ void nm_load_tile(const NmapParams &P, float *S, uint8_t *V, int R0, int C0, int HW, int HH,
                                             int db, int dh)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    int b = 0, hr = warp;
    for (;;) {
        while (hr >= HH) { hr -= HH; ++b; }
        if (b > P.nb) break;
        const int r = R0 + hr;
        const long long row = (long long)r * P.cols;
        for (int hc = lane; hc < HW; hc += 32) {
            const int c = C0 - P.nx + hc;
            const bool in = r < P.rows && c >= 0 && c < P.cols;
            if (b == P.nb) {
                V[hr * HW + hc] = in ? P.valid[row + c] : 0;
            } else {
                // zero-filled outside the scene
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(S + b * db + (hr * HW + hc) * dh);
                const float *src = P.sorted + (in ? b * P.plane + row + c : 0);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"(dst), "l"(src), "r"(in ? 4 : 0) : "memory");
            }
        }
        hr += nw;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// The forward results: one word per (row, 32-column group, forward tap), bit
// c of it for column c of the group.  Lane l of a warp keeps the ballot of
// tap 32 q + l and the warp stores 32 taps together.
struct FwdWords {
    uint32_t *out;       // words of this row and group
    uint32_t keep;
    __device__ __forceinline__ void put(bool set, int g, int glast, int lane)
    {
        const uint32_t m = __ballot_sync(0xffffffffu, set);
        if (lane == (g & 31)) keep = m;
        if ((g & 31) == 31 || g == glast) {
            if (out && lane <= (g & 31)) out[(g & ~31) + lane] = keep;
        }
    }
};
__device__ __forceinline__ FwdWords fwd_words(const NmapParams &P, int r, int tc)
{
    const int ntc = (P.cols + NM_TC - 1) / NM_TC;
    return FwdWords{r < P.rows ? P.fwd + ((long long)r * ntc + tc) * P.ntap : nullptr, 0u};
}

// Two-sample KS test, forward half window (see the file comment).  For
// samples a, b of n ascending values the statistic D = max_x |#{a <= x} -
// #{b <= x}| reaches k exactly when a_{i+k-1} < b_i or b_{i+k-1} < a_i for
// some i in [0, n-k] (x = the smaller value): no merge of the samples is needed.  With
// k the smallest D that fails the threshold, a pair fails iff some b_j lies
// above U_j = a_{j+k-1} or below L_j = a_{j-k+1} (+-inf where there is no
// such value).  The thread keeps U and L of PX vertically adjacent pixels in
// registers and reads each neighbour's b once for all of them; the sign bits
// of U_j - b_j and b_j - L_j are collected with one three-input OR (the FP32
// compare into a predicate issues at a quarter of the rate of these adds).
// No branch depends on the data.  An infinite b or bound gives inf - inf =
// NaN with a clear sign, the answer for equal values.  VEC: a pixel's dates
// lie P.sp floats apart from the next pixel's, P.sp = 2 mod 4, so that 32
// lanes' 8-byte loads fall in distinct banks and every date is an immediate
// offset; otherwise single loads, no padding (windows that fit no other way).
template <int NPAD, int PX, bool VEC>
__global__ void __launch_bounds__(32 * KS_MAX_WARPS, NPAD <= 16 ? 2 : 1) k_nmap_ks(NmapParams P)
{
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int NG = NPAD / 8;                      // groups of 8 dates
    static_assert(PX <= 2, "rows of the first, all, and the last pixel");
    const int HW = NM_TC + 2 * P.nx, HH = P.tr + P.ny, sp = P.sp;
    float *S = reinterpret_cast<float *>(smem);                                  // [HH * HW][sp]
    uint8_t *V = smem + sizeof(float) * (size_t)(HH * HW) * sp;                  // [HH * HW]
    const int ntc = (P.cols + NM_TC - 1) / NM_TC;
    const int tc = blockIdx.x % ntc, R0 = (blockIdx.x / ntc) * P.tr, C0 = tc * NM_TC;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    nm_load_tile(P, S, V, R0, C0, HW, HH, 1, sp);
    __syncthreads();
    const int wx = 2 * P.nx + 1, n = P.nb, k = P.ks_fail;
    const int r0 = R0 + PX * warp, c = C0 + lane;
    const int hp = PX * warp * HW + lane + P.nx;      // first pixel of the thread
    float U[PX][NPAD], Lo[PX][NPAD];
    bool pv[PX];
    FwdWords fw[PX];
#pragma unroll
    for (int u = 0; u < PX; ++u) {
        pv[u] = c < P.cols && r0 + u < P.rows && V[hp + u * HW] != 0;
        fw[u] = fwd_words(P, r0 + u, tc);
        const float *own = S + (hp + u * HW) * sp;
#pragma unroll
        for (int j = 0; j < NPAD; ++j) {
            const int ju = j + k - 1, jl = j - k + 1;
            U[u][j] = ju < n ? own[ju] : INFINITY;
            Lo[u][j] = (jl >= 0 && j < n) ? own[jl] : -INFINITY;
        }
    }
    const uint32_t Sa = (uint32_t)__cvta_generic_to_shared(S), Va = (uint32_t)__cvta_generic_to_shared(V);
    // groups with a bound: U in [0, n - k], L in [k - 1, n)
    const int gu = k <= n ? (n - k) / 8 : -1, gl = k <= n ? (k - 1) / 8 : NG, gn = (n - 1) / 8;
    const int glast = P.ny * wx + P.nx;
    // the pixels of mask M against the neighbour whose sample is at q.  Past
    // date n - 1 the loads run into the next pixel's sample (or the validity
    // bytes): whatever is there passes the infinite bounds, NaN included.
    auto test = [&](auto mask, uint32_t q, int (&acc)[PX]) {
        constexpr int M = decltype(mask)::value;
#pragma unroll
        for (int u = 0; u < PX; ++u) acc[u] = 0;
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            if (g > gn) break;
            float b[8];
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const uint32_t a = q + 4 * (8 * g + j);
                if (VEC) {
                    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(b[j]), "=f"(b[j + 1]) : "r"(a));
                } else {
                    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(b[j]) : "r"(a));
                    asm volatile("ld.shared.f32 %0, [%1 + 4];" : "=f"(b[j + 1]) : "r"(a));
                }
            }
            if (g <= gu) {
#pragma unroll
                for (int u = 0; u < PX; ++u)
                    if (M >> u & 1) {
#pragma unroll
                        for (int j = 0; j < 8; j += 2)
                            acc[u] |= __float_as_int(U[u][8 * g + j] - b[j]) |
                                      __float_as_int(U[u][8 * g + j + 1] - b[j + 1]);
                    }
            }
            if (g >= gl) {
#pragma unroll
                for (int u = 0; u < PX; ++u)
                    if (M >> u & 1) {
#pragma unroll
                        for (int j = 0; j < 8; j += 2)
                            acc[u] |= __float_as_int(b[j] - Lo[u][8 * g + j]) |
                                      __float_as_int(b[j + 1] - Lo[u][8 * g + j + 1]);
                    }
            }
        }
    };
    // neighbours of row rr below the thread's first pixel, columns from j0 on;
    // pixel u reaches them with the row offset rr - u
    auto row = [&](auto mask, int rr, int j0) {
        constexpr int M = decltype(mask)::value;
        const int hq = hp + rr * HW + j0;
        uint32_t q = Sa + 4 * hq * sp, v = Va + hq;
#pragma unroll 1
        for (int jj = j0; jj <= P.nx; ++jj, ++v, q += 4 * sp) {
            uint32_t qv;
            asm volatile("ld.shared.u8 %0, [%1];" : "=r"(qv) : "r"(v));
            int acc[PX];
            test(mask, q, acc);
#pragma unroll
            for (int u = 0; u < PX; ++u) {
                const int tap = (rr - u) * wx + jj;             // forward tap of pixel u
                // the centre is set whatever the test says (nmap.cpp:441-445)
                if ((M >> u & 1) && tap >= 0) fw[u].put(pv[u] && qv != 0 && (acc[u] >= 0 || tap == 0), tap, glast, lane);
            }
        }
    };
    row(std::integral_constant<int, 1>{}, 0, 0);
#pragma unroll 1
    for (int rr = 1; rr <= P.ny; ++rr) row(std::integral_constant<int, (1 << PX) - 1>{}, rr, -P.nx);
    if (PX == 2) row(std::integral_constant<int, 2>{}, P.ny + 1, -P.nx);
}

// AD2: the walk sum of the first sample a over the merged order of two
// ascending samples (ties: b first), in FP32: the terms d^2 w_j, d = 2 m_j -
// (j + 1).  The merge runs from both ends at once: the first n merged values
// need no bounds checks (neither sample can run out before), nor do the last
// n - 1, whose d from the end has the same square, and w_j = w_{2n-2-j}; the two
// chains of dependent loads overlap.  Issue-bound (84% of the slots): 13
// instructions per merged value.  a0, b0: shared-memory addresses of the samples, stb:
// bytes between their dates.
__device__ __forceinline__ float ad_walk_fast(uint32_t a0, uint32_t b0, uint32_t stb, int n, const float *w)
{
    // one step of each chain, predicated: the taken sample's pointer moves on
    // and its next value is loaded; d is +1 for the first sample, -1 for the second
    auto fwd = [&](uint32_t &pa, uint32_t &pb, float &va, float &vb) {
        float d;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %2, %3;\n\t@p add.u32 %0, %0, %5;\n\t@!p add.u32 %1, %1, %5;\n\t"
                     "@p ld.shared.f32 %2, [%0];\n\t@!p ld.shared.f32 %3, [%1];\n\tselp.f32 %4, 0f3F800000, 0fBF800000, p;\n\t}"
                     : "+r"(pa), "+r"(pb), "+f"(va), "+f"(vb), "=f"(d) : "r"(stb));
        return d;
    };
    auto bwd = [&](uint32_t &qa, uint32_t &qb, float &ya, float &yb) {
        float d;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.f32 p, %2, %3;\n\t@p sub.u32 %0, %0, %5;\n\t@!p sub.u32 %1, %1, %5;\n\t"
                     "@p ld.shared.f32 %2, [%0];\n\t@!p ld.shared.f32 %3, [%1];\n\tselp.f32 %4, 0f3F800000, 0fBF800000, p;\n\t}"
                     : "+r"(qa), "+r"(qb), "+f"(ya), "+f"(yb), "=f"(d) : "r"(stb));
        return d;
    };
    auto at = [](uint32_t p) {
        float v;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(p));
        return v;
    };
    uint32_t qa = a0 + (n - 1) * stb, qb = b0 + (n - 1) * stb;
    float va = at(a0), vb = at(b0), ya = at(qa), yb = at(qb), df = 0.f, db = 0.f, s = 0.f;
#pragma unroll 8
    for (int t = 0; t < n - 1; ++t) {
        df += fwd(a0, b0, va, vb);
        db += bwd(qa, qb, ya, yb);
        s = fmaf(fmaf(db, db, df * df), w[t], s);
    }
    df += (va < vb) ? 1.f : -1.f;
    return fmaf(df * df, w[n - 1], s);
}

// The same sum as the reference evaluates it (src/nmap/AD2unique.hpp:
// 295-309), operation for operation in FP64: bit-identical to the host's.
__device__ __noinline__ double ad_walk_exact(const float *A, const float *B, int st, int n)
{
    int ia = 0, ib = 0;
    const double N = 2.0 * n, dn = n;
    double m = 0.0, s = 0.0;
    for (int j = 0; j < 2 * n - 1; ++j) {
        const bool ta = ia < n && (ib >= n || A[ia * st] < B[ib * st]);
        if (ta) ++ia; else ++ib;
        m = __dadd_rn(m, ta ? 1.0 : 0.0);
        const double bj = j + 1;
        const double t = __dsub_rn(__dmul_rn(N, m), __dmul_rn(dn, bj));
        s = __dadd_rn(s, __ddiv_rn(__dmul_rn(t, t), __dmul_rn(bj, __dsub_rn(N, bj))));
    }
    return s;
}

// Two-sample AD test, forward half window: thread per pixel, one warp per
// row of the tile, both samples walked in shared memory.
__global__ void __launch_bounds__(NM_TC * NM_MAX_TR) k_nmap_ad(NmapParams P)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int HW = NM_TC + 2 * P.nx, HH = P.tr + P.ny, sp = P.sp;
    float *S = reinterpret_cast<float *>(smem);                                  // [nb][sp]
    uint8_t *V = smem + sizeof(float) * (size_t)P.nb * sp;                       // [HH * HW]
    const int ntc = (P.cols + NM_TC - 1) / NM_TC;
    const int tc = blockIdx.x % ntc, R0 = (blockIdx.x / ntc) * P.tr, C0 = tc * NM_TC;
    const int tr = threadIdx.x >> 5, lane = threadIdx.x & 31;
    nm_load_tile(P, S, V, R0, C0, HW, HH, sp, 1);
    __syncthreads();
    const int r = R0 + tr, c = C0 + lane;
    if (r >= P.rows) return;
    const int wx = 2 * P.nx + 1, glast = P.ny * wx + P.nx;
    FwdWords fw = fwd_words(P, r, tc);
    const uint32_t Sa = (uint32_t)__cvta_generic_to_shared(S);
    const int hp = tr * HW + lane + P.nx;
    const bool pv = c < P.cols && V[hp] != 0;
    int ii = 0, jj = 0;                               // offset of forward tap g
    for (int g = 0; g <= glast; ++g) {
        const int hq = hp + ii * HW + jj;
        bool set = false;
        if (pv && V[hq]) {
            if (g == 0) {
                set = true;                                  // the centre (nmap.cpp:441-445)
            } else if (P.ad_mode != 0) {
                set = P.ad_mode == 1;
            } else {
                // this pixel is the reference's first sample
                const float sf = ad_walk_fast(Sa + 4 * hp, Sa + 4 * hq, 4 * sp, P.nb, P.ad_w);
                if (sf < P.ad_lo) set = true;
                else if (sf > P.ad_hi) set = false;
                else set = ad_walk_exact(S + hp, S + hq, sp, P.nb) <= P.ad_star;
            }
        }
        fw.put(set, g, glast, lane);
        if (++jj > P.nx) {
            jj = -P.nx;
            ++ii;
        }
    }
}

// The map and count of every pixel from the forward results: a warp takes
// the 32 columns of a group of one row.  Lane l fetches tap 32 w + l of the
// whole group as one word -- a forward tap is the group's own, a backward
// one (nmap.cpp:459) the mirrored tap of the row above it, shifted by the column
// offset -- and a 32 x 32 bit transposition over the warp turns 32 taps of 32
// pixels into one map word per pixel.  The words are written through shared
// memory as one contiguous run.  Gathering every pixel's bits one at a time
// took 41 instructions per tap: 0.31 -> 0.04 ms at 1024^2, 11 x 21.
constexpr int MAP_WARPS = 8;
__global__ void __launch_bounds__(32 * MAP_WARPS) k_nmap_map(NmapParams P)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ntc = (P.cols + NM_TC - 1) / NM_TC;
    const long long item = (long long)blockIdx.x * MAP_WARPS + warp;
    if (item >= (long long)P.rows * ntc) return;
    const int r = int(item / ntc), tc = int(item - (long long)r * ntc), C0 = tc * NM_TC;
    const int wx = 2 * P.nx + 1, K = (2 * P.ny + 1) * wx, fc = P.ny * wx + P.nx, nul = P.nulong;
    uint32_t *buf = reinterpret_cast<uint32_t *>(smem) + warp * 32 * (nul | 1);   // odd rows: no bank conflicts
    int cnt = 0;
    for (int w = 0; w < nul; ++w) {
        const int f = 32 * w + lane;
        uint32_t m = 0;
        if (f >= fc && f < K) {
            m = __ldg(P.fwd + item * P.ntap + (f - fc));
        } else if (f < fc) {
            const int g = fc - f, ii = (g + P.nx) / wx, jj = g - ii * wx;
            const int pos = C0 - jj, rs = r - ii;             // group columns read bits pos .. pos + 31
            const int wl = pos >> 5;
            if (rs >= 0) {
                const uint32_t *src = P.fwd + (long long)rs * ntc * P.ntap + g;
                const uint32_t lo = (wl >= 0 && wl < ntc) ? __ldg(src + (long long)wl * P.ntap) : 0u;
                const uint32_t hi = (wl + 1 >= 0 && wl + 1 < ntc) ? __ldg(src + (long long)(wl + 1) * P.ntap) : 0u;
                m = __funnelshift_r(lo, hi, pos & 31);
            }
        }
        // bit b of lane l -> bit l of lane b
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
            const uint32_t keep = s == 16 ? 0x0000ffffu : s == 8 ? 0x00ff00ffu : s == 4 ? 0x0f0f0f0fu : s == 2 ? 0x33333333u : 0x55555555u;
            const uint32_t y = __shfl_xor_sync(0xffffffffu, m, s);
            m = (lane & s) ? ((m & ~keep) | ((y >> s) & keep)) : ((m & keep) | ((y << s) & ~keep));
        }
        cnt += __popc(m);
        buf[lane * (nul | 1) + w] = m;
    }
    __syncwarp();
    const int ncol = min(NM_TC, P.cols - C0);
    const long long q0 = (long long)r * P.cols + C0;
    if (P.count && lane < ncol) P.count[q0 + lane] = cnt;
    uint32_t *out = P.nmap + q0 * nul;
    int px = lane / nul, w = lane - px * nul;
    const int dp = 32 / nul, dw = 32 - dp * nul;
    for (int e = lane; e < ncol * nul; e += 32) {
        out[e] = buf[px * (nul | 1) + w];
        px += dp;
        w += dw;
        if (w >= nul) { w -= nul; ++px; }
    }
}

// The Kolmogorov distribution as the reference evaluates it
// (src/nmap/KS2sample.hpp:42-78, ROOT's KolmogorovProb series).
double kolmogorov_prob(double z)
{
    const double u = std::fabs(z);
    if (u < 0.2) return 1.0;
    if (u < 0.755) {
        const double v = 1.0 / (u * u);
        return 1.0 - 2.50662827 * (std::exp(-1.2337005501361697 * v) + std::exp(-11.103304951225528 * v) +
                                   std::exp(-30.842513753404244 * v)) / u;
    }
    if (u < 6.8116) {
        double r[4] = {0.0, 0.0, 0.0, 0.0};
        const double v = u * u;
        const int maxj = std::max(1, (int)std::round(3.0 / u));
        for (int j = 0; j < maxj; ++j) r[j] = std::exp(-2.0 * (j + 1) * (j + 1) * v);
        return 2.0 * (r[0] - r[1] + r[2] - r[3]);
    }
    return 0.0;
}

// Decisions for D = 0..n.  The reference accumulates the statistic as a
// double sum of +-1/n steps, which lands within a few units in the last
// place of k/n; a table entry is accepted only when the decision is the
// same over that whole interval (false: the threshold sits on the rounding
// of a table value).
// ---- AD2: the reference's p-value as a function of the walk sum ----------
// Scholz & Stephens (1987), "K-sample Anderson-Darling tests", JASA 82:918:
// the m = 1 column of their table of critical points of the standardised
// statistic (the entries the reference reads, src/nmap/AD2unique.hpp:8-48
// at indices 0, 8, .., 272), with the upper-tail probabilities it lists.
const double kAdCrit[35] = {
    -1.1954, -1.1786, -1.166, -1.1407, -1.1253, -1.0777, -1.0489, -0.9978, -0.9417, -0.8981, -0.8598, -0.7258,
    -0.5966, -0.4572, -0.2966, -0.1009, 0.1571, 0.5357, 1.2255, 1.5262, 1.9633, 2.7314, 3.7825, 4.1241, 4.6044,
    5.409, 6.4954, 6.8279, 7.2755, 8.1885, 9.3061, 9.6132, 10.0989, 10.8825, 11.8537};
const double kAdProb[35] = {
    .00001, .00005, .0001, .0005, .001, .005, .01, .025, .05, .075, .1, .2, .3, .4, .5, .6, .7, .8, .9,
    .925, .95, .975, .99, .9925, .995, .9975, .999, .99925, .9995, .99975, .9999, .999925, .99995, .999975,
    .99999};

// sigma_N of the standardised statistic (Scholz & Stephens eq. 4, k = 2,
// both samples of n; N = 2n < 2000, harmonic sums summed in the
// reference's order, src/nmap/AD2unique.hpp:173-219)
double ad_sigma(int n)
{
    const int N = 2 * n;
    const double kk = 2.0, H = 1.0 / (1.0 * n) + 1.0 / (1.0 * n);
    std::vector<double> inv(N > 1 ? N : 2, 0.0);
    double h = 0.0, g = 0.0;
    for (int i = 1; i < N; ++i) {
        inv[i] = 1.0 / i;
        h += inv[i];
    }
    for (int i = 1; i < N - 1; ++i) {
        const double t = inv[N - i];
        for (int j = i + 1; j < N; ++j) g += t * inv[j];
    }
    const double k2 = kk * kk;
    const double a = (4 * g - 6) * (kk - 1) + (10 - 6 * g) * H;
    const double b = (2 * g - 4) * k2 + 8 * h * kk + (2 * g - 14 * h - 4) * H - 8 * h + 4 * g - 6;
    const double c = (6 * h + 2 * g - 2) * k2 + (4 * h - 4 * g + 6) * kk + (2 * h - 6) * H + 4 * h;
    const double d = (2 * h + 6) * k2 - 4 * h * kk;
    const double dN = (double)N;
    double s2 = 0.0;
    s2 += a * (dN * dN * dN) + b * (dN * dN) + c * N + d;
    s2 /= ((double)(N - 1) * (double)(N - 2) * (double)(N - 3));
    return std::sqrt(s2);
}

// the reference's p-value of the standardised statistic t (linear in
// log((1 - p) / p) between the table's points, extrapolated past its ends)
double ad_pvalue(double t)
{
    int i1 = -1;
    for (int i = 0; i < 35; ++i) {
        i1 = i - 1;
        if (t <= kAdCrit[i]) break;
    }
    int i2 = i1 + 1;
    if (i1 < 0) { i1 = 0; i2 = 1; }
    if (i2 >= 35) { i1 = 33; i2 = 34; }
    const double l1 = std::log((1.0 - kAdProb[i1]) / kAdProb[i1]), l2 = std::log((1.0 - kAdProb[i2]) / kAdProb[i2]);
    const double t1 = kAdCrit[i1], t2 = kAdCrit[i2];
    const double l0 = (l1 - l2) * (t - t2) / (t1 - t2) + l2;
    return std::exp(l0) / (1. + std::exp(l0));
}

// does the walk sum s of a pair of n-date samples pass? (the chain of
// src/nmap/AD2unique.hpp:333-345: both samples' sums are s)
bool ad_pass(double s, int n, double sigma, double prob)
{
    double akn = 0.0;
    akn = akn + s / (n * 1.0);
    akn = akn + s / (n * 1.0);
    akn = akn / (2.0 * n);
    double t = akn - 1;
    t /= sigma;
    return ad_pvalue(t) >= prob;
}

// AD2 decision for this stack depth and threshold: the largest passing sum
// S* (the pass set is every sum up to it); false when the decisions
// within 4096 units in the last place of S* are not all on their side of it
// (the threshold sits on the rounding of the p-value there).
bool ad_table(int n, double prob, NmapParams *P)
{
    const double sigma = ad_sigma(n);
    std::memset(P->ad_w, 0, sizeof(P->ad_w));
    for (int j = 0; j < 2 * n - 1; ++j)
        P->ad_w[j] = (float)((double)n * n / ((double)(j + 1) * (double)(2 * n - j - 1)));
    const double top = 1e300;
    const bool p0 = ad_pass(0.0, n, sigma, prob), p1 = ad_pass(top, n, sigma, prob);
    P->ad_star = 0.0;
    P->ad_lo = P->ad_hi = 0.f;
    if (p0 == p1) {                       // one decision for every sum
        P->ad_mode = p0 ? 1 : 2;
        for (int k = 0; k < 64; ++k)
            if (ad_pass(top * k / 64.0, n, sigma, prob) != p0) return false;
        return true;
    }
    if (!p0) return false;                // the p-value must fall with the sum
    auto bits = [](double x) { uint64_t u; std::memcpy(&u, &x, 8); return u; };
    auto val = [](uint64_t u) { double x; std::memcpy(&x, &u, 8); return x; };
    uint64_t lo = bits(0.0), hi = bits(top);
    while (hi - lo > 1) {
        const uint64_t mid = lo + (hi - lo) / 2;
        if (ad_pass(val(mid), n, sigma, prob)) lo = mid; else hi = mid;
    }
    for (int64_t k = -4096; k <= 4096; ++k) {
        const int64_t u = (int64_t)lo + k;
        if (u < 0) continue;
        if (ad_pass(val((uint64_t)u), n, sigma, prob) != (k <= 0)) return false;
    }
    const double star = val(lo);
    P->ad_star = star;
    // the FP32 sum of n positive terms rounds by at most (n + 2) 2^-24 of its value
    const double band = (2 * n + 16) * 1.1920929e-7;
    P->ad_lo = (float)(star * (1.0 - band));
    P->ad_hi = (float)(star * (1.0 + band));
    P->ad_mode = 0;
    return true;
}

// The probabilities fall with D (checked for every depth up to 64 dates), so
// the decision is one number: the smallest D that fails.
bool ks_table(int n, double prob, int *fail)
{
    *fail = n + 1;
    const double rn = n, s = 1.0 / rn, scale = std::sqrt(rn * rn / (rn + rn));
    for (int k = 0; k <= n; ++k) {
        double acc = 0.0;
        for (int t = 0; t < k; ++t) acc += s;
        const double cand[4] = {acc, k * s, acc * (1.0 - 64 * 1.2e-16), acc * (1.0 + 64 * 1.2e-16)};
        int pass = -1;
        for (double x : cand) {
            const int p = kolmogorov_prob(x * scale) >= prob ? 1 : 0;
            if (pass < 0) pass = p;
            else if (p != pass) return false;
        }
        if (!pass && k < *fail) *fail = k;
    }
    return true;
}

constexpr size_t NM_SMEM_CTA = 227 * 1024, NM_SMEM_SM = 228 * 1024;

// Tile of the forward kernels: tr rows (px per warp) of 32 columns.  The
// samples lie sp floats apart: KS2 from pixel to pixel, at least n and 2 mod
// 4; AD2 from date to date, a multiple of 32 (lanes on consecutive columns
// never meet in a bank, whatever dates their walks have reached); packed: no
// padding.  The height with the most warps resident per SM (up to sm_warps), two CTAs before
// one, so that one's loads overlap the other's tests, and the taller tile,
// which shares its apron among more pixels; lower when the scene would leave
// SMs without a tile.  false when not even one warp's rows fit.
struct NmTile {
    int warps, tr, sp;
    size_t smem;
};
NmTile nm_tile(int warps, int px, int n, int ny, int nx, bool ad2, bool packed)
{
    NmTile t;
    t.warps = warps;
    t.tr = warps * px;
    const size_t hp = (size_t)(NM_TC + 2 * nx) * (t.tr + ny);
    const size_t sp = ad2 ? (packed ? hp : (hp + 31) & ~size_t(31)) : (packed ? n : (n + 1) / 4 * 4 + 2);
    t.sp = (int)sp;
    t.smem = sizeof(float) * (ad2 ? (size_t)n : hp) * sp + hp;
    return t;
}
bool nm_pick_tile(int cta_warps, int sm_warps, int px, int n, int ny, int nx, int rows, int cols, int num_sms,
                  bool ad2, bool packed, NmTile *best)
{
    int best_score = -1;
    for (int w = 1; w <= cta_warps; ++w) {
        const NmTile t = nm_tile(w, px, n, ny, nx, ad2, packed);
        if (t.smem > NM_SMEM_CTA) break;
        const int ctas = (int)std::min<size_t>(NM_SMEM_SM / (t.smem + 1024), sm_warps / w);
        const int resident = std::max(1, ctas) * w;
        const long long tiles = (long long)((cols + NM_TC - 1) / NM_TC) * ((rows + t.tr - 1) / t.tr);
        if (best_score >= 0 && tiles < num_sms) break;
        const int score = 16 * resident + (ctas >= 2 ? 12 : 0);
        if (score >= best_score) {
            best_score = score;
            *best = t;
        }
    }
    return best_score >= 0;
}

// raises a kernel's shared-memory limit, once per device
template <typename K> cudaError_t nm_configure(K kern, bool *done)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || (dev < 64 && done[dev])) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)NM_SMEM_CTA);
    if (e == cudaSuccess && dev < 64) done[dev] = true;
    return e;
}

template <int NPAD, int PX, bool VEC> cudaError_t nm_launch_ks(const NmapParams &P, const NmTile &t, cudaStream_t st)
{
    static bool done[64] = {false};
    cudaError_t e = nm_configure(k_nmap_ks<NPAD, PX, VEC>, done);
    if (e != cudaSuccess) return e;
    const long long ntiles = (long long)((P.cols + NM_TC - 1) / NM_TC) * ((P.rows + t.tr - 1) / t.tr);
    k_nmap_ks<NPAD, PX, VEC><<<(unsigned)ntiles, 32 * t.warps, t.smem, st>>>(P);
    return cudaGetLastError();
}

cudaError_t nm_launch_ad(const NmapParams &P, const NmTile &t, cudaStream_t st)
{
    static bool done[64] = {false};
    cudaError_t e = nm_configure(k_nmap_ad, done);
    if (e != cudaSuccess) return e;
    const long long ntiles = (long long)((P.cols + NM_TC - 1) / NM_TC) * ((P.rows + t.tr - 1) / t.tr);
    k_nmap_ad<<<(unsigned)ntiles, 32 * t.warps, t.smem, st>>>(P);
    return cudaGetLastError();
}

}  // namespace
}  // namespace fpl

extern "C" int fpl_nmap(fpl_ctx *ctx, const fpl_nmap_job *job)
{
    return fpl_guard([&]() -> int {
        using namespace fpl;
        if (!ctx || !job || !job->stack || !job->nmap) return FPL_ERR_NULL;
        if (job->rows <= 0 || job->cols <= 0 || job->nbands <= 0 || job->half_window_x < 0 ||
            job->half_window_y < 0)
            return FPL_ERR_OPTIONS;
        if (job->memory != FPL_MEM_HOST && job->memory != FPL_MEM_DEVICE) return FPL_ERR_OPTIONS;
        if (!(job->prob >= 0.0) || job->prob > 1.0) return FPL_ERR_OPTIONS;
        if (job->nbands > FPL_MAX_BANDS) return FPL_ERR_UNSUPPORTED;
        const int wx = 2 * job->half_window_x + 1, K = (2 * job->half_window_y + 1) * wx;
        const int nul = (K + 31) / 32;
        if (nul > FPL_MAX_NULONG) return FPL_ERR_UNSUPPORTED;
        NmapParams P;
        std::memset(&P, 0, sizeof(P));
        P.rows = job->rows;
        P.cols = job->cols;
        P.nb = job->nbands;
        P.ny = job->half_window_y;
        P.nx = job->half_window_x;
        P.nulong = nul;
        P.plane = (long long)job->rows * job->cols;
        // calibration constants normalised to the first band (nmap.cpp:204-230)
        double a[FPL_MAX_BANDS];
        for (int b = 0; b < P.nb; ++b) {
            const double cst = job->amp_const ? job->amp_const[b] : 1.0;
            a[b] = cst > 0.0 ? cst : 1.0;
        }
        const double a0 = a[0];
        for (int b = 0; b < P.nb; ++b) a[b] /= a0;
        a[0] = 1.0;
        P.unit_alpha = 1;
        for (int b = 0; b < P.nb; ++b) {
            P.alpha[b] = a[b];
            P.alpha_hi[b] = (float)a[b];
            P.alpha_lo[b] = (float)(a[b] - (double)P.alpha_hi[b]);
            if (a[b] != 1.0) P.unit_alpha = 0;
        }
        if (job->method != FPL_NMAP_KS2 && job->method != FPL_NMAP_AD2) return FPL_ERR_OPTIONS;
        const bool ad2 = job->method == FPL_NMAP_AD2;
        if (!ad2 && !ks_table(P.nb, job->prob, &P.ks_fail)) {
            ctx->last_error = "the threshold lies within rounding of a Kolmogorov table value for this stack depth";
            return FPL_ERR_OPTIONS;
        }
        if (ad2) {
            // the boundary depends on the depth and the threshold alone, and
            // checking it takes 8,000 p-values: the context keeps the last one
            NmapAdPlan &plan = ctx->nmap_ad;
            if (plan.n != P.nb || plan.prob != job->prob) {
                plan.n = 0;
                if (!ad_table(P.nb, job->prob, &P)) {
                    ctx->last_error =
                        "the threshold lies within rounding of the Anderson-Darling p-value for this stack depth";
                    return FPL_ERR_OPTIONS;
                }
                plan.star = P.ad_star;
                plan.lo = P.ad_lo;
                plan.hi = P.ad_hi;
                plan.mode = P.ad_mode;
                std::memcpy(plan.w, P.ad_w, sizeof(plan.w));
                plan.prob = job->prob;
                plan.n = P.nb;
            }
            P.ad_star = plan.star;
            P.ad_lo = plan.lo;
            P.ad_hi = plan.hi;
            P.ad_mode = plan.mode;
            std::memcpy(P.ad_w, plan.w, sizeof(plan.w));
        }
        if (cudaSetDevice(ctx->device) != cudaSuccess) return FPL_ERR_CUDA;
        // KS2: pixels per thread by the registers their bounds take.  Windows
        // so tall that the padded tile does not fit: one pixel per thread, packed.
        const int ks_px = P.nb <= 32 ? 2 : 1;
        NmTile tile = {};
        bool packed = false;
        auto pick = [&](int cta_warps, int sm_warps, int px) {
            return nm_pick_tile(cta_warps, sm_warps, px, P.nb, P.ny, P.nx, P.rows, P.cols, ctx->num_sms, ad2, packed, &tile);
        };
        bool fits = ad2 ? pick(NM_MAX_TR, NM_AD_SM_WARPS, 1)
                        : pick(KS_MAX_WARPS, P.nb <= 16 ? 2 * KS_MAX_WARPS : KS_MAX_WARPS, ks_px);
        if (!fits) {
            packed = true;
            fits = pick(1, 1, 1);
        }
        if (!fits) return FPL_ERR_UNSUPPORTED;
        P.tr = tile.tr;
        P.sp = tile.sp;
        cudaStream_t st = ctx->stream;
        const size_t b_stack = (size_t)P.plane * P.nb * 8, b_nmap = (size_t)P.plane * nul * 4;
        const size_t b_sorted = ((size_t)P.plane * P.nb * 4 + 255) & ~size_t(255);   // keeps every region 256-aligned
        // scratch: sorted amplitudes | validity | forward results | (host jobs)
        // mask, stack, nmap, count
        P.ntap = K - (P.ny * wx + P.nx);
        const size_t b_fwd = ((size_t)P.rows * ((P.cols + NM_TC - 1) / NM_TC) * P.ntap * 4 + 255) & ~size_t(255);
        size_t need = b_sorted + ((P.plane + 255) & ~255ll) + b_fwd;
        if (job->memory == FPL_MEM_HOST)
            need += ((b_stack + 255) & ~size_t(255)) + ((b_nmap + 255) & ~size_t(255)) +
                    (((size_t)P.plane * 4 + 255) & ~size_t(255)) + (((size_t)P.plane + 255) & ~size_t(255));
        if (ctx->cap_nm < need) {
            if (ctx->d_nm) cudaFree(ctx->d_nm);
            ctx->d_nm = nullptr;
            ctx->cap_nm = 0;
            if (cudaMalloc(&ctx->d_nm, need) != cudaSuccess) return FPL_ERR_NOMEM;
            ctx->cap_nm = need;
        }
        char *base = static_cast<char *>(ctx->d_nm);
        P.sorted = reinterpret_cast<float *>(base);
        base += b_sorted;
        P.valid = reinterpret_cast<uint8_t *>(base);
        base += (P.plane + 255) & ~255ll;
        P.fwd = reinterpret_cast<uint32_t *>(base);
        base += b_fwd;
        auto fail = [&](cudaError_t e, const char *what) {
            ctx->last_error = std::string(what) + ": " + cudaGetErrorString(e);
            return FPL_ERR_CUDA;
        };
        cudaError_t e;
        if (job->memory == FPL_MEM_HOST) {
            void *d_stack = base;
            base += (b_stack + 255) & ~size_t(255);
            P.nmap = reinterpret_cast<uint32_t *>(base);
            base += (b_nmap + 255) & ~size_t(255);
            P.count = job->count ? reinterpret_cast<int32_t *>(base) : nullptr;
            base += ((size_t)P.plane * 4 + 255) & ~size_t(255);
            uint8_t *d_mask = job->mask ? reinterpret_cast<uint8_t *>(base) : nullptr;
            if ((e = cudaMemcpyAsync(d_stack, job->stack, b_stack, cudaMemcpyHostToDevice, st)) != cudaSuccess)
                return fail(e, "copy stack");
            if (d_mask && (e = cudaMemcpyAsync(d_mask, job->mask, (size_t)P.plane, cudaMemcpyHostToDevice, st)) !=
                              cudaSuccess)
                return fail(e, "copy mask");
            P.stack = static_cast<const float2 *>(d_stack);
            P.mask = d_mask;
        } else {
            P.stack = static_cast<const float2 *>(job->stack);
            P.mask = job->mask;
            P.nmap = job->nmap;
            P.count = job->count;
        }
        const unsigned sblocks = (unsigned)((P.plane + NM_SORT_THREADS - 1) / NM_SORT_THREADS);
        if (P.nb <= 16) k_nmap_sort<16><<<sblocks, NM_SORT_THREADS, 0, st>>>(P);
        else if (P.nb <= 32) k_nmap_sort<32><<<sblocks, NM_SORT_THREADS, 0, st>>>(P);
        else k_nmap_sort<64><<<sblocks, NM_SORT_THREADS, 0, st>>>(P);
        if ((e = cudaGetLastError()) != cudaSuccess) return fail(e, "k_nmap_sort");
        if (ad2) e = nm_launch_ad(P, tile, st);
        else if (packed) e = nm_launch_ks<64, 1, false>(P, tile, st);
        else if (P.nb <= 16) e = nm_launch_ks<16, 2, true>(P, tile, st);
        else if (P.nb <= 32) e = nm_launch_ks<32, 2, true>(P, tile, st);
        else e = nm_launch_ks<64, 1, true>(P, tile, st);
        if (e != cudaSuccess) return fail(e, ad2 ? "k_nmap_ad" : "k_nmap_ks");
        const long long groups = (long long)P.rows * ((P.cols + NM_TC - 1) / NM_TC);
        k_nmap_map<<<(unsigned)((groups + MAP_WARPS - 1) / MAP_WARPS), 32 * MAP_WARPS,
                     sizeof(uint32_t) * MAP_WARPS * 32 * (nul | 1), st>>>(P);
        if ((e = cudaGetLastError()) != cudaSuccess) return fail(e, "k_nmap_map");
        if (job->memory == FPL_MEM_HOST) {
            if ((e = cudaMemcpyAsync(job->nmap, P.nmap, b_nmap, cudaMemcpyDeviceToHost, st)) != cudaSuccess)
                return fail(e, "copy nmap");
            if (job->count &&
                (e = cudaMemcpyAsync(job->count, P.count, (size_t)P.plane * 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess)
                return fail(e, "copy count");
        }
        if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return fail(e, "fpl_nmap");
        return FPL_OK;
    });
}
