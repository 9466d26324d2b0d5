// kernels.h -- host-side declarations of the kernel launchers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fpl {

struct KParams;
struct BoxSeg;
struct BatchEntry;

// padded order used for a stack depth (16, 32, 64; 0 = unsupported)
int pick_np(int nb);

// plain FP32 form, one warp per pixel end to end (windows the Gamma kernel
// does not take, and runs that may not allocate), over P.npix pixels starting at
// P.pix_begin
cudaError_t launch_fp32(const KParams &P, int num_sms, cudaStream_t st);

// FP64 form over the work list in P (or over every pixel if P.fb_list is null)
cudaError_t launch_fp64(const KParams &P, int num_sms, cudaStream_t st);

// is the tensor-core Gamma kernel available for this stack
// depth and window (nbands <= 64, window width <= 63, window union of an
// 8 x 16 pixel tile <= 2048 samples)
bool gram_box_supported(int nb, int ny, int nx);

// floats per Gamma record written by launch_gram_box
int gram_box_record(int nb);

// tensor-core Gamma records (P.parts bf16 parts per product) for the whole rows
// [P.pix_begin, P.pix_begin + P.npix) into P.cbuf / P.cinfo
cudaError_t launch_gram_box(const KParams &P, int num_sms, cudaStream_t st);

// eigen-solves and outputs from P.cbuf / P.cinfo
cudaError_t launch_solve(const KParams &P, int num_sms, cudaStream_t st);
// sets the attributes of its kernels (before a capture)
cudaError_t prepare_solve();
// Pieces of a batch or serving wave from this size on get solve launches of
// their own: the kernel for their depth (the combined one has one shape for 17 to 32
// and one for 33 to 64 dates) with its parameters in constant memory.  20 pieces of
// 10 to 45 dates, combined -> own launches: 512^2 106 -> 81 ms, 256^2 30.0 -> 23.9 ms,
// 180^2 17.1 -> 14.7 ms; of 30 dates all: 512^2 79.0 -> 71.1, 256^2 23.3 -> 22.0, but
// 180^2 14.08 -> 14.14 and 128^2 9.5 -> 10.2 ms; of 10 dates: 256^2 6.23 -> 6.06,
// 128^2 1.81 -> 2.09 ms.  From 2^16 pixels on every batch gains.
constexpr long long kOwnSolvePx = 1ll << 16;

// batched: a launch of the Gamma kernel covers gram_box_tiles(P)
// tiles and needs gram_box_smem bytes of shared memory.
long long gram_box_tiles(const KParams &P);
size_t gram_box_smem(const KParams &P);
// tiles of every segment in one persistent launch (smem: the largest
// gram_box_smem of the segments)
cudaError_t launch_gram_batch(const BoxSeg *segs, int nseg, long long total, size_t smem,
                              int num_sms, cudaStream_t st);
// kernel attributes of the batched solve for padded depth np (call
// before capturing a launch sequence)
cudaError_t prepare_mixed_batch(int np);
cudaError_t prepare_gram_batch();
// eigen-solves of every entry (one padded depth np); kinds: the union of the
// entries' solve_kind; warps: warps per CTA (0 = the most that fit; see solve_max_warps)
int solve_kind(const KParams &P);
cudaError_t launch_solve_batch(int np, const BatchEntry *ents, int nent, long long total, int kinds, int num_sms,
                               cudaStream_t st, int warps = 0);
int solve_max_warps(int np);

}  // namespace fpl
