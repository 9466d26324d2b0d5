// kernels_f32.cu -- FP32 instantiations of the pixel kernels.
#include <algorithm>

#include "kernels_impl.cuh"

namespace fpl {

int pick_np(int nb)
{
    if (nb <= 16) return 16;
    if (nb <= 32) return 32;
    if (nb <= 64) return 64;
    return 0;
}

cudaError_t launch_fp32(const KParams &P, int num_sms, cudaStream_t st)
{
    switch (pick_np(P.nb)) {
    case 16: return launch_t<float, 16>(P, num_sms, st);
    case 32: return launch_t<float, 32>(P, num_sms, st);
    case 64: return launch_t<float, 64>(P, num_sms, st);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_solve(const KParams &P, int num_sms, cudaStream_t st)
{
    // the smallest grid that holds the dates: its blocks per lane (3, 6, 10; 12,
    // 20) set the work of a step and the registers, so the warps per SM
    if (P.nb <= 16) return launch_solve_t<16, 2>(P, num_sms, st);
    if (P.nb <= 24) return launch_solve_t<16, 3>(P, num_sms, st);
    if (P.nb <= 32) return launch_solve_t<16, 4>(P, num_sms, st);
    if (P.nb <= 48) return launch_solve_t<32, 3>(P, num_sms, st);
    if (P.nb <= 64) return launch_solve_t<32, 4>(P, num_sms, st);
    return cudaErrorInvalidValue;
}

cudaError_t prepare_mixed_batch(int np)
{
    cudaError_t e = prepare_gram_batch();
    if (e != cudaSuccess) return e;
    switch (np) {
    case 16: return configure_solve_batch<16, 2>();
    case 32: return configure_solve_batch<16, 4>();
    case 64: return configure_solve_batch<32, 4>();
    }
    return cudaErrorInvalidValue;
}

int solve_max_warps(int np)
{
    switch (np) {
    case 16: return solve_warps<16, 2>();
    case 32: return solve_warps<16, 4>();
    case 64: return solve_warps<32, 4>();
    }
    return 1;
}

cudaError_t prepare_solve()
{
    const cudaError_t e[5] = {prepare_solve_t<16, 2>(), prepare_solve_t<16, 3>(), prepare_solve_t<16, 4>(),
                              prepare_solve_t<32, 3>(), prepare_solve_t<32, 4>()};
    for (cudaError_t r : e)
        if (r != cudaSuccess) return r;
    return cudaSuccess;
}

int solve_kind(const KParams &P) { return 1 << tile_kind(P); }

cudaError_t launch_solve_batch(int np, const BatchEntry *ents, int nent, long long total, int kinds, int num_sms,
                               cudaStream_t st, int warps)
{
    if (nent <= 0 || total <= 0) return cudaSuccess;
    switch (np) {
    case 16: return launch_solve_batch_t<16, 2>(ents, nent, total, kinds, num_sms, st, warps);
    case 32: return launch_solve_batch_t<16, 4>(ents, nent, total, kinds, num_sms, st, warps);
    case 64: return launch_solve_batch_t<32, 4>(ents, nent, total, kinds, num_sms, st, warps);
    }
    return cudaErrorInvalidValue;
}

}  // namespace fpl
