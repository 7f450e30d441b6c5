// columns_batched.cu -- the thin-film and fused y+z passes over many problems in one launch.
#include "columns_conv.cuh"

namespace fm {

namespace {

// work[blockIdx.x] = (problem, kx tile); KIND: see col_batched_kind -- one kernel per kind, so
// each gets its own register allocation
template <int KIND>
__global__ void __launch_bounds__(kThreads, KIND >= 9 ? 4 : KIND >= 6 || KIND == 2 ? 1 : 2) col_batched_kernel(
    const ColPass *__restrict__ ps, const int2 *__restrict__ work) {
    __shared__ __align__(16) unsigned char desc[sizeof(ColPass)];  // descriptor staged once per CTA
    const int2 w = work[blockIdx.x];
    // a finished problem (step size 0) keeps its tiles in the table until the round is
    // rebuilt; the whole CTA leaves before its first barrier
    const double *skip = ps[w.x].skip_dt;
    if (skip && *skip <= 0.0) return;
    const int *src = reinterpret_cast<const int *>(ps + w.x);
    for (int i = threadIdx.x; i < (int)(sizeof(ColPass) / sizeof(int)); i += blockDim.x)
        reinterpret_cast<int *>(desc)[i] = src[i];
    __syncthreads();
    const ColPass &p = *reinterpret_cast<const ColPass *>(desc);
    constexpr int N = -1 - KIND % 3;
    if constexpr (KIND == 9) {
        y_convolve_2d_general_body(p, w.y);
    } else if constexpr (KIND == 10) {
        yz_convolve_general_body(p, w.y);
    } else if constexpr (KIND < 3) {
#define FM_CASE(n) \
    case n: y_convolve_2d_fused<n, false, false>(p, w.y); return;
        FM_SELECT_LENGTH(N, FM_CASE)
#undef FM_CASE
    } else {
        yz_convolve_fused_body<N, (KIND >= 6)>(p, w.y);
    }
}

}  // namespace

int col_batched_kind(const Grid &g) {
    const int c = g.py <= 64 ? 0 : g.py <= 256 ? 1 : 2;
    if (g.thin) return y2d_fused_ok(g) && !g.per ? c : 9;
    return yz_fused_ok(g) ? (g.pz <= 8 ? 3 : 6) + c : 10;
}

cudaError_t launch_col_batched(const ColPass *ps, const int2 *work, int nwork, int kind, size_t smem, cudaStream_t s) {
    using Kernel = void (*)(const ColPass *, const int2 *);
    static constexpr Kernel fns[kColBatchedKinds] = {
        col_batched_kernel<0>, col_batched_kernel<1>, col_batched_kernel<2>, col_batched_kernel<3>,
        col_batched_kernel<4>, col_batched_kernel<5>, col_batched_kernel<6>, col_batched_kernel<7>,
        col_batched_kernel<8>, col_batched_kernel<9>, col_batched_kernel<10>};
    if (kind < 0 || kind >= kColBatchedKinds) return cudaErrorInvalidValue;
    cudaError_t e = ensure_smem((const void *)fns[kind], smem);
    if (e != cudaSuccess || nwork == 0) return e;
    fns[kind]<<<nwork, kThreads, smem, s>>>(ps, work);
    return cudaGetLastError();
}

}  // namespace fm
