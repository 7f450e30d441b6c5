// row_pass_batched.cu -- the row pass over many problems in one launch.
#include "row_pass.cuh"

namespace fm {

namespace {

// One launch for many problems: work[blockIdx.x] = (problem, block within problem).
template <int CLASS, bool LEAN>
__global__ void __launch_bounds__(kThreads, row_ctas(-CLASS)) row_pass_batched_kernel(const RowPass *__restrict__ ps,
                                                                    const int2 *__restrict__ work) {
    // stage the problem's descriptor in shared memory once per CTA: the body reads its
    // fields in every loop, and global reads could not be hoisted past the stores
    __shared__ __align__(16) unsigned char desc[sizeof(RowPass)];
    const int2 w = work[blockIdx.x];
    // a finished problem (step size 0 in its control block) keeps its blocks in the table
    // until the round is rebuilt; the whole CTA leaves before its first barrier
    const double *dtp = ps[w.x].dt_dev;
    if (dtp && *dtp <= 0.0) return;
    const int *src = reinterpret_cast<const int *>(ps + w.x);
    for (int i = threadIdx.x; i < (int)(sizeof(RowPass) / sizeof(int)); i += blockDim.x)
        reinterpret_cast<int *>(desc)[i] = src[i];
    __syncthreads();
    const RowPass &p = *reinterpret_cast<const RowPass *>(desc);
    row_pass_body<-CLASS, false, false, LEAN>(p, w.y, (p.g.ny * p.g.nz + p.rows - 1) / p.rows);
}

}  // namespace

int row_pass_class(const Grid &g, bool demag) {
    const int n = row_pass_length(g, demag);
    return n == 0 ? 0 : n <= 64 ? 1 : n <= 256 ? 2 : 3;
}

cudaError_t launch_row_pass_batched(const RowPass *ps, const int2 *work, int nwork, int cls, bool lean, size_t smem,
                                    cudaStream_t s) {
    using Kernel = void (*)(const RowPass *, const int2 *);
    static constexpr Kernel fns[4][2] = {{row_pass_batched_kernel<0, false>, row_pass_batched_kernel<0, true>},
                                         {row_pass_batched_kernel<1, false>, row_pass_batched_kernel<1, true>},
                                         {row_pass_batched_kernel<2, false>, row_pass_batched_kernel<2, true>},
                                         {row_pass_batched_kernel<3, false>, row_pass_batched_kernel<3, true>}};
    const Kernel fn = fns[cls][lean];
    cudaError_t e = ensure_smem((const void *)fn, smem);
    if (e != cudaSuccess || nwork == 0) return e;
    fn<<<nwork, kThreads, smem, s>>>(ps, work);
    return cudaGetLastError();
}

}  // namespace fm
