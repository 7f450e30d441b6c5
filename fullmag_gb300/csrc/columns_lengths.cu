// columns_lengths.cu -- thin-film and fused y+z kernels of a few y lengths; compiled once per
// group (FM_GROUP, build.py), so that the groups build in parallel.
#include "columns_conv.cuh"

namespace fm {

namespace {

// (from 320 on the inner pass of a film holds 3 x 10 to 3 x 32 complex values a thread)
template <int N, bool FULL, bool PER>
__global__ void __launch_bounds__(kThreads, N > 512 ? 1 : 2) y_convolve_2d_kernel(const ColPass p) {
    pdl_wait();
    if (p.early) pdl_trigger();
    y_convolve_2d_fused<N, FULL, PER>(p, blockIdx.x);
}
template <int N, bool BIG>
__global__ void __launch_bounds__(kThreads) yz_convolve_kernel(const ColPass p) {
    pdl_wait();
    if (p.early) pdl_trigger();
    yz_convolve_fused_body<N, BIG>(p, blockIdx.x);
}

template <int N>
ConvKernels conv_kernels() {
    return {y_convolve_2d_kernel<N, false, false>, y_convolve_2d_kernel<N, false, true>, y_convolve_2d_kernel<N, true, true>,
            yz_convolve_kernel<N, false>, yz_convolve_kernel<N, true>};
}

}  // namespace

#if FM_GROUP == 0
#define FM_GROUP_LENGTHS(F) F(16) F(20) F(24)
#elif FM_GROUP == 1
#define FM_GROUP_LENGTHS(F) F(28) F(32) F(40)
#elif FM_GROUP == 2
#define FM_GROUP_LENGTHS(F) F(48) F(56) F(64)
#elif FM_GROUP == 3
#define FM_GROUP_LENGTHS(F) F(80) F(96) F(112)
#elif FM_GROUP == 4
#define FM_GROUP_LENGTHS(F) F(128) F(160) F(192)
#elif FM_GROUP == 5
#define FM_GROUP_LENGTHS(F) F(224) F(256) F(320)
#elif FM_GROUP == 6
#define FM_GROUP_LENGTHS(F) F(384) F(448) F(512)
#elif FM_GROUP == 7
#define FM_GROUP_LENGTHS(F) F(640) F(768)
#else
#define FM_GROUP_LENGTHS(F) F(896) F(1024)
#endif

#define FM_ENTRY(n) \
    template <> \
    const ConvKernels &conv_kernels_of<n>() { \
        static const ConvKernels k = conv_kernels<n>(); \
        return k; \
    }
FM_GROUP_LENGTHS(FM_ENTRY)

}  // namespace fm
