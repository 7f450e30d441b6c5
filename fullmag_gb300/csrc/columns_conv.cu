// columns_conv.cu -- launchers of the thin-film pass and of the fused y+z pass of small 3-D
// grids, their batched forms, and their kernels for any length.
#include "columns_conv.cuh"

namespace fm {

#define FM_DECLARE(n) \
    template <> \
    const ConvKernels &conv_kernels_of<n>();
FM_LENGTHS_TO_256(FM_DECLARE) FM_LENGTHS_LONG(FM_DECLARE)
#undef FM_DECLARE

namespace {

// (two CTAs named as in long_butterflies; the y+z pass gains at every length, 60x45x6 24.7 -> 22.8 us
// per launch, 100x90x5 32.1 -> 30.9, unless its CTAs want more than two per SM: 300x2x20, 321 CTAs of
// 10 KB, 12.3 us at 64 registers and 16.3 at 96)
template <bool WIDE>
__global__ void __launch_bounds__(kThreads, general_ctas(WIDE)) yz_convolve_general_kernel(const ColPass p) {
    pdl_wait();
    if (p.early) pdl_trigger();
    yz_convolve_general_body(p, blockIdx.x);
}
template <bool WIDE>
__global__ void __launch_bounds__(kThreads, general_ctas(WIDE)) y_convolve_2d_general_kernel(const ColPass p) {
    pdl_wait();
    if (p.early) pdl_trigger();
    y_convolve_2d_general_body(p, blockIdx.x);
}
const ConvKernels &conv_kernels_for(int py) {
#define FM_CASE(n) \
    case n: return conv_kernels_of<n>();
    switch (py) { FM_LENGTHS_TO_256(FM_CASE) FM_LENGTHS_LONG(FM_CASE) }
#undef FM_CASE
    static const ConvKernels none{};
    return none;
}

}  // namespace

size_t yz_convolve_smem(const Grid &g, int tx) {
    const size_t a = (size_t)3 * tx * g.nz * skewed_len(g.py);
    if (yz_fused_ok(g)) return 2 * sizeof(float2) * a;
    const size_t b = (size_t)3 * tx * g.py * skewed_len(g.pz);
    return 2 * sizeof(float2) * (a > b ? a : b);
}

cudaError_t launch_yz_convolve(const ColPass &p, cudaStream_t s) {
    if (p.g.per) return cudaErrorInvalidValue;  // the fused y+z pass reads the octant kernel only
    const size_t sm = yz_convolve_smem(p.g, p.tx);
    const ConvKernels &k = conv_kernels_for(p.g.py);
    const bool wide = tiles(p) <= 2 * 152 || sm > kMaxSmem / 3;
    const ColKernel fn = yz_fused_ok(p.g) ? (p.g.pz <= 8 ? k.yz : k.yz_big)
                         : wide           ? yz_convolve_general_kernel<true>
                                          : yz_convolve_general_kernel<false>;
    cudaError_t e = ensure_smem((const void *)fn, sm);
    if (e != cudaSuccess) return e;
    return launch_pdl(fn, dim3(tiles(p)), dim3(kThreads), sm, s, p);
}

size_t y_convolve_2d_smem(const Grid &g, int tx) {
    const size_t one = sizeof(float2) * (size_t)3 * tx * skewed_len(g.py);
    return y2d_two_level(g) ? one : 2 * one;
}
size_t y_convolve_2d_batched_smem(const Grid &g, int tx) {
    const size_t one = sizeof(float2) * (size_t)3 * tx * skewed_len(g.py);
    return y2d_fused_ok(g) && !g.per ? one : 2 * one;
}

cudaError_t launch_y_convolve_2d(const ColPass &p, cudaStream_t s) {
    const size_t sm = y_convolve_2d_smem(p.g, p.tx);
    const ConvKernels &k = conv_kernels_for(p.g.py);
    const ColKernel general = long_butterflies(p.plan) ? y_convolve_2d_general_kernel<true> : y_convolve_2d_general_kernel<false>;
    const ColKernel fn = !y2d_two_level(p.g) ? general
                         : (p.g.per & 2)    ? k.film_full
                         : p.g.per          ? k.film_per
                                            : k.film;
    cudaError_t e = ensure_smem((const void *)fn, sm);
    if (e != cudaSuccess) return e;
    return launch_pdl(fn, dim3(tiles(p)), dim3(kThreads), sm, s, p);
}

}  // namespace fm
