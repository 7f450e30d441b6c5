// row_pass.cu -- launchers of the row pass (row_pass.cuh), and its kernels for any x length.
#include "row_pass.cuh"

namespace fm {

#define FM_DECLARE(n) \
    template <> \
    const RowKernels &row_kernels_of<n>();
FM_LENGTHS_TO_256(FM_DECLARE) FM_LENGTHS_LONG(FM_DECLARE)
#undef FM_DECLARE

// by half length; 0: any length
static const RowKernels &row_kernels_for(int half) {
#define FM_CASE(n) \
    case n: return row_kernels_of<n>();
    switch (half) { FM_LENGTHS_TO_256(FM_CASE) FM_LENGTHS_LONG(FM_CASE) }
#undef FM_CASE
    static const RowKernels general = row_kernels<0>();
    return general;
}

// an intermediate stage: what LEAN leaves out is not asked for
static bool row_lean(const RowPass &p, bool transforms) {
    return p.m_in && p.m0 && !p.partials && !p.n_err && !p.h_ex_out && !p.h_d_out && !p.adj_mode &&
           (!transforms || (p.x_in && p.x_out));
}

int row_pass_length(const Grid &g, bool demag) {
    return demag && (row_x_open_ok(g) || row_x_periodic_ok(g)) ? g.half : 0;
}

// ---- host launchers ----

size_t row_pass_smem(const RowPass &p) {
    const bool use_fft = (p.x_in != nullptr) || (p.x_out != nullptr);
    size_t b = 0;
    // one buffer for the two-level transforms of half lines (in place), else two
    if (use_fft) b += (row_pass_length(p.g, true) && !(p.g.per & 1) ? 1 : 2) * sizeof(float2) * (size_t)p.rows * 3 * skewed_len(p.g.half);
    b += sizeof(double) * kWarps * kNumStats;
    return b;
}

int row_pass_blocks(const RowPass &p) {
    const int nrows = p.g.ny * p.g.nz;
    return (nrows + p.rows - 1) / p.rows;
}

cudaError_t launch_row_pass(const RowPass &p, cudaStream_t s) {
    const size_t sm = row_pass_smem(p);
    const int length = row_pass_length(p.g, p.x_in || p.x_out);
    const RowKernels &k = row_kernels_for(length);
    const bool lean = row_lean(p, length > 0);
    const RowKernel fn = length && (p.g.per & 1)                                ? k.periodic[lean]
                         : !length && (p.x_in || p.x_out) && long_butterflies(p.xplan) ? k.wide[lean]
                         : lean && k.dense && row_pass_blocks(p) >= kDenseCtas ? k.dense
                                                                               : k.open[lean];
    cudaError_t e = ensure_smem((const void *)fn, sm);
    if (e != cudaSuccess) return e;
    return launch_pdl(fn, dim3(row_pass_blocks(p)), dim3(kThreads), sm, s, p);
}

cudaError_t launch_row_pass_adj(const RowPass &p, cudaStream_t s) {
    const size_t sm = row_pass_smem(p);
    const RowKernel fn = row_kernels_for(row_pass_length(p.g, p.x_in || p.x_out)).adj;
    cudaError_t e = ensure_smem((const void *)fn, sm);
    if (e != cudaSuccess) return e;
    return launch_pdl(fn, dim3(row_pass_blocks(p)), dim3(kThreads), sm, s, p);
}

}  // namespace fm
