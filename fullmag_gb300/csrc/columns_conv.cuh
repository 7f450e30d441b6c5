// columns_conv.cuh -- bodies of the column passes that convolve a kx tile X -> X in one go:
// thin films (y transform, multiply, inverse) and small 3-D grids (y and z).
#pragma once
#include "columns.cuh"

namespace fm {

// The kernels of one py, each length compiled in columns_lengths.cu: thin film with the open
// kernel, with the periodic kernel on an open y, on a periodic y; fused y+z with pz <= 8 and
// up to 24 (z columns of up to 144 registers a thread).
using ColKernel = void (*)(const ColPass);
struct ConvKernels {
    ColKernel film, film_per, film_full, yz, yz_big;
};
template <int N>
const ConvKernels &conv_kernels_of();

namespace {

// z convolution of the tile's (col, ky) columns in registers: component c, plane z of the
// column sits at line[(c*nz + z)*lstride].
template <int PZ>
__device__ __forceinline__ void z_small_phase(const ColPass &p, int kx0, int ncol, float2 *B, int ls) {
    constexpr int H = PZ / 2;
    const Grid &g = p.g;
    const int nz = g.nz;
    const size_t lstride = (size_t)p.tx * ls, kc = (size_t)g.nkz * g.nky * g.nkx;
    for (int it = threadIdx.x; it < g.py * ncol; it += blockDim.x) {
        int ky, col;
        tile_item(p, ncol, it, ky, col);
        float2 *line = B + (size_t)col * ls + sk(ky);
        float2 v[3][H];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int z = 0; z < H; ++z) v[c][z] = z < nz ? line[(c * nz + z) * lstride] : make_float2(0.f, 0.f);
        int kym;
        float sy;
        kernel_mirror(ky, g.py, kym, sy);
        const int kx = min(kx0 + col, g.nkx - 1);
        z_column_convolve<PZ, false>(v, p.kern + (size_t)kx * g.nky + kym, (size_t)g.nkx * g.nky, kc, sy,
                                     p.plan2.tw);  // ky-fastest kernel layout
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int z = 0; z < H; ++z)
                if (z < nz) line[(c * nz + z) * lstride] = v[c][z];
    }
}

__host__ __device__ __forceinline__ bool yz_fused_ok(const Grid &g) {
    return g.per == 0 && two_level_length(g.py) && 2 * g.ny <= g.py && z_register_length(g.pz) && 2 * g.nz <= g.pz;
}

// Small 3-D grids, py = N1 * N2: the pruned two-level y transforms of the nz physical
// planes around the register z convolution.  Lines (c, z, col) at L = (c*nz + z)*tx + col in
// two buffers: A holds the outer-pass slots, B the natural-order y spectrum.  Phases: outer
// half-input DFT from global memory -> A; inner DFTs A -> B; per (col, ky) z convolution in
// B; inner inverse B -> A; outer half-output inverse A -> global memory.
template <int N>
__device__ __forceinline__ void yz_forward(const ColPass &p, int kx0, int ncol, float2 *A, float2 *B) {
    constexpr int N1 = split_line(N), N2 = N / N1, H1 = N1 / 2;
    constexpr int ls = skewed_len(N);
    const Grid &g = p.g;
    const int tx = p.tx, nlive = 3 * g.nz * ncol;
    const size_t zstride = (size_t)g.ny * g.xs;
    const float2 *__restrict__ tw = p.plan.tw;
    for (int it = threadIdx.x; it < nlive * N2; it += blockDim.x) {
        int rest, col;
        tile_item(p, ncol, it, rest, col);
        const int n2 = rest % N2, cz = rest / N2;  // cz = c*nz + z
        const float2 *src = p.in + cz * zstride + kx0 + col;
        float2 e[H1];
#pragma unroll
        for (int y1 = 0; y1 < H1; ++y1) {
            const int y = N2 * y1 + n2;
            e[y1] = y < g.ny ? src[(size_t)y * g.xs] : make_float2(0.f, 0.f);
        }
        half_dft_store<N1, N2>(e, n2, A + (cz * tx + col) * ls, tw);
    }
    __syncthreads();
    for (int it = threadIdx.x; it < nlive * N1; it += blockDim.x) {
        int rest, col;
        tile_item(p, ncol, it, rest, col);
        const int k1 = rest % N1, cz = rest / N1;
        const float2 *sl = A + (cz * tx + col) * ls;
        float2 v[N2];
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) v[n2] = sl[sk(k1 * N2 + n2)];
        dft_small<N2>(v, false);
        float2 *bl = B + (cz * tx + col) * ls;
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) bl[sk(k1 + N1 * k2)] = v[k2];
    }
    __syncthreads();
}
template <int N>
__device__ __forceinline__ void yz_inverse(const ColPass &p, int kx0, int ncol, float2 *A, const float2 *B) {
    constexpr int N1 = split_line(N), N2 = N / N1, H1 = N1 / 2;
    constexpr int ls = skewed_len(N);
    const Grid &g = p.g;
    const int tx = p.tx, nlive = 3 * g.nz * ncol;
    const size_t zstride = (size_t)g.ny * g.xs;
    const float2 *__restrict__ tw = p.plan.tw;
    __syncthreads();
    for (int it = threadIdx.x; it < nlive * N1; it += blockDim.x) {
        int rest, col;
        tile_item(p, ncol, it, rest, col);
        const int k1 = rest % N1, cz = rest / N1;
        const float2 *bl = B + (cz * tx + col) * ls;
        float2 v[N2];
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) v[k2] = bl[sk(k1 + N1 * k2)];
        dft_small<N2>(v, true);
        float2 *sl = A + (cz * tx + col) * ls;
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) sl[sk(k1 * N2 + n2)] = (n2 && k1) ? cmul(v[n2], cconj(__ldg(tw + n2 * k1))) : v[n2];
    }
    __syncthreads();
    for (int it = threadIdx.x; it < nlive * N2; it += blockDim.x) {
        int rest, col;
        tile_item(p, ncol, it, rest, col);
        const int n2 = rest % N2, cz = rest / N2;
        float2 e[H1];
        half_idft_load<N1, N2>(e, n2, A + (cz * tx + col) * ls, tw);
        float2 *dst = p.out + cz * zstride + kx0 + col;
#pragma unroll
        for (int y1 = 0; y1 < H1; ++y1) {
            const int y = N2 * y1 + n2;
            if (y < g.ny) dst[(size_t)y * g.xs] = e[y1];
        }
    }
}

// One y length (N > 0), or a class of lengths by the grid's own (N = -1, -2, -3: the batched
// kernels, whose problems differ): F(n) for the grid's length.
#define FM_LENGTHS_CLASS1(F) F(16) F(20) F(24) F(28) F(32) F(40) F(48) F(56) F(64)
#define FM_LENGTHS_CLASS2(F) F(80) F(96) F(112) F(128) F(160) F(192) F(224) F(256)
#define FM_SELECT_LENGTH(N, F)                    \
    if constexpr (N == -1)                        \
        switch (p.g.py) { FM_LENGTHS_CLASS1(F) }  \
    else if constexpr (N == -2)                   \
        switch (p.g.py) { FM_LENGTHS_CLASS2(F) }  \
    else if constexpr (N == -3)                   \
        switch (p.g.py) { FM_LENGTHS_LONG(F) }

template <int N, bool BIG>
__device__ __forceinline__ void yz_convolve_fused_body(const ColPass &p, const int tile) {
    extern __shared__ __align__(16) unsigned char smem[];
    const Grid &g = p.g;
    const int kx0 = tile * p.tx, ncol = min(p.tx, g.nkx - kx0);
    const int ls = skewed_len(N > 0 ? N : g.py);
    float2 *A = reinterpret_cast<float2 *>(smem);
    float2 *B = A + (size_t)3 * g.nz * p.tx * ls;
#define FM_CASE(n) \
    case n: yz_forward<n>(p, kx0, ncol, A, B); break;
    if constexpr (N > 0) yz_forward<N>(p, kx0, ncol, A, B);
    else { FM_SELECT_LENGTH(N, FM_CASE) }
#undef FM_CASE
#define FM_CASE(n) \
    case n: z_small_phase<n>(p, kx0, ncol, B, ls); break;
    if constexpr (BIG)
        switch (g.pz) { FM_CASE(10) FM_CASE(12) FM_CASE(14) FM_CASE(16) FM_CASE(20) FM_CASE(24) }
    else
        switch (g.pz) { FM_CASE(2) FM_CASE(4) FM_CASE(6) FM_CASE(8) }
#undef FM_CASE
#define FM_CASE(n) \
    case n: yz_inverse<n>(p, kx0, ncol, A, B); break;
    if constexpr (N > 0) yz_inverse<N>(p, kx0, ncol, A, B);
    else { FM_SELECT_LENGTH(N, FM_CASE) }
#undef FM_CASE
}

// 3-D grids whose (y, z) plane fits in shared memory: forward y-transform of the nz
// physical planes, in-smem transpose, forward z, multiply, inverse z, transpose back,
// inverse y -- X -> X in place, one pass instead of three and no Y round trip.
// Lines: y-lines (c, col, z) at ((c*tx + col)*nz + z), z-lines (c, col, ky) at
// ((c*tx + col)*py + ky); both layouts share two ping-pong buffers of `half_buf`.
__device__ __forceinline__ void yz_convolve_general_body(const ColPass &p, const int tile) {
    extern __shared__ __align__(16) unsigned char smem[];
    const Grid &g = p.g;
    const FftPlan &plan_z = p.plan2;
    const int tx = p.tx, kx0 = tile * tx, ncol = min(tx, g.nkx - kx0);
    const int lsy = skewed_len(g.py), lsz = skewed_len(g.pz);
    const int nly = 3 * tx * g.nz, nlz = 3 * tx * g.py;
    const int half_buf = max(nly * lsy, nlz * lsz);
    float2 *P = reinterpret_cast<float2 *>(smem);
    float2 *Q = P + half_buf;
    const size_t cstride = (size_t)g.nz * g.ny * g.xs;
    batched_copy<8>(
        3 * g.nz * g.ny * tx,
        [&](int idx) {
            const int r = p.fd_tx.div(idx), col = idx - r * tx;
            const int r2 = g.fd_ny.div(r), y = r - r2 * g.ny;
            const int c = g.fd_nz.div(r2), z = r2 - c * g.nz;
            return col < ncol ? p.in[c * cstride + ((size_t)z * g.ny + y) * g.xs + kx0 + col] : make_float2(0.f, 0.f);
        },
        [&](int idx, float2 v) {
            const int r = p.fd_tx.div(idx), col = idx - r * tx;
            const int r2 = g.fd_ny.div(r), y = r - r2 * g.ny;
            const int c = g.fd_nz.div(r2), z = r2 - c * g.nz;
            P[((c * tx + col) * g.nz + z) * lsy + sk(y)] = v;
        });
    for (int line = threadIdx.x >> 5; line < nly; line += blockDim.x >> 5)
        for (int y = g.ny + (threadIdx.x & 31); y < g.py; y += 32) P[line * lsy + sk(y)] = make_float2(0.f, 0.f);
    __syncthreads();
    float2 *R = fft_lines(P, Q, nly, lsy, p.plan, false);
    float2 *O = (R == P) ? Q : P;
    // transpose to z-lines, zero planes z >= nz
    for (int idx = threadIdx.x; idx < nlz * g.pz; idx += blockDim.x) {
        const int lz = g.fd_pz.div(idx), z = idx - lz * g.pz;
        const int cc = g.fd_py.div(lz), ky = lz - cc * g.py;
        O[lz * lsz + sk(z)] = z < g.nz ? R[(cc * g.nz + z) * lsy + sk(ky)] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    float2 *R2 = fft_lines(O, R, nlz, lsz, plan_z, false);
    const size_t kc = (size_t)g.nkz * g.nky * g.nkx;
    for (int idx = threadIdx.x; idx < tx * g.py * g.pz; idx += blockDim.x) {
        const int r = g.fd_pz.div(idx), kz = idx - r * g.pz;
        const int col = g.fd_py.div(r), ky = r - col * g.py;
        const int kx = min(kx0 + col, g.nkx - 1);
        int kym, kzm;
        float sy, sz;
        kernel_mirror(ky, g.py, kym, sy);
        kernel_mirror(kz, g.pz, kzm, sz);
        const float *K = p.kern + ((size_t)kzm * g.nkx + kx) * g.nky + kym;  // ky-fastest layout
        const float kxx = __ldg(K), kyy = __ldg(K + kc), kzz = __ldg(K + 2 * kc);
        const float kxy = sy * __ldg(K + 3 * kc), kxz = sz * __ldg(K + 4 * kc), kyz = sy * sz * __ldg(K + 5 * kc);
        float2 *lx = R2 + ((0 * tx + col) * g.py + ky) * lsz + sk(kz);
        float2 *ly = R2 + ((1 * tx + col) * g.py + ky) * lsz + sk(kz);
        float2 *lz = R2 + ((2 * tx + col) * g.py + ky) * lsz + sk(kz);
        const float2 mx = *lx, my = *ly, mz = *lz;
        *lx = make_float2(-(kxx * mx.x + kxy * my.x + kxz * mz.x), -(kxx * mx.y + kxy * my.y + kxz * mz.y));
        *ly = make_float2(-(kxy * mx.x + kyy * my.x + kyz * mz.x), -(kxy * mx.y + kyy * my.y + kyz * mz.y));
        *lz = make_float2(-(kxz * mx.x + kyz * my.x + kzz * mz.x), -(kxz * mx.y + kyz * my.y + kzz * mz.y));
    }
    __syncthreads();
    float2 *R3 = fft_lines(R2, (R2 == P) ? Q : P, nlz, lsz, plan_z, true);
    float2 *O3 = (R3 == P) ? Q : P;
    // transpose back to y-lines, keeping the physical planes z < nz
    for (int idx = threadIdx.x; idx < nly * g.py; idx += blockDim.x) {
        const int ly = g.fd_py.div(idx), ky = idx - ly * g.py;
        const int cc = g.fd_nz.div(ly), z = ly - cc * g.nz;
        O3[ly * lsy + sk(ky)] = R3[(cc * g.py + ky) * lsz + sk(z)];
    }
    __syncthreads();
    float2 *R4 = fft_lines(O3, R3, nly, lsy, p.plan, true);
    for (int idx = threadIdx.x; idx < 3 * g.nz * g.ny * tx; idx += blockDim.x) {
        const int r = p.fd_tx.div(idx), col = idx - r * tx;
        const int r2 = g.fd_ny.div(r), y = r - r2 * g.ny;
        const int c = g.fd_nz.div(r2), z = r2 - c * g.nz;
        if (col < ncol)
            p.out[c * cstride + ((size_t)z * g.ny + y) * g.xs + kx0 + col] = R4[((c * tx + col) * g.nz + z) * lsy + sk(y)];
    }
}

// Thin film, py = N1 * N2: outer pass from global memory (half lines on an open y; FULL:
// periodic, ny = py), inner passes with the multiply in registers, outer inverse to global
// memory; X -> X in place.  PER: the complex kernel of a film periodic along x or y.
template <int N, bool FULL, bool PER>
__device__ __forceinline__ void y_convolve_2d_fused(const ColPass &p, const int tile) {
    constexpr int N1 = split_conv(N), N2 = N / N1, H1 = N1 / 2;
    constexpr int ls = skewed_len(N);
    extern __shared__ __align__(16) unsigned char smem[];
    float2 *buf = reinterpret_cast<float2 *>(smem);  // line (c, col) at (c*tx + col)*ls
    const Grid &g = p.g;
    const int tx = p.tx, kx0 = tile * tx, ncol = min(tx, g.nkx - kx0);
    const size_t cstride = (size_t)g.ny * g.xs;
    const float2 *__restrict__ tw = p.plan.tw;
    const int n13 = 3 * N2 * ncol;
    for (int it = threadIdx.x; it < n13; it += blockDim.x) {
        int rz, col;
        tile_item(p, ncol, it, rz, col);
        const int n2 = rz % N2, c = rz / N2;
        const float2 *src = p.in + c * cstride + kx0 + col;
        float2 e[H1];
#pragma unroll
        for (int n1 = 0; n1 < H1; ++n1) {
            const int y = N2 * n1 + n2;
            e[n1] = FULL || y < g.ny ? src[(size_t)y * g.xs] : make_float2(0.f, 0.f);
        }
        if constexpr (FULL) {
            float2 f[H1];
#pragma unroll
            for (int n1 = 0; n1 < H1; ++n1) f[n1] = src[(size_t)(N2 * (n1 + H1) + n2) * g.xs];
            full_dft_store<N1, N2>(e, f, n2, buf + (c * tx + col) * ls, tw);
        } else {
            half_dft_store<N1, N2>(e, n2, buf + (c * tx + col) * ls, tw);
        }
    }
    __syncthreads();
    const size_t kc = (size_t)(PER ? g.py : g.nky) * g.ks;
    for (int it = threadIdx.x; it < N1 * ncol; it += blockDim.x) {
        int k1, col;
        tile_item(p, ncol, it, k1, col);
        float2 m[3][N2];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 *line = buf + (c * tx + col) * ls;
#pragma unroll
            for (int n2 = 0; n2 < N2; ++n2) m[c][n2] = line[sk(k1 * N2 + n2)];
            dft_small<N2>(m[c], false);
        }
        const int kx = min(kx0 + col, g.nkx - 1);
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) {
            if constexpr (PER) {  // complex kernel K[c][ky][kx]
                multiply_periodic(reinterpret_cast<const float2 *>(p.kern) + (size_t)(k1 + N1 * k2) * g.ks + kx, kc, true,
                                  &m[0][k2], &m[1][k2], &m[2][k2]);
            } else {
                int kym;
                float sy;
                kernel_mirror(k1 + N1 * k2, N, kym, sy);
                const float *K = p.kern + (size_t)kym * g.ks + kx;
                const float kxx = __ldg(K), kyy = __ldg(K + kc), kzz = __ldg(K + 2 * kc), kxy = sy * __ldg(K + 3 * kc);
                const float2 mx = m[0][k2], my = m[1][k2], mz = m[2][k2];
                m[0][k2] = make_float2(-(kxx * mx.x + kxy * my.x), -(kxx * mx.y + kxy * my.y));
                m[1][k2] = make_float2(-(kxy * mx.x + kyy * my.x), -(kxy * mx.y + kyy * my.y));
                m[2][k2] = make_float2(-(kzz * mz.x), -(kzz * mz.y));
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            dft_small<N2>(m[c], true);
            float2 *line = buf + (c * tx + col) * ls;
#pragma unroll
            for (int n2 = 0; n2 < N2; ++n2)
                line[sk(k1 * N2 + n2)] = (n2 && k1) ? cmul(m[c][n2], cconj(__ldg(tw + n2 * k1))) : m[c][n2];
        }
    }
    __syncthreads();
    for (int it = threadIdx.x; it < n13; it += blockDim.x) {
        int rz, col;
        tile_item(p, ncol, it, rz, col);
        const int n2 = rz % N2, c = rz / N2;
        float2 e[H1], f[H1];
        idft_load<N1, N2, FULL>(e, f, n2, buf + (c * tx + col) * ls, tw);
        float2 *dst = p.out + c * cstride + kx0 + col;
#pragma unroll
        for (int n1 = 0; n1 < H1; ++n1) {
            const int y = N2 * n1 + n2;
            if (FULL || y < g.ny) dst[(size_t)y * g.xs] = e[n1];
            if (FULL) dst[(size_t)(y + N2 * H1) * g.xs] = f[n1];
        }
    }
}

__host__ __device__ __forceinline__ bool y2d_fused_ok(const Grid &g) {
    return two_level_length(g.py) && ((g.per & 2) ? g.ny == g.py : 2 * g.ny <= g.py);
}

// ... and is the better one for a film alone: not for long lines (film_y_long, engine.h) of few kx
// columns.  The two-level form of these lengths holds 3 x 28 to 3 x 32 complex values a thread and is
// one long chain, which a few CTAs only wait for; from about 40 columns its fewer instructions count.
// RK4 steps in one call, us, two-level / general at 1024: ny = 500, nx = 4: 99 / 65, nx = 32: 85 / 73,
// nx = 48: 84 / 91, nx = 64: 86 / 91; ny = 400: nx = 32: 80 / 68, nx = 48: 81 / 68, nx = 64: 80 / 83.
__host__ __device__ __forceinline__ bool y2d_two_level(const Grid &g) {
    return y2d_fused_ok(g) && !(film_y_long(g.py, (g.per & 2) != 0) && g.nkx <= kFilmColumns);
}

// Thin film, any py: Stockham transforms in shared memory.
__device__ __forceinline__ void y_convolve_2d_general_body(const ColPass &p, const int tile) {
    extern __shared__ __align__(16) unsigned char smem[];
    const Grid &g = p.g;
    const int tx = p.tx, kx0 = tile * tx, ncol = min(tx, g.nkx - kx0);
    const int ls = skewed_len(g.py);
    const int nl = 3 * tx;
    float2 *a = reinterpret_cast<float2 *>(smem);
    float2 *b = a + nl * ls;
    const size_t cstride = (size_t)g.ny * g.xs;
    batched_copy<8>(
        3 * g.ny * tx,
        [&](int idx) {
            const int r1 = p.fd_tx.div(idx), col = idx - r1 * tx;
            const int c = g.fd_ny.div(r1), y = r1 - c * g.ny;
            return col < ncol ? p.in[c * cstride + (size_t)y * g.xs + kx0 + col] : make_float2(0.f, 0.f);
        },
        [&](int idx, float2 v) {
            const int r1 = p.fd_tx.div(idx), col = idx - r1 * tx;
            const int c = g.fd_ny.div(r1), y = r1 - c * g.ny;
            a[(c * tx + col) * ls + sk(y)] = v;
        });
    for (int line = threadIdx.x >> 5; line < nl; line += blockDim.x >> 5)  // zero padding rows
        for (int y = g.ny + (threadIdx.x & 31); y < g.py; y += 32) a[line * ls + sk(y)] = make_float2(0.f, 0.f);
    __syncthreads();
    float2 *r = fft_lines(a, b, nl, ls, p.plan, false);
    float2 *o = (r == a) ? b : a;
    if (g.per) {  // complex kernel K[c][ky][kx]
        const size_t kcp = (size_t)g.py * g.ks;
        for (int idx = threadIdx.x; idx < g.py * tx; idx += blockDim.x) {
            const int ky = p.fd_tx.div(idx), col = idx - ky * tx;
            const int kx = min(kx0 + col, g.nkx - 1);
            const float2 *K = reinterpret_cast<const float2 *>(p.kern) + (size_t)ky * g.ks + kx;
            multiply_periodic(K, kcp, true, r + (0 * tx + col) * ls + sk(ky), r + (1 * tx + col) * ls + sk(ky),
                              r + (2 * tx + col) * ls + sk(ky));
        }
    }
    const size_t kc = (size_t)g.nky * g.ks;
    for (int idx = threadIdx.x; idx < (g.per ? 0 : g.py * tx); idx += blockDim.x) {
        const int ky = p.fd_tx.div(idx), col = idx - ky * tx;
        const int kx = min(kx0 + col, g.nkx - 1);
        int kym;
        float sy;
        kernel_mirror(ky, g.py, kym, sy);
        const float *K = p.kern + (size_t)kym * g.ks + kx;
        const float kxx = __ldg(K), kyy = __ldg(K + kc), kzz = __ldg(K + 2 * kc), kxy = sy * __ldg(K + 3 * kc);
        float2 *lx = r + (0 * tx + col) * ls + sk(ky);
        float2 *ly = r + (1 * tx + col) * ls + sk(ky);
        float2 *lz = r + (2 * tx + col) * ls + sk(ky);
        const float2 mx = *lx, my = *ly, mz = *lz;
        *lx = make_float2(-(kxx * mx.x + kxy * my.x), -(kxx * mx.y + kxy * my.y));
        *ly = make_float2(-(kxy * mx.x + kyy * my.x), -(kxy * mx.y + kyy * my.y));
        *lz = make_float2(-(kzz * mz.x), -(kzz * mz.y));
    }
    __syncthreads();
    float2 *q = fft_lines(r, o, nl, ls, p.plan, true);
    for (int idx = threadIdx.x; idx < 3 * g.ny * tx; idx += blockDim.x) {
        const int r1 = p.fd_tx.div(idx), col = idx - r1 * tx;
        const int c = g.fd_ny.div(r1), y = r1 - c * g.ny;
        if (col < ncol) p.out[c * cstride + (size_t)y * g.xs + kx0 + col] = q[(c * tx + col) * ls + sk(y)];
    }
}

}  // namespace

}  // namespace fm
