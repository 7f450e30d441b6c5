// columns_z.cu -- z transforms of the demag convolution with the tensor multiply between the
// forward and the inverse transform.  In the shared-memory passes the y-frequencies ky and
// py - ky share one CTA, so every octant kernel value is read from HBM once per evaluation.
#include "columns.cuh"

namespace fm {

namespace {

// 3-D: for y-frequencies (ky, py-ky) and a tile of kx, forward z-transform of the
// nz physical planes (zero-padded to pz), multiply by -N(k), inverse, keep nz planes.
__global__ void __launch_bounds__(kThreads) z_convolve_kernel(const ColPass p) {
    pdl_wait();
    if (p.early) pdl_trigger();
    extern __shared__ __align__(16) unsigned char smem[];
    const Grid &g = p.g;
    const int tx = p.tx, kx0 = blockIdx.x * tx, ncol = min(tx, g.nkx - kx0);
    const int kya = blockIdx.y;
    int kyb;
    const int np = ky_pair(kya, g.py, kyb);
    const int ls = skewed_len(g.pz);
    const int nl = np * 3 * tx;  // line (q, c, col) at ((q*3 + c)*tx + col)
    float2 *a = reinterpret_cast<float2 *>(smem);
    float2 *b = a + (size_t)2 * 3 * tx * ls;
    const size_t cstride = (size_t)g.nz * g.py * g.xs;  // component stride of Y
    const size_t zstride = (size_t)g.py * g.xs;
    batched_copy<8>(
        np * 3 * g.nz * tx,
        [&](int idx) {
            const int r1 = p.fd_tx.div(idx), col = idx - r1 * tx;
            const int r2 = g.fd_nz.div(r1), z = r1 - r2 * g.nz;
            const int q = r2 / 3, c = r2 - 3 * q;
            const int ky = q ? kyb : kya;
            return col < ncol ? p.in[c * cstride + z * zstride + (size_t)ky * g.xs + kx0 + col] : make_float2(0.f, 0.f);
        },
        [&](int idx, float2 v) {
            const int r1 = p.fd_tx.div(idx), col = idx - r1 * tx;
            const int r2 = g.fd_nz.div(r1), z = r1 - r2 * g.nz;
            a[(r2 * tx + col) * ls + sk(z)] = v;
        });
    // zero the padded planes z in [nz, pz): one warp per line
    for (int line = threadIdx.x >> 5; line < nl; line += blockDim.x >> 5)
        for (int z = g.nz + (threadIdx.x & 31); z < g.pz; z += 32) a[line * ls + sk(z)] = make_float2(0.f, 0.f);
    __syncthreads();
    float2 *r = fft_lines(a, b, nl, ls, p.plan, false);
    float2 *o = (r == a) ? b : a;
    if (g.per) {  // complex kernel K[c][kz][ky][kx]
        const size_t kcp = (size_t)g.pz * g.py * g.ks;
        for (int idx = threadIdx.x; idx < np * g.pz * tx; idx += blockDim.x) {
            const int r1 = p.fd_tx.div(idx), col = idx - r1 * tx;
            const int q = r1 >= g.pz ? 1 : 0, kz = r1 - q * g.pz;
            const int kx = min(kx0 + col, g.nkx - 1), ky = q ? kyb : kya;
            const float2 *K = reinterpret_cast<const float2 *>(p.kern) + ((size_t)kz * g.py + ky) * g.ks + kx;
            multiply_periodic(K, kcp, false, r + ((q * 3 + 0) * tx + col) * ls + sk(kz), r + ((q * 3 + 1) * tx + col) * ls + sk(kz),
                              r + ((q * 3 + 2) * tx + col) * ls + sk(kz));
        }
    }
    const size_t kc = (size_t)g.nkz * g.nky * g.ks;
    for (int idx = threadIdx.x; idx < (g.per ? 0 : g.pz * tx); idx += blockDim.x) {
        const int kz = p.fd_tx.div(idx), col = idx - kz * tx;
        const int kx = min(kx0 + col, g.nkx - 1);
        int kzm;
        float sz;
        kernel_mirror(kz, g.pz, kzm, sz);
        const float *K = p.kern + ((size_t)kzm * g.nky + kya) * g.ks + kx;
        const float kxx = __ldg(K), kyy = __ldg(K + kc), kzz = __ldg(K + 2 * kc);
        const float kxy0 = __ldg(K + 3 * kc), kxz = sz * __ldg(K + 4 * kc), kyz0 = sz * __ldg(K + 5 * kc);
        for (int q = 0; q < np; ++q) {
            // the second frequency of the pair is the y-mirror: odd-in-y components flip sign
            const float sy = q ? -1.f : 1.f;
            const float kxy = sy * kxy0, kyz = sy * kyz0;
            float2 *lx = r + ((q * 3 + 0) * tx + col) * ls + sk(kz);
            float2 *ly = r + ((q * 3 + 1) * tx + col) * ls + sk(kz);
            float2 *lz = r + ((q * 3 + 2) * tx + col) * ls + sk(kz);
            const float2 mx = *lx, my = *ly, mz = *lz;
            *lx = make_float2(-(kxx * mx.x + kxy * my.x + kxz * mz.x), -(kxx * mx.y + kxy * my.y + kxz * mz.y));
            *ly = make_float2(-(kxy * mx.x + kyy * my.x + kyz * mz.x), -(kxy * mx.y + kyy * my.y + kyz * mz.y));
            *lz = make_float2(-(kxz * mx.x + kyz * my.x + kzz * mz.x), -(kxz * mx.y + kyz * my.y + kzz * mz.y));
        }
    }
    __syncthreads();
    float2 *qb = fft_lines(r, o, nl, ls, p.plan, true);
    for (int idx = threadIdx.x; idx < np * 3 * g.nz * tx; idx += blockDim.x) {
        const int r1 = p.fd_tx.div(idx), col = idx - r1 * tx;
        const int r2 = g.fd_nz.div(r1), z = r1 - r2 * g.nz;
        const int q = r2 / 3, c = r2 - 3 * q;
        const int ky = q ? kyb : kya;
        if (col < ncol)
            p.out[c * cstride + z * zstride + (size_t)ky * g.xs + kx0 + col] = qb[((q * 3 + c) * tx + col) * ls + sk(z)];
    }
}

// Pruned two-level z convolution for pz = N1 * N2.  With z = N2 z1 + z2 and
// k = k1 + N1 k2 the transform of one z line is
//   X[k1 + N1 k2] = sum_z2 W_N2^{z2 k2} W_pz^{z2 k1} sum_z1 x[N2 z1 + z2] W_N1^{z1 k1}
// and its inverse runs the same factors backwards.  Inputs vanish for z >= pz/2 (z1 >=
// N1/2) and only z < nz <= pz/2 is kept, so the outer N1-point passes work on half
// lines: a half-input DFT is two N1/2-point DFTs (even and odd outputs), a half-output
// inverse is two N1/2-point inverses.  Phase 1 (line, z2): global loads straight into
// registers, half-input DFT, twiddle, one shared-memory write.  Phase 2 (ky of the pair,
// column, k1; all three components): N2-point DFTs, the tensor multiply, inverse
// N2-point DFTs, conjugate twiddle, in place.  Phase 3 (line, z2): half-output inverse
// straight to global memory.  Two barriers per tile, one buffer.
template <int N1, int N2>
__global__ void __launch_bounds__(kThreads, (N1 * N2 <= 128) ? 3 : 1) z_convolve_fused_kernel(const ColPass p) {
    pdl_wait();
    if (p.early) pdl_trigger();
    constexpr int N = N1 * N2, H1 = N1 / 2;
    constexpr int ls = skewed_len(N);
    extern __shared__ __align__(16) unsigned char smem[];
    float2 *buf = reinterpret_cast<float2 *>(smem);  // line (q, c, col) at ((q*3 + c)*tx + col)*ls
    const Grid &g = p.g;
    const int tx = p.tx, kx0 = blockIdx.x * tx, ncol = min(tx, g.nkx - kx0);
    const int kya = blockIdx.y;
    int kyb;
    const int np = ky_pair(kya, g.py, kyb);
    const int nz = g.nz;
    const size_t cstride = (size_t)nz * g.py * g.xs;  // component stride of Y
    const size_t zstride = (size_t)g.py * g.xs;
    const float2 *__restrict__ tw = p.plan.tw;        // e^{-2 pi i e / N}

    // phase 1: item (r2, z2, col), col fastest
    const int n13 = np * 3 * N2 * ncol;
    for (int it = threadIdx.x; it < n13; it += blockDim.x) {
        int rz, col;
        tile_item(p, ncol, it, rz, col);
        const int z2 = rz % N2, r2 = rz / N2;
        const int q = r2 >= 3, c = r2 - 3 * q;
        const int ky = q ? kyb : kya;
        const float2 *src = p.in + c * cstride + (size_t)ky * g.xs + kx0 + col;
        float2 e[H1];
#pragma unroll
        for (int z1 = 0; z1 < H1; ++z1) {
            const int z = N2 * z1 + z2;
            e[z1] = z < nz ? src[(size_t)z * zstride] : make_float2(0.f, 0.f);
        }
        half_dft_store<N1, N2>(e, z2, buf + (r2 * tx + col) * ls, tw);
    }
    __syncthreads();

    // phase 2: item (q, k1, col), col fastest; all three components of one frequency column
    const size_t kc = (size_t)g.nkz * g.nky * g.ks;
    const int n2 = np * N1 * ncol;
    for (int it = threadIdx.x; it < n2; it += blockDim.x) {
        int qk, col;
        tile_item(p, ncol, it, qk, col);
        const int k1 = qk % N1, q = qk / N1;
        float2 m[3][N2];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 *line = buf + ((q * 3 + c) * tx + col) * ls;
#pragma unroll
            for (int z2 = 0; z2 < N2; ++z2) m[c][z2] = line[sk(k1 * N2 + z2)];
            dft_small<N2>(m[c], false);
        }
        const int kx = min(kx0 + col, g.nkx - 1);
        // the second frequency of the pair is the y-mirror: odd-in-y components flip sign
        const float sy = q ? -1.f : 1.f;
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) {
            int kzm;
            float sz;
            kernel_mirror(k1 + N1 * k2, N, kzm, sz);
            const float *K = p.kern + ((size_t)kzm * g.nky + kya) * g.ks + kx;
            const float kxx = __ldg(K), kyy = __ldg(K + kc), kzz = __ldg(K + 2 * kc);
            const float kxy = sy * __ldg(K + 3 * kc), kxz = sz * __ldg(K + 4 * kc), kyz = sy * sz * __ldg(K + 5 * kc);
            const float2 mx = m[0][k2], my = m[1][k2], mz = m[2][k2];
            m[0][k2] = make_float2(-(kxx * mx.x + kxy * my.x + kxz * mz.x), -(kxx * mx.y + kxy * my.y + kxz * mz.y));
            m[1][k2] = make_float2(-(kxy * mx.x + kyy * my.x + kyz * mz.x), -(kxy * mx.y + kyy * my.y + kyz * mz.y));
            m[2][k2] = make_float2(-(kxz * mx.x + kyz * my.x + kzz * mz.x), -(kxz * mx.y + kyz * my.y + kzz * mz.y));
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            dft_small<N2>(m[c], true);
            float2 *line = buf + ((q * 3 + c) * tx + col) * ls;
#pragma unroll
            for (int z2 = 0; z2 < N2; ++z2)
                line[sk(k1 * N2 + z2)] = (z2 && k1) ? cmul(m[c][z2], cconj(__ldg(tw + z2 * k1))) : m[c][z2];
        }
    }
    __syncthreads();

    // phase 3: item (r2, z2, col), col fastest; outputs z1 < N1/2 with z < nz
    for (int it = threadIdx.x; it < n13; it += blockDim.x) {
        int rz, col;
        tile_item(p, ncol, it, rz, col);
        const int z2 = rz % N2, r2 = rz / N2;
        const int q = r2 >= 3, c = r2 - 3 * q;
        const int ky = q ? kyb : kya;
        float2 e[H1];
        half_idft_load<N1, N2>(e, z2, buf + (r2 * tx + col) * ls, tw);
        float2 *dst = p.out + c * cstride + (size_t)ky * g.xs + kx0 + col;
#pragma unroll
        for (int z1 = 0; z1 < H1; ++z1) {
            const int z = N2 * z1 + z2;
            if (z < nz) dst[(size_t)z * zstride] = e[z1];
        }
    }
}

__device__ __forceinline__ void cp_async16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The pruned two-level z convolution on y-frequency pairs in packed FP32x2 form: lane A
// is ky, lane B is py - ky (the two share every twiddle and, up to the sign of the
// odd-in-y components xy and yz, every kernel value).  Tiles of 8 kx columns; phase 1
// item (c, z2, col), phase 2 item (k1, col) with all three components of both lanes,
// phase 3 item (c, z2, col).  Shared memory holds pair elements (float4), so the
// buffer is the size of the unpaired kernel's.  For ky = 0 and ky = py/2 (no partner)
// lane B repeats lane A and is not stored.
template <int N1, int N2>
__global__ void __launch_bounds__(3 * N2 * 8, N2 >= 7 ? 2 : 3) z_convolve_pair_kernel(const ColPass p) {
    pdl_wait();
    if (p.early) pdl_trigger();
    constexpr int N = N1 * N2, H1 = N1 / 2, TX = 8;
    constexpr int ls = skewed_len(N);
    extern __shared__ __align__(16) unsigned char smem[];
    float4 *buf = reinterpret_cast<float4 *>(smem);  // line (c, col) at (c*TX + col)*ls
    const Grid &g = p.g;
    const int kx0 = blockIdx.x * TX, ncol = min(TX, g.nkx - kx0);
    const int kya = blockIdx.y;
    int kyb;
    const int np = ky_pair(kya, g.py, kyb);
    const int kyB = np == 2 ? kyb : kya;
    const int nz = g.nz;
    const size_t cstride = (size_t)nz * g.py * g.xs;  // component stride of Y
    const size_t zstride = (size_t)g.py * g.xs;
    const float2 *__restrict__ tw = p.plan.tw;        // e^{-2 pi i e / N}

    // the tile's kernel values [6][N/2 + 1][8], in flight during phase 1 (rows are 16-byte aligned)
    const size_t kc = (size_t)g.nkz * g.nky * g.ks;
    constexpr int NKZ = N / 2 + 1;
    float *kt = reinterpret_cast<float *>(buf + 3 * TX * ls);
    for (int r = threadIdx.x; r < 2 * 6 * NKZ; r += blockDim.x) {
        const int h = r & 1, ck = r >> 1, c = ck / NKZ, kz = ck - c * NKZ;
        if (kx0 + 4 * h < g.ks)
            cp_async16(kt + 4 * r, p.kern + c * kc + ((size_t)kz * g.nky + kya) * g.ks + kx0 + 4 * h);
    }

    // phase 1: item (c, z2, col), col fastest
    for (int it = threadIdx.x; it < 3 * N2 * TX; it += blockDim.x) {
        const int col = it & (TX - 1), cz = it >> 3;
        if (col >= ncol) continue;
        const int z2 = cz % N2, c = cz / N2;
        const float2 *srcA = p.in + c * cstride + (size_t)kya * g.xs + kx0 + col;
        const float2 *srcB = p.in + c * cstride + (size_t)kyB * g.xs + kx0 + col;
        cp2 e[H1];
#pragma unroll
        for (int z1 = 0; z1 < H1; ++z1) {
            const int z = N2 * z1 + z2;
            e[z1] = z < nz ? ppack(srcA[(size_t)z * zstride], srcB[(size_t)z * zstride]) : pzero();
        }
        phalf_dft_store<N1, N2>(e, z2, buf + (c * TX + col) * ls, tw);
    }
    cp_async_wait();
    __syncthreads();

    // phase 2: item (k1, col); inner DFTs, the tensor multiply, inverse inner DFTs
    for (int it = threadIdx.x; it < N1 * TX; it += blockDim.x) {
        const int col = it & (TX - 1), k1 = it >> 3;
        if (col >= ncol) continue;
        cp2 m[3][N2];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float4 *line = buf + (c * TX + col) * ls;
#pragma unroll
            for (int z2 = 0; z2 < N2; ++z2) m[c][z2] = pload(line[sk(k1 * N2 + z2)]);
            pdft<N2>(m[c], false);
        }
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) {
            int kzm;
            float sz;
            kernel_mirror(k1 + N1 * k2, N, kzm, sz);
            const float *K = kt + kzm * TX + col;
            const float kxx = K[0], kyy = K[NKZ * TX], kzz = K[2 * NKZ * TX];
            const float kxy = K[3 * NKZ * TX], kxz = sz * K[4 * NKZ * TX], kyz = sz * K[5 * NKZ * TX];
            // H = -N M; lane B (py - ky) flips the odd-in-y components xy and yz
            const float2 Nxx = pb(-kxx), Nyy = pb(-kyy), Nzz = pb(-kzz), Nxz = pb(-kxz);
            const float2 Nxy = make_float2(-kxy, kxy), Nyz = make_float2(-kyz, kyz);
            const cp2 mx = m[0][k2], my = m[1][k2], mz = m[2][k2];
            m[0][k2] = {__ffma2_rn(Nxz, mz.re, __ffma2_rn(Nxy, my.re, __fmul2_rn(Nxx, mx.re))),
                        __ffma2_rn(Nxz, mz.im, __ffma2_rn(Nxy, my.im, __fmul2_rn(Nxx, mx.im)))};
            m[1][k2] = {__ffma2_rn(Nyz, mz.re, __ffma2_rn(Nyy, my.re, __fmul2_rn(Nxy, mx.re))),
                        __ffma2_rn(Nyz, mz.im, __ffma2_rn(Nyy, my.im, __fmul2_rn(Nxy, mx.im)))};
            m[2][k2] = {__ffma2_rn(Nzz, mz.re, __ffma2_rn(Nyz, my.re, __fmul2_rn(Nxz, mx.re))),
                        __ffma2_rn(Nzz, mz.im, __ffma2_rn(Nyz, my.im, __fmul2_rn(Nxz, mx.im)))};
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            pdft<N2>(m[c], true);
            float4 *line = buf + (c * TX + col) * ls;
#pragma unroll
            for (int z2 = 0; z2 < N2; ++z2)
                line[sk(k1 * N2 + z2)] = pstore((z2 && k1) ? pmulw(m[c][z2], __ldg(tw + z2 * k1), true) : m[c][z2]);
        }
    }
    __syncthreads();

    // phase 3: item (c, z2, col); outputs z1 < N1/2 with z < nz
    for (int it = threadIdx.x; it < 3 * N2 * TX; it += blockDim.x) {
        const int col = it & (TX - 1), cz = it >> 3;
        if (col >= ncol) continue;
        const int z2 = cz % N2, c = cz / N2;
        cp2 e[H1];
        phalf_idft_load<N1, N2>(e, z2, buf + (c * TX + col) * ls, tw);
        float2 *dstA = p.out + c * cstride + (size_t)kya * g.xs + kx0 + col;
        float2 *dstB = p.out + c * cstride + (size_t)kyb * g.xs + kx0 + col;
#pragma unroll
        for (int z1 = 0; z1 < H1; ++z1) {
            const int z = N2 * z1 + z2;
            if (z < nz) {
                dstA[(size_t)z * zstride] = plane_a(e[z1]);
                if (np == 2) dstB[(size_t)z * zstride] = plane_b(e[z1]);
            }
        }
    }
}

// pz <= 24: one thread per (kx, ky) holds the three components' z columns in registers, so
// the pass is one read and one write of Y with no shared memory and no barrier.  3 nz
// independent loads a thread keep enough bytes in flight at two to four CTAs of 128 threads
// per SM.
template <int PZ, bool PER>
__global__ void __launch_bounds__(128, PZ <= 8 ? 4 : PZ <= 14 ? 3 : 2) z_convolve_register_kernel(const ColPass p) {
    pdl_wait();
    if (p.early) pdl_trigger();
    constexpr int H = PZ / 2;
    const Grid &g = p.g;
    const int idx = blockIdx.x * 128 + threadIdx.x;
    if (idx >= g.py * g.nkx) return;
    const int ky = g.fd_nkx.div(idx), kx = idx - ky * g.nkx, nz = g.nz;
    const size_t plane = (size_t)g.py * g.xs, at = (size_t)ky * g.xs + kx;
    float2 v[3][H];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int z = 0; z < H; ++z) v[c][z] = z < nz ? p.in[(size_t)(c * nz + z) * plane + at] : make_float2(0.f, 0.f);
    if constexpr (PER) {
        const size_t kp = (size_t)g.py * g.ks;
        z_column_convolve<PZ, true>(
            v, reinterpret_cast<const float *>(reinterpret_cast<const float2 *>(p.kern) + (size_t)ky * g.ks + kx), kp,
            PZ * kp, 1.f, p.plan.tw);
    } else {
        int kym;
        float sy;
        kernel_mirror(ky, g.py, kym, sy);
        z_column_convolve<PZ, false>(v, p.kern + (size_t)kym * g.ks + kx, (size_t)g.nky * g.ks,
                                     (size_t)g.nkz * g.nky * g.ks, sy, p.plan.tw);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int z = 0; z < H; ++z)
            if (z < nz) p.out[(size_t)(c * nz + z) * plane + at] = v[c][z];
}

}  // namespace

namespace {
template <int N1, int N2>
cudaError_t launch_z_fused(const ColPass &p, cudaStream_t s) {
    const size_t sm = sizeof(float2) * (size_t)2 * 3 * p.tx * skewed_len(N1 * N2);
    cudaError_t e = ensure_smem((const void *)z_convolve_fused_kernel<N1, N2>, sm);
    if (e != cudaSuccess) return e;
    return launch_pdl(z_convolve_fused_kernel<N1, N2>, dim3(tiles(p), p.g.nky), dim3(kThreads), sm, s, p);
}
// every physical plane in the lower half of an open z, the octant kernel
bool z_fused_ok(const Grid &g) { return g.per == 0 && two_level_length(g.pz) && 2 * g.nz <= g.pz; }
}  // namespace

size_t z_convolve_smem(const Grid &g, int tx) {
    const size_t one = sizeof(float2) * (size_t)2 * 3 * tx * skewed_len(g.pz);
    return z_fused_ok(g) ? one : 2 * one;
}

namespace {

template <int N1, int N2>
cudaError_t launch_z_pair(const ColPass &p, cudaStream_t s) {
    const void *fn = (const void *)z_convolve_pair_kernel<N1, N2>;
    const size_t sm = sizeof(float4) * (size_t)3 * 8 * skewed_len(N1 * N2) + sizeof(float) * 6 * (N1 * N2 / 2 + 1) * 8;
    cudaError_t e = ensure_smem(fn, sm);
    if (e != cudaSuccess) return e;
    return launch_pdl(z_convolve_pair_kernel<N1, N2>, dim3(tiles(p), p.g.nky), dim3(3 * N2 * 8), sm, s, p);
}

template <int PZ>
cudaError_t launch_z_register(const ColPass &p, cudaStream_t s) {
    const auto fn = p.g.per ? z_convolve_register_kernel<PZ, true> : z_convolve_register_kernel<PZ, false>;
    return launch_pdl(fn, dim3((unsigned)(p.g.py * p.g.nkx + 127) / 128), dim3(128), 0, s, p);
}
}  // namespace

// the packed ky-pair z pass: tile 8, inner radix 4 to 8, kernel rows at 16-byte boundaries (cp.async)
bool z_convolve_pair_ok(const Grid &g, int tx) {
    return tx == 8 && z_fused_ok(g) && g.pz >= 32 && g.pz <= 128 && g.ks % 4 == 0;
}
bool z_register_length_ok(int pz) { return z_register_length(pz); }
bool z_convolve_register_ok(const Grid &g) {
    return !(g.per & 4) && z_register_length(g.pz) && 2 * g.nz <= g.pz && (long long)g.py * g.nkx < (1ll << 30);
}

cudaError_t launch_z_convolve(const ColPass &p, cudaStream_t s) {
    if (p.pipe == 1) {
        if (!z_convolve_pair_ok(p.g, p.tx)) return cudaErrorInvalidValue;
        switch (p.g.pz) {
            case 32: return launch_z_pair<8, 4>(p, s);
            case 40: return launch_z_pair<8, 5>(p, s);
            case 48: return launch_z_pair<8, 6>(p, s);
            case 56: return launch_z_pair<8, 7>(p, s);
            case 64: return launch_z_pair<8, 8>(p, s);
            case 80: return launch_z_pair<10, 8>(p, s);
            case 96: return launch_z_pair<12, 8>(p, s);
            case 112: return launch_z_pair<14, 8>(p, s);
            default: return launch_z_pair<16, 8>(p, s);
        }
    }
    if (p.pipe == 2) {
        if (!z_convolve_register_ok(p.g)) return cudaErrorInvalidValue;
#define FM_CASE(n) \
    case n: return launch_z_register<n>(p, s);
        switch (p.g.pz) {
            FM_CASE(2) FM_CASE(4) FM_CASE(6) FM_CASE(8) FM_CASE(10) FM_CASE(12) FM_CASE(14) FM_CASE(16) FM_CASE(20) FM_CASE(24)
        }
#undef FM_CASE
        return cudaErrorInvalidValue;
    }
    if (z_fused_ok(p.g)) {
        if (p.split != 0) switch (p.g.pz) {  // radix split, as launch_y_dispatch
                case 16: return launch_z_fused<8, 2>(p, s);
                case 32: return launch_z_fused<4, 8>(p, s);
                case 64: return launch_z_fused<16, 4>(p, s);
                case 128: return launch_z_fused<32, 4>(p, s);
                case 256: return launch_z_fused<32, 8>(p, s);
            }
#define FM_CASE(n) \
    case n: return launch_z_fused<split_line(n), n / split_line(n)>(p, s);
        switch (p.g.pz) { FM_LENGTHS_TO_256(FM_CASE) FM_LENGTHS_LONG(FM_CASE) }
#undef FM_CASE
    }
    // room for a y-frequency pair: 2 x 3 lines per kx column, two ping-pong buffers
    const size_t sm = 2 * sizeof(float2) * (size_t)2 * 3 * p.tx * skewed_len(p.g.pz);
    cudaError_t e = ensure_smem((const void *)z_convolve_kernel, sm);
    if (e != cudaSuccess) return e;
    return launch_pdl(z_convolve_kernel, dim3(tiles(p), p.g.nky), dim3(kThreads), sm, s, p);
}

}  // namespace fm
