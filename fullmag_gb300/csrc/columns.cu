// columns.cu -- y transforms of the demag convolution, plus the deterministic final
// reduction of the per-block statistics of large grids and of batched problems.
//
// Reference behaviour restated (paths in mzrptu/fullmag):
//   multi-pass FP64 reductions                 native/backends/fdm/src/reductions_fp64.cu:30-84,354-393
#include "columns.cuh"
#include "stats.cuh"

namespace fm {

namespace {

// X[c][z][y<ny][kx] -> Y[c][z][ky<py][kx] (forward along y, zero rows pruned)
__global__ void __launch_bounds__(kThreads) y_forward_kernel(const ColPass p) {
    pdl_wait();
    if (p.early) pdl_trigger();
    extern __shared__ __align__(16) unsigned char smem[];
    const Grid &g = p.g;
    const int tx = p.tx, kx0 = blockIdx.x * tx, ncol = min(tx, g.nkx - kx0);
    const int z = blockIdx.y, c = blockIdx.z;
    const int ls = skewed_len(g.py);
    float2 *a = reinterpret_cast<float2 *>(smem);
    float2 *b = a + tx * ls;
    const float2 *src = p.in + ((size_t)c * g.nz + z) * g.ny * g.xs;
    batched_copy<8>(
        g.ny * tx,
        [&](int idx) {
            const int y = p.fd_tx.div(idx), col = idx - y * tx;
            return col < ncol ? src[(size_t)y * g.xs + kx0 + col] : make_float2(0.f, 0.f);
        },
        [&](int idx, float2 v) {
            const int y = p.fd_tx.div(idx), col = idx - y * tx;
            a[col * ls + sk(y)] = v;
        });
    for (int line = threadIdx.x >> 5; line < tx; line += blockDim.x >> 5)  // zero padding rows
        for (int y = g.ny + (threadIdx.x & 31); y < g.py; y += 32) a[line * ls + sk(y)] = make_float2(0.f, 0.f);
    __syncthreads();
    float2 *r = fft_lines(a, b, tx, ls, p.plan, false);
    float2 *dst = p.out + ((size_t)c * g.nz + z) * g.py * g.xs;
    for (int idx = threadIdx.x; idx < g.py * tx; idx += blockDim.x) {
        const int y = p.fd_tx.div(idx), col = idx - y * tx;
        if (col < ncol) dst[(size_t)y * g.xs + kx0 + col] = r[col * ls + sk(y)];
    }
}

// Y[c][z][ky][kx] -> X[c][z][y<ny][kx] (inverse along y, only physical rows kept)
// (WIDE: long_butterflies, columns.cuh; the forward pass loads in batches and needs no such help)
template <bool WIDE>
__global__ void __launch_bounds__(kThreads, general_ctas(WIDE)) y_inverse_kernel(const ColPass p) {
    pdl_wait();
    if (p.early) pdl_trigger();
    extern __shared__ __align__(16) unsigned char smem[];
    const Grid &g = p.g;
    const int tx = p.tx, kx0 = blockIdx.x * tx, ncol = min(tx, g.nkx - kx0);
    const int z = blockIdx.y, c = blockIdx.z;
    const int ls = skewed_len(g.py);
    float2 *a = reinterpret_cast<float2 *>(smem);
    float2 *b = a + tx * ls;
    const float2 *src = p.in + ((size_t)c * g.nz + z) * g.py * g.xs;
    batched_copy<8>(
        g.py * tx,
        [&](int idx) {
            const int y = p.fd_tx.div(idx), col = idx - y * tx;
            return col < ncol ? src[(size_t)y * g.xs + kx0 + col] : make_float2(0.f, 0.f);
        },
        [&](int idx, float2 v) {
            const int y = p.fd_tx.div(idx), col = idx - y * tx;
            a[col * ls + sk(y)] = v;
        });
    __syncthreads();
    float2 *r = fft_lines(a, b, tx, ls, p.plan, true);
    float2 *dst = p.out + ((size_t)c * g.nz + z) * g.ny * g.xs;
    for (int idx = threadIdx.x; idx < g.ny * tx; idx += blockDim.x) {
        const int y = p.fd_tx.div(idx), col = idx - y * tx;
        if (col < ncol) dst[(size_t)y * g.xs + kx0 + col] = r[col * ls + sk(y)];
    }
}

// ---- two-level transforms (fft_smem.cuh) ----

// CTA size: a tile of 16 columns gives every thread whole butterflies in the longer pass
__host__ __device__ constexpr int y_threads(int n1) { return n1 == 20 ? 320 : n1 == 24 ? 192 : n1 == 28 ? 224 : kThreads; }

// X[c][z][y<ny][kx] -> Y[c][z][ky<py][kx], py = N1 * N2: outer pass from global memory (half
// lines on an open y; FULL: periodic, ny = py), inner N2-point pass straight to global
// memory, one barrier.
template <int N1, int N2, bool FULL>
__global__ void __launch_bounds__(y_threads(N1), 2) y_forward_fused_kernel(const ColPass p) {
    pdl_wait();
    if (p.early) pdl_trigger();
    constexpr int N = N1 * N2, H1 = N1 / 2;
    constexpr int ls = skewed_len(N);
    extern __shared__ __align__(16) unsigned char smem[];
    float2 *buf = reinterpret_cast<float2 *>(smem);
    const Grid &g = p.g;
    const int tx = p.tx, kx0 = blockIdx.x * tx, ncol = min(tx, g.nkx - kx0);
    const int z = blockIdx.y, c = blockIdx.z;
    const float2 *__restrict__ tw = p.plan.tw;
    const float2 *src = p.in + ((size_t)c * g.nz + z) * g.ny * g.xs + kx0;
    for (int it = threadIdx.x; it < N2 * ncol; it += blockDim.x) {
        int n2, col;
        tile_item(p, ncol, it, n2, col);
        float2 e[H1];
#pragma unroll
        for (int n1 = 0; n1 < H1; ++n1) {
            const int y = N2 * n1 + n2;
            e[n1] = y < g.ny ? src[(size_t)y * g.xs + col] : make_float2(0.f, 0.f);
        }
        if constexpr (FULL) {
            float2 f[H1];
#pragma unroll
            for (int n1 = 0; n1 < H1; ++n1) f[n1] = src[(size_t)(N2 * (n1 + H1) + n2) * g.xs + col];
            full_dft_store<N1, N2>(e, f, n2, buf + col * ls, tw);
        } else {
            half_dft_store<N1, N2>(e, n2, buf + col * ls, tw);
        }
    }
    __syncthreads();
    float2 *dst = p.out + ((size_t)c * g.nz + z) * g.py * g.xs + kx0;
    for (int it = threadIdx.x; it < N1 * ncol; it += blockDim.x) {
        int k1, col;
        tile_item(p, ncol, it, k1, col);
        const float2 *line = buf + col * ls;
        float2 v[N2];
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) v[n2] = line[sk(k1 * N2 + n2)];
        dft_small<N2>(v, false);
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) dst[(size_t)(k1 + N1 * k2) * g.xs + col] = v[k2];
    }
}

// Y[c][z][ky][kx] -> X[c][z][y<ny][kx]: inner inverse N2-point pass from global memory,
// outer pass straight to global memory, one barrier.
template <int N1, int N2, bool FULL>
__global__ void __launch_bounds__(y_threads(N1), 2) y_inverse_fused_kernel(const ColPass p) {
    pdl_wait();
    if (p.early) pdl_trigger();
    constexpr int N = N1 * N2, H1 = N1 / 2;
    constexpr int ls = skewed_len(N);
    extern __shared__ __align__(16) unsigned char smem[];
    float2 *buf = reinterpret_cast<float2 *>(smem);
    const Grid &g = p.g;
    const int tx = p.tx, kx0 = blockIdx.x * tx, ncol = min(tx, g.nkx - kx0);
    const int z = blockIdx.y, c = blockIdx.z;
    const float2 *__restrict__ tw = p.plan.tw;
    const float2 *src = p.in + ((size_t)c * g.nz + z) * g.py * g.xs + kx0;
    for (int it = threadIdx.x; it < N1 * ncol; it += blockDim.x) {
        int k1, col;
        tile_item(p, ncol, it, k1, col);
        float2 v[N2];
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) v[k2] = src[(size_t)(k1 + N1 * k2) * g.xs + col];
        dft_small<N2>(v, true);
        float2 *line = buf + col * ls;
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2)
            line[sk(k1 * N2 + n2)] = (n2 && k1) ? cmul(v[n2], cconj(__ldg(tw + n2 * k1))) : v[n2];
    }
    __syncthreads();
    float2 *dst = p.out + ((size_t)c * g.nz + z) * g.ny * g.xs + kx0;
    for (int it = threadIdx.x; it < N2 * ncol; it += blockDim.x) {
        int n2, col;
        tile_item(p, ncol, it, n2, col);
        float2 e[H1], f[H1];
        idft_load<N1, N2, FULL>(e, f, n2, buf + col * ls, tw);
#pragma unroll
        for (int n1 = 0; n1 < H1; ++n1) {
            const int y = N2 * n1 + n2;
            if (y < g.ny) dst[(size_t)y * g.xs + col] = e[n1];
            if (FULL) dst[(size_t)(y + N2 * H1) * g.xs + col] = f[n1];
        }
    }
}

// Deterministic final reduction of the per-block partials (layout [stat][block] of
// float-float pairs): the threads stride over the blocks with compensated TwoSum
// accumulation for the energies and max for the norms, all nine statistics at once;
// warp butterflies and one barrier combine the threads in a fixed order.  GB300's FP64
// rate is a small fraction of its FP32 rate, so the compensation runs on FP32 pipes;
// only the final hi + lo is formed in FP64.
constexpr int kFinThreads = 1024;

// One butterfly level: float-float sums combined in lane order (every lane ends with
// the same bits), maxima by fmaxf.
__device__ __forceinline__ void fin_level(float (&h)[kNumStats], float (&l)[kNumStats], int o) {
    const bool low = (threadIdx.x & o) == 0;
#pragma unroll
    for (int s = 0; s < kNumStats; ++s) {
        const float oh = __shfl_xor_sync(0xffffffffu, h[s], o);
        const float ol = __shfl_xor_sync(0xffffffffu, l[s], o);
        if (s < 5) {
            float ah = low ? h[s] : oh, al = low ? l[s] : ol;
            ff_add(ah, al, low ? oh : h[s]);
            al += low ? ol : l[s];
            h[s] = ah;
            l[s] = al;
        } else {
            h[s] = fmaxf(h[s], oh);
        }
    }
}

__device__ __forceinline__ void finalize_body(const float2 *__restrict__ partials, int nblocks, double *__restrict__ out) {
    __shared__ float2 sh[kFinThreads / 32][kNumStats];
    float h[kNumStats], l[kNumStats];
#pragma unroll
    for (int s = 0; s < kNumStats; ++s) h[s] = l[s] = 0.f;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
#pragma unroll
        for (int s = 0; s < kNumStats; ++s) {
            const float2 v = partials[(size_t)s * nblocks + b];
            if (s < 5) {
                ff_add(h[s], l[s], v.x);
                l[s] += v.y;
            } else {
                h[s] = fmaxf(h[s], v.x);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) fin_level(h, l, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane == 0) {
#pragma unroll
        for (int s = 0; s < kNumStats; ++s) sh[wid][s] = make_float2(h[s], l[s]);
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int s = 0; s < kNumStats; ++s) {
            const float2 v = lane < nw ? sh[lane][s] : make_float2(0.f, 0.f);
            h[s] = v.x;
            l[s] = v.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) fin_level(h, l, o);
        if (lane == 0) {
#pragma unroll
            for (int s = 0; s < kNumStats; ++s) out[s] = (double)h[s] + (double)l[s];
        }
    }
}

// One problem; up to kFinInPass CTAs in the order of the row pass that reduces its own.
__global__ void __launch_bounds__(kFinThreads) finalize_stats_kernel(const float2 *__restrict__ partials, int nblocks,
                                                                     double *__restrict__ out, int early) {
    pdl_wait();
    if (early) pdl_trigger();
    if (nblocks > kFinInPass) finalize_body(partials, nblocks, out);
    else if (threadIdx.x >> 5 < kNumStats) finalize_stat(partials, nblocks, threadIdx.x >> 5, out);
}
// One block per problem; statistics land in out[problem * kNumStats + s].
__global__ void __launch_bounds__(kFinThreads) finalize_batched_kernel(const FinDesc *__restrict__ fd, double *__restrict__ out) {
    const FinDesc d = fd[blockIdx.x];
    finalize_body(d.partials, d.nblocks, out + (size_t)blockIdx.x * kNumStats);
}

}  // namespace

int col_tile(const Grid &g, int lines_per_col, int len) {
    // largest tile (<= 8 kx columns) whose two ping-pong buffers fit in 200 KB
    int tx = 8;
    while (tx > 1 && (size_t)2 * lines_per_col * tx * skewed_len(len) * sizeof(float2) > 200u * 1024u) tx >>= 1;
    return tx;
}

namespace {
// the two-level y passes: every physical row in the lower half of an open y, or a periodic y
bool y_fused_ok(const Grid &g) { return two_level_length(g.py) && ((g.per & 2) ? g.ny == g.py : 2 * g.ny <= g.py); }
template <int N1, int N2, bool INV, bool FULL>
cudaError_t launch_y_fused(const ColPass &p, cudaStream_t s) {
    const size_t sm = sizeof(float2) * (size_t)p.tx * skewed_len(N1 * N2);
    const auto fn = INV ? y_inverse_fused_kernel<N1, N2, FULL> : y_forward_fused_kernel<N1, N2, FULL>;
    cudaError_t e = ensure_smem((const void *)fn, sm);
    if (e != cudaSuccess) return e;
    // a narrower tile takes a smaller CTA (at least 64 threads), so more of them overlap on an SM
    const int threads = p.tx < 16 ? std::max(64, y_threads(N1) * p.tx / 16) : y_threads(N1);
    return launch_pdl(fn, dim3(tiles(p), p.g.nz, 3), dim3(threads), sm, s, p);
}
// Radix split N = N1 x N2 of the two-level passes: split 0 is the default, split 1 the
// alternative the autotuner times against it (open powers of two up to 256).
template <bool INV, bool FULL>
cudaError_t launch_y_dispatch(const ColPass &p, cudaStream_t s) {
    if (!FULL && p.split != 0) switch (p.g.py) {
            case 16: return launch_y_fused<8, 2, INV, false>(p, s);
            case 32: return launch_y_fused<4, 8, INV, false>(p, s);
            case 64: return launch_y_fused<16, 4, INV, false>(p, s);
            case 128: return launch_y_fused<32, 4, INV, false>(p, s);
            case 256: return launch_y_fused<32, 8, INV, false>(p, s);
        }
#define FM_CASE(n) \
    case n: return launch_y_fused<split_line(n), n / split_line(n), INV, FULL>(p, s);
    switch (p.g.py) { FM_LENGTHS_TO_256(FM_CASE) FM_LENGTHS_LONG(FM_CASE) }
#undef FM_CASE
    return cudaErrorInvalidValue;
}
}  // namespace

size_t y_pass_smem(const Grid &g, int tx) {
    const size_t one = sizeof(float2) * (size_t)tx * skewed_len(g.py);
    return y_fused_ok(g) ? one : 2 * one;
}

cudaError_t launch_y_forward(const ColPass &p, cudaStream_t s) {
    if (y_fused_ok(p.g)) return (p.g.per & 2) ? launch_y_dispatch<false, true>(p, s) : launch_y_dispatch<false, false>(p, s);
    const size_t sm = 2 * sizeof(float2) * (size_t)p.tx * skewed_len(p.g.py);
    cudaError_t e = ensure_smem((const void *)y_forward_kernel, sm);
    if (e != cudaSuccess) return e;
    return launch_pdl(y_forward_kernel, dim3(tiles(p), p.g.nz, 3), dim3(kThreads), sm, s, p);
}

cudaError_t launch_y_inverse(const ColPass &p, cudaStream_t s) {
    if (y_fused_ok(p.g)) return (p.g.per & 2) ? launch_y_dispatch<true, true>(p, s) : launch_y_dispatch<true, false>(p, s);
    const size_t sm = 2 * sizeof(float2) * (size_t)p.tx * skewed_len(p.g.py);
    const auto fn = long_butterflies(p.plan) ? y_inverse_kernel<true> : y_inverse_kernel<false>;
    cudaError_t e = ensure_smem((const void *)fn, sm);
    if (e != cudaSuccess) return e;
    return launch_pdl(fn, dim3(tiles(p), p.g.nz, 3), dim3(kThreads), sm, s, p);
}

cudaError_t load_finalize_stats() {
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, (const void *)finalize_stats_kernel);
}

cudaError_t launch_finalize_stats(const float2 *partials, int nblocks, double *out, cudaStream_t s, int early) {
    return launch_pdl(finalize_stats_kernel, dim3(1), dim3(kFinThreads), 0, s, partials, nblocks, out, early);
}

cudaError_t launch_finalize_batched(const FinDesc *fd, int nproblems, double *out, cudaStream_t s) {
    finalize_batched_kernel<<<nproblems, kFinThreads, 0, s>>>(fd, out);
    return cudaGetLastError();
}

namespace {
// [c][kz][ky][kx] -> [c][kz][kx][ky]; one launch at setup
__global__ void kern_ky_fast_kernel(const float *__restrict__ in, float *__restrict__ out, long long planes, int nky,
                                    int nkx) {
    const long long per = (long long)nky * nkx;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < planes * per; i += (long long)gridDim.x * blockDim.x) {
        const long long pl = i / per;
        const int r = (int)(i - pl * per), ky = r / nkx, kx = r - ky * nkx;
        out[pl * per + (long long)kx * nky + ky] = in[i];
    }
}
}  // namespace

cudaError_t launch_kern_ky_fast(const float *in, float *out, int ncomp, int nkz, int nky, int nkx, cudaStream_t s) {
    const long long total = (long long)ncomp * nkz * nky * nkx;
    const int blocks = (int)std::min<long long>((total + 255) / 256, 4096);
    kern_ky_fast_kernel<<<blocks, 256, 0, s>>>(in, out, (long long)ncomp * nkz, nky, nkx);
    return cudaGetLastError();
}

}  // namespace fm
