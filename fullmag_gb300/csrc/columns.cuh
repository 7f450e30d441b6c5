// columns.cuh -- what the column passes (columns.cu, columns_z.cu, columns_conv.cuh) share:
// the demag multiply with the octant or the periodic kernel, and the kx tiling.
//
// Reference behaviour restated (paths in mzrptu/fullmag):
//   tensor multiply H(k) = -N(k) M(k)          native/backends/fdm/src/demag_fp32.cu:138-164
//                                              crates/fullmag-engine/src/fdm_fields.rs:560-588
// The open-boundary kernel is real and octant-unique (6 floats per octant frequency), the
// multiply sits between the forward and inverse z (3-D) or y (thin film) transforms of one
// CTA.
#pragma once
#include <algorithm>

#include "engine.h"
#include "fft_pair.cuh"

namespace fm {

namespace {

constexpr int kThreads = 256;
constexpr size_t kMaxSmem = 227 * 1024;  // shared memory of an SM that CTAs can have

__device__ __forceinline__ void kernel_mirror(int k, int p, int &km, float &sg) {
    if (k > p / 2) {
        km = p - k;
        sg = -1.f;
    } else {
        km = k;
        sg = 1.f;
    }
}

// H = -K M with the complex kernel of a periodic grid: K points at component xx of one
// frequency, the other components follow at stride kc (xx yy zz xy xz yz; 2-D: the
// first four, xz = yz = 0).
__device__ __forceinline__ float2 cmadd(float2 k, float2 m, float2 acc) {
    return make_float2(acc.x + k.x * m.x - k.y * m.y, acc.y + k.x * m.y + k.y * m.x);
}
__device__ __forceinline__ void multiply_periodic(const float2 *K, size_t kc, bool thin, float2 *lx, float2 *ly,
                                                  float2 *lz) {
    const float2 kxx = __ldg(K), kyy = __ldg(K + kc), kzz = __ldg(K + 2 * kc), kxy = __ldg(K + 3 * kc);
    const float2 z0 = make_float2(0.f, 0.f);
    const float2 kxz = thin ? z0 : __ldg(K + 4 * kc), kyz = thin ? z0 : __ldg(K + 5 * kc);
    const float2 mx = *lx, my = *ly, mz = *lz;
    const float2 hx = cmadd(kxz, mz, cmadd(kxy, my, cmadd(kxx, mx, z0)));
    const float2 hy = cmadd(kyz, mz, cmadd(kyy, my, cmadd(kxy, mx, z0)));
    const float2 hz = cmadd(kzz, mz, cmadd(kyz, my, cmadd(kxz, mx, z0)));
    *lx = make_float2(-hx.x, -hx.y);
    *ly = make_float2(-hy.x, -hy.y);
    *lz = make_float2(-hz.x, -hz.y);
}

// Work item `it` of a kx tile -> (row, col), col fastest over the tile's ncol live
// columns.  nkx = px/2 + 1 is odd, so the last tile of a grid usually holds one live
// column; iterating rows * ncol items (not rows * tx) lets it skip the padding columns
// instead of computing them.  Only the last tile can be partial, so the divider is
// either the tile width's or the last tile's (fd_last, precomputed on the host).
// Shared-memory lines stay indexed by col within tx.
__device__ __forceinline__ void tile_item(const ColPass &p, int ncol, int it, int &row, int &col) {
    const FastDiv &fd = ncol == p.tx ? p.fd_tx : p.fd_last;
    row = fd.div(it);
    col = it - row * ncol;
}

// Number of y-frequencies a CTA handles: ky and py - ky (1 for ky = 0 and the Nyquist row).
__device__ __forceinline__ int ky_pair(int kya, int py, int &kyb) {
    kyb = py - kya;
    return (kya == 0 || kyb == kya) ? 1 : 2;
}


inline cudaError_t ensure_smem(const void *fn, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

inline unsigned tiles(const ColPass &p) { return (unsigned)((p.g.nkx + p.tx - 1) / p.tx); }

// z convolution of one (kx, ky) column in registers, pz = PZ <= 24 with 2 nz <= PZ: the nz
// physical values of the three components in v (zero from nz on), forward DFT from half
// lines (even and odd outputs as PZ/2-point DFTs of v and of v W^n), -N(k) multiply,
// inverse, back in v.  K points at component xx of frequency kz = 0 of the column; zs is
// the kz stride, kc the component stride, sy the sign of the odd-in-y components (open
// boundaries); PER: the complex kernel, all kz.  tw: e^{-2 pi i n / PZ}.
template <int PZ, bool PER>
__device__ __forceinline__ void z_column_convolve(float2 (&v)[3][PZ / 2], const float *__restrict__ kern, size_t zs,
                                                  size_t kc, float sy, const float2 *__restrict__ tw) {
    constexpr int H = PZ / 2;
    float2 o[3][H];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        o[c][0] = v[c][0];
#pragma unroll
        for (int n = 1; n < H; ++n) o[c][n] = cmul(v[c][n], __ldg(tw + n));
        dft_small<H>(v[c], false);
        dft_small<H>(o[c], false);
    }
#pragma unroll
    for (int kz = 0; kz < PZ; ++kz) {
        float2 &x = (kz & 1) ? o[0][kz / 2] : v[0][kz / 2];
        float2 &y = (kz & 1) ? o[1][kz / 2] : v[1][kz / 2];
        float2 &z = (kz & 1) ? o[2][kz / 2] : v[2][kz / 2];
        if constexpr (PER) {
            multiply_periodic(reinterpret_cast<const float2 *>(kern) + kz * zs, kc, false, &x, &y, &z);
        } else {
            const float sz = kz > H ? -1.f : 1.f;
            const float *K = kern + (kz > H ? PZ - kz : kz) * zs;
            const float kxx = __ldg(K), kyy = __ldg(K + kc), kzz = __ldg(K + 2 * kc);
            const float kxy = sy * __ldg(K + 3 * kc), kxz = sz * __ldg(K + 4 * kc), kyz = sy * sz * __ldg(K + 5 * kc);
            const float2 mx = x, my = y, mz = z;
            x = make_float2(-(kxx * mx.x + kxy * my.x + kxz * mz.x), -(kxx * mx.y + kxy * my.y + kxz * mz.y));
            y = make_float2(-(kxy * mx.x + kyy * my.x + kyz * mz.x), -(kxy * mx.y + kyy * my.y + kyz * mz.y));
            z = make_float2(-(kxz * mx.x + kyz * my.x + kzz * mz.x), -(kxz * mx.y + kyz * my.y + kzz * mz.y));
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        dft_small<H>(v[c], true);
        dft_small<H>(o[c], true);
#pragma unroll
        for (int n = 0; n < H; ++n) v[c][n] = cadd(v[c][n], n ? cmul(o[c][n], cconj(__ldg(tw + n))) : o[c][n]);
    }
}
__host__ __device__ constexpr bool z_register_length(int pz) {
    return (pz % 2 == 0 && pz >= 2 && pz <= 16) || pz == 20 || pz == 24;
}

}  // namespace

}  // namespace fm
