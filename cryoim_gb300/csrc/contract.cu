// contract.cu — the projection-matching contraction form of the global search.
//
// Score: for particle p, origin s and orientation R,
//     CC(p, s, R) = Re sum_h  A_ps(h) conj(B_R(h)) / (|A_p| |B_R|)
// over the half-plane band samples h (minR <= |h| <= maxR), with
//     A_ps(h) = CTF_p(h) P_p(h) exp(2 pi i h.(s + nx/2)/nx)     (the particle, its CTF and
//               the origin shift of img2d_FT_centshift.f90, so the reference's CTF
//               multiply and origin ramps sit on the particle side of the product)
//     B_R(h)  = M(R (hx, ky, 0))                                (trilinear central section
//               of the centred 3D Fourier map, project2d_FT3dTo2d.f90:30-83)
// Stacking (Re, Im) along K turns it into one real contraction
//     C[(p,s), R] = sum_k A[(p,s), k] B[R, k],   K = 2 x samples,
// which gemm_tc.cu runs on the tensor cores in BF16 or e4m3 with FP32 accumulation.  The local form
// contracts it so, a row of A per origin.  The global forms' rows of A are the particle under a
// basis of its origin grid (origin_basis.h), whose products the k_up_* kernels here expand to all
// origins in FP32, and where the grid's omegas pair up half a turn apart B holds the first of each
// pair: the two halves of K are contracted apart and summed or subtracted.  The normalisation sums
// are FP64; the best candidates are rescored in FP64 here and with the reference's phase residual
// by the driver.
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "geom.cuh"
#include "reduce.cuh"
#include "kernels.h"
#include "launch.h"
#include "origin_basis.h"

namespace cryoim {
namespace {

__device__ double block_sum_double(double v, double* sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    double r = 0;
    if (threadIdx.x < 32) {
        r = (l < nw) ? sh[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        if (l == 0) sh[0] = r;
    }
    __syncthreads();
    r = sh[0];
    __syncthreads();
    return r;
}

// 1 / sqrt of the block's FP64 sum of part (0 for 0); the root and the quotient by one thread: FP64
// work of every warp would take longer than a row's samples
__device__ float block_inv_norm(float part, double* sh) {
    __shared__ float inv;
    const double nrm = block_sum_double((double)part, sh);
    if (threadIdx.x == 0) inv = nrm > 0.0 ? (float)(1.0 / sqrt(nrm)) : 0.0f;
    __syncthreads();
    return inv;
}

// map * (-1)^(x+y+z) as complex, so the forward FFT is centred at nx/2
__global__ void k_map_checker(const float* __restrict__ map, int nx, float2* __restrict__ out) {
    const long n3 = (long)nx * nx * nx;
    for (long q = (long)blockIdx.x * blockDim.x + threadIdx.x; q < n3; q += (long)gridDim.x * blockDim.x) {
        int x = (int)(q % nx), y = (int)((q / nx) % nx), z = (int)(q / ((long)nx * nx));
        float v = map[q];
        out[q] = make_float2(((x + y + z) & 1) ? -v : v, 0.0f);
    }
}

// Band cube of the transform: frequencies -(R+1) .. R+1 per axis, phase referenced to
// the map centre ((-1)^(kx+ky+kz)), standard complex convention, scaled by 1/nx^3.
__global__ void k_map_band(const float2* __restrict__ ft, int nx, int R, float2* __restrict__ cube) {
    const int C = 2 * R + 3;
    const long total = (long)C * C * C;
    const float s = 1.0f / ((float)nx * (float)nx * (float)nx);
    for (long q = (long)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (long)gridDim.x * blockDim.x) {
        int x = (int)(q % C), y = (int)((q / C) % C), z = (int)(q / ((long)C * C));
        int kx = x - (R + 1), ky = y - (R + 1), kz = z - (R + 1);
        float2 v = ft[((long)freq_index(kz, nx) * nx + freq_index(ky, nx)) * nx + freq_index(kx, nx)];
        float sg = ((kx + ky + kz) & 1) ? -s : s;
        cube[q] = make_float2(v.x * sg, v.y * sg);
    }
}

// Gaussian-kernel interpolation of the band cube (C^3 float2, frequency k at index
// k + off): the 3 x 3 x 3 voxels around the nearest one to (x, y, z), each weighted by
// exp(-d^2 / (2 sigma^2)) (gk = 1 / (2 sigma^2); the weight is separable in x, y, z),
// normalised by the weights' sum.  |(x, y, z)| <= maxR keeps every tap inside the cube.
__device__ __forceinline__ float2 gauss_sample(const float2* __restrict__ cube, int C, int off, float x, float y,
                                               float z, float gk) {
    const float rx = rintf(x), ry = rintf(y), rz = rintf(z);
    float wx[3], wy[3], wz[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float ex = x - (rx + (float)(d - 1)), ey = y - (ry + (float)(d - 1)), ez = z - (rz + (float)(d - 1));
        wx[d] = expf(-gk * ex * ex);
        wy[d] = expf(-gk * ey * ey);
        wz[d] = expf(-gk * ez * ez);
    }
    const float2* b = cube + ((long)((int)rz + off - 1) * C + ((int)ry + off - 1)) * C + ((int)rx + off - 1);
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int dz = 0; dz < 3; ++dz)
#pragma unroll
        for (int dy = 0; dy < 3; ++dy) {
            const float2* r = b + ((long)dz * C + dy) * C;
            const float w = wz[dz] * wy[dy];
            const float2 v0 = r[0], v1 = r[1], v2 = r[2];
            acc.x += w * (wx[0] * v0.x + wx[1] * v1.x + wx[2] * v2.x);
            acc.y += w * (wx[0] * v0.y + wx[1] * v1.y + wx[2] * v2.y);
        }
    const float inv = 1.0f / ((wx[0] + wx[1] + wx[2]) * (wy[0] + wy[1] + wy[2]) * (wz[0] + wz[1] + wz[2]));
    return make_float2(acc.x * inv, acc.y * inv);
}

// Section rows are stored pre-swizzled: within each 128-byte block of K, the 16-byte
// chunk c of row r sits at chunk c ^ (r & 7), the order in which a TMA load with the
// 128-byte swizzle would place it in shared memory.  A row copied verbatim into a tile
// row of the same residue mod 8 (a TMA box without swizzle) is then already in the
// layout the tensor cores read; a row copied by index into any tile row has its chunks
// re-ordered by the XOR of the two residues (gemm_tc.cu, B rows by index).  Index of
// (Re, Im) pair i of a local grid's row r (interleaved pairs, 32 per block, 4 per chunk):
__device__ __forceinline__ long bf16_pair_at(long i, long r) {
    return (i & ~31L) | ((((i >> 2) & 7) ^ (r & 7)) << 2) | (i & 3);
}


// The section banks keep the parts of a row apart: elements [0, KH) are the real parts of
// the samples, [KH, 2 KH) the imaginary parts (KH = S rounded up to a 128-byte block), so
// that the products over each half of K come out separately (k_up_* below).  Index of
// element e (of 2 KH) of row r, pre-swizzled as above: BF16 64 elements per block, FP8 128.
__device__ __forceinline__ long bf16_at(long e, long r) {
    return (e & ~63L) | ((((e >> 3) & 7) ^ (r & 7)) << 3) | (e & 7);
}
__device__ __forceinline__ long fp8_at(long e, long r) {
    return (e & ~127L) | ((((e >> 4) & 7) ^ (r & 7)) << 4) | (e & 15);
}

// One CTA per bank row r = view * nomr + iomega (nomr omegas of each view: all of them, or
// the first half turn, the others being complex conjugates): section samples in shared
// memory, norm (FP32 per thread, FP64 across the block), then the unit-norm row in BF16
// (split, zero pad).  The trilinear interpolation runs on the texture
// units: the band cube is a float2 3D array with linear filtering (hardware weights in
// 1/256 steps, well inside the BF16 rounding of the row), texel centres at +0.5, zero
// outside the cube.
__global__ void __launch_bounds__(512) k_slice_bf16(cudaTextureObject_t cube, int R,
                                                    const int2* __restrict__ samples, int S, int KH,
                                                    const float* __restrict__ views, int nomr, float step,
                                                    float d2r, long n0, __nv_bfloat16* __restrict__ B,
                                                    const float2* __restrict__ lin, float gk, float sc) {
    extern __shared__ float2 ssec[];
    __shared__ double sh[32];
    __shared__ float rot[9];
    const long n = n0 + blockIdx.x;
    const int v = (int)(n / nomr), io = (int)(n % nomr);
    if (threadIdx.x == 0) {
        euler_mat(views[2 * v], views[2 * v + 1], step * (float)io, d2r, rot);
        for (int i = 0; i < 9; ++i) rot[i] *= sc;  // cube voxels per frequency unit
    }
    __syncthreads();
    const float off = (float)(R + 1) + 0.5f;
    float part = 0.0f;
    // four samples per step: their fetches are independent and in flight together
#pragma unroll 4
    for (int i = threadIdx.x; i < S; i += blockDim.x) {
        const int2 hk = samples[i];
        const float hx = (float)hk.x, ky = (float)hk.y;
        const float x = rot[0] * hx + rot[1] * ky, y = rot[3] * hx + rot[4] * ky, z = rot[6] * hx + rot[7] * ky;
        const float2 val = gk > 0.0f ? gauss_sample(lin, 2 * R + 3, R + 1, x, y, z, gk)
                                     : tex3D<float2>(cube, x + off, y + off, z + off);
        ssec[i] = val;
        part += val.x * val.x + val.y * val.y;
    }
    const float inv = block_inv_norm(part, sh);
    __nv_bfloat16* row = B + (long)blockIdx.x * (2 * KH);
    for (int i = 2 * threadIdx.x; i < KH; i += 2 * blockDim.x) {
        const float2 a = i < S ? ssec[i] : make_float2(0.f, 0.f);
        const float2 c = i + 1 < S ? ssec[i + 1] : make_float2(0.f, 0.f);
        *reinterpret_cast<__nv_bfloat162*>(row + bf16_at(i, n)) = __floats2bfloat162_rn(a.x * inv, c.x * inv);
        *reinterpret_cast<__nv_bfloat162*>(row + bf16_at(KH + i, n)) = __floats2bfloat162_rn(a.y * inv, c.y * inv);
    }
}

// Local grids: one CTA per (particle p, grid point l) with l = (i * n + j) * n + k,
// n = 2 m + 1, orientation (theta_p + (i - m) s, phi_p + (j - m) s, omega_p + (k - m) s)
// from centre[3 p ..]; particle p's rows start at row p * lpitch (lpitch >= n^3); the
// row is interpolated and normalised as k_slice_bf16 does it, in (Re, Im) pairs.
// With pctf (the CTF of each particle at each sample), a row is normalised by |CTF S|
// instead of |S|: the particle's own grid, so the contraction's score is the unbiased
// projection-matching correlation sum Re(P conj(CTF S)) / (|P| |CTF S|) (with A rows
// normalised by |P|), whose maximum lies at the particle's orientation.  Normalising by
// |S| (a section shared by every particle, as in the global bank) moves the maximum by
// a fraction of a degree on whole particles and by degrees on the local maps' sections.
__global__ void __launch_bounds__(512) k_slice_bf16_local(cudaTextureObject_t cube, int R,
                                                          const int2* __restrict__ samples, int S, int Kpad,
                                                          const float* __restrict__ centre, int m, float step,
                                                          float d2r, long n0, __nv_bfloat162* __restrict__ B,
                                                          const float2* __restrict__ lin, float gk, long lpitch,
                                                          const float* __restrict__ pctf, float sc) {
    extern __shared__ float2 ssec[];
    __shared__ double sh[32];
    __shared__ float rot[9];
    const int n = 2 * m + 1;
    const long nloc = (long)n * n * n;
    const long q = n0 + blockIdx.x;
    const int p = (int)(q / lpitch), l = (int)(q % lpitch);
    if (l >= nloc) return;  // padding row between particles' grids (never a valid column)
    const int i = l / (n * n), j = (l / n) % n, k = l % n;
    if (threadIdx.x == 0) {
        euler_mat(centre[3 * p] + step * (float)(i - m), centre[3 * p + 1] + step * (float)(j - m),
                  centre[3 * p + 2] + step * (float)(k - m), d2r, rot);
        for (int e = 0; e < 9; ++e) rot[e] *= sc;  // cube voxels per frequency unit
    }
    __syncthreads();
    const float off = (float)(R + 1) + 0.5f;
    float part = 0.0f;
#pragma unroll 4
    for (int t = threadIdx.x; t < S; t += blockDim.x) {
        const int2 hk = samples[t];
        const float hx = (float)hk.x, ky = (float)hk.y;
        const float x = rot[0] * hx + rot[1] * ky, y = rot[3] * hx + rot[4] * ky, z = rot[6] * hx + rot[7] * ky;
        const float2 val = gk > 0.0f ? gauss_sample(lin, 2 * R + 3, R + 1, x, y, z, gk)
                                     : tex3D<float2>(cube, x + off, y + off, z + off);
        ssec[t] = val;
        const float cw = pctf ? pctf[(long)p * S + t] : 1.0f;
        part += cw * cw * (val.x * val.x + val.y * val.y);
    }
    const float inv = block_inv_norm(part, sh);
    __nv_bfloat162* row = B + (long)blockIdx.x * (Kpad / 2);
    for (int t = threadIdx.x; t < Kpad / 2; t += blockDim.x) {
        float2 val = t < S ? ssec[t] : make_float2(0.f, 0.f);
        row[bf16_pair_at(t, q)] = __floats2bfloat162_rn(val.x * inv, val.y * inv);
    }
}

// The same rows, one CTA per (particle p, i, j) cutting the n rows k = 0 .. n - 1 (the
// omega steps) LSR_ROWS at a time: a thread holds its SPT samples (h, k, CTF^2) in registers
// across the rows and the rows' values in registers until their norms are known, so the CTA needs
// no shared-memory row and the SM's L1 stays large for the texture fetches, which
// neighbouring omegas share (0.25 degrees moves a sample by a fraction of a voxel).
// Each row's values, norm and BF16 row are k_slice_bf16_local's; the norm's FP32
// per-thread partials cover fewer samples (it agrees to FP32 rounding).
// Bound: the texture pipe (60 % busy, FP64 16 %).  With a row at a time, every warp summing in five
// FP64 steps and taking the root and the quotient for itself, the FP64 pipe was 70 % busy and
// the 15,625 rows of each of 24 particles (25 steps a side, 1,600
// samples a row) took 6.27 ms; now 3.66.  Two rows at a time 3.8 to 3.9, one 4.4, 512 threads 4.1.
constexpr int LSR_THREADS = 256, LSR_SPT = 8;  // rows of up to 2,048 samples (pairs)
constexpr int LSR_ROWS = 4;
template <int SPT>
__global__ void __launch_bounds__(LSR_THREADS, 2) k_slice_bf16_local_rows(
    cudaTextureObject_t cube, int R, const int2* __restrict__ samples, int S, int Kpad,
    const float* __restrict__ centre, int m, float step, float d2r, __nv_bfloat162* __restrict__ B,
    const float2* __restrict__ lin, float gk, long lpitch, const float* __restrict__ pctf, float sc) {
    extern __shared__ float rots[];  // [n][9]
    __shared__ double wsum[LSR_ROWS][LSR_THREADS / 32];
    __shared__ float sinv[LSR_ROWS];
    const int n = 2 * m + 1;
    const int p = blockIdx.y, ij = blockIdx.x;
    const int i = ij / n, j = ij % n;
    for (int k = threadIdx.x; k < n; k += LSR_THREADS) {
        float* rot = rots + 9 * k;
        euler_mat(centre[3 * p] + step * (float)(i - m), centre[3 * p + 1] + step * (float)(j - m),
                  centre[3 * p + 2] + step * (float)(k - m), d2r, rot);
        for (int e = 0; e < 9; ++e) rot[e] *= sc;  // cube voxels per frequency unit
    }
    float hx[SPT], ky[SPT], cw2[SPT];
#pragma unroll
    for (int s = 0; s < SPT; ++s) {
        const int t = threadIdx.x + s * LSR_THREADS;
        hx[s] = 0.0f;
        ky[s] = 0.0f;
        cw2[s] = 0.0f;
        if (t < S) {
            const int2 hk = samples[t];
            hx[s] = (float)hk.x;
            ky[s] = (float)hk.y;
            const float cw = pctf ? pctf[(long)p * S + t] : 1.0f;
            cw2[s] = cw * cw;
        }
    }
    __syncthreads();
    const float off = (float)(R + 1) + 0.5f;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int k0 = 0; k0 < n; k0 += LSR_ROWS) {
        float2 val[LSR_ROWS][SPT];
        double sums[LSR_ROWS];
#pragma unroll
        for (int q = 0; q < LSR_ROWS; ++q) {
            const float* rot = rots + 9 * min(k0 + q, n - 1);  // a row beyond the last is not written
            const float r0 = rot[0], r1 = rot[1], r3 = rot[3], r4 = rot[4], r6 = rot[6], r7 = rot[7];
            float part = 0.0f;
#pragma unroll
            for (int s = 0; s < SPT; ++s) {
                val[q][s] = make_float2(0.f, 0.f);
                if (threadIdx.x + s * LSR_THREADS < S && k0 + q < n) {
                    const float x = r0 * hx[s] + r1 * ky[s], y = r3 * hx[s] + r4 * ky[s], z = r6 * hx[s] + r7 * ky[s];
                    val[q][s] = gk > 0.0f ? gauss_sample(lin, 2 * R + 3, R + 1, x, y, z, gk)
                                          : tex3D<float2>(cube, x + off, y + off, z + off);
                }
            }
#pragma unroll
            for (int s = 0; s < SPT; ++s)
                if (threadIdx.x + s * LSR_THREADS < S)
                    part += cw2[s] * (val[q][s].x * val[q][s].x + val[q][s].y * val[q][s].y);
            sums[q] = (double)part;
        }
        // norms: FP64 across the block in a fixed order (warps, then the warps' sums)
        warp_sums<LSR_ROWS>(sums, lane);
        if (lane % (32 / LSR_ROWS) == 0) wsum[warp_sum_index<LSR_ROWS>(lane)][wid] = sums[0];
        __syncthreads();
        if (threadIdx.x < LSR_ROWS) {
            double nrm = 0.0;
#pragma unroll
            for (int w = 0; w < LSR_THREADS / 32; ++w) nrm += wsum[threadIdx.x][w];
            sinv[threadIdx.x] = nrm > 0.0 ? (float)(1.0 / sqrt(nrm)) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < LSR_ROWS; ++q) {
            if (k0 + q >= n) break;
            const float inv = sinv[q];
            const long r = (long)p * lpitch + (long)ij * n + k0 + q;
            __nv_bfloat162* row = B + r * (Kpad / 2);
#pragma unroll
            for (int s = 0; s < SPT; ++s) {
                const int t = threadIdx.x + s * LSR_THREADS;
                if (t < Kpad / 2) row[bf16_pair_at(t, r)] = __floats2bfloat162_rn(val[q][s].x * inv, val[q][s].y * inv);
            }
        }
    }
}

// FP64 sum over samples of |CTF * P|^2 per particle (the origin shift keeps it); with
// pc, also the samples CTF * (a, b) themselves in FP64, in sample order.
// With norm0, also the sum of |P|^2 without the CTF; with pctf, the CTF at each sample.
__global__ void k_particle_norm(const float2* __restrict__ band, const float* __restrict__ ctf, Band bd,
                                const int2* __restrict__ samples, int S, double* __restrict__ norm,
                                double2* __restrict__ pc, double* __restrict__ norm0, float* __restrict__ pctf) {
    __shared__ double sh[32];
    const int p = blockIdx.x, W = bd.W, R = bd.max_r;
    const float2* b = band + (long)p * W * W;
    const float* c = ctf ? ctf + (long)p * W * W : nullptr;
    double acc = 0.0, acc0 = 0.0;
    for (int i = threadIdx.x; i < S; i += blockDim.x) {
        const int2 hk = samples[i];
        const int q = (hk.y + R) * W + (hk.x + R);
        const double cv = c ? (double)c[q] : 1.0;
        const double re = b[q].x * cv, im = b[q].y * cv;
        acc += re * re + im * im;
        acc0 += (double)b[q].x * b[q].x + (double)b[q].y * b[q].y;
        if (pc) pc[(long)p * S + i] = make_double2(re, im);
        if (pctf) pctf[(long)p * S + i] = c ? c[q] : 1.0f;
    }
    acc = block_sum_double(acc, sh);
    if (threadIdx.x == 0) norm[p] = acc;
    if (norm0) {
        acc0 = block_sum_double(acc0, sh);
        if (threadIdx.x == 0) norm0[p] = acc0;
    }
}

// The origin phase exp(i 2pi/n (sx hx + sy ky)) of a row of A is separable: a block
// tabulates (cos, sin) of 2pi/n sx hx for hx in [0, R] and of 2pi/n sy ky for ky in
// [-R, R] (3R + 2 entries in shared memory) and multiplies the two per sample.
__device__ __forceinline__ void phasor_at(const float2* tab, int R, int2 hk, float* sn, float* cs) {
    const float2 ex = tab[hk.x], ey = tab[R + 1 + R + hk.y];
    *cs = ex.x * ey.x - ex.y * ey.y;
    *sn = ex.y * ey.x + ex.x * ey.y;
}

// Rows (p, o0 .. o0 + AO - 1) of A: CTF x particle x origin phase ramp, unit norm,
// BF16.  Each thread reads a sample's transform and CTF once and writes it for AO
// origins (phasor tables of all AO origins in shared memory).
constexpr int AO = 8;
__global__ void __launch_bounds__(256) k_build_a(const float2* __restrict__ band, const float* __restrict__ ctf,
                                                 Band bd, const int2* __restrict__ samples, int S, int Kpad,
                                                 const float* __restrict__ origins, int O,
                                                 const float* __restrict__ poff,
                                                 const double* __restrict__ norm, float two_pi_over_n,
                                                 __nv_bfloat162* __restrict__ A) {
    extern __shared__ float2 ptab[];  // [AO][3 R + 2]
    const int o0 = blockIdx.x * AO, p = blockIdx.y, W = bd.W, R = bd.max_r, nt = 3 * R + 2;
    const int no = min(AO, O - o0);
    const float2* b = band + (long)p * W * W;
    const float* c = ctf ? ctf + (long)p * W * W : nullptr;
    // origins relative to the particle's own (poff) or absolute
    const float hx = (float)(bd.nx / 2) + (poff ? poff[2 * p] : 0.0f);
    const float hy = (float)(bd.nx / 2) + (poff ? poff[2 * p + 1] : 0.0f);
    __shared__ float sinv;  // root and quotient once: FP64 by every warp outweighs a block's FP32 work
    if (threadIdx.x == 0) sinv = norm[p] > 0.0 ? (float)(1.0 / sqrt(norm[p])) : 0.0f;
    for (int j = 0; j < no; ++j) {
        const float sx = origins[2 * (o0 + j)] + hx, sy = origins[2 * (o0 + j) + 1] + hy;
        for (int i = threadIdx.x; i < nt; i += blockDim.x) {
            const float a = i <= R ? two_pi_over_n * (sx * (float)i)
                                   : two_pi_over_n * (sy * (float)(i - 2 * R - 1));
            float sn, cs;
            sincosf(a, &sn, &cs);
            ptab[j * nt + i] = make_float2(cs, sn);
        }
    }
    __syncthreads();
    const float inv = sinv;
    for (int i = threadIdx.x; i < Kpad / 2; i += blockDim.x) {
        if (i < S) {
            const int2 hk = samples[i];
            const int q = (hk.y + R) * W + (hk.x + R);
            const float2 ab = b[q];  // (a, b) = (Re F, -Im F) referenced to pixel 0
            const float cv = (c ? c[q] : 1.0f) * inv;
            for (int j = 0; j < no; ++j) {
                float sn, cs;
                phasor_at(ptab + j * nt, R, hk, &sn, &cs);
                // centshift: (a', b') = (a cos + b sin, -a sin + b cos); P = a' - i b'
                const float a2 = ab.x * cs + ab.y * sn, b2 = -ab.x * sn + ab.y * cs;
                A[((long)p * O + o0 + j) * (Kpad / 2) + i] = __floats2bfloat162_rn(a2 * cv, -b2 * cv);
            }
        } else {
            for (int j = 0; j < no; ++j)
                A[((long)p * O + o0 + j) * (Kpad / 2) + i] = __floats2bfloat162_rn(0.f, 0.f);
        }
    }
}

// ---- the origin grid's basis ---------------------------------------------------
// The global forms correlate ob.slots basis rows per particle instead of its origin grid
// (origin_basis.h has the argument), and a half turn of omega instead of the whole: the
// section at omega + 180 degrees is the complex conjugate of the section at omega (the map
// is real), so with u = A_re B_re^T and v = A_im B_im^T, the two halves of K apart, the
// scores are u + v at omega and u - v at omega + 180.  Where omega + 180 is not a grid point
// (an odd number of omegas) the bank holds every omega and K is one piece.
//
// Row b = (m of x, k of y, part) of a particle: P exp(i 2 pi h.(mid + n/2 + off) / n) f_m(hx)
// f_k(ky) i^(m odd + k odd) (the transform of q_m(x) q_k(y), f real by parity), times CTF and
// 1/|CTF P|.  Part 1 holds what rounding part 0 to the operand type left.
// HBM-write-bound: 160 rows x 25.6 KB a particle at box 256 (the origin grid is 625 rows:
// 247 us a 64-particle pass against 82).
constexpr int BO = 8;  // rows per block: a sample's transform, CTF and phase once for eight rows
// PACK: several particles to a block of rows (pack_rows), the rows in use alone.
template <bool F8, bool PACK>
__global__ void __launch_bounds__(256) k_build_basis(const float2* __restrict__ band, const float* __restrict__ ctf,
                                                     Band bd, const int2* __restrict__ samples, int S, int KH,
                                                     OriginDev ob, OriginPack pk, const float* __restrict__ poff,
                                                     const double* __restrict__ norm, const float* __restrict__ mulA,
                                                     const int* __restrict__ fexp, float two_pi_over_n,
                                                     void* __restrict__ Aout) {
    extern __shared__ float2 ptab[];  // [3 R + 2] origin phasors, then per row f_m [R + 1], f_k [2 R + 1]
    const int b0 = blockIdx.x * BO, p = blockIdx.y, W = bd.W, R = bd.max_r, nt = 3 * R + 2, R1 = ob.R;
    const long row0 = pk.at(ob.used, p) + b0;
    const int nrow = ob.used - b0;  // PACK: of this block's
    float* ft = reinterpret_cast<float*>(ptab + nt);
    const float2* b = band + (long)p * W * W;
    const float* c = ctf ? ctf + (long)p * W * W : nullptr;
    const float sx = (float)(bd.nx / 2) + ob.mid + (poff ? poff[2 * p] : 0.0f);
    const float sy = (float)(bd.nx / 2) + ob.mid + (poff ? poff[2 * p + 1] : 0.0f);
    __shared__ float sinv;  // root and quotient once: FP64 by every warp outweighs a block's FP32 work
    if (threadIdx.x == 0) sinv = norm[p] > 0.0 ? (float)(1.0 / sqrt(norm[p])) : 0.0f;
    const float pscale = F8 ? ldexpf(1.0f, fexp[p]) : 1.0f;
    int rot[BO], part[BO];  // rot: quarter turns of i^(...), part: -1 for an empty row
#pragma unroll
    for (int j = 0; j < BO; ++j) {
        const int rw = ob.row[b0 + j];  // (slots is a multiple of BO)
        const int m = rw & 0xfff, k = (rw >> 12) & 0xfff;
        part[j] = rw < 0 ? -1 : (rw >> 24) & 1;
        rot[j] = rw < 0 ? 0 : (m & 1) + (k & 1);
        if (rw >= 0) {  // (the table covers |h| <= ob.R, the samples' band; zero beyond)
            for (int i = threadIdx.x; i <= R; i += blockDim.x)
                ft[j * nt + i] = i <= R1 ? ob.f[(long)m * (2 * R1 + 1) + R1 + i] : 0.0f;
            for (int i = threadIdx.x; i < 2 * R + 1; i += blockDim.x)
                ft[j * nt + R + 1 + i] = abs(i - R) <= R1 ? ob.f[(long)k * (2 * R1 + 1) + R1 + i - R] : 0.0f;
        }
    }
    for (int i = threadIdx.x; i < nt; i += blockDim.x) {
        const float a = i <= R ? two_pi_over_n * (sx * (float)i) : two_pi_over_n * (sy * (float)(i - 2 * R - 1));
        float sn, cs;
        sincosf(a, &sn, &cs);
        ptab[i] = make_float2(cs, sn);
    }
    __syncthreads();
    const float inv = sinv;
    for (int i = 2 * threadIdx.x; i < KH; i += 2 * blockDim.x) {  // two samples a thread
        float2 z[2];
        int2 hk[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            z[u] = make_float2(0.f, 0.f);
            hk[u] = make_int2(0, 0);
            if (i + u < S) {
                hk[u] = samples[i + u];
                const int q = (hk[u].y + R) * W + (hk[u].x + R);
                const float2 ab = b[q];  // (a, b) = (Re F, -Im F) referenced to pixel 0
                const float cv = (c ? c[q] : 1.0f) * inv * (F8 ? mulA[i + u] * pscale : 1.0f);
                float sn, cs;
                phasor_at(ptab, R, hk[u], &sn, &cs);
                // centshift: (a', b') = (a cos + b sin, -a sin + b cos); P = a' - i b'
                z[u] = make_float2((ab.x * cs + ab.y * sn) * cv, (ab.x * sn - ab.y * cs) * cv);
            }
        }
#pragma unroll
        for (int j = 0; j < BO; ++j) {
            float re[2], im[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float fv = part[j] < 0 ? 0.0f : ft[j * nt + hk[u].x] * ft[j * nt + 2 * R + 1 + hk[u].y];
                const float x = z[u].x * fv, y = z[u].y * fv;
                re[u] = rot[j] == 0 ? x : (rot[j] == 1 ? -y : -x);
                im[u] = rot[j] == 0 ? y : (rot[j] == 1 ? x : -y);
            }
            if (PACK && j >= nrow) continue;
            const long row = row0 + j;
            if constexpr (F8) {
                unsigned char* A = (unsigned char*)Aout + row * (2 * KH);
                float2 vr = make_float2(re[0], re[1]), vi = make_float2(im[0], im[1]);
                if (part[j] == 1) {
                    const __half2 hr = __half2(__nv_cvt_fp8x2_to_halfraw2(__nv_cvt_float2_to_fp8x2(vr, __NV_SATFINITE, __NV_E4M3), __NV_E4M3));
                    const __half2 hi = __half2(__nv_cvt_fp8x2_to_halfraw2(__nv_cvt_float2_to_fp8x2(vi, __NV_SATFINITE, __NV_E4M3), __NV_E4M3));
                    vr = make_float2((vr.x - __low2float(hr)) * 16.0f, (vr.y - __high2float(hr)) * 16.0f);
                    vi = make_float2((vi.x - __low2float(hi)) * 16.0f, (vi.y - __high2float(hi)) * 16.0f);
                }
                *reinterpret_cast<unsigned short*>(A + i) = __nv_cvt_float2_to_fp8x2(vr, __NV_SATFINITE, __NV_E4M3);
                *reinterpret_cast<unsigned short*>(A + KH + i) = __nv_cvt_float2_to_fp8x2(vi, __NV_SATFINITE, __NV_E4M3);
            } else {
                __nv_bfloat16* A = (__nv_bfloat16*)Aout + row * (2 * KH);
                __nv_bfloat162 vr = __floats2bfloat162_rn(re[0], re[1]), vi = __floats2bfloat162_rn(im[0], im[1]);
                if (part[j] == 1) {
                    vr = __floats2bfloat162_rn(re[0] - __low2float(vr), re[1] - __high2float(vr));
                    vi = __floats2bfloat162_rn(im[0] - __low2float(vi), im[1] - __high2float(vi));
                }
                *reinterpret_cast<__nv_bfloat162*>(A + i) = vr;
                *reinterpret_cast<__nv_bfloat162*>(A + KH + i) = vi;
            }
        }
    }
}

// Expansion of the basis, one orientation per thread: C[o] = sum_mk c_mk q_m(x_o) q_k(y_o)
// in FP32, c_mk the products of the function's rows (u or u +- v).  The functions are even
// (m even) or odd, so a pair of mirror origins costs one pass: per pair of y the sums over
// even and odd k apart give T_m at both, per pair of x the same over m; (even, odd) sums ride
// in packed FP32x2 operations.  In one of origin_basis.h's fixed layouts the c_mk sit in
// registers; more functions (BF16 origin ranges beyond 6 px at maxR n/4, e4m3 beyond 7) lie in
// shared memory (UpAny below).
// emit(N, jy, jx, h[N], l[N]): (even, odd) sums over x at y hi and y lo for the pairs of x
// jx .. jx + N - 1; the value at x hi is their sum, at x lo their difference, where hi =
// n1/2 + j, lo = (n1-1)/2 - j.
constexpr int UP_THREADS = 256, UP_N1 = 1024;
// q at the upper half of the origins, [(n1 + 1) / 2][nb rounded up to even], zero beyond nb
template <int LY> __host__ __device__ inline int up_table_floats(int n1) {
    return (n1 + 1) / 2 * ((OB_LAYOUT[LY].nb + 1) / 2 * 2);
}
template <int LY> __device__ __forceinline__ void up_table(const OriginDev& ob, float* sm) {
    constexpr int NP = (OB_LAYOUT[LY].nb + 1) / 2 * 2;
    for (int i = threadIdx.x; i < up_table_floats<LY>(ob.n1); i += blockDim.x) {
        const int j = i / NP, m = i % NP;
        sm[i] = m < ob.nb ? ob.q[(long)m * ob.n1 + ob.n1 / 2 + j] : 0.0f;
    }
}
template <int LY> struct UpCoef {
    static constexpr int NB = OB_LAYOUT[LY].nb, CUT = OB_LAYOUT[LY].cut, L2 = OB_LAYOUT[LY].second,
                         ROWS = OB_LAYOUT[LY].rows, H = (NB + 1) / 2;
    static __host__ __device__ constexpr bool in(int m, int k) { return m < NB && k < NB && m + k <= CUT; }
    static __host__ __device__ constexpr bool twice(int m, int k) { return in(m, k) && m + k < L2; }
    static __host__ __device__ constexpr bool pair(int m, int k) { return in(m, 2 * k) || in(m, 2 * k + 1); }
    float2 c[2 * H][H];  // (k even, k odd) pairs; zero outside the layout
    // get(i): product of row i; lo: scale of the second rows
    template <class Get> __device__ __forceinline__ void load(float lo, Get get) {
        int b = 0;
#pragma unroll
        for (int m = 0; m < 2 * H; ++m)
#pragma unroll
            for (int k = 0; k < H; ++k) {
                c[m][k] = make_float2(0.f, 0.f);
                if (in(m, 2 * k)) c[m][k].x = get(b++);
                if (in(m, 2 * k + 1)) c[m][k].y = get(b++);
            }
#pragma unroll
        for (int m = 0; m < L2; ++m)
#pragma unroll
            for (int k = 0; k < L2; ++k)
                if (twice(m, k)) {
                    const float v = get(b++);
                    if (k & 1) c[m][k / 2].y = fmaf(v, lo, c[m][k / 2].y);
                    else c[m][k / 2].x = fmaf(v, lo, c[m][k / 2].x);
                }
    }
};
template <int LY, class Emit>
__device__ __forceinline__ void up_eval(const OriginDev& ob, const UpCoef<LY>& cf, const float* sm, Emit emit,
                                        int jy0 = 0, int jy1 = 0x7fffffff) {
    constexpr int H = UpCoef<LY>::H;
    const int hn = (ob.n1 + 1) / 2;
    const float2* q2 = reinterpret_cast<const float2*>(sm);
    for (int jy = jy0; jy < min(hn, jy1); ++jy) {
        float2 qy[H];
#pragma unroll
        for (int k = 0; k < H; ++k) qy[k] = q2[jy * H + k];
        float2 th[H], tl[H];  // (T_2k, T_2k+1) at y hi, y lo
#pragma unroll
        for (int m = 0; m < H; ++m) {
            float2 e = make_float2(0.f, 0.f), o = make_float2(0.f, 0.f);
#pragma unroll
            for (int k = 0; k < H; ++k) {
                if (UpCoef<LY>::pair(2 * m, k)) e = __ffma2_rn(cf.c[2 * m][k], qy[k], e);
                if (UpCoef<LY>::pair(2 * m + 1, k)) o = __ffma2_rn(cf.c[2 * m + 1][k], qy[k], o);
            }
            th[m] = make_float2(e.x + e.y, o.x + o.y);
            tl[m] = make_float2(e.x - e.y, o.x - o.y);
        }
        // pairs of x four (two where the coefficients leave no registers), two, one at a time
        auto pairs = [&](auto nc, int jx) {
            constexpr int N = decltype(nc)::value;
            float2 h[N], l[N];
#pragma unroll
            for (int u = 0; u < N; ++u) { h[u] = make_float2(0.f, 0.f); l[u] = make_float2(0.f, 0.f); }
#pragma unroll
            for (int k = 0; k < H; ++k)
#pragma unroll
                for (int u = 0; u < N; ++u) {
                    const float2 qx = q2[(jx + u) * H + k];
                    h[u] = __ffma2_rn(th[k], qx, h[u]);
                    l[u] = __ffma2_rn(tl[k], qx, l[u]);
                }
            emit(nc, jy, jx, h, l);
        };
        int jx = 0;
        constexpr int N = UpCoef<LY>::ROWS > 128 ? 2 : 4;
        for (; jx + N <= hn; jx += N) pairs(std::integral_constant<int, N>(), jx);
        if (N > 2 && jx + 2 <= hn) { pairs(std::integral_constant<int, 2>(), jx); jx += 2; }
        if (jx < hn) pairs(std::integral_constant<int, 1>(), jx);
    }
}
// product of function (m, k) at the column whose rows start at U, V (the two K shares; V null:
// one share), sgn V's sign
__device__ __forceinline__ float up_coef(const OriginDev& ob, const float* U, const float* V, float sgn, long pitch,
                                         int m, int k) {
    const int2 b = __ldg(ob.slot + (long)m * ob.nb + k);
    float s = 0.0f;
    if (b.x >= 0) {
        s = U[b.x * pitch];
        if (V) s = fmaf(sgn, V[b.x * pitch], s);
    }
    if (b.y >= 0) {
        float c = U[b.y * pitch];
        if (V) c = fmaf(sgn, V[b.y * pitch], c);
        s = fmaf(c, ob.lo, s);
    }
    return s;
}
// Any number of functions.  A warp has 32 columns (a lane each) and a pair of y: for UM_X or UL_X pairs
// of x at a time it goes through the functions m in (even, odd) couples, forms T_m at its y from the
// couple's products and adds T_m q_m(x) to the sums in registers, so that neither T nor the products
// need registers of their own and nothing bounds the number of functions.  The products are combined
// (u +- v, second rows) once for all warps of a block and lie in shared memory four to a 16-byte entry
// (OriginBasis::ent), in chunks of entries where they are too many.  Bound: shared memory, five 128-byte
// reads (an entry of 32 lanes and its q) for each four functions, and the instructions of few warps.
constexpr int UM_X = 16, UM_SHARES = 4, UL_X = 8, UL_THREADS = 256;  // exhaustive, lists
struct UpAny {
    const float4* c;        // the chunk's products: entry e of the chunk of this lane's column at c[e * cols]
    int cols;
    const float4 *qx, *qy;  // OriginBasis::qx, qy
    const int* off;         // [h + 1] entries
    int h;                  // (nb + 1) / 2
};
// q's tables (QSH: into shared memory; else they are read where they are) and the entry offsets, by the
// whole block: qx, qy, offsets from sm
template <bool QSH>
__device__ __forceinline__ UpAny up_any_tables(const OriginDev& ob, unsigned char* sm) {
    const int h = (ob.nb + 1) / 2;
    float4* q = reinterpret_cast<float4*>(sm);
    int* off = reinterpret_cast<int*>(q + (QSH ? ob.nqx + ob.nqy : 0));
    if (QSH) {
        for (int i = threadIdx.x; i < ob.nqx; i += blockDim.x) q[i] = ob.qx[i];
        for (int i = threadIdx.x; i < ob.nqy; i += blockDim.x) q[ob.nqx + i] = ob.qy[i];
    }
    for (int i = threadIdx.x; i <= h; i += blockDim.x) off[i] = ob.ent_off[i];
    return UpAny{nullptr, 0, QSH ? q : ob.qx, QSH ? q + ob.nqx : ob.qy, off, h};
}
// shared memory of the tables, a multiple of 16 bytes
__host__ __device__ inline size_t up_any_table_bytes(const OriginDev& ob, bool qsh) {
    const int h = (ob.nb + 1) / 2;
    return (qsh ? sizeof(float4) * (ob.nqx + ob.nqy) : 0) + (sizeof(int) * (h + 1) + 15) / 16 * 16;
}
// The rows of entry i: part 0, part 1 of its four functions.
__device__ __forceinline__ void up_any_rows(const OriginDev& ob, int i, int (&rows)[8]) {
    const int4 a = __ldg(ob.ent + 2 * i), b = __ldg(ob.ent + 2 * i + 1);
    rows[0] = a.x, rows[1] = a.y, rows[2] = a.z, rows[3] = a.w;
    rows[4] = b.x, rows[5] = b.y, rows[6] = b.z, rows[7] = b.w;
}
// the four functions' products of one sign of v
__device__ __forceinline__ float4 up_any_four(const float* u, const float* v, float sgn, float lo) {
    float c[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = fmaf(fmaf(sgn, v[2 * k + 1], u[2 * k + 1]), lo, fmaf(sgn, v[2 * k], u[2 * k]));
    return make_float4(c[0], c[1], c[2], c[3]);
}
// adds the chunk e0 .. e1 (even) to the sums of the pair of y jy over the N pairs of x from x0 (up to UM_X
// beyond the last: zeros): (even, odd) sums h, l at y hi, lo
template <int N>
__device__ __forceinline__ void up_any_add(const UpAny& A, int e0, int e1, int jy, int x0, float2 (&h)[N], float2 (&l)[N]) {
    const float4* qy = A.qy + jy * ((A.h + 1) / 2);
    for (int a = 0; a < A.h; ++a) {
        const int o = A.off[a], i0 = max(o, e0), i1 = min(A.off[a + 1], e1);
        if (i0 >= i1) continue;
        float2 e[2], d[2];  // (sums over even k, over odd k) of functions 2a and 2a + 1, of every other entry
        e[0] = e[1] = d[0] = d[1] = make_float2(0.f, 0.f);
        const float4* c = A.c + (i0 - e0) * A.cols;
        const float4* q = qy + (i0 - o) / 2;
#pragma unroll 2
        for (int i = i0; i < i1; i += 2, c += 2 * A.cols, ++q) {
            const float4 c0 = c[0], c1 = c[A.cols], v = *q;
            e[0] = __ffma2_rn(make_float2(c0.x, c0.y), make_float2(v.x, v.y), e[0]);
            d[0] = __ffma2_rn(make_float2(c0.z, c0.w), make_float2(v.x, v.y), d[0]);
            e[1] = __ffma2_rn(make_float2(c1.x, c1.y), make_float2(v.z, v.w), e[1]);
            d[1] = __ffma2_rn(make_float2(c1.z, c1.w), make_float2(v.z, v.w), d[1]);
        }
        e[0] = __fadd2_rn(e[0], e[1]);
        d[0] = __fadd2_rn(d[0], d[1]);
        const float2 th = make_float2(e[0].x + e[0].y, d[0].x + d[0].y), tl = make_float2(e[0].x - e[0].y, d[0].x - d[0].y);
        const float4* qx = A.qx + x0 / 2 * A.h + a;
#pragma unroll
        for (int u = 0; u < N; u += 2) {
            const float4 v = qx[u / 2 * A.h];
            h[u] = __ffma2_rn(th, make_float2(v.x, v.y), h[u]);
            l[u] = __ffma2_rn(tl, make_float2(v.x, v.y), l[u]);
            h[u + 1] = __ffma2_rn(th, make_float2(v.z, v.w), h[u + 1]);
            l[u + 1] = __ffma2_rn(tl, make_float2(v.z, v.w), l[u + 1]);
        }
    }
}

// Best origin's value of every orientation of every particle.  Persistent blocks of 256
// threads, one per SM; a tile is 128 bank rows, whose products (up to 160 rows of A x two K
// shares = 160 KB) the block copies into shared memory with 16-byte cp.async, threads 0-127
// taking the bank rows' omegas and threads 128-255 the ones half a turn on (one K share: 256
// bank rows, a thread each).  Once the products are in registers the next tile's copies are
// issued and land under the expansion.  FP32-issue-bound.  Measured at 625 origins and 2 x
// 119,520 orientations: 87 us a particle; 480 us with each function's row looked up and
// fetched by its thread (the loads' latency exposed), 118 us without the prefetch.
// blocks an SM: what the coefficients' registers leave (one where there are 96 of them and more)
constexpr int up_blocks(int ly) { return OB_LAYOUT[ly].rows <= 18 ? 4 : OB_LAYOUT[ly].rows < 96 ? 2 : 1; }
template <int LY>
__global__ void __launch_bounds__(UP_THREADS, up_blocks(LY)) k_up_max(OriginDev ob, OriginPack pk,
                                                                     const float* __restrict__ C, long pitch, long rows,
                                                                     int nom, int nomr, int B,
                                                                     float* __restrict__ ccmax) {
    constexpr int ROWS = OB_LAYOUT[LY].rows;
    extern __shared__ __align__(16) float smem[];  // [share][row of A][columns], then the table of q
    float* sq = smem + UP_THREADS * ROWS;
    up_table<LY>(ob, sq);
    const bool two = nom != nomr;
    const int cols = two ? UP_THREADS / 2 : UP_THREADS;  // bank rows of a tile
    const int ch = cols / 4;                             // 16-byte chunks of a row of a tile
    const long ntile = (rows + cols - 1) / cols, total = ntile * B;
    auto fetch = [&](long t) {
        const long p = t / ntile, r0 = (t - p * ntile) * cols;
        const float* src = C + pk.at_c(ROWS, (int)p, two ? 2 : 1) * pitch + r0;
        const int n = UP_THREADS * ROWS / 4;
        for (int i = threadIdx.x; i < n; i += UP_THREADS) {
            const int row = i / ch, c = i - row * ch;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem + 4 * i);
            const long at = row < ROWS ? row : row - ROWS + pk.rows;  // (the second share's)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + at * pitch + 4 * c) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    long t = blockIdx.x;
    if (t < total) fetch(t);
    const int cl = two ? threadIdx.x & (UP_THREADS / 2 - 1) : threadIdx.x, half = two ? threadIdx.x / (UP_THREADS / 2) : 0;
    const float sgn = half ? -1.0f : 1.0f;
    for (; t < total; t += gridDim.x) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        UpCoef<LY> c;
        if (two)
            c.load(ob.lo, [&](int i) { return fmaf(sgn, smem[(ROWS + i) * (UP_THREADS / 2) + cl], smem[i * (UP_THREADS / 2) + cl]); });
        else
            c.load(ob.lo, [&](int i) { return smem[i * UP_THREADS + cl]; });
        __syncthreads();
        if (t + gridDim.x < total) fetch(t + gridDim.x);
        float best = -3.0e38f;
        // the larger of e + o and e - o is e + |o|
        up_eval<LY>(ob, c, sq, [&](auto nc, int, int, const float2* h, const float2* l) {
#pragma unroll
            for (int u = 0; u < decltype(nc)::value; ++u)
                best = fmaxf(best, fmaxf(h[u].x + fabsf(h[u].y), l[u].x + fabsf(l[u].y)));
        });
        const long p = t / ntile, r = (t - p * ntile) * cols + cl;
        if (r < rows) ccmax[p * (rows / nomr * nom) + r / nomr * nom + r % nomr + (long)half * nomr] = best;
    }
}
// Any number of functions: blocks of 64 orientations (32 bank rows and the half turn, or 64 bank rows) by 4
// shares of y.  Issue 50 %, shared memory 60 %, the rest waits for the block's products.  A particle of
// box 256 on the 1-degree grid at +-6.5 px (320 rows): 0.23 ms, at +-10 px 0.68, its contraction 0.59;
// with every product read from C again for every pair of y 2.4 and 3.8 ms.  Two shares of y 0.19 and 0.90; two
// pairs of y a warp (fewer reads, half the warps) 0.26; pairs of x 8 at a time 0.26.
constexpr int UM_COLS = 64, UM_THREADS = UM_COLS * UM_SHARES;
template <bool QSH, int W>
__global__ void __launch_bounds__(UM_THREADS, 2) k_up_max_any(OriginDev ob, OriginPack pk, const float* __restrict__ C,
                                                              long pitch, long rows, int nom, int nomr, int chunk,
                                                              float* __restrict__ ccmax) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ float sbest[UM_SHARES - 1][UM_COLS];
    const int hn = (ob.n1 + 1) / 2, ne = ob.nent;
    float4* sc = reinterpret_cast<float4*>(smraw + up_any_table_bytes(ob, QSH));  // [chunk][UM_COLS]
    const bool two = nom != nomr;
    const int cols = two ? UM_COLS / 2 : UM_COLS;
    const int p = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long r0 = (long)blockIdx.x * cols;
    const float* U = C + pk.at_c(ob.used, p, two ? 2 : 1) * pitch + r0;  // (pitch: whole tiles of 256)
    const float* V = U + pk.rows * pitch;
    const int col = 32 * (warp & 1) + lane, share = warp >> 1;
    UpAny A = up_any_tables<QSH>(ob, smraw);
    A.c = sc + col;
    A.cols = UM_COLS;
    auto load = [&](int e0, int e1) {
        __syncthreads();
        // four columns of an entry a thread, 16 bytes a load
        const int lg = two ? 3 : 4;  // threads an entry
        for (int i = threadIdx.x; i < (e1 - e0) << lg; i += UM_THREADS) {
            const int e = i >> lg, c = 4 * (i & ((1 << lg) - 1));
            int row[8];
            up_any_rows(ob, e0 + e, row);
            float w[2][4][4];  // [sign][column][function]
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                float4 u[2], v[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    u[k] = v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                    const int at = row[2 * f + k];
                    if (at < 0) continue;
                    u[k] = __ldg(reinterpret_cast<const float4*>(U + at * pitch + c));
                    if (two) v[k] = __ldg(reinterpret_cast<const float4*>(V + at * pitch + c));
                }
                const float4 a = make_float4(fmaf(u[1].x, ob.lo, u[0].x), fmaf(u[1].y, ob.lo, u[0].y),
                                             fmaf(u[1].z, ob.lo, u[0].z), fmaf(u[1].w, ob.lo, u[0].w));
                const float4 b = make_float4(fmaf(v[1].x, ob.lo, v[0].x), fmaf(v[1].y, ob.lo, v[0].y),
                                             fmaf(v[1].z, ob.lo, v[0].z), fmaf(v[1].w, ob.lo, v[0].w));
                w[0][0][f] = a.x + b.x, w[0][1][f] = a.y + b.y, w[0][2][f] = a.z + b.z, w[0][3][f] = a.w + b.w;
                w[1][0][f] = a.x - b.x, w[1][1][f] = a.y - b.y, w[1][2][f] = a.z - b.z, w[1][3][f] = a.w - b.w;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float4* at = sc + e * UM_COLS + c + j;
                at[0] = make_float4(w[0][j][0], w[0][j][1], w[0][j][2], w[0][j][3]);
                if (two) at[UM_COLS / 2] = make_float4(w[1][j][0], w[1][j][1], w[1][j][2], w[1][j][3]);
            }
        }
        __syncthreads();
    };
    if (chunk >= ne) load(0, ne);
    float best = -3.0e38f;
    for (int x0 = 0; x0 < hn; x0 += W)
        for (int j0 = 0; j0 < hn; j0 += UM_SHARES) {
            float2 ah[W], al[W];
#pragma unroll
            for (int u = 0; u < W; ++u) ah[u] = al[u] = make_float2(0.f, 0.f);
            const int jy = j0 + share;
            for (int e0 = 0; e0 < ne; e0 += chunk) {
                const int e1 = min(ne, e0 + chunk);
                if (chunk < ne) load(e0, e1);
                if (jy >= hn) continue;
                up_any_add(A, e0, e1, jy, x0, ah, al);
            }
            if (jy >= hn) continue;
#pragma unroll
            for (int u = 0; u < W; ++u)
                if (x0 + u < hn) best = fmaxf(best, fmaxf(ah[u].x + fabsf(ah[u].y), al[u].x + fabsf(al[u].y)));
        }
    if (share) sbest[share - 1][col] = best;
    __syncthreads();
    if (share) return;
#pragma unroll
    for (int i = 0; i < UM_SHARES - 1; ++i) best = fmaxf(best, sbest[i][col]);
    const int half = two ? warp & 1 : 0;
    const long r = r0 + (two ? lane : col);
    if (r < rows) ccmax[(long)p * (rows / nomr * nom) + r / nomr * nom + r % nomr + (long)half * nomr] = best;
}

// Per (particle, block of 256 orientations): the best value and its orientation.
__global__ void __launch_bounds__(256) k_tile_best(const float* __restrict__ ccmax, long n_orient, int ntiles,
                                                   float* __restrict__ bv_out, int* __restrict__ bo_out) {
    __shared__ float sv[8];
    __shared__ int si[8];
    const int t = blockIdx.x, p = blockIdx.y;
    const long n = (long)t * 256 + threadIdx.x;
    float bv = n < n_orient ? ccmax[(long)p * n_orient + n] : -3.0e38f;
    int bi = bv > -3.0e38f ? (int)n : -1;
    for (int off = 16; off > 0; off >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, off);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
        if (ov > bv || (ov == bv && oi >= 0 && oi < bi)) { bv = ov; bi = oi; }
    }
    if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = bv; si[threadIdx.x >> 5] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 1; q < 8; ++q)
            if (sv[q] > sv[0]) { sv[0] = sv[q]; si[0] = si[q]; }
        bv_out[(long)p * ntiles + t] = sv[0];
        bo_out[(long)p * ntiles + t] = si[0];
    }
}

// Best origin (index iy n1 + ix) of the selected orientations: one block per (candidate,
// particle), a thread per row of origins in turn.
constexpr int UO_X = 32;  // origins of a row at a time
__global__ void __launch_bounds__(128) k_up_origin(OriginDev ob, OriginPack pk, const float* __restrict__ C, long pitch,
                                                   int nom, int nomr, const int* __restrict__ orient, int k,
                                                   int* __restrict__ origin) {
    __shared__ float sv[4];
    __shared__ int si[4];
    const int p = blockIdx.y, parts = nom / nomr, n = orient[p * k + blockIdx.x];
    float bv = -3.0e38f;
    int bi = 0x7fffffff;
    if (n >= 0) {
        const int io = n % nom;
        const long r = (long)(n / nom) * nomr + io % nomr;
        const float* U = C + pk.at_c(ob.used, p, parts) * pitch + r;
        const float* V = parts > 1 ? U + pk.rows * pitch : nullptr;
        for (int iy = threadIdx.x; iy < ob.n1; iy += blockDim.x)
            for (int x0 = 0; x0 < ob.n1; x0 += UO_X) {
                float s[UO_X];
#pragma unroll
                for (int j = 0; j < UO_X; ++j) s[j] = 0.0f;
                for (int m = 0; m < ob.nb; ++m) {
                    float t = 0.0f;
                    for (int q = 0; q < ob.nb; ++q)
                        t = fmaf(up_coef(ob, U, V, io >= nomr ? -1.0f : 1.0f, pitch, m, q), ob.q[(long)q * ob.n1 + iy], t);
                    const float* qx = ob.q + (long)m * ob.n1 + x0;
#pragma unroll
                    for (int j = 0; j < UO_X; ++j)
                        if (x0 + j < ob.n1) s[j] = fmaf(t, qx[j], s[j]);
                }
#pragma unroll
                for (int j = 0; j < UO_X; ++j)
                    if (x0 + j < ob.n1 && s[j] > bv) { bv = s[j]; bi = iy * ob.n1 + x0 + j; }
            }
    }
    for (int off = 16; off > 0; off >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, off);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = bv; si[threadIdx.x >> 5] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 1; q < 4; ++q)
            if (sv[q] > sv[0] || (sv[q] == sv[0] && si[q] < si[0])) { sv[0] = sv[q]; si[0] = si[q]; }
        origin[p * k + blockIdx.x] = bi == 0x7fffffff && si[0] == 0x7fffffff ? 0 : si[0];
    }
}

// Listed orientations (the proposal forms): one block per (block of 256 list positions,
// particle) gives, per origin, the best of its positions and which it is (the first of
// equal ones), as the argmax contraction does for a local grid's columns.  A warp takes 32
// positions at a time and keeps its running maxima over the origins in shared memory; the
// maximum of 32 lanes by redux on the
// order-preserving integer image of the value, up to 16 origins at a time so that their
// latencies overlap (one origin at a time, with its update in between: 185 us a 64-particle
// pass of the box-256 search; so: 137 us).  gridDim.z blocks share a tile's origins by rows (pairs of
// y about the middle) where a call has few tiles: one particle's three, 625 origins, 60 -> 23 us.

// The maxima of 4 N origins (up_eval's pairs of x jx .. jx + N - 1 at the pair of y jy) over a
// warp's 32 positions: they are independent, lane i keeps the i-th and hands it to put(y, x, value, lane of the
// maximum).
template <int N, class Put>
__device__ __forceinline__ void list_max(const float2* h, const float2* l, bool valid, int n1, int jy, int jx, Put put) {
    const int lane = threadIdx.x & 31;
    float mine = 0.0f;
    int who = -1;
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const float v[4] = {h[u].x + h[u].y, h[u].x - h[u].y, l[u].x + l[u].y, l[u].x - l[u].y};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const unsigned x = __float_as_uint(v[q]);
            const unsigned key = valid ? ((x & 0x80000000u) ? ~x : (x | 0x80000000u)) : 0u;
            const unsigned mx = __reduce_max_sync(0xffffffffu, key);
            const unsigned eq = __ballot_sync(0xffffffffu, key == mx);
            if (lane == 4 * u + q) {
                mine = __uint_as_float((mx & 0x80000000u) ? (mx & 0x7fffffffu) : ~mx);
                who = __ffs(eq) - 1;
            }
        }
    }
    const int jj = jx + (lane >> 2);
    if (who >= 0 && jj < (n1 + 1) / 2)
        put((lane & 2) ? (n1 - 1) / 2 - jy : n1 / 2 + jy, (lane & 1) ? (n1 - 1) / 2 - jj : n1 / 2 + jj, mine, who);
}
template <int LY>
__global__ void __launch_bounds__(256, 1) k_up_list(OriginDev ob, const float* __restrict__ C, int parts,
                                                    const UpGroup* __restrict__ groups, const int* __restrict__ map,
                                                    float* __restrict__ topv, int* __restrict__ topi) {
    extern __shared__ __align__(16) float smem[];
    const UpGroup g = groups[blockIdx.y];
    const int tile = blockIdx.x;
    if (tile >= g.ntiles) return;
    const int O = ob.n1 * ob.n1, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    float* sv = smem + up_table_floats<LY>(ob.n1) + warp * O;
    int* si = reinterpret_cast<int*>(smem + up_table_floats<LY>(ob.n1) + nw * O) + warp * O;
    float* ov = topv + g.topv_off + tile;  // stride ntiles
    int* oi = topi + g.topv_off + tile;
    const int hn = (ob.n1 + 1) / 2;
    const int jy0 = hn * (int)blockIdx.z / (int)gridDim.z, jy1 = hn * ((int)blockIdx.z + 1) / (int)gridDim.z;
    up_table<LY>(ob, smem);
    for (int o = lane; o < O; o += 32) { sv[o] = -3.0e38f; si[o] = -1; }
    __syncthreads();
    const long pitch = 256L * g.n_tiles;
    for (int c = warp; c < 8; c += nw) {
        const int j0 = tile * 256 + c * 32;
        if (j0 >= g.n_list) break;
        const int j = j0 + lane;
        const bool valid = j < g.n_list;
        const int mp = map[g.map_off + (valid ? j : 0)];
        const float* U = C + g.c_off + (mp >> 1);
        const float* V = parts > 1 ? U + ob.slots * pitch : nullptr;
        const float sgn = (mp & 1) ? -1.0f : 1.0f;
        // (neighbouring list positions mostly stand for neighbouring columns)
        UpCoef<LY> cf;
        cf.load(ob.lo, [&](int i) {
            const float u = __ldg(U + i * pitch);
            return V ? fmaf(sgn, __ldg(V + i * pitch), u) : u;
        });
        auto keep = [&](int y, int x, float v, int who) {
            const int o = y * ob.n1 + x;
            if (v > sv[o]) {
                sv[o] = v;
                si[o] = j0 + who;
            }
        };
        up_eval<LY>(ob, cf, smem,
                    [&](auto nc, int jy, int jx, const float2* h, const float2* l) {
                        list_max<decltype(nc)::value>(h, l, valid, ob.n1, jy, jx, keep);
                    },
                    jy0, jy1);
        __syncwarp();  // the next 32 positions update these maxima from other lanes
    }
    __syncthreads();
    sv = smem + up_table_floats<LY>(ob.n1);
    si = reinterpret_cast<int*>(sv + nw * O);
    for (int o = threadIdx.x; o < O; o += blockDim.x) {
        const int y = o / ob.n1, jy = y >= ob.n1 / 2 ? y - ob.n1 / 2 : (ob.n1 - 1) / 2 - y;
        if (jy < jy0 || jy >= jy1) continue;
        float bv = -3.0e38f;
        int bi = -1;
        for (int w = 0; w < nw; ++w) {
            const float x = sv[w * O + o];
            const int i = si[w * O + o];
            if (i >= 0 && (x > bv || (x == bv && i < bi))) { bv = x; bi = i; }
        }
        ov[(long)o * g.ntiles] = bv;
        oi[(long)o * g.ntiles] = bi;
    }
}

// The same for any number of functions and origins.  A task is a pair of y and UL_X pairs of x: 32 origins, a
// lane each.  A warp's tasks are its own for all positions of the tile, which the block goes through 32 at a
// time, so that an origin's maximum is one warp's alone.  blockIdx.z blocks share a tile's tasks.  One particle's
// lists of box 256 at +-8 px (33 x 33 origins): 73 us, 64 particles' 356; with every product read from C
// again for every pair of y 1.4 and 3.1 ms.  Two pairs of y and 16 of x a task 188 and 380 us.
template <bool QSH>
__global__ void __launch_bounds__(UL_THREADS, 2) k_up_list_any(OriginDev ob, const float* __restrict__ C, int parts,
                                                               const UpGroup* __restrict__ groups,
                                                               const int* __restrict__ map, int chunk,
                                                               float* __restrict__ topv, int* __restrict__ topi) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const UpGroup g = groups[blockIdx.y];
    const int tile = blockIdx.x;
    if (tile >= g.ntiles) return;
    const int hn = (ob.n1 + 1) / 2, ne = ob.nent, n1 = ob.n1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int NW = UL_THREADS / 32;
    const int nx = (hn + UL_X - 1) / UL_X, tasks = hn * nx;
    const int t0 = (int)((long)tasks * blockIdx.z / gridDim.z), t1 = (int)((long)tasks * (blockIdx.z + 1) / gridDim.z);
    float4* sc = reinterpret_cast<float4*>(smraw + up_any_table_bytes(ob, QSH));  // [chunk][32]
    float* sv = reinterpret_cast<float*>(sc + chunk * 32);                        // [t1 - t0][32]
    int* si = reinterpret_cast<int*>(sv + (t1 - t0) * 32);
    for (int t = t0 + warp; t < t1; t += NW) {
        sv[(t - t0) * 32 + lane] = -3.0e38f;
        si[(t - t0) * 32 + lane] = -1;
    }
    const long pitch = 256L * g.n_tiles;
    UpAny A = up_any_tables<QSH>(ob, smraw);
    A.c = sc + lane;
    A.cols = 32;
    for (int c = 0; c < 8; ++c) {
        const int j0 = tile * 256 + c * 32;
        if (j0 >= g.n_list) break;
        const bool valid = j0 + lane < g.n_list;
        const int mp = map[g.map_off + (valid ? j0 + lane : 0)];  // (of this lane's column, which it also loads)
        const float* U = C + g.c_off + (mp >> 1);
        const float* V = U + ob.slots * pitch;
        const float sgn = (mp & 1) ? -1.0f : 1.0f;
        auto load = [&](int e0, int e1) {
            __syncthreads();
            // an entry a warp, two at a time: up to 32 loads in flight
            for (int e = e0 + warp; e < e1; e += 2 * NW) {
                float u[2][8], v[2][8];
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    int row[8];
                    up_any_rows(ob, min(e + t * NW, e1 - 1), row);
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const bool in = row[k] >= 0 && e + t * NW < e1;
                        u[t][k] = in ? __ldg(U + row[k] * pitch) : 0.0f;
                        v[t][k] = in && parts > 1 ? __ldg(V + row[k] * pitch) : 0.0f;
                    }
                }
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    if (e + t * NW < e1) sc[(e + t * NW - e0) * 32 + lane] = up_any_four(u[t], v[t], sgn, ob.lo);
            }
            __syncthreads();
        };
        if (chunk >= ne) load(0, ne);
        for (int tb = t0; tb < t1; tb += NW) {
            const int t = tb + warp, jy = t / nx, x0 = (t - jy * nx) * UL_X;
            float2 ah[UL_X], al[UL_X];
#pragma unroll
            for (int u = 0; u < UL_X; ++u) ah[u] = al[u] = make_float2(0.f, 0.f);
            for (int e0 = 0; e0 < ne; e0 += chunk) {
                const int e1 = min(ne, e0 + chunk);
                if (chunk < ne) load(e0, e1);
                if (t < t1) up_any_add(A, e0, e1, jy, x0, ah, al);
            }
            if (t >= t1) continue;
            const int at = (t - t0) * 32 + lane;
            list_max<UL_X>(ah, al, valid, n1, jy, x0, [&](int, int, float v, int who) {
                if (v > sv[at]) {
                    sv[at] = v;
                    si[at] = j0 + who;
                }
            });
        }
    }
    float* ov = topv + g.topv_off + tile;  // stride ntiles
    int* oi = topi + g.topv_off + tile;
    for (int t = t0 + warp; t < t1; t += NW) {
        const int jy = t / nx, jx = (t - jy * nx) * UL_X + (lane >> 2), at = (t - t0) * 32 + lane;
        if (jx >= hn) continue;
        // (hi and lo are the same row, or column, in the middle of an odd grid: equal values)
        const int y = (lane & 2) ? (n1 - 1) / 2 - jy : n1 / 2 + jy, x = (lane & 1) ? (n1 - 1) / 2 - jx : n1 / 2 + jx;
        ov[((long)y * n1 + x) * g.ntiles] = sv[at];
        oi[((long)y * n1 + x) * g.ntiles] = si[at];
    }
}

// The larger (value, index) of a block's threads, the first of equal values, for every thread; index
// -1: none.  sv, si: 32 each and a place for the result.
__device__ __forceinline__ void block_best(float& v, int& i, float* sv, int* si) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
    auto warp = [&]() {
        for (int off = 16; off > 0; off >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, off);
            const int oi = __shfl_xor_sync(0xffffffffu, i, off);
            if (ov > v || (ov == v && oi >= 0 && (i < 0 || oi < i))) { v = ov; i = oi; }
        }
    };
    warp();
    if (l == 0) { sv[w] = v; si[w] = i; }
    __syncthreads();
    if (w == 0) {
        v = l < nw ? sv[l] : -3.0e38f;
        i = l < nw ? si[l] : -1;
        warp();
        if (l == 0) { sv[32] = v; si[32] = i; }
    }
    __syncthreads();
    v = sv[32];
    i = si[32];
}

// Per particle: the k best entries of cnt (value, orientation) pairs; a thread keeps the best of its
// entries and looks through them again (taken ones set to -inf in v, a scratch array) once one is taken.
__global__ void k_select_topk(float* __restrict__ v, const int* __restrict__ orient, int cnt, int k,
                              int* __restrict__ out_orient, float* __restrict__ out_cc) {
    __shared__ float sv[33];
    __shared__ int si[33];
    const int p = blockIdx.x;
    const long base = (long)p * cnt;
    float bv;
    int bi;
    auto scan = [&]() {
        bv = -3.0e38f;
        bi = -1;
        for (int q = threadIdx.x; q < cnt; q += blockDim.x) {
            const float x = v[base + q];
            if (x > bv) { bv = x; bi = q; }
        }
    };
    scan();
    for (int r = 0; r < k; ++r) {
        float x = bv;
        int i = bi;
        block_best(x, i, sv, si);
        if (threadIdx.x == 0) {
            out_orient[p * k + r] = i >= 0 ? orient[base + i] : -1;
            out_cc[p * k + r] = i >= 0 ? x : -3.0e38f;
        }
        if (i >= 0 && i == bi) {
            v[base + i] = -3.0e38f;
            scan();
        }
    }
}

// Proposal form, per particle: the k best (origin row, column tile) maxima with
// distinct orientations.  v[o * ntiles + t] is the best CC of tile t at origin o and
// col[...] its column in the gathered list; once a column is taken, every entry that
// names it is retired, so the candidates are k distinct orientations, each at its best
// origin.  Columns are remapped to orientations on the host.
// One block per particle of a group: seg[b] = (offset of its entries, its ntiles).  SHARED: the
// entries in shared memory (else v is scratch: retired entries are set to -inf).  Retiring a column
// and finding a thread's next best is one pass over its entries.  One particle of 1,875 entries, 16
// of them: 28 us with two passes over global memory and a serial comparison of the warps' bests a
// round, now 23; the 17,918 entries of each of 24 local grids 95, now 78.
template <bool SHARED>
__global__ void __launch_bounds__(512) k_select_distinct(float* __restrict__ v0, const int* __restrict__ col0, int O,
                                                        const int2* __restrict__ seg, int k,
                                                        int* __restrict__ out_col0, int* __restrict__ out_origin0,
                                                        float* __restrict__ out_cc0) {
    extern __shared__ float sent[];  // values, then columns
    __shared__ float sv[33];
    __shared__ int si[33];
    const int2 sg = seg[blockIdx.x];
    const int ntiles = sg.y, cnt = O * ntiles;
    float* v = v0 + sg.x;
    const int* col = col0 + sg.x;
    int* out_col = out_col0 + (long)blockIdx.x * k;
    int* out_origin = out_origin0 + (long)blockIdx.x * k;
    float* out_cc = out_cc0 + (long)blockIdx.x * k;
    if (SHARED) {  // a thread reads its own entries alone
        int* sc = reinterpret_cast<int*>(sent + cnt);
        for (int q = threadIdx.x; q < cnt; q += blockDim.x) {
            sent[q] = v[q];
            sc[q] = col[q];
        }
        v = sent;
        col = sc;
    }
    int taken = -1;
    for (int r = 0; r < k; ++r) {
        float bv = -3.0e38f;
        int bi = -1;
#pragma unroll 4
        for (int q = threadIdx.x; q < cnt; q += blockDim.x) {
            const int c = col[q];
            const float x = v[q];
            if (c < 0) continue;
            if (c == taken) v[q] = -3.0e38f;
            else if (x > bv) { bv = x; bi = q; }
        }
        block_best(bv, bi, sv, si);
        taken = -1;
        if (bi >= 0) taken = SHARED ? reinterpret_cast<const int*>(sent + cnt)[bi] : col[bi];
        if (threadIdx.x == 0) {
            out_col[r] = taken;
            out_origin[r] = bi >= 0 ? bi / ntiles : 0;
            out_cc[r] = bi >= 0 ? bv : -3.0e38f;
        }
    }
}

// FP64 rescoring of one (particle, candidate): the same CC with every product,
// interpolation and sum in double precision.
// FP64 rescoring, one (candidate, particle, sample chunk) per block: the three sums of
// the CC (p.q, |p|^2, |q|^2) over samples [S*s/NS, S*(s+1)/NS).  The section sample
// is interpolated at FP64-rotated coordinates; its trilinear blend of the FP32 cube runs
// in FP32 (the data's own precision), every product and sum after it in FP64.  The
// origin shift exp(-i 2pi (sx hx + sy ky)/n) is separable, so each block tabulates the
// per-hx and per-ky phasors in double once and multiplies them per sample.
constexpr int CC_SPLIT = 4;

__global__ void k_cc_fp64(const float2* __restrict__ cube, const double2* __restrict__ pcband, Band bd,
                          const int2* __restrict__ samples, int S, const float* __restrict__ cand, int k,
                          double* __restrict__ part, double gk, const float* __restrict__ pctf, int Rq, double sc) {
    extern __shared__ double2 ctab[];  // [R + 1] per hx, then [2R + 1] per ky
    __shared__ double sh[32];
    __shared__ double rot[9], trig[6];
    // R: the band; Rq: the cube's radius (its side C = 2 Rq + 3), sc cube voxels per frequency
    const int c = blockIdx.x, p = blockIdx.y, sp = blockIdx.z, R = bd.max_r, C = 2 * Rq + 3, off = Rq + 1;
    const float* cd = cand + ((long)p * k + c) * 5;
    if (threadIdx.x < 6) {  // cosines and sines of phi, theta, omega, a lane each
        const int e = threadIdx.x % 3;
        const double d2r = 3.14159265358979323846 / 180.0, ang = cd[e == 0 ? 1 : e == 1 ? 0 : 2] * d2r;
        trig[threadIdx.x] = threadIdx.x < 3 ? cos(ang) : sin(ang);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double c1 = trig[0], c2 = trig[1], c3 = trig[2], s1 = trig[3], s2 = trig[4], s3 = trig[5];
        rot[0] = c1 * c2 * c3 - s1 * s3; rot[1] = -c1 * c2 * s3 - c3 * s1; rot[2] = c1 * s2;
        rot[3] = c2 * c3 * s1 + c1 * s3; rot[4] = -c2 * s1 * s3 + c1 * c3; rot[5] = s1 * s2;
        rot[6] = -c3 * s2;               rot[7] = s2 * s3;                 rot[8] = c2;
        for (int i = 0; i < 9; ++i) rot[i] *= sc;
    }
    const double h = (double)(bd.nx / 2), sx = cd[3] + h, sy = cd[4] + h;
    const double tpn = 2.0 * 3.14159265358979323846 / (double)bd.nx;
    double2* tx = ctab;
    double2* ty = ctab + (R + 1);
    for (int i = threadIdx.x; i < 3 * R + 2; i += blockDim.x) {
        double th, sn, cs;
        if (i <= R) th = tpn * (sx * (double)i);
        else th = tpn * (sy * (double)(i - (R + 1) - R));
        sincos(th, &sn, &cs);
        ctab[i] = make_double2(cs, sn);
    }
    __syncthreads();
    const double2* pcb = pcband + (long)p * S;  // CTF x (a, b) per sample, FP64 (k_particle_norm)
    double dot = 0, nb = 0;  // the particle's norm is the same for every candidate: k_particle_norm
    const int i0 = (int)((long)S * sp / gridDim.z), i1 = (int)((long)S * (sp + 1) / gridDim.z);
    for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
        const int2 hk = samples[i];
        const double x = rot[0] * hk.x + rot[1] * hk.y, y = rot[3] * hk.x + rot[4] * hk.y,
                     z = rot[6] * hk.x + rot[7] * hk.y;
        double sr, si;
        if (gk > 0.0) {
            // Gaussian kernel in FP64 over the 27 voxels around the nearest one
            const double rx = rint(x), ry = rint(y), rz = rint(z);
            double wx[3], wy[3], wz[3];
            for (int d = 0; d < 3; ++d) {
                const double ex = x - (rx + (d - 1)), ey = y - (ry + (d - 1)), ez = z - (rz + (d - 1));
                wx[d] = exp(-gk * ex * ex);
                wy[d] = exp(-gk * ey * ey);
                wz[d] = exp(-gk * ez * ez);
            }
            const float2* b0 = cube + ((long)((int)rz + off - 1) * C + ((int)ry + off - 1)) * C + ((int)rx + off - 1);
            double ar = 0.0, ai = 0.0;
            for (int dz = 0; dz < 3; ++dz)
                for (int dy = 0; dy < 3; ++dy) {
                    const float2* rr = b0 + ((long)dz * C + dy) * C;
                    const double w = wz[dz] * wy[dy];
                    ar += w * (wx[0] * rr[0].x + wx[1] * rr[1].x + wx[2] * rr[2].x);
                    ai += w * (wx[0] * rr[0].y + wx[1] * rr[1].y + wx[2] * rr[2].y);
                }
            const double inv = 1.0 / ((wx[0] + wx[1] + wx[2]) * (wy[0] + wy[1] + wy[2]) * (wz[0] + wz[1] + wz[2]));
            sr = ar * inv;
            si = ai * inv;
        } else {
            // the cube holds FP32 values: its trilinear blend runs in FP32 at the FP64-rotated
            // coordinates rounded once to FP32 (|x| <= maxR + 1: within 2^-17 px), the products
            // and sums below in FP64
            const float xf = (float)x, yf = (float)y, zf = (float)z;
            const float fx = floorf(xf), fy = floorf(yf), fz = floorf(zf);
            const int ix = (int)fx + off, iy = (int)fy + off, iz = (int)fz + off;
            const float ax = xf - fx, ay = yf - fy, az = zf - fz;
            const float2* cb0 = cube + ((long)iz * C + iy) * C + ix;
            float2 r0, r1;
            {
                const float2 v000 = cb0[0], v001 = cb0[1], v010 = cb0[C], v011 = cb0[C + 1];
                const float2 v100 = cb0[C * C], v101 = cb0[C * C + 1], v110 = cb0[C * C + C], v111 = cb0[C * C + C + 1];
                const float2 a0 = make_float2(fmaf(ax, v001.x - v000.x, v000.x), fmaf(ax, v001.y - v000.y, v000.y));
                const float2 a1 = make_float2(fmaf(ax, v011.x - v010.x, v010.x), fmaf(ax, v011.y - v010.y, v010.y));
                const float2 a2 = make_float2(fmaf(ax, v101.x - v100.x, v100.x), fmaf(ax, v101.y - v100.y, v100.y));
                const float2 a3 = make_float2(fmaf(ax, v111.x - v110.x, v110.x), fmaf(ax, v111.y - v110.y, v110.y));
                r0 = make_float2(fmaf(ay, a1.x - a0.x, a0.x), fmaf(ay, a1.y - a0.y, a0.y));
                r1 = make_float2(fmaf(ay, a3.x - a2.x, a2.x), fmaf(ay, a3.y - a2.y, a2.y));
            }
            sr = (double)fmaf(az, r1.x - r0.x, r0.x);
            si = (double)fmaf(az, r1.y - r0.y, r0.y);
        }
        // cos/sin of tpn (sx hx + sy ky) from the two tabulated phasors
        const double2 ex = tx[hk.x], ey = ty[hk.y + R];
        const double cs = ex.x * ey.x - ex.y * ey.y, sn = ex.y * ey.x + ex.x * ey.y;
        // the origin-shifted particle sample (img2d_FT_centshift.f90, b = -Im convention)
        const double2 pc = pcb[i];
        const double pr = pc.x * cs + pc.y * sn, pi = pc.x * sn - pc.y * cs;
        dot += pr * sr + pi * si;
        const double cw = pctf ? (double)pctf[(long)p * S + i] : 1.0;
        nb += cw * cw * (sr * sr + si * si);
    }
    dot = block_sum_double(dot, sh);
    nb = block_sum_double(nb, sh);
    if (threadIdx.x == 0) {
        double* o = part + (((long)p * k + c) * gridDim.z + sp) * 3;
        o[0] = dot;
        o[1] = 0.0;
        o[2] = nb;
    }
}

// CC of each (particle, candidate) from its chunks' sums, in chunk order.
// CC = dot / sqrt(|P|^2 |S|^2): the chunks' dot and section norms, the particle's FP64 norm
// (sum over the samples of |CTF P|^2, k_particle_norm; the origin phase keeps it)
__global__ void k_cc_fp64_finish(const double* __restrict__ part, int n, int ns, const double* __restrict__ pnorm,
                                 int k, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double dot = 0, nb = 0;
    for (int s = 0; s < ns; ++s) {
        dot += part[((long)i * ns + s) * 3];
        nb += part[((long)i * ns + s) * 3 + 2];
    }
    const double na = pnorm[i / k];
    out[i] = (na > 0 && nb > 0) ? dot / sqrt(na * nb) : 0.0;
}

// ---- FP8-e4m3 operands ---------------------------------------------------------
// Both operands are unit-norm rows whose elements span a wide range: low-frequency
// samples carry most of the norm, high-frequency ones little.  Each radial band b =
// int(|h|) of the samples gets a power-of-two scale 2^e_b on the B side (the sections)
// and 2^-e_b on the A side (the particles), so every product, hence every score, is
// unchanged, while each band of B uses the top of the e4m3 range (max 448).  A whole A
// row is further scaled by 2^f_p per particle (its origins share it), which scales all
// of that particle's scores alike and is removed from the reported CC.

__device__ __forceinline__ int sample_band(int2 hk) {
    return (int)sqrtf((float)(hk.x * hk.x + hk.y * hk.y));
}

// Largest |Re| or |Im| of B per band over every stride-th row (float bits, non-negative,
// so unsigned order is float order).
__global__ void k_band_absmax(const __nv_bfloat16* __restrict__ B, long n, int KH, const int2* __restrict__ samples,
                              int S, int nband, int stride, unsigned* __restrict__ out) {
    extern __shared__ unsigned smax[];
    for (int b = threadIdx.x; b < nband; b += blockDim.x) smax[b] = 0u;
    __syncthreads();
    for (long r = (long)blockIdx.x * stride; r < n; r += (long)gridDim.x * stride) {
        const __nv_bfloat16* row = B + r * (2 * KH);
        for (int i = threadIdx.x; i < S; i += blockDim.x) {
            const float m = fmaxf(fabsf(__bfloat162float(row[bf16_at(i, r)])),
                                  fabsf(__bfloat162float(row[bf16_at(KH + i, r)])));
            atomicMax(&smax[sample_band(samples[i])], __float_as_uint(m));
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < nband; b += blockDim.x)
        if (smax[b]) atomicMax(&out[b], smax[b]);
}

// One CTA per row: B8[r] = e4m3(B[r] * mulB[sample]), both parts zero padded to KH8 bytes.
__global__ void k_b_to_e4m3(const __nv_bfloat16* __restrict__ B, int KH, int S, const float* __restrict__ mulB,
                            int KH8, unsigned char* __restrict__ B8) {
    const long r = blockIdx.x;
    const __nv_bfloat16* row = B + r * (2 * KH);
    unsigned char* out = B8 + r * (2 * KH8);
    for (int i = 2 * threadIdx.x; i < KH8; i += 2 * blockDim.x)
#pragma unroll
        for (int im = 0; im < 2; ++im) {
            float2 v = make_float2(0.f, 0.f);
            if (i < S) v.x = __bfloat162float(row[bf16_at(im * KH + i, r)]) * mulB[i];
            if (i + 1 < S) v.y = __bfloat162float(row[bf16_at(im * KH + i + 1, r)]) * mulB[i + 1];
            *reinterpret_cast<unsigned short*>(out + fp8_at(im * KH8 + i, r)) =
                __nv_cvt_float2_to_fp8x2(v, __NV_SATFINITE, __NV_E4M3);
        }
}

// Per particle: f_p = floor(log2(224 / max_i |A_i| mulA_i)) with |A_i| = |CTF P| / |A|.
__global__ void k_particle_exp8(const float2* __restrict__ band, const float* __restrict__ ctf, Band bd,
                                const int2* __restrict__ samples, int S, const double* __restrict__ norm,
                                const float* __restrict__ mulA, int* __restrict__ fexp) {
    __shared__ float sm[32];
    const int p = blockIdx.x, W = bd.W, R = bd.max_r;
    const float2* b = band + (long)p * W * W;
    const float* c = ctf ? ctf + (long)p * W * W : nullptr;
    const float inv = norm[p] > 0.0 ? (float)(1.0 / sqrt(norm[p])) : 0.0f;
    float m = 0.0f;
    for (int i = threadIdx.x; i < S; i += blockDim.x) {
        const int2 hk = samples[i];
        const int q = (hk.y + R) * W + (hk.x + R);
        const float a = sqrtf(b[q].x * b[q].x + b[q].y * b[q].y) * fabsf(c ? c[q] : 1.0f);
        m = fmaxf(m, a * inv * mulA[i]);
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmaxf(m, sm[w]);
        m = fmaxf(m, sm[0]);
        fexp[p] = m > 0.0f ? (int)floorf(log2f(224.0f / m)) : 0;
    }
}

inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

}  // namespace

cudaError_t launch_band_absmax(const void* B, long n, int KH, const int2* samples, int S, int nband, int stride,
                               unsigned* out, int sms, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(unsigned) * nband, st);
    if (e != cudaSuccess) return e;
    long rows = (n + stride - 1) / stride;
    int grid = (int)(rows < 4L * sms ? rows : 4L * sms);
    k_band_absmax<<<grid, 256, sizeof(unsigned) * nband, st>>>((const __nv_bfloat16*)B, n, KH, samples, S, nband,
                                                               stride, out);
    return cudaGetLastError();
}

cudaError_t launch_b_to_e4m3(const void* B, long n, int KH, int S, const float* mulB, int KH8, void* B8,
                             cudaStream_t st) {
    // (chunks of a multiple of 8 rows: a row's swizzle residue is its index in the bank)
    for (long r0 = 0; r0 < n; r0 += 1L << 30) {
        long nb = n - r0 < (1L << 30) ? n - r0 : (1L << 30);
        k_b_to_e4m3<<<(unsigned)nb, 256, 0, st>>>((const __nv_bfloat16*)B + r0 * (2 * KH), KH, S, mulB, KH8,
                                                  (unsigned char*)B8 + r0 * (2 * KH8));
    }
    return cudaGetLastError();
}

cudaError_t launch_build_basis(const float2* band, const float* ctf, Band bd, const int2* samples, int S, int KH,
                               const OriginDev& ob, OriginPack pk, const double* norm, int B, void* A, bool f8,
                               const float* mulA, int* fexp, cudaStream_t st, const float* poff) {
    const float tpn = 2.0f * host_angles().pi / (float)bd.nx;
    const bool pack = pk.per > 1;
    const dim3 g(((pack ? ob.used : ob.slots) + BO - 1) / BO, B);
    const size_t sm = (sizeof(float2) + sizeof(float) * BO) * (3 * (size_t)bd.max_r + 2);
    if (f8) k_particle_exp8<<<B, 256, 0, st>>>(band, ctf, bd, samples, S, norm, mulA, fexp);
    auto kern = f8 ? (pack ? k_build_basis<true, true> : k_build_basis<true, false>)
                   : (pack ? k_build_basis<false, true> : k_build_basis<false, false>);
    const cudaError_t e = allow_smem(kern, sm);
    if (e != cudaSuccess) return e;
    kern<<<g, 256, sm, st>>>(band, ctf, bd, samples, S, KH, ob, pk, poff, norm, mulA, fexp, tpn, A);
    return cudaGetLastError();
}

// the register kernels: a fixed layout, and origins whose table leaves room for the products
static int up_layout(const OriginDev& ob) { return ob.n1 <= UP_N1 ? ob.layout : -1; }

// f with the layout ly as a constant
template <int LY, class F>
static void up_dispatch(int ly, F& f) {
    if (ly == LY) f(std::integral_constant<int, LY>());
    else if constexpr (LY + 1 < OB_LAYOUTS) up_dispatch<LY + 1>(ly, f);
}

// Shared memory of the kernels for any number of functions: q's table where it is small, then as many
// entries of cols columns as leave two blocks an SM (113 KB each), at least 16.
struct UpAnyShape {
    bool qsh;
    int chunk;
    size_t smem;
};
static UpAnyShape up_any_shape(const OriginDev& ob, int cols, size_t more) {
    UpAnyShape s;
    const size_t room = 110 * 1024 - more, entry = sizeof(float4) * cols;
    s.qsh = up_any_table_bytes(ob, true) <= 32 * 1024;
    const size_t tab = up_any_table_bytes(ob, s.qsh);
    const size_t fit = room > tab + 16 * entry ? (room - tab) / entry : 16;
    s.chunk = (int)std::min<size_t>(fit / 2 * 2, std::max(2, ob.nent));
    s.smem = tab + s.chunk * entry + more;
    return s;
}

cudaError_t launch_up_topk(const OriginDev& ob, OriginPack pk, const float* C, long pitch, long rows, int nom, int nomr,
                           int B, int k, float* ccmax, int ntiles, float* tile_v, int* tile_o, int* orient, int* origin, float* cc,
                           bool want_origin, int num_sms, cudaStream_t st) {
    const long n_orient = rows / nomr * nom;
    cudaError_t e = cudaSuccess;
    const int ly = up_layout(ob);
    if (ly >= 0) {
        auto run = [&](auto lyc) {
            constexpr int LY = decltype(lyc)::value;
            const int cols = nom == nomr ? UP_THREADS : UP_THREADS / 2;
            const long tiles = (rows + cols - 1) / cols * B;
            const size_t sm = sizeof(float) * (up_table_floats<LY>(ob.n1) + (size_t)UP_THREADS * OB_LAYOUT[LY].rows);
            e = allow_smem(k_up_max<LY>, sm);
            if (e != cudaSuccess) return;
            k_up_max<LY><<<(unsigned)std::min<long>(tiles, num_sms * up_blocks(LY)), UP_THREADS, sm, st>>>(ob, pk, C, pitch, rows, nom, nomr, B,
                                                                                          ccmax);
        };
        up_dispatch<0>(ly, run);
        if (e != cudaSuccess) return e;
    } else {
        const int cols = nom == nomr ? UM_COLS : UM_COLS / 2;
        const UpAnyShape sh = up_any_shape(ob, UM_COLS, 0);
        // pairs of x at a time: as few turns as UM_X allows, in turns of one width
        const int hn = (ob.n1 + 1) / 2, turns = (hn + UM_X - 1) / UM_X, w = ((hn + turns - 1) / turns + 1) / 2 * 2;
        auto kern = !sh.qsh   ? k_up_max_any<false, UM_X>
                    : w <= 8  ? k_up_max_any<true, 8>
                    : w <= 10 ? k_up_max_any<true, 10>
                    : w <= 12 ? k_up_max_any<true, 12>
                    : w <= 14 ? k_up_max_any<true, 14>
                              : k_up_max_any<true, UM_X>;
        if ((e = allow_smem(kern, sh.smem)) != cudaSuccess) return e;
        kern<<<dim3((unsigned)((rows + cols - 1) / cols), B), UM_THREADS, sh.smem, st>>>(ob, pk, C, pitch, rows, nom, nomr,
                                                                                        sh.chunk, ccmax);
    }
    k_tile_best<<<dim3(ntiles, B), 256, 0, st>>>(ccmax, n_orient, ntiles, tile_v, tile_o);
    k_select_topk<<<B, 512, 0, st>>>(tile_v, tile_o, ntiles, k, orient, cc);
    if (want_origin)
        k_up_origin<<<dim3(k, B), 128, 0, st>>>(ob, pk, C, pitch, nom, nomr, orient, k, origin);
    else
        return cudaMemsetAsync(origin, 0, sizeof(int) * (size_t)B * k, st);
    return cudaGetLastError();
}

cudaError_t launch_up_list(const OriginDev& ob, const float* C, int parts, const UpGroup* groups, int ngroups,
                           int max_tiles, const int* map, float* topv, int* topi, cudaStream_t st) {
    const int O = ob.n1 * ob.n1, ly = up_layout(ob);
    // warps per block: the running maxima of each over the origins in shared memory
    const size_t tab = sizeof(float) * ((ob.n1 + 1) / 2 * ((ob.nb + 1) / 2 * 2));
    int nw = 8;
    while (nw > 1 && tab + (size_t)nw * O * 8 > 220 * 1024) nw /= 2;
    const size_t sm = tab + (size_t)nw * O * 8;
    if (ly < 0 || sm > 220 * 1024) {
        // blocks to a tile: as many as find an SM (each combines its positions' products again), and as
        // hold the maxima of their tasks in 48 KB
        const int hn = (ob.n1 + 1) / 2, tasks = hn * ((hn + UL_X - 1) / UL_X), nw = UL_THREADS / 32;
        const int most = 48 * 1024 / (32 * 8), fill = 2 * sm_count() / std::max(1, max_tiles * ngroups);
        const int z = std::max((tasks + most - 1) / most, std::min(fill, (tasks + nw - 1) / nw));
        const UpAnyShape sh = up_any_shape(ob, 32, (size_t)((tasks + z - 1) / z) * 32 * (sizeof(float) + sizeof(int)));
        auto kern = sh.qsh ? k_up_list_any<true> : k_up_list_any<false>;
        const cudaError_t e = allow_smem(kern, sh.smem);
        if (e != cudaSuccess) return e;
        kern<<<dim3(max_tiles, ngroups, z), UL_THREADS, sh.smem, st>>>(ob, C, parts, groups, map, sh.chunk, topv, topi);
        return cudaGetLastError();
    }
    void (*kern)(OriginDev, const float*, int, const UpGroup*, const int*, float*, int*) = nullptr;
    auto pick = [&](auto lyc) { kern = k_up_list<decltype(lyc)::value>; };
    up_dispatch<0>(ly, pick);
    cudaError_t e = allow_smem(kern, sm);
    if (e != cudaSuccess) return e;
    // blocks to a tile: as many as find an SM of their own (each reads its tile's products again, so that with
    // the SMs filled, by this launch or by other lanes', the pass takes longer: 14.0 -> 14.5 ms of the box-256
    // search with 192 tiles cut in three)
    int z = 1;
    z = std::max(1, std::min(std::min(8, (ob.n1 + 1) / 2), sm_count() / std::max(1, max_tiles * ngroups)));
    kern<<<dim3(max_tiles, ngroups, z), 32 * nw, sm, st>>>(ob, C, parts, groups, map, topv, topi);
    return cudaGetLastError();
}

void launch_map_checker(const float* map, int nx, float2* work, cudaStream_t st) {
    const long n3 = (long)nx * nx * nx;
    k_map_checker<<<cdiv(n3, 256) < 65535 ? cdiv(n3, 256) : 65535, 256, 0, st>>>(map, nx, work);
}

void launch_map_band(const float2* ft, int nx, int R, float2* cube, cudaStream_t st) {
    const long c3 = (long)(2 * R + 3) * (2 * R + 3) * (2 * R + 3);
    k_map_band<<<cdiv(c3, 256) < 65535 ? cdiv(c3, 256) : 65535, 256, 0, st>>>(ft, nx, R, cube);
}

// The band cube ((2R+3)^3 float2, x fastest) as a 3D array behind a linear-filtering
// texture (unnormalised coordinates, zero border).  Release with free_cube_texture.
cudaError_t make_cube_texture(const float2* cube, int R, cudaStream_t st, cudaArray_t* arr,
                              cudaTextureObject_t* tex) {
    const int C = 2 * R + 3;
    cudaChannelFormatDesc fd = cudaCreateChannelDesc<float2>();
    cudaError_t e = cudaMalloc3DArray(arr, &fd, make_cudaExtent(C, C, C));
    if (e != cudaSuccess) return e;
    cudaMemcpy3DParms cp{};
    cp.srcPtr = make_cudaPitchedPtr(const_cast<float2*>(cube), (size_t)C * sizeof(float2), C, C);
    cp.dstArray = *arr;
    cp.extent = make_cudaExtent(C, C, C);
    cp.kind = cudaMemcpyDeviceToDevice;
    if ((e = cudaMemcpy3DAsync(&cp, st)) != cudaSuccess) return e;
    cudaResourceDesc rd{};
    rd.resType = cudaResourceTypeArray;
    rd.res.array.array = *arr;
    cudaTextureDesc td{};
    td.addressMode[0] = td.addressMode[1] = td.addressMode[2] = cudaAddressModeBorder;
    td.filterMode = cudaFilterModeLinear;
    td.readMode = cudaReadModeElementType;
    td.normalizedCoords = 0;
    return cudaCreateTextureObject(tex, &rd, &td, nullptr);
}

void free_cube_texture(cudaArray_t arr, cudaTextureObject_t tex) {
    if (tex) cudaDestroyTextureObject(tex);
    if (arr) cudaFreeArray(arr);
}

constexpr int SLICE_THREADS = 256;  // threads per section row
cudaError_t launch_slice_bf16(cudaTextureObject_t cube, int R, const int2* samples, int S, int KH,
                              const float* views, int nomr, float step, long n0, long count, void* B,
                              cudaStream_t st, const float2* lin, float sigma, float sc) {
    const float gk = (lin && sigma > 0.0f) ? 1.0f / (2.0f * sigma * sigma) : 0.0f;
    size_t sm = (size_t)S * sizeof(float2);
    cudaError_t e = allow_smem(k_slice_bf16, sm);
    if (e != cudaSuccess) return e;
    k_slice_bf16<<<(unsigned)count, SLICE_THREADS, sm, st>>>(cube, R, samples, S, KH, views, nomr, step,
                                                             host_angles().deg2rad, n0, (__nv_bfloat16*)B, lin, gk,
                                                             sc);
    return cudaGetLastError();
}

// a local grid's rows are short (a few thousand samples at sub-particle sizes): fewer
// threads per row keep the per-row norm reduction from dominating
constexpr int LOCAL_SLICE_THREADS = 64;
cudaError_t launch_slice_bf16_local(cudaTextureObject_t cube, int R, const int2* samples, int S, int Kpad,
                                    const float* centre, int m, float step, long count, void* B, cudaStream_t st,
                                    const float2* lin, float sigma, long lpitch, const float* pctf, float sc) {
    if (lpitch <= 0) lpitch = (long)(2 * m + 1) * (2 * m + 1) * (2 * m + 1);
    const float gk = (lin && sigma > 0.0f) ? 1.0f / (2.0f * sigma * sigma) : 0.0f;
    const long n = 2L * m + 1;
    if (Kpad / 2 <= LSR_THREADS * LSR_SPT && count % lpitch == 0 && n * n <= 65535 && count / lpitch <= 65535) {
        // the whole grid of each of count / lpitch particles: rows by (p, i, j) lines of omegas
        dim3 grid((unsigned)(n * n), (unsigned)(count / lpitch));
        auto rows = [&](auto spt) {
            k_slice_bf16_local_rows<decltype(spt)::value><<<grid, LSR_THREADS, sizeof(float) * 9 * (size_t)n, st>>>(
                cube, R, samples, S, Kpad, centre, m, step, host_angles().deg2rad, (__nv_bfloat162*)B, lin, gk, lpitch,
                pctf, sc);
            return cudaGetLastError();
        };
        // registers for the samples there are (24 grids of 25 steps a side: at maxR 32, 7 a thread, 1-2 % of the
        // form against 8)
        switch ((Kpad / 2 + LSR_THREADS - 1) / LSR_THREADS) {
            case 1: return rows(std::integral_constant<int, 1>());
            case 2: return rows(std::integral_constant<int, 2>());
            case 3: return rows(std::integral_constant<int, 3>());
            case 4: return rows(std::integral_constant<int, 4>());
            case 5: return rows(std::integral_constant<int, 5>());
            case 6: return rows(std::integral_constant<int, 6>());
            case 7: return rows(std::integral_constant<int, 7>());
            default: return rows(std::integral_constant<int, LSR_SPT>());
        }
    }
    size_t sm = (size_t)S * sizeof(float2);
    cudaError_t e = allow_smem(k_slice_bf16_local, sm);
    if (e != cudaSuccess) return e;
    for (long c0 = 0; c0 < count; c0 += 65535) {
        long nb = count - c0 < 65535 ? count - c0 : 65535;
        k_slice_bf16_local<<<(unsigned)nb, LOCAL_SLICE_THREADS, sm, st>>>(cube, R, samples, S, Kpad, centre, m, step,
                                                         host_angles().deg2rad, c0,
                                                         (__nv_bfloat162*)B + c0 * (Kpad / 2), lin, gk, lpitch,
                                                         pctf, sc);
    }
    return cudaGetLastError();
}

void launch_particle_norm(const float2* band, const float* ctf, Band bd, const int2* samples, int S,
                          int B, double* norm, cudaStream_t st, double2* pc, double* norm0, float* pctf) {
    k_particle_norm<<<B, 256, 0, st>>>(band, ctf, bd, samples, S, norm, pc, norm0, pctf);
}

void launch_build_a(const float2* band, const float* ctf, Band bd, const int2* samples, int S, int Kpad,
                    const float* origins, int O, const double* norm, int B, void* A, cudaStream_t st,
                    const float* poff) {
    const float tpn = 2.0f * host_angles().pi / (float)bd.nx;
    dim3 ga((O + AO - 1) / AO, B);
    const int sm = (int)(sizeof(float2) * AO * (3 * bd.max_r + 2));
    allow_smem(k_build_a, sm);
    k_build_a<<<ga, 256, sm, st>>>(band, ctf, bd, samples, S, Kpad, origins, O, poff, norm, tpn,
                                   (__nv_bfloat162*)A);
}

void launch_select_distinct(float* topv, const int* topi, int O, const int2* seg, int B, int max_tiles, int k, int* col,
                            int* origin, float* cc, cudaStream_t st) {
    const size_t sm = (size_t)O * max_tiles * (sizeof(float) + sizeof(int));
    if (sm <= 200 * 1024 && allow_smem(k_select_distinct<true>, sm) == cudaSuccess)
        k_select_distinct<true><<<B, 512, sm, st>>>(topv, topi, O, seg, k, col, origin, cc);
    else
        k_select_distinct<false><<<B, 512, 0, st>>>(topv, topi, O, seg, k, col, origin, cc);
}

long cc_fp64_scratch(int k, int B) { return (long)k * B * CC_SPLIT * 3; }

void launch_cc_fp64(const float2* cube, const double2* pcband, Band bd, const int2* samples, int S,
                    const float* cand, int k, int B, const double* pnorm, double* scratch, double* out,
                    cudaStream_t st, float sigma, const float* pctf, int cube_r, float sc) {
    dim3 g(k, B, CC_SPLIT);
    const size_t sm = sizeof(double2) * (3 * bd.max_r + 2);
    const double gk = sigma > 0.0f ? 1.0 / (2.0 * (double)sigma * (double)sigma) : 0.0;
    k_cc_fp64<<<g, 256, sm, st>>>(cube, pcband, bd, samples, S, cand, k, scratch, gk, pctf,
                                  cube_r < 0 ? bd.max_r : cube_r, (double)sc);
    k_cc_fp64_finish<<<(k * B + 127) / 128, 128, 0, st>>>(scratch, k * B, CC_SPLIT, pnorm, k, out);
}

}  // namespace cryoim
