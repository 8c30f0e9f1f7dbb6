// Vector kernels on FP64 complex columns with fixed-order two-stage reductions, so that
// norms and dot products repeat bit for bit from run to run (the reference's results do
// not depend on its thread count, numerics/parallel.rs).
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace tcu {

constexpr int RG = 256;  // partial sums per reduction (grid size of stage 1)
constexpr int MAX_ROWS = 65535;  // of a grid: columns per launch of stage 1

__device__ __forceinline__ double block_sum(double v, double* sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) s += sh[q];
    __syncthreads();
    return s;  // valid in thread 0
}

// stage 1: partial[c * RG + b] = sum over the fixed slice of column c of f(i)
__global__ void norm_stage1(const cplx* __restrict__ x, size_t n, double* __restrict__ partial) {
    __shared__ double sh[32];
    int c = blockIdx.y, b = blockIdx.x;
    const cplx* xc = x + (size_t)c * n;
    double s = 0.0;
    for (size_t i = (size_t)b * blockDim.x + threadIdx.x; i < n; i += (size_t)RG * blockDim.x) s += cabs2(xc[i]);
    s = block_sum(s, sh);
    if (threadIdx.x == 0) partial[c * RG + b] = s;
}
__global__ void sum_stage2(const double* __restrict__ partial, int ncol, double* __restrict__ out, int do_sqrt) {
    __shared__ double sh[32];
    int c = blockIdx.x;
    double s = partial[(size_t)c * RG + threadIdx.x];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) out[c] = do_sqrt ? sqrt(s) : s;
}
void vec_norms(const cplx* x, size_t n, int ncol, double* out_dev, double* partial, cudaStream_t st) {
    for (int c = 0; c < ncol; c += MAX_ROWS)
        norm_stage1<<<dim3(RG, std::min(MAX_ROWS, ncol - c)), 256, 0, st>>>(x + c * n, n, partial + (size_t)c * RG);
    sum_stage2<<<ncol, RG, 0, st>>>(partial, ncol, out_dev, 1);
}

__global__ void rdot_stage1(const cplx* __restrict__ a, const cplx* __restrict__ b, size_t n, double* __restrict__ partial) {
    __shared__ double sh[32];
    int c = blockIdx.y, bl = blockIdx.x;
    const cplx* ac = a + (size_t)c * n;
    const cplx* bc = b + (size_t)c * n;
    double s = 0.0;
    for (size_t i = (size_t)bl * blockDim.x + threadIdx.x; i < n; i += (size_t)RG * blockDim.x)
        s += ac[i].x * bc[i].x + ac[i].y * bc[i].y;
    s = block_sum(s, sh);
    if (threadIdx.x == 0) partial[c * RG + bl] = s;
}
void vec_real_dots(const cplx* a, const cplx* b, size_t n, int ncol, double* out_dev, double* partial,
                   cudaStream_t st) {
    for (int c = 0; c < ncol; c += MAX_ROWS)
        rdot_stage1<<<dim3(RG, std::min(MAX_ROWS, ncol - c)), 256, 0, st>>>(a + c * n, b + c * n, n,
                                                                          partial + (size_t)c * RG);
    sum_stage2<<<ncol, RG, 0, st>>>(partial, ncol, out_dev, 0);
}

// complex dots out[i] = sum conj(V_i) w, i < nv
__global__ void dots_stage1(const cplx* __restrict__ V, size_t ldv, const cplx* __restrict__ w, size_t n,
                            cplx* __restrict__ partial) {
    __shared__ double sh[32];
    int i = blockIdx.y, b = blockIdx.x;
    const cplx* v = V + (size_t)i * ldv;
    double sr = 0.0, si = 0.0;
    for (size_t q = (size_t)b * blockDim.x + threadIdx.x; q < n; q += (size_t)RG * blockDim.x) {
        cplx a = v[q], c = w[q];
        sr += a.x * c.x + a.y * c.y;
        si += a.x * c.y - a.y * c.x;
    }
    sr = block_sum(sr, sh);
    si = block_sum(si, sh);
    if (threadIdx.x == 0) partial[i * RG + b] = mk(sr, si);
}
// w -= V h with h_i the sum of column i's partial dots, which every CTA forms itself in one fixed order
// (a warp per column); the first CTA stores h. NORM: npart[b] = this CTA's share of |w|^2.
template <bool NORM>
__global__ void __launch_bounds__(256) gram_schmidt_kernel(cplx* __restrict__ w, const cplx* __restrict__ V,
                                                           size_t ldv, int nv, const cplx* __restrict__ partial,
                                                           size_t n, cplx* __restrict__ h_out,
                                                           double* __restrict__ npart) {
    constexpr int GROUP = 64;  // columns at a time
    __shared__ cplx h[GROUP];
    __shared__ double sh[32];
    const int lane = threadIdx.x & 31;
    double norm = 0.0;
    for (int i0 = 0; i0 < nv; i0 += GROUP) {
        const int cols = min(GROUP, nv - i0);
        if (i0 > 0) __syncthreads();  // h of the columns before is used up
        for (int i = threadIdx.x >> 5; i < cols; i += 8) {
            cplx s = mk(0.0, 0.0);
#pragma unroll
            for (int q = 0; q < RG / 32; ++q) s = cadd(s, partial[(size_t)(i0 + i) * RG + q * 32 + lane]);
            for (int o = 16; o > 0; o >>= 1) {
                s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
                s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
            }
            if (lane == 0) {
                h[i] = s;
                if (blockIdx.x == 0) h_out[i0 + i] = s;
            }
        }
        __syncthreads();
        for (size_t q = (size_t)blockIdx.x * 256 + threadIdx.x; q < n; q += (size_t)gridDim.x * 256) {
            cplx acc = w[q];
            for (int i = 0; i < cols; ++i) {
                const cplx hv = h[i], v = V[(size_t)(i0 + i) * ldv + q];
                acc.x -= hv.x * v.x - hv.y * v.y;
                acc.y -= hv.x * v.y + hv.y * v.x;
            }
            w[q] = acc;
            if (NORM && i0 + cols == nv) norm += cabs2(acc);
        }
    }
    if (NORM) {
        norm = block_sum(norm, sh);
        if (threadIdx.x == 0) npart[blockIdx.x] = norm;
    }
}
// next = w / |w| and the norm itself (by the first CTA) from the partial sums of |w|^2
__global__ void __launch_bounds__(256) normalize_kernel(const cplx* __restrict__ w, const double* __restrict__ npart,
                                                        int parts, size_t n, cplx* __restrict__ next,
                                                        double* __restrict__ norm_out) {
    __shared__ double sh[32];
    __shared__ double total;
    double s = 0.0;
    for (int b = threadIdx.x; b < parts; b += 256) s += npart[b];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) {
        total = sqrt(s);
        if (blockIdx.x == 0) *norm_out = total;
    }
    __syncthreads();
    const double inv = 1.0 / total;
    for (size_t q = (size_t)blockIdx.x * 256 + threadIdx.x; q < n; q += (size_t)gridDim.x * 256)
        next[q] = cscale(w[q], inv);
}
// One Arnoldi step after the operator: w made orthogonal to V_0 .. V_{nv-1} by two classical Gram-Schmidt
// passes, next = w / |w| (not finite where the norm is 0). coef: the coefficients of both passes (nv each),
// then the norm as the real part of one more entry. Latency bounds it below some hundred thousand modes: five
// launches and one copy to the host, where the sums had their own launches and each pass and the norm were
// copied and waited for (11 launches, three waits): 300 spheres at lmax 6 (13 steps) 7.57 -> 7.15 ms a solve.
void vec_arnoldi_step(const cplx* V, size_t ldv, int nv, cplx* w, size_t n, cplx* next, cplx* coef, cplx* partial,
                      double* npart, cudaStream_t st) {
    const int ctas = (int)std::min<size_t>((n + 255) / 256, ARNOLDI_PARTS);
    dots_stage1<<<dim3(RG, nv), 256, 0, st>>>(V, ldv, w, n, partial);
    gram_schmidt_kernel<false><<<ctas, 256, 0, st>>>(w, V, ldv, nv, partial, n, coef, nullptr);
    dots_stage1<<<dim3(RG, nv), 256, 0, st>>>(V, ldv, w, n, partial);
    gram_schmidt_kernel<true><<<ctas, 256, 0, st>>>(w, V, ldv, nv, partial, n, coef + nv, npart);
    normalize_kernel<<<ctas, 256, 0, st>>>(w, npart, ctas, n, next, (double*)(coef + 2 * nv));
}
__global__ void lincomb_kernel(cplx* __restrict__ x, const cplx* __restrict__ V, size_t ldv, int nv,
                               const cplx* __restrict__ g, size_t n) {
    size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    cplx acc = x[q];
    for (int i = nv - 1; i >= 0; --i) cfma(acc, g[i], V[(size_t)i * ldv + q]);
    x[q] = acc;
}
void vec_lincomb(cplx* x, const cplx* V, size_t ldv, int nv, const cplx* g_dev, size_t n, cudaStream_t st) {
    lincomb_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(x, V, ldv, nv, g_dev, n);
}
__global__ void axpy_kernel(cplx* __restrict__ y, const cplx* __restrict__ x, size_t total) {
    size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < total) y[q] = cadd(y[q], x[q]);
}
void vec_axpy(cplx* y, const cplx* x, size_t n, int ncol, cudaStream_t st) {
    size_t t = n * ncol;
    axpy_kernel<<<(unsigned)((t + 255) / 256), 256, 0, st>>>(y, x, t);
}
__global__ void sub_kernel(cplx* o, const cplx* a, const cplx* b, size_t total) {  // o may alias a or b
    size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < total) o[q] = csub(a[q], b[q]);
}
void vec_sub(cplx* out, const cplx* a, const cplx* b, size_t n, int ncol, cudaStream_t st) {
    size_t t = n * ncol;
    sub_kernel<<<(unsigned)((t + 255) / 256), 256, 0, st>>>(out, a, b, t);
}
__global__ void scale_kernel(cplx* o, const cplx* x, size_t n, double s) {  // o may alias x
    size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) o[q] = cscale(x[q], s);
}
void vec_scale_copy(cplx* out, const cplx* x, size_t n, double s, cudaStream_t st) {
    scale_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, x, n, s);
}

}  // namespace tcu
