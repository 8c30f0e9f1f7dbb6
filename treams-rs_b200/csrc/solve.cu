// Triangular solves with the LU factors (FP64 or FP32 storage, FP64 arithmetic).
//
// After a factorization the diagonal 64 x 64 blocks of L (unit lower) and U (upper) are
// inverted once, in FP64 (tri_block_inverse_kernel). A forward or backward sweep is then a
// chain of block steps, each one launch: every CTA forms x_b = D_b^-1 r_b (a dense 64 x 64
// product, no serial recurrence) and subtracts the block column times x_b from its share
// of the remaining rows (read once, coalesced along the column). The right-hand side is
// updated in place while the block solutions go to a separate array, so no CTA reads a
// row that another CTA writes in the same step.
//
// The default is one persistent kernel per triangle instead (sweep_kernel), which also serves the
// adjoint solves; the block steps stay for TCU_SOLVE=steps and for a refused cooperative launch.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <string>

#include "common.cuh"
#include "kernels.h"

namespace tcu {

constexpr int SB = 64;      // diagonal block size
constexpr int SMAXC = 8;    // right-hand sides per block step
enum SweepOp { SW_L, SW_U, SW_UH, SW_LH };

template <typename C>
__device__ __forceinline__ double2 to_d2(C v) {
    return make_double2((double)v.x, (double)v.y);
}

// One CTA per diagonal block and triangle (blockIdx.y: 0 L, unit lower; 1 U): its FP64 inverse, out
// column-major 64 x 64 per block (identity beyond the matrix edge), all of L then all of U. U is
// turned into a lower triangle by reversing both indices. The four 16 x 16 diagonal blocks are
// inverted by a warp each (a lane per column of the inverse, a right-looking substitution), then
// neighbouring inverses are joined, [A 0; B C]^-1 = [A^-1 0; -C^-1 B A^-1 C^-1], at 16 and at 32 rows.
// One column after the other took 64 dependent steps with two barriers and 64 threads at work:
// 95 us for each triangle whatever n, against 28 for both.
constexpr int TBI_LD = SB + 1;
template <typename C>
__global__ void __launch_bounds__(256) tri_block_inverse_kernel(const C* __restrict__ A, size_t lda, int n,
                                                                double2* __restrict__ out) {
    extern __shared__ double2 tbi_smem[];
    double2* M = tbi_smem;                  // M[i * TBI_LD + k], lower triangle
    double2* T = tbi_smem + SB * TBI_LD;    // 32 x 32 (two 16 x 16 at the first level)
    const bool upper = blockIdx.y == 1;
    const int b0 = blockIdx.x * SB, bw = min(SB, n - b0), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto place = [&](int i) { return upper ? SB - 1 - i : i; };  // index in the matrix -> in M
    for (int idx = tid; idx < SB * SB; idx += blockDim.x) {
        const int i = idx % SB, k = idx / SB;  // matrix row and column inside the block
        const bool in = upper ? i <= k : i > k;
        double2 v = make_double2(0.0, 0.0);
        if (in && i < bw && k < bw) v = to_d2(A[(size_t)(b0 + k) * lda + b0 + i]);
        if (i == k && (!upper || i >= bw)) v = make_double2(1.0, 0.0);
        M[place(i) * TBI_LD + place(k)] = v;
    }
    __syncthreads();
    if (warp < SB / 16 && lane < 16) {
        const int o = warp * 16;
        double2 x[16], inv[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            x[i] = make_double2(i == lane ? 1.0 : 0.0, 0.0);
            inv[i] = cinv(M[(o + i) * TBI_LD + o + i]);
        }
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            x[k] = cmul(x[k], inv[k]);
#pragma unroll
            for (int i = k + 1; i < 16; ++i) cfma(x[i], cneg(M[(o + i) * TBI_LD + o + k]), x[k]);
        }
        __syncwarp(0xffffu);  // every lane has read the block
#pragma unroll
        for (int i = 0; i < 16; ++i) M[(o + i) * TBI_LD + o + lane] = x[i];
    }
    __syncthreads();
    for (int s = 16; s < SB; s *= 2) {
        const int pairs = SB / (2 * s);
        for (int idx = tid; idx < pairs * s * s; idx += blockDim.x) {  // T = B A^-1
            const int q = idx / (s * s), e = idx - q * s * s, k = e % s, i = e / s, a0 = 2 * s * q, c0 = a0 + s;
            double2 t = make_double2(0.0, 0.0);
            for (int m = k; m < s; ++m) cfma(t, M[(c0 + i) * TBI_LD + a0 + m], M[(a0 + m) * TBI_LD + a0 + k]);
            T[idx] = t;
        }
        __syncthreads();
        for (int idx = tid; idx < pairs * s * s; idx += blockDim.x) {  // -C^-1 T over B
            const int q = idx / (s * s), e = idx - q * s * s, k = e % s, i = e / s, a0 = 2 * s * q, c0 = a0 + s;
            double2 t = make_double2(0.0, 0.0);
            for (int m = 0; m <= i; ++m) cfma(t, M[(c0 + i) * TBI_LD + c0 + m], T[q * s * s + m * s + k]);
            M[(c0 + i) * TBI_LD + a0 + k] = cneg(t);
        }
        __syncthreads();
    }
    double2* o = out + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * SB * SB;
    for (int idx = tid; idx < SB * SB; idx += blockDim.x) {
        const int i = idx % SB, k = idx / SB;
        const bool in = upper ? i <= k : i >= k;
        o[idx] = in ? M[place(i) * TBI_LD + place(k)] : make_double2(0.0, 0.0);
    }
}

__global__ void gather_kernel(const double2* __restrict__ x, double2* __restrict__ y, const int* __restrict__ perm,
                              int n, int ncol) {
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (size_t)n * ncol) return;
    int c = (int)(t / n), i = (int)(t % n);
    y[t] = x[(size_t)c * n + perm[i]];
}

// One block step: sol_b = Dinv_b r_b; r[other rows] -= A[other rows, block] sol_b.
// Every load that does not depend on the block solution (the Dinv quarter of each thread,
// the right-hand side block, the first half of the thread's row of the block column) is
// issued up front, so a step costs about two memory round trips.
template <typename C, bool LOWER, int NC>
__global__ void __launch_bounds__(256) trsv_inv_step_kernel(const C* __restrict__ A, size_t lda, int n, int b0, int bw,
                                                            const double2* __restrict__ dinv, double2* __restrict__ r,
                                                            double2* __restrict__ sol) {
    __shared__ double2 rb[NC][SB];
    __shared__ double2 part[4][NC][SB];
    __shared__ double2 xb[NC][SB];
    constexpr int KH = 16;  // preloaded first chunk of the block column
    // Programmatic dependent launch: the next step may start its read-only preloads (its
    // Dinv quarter and block column) while this one runs; it reads the right-hand side only
    // after griddepcontrol.wait, i.e. after this grid has completed and its writes are visible.
    asm volatile("griddepcontrol.launch_dependents;");
    const int tid = threadIdx.x;
    const int i = tid % SB, kq = tid / SB;  // Dinv row and K quarter
    double2 d[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) d[u] = dinv[(size_t)(kq * 16 + u) * SB + i];
    const int lo = LOWER ? b0 + bw : 0, hi = LOWER ? n : b0;
    const int row = lo + blockIdx.x * blockDim.x + tid;
    const bool has_row = row < hi;
    C av[KH];
#pragma unroll
    for (int u = 0; u < KH; ++u) {
        if (has_row && u < bw)
            av[u] = A[(size_t)(b0 + u) * lda + row];
        else {
            av[u].x = 0;
            av[u].y = 0;
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int idx = tid; idx < SB * NC; idx += blockDim.x) {
        int ii = idx % SB, c = idx / SB;
        rb[c][ii] = ii < bw ? r[(size_t)c * n + b0 + ii] : make_double2(0.0, 0.0);
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        double2 acc = make_double2(0.0, 0.0);
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            double2 v = rb[c][kq * 16 + u];
            acc.x += d[u].x * v.x - d[u].y * v.y;
            acc.y += d[u].x * v.y + d[u].y * v.x;
        }
        part[kq][c][i] = acc;
    }
    __syncthreads();
    for (int idx = tid; idx < SB * NC; idx += blockDim.x) {
        int ii = idx % SB, c = idx / SB;
        double2 s = part[0][c][ii];
#pragma unroll
        for (int q = 1; q < 4; ++q) {
            s.x += part[q][c][ii].x;
            s.y += part[q][c][ii].y;
        }
        xb[c][ii] = s;
    }
    __syncthreads();
    if (blockIdx.x == 0)
        for (int idx = tid; idx < bw * NC; idx += blockDim.x) {
            int ii = idx % bw, c = idx / bw;
            sol[(size_t)c * n + b0 + ii] = xb[c][ii];
        }
    // rows beyond the first pass of the grid (n > 148 * 256) load their first chunk here too
    for (int rr = row; rr < hi; rr += gridDim.x * blockDim.x) {
        const bool first = rr == row;
        double2 acc[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[c] = make_double2(0, 0);
#pragma unroll 1
        for (int kc = 0; kc < SB; kc += KH) {
            C v[KH];
#pragma unroll
            for (int u = 0; u < KH; ++u) {
                if (kc == 0 && first)
                    v[u] = av[u];
                else if (kc + u < bw)
                    v[u] = A[(size_t)(b0 + kc + u) * lda + rr];
                else {
                    v[u].x = 0;
                    v[u].y = 0;
                }
            }
#pragma unroll
            for (int u = 0; u < KH; ++u) {
                double lr = v[u].x, li = v[u].y;
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    double2 x = xb[c][kc + u];
                    acc[c].x += lr * x.x - li * x.y;
                    acc[c].y += lr * x.y + li * x.x;
                }
            }
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            double2* p = r + (size_t)c * n + rr;
            double2 v = *p;
            v.x -= acc[c].x;
            v.y -= acc[c].y;
            *p = v;
        }
    }
}

// ---- persistent sweeps -----------------------------------------------------------------
// One cooperative launch per triangle and direction. Grid (G, chunks): chunk y solves NC of the
// right-hand-side columns, its CTA x takes the block rows x, x + G, ... in solve order. A block
// row t accumulates s = b_t - sum_(j < t) T_tj y_j tile by tile (64 x 64, a fixed order) and ends
// with y_t = Dinv_t s. The block solutions are their own completion flags: the solution array
// starts as all-ones bit patterns (a NaN no computation produces), a consumer polls the entries it
// needs until both halves differ, so a step of the chain costs one store and one load through L2
// and no fence, flag or second read.
//
// This kernel serves one and two columns, where the chain of n / 64 dependent steps bounds it (a step:
// poll, one tile, reduction, the diagonal product: 1.4 us at one column, 1.8 at two) or, with few CTAs, its
// 0.8 us a tile.
// Tiles arrive by cp.async (3 stages of 32 KB for FP32 factors, 2 of 64 KB for FP64), padded to 65
// rows so that the transposed reads of the adjoint sweeps have no bank conflicts either.
// Measured against one launch per 8 columns with completion flags behind fences: one column
// 2.6 -> 1.5 us per block step.
// Every poll is bounded (4 s): status 8 and all CTAs return.
constexpr int SW_THREADS = 512;
constexpr int SW_Q = SW_THREADS / SB;  // contraction groups of a tile
constexpr int SW_K = SB / SW_Q;        // contraction entries per thread and tile
constexpr int SW_LD = SB + 1;
constexpr int SW_MAXC = 2;             // columns per chunk

__device__ __forceinline__ unsigned long long sw_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ double2 sw_load(const double2* p) {
    double2 v;
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void sw_store(double2* p, double2 v) {
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ bool sw_empty(double v) { return __double_as_longlong(v) == -1ll; }
__device__ __forceinline__ double sw_value(double v) {  // never the empty pattern
    return sw_empty(v) ? __longlong_as_double(0x7ff8000000000000ll) : v;
}
// Polls one entry until it is written; false (and status 8) after 4 s or when another wait gave up.
__device__ __forceinline__ bool sw_wait(const double2* p, double2& v, int* status,
                                        unsigned long long limit_ns = 4000000000ull) {
    unsigned long long t0 = 0;
    for (unsigned spins = 1; sw_empty(v.x) || sw_empty(v.y); ++spins) {
        if ((spins & 255u) == 0) {  // the clock is read on long waits only: it costs about a microsecond
            const unsigned long long now = sw_ns();
            if (!t0) t0 = now;
            if (*(volatile int*)status == 8 || now - t0 > limit_ns) {
                atomicExch(status, 8);
                return false;
            }
        }
        v = sw_load(p);
    }
    return true;
}
template <typename C>
__device__ __forceinline__ void sw_copy(C* smem, const C* gmem, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int sz = valid ? (int)sizeof(C) : 0;
    if (sizeof(C) == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(sz) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(s), "l"(gmem), "r"(sz) : "memory");
}

template <typename C>
constexpr int sw_stages() {
    return sizeof(C) == 8 ? 3 : 2;
}
template <typename C>
constexpr size_t sweep_smem_bytes(int nc) {
    return (size_t)sw_stages<C>() * SB * SW_LD * sizeof(C) + (size_t)(2 + SW_Q + 1) * nc * SB * sizeof(double2);
}

// sol = op(T)^-1 rhs for ncol columns (n x ncol, sol preset to the empty pattern) with T the unit
// lower or the upper triangle of the factor. OP: SW_L and SW_UH run down the block rows (L y = b,
// U^H y = b), SW_U and SW_LH up. clear: presets the solution array of the next sweep.
template <typename C, int OP, int NC>
__global__ void __launch_bounds__(SW_THREADS, 1)
    sweep_kernel(const C* __restrict__ A, size_t lda, int n, int nb, int ncol, const double2* __restrict__ dinv,
                 const double2* __restrict__ rhs, double2* sol, double2* clear, int* status) {
    constexpr bool DOWN = OP == SW_L || OP == SW_UH, ADJ = OP == SW_UH || OP == SW_LH;
    constexpr int ST = sw_stages<C>();
    extern __shared__ __align__(16) unsigned char sw_smem[];
    double2* ys = reinterpret_cast<double2*>(sw_smem);  // [2][NC][SB]
    double2* part = ys + 2 * NC * SB;                   // [SW_Q][NC][SB]
    double2* sb = part + SW_Q * NC * SB;                // [NC][SB]
    C* tiles = reinterpret_cast<C*>(sb + NC * SB);      // [ST][SB][SW_LD]: column k at k * SW_LD
    const int tid = threadIdx.x, o = tid % SB, q = tid / SB;
    const int col0 = blockIdx.y * NC, nc = min(NC, ncol - col0);
    rhs += (size_t)col0 * n;
    sol += (size_t)col0 * n;
    if (clear) {
        clear += (size_t)col0 * n;
        const double e = __longlong_as_double(-1ll);
        for (size_t i = (size_t)blockIdx.x * SW_THREADS + tid; i < (size_t)nc * n; i += (size_t)gridDim.x * SW_THREADS)
            clear[i] = make_double2(e, e);
    }
    auto blk = [&](int t) { return DOWN ? t : nb - 1 - t; };
    // this thread's entry (column q, row o of a block) of the solution and right-hand-side blocks
    const bool entry = q < nc;
    for (int t = blockIdx.x; t < nb; t += gridDim.x) {
        const int bi = blk(t), r0 = bi * SB;
        double2 d[SW_K], rb = make_double2(0.0, 0.0);
#pragma unroll
        for (int u = 0; u < SW_K; ++u) {
            const size_t at = ADJ ? (size_t)o * SB + q * SW_K + u : (size_t)(q * SW_K + u) * SB + o;
            d[u] = __ldg(&dinv[(size_t)bi * SB * SB + at]);
        }
        if (entry && r0 + o < n) rb = rhs[(size_t)q * n + r0 + o];
        auto load_tile = [&](int ts) {  // T_(t, ts), or the tile it is the adjoint of
            if (ts < t) {
                const int ri = ADJ ? blk(ts) * SB : r0, ci = ADJ ? r0 : blk(ts) * SB;
                C* dst = tiles + (size_t)(ts % ST) * SB * SW_LD;
                const bool rok = ri + o < n;
#pragma unroll
                for (int u = 0; u < SW_K; ++u) {
                    const int k = q + SW_Q * u;
                    const bool ok = rok && ci + k < n;
                    sw_copy(&dst[k * SW_LD + o], ok ? &A[(size_t)(ci + k) * lda + ri + o] : A, ok);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int s = 0; s < ST - 1; ++s) load_tile(s);
        double2 acc[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[c] = make_double2(0.0, 0.0);
        const double2* yp = sol + (size_t)(entry ? q : 0) * n + o;
        double2 pre = make_double2(0.0, 0.0);
        auto in_range = [&](int ts) { return entry && blk(ts) * SB + o < n; };
        if (t > 0 && in_range(0)) pre = sw_load(yp + blk(0) * SB);
        for (int ts = 0; ts < t; ++ts) {
            int gave_up = 0;
            if (q < NC) {
                if (in_range(ts))
                    gave_up = !sw_wait(yp + blk(ts) * SB, pre, status);
                else
                    pre = make_double2(0.0, 0.0);
                ys[((ts & 1) * NC + q) * SB + o] = pre;
            }
            asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
            // tile ts and y_ts are in shared memory; the stage of tile ts - 1 is free
            if (__syncthreads_or(gave_up)) {
                asm volatile("cp.async.wait_all;" ::: "memory");
                return;
            }
            load_tile(ts + ST - 1);
            if (ts + 1 < t && in_range(ts + 1)) pre = sw_load(yp + blk(ts + 1) * SB);
            const C* tile = tiles + (size_t)(ts % ST) * SB * SW_LD;
            const double2* yv = ys + (ts & 1) * NC * SB + q * SW_K;
#pragma unroll
            for (int u = 0; u < SW_K; ++u) {
                const double2 v = to_d2(ADJ ? tile[o * SW_LD + q * SW_K + u] : tile[(q * SW_K + u) * SW_LD + o]);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (ADJ)
                        cfma_conj(acc[c], v, yv[c * SB + u]);
                    else
                        cfma(acc[c], v, yv[c * SB + u]);
                }
            }
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) part[(q * NC + c) * SB + o] = acc[c];
        __syncthreads();
        if (q < NC) {
            double2 s = rb;
#pragma unroll
            for (int g = 0; g < SW_Q; ++g) s = csub(s, part[(g * NC + q) * SB + o]);
            sb[q * SB + o] = s;
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            double2 y = make_double2(0.0, 0.0);
#pragma unroll
            for (int u = 0; u < SW_K; ++u) {
                if (ADJ)
                    cfma_conj(y, d[u], sb[c * SB + q * SW_K + u]);
                else
                    cfma(y, d[u], sb[c * SB + q * SW_K + u]);
            }
            part[(q * NC + c) * SB + o] = y;
        }
        __syncthreads();
        if (entry && r0 + o < n) {
            double2 y = part[q * SB + o];
#pragma unroll
            for (int g = 1; g < SW_Q; ++g) y = cadd(y, part[(g * NC + q) * SB + o]);
            sw_store(&sol[(size_t)q * n + r0 + o], make_double2(sw_value(y.x), sw_value(y.y)));
        }
        __syncthreads();  // part and the tile stages are free for the next block row
    }
}

// ---- persistent sweeps on the FP64 tensor cores -------------------------------------------
// The same chain for three and more columns, in chunks of four: the 4 complex columns are the 8 real columns
// [re y | im y] of m8n8k4 products, acc1 = Re T [re y | im y] and acc2 = Im T [re y | im y], two products per 8
// rows and 4 entries. Roles instead of CTA-wide barriers: 8 product warps (a row octet each, so no
// sums cross warps), four that stream the tiles into a ring (16-byte copies; one bulk copy per column of a tile
// took 2.3 us a tile whatever its size), and four that poll the block solutions, a column each, and lay them out as fragments in a second ring.
// Bound by the FP64 rate, 0.53 us a tile (1.0 measured), with many block rows per CTA; by the chain (poll, tile,
// diagonal product, 2.2 us) with few. us per triangle against sweep_kernel at 4 columns a chunk, whose
// 8-byte copies, conversions and CTA barrier took 1.9 us a tile: n = 9600, 17 columns, FP32 factor 840 -> 485,
// 64 columns 2305 -> 1230; n = 1920, 96 columns, FP64 190 -> 105; n = 24576, 3 columns, FP32 1140 -> 935.
// Several chains of products per warp or twice the warps with half of the entries each: no faster.
// Tile columns are SD_LD entries apart, so that the fragments of a tile and of its adjoint (FP64: of the one
// the sweep reads) come without bank conflicts. n is even (checked by the launch), so that every column of
// a tile starts on 16 bytes and is a multiple of them long.
constexpr int SD_COLS = 4, SD_WARPS = 8, SD_LOADERS = 4, SD_THREADS = (SD_WARPS + SD_COLS + SD_LOADERS) * 32;
template <typename C>
constexpr int sd_stages() {
    return sizeof(C) == 8 ? 5 : 3;
}
template <typename C>
constexpr int sd_yring() {
    return sizeof(C) == 8 ? 4 : 3;
}
template <typename C, bool ADJ>
constexpr int sd_ld() {
    return sizeof(C) == 8 || ADJ ? 68 : 66;
}
template <typename C, bool ADJ>
constexpr size_t sd_smem_bytes() {
    return (size_t)sd_stages<C>() * SB * sd_ld<C, ADJ>() * sizeof(C) + (size_t)(sd_yring<C>() + 2) * 512 * sizeof(double);
}
__device__ __forceinline__ void sd_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(bar)), "r"(count)
                 : "memory");
}
__device__ __forceinline__ void sd_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"((unsigned)__cvta_generic_to_shared(bar)) : "memory");
}
__device__ __forceinline__ bool sd_try(uint64_t* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"((unsigned)__cvta_generic_to_shared(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// false when the CTA has given up or after 5 s (a poll gives up after 4)
__device__ __forceinline__ bool sd_wait(uint64_t* bar, unsigned parity, volatile int* gave_up,
                                        unsigned long long limit_ns = 5000000000ull) {
    if (sd_try(bar, parity)) return true;
    unsigned long long t0 = 0;
    for (unsigned it = 1;; ++it) {
        if (sd_try(bar, parity)) return true;
        if ((it & 63u) == 0) {
            if (*gave_up) return false;
            const unsigned long long now = sw_ns();
            if (!t0) t0 = now;
            if (now - t0 > limit_ns) {
                *gave_up = 1;
                return false;
            }
        }
    }
}
__device__ __forceinline__ void sd_dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}
// acc1, acc2 -> this lane's two entries of the complex product: columns 2 q, 2 q + 1 of [re | im], q = lane % 4
template <bool ADJ>
__device__ __forceinline__ void sd_join(const double (&a1)[2], const double (&a2)[2], int q, double (&v)[2]) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const double o = __shfl_xor_sync(0xffffffffu, a2[u], 2);
        v[u] = ((q < 2) != ADJ) ? a1[u] - o : a1[u] + o;
    }
}

template <typename C, int OP>
__global__ void __launch_bounds__(SD_THREADS, 1)
    sweep_dmma_kernel(const C* __restrict__ A, size_t lda, int n, int nb, int ncol, const double2* __restrict__ dinv,
                      const double2* __restrict__ rhs, double2* sol, double2* clear, int* status) {
    constexpr bool DOWN = OP == SW_L || OP == SW_UH, ADJ = OP == SW_UH || OP == SW_LH;
    constexpr int ST = sd_stages<C>(), YR = sd_yring<C>(), LD = sd_ld<C, ADJ>(), TILE = SB * LD;
    extern __shared__ __align__(128) unsigned char sd_smem[];
    C* tiles = reinterpret_cast<C*>(sd_smem);                    // [ST][SB][LD]: column k at k * LD
    double* ys = reinterpret_cast<double*>(tiles + ST * TILE);   // [YR][16][32]: fragments of y
    double* ss = ys + YR * 512;                            // [2][16][32]: fragments of a block's sums
    __shared__ __align__(8) uint64_t bars[2 * ST + 2 * YR];
    __shared__ int s_gave_up;
    uint64_t *full = bars, *empty = bars + ST, *yfull = bars + 2 * ST, *yempty = yfull + YR;
    volatile int* gave_up = &s_gave_up;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int col0 = blockIdx.y * SD_COLS, nc = min(SD_COLS, ncol - col0);
    rhs += (size_t)col0 * n;
    sol += (size_t)col0 * n;
    if (clear) {
        clear += (size_t)col0 * n;
        const double e = __longlong_as_double(-1ll);
        for (size_t i = (size_t)blockIdx.x * SD_THREADS + tid; i < (size_t)nc * n; i += (size_t)gridDim.x * SD_THREADS)
            clear[i] = make_double2(e, e);
    }
    if (tid == 0) {
        for (int i = 0; i < ST; ++i) {
            sd_init(full + i, 32 * SD_LOADERS);
            sd_init(empty + i, SD_WARPS);
        }
        for (int i = 0; i < YR; ++i) {
            sd_init(yfull + i, 32 * SD_COLS);
            sd_init(yempty + i, SD_WARPS);
        }
        s_gave_up = 0;
    }
    __syncthreads();
    auto blk = [&](int t) { return DOWN ? t : nb - 1 - t; };
    if (warp >= SD_WARPS + SD_COLS) {  // tiles
        constexpr int PER = 16 / sizeof(C), COLS = 32 * PER == SB ? 1 : 2;  // entries a copy, instructions a column
        const int lw = warp - SD_WARPS - SD_COLS;
        int seq = 0;
        bool ok = true;
        for (int t = blockIdx.x; ok && t < nb; t += gridDim.x)
            for (int ts = 0; ts < t; ++ts, ++seq) {
                const int s = seq % ST;
                if (!(ok = __all_sync(0xffffffffu, sd_wait(empty + s, ((seq / ST) & 1) ^ 1, gave_up)))) break;
                const int ri = (ADJ ? blk(ts) : blk(t)) * SB, ci = (ADJ ? blk(t) : blk(ts)) * SB;
                C* dst = tiles + s * TILE;
#pragma unroll 8
                for (int k = lw; k < SB; k += SD_LOADERS)
#pragma unroll
                    for (int h = 0; h < COLS; ++h) {
                        const int row = (h * 32 + lane) * PER;
                        const bool in = ci + k < n && ri + row < n;  // n is even: both entries of a copy or none
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                                         (unsigned)__cvta_generic_to_shared(dst + k * LD + row)),
                                     "l"(in ? A + (size_t)(ci + k) * lda + ri + row : A), "r"(in ? 16 : 0)
                                     : "memory");
                    }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(
                                 (unsigned)__cvta_generic_to_shared(full + s))
                             : "memory");
            }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp >= SD_WARPS) {  // block solutions: a column each, two entries a lane
        const int c = warp - SD_WARPS;
        const double2* yp = sol + (size_t)min(c, nc - 1) * n;
        int seq = 0;
        bool ok = true;
        double2 pre[2];
        auto fetch = [&](int ts) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int at = blk(ts) * SB + lane + 32 * u;
                pre[u] = c < nc && at < n ? sw_load(yp + at) : make_double2(0.0, 0.0);
            }
        };
        for (int t = blockIdx.x; ok && t < nb; t += gridDim.x) {
            if (t > 0) fetch(0);
            for (int ts = 0; ts < t; ++ts, ++seq) {
                const int s = seq % YR;
                unsigned long long t0 = 0;
                for (unsigned spins = 1;; ++spins) {
                    const bool e0 = sw_empty(pre[0].x) || sw_empty(pre[0].y), e1 = sw_empty(pre[1].x) || sw_empty(pre[1].y);
                    if (!__any_sync(0xffffffffu, e0 || e1)) break;
                    if ((spins & 255u) == 0) {  // the clock is read on long waits only
                        const unsigned long long now = sw_ns();
                        if (!t0) t0 = now;
                        if (__any_sync(0xffffffffu, *(volatile int*)status == 8 || now - t0 > 4000000000ull)) {
                            atomicExch(status, 8);
                            ok = false;
                            break;
                        }
                    }
                    if (e0) pre[0] = sw_load(yp + blk(ts) * SB + lane);
                    if (e1) pre[1] = sw_load(yp + blk(ts) * SB + lane + 32);
                }
                const double2 v0 = pre[0], v1 = pre[1];
                if (ok && ts + 1 < t) fetch(ts + 1);
                if (ok) ok = __all_sync(0xffffffffu, sd_wait(yempty + s, ((seq / YR) & 1) ^ 1, gave_up));
                if (!ok) {
                    *gave_up = 1;
                    break;
                }
                double* y = ys + s * 512 + (lane >> 2) * 32 + c * 4 + (lane & 3);
                y[0] = v0.x;
                y[16] = v0.y;
                y[256] = v1.x;
                y[256 + 16] = v1.y;
                sd_arrive(yfull + s);
            }
        }
    } else {
        const int r = lane >> 2, q = lane & 3, o = warp * 8 + r;  // this lane's row of a block
        const int c = (2 * q) & 3;                                // its columns c, c + 1 (re: q < 2, im: q >= 2)
        int seq = 0, turn = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < nb; t += gridDim.x, ++turn) {
            const int bi = blk(t), r0 = bi * SB;
            double2 d[16];
#pragma unroll
            for (int g = 0; g < 16; ++g)
                d[g] = __ldg(&dinv[(size_t)bi * SB * SB + (ADJ ? o * SB + 4 * g + q : (4 * g + q) * SB + o)]);
            double b[2] = {0.0, 0.0};
            const bool in = r0 + o < n;
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (in && c + u < nc) {
                    const double2 v = rhs[(size_t)(c + u) * n + r0 + o];
                    b[u] = q < 2 ? v.x : v.y;
                }
            double a1[2] = {0.0, 0.0}, a2[2] = {0.0, 0.0}, v[2];
            for (int ts = 0; ts < t; ++ts, ++seq) {
                const int s = seq % ST, sy = seq % YR;
                // (a warp that gives up goes on to the barrier of every block row, so that none waits there)
                ok = ok && sd_wait(full + s, (seq / ST) & 1, gave_up) && sd_wait(yfull + sy, (seq / YR) & 1, gave_up);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                const C* tile = tiles + s * TILE + (ADJ ? o * LD + q : q * LD + o);
                const double* y = ys + sy * 512 + lane;
#pragma unroll
                for (int g = 0; g < 16; ++g) {
                    const double2 m = to_d2(tile[ADJ ? 4 * g : 4 * g * LD]);
                    const double yv = y[g * 32];
                    sd_dmma(a1, m.x, yv);
                    sd_dmma(a2, m.y, yv);
                }
                __syncwarp();
                if (lane == 0) {
                    sd_arrive(empty + s);
                    sd_arrive(yempty + sy);
                }
            }
            sd_join<ADJ>(a1, a2, q, v);
            double* sf = ss + (turn & 1) * 512;
#pragma unroll
            for (int u = 0; u < 2; ++u) sf[(o >> 2) * 32 + (2 * q + u) * 4 + (o & 3)] = in ? b[u] - v[u] : 0.0;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            a1[0] = a1[1] = a2[0] = a2[1] = 0.0;
#pragma unroll
            for (int g = 0; g < 16; ++g) {
                const double sv = sf[g * 32 + lane];
                sd_dmma(a1, d[g].x, sv);
                sd_dmma(a2, d[g].y, sv);
            }
            sd_join<ADJ>(a1, a2, q, v);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const double im = __shfl_xor_sync(0xffffffffu, v[u], 2);
                if (in && q < 2 && c + u < nc)
                    sw_store(&sol[(size_t)(c + u) * n + r0 + o], make_double2(sw_value(v[u]), sw_value(im)));
            }
        }
    }
    __syncthreads();
    if (tid == 0 && s_gave_up) atomicExch(status, 8);
}

// The sweeps' two waits on what never comes: a solution entry (the empty pattern, preset here) and a ring
// stage (an mbarrier without arrivals).
__global__ void sweep_wait_selftest_kernel(double2* entry, int* entry_status, int* ring_status,
                                           unsigned long long limit_ns) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ int gave_up;
    if (threadIdx.x == 0) {
        const double e = __longlong_as_double(-1ll);
        *entry = make_double2(e, e);
        sd_init(&bar, 1);
        gave_up = 0;
        __threadfence();
    }
    __syncthreads();
    double2 v = sw_load(entry);
    sw_wait(entry, v, entry_status, limit_ns);
    if (!sd_wait(&bar, 0, &gave_up, limit_ns)) atomicExch(ring_status, 8);
}
void launch_sweep_wait_selftest(int* entry_status, int* ring_status, void* entry, double limit_s, cudaStream_t st) {
    sweep_wait_selftest_kernel<<<1, 32, 0, st>>>((double2*)entry, entry_status, ring_status, selftest_ns(limit_s));
}

static int g_sms = 0;

template <typename C, bool LOWER, int NC>
static void step_launch_nc(cudaStream_t st, const C* A, int n, int b0, int bw, const double2* dinv, double2* r,
                           double2* sol) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g_sms);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, trsv_inv_step_kernel<C, LOWER, NC>, A, (size_t)n, n, b0, bw, dinv, r, sol);
}

template <typename C, bool LOWER>
static void step_launch(int nc, cudaStream_t st, const C* A, int n, int b0, int bw, const double2* dinv, double2* r,
                        double2* sol) {
    switch (nc) {
#define TV_CASE(K) \
    case K: step_launch_nc<C, LOWER, K>(st, A, n, b0, bw, dinv, r, sol); break;
        TV_CASE(1) TV_CASE(2) TV_CASE(3) TV_CASE(4) TV_CASE(5) TV_CASE(6) TV_CASE(7) TV_CASE(8)
#undef TV_CASE
    }
}

// the two sets of block inverses
size_t lu_inverse_bytes(int n) {
    const size_t nb = (n + SB - 1) / SB;
    return (size_t)2 * nb * SB * SB * sizeof(double2);
}

template <typename C>
static void inverses_impl(const C* A, int n, double2* inv, cudaStream_t st, long long* launches) {
    int nb = (n + SB - 1) / SB;
    StageScope sc(ST_SOLVE, st);
    const size_t smem = (size_t)(SB * TBI_LD + 32 * 32) * sizeof(double2);
    static PerDeviceOnce attr;
    once_per_device(attr, [&] {
        cudaFuncSetAttribute(tri_block_inverse_kernel<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(tri_block_inverse_kernel<float2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    });
    tri_block_inverse_kernel<C><<<dim3(nb, 2), 256, smem, st>>>(A, n, n, inv);
    *launches += 1;
}
void lu_block_inverses_fp64(const double2* A, int n, double2* inv, cudaStream_t st, long long* launches) {
    inverses_impl<double2>(A, n, inv, st, launches);
}
void lu_block_inverses_fp32(const float2* A, int n, double2* inv, cudaStream_t st, long long* launches) {
    inverses_impl<float2>(A, n, inv, st, launches);
}

// Persistent sweeps unless TCU_SOLVE=steps asks for one launch per block step.
static bool chain_enabled() {
    static const bool v = [] {
        const char* e = getenv("TCU_SOLVE");
        return !(e && std::string(e) == "steps");
    }();
    return v;
}

static void sweep_init() {
    static PerDeviceOnce sms_once;
    once_per_device(sms_once, [] {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
    });
}

template <typename C, int OP, int NC>
static bool sweep_launch_nc(cudaStream_t st, const C* A, int n, const double2* dinv, const double2* rhs, double2* sol,
                            double2* clear, int ncol, int* status) {
    static PerDeviceOnce attr;
    const size_t smem = sweep_smem_bytes<C>(NC);
    // a refused attribute makes the cooperative launch below fail, and the caller takes the step path
    once_per_device(attr, [&] {
        cudaFuncSetAttribute(sweep_kernel<C, OP, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    });
    const int nb = (n + SB - 1) / SB, chunks = (ncol + NC - 1) / NC;
    const int G = std::min(nb, g_sms / chunks);
    if (G < 1) return false;
    size_t lda = (size_t)n;
    void* args[] = {(void*)&A, &lda, &n, (void*)&nb, &ncol, (void*)&dinv, (void*)&rhs, &sol, &clear, &status};
    return cudaLaunchCooperativeKernel((void*)sweep_kernel<C, OP, NC>, dim3(G, chunks), dim3(SW_THREADS), args, smem,
                                       st) == cudaSuccess;
}

template <typename C, int OP>
static bool sweep_dmma_launch(cudaStream_t st, const C* A, int n, const double2* dinv, const double2* rhs, double2* sol,
                              double2* clear, int ncol, int* status) {
    static PerDeviceOnce attr;
    constexpr size_t smem = sd_smem_bytes<C, OP == SW_UH || OP == SW_LH>();
    once_per_device(attr, [&] {
        cudaFuncSetAttribute(sweep_dmma_kernel<C, OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    });
    const int nb = (n + SB - 1) / SB, chunks = (ncol + SD_COLS - 1) / SD_COLS;
    const int G = std::min(nb, g_sms / chunks);
    if (G < 1) return false;
    size_t lda = (size_t)n;
    void* args[] = {(void*)&A, &lda, &n, (void*)&nb, &ncol, (void*)&dinv, (void*)&rhs, &sol, &clear, &status};
    return cudaLaunchCooperativeKernel((void*)sweep_dmma_kernel<C, OP>, dim3(G, chunks), dim3(SD_THREADS), args, smem,
                                       st) == cudaSuccess;
}

template <typename C, int OP>
static bool sweep_launch(cudaStream_t st, const C* A, int n, const double2* dinv, const double2* rhs, double2* sol,
                         double2* clear, int ncol, int* status) {
    // the tensor cores from 3 columns on: they take the time of 4 however many there are (us per triangle at 1, 2, 3
    // and 4 columns, n = 1920 FP32: 64, 65, 66, 67 against 47, 61, 75, 89; 9600: 315, 315, 330, 341 against
    // 217, 273, 345, 419). n = 2 nlm spheres is even; an odd order would stay on the other kernel.
    if (n % 2 == 0 && ncol > SW_MAXC) return sweep_dmma_launch<C, OP>(st, A, n, dinv, rhs, sol, clear, ncol, status);
    switch (std::min(ncol, SW_MAXC)) {
#define SW_CASE(K) \
    case K: return sweep_launch_nc<C, OP, K>(st, A, n, dinv, rhs, sol, clear, ncol, status);
        SW_CASE(1) SW_CASE(2)
#undef SW_CASE
    }
    return false;
}

// The two sweeps of a solve over ncol <= SOLVE_MAXC columns, rhs -> mid -> out; false when they are
// turned off or a launch was refused (mid and out are then undefined, rhs is intact).
template <typename C>
bool lu_sweeps(const C* A, int n, const double2* inv, const double2* rhs, double2* mid, double2* out, int ncol,
               bool adjoint, int* status, cudaStream_t st, long long* launches) {
    if (!chain_enabled() || !status || ncol > SOLVE_MAXC) return false;
    sweep_init();
    const size_t nb = (n + SB - 1) / SB;
    const double2 *linv = inv, *uinv = inv + nb * SB * SB;
    cudaMemsetAsync(mid, 0xff, (size_t)n * ncol * sizeof(double2), st);  // the empty pattern
    const bool ok = adjoint ? sweep_launch<C, SW_UH>(st, A, n, uinv, rhs, mid, out, ncol, status) &&
                                  sweep_launch<C, SW_LH>(st, A, n, linv, mid, out, nullptr, ncol, status)
                            : sweep_launch<C, SW_L>(st, A, n, linv, rhs, mid, out, ncol, status) &&
                                  sweep_launch<C, SW_U>(st, A, n, uinv, mid, out, nullptr, ncol, status);
    if (ok) {
        if (launches) *launches += 2;
    } else {
        cudaGetLastError();  // a launch that was refused leaves no work behind
    }
    return ok;
}
template bool lu_sweeps<float2>(const float2*, int, const double2*, const double2*, double2*, double2*, int, bool, int*,
                                cudaStream_t, long long*);
template bool lu_sweeps<double2>(const double2*, int, const double2*, const double2*, double2*, double2*, int, bool,
                                 int*, cudaStream_t, long long*);

// x (n x ncol) <- A^-1 x; tmp holds 2 n ncol complex.
template <typename C>
static void solve_impl(const C* A, int n, const int* perm, const double2* inv, double2* x, double2* tmp, int ncol,
                       cudaStream_t st, long long* launches, int* status) {
    sweep_init();
    StageScope sc(ST_SOLVE, st);
    const int nb = (n + SB - 1) / SB;
    const size_t tot = (size_t)n * ncol;
    gather_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(x, tmp, perm, n, ncol);
    ++*launches;
    if (lu_sweeps<C>(A, n, inv, tmp, tmp + tot, x, ncol, false, status, st, launches)) return;
    const double2* linv = inv;
    const double2* uinv = inv + (size_t)nb * SB * SB;
    for (int c0 = 0; c0 < ncol; c0 += SMAXC) {
        const int nc = std::min(SMAXC, ncol - c0);
        double2* xc = x + (size_t)c0 * n;
        double2* y = tmp + (size_t)c0 * n;        // P b, then updated in place by the forward sweep
        double2* z = tmp + tot + (size_t)c0 * n;  // forward solution, updated in place by the backward sweep
        for (int b = 0; b < nb; ++b) {
            int b0 = b * SB, bw = std::min(SB, n - b0);
            step_launch<C, true>(nc, st, A, n, b0, bw, linv + (size_t)b * SB * SB, y, z);
            ++*launches;
        }
        for (int b = nb - 1; b >= 0; --b) {
            int b0 = b * SB, bw = std::min(SB, n - b0);
            step_launch<C, false>(nc, st, A, n, b0, bw, uinv + (size_t)b * SB * SB, z, xc);
            ++*launches;
        }
    }
}

void lu_solve_fp64(const double2* A, int n, const int* perm, const double2* inv, double2* x, double2* tmp, int ncol,
                   cudaStream_t st, long long* launches, int* status) {
    solve_impl<double2>(A, n, perm, inv, x, tmp, ncol, st, launches, status);
}
void lu_solve_fp32(const float2* A, int n, const int* perm, const double2* inv, double2* x, double2* tmp, int ncol,
                   cudaStream_t st, long long* launches, int* status) {
    solve_impl<float2>(A, n, perm, inv, x, tmp, ncol, st, launches, status);
}

}  // namespace tcu
