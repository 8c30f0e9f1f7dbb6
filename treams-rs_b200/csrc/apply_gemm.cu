// Matrix-free operator x - T C x in product form, for lmax 2..5, and its dipole blocks (any
// lmax): the columns of the dipole sources (the coarse correction of the two-level
// preconditioner) and the dipole-to-dipole block (its coarse operator).
//
// The coupling of destination sphere i is, per destination mode d and helicity,
//   (C x)_i[d, +] = sum_{j != i} sum_s (A_ij(s,d) + B_ij(s,d)) x_j[2s]
//   (C x)_i[d, -] = sum_{j != i} sum_s (A_ij(s,d) - B_ij(s,d)) x_j[2s+1]
// with A and B the plan's term sums over the pair's harmonic table Z_ij (sw/plan.rs:224-251,
// sw/coupling.rs:127-140). Exchanging the sums over j and over the plan's terms gives
//   G_i[idx, e] = sum_{j != i} Z_ij[idx] x_j[e]            (tsize x 2 nlm per destination)
//   (C x)_i[d, +] = sum_s sum_{t in A(s,d) + B(s,d)} w_t G_i[idx_t, 2s]   (and - for B at 2s+1)
// The first line is a complex product of the generated table matrix Z_i (tsize x N) with the
// coefficients X (N x 2 nlm): a register-tiled FP64 product whose A operand is built in shared
// memory chunk by chunk and never stored. The plan's term lists then run once per destination
// instead of once per pair. Work per ordered pair: tsize * 2 nlm complex multiply-adds
// (1,470 at lmax 3, 3,888 at lmax 4) plus one harmonic table.
//
// CTA = DI destination spheres x one right-hand side, RG x CG threads in whole warps; thread (rg, cg) owns
// G rows rg + RG u (u < TR) and columns cg + CG t (t < TC). Per chunk of KJ sources:
//   A) thread per pair: direction and radial sequence z_p(k r), p <= 2 lmax, to shared memory;
//   B) thread per (pair, order m >= 0): the order column of the solid harmonics times z_p,
//      written into the chunk's table matrix (rows dest * tsize + idx, one column per source);
//   C) the chunk's product update from shared memory.
// Finally G goes to shared memory and thread per (destination, d) applies the term lists,
// the Mie block and the alpha / beta / zadd epilogue of the operator.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "apply_shapes.h"
#include "common.cuh"
#include "kernels.h"
#include "pairtable.cuh"
#include "plan.h"

namespace tcu {

namespace {

size_t gemm_smem(const SubOp& o, const GemmShape& s) {
    const size_t tsz = (size_t)(o.order + 1) * (o.order + 1);
    const size_t rows = (size_t)s.TR * s.RG + 1, cols = (size_t)s.TC * s.CG, npair = (size_t)s.DI * s.KJ;
    const size_t chunk = ((size_t)s.KJ * rows + (size_t)s.KJ * cols + npair * (o.order + 1)) * sizeof(cplx) +
                         npair * sizeof(double4) + tsz * sizeof(double2);
    const size_t g = (size_t)s.DI * tsz * 2 * o.nsrc * sizeof(cplx);
    return chunk > g ? chunk : g;
}

// Coefficients of the degree recurrence P_deg = a z P_(deg-1) - b r^2 P_(deg-2) of order column m,
// at m (order + 1) + deg: the divisions once per CTA instead of once per pair and degree.
__device__ __forceinline__ void recurrence_table(int order, double2* rec, int tid, int nthr) {
    const int ord1 = order + 1;
    for (int t = tid; t < ord1 * ord1; t += nthr) {
        const int m = t / ord1, deg = t - m * ord1;
        rec[t] = deg > m ? make_double2(double(2 * deg - 1) / double(deg - m), double(deg + m - 1) / double(deg - m))
                         : make_double2(0.0, 0.0);
    }
}

// Phases A and B of one chunk: the harmonic tables of the pairs (i0 + il, j0 + jj), il < DI,
// jj < KJ, into Zs (row il * ts + idx, column jj, leading dimension ZLD); Rs (entry q of pair p at
// q npair + p) and Ds hold the radial sequences and directions, rec the recurrence_table. One
// barrier inside (between A and B), none at the end.
__device__ __forceinline__ void build_chunk(const DevPlan& P, int order, int N, double k,
                                            const double* __restrict__ pos, bool singular, int i0, int j0,
                                            int DI, int KJ, int ZLD, cplx* Zs, cplx* Rs, double4* Ds,
                                            const double2* rec, int tid, int nthr) {
    const int ord1 = order + 1, ts = ord1 * ord1, npair = DI * KJ;
    // A) per pair: state 2 = a table, 1 = coincident centres of the regular kind (Z = e_0),
    //    0 = no coupling (the pair i = j, sources or destinations past N, coincident outgoing)
    for (int p = tid; p < npair; p += nthr) {
        const int il = p / KJ, jj = p - il * KJ, i = i0 + il, j = j0 + jj;
        double u[3] = {0.0, 0.0, 0.0}, state = 0.0;
        if (i < N && j < N && j != i) {
            double r;
            if (unit_direction(pos[3 * i] - pos[3 * j], pos[3 * i + 1] - pos[3 * j + 1],
                               pos[3 * i + 2] - pos[3 * j + 2], r, u)) {
                state = 2.0;
                if (singular && k * r >= 0.5) {
                    // the recurrence of hankel_sequence, stored as it runs (no local array)
                    const double inv = 1.0 / (k * r);
                    double sn, cs;
                    sincos(k * r, &sn, &cs);
                    cplx prev = mk(cs * inv, sn * inv), cur = mk(sn * inv, -cs * inv);
                    for (int q = 0; q <= order; ++q) {
                        Rs[(size_t)q * npair + p] = cur;
                        const double f = double(2 * q + 1) * inv;
                        const cplx next = mk(f * cur.x - prev.x, f * cur.y - prev.y);
                        prev = cur;
                        cur = next;
                    }
                } else if (singular) {
                    cplx h[MAXP];
                    hankel_sequence<MAXP>(order, k * r, h);
                    for (int q = 0; q <= order; ++q) Rs[(size_t)q * npair + p] = h[q];
                } else {
                    double jv[MAXP];
                    bessel_j_sequence<MAXP>(order, k * r, jv);
                    for (int q = 0; q <= order; ++q) Rs[(size_t)q * npair + p] = mk(jv[q], 0.0);
                }
            } else if (!singular) {
                state = 1.0;
            }
        }
        Ds[p] = make_double4(u[0], u[1], u[2], state);
    }
    __syncthreads();
    // B) per (order m >= 0, pair), consecutive threads on consecutive pairs so that a warp runs one
    //    column length: entries deg = m..order at deg^2 + deg + m and deg^2 + deg - m
    for (int it = tid; it < npair * ord1; it += nthr) {
        const int m = it / npair, p = it - m * npair;
        const int il = p / KJ, jj = p - il * KJ;
        cplx* Zp = Zs + (size_t)jj * ZLD + (size_t)il * ts;
        const double4 D = Ds[p];
        if (D.w == 2.0) {
            const cplx* rad = Rs + p;
            const cplx xy = mk(D.x, D.y);
            const double z = D.z, r2 = D.x * D.x + D.y * D.y + D.z * D.z;
            cplx diag = mk(1.0, 0.0);
            for (int q = 1; q <= m; ++q) diag = cscale(cmul(diag, xy), -double(2 * q - 1));
            cplx pc = diag, prev = mk(0.0, 0.0);
            for (int deg = m; deg <= order; ++deg) {
                if (deg > m) {
                    const double2 ab = rec[m * ord1 + deg];
                    const double az = ab.x * z, br = ab.y * r2;
                    const cplx next = mk(az * pc.x - br * prev.x, az * pc.y - br * prev.y);
                    prev = pc;
                    pc = next;
                }
                const cplx rd = rad[(size_t)deg * npair];
                Zp[deg * deg + deg + m] = cmul(rd, pc);
                if (m > 0) {
                    const int idx = deg * deg + deg - m;
                    Zp[idx] = cmul(rd, cscale(cconj(pc), __ldg(&P.reflection[idx])));
                }
            }
        } else {
            for (int deg = m; deg <= order; ++deg) {
                Zp[deg * deg + deg + m] = mk((D.w == 1.0 && deg == 0) ? 1.0 : 0.0, 0.0);
                if (m > 0) Zp[deg * deg + deg - m] = mk(0.0, 0.0);
            }
        }
    }
}

// Term lists of the plan, Mie block and the alpha / beta / zadd epilogue: W lanes per (destination, d)
// of the DI destinations from i0, each lane the source lm s = lane, lane + W, ..., summed by shuffles in
// a fixed order, with G of destination il at Gs + il * tsize * 2 nsrc (rows: table index, columns:
// source lm and helicity). W is what the CTA's threads allow, at most 16: a thread alone walks a
// chain of 200 dependent gathers at lmax 4, about 5 us, as long as the product itself below some
// hundred spheres (40 spheres, 96 columns: 0.71 -> 0.45 ms an application).
__device__ __forceinline__ void terms_epilogue(const DevPlan& P, const SubOp& O, const cplx* Gs, int DI, int i0,
                                               int N, const cplx* __restrict__ T, const cplx* __restrict__ xc,
                                               size_t coff, const cplx* __restrict__ zadd, double alpha,
                                               double beta, bool singular, cplx* __restrict__ y, int tid,
                                               int nthr) {
    const int nlm = P.nlm, M = 2 * O.nsrc, ts = (O.order + 1) * (O.order + 1);
    const int ndst = O.ndst, tasks = DI * ndst;
    const int W = epilogue_lanes(tasks, nthr, O.nsrc);
    const int end = (tasks * W + 31) / 32 * 32;  // whole warps take part in the shuffles
    for (int t0 = tid; t0 < end; t0 += nthr) {
        const int it = min(t0 / W, tasks - 1), part = t0 % W;
        const int il = it / ndst, d = it - il * ndst, i = i0 + il;
        const cplx* G = Gs + (size_t)il * ts * M;
        cplx sp = mk(0.0, 0.0), sn = mk(0.0, 0.0);
        if (i < N)
            for (int s = part; s < O.nsrc; s += W) {
                const int2 cb = __ldg(&P.combo[s * nlm + d]);
                int t = cb.x;
                const int na = cb.y & 0xffff, nb = cb.y >> 16;
                const cplx* g = G + 2 * s;
                for (int e = 0; e < na; ++e, ++t) {
                    const cplx w = __ldg(&P.w[t]);
                    const cplx* ge = g + (size_t)__ldg(&P.idx[t]) * M;
                    cfma(sp, w, ge[0]);
                    cfma(sn, w, ge[1]);
                }
                for (int e = 0; e < nb; ++e, ++t) {
                    const cplx w = __ldg(&P.w[t]);
                    const cplx* ge = g + (size_t)__ldg(&P.idx[t]) * M;
                    cfma(sp, w, ge[0]);
                    cfma(sn, cneg(w), ge[1]);
                }
            }
        for (int o = W / 2; o > 0; o >>= 1) {
            sp.x += __shfl_xor_sync(0xffffffffu, sp.x, o);
            sp.y += __shfl_xor_sync(0xffffffffu, sp.y, o);
            sn.x += __shfl_xor_sync(0xffffffffu, sn.x, o);
            sn.y += __shfl_xor_sync(0xffffffffu, sn.y, o);
        }
        if (i >= N || part != 0 || t0 >= tasks * W) continue;
        // the input at (i, d) exists for source lm only (d < nsrc), the output for d < ndst
        const size_t row = (size_t)i * O.ldout + 2 * d, rin = (size_t)i * O.ldin + 2 * d;
        const cplx x0 = d < O.nsrc ? xc[rin] : mk(0.0, 0.0), x1 = d < O.nsrc ? xc[rin + 1] : mk(0.0, 0.0);
        cplx y0, y1;
        if (singular) {
            cplx tc0 = sp, tc1 = sn;  // T null: the coupling alone
            if (T) {
                const int lam = degree_of(d);
                const cplx* t4 = T + ((size_t)i * P.L + lam - 1) * 4;
                tc0 = cadd(cmul(t4[0], sp), cmul(t4[1], sn));
                tc1 = cadd(cmul(t4[2], sp), cmul(t4[3], sn));
            }
            y0 = cadd(cscale(x0, alpha), cscale(tc0, beta));
            y1 = cadd(cscale(x1, alpha), cscale(tc1, beta));
            if (zadd) {
                y0 = cadd(y0, zadd[coff + row]);
                y1 = cadd(y1, zadd[coff + row + 1]);
            }
        } else {
            y0 = cadd(x0, sp);
            y1 = cadd(x1, sn);
        }
        y[coff + row] = y0;
        y[coff + row + 1] = y1;
    }
}

template <int TR, int TC>
__global__ void __launch_bounds__(512, 1)
    apply_gemm_kernel(DevPlan P, SubOp O, int N, double k, const double* __restrict__ pos, const cplx* __restrict__ T,
                      const cplx* __restrict__ x, size_t ldx, const cplx* __restrict__ zadd, double alpha, double beta,
                      bool singular, cplx* __restrict__ y, int DI, int RG, int CG, int KJ) {
    extern __shared__ __align__(16) unsigned char ag_smem[];
    const int M = 2 * O.nsrc, order = O.order, ord1 = order + 1, ts = ord1 * ord1;
    // ZLD = ROWS + 1: the builder's writes of different sources (one column each) fall into
    // different banks; the product reads consecutive rows of one column
    const int ROWS = TR * RG, ZLD = ROWS + 1, COLS = TC * CG, npair = DI * KJ;
    cplx* Zs = reinterpret_cast<cplx*>(ag_smem);                     // KJ x ZLD (source-major)
    cplx* Xs = Zs + (size_t)KJ * ZLD;                                // KJ x COLS
    cplx* Rs = Xs + (size_t)KJ * COLS;                               // npair x (order + 1)
    double4* Ds = reinterpret_cast<double4*>(Rs + (size_t)npair * ord1);  // direction, state
    double2* rec = reinterpret_cast<double2*>(Ds + npair);           // ts
    cplx* Gs = reinterpret_cast<cplx*>(ag_smem);                     // at the end: DI * ts x M
    const int tid = threadIdx.x, nthr = blockDim.x;
    recurrence_table(order, rec, tid, nthr);
    const int rg = tid / CG, cg = tid - (tid / CG) * CG;
    const bool worker = rg < RG;
    const int i0 = blockIdx.x * DI;
    const size_t coff = (size_t)blockIdx.y * ldx;  // column offset, input and output alike
    const cplx* xc = x + coff;

    cplx acc[TR][TC];
#pragma unroll
    for (int u = 0; u < TR; ++u)
#pragma unroll
        for (int t = 0; t < TC; ++t) acc[u][t] = mk(0.0, 0.0);
    for (int t = tid; t < KJ * ZLD; t += nthr) Zs[t] = mk(0.0, 0.0);  // padding rows stay zero

    for (int j0 = 0; j0 < N; j0 += KJ) {
        __syncthreads();  // the previous chunk's product is done with Zs / Xs
        for (int t = tid; t < KJ * COLS; t += nthr) {
            const int jj = t / COLS, col = t - jj * COLS, j = j0 + jj;
            Xs[t] = (col < M && j < N) ? xc[(size_t)j * O.ldin + col] : mk(0.0, 0.0);
        }
        build_chunk(P, order, N, k, pos, singular, i0, j0, DI, KJ, ZLD, Zs, Rs, Ds, rec, tid, nthr);
        __syncthreads();
        // C) G += Z_chunk X_chunk
        if (worker) {
            const cplx* zr = Zs + rg;
            const cplx* xr = Xs + cg;
            for (int kk = 0; kk < KJ; ++kk) {
                cplx a[TR], b[TC];
#pragma unroll
                for (int u = 0; u < TR; ++u) a[u] = zr[(size_t)kk * ZLD + u * RG];
#pragma unroll
                for (int t = 0; t < TC; ++t) b[t] = xr[(size_t)kk * COLS + t * CG];
#pragma unroll
                for (int u = 0; u < TR; ++u)
#pragma unroll
                    for (int t = 0; t < TC; ++t) cfma(acc[u][t], a[u], b[t]);
            }
        }
    }
    __syncthreads();
    if (worker) {
#pragma unroll
        for (int u = 0; u < TR; ++u) {
            const int row = rg + u * RG;
#pragma unroll
            for (int t = 0; t < TC; ++t) {
                const int col = cg + t * CG;
                if (row < DI * ts && col < M) Gs[(size_t)row * M + col] = acc[u][t];
            }
        }
    }
    __syncthreads();
    terms_epilogue(P, O, Gs, DI, i0, N, T, xc, coff, zadd, alpha, beta, singular, y, tid, nthr);
}

// ---- stored tables -------------------------------------------------------------------------
// For repeated applications (GMRES) the tables of all ordered pairs are built once and kept in
// HBM, laid out for the FP64 tensor-core product: per block of DI destinations (RO row octets
// of 8 table rows, rows il * tsize + idx) and per chunk of 16 sources, a contiguous 2 KB slab
// per row octet and group of 4 sources in the m8n8k4 A-fragment order (lane = 4 * row % 8 +
// source % 4). The inputs are packed per call in the B-fragment order (lane = 4 * column % 8 +
// source % 4), so every fragment load of a warp reads 512 contiguous bytes.
constexpr int SRC_CHUNK = 16;  // sources per stored chunk
constexpr int AS_STAGES = 3;   // ring of the stored product (2 CTAs per SM at lmax <= 4)

// c += a b on one 8 x 8 FP64 tile (m8n8k4, A row-major, B column-major)
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// CTA = one block of DI destinations x a range of source chunks: builds the chunk tables
// (degrees <= order) exactly as the on-the-fly product does and writes them out in the stored
// order: the block's destinations side by side, row t * DI + destination, so that row octets ascend in
// degree (stored_product_blocks).
__global__ void __launch_bounds__(256) table_store_kernel(DevPlan P, int order, int N, double k,
                                                          const double* __restrict__ pos, bool singular, int DI,
                                                          int KJ, int RO, int NC, int span, cplx* __restrict__ Z) {
    extern __shared__ __align__(16) unsigned char ts_smem[];
    const int ord1 = order + 1, ts = ord1 * ord1, rows = DI * ts;
    const int ZLD = RO * 8 + 1, npair = DI * KJ;
    cplx* Zs = reinterpret_cast<cplx*>(ts_smem);                          // KJ x ZLD
    cplx* Rs = Zs + (size_t)KJ * ZLD;                                     // npair x (order + 1)
    double4* Ds = reinterpret_cast<double4*>(Rs + (size_t)npair * ord1);  // direction, state
    double2* rec = reinterpret_cast<double2*>(Ds + npair);                // ts
    __shared__ unsigned char place[128];                                  // stored row -> row of Zs
    const int tid = threadIdx.x, nthr = blockDim.x;
    recurrence_table(order, rec, tid, nthr);
    const int i0 = blockIdx.x * DI;
    for (int t = tid; t < KJ * ZLD; t += nthr) Zs[t] = mk(0.0, 0.0);  // padding rows stay zero
    if (DI > 1)  // at most 128 rows
        for (int row = tid; row < RO * 8; row += nthr) place[row] = row < rows ? row % DI * ts + row / DI : row;
    const int jbeg = blockIdx.y * span, jend = min(N, jbeg + span);
    cplx* Zb = Z + (size_t)blockIdx.x * NC * RO * 128;
    for (int j0 = jbeg; j0 < jend; j0 += KJ) {
        __syncthreads();  // the previous chunk is written out
        build_chunk(P, order, N, k, pos, singular, i0, j0, DI, KJ, ZLD, Zs, Rs, Ds, rec, tid, nthr);
        __syncthreads();
        // out: per 16-source chunk c, group q of 4 sources, row octet o, lane
        const int total = (KJ / SRC_CHUNK) * 4 * RO * 32;
        for (int it = tid; it < total; it += nthr) {
            const int lane = it & 31, w = it >> 5, o = w % RO, qc = w / RO;
            const int row = o * 8 + (lane >> 2), kk = qc * 4 + (lane & 3);  // qc = 4 c + q
            const cplx v = row < rows ? Zs[(size_t)kk * ZLD + (DI > 1 ? place[row] : row)] : mk(0.0, 0.0);
            const size_t slab = (size_t)(j0 / SRC_CHUNK) * 4 + qc;  // chunk * 4 + q
            if (slab < (size_t)NC * 4) Zb[(slab * RO + o) * 32 + lane] = v;  // the last build chunk may be half past N
        }
    }
}

// Inputs of ncol columns in the B-fragment order: per chunk, group q, column octet c, lane. With
// parts > 1 (the split product below) part h + 2 r holds the helicity-h entries of the sources'
// lm from r * cnt on, cnt of them.
__global__ void pack_sources_kernel(const cplx* __restrict__ x, size_t ldx, int ldin, int N, int M, int NC, int CT,
                                    int parts, int cnt, size_t per_col, cplx* __restrict__ Xf) {
    const size_t per = (size_t)NC * 4 * CT * 32;
    const cplx* xc = x + (size_t)blockIdx.y * ldx;
    const int part = blockIdx.z, s0 = (part >> 1) * cnt;
    cplx* out = Xf + (size_t)blockIdx.y * per_col + part * per;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < per; t += (size_t)gridDim.x * blockDim.x) {
        const int lane = (int)(t & 31);
        const size_t w = t >> 5;
        const int c = (int)(w % CT);
        const size_t g = w / CT;  // chunk * 4 + q
        const size_t j = g * 4 + (lane & 3);
        int col = c * 8 + (lane >> 2);
        bool ok = j < (size_t)N;
        if (parts > 1) {
            ok = ok && col < cnt && s0 + col < M / 2;
            col = 2 * (s0 + col) + (part & 1);
        } else {
            ok = ok && col < M;
        }
        out[t] = ok ? xc[j * ldin + col] : mk(0.0, 0.0);
    }
}

// y = zadd + alpha x + beta T C x (or the sub-operator O) from the stored tables: CTA = DI
// destinations x one column, complex accumulators as re and im 8 x 8 FP64 tiles, four m8n8k4 products
// per complex step: re += a.re b.re + a.im (-b.im), im += a.re b.im + a.im b.re; then the term lists.
// ---- bulk-copy pipeline of the stored product ---------------------------------------------
__device__ __forceinline__ uint32_t as_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void as_mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void as_mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void as_mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool as_mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait on a phase: false after 2 s (recorded in abort_flag) or once another warp gave up.
__device__ __forceinline__ bool as_mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                             unsigned long long limit_ns = 2000000000ull) {
    if (as_mbar_try(bar, parity)) return true;
    unsigned long long t0;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (unsigned it = 1;; ++it) {
        if (as_mbar_try(bar, parity)) return true;
        if ((it & 63u) == 0) {
            if (*abort_flag) return false;
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t - t0 > limit_ns) {
                *abort_flag = 1;
                return false;
            }
        }
    }
}
// This wait on a barrier without arrivals.
__global__ void product_wait_selftest_kernel(int* status, unsigned long long limit_ns) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ int abort_flag;
    as_mbar_init(as_smem_u32(&bar), 1);
    abort_flag = 0;
    if (!as_mbar_wait(as_smem_u32(&bar), 0, &abort_flag, limit_ns)) atomicExch(status, 8);
}
// contiguous global -> shared copy completing on an mbarrier (16-byte aligned, size % 16 == 0)
__device__ __forceinline__ void as_bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}

// most blocks a warp takes (stored_product_blocks over the product warps): 16 / 8, 30 / 8, 41 / 8, 52 / 8,
// 109 / 16, 103 / 16, 106 / 16. A block past the last slot would be dropped: stored_product_blocks refuses
// lists that product_capacity does not hold.
constexpr int SLOTS_DIPOLE = 2, SLOTS_L2 = 4, SLOTS_L3 = 6, SLOTS_L4 = 7, SLOTS_L5 = 7, SLOTS_L6 = 7, SLOTS_L7 = 7;

// The stored product with a producer warp: lane 0 of the last warp streams the 16-source chunks
// (table slab and packed inputs, each one contiguous bulk copy) into a 3-stage ring, each stage
// completing on its full barrier; the product warps take a stage once its full barrier flips
// and release it through its empty barrier (one arrival per warp), so no CTA-wide barrier
// sits in the loop. Every wait is bounded (2 s): on a timeout the kernel records status 8,
// waits (bounded) for the copies in flight and returns without writing y.
// On success the product Z X is in Gs = smem (rows < rows, columns < cols, row-major, the rows of
// destination 0 first), wherever a term reads it.
// Work: the 8 x 8 blocks of `blocks`, dealt out evenly to the product warps in row order, at most SLOTS each
// with its accumulators in registers. A source of degree l reads table degrees l - lmax .. l + lmax only,
// so a fifth of the blocks are never read (lmax 3: 41 of 52 remain, 4: 52 of 66, 5: 109 of 144, 6: 103 of
// 132), and warps of equal work keep the four DMMA pipes equally busy (warp w runs on scheduler w % 4; row
// octets by twos left them 4, 4, 3 and 2 octets at lmax 3). Both fragments of a slot are loaded for four
// products, 39 % of the shared-memory rate, two slots ahead and without a branch in between: 13 % of the
// time at lmax 3 and 6. One column: 1184 spheres lmax 3 0.64 -> 0.44 ms, 296 lmax 6 0.43 -> 0.345;
// 4096 lmax 3 7.6 -> 5.3, the DMMA pipe 84 % busy.
// A chunk's products of the first USED slots (of the first cnt of them), fragments read two slots ahead.
template <int SLOTS, int USED>
__device__ __forceinline__ void product_chunk(const cplx* stage, int da, int db, const int (&oa)[SLOTS],
                                              const int (&ob)[SLOTS], double (&re)[SLOTS][2], double (&im)[SLOTS][2],
                                              int cnt = USED) {
    constexpr int AHEAD = 2, STEPS = 4 * USED;
    cplx a[AHEAD + 1], b[AHEAD + 1];
#pragma unroll
    for (int n = 0; n < STEPS + AHEAD; ++n) {
        if (n < STEPS) {
            a[n % (AHEAD + 1)] = stage[n / USED * da + oa[n % USED]];
            b[n % (AHEAD + 1)] = stage[n / USED * db + ob[n % USED]];
        }
        if (n >= AHEAD) {
            const int j = (n - AHEAD) % USED;
            const cplx x = a[(n - AHEAD) % (AHEAD + 1)], z = b[(n - AHEAD) % (AHEAD + 1)];
            if (j < cnt) {
                dmma(re[j], x.x, z.x);
                dmma(im[j], x.x, z.y);
                dmma(re[j], x.y, -z.y);
                dmma(im[j], x.y, z.x);
            }
        }
    }
}
template <int SLOTS>
__device__ __forceinline__ bool stored_product(unsigned char* smem, const cplx* __restrict__ Zb,
                                               const cplx* __restrict__ Xb, int NC, int RO, int CT,
                                               const ProductBlocks& blocks, int list, int DI, int ts, int cols,
                                               int* __restrict__ status) {
    __shared__ __align__(8) uint64_t bars[2 * AS_STAGES];
    __shared__ int s_abort;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int W = (blockDim.x >> 5) - 1;  // product warps; warp W loads
    const int ABLK = RO * 128, BBLK = CT * 128, SBLK = ABLK + BBLK;  // complex entries per chunk
    cplx* ring = reinterpret_cast<cplx*>(smem);
    const uint32_t full0 = as_smem_u32(bars), empty0 = full0 + 8 * AS_STAGES;
    if (tid == 0) {
        for (int s = 0; s < AS_STAGES; ++s) {
            as_mbar_init(full0 + 8 * s, 1);
            as_mbar_init(empty0 + 8 * s, W);
        }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    volatile int* abort_flag = &s_abort;
    double re[SLOTS][2], im[SLOTS][2];
    int oa[SLOTS], ob[SLOTS];  // places of the slots' fragments in a group of 4 sources
    int cnt = 0, first = 0;
    if (warp < W) {
        const int total = blocks.count[list], base = total / W, extra = total - base * W;
        cnt = base + (warp < extra ? 1 : 0);
        first = warp * base + min(warp, extra);
#pragma unroll
        for (int j = 0; j < SLOTS; ++j) {
            const int at = min(first + j, total - 1);
            oa[j] = blocks.row[list][at] * 32 + lane;
            ob[j] = ABLK + blocks.col[list][at] * 32 + lane;
            re[j][0] = re[j][1] = im[j][0] = im[j][1] = 0.0;
        }
    }
    if (warp == W) {
        if (lane == 0) {
            int kc = 0;
            for (; kc < NC; ++kc) {
                const int s = kc % AS_STAGES;
                if (!as_mbar_wait(empty0 + 8 * s, ((kc / AS_STAGES) & 1) ^ 1, abort_flag)) break;
                const uint32_t dst = as_smem_u32(ring + (size_t)s * SBLK);
                as_mbar_expect_tx(full0 + 8 * s, (uint32_t)SBLK * 16u);
                as_bulk_load(dst, Zb + (size_t)kc * ABLK, (uint32_t)ABLK * 16u, full0 + 8 * s);
                as_bulk_load(dst + (uint32_t)ABLK * 16u, Xb + (size_t)kc * BBLK, (uint32_t)BBLK * 16u, full0 + 8 * s);
            }
            if (*abort_flag) {
                // drain: the last load issued into every stage lands before the CTA exits
                volatile int never = 0;
                for (int s = 0; s < AS_STAGES; ++s) {
                    const int last = kc - 1 - ((kc - 1 - s) % AS_STAGES + AS_STAGES) % AS_STAGES;
                    if (last >= 0) as_mbar_wait(full0 + 8 * s, (last / AS_STAGES) & 1, &never);
                }
            }
        }
    } else {
        for (int kc = 0; kc < NC; ++kc) {
            const int s = kc % AS_STAGES;
            if (!as_mbar_wait(full0 + 8 * s, (kc / AS_STAGES) & 1, abort_flag)) break;
            const cplx* stage = ring + (size_t)s * SBLK;
            if (cnt == SLOTS)
                product_chunk<SLOTS, SLOTS>(stage, RO * 32, CT * 32, oa, ob, re, im);
            else if (cnt == SLOTS - 1)
                product_chunk<SLOTS, SLOTS - 1>(stage, RO * 32, CT * 32, oa, ob, re, im);
            else  // lmax 7, first half of the sources
                product_chunk<SLOTS, (SLOTS > 2 ? SLOTS - 2 : 1)>(stage, RO * 32, CT * 32, oa, ob, re, im, cnt);
            __syncwarp();
            if (lane == 0) as_mbar_arrive(empty0 + 8 * s);
        }
    }
    __syncthreads();  // every chunk consumed: no copy in flight, the ring is free for G
    if (s_abort) {
        if (tid == 0 && status) atomicExch(status, 8);
        return false;
    }
    cplx* Gs = ring;
    if (warp < W) {
#pragma unroll
        for (int j = 0; j < SLOTS; ++j) {
            const int row = blocks.row[list][min(first + j, blocks.count[list] - 1)] * 8 + (lane >> 2);
            const int col = blocks.col[list][min(first + j, blocks.count[list] - 1)] * 8 + 2 * (lane & 3);
            if (j < cnt && row < DI * ts) {
                cplx* g = Gs + (size_t)(DI > 1 ? row % DI * ts + row / DI : row) * cols;
                if (col < cols) g[col] = mk(re[j][0], im[j][0]);
                if (col + 1 < cols) g[col + 1] = mk(re[j][1], im[j][1]);
            }
        }
    }
    __syncthreads();
    return true;
}

template <int SLOTS, int WARPS>
__global__ void __launch_bounds__(WARPS * 32 + 32, WARPS == 8 ? 2 : 1)
    apply_stored_tma_kernel(DevPlan P, SubOp O, int N, const cplx* __restrict__ Z, const cplx* __restrict__ Xf,
                            int NC, int DI, int RO, int CT, const __grid_constant__ ProductBlocks blocks,
                            const cplx* __restrict__ T, const cplx* __restrict__ x, size_t ldx,
                            const cplx* __restrict__ zadd, double alpha, double beta, bool singular,
                            cplx* __restrict__ y, int* __restrict__ status) {
    extern __shared__ __align__(128) unsigned char at_smem[];
    const int M = 2 * O.nsrc, ts = (O.order + 1) * (O.order + 1);
    if (!stored_product<SLOTS>(at_smem, Z + (size_t)blockIdx.x * NC * RO * 128,
                               Xf + (size_t)blockIdx.y * NC * CT * 128, NC, RO, CT, blocks, 0, DI, ts, M, status))
        return;
    const size_t coff = (size_t)blockIdx.y * ldx;
    terms_epilogue(P, O, reinterpret_cast<const cplx*>(at_smem), DI, blockIdx.x * DI, N, T, x + coff, coff, zadd, alpha,
                   beta, singular, y, threadIdx.x, blockDim.x);
}

// ---- split product (lmax 6 and 7) -----------------------------------------------------------
// One destination's G (169 x 96 complex at lmax 6) exceeds a CTA's registers, so `parts` CTAs share
// it: helicity h of the coupling reads the helicity-h source columns only, (C x)[d, +-] =
// sum_s sum_t +- w_t G[idx_t, s], so part h + 2 r takes helicity h and the cnt source lm from r cnt
// on (all 48 at lmax 6, 32 at lmax 7) and writes its sums over them to Cp; split_finish_kernel
// adds the parts in a fixed order and applies the Mie block and the epilogue. The DMMA pipe
// bounds it as it bounds lmax 2..5. 300 spheres lmax 6, one application: 4.3 ms with the per-pair
// term sums (CUDA cores, an index, a weight and a gather per term and pair), 0.38 ms here.
// One CTA fits an SM. Where the last wave of the (column, destination, part) tiles would leave half of the SMs
// or more idle, each of its tiles is cut into pieces of the source chunks, as many as there are SMs for them:
// tiles from `whole` on, whose pieces' sums go to Cx and are added by split_finish_kernel. 300 spheres at lmax 6
// are 600 tiles on 148 SMs, 4.05 waves: 0.43 -> 0.38 ms a product with 8 tiles in 18 pieces each.
struct SplitTail {
    int whole, pieces;
};
template <int SLOTS, int WARPS>
__global__ void __launch_bounds__(WARPS * 32 + 32, 1)
    apply_split_kernel(DevPlan P, int N, const cplx* __restrict__ Z, const cplx* __restrict__ Xf, size_t per_col,
                       int NC, int RO, int CT, const __grid_constant__ ProductBlocks blocks, int parts, int cnt,
                       SplitTail tail, cplx* __restrict__ Cp, cplx* __restrict__ Cx, int* __restrict__ status) {
    extern __shared__ __align__(128) unsigned char sp_smem[];
    const int b = blockIdx.x, over = b - tail.whole, q = over >= 0 ? over / tail.pieces : 0;
    const int tile = over >= 0 ? tail.whole + q : b, piece = over - q * tail.pieces;
    const int col = tile / (N * parts), i = tile / parts - col * N, part = tile % parts, s0 = (part >> 1) * cnt;
    const int c0 = over >= 0 ? piece * NC / tail.pieces : 0;
    const int c1 = over >= 0 ? (piece + 1) * NC / tail.pieces : NC;
    const int ns = min(cnt, P.nlm - s0), nlm = P.nlm;
    if (!stored_product<SLOTS>(sp_smem, Z + ((size_t)i * NC + c0) * RO * 128,
                               Xf + (size_t)col * per_col + ((size_t)part * NC + c0) * CT * 128, c1 - c0, RO, CT,
                               blocks, part >> 1, 1, P.tsize, cnt, status))
        return;
    cplx* out = over >= 0 ? Cx + (size_t)over * nlm : Cp + (((size_t)col * parts + part) * N + i) * nlm;
    const cplx* G = reinterpret_cast<const cplx*>(sp_smem);
    // thread (d, group): the group's source lm s = group, group + groups, ...; then a fixed-order sum
    __shared__ cplx sums[512];
    const int groups = min((int)blockDim.x / nlm, 8), d = threadIdx.x % nlm, grp = threadIdx.x / nlm;
    if (grp < groups) {
        const double sgn = (part & 1) ? -1.0 : 1.0;
        cplx a = mk(0.0, 0.0), b = mk(0.0, 0.0);
        for (int s = grp; s < ns; s += groups) {
            const int2 cb = __ldg(&P.combo[(s0 + s) * nlm + d]);
            int t = cb.x;
            const int na = cb.y & 0xffff, nb = cb.y >> 16;
            for (int e = 0; e < na; ++e, ++t) cfma(a, __ldg(&P.w[t]), G[(size_t)__ldg(&P.idx[t]) * cnt + s]);
            for (int e = 0; e < nb; ++e, ++t) cfma(b, __ldg(&P.w[t]), G[(size_t)__ldg(&P.idx[t]) * cnt + s]);
        }
        sums[grp * nlm + d] = mk(fma(sgn, b.x, a.x), fma(sgn, b.y, a.y));
    }
    __syncthreads();
    if (threadIdx.x < nlm) {
        cplx c = sums[threadIdx.x];
        for (int g = 1; g < groups; ++g) c = cadd(c, sums[g * nlm + threadIdx.x]);
        out[threadIdx.x] = c;
    }
}

// y from the parts' coupling sums: outgoing, y = zadd + alpha x + beta T c; regular, y = x + c.
__global__ void split_finish_kernel(DevPlan P, int N, int parts, SplitTail tail, const cplx* __restrict__ Cp,
                                    const cplx* __restrict__ Cx, const cplx* __restrict__ T, const cplx* __restrict__ x, size_t ldx,
                                    const cplx* __restrict__ zadd, double alpha, double beta, bool singular,
                                    cplx* __restrict__ y) {
    const int nlm = P.nlm;
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (size_t)N * nlm) return;
    const size_t i = t / nlm, per = (size_t)N * nlm;
    const int d = (int)(t - i * nlm);
    const int tile = ((int)blockIdx.y * N + (int)i) * parts;
    auto sum_of = [&](int p) {
        const int over = tile + p - tail.whole;
        if (over < 0) return Cp[((size_t)blockIdx.y * parts + p) * per + t];
        const cplx* c = Cx + (size_t)over * tail.pieces * nlm + d;
        cplx v = c[0];
        for (int k = 1; k < tail.pieces; ++k) v = cadd(v, c[(size_t)k * nlm]);
        return v;
    };
    cplx sp = sum_of(0), sn = sum_of(1);
    for (int p = 2; p < parts; p += 2) {
        sp = cadd(sp, sum_of(p));
        sn = cadd(sn, sum_of(p + 1));
    }
    const size_t row = (size_t)blockIdx.y * ldx + 2 * t;
    const cplx x0 = x[row], x1 = x[row + 1];
    if (!singular) {
        y[row] = cadd(x0, sp);
        y[row + 1] = cadd(x1, sn);
        return;
    }
    cplx tc0 = sp, tc1 = sn;  // T null: the coupling alone
    if (T) {
        const cplx* t4 = T + (i * P.L + degree_of(d) - 1) * 4;
        tc0 = cadd(cmul(t4[0], sp), cmul(t4[1], sn));
        tc1 = cadd(cmul(t4[2], sp), cmul(t4[3], sn));
    }
    cplx y0 = cadd(cscale(x0, alpha), cscale(tc0, beta)), y1 = cadd(cscale(x1, alpha), cscale(tc1, beta));
    if (zadd) {
        y0 = cadd(y0, zadd[row]);
        y1 = cadd(y1, zadd[row + 1]);
    }
    y[row] = y0;
    y[row + 1] = y1;
}

}  // namespace

bool stored_tables_enabled() {
    const char* e = getenv("TCU_APPLY");
    return !(e && (strcmp(e, "fly") == 0 || strcmp(e, "terms") == 0));
}

static bool product_forms_enabled() {
    const char* e = getenv("TCU_APPLY");  // "terms": the per-pair term-sum kernels instead
    return !(e && strcmp(e, "terms") == 0);
}
bool apply_gemm_supported(const DevPlan& P) { return P.L >= 2 && P.L <= 5 && product_forms_enabled(); }
bool stored_full_supported(const DevPlan& P) { return P.L >= 2 && P.L <= 7 && product_forms_enabled(); }

template <int TR, int TC>
static void launch_shape(const DevPlan& P, const SubOp& O, const GemmShape& s, int N, double k, const double* pos,
                         const cplx* T, const cplx* x, size_t ldx, int ncol, const cplx* zadd, double alpha,
                         double beta, bool singular, cplx* y, cudaStream_t st) {
    const dim3 grid((unsigned)((N + s.DI - 1) / s.DI), (unsigned)ncol);
    apply_gemm_kernel<TR, TC><<<grid, shape_threads(s), gemm_smem(O, s), st>>>(P, O, N, k, pos, T, x, ldx, zadd, alpha,
                                                                          beta, singular, y, s.DI, s.RG, s.CG, s.KJ);
}

void launch_apply_gemm(const DevPlan& P, int N, double k, const double* pos, const cplx* T, const cplx* x, size_t ldx,
                       int ncol, const cplx* zadd, double alpha, double beta, bool singular, cplx* y,
                       cudaStream_t st) {
    if (N <= 0 || ncol <= 0) return;
    const GemmShape s = gemm_shape(P.L);
    const SubOp O{P.nlm, P.nlm, P.order, 2 * P.nlm, 2 * P.nlm};
    switch (P.L) {
        case 2: launch_shape<4, 2>(P, O, s, N, k, pos, T, x, ldx, ncol, zadd, alpha, beta, singular, y, st); break;
        case 3: launch_shape<4, 3>(P, O, s, N, k, pos, T, x, ldx, ncol, zadd, alpha, beta, singular, y, st); break;
        case 4: launch_shape<4, 4>(P, O, s, N, k, pos, T, x, ldx, ncol, zadd, alpha, beta, singular, y, st); break;
        default: launch_shape<4, 5>(P, O, s, N, k, pos, T, x, ldx, ncol, zadd, alpha, beta, singular, y, st); break;
    }
}

void launch_product_wait_selftest(int* status, double limit_s, cudaStream_t st) {
    product_wait_selftest_kernel<<<1, 1, 0, st>>>(status, selftest_ns(limit_s));
}

void launch_apply_dipole(const DevPlan& P, int N, double k, const double* pos, const cplx* T, const cplx* z,
                         bool dipole_rows, const cplx* zadd, double alpha, double beta, cplx* y, cudaStream_t st) {
    if (N <= 0) return;
    StageScope sc(ST_COARSE, st);
    const int ndst = dipole_rows ? 3 : P.nlm;
    const SubOp O{3, ndst, 1 + (dipole_rows ? 1 : P.L), 6, 2 * ndst};
    const GemmShape s = sub_shape((O.order + 1) * (O.order + 1));
    launch_shape<4, 2>(P, O, s, N, k, pos, T, z, 0, 1, zadd, alpha, beta, true, y, st);
}

// ---- stored tables: host side ----------------------------------------------------------------
namespace {
SubOp stored_subop(const DevPlan& P, int kind) {
    switch (kind) {
        case STORED_DIPOLE_SOURCES: return {3, P.nlm, 1 + P.L, 6, 2 * P.nlm};
        case STORED_DIPOLE_BLOCK: return {3, 3, 2, 6, 6};
        default: return {P.nlm, P.nlm, P.order, 2 * P.nlm, 2 * P.nlm};
    }
}
// full operator: lmax 2..5, and in parts lmax 6 and 7; dipole blocks: tables of at most 128 entries (one destination per
// block then fills at most 16 row octets, the 8 warps of the product)
bool stored_kind_ok(const DevPlan& P, int kind) {
    if (kind == STORED_FULL) return P.L >= 2 && P.L <= 7;
    if (kind != STORED_DIPOLE_SOURCES && kind != STORED_DIPOLE_BLOCK) return false;
    const int order = stored_subop(P, kind).order;
    return (order + 1) * (order + 1) <= 128;
}
struct StoredLayout {
    SubOp O;
    int DI, KJ, RO, CT, NC, nblk;
    int parts, cnt;                     // split product: CTAs per destination, source lm of each (else 1, 0)
    size_t z_elems, xf_per_col, cp_per_col;  // cp: the split product's coupling sums
};
StoredLayout stored_layout(const DevPlan& P, int N, int kind) {
    StoredLayout l;
    l.O = stored_subop(P, kind);
    const int ts = (l.O.order + 1) * (l.O.order + 1);
    l.DI = std::max(1, 128 / ts);  // about 128 table rows per destination block
    l.KJ = 32;
    l.RO = (l.DI * ts + 7) / 8;
    l.parts = 1;
    l.cnt = 0;
    if (kind == STORED_FULL && P.L > 5) {
        const int halves = P.L == 6 ? 1 : 2;  // of the source lm, per helicity
        l.parts = 2 * halves;
        l.cnt = (l.O.nsrc + halves - 1) / halves;
    }
    l.CT = ((l.parts > 1 ? l.cnt : 2 * l.O.nsrc) + 7) / 8;
    l.NC = (N + SRC_CHUNK - 1) / SRC_CHUNK;
    l.nblk = (N + l.DI - 1) / l.DI;
    l.z_elems = (size_t)l.nblk * l.NC * l.RO * 128;
    l.xf_per_col = (size_t)l.parts * l.NC * l.CT * 128;
    l.cp_per_col = l.parts > 1 ? (size_t)l.parts * N * P.nlm : 0;
    return l;
}
size_t stored_smem(const StoredLayout& l) {
    const size_t ring = (size_t)AS_STAGES * (l.RO + l.CT) * 128 * sizeof(cplx);
    const size_t g = (size_t)l.DI * (l.O.order + 1) * (l.O.order + 1) * (l.parts > 1 ? l.cnt : 2 * l.O.nsrc) *
                     sizeof(cplx);
    return ring > g ? ring : g;
}
size_t store_smem(const StoredLayout& l) {
    const size_t npair = (size_t)l.DI * l.KJ;
    return ((size_t)l.KJ * (l.RO * 8 + 1) + npair * (l.O.order + 1)) * sizeof(cplx) + npair * sizeof(double4) +
           (size_t)(l.O.order + 1) * (l.O.order + 1) * sizeof(double2);
}
}  // namespace

// blocks that the warps of the full operator's product take (launch_apply_stored)
static int product_capacity(int L) {
    switch (L) {
        case 2: return 8 * SLOTS_L2;
        case 3: return 8 * SLOTS_L3;
        case 4: return 8 * SLOTS_L4;
        case 5: return 16 * SLOTS_L5;
        case 6: return 16 * SLOTS_L6;
        default: return 16 * SLOTS_L7;
    }
}
// The blocks of the full coupling operator's product that a term of the plan reads: source lm s and table
// entry t meet in the term lists of some destination. Natural order of both already gathers them (of
// random exchanges of rows and columns none found fewer). False when the product's warps cannot hold them.
bool stored_product_blocks(const DevPlan& P, const HostPlan& h, ProductBlocks* b) {
    b->count[0] = b->count[1] = 0;
    if (P.L < 2 || P.L > 7) return true;
    const StoredLayout l = stored_layout(P, 1, STORED_FULL);
    std::vector<char> read((size_t)h.nlm * P.tsize, 0);
    for (int c = 0; c < h.nlm * h.nlm; ++c) {
        const int n = (h.combo[2 * c + 1] & 0xffff) + (h.combo[2 * c + 1] >> 16);
        for (int e = 0; e < n; ++e) read[(size_t)(c / h.nlm) * P.tsize + h.idx[h.combo[2 * c] + e]] = 1;
    }
    for (int list = 0; list < std::max(1, l.parts / 2); ++list)
        for (int o = 0; o < l.RO; ++o)
            for (int c = 0; c < l.CT; ++c) {
                bool any = false;
                for (int row = o * 8; row < std::min(o * 8 + 8, l.DI * P.tsize); ++row)
                    for (int col = c * 8; col < c * 8 + 8; ++col) {
                        if (l.parts > 1 && col >= l.cnt) break;
                        const int s = l.parts > 1 ? list * l.cnt + col : col / 2;
                        any = any || (s < h.nlm && read[(size_t)s * P.tsize + row / l.DI]);
                    }
                if (!any) continue;
                if (b->count[list] == std::min(product_capacity(P.L), (int)ProductBlocks::MAX)) return false;
                b->row[list][b->count[list]] = (unsigned char)o;
                b->col[list][b->count[list]++] = (unsigned char)c;
            }
    return true;
}
// every block of a product (the dipole operators: one column octet)
static ProductBlocks all_blocks(const StoredLayout& l) {
    ProductBlocks b;
    b.count[0] = b.count[1] = 0;
    for (int o = 0; o < l.RO; ++o)
        for (int c = 0; c < l.CT; ++c) {
            b.row[0][b.count[0]] = (unsigned char)o;
            b.col[0][b.count[0]++] = (unsigned char)c;
        }
    return b;
}

size_t stored_tables_bytes(const DevPlan& P, int N, int kind) {
    if (!stored_kind_ok(P, kind) || N <= 0) return 0;
    return stored_layout(P, N, kind).z_elems * sizeof(cplx);
}

static int num_sms() {
    static const int sms = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v;
    }();
    return sms;
}

size_t stored_inputs_bytes(const DevPlan& P, int N, int kind, int ncol) {
    if (!stored_kind_ok(P, kind) || N <= 0) return 0;
    const StoredLayout l = stored_layout(P, N, kind);
    // the pieces of the split product's tail: one coupling sum per SM at most
    const size_t cx = l.parts > 1 ? (size_t)num_sms() * P.nlm : 0;
    return ((l.xf_per_col + l.cp_per_col) * (size_t)ncol + cx) * sizeof(cplx);
}

void build_stored_tables(const DevPlan& P, int N, double k, const double* pos, int kind, cplx* Z, cudaStream_t st,
                         bool singular) {
    if (N <= 0 || !stored_kind_ok(P, kind)) return;
    StageScope sc(kind == STORED_FULL ? ST_APPLY : ST_COARSE, st);
    const StoredLayout l = stored_layout(P, N, kind);
    const int nchunk = (N + l.KJ - 1) / l.KJ;
    const int ysplit = std::min(nchunk, std::max(1, (4 * 148 + l.nblk - 1) / l.nblk));
    const int span = (nchunk + ysplit - 1) / ysplit * l.KJ;
    const dim3 grid((unsigned)l.nblk, (unsigned)((nchunk * l.KJ + span - 1) / span));
    table_store_kernel<<<grid, 256, store_smem(l), st>>>(P, l.O.order, N, k, pos, singular, l.DI, l.KJ, l.RO, l.NC, span,
                                                         Z);
}

void launch_apply_stored(const DevPlan& P, int N, int kind, const cplx* Z, const cplx* T, const cplx* x, size_t ldx,
                         int ncol, const cplx* zadd, double alpha, double beta, cplx* y, cplx* Xf, int* status,
                         cudaStream_t st, bool singular) {
    if (N <= 0 || ncol <= 0 || !stored_kind_ok(P, kind)) return;
    StageScope sc(kind == STORED_FULL ? ST_APPLY : ST_COARSE, st);
    const StoredLayout l = stored_layout(P, N, kind);
    const int M = 2 * l.O.nsrc;
    const dim3 pgrid((unsigned)std::min<size_t>((l.xf_per_col / l.parts + 255) / 256, 1024), (unsigned)ncol,
                     (unsigned)l.parts);
    pack_sources_kernel<<<pgrid, 256, 0, st>>>(x, ldx, l.O.ldin, N, M, l.NC, l.CT, l.parts, l.cnt, l.xf_per_col, Xf);
    const size_t smem = stored_smem(l);
    const ProductBlocks blocks = kind == STORED_FULL ? *P.blocks : all_blocks(l);
    if (l.parts > 1) {
        cplx* Cp = Xf + l.xf_per_col * ncol;
        cplx* Cx = Cp + l.cp_per_col * ncol;
        const int tiles = N * l.parts * ncol, sms = num_sms(), last = tiles % sms;
        SplitTail tail{tiles, 1};
        if (last > 0 && 2 * last <= sms && l.NC > 1) tail = {tiles - last, std::min(sms / last, l.NC)};
        const int ctas = tail.whole + (tiles - tail.whole) * tail.pieces;
        auto split = [&](auto kernel, int warps) {
            kernel<<<ctas, warps * 32 + 32, smem, st>>>(P, N, Z, Xf, l.xf_per_col, l.NC, l.RO, l.CT, blocks, l.parts,
                                                        l.cnt, tail, Cp, Cx, status);
        };
        if (P.L == 6)
            split(apply_split_kernel<SLOTS_L6, 16>, 16);
        else
            split(apply_split_kernel<SLOTS_L7, 16>, 16);
        const dim3 fg((unsigned)(((size_t)N * P.nlm + 255) / 256), (unsigned)ncol);
        split_finish_kernel<<<fg, 256, 0, st>>>(P, N, l.parts, tail, Cp, Cx, T, x, ldx, zadd, alpha, beta, singular, y);
        return;
    }
    const dim3 grid((unsigned)l.nblk, (unsigned)ncol);
    auto apply = [&](auto kernel, int warps) {
        kernel<<<grid, warps * 32 + 32, smem, st>>>(P, l.O, N, Z, Xf, l.NC, l.DI, l.RO, l.CT, blocks, T, x, ldx, zadd,
                                                    alpha, beta, singular, y, status);
    };
    // 8 warps and two CTAs per SM while the ring allows (lmax 5: 153 KB), 16 warps beyond
    switch (l.CT) {
        case 1: apply(apply_stored_tma_kernel<SLOTS_DIPOLE, 8>, 8); break;
        case 2: apply(apply_stored_tma_kernel<SLOTS_L2, 8>, 8); break;
        case 4: apply(apply_stored_tma_kernel<SLOTS_L3, 8>, 8); break;
        case 6: apply(apply_stored_tma_kernel<SLOTS_L4, 8>, 8); break;
        default: apply(apply_stored_tma_kernel<SLOTS_L5, 16>, 16); break;
    }
}

void apply_gemm_init_attributes() {
    cudaFuncSetAttribute(apply_gemm_kernel<4, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(apply_gemm_kernel<4, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(apply_gemm_kernel<4, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(apply_gemm_kernel<4, 5>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(table_store_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    auto allow = [](auto kernel) { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); };
    allow(apply_stored_tma_kernel<SLOTS_DIPOLE, 8>);
    allow(apply_stored_tma_kernel<SLOTS_L2, 8>);
    allow(apply_stored_tma_kernel<SLOTS_L3, 8>);
    allow(apply_stored_tma_kernel<SLOTS_L4, 8>);
    allow(apply_stored_tma_kernel<SLOTS_L5, 16>);
    allow(apply_split_kernel<SLOTS_L6, 16>);
    allow(apply_split_kernel<SLOTS_L7, 16>);
}

}  // namespace tcu
