// LU panel factorization on thread-block clusters (included by lu.cu).
//
// A panel column needs one exchange between all CTAs that hold its rows: the largest |a| and the
// row it sits in. Through global memory (panel_kernel in lu.cu: a grid barrier, then the key, then
// the row) that exchange is five dependent L2 round trips and serialised arrivals on one counter,
// 2.5 us a column on 4 CTAs and 3.4 us on 148, which is nearly all of the kernel's time. Here the
// CTAs of a cluster push their candidates into each other's shared memory instead:
//  - thread = row. A 16-column sub-block of the row sits in the thread's registers; the rank-1
//    update of a column shifts it by one entry, so the column loop is the same code for every
//    column. The multiplier goes to the shared-memory slab (chunk x (NB + 1), row-major) at once.
//  - per column every CTA finds its candidate (redux.sync, one __syncthreads) and sends it to every
//    CTA of the cluster with st.async: 16 entries, the key (|a|^2 as FP32 bits, + 1), the row and the
//    FP64 reciprocal of its pivot. An mbarrier counts the bytes; every warp then picks the winner
//    among at most 16 keys. One one-way message per column, no barrier.
//  - panels beyond one cluster's shared memory take several clusters of 16: the CTA that holds its
//    cluster's winner publishes it in global words that carry their own flags (4 bytes of value
//    and the epoch in one 8-byte word, no fence), and every CTA reads the clusters' winners.
//  - rows do not move. A pivot row stays in its slab, its entries over the panel's remaining columns
//    go to global memory behind the next column's exchange, and after 16 columns every CTA reads the
//    16 rows, forms their U part (forward substitution) and applies one rank-16 update to its rows.
//    Row interchanges become a permutation of the destination rows when the slab is written back.
// Measured per column (us, panel_kernel -> this): n = 240 FP64 2.60 -> 1.19, 1920 FP64 3.04 -> 1.35, 4272
// FP64 3.02 -> 1.63, 1920 FP32 2.87 -> 1.22, 12288 FP32 3.13 -> 1.79, 24576 FP32 3.42 -> 2.27. A column of
// a 4-CTA cluster is about 2300 cycles: candidate 370, message 700, pick 130, rank-1 update 450, a 16th
// of the sub-block's end 460; several clusters add 500 to 1200 for the global exchange.
// Pivots: the largest |a| in FP32 bits of |a|^2, ties to the lower original row.
// Every wait is bounded (4 s): status 8; the CTAs then run to the end without waiting, so that none
// exits while another may still send to it.
#pragma once

#include "panel_shape.h"

namespace tcu {

// A candidate message in 16-byte units: 16 entries, {key, row} in the first word of the next unit, the
// reciprocal. Words are 8 bytes.
template <typename C>
struct PcMsg {
    static constexpr int E = sizeof(C) / 8;
    static constexpr int UNITS = PC_SUB * E / 2;  // of the entries: 8 or 16, a thread each per CTA
    static constexpr int KEY = PC_SUB * E, INV = KEY + 2, WORDS = INV + 2, BYTES = WORDS * 8;
    static_assert(BYTES == panel_message_bytes(sizeof(C)), "the launch sizes shared memory by it");
};

typedef unsigned long long pc_word;

__device__ __forceinline__ uint32_t pc_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t pc_map(uint32_t addr, uint32_t cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
    return r;
}
__device__ __forceinline__ void pc_send2(uint32_t dst, pc_word v0, pc_word v1, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "l"(v0), "l"(v1), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void pc_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool pc_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void pc_cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// A long wait checks the clock and the status word; true when the caller has to give up.
__device__ __forceinline__ bool pc_expired(unsigned long long& t0, unsigned spins, int* status, volatile int* quit,
                                           unsigned long long limit_ns = BARRIER_LIMIT_NS) {
    if ((spins & 255u) != 0) return false;
    if (*quit) return true;
    const unsigned long long now = global_ns();
    if (!t0) t0 = now;
    if (*(volatile int*)status != 8 && now - t0 <= limit_ns) return false;
    atomicExch(status, 8);
    *quit = 1;
    return true;
}
__device__ __forceinline__ void pc_wait(uint32_t bar, uint32_t parity, int* status, volatile int* quit,
                                        unsigned long long limit_ns = BARRIER_LIMIT_NS) {
    unsigned long long t0 = 0;
    for (unsigned spins = 1; !pc_try(bar, parity); ++spins)
        if (*quit || pc_expired(t0, spins, status, quit, limit_ns)) return;
}
// global words that carry their own flag
__device__ __forceinline__ void pc_put(uint4* p, pc_word v, unsigned flag) {
    asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"((unsigned)v), "r"(flag),
                 "r"((unsigned)(v >> 32)), "r"(flag)
                 : "memory");
}
__device__ __forceinline__ uint4 pc_peek(const uint4* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}
__device__ __forceinline__ pc_word pc_get(const uint4* p, uint4 v, unsigned flag, int* status, volatile int* quit,
                                          unsigned long long limit_ns = BARRIER_LIMIT_NS) {
    unsigned long long t0 = 0;
    for (unsigned spins = 1; v.y != flag || v.w != flag; ++spins) {
        if (*quit || pc_expired(t0, spins, status, quit, limit_ns)) break;
        v = pc_peek(p);
    }
    return (pc_word)v.x | ((pc_word)v.z << 32);
}
// lowest lane with the largest key
__device__ __forceinline__ int pc_best(unsigned key) {
    const unsigned m = __reduce_max_sync(0xffffffffu, key);
    return __ffs(__ballot_sync(0xffffffffu, key == m)) - 1;
}
__device__ __forceinline__ void pc_store2(float2* p, float2 a, float2 b) {
    *reinterpret_cast<float4*>(p) = make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void pc_store2(double2* p, double2 a, double2 b) {
    p[0] = a;
    p[1] = b;
}
__device__ __forceinline__ void pc_load2(const float2* p, float2& a, float2& b) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    a = make_float2(v.x, v.y);
    b = make_float2(v.z, v.w);
}
__device__ __forceinline__ void pc_load2(const double2* p, double2& a, double2& b) {
    a = p[0];
    b = p[1];
}
// x - l u
__device__ __forceinline__ float2 pc_sub(float2 x, float2 l, float2 u) {
    return make_float2(fmaf(-l.x, u.x, fmaf(l.y, u.y, x.x)), fmaf(-l.x, u.y, fmaf(-l.y, u.x, x.y)));
}
__device__ __forceinline__ double2 pc_sub(double2 x, double2 l, double2 u) {
    return make_double2(fma(-l.x, u.x, fma(l.y, u.y, x.x)), fma(-l.x, u.y, fma(-l.y, u.x, x.y)));
}

// global words of the clusters' exchange and of the pivot rows (uint4 each)
constexpr size_t PC_GKEY = 2 * PC_MAXCL * 36, PC_GROW = 2 * PC_SUB * 128;

template <typename R, int NB>
__global__ void __launch_bounds__(PC_T, 1)
    panel_cluster_kernel(typename Cx<R>::T* A, size_t lda, int k0, int n, int w, int chunk, int cs, unsigned epoch,
                         int* __restrict__ piv, uint4* gkey, uint4* grow, int* status) {
    typedef typename Cx<R>::T C;
    typedef PcMsg<C> M;
    constexpr int LD = NB + 1, E = M::E;
    extern __shared__ __align__(16) unsigned char pc_raw[];
    pc_word* recvA = reinterpret_cast<pc_word*>(pc_raw);   // [2][cs] messages of the cluster's CTAs
    pc_word* gmsg = recvA + 2 * cs * M::WORDS;             // the clusters' winners
    // the warps' candidates are double-buffered by column parity: a warp may reach the next column
    // while another one still sends this one's
    C* srow = reinterpret_cast<C*>(gmsg + PC_MAXCL * M::WORDS);  // [2][warp][16] their rows
    C* pbuf = srow + 2 * PC_WARPS * PC_SUB;                // [16][NB] the sub-block's pivot rows
    C* tile = pbuf + PC_SUB * NB;                          // chunk x LD
    __shared__ __align__(8) uint64_t s_bar[2];
    __shared__ unsigned s_key[2][PC_WARPS], s_row[2][PC_WARPS];
    __shared__ short s_done[PC_T];           // 1 + pivot index of a local row, 0: not a pivot
    __shared__ int s_at[NB], s_pos[NB];      // row at a top position, position of a top row
    __shared__ int s_prow[PC_SUB];
    __shared__ int s_quit;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = blockIdx.x % cs, cl = blockIdx.x / cs, ncl = gridDim.x / cs;
    const int rows = n - k0, row0 = k0 + blockIdx.x * chunk;
    const int myrows = max(0, min(chunk, rows - (int)blockIdx.x * chunk));
    const uint32_t barA = pc_smem(s_bar);
    volatile int* quit = &s_quit;
    if (tid == 0) {
        for (int i = 0; i < 2; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(barA + 8 * i) : "memory");
        s_quit = 0;
        for (int i = 0; i < 2 && i < w; ++i) pc_expect(barA + 8 * i, cs * M::BYTES);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    s_done[tid] = 0;
    for (int t = tid; t < w; t += PC_T) s_at[t] = s_pos[t] = k0 + t;
    // the slab, transposed on the way in; all copies in flight at once
    for (int c = warp; c < w; c += PC_WARPS)
        for (int r = lane; r < myrows; r += 32) {
            const uint32_t dst = pc_smem(&tile[(size_t)r * LD + c]);
            const C* src = &A[(size_t)(k0 + c) * lda + row0 + r];
            if (sizeof(C) == 16)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
            else
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
        }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    pc_cluster_barrier();  // every CTA's barriers are initialised

    // where this thread sends: unit `unit` of the message to CTA `peer`; the last 16 threads also send
    // key and reciprocal to CTA `kpeer`
    const int peer = tid / M::UNITS, unit = tid % M::UNITS, kpeer = tid - (PC_T - 16);
    const uint32_t my_msg = pc_smem(recvA + rank * M::WORDS);
    const uint32_t dst_e = pc_map(my_msg + 16 * unit, peer < cs ? peer : 0), bar_e = pc_map(barA, peer < cs ? peer : 0);
    const uint32_t dst_k = pc_map(my_msg, kpeer >= 0 && kpeer < cs ? kpeer : 0);
    const uint32_t bar_k = pc_map(barA, kpeer >= 0 && kpeer < cs ? kpeer : 0);
    const C zero = cx_make<C>(0.0, 0.0);
    for (int jb = 0; jb < w; jb += PC_SUB) {
        const int sw = min(PC_SUB, w - jb), cend = jb + sw, sbp = (jb / PC_SUB) & 1;
        const bool trailing = cend < w;
        bool active = tid < myrows && s_done[tid] == 0;
        C a[PC_SUB];
#pragma unroll
        for (int k = 0; k < PC_SUB; ++k) a[k] = active && k < sw ? tile[(size_t)tid * LD + jb + k] : zero;
        int pend = -1, pend_k = 0;  // a pivot row of this CTA whose entries still have to go to the others
        auto publish = [&]() {
            if (pend < 0 || !trailing) return;
            for (int c = jb + tid; c < w; c += PC_T) {
                uint4* dst = grow + ((size_t)(sbp * PC_SUB + pend_k) * NB + (c - jb)) * E;
                const pc_word* v = reinterpret_cast<const pc_word*>(&tile[(size_t)pend * LD + c]);
#pragma unroll
                for (int e = 0; e < E; ++e) pc_put(dst + e, v[e], epoch + jb + pend_k + 1);
            }
        };
        for (int jj = 0; jj < sw; ++jj) {
            const int j = jb + jj, par = j & 1;
            const uint32_t ph = (j >> 1) & 1, bA = barA + 8 * par;
            // the warp's candidate: lanes are in row order, so the lowest lane is the lowest row
            const unsigned key = active ? __float_as_uint((float)cx_abs2<R>(a[0])) + 1u : 0u;
            const int top = pc_best(key), rem = sw - jj;  // rem: live entries of a
            C* sr = srow + par * PC_WARPS * PC_SUB;
            if (lane == top) {
                C* out = sr + warp * PC_SUB;
#pragma unroll
                for (int g = 0; g < PC_SUB; g += 4)
                    if (g < rem) {
#pragma unroll
                        for (int k = g; k < g + 4; k += 2) pc_store2(out + k, a[k], a[k + 1]);
                    }
                s_key[par][warp] = key;
                s_row[par][warp] = (unsigned)(row0 + tid);
            }
            __syncthreads();
            {
                // this CTA's candidate to every CTA of the cluster
                const int from = pc_best(lane < PC_WARPS ? s_key[par][lane] : 0u);
                const pc_word* cand = reinterpret_cast<const pc_word*>(sr + from * PC_SUB);
                const uint32_t at = par * cs * M::BYTES;
                if (peer < cs) pc_send2(dst_e + at, cand[2 * unit], cand[2 * unit + 1], bar_e + 8 * par);
                if (kpeer >= 0 && kpeer < cs) {  // the reciprocal follows while the entries travel
                    pc_send2(dst_k + at + 8 * M::KEY,
                             (pc_word)s_key[par][from] | ((pc_word)s_row[par][from] << 32), 0ull, bar_k + 8 * par);
                    const C pv = sr[from * PC_SUB];
                    const double den = (double)pv.x * pv.x + (double)pv.y * pv.y;
                    const double rd = __drcp_rn(den);
                    const double ir = den > 0.0 ? pv.x * rd : 0.0, ii = den > 0.0 ? -pv.y * rd : 0.0;
                    pc_send2(dst_k + at + 8 * M::INV, (pc_word)__double_as_longlong(ir),
                             (pc_word)__double_as_longlong(ii), bar_k + 8 * par);
                }
            }
            publish();
            pend = -1;
            pc_wait(bA, ph, status, quit);
            int from = pc_best(lane < cs ? (unsigned)recvA[(par * cs + lane) * M::WORDS + M::KEY] : 0u);
            const pc_word* msg = recvA + (par * cs + from) * M::WORDS;
            if (ncl > 1) {
                // the clusters' winners: the CTA that holds one publishes it, everyone reads them all
                uint4* slot = gkey + (size_t)par * PC_MAXCL * 36;
                const unsigned flag = epoch + j + 1;
                if (from == rank)
                    for (int t = tid; t < M::WORDS; t += PC_T) pc_put(slot + cl * 36 + t, msg[t], flag);
                for (int t = tid; t < ncl * M::WORDS; t += PC_T) {
                    const int c = t / M::WORDS, q = t - c * M::WORDS;
                    const uint4* src = slot + c * 36 + q;
                    gmsg[t] = c == cl ? msg[q] : pc_get(src, pc_peek(src), flag, status, quit);
                }
                __syncthreads();
                msg = gmsg + pc_best(lane < ncl ? (unsigned)gmsg[lane * M::WORDS + M::KEY] : 0u) * M::WORDS;
            }
            const int pr = (int)(msg[M::KEY] >> 32);
            const double ir = __longlong_as_double((long long)msg[M::INV]);
            const double ii = __longlong_as_double((long long)msg[M::INV + 1]);
            const bool nonzero = ir != 0.0 || ii != 0.0;
            if (active && row0 + tid == pr) {
                active = false;
                s_done[tid] = (short)(j + 1);
            } else if (active) {
                const C* u = reinterpret_cast<const C*>(msg);
                C l;
                l.x = (R)(a[0].x * ir - a[0].y * ii);
                l.y = (R)(a[0].x * ii + a[0].y * ir);
                tile[(size_t)tid * LD + j] = nonzero ? l : a[0];
                if (!nonzero) l = zero;
#pragma unroll
                for (int g = 0; g < PC_SUB; g += 4)
                    if (g + 1 < rem) {
#pragma unroll
                        for (int k = g; k < g + 4 && k + 1 < PC_SUB; ++k) a[k] = pc_sub(a[k + 1], l, u[k + 1]);
                    }
            }
            if (pr >= row0 && pr < row0 + myrows) {
                pend = pr - row0;
                pend_k = jj;
                // the row's U entries, from the message that carries them
                const int k = tid - (PC_T - 64);
                if (k >= 0 && k < rem) tile[(size_t)pend * LD + j + k] = reinterpret_cast<const C*>(msg)[k];
            }
            if (tid == PC_T - 1) {
                if (j + 2 < w) pc_expect(bA, cs * M::BYTES);  // this barrier's next column
                // the interchanges: piv[k0 + j] is the position that row pr has now
                s_prow[jj] = pr;
                if (pr >= k0 && pr < n) {
                    const int at = pr < k0 + w ? s_pos[pr - k0] : pr, s = s_at[j];
                    s_pos[s - k0] = at;
                    if (at < k0 + w) s_at[at - k0] = s;
                    if (blockIdx.x == 0) {
                        piv[k0 + j] = at;
                        if (!nonzero) atomicCAS(status, 0, 5);
                    }
                }
            }
        }
        __syncthreads();
        if (!trailing) continue;
        publish();
        {
            // the 16 pivot rows over columns jb .. w - 1
            constexpr int RW = NB * E, RP = PC_T / RW;  // words of a row, rows per pass
            static_assert(RW * RP == PC_T && PC_SUB % RP == 0, "threads cover whole rows");
            const int e = tid % RW, kr = tid / RW;
            const uint4* src = grow + (size_t)sbp * PC_SUB * RW + e;
            if (e < (w - jb) * E) {
                uint4 v[PC_SUB / RP];
#pragma unroll
                for (int q = 0; q < PC_SUB / RP; ++q) v[q] = pc_peek(src + (size_t)(kr + q * RP) * RW);
#pragma unroll
                for (int q = 0; q < PC_SUB / RP; ++q) {
                    const int k = kr + q * RP;
                    reinterpret_cast<pc_word*>(pbuf + (size_t)k * NB + jb)[e] =
                        pc_get(src + (size_t)k * RW, v[q], epoch + jb + k + 1, status, quit);
                }
            }
        }
        __syncthreads();
        for (int c = cend + tid; c < w; c += PC_T) {  // forward substitution, a column per thread
            C u[PC_SUB];
#pragma unroll
            for (int k = 0; k < PC_SUB; ++k) u[k] = pbuf[(size_t)k * NB + c];
#pragma unroll
            for (int k = 0; k < PC_SUB; ++k) {
#pragma unroll
                for (int i = k + 1; i < PC_SUB; ++i) u[i] = pc_sub(u[i], pbuf[(size_t)i * NB + jb + k], u[k]);
                pbuf[(size_t)k * NB + c] = u[k];
            }
        }
        __syncthreads();
        const int nt = w - cend;
        for (int k = warp; k < PC_SUB; k += PC_WARPS) {
            const int r = s_prow[k] - row0;
            if (r >= 0 && r < myrows)
                for (int c = cend + lane; c < w; c += 32) tile[(size_t)r * LD + c] = pbuf[(size_t)k * NB + c];
        }
        // rank-16 update of the other rows: lanes over rows, warps over groups of G columns
        constexpr int G = sizeof(R) == 4 ? 8 : 4;
        const int ng = (nt + G - 1) / G;
        for (int gq = warp; gq < ng; gq += PC_WARPS) {
            const int c0 = cend + gq * G;
            for (int r = lane; r < myrows; r += 32) {
                if (s_done[r]) continue;
                C* trow = tile + (size_t)r * LD;
                C acc[G];
#pragma unroll
                for (int k = 0; k < G; ++k) acc[k] = trow[c0 + k];
#pragma unroll 4
                for (int i = 0; i < PC_SUB; ++i) {
                    const C l = trow[jb + i];
                    const C* u = pbuf + (size_t)i * NB + c0;
#pragma unroll
                    for (int k = 0; k < G; k += 2) {
                        C u0, u1;
                        pc_load2(u + k, u0, u1);
                        acc[k] = pc_sub(acc[k], l, u0);
                        acc[k + 1] = pc_sub(acc[k + 1], l, u1);
                    }
                }
#pragma unroll
                for (int k = 0; k < G; ++k)
                    if (c0 + k < w) trow[c0 + k] = acc[k];
            }
        }
        __syncthreads();
    }
    // every CTA has read its rows of A long ago (it took part in the exchanges): write them back
    for (int r = lane; r < myrows; r += 32) {
        const int g = row0 + r, d = s_done[r];
        const int dst = d ? k0 + d - 1 : (g < k0 + w ? s_pos[g - k0] : g);
        for (int c = warp; c < w; c += PC_WARPS) A[(size_t)(k0 + c) * lda + dst] = tile[(size_t)r * LD + c];
    }
    if (*quit) __nanosleep(20000);  // messages on their way when the waits gave up
    __syncthreads();
    pc_cluster_barrier();  // no CTA leaves while another may still send to it
}

}  // namespace tcu
