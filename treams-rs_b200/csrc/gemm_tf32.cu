// Trailing update of the mixed-precision LU on the 5th-generation tensor cores:
//   A22 -= L21 U12   (complex64, column-major, in place)
// as one real GEMM D = Lemb * U^T with
//   Lemb[2mu+c][2k+c'] = { Re L, -Im L ; Im L, Re L }   (2m x 2w, K-major)
//   U[nu][2k+c']       = interleaved (Re, Im) of column nu of U12   (n' x 2w, K-major)
// so that D[2mu+c][nu] is part c of (L21 U12)[mu][nu] and the 2m x n' result maps onto
// the interleaved storage of A22 (real leading dimension 2n).
//
// Precision: every operand is split x = hi + lo into two pieces and the passes accumulate in FP32
// in TMEM. Formats (TCU_SPLIT):
//   bfloat16 (default): hi = bf16(x), lo = bf16(x - hi), 16 significant bits at the FP32 exponent range;
//     three passes hi*hi + hi*lo + lo*hi of tcgen05.mma kind::f16, the dropped lo*lo and the rounding
//     of lo leave about 2^-17 of |a||b| per term. Twice the TF32 rate: 1.5 TF32 passes of tensor time.
//   tf32x2: hi = tf32(x), lo = tf32(x - hi), two passes hi*hi + lo*hi of kind::tf32, the B operand rounded
//     to TF32: about 2^-12 per term at 2 TF32 passes. 24576 modes, all updates of a factorization: 128 ms
//     and a first residual of 2.5e-6, against 105 ms and 2.1e-7 of the bfloat16 pieces on single CTAs (9600 modes: 8.7 ms and
//     1.6e-6 against 7.2 ms and 1.7e-7), and the packing kernels write half the bytes (8.1 against 7.0 ms).
//   tf32x3: the same pieces in three passes, 2^-22 per term; the format of fallback factors.
//   f16: each row of each operand (a complex row of L21, a column of U12) is first scaled by its own
//     power of two 2^(14 - ceil log2 max|row|) (computed in the packing kernels; no host round trip),
//     hi = f16(x s), lo = f16(x s - hi); three passes of kind::f16, and the epilogue multiplies each
//     accumulator entry by the exact power of two 1/(s_row s_col). Pieces below the FP16 normal
//     range only lose absolute accuracy under 2^-38 of their row's maximum.
//
// Kernel layout (persistent, one CTA per SM, 192 threads, CTAs in pairs): a pair forms a 256 x 256 tile with
// cta_group::2 products, each CTA staging its 128 rows of the A pieces and half of the B rows, so a chunk
// brings 32 KB into an SM instead of 48. One CTA per 128 x 256 tile drew 64 bytes a clock and SM from L2, more than
// L2 gives: 24576 modes 105 -> 90 ms (1.33 PFLOP/s executed, 94 % of the sustained bf16 rate), 17150 modes 37 -> 32.
//   warp 0     TMA producer of each CTA: 64-byte-swizzled boxes (64-byte K rows) of the four packed operands
//              into a 6-stage shared-memory ring (32 KB per stage), complete_tx on the leader's mbarrier;
//   warp 1     TMEM allocator; in the leader the MMA issuer (one thread): 2 K-steps x 2 or 3 passes per stage
//              into both CTAs' 128 x 256 FP32 accumulators, double-buffered in TMEM (512 columns); its
//              commits free the stages and publish the accumulators in both CTAs;
//   warps 2-5  epilogue of the CTA's 128 rows: tcgen05.ld 32 columns at a time into a shared-memory staging
//              buffer, TMA reduce-add of -D into A22.
// Every mbarrier wait is bounded; on timeout the kernel records status 8, drains its TMA
// loads, frees TMEM and returns (the pair's last barrier is reached by both CTAs in any case).
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>

#include "kernels.h"
#include "precond.h"

namespace tcu {

constexpr int TB_M = 128;       // real rows of a CTA (64 complex rows); a pair of CTAs takes 256
constexpr int TB_N = 256;       // columns per tile; each CTA of the pair stages half of them
constexpr int TB_K = 16;        // floats per K chunk (one 64-byte swizzle row); 32 for 2-byte pieces
constexpr int TB_STAGES = 6;
constexpr int A_BYTES = TB_M * TB_K * 4;   // 8 KB
constexpr int B_BYTES = TB_N / 2 * TB_K * 4;  // 8 KB
constexpr int STAGE_BYTES = 2 * A_BYTES + 2 * B_BYTES;  // 32 KB
constexpr int TMEM_COLS = 2 * TB_N;        // two accumulators
constexpr int EPI_COLS = 32;                         // columns per epilogue staging buffer
constexpr int EPI_BYTES = TB_M * EPI_COLS * 4;         // 16 KB
constexpr size_t TF32_SMEM = (size_t)TB_STAGES * STAGE_BYTES + 2 * EPI_BYTES + 1024 + 256;

// ---- device helpers ---------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
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
// Bounded wait: false after 2 s or when another role has aborted.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          unsigned long long limit_ns = 2000000000ull) {
    if (mbar_try(bar, parity)) return true;
    unsigned long long t0 = gtimer();
    for (unsigned it = 1;; ++it) {
        if (mbar_try(bar, parity)) return true;
        if ((it & 63u) == 0) {
            if (*abort_flag) return false;
            if (gtimer() - t0 > limit_ns) {
                *abort_flag = 1;
                return false;
            }
        }
    }
}

// This wait on a barrier without arrivals.
__global__ void update_wait_selftest_kernel(int* status, unsigned long long limit_ns) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ int abort_flag;
    mbar_init(smem_u32(&bar), 1);
    abort_flag = 0;
    if (!mbar_wait(smem_u32(&bar), 0, &abort_flag, limit_ns)) atomicExch(status, 8);
}
void launch_update_wait_selftest(int* status, double limit_s, cudaStream_t st) {
    update_wait_selftest_kernel<<<1, 1, 0, st>>>(status, selftest_ns(limit_s));
}

// The leader's (rank 0) barrier of the pair, as a shared::cluster address.
__device__ __forceinline__ uint32_t leader_bar(uint32_t bar) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(bar));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void pair_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// into this CTA's shared memory, completing on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];" ::"r"(dst),
        "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// K-major, 64-byte swizzled operand tile: rows of 16 floats, 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t swz_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;             // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(512 >> 4) << 32;    // stride byte offset: next 8-row group
    d |= (uint64_t)1 << 46;             // descriptor version (sm_100)
    d |= (uint64_t)4 << 61;             // SWIZZLE_64B
    return d;
}

// Tile t of the persistent loop: groups of 16 M-tiles (of 256 rows) sweep all N-tiles, so the CTAs in
// flight share a few A and B tiles in L2.
constexpr int TILE_GROUP = 16;
__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int& tm, int& tn) {
    int per_group = TILE_GROUP * tiles_n;
    int g = t / per_group;
    int first = g * TILE_GROUP;
    int gm = min(TILE_GROUP, tiles_m - first);
    int local = t - g * per_group;
    tm = first + local % gm;
    tn = local / gm;
}

__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
template <bool HALF>
__device__ __forceinline__ void mma_split(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    if (HALF)
        mma_f16(d_tmem, a, b, idesc, acc);
    else
        mma_tf32(d_tmem, a, b, idesc, acc);
}
// Power-of-two scale that maps max |x| to (2^13, 2^14]: exact, and far inside the FP16 range.
__device__ __forceinline__ float f16_scale(float mx) {
    if (!(mx > 0.0f) || !isfinite(mx)) return 1.0f;
    int e;
    frexpf(mx, &e);  // mx = f 2^e, 0.5 <= f < 1
    return ldexpf(1.0f, 14 - e);
}
// arrives on the barrier at this place in both CTAs of the pair
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
        "h"((uint16_t)3)
        : "memory");
}
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// ---- the GEMM ---------------------------------------------------------------------------
struct Tf32Args {
    float* C;        // A viewed as floats
    size_t ldc;      // 2n (floats per column)
    int row0;        // 2 r0: first real row of A22
    int col0;        // r0
    int m2;          // real rows of A22 (2m)
    int ncols;       // columns of A22
    int kchunks;     // K / TB_K
    int tiles_m, tiles_n, tiles;
    int* status;
    const float* sA;      // FP16 pieces: scale of each complex row of the A operand (m2 / 2), else null
    const float* sB;      // FP16 pieces: scale of each row of the B operand (ncols)
};

template <int PIECES>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(192, 1) tf32_update_kernel(const __grid_constant__ CUtensorMap mAhi,
                                                             const __grid_constant__ CUtensorMap mAlo,
                                                             const __grid_constant__ CUtensorMap mBhi,
                                                             const __grid_constant__ CUtensorMap mBlo,
                                                             const __grid_constant__ CUtensorMap mC, Tf32Args args) {
    // 2-byte pieces (kind::f16), rows with scales, two passes
    constexpr bool HALF = PIECES == PIECES_F16 || PIECES == PIECES_BF16, F16 = PIECES == PIECES_F16;
    constexpr bool TWO = PIECES == PIECES_TF32X2;
    constexpr int KC = HALF ? 2 * TB_K : TB_K;  // K elements of a chunk (64 bytes)
    extern __shared__ uint8_t smem_raw[];
    uint32_t base = smem_u32(smem_raw);
    uint32_t tiles_smem = (base + 1023u) & ~1023u;  // 1024-byte aligned stage ring
    const uint32_t epi_smem = tiles_smem + TB_STAGES * STAGE_BYTES;  // 2 staging buffers
    float* epi = (float*)(smem_raw + (epi_smem - base));
    uint8_t* ctrl = smem_raw + (tiles_smem - base) + TB_STAGES * STAGE_BYTES + 2 * EPI_BYTES;
    // barriers: full[S], empty[S], tmem_full[2], tmem_empty[2]
    uint64_t* bars = (uint64_t*)ctrl;
    uint32_t* tmem_slot = (uint32_t*)(ctrl + 8 * (2 * TB_STAGES + 4));
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)cta_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    auto bar = [&](int i) { return smem_u32(&bars[i]); };
    constexpr int EMPTY = TB_STAGES, TFULL = 2 * TB_STAGES, TEMPTY = 2 * TB_STAGES + 2;
    if (threadIdx.x == 0) {
        for (int s = 0; s < TB_STAGES; ++s) {
            mbar_init(bar(s), 1);
            mbar_init(bar(EMPTY + s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(bar(TFULL + a), 1);
            mbar_init(bar(TEMPTY + a), 2);  // (the leader's: one arrival per CTA)
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    __syncthreads();
    pair_sync();  // both CTAs' barriers are ready, both have their TMEM
    fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int step = 0;
            for (int t = pair; t < args.tiles && !*abort_flag; t += pairs) {
                int tm, tn;
                tile_coords(t, args.tiles_m, args.tiles_n, tm, tn);
                for (int kb = 0; kb < args.kchunks; ++kb, ++step) {
                    int s = step % TB_STAGES;
                    uint32_t ph = (step / TB_STAGES) & 1;
                    if (!mbar_wait(bar(EMPTY + s), ph ^ 1, abort_flag)) break;
                    uint32_t st = tiles_smem + s * STAGE_BYTES;
                    // the leader's barrier counts the bytes of both CTAs (the other's may come before this)
                    if (rank == 0) mbar_expect_tx(bar(s), 2 * (TWO ? STAGE_BYTES - B_BYTES : STAGE_BYTES));
                    const uint32_t fb = leader_bar(bar(s));
                    const int ya = (2 * tm + rank) * TB_M, yb = tn * TB_N + rank * (TB_N / 2);
                    tma_load_2d(st, &mAhi, kb * KC, ya, fb);
                    tma_load_2d(st + A_BYTES, &mAlo, kb * KC, ya, fb);
                    tma_load_2d(st + 2 * A_BYTES, &mBhi, kb * KC, yb, fb);
                    if (!TWO) tma_load_2d(st + 2 * A_BYTES + B_BYTES, &mBlo, kb * KC, yb, fb);
                }
            }
            if (*abort_flag && rank == 0) {
                // drain: wait (bounded) for both CTAs' loads of every stage still in flight; the other CTA
                // stays until the pair's last barrier
                volatile int never = 0;
                for (int s = 0; s < TB_STAGES; ++s) {
                    int last = step - 1 - ((step - 1 - s) % TB_STAGES + TB_STAGES) % TB_STAGES;
                    if (last >= 0) mbar_wait(bar(s), (last / TB_STAGES) & 1, &never);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            // D F32; A, B TF32 (2), BF16 (1) or F16 (0); K-major; N >> 3 at bit 17, M >> 4 at bit 24
            const uint32_t ab = F16 ? 0u : (HALF ? 1u : 2u);
            const uint32_t idesc = (1u << 4) | (ab << 7) | (ab << 10) | ((uint32_t)(TB_N >> 3) << 17) |
                                   ((uint32_t)(2 * TB_M >> 4) << 24);
            int step = 0, it = 0;
            for (int t = pair; t < args.tiles && !*abort_flag; t += pairs, ++it) {
                int acc = it & 1;
                uint32_t aph = (it >> 1) & 1;
                if (!mbar_wait(bar(TEMPTY + acc), aph ^ 1, abort_flag)) break;
                fence_after();
                uint32_t d = tmem_base + (uint32_t)(acc * TB_N);
                bool ok = true;
                for (int kb = 0; kb < args.kchunks; ++kb, ++step) {
                    int s = step % TB_STAGES;
                    uint32_t ph = (step / TB_STAGES) & 1;
                    if (!mbar_wait(bar(s), ph, abort_flag)) {
                        ok = false;
                        break;
                    }
                    fence_after();
                    uint32_t st = tiles_smem + s * STAGE_BYTES;
#pragma unroll
                    for (int ks = 0; ks < 2; ++ks) {  // two 32-byte K-steps per 64-byte row
                        uint64_t ahi = swz_desc(st + ks * 32), alo = swz_desc(st + A_BYTES + ks * 32);
                        uint64_t bhi = swz_desc(st + 2 * A_BYTES + ks * 32);
                        uint64_t blo = swz_desc(st + 2 * A_BYTES + B_BYTES + ks * 32);
                        uint32_t first = (kb == 0 && ks == 0) ? 0u : 1u;
                        mma_split<HALF>(d, ahi, bhi, idesc, first);
                        if (!TWO) mma_split<HALF>(d, ahi, blo, idesc, 1u);
                        mma_split<HALF>(d, alo, bhi, idesc, 1u);
                    }
                    mma_commit(bar(EMPTY + s));
                }
                if (!ok) break;
                mma_commit(bar(TFULL + acc));
            }
        }
    } else {
        // Epilogue: -D goes through a shared-memory staging buffer ([64 columns][128 rows])
        // and a TMA reduce-add into A22 in L2, so no thread waits on a load of A22.
        const int q = warp & 3;  // TMEM lane quarter of this warp
        const int R = q * 32 + lane;
        const bool issuer = (warp == 2 && lane == 0);
        volatile int* s_go = abort_flag + 1;  // the issuer's wait result, shared by the 4 warps
        // FP16 pieces: -1 / (row scale x column scale) undoes the operand scaling exactly
        const int grow = R;  // row of the tile this thread stores
        int it = 0, e = 0;
        for (int t = pair; t < args.tiles; t += pairs, ++it) {
            int acc = it & 1;
            uint32_t aph = (it >> 1) & 1;
            // one thread waits (bounded) and the four warps take its decision together, so a
            // time-out cannot leave some of them at the named barrier
            if (issuer) *s_go = (!*abort_flag && mbar_wait(bar(TFULL + acc), aph, abort_flag)) ? 1 : 0;
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (!*s_go) break;
            fence_after();
            int tm, tn;
            tile_coords(t, args.tiles_m, args.tiles_n, tm, tn);
            const int row0 = (2 * tm + rank) * TB_M;  // this CTA's first row
            float rowneg = -1.0f;
            if (F16) {
                const int mu = (row0 + grow) >> 1;
                rowneg = mu < (args.m2 >> 1) ? -1.0f / __ldg(&args.sA[mu]) : -1.0f;
            }
            // columns and rows past the block: nothing to add
            const int subs = row0 < args.m2 ? (min(TB_N, args.ncols - tn * TB_N) + EPI_COLS - 1) / EPI_COLS : 0;
            for (int sub = 0; sub < subs; ++sub, ++e) {
                const int buf = e & 1;
                if (issuer) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                asm volatile("bar.sync 1, 128;" ::: "memory");
                float* stage = epi + buf * (TB_M * EPI_COLS);
#pragma unroll
                for (int cb = 0; cb < EPI_COLS / 32; ++cb) {
                    float v[32];
                    uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) +
                                     (uint32_t)(acc * TB_N + sub * EPI_COLS + cb * 32);
                    tmem_ld32(taddr, v);
#pragma unroll
                    for (int jj = 0; jj < 32; ++jj) {
                        float f = rowneg;
                        if (F16) {
                            const int col = tn * TB_N + sub * EPI_COLS + cb * 32 + jj;
                            f = col < args.ncols ? rowneg / __ldg(&args.sB[col]) : rowneg;
                        }
                        stage[(cb * 32 + jj) * TB_M + R] = f * v[jj];
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (issuer) {
                    int x = args.row0 + row0, y = args.col0 + tn * TB_N + sub * EPI_COLS;
                    asm volatile(
                        "cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                            (uint64_t)&mC),
                        "r"(x), "r"(y), "r"(epi_smem + buf * EPI_BYTES)
                        : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
            fence_before();
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (issuer) mbar_arrive_cluster(leader_bar(bar(TEMPTY + acc)));
        }
        if (issuer) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    pair_sync();  // no product still reads the other CTA's stages, no arrival is on its way there
    if (*abort_flag && threadIdx.x == 0) atomicExch(args.status, 8);
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS));
    }
}

// ---- operand packing ----------------------------------------------------------------------
__device__ __forceinline__ float tf32_rna(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}
__device__ __forceinline__ void split(float x, float& hi, float& lo) {
    hi = tf32_rna(x);
    lo = tf32_rna(x - hi);
}

// Lemb hi/lo (2m x kp floats, row-major): a 32 x 32 complex tile through shared memory.
__global__ void pack_l_kernel(const float2* __restrict__ A, size_t lda, int r0, int k0, int m, int w, int kp,
                              float* __restrict__ hi, float* __restrict__ lo) {
    __shared__ float2 tile[32][33];
    int mu0 = blockIdx.x * 32, k00 = blockIdx.y * 32;
    int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    for (int r = ty; r < 32; r += 8) {
        int kk = k00 + r, mu = mu0 + tx;
        tile[r][tx] = (kk < w && mu < m) ? A[(size_t)(k0 + kk) * lda + r0 + mu] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        int mu = mu0 + r, kk = k00 + tx;
        if (mu >= m || 2 * kk >= kp) continue;
        float2 l = tile[tx][r];
        float rh, rl, ih, il;
        split(l.x, rh, rl);
        split(l.y, ih, il);
        size_t o0 = (size_t)(2 * mu) * kp + 2 * kk, o1 = o0 + kp;
        *(float2*)(hi + o0) = make_float2(rh, -ih);
        *(float2*)(hi + o1) = make_float2(ih, rh);
        *(float2*)(lo + o0) = make_float2(rl, -il);
        *(float2*)(lo + o1) = make_float2(il, rl);
    }
}

// U hi/lo (n' x kp floats, row-major): row nu = interleaved column nu of U12. lo may be null
// (the two-pass split reads only hi, U12 rounded to TF32).
__global__ void pack_u_kernel(const float2* __restrict__ A, size_t lda, int r0, int k0, int ncols, int w, int kp,
                              float* __restrict__ hi, float* __restrict__ lo) {
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    int half = kp / 2;
    if (t >= (size_t)ncols * half) return;
    int nu = (int)(t / half), kk = (int)(t % half);
    float2 u = kk < w ? A[(size_t)(r0 + nu) * lda + k0 + kk] : make_float2(0.f, 0.f);
    float rh, rl, ih, il;
    split(u.x, rh, rl);
    split(u.y, ih, il);
    size_t o = (size_t)nu * kp + 2 * kk;
    *(float2*)(hi + o) = make_float2(rh, ih);
    if (lo) *(float2*)(lo + o) = make_float2(rl, il);
}

// The same operands as bfloat16 pieces (kp multiple of 32; K of any number of panels).
__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16& hi, __nv_bfloat16& lo) {
    hi = __float2bfloat16_rn(x);
    lo = __float2bfloat16_rn(x - __bfloat162float(hi));
}
__global__ void pack_l_bf16_kernel(const float2* __restrict__ A, size_t lda, int r0, int k0, int m, int w, int kp,
                                   __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo) {
    __shared__ float2 tile[32][33];
    const int mu0 = blockIdx.x * 32, k00 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    for (int r = ty; r < 32; r += 8) {
        const int kk = k00 + r, mu = mu0 + tx;
        tile[r][tx] = (kk < w && mu < m) ? A[(size_t)(k0 + kk) * lda + r0 + mu] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int mu = mu0 + r, kk = k00 + tx;
        if (mu >= m || 2 * kk >= kp) continue;
        const float2 l = tile[tx][r];
        __nv_bfloat16 rh, rl, ih, il;
        split_bf16(l.x, rh, rl);
        split_bf16(l.y, ih, il);
        const size_t o0 = (size_t)(2 * mu) * kp + 2 * kk, o1 = o0 + kp;
        *(__nv_bfloat162*)(hi + o0) = __halves2bfloat162(rh, __hneg(ih));
        *(__nv_bfloat162*)(hi + o1) = __halves2bfloat162(ih, rh);
        *(__nv_bfloat162*)(lo + o0) = __halves2bfloat162(rl, __hneg(il));
        *(__nv_bfloat162*)(lo + o1) = __halves2bfloat162(il, rl);
    }
}
__global__ void pack_u_bf16_kernel(const float2* __restrict__ A, size_t lda, int r0, int k0, int ncols, int w, int kp,
                                   __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo) {
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int half = kp / 2;
    if (t >= (size_t)ncols * half) return;
    const int nu = (int)(t / half), kk = (int)(t % half);
    const float2 u = kk < w ? A[(size_t)(r0 + nu) * lda + k0 + kk] : make_float2(0.f, 0.f);
    __nv_bfloat16 rh, rl, ih, il;
    split_bf16(u.x, rh, rl);
    split_bf16(u.y, ih, il);
    const size_t o = (size_t)nu * kp + 2 * kk;
    *(__nv_bfloat162*)(hi + o) = __halves2bfloat162(rh, ih);
    *(__nv_bfloat162*)(lo + o) = __halves2bfloat162(rl, il);
}

// ---- FP16 pieces -----------------------------------------------------------------------
// Every row of the A operand (complex row mu of L21, both its real rows) and every row of the
// B operand (column nu of U12) gets its own power-of-two scale f16_scale(max over its K
// entries), so each row's pieces keep 22 bits relative to that row's largest entry.

__device__ __forceinline__ void split16(float x, float s, __half& hi, __half& lo) {
    float xs = x * s;
    hi = __float2half_rn(xs);
    lo = __float2half_rn(xs - __half2float(hi));
}

// Lemb pieces (2m x kp halves, row-major) of 32 complex rows per CTA (K <= 256 real, i.e.
// w <= 128); sign -1 negates. sA[mu] receives the row's scale.
__global__ void __launch_bounds__(256) pack_l16_kernel(const float2* __restrict__ A, size_t lda, int r0, int k0, int m,
                                                       int w, int kp, float sign, __half* __restrict__ hi,
                                                       __half* __restrict__ lo, float* __restrict__ sA) {
    __shared__ float2 tile[128][33];  // [kk][mu]
    __shared__ float scale[32];
    const int mu0 = blockIdx.x * 32, half = kp / 2;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    for (int kk = ty; kk < half; kk += 8) {
        int mu = mu0 + tx;
        tile[kk][tx] = (kk < w && mu < m) ? A[(size_t)(k0 + kk) * lda + r0 + mu] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {  // warp ty: rows r; lanes over K
        float mx = 0.0f;
        for (int kk = tx; kk < half; kk += 32) mx = fmaxf(mx, fmaxf(fabsf(tile[kk][r].x), fabsf(tile[kk][r].y)));
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (tx == 0) {
            float sc = f16_scale(mx);
            scale[r] = sign * sc;
            if (mu0 + r < m) sA[mu0 + r] = sc;
        }
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int mu = mu0 + r;
        if (mu >= m) continue;
        const float sc = scale[r];
        for (int kk = tx; kk < half; kk += 32) {
            float2 l = tile[kk][r];
            __half rh, rl, ih, il;
            split16(l.x, sc, rh, rl);
            split16(l.y, sc, ih, il);
            size_t o0 = (size_t)(2 * mu) * kp + 2 * kk, o1 = o0 + kp;
            *(__half2*)(hi + o0) = __halves2half2(rh, __hneg(ih));
            *(__half2*)(hi + o1) = __halves2half2(ih, rh);
            *(__half2*)(lo + o0) = __halves2half2(rl, __hneg(il));
            *(__half2*)(lo + o1) = __halves2half2(il, rl);
        }
    }
}

// U pieces (n' x kp halves, row-major): row nu = interleaved column nu of U12; one warp per
// row, sB[nu] its scale.
__global__ void __launch_bounds__(256) pack_u16_kernel(const float2* __restrict__ A, size_t lda, int r0, int k0,
                                                       int ncols, int w, int kp, __half* __restrict__ hi,
                                                       __half* __restrict__ lo, float* __restrict__ sB) {
    const int nu = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (nu >= ncols) return;
    const int half = kp / 2;
    float2 u[4];  // kp / 2 <= 128 values per row
    float mx = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        int kk = lane + 32 * q;
        u[q] = (kk < w && kk < half) ? A[(size_t)(r0 + nu) * lda + k0 + kk] : make_float2(0.f, 0.f);
        mx = fmaxf(mx, fmaxf(fabsf(u[q].x), fabsf(u[q].y)));
    }
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float sc = f16_scale(mx);
    if (lane == 0) sB[nu] = sc;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        int kk = lane + 32 * q;
        if (kk >= half) continue;
        __half rh, rl, ih, il;
        split16(u[q].x, sc, rh, rl);
        split16(u[q].y, sc, ih, il);
        size_t o = (size_t)nu * kp + 2 * kk;
        *(__half2*)(hi + o) = __halves2half2(rh, ih);
        *(__half2*)(lo + o) = __halves2half2(rl, il);
    }
}

// ---- host -------------------------------------------------------------------------------
typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiled encoder() {
    static const EncodeTiled fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return (EncodeTiled)p;
        return (EncodeTiled) nullptr;
    }();
    return fn;
}

// K-major operand of `rows` rows of kp elements (4-byte TF32 pieces or 2-byte FP16 or bfloat16 pieces);
// boxes are one 64-byte swizzle row deep (16 or 32 elements).
static bool make_map(CUtensorMap* map, void* base, int rows, int kp, int box_rows, PieceFormat pieces) {
    EncodeTiled enc = encoder();
    if (!enc) return false;
    const int eb = pieces == PIECES_F16 || pieces == PIECES_BF16 ? 2 : 4;
    const CUtensorMapDataType type = pieces == PIECES_F16    ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                     : pieces == PIECES_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                             : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    cuuint64_t dims[2] = {(cuuint64_t)kp, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)kp * eb};
    cuuint32_t box[2] = {(cuuint32_t)(64 / eb), (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return enc(map, type, 2, base, dims, strides, box,
               estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr int TI_W = 128, TI_LD = TI_W + 1;  // order of L11, its row pitch
constexpr int TI_S = 16, TI_C = 8;           // rows of a block, columns of the inverse per CTA
constexpr size_t TI_SMEM = (size_t)(TI_W * TI_LD + TI_W * (TI_S + 1) + (TI_W + TI_S) * TI_C) * sizeof(float2);
__global__ void tri_inverse_l_kernel(const float2* __restrict__ A, size_t lda, int k0, float* __restrict__ hi,
                                     float* __restrict__ lo, float2* __restrict__ N);

// bfloat16 pieces are the fastest and as accurate as FP32 panels allow (see the top). FP16 pieces reach the
// same residuals, but their epilogue divides every entry by its scales and they keep one update per panel:
// 380 ms of updates at 24576 modes. A refinement that stalls on any other format falls back to a three-pass
// TF32 factor.
PieceFormat split_default() {
    static const PieceFormat f = [] {
        const char* e = getenv("TCU_SPLIT");
        if (e && std::strcmp(e, "tf32x3") == 0) return PIECES_TF32X3;
        if (e && std::strcmp(e, "tf32x2") == 0) return PIECES_TF32X2;
        if (e && std::strcmp(e, "f16") == 0) return PIECES_F16;
        return PIECES_BF16;
    }();
    return f;
}

bool tf32_enabled() {
    static const int on = [] {
        const char* e = getenv("TCU_DISABLE_TCGEN05");
        return (e && e[0] == '1') || !encoder() ? 0 : 1;
    }();
    if (on == 1) {
        static PerDeviceOnce attr;
        once_per_device(attr, [] {
            cudaFuncSetAttribute(tf32_update_kernel<PIECES_TF32X3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)TF32_SMEM);
            cudaFuncSetAttribute(tf32_update_kernel<PIECES_TF32X2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)TF32_SMEM);
            cudaFuncSetAttribute(tf32_update_kernel<PIECES_F16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)TF32_SMEM);
            cudaFuncSetAttribute(tf32_update_kernel<PIECES_BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)TF32_SMEM);
            cudaFuncSetAttribute(tri_inverse_l_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TI_SMEM);
        });
    }
    return on == 1;
}

// N = L11^-1 - I for the unit lower 128 x 128 diagonal block of a panel, in FP32: one CTA per 8 columns of
// the inverse, none waiting for another. Each inverts the 16 x 16 diagonal blocks it needs (a warp per block,
// a lane per row and 8 columns) and substitutes downwards block by block, X_i = L_ii^-1 R_i, R -= L_:i X_i,
// with R in registers (a thread per row and 4 columns): one shared-memory load of L serves four products.
// U12 = L11^-1 A12 = A12 + N A12 then runs on the tensor cores: hi/lo receive the TF32 pieces of -N,
// embedded as in pack_l_kernel, and N (where not null) the matrix, column-major.
// A chain of 16 short steps bounds it. One CTA that joined inverted blocks at 16, 32 and 64 rows read two
// operands from shared memory per product: 50 us against 13, and packing and negating took two more launches.
__device__ __forceinline__ void fmac(float2& s, float2 a, float2 b) {
    s.x += a.x * b.x - a.y * b.y;
    s.y += a.x * b.y + a.y * b.x;
}
__global__ void __launch_bounds__(256) tri_inverse_l_kernel(const float2* __restrict__ A, size_t lda, int k0,
                                                            float* __restrict__ hi, float* __restrict__ lo,
                                                            float2* __restrict__ N) {
    extern __shared__ __align__(16) float2 ti_smem[];
    float2* X = ti_smem;               // this CTA's columns of the inverse, X[i * TI_C + c]
    float2* S = X + TI_W * TI_C;       // R of the block in turn
    float2* M = S + TI_S * TI_C;       // L11, M[i * TI_LD + k], i > k
    float2* D = M + TI_W * TI_LD;      // inverted diagonal blocks, D[i * (TI_S + 1) + m], i < 128
    const int o = blockIdx.x * TI_C, b0 = o / TI_S;  // first column, first block
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row = tid & (TI_W - 1), g = tid >> 7;  // this thread's R: columns 4 g .. 4 g + 3 of the row
    for (int k = b0 * TI_S + g; k < row; k += 2)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(&M[row * TI_LD + k])),
                     "l"(A + (size_t)(k0 + k) * lda + k0 + row)
                     : "memory");
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (warp >= b0) {
        const int d = warp * TI_S, r = lane & 15, c0 = (lane >> 4) * 8;
        float2 x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = make_float2(r == c0 + u ? 1.0f : 0.0f, 0.0f);
#pragma unroll 1
        for (int k = 0; k < TI_S - 1; ++k) {
            float2 l = make_float2(0.0f, 0.0f);
            if (r > k) l = M[(d + r) * TI_LD + d + k];
            l.x = -l.x;
            l.y = -l.y;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float2 xk = make_float2(__shfl_sync(0xffffffffu, x[u].x, k, 16),
                                              __shfl_sync(0xffffffffu, x[u].y, k, 16));
                fmac(x[u], l, xk);
            }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) D[(d + r) * (TI_S + 1) + c0 + u] = x[u];
    }
    float2 R[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) R[u] = make_float2(row == o + 4 * g + u ? 1.0f : 0.0f, 0.0f);
    const int pr = tid >> 4, pc = (tid >> 1) & 7, ph = tid & 1;  // product: row, column, half of the sum
#pragma unroll 1
    for (int b = b0; b < TI_W / TI_S; ++b) {
        if (row >> 4 == b) {
#pragma unroll
            for (int u = 0; u < 4; ++u) S[(row & 15) * TI_C + 4 * g + u] = R[u];
        }
        __syncthreads();
        float2 s = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int m = 0; m < 8; ++m) fmac(s, D[(b * TI_S + pr) * (TI_S + 1) + ph * 8 + m], S[(ph * 8 + m) * TI_C + pc]);
        s.x += __shfl_xor_sync(0xffffffffu, s.x, 1);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, 1);
        if (ph == 0) X[(b * TI_S + pr) * TI_C + pc] = s;
        __syncthreads();
        if (row >> 4 > b) {
#pragma unroll
            for (int k = 0; k < TI_S; ++k) {
                float2 l = M[row * TI_LD + b * TI_S + k];
                l.x = -l.x;
                l.y = -l.y;
                const float4 x01 = *(const float4*)&X[(b * TI_S + k) * TI_C + 4 * g];
                const float4 x23 = *(const float4*)&X[(b * TI_S + k) * TI_C + 4 * g + 2];
                fmac(R[0], l, make_float2(x01.x, x01.y));
                fmac(R[1], l, make_float2(x01.z, x01.w));
                fmac(R[2], l, make_float2(x23.x, x23.y));
                fmac(R[3], l, make_float2(x23.z, x23.w));
            }
        }
    }
    constexpr int kp = 2 * TI_W;
    for (int idx = tid; idx < TI_W * TI_C; idx += 256) {
        const int k = idx % TI_C, i = idx / TI_C;
        const float2 v = i > o + k ? X[idx] : make_float2(0.0f, 0.0f);
        float rh, rl, ih, il;
        split(-v.x, rh, rl);
        split(-v.y, ih, il);
        const size_t o0 = (size_t)(2 * i) * kp + 2 * (o + k), o1 = o0 + kp;
        *(float2*)(hi + o0) = make_float2(rh, -ih);
        *(float2*)(hi + o1) = make_float2(ih, rh);
        *(float2*)(lo + o0) = make_float2(rl, -il);
        *(float2*)(lo + o1) = make_float2(il, rl);
        if (N) N[(size_t)(o + k) * TI_W + i] = v;
    }
}
size_t tf32_pack_bytes(int n) {
    size_t kp = 512;  // two 128-column panels per trailing update
    return ((size_t)2 * n * kp + (size_t)n * kp) * 2 * 4 + (size_t)128 * 128 * 8 + 8192;
}

// CTA pairs the device holds at once
static int num_pairs() {
    static const int pairs = [] {
        int dev = 0, sms = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2 * (sms / 2));
        cfg.blockDim = dim3(192);
        cfg.dynamicSmemBytes = TF32_SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, tf32_update_kernel<PIECES_BF16>, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = sms / 2;
        }
        return std::min(n, sms / 2);
    }();
    return pairs;
}

// The packed operands live in the buffer the factor allocated from its context's pool
// (tf32_pack_bytes(n), enough for every step of an n x n factorization); a step that would
// need more records status 6 (out of memory) instead of reallocating outside the pool.
static bool ensure_pack(LuWork& wk, size_t need, cudaStream_t st) {
    if (wk.pack && wk.pack_bytes >= need) return true;
    cudaMemsetAsync(wk.status, 6, 1, st);
    return false;
}

// C[row0 .. row0+m2) x [col0 .. col0+ncols) -= Apack (m2 x kp) * Bpack (ncols x kp)^T;
// FP16 pieces have the row scales sA of the A operand, sB of the B operand.
static void run_gemm(float2* A, int n, int row0, int col0, int m2, int ncols, int kp, void* ahi, void* alo, void* bhi,
                     void* blo, const float* sA, const float* sB, LuWork& wk, cudaStream_t st, long long* launches,
                     PieceFormat pieces) {
    const bool half = pieces == PIECES_F16 || pieces == PIECES_BF16;
    CUtensorMap mAhi, mAlo, mBhi, mBlo;
    bool ok = make_map(&mAhi, ahi, m2, kp, TB_M, pieces) && make_map(&mAlo, alo, m2, kp, TB_M, pieces) &&
              make_map(&mBhi, bhi, ncols, kp, TB_N / 2, pieces) && make_map(&mBlo, blo, ncols, kp, TB_N / 2, pieces);
    // A viewed as a 2n x n float matrix (column-major): box of 128 real rows x 64 columns
    CUtensorMap mC;
    {
        EncodeTiled enc = encoder();
        cuuint64_t dims[2] = {(cuuint64_t)2 * n, (cuuint64_t)n};
        cuuint64_t strides[1] = {(cuuint64_t)2 * n * 4};
        cuuint32_t box[2] = {(cuuint32_t)TB_M, (cuuint32_t)EPI_COLS};
        cuuint32_t estr[2] = {1, 1};
        ok = ok && enc && enc(&mC, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)A, dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    }
    if (!ok) {
        cudaMemsetAsync(wk.status, 7, 1, st);
        return;
    }
    Tf32Args a;
    a.C = (float*)A;
    a.ldc = (size_t)2 * n;
    a.row0 = row0;
    a.col0 = col0;
    a.m2 = m2;
    a.ncols = ncols;
    a.kchunks = kp / (half ? 32 : TB_K);
    a.tiles_m = (m2 + 2 * TB_M - 1) / (2 * TB_M);
    a.tiles_n = (ncols + TB_N - 1) / TB_N;
    a.tiles = a.tiles_m * a.tiles_n;
    a.status = wk.status;
    a.sA = sA;
    a.sB = sB;
    const int grid = 2 * std::min(num_pairs(), a.tiles);
    auto launch = [&](auto kernel) { kernel<<<grid, 192, TF32_SMEM, st>>>(mAhi, mAlo, mBhi, mBlo, mC, a); };
    switch (pieces) {
        case PIECES_BF16: launch(tf32_update_kernel<PIECES_BF16>); break;
        case PIECES_F16: launch(tf32_update_kernel<PIECES_F16>); break;
        case PIECES_TF32X2: launch(tf32_update_kernel<PIECES_TF32X2>); break;
        default: launch(tf32_update_kernel<PIECES_TF32X3>); break;
    }
    *launches += 1;
}

// U12 = L11^-1 A12 on the tensor cores: invert L11, then A12 -= (-(L11^-1 - I)) A12 with the
// operands packed (A12 is read from its packed copy, so the in-place update is race free).
// Places of one TRSM step in the factor's operand buffer (a trailing block means a full panel, w = 128):
// the pieces of A12 first, then those of -N and N itself, beyond what the updates between the inverse's
// launch and the TRSM write (panel b's block rows, the packing of A12). False when the buffer is too small.
struct TrsmPlaces {
    float *bhi, *blo, *nhi, *nlo;
    float2* N;
};
static bool trsm_places(int n, int k0, LuWork& wk, cudaStream_t st, TrsmPlaces* t) {
    const size_t ncols = n - k0 - TI_W, kp = 2 * TI_W, piece = 2 * TI_W * kp;
    // panel b's update with panel a: pieces of its 128 complex rows and of ncols columns (the largest of them)
    const size_t before = 2 * (piece + ncols * kp);
    if (!ensure_pack(wk, (before + 2 * piece) * 4 + (size_t)TI_W * TI_W * 8 + 8192, st)) return false;
    t->bhi = (float*)wk.pack;
    t->blo = t->bhi + ncols * kp;
    t->nhi = (float*)(((uintptr_t)((float*)wk.pack + before) + 255) & ~(uintptr_t)255);
    t->nlo = t->nhi + piece;
    t->N = (float2*)(t->nlo + piece);
    return true;
}

bool launch_tf32_trsm_inverse(float2* A, int n, int k0, LuWork& wk, cudaStream_t st, cudaStream_t side,
                              long long* launches) {
    TrsmPlaces t;
    if (!trsm_places(n, k0, wk, st, &t)) return false;
    tri_inverse_l_kernel<<<TI_W / TI_C, 256, TI_SMEM, side>>>(A, (size_t)n, k0, t.nhi, t.nlo,
                                                        wk.pieces == PIECES_F16 ? t.N : nullptr);
    ++*launches;
    // a refused launch leaves the inverse to the main stream (launch_tf32_trsm, inverse_done false)
    return cudaGetLastError() == cudaSuccess;
}

// The TRSM's right-hand side A12 as TF32 pieces, packed before the main stream waits for the
// inverse of L11 (which it does not need); launch_tf32_trsm(..., rhs_packed = true) then skips
// it. FP16 pieces keep their packing in launch_tf32_trsm (false here).
static void pack_trsm_rhs(float2* A, int n, int k0, const TrsmPlaces& t, cudaStream_t st, long long* launches) {
    const int r0 = k0 + TI_W, ncols = n - r0;
    const size_t tot = (size_t)ncols * TI_W;
    pack_u_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(A, (size_t)n, r0, k0, ncols, TI_W, 2 * TI_W, t.bhi,
                                                                 t.blo);
    ++*launches;
}
bool launch_tf32_trsm_rhs(float2* A, int n, int k0, LuWork& wk, cudaStream_t st, long long* launches) {
    TrsmPlaces t;
    if (wk.pieces == PIECES_F16 || !trsm_places(n, k0, wk, st, &t)) return false;
    StageScope sc(ST_TRSM, st);
    pack_trsm_rhs(A, n, k0, t, st, launches);
    return true;
}

void launch_tf32_trsm(float2* A, int n, int k0, LuWork& wk, cudaStream_t st, long long* launches, bool inverse_done,
                      bool rhs_packed) {
    constexpr int w = TI_W, kp = 2 * TI_W;
    const int r0 = k0 + w, ncols = n - r0;
    TrsmPlaces t;
    if (!trsm_places(n, k0, wk, st, &t)) return;
    StageScope sc(ST_TRSM, st);
    if (!inverse_done && !launch_tf32_trsm_inverse(A, n, k0, wk, st, st, launches)) {
        cudaMemsetAsync(wk.status, 7, 1, st);  // U12 would use a stale inverse: stop the factorization
        return;
    }
    if (wk.pieces == PIECES_F16) {
        // A operand: -N embedded, so that the update C -= (-N) A12 adds N A12
        __half *h_ahi = (__half*)wk.pack, *h_alo = h_ahi + (size_t)2 * w * kp;
        __half *h_bhi = h_alo + (size_t)2 * w * kp, *h_blo = h_bhi + (size_t)ncols * kp;
        float* sA = (float*)(((uintptr_t)(h_blo + (size_t)ncols * kp) + 255) & ~(uintptr_t)255);
        float* sB = (float*)(((uintptr_t)(sA + w) + 255) & ~(uintptr_t)255);
        pack_l16_kernel<<<(w + 31) / 32, 256, 0, st>>>(t.N, (size_t)w, 0, 0, w, w, kp, -1.0f, h_ahi, h_alo, sA);
        pack_u16_kernel<<<(unsigned)(((size_t)ncols * 32 + 255) / 256), 256, 0, st>>>(A, (size_t)n, r0, k0, ncols, w, kp,
                                                                                     h_bhi, h_blo, sB);
        run_gemm(A, n, 2 * k0, r0, 2 * w, ncols, kp, h_ahi, h_alo, h_bhi, h_blo, sA, sB, wk, st, launches, PIECES_F16);
        *launches += 2;
    } else {
        if (!rhs_packed) pack_trsm_rhs(A, n, k0, t, st, launches);
        run_gemm(A, n, 2 * k0, r0, 2 * w, ncols, kp, t.nhi, t.nlo, t.bhi, t.blo, nullptr, nullptr, wk, st, launches,
                 PIECES_TF32X3);
    }
}

// A[r0 .. r0+m) x [c0 .. c0+ncols) -= A[r0.., k0 .. k0+w) A[k0 .. k0+w, c0..): the trailing
// update of panel columns k0 .. k0+w restricted to a block of rows and columns.
void launch_tf32_update_region(float2* A, int n, int k0, int w, int r0, int m, int c0, int ncols, LuWork& wk,
                               cudaStream_t st, long long* launches) {
    if (m <= 0 || ncols <= 0) return;
    int kp = ((2 * w + 31) / 32) * 32;  // whole 64-byte K rows of FP16 pieces (and of TF32)
    size_t need = ((size_t)2 * m * kp + (size_t)ncols * kp) * 2 * 4 + 4096;
    if (!ensure_pack(wk, need, st)) return;
    float* ahi = (float*)wk.pack;
    float* alo = ahi + (size_t)2 * m * kp;
    float* bhi = alo + (size_t)2 * m * kp;
    float* blo = bhi + (size_t)ncols * kp;
    __half *h_ahi = (__half*)ahi, *h_alo = h_ahi + (size_t)2 * m * kp;
    __half *h_bhi = h_alo + (size_t)2 * m * kp, *h_blo = h_bhi + (size_t)ncols * kp;
    float* sA = (float*)(((uintptr_t)(h_blo + (size_t)ncols * kp) + 255) & ~(uintptr_t)255);
    float* sB = (float*)(((uintptr_t)(sA + m) + 255) & ~(uintptr_t)255);
    {
        StageScope sc(ST_PACK, st);
        if (wk.pieces == PIECES_BF16) {
            const dim3 g1((m + 31) / 32, (kp / 2 + 31) / 32);
            const size_t tot = (size_t)ncols * (kp / 2);
            pack_l_bf16_kernel<<<g1, 256, 0, st>>>(A, (size_t)n, r0, k0, m, w, kp, (__nv_bfloat16*)h_ahi,
                                                   (__nv_bfloat16*)h_alo);
            pack_u_bf16_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(
                A, (size_t)n, c0, k0, ncols, w, kp, (__nv_bfloat16*)h_bhi, (__nv_bfloat16*)h_blo);
        } else if (wk.pieces == PIECES_F16) {
            pack_l16_kernel<<<(m + 31) / 32, 256, 0, st>>>(A, (size_t)n, r0, k0, m, w, kp, 1.0f, h_ahi, h_alo, sA);
            pack_u16_kernel<<<(unsigned)(((size_t)ncols * 32 + 255) / 256), 256, 0, st>>>(A, (size_t)n, c0, k0, ncols, w,
                                                                                         kp, h_bhi, h_blo, sB);
        } else {
            dim3 g1((m + 31) / 32, (kp / 2 + 31) / 32);
            size_t tot = (size_t)ncols * (kp / 2);
            pack_l_kernel<<<g1, 256, 0, st>>>(A, (size_t)n, r0, k0, m, w, kp, ahi, alo);
            pack_u_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(A, (size_t)n, c0, k0, ncols, w, kp, bhi,
                                                                         wk.pieces == PIECES_TF32X2 ? nullptr : blo);
        }
        *launches += 2;
    }
    StageScope sc(ST_GEMM, st);
    if (wk.pieces == PIECES_BF16 || wk.pieces == PIECES_F16)
        run_gemm(A, n, 2 * r0, c0, 2 * m, ncols, kp, h_ahi, h_alo, h_bhi, h_blo, sA, sB, wk, st, launches, wk.pieces);
    else
        run_gemm(A, n, 2 * r0, c0, 2 * m, ncols, kp, ahi, alo, bhi, blo, nullptr, nullptr, wk, st, launches, wk.pieces);
}

void launch_tf32_update(float2* A, int n, int k0, int w, LuWork& wk, cudaStream_t st, long long* launches) {
    const int r0 = k0 + w;
    launch_tf32_update_region(A, n, k0, w, r0, n - r0, r0, n - r0, wk, st, launches);
}

}  // namespace tcu
