// Host-side launchers of the device kernels (one header for the C ABI layer).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include "../../include/treams_cuda.h"
#include "plan.h"

#include <atomic>
#include <mutex>
#include <vector>

namespace tcu {

typedef double2 cplx;

// Kernel attributes (large dynamic shared memory) are per device: each site keeps one bit per
// device in `mask`, and this returns true the first time it runs with that device current.
struct PerDeviceOnce {
    std::mutex mu;
    unsigned long long done = 0;  // bit d: done on device d
};
// Runs f once per process and current device; callers on other threads wait until it is done
// (the batched solve launches from several host threads).
template <class F>
inline void once_per_device(PerDeviceOnce& o, F&& f) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        f();
        return;
    }
    const unsigned long long bit = 1ull << dev;
    std::lock_guard<std::mutex> g(o.mu);
    if (o.done & bit) return;
    f();
    o.done |= bit;
}

// Per-stage CUDA-event timing (tcu_context_set_profiling). The API layer installs the
// context's profiler as the calling thread's current one for the duration of a call; the
// launch sites bracket their kernels with a StageScope.
enum Stage { ST_ASSEMBLE = 0, ST_PANEL, ST_SWAP, ST_TRSM, ST_GEMM, ST_PACK, ST_SOLVE, ST_APPLY, ST_MIE, ST_LATTICE,
             ST_SMALL_LU, ST_COARSE, ST_NEAR, ST_COUNT };
struct Profiler {
    bool on = false;
    struct Rec {
        int stage;
        cudaEvent_t a, b;
    };
    std::vector<Rec> recs;
    std::vector<cudaEvent_t> pool;
    double total_ms[ST_COUNT] = {};
    long long count[ST_COUNT] = {};
    cudaEvent_t take() {
        if (!pool.empty()) {
            cudaEvent_t e = pool.back();
            pool.pop_back();
            return e;
        }
        cudaEvent_t e;
        cudaEventCreate(&e);
        return e;
    }
    void collect() {
        for (auto& r : recs) {
            cudaEventSynchronize(r.b);
            float ms = 0.f;
            cudaEventElapsedTime(&ms, r.a, r.b);
            total_ms[r.stage] += ms;
            count[r.stage] += 1;
            pool.push_back(r.a);
            pool.push_back(r.b);
        }
        recs.clear();
    }
    ~Profiler() {
        collect();
        for (auto e : pool) cudaEventDestroy(e);
    }
};
extern thread_local Profiler* g_prof;

// Device memory of objects that live within one API call (preconditioners, their graphs and
// coarse solvers): the context's caching pool while the call has installed it (PoolScope),
// else cudaMalloc / cudaFree. Each allocation remembers where it came from.
struct DeviceAllocator {
    virtual cudaError_t alloc(void** p, size_t bytes) = 0;
    virtual void release(void* p) = 0;

   protected:
    ~DeviceAllocator() = default;
};
extern thread_local DeviceAllocator* g_call_pool;
struct PoolScope {
    DeviceAllocator* prev;
    explicit PoolScope(DeviceAllocator* a) : prev(g_call_pool) { g_call_pool = a; }
    ~PoolScope() { g_call_pool = prev; }
};
inline cudaError_t call_malloc(void** p, size_t bytes, DeviceAllocator** owner) {
    *owner = g_call_pool;
    return *owner ? (*owner)->alloc(p, bytes) : cudaMalloc(p, bytes);
}
inline void call_free(void* p, DeviceAllocator* owner) {
    if (!p) return;
    if (owner)
        owner->release(p);
    else
        cudaFree(p);
}
struct StageScope {
    Profiler* p;
    int stage;
    cudaStream_t st;
    cudaEvent_t a = nullptr;
    StageScope(int stage_, cudaStream_t st_) : p(g_prof), stage(stage_), st(st_) {
        if (p && p->on) {
            a = p->take();
            cudaEventRecord(a, st);
        }
    }
    ~StageScope() {
        if (a) {
            cudaEvent_t b = p->take();
            cudaEventRecord(b, st);
            p->recs.push_back({stage, a, b});
        }
    }
};

// pairs.cu
void launch_assemble(const DevPlan& P, int N, double k, const double* pos, const cplx* T, void* out, size_t ld,
                     bool fp32, cudaStream_t st);
void launch_apply(const DevPlan& P, int N, double k, const double* pos, const cplx* T, const cplx* x, size_t ldx,
                  int ncol, const cplx* zadd, double alpha, double beta, bool singular, cplx* y, cudaStream_t st);
size_t apply_smem_bytes(const DevPlan& P, int ncol);
// Product form of the same operator (lmax 2..5; TCU_APPLY=terms selects the term-sum kernels)
bool apply_gemm_supported(const DevPlan& P);
void launch_apply_gemm(const DevPlan& P, int N, double k, const double* pos, const cplx* T, const cplx* x, size_t ldx,
                       int ncol, const cplx* zadd, double alpha, double beta, bool singular, cplx* y, cudaStream_t st);
void apply_gemm_init_attributes();
// Dipole blocks of the operator in product form, one vector: z holds the 6 dipole modes of every
// sphere; y = zadd + alpha (z on the dipole modes) + beta T (C P z), on all modes (y: n) or, with
// dipole_rows, on the dipole modes only (y: 6N). P z is z on the dipole modes, zero elsewhere.
void launch_apply_dipole(const DevPlan& P, int N, double k, const double* pos, const cplx* T, const cplx* z,
                         bool dipole_rows, const cplx* zadd, double alpha, double beta, cplx* y, cudaStream_t st);
// Stored-table form of the singular operator and of its two dipole blocks (for repeated
// applications; singular false: the regular operator x + C x): the harmonic tables of all ordered pairs built once into Z
// (stored_tables_bytes), then every application is an FP64 tensor-core product over Z plus the
// term lists. kind: STORED_FULL (lmax 2..7) is launch_apply's operator; STORED_DIPOLE_SOURCES and
// STORED_DIPOLE_BLOCK are launch_apply_dipole with dipole_rows false and true (input ldin 6).
// Xf: scratch of stored_inputs_bytes for the packed inputs. Sizes are 0 where a kind does not
// apply.
enum StoredKind { STORED_FULL = 0, STORED_DIPOLE_SOURCES = 1, STORED_DIPOLE_BLOCK = 2 };
bool stored_full_supported(const DevPlan& P);  // STORED_FULL exists for this lmax and TCU_APPLY allows it
bool stored_tables_enabled();  // false when TCU_APPLY is "fly" or "terms" (read at every call)
// the list of blocks that the full operator's product forms; false when its warps cannot hold them
bool stored_product_blocks(const DevPlan& P, const HostPlan& h, ProductBlocks* b);
size_t stored_tables_bytes(const DevPlan& P, int N, int kind);
size_t stored_inputs_bytes(const DevPlan& P, int N, int kind, int ncol);
void build_stored_tables(const DevPlan& P, int N, double k, const double* pos, int kind, cplx* Z, cudaStream_t st,
                         bool singular = true);
// status (may be null) receives 8 when a bounded wait of the product gave up (y not written).
void launch_apply_stored(const DevPlan& P, int N, int kind, const cplx* Z, const cplx* T, const cplx* x, size_t ldx,
                         int ncol, const cplx* zadd, double alpha, double beta, cplx* y, cplx* Xf, int* status,
                         cudaStream_t st, bool singular = true);
void launch_block(const DevPlan& P, double k, const double* d, bool singular, bool helicity, cplx* out,
                  cudaStream_t st);
void launch_mie(int L, double k0, int N, const double* radii, const cplx* eps, cplx* T, int* status, cudaStream_t st);
void launch_plane_wave(int L, int N, const double* pos, int ncol, const cplx* kvecs, const int* pols,
                       const double* lfac, cplx* out, cudaStream_t st);
void launch_apply_t(int L, int N, const cplx* T, const cplx* x, int ncol, cplx* y, cudaStream_t st);
// regular translation blocks between the N spheres (nlm_loc lm per sphere) and the origin
// (nlm_glob lm), cut from blocks of the plan P (P.nlm >= both): Ein n x Mg, Eout Mg x n
// (cleared by the caller); and a small complex FP64 GEMM C = A B (column-major)
void launch_expand_blocks(const DevPlan& P, int N, double k, const double* pos, const double* origin, int nlm_loc,
                          int nlm_glob, cplx* Ein, cplx* Eout, cudaStream_t st);
void launch_zgemm_small(int m, int n, int k, const cplx* A, size_t lda, const cplx* B, size_t ldb, cplx* C,
                        size_t ldc, cudaStream_t st);
void pairs_init_attributes();
// translate.cu — per-entry translation coefficients: labels 6 ints per element (lambda, mu,
// pol, l, m, qol), args 3 complex per element (kr, theta, phi)
void launch_translate(const DevPlan& P, size_t count, const int* labels, const cplx* args, bool helicity,
                      bool singular, cplx* out, cudaStream_t st);

// adjoint.cu — y = (I - T C)^H x for ncol columns of leading dimension ldx (t1, t2: ldx x ncol
// scratch; with stored pair tables Z (STORED_FULL) the coupling product runs over them, Xf:
// stored_inputs_bytes for ncol columns, status as for launch_apply_stored), y = T^H x, and
// x <- A^-H x with the LU factors (tmp: adjoint_solve_tmp(n, ncol))
void launch_apply_adjoint(const DevPlan& P, int N, double k0, const double* pos, const cplx* T, const cplx* x,
                          size_t ldx, int ncol, cplx* y, cplx* t1, cplx* t2, cudaStream_t st, long long* launches,
                          const cplx* Z = nullptr, cplx* Xf = nullptr, int* status = nullptr);
void launch_apply_th(int L, int N, const cplx* T, const cplx* x, size_t ldx, int ncol, cplx* y, cudaStream_t st);
size_t adjoint_solve_tmp(int n, int ncol);
void lu_solve_adjoint_fp64(const double2* A, int n, const int* perm, const double2* inv, double2* x, double2* tmp,
                           int ncol, cudaStream_t st, long long* launches, int* status);
void lu_solve_adjoint_fp32(const float2* A, int n, const int* perm, const double2* inv, double2* x, double2* tmp,
                           int ncol, cudaStream_t st, long long* launches, int* status);

// equil.cu — power-of-two row/column equilibration of an n x n column-major matrix (FP64 or
// FP32 storage) when its largest entry exceeds `threshold`; r, c: n scales each.
size_t equilibrate_scratch_doubles(int n);
tcu_status equilibrate(void* A, bool fp32, int n, double threshold, double* r, double* c, double* partial,
                       bool* applied, cudaStream_t st, long long* launches);
void scale_rows(cplx* v, const double* s, size_t n, int ncol, cudaStream_t st);

// lattice.cu — 2D lattice sums (any real shift) and the batched periodic-array solve
constexpr int LS_MAXL = 14;                // largest degree of a lattice sum
constexpr int LS_NMAX = LS_MAXL / 2 + 1;   // reciprocal orders n per (l, m) in the plane
constexpr int LS_FMAX = LS_MAXL + 1;       // reciprocal orders n per (l, m) off the plane
constexpr int LS_PMAX = LS_MAXL / 2 + 1;   // powers of beta^2 in S_lmn off the plane
constexpr int LS_TMAX = 64;                // most terms of the t-series of F_(1/2-n)(v, t)
struct LatticeSumArgs {
    int lsum = 0;                          // degrees l <= lsum, T = (lsum+1)^2 outputs
    double k = 0, eta = 0;
    int NR = 0;                            // real-space lattice points (R != 0)
    const double2* R = nullptr;
    const double2* realtab = nullptr;      // NR x pairs x 2 real-space terms (lattice_pair_index)
    int NG = 0;                            // reciprocal lattice vectors
    const double2* G = nullptr;
    const double2* Glo = nullptr;          // their low parts (G = G + Glo to twice FP64 precision)
    const double2* coef = nullptr;         // slots x pairs: polynomial coefficients (lattice_coefficients)
    const double2* pref = nullptr;         // T reciprocal prefactors
    double2 self0{0, 0};                   // self term of l = 0 (zero for a nonzero shift)
    double sx = 0, sy = 0;                 // in-plane shift r' (reciprocal phase e^{-i q.r'})
    double R0x = 0, R0y = 0;               // lattice vector taken off the shift: e^{-i kpar.R0}
    // shift off the plane (r_z != 0): every order n <= lsum, F'_n from the t-series of
    // F_(1/2-n)(v, t) with t = (k r_z eta)^2 (J + 1 terms)
    bool offplane = false;
    int J = 0;
    double t = 0;
    int nk = 0;
    const double2* kpar = nullptr;
    double2* out = nullptr;                // out[kp * ldo + l*l+l+m]
    size_t ldo = 0;
    int* status = nullptr;                 // 9: a diffraction order on its threshold
};
// lattice_ck.cu — the same sums at a complex wavenumber (Im k >= 0), any shift, real split
struct LatticeSumCkArgs {
    int lsum = 0;
    double2 k{0, 0};
    double eta = 0;
    int NR = 0;
    const double2* R = nullptr;
    const double2* realtab = nullptr;      // NR x pairs x 2 real-space terms (lattice_pair_index)
    int NG = 0;
    const double2* G = nullptr;
    const double2* Glo = nullptr;          // low parts of the reciprocal vectors
    const double2* coef = nullptr;         // slots x pairs: polynomial coefficients (lattice_coefficients)
    bool offplane = false;                 // shift off the plane: every order n <= lsum
    const double2* pref = nullptr;         // T reciprocal prefactors (1/k^2 included)
    double2 self0{0, 0};
    double sx = 0, sy = 0, R0x = 0, R0y = 0;
    int J = 0;                             // t-series terms (0 in the plane)
    double2 t{0, 0};                       // (k r_z eta)^2
    double2 ksq{0, 0};                     // k^2
    double turn = 0, near = 0;             // sheet split: arg (k eta)^2, tan^2 of the near sector
    int has_near = 0;
    int nk = 0;
    const double2* kpar = nullptr;
    double2* out = nullptr;
    size_t ldo = 0;
    int* status = nullptr;                 // 9: a diffraction order on its threshold
};
void launch_real_table_ck(int lsum, double2 k, double eta, int NR, const double2* R, double sx, double sy, double sz,
                          const double* norm, const double* reflection, bool offplane, double2* tab, cudaStream_t st);
void launch_real_table(int lsum, double k, double eta, int NR, const double2* R, double sx, double sy, double sz,
                       const double* norm, const double* reflection, bool offplane, double2* tab, cudaStream_t st);
// lattice_sum.cu — the reciprocal part and the reduction. The sums run over the (l, |m|) pairs of
// even l - |m| in the plane, of all off it, in the order of l - |m|, then |m|.
int lattice_pairs(int lsum, bool offplane);
int lattice_orders(int lsum, bool offplane);  // F'_n kept per reciprocal vector
size_t lattice_order_bytes(int lsum, bool offplane, int NG, size_t nk);  // scratch F of the launches
// entry of (l, m) in a table row of 2 lattice_pairs entries (-1: vanishes); hstep 2 in the plane, else 1
#ifdef __CUDACC__
__host__ __device__
#endif
inline int lattice_pair_index(int lsum, int l, int m, int hstep) {
    const int am = m < 0 ? -m : m, h = l - am;
    if (h % hstep) return -1;
    const int before = hstep == 2 ? h / 2 * (lsum + 1) - h / 2 * (h / 2 - 1) : h * (lsum + 1) - h * (h - 1) / 2;
    return 2 * (before + am) + (m < 0 ? 1 : 0);
}
void launch_lattice_sum(const LatticeSumArgs& a, cplx* F, cudaStream_t st, long long* launches);
void launch_lattice_sum_ck(const LatticeSumCkArgs& a, cplx* F, cudaStream_t st, long long* launches);
void launch_array_solve(const DevPlan& P, const double2* D, size_t ldd, const double* norm, const double2* Tm, int nk,
                        double2* X, int* status, int grid, cudaStream_t st);

// lu.cu — dense LU of an n x n column-major complex matrix (lda = n) in FP64 (double2)
// or FP32 (float2) storage, row permutation kept as perm (row i of P A is row perm[i]).
// Operand pieces of the mixed path's trailing updates (gemm_tf32.cu): three passes of bfloat16, of FP16
// (scaled rows) or of TF32 pieces, or two of TF32
enum PieceFormat { PIECES_TF32X3, PIECES_TF32X2, PIECES_F16, PIECES_BF16 };
struct LuWork {
    int* piv = nullptr;        // n
    int* perm = nullptr;       // n
    unsigned* barrier = nullptr;
    int* status = nullptr;     // device status word
    void* cand = nullptr;      // candidate values/rows, double-buffered
    void* pack = nullptr;      // packed GEMM operands (mixed path)
    size_t pack_bytes = 0;
    PieceFormat pieces = PIECES_TF32X3;  // mixed path: the split of the trailing updates' operands
    int panel_rows = 0;        // least rows per panel CTA (0: the default of the panel's kernel)
};
// bfloat16 unless TCU_SPLIT names another format (tf32x3, tf32x2, f16)
PieceFormat split_default();
int lu_factor_fp64(double2* A, int n, LuWork& w, cudaStream_t st, long long* launches);
// Self-tests of the bounded waits: each waits for what never comes, gives up after limit_s (clamped to
// [0, 4] s) and records status 8. zeros: 16 zeroed bytes of device memory.
inline unsigned long long selftest_ns(double limit_s) {
    return (unsigned long long)((limit_s < 0.0 ? 0.0 : limit_s > 4.0 ? 4.0 : limit_s) * 1e9);
}
void launch_panel_wait_selftest(const void* zeros, int* status, double limit_s, cudaStream_t st);  // status: 2 words
void launch_sweep_wait_selftest(int* entry_status, int* ring_status, void* entry, double limit_s, cudaStream_t st);
void launch_update_wait_selftest(int* status, double limit_s, cudaStream_t st);
void launch_product_wait_selftest(int* status, double limit_s, cudaStream_t st);
// The panel's grid barrier with one arrival missing (bar: a zeroed counter); it gives up
// after limit_s (clamped to [0, 4] s) and records status 8.
void launch_barrier_selftest(unsigned* bar, int* status, double limit_s, cudaStream_t st);
// The row interchanges of a panel that gave up: status 9 if a pivot out of range moved anything.
// work: swap_selftest_bytes() of device memory.
size_t swap_selftest_bytes();
void launch_swap_selftest(void* work, int* status, cudaStream_t st);
int lu_factor_fp32(float2* A, int n, LuWork& w, cudaStream_t st, long long* launches, bool tensor_cores);
// solve.cu — inverses of the 64 x 64 diagonal blocks of L and U (FP64, lu_inverse_bytes),
// then x (n x ncol, FP64) <- A^-1 x, ncol <= SOLVE_MAXC; tmp holds 2 n ncol complex.
constexpr int SOLVE_MAXC = 128;
size_t lu_inverse_bytes(int n);
void lu_block_inverses_fp64(const double2* A, int n, double2* inv, cudaStream_t st, long long* launches);
void lu_block_inverses_fp32(const float2* A, int n, double2* inv, cudaStream_t st, long long* launches);
// status: a device status word (8 when a sweep's bounded wait gave up); null selects one launch
// per block step.
void lu_solve_fp64(const double2* A, int n, const int* perm, const double2* inv, double2* x, double2* tmp, int ncol,
                   cudaStream_t st, long long* launches, int* status = nullptr);
void lu_solve_fp32(const float2* A, int n, const int* perm, const double2* inv, double2* x, double2* tmp, int ncol,
                   cudaStream_t st, long long* launches, int* status = nullptr);
// The persistent sweeps alone (no permutation): out = (L U)^-1 rhs or its adjoint, through mid;
// false when they cannot run (TCU_SOLVE=steps, no status word, a refused launch; rhs is intact).
template <typename C>
bool lu_sweeps(const C* A, int n, const double2* inv, const double2* rhs, double2* mid, double2* out, int ncol,
               bool adjoint, int* status, cudaStream_t st, long long* launches);
size_t lu_workspace_bytes(int n, bool fp32);
size_t tf32_pack_bytes(int n);  // packed tensor-core operands of the mixed LU
void lu_init_attributes();

// blas.cu — fixed-order reductions and vector updates on FP64 complex vectors
void vec_norms(const cplx* x, size_t n, int ncol, double* out_dev, double* partial, cudaStream_t st);
void vec_axpy(cplx* y, const cplx* x, size_t n, int ncol, cudaStream_t st);
void vec_sub(cplx* out, const cplx* a, const cplx* b, size_t n, int ncol, cudaStream_t st);
constexpr int ARNOLDI_PARTS = 592;  // partial sums of a norm: four CTAs per SM
// coef: 2 nv + 1 entries, partial: 256 nv, npart: ARNOLDI_PARTS
void vec_arnoldi_step(const cplx* V, size_t ldv, int nv, cplx* w, size_t n, cplx* next, cplx* coef, cplx* partial,
                      double* npart, cudaStream_t st);
void vec_scale_copy(cplx* out, const cplx* x, size_t n, double s, cudaStream_t st);
void vec_lincomb(cplx* x, const cplx* V, size_t ldv, int nv, const cplx* g_dev, size_t n, cudaStream_t st);
void vec_real_dots(const cplx* a, const cplx* b, size_t n, int ncol, double* out_dev, double* partial,
                   cudaStream_t st);

}  // namespace tcu
