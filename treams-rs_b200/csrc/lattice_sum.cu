// The lattice sums' two device stages behind the real-space tables (lattice.cu for a real
// wavenumber, lattice_ck.cu for a complex one, which also state the formulas):
//   lattice_orders_kernel  F'_n of every (Bloch vector, reciprocal vector) pair, a thread each;
//   lattice_reduce_kernel  D_lm of every Bloch vector from them and from the real-space table.
//
// Orders. F_(1/2-i)(v, 0) for i = 0..I (I = the largest n, plus the terms of the t-series off the
// plane) comes from ONE evaluation at i0 = min(I, round |v|) and the two-term recurrence of the
// incomplete gamma function (DLMF 8.8.2) in both directions: with b_i = 1/2 - i and
// Q_i = Gamma(b_i, z) / z^b_i,
//   Q_(i+1) = (z Q_i - e^-z) / b_(i+1),   Q_i = (b_(i+1) Q_(i+1) + e^-z) / z,
// and the same with -e^-z for the power series S_i (DLMF 8.7.3), Q_i = Gamma(b_i) z^-b_i - S_i. Above
// i0 the first contracts errors by |z| / (i + 1/2), below it the second adds terms of one sign for
// Re z > 0: against 113-bit values both stay at the error of the direct evaluation (1.5e-14 over
// |z| in 2..45, every i <= 24; starting at |z| / 2 instead loses one to three digits). Evaluating
// every order by itself took 7 (in the plane) to 40 (off it) fractions or series per pair, with only
// the threads of one Bloch vector's reciprocal vectors at work: it bound the whole call.
// The fraction runs backward from a level that its convergence rate exp(-4 sqrt(N |z|) cos(arg z / 2))
// fixes beforehand: one reciprocal a level instead of the two divisions of Lentz's algorithm.
// Threads of a warp share the reciprocal vector and differ in the Bloch vector, so they mostly agree
// on the branch and on the number of levels.
//
// Reduction. A thread takes one (l, |m|) of one Bloch vector with both signs of m: the polynomial
// S_lmn is the same for +-m. Orders, powers ((q_x +- i q_y)/k)^m and Bloch phases of a tile of lattice
// points sit in shared memory. Pairs are sorted by l - |m|, so a warp runs one polynomial length; in the lattice plane
// only even l - |m| exist (the others vanish). Every sum has a fixed order.
//
// Measured (B200): 4096 Bloch vectors, l <= 12 in the plane: 2.63 ms -> 0.28 ms for all stages;
// 1000 at k0 (1 + 0.05 i) off the plane, l <= 8: 2.79 -> 0.27 ms.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace tcu {

namespace {

constexpr int LO_T = 128;      // threads of the order kernel
constexpr int LO_TAB = 128;    // reciprocals kept in shared memory
constexpr double LS_PI = 3.14159265358979323846;

// Real and complex arithmetic of the recurrences (F: double or cplx)
__device__ __forceinline__ double f_mul(double a, double b) { return a * b; }
__device__ __forceinline__ cplx f_mul(cplx a, cplx b) { return cmul(a, b); }
__device__ __forceinline__ double f_scale(double a, double s) { return a * s; }
__device__ __forceinline__ cplx f_scale(cplx a, double s) { return cscale(a, s); }
__device__ __forceinline__ double f_add(double a, double b) { return a + b; }
__device__ __forceinline__ cplx f_add(cplx a, cplx b) { return cadd(a, b); }
__device__ __forceinline__ double f_add1(double a, double s) { return a + s; }
__device__ __forceinline__ cplx f_add1(cplx a, double s) { return mk(a.x + s, a.y); }
__device__ __forceinline__ double f_neg(double a) { return -a; }
__device__ __forceinline__ cplx f_neg(cplx a) { return cneg(a); }
__device__ __forceinline__ double f_inv(double a) { return __drcp_rn(a); }
__device__ __forceinline__ cplx f_inv(cplx a) {
    const double r = __drcp_rn(cabs2(a));
    return mk(a.x * r, -a.y * r);
}
__device__ __forceinline__ double f_exp(double a) { return exp(a); }
__device__ __forceinline__ cplx f_exp(cplx a) { return cexpz(a); }
__device__ __forceinline__ double f_re(double a) { return a; }
__device__ __forceinline__ double f_re(cplx a) { return a.x; }
__device__ __forceinline__ double f_size(double a) { return fabs(a); }
__device__ __forceinline__ double f_size(cplx a) { return fabs(a.x) + fabs(a.y); }

struct Recip {
    const double* one;   // 1 / k
    const double* half;  // 1 / (k + 1/2)
    __device__ double at(int k) const { return k < LO_TAB ? one[k] : 1.0 / k; }
    __device__ double at_half(int k) const {  // 1 / (k + 1/2), any sign of k
        const int m = k < 0 ? -1 - k : k;
        const double r = m < LO_TAB ? half[m] : 1.0 / (m + 0.5);
        return k < 0 ? -r : r;
    }
};

// Legendre's continued fraction of Gamma(b, z) e^z z^-b (DLMF 8.9.2, even contraction) from level
// n down
template <typename F>
__device__ F fraction_down(double b, F z, double az) {
    const double cos2 = 0.5 * (1.0 + f_re(z) / az);
    const int n = min(2000, (int)(85.0 / (az * cos2)) + 6);
    F t = f_scale(z, 0.0);
    for (int i = n; i > 0; --i) t = f_scale(f_inv(f_add(f_add1(z, (2 * i + 1) - b), t)), -(double)i * ((double)i - b));
    return f_inv(f_add(f_add1(z, 1.0 - b), t));
}

// sum_k (-z)^k / (k! (b + k)), b = 1/2 - i (DLMF 8.7.3 without its leading power)
template <typename F>
__device__ F series_sum(int i, F z, double az, const Recip& rc) {
    F term = f_add1(f_scale(z, 0.0), 1.0), s = f_scale(term, rc.at_half(-i));
    const F mz = f_neg(z);
    for (int k = 1; k < 600; ++k) {
        term = f_scale(f_mul(term, mz), rc.at(k));
        const F add = f_scale(term, rc.at_half(k - i));
        s = f_add(s, add);
        if (k > az && f_size(add) < 1e-18 * f_size(s)) break;
    }
    return s;
}

// where the fraction converges fast (the series elsewhere; real z: from 2 on)
__device__ __forceinline__ bool by_fraction(cplx z, double az) { return z.x >= 2.0 || (az >= 4.0 && z.x >= -0.3 * az); }

// Calls emit(i, Q_i or S_i) for i = 0..I: from i0 up, then from i0 - 1 down.
template <typename F, typename Emit>
__device__ void order_ladder(int I, F z, double az, bool frac, const Recip& rc, Emit emit) {
    const int i0 = min(I, (int)(az + 0.5));
    const F ez = f_exp(f_neg(z));
    const F e = frac ? f_neg(ez) : ez;  // Q_(i+1) = (z Q_i - e^-z) / b_(i+1), S_(i+1) = (z S_i + e^-z) / b_(i+1)
    const F start = frac ? f_mul(ez, fraction_down(0.5 - i0, z, az)) : series_sum(i0, z, az, rc);
    F q = start;
    emit(i0, q);
    for (int i = i0; i < I; ++i) {
        q = f_scale(f_add(f_mul(z, q), e), -rc.at_half(i));
        emit(i + 1, q);
    }
    if (i0 > 0) {
        const F zi = f_inv(z);
        q = start;
        for (int i = i0 - 1; i >= 0; --i) {
            q = f_mul(f_add(f_scale(q, -(i + 0.5)), f_neg(e)), zi);
            emit(i, q);
        }
    }
}

// Whole turns of v on the outgoing sheet of an order (lattice/sheets.rs): orders whose k^2 - q.q
// lies in the near sector of the split (|arg| of (k eta)^2 + 1/2 < pi/2) follow arg(k^2 - q.q);
// the others stay on the principal sheet. Returns whether the number of turns is odd.
__device__ bool odd_turns_of(const LatticeSumCkArgs& A, double q2, cplx v) {
    const cplx sq = mk(A.ksq.x - q2, A.ksq.y);
    const bool near = sq.x > 0.0 && sq.y * sq.y <= A.near * sq.x * sq.x;
    if (A.has_near && !near) return false;
    double turn;
    if (sq.y == 0.0) {
        turn = sq.x > 0.0 ? 0.0 : LS_PI;
    } else {
        turn = atan2(sq.y, sq.x);
        if (turn < 0.0) turn += 2.0 * LS_PI;
    }
    const double sheet = turn - LS_PI - A.turn;
    const double turns = rint((sheet - atan2(v.y, v.x)) / (2.0 * LS_PI));
    return fmod(fabs(turns), 2.0) == 1.0;
}

// Orders and their sinks. The limits L_i = F_(1/2-i)(v, 0) go either straight to F'_i (in the plane)
// or into the t-series sums of every F'_n they reach (off it), kept per thread in shared memory.
struct OrderSink {
    cplx* out;         // F + base of this (g, k)
    size_t stride;     // between orders
    const double* pw;  // (2 eta^2)^n / (sqrt 2 eta)
    cplx phase;        // e^{-i q.r'}
    const cplx* tw;    // (t/2)^j / j!, off the plane
    cplx* sums;        // this thread's column of the t-series sums (stride LO_T), off the plane
    int nmax, J;
    bool series;
    __device__ void operator()(int i, cplx L) const {
        if (!series) {
            out[i * stride] = cmul(cscale(L, pw[i]), phase);
            return;
        }
        for (int n = max(0, i - J); n <= min(nmax, i); ++n) cfma(sums[n * LO_T], tw[i - n], L);
    }
    __device__ void finish() const {
        if (!series) return;
        for (int n = 0; n <= nmax; ++n) out[n * stride] = cmul(cscale(sums[n * LO_T], pw[n]), phase);
    }
};

// real wavenumber: F_(1/2-i)(v, 0) on the lower side of the cut, v > 0: -i (-1)^i Q_i; v < 0
// (propagating orders, y = -v): Gamma(b_i) y^-b_i + i (-1)^i S_i
__device__ void real_limits(int I, double v, const Recip& rc, const OrderSink& sink) {
    const double az = fabs(v);
    const bool frac = v >= 2.0;
    double g = 0.0;
    int gi = -1;  // g = Gamma(b_gi) az^-b_gi
    order_ladder(I, v, az, frac, rc, [&](int i, double q) {
        if (!frac) {
            if (gi < 0) {
                g = 1.7724538509055160273 / sqrt(az);
                for (int j = 0; j < i; ++j) g *= -az * rc.at_half(j);
            } else {
                for (; gi < i; ++gi) g *= -az * rc.at_half(gi);
                for (; gi > i; --gi) g *= -(gi - 0.5) / az;
            }
            gi = i;
        }
        if (v < 0.0) {
            sink(i, mk(g, (i & 1) ? -q : q));
        } else {
            const double r = frac ? q : g - q;
            sink(i, mk(0.0, (i & 1) ? r : -r));
        }
    });
}

// complex wavenumber: Gamma(b, z)/(-z)^b, e^(i pi b) = +-i (-1)^i for Im z > 0 / below the axis; odd
// turns add -2 Gamma(b)/(-z)^b, Im z > 0 flips the sign (lattice/reduced.rs:18-100, lattice/sheets.rs)
__device__ void complex_limits(int I, cplx z, bool odd_turns, const Recip& rc, const OrderSink& sink) {
    const double az = hypot(z.x, z.y);
    const bool frac = by_fraction(z, az), above = z.y > 0.0;
    const cplx mz = cneg(z), root = cscale(cinv(csqrt_p(mz)), 1.7724538509055160273);
    const bool lead = !frac || odd_turns;  // whether Gamma(b_i)/(-z)^b_i is needed
    cplx g = root;
    int gi = 0;
    order_ladder(I, z, az, frac, rc, [&](int i, cplx q) {
        if (lead) {
            if (gi > i) {  // the downward half starts below i0: again from i = 0
                g = root;
                gi = 0;
            }
            for (; gi < i; ++gi) g = cscale(cmul(g, mz), -rc.at_half(gi));
        }
        const double s = (above ? 1.0 : -1.0) * ((i & 1) ? -1.0 : 1.0);  // phase = i s
        const cplx pq = mk(-s * q.y, s * q.x);
        cplx r = frac ? pq : csub(g, pq);
        if (odd_turns) r = csub(r, cscale(g, 2.0));
        sink(i, above ? cneg(r) : r);
    });
}

template <bool CK, typename Args>
__global__ void __launch_bounds__(LO_T) lattice_orders_kernel(Args A, int nF, int k_first, int k_count, int kw,
                                                              cplx* __restrict__ F) {
    __shared__ double one[LO_TAB], half[LO_TAB], pw[LS_FMAX];
    __shared__ cplx tw[LS_TMAX + 1];
    extern __shared__ __align__(16) unsigned char lo_raw[];
    cplx* sums = reinterpret_cast<cplx*>(lo_raw) + threadIdx.x;  // off the plane: nF columns of LO_T
    const int tid = threadIdx.x;
    const bool series = A.J > 0;
    if (tid < LO_TAB) {
        one[tid] = tid ? 1.0 / tid : 0.0;
        half[tid] = 1.0 / (tid + 0.5);
    }
    if (tid == 0) {
        double f = 1.0 / (1.4142135623730950488 * A.eta);
        for (int n = 0; n < nF; ++n) {
            pw[n] = f;
            f *= 2.0 * A.eta * A.eta;
        }
    }
    if (tid == 32 && series) {
        cplx w = mk(1.0, 0.0), half_t;
        if constexpr (CK)
            half_t = cscale(A.t, 0.5);
        else
            half_t = mk(0.5 * A.t, 0.0);
        for (int j = 0; j <= A.J; ++j) {
            if (j > 0) w = cscale(cmul(w, half_t), 1.0 / j);
            tw[j] = w;
        }
    }
    __syncthreads();
    const long long idx = (long long)blockIdx.x * LO_T + tid;
    const int g = (int)(idx / kw), kk = (int)(idx - (long long)g * kw);
    if (g >= A.NG || kk >= k_count) return;
    const double2 kpar = A.kpar[k_first + kk];
    const double2 G = A.G[g], Gl = A.Glo[g];
    double qx, qy, ex, ey;
    bloch_order(kpar.x, G.x, Gl.x, qx, ex);
    bloch_order(kpar.y, G.y, Gl.y, qy, ey);
    const size_t stride = kw;
    cplx* out = F + (size_t)g * (nF + 1) * stride + kk;
    out[nF * stride] = mk(qx, qy);
    OrderSink sink;
    sink.out = out;
    sink.stride = stride;
    sink.pw = pw;
    sink.tw = tw;
    sink.sums = sums;
    sink.nmax = nF - 1;
    sink.J = A.J;
    sink.series = series;
    double ps, pc;
    sincos(-(qx * A.sx + qy * A.sy), &ps, &pc);
    sink.phase = mk(pc, ps);
    if (series)
        for (int n = 0; n < nF; ++n) sums[n * LO_T] = mk(0.0, 0.0);
    const Recip rc{one, half};
    bool threshold;
    if constexpr (CK) {
        const cplx kinv = cinv(A.k), kinv2 = cmul(kinv, kinv);
        // v = (q.q - k^2) / (2 eta^2 k^2): Re(q.q - k^2) = (q.q - Re(k)^2) + Im(k)^2 compensated
        const cplx d = mk(q2_minus_k2(qx, ex, qy, ey, A.k.x) + A.k.y * A.k.y, -2.0 * A.k.x * A.k.y);
        cplx v = cscale(cmul(d, kinv2), 1.0 / (2.0 * A.eta * A.eta));
        if (v.y == 0.0) v.y = -0.0;  // lower side (lattice/sheets.rs:12-17)
        threshold = hypot(v.x, v.y) <= 1e-14;
        if (!threshold) complex_limits(nF - 1 + A.J, v, odd_turns_of(A, qx * qx + qy * qy, v), rc, sink);
    } else {
        // v = (q.q - k^2) / (2 eta^2 k^2), the difference compensated near a threshold
        const double v = q2_minus_k2(qx, ex, qy, ey, A.k) / (2.0 * A.eta * A.eta * A.k * A.k);
        threshold = fabs(v) <= 1e-14;
        if (!threshold) real_limits(nF - 1 + A.J, v, rc, sink);
    }
    if (threshold) {
        atomicExch(A.status, 9);  // on a diffraction threshold (reciprocal.rs:236-241)
        for (int n = 0; n < nF; ++n) out[n * stride] = mk(0.0, 0.0);
        return;
    }
    sink.finish();
}

// ---- reduction ------------------------------------------------------------------------------
struct ReduceArgs {
    int lsum, hstep, npair;     // hstep: 2 in the plane (even l - |m| only), else 1
    int NR, NG, nF, nk, k_first, k_count, kw;
    const double2* R;
    const double2* tab;         // NR x npair x 2: the table entries of +m and -m
    const cplx* F;
    const double2* coef;        // slots x npair: the polynomial coefficients in the order of their use
    const double2* kpar;
    double2 kinv;
    const double2* pref;        // by lm
    double2 self0;
    double R0x, R0y;
    double2* out;
    size_t ldo;
};
constexpr int LR_T = 256;
constexpr int LR_TILE = 16;  // reciprocal vectors per tile
constexpr int LR_RT = 32;    // real-space points per tile

// PLANE: the shift lies in the lattice plane; the at most 8 coefficients of a pair then sit in
// registers and the polynomial is unrolled (loops over both with coefficients from L1: 1021 Bloch
// vectors 183 us, unrolled 99). Two Bloch vectors a thread, which would share coefficients and table
// entries, measured slower (4096: 0.33 ms against 0.28): the FP64 arithmetic and its latency bound it.
template <bool CK, bool PLANE>
__global__ void __launch_bounds__(LR_T) lattice_reduce_kernel(ReduceArgs A, int tpk) {
    extern __shared__ __align__(16) unsigned char lr_raw[];
    const int kblk = LR_T / tpk;  // Bloch vectors of the CTA, one per group of tpk threads
    const int np = A.lsum + 1;
    cplx* sF = reinterpret_cast<cplx*>(lr_raw);          // [tile][nF][kblk]
    cplx* sZ = sF + (size_t)LR_TILE * A.nF * kblk;       // [tile][np][kblk]: ((q_x + i q_y)/k)^m
    cplx* sZm = sZ + (size_t)LR_TILE * np * kblk;        // the same of q_x - i q_y (complex k only)
    cplx* sB = sZm + (CK ? (size_t)LR_TILE * np * kblk : 0);  // [tile][kblk]: beta^2
    cplx* sP = sB + LR_TILE * kblk;                      // [LR_RT][kblk]: e^{i kpar.R}
    const int tid = threadIdx.x, kl = tid / tpk, p = tid - kl * tpk;
    const int kb0 = blockIdx.x * kblk;  // first Bloch vector (of this chunk)
    const bool active = kl < kblk && p < A.npair;
    // pair p: h = l - |m| ascending (in steps of hstep), |m| ascending
    int h = 0, am = active ? p : 0;
    if (active)
        while (am >= A.lsum - h + 1) {
            am -= A.lsum - h + 1;
            h += A.hstep;
        }
    const int l = h + am;
    cplx accp = mk(0.0, 0.0), accm = mk(0.0, 0.0);
    // reciprocal part
    const cplx kinv2 = cmul(A.kinv, A.kinv);
    const int steps = h / 2;  // Horner steps in beta^2
    cplx creg[PLANE ? LS_NMAX : 1];
    if (PLANE) {
#pragma unroll
        for (int n = 0; n < LS_NMAX; ++n) creg[n] = active && n <= steps ? A.coef[n * A.npair + p] : mk(0.0, 0.0);
    }
    for (int g0 = 0; g0 < A.NG; g0 += LR_TILE) {
        const int cnt = min(LR_TILE, A.NG - g0);
        __syncthreads();
        for (int t = tid; t < cnt * A.nF * kblk; t += LR_T) {
            const int kk = t % kblk, w = t / kblk, g = w / A.nF, n = w - g * A.nF;
            sF[t] = kb0 + kk < A.k_count ? A.F[((size_t)(g0 + g) * (A.nF + 1) + n) * A.kw + kb0 + kk] : mk(0.0, 0.0);
        }
        for (int t = tid; t < cnt * kblk; t += LR_T) {
            const int kk = t % kblk, g = t / kblk;
            const cplx q = kb0 + kk < A.k_count ? A.F[((size_t)(g0 + g) * (A.nF + 1) + A.nF) * A.kw + kb0 + kk]
                                                : mk(0.0, 0.0);
            const double q2 = q.x * q.x + q.y * q.y;
            const cplx zp = cmul(q, A.kinv);
            sB[g * kblk + kk] = cscale(kinv2, q2);
            cplx w = mk(1.0, 0.0);
            for (int m = 0; m < np; ++m) {
                sZ[(g * np + m) * kblk + kk] = w;
                w = cmul(w, zp);
            }
            if (CK) {
                const cplx zm = cmul(cconj(q), A.kinv);
                w = mk(1.0, 0.0);
                for (int m = 0; m < np; ++m) {
                    sZm[(g * np + m) * kblk + kk] = w;
                    w = cmul(w, zm);
                }
            }
        }
        __syncthreads();
        if (!active) continue;
        for (int g = 0; g < cnt; ++g) {
            const cplx* f = sF + (size_t)g * A.nF * kblk + kl;
            const cplx b2 = sB[g * kblk + kl];
            cplx s = mk(0.0, 0.0);
            // Horner in beta^2 over pp = (l - |m| - s)/2; in the plane the order n = s/2, off it n <= s <= 2n
            if (PLANE) {
#pragma unroll
                for (int n = 0; n < LS_NMAX; ++n)
                    if (n <= steps) {
                        const cplx fv = f[n * kblk];
                        if (CK) {
                            if (n > 0) s = cmul(s, b2);
                            cfma(s, creg[n], fv);
                        } else {
                            s.x = fma(s.x, b2.x, creg[n].x * fv.x);
                            s.y = fma(s.y, b2.x, creg[n].x * fv.y);
                        }
                    }
            } else {
                const double2* cf = A.coef + p;
                for (int pp = steps; pp >= 0; --pp) {
                    const int sidx = h - 2 * pp;
                    if (pp < steps) s = CK ? cmul(s, b2) : cscale(s, b2.x);
                    for (int n = (sidx + 1) / 2; n <= sidx; ++n, cf += A.npair) {
                        const double2 c = __ldg(cf);
                        const cplx fv = f[n * kblk];
                        if (CK) {
                            cfma(s, c, fv);
                        } else {
                            s.x = fma(c.x, fv.x, s.x);
                            s.y = fma(c.x, fv.y, s.y);
                        }
                    }
                }
            }
            const int zi = (g * np + am) * kblk + kl;
            const cplx z = sZ[zi];
            cfma(accp, s, z);
            cfma(accm, s, CK ? sZm[zi] : cconj(z));
        }
    }
    const int lmp = l * l + l + am, lmm = l * l + l - am;
    if (active) {
        accp = cmul(A.pref[lmp], accp);
        accm = cmul(A.pref[lmm], accm);
    }
    // real-space part
    cplx rp = mk(0.0, 0.0), rm = mk(0.0, 0.0);
    for (int r0 = 0; r0 < A.NR; r0 += LR_RT) {
        const int cnt = min(LR_RT, A.NR - r0);
        __syncthreads();
        for (int t = tid; t < cnt * kblk; t += LR_T) {
            const int kk = t % kblk, r = t / kblk;
            if (kb0 + kk < A.k_count) {
                const double2 kp = A.kpar[A.k_first + kb0 + kk], R = A.R[r0 + r];
                sP[t] = cexp_i(kp.x * R.x + kp.y * R.y);
            } else {
                sP[t] = mk(0.0, 0.0);
            }
        }
        __syncthreads();
        if (!active) continue;
#pragma unroll 4
        for (int r = 0; r < cnt; ++r) {
            const double2* e = A.tab + ((size_t)(r0 + r) * A.npair + p) * 2;
            const cplx ph = sP[r * kblk + kl];
            cfma(rp, __ldg(e), ph);
            cfma(rm, __ldg(e + 1), ph);
        }
    }
    if (active && kb0 + kl < A.k_count) {
        const size_t row = (size_t)(A.k_first + kb0 + kl);
        const double2 kp = A.kpar[row];
        const cplx back = cexp_i(-(kp.x * A.R0x + kp.y * A.R0y));  // the shift reduced into the cell
        cplx vp = cadd(rp, accp);
        if (l == 0) vp = cadd(vp, A.self0);
        A.out[row * A.ldo + lmp] = cmul(vp, back);
        if (am > 0) A.out[row * A.ldo + lmm] = cmul(cadd(rm, accm), back);
    }
    if (PLANE)  // odd l - |m| vanish in the plane
        for (int t = tid; t < kblk * np * np; t += LR_T) {
            const int kk = t / (np * np), lm = t - kk * np * np;
            int ll = 0;
            while ((ll + 1) * (ll + 1) <= lm) ++ll;
            if (kb0 + kk < A.k_count && ((lm - ll * ll) & 1))  // l + m odd
                A.out[(size_t)(A.k_first + kb0 + kk) * A.ldo + lm] = mk(0.0, 0.0);
        }
}

size_t reduce_smem(bool ck, int lsum, int nF, int kblk) {
    const size_t np = lsum + 1;
    return ((size_t)LR_TILE * kblk * (nF + (ck ? 2 : 1) * np + 1) + (size_t)LR_RT * kblk) * sizeof(cplx);
}

template <bool CK, bool PLANE>
void launch_reduce(const ReduceArgs& r, int tpk, cudaStream_t st) {
    const int kblk = LR_T / tpk;
    static PerDeviceOnce attr;
    once_per_device(attr, [] {
        cudaFuncSetAttribute(lattice_reduce_kernel<CK, PLANE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    });
    lattice_reduce_kernel<CK, PLANE>
        <<<(r.k_count + kblk - 1) / kblk, LR_T, reduce_smem(CK, r.lsum, r.nF, kblk), st>>>(r, tpk);
}

template <bool CK, typename Args>
void launch_sum(const Args& a, double2 kinv, cplx* F, int k_chunk, cudaStream_t st, long long* launches) {
    StageScope sc(ST_LATTICE, st);
    ReduceArgs r;
    r.lsum = a.lsum;
    r.hstep = a.offplane ? 1 : 2;
    r.npair = lattice_pairs(a.lsum, a.offplane);
    r.nF = lattice_orders(a.lsum, a.offplane);
    r.NR = a.NR;
    r.NG = a.NG;
    r.nk = a.nk;
    r.kw = k_chunk;
    r.R = a.R;
    r.tab = a.realtab;
    r.F = F;
    r.coef = a.coef;
    r.kpar = a.kpar;
    r.kinv = kinv;
    r.pref = a.pref;
    r.self0 = a.self0;
    r.R0x = a.R0x;
    r.R0y = a.R0y;
    r.out = a.out;
    r.ldo = a.ldo;
    const int tpk = std::max(32, std::min(LR_T, (r.npair + 31) / 32 * 32));
    const size_t osm = a.J > 0 ? (size_t)r.nF * LO_T * sizeof(cplx) : 0;
    for (int k0 = 0; k0 < a.nk; k0 += k_chunk) {
        r.k_first = k0;
        r.k_count = std::min(k_chunk, a.nk - k0);
        const long long items = (long long)a.NG * k_chunk;
        lattice_orders_kernel<CK, Args><<<(unsigned)((items + LO_T - 1) / LO_T), LO_T, osm, st>>>(a, r.nF, k0, r.k_count,
                                                                                                k_chunk, F);
        if (a.offplane)
            launch_reduce<CK, false>(r, tpk, st);
        else
            launch_reduce<CK, true>(r, tpk, st);
        if (launches) *launches += 2;
    }
}

}  // namespace

int lattice_pairs(int lsum, bool offplane) {
    int n = 0;
    for (int h = 0; h <= lsum; h += offplane ? 1 : 2) n += lsum - h + 1;
    return n;
}
int lattice_orders(int lsum, bool offplane) { return offplane ? lsum + 1 : lsum / 2 + 1; }
// Bloch vectors per pass: the orders of a pass take at most 64 MB (they stay in L2), or one vector's
int lattice_chunk(int lsum, bool offplane, int NG, size_t nk) {
    const size_t per = (size_t)std::max(1, NG) * (lattice_orders(lsum, offplane) + 1) * sizeof(cplx);
    const size_t fit = ((size_t)64 << 20) / per;
    if (fit < 32) return (int)std::max<size_t>(1, std::min(fit, nk));
    return (int)std::min(fit / 32 * 32, (nk + 31) / 32 * 32);
}
size_t lattice_order_bytes(int lsum, bool offplane, int NG, size_t nk) {
    return (size_t)lattice_chunk(lsum, offplane, NG, nk) * std::max(1, NG) * (lattice_orders(lsum, offplane) + 1) *
           sizeof(cplx);
}

void launch_lattice_sum(const LatticeSumArgs& a, cplx* F, cudaStream_t st, long long* launches) {
    launch_sum<false>(a, make_double2(1.0 / a.k, 0.0), F, lattice_chunk(a.lsum, a.offplane, a.NG, a.nk), st, launches);
}
void launch_lattice_sum_ck(const LatticeSumCkArgs& a, cplx* F, cudaStream_t st, long long* launches) {
    const double d = a.k.x * a.k.x + a.k.y * a.k.y;
    launch_sum<true>(a, make_double2(a.k.x / d, -a.k.y / d), F, lattice_chunk(a.lsum, a.offplane, a.NG, a.nk), st,
                     launches);
}

}  // namespace tcu
