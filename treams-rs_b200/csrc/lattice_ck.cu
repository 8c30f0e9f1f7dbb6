// 2D Ewald lattice sums of outgoing spherical waves at a complex wavenumber k (lossy embedding,
// Im k >= 0) and any shift r, with a real split eta (lattice::sum, lattice/mod.rs:283).
//
// The same split as the real-wavenumber kernels of lattice.cu (real space lattice/real.rs:149-187,
// reciprocal space lattice/reciprocal.rs:288-334 with S_lmn of reciprocal.rs:22-60 and the t-series
// of lattice/reduced.rs:223 off the plane, the self term at r' = 0), with every quantity that
// involves k complex:
//   real space   Treal_lm(rho) = -i sqrt(2/pi) (k |rho|)^l N_lm Y_lm(-rho/|rho|) I_2l(k |rho|, eta),
//                I_2l(z, eta) = eta^(2l+1)/2 sum_j c^j/j! R(l + 1/2 - j), R(d) = Gamma(d, a)/a^d at the
//                complex a = (z eta)^2/2 (special/integrals/kambe.rs:36-120). Re(k) > 0 and
//                Im(k) >= 0 with a real eta put z eta in the first quadrant, where z eta/sqrt 2 is the
//                principal root of a, so no reflected ladder arises.
//   reciprocal   F_(1/2-n)(v, 0) = Gamma(1/2-n, v)/(-v)^(1/2-n) at the complex v = (q.q/k^2 - 1)/(2 eta^2)
//                on the outgoing sheet of each diffraction order (lattice/sheets.rs): orders whose
//                k^2 - q.q lies in the near sector of the split take whole turns from the principal
//                argument, an odd number of turns adds -2 Gamma(1/2-n)/(-v)^(1/2-n), and a value
//                above the real axis changes sign (lattice/reduced.rs:18-100).
// Special functions, FP64 complex, from published methods: Gamma(d, z) for half-integer d <= 1/2
// by the power series (DLMF 8.7.3) near the origin and where Re z < 0, else by Legendre's
// continued fraction (DLMF 8.9.2, modified Lentz); R(d) for d > 1/2 by the upward recurrence
// R(d+1) = (d R(d) + e^-a)/a.
//
// Device layout as in lattice.cu: one launch tabulates Treal for the lattice points within the
// cutoff (a warp per point); lattice_sum.cu evaluates the reduced integrals and reduces both parts.
// S_lmn is a polynomial in beta^2 whose coefficients (powers of -k r_z folded in) come from the
// host, so shifts on and off the plane take the same path.
#include <cuda_runtime.h>

#include "common.cuh"
#include "kernels.h"

namespace tcu {

namespace {

constexpr int CK_JMAX = 64;   // Kambe series terms
constexpr int CK_LADDER = LS_MAXL + 1 + CK_JMAX;

__device__ __forceinline__ cplx clog_c(cplx z) { return mk(log(hypot(z.x, z.y)), atan2(z.y, z.x)); }
__device__ __forceinline__ cplx cpow_c(cplx z, double a) {  // principal z^a
    if (z.x == 0.0 && z.y == 0.0) return mk(0.0, 0.0);
    return cexpz(cscale(clog_c(z), a));
}
__device__ __forceinline__ cplx cpowi_c(cplx z, int n) {
    cplx r = mk(1.0, 0.0), b = z;
    unsigned e = (unsigned)(n < 0 ? -n : n);
    while (e) {
        if (e & 1u) r = cmul(r, b);
        b = cmul(b, b);
        e >>= 1;
    }
    return n < 0 ? cinv(r) : r;
}

// Legendre's continued fraction of Gamma(d, z) e^z z^-d (DLMF 8.9.2, even contraction), modified
// Lentz; converges off the negative real axis
__device__ cplx gamma_fraction_c(double d, cplx z) {
    const double tiny = 1e-300;
    cplx b = mk(z.x + 1.0 - d, z.y), c = mk(1.0 / tiny, 0.0), dd = cinv(b), h = dd;
    for (int i = 1; i < 2000; ++i) {
        const double an = -(double)i * ((double)i - d);
        b.x += 2.0;
        dd = cadd(cscale(dd, an), b);
        if (cabs2(dd) < 1e-300) dd = mk(tiny, 0.0);
        c = cadd(b, cscale(cinv(c), an));
        if (cabs2(c) < 1e-300) c = mk(tiny, 0.0);
        dd = cinv(dd);
        const cplx del = cmul(dd, c);
        h = cmul(h, del);
        if (fabs(del.x - 1.0) + fabs(del.y) < 1e-16) break;
    }
    return h;
}

// sum_k (-z)^k / (k! (d + k)) (DLMF 8.7.3 without its leading power)
__device__ cplx gamma_series_sum_c(double d, cplx z) {
    cplx s = mk(1.0 / d, 0.0), term = mk(1.0, 0.0);
    const double az = hypot(z.x, z.y);
    for (int k = 1; k < 600; ++k) {
        term = cscale(cmul(term, cneg(z)), 1.0 / k);
        const cplx add = cscale(term, 1.0 / (d + k));
        s = cadd(s, add);
        if (k > az && cabs2(add) < 1e-36 * cabs2(s)) break;
    }
    return s;
}

__device__ __forceinline__ bool use_fraction(cplx z) {
    const double az = hypot(z.x, z.y);
    return z.x >= 2.0 || (az >= 4.0 && z.x >= -0.3 * az);
}

// R(d) = Gamma(d, a)/a^d for half-integer d <= 1/2 and Re a > 0 (the Kambe ladder below 1/2)
__device__ cplx scaled_gamma_c(double d, cplx a) {
    if (use_fraction(a)) return cmul(cexpz(cneg(a)), gamma_fraction_c(d, a));
    return csub(cscale(cpow_c(a, -d), tgamma(d)), gamma_series_sum_c(d, a));
}

// One warp per lattice point: Treal_lm(R) for every l <= lsum, |m| <= l, complex k.
__global__ void __launch_bounds__(128) real_table_ck_kernel(int lsum, cplx k, double eta, int NR,
                                                            const double2* __restrict__ R, double sx, double sy,
                                                            double sz, const double* __restrict__ norm,
                                                            const double* __restrict__ reflection, int hstep,
                                                            int row, double2* __restrict__ tab) {
    __shared__ cplx ladder[4][CK_LADDER];
    __shared__ cplx kam[4][LS_MAXL + 1];
    __shared__ cplx Y[4][(LS_MAXL + 1) * (LS_MAXL + 1)];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * 4 + warp;
    if (r >= NR) return;
    const int T = (lsum + 1) * (lsum + 1);
    const double2 p = R[r];
    double dist, u[3];
    unit_direction(-p.x - sx, -p.y - sy, -sz, dist, u);  // rho = -r' - R
    const cplx ze = cscale(k, dist * eta);
    const cplx a = cscale(cmul(ze, ze), 0.5);
    const double c = 0.5 / (eta * eta);
    // ladder[i] = R(lsum + 1/2 - i): R(1/2) and below from the series / fraction, above by recurrence
    const int nlad = lsum + 1 + CK_JMAX;
    for (int i = lsum + lane; i < nlad; i += 32) ladder[warp][i] = scaled_gamma_c(lsum + 0.5 - i, a);
    __syncwarp();
    if (lane == 0) {
        const cplx ea = cexpz(cneg(a)), ainv = cinv(a);
        cplx rr = ladder[warp][lsum];
        double d = 0.5;
        for (int i = lsum - 1; i >= 0; --i) {
            rr = cmul(cadd(cscale(rr, d), ea), ainv);
            d += 1.0;
            ladder[warp][i] = rr;
        }
    }
    if (lane <= lsum) solid_column(lsum, lane, u, reflection, Y[warp]);
    __syncwarp();
    if (lane <= lsum) {
        const int l = lane;
        cplx sum = mk(0.0, 0.0);
        double coef = 1.0;
        for (int j = 0; j < CK_JMAX; ++j) {
            if (j > 0) coef *= c / j;
            const cplx term = cscale(ladder[warp][lsum - l + j], coef);
            sum = cadd(sum, term);
            if (j > c + 3.0 && cabs2(term) <= 1e-34 * cabs2(sum)) break;
        }
        kam[warp][l] = cscale(sum, 0.5 * pow(eta, 2 * l + 1));
    }
    __syncwarp();
    const double s2p = 0.79788456080286535588;  // sqrt(2/pi)
    const cplx kd = cscale(k, dist);
    for (int lm = lane; lm < T; lm += 32) {
        int l = (int)sqrt((double)lm);
        while (l * l > lm) --l;
        while ((l + 1) * (l + 1) <= lm) ++l;
        const cplx f = cscale(cmul(cpowi_c(kd, l), kam[warp][l]), s2p * norm[lm]);
        const cplx fy = cmul(f, Y[warp][lm]);
        // -i f y, where the reduction reads it (in the plane odd l - |m| vanish)
        const int at = lattice_pair_index(lsum, l, lm - l * l - l, hstep);
        if (at >= 0) tab[(size_t)r * row + at] = mk(fy.y, -fy.x);
    }
}

}  // namespace

void launch_real_table_ck(int lsum, cplx k, double eta, int NR, const double2* R, double sx, double sy, double sz,
                          const double* norm, const double* reflection, bool offplane, double2* tab, cudaStream_t st) {
    StageScope sc(ST_LATTICE, st);
    real_table_ck_kernel<<<(NR + 3) / 4, 128, 0, st>>>(lsum, k, eta, NR, R, sx, sy, sz, norm, reflection,
                                                       offplane ? 1 : 2, 2 * lattice_pairs(lsum, offplane), tab);
}

}  // namespace tcu
