// boys.cuh -- device Boys function F_0..F_m(x) in FP64.
//
// Same scheme as the reference (src/integrals/boys.f90:202-281): x < 25 ->
// 5-point Chebyshev interpolation of F_m on one of 500 intervals
// (cheb_approx_5, chebinterp.f90:122-149), then downward recursion
// F_{k-1} = (2x F_k + e^{-x}) / (2k-1); x >= 25 -> F_0 = sqrt(pi/x)/2 and
// upward recursion.  The coefficient table is built on the host
// (host_math.cpp) and read through the read-only data path.
#pragma once
#include "gci_common.h"

namespace gci {

// Factors of a primitive quartet with exponent sums P and Q (auto2e_WMatrix_part1.f90:134):
// alpha = PQ / (P + Q + kappa PQ) and 2 pi^{5/2} / (PQ sqrt(P + Q + kappa PQ)), both from
// r = 1 / (PQ sqrt(..)): alpha = (PQ)^3 r^2.  One reciprocal square root where the quotients and
// the root as written take three times the FP64 instructions (with the one in boys_fm: Coulomb
// gradient of 280 AOs 38.3 -> 32.6 ms, which this pipe bounds).  PQ PQ (P + Q + kappa PQ) has to
// stay a finite number: exponent sums below 1e60.  The class kernels keep the quotients, because the
// order of tied pivots follows the last bits of the diagonal they evaluate (arguments of boys_fm from
// kBoysXAsym on changed bits there with its reciprocal root).
__device__ __forceinline__ void quartet_factors(double P, double Q, double kappa, double& alpha, double& pref)
{
    const double PQ = P * Q;
    const double den = fma(kappa, PQ, P + Q);
    const double r = rsqrt(PQ * PQ * den);
    alpha = PQ * ((PQ * r) * (PQ * r));
    pref = 34.986836655249725 * r;
}

template <int M>
__device__ __forceinline__ void boys_fm(double x, const double* __restrict__ table, double (&F)[M + 1])
{
    // both branches need it where M > 0, and a warp often takes both
    const double expmx = M > 0 ? exp(-x) : 0.0;
    if (x < kBoysXAsym) {
        const int k = static_cast<int>(x * (1.0 / kBoysDelta));
        const int kk = k < kBoysNInt ? k : kBoysNInt - 1;
        const double* c = table + (static_cast<size_t>(M) * kBoysNInt + kk) * 5;
        const double ab_sum = static_cast<double>(2 * kk + 1) * kBoysDelta;
        const double y = (2.0 * x - ab_sum) * (1.0 / kBoysDelta);
        const double twoy = 2.0 * y;
        const double d5 = __ldg(c + 4);
        const double d4 = twoy * d5 + __ldg(c + 3);
        const double d3 = twoy * d4 - d5 + __ldg(c + 2);
        const double d2 = twoy * d3 - d4 + __ldg(c + 1);
        double f = y * d2 - d3 + 0.5 * __ldg(c + 0);
        F[M] = f;
        if constexpr (M > 0) {
            const double twox = 2.0 * x;
#pragma unroll
            for (int l = M; l >= 1; --l) {
                f = (twox * f + expmx) * (1.0 / static_cast<double>(2 * l - 1));
                F[l - 1] = f;
            }
        }
    } else {
        const double r = rsqrt(x);
        double f = 0.88622692545275801365 * r;   // sqrt(pi) / 2
        F[0] = f;
        if constexpr (M > 0) {
            const double beta = 0.5 * r * r;
#pragma unroll
            for (int l = 1; l <= M; ++l) {
                f = beta * (static_cast<double>(2 * l - 1) * f - expmx);
                F[l] = f;
            }
        }
    }
}

} // namespace gci
