// dem_div.cuh -- divisions of the contact law that share a denominator, with the bits of three `/`.
//
// The FP64 pair law divides four vectors by a length or a stiffness: twelve of its eighteen divisions,
// each a chain of some fourteen dependent instructions behind a branch of its own, so that they run one
// after another (114 cycles each).  Here one division gives y = RN(1/b) and each quotient follows by
// multiplications: q0 = RN(a y) is within 1.5 ulp of a/b, one residual step makes it faithful (within
// 0.5 ulp and a hair), and a second one rounds correctly by Markstein's theorem (P. W. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34,
// 1990): for y = RN(1/b) and a faithful q, RN(q + RN(a - q b) y) = RN(a/b).  The three chains overlap.
// The theorem asks that nothing overflows and no residual loses bits: b and each a in [2^-500, 2^500),
// or a = 0; anything else (a NaN among them) takes the plain divisions.
//
// Measured (B200, FP64): see pp_pair in dem_particle.cuh.
#pragma once

namespace b200dem {
namespace {

__device__ __forceinline__ bool div_plain_range(const double v) {   // 2^-500 <= |v| < 2^500
    return (((unsigned)__double2hiint(v) >> 20) & 0x7ffu) - 523u < 1000u;
}

__device__ __forceinline__ double div_by(const double a, const double b, const double y) {
    const double q0 = a * y;
    const double q1 = __fma_rn(__fma_rn(-q0, b, a), y, q0);
    const double q2 = __fma_rn(__fma_rn(-q1, b, a), y, q1);
    return a == 0. ? q0 : q2;   // a zero keeps its sign
}

// q[d] = a[d] / b
__device__ __forceinline__ void div3(const double a0, const double a1, const double a2, const double b, double &q0,
                                     double &q1, double &q2) {
    if (div_plain_range(b) && (div_plain_range(a0) || a0 == 0.) && (div_plain_range(a1) || a1 == 0.) &&
        (div_plain_range(a2) || a2 == 0.)) {
        const double y = 1. / b;
        q0 = div_by(a0, b, y);
        q1 = div_by(a1, b, y);
        q2 = div_by(a2, b, y);
    } else {
        q0 = a0 / b;
        q1 = a1 / b;
        q2 = a2 / b;
    }
}

}  // namespace
}  // namespace b200dem
