// dem_flight.cuh -- steps of particles that nothing can touch, many at a time.
//
// In a sparse system most particles have no neighbour close enough to be reached before the next
// list build: a build with quiet classes (ClassSpec::walls) puts those whose every listed
// neighbour, and every wall, keeps a gap above g, and that track no contact, first in the storage
// ([0, nlone + nclear)).  Two particles approach by at most twice the displacement bound, so until
// that reaches g (Ctl::clear_until = g / 2) such a particle only falls freely.  The streaming kernel
// moves its 120 bytes through HBM every step for that; here k_steps_live steps the few others (quiet
// = 1) for up to kFlightSteps steps in one launch, and k_flight then reads each quiet particle once,
// takes the same number of free steps in registers (stream_free_step's arithmetic, so the same
// bits) and writes it once.
//
// What the others see meanwhile: a listed quiet particle's position is up to kFlightSteps old, or
// older in the buffer an even number of steps leaves alone (launch_quiet_begin fills both after a
// build).  Any position it had since the build answers their overlap tests alike: it and they have
// each moved by less than g / 2, so they do not overlap.  Its velocity is read by nobody.  The
// displacement bound needs the quiet ones' largest speed of each step: Ctl::vq2 bounds it at the
// launch's start (the largest |u|^2 seen at a build, a run's start and the end of each flight; |u|^2
// is convex in time under a constant force, so its ends bound a flight), and each step adds at most
// dt |g| to the speed.
//
// Bounds: 120 bytes per particle and flight (HBM), and four FP64 operations per particle, step and
// axis along a force, one along the others; at kFlightSteps = 64 about as long.  Measured (B200, device us per
// step, three-kernel step / this one): 2,000,000 spheres 57 / 7.4; 300,007, FP32 forces 19 / 5.4; 70,001
// 14.3 / 4.6.
#pragma once
#include "dem_particle.cuh"

namespace b200dem {
namespace {

__device__ __forceinline__ void fold_v2(unsigned long long *word, double v2) {
    for (int o = 16; o > 0; o >>= 1) v2 = fmax(v2, __shfl_xor_sync(0xffffffffu, v2, o));
    const unsigned long long b = (unsigned long long)__double_as_longlong(v2);
    if ((threadIdx.x & 31) == 0 && b > *reinterpret_cast<volatile unsigned long long *>(word)) atomicMax(word, b);
}

__global__ void __launch_bounds__(kBlock) k_quiet_begin(Particles P, Ctl *ctl) {
    const int cur = ctl->cur, vcur = ctl->vcur, nq = ctl->nlone + ctl->nclear, cap = P.cap;
    double vq = 0.0, vr = 0.0;   // of the quiet ones, of the others
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P.n; i += gridDim.x * blockDim.x) {
        const double a = P.vel[vcur][i], b = P.vel[vcur][cap + i], c = P.vel[vcur][2 * cap + i];
        const double v2 = a * a + b * b + c * c;
        if (i < nq) {
            st4(P.pos[cur ^ 1], i, ld4(P.pos[cur], i));
            vq = fmax(vq, v2);
        } else {
            vr = fmax(vr, v2);
        }
    }
    fold_v2(&ctl->vq2, vq);
    fold_v2(&ctl->vr2, vr);
}

__global__ void __launch_bounds__(256) k_flight(Particles P, Ctl *ctl, ForceConsts fc) {
    const int steps = ctl->flight_steps;
    if (steps <= 0) return;
    const int nq = ctl->nlone + ctl->nclear, cap = P.cap, last = ctl->flight_last;
    const double4 *pc = P.pos[ctl->flight_cur];
    double4 *pn = P.pos[ctl->cur];
    double *vel = P.vel[ctl->vcur];
    double v2 = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nq; i += gridDim.x * blockDim.x) {
        D4 p = ld4(pc, i);
        const double m = P.mI[i], m_inverse = 1. / m;
        const bool held = fc.has_fix && (P.fix[i] & DEM_FIX_FORCE);
        double u[3], a[3], F[3], x[3] = {p.x, p.y, p.z};
        for (int d = 0; d < 3; ++d) {
            u[d] = vel[d * cap + i];
            F[d] = fc.has_gravity ? dadd(0., dmul(m, fc.g[d])) : 0.;
            if (held) F[d] = 0.;
            a[d] = dmul(dmul(fc.half_dt, F[d]), m_inverse);
        }
        for (int d = 0; d < 3; ++d) {
            if (a[d] == 0.) {   // along no force: the speed stays (a zero's sign aside), and so does the drift
                if (steps > last) u[d] = dadd(dadd(u[d], a[d]), a[d]);
                const double du = dmul(fc.dt, u[d]);
                for (int k = 0; k < steps - last; ++k) x[d] = dadd(x[d], du);
            } else {
                for (int k = 0; k < steps - last; ++k) {
                    u[d] = dadd(dadd(u[d], a[d]), a[d]);
                    x[d] = dadd(x[d], dmul(fc.dt, u[d]));
                }
            }
        }
        if (last)   // the run's last step: no drift, F and tau stored
            for (int d = 0; d < 3; ++d) {
                u[d] = dadd(u[d], a[d]);
                P.force[d * cap + i] = F[d];
                P.torque[d * cap + i] = 0.;
            }
        p.x = x[0];
        p.y = x[1];
        p.z = x[2];
        st4(pn, i, p);
        for (int d = 0; d < 3; ++d) vel[d * cap + i] = u[d];
        v2 = fmax(v2, u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
    }
    fold_v2(&ctl->vq2, v2);
}

}  // namespace

void launch_quiet_begin(const Particles &P, Ctl *ctl, cudaStream_t s) { k_quiet_begin<<<148 * 12, kBlock, 0, s>>>(P, ctl); }
void launch_flight(const Particles &P, Ctl *ctl, const ForceConsts &fc, cudaStream_t s) {
    k_flight<<<148 * 8, 256, 0, s>>>(P, ctl, fc);
}

}  // namespace b200dem
