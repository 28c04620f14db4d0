// dem_bonded.cu -- bonded-DEM bond build and fused bond-force step on sm_100a (FP64,
// built with --fmad=false; the expressions follow the reference's order).
//
//   k_bond_setup   setupBonds (src/CabanaBondedDEM_Particles.hpp:118-137): over the
//                  neighbour list (ascending caller index) bond every j with
//                  rij < factor * rad(i), rest length = rij
//   k_bond_step    one bonded step in the order of tst_01_BDEM:295-306: force reset, external
//                  force, computeBondedForce (src/CabanaBondedDEM_Force.hpp:86-341), boundary
//                  hook, stage3, then stage1 + stage2 of the next step (ping-pong buffers)
//   k_bond_force   computeBondedForce alone, for callers that drive the bonded loop phase by
//                  phase (with k_add_ext_force and k_post_hooks for the example's hooks)
//
// Bond slots are slot-major per particle: partner (sorted index), rest length, and the 9 live
// history components (tangential force, normal and tangential moments; the reference's
// bond_fn_* arrays are never written, :69-71).  Breakage (no reference counterpart): a bond
// whose FP64 strain (rij - L0) / L0 exceeds the threshold is flagged and skipped from then on;
// both ends compute the same strain bit for bit, so they break in the same step.
#include "dem_bulk.cuh"
#include "dem_gridstep.cuh"
#include "dem_particle.cuh"

namespace b200dem {

namespace {

constexpr int kBondBlock = 128;

__global__ void k_bond_setup(Particles P, NbrList L, Bonds B, Ctl *ctl, double factor) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    const int cur = ctl->cur, cap = P.cap;
    const D4 pi = ld4(P.pos[cur], i);
    int cnt = 0;
    int status = 0;
    for (int kk = 0; kk < L.nn[i]; ++kk) {
        const int j = L.idx[(long)kk * cap + i];
        const D4 pj = ld4(P.pos[cur], j);
        const double px = pi.x - pj.x, py = pi.y - pj.y, pz = pi.z - pj.z;
        const double r2ij = px * px + py * py + pz * pz;
        const double rij = sqrt(r2ij);
        const double bond_cond = factor * pi.w;
        if (rij < bond_cond) {
            if (cnt >= B.mb) {
                status |= DEM_ERR_BOND_OVERFLOW;
                continue;
            }
            B.idx[(long)cnt * cap + i] = j;
            B.init_len[(long)cnt * cap + i] = rij;
            ++cnt;
        }
    }
    B.count[i] = cnt;
    for (int k = cnt; k < B.mb; ++k) B.idx[(long)k * cap + i] = -1;
    if (status) atomicOr(&ctl->status, status);
}

// R = double: the reference's FP64 arithmetic (bitwise parity with the oracle).  R = float
// (mixed precision): strain, geometry and relative kinematics stay FP64 (rij - L0 and the
// breakage test are exact), the bond force/moment history is stored and updated in FP32
// (half the history traffic), per-particle sums and integration are FP64.
template <typename R>
__device__ __forceinline__ R *bond_hist(const Bonds &B);
template <>
__device__ __forceinline__ double *bond_hist<double>(const Bonds &B) { return B.hist; }
template <>
__device__ __forceinline__ float *bond_hist<float>(const Bonds &B) { return B.hist32; }

// What a bond reads of its partner.
struct BondPartner {
    D4 p;
    double u[3], w[3];
};
__device__ __forceinline__ BondPartner bond_partner(const double4 *pc, const double *vc, const double *wc, const int cap,
                                                    const int j) {
    BondPartner q;
    q.p = ld4(pc, j);
    for (int d = 0; d < 3; ++d) {
        q.u[d] = vc[d * cap + j];
        q.w[d] = wc[d * cap + j];
    }
    return q;
}

// Bond stiffnesses (BondedDEM_Force.hpp:186-198, or the given ones) for the smaller radius rmin.
struct BondStiff {
    double n, t, tor, ben;
};
__device__ __forceinline__ BondStiff bond_stiff(const BondConsts &bc, const double rmin, const double rad_sum,
                                                const double Ei, const double Gi) {
    const double bond_rad = rmin * bc.radius_factor;
    const double A_bond = M_PI * (bond_rad * bond_rad);
    const double I_bond = M_PI * ((bond_rad * bond_rad) * (bond_rad * bond_rad)) / 4.0;
    const double I_p_bond = I_bond * 2.0;
    BondStiff s;
    if (bc.quirks & BQ11_HARDCODED_K) {
        s.n = Ei * A_bond / rad_sum;
        s.t = Gi * A_bond / rad_sum;
        s.tor = Gi * I_p_bond / rad_sum;
        s.ben = Ei * I_bond / rad_sum;
    } else {
        s.n = bc.kn;
        s.t = bc.kt;
        s.tor = bc.kt * I_p_bond / A_bond;
        s.ben = bc.kn * I_bond / A_bond;
    }
    return s;
}

// One bond of particle i (BondedDEM_Force.hpp:53-348) with rest length L0 and history h[9] (tangential
// force, twisting and bending moments; in and out): strain and breakage, normal force, incremental
// shear force, moments.  Returns false when it breaks now (nothing changed); else cf receives the
// bond's contribution to F (0..2) and tau (3..5) of i, which the caller adds in slot order.  `own`:
// bond_stiff for i's own radius, taken when that is the smaller one and only it counts.  Divisions
// bound the law: what a bond repeats step after step (the stiffnesses' two, the strain's while it is
// clearly below the threshold, the two of a ratio that is multiplied by zero) is left out, with the
// same results.
template <typename R>
__device__ __forceinline__ bool bond_law(const BondConsts &bc, const BondStiff &own, const D4 &pi, const double ui0, const double ui1,
                                         const double ui2, const double wi0, const double wi1, const double wi2,
                                         const double Ei, const double Gi, const BondPartner &q, const double L0,
                                         const double dt, R (&h)[9], double (&cf)[6]) {
    const double px = pi.x - q.p.x, py = pi.y - q.p.y, pz = pi.z - q.p.z;
    const double r2ij = px * px + py * py + pz * pz;
    const double rij = sqrt(r2ij);
    if (bc.break_strain > 0.0) {
        // (rij - L0) / L0 > break_strain; the quotient only where it can be near the threshold
        if (!(rij - L0 < 0.999999 * bc.break_strain * L0 && L0 > 0.) && (rij - L0) / L0 > bc.break_strain) {
            return false;
        }
    }
    const double g_c = rij - pi.w - q.p.w;
    const double a_i = pi.w + g_c / 2.;
    const double a_j = q.p.w + g_c / 2.;
    const double n0 = px / rij, n1 = py / rij, n2 = pz / rij;
    const double uj0 = q.u[0];
    const double uj1 = (bc.quirks & BQ1_VELJ_USES_UI) ? ui1 : q.u[1];
    const double uj2 = (bc.quirks & BQ1_VELJ_USES_UI) ? ui2 : q.u[2];
    const double wj0 = q.w[0], wj1 = q.w[1], wj2 = q.w[2];
    const double vi0 = ui0 + (wi1 * n2 - wi2 * n1) * a_i;
    const double vi1 = ui1 + (wi2 * n0 - wi0 * n2) * a_i;
    const double vi2 = ui2 + (wi0 * n1 - wi1 * n0) * a_i;
    const double vj0 = uj0 + (-wj1 * n2 + wj2 * n1) * a_j;
    const double vj1 = uj1 + (-wj2 * n0 + wj0 * n2) * a_j;
    const double vj2 = uj2 + (-wj0 * n1 + wj1 * n0) * a_j;
    const double vr0 = vi0 - vj0, vr1 = vi1 - vj1, vr2 = vi2 - vj2;
    const double vdp = vr0 * n0 + vr1 * n1 + vr2 * n2;
    const double vn0 = vdp * n0, vn1 = vdp * n1, vn2 = vdp * n2;
    const double vt0 = vr0 - vn0, vt1 = vr1 - vn1, vt2 = vr2 - vn2;
    const double wr0 = wi0 - wj0, wr1 = wi1 - wj1, wr2 = wi2 - wj2;
    const double wdp = wr0 * n0 + wr1 * n1 + wr2 * n2;
    const double wn0 = wdp * n0, wn1 = wdp * n1, wn2 = wdp * n2;
    const double wt0 = wr0 - wn0, wt1 = wr1 - wn1, wt2 = wr2 - wn2;
    const double rad_sum = pi.w + q.p.w;
    const double beta_bond = bc.beta;
    const BondStiff ks = (pi.w <= q.p.w && !(bc.quirks & BQ11_HARDCODED_K)) ? own
                                                                           : bond_stiff(bc, pi.w < q.p.w ? pi.w : q.p.w,
                                                                                        rad_sum, Ei, Gi);
    const double k_n_bond = ks.n, k_t_bond = ks.t, k_tor_bond = ks.tor, k_ben_bond = ks.ben;
    // normal bond force (:205-222)
    const double overlap_n = rij - L0;
    const R rn0 = (R)n0, rn1 = (R)n1, rn2 = (R)n2;
    const R fn0 = -(R)k_n_bond * (R)overlap_n * rn0;
    const R fn1 = -(R)k_n_bond * (R)overlap_n * rn1;
    const R fn2 = -(R)k_n_bond * (R)overlap_n * rn2;
    const R beta_b = (R)beta_bond;
    R mX = (vn0 >= 0.0) ? (R)1 : (R)-1;
    R mY = (vn1 >= 0.0) ? (R)1 : (R)-1;
    R mZ = (vn2 >= 0.0) ? (R)1 : (R)-1;
    const R fd0 = fn0 + beta_b * fabs(fn0) * mX;
    const R fd1 = fn1 + beta_b * fabs(fn1) * mY;
    const R fd2 = fn2 + beta_b * fabs(fn2) * mZ;
    // tangential bond force (:231-260)
    R ft0 = h[0], ft1 = h[1], ft2 = h[2];
    const R fdp = ft0 * rn0 + ft1 * rn1 + ft2 * rn2;
    ft0 -= fdp * rn0;
    ft1 -= fdp * rn1;
    ft2 -= fdp * rn2;
    R tmp = (R)k_t_bond * (R)dt;
    ft0 += -(R)vt0 * tmp;
    ft1 += -(R)vt1 * tmp;
    ft2 += -(R)vt2 * tmp;
    mX = (vt0 >= 0.0) ? (R)1 : (R)-1;
    mY = (vt1 >= 0.0) ? (R)1 : (R)-1;
    mZ = (vt2 >= 0.0) ? (R)1 : (R)-1;
    const R ftd0 = ft0 - beta_b * fabs(ft0) * mX;
    const R ftd1 = ft1 - beta_b * fabs(ft1) * mY;
    const R ftd2 = ft2 - beta_b * fabs(ft2) * mZ;
    h[0] = ftd0;
    h[1] = ftd1;
    h[2] = ftd2;
    // twisting moment (:267-291)
    R tn0 = h[3], tn1 = h[4], tn2 = h[5];
    R tdp = tn0 * rn0 + tn1 * rn1 + tn2 * rn2;
    tn0 = tdp * rn0;
    tn1 = tdp * rn1;
    tn2 = tdp * rn2;
    tmp = (R)k_tor_bond * (R)dt;
    tn0 += -(R)wn0 * tmp;
    tn1 += -(R)wn1 * tmp;
    tn2 += -(R)wn2 * tmp;
    mX = (wn0 >= 0.0) ? (R)1 : (R)-1;
    mY = (wn1 >= 0.0) ? (R)1 : (R)-1;
    mZ = (wn2 >= 0.0) ? (R)1 : (R)-1;
    const R nd0 = tn0 - beta_b * fabs(tn0) * mX;
    const R nd1 = tn1 - beta_b * fabs(tn1) * mY;
    const R nd2 = tn2 - beta_b * fabs(tn2) * mZ;
    h[3] = nd0;
    h[4] = nd1;
    h[5] = nd2;
    // bending moment (:298-322)
    R tt0 = h[6], tt1 = h[7], tt2 = h[8];
    tdp = tt0 * rn0 + tt1 * rn1 + tt2 * rn2;
    tt0 -= tdp * rn0;
    tt1 -= tdp * rn1;
    tt2 -= tdp * rn2;
    tmp = (R)k_ben_bond * (R)dt;
    tt0 += -(R)wt0 * tmp;
    tt1 += -(R)wt1 * tmp;
    tt2 += -(R)wt2 * tmp;
    mX = (wt0 >= 0.0) ? (R)1 : (R)-1;
    mY = (wt1 >= 0.0) ? (R)1 : (R)-1;
    mZ = (wt2 >= 0.0) ? (R)1 : (R)-1;
    const R td0 = tt0 - beta_b * fabs(tt0) * mX;
    const R td1 = tt1 - beta_b * fabs(tt1) * mY;
    const R td2 = tt2 - beta_b * fabs(tt2) * mZ;
    h[6] = td0;
    h[7] = td1;
    h[8] = td2;
    // the reference's cri * 0: zero unless the ratio is not finite
    double cri = 0.0;
    if (!(pi.w > 1e-100 && rad_sum > 1e-100 && rij < 1e100)) cri = rij * 1. / pi.w * 1. / (pi.w + q.p.w);
    cf[0] = (double)(fd0 + ftd0);
    cf[1] = (double)(fd1 + ftd1);
    cf[2] = (double)(fd2 + ftd2);
    cf[3] = (double)(nd0 + td0) - cri * 0.0;
    cf[4] = (double)(nd1 + td1) - cri * 0.0;
    cf[5] = (double)(nd2 + td2) - cri * 0.0;
    return true;
}

// bond_law on slot k of particle i in global memory.  Returns false when the slot holds no live bond
// (empty, broken now or before, or its partner-indexed history slot overflows).
template <typename R>
__device__ __forceinline__ bool bond_term(const Particles &P, const Bonds &B, const BondConsts &bc, R *__restrict__ hist,
                                          const double4 *__restrict__ pc, const double *__restrict__ vc,
                                          const double *__restrict__ wc, const int cap, const int i, const int k,
                                          const D4 &pi, const double ui0, const double ui1, const double ui2,
                                          const double wi0, const double wi1, const double wi2, const double Ei,
                                          const double Gi, const double dt, int &status, double (&cf)[6]) {
    const long slot = (long)k * cap + i;
    const int j = B.idx[slot];
    if (j < 0 || B.broken[slot]) return false;
    long hs = slot;
    if (bc.quirks & BQ10_INDEX_BY_J) {
        const int jc = P.perm[j];
        if (jc >= B.mb) {
            status |= DEM_ERR_BOND_OVERFLOW;
            return false;
        }
        hs = (long)jc * cap + i;
    }
    R h[9];
    for (int c = 0; c < 9; ++c) h[c] = hist[((long)c * B.mb) * cap + hs];
    const BondStiff own = bond_stiff(bc, pi.w, 1., Ei, Gi);
    if (!bond_law<R>(bc, own, pi, ui0, ui1, ui2, wi0, wi1, wi2, Ei, Gi, bond_partner(pc, vc, wc, cap, j), B.init_len[hs], dt, h,
                     cf)) {
        B.broken[slot] = 1;
        return false;
    }
    for (int c = 0; c < 9; ++c) hist[((long)c * B.mb) * cap + hs] = h[c];
    return true;
}

// Hooks (gravity, applyBoundaryConditions of tst_01_BDEM:50-60) and the velocity-Verlet
// update of particle i after its bond pass; u, omega to the other velocity buffer.
__device__ __forceinline__ void bond_finish_particle(const Particles &P, const ForceConsts &fc, const int i,
                                                     const int nxt, const int vcur, const bool last, const D4 &pi,
                                                     double ui0, double ui1, double ui2, double wi0, double wi1,
                                                     double wi2, const double2 mIi, double F0, double F1, double F2,
                                                     double T0, double T1, double T2, double &vmax2) {
    const int cap = P.cap;
    if (fc.has_gravity) {
        F0 += mIi.x * fc.g[0];
        F1 += mIi.x * fc.g[1];
        F2 += mIi.x * fc.g[2];
    }
    if (fc.has_fix) {   // applyBoundaryConditions (tst_01_BDEM:50-60)
        const int f = P.fix[i];
        if (f & DEM_FIX_FORCE) F0 = F1 = F2 = 0.;
        if (f & DEM_FIX_TORQUE) T0 = T1 = T2 = 0.;
    }
    const double m_inverse = 1. / mIi.x, I_inverse = 1. / mIi.y, h = fc.half_dt;
    ui0 += h * F0 * m_inverse;
    ui1 += h * F1 * m_inverse;
    ui2 += h * F2 * m_inverse;
    wi0 += h * T0 * I_inverse;
    wi1 += h * T1 * I_inverse;
    wi2 += h * T2 * I_inverse;
    D4 pn = pi;
    if (last) {
        P.force[i] = F0;
        P.force[cap + i] = F1;
        P.force[2 * cap + i] = F2;
        P.torque[i] = T0;
        P.torque[cap + i] = T1;
        P.torque[2 * cap + i] = T2;
    } else {
        ui0 += h * F0 * m_inverse;
        ui1 += h * F1 * m_inverse;
        ui2 += h * F2 * m_inverse;
        wi0 += h * T0 * I_inverse;
        wi1 += h * T1 * I_inverse;
        wi2 += h * T2 * I_inverse;
        pn.x += fc.dt * ui0;
        pn.y += fc.dt * ui1;
        pn.z += fc.dt * ui2;
        vmax2 = ui0 * ui0 + ui1 * ui1 + ui2 * ui2;
    }
    st4(P.pos[nxt], i, pn);
    double *vn = P.vel[vcur ^ 1], *wn = P.omg[vcur ^ 1];
    vn[i] = ui0;
    vn[cap + i] = ui1;
    vn[2 * cap + i] = ui2;
    wn[i] = wi0;
    wn[cap + i] = wi1;
    wn[2 * cap + i] = wi2;
}

template <typename R>
__global__ void __launch_bounds__(kBondBlock) k_bond_step(Particles P, Bonds B, Ctl *ctl, ForceConsts fc, BondConsts bc) {
    grid_dep_wait();   // launched as a dependent (launch_k): the kernel before has completed
    grid_dep_release();
    R *__restrict__ hist = bond_hist<R>(B);
    const CtlSnap cs_ = read_ctl(ctl, true);
    if (!cs_.go) return;
    const int cur = cs_.cur, nxt = cur ^ 1, vcur = ctl->vcur;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int cap = P.cap;
    double vmax2 = 0.0;
    int status = 0;
    if (i < P.n) {
        const double4 *__restrict__ pc = P.pos[cur];
        const double *__restrict__ vc = P.vel[vcur];
        const double *__restrict__ wc = P.omg[vcur];
        const D4 pi = ld4(pc, i);
        double ui0 = vc[i], ui1 = vc[cap + i], ui2 = vc[2 * cap + i];
        double wi0 = wc[i], wi1 = wc[cap + i], wi2 = wc[2 * cap + i];
        const double2 mIi = load_mI(P, i);
        double F0 = 0., F1 = 0., F2 = 0., T0 = 0., T1 = 0., T2 = 0.;
        if (fc.has_ext) {   // applyTensileForce (tst_01_BDEM:101-111) before the bond pass
            F0 += P.ext[i];
            F1 += P.ext[cap + i];
            F2 += P.ext[2 * cap + i];
        }
        const double Ei = B.E[i], Gi = B.G[i];
        const int no_bonds_i = B.count[i];
        for (int k = 0; k < no_bonds_i; k++) {
            double cf[6];
            if (!bond_term<R>(P, B, bc, hist, pc, vc, wc, cap, i, k, pi, ui0, ui1, ui2, wi0, wi1, wi2, Ei, Gi, fc.dt,
                              status, cf))
                continue;
            F0 += cf[0];
            F1 += cf[1];
            F2 += cf[2];
            T0 += cf[3];
            T1 += cf[4];
            T2 += cf[5];
        }
        bond_finish_particle(P, fc, i, nxt, vcur, cs_.last, pi, ui0, ui1, ui2, wi0, wi1, wi2, mIi, F0, F1, F2, T0, T1,
                             T2, vmax2);
    }
    finish_step(ctl, P.vslots, vmax2, fc.dt, status, true, true);
}

// The fused step with a tile's bonds staged in shared memory: a block takes kBondBlock consecutive
// particles, and one bulk copy per row brings in their partners, rest lengths, break flags and
// histories, kBondRing slots ahead of the law, each slot on a barrier of its own.  A thread then waits
// for its partner's state only, where it waited for the partner's index, the partner and the history
// of each bond in turn.  Histories are stored from registers.  Slot-indexed histories only (BQ10
// clear); `slots`: the largest bond count.  Waits are bounded: one that gives up sets DEM_ERR_TIMEOUT
// and leaves the step unfinished.
// What bounds it: resident warps (16 per SM at 128 registers) against partners' loads and the law's
// dependent FP64 chain.  131,072 particles, us per step, FP64 / FP32 history (B200): 33.4 / 33.4 without
// the staging (and with five more divisions per bond, see bond_law), 27.6 / 23.4 with it; all slots
// staged at once (three blocks per SM) 32.4 / 29.5; the next bond's partner read ahead into registers
// 29.8 / 25.2; five blocks per SM 28.9 / 25.4 (spills).
template <typename R>
struct BondTile {
    static constexpr int T = kBondBlock;
    static constexpr int HIST = 0, LEN = 9 * T * (int)sizeof(R), IDX = LEN + 8 * T, BROKEN = IDX + 4 * T,
                         BYTES = BROKEN + T;   // of one slot
};
constexpr int kBondRing = 4;   // slots of a tile in shared memory at a time
constexpr int kBondWaitLimit = 1 << 18;

template <typename R>
__global__ void __launch_bounds__(kBondBlock, 4) k_bond_step_tile(Particles P, Bonds B, Ctl *ctl, ForceConsts fc,
                                                               BondConsts bc, int slots) {
    using BT = BondTile<R>;
    constexpr int T = BT::T;
    grid_dep_wait();   // launched as a dependent (launch_k): the kernel before has completed
    grid_dep_release();
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ uint64_t full[kBondRing];
    R *__restrict__ hist = bond_hist<R>(B);
    const CtlSnap cs_ = read_ctl(ctl, true);
    if (!cs_.go) return;
    const int cap = P.cap, i0 = blockIdx.x * T, i = i0 + threadIdx.x;
    if (threadIdx.x < kBondRing) bulk::bar_init(&full[threadIdx.x], 1);
    bulk::bar_init_fence();
    __syncthreads();
    auto issue = [&](int k) {   // one thread: the rows of slot k into place k % kBondRing
        const uint32_t m = (uint32_t)min(T, cap - i0);   // 64 or T: cap is a multiple of 64
        unsigned char *s = sm + (long)(k % kBondRing) * BT::BYTES;
        uint64_t *bar = &full[k % kBondRing];
        const long row = (long)k * cap + i0;
        bulk::bar_arrive_expect(bar, m * (9u * (uint32_t)sizeof(R) + 8u + 4u + 1u));
        if (fc.drop_copies) return;   // testing the bounded waits: nothing will arrive
        bulk::copy_g2s(s + BT::IDX, B.idx + row, 4u * m, bar);
        bulk::copy_g2s(s + BT::BROKEN, B.broken + row, m, bar);
        bulk::copy_g2s(s + BT::LEN, B.init_len + row, 8u * m, bar);
        for (int c = 0; c < 9; ++c)
            bulk::copy_g2s(s + BT::HIST + c * T * (int)sizeof(R), hist + ((long)c * B.mb * cap + row), m * (uint32_t)sizeof(R),
                           bar);
    };
    if (threadIdx.x < kBondRing && threadIdx.x < slots) issue(threadIdx.x);
    const int cur = cs_.cur, nxt = cur ^ 1, vcur = ctl->vcur;
    double vmax2 = 0.0;
    bool ok = true;
    const double4 *__restrict__ pc = P.pos[cur];
    const double *__restrict__ vc = P.vel[vcur];
    const double *__restrict__ wc = P.omg[vcur];
    const bool have = i < P.n;
    const int ii = have ? i : i0;
    const D4 pi = ld4(pc, ii);
    const double ui0 = vc[ii], ui1 = vc[cap + ii], ui2 = vc[2 * cap + ii];
    const double wi0 = wc[ii], wi1 = wc[cap + ii], wi2 = wc[2 * cap + ii];
    const double2 mIi = load_mI(P, ii);
    double F0 = 0., F1 = 0., F2 = 0., T0 = 0., T1 = 0., T2 = 0.;
    if (fc.has_ext) {   // applyTensileForce (tst_01_BDEM:101-111) before the bond pass
        F0 += P.ext[ii];
        F1 += P.ext[cap + ii];
        F2 += P.ext[2 * cap + ii];
    }
    const double Ei = B.E[ii], Gi = B.G[ii];
    const BondStiff own = bond_stiff(bc, pi.w, 1., Ei, Gi);
    const int count = have ? B.count[i] : 0;
    // partner of slot k, -1 without a live bond there
    auto partner_of = [&](int k) {
        if (k >= count) return -1;
        const unsigned char *s = sm + (long)(k % kBondRing) * BT::BYTES;
        const int j = reinterpret_cast<const int *>(s + BT::IDX)[threadIdx.x];
        return s[BT::BROKEN + threadIdx.x] ? -1 : j;
    };
    const int limit = fc.wait_polls > 0 ? fc.wait_polls : kBondWaitLimit;
    int k = 0;
    for (; k < slots; ++k) {
        ok = ok && bulk::bar_wait(&full[k % kBondRing], (k / kBondRing) & 1, limit);
        const int j = ok ? partner_of(k) : -1;
        BondPartner q = {};
        if (j >= 0) q = bond_partner(pc, vc, wc, cap, j);
        const unsigned char *s = sm + (long)(k % kBondRing) * BT::BYTES;
        R h[9];
        double L0 = 0.;
        if (j >= 0) {
            const R *sh = reinterpret_cast<const R *>(s + BT::HIST) + threadIdx.x;
#pragma unroll
            for (int c = 0; c < 9; ++c) h[c] = sh[c * T];
            L0 = reinterpret_cast<const double *>(s + BT::LEN)[threadIdx.x];
        }
        if (k + kBondRing < slots) {   // place k % kBondRing is read: its next slot
            if (__syncthreads_or(ok ? 0 : 1)) break;
            if (threadIdx.x == 0) issue(k + kBondRing);
        }
        if (j < 0) continue;
        double cf[6];
        const long slot = (long)k * cap + i;
        if (!bond_law<R>(bc, own, pi, ui0, ui1, ui2, wi0, wi1, wi2, Ei, Gi, q, L0, fc.dt, h, cf)) {
            B.broken[slot] = 1;
            continue;
        }
#pragma unroll
        for (int c = 0; c < 9; ++c) hist[(long)c * B.mb * cap + slot] = h[c];
        F0 += cf[0];
        F1 += cf[1];
        F2 += cf[2];
        T0 += cf[3];
        T1 += cf[4];
        T2 += cf[5];
    }
    if (__syncthreads_or(ok ? 0 : 1)) {   // report, and let the copies in flight land before the block leaves
        if (threadIdx.x == 0) atomicOr(&ctl->status, DEM_ERR_TIMEOUT);
        const int issued = min(slots, k + kBondRing);   // the last copies into each place of the ring
        for (int r = max(0, issued - kBondRing); r < issued; ++r)
            bulk::bar_wait(&full[r % kBondRing], (r / kBondRing) & 1, limit);
        return;
    }
    if (have)
        bond_finish_particle(P, fc, i, nxt, vcur, cs_.last, pi, ui0, ui1, ui2, wi0, wi1, wi2, mIi, F0, F1, F2, T0, T1, T2,
                             vmax2);
    finish_step(ctl, P.vslots, vmax2, fc.dt, 0, true, true);
}

// A run of a small specimen in one cooperative launch: eight lanes per particle, a bond each, with the
// bond's history, rest length and partner and the particle's state in registers for the whole run.
// Per step a lane reads its partner, evaluates its bond, and the eight add the terms in slot order
// (each lane all of them, so that each holds the new state); lanes 0, 1 and 2 store position,
// velocity and spin for the partners, and a grid barrier ends the step.  Slot-indexed histories, at
// most eight bonds per particle, at most the particles resident at once (bond_loop_capacity).
// One thread per particle walking its bonds, a launch per step: 18.7 us per step on 3,003 particles
// (FP32 history) and 19.5 on 7,200 (FP64); this form 3.5 and 4.2 (B200), of which 1.2 is the barrier.
template <typename R>
__global__ void __launch_bounds__(kBondBlock, 4) k_bond_loop(Particles P, Bonds B, Ctl *ctl, ForceConsts fc,
                                                             BondConsts bc, int max_steps, unsigned long long *scratch) {
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ GridStep<kBondBlock> bar;
    R *hist = bond_hist<R>(B);
    const int lane = threadIdx.x & 31, k = lane & 7, g0 = lane & 24, n = P.n, cap = P.cap;
    const int i = (blockIdx.x * kBondBlock + threadIdx.x) / 8;
    const bool have = i < n;
    const int ii = have ? i : 0;
    int cur = ctl->cur, vcur = ctl->vcur, done = ctl->steps_done, steps = 0;
    const int target = ctl->target;
    const bool stopped = (ctl->status & kStopBits) != 0;
    const double half = ctl->half_skin;
    double disp = ctl->disp;
    D4 x = ld4(P.pos[cur], ii);
    double u[3], w[3];
    for (int d = 0; d < 3; ++d) {
        u[d] = P.vel[vcur][d * cap + ii];
        w[d] = P.omg[vcur][d * cap + ii];
    }
    const double2 mI = load_mI(P, ii);
    const double m_inverse = 1. / mI.x, I_inverse = 1. / mI.y, hdt = fc.half_dt;
    const double Ei = B.E[ii], Gi = B.G[ii];
    const int fix = fc.has_fix ? P.fix[ii] : 0;
    double ext[3] = {0., 0., 0.};
    if (fc.has_ext)
        for (int d = 0; d < 3; ++d) ext[d] = P.ext[d * cap + ii];
    const BondStiff own = bond_stiff(bc, x.w, 1., Ei, Gi);
    // this lane's bond
    const int count = have ? B.count[ii] : 0;
    const long slot = (long)k * cap + ii;
    int j = -1;
    double L0 = 0.;
    R h[9] = {};
    if (k < count) {
        j = B.broken[slot] ? -1 : B.idx[slot];
        L0 = B.init_len[slot];
        for (int c = 0; c < 9; ++c) h[c] = hist[(long)c * B.mb * cap + slot];
    }
    const int most = (int)__reduce_max_sync(FULL, (unsigned)count);
    bool ok = true;
    for (int s = 0; s < max_steps; ++s) {
        if (!(done < target && !stopped && disp < half && ok)) break;   // the same in every block
        const bool last = done + 1 >= target;
        double cf[6] = {0., 0., 0., 0., 0., 0.};
        bool acts = false;
        if (j >= 0) {
            acts = bond_law<R>(bc, own, x, u[0], u[1], u[2], w[0], w[1], w[2], Ei, Gi,
                               bond_partner(P.pos[cur], P.vel[vcur], P.omg[vcur], cap, j), L0, fc.dt, h, cf);
            if (!acts) {   // broken now, skipped from here on
                B.broken[slot] = 1;
                j = -1;
            }
        }
        const unsigned act = __ballot_sync(FULL, acts) >> g0;
        double F[3] = {0., 0., 0.}, T[3] = {0., 0., 0.};
        if (fc.has_ext)   // applyTensileForce (tst_01_BDEM:101-111) before the bond pass
            for (int d = 0; d < 3; ++d) F[d] += ext[d];
        for (int q = 0; q < most; ++q) {
            double t[6];
#pragma unroll
            for (int c = 0; c < 6; ++c) t[c] = __shfl_sync(FULL, cf[c], g0 + q);
            if ((act >> q) & 1u)
                for (int d = 0; d < 3; ++d) {
                    F[d] += t[d];
                    T[d] += t[3 + d];
                }
        }
        if (fc.has_gravity)
            for (int d = 0; d < 3; ++d) F[d] += mI.x * fc.g[d];
        if (fix & DEM_FIX_FORCE) F[0] = F[1] = F[2] = 0.;
        if (fix & DEM_FIX_TORQUE) T[0] = T[1] = T[2] = 0.;
        double v2 = 0.0;
        for (int d = 0; d < 3; ++d) {
            const double a = hdt * F[d] * m_inverse, b = hdt * T[d] * I_inverse;
            u[d] += a;
            w[d] += b;
            if (!last) {
                u[d] += a;
                w[d] += b;
            }
        }
        if (!last) {
            x.x += fc.dt * u[0];
            x.y += fc.dt * u[1];
            x.z += fc.dt * u[2];
            if (have) v2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
        }
        if (have) {
            if (k == 0) st4(P.pos[cur ^ 1], i, x);
            if (k == 1)
                for (int d = 0; d < 3; ++d) P.vel[vcur ^ 1][d * cap + i] = u[d];
            if (k == 2)
                for (int d = 0; d < 3; ++d) P.omg[vcur ^ 1][d * cap + i] = w[d];
            if (last && k == 3)
                for (int d = 0; d < 3; ++d) {
                    P.force[d * cap + i] = F[d];
                    P.torque[d * cap + i] = T[d];
                }
        }
        unsigned long long big;
        int total;
        ok = grid_step<kBondBlock>(bar, ctl, fc, scratch, s, v2, 0, big, total);
        if (!ok) break;
        disp = disp + fc.dt * sqrt(__longlong_as_double((long long)big)) * (1.0 + 1e-9);
        cur ^= 1;
        vcur ^= 1;
        done += 1;
        steps += 1;
    }
    if (k < count)
        for (int c = 0; c < 9; ++c) hist[(long)c * B.mb * cap + slot] = h[c];
    if (blockIdx.x == 0 && threadIdx.x == 0) {   // the control word as finish_step leaves it
        ctl->cur = cur;
        ctl->vcur = vcur;
        ctl->steps_done = done;
        ctl->total_steps += steps;
        ctl->disp = disp;
        ctl->ndefer = 0;
    }
}

// computeBondedForce as a phase of its own (src/CabanaBondedDEM_Force.hpp:53-348): for every
// particle, F and tau += the bond terms in slot order, starting from the F and tau the earlier
// phases left (resetForcesAndTorques, then the caller's hooks).  Same per-bond arithmetic as
// the fused step (bond_term), so a loop of phases equals the fused step bit for bit.
template <typename R>
__global__ void __launch_bounds__(kBondBlock) k_bond_force(Particles P, Bonds B, Ctl *ctl, BondConsts bc, double dt) {
    R *__restrict__ hist = bond_hist<R>(B);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    const int cur = ctl->cur, vcur = ctl->vcur, cap = P.cap;
    const double4 *__restrict__ pc = P.pos[cur];
    const double *__restrict__ vc = P.vel[vcur];
    const double *__restrict__ wc = P.omg[vcur];
    const D4 pi = ld4(pc, i);
    const double ui0 = vc[i], ui1 = vc[cap + i], ui2 = vc[2 * cap + i];
    const double wi0 = wc[i], wi1 = wc[cap + i], wi2 = wc[2 * cap + i];
    double F0 = P.force[i], F1 = P.force[cap + i], F2 = P.force[2 * cap + i];
    double T0 = P.torque[i], T1 = P.torque[cap + i], T2 = P.torque[2 * cap + i];
    const double Ei = B.E[i], Gi = B.G[i];
    int status = 0;
    const int no_bonds_i = B.count[i];
    for (int k = 0; k < no_bonds_i; k++) {
        double cf[6];
        if (!bond_term<R>(P, B, bc, hist, pc, vc, wc, cap, i, k, pi, ui0, ui1, ui2, wi0, wi1, wi2, Ei, Gi, dt, status,
                          cf))
            continue;
        F0 += cf[0];
        F1 += cf[1];
        F2 += cf[2];
        T0 += cf[3];
        T1 += cf[4];
        T2 += cf[5];
    }
    P.force[i] = F0;
    P.force[cap + i] = F1;
    P.force[2 * cap + i] = F2;
    P.torque[i] = T0;
    P.torque[cap + i] = T1;
    P.torque[2 * cap + i] = T2;
    if (status) atomicOr(&ctl->status, status);
}

// The hook in the position of tst_01_BDEM's applyTensileForce (:101-111): F += the external
// force (DEM_F_EXT_FORCE).
__global__ void k_add_ext_force(Particles P) {
    const int cap = P.cap;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P.n; i += gridDim.x * blockDim.x) {
        P.force[i] += P.ext[i];
        P.force[cap + i] += P.ext[cap + i];
        P.force[2 * cap + i] += P.ext[2 * cap + i];
    }
}

// The hooks in the position of tst_01_BDEM's applyBoundaryConditions (:19-67): gravity (m g
// added), then the DEM_FIX_* flags zero F and/or tau -- the order of the fused step.
__global__ void k_post_hooks(Particles P, ForceConsts fc) {
    const int cap = P.cap;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P.n; i += gridDim.x * blockDim.x) {
        if (fc.has_gravity) {
            const double m = load_mI(P, i).x;
            P.force[i] += m * fc.g[0];
            P.force[cap + i] += m * fc.g[1];
            P.force[2 * cap + i] += m * fc.g[2];
        }
        if (fc.has_fix) {
            const int f = P.fix[i];
            if (f & DEM_FIX_FORCE) P.force[i] = P.force[cap + i] = P.force[2 * cap + i] = 0.;
            if (f & DEM_FIX_TORQUE) P.torque[i] = P.torque[cap + i] = P.torque[2 * cap + i] = 0.;
        }
    }
}

__global__ void k_bond_broken_count(Bonds B, int n, unsigned long long *out) {
    unsigned long long c = 0;
    for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < (long)B.mb * B.cap; t += (long)gridDim.x * blockDim.x)
        c += B.broken[t] ? 1 : 0;
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

}  // namespace

void launch_bond_setup(const Particles &P, const NbrList &L, const Bonds &B, Ctl *ctl, double factor, cudaStream_t s) {
    k_bond_setup<<<(P.n + 127) / 128, 128, 0, s>>>(P, L, B, ctl, factor);
}

template <typename R>
static bool bond_step_tile(const Particles &P, const Bonds &B, Ctl *ctl, const ForceConsts &fc, const BondConsts &bc,
                           int slots, cudaStream_t s) {
    constexpr int bytes = kBondRing * BondTile<R>::BYTES;
    if (bc.quirks & BQ10_INDEX_BY_J) return false;
    if (cudaFuncSetAttribute((const void *)k_bond_step_tile<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) !=
        cudaSuccess)
        return false;
    return launch_k(k_bond_step_tile<R>, (P.n + kBondBlock - 1) / kBondBlock, kBondBlock, (size_t)bytes, s, fc.pdl, P, B, ctl,
                    fc, bc, slots) == cudaSuccess;
}

// `slots`: the largest bond count of a particle.
void launch_bond_step(const Particles &P, const Bonds &B, Ctl *ctl, const ForceConsts &fc, const BondConsts &bc, int slots,
                      cudaStream_t s) {
    if (B.hist32 ? bond_step_tile<float>(P, B, ctl, fc, bc, slots, s) : bond_step_tile<double>(P, B, ctl, fc, bc, slots, s))
        return;
    const int g = (P.n + kBondBlock - 1) / kBondBlock;
    if (B.hist32)
        launch_k(k_bond_step<float>, g, kBondBlock, 0, s, fc.pdl, P, B, ctl, fc, bc);
    else
        launch_k(k_bond_step<double>, g, kBondBlock, 0, s, fc.pdl, P, B, ctl, fc, bc);
}

template <typename R>
static int bond_loop_fit() {   // particles resident at once
    static thread_local PerDevice fit;
    return resident_blocks(fit, (const void *)k_bond_loop<R>, kBondBlock) * (kBondBlock / 8);
}
int bond_loop_capacity(const Bonds &B, const BondConsts &bc, int slots) {
    if (slots > 8 || (bc.quirks & BQ10_INDEX_BY_J)) return 0;
    return B.hist32 ? bond_loop_fit<float>() : bond_loop_fit<double>();
}
cudaError_t launch_bond_loop(const Particles &P, const Bonds &B, Ctl *ctl, const ForceConsts &fc, const BondConsts &bc,
                             int max_steps, unsigned long long *scratch, cudaStream_t s) {
    const cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(unsigned long long) * 6, s);
    if (e != cudaSuccess) return e;
    Particles p = P;
    Bonds b = B;
    ForceConsts f = fc;
    BondConsts c = bc;
    void *args[] = {&p, &b, &ctl, &f, &c, &max_steps, &scratch};
    const void *kernel = B.hist32 ? (const void *)k_bond_loop<float> : (const void *)k_bond_loop<double>;
    return cudaLaunchCooperativeKernel(kernel, dim3((8 * P.n + kBondBlock - 1) / kBondBlock), dim3(kBondBlock), args, 0, s);
}

void launch_bond_force(const Particles &P, const Bonds &B, Ctl *ctl, const BondConsts &bc, double dt, cudaStream_t s) {
    if (B.hist32)
        k_bond_force<float><<<(P.n + kBondBlock - 1) / kBondBlock, kBondBlock, 0, s>>>(P, B, ctl, bc, dt);
    else
        k_bond_force<double><<<(P.n + kBondBlock - 1) / kBondBlock, kBondBlock, 0, s>>>(P, B, ctl, bc, dt);
}

void launch_add_ext_force(const Particles &P, cudaStream_t s) {
    if (P.ext) k_add_ext_force<<<(P.n + 255) / 256, 256, 0, s>>>(P);
}

void launch_post_hooks(const Particles &P, const ForceConsts &fc, cudaStream_t s) {
    if (fc.has_gravity || fc.has_fix) k_post_hooks<<<(P.n + 255) / 256, 256, 0, s>>>(P, fc);
}

void launch_bond_broken_count(const Bonds &B, int n, unsigned long long *out, cudaStream_t s) {
    cudaMemsetAsync(out, 0, sizeof(unsigned long long), s);
    k_bond_broken_count<<<148 * 4, 256, 0, s>>>(B, n, out);
}

}  // namespace b200dem
