// dem_live.cuh -- the step loop of a small system in one cooperative launch, each particle in a
// thread's registers.
//
// A thread holds its particle's position, velocity, gravity increment and first list entries for
// the whole launch.  Per step it reads its listed partners' positions and marks the entries and
// walls that may overlap; a particle that tracks no contact and has no mark takes the free step
// (free_step's arithmetic: two adds of the constant half-kick, the drift), the others live_contact,
// which is particle_full's sequence for the marked entries and walls.  New positions and
// velocities are stored for the partners, and one grid barrier ends the step.
//
// k_steps_coop_lean (dem_persist.cuh) reloads each particle's state and runs the full body in every
// thread.  Measured (B200, device us per step, that form / this one): 4,096 spheres, no pair in
// contact 6.6 / 4.8, some 9.0 / 5.6; 30,011 spheres 11.0 / 6.9, FP32 forces 9.8 / 5.8; 200 spheres
// 7.5 / 5.4; a column of disks with most in contact, 5,000 29.5 / 20.6, 56,000 36.0 / 26.2
// (some of it the pair law's).  Contacts
// by eight lanes each (particle_coop) instead took 11.2 us on the 4,096: some 1,400 dependent
// instructions of a contact, staged through shared memory, where a thread has its own state at hand.
// What bounds it: the barrier (1.2 us) and the chain of one contact's divisions and square roots.
//
// Velocities alternate between two buffers, since a contact reads its partner's velocities of the
// step; only particles in contact are read, so a free particle's spin, which does not change, is
// copied over only in the step after a contact.
//
// quiet (dem_flight.cuh): only the particles [nlone + nclear, n) are stepped; the others cannot
// touch anything until the displacement bound reaches ctl->clear_until, and k_flight advances them
// afterwards by the steps taken.  The second buffer is then the deferred-velocity arrays, and the
// bound on the quiet ones' speed enters the displacement bound.
#pragma once
#include "dem_gridstep.cuh"
#include "dem_particle.cuh"

namespace b200dem {
namespace {

// The step of a particle that tracks or may have contacts, from the thread's registers: the
// statements of particle_full, for the list entries of `pairs` (bit kk: entry kk may overlap; all
// entries from 31 on when bit 31 is set) and the walls of `near` (bit lw) or of the history only,
// since the others' are skipped there as well.  x and u are updated, v2 is |u|^2 of the drift.
template <bool MIXED>
__device__ __forceinline__ void live_contact(const Particles &P, const NbrList &L, const ForceConsts &fc,
                                             const PairConst *__restrict__ pp, const PairConst *__restrict__ pw,
                                             const WallGeom *__restrict__ walls, const double4 *pc, double4 *pn,
                                             const double *vc, const double *wc, double *vn, double *wn, const int last,
                                             const int i, const int j0, const int j1, const int nn, const unsigned pairs,
                                             const unsigned near, const int wall0, const double m, D4 &x, double (&u)[3],
                                             int &cs, double &v2, int &status) {
    const int cap = P.cap;
    const unsigned q = fc.quirks;
    double w[3];
    for (int d = 0; d < 3; ++d) w[d] = wc[d * cap + i];
    const double I = P.mI[(long)cap + i];
    const SceneConst *scn = fc.scenes ? fc.scenes + (P.scene ? P.scene[i] : 0) : nullptr;
    const int mi = fc.nmat > 1 ? (int)P.mat[i] : 0;
    int cnt = cs & 0xff;
    unsigned wmask = (unsigned)cs >> 8;
    int *tidx = P.tidx + i;
    double *thx = P.th + i, *thy = P.th + (long)P.mc * cap + i, *thz = P.th + 2L * P.mc * cap + i;
    // One tracked partner, and it is the first marked entry (most steps of a contact): the list's test
    // decides whether its slot stays, so the partner's position is not read for the compaction first (4,096
    // spheres 5.94 -> 5.64 us per step; columns, with several contacts each, 1 % slower).
    const int kf = pairs ? __ffs(pairs) - 1 : nn;
    const int t0 = cnt == 1 ? tidx[0] : -1;
    const bool early = !MIXED && cnt == 1;   // its history with it (FP32 forces: 5.88 us with, 5.81 without)
    const double g0 = early ? thx[0] : 0., g1 = early ? thy[0] : 0., g2 = early ? thz[0] : 0.;
    const bool lone = t0 >= 0 && kf < nn && t0 == (kf == 0 ? j0 : kf == 1 ? j1 : L.idx[(long)kf * cap + i]);
    double F0 = 0., F1 = 0., F2 = 0., T0 = 0., T1 = 0., T2 = 0.;
    if (fc.has_ext) {
        F0 += P.ext[i];
        F1 += P.ext[cap + i];
        F2 += P.ext[2 * cap + i];
    }
    // ---- update_tangential_contacts (Force.hpp:364-441)
    if (cnt > 0 && !lone) {
        int count = 0, k = 0;
        const int total = cnt;
        int back = cnt - 1;
        while (count < total) {
            const int sidx = tidx[(long)k * cap];
            if (sidx == -1) break;
            const D4 pj = ld4(pc, sidx);
            const double px = x.x - pj.x, py = x.y - pj.y, pz = x.z - pj.z;
            const double r2ij = px * px + py * py + pz * pz;
            const double rij = sqrt(r2ij);
            const double overlap = x.w + pj.w - rij;
            if (overlap <= 0.) {
                const long a = (long)k * cap, b = (long)back * cap;
                if (k == back) {
                    tidx[a] = -1;
                    thx[a] = 0.;
                    thy[a] = 0.;
                    thz[a] = 0.;
                } else {
                    tidx[a] = tidx[b];
                    tidx[b] = -1;
                    thx[a] = thx[b];
                    thx[b] = 0.;
                    thy[a] = thy[b];
                    thy[b] = 0.;
                    thz[a] = thz[b];
                    thz[b] = 0.;
                    back -= 1;
                }
                cnt -= 1;
            } else {
                k = k + 1;
            }
            count += 1;
        }
    }
    // ---- particle-particle (Force.hpp:73-329), list in ascending caller index
    unsigned todo = pairs;
    for (int kk = kf; kk < nn;) {
        const int j = kk == 0 ? j0 : kk == 1 ? j1 : L.idx[(long)kk * cap + i];
        const D4 pj = ld4(pc, j);
        const Mate b = load_mate(P.mI, vc, wc, cap, j);   // most marked entries are in contact
        const double px = x.x - pj.x, py = x.y - pj.y, pz = x.z - pj.z;
        const double r2ij = px * px + py * py + pz * pz;
        const double sr = x.w + pj.w;
        const double rij = sqrt(r2ij);
        const double overlap = sr - rij;
        if (!(r2ij >= sr * sr * 1.0000000001) && overlap > 0.) {
            // slot lookup / insert (Force.hpp:166-192)
            int found_at = lone && kk == kf ? 0 : -1;
            if (found_at < 0)
                for (int s = 0; s < cnt; ++s)
                    if (tidx[(long)s * cap] == j) found_at = s;
            double h0 = 0., h1 = 0., h2 = 0.;
            if (found_at < 0) {
                if (cnt < P.mc) {
                    found_at = cnt;
                    cnt += 1;
                    tidx[(long)found_at * cap] = j;
                } else {
                    status |= DEM_ERR_CONTACT_OVERFLOW;
                }
            } else if (!MIXED && lone && kk == kf) {
                h0 = g0;
                h1 = g1;
                h2 = g2;
            } else {
                const long a = (long)found_at * cap;
                h0 = thx[a];
                h1 = thy[a];
                h2 = thz[a];
            }
            const int mj = fc.nmat > 1 ? (int)P.mat[j] : 0;
            const PairConst c = pp[mi * fc.nmat + mj];
            double cf[6];
            pp_pair<MIXED>(b, q, x, pj, px, py, pz, rij, overlap, u[0], u[1], u[2], w[0], w[1], w[2], m,
                           c, scn ? scn->K_n_pp : fc.K_n_pp, scn ? scn->K_t_pp : fc.K_t_pp, scn ? scn->mu_pp : fc.mu_pp,
                           fc.dt, h0, h1, h2, cf);
            if (found_at >= 0) {
                const long a = (long)found_at * cap;
                thx[a] = h0;
                thy[a] = h1;
                thz[a] = h2;
            }
            F0 += cf[0];
            F1 += cf[1];
            F2 += cf[2];
            if (!(q & DEM_Q3_NO_PP_TORQUE)) {
                T0 += cf[3];
                T1 += cf[4];
                T2 += cf[5];
            }
        } else if (lone && kk == kf && x.w + pj.w - rij <= 0.) {   // the compaction of the lone slot
            tidx[0] = -1;
            thx[0] = 0.;
            thy[0] = 0.;
            thz[0] = 0.;
            cnt = 0;
        }
        if (kk < 31) {   // the next marked entry; from 31 on every entry
            todo &= todo - 1u;
            kk = todo ? __ffs(todo) - 1 : nn;
        } else {
            ++kk;
        }
    }
    // ---- particle-infinite wall (Force.hpp:475-673)
    for (unsigned ws = near | wmask; ws; ws &= ws - 1u) {
        const int lw = __ffs(ws) - 1;
        const WallGeom g = walls[wall0 + lw];
        const double px = x.x - g.x[0], py = x.y - g.x[1], pz = x.z - g.x[2];
        const double nx = g.n[0], ny = g.n[1], nz = g.n[2];
        const double tmp = px * nx + py * ny + pz * nz;
        const double overlap = x.w - tmp;
        const unsigned bit = 1u << lw;
        double *swx = P.sw + (long)lw * cap + i;
        double *swy = P.sw + (long)(P.mw + lw) * cap + i;
        double *swz = P.sw + (long)(2 * P.mw + lw) * cap + i;
        if (overlap > 0.) {
            double cf[6];
            pw_wall<MIXED>(q, x, nx, ny, nz, overlap, u[0], u[1], u[2], w[0], w[1], w[2], g.u[0], g.u[1], g.u[2], m,
                           pw[mi * fc.nwall + wall0 + lw], scn ? scn->K_n_pw : fc.K_n_pw, scn ? scn->K_t_pw : fc.K_t_pw,
                           scn ? scn->mu_pw : fc.mu_pw, fc.dt, (wmask & bit) != 0u, swx, swy, swz, cf);
            wmask |= bit;
            F0 += cf[0];
            F1 += cf[1];
            F2 += cf[2];
            T0 += cf[3];
            T1 += cf[4];
            T2 += cf[5];
        } else if (wmask & bit) {
            *swx = 0.;
            *swy = 0.;
            *swz = 0.;
            wmask &= ~bit;
        }
    }
    const int cs1 = cnt | (int)(wmask << 8);
    if (cs1 != cs) P.cstate[i] = cs1;
    cs = cs1;
    // ---- hooks after the pair forces, stage3 and the next step's stage1 + stage2
    double F[3] = {F0, F1, F2}, T[3] = {T0, T1, T2};
    if (fc.has_gravity)
        for (int d = 0; d < 3; ++d) F[d] = dadd(F[d], dmul(m, fc.g[d]));
    if (fc.has_fix) {
        const int f = P.fix[i];
        if (f & DEM_FIX_FORCE) F[0] = F[1] = F[2] = 0.;
        if (f & DEM_FIX_TORQUE) T[0] = T[1] = T[2] = 0.;
    }
    const double m_inverse = 1. / m, I_inverse = 1. / I, h = fc.half_dt;
    for (int d = 0; d < 3; ++d) {
        const double a = dmul(dmul(h, F[d]), m_inverse), b = dmul(dmul(h, T[d]), I_inverse);
        u[d] = dadd(u[d], a);
        w[d] = dadd(w[d], b);
        if (last) {
            P.force[d * cap + i] = F[d];
            P.torque[d * cap + i] = T[d];
        } else {
            u[d] = dadd(u[d], a);
            w[d] = dadd(w[d], b);
        }
    }
    if (!last) {
        x.x = dadd(x.x, dmul(fc.dt, u[0]));
        x.y = dadd(x.y, dmul(fc.dt, u[1]));
        x.z = dadd(x.z, dmul(fc.dt, u[2]));
        v2 = dadd(dadd(dmul(u[0], u[0]), dmul(u[1], u[1])), dmul(u[2], u[2]));
    }
    st4(pn, i, x);
    for (int d = 0; d < 3; ++d) {
        vn[d * cap + i] = u[d];
        wn[d * cap + i] = w[d];
    }
}

// List entries of particle i at x that may overlap (bit kk, 31 for all from 31 on; the exact early-out
// of the contact loop) and walls it may touch (bit lw; a margin above the law's own test).
__device__ __forceinline__ void live_marks(const NbrList &L, const int cap, const WallGeom *__restrict__ walls,
                                           const double4 *pc, const D4 &x, const int i, const int nn, const int j0,
                                           const int j1, const int wall0, const int wall1, unsigned &pairs,
                                           unsigned &near) {
    auto touches = [&](const D4 &pj) {
        const double px = dadd(x.x, -pj.x), py = dadd(x.y, -pj.y), pz = dadd(x.z, -pj.z);
        const double r2 = dadd(dadd(dmul(px, px), dmul(py, py)), dmul(pz, pz));
        const double sr = dadd(x.w, pj.w);
        return !(r2 >= dmul(dmul(sr, sr), 1.0000000001));
    };
    pairs = near = 0u;
    if (nn > 0) {
        const D4 pa = ld4(pc, j0), pb = ld4(pc, nn > 1 ? j1 : j0);
        pairs = (touches(pa) ? 1u : 0u) | (nn > 1 && touches(pb) ? 2u : 0u);
        for (int k0 = 2; k0 < nn; k0 += 4) {   // four entries' indices, then their positions, in flight
            int j[4];
            D4 p[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) j[c] = L.idx[(long)min(k0 + c, nn - 1) * cap + i];
#pragma unroll
            for (int c = 0; c < 4; ++c) p[c] = ld4(pc, j[c]);
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (touches(p[c])) pairs |= 1u << min(min(k0 + c, nn - 1), 31);
        }
    }
    for (int q = wall0; q < wall1; ++q) {
        const WallGeom &g = walls[q];
        const double at = (x.x - g.x[0]) * g.n[0] + (x.y - g.x[1]) * g.n[1] + (x.z - g.x[2]) * g.n[2];
        near |= !(at > x.w * 1.000001) ? 1u << (q - wall0) : 0u;
    }
}

template <bool MIXED>
__global__ void __launch_bounds__(kBlock, 3) k_steps_live(Particles P, NbrList L, Ctl *ctl, ForceConsts fc,
                                                          const PairConst *__restrict__ pp,
                                                          const PairConst *__restrict__ pw,
                                                          const WallGeom *__restrict__ walls, int max_steps,
                                                          unsigned long long *scratch, int quiet) {
    __shared__ GridStep<kBlock> bar;
    const int n = P.n, cap = P.cap;
    const int cur0 = ctl->cur, vcur0 = ctl->vcur, target = ctl->target;
    const int first = quiet ? ctl->nlone + ctl->nclear : 0;
    const bool stopped = (ctl->status & kStopBits) != 0;
    const double half = ctl->half_skin, until = quiet ? fmin(half, ctl->clear_until) : half;
    const bool wfar_ok = ctl->wfar_build == ctl->rebuilds;
    const double vq = quiet ? sqrt(__longlong_as_double((long long)ctl->vq2)) : 0.0;
    const double ga = sqrt(fc.g[0] * fc.g[0] + fc.g[1] * fc.g[1] + fc.g[2] * fc.g[2]);
    double disp = ctl->disp;
    int done = ctl->steps_done, cur = cur0, steps = 0, ncon = 0;
    double *v0 = P.vel[vcur0], *w0 = P.omg[vcur0];   // velocities of the step, and of the next
    double *v1 = quiet ? L.defer_v : P.vel[vcur0 ^ 1], *w1 = quiet ? L.defer_w : P.omg[vcur0 ^ 1];
    // this thread's particle
    const int i = first + blockIdx.x * kBlock + threadIdx.x;
    const bool have = i < n;
    D4 x = {0., 0., 0., 0.};
    double u[3] = {0., 0., 0.}, a[3] = {0., 0., 0.}, m = 1.;
    int cs = 0, nn = 0, j0 = 0, j1 = 0, wall0 = 0, wall1 = 0;
    bool far = true, spin = false;
    if (have) {
        x = ld4(P.pos[cur], i);
        m = P.mI[i];
        cs = P.cstate[i];
        nn = L.nn[i];
        far = L.wfar[i] != 0;
        j0 = nn > 0 ? L.idx[i] : 0;
        j1 = nn > 1 ? L.idx[cap + i] : 0;
        const int scene_i = P.scene ? P.scene[i] : 0;
        wall0 = fc.wps ? scene_i * fc.wps : 0;
        wall1 = fc.wps ? wall0 + fc.wps : fc.nwall;
        const bool held = fc.has_fix && (P.fix[i] & DEM_FIX_FORCE);
        const double m_inverse = 1. / m;
        for (int d = 0; d < 3; ++d) {
            u[d] = v0[d * cap + i];
            w1[d * cap + i] = w0[d * cap + i];
            double F = 0.;
            if (fc.has_ext) F = dadd(F, P.ext[d * cap + i]);
            if (fc.has_gravity) F = dadd(F, dmul(m, fc.g[d]));
            if (held) F = 0.;
            a[d] = dmul(dmul(fc.half_dt, F), m_inverse);
        }
    }
    bool ok = true;
    for (int k = 0; k < max_steps; ++k) {
        // the same in every block
        if (!(done < target && !stopped && disp < until && ok)) break;
        const int last = done + 1 >= target;
        const bool wfar = wfar_ok && 2.0 * disp < half;
        const double4 *pc = P.pos[cur];
        double v2 = 0.0;
        int status = 0;
        bool full = false;
        if (have) {
            unsigned pairs, near;
            live_marks(L, cap, walls, pc, x, i, nn, j0, j1, wall0, wfar && far ? wall0 : wall1, pairs, near);
            full = cs != 0 || pairs != 0u || near != 0u;
            if (!full) {
                if (last) {
                    v2 = free_step(P, fc, i, 1, m, u, x);
                } else {
                    for (int d = 0; d < 3; ++d) u[d] = dadd(dadd(u[d], a[d]), a[d]);
                    x.x = dadd(x.x, dmul(fc.dt, u[0]));
                    x.y = dadd(x.y, dmul(fc.dt, u[1]));
                    x.z = dadd(x.z, dmul(fc.dt, u[2]));
                    v2 = dadd(dadd(dmul(u[0], u[0]), dmul(u[1], u[1])), dmul(u[2], u[2]));
                }
                st4(P.pos[cur ^ 1], i, x);
                for (int d = 0; d < 3; ++d) v1[d * cap + i] = u[d];
                if (spin) {   // the spin a contact wrote last step, in both buffers again
                    for (int d = 0; d < 3; ++d) w1[d * cap + i] = w0[d * cap + i];
                    spin = false;
                }
            } else {
                live_contact<MIXED>(P, L, fc, pp, pw, walls, pc, P.pos[cur ^ 1], v0, w0, v1, w1, last, i, j0, j1, nn,
                                    pairs, near, wall0, m, x, u, cs, v2, status);
                spin = true;
            }
        }
        const unsigned busy = __ballot_sync(0xffffffffu, full);
        if (status) atomicOr(&ctl->status, status);
        unsigned long long big;
        ok = grid_step<kBlock>(bar, ctl, fc, scratch, k, v2, __popc(busy), big, ncon);
        if (!ok) break;
        double v = sqrt(__longlong_as_double((long long)big));
        if (quiet) v = fmax(v, vq + (k + 1) * fc.dt * ga * (1.0 + 1e-9));
        disp = disp + fc.dt * v * (1.0 + 1e-9);
        cur ^= 1;
        double *tv = v0, *tw = w0;
        v0 = v1;
        w0 = w1;
        v1 = tv;
        w1 = tw;
        done += 1;
        steps += 1;
    }
    if (quiet && (steps & 1) && have)   // the velocities back into their arrays
        for (int d = 0; d < 3; ++d) {
            v1[d * cap + i] = v0[d * cap + i];
            w1[d * cap + i] = w0[d * cap + i];
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) {   // the control word as the per-step finaliser leaves it
        ctl->cur = cur;
        if (!quiet) ctl->vcur = vcur0 ^ (steps & 1);
        ctl->steps_done = done;
        ctl->total_steps += steps;
        ctl->disp = disp;
        if (steps > 0) ctl->last_ndefer = ncon;
        ctl->ndefer = 0;
        ctl->npairs = 0;
        ctl->flight_cur = cur0;      // what k_flight continues from
        ctl->flight_steps = steps;
        ctl->flight_last = done >= target;
    }
}

// The same loop for up to kLiveMany particles per thread, their state in memory: a thread first takes
// the free step of those nothing marks, then the warp's threads each take their marked ones, one after
// another (live_contact), so that particles in contact in different rounds share one pass.  Ends
// early once more than `dense` particles of a step were in contact.
//
// Bounded by the list and position gathers of a thread's rounds and by the barrier.  Measured (B200,
// device us per step, the three-kernel step in graph replays / this one): 151 scenes of 1,166 spheres
// in their boxes (176,000, FP32 forces) 25 / 14.4; four entries' gathers in flight at a time instead of
// one after another 16.6 -> 14.4.
template <bool MIXED>
__global__ void __launch_bounds__(kBlock, 3) k_steps_live_many(Particles P, NbrList L, Ctl *ctl, ForceConsts fc,
                                                               const PairConst *__restrict__ pp,
                                                               const PairConst *__restrict__ pw,
                                                               const WallGeom *__restrict__ walls, int max_steps,
                                                               unsigned long long *scratch, int quiet, int dense) {
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ GridStep<kBlock> bar;
    const int n = P.n, cap = P.cap, T = gridDim.x * kBlock;
    const int cur0 = ctl->cur, vcur0 = ctl->vcur, target = ctl->target;
    const int first = quiet ? ctl->nlone + ctl->nclear : 0;
    const bool stopped = (ctl->status & kStopBits) != 0;
    const double half = ctl->half_skin, until = quiet ? fmin(half, ctl->clear_until) : half;
    const bool wfar_ok = ctl->wfar_build == ctl->rebuilds;
    const double vq = quiet ? sqrt(__longlong_as_double((long long)ctl->vq2)) : 0.0;
    const double ga = sqrt(fc.g[0] * fc.g[0] + fc.g[1] * fc.g[1] + fc.g[2] * fc.g[2]);
    double disp = ctl->disp;
    int done = ctl->steps_done, cur = cur0, steps = 0, ncon = 0;
    double *v0 = P.vel[vcur0], *w0 = P.omg[vcur0];   // velocities of the step, and of the next
    double *v1 = quiet ? L.defer_v : P.vel[vcur0 ^ 1], *w1 = quiet ? L.defer_w : P.omg[vcur0 ^ 1];
    const int i0 = first + blockIdx.x * kBlock + threadIdx.x;
    unsigned spin = 0u;   // bit r: the particle of round r was in contact in the last step
    for (int i = i0; i < n; i += T)
        for (int d = 0; d < 3; ++d) w1[d * cap + i] = w0[d * cap + i];
    bool ok = true;
    for (int k = 0; k < max_steps; ++k) {
        // the same in every block
        if (!(done < target && !stopped && disp < until && ok && ncon <= dense)) break;
        const int last = done + 1 >= target;
        const bool wfar = wfar_ok && 2.0 * disp < half;
        const double4 *pc = P.pos[cur];
        double vmax = 0.0;
        int status = 0;
        unsigned pend = 0u;
        // particle i's state and marks
        auto read = [&](const int i, D4 &x, double &m, double (&u)[3], int &cs, int &nn, int &j0, int &j1, int &wall0,
                        unsigned &pairs, unsigned &near) {
            x = ld4(pc, i);
            cs = P.cstate[i];
            nn = L.nn[i];
            const bool far = wfar && L.wfar[i];
            j0 = L.maxnb > 0 ? L.idx[i] : 0;   // used below the list length only
            j1 = L.maxnb > 1 ? L.idx[cap + i] : 0;
            m = P.mI[i];
            for (int d = 0; d < 3; ++d) u[d] = v0[d * cap + i];
            const int scene_i = P.scene ? P.scene[i] : 0;
            wall0 = fc.wps ? scene_i * fc.wps : 0;
            const int wall1 = far ? wall0 : fc.wps ? wall0 + fc.wps : fc.nwall;
            live_marks(L, cap, walls, pc, x, i, nn, j0, j1, wall0, wall1, pairs, near);
        };
        int r = 0;
        for (int i = i0; i < n; i += T, ++r) {
            D4 x;
            double m, u[3];
            int cs, nn, j0, j1, wall0;
            unsigned pairs, near;
            read(i, x, m, u, cs, nn, j0, j1, wall0, pairs, near);
            if (cs != 0 || pairs != 0u || near != 0u) {
                pend |= 1u << r;
                continue;
            }
            vmax = fmax(vmax, free_step(P, fc, i, last, m, u, x));
            st4(P.pos[cur ^ 1], i, x);
            for (int d = 0; d < 3; ++d) v1[d * cap + i] = u[d];
            if ((spin >> r) & 1u) {   // the spin a contact wrote last step, in both buffers again
                for (int d = 0; d < 3; ++d) w1[d * cap + i] = w0[d * cap + i];
                spin &= ~(1u << r);
            }
        }
        const int busy = (int)__reduce_add_sync(FULL, (unsigned)__popc(pend));
        spin |= pend;
        while (__any_sync(FULL, pend != 0u)) {
            if (pend) {
                const int i = i0 + (__ffs(pend) - 1) * T;
                pend &= pend - 1u;
                D4 x;
                double m, u[3], v2 = 0.0;
                int cs, nn, j0, j1, wall0;
                unsigned pairs, near;
                read(i, x, m, u, cs, nn, j0, j1, wall0, pairs, near);
                live_contact<MIXED>(P, L, fc, pp, pw, walls, pc, P.pos[cur ^ 1], v0, w0, v1, w1, last, i, j0, j1, nn,
                                    pairs, near, wall0, m, x, u, cs, v2, status);
                vmax = fmax(vmax, v2);
            }
        }
        if (status) atomicOr(&ctl->status, status);
        unsigned long long big;
        ok = grid_step<kBlock>(bar, ctl, fc, scratch, k, vmax, busy, big, ncon);
        if (!ok) break;
        double v = sqrt(__longlong_as_double((long long)big));
        if (quiet) v = fmax(v, vq + (k + 1) * fc.dt * ga * (1.0 + 1e-9));
        disp = disp + fc.dt * v * (1.0 + 1e-9);
        cur ^= 1;
        double *tv = v0, *tw = w0;
        v0 = v1;
        w0 = w1;
        v1 = tv;
        w1 = tw;
        done += 1;
        steps += 1;
    }
    if (quiet && (steps & 1))   // the velocities back into their arrays
        for (int i = i0; i < n; i += T)
            for (int d = 0; d < 3; ++d) {
                v1[d * cap + i] = v0[d * cap + i];
                w1[d * cap + i] = w0[d * cap + i];
            }
    if (blockIdx.x == 0 && threadIdx.x == 0) {   // as k_steps_live leaves it
        ctl->cur = cur;
        if (!quiet) ctl->vcur = vcur0 ^ (steps & 1);
        ctl->steps_done = done;
        ctl->total_steps += steps;
        ctl->disp = disp;
        if (steps > 0) ctl->last_ndefer = ncon;
        ctl->ndefer = 0;
        ctl->npairs = 0;
        ctl->flight_cur = cur0;
        ctl->flight_steps = steps;
        ctl->flight_last = done >= target;
    }
}

// Blocks resident at once.
template <bool MIXED>
static int live_blocks(bool many) {
    static thread_local PerDevice fit[2];
    return resident_blocks(fit[many], many ? (const void *)k_steps_live_many<MIXED> : (const void *)k_steps_live<MIXED>, kBlock);
}

template <bool MIXED>
static int live_threads() { return live_blocks<MIXED>(false) * kBlock; }

template <bool MIXED>
static cudaError_t steps_live_t(const Particles &P, const NbrList &L, Ctl *ctl, const ForceConsts &fc,
                                const PairConst *pp, const PairConst *pw, const WallGeom *walls, int count, int max_steps,
                                unsigned long long *scratch, int quiet, int dense, cudaStream_t s) {
    const int need = count > 0 ? (count + kBlock - 1) / kBlock : 1;
    const bool many = need > live_blocks<MIXED>(false);
    // every thread the same number of rounds: the fewest rounds, then no more blocks than those need
    const int most = live_blocks<MIXED>(true), rounds = (need + most - 1) / most;
    const int grid = many ? (need + rounds - 1) / rounds : need;
    if (many && rounds > kLiveMany) return cudaErrorInvalidValue;
    const cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(unsigned long long) * 6, s);
    if (e != cudaSuccess) return e;
    Particles p = P;
    NbrList l = L;
    ForceConsts f = fc;
    void *args[] = {&p, &l, &ctl, &f, (void *)&pp, (void *)&pw, (void *)&walls, &max_steps, &scratch, &quiet, &dense};
    return cudaLaunchCooperativeKernel(many ? (const void *)k_steps_live_many<MIXED> : (const void *)k_steps_live<MIXED>,
                                       dim3(grid), dim3(kBlock), args, 0, s);   // k_steps_live takes no `dense`
}

}  // namespace
}  // namespace b200dem
