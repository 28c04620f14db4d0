// dem_refloop.cuh -- the rebuild-every-step mode's loop (the reference's: a new neighbour search
// before every force pass, src/CabanaDEM_Solver.hpp:79-97) in one cooperative launch.
//
// As a graph, such a step is 13 build kernels and the step kernel: 36 us for 2 spheres, 109 us for
// 3,000, nearly all of it launches and dependent round trips of nearly empty grids.  Here a step is
// one search-and-force pass of a resident grid and one grid barrier.  A group of NL lanes (32, 16
// or 8) takes a particle: its lanes read the 27 cells around it and test their particles, the
// candidates that can overlap go to the group's list in shared memory in ascending caller index
// (the order of every sum), and particle_coop does the step with that list.  The group then enters
// the new position into the next step's cell table, so the barrier at the end of a step separates
// the table's writers from its readers.  Three tables rotate: step k reads table k mod 3, enters
// into table (k + 1) mod 3 and clears its own entry of step k - 1 in table (k + 2) mod 3.
//
// Cells have a fixed capacity (kRefCell), so entering a particle is one atomic and no scan is
// needed.  The grid is taken from the positions at the launch; a particle that leaves it counts to
// the cell at the border (a clamped coordinate never separates two cells that touch, so no pair is
// missed).  A full cell, a list over the solver's capacity or a position that is not finite ends
// the launch at the step boundary.  The host then makes the lists larger where that is what it takes, and
// launches again on a fresh grid; a launch that can take no step hands the rest of the run to the graph
// of build and step kernels, which reports the error if there is one.  The run's last step writes the lists (all
// candidates within the cutoff) where the build kernels leave them.
//
// Measured (B200, FP64, us per step over 1,000 steps, graph / this loop): 2 spheres 37 / 4.2, a dense
// cloud of 200 94 / 8.5, of 3,000 113 / 11.0, of 12,000 115 / 22.9, of 65,000 134 / 78; a gas of 65,000
// 69 / 50: faster at every size the mode's one-kernel step takes.  What bounds it: the grid barrier
// (1.2 us: two L2 round trips and a fence) and, below some 10,000 particles, the instructions of the
// slowest warp (a search and a contact, about 1,800 instructions at 6-8 cycles each); above, those of
// all warps.
#pragma once
#include "dem_cells.cuh"
#include "dem_contact_coop.cuh"
#include "dem_persist.cuh"

namespace b200dem {
namespace {

// Lanes per particle and the block's shape: a warp each (8 warps per SM, no register cap), then 16 lanes
// (12 warps per SM), while every particle's lanes are resident at once, else 8 lanes.
// A warp each at 3,000 and 12,000 spheres took 15.2 and 37 us against 12.8 and 22.7 with 8 lanes; 8 lanes at 2
// and 200 spheres 11.9 and 12.9 against 7.9 and 8.4.  16 lanes, two cells each, against 8: 1,185 spheres 10.0,
// 12.2; 3,000 11.0, 13.0; 3,552 11.3, 13.2.
constexpr int kRefWideMax = 148 * 8;        // a warp each: 8 warps per SM
constexpr int kRefMidMax = 148 * 12 * 2;    // 16 lanes each: 12 warps per SM
template <int NL>
struct RefShape {
    static constexpr int block = NL == 32 ? 256 : 128, min_blocks = NL == 32 ? 1 : 3;
};
constexpr int kRefMaxList = 128;   // candidates a group can hold (the build's kMaxCand)

// Linear cell index: no storage order hangs on it, and it takes a fraction of the Morton key's
// instructions.  Never more cells than the grid's keys (k_grid takes Morton keys only when those,
// which are no fewer, fit).
__device__ __forceinline__ int ref_key(const Grid &g, int x, int y, int z) { return (z * g.dims[1] + y) * g.dims[0] + x; }

// Enters particle i at position p into table `tab` (counts zeroed before; table 0 by k_ref_enter).
__device__ __forceinline__ void ref_enter(const RefTables &R, const Grid &G, int tab, int n_codes, int i, const D4 &p,
                                          int *key_of, bool &stop) {
    int c[3];
    cell_of(G, p, c);
    const int key = ref_key(G, c[0], c[1], c[2]);
    const int slot = atomicAdd(R.count + (long)tab * n_codes + key, 1);
    if (slot < kRefCell) R.item[((long)tab * n_codes + key) * kRefCell + slot] = i;
    key_of[i] = key;
    const double big = 1e300;   // also false for a NaN
    if (slot >= kRefCell || !(fabs(p.x) < big && fabs(p.y) < big && fabs(p.z) < big)) stop = true;
}

__global__ void k_ref_enter(Particles P, const Ctl *ctl, RefTables R, unsigned long long *arrive) {
    const Grid G = *R.grid;
    const int codes = *R.total;
    bool stop = (ctl->status & (DEM_ERR_NAN | kStopBits)) != 0;
    if (codes > R.codes) stop = true;   // the tables hold R.codes cells
    else
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P.n; i += gridDim.x * blockDim.x)
            ref_enter(R, G, 0, R.codes, i, ld4(P.pos[ctl->cur], i), R.key, stop);
    if (stop) atomicOr(arrive, 1ull << 62);   // seen at barrier 0
}

// Barrier number `b` of the launch: every block's writes before, every block's reads after.
// Returns false when some block asked to stop before it, or when the wait gave up.  The low half
// of the arrival word counts arrivals; bit 62 + (b & 1) is the stop request of barrier b (a block
// may already be one barrier ahead of one that still polls, so the two need bits of their own).
// fc: as for grid_step.
__device__ __forceinline__ bool ref_barrier(Ctl *ctl, const ForceConsts &fc, unsigned long long *arrive, unsigned b, bool stop) {
    __shared__ int s_go;
    const int any = __syncthreads_or(stop ? 1 : 0);
    if (gridDim.x == 1) return !any;   // one block: its own barrier is the grid's
    if (threadIdx.x == 0) {
        const unsigned want = gridDim.x * (b + 1);
        const int bit = 62 + (int)(b & 1);
        unsigned long long v;
        if (any) atomicOr(arrive, 1ull << bit);
        asm volatile("atom.release.gpu.global.add.u64 %0, [%1], %2;"
                     : "=l"(v) : "l"(arrive), "l"(fc.drop_copies ? 0ull : 1ull) : "memory");
        const int limit = fc.wait_polls > 0 ? fc.wait_polls : kCoopWaitPolls;
        int k = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(arrive) : "memory");
        } while ((unsigned)v < want && ++k < limit);
        int go = ((v >> bit) & 1) == 0;
        if (k == limit) {
            atomicOr(&ctl->status, DEM_ERR_TIMEOUT);
            go = 0;
        }
        s_go = go;
    }
    __syncthreads();
    return s_go != 0;
}

struct RefGroup {   // a group's share of the block's shared memory
    double h[3 * kCoopSlots + 1];
    int tidx[kCoopSlots + 1];
    int n, all;                                 // candidates kept; candidates within the cutoff
    int j[kRefMaxList], key[kRefMaxList], list[kRefMaxList];
};

template <int NL, bool MIXED>
__global__ void __launch_bounds__(RefShape<NL>::block, RefShape<NL>::min_blocks) k_steps_ref(Particles P, NbrList L, Ctl *ctl, ForceConsts fc,
                                                            const PairConst *__restrict__ pp,
                                                            const PairConst *__restrict__ pw,
                                                            const WallGeom *__restrict__ walls, RefTables R,
                                                            double delta, double skin, int max_steps,
                                                            unsigned long long *arrive) {
    constexpr int GPB = RefShape<NL>::block / NL;        // groups of a block
    constexpr int CPL = (27 + NL - 1) / NL;        // cells per lane
    extern __shared__ __align__(128) unsigned char sm[];
    RefGroup &S = reinterpret_cast<RefGroup *>(sm)[threadIdx.x / NL];
    const Grid G = *R.grid;
    const int gl = threadIdx.x % NL, grp = threadIdx.x / NL;
    const int ngroups = gridDim.x * GPB, wgroups = 32 / NL;
    const int g0 = blockIdx.x * GPB + grp;
    const int n = P.n, cap = P.cap;
    int cur = ctl->cur, vcur = ctl->vcur, done = ctl->steps_done;
    const int target = ctl->target;
    unsigned bar = 0;
    bool go = !(ctl->status & (kStopBits | DEM_ERR_NAN)) && !((*arrive >> 62) & 1);
    go = ref_barrier(ctl, fc, arrive, bar++, !go);
    int steps = 0, status = 0;
    // at most 2^31 - 1 arrivals per launch (the host goes on with another)
    const int kmax = min(max_steps, (int)(0x7fffffffu / gridDim.x) - 2);
    for (int k = 0; k < kmax && go && done < target; ++k) {
        const int last = done + 1 >= target;
        const int tr = k % 3, tw = (k + 1) % 3, tz = (k + 2) % 3;
        const int *cnt_r = R.count + (long)tr * R.codes;
        const int *item_r = R.item + (long)tr * R.codes * kRefCell;
        const double4 *pc = P.pos[cur];
        bool stop = false;
        for (int base = 0; base < n; base += ngroups) {
            if (base + g0 - (g0 % wgroups) >= n) break;   // no particle left for this warp
            const int i = base + g0 < n ? base + g0 : -1;
            if (gl == 0) S.n = S.all = 0;
            __syncwarp();
            bool busy = false;   // tracked contacts, a wall within reach (or candidates, below)
            CoopOwn o = {{0., 0., 0., 0.}, {0., 0., 0.}, {0., 0., 0.}, 1., 1., 0};
            D4 &pi = o.p;
            if (i >= 0) {
                pi = ld4(pc, i);
                o.cs = P.cstate[i];
                o.m = P.mI[i];
                o.I = P.mI[(long)cap + i];
                for (int d = 0; d < 3; ++d) {
                    o.u[d] = P.vel[vcur][d * cap + i];
                    o.w[d] = P.omg[vcur][d * cap + i];
                }
                busy = o.cs != 0;
                for (int q = gl; q < fc.nwall; q += NL) {   // a margin above the law's own test
                    const WallGeom &g = walls[q];
                    const double at = (pi.x - g.x[0]) * g.n[0] + (pi.y - g.x[1]) * g.n[1] + (pi.z - g.x[2]) * g.n[2];
                    busy = busy || !(at > pi.w * 1.000001);
                }
                int c[3];
                cell_of(G, pi, c);
                int m[CPL];
                const int4 *it[CPL];
                int4 a[CPL];
#pragma unroll
                for (int r = 0; r < CPL; ++r) {   // the cells' counts and first entries in one round trip
                    const int cc = gl + r * NL;
                    const int x = c[0] + cc % 3 - 1, y = c[1] + (cc / 3) % 3 - 1, z = c[2] + cc / 9 - 1;
                    const bool in = cc < 27 && (unsigned)x < (unsigned)G.dims[0] && (unsigned)y < (unsigned)G.dims[1] &&
                                    (unsigned)z < (unsigned)G.dims[2];
                    const int key = in ? ref_key(G, x, y, z) : 0;
                    m[r] = in ? min(cnt_r[key], kRefCell) : 0;
                    it[r] = reinterpret_cast<const int4 *>(item_r) + (long)key * (kRefCell / 4);
                    a[r] = it[r][0];
                }
                int within = 0;
                auto test = [&](const int j, const D4 &pj) {
                    // the build's expression, never contracted: the same candidates in both precisions
                    const double px = dadd(pi.x, -pj.x), py = dadd(pi.y, -pj.y), pz = dadd(pi.z, -pj.z);
                    const double r2 = dadd(dadd(dmul(px, px), dmul(py, py)), dmul(pz, pz));
                    const double sr = dadd(pi.w, pj.w);
                    const double cut = delta > 0.0 ? delta : dadd(sr, skin);
                    if (!(r2 <= dmul(cut, cut)) || j == i) return;
                    ++within;
                    // the last step keeps every listed candidate, the others those that can overlap
                    if (last || r2 < sr * sr * 1.000001) {
                        const int s = atomicAdd(&S.n, 1);
                        if (s < kRefMaxList) {
                            S.j[s] = j;
                            S.key[s] = P.perm[j];
                        }
                    }
                };
#pragma unroll
                for (int r = 0; r < CPL; ++r) {
                    int4 e = a[r];
#pragma unroll 1
                    for (int s = 0; s < m[r]; s += 4) {   // four positions in flight
                        const int left = m[r] - s;
                        if (s) e = it[r][s / 4];
                        const int j1 = left > 1 ? e.y : e.x, j2 = left > 2 ? e.z : e.x, j3 = left > 3 ? e.w : e.x;
                        const D4 q0 = ld4(pc, e.x), q1 = ld4(pc, j1), q2 = ld4(pc, j2), q3 = ld4(pc, j3);
                        test(e.x, q0);
                        if (left > 1) test(j1, q1);
                        if (left > 2) test(j2, q2);
                        if (left > 3) test(j3, q3);
                    }
                }
                if (within) atomicAdd(&S.all, within);
            }
            __syncwarp();
            const int nc = min(S.n, kRefMaxList), all = S.all;
            if (i >= 0 && all > min(L.maxnb, kRefMaxList)) {   // the host grows the lists, or reports more than 128
                status |= DEM_ERR_NEIGHBOR_OVERFLOW;
                stop = true;
            }
            // ascending caller index: the rank of each candidate
            for (int a = gl; a < nc; a += NL) {
                const int ka = S.key[a];
                int r = 0;
                for (int b = 0; b < nc; ++b) r += S.key[b] < ka ? 1 : 0;
                S.list[r] = S.j[a];
            }
            __syncwarp();
            if (i >= 0 && (last || stop)) {
                const int keep = min(nc, L.maxnb);
                for (int a = gl; last && a < keep; a += NL) L.idx[(long)a * cap + i] = S.list[a];
                if (gl == 0) {
                    if (last) L.nn[i] = keep;
                    atomicMax(&ctl->max_nbr, all);
                }
            }
            D4 pn = pi;
            if (__any_sync(0xffffffffu, busy || nc > 0)) {
                double v2 = 0.0;
                particle_coop<NL, MIXED, false>(P, GroupList{S.list, i >= 0 ? nc : 0}, fc, pp, pw, walls, cur, cur ^ 1,
                                                vcur, last, i, i, S.tidx, S.h, P.vel[vcur ^ 1], P.omg[vcur ^ 1], v2,
                                                status, &pn, &o);
            } else if (i >= 0 && gl == 0) {
                // nothing touches this particle: the step of particle_coop without contacts
                free_step(P, fc, i, last, o.m, o.u, pn);
                st4(P.pos[cur ^ 1], i, pn);
                for (int d = 0; d < 3; ++d) {
                    P.vel[vcur ^ 1][d * cap + i] = o.u[d];
                    P.omg[vcur ^ 1][d * cap + i] = o.w[d];
                }
            }
            if (i >= 0 && gl == 0) {
                if (k > 0) R.count[(long)tz * R.codes + R.key[(long)tz * cap + i]] = 0;
                if (!last) ref_enter(R, G, tw, R.codes, i, pn, R.key + (long)tw * cap, stop);
            }
            __syncwarp();
        }
        go = ref_barrier(ctl, fc, arrive, bar++, stop);
        cur ^= 1;
        vcur ^= 1;
        done += 1;
        steps += 1;
    }
    if (status) atomicOr(&ctl->status, status);
    if (blockIdx.x == 0 && threadIdx.x == 0) {   // the control word as the build and step kernels leave it
        ctl->cur = cur;
        ctl->vcur = vcur;
        ctl->steps_done = done;
        ctl->total_steps += steps;
        ctl->rebuilds += steps;
        ctl->disp = 0.0;
        ctl->ndefer = 0;
        ctl->npairs = 0;
        ctl->nlone = 0;
        ctl->nclear = 0;
    }
}

}  // namespace

template <int NL, bool MIXED>
static cudaError_t steps_ref_t(const Particles &P, const NbrList &L, Ctl *ctl, const ForceConsts &fc,
                               const PairConst *pp, const PairConst *pw, const WallGeom *walls, const RefTables &R,
                               double delta, double skin, int max_steps, unsigned long long *arrive, cudaStream_t s) {
    const void *kernel = (const void *)k_steps_ref<NL, MIXED>;
    static thread_local PerDevice kept;
    const int smem = (RefShape<NL>::block / NL) * (int)sizeof(RefGroup);
    const int fit = resident_blocks(kept, kernel, RefShape<NL>::block, smem);
    const int need = (P.n + RefShape<NL>::block / NL - 1) / (RefShape<NL>::block / NL);
    const int grid = need < fit ? need : fit;
    cudaError_t e = cudaMemsetAsync(arrive, 0, sizeof(unsigned long long), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(R.count, 0, sizeof(int) * 3 * (size_t)R.codes, s);
    if (e != cudaSuccess) return e;
    const int ge = (P.n + 255) / 256;
    k_ref_enter<<<ge < 148 * 4 ? ge : 148 * 4, 256, 0, s>>>(P, ctl, R, arrive);
    Particles p = P;
    NbrList l = L;
    ForceConsts f = fc;
    RefTables r = R;
    void *args[] = {&p, &l, &ctl, &f, (void *)&pp, (void *)&pw, (void *)&walls, &r, &delta, &skin, &max_steps, &arrive};
    return cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(RefShape<NL>::block), args, smem, s);
}

}  // namespace b200dem
