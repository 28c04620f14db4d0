// dem_nn.cu -- dense layers of the learned surrogate on the 5th-generation tensor cores.
//
// Every dense block of the message-passing network is a two-layer perceptron over rows
// (edges or particles):  y = W2 relu(W1 x + b1) + b2 (+ residual), hidden width 128,
// BF16 operands, FP32 accumulation in TMEM.  Three kernels cover training and inference:
//
//   k_mlp_fwd    gather the input row tile (up to three sources, e.g. [e_ij, h_i, h_j]),
//                GEMM1 -> bias + ReLU -> GEMM2 -> bias (+ residual); the hidden tile never
//                leaves shared memory/TMEM (saved to HBM only when training).
//   k_mlp_bwd    dH = dY W2^T, dZ = dH * [h > 0], dX = dZ W1^T (input gradient, split into
//                128-wide N chunks).
//   k_mlp_wgrad  dW1^T = dZ^T X, dW2^T = dY^T H (or dW2 = H^T dY for a 16-wide output) and
//                the bias sums, accumulated in TMEM over each CTA's row tiles; per-CTA
//                partials are then summed in a fixed order (k_wgrad_reduce), so the
//                gradients are deterministic.
//
// Persistent CTAs over row tiles, one per SM for the wide shapes: threads t, t + 128, ... share tile row
// t, which is TMEM lane t of the M = 128 accumulators.  One elected thread issues tcgen05.mma and
// commits to an mbarrier; every wait is bounded and a timeout raises the context's error
// word instead of hanging.
#include <cuda.h>   // CUtensorMap (encoded on the host through the driver entry point)
#include <cuda_bf16.h>
#include <cstdint>

#include "b200dem.h"
#include "dem_internal.cuh"
#include "nn_tc.cuh"

namespace b200dem {
namespace {

using bf16 = __nv_bfloat16;
constexpr int kRows = 128;      // rows per tile (= MMA M)
constexpr int kHidden = 128;    // hidden width
constexpr int kFwdThreads = 256;   // k_edge_fwd: warps w and w + 4 split a TMEM lane quarter's columns
constexpr int kLinThreads = 512;   // the other kernels: warps w, w + 4, w + 8 and w + 12 do
constexpr int kBwdThreads = 512;

struct RowSrc {
    const bf16 *p;
    const int *idx;
    int width;   // features taken from this source (multiple of 8)
};

struct MlpW {
    const bf16 *w1t, *w1, *w2t, *w2;
    const float *b1, *b2;
};

// ---- asynchronous staging (cp.async: every chunk copy of a tile in flight at once) ----
__device__ __forceinline__ void cp16(void *smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_u32(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Element q of a tile of R rows (a multiple of 8) and C chunks: eight consecutive threads take eight
// consecutive rows of one chunk (conflict-free 128-byte runs in shared memory), the warp four chunks of
// them, so that its access covers whole 32-byte sectors of global memory.
__device__ __forceinline__ void tile_element(int q, int R, int C, int &row, int &kc) {
    const int G = C < 4 ? C : 4, rest = (q >> 3) / G;
    row = (rest % (R / 8)) * 8 + (q & 7);
    kc = (rest / (R / 8)) * G + (q >> 3) % G;
}

// Feature f of the concatenated sources: the source's number, and f within it.  (The sources are
// picked by comparisons: an index into the kernel's argument array would put a copy of it in local memory.)
__device__ __forceinline__ RowSrc pick_source(const RowSrc *src, int nsrc, int &f, int &s) {
    RowSrc r = src[0];
    s = 0;
    if (nsrc > 1 && f >= r.width) {
        f -= r.width;
        r = src[1];
        s = 1;
        if (nsrc > 2 && f >= r.width) {
            f -= r.width;
            r = src[2];
            s = 2;
        }
    }
    return r;
}

// Queue the copies of a dense row-major block [R rows][F features] (row stride F) into a row
// tile of R rows; rows past `rows` are zero-filled.
__device__ __forceinline__ void stage_dense(unsigned char *tile, const bf16 *g, int R, int F, long row0, long rows) {
    const int C = F / 8;
    for (int q = threadIdx.x; q < R * C; q += blockDim.x) {
        int row, kc;
        tile_element(q, R, C, row, kc);
        unsigned char *dst = tile + tc::tile_off(R, row, kc);
        if (row0 + row < rows) cp16(dst, g + (row0 + row) * F + kc * 8);
        else *reinterpret_cast<uint4 *>(dst) = make_uint4(0, 0, 0, 0);
    }
}

// The same into the swizzled layout (F a multiple of 64): a warp takes whole rows, four lines of global
// memory, where the layout above makes it touch eight rows: there the copies of a 32 KB tile occupied an
// SM's load path for some 2,000 cycles, most of the gradient kernels' time.
__device__ __forceinline__ void stage_sw(unsigned char *tile, const bf16 *g, int R, int F, long row0, long rows) {
    const int C = F / 8;
    for (int q = threadIdx.x; q < R * C; q += blockDim.x) {
        const int row = q / C, c = q % C;
        unsigned char *dst = tile + tc::sw_off(R, row, c);
        if (row0 + row < rows) cp16(dst, g + (row0 + row) * F + c * 8);
        else *reinterpret_cast<uint4 *>(dst) = make_uint4(0, 0, 0, 0);
    }
}
__device__ __forceinline__ unsigned char *align1024(unsigned char *p) {
    return p + ((1024u - (tc::smem_u32(p) & 1023u)) & 1023u);
}

// Completes this thread's queued copies and publishes the tiles to the tensor core.
__device__ __forceinline__ void stage_done() {
    cp_wait_all();
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
}

// Row-major output tile in shared memory (128 rows x 256 bytes), 16-byte chunks XOR-swizzled
// by the row so that thread t writing its row and 16 threads reading one row are both free of
// bank conflicts; copy_out then writes whole 256-byte rows (coalesced).
__device__ __forceinline__ void out_put(unsigned char *tile, int row, int chunk, uint4 v) {
    *reinterpret_cast<uint4 *>(tile + row * 256 + ((chunk ^ (row & 15)) << 4)) = v;
}
__device__ __forceinline__ void copy_out(const unsigned char *tile, bf16 *g, long row0, long rows) {
    for (int q = threadIdx.x; q < kRows * 16; q += blockDim.x) {
        const int row = q >> 4, chunk = q & 15;
        if (row0 + row < rows)
            *reinterpret_cast<uint4 *>(g + (row0 + row) * kHidden + chunk * 8) =
                *reinterpret_cast<const uint4 *>(tile + row * 256 + ((chunk ^ (row & 15)) << 4));
    }
}

// Eight floats of shared memory in two loads (p on a 16-byte boundary).
__device__ __forceinline__ void load8(const float *p, float v[8]) {
    const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}

// Thread t reads 16 accumulator columns [col, col + 16) of its TMEM lane.
__device__ __forceinline__ void acc16(uint32_t tm, int col, float v[16]) {
    tc::tmem_ld16(tc::tmem_warp_addr(tm, col), v);
    tc::tmem_wait_ld();
}

// 32 accumulator columns [col, col + 32) of thread t's lane.
__device__ __forceinline__ void acc32(uint32_t tm, int col, float v[32]) {
    uint32_t r[32];
    tc::tmem_ld32_nowait(tc::tmem_warp_addr(tm, col), r);
    tc::tmem_wait_ld();
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = __uint_as_float(r[k]);
}

// 64 accumulator columns [col, col + 64) of thread t's lane with one wait (two x32 loads).
__device__ __forceinline__ void acc64(uint32_t tm, int col, float v[64]) {
    uint32_t r[64];
    tc::tmem_ld32_nowait(tc::tmem_warp_addr(tm, col), r);
    tc::tmem_ld32_nowait(tc::tmem_warp_addr(tm, col + 32), r + 32);
    tc::tmem_wait_ld();
#pragma unroll
    for (int k = 0; k < 64; ++k) v[k] = __uint_as_float(r[k]);
}

// Shared-memory prologue of every kernel: mbarrier, TMEM allocation (warp 0).
__device__ __forceinline__ uint32_t tc_setup(uint64_t *mbar, uint32_t *tslot, int ncols) {
    if (threadIdx.x == 0) tc::mbar_init(mbar, 1);
    if (threadIdx.x < 32) {
        tc::tmem_alloc(tslot, ncols);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    return *tslot;
}

// Bounded waits of the tensor-core kernels: polls of mbarrier.try_wait per wait, and a
// diagnostic switch under which the kernels issue no MMA and no commit (so every wait runs
// out with nothing in flight).  Process-wide per device; set by dem_nn_debug_waits.
__device__ int g_tc_wait_limit = 1 << 22;
__device__ int g_tc_drop_mma = 0;

// The elected thread's MMA issue and commit, skipped under the diagnostic switch.
__device__ __forceinline__ void mma_issue(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    if (!g_tc_drop_mma) tc::mma_bf16(tmem_d, adesc, bdesc, idesc, accumulate);
}
__device__ __forceinline__ void mma_issue_tmem_a(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                                 uint32_t accumulate) {
    if (!g_tc_drop_mma) tc::mma_bf16_tmem_a(tmem_d, tmem_a, bdesc, idesc, accumulate);
}
__device__ __forceinline__ void mma_commit_issue(uint64_t *mbar) {
    if (!g_tc_drop_mma) tc::mma_commit(mbar);
}

// End of every kernel: free the block's TMEM.  When a wait gave up (ok false), the MMA batch
// of that wait may still be running and writing TMEM: the block first waits once more, with
// the same bound, for that batch's commit (parity `phase ^ 1`: mma_wait flipped it), so TMEM
// is freed after the batch completes.  If that wait gives up too, TMEM is freed anyway and the
// error word carries DEM_ERR_TIMEOUT; the host learns of it from dem_nn_status.
__device__ __forceinline__ void tc_teardown(uint32_t tm, int ncols, bool ok, int *err, uint64_t *mbar,
                                            uint32_t phase) {
    if (!ok) {
        if (threadIdx.x == 0) (void)tc::mbar_wait(mbar, phase ^ 1u, g_tc_wait_limit);
        __syncthreads();
    }
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tm, ncols);
    }
    if (!ok && threadIdx.x == 0 && err) atomicOr(err, DEM_ERR_TIMEOUT);
}

// All threads wait for the MMA batch committed last; uniform result across the block.
__device__ __forceinline__ bool mma_wait(uint64_t *mbar, uint32_t &phase) {
    const bool ok = tc::mbar_wait(mbar, phase, g_tc_wait_limit);
    phase ^= 1u;
    const bool all = __syncthreads_and(ok) != 0;
    tc::fence_after_sync();
    return all;
}

// ------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------
struct FwdArgs {
    long rows;
    RowSrc src[3];
    int nsrc;
    MlpW w;
    const bf16 *resid;   // [rows][NOUT] or null
    int resid_src0;      // the residual is source 0 of the input (read from the staged tile)
    bf16 *out;           // [rows][NOUT] or null
    float *out_f32;      // [rows][NOUT] or null
    bf16 *h1;            // [rows][128] or null
    int *err;
};

// Input tiles in flight (384 features leave room for one) and threads: an SM's shared memory holds one CTA
// of the wide shapes, so its own warps have to hide the latencies; of the narrow ones several.
template <int KIN>
__host__ __device__ constexpr int fwd_bufs() { return KIN > 2 * kHidden ? 1 : 2; }
template <int KIN>
__host__ __device__ constexpr int fwd_threads() { return KIN >= kHidden ? 512 : 256; }
// The hidden tile lies in the input tile when that is wide enough: behind source 0 when the input is two
// sources wide, so that a residual taken from source 0 is still there for the second epilogue.
template <int KIN>
__host__ __device__ constexpr bool fwd_own_hidden() { return KIN < kHidden; }
template <int KIN, int NOUT>
constexpr size_t fwd_smem() {
    return (size_t)kHidden * KIN * 2 + (size_t)NOUT * kHidden * 2 + fwd_bufs<KIN>() * (size_t)kRows * KIN * 2 +
           (fwd_own_hidden<KIN>() ? (size_t)kRows * kHidden * 2 : 0) + 1024 + 64;
}

// The next tile's rows arrive while this one is worked on.  Tiles of 64 features and more, the hidden and
// the output tile are in the swizzled layout (see stage_sw).  One tile at a time, chunk-major, 200,000
// particles took 90 us with 256 inputs (B200), now 62; 1.2 M edges and 200,000 particles with 16 inputs 222,
// now 156.
template <int KIN, int NOUT>
__global__ void __launch_bounds__(fwd_threads<KIN>(), 1) k_mlp_fwd(FwdArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int NB = fwd_bufs<KIN>(), NT = fwd_threads<KIN>(), NP = NT / kRows;   // NP threads per row
    constexpr bool SW = KIN % 64 == 0;
    constexpr uint32_t TA = (uint32_t)kRows * KIN * 2;
    unsigned char *sIn = align1024(smem_raw);                          // NB input tiles
    unsigned char *sHid = sIn + NB * TA;                               // hidden tile of its own
    unsigned char *sW1 = sHid + (fwd_own_hidden<KIN>() ? kRows * kHidden * 2 : 0);   // W1^T: 128 rows x KIN
    unsigned char *sW2 = sW1 + (size_t)kHidden * KIN * 2;              // W2^T: NOUT rows x 128
    uint64_t *mbar = reinterpret_cast<uint64_t *>(sW2 + (size_t)NOUT * kHidden * 2);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(mbar + 1);
    __shared__ float s_b1[kHidden], s_b2[kHidden];
    const int tid = threadIdx.x;
    const int t = tid & (kRows - 1);   // tile row (TMEM lane) of this thread
    const int part = tid >> 7;         // columns [128 / NP part, + 128 / NP) of the epilogues
    if (tid < kHidden) s_b1[t] = a.w.b1[t];
    else if (tid < kHidden + NOUT) s_b2[t] = a.w.b2[t];
    const long ntiles = (a.rows + kRows - 1) / kRows;
    auto stage = [&](long tile, int b) {
        const long row0 = tile * kRows;
        for (int q = tid; q < kRows * (KIN / 8); q += NT) {
            int row = q / (KIN / 8), kc = q % (KIN / 8);
            if (!SW) tile_element(q, kRows, KIN / 8, row, kc);
            unsigned char *dst = sIn + b * TA + (SW ? tc::sw_off(kRows, row, kc) : tc::tile_off(kRows, row, kc));
            const long grow = row0 + row;
            if (grow < a.rows) {
                int f = kc * 8, k;
                const RowSrc r = pick_source(a.src, a.nsrc, f, k);
                cp16(dst, r.p + (r.idx ? (long)r.idx[grow] : grow) * r.width + f);
            } else {
                *reinterpret_cast<uint4 *>(dst) = make_uint4(0, 0, 0, 0);
            }
        }
    };
    stage_dense(sW1, a.w.w1t, kHidden, KIN, 0, kHidden);
    stage_dense(sW2, a.w.w2t, NOUT, kHidden, 0, NOUT);
    if (NB > 1 && blockIdx.x < ntiles) stage(blockIdx.x, 0);
    cp_commit();
    const uint32_t tm = tc_setup(mbar, tslot, 128);
    const uint32_t aW1 = tc::smem_u32(sW1), aW2 = tc::smem_u32(sW2);
    constexpr uint32_t id1 = tc::idesc_bf16(kRows, kHidden, false, false);
    constexpr uint32_t id2 = tc::idesc_bf16(kRows, NOUT, false, false);
    uint32_t phase = 0;
    bool ok = true;
    int b = 0;
    for (long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, b = NB > 1 ? b ^ 1 : 0) {
        const long row0 = tile * kRows;
        const long grow = row0 + t;
        unsigned char *sA = sIn + b * TA;
        unsigned char *sH = fwd_own_hidden<KIN>() ? sHid : sA + (KIN >= 2 * kHidden ? kRows * kHidden * 2 : 0);
        const uint32_t aA = tc::smem_u32(sA), aH = tc::smem_u32(sH);
        if (NB > 1) {
            if (tile + gridDim.x < ntiles) stage(tile + gridDim.x, b ^ 1);
            cp_commit();
            cp_wait<1>();
        } else {
            stage(tile, 0);
            cp_wait_all();
        }
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
            for (int ks = 0; ks < KIN / 16; ++ks)
                mma_issue(tm, SW ? tc::kmajor_sw(aA, kRows, ks) : tc::kmajor_desc(aA, kRows, ks), tc::kmajor_desc(aW1, kHidden, ks),
                          id1, ks > 0);
            mma_commit_issue(mbar);
        }
        ok = mma_wait(mbar, phase);
        if (!ok) break;
        // hidden = relu(acc + b1) -> bf16 tile (A operand of GEMM2), optionally saved
#pragma unroll
        for (int c32 = 0; c32 < 4 / NP; ++c32) {
            const int c0 = (part * (4 / NP) + c32) * 32;
            float w[32];
            acc32(tm, c0, w);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float *v = w + 8 * c;
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = fmaxf(v[k] + s_b1[c0 + 8 * c + k], 0.f);
                *reinterpret_cast<uint4 *>(sH + tc::sw_off(kRows, t, c0 / 8 + c)) = tc::pack8(v);
            }
        }
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
            for (int ks = 0; ks < kHidden / 16; ++ks)
                mma_issue(tm, tc::kmajor_sw(aH, kRows, ks), tc::kmajor_desc(aW2, NOUT, ks), id2, ks > 0);
            mma_commit_issue(mbar);
        }
        auto rows_out = [&](bf16 *g) {   // the hidden tile's rows, or the output's in its place
            for (int q = tid; q < kRows * 16; q += NT) {
                const int row = q >> 4, c = q & 15;
                if (row0 + row < a.rows)
                    *reinterpret_cast<uint4 *>(g + (row0 + row) * kHidden + c * 8) =
                        *reinterpret_cast<const uint4 *>(sH + tc::sw_off(kRows, row, c));
            }
        };
        if (a.h1) rows_out(a.h1);   // while the tensor core reads them too
        ok = mma_wait(mbar, phase);
        if (!ok) break;
        constexpr bool kStaged = NOUT == kHidden;   // bf16 rows written through the output tile
        constexpr int CB = kStaged ? 32 : NOUT;      // columns per TMEM wait
        static_assert(kStaged || NOUT == 16, "a narrow output is one block of 16 columns");
#pragma unroll
        for (int cb = 0; cb < (kStaged ? 4 / NP : 1); ++cb) {
            if (!kStaged && part > 0) break;
            const int c0 = kStaged ? (part * (4 / NP) + cb) * 32 : 0;
            float w[32];
            if (kStaged) acc32(tm, c0, w);
            else acc16(tm, 0, w);
            if (grow >= a.rows) continue;
#pragma unroll
            for (int c = 0; c < CB / 8; ++c) {
                float *v = w + 8 * c;
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] += s_b2[c0 + 8 * c + k];
                if (a.resid) {
                    float r[8];
                    if (KIN >= 2 * kHidden && a.resid_src0)   // source 0 is still staged in chunks [0, 16)
                        tc::unpack8(*reinterpret_cast<const uint4 *>(sA + tc::sw_off(kRows, t, c0 / 8 + c)), r);
                    else
                        tc::unpack8(*reinterpret_cast<const uint4 *>(a.resid + grow * NOUT + c0 + 8 * c), r);
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[k] += r[k];
                }
                if (a.out && kStaged) *reinterpret_cast<uint4 *>(sH + tc::sw_off(kRows, t, c0 / 8 + c)) = tc::pack8(v);
                else if (a.out) *reinterpret_cast<uint4 *>(a.out + grow * NOUT + c0 + 8 * c) = tc::pack8(v);
                if (a.out_f32) {
                    float4 *dst = reinterpret_cast<float4 *>(a.out_f32 + grow * NOUT + c0 + 8 * c);
                    dst[0] = make_float4(v[0], v[1], v[2], v[3]);
                    dst[1] = make_float4(v[4], v[5], v[6], v[7]);
                }
            }
        }
        tc::fence_before_sync();
        __syncthreads();   // TMEM and the tiles are reused by the next tile
        if (a.out && kStaged) {
            rows_out(a.out);
            __syncthreads();
        }
    }
    cp_wait_all();
    tc_teardown(tm, 128, ok, a.err, mbar, phase);
}

// ------------------------------------------------------------------------------------
// backward: input gradient
// ------------------------------------------------------------------------------------
struct BwdArgs {
    long rows;
    MlpW w;
    const bf16 *dy;   // [rows][NOUT]
    const bf16 *h1;   // [rows][128]
    bf16 *dz1;        // [rows][128]
    float *dx;        // [rows][KIN] or null
    DxSum sum;        // what dX is added to (the SUM form)
    int *err;
};

// Tiles in flight per CTA (384 inputs leave room for one), and whether the dX rows leave through a
// buffer of their own (else through the dY tile, which is spent by then).
template <int KIN>
__host__ __device__ constexpr int bwd_bufs() { return KIN > 2 * kHidden ? 1 : 2; }
template <int KIN, int NOUT>
constexpr size_t bwd_smem() {
    return (size_t)kHidden * NOUT * 2 + (size_t)KIN * kHidden * 2 +
           bwd_bufs<KIN>() * ((size_t)kRows * NOUT * 2 + (size_t)kRows * kHidden * 2) + (NOUT < kHidden ? 32768 : 0) + 1024 + 64;
}

// The next tile's dY and H arrive while this one is worked on; dZ takes H's place in the tile (each
// chunk by the thread that read it) and leaves from there, dX through a 2 KB buffer per warp, both in
// whole sectors.  One CTA fills an SM's shared memory, so the epilogues' warps are all there is to hide
// latency: four per scheduler.  With 128 threads, one tile at a time and rows written by the thread that
// owned them, 240,000 edges took 129 us (B200); with 512 threads and this order 120, in the swizzled layout
// 74.  HBM: 306 MB, 47 us at the copy rate.  SUM: dX is added to a running sum here instead of in a pass of
// its own (k_edge_grad 57 -> 36 us, one pass of four less) for 74 -> 105 us; the sum's loads are issued behind
// the first product (after the second one 145).
template <int KIN, int NOUT, bool SUM>
__global__ void __launch_bounds__(kBwdThreads, 1) k_mlp_bwd(BwdArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char *smem = align1024(smem_raw);
    constexpr int NB = bwd_bufs<KIN>();
    constexpr uint32_t TY = (uint32_t)kRows * NOUT * 2, TH = (uint32_t)kRows * kHidden * 2;
    unsigned char *sW2 = smem;                                  // W2: 128 rows (in) x NOUT
    unsigned char *sW1 = sW2 + (size_t)kHidden * NOUT * 2;      // W1: KIN rows (in) x 128
    unsigned char *sIn = sW1 + (size_t)KIN * kHidden * 2;       // per tile in flight: dY 128 x NOUT, H (then dZ) 128 x 128
    unsigned char *sOut = sIn + (size_t)NB * (TY + TH);         // dX buffers of the warps (NOUT < 128)
    uint64_t *mbar = reinterpret_cast<uint64_t *>(sOut + (NOUT < kHidden ? 32768 : 0));
    uint32_t *tslot = reinterpret_cast<uint32_t *>(mbar + 1);
    const int tid = threadIdx.x, t = tid & (kRows - 1), part = tid >> 7, lane = tid & 31;
    const bool want_dx = a.dx != nullptr;
    const long ntiles = (a.rows + kRows - 1) / kRows;
    auto stage = [&](long tile, int b) {
        unsigned char *y = sIn + (size_t)b * (TY + TH);
        if (NOUT == kHidden) stage_sw(y, a.dy, kRows, NOUT, tile * kRows, a.rows);
        else stage_dense(y, a.dy, kRows, NOUT, tile * kRows, a.rows);
        stage_sw(y + TY, a.h1, kRows, kHidden, tile * kRows, a.rows);
    };

    stage_dense(sW2, a.w.w2, kHidden, NOUT, 0, kHidden);
    if (want_dx) stage_dense(sW1, a.w.w1, KIN, kHidden, 0, KIN);
    if (NB > 1 && blockIdx.x < ntiles) stage(blockIdx.x, 0);
    cp_commit();
    const uint32_t tm = tc_setup(mbar, tslot, 512);
    const uint32_t aW1 = tc::smem_u32(sW1), aW2 = tc::smem_u32(sW2);
    constexpr uint32_t id1 = tc::idesc_bf16(kRows, kHidden, false, false);
    constexpr int NX = KIN < 128 ? KIN : 128;   // N of one input-gradient chunk
    constexpr uint32_t idx = tc::idesc_bf16(kRows, NX, false, false);
    uint32_t phase = 0;
    bool ok = true;
    int b = 0;
    for (long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, b = NB > 1 ? b ^ 1 : 0) {
        const long row0 = tile * kRows;
        const long grow = row0 + t;
        unsigned char *sY = sIn + (size_t)b * (TY + TH), *sZ = sY + TY;
        const uint32_t aY = tc::smem_u32(sY), aZ = tc::smem_u32(sZ);
        if (NB > 1) {
            if (tile + gridDim.x < ntiles) stage(tile + gridDim.x, b ^ 1);
            cp_commit();
            cp_wait<1>();
        } else {
            stage(tile, 0);
            cp_wait_all();
        }
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
            for (int ks = 0; ks < NOUT / 16; ++ks)
                mma_issue(tm, NOUT == kHidden ? tc::kmajor_sw(aY, kRows, ks) : tc::kmajor_desc(aY, kRows, ks), tc::kmajor_desc(aW2, kHidden, ks), id1, ks > 0);
            mma_commit_issue(mbar);
        }
        // what dX is added to, of the rows and columns this lane stores, while the products run
        [[maybe_unused]] float4 base[8];
        [[maybe_unused]] const DxSum &S = a.sum;
        if constexpr (SUM) {
            static_assert(KIN == kHidden, "one block of 32 columns per thread");
            const int col = part * 32 + (lane & 7) * 4;
            float4 d[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const long r = row0 + (t & ~31) + 4 * k + (lane >> 3), rr = r < a.rows ? r : 0;
                base[k] = S.run ? *reinterpret_cast<const float4 *>(S.run + rr * KIN + col) : make_float4(0.f, 0.f, 0.f, 0.f);
                d[k] = *reinterpret_cast<const float4 *>(S.add + (long)S.idx[rr] * S.ld + S.col + col);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                base[k].x += d[k].x;
                base[k].y += d[k].y;
                base[k].z += d[k].z;
                base[k].w += d[k].w;
            }
        }
        ok = mma_wait(mbar, phase);
        if (!ok) break;
        {
            float w[32], h[8];
            acc32(tm, part * 32, w);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                unsigned char *at = sZ + tc::sw_off(kRows, t, part * 4 + c);
                float *v = w + 8 * c;
                tc::unpack8(*reinterpret_cast<const uint4 *>(at), h);
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = grow < a.rows && h[k] > 0.f ? v[k] : 0.f;
                *reinterpret_cast<uint4 *>(at) = tc::pack8(v);
            }
        }
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        if (want_dx && tid == 0) {
            tc::fence_after_sync();
            for (int j = 0; j < KIN / NX; ++j)   // N chunk j: input features [j*NX, j*NX + NX)
                for (int ks = 0; ks < kHidden / 16; ++ks)
                    mma_issue(tm + kHidden + j * NX, tc::kmajor_sw(aZ, kRows, ks),
                                 tc::kmajor_desc(aW1 + (uint32_t)(j * NX * 16), KIN, ks), idx, ks > 0);
            mma_commit_issue(mbar);
        }
        for (int q = tid; q < kRows * (kHidden / 8); q += kBwdThreads) {   // dZ rows, while the tensor core reads them too
            const int row = q >> 4, c = q & 15;
            if (row0 + row < a.rows)
                *reinterpret_cast<uint4 *>(a.dz1 + (row0 + row) * kHidden + c * 8) =
                    *reinterpret_cast<const uint4 *>(sZ + tc::sw_off(kRows, row, c));
        }
        if (want_dx) {
            ok = mma_wait(mbar, phase);
            if (!ok) break;
            if constexpr (KIN >= 64) {
                // 32 columns of 16 rows at a time
                float4 *buf = reinterpret_cast<float4 *>((NOUT < kHidden ? sOut : sY) + (tid >> 5) * 2048);
                const long wrow0 = row0 + (t & ~31);
                for (int c = part; c < KIN / 32; c += 4) {
                    float v[32];
                    acc32(tm, kHidden + c * 32, v);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if ((lane >> 4) == h)
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                buf[(lane & 15) * 8 + ((k ^ lane) & 7)] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
                        __syncwarp();
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const int r = 4 * k + (lane >> 3), f = lane & 7;
                            const long grow_r = wrow0 + 16 * h + r;
                            float4 o = buf[r * 8 + ((f ^ r) & 7)];
                            if constexpr (SUM) {
                                const float4 &s = base[4 * h + k];
                                o = make_float4(s.x + o.x, s.y + o.y, s.z + o.z, s.w + o.w);
                            }
                            if (grow_r < a.rows) {
                                if (SUM && S.out_bf) {
                                    const __nv_bfloat162 lo = __floats2bfloat162_rn(o.x, o.y), hi = __floats2bfloat162_rn(o.z, o.w);
                                    *reinterpret_cast<uint2 *>((bf16 *)S.out_bf + grow_r * KIN + c * 32 + f * 4) =
                                        make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
                                } else {
                                    *reinterpret_cast<float4 *>(a.dx + grow_r * KIN + c * 32 + f * 4) = o;
                                }
                            }
                        }
                        __syncwarp();
                    }
                }
            } else if (part == 0) {
                for (int c = 0; c < KIN / 16; ++c) {
                    float v[16];
                    acc16(tm, kHidden + c * 16, v);
                    if (grow < a.rows) {
                        float4 *dst = reinterpret_cast<float4 *>(a.dx + grow * KIN + c * 16);
                        for (int k = 0; k < 4; ++k) dst[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
                    }
                }
            }
        }
        tc::fence_before_sync();
        __syncthreads();
    }
    cp_wait_all();
    tc_teardown(tm, 512, ok, a.err, mbar, phase);
}

// ------------------------------------------------------------------------------------
// backward: weight and bias gradients (per-CTA partials)
// ------------------------------------------------------------------------------------
struct WgradArgs {
    long rows;
    RowSrc src[3];
    int nsrc;
    const bf16 *dz1;   // [rows][128]
    const bf16 *h1;    // [rows][128]
    const bf16 *dy;    // [rows][NOUT]
    float *part;       // per CTA: [128][KIN + NW2]: dW1^T | dW2 block, then db1 [128], db2 [128]
    int *err;
};

template <int NOUT>
__host__ __device__ constexpr int wgrad_w2_cols() { return NOUT == kHidden ? kHidden : NOUT; }
template <int KIN, int NOUT>
__host__ __device__ constexpr int wgrad_cols() { return KIN + wgrad_w2_cols<NOUT>() + 2; }
template <int KIN, int NOUT>
__host__ __device__ constexpr int wgrad_tmem_cols() {
    return (KIN + wgrad_w2_cols<NOUT>()) <= 256 ? 256 : 512;
}
// Rows of a stage and stages in flight: all the shared memory holds.
constexpr int kWgRows = 64;
template <int KIN, int NOUT>
__host__ __device__ constexpr size_t wgrad_stage() { return (size_t)kWgRows * (2 * kHidden + KIN + NOUT) * 2; }
template <int KIN>
__host__ __device__ constexpr int wgrad_stages() { return KIN >= 2 * kHidden ? 2 : 3; }
template <int KIN, int NOUT>
constexpr size_t wgrad_smem() { return wgrad_stages<KIN>() * wgrad_stage<KIN, NOUT>() + 1024 + 64; }

// The rows pass through a ring of stages of 64, each a K = 64 step of both products: while the tensor
// core and the bias sums take one, the copies of the next one or two are in flight.  A stage's buffer is
// filled again once its own products are done, a stage later.  One tile of 128 rows at a time, loaded by
// 128 threads and summed by one thread per column, 240,000 edges took 157 us (B200); the ring with 512
// threads 107, in the swizzled layout 64, with the accumulators' rows written in whole sectors 55 (256 inputs,
// 40,000 rows: 73 -> 24).  HBM: 246 MB, 38 us at the copy rate.
template <int KIN, int NOUT>
__global__ void __launch_bounds__(kBwdThreads, 1) k_mlp_wgrad(WgradArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char *smem = align1024(smem_raw);
    constexpr int NS = wgrad_stages<KIN>(), R = kWgRows;
    constexpr uint32_t SB = (uint32_t)wgrad_stage<KIN, NOUT>();
    constexpr uint32_t OH = R * kHidden * 2, OX = 2 * OH, OY = OX + R * KIN * 2;   // dZ at 0, H, X, dY
    uint64_t *mbar = reinterpret_cast<uint64_t *>(smem + (size_t)NS * SB);         // one per stage
    uint32_t *tslot = reinterpret_cast<uint32_t *>(mbar + NS);
    const int tid = threadIdx.x;
    constexpr int TC = wgrad_tmem_cols<KIN, NOUT>();
    if (tid > 0 && tid < NS) tc::mbar_init(mbar + tid, 1);
    const uint32_t tm = tc_setup(mbar, tslot, TC);
    constexpr int NX = KIN < 128 ? KIN : 128;
    constexpr bool SWX = KIN % 64 == 0, SWY = NOUT == kHidden;   // swizzled tiles (16 features: plain ones)
    constexpr uint32_t idx = tc::idesc_bf16(kRows, NX, true, true);
    constexpr uint32_t id2 = tc::idesc_bf16(kRows, NOUT == kHidden ? kHidden : NOUT, true, true);
    const long ntiles = (a.rows + kRows - 1) / kRows;
    const long units = 2 * ((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x);   // the grid has no more CTAs than tiles
    auto fill = [&](long u) {
        unsigned char *s = smem + (size_t)(u % NS) * SB;
        const long row0 = (blockIdx.x + (u >> 1) * gridDim.x) * kRows + (u & 1) * R;
        stage_sw(s, a.dz1, R, kHidden, row0, a.rows);
        stage_sw(s + OH, a.h1, R, kHidden, row0, a.rows);
        for (int q = tid; q < R * (KIN / 8); q += kBwdThreads) {   // the concatenated input row
            const int row = q / (KIN / 8), kc = q % (KIN / 8);
            unsigned char *dst = s + OX + (SWX ? tc::sw_off(R, row, kc) : tc::tile_off(R, row, kc));
            const long grow = row0 + row;
            if (grow < a.rows) {
                int f = kc * 8, k;
                const RowSrc src = pick_source(a.src, a.nsrc, f, k);
                cp16(dst, src.p + (src.idx ? (long)src.idx[grow] : grow) * src.width + f);
            } else {
                *reinterpret_cast<uint4 *>(dst) = make_uint4(0, 0, 0, 0);
            }
        }
        if (SWY) stage_sw(s + OY, a.dy, R, NOUT, row0, a.rows);
        else stage_dense(s + OY, a.dy, R, NOUT, row0, a.rows);
    };
    // bias sums: features [8 kc, 8 kc + 8) of rows r0 and r0 + 32
    const int kc = (tid >> 4) & 15, r0 = (tid & 15) + 16 * (tid >> 8);
    float z[8], y[8];
    for (int k = 0; k < 8; ++k) z[k] = y[k] = 0.f;
    bool ok = true;
    long u = 0;
    for (; u < NS - 1; ++u) {
        if (u < units) fill(u);
        cp_commit();
    }
    for (u = 0; u < units; ++u) {
        cp_wait<NS - 2>();   // this thread's share of stage u has landed
        tc::fence_async_smem();
        tc::fence_before_sync();
        ok = __syncthreads_and(ok) != 0;
        if (!ok) break;
        unsigned char *s = smem + (size_t)(u % NS) * SB;
        if (tid == 0) {
            tc::fence_after_sync();
            const uint32_t aZ = tc::smem_u32(s), aH = aZ + OH, aX = aZ + OX, aY = aZ + OY;
            for (int j = 0; j < KIN / NX; ++j)   // dW1^T[:, j*NX .. ] += dZ^T X_j
                for (int ks = 0; ks < R / 16; ++ks)
                    mma_issue(tm + j * NX, tc::mnmajor_sw(aZ, R, ks),
                                 SWX ? tc::mnmajor_sw(aX + (uint32_t)(j * NX * R * 2), R, ks) : tc::mnmajor_desc(aX, R, ks), idx,
                                 (u > 0 || ks > 0) ? 1u : 0u);
            for (int ks = 0; ks < R / 16; ++ks) {
                if (NOUT == kHidden)   // dW2^T += dY^T H
                    mma_issue(tm + KIN, tc::mnmajor_sw(aY, R, ks), tc::mnmajor_sw(aH, R, ks), id2,
                                 (u > 0 || ks > 0) ? 1u : 0u);
                else                   // dW2 += H^T dY (M = 128 hidden, N = NOUT)
                    mma_issue(tm + KIN, tc::mnmajor_sw(aH, R, ks), tc::mnmajor_desc(aY, R, ks), id2,
                                 (u > 0 || ks > 0) ? 1u : 0u);
            }
            mma_commit_issue(mbar + u % NS);
        }
        // stage u - 1's products are done and its sums were taken before the barrier: fill its buffer again
        if (u > 0) ok = tc::mbar_wait(mbar + (u - 1) % NS, (uint32_t)((u - 1) / NS) & 1u, g_tc_wait_limit);
        if (u + NS - 1 < units) fill(u + NS - 1);
        cp_commit();
        // bias sums from the stage while the tensor core runs (fixed row order)
#pragma unroll
        for (int i = 0; i < R / 32; ++i) {
            float v[8];
            tc::unpack8(*reinterpret_cast<const uint4 *>(s + tc::sw_off(R, r0 + 32 * i, kc)), v);
#pragma unroll
            for (int k = 0; k < 8; ++k) z[k] += v[k];
            if (kc < NOUT / 8) {
                tc::unpack8(*reinterpret_cast<const uint4 *>(s + OY + (SWY ? tc::sw_off(R, r0 + 32 * i, kc) : tc::tile_off(R, r0 + 32 * i, kc))), v);
#pragma unroll
                for (int k = 0; k < 8; ++k) y[k] += v[k];
            }
        }
    }
    cp_wait_all();
    // the last stage's products (after a wait that gave up: of the stages issued, again with a limit)
    if (u > 0) ok = tc::mbar_wait(mbar + (u - 1) % NS, (uint32_t)((u - 1) / NS) & 1u, g_tc_wait_limit) && ok;
    ok = __syncthreads_and(ok) != 0;
    constexpr int NM = KIN + wgrad_w2_cols<NOUT>(), NC = NM + 2;
    float *part = a.part + (long)blockIdx.x * kRows * NC;
    const int t = tid & (kRows - 1), lane = tid & 31;
    __shared__ float s_db[2][2][kHidden];   // [rows 16 (tid / 256) ..][layer]
#pragma unroll
    for (int k = 0; k < 8; ++k)
        for (int o = 8; o > 0; o >>= 1) {
            z[k] += __shfl_xor_sync(0xffffffffu, z[k], o);
            y[k] += __shfl_xor_sync(0xffffffffu, y[k], o);
        }
    if ((tid & 15) == 0)
        for (int k = 0; k < 8; ++k) {
            s_db[tid >> 8][0][kc * 8 + k] = z[k];
            s_db[tid >> 8][1][kc * 8 + k] = y[k];
        }
    __syncthreads();
    if (ok) {
        tc::fence_after_sync();
        // the accumulators' rows through a buffer per warp in the spent stages, 16 columns at a time
        float4 *buf = reinterpret_cast<float4 *>(smem + (tid >> 5) * 2048);
        for (int c = tid >> 7; c < NM / 16; c += 4) {
            float v[16];
            acc16(tm, c * 16, v);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                buf[lane * 4 + ((k + (lane >> 1)) & 3)] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int r = 8 * k + (lane >> 2), f = lane & 3;
                *reinterpret_cast<float4 *>(part + (long)((t & ~31) + r) * NM + c * 16 + f * 4) = buf[r * 4 + ((f + (r >> 1)) & 3)];
            }
            __syncwarp();
        }
    } else {
        for (int c = tid; c < kRows * NC; c += kBwdThreads) part[c] = 0.f;
        __syncthreads();
    }
    if (tid < kRows) {
        part[(long)kRows * NM + tid] = s_db[0][0][tid] + s_db[1][0][tid];
        part[(long)kRows * NM + kRows + tid] = s_db[0][1][tid] + s_db[1][1][tid];
    }
    tc::fence_before_sync();
    __syncthreads();
    if (tid < 32) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tm, TC);
    }
    if (!ok && tid == 0 && a.err) atomicOr(a.err, DEM_ERR_TIMEOUT);
}

// p[0] + p[stride] + ... over the blocks in order, eight loads in flight.
__device__ __forceinline__ float sum_blocks(const float *p, long stride, int nblocks) {
    float s = 0.f;
    int b = 0;
    for (; b + 8 <= nblocks; b += 8) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = p[(b + k) * stride];
#pragma unroll
        for (int k = 0; k < 8; ++k) s += v[k];
    }
    for (; b < nblocks; ++b) s += p[b * stride];
    return s;
}

// Sum the per-CTA partials in block order and add them to the gradient buffers:
// g_w1t [128][KIN], g_b1 [128], g_w2t [NOUT][128], g_b2 [NOUT].
__global__ void k_wgrad_reduce(const float *part, int nblocks, int kin, int nout, float *g_w1t, int ld_w1, float *g_b1,
                               float *g_w2t, float *g_b2) {
    const int nw2 = nout == kHidden ? kHidden : nout;
    const int nm = kin + nw2, nc = nm + 2;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < kRows * nc; e += gridDim.x * blockDim.x) {
        const int bias = e - kRows * nm;   // from 0 on: db1, then db2
        const int r = bias < 0 ? e / nm : bias % kRows, c = bias < 0 ? e % nm : nm + bias / kRows;
        const float s = sum_blocks(part + e, (long)kRows * nc, nblocks);
        if (c < kin) g_w1t[(long)r * ld_w1 + c] += s;
        else if (c < kin + nw2) {
            const int cc = c - kin;
            if (nout == kHidden) g_w2t[r * kHidden + cc] += s;   // row r = output unit
            else g_w2t[cc * kHidden + r] += s;                   // row r = hidden unit
        } else if (c == kin + nw2) g_b1[r] += s;
        else if (r < nout) g_b2[r] += s;
    }
}

// Dynamic shared memory is raised so that the CTAs one SM can hold never ask for more TMEM
// columns than its 512 (an allocation that cannot be met would wait for another CTA).
// 228 KB of shared memory per SM: > 114 KB leaves one CTA, > 76 KB two, > 57 KB three.
// ------------------------------------------------------------------------------------
// factorised edge layer:  z = W1e e + P[recv] + Q[send] + b1,  PQ = [W1i h | W1j h]
// (W1 = [W1e | W1i | W1j] of the 384-wide edge-update perceptron), e' = e + W2 relu(z) + b2
// ------------------------------------------------------------------------------------
struct LinArgs {
    long rows;
    const bf16 *x;      // [rows][KIN]
    const bf16 *wt;     // [NOUT][KIN] (out x in)
    bf16 *out;          // [rows][NOUT]
    float *acc_out;     // [rows][NOUT] FP32, added to (used instead of out when set)
    int *err;
};

// out = x W^T (no bias), M = 128 rows per tile, N = NOUT (<= 256), K = KIN.  The next tile's rows arrive
// while this one is worked on (swizzled layout, see stage_sw); the output leaves through a buffer per warp
// in whole lines.  One tile at a time, chunk-major and rows written by the thread that owned them, 200,000
// rows took 65 us with 128 in and 256 out (B200), now 35, and the 40,000 rows of the backward product,
// added to FP32, 39, now 17.
template <int KIN, int NOUT>
constexpr size_t lin_smem() {
    return (size_t)NOUT * KIN * 2 + 2 * (size_t)kRows * KIN * 2 + (kLinThreads / 32) * 2048 + 1024 + 64;
}

template <int KIN, int NOUT>
__global__ void __launch_bounds__(kLinThreads, 1) k_linear(LinArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char *sA = align1024(smem_raw);                   // two tiles of 128 rows x KIN
    constexpr uint32_t TA = (uint32_t)kRows * KIN * 2;
    unsigned char *sW = sA + 2 * TA;                           // NOUT rows x KIN
    unsigned char *sBuf = sW + (size_t)NOUT * KIN * 2;         // 2 KB per warp
    uint64_t *mbar = reinterpret_cast<uint64_t *>(sBuf + (kLinThreads / 32) * 2048);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(mbar + 1);
    const int tid = threadIdx.x, t = tid & (kRows - 1), part = tid >> 7, lane = tid & 31;
    constexpr int TC = NOUT <= 128 ? 128 : 256, NP = kLinThreads / kRows;
    const long ntiles = (a.rows + kRows - 1) / kRows;
    stage_sw(sW, a.wt, NOUT, KIN, 0, NOUT);
    if (blockIdx.x < ntiles) stage_sw(sA, a.x, kRows, KIN, (long)blockIdx.x * kRows, a.rows);
    cp_commit();
    const uint32_t tm = tc_setup(mbar, tslot, TC);
    const uint32_t aW = tc::smem_u32(sW);
    constexpr uint32_t id = tc::idesc_bf16(kRows, NOUT, false, false);
    uint32_t phase = 0;
    bool ok = true;
    int b = 0;
    for (long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, b ^= 1) {
        const uint32_t aA = tc::smem_u32(sA) + (uint32_t)b * TA;
        if (tile + gridDim.x < ntiles) stage_sw(sA + (b ^ 1) * TA, a.x, kRows, KIN, (tile + gridDim.x) * kRows, a.rows);
        cp_commit();
        cp_wait<1>();
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
            for (int ks = 0; ks < KIN / 16; ++ks)
                mma_issue(tm, tc::kmajor_sw(aA, kRows, ks), tc::kmajor_sw(aW, NOUT, ks), id, ks > 0);
            mma_commit_issue(mbar);
        }
        ok = mma_wait(mbar, phase);
        if (!ok) break;
        const long wrow0 = tile * kRows + (t & ~31);
        uint4 *buf = reinterpret_cast<uint4 *>(sBuf + (tid >> 5) * 2048);
        if (a.acc_out) {   // 32 columns of 16 rows at a time
            for (int c = part; c < NOUT / 32; c += NP) {
                float v[32];
                acc32(tm, c * 32, v);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if ((lane >> 4) == h)
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            reinterpret_cast<float4 *>(buf)[(lane & 15) * 8 + ((k ^ lane) & 7)] =
                                make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
                    __syncwarp();
                    float4 o[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const long grow = wrow0 + 16 * h + 4 * k + (lane >> 3);
                        if (grow < a.rows) o[k] = *reinterpret_cast<const float4 *>(a.acc_out + grow * NOUT + c * 32 + (lane & 7) * 4);
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int r = 4 * k + (lane >> 3), f = lane & 7;
                        const long grow = wrow0 + 16 * h + r;
                        const float4 s = reinterpret_cast<const float4 *>(buf)[r * 8 + ((f ^ r) & 7)];
                        if (grow < a.rows) {
                            o[k].x += s.x;
                            o[k].y += s.y;
                            o[k].z += s.z;
                            o[k].w += s.w;
                            *reinterpret_cast<float4 *>(a.acc_out + grow * NOUT + c * 32 + f * 4) = o[k];
                        }
                    }
                    __syncwarp();
                }
            }
        } else {           // 64 columns of 16 rows at a time
            for (int c = part; c < NOUT / 64; c += NP) {
                float v[64];
                acc64(tm, c * 64, v);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if ((lane >> 4) == h)
#pragma unroll
                        for (int k = 0; k < 8; ++k) buf[(lane & 15) * 8 + ((k ^ lane) & 7)] = tc::pack8(v + 8 * k);
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int r = 4 * k + (lane >> 3), f = lane & 7;
                        const long grow = wrow0 + 16 * h + r;
                        if (grow < a.rows)
                            *reinterpret_cast<uint4 *>(a.out + grow * NOUT + c * 64 + f * 8) = buf[r * 8 + ((f ^ r) & 7)];
                    }
                    __syncwarp();
                }
            }
        }
        tc::fence_before_sync();
        __syncthreads();
    }
    cp_wait_all();
    tc_teardown(tm, TC, ok, a.err, mbar, phase);
}

struct EdgeArgs {
    long rows;
    const bf16 *e;       // [rows][128] input latent, also the residual
    const bf16 *pq;      // [nodes][256]
    const int *recv, *send;
    const bf16 *w1e_t;   // [128][128]
    const float *b1;
    const bf16 *w2t;     // [128][128]
    const float *b2;
    bf16 *out;           // [rows][128]
    bf16 *h1;            // [rows][128] or null
    int *err;
};

constexpr size_t edge_smem() { return 3 * (size_t)kRows * kHidden * 2 + 64; }

// Two CTAs of 256 threads per SM (96 KB of shared memory each), so that one CTA's tensor-core
// and memory waits overlap the other's epilogues.  Thread (row t, half) prefetches the half
// rows of P[recv] and Q[send] it needs into registers before the first product, reloads its
// residual half row (an L2 hit) while the second product runs, and writes its output through
// the spent tile so that whole 256-byte rows leave the SM.
__global__ void __launch_bounds__(kFwdThreads, 2) k_edge_fwd(EdgeArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr size_t T = (size_t)kRows * kHidden * 2;
    unsigned char *sW1 = smem;          // W1e^T 128 x 128
    unsigned char *sW2 = sW1 + T;       // W2^T 128 x 128
    unsigned char *sA = sW2 + T;        // e tile -> hidden tile -> output tile
    uint64_t *mbar = reinterpret_cast<uint64_t *>(sA + T);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(mbar + 1);
    __shared__ float s_b1[kHidden], s_b2[kHidden];
    const int tid = threadIdx.x;
    const int t = tid & (kRows - 1);   // tile row (TMEM lane)
    const int half = tid >> 7;         // features [64 half, 64 half + 64)
    if (half == 0) s_b1[t] = a.b1[t];
    else s_b2[t] = a.b2[t];
    stage_dense(sW1, a.w1e_t, kHidden, kHidden, 0, kHidden);
    stage_dense(sW2, a.w2t, kHidden, kHidden, 0, kHidden);
    cp_wait_all();
    const uint32_t tm = tc_setup(mbar, tslot, 128);
    const uint32_t aW1 = tc::smem_u32(sW1), aW2 = tc::smem_u32(sW2), aA = tc::smem_u32(sA);
    constexpr uint32_t id = tc::idesc_bf16(kRows, kHidden, false, false);
    uint32_t phase = 0;
    bool ok = true;
    const long ntiles = (a.rows + kRows - 1) / kRows;
    for (long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const long row0 = tile * kRows, grow = row0 + t;
        const bool live = grow < a.rows;
        stage_dense(sA, a.e, kRows, kHidden, row0, a.rows);
        uint4 p[8], q[8];
        {
            const long r = live ? a.recv[grow] : 0, c = live ? a.send[grow] : 0;
            const uint4 *ps = reinterpret_cast<const uint4 *>(a.pq + r * 2 * kHidden + half * 64);
            const uint4 *qs = reinterpret_cast<const uint4 *>(a.pq + c * 2 * kHidden + kHidden + half * 64);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                p[k] = ps[k];
                q[k] = qs[k];
            }
        }
        stage_done();
        if (tid == 0) {
            tc::fence_after_sync();
            for (int ks = 0; ks < kHidden / 16; ++ks)
                mma_issue(tm, tc::kmajor_desc(aA, kRows, ks), tc::kmajor_desc(aW1, kHidden, ks), id, ks > 0);
            mma_commit_issue(mbar);
        }
        ok = mma_wait(mbar, phase);
        if (!ok) break;
#pragma unroll
        for (int b = 0; b < 2; ++b) {   // two batches of 32 columns keep the P/Q registers live
            float w[32];
            acc32(tm, half * 64 + b * 32, w);
#pragma unroll
            for (int c2 = 0; c2 < 2; ++c2) {
                const int cc = 2 * b + c2;
                const int c = half * 4 + cc;   // 16-feature group
                float *v = w + 16 * c2, pf[8], qf[8];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    tc::unpack8(p[2 * cc + h], pf);
                    tc::unpack8(q[2 * cc + h], qf);
                    for (int k = 0; k < 8; ++k)
                        v[8 * h + k] = fmaxf(v[8 * h + k] + s_b1[c * 16 + 8 * h + k] + pf[k] + qf[k], 0.f);
                }
                const uint4 lo = tc::pack8(v), hi = tc::pack8(v + 8);
                *reinterpret_cast<uint4 *>(sA + tc::tile_off(kRows, t, 2 * c)) = lo;
                *reinterpret_cast<uint4 *>(sA + tc::tile_off(kRows, t, 2 * c + 1)) = hi;
                if (a.h1 && live) {
                    uint4 *dst = reinterpret_cast<uint4 *>(a.h1 + grow * kHidden + c * 16);
                    dst[0] = lo;
                    dst[1] = hi;
                }
            }
        }
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after_sync();
            for (int ks = 0; ks < kHidden / 16; ++ks)
                mma_issue(tm, tc::kmajor_desc(aA, kRows, ks), tc::kmajor_desc(aW2, kHidden, ks), id, ks > 0);
            mma_commit_issue(mbar);
        }
        {   // residual half row while the second product runs
            const uint4 *es = reinterpret_cast<const uint4 *>(a.e + (live ? grow : 0) * kHidden + half * 64);
#pragma unroll
            for (int k = 0; k < 8; ++k) p[k] = es[k];
        }
        ok = mma_wait(mbar, phase);
        if (!ok) break;
        {
            float w[64];
            acc64(tm, half * 64, w);
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                const int c = half * 4 + cc;
                float *v = w + 16 * cc, r[8];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    tc::unpack8(p[2 * cc + h], r);
                    for (int k = 0; k < 8; ++k) v[8 * h + k] += s_b2[c * 16 + 8 * h + k] + r[k];
                }
                out_put(sA, t, 2 * c, tc::pack8(v));
                out_put(sA, t, 2 * c + 1, tc::pack8(v + 8));
            }
        }
        tc::fence_before_sync();
        __syncthreads();
        copy_out(sA, a.out, row0, a.rows);
        __syncthreads();
    }
    tc_teardown(tm, 128, ok, a.err, mbar, phase);
}

// The same layer with its row tiles brought in by the tensor copy engine and the hidden tile
// kept in tensor memory.  One CTA of 512 threads per SM: two groups of 256, each with a tile of its
// own in flight (its e tiles, accumulator, barriers), share the weights.  Per tile the e rows arrive as
// two 64-feature boxes of a tiled tensor copy in the 128-byte swizzle layout (one elected thread
// issues them on an mbarrier, one tile ahead, into the other of the group's two buffers); the first
// product reads them from shared memory while the group gathers P and Q; the epilogue writes the
// hidden activations as BF16 pairs into tensor memory (tcgen05.st), which is the A operand of
// the second product; the output rows take the place of the residual's in the e tile and leave by a
// tensor copy, which leaves out rows past the end.  Same arithmetic, in the same order, as k_edge_fwd.
//
// P, Q and the saved hidden rows pass through a 2 KB buffer per warp: eight lanes read or write one
// row's 128 bytes in global memory, and a thread takes its own row's eight chunks from the buffer
// (chunks XOR-swizzled by the row, no bank conflicts).  A thread reading its own row directly touched
// 32 lines per instruction: 1,024 L1 wavefronts per warp and tile.  What bounds it now: latency, with
// no unit above 40 %: the gathers, two products and two epilogues of a tile follow one another, and
// two groups are all that shared memory holds.  Measured (B200, 1.2 M edges): rows read directly 358 us,
// through the buffers 277, with the gather behind the first product and the residual from the e tile
// 268.  Not kept: 1,024 threads, 32 features each (64-byte gathers) 325; prefetches of the next rows
// 269; the weights in the chunk-major layout 268.
constexpr int kEdgeThreads = 512, kEdgeGroup = 256;
constexpr size_t edge_tma_smem() {
    return 1024 + 6 * (size_t)kRows * kHidden * 2 + (size_t)(kEdgeThreads / 32) * 2048 + 128;
}

// Barrier of one group of 256 threads (ids 1 and 2), and the same with a vote.
__device__ __forceinline__ void group_sync(int id) { asm volatile("bar.sync %0, 256;" ::"r"(id) : "memory"); }
__device__ __forceinline__ bool group_and(int id, bool p) {
    uint32_t r;
    asm volatile(
        "{\n\t"
        ".reg .pred a, b;\n\t"
        "setp.ne.u32 a, %1, 0;\n\t"
        "bar.red.and.pred b, %2, 256, a;\n\t"
        "selp.u32 %0, 1, 0, b;\n\t"
        "}\n"
        : "=r"(r)
        : "r"(p ? 1u : 0u), "r"(id)
        : "memory");
    return r != 0;
}

// A warp's 32 half rows of 64 features, row r of lane r: coalesced between global memory and the
// buffer (row_in_lane: the row, of the lane's 4 k + lane / 8, chunk lane % 8), own rows between the
// buffer and registers.
__device__ __forceinline__ unsigned char *warp_chunk(unsigned char *buf, int row, int c) {
    return buf + row * 128 + ((c ^ (row & 7)) << 4);
}
__device__ __forceinline__ void warp_rows_issue(const bf16 *base, long stride, int own_row, uint4 v[8]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const long r = __shfl_sync(0xffffffffu, own_row, 4 * k + (lane >> 3));
        v[k] = *reinterpret_cast<const uint4 *>(base + r * stride + (lane & 7) * 8);
    }
}
__device__ __forceinline__ void warp_rows_take(unsigned char *buf, const uint4 v[8], uint4 own[8]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int h = 0; h < 2; ++h) {   // 16 rows at a time
#pragma unroll
        for (int k = 0; k < 4; ++k)
            *reinterpret_cast<uint4 *>(warp_chunk(buf, 4 * k + (lane >> 3), lane & 7)) = v[4 * h + k];
        __syncwarp();
        if ((lane >> 4) == h)
#pragma unroll
            for (int c = 0; c < 8; ++c) own[c] = *reinterpret_cast<const uint4 *>(warp_chunk(buf, lane & 15, c));
        __syncwarp();
    }
}
__device__ __forceinline__ void warp_rows_store(unsigned char *buf, const uint4 own[8], bf16 *g, long row0, long rows) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if ((lane >> 4) == h)
#pragma unroll
            for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4 *>(warp_chunk(buf, lane & 15, c)) = own[c];
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int row = 4 * k + (lane >> 3);
            const long grow = row0 + 16 * h + row;
            if (grow < rows)
                *reinterpret_cast<uint4 *>(g + grow * kHidden + (lane & 7) * 8) =
                    *reinterpret_cast<const uint4 *>(warp_chunk(buf, row, lane & 7));
        }
        __syncwarp();
    }
}

template <bool SAVE_H1>
__global__ void __launch_bounds__(kEdgeThreads, 1) k_edge_fwd_tma(const __grid_constant__ CUtensorMap tm_e, const __grid_constant__ CUtensorMap tm_out,
                                                                    EdgeArgs a) {
    // 1,024-byte alignment by hand: an extern array declared with it would raise the alignment of
    // every kernel's dynamic shared memory in this file (and their static padding with it)
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr uint32_t T = (uint32_t)kRows * kHidden * 2;   // one 128 x 128 BF16 tile
    unsigned char *sE0 = align1024(smem_raw);
    unsigned char *sW1 = sE0 + 4 * T;   // W1e^T 128 x 128 (row tile), after the groups' two e tiles each
    unsigned char *sW2 = sW1 + T;       // W2^T 128 x 128 (row tile)
    unsigned char *sBuf = sW2 + T;      // 2 KB per warp
    uint64_t *bars = reinterpret_cast<uint64_t *>(sBuf + (kEdgeThreads / 32) * 2048);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bars + 6);
    __shared__ __align__(16) float s_b1[kHidden], s_b2[kHidden];
    const int group = threadIdx.x / kEdgeGroup, tid = threadIdx.x % kEdgeGroup, bid = 1 + group;
    const int t = tid & (kRows - 1);   // tile row (TMEM lane)
    const int half = tid >> 7;         // features [64 half, 64 half + 64)
    unsigned char *sEg = sE0 + group * 2 * T, *buf = sBuf + (threadIdx.x >> 5) * 2048;
    uint64_t *bar_mma = bars + 3 * group, *bar_e = bar_mma + 1;   // bar_e: one per e tile
    if (threadIdx.x < kHidden) s_b1[threadIdx.x] = a.b1[threadIdx.x];
    else if (threadIdx.x < 2 * kHidden) s_b2[threadIdx.x - kHidden] = a.b2[threadIdx.x - kHidden];
    stage_sw(sW1, a.w1e_t, kHidden, kHidden, 0, kHidden);
    stage_sw(sW2, a.w2t, kHidden, kHidden, 0, kHidden);
    cp_wait_all();
    if (tid == 0) {
        tc::mbar_init(bar_mma, 1);
        tc::mbar_init(bar_e, 1);
        tc::mbar_init(bar_e + 1, 1);
        tc::mbar_init_fence();
    }
    if (threadIdx.x < 32) {
        tc::tmem_alloc(tslot, 512);
        tc::tmem_relinquish();
    }
    tc::fence_async_smem();   // the weight tiles, complete, visible to the tensor core
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tm = *tslot;
    const uint32_t tacc = tm + 256u * group;   // accumulator, 128 columns (both products)
    const uint32_t ta = tacc + 128;            // hidden tile as the second product's A operand, 64 columns
    const uint32_t aW1 = tc::smem_u32(sW1), aW2 = tc::smem_u32(sW2);
    constexpr uint32_t id = tc::idesc_bf16(kRows, kHidden, false, false);
    const long ntiles = (a.rows + kRows - 1) / kRows, step = 2L * gridDim.x;
    auto issue_e = [&](long tile, int b) {   // the group's thread 0: the tile's two feature boxes
        unsigned char *sE = sEg + b * T;
        tc::mbar_arrive_expect(bar_e + b, T);
        tc::tma_load_2d(sE, &tm_e, 0, (int)(tile * kRows), bar_e + b);
        tc::tma_load_2d(sE + T / 2, &tm_e, 64, (int)(tile * kRows), bar_e + b);
    };
    uint32_t ph_mma = 0, ph_e = 0;
    bool ok = true, e_pending = false, mma_pending = false;   // of thread 0: not yet waited for
    const long tile0 = 2L * blockIdx.x + group;
    if (tid == 0 && tile0 < ntiles) {
        issue_e(tile0, 0);
        e_pending = true;
    }
    int b = 0, e_buf = 0;   // the e tile in work (ph_e: bit b its barrier's phase), and the one pending
    int ir = 0, ic = 0;
    if (tile0 * kRows + t < a.rows) {
        ir = a.recv[tile0 * kRows + t];
        ic = a.send[tile0 * kRows + t];
    }
    auto wait_mma = [&]() {
        const bool w = tc::mbar_wait(bar_mma, ph_mma, g_tc_wait_limit);
        const bool all = group_and(bid, w);
        if (all) {
            ph_mma ^= 1u;
            mma_pending = false;
        }
        tc::fence_after_sync();
        return all;
    };
    for (long tile = tile0; tile < ntiles; tile += step, b ^= 1) {
        const long row0 = tile * kRows, grow = row0 + t, wrow0 = row0 + (t & ~31);   // the warp's first row
        unsigned char *sE = sEg + b * T;
        const uint32_t aE = tc::smem_u32(sE);
        // the e tile; the group's barrier also orders every thread's reads of the previous tile's
        // accumulator before this tile's first product
        const bool e_ok = tc::mbar_wait(bar_e + b, (ph_e >> b) & 1u, g_tc_wait_limit);
        if (!group_and(bid, e_ok)) {
            ok = false;
            break;
        }
        ph_e ^= 1u << b;
        if (tid == 0) {
            e_pending = false;
            tc::fence_after_sync();
            for (int ks = 0; ks < kHidden / 16; ++ks)
                mma_issue(tacc, tc::sdesc_sw128(aE + (uint32_t)(ks >> 2) * (T / 2) + (uint32_t)(ks & 3) * 32u),
                          tc::kmajor_sw(aW1, kHidden, ks), id, ks > 0);
            mma_commit_issue(bar_mma);
            mma_pending = true;
            // the next tile's copy, once the previous tile's output has left that buffer
            if (tile + step < ntiles) {
                tc::bulk_wait_read();
                issue_e(tile + step, b ^ 1);
                e_pending = true;
                e_buf = b ^ 1;
            }
        }
        uint4 p[8], q[8];   // P and Q of the row while the first product runs; the next tile's indices
        {
            uint4 vp[8], vq[8];
            warp_rows_issue(a.pq + half * 64, 2 * kHidden, ir, vp);
            warp_rows_issue(a.pq + kHidden + half * 64, 2 * kHidden, ic, vq);
            const long gnext = grow + step * kRows;
            ir = gnext < a.rows ? a.recv[gnext] : 0;
            ic = gnext < a.rows ? a.send[gnext] : 0;
            warp_rows_take(buf, vp, p);
            warp_rows_take(buf, vq, q);
        }
        ok = wait_mma();
        if (!ok) break;
        uint4 hv[8];   // the thread's hidden half row
#pragma unroll
        for (int g = 0; g < 2; ++g) {   // two batches of 32 columns keep the P/Q registers live
            float w[32];
            acc32(tacc, half * 64 + g * 32, w);
            uint32_t hw[16];
#pragma unroll
            for (int c2 = 0; c2 < 2; ++c2) {
                const int cc = 2 * g + c2;
                const int c = half * 4 + cc;   // 16-feature group
                float *v = w + 16 * c2, pf[8], qf[8];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    tc::unpack8(p[2 * cc + h], pf);
                    tc::unpack8(q[2 * cc + h], qf);
                    float bias[8];
                    load8(s_b1 + c * 16 + 8 * h, bias);
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[8 * h + k] = fmaxf(v[8 * h + k] + bias[k] + pf[k] + qf[k], 0.f);
                }
                const uint4 lo = tc::pack8(v), hi = tc::pack8(v + 8);
                hw[8 * c2 + 0] = lo.x;
                hw[8 * c2 + 1] = lo.y;
                hw[8 * c2 + 2] = lo.z;
                hw[8 * c2 + 3] = lo.w;
                hw[8 * c2 + 4] = hi.x;
                hw[8 * c2 + 5] = hi.y;
                hw[8 * c2 + 6] = hi.z;
                hw[8 * c2 + 7] = hi.w;
                hv[2 * cc] = lo;
                hv[2 * cc + 1] = hi;
            }
            // features [64 half + 32 g, + 32) as 16 columns of BF16 pairs
            tc::tmem_st16(tc::tmem_warp_addr(ta, half * 32 + g * 16), hw);
        }
        tc::tmem_wait_st();
        tc::fence_before_sync();
        group_sync(bid);
        if (tid == 0) {
            tc::fence_after_sync();
            for (int ks = 0; ks < kHidden / 16; ++ks)
                mma_issue_tmem_a(tacc, ta + (uint32_t)ks * 8u, tc::kmajor_sw(aW2, kHidden, ks), id, ks > 0);
            mma_commit_issue(bar_mma);
            mma_pending = true;
        }
        // hidden rows out (training), while the second product runs
        if constexpr (SAVE_H1) warp_rows_store(buf, hv, a.h1 + half * 64, wrow0, a.rows);
        ok = wait_mma();
        if (!ok) break;
        {   // the output half row takes the place of the residual's in the e tile
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                float w[32];
                acc32(tacc, half * 64 + g * 32, w);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint4 *at = reinterpret_cast<uint4 *>(sE + tc::sw_off(kRows, t, half * 8 + g * 4 + c));
                    float *v = w + 8 * c, r[8];
                    tc::unpack8(*at, r);
                    float bias[8];
                    load8(s_b2 + half * 64 + g * 32 + 8 * c, bias);
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[k] += bias[k] + r[k];
                    *at = tc::pack8(v);
                }
            }
        }
        tc::fence_async_smem();
        tc::fence_before_sync();
        group_sync(bid);
        if (tid == 0) {
            tc::tma_store_2d(&tm_out, 0, (int)row0, sE);
            tc::tma_store_2d(&tm_out, 64, (int)row0, sE + T / 2);
            tc::bulk_commit();
        }
    }
    if (tid == 0) tc::bulk_wait();
    // a wait gave up: let the group's copy and product in flight land before the block's memory goes
    if (tid == 0 && e_pending) (void)tc::mbar_wait(bar_e + e_buf, (ph_e >> e_buf) & 1u, g_tc_wait_limit);
    if (tid == 0 && mma_pending) (void)tc::mbar_wait(bar_mma, ph_mma, g_tc_wait_limit);
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tm, 512);
    }
    if (!ok && tid == 0 && a.err) atomicOr(a.err, DEM_ERR_TIMEOUT);
}

// dW^T [256][128] partials: D_half[o][k] = sum_rows A[row][128 half + o] B[row][k]
struct LinWgradArgs {
    long rows;
    const bf16 *a;     // [rows][256]
    const bf16 *b;     // [rows][128]
    float *part;       // [gridDim.x][128][256]
    int *err;
};
constexpr uint32_t kLinwStage = kWgRows * (256 + kHidden) * 2;
constexpr int kLinwStages = 4;
constexpr size_t linw_smem() { return kLinwStages * (size_t)kLinwStage + 1024 + 64; }

// The row pipeline of k_mlp_wgrad.  One tile of 128 rows at a time, 40,000 rows took 42 us (B200),
// now 15.
__global__ void __launch_bounds__(kBwdThreads, 1) k_linear_wgrad(LinWgradArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char *smem = align1024(smem_raw);
    constexpr int NS = kLinwStages, R = kWgRows;
    constexpr uint32_t SB = kLinwStage, OB = R * 256 * 2;    // A rows, then B rows
    uint64_t *mbar = reinterpret_cast<uint64_t *>(smem + (size_t)NS * SB);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(mbar + NS);
    const int tid = threadIdx.x;
    if (tid > 0 && tid < NS) tc::mbar_init(mbar + tid, 1);
    const uint32_t tm = tc_setup(mbar, tslot, 256);
    constexpr uint32_t id = tc::idesc_bf16(kRows, kHidden, true, true);
    const long ntiles = (a.rows + kRows - 1) / kRows;
    const long units = 2 * ((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x);   // the grid has no more CTAs than tiles
    auto fill = [&](long u) {
        unsigned char *s = smem + (size_t)(u % NS) * SB;
        const long row0 = (blockIdx.x + (u >> 1) * gridDim.x) * kRows + (u & 1) * R;
        stage_sw(s, a.a, R, 256, row0, a.rows);
        stage_sw(s + OB, a.b, R, kHidden, row0, a.rows);
    };
    bool ok = true;
    long u = 0;
    for (; u < NS - 1; ++u) {
        if (u < units) fill(u);
        cp_commit();
    }
    for (u = 0; u < units; ++u) {
        cp_wait<NS - 2>();
        tc::fence_async_smem();
        tc::fence_before_sync();
        ok = __syncthreads_and(ok) != 0;
        if (!ok) break;
        if (tid == 0) {
            tc::fence_after_sync();
            const uint32_t aA = tc::smem_u32(smem + (size_t)(u % NS) * SB), aB = aA + OB;
            for (int h = 0; h < 2; ++h)
                for (int ks = 0; ks < R / 16; ++ks)
                    mma_issue(tm + h * kHidden, tc::mnmajor_sw(aA + (uint32_t)(h * kHidden * R * 2), R, ks),
                                 tc::mnmajor_sw(aB, R, ks), id, (u > 0 || ks > 0) ? 1u : 0u);
            mma_commit_issue(mbar + u % NS);
        }
        if (u > 0) ok = tc::mbar_wait(mbar + (u - 1) % NS, (uint32_t)((u - 1) / NS) & 1u, g_tc_wait_limit);
        if (u + NS - 1 < units) fill(u + NS - 1);
        cp_commit();
    }
    cp_wait_all();
    if (u > 0) ok = tc::mbar_wait(mbar + (u - 1) % NS, (uint32_t)((u - 1) / NS) & 1u, g_tc_wait_limit) && ok;
    ok = __syncthreads_and(ok) != 0;
    float *part = a.part + (long)blockIdx.x * kRows * 256;
    const int t = tid & (kRows - 1), lane = tid & 31;
    if (ok) {
        tc::fence_after_sync();
        float4 *buf = reinterpret_cast<float4 *>(smem + (tid >> 5) * 2048);   // as in k_mlp_wgrad
        for (int c = tid >> 7; c < 256 / 16; c += 4) {
            float v[16];
            acc16(tm, c * 16, v);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                buf[lane * 4 + ((k + (lane >> 1)) & 3)] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int r = 8 * k + (lane >> 2), f = lane & 3;
                *reinterpret_cast<float4 *>(part + (long)((t & ~31) + r) * 256 + c * 16 + f * 4) = buf[r * 4 + ((f + (r >> 1)) & 3)];
            }
            __syncwarp();
        }
    } else {
        for (int c = tid; c < kRows * 256; c += kBwdThreads) part[c] = 0.f;
    }
    tc::fence_before_sync();
    __syncthreads();
    if (tid < 32) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tm, 256);
    }
    if (!ok && tid == 0 && a.err) atomicOr(a.err, DEM_ERR_TIMEOUT);
}

// g[o * ld + col0 + c] += sum over blocks of part[b][o][c]   (o < 128, c < 256)
__global__ void k_linw_reduce(const float *part, int nblocks, float *g, int ld, int col0) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < kRows * 256; e += gridDim.x * blockDim.x) {
        const int o = e / 256, c = e % 256;
        g[(long)o * ld + col0 + c] += sum_blocks(part + (long)o * 256 + c, kRows * 256L, nblocks);
    }
}

template <typename K, typename A>
int launch_tc(K kernel, size_t smem, int tmem_cols, long rows, A args, cudaStream_t s, int max_blocks, int threads) {
    if (rows <= 0) return DEM_OK;
    const size_t floor_bytes = tmem_cols >= 512 ? 116 * 1024 : (tmem_cols >= 256 ? 80 * 1024 : 0);
    if (smem < floor_bytes) smem = floor_bytes;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return DEM_ERR_CUDA;
    const long ntiles = (rows + kRows - 1) / kRows;
    if (max_blocks <= 0) {   // as many CTAs as the SMs hold (shared memory and TMEM), persistent
        cudaFuncAttributes fa{};
        if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) return DEM_ERR_CUDA;
        const size_t per = smem + fa.sharedSizeBytes + 1024;
        int fit = (int)((228 * 1024) / per);
        fit = fit < 512 / tmem_cols ? fit : 512 / tmem_cols;
        max_blocks = 148 * (fit > 0 ? fit : 1);
    }
    const int grid = (int)(ntiles < max_blocks ? ntiles : max_blocks);
    kernel<<<grid, threads, smem, s>>>(args);
    return cudaGetLastError() == cudaSuccess ? DEM_OK : DEM_ERR_CUDA;
}

}  // namespace

// ---- dispatch over the (KIN, NOUT) shapes the surrogate uses ----
#define B200_NN_SHAPES(X) X(16, 128) X(128, 128) X(256, 128) X(384, 128) X(128, 16)

int nn_mlp_forward(const dem_nn_mlp &m, long rows, const dem_nn_rows *src, int nsrc, const void *resid, void *out,
                   float *out_f32, void *h1, int *err, cudaStream_t s) {
    FwdArgs a{};
    a.rows = rows;
    a.nsrc = nsrc;
    int kin = 0;
    for (int k = 0; k < nsrc && k < 3; ++k) {
        a.src[k] = RowSrc{(const bf16 *)src[k].data, src[k].index, src[k].width};
        kin += src[k].width;
    }
    if (kin != m.kin) return DEM_ERR_INVALID;
    a.w = MlpW{(const bf16 *)m.w1t, (const bf16 *)m.w1, (const bf16 *)m.w2t, (const bf16 *)m.w2, m.b1, m.b2};
    a.resid = (const bf16 *)resid;
    a.resid_src0 = (resid && resid == src[0].data && !src[0].index && src[0].width == m.nout) ? 1 : 0;
    a.out = (bf16 *)out;
    a.out_f32 = out_f32;
    a.h1 = (bf16 *)h1;
    a.err = err;
#define X(KI, NO) \
    if (m.kin == KI && m.nout == NO)                                                                        \
        return launch_tc(k_mlp_fwd<KI, NO>, fwd_smem<KI, NO>(), 128, rows, a, s, 0, fwd_threads<KI>());
    B200_NN_SHAPES(X)
#undef X
    return DEM_ERR_UNSUPPORTED;
}

int nn_mlp_backward(const dem_nn_mlp &m, long rows, const dem_nn_rows *src, int nsrc, const void *dy, const void *h1,
                    void *dz1, float *dx, float *g_w1t, int ld_w1, float *g_b1, float *g_w2t, float *g_b2,
                    float *part, int *err, cudaStream_t s, const DxSum *sum) {
    BwdArgs b{};
    if (sum) b.sum = *sum;
    b.rows = rows;
    b.w = MlpW{(const bf16 *)m.w1t, (const bf16 *)m.w1, (const bf16 *)m.w2t, (const bf16 *)m.w2, m.b1, m.b2};
    b.dy = (const bf16 *)dy;
    b.h1 = (const bf16 *)h1;
    b.dz1 = (bf16 *)dz1;
    b.dx = dx;
    b.err = err;
    WgradArgs g{};
    g.rows = rows;
    g.nsrc = nsrc;
    int kin = 0;
    for (int k = 0; k < nsrc && k < 3; ++k) {
        g.src[k] = RowSrc{(const bf16 *)src[k].data, src[k].index, src[k].width};
        kin += src[k].width;
    }
    if (kin != m.kin) return DEM_ERR_INVALID;
    g.dz1 = (const bf16 *)dz1;
    g.h1 = (const bf16 *)h1;
    g.dy = (const bf16 *)dy;
    g.part = part;
    g.err = err;
    const long ntiles = (rows + kRows - 1) / kRows;
    const int nblocks = (int)(ntiles < 148 ? ntiles : 148);
    int st = DEM_ERR_UNSUPPORTED;
#define X(KI, NO)                                                                             \
    if (m.kin == KI && m.nout == NO) {                                                        \
        if (KI == kHidden && NO == kHidden && sum)                                            \
            st = launch_tc(k_mlp_bwd<kHidden, kHidden, true>, bwd_smem<KI, NO>(), 512, rows, b, s, 148, kBwdThreads); \
        else if (!sum)                                                                        \
            st = launch_tc(k_mlp_bwd<KI, NO, false>, bwd_smem<KI, NO>(), 512, rows, b, s, 148, kBwdThreads);  \
        if (st == DEM_OK)                                                                     \
            st = launch_tc(k_mlp_wgrad<KI, NO>, wgrad_smem<KI, NO>(), wgrad_tmem_cols<KI, NO>(), rows, g, s, 148, kBwdThreads); \
    }
    B200_NN_SHAPES(X)
#undef X
    if (st != DEM_OK || rows <= 0) return st;
    // a thread per element: 64 blocks that looped over them took 62 us on average
    const int nc = m.kin + (m.nout == kHidden ? kHidden : m.nout) + 2;
    k_wgrad_reduce<<<(kRows * nc + 127) / 128, 128, 0, s>>>(part, nblocks, m.kin, m.nout, g_w1t, ld_w1, g_b1, g_w2t, g_b2);
    return cudaGetLastError() == cudaSuccess ? DEM_OK : DEM_ERR_CUDA;
}

// PQ[rows][256] = h W1ij^T (W1ij^T: [256][128]).
int nn_linear_pq(long rows, const void *h, const void *w1ij_t, void *pq, int *err, cudaStream_t s) {
    LinArgs a{rows, (const bf16 *)h, (const bf16 *)w1ij_t, (bf16 *)pq, nullptr, err};
    return launch_tc(k_linear<128, 256>, lin_smem<128, 256>(), 256, rows, a, s, 0, kLinThreads);
}

// dh[rows][128] += dPQ W1ij (dPQ: [rows][256] bf16, W1ij: [128][256]).
int nn_linear_pq_backward(long rows, const void *dpq, const void *w1ij, float *dh, int *err, cudaStream_t s) {
    LinArgs a{rows, (const bf16 *)dpq, (const bf16 *)w1ij, nullptr, dh, err};
    return launch_tc(k_linear<256, 128>, lin_smem<256, 128>(), 128, rows, a, s, 0, kLinThreads);
}

// g_w1t[o][col0 + c] += sum_rows dPQ[row][c'] h[row][k] arranged as dW1ij^T (ld = row stride).
int nn_linear_pq_wgrad(long rows, const void *dpq, const void *h, float *g_w1t, int ld, int col0, float *part,
                       int *err, cudaStream_t s) {
    if (rows <= 0) return DEM_OK;
    LinWgradArgs a{rows, (const bf16 *)dpq, (const bf16 *)h, part, err};
    const int st = launch_tc(k_linear_wgrad, linw_smem(), 256, rows, a, s, 148, kBwdThreads);
    if (st) return st;
    const long ntiles = (rows + kRows - 1) / kRows;
    k_linw_reduce<<<kRows * 256 / 128, 128, 0, s>>>(part, (int)(ntiles < 148 ? ntiles : 148), g_w1t, ld, col0);
    return cudaGetLastError() == cudaSuccess ? DEM_OK : DEM_ERR_CUDA;
}

namespace {
// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against the driver
// library); null when the driver does not provide it.
using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled() {
    static EncodeTiled fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return (EncodeTiled) nullptr;
        return reinterpret_cast<EncodeTiled>(p);
    }();
    return fn;
}

// Tensor map of e [rows][128] BF16 with 64 x 128 boxes in the 128-byte swizzle layout.
bool edge_map(CUtensorMap *m, const void *e, long rows) {
    const EncodeTiled enc = encode_tiled();
    if (!enc || (reinterpret_cast<uintptr_t>(e) & 15u) || rows <= 0 || rows > 0x7FFFFFFFL - kRows) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)kHidden, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)kHidden * 2};
    const cuuint32_t box[2] = {64u, (cuuint32_t)kRows};
    const cuuint32_t elem[2] = {1u, 1u};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(e), dims, strides, box, elem,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace

// form 0: the tensor-copy kernel (k_edge_fwd_tma) where the tensor map can be made, else the
// staged kernel; form 1: the staged kernel (k_edge_fwd); -1: the build's default
// (EDGE_FORM_DEFAULT).  Same results.
#ifndef EDGE_FORM_DEFAULT
#define EDGE_FORM_DEFAULT 0
#endif
int nn_edge_forward(long rows, const void *e, const void *pq, const int *recv, const int *send, const void *w1e_t,
                    const float *b1, const void *w2t, const float *b2, void *out, void *h1, int *err, cudaStream_t s,
                    int form) {
    EdgeArgs a{rows, (const bf16 *)e, (const bf16 *)pq, recv, send, (const bf16 *)w1e_t, b1, (const bf16 *)w2t, b2,
               (bf16 *)out, (bf16 *)h1, err};
    if (rows <= 0) return DEM_OK;
    if (form < 0) form = EDGE_FORM_DEFAULT;
    CUtensorMap m, mo;
    if (form == 0 && edge_map(&m, e, rows) && edge_map(&mo, out, rows)) {
        const size_t smem = edge_tma_smem();
        const auto kernel = h1 ? k_edge_fwd_tma<true> : k_edge_fwd_tma<false>;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
            return DEM_ERR_CUDA;
        int sms = 148, dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const long pairs = ((rows + kRows - 1) / kRows + 1) / 2, cap = sms > 0 ? sms : 148;   // a CTA steps two tiles
        kernel<<<(int)(pairs < cap ? pairs : cap), kEdgeThreads, smem, s>>>(m, mo, a);
        return cudaGetLastError() == cudaSuccess ? DEM_OK : DEM_ERR_CUDA;
    }
    return launch_tc(k_edge_fwd, edge_smem(), 128, rows, a, s, 0, kFwdThreads);
}

long nn_linear_wgrad_scratch() { return 148L * kRows * 256; }

// Scratch floats the per-CTA weight-gradient partials of one backward call need.
int nn_debug_waits(int poll_limit, int drop_mma, cudaStream_t s) {
    const int lim = poll_limit > 0 ? poll_limit : (1 << 22);
    const int drop = drop_mma ? 1 : 0;
    if (cudaMemcpyToSymbolAsync(g_tc_wait_limit, &lim, sizeof(int), 0, cudaMemcpyHostToDevice, s) != cudaSuccess ||
        cudaMemcpyToSymbolAsync(g_tc_drop_mma, &drop, sizeof(int), 0, cudaMemcpyHostToDevice, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return DEM_ERR_CUDA;
    return DEM_OK;
}

long nn_wgrad_scratch(int kin, int nout) {
    const int nw2 = nout == kHidden ? kHidden : nout;
    return 148L * kRows * (kin + nw2 + 2);
}

}  // namespace b200dem
