// Verification: for every candidate user of a query, count the facilities
// strictly nearer than the query facility q and keep the user when the count
// is below k (rknn-inf-gpu/inf_kernel.cu:41-66 counts bisector violations per
// user; rknn-rt/rt.cu:95-111 counts half-plane hits and stops at k).
//
// Stage 1 (half-plane filter).  A user is tested against the zone's
// bisectors written as exact half-planes relative to q,
//     m_f(u) = a (ux-qx) + b (uy-qy) + c = d2(u,f) - d2(u,q),
// two FMAs per (user, half-plane).  m_f(u) < -bound certifies that f is
// strictly nearer; k certified half-planes reject the user.  The bound
//     8u (2F'(|x'|+|y'|) + F'^2),  F' = max |f - q| over the bisectors,
// exceeds the float (or double) evaluation error of m_f (at most
// 4.01u(|a x'| + |b y'| + |c|)).  Lanes own users (coalesced float2 loads,
// four per lane); the warp leaves the half-plane loop as soon as every lane
// has k certified violations for all its users (__all_sync).  Where it is
// cheaper (boxes_first), and in FP64 always, the users' bounding boxes are tested
// first (verify_box.cuh).
//
// Stage 2 (exact count).  Users that survive stage 1 go to a survivor list,
// and recount_kernel counts each one exactly, a warp (or a group of up to
// eight warps, when warps outnumber survivors) per survivor: the facility
// cells covering the disc of radius d(u,q) around u, row by row (one
// contiguous range of the cell-sorted facility array per row, trimmed to the
// disc's chord), 32 facilities a round, counting d2(u,f) < d2(u,q) and
// stopping at k.  Each comparison is decided in float (or double) with its
// error bound, and the undecided ones by the exact expansion predicate.
// Accepted users are appended to their query's result region.  When the
// survivor list is full, the warp counts its own survivors, one lane per
// facility.  The item code itself lives in verify_item.cuh (the user-by-user
// form is shared with the slice filter's fused verification).
#include "verify_box.cuh"
#include <climits>

namespace rknn {

using namespace vitem;

template <int UPT, bool F64>
__device__ __forceinline__ void verify_body(const VerifyArgs& A)
{
    extern __shared__ __align__(16) char smem[];
    // every st-th work-item offset, for the item -> slot lookup
    __shared__ int csmp[VERIFY_SAMPLES];
    pdl_wait();
    pdl_trigger();
    // a fused batch with no slot left over: nothing to do here
    if (A.deflist && __ldcg(A.ndef) == 0) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // per warp (verify_warp_bytes): the boxes' scratch, seg_stage segments,
    // the slot's 32 slice bounds
    char* wsm = smem + w * verify_warp_bytes(A.stage_cap, A.seg_stage);
    const BoxScratch BS = {(uint16_t*)(wsm + BOX_STAGE_BYTES + BOX_MASK_BYTES + BOX_QBOX_BYTES), wsm,
                           (unsigned*)(wsm + BOX_STAGE_BYTES), (float4*)(wsm + BOX_STAGE_BYTES + BOX_MASK_BYTES)};
    int2* ssg = (int2*)(wsm + verify_box_bytes(A.stage_cap));
    float* sr = (float*)(ssg + A.seg_stage);
    // the listed slots: every slot, or those the fused slice filter left
    const int nl = A.deflist ? __ldcg(A.ndef) : A.nq;
    const int st = max(1, (nl + VERIFY_SAMPLES) / VERIFY_SAMPLES);       // ceil((nl + 1) / samples)
    const int nsmp = nl / st + 1;                                         // samples i * st <= nl
    if (nl > 0)
        for (int i = threadIdx.x; i < nsmp; i += blockDim.x) csmp[i] = A.chunk_off[i * st];
    __syncthreads();
    int cur = -1;
    bool seg_staged = false, boxed = false, listed = false;
    int nsp = 0;
    // per-warp statistics (32-bit here, 64-bit in the totals)
    VCount vc = {};
    const int total = nl > 0 ? A.chunk_off[nl] : 0;
    // A warp's first item is its number, counted over the blocks first so that
    // a small batch's items spread over all SMs (FP64, 1000 queries of about
    // two items: 47 -> 43 us); later items come from the counter,
    // numbered after the nwarps taken that way, and only when items
    // outnumber warps.  (Thousands of warps taking even their first item
    // from one counter queue their atomics on one address for many
    // microseconds, and a small batch's few items wait behind them.)
    const int nwarps = gridDim.x * (blockDim.x >> 5);
    int g = w * gridDim.x + blockIdx.x;
    for (bool first = true;; first = false) {
        if (!first) {
            if (total <= nwarps) break;
            int nx = 0;
            if (lane == 0) nx = nwarps + atomicAdd(A.work_counter, 1);
            g = __shfl_sync(FULL, nx, 0);
        }
        if (g >= total) break;
        // list entry e of item g: chunk_off[e] <= g < chunk_off[e+1].  The
        // samples narrow it to [ws, ws + st); there the count of offsets <= g
        // places it (offsets never decrease).
        int lo = 0, hi = nsmp;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (csmp[mid] <= g) lo = mid; else hi = mid;
        }
        int e = lo, c_off = 0;      // c_off = chunk_off[e]
        if (st > 1) {
            const int ws = lo * st, we = min(ws + st, nl);
            if (st <= 31) {
                const int j = ws + lane;
                const int co = j <= we ? A.chunk_off[VX(j, nl + 1, 215)] : INT_MAX;
                e = ws + __popc(__ballot_sync(FULL, co <= g)) - 1;
                c_off = __shfl_sync(FULL, co, e - ws);
            } else {
                int l = ws, h = we;
                while (h - l > 1) {
                    const int mid = (l + h) >> 1;
                    if (A.chunk_off[mid] <= g) l = mid; else h = mid;
                }
                e = l;
                c_off = A.chunk_off[e];
            }
        } else {
            c_off = csmp[e];
        }
        const int s = A.deflist ? A.deflist[VX(e, A.nq, 222)] : e;
        const QDesc d = A.qd[s];
        if (s != cur) {
            // the slot's segments and slice bounds, and the half-planes, each
            // lane's loads issued together: staged (the first nsp) for the
            // user-by-user test, brought to L1 (one lane a line) for the boxes
            __syncwarp();
            const float4* src = A.planes + (size_t)s * A.lc;
            const int nst = min(d.nb, A.stage_cap);
            listed = A.list_cand >= d.ncand || (!F64 && !(d.kf2 < INFINITY));
            boxed = listed || F64 || (A.box_batch ? d.ncand >= BOX_MIN_CAND : boxes_first(d.k, d.ncand));
            if (listed) {
                // no half-planes needed
            } else if (boxed) {
                if (nst > 0)
                    for (int m = 8 * lane; m < nst + 7; m += 8 * 32) prefetch_l1(src + min(m, nst - 1));
            } else {
                nsp = min(nst, (int)(verify_box_bytes(A.stage_cap) / sizeof(float4)) & ~1);
                for (int m0 = lane; m0 < nsp; m0 += 32 * 8) {
                    float4 p[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int m = m0 + 32 * j;
                        p[j] = m < nsp ? src[m] : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int m = m0 + 32 * j;
                        if (m < nsp) ((float4*)wsm)[m] = p[j];
                    }
                }
            }
            // the slot's segments (nseg ranges and the terminal entry), when
            // they fit; the record has arrived with the half-planes in flight
            const int2* gsg = A.segs + (size_t)s * A.seg_cap;
            seg_staged = d.nseg + 1 <= A.seg_stage;
            const int nss = seg_staged ? d.nseg + 1 : 0;
            for (int m0 = lane; m0 < nss; m0 += 32 * 8) {
                int2 e[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int m = m0 + 32 * j;
                    e[j] = m < nss ? gsg[m] : make_int2(0, 0);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (m0 + 32 * j < nss) ssg[m0 + 32 * j] = e[j];
            }
            if (A.slice_r) sr[lane] = A.slice_r[(size_t)s * 32 + lane];
            cur = s;
            __syncwarp();
        }
        const int2* sg = seg_staged ? ssg : A.segs + (size_t)s * A.seg_cap;
        const int nbs = min(d.nb, A.stage_cap);
        const float4* gp = A.planes + (size_t)s * A.lc;
        const float rho2 = item_rho2(d, nbs);
        // a work item is A.parts parts of 32 UPT users
        const int vbeg = (g - c_off) * (32 * UPT * A.parts), vend = min(vbeg + 32 * UPT * A.parts, d.ncand);
        for (int v0 = vbeg; v0 < vend; v0 += 32 * UPT) {
            if (!boxed) {
                if constexpr (!F64) verify_item<UPT, true>(A, d, s, v0, wsm, nsp, gp, sg, sr, nbs, -1, -1, vc);
                continue;
            }
            int pos[UPT];
            float2 u[UPT];
            bool valid[UPT], direct[UPT], surv[UPT];
            item_users<UPT>(A, d, s, v0, sg, sr, false, pos, u, valid, vc);
            if (listed) {
#pragma unroll
                for (int t = 0; t < UPT; ++t) { direct[t] = false; surv[t] = valid[t]; }
            } else
            filter_boxed<UPT, F64>(A, d, nbs, gp, A.bis_pos + (size_t)s * A.lc, BS, u, valid, direct, surv, vc.evals,
                                   rho2);
            item_emit<UPT, F64>(A, d, s, pos, direct, surv, -1, -1, vc);
        }
    }
    vc.flush(A.vstats);
}

// The verification kernel with 2, 4 or 8 users per lane per work item
// (32 * UPT users per item), for either precision mode; blocks of up to 16
// warps.  80 registers (24 warps an SM), which spill about 25 registers each
// (94 bytes of stores and 176 of loads a thread in FP32, 104 and 164 in FP64):
// FP64 needs the warps to issue beside the FP64 pipe (street layout with 126 / 80 /
// 64 registers: 2.49 / 2.27 / 2.25 ms; 1000 uniform queries: 41 / 43 / 45 us), FP32
// with 64 spills still more (1.46 -> 1.54 ms).
__global__ void __maxnreg__(80) verify_kernel(VerifyArgs a) { verify_body<4, false>(a); }
__global__ void __maxnreg__(80) verify_kernel_u2(VerifyArgs a) { verify_body<2, false>(a); }
__global__ void __launch_bounds__(512) verify_kernel_u8(VerifyArgs a) { verify_body<8, false>(a); }
__global__ void __maxnreg__(80) verify64_kernel(VerifyArgs a) { verify_body<4, true>(a); }
__global__ void __maxnreg__(80) verify64_kernel_u2(VerifyArgs a) { verify_body<2, true>(a); }
__global__ void __launch_bounds__(512) verify64_kernel_u8(VerifyArgs a) { verify_body<8, true>(a); }

// One warp per listed survivor.  Lane r computes the facility range of
// disc row r (trimmed to the chord), a warp prefix sum flattens the rows,
// and each round tests 32 facilities (__ballot_sync/__popc), stopping at k:
// the survivor costs a couple of load latencies, not one per facility.
__device__ __forceinline__ void group_barrier(int id, int nthreads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// Exact count of the facilities strictly nearer to u than q, stopping at k,
// by a group of G warps (G = 1, 2, 4, 8; gi this warp's index in it): lane r
// computes the facility range of disc row r (trimmed to the disc's chord), a
// warp prefix sum flattens the rows, and the group's warps take alternate
// rounds of 32 facilities (__ballot_sync/__popc), adding their counts to the
// group's shared counter *sc and stopping once it reaches k.  The count is
// exact below k and at least k otherwise, whatever G.  Groups of more than
// one warp synchronise on named barrier bar (G * 32 threads).
struct Counted {
    float ux, uy, qx, qy;   // the user and the query
    int qpos, k;            // the query's position among the facilities, its k
};
template <bool F64>
__device__ __forceinline__ int group_exact_count(const Counted& d, const VerifyArgs& A, int G, int gi, int bar,
                                                 int* sc, unsigned long long& fac, unsigned long long& rech)
{
    const int lane = threadIdx.x & 31;
    const float ux = d.ux, uy = d.uy, qx = d.qx, qy = d.qy;
    const float slack = 4.0f * kU32 * (fabsf(ux) + fabsf(uy) + fabsf(qx) + fabsf(qy)) + 1e-30f;
    // the disc's radius, above |u - q|
    const float ddx = ux - qx, ddy = uy - qy;
    const float Dq = fmaf(ddx, ddx, ddy * ddy);
    const float r = disc_radius(Dq, slack);
    Near64 near;
    if (F64) near = near64(ux, uy, qx, qy);
    if (G > 1) {
        if (gi == 0 && lane == 0) *sc = 0;
        group_barrier(bar, G * 32);
    }
    const Grid& g = A.gf;
    const float ym = 1e-5f * g.cs + 8.0f * kU32 * (fabsf(g.y0) + fabsf(uy) + g.cs * (float)g.gy);
    const int cy0 = cell_coord(uy - r, g.y0, g.inv, g.gy), cy1 = cell_coord(uy + r, g.y0, g.inv, g.gy);
    int cnt = 0;
    bool stop = false;
    for (int rb = cy0; rb <= cy1 && !stop; rb += 32) {
        const int cy = rb + lane;
        int f0 = 0, len = 0;
        if (cy <= cy1) {
            const float ylo = g.y0 + (float)cy * g.cs - ym, yhi = g.y0 + (float)(cy + 1) * g.cs + ym;
            const float dyn = fmaxf(fmaxf(ylo - uy, uy - yhi), 0.0f) * (1.0f - 1e-6f);
            // (r^2 - dyn^2 as a product: the squares overflow from 1.8e19 on)
            const float w = sqrtf(fmaxf((r - dyn) * (r + dyn), MIN_SQUARE)) * (1.0f + 1e-6f) + slack;
            const int cx0 = cell_coord(ux - w, g.x0, g.inv, g.gx), cx1 = cell_coord(ux + w, g.x0, g.inv, g.gx);
            f0 = A.fstart[VX(cy * g.gx + cx0, A.ncf + 1, 211)];
            len = A.fstart[VX(cy * g.gx + cx1 + 1, A.ncf + 1, 212)] - f0;
        }
        int incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += v;
        }
        const int total = __shfl_sync(FULL, incl, 31);
        for (int t0 = gi * 32; t0 < total; t0 += G * 32) {
            const int j = t0 + lane;
            int lo = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const int probe = __shfl_sync(FULL, incl, lo + step - 1);
                if (probe <= j) lo += step;
            }
            const int rs = __shfl_sync(FULL, f0, lo & 31);
            const int ri = __shfl_sync(FULL, incl, lo & 31);
            const int rl = __shfl_sync(FULL, len, lo & 31);
            const int i = rs + (j - (ri - rl));
            bool c = false;
            if (j < total && i != d.qpos) {
                const float2 f = A.fxy[VX(i, A.nf, 213)];
                c = F64 ? closer_f64(near, ux, uy, f.x, f.y, qx, qy, &rech)
                        : closer_f32(ux, uy, f.x, f.y, qx, qy, Dq, &rech);
            }
            const int pc = __popc(__ballot_sync(FULL, c));
            fac += (unsigned long long)min(32, total - t0);
            if (G == 1) {
                cnt += pc;
            } else {
                int now = 0;
                if (lane == 0) now = atomicAdd(sc, pc) + pc;
                cnt = __shfl_sync(FULL, now, 0);
            }
            if (cnt >= d.k) { stop = true; break; }
        }
    }
    if (G > 1) {
        group_barrier(bar, G * 32);
        cnt = *(volatile int*)sc;
        group_barrier(bar, G * 32);      // the counter is read before the next survivor resets it
    }
    return cnt;
}

// Exact recount of the listed survivors; accepted users are appended with
// one atomic per survivor.  A survivor gets a group of G warps of one block
// (G a power of two up to the block's warps, as large as the grid's warps
// allow for all survivors at once), which split its rounds of facilities:
// the count's latency, not its work, bounds a small batch.  sc: one shared
// counter per group.
template <bool F64>
__device__ __forceinline__ void recount_listed(const VerifyArgs& A, VCount& vc, int* sc, Counted* run_c, int2* run_e)
{
    const int lane = threadIdx.x & 31;
    const int n = min(*A.surv_count, A.surv_cap);
    unsigned long long s_fac = 0, s_rech = 0, s_res = 0;
    const int wpb = blockDim.x >> 5, w = threadIdx.x >> 5;
    const int nw = gridDim.x * wpb;
    int G = 1;
    while (2 * G <= wpb && (long long)n * 2 * G <= nw) G *= 2;
    const int gi = w % G, gid = w / G, gpb = wpb / G;
    // more survivors than warps: each warp takes a run of them, its first run
    // by its number and later ones from a queue (a survivor far from every
    // facility walks a large disc, so shares fixed beforehand end unevenly);
    // short runs where survivors are few, up to 32 where the queue's counter
    // would be the bound: about three runs a warp in FP32, eight in FP64, whose
    // counts are longer (zone batches of 50 k / 100 k / 250 k survivors, us, with
    // eight / four / three / two: FP32 57 / 47 / 45 / 45, 70 / 61 / 61 / 64, 127 /
    // 119 / 123 / 135, FP64 70 / 65 / 64 / 68, 115 / 111 / 119 / 127, 283 / 297 /
    // 307 / 324; fixed shares took 43, 66 and 131 in FP32).  Survivors of one
    // query are neighbours in the list and alike, so a run takes every nruns-th.
    // A run's records are loaded by its lanes at once and kept in shared memory,
    // where the count's registers leave room for more warps.  Clustered workload,
    // 209 k survivors (eight runs a warp): 0.64 ms with fixed shares, 0.51 with
    // runs of neighbours, 0.46 so.
    const int run = G == 1 ? max(1, min(32, n / ((F64 ? 8 : 3) * nw))) : 1;
    const int nruns = (n + run - 1) / run;
    const int ngroups = gridDim.x * gpb;
    int r = blockIdx.x * gpb + gid;
    while (r < nruns) {
        const int m = (n - 1 - r) / nruns + 1;
        __syncwarp();                    // the last run's records have been read
        if (lane < m) {
            const int2 e = A.surv[VX(r + lane * nruns, A.surv_cap, 215)];
            Counted c = {};
            if (e.x >= 0) {
                const QDesc* d = A.qd + e.x;
                const float2 u = A.uxy[VX(e.y, A.nu, 216)];
                c = {u.x, u.y, d->qx, d->qy, d->qpos, d->k};
            }
            run_c[lane] = c;
            run_e[lane] = e;
        }
        __syncwarp();
        for (int j = 0; j < m; ++j) {
            const int slot = run_e[j].x, pos = run_e[j].y;
            if (slot < 0) continue;      // the group's warps skip it alike
            const Counted c = run_c[j];
            const int cnt = group_exact_count<F64>(c, A, G, gi, 1 + gid, sc + gid, s_fac, s_rech);
            if (cnt < c.k && gi == 0 && lane == 0) {
                const int at = atomicAdd(A.res_count + slot, 1);
                const long long r0 = A.cand_off[slot], region = A.reg_len[slot];
                if (at < region) A.res_pool[VX(r0 + at, A.pool_cap, 217)] = A.uid[VX(pos, A.nu, 218)];
                else atomicOr(A.dropped, 1);
                s_res += 1;
            }
        }
        if (nruns <= ngroups) break;
        if (!F64 && A.alike && n < 6 * nw) {
            // a few alike survivors a warp: fixed shares (zone batches of 24 k
            // survivors 45 -> 35 us, of 19 k 36 -> 33: an atomic each on one counter
            // takes longer than the shares differ).  Those of slice batches are
            // the odd ones (clustered ties, k=1: 118 us from the queue, 130 so)
            r += ngroups;
            continue;
        }
        if (lane == 0) r = ngroups + atomicAdd(A.recount_counter, 1);
        r = __shfl_sync(FULL, r, 0);
    }
    vc.fac += (unsigned)s_fac;
    vc.rech += (unsigned)s_rech;
    vc.res += (unsigned)s_res;
}

template <bool F64>
__device__ __forceinline__ void recount_body(const VerifyArgs& A)
{
    pdl_wait();
    pdl_trigger();
    __shared__ int sc[8];
    __shared__ Counted run_c[8][32];
    __shared__ int2 run_e[8][32];
    VCount vc = {};
    recount_listed<F64>(A, vc, sc, run_c[threadIdx.x >> 5], run_e[threadIdx.x >> 5]);
    vc.flush(A.vstats);
}

// FP32 with four blocks an SM (64 registers, spills in the exact predicate's
// rare call), FP64 with three (79): FP32 waits for its loads, FP64 for its pipe.
// ms, four / three blocks: FP32 uniform k=500, 400 queries 2.50 / 3.15, street
// zones k=25, 1000 queries 1.00 / 1.26; FP64 the same 2.72 / 2.72 (a grid of four
// blocks an SM over three resident ones: 2.74, and 4 us more on small batches).
__global__ void __launch_bounds__(256, 4) recount_kernel(VerifyArgs A) { recount_body<false>(A); }
__global__ void __launch_bounds__(256) recount64_kernel(VerifyArgs A) { recount_body<true>(A); }

// ---------------------------------------------------------------- scans
// Scans over the batch's slots: SCAN_THREADS slots a block, one a thread.  A
// block sums the values of every slot before its own itself (coalesced, from
// L2), so no block waits for another.  One block that walked all slots in
// tiles took 31 us (plan) and 16 to 25 us (offsets) for 16,384 slots, against
// 11 and 8 us so.
namespace {
// Sum of v over the block, in every thread (one barrier before, one after).
template <typename T>
__device__ __forceinline__ T block_sum(T v, T* tmp)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    if (lane == 0) tmp[w] = v;
    __syncthreads();
    T r = tmp[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(FULL, r, o);
    __syncthreads();
    return r;
}
}  // namespace

// Result region of each slot: min(candidates, rcap) entries, at 64-bit
// offsets; slots whose region does not fit the pool are flagged and skipped
// (the host grows the pool and runs the batch again).  Work items of chunk
// users cover every candidate of the slots that fit.
__global__ void __launch_bounds__(SCAN_THREADS)
plan_kernel(QDesc* qd, const int* ncand, int nq, long long* cand_off, int* reg_len, long long* region_top,
            int* chunk_off, long long pool_cap, int rcap, int chunk)
{
    pdl_wait();
    pdl_trigger();
    __shared__ long long tmp64[32];
    __shared__ int tmp[32];
    const int tid = threadIdx.x, first = blockIdx.x * SCAN_THREADS;
    const int n = first + tid < nq ? ncand[first + tid] : 0;
    long long before = 0;
    int items = 0;
    if (first > 0) {
        for (int i0 = tid; i0 < first; i0 += 4 * SCAN_THREADS) {
            int v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = i0 + j * SCAN_THREADS < first ? ncand[i0 + j * SCAN_THREADS] : 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                before += min(v[j], rcap);
                items += (v[j] + chunk - 1) / chunk;
            }
        }
        before = block_sum<long long>(before, tmp64);
        items = block_sum<int>(items, tmp);
    }
    const int r = min(n, rcap);
    long long tot64 = 0;
    const long long off = before + block_scan_excl<long long>(r, tmp64, &tot64);
    if (before + tot64 > pool_cap) {
        // the pool ends in or before this block's slots: the items of those
        // that fit, tile by tile (the batch runs again)
        items = 0;
        long long at = 0;
        for (int t0 = 0; t0 < first; t0 += SCAN_THREADS) {
            const int m = ncand[t0 + tid], rm = min(m, rcap);
            long long t64 = 0;
            const bool ok = at + block_scan_excl<long long>(rm, tmp64, &t64) + rm <= pool_cap;
            items += block_sum<int>(ok ? (m + chunk - 1) / chunk : 0, tmp);
            at += t64;
        }
    }
    const bool fits = off + r <= pool_cap;
    int tot = 0;
    const int coff = items + block_scan_excl<int>(fits ? (n + chunk - 1) / chunk : 0, tmp, &tot);
    const int i = first + tid;
    if (i < nq) {
        cand_off[i] = off;
        reg_len[i] = r;
        chunk_off[i] = coff;
        if (!fits) qd[i].flags |= QF_RESULT_OVERFLOW;
    }
    if (blockIdx.x == gridDim.x - 1 && tid == 0) {
        *region_top = before + tot64;
        chunk_off[nq] = items + tot;
    }
}

// Output offsets of the stored results (a slot stores at most its region),
// then the total and the run's flags.
__global__ void __launch_bounds__(SCAN_THREADS)
scan_counts_kernel(const int* res_count, const int* reg_len, const long long* region_top, int nq, int* out_off,
                   const int* counters, int* out_off_host)
{
    pdl_wait();
    pdl_trigger();
    __shared__ int tmp[32];
    const int tid = threadIdx.x, first = blockIdx.x * SCAN_THREADS, i = first + tid;
    const int n = i < nq ? min(res_count[i], reg_len[i]) : 0;
    int before = 0;
    if (first > 0) {
        for (int i0 = tid; i0 < first; i0 += 4 * SCAN_THREADS) {
            int v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int e = i0 + j * SCAN_THREADS;
                v[j] = e < first ? min(res_count[e], reg_len[e]) : 0;
            }
            before += v[0] + v[1] + v[2] + v[3];
        }
        before = block_sum<int>(before, tmp);
    }
    int tot = 0;
    const int off = before + block_scan_excl<int>(n, tmp, &tot);
    if (i < nq) {
        out_off[i] = off;
        if (out_off_host) out_off_host[i] = off;
    }
    if (blockIdx.x == gridDim.x - 1 && tid <= OFF_TAIL) {
        const unsigned long long rt = (unsigned long long)*region_top;
        const int tail[1 + OFF_TAIL] = {before + tot, (int)(unsigned)(rt & 0xffffffffu), (int)(unsigned)(rt >> 32),
                                        counters[2], counters[3]};
        out_off[nq + tid] = tail[tid];
        if (out_off_host) out_off_host[nq + tid] = tail[tid];
    }
}

// ---------------------------------------------------------------- finalize
namespace {
__device__ __forceinline__ unsigned okey(int v) { return (unsigned)v ^ 0x80000000u; }

// LSD radix sort of one slot's ids by its warp: 8-bit digits over the bits
// in which the keys differ (key - min), stable passes of 32 keys at a time
// in order, ping-ponging between the slot's pool region (scratch by now)
// and its range of the device staging array tmp; bins: the warp's 256 shared
// counters.  Work linear in n (about three passes for ids below 2^24), where
// a bitonic network pads to a power of two and takes log^2 steps.
// The passes scatter single words and read them back, so they stay in device
// memory: through an output in page-locked host memory each pass crosses the
// CPU link word by word (35 M ids of the street workload: finalize 22.3 ms,
// against 1.6 ms staged, where only the sorted ids cross, whole 128-byte
// lines at a time).  out may be tmp's range itself.
__device__ void warp_radix_slot(unsigned* src, unsigned* tmp, unsigned* out, int n, int lane, unsigned* bins)
{
    unsigned mn = 0xffffffffu, mx = 0u;
    for (int i = lane; i < n; i += 32) {
        const unsigned k = okey((int)src[i]);
        src[i] = k;
        mn = min(mn, k);
        mx = max(mx, k);
    }
    mn = __reduce_min_sync(FULL, mn);
    mx = __reduce_max_sync(FULL, mx);
    const unsigned span = mx - mn;
    const int passes = span ? (32 - __clz((int)span) + 7) / 8 : 0;
    unsigned* a = src;
    unsigned* b = tmp;
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p;
        for (int j = lane; j < 256; j += 32) bins[j] = 0u;
        __syncwarp();
        for (int i = lane; i < n; i += 32) atomicAdd(&bins[((a[i] - mn) >> shift) & 255u], 1u);
        __syncwarp();
        // exclusive scan of the bins: lane l owns bins 8l .. 8l + 7
        unsigned v[8], sum = 0u;
#pragma unroll
        for (int j = 0; j < 8; ++j) { v[j] = bins[8 * lane + j]; sum += v[j]; }
        unsigned incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
        }
        unsigned run = incl - sum;
#pragma unroll
        for (int j = 0; j < 8; ++j) { bins[8 * lane + j] = run; run += v[j]; }
        __syncwarp();
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            const bool ok = i < n;
            const unsigned key = ok ? a[i] : 0u;
            const unsigned d = ok ? ((key - mn) >> shift) & 255u : 256u + (unsigned)lane;   // idle lanes: own groups
            const unsigned mm = __match_any_sync(FULL, d);
            const unsigned base = ok ? bins[d] : 0u;
            __syncwarp();
            if (ok) {
                b[base + __popc(mm & ((1u << lane) - 1))] = key;
                if ((mm >> lane) == 1u) bins[d] = base + __popc(mm);   // the group's last lane moves the bin on
            }
            __syncwarp();
        }
        unsigned* t = a;
        a = b;
        b = t;
    }
    // a is src or tmp, element for element; the warp's stores start on out's
    // 128-byte lines
    const int lead = (int)(((unsigned long long)out >> 2) & 31ull);
    for (int i = lane - lead; i < n; i += 32)
        if (i >= 0) out[i] = a[i] ^ 0x80000000u;
}
}  // namespace

namespace {
// Ascending bitonic sort of 32*E keys held by one warp in registers, key
// t*32 + lane in x[t] (coalesced loads and stores).  Pairs 32 or more apart
// sit in one lane's registers; nearer pairs are exchanged by shuffles.
template <int E>
__device__ __forceinline__ void warp_sort_regs(unsigned (&x)[E], int lane)
{
#pragma unroll
    for (int kk = 2; kk <= 32 * E; kk <<= 1) {
#pragma unroll
        for (int j = kk >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
                const int tj = j >> 5;
#pragma unroll
                for (int t = 0; t < E; ++t) {
                    if ((t & tj) == 0) {
                        const bool up = (((t << 5) | lane) & kk) == 0;
                        const unsigned a = x[t], b = x[t | tj];
                        x[t] = up ? min(a, b) : max(a, b);
                        x[t | tj] = up ? max(a, b) : min(a, b);
                    }
                }
            } else {
                const bool lower = (lane & j) == 0;
#pragma unroll
                for (int t = 0; t < E; ++t) {
                    const unsigned o = __shfl_xor_sync(FULL, x[t], j);
                    const bool up = (((t << 5) | lane) & kk) == 0;
                    x[t] = (lower == up) ? min(x[t], o) : max(x[t], o);
                }
            }
        }
    }
}

template <int E, bool TWIN>
__device__ __forceinline__ void warp_sort_slot(const unsigned* src, unsigned* dst, unsigned* twin, int n, int lane)
{
    unsigned x[E];
#pragma unroll
    for (int t = 0; t < E; ++t) {
        const int i = (t << 5) | lane;
        x[t] = i < n ? okey((int)src[i]) : 0xffffffffu;
    }
    warp_sort_regs<E>(x, lane);
#pragma unroll
    for (int t = 0; t < E; ++t) {
        const int i = (t << 5) | lane;
        if (i < n) {
            dst[i] = x[t] ^ 0x80000000u;
            if (TWIN && twin) twin[i] = x[t] ^ 0x80000000u;
        }
    }
}
}  // namespace

// One warp per slot sorts the slot's stored ids into its output range: up to
// 32 ids by rank counting in registers, up to FIN_WCAP by a bitonic network
// in registers; larger sets are listed for sort_large_kernel where the batch
// launches it, else radix sorted through the slot's pool region.
template <bool TWIN>
__device__ __forceinline__ void finalize_body(int* res_pool, const long long* cand_off, const int* reg_len,
                                              const int* res_count, int* out_off, int* out, int* stage, int nq,
                                              long long out_cap, int* zero, long long zero_n, const FinScan& S)
{
    // the next batch's counters (no kernel of this batch uses them), while
    // the predecessor drains
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < zero_n;
         i += (long long)gridDim.x * blockDim.x)
        zero[i] = 0;
    pdl_wait();
    __shared__ unsigned bins[FIN_WARPS][256];
    __shared__ int s_part[FIN_WARPS];
    __shared__ int s_off[FIN_WARPS];      // this block's slots' output offsets
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int first = blockIdx.x * FIN_WARPS;
    if (S.on) {
        // stored ids of the slots before this block's (four loads in flight
        // per thread)
        int part = 0;
        for (int i0 = tid; i0 < first; i0 += 4 * (int)blockDim.x) {
            int v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = i0 + j * (int)blockDim.x;
                v[j] = i < first ? min(res_count[i], reg_len[i]) : 0;
            }
            part += v[0] + v[1] + v[2] + v[3];
        }
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(FULL, part, o);
        if (lane == 0) s_part[w] = part;
        __syncthreads();
        if (w == 0) {
            int base = lane < FIN_WARPS ? s_part[lane] : 0;
            for (int o = 16; o > 0; o >>= 1) base += __shfl_xor_sync(FULL, base, o);
            const int sj = first + lane;
            const int nj = (lane < FIN_WARPS && sj < nq) ? min(res_count[sj], reg_len[sj]) : 0;
            int incl = nj;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += y;
            }
            const int excl = base + incl - nj;
            if (lane < FIN_WARPS) s_off[lane] = excl;
            if (lane < FIN_WARPS && sj < nq) {
                out_off[sj] = excl;
                if (S.out_off_host) S.out_off_host[sj] = excl;
            }
            const int total = base + __shfl_sync(FULL, incl, 31);
            if (blockIdx.x == gridDim.x - 1 && lane <= OFF_TAIL) {
                // the total and the run's flags (as scan_counts_kernel)
                const unsigned long long rt = (unsigned long long)*S.region_top;
                const int tail[1 + OFF_TAIL] = {total, (int)(unsigned)(rt & 0xffffffffu), (int)(unsigned)(rt >> 32),
                                                S.counters[2], S.counters[3]};
                out_off[nq + lane] = tail[lane];
                if (S.out_off_host) S.out_off_host[nq + lane] = tail[lane];
            }
        }
    }
    __syncthreads();
    const int s = first + w;
    if (s < nq) {
        const int n = min(res_count[s], reg_len[s]);
        const int os = S.on ? s_off[w] : out_off[s];
        unsigned* src = (unsigned*)(res_pool + cand_off[s]);
        unsigned* dst = (unsigned*)(out + os);
        unsigned* twin = TWIN && (long long)os + n <= S.twin_cap ? (unsigned*)(S.twin + os) : nullptr;
        if ((long long)os + n > out_cap) {
            // past the output's capacity: left out (the batch fails on the host)
        } else if (n <= 32) {
            // stable rank: smaller keys, and equal keys in lower lanes
            const unsigned key = lane < n ? okey((int)src[lane]) : 0xffffffffu;
            int rank = 0;
            for (int j = 0; j < 32; ++j) {
                const unsigned o = __shfl_sync(FULL, key, j);
                rank += (o < key) || (o == key && j < lane);
            }
            if (lane < n) {
                dst[rank] = key ^ 0x80000000u;
                if (TWIN && twin) twin[rank] = key ^ 0x80000000u;
            }
        } else if (n <= 64) {
            warp_sort_slot<2, TWIN>(src, dst, twin, n, lane);
        } else if (n <= 128) {
            warp_sort_slot<4, TWIN>(src, dst, twin, n, lane);
        } else if (n <= 256) {
            warp_sort_slot<8, TWIN>(src, dst, twin, n, lane);
        } else if (n <= FIN_WCAP) {
            warp_sort_slot<16, TWIN>(src, dst, twin, n, lane);
        } else if (S.large) {
            // left to sort_large_kernel
            if (lane == 0) S.large[atomicAdd(S.nlarge, 1)] = s;
        } else {
            warp_radix_slot(src, (unsigned*)(stage + os), dst, n, lane, bins[w]);
            __syncwarp();
            if (TWIN && twin)
                for (int i = lane; i < n; i += 32) twin[i] = dst[i];
        }
    }
}

__global__ void __launch_bounds__(32 * FIN_WARPS, 1)
finalize_kernel(int* res_pool, const long long* cand_off, const int* reg_len, const int* res_count,
                int* out_off, int* out, int* stage, int nq, long long out_cap, int* zero, long long zero_n, FinScan S)
{
    finalize_body<false>(res_pool, cand_off, reg_len, res_count, out_off, out, stage, nq, out_cap, zero, zero_n, S);
}
__global__ void __launch_bounds__(32 * FIN_WARPS, 1)
finalize_twin_kernel(int* res_pool, const long long* cand_off, const int* reg_len, const int* res_count,
                     int* out_off, int* out, int* stage, int nq, long long out_cap, int* zero, long long zero_n, FinScan S)
{
    finalize_body<true>(res_pool, cand_off, reg_len, res_count, out_off, out, stage, nq, out_cap, zero, zero_n, S);
}

// ------------------------------------------------------- large result sets
// Sorts one slot's n > 0 ids with a block.  A set of one tile is sorted by
// buckets in shared memory (sort_buckets).  Larger ones, and ids in narrow
// groups: LSD radix, SORT_BITS bits a pass over the bits in which the ids
// differ, in tiles of SORT_TILE ids; in a pass each thread takes SORT_PT ids at
// most (a warp's are consecutive runs of 32), ranks them within its warp's digit
// counts by ballots, and the block's scan of those counts places every id; a set
// of one tile ping-pongs between two shared-memory buffers, a larger one between
// src and tmp in device memory, its tiles in order after a histogram of the
// whole set.  The sorted ids go to out on its 128-byte lines (ids written to
// page-locked host memory from their buckets, out of line: 0.92 ms for 0.76).
//
// Why a block: a warp that sorts a set alone is a chain of dependent loads,
// votes and shared-memory updates, and the last large set that starts ends the
// batch.  Street workload, 16,384 sets, 35 M ids, finalize with a warp a set /
// radix passes / buckets: 1.42 / 0.81 / 0.76 ms into page-locked host memory,
// - / 0.78 / 0.47 into device memory.  The first is bound by the link to the
// host (140 MB at 190 GB/s, as a copy of the same bytes: 0.74 ms), the second by
// the block's barriers.
namespace {
constexpr int SORT_WARPS = SORT_THREADS / 32;
constexpr int SORT_PT = SORT_TILE / SORT_THREADS;
constexpr int SORT_DIGITS = 1 << SORT_BITS;
constexpr int SORT_BUCKET_BITS = 12, SORT_BUCKETS = 1 << SORT_BUCKET_BITS, SORT_BUCKET_MAX = 32;
static_assert(SORT_BUCKETS % SORT_THREADS == 0, "whole buckets a thread");
static_assert(SORT_THREADS >= SORT_DIGITS && SORT_DIGITS % 32 == 0, "a thread a digit in the scans");
static_assert(SORT_TILE % SORT_THREADS == 0 && SORT_TILE <= 65536, "whole rounds of ids, 16-bit counts");

struct SortShared {
    unsigned key[2][SORT_TILE];
    union {
        uint16_t cnt[SORT_WARPS][SORT_DIGITS];  // a warp's digit counts, then its first places
        unsigned bucket[SORT_BUCKETS];          // a bucket's count, then its first place
    };
    unsigned base[SORT_DIGITS];                 // tiled sets: where a digit's next id goes
    unsigned place[SORT_DIGITS];                // where the tile's first id of a digit goes
    unsigned ws[SORT_WARPS], mn, mx;
    int slot;
};

// Exclusive scan of v over the block's first SORT_DIGITS threads (the others
// pass 0); begins and ends at a barrier.
__device__ __forceinline__ unsigned sort_scan(unsigned v, SortShared& sh)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh.ws[w] = x;
    __syncthreads();
    unsigned b = 0;
#pragma unroll
    for (int j = 0; j < SORT_DIGITS / 32; ++j)
        if (j < w) b += sh.ws[j];
    __syncthreads();
    return b + x - v;
}

// Sorts a tile's ids into sh.key[0] by buckets: their range is cut into
// SORT_BUCKETS equal parts, each id goes to its part (an atomic to count it and
// one to place it, a scan between) and from there to its rank among the few in
// that part.  False, with the ids untouched, when a part holds more than
// SORT_BUCKET_MAX (ids in narrow groups): the digits' passes are left.
__device__ __forceinline__ bool sort_buckets(SortShared& sh, const int* src, unsigned mn, int bits, int n)
{
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    unsigned *at = sh.bucket, *key = sh.key[1];
    const int shift = max(0, bits - SORT_BUCKET_BITS);
    constexpr int PER = SORT_BUCKETS / SORT_THREADS;
    for (int i = tid; i < SORT_BUCKETS; i += SORT_THREADS) at[i] = 0u;
    __syncthreads();
#pragma unroll 4
    for (int i = tid; i < n; i += SORT_THREADS) atomicAdd(&at[(okey(src[i]) - mn) >> shift], 1u);
    __syncthreads();
    unsigned c[PER], sum = 0u, top = 0u;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        c[j] = at[PER * tid + j];
        sum += c[j];
        top = max(top, c[j]);
    }
    if (__syncthreads_or(top > SORT_BUCKET_MAX)) return false;
    unsigned x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh.ws[w] = x;
    __syncthreads();
    x -= sum;
#pragma unroll
    for (int j = 0; j < SORT_WARPS; ++j) x += j < w ? sh.ws[j] : 0u;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        at[PER * tid + j] = x;
        x += c[j];
    }
    __syncthreads();
#pragma unroll 4
    for (int i = tid; i < n; i += SORT_THREADS) {
        const unsigned k = okey(src[i]);
        key[atomicAdd(&at[(k - mn) >> shift], 1u)] = k;
    }
    __syncthreads();
    // at[b] is now the end of bucket b
    for (int i = tid; i < n; i += SORT_THREADS) {
        const unsigned k = key[i], b = (k - mn) >> shift;
        const int i0 = b ? (int)at[b - 1] : 0, i1 = (int)at[b];
        int r = i0;
        for (int j = i0; j < i1; ++j) {
            const unsigned o = key[j];
            r += o < k || (o == k && j < i);
        }
        sh.key[0][r] = k;
    }
    __syncthreads();
    return true;
}

__device__ __forceinline__ void sort_slot(SortShared& sh, const unsigned* src0, unsigned* tmp, unsigned* out, int n)
{
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    unsigned* src = (unsigned*)src0;
    const bool one = n <= SORT_TILE;
    // the range of the keys (unsigned, in the ids' order)
    unsigned mn = 0xffffffffu, mx = 0u;
    if (tid == 0) { sh.mn = 0xffffffffu; sh.mx = 0u; }
#pragma unroll 4
    for (int i = tid; i < n; i += SORT_THREADS) {
        const unsigned k = okey((int)src[i]);
        mn = min(mn, k);
        mx = max(mx, k);
    }
    mn = __reduce_min_sync(FULL, mn);
    mx = __reduce_max_sync(FULL, mx);
    __syncthreads();
    if (lane == 0) { atomicMin(&sh.mn, mn); atomicMax(&sh.mx, mx); }
    __syncthreads();
    mn = sh.mn;
    const unsigned span = sh.mx - mn;
    const int bits = span ? 32 - __clz((int)span) : 0;
    int passes = (bits + SORT_BITS - 1) / SORT_BITS;
    if (one && span && sort_buckets(sh, (const int*)src, mn, bits, n)) {
        passes = 0;
    } else {
        for (int i = tid; i < n; i += SORT_THREADS) {
            const unsigned k = okey((int)src[i]);
            if (one) sh.key[0][i] = k;
            else src[i] = k;
        }
        __syncthreads();
    }
    int cur = 0;                        // one tile: the buffer that holds the keys
    unsigned *a = src, *b = tmp;        // more: the arrays, a holding the keys
    for (int p = 0; p < passes; ++p) {
        const int shift = SORT_BITS * p;
        if (!one) {
            // the whole set's digit counts place its tiles
            for (int i = tid; i < SORT_DIGITS; i += SORT_THREADS) sh.base[i] = 0u;
            __syncthreads();
            for (int i = tid; i < n; i += SORT_THREADS)
                atomicAdd(&sh.base[((a[i] - mn) >> shift) & (SORT_DIGITS - 1)], 1u);
            __syncthreads();
            const unsigned e = sort_scan(tid < SORT_DIGITS ? sh.base[tid] : 0u, sh);
            if (tid < SORT_DIGITS) sh.base[tid] = e;
            __syncthreads();
        }
        for (int t0 = 0; t0 < n; t0 += SORT_TILE) {
            const int m = min(SORT_TILE, n - t0);
            for (int i = lane; i < SORT_DIGITS / 2; i += 32) ((unsigned*)sh.cnt[w])[i] = 0u;
            __syncwarp();
            unsigned key[SORT_PT];
            uint16_t rank[SORT_PT];
            const int pt = (m + SORT_THREADS - 1) / SORT_THREADS;      // ids a thread takes
            const int i0 = w * (32 * pt) + lane;
#pragma unroll
            for (int j = 0; j < SORT_PT; ++j) {
                if (j >= pt) break;
                const int i = i0 + 32 * j;
                const bool ok = i < m;
                key[j] = ok ? (one ? sh.key[cur][i] : a[t0 + i]) : 0u;
                const unsigned d = ((key[j] - mn) >> shift) & (SORT_DIGITS - 1);
                // lanes with the same digit, a ballot a bit
                unsigned mm = __ballot_sync(FULL, ok);
#pragma unroll
                for (int t = 0; t < SORT_BITS; ++t) {
                    const bool bit = (d >> t) & 1u;
                    const unsigned v = __ballot_sync(FULL, bit);
                    mm &= bit ? v : ~v;
                }
                const int r = __popc(mm & ((1u << lane) - 1));
                const int old = ok ? sh.cnt[w][d] : 0;
                __syncwarp();
                if (ok && r == 0) sh.cnt[w][d] = (uint16_t)(old + __popc(mm));
                __syncwarp();
                rank[j] = (uint16_t)(old + r);
            }
            __syncthreads();
            // a digit's ids: warp by warp, after those of smaller digits
            unsigned tot = 0;
            if (tid < SORT_DIGITS) {
#pragma unroll
                for (int j = 0; j < SORT_WARPS; ++j) {
                    const unsigned c = sh.cnt[j][tid];
                    sh.cnt[j][tid] = (uint16_t)tot;
                    tot += c;
                }
            }
            unsigned first = 0;
            if (one) {
                first = sort_scan(tot, sh);
            } else if (tid < SORT_DIGITS) {
                first = sh.base[tid];
                sh.base[tid] = first + tot;
            }
            if (tid < SORT_DIGITS) sh.place[tid] = first;
            __syncthreads();
#pragma unroll
            for (int j = 0; j < SORT_PT; ++j) {
                const int i = i0 + 32 * j;
                if (j < pt && i < m) {
                    const unsigned d = ((key[j] - mn) >> shift) & (SORT_DIGITS - 1);
                    const unsigned at = sh.place[d] + sh.cnt[w][d] + rank[j];
                    if (one) sh.key[cur ^ 1][at] = key[j];
                    else b[at] = key[j];
                }
            }
            __syncthreads();
        }
        cur ^= 1;
        unsigned* t = a;
        a = b;
        b = t;
    }
    const int lead = (int)(((unsigned long long)out >> 2) & 31ull);
    for (int i = tid - lead; i < n; i += SORT_THREADS)
        if (i >= 0) out[i] = (one ? sh.key[cur][i] : a[i]) ^ 0x80000000u;
    __syncthreads();
}
}  // namespace

// Blocks take the slots of more than FIN_WCAP ids that finalize_kernel listed.
__global__ void __launch_bounds__(SORT_THREADS)
sort_large_kernel(int* res_pool, const long long* cand_off, const int* reg_len, const int* res_count,
                  const int* out_off, int* out, int* stage, long long out_cap, const int* list, const int* nlist,
                  int* queue)
{
    extern __shared__ __align__(16) char smem[];
    SortShared& sh = *(SortShared*)smem;
    pdl_wait();
    pdl_trigger();
    const int nl = *nlist;
    for (int e = blockIdx.x; e < nl;) {
        const int s = list[e];
        const int n = min(res_count[s], reg_len[s]), os = out_off[s];
        if ((long long)os + n <= out_cap)
            sort_slot(sh, (const unsigned*)(res_pool + cand_off[s]), (unsigned*)(stage + os), (unsigned*)(out + os), n);
        if (nl <= (int)gridDim.x) break;
        if (threadIdx.x == 0) sh.slot = (int)gridDim.x + atomicAdd(queue, 1);
        __syncthreads();
        e = sh.slot;
        __syncthreads();
    }
}

size_t sort_large_smem() { return sizeof(SortShared); }

}  // namespace rknn
