// Verification of an item's users by bounding boxes first: a group of
// consecutive candidates (a few grid cells of one row) lies in a small box,
// and most half-planes either hold the whole box or miss it.  Lanes own
// half-planes (32 a step) and classify them against each group's box; only
// the half-planes whose line crosses the box are evaluated user by user, and
// a group whose certain violations reach k, or whose certain and crossing
// ones together stay below k, needs no evaluation at all.
//
// What bounds it: instruction issue in FP32 (street layout, 16,384 queries of
// 2,768 candidates: 9.3 steps of 32 half-planes an item of 128 users, 1.8 of
// its 4 groups left open, about 10 evaluations a user instead of 237;
// 3.08 -> 1.48 ms), the FP64 pipe and issue in FP64 (110.4 -> 2.27 ms; uniform
// k=10, 1000 queries: 348 -> 43 us).
//
// The box test is a certified float test in both precision modes: it decides
// a (box, half-plane) pair only when every user of the box is on one side by
// more than the evaluation's error; what it leaves open is decided user by
// user in the mode's own precision.
#pragma once
#include "verify_item.cuh"

namespace rknn {
namespace vitem {

// Least and largest of a float over the warp.
__device__ __forceinline__ float warp_fmin(float v)
{
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_fmax(float v)
{
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// A box of user offsets from q: centre, half extents (rounded up) and the FP32
// evaluation bound of its users.
struct UserBox {
    float cx, cy, hx, hy, b;
};

__device__ __forceinline__ UserBox make_box(const QDesc& d, float x0, float x1, float y0, float y1)
{
    UserBox r;
    r.cx = 0.5f * x0 + 0.5f * x1;
    r.cy = 0.5f * y0 + 0.5f * y1;
    r.hx = fmaxf(__fsub_ru(x1, r.cx), __fsub_ru(r.cx, x0));
    r.hy = fmaxf(__fsub_ru(y1, r.cy), __fsub_ru(r.cy, y0));
    r.b = __fmaf_ru(d.k2f, __fadd_ru(fmaxf(fabsf(x0), fabsf(x1)), fmaxf(fabsf(y0), fabsf(y1))), d.kf2);
    return r;
}

// Half-plane p = (a, b, c, w) against a box.  cert: its facility is strictly
// nearer than q to every user of the box; cross: the box does not decide it.
// (Neither: it is strictly nearer to none of them.)
// For a user at float offsets (x, y) in the box, with M = a cx + b cy + c in
// real arithmetic, the exact m(u) differs from M by at most |a| hx + |b| hy
// plus, for the rounding of the coefficients (u for a and b, 5u for c) and of
// x and y, 2u|a|X + 2u|b|Y + 5u|c|; the two FMAs below add u|a|X + 2u|b|Y +
// 2u|c|.  With |a|, |b| <= 2F' and |c| <= F'^2 that is at most
// 8uF'(X + Y) + 7uF'^2, below the box's bound 8u (2F'(X + Y) + F'^2).
// Where something may overflow the bound is infinite (filter_bound), which
// leaves the pair undecided (mc + r < -inf is false, and so is mc - r > inf; NaNs
// compare false).
// NO_PLANE is neither (and undecided where the bound overflows: callers mask
// the lanes that hold it).
#define NO_PLANE make_float4(0.0f, 0.0f, INFINITY, 0.0f)
__device__ __forceinline__ void box_test(const float4 p, const UserBox& q, bool& cert, bool& cross)
{
    const float mc = fmaf(p.x, q.cx, fmaf(p.y, q.cy, p.z));
    const float r = __fmaf_ru(fabsf(p.x), q.hx, __fmul_ru(fabsf(p.y), q.hy));
    cert = __fadd_ru(mc, r) < -q.b;
    cross = !cert && !(__fsub_rd(mc, r) > q.b);
}

// What the boxes of an item's groups (group t: the warp's users t) decided.
template <int UPT>
struct GroupState {
    UserBox box[UPT];
    int cert[UPT];          // half-planes certain for the whole group
    unsigned cm[UPT];       // lane s: the open ones among half-planes 32s .. 32s + 31
    int ns;                 // steps of 32 half-planes taken
    unsigned open;          // groups (bit t) that need evaluations user by user
};

// planes: the slot's first nb <= 1024 half-planes.
template <int UPT>
__device__ __forceinline__ void group_boxes(const QDesc& d, int nb, const float4* planes, const float2* u,
                                            const bool* valid, GroupState<UPT>& G, unsigned& evals)
{
    const int lane = threadIdx.x & 31;
    const int k = d.k;
    float limtop = 0.0f;
#pragma unroll
    for (int t = 0; t < UPT; ++t) {
        const bool any = __any_sync(FULL, valid[t]);
        const float x = u[t].x - d.qx, y = u[t].y - d.qy;
        const float x0 = warp_fmin(valid[t] ? x : INFINITY), x1 = warp_fmax(valid[t] ? x : -INFINITY);
        const float y0 = warp_fmin(valid[t] ? y : INFINITY), y1 = warp_fmax(valid[t] ? y : -INFINITY);
        const float l = warp_fmax(valid[t] ? user_lim(x, y) : 0.0f);
        G.box[t] = make_box(d, x0, x1, y0, y1);
        G.cert[t] = any ? 0 : INT_MAX / 2;
        G.cm[t] = 0u;
        limtop = fmaxf(limtop, l);
    }
    G.ns = 0;
    // a lane counts its own half-planes; the warp sums at the end, and every
    // eighth step for the early exit
    int mine[UPT];
#pragma unroll
    for (int t = 0; t < UPT; ++t) mine[t] = 0;
    for (int m0 = 0; m0 < nb; m0 += 32, ++G.ns) {
        const int m = m0 + lane;
        const bool in = m < nb;
        const float4 p = in ? planes[m] : NO_PLANE;
        const unsigned inm = __ballot_sync(FULL, in);
        // the fourth component bounds |f - q|^2 for this and every later one
        if (__shfl_sync(FULL, p.w, 0) > limtop) break;
        if ((G.ns & 7) == 7) {
            bool left = false;
#pragma unroll
            for (int t = 0; t < UPT; ++t) left |= G.cert[t] + __reduce_add_sync(FULL, mine[t]) < k;
            if (!left) break;
        }
        evals += in ? UPT : 0;
#pragma unroll
        for (int t = 0; t < UPT; ++t) {
            bool ce, cr;
            box_test(p, G.box[t], ce, cr);
            mine[t] += ce;
            const unsigned c = __ballot_sync(FULL, cr) & inm;
            if (lane == G.ns) G.cm[t] = c;
        }
    }
    G.open = 0u;
#pragma unroll
    for (int t = 0; t < UPT; ++t) {
        G.cert[t] += __reduce_add_sync(FULL, mine[t]);
        const int cross = __reduce_add_sync(FULL, __popc(G.cm[t]));
        if (G.cert[t] < k && G.cert[t] + cross >= k) G.open |= 1u << t;
    }
}

// -2 v for a double that is zero or normal (v is a difference of floats), by
// its bits.
__device__ __forceinline__ double neg_twice(double v)
{
    const int hi = __double2hiint(v);
    return (hi & 0x7ff00000) ? __hiloint2double((hi + 0x00100000) ^ 0x80000000, __double2loint(v)) : 0.0;
}

// v[t] for a t all lanes share, without an array in memory.
template <int UPT, typename T>
__device__ __forceinline__ T pick(const T* v, int t)
{
    T r = v[0];
#pragma unroll
    for (int i = 1; i < UPT; ++i)
        if (t == i) r = v[i];
    return r;
}

// A warp's scratch for the half-planes that cross a group's box.
struct BoxScratch {
    uint16_t* list;         // their indices
    char* stage;            // 32 of them, as the evaluation reads them
    unsigned* mask;         // [quarter][chunk of 32]: those that cross a quarter's box
    float4* box;            // [quarter][2]: (cx, cy, hx, hy), (b, -, -, -)
};

// Stage 1 with boxes, over the slot's first nb half-planes gp (float, global
// memory; pos_of: their facilities).  direct[t]: the half-planes show the
// user to be a result; surv[t]: they leave it open (see filter_users).
//
// A group of 32 users that its box leaves open lists its crossing half-planes
// and tests them against the boxes of its quarters (8 users, about a cell);
// the quarters then evaluate their own crossing half-planes side by side, so a
// trip serves four half-planes, and stop once every user of theirs is
// decided.
//
// FP64: a warp's FP64 instruction holds its sub-partition's FP64 pipe for
// about 64 cycles on GB300, whatever the number of lanes, so what counts is
// how many are issued: two FMAs a trip, and four for each 32 half-planes made
// in double (the compares are integer compares of the bits: mv is finite and
// bu > 0, so mv < -bu is order_key(mv) < ~bits(bu), and |mv| <= bu compares
// the magnitude bits).  bu is the double bound rounded up to a float.
template <int UPT, bool F64>
__device__ __forceinline__ void filter_boxed(const VerifyArgs& A, const QDesc& d, int nb, const float4* gp,
                                             const int* pos_of, const BoxScratch& S, const float2* u,
                                             const bool* valid, bool* direct, bool* surv, unsigned& evals, float rho2)
{
    const int lane = threadIdx.x & 31;
    GroupState<UPT> G;
    group_boxes<UPT>(d, nb, gp, u, valid, G, evals);
    const int k = d.k;
    unsigned dbits = 0u, sbits = 0u;        // direct, surv: bit t
#pragma unroll
    for (int t = 0; t < UPT; ++t) {
        // no group evaluation needed: certain for all, or fewer than k even
        // if every half-plane left open were a violation
        const bool in = valid[t] && G.cert[t] < k,
                   dir = in && !(user_lim(u[t].x - d.qx, u[t].y - d.qy) > rho2);
        dbits |= (unsigned)dir << t;
        sbits |= (unsigned)(in && !dir) << t;
    }
    // one copy of the evaluation's code for all groups: unrolled, the kernel
    // outgrew the instruction caches (9 of 16 cycles an instruction waited for
    // them, street workload)
#pragma unroll 1
    for (unsigned todo = G.open; todo; todo &= todo - 1) {
        const int t = __ffs(todo) - 1;
        const float2 ut = make_float2(pick<UPT>(u, t).x, pick<UPT>(u, t).y);
        const float xt = ut.x - d.qx, yt = ut.y - d.qy;
        const bool vt = pick<UPT>(valid, t);
        int cnt = pick<UPT>(G.cert, t), rem = 0;
        const unsigned cmt = pick<UPT>(G.cm, t);
        {
            // boxes of the group's quarters
            float x0 = vt ? xt : INFINITY, x1 = vt ? xt : -INFINITY;
            float y0 = vt ? yt : INFINITY, y1 = vt ? yt : -INFINITY;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                x0 = fminf(x0, __shfl_xor_sync(FULL, x0, o));
                x1 = fmaxf(x1, __shfl_xor_sync(FULL, x1, o));
                y0 = fminf(y0, __shfl_xor_sync(FULL, y0, o));
                y1 = fmaxf(y1, __shfl_xor_sync(FULL, y1, o));
            }
            const UserBox own = make_box(d, x0, x1, y0, y1);
            if ((lane & 7) == 0) {
                S.box[lane >> 2] = make_float4(own.cx, own.cy, own.hx, own.hy);
                S.box[(lane >> 2) + 1].x = own.b;
            }
            if (lane == 0) {
                // the stage's entry 0: no violation, not too close (a NaN
                // that compares above every bound)
                if constexpr (F64) {
                    double* v = (double*)S.stage;
                    v[0] = v[BOX_STAGE] = 0.0;
                    v[2 * BOX_STAGE] = INFINITY;
                } else {
                    ((float4*)S.stage)[0] = make_float4(0.0f, 0.0f, NAN, 0.0f);
                }
            }
            int ce4[4], cr4[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) { ce4[j] = cnt; cr4[j] = 0; }
            // the group's crossing half-planes, in order
            int n = 0;
            for (int s = 0; s < G.ns; ++s) {
                const unsigned M = __shfl_sync(FULL, cmt, s);
                if ((M >> lane) & 1u) S.list[n + __popc(M & ((1u << lane) - 1))] = (uint16_t)(32 * s + lane);
                n += __popc(M);
            }
            __syncwarp();
            const int nc = (n + 31) >> 5;
            for (int c = 0; c < nc; ++c) {
                const int i = 32 * c + lane;
                const bool in = i < n;
                const float4 p = in ? gp[S.list[i]] : NO_PLANE;
                const unsigned inm = __ballot_sync(FULL, in);
                evals += in ? 4 : 0;
                unsigned mine = 0u;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    bool ce, cr;
                    const float4 b0 = S.box[2 * j];
                    box_test(p, UserBox{b0.x, b0.y, b0.z, b0.w, S.box[2 * j + 1].x}, ce, cr);
                    ce4[j] += __popc(__ballot_sync(FULL, ce));
                    const unsigned m = __ballot_sync(FULL, cr) & inm;
                    cr4[j] += __popc(m);
                    if (lane == j) mine = m;
                }
                if (lane < 4) S.mask[32 * lane + c] = mine;
            }
            __syncwarp();
            const int g = lane >> 3;
            cnt = g == 0 ? ce4[0] : g == 1 ? ce4[1] : g == 2 ? ce4[2] : ce4[3];
            rem = g == 0 ? cr4[0] : g == 1 ? cr4[1] : g == 2 ? cr4[2] : cr4[3];
            if (!vt) cnt = INT_MAX / 2;
            // bit 0: fewer than k certain, bit 1: also with all those open
            const int closed = (cnt < k ? 1 : 0) | (cnt + rem < k ? 2 : 0);
            int state = closed;
            if (__any_sync(FULL, state == 1)) {
                // Eight lanes a quarter.  FP64: with one or two quarters open
                // (1.8 of 4 on average on the street layout), four or two times
                // eight lanes share a quarter's half-planes, which halves the
                // FP64 trips; in FP32 the sums cost more than the trips saved
                // (1.46 -> 1.51 ms).
                unsigned act = 0u;      // the open quarters (their first lane's bit)
                int na = 4, q1 = 0, q2 = 0, qs = g;
                unsigned share = ~0u;
                float2 us = ut;
                int base = cnt, later = rem;
                bool open = state == 1;
                if constexpr (F64) {
                    act = __ballot_sync(FULL, open);
                    act |= act >> 4;
                    act |= act >> 2;
                    act = (act | act >> 1) & 0x01010101u;
                    na = __popc(act);
                    q1 = (__ffs(act) - 1) >> 3;
                    q2 = (31 - __clz(act)) >> 3;
                    if (na <= 2) {
                        qs = g < 2 ? q1 : q2;
                        share = na == 2 ? 0x55555555u << (g & 1) : 0x11111111u << g;
                        const int src = 8 * qs + (lane & 7);
                        us = make_float2(__shfl_sync(FULL, ut.x, src), __shfl_sync(FULL, ut.y, src));
                        base = __shfl_sync(FULL, cnt, src);
                        later = __shfl_sync(FULL, rem, src);
                        open = __shfl_sync(FULL, open, src);
                    }
                }
                const float xs = us.x - d.qx, ys = us.y - d.qy;
                double qx = 0.0, qy = 0.0, xx = 0.0, yy = 0.0;
                long long bb = 0;
                float bu = 0.0f;
                unsigned bu2 = 0u;
                if constexpr (F64) {
                    qx = f2d_bits(d.qx);
                    qy = f2d_bits(d.qy);
                    xx = f2d_bits(us.x) - qx;
                    yy = f2d_bits(us.y) - qy;
                    // |x| + |y| above the floats' rounding, then every step up
                    const float ax = __fmul_ru(__fadd_ru(fabsf(xs), fabsf(ys)), 1.0f + 0x1p-22f);
                    bb = __double_as_longlong(f2d_bits(
                        __fmaf_ru(__double2float_ru(d.k2f64), ax, __double2float_ru(d.kf264))));
                } else {
                    bu = fmaf(d.k2f, fabsf(xs) + fabsf(ys), d.kf2);
                    bu2 = min(__float_as_uint(__fmul_ru(bu, 2.0f * (1.0f + 0x1p-20f))), 0x7f800000u);
                }
                // a lane's counts over its half-planes, and the sums over those
                // that share the user: certified in bits 0-10 (at most 1024),
                // too close to call in 11-21, still to do in 22-27
                unsigned mine = 0u, sum = 0u;
                int ne = 0;
                for (int c = 0; c < nc; ++c) {
                    unsigned mm = S.mask[32 * qs + c];
                    // a quarter goes on while one of its users is open
                    const unsigned go = __ballot_sync(FULL, open);
                    if (!go) break;
                    if (!((go >> (lane & 24)) & 0xffu)) mm = 0u;
                    if (!__any_sync(FULL, mm != 0u)) continue;
                    later -= __popc(mm);
                    mm &= share;
                    // the chunk's half-planes, one per lane
                    const int i = 32 * c + lane;
                    if (i < n) {
                        if constexpr (F64) {
                            const float2 f = A.fxy[VX(pos_of[S.list[i]], A.nf, 204)];
                            const double dx = f2d_bits(f.x) - qx, dy = f2d_bits(f.y) - qy;
                            double* v = (double*)S.stage + 1 + lane;
                            v[0] = neg_twice(dx);
                            v[BOX_STAGE] = neg_twice(dy);
                            v[2 * BOX_STAGE] = fma(dx, dx, dy * dy);
                        } else {
                            ((float4*)S.stage)[1 + lane] = gp[S.list[i]];
                        }
                    }
                    __syncwarp();
                    // lanes out of half-planes evaluate entry 0: without
                    // branches around the evaluations 1.67 -> 1.52 ms
                    ne += __popc(mm);
                    auto settle = [&]() {
                        sum = mine + ((unsigned)__popc(mm) << 22);
                        if constexpr (F64) {
                            if (na <= 2) sum += __shfl_xor_sync(FULL, sum, 8);
                            if (na == 1) sum += __shfl_xor_sync(FULL, sum, 16);
                        }
                        const int ce = base + (int)(sum & 0x7ffu);
                        open = ce < k && ce + (int)((sum >> 11) & 0x7ffu) + (int)(sum >> 22) + later >= k;
                        const unsigned more = __ballot_sync(FULL, open);
                        if (!((more >> (lane & 24)) & 0xffu)) {
                            ne -= __popc(mm);
                            mm = 0u;
                        }
                    };
                    if constexpr (F64) {
                        while (__any_sync(FULL, mm != 0u)) {
                            const double* v = (const double*)S.stage + __ffs(mm);
                            mm &= mm - 1;
                            const double mv = fma(v[0], xx, fma(v[BOX_STAGE], yy, v[2 * BOX_STAGE]));
                            mine += order_key(mv) < ~bb;
                            mine += (__double_as_longlong(mv) & 0x7fffffffffffffffll) <= bb ? 1u << 11 : 0u;
                            settle();
                        }
                    } else {
                        // r = m(u) + bu: negative for a certified violation, in
                        // [0, 2 bu] for one too close to call (filter_users)
                        while (__any_sync(FULL, mm != 0u)) {
#pragma unroll
                            for (int j = 0; j < BOX_TRIP; ++j) {
                                const float4 p = ((const float4*)S.stage)[__ffs(mm)];
                                mm &= mm - 1;
                                const float r = fmaf(p.x, xs, fmaf(p.y, ys, p.z)) + bu;
                                mine += __float_as_uint(r) >> 31;
                                mine += __float_as_uint(r) <= bu2 ? 1u << 11 : 0u;
                            }
                            settle();
                        }
                    }
                    __syncwarp();
                }
                evals += base < INT_MAX / 2 ? ne : 0;
                // back to the users' own lanes
                const int ce = base + (int)(sum & 0x7ffu);
                state = (ce < k ? 1 : 0) |
                        (ce + (int)((sum >> 11) & 0x7ffu) + (int)(sum >> 22) + later < k ? 2 : 0);
                if constexpr (F64)
                    if (na <= 2) {
                        // back to the users' own lanes
                        const int back = __shfl_sync(FULL, state, (na == 2 && g == q2 ? 16 : 0) + (lane & 7));
                        state = ((act >> (8 * g)) & 1u) ? back : closed;
                    }
            }
            __syncwarp();           // the scratch is free again
            // fewer than k even if every half-plane left open were a violation
            const bool in = vt && (state & 1), dir = in && (state & 2) && !(user_lim(xt, yt) > rho2);
            const unsigned bit = 1u << t;
            dbits = (dbits & ~bit) | (dir ? bit : 0u);
            sbits = (sbits & ~bit) | (in && !dir ? bit : 0u);
        }
    }
#pragma unroll
    for (int t = 0; t < UPT; ++t) {
        direct[t] = (dbits >> t) & 1u;
        surv[t] = (sbits >> t) & 1u;
    }
}

}  // namespace vitem
}  // namespace rknn
