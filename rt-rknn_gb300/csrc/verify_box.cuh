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
// 3.08 -> 1.75 ms), the FP64 pipe in FP64 (110.4 -> 2.94 ms; uniform k=10,
// 1000 queries: 348 -> 47 us).
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

// A box of user offsets from q: centre, half extents (rounded up), the FP32
// evaluation bound of its users and the largest of their lims.
struct UserBox {
    float cx, cy, hx, hy, b, lim;
};

__device__ __forceinline__ UserBox make_box(const QDesc& d, float x0, float x1, float y0, float y1, float lim)
{
    UserBox r;
    r.cx = 0.5f * x0 + 0.5f * x1;
    r.cy = 0.5f * y0 + 0.5f * y1;
    r.hx = fmaxf(__fsub_ru(x1, r.cx), __fsub_ru(r.cx, x0));
    r.hy = fmaxf(__fsub_ru(y1, r.cy), __fsub_ru(r.cy, y0));
    r.b = __fmaf_ru(d.k2f, __fadd_ru(fmaxf(fabsf(x0), fabsf(x1)), fmaxf(fabsf(y0), fabsf(y1))), d.kf2);
    r.lim = lim;
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
// Values that overflow leave the pair undecided (every compare is false).
__device__ __forceinline__ void box_test(const float4 p, const UserBox& q, bool in, bool& cert, bool& cross)
{
    const float mc = fmaf(p.x, q.cx, fmaf(p.y, q.cy, p.z));
    const float r = __fmaf_ru(fabsf(p.x), q.hx, __fmul_ru(fabsf(p.y), q.hy));
    // a facility with |f - q| beyond 2|u - q| for every user decides nothing
    const bool on = in && !(p.w > q.lim);
    cert = on && __fadd_ru(mc, r) < -q.b;
    cross = on && !cert && !(__fsub_rd(mc, r) > q.b);
}

// What the boxes of an item's groups (group t: the warp's users t) decided.
template <int UPT>
struct GroupState {
    UserBox box[UPT];
    int cert[UPT];          // half-planes certain for the whole group
    int cross[UPT];         // half-planes left open
    unsigned cm[UPT];       // lane s: the open ones among half-planes 32s .. 32s + 31
    int ns;                 // steps of 32 half-planes taken
    unsigned open;          // groups (bit t) that need evaluations user by user
};

// planes: the slot's first nb <= 1024 half-planes.
template <int UPT>
__device__ __forceinline__ void group_boxes(const QDesc& d, int nb, const float4* planes, const float* x,
                                            const float* y, const float* lim, const bool* valid, GroupState<UPT>& G,
                                            unsigned& evals)
{
    const int lane = threadIdx.x & 31;
    const int k = d.k;
    float limtop = 0.0f;
#pragma unroll
    for (int t = 0; t < UPT; ++t) {
        const bool any = __any_sync(FULL, valid[t]);
        const float x0 = warp_fmin(valid[t] ? x[t] : INFINITY), x1 = warp_fmax(valid[t] ? x[t] : -INFINITY);
        const float y0 = warp_fmin(valid[t] ? y[t] : INFINITY), y1 = warp_fmax(valid[t] ? y[t] : -INFINITY);
        const float l = warp_fmax(valid[t] ? lim[t] : 0.0f);
        G.box[t] = make_box(d, x0, x1, y0, y1, l);
        G.cert[t] = any ? 0 : INT_MAX / 2;
        G.cross[t] = 0;
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
        const float4 p = in ? planes[m] : make_float4(0.f, 0.f, 0.f, 0.f);
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
            box_test(p, G.box[t], in, ce, cr);
            mine[t] += ce;
            const unsigned c = __ballot_sync(FULL, cr);
            if (lane == G.ns) G.cm[t] = c;
        }
    }
#pragma unroll
    for (int t = 0; t < UPT; ++t) {
        G.cert[t] += __reduce_add_sync(FULL, mine[t]);
        G.cross[t] = __reduce_add_sync(FULL, __popc(G.cm[t]));
    }
    G.open = 0u;
#pragma unroll
    for (int t = 0; t < UPT; ++t)
        if (G.cert[t] < k && G.cert[t] + G.cross[t] >= k) G.open |= 1u << t;
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
    float4* box;            // [quarter][2]: (cx, cy, hx, hy), (b, lim, 0, 0)
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
    float x[UPT], y[UPT], lim[UPT];
#pragma unroll
    for (int t = 0; t < UPT; ++t) {
        x[t] = u[t].x - d.qx;
        y[t] = u[t].y - d.qy;
        lim[t] = user_lim(x[t], y[t]);
    }
    GroupState<UPT> G;
    group_boxes<UPT>(d, nb, gp, x, y, lim, valid, G, evals);
    const int k = d.k;
    unsigned dbits = 0u, sbits = 0u;        // direct, surv: bit t
#pragma unroll
    for (int t = 0; t < UPT; ++t) {
        // no group evaluation needed: certain for all, or fewer than k even
        // if every half-plane left open were a violation
        const bool in = valid[t] && G.cert[t] < k, dir = in && !(lim[t] > rho2);
        dbits |= (unsigned)dir << t;
        sbits |= (unsigned)(in && !dir) << t;
    }
    // one copy of the evaluation's code for all groups: unrolled, the kernel
    // outgrew the instruction caches (9 of 16 cycles an instruction waited for
    // them, street workload)
#pragma unroll 1
    for (unsigned todo = G.open; todo; todo &= todo - 1) {
        const int t = __ffs(todo) - 1;
        const float xt = pick<UPT>(x, t), yt = pick<UPT>(y, t), lt = pick<UPT>(lim, t);
        const bool vt = pick<UPT>(valid, t);
        int cnt = pick<UPT>(G.cert, t), rem = pick<UPT>(G.cross, t), und = 0;
        const unsigned cmt = pick<UPT>(G.cm, t);
        {
            // boxes of the group's quarters
            float x0 = vt ? xt : INFINITY, x1 = vt ? xt : -INFINITY;
            float y0 = vt ? yt : INFINITY, y1 = vt ? yt : -INFINITY;
            float l = vt ? lt : 0.0f;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                x0 = fminf(x0, __shfl_xor_sync(FULL, x0, o));
                x1 = fmaxf(x1, __shfl_xor_sync(FULL, x1, o));
                y0 = fminf(y0, __shfl_xor_sync(FULL, y0, o));
                y1 = fmaxf(y1, __shfl_xor_sync(FULL, y1, o));
                l = fmaxf(l, __shfl_xor_sync(FULL, l, o));
            }
            const UserBox own = make_box(d, x0, x1, y0, y1, l);
            if ((lane & 7) == 0) {
                S.box[lane >> 2] = make_float4(own.cx, own.cy, own.hx, own.hy);
                S.box[(lane >> 2) + 1] = make_float4(own.b, own.lim, 0.0f, 0.0f);
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
                const float4 p = in ? gp[S.list[i]] : make_float4(0.f, 0.f, 0.f, 0.f);
                evals += in ? 4 : 0;
                unsigned mine = 0u;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    bool ce, cr;
                    const float4 b0 = S.box[2 * j];
                    const float2 b1 = *(const float2*)(S.box + 2 * j + 1);
                    box_test(p, UserBox{b0.x, b0.y, b0.z, b0.w, b1.x, b1.y}, in, ce, cr);
                    ce4[j] += __popc(__ballot_sync(FULL, ce));
                    const unsigned m = __ballot_sync(FULL, cr);
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
            double qx = 0.0, qy = 0.0, xx = 0.0, yy = 0.0;
            long long bb = 0;
            float bu = 0.0f;
            unsigned bu2 = 0u;
            int done = 0;
            for (int c = 0; c < nc; ++c) {
                unsigned mm = S.mask[32 * g + c];
                // a quarter goes on while one of its users is open
                const unsigned act = __ballot_sync(FULL, cnt < k && cnt + und + rem >= k);
                if (!act) break;
                if (!((act >> (lane & 24)) & 0xffu)) mm = 0u;
                if (!__any_sync(FULL, mm != 0u)) continue;
                // the chunk's half-planes, one per lane
                const int i = 32 * c + lane;
                if constexpr (F64) {
                    if (done == 0) {
                        qx = f2d_bits(d.qx);
                        qy = f2d_bits(d.qy);
                        xx = f2d_bits(pick<UPT>(u, t).x) - qx;
                        yy = f2d_bits(pick<UPT>(u, t).y) - qy;
                        // |x| + |y| above the floats' rounding, then every step up
                        const float ax = __fmul_ru(__fadd_ru(fabsf(xt), fabsf(yt)), 1.0f + 0x1p-22f);
                        bb = __double_as_longlong(f2d_bits(
                            __fmaf_ru(__double2float_ru(d.k2f64), ax, __double2float_ru(d.kf264))));
                    }
                    if (i < n) {
                        const float2 f = A.fxy[VX(pos_of[S.list[i]], A.nf, 204)];
                        const double dx = f2d_bits(f.x) - qx, dy = f2d_bits(f.y) - qy;
                        double* v = (double*)S.stage + lane;
                        v[0] = neg_twice(dx);
                        v[32] = neg_twice(dy);
                        v[64] = fma(dx, dx, dy * dy);
                    }
                } else {
                    if (done == 0) {
                        bu = fmaf(d.k2f, fabsf(xt) + fabsf(yt), d.kf2);
                        bu2 = __float_as_uint(__fmul_ru(bu, 2.0f * (1.0f + 0x1p-20f)));
                    }
                    if (i < n) ((float4*)S.stage)[lane] = gp[S.list[i]];
                }
                done = 1;
                __syncwarp();
                int ne = 0;
                if constexpr (F64) {
                    while (__any_sync(FULL, mm != 0u)) {
                        if (mm) {
                            const double* v = (const double*)S.stage + (__ffs(mm) - 1);
                            mm &= mm - 1;
                            --rem;
                            ++ne;
                            const double mv = fma(v[0], xx, fma(v[32], yy, v[64]));
                            cnt += order_key(mv) < ~bb;
                            und += (__double_as_longlong(mv) & 0x7fffffffffffffffll) <= bb;
                        }
                        const unsigned more = __ballot_sync(FULL, cnt < k && cnt + und + rem >= k);
                        if (!((more >> (lane & 24)) & 0xffu)) mm = 0u;
                    }
                } else {
                    // two a trip; r = m(u) + bu: negative for a certified
                    // violation, in [0, 2 bu] for one too close to call
                    // (filter_users)
                    auto eval = [&]() {
                        const float4 p = ((const float4*)S.stage)[__ffs(mm) - 1];
                        mm &= mm - 1;
                        --rem;
                        ++ne;
                        const float r = fmaf(p.x, xt, fmaf(p.y, yt, p.z)) + bu;
                        cnt += (int)(__float_as_uint(r) >> 31);
                        und += __float_as_uint(r) <= bu2;
                    };
                    while (__any_sync(FULL, mm != 0u)) {
                        if (mm) eval();
                        if (mm) eval();
                        const unsigned more = __ballot_sync(FULL, cnt < k && cnt + und + rem >= k);
                        if (!((more >> (lane & 24)) & 0xffu)) mm = 0u;
                    }
                }
                evals += vt ? ne : 0;
                __syncwarp();
            }
            __syncwarp();           // the scratch is free again
        }
        // fewer than k even if every half-plane left open were a violation
        const bool in = vt && cnt < k, dir = in && cnt + und + rem < k && !(lt > rho2);
        const unsigned bit = 1u << t;
        dbits = (dbits & ~bit) | (dir ? bit : 0u);
        sbits = (sbits & ~bit) | (in && !dir ? bit : 0u);
    }
#pragma unroll
    for (int t = 0; t < UPT; ++t) {
        direct[t] = (dbits >> t) & 1u;
        surv[t] = (sbits >> t) & 1u;
    }
}

}  // namespace vitem
}  // namespace rknn
