// Uniform-grid index: a stable LSD radix sort of the points on their cell
// number (digits of up to 8 bits), cell start offsets and per-cell facility
// MBRs.  It replaces the reference's per-process R*-tree
// (rknn-inf/RStarTree2D.cpp, insert 106-114): the zone kernel treats grid cells
// as leaf nodes and the verification reads each grid row of cells as one
// contiguous range.
//
// The sort moves whole records (point and id) and makes the cell number again
// from the point in each pass: no key is stored, and the last pass writes the
// index's own arrays, where sorting (cell, input index) pairs ended in a gather
// of 12 scattered bytes a point.  Bound by memory traffic: 10 M points into
// 1.25 M cells take 0.33 ms (a scatter 65 us for 240 MB), with pairs 0.75 (the
// gather 0.17).
#include "index.cuh"
#include <algorithm>
#include <climits>
#include <vector>

namespace rknn {

namespace {
constexpr unsigned FULL = 0xffffffffu;
constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_ITEMS = 8;            // items of a thread
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_BITS = 8;             // most bits of a digit
constexpr int RS_DIGITS = 1 << RS_BITS;
static_assert(RS_DIGITS == RS_THREADS, "a thread a digit");

__device__ __forceinline__ uint32_t cell_of(const float2 p, const Grid& g)
{
    return (uint32_t)(cell_coord(p.y, g.y0, g.inv, g.gy) * g.gx + cell_coord(p.x, g.x0, g.inv, g.gx));
}

// Digit counts of each tile of RS_TILE points: hist[digit][tile].
__global__ void __launch_bounds__(RS_THREADS) k_rs_hist(const float2* xy, int n, Grid g, int shift, int nd,
                                                        uint32_t* hist, int ntiles)
{
    __shared__ uint32_t h[RS_DIGITS];
    h[threadIdx.x] = 0;
    __syncthreads();
    const long long base = (long long)blockIdx.x * RS_TILE + threadIdx.x;
    float2 p[RS_ITEMS];
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
        const long long i = base + j * RS_THREADS;
        p[j] = i < n ? xy[i] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j)
        if (base + j * RS_THREADS < n) atomicAdd(&h[(cell_of(p[j], g) >> shift) & (nd - 1)], 1u);
    __syncthreads();
    if (threadIdx.x < nd) hist[(size_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// Stable scatter of one tile by a digit.  A warp takes 256 consecutive items,
// 32 at a time, and ranks each among its own (ballots on the digit's bits); the
// digits' counts of all warps then place the tile's records in order in shared
// memory, from where they go out in runs of one digit (written from the
// registers, each store of a warp touched up to 32 sectors).
// offs: the exclusive scan of hist.  w: the records' ids (null: their index).
__global__ void __launch_bounds__(RS_THREADS) k_rs_scatter(const float2* xy, const int* w, float2* xy_out, int* w_out,
                                                           int* pos_of, int n, Grid g, int shift, int nd,
                                                           const uint32_t* offs, int ntiles)
{
    __shared__ float2 sxy[RS_TILE];
    __shared__ int sw[RS_TILE];
    __shared__ uint8_t sd[RS_TILE];
    __shared__ uint32_t wc[RS_WARPS][RS_DIGITS];
    __shared__ uint32_t go[RS_DIGITS];
    __shared__ uint32_t ws[RS_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, wi = tid >> 5;
    const long long base = (long long)blockIdx.x * RS_TILE;
    const int cnt = (int)(n - base < RS_TILE ? n - base : RS_TILE);
    float2 p[RS_ITEMS];
    int v[RS_ITEMS];
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
        const int i = wi * (32 * RS_ITEMS) + 32 * j + lane;
        p[j] = i < cnt ? xy[base + i] : make_float2(0.f, 0.f);
        v[j] = i < cnt ? (w ? w[base + i] : (int)(base + i)) : 0;
    }
    const uint32_t first = tid < nd ? offs[(size_t)tid * ntiles + blockIdx.x] : 0u;
#pragma unroll
    for (int j = 0; j < RS_DIGITS / 32; ++j) wc[wi][32 * j + lane] = 0u;
    __syncwarp();
    uint32_t dl[RS_ITEMS];          // digit, and rank among the warp's items of it (bits 8 up)
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
        const bool ok = wi * (32 * RS_ITEMS) + 32 * j + lane < cnt;
        const uint32_t dg = (cell_of(p[j], g) >> shift) & (uint32_t)(nd - 1);
        unsigned same = __ballot_sync(FULL, ok);
#pragma unroll
        for (int b = 0; b < RS_BITS; ++b) {
            const unsigned m = __ballot_sync(FULL, (dg >> b) & 1u);
            same &= ((dg >> b) & 1u) ? m : ~m;
        }
        const uint32_t old = wc[wi][dg];
        __syncwarp();
        if (ok && (same & ((1u << lane) - 1)) == 0u) wc[wi][dg] = old + __popc(same);
        __syncwarp();
        dl[j] = dg | (old + __popc(same & ((1u << lane) - 1))) << RS_BITS;
    }
    __syncthreads();
    {
        // thread tid: digit tid's first place in the tile, for each warp
        uint32_t sum = 0u;
#pragma unroll
        for (int j = 0; j < RS_WARPS; ++j) sum += wc[j][tid];
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) ws[wi] = x;
        __syncthreads();
        uint32_t at = x - sum;
#pragma unroll
        for (int j = 0; j < RS_WARPS; ++j) at += j < wi ? ws[j] : 0u;
        go[tid] = first - at;
#pragma unroll
        for (int j = 0; j < RS_WARPS; ++j) {
            const uint32_t c = wc[j][tid];
            wc[j][tid] = at;
            at += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
        if (wi * (32 * RS_ITEMS) + 32 * j + lane >= cnt) continue;
        const uint32_t dg = dl[j] & (RS_DIGITS - 1), at = wc[wi][dg] + (dl[j] >> RS_BITS);
        sxy[at] = p[j];
        sw[at] = v[j];
        sd[at] = (uint8_t)dg;
    }
    __syncthreads();
    for (int i = tid; i < cnt; i += RS_THREADS) {
        const uint32_t to = go[sd[i]] + (uint32_t)i;
        xy_out[to] = sxy[i];
        w_out[to] = sw[i];
        if (pos_of) pos_of[sw[i]] = (int)to;
    }
}

// exclusive scan, 1024 items per block, block totals to sums
__global__ void k_scan_block(const uint32_t* in, uint32_t* out, int n, uint32_t* sums)
{
    __shared__ uint32_t ws[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int i = blockIdx.x * 1024 + tid;
    uint32_t v = i < n ? in[i] : 0u, x = v;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (w == 0) {
        uint32_t t = ws[lane];
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(FULL, t, o);
            if (lane >= o) t += y;
        }
        ws[lane] = t;
    }
    __syncthreads();
    uint32_t excl = x - v + (w ? ws[w - 1] : 0u);
    if (i < n) out[i] = excl;
    if (tid == 1023 && sums) sums[blockIdx.x] = ws[31];
}

__global__ void k_scan_add(uint32_t* out, int n, const uint32_t* sums)
{
    int i = blockIdx.x * 1024 + threadIdx.x;
    if (i < n && blockIdx.x > 0) out[i] += sums[blockIdx.x];
}

// First point of the sorted n whose cell is at least c, by a warp: 32 probes a
// round.
__device__ __forceinline__ int warp_lower_bound(const float2* xy, int n, const Grid& g, uint32_t c)
{
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = n;             // the answer lies in [lo, hi]
    while (lo < hi) {
        const int step = (int)(((long long)hi - lo + 31) >> 5);
        const long long i = lo + (long long)(lane + 1) * step - 1;
        const bool less = i < hi && cell_of(xy[i], g) < c;
        lo = (int)min((long long)hi, lo + (long long)__popc(__ballot_sync(FULL, less)) * step);
        hi = (int)min((long long)hi, (long long)lo + step - 1);
    }
    return lo;
}

// Cell starts from the sorted points: a block finds the points of its ST_CELLS
// cells, a thread its cells' first ones among them by bisection, side by side.
// The work follows the cells, however the points crowd in them.  Bound by the
// scattered probes (10 M points, 1.25 M cells: 44 us; one cell after the other
// 49, a thread a point 65, counting with atomics and scanning the counts 57).
constexpr int ST_THREADS = 256, ST_CELLS = 1024;
__global__ void __launch_bounds__(ST_THREADS) k_starts(const float2* xy, int n, Grid g, int nc, int* start)
{
    __shared__ int range[2];
    const int c0 = blockIdx.x * ST_CELLS, c1 = min(c0 + ST_CELLS, nc + 1);
    const int wi = threadIdx.x >> 5;
    if (wi < 2) {
        const int r = warp_lower_bound(xy, n, g, (uint32_t)(wi ? c1 : c0));
        if ((threadIdx.x & 31) == 0) range[wi] = r;
    }
    __syncthreads();
    constexpr int C = ST_CELLS / ST_THREADS;
    int lo[C], len = range[1] - range[0];
#pragma unroll
    for (int j = 0; j < C; ++j) lo[j] = range[0];
    while (len > 0) {
        const int half = (len + 1) >> 1;
#pragma unroll
        for (int j = 0; j < C; ++j)
            if (cell_of(xy[lo[j] + half - 1], g) < (uint32_t)(c0 + j * ST_THREADS + threadIdx.x)) lo[j] += half;
        len -= half;
    }
#pragma unroll
    for (int j = 0; j < C; ++j) {
        const int c = c0 + j * ST_THREADS + threadIdx.x;
        if (c < c1) start[c] = lo[j];
    }
}

// Box of each cell's points; *filled counts the cells that have any.
__global__ void k_mbr(const float2* xy, const int* start, int nc, float4* mbr, int* filled)
{
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = __syncthreads_count(c < nc && start[c + 1] > start[c]);
    if (threadIdx.x == 0 && n) atomicAdd(filled, n);
    if (c >= nc) return;
    float4 r = make_float4(INFINITY, INFINITY, -INFINITY, -INFINITY);
    for (int i = start[c]; i < start[c + 1]; ++i) {
        float2 p = xy[i];
        r.x = fminf(r.x, p.x); r.y = fminf(r.y, p.y);
        r.z = fmaxf(r.z, p.x); r.w = fmaxf(r.w, p.y);
    }
    mbr[c] = r;
}

// Integer key with a finite float's order.
__device__ __forceinline__ unsigned float_key(float f)
{
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : u | 0x80000000u;
}

// Bounding box of n points and whether any coordinate is not finite.  One
// pass over the points, bound by their reads (0.15 ms for 11 M points with its
// copies and waits, where one host core took 20.8 ms).
constexpr int BB_THREADS = 256;
__global__ void __launch_bounds__(BB_THREADS) k_bbox(const float2* xy, int n, PointBox* box, int* bad)
{
    unsigned x0 = 0xffffffffu, y0 = 0xffffffffu, x1 = 0u, y1 = 0u;
    bool nf = false;
    const int stride = gridDim.x * BB_THREADS;
    for (int i = blockIdx.x * BB_THREADS + threadIdx.x; i < n; i += 4 * stride) {
        float2 p[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] = (long long)i + (long long)j * stride < n ? xy[i + j * stride] : xy[i];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!isfinite(p[j].x) || !isfinite(p[j].y)) { nf = true; continue; }
            const unsigned kx = float_key(p[j].x), ky = float_key(p[j].y);
            x0 = min(x0, kx); x1 = max(x1, kx);
            y0 = min(y0, ky); y1 = max(y1, ky);
        }
    }
    __shared__ unsigned s[4][BB_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    x0 = __reduce_min_sync(FULL, x0); y0 = __reduce_min_sync(FULL, y0);
    x1 = __reduce_max_sync(FULL, x1); y1 = __reduce_max_sync(FULL, y1);
    if (__any_sync(FULL, nf) && lane == 0) atomicOr(bad, 1);
    if (lane == 0) { s[0][w] = x0; s[1][w] = y0; s[2][w] = x1; s[3][w] = y1; }
    __syncthreads();
    if (threadIdx.x < 4) {
        unsigned v = s[threadIdx.x][0];
        for (int j = 1; j < BB_THREADS / 32; ++j)
            v = threadIdx.x < 2 ? min(v, s[threadIdx.x][j]) : max(v, s[threadIdx.x][j]);
        if (threadIdx.x < 2) atomicMin(box->key + threadIdx.x, v);
        else atomicMax(box->key + threadIdx.x, v);
    }
}

inline int nblk(long long n, int b) { return (int)((n + b - 1) / b); }
}  // namespace

// Exclusive scan of n values in place; sums: room for scan_room(n) values.
namespace {
size_t scan_room(size_t n)
{
    size_t r = 0;
    while (n > 1024) r += n = (n + 1023) / 1024;
    return r;
}
void scan_exclusive_u32(uint32_t* v, int n, uint32_t* sums, cudaStream_t st)
{
    const int nb = nblk(n, 1024);
    k_scan_block<<<nb, 1024, 0, st>>>(v, v, n, nb > 1 ? sums : nullptr);
    if (nb > 1) {
        scan_exclusive_u32(sums, nb, sums + nb, st);
        k_scan_add<<<nb, 1024, 0, st>>>(v, n, sums);
    }
}

// grid_sort's passes and its scratch: the digit counts, their scan's sums, and
// the records between passes (the outputs hold every second pass's).
struct SortPlan {
    int passes, bits, nd, ntiles;
    size_t nh, xy_at, w_at, bytes;
    SortPlan(int n, const Grid& g)
    {
        const long long nc = (long long)g.gx * g.gy;
        int all = 1;
        while ((1ll << all) < nc) ++all;
        passes = (all + RS_BITS - 1) / RS_BITS;
        bits = (all + passes - 1) / passes;
        nd = 1 << bits;
        ntiles = nblk(n, RS_TILE);
        nh = (size_t)nd * ntiles;
        auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
        xy_at = up(sizeof(uint32_t) * (nh + scan_room(nh)));
        w_at = xy_at + (passes > 1 ? up(sizeof(float2) * (size_t)n) : 0);
        bytes = w_at + (passes > 1 ? up(sizeof(int) * (size_t)n) : 0);
    }
};
}  // namespace

size_t grid_sort_bytes(int n, const Grid& g) { return n > 0 ? SortPlan(n, g).bytes : 0; }

// Sort n points into g's cells, stable.  d_ids: their ids (null: their
// index).  ws: grid_sort_bytes(n, g) bytes.  Outputs (device,
// caller-allocated): xy_s[n], ids_s[n], pos_of[n] (may be null: each id's
// place), start[nc+1].
cudaError_t grid_sort(const float2* d_xy, const int* d_ids, int n, const Grid& g, char* ws,
                      float2* xy_s, int* ids_s, int* pos_of, int* start, cudaStream_t st)
{
    const int nc = g.gx * g.gy;
    if (n > 0) {
        const SortPlan p(n, g);
        uint32_t* hist = (uint32_t*)ws;
        const float2* in = d_xy;
        const int* w = d_ids;
        for (int i = 0; i < p.passes; ++i) {
            const bool last = i == p.passes - 1, direct = (p.passes - 1 - i) % 2 == 0;
            float2* out = direct ? xy_s : (float2*)(ws + p.xy_at);
            int* wout = direct ? ids_s : (int*)(ws + p.w_at);
            k_rs_hist<<<p.ntiles, RS_THREADS, 0, st>>>(in, n, g, i * p.bits, p.nd, hist, p.ntiles);
            scan_exclusive_u32(hist, (int)p.nh, hist + p.nh, st);
            k_rs_scatter<<<p.ntiles, RS_THREADS, 0, st>>>(in, w, out, wout, last ? pos_of : nullptr, n, g,
                                                          i * p.bits, p.nd, hist, p.ntiles);
            in = out;
            w = wout;
        }
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    k_starts<<<nblk(nc + 1, ST_CELLS), ST_THREADS, 0, st>>>(xy_s, n, g, nc, start);
    return cudaGetLastError();
}

cudaError_t cell_mbrs(const float2* xy_s, const int* start, const Grid& g, float4* mbr, int* filled, cudaStream_t st)
{
    int nc = g.gx * g.gy;
    const cudaError_t e = cudaMemsetAsync(filled, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    k_mbr<<<nblk(nc, 256), 256, 0, st>>>(xy_s, start, nc, mbr, filled);
    return cudaGetLastError();
}

cudaError_t points_box(const float2* xy, int n, PointBox* box, int* bad, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    k_bbox<<<std::min(nblk(n, BB_THREADS), 8 * 152), BB_THREADS, 0, st>>>(xy, n, box, bad);
    return cudaGetLastError();
}

// Grid over [x0,x1]x[y0,y1] with about `per_cell` points per cell.
Grid make_grid(double x0, double y0, double x1, double y1, long long n, double per_cell, int max_side)
{
    Grid g;
    double w = x1 - x0, h = y1 - y0;
    double ext = w > h ? w : h;
    if (!(ext > 0)) ext = 1.0;
    double ww = w > 0 ? w : ext * 1e-3, hh = h > 0 ? h : ext * 1e-3;
    double cs = n > 0 ? sqrt(ww * hh * per_cell / (double)n) : ext;
    if (!(cs > 0)) cs = ext;
    if (ext / cs > max_side) cs = ext / max_side;
    float inv = (float)(1.0 / cs);
    g.x0 = (float)x0;
    g.y0 = (float)y0;
    g.inv = inv;
    g.cs = (float)(1.0 / (double)inv);
    // cells needed so that every coordinate maps inside without clamping
    g.gx = (int)floorf(((float)x1 - g.x0) * inv) + 1;
    g.gy = (int)floorf(((float)y1 - g.y0) * inv) + 1;
    if (g.gx < 1) g.gx = 1;
    if (g.gy < 1) g.gy = 1;
    return g;
}

}  // namespace rknn
