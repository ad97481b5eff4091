// Verification kernels: half-plane filter, exact recount, result finalize.
#pragma once
#include "rknn_common.cuh"

namespace rknn {

constexpr int VERIFY_UPT = 4;                       // default users per lane per work item
constexpr int VERIFY_CHUNK = 32 * VERIFY_UPT;       // default users per work item
constexpr int VERIFY_WARPS = 8;                     // default warps per block
constexpr int VERIFY_SAMPLES = 1024;                // work-item offsets cached per block
// FP32: whether boxes come first in a slot of n candidates.  Measured over 128
// users (ns of verification, 16,384 queries), user by user costs about 1 + 0.14 k
// (each user meets some 6 k half-planes before it is decided) and with boxes
// about 2.6 + 105 k / n (the fewer users a facility has, the wider their boxes):
// uniform layout with 10 users a facility k=60 9.9 / 9.9, k=80 13.0 / 10.9, with
// 50 k=7 1.9 / 3.7, k=24 3.9 / 4.1, street layout k=6 2.0 / 3.4, k=20 3.3 / 3.5.
// The line lies where both cost the same on these and on the clustered layout
// (k=16 160 / 162 us, k=32 297 / 272).
__host__ __device__ __forceinline__ bool boxes_first(int k, int n)
{
    return (float)k * (float)(n - 750) > 16.0f * (float)n;
}
// A batch whose largest k is beyond that line by a factor of two, at the 1.5
// candidates for each of the users that k facilities have (1.4 to 1.5 on uniform
// and street layouts), takes the boxes from this many candidates on instead:
// slots of both kinds side by side miss the instruction caches (verification of
// 16,384 queries of k from 1 to a largest one, us, so / by the line: street layout
// k to 24 547 / 416, to 50 864 / 997, to 100 1488 / 1787, 50 users a facility
// k to 32 432 / 346, to 64 684 / 746, clustered k to 50 860 / 839, to 100 1743 / 1840).
constexpr int BOX_MIN_CAND = 512;
// Most queries of an FP64 influence-zone batch, and candidates of a query, that
// go to the recount without a half-plane test.  The zone's half-planes reject
// about half of the candidates and accept none (its pruning may have dropped a
// needed facility, so those left are counted anyway), and a few queries leave
// most warps idle: counting all candidates takes the recount no longer, and the
// half-plane tests' chain is saved (one FP64 query at k=10: verification
// 26 -> 8 us; single queries at k=10, uniform 499 -> 468 us, clustered 571 -> 538,
// street 522 -> 490, ten at a time 563 -> 530, 1146 -> 1138, 646 -> 609).  In FP32
// the chain is short: one query takes 406 us either way, sixteen with 50 users a
// facility at k=3 229 listed, 223 tested.
constexpr int LIST_QUERIES = 16, LIST_CAND = 4096;
constexpr int VERIFY_PLANES_MAX = 1024;             // half-planes used per slot (32 box masks of 32)
constexpr int FIN_WARPS = 8;                        // finalize: slots per block (one warp each)
constexpr int FIN_WCAP = 512;                       // ids one warp sorts in registers

enum { MODE_FP64 = 0, MODE_FP32 = 1 };

struct VerifyArgs {
    const QDesc* qd;
    const float4* planes;    // [slot][lc] float half-planes relative to q
    const int* bis_pos;      // [slot][lc] facility positions (FP64 planes are rebuilt from these)
    int lc;                  // row stride of planes / bis_pos
    int stage_cap;           // half-planes used per slot, at most 1024 (the first ones;
                             // fewer only means more users reach the exact recount)
    int list_cand = -1;      // slots of up to this many candidates go to the recount whole
    bool box_batch = false;  // FP32: see BOX_MIN_CAND
    int parts = 1;           // parts of 32 * (users per lane) users in a work item
    const int2* segs;        // [slot][seg_cap]
    int seg_cap;
    int seg_stage = 0;       // user segments staged per warp beside the half-planes
                             // (a slot with more reads them from global memory)
    const int* chunk_off;    // [nq+1]
    const long long* cand_off;   // [nq] start of each slot's result region in res_pool
    const int* reg_len;          // [nq] its length (ids the slot stores at most)
    int nq;
    const float2* uxy;       // cell-sorted users
    const int* uid;          // their ids
    const float2* fxy;       // cell-sorted facilities
    const int* fstart;
    Grid gf;
    int* res_count;          // [nq]
    int* res_pool;           // results, region per slot
    int* work_counter;
    VStats* vstats;
    int mode;
    int nu, nf, ncf;         // array sizes (bounds-checked builds)
    long long pool_cap;
    int* dropped;            // set when a slot had more results than its region
    const float* slice_r;    // [slot][32] slice bounds (queries flagged QF_SLICE_R)
    int2* surv;              // survivors of the half-plane filter: (slot, user position)
    int surv_cap;            // 0: no list (the verification kernel recounts in-warp)
    int* surv_count;
    int* recount_counter = nullptr;    // recount_kernel's queue
    bool alike = false;      // an influence-zone batch: its survivors cost much the same
    int* fault;              // checked builds: {flag, array id, index, size, line}
    // slots to verify: chunk_off indexes deflist[0 .. *ndef) when deflist is
    // set (the fused slice filter verified the others), else slots 0 .. nq
    const int* deflist = nullptr;
    const int* ndef = nullptr;
    long long* region_top = nullptr;   // total of the result regions (fused claims)
    int* done = nullptr;               // fused filter: its blocks finished
};

__global__ void verify_kernel(VerifyArgs a);        // FP32, 4 users per lane per work item
__global__ void verify_kernel_u2(VerifyArgs a);     // 2
__global__ void verify_kernel_u8(VerifyArgs a);     // 8
__global__ void verify64_kernel(VerifyArgs a);      // FP64, 4 users per lane per work item
__global__ void verify64_kernel_u2(VerifyArgs a);   // 2
__global__ void verify64_kernel_u8(VerifyArgs a);   // 8

// Shared memory of one warp of a verification kernel: the box filter's
// staged half-planes (three doubles each at most), its masks, boxes and list
// of half-plane indices; the segments; the slice bounds.
constexpr int BOX_STAGE = 34;          // staged entries: one that decides nothing, 32 half-planes, padding
// FP32: half-planes a lane evaluates between two tests (street layout, ms: two
// 1.55, three 1.53, four 1.52, six 1.56)
constexpr int BOX_TRIP = 4;
constexpr int BOX_STAGE_BYTES = BOX_STAGE * 3 * (int)sizeof(double);
constexpr int BOX_MASK_BYTES = 4 * 32 * (int)sizeof(unsigned);
constexpr int BOX_QBOX_BYTES = 4 * 2 * (int)sizeof(float4);
__host__ __device__ __forceinline__ size_t verify_box_bytes(int stage_cap)
{
    return BOX_STAGE_BYTES + BOX_MASK_BYTES + BOX_QBOX_BYTES + (((size_t)stage_cap * sizeof(uint16_t) + 15) & ~(size_t)15);
}
__host__ __device__ __forceinline__ size_t verify_warp_bytes(int stage_cap, int seg_stage)
{
    const size_t b = verify_box_bytes(stage_cap) + (size_t)seg_stage * sizeof(int2) + 32 * sizeof(float);
    return (b + 15) & ~(size_t)15;
}

// exact recount of the listed survivors, a warp or a group of warps each
__global__ void recount_kernel(VerifyArgs a);       // FP32 filter
__global__ void recount64_kernel(VerifyArgs a);     // FP64 filter

// slots a block of the two scan kernels takes
constexpr int SCAN_THREADS = 1024;
inline int scan_blocks(int nq) { return (nq + SCAN_THREADS - 1) / SCAN_THREADS; }

// result regions (min(candidates, rcap) ids at 64-bit offsets, their lengths
// and *region_top = their total) and work-item offsets from the slots'
// candidate counts; flags slots whose region does not fit the pool
__global__ void plan_kernel(QDesc* qd, const int* ncand, int nq, long long* cand_off, int* reg_len,
                            long long* region_top, int* chunk_off, long long pool_cap, int rcap, int chunk);

// exclusive scan of the stored result counts into out_off
// out_off: nq+1 offsets, then OFF_TAIL ints: the region total (low and high
// halves of *region_top), the dropped flag and the listed survivors
// (counters[2], counters[3]), so that one copy brings back all of them.
constexpr int OFF_TAIL = 4;
// out_off_host (or null): device-accessible host memory that receives a
// copy of the same nq+1+OFF_TAIL ints.
__global__ void scan_counts_kernel(const int* res_count, const int* reg_len, const long long* region_top, int nq,
                                   int* out_off, const int* counters, int* out_off_host);

// Output offsets computed by finalize_kernel itself (batches of up to
// FIN_SCAN_MAX slots, which then need no scan_counts_kernel): each block sums
// the stored ids of the slots before its own, writes its slots' offsets to
// out_off (and out_off_host) and the last block the total and the run's
// flags, as scan_counts_kernel does.
constexpr int FIN_SCAN_MAX = 4096;
struct FinScan {
    int on = 0;
    int* out_off_host = nullptr;
    const long long* region_top = nullptr;
    const int* counters = nullptr;
    // sets above FIN_WCAP ids are listed here for sort_large_kernel (null:
    // sorted by their warps)
    int* large = nullptr;
    int* nlarge = nullptr;
    // a second copy of the sorted ids, in device-accessible host memory of
    // twin_cap ids (null: none; not with large): slots that would pass its end
    // are left out of it
    int* twin = nullptr;
    long long twin_cap = 0;
};

// Sets above FIN_WCAP ids, a block each (persistent blocks, *queue counts the
// slots taken after each block's first).  Launched for batches whose largest k
// gives SORT_MIN_MEAN results on average: below it large sets are few, and the
// launch would cost more than their warps' sorts.
// (finalize of the street workload, ms into host / device memory, by threads /
// tile / blocks an SM: 1024 / 16384 / 1 0.756 / 0.471, 1024 / 12288 / 1 0.770 /
// 0.485, 512 / 12288 / 2 0.770 / 0.405, 512 / 8192 / 2 0.793 / 0.489)
constexpr int SORT_BITS = 8, SORT_THREADS = 1024, SORT_TILE = 16384;
constexpr int SORT_MIN_MEAN = 1024;
__global__ void sort_large_kernel(int* res_pool, const long long* cand_off, const int* reg_len, const int* res_count,
                                  const int* out_off, int* out, int* stage, long long out_cap, const int* list,
                                  const int* nlist, int* queue);
size_t sort_large_smem();

// one block per slot: sort the slot's results into out[out_off[s] ...]
// out may be device-accessible host memory of out_cap ids: a slot whose range
// would pass out_cap is left out (the caller sees the total and fails the
// batch).  stage: device memory for every stored id (at least the total of
// the result regions), where large sets are sorted; it may be out itself.
// zero[0 .. zero_n) (another batch's counters, unused by this one) is cleared
// for the next batch.
__global__ void finalize_kernel(int* res_pool, const long long* cand_off, const int* reg_len, const int* res_count,
                                int* out_off, int* out, int* stage, int nq, long long out_cap, int* zero,
                                long long zero_n, FinScan S);
// the same with the second copy (S.twin)
__global__ void finalize_twin_kernel(int* res_pool, const long long* cand_off, const int* reg_len,
                                     const int* res_count, int* out_off, int* out, int* stage, int nq,
                                     long long out_cap, int* zero, long long zero_n, FinScan S);


}  // namespace rknn
