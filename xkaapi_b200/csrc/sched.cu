// Device-side ready-queue scheduler and the three execution forms of a resolved task graph.
//
// Reference behaviour replaced (XKRT, file:line): a task becomes ready when its wait counter
// reaches 0 (include/xkrt/task/task.hpp:518-551), is queued (src/sched.cc:413-455), executed
// by a device thread that launches its kernel (src/sched.cc:249-351, :469-505), and on
// completion decrements each successor's counter, queueing those that reach 0
// (src/task.cc:160-247).
//
//  * PERSISTENT: one kernel whose warps are the workers. A task is split into 2^k UNITS (column
//    slabs of a heat tile, pieces of an axpby range; k is fixed for a run, see split_log2). A
//    warp takes the next ticket (atomicAdd on head): unit (ticket mod 2^k) of task number
//    (ticket / 2^k). Two orders, chosen on the device before the run (sched_plan_kernel):
//      - IN ORDER, for graphs spawned level by level (the heat graphs): tasks are taken in spawn
//        order; a warp waits, with a time limit, for its task's counter of unfinished
//        predecessor units, runs the unit and decrements the successors' counters.
//      - QUEUE, for any graph: tasks are taken in the order they became ready. A warp waits for
//        a task id to be published in its queue slot; the warp that ends a task's last unit
//        decrements the successors' counters and publishes those that reach zero. Every slot
//        is written once (a task is pushed once): a plain array of ntasks slots.
//    Tile data written inside the kernel is read back with L1-bypassing loads.
//  * PLAIN: the host launches one kernel per task in spawn order (a topological order) on one
//    stream -- the reference's one-launch-per-task device path.
//  * GRAPH: the task graph becomes a CUDA graph (one kernel node per task, one edge per
//    dependency), instantiated once and replayed.
#include "common.cuh"
#include "heat.cuh"
#include "heat_bulk.cuh"
#include "internal.h"

#include <cuda.h>

#include <cmath>
#include <mutex>
#include <new>
#include <vector>

namespace xkb {

template <bool CG>
__device__ __forceinline__ double axpby1(double a, double x, double b, double y) { return __dadd_rn(__dmul_rn(a, x), __dmul_rn(b, y)); }

template <bool CG>
__device__ __forceinline__ void axpby_team(int64_t lo, int64_t hi, double a, const double * __restrict__ x,
                                           double b, double * __restrict__ y, int64_t tid, int64_t nth)
{
    if (lo >= hi) return;
    const bool same_phase = (((uintptr_t) (x + lo)) & 15) == (((uintptr_t) (y + lo)) & 15);
    int64_t head = lo;
    if (same_phase && (((uintptr_t) (y + lo)) & 15)) head = lo + 1;
    if (!same_phase) head = hi;
    if (head > hi) head = hi;
    for (int64_t i = lo + tid; i < head; i += nth)
        y[i] = axpby1<CG>(a, CG ? __ldcg(x + i) : __ldg(x + i), b, CG ? __ldcg(y + i) : y[i]);
    const int64_t nv = (hi - head) / 2;
    const double2 * xv = (const double2 *) (x + head);
    double2 * yv = (double2 *) (y + head);
    // Four vectors of each operand in flight per lane: with one (32 bytes per lane, 16 KB per SM
    // at 16 warps) a team waited out a DRAM round trip per step of the loop.
    int64_t v = tid;
    for (; v + 3 * nth < nv; v += 4 * nth)
    {
        double2 xx[4], yy[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            xx[k] = CG ? __ldcg(xv + v + k * nth) : __ldg(xv + v + k * nth);
            yy[k] = CG ? __ldcg(yv + v + k * nth) : yv[v + k * nth];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            yv[v + k * nth] = make_double2(axpby1<CG>(a, xx[k].x, b, yy[k].x), axpby1<CG>(a, xx[k].y, b, yy[k].y));
    }
    for (; v < nv; v += nth)
    {
        const double2 xx = CG ? __ldcg(xv + v) : __ldg(xv + v);
        const double2 yy = CG ? __ldcg(yv + v) : yv[v];
        yv[v] = make_double2(axpby1<CG>(a, xx.x, b, yy.x), axpby1<CG>(a, xx.y, b, yy.y));
    }
    for (int64_t i = head + 2 * nv + tid; i < hi; i += nth)
        y[i] = axpby1<CG>(a, CG ? __ldcg(x + i) : __ldg(x + i), b, CG ? __ldcg(y + i) : y[i]);
}

constexpr int SCHED_THREADS = 256;
// log2 of the units of one task that the warps of one CTA run together (team runs).
constexpr int TEAM_LOG2 = 3;
static_assert((1 << TEAM_LOG2) * 32 == SCHED_THREADS, "a team is a CTA");

constexpr int SCHED_BULK_NBUF = 8;       // staged columns in flight per warp (bulk tile body)
#ifndef XKB_TILE_PF
#define XKB_TILE_PF 5                    // east columns an FP32 tile strip loads ahead into registers (us per step of the 8192^2 graph: 3 104, 4 95, 5 95, 6 93, 8 93)
#endif
#ifndef XKB_F64_VEC
#define XKB_F64_VEC 4                    // rows per lane of the FP64 tile body: one warp covers 128 rows
#endif
#ifndef XKB_F64_PF
#define XKB_F64_PF 2                     // east columns the FP64 tile strip loads ahead (32 B per lane each)
#endif
#ifndef XKB_SCHED_MINB
#define XKB_SCHED_MINB 2                 // persistent CTAs resident per SM (register budget)
#endif
constexpr unsigned SCHED_POLL_NS = 100;  // between two looks at a counter or slot (20 or 200: within 1 %)
constexpr int SCHED_PFD_DEFAULT = 4;     // L2 prefetch distance of heat tiles in columns (3-5 measured best)
constexpr double SCHED_TIMEOUT_MAX_S = 3600.0;   // longest device wait a caller may ask for

// A device wait limit in seconds is usable when finite, positive and at most an hour.
static inline bool timeout_ok(double s) { return std::isfinite(s) && s > 0 && s <= SCHED_TIMEOUT_MAX_S; }

constexpr int TEAM_PF = 4;               // columns a strip of a team run loads ahead: its units are 4 to 16 columns wide
// Piece of an axpby range that unit `unit` of `nunits` runs: contiguous, a multiple of
// AXPBY_PIECE elements (so every piece keeps the range's alignment phase; the last one ends the
// range), empty for the units a short range does not need.
constexpr int64_t AXPBY_PIECE = 8192;    // 192 KiB of traffic: 30 us for one warp of a full device
__device__ __forceinline__ void axpby_piece(int64_t lo, int64_t hi, int unit, int nunits, int64_t & plo, int64_t & phi)
{
    const int64_t pieces = (hi - lo + AXPBY_PIECE - 1) / AXPBY_PIECE;
    const int64_t per = (pieces + nunits - 1) / nunits * AXPBY_PIECE;
    plo = lo + unit * per;
    phi = plo + per < hi ? plo + per : hi;
}

// Which task bodies a kernel holds. A kernel of one body keeps all of the SM's registers for it: with
// both heat bodies and the row-by-row strips in one kernel every tile pays for what the others spill:
// with the row-by-row strips of 3 and 4 columns ahead called from one kernel for all, the 8192^2 FP32
// graph took 132 us per step, alone 107; 8191 x 4001 (odd ld) FP32 123 against 68, FP64 135 against 99.
enum class Body { ANY, F64, F32, ROWS64, ROWS32, AXPBY };

// The kernel for tasks that need the bodies `seen` (XKB_BODY_*).
static inline Body body_for(unsigned seen)
{
    switch (seen)
    {
        case 0: case XKB_BODY_F64: return Body::F64;
        case XKB_BODY_F32: return Body::F32;
        case XKB_BODY_ROWS64: return Body::ROWS64;
        case XKB_BODY_ROWS32: return Body::ROWS32;
        case XKB_BODY_AXPBY: return Body::AXPBY;
        default: return Body::ANY;
    }
}

// Run unit `unit` of the `nunits` (a power of two) a task is split into, with one warp. PF64, PF32:
// columns a heat strip loads ahead into registers. A kernel of one body passes the other kinds by:
// the host chose it for tasks that have none.
template <Body B, int PF64, int PF32>
__device__ __forceinline__ void run_unit(const xkb_task_desc_t & d, int unit, int nunits, int pfd)
{
    const auto & h = d.u.heat;
    if constexpr (B == Body::ANY || B == Body::F64)
        if (d.kind == XKB_TASK_HEAT_F64)
        {
            const bool vok = (h.ld % 2 == 0) && (h.src % 16 == 0) && (h.dst % 16 == 0);
            heat_tile_team<double, XKB_F64_VEC, PF64, true>((const double *) h.src, (double *) h.dst, h.ld, h.nx, h.ny,
                                               h.x0, h.x1, h.y0, h.y1, h.c, vok, pfd, unit, nunits);
            return;
        }
    if constexpr (B == Body::ROWS64)
        if (d.kind == XKB_TASK_HEAT_F64)
            heat_tile_team<double, XKB_F64_VEC, ROWS_PF<double>, true, Strips::ROWS>((const double *) h.src, (double *) h.dst, h.ld, h.nx, h.ny,
                                               h.x0, h.x1, h.y0, h.y1, h.c, false, 0, unit, nunits);
    if constexpr (B == Body::ANY || B == Body::F32)
        if (d.kind == XKB_TASK_HEAT_F32)
        {
            const bool vok = (h.ld % 4 == 0) && (h.src % 16 == 0) && (h.dst % 16 == 0);
            // an FP32 column is half the bytes of an FP64 one: prefetch twice as many columns ahead
            heat_tile_team<float, 4, PF32, true>((const float *) h.src, (float *) h.dst, h.ld, h.nx, h.ny,
                                              h.x0, h.x1, h.y0, h.y1, h.c, vok, 2 * pfd, unit, nunits);
            return;
        }
    if constexpr (B == Body::ROWS32)
        if (d.kind == XKB_TASK_HEAT_F32)
            heat_tile_team<float, 4, ROWS_PF<float>, true, Strips::ROWS>((const float *) h.src, (float *) h.dst, h.ld, h.nx, h.ny,
                                              h.x0, h.x1, h.y0, h.y1, h.c, false, 0, unit, nunits);
    if constexpr (B == Body::ANY || B == Body::AXPBY)
        if (d.kind == XKB_TASK_AXPBY)
        {
            const auto & a = d.u.axpby;
            int64_t lo, hi;
            axpby_piece(a.lo, a.hi, unit, nunits, lo, hi);
            axpby_team<true>(lo, hi, a.a, (const double *) a.x, a.b, (double *) a.y, threadIdx.x & 31, 32);
        }
    // (XKB_TASK_NOOP: first-touch / placement tasks)
}

// Counters of a run (device memory): ready-queue tickets and tasks published, status, tasks
// executed; then what the seed kernel learnt about the tasks that are ready at the start, and of the kinds
// of all tasks (CTR_HEAT, CTR_AXPBY, CTR_PIECES of 64 bits; only where there may be axpby tasks).
// Head and tail have cache lines of their own: every warp's ticket and every release is an atomic there.
// CTR_EXECUTED counts units of an in-order run, tasks of a queue run (executed_tasks); a run goes in order
// when the plan kernel has left CTR_QUEUE and CTR_NEAR at 0 (run_in_order).
enum { CTR_HEAD = 0, CTR_TAIL = 32, CTR_STATUS = 48, CTR_EXECUTED, CTR_BAD_TASK, CTR_SEEDS, CTR_SEED_LAST, CTR_SEED_WIDTH, CTR_SEED_HEAT,
       CTR_HEAT, CTR_PIECES, CTR_PIECES_HI, CTR_AXPBY, CTR_QUEUE, CTR_NEAR, CTR_SPLIT, CTR_TEAM, CTR_RUN, CTR_COUNT };
static_assert(CTR_COUNT <= 64, "the no-allocation run's array has 64");
static_assert(CTR_PIECES % 2 == 0, "64 bits");

// A run covers `ntasks` tasks numbered w * period + t (window w, task t of the window's
// `period` descriptors). A plain graph is one window (period = ntasks); a periodic graph adds
// cross-window successors (xsucc) and a wait count for tasks of later windows (npred_next).
struct SchedArgs {
    const xkb_task_desc_t * tasks;
    uint32_t ntasks;
    uint32_t period;
    const uint32_t * succ_ptr;
    const uint32_t * succ;
    const uint32_t * xsucc_ptr;    // null for a plain graph
    const uint32_t * xsucc;
    const uint32_t * npred_first;
    const uint32_t * npred_next;
    int * wc;                  // wait counters; in a queue run, below 0: units of the task that ended
    int * queue;
    unsigned * ctr;            // CTR_*
    uint64_t timeout_ns;
    int pfd;                   // L2 prefetch distance of the tile bodies, in columns
    int allow_team;            // narrow graphs may go to sched_team_kernel
    unsigned bodies;           // the bodies the tasks need (XKB_BODY_*), as far as the host knows
    int units;                 // the caller's warps per task (xkb_sched_set_team): this many units; 0: chosen here,
    int min_units;             // at least this many
};

__global__ void sched_init_kernel(SchedArgs a)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.ntasks) return;
    a.queue[t] = -1;
    const uint32_t w = t / a.period, l = t - w * a.period;
    a.wc[t] = (int) (w == 0 ? a.npred_first[l] : a.npred_next[l]);
}

// Eighths of the tasks that seed l releases, as far as its successors show: each counts for its share of
// their predecessors, estimated on up to 16 of them. Few successors count an eighth each (a tile task has about
// eight that each wait for as many tasks), without a look at them.
__device__ __forceinline__ unsigned seed_width(const SchedArgs & a, uint32_t l)
{
    constexpr unsigned SAMPLE = 16;
    const uint32_t b = a.succ_ptr[l], deg = a.succ_ptr[l + 1] - b;
    if (deg <= SAMPLE) return deg;
    float share = 0;
#pragma unroll 8
    for (unsigned i = 0; i < SAMPLE; ++i)
    {
        const uint32_t s = a.succ[b + (uint64_t) deg * i / SAMPLE];
        if (s < a.period) share += 1.0f / (float) max(a.npred_first[s], 1u);
    }
    return (unsigned) fminf(8.0f / SAMPLE * share * (float) deg, 65536.0f);
}

__global__ void __launch_bounds__(256) sched_seed_kernel(SchedArgs a)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31;
    const bool ok = *(volatile unsigned *) (a.ctr + CTR_STATUS) == 0;   // a check before the run failed: nothing becomes ready
    const uint32_t w = t / a.period, l = t - w * a.period;
    const bool seed = ok && t < a.ntasks && (w == 0 ? a.npred_first[l] : a.npred_next[l]) == 0;
    const bool scan = a.bodies & XKB_BODY_AXPBY;           // (the host knows of heat tiles alone: no look at each task)
    bool heat = false;
    unsigned pieces = 0;
    if (seed || (scan && t < a.period && t < a.ntasks))
    {
        const xkb_task_desc_t & d = a.tasks[l];
        heat = d.kind == XKB_TASK_HEAT_F64 || d.kind == XKB_TASK_HEAT_F32;
        if (scan && w == 0 && d.kind == XKB_TASK_AXPBY)
            pieces = (unsigned) max(min((d.u.axpby.hi - d.u.axpby.lo + AXPBY_PIECE - 1) / AXPBY_PIECE, (int64_t) 65536), (int64_t) 1);
    }
    if (scan)
    {
        if (__syncthreads_or(heat) && threadIdx.x == 0 && *(volatile unsigned *) (a.ctr + CTR_HEAT) == 0) atomicExch(a.ctr + CTR_HEAT, 1u);
        const int naxpby = __syncthreads_count(pieces > 0);
        if (naxpby)
        {
            const unsigned sum = __reduce_add_sync(0xffffffffu, pieces);
            if (lane == 0 && sum) atomicAdd((unsigned long long *) (a.ctr + CTR_PIECES), (unsigned long long) sum);
            if (threadIdx.x == 0) atomicAdd(a.ctr + CTR_AXPBY, (unsigned) naxpby);
        }
    }
    const unsigned m = __ballot_sync(0xffffffffu, seed);
    if (!m) return;
    const unsigned width = __reduce_add_sync(0xffffffffu, seed ? seed_width(a, l) : 0u);
    const unsigned last = __reduce_max_sync(0xffffffffu, seed ? t + 1 : 0u);
    const unsigned nheat = __popc(__ballot_sync(0xffffffffu, seed && heat));
    unsigned pos = 0;
    if (lane == 0)
    {
        pos = atomicAdd(a.ctr + CTR_TAIL, (unsigned) __popc(m));
        atomicAdd(a.ctr + CTR_SEEDS, (unsigned) __popc(m));
        atomicMax(a.ctr + CTR_SEED_LAST, last);
        if (width) atomicAdd(a.ctr + CTR_SEED_WIDTH, width);
        if (nheat) atomicAdd(a.ctr + CTR_SEED_HEAT, nheat);
    }
    pos = __shfl_sync(0xffffffffu, pos, 0);
    if (seed) a.queue[pos + __popc(m & ((1u << lane) - 1))] = (int) t;
}

// log2 of the units a run's tasks are split into, from `width` = how many tasks the graph runs side
// by side, `heat` whether there are heat tiles among them, its `tasks`, the axpby ones' number `naxpby`
// and AXPBY_PIECE `pieces`, `warps` the run's workers, and the caller's least.
//  * heat tiles, few: as many units as there are warps, 32 at most (128^2 FP64 tiles, us per step:
//    64 tiles, 32 units of 4 columns 5.4, 16 units 7.6, one warp per tile 59; 256 tiles, 8 units
//    12.3, one warp 62);
//  * heat tiles, more than an eighth of the warps: up to two units per warp, 8 per tile at most, as
//    a warp alone does not keep its memory requests in flight (576 tiles: 28.5 with 8 units, 40.5
//    with 4, 70 with one; 1024 tiles: 45.3 with 4, 49.3 with 2, 49.7 with 8); a tile per warp or
//    more is not split (4096 tiles: 174 with one or two units);
//  * axpby: units of about AXPBY_PIECE elements, twice as many as the mean axpby task needs, so that
//    the largest chunk of a mixed graph spreads too (10 passes over 2^26 elements in chunks of 64 KiB
//    to 16 MiB: 2.5 ms against 142 ms with one warp per chunk). Every task gets as many units, empty ones
//    where it has no work for them, so where most tasks are not long axpby ones (more than four units per piece) the
//    units are fewer: until what they cost, about a sixteenth of a piece each, is no more than the pieces that
//    one unit of the mean axpby task runs.
constexpr int SPLIT_MAX_HEAT = 5, SPLIT_MAX = 8, PIECE_UNITS = 16;
__host__ __device__ __forceinline__ int split_log2(unsigned width, bool heat, uint64_t tasks, unsigned naxpby, uint64_t pieces,
                                                   unsigned warps, int min_units)
{
    int k = 0;
    if (heat)
    {
        while (k < SPLIT_MAX_HEAT && ((uint64_t) width << (k + 1)) <= warps) ++k;
        if (k < TEAM_LOG2) while (k < TEAM_LOG2 && ((uint64_t) width << (k + 1)) <= 2 * (uint64_t) warps) ++k;
    }
    if (pieces > naxpby)
    {
        const uint64_t mean = (pieces + naxpby - 1) / naxpby;
        int q = 0;
        while (q < SPLIT_MAX && (1ull << q) < 2 * mean) ++q;
        while (q > 0 && (tasks << q) > 4 * pieces && (tasks << 2 * q) > PIECE_UNITS * mean * warps) --q;
        if (q > k) k = q;
    }
    while ((1 << k) < min_units) ++k;
    return k;
}

// The split of a run, from the seed kernel's counters. The width is the number of tasks ready at the
// start, or what those release if that is more (a graph with one root and a wide second level).
__device__ __forceinline__ int run_split_log2(const SchedArgs & a, unsigned warps)
{
    const bool heat = a.bodies & XKB_BODY_AXPBY ? a.ctr[CTR_HEAT] != 0 : (a.bodies & XKB_BODY_ALL) != 0;
    int k = a.units ? (a.units == 8 ? 3 : a.units / 2)
                    : split_log2(max(a.ctr[CTR_SEEDS], a.ctr[CTR_SEED_WIDTH] / 8), heat, min(a.period, a.ntasks), a.ctr[CTR_AXPBY],
                                 *(unsigned long long *) (a.ctr + CTR_PIECES), warps, a.min_units);
    while (k > 0 && ((uint64_t) a.ntasks << k) > 0xf0000000ull) --k;      // tickets are 32-bit
    return k;
}

// Chooses the order of the run. Let W be the number of tasks ready at the start. The run goes in
// order when those are tasks 0 .. W-1, every edge leads from one block of W consecutive tasks to a
// later one, and every other task has a predecessor at most 2 W tasks before it (a heat tile, the same tile a
// step earlier, in graphs that begin inside a step too). Then the tasks of a block are independent
// of one another, and no task is ready more than 2 W tasks behind the last one taken, so spawn order keeps
// about as many tasks runnable as the queue could. (Without the last condition a graph with one root
// passes whatever follows: 64 chains of 100 tiles behind a common first task, spawned chain by chain,
// ran one after another, 10.4 ms against 5.7 through the queue.) In order, nothing is published, a warp
// knows its task -- descriptor and successors -- before it may run, and every unit decrements its
// successors itself, without waiting for the answer: 13.0 us per step of the 2048^2 FP64 graph against
// 18.5 through the queue with the same units, 176 against 187 for 8192^2, 661 against 725 for 16384^2.
// In order, a counter starts at the task's number of predecessors n and every one of their 2^k units
// takes one off, so the task may run at n - n * 2^k.
constexpr unsigned INORDER_MAX_NPRED = 1u << 20;      // keeps that inside an int

// Successor lists are looked at by their task's thread up to PLAN_LIST entries, and past them by the
// whole warp (60,000 successors of one task by one thread: 4 ms before the run).
constexpr uint32_t PLAN_LIST = 32;
constexpr int PLAN_BATCH = 12;           // successors looked at together (a tile has 9)

__global__ void __launch_bounds__(256) sched_plan_kernel(SchedArgs a, unsigned warps)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31;
    const bool mine = t < a.period;
    if (t == 0)
    {
        const int k = run_split_log2(a, warps);
        a.ctr[CTR_SPLIT] = (unsigned) k;
        a.ctr[CTR_TEAM] = a.allow_team && a.ctr[CTR_SEED_HEAT] > 0 && a.ctr[CTR_AXPBY] == 0 && k >= TEAM_LOG2 &&
                          ((uint64_t) a.ctr[CTR_SEEDS] << k) <= warps;
    }
    const uint32_t W = a.ctr[CTR_SEEDS];
    const bool level = W > 0 && a.ctr[CTR_SEED_LAST] == W && (a.xsucc_ptr == nullptr || a.period % W == 0);   // (the same for every thread)
    bool ok = level;
    if (level)
    {
        // tasks found to have a near predecessor are marked in the queue, whose places from W on are still
        // empty (anything below 0); CTR_NEAR ends at 0 when all of them were
        __shared__ unsigned marked;
        if (threadIdx.x == 0) marked = 0;
        __syncthreads();
        const uint32_t own = min(a.period, a.ntasks), ahead = a.ntasks > a.period ? min(W, a.ntasks - a.period) : 0u;
        if (t == 0) atomicSub(a.ctr + CTR_NEAR, (own > W ? own - W : 0u) + ahead);
        unsigned near = 0;
        // marks the near ones among N tasks behind `from`; every load is under way before one is looked at, and so
        // is every exchange (one edge after the other: 5 us more before each run)
        auto mark = [&](uint32_t from, const uint32_t (&to)[PLAN_BATCH], unsigned which) {
            int q[PLAN_BATCH];
#pragma unroll
            for (int j = 0; j < PLAN_BATCH; ++j) q[j] = which >> j & 1u && to[j] - from <= 2 * (uint64_t) W ? *(volatile int *) (a.queue + to[j]) : 0;
#pragma unroll
            for (int j = 0; j < PLAN_BATCH; ++j) q[j] = q[j] == -1 ? atomicExch(a.queue + to[j], -2) : 0;
#pragma unroll
            for (int j = 0; j < PLAN_BATCH; ++j) near += q[j] == -1;
        };
        // the successors [i, n) of task `from` that are `step` apart: whether all of them are in later blocks
        auto edges = [&](uint32_t from, uint32_t i, uint32_t n, uint32_t step) -> bool {
            bool later = true;
            for (; i < n; i += PLAN_BATCH * step)
            {
                uint32_t to[PLAN_BATCH];
                unsigned which = 0;
#pragma unroll
                for (int j = 0; j < PLAN_BATCH; ++j) to[j] = i + j * (uint64_t) step < n ? a.succ[i + j * step] : 0xffffffffu;
#pragma unroll
                for (int j = 0; j < PLAN_BATCH; ++j)
                {
                    const bool there = to[j] != 0xffffffffu, ok = to[j] / W > from / W;
                    later = later && (!there || ok);
                    which |= (there && ok && to[j] < own) << j;
                }
                mark(from, to, which);
            }
            return later;
        };
        const uint32_t b = mine ? a.succ_ptr[t] : 0u, e = mine ? a.succ_ptr[t + 1] : 0u;
        if (mine) ok = a.npred_first[t] < INORDER_MAX_NPRED && a.npred_next[t] < INORDER_MAX_NPRED;
        ok = edges(t, b, min(e, b + PLAN_LIST), 1) && ok;
        for (unsigned rest = __ballot_sync(0xffffffffu, e - b > PLAN_LIST); rest; rest &= rest - 1)
        {
            const int src = __ffs(rest) - 1;
            const uint32_t lb = __shfl_sync(0xffffffffu, b, src), le = __shfl_sync(0xffffffffu, e, src);
            const bool lok = __all_sync(0xffffffffu, edges(t - lane + (uint32_t) src, lb + PLAN_LIST + lane, le, 32));
            if ((int) lane == src) ok = ok && lok;
        }
        // into the next window: its first W tasks have no predecessor in their own
        if (mine && a.xsucc_ptr && ahead && t + 2 * (uint64_t) W >= a.period)
            for (uint32_t i = a.xsucc_ptr[t], n = a.xsucc_ptr[t + 1]; i < n; i += PLAN_BATCH)
            {
                uint32_t to[PLAN_BATCH];
                unsigned which = 0;
#pragma unroll
                for (int j = 0; j < PLAN_BATCH; ++j)
                {
                    const uint32_t x = i + j < n ? a.xsucc[i + j] : ahead;
                    to[j] = a.period + x;
                    which |= (x < ahead) << j;
                }
                mark(t, to, which);
            }
        if (near) atomicAdd(&marked, near);
        __syncthreads();
        if (threadIdx.x == 0 && marked) atomicAdd(a.ctr + CTR_NEAR, marked);
    }
    if (!mine) return;
    if (!ok && *(volatile unsigned *) (a.ctr + CTR_QUEUE) == 0) atomicExch(a.ctr + CTR_QUEUE, 1u);
    // the first place among the ready tasks where the tiles' rows change (block_order); ~ so that 0 is none
    if (ok && t + 1 < W && a.ctr[CTR_SEED_HEAT] == W && a.tasks[t].u.heat.x0 != a.tasks[t + 1].u.heat.x0)
        atomicMax(a.ctr + CTR_RUN, ~(t + 1));
}

// Order of the tasks of a block in an in-order run. Tiles spawned column by column within a row of
// tiles (the examples' loop: consecutive tasks work on the same 1 KB of every column) are taken row by
// row within a column of tiles instead, so that the tasks in flight read and write whole columns,
// which are contiguous (16384^2 FP64 graph 698 -> 658 us per step, 6.53 TB/s; 8192^2 175 -> 168). Any order of a block is valid, its tasks are
// independent; a part of a block keeps spawn order.
struct BlockOrder {
    uint32_t W, rows, cols, whole;         // tiles: rows x cols per block; tasks in whole blocks

    // blocks of rows x cols tiles spawned row of tiles by row of tiles, ntasks in whole blocks
    __device__ __forceinline__ BlockOrder(uint32_t rows_, uint32_t cols_, uint32_t ntasks) : W(rows_ * cols_), rows(rows_), cols(cols_), whole(ntasks) {}
    __device__ __forceinline__ BlockOrder(const SchedArgs & a)
    {
        W = a.ctr[CTR_SEEDS];
        const uint32_t run = a.ctr[CTR_RUN] ? ~a.ctr[CTR_RUN] : 0u;
        const bool grid = run > 1 && W % run == 0;
        cols = grid ? run : 1u;
        rows = grid ? W / run : 1u;
        whole = grid ? a.ntasks - a.ntasks % W : 0u;
    }
    __device__ __forceinline__ uint32_t task(uint32_t slot) const
    {
        if (slot >= whole) return slot;
        const uint32_t b = slot / W, p = slot - b * W, c = p / rows, r = p - c * rows;
        return b * W + r * cols + c;
    }
};

// Whether the run goes in order, from its counters.
__host__ __device__ __forceinline__ bool run_in_order(const unsigned * ctr) { return ctr[CTR_QUEUE] == 0 && ctr[CTR_NEAR] == 0; }

// Whether sched_team_kernel has the run.
__device__ __forceinline__ bool team_run(const SchedArgs & a) { return a.ctr[CTR_TEAM] != 0 && run_in_order(a.ctr); }

// Tasks run, from the counters of a run that ended.
__host__ __device__ __forceinline__ unsigned executed_tasks(const unsigned * ctr)
{
    return run_in_order(ctr) ? ctr[CTR_EXECUTED] >> ctr[CTR_SPLIT] : ctr[CTR_EXECUTED];
}

__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ __forceinline__ int atom_add_relaxed(int * p, int v)
{
    int old;
    asm volatile("atom.relaxed.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

__device__ __forceinline__ void red_add_relaxed(int * p, int v)
{
    asm volatile("red.relaxed.gpu.global.add.s32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}

// The successor graph of a run (see SchedArgs) and the entry i of a task's successors: those of
// its own window, then those of the next window. A successor at or beyond ntasks -- past the tail of
// the last window -- is not part of the run.
struct SuccGraph {
    const uint32_t * succ_ptr, * succ, * xsucc_ptr, * xsucc;
    uint32_t period, ntasks;

    __device__ __forceinline__ uint32_t count(uint32_t l) const
    {
        return succ_ptr[l + 1] - succ_ptr[l] + (xsucc_ptr ? xsucc_ptr[l + 1] - xsucc_ptr[l] : 0u);
    }
    __device__ __forceinline__ uint32_t entry(uint32_t l, uint32_t base, uint32_t i) const
    {
        const uint32_t b = succ_ptr[l], n = succ_ptr[l + 1] - b;
        return i < n ? base + succ[b + i] : base + period + xsucc[xsucc_ptr[l] + i - n];
    }
    // the lane's entry, loaded ahead (almost every task has at most 32 successors)
    __device__ __forceinline__ uint32_t first(uint32_t l, uint32_t base, int lane, bool & more) const
    {
        const uint32_t n = count(l);
        more = n > 32;
        return (uint32_t) lane < n ? entry(l, base, (uint32_t) lane) : 0xffffffffu;
    }
};

// One warp: decrement the counters of the tasks s (one per lane and place; none at or beyond ntasks) and
// publish those that became ready. The fence orders the writes of their other predecessors before the
// queue slot.
template <int N>
__device__ __forceinline__ void release_batch(const uint32_t (&s)[N], uint32_t ntasks, int * wc, int * queue, unsigned * tail, int lane)
{
    bool ready[N];
    unsigned m[N], total = 0;
#pragma unroll
    for (int j = 0; j < N; ++j) ready[j] = s[j] < ntasks && atom_add_relaxed(wc + s[j], -1) == 1;
#pragma unroll
    for (int j = 0; j < N; ++j) { m[j] = __ballot_sync(0xffffffffu, ready[j]); total += __popc(m[j]); }
    if (!total) return;
    fence_acq_rel_gpu();
    unsigned pos = 0;
    if (lane == 0) pos = atomicAdd(tail, total);
    pos = __shfl_sync(0xffffffffu, pos, 0);
#pragma unroll
    for (int j = 0; j < N; ++j)
    {
        if (ready[j])
            asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" :: "l"(queue + pos + __popc(m[j] & ((1u << lane) - 1))), "r"((int) s[j]) : "memory");
        pos += __popc(m[j]);
    }
}

// A task's successors past the first 32, four times 32 at a time: each batch waits out a load, an atomic, a
// fence and another atomic, 2 to 4 us, whatever its size (60,000 successors of one task: 8.3 ms 32 at a time).
__device__ __noinline__ void release_more(const SuccGraph g, uint32_t t, int * wc, int * queue, unsigned * tail, int lane)
{
    constexpr int N = 4;
    const uint32_t w = t / g.period, l = t - w * g.period, base = w * g.period;
    const uint32_t b = g.succ_ptr[l], own = g.succ_ptr[l + 1] - b, xb = g.xsucc_ptr ? g.xsucc_ptr[l] : 0u;
    const uint32_t n = own + (g.xsucc_ptr ? g.xsucc_ptr[l + 1] - xb : 0u);
    for (uint32_t i0 = 32; i0 < n; i0 += 32 * N)
    {
        uint32_t s[N];
#pragma unroll
        for (int j = 0; j < N; ++j)
        {
            const uint32_t i = i0 + 32 * j + lane;
            s[j] = i < own ? base + g.succ[b + i] : i < n ? base + g.period + g.xsucc[xb + i - own] : 0xffffffffu;
        }
        release_batch(s, g.ntasks, wc, queue, tail, lane);
    }
}

// One warp, after task t's last unit: release its successors, the lanes' entries of the first 32 loaded
// ahead. The caller's fence, by every lane, orders the writes of all of the task's units before the counters.
__device__ __forceinline__ void release_successors(const SuccGraph & g, uint32_t t, uint32_t first, bool more, int * wc, int * queue,
                                                   unsigned * tail, int lane)
{
    const uint32_t s[1] = {first};
    release_batch(s, g.ntasks, wc, queue, tail, lane);
    if (more) release_more(g, t, wc, queue, tail, lane);
}

// One warp, after a unit of task t of an in-order run.
__device__ __forceinline__ void count_down_successors(const SuccGraph & g, uint32_t t, uint32_t first, bool more, int * wc, int lane)
{
    if (first < g.ntasks) red_add_relaxed(wc + first, -1);
    if (!more) return;
    const uint32_t w = t / g.period, l = t - w * g.period, n = g.count(l);
    for (uint32_t i = 32 + lane; i < n; i += 32)
    {
        const uint32_t s = g.entry(l, w * g.period, i);
        if (s < g.ntasks) red_add_relaxed(wc + s, -1);
    }
}

// 64-byte descriptor as four independent 16-byte loads
__device__ __forceinline__ xkb_task_desc_t load_desc(const xkb_task_desc_t * p)
{
    static_assert(sizeof(xkb_task_desc_t) == 64, "descriptor size");
    union { int4 v[4]; xkb_task_desc_t d; } q;
#pragma unroll
    for (int k = 0; k < 4; ++k) q.v[k] = __ldg((const int4 *) p + k);
    return q.d;
}

// Wait (one lane) until *p <= target, polling with acquire loads; false when the time limit ran out
// here or anywhere (the status word, looked at now and then).
__device__ __forceinline__ bool wait_at_most(const int * p, int target, unsigned * status, uint64_t timeout_ns)
{
    if (xkb_ld_acquire(p) <= target) return true;
    const uint64_t t0 = xkb_globaltimer();
    for (uint32_t spins = 1;; ++spins)
    {
        __nanosleep(SCHED_POLL_NS);
        if (xkb_ld_acquire(p) <= target) return true;
        if ((spins & 63) == 0)
        {
            if (*(volatile unsigned *) status != 0) return false;
            if (xkb_globaltimer() - t0 > timeout_ns) { atomicCAS(status, 0u, (unsigned) -XKB_ETIMEDOUT); return false; }
        }
    }
}

// Wait (one lane) until queue slot *p holds a task id; -1 when the time limit ran out.
__device__ __forceinline__ int wait_published(const int * p, unsigned * status, uint64_t timeout_ns)
{
    int t = xkb_ld_acquire(p);
    if (t >= 0) return t;
    const uint64_t t0 = xkb_globaltimer();
    for (uint32_t spins = 1;; ++spins)
    {
        __nanosleep(SCHED_POLL_NS);
        if ((t = xkb_ld_acquire(p)) >= 0) return t;
        if ((spins & 63) == 0)
        {
            if (*(volatile unsigned *) status != 0) return -1;
            if (xkb_globaltimer() - t0 > timeout_ns) { atomicCAS(status, 0u, (unsigned) -XKB_ETIMEDOUT); return -1; }
        }
    }
}

// Warps never wait for one another except through the counters or the queue, so while one takes or
// releases a task the others keep HBM busy.
//
// BULK: heat tiles whose layout allows it run the bulk-staged body (heat_bulk.cuh): each warp
// streams its strips' columns through its own ring of shared-memory slots; other tasks run the
// register body.
// Dynamic shared memory of the BULK variant with NBUF slots per warp: the slots, then the mbarriers.
constexpr size_t bulk_smem_bytes(int nbuf) { return (size_t) (SCHED_THREADS / 32) * nbuf * (BULK_SLOT_BYTES + 8); }

template <Body B, bool BULK = false, int NBUF = SCHED_BULK_NBUF>
__global__ void __launch_bounds__(SCHED_THREADS, XKB_SCHED_MINB) sched_persistent_kernel(SchedArgs a)
{
    constexpr int NWARPS = SCHED_THREADS / 32;
    extern __shared__ __align__(128) unsigned char bulk_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool inorder = run_in_order(a.ctr);
    const int k = (int) a.ctr[CTR_SPLIT];
    const int nunits = 1 << k;
    unsigned executed = 0;
    BulkRing<NBUF> ring;
    if constexpr (BULK)
    {
        ring.slots = bulk_smem + (size_t) warp * NBUF * BULK_SLOT_BYTES;
        ring.bars = (uint64_t *) (bulk_smem + (size_t) NWARPS * NBUF * BULK_SLOT_BYTES) + warp * NBUF;
        bulk_ring_init(ring);
    }
    // (a check before the run that failed left its status: nothing runs)
    if (team_run(a) || *(volatile unsigned *) (a.ctr + CTR_STATUS) != 0) return;
    const BlockOrder order(a);
    unsigned ticket = 0;
    if (lane == 0) ticket = atomicAdd(a.ctr + CTR_HEAD, 1u);
    for (;;)
    {
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        const uint32_t slot = ticket >> k;
        const int unit = (int) (ticket & (nunits - 1));
        if (slot >= a.ntasks) break;
        int t = (int) order.task(slot);
        if (!inorder)
        {
            if (lane == 0) t = wait_published(a.queue + slot, a.ctr + CTR_STATUS, a.timeout_ns);
            t = __shfl_sync(0xffffffffu, t, 0);
            if (t < 0) break;
        }
        const uint32_t w = (uint32_t) t / a.period, l = (uint32_t) t - w * a.period;
        const xkb_task_desc_t d = load_desc(a.tasks + l);
        const SuccGraph g{a.succ_ptr, a.succ, a.xsucc_ptr, a.xsucc, a.period, a.ntasks};
        bool more;
        const uint32_t first = g.first(l, w * a.period, lane, more);
        if (inorder)
        {
            int ok = 1;
            if (lane == 0)
            {
                const int np = (int) (w == 0 ? a.npred_first[l] : a.npred_next[l]);
                ok = wait_at_most(a.wc + t, np - np * nunits, a.ctr + CTR_STATUS, a.timeout_ns);
            }
            if (!__shfl_sync(0xffffffffu, ok, 0)) break;
        }
        __syncwarp();
        if constexpr (BULK)
        {
            const auto & h = d.u.heat;
            // once a wait has run out anywhere, the remaining tasks are passed over quickly
            bool done = *(volatile unsigned *) (a.ctr + CTR_STATUS) != 0;
            if (d.kind == XKB_TASK_HEAT_F64 && bulk_ok<double, 2>((const double *) h.src, h.ld, h.nx) && h.dst % 16 == 0)
            {
                done = true;
                if (!heat_tile_team_bulk<double, 2, NBUF>((const double *) h.src, (double *) h.dst, h.ld, h.nx, h.ny, h.x0, h.x1,
                                                          h.y0, h.y1, h.c, unit, nunits, ring, xkb_globaltimer() + a.timeout_ns))
                    atomicCAS(a.ctr + CTR_STATUS, 0u, (unsigned) -XKB_ETIMEDOUT);
            }
            else if (d.kind == XKB_TASK_HEAT_F32 && bulk_ok<float, 4>((const float *) h.src, h.ld, h.nx) && h.dst % 16 == 0)
            {
                done = true;
                if (!heat_tile_team_bulk<float, 4, NBUF>((const float *) h.src, (float *) h.dst, h.ld, h.nx, h.ny, h.x0, h.x1,
                                                         h.y0, h.y1, h.c, unit, nunits, ring, xkb_globaltimer() + a.timeout_ns))
                    atomicCAS(a.ctr + CTR_STATUS, 0u, (unsigned) -XKB_ETIMEDOUT);
            }
            if (!done) run_unit<B, XKB_F64_PF, XKB_TILE_PF>(d, unit, nunits, a.pfd);
        }
        else
            run_unit<B, XKB_F64_PF, XKB_TILE_PF>(d, unit, nunits, a.pfd);
        // the next ticket arrives while the fence waits for the unit's stores
        if (lane == 0) ticket = atomicAdd(a.ctr + CTR_HEAD, 1u);
        __syncwarp();
        fence_acq_rel_gpu();
        if (inorder) count_down_successors(g, (uint32_t) t, first, more, a.wc, lane);
        else
        {
            if (k > 0)
            {
                // (the counter of a published task stands at 0, and counts its units from there on)
                int last = 0;
                if (lane == 0) last = atom_add_relaxed(a.wc + t, -1) == 1 - nunits;
                if (!__shfl_sync(0xffffffffu, last, 0)) continue;
                __syncwarp();
                // every lane decrements counters below, so every lane fences: the other units' writes, which
                // the count has shown to be done, come before its decrements too
                fence_acq_rel_gpu();
            }
            release_successors(g, (uint32_t) t, first, more, a.wc, a.queue, a.ctr + CTR_TAIL, lane);
        }
        ++executed;
    }
    if (lane == 0 && executed) atomicAdd(a.ctr + CTR_EXECUTED, executed);
}

// In-order runs of narrow heat graphs: the 8 warps of a CTA run 8 units of one task together. One
// thread takes the group's ticket and waits for the task's counter, one barrier before and one after
// the units, one fence and one round of counter updates for the group: an eighth of the polling,
// tickets and counter updates of one warp per unit, whose atomics are what bounds a step of a few
// microseconds (1024^2 FP64, 64 tiles of 32 units: 5.4 us per step against 11.2). Every run launches
// both kernels, and the one that does not have it returns at once.
template <Body B>
__global__ void __launch_bounds__(SCHED_THREADS, XKB_SCHED_MINB) sched_team_kernel(SchedArgs a)
{
    constexpr int NWARPS = SCHED_THREADS / 32;
    if (!team_run(a) || *(volatile unsigned *) (a.ctr + CTR_STATUS) != 0) return;
    __shared__ unsigned next_ticket;
    __shared__ int ready;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k = (int) a.ctr[CTR_SPLIT];
    const int nunits = 1 << k;
    const SuccGraph g{a.succ_ptr, a.succ, a.xsucc_ptr, a.xsucc, a.period, a.ntasks};
    unsigned executed = 0;
    if (threadIdx.x == 0) next_ticket = atomicAdd(a.ctr + CTR_HEAD, (unsigned) NWARPS);
    for (;;)
    {
        __syncthreads();                                       // the group's ticket
        const unsigned ticket = next_ticket;
        const uint32_t t = ticket >> k;
        const int unit = (int) (ticket & (nunits - 1)) + warp;
        if (t >= a.ntasks) break;
        const uint32_t w = t / a.period, l = t - w * a.period;
        const xkb_task_desc_t d = load_desc(a.tasks + l);
        uint32_t first = 0xffffffffu;
        bool more = false;
        if (warp == 0)
        {
            first = g.first(l, w * a.period, lane, more);
            if (lane == 0)
            {
                const int np = (int) (w == 0 ? a.npred_first[l] : a.npred_next[l]);
                ready = wait_at_most(a.wc + t, np - np * (nunits / NWARPS), a.ctr + CTR_STATUS, a.timeout_ns);
            }
        }
        __syncthreads();
        if (!ready) break;
        run_unit<B, TEAM_PF, TEAM_PF>(d, unit, nunits, 0);
        __syncthreads();                                       // the group's units are done
        ++executed;
        if (warp != 0) continue;
        if (lane == 0) next_ticket = atomicAdd(a.ctr + CTR_HEAD, (unsigned) NWARPS);
        fence_acq_rel_gpu();
        count_down_successors(g, t, first, more, a.wc, lane);
    }
    if (lane == 0 && executed) atomicAdd(a.ctr + CTR_EXECUTED, executed);
}

// Both kernels of a run (see sched_team_kernel); teams are of heat tiles only.
template <Body B>
static void launch_run(const SchedArgs & a, unsigned grid, cudaStream_t stream)
{
    sched_persistent_kernel<B><<<grid, SCHED_THREADS, 0, stream>>>(a);
    if constexpr (B != Body::AXPBY) sched_team_kernel<B><<<grid, SCHED_THREADS, 0, stream>>>(a);
}

// per-task kernels (PLAIN and GRAPH forms)
__global__ void __launch_bounds__(SCHED_THREADS, 2) task_kernel(xkb_task_desc_t d, int nslabs)
{
    // blockIdx.x selects a column slab of a heat tile / a chunk of an axpby range
    if (d.kind == XKB_TASK_HEAT_F64 || d.kind == XKB_TASK_HEAT_F32)
    {
        xkb_task_desc_t q = d;
        const int64_t cols = (int64_t) d.u.heat.y1 - d.u.heat.y0;
        const int64_t per = (cols + nslabs - 1) / nslabs;
        q.u.heat.y0 = (int32_t) (d.u.heat.y0 + blockIdx.x * per);
        { const int64_t e = (int64_t) q.u.heat.y0 + per; q.u.heat.y1 = (int32_t) (e < d.u.heat.y1 ? e : d.u.heat.y1); }
        if (q.u.heat.y0 >= q.u.heat.y1) return;
        if (d.kind == XKB_TASK_HEAT_F64) {
            const auto & h = q.u.heat;
            const bool vok = (h.ld % 2 == 0) && (h.src % 16 == 0) && (h.dst % 16 == 0);
            heat_tile_cta<double, 2, 4, false>((const double *) h.src, (double *) h.dst, h.ld, h.nx, h.ny, h.x0, h.x1, h.y0, h.y1, h.c, vok, 8);
        } else {
            const auto & h = q.u.heat;
            const bool vok = (h.ld % 4 == 0) && (h.src % 16 == 0) && (h.dst % 16 == 0);
            heat_tile_cta<float, 4, 4, false>((const float *) h.src, (float *) h.dst, h.ld, h.nx, h.ny, h.x0, h.x1, h.y0, h.y1, h.c, vok, 8);
        }
    }
    else if (d.kind == XKB_TASK_AXPBY)
    {
        const auto & a = d.u.axpby;
        const int64_t n = a.hi - a.lo, per = ((n + nslabs - 1) / nslabs + 1) & ~(int64_t) 1;
        const int64_t lo = a.lo + blockIdx.x * per;
        const int64_t hi = (lo + per < a.hi) ? lo + per : a.hi;
        axpby_team<false>(lo, hi, a.a, (const double *) a.x, a.b, (double *) a.y, threadIdx.x, blockDim.x);
    }
}

static int task_slabs(const xkb_task_desc_t & d)
{
    if (d.kind == XKB_TASK_HEAT_F64 || d.kind == XKB_TASK_HEAT_F32)
    {
        const int64_t cols = (int64_t) d.u.heat.y1 - d.u.heat.y0;
        return (int) std::max<int64_t>(1, (cols + 31) / 32);
    }
    if (d.kind == XKB_TASK_AXPBY)
    {
        const int64_t n = d.u.axpby.hi - d.u.axpby.lo;
        return (int) std::min<int64_t>(std::max<int64_t>(1, n / 4096), 1184);
    }
    return 1;
}

template <typename T>
struct Dev {
    T * p = nullptr; size_t cap = 0;
    ~Dev() { if (p) cudaFree(p); }
    int reserve(size_t n) {
        if (n <= cap) return XKB_OK;
        if (p) { cudaFree(p); p = nullptr; cap = 0; }
        cudaError_t e = cudaMalloc(&p, n * sizeof(T));
        if (e != cudaSuccess) return xkb_set_cuda_error(e);
        cap = n; return XKB_OK;
    }
};

} // namespace xkb

using namespace xkb;

struct xkb_sched {
    cudaStream_t stream = nullptr;
    std::vector<xkb_task_desc_t> host_tasks;  // host copy for the per-task forms (empty: device only)
    size_t ntasks = 0;                        // descriptors set
    unsigned bodies = XKB_BODY_ALL;           // the bodies they need
    Dev<xkb_task_desc_t> tasks;
    Dev<int> wc, queue;
    Dev<unsigned> ctr;
    Dev<unsigned long long> wsum;             // windows run without waiting: [0] first status, [1] executed
    cudaGraphExec_t gexec = nullptr;
    cudaGraph_t graph = nullptr;
    const void * graph_key = nullptr;
    int last_form = -1;
    int grid = 0;
    int team_warps = 0;                       // units (warps) per task, if the caller has set them
    int min_units = 1;                        // else at least this many
    int bulk = 0;                             // 1: bulk-staged heat tile body (measured slower; opt-in)
    int pfd = SCHED_PFD_DEFAULT;              // L2 prefetch distance in columns
    uint64_t last_total = 0;                  // tasks of the last run
    cudaEvent_t ev[2] = {nullptr, nullptr};   // around the persistent kernel of the last run
    uint64_t timeout_ns = 10ull * 1000 * 1000 * 1000;
    ~xkb_sched() {
        if (ev[0]) cudaEventDestroy(ev[0]);
        if (ev[1]) cudaEventDestroy(ev[1]);
        if (gexec) cudaGraphExecDestroy(gexec);
        if (graph) cudaGraphDestroy(graph);
    }
};

static int check_tasks(const xkb_task_desc_t * t, size_t n, unsigned & bodies)
{
    bodies = 0;
    for (size_t i = 0; i < n; ++i)
    {
        if (!xkb_internal_task_valid(t[i]))
        {
            const uint32_t k = t[i].kind;
            if (k == XKB_TASK_HEAT_F64 || k == XKB_TASK_HEAT_F32) return xkb_set_error(XKB_EINVAL, "sched: task %zu: bad heat tile", i);
            if (k == XKB_TASK_AXPBY) return xkb_set_error(XKB_EINVAL, "sched: task %zu: bad axpby range", i);
            return xkb_set_error(XKB_EINVAL, "sched: task %zu: unknown kind %u", i, k);
        }
        bodies |= xkb_internal_body_of(t[i]);
    }
    return XKB_OK;
}

extern "C" int xkb_sched_create(xkb_sched_t ** out, void * stream)
{
    if (!out) return xkb_set_error(XKB_EINVAL, "sched_create: null output");
    int dev;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return xkb_set_cuda_error(e);
    xkb_sched * S = new (std::nothrow) xkb_sched();
    if (!S) return xkb_set_error(XKB_ENOMEM, "sched_create: out of host memory");
    S->stream = (cudaStream_t) stream;
    int sms = 148, per = 2;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, sched_persistent_kernel<Body::ANY>, SCHED_THREADS, 0);
    S->grid = sms * (per > 0 ? per : 1);
    *out = S;
    return XKB_OK;
}

extern "C" int xkb_sched_destroy(xkb_sched_t * S)
{
    if (S) { cudaStreamSynchronize(S->stream); delete S; }
    return XKB_OK;
}

extern "C" int xkb_sched_set_tasks(xkb_sched_t * S, const xkb_task_desc_t * tasks, size_t ntasks)
{
    if (!S || (ntasks && !tasks)) return xkb_set_error(XKB_EINVAL, "sched_set_tasks: bad arguments");
    unsigned bodies;
    int rc = check_tasks(tasks, ntasks, bodies);
    if (rc) return rc;
    S->bodies = bodies;
    S->host_tasks.assign(tasks, tasks + ntasks);
    S->ntasks = ntasks;
    if ((rc = S->tasks.reserve(ntasks ? ntasks : 1))) return rc;
    if (ntasks) XKB_CUDA_TRY(cudaMemcpyAsync(S->tasks.p, tasks, ntasks * sizeof(xkb_task_desc_t), cudaMemcpyHostToDevice, S->stream));
    XKB_CUDA_TRY(cudaStreamSynchronize(S->stream));
    if (S->gexec) { cudaGraphExecDestroy(S->gexec); S->gexec = nullptr; }
    if (S->graph) { cudaGraphDestroy(S->graph); S->graph = nullptr; }
    S->graph_key = nullptr;
    return XKB_OK;
}

// Library-internal: the descriptors go to the device only (no host copy, so only the persistent
// forms can run them); for callers that hand over millions of descriptors for one run.
int xkb_internal_sched_set_tasks_device(xkb_sched_t * S, const xkb_task_desc_t * tasks, size_t ntasks, unsigned bodies)
{
    if (!S || (ntasks && !tasks)) return xkb_set_error(XKB_EINVAL, "sched_set_tasks: bad arguments");
    int rc;
    S->bodies = bodies;
    S->host_tasks.clear(); S->host_tasks.shrink_to_fit();
    S->ntasks = ntasks;
    if ((rc = S->tasks.reserve(ntasks ? ntasks : 1))) return rc;
    if (ntasks) XKB_CUDA_TRY(cudaMemcpyAsync(S->tasks.p, tasks, ntasks * sizeof(xkb_task_desc_t), cudaMemcpyHostToDevice, S->stream));
    XKB_CUDA_TRY(cudaStreamSynchronize(S->stream));
    if (S->gexec) { cudaGraphExecDestroy(S->gexec); S->gexec = nullptr; }
    if (S->graph) { cudaGraphDestroy(S->graph); S->graph = nullptr; }
    S->graph_key = nullptr;
    return XKB_OK;
}

extern "C" int xkb_sched_set_timeout(xkb_sched_t * S, double seconds)
{
    if (!S || !timeout_ok(seconds)) return xkb_set_error(XKB_EINVAL, "sched_set_timeout: the limit must be finite, above 0 and at most 3600 s");
    S->timeout_ns = (uint64_t) (seconds * 1e9);
    return XKB_OK;
}

extern "C" int xkb_sched_set_grid(xkb_sched_t * S, int ctas)
{
    if (!S || ctas <= 0) return xkb_set_error(XKB_EINVAL, "sched_set_grid: bad arguments");
    S->grid = ctas;
    return XKB_OK;
}

extern "C" int xkb_sched_set_prefetch(xkb_sched_t * S, int columns)
{
    if (!S || columns < 0 || columns > 256) return xkb_set_error(XKB_EINVAL, "sched_set_prefetch: 0..256 columns");
    S->pfd = columns;
    return XKB_OK;
}

extern "C" int xkb_sched_set_team(xkb_sched_t * S, int warps_per_task)
{
    if (!S || (warps_per_task != 1 && warps_per_task != 2 && warps_per_task != 4 && warps_per_task != 8))
        return xkb_set_error(XKB_EINVAL, "sched_set_team: warps per task must be 1, 2, 4 or 8");
    S->team_warps = warps_per_task;
    return XKB_OK;
}

void xkb_internal_sched_min_units(xkb_sched_t * S, int units) { if (S) S->min_units = units; }

extern "C" int xkb_sched_set_staging(xkb_sched_t * S, int bulk)
{
    if (!S || bulk < 0 || bulk > 1) return xkb_set_error(XKB_EINVAL, "sched_set_staging: 0 (register body) or 1 (bulk-staged body)");
    S->bulk = bulk;
    return XKB_OK;
}

static int launch_persistent(xkb_sched * S, SchedArgs & a);

static int launch_bulk(xkb_sched * S, SchedArgs & a)
{
    const size_t smem = bulk_smem_bytes(SCHED_BULK_NBUF);
    XKB_CUDA_TRY(cudaFuncSetAttribute(sched_persistent_kernel<Body::ANY, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    sched_persistent_kernel<Body::ANY, true><<<S->grid, SCHED_THREADS, smem, S->stream>>>(a);
    return XKB_OK;
}

// Working memory of runs of up to n tasks: wait counters, queue slots, counters.
static int reserve_run(xkb_sched * S, size_t n)
{
    if (n < 1) n = 1;
    int rc;
    if ((rc = S->wc.reserve(n)) || (rc = S->queue.reserve(n)) || (rc = S->ctr.reserve(CTR_COUNT))) return rc;
    return XKB_OK;
}

static SchedArgs run_args(xkb_sched * S, uint32_t ntasks, uint32_t period)
{
    SchedArgs a;
    a.tasks = S->tasks.p; a.ntasks = ntasks; a.period = period;
    a.wc = S->wc.p; a.queue = S->queue.p; a.ctr = S->ctr.p;
    a.timeout_ns = S->timeout_ns; a.pfd = S->pfd; a.units = S->team_warps; a.min_units = S->min_units;
    a.allow_team = !S->bulk; a.bodies = S->bodies;
    return a;
}

static void plain_graph(SchedArgs & a, const xkb_task_graph_t * g)
{
    a.succ_ptr = g->succ_ptr; a.succ = g->succ; a.xsucc_ptr = nullptr; a.xsucc = nullptr;
    a.npred_first = g->npred; a.npred_next = g->npred;
}

static int run_persistent(xkb_sched * S, const xkb_task_graph_t * g)
{
    const uint32_t n = (uint32_t) g->ntasks;
    if (int rc = reserve_run(S, n)) return rc;
    SchedArgs a = run_args(S, n, n ? n : 1);
    plain_graph(a, g);
    return launch_persistent(S, a);
}

static int launch_persistent(xkb_sched * S, SchedArgs & a)
{
    const uint32_t n = a.ntasks;
    XKB_CUDA_TRY(cudaMemsetAsync(S->ctr.p, 0, CTR_COUNT * sizeof(unsigned), S->stream));
    if (n)
    {
        sched_init_kernel<<<(n + 255) / 256, 256, 0, S->stream>>>(a);
        sched_seed_kernel<<<(n + 255) / 256, 256, 0, S->stream>>>(a);
        sched_plan_kernel<<<(a.period + 255) / 256, 256, 0, S->stream>>>(a, (unsigned) S->grid * (SCHED_THREADS / 32));
        if (!S->ev[0]) { XKB_CUDA_TRY(cudaEventCreate(&S->ev[0])); XKB_CUDA_TRY(cudaEventCreate(&S->ev[1])); }
        XKB_CUDA_TRY(cudaEventRecord(S->ev[0], S->stream));
        if (S->bulk)
        {
            int rc = launch_bulk(S, a);
            if (rc) return rc;
        }
        else
            switch (body_for(S->bodies))
            {
                case Body::F64: launch_run<Body::F64>(a, S->grid, S->stream); break;
                case Body::F32: launch_run<Body::F32>(a, S->grid, S->stream); break;
                case Body::ROWS64: launch_run<Body::ROWS64>(a, S->grid, S->stream); break;
                case Body::ROWS32: launch_run<Body::ROWS32>(a, S->grid, S->stream); break;
                case Body::AXPBY: launch_run<Body::AXPBY>(a, S->grid, S->stream); break;
                default: launch_run<Body::ANY>(a, S->grid, S->stream);
            }
        XKB_CUDA_TRY(cudaEventRecord(S->ev[1], S->stream));
    }
    XKB_CUDA_TRY(cudaGetLastError());
    return XKB_OK;
}

static int run_plain(xkb_sched * S)
{
    for (const xkb_task_desc_t & d : S->host_tasks)
    {
        if (d.kind == XKB_TASK_NOOP) continue;
        task_kernel<<<task_slabs(d), SCHED_THREADS, 0, S->stream>>>(d, task_slabs(d));
    }
    XKB_CUDA_TRY(cudaGetLastError());
    return XKB_OK;
}

static int build_cuda_graph(xkb_sched * S, const xkb_task_graph_t * g)
{
    const size_t n = S->host_tasks.size();
    std::vector<uint32_t> ptr(n + 1), succ(g->nedges);
    XKB_CUDA_TRY(cudaMemcpy(ptr.data(), g->succ_ptr, (n + 1) * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    if (g->nedges) XKB_CUDA_TRY(cudaMemcpy(succ.data(), g->succ, g->nedges * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    cudaGraph_t graph;
    XKB_CUDA_TRY(cudaGraphCreate(&graph, 0));
    std::vector<cudaGraphNode_t> nodes(n);
    for (size_t i = 0; i < n; ++i)
    {
        xkb_task_desc_t d = S->host_tasks[i];
        int slabs = task_slabs(d);
        void * args[2] = {&d, &slabs};
        cudaKernelNodeParams p = {};
        p.func = (void *) task_kernel;
        p.gridDim = dim3(d.kind == XKB_TASK_NOOP ? 1 : slabs);
        p.blockDim = dim3(SCHED_THREADS);
        p.kernelParams = args;
        cudaError_t e = cudaGraphAddKernelNode(&nodes[i], graph, nullptr, 0, &p);
        if (e != cudaSuccess) { cudaGraphDestroy(graph); return xkb_set_cuda_error(e); }
    }
    std::vector<cudaGraphNode_t> from, to;
    from.reserve(g->nedges); to.reserve(g->nedges);
    for (size_t t = 0; t < n; ++t)
        for (uint32_t i = ptr[t]; i < ptr[t + 1]; ++i) { from.push_back(nodes[t]); to.push_back(nodes[succ[i]]); }
    if (!from.empty())
    {
        cudaError_t e = cudaGraphAddDependencies(graph, from.data(), to.data(), from.size());
        if (e != cudaSuccess) { cudaGraphDestroy(graph); return xkb_set_cuda_error(e); }
    }
    cudaGraphExec_t exec;
    cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
    if (e != cudaSuccess) { cudaGraphDestroy(graph); return xkb_set_cuda_error(e); }
    if (S->gexec) cudaGraphExecDestroy(S->gexec);
    if (S->graph) cudaGraphDestroy(S->graph);
    S->graph = graph; S->gexec = exec; S->graph_key = g->succ;
    return XKB_OK;
}

extern "C" int xkb_sched_run(xkb_sched_t * S, const xkb_task_graph_t * g, int form)
{
    if (!S || !g) return xkb_set_error(XKB_EINVAL, "sched_run: bad arguments");
    if (g->ntasks != S->ntasks)
        return xkb_set_error(XKB_EINVAL, "sched_run: graph has %llu tasks, %zu descriptors set",
                             (unsigned long long) g->ntasks, S->ntasks);
    if (form != XKB_FORM_PERSISTENT && S->host_tasks.size() != S->ntasks)
        return xkb_set_error(XKB_EINVAL, "sched_run: the descriptors were set for the persistent form only");
    S->last_form = form;
    S->last_total = g->ntasks;
    switch (form)
    {
        case XKB_FORM_PERSISTENT: return run_persistent(S, g);
        case XKB_FORM_PLAIN: return run_plain(S);
        case XKB_FORM_GRAPH:
            if (!S->gexec || S->graph_key != g->succ) { int rc = build_cuda_graph(S, g); if (rc) return rc; }
            XKB_CUDA_TRY(cudaGraphLaunch(S->gexec, S->stream));
            return XKB_OK;
        default: return xkb_set_error(XKB_EINVAL, "sched_run: unknown form %d", form);
    }
}

extern "C" int xkb_sched_run_periodic(xkb_sched_t * S, const xkb_periodic_graph_t * g, uint32_t repeats, uint32_t tail)
{
    if (!S || !g || repeats == 0 || tail == 0 || tail > g->period)
        return xkb_set_error(XKB_EINVAL, "sched_run_periodic: bad arguments");
    if (g->period != S->ntasks)
        return xkb_set_error(XKB_EINVAL, "sched_run_periodic: period %llu but %zu descriptors set",
                             (unsigned long long) g->period, S->ntasks);
    const uint64_t total = (uint64_t) (repeats - 1) * g->period + tail;
    if (total >= (1ull << 31)) return xkb_set_error(XKB_ERANGE, "sched_run_periodic: %llu tasks in one run", (unsigned long long) total);
    if (int rc = reserve_run(S, total)) return rc;
    SchedArgs a = run_args(S, (uint32_t) total, (uint32_t) g->period);
    a.succ_ptr = g->succ_ptr; a.succ = g->succ; a.xsucc_ptr = g->xsucc_ptr; a.xsucc = g->xsucc;
    a.npred_first = g->npred_first; a.npred_next = g->npred_next;
    S->last_form = XKB_FORM_PERSISTENT;
    S->last_total = total;
    return launch_persistent(S, a);
}

// Fold one launch's status and executed count into the windows' running totals.
__global__ void window_status_kernel(const unsigned * __restrict__ ctr, unsigned long long * sum)
{
    if (threadIdx.x != 0) return;
    if (sum[0] == 0 && ctr[CTR_STATUS] != 0) sum[0] = ctr[CTR_STATUS];
    sum[1] += executed_tasks(ctr);
}

int xkb_internal_sched_reserve(xkb_sched_t * S, size_t ntasks)
{
    if (!S) return xkb_set_error(XKB_EINVAL, "sched_reserve: null scheduler");
    int rc;
    if ((rc = S->tasks.reserve(ntasks)) || (rc = reserve_run(S, ntasks))) return rc;
    if (!S->wsum.p)
    {
        if ((rc = S->wsum.reserve(2))) return rc;
        XKB_CUDA_TRY(cudaMemsetAsync(S->wsum.p, 0, 2 * sizeof(unsigned long long), S->stream));
    }
    return XKB_OK;
}

int xkb_internal_sched_upload_window(xkb_sched_t * S, const xkb_task_desc_t * tasks, size_t ntasks, unsigned bodies)
{
    if (!S || (ntasks && !tasks) || ntasks >= (size_t(1) << 31)) return xkb_set_error(XKB_EINVAL, "sched_upload_window: bad arguments");
    int rc;
    if (ntasks > S->tasks.cap || ntasks > S->wc.cap || ntasks > S->queue.cap)
    {
        // earlier windows may still be reading these buffers
        XKB_CUDA_TRY(cudaStreamSynchronize(S->stream));
        const size_t c = ntasks + ntasks / 2;
        if ((rc = S->tasks.reserve(c)) || (rc = reserve_run(S, c))) return rc;
    }
    if (ntasks) XKB_CUDA_TRY(cudaMemcpyAsync(S->tasks.p, tasks, ntasks * sizeof(xkb_task_desc_t), cudaMemcpyHostToDevice, S->stream));
    S->host_tasks.clear();
    S->ntasks = ntasks;
    S->bodies = bodies;
    S->graph_key = nullptr;
    return XKB_OK;
}

int xkb_internal_sched_launch_window(xkb_sched_t * S, const xkb_task_graph_t * g)
{
    if (!S || !g || g->ntasks != S->ntasks) return xkb_set_error(XKB_EINVAL, "sched_launch_window: the graph and the uploaded window differ");
    int rc;
    if (!S->wsum.p)
    {
        if ((rc = S->wsum.reserve(2))) return rc;
        XKB_CUDA_TRY(cudaMemsetAsync(S->wsum.p, 0, 2 * sizeof(unsigned long long), S->stream));
    }
    const size_t ntasks = S->ntasks;
    if (ntasks == 0) return XKB_OK;
    if ((rc = reserve_run(S, ntasks))) return rc;      // (no-op: xkb_internal_sched_upload_window made room)
    SchedArgs a = run_args(S, (uint32_t) ntasks, (uint32_t) ntasks);
    plain_graph(a, g);
    if ((rc = launch_persistent(S, a))) return rc;
    window_status_kernel<<<1, 32, 0, S->stream>>>(S->ctr.p, S->wsum.p);
    XKB_CUDA_TRY(cudaGetLastError());
    S->last_form = XKB_FORM_PERSISTENT;
    S->last_total = ntasks;
    return XKB_OK;
}

int xkb_internal_sched_run_window(xkb_sched_t * S, const xkb_task_desc_t * tasks, size_t ntasks, unsigned bodies, const xkb_task_graph_t * g)
{
    if (!S || (ntasks && !tasks) || !g || g->ntasks != ntasks || ntasks >= (size_t(1) << 31))
        return xkb_set_error(XKB_EINVAL, "sched_run_window: bad arguments");
    int rc = xkb_internal_sched_upload_window(S, tasks, ntasks, bodies);
    return rc ? rc : xkb_internal_sched_launch_window(S, g);
}

int xkb_internal_sched_windows_wait(xkb_sched_t * S, uint64_t * executed)
{
    if (!S) return xkb_set_error(XKB_EINVAL, "sched_windows_wait: null scheduler");
    XKB_CUDA_TRY(cudaStreamSynchronize(S->stream));
    unsigned long long sum[2] = {0, 0};
    if (S->wsum.p)
    {
        XKB_CUDA_TRY(cudaMemcpy(sum, S->wsum.p, sizeof(sum), cudaMemcpyDeviceToHost));
        XKB_CUDA_TRY(cudaMemset(S->wsum.p, 0, sizeof(sum)));
    }
    if (executed) *executed = sum[1];
    if (sum[0] != 0) return xkb_set_error(-(int) sum[0], "sched: a device wait ran out of time in a window run");
    return XKB_OK;
}

extern "C" int xkb_sched_wait(xkb_sched_t * S, uint64_t * executed)
{
    if (!S) return xkb_set_error(XKB_EINVAL, "sched_wait: null scheduler");
    XKB_CUDA_TRY(cudaStreamSynchronize(S->stream));
    unsigned ctr[CTR_COUNT] = {};
    ctr[CTR_EXECUTED] = (unsigned) S->last_total;               // the other forms count nothing
    if (S->ctr.p && S->last_form == XKB_FORM_PERSISTENT) XKB_CUDA_TRY(cudaMemcpy(ctr, S->ctr.p, sizeof(ctr), cudaMemcpyDeviceToHost));
    if (executed) *executed = executed_tasks(ctr);
    if (ctr[CTR_STATUS] != 0)
        return xkb_set_error(-(int) ctr[CTR_STATUS], "sched: a device wait ran out of time (%u of %llu tasks ran)", executed_tasks(ctr),
                             (unsigned long long) S->last_total);
    return XKB_OK;
}

extern "C" int xkb_sched_kernel_ms(xkb_sched_t * S, double * ms)
{
    if (!S || !ms) return xkb_set_error(XKB_EINVAL, "sched_kernel_ms: bad arguments");
    *ms = 0;
    if (S->last_form != XKB_FORM_PERSISTENT || !S->ev[0]) return XKB_OK;
    float f = 0;
    XKB_CUDA_TRY(cudaEventSynchronize(S->ev[1]));
    XKB_CUDA_TRY(cudaEventElapsedTime(&f, S->ev[0], S->ev[1]));
    *ms = f;
    return XKB_OK;
}

// ------------------------------------------------------------------------------------------
// Persistent run without any allocation.
//
// Some callers cannot allocate device memory when they run a graph: a task runtime that has
// reserved most of the GPU's memory for its own allocator at start-up (XKRT reserves 90 % of
// HBM for its device memory areas), or a serving loop whose device memory is already carved
// into fixed pools, gets a failed or competing cudaMalloc; and cudaMalloc/cudaFree can
// synchronise the device in the middle of a latency-critical loop. This entry point keeps the
// scheduler's working set -- wait counters, queue slots and the run's counters -- in the file-scope
// array below instead, sized for at most XKB_NOALLOC_MAX_TASKS tasks (8 MiB + 256 B held by
// every GPU that loads the library, until the process exits).
static __device__ __align__(256) int g_sched_noalloc_scratch[2 * XKB_NOALLOC_MAX_TASKS + 64];   // + counters

// (the counters CTR_* stand after the wait counters and the queue; CTR_BAD_TASK is the lowest task
// index whose descriptor failed the check)

// Every descriptor of a no-allocation run is checked on the device with the host checks of
// xkb_sched_set_tasks before anything runs: a bad one sets the status to XKB_EINVAL, records
// the lowest such index, and the seed kernel then makes no task ready, so no tile is touched.
__global__ void noalloc_check_kernel(const xkb_task_desc_t * __restrict__ tasks, uint32_t n, unsigned * ctr)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    if (!xkb_internal_task_valid(tasks[t]))
    {
        atomicCAS(ctr + CTR_STATUS, 0u, (unsigned) -XKB_EINVAL);
        atomicMin(ctr + CTR_BAD_TASK, t);
    }
}

// Device address of the scratch array in the current context. In host code the array's name
// only stands for it; its device address is looked up with the device current, on the first
// call made in each CUDA context (a context destroyed by cudaDeviceReset and made again gets a
// fresh lookup). The same set-up loads the kernels the run launches, so that with lazy module
// loading a later call needs no module memory either.
struct NoallocSlot { CUcontext ctx = nullptr; int * ptr = nullptr; };

static int noalloc_scratch(int ** out)
{
    static std::mutex mu;
    static NoallocSlot slots[256];
    static CUresult (*ctx_current)(CUcontext *) = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        cudaDriverEntryPointQueryResult q;
        void * f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            ctx_current = (CUresult (*)(CUcontext *)) f;
        else
            cudaGetLastError();
    });
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return xkb_set_cuda_error(e);
    if (dev < 0 || dev >= 256) return xkb_set_error(XKB_ENODEV, "sched_run_noalloc: device %d out of range", dev);
    e = cudaSetDevice(dev);                     // makes the device's primary context current (CUDA 12)
    if (e != cudaSuccess) return xkb_set_cuda_error(e);
    CUcontext ctx = nullptr;
    if (!ctx_current || ctx_current(&ctx) != CUDA_SUCCESS || !ctx)
        return xkb_set_error(XKB_ENODEV, "sched_run_noalloc: no current CUDA context on device %d", dev);
    std::lock_guard<std::mutex> lock(mu);
    NoallocSlot & sl = slots[dev];
    if (sl.ctx != ctx || !sl.ptr)
    {
        void * p = nullptr;
        e = cudaGetSymbolAddress(&p, g_sched_noalloc_scratch);
        if (e != cudaSuccess) return xkb_set_cuda_error(e);
        cudaFuncAttributes fa;
        const void * kernels[] = {(const void *) noalloc_check_kernel, (const void *) sched_init_kernel,
                                  (const void *) sched_seed_kernel, (const void *) sched_plan_kernel,
                                  (const void *) sched_persistent_kernel<Body::ANY>, (const void *) sched_team_kernel<Body::ANY>};
        for (const void * k : kernels)
            if ((e = cudaFuncGetAttributes(&fa, k)) != cudaSuccess) return xkb_set_cuda_error(e);
        sl.ctx = ctx;
        sl.ptr = (int *) p;
    }
    *out = sl.ptr;
    return XKB_OK;
}

extern "C" int xkb_sched_run_noalloc(const xkb_task_desc_t * tasks, const xkb_task_graph_t * graph, int warps_per_task,
                                     double timeout_s, void * stream, uint64_t * executed)
{
    if (!graph || (graph->ntasks && (!tasks || !graph->succ_ptr || !graph->npred)))
        return xkb_set_error(XKB_EINVAL, "sched_run_noalloc: bad arguments");
    if (!timeout_ok(timeout_s))
        return xkb_set_error(XKB_EINVAL, "sched_run_noalloc: the time limit must be finite, above 0 and at most 3600 s");
    if (warps_per_task != 1 && warps_per_task != 2 && warps_per_task != 4 && warps_per_task != 8)
        return xkb_set_error(XKB_EINVAL, "sched_run_noalloc: warps per task must be 1, 2, 4 or 8");
    if (graph->ntasks > XKB_NOALLOC_MAX_TASKS)
        return xkb_set_error(XKB_ERANGE, "sched_run_noalloc: %llu tasks exceed the fixed capacity of %u tasks",
                             (unsigned long long) graph->ntasks, (unsigned) XKB_NOALLOC_MAX_TASKS);
    int * scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    cudaStream_t st = xkb_stream(stream);
    const uint32_t n = (uint32_t) graph->ntasks;
    SchedArgs a;
    a.tasks = tasks; a.ntasks = n; a.period = n ? n : 1; a.succ_ptr = graph->succ_ptr; a.succ = graph->succ;
    a.xsucc_ptr = nullptr; a.xsucc = nullptr; a.npred_first = graph->npred; a.npred_next = graph->npred;
    a.wc = scratch; a.queue = scratch + XKB_NOALLOC_MAX_TASKS;
    a.units = 0; a.min_units = warps_per_task;
    a.allow_team = 1; a.bodies = XKB_BODY_ALL;
    a.ctr = (unsigned *) (scratch + 2 * XKB_NOALLOC_MAX_TASKS);
    a.timeout_ns = (uint64_t) (timeout_s * 1e9);
    a.pfd = SCHED_PFD_DEFAULT;
    // the array keeps the previous call's contents: the counters are cleared here (the lowest bad
    // index to all ones), and the init kernel rewrites every wait counter and queue slot this run uses
    XKB_CUDA_TRY(cudaMemsetAsync(a.ctr, 0, CTR_COUNT * sizeof(unsigned), st));
    XKB_CUDA_TRY(cudaMemsetAsync(a.ctr + CTR_BAD_TASK, 0xff, sizeof(unsigned), st));
    if (n)
    {
        int dev = 0, sms = 148, per = 2;
        XKB_CUDA_TRY(cudaGetDevice(&dev));
        XKB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        XKB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, sched_persistent_kernel<Body::ANY>, SCHED_THREADS, 0));
        const unsigned grid = (unsigned) (sms * (per > 0 ? per : 1));
        noalloc_check_kernel<<<(n + 255) / 256, 256, 0, st>>>(tasks, n, a.ctr);
        sched_init_kernel<<<(n + 255) / 256, 256, 0, st>>>(a);
        sched_seed_kernel<<<(n + 255) / 256, 256, 0, st>>>(a);
        sched_plan_kernel<<<(n + 255) / 256, 256, 0, st>>>(a, grid * (SCHED_THREADS / 32));
        launch_run<Body::ANY>(a, grid, st);
        XKB_CUDA_TRY(cudaGetLastError());
    }
    unsigned ctr[CTR_COUNT] = {};
    XKB_CUDA_TRY(cudaMemcpyAsync(ctr, a.ctr, sizeof(ctr), cudaMemcpyDeviceToHost, st));
    XKB_CUDA_TRY(cudaStreamSynchronize(st));
    if (executed) *executed = executed_tasks(ctr);
    if (ctr[CTR_STATUS] == (unsigned) -XKB_EINVAL)
        return xkb_set_error(XKB_EINVAL, "sched_run_noalloc: task %u: bad descriptor (unknown kind, bad heat tile or axpby range); nothing ran", ctr[CTR_BAD_TASK]);
    if (ctr[CTR_STATUS] != 0)
        return xkb_set_error(-(int) ctr[CTR_STATUS], "sched_run_noalloc: a device wait ran out of time (%u of %u tasks ran)", executed_tasks(ctr), n);
    return XKB_OK;
}

// ------------------------------------------------------------------------------------------
// Device-resident serving loop: ONE persistent kernel runs the tile tasks of every admitted
// request. The host admits a request by writing its slot record (descriptors, periodic graph,
// counter array, the grid to duplicate) and then the slot's state word. Idle CTAs take the slot's
// set-up chunks (wait counters, second grid), and the one that finishes the last chunk starts the
// request. From then on idle CTAs ATTACH to it, as many as its steps can keep busy or its share of the
// device when requests compete, and run it like an in-order batch run (the heat graph is spawned level
// by level): tickets from the slot's counter, a wait for the task's predecessors, the unit, the
// successors' counters -- a CTA at a time where a task has 8 units or more, else warp by warp. A CTA
// leaves when the tickets run out, or between tickets when its request holds more than its share (a
// look every SRV_LOOK_NS); the one that counts the last unit marks the slot done and reports the
// admission number to mapped host memory, and the host copies the result out. CTAs stop when the host
// has said no request will come and every slot is idle or done, on an error, or at the time limit;
// every wait is bounded. (Warps that each looked for their next unit through every slot's queue kept
// the counters' lines busy: 24 requests of 256^2 to 2048^2, 8 in flight, 10.1 ms
// against 6.3; one 1024^2 request of 40 steps 1.27 ms against 0.83.)

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned * p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release_u32(unsigned * p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}

constexpr uint64_t SRV_LOOK_NS = 50000;      // between two looks of an attached CTA at its share
constexpr int SRV_PF32 = 4;                  // columns an FP32 strip loads ahead beside the FP64 body (5 spills: 4.71 against 4.75 TB/s)
constexpr unsigned SRV_NAP_MAX = 1024;       // longest nap of an idle CTA, ns
constexpr unsigned SRV_LEAVE = 0xffffffffu;  // a ticket past every task

// One warp, the slots spread over its lanes: the most CTAs any one request may hold now. Requests that
// keep fewer busy take what they need, the others share the rest of the grid evenly (a few rounds of
// water-filling; rounded up, so that no CTA is left without a request).
__device__ __forceinline__ unsigned srv_share(const XkbSrvArgs & a, int lane)
{
    unsigned need[2] = {0, 0};                 // at most 64 slots
#pragma unroll
    for (int h = 0; h < 2; ++h)
    {
        const int q = lane + 32 * h;
        if (q >= a.nslots) continue;
        const unsigned w = *(volatile uint32_t *) &a.slots[q].ctas, st = ld_acquire_u32(&a.ctl[q].state);
        if (st == 1 || st == 2) need[h] = w;
    }
    unsigned share = 0;
    for (int round = 0; round < 4; ++round)
    {
        unsigned few = 0, many = 0;            // CTAs of the requests content with the share, number of the others
#pragma unroll
        for (int h = 0; h < 2; ++h) { if (need[h] > share) ++many; else few += need[h]; }
        few = __reduce_add_sync(0xffffffffu, few);
        many = __reduce_add_sync(0xffffffffu, many);
        if (many == 0) return gridDim.x;
        share = max(share, (gridDim.x - min(few, gridDim.x) + many - 1) / many);
    }
    return share;
}

// One thread: whether the kernel has to end (an error, the host gave up, the time limit), recorded in the
// status word, which every wait looks at.
__device__ __forceinline__ bool srv_ended(const XkbSrvArgs & a, uint64_t t_start)
{
    if (*(volatile unsigned *) a.status != 0) return true;
    if (*(volatile unsigned *) (a.status + 2) < 2 && xkb_globaltimer() - t_start <= a.run_ns) return false;
    atomicCAS(a.status, 0u, (unsigned) -XKB_ETIMEDOUT);
    return true;
}

__global__ void __launch_bounds__(SCHED_THREADS, XKB_SCHED_MINB) server_kernel(XkbSrvArgs a)
{
    constexpr int NWARPS = SCHED_THREADS / 32;
    enum { STOP, SETUP, ATTACH, NAP };
    __shared__ int job, job_slot, job_idx, ready;
    __shared__ volatile int leave;
    __shared__ unsigned next_ticket, units_run;
    __shared__ XkbSrvSlot S;                   // the record of the request worked on
    __shared__ XkbSrvCtl * c;                  // ... and its counters
    // state that lasts over a tile stands here too: every register it took would be spilled in the body
    __shared__ uint64_t t_start, looked;       // start of the kernel, last look at the share
    __shared__ unsigned counted;               // this CTA counts in `attached`
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint32_t nap = 64;
    if (tid == 0) t_start = xkb_globaltimer();
    for (;;)
    {
        if (warp == 0)
        {
            // every lane looks at its slots; the first in turn (a different one for each CTA) that has
            // something to do is tried
            const unsigned share = srv_share(a, lane);
            unsigned best = 0xffffffffu;
            bool busy = false;
            for (int q = lane; q < a.nslots; q += 32)
            {
                const unsigned st = ld_acquire_u32(&a.ctl[q].state);
                busy = busy || st == 1 || st == 2;
                const bool chunk = st == 1 && *(volatile unsigned *) &a.ctl[q].init_next < *(volatile uint32_t *) &a.slots[q].nchunks;
                const bool run = st == 2 && *(volatile unsigned *) &a.ctl[q].attached < min(share, *(volatile uint32_t *) &a.slots[q].ctas);
                if (chunk || run) best = min(best, (unsigned) ((q + a.nslots - (int) (blockIdx.x % a.nslots)) % a.nslots) << 8 | (unsigned) q);
            }
            best = __reduce_min_sync(0xffffffffu, best);
            busy = __any_sync(0xffffffffu, busy);
            if (lane == 0)
            {
                int kind = NAP, sl = -1, idx = -1;
                if (srv_ended(a, t_start)) kind = STOP;
                else if (best != 0xffffffffu)
                {
                    const int q = (int) (best & 0xff);
                    XkbSrvCtl * c = a.ctl + q;
                    // counted before the state is looked at (again): the slot is not reused while this CTA
                    // counts. Whoever ends the request stores state 3 and then looks at the count; the
                    // sequentially consistent fence between the two on either side makes one see the other.
                    const unsigned n = atomicAdd(&c->attached, 1u);
                    __threadfence();
                    const unsigned st = ld_acquire_u32(&c->state);
                    if (st == 2 && n < a.slots[q].ctas) { kind = ATTACH; sl = q; }
                    else
                    {
                        if (st == 1)
                        {
                            // (a claimed chunk holds the request in state 1 by itself)
                            const unsigned ch = atomicAdd(&c->init_next, 1u);
                            if (ch < a.slots[q].nchunks) { kind = SETUP; sl = q; idx = (int) ch; }
                        }
                        atomicSub(&c->attached, 1u);
                    }
                }
                else if (!busy && *(volatile unsigned *) (a.status + 2) != 0) kind = STOP;
                if (kind == NAP) { __nanosleep(nap); if (nap < SRV_NAP_MAX) nap *= 2; } else nap = 64;
                job = kind; job_slot = sl; job_idx = idx; leave = 0; units_run = 0;
                c = a.ctl + sl; counted = 1; looked = xkb_globaltimer();
            }
        }
        __syncthreads();
        const int kind = job;
        if (kind == STOP) break;
        if (kind == NAP) { __syncthreads(); continue; }
        for (int k = tid; k < (int) (sizeof(XkbSrvSlot) / 4); k += SCHED_THREADS)
            ((uint32_t *) &S)[k] = __ldcg((const uint32_t *) (a.slots + job_slot) + k);
        __syncthreads();
        if (kind == SETUP)
        {
            // set-up chunk: wait counters of its tasks, and its share of the second grid (a copy of the
            // first, which the host copied in)
            const uint32_t idx = (uint32_t) job_idx, t0 = idx * S.chunk_tasks, t1 = min(S.ntasks, t0 + S.chunk_tasks);
            for (uint32_t t = t0 + tid; t < t1; t += SCHED_THREADS)
            {
                const uint32_t w = t / S.period, l = t - w * S.period;
                S.wc[t] = (int) (w == 0 ? S.npred_first[l] : S.npred_next[l]);
            }
            const uint64_t per = ((S.copy_bytes + S.nchunks - 1) / S.nchunks + 15) & ~(uint64_t) 15;
            const uint64_t b0 = min(S.copy_bytes, (uint64_t) idx * per), b1 = min(S.copy_bytes, b0 + per);
            const uint4 * src = (const uint4 *) (S.copy_src + b0);
            uint4 * dst = (uint4 *) (S.copy_dst + b0);
            const uint64_t nv = (b1 - b0) / 16;
            uint64_t k = tid;
            for (; k + 3 * SCHED_THREADS < nv; k += 4 * SCHED_THREADS)   // four 16-byte loads in flight per lane
            {
                const uint4 v0 = __ldcg(src + k), v1 = __ldcg(src + k + SCHED_THREADS), v2 = __ldcg(src + k + 2 * SCHED_THREADS),
                            v3 = __ldcg(src + k + 3 * SCHED_THREADS);
                dst[k] = v0; dst[k + SCHED_THREADS] = v1; dst[k + 2 * SCHED_THREADS] = v2; dst[k + 3 * SCHED_THREADS] = v3;
            }
            for (; k < nv; k += SCHED_THREADS) dst[k] = __ldcg(src + k);
            for (uint64_t r = ((b1 - b0) & ~(uint64_t) 15) + tid; r < b1 - b0; r += SCHED_THREADS)
                S.copy_dst[b0 + r] = __ldcg(S.copy_src + b0 + r);
            __syncthreads();
            if (tid == 0)
            {
                fence_acq_rel_gpu();
                if (atomicAdd(&c->init_done, 1u) + 1 == S.nchunks)
                {
                    fence_acq_rel_gpu();
                    st_release_u32(&c->state, 2u);
                }
            }
            continue;                                          // (the smem record is rewritten after the next barrier)
        }
        // attached: an in-order run of the request's tasks
        const int k = (int) S.units_log2, nunits = 1 << k;
        const bool team = k >= TEAM_LOG2;
        const SuccGraph g{S.succ_ptr, S.succ, S.xsucc_ptr, S.xsucc, S.period, S.ntasks};
        // warp 0, between two tickets: whether the CTA has to leave
        auto look = [&]() -> bool {
            if (!__shfl_sync(0xffffffffu, (int) (xkb_globaltimer() - looked >= SRV_LOOK_NS), 0)) return false;
            const unsigned share = srv_share(a, lane);
            int out = 0;
            if (lane == 0)
            {
                looked = xkb_globaltimer();
                const unsigned keep = share + share / 8;
                if (srv_ended(a, t_start)) out = 1;
                else if (*(volatile unsigned *) &c->attached > keep)
                {
                    // counted out at once, so that no more leave than have to; the slot stays this
                    // request's until the units this CTA has run are counted
                    if (atomicSub(&c->attached, 1u) > keep) { out = 1; counted = 0; }
                    else atomicAdd(&c->attached, 1u);
                }
            }
            return __shfl_sync(0xffffffffu, out, 0) != 0;
        };
        unsigned ticket = 0;
        if (team) { if (tid == 0) next_ticket = atomicAdd(&c->head, (unsigned) NWARPS); }
        else if (lane == 0) ticket = atomicAdd(&c->head, 1u);
        for (;;)
        {
            if (team) { __syncthreads(); ticket = next_ticket == SRV_LEAVE ? SRV_LEAVE : next_ticket + warp; }
            else ticket = __shfl_sync(0xffffffffu, ticket, 0);
            if ((ticket >> k) >= S.ntasks) break;
            const uint32_t t = team ? ticket >> k : BlockOrder(S.rows, S.cols, S.ntasks).task(ticket >> k);
            const int unit = (int) (ticket & (nunits - 1));
            const uint32_t w = t / S.period, l = t - w * S.period;
            const xkb_task_desc_t d = load_desc(S.tasks + l);
            uint32_t first = 0xffffffffu;
            bool more = false;
            if (!team || warp == 0) first = g.first(l, w * S.period, lane, more);
            int ok = 1;
            if (lane == 0 && (!team || warp == 0))
            {
                const int np = (int) (w == 0 ? S.npred_first[l] : S.npred_next[l]);
                ok = wait_at_most(S.wc + t, np - np * (team ? nunits / NWARPS : nunits), a.status, a.timeout_ns);
                if (team) ready = ok;
            }
            if (team) { __syncthreads(); ok = ready; }
            else ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            __syncwarp();
            run_unit<Body::ANY, XKB_F64_PF, SRV_PF32>(d, unit, nunits, team ? 0 : S.pfd);
            if (lane == 0) atomicAdd(&units_run, 1u);
            if (team) { __syncthreads(); if (warp != 0) continue; }        // the group's units are done
            const bool out = warp == 0 && look();
            if (lane == 0)
            {
                if (out) { leave = 1; ticket = SRV_LEAVE; }
                else if (!team && leave) ticket = SRV_LEAVE;
                else ticket = atomicAdd(&c->head, team ? (unsigned) NWARPS : 1u);
                if (team) next_ticket = ticket;
            }
            __syncwarp();
            fence_acq_rel_gpu();
            count_down_successors(g, t, first, more, S.wc, lane);
        }
        // the last writes of this CTA come before its count, and the count of the request's last unit
        // before the slot is reported done
        __syncthreads();
        if (tid == 0)
        {
            fence_acq_rel_gpu();
            const unsigned all = S.ntasks << k, mine = units_run;
            if (mine && atomicAdd(&c->executed, mine) + mine == all)
            {
                fence_acq_rel_gpu();
                st_release_u32(&c->state, 3u);
                __threadfence();                               // (see where a CTA counts itself in)
                // CTAs that saw state 2 before the store above find no ticket, or the new state, and
                // leave; wait (bounded) until none but this one counts
                const uint64_t tw = xkb_globaltimer();
                for (uint32_t spins = 1; ld_acquire_u32(&c->attached) != counted; ++spins)
                    if ((spins & 63) == 0 && xkb_globaltimer() - tw > a.timeout_ns)
                    {
                        atomicCAS(a.status, 0u, (unsigned) -XKB_ETIMEDOUT);
                        break;
                    }
                atomicAdd(a.status + 1, S.ntasks);
                __threadfence_system();
                a.host_done[job_slot] = S.gen;
            }
            if (counted) atomicSub(&c->attached, 1u);
        }
        __syncthreads();
    }
}

int xkb_internal_server_launch(const XkbSrvArgs & a, int grid, cudaStream_t stream)
{
    server_kernel<<<grid, SCHED_THREADS, 0, stream>>>(a);
    XKB_CUDA_TRY(cudaGetLastError());
    return XKB_OK;
}

int xkb_internal_split_log2(uint64_t width, uint64_t warps)
{
    return split_log2((unsigned) std::min<uint64_t>(width, 1u << 30), true, 0, 0, 0, (unsigned) warps, 1);
}

int xkb_internal_launch_task(const xkb_task_desc_t * d, cudaStream_t stream)
{
    if (d->kind == XKB_TASK_NOOP) return XKB_OK;
    const int slabs = task_slabs(*d);
    task_kernel<<<slabs, SCHED_THREADS, 0, stream>>>(*d, slabs);
    XKB_CUDA_TRY(cudaGetLastError());
    return XKB_OK;
}
