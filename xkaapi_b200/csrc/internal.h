// Library-internal entry points shared between translation units (not exported).
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>
#include <thread>

#include "../../include/xkrt_b200.h"

// Launch one task descriptor as its own kernel (the plain per-task form) on `stream`.
int xkb_internal_launch_task(const xkb_task_desc_t * d, cudaStream_t stream);
// xkb_plan_execute with host cuts (sorted addresses): no two copies whose host bytes lie on
// different sides of a cut are merged into one (each copy given must lie between two cuts).
// Host copies issued by the plan executor so far, after coalescing (traces).
uint64_t xkb_internal_issued_host_copies();
int xkb_internal_plan_execute_cut(const xkb_copy_t * copies, size_t n, void * const * alloc_ptrs, size_t nallocs,
                                  cudaStream_t stream, const uint64_t * cuts, size_t ncuts);

// Set a scheduler's descriptors on the device only (persistent forms only; no host copy). The
// caller validated every descriptor with xkb_internal_task_valid; bodies: every task's
// xkb_internal_body_of, or-ed.
int xkb_internal_sched_set_tasks_device(xkb_sched_t * S, const xkb_task_desc_t * tasks, size_t ntasks, unsigned bodies);

#ifdef __CUDACC__
#define XKB_HD __host__ __device__
#else
#define XKB_HD
#endif

// The descriptor checks of xkb_sched_set_tasks: a known kind with a well-formed tile or range.
// (Heat tile bodies clip their tile to the grid's interior, so a tile beyond nx/ny is harmless
// once ld >= nx.) Also evaluated on the device by xkb_sched_run_noalloc.
static inline XKB_HD bool xkb_internal_task_valid(const xkb_task_desc_t & d)
{
    if (d.kind == XKB_TASK_HEAT_F64 || d.kind == XKB_TASK_HEAT_F32)
    {
        const auto & h = d.u.heat;
        return h.src && h.dst && h.src != h.dst && h.ld >= h.nx && h.nx >= 0 && h.ny >= 0 && h.x0 <= h.x1 && h.y0 <= h.y1;
    }
    if (d.kind == XKB_TASK_AXPBY)
    {
        const auto & a = d.u.axpby;
        return a.lo >= 0 && a.lo <= a.hi && (a.hi == a.lo || (a.x && a.y));
    }
    return d.kind == XKB_TASK_NOOP;
}

// The body a task needs in the persistent kernels: FP64 or FP32 heat tiles of grids that allow aligned
// 16-byte accesses or of any grid (row by row), axpby; 0 for a task without a body. The scheduler runs
// a kernel built for the bodies its tasks need.
constexpr unsigned XKB_BODY_F64 = 1, XKB_BODY_F32 = 2, XKB_BODY_ROWS64 = 4, XKB_BODY_ROWS32 = 8, XKB_BODY_AXPBY = 16, XKB_BODY_ALL = 31;
static inline unsigned xkb_internal_body_of(const xkb_task_desc_t & d)
{
    const auto & h = d.u.heat;
    const bool aligned = h.src % 16 == 0 && h.dst % 16 == 0;
    switch (d.kind)
    {
        case XKB_TASK_HEAT_F64: return aligned && h.ld % 2 == 0 ? XKB_BODY_F64 : XKB_BODY_ROWS64;
        case XKB_TASK_HEAT_F32: return aligned && h.ld % 4 == 0 ? XKB_BODY_F32 : XKB_BODY_ROWS32;
        case XKB_TASK_AXPBY: return XKB_BODY_AXPBY;
        default: return 0;
    }
}

// Host threads for the parallel passes of background work (resolution, coherency, descriptor
// translation): XKB_HELPERS, else the hardware threads minus four (the spawning thread, the
// worker and the page-fault helpers keep theirs), between 1 and 16.
static inline unsigned xkb_internal_helpers()
{
    if (const char * e = getenv("XKB_HELPERS")) { const int v = atoi(e); if (v > 0) return v < 64 ? (unsigned) v : 64u; }
    const unsigned hw = std::thread::hardware_concurrency();
    return hw > 5 ? (hw - 4 < 16 ? hw - 4 : 16) : 1;
}

// Reset a resolver to no tasks, keeping its device buffers for the next graph.
int xkb_internal_resolver_reset(xkb_resolver_t * R);

// A point of a resolver's edge store: the tasks added so far and where the next unique edge goes.
typedef struct xkb_edge_mark_t { size_t seg, off; uint32_t ntasks; } xkb_edge_mark_t;
int xkb_internal_resolver_edge_mark(xkb_resolver_t * R, xkb_edge_mark_t * m);
// Reserve the working memory of a batch of about nops ops up front.
int xkb_internal_resolver_prepare(xkb_resolver_t * R, size_t nops);
// Units (1, 2, 4 or 8) a task is split into at least where the scheduler chooses their number itself.
void xkb_internal_sched_min_units(xkb_sched_t * S, int units);
// Reserve the device buffers of runs of up to ntasks tasks up front.
int xkb_internal_sched_reserve(xkb_sched_t * S, size_t ntasks);
// Unique edges stored so far (no graph build).
size_t xkb_internal_resolver_nedges(const xkb_resolver_t * R);
// The window of the graph from the mark's first task to the last task added: successor CSR of
// tasks [m->ntasks, ntasks) renumbered from 0, with the edges stored since the mark whose both
// ends lie in the window (every edge into a task is stored by the batch that added the task, so
// the window keeps all edges among its tasks and drops those from earlier tasks). Device buffers
// owned by the resolver, valid until the next window (in stream order) or reset.
int xkb_internal_resolver_window_graph(xkb_resolver_t * R, const xkb_edge_mark_t * m, xkb_task_graph_t * g);

// Run tasks as one persistent launch on the scheduler's stream without waiting for it: the
// descriptors are copied in stream order (host memory may be pageable), the launch's status and
// executed count are added to the scheduler's running totals, read and cleared by
// xkb_internal_sched_windows_wait.
int xkb_internal_sched_run_window(xkb_sched_t * S, const xkb_task_desc_t * tasks, size_t ntasks, unsigned bodies, const xkb_task_graph_t * g);
// The two halves of a window run: the descriptors' copy (queued now, so that it can go ahead of
// the window's graph), then the launch on the graph of the same ntasks tasks.
int xkb_internal_sched_upload_window(xkb_sched_t * S, const xkb_task_desc_t * tasks, size_t ntasks, unsigned bodies);
int xkb_internal_sched_launch_window(xkb_sched_t * S, const xkb_task_graph_t * g);
int xkb_internal_sched_windows_wait(xkb_sched_t * S, uint64_t * executed);

// The heat update of the cells [i0, i0 + w) x [j0, j0 + h) of an nx x ny grid (interior cells
// only) on per-access replicas: src and dst point at cell (i0, j0) of theirs, each with its own
// leading dimension (xkb_diffusion_views with an explicit box).
int xkb_internal_diffusion_box(int dtype, cudaStream_t stream, const void * src, int64_t ld_src, void * dst, int64_t ld_dst,
                               int64_t i0, int64_t j0, int64_t w, int64_t h, int64_t nx, int64_t ny, double c);

// ---- device-resident serving loop (one persistent kernel for every admitted request) --------
// One admitted request, in device memory. The host writes it, then the slot's counters, then the
// slot's state word (three copies in stream order), so a team that sees the state sees the rest.
struct XkbSrvSlot {
    const xkb_task_desc_t * tasks;       // the periodic window's `period` descriptors
    const uint32_t * succ_ptr, * succ, * xsucc_ptr, * xsucc, * npred_first, * npred_next;
    int * wc;                            // ntasks wait counters
    const uint8_t * copy_src;            // the grid the host copied in ...
    uint8_t * copy_dst;                  //   ... duplicated here by the set-up chunks (second grid)
    uint64_t copy_bytes;
    uint32_t period, ntasks;
    uint32_t nchunks;                    // set-up chunks (wait counters, grid copy)
    uint32_t chunk_tasks;                // tasks whose counters one chunk sets up
    uint32_t gen;                        // admission number, reported back when the request ends
    uint32_t units_log2;                 // a task is 2^units_log2 units, each run by one warp
    uint32_t rows, cols;                 // tiles of a step (rows x cols tasks, row by row)
    uint32_t ctas;                       // CTAs its steps keep busy: units per step / warps per CTA, at least 1
    int32_t pfd;
};
// The slot's counters (device memory), one cache line for each kind of traffic. state: 0 idle, 1 admitted
// (set-up pending), 2 running, 3 done; set-up chunks claimed / finished; tickets taken; units executed;
// CTAs that work on the request, or are about to find that they cannot. The host writes what stands
// before `attached` when it admits a request; `attached` counts up and down over the whole run, as a CTA
// may look at a slot while the host refills it.
struct XkbSrvCtl {
    alignas(128) unsigned state;
    alignas(128) unsigned init_next;
    unsigned init_done;
    alignas(128) unsigned head;
    alignas(128) unsigned executed;
    alignas(128) unsigned attached;
};
struct XkbSrvArgs {
    XkbSrvSlot * slots;
    XkbSrvCtl * ctl;
    int nslots;
    volatile unsigned * host_done;       // mapped host memory: gen of the last request each slot ended
    unsigned * status;                   // [0] first error (XKB_ETIMEDOUT), [1] tasks executed,
                                         // [2] set by the host: 1 once no request will come,
                                         //     2 to stop at once (the host gave up)
    uint64_t run_ns;                     // how long a CTA may run before it gives up
    uint64_t timeout_ns;                 // longest wait for one task's predecessors
};
// At most this many tasks and bytes of the grid copy per set-up chunk (one CTA) of a served request.
constexpr uint32_t XKB_SRV_CHUNK = 8192;
constexpr uint64_t XKB_SRV_COPY_CHUNK = uint64_t(128) << 10;
// Launch the serving kernel (grid CTAs of 256 threads).
int xkb_internal_server_launch(const XkbSrvArgs & a, int grid, cudaStream_t stream);
// log2 of the units heat tile tasks are split into when `width` of them run side by side on `warps` warps.
int xkb_internal_split_log2(uint64_t width, uint64_t warps);
