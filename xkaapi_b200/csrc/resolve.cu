// Batched dependency resolver for R/W/RW accesses on LD-strided matrices and segments.
//
// Semantics (what the reference's dependency domains compute; file:line in XKRT):
//  * per task: LINK every access, then PUT every access (src/task/task.cc:285-299);
//  * one interval domain for segments, one BLAS domain per (ld, sizeof) created by the first
//    matrix access naming it, during that task's LINK pass (src/task/task.cc:153-201); a
//    segment also goes to every BLAS domain that exists at that moment (:240-259), and a new
//    BLAS domain first replays the PUT of every earlier segment newest-first
//    (interval/dependency-tree.hpp:355-360 push_front, task.cc:177-198);
//  * frames: matrix tile -> 1-2 rects (byte row mod ld*s, column) (access.hpp:204-287);
//    segment -> [a, b) in the interval domain, 3 rects in a BLAS frame (access.hpp:76-139);
//    a segment's PUT in a BLAS domain only touches rows [a, b) of column 0 of that frame,
//    because BLAS on_insert tests the access's own rects, which a segment keeps in the
//    ld = SIZE_MAX frame (access.hpp:479-514, blas/dependency-tree.hpp:228-256);
//  * per point: LINK(A): W-mode A with readers -> edges from every reader, else edge from
//    the writer; PUT(A): W-mode -> writer = A, readers = {}; mode == R exactly -> readers += A
//    (blas/dependency-tree.hpp:295-355);
//  * handles: one DependencyMap per domain task (src/task/task.cc:226-236), a point per handle
//    with the same LINK/PUT except that any mode with R and without W is recorded as a reader
//    (handle/dependency-map.hpp:157-297; sequential and commutative accesses -- a stream with
//    concurrent ones is expanded first by xkb_handle_map_expand, handles.h).
//
// Method (B200): the host turns the accesses of a batch into each domain's ordered op list
// and keeps a coordinate compression of the domain (elementary cells between all rect
// boundaries seen so far). On the GPU the ops are binned to regions of RX x RY cells, in op order; a
// CTA takes a segment of a region's list, finds each cell's state at the segment's start by looking
// back for its last write, and each thread then applies the ops to its own cell's writer/readers
// state, emitting (pred, succ) pairs; lanes emitting the same pred for the same op are merged with
// __match_any_sync. A GPU hash set keeps the unique pairs; finalising counts predecessors,
// scans and scatters the pairs into a successor CSR. Cell state stays in HBM between batches.
#include "common.cuh"
#include "internal.h"
#include "op_windows.h"
#include "scan.cuh"
#include "workpool.h"

#if defined(__x86_64__)
#include <emmintrin.h>
#endif

#include <cuda.h>

#include <algorithm>
#include <climits>
#include <chrono>
#include <string>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <map>
#include <memory>
#include <new>
#include <thread>
#include <utility>
#include <vector>

namespace xkb {

constexpr uint8_t M_R = 1, M_W = 2;
constexpr int RES_CHUNK_PER_THREAD = 4;
constexpr unsigned long long EDGE_EMPTY = ~0ull;

struct DOp {            // one op in cell coordinates (24 bytes)
    int32_t task;
    uint8_t link;
    uint8_t mode;
    uint16_t pad;
    int32_t cx0, cx1, cy0, cy1;
};

// Cell state: writer, number of readers since that write, head and tail of the reader spill
// chain, and the first RCAP readers. Readers past RCAP go to chains of SPILL-int chunks
// (next chunk, then SPILL - 1 readers) drawn from one pool per resolver, so a cell can collect
// any number of readers (a region that is read every step and never written) while the state
// and the region kernel's shared memory stay small. Chunks of a chain that a write clears are
// not reused.
#ifndef XKB_REGION_RY
#define XKB_REGION_RY 8                 // cell rows of a 2-D region (8 columns each): 8 = two warps per CTA
#endif
constexpr int RCAP = 32;
constexpr int SHDR = 4;
constexpr int STRIDE = SHDR + RCAP;
constexpr int SPILL = 32;
constexpr int SPILL_R = SPILL - 1;

struct ResolveArgs {
    const DOp * ops;
    int nops;
    int ncx, ncy, nrx;
    const int * state_in;     // STRIDE ints per cell
    int * state_out;
    unsigned long long * emit;
    unsigned long long * emit_count;
    unsigned long long emit_cap;
    int * spill;              // chunk pool
    unsigned * spill_ctr;     // [0] chunks handed out, [1] set when the pool ran out
    unsigned spill_cap;       // chunks in the pool
};

// A fresh spill chunk (its next link cleared), or -1 with the out-of-pool flag set.
__device__ __forceinline__ int spill_alloc(int * spill, unsigned * ctr, unsigned cap)
{
    const unsigned c = atomicAdd(ctr, 1u);
    if (c >= cap) { atomicExch(ctr + 1, 1u); return -1; }
    spill[(size_t) c * SPILL] = -1;
    return (int) c;
}

// Pairs are staged per warp in shared memory and appended to a.emit EMIT_BUF - 32 or more at a
// time, with one atomic on the batch's counter per flush instead of one per emitting step.
constexpr int EMIT_BUF = 256;

// Append this warp's n staged pairs to a.emit (coalesced); every lane of the warp calls it.
__device__ __forceinline__ void emit_flush(const ResolveArgs & a, const unsigned long long * buf, int n, int lane)
{
    __syncwarp();
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(a.emit_count, (unsigned long long) n);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (int j = lane; j < n; j += 32)
        if (base + j < a.emit_cap) a.emit[base + j] = buf[j];
    __syncwarp();
}

// ---- a region's ops applied to its cells, cut in time -----------------------------------------
// One CTA per region (RX x RY cells, a thread per cell) and SEGMENT of the region's op list (cut s at
// lo + (hi - lo) * s / nseg), so that a batch of few regions still fills the device. A segment
// applies its ops in order: PUT ops update the cell's state, LINK ops emit the edges from it.
// The state at its cut is not handed over by the segment before: a cell's state is its last write and
// the reads since, so the CTA looks back from the cut for each cell's last write (a handful of ops
// where tasks write what they read) and applies the PUT ops from there on; a cell without one starts
// from the state before the batch. (One CTA per region applying all PUT ops first, to leave a snapshot
// at every cut, was 2.06 of 2.65 ms on the 65,536-task stream of 128 x 128 cells; this is 0.66.) The readers matter
// to LINK ops that write only, so a segment without one skips them, unless it is the region's last
// segment, whose state is the batch's final one.
//  * Readers past RCAP: a cell that starts from the state before the batch finds the first of them on
//    that state's spill chain, which only the last segment appends to (past the count the others
//    use; a write drops a chain without reusing its chunks); the readers a segment adds go to a chain
//    of its own. The last segment's chain is kept.
__device__ __forceinline__ int seg_cut(int lo, int hi, int s, int nseg)
{
    return lo + (int) ((long long) (hi - lo) * s / nseg);
}

template <int RX, int RY>
__global__ void __launch_bounds__(RX * RY)
resolve_segment_kernel(ResolveArgs a, const unsigned * __restrict__ roff, const int * __restrict__ rlist, int nseg)
{
    constexpr int NT = RX * RY;
    constexpr int NW = NT / 32;
    constexpr int CHUNK = NT * RES_CHUNK_PER_THREAD;
    extern __shared__ int rd[];                  // readers: rd[k * NT + tid]
    __shared__ DOp list[CHUNK];
    __shared__ unsigned long long ebuf[NW][EMIT_BUF];   // each warp's pairs not yet in a.emit
    __shared__ int first_s;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int region = blockIdx.x / nseg, s = blockIdx.x % nseg;
    const bool last = s == nseg - 1;
    const int rx = region % a.nrx, ry = region / a.nrx;
    const int cx = rx * RX + tid % RX, cy = ry * RY + tid / RX;
    const bool valid = cx < a.ncx && cy < a.ncy;
    const size_t cell = valid ? (size_t) cy * a.ncx + cx : 0;
    const int lo = (int) roff[region], hi = (int) roff[region + 1];
    const int from = seg_cut(lo, hi, s, nseg), to = seg_cut(lo, hi, s + 1, nseg);
    auto covers = [&](const DOp & op) { return valid && op.cx0 <= cx && cx < op.cx1 && op.cy0 <= cy && cy < op.cy1; };

    // the cell's last write before the cut
    int wpos = -1;
    int start = from;
    bool readers = true;
    if (from > lo)
    {
        for (int e = from; e > lo;)
        {
            const int b = max(lo, e - NT), n = e - b;
            if (tid < n) list[tid] = a.ops[rlist[b + tid]];
            __syncthreads();
            for (int k = n - 1; k >= 0 && wpos < 0; --k)
            {
                const DOp op = list[k];
                if (!op.link && (op.mode & M_W) && covers(op)) wpos = b + k;
            }
            e = b;
            if (__syncthreads_and(wpos >= 0 || !valid)) break;
        }
        if (!last)
        {
            int w = 0;
            for (int i = from + tid; i < to; i += NT) { const DOp op = a.ops[rlist[i]]; w |= op.link && (op.mode & M_W); }
            readers = __syncthreads_or(w) != 0;
        }
        if (readers)
        {
            if (tid == 0) first_s = from;
            __syncthreads();
            const int mine = !valid ? from : wpos >= 0 ? wpos : lo;
            atomicMin(&first_s, mine);
            __syncthreads();
            start = first_s;
        }
    }

    int writer = -1, nr = 0;
    int shead = -1, nsnap = 0;                   // readers [RCAP, nsnap) are on the chain of the state before the batch
    int phead = -1, ptail = -1;                  // readers from max(RCAP, nsnap) on
    if (valid && wpos < 0)
    {
        const int * st = a.state_in + cell * STRIDE;
        writer = st[0]; nr = st[1]; shead = st[2];
        for (int k = 0; k < nr && k < RCAP; ++k) rd[k * NT + tid] = st[SHDR + k];
        if (last) { phead = shead; ptail = st[3]; } else nsnap = nr;
    }
    if (valid && wpos >= 0 && !readers) writer = a.ops[rlist[wpos]].task;
    int nbuf = 0;                                // pairs in this warp's ebuf (same in every lane)

    for (int base = start; base < to; base += CHUNK)
    {
        const int n = min(CHUNK, to - base);
        for (int j = tid; j < n; j += NT) list[j] = a.ops[rlist[base + j]];
        __syncthreads();
        for (int k = 0; k < n; ++k)
        {
            const DOp op = list[k];
            const bool in = covers(op) && base + k >= wpos;
            const int pbase = max(RCAP, nsnap);
            if (op.link)
            {
                if (base + k < from) continue;
                const bool from_readers = in && (op.mode & M_W) && nr > 0;
                const int cnt = from_readers ? nr : ((in && writer >= 0) ? 1 : 0);
                const int maxcnt = __reduce_max_sync(0xffffffffu, cnt);
                int chunk = shead, ci = 0;                // walk of the spill chain past RCAP
                for (int q = 0; q < maxcnt; ++q)
                {
                    int p = -1;
                    if (q < cnt)
                    {
                        if (!from_readers) p = writer;
                        else if (q < RCAP) p = rd[q * NT + tid];
                        else
                        {
                            if (q == pbase) { chunk = phead; ci = 0; }
                            else if (ci == SPILL_R) { chunk = chunk >= 0 ? a.spill[(size_t) chunk * SPILL] : -1; ci = 0; }
                            p = chunk >= 0 ? a.spill[(size_t) chunk * SPILL + 1 + ci] : -1;   // -1: pool ran out, batch redone
                            ++ci;
                        }
                    }
                    const unsigned peers = __match_any_sync(0xffffffffu, p);
                    const bool leader = p >= 0 && lane == __ffs(peers) - 1;
                    const unsigned em = __ballot_sync(0xffffffffu, leader);
                    if (leader)
                        ebuf[warp][nbuf + __popc(em & ((1u << lane) - 1))] = ((unsigned long long) (uint32_t) p << 32) | (uint32_t) op.task;
                    nbuf += __popc(em);
                    if (nbuf > EMIT_BUF - 32) { emit_flush(a, ebuf[warp], nbuf, lane); nbuf = 0; }
                }
            }
            else if (in)
            {
                if (op.mode & M_W) { writer = op.task; nr = 0; nsnap = 0; phead = ptail = -1; }
                else if (op.mode == M_R && readers)
                {
                    if (nr < RCAP) rd[nr * NT + tid] = op.task;
                    else
                    {
                        const int slot = (nr - pbase) % SPILL_R;
                        if (slot == 0)
                        {
                            const int c = spill_alloc(a.spill, a.spill_ctr, a.spill_cap);
                            if (c >= 0) { if (ptail >= 0) a.spill[(size_t) ptail * SPILL] = c; else phead = c; }
                            ptail = c;
                        }
                        if (ptail >= 0) a.spill[(size_t) ptail * SPILL + 1 + slot] = op.task;
                    }
                    ++nr;
                }
            }
        }
        __syncthreads();
    }

    if (nbuf) emit_flush(a, ebuf[warp], nbuf, lane);
    if (valid && last)
    {
        int * st = a.state_out + cell * STRIDE;
        st[0] = writer; st[1] = nr; st[2] = nr > RCAP ? phead : -1; st[3] = nr > RCAP ? ptail : -1;
        for (int k = 0; k < nr && k < RCAP; ++k) st[SHDR + k] = rd[k * NT + tid];
    }
}

// ---- binning of ops to regions ----------------------------------------------------------------
// The regions of an op: the RX x RY cell blocks its cell rect overlaps.
__global__ void bin_count_kernel(const DOp * __restrict__ ops, int nops, int RX, int RY, int nrx, unsigned * rcount)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nops) return;
    const DOp o = ops[i];
    if (o.cx0 >= o.cx1 || o.cy0 >= o.cy1) return;
    for (int ry = o.cy0 / RY; ry <= (o.cy1 - 1) / RY; ++ry)
        for (int rx = o.cx0 / RX; rx <= (o.cx1 - 1) / RX; ++rx)
            atomicAdd(rcount + ry * nrx + rx, 1u);
}

__global__ void bin_fill_kernel(const DOp * __restrict__ ops, int nops, int RX, int RY, int nrx, const unsigned * __restrict__ roff,
                                unsigned * cursor, int * list)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nops) return;
    const DOp o = ops[i];
    if (o.cx0 >= o.cx1 || o.cy0 >= o.cy1) return;
    for (int ry = o.cy0 / RY; ry <= (o.cy1 - 1) / RY; ++ry)
        for (int rx = o.cx0 / RX; rx <= (o.cx1 - 1) / RX; ++rx)
        {
            const int r = ry * nrx + rx;
            list[roff[r] + atomicAdd(cursor + r, 1u)] = i;
        }
}

// Block-local binning: with at most BIN_SMEM_REGIONS regions, a block of the count / fill kernels
// counts its ops' regions in shared memory and touches each region's global counter once (the
// kernels above do one global atomic per (op, region) on a few hundred shared counters).
constexpr int BIN_SMEM_REGIONS = 12288;

__global__ void bin_count_smem_kernel(const DOp * __restrict__ ops, int nops, int RX, int RY, int nrx, int nregions,
                                      unsigned * rcount)
{
    extern __shared__ unsigned h[];
    for (int r = threadIdx.x; r < nregions; r += blockDim.x) h[r] = 0;
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nops; i += gridDim.x * blockDim.x)
    {
        const DOp o = ops[i];
        if (o.cx0 >= o.cx1 || o.cy0 >= o.cy1) continue;
        for (int ry = o.cy0 / RY; ry <= (o.cy1 - 1) / RY; ++ry)
            for (int rx = o.cx0 / RX; rx <= (o.cx1 - 1) / RX; ++rx)
                atomicAdd(h + ry * nrx + rx, 1u);
    }
    __syncthreads();
    for (int r = threadIdx.x; r < nregions; r += blockDim.x)
        if (h[r]) atomicAdd(rcount + r, h[r]);
}

// Each block counts its own ops' regions, reserves one range per region with one global atomic,
// and places its ops inside its ranges (any op-to-block split works: each region's list is put
// back in op order afterwards).
__global__ void bin_fill_smem_kernel(const DOp * __restrict__ ops, int nops, int RX, int RY, int nrx, int nregions,
                                     const unsigned * __restrict__ roff, unsigned * cursor, int * list)
{
    extern __shared__ unsigned h[];                       // [nregions] counts, then [nregions] bases
    unsigned * base = h + nregions;
    for (int r = threadIdx.x; r < nregions; r += blockDim.x) h[r] = 0;
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nops; i += gridDim.x * blockDim.x)
    {
        const DOp o = ops[i];
        if (o.cx0 >= o.cx1 || o.cy0 >= o.cy1) continue;
        for (int ry = o.cy0 / RY; ry <= (o.cy1 - 1) / RY; ++ry)
            for (int rx = o.cx0 / RX; rx <= (o.cx1 - 1) / RX; ++rx)
                atomicAdd(h + ry * nrx + rx, 1u);
    }
    __syncthreads();
    for (int r = threadIdx.x; r < nregions; r += blockDim.x)
    {
        base[r] = h[r] ? roff[r] + atomicAdd(cursor + r, h[r]) : 0u;
        h[r] = 0;
    }
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nops; i += gridDim.x * blockDim.x)
    {
        const DOp o = ops[i];
        if (o.cx0 >= o.cx1 || o.cy0 >= o.cy1) continue;
        for (int ry = o.cy0 / RY; ry <= (o.cy1 - 1) / RY; ++ry)
            for (int rx = o.cx0 / RX; rx <= (o.cx1 - 1) / RX; ++rx)
            {
                const int r = ry * nrx + rx;
                list[base[r] + atomicAdd(h + r, 1u)] = i;
            }
    }
}

constexpr int MAX_SEGMENTS = 24;             // segments per region at most
constexpr int SEGMENT_OPS = 512;             // ops per segment aimed at (12 or 32 segments, 256 ops: within 3 %)
constexpr int BIN_SORT_THREADS = 1024;
constexpr int BIN_SORT_SHORT = 1024;         // a list of up to this many ops is sorted as keys
constexpr int BIN_SORT_WORDS = 40960;        // words of the bitmap of a longer one at most (160 KB: 1.3 M ops a pass)

// Put each region's list back in op order (the fill appends in arbitrary order), from `in` to `out`.
// A short list: bitonic sort in shared memory. A longer one: its ops set their bits in a bitmap of the
// batch's ops, whose set bits are then written out in order -- the list is a set of distinct numbers
// below nops -- `words` words of it at a time. (Bitonic sorts of 12,800 ops per region took 264 us; this
// 24.)
__global__ void __launch_bounds__(BIN_SORT_THREADS) bin_sort_kernel(const unsigned * __restrict__ roff, const int * __restrict__ in,
                                                                    int * __restrict__ out, int nops, int words)
{
    extern __shared__ unsigned bits[];
    __shared__ uint32_t wt[32];
    const unsigned b = roff[blockIdx.x], e = roff[blockIdx.x + 1];
    const int n = (int) (e - b);
    if (n == 0) return;
    if (n <= BIN_SORT_SHORT)
    {
        int * keys = (int *) bits;
        int p2 = 1;
        while (p2 < n) p2 <<= 1;
        const int i = threadIdx.x;
        if (i < p2) keys[i] = i < n ? in[b + i] : 0x7fffffff;
        __syncthreads();
        for (int k = 2; k <= p2; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1)
            {
                const int l = i ^ j;
                if (i < p2 && l > i)
                {
                    const int x = keys[i], y = keys[l];
                    if (((i & k) == 0) == (x > y)) { keys[i] = y; keys[l] = x; }
                }
                __syncthreads();
            }
        if (i < n) out[b + i] = keys[i];
        return;
    }
    unsigned pos = b;
    for (int at = 0; at < nops;)
    {
        const OpWindow win = OpWindow::from(at, words, nops);
        for (int w = threadIdx.x; w < words; w += BIN_SORT_THREADS) bits[w] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += BIN_SORT_THREADS)
        {
            const int op = in[b + i];
            if (win.holds(op)) atomicOr(bits + ((op - win.first) >> 5), 1u << ((op - win.first) & 31));
        }
        __syncthreads();
        const int used = (win.last - win.first + 31) / 32;
        for (int w = threadIdx.x; w < ((used + BIN_SORT_THREADS - 1) / BIN_SORT_THREADS) * BIN_SORT_THREADS; w += BIN_SORT_THREADS)
        {
            unsigned m = w < used ? bits[w] : 0u;
            uint32_t total;
            unsigned to = pos + block_exclusive_scan((uint32_t) __popc(m), wt, total);
            pos += total;
            for (; m; m &= m - 1) out[to++] = win.first + w * 32 + __ffs(m) - 1;
        }
        __syncthreads();
        at = win.last;
    }
}

// New compression refines the old one: every new cell lies inside exactly one old cell (or
// outside the old domain, where the state is empty).
// Every new cell takes the state of the old cell it lies in; a spill chain is copied into fresh
// chunks, since several new cells can come from one old cell and each appends on its own.
__global__ void refine_state_kernel(const int * __restrict__ old_state, int * __restrict__ new_state,
                                    const int * __restrict__ map_x, const int * __restrict__ map_y, int ncx, int ncy, int old_ncx,
                                    int * spill, unsigned * spill_ctr, unsigned spill_cap)
{
    const size_t cell = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (cell >= (size_t) ncx * ncy) return;
    const int cx = (int) (cell % ncx), cy = (int) (cell / ncx);
    const int ox = map_x[cx], oy = map_y[cy];
    int * dst = new_state + cell * STRIDE;
    if (ox < 0 || oy < 0) { dst[0] = -1; dst[1] = 0; dst[2] = -1; dst[3] = -1; return; }
    const int * src = old_state + ((size_t) oy * old_ncx + ox) * STRIDE;
    const int n = src[1];
    dst[0] = src[0]; dst[1] = n;
    for (int k = 0; k < n && k < RCAP; ++k) dst[SHDR + k] = src[SHDR + k];
    int head = -1, tail = -1;
    int from = src[2];
    for (int left = n - RCAP; left > 0 && from >= 0; left -= SPILL_R)
    {
        const int c = spill_alloc(spill, spill_ctr, spill_cap);
        if (c < 0) { head = tail = -1; break; }                 // pool ran out: redone after growing
        for (int k = 1; k < SPILL; ++k) spill[(size_t) c * SPILL + k] = spill[(size_t) from * SPILL + k];
        if (tail >= 0) spill[(size_t) tail * SPILL] = c; else head = c;
        tail = c;
        from = spill[(size_t) from * SPILL];
    }
    dst[2] = head; dst[3] = tail;
}

__global__ void init_state_kernel(int * state, size_t ncells)
{
    const size_t cell = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (cell < ncells) { int * st = state + cell * STRIDE; st[0] = -1; st[1] = 0; st[2] = -1; st[3] = -1; }
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long k)
{
    k ^= k >> 33; k *= 0xff51afd7ed558ccdull; k ^= k >> 33; k *= 0xc4ceb9fe1a85ec53ull; k ^= k >> 33;
    return k;
}

// Results of a batch's device work, read back together: pairs emitted, unique pairs stored so far in
// the segment, and whether the hash set or the segment had no room.
enum { CNT_EMIT, CNT_UNIQ, CNT_FULL, CNT_COUNT };

// Unique the emitted pairs into a hash set and append the new ones to `uniq`. The count is read on the
// device; nothing is done when the pairs did not fit their buffer (the host redoes the batch). Most
// pairs are already there (a pair is emitted by every region the two tasks share): a plain load finds
// them without an atomic (8.2 M pairs, 1.4 M unique: 544 us with an atomic each, 372 so).
constexpr int DEDUPE_PROBES = 128;
__global__ void __launch_bounds__(256) dedupe_kernel(const unsigned long long * __restrict__ emit, unsigned long long emit_cap,
                                                     unsigned long long * table, unsigned long long mask, unsigned long long * uniq,
                                                     unsigned long long * cnt, unsigned long long uniq_cap)
{
    const unsigned long long n = cnt[CNT_EMIT];
    if (n > emit_cap) return;
    const int lane = threadIdx.x & 31;
    const unsigned long long stride = (unsigned long long) gridDim.x * blockDim.x;
    for (unsigned long long i0 = (unsigned long long) blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < n; i0 += stride)
    {
        const unsigned long long i = i0 + lane;
        bool fresh = false;
        unsigned long long key = 0;
        if (i < n)
        {
            key = emit[i];
            unsigned long long h = mix64(key) & mask;
            bool done = false;
            for (int probe = 0; probe < DEDUPE_PROBES && !done; ++probe)
            {
                unsigned long long v = *(volatile unsigned long long *) (table + h);
                if (v == EDGE_EMPTY) { v = atomicCAS(table + h, EDGE_EMPTY, key); fresh = done = v == EDGE_EMPTY; }
                done = done || v == key;
                h = (h + 1) & mask;
            }
            if (!done) cnt[CNT_FULL] = 1;
        }
        // one atomic per warp on the shared counter for the warp's new pairs
        const unsigned nb = __ballot_sync(0xffffffffu, fresh);
        if (!nb) continue;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(cnt + CNT_UNIQ, (unsigned long long) __popc(nb));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (fresh)
        {
            const unsigned long long at = base + __popc(nb & ((1u << lane) - 1));
            if (at < uniq_cap) uniq[at] = key; else cnt[CNT_FULL] = 1;
        }
    }
}

__global__ void count_edges_kernel(const unsigned long long * __restrict__ e, size_t n, uint32_t * nsucc, uint32_t * npred)
{
    const size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long k = e[i];
    atomicAdd(nsucc + (uint32_t) (k >> 32), 1u);
    atomicAdd(npred + (uint32_t) k, 1u);
}

__global__ void scatter_edges_kernel(const unsigned long long * __restrict__ e, size_t n, uint32_t * cursor, uint32_t * succ)
{
    const size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long k = e[i];
    const uint32_t pos = atomicAdd(cursor + (uint32_t) (k >> 32), 1u);
    succ[pos] = (uint32_t) k;
}

// A window of the graph: edges whose ends are both >= first, renumbered from first.
__global__ void count_window_edges_kernel(const unsigned long long * __restrict__ e, size_t n, uint32_t first, uint32_t * nsucc,
                                          uint32_t * npred)
{
    const size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long k = e[i];
    const uint32_t p = (uint32_t) (k >> 32), q = (uint32_t) k;
    if (p < first || q < first) return;
    atomicAdd(nsucc + (p - first), 1u);
    atomicAdd(npred + (q - first), 1u);
}

__global__ void scatter_window_edges_kernel(const unsigned long long * __restrict__ e, size_t n, uint32_t first, uint32_t * cursor,
                                            uint32_t * succ)
{
    const size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long k = e[i];
    const uint32_t p = (uint32_t) (k >> 32), q = (uint32_t) k;
    if (p < first || q < first) return;
    succ[atomicAdd(cursor + (p - first), 1u)] = q - first;
}

// Sort each successor list ascending (deterministic CSR), a warp per task: up to 32 successors by
// counting the smaller ones over shuffles, up to SORT_LIST by a bitonic sort in the warp's share of
// shared memory, longer lists in place in global memory by the same network. (Successors of a task are
// distinct.) 45 us for 1.4 M edges of 65,536 tasks; one thread per task with an insertion sort took 235.
constexpr uint32_t SORT_LIST = 512;
__global__ void __launch_bounds__(256) sort_segments_kernel(const uint32_t * __restrict__ ptr, uint32_t * succ, uint32_t ntasks)
{
    __shared__ uint32_t keys_s[8][SORT_LIST];
    const uint32_t t = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= ntasks) return;
    const uint32_t b = ptr[t], n = ptr[t + 1] - b;
    if (n < 2) return;
    if (n <= 32)
    {
        const uint32_t v = (uint32_t) lane < n ? succ[b + lane] : 0xffffffffu;
        int rank = 0;
        for (uint32_t k = 0; k < n; ++k) rank += __shfl_sync(0xffffffffu, v, (int) k) < v;
        if ((uint32_t) lane < n) succ[b + rank] = v;
        return;
    }
    uint32_t * keys = n <= SORT_LIST ? keys_s[threadIdx.x >> 5] : succ + b;
    if (n <= SORT_LIST) for (uint32_t i = lane; i < n; i += 32) keys[i] = succ[b + i];
    __syncwarp();
    // bitonic network for any n: every merge step compares ascending (the first one of a merge mirrored),
    // so places past the end, which would hold the largest keys, never move
    uint32_t p2 = 64;
    while (p2 < n) p2 <<= 1;
    for (uint32_t k = 2; k <= p2; k <<= 1)
        for (uint32_t j = k; j > 1; j >>= 1)
        {
            for (uint32_t q = lane; q < p2 / 2; q += 32)
            {
                // the q-th pair: mirrored within blocks of k, then at distance j / 2 within blocks of j
                const uint32_t blk = q / (j / 2), o = q % (j / 2), i = blk * j + o, l = j == k ? blk * j + j - 1 - o : i + j / 2;
                if (l < n)
                {
                    const uint32_t x = keys[i], y = keys[l];
                    if (x > y) { keys[i] = y; keys[l] = x; }
                }
            }
            __syncwarp();
        }
    if (n <= SORT_LIST) for (uint32_t i = lane; i < n; i += 32) succ[b + i] = keys[i];
}

// ------------------------------------------------------------------------------------------
// host side

struct HRect { uint64_t x0, x1, y0, y1; };
// An op in byte coordinates. PAIRED ops (staged batches) stand for a LINK and a PUT op each.
struct HOp { uint32_t task; uint8_t link; uint8_t mode; HRect r; };

// Store an op past the caches: the page-locked staging buffer is read by the GPU next, and reading
// lines that lie modified in the caches of a dozen cores ran at 5 GB/s instead of 53 (13 MB: 2.3 ms
// against 0.26). stream_fence() before the copy is queued.
static inline void stream_op(HOp * p, const HOp & op)
{
#if defined(__x86_64__)
    static_assert(sizeof(HOp) == 40, "five 8-byte stores");
    long long w[5];
    memcpy(w, &op, sizeof(op));
    for (int k = 0; k < 5; ++k) _mm_stream_si64((long long *) p + k, w[k]);
#else
    *p = op;
#endif
}
static inline void stream_fence()
{
#if defined(__x86_64__)
    _mm_sfence();
#endif
}

static size_t g_realloc_bytes = 0;               // device bytes allocated by reserve (trace)

// Number of the CUDA context current on this thread (the device's own is made so if there is none): never
// used twice in a process, unlike a context's address. 0: the driver cannot tell.
static uint64_t context_id()
{
    typedef CUresult (*get_id_t)(CUcontext, unsigned long long *);
    static const get_id_t get_id = [] {
        cudaDriverEntryPointQueryResult q;
        void * f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            return (get_id_t) f;
        cudaGetLastError();
        return (get_id_t) nullptr;
    }();
    unsigned long long id = 0;
    if (!get_id || get_id(nullptr, &id) == CUDA_SUCCESS) return id;
    return cudaFree(nullptr) == cudaSuccess && get_id(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

// Device memory pool of the resolver's work buffers on the current device (made on first use).
// Buffers only the resolver's own stream touches are allocated from it in stream order, so
// growing one neither waits for the whole device (as cudaFree does) nor asks the driver for
// memory while copies and kernels of other streams run: a runtime streaming windows of tasks
// had its resolution stall for up to 0.3 s in cudaMalloc / cudaFree of a domain's cell states.
// Freed memory stays in the pool for the next resolver of the process, up to 4 GiB
// (XKB_POOL_CACHE=0: none). A pool ends with its context (cudaDeviceReset), and the next context of the
// device gets one of its own.
static cudaMemPool_t resolver_pool()
{
    static std::mutex mu;
    static auto * pools = new std::map<std::pair<int, uint64_t>, cudaMemPool_t>;       // by device and context
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    const uint64_t ctx = context_id();
    std::lock_guard<std::mutex> lk(mu);
    const auto known = pools->find({dev, ctx});
    if (known != pools->end()) return known->second;
    cudaMemPoolProps props;
    memset(&props, 0, sizeof(props));
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) { cudaGetLastError(); pool = nullptr; }
    else
    {
        const char * e = getenv("XKB_POOL_CACHE");
        uint64_t keep = (e && atoi(e) == 0) ? 0 : (uint64_t(4) << 30);
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    (*pools)[{dev, ctx}] = pool;
    return pool;
}

// Page-locked host memory the resolvers of the process share: a batch takes blocks for its staging and
// its read-backs and gives them back when it has been waited for, so a resolver holds none between
// batches and a new one finds them there (page-locking costs about 0.5 ms per MB and waits for the
// device; a server keeps a resolver per graph shape). Given-back blocks are kept up to PINNED_KEEP
// bytes while there are resolvers, and PINNED_REST once there is none (XKB_POOL_CACHE=0: none); a block
// in use belongs to one batch. A block up to four times the size asked for will do, and a block given back
// displaces larger ones rather than being unlocked, so a stream of batches finds its blocks again
// whatever an earlier one left: unlocking and locking 64 MB behind a running window costs 35 to 90 ms a
// batch (16384^2 x 500 heat graph spawned through the C API: 1.6 to 2.7 s to the end of the wait when a
// 128 MB block no batch asked for filled the room, 0.63 s now).
// Blocks end with the context they were made in (cudaDeviceReset), so each context has its own, and those of
// one that ended are neither handed out nor unlocked again.
class PinnedBlocks {
public:
    static constexpr size_t PINNED_KEEP = size_t(256) << 20, PINNED_REST = size_t(64) << 20, MIN_BLOCK = size_t(1) << 18;

    static int take(size_t bytes, void ** p, size_t * cap, uint64_t * ctx)
    {
        size_t c = MIN_BLOCK;
        while (c < bytes) c *= 2;
        *ctx = context_id();
        std::vector<void *> due;
        {
            std::lock_guard<std::mutex> lk(mu());
            Kept & k = kept(*ctx);
            due.swap(k.due);
            auto it = k.blocks.lower_bound(c);
            if (it != k.blocks.end() && it->first <= 4 * c)
            {
                *p = it->second; *cap = it->first;
                k.bytes -= it->first;
                k.blocks.erase(it);
            }
            else *p = nullptr;
        }
        unlock(due);
        if (*p) return XKB_OK;
        cudaError_t e = cudaHostAlloc(p, c, cudaHostAllocPortable);
        if (e != cudaSuccess) { *p = nullptr; return xkb_set_cuda_error(e); }
        *cap = c;
        return XKB_OK;
    }
    // Whether a block of this size is kept when it is given back; one that is not is unlocked.
    static bool keeps(size_t cap)
    {
        static const bool none = getenv("XKB_POOL_CACHE") && atoi(getenv("XKB_POOL_CACHE")) == 0;
        return !none && cap <= PINNED_KEEP;
    }
    static void give(void * p, size_t cap, uint64_t ctx)
    {
        if (!p) return;
        const bool current = ctx == context_id();
        std::vector<void *> due;
        {
            std::lock_guard<std::mutex> lk(mu());
            Kept & k = kept(ctx);
            if (!keeps(cap)) k.due.push_back(p);
            else
            {
                k.blocks.emplace(cap, p);
                k.bytes += cap;
                k.keep(k.resolvers ? PINNED_KEEP : PINNED_REST, p);
            }
            if (current) due.swap(k.due);                        // (else when the context is current again)
        }
        unlock(due);
    }

    // A resolver of context ctx begins, and ends.
    static void enter(uint64_t ctx) { std::lock_guard<std::mutex> lk(mu()); ++kept(ctx).resolvers; }
    static void leave(uint64_t ctx)
    {
        const bool current = ctx == context_id();
        std::vector<void *> due;
        {
            std::lock_guard<std::mutex> lk(mu());
            Kept & k = kept(ctx);
            if (--k.resolvers == 0) k.keep(PINNED_REST, nullptr);
            if (current) due.swap(k.due);
        }
        unlock(due);
    }

private:                                        // (never destroyed: resolvers may outlive static objects)
    struct Kept {
        std::multimap<size_t, void *> blocks;
        size_t bytes = 0, resolvers = 0;
        std::vector<void *> due;                                 // to be unlocked
        // the smallest blocks, `limit` bytes of them at most; `last` is the last to go
        void keep(size_t limit, void * last)
        {
            while (bytes > limit)
            {
                auto it = std::prev(blocks.end());
                if (it->second == last && it != blocks.begin()) --it;
                bytes -= it->first;
                due.push_back(it->second);
                blocks.erase(it);
            }
        }
    };
    static std::mutex & mu() { static std::mutex * m = new std::mutex; return *m; }
    static void unlock(const std::vector<void *> & due) { for (void * q : due) cudaFreeHost(q); }     // (may wait for the device)
    static Kept & kept(uint64_t ctx) { static auto * k = new std::map<uint64_t, Kept>; return (*k)[ctx]; }
};

template <typename T>
struct DevBuf {
    T * p = nullptr;
    size_t cap = 0;
    cudaStream_t st = nullptr;       // pooled: the one stream that uses the buffer
    bool pooled = false;
    ~DevBuf()
    {
        if (!p) return;
        if (!pooled) cudaFree(p);
        else if (cudaFreeAsync(p, st) != cudaSuccess) { cudaGetLastError(); cudaFree(p); }
    }
    // Allocate from the resolver's pool in the order of `s` (before the first allocation only).
    void use_pool(cudaStream_t s)
    {
        if (p) return;
        pooled = resolver_pool() != nullptr;
        st = s;
    }
    int reserve(size_t n)
    {
        if (n <= cap) return XKB_OK;
        size_t c = cap ? cap : 1024;
        while (c < n) c *= 2;
        T * q = nullptr;
        g_realloc_bytes += c * sizeof(T);
        if (pooled)
        {
            cudaError_t e = cudaMallocFromPoolAsync((void **) &q, c * sizeof(T), resolver_pool(), st);
            if (e != cudaSuccess) return xkb_set_cuda_error(e);
            if (p) cudaFreeAsync(p, st);      // after the stream's work queued so far
        }
        else
        {
            cudaError_t e = cudaMalloc(&q, c * sizeof(T));
            if (e != cudaSuccess) return xkb_set_cuda_error(e);
            if (p) cudaFree(p);
        }
        p = q; cap = c;
        return XKB_OK;
    }
};

// ---- coordinate compression on the device ----------------------------------------------------
// Every op's rect boundaries go into two open-addressing hash sets (x and y); each first insert
// appends the key to a compact list, so the host only sorts the distinct boundaries of the batch.
// The tables hold at least twice as many slots as keys can be inserted, so a probe always ends at
// an empty slot. Slots only ever change from empty to a key, so a stale read sees empty at worst
// and the CAS settles it. The key ~0 (the empty marker) is reported through a flag bit instead.
constexpr uint64_t KEY_EMPTY = ~0ull;

__device__ __forceinline__ void hset_insert(uint64_t * tab, uint32_t mask, uint64_t key, uint64_t * out, unsigned * count,
                                            unsigned * flags, unsigned max_bit)
{
    if (key == KEY_EMPTY) { atomicOr(flags, max_bit); return; }
    uint32_t h = (uint32_t) ((key * 0x9e3779b97f4a7c15ull) >> 32) & mask;
    for (;;)
    {
        const uint64_t v = *(volatile uint64_t *) (tab + h);
        if (v == key) return;
        if (v == KEY_EMPTY)
        {
            const uint64_t prev = atomicCAS((unsigned long long *) (tab + h), (unsigned long long) KEY_EMPTY,
                                            (unsigned long long) key);
            if (prev == KEY_EMPTY) { out[atomicAdd(count, 1u)] = key; return; }
            if (prev == key) return;
        }
        h = (h + 1) & mask;
    }
}

// counts[0] / counts[1]: distinct x / y keys appended; counts[2]: bit 1 / 2 when ~0 was an x / y key
__global__ void collect_bounds_kernel(const HOp * __restrict__ ops, int n, uint64_t * tx, uint64_t * ty, uint32_t mask,
                                      uint64_t * ux, uint64_t * uy, unsigned * counts)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const HRect r = ops[i].r;
    // neighbouring ops mostly share their boundaries (tiles of one grid): one lane per distinct
    // key of the warp probes the table
    const unsigned act = __activemask(), lane = threadIdx.x & 31;
    auto once = [&](uint64_t key, uint64_t * tab, uint64_t * out, unsigned * count, unsigned bit) {
        const unsigned same = __match_any_sync(act, key);
        if ((unsigned) (__ffs(same) - 1) == lane) hset_insert(tab, mask, key, out, count, counts + 2, bit);
    };
    once(r.x0, tx, ux, counts + 0, 1u);
    once(r.x1, tx, ux, counts + 0, 1u);
    once(r.y0, ty, uy, counts + 1, 2u);
    once(r.y1, ty, uy, counts + 1, 2u);
}

__device__ __forceinline__ int32_t lower_index(const uint64_t * __restrict__ v, int n, uint64_t key)
{
    int lo = 0, hi = n;
    while (lo < hi) { const int mid = (lo + hi) >> 1; if (__ldg(v + mid) < key) lo = mid + 1; else hi = mid; }
    return lo;
}

// Ops in cell coordinates: each boundary's index in the domain's sorted boundary lists. PAIRED: op e
// of a task's ops [b, f) (ops are in task order) becomes the LINK op b + e and the PUT op f + e -- all
// of a task's LINK ops before its PUT ops.
template <bool PAIRED>
__global__ void map_ops_kernel(const HOp * __restrict__ ops, int n, const uint64_t * __restrict__ xs, int nxs,
                               const uint64_t * __restrict__ ys, int nys, DOp * out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const HOp o = ops[i];
    DOp q;
    q.task = (int32_t) o.task; q.link = PAIRED ? 1 : o.link; q.mode = o.mode; q.pad = 0;
    q.cx0 = lower_index(xs, nxs, o.r.x0); q.cx1 = lower_index(xs, nxs, o.r.x1);
    q.cy0 = lower_index(ys, nys, o.r.y0); q.cy1 = lower_index(ys, nys, o.r.y1);
    if constexpr (!PAIRED) { out[i] = q; return; }
    // the task's first and one past its last op: most tasks have a few, others are bisected for
    auto edge = [&](int dir) {
        int k = i;
        for (int step = 1; step <= 8; ++step)
        {
            const int m = i + dir * step;
            if (m < 0 || m >= n || ops[m].task != o.task) return k;
            k = m;
        }
        int in = k, outside = dir < 0 ? -1 : n;
        while (in - outside > 1 || outside - in > 1)
        {
            const int m = in + (outside - in) / 2;
            if (ops[m].task == o.task) in = m; else outside = m;
        }
        return in;
    };
    const int b = edge(-1), f = edge(1) + 1;
    out[b + i] = q;
    q.link = 0;
    out[f + i] = q;
}

struct Domain {
    bool interval = false;
    uint64_t ld = 0, s = 0;
    std::vector<uint64_t> xs, ys;       // compression (sorted unique boundaries)
    DevBuf<int> state[2];
    int cur = 0;
    size_t ncells = 0;
    std::vector<HOp> ops;               // ops of the batch being resolved (sequential build)
    size_t nops = 0;                    // ops of the batch
    size_t nhops = 0;                   // as they are uploaded: nops, or half of them (staged: PAIRED)
};

// A block of a resolver. rest(), between batches, gives it back where it is kept for whoever asks next, and
// holds on to it where it would be unlocked and locked again for the next batch (more than PINNED_KEEP
// bytes, or no block is kept: 1.56 ms against 0.40 for an add of 1,280 records).
struct PinnedBlock {
    uint8_t * p = nullptr;
    size_t cap = 0;
    uint64_t ctx = 0;
    PinnedBlock() = default;
    PinnedBlock(const PinnedBlock &) = delete;
    PinnedBlock & operator=(const PinnedBlock &) = delete;
    ~PinnedBlock() { drop(); }
    void drop() { PinnedBlocks::give(p, cap, ctx); p = nullptr; cap = 0; }
    void rest() { if (PinnedBlocks::keeps(cap)) drop(); }
    // at least n bytes; what the block held is gone
    int take(size_t n)
    {
        if (p && n <= cap) return XKB_OK;
        drop();
        return PinnedBlocks::take(n, (void **) &p, &cap, &ctx);
    }
};

// Page-locked host memory the staged build writes the batch's ops into, so that their upload runs at
// DMA speed.
struct HostStage {
    PinnedBlock block;
    HOp * ops() { return (HOp *) block.p; }
    int take(size_t n) { return block.take(n * sizeof(HOp)); }
    void rest() { block.rest(); }
    void drop() { block.drop(); }
};

// Page-locked host memory for what the device reports back and for the small arrays it is given, so
// that neither waits for a staging copy: results (first, fixed places), then `used` bytes handed out
// to arrays whose copies are in flight; release() once the stream has been waited for.
struct HostScratch {
    static constexpr size_t RESULTS = 256, KEYS = 2048;           // bytes; keys of each axis read back with the counts
    PinnedBlock block;
    size_t used = 0;
    void rest() { block.rest(); }
    void drop() { block.drop(); }
    uint64_t * results() { return (uint64_t *) block.p; }
    uint64_t * keys(int axis) { return (uint64_t *) (block.p + RESULTS) + axis * KEYS; }
    void release() { used = RESULTS + 2 * KEYS * sizeof(uint64_t); }
    int init() { return grow(size_t(1) << 17); }
    // n bytes for a copy to the device queued on `st`; a full scratch waits for the copies so far
    int take(size_t n, cudaStream_t st, void ** out)
    {
        n = (n + 15) & ~(size_t) 15;
        if (used + n > block.cap)
        {
            XKB_CUDA_TRY(cudaStreamSynchronize(st));
            release();
            if (used + n > block.cap) if (int rc = grow(2 * (used + n))) return rc;
        }
        *out = block.p + used;
        used += n;
        return XKB_OK;
    }
private:
    int grow(size_t n)
    {
        const int rc = block.take(n);
        release();
        return rc;
    }
};

} // namespace xkb

using namespace xkb;

struct xkb_resolver {
    cudaStream_t stream = nullptr;
    Domain interval;
    Domain handles;                             // handle accesses: one point per handle
    std::vector<std::unique_ptr<Domain>> blas;
    std::map<std::pair<uint64_t, uint64_t>, size_t> blas_index;
    std::vector<xkb_access_rec_t> segments;     // every segment so far, spawn order (replay)
    uint32_t ntasks = 0;
    // device work buffers
    DevBuf<DOp> dops;
    DevBuf<HOp> hops;                           // the batch's ops in byte coordinates
    DevBuf<uint64_t> hset, ukeys, bounds;       // compression: hash sets, distinct keys, sorted boundaries
    DevBuf<unsigned> ucount;
    DevBuf<unsigned long long> emit, table;
    // unique edges, appended batch by batch into segments (a batch's edges all end in the
    // batch's own tasks, so batches never repeat each other's pairs); a new segment starts when
    // the last one cannot take a batch's worst case, so stored edges are never moved
    std::vector<std::unique_ptr<DevBuf<unsigned long long>>> useg;
    std::vector<size_t> useg_n;
    DevBuf<unsigned long long> counters;        // CNT_*
    DevBuf<int> maps;                           // refinement: the old cell row / column of each new one
    DevBuf<int> spill;                          // reader spill chunks (SPILL ints each)
    DevBuf<unsigned> spill_ctr;                 // [0] chunks handed out, [1] ran-out flag
    size_t spill_chunks = 0;                    // pool capacity in chunks
    unsigned spill_used = 0;                    // chunks in use after the last completed step
    size_t nuniq = 0;
    // graph
    DevBuf<uint32_t> succ_ptr, succ, npred, tmp;
    DevBuf<uint32_t> win_ptr, win_succ, win_npred, win_tmp;   // window graphs (a runtime running the graph in pieces)
    DevBuf<uint32_t> periodic;                  // packed arrays of the periodic form
    DevBuf<unsigned> bin_off, bin_cur;          // ops binned to regions: offsets, fill cursors
    DevBuf<int> bin_list, bin_sorted;           // op indices per region, as filled and in op order
    bool graph_valid = false;
    double last_device_ms = 0;
    double last_ops_ms = 0, last_compress_ms = 0;   // host phases of the last batch
    double emit_per_op = 32.0;                  // emitted-pair estimate per op (from the last batch)
    double uniq_per_op = 8.0;                   // unique-pair estimate per op
    HostScratch host;
    cudaEvent_t ev[2] = {nullptr, nullptr};     // around the last batch
    const uint64_t ctx = context_id();
    xkb_resolver() { PinnedBlocks::enter(ctx); }
    ~xkb_resolver()
    {
        for (cudaEvent_t e : ev) if (e) cudaEventDestroy(e);
        host.drop(); stage.drop();
        PinnedBlocks::leave(ctx);
    }
    // parallel host passes (validation, op build): the host team and the page-locked staging buffer
    std::unique_ptr<WorkPool> pool;
    HostStage stage;
    bool staged = false;                        // this batch's ops are in `stage`
};

namespace xkb {

static int seg_rects_blas(uint64_t a, uint64_t b, uint64_t ld, uint64_t s, HRect out[3])
{
    const uint64_t LDs = ld * s, size = b - a;
    const uint64_t x0 = a % LDs, x1 = std::min(x0 + size, LDs), dx10 = x1 - x0;
    const uint64_t x3 = (size - dx10) % LDs;
    const uint64_t y0 = a / LDs, y1 = y0 + 1;
    const uint64_t y3 = y0 + (size - dx10 - x3) / LDs + 2, y2 = y3 - 1;
    const HRect r[3] = {{x0, x1, y0, y1}, {0, LDs, y1, y2}, {0, x3, y2, y3}};
    int n = 0;
    for (const HRect & q : r) if (q.x0 < q.x1 && q.y0 < q.y1) out[n++] = q;
    return n;
}

static int mat_rects(const xkb_access_rec_t & r, HRect out[2])
{
    const uint64_t s = r.sizeof_type, ld = r.ld, LDs = ld * s;
    const uint64_t A = r.addr + (r.offset_n * ld + r.offset_m) * s;
    const uint64_t x0 = A % LDs, y0 = A / LDs;
    if (x0 + r.m * s <= LDs) { out[0] = {x0, x0 + r.m * s, y0, y0 + r.n}; return 1; }
    out[0] = {x0, LDs, y0, y0 + r.n};
    out[1] = {0, r.m * s - (LDs - x0), y0 + 1, y0 + r.n + 1};
    return 2;
}

static void push_ops(Domain & d, bool link, const xkb_access_rec_t & r)
{
    HRect rects[3];
    int n;
    if (r.type == XKB_ACCESS_TYPE_HANDLE)
    {
        // a handle is one point of its own domain; the handle map records every access with
        // the R bit and no W bit as a reader (dependency-map.hpp put()), so such modes count as R
        const uint8_t m = ((r.mode & M_R) && !(r.mode & M_W)) ? M_R : r.mode;
        d.ops.push_back({r.task, (uint8_t) link, m, HRect{r.addr, r.addr + 1, 0, 1}});
        return;
    }
    if (d.interval) { rects[0] = {r.addr, r.ld, 0, 1}; n = 1; }
    else if (r.type == XKB_ACCESS_TYPE_SEGMENT) n = seg_rects_blas(r.addr, r.ld, d.ld, d.s, rects);
    else n = mat_rects(r, rects);
    for (int i = 0; i < n; ++i)
    {
        HRect q = rects[i];
        if (!link && !d.interval && r.type == XKB_ACCESS_TYPE_SEGMENT)
        {
            q.x0 = std::max(q.x0, r.addr); q.x1 = std::min(q.x1, r.ld);
            q.y1 = std::min<uint64_t>(q.y1, 1);
            if (q.x0 >= q.x1 || q.y0 >= q.y1) continue;
        }
        d.ops.push_back({r.task, (uint8_t) link, r.mode, q});
    }
}

// First record of [b, e) that is malformed or breaks the dense task numbering (its task must be
// the previous record's or the next one, starting at first_task), with the reason; e if none.
static size_t first_invalid(const xkb_access_rec_t * recs, size_t b, size_t e, uint32_t first_task, const char ** why)
{
    for (size_t i = b; i < e; ++i)
    {
        const xkb_access_rec_t & r = recs[i];
        const uint32_t prev = i == 0 ? first_task : recs[i - 1].task;
        if (r.task < prev || r.task > prev + 1 || (i == 0 && r.task != first_task)) { *why = "task ids must be dense, in spawn order"; return i; }
        if (r.mode == 0 || (r.mode & ~15u)) { *why = "bad mode"; return i; }
        const unsigned conc = r.reserved >> 8;      // sequential (0, 1) or commutative (2)
        if (conc == 4) { *why = "a concurrent access: expand the stream with xkb_handle_map_expand first"; return i; }
        if (conc > 2) { *why = "bad concurrency"; return i; }
        if (r.type == XKB_ACCESS_TYPE_SEGMENT) {
            if (r.ld <= r.addr) { *why = "empty segment"; return i; }
        } else if (r.type == XKB_ACCESS_TYPE_BLAS_MATRIX) {
            if (!r.ld || !r.sizeof_type || !r.m || !r.n || r.m > r.ld) { *why = "bad matrix tile"; return i; }
        } else if (r.type == XKB_ACCESS_TYPE_HANDLE) {
            if (r.addr == ~0ull) { *why = "handle ~0 is reserved"; return i; }
        } else { *why = "unsupported access type"; return i; }
    }
    return e;
}

// Validate a batch (on the host team when it is large).
static int validate(xkb_resolver * R, const xkb_access_rec_t * recs, size_t n, uint32_t first_task)
{
    const char * why = "";
    size_t bad = n;
    if (n >= 65536 && R->pool && R->pool->size() > 1)
    {
        const unsigned nc = R->pool->size();
        std::vector<size_t> at(nc, n);
        std::vector<const char *> w(nc, "");
        R->pool->run([&](unsigned c) {
            const size_t e = n * (c + 1) / nc;
            const size_t x = first_invalid(recs, n * c / nc, e, first_task, &w[c]);
            at[c] = x == e ? n : x;
        });
        for (unsigned c = 0; c < nc; ++c) if (at[c] < bad) { bad = at[c]; why = w[c]; }
    }
    else bad = first_invalid(recs, 0, n, first_task, &why);
    if (bad < n) return xkb_set_error(XKB_EINVAL, "resolver: access %zu: %s (tasks continue at %u)", bad, why, first_task);
    return XKB_OK;
}

// Rects of a matrix record in its frame (mat_rects' count only).
static inline int mat_nrects(const xkb_access_rec_t & r)
{
    const uint64_t LDs = r.ld * r.sizeof_type, A = r.addr + (r.offset_n * r.ld + r.offset_m) * r.sizeof_type;
    return (A % LDs) + r.m * r.sizeof_type <= LDs ? 1 : 2;
}

// Refuse a batch with more ops in one domain than the kernels can number; none of its ops is kept.
static int check_ops(xkb_resolver * R)
{
    uint64_t most = std::max<uint64_t>(R->interval.nops, R->handles.nops);
    for (auto & d : R->blas) most = std::max<uint64_t>(most, d->nops);
    if (most <= RESOLVE_MAX_OPS) return XKB_OK;
    auto drop = [](Domain & d) { d.ops.clear(); d.nops = d.nhops = 0; };
    drop(R->interval); drop(R->handles);
    for (auto & d : R->blas) drop(*d);
    return xkb_set_error(XKB_ERANGE, "resolver: %llu ops of one domain in a batch (at most %llu): add it in smaller batches",
                         (unsigned long long) most, (unsigned long long) RESOLVE_MAX_OPS);
}

// Matrix-only batches whose every (ld, sizeof) already has a domain: each record's ops go to its
// own domain only (LINK ops of a task's records, then their PUT ops), so chunks of whole tasks
// are built on their own -- by the host team when the batch is large: a counting pass, then every
// chunk writes its ops straight into the page-locked staging buffer, domain after domain and chunks
// in order within a domain, one per rect: the device makes the LINK and the PUT op of it
// (map_ops_kernel). Counters and cursors live on each member's own stack while it runs (members
// sharing cache lines would serialise on them). Returns 1 (built), 0 (the batch needs the
// sequential path: a segment or handle, or a matrix key seen for the first time after a segment -- a
// new domain replays earlier segments at that point of the stream), or an error.
constexpr size_t TEAM_RECORDS = 16384;      // records from which the host team pays (waking it: about 20 us a pass)

static int build_ops_staged(xkb_resolver * R, const xkb_access_rec_t * recs, size_t n)
{
    const unsigned nc = n >= TEAM_RECORDS && R->pool ? R->pool->size() : 1;
    auto team = [&](const std::function<void(unsigned)> & fn) { if (nc > 1) R->pool->run(fn); else fn(0); };
    if (R->segments.empty())
    {
        // no segment seen yet, so a new matrix domain replays nothing: create the batch's new
        // ones up front, in the order the sequential build would meet them
        std::vector<char> other(nc, 0), fresh(nc, 0);
        team([&](unsigned c) {
            uint64_t lk = ~0ull, ls = ~0ull;
            for (size_t i = n * c / nc; i < n * (c + 1) / nc; ++i)
            {
                const xkb_access_rec_t & r = recs[i];
                if (r.type != XKB_ACCESS_TYPE_BLAS_MATRIX) { other[c] = 1; return; }
                if (r.ld == lk && r.sizeof_type == ls) continue;
                lk = r.ld; ls = r.sizeof_type;
                if (!R->blas_index.count(std::make_pair(r.ld, r.sizeof_type))) fresh[c] = 1;
            }
        });
        for (char o : other) if (o) return 0;
        bool any = false;
        for (char f : fresh) any = any || f;
        uint64_t lk = ~0ull, ls = ~0ull;
        if (any)
            for (size_t i = 0; i < n; ++i)
            {
                if (recs[i].ld == lk && recs[i].sizeof_type == ls) continue;
                lk = recs[i].ld; ls = recs[i].sizeof_type;
                const auto key = std::make_pair(lk, ls);
                if (R->blas_index.count(key)) continue;
                std::unique_ptr<Domain> d(new Domain());
                d->ld = key.first; d->s = key.second;
                d->state[0].use_pool(R->stream); d->state[1].use_pool(R->stream);
                R->blas.push_back(std::move(d));
                R->blas_index.emplace(key, R->blas.size() - 1);
            }
    }
    if (R->blas.empty()) return 0;
    const size_t nd = R->blas.size();
    std::vector<uint64_t> keys(2 * nd);
    for (size_t k = 0; k < nd; ++k) { keys[2 * k] = R->blas[k]->ld; keys[2 * k + 1] = R->blas[k]->s; }
    auto dom_of = [&](const xkb_access_rec_t & r, uint64_t & lk, uint64_t & ls, size_t & li) {
        if (r.ld == lk && r.sizeof_type == ls) return true;
        for (size_t k = 0; k < nd; ++k)
            if (keys[2 * k] == r.ld && keys[2 * k + 1] == r.sizeof_type) { lk = r.ld; ls = r.sizeof_type; li = k; return true; }
        return false;
    };
    std::vector<size_t> cut(nc + 1, n);
    cut[0] = 0;
    for (unsigned t = 1; t < nc; ++t)
    {
        size_t c = std::max(cut[t - 1], n * t / nc);
        while (c > cut[t - 1] && c < n && recs[c].task == recs[c - 1].task) ++c;     // whole tasks per chunk
        cut[t] = c;
    }
    std::vector<size_t> cnt(nc * nd, 0);
    std::vector<char> ok(nc, 1);
    team([&](unsigned c) {
        uint64_t lk = ~0ull, ls = ~0ull;
        size_t li = 0;
        std::vector<size_t> my(nd, 0);
        for (size_t i = cut[c]; i < cut[c + 1]; ++i)
        {
            const xkb_access_rec_t & r = recs[i];
            if (r.type != XKB_ACCESS_TYPE_BLAS_MATRIX || !dom_of(r, lk, ls, li)) { ok[c] = 0; return; }
            my[li] += (size_t) mat_nrects(r);
        }
        std::copy(my.begin(), my.end(), cnt.begin() + c * nd);
    });
    for (char o : ok) if (!o) return 0;
    std::vector<size_t> pos(nc * nd);
    size_t total = 0;
    for (size_t k = 0; k < nd; ++k)
    {
        const size_t first = total;
        for (unsigned c = 0; c < nc; ++c) { pos[c * nd + k] = total; total += cnt[c * nd + k]; }
        R->blas[k]->nhops = total - first;
        R->blas[k]->nops = 2 * R->blas[k]->nhops;
    }
    if (int rc = check_ops(R)) return rc;
    if (int rc = R->stage.take(total ? total : 1)) return rc;
    HOp * out = R->stage.ops();
    team([&](unsigned c) {
        uint64_t lk = ~0ull, ls = ~0ull;
        size_t li = 0;
        std::vector<size_t> p(pos.begin() + c * nd, pos.begin() + (c + 1) * nd);
        for (size_t i = cut[c]; i < cut[c + 1]; ++i)
        {
            dom_of(recs[i], lk, ls, li);
            HRect rr[2];
            const int nr = mat_rects(recs[i], rr);
            for (int q = 0; q < nr; ++q) stream_op(out + p[li]++, HOp{recs[i].task, 1, recs[i].mode, rr[q]});
        }
        stream_fence();
    });
    R->staged = true;
    return 1;
}

// Build every domain's op list for the batch, in the order the reference performs them.
static void build_ops(xkb_resolver * R, const xkb_access_rec_t * recs, size_t n)
{
    for (size_t i = 0; i < n;)
    {
        size_t j = i;
        while (j < n && recs[j].task == recs[i].task) ++j;
        for (size_t a = i; a < j; ++a)                          // LINK pass
        {
            const xkb_access_rec_t & r = recs[a];
            if (r.type == XKB_ACCESS_TYPE_HANDLE) push_ops(R->handles, true, r);
            else if (r.type == XKB_ACCESS_TYPE_SEGMENT)
            {
                push_ops(R->interval, true, r);
                for (auto & d : R->blas) push_ops(*d, true, r);
            }
            else
            {
                const auto key = std::make_pair(r.ld, r.sizeof_type);
                auto it = R->blas_index.find(key);
                if (it == R->blas_index.end())
                {
                    std::unique_ptr<Domain> d(new Domain());
                    d->ld = r.ld; d->s = r.sizeof_type;
                    d->state[0].use_pool(R->stream); d->state[1].use_pool(R->stream);
                    for (auto k = R->segments.rbegin(); k != R->segments.rend(); ++k) push_ops(*d, false, *k);
                    R->blas.push_back(std::move(d));
                    it = R->blas_index.emplace(key, R->blas.size() - 1).first;
                }
                push_ops(*R->blas[it->second], true, r);
            }
        }
        for (size_t a = i; a < j; ++a)                          // PUT pass
        {
            const xkb_access_rec_t & r = recs[a];
            if (r.type == XKB_ACCESS_TYPE_HANDLE) push_ops(R->handles, false, r);
            else if (r.type == XKB_ACCESS_TYPE_SEGMENT)
            {
                push_ops(R->interval, false, r);
                for (auto & d : R->blas) push_ops(*d, false, r);
                R->segments.push_back(r);
            }
            else
                push_ops(*R->blas[R->blas_index.at({r.ld, r.sizeof_type})], false, r);
        }
        i = j;
    }
}

// Extend the domain's compression with the batch's boundaries; remap the device state when
// the cell grid changes.
// The spill pool: created on first use; grown keeping its chunks (cell states name them by
// index). reset_spill() rewinds the hand-out counter to the last completed step before a kernel
// that may run out of chunks and be redone.
static int spill_reserve(xkb_resolver * R, size_t chunks)
{
    if (!R->spill_ctr.p)
    {
        int rc = R->spill_ctr.reserve(2);
        if (rc) return rc;
        XKB_CUDA_TRY(cudaMemsetAsync(R->spill_ctr.p, 0, 2 * sizeof(unsigned), R->stream));
    }
    if (chunks <= R->spill_chunks) return XKB_OK;
    size_t c = R->spill_chunks ? R->spill_chunks : 65536;
    while (c < chunks) c *= 2;
    if (c > 0xffffffffu / 2) return xkb_set_error(XKB_ERANGE, "resolver: reader spill pool exceeds 2^31 chunks");
    int * q = nullptr;
    cudaError_t e = cudaMalloc(&q, c * SPILL * sizeof(int));
    if (e != cudaSuccess) return xkb_set_cuda_error(e);
    if (R->spill.p && R->spill_used)
    {
        e = cudaMemcpyAsync(q, R->spill.p, (size_t) R->spill_used * SPILL * sizeof(int), cudaMemcpyDeviceToDevice, R->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(R->stream);
        if (e != cudaSuccess) { cudaFree(q); return xkb_set_cuda_error(e); }
    }
    if (R->spill.p) cudaFree(R->spill.p);
    R->spill.p = q; R->spill.cap = c * SPILL; R->spill_chunks = c;
    return XKB_OK;
}

__global__ void set_spill_kernel(unsigned * ctr, unsigned used) { ctr[0] = used; ctr[1] = 0; }

static int reset_spill(xkb_resolver * R)
{
    set_spill_kernel<<<1, 1, 0, R->stream>>>(R->spill_ctr.p, R->spill_used);
    XKB_CUDA_TRY(cudaGetLastError());
    return XKB_OK;
}

// After a kernel that draws chunks: true (and the pool grown) if it ran out and must be redone;
// else the chunks it drew become part of the kept state.
static int spill_check(xkb_resolver * R, bool & redo)
{
    unsigned v[2];
    XKB_CUDA_TRY(cudaMemcpyAsync(v, R->spill_ctr.p, sizeof(v), cudaMemcpyDeviceToHost, R->stream));
    XKB_CUDA_TRY(cudaStreamSynchronize(R->stream));
    redo = v[1] != 0;
    if (redo) return spill_reserve(R, (size_t) v[0] + 1);
    R->spill_used = v[0];
    return XKB_OK;
}

// XKB_TRACE_RESOLVE=2: the time each step of a batch's compression and region pass takes
// (host clock, so a step that synchronises includes the device work queued before it).
struct PhaseTrace {
    const bool on;
    const char * what;
    std::chrono::steady_clock::time_point t = std::chrono::steady_clock::now();
    std::string line;
    explicit PhaseTrace(const char * w) : on(trace_level() >= 2), what(w) {}
    static int trace_level() { static const int l = getenv("XKB_TRACE_RESOLVE") ? atoi(getenv("XKB_TRACE_RESOLVE")) : 0; return l; }
    void mark(const char * step)
    {
        if (!on) return;
        const auto n = std::chrono::steady_clock::now();
        char b[96];
        snprintf(b, sizeof(b), " %s %.1f", step, std::chrono::duration<double, std::milli>(n - t).count());
        line += b; t = n;
    }
    ~PhaseTrace() { if (on) fprintf(stderr, "  %s (ms):%s\n", what, line.c_str()); }
};

static int refine_domain(xkb_resolver * R, Domain & d, std::vector<uint64_t> & xs, std::vector<uint64_t> & ys)
{
    if (xs.size() < 2 || ys.size() < 2) { d.xs = xs; d.ys = ys; return XKB_OK; }
    const bool same = xs == d.xs && ys == d.ys;
    const size_t ncx = xs.size() - 1, ncy = ys.size() - 1, ncells = ncx * ncy;
    if (same && d.ncells == ncells) return XKB_OK;
    int rc;
    PhaseTrace pt("refine");
    DevBuf<int> & out = d.state[d.cur ^ 1];
    if ((rc = out.reserve(ncells * STRIDE))) return rc;
    pt.mark("state-reserve");
    if (d.ncells == 0)
    {
        init_state_kernel<<<(unsigned) ((ncells + 255) / 256), 256, 0, R->stream>>>(out.p, ncells);
    }
    else
    {
        const size_t old_ncx = d.xs.size() - 1;
        if ((rc = R->maps.reserve(ncx + ncy))) return rc;
        void * m = nullptr;
        if ((rc = R->host.take((ncx + ncy) * sizeof(int), R->stream, &m))) return rc;
        int * mx = (int *) m, * my = mx + ncx;
        for (size_t i = 0; i < ncx; ++i) {
            const uint64_t v = xs[i];
            if (v < d.xs.front() || v >= d.xs.back()) mx[i] = -1;
            else mx[i] = (int) (std::upper_bound(d.xs.begin(), d.xs.end(), v) - d.xs.begin()) - 1;
        }
        for (size_t i = 0; i < ncy; ++i) {
            const uint64_t v = ys[i];
            if (v < d.ys.front() || v >= d.ys.back()) my[i] = -1;
            else my[i] = (int) (std::upper_bound(d.ys.begin(), d.ys.end(), v) - d.ys.begin()) - 1;
        }
        XKB_CUDA_TRY(cudaMemcpyAsync(R->maps.p, mx, (ncx + ncy) * sizeof(int), cudaMemcpyHostToDevice, R->stream));
        pt.mark("maps");
        if ((rc = spill_reserve(R, 1))) return rc;
        pt.mark("spill-reserve");
        for (bool redo = true; redo;)
        {
            if ((rc = reset_spill(R))) return rc;
            refine_state_kernel<<<(unsigned) ((ncells + 255) / 256), 256, 0, R->stream>>>(
                d.state[d.cur].p, out.p, R->maps.p, R->maps.p + ncx, (int) ncx, (int) ncy, (int) old_ncx, R->spill.p, R->spill_ctr.p,
                (unsigned) R->spill_chunks);
            XKB_CUDA_TRY(cudaGetLastError());
            if ((rc = spill_check(R, redo))) return rc;
            pt.mark("refine-kernel+sync");
        }
    }
    XKB_CUDA_TRY(cudaGetLastError());
    d.cur ^= 1;
    d.xs.swap(xs); d.ys.swap(ys); d.ncells = ncells;
    return XKB_OK;
}

// Let a launch on the current device ask for `bytes` of dynamic shared memory. The limit is the
// kernel's, for every host thread, so it is always set to `most`, what the kernel may ever need: a
// limit of just this call's bytes would take it from another thread's batch before its launch.
template <typename K>
static int allow_smem(K kernel, size_t bytes, size_t most)
{
    if (bytes > 48 * 1024) XKB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) most));
    return XKB_OK;
}

static int device_sms()
{
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// Bin the batch's ops to regions (counts, offsets, fill, per-region sort) and run the segment kernel
// over each region's own list.
template <int RX, int RY>
static int launch_region(xkb_resolver * R, ResolveArgs & a, int nregions)
{
    const size_t smem = (size_t) RCAP * RX * RY * sizeof(int);
    cudaStream_t st = R->stream;
    const size_t nb = (size_t) nregions + 1;
    int rc;
    PhaseTrace pt("regions");
    if ((rc = R->bin_off.reserve(nb)) || (rc = R->bin_cur.reserve(nb)) || (rc = R->tmp.reserve(nb / SCAN_TILE + 2))) return rc;
    pt.mark("reserve");
    XKB_CUDA_TRY(cudaMemsetAsync(R->bin_off.p, 0, nb * sizeof(unsigned), st));
    XKB_CUDA_TRY(cudaMemsetAsync(R->bin_cur.p, 0, nb * sizeof(unsigned), st));
    const unsigned g = (unsigned) ((a.nops + 255) / 256);
    // block-local binning: a grid of a few blocks per SM, each walking its share of the ops
    const char * gb = getenv("XKB_RESOLVE_BIN_GLOBAL");             // 1: the global-atomic binning (tests)
    const bool smem_bins = nregions <= BIN_SMEM_REGIONS && !(gb && atoi(gb) == 1);
    const unsigned gs = std::min<unsigned>(g, (unsigned) (2 * device_sms()));
    const size_t bins = (size_t) nregions * sizeof(unsigned), bins_most = BIN_SMEM_REGIONS * sizeof(unsigned);
    if (smem_bins)
    {
        if ((rc = allow_smem(bin_count_smem_kernel, bins, bins_most))) return rc;
        bin_count_smem_kernel<<<gs, 256, bins, st>>>(a.ops, a.nops, RX, RY, a.nrx, nregions, R->bin_off.p);
    }
    else
        bin_count_kernel<<<g, 256, 0, st>>>(a.ops, a.nops, RX, RY, a.nrx, R->bin_off.p);
    if ((rc = device_exclusive_scan(R->bin_off.p, R->bin_off.p, nb, R->tmp.p, nullptr, st))) return rc;
    unsigned * total_p = (unsigned *) R->host.results();
    XKB_CUDA_TRY(cudaMemcpyAsync(total_p, R->bin_off.p + nregions, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    XKB_CUDA_TRY(cudaStreamSynchronize(st));
    R->host.release();
    const unsigned total = *total_p;
    pt.mark("count+sync");
    if (total)
    {
        if ((rc = R->bin_list.reserve(total)) || (rc = R->bin_sorted.reserve(total))) return rc;
        if (smem_bins)
        {
            if ((rc = allow_smem(bin_fill_smem_kernel, 2 * bins, 2 * bins_most))) return rc;
            bin_fill_smem_kernel<<<gs, 256, 2 * bins, st>>>(a.ops, a.nops, RX, RY, a.nrx, nregions, R->bin_off.p, R->bin_cur.p,
                                                            R->bin_list.p);
        }
        else
            bin_fill_kernel<<<g, 256, 0, st>>>(a.ops, a.nops, RX, RY, a.nrx, R->bin_off.p, R->bin_cur.p, R->bin_list.p);
        const int words = std::max(BIN_SORT_SHORT, std::min(BIN_SORT_WORDS, (a.nops + 31) / 32));
        if ((rc = allow_smem(bin_sort_kernel, (size_t) words * sizeof(unsigned), BIN_SORT_WORDS * sizeof(unsigned)))) return rc;
        bin_sort_kernel<<<(unsigned) nregions, BIN_SORT_THREADS, (size_t) words * sizeof(unsigned), st>>>(R->bin_off.p, R->bin_list.p,
                                                                                                          R->bin_sorted.p, a.nops, words);
    }
    // segments per region from the mean list length (a segment of a few hundred ops still amortises its
    // look-back); XKB_RESOLVE_SEGMENTS overrides (1 = one pass per region)
    const char * seg_s = getenv("XKB_RESOLVE_SEGMENTS");
    const int seg_env = seg_s ? atoi(seg_s) : 0;
    int nseg = seg_env > 0 ? seg_env : (int) std::min<size_t>(MAX_SEGMENTS, std::max<size_t>(1, (size_t) total / nregions / SEGMENT_OPS));
    nseg = std::max(1, std::min(nseg, MAX_SEGMENTS));
    resolve_segment_kernel<RX, RY><<<(unsigned) (nregions * nseg), RX * RY, smem, st>>>(a, R->bin_off.p, R->bin_sorted.p, nseg);
    XKB_CUDA_TRY(cudaGetLastError());
    return XKB_OK;
}

static int launch_domain(xkb_resolver * R, Domain & d, size_t op_offset, size_t nops)
{
    const int ncx = (int) d.xs.size() - 1, ncy = (int) d.ys.size() - 1;
    ResolveArgs a;
    a.ops = R->dops.p + op_offset; a.nops = (int) nops;
    a.ncx = ncx; a.ncy = ncy;
    a.state_in = d.state[d.cur].p; a.state_out = d.state[d.cur ^ 1].p;
    a.emit = R->emit.p; a.emit_count = R->counters.p; a.emit_cap = R->emit.cap;
    a.spill = R->spill.p; a.spill_ctr = R->spill_ctr.p; a.spill_cap = (unsigned) R->spill_chunks;
    if (ncy == 1)
    {
        constexpr int RX = 64, RY = 1;
        a.nrx = (ncx + RX - 1) / RX;
        return launch_region<RX, RY>(R, a, a.nrx);
    }
    constexpr int RX = 8, RY = XKB_REGION_RY;
    a.nrx = (ncx + RX - 1) / RX;
    const int nry = (ncy + RY - 1) / RY;
    return launch_region<RX, RY>(R, a, a.nrx * nry);
}

// Compress the domain's coordinates with the batch's boundaries (found on the device, merged with
// the domain's earlier ones on the host), refine the cell state, and write the batch's ops in cell
// coordinates to dops. hops: this domain's nops uploaded ops on the device, each two of dops if paired.
static int compress_domain(xkb_resolver * R, Domain & d, const HOp * hops, DOp * dops, size_t nops, bool paired)
{
    cudaStream_t st = R->stream;
    size_t cap = 1024;
    while (cap < 4 * nops) cap *= 2;
    int rc;
    PhaseTrace pt("compress");
    if ((rc = R->hset.reserve(2 * cap)) || (rc = R->ukeys.reserve(4 * nops)) || (rc = R->ucount.reserve(3))) return rc;
    pt.mark("reserve");
    XKB_CUDA_TRY(cudaMemsetAsync(R->hset.p, 0xff, 2 * cap * sizeof(uint64_t), st));
    XKB_CUDA_TRY(cudaMemsetAsync(R->ucount.p, 0, 3 * sizeof(unsigned), st));
    const unsigned g = (unsigned) ((nops + 255) / 256);
    collect_bounds_kernel<<<g, 256, 0, st>>>(hops, (int) nops, R->hset.p, R->hset.p + cap, (uint32_t) (cap - 1),
                                             R->ukeys.p, R->ukeys.p + 2 * nops, R->ucount.p);
    XKB_CUDA_TRY(cudaGetLastError());
    // the counts and the first keys come back together: most batches have no more
    unsigned * cnt = (unsigned *) R->host.results();
    const size_t some = std::min<size_t>(HostScratch::KEYS, 2 * nops);
    XKB_CUDA_TRY(cudaMemcpyAsync(cnt, R->ucount.p, 3 * sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    XKB_CUDA_TRY(cudaMemcpyAsync(R->host.keys(0), R->ukeys.p, some * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    XKB_CUDA_TRY(cudaMemcpyAsync(R->host.keys(1), R->ukeys.p + 2 * nops, some * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    XKB_CUDA_TRY(cudaStreamSynchronize(st));
    R->host.release();
    pt.mark("collect+sync");
    std::vector<uint64_t> xs(d.xs.size() + cnt[0] + 1), ys(d.ys.size() + cnt[1] + 1);
    std::copy(d.xs.begin(), d.xs.end(), xs.begin());
    std::copy(d.ys.begin(), d.ys.end(), ys.begin());
    std::copy_n(R->host.keys(0), std::min<size_t>(cnt[0], some), xs.begin() + d.xs.size());
    std::copy_n(R->host.keys(1), std::min<size_t>(cnt[1], some), ys.begin() + d.ys.size());
    if (cnt[0] > some) XKB_CUDA_TRY(cudaMemcpyAsync(xs.data() + d.xs.size() + some, R->ukeys.p + some, (cnt[0] - some) * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    if (cnt[1] > some) XKB_CUDA_TRY(cudaMemcpyAsync(ys.data() + d.ys.size() + some, R->ukeys.p + 2 * nops + some, (cnt[1] - some) * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    if (cnt[0] > some || cnt[1] > some) XKB_CUDA_TRY(cudaStreamSynchronize(st));
    if (cnt[2] & 1u) xs.back() = KEY_EMPTY; else xs.pop_back();
    if (cnt[2] & 2u) ys.back() = KEY_EMPTY; else ys.pop_back();
    for (std::vector<uint64_t> * v : {&xs, &ys})
    {
        std::sort(v->begin(), v->end());
        v->erase(std::unique(v->begin(), v->end()), v->end());
    }
    pt.mark("keys+sort");
    if ((rc = refine_domain(R, d, xs, ys))) return rc;
    pt.mark("refine");
    if ((rc = R->bounds.reserve(d.xs.size() + d.ys.size()))) return rc;
    void * hb = nullptr;
    const size_t nbounds = d.xs.size() + d.ys.size();
    if ((rc = R->host.take(nbounds * sizeof(uint64_t), st, &hb))) return rc;
    std::copy(d.ys.begin(), d.ys.end(), std::copy(d.xs.begin(), d.xs.end(), (uint64_t *) hb));
    XKB_CUDA_TRY(cudaMemcpyAsync(R->bounds.p, hb, nbounds * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
    (paired ? map_ops_kernel<true> : map_ops_kernel<false>)<<<g, 256, 0, st>>>(hops, (int) nops, R->bounds.p, (int) d.xs.size(),
                                                                               R->bounds.p + d.xs.size(), (int) d.ys.size(), dops);
    XKB_CUDA_TRY(cudaGetLastError());
    pt.mark("map");
    return XKB_OK;
}

__global__ void set_uniq_kernel(unsigned long long * cnt, unsigned long long n) { cnt[CNT_UNIQ] = n; cnt[CNT_FULL] = 0; }

static int resolve_batch(xkb_resolver * R, const xkb_access_rec_t * recs, size_t n)
{
    int rc;
    using clk = std::chrono::steady_clock;
    const auto t0 = clk::now();
    if ((rc = R->host.init())) return rc;
    R->staged = false;
    rc = build_ops_staged(R, recs, n);
    if (rc < 0) return rc;
    if (!R->staged)
    {
        build_ops(R, recs, n);
        R->interval.nops = R->interval.nhops = R->interval.ops.size();
        R->handles.nops = R->handles.nhops = R->handles.ops.size();
        for (auto & d : R->blas) d->nops = d->nhops = d->ops.size();
        if ((rc = check_ops(R))) return rc;
    }
    const auto t1 = clk::now();
    std::vector<Domain *> doms;
    if (R->interval.nops) doms.push_back(&R->interval);
    if (R->handles.nops) doms.push_back(&R->handles);
    for (auto & d : R->blas) if (d->nops) doms.push_back(d.get());

    std::vector<size_t> offs, hoffs;            // each domain's first op, and first uploaded op
    size_t total = 0, htotal = 0;
    for (Domain * d : doms) { offs.push_back(total); hoffs.push_back(htotal); total += d->nops; htotal += d->nhops; }
    if ((rc = R->hops.reserve(htotal ? htotal : 1)) || (rc = R->dops.reserve(total ? total : 1))) return rc;
    if (R->staged)          // domain-major in the staging buffer, in the order of `doms`
    {
        if (htotal) XKB_CUDA_TRY(cudaMemcpyAsync(R->hops.p, R->stage.ops(), htotal * sizeof(HOp), cudaMemcpyHostToDevice, R->stream));
    }
    else
        for (size_t k = 0; k < doms.size(); ++k)
            XKB_CUDA_TRY(cudaMemcpyAsync(R->hops.p + hoffs[k], doms[k]->ops.data(), doms[k]->nhops * sizeof(HOp),
                                         cudaMemcpyHostToDevice, R->stream));
    for (size_t k = 0; k < doms.size(); ++k)
        if ((rc = compress_domain(R, *doms[k], R->hops.p + hoffs[k], R->dops.p + offs[k], doms[k]->nhops, R->staged))) return rc;
    R->last_ops_ms = std::chrono::duration<double, std::milli>(t1 - t0).count();
    R->last_compress_ms = std::chrono::duration<double, std::milli>(clk::now() - t1).count();

    static const bool trace = getenv("XKB_TRACE_RESOLVE") != nullptr;
    const size_t realloc0 = g_realloc_bytes;
    // the emit buffer, the hash set and the room for unique pairs are sized from the pairs per op of the
    // last batch (32 emitted and 8 unique per op before the first), within 2^28 pairs, so that nothing is read back between
    // the steps; what turns out too small is redone with what it needs
    size_t emit_guess = std::max<size_t>(1 << 16, std::min<size_t>(size_t(1) << 28, (size_t) (total * R->emit_per_op)));
    size_t uniq_guess = std::min<size_t>(emit_guess, std::max<size_t>(1 << 14, (size_t) (total * R->uniq_per_op)));
    bool regions = true;                       // false: only the unique step is redone
    auto ta = clk::now();
    for (int attempt = 0; attempt < 24; ++attempt)
    {
        if (regions)
        {
            ta = clk::now();
            if ((rc = R->emit.reserve(emit_guess)) || (rc = R->counters.reserve(CNT_COUNT))) return rc;
            if ((rc = spill_reserve(R, 1)) || (rc = reset_spill(R))) return rc;
            XKB_CUDA_TRY(cudaMemsetAsync(R->counters.p, 0, CNT_COUNT * sizeof(unsigned long long), R->stream));
            for (size_t k = 0; k < doms.size(); ++k)
            {
                const size_t nops = doms[k]->nops;
                // states must exist for every cell (ncells > 0 when the domain has >= 1 op)
                if (doms[k]->ncells == 0) continue;
                if ((rc = doms[k]->state[doms[k]->cur ^ 1].reserve(doms[k]->ncells * STRIDE))) return rc;
                if ((rc = launch_domain(R, *doms[k], offs[k], nops))) return rc;
            }
        }
        // unique the emitted pairs into the accumulated edge list
        size_t tcap = 1024;
        while (tcap < 2 * uniq_guess) tcap *= 2;
        if ((rc = R->table.reserve(tcap))) return rc;
        if (R->useg.empty() || R->useg.back()->cap - R->useg_n.back() < uniq_guess)
        {
            std::unique_ptr<DevBuf<unsigned long long>> seg(new (std::nothrow) DevBuf<unsigned long long>());
            if (!seg) return xkb_set_error(XKB_ENOMEM, "resolver: out of host memory");
            seg->use_pool(R->stream);
            // segments double in size, so a long stream allocates a few of them, not one per batch
            const size_t last = R->useg.empty() ? 0 : R->useg.back()->cap;
            if ((rc = seg->reserve(std::max<size_t>({uniq_guess, size_t(1) << 24, 2 * last})))) return rc;
            R->useg.push_back(std::move(seg));
            R->useg_n.push_back(0);
        }
        DevBuf<unsigned long long> & seg = *R->useg.back();
        const unsigned long long nu0 = R->useg_n.back();
        XKB_CUDA_TRY(cudaMemsetAsync(R->table.p, 0xff, tcap * sizeof(unsigned long long), R->stream));
        set_uniq_kernel<<<1, 1, 0, R->stream>>>(R->counters.p, nu0);
        dedupe_kernel<<<(unsigned) std::min<size_t>((emit_guess + 255) / 256, (size_t) device_sms() * 8), 256, 0, R->stream>>>(
            R->emit.p, R->emit.cap, R->table.p, tcap - 1, seg.p, R->counters.p, seg.cap);
        XKB_CUDA_TRY(cudaGetLastError());
        unsigned long long * cnt = (unsigned long long *) R->host.results();
        unsigned * sp = (unsigned *) (cnt + CNT_COUNT);
        XKB_CUDA_TRY(cudaMemcpyAsync(cnt, R->counters.p, CNT_COUNT * sizeof(unsigned long long), cudaMemcpyDeviceToHost, R->stream));
        XKB_CUDA_TRY(cudaMemcpyAsync(sp, R->spill_ctr.p, 2 * sizeof(unsigned), cudaMemcpyDeviceToHost, R->stream));
        XKB_CUDA_TRY(cudaStreamSynchronize(R->stream));
        R->host.release();
        const unsigned long long nemit = cnt[CNT_EMIT], nu = cnt[CNT_UNIQ];
        if (regions && sp[1])
        {
            // the reader spill pool ran out: grow it (keeping its chunks) and redo the batch
            if ((rc = spill_reserve(R, (size_t) sp[0] + 1))) return rc;
            continue;
        }
        if (nemit > R->emit.cap) { emit_guess = (size_t) nemit; uniq_guess = std::min<size_t>(2 * uniq_guess, emit_guess); regions = true; continue; }
        if (cnt[CNT_FULL])
        {
            // no room in the hash set or the segment: four times as much
            uniq_guess *= 4;
            regions = false;
            continue;
        }
        const auto tb = clk::now();
        R->spill_used = sp[0];
        if (total)
        {
            R->emit_per_op = std::max(2.0, 1.25 * (double) nemit / (double) total);
            R->uniq_per_op = std::max(1.0, 1.5 * (double) (nu - nu0) / (double) total);
        }
        R->nuniq += nu - nu0;
        R->useg_n.back() = nu;
        for (Domain * d : doms) { d->cur ^= 1; d->ops.clear(); d->nops = d->nhops = 0; }
        if (trace)
            fprintf(stderr, "resolver batch: %zu ops (built in %.2f ms, compressed in %.2f ms), attempt %d, regions and unique %.2f ms, "
                    "%llu emitted, %llu unique, %.1f MB allocated\n",
                    total, R->last_ops_ms, R->last_compress_ms, attempt, std::chrono::duration<double, std::milli>(tb - ta).count(),
                    nemit, nu - nu0, (g_realloc_bytes - realloc0) / 1e6);
        return XKB_OK;
    }
    return xkb_set_error(XKB_ERANGE, "resolver: batch did not fit after resizing");
}

static int build_graph(xkb_resolver * R)
{
    int rc;
    const size_t nt = R->ntasks, ne = R->nuniq;
    if ((rc = R->succ_ptr.reserve(nt + 1))) return rc;
    if ((rc = R->npred.reserve(nt + 1))) return rc;
    if ((rc = R->succ.reserve(ne ? ne : 1))) return rc;
    if ((rc = R->tmp.reserve(nt + 1 + (nt + 1) / SCAN_TILE + 2))) return rc;
    cudaStream_t st = R->stream;
    XKB_CUDA_TRY(cudaMemsetAsync(R->succ_ptr.p, 0, (nt + 1) * sizeof(uint32_t), st));
    XKB_CUDA_TRY(cudaMemsetAsync(R->npred.p, 0, (nt + 1) * sizeof(uint32_t), st));
    for (size_t k = 0; k < R->useg.size(); ++k)
        if (R->useg_n[k])
            count_edges_kernel<<<(unsigned) ((R->useg_n[k] + 255) / 256), 256, 0, st>>>(R->useg[k]->p, R->useg_n[k], R->succ_ptr.p,
                                                                                       R->npred.p);
    if ((rc = device_exclusive_scan(R->succ_ptr.p, R->succ_ptr.p, nt + 1, R->tmp.p + nt + 1, nullptr, st))) return rc;
    XKB_CUDA_TRY(cudaMemcpyAsync(R->tmp.p, R->succ_ptr.p, (nt + 1) * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
    for (size_t k = 0; k < R->useg.size(); ++k)
        if (R->useg_n[k])
            scatter_edges_kernel<<<(unsigned) ((R->useg_n[k] + 255) / 256), 256, 0, st>>>(R->useg[k]->p, R->useg_n[k], R->tmp.p,
                                                                                         R->succ.p);
    if (nt) sort_segments_kernel<<<(unsigned) ((nt + 7) / 8), 256, 0, st>>>(R->succ_ptr.p, R->succ.p, (uint32_t) nt);
    XKB_CUDA_TRY(cudaGetLastError());
    XKB_CUDA_TRY(cudaStreamSynchronize(st));
    R->graph_valid = true;
    return XKB_OK;
}

} // namespace xkb

extern "C" int xkb_resolver_create(xkb_resolver_t ** out, void * stream)
{
    if (!out) return xkb_set_error(XKB_EINVAL, "resolver_create: null output");
    int dev;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return xkb_set_cuda_error(e);
    xkb_resolver * R = new (std::nothrow) xkb_resolver();
    if (!R) return xkb_set_error(XKB_ENOMEM, "resolver_create: out of host memory");
    R->interval.interval = true;
    R->handles.interval = true;
    R->stream = (cudaStream_t) stream;
    // work buffers only this resolver's stream touches come from the pool in stream order (the
    // window graphs too: the runtime runs them on this stream); the graph it hands out
    // (succ_ptr, succ, npred, periodic form) stays in plain allocations, as a caller may read it
    // on other streams
    for (Domain * d : {&R->interval, &R->handles}) { d->state[0].use_pool(R->stream); d->state[1].use_pool(R->stream); }
    R->dops.use_pool(R->stream); R->hops.use_pool(R->stream);
    R->hset.use_pool(R->stream); R->ukeys.use_pool(R->stream); R->bounds.use_pool(R->stream); R->ucount.use_pool(R->stream);
    R->emit.use_pool(R->stream); R->table.use_pool(R->stream); R->counters.use_pool(R->stream);
    R->tmp.use_pool(R->stream); R->bin_off.use_pool(R->stream); R->bin_cur.use_pool(R->stream);
    R->bin_list.use_pool(R->stream); R->bin_sorted.use_pool(R->stream); R->maps.use_pool(R->stream);
    R->win_ptr.use_pool(R->stream); R->win_succ.use_pool(R->stream); R->win_npred.use_pool(R->stream);
    R->win_tmp.use_pool(R->stream);
    *out = R;
    return XKB_OK;
}

extern "C" int xkb_resolver_destroy(xkb_resolver_t * R)
{
    if (R) { cudaStreamSynchronize(R->stream); delete R; }
    return XKB_OK;
}

// Library-internal: forget every task and domain but keep the device work buffers, so the
// next graph resolves without allocating them again.
// Reserve, up front, the working memory one batch of about `nops` ops uses (the buffers grow on
// demand otherwise): op lists, compression hash sets, emitted and unique edges, staging, the host
// team. The cell states of each domain depend on its boundaries and still grow on demand.
int xkb_internal_resolver_prepare(xkb_resolver_t * R, size_t nops)
{
    if (!R) return xkb_set_error(XKB_EINVAL, "resolver_prepare: null resolver");
    if (nops == 0) return XKB_OK;
    if (!R->pool)
    {
        R->pool.reset(new (std::nothrow) WorkPool(xkb_internal_helpers()));
    }
    size_t cap = 1024;
    while (cap < 4 * nops) cap *= 2;
    // edge pairs: about 9 per op on tile stencils (the emit estimate after the first batches)
    const size_t emit = std::max<size_t>(1 << 16, nops * 12);
    size_t tcap = 1024;
    while (tcap < 2 * emit) tcap *= 2;
    int rc;
    if ((rc = R->hops.reserve(nops)) || (rc = R->dops.reserve(nops)) || (rc = R->hset.reserve(2 * cap)) ||
        (rc = R->ukeys.reserve(4 * nops)) || (rc = R->ucount.reserve(3)) || (rc = R->emit.reserve(emit)) ||
        (rc = R->counters.reserve(CNT_COUNT)) || (rc = R->table.reserve(tcap)) || (rc = R->stage.take((nops + 1) / 2)) || (rc = spill_reserve(R, 1)))
        return rc;
    R->stage.rest();                            // (kept for the batches to come; one op per LINK and PUT pair is staged)
    if (R->useg.empty())
    {
        std::unique_ptr<DevBuf<unsigned long long>> seg(new (std::nothrow) DevBuf<unsigned long long>());
        if (seg) seg->use_pool(R->stream);
        if (!seg) return xkb_set_error(XKB_ENOMEM, "resolver: out of host memory");
        if ((rc = seg->reserve(std::max<size_t>(emit, size_t(1) << 24)))) return rc;
        R->useg.push_back(std::move(seg));
        R->useg_n.push_back(0);
    }
    // the buffers still to come (cell states of each domain, region bins,
    // window graphs) grow from the pool: give it room now rather than while batches run
    if (cudaMemPool_t pool = resolver_pool())
    {
        void * w = nullptr;
        if (cudaMallocFromPoolAsync(&w, size_t(256) << 20, pool, R->stream) == cudaSuccess) cudaFreeAsync(w, R->stream);
        else cudaGetLastError();
    }
    XKB_CUDA_TRY(cudaStreamSynchronize(R->stream));
    return XKB_OK;
}

int xkb_internal_resolver_reset(xkb_resolver_t * R)
{
    if (!R) return xkb_set_error(XKB_EINVAL, "resolver_reset: null resolver");
    XKB_CUDA_TRY(cudaStreamSynchronize(R->stream));
    R->interval.xs.clear(); R->interval.ys.clear(); R->interval.ncells = 0; R->interval.ops.clear(); R->interval.nops = 0;
    R->handles.xs.clear(); R->handles.ys.clear(); R->handles.ncells = 0; R->handles.ops.clear(); R->handles.nops = 0;
    R->blas.clear(); R->blas_index.clear(); R->segments.clear();
    R->ntasks = 0; R->nuniq = 0; R->graph_valid = false;
    if (R->useg.size() > 1) { R->useg.resize(1); R->useg_n.resize(1); }   // keep the first edge segment
    for (size_t & n : R->useg_n) n = 0;
    R->spill_used = 0;
    return XKB_OK;
}

extern "C" int xkb_resolver_reset(xkb_resolver_t * R)
{
    return xkb_internal_resolver_reset(R);
}

extern "C" int xkb_resolver_add(xkb_resolver_t * R, const xkb_access_rec_t * recs, size_t n)
{
    if (!R || (n && !recs)) return xkb_set_error(XKB_EINVAL, "resolver_add: bad arguments");
    if (n == 0) return XKB_OK;
    if (!R->pool && n >= TEAM_RECORDS)
    {
        R->pool.reset(new (std::nothrow) WorkPool(xkb_internal_helpers()));
    }
    int rc = validate(R, recs, n, R->ntasks);
    if (rc) return rc;
    for (cudaEvent_t & e : R->ev) if (!e) XKB_CUDA_TRY(cudaEventCreate(&e));
    cudaEventRecord(R->ev[0], R->stream);
    rc = resolve_batch(R, recs, n);
    if (rc == XKB_OK) { R->ntasks = recs[n - 1].task + 1; R->graph_valid = false; }
    cudaEventRecord(R->ev[1], R->stream);
    cudaEventSynchronize(R->ev[1]);
    R->host.rest();                             // no copy of the batch is in flight any more
    R->stage.rest();
    float ms = 0; cudaEventElapsedTime(&ms, R->ev[0], R->ev[1]);
    R->last_device_ms = ms;
    return rc;
}

size_t xkb_internal_resolver_nedges(const xkb_resolver_t * R) { return R ? R->nuniq : 0; }

int xkb_internal_resolver_edge_mark(xkb_resolver_t * R, xkb_edge_mark_t * m)
{
    if (!R || !m) return xkb_set_error(XKB_EINVAL, "resolver_edge_mark: bad arguments");
    m->seg = R->useg.empty() ? 0 : R->useg.size() - 1;
    m->off = R->useg.empty() ? 0 : R->useg_n.back();
    m->ntasks = R->ntasks;
    return XKB_OK;
}

int xkb_internal_resolver_window_graph(xkb_resolver_t * R, const xkb_edge_mark_t * m, xkb_task_graph_t * g)
{
    if (!R || !m || !g || m->ntasks > R->ntasks) return xkb_set_error(XKB_EINVAL, "resolver_window_graph: bad arguments");
    const uint32_t first = m->ntasks;
    const size_t nt = R->ntasks - first;
    int rc;
    if ((rc = R->win_ptr.reserve(nt + 1)) || (rc = R->win_npred.reserve(nt + 1)) ||
        (rc = R->win_tmp.reserve(nt + 1 + (nt + 1) / SCAN_TILE + 2)))
        return rc;
    cudaStream_t st = R->stream;
    XKB_CUDA_TRY(cudaMemsetAsync(R->win_ptr.p, 0, (nt + 1) * sizeof(uint32_t), st));
    XKB_CUDA_TRY(cudaMemsetAsync(R->win_npred.p, 0, (nt + 1) * sizeof(uint32_t), st));
    // the edges stored since the mark: the rest of its segment, then every later segment
    auto each_range = [&](auto && fn) {
        for (size_t k = m->seg; k < R->useg.size(); ++k)
        {
            const size_t b = k == m->seg ? m->off : 0;
            if (R->useg_n[k] > b) fn(R->useg[k]->p + b, R->useg_n[k] - b);
        }
    };
    each_range([&](const unsigned long long * e, size_t n) {
        count_window_edges_kernel<<<(unsigned) ((n + 255) / 256), 256, 0, st>>>(e, n, first, R->win_ptr.p, R->win_npred.p);
    });
    if ((rc = device_exclusive_scan(R->win_ptr.p, R->win_ptr.p, nt + 1, R->win_tmp.p + nt + 1, nullptr, st))) return rc;
    uint32_t ne = 0;
    XKB_CUDA_TRY(cudaMemcpyAsync(&ne, R->win_ptr.p + nt, sizeof(ne), cudaMemcpyDeviceToHost, st));
    XKB_CUDA_TRY(cudaStreamSynchronize(st));
    if ((rc = R->win_succ.reserve(ne ? ne : 1))) return rc;
    XKB_CUDA_TRY(cudaMemcpyAsync(R->win_tmp.p, R->win_ptr.p, (nt + 1) * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
    each_range([&](const unsigned long long * e, size_t n) {
        scatter_window_edges_kernel<<<(unsigned) ((n + 255) / 256), 256, 0, st>>>(e, n, first, R->win_tmp.p, R->win_succ.p);
    });
    if (nt) sort_segments_kernel<<<(unsigned) ((nt + 7) / 8), 256, 0, st>>>(R->win_ptr.p, R->win_succ.p, (uint32_t) nt);
    XKB_CUDA_TRY(cudaGetLastError());
    g->ntasks = nt;
    g->nedges = ne;
    g->succ_ptr = R->win_ptr.p;
    g->succ = R->win_succ.p;
    g->npred = R->win_npred.p;
    return XKB_OK;
}

extern "C" int xkb_resolver_graph(xkb_resolver_t * R, xkb_task_graph_t * g)
{
    if (!R || !g) return xkb_set_error(XKB_EINVAL, "resolver_graph: bad arguments");
    if (!R->graph_valid) { int rc = build_graph(R); if (rc) return rc; }
    g->ntasks = R->ntasks;
    g->nedges = R->nuniq;
    g->succ_ptr = R->succ_ptr.p;
    g->succ = R->succ.p;
    g->npred = R->npred.p;
    return XKB_OK;
}

extern "C" int xkb_resolver_edges(xkb_resolver_t * R, uint32_t * pairs, size_t cap_pairs, size_t * nedges)
{
    if (!R || !nedges) return xkb_set_error(XKB_EINVAL, "resolver_edges: bad arguments");
    if (!R->graph_valid) { int rc = build_graph(R); if (rc) return rc; }
    *nedges = R->nuniq;
    if (R->nuniq > cap_pairs) return xkb_set_error(XKB_ERANGE, "resolver_edges: %zu pairs needed", R->nuniq);
    if (!pairs || R->nuniq == 0) return XKB_OK;
    std::vector<uint32_t> ptr(R->ntasks + 1), succ(R->nuniq);
    XKB_CUDA_TRY(cudaMemcpy(ptr.data(), R->succ_ptr.p, ptr.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    XKB_CUDA_TRY(cudaMemcpy(succ.data(), R->succ.p, succ.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    size_t k = 0;
    for (uint32_t t = 0; t < R->ntasks; ++t)
        for (uint32_t i = ptr[t]; i < ptr[t + 1]; ++i) { pairs[2 * k] = t; pairs[2 * k + 1] = succ[i]; ++k; }
    return XKB_OK;
}

extern "C" int xkb_resolver_stats(xkb_resolver_t * R, uint64_t * ntasks, uint64_t * nedges, double * last_batch_ms)
{
    if (!R) return xkb_set_error(XKB_EINVAL, "resolver_stats: null resolver");
    if (ntasks) *ntasks = R->ntasks;
    if (nedges) *nedges = R->nuniq;
    if (last_batch_ms) *last_batch_ms = R->last_device_ms;
    return XKB_OK;
}

extern "C" int xkb_resolver_timing(xkb_resolver_t * R, double * ops_ms, double * compress_ms, double * batch_ms)
{
    if (!R) return xkb_set_error(XKB_EINVAL, "resolver_timing: null resolver");
    if (ops_ms) *ops_ms = R->last_ops_ms;
    if (compress_ms) *compress_ms = R->last_compress_ms;
    if (batch_ms) *batch_ms = R->last_device_ms;
    return XKB_OK;
}

extern "C" int xkb_resolver_periodic(xkb_resolver_t * R, uint64_t period, xkb_periodic_graph_t * out)
{
    if (!R || !out || period == 0) return xkb_set_error(XKB_EINVAL, "resolver_periodic: bad arguments");
    if (R->ntasks != 3 * period)
        return xkb_set_error(XKB_EINVAL, "resolver_periodic: the resolver must hold exactly 3 windows (%llu tasks), it holds %u",
                             (unsigned long long) (3 * period), R->ntasks);
    if (!R->graph_valid) { int rc = build_graph(R); if (rc) return rc; }
    const size_t nt = R->ntasks, P = period;
    std::vector<uint32_t> ptr(nt + 1), succ(R->nuniq ? R->nuniq : 1), npred(nt);
    XKB_CUDA_TRY(cudaMemcpy(ptr.data(), R->succ_ptr.p, (nt + 1) * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    if (R->nuniq) XKB_CUDA_TRY(cudaMemcpy(succ.data(), R->succ.p, R->nuniq * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    XKB_CUDA_TRY(cudaMemcpy(npred.data(), R->npred.p, nt * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    // split the successors of window w into its own window and the next one
    auto split = [&](size_t w, std::vector<uint32_t> & ip, std::vector<uint32_t> & is,
                     std::vector<uint32_t> & xp, std::vector<uint32_t> & xs) -> bool {
        ip.assign(1, 0); xp.assign(1, 0); is.clear(); xs.clear();
        for (size_t t = w * P; t < (w + 1) * P; ++t)
        {
            for (uint32_t i = ptr[t]; i < ptr[t + 1]; ++i)
            {
                const uint32_t s = succ[i];
                if (s < (w + 1) * P) is.push_back((uint32_t) (s - w * P));
                else if (s < (w + 2) * P) xs.push_back((uint32_t) (s - (w + 1) * P));
                else return false;                              // an edge skips a window
            }
            ip.push_back((uint32_t) is.size()); xp.push_back((uint32_t) xs.size());
        }
        return true;
    };
    std::vector<uint32_t> ip0, is0, xp0, xs0, ip1, is1, xp1, xs1;
    if (!split(0, ip0, is0, xp0, xs0) || !split(1, ip1, is1, xp1, xs1))
        return xkb_set_error(XKB_EINVAL, "resolver_periodic: an edge skips a window");
    std::vector<uint32_t> ip2, is2, xp2, xs2;
    {   // window 2's own edges (no next window was resolved)
        ip2.assign(1, 0);
        for (size_t t = 2 * P; t < 3 * P; ++t)
        {
            for (uint32_t i = ptr[t]; i < ptr[t + 1]; ++i) is2.push_back((uint32_t) (succ[i] - 2 * P));
            ip2.push_back((uint32_t) is2.size());
        }
    }
    if (ip0 != ip1 || is0 != is1 || xp0 != xp1 || xs0 != xs1 || ip0 != ip2 || is0 != is2 ||
        !std::equal(npred.begin() + P, npred.begin() + 2 * P, npred.begin() + 2 * P))
        return xkb_set_error(XKB_EINVAL, "resolver_periodic: the windows do not repeat");
    // pack: succ_ptr | succ | xsucc_ptr | xsucc | npred_first | npred_next
    const size_t total = (P + 1) + is0.size() + (P + 1) + xs0.size() + P + P;
    int rc = R->periodic.reserve(total ? total : 1);
    if (rc) return rc;
    std::vector<uint32_t> h;
    h.reserve(total);
    h.insert(h.end(), ip0.begin(), ip0.end());
    h.insert(h.end(), is0.begin(), is0.end());
    h.insert(h.end(), xp0.begin(), xp0.end());
    h.insert(h.end(), xs0.begin(), xs0.end());
    h.insert(h.end(), npred.begin(), npred.begin() + P);
    h.insert(h.end(), npred.begin() + P, npred.begin() + 2 * P);
    XKB_CUDA_TRY(cudaMemcpy(R->periodic.p, h.data(), h.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    const uint32_t * d = R->periodic.p;
    out->period = P;
    out->succ_ptr = d; d += P + 1;
    out->succ = d; d += is0.size();
    out->xsucc_ptr = d; d += P + 1;
    out->xsucc = d; d += xs0.size();
    out->npred_first = d; d += P;
    out->npred_next = d;
    return XKB_OK;
}
