// axpby tile body as its own launch: y = a*x + b*y over FP64 vectors.
#include "common.cuh"

#include <type_traits>

namespace xkb {

__device__ __forceinline__ double axpby1(double a, double x, double b, double y)
{
    return __dadd_rn(__dmul_rn(a, x), __dmul_rn(b, y));   // (a*x) + (b*y), no FMA
}

// One CTA per AXPBY_CTA elements, handed out as others end (a fixed grid that strides through the
// vectors with one of each operand in flight per thread: 10^8 elements 393 us against 345, 6.95 TB/s;
// 2 or 8 vectors per thread instead of 4: within 1 %). A thread loads its share of both operands
// before it uses any. VECTOR: the operands are 16-byte aligned together from element `head` on, and
// go two elements at a time; `head` (at most one) element before and an odd one at the end go alone.
// Else they go one at a time, which costs nothing but the instructions (355 us at the same length, 546 before).
constexpr int AXPBY_THREADS = 256, AXPBY_CTA = 8 * AXPBY_THREADS;

template <bool VECTOR>
__global__ void __launch_bounds__(AXPBY_THREADS) axpby_kernel(int64_t n, int64_t head, double a, const double * __restrict__ x,
                                                              double b, double * __restrict__ y)
{
    constexpr int PER = VECTOR ? 4 : 8;
    using V = typename std::conditional<VECTOR, double2, double>::type;
    const int64_t nv = VECTOR ? (n - head) / 2 : n, v0 = (int64_t) blockIdx.x * (AXPBY_THREADS * PER) + threadIdx.x;
    const V * xv = (const V *) (x + head);
    V * yv = (V *) (y + head);
    V xx[PER], yy[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k)
    {
        const int64_t v = v0 + k * AXPBY_THREADS;
        if (v < nv) { xx[k] = __ldcs(xv + v); yy[k] = __ldcs(yv + v); }
    }
#pragma unroll
    for (int k = 0; k < PER; ++k)
    {
        const int64_t v = v0 + k * AXPBY_THREADS;
        if (v >= nv) break;
        if constexpr (VECTOR) yv[v] = make_double2(axpby1(a, xx[k].x, b, yy[k].x), axpby1(a, xx[k].y, b, yy[k].y));
        else yv[v] = axpby1(a, xx[k], b, yy[k]);
    }
    if (VECTOR && blockIdx.x == 0 && threadIdx.x < 2)
    {
        const int64_t i = threadIdx.x == 0 ? 0 : n - 1;
        if (threadIdx.x == 0 ? head == 1 : head + 2 * nv < n) y[i] = axpby1(a, __ldg(x + i), b, y[i]);
    }
}

} // namespace xkb

extern "C" int xkb_axpby(int64_t n, double a, const double * x, double b, double * y, void * stream)
{
    if (n < 0 || (n > 0 && (!x || !y))) return xkb_set_error(XKB_EINVAL, "axpby: bad arguments");
    if (n == 0) return XKB_OK;
    const int64_t ctas = (n + xkb::AXPBY_CTA - 1) / xkb::AXPBY_CTA;
    if (ctas > INT32_MAX) return xkb_set_error(XKB_EINVAL, "axpby: vectors too long");
    const bool vector = ((uintptr_t) x & 15) == ((uintptr_t) y & 15);
    if (vector)
        xkb::axpby_kernel<true><<<(unsigned) ctas, xkb::AXPBY_THREADS, 0, xkb_stream(stream)>>>(n, ((uintptr_t) y & 15) ? 1 : 0, a, x, b, y);
    else
        xkb::axpby_kernel<false><<<(unsigned) ctas, xkb::AXPBY_THREADS, 0, xkb_stream(stream)>>>(n, 0, a, x, b, y);
    XKB_CUDA_TRY(cudaGetLastError());
    return XKB_OK;
}
