// Heat-diffusion-2d kernels: per-task tile launch (the plain form, one launch per tile task)
// and the whole-step launch (all tile tasks of one step fused into one grid).
#include "heat.cuh"

namespace xkb {

constexpr int HEAT_THREADS = 256;   // 8 warps per CTA

constexpr int HEAT_VEC = 4;         // rows per lane of the box kernel: a warp strip is 128 rows
constexpr int BOX_COLS_F64 = 48, BOX_COLS_F32 = 96;   // columns of a strip of a large box
constexpr int BOX_PFD_F64 = 3, BOX_PFD_F32 = 6;       // its L2 prefetch distance in columns
constexpr int HEAT_NARROW = 16;     // columns of a strip up to which all of them are loaded 4 ahead, without L2 prefetch

// The cells of a box (a tile, or the whole interior), split into strips of 128 rows x `cols` columns,
// one warp each, consecutive warps down a column chunk so that the warps in flight read and write
// whole columns (across the columns of a row of strips instead: 16384^2 FP64 701 us against 662). The
// strips are the tile bodies' of the persistent scheduler (heat.cuh): four rows per lane, twice the
// bytes per request of the two-row overlapping strips of heat_step_kernel, which this replaces as
// the default. A step, us: 16384^2 FP64 762 -> 651 (6.6 TB/s), 8192^2 197 -> 172, 8192^2 FP32
// 118 -> 113, 1024^2 FP64 29 -> 6, 5003 x 4001 (odd ld) FP32 78 -> 47, FP64 106 -> 62.
template <typename T, int PF, Strips K>
__global__ void __launch_bounds__(HEAT_THREADS, 2)
heat_box_kernel(const T * __restrict__ src, T * __restrict__ dst, int64_t ld, int64_t nx, int64_t ny, TileBox b,
                int64_t rbase0, int nrg, int ncg, int cols, double c, int pfd)
{
    const int s = (int) blockIdx.x * (HEAT_THREADS / 32) + (int) (threadIdx.x >> 5);
    if (s < nrg * ncg)
    {
        const int cg = (int) ((uint32_t) s / (uint32_t) nrg), rg = s - cg * nrg;
        const int64_t cy0 = b.cy0 + (int64_t) cg * cols, rbase = rbase0 + (int64_t) rg * 32 * HEAT_VEC;
        int64_t cy1 = cy0 + cols; if (cy1 > b.cy1) cy1 = b.cy1;
        if constexpr (K == Strips::ROWS)
            heat_strip_rows<T, HEAT_VEC, PF, false>(src, dst, ld, nx, rbase, b.rx0, b.rx1, cy0, cy1, c);
        else if (rbase + 32 * HEAT_VEC <= nx || nx % HEAT_VEC == 0 || cy1 < ny - 1)
            heat_strip_halo_impl<T, HEAT_VEC, PF, false>(src, dst, ld, nx, rbase, b.rx0, b.rx1, cy0, cy1, c, pfd);
        else
            heat_strip_rows_call<T, HEAT_VEC, false>(src, dst, ld, nx, rbase, b.rx0, b.rx1, cy0, cy1, c);
    }
}

template <typename T, int VEC, int PF, int MINB>
__global__ void __launch_bounds__(HEAT_THREADS, MINB)
heat_step_kernel(const T * __restrict__ src, T * __restrict__ dst, int64_t ld, int64_t nx, int64_t ny,
                 int64_t nrg, int64_t ncc, int64_t cols, double c, bool vec_ok, int pfd)
{
    const int64_t warps = (int64_t) gridDim.x * (HEAT_THREADS / 32);
    const int64_t nstrips = nrg * ncc;
    for (int64_t s = (int64_t) blockIdx.x * (HEAT_THREADS / 32) + (threadIdx.x >> 5); s < nstrips; s += warps)
    {
        // consecutive warps take consecutive row groups of the same column chunk, so a CTA
        // sweeps a contiguous panel of the grid
        const int64_t rg = s % nrg, cc = s / nrg;
        const int64_t cy0 = 1 + cc * cols;
        int64_t cy1 = cy0 + cols; if (cy1 > ny - 1) cy1 = ny - 1;
        heat_strip<T, VEC, PF, false>(src, dst, ld, nx, ny, rg * StripGeom<VEC>::OUT, 1, nx - 1, cy0, cy1, c, vec_ok, pfd);
    }
}

template <typename T>
static bool vec_ok_for(const void * src, const void * dst, int64_t ld)
{
    constexpr int VEC = HeatVec<T>::N;
    return (ld % VEC == 0) && ((uintptr_t) src % 16 == 0) && ((uintptr_t) dst % 16 == 0);
}

static int sm_count()
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    }
    return sms;
}

// Launch the box kernel, a CTA per 8 strips (CTAs are handed out as others end: with the strips dealt
// to resident warps in advance the slowest warp made 16384^2 FP64 767 us). Strips of about BOX_COLS
// columns, their number rounded to whole waves of the device's warps; a box of less than a wave gets a
// strip per warp, of 4 columns at least. (FP64 strips of 32 / 48 / 64 / 96 / 128 columns: 649 / 651 /
// 654 / 659 / 767 us at 16384^2, 170 / 172 / 178 / 189 / 204 at 8192^2; FP32 strips of 32 / 64 / 96:
// 119 / 114 / 113 at 8192^2.)
template <typename T>
static int launch_box(const void * src, void * dst, int64_t ld, int64_t nx, int64_t ny, const TileBox & b, double c, cudaStream_t st)
{
    if (b.rx0 >= b.rx1 || b.cy0 >= b.cy1) return XKB_OK;
    const int64_t rbase0 = b.rx0 - b.rx0 % HEAT_VEC, width = b.cy1 - b.cy0, warps = (int64_t) sm_count() * 2 * (HEAT_THREADS / 32);
    const int64_t nrg = (b.rx1 - rbase0 + 32 * HEAT_VEC - 1) / (32 * HEAT_VEC);
    const int64_t target = sizeof(T) == 8 && vec_ok_for<T>(src, dst, ld) ? BOX_COLS_F64 : BOX_COLS_F32;
    const int64_t waves = std::max<int64_t>(1, (nrg * width + target / 2 * warps) / (target * warps));
    int64_t ncg = std::max<int64_t>(1, waves * warps / nrg);
    const int64_t cols = std::max<int64_t>(4, (width + ncg - 1) / ncg);
    ncg = (width + cols - 1) / cols;
    if (nrg > INT32_MAX / ncg - 8 || cols > INT32_MAX) return xkb_set_error(XKB_EINVAL, "heat: grid too large");
    const unsigned grid = (unsigned) ((nrg * ncg + HEAT_THREADS / 32 - 1) / (HEAT_THREADS / 32));
    auto run = [&](auto kernel, int pfd) {
        kernel<<<grid, HEAT_THREADS, 0, st>>>((const T *) src, (T *) dst, ld, nx, ny, b, rbase0, (int) nrg, (int) ncg, (int) cols, c, pfd);
    };
    if (!vec_ok_for<T>(src, dst, ld)) run(heat_box_kernel<T, ROWS_PF<T>, Strips::ROWS>, 0);
    else if (cols <= HEAT_NARROW) run(heat_box_kernel<T, 4, Strips::VECTOR>, 0);
    else run(heat_box_kernel<T, sizeof(T) == 8 ? 2 : 5, Strips::VECTOR>, sizeof(T) == 8 ? BOX_PFD_F64 : BOX_PFD_F32);
    XKB_CUDA_TRY(cudaGetLastError());
    return XKB_OK;
}

template <typename T, int PF, int MINB>
static void step_launch(dim3 g, cudaStream_t st, const void * src, void * dst, int64_t ld, int64_t nx, int64_t ny,
                        int64_t nrg, int64_t ncc, int64_t cols, double c, bool vok, int pfd)
{
    heat_step_kernel<T, HeatVec<T>::N, PF, MINB><<<g, HEAT_THREADS, 0, st>>>((const T *) src, (T *) dst, ld, nx, ny,
                                                                          nrg, ncc, cols, c, vok, pfd);
}

template <typename T>
static int launch_step(const void * src, void * dst, int64_t ld, int64_t nx, int64_t ny, double c,
                       const xkb_heat_cfg_t & cfg, cudaStream_t st)
{
    constexpr int VEC = HeatVec<T>::N;
    if (nx < 3 || ny < 3) return XKB_OK;
    const int64_t cols = cfg.cols_per_strip > 0 ? cfg.cols_per_strip : 64;
    const int64_t nrg = (nx - 2 + StripGeom<VEC>::OUT - 1) / StripGeom<VEC>::OUT;
    const int64_t ncc = (ny - 2 + cols - 1) / cols;
    const int64_t ctas_needed = (nrg * ncc + (HEAT_THREADS / 32) - 1) / (HEAT_THREADS / 32);
    int64_t grid = (int64_t) sm_count() * (cfg.ctas_per_sm > 0 ? cfg.ctas_per_sm : 8);
    if (grid > ctas_needed) grid = ctas_needed;
    const bool vok = vec_ok_for<T>(src, dst, ld);
    const dim3 g((unsigned) grid);
    const int pfd = cfg.l2_prefetch_cols;
    switch (cfg.pf * 10 + cfg.min_blocks)
    {
        case 21: step_launch<T, 2, 1>(g, st, src, dst, ld, nx, ny, nrg, ncc, cols, c, vok, pfd); break;
        case 22: step_launch<T, 2, 2>(g, st, src, dst, ld, nx, ny, nrg, ncc, cols, c, vok, pfd); break;
        case 24: step_launch<T, 2, 4>(g, st, src, dst, ld, nx, ny, nrg, ncc, cols, c, vok, pfd); break;
        case 41: step_launch<T, 4, 1>(g, st, src, dst, ld, nx, ny, nrg, ncc, cols, c, vok, pfd); break;
        case 42: step_launch<T, 4, 2>(g, st, src, dst, ld, nx, ny, nrg, ncc, cols, c, vok, pfd); break;
        case 81: step_launch<T, 8, 1>(g, st, src, dst, ld, nx, ny, nrg, ncc, cols, c, vok, pfd); break;
        case 82: step_launch<T, 8, 2>(g, st, src, dst, ld, nx, ny, nrg, ncc, cols, c, vok, pfd); break;
        default: return xkb_set_error(XKB_EINVAL, "heat_step: unsupported (pf=%d, min_blocks=%d)", cfg.pf, cfg.min_blocks);
    }
    XKB_CUDA_TRY(cudaGetLastError());
    return XKB_OK;
}

} // namespace xkb

using namespace xkb;

static int heat_check(int dtype, const void * src, const void * dst, int64_t ld, int64_t nx, int64_t ny)
{
    if (dtype != XKB_F64 && dtype != XKB_F32) return xkb_set_error(XKB_EINVAL, "heat: dtype must be XKB_F64 or XKB_F32");
    if (!src || !dst || src == dst) return xkb_set_error(XKB_EINVAL, "heat: src and dst must be distinct device grids");
    if (nx < 0 || ny < 0 || ld < nx) return xkb_set_error(XKB_EINVAL, "heat: need 0 <= nx <= ld and ny >= 0");
    return XKB_OK;
}

extern "C" int xkb_heat_tile(int dtype, const void * src, void * dst, int64_t ld, int64_t nx, int64_t ny,
                             int64_t tile_x, int64_t tile_y, int64_t tsx, int64_t tsy, double c, void * stream)
{
    int rc = heat_check(dtype, src, dst, ld, nx, ny);
    if (rc) return rc;
    if (tsx <= 0 || tsy <= 0 || tile_x < 0 || tile_y < 0) return xkb_set_error(XKB_EINVAL, "heat_tile: bad tile");
    const int64_t x0 = tile_x * tsx, y0 = tile_y * tsy;
    const int64_t x1 = x0 + tsx, y1 = y0 + tsy;
    const TileBox b = heat_tile_box(nx, ny, x0, x1, y0, y1);
    return dtype == XKB_F64 ? launch_box<double>(src, dst, ld, nx, ny, b, c, xkb_stream(stream))
                            : launch_box<float>(src, dst, ld, nx, ny, b, c, xkb_stream(stream));
}

extern "C" int xkb_heat_step(int dtype, const void * src, void * dst, int64_t ld, int64_t nx, int64_t ny,
                             double c, void * stream)
{
    return xkb_heat_step_cfg(dtype, src, dst, ld, nx, ny, c, nullptr, stream);
}

extern "C" int xkb_heat_step_cfg(int dtype, const void * src, void * dst, int64_t ld, int64_t nx, int64_t ny,
                                 double c, const xkb_heat_cfg_t * cfg, void * stream)
{
    int rc = heat_check(dtype, src, dst, ld, nx, ny);
    if (rc) return rc;
    if (!cfg)
    {
        const TileBox b = heat_tile_box(nx, ny, 0, nx, 0, ny);
        return dtype == XKB_F64 ? launch_box<double>(src, dst, ld, nx, ny, b, c, xkb_stream(stream))
                                : launch_box<float>(src, dst, ld, nx, ny, b, c, xkb_stream(stream));
    }
    const xkb_heat_cfg_t & k = *cfg;
    if (k.l2_prefetch_cols < 0 || k.l2_prefetch_cols > 256 || k.cols_per_strip < 0)
        return xkb_set_error(XKB_EINVAL, "heat_step: bad configuration");
    return dtype == XKB_F64 ? launch_step<double>(src, dst, ld, nx, ny, c, k, xkb_stream(stream))
                            : launch_step<float>(src, dst, ld, nx, ny, c, k, xkb_stream(stream));
}

// ---- FP64 checks of a step's result ---------------------------------------------------------
namespace {

// Non-negative doubles order like their bit patterns, so an integer max is a double max.
__device__ __forceinline__ void atomic_max_nonneg(double * p, double v)
{
    atomicMax((unsigned long long *) p, (unsigned long long) __double_as_longlong(v));
}

// out[0] max |dst| on the boundary, out[1] sum of dst^2 over the interior, out[2] max over the
// interior of |dst - (src + c*lap(src))| with src promoted to double, out[3] max |dst| interior.
// One block per column band; threads over rows; all arithmetic in double.
template <typename T>
__global__ void __launch_bounds__(256) heat_norms_kernel(const T * __restrict__ src, const T * __restrict__ dst, int64_t ld,
                                                         int64_t nx, int64_t ny, double c, double * out)
{
    double bmax = 0, sum = 0, rmax = 0, vmax = 0;
    for (int64_t j = blockIdx.x; j < ny; j += gridDim.x)
        for (int64_t i = threadIdx.x; i < nx; i += blockDim.x)
        {
            const double d = (double) dst[j * ld + i];
            if (i == 0 || j == 0 || i == nx - 1 || j == ny - 1) { bmax = fmax(bmax, fabs(d)); continue; }
            const T * s = src + j * ld + i;
            const double v = (double) s[0];
            const double a = __dadd_rn(__dsub_rn((double) s[1], __dmul_rn(2.0, v)), (double) s[-1]);
            const double b = __dadd_rn(__dsub_rn((double) s[ld], __dmul_rn(2.0, v)), (double) s[-ld]);
            const double e = __dadd_rn(v, __dmul_rn(c, __dadd_rn(a, b)));
            rmax = fmax(rmax, fabs(d - e));
            vmax = fmax(vmax, fabs(d));
            sum += d * d;
        }
    for (int o = 16; o > 0; o >>= 1)
    {
        bmax = fmax(bmax, __shfl_xor_sync(0xffffffffu, bmax, o));
        rmax = fmax(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
        vmax = fmax(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
    }
    if ((threadIdx.x & 31) == 0)
    {
        atomic_max_nonneg(out + 0, bmax);
        atomicAdd(out + 1, sum);
        atomic_max_nonneg(out + 2, rmax);
        atomic_max_nonneg(out + 3, vmax);
    }
}

} // namespace

extern "C" int xkb_heat_norms(int dtype, const void * src, const void * dst, int64_t ld, int64_t nx, int64_t ny, double c,
                              double * out, void * stream)
{
    int rc = heat_check(dtype, src, dst, ld, nx, ny);
    if (rc) return rc;
    if (!out) return xkb_set_error(XKB_EINVAL, "heat_norms: null output");
    cudaStream_t st = xkb_stream(stream);
    XKB_CUDA_TRY(cudaMemsetAsync(out, 0, 4 * sizeof(double), st));
    if (nx == 0 || ny == 0) return XKB_OK;
    int dev = 0, sms = 148;
    XKB_CUDA_TRY(cudaGetDevice(&dev));
    XKB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const unsigned grid = (unsigned) std::min<int64_t>(ny, (int64_t) sms * 8);
    if (dtype == XKB_F64) heat_norms_kernel<double><<<grid, 256, 0, st>>>((const double *) src, (const double *) dst, ld, nx, ny, c, out);
    else heat_norms_kernel<float><<<grid, 256, 0, st>>>((const float *) src, (const float *) dst, ld, nx, ny, c, out);
    XKB_CUDA_TRY(cudaGetLastError());
    return XKB_OK;
}
