// Auxiliary kernels: state transposes between the host dump order and the
// device SoA storage, deterministic statistics partial sums, conserved
// moments.  Templated on arithmetic type T and storage type S like the step.
#pragma once
#include "dugks_kernels.cuh"
#include "fixed_kernels.cuh"

namespace dg {

// dump order f[((k*ny+j)*nx+i)*19+p] (double)  ->  SoA storage
template <class T, class S>
__global__ void __launch_bounds__(256) aos_to_soa_kernel(const double *__restrict__ src, S *__restrict__ dst,
                                                         const StepParams<T, S> P)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    if (i >= P.nx) return;
    const size_t cell = ((size_t)k * P.ny + j) * P.nx + i;
    const long long c = ((long long)k * P.ny + j) * P.pitch + i;
#pragma unroll
    for (int p = 0; p < NPOP; ++p) P.codec.store(dst, p * P.ps + c, p, T(src[cell * NPOP + p]));
}

// SoA storage -> dump order (double)
template <class T, class S>
__global__ void __launch_bounds__(256) soa_to_aos_kernel(const S *__restrict__ src, double *__restrict__ dst,
                                                         const StepParams<T, S> P)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    if (i >= P.nx) return;
    const size_t cell = ((size_t)k * P.ny + j) * P.nx + i;
    const long long c = ((long long)k * P.ny + j) * P.pitch + i;
#pragma unroll
    for (int p = 0; p < NPOP; ++p) dst[cell * NPOP + p] = double(P.codec.load_nc(src, p * P.ps + c, p));
}

// Number of FP64 partial sums per x index written by stats_partials_kernel:
//  0 rho, 1 u, 2 v, 3 w, 4 uw, 5 uv, 6 vw, 7 uu, 8 vv, 9 ww,
//  10..13 min rho,u,v,w, 14..17 max rho,u,v,w, 18 non-finite count
constexpr int NSTAT = 19;

// Density and output velocity of a cell in FP64 (src/output.cu:223-260 on the
// arrays of src/dugks.cu:1021-1064)
__device__ __forceinline__ void stats_cell(const double v[NPOP], const double shift[3], double q[4])
{
    double r, jx, jy, jz;
    moments(v, r, jx, jy, jz);
    q[0] = r;
    q[1] = jx / r + shift[0];
    q[2] = jy / r + shift[1];
    q[3] = jz / r + shift[2];
}

__device__ __forceinline__ void stats_init(double acc[NSTAT])
{
#pragma unroll
    for (int s = 0; s < NSTAT; ++s) acc[s] = s < 10 || s == 18 ? 0.0 : (s < 14 ? 1e300 : -1e300);
}
__device__ __forceinline__ void stats_add(double acc[NSTAT], const double q[4])
{
    const double r = q[0], u = q[1], vv = q[2], w = q[3];
    acc[0] += r; acc[1] += u; acc[2] += vv; acc[3] += w;
    acc[4] += u * w; acc[5] += u * vv; acc[6] += vv * w;
    acc[7] += u * u; acc[8] += vv * vv; acc[9] += w * w;
}
__device__ __forceinline__ void stats_extremes(double acc[NSTAT], const double q[4])
{
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        acc[10 + a] = fmin(acc[10 + a], q[a]);
        acc[14 + a] = fmax(acc[14 + a], q[a]);
    }
    if (!isfinite(q[0]) || !isfinite(q[1]) || !isfinite(q[2]) || !isfinite(q[3])) acc[18] += 1.0;
}

// Block (b, by) sums rows (j,k) = b, b+gridDim.x, ... ; thread owns x index
// i = by*blockDim.x + threadIdx.x.  Output partial[b][NSTAT][i].  The fixed assignment and
// the ordered second pass make the result independent of scheduling.
template <class T, class S>
__global__ void __launch_bounds__(1024) stats_partials_kernel(const S *__restrict__ f, const StepParams<T, S> P,
                                                              double hdt, double fxa, double fya, double fza,
                                                              double *__restrict__ partial)
{
    const int i = blockIdx.y * blockDim.x + threadIdx.x;
    if (i >= P.nx) return;
    const double shift[3] = {fxa * hdt, fya * hdt, fza * hdt};
    double acc[NSTAT];
    stats_init(acc);
    const int rows = P.ny * P.nz;
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {
        const long long c = (long long)row * P.pitch + i;
        double v[NPOP], q[4];
#pragma unroll
        for (int p = 0; p < NPOP; ++p) v[p] = double(P.codec.load_nc(f, p * P.ps + c, p));
        stats_cell(v, shift, q);
        stats_add(acc, q);
        stats_extremes(acc, q);
    }
    double *out = partial + (size_t)blockIdx.x * NSTAT * P.nx + i;
#pragma unroll
    for (int s = 0; s < NSTAT; ++s) out[(size_t)s * P.nx] = acc[s];
}

// The same with density and velocity of a cell in fixed point (fixed.cuh) where its
// values are in the range of fixed_kernels.cuh, and its extremes as integers: 11
// FP64 instructions per cell (the density's conversion, ten sums), one more per axis with a
// force, instead of about 130, most of them the three divisions.  The moments are exact; a
// velocity is their quotient formed at a scale of its own and rounded once to FP64 (relative
// error below 2^-52 at any size, no bias).  Other cells take stats_cell.  Both sums of
// products and the reduction stay in FP64.  dg_stats_values of 256 x 128 x 128 FP64 cells: 174
// us, against 1654 us with FP64 cells and one chain; the reads alone take 95 us.  Bound by
// latency at 16 warps per SM (99 registers; 24 warps, at 80, 185 us).  210 us with the
// velocities' conversions and the test for a force as FP64 instructions.
// one stored value, scaled 2^62 (FP64) or 2^30 (float values of 2^-7 and more are
// multiples of 2^-30: their moments fit 32-bit integers exactly)
__device__ __forceinline__ i64 stats_int(double x) { return fx_from_double(x); }
__device__ __forceinline__ int stats_int(float x)
{
    const unsigned b = __float_as_uint(x);
    return int(((b & 0x7fffffu) | 0x800000u) << ((b >> 23) - 120));
}
__device__ __forceinline__ bool stats_bad(double x, int p) { return fx_bad_double(x, p); }
__device__ __forceinline__ bool stats_bad(float x, int p)
{
    const double w = weight<double>(p);
    const unsigned lo = __float_as_uint(float(w * FX_LO)) + 1, hi = __float_as_uint(float(w * FX_HI));
    return __float_as_uint(x) - lo >= hi - lo;
}

// The FP64 value nearest to v / 2^s, |v| < 2^63, in integer operations
__device__ __forceinline__ double fx_pack(i64 v, int s)
{
    const u64 m = v < 0 ? -v : v;
    const int c = __clzll(m);
    const u64 t = m << (c & 63);
    const u64 b = (t >> 11) + ((t >> 10) & 1) + (u64(1023 + 62 - c - s) << 52);  // the leading one adds 1 to the exponent
    return __longlong_as_double(m ? i64(b) | (v & (1ll << 63)) : 0);
}

// FP64 numbers as integers that compare alike, and back
__device__ __forceinline__ i64 stats_key(double x)
{
    const i64 b = __double_as_longlong(x);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double stats_unkey(i64 k) { return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll)); }

template <class T, class S>
__global__ void __launch_bounds__(256) stats_fx_kernel(const S *__restrict__ f, const StepParams<T, S> P,
                                                       double sx, double sy, double sz, double *__restrict__ partial)
{
    using I = decltype(stats_int(T(0)));
    const int i = blockIdx.y * blockDim.x + threadIdx.x;
    if (i >= P.nx) return;
    const FxMul third = fx_split(0x5555555555555555ll);
    double acc[NSTAT];
    stats_init(acc);
    const double shift[3] = {sx, sy, sz};
    // compared as integers: the compiler would compare the doubles in every cell
    const bool forced[3] = {__double_as_longlong(sx) != 0, __double_as_longlong(sy) != 0, __double_as_longlong(sz) != 0};
    i64 lo[4], hi[4], key[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) lo[a] = 0x7fffffffffffffffll, hi[a] = -0x7fffffffffffffffll;
    const int rows = P.ny * P.nz;
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {
        const long long c = (long long)row * P.pitch + i;
        T v[NPOP];
        bool bad = false;
#pragma unroll
        for (int p = 0; p < NPOP; ++p) {
            v[p] = P.codec.load_nc(f, p * P.ps + c, p);
            bad |= stats_bad(v[p], p);
        }
        double q[4];
        if (!bad) {
            I r = 0, j[3] = {0, 0, 0};
#pragma unroll
            for (int p = 0; p < NPOP; ++p) {
                const I x = stats_int(v[p]);
                r += x;
#pragma unroll
                for (int a = 0; a < 3; ++a)
                    if (cc(a, p)) j[a] += cc(a, p) > 0 ? x : -x;
            }
            constexpr int up = sizeof(I) == 8 ? 0 : 32;
            const i64 rho = i64(r) << up;
            const FxMul M3 = fx_recip3(rho);  // 3 / (16 rho)
            const FxMul M = fx_split(fx_mul(i64(M3.h) * (1ll << 32) + M3.l, third));
            q[0] = fx_to_double(rho, 62);
            key[0] = rho;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const i64 ja = i64(j[a]) << up;
                const int n = __clzll(ja < 0 ? -ja : ja) - 2;  // |j| < 2^61: shifted to 2^61 .. 2^62
                q[a + 1] = fx_pack(fx_madr(ja << n, M, 0), 58 + n);
                if (forced[a]) q[a + 1] += shift[a];
                key[a + 1] = stats_key(q[a + 1]);
            }
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                lo[a] = min(lo[a], key[a]);
                hi[a] = max(hi[a], key[a]);
            }
        } else {
            double d[NPOP];
#pragma unroll
            for (int p = 0; p < NPOP; ++p) d[p] = double(v[p]);
            stats_cell(d, shift, q);
            stats_extremes(acc, q);
        }
        stats_add(acc, q);
    }
    if (lo[0] <= hi[0]) {
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            acc[10 + a] = fmin(acc[10 + a], a ? stats_unkey(lo[a]) : fx_to_double(lo[a], 62));
            acc[14 + a] = fmax(acc[14 + a], a ? stats_unkey(hi[a]) : fx_to_double(hi[a], 62));
        }
    }
    double *out = partial + (size_t)blockIdx.x * NSTAT * P.nx + i;
#pragma unroll
    for (int s = 0; s < NSTAT; ++s) out[(size_t)s * P.nx] = acc[s];
}

// Ordered reduction over blocks of the statistics partials of x index i:
// sum / min / max over b0 <= b < b1 of partial[b][s][i] (b ascending).  Shared by
// stats_reduce_kernel, over one chain or several (launch_stats_reduce), and the
// allocation-free statistics, over one.
__device__ __forceinline__ double stats_combine(const double *__restrict__ partial, int b0, int b1, int nx, int i, int s)
{
    const double *q = partial + size_t(s) * nx + i;
    const size_t step = size_t(nx) * NSTAT;
    double acc = q[b0 * step];
    if (s < 10 || s == 18) {
#pragma unroll 16
        for (int b = b0 + 1; b < b1; ++b) acc += q[b * step];
    } else if (s < 14) {
#pragma unroll 16
        for (int b = b0 + 1; b < b1; ++b) acc = fmin(acc, q[b * step]);
    } else {
#pragma unroll 16
        for (int b = b0 + 1; b < b1; ++b) acc = fmax(acc, q[b * step]);
    }
    return acc;
}
__device__ __forceinline__ void stats_combine_blocks(const double *__restrict__ partial, int nblocks, int nx, int i,
                                                     double acc[NSTAT])
{
    for (int s = 0; s < NSTAT; ++s) acc[s] = stats_combine(partial, 0, nblocks, nx, i, s);
}

// Ordered reduction over blocks: total[i][s] = sum/min/max over b of partial[b][s][i].
// A warp holds 32 x indices of one sum s (blockIdx.y); the warps of a CTA (blockDim.y)
// take consecutive ranges of blocks, combined in order.
constexpr int kStatsWarps = 16;
__global__ void stats_reduce_kernel(const double *__restrict__ partial, int nblocks, int nx, double *__restrict__ total);
// acc[i][s] += total[i][s] for the 10 sums
__global__ void stats_accumulate_kernel(const double *__restrict__ total, int nx, double *__restrict__ acc);

// Conserved moments: block partial sums of (rho, jx, jy, jz) over cells; a
// fixed assignment of cells to threads and a fixed-order tree make the sums
// reproducible.
// Warp-shuffle sum of a double over the 32 lanes (fixed order: deterministic).
__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Mass and momentum partial sums, one per block (deterministic order).  Every
// thread takes cells t, t + gridDim.x*blockDim.x, ... of the interior in x-fastest
// order (coalesced).  FP64 form: one FP64 sum per population over the thread's
// cells, combined into (rho, j) at the end: 19 additions per cell instead of
// the per-cell moments (46) plus four accumulations, on GB300's reduced-rate
// FP64 pipe.  Other forms: moments per cell in the arithmetic type, summed over
// cells in FP64.  Warps reduce with shuffles, warp 0 combines the warps.
template <class T, class S>
__global__ void __launch_bounds__(256) moments_partials_kernel(const S *__restrict__ f, const StepParams<T, S> P,
                                                               double *__restrict__ partial)
{
    __shared__ double red[8][4];
    double a[4] = {0, 0, 0, 0};
    const long long ncell = (long long)P.nx * P.ny * P.nz;
    const long long stride = (long long)gridDim.x * blockDim.x;
    if (sizeof(T) == 8) {
        double sp[NPOP];
#pragma unroll
        for (int p = 0; p < NPOP; ++p) sp[p] = 0.0;
        for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < ncell; t += stride) {
            const long long row = t / P.nx;
            const long long c = row * P.pitch + (t - row * P.nx);
#pragma unroll
            for (int p = 0; p < NPOP; ++p) sp[p] += double(P.codec.load_nc(f, p * P.ps + c, p));
        }
#pragma unroll
        for (int p = 0; p < NPOP; ++p) {
            a[0] += sp[p];
            if (cx(p)) a[1] += cx(p) > 0 ? sp[p] : -sp[p];
            if (cy(p)) a[2] += cy(p) > 0 ? sp[p] : -sp[p];
            if (cz(p)) a[3] += cz(p) > 0 ? sp[p] : -sp[p];
        }
    } else {
        for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < ncell; t += stride) {
            const long long row = t / P.nx;
            const long long c = row * P.pitch + (t - row * P.nx);
            T v[NPOP];
#pragma unroll
            for (int p = 0; p < NPOP; ++p) v[p] = P.codec.load_nc(f, p * P.ps + c, p);
            T r, jx, jy, jz;
            moments(v, r, jx, jy, jz);
            a[0] += double(r); a[1] += double(jx); a[2] += double(jy); a[3] += double(jz);
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const double s = warp_sum(a[m]);
        if (lane == 0) red[warp][m] = s;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const double s = warp_sum(lane < 8 ? red[lane][m] : 0.0);
            if (lane == 0) partial[blockIdx.x * 4 + m] = s;
        }
    }
}

}  // namespace dg
