// The FP64 step in 64-bit fixed point (fixed.cuh): stage (a) and the flux / update
// kernel of dugks_kernels.cuh with every distribution value an integer scaled 2^62.
//
// What bounds the FP64 step is FP64 issue (2.1 lanes per SM and clock, 861
// instructions per cell), not memory; integer adds and products run on pipes that
// are 4 to 30 times wider (fixed.cuh).  f-tilde stays FP64 in memory; it is read
// exactly (its values have fewer bits than the fixed point) and rounded once when
// written.  f-bar-plus, written and read by these two kernels only, is held in
// fixed point.  Step of the 256 x 128 x 128 channel: 6.65 ms with the FP64 kernels,
// 1.22 ms here (stage (a) 0.21, flux 1.01); 64^3 box 0.63 -> 0.104 ms, 64 x 32 x 32
// channel 0.229 -> 0.037 ms.
//
// Error of the state against the double scheme in extended precision (the reference's double
// coefficients, no rounding of the arithmetic; relative 2-norm, channel and periodic box):
// 5e-17 after one step, the rounding of the stored values (FP64 kernels 1.7e-16 to 2.3e-16),
// 1.1e-16 after 100 (5.6e-15); tests/test_extended_oracle.py.  After 10^4 steps the state is
// within 1e-14 of the oracle in double (FP64 kernels 5.6e-13), mass included, which those
// coefficients let drift by 1.4e-16 a step in the channel; tests/test_gpu_fixed_long.py.
//
// Range.  The scaling is chosen for states near unit density: every f-tilde and
// f-bar-plus (wall ghosts included) within (FX_LO, FX_HI) w_p, which holds up to
// velocities of about 0.25.  Face values are convex combinations of f-bar-plus and
// stay in that box, which bounds density (0.4 .. 1.98), momentum (|j| < 0.27),
// 3 c_p.u (< 1.67, reached with the populations moving along c_p at the upper and
// the others at the lower end) and the equilibrium polynomial (< 3.9) at every cell
// and face, so that no sum or product overflows (the sums over the populations that do not
// cross a face reach 1.32, see fx_mean).  Stage (a) checks the box per value
// (NaN and infinities fail it) and raises a device flag; the flux kernel then does stage
// (a) again in FP64 and fp64_redo_kernel the rest of the step.  The parameters have to
// fit too (make_fixed_plan in engine.cu): a single force axis, interpolation weights
// within (0, 1/2), dt/dx below about 1/2.
#pragma once
#ifdef __CUDACC__
#include <cuda_runtime.h>
#endif

#include "d3q19.cuh"
#include "fixed.cuh"
#ifdef __CUDACC__
#include "dugks_kernels.cuh"
#endif

namespace dg {

constexpr double FX_LO = 0.4, FX_HI = 1.98;
constexpr i64 FX_ONE = 1ll << 62;

// Equilibrium coefficients of a cell (stage (a)) or a face:
//   K_p = w_p rho (B + c_p.Kf - Cf u), see fx_eq.
struct FxForce {
    i64 shift;   // 3 x velocity shift along the force axis, scaled 2^61
    i64 B;       // (coefficient of feq without force) / 18, scaled 2^64
    FxMul C;     // 3 u_a (scaled 2^61) -> its share of B (scaled 2^64)
    FxMul Kf;    // rho (2^62) -> force term of K of an axis population along +a, scaled 2^62
};

struct FxParams {
    int nx, ny, nz, pitch;  // f-tilde as in StepParams
    long long ps;
    int pitch_b, rs;        // f-bar-plus: columns per row (nx + 2 rounded up to 16), elements per row (19 pitch_b)
    int periodic_x;
    int esh;                // fluxes are held divided by fw1 2^esh, fw1 2^esh in (1/4, 1]
    int stretched;          // x-face weights of the c_x = 0 populations differ from 1/2
    int drift;              // sum f-bar-plus / rho - 1, scaled 2^78 (see fx_stage_a)
    FxForce cell, face;
    FxMul bw1;              // 2 f (2^63) -> bw1 f (2^62)
    FxMul third;            // 1/3
    FxMul ty, tz;           // transverse weights hdt/dy, hdt/dz
    FxMul my, mz;           // normal weight of the upwind-side cell, 1/2 - hdt/dy, 1/2 - hdt/dz
    FxMul cy, cz;           // fw1 2^esh dt/dy, dt/dz
    FxMul q0, q1;           // wall ghosts: extrapolation weight q, less 2
    const FxMul *tab;       // [FXT_ROWS][nx + 2] per column / x face
    const void *step;       // StepParams<double, double> on the device, for steps out of range
};
constexpr int FXT_TXP = 0;  // transverse x weight of c_x > 0 at column i
constexpr int FXT_TXM = 1;  // ... of c_x < 0
constexpr int FXT_MP = 2;   // x face I: weight of cell I+1 for c_x > 0
constexpr int FXT_MM = 3;   // ... of cell I for c_x < 0
constexpr int FXT_D0 = 4;   // ... of cell I+1 for c_x = 0, less 1/2
constexpr int FXT_CX = 5;   // column i: fw1 2^esh dt/dx
constexpr int FXT_ROWS = 6;

// f-bar-plus layout: row (k, j) of 0-based cells holds pitch_b columns in blocks of
// 16, the 19 populations of a block one after another: a population step is the
// constant 16 elements (an immediate of the load) and a warp's 32 cells are two
// 128-byte pieces.  Column c = 0 .. nx-1: cells; nx: the ghost past the upper
// wall (or image); nx + 1: the lower ghost.
DG_FX int fx_col(int c) { return (c >> 4) * (NPOP * 16) + (c & 15); }

// K_p coefficients, velocities and the equilibrium polynomial of a cell or face:
//   feq_p = w_p rho (1 + x + x^2/2 - 1.5 u.u), x = 3 c_p.u
struct FxEq {
    i64 u3[3];       // 3 u, scaled 2^61 (force shift included)
    i64 sq[3];       // (3 u_a)^2 / 2, scaled 2^61
    i64 base;        // 1 - 1.5 u.u, scaled 2^61
    FxMul K1[3], K2[3];  // K of axis / diagonal populations with c_a = 0, +1, -1 along the force axis, scaled 2^65
};

template <int FAX>
DG_FX FxEq fx_eq(i64 rho, const i64 j[3], const FxForce &c, FxMul third)
{
    FxEq E;
    const FxMul M = fx_recip3(rho);
DG_UNROLL
    for (int a = 0; a < 3; ++a) {
        E.u3[a] = fx_mul(j[a] << 2, M) << 1;  // 4 j (2^62) x 3 / (16 rho) = 3 u 2^60
        if (a == FAX) E.u3[a] += c.shift;
        E.sq[a] = fx_sq(E.u3[a] << 1);
    }
    E.base = (1ll << 61) - fx_mul(E.sq[0] + E.sq[1] + E.sq[2], third);
    if (FAX < 3) {
        const i64 k = fx_mul(rho, fx_split(c.B - fx_mul(E.u3[FAX < 3 ? FAX : 0], c.C)));
        const i64 d = fx_mul(rho, c.Kf);
        E.K1[0] = fx_split(k << 3), E.K1[1] = fx_split((k + d) << 3), E.K1[2] = fx_split((k - d) << 3);
        E.K2[0] = fx_split(k << 2), E.K2[1] = fx_split((k + d) << 2), E.K2[2] = fx_split((k - d) << 2);
    } else {
        const i64 k = fx_mul(rho, fx_split(c.B));
        E.K1[0] = E.K1[1] = E.K1[2] = fx_split(k << 3);
        E.K2[0] = E.K2[1] = E.K2[2] = fx_split(k << 2);
    }
    return E;
}

// acc_p += K_p (polynomial at +-x) for the opposite pair (p, opp(p))
template <int FAX>
DG_FX void fx_pair(const FxEq &E, int p, i64 &accp, i64 &accq)
{
    const int ax = cx(p), ay = cy(p), az = cz(p);
    i64 x = 0;
    if (ax) x += ax > 0 ? E.u3[0] : -E.u3[0];
    if (ay) x += ay > 0 ? E.u3[1] : -E.u3[1];
    if (az) x += az > 0 ? E.u3[2] : -E.u3[2];
    const i64 t = E.base + (p <= 6 ? (ax ? E.sq[0] : (ay ? E.sq[1] : E.sq[2])) : fx_sq(x << 1));
    const int ca = FAX < 3 ? cc(FAX, p) : 0;
    const int sp = ca == 0 ? 0 : (ca > 0 ? 1 : 2), sq = ca == 0 ? 0 : (ca > 0 ? 2 : 1);
    accp = fx_mad(t + x, p <= 6 ? E.K1[sp] : E.K2[sp], accp);
    accq = fx_mad(t - x, p <= 6 ? E.K1[sq] : E.K2[sq], accq);
}

// Density and momentum of 19 values.
DG_FX void fx_moments(const i64 v[NPOP], i64 &r, i64 j[3])
{
    r = v[0];
    j[0] = j[1] = j[2] = 0;
DG_UNROLL
    for (int p = 1; p < NPOP; ++p) {
        r += v[p];
DG_UNROLL
        for (int a = 0; a < 3; ++a)
            if (cc(a, p)) j[a] += cc(a, p) > 0 ? v[p] : -v[p];
    }
}

// f-bar-plus of one cell from f-tilde: bw1 f + K feq-polynomial; the rest
// population from the density: the sum of f-bar-plus is rho (1 + drift).  The scheme
// conserves mass (drift 0), but its coefficients as doubles (weights, bw1, bw2) miss their
// sums by about 1e-16, which is 1.4e-12 of the mass after 10^4 steps, and the parity of this
// form is with the reference's step, which has these doubles (make_fixed_plan in engine.cu).
template <int FAX>
DG_FX void fx_stage_a(const FxParams &P, const i64 v[NPOP], i64 ob[NPOP])
{
    i64 rho, j[3];
    fx_moments(v, rho, j);
    const FxEq E = fx_eq<FAX>(rho, j, P.cell, P.third);
    i64 rest = rho + (fx_wide(int(rho >> 32), P.drift, 1ll << 45) >> 46);
DG_UNROLL
    for (int p = 1; p < NPOP; ++p) {
        const int q = opp(p);
        if (q < p) continue;
        ob[p] = fx_mul(v[p] << 1, P.bw1);
        ob[q] = fx_mul(v[q] << 1, P.bw1);
        fx_pair<FAX>(E, p, ob[p], ob[q]);
        rest -= ob[p] + ob[q];
    }
    ob[0] = rest;
}

// Face fluxes divided by fw1 2^esh, in place: v holds the 10 face values that
// cross the face (flux_pop order), m the sums over the other 9 of their values
// and of their tangential momenta.
template <int AX, int FAX>
DG_FX void fx_face_flux(const FxParams &P, i64 v[10], const i64 m[3])
{
    constexpr int T1 = AX == 0 ? 1 : 0, T2 = AX == 2 ? 1 : 2;
    i64 rho = m[0], j[3];
    j[AX] = 0;
    j[T1] = m[1];
    j[T2] = m[2];
DG_UNROLL
    for (int s = 0; s < 10; ++s) {
        const int p = flux_pop(AX, s);
        rho += v[s];
DG_UNROLL
        for (int a = 0; a < 3; ++a)
            if (cc(a, p)) j[a] += cc(a, p) > 0 ? v[s] : -v[s];
    }
    const FxEq E = fx_eq<FAX>(rho, j, P.face, P.third);
DG_UNROLL
    for (int s = 0; s < 10; ++s) {
        const int p = flux_pop(AX, s), q = opp(p), sq = flux_slot(AX, q);
        if (q < p) continue;
        i64 fp = v[s] >> P.esh, fq = v[sq] >> P.esh;
        fx_pair<FAX>(E, p, fp, fq);
        v[s] = fp;
        v[sq] = fq;
    }
}

#ifdef __CUDACC__

// Outside the box of the range comment.  f-tilde as FP64: positive values compare
// like their high words.
__device__ __forceinline__ bool fx_bad_double(double x, int p)
{
    const double w = weight<double>(p);
    const unsigned lo = unsigned(__double2hiint(w * FX_LO)) + 1, hi = unsigned(__double2hiint(w * FX_HI));
    return unsigned(__double2hiint(x)) - lo >= hi - lo;
}
__device__ __forceinline__ bool fx_bad(i64 x, int p)
{
    const double w = weight<double>(p);
    const unsigned lo = unsigned(w * FX_LO * 1073741824.0) + 1, hi = unsigned(w * FX_HI * 1073741824.0);
    return unsigned(x >> 32) - lo >= hi - lo;
}

// Device words of a handle: the range flag, raised by stage (a) and lowered by the step
// that it redoes; what f-bar-plus holds (0: FP64, 1: fixed point); CTAs of fp64_redo_kernel that
// have read the flag; whether the caller has f-bar-plus's address (every step runs in FP64).
constexpr int FXW_FLAG = 0, FXW_FIXED = 1, FXW_DONE = 2, FXW_SHOWN = 3, FXW_WORDS = 4;
__device__ __forceinline__ bool fx_in_fp64(const int *words) { return __ldcg(words + FXW_FLAG) | __ldcg(words + FXW_SHOWN); }

// Stage (a), one thread per cell, x ghost columns included.  xoff: cells shifted by
// one thread when nx = 1 (mod 32), so that cells nx-2 and nx-1 share a warp.
template <int FAX>
__global__ void __launch_bounds__(128) fbar_fx_kernel(const double *__restrict__ f, i64 *__restrict__ fb,
                                                      const FxParams P, int xoff, int *words)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x - xoff;
    const int j = blockIdx.y, k = blockIdx.z, nx = P.nx;
    const bool in = i >= 0 && i < nx;
    const int ic = in ? i : (i < 0 ? 0 : nx - 1);
    const double *src = f + ((long long)k * P.ny + j) * P.pitch + ic;
    i64 v[NPOP], ob[NPOP];
    bool bad = false;
#pragma unroll
    for (int p = 0; p < NPOP; ++p) {
        const double x = __ldg(src + p * P.ps);
        bad |= fx_bad_double(x, p);
        v[p] = fx_from_double(x);
    }
    // another block's cell is out of range already (or all steps run in FP64): nothing here is read
    if (__any_sync(0xffffffffu, fx_in_fp64(words))) return;
    fx_stage_a<FAX>(P, v, ob);
    i64 *row = fb + ((long long)k * P.ny + j) * P.rs;
    i64 *dst = row + fx_col(ic);
#pragma unroll
    for (int p = 0; p < NPOP; ++p) {
        bad |= fx_bad(ob[p], p);
        if (in) dst[p * 16] = ob[p];
    }
    const int w0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31) - xoff;  // cell of lane 0
    if (w0 <= 0) {  // the warp of cell 0: the ghost below it, or the image of cell 0 above cell nx-1
        i64 *g = row + fx_col(P.periodic_x ? nx : nx + 1);
#pragma unroll
        for (int p = 0; p < NPOP; ++p) {
            const i64 n = __shfl_down_sync(0xffffffffu, ob[p], 1);
            const i64 e = P.periodic_x ? ob[p] : fx_mad(ob[p] - n, P.q0, ob[p] + (ob[p] - n));
            if (i == 0) {
                bad |= fx_bad(e, p);
                g[p * 16] = e;
            }
        }
    }
    if (w0 <= nx - 1 && w0 + 31 >= nx - 1) {  // the warp of cell nx-1
        i64 *g = row + fx_col(P.periodic_x ? nx + 1 : nx);
#pragma unroll
        for (int p = 0; p < NPOP; ++p) {
            const i64 n = __shfl_up_sync(0xffffffffu, ob[p], 1);
            const i64 e = P.periodic_x ? ob[p] : fx_mad(ob[p] - n, P.q1, ob[p] + (ob[p] - n));
            if (i == nx - 1) {
                bad |= fx_bad(e, p);
                g[p * 16] = e;
            }
        }
    }
    if (bad && in) atomicOr(words + FXW_FLAG, 1);
}

// Where f-bar-plus is read around a cell: plane pointers k-1..k+1, row and column
// offsets of the neighbours (periodic in y and z, ghosts stored in x).
struct FxAt {
    const i64 *pl[3];
    int row[3], col[3];
    __device__ __forceinline__ i64 operator()(int p, int dx, int dy, int dz) const
    {
        return __ldg(pl[dz + 1] + (row[dy + 1] + col[dx + 1]) + p * 16);
    }
};

// Population p interpolated within plane dz of A, transversely to the faces normal to AX.
template <int AX>
__device__ __forceinline__ i64 fx_inplane(const FxParams &P, const FxAt &A, FxMul txp, FxMul txm, int p, int dz)
{
    const int ax = AX == 0 ? 0 : cx(p), ay = AX == 1 ? 0 : cy(p);
    const FxMul tx = ax > 0 ? txp : txm;
    i64 a = A(p, 0, 0, dz);
    if (ax) a = fx_lerp(a, A(p, -ax, 0, dz), tx);
    if (ay) {
        i64 b = A(p, 0, -ay, dz);
        if (ax) b = fx_lerp(b, A(p, -ax, -ay, dz), tx);
        a = fx_lerp(a, b, P.ty);
    }
    return a;
}

// In-plane part of the z-moving populations at plane k (A's middle plane) where c_z > 0,
// at k + 1 where c_z < 0.  A transverse value at plane k lies between this at k and at
// k - 1 (both kinds reach back one of the two), so the march along z forms it once per
// plane and keeps the last one.
template <int AX>
__device__ __forceinline__ void fx_zparts(const FxParams &P, const FxAt &A, FxMul txp, FxMul txm, i64 old[10])
{
#pragma unroll
    for (int s = 0; s < 10; ++s) {
        const int p = flux_pop(2, s);
        old[s] = fx_inplane<AX>(P, A, txp, txm, p, cz(p) > 0 ? 0 : 1);
    }
}

constexpr int FXG = 13;

// Transverse interpolation of every population at one cell for the faces normal to
// AX: put(n, x), n = 0..9 the populations that cross such a face, n = 10..12 the sums over
// the others of their values and tangential momenta (their normal weights are equal, so
// the face needs the sums only).  A face value is then one interpolation between
// the two cells across it: each cell's transverse values are formed once per axis
// and used by both of its faces.  AX < 2, old: fx_zparts of plane k - 1, becomes that of k.
template <int AX, class Put>
__device__ __forceinline__ void fx_cell_values(const FxParams &P, const FxAt &A, FxMul txp, FxMul txm, i64 *old, Put put)
{
    constexpr int T1 = AX == 0 ? 1 : 0, T2 = AX == 2 ? 1 : 2;
    i64 m[3] = {A(0, 0, 0, 0), 0, 0};
#pragma unroll
    for (int p = 1; p < NPOP; ++p) {
        const bool z = AX < 2 && cz(p) != 0;
        i64 x = fx_inplane<AX>(P, A, txp, txm, p, z && cz(p) < 0 ? 1 : 0);
        if (z) {
            i64 &o = old[flux_slot(2, p) < 0 ? 0 : flux_slot(2, p)];
            const i64 n = x;
            x = cz(p) > 0 ? fx_lerp(n, o, P.tz) : fx_lerp(o, n, P.tz);
            o = n;
        }
        if (cc(AX, p)) {
            put(flux_slot(AX, p), x);
            continue;
        }
        m[0] += x;
        if (cc(T1, p)) m[1] += cc(T1, p) > 0 ? x : -x;
        if (cc(T2, p)) m[2] += cc(T2, p) > 0 ? x : -x;
    }
#pragma unroll
    for (int s = 0; s < 3; ++s) put(10 + s, m[s]);
}

// mean of the two cells' sum s (0: values, 1 and 2: tangential momenta).  The values' sums
// are positive and below 1.32 each, not below 2 together: added as unsigned numbers
DG_FX i64 fx_mean(int s, i64 a, i64 b) { return s == 0 ? i64((u64(a) + u64(b)) >> 1) : (a + b) >> 1; }

// face value of crossing population p between the lower cell's a and the upper cell's b
template <int AX>
__device__ __forceinline__ i64 fx_normal(int s, i64 a, i64 b, FxMul mp, FxMul mm)
{
    return cc(AX, flux_pop(AX, s)) > 0 ? fx_lerp(a, b, mp) : fx_lerp(b, a, mm);
}

// shared memory of flux_fx_kernel, in elements
template <int R>
struct FxSmem {
    static constexpr int GX = 0, GY = GX + R * FXG * 34, YS = GY + (R + 2) * FXG * 32, XZ = YS + 2 * (R + 1) * 10 * 32,
                         X0 = XZ + 2 * R * 4 * 33, DZ = X0 + 2 * R * 6, GZ = DZ + 2 * R * 4 * 32, N = GZ + R * FXG * 32;
    static constexpr size_t bytes = sizeof(i64) * size_t(N);
};

// barrier of one group of warps
__device__ __forceinline__ void fx_bar(int id, int threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Stage (a) in FP64 with its ghost layer (fbar_kernel and fb_ghost_kernel in one pass), tasks
// t, t + step, ...: first every cell with its periodic images, then, between walls, the
// ghost of every row's end, which forms the values of its two cells again (in tasks of
// their own: beside a row's other cells they would take the whole warp's time twice).  A
// call, so that its registers are not the flux kernel's.
template <int R>
__device__ __noinline__ void fp64_stage_a(const double *f, double *fb, const StepParams<double, double> &P, long long t,
                                          long long step)
{
    const int nx = P.nx, ny = P.ny, nz = P.nz;
    const long long n = (long long)nx * ny * nz, tasks = n + (P.periodic_x ? 0 : 2LL * ny * nz);
    for (; t < tasks; t += step) {
        const bool cell = t < n;
        const long long r = cell ? t / nx : (t - n) >> 1;
        const int i = cell ? int(t - r * nx) : ((t - n) & 1 ? nx - 1 : 0), j = int(r % ny), k = int(r / ny);
        const double q = i == 0 ? P.q0 : P.q1;
        double ob[NPOP];
#pragma unroll 1
        for (int m = cell; m < 2; ++m) {  // the cell itself last
            const int c = m ? i : (i == 0 ? 1 : nx - 2);
            const double *src = f + ((long long)k * ny + j) * P.pitch + c;
            double v[NPOP], o[NPOP];
#pragma unroll
            for (int p = 0; p < NPOP; ++p) v[p] = src[p * P.ps];
            fbar_cell(P, c, j, k, v, o);
#pragma unroll
            for (int p = 0; p < NPOP; ++p) ob[p] = cell ? o[p] : (m ? q * o[p] + ob[p] : (1.0 - q) * o[p]);
        }
        auto put = [&](int I) {
            fb_images(j, k, ny, nz, [&](int J, int K) {
                double *d = fb + ((long long)K * (ny + 2) + J) * P.pitch_b + I;
#pragma unroll
                for (int p = 0; p < NPOP; ++p) d[p * P.ps_b] = ob[p];
            });
        };
        put(cell ? i + 1 : (i == 0 ? 0 : nx + 1));
        if (cell && P.periodic_x && i == 0) put(nx + 1);
        if (cell && P.periodic_x && i == nx - 1) put(0);
    }
}

// Stages (b)-(e).  A CTA holds R rows of 32 cells (lane = x) and marches a chunk of z
// planes.  Each axis has warps of its own: R + 1 for x (the last one, the halo warp, the
// columns left and right of the tile), R + 2 for y (the rows -1 .. R), R for z.  Per plane:
//   1. every warp forms its cells' transverse values; those of x and y are published in
//      shared memory (gx, gy), those of z carried from plane to plane in registers;
//   2. after a barrier of the axis' own warps it evaluates its faces (x: +x, the halo warp
//      -x of the first column; y: the face below its row; z: +z) and publishes the fluxes
//      that other warps need;
//   3. after a barrier of the CTA the x, y and z warp of a row update a third of its
//      populations each: those whose flux differences they hold, so that four of the ten
//      fluxes of an axis cross over (fxz, ysh, dzs; double-buffered, read until the
//      next such barrier).
// Bound by latency: with one warp per row doing all of it (values of all three axes and
// z carries in registers) the loads' latency showed between spills, issue 33 %; split by
// axis a thread carries few values, three times the warps share a tile and their phases
// overlap, issue 40 to 45 %, ALU pipe 40 %.  256 x 128 x 128 channel: 1.45 -> 1.01 ms; 64 x 32 x
// 32: a step 78 -> 37 us (R = 7 and 4, see flux_fx_tiling; R = 5 and 6, with warps that do
// not divide evenly over the schedulers, 1.2 to 1.3 ms).  Waits split into arrive and wait (mbarriers), with the
// next plane's values in between, were slower (1.5 ms), and so was an even split of all
// planes over one CTA per SM (1.09 ms: tiles next to each other, at different planes, no
// longer share rows in L2).
template <int R, int FAX>
__global__ void __launch_bounds__(32 * (3 * R + 3)) flux_fx_kernel(i64 *fb, const double *f_in, double *f_out,
                                                                   const FxParams P, const int *words)
{
    using L = FxSmem<R>;
    constexpr int ALL = 32 * (3 * R + 3);  // threads of the CTA, which meet at barrier 0 from the branches of the three axes
    extern __shared__ __align__(16) i64 sm[];
    i64(*gx)[FXG][34] = reinterpret_cast<i64(*)[FXG][34]>(sm + L::GX);               // [row]
    i64(*gy)[FXG][32] = reinterpret_cast<i64(*)[FXG][32]>(sm + L::GY);               // [row + 1]
    i64(*ysh)[R + 1][10][32] = reinterpret_cast<i64(*)[R + 1][10][32]>(sm + L::YS);  // [parity][face below row]
    i64(*fxz)[R][4][33] = reinterpret_cast<i64(*)[R][4][33]>(sm + L::XZ);            // x fluxes of populations 11..14
    i64(*xs0)[R][6] = reinterpret_cast<i64(*)[R][6]>(sm + L::X0);                    // -x fluxes of the first column, 1, 2, 7..10
    i64(*dzs)[R][4][32] = reinterpret_cast<i64(*)[R][4][32]>(sm + L::DZ);            // z differences of populations 15..18
    if (fx_in_fp64(words)) {  // a value out of range: fp64_redo_kernel does the rest of the step
        // a warp takes every n-th 32 tasks, neighbours on different SMs: an incomplete last round spreads over all
        const long long ctas = (long long)gridDim.x * gridDim.y * gridDim.z;
        const long long cta = blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z);
        fp64_stage_a<R>(f_in, reinterpret_cast<double *>(fb), *static_cast<const StepParams<double, double> *>(P.step),
                        (threadIdx.y * ctas + cta) * 32 + threadIdx.x, ctas * ALL);
        return;
    }

    const int lane = threadIdx.x, wr = threadIdx.y;
    const int nx = P.nx, ny = P.ny, nz = P.nz, xs = nx + 2;
    const long long plane = (long long)ny * P.rs;
    auto wrap = [](int a, int n) { return a < 0 ? a + n : (a >= n ? a - n : a); };
    auto wrapc = [&](int a, int n) { a = wrap(a, n); return a < n ? a : n - 1; };  // rows past a ragged last tile: any valid row
    FxAt A;
    auto rows = [&](int j) {
        A.row[0] = wrap(j - 1, ny) * P.rs;
        A.row[1] = j * P.rs;
        A.row[2] = wrap(j + 1, ny) * P.rs;
    };
    auto cols = [&](int c) {  // c = -1 .. nx (ghost columns at nx + 1 and nx)
        A.col[0] = fx_col(c <= 0 ? nx + 1 : c - 1);
        A.col[1] = fx_col(c < 0 ? nx + 1 : c);
        A.col[2] = fx_col(min(c + 1, nx));
    };
    auto planes = [&](int k) {  // k = -1 .. nz
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            int q = k + d - 1;
            q = wrap(wrap(q, nz), nz);
            A.pl[d] = fb + q * plane;
        }
    };
    auto at_x = [&](int I, int row) {
        const int2 m = __ldg(reinterpret_cast<const int2 *>(P.tab) + row * xs + I);
        return FxMul{m.x, m.y};
    };
    const int c0 = blockIdx.x * 32;  // first column of the tile (0-based cell)
    const int j0 = blockIdx.y * R;   // first row
    const int kb = int((long long)nz * blockIdx.z / gridDim.z), ke = int((long long)nz * (blockIdx.z + 1) / gridDim.z);
    const int gc = c0 + lane, cc1 = min(gc, nx - 1);
    // f = 4/3 f-bar-plus - 1/3 f (less the flux differences) of population p of the cell at A
    auto base = [&](int p, long long c) {
        const i64 b = A(p, 0, 0, 0);
        return fx_madr(b - fx_from_double(f_in[p * P.ps + c]), P.third, b);
    };

    if (wr <= R) {
        // --- x: cell whose values the thread forms: its own; in the halo warp, lane by
        // lane, the column left of the tile (lanes 0..R-1) and the one right of it
        const bool halo = wr == R;
        const int hs = lane >= R, hr = min(hs ? lane - R : lane, R - 1);
        const int row = wrapc(j0 + (halo ? hr : wr), ny);
        const int r = halo ? hr : wr;
        i64 *gxw = &gx[r][0][halo ? (hs ? 33 : 0) : lane + 1];
        const bool gxs = !halo || lane < 2 * R;
        // x face the thread evaluates: I (between 1-based columns I and I+1) of tile row
        // xr; a lane past the last column takes that column's face, a valid one
        const int I = halo ? c0 : min(gc + 1, nx), xr = halo ? min(lane, R - 1) : wr, q = I - c0;
        const FxMul mp = at_x(I, FXT_MP), mm = at_x(I, FXT_MM), cxm = at_x(cc1 + 1, FXT_CX);
        const bool cell = !halo && gc < nx && j0 + wr < ny;
        const int restrow = wrapc(j0 + xr, ny) * P.rs;
        rows(row);
        cols(halo ? (hs ? min(c0 + 32, nx) : c0 - 1) : min(gc, nx));
        i64 old[10];
        planes(kb - 1);
        fx_zparts<0>(P, A, FxMul{}, FxMul{}, old);
        for (int k = kb; k < ke; ++k) {
            planes(k);
            fx_cell_values<0>(P, A, FxMul{}, FxMul{}, old, [&](int n, i64 x) {
                if (gxs) gxw[n * 34] = x;
            });
            fx_bar(1, 32 * (R + 1));
            i64 v[10], m[3];
#pragma unroll
            for (int s = 0; s < 10; ++s) v[s] = fx_normal<0>(s, gx[xr][s][q], gx[xr][s][q + 1], mp, mm);
            if (P.stretched) {
                // weight 1/2 + d on the upper cell, except for the rest population (1/2)
                const FxMul d = at_x(I, FXT_D0);
                const i64 *rr = A.pl[1] + restrow;
                const i64 rest = __ldg(rr + fx_col(I)) - __ldg(rr + fx_col(I == 0 ? nx + 1 : I - 1));
#pragma unroll
                for (int s = 0; s < 3; ++s) {
                    const i64 a = gx[xr][10 + s][q], b = gx[xr][10 + s][q + 1];
                    m[s] = fx_mad(b - a - (s == 0 ? rest : 0), d, fx_mean(s, a, b));
                }
            } else {
#pragma unroll
                for (int s = 0; s < 3; ++s) m[s] = fx_mean(s, gx[xr][10 + s][q], gx[xr][10 + s][q + 1]);
            }
            if (!P.periodic_x) {
                // bounce-back on the walls: populations entering the fluid take their opposites' values
                if (I == 0) {
                    v[0] = v[1]; v[2] = v[5]; v[4] = v[3]; v[6] = v[9]; v[8] = v[7];
                }
                if (I == nx) {
                    v[1] = v[0]; v[5] = v[2]; v[3] = v[4]; v[9] = v[6]; v[7] = v[8];
                }
            }
            fx_face_flux<0, FAX>(P, v, m);
            const int b = k & 1;
            if (halo) {
                if (lane < R) {
#pragma unroll
                    for (int s = 0; s < 6; ++s) xs0[b][lane][s] = v[s];
#pragma unroll
                    for (int s = 0; s < 4; ++s) fxz[b][lane][s][0] = v[6 + s];
                }
                fx_bar(0, ALL);
                continue;
            }
#pragma unroll
            for (int s = 0; s < 4; ++s) fxz[b][wr][s][lane + 1] = v[6 + s];
            const long long c = ((long long)k * ny + min(j0 + wr, ny - 1)) * P.pitch + cc1;
            i64 acc[7];  // populations 0, 1, 2, 7..10
#pragma unroll
            for (int n = 0; n < 7; ++n) acc[n] = base(n < 3 ? n : n + 4, c);
            fx_bar(0, ALL);
#pragma unroll
            for (int n = 0; n < 7; ++n) {
                const int p = n < 3 ? n : n + 4;
                i64 a = acc[n];
                if (cx(p)) {
                    const int s = flux_slot(0, p) < 0 ? 0 : flux_slot(0, p);
                    i64 l = __shfl_up_sync(0xffffffffu, v[s], 1);
                    if (lane == 0) l = xs0[b][wr][s];
                    a = fx_madr(cx(p) > 0 ? l - v[s] : v[s] - l, cxm, a);
                }
                if (cy(p)) {
                    const int s = flux_slot(1, p);
                    const i64 l = ysh[b][wr][s][lane], u = ysh[b][wr + 1][s][lane];
                    a = fx_madr(cy(p) > 0 ? l - u : u - l, P.cy, a);
                }
                if (cell) f_out[p * P.ps + c] = fx_to_double(a);
            }
        }
    } else if (wr <= 2 * R + 2) {
        // --- y: tile row yr - 1; the face below it (none for the last warp)
        const int yr = wr - (R + 1), gj = j0 + yr - 1;
        const FxMul txp = at_x(cc1 + 1, FXT_TXP), txm = at_x(cc1 + 1, FXT_TXM);
        const bool cell = yr >= 1 && yr <= R && gc < nx && gj < ny;
        rows(wrapc(gj, ny));
        cols(cc1);
        i64 *gyw = &gy[yr][0][lane];
        // plane k's f-bar-plus rows of the tile and f-tilde into L2 (last warp), two planes ahead of use
        auto prefetch = [&](int k) {
            const int q = wrap(k, nz);
            if (lane < R + 2)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(fb + q * plane + wrapc(wrap(j0 - 1 + lane, ny), ny) * (long long)P.rs + fx_col(c0)),
                             "r"(unsigned(min(2, (P.pitch_b - c0) >> 4) * NPOP * 16 * 8)));
            if (k < ke)
                for (int t = lane; t < NPOP * R * 2; t += 32) {
                    const int p = t / (2 * R), r = (t >> 1) % R;
                    const long long o = p * P.ps + ((long long)k * ny + min(j0 + r, ny - 1)) * P.pitch + min(c0 + 16 * (t & 1), nx - 1);
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(f_in + o));
                }
        };
        i64 old[10];
        planes(kb - 1);
        fx_zparts<1>(P, A, txp, txm, old);
        for (int k = kb; k < ke; ++k) {
            planes(k);
            fx_cell_values<1>(P, A, txp, txm, old, [&](int n, i64 x) { gyw[n * 32] = x; });
            fx_bar(2, 32 * (R + 2));
            if (yr > R) {
                if (k + 2 <= ke) prefetch(k + 2);
                fx_bar(0, ALL);
                continue;
            }
            // face between tile rows yr - 1 (gy[yr]) and yr
            i64 v[10], m[3];
#pragma unroll
            for (int s = 0; s < 10; ++s) v[s] = fx_normal<1>(s, gy[yr][s][lane], gy[yr + 1][s][lane], P.my, P.my);
#pragma unroll
            for (int s = 0; s < 3; ++s) m[s] = fx_mean(s, gy[yr][10 + s][lane], gy[yr + 1][10 + s][lane]);
            fx_face_flux<1, FAX>(P, v, m);
            const int b = k & 1;
#pragma unroll
            for (int s = 0; s < 10; ++s) ysh[b][yr][s][lane] = v[s];
            if (yr == 0) {
                fx_bar(0, ALL);
                continue;
            }
            const long long c = ((long long)k * ny + min(gj, ny - 1)) * P.pitch + cc1;
            i64 acc[6];  // populations 3, 4, 15..18
#pragma unroll
            for (int n = 0; n < 6; ++n) acc[n] = base(n < 2 ? 3 + n : 13 + n, c);
            fx_bar(0, ALL);
#pragma unroll
            for (int n = 0; n < 6; ++n) {
                const int p = n < 2 ? 3 + n : 13 + n, s = flux_slot(1, p);
                const i64 l = ysh[b][yr - 1][s][lane];
                i64 a = fx_madr(cy(p) > 0 ? l - v[s] : v[s] - l, P.cy, acc[n]);
                if (cz(p)) a = fx_madr(dzs[b][yr - 1][flux_slot(2, p) - 6][lane], P.cz, a);
                if (cell) f_out[p * P.ps + c] = fx_to_double(a);
            }
        }
    } else {
        // --- z
        const int r = wr - (2 * R + 3), gj = j0 + r;
        const FxMul txp = at_x(cc1 + 1, FXT_TXP), txm = at_x(cc1 + 1, FXT_TXM), cxm = at_x(cc1 + 1, FXT_CX);
        const bool cell = gc < nx && gj < ny;
        rows(wrapc(gj, ny));
        cols(cc1);
        i64 *gz = sm + L::GZ + r * FXG * 32 + lane;  // the thread's values of the last plane
        i64 fz[10];                                  // flux below plane k
        planes(kb - 1);
        fx_cell_values<2>(P, A, txp, txm, nullptr, [&](int n, i64 x) { gz[n * 32] = x; });
        // one round ahead of the first plane for the flux below it
        for (int k = kb - 1; k < ke; ++k) {
            i64 v[10], m[3];
            planes(k + 1);
            fx_cell_values<2>(P, A, txp, txm, nullptr, [&](int n, i64 x) {
                const i64 o = gz[n * 32];
                gz[n * 32] = x;
                if (n < 10)
                    v[n < 10 ? n : 0] = fx_normal<2>(n < 10 ? n : 0, o, x, P.mz, P.mz);
                else
                    m[n < 10 ? 0 : n - 10] = fx_mean(n - 10, o, x);
            });
            fx_face_flux<2, FAX>(P, v, m);
            if (k >= kb) {
                const int b = k & 1;
#pragma unroll
                for (int s = 0; s < 10; ++s) fz[s] = cz(flux_pop(2, s)) > 0 ? fz[s] - v[s] : v[s] - fz[s];
#pragma unroll
                for (int s = 0; s < 4; ++s) dzs[b][r][s][lane] = fz[6 + s];
                planes(k);
                const long long c = ((long long)k * ny + min(gj, ny - 1)) * P.pitch + cc1;
                i64 acc[6];  // populations 5, 6, 11..14
#pragma unroll
                for (int n = 0; n < 6; ++n) acc[n] = fx_madr(fz[n], P.cz, base(n < 2 ? 5 + n : 9 + n, c));
                fx_bar(0, ALL);
#pragma unroll
                for (int n = 0; n < 6; ++n) {
                    const int p = n < 2 ? 5 + n : 9 + n;
                    i64 a = acc[n];
                    if (cx(p)) {
                        const i64 l = fxz[b][r][n - 2 < 0 ? 0 : n - 2][lane], u = fxz[b][r][n - 2 < 0 ? 0 : n - 2][lane + 1];
                        a = fx_madr(cx(p) > 0 ? l - u : u - l, cxm, a);
                    }
                    if (cell) f_out[p * P.ps + c] = fx_to_double(a);
                }
            }
#pragma unroll
            for (int s = 0; s < 10; ++s) fz[s] = v[s];
        }
    }
}

#endif  // __CUDACC__

}  // namespace dg
