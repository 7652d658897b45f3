// Stages (b)-(e) of the float forms (FP32 and the 16-bit storage forms) with the
// central-difference ("gradient") reconstruction, f_face = mean - hdt (c . grad): face
// values, face flux and finite-volume update (src/dugks.cu:421-649, calc_fx).
//
// What bounds it is instruction issue and shared-memory reads, so the transverse
// derivatives are formed once per cell and axis: a cell contributes the same value,
// f - hdt (c_t d/dt) over the two transverse axes, to both of its faces normal to an
// axis, and the face adds the mean of two such values and the normal derivative.  The 9
// populations that do not cross a face enter it only through its density and
// tangential momentum, so a cell contributes their three sums.  A step of the 97 x 66 x
// 130 channel on the stretched mesh, FP32: 0.174 -> 0.129 ms against faces that each
// form their own derivatives.  (The trilinear reconstruction gains too, FP32 15 % a
// step, but in another order of its lerps: its results would change in the last place
// of FP32, so it keeps flux_tma_kernel.)
#pragma once
#include "dugks_kernels.cuh"

namespace dg {

// ---------------------------------------------------------------------------
// packed arithmetic on population pairs (2m-1, 2m): sm_100+ FADD2 / FMUL2 / FFMA2
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float sub_stored(float b, float a) { return b - a; }

// The population pairs of the packed code: crossing pairs (flux_pop(AX, 2n), + 1) and
// these four that do not cross a face normal to AX -- along the first transverse
// axis t1, along the second t2, and the diagonals with c_t2 = +1 and -1 (c_t1 is
// (+, -) within the pair).
__host__ __device__ constexpr int nc_pair(int ax, int n)
{
    return ax == 0 ? (n == 0 ? 3 : n == 1 ? 5 : n == 2 ? 15 : 17)
         : ax == 1 ? (n == 0 ? 1 : n == 1 ? 5 : n == 2 ? 11 : 13)
                   : (n == 0 ? 1 : n == 1 ? 3 : n == 2 ? 7 : 9);
}
__host__ __device__ constexpr int axis_t1(int ax) { return ax == 0 ? 1 : 0; }
__host__ __device__ constexpr int axis_t2(int ax) { return ax == 2 ? 1 : 2; }

// The pairing rule: crossing pairs share their transverse axes and every pair moving
// along x transversally is (c_x > 0, c_x < 0); crossing diagonals are (t1 axis: D1, D2
// with c_n or c_t1 dup), laid out as face_flux_sh takes them.
__host__ __device__ constexpr bool sh_pairs_ok()
{
    for (int ax = 0; ax < 3; ++ax) {
        const int t1 = axis_t1(ax), t2 = axis_t2(ax);
        for (int n = 0; n < 9; ++n) {
            const int p = n < 5 ? flux_pop(ax, 2 * n) : nc_pair(ax, n - 5), q = p + 1;
            if (n < 5 && (flux_pop(ax, 2 * n + 1) != q || p % 2 != 1)) return false;
            for (int t = 0; t < 3; ++t)
                if ((cc(t, p) != 0) != (cc(t, q) != 0)) return false;
            if (ax != 0 && cx(p) != 0 && !(cx(p) == 1 && cx(q) == -1)) return false;
            if (n >= 5 && cc(ax, p) != 0) return false;
        }
        for (int n = 0; n < 4; ++n) {
            const int p = nc_pair(ax, n), q = p + 1;
            if (n != 1 && !(cc(t1, p) == 1 && cc(t1, q) == -1)) return false;
            if (n == 1 && !(cc(t2, p) == 1 && cc(t2, q) == -1)) return false;
            if (n == 2 && !(cc(t2, p) == 1 && cc(t2, q) == 1)) return false;
            if (n == 3 && !(cc(t2, p) == -1 && cc(t2, q) == -1)) return false;
        }
    }
    return true;
}
static_assert(sh_pairs_ok(), "population pairs of the shared-transverse flux kernel");

// ---------------------------------------------------------------------------
// f-bar-plus around one cell of the tile: its population 0 in the planes k-1, k, k+1
// ---------------------------------------------------------------------------
template <class S, int W>
struct TileAt {
    static constexpr int BXT = TmaTile<S>::BXT, POPS = BXT * (W + 1);
    static constexpr int STAGE_BYTES = ((NPOP * POPS * int(sizeof(S))) + 127) / 128 * 128;
    static constexpr int STAGE = STAGE_BYTES / int(sizeof(S));
    const S *b[3];
    __device__ __forceinline__ S operator()(int p, int dx, int dy, int dz) const
    {
        return b[dz + 1][p * POPS + dy * BXT + dx];
    }
};

// hdt times the weights of the x derivative at a column on columns i-1, i, i+1
struct XDeriv {
    float wm, w0, wp;
};

// The pair (p, p + 1) at a cell less hdt c_t d/dt along the axes transverse to AX, by
// central differences (src/dugks.cu:459-583).
template <class S, int W, int AX>
__device__ __forceinline__ float2 pair_value(const StepParams<float, S> &P, const TileAt<S, W> &A, const XDeriv &X, int p)
{
    const int q = p + 1;
    const bool ax = AX != 0 && cx(p) != 0, ay = AX != 1 && cy(p) != 0, az = AX != 2 && cz(p) != 0;
    const float2 f = make_float2(float(A(p, 0, 0, 0)), float(A(q, 0, 0, 0)));
    float2 v = f;
    if (ax) {  // c_x = (+, -)
        const float2 a = make_float2(float(A(p, -1, 0, 0)), float(A(q, -1, 0, 0)));
        const float2 b = make_float2(float(A(p, 1, 0, 0)), float(A(q, 1, 0, 0)));
        const float2 d = __ffma2_rn(dup2(X.wp), b, __ffma2_rn(dup2(X.w0), f, __fmul2_rn(dup2(X.wm), a)));
        v = __ffma2_rn(make_float2(-1.0f, 1.0f), d, v);
    }
    // c (f(+1) - f(-1)) = f(+c) - f(-c)
    if (ay) {
        const float2 d = make_float2(sub_stored(A(p, 0, -cy(p), 0), float(A(p, 0, cy(p), 0))),
                                     sub_stored(A(q, 0, -cy(q), 0), float(A(q, 0, cy(q), 0))));
        v = __ffma2_rn(dup2(P.hdt * P.g_i2dy), d, v);
    }
    if (az) {
        const float2 d = make_float2(sub_stored(A(p, 0, 0, -cz(p)), float(A(p, 0, 0, cz(p)))),
                                     sub_stored(A(q, 0, 0, -cz(q)), float(A(q, 0, 0, cz(q)))));
        v = __ffma2_rn(dup2(P.hdt * P.g_i2dz), d, v);
    }
    return v;
}

constexpr int SHG = 13;

// What a cell contributes to its faces normal to AX (16-bit forms: less the rest
// state): g[0..9] the crossing populations in flux_pop order, g[10] the sum of the
// others, g[11], g[12] their momenta along t1, t2.
template <class S, int W, int AX>
__device__ __forceinline__ void cell_values(const StepParams<float, S> &P, const TileAt<S, W> &A, const XDeriv &X,
                                            float g[SHG])
{
#pragma unroll
    for (int n = 0; n < 5; ++n) {
        const int p = flux_pop(AX, 2 * n);
        const float2 v = P.codec.dec_e2(p, p + 1, pair_value<S, W, AX>(P, A, X, p));
        g[2 * n] = v.x;
        g[2 * n + 1] = v.y;
    }
    float2 v[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        const int p = nc_pair(AX, n);
        v[n] = P.codec.dec_e2(p, p + 1, pair_value<S, W, AX>(P, A, X, p));
    }
    const float2 t1 = __fadd2_rn(v[0], __fadd2_rn(v[2], v[3]));
    const float2 all = __fadd2_rn(t1, v[1]), d = sub_x2(v[2], v[3]);
    g[10] = (all.x + all.y) + P.codec.dec_e(0, float(A(0, 0, 0, 0)));
    g[11] = t1.x - t1.y;
    g[12] = (v[1].x - v[1].y) + (d.x + d.y);
}

// Face equilibrium and flux divided by fw1 (src/dugks.cu:675-709, 912-943) of the 10
// crossing populations, in place, from their face values and the sums m over the
// others (density, t1 and t2 momentum).  face_flux of dugks_kernels.cuh for float.
template <class S, int AX, bool FF>
__device__ __forceinline__ void face_flux_sh(const StepParams<float, S> &P, float v[10], const float m[3], float fadd)
{
    auto V = [&](int n) { return make_float2(v[2 * n], v[2 * n + 1]); };
    float r, j[3];
    const float2 d12 = sub_x2(V(1), V(2)), d34 = sub_x2(V(3), V(4));
    const float2 s12 = __fadd2_rn(V(1), V(2)), s34 = __fadd2_rn(V(3), V(4));
    const float2 all = __fadd2_rn(V(0), __fadd2_rn(s12, s34));
    r = m[0] + (all.x + all.y);
    if constexpr (Codec<float, S>::deviation) r += 1.0f;
    if (AX == 0) {         // pairs (+,-) along x; (7,8)-(9,10) along y, (11,12)-(13,14) along z
        j[0] = all.x - all.y;
        j[1] = m[1] + (d12.x + d12.y);
        j[2] = m[2] + (d34.x + d34.y);
    } else if (AX == 1) {  // (3,4), (15..18) (+,-) along y; (7,8)-(9,10) along y, (+,-) along x; (15,16)-(17,18) along z
        const float2 n = __fadd2_rn(V(0), s34);
        j[0] = m[1] + (s12.x - s12.y);
        j[1] = (n.x - n.y) + (d12.x + d12.y);
        j[2] = m[2] + (d34.x + d34.y);
    } else {               // (5,6) (+,-) along z; (11,12)-(13,14), (15,16)-(17,18) along z; (+,-) along x, y
        const float2 n = __fadd2_rn(d12, d34);
        j[0] = m[1] + (s12.x - s12.y);
        j[1] = m[2] + (s34.x - s34.y);
        j[2] = (v[0] - v[1]) + (n.x + n.y);
    }
    const float inv = recip(r);
    float u = j[0] * inv, vv = j[1] * inv, w = j[2] * inv;
    float B = P.fw2s;
    float F[3] = {P.F[0], P.F[1], P.F[2]};
    if (FF) {
        F[0] += P.ffaxis == 0 ? fadd : 0.0f;
        F[1] += P.ffaxis == 1 ? fadd : 0.0f;
        F[2] += P.ffaxis == 2 ? fadd : 0.0f;
        const float hh = 0.5f * P.hdt;
        u = fmaf(hh, F[0], u);
        vv = fmaf(hh, F[1], vv);
        w = fmaf(hh, F[2], w);
        B = fmaf(-P.fw0x3s, fmaf(F[0], u, fmaf(F[1], vv, F[2] * w)), P.fw2s);
    } else if (P.force_on) {
        u += P.hF[0];
        vv += P.hF[1];
        w += P.hF[2];
        B = fmaf(-P.fw0x3s, fmaf(F[0], u, fmaf(F[1], vv, F[2] * w)), P.fw2s);
    }
    const float c3[3] = {3.0f * u, 3.0f * vv, 3.0f * w};
    const float base = fmaf(-1.5f, fmaf(u, u, fmaf(vv, vv, w * w)), 1.0f);
    const float wr1 = weight<float>(1) * r, wr2 = weight<float>(7) * r;
#pragma unroll
    for (int n = 0; n < 5; ++n) {
        const int p = flux_pop(AX, 2 * n), q = p + 1;
        // 3 c.u of the pair: one axis (+, -) and, on the diagonals, one shared
        float2 e = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int a = 0; a < 3; ++a)
            if (cc(a, p) && cc(a, p) != cc(a, q)) e = make_float2(c3[a], -c3[a]);
#pragma unroll
        for (int a = 0; a < 3; ++a)
            if (cc(a, p) && cc(a, p) == cc(a, q)) e = cc(a, p) > 0 ? __fadd2_rn(e, dup2(c3[a])) : sub_x2(e, dup2(c3[a]));
        float kp = P.Kfs[p], kq = P.Kfs[q];
        if (FF) {
            const int a = P.ffaxis;
            const int cp = a == 0 ? cx(p) : (a == 1 ? cy(p) : cz(p)), cq = a == 0 ? cx(q) : (a == 1 ? cy(q) : cz(q));
            kp = fmaf(float(cp) * P.fw0x3s, fadd, kp);
            kq = fmaf(float(cq) * P.fw0x3s, fadd, kq);
        }
        const float2 k = __fmul2_rn(__fadd2_rn(dup2(B), make_float2(kp, kq)), dup2(p <= 6 ? wr1 : wr2));
        const float2 t = __ffma2_rn(e, __ffma2_rn(dup2(0.5f), e, dup2(1.0f)), dup2(base));  // feq / (w rho)
        const float2 o = __ffma2_rn(k, t, V(n));
        v[2 * n] = o.x;
        v[2 * n + 1] = o.y;
    }
}

// A CTA is W warps: warps 1..W-1 one row of 32 cells each (lane = x), marching a
// chunk of z planes; warp 0 is the halo.  f-bar-plus planes of the tile (columns
// i0-1 .. i0+32, rows j0-1 .. j0+W-1, 19 populations) arrive in a 3-stage
// shared-memory ring through cp.async.bulk.tensor with mbarrier completion.  Per plane:
//   1. every thread forms what its cell contributes to x and y faces and publishes it
//      (gx, gy); the halo warp does so for the rows below and above the tile and the
//      columns left and right of it;
//   2. after a barrier plane k+2 is requested into the stage of plane k-1, and every
//      thread evaluates its +x, +z and +y faces, the halo warp the -y faces of the
//      first row and the -x faces of the first column;
//   3. after a second barrier the cells are updated.
// The z contributions and the z flux are carried from plane to plane in registers.
template <class S, int W>
constexpr size_t flux_sh_smem_bytes()
{
    return 3 * size_t(TileAt<S, W>::STAGE_BYTES) +
           sizeof(float) * ((W - 1) * SHG * 34 + (W + 1) * SHG * 32 + W * 10 * 32 + (W - 1) * 10) + 3 * 8 + 8;
}

template <class S, int W, int MINB, bool FF>
__global__ void __launch_bounds__(32 * W, MINB) flux_sh_kernel(const __grid_constant__ CUtensorMap tmap, const S *f_in,
                                                               S *f_out, const StepParams<float, S> P, int kchunk)
{
    using AT = TileAt<S, W>;
    // FP32: f-tilde fetched into L2 a plane ahead (256 x 128 x 128 channel 0.290 -> 0.286 ms).  A
    // cell's x, y and z contributions in one go, which shares a third of their reads, were
    // slower for the registers they take: 0.314 ms, FP16 0.410 against 0.370.
    constexpr bool PREFETCH = sizeof(S) == 4;
    constexpr int R = W - 1, BXT = AT::BXT;
    extern __shared__ __align__(128) unsigned char smem[];
    S *ring = reinterpret_cast<S *>(smem);
    float *ex = reinterpret_cast<float *>(smem + 3 * AT::STAGE_BYTES);
    float(*gx)[SHG][34] = reinterpret_cast<float(*)[SHG][34]>(ex);
    float(*gy)[SHG][32] = reinterpret_cast<float(*)[SHG][32]>(ex + R * SHG * 34);
    float(*ysh)[10][32] = reinterpret_cast<float(*)[10][32]>(ex + R * SHG * 34 + (R + 2) * SHG * 32);
    float(*xsh)[10] = reinterpret_cast<float(*)[10]>(ex + R * SHG * 34 + (R + 2) * SHG * 32 + W * 10 * 32);
    constexpr int EX = R * SHG * 34 + (R + 2) * SHG * 32 + W * 10 * 32 + R * 10;
    unsigned long long *mbar = reinterpret_cast<unsigned long long *>(ex + (EX + 1) / 2 * 2);
    constexpr unsigned TILE_BYTES = unsigned(NPOP * AT::POPS * sizeof(S));

    const int lane = threadIdx.x, wr = threadIdx.y, tid = wr * 32 + lane;
    const int nx = P.nx, ny = P.ny, nz = P.nz;
    const int i0 = blockIdx.x * 32 + 1, j0 = blockIdx.y * R + 1;
    const int kb = blockIdx.z * kchunk + 1, ke = min(kb + kchunk, nz + 1);
    if (kb >= ke) return;

    if (tid == 0) {
        for (int s = 0; s < 3; ++s)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar + s)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto issue = [&](int g, int s) {  // stored plane g -> stage s
        if (tid == 0 && g <= ke) {
            const unsigned bar = smem_u32(mbar + s);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(TILE_BYTES)
                         : "memory");
            asm volatile(
                "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
                "[%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(ring + s * AT::STAGE)),
                "l"(reinterpret_cast<unsigned long long>(&tmap)), "r"(i0 - 1), "r"(j0 - 1), "r"(g), "r"(0), "r"(bar)
                : "memory");
        }
    };
    unsigned phase = 0;  // bit s: parity of the next completion of stage s
    int wait_limit = kWaitPolls;
    auto wait = [&](int s) {
        if (!mbar_wait(smem_u32(mbar + s), (phase >> s) & 1u, wait_limit)) {
            atomicOr(P.err, 1);
            wait_limit = kWaitPollsAfterFailure;
        }
        phase ^= 1u << s;
    };

    // 16-bit forms between walls: the wall ghost columns 0 and nx+1 of f-bar-plus are
    // not stored (stage (a) writes the interior and its y / z images only); the tiles
    // that read them form them in shared memory from the landed plane, g0 = q0 d(1) +
    // (1-q0) d(2), g_{nx+1} = q1 d(nx) + (1-q1) d(nx-1) (src/dugks.cu:1234-1251;
    // stretched mesh src/fortran/channel/src/dugks.cuf:365-374), on the stored deviations
    // (the decode is affine) and rounded as the engine rounds every stored value
    // (stochastically, from the ghost cell's index; every tile that forms the same ghost
    // gets the same value).  Column 0 is read only by the first tile, column nx+1 only by
    // the tiles holding nx or starting past it.  (Formed by the whole CTA after each plane
    // lands, with one more block barrier in those tiles.)
    constexpr bool WALL_GHOST = sizeof(S) == 2;
    const int cwall_lo = (WALL_GHOST && !P.periodic_x && i0 == 1) ? 0 : -1;
    const int cwall_hi = (WALL_GHOST && !P.periodic_x && i0 <= nx && nx <= i0 + 31) ? nx + 1 - (i0 - 1) : -1;
    const bool wall_tile = cwall_lo >= 0 || cwall_hi >= 0;  // the same for the whole CTA
    auto wall_ghosts = [&](int g, int s) {
        if constexpr (WALL_GHOST) {
            S *st = ring + s * AT::STAGE;
            for (int t = tid; t < 2 * NPOP * (W + 1); t += 32 * W) {
                const int side = t / (NPOP * (W + 1)), seg = t - side * (NPOP * (W + 1));
                const int c = side ? cwall_hi : cwall_lo;
                if (c < 0) continue;
                S *row = st + seg * BXT;  // segment = one row of one population
                const int d = side ? -1 : 1;
                const float q = side ? P.q1 : P.q0;
                const float a = float(row[c + d]), b = float(row[c + 2 * d]);
                const int p = seg / (W + 1), r = seg - p * (W + 1);
                const long long dst = ((long long)g * (ny + 2) + (j0 - 1 + r)) * P.pitch_b + (i0 - 1 + c);
                row[c] = P.codec.encode_dev(p * P.ps_b + dst, p, q * a + (1.0f - q) * b);
            }
            // these writes before the stage's next TMA load
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
    };

    const int gi = i0 + lane, gj = j0 + wr - 1;
    const bool cell = wr >= 1 && gi <= nx && gj <= ny;
    const int ci = min(gi, nx);
    const int tx = ci - (i0 - 1);                     // tile column of the thread's cell (clamped)
    // cell whose contributions the thread forms: its own (or the ghost column); in the
    // halo warp, for x faces, lane by lane the column left of the tile (lanes 0..R-1) and right of it
    const int hs = lane >= R, hr = min(hs ? lane - R : lane, R - 1);
    const int xcol = wr ? min(gi, nx + 1) - (i0 - 1) : (hs ? 33 : 0);
    const int xoff = (wr ? wr : hr + 1) * BXT + xcol, yoff = wr * BXT + tx;
    float *gxw = &gx[wr ? wr - 1 : hr][0][wr ? lane + 1 : xcol];
    // x face the thread evaluates: between columns I and I+1 of tile row xr
    const int I = wr ? ci : i0 - 1, xr = wr ? wr - 1 : min(lane, R - 1), xq = I - (i0 - 1);
    const int xs = P.xws;
    XDeriv X;
    if (P.grad_st) {
        X.wm = P.hdt * __ldg(P.gw + GW_WM * xs + ci);
        X.w0 = P.hdt * __ldg(P.gw + GW_W0 * xs + ci);
        X.wp = P.hdt * __ldg(P.gw + GW_WP * xs + ci);
    } else {
        X.wm = -P.hdt * P.g_i2dx;
        X.w0 = 0.0f;
        X.wp = P.hdt * P.g_i2dx;
    }

    // cell of f-tilde: the tile's first cell in plane k (uniform over the CTA) and the thread's offset
    auto tile_cell = [&](int k) { return ((long long)(k - 1) * ny + (j0 - 1)) * P.pitch + (i0 - 1); };
    const unsigned coff = unsigned((wr - 1) * P.pitch + lane);
    AT A;
    auto at = [&](int o, int sm1, int s0, int s1) {
        A.b[0] = ring + sm1 * AT::STAGE + o;
        A.b[1] = ring + s0 * AT::STAGE + o;
        A.b[2] = ring + s1 * AT::STAGE + o;
    };
    // -hdt c_n d/dn of the crossing pair p across a face, added to its mean
    auto normal_grad = [&](int AXn, int p, const S *lo, const S *hi, int step, float k) {
        const float2 d = make_float2(sub_stored(hi[p * AT::POPS + step], float(lo[p * AT::POPS])),
                                     sub_stored(hi[(p + 1) * AT::POPS + step], float(lo[(p + 1) * AT::POPS])));
        return P.codec.dec_e2(p, p + 1, __fmul2_rn(make_float2(-float(cc(AXn, p)) * k, -float(cc(AXn, p + 1)) * k), d));
    };

    // the tile's f-tilde of plane k into L2 (halo warp), a plane ahead of its use
    auto prefetch = [&](int k) {
        const int seg = lane & 1 ? 128 / int(sizeof(S)) : 0;  // rows of 32 cells cover one or two lines
        for (int t = lane >> 1; t < NPOP * R; t += 16) {
            const int p = t / R, r = t - p * R;
            if (seg < 32)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(f_in + p * P.ps + ((long long)(k - 1) * ny + min(j0 - 1 + r, ny - 1)) * P.pitch + min(i0 - 1 + seg, nx - 1)));
        }
    };
    for (int s = 0; s < 3; ++s) issue(kb - 1 + s, s);
    float gz[SHG], fz[10], fo[NPOP];
    int sm1 = 1, s0 = 2, s1 = 0;  // stages of planes k-1, k, k+1
    // two rounds ahead of the first plane for the z contributions and flux below it
    for (int k = kb - 2; k < ke; ++k) {
        wait(s1);
        if (wall_tile) {
            wall_ghosts(k + 1, s1);
            __syncthreads();
        }
        float fx[10], dz[10], gax[SHG], gay[SHG], gzn[SHG];
        if (k >= kb) {
            // 1. contributions to the faces
            at(xoff, sm1, s0, s1);
            cell_values<S, W, 0>(P, A, X, gax);
            if (wr || lane < 2 * R) {
#pragma unroll
                for (int s = 0; s < SHG; ++s) gxw[s * 34] = gax[s];
            }
#pragma unroll 1
            for (int t = wr ? 0 : 1; t >= 0; --t) {  // the halo warp: the rows above and below the tile
                at(t ? (R + 1) * BXT + tx : yoff, sm1, s0, s1);
                cell_values<S, W, 1>(P, A, X, gay);
                float *w = &gy[t ? R + 1 : wr][0][lane];
#pragma unroll
                for (int s = 0; s < SHG; ++s) w[s * 32] = gay[s];
            }
            __syncthreads();
            issue(k + 2, sm1);  // plane k-1 is no longer read
            // 2. faces: x
            {
                const float *b = &gx[xr][0][xq + 1];
                float m[3];
                const S *cl = ring + s0 * AT::STAGE + (xr + 1) * BXT + xq;  // population 0 of cell I
                float om = 0.5f, mm = 0.5f, idn = P.g_idx;
                if (P.grad_st) {
                    // values interpolated to the face, normal difference over the centre spacing
                    mm = __ldg(P.gw + GW_LAM * xs + I);
                    om = 1.0f - mm;
                    idn = __ldg(P.gw + GW_IDX * xs + I);
                }
#pragma unroll
                for (int n = 0; n < 5; ++n) {
                    const int p = flux_pop(0, 2 * n);
                    const float2 v = lerp_x2(dup2(om), dup2(mm), make_float2(gax[2 * n], gax[2 * n + 1]),
                                             make_float2(b[2 * n * 34], b[(2 * n + 1) * 34]));
                    const float2 d = __fadd2_rn(v, normal_grad(0, p, cl, cl, 1, P.hdt * idn));
                    fx[2 * n] = d.x;
                    fx[2 * n + 1] = d.y;
                }
#pragma unroll
                for (int s = 0; s < 3; ++s) m[s] = om * gax[10 + s] + mm * b[(10 + s) * 34];
                if (!P.periodic_x) {
                    // bounce-back on the walls (src/dugks.cu:807-823)
                    if (I == 0) {
                        fx[0] = fx[1]; fx[2] = fx[5]; fx[4] = fx[3]; fx[6] = fx[9]; fx[8] = fx[7];
                    }
                    if (I == nx) {
                        fx[1] = fx[0]; fx[5] = fx[2]; fx[3] = fx[4]; fx[9] = fx[6]; fx[7] = fx[8];
                    }
                }
                face_flux_sh<S, 0, FF>(P, fx, m, FF ? face_field<float, S, 0>(P, I, min(j0 + xr, ny), k) : 0.0f);
                if (wr == 0 && lane < R) {
#pragma unroll
                    for (int s = 0; s < 10; ++s) xsh[lane][s] = fx[s];
                }
            }
            // y
            {
                const float *b = &gy[wr + 1][0][lane];
                float v[10], m[3];
                const S *cl = ring + s0 * AT::STAGE + yoff;
#pragma unroll
                for (int n = 0; n < 5; ++n) {
                    const int p = flux_pop(1, 2 * n);
                    float2 x = lerp_x2(dup2(0.5f), dup2(0.5f), make_float2(gay[2 * n], gay[2 * n + 1]),
                                       make_float2(b[2 * n * 32], b[(2 * n + 1) * 32]));
                    x = __fadd2_rn(x, normal_grad(1, p, cl, cl, BXT, P.hdt * P.g_idy));
                    v[2 * n] = x.x;
                    v[2 * n + 1] = x.y;
                }
#pragma unroll
                for (int s = 0; s < 3; ++s) m[s] = 0.5f * (gay[10 + s] + b[(10 + s) * 32]);
                face_flux_sh<S, 1, FF>(P, v, m, FF ? face_field<float, S, 1>(P, ci, wr ? min(gj, ny) : j0 - 1, k) : 0.0f);
#pragma unroll
                for (int s = 0; s < 10; ++s) ysh[wr][s][lane] = v[s];
            }
        }
        // z, between planes k and k+1
        if (wr >= 1) {
            at(xoff, sm1, s0, s1);
            {
                AT B = A;
                B.b[1] = A.b[2];
                cell_values<S, W, 2>(P, B, X, gzn);
            }
            if (k >= kb - 1) {
                float v[10], m[3];
#pragma unroll
                for (int n = 0; n < 5; ++n) {
                    const int p = flux_pop(2, 2 * n);
                    float2 x = lerp_x2(dup2(0.5f), dup2(0.5f), make_float2(gz[2 * n], gz[2 * n + 1]), make_float2(gzn[2 * n], gzn[2 * n + 1]));
                    x = __fadd2_rn(x, normal_grad(2, p, A.b[1], A.b[2], 0, P.hdt * P.g_idz));
                    v[2 * n] = x.x;
                    v[2 * n + 1] = x.y;
                }
#pragma unroll
                for (int s = 0; s < 3; ++s) m[s] = 0.5f * (gz[10 + s] + gzn[10 + s]);
                face_flux_sh<S, 2, FF>(P, v, m, FF ? face_field<float, S, 2>(P, ci, min(gj, ny), k) : 0.0f);
#pragma unroll
                for (int s = 0; s < 10; ++s) {
                    dz[s] = v[s] - fz[s];
                    fz[s] = v[s];
                }
            }
#pragma unroll
            for (int s = 0; s < SHG; ++s) gz[s] = gzn[s];
            // the cell's f-tilde, loaded before the barrier so its latency overlaps the exchange
            if (cell && k >= kb) {
                const S *fi = f_in + tile_cell(k);
#pragma unroll
                for (int p = 0; p < NPOP; ++p) fo[p] = P.codec.raw(fi + p * P.ps, coff);
            }
        }
        if (k >= kb) {
            __syncthreads();
            // 3. update
            if (wr >= 1) {
                float fxl[10];
#pragma unroll
                for (int s = 0; s < 10; ++s) {
                    const float up = __shfl_up_sync(0xffffffffu, fx[s], 1);
                    fxl[s] = lane == 0 ? xsh[wr - 1][s] : up;
                }
                if (cell) {
                    S *out = f_out + tile_cell(k);
                    const unsigned hc = P.codec.cell_hash(tile_cell(k) + coff);
                    const S *own = ring + s0 * AT::STAGE + yoff;
                    const float cxg = __ldg(P.cxuf + gi);
                    {
                        const UpdateSum<float, S> u(upd_base(float(own[0]), fo[0], 4.0f / 3.0f, 1.0f / 3.0f));
                        out[coff] = u.encode(P.codec, 0, hc);  // rest population
                    }
                    auto sgn = [](int a, float cval) { return a > 0 ? -cval : cval; };
#pragma unroll
                    for (int m = 1; m <= 9; ++m) {
                        const int p = 2 * m - 1, q = 2 * m;
                        UpdatePair<S> u(make_float2(float(own[p * AT::POPS]), float(own[q * AT::POPS])),
                                        make_float2(fo[p], fo[q]));
                        if (cx(p)) {
                            const int s = flux_slot(0, p);
                            u.add(make_float2(sgn(cx(p), cxg), sgn(cx(q), cxg)),
                                  sub_x2(make_float2(fx[s], fx[s + 1]), make_float2(fxl[s], fxl[s + 1])));
                        }
                        if (cy(p)) {
                            const int s = flux_slot(1, p);
                            u.add(make_float2(sgn(cy(p), P.cyuf), sgn(cy(q), P.cyuf)),
                                  sub_x2(make_float2(ysh[wr][s][lane], ysh[wr][s + 1][lane]),
                                         make_float2(ysh[wr - 1][s][lane], ysh[wr - 1][s + 1][lane])));
                        }
                        if (cz(p)) {
                            const int s = flux_slot(2, p);
                            u.add(make_float2(sgn(cz(p), P.czuf), sgn(cz(q), P.czuf)), make_float2(dz[s], dz[s + 1]));
                        }
                        u.store(P.codec, out, p * P.ps + coff, q * P.ps + coff, p, q, hc);
                    }
                }
            }
        }
        if (PREFETCH && wr == 0 && k + 1 < ke && k + 1 >= kb) prefetch(k + 1);
        const int s = sm1;
        sm1 = s0;
        s0 = s1;
        s1 = s;
    }
    // every plane issued (g <= ke) has been waited for: no bulk copy is left in flight
}

}  // namespace dg
