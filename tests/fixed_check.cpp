// CPU check of the fixed-point FP64 arithmetic (csrc/fixed_kernels.cuh): stage (a)
// of a cell and the flux of a face against quadruple precision, next to the same
// formulas in double.  Prints, per force axis and orientation, the largest error of
// both in units of 2^-62; run by tests/test_fixed_cpu.py.
//   fixed_check VISC DT F
#define __host__
#define __device__
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../dugks-gpu_gb300/csrc/fixed_kernels.cuh"

using namespace dg;
#ifdef __x86_64__
typedef __float128 quad;
#else
typedef long double quad;
#endif
static double mag(quad x) { return double(x < 0 ? -x : x); }

template <class R>
struct Coef {
    R w0, w1, w2, shift;
};
// stage (a) and face coefficients from viscosity, time step and force
template <class R>
static Coef<R> cell_coef(double visc, double dt, double F)
{
    const R tau = R(3) * R(visc), h = R(dt) / R(2), d = R(2) * tau + R(dt);
    return {R(3) * tau * h / d, (R(2) * tau - h) / d, R(3) * h / d, h * R(F)};
}
template <class R>
static Coef<R> face_coef(double visc, double dt, double F)
{
    const R tau = R(3) * R(visc), h = R(dt) / R(2), d = R(2) * tau + h;
    return {tau * h / d, R(2) * tau / d, h / d, h * R(F) / R(2)};
}

// w1 v_p + (w2 + 3 w0 F.(c - u)) feq_p for the values v, u = j / rho + shift
template <class R>
static void relax(const R v[NPOP], const Coef<R> &c, double F, int fax, R out[NPOP])
{
    R r = 0, j[3] = {0, 0, 0};
    for (int p = 0; p < NPOP; ++p) {
        r += v[p];
        for (int a = 0; a < 3; ++a) j[a] += R(cc(a, p)) * v[p];
    }
    R u[3];
    for (int a = 0; a < 3; ++a) u[a] = j[a] / r + (a == fax ? c.shift : R(0));
    const R uu = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
    for (int p = 0; p < NPOP; ++p) {
        const R w = p == 0 ? R(1) / R(3) : (p <= 6 ? R(1) / R(18) : R(1) / R(36));
        const R x = R(3) * (R(cx(p)) * u[0] + R(cy(p)) * u[1] + R(cz(p)) * u[2]);
        const R feq = w * r * (R(1) + x + x * x / R(2) - R(3) * uu / R(2));
        const R k = fax < 3 ? c.w2 + R(3) * c.w0 * R(F) * (R(cc(fax, p)) - u[fax]) : c.w2;
        out[p] = c.w1 * v[p] + k * feq;
    }
}

static FxMul mul(double m, double unit) { return fx_split(i64(std::llrint(std::ldexp(m / unit, 64)))); }

static FxForce force(const Coef<double> &c, double s, double F)
{
    FxForce f;
    f.shift = i64(std::llrint(std::ldexp(3 * c.shift, 61)));
    f.B = i64(std::llrint(std::ldexp(c.w2 / s / 18, 64)));
    f.C = mul(c.w0 / s * F / 18, 1.0 / 8);
    f.Kf = mul(3 * c.w0 / s * F / 18, 1);
    return f;
}

template <int FAX>
static void check(double visc, double dt, double F)
{
    if (FAX == 3) F = 0;
    const Coef<double> b = cell_coef<double>(visc, dt, F), g = face_coef<double>(visc, dt, F);
    const Coef<quad> bq = cell_coef<quad>(visc, dt, F), gq = face_coef<quad>(visc, dt, F);
    FxParams P{};
    while (std::ldexp(g.w1, P.esh) <= 0.5) ++P.esh;
    const double s = std::ldexp(g.w1, P.esh);
    P.cell = force(b, 1, F);
    P.face = force(g, s, F);
    P.bw1 = fx_split(i64((1ull << 63) - 9ull * u64(P.cell.B)));  // 1 - w2
    P.third = fx_split(0x5555555555555555ll);
    std::mt19937_64 rng(FAX + 1);
    std::uniform_real_distribution<double> U(-1, 1);
    double ea = 0, da = 0, ef[3] = {0, 0, 0}, df[3] = {0, 0, 0};
    for (int n = 0; n < 40000; ++n) {
        // from the whole box (large n) down to small deviations
        const double dev = std::pow(10.0, -3.0 * (n % 4) / 3.0);
        double v[NPOP];
        i64 x[NPOP];
        quad vq[NPOP], oq[NPOP];
        for (int p = 0; p < NPOP; ++p) {
            const double r = U(rng);
            v[p] = weight<double>(p) * (1 + dev * 0.999 * r * (r > 0 ? FX_HI - 1 : 1 - FX_LO));
            x[p] = fx_from_double(v[p]);
            vq[p] = v[p];
        }
        double od[NPOP];
        i64 o[NPOP];
        relax<quad>(vq, bq, F, FAX, oq);
        relax<double>(v, b, F, FAX, od);
        fx_stage_a<FAX>(P, x, o);
        const quad one = quad(FX_ONE);
        for (int p = 0; p < NPOP; ++p) {
            ea = std::max(ea, mag(quad(o[p]) - oq[p] * one));
            da = std::max(da, mag((quad(od[p]) - oq[p]) * one));
        }
        relax<quad>(vq, gq, F, FAX, oq);
        relax<double>(v, g, F, FAX, od);
        auto face = [&](auto axis) {
            constexpr int AX = decltype(axis)::value;
            i64 y[10], m[3] = {0, 0, 0};
            for (int p = 0; p < NPOP; ++p) {
                if (cc(AX, p)) {
                    y[flux_slot(AX, p)] = x[p];
                } else {
                    m[0] += x[p];
                    m[1] += cc(AX == 0 ? 1 : 0, p) * x[p];
                    m[2] += cc(AX == 2 ? 1 : 2, p) * x[p];
                }
            }
            fx_face_flux<AX, FAX>(P, y, m);
            for (int q = 0; q < 10; ++q) {
                const int p = flux_pop(AX, q);
                ef[AX] = std::max(ef[AX], mag(quad(y[q]) * quad(s) - oq[p] * one));
                df[AX] = std::max(df[AX], mag((quad(od[p]) - oq[p]) * one));
            }
        };
        face(std::integral_constant<int, 0>());
        face(std::integral_constant<int, 1>());
        face(std::integral_constant<int, 2>());
    }
    std::printf("%d a %.3f %.3f x %.3f %.3f y %.3f %.3f z %.3f %.3f\n", FAX, ea, da, ef[0], df[0], ef[1], df[1], ef[2], df[2]);
}

int main(int argc, char **argv)
{
    if (argc < 4) return 2;
    const double visc = std::atof(argv[1]), dt = std::atof(argv[2]), F = std::atof(argv[3]);
    check<0>(visc, dt, F);
    check<1>(visc, dt, F);
    check<2>(visc, dt, F);
    check<3>(visc, dt, F);
    return 0;
}
