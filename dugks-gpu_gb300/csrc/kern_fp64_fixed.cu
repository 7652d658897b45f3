// Launchers of the fixed-point FP64 step (fixed_kernels.cuh) and of the FP64
// kernel that redoes a step whose state left its range.
#include <cooperative_groups.h>

#include "fixed_launch.cuh"
#include "launch_impl.cuh"

namespace dg {
namespace {

// A whole FP64 step in one cooperative launch, run by every step of the fixed-point
// path behind its two kernels: returns at once unless stage (a) raised the flag.
// Then f-tilde is still the step's input, and stage (a), the ghost layer and the
// flux / update follow with grid-wide barriers in between; the flag is lowered.
// flag[1]: whether the last step was redone (f-bar-plus is then FP64).
template <int W, int MINB>
__global__ void __launch_bounds__(32 * W, MINB) fp64_redo_kernel(const double *f_in, double *f_out, double *fb,
                                                                 const StepParams<double, double> P, int *flag)
{
    const int tid = threadIdx.y * 32 + threadIdx.x, nb = gridDim.x;
    const int redo = flag[0];
    if (blockIdx.x == 0 && tid == 0) flag[1] = redo;
    if (!redo) return;
    namespace cg = cooperative_groups;
    const cg::grid_group grid = cg::this_grid();
    const int gx = (P.nx + 32 * W - 1) / (32 * W);
    const long long blocks = (long long)gx * P.ny * P.nz;
    for (long long b = blockIdx.x; b < blocks; b += nb) {
        const long long r = b / gx;
        fbar_block<double, double>(f_in, fb, P, tid, int(b - r * gx), 32 * W, int(r % P.ny), int(r / P.ny));
    }
    grid.sync();
    const long long ghosts = fb_ghosts(P.nx, P.ny, P.nz);
    for (long long q = (long long)blockIdx.x * (32 * W) + tid; q < ghosts; q += (long long)nb * (32 * W))
        fb_ghost_cell(fb, P, q);
    grid.sync();
    if (blockIdx.x == 0 && tid == 0) flag[0] = 0;
    const int tx = (P.nx + 31) / 32, ty = (P.ny + W - 2) / (W - 1);
    constexpr int kc = 8;
    const long long tiles = (long long)tx * ty * ((P.nz + kc - 1) / kc);
    for (long long b = blockIdx.x; b < tiles; b += nb) {
        const long long r = b / tx;
        flux_block<double, double, W, 0, false, FbReadCoherent<double, double>>(
            fb, f_in, f_out, P, kc, int(b - r * tx), int(r % ty), int(r / ty));
        __syncthreads();  // the next tile reuses the shared flux rows
    }
}

// f-bar-plus as the FP64 kernels store it (interior cells)
__global__ void fx_decode_kernel(const i64 *__restrict__ fb, double *__restrict__ dst, const FxParams P,
                                 const StepParams<double, double> D)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
    if (i >= P.nx) return;
    const i64 *src = fb + ((long long)k * P.ny + j) * P.rs + fx_col(i);
    double *q = dst + ((long long)(k + 1) * (P.ny + 2) + (j + 1)) * D.pitch_b + i + 1;
    for (int p = 0; p < NPOP; ++p) q[p * D.ps_b] = fx_to_double(src[p * 16]);
}

constexpr int REDO_W = 8, REDO_MINB = 2;

// The flux kernel has tiles of four rows (128 registers, no spills) and of seven (80, 24
// warps per SM, fewer rows formed twice).  A plane of a seven-row tile takes 1.65 times one
// of four rows (7.8 against 4.7 us), and beginning a z chunk costs about 1.5 planes (two
// rounds of the z warps, part of one of the others).  Rows and chunk count are those whose
// waves of CTAs take the least time: 256 x 128 x 128 channel 1.01 ms with seven rows, 1.06
// with four; 64 x 32 x 32 channel, whole step, 43 and 37 us; 64^3 box 107 and 104 us.
struct FxTiling {
    int rows, chunks;
};
FxTiling flux_fx_tiling(int nx, int ny, int nz, int slots)
{
    FxTiling best{4, 1};
    double least = 1e300;
    for (int rows : {4, 7}) {
        const long long tiles = (long long)((nx + 31) / 32) * ((ny + rows - 1) / rows);
        for (int c = 1; c <= nz; ++c) {
            const double cost = double((tiles * c + slots - 1) / slots) * ((nz + c - 1) / c + 1.5) * (rows == 7 ? 1.65 : 1.0);
            if (cost < least) {
                least = cost;
                best = FxTiling{rows, c};
            }
        }
    }
    return best;
}

template <int FAX, int R>
cudaError_t allow_smem()
{
    return cudaFuncSetAttribute(flux_fx_kernel<R, FAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(FxSmem<R>::bytes));
}

template <int FAX>
cudaError_t setup(FxPlan &L, int sms)
{
    const FxTiling t = flux_fx_tiling(L.P.nx, L.P.ny, L.P.nz, sms);  // one CTA per SM
    L.flux_rows = t.rows;
    L.flux_chunks = t.chunks;
    return t.rows == 4 ? allow_smem<FAX, 4>() : allow_smem<FAX, 7>();
}

template <int FAX>
cudaError_t stage_a(const FxPlan &L, const double *f_in, i64 *fb, int *flag, cudaStream_t st)
{
    const FxParams &P = L.P;
    const int xoff = P.nx % 32 == 1 ? 1 : 0;
    const int bx = P.nx + xoff >= 128 ? 128 : ((P.nx + xoff + 31) / 32) * 32;
    fbar_fx_kernel<FAX><<<dim3((P.nx + xoff + bx - 1) / bx, P.ny, P.nz), bx, 0, st>>>(f_in, fb, P, xoff, flag);
    return cudaGetLastError();
}

template <int FAX, int R>
cudaError_t flux_rows(const FxPlan &L, const i64 *fb, const double *f_in, double *f_out, int *flag, cudaStream_t st)
{
    const FxParams &P = L.P;
    const dim3 grid((P.nx + 31) / 32, (P.ny + R - 1) / R, L.flux_chunks);
    flux_fx_kernel<R, FAX><<<grid, dim3(32, 3 * R + 3), FxSmem<R>::bytes, st>>>(fb, f_in, f_out, P, flag);
    return cudaGetLastError();
}

template <int FAX>
cudaError_t flux(const FxPlan &L, const i64 *fb, const double *f_in, double *f_out, int *flag, cudaStream_t st)
{
    return L.flux_rows == 4 ? flux_rows<FAX, 4>(L, fb, f_in, f_out, flag, st)
                            : flux_rows<FAX, 7>(L, fb, f_in, f_out, flag, st);
}

}  // namespace

cudaError_t fixed_plan_setup(FxPlan &L)
{
    const int sms = device_sms();
    cudaError_t e = L.fax == 0 ? setup<0>(L, sms) : L.fax == 1 ? setup<1>(L, sms) : L.fax == 2 ? setup<2>(L, sms) : setup<3>(L, sms);
    int occ = 1;
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fp64_redo_kernel<REDO_W, REDO_MINB>, 32 * REDO_W, 0);
    L.redo_blocks = sms * std::max(occ, 1);
    return e;
}

cudaError_t launch_fixed_a(const FxPlan &L, const double *f_in, void *fb, int *flag, cudaStream_t st)
{
    i64 *b = static_cast<i64 *>(fb);
    return L.fax == 0   ? stage_a<0>(L, f_in, b, flag, st)
           : L.fax == 1 ? stage_a<1>(L, f_in, b, flag, st)
           : L.fax == 2 ? stage_a<2>(L, f_in, b, flag, st)
                        : stage_a<3>(L, f_in, b, flag, st);
}

cudaError_t launch_fixed_flux(const FxPlan &L, const double *f_in, double *f_out, void *fb, int *flag, cudaStream_t st)
{
    const i64 *b = static_cast<const i64 *>(fb);
    const cudaError_t e = L.fax == 0   ? flux<0>(L, b, f_in, f_out, flag, st)
                          : L.fax == 1 ? flux<1>(L, b, f_in, f_out, flag, st)
                          : L.fax == 2 ? flux<2>(L, b, f_in, f_out, flag, st)
                                       : flux<3>(L, b, f_in, f_out, flag, st);
    if (e != cudaSuccess) return e;
    double *fbd = static_cast<double *>(fb);
    void *args[] = {const_cast<const double **>(&f_in), &f_out, &fbd, const_cast<StepParams<double, double> *>(&L.D), &flag};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(fp64_redo_kernel<REDO_W, REDO_MINB>),
                                       dim3(L.redo_blocks), dim3(32, REDO_W), args, 0, st);
}

cudaError_t launch_fixed_decode(const FxPlan &L, const void *fb, double *dst, cudaStream_t st)
{
    const int nx = L.P.nx, ny = L.P.ny, nz = L.P.nz;
    fx_decode_kernel<<<dim3((nx + 127) / 128, ny, nz), 128, 0, st>>>(static_cast<const i64 *>(fb), dst, L.P, L.D);
    const long long g = fb_ghosts(nx, ny, nz);
    fb_ghost_kernel<double, double><<<unsigned((g + 255) / 256), 256, 0, st>>>(dst, L.D);
    return cudaGetLastError();
}

}  // namespace dg
