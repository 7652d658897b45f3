// Launchers of the fixed-point FP64 step (fixed_kernels.cuh) and of the FP64
// kernel that redoes a step whose state left its range.
#include "fixed_launch.cuh"
#include "launch_impl.cuh"

namespace dg {
namespace {

constexpr int REDO_W = TileCfg<double, double>::W, REDO_MINB = TileCfg<double, double>::MINB;

// Stages (b)-(e) in FP64 of a step out of range, whose f-bar-plus the flux kernel has formed
// in FP64: the tiles of flux_kernel, each CTA every gridDim.x-th.  Run behind every
// fixed-point flux kernel, it returns at once after a step in range.  (An ordinary launch: a
// step needs no more of the GPU than is free.)  A step out of range takes, with all three
// kernels, 237 us on 64 x 32 x 32 cells, 683 us on 64^3 and 6.76 ms on 256 x 128 x 128, against
// 221, 635 and 6.63 with the FP64 kernels alone; as one cooperative launch with grid-wide
// barriers it took 749, 840 and 7.02.
__global__ void __launch_bounds__(32 * REDO_W, REDO_MINB)
    fp64_redo_kernel(const double *__restrict__ fb, const double *f_in, double *f_out, const StepParams<double, double> P,
                     int kc, int *words)
{
    const int tid = threadIdx.y * 32 + threadIdx.x;
    if (!fx_in_fp64(words)) {
        if (blockIdx.x == 0 && tid == 0) words[FXW_FIXED] = 1;
        return;
    }
    __syncthreads();
    // the last CTA to have read the flag lowers it
    if (tid == 0 && atomicAdd(words + FXW_DONE, 1) == int(gridDim.x) - 1) {
        words[FXW_FLAG] = 0;
        words[FXW_FIXED] = 0;
        words[FXW_DONE] = 0;
    }
    const int tx = (P.nx + 31) / 32, ty = (P.ny + REDO_W - 2) / (REDO_W - 1);
    const long long tiles = (long long)tx * ty * ((P.nz + kc - 1) / kc);
    for (long long b = blockIdx.x; b < tiles; b += gridDim.x) {
        const long long r = b / tx;
        flux_block<double, double, REDO_W, 0, false>(fb, f_in, f_out, P, kc, int(b - r * tx), int(r % ty), int(r / ty));
        __syncthreads();  // the next tile reuses the shared flux rows
    }
}

// f-bar-plus as the FP64 kernels store it, a block per row: the cells, the two ghost columns
// and their periodic images
__global__ void __launch_bounds__(128) fx_decode_kernel(const i64 *__restrict__ copy, double *__restrict__ dst,
                                                        const FxParams P, const StepParams<double, double> D,
                                                        const int *words)
{
    if (!words[FXW_FIXED]) return;
    const int j = blockIdx.x, k = blockIdx.y, ny = P.ny, nz = P.nz;
    const i64 *row = copy + ((long long)k * ny + j) * P.rs;
    for (int c = threadIdx.x; c < P.nx + 2; c += blockDim.x) {
        const int I = c == P.nx + 1 ? 0 : c + 1;  // the lower ghost is the last column there, the first here
        const i64 *src = row + fx_col(c);
        fb_images(j, k, ny, nz, [&](int J, int K) {
            double *q = dst + ((long long)K * (ny + 2) + J) * D.pitch_b + I;
            for (int p = 0; p < NPOP; ++p) q[p * D.ps_b] = fx_to_double(src[p * 16]);
        });
    }
}
__global__ void fx_shown_kernel(int *words)
{
    words[FXW_FIXED] = 0;
    words[FXW_SHOWN] = 1;
}

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
cudaError_t stage_a(const FxPlan &L, const double *f_in, i64 *fb, int *words, cudaStream_t st)
{
    const FxParams &P = L.P;
    const int xoff = P.nx % 32 == 1 ? 1 : 0;
    const int bx = P.nx + xoff >= 128 ? 128 : ((P.nx + xoff + 31) / 32) * 32;
    fbar_fx_kernel<FAX><<<dim3((P.nx + xoff + bx - 1) / bx, P.ny, P.nz), bx, 0, st>>>(f_in, fb, P, xoff, words);
    return cudaGetLastError();
}

template <int FAX, int R>
cudaError_t flux_rows(const FxPlan &L, i64 *fb, const double *f_in, double *f_out, int *words, cudaStream_t st)
{
    const FxParams &P = L.P;
    const dim3 grid((P.nx + 31) / 32, (P.ny + R - 1) / R, L.flux_chunks);
    flux_fx_kernel<R, FAX><<<grid, dim3(32, 3 * R + 3), FxSmem<R>::bytes, st>>>(fb, f_in, f_out, P, words);
    return cudaGetLastError();
}

template <int FAX>
cudaError_t flux(const FxPlan &L, i64 *fb, const double *f_in, double *f_out, int *words, cudaStream_t st)
{
    return L.flux_rows == 4 ? flux_rows<FAX, 4>(L, fb, f_in, f_out, words, st)
                            : flux_rows<FAX, 7>(L, fb, f_in, f_out, words, st);
}

}  // namespace

cudaError_t fixed_plan_setup(FxPlan &L)
{
    const int sms = device_sms();
    cudaError_t e = L.fax == 0 ? setup<0>(L, sms) : L.fax == 1 ? setup<1>(L, sms) : L.fax == 2 ? setup<2>(L, sms) : setup<3>(L, sms);
    int occ = 1;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fp64_redo_kernel, 32 * REDO_W, 0);
    const long long cols = (long long)((L.P.nx + 31) / 32) * ((L.P.ny + REDO_W - 2) / (REDO_W - 1));
    const long long slots = (long long)sms * std::max(occ, 1);
    L.redo_kchunk = choose_kchunk(L.P.nz, cols, slots);
    L.redo_blocks = int(std::min(slots, cols * ((L.P.nz + L.redo_kchunk - 1) / L.redo_kchunk)));
    return e;
}

cudaError_t launch_fixed_a(const FxPlan &L, const double *f_in, void *fb, int *words, cudaStream_t st)
{
    i64 *b = static_cast<i64 *>(fb);
    return L.fax == 0   ? stage_a<0>(L, f_in, b, words, st)
           : L.fax == 1 ? stage_a<1>(L, f_in, b, words, st)
           : L.fax == 2 ? stage_a<2>(L, f_in, b, words, st)
                        : stage_a<3>(L, f_in, b, words, st);
}

cudaError_t launch_fixed_flux(const FxPlan &L, const double *f_in, double *f_out, void *fb, int *words, cudaStream_t st)
{
    i64 *b = static_cast<i64 *>(fb);
    const cudaError_t e = L.fax == 0   ? flux<0>(L, b, f_in, f_out, words, st)
                          : L.fax == 1 ? flux<1>(L, b, f_in, f_out, words, st)
                          : L.fax == 2 ? flux<2>(L, b, f_in, f_out, words, st)
                                       : flux<3>(L, b, f_in, f_out, words, st);
    if (e != cudaSuccess) return e;
    fp64_redo_kernel<<<L.redo_blocks, dim3(32, REDO_W), 0, st>>>(static_cast<const double *>(fb), f_in, f_out, L.D,
                                                                 L.redo_kchunk, words);
    return cudaGetLastError();
}

cudaError_t launch_fixed_decode(const FxPlan &L, const void *copy, void *fb, int *words, cudaStream_t st)
{
    fx_decode_kernel<<<dim3(L.P.ny, L.P.nz), 128, 0, st>>>(static_cast<const i64 *>(copy), static_cast<double *>(fb), L.P,
                                                           L.D, words);
    fx_shown_kernel<<<1, 1, 0, st>>>(words);
    return cudaGetLastError();
}

}  // namespace dg
