// ragged_pipe.cu -- the transforms of one size, n = 2^16 .. 2^18, of a packed
// ragged batch: the pipelined column and row passes (tiles_pipe.cuh) with the
// transforms' starts read from a table.
//
// HBM-bound like the passes of a uniform batch: 512-point columns and rows of
// 512 or 256 points (2^16: 256 x 256), tiles of 16 columns (rows), 32 points a
// thread, two passes and one exchange where the 4096-point tiles of the
// persistent ragged kernel (16 points a thread) take three and two.  GB300,
// us an exec of 2^26 points of one size, persistent kernel / these passes:
// 2^16 417 / 365, 2^17 448 / 350, 2^18 490 / 359; 10000 transforms of
// 2^6 .. 2^18, forward and inverse, 5400 / 4210 (the rest unchanged).
#include <algorithm>

#include "internal.h"
#include "plan.h"
#include "tiles_pipe.cuh"
#include "tiles_registry.h"

namespace gfft {

using c32 = cpx<float>;

namespace {
constexpr int C = RAGGED_PIPE_C, E = 32;
// log2 of the column length of n = 2^logn (C2CCore::init's split)
constexpr int log_a(int logn) { return logn == 16 ? 8 : 9; }
// groups (and stages) a CTA: 512 threads
constexpr int groups(int logl) { return logl == 8 ? 4 : 2; }

template <int L, bool INV>
const void *col_fn()
{
    return (const void *)&pipe::k_colpass_tma<float, L, C, E, groups(L), groups(L), INV, 3, false, true>;
}
template <int L, bool INV>
const void *row_fn()
{
    return (const void *)&pipe::k_rowpass_tma<float, L, C, E, groups(L), groups(L), INV, true>;
}
template <int L, int LD>
using Cfg = PipeCfg<float, L, C, E, groups(L), groups(L), LD>;
static_assert(Cfg<8, LAND_COL>::THREADS == 512 && Cfg<9, LAND_COL>::THREADS == 512, "one CTA an SM");
static_assert(2 * Cfg<8, LAND_COL>::SMEM > 228 * 1024 && 2 * Cfg<9, LAND_COL>::SMEM > 228 * 1024 &&
                  2 * Cfg<8, LAND_ROW>::SMEM > 228 * 1024 && 2 * Cfg<9, LAND_ROW>::SMEM > 228 * 1024,
              "one CTA an SM");

// copies run ahead of a tile's stores only while the passes stay in L2
// (C2CCore::run)
unsigned late(int logn, long long count) { return (count << (logn + 3)) > (200LL << 20) && log_a(logn) <= 9; }
}  // namespace

RaggedPipeTables ragged_pipe_tables(int logn)
{
    const int la = log_a(logn), lb = logn - la;
    const TileKernel *kc = tile_find(GFFT_F32, TILE_COL_TWP, la, C), *kr = tile_find(GFFT_F32, TILE_ROW_PIPE, lb, C);
    if (!kc || !kr || kc->e != E || kr->e != E) fail(GFFT_ERR_UNSUPPORTED, "no pipelined tiles for ragged batches");
    RaggedPipeTables tb;
    tb.col = tile_table(GFFT_F32, kc, la, C);
    tb.row = tile_table(GFFT_F32, kr, lb, C);
    t12_tables(GFFT_F32, logn, kc, &tb.t1, &tb.t2);
    return tb;
}

cudaError_t launch_ragged_col(int logn, int inverse, const void *in, long long total, void *ws, const long long *off,
                              long long count, const RaggedPipeTables &tb, cudaStream_t st)
{
    const int la = log_a(logn);
    const void *fn = la == 8 ? (inverse ? col_fn<8, true>() : col_fn<8, false>())
                             : (inverse ? col_fn<9, true>() : col_fn<9, false>());
    const size_t smem = la == 8 ? Cfg<8, LAND_COL>::SMEM : Cfg<9, LAND_COL>::SMEM;
    cudaError_t e = ensure_smem(fn, smem);
    if (e != cudaSuccess) return e;
    long long B = 1LL << (logn - la), odist = 1LL << logn;
    // the packed input as rows of B elements (the last one may be short: no
    // tile reaches past its own transform)
    const unsigned long long rows = (unsigned long long)((total + B - 1) / B);
    CUtensorMap map;
    const int boxr = la == 8 ? Cfg<8, LAND_COL>::BOXR : Cfg<9, LAND_COL>::BOXR;
    if (!make_tensor_map_3d(&map, in, (unsigned long long)B, rows, 1, (unsigned long long)B * sizeof(c32),
                            rows * (unsigned long long)B * sizeof(c32), C, (unsigned)boxr))
        return cudaErrorInvalidValue;
    unsigned *err = device_error_word();
    float scale = 1.f;
    int skew = 0;
    unsigned lt = late(logn, count);
    const long long grid = std::min<long long>(B / C * count, sm_count());
    void *args[] = {(void *)&map, (void *)&ws, (void *)&B, (void *)&B, (void *)&odist, (void *)&count,
                    (void *)&tb.col, (void *)&tb.t1, (void *)&tb.t2, (void *)&skew, (void *)&lt, (void *)&err,
                    (void *)&scale, (void *)&map, (void *)&off};
    return launch_pdl(fn, dim3((unsigned)grid), dim3(512), args, smem, st);
}

cudaError_t launch_ragged_row(int logn, int inverse, const void *ws, void *out, const long long *off, long long count,
                              const RaggedPipeTables &tb, cudaStream_t st)
{
    const int la = log_a(logn), lb = logn - la;
    const void *fn = lb == 8 ? (inverse ? row_fn<8, true>() : row_fn<8, false>())
                             : (inverse ? row_fn<9, true>() : row_fn<9, false>());
    const size_t smem = lb == 8 ? Cfg<8, LAND_ROW>::SMEM : Cfg<9, LAND_ROW>::SMEM;
    cudaError_t e = ensure_smem(fn, smem);
    if (e != cudaSuccess) return e;
    long long A = 1LL << la, B = 1LL << lb, N = 1LL << logn;
    unsigned *err = device_error_word();
    float scale = 1.f;
    unsigned lt = late(logn, count);
    const long long grid = std::min<long long>(A / C * count, sm_count());
    void *args[] = {(void *)&ws, (void *)&out, (void *)&A, (void *)&B, (void *)&A, (void *)&N, (void *)&N,
                    (void *)&count, (void *)&tb.row, (void *)&err, (void *)&scale, (void *)&lt, (void *)&off};
    return launch_pdl(fn, dim3((unsigned)grid), dim3(512), args, smem, st);
}

}  // namespace gfft
