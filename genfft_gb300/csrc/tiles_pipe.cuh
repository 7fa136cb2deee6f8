// tiles_pipe.cuh -- persistent tile kernels for fp32 columns and rows of
// 2^9 .. 2^12 points with 32 or 64 points a thread: two Stockham passes and
// one shared-memory exchange where 16 points a thread need three and two.
//
// A CTA (one per SM) holds NG thread groups and NB >= NG shared-memory stages.
// A group works on a tile of C columns (rows) by itself, on its own named
// barriers; tile i of the CTA goes to group i mod NG and stage i mod NB.  A
// tile's TMA copy lands in its stage, the exchange runs in place there, and
// once the group has read its last exchange values one thread starts the copy
// of tile i + NB into the stage.  So one group's butterflies and stores
// overlap the others' and the copies in flight, and a barrier never stops the
// whole SM.  The four-step passes take a stage a group, the column FFTs of the
// 2D and column transforms, whose data is in L2 more often, one more (GB300,
// us, with / without it: 2^10 columns 5000 16.6 / 19.8; C2C 2^20 x 128
// 794 / 733, 2^19 x 128 389 / 355: more copies in flight than HBM serves well).
//
// What bounds them (GB300; 6683 GB/s is the copy rate; GB/s of one pass over
// a 1 GB batch in a kernel probe):
//   columns  512 x 16 (2 groups of 256)            6094   HBM
//           1024 x  8 (2 groups of 256)            5563   HBM, 64-byte runs
//           2048 x  8 (1 group of 256, 64 points)  5674   issue, 8 warps
//           4096 x  4 (1 group of 256, 64 points)  4655   32-byte runs
//   rows     512 x 16  6312, 1024 x 8  6139, 2048 x 8  5998
// With 32 points a thread a 2048 x 8 tile takes three passes and 512
// threads: 4417 (columns) and 5252 (rows).  A whole stage beside a
// half-size exchange buffer (re and im in turn) frees the stage a pass
// earlier but doubles the barriers: 3801 and 3928.  Column copies by
// cp.async instead of TMA: 0.95x with 16-byte, 0.62 - 0.75x with 8-byte
// pieces.
//
// C2C through two such passes, GB300, GB/s forward, against the paths before
// (persistent four-step 2^17 .. 2^19, 16-point tiles 2^20, three passes of
// short tiles 2^21 .. 2^24), 1 GB batches:
//   2^17 3157 / 2385   2^18 3189 / 2103   2^19 3024 / 1951   2^20 2931 / 2110
//   2^21 2925 / 2098   2^22 2851 / 2071   2^23 2788 / 2003   2^24 2651 / 1916
// and one transform: 2^17 8.9 us / 16.2, 2^20 11.4 / 20.6, 2^24 115 / 146.
//
// Inter-pass twiddle W_N^(f k), k = t + q G, f the column (TWM 3):
// W_N^(f t) * W_N^(G f q) from two tables of directly
// rounded roots, t1[f][t] (G a row) and t2[f][q] (E a row).  A thread loads
// one t1 value a tile and the group stages the E x C t2 values it needs,
// where the hi / lo split costs two scattered loads a point.  (Indexed by the
// products f t and f q the tables are as small, but every load is a sector of
// its own: a third of the column pass's L2 reads.)
#pragma once

#include "tiles_tma.cuh"

namespace gfft {

// named barriers of a thread group (ids 1 .. 15; 0 is __syncthreads)
__device__ __forceinline__ void bar_group(int id, int nthreads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ void bar_group_arrive(int id, int nthreads)
{
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
// bar_group returning the AND of the group's predicates
__device__ __forceinline__ bool bar_group_and(int id, int nthreads, bool pred)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.red.and.pred q, %3, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)pred), "r"(nthreads), "r"(id)
        : "memory");
    return r != 0;
}

// how a tile lands: columns whose rows all start on 16-byte boundaries,
// columns whose rows may not, rows
enum PipeLand { LAND_COL = 0, LAND_COLU = 1, LAND_ROW = 2 };

template <typename T, int LOGL, int C, int E_, int NG_, int NB_, int LD>
struct PipeCfg {
    using SP = StockhamPlan<T, LOGL, E_>;
    static constexpr int N = SP::N, NG = NG_, NB = NB_;
    static constexpr int GT = SP::G * C;        // threads of a group
    static constexpr int THREADS = GT * NG;
    // Exchange layout: column s at s * PITCH, element i at i + i / R0.  A
    // half-warp holds C columns (8 rows of a 16-row tile) by 16 / C values of
    // t; with PITCH = 16 / C (mod 16) its reads (stride 1 in t) and its
    // writes after the first pass (stride R0 + 1 in t) fall on different
    // banks, where padding every 16 elements makes the writes of 32- and
    // 64-point first passes collide two and four ways.  (16 columns: one t a
    // half-warp, only the pitch matters.)
    static constexpr int CB = LD == LAND_ROW && C > 8 ? 8 : C;
    __host__ __device__ static constexpr int padded(int i) { return CB == 16 ? i : i + (i >> ilog2c(SP::R0)); }
    static constexpr int PITCH = (padded(N) + 15) / 16 * 16 + 16 / CB;
    // pitch of the rows a row tile lands on: a multiple of 16 bytes (bulk
    // copies), 16 / CB banks apart
    static constexpr int RP = N + 16 / CB;
    // LAND_COLU: an 8-byte element may sit in the second half of its 16-byte
    // granule, so a row's box is one granule wider than C
    static constexpr int BW = LD == LAND_COLU ? C + 2 : C;
    static constexpr int LAND = LD == LAND_ROW ? RP * C : N * BW;
    static constexpr int STAGE = StageRound<T, cmax<PITCH * C, LAND>::value>::value;
    static constexpr int T2 = LD == LAND_COL ? C * SP::E : 0;  // staged t2 values of a group's tile (two buffers)
    // rows per tensor box (LAND_COLU: of the even or the odd rows)
    static constexpr int BOXR = N < 256 ? N : 256;
    static constexpr size_t BAR_OFF = ((size_t)NB * STAGE + (size_t)NG * 2 * T2 + SP::TW) * sizeof(cpx<T>);
    static constexpr size_t SMEM = BAR_OFF + 128;  // + barriers and sequence numbers
    static_assert(SMEM <= 227 * 1024, "stages and tables must fit one CTA");
    static_assert(GT % 32 == 0 && 1 + 2 * NG <= 16 && NB >= NG && NB * 12 <= 128, "whole warps, barrier ids, barrier words");
};

// Stage hand-over.  An mbarrier's parity names two phases, so a group may
// wait for tile i only once the copy of tile i has been armed: with NB > NG a
// stage goes from group to group, and a group that got there while the copy of
// tile i - NB was still in flight would take that phase's parity for its own.
// Whoever arms tile i's copy publishes i in seq[i mod NB] first thing after.
__device__ __forceinline__ void seq_publish(int *seq, int i)
{
    asm volatile("st.release.cta.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(seq)), "r"(i) : "memory");
}
__device__ __forceinline__ int seq_read(const int *seq)
{
    int v;
    asm volatile("ld.acquire.cta.shared::cta.b32 %0, [%1];" : "=r"(v) : "r"(smem_u32(seq)) : "memory");
    return v;
}
// wait (bounded) until tile i's copy is armed and has landed; the warp leaves
// it converged
__device__ __forceinline__ bool stage_wait(uint64_t *full, const int *seq, int i, uint32_t parity)
{
    bool ok = true;
    if (seq_read(seq) != i) {
        const unsigned long long t0 = global_ns();
        while (ok && seq_read(seq) != i) ok = global_ns() - t0 <= TMA_WAIT_NS;
    }
    if (ok) ok = mbar_wait(full, parity);
    __syncwarp();
    return ok;
}

// The loop the passes share: tile i of the CTA is tile w0 + i step of the
// launch.  issue(i) starts its copy (one thread; nothing past the last tile),
// body(i, stage, parity) transforms and stores it, starts the copy of tile
// i + NB and returns false when its own did not land in time.
template <typename Cfg, typename Issue, typename Body>
__device__ __forceinline__ void pipe_loop(uint64_t *full, const int *seq, unsigned *err, int w0, int step, int total,
                                          Issue issue, Body body)
{
    constexpr int NB = Cfg::NB, NG = Cfg::NG;
    const int grp = threadIdx.x / Cfg::GT;
    if (threadIdx.x == 0)
        for (int i = 0; i < NB; i++) issue(i);
    for (int i = grp; w0 + i * step < total; i += NG) {
        const int buf = i % NB;
        if (body(i, buf, (uint32_t)((i / NB) & 1))) continue;
        // timed out: report, let the copies in flight land (bounded), leave
        if (threadIdx.x == grp * Cfg::GT) {
            atomicOr(err, DEV_ERR_TMA_TIMEOUT);
            for (int j = i; j < i + NB && w0 + j * step < total; j++)
                if (seq_read(&seq[j % NB]) == j) mbar_wait(&full[j % NB], (uint32_t)((j / NB) & 1));
        }
        break;
    }
}

// 8-byte asynchronous copy global -> shared, and the wait for this thread's
__device__ __forceinline__ void cp_async8(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Frees a stage once the whole group has read it and starts the next copy
// into it.  Every warp calls stage_read after its last read; the issuing warp
// calls stage_refill, the only one to wait for the others, right after it or
// (`late`, see C2CCore::run) once its own stores are out.
__device__ __forceinline__ void stage_read(int bar, int nthreads, int tid)
{
    if (tid >= 32) bar_group_arrive(bar, nthreads);
}
template <typename Issue>
__device__ __forceinline__ void stage_refill(int bar, int nthreads, int tid, bool landed, int next, Issue issue)
{
    if (tid >= 32) return;
    bar_group(bar, nthreads);
    if (tid == 0 && landed) {
        fence_proxy_async_smem();
        issue(next);
    }
    __syncwarp();
}

namespace pipe {

// Column pass: see k_colpass (tiles.cuh); the tensor map views the input as
// [batch][rows][ncols] 8-byte elements.
// U: row starts that alternate between 16-byte boundaries and the 8 bytes
// after them (an odd row stride, as the W/2 + 1 bins of a real image's
// half spectrum have).  TMA wants 16-byte strides and starts, so the even
// rows come through `map` and the odd rows through `map1`, each of twice the
// row stride and rounded down to a boundary; bit r of `skew` says that the
// rows of parity r start 8 bytes in.  They land in two blocks of boxes one
// granule wider than the tile.  (GB300, us: 5001 columns of 2^10 points 21.3
// against 29.5 for 16-point tiles of plain loads, of 2^11 51.8 / 69.3; an
// even count takes 16.6 and 38.4.)
// AT: transform b starts at element off[b] of the packed input, a multiple of
// C, which the tensor map views as rows of ncols elements (a power of two); a
// tile then lies in rows that start off[b] / ncols down and never straddles
// two of them.
template <typename T, int LOGL, int C, int E_, int NG, int NB, bool INV, int TWM, bool U = false, bool AT = false>
__global__ void __launch_bounds__(PipeCfg<T, LOGL, C, E_, NG, NB, U ? LAND_COLU : LAND_COL>::THREADS, 1)
    k_colpass_tma(const __grid_constant__ CUtensorMap map, cpx<T> *__restrict__ out, long long ncols, long long ld_out,
              long long odist, long long nbatch, const cpx<T> *__restrict__ tw, const cpx<T> *__restrict__ t1,
              const cpx<T> *__restrict__ t2, int skew, unsigned late, unsigned *err, T scale,
              const __grid_constant__ CUtensorMap map1, const long long *__restrict__ off = nullptr)
{
    using Cfg = PipeCfg<T, LOGL, C, E_, NG, NB, U ? LAND_COLU : LAND_COL>;
    static_assert(!U || (TWM == 0 && !AT), "plain columns");
    using SP = typename Cfg::SP;
    static_assert(sizeof(cpx<T>) == 8 && (TWM == 0 || TWM == 3), "fp32; no twiddle, or from t1 / t2");
    constexpr int E = SP::E, G = SP::G, N = SP::N, GT = Cfg::GT;
    constexpr int W2 = TWM != 0 ? (Cfg::T2 + GT - 1) / GT : 1;  // t2 values a thread stages
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    cpx<T> *const stage0 = reinterpret_cast<cpx<T> *>(smem_raw);
    cpx<T> *const tws = stage0 + (size_t)NB * Cfg::STAGE;
    uint64_t *const full = reinterpret_cast<uint64_t *>(smem_raw + Cfg::BAR_OFF);
    int *const seq = reinterpret_cast<int *>(full + NB);
    const int grp = threadIdx.x / GT, tid = threadIdx.x - grp * GT;
    cpx<T> *const t2b = tws + SP::TW + grp * 2 * Cfg::T2;
    const int bar = 1 + 2 * grp;
    const int s = tid % C, t = tid / C;
    // (tiles of 4096 points and more: their count fits 31 bits, and 32-bit
    // divisions find a tile's place)
    const int tiles = (int)((ncols + C - 1) / C), total = tiles * (int)nbatch;
    const int w0 = blockIdx.x, step = gridDim.x;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NB; i++) {
            mbar_init(&full[i], 1);
            seq[i] = -1;
        }
        fence_barrier_init();
    }
    for (int i = threadIdx.x; i < SP::TW; i += Cfg::THREADS) tws[i] = ldg_c(tw + i);
    pdl_enter();  // launched by launch_pdl: waits for the previous kernel
    __syncthreads();

    // AT: the start of tile i's transform, read ahead of its copy
    auto start_of = [&](int i) {
        const int w = w0 + i * step;
        return w < total ? __ldg(off + (unsigned)w / (unsigned)tiles) : 0LL;
    };
    long long next_off = 0;
    auto issue = [&](int i) {
        const int w = w0 + i * step;
        if (w >= total) return;
        const int buf = i % NB;
        cpx<T> *const S = stage0 + (size_t)buf * Cfg::STAGE;
        const int b = (int)((unsigned)w / (unsigned)tiles), c0 = (w - b * tiles) * C;
        // out-of-range columns of the last tile are zero-filled and still counted
        mbar_arrive_expect_tx(&full[buf], (uint32_t)(N * Cfg::BW * sizeof(cpx<T>)));
        seq_publish(&seq[buf], i);
        if constexpr (U) {
            for (int r = 0; r < N / 2; r += Cfg::BOXR) {
                tensor_load_3d(S + r * Cfg::BW, &map, c0, r, b, &full[buf]);
                tensor_load_3d(S + (N / 2 + r) * Cfg::BW, &map1, c0, r, b, &full[buf]);
            }
        } else if constexpr (AT) {
            const long long at = (i < NB ? start_of(i) : next_off) + c0;
            const int y = (int)(at / ncols), x = (int)(at & (ncols - 1));
            for (int r = 0; r < N; r += Cfg::BOXR) tensor_load_3d(S + r * C, &map, x, y + r, 0, &full[buf]);
        } else {
            for (int r = 0; r < N; r += Cfg::BOXR) tensor_load_3d(S + r * C, &map, c0, r, b, &full[buf]);
        }
    };
    pipe_loop<Cfg>(full, seq, err, w0, step, total, issue, [&](int i, int buf, uint32_t par) {
        const int w = w0 + i * step;
        cpx<T> *const S = stage0 + (size_t)buf * Cfg::STAGE;
        const int wb = (int)((unsigned)w / (unsigned)tiles);
        const long long b = wb, col = (long long)(w - wb * tiles) * C + s;
        const bool active = col < ncols;
        // the tile's t2 values go to the group's two buffers in turn: slower warps of
        // the group may still read the other one for the tile before
        cpx<T> *const t2s = t2b + (i / NG & 1) * Cfg::T2;
        if constexpr (AT) next_off = start_of(i + NB);
        cpx<T> w1{(T)0, (T)0};
        if constexpr (TWM != 0) {
            const unsigned f = (unsigned)(active ? col : 0);
            w1 = ldg_c(t1 + f * (unsigned)G + t);
#pragma unroll
            for (int j = 0; j < W2; j++)
                if (W2 * GT == Cfg::T2 || tid + j * GT < Cfg::T2) cp_async8(t2s + tid + j * GT, t2 + f * (unsigned)E + (t + j * G));
        }
        const bool ok = stage_wait(&full[buf], &seq[buf], i, par);
        cpx<T> v[E];
#pragma unroll
        for (int q = 0; q < E; q++) {
            const int r = t + q * G;  // (G is even: its parity is t's)
            if constexpr (U) v[q] = S[((t & 1) * (N / 2) + (r >> 1)) * Cfg::BW + s + ((skew >> (t & 1)) & 1)];
            else v[q] = S[r * C + s];
        }
        bool landed = true;
        cpx<T> *const my = S + s * Cfg::PITCH;
        stockham_run<T, LOGL, E_, INV, TwShared>(
            v, t, [my](int k) -> cpx<T> & { return my[Cfg::padded(k)]; }, tws, [bar]() { bar_group(bar, GT); },
            [&]() {
                stage_read(bar + 1, GT, tid);
                if (!late) stage_refill(bar + 1, GT, tid, landed, i + NB, issue);
            },
            [&]() {
                // every thread of the group holds its inputs: the stage
                // takes the exchange
                if constexpr (TWM != 0) cp_async_wait();
                landed = bar_group_and(bar, GT, ok);
            });
        if (!landed) return false;
        if (active) {
            cpx<T> *dst = out + b * odist + col + (long long)t * ld_out;
            const long long st = (long long)G * ld_out;
#pragma unroll
            for (int q = 0; q < E; q++, dst += st) {
                if constexpr (TWM != 0) {
                    st_c(dst, twmul<INV>(v[q], cmul(w1, t2s[q * C + s])));
                    if ((q & 7) == 7) asm volatile("" ::: "memory");  // bounds the staged twiddles in registers
                } else {
                    st_c(dst, scl(v[q], scale));
                }
            }
        }
        if (late) stage_refill(bar + 1, GT, tid, landed, i + NB, issue);
        return true;
    });
}

// Row pass with transposed store: see k_rowpass (tiles.cuh).  The rows land
// RP apart and thread (s, t) holds points of row s, s fastest, so the
// outputs leave the registers in runs of C without a transpose.  AT: the
// output of transform b starts at element off[b].
template <typename T, int LOGL, int C, int E_, int NG, int NB, bool INV, bool AT = false>
__global__ void __launch_bounds__(PipeCfg<T, LOGL, C, E_, NG, NB, LAND_ROW>::THREADS, 1)
    k_rowpass_tma(const cpx<T> *__restrict__ in, cpx<T> *__restrict__ out, long long nrows, long long ld_in,
              long long ostride, long long idist, long long odist, long long nbatch, const cpx<T> *__restrict__ tw,
              unsigned *err, T scale, unsigned late, const long long *__restrict__ off = nullptr)
{
    using Cfg = PipeCfg<T, LOGL, C, E_, NG, NB, LAND_ROW>;
    using SP = typename Cfg::SP;
    constexpr int E = SP::E, G = SP::G, N = SP::N, GT = Cfg::GT;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    cpx<T> *const stage0 = reinterpret_cast<cpx<T> *>(smem_raw);
    cpx<T> *const tws = stage0 + (size_t)NB * Cfg::STAGE;
    uint64_t *const full = reinterpret_cast<uint64_t *>(smem_raw + Cfg::BAR_OFF);
    int *const seq = reinterpret_cast<int *>(full + NB);
    const int grp = threadIdx.x / GT, tid = threadIdx.x - grp * GT;
    const int bar = 1 + 2 * grp;
    // a half-warp takes at most 8 rows (Cfg::CB) and 16 / CB values of t
    const int s = C <= 8 ? tid % C : (tid & 7) + (tid >> 4 & 1) * 8;
    const int t = C <= 8 ? tid / C : (tid >> 5) * 2 + (tid >> 3 & 1);
    static_assert(C <= 8 || C == 16, "row mapping");
    const int tiles = (int)((nrows + C - 1) / C), total = tiles * (int)nbatch;
    const int w0 = blockIdx.x, step = gridDim.x;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NB; i++) {
            mbar_init(&full[i], 1);
            seq[i] = -1;
        }
        fence_barrier_init();
    }
    for (int i = threadIdx.x; i < SP::TW; i += Cfg::THREADS) tws[i] = ldg_c(tw + i);
    pdl_enter();  // launched by launch_pdl: waits for the previous kernel
    __syncthreads();

    auto issue = [&](int i) {
        const int w = w0 + i * step;
        if (w >= total) return;
        const int buf = i % NB;
        cpx<T> *const S = stage0 + (size_t)buf * Cfg::STAGE;
        const int b = (int)((unsigned)w / (unsigned)tiles), row0 = (w - b * tiles) * C;
        const int rows = (int)(nrows - row0 < C ? nrows - row0 : C);
        mbar_arrive_expect_tx(&full[buf], (uint32_t)(rows * N * sizeof(cpx<T>)));
        seq_publish(&seq[buf], i);
        const cpx<T> *src = in + (long long)b * idist + (long long)row0 * ld_in;
        for (int r = 0; r < rows; r++)
            bulk_load(S + r * Cfg::RP, src + r * ld_in, N * sizeof(cpx<T>), &full[buf]);
    };
    pipe_loop<Cfg>(full, seq, err, w0, step, total, issue, [&](int i, int buf, uint32_t par) {
        const int w = w0 + i * step;
        cpx<T> *const S = stage0 + (size_t)buf * Cfg::STAGE;
        const int wb = (int)((unsigned)w / (unsigned)tiles);
        const long long b = wb, row = (long long)(w - wb * tiles) * C + s;
        long long start;
        if constexpr (AT) start = __ldg(off + b);
        else start = b * odist;
        const bool ok = stage_wait(&full[buf], &seq[buf], i, par);
        cpx<T> v[E];
#pragma unroll
        for (int q = 0; q < E; q++) v[q] = S[s * Cfg::RP + t + q * G];
        bool landed = true;
        cpx<T> *const my = S + s * Cfg::PITCH;
        stockham_run<T, LOGL, E_, INV, TwShared>(
            v, t, [my](int k) -> cpx<T> & { return my[Cfg::padded(k)]; }, tws, [bar]() { bar_group(bar, GT); },
            [&]() {
                stage_read(bar + 1, GT, tid);
                if (!late) stage_refill(bar + 1, GT, tid, landed, i + NB, issue);
            },
            [&]() { landed = bar_group_and(bar, GT, ok); });
        if (!landed) return false;
        if (row < nrows) {
            cpx<T> *dst = out + start + row + (long long)t * ostride;
            const long long st = (long long)G * ostride;
#pragma unroll
            for (int q = 0; q < E; q++, dst += st) stcs_c(dst, scl(v[q], scale));
        }
        if (late) stage_refill(bar + 1, GT, tid, landed, i + NB, issue);
        return true;
    });
}

}  // namespace pipe
}  // namespace gfft
