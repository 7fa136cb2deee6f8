// real_pipe.cu -- fp32 real-input transforms and half-spectrum inverses of
// n = 2^18 .. 2^22 on the pipelined tiles (tiles_pipe.cuh), with the
// real-FFT adjustment inside the pass that touches the spectrum
// (RealFFT<T>::forward, FFTReal.h:186-221).
//
// H = n/2 = A B complex points, k = k1 + A k2 (spectrum), B a + b (input):
//   forward   column pass over A (TILE_COL_TWP), then k_rowdit_pipe over
//             rows of B = 512: a tile holds 8 rows k1 and their mirrors
//             A - k1, whose bins k and H - k the adjustment (dit.cuh) pairs;
//   inverse   k_c2rcol_pipe over columns of A = 512: a tile holds 8 columns
//             b and their mirrors B - b, forms Z'_k from F_k and F_(H-k)
//             (c2r.cu) as it reads them from the stage, and goes on as a
//             column pass; then the row pass (TILE_ROW_PIPE) over B.
// Row (column) 0 is its own mirror and has a tile of its own.
//
// The adjustment's twiddle t_k = i W_n^k needs one table value a thread: the
// thread's 32 points are n / 64 apart in k, so the rest are its products
// with the constants W_64^q, where one table load a bin read as many bytes
// from L2 as the spectrum itself.
//
// HBM-bound: each pass reads and writes the H points once.  GB300, GB/s of one
// read and one write of the reals, against the 16-point passes before (column
// tiles + row pass with the DIT; pre-pass + C2C of n/2):
//            forward                     inverse
//   2^18     x 64      2488 / 1896       2276 / 1454
//   2^20     x 64      2370 / 1712       2534 / 1483
//   2^20     x 1       10.1 us / 19.2    11.2 us / 24.6
// Its partial 64-byte runs (the half spectrum has H + 1 bins, so every other
// transform starts 8 bytes off a boundary) cost 1.4x the L2 write sectors.
#include <algorithm>

#include "dit.cuh"
#include "internal.h"
#include "plan.h"
#include "tiles_pipe.cuh"
#include "twiddle.h"

namespace gfft {

using c32 = cpx<float>;

namespace {
constexpr int RL = 9;       // log2 of the row (forward) / column (inverse) length
constexpr int RC = 16;      // rows (columns) a tile: 8 and their mirrors
constexpr int RE = 32;      // points a thread
}  // namespace

// ---------------------------------------------------------------------------
// forward: row pass with the adjustment

struct RowDitPipeCfg : PipeCfg<float, RL, RC, RE, 2, 2, LAND_ROW> {
    using Base = PipeCfg<float, RL, RC, RE, 2, 2, LAND_ROW>;
    static constexpr size_t Z0_OFF = Base::BAR_OFF + 128;  // row 0 of each group's tile
    static constexpr size_t SMEM = Z0_OFF + (size_t)NG * N * sizeof(c32);
    static_assert(SMEM <= 227 * 1024, "fits one CTA");
};

// in: the column pass's output, rows of 512; out: H + 1 bins a transform.
// TMA false (GFFT_NO_TMA): each thread loads its own points.
template <bool TMA>
__global__ void __launch_bounds__(RowDitPipeCfg::THREADS, 1)
    k_rowdit_pipe(const c32 *__restrict__ in, c32 *__restrict__ out, int A, long long idist, long long odist,
                  int nbatch, const c32 *__restrict__ tw, const c32 *__restrict__ dtw, unsigned *err, float scale)
{
    using Cfg = RowDitPipeCfg;
    using SP = Cfg::SP;
    constexpr int E = SP::E, G = SP::G, N = SP::N, GT = Cfg::GT, NG = Cfg::NG, NB = Cfg::NB;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    c32 *const stage0 = reinterpret_cast<c32 *>(smem_raw);
    c32 *const tws = stage0 + (size_t)NB * Cfg::STAGE;
    uint64_t *const full = reinterpret_cast<uint64_t *>(smem_raw + Cfg::BAR_OFF);
    int *const seq = reinterpret_cast<int *>(full + NB);
    const int grp = threadIdx.x / GT, tid = threadIdx.x - grp * GT;
    c32 *const z0 = reinterpret_cast<c32 *>(smem_raw + Cfg::Z0_OFF) + grp * N;
    const int bar = 1 + 2 * grp;
    // slot s: rows 1 + 8 p + s (s < 8) and their mirrors; t and its mirror
    // G - 1 - t sit 8 lanes apart, so a bin's partner is lane ^ 24
    const int s = (tid & 7) + (tid >> 4 & 1) * 8;
    const int t = tid >> 3 & 1 ? G - 1 - (tid >> 5) : tid >> 5;
    const int P = A / RC;  // pair tiles a transform; tile P is row 0's
    const int tiles = P + 1, total = tiles * nbatch;
    const int w0 = blockIdx.x, step = gridDim.x;
    const long long H = (long long)A * N;
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
        if (!TMA || w >= total) return;
        const int buf = i % NB;
        c32 *const S = stage0 + (size_t)buf * Cfg::STAGE;
        const int b = (int)((unsigned)w / (unsigned)tiles), p = w - b * tiles;
        const int rows = p < P ? RC : 1;
        const c32 *src = in + (long long)b * idist;
        mbar_arrive_expect_tx(&full[buf], (uint32_t)(rows * N * sizeof(c32)));
        seq_publish(&seq[buf], i);
        for (int r = 0; r < rows; r++) {
            const int k1 = p == P ? 0 : r < 8 ? 1 + 8 * p + r : A - 1 - 8 * p - (r - 8);
            bulk_load(S + r * Cfg::RP, src + (long long)k1 * N, N * sizeof(c32), &full[buf]);
        }
    };
    pipe_loop<Cfg>(full, seq, err, w0, step, total, issue, [&](int i, int buf, uint32_t par) {
        const int w = w0 + i * step;
        c32 *const S = stage0 + (size_t)buf * Cfg::STAGE;
        const int b = (int)((unsigned)w / (unsigned)tiles), p = w - b * tiles;
        const bool row0 = p == P;
        const int k1 = row0 ? 0 : s < 8 ? 1 + 8 * p + s : A - 1 - 8 * p - (s - 8);
        // t_k of this thread's point 0 (bins k1 + A (t + G q))
        const c32 t0 = ldg_c(dtw + k1 + (long long)A * t);
        const bool ok = TMA ? stage_wait(&full[buf], &seq[buf], i, par) : true;
        const bool active = !row0 || s == 0;
        c32 v[E];
        if constexpr (TMA) {
#pragma unroll
            for (int q = 0; q < E; q++) v[q] = active ? S[s * Cfg::RP + t + q * G] : c32{0.f, 0.f};
        } else {
            const c32 *const row = in + (long long)b * idist + (long long)k1 * N;
#pragma unroll
            for (int q = 0; q < E; q++) v[q] = active ? ldcg_c(row + t + q * G) : c32{0.f, 0.f};
        }
        bool landed = true;
        c32 *const my = S + s * Cfg::PITCH;
        stockham_run<float, RL, RE, false, TwShared>(
            v, t, [my](int k) -> c32 & { return my[Cfg::padded(k)]; }, tws, [bar]() { bar_group(bar, GT); },
            [&]() {
                if constexpr (TMA) {
                    stage_read(bar + 1, GT, tid);
                    stage_refill(bar + 1, GT, tid, landed, i + NB, issue);
                }
            },
            [&]() { landed = bar_group_and(bar, GT, ok); });
        if (!landed) return false;
        c32 *const dst = out + (long long)b * odist;
        if (!row0) {
            // bin k = k1 + A (t + G q), q < E/2, with the partner's point
            // E - 1 - q: both bins of the pair are this thread's
            const long long k0 = k1 + (long long)A * t;
            c32 *lo = dst + k0, *hi = dst + (H - k0);
            const long long st = (long long)A * G;
            static_for<0, E / 2>([&](auto qc) {
                constexpr int q = decltype(qc)::value;
                const c32 mine = v[E - 1 - q];
                const c32 zj{__shfl_xor_sync(0xffffffffu, mine.x, 24), __shfl_xor_sync(0xffffffffu, mine.y, 24)};
                const c32 tk = rot64<q, false, float>(t0);
                st_c(lo + q * st, scl(dit_value(v[q], zj, tk), scale));
                st_c(hi - q * st, scl(dit_value(zj, v[q], c32{tk.x, -tk.y}), scale));
            });
        } else {
            // row 0: bins A k2 and A (N - k2), k2 = 0 .. N/2 (k2 = 0 also
            // gives the Nyquist bin H), through shared memory
            if (s == 0) {
#pragma unroll
                for (int q = 0; q < E; q++) z0[t + q * G] = v[q];
            }
            bar_group(bar, GT);
            for (int k2 = tid; k2 <= N / 2; k2 += GT) {
                const long long k = (long long)A * k2, j = H - k;
                const c32 zk = z0[k2], zj = z0[(N - k2) & (N - 1)];
                st_c(dst + k, scl(dit_value(zk, zj, ldg_c(dtw + k)), scale));
                st_c(dst + j, scl(dit_value(zj, zk, ldg_c(dtw + j)), scale));
            }
            bar_group(bar, GT);  // z0 is free again
        }
        return true;
    });
}

// ---------------------------------------------------------------------------
// inverse: column pass that forms Z' from the half spectrum

// columns land in two blocks (the 8 columns and their mirrors) of boxes one
// 16-byte granule wider than 8: columns 1 + 8 p start off a boundary
constexpr int CBW = 10;
struct C2RColCfg : PipeCfg<float, RL, RC, RE, 2, 2, LAND_ROW> {
    using Base = PipeCfg<float, RL, RC, RE, 2, 2, LAND_ROW>;
    static constexpr int STAGE = StageRound<float, cmax<PITCH * RC, N * 2 * CBW>::value>::value;
    static constexpr int T2 = RC * SP::E;
    static constexpr size_t BAR_OFF = ((size_t)NB * STAGE + (size_t)NG * 2 * T2 + SP::TW) * sizeof(c32);
    static constexpr size_t SMEM = BAR_OFF + 128;
    static_assert(SMEM <= 227 * 1024, "fits one CTA");
};

// Z'_k from bins k and H - k weighted by f, 1 or 1/2 (c2r.cu).  The weight
// comes first, in the adds' multiply-adds: the sum of two bins may overflow
// where that of their halves does not.
__device__ __forceinline__ c32 c2r_value(c32 fk, c32 fp, c32 tk, float f)
{
    const c32 h = scl(fp, f);
    const c32 sm{fma_(fk.x, f, h.x), fma_(fk.y, f, -h.y)};   // F_k + conj F_p
    const c32 df{fma_(-fk.x, f, h.x), fma_(-fk.y, f, -h.y)};  // conj F_p - F_k
    return sm + cmulc(df, tk);
}

// in: H + 1 bins a transform, H = 512 B (map / map1: the even / odd
// transforms as [512 rows][B], rounded down to 16 bytes; bit r of skew: those
// of parity r start 8 bytes in); out: the workspace, rows of B.
// interior = 0.5: the adjoint of the half-spectrum R2C halves every bin but
// F_0 and F_H.  TMA false (GFFT_NO_TMA, or no tensor map for this input): each
// thread loads its own bins.
template <bool TMA>
__global__ void __launch_bounds__(C2RColCfg::THREADS, 1)
    k_c2rcol_pipe(const __grid_constant__ CUtensorMap map, const __grid_constant__ CUtensorMap map1, int skew,
                  const c32 *__restrict__ in, long long idist, c32 *__restrict__ out, int B, int nbatch,
                  const c32 *__restrict__ tw, const c32 *__restrict__ t1, const c32 *__restrict__ t2,
                  const c32 *__restrict__ dtw, unsigned *err, float interior)
{
    using Cfg = C2RColCfg;
    using SP = Cfg::SP;
    constexpr int E = SP::E, G = SP::G, N = SP::N, GT = Cfg::GT, NG = Cfg::NG, NB = Cfg::NB;
    constexpr int W2 = Cfg::T2 / GT;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    c32 *const stage0 = reinterpret_cast<c32 *>(smem_raw);
    c32 *const tws = stage0 + (size_t)NB * Cfg::STAGE;
    uint64_t *const full = reinterpret_cast<uint64_t *>(smem_raw + Cfg::BAR_OFF);
    int *const seq = reinterpret_cast<int *>(full + NB);
    const int grp = threadIdx.x / GT, tid = threadIdx.x - grp * GT;
    c32 *const t2b = tws + SP::TW + grp * 2 * Cfg::T2;
    const int bar = 1 + 2 * grp;
    const int s = (tid & 7) + (tid >> 4 & 1) * 8;
    const int t = (tid >> 5) * 2 + (tid >> 3 & 1);
    const int P = B / RC;  // pair tiles a transform; tile P is column 0's
    const int tiles = P + 1, total = tiles * nbatch;
    const int w0 = blockIdx.x, step = gridDim.x;
    const long long H = (long long)B * N;
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

    // where columns 1 + 8 p .. (lo) and B - 8 - 8 p .. (hi) of transform b
    // start in their boxes: the box starts on an even element
    auto lo_x = [&](int b, int p) { return 1 + 8 * p + (skew >> (b & 1) & 1); };
    auto hi_x = [&](int b, int p) { return B - 8 - 8 * p + (skew >> (b & 1) & 1); };
    auto issue = [&](int i) {
        const int w = w0 + i * step;
        if (!TMA || w >= total) return;
        const int buf = i % NB;
        c32 *const S = stage0 + (size_t)buf * Cfg::STAGE;
        const int b = (int)((unsigned)w / (unsigned)tiles), p = w - b * tiles;
        if (p == P) {  // column 0: its threads load it themselves
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full[buf])) : "memory");
            seq_publish(&seq[buf], i);
            return;
        }
        mbar_arrive_expect_tx(&full[buf], (uint32_t)(N * 2 * CBW * sizeof(c32)));
        seq_publish(&seq[buf], i);
        const CUtensorMap *m = b & 1 ? &map1 : &map;
        for (int r = 0; r < N; r += Cfg::BOXR) {
            tensor_load_3d(S + r * CBW, m, lo_x(b, p) & ~1, r, b >> 1, &full[buf]);
            tensor_load_3d(S + (N + r) * CBW, m, hi_x(b, p) & ~1, r, b >> 1, &full[buf]);
        }
    };
    pipe_loop<Cfg>(full, seq, err, w0, step, total, issue, [&](int i, int buf, uint32_t par) {
        const int w = w0 + i * step;
        c32 *const S = stage0 + (size_t)buf * Cfg::STAGE;
        const int b = (int)((unsigned)w / (unsigned)tiles), p = w - b * tiles;
        const bool col0 = p == P;
        const int col = col0 ? 0 : s < 8 ? 1 + 8 * p + s : B - 1 - 8 * p - (s - 8);
        const bool active = !col0 || s == 0;
        // t_k of this thread's point 0 (bins B (t + G q) + col)
        const c32 t0 = ldg_c(dtw + (long long)B * t + col);
        const c32 w1 = ldg_c(t1 + col * G + t);
        // t2s[q * 16 + slot]: the values the group's thread of that slot uses
        c32 *const t2s = t2b + (i / NG & 1) * Cfg::T2;
#pragma unroll
        for (int j = 0; j < W2; j++) {
            const int idx = tid + j * GT, sl = idx % RC, q = idx / RC;
            const int cl = col0 ? 0 : sl < 8 ? 1 + 8 * p + sl : B - 1 - 8 * p - (sl - 8);
            cp_async8(t2s + idx, t2 + cl * E + q);
        }
        const bool ok = TMA ? stage_wait(&full[buf], &seq[buf], i, par) : true;
        c32 v[E];
        if (!col0) {
            // own column and its mirror: element a pairs with N - 1 - a
            const int lx = lo_x(b, p) & 1, hx = hi_x(b, p) & 1;
            const int own = s < 8 ? lx + s : N * CBW + hx + 7 - (s - 8);
            const int mir = s < 8 ? N * CBW + hx + 7 - s : lx + (s - 8);
            static_for<0, E>([&](auto qc) {
                constexpr int q = decltype(qc)::value;
                const int a = t + q * G;
                c32 fk, fp;
                if constexpr (TMA) {
                    fk = S[own + a * CBW];
                    fp = S[mir + (N - 1 - a) * CBW];
                } else {
                    const long long k = (long long)B * a + col;
                    fk = ldcg_c(in + (long long)b * idist + k);
                    fp = ldcg_c(in + (long long)b * idist + (H - k));
                }
                v[q] = c2r_value(fk, fp, rot64<q, false, float>(t0), interior);
            });
        } else if (active) {
            // (eight pairs of bins in flight a thread)
            const c32 *F = in + (long long)b * idist;
            constexpr int CH = 8;
#pragma unroll
            for (int q0 = 0; q0 < E; q0 += CH) {
                c32 fk[CH], fp[CH];
#pragma unroll
                for (int j = 0; j < CH; j++) {
                    const long long a = t + (q0 + j) * G;
                    fk[j] = ldcg_c(F + B * a);
                    fp[j] = ldcg_c(F + B * (N - a));
                }
#pragma unroll
                for (int j = 0; j < CH; j++) {
                    const int a = t + (q0 + j) * G;
                    if (a == 0) {  // F_0 and F_H count as real, and whole
                        fk[j].y = 0.f;
                        fp[j].y = 0.f;
                    }
                    v[q0 + j] = c2r_value(fk[j], fp[j], ldg_c(dtw + (long long)B * a), a == 0 ? 1.f : interior);
                }
            }
        } else {
#pragma unroll
            for (int q = 0; q < E; q++) v[q] = c32{0.f, 0.f};
        }
        bool landed = true;
        c32 *const my = S + s * Cfg::PITCH;
        stockham_run<float, RL, RE, true, TwShared>(
            v, t, [my](int k) -> c32 & { return my[Cfg::padded(k)]; }, tws, [bar]() { bar_group(bar, GT); },
            [&]() {
                if constexpr (TMA) {
                    stage_read(bar + 1, GT, tid);
                    stage_refill(bar + 1, GT, tid, landed, i + NB, issue);
                }
            },
            [&]() {
                cp_async_wait();
                landed = bar_group_and(bar, GT, ok);
            });
        if (!landed) return false;
        if (active) {
            c32 *dst = out + (long long)b * H + col + (long long)t * B;
            const long long st = (long long)G * B;
#pragma unroll
            for (int q = 0; q < E; q++, dst += st) {
                st_c(dst, twmul<true>(v[q], cmul(w1, t2s[q * RC + s])));
                if ((q & 7) == 7) asm volatile("" ::: "memory");
            }
        }
        return true;
    });
}

// ---------------------------------------------------------------------------
// host side

int realpipe_logl() { return RL; }
size_t realpipe_twiddle_count() { return RowDitPipeCfg::SP::TW; }
void realpipe_twiddle_fill(void *buf)
{
    stockham_fill_twiddles<float, RL, RE>(static_cast<c32 *>(buf), [](long long k, long long M, c32 *w) {
        forward_root<float>(k, M, &w->x, &w->y);
    });
}

cudaError_t launch_rowdit_pipe(const void *in, void *out, long long A, long long batch, long long idist,
                               long long odist, const void *tw, const void *dtw, cudaStream_t st, double scale)
{
    const void *fn = tma_enabled() ? (const void *)&k_rowdit_pipe<true> : (const void *)&k_rowdit_pipe<false>;
    cudaError_t e = ensure_smem(fn, RowDitPipeCfg::SMEM);
    if (e != cudaSuccess) return e;
    int a = (int)A, nb = (int)batch;
    float sc = (float)scale;
    unsigned *err = device_error_word();
    const long long grid = std::min<long long>((A / RC + 1) * batch, sm_count());
    void *args[] = {(void *)&in, (void *)&out, (void *)&a, (void *)&idist, (void *)&odist, (void *)&nb, (void *)&tw,
                    (void *)&dtw, (void *)&err, (void *)&sc};
    return launch_pdl(fn, dim3((unsigned)grid), dim3(RowDitPipeCfg::THREADS), args, RowDitPipeCfg::SMEM, st);
}

cudaError_t launch_c2rcol_pipe(const void *in, void *ws, long long B, long long batch, long long idist, const void *tw,
                               const void *t1, const void *t2, const void *dtw, bool half_interior, cudaStream_t st)
{
    CUtensorMap map[2] = {};
    int skew = 0;
    constexpr int N = C2RColCfg::N;
    bool tma = tensor_maps_enabled();
    for (int r = 0; r < 2 && tma; r++) {
        if (r == 1 && batch == 1) {
            map[1] = map[0];
            break;
        }
        const uintptr_t base = (uintptr_t)in + (uintptr_t)(r * idist) * sizeof(c32);
        const int off = (int)(base >> 3 & 1);
        skew |= off << r;
        tma = make_tensor_map_3d(&map[r], (const void *)(base & ~(uintptr_t)15), (unsigned long long)(B + off), N,
                                 (unsigned long long)((batch + 1 - r) / 2), (unsigned long long)B * sizeof(c32),
                                 (unsigned long long)(2 * idist) * sizeof(c32), CBW, C2RColCfg::BOXR);
    }
    const void *fn = tma ? (const void *)&k_c2rcol_pipe<true> : (const void *)&k_c2rcol_pipe<false>;
    cudaError_t e = ensure_smem(fn, C2RColCfg::SMEM);
    if (e != cudaSuccess) return e;
    int b = (int)B, nb = (int)batch;
    float interior = half_interior ? 0.5f : 1.0f;
    unsigned *err = device_error_word();
    const long long grid = std::min<long long>((B / RC + 1) * batch, sm_count());
    void *args[] = {(void *)&map[0], (void *)&map[1], (void *)&skew, (void *)&in, (void *)&idist, (void *)&ws,
                    (void *)&b, (void *)&nb, (void *)&tw, (void *)&t1, (void *)&t2, (void *)&dtw, (void *)&err,
                    (void *)&interior};
    return launch_pdl(fn, dim3((unsigned)grid), dim3(C2RColCfg::THREADS), args, C2RColCfg::SMEM, st);
}

}  // namespace gfft
