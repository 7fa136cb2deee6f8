// fused_tma.cu -- fp32 C2C, R2C and half-spectrum C2R whose complex length is
// 2^12 .. 2^14, dense and on 16-byte boundaries: the arithmetic of k_c2c_fused,
// k_r2c_fused and k_c2r_fused, bit for bit, in a persistent kernel that copies
// a group's next transform in while it stores this one and keeps the twiddles
// on chip.  (The same points a thread as the plain kernels, so that a
// transform's bits do not depend on how many others stand beside it, nor on
// whether it came from a host buffer, which goes through in chunks.)
//
// What bounded the plain kernels at 2^13 and 2^14 (32 points a thread) is the
// last pass: its table (31 / 32 of N values, 65 KB at 2^13, 129 KB at 2^14) is
// read once a transform through L1, which the exchange buffers leave no room,
// so a load a point goes to L2 and is waited for.  Thread t of a group needs
// the same 31 values for every transform (W_N^(t r)), more than its registers
// hold -- but a persistent CTA has 256 KB of tensor memory beside its registers
// and shared memory, which tcgen05.st fills once and tcgen05.ld reads back 16
// twiddles at a time.  The real transforms' adjustment twiddles (dit.cuh)
// lie beside them.  GB300, GB/s, C2C, 1 GB batches: 2^14 5430 - 5660 from run
// to run with tensor memory, 5110 without it, 3994 the plain kernel; 2^13 6120 -
// 6250 / 5044 / 4807.
// 64 points a thread: 4498 at 2^14, 4506 at 2^13.  Real transforms, n = 2^14 /
// 2^15, 512 MB - 1 GB: R2C 4896 / 4130 against 4032 / 3453, C2R 5293 / 4945
// against 3730 / 2982.
//
// At 2^12 (16 points a thread) all tables fit shared memory, beside the stages
// of three transforms (C2C, 80 registers a thread) or four (real, 64).  GB300,
// us, plain / three / four groups: C2C x 16384 169.7 / 159.6 / 172.7, x 4096
// 46.3 / 43.9 / 44.7; R2C x 16384 207.2 / 198.4 / 182.4; C2R 212.7 / 207.7 /
// 180.1.  With 32 points and tensor memory 165.8, 185.9 and 181.3, and the
// plain kernels are 7 - 20 % slower with 32.
//
// Replaces FFT<float>::transform<inv> (fft.h:80-85) and RealFFT<float>::forward
// (FFTReal.h:186-221) for these lengths.
#include <algorithm>
#include <cstdint>

#include "internal.h"
#include "tiles_registry.h"
#include "dit.cuh"
#include "stockham.cuh"
#include "tc.cuh"
#include "tiles_pipe.cuh"
#include "twiddle.h"

namespace gfft {

using c32 = cpx<float>;

enum FusedKind { FUSED_C2C = 0, FUSED_R2C = 1, FUSED_C2R = 2 };

// NG transforms at a time, a group of N / E threads and a stage each
template <int LOGN, int NG_, int KIND>
struct FusedTmaCfg {
    // TM: 32 points a thread, the last pass's and the adjustment's twiddles in
    // tensor memory; 2^12: the 16 points of the plain kernels, all twiddles in
    // shared memory
    static constexpr bool TM = LOGN > 12;
    using SP = StockhamPlan<float, LOGN, TM ? 32 : 16>;
    static constexpr int N = SP::N, E = SP::E, G = SP::G, NG = NG_, THREADS = G * NG;
    static constexpr int STAGE = (spad_size<float>(N) + 15) / 16 * 16;
    static constexpr int TWS = TM ? SP::twiddle_offset(SP::P - 1) : SP::TW;  // Stockham twiddles in shared memory
    static constexpr int DTS = TM || KIND == FUSED_C2C ? 0 : KIND == FUSED_R2C ? N / 2 : N;  // adjustment twiddles there
    // tensor memory: a warp reaches the 32 lanes of its number modulo 4, so
    // warps 4 apart stack their 2 E columns
    // (R2C adds 16 adjustment twiddles a thread, C2R 32)
    static constexpr int WCOLS = KIND == FUSED_C2C ? 2 * E : 4 * E;
    static constexpr int COLS = WCOLS * (THREADS / 128);
    static constexpr size_t BAR_OFF = ((size_t)NG * STAGE + (TWS + DTS + 1) / 2 * 2) * sizeof(c32);
    static constexpr size_t SMEM = BAR_OFF + 128;
    static constexpr int PIECE = 4096;  // elements a bulk copy
    static_assert(SP::P == 3 && (TM ? E == 32 && THREADS == 512 : THREADS <= 1024), "three passes");
    static_assert(!TM || (COLS <= 512 && (COLS & (COLS - 1)) == 0), "columns");
    static_assert(SMEM <= 227 * 1024 && 2 * SMEM > 228 * 1024,
                  "one CTA an SM: its tensor memory is never waited for by its own grid");
};

// 32 consecutive 32-bit columns of this thread's tensor-memory lane
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float (&r)[32])
{
    uint32_t u[32];
#pragma unroll
    for (int i = 0; i < 32; i++) u[i] = __float_as_uint(r[i]);
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};" ::"r"(u[0]),
        "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]), "r"(u[9]), "r"(u[10]),
        "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15]), "r"(u[16]), "r"(u[17]), "r"(u[18]), "r"(u[19]),
        "r"(u[20]), "r"(u[21]), "r"(u[22]), "r"(u[23]), "r"(u[24]), "r"(u[25]), "r"(u[26]), "r"(u[27]), "r"(u[28]),
        "r"(u[29]), "r"(u[30]), "r"(u[31]), "r"(taddr)
        : "memory");
}

// In: `batch` transforms idist elements apart (C2C, R2C: complex elements,
// even, from a 16-byte boundary; C2R: bins, from any).  Out: odist apart (R2C:
// bins; C2R: complex elements).  interior: the factor of bins 1 .. N - 1, 2
// for the adjoint of C2R (R2C), 1/2 for the adjoint of R2C (C2R), else 1.
// AT (C2C): transform w is at element off[w], even, of in and out instead.
template <int LOGN, int NG, int KIND, bool INV, bool AT = false>
__global__ void __launch_bounds__(FusedTmaCfg<LOGN, NG, KIND>::THREADS, 1)
    k_fused_tma(const c32 *__restrict__ in, c32 *__restrict__ out, int batch, long long idist, long long odist,
                const c32 *__restrict__ tw, const c32 *__restrict__ dtw, unsigned *err, float scale, float interior,
                const long long *__restrict__ off)
{
    using Cfg = FusedTmaCfg<LOGN, NG, KIND>;
    static_assert(!AT || KIND == FUSED_C2C, "packed transforms are C2C");
    using SP = typename Cfg::SP;
    constexpr int N = Cfg::N, E = Cfg::E, G = Cfg::G, R0 = SP::R0;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    c32 *const stage0 = reinterpret_cast<c32 *>(smem_raw);
    c32 *const tws = stage0 + (size_t)NG * Cfg::STAGE;
    uint64_t *const bars = reinterpret_cast<uint64_t *>(smem_raw + Cfg::BAR_OFF);
    uint32_t *const tmem_slot = reinterpret_cast<uint32_t *>(bars + NG);

    const int grp = threadIdx.x / G, t = threadIdx.x - grp * G;
    c32 *const S = stage0 + (size_t)grp * Cfg::STAGE;
    uint64_t *const full = bars + grp;
    const int bar = 1 + 2 * grp;
    const int first = blockIdx.x + grp * gridDim.x, step = NG * gridDim.x;
    if (t == 0) {
        mbar_init(full, 1);
        fence_barrier_init();
    }
    for (int i = threadIdx.x; i < Cfg::TWS; i += Cfg::THREADS) tws[i] = ldg_c(tw + i);
    const c32 *const dts = tws + Cfg::TWS;
    for (int i = threadIdx.x; i < Cfg::DTS; i += Cfg::THREADS) tws[Cfg::TWS + i] = ldg_c(dtw + i);
    // Tensor memory is taken only once every earlier grid is through (a CTA of
    // one that still had its own to allocate would wait for ours while we wait
    // for it), and later grids may come in only once it is taken.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // AT: where this transform and the next one start, read ahead of the copy
    auto start_of = [&](int w) { return w < batch ? __ldg(off + w) : 0LL; };
    long long at = 0, next_at = 0;
    if constexpr (AT) next_at = start_of(first);
    auto issue = [&](int w) {
        if (w >= batch) return;
        const c32 *src = in + (AT ? next_at : (long long)w * idist);
        if constexpr (KIND == FUSED_C2R) {
            // N + 1 bins and what shares their first and last 16 bytes
            const uintptr_t a = (uintptr_t)src & ~(uintptr_t)15, e = ((uintptr_t)(src + N + 1) + 15) & ~(uintptr_t)15;
            mbar_arrive_expect_tx(full, (uint32_t)(e - a));
            for (uint32_t o = 0; o < (uint32_t)(e - a); o += Cfg::PIECE * 8) {
                const uint32_t len = (uint32_t)(e - a) - o;
                bulk_load(reinterpret_cast<char *>(S) + o, reinterpret_cast<const char *>(a) + o,
                          len < Cfg::PIECE * 8 ? len : Cfg::PIECE * 8, full);
            }
        } else {
            mbar_arrive_expect_tx(full, (uint32_t)(N * sizeof(c32)));
            for (int r = 0; r < N; r += Cfg::PIECE) bulk_load(S + r, src + r, Cfg::PIECE * sizeof(c32), full);
        }
    };
    if (t == 0) issue(first);
    __syncwarp();
    if constexpr (Cfg::TM)
        if (threadIdx.x < 32) tc::tmem_alloc(tmem_slot, Cfg::COLS);
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    uint32_t tm = 0;
    if constexpr (Cfg::TM) {
        tc::fence_after_sync();
        const int warp = threadIdx.x >> 5;
        tm = *tmem_slot + ((uint32_t)(warp & 3) << 21) + (uint32_t)(warp >> 2) * Cfg::WCOLS;
        // this thread's last-pass twiddles W_N^(t r) (r = 0: 1, not used),
        // then the adjustment twiddles of bins t + q G
        const c32 *const twl = tw + Cfg::TWS + t;
        constexpr int CH = KIND == FUSED_C2C ? 2 : KIND == FUSED_R2C ? 3 : 4;
#pragma unroll
        for (int c = 0; c < CH; c++) {
            float r[32];
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const int q = (c * 16 + j) % E;
                const c32 w = c >= 2 ? ldg_c(dtw + t + q * G) : q == 0 ? c32{1.f, 0.f} : ldg_c(twl + (q - 1) * G);
                r[2 * j] = w.x;
                r[2 * j + 1] = w.y;
            }
            tmem_st32(tm + c * 32, r);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }

    uint32_t par = 0;
    for (int w = first; w < batch; w += step, par ^= 1) {
        if constexpr (AT) {
            at = next_at;
            next_at = start_of(w + step);
        }
        const bool ok = mbar_wait(full, par);
        __syncwarp();
        c32 v[E];
        if constexpr (KIND == FUSED_C2R) {
            // Z'_k from bins k and N - k (c2r.cu)
            const c32 *const F = S + ((uintptr_t)(in + (long long)w * idist) >> 3 & 1);
#pragma unroll
            for (int c = 0; c < E / 16; c++) {
                float r[32];
                if constexpr (Cfg::TM) tc::tmem_ld32(tm + (2 + c) * 32, r);
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const int q = c * 16 + j, k = t + q * G;
                    const c32 tk = Cfg::TM ? c32{r[2 * j], r[2 * j + 1]} : dts[k];
                    c32 fk = F[k], fp = F[N - k];
                    if (q == 0 && t == 0) {  // bins 0 and N count as real, and whole
                        fk.y = 0.f;
                        fp.y = 0.f;
                    } else {
                        fk = scl(fk, interior);
                        fp = scl(fp, interior);
                    }
                    const c32 sm{fk.x + fp.x, fk.y - fp.y}, df{fp.x - fk.x, -fp.y - fk.y};
                    const c32 m = cmul(c32{tk.x, -tk.y}, df);
                    v[q] = {sm.x + m.x, sm.y + m.y};
                }
            }
        } else {
#pragma unroll
            for (int q = 0; q < E; q++) v[q] = S[t + q * G];
        }
        if (!bar_group_and(bar, G, ok)) {
            if (t == 0) {
                atomicOr(err, DEV_ERR_TMA_TIMEOUT);
                mbar_wait(full, par);  // let the copy in flight land (bounded)
            }
            break;
        }
        // pass 0: radix R0
#pragma unroll
        for (int m = 0; m < E / R0; m++) {
            c32 u[R0];
#pragma unroll
            for (int r = 0; r < R0; r++) u[r] = v[m + r * (E / R0)];
            dft<R0, INV, float>(u);
#pragma unroll
            for (int r = 0; r < R0; r++) S[spad<float>((t + m * G) * R0 + r)] = u[r];
        }
        // pass 1: radix E, twiddles from shared memory
        bar_group(bar, G);
#pragma unroll
        for (int q = 0; q < E; q++) v[q] = S[spad<float>(t + q * G)];
        {
            const c32 *const twp = tws + t % R0;
#pragma unroll
            for (int r = 1; r < E; r++) v[r] = twmul<INV>(v[r], twp[(r - 1) * R0]);
            dft<E, INV, float>(v);
            bar_group(bar, G);
            const int base = (t / R0) * R0 * E + t % R0;
#pragma unroll
            for (int r = 0; r < E; r++) S[spad<float>(base + r * R0)] = v[r];
        }
        // pass 2: radix E, twiddles from tensor memory (2^12: from shared)
        bar_group(bar, G);
#pragma unroll
        for (int q = 0; q < E; q++) v[q] = S[spad<float>(t + q * G)];
        if constexpr (KIND != FUSED_R2C) {
            stage_read(bar + 1, G, t);
            stage_refill(bar + 1, G, t, true, w + step, issue);
        }
        if constexpr (Cfg::TM) {
#pragma unroll
            for (int c = 0; c < E / 16; c++) {
                float r[32];
                tc::tmem_ld32(tm + c * 32, r);
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (c * 16 + j > 0) v[c * 16 + j] = twmul<INV>(v[c * 16 + j], c32{r[2 * j], r[2 * j + 1]});
            }
        } else {
            const c32 *const twp = tws + SP::twiddle_offset(SP::P - 1) + t;
#pragma unroll
            for (int r = 1; r < E; r++) v[r] = twmul<INV>(v[r], twp[(r - 1) * G]);
        }
        dft<E, INV, float>(v);
        c32 *const dst = out + (AT ? at : (long long)w * odist);
        if constexpr (KIND != FUSED_R2C) {
#pragma unroll
            for (int q = 0; q < E; q++) stcs_c(dst + t + q * G, scl(v[q], scale));
        } else {
            // bins k = t + q G, q < E/2, and N - k: the partner's values are
            // the upper half of thread G - t, through the stage (thread 0's
            // are its own, N / 2 its own partner)
            bar_group(bar, G);
#pragma unroll
            for (int q = E / 2; q < E; q++) S[spad<float>(t + (q - E / 2) * G)] = v[q];
            bar_group(bar, G);
            c32 z[E / 2];
#pragma unroll
            for (int q = 0; q < E / 2; q++) {
                const int j = N - (t + q * G);
                z[q] = q == 0 && t == 0 ? v[0] : S[spad<float>(j - N / 2 - (q == 0 && t == 0 ? N / 2 : 0))];
            }
            stage_read(bar + 1, G, t);
            stage_refill(bar + 1, G, t, true, w + step, issue);
            float r[32];
            if constexpr (Cfg::TM) tc::tmem_ld32(tm + 2 * 32, r);
            const float wt = scale * interior;
#pragma unroll
            for (int q = 0; q < E / 2; q++) {
                const int k = t + q * G;
                const c32 tk = Cfg::TM ? c32{r[2 * q], r[2 * q + 1]} : dts[k];
                const bool ends = q == 0 && t == 0;  // bins 0 and N
                const float f = ends ? scale : wt;
                stcs_c(dst + k, scl(dit_value(v[q], z[q], tk), f));
                stcs_c(dst + (N - k), scl(dit_value(z[q], v[q], c32{tk.x, -tk.y}), f));
            }
            if (t == 0) stcs_c(dst + N / 2, scl(dit_value(v[E / 2], v[E / 2], ldg_c(dtw + N / 2)), wt));
        }
    }
    if constexpr (Cfg::TM) {
        tc::fence_before_sync();
        __syncthreads();
        if (threadIdx.x < 32) tc::tmem_dealloc(*tmem_slot, Cfg::COLS);
    }
}

namespace {
struct Entry {
    const void *fn[6];  // C2C forward and inverse, R2C, C2R, packed C2C forward and inverse
    int groups[3], threads[3];  // by kind
    size_t smem[3];
};
// (packed: 2^13 and 2^14 only, see ragged.cu)
template <int LOGN, int NG, bool INV>
const void *packed_fn()
{
    if constexpr (LOGN > 12) return (const void *)&k_fused_tma<LOGN, NG, FUSED_C2C, INV, true>;
    else return nullptr;
}
// NG groups for C2C, NGR for the real transforms
template <int LOGN, int NG, int NGR>
Entry make_entry()
{
    using C = FusedTmaCfg<LOGN, NG, FUSED_C2C>;
    using R = FusedTmaCfg<LOGN, NGR, FUSED_R2C>;
    using I = FusedTmaCfg<LOGN, NGR, FUSED_C2R>;
    return Entry{{(const void *)&k_fused_tma<LOGN, NG, FUSED_C2C, false>, (const void *)&k_fused_tma<LOGN, NG, FUSED_C2C, true>,
                  (const void *)&k_fused_tma<LOGN, NGR, FUSED_R2C, false>, (const void *)&k_fused_tma<LOGN, NGR, FUSED_C2R, true>,
                  packed_fn<LOGN, NG, false>(), packed_fn<LOGN, NG, true>()},
                 {NG, NGR, NGR},
                 {C::THREADS, R::THREADS, I::THREADS},
                 {C::SMEM, R::SMEM, I::SMEM}};
}
const Entry &entry(int logn)
{
    static const Entry tab[3] = {make_entry<12, 3, 4>(), make_entry<13, 2, 2>(), make_entry<14, 1, 1>()};
    return tab[logn - FUSED_TMA_MIN];
}

cudaError_t launch(int logn, int kind, int fn_i, const void *in, void *out, long long nbatch, long long idist,
                   long long odist, const void *tw, const void *dtw, double sc, float interior, cudaStream_t st,
                   const long long *off = nullptr)
{
    const Entry &e = entry(logn);
    const void *fn = e.fn[fn_i];
    cudaError_t r = ensure_smem(fn, e.smem[kind]);
    if (r != cudaSuccess) return r;
    int batch = (int)nbatch;
    unsigned *err = device_error_word();
    float scale = (float)sc;
    const long long grid = std::min<long long>((nbatch + e.groups[kind] - 1) / e.groups[kind], sm_count());
    void *args[] = {(void *)&in, (void *)&out, (void *)&batch, (void *)&idist, (void *)&odist, (void *)&tw,
                    (void *)&dtw, (void *)&err, (void *)&scale, (void *)&interior, (void *)&off};
    return launch_pdl(fn, dim3((unsigned)grid), dim3(e.threads[kind]), args, e.smem[kind], st);
}
}  // namespace

size_t fused_tma_twiddle_count(int logn)
{
    return logn == 12 ? (size_t)StockhamPlan<float, 12, 16>::TW
         : logn == 13 ? (size_t)StockhamPlan<float, 13, 32>::TW : (size_t)StockhamPlan<float, 14, 32>::TW;
}
template <int L>
static void fill(void *buf)
{
    stockham_fill_twiddles<float, L, (L > 12 ? 32 : 16)>(static_cast<c32 *>(buf), [](long long k, long long M, c32 *w) {
        forward_root<float>(k, M, &w->x, &w->y);
    });
}
void fused_tma_twiddle_fill(int logn, void *buf) { (logn == 12 ? fill<12> : logn == 13 ? fill<13> : fill<14>)(buf); }

// The persistent kernels pay for filling their tables once a CTA and want
// transforms to reuse them: more than one wave of the SMs at 2^14, three at
// 2^13, four (C2C) or two (real) at 2^12.  GB300, us, plain / persistent: C2C
// 2^14 x 152 12.9 / 13.2, x 304 24.2 / 22.7; 2^13 x 608 21.4 / 21.7, x 1000
// 33.9 / 32.7; 2^12 x 1217 14.3 / 14.5, x 2000 24.6 / 23.8; R2C of 2^14 reals
// x 1000 39.9 / 39.7, x 1501 55.5 / 50.9; of 2^13 x 608 9.0 / 9.9, x 1217
// 17.5 / 17.1, x 2000 29.7 / 27.8; C2R of 2^13 x 1217 18.3 / 18.1, x 2000
// 32.5 / 28.7.
bool fused_tma_takes(int logn, bool real, long long batch)
{
    if (logn < FUSED_TMA_MIN || logn > FUSED_TMA_MAX || batch >= (1LL << 30) || !tma_enabled()) return false;
    const int waves = logn == 14 ? 1 : logn == 13 ? 3 : real ? 2 : 4;
    return batch > waves * entry(logn).groups[real ? FUSED_R2C : FUSED_C2C] * (long long)sm_count();
}

cudaError_t launch_fused_tma_c2c(int logn, int inverse, const FusedC2CArgs &a, cudaStream_t st)
{
    return launch(logn, FUSED_C2C, inverse ? 1 : 0, a.in, a.out, a.batch, a.idist, a.odist, a.tw_tma, nullptr, a.scale,
                  1.f, st);
}
cudaError_t launch_fused_tma_at(int logn, int inverse, const void *in, void *out, const long long *off, long long count,
                                const void *tw, cudaStream_t st)
{
    return launch(logn, FUSED_C2C, inverse ? 5 : 4, in, out, count, 0, 0, tw, nullptr, 1.0, 1.f, st, off);
}
cudaError_t launch_fused_tma_r2c(int logh, bool x2, const void *in, void *out, long long batch, long long idist,
                                 long long odist, const void *tw, const void *dtw, cudaStream_t st, double scale)
{
    return launch(logh, FUSED_R2C, 2, in, out, batch, idist, odist, tw, dtw, scale, x2 ? 2.f : 1.f, st);
}
cudaError_t launch_fused_tma_c2r(int logh, bool half, const void *in, void *out, long long batch, long long idist,
                                 long long odist, const void *tw, const void *dtw, cudaStream_t st, double scale)
{
    return launch(logh, FUSED_C2R, 3, in, out, batch, idist, odist, tw, dtw, scale, half ? 0.5f : 1.f, st);
}

}  // namespace gfft
