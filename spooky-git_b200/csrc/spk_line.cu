// spk_line.cu -- strided-axis FFT pass between pass buffers (y inverse, y
// forward, x forward), on the warp-owned transforms of spk_line.cuh.
//
// The pass moves each element once in and once out, so its floor is HBM; as
// the CTA-wide k_axis2 it was bound by latency instead (four CTA barriers a
// tile, 16 warps, 38-43% of issue slots, 51-69% of the copy bandwidth).
// Here a tile of 128-byte rows is loaded by TMA (swizzled) and transformed in
// place by the warps that own its columns: no exchange buffer, 24 warps per
// SM (16 for the FP64 lengths 3 2^k), one barrier of the tile's warps per tile.  The inverse, which writes
// every row, stores the tile by TMA; the forward passes, which write the kept
// rows, copy them out in 16-byte pieces (TMA boxes of the kept rows measured
// 0.149 ms at 256^3 FP32, the copy 0.141).  Loads take the rows and columns
// the pass needs (the kept ky rows of a trimmed inverse, kz < kz_keep).
// Measured, k_axis2 -> here (MHD; y inverse, y forward, x forward, ms):
//   256^3 FP64  0.241 0.257 0.180 -> 0.178 0.244 0.167
//   256^3 FP32  0.130 0.134 0.095 -> 0.104 0.144 0.096
//   128^3 FP32  0.029 0.027 0.021 -> 0.021 0.019 0.015
//   64^3  FP32  0.012 0.011 0.011 -> 0.009 0.008 0.008
// At 256^3 both directions wait for memory (long-scoreboard stalls of the
// tile waits, 4.5-4.9 TB/s moved, 51-55% of issue slots).  The FP32 forward
// passes of 256 points gain nothing by themselves, but the step is no slower
// with them (four steps 10.286 ms, 10.287 with k_axis2's) and other lengths
// are faster (192^3 5.82 ms against 6.11): one rule for all.  Refilling a stage before the next tile's
// wait, more tiles of fewer warps, and L2 promotion of 64 to 256 bytes
// measured no better.
//
// Warps form groups of W (the warps of one tile); each group runs its own
// ring of nst tiles, loaded by its first thread.  A stage is loaded again once
// its rows are out.  Every wait is bounded: a group whose wait ran out stops
// touching its tiles, still meets its barriers, and the pass ends with
// DevScalars.err = 2.
#include "spk_line.cuh"
#include "spk_ring.cuh"

namespace spk {

// Rows [row, row + n * rows) of a tile as n TMA boxes of `rows` rows through
// map `m` (n = 0: nothing).
struct LineSeg { int row, rows, n, map; };

struct LineJob { int ch_in, ch_out, deriv; };   // channels of the input and output maps; deriv 1: times i k

struct LineArgs {
    alignas(64) CUtensorMap map[4];   // the input in boxes of all rows, of the kept prefix and suffix; the output
    DevGrid g;
    FftPlan plan;
    int axis, kcols, nb, njobs, nst;
    int in_box_ch, out_box_ch;
    int outer_filter, trim, tr_always, tr_nouter, tr_nkb;
    const int* tr_outer;
    FastDiv fd_job, fd_box, fd_kb, tr_fd_job, tr_fd_box, tr_fd_kb;
    double scale;
    const DevScalars* gate;
    int gate_stage;
    int* err;
    const DevScalars* scs;
    LineSeg in[2];          // every row (in[1] unused)
    LineSeg in_trim[2];     // the rows that can be nonzero when the box has no masked content
    int out_rows;           // inverse: rows of an output box
    int out_pre, out_suf;   // forward: the rows to store, [0, out_pre) and [out_suf, N)
    void* out;
    LineJob job[SPK_MAXJOBS];
};

template <typename T, int N> struct LineCfg {
    using G = Line<T, N, 128>;
    static constexpr int WARPS = G::W > 8 ? G::W : 8;
    static constexpr int NG = WARPS / G::W;            // groups (tiles in work) of a CTA, at most
    // CTAs per SM: three at 80 registers; the FP64 3 2^k transforms (12
    // elements a lane) would spill there
    static constexpr int MINB = WARPS > 8 ? 1 : (sizeof(T) == 8 && !RegFft<T, N>::P2 ? 2 : 3);
};

template <typename T, int N, int DIR>
__global__ void __launch_bounds__(LineCfg<T, N>::WARPS * 32, LineCfg<T, N>::MINB) k_line(const __grid_constant__ LineArgs a) {
    using F = RegFft<T, N>;
    using G = Line<T, N, 128>;
    constexpr int KT = G::KT, W = G::W;
    constexpr bool TOUT = DIR > 0;   // all rows go out: by TMA
    extern __shared__ __align__(1024) unsigned char smem_line[];
    if (a.gate && a.gate_stage > a.gate->s_rkl) return;
    const int nst = a.nst;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ng = blockDim.x / (W * 32);
    const int grp = warp / W, w = warp % W;
    const int q = lane / G::CW, co = G::coff(G::column(lane % G::CW, w));
    const bool lead = w == 0 && lane == 0;
    unsigned char* base = smem_line + ((1024 - (smem_u32(smem_line) & 1023)) & 1023);
    unsigned char* ring = base + (size_t)grp * nst * G::TILE;
    C2<T>* tw = reinterpret_cast<C2<T>*>(base + (size_t)ng * nst * G::TILE);
    T* kax = reinterpret_cast<T*>(tw + F::TWN);
    // per stage: loaded (TMA bytes), then read out by every warp of the group
    uint64_t* bar = reinterpret_cast<uint64_t*>(kax + ((N + 1) & ~1)) + 2 * grp * nst;
    uint64_t* empty = bar + nst;
    // the group's loads so far (its first thread's; in shared memory, off the registers)
    int* issued = reinterpret_cast<int*>(reinterpret_cast<uint64_t*>(kax + ((N + 1) & ~1)) + 2 * ng * nst) + grp;

    // a pass whose boxes all have no masked content walks only the tiles it keeps
    bool all_clear = a.trim != 0;
    for (int b = 0; all_clear && b < a.nb; b++) all_clear = !a.scs[b].masked_live;
    const bool ctile = a.tr_always || all_clear;
    const bool couter = a.tr_always != 0;
    const int nkb = ctile ? a.tr_nkb : (a.kcols + KT - 1) / KT;
    const int nouter = couter ? a.tr_nouter : (a.axis == 0 ? a.g.ny : a.g.nx);
    const FastDiv fdj = ctile ? a.tr_fd_job : a.fd_job, fdb = ctile ? a.tr_fd_box : a.fd_box;
    const FastDiv fdk = ctile ? a.tr_fd_kb : a.fd_kb;
    const int per_box = nouter * nkb, per_job = a.nb * per_box, total = a.njobs * per_job;
    const int first = blockIdx.x * ng + grp, step = gridDim.x * ng;
    const double* om = a.axis == 0 ? a.g.my : a.g.mx;   // mask factors of the outer index

    struct Where { int job, box, o, kb; bool skip, clear; };
    auto where = [&](int t) {
        Where x;
        x.job = (int)fdj.div((unsigned)t);
        const int rb = t - x.job * per_job;
        x.box = (int)fdb.div((unsigned)rb);
        const int rem = rb - x.box * per_box;
        const int oe = (int)fdk.div((unsigned)rem);
        x.kb = rem - oe * nkb;
        x.o = couter ? a.tr_outer[oe] : oe;
        x.clear = a.trim && (all_clear || !a.scs[x.box].masked_live);
        x.skip = (a.outer_filter && !couter && om[x.o] == 0.0) || (x.clear && x.kb * KT >= a.g.kz_keep);
        return x;
    };
    auto segment = [&](const LineSeg& s, unsigned char* dst, uint64_t* b, const Where& x, int ch) {
        for (int i = 0; i < s.n; i++) {
            const int row = s.row + i * s.rows;
            tma_load_4d(dst + row * 128, &a.map[s.map], b, 2 * x.kb * KT, a.axis == 0 ? x.o : row,
                        a.axis == 0 ? row : x.o, ch);
        }
    };
    auto issue = [&](int t, int s, int j) {   // load j of the group, by its first thread
        *issued = j + 1;
        const Where x = where(t);
        if (x.skip) { mbar_expect_tx(&bar[s], 0); return; }
        const LineSeg* seg = x.clear ? a.in_trim : a.in;
        mbar_expect_tx(&bar[s], (uint32_t)((seg[0].rows * seg[0].n + seg[1].rows * seg[1].n) * 128));
        const int ch = a.job[x.job].ch_in + x.box * a.in_box_ch;
        segment(seg[0], ring + (size_t)s * G::TILE, &bar[s], x, ch);
        segment(seg[1], ring + (size_t)s * G::TILE, &bar[s], x, ch);
    };

    if (lead) {
        *issued = 0;
        for (int s = 0; s < nst; s++) { mbar_init(&bar[s], 1); mbar_init(&empty[s], W); }
        fence_mbar_init();
        for (int s = 0; s < nst; s++)
            if (first + s * step < total) issue(first + s * step, s, s);
    }
    regfft_fill_twiddles<T, N>(tw, (const C2<T>*)a.plan.tw, tid, blockDim.x);
    for (int i = tid; i < N; i += blockDim.x) kax[i] = (T)(a.axis == 0 ? a.g.kx : a.g.ky)[i];
    // bit e: this thread's e-th input row is inside the mask (inverse passes)
    uint32_t keepm = ~0u;
    if constexpr (DIR > 0) {
        const double* mg = a.axis == 0 ? a.g.mx : a.g.my;
        keepm = regfft_load_mask<T, N>(q, [&](int n) { return mg[n] != 0.0; });
    }
    __syncthreads();

    const T scale = (T)a.scale;
    bool dead = false;
    int it = 0;
    for (int t = first; t < total; t += step, it++) {
        const int s = it % nst;
        const Where x = where(t);
        unsigned char* tile = ring + (size_t)s * G::TILE;
        bool ok = !dead;
        if (ok) ok = mbar_wait(&bar[s], (uint32_t)((it / nst) & 1), SPK_WAIT_ITERS);
        dead = __any_sync(0xffffffffu, !ok);   // alike for the whole warp
        // the previous tile's stage, once its rows are out: the next load
        auto refill = [&]() {
            const int tn = t + (nst - 1) * step, sp = (it - 1) % nst;
            if (lead && it > 0 && !dead && tn < total) {
                if constexpr (TOUT) bulk_wait_read<0>();
                else dead = !mbar_wait(&empty[sp], (uint32_t)(((it - 1) / nst) & 1), SPK_WAIT_ITERS);
                if (!dead) {
                    fence_proxy_async_smem();
                    issue(tn, sp, it + nst - 1);
                }
            }
        };
        if (!dead && !x.skip) {
            const bool zrows = DIR > 0 && x.clear;
            const bool deriv = DIR > 0 && a.job[x.job].deriv != 0;
            C2<T> r[F::E];
            if (!zrows && !deriv) {
                line_load<T, N, 128>(r, q, tile, co, [&](C2<T> v, int) { return mk<T>(v.x * scale, v.y * scale); });
            } else if (!deriv) {
                line_load<T, N, 128>(r, q, tile, co, [&](C2<T> v, int e) {
                    return ((keepm >> e) & 1u) ? mk<T>(v.x * scale, v.y * scale) : mk<T>((T)0, (T)0);
                });
            } else {
                constexpr int R = F::radix(0);
                line_load<T, N, 128>(r, q, tile, co, [&](C2<T> v, int e) {
                    const T k = scale * kax[regfft_in_index<T, N, 0>(q, e / R, e % R)];
                    return (!zrows || ((keepm >> e) & 1u)) ? mk<T>(-k * v.y, k * v.x) : mk<T>((T)0, (T)0);
                });
            }
            line_from<T, N, 128, DIR, 0>(r, q, tw, tile, co, refill);
            if constexpr (TOUT) fence_proxy_async_smem();
        } else {
            refill();
        }
        if constexpr (W > 1) named_barrier(1 + grp, W * 32);
        else __syncwarp();
        const int cho = a.job[x.job].ch_out + x.box * a.out_box_ch;
        if constexpr (TOUT) {
            if (lead && !dead) {
                if (!x.skip)
                    for (int row = 0; row < N; row += a.out_rows)
                        tma_store_4d(&a.map[3], tile + row * 128, 2 * x.kb * KT, a.axis == 0 ? x.o : row,
                                     a.axis == 0 ? row : x.o, cho);
                bulk_commit();
            }
        } else {
            if (!dead && !x.skip) {
                // the kept rows, 16 bytes a lane (whole chunks that begin inside
                // kcols; a row's padding takes the odd column)
                const int chunk = lane & 7, k0 = x.kb * KT + chunk * G::EPC;
                const int npre = a.out_pre, nrow = npre + N - a.out_suf;
                const size_t pitch = a.axis == 0 ? (size_t)a.g.ny * a.g.nzs : (size_t)a.g.nzs;
                C2<T>* out = (C2<T>*)a.out + (size_t)cho * a.g.ncs +
                             (size_t)x.o * (a.axis == 0 ? (size_t)a.g.nzs : (size_t)a.g.ny * a.g.nzs) + k0;
                if (k0 < a.kcols)
                    for (int i = w * 4 + (lane >> 3); i < nrow; i += W * 4) {
                        const int row = i < npre ? i : i - npre + a.out_suf;
                        *reinterpret_cast<float4*>(out + row * pitch) =
                            *reinterpret_cast<const float4*>(tile + row * 128 + ((chunk ^ (row & 7)) << 4));
                    }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
        }
    }
    if (TOUT && lead) bulk_wait<0>();
    if (dead) {
        if (lane == 0) atomicExch(a.err, 2);
        // bounded drain of the loads in flight: the group has walked its tiles
        // to the end without loading, so they are counted by what went out
        if (lead)
            for (int j = ring_first_pending(*issued, nst); j < *issued; j++)
                mbar_wait(&bar[ring_stage(j, nst)], ring_parity(j, nst), SPK_WAIT_ITERS);
    }
}

}  // namespace spk
