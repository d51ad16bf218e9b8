// spk_xrhs.cu -- x forward, right-hand side and x inverse of one RK3 stage in
// one pass (HD and MHD steps with deferred masked modes, stages 0 and 1).
//
// The right-hand side and the low-storage update act mode by mode, and the x
// transforms on either side of them act on the x lines of fixed (ky, kz).  A
// tile is one ky, KT consecutive kz columns and all x, of one field triple
// (velocity: 5 stress channels in; magnetic field: 3 EMF channels in; 3 out):
//   1. TMA loads of the product channels after the y forward;
//   2. x forward in shared memory (warp-owned transforms, spk_line.cuh);
//   3. every kept mode: contraction, diffusion, Leray projection and RK
//      update (k_rhs's arithmetic in the same order), the new state to HBM
//      and, scaled and rounded as the x inverse reads it, to the tile;
//   4. x inverse of the three fields, TMA stores to the pass buffer.
// As separate passes the products and the new state each made a round trip
// through HBM: at 256^3 MHD, FP32, 2.0 GB per stage and 0.37 ms (x forward
// 0.096, RHS 0.158, x inverse 0.112) against 1.1 GB and 0.27 ms here; the step
// goes from 2.75 to 2.59 ms, plain 5.04 to 4.87, 64^3 FP32 0.134 to 0.115
// (two launches fewer a stage).
// The pass is bound by latency: 64-byte rows keep five channels of N = 256
// within 80 KB, so two CTAs of 256 threads (128 registers) share an SM and
// overlap their phases.  Prefetching the state's rows into L2 while the
// products arrive measured slower (four steps 10.42 ms without, 10.56 by TMA,
// 10.60 per thread), and so did loading the products by cp.async (10.59).
// Three fifths of a tile's time go to step 3 (phase clocks at 256^3 FP32: 23k
// of 39k cycles), whose rows lie in 45 pages per array: the loads of one mode
// ahead cover part of their latency.
//
// Boxes with masked content (DevScalars::masked_live) walk every (ky, kz)
// tile: their masked modes enter the inverse scaled to the next stage, as in
// k_axis2's deferred x inverse.
#include "spk_line.cuh"

namespace spk {

struct XrArgs {
    alignas(64) CUtensorMap in, out;     // products, x-inverse output: boxes of N rows
    XfArgs x;
    int in_box_ch, out_box_ch;           // channels of a box in the maps
    int ch_T, ch_E, ch_u, ch_b;          // first channels: stress, EMF (in); u, B (out)
    double scale;                        // the x inverse's 1/N^3
    FastDiv fd_kb, fd_outer, tr_fd_kb, tr_fd_outer;   // k blocks, ky rows: all, and the kept ones
    int* err;
};

// 64-byte rows where a warp's columns fit them, else 128
template <typename T, int N> __host__ __device__ constexpr int xr_rb() { return line_ok<T, N, 64>() ? 64 : 128; }
template <typename T, int N> __host__ __device__ constexpr bool xr_ok() {
    return line_ok<T, N, xr_rb<T, N>()>() && 5 * N * xr_rb<T, N>() <= 96 * 1024;
}

template <typename T, int N>
__global__ void __launch_bounds__(256, 2) k_xrhs(const __grid_constant__ XrArgs a) {
    using F = RegFft<T, N>;
    constexpr int RB = xr_rb<T, N>();
    using G = Line<T, N, RB>;
    constexpr int KT = G::KT, W = G::W;
    extern __shared__ __align__(1024) unsigned char smem_line[];
    unsigned char* tiles = smem_line + ((1024 - (smem_u32(smem_line) & 1023)) & 1023);
    C2<T>* tw = reinterpret_cast<C2<T>*>(tiles + 5 * G::TILE);
    double* kxs = reinterpret_cast<double*>(tw + ((F::TWN + 1) & ~1));
    unsigned char* keep = reinterpret_cast<unsigned char*>(kxs + N);
    uint64_t* bar = reinterpret_cast<uint64_t*>(keep + ((N + 7) & ~7));
    const XfArgs& x = a.x;
    const DevGrid& g = x.g;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int q = lane / G::CW;
    const int kzk = g.kz_keep;
    const size_t nc = g.nc;

    bool all_clear = true;
    for (int b = 0; all_clear && b < x.nb; b++) all_clear = !x.sc[b].masked_live;
    const int nkb = ((all_clear ? kzk : g.nzh) + KT - 1) / KT, nouter = all_clear ? x.nky : g.ny;
    const FastDiv fdk = all_clear ? a.tr_fd_kb : a.fd_kb, fdo = all_clear ? a.tr_fd_outer : a.fd_outer;
    const int per_group = x.nb * nouter * nkb, total = (x.mhd ? 2 : 1) * per_group;

    struct Where { int mag, box, o, kb; bool kept, live; };
    auto where = [&](int t) {
        Where w;
        w.mag = t >= per_group;   // velocity tiles first, then magnetic ones: every CTA gets its share of both
        const int r = w.mag ? t - per_group : t;
        const int r1 = (int)fdk.div((unsigned)r);
        w.kb = r - r1 * nkb;
        w.box = (int)fdo.div((unsigned)r1);
        const int oe = r1 - w.box * nouter;
        w.o = all_clear ? x.kyi[oe] : oe;
        w.live = !all_clear && x.sc[w.box].masked_live;
        w.kept = all_clear || (g.my[w.o] != 0.0 && w.kb * KT < kzk);
        return w;
    };
    auto issue = [&](int t) {   // thread 0: the products of tile t
        const Where w = where(t);
        if (!w.kept) return;
        const int nch = w.mag ? 3 : 5, ch = (w.mag ? a.ch_E : a.ch_T) + w.box * a.in_box_ch;
        mbar_expect_tx(bar, (uint32_t)(nch * G::TILE));
        for (int c = 0; c < nch; c++)
            tma_load_4d(tiles + c * G::TILE, &a.in, bar, 2 * w.kb * KT, w.o, 0, ch + c);
    };
    if (tid == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
        if ((int)blockIdx.x < total) issue(blockIdx.x);
    }
    regfft_fill_twiddles<T, N>(tw, (const C2<T>*)x.plan.tw, tid, 256);
    for (int i = tid; i < N; i += 256) {
        kxs[i] = g.kx[i];
        keep[i] = g.mx[i] != 0.0;
    }
    __syncthreads();
    const uint32_t keepm = regfft_load_mask<T, N>(q, [&](int n) { return keep[n] != 0; });

    int phase = 0;
    bool aborted = false;
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        const Where w = where(t);
        const int k0 = w.kb * KT;
        if (w.kept) {
            const bool ok = mbar_wait(bar, (uint32_t)(phase & 1), SPK_WAIT_ITERS);
            phase++;
            if (__syncthreads_or(!ok)) { aborted = true; break; }
            // x forward of the products
            const int ntask = (w.mag ? 3 : 5) * W;
#pragma unroll 1
            for (int k = warp; k < ntask; k += 8) {
                const int ch = k / W;
                const int co = G::coff(G::column(lane % G::CW, k - ch * W));
                C2<T> r[F::E];
                line_load<T, N, RB>(r, q, tiles + ch * G::TILE, co, [](C2<T> v, int) { return v; });
                line_from<T, N, RB, -1, 0>(r, q, tw, tiles + ch * G::TILE, co, []() {});
            }
            __syncthreads();
        } else {
            __syncthreads();   // the previous tile's stores have read the buffer (thread 0 waited)
        }
        const size_t bo = (size_t)w.box * x.box_state + (size_t)(w.mag ? x.MAG : x.VEL) * nc;
        const DevScalars& sc = x.sc[w.box];
        const double dt = sc.dt, visc = w.mag ? sc.nu_m : sc.nu;
        const double ky = g.ky[w.o];
        auto cell = [&](int ch, int i, int c) -> C2<T>& {
            return *reinterpret_cast<C2<T>*>(tiles + ch * G::TILE + (G::swz(i) ^ G::coff(c)));
        };
        auto to_tile = [&](int ch, int i, int c, double2 v) { cell(ch, i, c) = mk<T>((T)(v.x * a.scale), (T)(v.y * a.scale)); };
        if (w.kept) {
            const int c = tid % KT, k = k0 + c;
            const double kz = g.kz[min(k, g.nzh - 1)];
            if (k < kzk) {
                // one mode ahead: its loads go out before this mode's stores
                // (the compiler cannot move them across)
                double2 Xn[3] = {d2(0.0, 0.0), d2(0.0, 0.0), d2(0.0, 0.0)}, Sn[3] = {Xn[0], Xn[0], Xn[0]};
                int in = 0;
                size_t gn = 0;
                auto fetch = [&](int ix) {
                    if (ix >= x.nkx) return;
                    in = x.kxi[ix];
                    gn = bo + ((size_t)in * g.ny + w.o) * g.nzh + k;
#pragma unroll
                    for (int d = 0; d < 3; d++) Xn[d] = x.U[gn + d * nc];
                    if (x.mode == XM_RK1)
#pragma unroll
                        for (int d = 0; d < 3; d++) Sn[d] = x.S[gn + d * nc];
                };
                fetch(tid / KT);
                for (int ix = tid / KT; ix < x.nkx; ix += 256 / KT) {
                    const int i = in;
                    const size_t gi = gn;
                    const double2 X[3] = {Xn[0], Xn[1], Xn[2]}, S[3] = {Sn[0], Sn[1], Sn[2]};
                    double2 R[3], Un[3];
                    fetch(ix + 256 / KT);
                    const double kx = kxs[i];
                    const double k2 = kx * kx + ky * ky + kz * kz;
                    const double f = -visc * k2;
                    if (!w.mag) {
                        const double2 t0 = to_d2(cell(0, i, c)), t1 = to_d2(cell(1, i, c)), t2 = to_d2(cell(2, i, c));
                        const double2 t3 = to_d2(cell(3, i, c)), t4 = to_d2(cell(4, i, c));
                        const double2 s0 = d2(kx * t0.x + ky * t1.x + kz * t2.x, kx * t0.y + ky * t1.y + kz * t2.y);
                        const double2 s1 = d2(kx * t1.x + ky * t3.x + kz * t4.x, kx * t1.y + ky * t3.y + kz * t4.y);
                        const double2 s2 = d2(kx * t2.x + ky * t4.x - kz * (t0.x + t3.x), kx * t2.y + ky * t4.y - kz * (t0.y + t3.y));
                        R[0] = d2(s0.y, -s0.x);
                        R[1] = d2(s1.y, -s1.x);
                        R[2] = d2(s2.y, -s2.x);
#pragma unroll
                        for (int d = 0; d < 3; d++) R[d] = d2(R[d].x + f * X[d].x, R[d].y + f * X[d].y);
                        const double ik2 = k2 > 0.0 ? 1.0 / k2 : 1.0;
                        const double sx = kx * R[0].x + ky * R[1].x + kz * R[2].x;
                        const double sy = kx * R[0].y + ky * R[1].y + kz * R[2].y;
                        const double kk[3] = {kx, ky, kz};
#pragma unroll
                        for (int d = 0; d < 3; d++) R[d] = d2(R[d].x - kk[d] * ik2 * sx, R[d].y - kk[d] * ik2 * sy);
                    } else {
                        const double2 e0 = to_d2(cell(0, i, c)), e1 = to_d2(cell(1, i, c)), e2 = to_d2(cell(2, i, c));
                        const double2 S3[3] = {d2(ky * e2.x - kz * e1.x, ky * e2.y - kz * e1.y),
                                               d2(kz * e0.x - kx * e2.x, kz * e0.y - kx * e2.y),
                                               d2(kx * e1.x - ky * e0.x, kx * e1.y - ky * e0.y)};
#pragma unroll
                        for (int d = 0; d < 3; d++) R[d] = d2(-S3[d].y + f * X[d].x, S3[d].x + f * X[d].y);
                    }
#pragma unroll
                    for (int d = 0; d < 3; d++) {
                        Un[d] = rk_value(x, gi + d * nc, X[d], S[d], R[d], dt);
                        x.U[gi + d * nc] = Un[d];
                        to_tile(d, i, c, Un[d]);
                    }
                }
            }
        }
        if (w.live) {
            // masked modes at the next stage's value (see the deferred x inverse in k_axis2)
            const T dnu = (T)(-visc * dt);
            const int c = tid % KT, k = k0 + c;
            const bool inside = w.kept && k < kzk;    // the column has kept modes
            const double kzc = g.kz[min(k, g.nzh - 1)];
            const T k2yz = (T)(ky * ky + kzc * kzc);
#pragma unroll 4
            for (int i = tid / KT; i < N; i += 256 / KT) {
                const bool mine = !(inside && keep[i]);
                double2 X[3];
#pragma unroll
                for (int d = 0; d < 3; d++)
                    X[d] = mine && k < g.nzh ? x.U[bo + d * nc + ((size_t)i * g.ny + w.o) * g.nzh + k] : d2(0.0, 0.0);
                const T kxn = (T)kxs[i];
                const T z = dnu * (kxn * kxn + k2yz);
                const T c1 = (T)1 + (T)(8.0 / 15.0) * z;
                const T fac = x.mode == XM_RK0 ? c1 : c1 + (T)(-17.0 / 60.0) * z + (T)(5.0 / 12.0) * z * c1;
                if (mine)
#pragma unroll
                    for (int d = 0; d < 3; d++) {
                        const C2<T> v = mk<T>((T)(X[d].x * a.scale), (T)(X[d].y * a.scale));
                        cell(d, i, c) = mk<T>(fac * v.x, fac * v.y);
                    }
            }
        }
        __syncthreads();
        if (w.kept || w.live) {
            // x inverse of the three fields (masked rows are zero without masked content)
#pragma unroll 1
            for (int k = warp; k < 3 * W; k += 8) {
                const int ch = k / W;
                const int co = G::coff(G::column(lane % G::CW, k - ch * W));
                C2<T> r[F::E];
                line_load<T, N, RB>(r, q, tiles + ch * G::TILE, co, [&](C2<T> v, int e) {
                    return (w.live || ((keepm >> e) & 1u)) ? v : mk<T>((T)0, (T)0);
                });
                line_from<T, N, RB, +1, 0>(r, q, tw, tiles + ch * G::TILE, co, []() {});
            }
            fence_proxy_async_smem();
        }
        __syncthreads();
        if (tid == 0) {
            if (w.kept || w.live) {
                const int ch = (w.mag ? a.ch_b : a.ch_u) + w.box * a.out_box_ch;
                for (int d = 0; d < 3; d++)
                    tma_store_4d(&a.out, tiles + d * G::TILE, 2 * k0, w.o, 0, ch + d);
                bulk_commit();
                bulk_wait_read<0>();
            }
            if (t + (int)gridDim.x < total) issue(t + gridDim.x);
        }
    }
    if (tid == 0) bulk_wait<0>();
    if (aborted) {
        if (tid == 0) {
            atomicExch(a.err, 2);
            mbar_wait(bar, (uint32_t)((phase - 1) & 1), SPK_WAIT_ITERS);   // bounded drain
        }
        __syncthreads();
    }
}

}  // namespace spk
