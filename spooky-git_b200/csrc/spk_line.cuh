// spk_line.cuh -- transforms that one warp owns, on a swizzled shared-memory
// tile (sm_100a).
//
// A tile holds N rows (the positions along the transformed axis) of RB bytes
// (KT = RB / sizeof(C2<T>) consecutive kz columns), as a TMA load with the
// RB-byte swizzle leaves it: the 16-byte chunk j of row n sits at chunk
// j ^ (n & 7) (RB = 128) or j ^ ((n >> 1) & 3) (RB = 64).  TPC = N/E lanes
// share a transform and a warp takes CW = 32/TPC columns, so a transform
// never leaves its warp: it reads its columns, exchanges its stages and
// writes its result in the cells of its own columns, with __syncwarp()
// between the stages instead of barriers of the CTA, and needs no exchange
// buffer.  The tile goes back to memory by a TMA store.
//
// Exchange element L lives in row L ^ ((L >> SH) & 7).  SH per length, and
// the columns of a warp (chunk (i / EPC) * W + warp for its i-th column where
// several warps share a tile), are chosen so that every access of the
// transform (first loads, exchanges, last stores) is free of bank conflicts;
// the exceptions are one exchange of the FP64 transforms of N = 128 and 384
// (2-way).
//
// All row indices split as (part of q) | (compile-time part) in disjoint
// bits, so an access is one XOR of the low row and chunk bits (at most eight
// distinct) and an immediate offset.
#pragma once
#include "spk_regfft.cuh"

namespace spk {

template <typename T, int N, int RB>
struct Line {
    using F = RegFft<T, N>;
    static constexpr int ES = (int)sizeof(C2<T>);
    static constexpr int KT = RB / ES;              // columns of a tile
    static constexpr int CW = 32 / F::TPC;          // columns of a warp
    static constexpr int W = KT / CW;               // warps of a tile
    static constexpr int EPC = 16 / ES;             // columns of a 16-byte chunk
    static constexpr int TILE = N * RB;             // bytes
    // row shift of the exchange layout (0: none), found by counting the
    // bank conflicts of every access for every length
    static constexpr int SH = sizeof(T) == 4
        ? (N <= 32 ? 0 : (!F::P2 ? 2 : (N == 64 ? 2 : (N == 128 ? 3 : 4))))
        : (N <= 48 ? 0 : (N == 64 || N == 256 ? 3 : (N == 192 ? 2 : 1)));
    __host__ __device__ static constexpr int xrow(int L) { return SH ? (L ^ ((L >> SH) & 7)) : L; }
    // byte offset of row n's chunk 0 in the swizzled tile
    __host__ __device__ static constexpr int swz(int n) {
        return RB == 128 ? n * 128 + ((n & 7) << 4) : n * 64 + (((n >> 1) & 3) << 4);
    }
    // column of the warp's i-th column; w: the warp within the tile
    __device__ static __forceinline__ int column(int i, int w) {
        if constexpr (W > 1 && CW > EPC) return ((i / EPC) * W + w) * EPC + i % EPC;
        else return w * CW + i;
    }
    // offset of column c within row 0
    __device__ static __forceinline__ int coff(int c) { return (c / EPC) * 16 + (c % EPC) * ES; }
    // cell of compile-time row part R from the thread's base offset b =
    // coff(c) ^ swz(q's row part): the low row bits by XOR, the rest added
    __device__ static __forceinline__ C2<T>& cell(unsigned char* tile, int b, int R) {
        return *reinterpret_cast<C2<T>*>(tile + (b ^ swz(R & 7)) + (R & ~7) * RB);
    }
};

// The lengths a warp can own: a warp's columns are whole 16-byte chunks (FP32
// at N = 384 and 512, one 8-byte column a warp, would use half of each shared-
// memory wavefront: 512^3 HD 39.3 -> 39.9 ms for two steps) and fit the tile.
template <typename T, int N, int RB> __host__ __device__ constexpr bool line_ok() {
    return N >= 24 && RegFft<T, N>::TPC <= 32 && (32 / RegFft<T, N>::TPC) * (int)sizeof(C2<T>) >= 16 &&
           32 / RegFft<T, N>::TPC <= RB / (int)sizeof(C2<T>);
}

// Stages S.. of the transform whose stage-S legs are in a[]; the result goes
// to the tile (row k, this thread's column).  mid(): called once, between
// the first stage and its exchange.
template <typename T, int N, int RB, int DIR, int S, typename MID>
__device__ __forceinline__ void line_from(C2<T>* a, int q, const C2<T>* tw, unsigned char* tile, int co, MID mid) {
    using F = RegFft<T, N>;
    using G = Line<T, N, RB>;
    regfft_stage_math<T, N, DIR, S>(a, q, tw);
    constexpr int R = F::radix(S), BPT = F::E / R;
    if constexpr (S == 0) mid();
    if constexpr (S + 1 < F::NS) {
        __syncwarp();   // every lane has read the legs it overwrites
        {
            const int b = co ^ G::swz(G::xrow(regfft_out_index<T, N, S>(q, 0, 0)));
#pragma unroll
            for (int u = 0; u < BPT; u++)
#pragma unroll
                for (int t = 0; t < R; t++) G::cell(tile, b, G::xrow(regfft_out_index<T, N, S>(0, u, t))) = a[u * R + t];
        }
        __syncwarp();
        constexpr int R1 = F::radix(S + 1), BPT1 = F::E / R1;
        {
            const int b = co ^ G::swz(G::xrow(regfft_in_index<T, N, S + 1>(q, 0, 0)));
#pragma unroll
            for (int u = 0; u < BPT1; u++)
#pragma unroll
                for (int r = 0; r < R1; r++) a[u * R1 + r] = G::cell(tile, b, G::xrow(regfft_in_index<T, N, S + 1>(0, u, r)));
        }
        line_from<T, N, RB, DIR, S + 1>(a, q, tw, tile, co, mid);
    } else {
        constexpr int P = F::P(S);
        __syncwarp();
        const int b = co ^ G::swz(q);
#pragma unroll
        for (int u = 0; u < BPT; u++)
#pragma unroll
            for (int t = 0; t < R; t++) G::cell(tile, b, u * F::TPC + P * t) = a[u * R + t];
    }
}

// The first-stage legs from the tile; f(value, e) maps the e-th one (e is a
// constant once the loop is unrolled).
template <typename T, int N, int RB, typename FN>
__device__ __forceinline__ void line_load(C2<T>* a, int q, unsigned char* tile, int co, FN f) {
    using F = RegFft<T, N>;
    using G = Line<T, N, RB>;
    constexpr int R = F::radix(0), BPT = F::E / R;
    const int b = co ^ G::swz(q);
#pragma unroll
    for (int u = 0; u < BPT; u++)
#pragma unroll
        for (int r = 0; r < R; r++)
            a[u * R + r] = f(G::cell(tile, b, regfft_in_index<T, N, 0>(0, u, r)), u * R + r);
}

}  // namespace spk
