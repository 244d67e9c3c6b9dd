// cvm_lines.cuh -- rows of 2^7 .. 2^11 points with N/16 threads per line:
// the geometry that the forward (cvm_rows.cu) and inverse (cvm_lines.cu)
// kernels share.
//
// Layout of the line buffer: pass 1's unit of natural index k0 (logical
// block v = brev(k0)) stores output i at i * PITCH + k0.  Pass 2's unit
// (block b, column j) reads its 16 elements at j * PITCH + brev4(i) * NB +
// brev(b) and stores them in place, output i at j * PITCH + i * NB +
// brev(b); pass 3's unit jj = j + R1 * i then reads NB consecutive
// elements.  PITCH keeps the three access patterns free of bank conflicts.
#pragma once

#include "cvm_device.cuh"

namespace cvm {
namespace {

template <int L>
struct Lines {
    static constexpr int N = 1 << L;
    static constexpr int R1 = (L & 1) ? 8 : 16;           // pass 1: the head, or radix 16 at quarter 1
    static constexpr int K1 = N / R1;                     // its units
    static constexpr int NB = N / (16 * R1);              // blocks of pass 2 = pass 3's radix (1: no pass 3)
    static constexpr int H2 = R1, H3 = 16 * R1;           // quarters of passes 2 and 3
    // line pitch: conflict-free for pass 2's reads (8-byte words of NB-wide
    // blocks) and pass 3's 16-byte reads over consecutive columns
    static constexpr int PITCH = NB == 1 ? K1 + 1 : (NB == 4 ? K1 + 6 : K1 + 2);
    static constexpr int LINE = (R1 * PITCH + 1) & ~1;    // elements
    static constexpr int G = N / 16;                      // threads of a line
    static constexpr int CTA = G > 64 ? G : 64;
    static constexpr int NL = CTA / G;                    // lines of a CTA at a time
    static constexpr size_t SMEM = (size_t)NL * LINE * sizeof(float2);  // + TABLE's bounds
};

// The barrier of a line's threads: the CTA (one line at a time) or the
// group's lanes of its warp.
template <int G>
__device__ __forceinline__ void group_sync(unsigned int mask) {
    if constexpr (G <= 32)
        __syncwarp(mask);
    else
        __syncthreads();
}

// Pass 2 of a line in the thread's registers: its unit's column j and block
// place bb, lanes over the blocks first (NB = 4: even columns, then odd ones,
// in groups of eight, keep the half-warps on distinct banks).
template <int L>
__device__ __forceinline__ void pass2_unit(int lt, int &j, int &bb) {
    constexpr int NB = Lines<L>::NB;
    const int jl = lt / NB;
    bb = lt & (NB - 1);
    j = NB == 4 ? (jl & 8) | ((jl & 3) << 1) | ((jl >> 2) & 1) : jl;
}

template <int L, bool INV, bool F>
__device__ __forceinline__ void pass2(float2 *ln, int j, int bb, float2 *z, const float2 *__restrict__ tri) {
    using S = Lines<L>;
    float2 *q = ln + j * S::PITCH + bb;
#pragma unroll
    for (int i = 0; i < 16; i++) z[i] = q[brevk(i, 4) * S::NB];
    math16<INV, S::H2, F>(z, tri + tw_off(L, S::H2) + j);
    if constexpr (S::NB > 1) {
#pragma unroll
        for (int i = 0; i < 16; i++) q[i * S::NB] = z[i];
    }
}

// Pass 3's unit jj (NB elements at quarter H3) into z.
template <int L, bool INV, bool F>
__device__ __forceinline__ void pass3(const float2 *ln, int jj, float2 *z, const float2 *__restrict__ tri) {
    using S = Lines<L>;
    const float4 *q = reinterpret_cast<const float4 *>(ln + (jj & (S::R1 - 1)) * S::PITCH + (jj / S::R1) * S::NB);
#pragma unroll
    for (int i = 0; i < S::NB / 2; i++) {
        const float4 w = q[i];
        // block b sits at brev(b)
        z[brevk(2 * i, ilog2k(S::NB))] = make_float2(w.x, w.y);
        z[brevk(2 * i + 1, ilog2k(S::NB))] = make_float2(w.z, w.w);
    }
    if constexpr (S::NB == 16)
        math16<INV, S::H3, F>(z, tri + tw_off(L, S::H3) + jj);
    else
        math4<INV, S::H3, F>(z, tri + tw_off(L, S::H3) + jj);
}

}  // namespace
}  // namespace cvm
