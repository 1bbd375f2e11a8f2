// deposit.cuh -- the corner sums of a group of cells by one warp, shared by the
// step's deposit (kernels.cu) and the allocation-free one (noalloc.cu).
//
// DepositAtom (src/cuda_Deposit.cu:289-317): per-cell sums of the four CIC
// weights.  Each lane adds its slots lane, lane + 32, ... of a cell in that
// order in FP32; the lanes are then added in FP64 by the xor tree (16, 8, 4,
// 2, 1), and one double4 per cell is written, which the node pass gathers in
// a fixed order.
//
// The adding of the lanes is most of the work of a cell with few particles
// (four trees of five shuffled doubles).  So a warp takes DEP_G = 4 cells, and
// the 16 sums go through the tree together: at each level a lane gives half
// of its sums to its partner and keeps the other half, so that 16 trees cost
// 8 + 4 + 2 + 1 + 1 additions and 24 shuffles (the first level exchanges the
// FP32 sums) instead of 80 and 160.  Every sum adds the same pairs as its
// own tree, so the bits are the same.
// Measured on a B200, two cells per warp with a tree per sum against this form:
// 0.118 and 0.104 ms on the 513x257 case with 200 particles per cell and
// species, 0.065 and 0.034 ms with 20, 0.041 and 0.031 ms on the 257x129 Ar/O2
// case.
#pragma once
#include "devutil.cuh"

namespace hp {
namespace dv {

constexpr int DEP_G = 4; // cells per warp

// Lane g < DEP_G holds cell g: its particle count, slots (null: no cell) and
// where its sums go.
__device__ __forceinline__ void deposit_group(int my_n, const float2 *my_xy, double4 *my_cw) {
    constexpr int G = DEP_G;
    const int lane = threadIdx.x & 31;
    int n[G];
    const float2 *xy[G];
    float w[4 * G]; // WS, WN, ES, EN of each cell
#pragma unroll
    for (int g = 0; g < G; g++) {
        n[g] = __shfl_sync(FULL, my_n, g);
        xy[g] = (const float2 *)__shfl_sync(FULL, (unsigned long long)my_xy, g);
    }
    // the first chunk of every cell together, then, where a cell has more, blocks
    // of four chunks, the next block's loads (of this cell or the next one) in
    // flight while a block is added
    float2 f0[G], f[4];
#pragma unroll
    for (int g = 0; g < G; g++) f0[g] = lane < n[g] ? xy[g][lane] : make_float2(0.f, 0.f);
    auto load = [&](const float2 *from, int k0, int ng, float2 *to) {
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const int k = k0 + 32 * h + lane;
            to[h] = k < ng ? from[k] : make_float2(0.f, 0.f);
        }
    };
    if (n[0] > 32) load(xy[0], 32, n[0], f);
#pragma unroll
    for (int g = 0; g < G; g++) {
        float WS = 0.f, WN = 0.f, ES = 0.f, EN = 0.f;
        auto add = [&](float2 at) {
            const float lx = at.x, ly = at.y;
            WS += (1 - lx) * (1 - ly);
            WN += (1 - lx) * ly;
            ES += lx * (1 - ly);
            EN += lx * ly;
        };
        const int ng = n[g], gn = g + 1 < G ? g + 1 : g;
        if (lane < ng) add(f0[g]);
        for (int k0 = 32; k0 < ng; k0 += 128) {
            float2 nf[4];
            if (k0 + 128 < ng) load(xy[g], k0 + 128, ng, nf);
            else if (gn > g && n[gn] > 32) load(xy[gn], 32, n[gn], nf);
#pragma unroll
            for (int h = 0; h < 4; h++)
                if (k0 + 32 * h + lane < ng) add(f[h]);
#pragma unroll
            for (int h = 0; h < 4; h++) f[h] = nf[h];
        }
        if (ng <= 32 && gn > g && n[gn] > 32) load(xy[gn], 32, n[gn], f);
        w[4 * g] = WS;
        w[4 * g + 1] = WN;
        w[4 * g + 2] = ES;
        w[4 * g + 3] = EN;
    }
    // the tree: a lane with bit o set keeps the upper half of the sums
    double a[2 * G], b[G], e[G / 2];
    {
        const bool up = (lane & 16) != 0;
#pragma unroll
        for (int k = 0; k < 2 * G; k++) {
            const float give = up ? w[k] : w[k + 2 * G], keep = up ? w[k + 2 * G] : w[k];
            a[k] = (double)keep + (double)__shfl_xor_sync(FULL, give, 16);
        }
    }
    {
        const bool up = (lane & 8) != 0;
#pragma unroll
        for (int k = 0; k < G; k++) {
            const double give = up ? a[k] : a[k + G], keep = up ? a[k + G] : a[k];
            b[k] = keep + __shfl_xor_sync(FULL, give, 8);
        }
    }
    {
        const bool up = (lane & 4) != 0;
#pragma unroll
        for (int k = 0; k < G / 2; k++) {
            const double give = up ? b[k] : b[k + G / 2], keep = up ? b[k + G / 2] : b[k];
            e[k] = keep + __shfl_xor_sync(FULL, give, 4);
        }
    }
    const bool up = (lane & 2) != 0;
    const double give = up ? e[0] : e[1], keep = up ? e[1] : e[0];
    double t = keep + __shfl_xor_sync(FULL, give, 2);
    t += __shfl_xor_sync(FULL, t, 1);
    // lanes 2q, 2q + 1 hold sum q' of the 16: bit 16 of the lane is its top bit
    const int q = ((lane & 16) >> 1) | ((lane & 8) >> 1) | ((lane & 4) >> 1) | ((lane & 2) >> 1);
    double *cw = (double *)__shfl_sync(FULL, (unsigned long long)my_cw, q >> 2);
    if (cw && !(lane & 1)) cw[q & 3] = t;
}
static_assert(DEP_G == 4, "the tree takes 16 sums");

} // namespace dv
} // namespace hp
