// Device pieces of the row orthonormalisation (CholeskyQR): the one-warp
// Cholesky with its inverse, and the Gram that the kernel producing the rows
// finishes by itself.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace dt {

// 1 / sqrt(d) for a normal d > 0, from the hardware's approximation y0 by the
// series of (1 - e)^(-1/2) = 1 + e/2 + 3 e^2 / 8 + 5 e^3 / 16 + ..., e = 1 - d
// y0^2 (|e| < 2^-19, so the next term is below 2^-77): straight-line code that
// the caller's shuffles and updates fill.
__device__ __forceinline__ double rsqrt_seed(double d) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    return y;
}
__device__ __forceinline__ double rsqrt_refine(double d, double y0) {
    const double e = fma(-(d * y0), y0, 1.0);
    const double p = fma(fma(e, 0.3125, 0.375), e, 0.5);
    return fma(p, y0 * e, y0);
}

// G = L L^T of the symmetric r x r matrix G (row i at G + i ldg; r <= RT), by
// one warp: lane c holds column c of G in registers and gets column c of
// L^{-1} in y (columns c >= r are those of the identity).  The row operations
// that eliminate G are applied to the identity as well, so the inverse needs no
// exchange and no chain of its own.  The next pivot is formed first, from
// values exchanged before this pivot's root is known, and its approximation
// starts before the rows are updated: the chain of a pivot is the refinement,
// one multiplication and one FMA.  No branch stands between the rows (r < RT
// rows have zero multipliers).  RT = r = 16: 2200 cycles, against 7400 for a
// CTA-wide Cholesky of two barriers a pivot and a back substitution.  Returns
// false on a pivot that is not positive (or not a normal number).
template <int RT>
__device__ __forceinline__ bool warp_chol_linv(const double *G, int ldg, int r, double (&y)[RT]) {
    const int lane = threadIdx.x & 31;
    double g[RT];
#pragma unroll
    for (int i = 0; i < RT; i++) {
        g[i] = (i < r && lane < r) ? G[i * ldg + lane] : 0.0;
        y[i] = i == lane ? 1.0 : 0.0;
    }
    double d = __shfl_sync(0xffffffffu, g[0], 0);
    double seed = rsqrt_seed(d);
    const double least = fmax(1e-28 * d, 2.3e-308);
    bool ok = true;
#pragma unroll
    for (int k = 0; k < RT; k++) {
        if (k >= r) break;
        double s[RT], next = 0.0;
#pragma unroll
        for (int i = k + 1; i < RT; i++) s[i] = __shfl_sync(0xffffffffu, g[k], i);
        if (k + 1 < RT) next = __shfl_sync(0xffffffffu, g[k + 1], k + 1);
        ok = ok && d > least;
        const double ri = rsqrt_refine(d, seed);
        if (k + 1 < RT) {
            const double l = s[k + 1] * ri;
            d = fma(-l, l, next);
            seed = rsqrt_seed(d);
        }
        const double gk = g[k] * ri, yk = y[k] * ri;
        y[k] = yk;
#pragma unroll
        for (int i = k + 1; i < RT; i++) {
            const double l = s[i] * ri;
            g[i] = fma(-l, gk, g[i]);
            y[i] = fma(-l, yk, y[i]);
        }
    }
    return ok;
}

// Scratch of the Gram that its producers finish: one r x r partial per CTA,
// one per group of GRAM_GROUP CTAs, and arrival counters (zero before the
// first use; the last CTA leaves them zero).
constexpr int GRAM_GROUP = 16;
constexpr int GRAM_MAX_BLOCKS = 1024;
struct GramFinish {
    double *part;       // gridDim.x x r x r
    double *group;      // ceil(gridDim.x / GRAM_GROUP) x r x r (one group: may be `part`)
    int *counters;      // one and one for each group
    double *Linv;       // r x r, col-major
    int *flag;          // bit 0: the rows are linearly dependent
};

// out[e] = sum over the n partials, in order, 16 loads in flight (the partials
// come from other CTAs of this launch: read from L2).
__device__ __forceinline__ void sum_partials_in_order(const double *part, int n, int rr,
                                                      double *out) {
    for (int e = threadIdx.x; e < rr; e += blockDim.x) {
        double s = 0.0;
        for (int b = 0; b < n; b += 16) {
            double v[16];
#pragma unroll
            for (int q = 0; q < 16; q++)
                v[q] = b + q < n ? __ldcg(part + (int64_t)(b + q) * rr + e) : 0.0;
#pragma unroll
            for (int q = 0; q < 16; q++) s += v[q];
        }
        out[e] = s;
    }
}

// Every CTA of the launch (256 threads, gridDim.x <= GRAM_MAX_BLOCKS) comes
// here with its warps' Gram tiles: acc[a][b] is the 8 x 8 tile of rows 8 a and
// columns 8 b.  The warps' tiles are added in a fixed order; the last CTA of
// a group adds the group's partials and the last group's CTA adds those,
// factors G = L L^T and writes L^{-1}.  Bound by latency (two sums of up to 37
// partials each, 16 loads in flight, and the pivots' chain): r = 16, 592 CTAs,
// about 11 us at the end of the producing kernel, where a Gram launch, a
// reduction launch and a factorisation by a division-based Cholesky took 11 + 8
// + 38 us.  The sums do not depend on the order of arrival.
template <int TT>
__device__ void gram_finish(double (&acc)[TT][TT][2], int r, const GramFinish &f) {
    constexpr int RT = 8 * TT;
    __shared__ double red[4][RT * RT];
    __shared__ int last;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, g = lane >> 2, t4 = lane & 3;
    const int rr = r * r;
#pragma unroll
    for (int half = 0; half < 2; half++) {
        if ((w >> 2) == half) {
#pragma unroll
            for (int a = 0; a < TT; a++)
#pragma unroll
                for (int b = 0; b < TT; b++)
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        double &dst = red[w & 3][(8 * a + g) * RT + 8 * b + 2 * t4 + q];
                        dst = half ? dst + acc[a][b][q] : acc[a][b][q];
                    }
        }
        __syncthreads();
    }
    for (int e = t; e < rr; e += blockDim.x) {
        const int i = e / r, j = e - i * r, o = i * RT + j;
        f.part[(int64_t)blockIdx.x * rr + e] = (red[0][o] + red[1][o]) + (red[2][o] + red[3][o]);
    }
    const int grp = blockIdx.x / GRAM_GROUP, ngrp = (gridDim.x + GRAM_GROUP - 1) / GRAM_GROUP;
    const int first = grp * GRAM_GROUP, size = min(GRAM_GROUP, (int)gridDim.x - first);
    __threadfence();
    __syncthreads();
    if (t == 0) last = atomicAdd(f.counters + 1 + grp, 1) == size - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    sum_partials_in_order(f.part + (int64_t)first * rr, size, rr, f.group + (int64_t)grp * rr);
    __threadfence();
    __syncthreads();
    if (t == 0) {
        f.counters[1 + grp] = 0;
        last = atomicAdd(f.counters, 1) == ngrp - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double *G = red[0];
    sum_partials_in_order(f.group, ngrp, rr, G);
    __syncthreads();
    if (t < 32) {
        double y[RT];
        const bool ok = warp_chol_linv<RT>(G, r, r, y);
#pragma unroll
        for (int i = 0; i < RT; i++)
            if (i < r && lane < r) f.Linv[i + r * lane] = i >= lane ? y[i] : 0.0;
        if (lane == 0) {
            if (!ok) atomicOr(f.flag, 1);
            f.counters[0] = 0;
        }
    }
}

}  // namespace dt
