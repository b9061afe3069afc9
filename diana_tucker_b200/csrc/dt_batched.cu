// Batched dense HOOI: many small 3-way tensors of uneven shapes and ranks
// decomposed in one persistent launch.
//
// Work items.  The host sorts the tensors by estimated cost (longest first,
// so the persistent CTAs finish together) and packs them into items: an item
// is one tensor worked on by the whole CTA, or two or four small tensors
// worked on side by side by equal thread groups of the CTA (each group with
// its own named barrier, its own slice of shared memory and of the global
// scratch).  Each CTA pulls items from an atomic queue.
//
// Per tensor, the whole HOOI runs inside its thread group: the
// dimension-tree TTM chain (T = X x_3 U_3^T shared by modes 1 and 2,
// X x_1 U_1^T x_2 U_2^T for mode 3), the Gram Y_(n) Y_(n)^T, the subspace
// iteration of ALS_ (hooi_als.tpp:7-34) with CholeskyQR, and finally the FP64
// core and relative error.  Arithmetic is FP64 throughout, on the FP64 tensor
// cores (mma.sync m8n8k4): every product is cut into 8 x 8 tiles, dealt over the
// group's warps.  X is FP32, read from global memory (from L2 while its group
// works on it) straight into fragments, 16 loads in flight per lane; the one
// large intermediate (I_1 x I_2 x R_3) is in the group's slice of global scratch;
// the factors, Y_(n) and its Gram (which takes Y_(n)'s place) live in shared
// memory.  In a subspace step each warp keeps its rows of S L in registers, laid
// out as the next products' fragments, from the product to the new factor.  Every
// sum goes in an order of the tensor's own (over its 8 x 8 tiles; over 512 classes
// of entries, as many as the largest block has threads): the results are the same
// bit for bit for every block size and packing, whatever the tuner takes.  4096
// tensors (modes 8 to 64, ranks 2 to 8, 10 sweeps): 11.5 ms, of it about half the
// two passes over X at 0.8 of the FP64 tensor rate (ranks padded to 8 columns); 100
// tensors 1.14 ms.  With one FMA chain per thread and entry on the CUDA cores 23.3
// and 2.4 ms.
//
// Autotuning.  The block size (128, 256, 512 threads) and the packing (one
// tensor per CTA; pairs, and quads, of the tensors small enough to share the
// CTA's shared memory: largest mode <= 32, <= 16) are chosen by timing every
// combination on the batch (a stratified sample of 8192 tensors of larger
// batches); the choice is cached per batch signature on the context.
//
// The launch (queue reset + persistent kernel) is a CUDA graph instantiated
// once per launch shape and kept on the context: the kernel reads its
// arguments from a device-resident block that each call rewrites, so a later
// call with the same launch shape replays the graph without re-capturing.
// On the legacy or per-thread default stream, which cannot be captured, the
// two are launched directly.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <numeric>
#include <tuple>
#include <vector>

#include "dt_kernels.cuh"

namespace dt {
namespace {

constexpr int BMAX_I = 64;               // largest mode size
constexpr int BMAX_R = 8;                // largest rank
constexpr int BMAX_K = BMAX_R * BMAX_R;  // largest product of two ranks

// Shared-memory doubles one tensor of largest mode size m needs: the factors
// (rows padded to whole tiles, 8 columns), Y_(n) or its Gram (rows of up to 64
// at a pitch of 4 mod 16; before and after the sweeps the classes of a sum).  The
// Gram shares of a subspace step, two tiles of 64 doubles a warp, come on top for
// the whole CTA.
__host__ __device__ constexpr int tile8(int n) { return (n + 7) / 8 * 8; }
__host__ __device__ constexpr int pitch16(int n) { return (n + 11) / 16 * 16 + 4; }
__host__ __device__ constexpr int slot_doubles(int m) {
    return 3 * tile8(m) * BMAX_R + tile8(m) * pitch16(BMAX_K);
}
constexpr int SLOT = slot_doubles(BMAX_I);                    // one CTA
// Room for four of the largest tensors that go four to a CTA.
constexpr int SLOT_ALL = SLOT > 4 * slot_doubles(16) ? SLOT : 4 * slot_doubles(16);
constexpr int WARP_SCR = 128;
// Global scratch per CTA: the intermediate and the last Y_(3).
constexpr int64_t SCR = (int64_t)BMAX_I * BMAX_I * BMAX_R + BMAX_I * BMAX_K;
// Largest mode size a tensor may have to share a CTA with 1 / 3 others.
constexpr int PAIR_MAX_I = 32, QUAD_MAX_I = 16;
static_assert(slot_doubles(PAIR_MAX_I) <= SLOT_ALL / 2 / 2 * 2 &&
                  slot_doubles(QUAD_MAX_I) <= SLOT_ALL / 4 / 2 * 2,
              "packing limits");
static_assert((int64_t)PAIR_MAX_I * PAIR_MAX_I * BMAX_R + PAIR_MAX_I * BMAX_K <= SCR / 2,
              "pair scratch");
static_assert((int64_t)QUAD_MAX_I * QUAD_MAX_I * BMAX_R + QUAD_MAX_I * BMAX_K <= SCR / 4,
              "quad scratch");

struct Item {
    int g;     // tensors worked on side by side (1, 2 or 4)
    int t[4];  // tensor ids, -1 where a group has none
};

struct BatchArgs {
    int count, nitems;
    const int64_t *shape;  // count x 3
    const int64_t *rank;   // count x 3
    const float *X;
    const int64_t *xoff;   // element offsets of each tensor
    double *U;             // factors, I_n x R_n col-major blocks
    const int64_t *uoff;   // count x 3 element offsets
    double *G;             // cores
    const int64_t *goff;
    double *relerr;
    const Item *items;
    int sweeps, inner;
    double *scratch;       // gridDim.x x SCR doubles
    int *queue;
};

// Shared memory goes by offsets into this array: the functions that are not
// inlined (to keep their registers apart) then still address it as such.
extern __shared__ __align__(16) double bt_sm[];

// A thread group working on one tensor: its threads are a contiguous run of
// whole warps of the CTA, synchronised by their own named barrier.
struct Grp {
    int lt;   // thread index in the group
    int gs;   // threads in the group (a multiple of 32)
    int bar;  // named barrier id (1..4; 0 is __syncthreads)
    int w, W;          // this warp, warps
    int g, t;          // fragment row / column of the lane
    int part;          // offset of W x WARP_SCR: the tiles' Gram shares
};

__device__ __forceinline__ void gsync(const Grp &g) {
    asm volatile("bar.sync %0, %1;" ::"r"(g.bar), "r"(g.gs) : "memory");
}

// Sum of the group's 512 classes in `cls` (shared memory), an order that does not
// depend on the group's size.
constexpr int CLASSES = 512;
static_assert(tile8(1) * pitch16(BMAX_K) >= CLASSES, "the classes take Y_(n)'s place");
__device__ double gsum(double *cls, const Grp &g) {
    gsync(g);
    if (g.w == 0) {
        double s = 0.0;
        for (int i = g.lt; i < CLASSES; i += 32) s += cls[i];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (g.lt == 0) cls[0] = s;
    }
    gsync(g);
    const double r = cls[0];
    gsync(g);
    return r;
}

__device__ __forceinline__ void bt_dmma(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// Factor entry (i, c): rows of 8, columns 4 apart swapped in every other pair of
// rows, so the four rows and eight columns of a fragment load hit distinct banks.
__device__ __forceinline__ int u_at(int i, int c) { return i * BMAX_R + (c ^ ((i & 2) << 1)); }

// dst(i, c, o) = sum_k src(i, o, k) U(k, c) for rows i < ni of no outer indices, K
// columns k and R <= 8 results c: every contraction of the chain.  Element (i, o,
// k) is at src[i si + o so + k sk], result (i, c, o) goes to dst[i di + c dc + o dw].
// A tile is 8 rows of one outer index; a warp takes four at a time, which share
// the factor's fragments, 16 columns in a block.  The next block's 16 loads per
// lane (of the same tiles or the next ones) are in flight while a block is
// multiplied: a block is 64 cycles of an SM's FP64 tensor rate, its loads come
// from L2.  Past K the last column is read again and meets zeros.
template <class TX>
__device__ __noinline__ void contract(const TX *src, int ni, int si, int no, int so, int K, int sk,
                                      int uo, double *dst, int di, int dc, int dw, int R, Grp g) {
    const double *U = bt_sm + uo;
    const int nti = (ni + 7) >> 3, ntile = nti * no, njobs = (ntile + 3) >> 2;
    auto tile = [&](int tau, int &i, int &o) {  // the lane's row and outer index
        tau = min(tau, ntile - 1);
        o = no == 1 ? 0 : tau / nti;
        i = 8 * (tau - o * nti) + g.g;
    };
    const TX *p[4];
    auto aim = [&](int job) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            int i, o;
            tile(4 * job + j, i, o);
            p[j] = src + min(i, ni - 1) * si + o * so;
        }
    };
    TX v[4][4], w[4][4];
    auto load = [&](TX (&x)[4][4], int k0) {
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const int k = min(k0 + 4 * s + g.t, K - 1) * sk;
#pragma unroll
            for (int j = 0; j < 4; j++) x[s][j] = p[j][k];
        }
    };
    int job = g.w, lj = g.w, lk = 0;
    if (job >= njobs) return;
    aim(job);
    load(v, 0);
    double acc[4][2] = {};
#pragma unroll 1
    for (int k0 = 0;;) {
        lk += 16;
        if (lk >= K) {
            lk = 0;
            lj += g.W;
            if (lj < njobs) aim(lj);
        }
        if (lj < njobs) load(w, lk);
#pragma unroll
        for (int s = 0; s < 4; s++) {
            if (k0 + 4 * s >= K) break;
            const int k = k0 + 4 * s + g.t;
            const double u = U[u_at(min(k, K - 1), g.g)];
            const double b = k < K ? u : 0.0;
#pragma unroll
            for (int j = 0; j < 4; j++) bt_dmma(acc[j][0], acc[j][1], (double)v[s][j], b);
        }
        k0 += 16;
        if (k0 >= K) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                int i, o;
                tile(4 * job + j, i, o);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int c = 2 * g.t + h;
                    if (4 * job + j < ntile && i < ni && c < R)
                        dst[i * di + c * dc + o * dw] = acc[j][h];
                    acc[j][h] = 0.0;
                }
            }
            k0 = 0;
            job += g.W;
            if (job >= njobs) return;
        }
#pragma unroll
        for (int s = 0; s < 4; s++)
#pragma unroll
            for (int j = 0; j < 4; j++) v[s][j] = w[s][j];
    }
}

// Zeroes what a Y_(n) of n x K does not fill of its whole tiles.
__device__ __forceinline__ void zero_pads(double *Y, int n, int K, int pitch, const Grp &g) {
    const int n8 = tile8(n), K4 = (K + 3) & ~3;
    for (int e = g.lt; e < n8 * K4; e += g.gs) {
        const int i = e / K4, k = e - i * K4;
        if (i >= n || k >= K) Y[i * pitch + k] = 0.0;
    }
}

// S (n x n, pitch ps) = Y Y^T in Y's place (pitch py, whole tiles zero padded).
// The upper triangle's tiles are dealt over the warps, at most 9 each, kept in
// registers until every warp has read Y.
__device__ __noinline__ void ggram(int ys, int n, int K, int py, int ps, Grp g) {
    double *YS = bt_sm + ys;
    const int nt = tile8(n) / 8, total = nt * (nt + 1) / 2, ks = (K + 3) / 4;
    double acc[9][2];
    int at[9];  // tile row | column << 4, -1: none
#pragma unroll
    for (int x = 0; x < 9; x++) {
        int s = g.w + x * g.W;
        at[x] = -1;
        if (s < total) {
            int r = 0;
            while (s >= nt - r) {
                s -= nt - r;
                r++;
            }
            at[x] = r | (r + s) << 4;
        }
    }
#pragma unroll
    for (int b = 0; b < 9; b += 3) {
        if (at[b] < 0) continue;
        const double *pr[3], *pc[3];
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const int q = at[b + x] < 0 ? at[b] : at[b + x];
            pr[x] = YS + (8 * (q & 15) + g.g) * py + g.t;
            pc[x] = YS + (8 * (q >> 4) + g.g) * py + g.t;
            acc[b + x][0] = acc[b + x][1] = 0.0;
        }
#pragma unroll 2
        for (int k = 0; k < ks; k++)
#pragma unroll
            for (int x = 0; x < 3; x++)
                bt_dmma(acc[b + x][0], acc[b + x][1], pr[x][4 * k], pc[x][4 * k]);
    }
    gsync(g);
#pragma unroll
    for (int x = 0; x < 9; x++) {
        if (at[x] < 0) continue;
        const int i = 8 * (at[x] & 15) + g.g, j = 8 * (at[x] >> 4) + 2 * g.t;
        *reinterpret_cast<double2 *>(YS + i * ps + j) = make_double2(acc[x][0], acc[x][1]);
        if ((at[x] & 15) != (at[x] >> 4)) {
            YS[j * ps + i] = acc[x][0];
            YS[(j + 1) * ps + i] = acc[x][1];
        }
    }
    gsync(g);
}

// Modified Gram-Schmidt of the n x r factor in place, zero columns kept zero: a
// product whose Gram is not positive definite.
__device__ __noinline__ void gmgs(int uo, int n, int r, int lt) {
    double *U = bt_sm + uo;
    if (lt == 0) {
        for (int c = 0; c < r; c++) {
            for (int p = 0; p < c; p++) {
                double d = 0.0;
                for (int i = 0; i < n; i++) d += U[u_at(i, c)] * U[u_at(i, p)];
                for (int i = 0; i < n; i++) U[u_at(i, c)] -= d * U[u_at(i, p)];
            }
            double nr = 0.0;
            for (int i = 0; i < n; i++) nr += U[u_at(i, c)] * U[u_at(i, c)];
            nr = sqrt(nr);
            for (int i = 0; i < n; i++) U[u_at(i, c)] = nr > 0 ? U[u_at(i, c)] / nr : 0.0;
        }
    }
}

// Leading subspace of S (n x n symmetric, pitch ps, whole tiles zero padded)
// from the factor U (n x r), `iters` steps of U <- orth(S U), in place.  Warp w
// owns the 8-row tiles w and w + W (n <= 64 and W >= 4, n <= 32 and W = 2, n <= 16
// and W = 1: two are enough).  It computes (S U)^T there: with U as the A operand
// a lane holds column g of Z = S U at rows 2 t, 2 t + 1, which are the fragments
// of Z^T Z as they stand (even rows one k-step, odd rows another).  Three barriers
// a step: each tile's share of the Gram (then Z takes U's place), the first warp's
// L^{-1}, the new U.  Bound by latency: a step of 40 x 4 takes about 2700 cycles alone on an SM
// with 4 warps, 3500 with four tensors on it; shuffles in place of the trip of Z
// through shared memory, or every warp factoring the sum for itself, were slower.
__device__ __noinline__ void gsubspace(int ys, int n, int ps, int uo, int r, int iters, Grp g) {
    const double *S = bt_sm + ys;
    double *U = bt_sm + uo;
    const int nt = tile8(n) / 8, m0 = g.w, m1 = g.w + g.W;
    const bool have0 = m0 < nt, have1 = m1 < nt;
    const double *s0 = S + (8 * (have0 ? m0 : 0) + g.g) * ps + g.t;
    const double *s1 = S + (8 * (have1 ? m1 : 0) + g.g) * ps + g.t;
    const double *u0 = U + u_at(g.t, g.g), *u1 = U + u_at(4 + g.t, g.g);
    double *const Li = bt_sm + g.part, *const mine = Li + g.g * 8 + 2 * g.t;
#pragma unroll 1
    for (int it = 0; it < iters; it++) {
        // Z's tiles, two chains each (even and odd k-steps); what is past n is zero.
        double z[2][2] = {}, y[2][2] = {};
        if (have0) {
#pragma unroll 1
            for (int k = 0; k < nt; k++) {
                const double a0 = u0[64 * k], a1 = u1[64 * k], b0 = s0[8 * k], b1 = s0[8 * k + 4];
                bt_dmma(z[0][0], z[0][1], a0, b0);
                bt_dmma(y[0][0], y[0][1], a1, b1);
                if (have1) {
                    const double c0 = s1[8 * k], c1 = s1[8 * k + 4];
                    bt_dmma(z[1][0], z[1][1], a0, c0);
                    bt_dmma(y[1][0], y[1][1], a1, c1);
                }
            }
        }
        double d[2][2][2] = {};
#pragma unroll
        for (int m = 0; m < 2; m++) {
#pragma unroll
            for (int q = 0; q < 2; q++) {
                z[m][q] += y[m][q];
                bt_dmma(d[m][q][0], d[m][q][1], z[m][q], z[m][q]);
            }
            if (m ? have1 : have0)
                *reinterpret_cast<double2 *>(mine + 64 * (m ? m1 : m0)) =
                    make_double2(d[m][0][0] + d[m][1][0], d[m][0][1] + d[m][1][1]);
        }
        gsync(g);
#pragma unroll
        for (int m = 0; m < 2; m++)
            if (m ? have1 : have0) {
                const int i = 8 * (m ? m1 : m0) + 2 * g.t;
                U[u_at(i, g.g)] = z[m][0];
                U[u_at(i + 1, g.g)] = z[m][1];
            }
        // The first warp adds the tiles' shares in order and factors the sum, in the
        // first share's place.
        if (g.w == 0) {
            double2 a = *reinterpret_cast<const double2 *>(mine);
#pragma unroll 4
            for (int k = 1; k < nt; k++) {
                const double2 p = *reinterpret_cast<const double2 *>(mine + 64 * k);
                a.x += p.x;
                a.y += p.y;
            }
            *reinterpret_cast<double2 *>(mine) = a;
            __syncwarp();
            double c[BMAX_R];
            const bool ok = warp_chol_linv<BMAX_R>(Li, BMAX_R, r, c);
            __syncwarp();
            // Lane j holds column j of L^{-1}; above the diagonal it holds zeros.
            const int j = 4 * g.g + g.t;
            if (j < BMAX_R) {
#pragma unroll
                for (int i = 0; i < BMAX_R; i++) Li[i * BMAX_R + j] = c[i];
            }
            if (j == 0 && !ok) Li[0] = -1.0;  // (a factor's is positive)
        }
        gsync(g);
        if (!(Li[0] > 0.0)) {
            gmgs(uo, n, r, g.lt);
            gsync(g);
            continue;
        }
        // Q^T = L^{-1} Z^T over the warp's own rows.
        const double l0 = Li[g.g * 8 + g.t], l1 = Li[g.g * 8 + 4 + g.t];
#pragma unroll
        for (int m = 0; m < 2; m++)
            if (m ? have1 : have0) {
                const int i0 = 8 * (m ? m1 : m0);
                const double b0 = U[u_at(i0 + g.g, g.t)], b1 = U[u_at(i0 + g.g, 4 + g.t)];
                double q0 = 0.0, q1 = 0.0;
                bt_dmma(q0, q1, l0, b0);
                bt_dmma(q0, q1, l1, b1);
                __syncwarp();
                U[u_at(i0 + 2 * g.t, g.g)] = q0;
                U[u_at(i0 + 2 * g.t + 1, g.g)] = q1;
            }
        gsync(g);
    }
}

// The whole HOOI of tensor t by one thread group.  `slot` is the offset of the
// group's shared-memory slice (slot_doubles(largest mode) doubles at least), `T`
// its global scratch slice.
__device__ __forceinline__ void hooi_one(const BatchArgs &a, int t, int slot, double *T,
                                         const Grp &g) {
    const int I0 = (int)a.shape[3 * t], I1 = (int)a.shape[3 * t + 1], I2 = (int)a.shape[3 * t + 2];
    const int R0 = (int)a.rank[3 * t], R1 = (int)a.rank[3 * t + 1], R2 = (int)a.rank[3 * t + 2];
    const int m = max(I0, max(I1, I2)), m8 = tile8(m);
    const int uo = slot, us = m8 * BMAX_R, ys = slot + 3 * us;
    double *U0 = bt_sm + uo, *U1 = U0 + us, *U2 = U1 + us;
    double *YS = bt_sm + ys;                      // Y_(n), then its Gram
    double *Ylast = T + (int64_t)m * m * BMAX_R;  // the final Y_(3), I2 x K
    const float *X = a.X + a.xoff[t];
    double *ug[3] = {a.U + a.uoff[3 * t], a.U + a.uoff[3 * t + 1], a.U + a.uoff[3 * t + 2]};
    for (int e = g.lt; e < 3 * m8 * BMAX_R; e += g.gs) U0[e] = 0.0;
    gsync(g);
    for (int e = g.lt; e < I0 * R0; e += g.gs) U0[u_at(e % I0, e / I0)] = ug[0][e];
    for (int e = g.lt; e < I1 * R1; e += g.gs) U1[u_at(e % I1, e / I1)] = ug[1][e];
    for (int e = g.lt; e < I2 * R2; e += g.gs) U2[u_at(e % I2, e / I2)] = ug[2][e];
    const int nx = I0 * I1 * I2;
    for (int c = g.lt; c < CLASSES; c += g.gs) {
        double s = 0.0;
#pragma unroll 8
        for (int e = c; e < nx; e += CLASSES) s = fma((double)X[e], (double)X[e], s);
        YS[c] = s;
    }
    const double x2 = gsum(YS, g);
    const int I01 = I0 * I1, I12 = I1 * I2;
    for (int sw = 0; sw < a.sweeps; sw++) {
        // T = X x_3 U_3^T  (I0 x I1 x R2): rows (i0, i1).
        contract<float>(X, I01, 1, 1, 0, I2, I01, uo + 2 * us, T, 1, I01, 0, R2, g);
        // Modes 1 and 2 from T: Y_(1)[i0, r1 + R1 r2], Y_(2)[i1, r0 + R0 r2].
#pragma unroll 1
        for (int n = 0; n < 2; n++) {
            const int I = n ? I1 : I0, R = n ? R0 : R1, K = R * R2, py = pitch16(K);
            const int ps = pitch16(tile8(I));
            gsync(g);
            zero_pads(YS, I, K, py, g);
            contract<double>(T, I, n ? I0 : 1, R2, I01, n ? I0 : I1, n ? 1 : I0, n ? uo : uo + us, YS,
                             py, 1, R, R, g);
            gsync(g);
            ggram(ys, I, K, py, ps, g);
            gsubspace(ys, I, ps, n ? uo + us : uo, n ? R1 : R0, a.inner, g);
        }
        // Mode 3 from X: T2[i1, i2, r0] = X x_1 U0^T, rows (i1, i2), then
        // Y_(3)[i2, r0 + R0 r1] = sum_i1 T2[i1, i2, r0] U1[i1, r1], rows i2.
        contract<float>(X, I12, I0, 1, 0, I0, 1, uo, T, 1, I12, 0, R0, g);
        gsync(g);
        const int K = R0 * R1, py = pitch16(K);
        zero_pads(YS, I2, K, py, g);
        contract<double>(T, I2, I1, R0, I12, I1, 1, uo + us, YS, py, R0, 1, R1, g);
        gsync(g);
        if (sw == a.sweeps - 1)
            for (int e = g.lt; e < I2 * K; e += g.gs) Ylast[e] = YS[(e % I2) * py + e / I2];
        ggram(ys, I2, K, py, pitch16(tile8(I2)), g);
        gsubspace(ys, I2, pitch16(tile8(I2)), uo + 2 * us, R2, a.inner, g);
    }
    // Core G[k + K r2] = sum_i2 Y_(3)[i2, k] U2[i2, r2] (the last Y_(3) and U2
    // are those of the final sweep), relative error in FP64.
    const int K = R0 * R1;
    double *Gout = a.G + a.goff[t];
    for (int e = g.lt; e < K * R2; e += g.gs) {
        const int k = e % K, r2 = e / K;
        double acc = 0.0;
        for (int i2 = 0; i2 < I2; i2++) acc = fma(Ylast[i2 + I2 * k], U2[u_at(i2, r2)], acc);
        Gout[e] = acc;
        YS[e] = acc * acc;  // at most 512 entries
    }
    for (int e = K * R2 + g.lt; e < CLASSES; e += g.gs) YS[e] = 0.0;
    const double g2 = gsum(YS, g);
    // A non-finite input gives a NaN error (fmax would turn NaN into 0).
    const double q = 1.0 - g2 / x2;
    if (g.lt == 0) a.relerr[t] = isnan(q) ? q : sqrt(fmax(0.0, q));
    for (int e = g.lt; e < I0 * R0; e += g.gs) ug[0][e] = U0[u_at(e % I0, e / I0)];
    for (int e = g.lt; e < I1 * R1; e += g.gs) ug[1][e] = U1[u_at(e % I1, e / I1)];
    for (int e = g.lt; e < I2 * R2; e += g.gs) ug[2][e] = U2[u_at(e % I2, e / I2)];
}

template <int NT>
__global__ void __launch_bounds__(NT, 512 / NT) batched_hooi_kernel(const BatchArgs *__restrict__ ap) {
    __shared__ int cur;
    const BatchArgs a = *ap;
    double *scr = a.scratch + (int64_t)blockIdx.x * SCR;
    for (;;) {
        if (threadIdx.x == 0) cur = atomicAdd(a.queue, 1);
        __syncthreads();
        const int it = cur;
        __syncthreads();
        if (it >= a.nitems) break;
        const Item item = a.items[it];
        const int gsz = NT / item.g;
        const int gid = threadIdx.x / gsz;
        const int lt = (int)threadIdx.x % gsz, lane = lt & 31;
        const Grp g{lt, gsz, 1 + gid, lt >> 5, gsz >> 5, lane >> 2, lane & 3,
                    SLOT_ALL + gid * (gsz >> 5) * WARP_SCR};
        const int t = item.t[gid];
        if (t >= 0)
            hooi_one(a, t, (SLOT_ALL / item.g / 2 * 2) * gid, scr + (SCR / item.g) * gid, g);
        __syncthreads();
    }
}

size_t batched_smem(int nt) { return ((size_t)SLOT_ALL + nt / 32 * WARP_SCR) * sizeof(double); }

template <int NT>
void kernel_attrs(dt_ctx *ctx, int *per_sm) {
    smem_limit(ctx, batched_hooi_kernel<NT>, batched_smem(NT));
    DT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, batched_hooi_kernel<NT>, NT,
                                                          batched_smem(NT)));
}

// Resident CTAs per SM x SMs for a block size.
unsigned batched_grid(dt_ctx *ctx, int nt) {
    int per_sm = 1;
    if (nt == 128)
        kernel_attrs<128>(ctx, &per_sm);
    else if (nt == 512)
        kernel_attrs<512>(ctx, &per_sm);
    else
        kernel_attrs<256>(ctx, &per_sm);
    return (unsigned)(std::max(1, per_sm) * ctx->num_sms);
}

void enqueue_kernel(dt_ctx *ctx, int nt, unsigned grid, const BatchArgs *dargs, int *queue) {
    DT_CUDA(cudaMemsetAsync(queue, 0, sizeof(int), ctx->stream));
    const size_t smem = batched_smem(nt);
    if (nt == 128)
        DT_LAUNCH(ctx, batched_hooi_kernel<128>, grid, 128, smem, dargs);
    else if (nt == 512)
        DT_LAUNCH(ctx, batched_hooi_kernel<512>, grid, 512, smem, dargs);
    else
        DT_LAUNCH(ctx, batched_hooi_kernel<256>, grid, 256, smem, dargs);
}

// Estimated cost of one tensor's sweep (FP64 FMAs): the two passes over X, the
// small contractions, the Grams and the subspace steps.
double tensor_cost(const int64_t *I, const int64_t *R, int inner) {
    const double x = (double)I[0] * I[1] * I[2];
    double c = x * (R[2] + R[0]);
    c += (double)I[0] * I[1] * R[2] * (R[1] + R[0]) + (double)R[0] * I[1] * I[2] * R[1];
    for (int n = 0; n < 3; n++) {
        const double K = (double)R[(n + 1) % 3] * R[(n + 2) % 3];
        c += (double)I[n] * I[n] * K * 0.5 + inner * (double)I[n] * I[n] * R[n] * 2.0;
    }
    return c;
}

// Packs tensors (sorted by cost, descending) into items.  pack >= 1 pairs
// tensors with largest mode <= PAIR_MAX_I, pack >= 2 puts those with largest
// mode <= QUAD_MAX_I four to an item.  Items come out cost-descending.
std::vector<Item> make_items(const std::vector<int> &order, const std::vector<double> &cost,
                             const std::vector<int> &maxI, int pack) {
    std::vector<std::pair<double, Item>> v;
    std::vector<int> pairs, quads;
    for (int t : order) {
        if (pack >= 2 && maxI[t] <= QUAD_MAX_I)
            quads.push_back(t);
        else if (pack >= 1 && maxI[t] <= PAIR_MAX_I)
            pairs.push_back(t);
        else
            v.push_back({cost[t], Item{1, {t, -1, -1, -1}}});
    }
    auto group = [&](const std::vector<int> &ts, int g) {
        for (size_t i = 0; i < ts.size(); i += g) {
            Item it{g, {-1, -1, -1, -1}};
            double c = 0.0;
            for (int k = 0; k < g && i + k < ts.size(); k++) {
                it.t[k] = ts[i + k];
                c = std::max(c, cost[ts[i + k]]);
            }
            // A group of g shares the CTA: it runs about as long as its most
            // expensive member with g times fewer threads.
            v.push_back({c * g, it});
        }
    };
    group(pairs, 2);
    group(quads, 4);
    std::stable_sort(v.begin(), v.end(),
                     [](const std::pair<double, Item> &a, const std::pair<double, Item> &b) {
                         return a.first > b.first;
                     });
    std::vector<Item> out;
    out.reserve(v.size());
    for (auto &p : v) out.push_back(p.second);
    return out;
}

}  // namespace

// Per-context state: tuned configurations per batch signature, the
// instantiated graphs per launch shape, and the device buffers they read.
struct BatchedState {
    std::map<std::vector<int64_t>, std::pair<int, int>> tuned;  // -> (threads, pack)
    std::map<std::pair<int, unsigned>, cudaGraphExec_t> graphs;  // (threads, grid)
    DevMem args, queue, scratch, tables;
    size_t tables_bytes = 0;
    unsigned scratch_grid = 0;
    ~BatchedState() {
        for (auto &kv : graphs) cudaGraphExecDestroy(kv.second);
    }
};

bool release_batched_scratch(dt_ctx *ctx) {
    if (ctx->batched.use_count() != 1) return false;  // none, or a running call's
    BatchedState &st = *std::static_pointer_cast<BatchedState>(ctx->batched);
    if (!st.scratch.get()) return false;
    DT_CUDA(cudaStreamSynchronize(ctx->stream));
    st.scratch.release();
    st.scratch_grid = 0;
    return true;
}

}  // namespace dt

using namespace dt;

extern "C" {

int dt_hooi_batched(dt_ctx *ctx, int count, const int64_t *shapes, const int64_t *ranks,
                    const float *X, const int64_t *x_offsets, int sweeps, int inner_iters,
                    double *U, const int64_t *u_offsets, double *G, const int64_t *g_offsets,
                    double *relerr, int block_threads, dt_batched_report *report) {
    return guard([&] {
        check_ctx(ctx);
        DT_CHECK_ARG(count >= 1 && shapes && ranks && X && x_offsets && U && u_offsets && G &&
                         g_offsets && relerr,
                     "dt_hooi_batched: bad arguments");
        DT_CHECK_ARG(sweeps >= 1 && inner_iters >= 1, "dt_hooi_batched: sweeps/inner must be >= 1");
        DT_CHECK_ARG(block_threads == 0 || block_threads == 128 || block_threads == 256 ||
                         block_threads == 512,
                     "dt_hooi_batched: block_threads must be 0 (autotune), 128, 256 or 512");
        int64_t xn = 0, un = 0, gn = 0;
        int64_t maxI = 0, maxR = 0;
        std::vector<double> cost(count);
        std::vector<int> tmaxI(count);
        int n_pair = 0, n_quad = 0;
        for (int t = 0; t < count; t++) {
            int64_t xs = 1, gs = 1, mi = 0;
            for (int m = 0; m < 3; m++) {
                const int64_t I = shapes[3 * t + m], R = ranks[3 * t + m];
                DT_CHECK_ARG(I >= 1 && I <= BMAX_I && R >= 1 && R <= BMAX_R && R <= I,
                             "dt_hooi_batched: tensor %d mode %d: need 1 <= R <= I, I <= %d, R <= %d",
                             t, m, BMAX_I, BMAX_R);
                DT_CHECK_ARG(u_offsets[3 * t + m] >= 0, "dt_hooi_batched: negative U offset");
                xs *= I;
                gs *= R;
                un = std::max(un, u_offsets[3 * t + m] + I * R);
                mi = std::max(mi, I);
                maxR = std::max(maxR, R);
            }
            DT_CHECK_ARG(x_offsets[t] >= 0 && g_offsets[t] >= 0,
                         "dt_hooi_batched: negative X or G offset");
            maxI = std::max(maxI, mi);
            tmaxI[t] = (int)mi;
            n_pair += mi <= PAIR_MAX_I;
            n_quad += mi <= QUAD_MAX_I;
            cost[t] = tensor_cost(shapes + 3 * t, ranks + 3 * t, inner_iters);
            xn = std::max(xn, x_offsets[t] + xs);
            gn = std::max(gn, g_offsets[t] + gs);
        }
        std::vector<int> order(count);
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(),
                         [&](int a, int b) { return cost[a] > cost[b]; });
        const std::vector<int64_t> sig = {count, maxI, maxR, sweeps, inner_iters, n_pair, n_quad};
        DT_CUDA(cudaSetDevice(ctx->device));
        if (!ctx->batched) ctx->batched = std::make_shared<BatchedState>();
        const auto state = std::static_pointer_cast<BatchedState>(ctx->batched);
        BatchedState &st = *state;
        DevView xv(ctx, X, xn * sizeof(float), true, false);
        DevView uv(ctx, U, un * sizeof(double), true, true);
        DevView gv(ctx, G, gn * sizeof(double), false, true);
        DevView ev(ctx, relerr, count * sizeof(double), false, true);
        if (!st.args.get()) st.args.alloc(ctx, sizeof(BatchArgs));
        if (!st.queue.get()) st.queue.alloc(ctx, sizeof(int));
        const int64_t launches0 = ctx->launches;

        // Descriptor tables (shapes, ranks, offsets, items) in one device
        // buffer kept on the context; `items` is rebuilt per configuration.
        auto upload = [&](const std::vector<Item> &items, BatchArgs &a) {
            const size_t n3 = 3 * (size_t)count;
            const size_t bytes = (3 * n3 + 2 * (size_t)count) * sizeof(int64_t) +
                                 items.size() * sizeof(Item);
            std::vector<char> h(bytes);
            int64_t *p = reinterpret_cast<int64_t *>(h.data());
            std::memcpy(p, shapes, n3 * sizeof(int64_t));
            std::memcpy(p + n3, ranks, n3 * sizeof(int64_t));
            std::memcpy(p + 2 * n3, u_offsets, n3 * sizeof(int64_t));
            std::memcpy(p + 3 * n3, x_offsets, count * sizeof(int64_t));
            std::memcpy(p + 3 * n3 + count, g_offsets, count * sizeof(int64_t));
            std::memcpy(p + 3 * n3 + 2 * count, items.data(), items.size() * sizeof(Item));
            if (st.tables_bytes < bytes) {
                st.tables_bytes = 0;  // (also when the allocation fails)
                st.tables.alloc(ctx, bytes);
                st.tables_bytes = bytes;
            }
            DT_CUDA(cudaMemcpyAsync(st.tables.get(), h.data(), bytes, cudaMemcpyHostToDevice,
                                    ctx->stream));
            const int64_t *d = st.tables.as<int64_t>();
            a.count = count;
            a.nitems = (int)items.size();
            a.shape = d;
            a.rank = d + n3;
            a.uoff = d + 2 * n3;
            a.xoff = d + 3 * n3;
            a.goff = d + 3 * n3 + count;
            a.items = reinterpret_cast<const Item *>(d + 3 * n3 + 2 * count);
            // The host copy must outlive the asynchronous copy from pageable
            // memory only until the call returns; the runtime stages it.
            DT_CUDA(cudaStreamSynchronize(ctx->stream));
        };
        // Scratch for `grid` CTAs, or for as many as there is room for; how many.
        auto with_scratch = [&](unsigned grid) {
            if (st.scratch_grid >= grid) return grid;
            st.scratch_grid = 0;
            while (!st.scratch.try_alloc(ctx, (size_t)grid * SCR * sizeof(double))) {
                if (grid == 1) st.scratch.alloc(ctx, SCR * sizeof(double));  // (fails)
                grid = std::max(1u, grid * 3 / 4);
            }
            st.scratch_grid = grid;
            return grid;
        };
        BatchArgs base{};
        base.X = xv.as<float>();
        base.G = gv.as<double>();
        base.relerr = ev.as<double>();
        base.sweeps = sweeps;
        base.inner = inner_iters;
        base.queue = st.queue.as<int>();

        int nt = block_threads, pack = 0;
        int timed = 0;
        double tune_best = 0.0, tune_worst = 0.0;
        if (nt != 0) {
            pack = 2;  // pairs and quads where they fit; no autotuning
        } else {
            auto itc = st.tuned.find(sig);
            if (itc != st.tuned.end()) {
                nt = itc->second.first;
                pack = itc->second.second;
            } else {
                // Autotune on a stratified sample (every k-th tensor of the
                // cost order) with a scratch copy of U.  The sample must fill
                // the largest grid several times over, or configurations with
                // few large CTAs win on the sample and lose on the batch: up
                // to 8192 tensors, the whole batch is timed.
                const int sample = std::min(count, 8192);
                std::vector<int> sord;
                for (int i = 0; i < sample; i++)
                    sord.push_back(order[(int64_t)i * count / sample]);
                DevMem ucopy(ctx, un * sizeof(double));
                float best = 1e30f, worst = 0.f;
                const int cand_nt[3] = {128, 256, 512};
                for (int c = 0; c < 3; c++) {
                    for (int pk = 0; pk <= 2; pk++) {
                        if (pk == 1 && n_pair == 0) continue;
                        if (pk == 2 && n_quad == 0) continue;
                        BatchArgs b = base;
                        upload(make_items(sord, cost, tmaxI, pk), b);
                        b.U = ucopy.as<double>();
                        const unsigned grid = with_scratch(batched_grid(ctx, cand_nt[c]));
                        b.scratch = st.scratch.as<double>();
                        DT_CUDA(cudaMemcpyAsync(st.args.get(), &b, sizeof(b),
                                                cudaMemcpyHostToDevice, ctx->stream));
                        float ms = 0.f;
                        for (int rep = 0; rep < 2; rep++) {  // warm, then timed
                            DT_CUDA(cudaMemcpyAsync(ucopy.get(), uv.ptr(), un * sizeof(double),
                                                    cudaMemcpyDeviceToDevice, ctx->stream));
                            DT_CUDA(cudaEventRecord(ctx->ev_start, ctx->stream));
                            enqueue_kernel(ctx, cand_nt[c], grid, st.args.as<BatchArgs>(),
                                           st.queue.as<int>());
                            DT_CUDA(cudaEventRecord(ctx->ev_stop, ctx->stream));
                            DT_CUDA(cudaEventSynchronize(ctx->ev_stop));
                            DT_CUDA(cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
                        }
                        timed++;
                        worst = std::max(worst, ms);
                        if (ms < best) {
                            best = ms;
                            nt = cand_nt[c];
                            pack = pk;
                        }
                    }
                }
                tune_best = best;
                tune_worst = worst;
                st.tuned[sig] = {nt, pack};
            }
        }
        const unsigned grid = with_scratch(batched_grid(ctx, nt));
        const std::vector<Item> items = make_items(order, cost, tmaxI, pack);
        BatchArgs a = base;
        upload(items, a);
        a.U = uv.as<double>();
        a.scratch = st.scratch.as<double>();
        DT_CUDA(cudaMemcpyAsync(st.args.get(), &a, sizeof(a), cudaMemcpyHostToDevice,
                                ctx->stream));
        // The graph (queue reset + persistent kernel) for this launch shape:
        // captured once, replayed by every later call.
        const std::pair<int, unsigned> gkey(nt, grid);
        int reused = 1;
        // Streams that cannot be captured (the legacy and per-thread default
        // streams) run the launch directly.
        const bool capturable = ctx->stream != nullptr && ctx->stream != cudaStreamLegacy &&
                                ctx->stream != cudaStreamPerThread;
        if (!capturable) {
            DT_CUDA(cudaEventRecord(ctx->ev_start, ctx->stream));
            enqueue_kernel(ctx, nt, grid, st.args.as<BatchArgs>(), st.queue.as<int>());
            DT_CUDA(cudaEventRecord(ctx->ev_stop, ctx->stream));
            reused = 0;
        }
        auto itg = capturable ? st.graphs.find(gkey) : st.graphs.end();
        if (capturable && itg == st.graphs.end()) {
            reused = 0;
            cudaGraph_t graph;
            cudaGraphExec_t exec;
            DT_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
            const int64_t l0 = ctx->launches;
            try {
                enqueue_kernel(ctx, nt, grid, st.args.as<BatchArgs>(), st.queue.as<int>());
            } catch (...) {
                cudaStreamEndCapture(ctx->stream, &graph);
                throw;
            }
            ctx->launches = l0;  // counted when the graph is launched
            DT_CUDA(cudaStreamEndCapture(ctx->stream, &graph));
            const cudaError_t ie = cudaGraphInstantiate(&exec, graph, 0);
            cudaGraphDestroy(graph);
            DT_CUDA(ie);
            itg = st.graphs.emplace(gkey, exec).first;
        }
        if (capturable) {
            DT_CUDA(cudaEventRecord(ctx->ev_start, ctx->stream));
            DT_CUDA(cudaGraphLaunch(itg->second, ctx->stream));
            ctx->launches++;
            DT_CUDA(cudaEventRecord(ctx->ev_stop, ctx->stream));
        }
        DT_CUDA(cudaStreamSynchronize(ctx->stream));
        float ms = 0.f;
        DT_CUDA(cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
        uv.finish();
        gv.finish();
        ev.finish();
        if (report) {
            std::memset(report, 0, sizeof(*report));
            report->device_ms = ms;
            report->block_threads = nt;
            report->grid = (int)grid;
            report->kernel_launches = (int)(ctx->launches - launches0);
            report->pack = pack;
            report->items = (int)items.size();
            report->candidates_timed = timed;
            report->tune_best_ms = tune_best;
            report->tune_worst_ms = tune_worst;
            report->graph_reused = reused;
        }
    });
}

}  // extern "C"
