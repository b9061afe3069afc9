// Small dense FP64 linear algebra on the GPU: the reference's LAPACK calls
// (src/operator/operator_double.cpp:84-155) and its ALS_ leading-subspace step
// (template/algorithm/tucker/hooi_als.tpp:7-34), kept on the device so a HOOI
// sweep never round-trips to the host.  These matrices are tiny (R x R, I_n x R,
// I_n x I_n): one CTA or one cluster per problem, latency-bound, so the code
// shortens dependency chains and barriers rather than saving flops.
#include <vector>

#include "dt_kernels.cuh"

namespace dt {
namespace {

constexpr int LA_NT = 512;

__device__ double block_sum(double v, double *red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        v = l < (int)(blockDim.x >> 5) ? red[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (l == 0) red[32] = v;
    }
    __syncthreads();
    return red[32];
}

// Householder QR of the m x n col-major W (in place: R in the upper triangle,
// reflector tails below the diagonal, tau[j]), then Q (m x n) formed by
// applying H_0 ... H_{n-1} to [I; 0] backwards -- the dgeqrf/dorgqr sequence.
// Reflector (dlarfg): beta = -sign(alpha) ||(alpha, x)||, tau = (beta-alpha)/beta,
// v = [1; x/(alpha-beta)]; tau = 0 when x == 0.
__device__ void hqr_device(double *W, int64_t m, int64_t n, double *tau, double *Q,
                           double *red) {
    const int t = threadIdx.x;
    const int warp = t >> 5, lane = t & 31, nwarps = blockDim.x >> 5;
    for (int64_t j = 0; j < n; j++) {
        double *col = W + j * m;
        double s = 0.0;
        for (int64_t i = j + 1 + t; i < m; i += blockDim.x) s = fma(col[i], col[i], s);
        const double xnorm2 = block_sum(s, red);
        const double alpha = col[j];
        double tj, scale;
        if (xnorm2 == 0.0) {
            tj = 0.0;
            scale = 0.0;
        } else {
            const double beta = -copysign(sqrt(alpha * alpha + xnorm2), alpha);
            tj = (beta - alpha) / beta;
            scale = 1.0 / (alpha - beta);
        }
        __syncthreads();
        if (tj != 0.0) {
            for (int64_t i = j + 1 + t; i < m; i += blockDim.x) col[i] *= scale;
        }
        __syncthreads();
        if (t == 0) {
            tau[j] = tj;
            if (tj != 0.0) col[j] = -copysign(sqrt(alpha * alpha + xnorm2), alpha);
        }
        // Apply H_j to the trailing columns, one warp per column.
        if (tj != 0.0) {
            for (int64_t c = j + 1 + warp; c < n; c += nwarps) {
                double *cc = W + c * m;
                const double cj = cc[j];  // read before lane 0 rewrites it
                double w = 0.0;
                for (int64_t i = j + 1 + lane; i < m; i += 32) w = fma(col[i], cc[i], w);
                for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
                w += cj;
                w *= tj;
                if (lane == 0) cc[j] -= w;
                for (int64_t i = j + 1 + lane; i < m; i += 32) cc[i] = fma(-w, col[i], cc[i]);
            }
        }
        __syncthreads();
    }
    if (!Q) return;
    for (int64_t e = t; e < m * n; e += blockDim.x) {
        const int64_t i = e % m, c = e / m;
        Q[e] = (i == c) ? 1.0 : 0.0;
    }
    __syncthreads();
    for (int64_t j = n - 1; j >= 0; j--) {
        const double tj = tau[j];
        if (tj != 0.0) {
            const double *v = W + j * m;
            for (int64_t c = j + warp; c < n; c += nwarps) {
                double *qc = Q + c * m;
                const double qj = qc[j];  // read before lane 0 rewrites it
                double w = 0.0;
                for (int64_t i = j + 1 + lane; i < m; i += 32) w = fma(v[i], qc[i], w);
                for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
                w += qj;
                w *= tj;
                if (lane == 0) qc[j] -= w;
                for (int64_t i = j + 1 + lane; i < m; i += 32) qc[i] = fma(-w, v[i], qc[i]);
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(LA_NT) hqr_kernel(const double *A, int64_t m, int64_t n,
                                                    double *Q, double *R, double *work) {
    __shared__ double red[33];
    double *W = work;
    double *tau = work + m * n;
    for (int64_t e = threadIdx.x; e < m * n; e += blockDim.x) W[e] = A[e];
    __syncthreads();
    hqr_device(W, m, n, tau, Q, red);
    if (R) {
        for (int64_t e = threadIdx.x; e < n * n; e += blockDim.x) {
            const int64_t i = e % n, c = e / n;
            R[e] = (i <= c) ? W[i + c * m] : 0.0;
        }
    }
}

// Cholesky G = R^T R of the r x r SPD matrix in smem (row-major G[i*r+c]), R in
// G's place, by one warp.  Lane c keeps column c in registers and rows are
// exchanged with shuffles, so the r pivots form one short dependency chain (one
// sqrt and one reciprocal per pivot).  Returns false on a non-positive pivot.
// Runs in warp 0 only; r <= 32.
template <int RMAX>
__device__ bool warp_chol(double *G, int r) {
    const int lane = threadIdx.x & 31;
    double g[RMAX];
#pragma unroll
    for (int i = 0; i < RMAX; i++) g[i] = (i < r && lane < r) ? G[i * r + lane] : 0.0;
    const double g00 = __shfl_sync(0xffffffffu, g[0], 0);
    bool ok = true;
#pragma unroll
    for (int k = 0; k < RMAX; k++) {
        if (k >= r) break;
        const double d = __shfl_sync(0xffffffffu, g[k], k);
        if (!(d > 1e-28 * g00)) ok = false;
        const double rkk = sqrt(fmax(d, 1e-300));
        const double inv = 1.0 / rkk;
        if (lane > k) g[k] *= inv;
        if (lane == k) g[k] = rkk;
#pragma unroll
        for (int i = k + 1; i < RMAX; i++) {
            if (i >= r) break;
            const double rki = __shfl_sync(0xffffffffu, g[k], i);
            if (lane >= i) g[i] = fma(-rki, g[k], g[i]);
        }
    }
    if (lane < r) {
#pragma unroll
        for (int i = 0; i < RMAX; i++)
            if (i < r) G[i * r + lane] = i <= lane ? g[i] : 0.0;
    }
    __syncwarp();
    return ok;
}

// Subspace iteration L <- orth(S L), `iters` times, one CTA: more than 256 rows (fewer
// go to subspace_cluster_kernel), up to 32 columns.  S (n x n, symmetric) is read
// from L2 for every product, which bounds it (n = 256, before the cluster kernel took
// that size: 112 us for 12 columns and 5 steps); L and Z (n x r) live in shared memory
// when they fit.  Intermediate steps orthonormalise with one CholeskyQR pass (only
// conditioning matters there), the last step with two (CholeskyQR2, orthonormal to
// FP64 rounding); a Cholesky breakdown (rank-deficient S L) switches that step to
// Householder.

// Forward substitution Q[i, :] = Z[i, :] R^{-1} for every row i (R upper,
// row-major r x r in smem, Rinv_diag its reciprocal diagonal), one thread per
// row: the r-step chain runs on 96+ rows at once instead of one warp.
__device__ __forceinline__ void rows_trsm(const double *Z, double *Q, int64_t n, int64_t r,
                                          const double *R) {
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        double q[32];
#pragma unroll
        for (int c = 0; c < 32; c++) {
            if (c >= r) break;
            double acc = Z[i + c * n];
#pragma unroll
            for (int k = 0; k < 32; k++) {
                if (k >= c) break;
                acc = fma(-q[k], R[k * r + c], acc);
            }
            q[c] = acc / R[c * r + c];
            Q[i + c * n] = q[c];
        }
    }
}

template <int RMAX>
__global__ void __launch_bounds__(LA_NT) subspace_kernel(const double *S, int64_t n,
                                                         double *Lg, int64_t r, int iters,
                                                         double *work, int zl_in_smem,
                                                         int *flag) {
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[33];
    __shared__ int bad;
    const int t = threadIdx.x;
    double *G = sm;  // r*r
    double *L, *Z;
    if (zl_in_smem) {
        L = sm + r * r;
        Z = L + n * r;
    } else {
        L = work;
        Z = work + n * r;
    }
    double *hwork = work + 2 * n * r;  // n*r + r for the Householder fallback
    for (int64_t e = t; e < n * r; e += blockDim.x) L[e] = Lg[e];
    __syncthreads();
    const int64_t cgroups = (r + 3) / 4;
    const int npairs = (int)(r * (r + 1) / 2);

    // One CholeskyQR pass: dst = orth(src) through G = src^T src = R^T R.
    auto cholqr = [&](const double *src, double *dst) -> bool {
        for (int task = t; task < 4 * ((npairs + 7) / 8) * 8; task += blockDim.x) {
            const int pr = task >> 2, part = task & 3;
            double sacc = 0.0;
            int a = 0, b = 0;
            if (pr < npairs) {
                int rem = pr;
                while (rem >= (int)r - a) {
                    rem -= (int)r - a;
                    a++;
                }
                b = a + rem;
                const double *ca = src + (int64_t)a * n, *cb = src + (int64_t)b * n;
                for (int64_t k = part; k < n; k += 4) sacc = fma(ca[k], cb[k], sacc);
            }
            sacc += __shfl_xor_sync(0xffffffffu, sacc, 1);
            sacc += __shfl_xor_sync(0xffffffffu, sacc, 2);
            if (pr < npairs && part == 0) {
                G[a * r + b] = sacc;
                G[b * r + a] = sacc;
            }
        }
        __syncthreads();
        if (t < 32) {
            const bool ok = warp_chol<RMAX>(G, (int)r);
            if (t == 0) bad = ok ? 0 : 1;
        }
        __syncthreads();
        if (bad) return false;
        rows_trsm(src, dst, n, r, G);
        __syncthreads();
        return true;
    };

    // span(S^iters L): products Z <- S Z, orthonormalised after the second
    // product (conditioning stays within (l1/lr)^2) and at the end (two passes).
    bool broke = false;
    double *cur_in = L, *cur_out = Z;
    for (int it = 0; it < iters && !broke; it++) {
        for (int64_t task = t; task < n * cgroups; task += blockDim.x) {
            const int64_t i = task % n, c0 = 4 * (task / n);
            double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
            const double *l0 = cur_in + c0 * n;
            const bool h1 = c0 + 1 < r, h2 = c0 + 2 < r, h3 = c0 + 3 < r;
#pragma unroll 4
            for (int64_t k = 0; k < n; k++) {
                const double sv = S[i + n * k];
                a0 = fma(sv, l0[k], a0);
                if (h1) a1 = fma(sv, l0[k + n], a1);
                if (h2) a2 = fma(sv, l0[k + 2 * n], a2);
                if (h3) a3 = fma(sv, l0[k + 3 * n], a3);
            }
            cur_out[i + c0 * n] = a0;
            if (h1) cur_out[i + (c0 + 1) * n] = a1;
            if (h2) cur_out[i + (c0 + 2) * n] = a2;
            if (h3) cur_out[i + (c0 + 3) * n] = a3;
        }
        __syncthreads();
        double *tmp = cur_in;
        cur_in = cur_out;
        cur_out = tmp;
        const bool last = it == iters - 1;
        if (last || (it % 2) == 1) {
            // cur_in holds the product; orthonormalise into cur_out, then back.
            if (!cholqr(cur_in, cur_out)) {
                broke = true;
                break;
            }
            if (last) {
                if (!cholqr(cur_out, cur_in)) {
                    broke = true;
                    break;
                }
            } else {
                tmp = cur_in;
                cur_in = cur_out;
                cur_out = tmp;
            }
        }
    }
    if (broke) {
        // Rank-deficient or badly conditioned: restart from the caller's L and
        // run every step with Householder orthonormalisation.
        for (int64_t e = t; e < n * r; e += blockDim.x) L[e] = Lg[e];
        __syncthreads();
        for (int it = 0; it < iters; it++) {
            for (int64_t e = t; e < n * r; e += blockDim.x) {
                const int64_t i = e % n, c = e / n;
                double acc = 0.0;
                for (int64_t k = 0; k < n; k++) acc = fma(S[i + n * k], L[k + c * n], acc);
                hwork[e] = acc;
            }
            __syncthreads();
            hqr_device(hwork, n, r, hwork + n * r, L, red);
            __syncthreads();
        }
        if (t == 0 && flag) atomicOr(flag, 2);
        for (int64_t e = t; e < n * r; e += blockDim.x) Lg[e] = L[e];
        return;
    }
    for (int64_t e = t; e < n * r; e += blockDim.x) Lg[e] = cur_in[e];
}

// ---------------------------------------------------------------------------
// Subspace iteration on the FP64 tensor-core path (mma.sync m8n8k4 .f64) for
// n <= 256 and r <= RT (8, 16 or 32), one thread-block cluster of C CTAs of 8
// warps.  One SM's FP64 rate bounds a product S Z (96 x 96 x 16: 2300 cycles
// at 64 FMA a cycle) and its shared memory holds S up to n = 130 only, so the
// rows are dealt out: each CTA keeps its rows of S (S is symmetric: its
// columns, contiguous in memory) in shared memory, computes its rows of every
// product from its own full copy of Z and sends them to all CTAs.  The r x r
// Gram, its factorisation by one warp and Z R^{-1} are small and done by every
// CTA alike, so rows of products are all that crosses SMs.  Each sum is taken
// in the order that one CTA would take: the results do not depend on the
// cluster's size.  Same schedule as subspace_kernel: CholeskyQR after every
// second product, CholeskyQR and a correction after the last.  Z goes through a
// ring of three buffers, so a CTA may send its rows of the next product while
// another still applies R^{-1}; with two (a third does not fit) a cluster
// barrier follows R^{-1}.  Shared-memory layout:
//  * the CTA's rows of S with a pitch = 4 (mod 16) and Z, Q row-major n8 x RT
//    with pitch RT + 4: the 8 x 4 and 4 x 8 operand fragments then hit 16
//    distinct 8-byte bank pairs per half-warp;
//  * rows n..n8-1 and columns r..RT-1 are zero padding, so every product,
//    Gram and solve runs on whole 8 x 8 tiles.
// A Cholesky breakdown restarts from the caller's L with Householder steps, on
// the first CTA alone.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void la_cp_async16(void *smem, const void *gmem) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem) : "memory");
}
__device__ __forceinline__ void la_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void la_cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A batch of matrices as a kernel argument (no table to copy to the device
// and keep until the kernel is done).
constexpr int ORTH_MAX = 16;
struct OrthTable {
    const double *A[ORTH_MAX];
    double *Q[ORTH_MAX];
    double *work[ORTH_MAX];  // m n + n doubles each
    int64_t m[ORTH_MAX], n[ORTH_MAX];
};

constexpr int SM_WARPS = 8;
constexpr int SM_NT = SM_WARPS * 32;
constexpr int SM_GP = 512;  // doubles of Gram partials (K split only below 8 tiles)

__device__ __forceinline__ void dmma884(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

template <int RT>
struct SmTile {
    static constexpr int LDQ = RT + 4;  // Z / Q pitch (= 4 mod 16 for RT in {16, 32}; 12 for 8)
    static constexpr int LDR = RT + 4;  // R^{-1} pitch
    static constexpr int NT = RT / 8;   // n-tiles
};

// dst = src Ri   (n8 x RT times RT x RT upper).
template <int RT>
__device__ __forceinline__ void sm_apply(const double *src, const double *Ri, int n8,
                                         double *dst) {
    using T = SmTile<RT>;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int mtiles = n8 / 8;
    for (int mt = w; mt < mtiles; mt += SM_WARPS) {
        double acc[T::NT][2];
#pragma unroll
        for (int j = 0; j < T::NT; j++) acc[j][0] = acc[j][1] = 0.0;
        const int row = 8 * mt + g;
#pragma unroll
        for (int kk = 0; kk < RT / 4; kk++) {
            const double a = src[row * T::LDQ + 4 * kk + t];
#pragma unroll
            for (int j = 0; j < T::NT; j++)
                dmma884(acc[j][0], acc[j][1], a, Ri[(4 * kk + t) * T::LDR + 8 * j + g]);
        }
#pragma unroll
        for (int j = 0; j < T::NT; j++)
            *reinterpret_cast<double2 *>(dst + row * T::LDQ + 8 * j + 2 * t) =
                make_double2(acc[j][0], acc[j][1]);
    }
}

// G = src^T src (RT x RT row-major); rows/columns >= r replaced by the identity.
template <int RT>
__device__ __forceinline__ void sm_gram(const double *src, int n, int r, double *Gp, double *G) {
    using T = SmTile<RT>;
    constexpr int TILES = T::NT * T::NT;
    constexpr int KSP = TILES >= SM_WARPS ? 1 : SM_WARPS / TILES;
    static_assert(KSP == 1 || KSP * RT * RT <= SM_GP, "Gram partials");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int ksteps = (n + 3) / 4;
    if (KSP == 1) {
        for (int tt = w; tt < TILES; tt += SM_WARPS) {
            const int ta = tt % T::NT, tb = tt / T::NT;
            double d0 = 0.0, d1 = 0.0;
            for (int kk = 0; kk < ksteps; kk++) {
                const int k = 4 * kk + t;
                dmma884(d0, d1, src[k * T::LDQ + 8 * ta + g], src[k * T::LDQ + 8 * tb + g]);
            }
            const int a = 8 * ta + g, b = 8 * tb + 2 * t;
            G[a * RT + b] = d0;
            G[a * RT + b + 1] = d1;
        }
        __syncthreads();
    } else {
        const int tt = w % TILES, part = w / TILES;
        const int ta = tt % T::NT, tb = tt / T::NT;
        double d0 = 0.0, d1 = 0.0;
        for (int kk = part; kk < ksteps; kk += KSP) {
            const int k = 4 * kk + t;
            dmma884(d0, d1, src[k * T::LDQ + 8 * ta + g], src[k * T::LDQ + 8 * tb + g]);
        }
        const int a = 8 * ta + g, b = 8 * tb + 2 * t;
        Gp[part * RT * RT + a * RT + b] = d0;
        Gp[part * RT * RT + a * RT + b + 1] = d1;
        __syncthreads();
        for (int e = threadIdx.x; e < RT * RT; e += SM_NT) {
            double s = 0.0;
#pragma unroll
            for (int p = 0; p < KSP; p++) s += Gp[p * RT * RT + e];
            G[e] = s;
        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < RT * RT; e += SM_NT) {
        const int a = e / RT, b = e % RT;
        if (a >= r || b >= r) G[e] = (a == b) ? 1.0 : 0.0;
    }
    __syncthreads();
}

// Ri = R^{-1} (row-major, pitch LDR) of G = R^T R, by warp 0 (all threads call
// it; ends with a barrier; G is overwritten).  32 / RT groups of RT lanes share
// the rows (row i belongs to group i mod 32 / RT), lane c of a group holds column c
// of its rows in registers.  The next pivot is formed first, from values exchanged
// before this pivot's root is known, and no branch stands between the rows'
// updates.  Then lane c solves column c of the inverse by back substitution, R
// read from shared memory.  Every operation and its rounding is that of the plain
// elimination (products and differences rounded one by one, two alternating
// sums in the back substitution): the callers' factors go on to be rounded to
// BF16 halves, where another rounding of FP64 would show.  Bound by the pivots'
// chain (a root, two products, a difference) and by what a warp can issue:
// r = 16 takes 4800 cycles (860 of them the back substitution), r = 5 1500; CTA-wide,
// with two barriers a pivot, r = 16 took 7400.  Returns false on a non-positive
// pivot.
template <int RT>
__device__ __forceinline__ bool sm_chol_inv(double *G, double *Ri, int r) {
    constexpr int LDR = SmTile<RT>::LDR;
    constexpr int GR = 32 / RT, NR = RT / GR;
    __shared__ int good;
    const int lane = threadIdx.x;
    if (lane < 32) {
        const int c = lane % RT, h = lane / RT;
        double g[NR], dinv[RT];
#pragma unroll
        for (int q = 0; q < NR; q++) g[q] = G[(q * GR + h) * RT + c];
#pragma unroll
        for (int i = 0; i < RT; i++) dinv[i] = 1.0;
        double d = __shfl_sync(0xffffffffu, g[0], 0);
        const double least = 1e-28 * d;
        bool ok = d > 0.0;
#pragma unroll
        for (int k = 0; k < RT; k++) {
            if (k >= r) break;
            constexpr unsigned ALL = 0xffffffffu;
            const int qk = k / GR, at = RT * (k % GR);  // row k's lanes: at, at + 1, ...
            double s[NR], next = 0.0, s1 = 0.0;
            if (k + 1 < RT) {
                s1 = __shfl_sync(ALL, g[qk], at + k + 1);
                next = __shfl_sync(ALL, g[(k + 1) / GR], RT * ((k + 1) % GR) + k + 1);
            }
            const double raw = __shfl_sync(ALL, g[qk], at + c);
#pragma unroll
            for (int q = qk; q < NR; q++) s[q] = __shfl_sync(ALL, g[qk], at + q * GR + h);
            ok = ok && d > least;
            const double ri = rsqrt(fmax(d, 1e-300));
            dinv[k] = ri;
            if (k + 1 < RT) {
                const double l = __dmul_rn(s1, ri);
                d = __dsub_rn(next, __dmul_rn(l, l));
            }
            const double gk = __dmul_rn(raw, ri);
#pragma unroll
            for (int q = qk; q < NR; q++) {
                const double u = __dsub_rn(g[q], __dmul_rn(__dmul_rn(s[q], ri), gk));
                if (q > qk || h > k % GR) g[q] = u;
                else if (h == k % GR) g[q] = gk;
            }
        }
#pragma unroll
        for (int q = 0; q < NR; q++) G[(q * GR + h) * RT + c] = g[q];
        __syncwarp();
        // x_i = (delta_{i,c} - sum_{j>i} R(i, j) x_j) dinv_i
        double x[RT];
#pragma unroll
        for (int i = RT - 1; i >= 0; i--) {
            double s0 = (i == lane) ? 1.0 : 0.0, s1 = 0.0;
#pragma unroll
            for (int j = i + 1; j < RT; j++) {
                const double rij = G[i * RT + j];
                if (j & 1)
                    s1 = fma(-rij, x[j], s1);
                else
                    s0 = fma(-rij, x[j], s0);
            }
            x[i] = (s0 + s1) * dinv[i];
        }
        if (lane < RT) {
#pragma unroll
            for (int i = 0; i < RT; i++) Ri[i * LDR + lane] = i <= lane ? x[i] : 0.0;
        }
        if (lane == 0) good = ok;
    }
    __syncthreads();
    return good != 0;
}

// The same by warp_chol_linv: the identity is eliminated along with G, with fused
// products and the hardware's root refined in line.  r = 16: 2200 cycles against
// 4800, three of them per subspace of 5 steps: 96^4 sweeps 1604 -> 1575 us, 256-cube
// warm start 1489 -> 1458 us.  For results that stay FP64, where another rounding of
// the last bit does no harm.
template <int RT>
__device__ __forceinline__ bool sm_chol_inv_fused(const double *G, double *Ri, int r) {
    constexpr int LDR = SmTile<RT>::LDR;
    __shared__ int good;
    const int lane = threadIdx.x;
    if (lane < 32) {
        double y[RT];
        const bool ok = warp_chol_linv<RT>(G, RT, r, y);
        // Lane c holds column c of L^{-1} = row c of R^{-1}.
        if (lane < RT) {
#pragma unroll
            for (int i = 0; i < RT; i++) Ri[lane * LDR + i] = i >= lane ? y[i] : 0.0;
        }
        if (lane == 0) good = ok;
    }
    __syncthreads();
    return good != 0;
}

// After one CholeskyQR pass, Q^T Q = I + E with E tiny.  When max |E| <= 1e-8,
// C = I - E/2 + 3E^2/8 (the series of (I + E)^{-1/2}) makes Q C orthonormal to
// rounding; C goes to Ri (pitch LDR) for sm_apply.  Returns false when E is too
// large, and the caller runs a second CholeskyQR pass instead.  All threads.
template <int RT>
__device__ __forceinline__ bool sm_polar_fix(const double *G, double *Ri, double *red) {
    constexpr int LDR = SmTile<RT>::LDR;
    const int t = threadIdx.x;
    double emax = 0.0;
    for (int e = t; e < RT * RT; e += SM_NT) {
        const int a = e / RT, b = e % RT;
        emax = fmax(emax, fabs(G[e] - (a == b ? 1.0 : 0.0)));
    }
    for (int o = 16; o > 0; o >>= 1) emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, o));
    if ((t & 31) == 0) red[t >> 5] = emax;
    __syncthreads();
    double m = 0.0;
#pragma unroll
    for (int w = 0; w < SM_WARPS; w++) m = fmax(m, red[w]);
    if (!(m <= 1e-8)) {
        __syncthreads();
        return false;
    }
    for (int e = t; e < RT * RT; e += SM_NT) {
        const int a = e / RT, b = e % RT;
        double e2 = 0.0;
#pragma unroll
        for (int k = 0; k < RT; k++)
            e2 = fma(G[a * RT + k] - (a == k ? 1.0 : 0.0), G[k * RT + b] - (k == b ? 1.0 : 0.0), e2);
        const double eab = G[e] - (a == b ? 1.0 : 0.0);
        Ri[a * LDR + b] = (a == b ? 1.0 : 0.0) - 0.5 * eab + 0.375 * e2;
    }
    __syncthreads();
    return true;
}

// The cluster's CTAs: rank, size, barrier, and this CTA's address of shared
// memory in another one.
__device__ __forceinline__ unsigned cl_rank() {
    unsigned v;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(v));
    return v;
}
__device__ __forceinline__ void cl_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                     : "memory");
}
__device__ __forceinline__ uint32_t cl_map(const void *p, unsigned rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), out;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(a), "r"(rank));
    return out;
}
// Sends `bytes` of this CTA's shared memory at p to the same place in the CTAs
// of the cluster and waits for what all of them send, `bytes_in` in sum (each
// sends its own part of the same array).  The copies are the hardware's bulk
// copies between shared memories and complete on the receiver's mbarrier, so an
// exchange is one way across the SM network: rows stored one 16-byte word per
// lane into every CTA and a cluster barrier took 1900 cycles more than the
// product alone for 96 x 16 on four CTAs, 4400 for 200 x 16 on eight.  Steps
// alternate between two mbarriers: a CTA can be one step ahead of another,
// never two (its second step needs the other's first).  The sender's rows are
// read before anybody can answer with the next step's data.  Returns false when
// the bounded wait ran out (about a second) for any thread of the CTA.  All
// threads; the verdict is the CTA's, so the threads go on or leave together, and
// taking it is a barrier.
struct ClExchange {
    uint64_t *bar;  // two mbarriers, arrival count 1
    int step;
    unsigned csize, rank;
    long long limit = 2000000000LL;  // cycles
};

__device__ __forceinline__ bool cl_exchange(ClExchange &x, const void *p, uint32_t bytes,
                                            uint32_t bytes_in) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (x.csize == 1) return true;
    uint64_t *bar = x.bar + (x.step & 1);
    const uint32_t parity = (x.step >> 1) & 1;
    x.step++;
    const uint32_t barl = (uint32_t)__cvta_generic_to_shared(bar);
    if (threadIdx.x == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(barl),
                     "r"(bytes_in)
                     : "memory");
    if (threadIdx.x < x.csize && threadIdx.x != x.rank && bytes > 0)
        asm volatile(
            "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, "
            "[%3];" ::"r"(cl_map(p, threadIdx.x)),
            "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(bytes), "r"(cl_map(bar, threadIdx.x))
            : "memory");
    long long t0 = 0;
    uint32_t ok;
    for (;;) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(barl), "r"(parity)
            : "memory");
        if (ok) break;
        if (t0 == 0) t0 = clock64();
        else if (clock64() - t0 > x.limit) break;
    }
    return !__syncthreads_or(!ok);
}

// A cluster of two CTAs that each wait for data nobody sends: adds up the threads
// that take the exchange for late.
__global__ void __launch_bounds__(SM_NT) exchange_selftest_kernel(int *late, long long limit) {
    __shared__ __align__(16) double data[2];
    __shared__ __align__(8) uint64_t bars[2];
    if (threadIdx.x == 0) {
        for (int q = 0; q < 2; q++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(bars + q))
                         : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cl_sync();
    ClExchange ex{bars, 0, 2u, cl_rank(), limit};
    if (!cl_exchange(ex, data, 0, sizeof(data))) atomicAdd(late, 1);
    cl_sync();
}

// Rows of S a CTA of a cluster of c owns (whole 8-row tiles), and the pitch of
// a staged row.
__host__ __device__ inline int sub_rows(int n, int c) { return 8 * (((n + 7) / 8 + c - 1) / c); }
__host__ __device__ inline int sub_pitch(int n) { return ((n + 11) / 16) * 16 + 4; }
template <int RT>
__host__ inline size_t sub_smem_bytes(int n, int c, bool s_in_smem, int bufs) {
    const int n8 = (n + 7) / 8 * 8;
    size_t d = bufs * (size_t)n8 * SmTile<RT>::LDQ          // Z
               + (size_t)SM_GP                              // Gram partials
               + (size_t)RT * RT                            // G
               + (size_t)RT * SmTile<RT>::LDR;              // R^{-1}
    if (s_in_smem) d += (size_t)sub_rows(n, c) * sub_pitch(n);
    return d * sizeof(double);
}

// Independent problems of one launch, a cluster each.
constexpr int SUB_MAX = 8;
struct SubBatch {
    const double *S[SUB_MAX];
    double *L[SUB_MAX], *work[SUB_MAX];
    int n[SUB_MAX], r[SUB_MAX];
};

// PLAIN: the factorisation that rounds as the plain elimination does.
template <int RT, bool SSM, bool PLAIN>
__global__ void __launch_bounds__(SM_NT, 1) subspace_cluster_kernel(SubBatch batch, int iters,
                                                                    int *flag, int csize, int bufs) {
    using T = SmTile<RT>;
    const int prob = blockIdx.x / csize;
    const double *const Sg = batch.S[prob];
    double *const Lg = batch.L[prob], *const work = batch.work[prob];
    const int n = batch.n[prob], r = batch.r[prob];
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[33];
    __shared__ __align__(8) uint64_t bars[2];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, g = lane >> 2, t4 = lane & 3;
    const unsigned rank = cl_rank();
    if (t == 0) {
        for (int q = 0; q < 2; q++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(bars + q))
                         : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    ClExchange ex{bars, 0, (unsigned)csize, rank};
    const int n8 = (n + 7) / 8 * 8, lds = sub_pitch(n);
    const int own0 = (int)rank * sub_rows(n, csize);
    const int own = max(0, min(n8 - own0, sub_rows(n, csize)));  // this CTA's rows
    const int mt = own / 8, ksteps = (n + 3) / 4;
    double *const ring = sm;  // `bufs` copies of Z
    double *Gp = ring + bufs * n8 * T::LDQ;
    double *G = Gp + SM_GP;
    double *Ri = G + RT * RT;
    double *Ss = Ri + RT * T::LDR;
    for (int e = t; e < bufs * n8 * T::LDQ; e += SM_NT) ring[e] = 0.0;
    if (SSM) {
        // Padding of the staged rows: k = n .. 4 ksteps - 1, and rows past n.
        for (int e = t; e < own * (4 * ksteps - n); e += SM_NT) {
            const int pr = 4 * ksteps - n;
            Ss[(e / pr) * lds + n + e % pr] = 0.0;
        }
        for (int i = max(0, n - own0); i < own; i++)
            for (int k = t; k < n; k += SM_NT) Ss[i * lds + k] = 0.0;
    }
    pdl_wait();
    const int have = min(own, n - own0);  // rows of S there are (may be <= 0)
    if (SSM) {
        const double *src = Sg + (int64_t)n * own0;
        // 16-byte copies: an even n on an S that is 16-byte aligned.
        if ((n & 1) == 0 && (reinterpret_cast<uintptr_t>(Sg) & 15) == 0) {
            const int hc = n / 2;
            for (int e = t; e < hc * have; e += SM_NT) {
                const int i = e / hc, q = e - i * hc;
                la_cp_async16(Ss + lds * i + 2 * q, src + (int64_t)n * i + 2 * q);
            }
            la_cp_commit();
        } else {
            for (int e = t; e < n * have; e += SM_NT) {
                const int i = e / n, k = e - i * n;
                Ss[lds * i + k] = src[e];
            }
        }
    }
    __syncthreads();  // the zeroed buffers
    {
        // L (n x r col-major) -> the ring's first (row-major, zero padded): all loads of a
        // thread are issued before its stores.
        constexpr int MAXQ = RT;  // n * r <= 256 * RT = SM_NT * MAXQ
        double v[MAXQ];
#pragma unroll
        for (int q = 0; q < MAXQ; q++) {
            const int e = t + SM_NT * q;
            v[q] = e < n * r ? Lg[e] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < MAXQ; q++) {
            const int e = t + SM_NT * q;
            if (e < n * r) {
                const int c = e / n, i = e - c * n;
                ring[i * T::LDQ + c] = v[q];
            }
        }
    }
    if (SSM) la_cp_wait_all();
    // Every CTA's buffers are ready before any CTA writes into them.
    if (csize > 1) cl_sync();
    else __syncthreads();

    // dst(own rows) = S(own rows, :) src, k-steps in order.
    auto product = [&](const double *src, double *dst) {
        for (int job = w; job < mt * T::NT; job += SM_WARPS) {
            const int m = job / T::NT, j = job - m * T::NT;
            double d0 = 0.0, d1 = 0.0;
            const double *bs = src + t4 * T::LDQ + 8 * j + g;
            if (SSM) {
                const double *as = Ss + (8 * m + g) * lds + t4;
#pragma unroll 8
                for (int k = 0; k < ksteps; k++) dmma884(d0, d1, as[4 * k], bs[4 * k * T::LDQ]);
            } else {
                const int i = own0 + 8 * m + g;
#pragma unroll 8
                for (int k = 0; k < ksteps; k++) {
                    const int kk = 4 * k + t4;
                    const double av = i < n && kk < n ? __ldg(Sg + (int64_t)n * i + kk) : 0.0;
                    dmma884(d0, d1, av, bs[4 * k * T::LDQ]);
                }
            }
            *reinterpret_cast<double2 *>(dst + (own0 + 8 * m + g) * T::LDQ + 8 * j + 2 * t4) =
                make_double2(d0, d1);
        }
    };
    const uint32_t row_bytes = T::LDQ * sizeof(double);
    int at = 0;  // Z's place in the ring
    auto z = [&](int k) { return ring + ((at + k) % bufs) * n8 * T::LDQ; };

    bool bad = false, late = false;
    int it = 0;
    for (; it < iters && !bad; it++) {
        const bool last = it == iters - 1;
        product(z(0), z(1));
        // Everybody's rows to everybody.
        late = !cl_exchange(ex, z(1) + own0 * T::LDQ, own * row_bytes, (n8 - own) * row_bytes);
        if (late) break;
        at = (at + 1) % bufs;
        if (!last && !(it & 1)) continue;
        for (int p = 0; p < (last ? 2 : 1); p++) {
            sm_gram<RT>(z(0), n, r, Gp, G);
            // The second pass is usually a tiny correction (polar fix).
            if (!(p == 1 && sm_polar_fix<RT>(G, Ri, red)) &&
                !(PLAIN ? sm_chol_inv<RT>(G, Ri, r) : sm_chol_inv_fused<RT>(G, Ri, r))) {
                bad = true;  // the same G, so the same answer, in every CTA
                break;
            }
            sm_apply<RT>(z(0), Ri, n8, z(1));
            __syncthreads();
            at = (at + 1) % bufs;
        }
        if (bufs == 2 && csize > 1 && !last && !bad) cl_sync();
    }
    // No CTA leaves while another still reads or fills its shared memory: a late one
    // takes part in the barriers of the steps it leaves out.
    if (late && bufs == 2)
        for (int k = it; k < iters - 1; k++)
            if (k & 1) cl_sync();
    if (csize > 1) cl_sync();
    if (late) {
        // An exchange never came: NaN factors, which the driver reports.
        for (int e = t; e < n * r; e += SM_NT) Lg[e] = __longlong_as_double(0x7ff8000000000000LL);
        return;
    }
    // Dependents launch once the iteration is done (launched at the start,
    // they took SM slots for the whole kernel; about 1 % of a decomposition).
    pdl_trigger();
    if (!bad) {
        for (int e = t; e < have * r; e += SM_NT) {
            const int c = e / have, i = own0 + (e - c * have);
            Lg[(int64_t)n * c + i] = z(0)[i * T::LDQ + c];
        }
        return;
    }
    if (rank != 0) return;
    // Rank-deficient or badly conditioned: restart from the caller's L and run
    // every step with Householder orthonormalisation (col-major, in `work`).
    double *Lw = work, *hw = work + 2 * (int64_t)n * r;
    for (int e = t; e < n * r; e += SM_NT) Lw[e] = Lg[e];
    __syncthreads();
    for (int it = 0; it < iters; it++) {
        for (int e = t; e < n * r; e += SM_NT) {
            const int i = e % n, c = e / n;
            double acc = 0.0;
            for (int k = 0; k < n; k++)
                acc = fma(__ldg(Sg + i + (int64_t)n * k), Lw[k + n * c], acc);
            hw[e] = acc;
        }
        __syncthreads();
        hqr_device(hw, n, r, hw + (int64_t)n * r, Lw, red);
        __syncthreads();
    }
    if (t == 0 && flag) atomicOr(flag, 2);
    for (int e = t; e < n * r; e += SM_NT) Lg[e] = Lw[e];
}

// Q[b] = orth(A[b]) for a batch of m x n (n <= RT) col-major matrices, one CTA
// each: CholeskyQR2 with the mma.sync Gram / apply above; a Cholesky
// breakdown falls back to Householder on work[b] (m n + n doubles).  The span
// is that of A, as with Householder QR; the basis may differ by a rotation.
template <int RT>
__global__ void __launch_bounds__(SM_NT, 1) cholqr2_batch_kernel(OrthTable tab) {
    using T = SmTile<RT>;
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[33];
    __shared__ int bad;
    const int b = blockIdx.x, t = threadIdx.x;
    const int M = (int)tab.m[b], r = (int)tab.n[b];
    const double *Ab = tab.A[b];
    double *Qb = tab.Q[b];
    const int M8 = (M + 7) / 8 * 8;
    double *Z0 = sm;
    double *Z1 = Z0 + M8 * T::LDQ;
    double *Gp = Z1 + M8 * T::LDQ;
    double *G = Gp + SM_GP;
    double *Ri = G + RT * RT;
    for (int e = t; e < M8 * T::LDQ; e += SM_NT) {
        const int i = e / T::LDQ, c = e % T::LDQ;
        Z0[e] = (i < M && c < r) ? Ab[i + (int64_t)M * c] : 0.0;
    }
    if (t == 0) bad = 0;
    __syncthreads();
    double *cur = Z0, *oth = Z1;
    for (int p = 0; p < 2; p++) {
        sm_gram<RT>(cur, M, r, Gp, G);
        if (!sm_chol_inv<RT>(G, Ri, r)) {
            bad = 1;
            break;
        }
        sm_apply<RT>(cur, Ri, M8, oth);
        __syncthreads();
        double *tmp = cur;
        cur = oth;
        oth = tmp;
    }
    if (!bad) {
        for (int e = t; e < M * r; e += SM_NT) {
            const int i = e % M, c = e / M;
            Qb[e] = cur[i * T::LDQ + c];
        }
        return;
    }
    double *W = tab.work[b];
    for (int e = t; e < M * r; e += SM_NT) W[e] = Ab[e];
    __syncthreads();
    hqr_device(W, M, r, W + (int64_t)M * r, Qb, red);
}

template <int RT, bool SSM>
void launch_subspace(dt_ctx *ctx, const SubBatch &batch, int count, int n, int iters, int *flag,
                     int csize, int bufs, bool plain) {
    const size_t smem = sub_smem_bytes<RT>(n, csize, SSM, bufs);
    auto kern = plain ? subspace_cluster_kernel<RT, SSM, true>
                      : subspace_cluster_kernel<RT, SSM, false>;
    smem_limit(ctx, kern, smem);
    launch_pdl_cluster(ctx, kern, count * csize, SM_NT, smem, csize, batch, iters, flag, csize, bufs);
}

// `count` problems of up to n rows.
template <int RT>
void subspace_mma(dt_ctx *ctx, const SubBatch &batch, int count, int n, int iters, int *flag,
                  bool plain) {
    const size_t cap = 220 * 1024;
    // Up to 64 rows one CTA: an exchange costs more than the part of a product
    // it saves (64 x 8, 5 steps: 13.6 us on one CTA, 14.8 on eight).  Above,
    // eight: 96 x 16, 5 steps 32.0 us on one CTA, 29.7 on two, 26.5 on four, 26.1 on
    // eight; 200 x 10, 30 steps 154 on four, 128 on eight.  The single-CTA kernel
    // before this one took 35 us for 96 x 16 in 5 steps and 20 in 2 (15.2 here),
    // and 112 us for 256 x 12 with S read from L2 (37 here).
    const int c = n <= 64 ? 1 : 8;
    if (sub_smem_bytes<RT>(n, c, true, 3) <= cap)
        launch_subspace<RT, true>(ctx, batch, count, n, iters, flag, c, 3, plain);
    else if (sub_smem_bytes<RT>(n, c, true, 2) <= cap)
        launch_subspace<RT, true>(ctx, batch, count, n, iters, flag, c, 2, plain);
    else  // r > 16 and n > 230 or so: S stays in L2
        launch_subspace<RT, false>(ctx, batch, count, n, iters, flag, c, 2, plain);
}

void subspace_mma(dt_ctx *ctx, const SubBatch &batch, int count, int iters, int *flag, bool plain) {
    int n = 0, r = 0;
    for (int b = 0; b < count; b++) {
        n = std::max(n, batch.n[b]);
        r = std::max(r, batch.r[b]);
    }
    if (r <= 8) subspace_mma<8>(ctx, batch, count, n, iters, flag, plain);
    else if (r <= 16) subspace_mma<16>(ctx, batch, count, n, iters, flag, plain);
    else subspace_mma<32>(ctx, batch, count, n, iters, flag, plain);
}

// Subspace iteration for ranks above 32: Householder QR every step, S, L and Z
// in global memory (L2-resident).  work >= 3*n*r + r.
__global__ void __launch_bounds__(LA_NT) subspace_wide_kernel(const double *S, int64_t n,
                                                              double *L, int64_t r, int iters,
                                                              double *work) {
    __shared__ double red[33];
    double *Z = work, *W = work + n * r, *tau = work + 2 * n * r;
    for (int it = 0; it < iters; it++) {
        for (int64_t e = threadIdx.x; e < n * r; e += blockDim.x) {
            const int64_t i = e % n, c = e / n;
            double acc = 0.0;
            for (int64_t k = 0; k < n; k++) acc = fma(S[i + n * k], L[k + n * c], acc);
            Z[e] = acc;
        }
        __syncthreads();
        for (int64_t e = threadIdx.x; e < n * r; e += blockDim.x) W[e] = Z[e];
        __syncthreads();
        hqr_device(W, n, r, tau, L, red);
        __syncthreads();
    }
}

// LU with partial pivoting on W (n x n col-major copy of A), then Ainv by
// solving for the identity columns.
__global__ void __launch_bounds__(LA_NT) lu_inverse_kernel(const double *A, int64_t n,
                                                           double *Ainv, double *W,
                                                           int *flag) {
    __shared__ double red_v[32];
    __shared__ int red_i[32];
    __shared__ int piv_row;
    extern __shared__ int perm[];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int64_t e = t; e < n * n; e += blockDim.x) W[e] = A[e];
    for (int64_t i = t; i < n; i += blockDim.x) perm[i] = (int)i;
    __syncthreads();
    for (int64_t k = 0; k < n; k++) {
        double best = -1.0;
        int bi = (int)k;
        for (int64_t i = k + t; i < n; i += blockDim.x) {
            const double v = fabs(W[i + k * n]);
            if (v > best) {
                best = v;
                bi = (int)i;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_down_sync(0xffffffffu, best, o);
            const int oi = __shfl_down_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) {
                best = ov;
                bi = oi;
            }
        }
        if (lane == 0) {
            red_v[warp] = best;
            red_i[warp] = bi;
        }
        __syncthreads();
        if (t == 0) {
            double bv = -1.0;
            int bb = (int)k;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++)
                if (red_v[w] > bv || (red_v[w] == bv && red_i[w] < bb)) {
                    bv = red_v[w];
                    bb = red_i[w];
                }
            piv_row = bb;
            if (!(bv > 0.0)) atomicOr(flag, 1);
        }
        __syncthreads();
        const int p = piv_row;
        if (p != k) {
            for (int64_t c = t; c < n; c += blockDim.x) {
                const double tmp = W[k + c * n];
                W[k + c * n] = W[p + c * n];
                W[p + c * n] = tmp;
            }
            if (t == 0) {
                const int tp = perm[k];
                perm[k] = perm[p];
                perm[p] = tp;
            }
        }
        __syncthreads();
        const double d = W[k + k * n];
        for (int64_t i = k + 1 + t; i < n; i += blockDim.x) W[i + k * n] /= d;
        __syncthreads();
        for (int64_t e = t; e < (n - k - 1) * (n - k - 1); e += blockDim.x) {
            const int64_t i = k + 1 + e % (n - k - 1), c = k + 1 + e / (n - k - 1);
            W[i + c * n] = fma(-W[i + k * n], W[k + c * n], W[i + c * n]);
        }
        __syncthreads();
    }
    // Solve L U x = P e_c for every column c (one thread per column).
    for (int64_t c = t; c < n; c += blockDim.x) {
        double *x = Ainv + c * n;
        for (int64_t i = 0; i < n; i++) {
            double s = (perm[i] == c) ? 1.0 : 0.0;
            for (int64_t j = 0; j < i; j++) s = fma(-W[i + j * n], x[j], s);
            x[i] = s;
        }
        for (int64_t i = n - 1; i >= 0; i--) {
            double s = x[i];
            for (int64_t j = i + 1; j < n; j++) s = fma(-W[i + j * n], x[j], s);
            x[i] = s / W[i + i * n];
        }
    }
}

// Householder QR of several small matrices at once (one CTA each, 128
// threads so the per-column barriers stay cheap): Q[b] = Q of A[b].
__global__ void __launch_bounds__(128) hqr_batch_kernel(OrthTable tab) {
    __shared__ double red[33];
    const int b = blockIdx.x;
    const int64_t mb = tab.m[b], nb = tab.n[b];
    double *W = tab.work[b];
    for (int64_t e = threadIdx.x; e < mb * nb; e += blockDim.x) W[e] = tab.A[b][e];
    __syncthreads();
    hqr_device(W, mb, nb, W + mb * nb, tab.Q[b], red);
}

// Cholesky of the r x r SPD G (col-major, its lower triangle overwritten) and L^{-1}
// (lower, col-major) for the orthonormalisation of more than 32 rows; one CTA of 1024
// threads, r <= 1024, both matrices in global memory (L2).  The row operations that
// eliminate G are applied to the identity as well.  Not on a measured path: bound
// by one SM's traffic with L2.
__global__ void __launch_bounds__(1024) chol_lower_inv_kernel(double *G, int r, double *Linv,
                                                              int *flag) {
    __shared__ double l[1024], y[1024];  // column k of L below k, row k of L^{-1}
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    const double least = fmax(1e-28 * G[0], 2.3e-308);
    for (int c = w; c < r; c += 32)
        for (int i = lane; i < r; i += 32) Linv[i + (int64_t)r * c] = i == c ? 1.0 : 0.0;
    __syncthreads();
    for (int k = 0; k < r; k++) {
        const double d = G[k + (int64_t)r * k];
        if (t == 0 && !(d > least)) atomicOr(flag, 1);
        const double ri = 1.0 / sqrt(d);
        for (int i = t; i < r; i += 1024) {
            if (i > k) {
                l[i] = G[i + (int64_t)r * k] * ri;
            } else {
                y[i] = Linv[k + (int64_t)r * i] * ri;
                Linv[k + (int64_t)r * i] = y[i];
            }
        }
        __syncthreads();
        for (int c = w; c < r; c += 32) {
            double *col = c > k ? G + (int64_t)r * c : Linv + (int64_t)r * c;
            const double f = c > k ? l[c] : y[c];
            for (int i = (c > k ? c : k + 1) + lane; i < r; i += 32) col[i] = fma(-l[i], f, col[i]);
        }
        __syncthreads();
    }
}

// Row Gram on the FP64 tensor cores (mma.sync m8n8k4): A is r x m col-major
// (factor row k = column k), G = sum_k a_k a_k^T, finished to L^{-1} of its
// Cholesky factor (gram_finish).  With 4 columns per k-step, the fragment
// A[g][t] = a_{4kk+t}(8h + g) is also the B fragment B[t][g] of tile h, so
// each lane loads TT values per k-step for TT x TT MMAs.  Warps of a block
// take interleaved k-steps of the block's column range.
template <int RT>
__global__ void __launch_bounds__(256) rows_gram_kernel(const double *__restrict__ A, int r,
                                                        int64_t m, int64_t cols_per_block,
                                                        GramFinish f) {
    constexpr int TT = RT / 8;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    pdl_wait();
    const int64_t k0 = blockIdx.x * cols_per_block;
    const int64_t k1 = min(m, k0 + cols_per_block);
    double acc[TT][TT][2];
#pragma unroll
    for (int a = 0; a < TT; a++)
#pragma unroll
        for (int b = 0; b < TT; b++) acc[a][b][0] = acc[a][b][1] = 0.0;
#pragma unroll 4
    for (int64_t c0 = k0 + 4 * w; c0 < k1; c0 += 32) {
        const int64_t col = c0 + t;
        double v[TT];
#pragma unroll
        for (int h = 0; h < TT; h++)
            v[h] = (col < k1 && 8 * h + g < r) ? A[col * r + 8 * h + g] : 0.0;
#pragma unroll
        for (int a = 0; a < TT; a++)
#pragma unroll
            for (int b = 0; b < TT; b++) dmma884(acc[a][b][0], acc[a][b][1], v[a], v[b]);
    }
    gram_finish<TT>(acc, r, f);
}

// T = Linv A: Linv (r x r lower, col-major) is the A operand (held in
// registers), 8-column blocks of A (r x m col-major) the B operand; one warp
// per 8-column block.  Column k goes to column rows[k] of T when `rows` is
// given.  GRAM: the Gram of T is taken on the way and finished to the next
// pass's L^{-1}.  A lane's results are T(8 h + g, columns 2 t + q): taking the
// block's even columns as one k-step and the odd ones as another, these are
// its Gram fragments as they stand.
template <int RT, bool GRAM>
__global__ void __launch_bounds__(256) rows_apply_kernel(const double *__restrict__ A, int r,
                                                         int64_t m,
                                                         const double *__restrict__ Linv,
                                                         double *__restrict__ T,
                                                         const int32_t *__restrict__ rows,
                                                         GramFinish f) {
    constexpr int TT = RT / 8, KS = RT / 4;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    pdl_wait();
    double la[TT][KS];
#pragma unroll
    for (int h = 0; h < TT; h++)
#pragma unroll
        for (int kk = 0; kk < KS; kk++) {
            const int i = 8 * h + g, c = 4 * kk + t;
            la[h][kk] = (i < r && c < r) ? Linv[i + (int64_t)r * c] : 0.0;
        }
    double gacc[TT][TT][2];
#pragma unroll
    for (int a = 0; a < TT; a++)
#pragma unroll
        for (int b = 0; b < TT; b++) gacc[a][b][0] = gacc[a][b][1] = 0.0;
    const int64_t warp0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t nblk = (m + 7) / 8;
    for (int64_t cb = warp0; cb < nblk; cb += nwarps) {
        double acc[TT][2];
#pragma unroll
        for (int h = 0; h < TT; h++) acc[h][0] = acc[h][1] = 0.0;
        const int64_t colb = 8 * cb + g;
        double b[KS];
#pragma unroll
        for (int kk = 0; kk < KS; kk++) {
            const int c = 4 * kk + t;
            b[kk] = (colb < m && c < r) ? A[colb * r + c] : 0.0;
        }
#pragma unroll
        for (int kk = 0; kk < KS; kk++)
#pragma unroll
            for (int h = 0; h < TT; h++) dmma884(acc[h][0], acc[h][1], la[h][kk], b[kk]);
        if (GRAM) {
#pragma unroll
            for (int q = 0; q < 2; q++)
#pragma unroll
                for (int x = 0; x < TT; x++)
#pragma unroll
                    for (int z = 0; z < TT; z++)
                        dmma884(gacc[x][z][0], gacc[x][z][1], acc[x][q], acc[z][q]);
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int64_t col = 8 * cb + 2 * t + q;
            if (col >= m) continue;
            double *dst = T + (rows ? (int64_t)rows[col] : col) * r;
#pragma unroll
            for (int h = 0; h < TT; h++)
                if (8 * h + g < r) dst[8 * h + g] = acc[h][q];
        }
    }
    if (GRAM) gram_finish<TT>(gacc, r, f);
}

}  // namespace

void householder_qr(dt_ctx *ctx, const double *A, int64_t m, int64_t n, double *Q, double *R,
                    double *work) {
    DT_CHECK_ARG(m >= n && n > 0, "householder_qr: need m >= n > 0 (m=%lld n=%lld)",
                 (long long)m, (long long)n);
    DT_LAUNCH(ctx, hqr_kernel, 1, LA_NT, 0, A, m, n, Q, R, work);
}

namespace {

// The batch's table, its workspaces in one allocation.
OrthTable orth_table(dt_ctx *ctx, int count, const double *const *A, double *const *Q,
                     const int64_t *m, const int64_t *n, DevMem &ws) {
    DT_CHECK_ARG(count >= 1 && count <= ORTH_MAX, "orth_batch: %d matrices", count);
    OrthTable tab{};
    int64_t total = 0;
    for (int b = 0; b < count; b++) {
        DT_CHECK_ARG(m[b] >= n[b] && n[b] > 0, "orth_batch: need m >= n > 0");
        total += m[b] * n[b] + n[b];
    }
    ws.alloc(ctx, total * sizeof(double));
    double *w = ws.as<double>();
    for (int b = 0; b < count; b++) {
        tab.A[b] = A[b];
        tab.Q[b] = Q[b];
        tab.work[b] = w;
        tab.m[b] = m[b];
        tab.n[b] = n[b];
        w += m[b] * n[b] + n[b];
    }
    return tab;
}

}  // namespace

void orth_batch(dt_ctx *ctx, int count, const double *const *A, double *const *Q,
                const int64_t *m, const int64_t *n) {
    DevMem ws;
    const OrthTable tab = orth_table(ctx, count, A, Q, m, n, ws);
    int64_t maxm = 0, maxn = 0;
    for (int b = 0; b < count; b++) {
        maxm = std::max(maxm, m[b]);
        maxn = std::max(maxn, n[b]);
    }
    const int RT = maxn <= 8 ? 8 : (maxn <= 16 ? 16 : 32);
    const int64_t M8 = (maxm + 7) / 8 * 8;
    const size_t smem =
        (2 * (size_t)M8 * (RT + 4) + SM_GP + RT * RT + RT * (RT + 4)) * sizeof(double);
    if (maxn > 32 || smem > 220 * 1024) {
        DT_LAUNCH(ctx, hqr_batch_kernel, count, 128, 0, tab);
        return;
    }
#define DT_CQR(R)                                            \
    do {                                                     \
        auto kern = cholqr2_batch_kernel<R>;                 \
        smem_limit(ctx, kern, smem);                         \
        DT_LAUNCH(ctx, kern, count, SM_NT, smem, tab);       \
    } while (0)
    if (RT == 8) DT_CQR(8);
    else if (RT == 16) DT_CQR(16);
    else DT_CQR(32);
#undef DT_CQR
}

void subspace_iter(dt_ctx *ctx, const double *S, int64_t n, double *L, int64_t r, int iters,
                   double *work, int *flag, bool plain) {
    DT_CHECK_ARG(n >= r && r > 0, "subspace_iter: bad sizes n=%lld r=%lld", (long long)n,
                 (long long)r);
    if (r > 32) {
        DT_LAUNCH(ctx, subspace_wide_kernel, 1, LA_NT, 0, S, n, L, r, iters, work);
        return;
    }
    if (n <= 256) {
        SubBatch one{};
        one.S[0] = S;
        one.L[0] = L;
        one.work[0] = work;
        one.n[0] = (int)n;
        one.r[0] = (int)r;
        subspace_mma(ctx, one, 1, iters, flag, plain);
        return;
    }
    const size_t zl_bytes = 2 * n * r * sizeof(double), base = r * r * sizeof(double);
    const int zl_in = base + zl_bytes <= 220 * 1024;
    const size_t smem = base + (zl_in ? zl_bytes : 0);
    if (r <= 16) {
        smem_limit(ctx, subspace_kernel<16>, smem);
        DT_LAUNCH(ctx, subspace_kernel<16>, 1, LA_NT, smem, S, n, L, r, iters, work, zl_in,
                  flag);
    } else {
        smem_limit(ctx, subspace_kernel<32>, smem);
        DT_LAUNCH(ctx, subspace_kernel<32>, 1, LA_NT, smem, S, n, L, r, iters, work, zl_in,
                  flag);
    }
}

void subspace_iter_batch(dt_ctx *ctx, int count, const double *const *S, const int64_t *n,
                         double *const *L, const int64_t *r, int iters, double *const *work,
                         int *flag) {
    SubBatch batch{};
    int k = 0;
    for (int b = 0; b < count; b++) {
        DT_CHECK_ARG(n[b] >= r[b] && r[b] > 0, "subspace_iter: bad sizes n=%lld r=%lld",
                     (long long)n[b], (long long)r[b]);
        if (n[b] > 256 || r[b] > 32) {
            subspace_iter(ctx, S[b], n[b], L[b], r[b], iters, work[b], flag);
            continue;
        }
        batch.S[k] = S[b];
        batch.L[k] = L[b];
        batch.work[k] = work[b];
        batch.n[k] = (int)n[b];
        batch.r[k] = (int)r[b];
        if (++k == SUB_MAX) {
            subspace_mma(ctx, batch, k, iters, flag, false);
            k = 0;
        }
    }
    if (k) subspace_mma(ctx, batch, k, iters, flag, false);
}

void exchange_selftest(dt_ctx *ctx, int *late, long long limit_cycles) {
    launch_pdl_cluster(ctx, exchange_selftest_kernel, 2, SM_NT, 0, 2, late, limit_cycles);
}

void lu_inverse(dt_ctx *ctx, const double *A, int64_t n, double *Ainv, double *work,
                int *flag) {
    DT_CHECK_ARG(n > 0 && n <= 8192, "lu_inverse: bad size %lld", (long long)n);
    DT_LAUNCH(ctx, lu_inverse_kernel, 1, LA_NT, n * sizeof(int), A, n, Ainv, work, flag);
}

namespace {

int64_t gram_groups(int64_t blocks) { return (blocks + GRAM_GROUP - 1) / GRAM_GROUP; }
// The arrival counters, in front, in doubles.
int64_t gram_counters(int64_t blocks) { return (gram_groups(blocks) + 2) / 2; }

size_t orth_scratch_bytes(int r, int64_t blocks) {
    const int64_t rr = (int64_t)r * r, groups = gram_groups(blocks);
    return (size_t)(gram_counters(blocks) + rr * (blocks + (groups > 1 ? groups : 0) + 2)) *
           sizeof(double);
}

}  // namespace

int64_t orth_blocks(const dt_ctx *ctx, int64_t m) {
    return std::max<int64_t>(
        1, std::min<int64_t>({((m + 7) / 8 + 7) / 8, GRAM_MAX_BLOCKS, 4LL * ctx->num_sms}));
}

int64_t orth_alloc(dt_ctx *ctx, DevMem &mem, int r, int64_t blocks, bool may_fail) {
    while (!mem.try_alloc(ctx, orth_scratch_bytes(r, blocks))) {
        if (blocks == 1 && may_fail) return 0;
        if (blocks == 1) mem.alloc(ctx, orth_scratch_bytes(r, 1));  // (fails)
        blocks = (blocks + 3) / 4;
    }
    DT_CUDA(cudaMemsetAsync(mem.get(), 0, gram_counters(blocks) * sizeof(double), ctx->stream));
    return blocks;
}

OrthScratch orth_scratch(void *mem, double *T, int r, int64_t blocks, int *flag) {
    const int64_t rr = (int64_t)r * r, groups = gram_groups(blocks);
    OrthScratch s;
    s.f.counters = static_cast<int *>(mem);
    double *p = static_cast<double *>(mem) + gram_counters(blocks);
    s.T = T;
    s.blocks = blocks;
    s.f.part = s.f.group = p;
    p += rr * blocks;
    if (groups > 1) {
        s.f.group = p;
        p += rr * groups;
    }
    s.f.Linv = p;
    s.Linv2 = p + rr;
    s.f.flag = flag;
    return s;
}

void orth_finish(dt_ctx *ctx, const double *A, int r, int64_t m, const OrthScratch &s, double *out,
                 const int32_t *rows) {
    DT_CHECK_ARG(r > 0 && r <= 32, "orth_finish: bad row count %d", r);
    GramFinish f2 = s.f;
    f2.Linv = s.Linv2;
    const unsigned gblocks = (unsigned)std::max<int64_t>(
        1, std::min<int64_t>(((m + 7) / 8 + 7) / 8, s.blocks));
    const unsigned ablocks = (unsigned)std::max<int64_t>(
        1, std::min<int64_t>(((m + 7) / 8 + 7) / 8, 8LL * ctx->num_sms));
#define DT_ROWS(R)                                                                          \
    do {                                                                                    \
        DT_LAUNCH_PDL(ctx, (rows_apply_kernel<R, true>), gblocks, 256, 0, A, r, m,          \
                      (const double *)s.f.Linv, s.T, nullptr, f2);                          \
        DT_LAUNCH_PDL(ctx, (rows_apply_kernel<R, false>), ablocks, 256, 0,                  \
                      (const double *)s.T, r, m, (const double *)s.Linv2, out, rows, f2);   \
    } while (0)
    if (r <= 8) DT_ROWS(8);
    else if (r <= 16) DT_ROWS(16);
    else if (r <= 24) DT_ROWS(24);
    else DT_ROWS(32);
#undef DT_ROWS
}

void orth_check(dt_ctx *ctx, const int *flag) {
    int h = 0;
    DT_CUDA(cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    DT_CUDA(cudaStreamSynchronize(ctx->stream));
    if (h) fail(DT_ERR_NUMERIC, "orth2: rows are linearly dependent");
}

void orth2_rows(dt_ctx *ctx, double *A, int64_t len1, int64_t len2) {
    // Gram-Schmidt over the rows of A (len1 x len2) equals A = L Q with L the
    // Cholesky factor of A A^T; two passes (CholeskyQR2) for FP64 accuracy.
    DT_CHECK_ARG(len1 > 0 && len1 <= 1024 && len2 >= len1, "orth2: bad sizes %lld x %lld",
                 (long long)len1, (long long)len2);
    if (len1 <= 32) {
        // Three launches: the Gram of A; T = L^{-1} A with the Gram of T; and
        // the second pass's product.
        const int r = (int)len1;
        DevMem T(ctx, (size_t)r * len2 * sizeof(double)), mem;
        const int64_t blocks = orth_alloc(ctx, mem, r, orth_blocks(ctx, len2));
        DevMem flag(ctx, sizeof(int));
        DT_CUDA(cudaMemsetAsync(flag.get(), 0, sizeof(int), ctx->stream));
        const OrthScratch s = orth_scratch(mem.get(), T.as<double>(), r, blocks, flag.as<int>());
        const int64_t cpb = std::max<int64_t>(256, (len2 + blocks - 1) / blocks);
        const unsigned nblk = (unsigned)((len2 + cpb - 1) / cpb);
        if (r <= 8) DT_LAUNCH_PDL(ctx, rows_gram_kernel<8>, nblk, 256, 0, A, r, len2, cpb, s.f);
        else if (r <= 16)
            DT_LAUNCH_PDL(ctx, rows_gram_kernel<16>, nblk, 256, 0, A, r, len2, cpb, s.f);
        else if (r <= 24)
            DT_LAUNCH_PDL(ctx, rows_gram_kernel<24>, nblk, 256, 0, A, r, len2, cpb, s.f);
        else
            DT_LAUNCH_PDL(ctx, rows_gram_kernel<32>, nblk, 256, 0, A, r, len2, cpb, s.f);
        orth_finish(ctx, A, r, len2, s, A, nullptr);
        orth_check(ctx, s.f.flag);
        return;
    }
    DevMem G(ctx, len1 * len1 * sizeof(double));
    DevMem Li(ctx, len1 * len1 * sizeof(double));
    DevMem flag(ctx, sizeof(int));
    DT_CUDA(cudaMemsetAsync(flag.get(), 0, sizeof(int), ctx->stream));
    DevMem T(ctx, len1 * len2 * sizeof(double));
    for (int pass = 0; pass < 2; pass++) {
        gemm_f64(ctx, 0, 1, len1, len1, len2, A, len1, A, len1, G.as<double>(), len1, 0.0);
        DT_LAUNCH(ctx, chol_lower_inv_kernel, 1, 1024, 0, G.as<double>(), (int)len1,
                  Li.as<double>(), flag.as<int>());
        gemm_f64(ctx, 0, 0, len1, len2, len1, Li.as<double>(), len1, A, len1, T.as<double>(),
                 len1, 0.0);
        DT_CUDA(cudaMemcpyAsync(A, T.get(), len1 * len2 * sizeof(double),
                                cudaMemcpyDeviceToDevice, ctx->stream));
    }
    orth_check(ctx, flag.as<int>());
}

}  // namespace dt
