// FP64 dense kernels: the stride-aware TTM, the Gram of an unfolding, the GEMM
// behind ttt_except / matmul (all on the FP64 tensor cores), and deterministic
// norms.
//
// The reference's Function::ttm (template/function/tensor.tpp:272-335) first
// permutes A into A_(n)^T with Operator::tenmatt (operator_cpu.tpp:83-103),
// runs dgemm, then folds back with mattten (operator_cpu.tpp:115-135).  Here the
// mode-n unfolding is never materialised: X is read as the 3-way array
// X[l, i, b] (l < prod_{m<n} I_m unit-stride, i = mode-n index with stride L,
// b the trailing modes) and the result is written straight into the folded
// layout Y[l, j, b].
#include "dt_kernels.cuh"

namespace dt {

// ---------------------------------------------------------------------------
// TTM: Y[l, j, b] = sum_i M(j, i) X[l, i, b], M(j, i) = M[j*msj + i*msi], on the
// FP64 tensor cores (mma.sync m8n8k4).  One CTA of 8 warps owns 64 MT output
// rows p = l + L b and 8 NT outputs j; warp w owns rows 8 MT w .. + 8 MT - 1 as
// MT x NT tiles.  Chunks of 16 i go through a ring of ST stages by cp.async
// (zero-filled past the end), one barrier per chunk.  Bound by memory for a
// large X (one read of X and NT >= J / 8, so X is read once for up to 32
// outputs); the FP64 tensor rate comes next.
//   KF (L == 1, mode 0): i is contiguous; rows are staged with k contiguous,
//        pitch 20.
//   else: rows are contiguous in runs of L; a thread keeps one row (or one
//        group of EV rows) and its address, found by one division, and walks
//        along i.  A tile's rows may lie in several b.
// Either way the four k-columns and eight rows of a fragment load hit distinct
// banks.  VEC: 16-byte copies, where L (KF: I) is a multiple of the elements
// in 16 bytes and X is aligned; else one element a copy.
// 96^4 FP64, 16 outputs: mode 0 243 -> 136 us, mode 1 295 -> 127, mode 3 132 -> 127
// (6.2 TB/s), FP32 215 -> 100 and 119 -> 105; 181 x 203 x 157, 24 outputs 47 -> 29;
// 96 x 16 x 96 x 96, 16 outputs 75 -> 44: before, only runs of L % 256 == 0 rows ran on
// the tensor cores, other layouts on the CUDA cores, ragged ones without a
// pipeline, and few rows split the contraction over two launches.
// ---------------------------------------------------------------------------
namespace {

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, int src_bytes) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem),
                 "r"(src_bytes)
                 : "memory");
}
// One element (4 or 8 bytes), through L1: neighbours in a line come later.
template <int BYTES>
__device__ __forceinline__ void cp_async_el(void *smem, const void *gmem, int src_bytes) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;" ::"r"(s), "l"(gmem),
                 "r"(src_bytes), "n"(BYTES)
                 : "memory");
}
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem, int src_bytes) {
    cp_async_el<8>(smem, gmem, src_bytes);
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void gm_dmma884(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}
// q / d, in 32 bits where both fit (a 64-bit division takes several times as
// many instructions).
__device__ __forceinline__ int64_t div_pos(int64_t q, int64_t d) {
    if (((q | d) >> 32) == 0) return (uint32_t)q / (uint32_t)d;
    return q / d;
}

constexpr int TTM_NT = 256;
constexpr int TTM_BK = 16;
constexpr int TTM_KP = TTM_BK + 4;
// Rows per CTA, ring depth, pitch of a staged k-row and elements of a stage.
__host__ __device__ constexpr int ttm_rows(int mt) { return 64 * mt; }
__host__ __device__ constexpr int ttm_stages(int mt) { return mt == 1 ? 6 : mt == 2 ? 3 : 2; }
template <class TX>
__host__ __device__ constexpr int ttm_pitch(int mt) { return ttm_rows(mt) + (sizeof(TX) == 8 ? 4 : 8); }
template <class TX>
__host__ __device__ constexpr int ttm_xstage(int mt, bool kf) {
    return kf ? ttm_rows(mt) * TTM_KP : TTM_BK * ttm_pitch<TX>(mt);
}
template <class TX>
__host__ __device__ constexpr size_t ttm_smem(int mt, int nt, bool kf) {
    return (size_t)ttm_stages(mt) *
           (ttm_xstage<TX>(mt, kf) * sizeof(TX) + TTM_BK * (8 * nt + 4) * sizeof(double));
}

template <class TX, int MT, int NT, bool KF, bool VEC>
__global__ void __launch_bounds__(TTM_NT) ttm_kernel(const TX *__restrict__ X, int64_t L,
                                                     int64_t I, int64_t P,
                                                     const double *__restrict__ M, int64_t msj,
                                                     int64_t msi, int64_t J,
                                                     double *__restrict__ Y, int64_t kchunk,
                                                     int64_t ysize, const void *const *slot) {
    constexpr int BP = ttm_rows(MT), ST = ttm_stages(MT), MP = 8 * NT + 4;
    constexpr int PITCH = ttm_pitch<TX>(MT), XSTAGE = ttm_xstage<TX>(MT, KF);
    constexpr int EV = VEC ? 16 / (int)sizeof(TX) : 1;
    if (slot) X = static_cast<const TX *>(*slot);
    extern __shared__ __align__(16) uint8_t ttm_sm[];
    TX *Xs = reinterpret_cast<TX *>(ttm_sm);
    double *Ms = reinterpret_cast<double *>(ttm_sm + (size_t)ST * XSTAGE * sizeof(TX));
    const int t = threadIdx.x, w = t >> 5, lane = t & 31, g = lane >> 2, t4 = lane & 3;
    const int64_t p0 = (int64_t)blockIdx.x * BP;
    const int64_t j0 = (int64_t)blockIdx.y * 8 * NT;
    const int64_t ibeg = (int64_t)blockIdx.z * kchunk;
    const int64_t iend = min(I, ibeg + kchunk);
    const int nch = (int)((iend - ibeg + TTM_BK - 1) / TTM_BK);
    Y += (int64_t)blockIdx.z * ysize;

    // Loader.  !KF: RS row slots of EV rows, KP = 256 / RS k-rows per pass;
    // KF: KS slots of EV k, RP = 256 / KS rows per pass.
    constexpr int RS = KF ? TTM_BK / EV : BP / EV;
    constexpr int PER = TTM_NT / RS;
    const int ls = t % RS, other = t / RS;
    const TX *src;
    bool row_ok = true;
    if (KF) {
        src = X + (p0 + other) * I + ibeg + EV * ls;
    } else {
        const int64_t p = p0 + EV * ls;
        row_ok = p < P;
        const int64_t b = row_ok ? div_pos(p, L) : 0;
        src = X + (row_ok ? p - b * L + L * I * b : 0) + (ibeg + other) * L;
    }
    const int mi = t & 15, mj = t >> 4;  // M: one i, j = mj (+ 16)
    const double *msrc = M + (ibeg + mi) * msi + (j0 + mj) * msj;
    auto issue = [&](int c) {
        TX *xd = Xs + (c % ST) * XSTAGE;
        const int left = (int)min((int64_t)TTM_BK, iend - ibeg - (int64_t)c * TTM_BK);
        if (KF) {
            const bool k_ok = EV * ls < left;
#pragma unroll
            for (int q = 0; q < BP / PER; q++) {
                const int r = other + q * PER;
                if (p0 + r < P) {
                    const TX *s = k_ok ? src + (int64_t)q * PER * I : X;
                    TX *d = xd + r * TTM_KP + EV * ls;
                    if (VEC) cp_async16(d, s, k_ok ? 16 : 0);
                    else cp_async_el<sizeof(TX)>(d, s, k_ok ? (int)sizeof(TX) : 0);
                }
            }
            src += TTM_BK;
        } else {
            if (row_ok) {
#pragma unroll
                for (int q = 0; q < TTM_BK / PER; q++) {
                    const int k = other + q * PER;
                    const bool k_ok = k < left;
                    const TX *s = k_ok ? src + (int64_t)q * PER * L : X;
                    TX *d = xd + k * PITCH + EV * ls;
                    if (VEC) cp_async16(d, s, k_ok ? 16 : 0);
                    else cp_async_el<sizeof(TX)>(d, s, k_ok ? (int)sizeof(TX) : 0);
                }
            }
            src += TTM_BK * L;
        }
        double *md = Ms + (c % ST) * TTM_BK * MP + mi * MP;
#pragma unroll
        for (int q = 0; q < (NT + 1) / 2; q++) {
            const int j = mj + 16 * q;
            if (j < 8 * NT) {
                const bool ok = mi < left && j0 + j < J;
                cp_async8(md + j, ok ? msrc + 16 * q * msj : M, ok ? 8 : 0);
            }
        }
        msrc += TTM_BK * msi;
        cp_async_commit();
    };

    double acc[MT][NT][2];
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int n = 0; n < NT; n++) acc[m][n][0] = acc[m][n][1] = 0.0;

    pdl_wait();
#pragma unroll
    for (int c = 0; c < ST - 1; c++) {
        if (c < nch) issue(c);
        else cp_async_commit();
    }
    const int wrow = 8 * MT * w + g;
    for (int c = 0; c < nch; c++) {
        cp_async_wait<ST - 2>();
        __syncthreads();
        if (c + ST - 1 < nch) issue(c + ST - 1);
        else cp_async_commit();
        const TX *xs = Xs + (c % ST) * XSTAGE + (KF ? wrow * TTM_KP + t4 : t4 * PITCH + wrow);
        const double *ms = Ms + (c % ST) * TTM_BK * MP + t4 * MP + g;
#pragma unroll
        for (int kk = 0; kk < TTM_BK / 4; kk++) {
            double bv[NT];
#pragma unroll
            for (int n = 0; n < NT; n++) bv[n] = ms[4 * kk * MP + 8 * n];
#pragma unroll
            for (int m = 0; m < MT; m++) {
                const double av =
                    (double)(KF ? xs[8 * m * TTM_KP + 4 * kk] : xs[4 * kk * PITCH + 8 * m]);
#pragma unroll
                for (int n = 0; n < NT; n++) gm_dmma884(acc[m][n][0], acc[m][n][1], av, bv[n]);
            }
        }
    }

    pdl_trigger();  // dependents may launch while the outputs are stored
    // D[row g][col 2 t + h] of tile (m, n).
    const bool pairs = KF && (J & 1) == 0 && (reinterpret_cast<uintptr_t>(Y) & 15) == 0;
#pragma unroll
    for (int m = 0; m < MT; m++) {
        const int64_t p = p0 + wrow + 8 * m;
        if (p >= P) continue;
        const int64_t b = KF ? p : div_pos(p, L);
        double *y = Y + (p - b * L) + L * J * b;
#pragma unroll
        for (int n = 0; n < NT; n++) {
            const int64_t j = j0 + 8 * n + 2 * t4;
            if (pairs) {
                if (j < J)
                    *reinterpret_cast<double2 *>(y + j) = make_double2(acc[m][n][0], acc[m][n][1]);
            } else {
                if (j < J) y[L * j] = acc[m][n][0];
                if (j + 1 < J) y[L * (j + 1)] = acc[m][n][1];
            }
        }
    }
}

__global__ void sum_splits_kernel(const double *__restrict__ part, int nsplit, int64_t n,
                                  double *__restrict__ out) {
    pdl_wait();
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
         e += (int64_t)gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int z = 0; z < nsplit; z++) s += part[z * n + e];
        out[e] = s;
    }
    pdl_trigger();
}

template <class TX, int MT, int NT, bool KF>
void ttm_launch(dt_ctx *ctx, dim3 grid, bool vec, const TX *X, int64_t L, int64_t I, int64_t P,
                const double *M, int64_t msj, int64_t msi, int64_t J, double *Y, int64_t kchunk,
                int64_t ysize, const void *const *slot) {
    constexpr size_t smem = ttm_smem<TX>(MT, NT, KF);
    if (vec) {
        smem_limit(ctx, ttm_kernel<TX, MT, NT, KF, true>, smem);
        DT_LAUNCH_PDL(ctx, (ttm_kernel<TX, MT, NT, KF, true>), grid, TTM_NT, smem, X, L, I, P, M,
                      msj, msi, J, Y, kchunk, ysize, slot);
    } else {
        smem_limit(ctx, ttm_kernel<TX, MT, NT, KF, false>, smem);
        DT_LAUNCH_PDL(ctx, (ttm_kernel<TX, MT, NT, KF, false>), grid, TTM_NT, smem, X, L, I, P, M,
                      msj, msi, J, Y, kchunk, ysize, slot);
    }
}

template <class TX, int NT>
void ttm_sized(dt_ctx *ctx, const TX *X, int64_t L, int64_t I, int64_t B, const double *M,
               int64_t msj, int64_t msi, int64_t J, double *Y, const void *const *slot) {
    const int64_t P = L * B, jt = ceil_div(J, 8 * NT);
    // 128 rows a CTA (three of them fit an SM) once these fill the GPU, else
    // 64: a short contraction over few rows is a matter of latency.  256 rows in
    // a ring of two for runs of an FP64 X (M is read half as often): 127 against
    // 148 us for one mode of 96^4 with 16 outputs; no gain for FP32 (105 us both)
    // or mode 0 (139 against 136).
    int mt = ceil_div(P, 128) * jt >= 2 * ctx->num_sms ? 2 : 1;
    const bool four = sizeof(TX) == 8 && NT <= 2 && L > 1 && ceil_div(P, 256) * jt >= 4 * ctx->num_sms;
    if (four) mt = 4;
    const int64_t base = ceil_div(P, 64 * mt) * jt;
    // A long contraction over few rows is split, and the partial outputs are
    // summed in a fixed order (deterministic).  Up to 512 the chunks' latencies
    // cost less than the second launch.
    int64_t nsplit = 1;
    if (2 * base <= ctx->num_sms && I > 512)
        nsplit = std::max<int64_t>(1, std::min<int64_t>(ctx->num_sms / base, I / 128));
    const int64_t kchunk = ((I + nsplit - 1) / nsplit + TTM_BK - 1) / TTM_BK * TTM_BK;
    nsplit = (I + kchunk - 1) / kchunk;
    const int64_t ysize = P * J;
    const dim3 grid(ceil_div(P, 64 * mt), (unsigned)jt, (unsigned)nsplit);
    const bool kf = L == 1;
    const bool vec = reinterpret_cast<uintptr_t>(X) % 16 == 0 &&
                     (kf ? I : L) % (int64_t)(16 / sizeof(TX)) == 0;
    auto launch = [&](double *dst) {
        if (kf && mt == 1)
            ttm_launch<TX, 1, NT, true>(ctx, grid, vec, X, L, I, P, M, msj, msi, J, dst, kchunk, ysize, slot);
        else if (kf)
            ttm_launch<TX, 2, NT, true>(ctx, grid, vec, X, L, I, P, M, msj, msi, J, dst, kchunk, ysize, slot);
        else if (four) {
            if constexpr (sizeof(TX) == 8 && NT <= 2)
                ttm_launch<TX, 4, NT, false>(ctx, grid, vec, X, L, I, P, M, msj, msi, J, dst, kchunk,
                                             ysize, slot);
        } else if (mt == 1)
            ttm_launch<TX, 1, NT, false>(ctx, grid, vec, X, L, I, P, M, msj, msi, J, dst, kchunk, ysize, slot);
        else
            ttm_launch<TX, 2, NT, false>(ctx, grid, vec, X, L, I, P, M, msj, msi, J, dst, kchunk, ysize, slot);
    };
    if (nsplit == 1) {
        launch(Y);
        return;
    }
    DevMem part(ctx, (size_t)nsplit * ysize * sizeof(double));
    launch(part.as<double>());
    const unsigned blocks = std::max(1u, std::min<unsigned>(ceil_div(ysize, 256), 8u * ctx->num_sms));
    DT_LAUNCH_PDL(ctx, sum_splits_kernel, blocks, 256, 0, part.as<double>(), (int)nsplit, ysize, Y);
}

}  // namespace

template <class TX>
void ttm_f64(dt_ctx *ctx, const TX *X, int64_t L, int64_t I, int64_t B, const double *M,
             int64_t msj, int64_t msi, int64_t J, double *Y, const void *const *slot) {
    if (L * B == 0 || J == 0) return;
    // One pass over X for up to 32 outputs.
    if (J <= 8)
        ttm_sized<TX, 1>(ctx, X, L, I, B, M, msj, msi, J, Y, slot);
    else if (J <= 16)
        ttm_sized<TX, 2>(ctx, X, L, I, B, M, msj, msi, J, Y, slot);
    else if (J <= 24)
        ttm_sized<TX, 3>(ctx, X, L, I, B, M, msj, msi, J, Y, slot);
    else
        ttm_sized<TX, 4>(ctx, X, L, I, B, M, msj, msi, J, Y, slot);
}
template void ttm_f64<double>(dt_ctx *, const double *, int64_t, int64_t, int64_t,
                              const double *, int64_t, int64_t, int64_t, double *,
                              const void *const *);
template void ttm_f64<float>(dt_ctx *, const float *, int64_t, int64_t, int64_t,
                             const double *, int64_t, int64_t, int64_t, double *,
                             const void *const *);

// ---------------------------------------------------------------------------
// Generic FP64 GEMM C(i, j) = sum_q a(i, q) b(j, q) over operands addressed as
//   a(i, q) = A[koff(q) + i * si],  koff(q) = q * sk            (plain matrix)
//                                   koff(q) = (q % L) + LI*(q / L)  (unfolding)
// This covers Function::gram / ttt_except (both operands are mode-n
// unfoldings X_(n), q running over the other modes) and matmulNN/NT/TN.
// 64 x 64 output tiles on the FP64 tensor cores, split-K over gridDim.z with
// a deterministic reduction of the partial tiles.
// ---------------------------------------------------------------------------
namespace {

struct Operand {
    const double *p;
    int64_t si;   // stride of the output index (i or j)
    int64_t sk;   // stride of q for a plain matrix
    int64_t L;    // unfolding: run length of q with unit stride
    int64_t LI;   // unfolding: stride of q / L
    int unfold;
    int kfast;    // consecutive q are adjacent in memory
};

__device__ __forceinline__ int64_t koff(const Operand &o, int64_t q) {
    if (o.unfold) {
        const int64_t b = q / o.L;
        return (q - b * o.L) + o.LI * b;
    }
    return q * o.sk;
}

constexpr int GM_B = 64;
constexpr int GM_BK = 16;
constexpr int GM_NT = 256;
// Staged rows are 68 doubles apart: the four k-rows of an mma.sync fragment
// load (lanes g + 8 t, 64-bit loads served per half-warp) fall in different
// banks.
constexpr int GM_P = GM_B + 4;

// One thread's four elements of a 16 x 64 operand tile: fetched into
// registers (fetch) while the previous tile is consumed, then stored (store).
struct TileRegs {
    double v[4];
};

__device__ __forceinline__ void fetch_tile(TileRegs &r, const Operand &o, int64_t i0, int64_t nI,
                                           int64_t q0, int64_t qend, int t) {
    if (o.kfast) {
        // 16 consecutive q per row, 16 rows per pass.
        const int k = t & 15;
        const int64_t q = q0 + k;
        const bool qok = q < qend;
        const int64_t off = qok ? koff(o, q) : 0;
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const int64_t i = i0 + (t >> 4) + 16 * s;
            r.v[s] = (qok && i < nI) ? o.p[off + i * o.si] : 0.0;
        }
    } else {
        // 64 consecutive output indices per q, 4 q per pass.
        const int64_t i = i0 + (t & 63);
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const int64_t q = q0 + (t >> 6) + 4 * s;
            r.v[s] = (q < qend && i < nI) ? o.p[koff(o, q) + i * o.si] : 0.0;
        }
    }
}

__device__ __forceinline__ void store_tile(double (*dst)[GM_P], const TileRegs &r,
                                           const Operand &o, int t) {
    if (o.kfast) {
#pragma unroll
        for (int s = 0; s < 4; s++) dst[t & 15][(t >> 4) + 16 * s] = r.v[s];
    } else {
#pragma unroll
        for (int s = 0; s < 4; s++) dst[(t >> 6) + 4 * s][t & 63] = r.v[s];
    }
}

// 64 x 64 output tile per CTA on the FP64 tensor cores (mma.sync m8n8k4):
// warp w owns rows 32 (w % 2) .. + 31 and columns 16 (w / 2) .. + 15 as 4 x 2
// tiles of 8 x 8.  Lane (g, t) supplies a(row g, q = t) and b(col g, q = t)
// and holds D[row g][cols 2 t, 2 t + 1].  The next 16 q of both operands are
// fetched into registers while the current ones are multiplied.
__global__ void __launch_bounds__(GM_NT) gemm_kernel(Operand A, Operand B, int64_t M,
                                                     int64_t N, int64_t K, int64_t kchunk,
                                                     double *__restrict__ C, int64_t ldc,
                                                     double beta, double *__restrict__ part) {
    __shared__ __align__(16) double As[GM_BK][GM_P];
    __shared__ __align__(16) double Bs[GM_BK][GM_P];
    const int t = threadIdx.x, w = t >> 5, lane = t & 31, g = lane >> 2, t4 = lane & 3;
    const int rb = 32 * (w & 1), cb = 16 * (w >> 1);
    const int64_t i0 = (int64_t)blockIdx.x * GM_B;
    const int64_t j0 = (int64_t)blockIdx.y * GM_B;
    const int64_t qbeg = (int64_t)blockIdx.z * kchunk;
    const int64_t qend = min(K, qbeg + kchunk);
    double acc[4][2][2];
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
        for (int n = 0; n < 2; n++) acc[m][n][0] = acc[m][n][1] = 0.0;
    TileRegs ra, rb_;
    if (qbeg < qend) {
        fetch_tile(ra, A, i0, M, qbeg, qend, t);
        fetch_tile(rb_, B, j0, N, qbeg, qend, t);
    }
    for (int64_t q0 = qbeg; q0 < qend; q0 += GM_BK) {
        store_tile(As, ra, A, t);
        store_tile(Bs, rb_, B, t);
        __syncthreads();
        if (q0 + GM_BK < qend) {
            fetch_tile(ra, A, i0, M, q0 + GM_BK, qend, t);
            fetch_tile(rb_, B, j0, N, q0 + GM_BK, qend, t);
        }
#pragma unroll
        for (int kk = 0; kk < GM_BK / 4; kk++) {
            const int k = 4 * kk + t4;
            const double b0 = Bs[k][cb + g], b1 = Bs[k][cb + 8 + g];
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const double a = As[k][rb + 8 * m + g];
                gm_dmma884(acc[m][0][0], acc[m][0][1], a, b0);
                gm_dmma884(acc[m][1][0], acc[m][1][1], a, b1);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const int64_t i = i0 + rb + 8 * m + g;
        if (i >= M) continue;
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int64_t j = j0 + cb + 8 * n + 2 * t4 + h;
                if (j >= N) continue;
                if (part)
                    part[(int64_t)blockIdx.z * M * N + i + M * j] = acc[m][n][h];
                else
                    C[i + ldc * j] = acc[m][n][h] + (beta != 0.0 ? beta * C[i + ldc * j] : 0.0);
            }
    }
}

__global__ void splitk_reduce_kernel(const double *__restrict__ part, int nsplit, int64_t M,
                                     int64_t N, double *__restrict__ C, int64_t ldc,
                                     double beta) {
    const int64_t MN = M * N;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < MN;
         e += (int64_t)gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int z = 0; z < nsplit; z++) s += part[z * MN + e];
        const int64_t i = e % M, j = e / M;
        C[i + ldc * j] = s + (beta != 0.0 ? beta * C[i + ldc * j] : 0.0);
    }
}

void gemm_generic(dt_ctx *ctx, const Operand &A, const Operand &B, int64_t M, int64_t N,
                  int64_t K, double *C, int64_t ldc, double beta) {
    if (M == 0 || N == 0) return;
    const int64_t tiles = (int64_t)ceil_div(M, GM_B) * ceil_div(N, GM_B);
    const int64_t target = 2LL * ctx->num_sms;
    int64_t nsplit = 1;
    if (tiles < target && K > 256) {
        nsplit = (target + tiles - 1) / tiles;
        nsplit = std::min<int64_t>(nsplit, (K + 127) / 128);
        nsplit = std::max<int64_t>(nsplit, 1);
    }
    int64_t kchunk = (K + nsplit - 1) / nsplit;
    kchunk = ((kchunk + GM_BK - 1) / GM_BK) * GM_BK;
    if (kchunk == 0) kchunk = GM_BK;
    nsplit = (K + kchunk - 1) / kchunk;
    if (nsplit < 1) nsplit = 1;
    dim3 grid(ceil_div(M, GM_B), ceil_div(N, GM_B), (unsigned)nsplit);
    if (nsplit == 1) {
        DT_LAUNCH(ctx, gemm_kernel, grid, GM_NT, 0, A, B, M, N, K, kchunk, C, ldc, beta,
                  (double *)nullptr);
    } else {
        DevMem part(ctx, (size_t)nsplit * M * N * sizeof(double));
        DT_LAUNCH(ctx, gemm_kernel, grid, GM_NT, 0, A, B, M, N, K, kchunk, C, ldc, beta,
                  part.as<double>());
        const unsigned blocks = std::min<unsigned>(ceil_div(M * N, 256), 4096u);
        DT_LAUNCH(ctx, splitk_reduce_kernel, blocks, 256, 0, part.as<double>(), (int)nsplit, M,
                  N, C, ldc, beta);
    }
}

Operand plain(const double *p, int64_t si, int64_t sk) {
    Operand o{p, si, sk, 1, 0, 0, sk == 1 ? 1 : 0};
    return o;
}

Operand unfolding(const double *p, int64_t L, int64_t I) {
    Operand o{p, L, 0, L, L * I, 1, L >= 16 ? 1 : 0};
    return o;
}

}  // namespace

// ---------------------------------------------------------------------------
// Gram of a mode-n unfolding, S(i, j) = sum_q X_(n)(i, q) X_(n)(j, q), on the
// FP64 tensor cores.  S is symmetric: only the 8 x 8 tiles of its upper block
// triangle are computed, dealt out evenly over the CTA's warps, and every staged
// row serves all of them: the CTA stages GR_K columns of all rows of X_(n) (n <=
// 256) or of the two 128-row blocks of its block pair, GR_ST chunks deep by
// cp.async, so X is read once up to 200 rows (two CTAs share the tiles up to 256).
// The list takes row r together with row nt - 1 - r (nt + 1 tiles in all), so a
// warp's run of tiles lies in at most three rows: it loads three A fragments a
// k-step and each tile selects one and loads its B fragment, without a branch.
// K is split over the CTAs; a second launch adds the partial tiles in order and
// mirrors them.  The column index q = (l, b) is carried along chunk by chunk (no
// divisions).  Bound by the FP64 tensor rate (64 FMA a cycle and SM): 200 rows, K =
// 40000: 83 us (20 TFLOP/s, of about 37) against 392 us for the whole square on
// 64 x 64 tiles with two divisions per loaded element; 203 rows, K = 28417: 78
// against 276 us.
// KF: q is contiguous in memory for at least 16 columns (L >= 16); rows are
// staged with k contiguous, pitch 20.  Else (L < 16, the first modes) k-rows of
// all i, pitch = 4 (mod 16).  Either way the four k-columns and the rows of a
// fragment load hit distinct banks.  VEC: 16-byte copies (even L, or L = 1 and
// an even I, on a 16-byte aligned X), else 8-byte ones.
// ---------------------------------------------------------------------------
namespace {

constexpr int GR_K = 16;    // columns per chunk
constexpr int GR_ST = 3;    // chunks in the ring
constexpr int GR_KP = GR_K + 4;
constexpr int GR_BLOCK = 128;  // rows of a block when there are several

struct GramArgs {
    const double *X;
    int64_t L, LI, K, kchunk;
    int n;        // rows
    int tiles;    // partial tiles per split (stride of the splits)
    int multi;    // several row blocks, a CTA per pair of them
    int parts;    // one block: CTAs that share its tiles
    int pitch;    // !KF: pitch of a staged k-row
    double *C;    // n x n col-major, written directly when part is null
    double *part;
};

// Block pair p of the upper triangle of nb blocks, row by row.
__host__ __device__ inline void gram_pair(int p, int nb, int &bi, int &bj) {
    bi = 0;
    while (p >= nb - bi) {
        p -= nb - bi;
        bi++;
    }
    bj = bi + p;
}
// Tile s of the upper triangle of nt x nt tiles: rows r and nt - 1 - r in turn.
__host__ __device__ inline void gram_tri(int s, int nt, int &r, int &c) {
    const int f = s / (nt + 1), o = s - f * (nt + 1);
    if (o < nt - f) {
        r = f;
        c = f + o;
    } else {
        r = nt - 1 - f;
        c = r + o - (nt - f);
    }
}

template <int W, int NACC, bool KF, bool VEC>
__global__ void __launch_bounds__(32 * W, W == 8 ? 2 : 1) gram_kernel(GramArgs a) {
    extern __shared__ __align__(16) double gs[];
    constexpr int NT = 32 * W;
    const int t = threadIdx.x, w = t >> 5, lane = t & 31, g = lane >> 2, t4 = lane & 3;
    int bi = 0, bj = 0;
    if (a.multi) gram_pair(blockIdx.x, (a.n + GR_BLOCK - 1) / GR_BLOCK, bi, bj);
    const bool rect = bi != bj;
    const int i0 = bi * GR_BLOCK, j0 = bj * GR_BLOCK;
    const int ni = a.multi ? min(GR_BLOCK, a.n - i0) : a.n;   // rows of the first block
    const int nj = rect ? min(GR_BLOCK, a.n - j0) : 0;        // staged rows of the second
    const int nti = (ni + 7) / 8, ntj = rect ? (nj + 7) / 8 : nti;
    const int rows = 8 * (rect ? nti + ntj : nti);            // staged rows
    const int stage = KF ? rows * GR_KP : GR_K * a.pitch;
    const int64_t qbeg = (int64_t)blockIdx.y * a.kchunk, qend = min(a.K, qbeg + a.kchunk);
    const int nch = (int)((qend - qbeg + GR_K - 1) / GR_K);
    // Staged rows past n are zero in every chunk.
    for (int q = 0; q < GR_ST; q++) {
        const int pi = 8 * nti - ni, pj = rect ? 8 * ntj - nj : 0;
        for (int e = t; e < (pi + pj) * GR_K; e += NT) {
            const int x = e / GR_K, k = e % GR_K;
            const int at = x < pi ? ni + x : 8 * nti + nj + (x - pi);
            gs[q * stage + (KF ? at * GR_KP + k : k * a.pitch + at)] = 0.0;
        }
    }

    // This warp's tiles: [s0, s1) of the list, in at most three rows; tile x
    // is in the first up to x = x1, in the second up to x2.
    const int total = rect ? nti * ntj : nti * (nti + 1) / 2;
    const int wt = W * a.parts, wi = W * (a.multi ? 0 : blockIdx.x) + w;
    const int s0 = (int)((int64_t)wi * total / wt), s1 = (int)((int64_t)(wi + 1) * total / wt);
    int row[3], col[3], x1 = NACC, x2 = NACC;  // col: column tile of x = 0 continued
    if (rect) {  // the first block is whole: one row of ntj tiles per warp
        row[0] = row[1] = row[2] = w;
        col[0] = col[1] = col[2] = nti;  // staged after the row tiles
    } else {
        gram_tri(min(s0, total - 1), nti, row[0], col[0]);
        x1 = min(nti - col[0], NACC);
        gram_tri(min(s0 + x1, total - 1), nti, row[1], col[1]);
        x2 = min(x1 + nti - col[1], NACC);
        gram_tri(min(s0 + x2, total - 1), nti, row[2], col[2]);
        col[1] -= x1;
        col[2] -= x2;
    }

    // Loader: KF: k = (VEC ? 2 : 1) (t % KT), rows t / KT + ...; else warp w
    // stages k = w, w + W, lanes along i.
    constexpr int EV = VEC ? 2 : 1;
    constexpr int KT = GR_K / EV;             // KF: threads along k
    constexpr int KPW = KF ? 1 : GR_K / W;    // !KF: k-rows per warp
    const int nq = (int)(qend - qbeg);  // this split's columns
    const double *src[KPW];             // the next chunk's column, l of it
    int64_t ql[KPW];
    for (int x = 0; x < KPW; x++) {
        const int64_t q = qbeg + (KF ? EV * (t % KT) : w + x * W);
        const int64_t b = q / a.L;
        ql[x] = q - b * a.L;
        src[x] = a.X + ql[x] + a.LI * b + (int64_t)i0 * a.L;
    }
    const int64_t jump = rect ? (int64_t)(j0 - i0 - ni) * a.L : 0;  // to the second block's rows
    auto issue = [&](int c) {
        double *dst = gs + (c % GR_ST) * stage;
#pragma unroll
        for (int x = 0; x < KPW; x++) {
            const int k = KF ? EV * (t % KT) : w + x * W;
            const int left = nq - c * GR_K - k;
            // A pair is cut only where nq is odd.
            const int bytes = left <= 0 ? 0 : KF && left < EV ? 8 : 8 * EV;
            for (int i = KF ? t / KT : EV * lane; i < ni + nj; i += KF ? NT / KT : 32 * EV) {
                const bool second = i >= ni;
                const int at = second ? 8 * nti + (i - ni) : i;
                const double *p = bytes ? src[x] + i * a.L + (second ? jump : 0) : a.X;
                double *o = dst + (KF ? at * GR_KP + k : k * a.pitch + at);
                if (VEC) cp_async16(o, p, bytes);
                else cp_async8(o, p, bytes);
            }
            ql[x] += GR_K;
            src[x] += GR_K;
            while (ql[x] >= a.L) {
                ql[x] -= a.L;
                src[x] += a.LI - a.L;
            }
        }
        cp_async_commit();
    };

    double acc[NACC][2];
#pragma unroll
    for (int x = 0; x < NACC; x++) acc[x][0] = acc[x][1] = 0.0;
    const int RS = KF ? 8 * GR_KP : 8;             // a row tile further
    const int KS = KF ? 4 : 4 * a.pitch;           // a k-step further
    const int lane_off = KF ? g * GR_KP + t4 : t4 * a.pitch + g;
    const int ar0 = lane_off + row[0] * RS, ar1 = lane_off + row[1] * RS,
              ar2 = lane_off + row[2] * RS;
    const int bc0 = lane_off + col[0] * RS, bc1 = lane_off + col[1] * RS,
              bc2 = lane_off + col[2] * RS;

    pdl_wait();
    for (int c = 0; c < GR_ST - 1; c++) {
        if (c < nch) issue(c);
        else cp_async_commit();
    }
    for (int c = 0; c < nch; c++) {
        cp_async_wait<GR_ST - 2>();
        __syncthreads();
        if (c + GR_ST - 1 < nch) issue(c + GR_ST - 1);
        else cp_async_commit();
        const double *base = gs + (c % GR_ST) * stage;
#pragma unroll
        for (int kk = 0; kk < GR_K / 4; kk++) {
            const double *p = base + kk * KS;
            const double a0 = p[ar0], a1 = p[ar1], a2 = p[ar2];
            // Selected anew each k-step: kept, the tiles' addresses cost more
            // registers than a thread has.
            asm volatile("" : "+r"(x1), "+r"(x2));
            // Tiles past s1 read what lies there (within the allocation) and
            // are not stored.
#pragma unroll
            for (int x = 0; x < NACC; x++) {
                const double av = x < x1 ? a0 : x < x2 ? a1 : a2;
                const int bc = x < x1 ? bc0 : x < x2 ? bc1 : bc2;
                gm_dmma884(acc[x][0], acc[x][1], av, p[bc + x * RS]);
            }
        }
    }
    pdl_trigger();
    // D[row g][cols 2 t, 2 t + 1] of tile x.
#pragma unroll
    for (int x = 0; x < NACC; x++) {
        if (s0 + x >= s1) continue;
        if (a.part) {
            const int64_t tile = (int64_t)blockIdx.y * a.tiles +
                                 (a.multi ? 256 * (int64_t)blockIdx.x : 0) + s0 + x;
            *reinterpret_cast<double2 *>(a.part + tile * 64 + g * 8 + 2 * t4) =
                make_double2(acc[x][0], acc[x][1]);
        } else {
            const int r = x < x1 ? row[0] : x < x2 ? row[1] : row[2];
            const int c = x + (x < x1 ? col[0] : x < x2 ? col[1] : col[2]) - (rect ? nti : 0);
            const int64_t i = i0 + 8 * r + g;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int64_t j = j0 + 8 * c + 2 * t4 + h;
                if (i < a.n && j < a.n) {
                    a.C[i + (int64_t)a.n * j] = acc[x][h];
                    if (rect || r != c) a.C[j + (int64_t)a.n * i] = acc[x][h];
                }
            }
        }
    }
}

// One CTA per tile: four threads an entry, each adding every fourth split (16
// loads in flight), then the four in order; the tile and its mirror go to C.
__global__ void __launch_bounds__(256) gram_sum_kernel(const double *__restrict__ part, int nsplit,
                                                       int tiles, int n, int multi,
                                                       double *__restrict__ C) {
    __shared__ double red[4][64];
    const int t = threadIdx.x, e = t & 63, q = t >> 6;
    int bi = 0, bj = 0, s = blockIdx.x;
    if (multi) {
        gram_pair(s / 256, (n + GR_BLOCK - 1) / GR_BLOCK, bi, bj);
        s %= 256;
    }
    const int ni = multi ? min(GR_BLOCK, n - bi * GR_BLOCK) : n;
    const int nti = (ni + 7) / 8;
    const int ntj = bi != bj ? (min(GR_BLOCK, n - bj * GR_BLOCK) + 7) / 8 : nti;
    if (s >= (bi != bj ? nti * ntj : nti * (nti + 1) / 2)) return;
    int r, c;
    if (bi != bj) {
        r = s / ntj;
        c = s - r * ntj;
    } else {
        gram_tri(s, nti, r, c);
    }
    pdl_wait();
    const double *p = part + (int64_t)blockIdx.x * 64 + e;
    double sum = 0.0;
    for (int z = q; z < nsplit; z += 64) {
        double v[16];
#pragma unroll
        for (int x = 0; x < 16; x++)
            v[x] = z + 4 * x < nsplit ? p[(int64_t)(z + 4 * x) * tiles * 64] : 0.0;
#pragma unroll
        for (int x = 0; x < 16; x++) sum += v[x];
    }
    red[q][e] = sum;
    __syncthreads();
    pdl_trigger();
    if (q == 0) {
        const double v = (red[0][e] + red[1][e]) + (red[2][e] + red[3][e]);
        const int64_t i = bi * GR_BLOCK + 8 * r + (e >> 3), j = bj * GR_BLOCK + 8 * c + (e & 7);
        if (i < n && j < n) {
            C[i + (int64_t)n * j] = v;
            if (bi != bj || r != c) C[j + (int64_t)n * i] = v;
        }
    }
}

template <int W, int NACC>
void launch_gram(dt_ctx *ctx, const GramArgs &a, dim3 grid, bool kf, bool vec) {
    // The ring, and room for the tiles a warp computes past its last.
    const int rows = a.multi ? 2 * GR_BLOCK : (a.n + 7) / 8 * 8;
    const size_t smem = ((size_t)GR_ST * (kf ? rows * GR_KP : GR_K * a.pitch) +
                         (size_t)NACC * (kf ? 8 * GR_KP : 8)) * sizeof(double);
#define DT_GRAM(KF, VEC)                                                   \
    do {                                                                   \
        auto kern = gram_kernel<W, NACC, KF, VEC>;                         \
        smem_limit(ctx, kern, smem);                                       \
        DT_LAUNCH_PDL(ctx, kern, grid, 32 * W, smem, a);                   \
    } while (0)
    if (kf && vec) DT_GRAM(true, true);
    else if (kf) DT_GRAM(true, false);
    else if (vec) DT_GRAM(false, true);
    else DT_GRAM(false, false);
#undef DT_GRAM
}

// S = X_(n) X_(n)^T; the partial tiles go to `scratch` (scratch_doubles) or, when
// it is null, to a stream-ordered allocation.
void gram_f64(dt_ctx *ctx, const double *X, int64_t L, int64_t I, int64_t B, double *C,
              double *scratch, int64_t scratch_doubles) {
    DT_CHECK_ARG(I < (int64_t(1) << 24), "gram: mode size %lld", (long long)I);
    GramArgs a{};
    a.X = X;
    a.L = L;
    a.LI = L * I;
    a.K = L * B;
    a.n = (int)I;
    a.C = C;
    const int nt = (a.n + 7) / 8;
    a.multi = nt > 32;
    // Above 25 tiles a row (325 in all, 21 per warp of 16) two CTAs share them:
    // more accumulators do not fit a thread's 128 registers.
    a.parts = !a.multi && nt > 25 ? 2 : 1;
    const int nb = (a.n + GR_BLOCK - 1) / GR_BLOCK;
    const int64_t pairs = a.multi ? (int64_t)nb * (nb + 1) / 2 : a.parts;
    DT_CHECK_ARG(256 * pairs <= INT32_MAX, "gram: mode size %lld", (long long)I);
    a.tiles = (int)(a.multi ? 256 * pairs : nt * (nt + 1) / 2);
    const bool kf = L >= GR_K;
    const bool vec = reinterpret_cast<uintptr_t>(X) % 16 == 0 &&
                     (kf ? L % 2 == 0 : L == 1 && I % 2 == 0);
    const int staged = a.multi ? 2 * GR_BLOCK : 8 * nt;
    a.pitch = (staged + 11) / 16 * 16 + 4;
    // Enough splits for the CTAs that fit (two of 8 warps or one of 16 per
    // SM), of at least two chunks each.
    const int tiles8 = nt * (nt + 1) / 2;
    const bool wide = a.multi || nt > 16;
    const int64_t target = (wide ? 1LL : 2LL) * ctx->num_sms;
    int64_t nsplit = std::max<int64_t>(1, std::min<int64_t>(target / pairs, (a.K + 2 * GR_K - 1) / (2 * GR_K)));
    if (scratch) nsplit = std::max<int64_t>(1, std::min<int64_t>(nsplit, scratch_doubles / (64LL * a.tiles)));
    // A split's columns are counted in 32 bits.
    const int64_t least = std::max<int64_t>(1, (a.K + (int64_t(1) << 30) - 1) >> 30);
    nsplit = std::max(nsplit, least);
    DevMem part;
    for (;; nsplit = std::max(least, nsplit / 2)) {
        a.kchunk = std::max<int64_t>(GR_K, ((a.K + nsplit - 1) / nsplit + GR_K - 1) / GR_K * GR_K);
        nsplit = std::max<int64_t>(1, (a.K + a.kchunk - 1) / a.kchunk);
        // Fewer splits where there is no room for their tiles; one needs none.
        const size_t bytes = (size_t)nsplit * a.tiles * 64 * sizeof(double);
        if (nsplit == 1 || scratch || part.try_alloc(ctx, bytes)) break;
        if (nsplit <= least) part.alloc(ctx, bytes);  // (fails)
    }
    if (nsplit > 1) a.part = scratch ? scratch : part.as<double>();
    const dim3 grid((unsigned)pairs, (unsigned)nsplit);
    // Tiles per warp, rounded up to the next size there is a kernel for.
    const int per8 = (tiles8 + 7) / 8, per16 = (tiles8 + 16 * a.parts - 1) / (16 * a.parts);
    if (a.multi) launch_gram<16, 16>(ctx, a, grid, kf, vec);
    else if (wide && per16 <= 12) launch_gram<16, 12>(ctx, a, grid, kf, vec);
    else if (wide && per16 <= 17) launch_gram<16, 17>(ctx, a, grid, kf, vec);
    else if (wide) launch_gram<16, 21>(ctx, a, grid, kf, vec);
    else if (per8 <= 2) launch_gram<8, 2>(ctx, a, grid, kf, vec);
    else if (per8 <= 4) launch_gram<8, 4>(ctx, a, grid, kf, vec);
    else if (per8 <= 7) launch_gram<8, 7>(ctx, a, grid, kf, vec);
    else if (per8 <= 10) launch_gram<8, 10>(ctx, a, grid, kf, vec);
    else if (per8 <= 14) launch_gram<8, 14>(ctx, a, grid, kf, vec);
    else launch_gram<8, 17>(ctx, a, grid, kf, vec);
    if (a.part)
        DT_LAUNCH_PDL(ctx, gram_sum_kernel, (unsigned)a.tiles, 256, 0, (const double *)a.part,
                      (int)nsplit, a.tiles, a.n, a.multi, C);
}

}  // namespace

void ttt_f64(dt_ctx *ctx, const double *A, const double *Bt, int64_t L, int64_t IA,
             int64_t IB, int64_t B, double *C) {
    if (A == Bt && IA == IB && IA > 0)
        gram_f64(ctx, A, L, IA, B, C, nullptr, 0);
    else
        gemm_generic(ctx, unfolding(A, L, IA), unfolding(Bt, L, IB), IA, IB, L * B, C, IA, 0.0);
}

void gram_f64_scratch(dt_ctx *ctx, const double *A, int64_t L, int64_t I, int64_t B, double *C,
                      double *scratch, int64_t scratch_doubles) {
    gram_f64(ctx, A, L, I, B, C, scratch, scratch_doubles);
}

void gemm_f64(dt_ctx *ctx, int transA, int transB, int64_t m, int64_t n, int64_t k,
              const double *A, int64_t lda, const double *B, int64_t ldb, double *C,
              int64_t ldc, double beta) {
    // a(i, q) = op(A)(i, q); b(j, q) = op(B)(q, j).
    const Operand a = transA ? plain(A, lda, 1) : plain(A, 1, lda);
    const Operand b = transB ? plain(B, 1, ldb) : plain(B, ldb, 1);
    gemm_generic(ctx, a, b, m, n, k, C, ldc, beta);
}

// ---------------------------------------------------------------------------
// Norms and conversions.
// ---------------------------------------------------------------------------
namespace {

template <class T>
__global__ void sumsq_partial_kernel(const T *__restrict__ x, int64_t n,
                                     double *__restrict__ part) {
    pdl_wait();
    double s = 0.0;
#pragma unroll 8
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
         e += (int64_t)gridDim.x * blockDim.x) {
        const double v = (double)x[e];
        s = fma(v, v, s);
    }
    pdl_trigger();
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) part[blockIdx.x] = s;
    }
}

__global__ void sum_partials_kernel(const double *__restrict__ part, int n,
                                    double *__restrict__ out) {
    pdl_wait();
    double s = 0.0;
    for (int e = threadIdx.x; e < n; e += blockDim.x) s += part[e];
    pdl_trigger();
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) out[0] = s;
    }
}

__global__ void f32_to_f64_kernel(const float *__restrict__ x, int64_t n,
                                  double *__restrict__ y) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
         e += (int64_t)gridDim.x * blockDim.x)
        y[e] = (double)x[e];
}

}  // namespace

void sumsq(dt_ctx *ctx, const void *x, int dtype, int64_t n, double *out) {
    // One block up to 4096 entries (16 a thread): its partial sum is the result.
    const int blocks =
        n <= 4096 ? 1 : std::min<int>(4 * ctx->num_sms, (int)ceil_div(n, 256));
    DevMem part;
    double *dst = out;
    if (blocks > 1) {
        part.alloc(ctx, (size_t)blocks * sizeof(double));
        dst = part.as<double>();
    }
    if (dtype == DT_F64)
        DT_LAUNCH_PDL(ctx, sumsq_partial_kernel<double>, blocks, 256, 0,
                      static_cast<const double *>(x), n, dst);
    else
        DT_LAUNCH_PDL(ctx, sumsq_partial_kernel<float>, blocks, 256, 0,
                      static_cast<const float *>(x), n, dst);
    if (blocks > 1)
        DT_LAUNCH_PDL(ctx, sum_partials_kernel, 1, 1024, 0, (const double *)dst, blocks, out);
}

void f32_to_f64(dt_ctx *ctx, const float *x, int64_t n, double *y) {
    const int blocks = std::max(1, std::min<int>(8 * ctx->num_sms, (int)ceil_div(n, 256)));
    DT_LAUNCH(ctx, f32_to_f64_kernel, blocks, 256, 0, x, n, y);
}

}  // namespace dt
