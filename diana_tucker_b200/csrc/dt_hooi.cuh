// Dense HOOI drivers (FP64 and the tensor-core mixed-precision variant).
#pragma once

#include <algorithm>
#include <functional>
#include <vector>

#include "dt_core.cuh"

namespace dt {

// The FP64 HOOI: TTM chain over a dimension tree, FP64 Gram and
// subspace iteration.  X may be FP64 or FP32 (read as FP32, computed in FP64).
// The GNU C library's rand() sequence after srand(seed), restated (dt_hooi.cu).
class LibcRand {
   public:
    explicit LibcRand(unsigned seed);
    int32_t next();  // in [0, 2^31 - 1], as rand()

   private:
    int32_t s_[31];
    int f_ = 3, r_ = 0;
};

// The state of a device-side sweep loop: what the call asked for, the sweeps
// done, the last residual and the residual of every sweep.
struct LoopState {
    int it, max_sweeps;
    double prev, thr;
    const void *x;  // this call's X (the captured kernels take it from here)
    double hist[DT_MAX_HIST];
};

// A sweep loop as one graph: a WHILE node whose body is one captured sweep
// followed by a kernel that computes the sweep's residual from scal[0] =
// ||X||^2 and scal[1] = ||G||^2, applies the stop rule (residual change below
// thr, or max_sweeps done) and sets the loop's condition.  One graph launch
// runs every sweep with no host round trip.  The stop rule's numbers and X's
// address are in the LoopState that launch() writes, so one graph serves every
// call of a plan.
class SweepLoop {
   public:
    SweepLoop() = default;
    SweepLoop(const SweepLoop &) = delete;
    SweepLoop &operator=(const SweepLoop &) = delete;
    ~SweepLoop();
    // Captures sweep's launches; false (and no further attempts) when the
    // runtime refuses any step: the host drives the sweeps then.
    bool build(dt_ctx *ctx, const double *scal, const std::function<void()> &sweep);
    void launch(dt_ctx *ctx, double thr, int max_sweeps, const void *x);
    LoopState *state(dt_ctx *ctx);       // device memory, allocated on first use
    int64_t launches_per_sweep() const { return launches_; }

   private:
    cudaGraphExec_t exec_ = nullptr;
    bool failed_ = false;
    int64_t launches_ = 0;
    DevMem state_;
};

struct DenseHooi {
    dt_ctx *ctx = nullptr;
    int dtype = DT_F64;
    int N = 0;
    int64_t I[16] = {}, R[16] = {};
    int64_t xsize = 0;
    dt_hooi_opts opts{};
    const void *Xdev = nullptr;
    DevMem X64;               // FP64 copy when needed
    std::vector<DevMem> U;    // I_n x R_n col-major
    DevMem S, work, flag, scal, G;
    bool allocated = false;
    // Orthonormal initial factors of the last explicit seed (DT_INIT_RANDN_LIBC).
    DevMem init_cache;
    bool init_cached = false;
    unsigned init_seed = 0;
    int hosvd_iters = 30;
    LaunchTimer *xtimer = nullptr;  // times the TTM launches that read X
    DevArena arena;                 // a captured sweep's intermediates
    DevMem arena_mem;
    const void *const *xslot = nullptr;  // where a captured sweep finds X
    DevMem hosvd_start;             // HOSVD's Gaussian starts, mode after mode
    // Where a call keeps its random draws, so that starting over draws no more
    // (null: not kept).
    std::vector<double> *drawn = nullptr;

    // Allocates the buffers on the first call; a later call on the same
    // object (same shapes and ranks) keeps them, so a captured sweep graph
    // stays valid.
    void setup(dt_ctx *c, const void *X, int dtype, int n, const int64_t *shape,
               const int64_t *ranks, const dt_hooi_opts &o);
    // Writes the initial factors into dst[m] (I_m x R_m col-major device
    // buffers; null: this object's U).
    void init_factors(double *const *U_user, double *const *dst = nullptr);
    // loop: runs the sweeps as one captured device-side loop (null, or where
    // each sweep needs the host: launches them directly).
    void run(double *G_user, double *const *U_user, dt_hooi_report *rep,
             SweepLoop *loop = nullptr);

   private:
    DevMem contract(const void *t, int tdtype, int64_t *shape, int m);
    DevMem contract_all(const void *t, int tdtype, int64_t *shape, std::vector<int> modes);
    void node(int lo, int hi, const void *T, int tdtype, const int64_t *shape);
    void leaf(int n, const double *Y, const int64_t *shape);
    void sweep();
    double read_scalar(int k);
    void read_scalars(int k, int n, double *out);
    double x_pass_flop() const;
    double x_pass_bytes() const;
    bool build_loop(SweepLoop &loop);
};

// BF16 / split-BF16 tensor-core HOOI (dt_hooi_tc.cu).
// upload: X (FP32) is still arriving from the host through it; its chunks
// are rounded to BF16 as they land (only where hooi_lowprec_tc_ok holds).
void hooi_dense_lowprec(dt_ctx *ctx, const void *X, int dtype, int ndim, const int64_t *shape,
                        const int64_t *ranks, const dt_hooi_opts &opts, double *G,
                        double *const *U, dt_hooi_report *report,
                        ChunkedUpload *upload = nullptr);
// Whether the tensor-core HOOI runs these shapes (otherwise it falls back to
// the FP64 engine).
bool hooi_lowprec_tc_ok(int ndim, const int64_t *shape, const int64_t *ranks);

}  // namespace dt
