"""Failure handling, with every failure made on the host or by a wait that
nothing completes: no test faults, traps or hangs the GPU.

- A bounded device wait that runs out (dt_selftest_wait_timeout: an mbarrier
  that nothing arrives on, a limit of 2e6 cycles, about 1 ms) returns
  DT_ERR_TIMEOUT; the context's next calls give the same results as before.
- A device-memory cap (dt_ctx_set_mem_limit) below a call's needs fails the
  call with DT_ERR_NOMEM before it allocates past the cap; the bytes the
  context holds come back to where they were, and lifting the cap gives the
  uncapped results bit for bit.
- NaN inputs: dense HOOI (FP64 and the tensor-core path) and sparse HOOI
  fail with DT_ERR_NUMERIC; a NaN tensor in a batch gives a NaN relative
  error for that tensor alone, the others bit-identical to a clean batch.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _codes():
    from diana_tucker_b200 import _lib
    return _lib


def _dense(shape=(40, 36, 32), seed=0):
    rng = np.random.default_rng(seed)
    return np.asfortranarray(rng.standard_normal(shape))


def test_bounded_wait_runs_out_and_context_survives(ctx):
    from diana_tucker_b200 import DTError
    L = _codes()
    X = _dense()
    G1, U1, _ = ctx.hooi_dense(X, (4, 4, 4), max_sweeps=3)
    with pytest.raises(DTError) as e:
        ctx.selftest_wait_timeout(2_000_000)
    assert e.value.code == L.DT_ERR_TIMEOUT
    # A limit above the library's own budget is refused before any launch.
    with pytest.raises(DTError) as e:
        ctx.selftest_wait_timeout(4_000_000_000)
    assert e.value.code == L.DT_ERR_ARG
    G2, U2, _ = ctx.hooi_dense(X, (4, 4, 4), max_sweeps=3)
    assert np.array_equal(G1, G2)
    for a, b in zip(U1, U2):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("limit", [0, 20_000, 2_000_000])
def test_cluster_exchange_that_runs_out_is_late_for_all_threads(ctx, limit):
    """The self-test's second kernel waits in the exchange of the subspace
    iteration for data that nobody sends: whatever the limit, all threads of both
    CTAs leave with the same verdict (the call reports the timeout, not a
    disagreement), and the iteration on a cluster runs as before."""
    from diana_tucker_b200 import DTError
    L = _codes()
    rng = np.random.default_rng(8)
    Y = np.asfortranarray(rng.standard_normal((96, 12, 20)))
    L0, _ = np.linalg.qr(rng.standard_normal((96, 16)))
    q = ctx.als(Y, 0, L0, 5)
    n0 = ctx.kernel_launches()
    with pytest.raises(DTError) as e:
        ctx.selftest_wait_timeout(limit)
    assert e.value.code == L.DT_ERR_TIMEOUT
    assert ctx.kernel_launches() - n0 == 2
    assert np.array_equal(ctx.als(Y, 0, L0, 5), q)


XBYTES = 40 * 36 * 32 * 8


@pytest.mark.parametrize("tiled,cap", [(True, 1 << 20), (False, XBYTES + (16 << 10))])
def test_memory_cap_fails_cleanly_then_lifts(ctx, tiled, cap):
    """A 1.5 MB X under a 1 MiB cap fails at its staging; a 369 KB X under a
    cap of X + 16 KiB fails further into the call, in the HOOI's buffers."""
    from diana_tucker_b200 import Context, DTError
    L = _codes()
    X = _dense()
    Xc = np.asfortranarray(np.tile(X, (4, 1, 1))) if tiled else X
    Gref, Uref, _ = ctx.hooi_dense(X, (4, 4, 4), max_sweeps=3)
    c = Context(0)
    try:
        before = c.mem_usage()[0]
        c.set_mem_limit(cap)
        for _ in range(2):  # a repeated failure holds nothing more
            with pytest.raises(DTError) as e:
                c.hooi_dense(Xc, (4, 4, 4), max_sweeps=3)
            assert e.value.code == L.DT_ERR_NOMEM
            c.synchronize()
            assert c.mem_usage()[0] == before
        c.set_mem_limit(0)
        G, U, _ = c.hooi_dense(X, (4, 4, 4), max_sweeps=3)
        assert np.array_equal(G, Gref)
        for a, b in zip(U, Uref):
            assert np.array_equal(a, b)
        assert c.mem_usage()[1] > 0
    finally:
        c.close()


def test_memory_cap_on_sparse_tensor_and_tensor_core_path(ctx):
    from diana_tucker_b200 import DT_PREC_BF16XH, Context, DTError
    L = _codes()
    rng = np.random.default_rng(3)
    shape = (64, 48, 40)
    X = rng.standard_normal(shape).astype(np.float32)
    kw = dict(precision=DT_PREC_BF16XH, max_sweeps=4, tol=1e-9, inner_iters=2)
    Gref, Uref, _ = ctx.hooi_dense(X, (8, 8, 8), **kw)
    idx = [rng.integers(0, s, 5000) for s in (300, 200, 100)]
    vals = rng.standard_normal(5000)
    c = Context(0)
    try:
        c.set_mem_limit(64 << 10)
        with pytest.raises(DTError) as e:
            c.sptensor(idx, vals, (300, 200, 100))
        assert e.value.code == L.DT_ERR_NOMEM
        with pytest.raises(DTError) as e:
            c.hooi_dense(X, (8, 8, 8), **kw)
        assert e.value.code == L.DT_ERR_NOMEM
        c.set_mem_limit(0)
        G, U, _ = c.hooi_dense(X, (8, 8, 8), **kw)
        assert np.array_equal(G, Gref)
        sp = c.sptensor(idx, vals, (300, 200, 100))
        sp.close()
    finally:
        c.close()


@pytest.mark.parametrize("prec", ["FP64", "BF16XH"])
def test_nan_input_dense_hooi(ctx, prec):
    import diana_tucker_b200 as dtb
    from diana_tucker_b200 import DTError
    L = _codes()
    rng = np.random.default_rng(5)
    X = rng.standard_normal((64, 48, 40)).astype(np.float32 if prec != "FP64" else np.float64)
    X[10, 7, 3] = np.nan
    with pytest.raises(DTError) as e:
        ctx.hooi_dense(X, (8, 8, 8), max_sweeps=3, precision=getattr(dtb, "DT_PREC_" + prec),
                       inner_iters=2)
    assert e.value.code == L.DT_ERR_NUMERIC
    X[10, 7, 3] = 0.0
    G, U, rep = ctx.hooi_dense(X, (8, 8, 8), max_sweeps=3,
                               precision=getattr(dtb, "DT_PREC_" + prec), inner_iters=2)
    assert np.isfinite(rep["residual"]) and np.all(np.isfinite(G))


def test_nan_input_sparse_hooi(ctx):
    from diana_tucker_b200 import DTError, datasets
    L = _codes()
    idx, vals, shape = datasets.sparse_zipf((500, 400, 300), 20_000, seed=2)
    vals = np.array(vals, dtype=np.float64)
    vals[123] = np.nan
    R = (4, 4, 4)
    Ut0 = datasets.random_orthonormal_transposed(shape, R, 1)
    sp = ctx.sptensor(idx, vals, shape)
    try:
        with pytest.raises(DTError) as e:
            sp.hooi(R, 2, Ut0)
        assert e.value.code == L.DT_ERR_NUMERIC
    finally:
        sp.close()


def test_nan_tensor_in_a_batch_stays_in_its_slot(ctx):
    from diana_tucker_b200 import datasets
    items = datasets.batched_small(count=32, seed=9)
    rng = np.random.default_rng(109)
    U0 = [[np.linalg.qr(rng.standard_normal((X.shape[n], r[n])))[0] for n in range(3)]
          for X, r in items]
    tensors = [X.copy() for X, _ in items]
    ranks = [r for _, r in items]
    _, G1, e1, _ = ctx.hooi_batched(tensors, ranks, U0, sweeps=3, block_threads=256)
    tensors[5][1, 2, 0] = np.nan
    _, G2, e2, _ = ctx.hooi_batched(tensors, ranks, U0, sweeps=3, block_threads=256)
    assert np.isnan(e2[5])
    keep = [t for t in range(len(items)) if t != 5]
    assert np.array_equal(e1[keep], e2[keep])
    for t in keep:
        assert np.array_equal(G1[t], G2[t])


def _device(shape, seed, dtype="float64"):
    import torch
    X = np.random.default_rng(seed).standard_normal(shape)
    return torch.from_numpy(X.reshape(-1, order="F").copy()).cuda().to(getattr(torch, dtype))


def _peak(shape, ranks, **kw):
    """Bytes that one call takes in a context that keeps nothing yet."""
    from diana_tucker_b200 import Context
    with Context(0) as c:
        c.hooi_dense(_device(shape, 1), ranks, shape=shape, **kw)
        return c.mem_usage()[1]


@pytest.mark.parametrize("then", ["fp64", "bf16xh", "sparse", "batched"])
def test_kept_plans_make_room(ctx, then):
    """Two FP64 shapes, whose plans the context keeps, then a call of a third kind
    under a cap that it fits by itself: the plans go, the call gives what it gives
    in a fresh context, and the first shape builds its plan again."""
    from diana_tucker_b200 import DT_PREC_BF16XH, Context, datasets
    kw = dict(max_sweeps=3, seed=2)
    shapes, ranks = [(60, 52, 44), (52, 60, 44)], (6, 5, 4)
    Xs = [_device(s, k) for k, s in enumerate(shapes)]
    rng = np.random.default_rng(4)

    def third(c):
        if then == "fp64":
            return c.hooi_dense(_device((44, 52, 60), 7), ranks, shape=(44, 52, 60), **kw)[:2]
        if then == "bf16xh":
            return c.hooi_dense(_device((64, 48, 40), 7, "float32"), (8, 8, 8), shape=(64, 48, 40),
                                precision=DT_PREC_BF16XH, inner_iters=2, **kw)[:2]
        if then == "sparse":
            shape, R = (3000, 500, 200), (8, 8, 8)
            idx, vals, _ = datasets.sparse_zipf(shape, 20000, alpha=1.1, seed=12)
            sp = c.sptensor(idx, vals, shape)
            out = sp.hooi(R, 2, datasets.random_orthonormal_transposed(shape, R, 3))[:2]
            sp.close()
            return out
        X = [np.asfortranarray(np.random.default_rng(k).standard_normal((12, 11, 10)), dtype=np.float32)
             for k in range(4)]
        r = np.random.default_rng(6)
        U0 = [[np.linalg.qr(r.standard_normal((s, 3)))[0] for s in x.shape] for x in X]
        return c.hooi_batched(X, [(3, 3, 3)] * 4, U0, sweeps=2, block_threads=128)[:2]

    def flat(out):
        for v in out:
            if isinstance(v, (list, tuple)):
                yield from flat(v)
            else:
                yield np.asarray(v)

    with Context(0) as c:
        want = list(flat(third(c)))
        cap = c.mem_usage()[1]
    with Context(0) as c:
        first = [c.hooi_dense(X, ranks, shape=s, **kw) for X, s in zip(Xs, shapes)]
        assert c.mem_usage()[0] > 0
        c.set_mem_limit(cap)
        for a, b in zip(flat(third(c)), want, strict=True):
            assert np.array_equal(a, b)
        c.set_mem_limit(0)
        G, U, _ = c.hooi_dense(Xs[0], ranks, shape=shapes[0], **kw)
        assert np.array_equal(G, first[0][0])
        assert all(np.array_equal(a, b) for a, b in zip(U, first[0][1]))


@pytest.mark.parametrize("shape,ranks,dtype,cap", [
    ((60, 50, 40), (6, 5, 4), "float64", 505956), ((60, 50, 40), (6, 5, 4), "float32", 1465956),
    ((300, 280, 20), (6, 5, 4), "float64", 9430996), ((300, 280, 20), (6, 5, 4), "float64", 1800000),
    ((40, 36, 32, 28), (5, 5, 5, 5), "float64", 1934868)])
def test_hosvd_start_one_mode_at_a_time(shape, ranks, dtype, cap):
    """A cap that holds the largest mode's Gram, or that and an FP64 copy of X, but
    not all modes' Grams side by side: the HOSVD start takes one mode after
    another.  Other splits and another order of the modes' work: 1e-12 of the
    core's norm, 1e-10 of the subspaces."""
    import torch

    from diana_tucker_b200 import Context, datasets
    from oracle import dense
    X = datasets.tucker_dense(shape, ranks, noise_var=1e-4, seed=5, dtype=np.float64)
    Xd = torch.from_numpy(X.reshape(-1, order="F").copy()).cuda().to(getattr(torch, dtype))
    kw = dict(init="hosvd", max_sweeps=2, shape=shape)
    with Context(0) as c:
        G0, U0, r0 = c.hooi_dense(Xd, ranks, **kw)
        assert c.mem_usage()[1] > cap
        for _ in range(2):
            c.set_mem_limit(cap)
            G, U, r = c.hooi_dense(Xd, ranks, **kw)
            assert abs(r["g_norm"] - r0["g_norm"]) <= 1e-12 * r0["g_norm"]
            for a, b in zip(U, U0):
                assert dense.principal_angle_max(a, b) <= 1e-10


def _small_batch(count):
    from diana_tucker_b200 import datasets
    items = datasets.batched_small(count=count, seed=9)
    rng = np.random.default_rng(1)
    U0 = [[np.linalg.qr(rng.standard_normal((x.shape[n], r[n])))[0] for n in range(3)]
          for x, r in items]
    return [x for x, _ in items], [r for _, r in items], U0


@pytest.mark.parametrize("block", [0, 128, 256, 512])
def test_batch_in_little_room(block):
    """A cap below the scratch of every CTA that fits the GPU: fewer CTAs, the same
    results (block 0 may choose another shape: 1e-10)."""
    from diana_tucker_b200 import Context
    args = _small_batch(100)
    with Context(0) as c:
        want = c.hooi_batched(*args, sweeps=3, block_threads=block)
    with Context(0) as c:
        c.set_mem_limit(60_000_000)
        got = c.hooi_batched(*args, sweeps=3, block_threads=block)
        assert c.mem_usage()[1] <= 60_000_000
        assert got[3]["grid"] < want[3]["grid"] or block == 0
    if block:
        assert np.array_equal(got[2], want[2])
        assert all(np.array_equal(a, b) for a, b in zip(got[1], want[1]))
    np.testing.assert_allclose(got[2], want[2], atol=1e-10)


def test_batch_after_one_that_found_no_room(ctx):
    """A batch whose scratch cannot grow fails; what it gave up on the way is not
    taken for there by the next."""
    import torch

    from diana_tucker_b200 import Context, DTError
    L = _codes()
    tensors, ranks, U0 = _small_batch(24)
    with Context(0) as c:
        pk = c.pack_batched(tensors, ranks, U0)
        Xd, U0d = torch.from_numpy(pk["X"]).cuda(), torch.from_numpy(pk["U"]).cuda()
        Gd = torch.zeros(pk["g_size"], dtype=torch.float64, device="cuda")
        Ed = torch.zeros(pk["count"], dtype=torch.float64, device="cuda")

        def call(block):
            Ud = U0d.clone()
            torch.cuda.synchronize()
            c.hooi_batched_packed(pk, Ud, Gd, Ed, X=Xd, sweeps=2, block_threads=block)
            return Ed.cpu().numpy()

        want = call(512)
        c.set_mem_limit(1)
        for _ in range(2):
            with pytest.raises(DTError) as e:
                call(128)
            assert e.value.code == L.DT_ERR_NOMEM
        c.set_mem_limit(0)
        assert np.array_equal(call(512), want)


@pytest.mark.parametrize("r,n,cap", [(5, 300, 24804), (16, 100_000, 26_210_308), (32, 50_000, 27_222_020)])
def test_row_orthonormalisation_in_little_room(r, n, cap):
    """A cap that holds the matrix and its copy and little else: the Gram's partial
    sums of fewer CTAs, at last of one.  Orthonormal to 1e-13 as without a cap."""
    from diana_tucker_b200 import Context
    W = np.random.default_rng(r).standard_normal((r, n))
    with Context(0) as c:
        c.set_mem_limit(cap)
        out = c.orth2(W)
        np.testing.assert_allclose(out @ out.T, np.eye(r), atol=1e-13)
        Lm = W @ out.T
        assert np.max(np.abs(np.triu(Lm, 1))) < 1e-12 * np.sqrt(n) and np.all(np.diag(Lm) > 0)


@pytest.mark.parametrize("shape,R,nnz,cap", [
    ((20000, 3000, 200), (16, 8, 8), 60000, 13664764), ((3001, 2003, 1009, 501), (5, 7, 6, 3), 30000, 6345860),
    ((3000, 2000), (5, 5), 20000, 1223136), ((20000, 300, 200), (32, 32, 32), 60000, 106931420)])
def test_sparse_hooi_in_little_room(shape, R, nnz, cap):
    """A cap that holds the tensor, the factors, Y_(n) and one product of a factor's
    size: the sweep fits, with the residual and subspaces of the uncapped call
    (other partial sums: 1e-12, 1e-10)."""
    from diana_tucker_b200 import Context, datasets
    from oracle import dense
    idx, vals, shape = datasets.sparse_zipf(shape, nnz, alpha=1.1, seed=3)
    Ut0 = datasets.random_orthonormal_transposed(shape, R, 1)
    with Context(0) as c:
        sp = c.sptensor(idx, vals, shape)
        G0, U0, r0 = sp.hooi(R, 2, Ut0)
        c.set_mem_limit(cap)
        G, U, r = sp.hooi(R, 2, Ut0)
        sp.close()
    assert abs(r["residual"] - r0["residual"]) <= 1e-12
    for a, b in zip(U, U0):
        assert dense.principal_angle_max(a, b) <= 1e-10


@pytest.mark.parametrize("shape,mode,spare", [((200, 40, 21), 0, 1 << 20), ((181, 203, 157), 1, 0),
                                              ((500, 100, 24), 0, 1 << 21), ((40, 50), 0, 0),
                                              ((300, 200, 5), 1, 1 << 22)])
def test_gram_in_any_room(shape, mode, spare):
    """The Gram takes fewer splits, at last one, under a cap that leaves its partial
    tiles little room beside X and the result, or none.  Sums of up to 28417
    products: 1e-12 of the largest entry."""
    from diana_tucker_b200 import Context
    X = np.asfortranarray(np.random.default_rng(sum(shape)).standard_normal(shape))
    A = np.moveaxis(X, mode, 0).reshape(shape[mode], -1)
    with Context(0) as c:
        c.gram(X, mode)
        cap = 8 * (X.size + shape[mode] ** 2) + spare
        assert c.mem_usage()[1] > cap
        c.set_mem_limit(cap)
        G = c.gram(X, mode)
        assert np.array_equal(G, G.T)
        np.testing.assert_allclose(G, A @ A.T, rtol=0, atol=1e-12 * np.max(np.abs(A @ A.T)))


@pytest.mark.parametrize("shape,ranks,cap", [((40, 36, 32, 28), (5, 5, 5, 5), 1934868),
                                             ((8, 8, 8), (2, 2, 2), 3580)])
@pytest.mark.parametrize("stream", ["legacy", "side"])
def test_cap_without_room_for_a_plan(ctx, shape, ranks, cap, stream):
    """A cap that holds a call's own buffers and the largest intermediates that
    live at one time, but no plan beside them (the driver's state, all
    intermediates): the call runs without one, the second time too.  The process's
    rand() is drawn from once."""
    import ctypes

    import torch

    from diana_tucker_b200 import Context
    libc = ctypes.CDLL(None)
    assert _peak(shape, ranks, max_sweeps=3) > cap
    X = _device(shape, 3)
    s = torch.cuda.default_stream() if stream == "legacy" else torch.cuda.Stream()
    torch.cuda.synchronize()
    with Context(0) as c, torch.cuda.stream(s):
        outs = []
        for limit in (0, cap, cap):
            c.set_mem_limit(limit)
            libc.srand(5)
            G, U, rep = c.hooi_dense(X, ranks, shape=shape, seed=0xFFFFFFFF, max_sweeps=3)
            outs.append((G, U, rep["residual"], libc.rand()))
            assert rep["sweeps"] == 3
        for G, U, res, after in outs[1:]:
            assert after == outs[0][3] and abs(res - outs[0][2]) <= 1e-12
            assert np.linalg.norm(G - outs[0][0]) <= 1e-12 * np.linalg.norm(G)
            for a, b in zip(U, outs[0][1]):
                assert np.linalg.norm(a - b) <= 1e-12
