"""Sparse TTMc and sparse HOOI on the GPU vs the C restatement (oracle).

Tolerance: 1e-12 relative (FP64; only the summation order differs)."""
import numpy as np
import pytest

from oracle import dense

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.max(np.abs(np.asarray(a) - np.asarray(b))) / max(1e-300, np.max(np.abs(b)))


@pytest.fixture(scope="module")
def zipf_small():
    from diana_tucker_b200 import datasets
    # Zipf heads give rows far longer than one 512-nonzero chunk.
    return datasets.sparse_zipf((3000, 500, 200), 40000, alpha=1.1, seed=12)


def _factors(shape, R, seed):
    from diana_tucker_b200 import datasets
    return datasets.random_orthonormal_transposed(shape, R, seed)


@pytest.mark.parametrize("R", [(16, 16, 16), (8, 4, 2), (5, 3, 7), (8, 16, 16), (16, 8, 8),
                               (32, 32, 32), (10, 10, 10), (12, 12, 12), (4, 4, 4)])
def test_ttmc_rows_mtr_mtl(ctx, oracle_sparse, zipf_small, R):
    idx, vals, shape = zipf_small
    sp = ctx.sptensor(idx, vals, shape)
    Ut = _factors(shape, R, 1)
    assert abs(sp.fnorm() - np.linalg.norm(vals)) < 1e-12 * np.linalg.norm(vals)
    for mode in range(3):
        Y = sp.ttmc_rows(Ut, R, mode)
        Yo = oracle_sparse.ttmc_rows(idx, vals, shape, Ut, R, mode)
        assert _rel(Y, Yo) < 1e-12
        L = sp.ttmc_mTR(Ut, R, mode)
        Lo = oracle_sparse.ttmc_mTR(idx, vals, shape, Ut, R, mode)
        assert _rel(L, Lo) < 1e-12
        out = sp.ttmc_mTL(Ut, R, mode, Lo)
        outo = oracle_sparse.ttmc_mTL(idx, vals, shape, Ut, R, mode, Lo)
        assert _rel(out, outo) < 1e-12
    sp.close()


@pytest.mark.parametrize("R", [(4, 40, 24), (33, 2, 30)])
def test_ttmc_wide_ranks(ctx, oracle_sparse, zipf_small, R):
    """Other-mode ranks above 32 (P <= 1024) take the wide fibre kernel."""
    idx, vals, shape = zipf_small
    sp = ctx.sptensor(idx, vals, shape)
    Ut = _factors(shape, R, 7)
    for mode in range(3):
        P = int(np.prod([R[m] for m in range(3) if m != mode]))
        if P > 1024:
            continue
        Y = sp.ttmc_rows(Ut, R, mode)
        assert _rel(Y, oracle_sparse.ttmc_rows(idx, vals, shape, Ut, R, mode)) < 1e-12
    sp.close()


def test_sparse_four_way_generic_path(ctx, oracle_sparse):
    from diana_tucker_b200 import datasets
    idx, vals, shape = datasets.sparse_zipf((60, 40, 30, 20), 5000, alpha=1.1, seed=4)
    R = (3, 2, 4, 2)
    Ut = _factors(shape, R, 2)
    sp = ctx.sptensor(idx, vals, shape)
    for mode in range(4):
        assert _rel(sp.ttmc_rows(Ut, R, mode),
                    oracle_sparse.ttmc_rows(idx, vals, shape, Ut, R, mode)) < 1e-12
        assert _rel(sp.ttmc_mTR(Ut, R, mode),
                    oracle_sparse.ttmc_mTR(idx, vals, shape, Ut, R, mode)) < 1e-12


@pytest.mark.parametrize("shape,R", [
    ((700, 90), (8, 31)), ((700, 90), (3, 1)), ((60, 40, 30, 20), (9, 8, 7, 5)),
    ((60, 40, 30, 20), (1, 16, 4, 16)), ((60, 40, 30, 25), (2, 6, 7, 24)),
    ((2000, 5, 6, 7), (10, 5, 6, 7)), ((30, 20, 12, 9, 7), (3, 5, 2, 4, 7)),
    ((9, 8, 7, 6, 5, 4), (2, 3, 4, 2, 3, 4)), ((6, 5, 4, 4, 3, 3, 3, 2), (2, 2, 3, 2, 2, 3, 2, 2))])
def test_row_kernel_orders_and_tile_edges(ctx, oracle_sparse, shape, R):
    """The row kernel over two to eight modes: rows of one nonzero and rows of
    several chunks, sides of the Kronecker cut at, below and above a tile.
    Sums of up to a few thousand products with factors below 1: 1e-12."""
    from diana_tucker_b200 import datasets
    idx, vals, shape = datasets.sparse_zipf(shape, 6000, alpha=1.1, seed=len(shape))
    Ut = _factors(shape, R, 21)
    sp = ctx.sptensor(idx, vals, shape)
    for mode in range(len(shape)):
        assert _rel(sp.ttmc_rows(Ut, R, mode),
                    oracle_sparse.ttmc_rows(idx, vals, shape, Ut, R, mode)) < 1e-12
    Ut0 = _factors(shape, R, 22)
    if all(R[m] <= np.prod([r for k, r in enumerate(R) if k != m]) for m in range(len(R))):
        G, U, rep = sp.hooi(R, 2, Ut0)
        Go, Uo, res = oracle_sparse.hooi(idx, vals, shape, R, 2, Ut0)
        assert abs(rep["residual"] - res) < 1e-10
        for n in range(len(shape)):
            np.testing.assert_allclose(U[n].T @ U[n], np.eye(R[n]), atol=1e-12)
    sp.close()


@pytest.mark.parametrize("R", [(16, 9, 16), (31, 17, 1), (25, 32, 32), (24, 15, 10), (7, 8, 23)])
def test_fibre_kernel_tiles(ctx, oracle_sparse, R):
    """The fibre kernel over ranks at and around its column tiles (even and odd
    tile counts lay the columns out differently), with fibres of one nonzero and
    fibres of several pieces.  Sums of up to a thousand products: 1e-12."""
    shape = (40, 36, 34)
    rng = np.random.default_rng(31)
    keep = np.concatenate([rng.choice(36 * 34 * 20, 9000, replace=False),
                           36 * 34 * 20 + rng.choice(36 * 34 * 20, 700, replace=False)])
    idx = [i.astype(np.int64) for i in np.unravel_index(keep, shape)]
    vals = rng.standard_normal(keep.size)
    Ut = _factors(shape, R, 32)
    sp = ctx.sptensor(idx, vals, shape)
    for mode in range(3):
        assert _rel(sp.ttmc_rows(Ut, R, mode),
                    oracle_sparse.ttmc_rows(idx, vals, shape, Ut, R, mode)) < 1e-12
    sp.close()


def test_sparse_hooi_vs_oracle(ctx, oracle_sparse, zipf_small):
    idx, vals, shape = zipf_small
    R = (8, 8, 8)
    Ut0 = _factors(shape, R, 3)
    sp = ctx.sptensor(idx, vals, shape)
    G, Ut, rep = sp.hooi(R, 3, Ut0)
    Go, Uto, res = oracle_sparse.hooi(idx, vals, shape, R, 3, Ut0)
    assert abs(rep["residual"] - res) < 1e-10
    assert abs(np.linalg.norm(G) - np.linalg.norm(Go)) < 1e-10 * np.linalg.norm(Go)
    for n in range(3):
        assert dense.principal_angle_max(Ut[n], Uto[n]) < 1e-8
        np.testing.assert_allclose(Ut[n].T @ Ut[n], np.eye(R[n]), atol=1e-12)


def test_single_nonzero_and_empty_rows(ctx, oracle_sparse):
    idx = [np.array([3], dtype=np.int64), np.array([0], dtype=np.int64),
           np.array([4], dtype=np.int64)]
    vals = np.array([2.5])
    shape = [5, 4, 6]
    R = (2, 2, 2)
    Ut = _factors(shape, R, 4)
    sp = ctx.sptensor(idx, vals, shape)
    for mode in range(3):
        Y = sp.ttmc_rows(Ut, R, mode)
        assert _rel(Y, oracle_sparse.ttmc_rows(idx, vals, shape, Ut, R, mode)) < 1e-14
        assert np.count_nonzero(np.abs(Y).sum(axis=1)) == 1


def test_out_of_range_index_is_rejected(ctx):
    from diana_tucker_b200 import DTError
    idx = [np.array([0, 5], dtype=np.int64), np.array([0, 1], dtype=np.int64)]
    with pytest.raises(DTError) as e:
        ctx.sptensor(idx, np.array([1.0, 2.0]), [5, 4])
    assert e.value.code == 1


def test_sptensor_outlives_its_context(oracle_sparse):
    """Destroying a context first detaches its sparse tensors: later calls fail
    with an error and closing the tensor is safe."""
    from diana_tucker_b200 import Context, DTError, datasets
    idx, vals, shape = datasets.sparse_zipf((50, 40, 30), 500, alpha=1.1, seed=5)
    c2 = Context(0)
    sp = c2.sptensor(idx, vals, shape)
    c2.close()
    with pytest.raises(DTError) as e:
        sp.ttmc_rows(_factors(shape, (2, 2, 2), 6), (2, 2, 2), 0)
    assert e.value.code == 1
    sp.close()


@pytest.mark.parametrize("rows", [100, 20_000, 300_011])
def test_hooi_factor_transfers(ctx, rows):
    """Factors below the staging threshold, within the staging buffer and
    larger than it: the start stays as it was, and the in-place entry point
    (device buffers, no staging) gives the same bits."""
    import ctypes

    import torch

    from diana_tucker_b200 import _lib, datasets
    R = (16, 8, 8)
    idx, vals, shape = datasets.sparse_zipf((rows, 300, 200), 20_000, alpha=1.1, seed=3)
    Ut0 = _factors(shape, R, 9)
    kept = [u.copy() for u in Ut0]
    sp = ctx.sptensor(idx, vals, shape)
    G, Ut, rep = sp.hooi(R, 2, Ut0)
    assert all(np.array_equal(a, b) for a, b in zip(Ut0, kept))
    dev = [torch.from_numpy(u).cuda() for u in Ut0]
    torch.cuda.synchronize()
    ptrs = (ctypes.c_void_p * 3)(*[d.data_ptr() for d in dev])
    r = (ctypes.c_int64 * 3)(*R)
    Gd = np.zeros_like(G)
    _lib.check(ctx.lib.dt_sp_hooi(ctx.h, sp.h, r, 2, ptrs, Gd.ctypes.data,
                                  ctypes.byref(_lib.HooiReport())))
    assert np.array_equal(G, Gd)
    for a, b in zip(Ut, dev):
        assert np.array_equal(a, b.cpu().numpy())
    sp.close()


@pytest.mark.parametrize("rows", [20_000, 300_011])
def test_hooi_factor_transfers_on_the_per_thread_stream(rows):
    """The handle of the per-thread default stream names another stream in each of
    the threads that copy the factors: the transfers have to be in order with the
    calling thread's all the same.  Other starts in turn, so what a call before
    left in the buffers does not pass for this one's; the in-place entry point
    (device buffers, no staging) on the context's own stream gives the same bits."""
    import ctypes

    import torch

    from diana_tucker_b200 import Context, _lib, datasets
    per_thread = ctypes.c_void_p(2)  # cudaStreamPerThread
    R = (16, 8, 8)
    idx, vals, shape = datasets.sparse_zipf((rows, 300, 200), 20_000, alpha=1.1, seed=3)
    r = (ctypes.c_int64 * 3)(*R)
    with Context(0) as c:
        sp = c.sptensor(idx, vals, shape)
        for seed in range(9, 15):
            Ut0 = _factors(shape, R, seed)
            _lib.check(c.lib.dt_ctx_set_stream(c.h, per_thread))
            G, Ut, _ = sp.hooi(R, 1, Ut0)
            _lib.check(c.lib.dt_ctx_set_stream(c.h, None))
            dev = [torch.from_numpy(u).cuda() for u in Ut0]
            torch.cuda.synchronize()
            ptrs = (ctypes.c_void_p * 3)(*[d.data_ptr() for d in dev])
            Gd = np.zeros_like(G)
            _lib.check(c.lib.dt_sp_hooi(c.h, sp.h, r, 1, ptrs, Gd.ctypes.data,
                                        ctypes.byref(_lib.HooiReport())))
            assert np.array_equal(G, Gd)
            for a, b in zip(Ut, dev):
                assert np.array_equal(a, b.cpu().numpy())
        sp.close()
