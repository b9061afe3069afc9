"""Dense FP64 path on the GPU vs the oracle (through the C ABI).

Tolerances: operators 1e-12 relative (FP64, different summation order);
HOOI invariants as the spec states them for the FP64 path -- relative
reconstruction error and core norm within 1e-10, largest principal angle
between factor subspaces <= 1e-8."""
import json
import os

import numpy as np
import pytest

from oracle import dense

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")


def _rel(a, b):
    return np.max(np.abs(np.asarray(a) - np.asarray(b))) / max(1e-300, np.max(np.abs(b)))


def test_ttm1_gram1_known_answers(ctx):
    ka = json.load(open(os.path.join(GOLD, "ref_known_answers.json")))
    t = np.reshape(np.array(ka["tensor_colmajor"]), ka["shape"], order="F")
    m1 = np.reshape(np.arange(16.0), (4, 4), order="F")
    m2 = np.reshape(np.arange(6.0), (2, 3), order="F")
    y = ctx.ttm(ctx.ttm(t, m1, 1), m2, 2)
    assert np.array_equal(y.reshape(-1, order="F"), np.array(ka["ttm1"]["expected_colmajor"]))
    g = ctx.gram(t, 1)
    assert np.array_equal(g.reshape(-1, order="F"), np.array(ka["gram1"]["expected_colmajor"]))


def test_ops_vs_reference_fixture(ctx):
    z = np.load(os.path.join(GOLD, "ref_hooi_small.npz"))
    X = z["ttm_X"]
    for n in range(3):
        assert _rel(ctx.ttm(X, z[f"ttm_M{n}"], n), z[f"ttm_Y{n}"]) < 1e-13
        assert _rel(ctx.gram(X, n), z[f"gram_{n}"]) < 1e-13
        assert _rel(ctx.ttt_except(X, z[f"ttt_B{n}"], n), z[f"ttt_{n}"]) < 1e-13


@pytest.mark.parametrize("shape,J", [
    ((200, 200, 10), 10), ((37, 19, 23), 20), ((96, 96, 96), 16), ((1, 5, 7), 3),
    ((5, 1, 7), 2), ((6, 5, 4, 3, 2), 4), ((300,), 7), ((17, 33), 33), ((4, 1000), 1),
    # Runs of 256 rows with 9..16 outputs: the FP64 tensor-core kernel, with
    # and without split contraction, with a ragged J tile.
    ((256, 40, 3), 12), ((512, 300), 16), ((16, 16, 33, 2), 9), ((256, 2, 70), 25)])
def test_ttm_shapes(ctx, shape, J):
    rng = np.random.default_rng(hash((shape, J)) % 2**32)
    X = np.asfortranarray(rng.standard_normal(shape))
    for n in range(len(shape)):
        M = np.asfortranarray(rng.standard_normal((J, shape[n])))
        assert _rel(ctx.ttm(X, M, n), dense.ttm(X, M, n)) < 1e-12


def test_ttm_device_pointers(ctx):
    import torch
    rng = np.random.default_rng(0)
    X = np.asfortranarray(rng.standard_normal((40, 30, 20)))
    M = np.asfortranarray(rng.standard_normal((8, 30)))
    # Column-major device copies: reversed-shape contiguous tensors, transposed.
    Xt = torch.from_numpy(np.ascontiguousarray(X.T)).cuda().permute(2, 1, 0)
    Mt = torch.from_numpy(np.ascontiguousarray(M.T)).cuda().permute(1, 0)
    Y = ctx.ttm(Xt, Mt, 1)
    torch.cuda.synchronize()
    Yh = Y.permute(2, 1, 0).contiguous().cpu().numpy().T
    assert _rel(Yh, dense.ttm(X, M, 1)) < 1e-12


@pytest.mark.parametrize("shape", [(200, 100, 30), (96, 16, 16, 16), (7, 1, 9), (3, 500)])
def test_gram_and_ttt(ctx, shape):
    rng = np.random.default_rng(7)
    X = np.asfortranarray(rng.standard_normal(shape))
    for n in range(len(shape)):
        assert _rel(ctx.gram(X, n), dense.gram(X, n)) < 1e-12
        bshape = tuple(5 if m == n else s for m, s in enumerate(shape))
        B = np.asfortranarray(rng.standard_normal(bshape))
        assert _rel(ctx.ttt_except(X, B, n), dense.ttt_except(X, B, n)) < 1e-12


def test_small_linear_algebra(ctx, oracle_ref):
    rng = np.random.default_rng(3)
    A = rng.standard_normal((50, 7))
    B = rng.standard_normal((7, 9))
    assert _rel(ctx.matmul(A, B), A @ B) < 1e-13
    C = rng.standard_normal((9, 7))
    assert _rel(ctx.matmul(A, C, transB=True), A @ C.T) < 1e-13
    D = rng.standard_normal((50, 4))
    assert _rel(ctx.matmul(A, D, transA=True), A.T @ D) < 1e-13
    Q, R = ctx.reduced_qr(A)
    Qr, Rr = oracle_ref.reduced_qr(A)
    # Same reflector convention as LAPACK: identical Q and R up to rounding.
    assert _rel(Q, Qr) < 1e-12 and _rel(R, Rr) < 1e-12
    S = rng.standard_normal((12, 12)) + 4 * np.eye(12)
    assert _rel(ctx.inverse(S), oracle_ref.inverse(S)) < 1e-11
    W = rng.standard_normal((5, 300))  # R x I, rows orthonormalised
    O = ctx.orth2(W)
    np.testing.assert_allclose(O @ O.T, np.eye(5), atol=1e-13)
    # Same row space, same triangular relation as Gram-Schmidt: W = L O.
    Lm = W @ O.T
    assert np.max(np.abs(np.triu(Lm, 1))) < 1e-12 and np.all(np.diag(Lm) > 0)


@pytest.mark.parametrize("r,n", [(1, 1), (8, 40), (31, 200), (32, 128), (33, 140), (40, 160), (64, 256),
                                 (97, 400), (257, 1100)])
def test_orth2_row_counts(ctx, r, n):
    """Row orthonormalisation on the tensor cores (up to 32 rows) and above: the
    rows of Gram-Schmidt, which are those of the triangular factorisation with a
    positive diagonal.  Gaussian rows four times as long as there are rows have a
    condition below 10: 1e-12."""
    W = np.random.default_rng(r).standard_normal((r, n))
    Q, R = np.linalg.qr(W.T)
    O = ctx.orth2(W)
    np.testing.assert_allclose(O, (Q * np.sign(np.diag(R))).T, rtol=0, atol=1e-12)
    np.testing.assert_allclose(O @ O.T, np.eye(r), atol=1e-13)


def test_orth2_zero_row(ctx):
    from diana_tucker_b200 import DTError
    for r in (20, 50):
        W = np.random.default_rng(r).standard_normal((r, 300))
        W[-1] = 0.0
        with pytest.raises(DTError) as e:
            ctx.orth2(W)
        assert e.value.code == 4


@pytest.mark.parametrize("shape,mode,J", [
    ((5, 7), 0, 1), ((16, 64), 0, 8), ((17, 65), 0, 9), ((33, 129, 3), 0, 24), ((48, 900, 50), 0, 16),
    ((2, 31, 40), 1, 7), ((3, 16, 43), 1, 17), ((63, 15, 9), 1, 16), ((64, 32, 11), 1, 33),
    ((130, 50, 300), 1, 12), ((131, 49, 300), 1, 25), ((256, 20, 700), 1, 16), ((255, 21, 700), 1, 8),
    ((300, 700), 1, 40), ((9, 2000), 1, 5), ((1500, 3), 0, 10)])
def test_ttm_tiles_and_layouts(ctx, shape, mode, J):
    """Rows and contractions at and past the tiles' edges, runs shorter than a
    tile and odd ones, one to several output tiles, 64, 128 and 256 rows a CTA,
    and a split contraction.  Sums of up to 2000 products: 1e-12 of the largest
    entry; FP32 X through one sweep of the FP64 driver."""
    rng = np.random.default_rng(sum(shape) + mode)
    X = np.asfortranarray(rng.standard_normal(shape))
    M = np.asfortranarray(rng.standard_normal((J, shape[mode])))
    want = np.moveaxis(np.tensordot(M, X, axes=([1], [mode])), 0, mode)
    np.testing.assert_allclose(ctx.ttm(X, M, mode), want, rtol=0, atol=1e-12 * np.max(np.abs(want)))
    ranks = [min(3, s) for s in shape]
    if len(shape) > 2:
        X32 = X.astype(np.float32)
        kw = dict(init="randn", max_sweeps=1)
        _, _, a = ctx.hooi_dense(X32, ranks, **kw)
        _, _, b = ctx.hooi_dense(X32.astype(np.float64), ranks, **kw)
        assert abs(a["g_norm"] - b["g_norm"]) <= 1e-12 * b["g_norm"]


@pytest.mark.parametrize("shape,mode", [
    ((7, 5, 3), 0), ((8, 33), 0), ((33, 8), 1), ((12, 64, 9), 1), ((15, 65, 7), 1), ((16, 66, 7), 1),
    ((17, 96, 5), 1), ((97, 31, 3), 0), ((3, 128, 50), 1), ((18, 129, 4), 1), ((200, 40, 21), 0),
    ((20, 200, 17), 1), ((22, 30, 201), 2), ((41, 256, 3), 1), ((256, 9, 9), 0), ((16, 257, 5), 1),
    ((300, 20), 0), ((6, 385, 4), 1), ((500, 1000, 24), 2)])
def test_gram_tiles_and_layouts(ctx, shape, mode):
    """Rows at, below and above the tile lists' sizes (one CTA, two sharing,
    block pairs), both staging layouts, 8- and 16-byte copies, one split and
    many, remainders of the columns.  Sums of up to 5e5 products: 1e-12 of the
    largest entry."""
    rng = np.random.default_rng(sum(shape) + mode)
    X = np.asfortranarray(rng.standard_normal(shape))
    A = np.moveaxis(X, mode, 0).reshape(shape[mode], -1)
    G = ctx.gram(X, mode)
    np.testing.assert_allclose(G, A @ A.T, rtol=0, atol=1e-12 * np.max(np.abs(A @ A.T)))
    assert np.array_equal(G, G.T)


def test_inverse_singular_reports_error(ctx):
    from diana_tucker_b200 import DTError
    with pytest.raises(DTError) as e:
        ctx.inverse(np.zeros((3, 3)))
    assert e.value.code == 4


def test_als_vs_reference(ctx, oracle_ref):
    rng = np.random.default_rng(4)
    Y = np.asfortranarray(rng.standard_normal((30, 6, 5)))
    L0, _ = np.linalg.qr(rng.standard_normal((30, 4)))
    q = ctx.als(Y, 0, L0, 5)
    qr_ = oracle_ref.als(Y, 0, L0, 5)
    assert dense.principal_angle_max(q, qr_) < 1e-10
    np.testing.assert_allclose(q.T @ q, np.eye(4), atol=1e-13)


@pytest.mark.parametrize("n,r", [(96, 16), (97, 13), (150, 16), (200, 10), (256, 8), (64, 32),
                                 (40, 20), (5, 5), (33, 1), (300, 12)])
def test_als_subspace_sizes_vs_oracle(ctx, n, r):
    """dt_als_f64 over the subspace kernel's shapes: S staged whole, packed, or
    read from L2; ranks padded to 8, 16 and 32; n above the tiled kernel's 256."""
    rng = np.random.default_rng(n * 100 + r)
    Y = np.asfortranarray(rng.standard_normal((n, 12, max(4, (2 * n) // 12 + 1))))
    L0, _ = np.linalg.qr(rng.standard_normal((n, r)))
    q = ctx.als(Y, 0, L0, 5)
    want = dense.als(Y, 0, L0, 5)
    assert dense.principal_angle_max(q, want) < 1e-10
    np.testing.assert_allclose(q.T @ q, np.eye(r), atol=1e-13)


@pytest.mark.parametrize("n,r,iters", [(64, 8, 1), (65, 9, 2), (72, 16, 3), (121, 3, 4), (129, 17, 6),
                                       (255, 16, 5), (256, 32, 2), (9, 8, 5)])
def test_als_cluster_edges(ctx, n, r, iters):
    """The subspace kernel on one CTA and on a cluster of eight: CTAs with one
    tile less than others or none, an odd n, S kept or read from L2, and every
    place the last step can have in the schedule.  Singular values fall by
    less than 30 in all, so ten powers of S stay far from breakdown."""
    rng = np.random.default_rng(n + iters)
    V, _ = np.linalg.qr(rng.standard_normal((n, n)))
    W, _ = np.linalg.qr(rng.standard_normal((2 * n, n)))
    Y = np.asfortranarray((V * np.geomspace(30.0, 1.0, n)) @ W.T)
    L0, _ = np.linalg.qr(rng.standard_normal((n, r)))
    q = ctx.als(Y, 0, L0, iters)
    assert dense.principal_angle_max(q, dense.als(Y, 0, L0, iters)) < 1e-10
    np.testing.assert_allclose(q.T @ q, np.eye(r), atol=1e-13)


def _check_hooi(G, U, rep, gn_ref, U_ref, xn):
    assert abs(rep["g_norm"] - gn_ref) <= 1e-10 * gn_ref
    assert abs(np.linalg.norm(G) - gn_ref) <= 1e-10 * gn_ref
    assert abs(rep["x_norm"] - xn) <= 1e-12 * xn
    res_ref = dense.residual(xn, gn_ref)
    assert abs(rep["residual"] - res_ref) <= 1e-10
    for n in range(len(U)):
        assert dense.principal_angle_max(U[n], U_ref[n]) <= 1e-8
        np.testing.assert_allclose(U[n].T @ U[n], np.eye(U[n].shape[1]), atol=1e-12)


def test_hooi_dropin_vs_reference_fixture(ctx):
    """HOOI_ALS semantics (libc-seeded random init, fixed sweeps) against the
    reference's own HOOI_ALS output stored in the golden fixture."""
    z = np.load(os.path.join(GOLD, "ref_hooi_small.npz"))
    X = z["hooi_X"]
    G, U, rep = ctx.hooi_dense(X, (4, 3, 5), init="randn", seed=7, max_sweeps=8)
    gn, xn = z["hooi_norms"]
    _check_hooi(G, U, rep, gn, [z[f"hooi_U{n}"] for n in range(3)], xn)
    assert rep["sweeps"] == 8


def test_hooi_dropin_vs_live_reference(ctx, oracle_ref):
    from diana_tucker_b200 import datasets
    X = datasets.tucker_dense((30, 25, 20, 12), (5, 4, 3, 2), noise_var=1e-3, seed=21)
    Gr, Ur, gn, xn = oracle_ref.hooi_als(X, (5, 4, 3, 2), 6, seed=3)
    G, U, rep = ctx.hooi_dense(X, (5, 4, 3, 2), init="randn", seed=3, max_sweeps=6)
    _check_hooi(G, U, rep, gn, Ur, xn)


def test_hooi_200cube_hosvd_tol_vs_reference_harness(ctx, oracle_ref):
    """The 200^3 FP64 rank-(10,10,10) configuration: HOSVD init, <= 25 sweeps or
    residual change < 1e-8, against the reference-built harness."""
    from diana_tucker_b200 import datasets
    X = datasets.dense_200cube_fp64()
    Gr, Ur, hist = oracle_ref.hooi_harness(X, (10, 10, 10), 25, 1e-8)
    G, U, rep = ctx.hooi_dense(X, (10, 10, 10), init="hosvd", max_sweeps=25, tol=1e-8)
    xn = float(np.linalg.norm(X))
    _check_hooi(G, U, rep, float(np.linalg.norm(Gr)), Ur, xn)
    assert abs(rep["residual"] - hist[-1]) <= 1e-10


@pytest.mark.parametrize("shape,ranks", [((24, 20, 16), (4, 4, 3)),
                                         ((16, 16, 48), (12, 12, 10))])
def test_hooi_fp32_input_equals_upcast(ctx, shape, ranks):
    from diana_tucker_b200 import datasets
    X32 = datasets.tucker_dense(shape, ranks, noise_var=1e-4, seed=9, dtype=np.float32)
    G1, U1, r1 = ctx.hooi_dense(X32, ranks, init="hosvd", max_sweeps=5)
    G2, U2, r2 = ctx.hooi_dense(X32.astype(np.float64), ranks, init="hosvd", max_sweeps=5)
    assert abs(r1["g_norm"] - r2["g_norm"]) <= 1e-12 * r2["g_norm"]
    for n in range(3):
        assert dense.principal_angle_max(U1[n], U2[n]) < 1e-10


def test_hooi_given_init_and_zero_sweeps(ctx):
    from diana_tucker_b200 import datasets
    X = datasets.tucker_dense((15, 14, 13), (3, 3, 3), noise_var=1e-4, seed=2)
    rng = np.random.default_rng(0)
    U0 = [np.linalg.qr(rng.standard_normal((s, 3)))[0] for s in X.shape]
    G, U, rep = ctx.hooi_dense(X, (3, 3, 3), U0=U0, max_sweeps=0)
    Gd = dense.core(X, U0)
    assert _rel(G, Gd) < 1e-12
    G, U, rep = ctx.hooi_dense(X, (3, 3, 3), U0=U0, max_sweeps=4)
    G2, U2, hist = dense.hooi(X, (3, 3, 3), 4, U0)
    assert abs(rep["g_norm"] - np.linalg.norm(G2)) < 1e-10 * np.linalg.norm(G2)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("shape,ranks", [
    ((25, 20, 16), (4, 5, 3)),       # an odd mode before even ones
    ((61, 48, 83), (5, 4, 6)),       # odd, even, odd
    ((17, 33, 20), (3, 4, 3)),       # odd, odd, even
    ((9, 70, 7, 24), (3, 5, 2, 4)),  # even modes after one and after two odd ones, one on a cluster
    ((5, 257, 18), (3, 6, 4)),       # a mode above the batched launch's sizes
    ((15, 14), (4, 4))])
def test_hooi_hosvd_start_of_mixed_parity(ctx, shape, ranks, dtype):
    """The HOSVD start of all modes in one launch, whose Grams lie behind one
    another: even modes after odd ones, modes of one tile beside modes that a
    cluster shares.  Zero sweeps give the start itself, whose subspaces are the
    oracle's leading eigenvectors (well separated by the model: 1e-8)."""
    from diana_tucker_b200 import datasets
    X = datasets.tucker_dense(shape, ranks, noise_var=1e-4, seed=11, dtype=dtype)
    Xd = X.astype(np.float64)
    want = dense.hosvd_init(Xd, ranks)
    G, U, rep = ctx.hooi_dense(X, ranks, init="hosvd", max_sweeps=0)
    for u, w in zip(U, want):
        assert dense.principal_angle_max(u, w) < 1e-8
        np.testing.assert_allclose(u.T @ u, np.eye(u.shape[1]), atol=1e-12)
    assert _rel(G, dense.core(Xd, U)) < 1e-12
    G, U, rep = ctx.hooi_dense(X, ranks, init="hosvd", max_sweeps=3)
    Go, Uo, _ = dense.hooi(Xd, ranks, 3, want)
    _check_hooi(G, U, rep, float(np.linalg.norm(Go)), Uo, float(np.linalg.norm(Xd)))


def test_hooi_rejects_bad_ranks(ctx):
    from diana_tucker_b200 import DTError
    with pytest.raises(DTError) as e:
        ctx.hooi_dense(np.ones((4, 5, 6)), (5, 2, 2))
    assert e.value.code == 1


@pytest.mark.parametrize("rows", [7, 6528, 6529])
def test_hooi_host_outputs_through_the_staging(ctx, rows):
    """Host outputs are stored by one kernel into 1 MiB of pinned staging and
    copied from there (6528 rows: 131060 words of 131072), larger ones by one
    copy each: both are what device outputs hold."""
    import torch
    shape, ranks = (rows, 12, 10), (min(rows, 20), 5, 4)
    X = np.random.default_rng(rows).standard_normal(shape)
    Xd = torch.from_numpy(X.reshape(-1, order="F").copy()).cuda()
    kw = dict(init="randn", seed=4, max_sweeps=1, shape=shape)
    Gd, Ud, repd = ctx.hooi_dense(Xd, ranks, device_out=True, **kw)
    G, U, rep = ctx.hooi_dense(Xd, ranks, **kw)
    assert rep["residual"] == repd["residual"]
    assert np.array_equal(G, Gd.cpu().numpy())
    for a, b in zip(U, Ud):
        assert np.array_equal(a, b.cpu().numpy())
