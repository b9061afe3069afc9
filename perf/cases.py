"""Measured workloads: what programs have this library do, through its public
Python entry points.

A program keeps one Context per process, makes tensors on the GPU (dense and
batched ones) or reads nonzeros on the host (sparse ones), and decomposes one
tensor after another.  The families:

fp64     Context.hooi_dense in plain FP64: from a tensor of some ten thousand
         entries, where launches and latency count, to 96^4.  X in float64, or
         in float32 as measured data often is; random start (the default) or
         HOSVD start; a fixed number of sweeps (the default) or a stop on the
         residual's change.
mixed    Context.hooi_dense with BF16 tensor-core sweeps of a float32 tensor.
batched  Context.hooi_batched_packed: many small tensors of uneven sizes.
sparse   SpTensor.hooi: power sweeps from random orthonormal factors, three
         modes and four.
ops      The operators a program that writes its own algorithm calls: one
         contraction (Context.ttm) and one Gram (Context.gram) of an FP64
         tensor.
warm     Context.ws_init with a decoder that was trained before, then the
         plain HOOI that finishes from it.

"stream" says whether the program calls from torch's default stream or from a
side stream of its own.
"""
import ctypes
import math

import numpy as np
import torch

import diana_tucker_b200 as dtb

_PREC = {"fp64": dtb.DT_PREC_FP64, "xh": dtb.DT_PREC_BF16XH, "x2": dtb.DT_PREC_BF16X2}
_kept = {}


def _context():
    if "ctx" not in _kept:
        _kept["ctx"] = dtb.Context(torch.cuda.current_device())
    return _kept["ctx"]


def _stream(case):
    if case.get("stream") != "side":
        return torch.cuda.default_stream()
    if "side" not in _kept:
        _kept["side"] = torch.cuda.Stream()
    return _kept["side"]


def _ints(text):
    return [int(v) for v in text.split("x")]


def _text(values):
    return "x".join(str(int(v)) for v in values)


def listed():
    return [
        # The smallest tensors: each of the launches of a decomposition is short.
        dict(name="fp64_small", kind="fp64", shape="40x32x24", ranks="5x4x3", dtype="f64",
             init="randn", sweeps=5, tol=0.0, noise=1e-4, decay=1.0, stream="default"),
        # The 200^3 rank-10 configuration: HOSVD start, stop on the residual's change.
        dict(name="fp64_200_hosvd", kind="fp64", shape="200x200x200", ranks="10x10x10",
             dtype="f64", init="hosvd", sweeps=25, tol=1e-8, noise=1e-4, decay=1.0,
             stream="side"),
        # Odd sizes, measured data in float32: no mode is a multiple of a tile.
        dict(name="fp64_ragged_4way", kind="fp64", shape="61x47x83x35", ranks="7x9x11x5",
             dtype="f32", init="randn", sweeps=4, tol=0.0, noise=1e-4, decay=1.0,
             stream="default"),
        # The largest dense tensor, plain FP64.
        dict(name="fp64_96x4", kind="fp64", shape="96x96x96x96", ranks="16x16x16x16",
             dtype="f64", init="randn", sweeps=30, tol=1e-9, noise=1e-6, decay=0.9,
             stream="side"),
        # The same tensor in float32, tensor-core sweeps: the headline configuration.
        dict(name="mixed_96x4", kind="mixed", shape="96x96x96x96", ranks="16x16x16x16",
             prec="xh", sweeps=30, tol=1e-9, noise=1e-6, decay=0.9, stream="side"),
        # Tensor-core sweeps of an ordinary size, called from the default stream.
        dict(name="mixed_3way", kind="mixed", shape="128x112x96", ranks="16x8x16", prec="x2",
             sweeps=5, tol=0.0, noise=1e-6, decay=0.9, stream="default"),
        # The batch configuration: 4096 tensors.
        dict(name="batched_4096", kind="batched", count=4096, lo=8, hi=64, rlo=2, rhi=8,
             sweeps=10, stream="side"),
        # A batch that does not fill the GPU.
        dict(name="batched_100", kind="batched", count=100, lo=8, hi=64, rlo=2, rhi=8,
             sweeps=10, stream="default"),
        # The sparse configuration's index law at an eighth of its sizes and draws.
        dict(name="sparse_zipf", kind="sparse", shape="250000x25000x6250", ranks="16x16x16",
             draws=6250000, sweeps=10),
        # Four modes, odd ranks.
        dict(name="sparse_4way", kind="sparse", shape="3001x2003x1009x501", ranks="5x7x6x3",
             draws=300000, sweeps=5),
        # One contraction and one Gram over the middle mode of an odd-sized tensor.
        dict(name="ops_ragged", kind="ops", shape="181x203x157", mode=1, rows=24,
             stream="default"),
        # The learned warm start of the 256^3 family.
        dict(name="warm_256", kind="warm", size=256, rank=12, latent=24, sketch_sweeps=2,
             sweeps=3, stream="side"),
    ]


def _capped(ranks):
    """A Tucker model needs R_n <= the product of the other ranks."""
    ranks = list(ranks)
    for n in range(len(ranks)):
        ranks[n] = min(ranks[n], math.prod(r for m, r in enumerate(ranks) if m != n))
    return ranks


def _log_between(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["fp64", "fp64", "mixed", "batched", "sparse", "ops", "warm"])
    stream = rng.choice(["default", "side"])
    if kind == "fp64":
        nd = rng.choice([3, 3, 4])
        side = _log_between(rng, 2e4, 2e7) ** (1.0 / nd)
        shape = [max(6, int(side * rng.uniform(0.7, 1.4))) for _ in range(nd)]
        ranks = _capped(rng.randint(3, min(16, s // 2)) for s in shape)
        init = rng.choice(["randn", "randn", "hosvd"])
        return dict(kind="fp64", shape=_text(shape), ranks=_text(ranks),
                    dtype=rng.choice(["f64", "f32"]), init=init, sweeps=rng.randint(2, 5),
                    tol=0.0, noise=1e-4, decay=1.0, stream=stream)
    if kind == "mixed":
        nd = rng.choice([3, 4])
        # Modes the tensor cores take: multiples of 8 up to 128, the first from 64.
        shape = [8 * rng.randint(8, 16)]
        side = (_log_between(rng, 1e6, 6e7) / shape[0]) ** (1.0 / (nd - 1))
        shape += [8 * min(16, max(2, int(side * rng.uniform(0.8, 1.25) / 8))) for _ in range(nd - 1)]
        ranks = [rng.choice([8, 16]) for _ in shape]
        return dict(kind="mixed", shape=_text(shape), ranks=_text(ranks),
                    prec=rng.choice(["xh", "x2"]), sweeps=rng.randint(2, 5), tol=0.0, noise=1e-6,
                    decay=0.9, stream=stream)
    if kind == "batched":
        lo = rng.randint(5, 16)
        return dict(kind="batched", count=int(_log_between(rng, 20, 4000)), lo=lo,
                    hi=rng.randint(lo + 8, 64), rlo=2, rhi=rng.randint(3, 8),
                    sweeps=rng.randint(3, 10), stream=stream)
    if kind == "sparse":
        nd = rng.choice([3, 3, 4])
        draws = int(_log_between(rng, 5e4, 6e6 if nd == 3 else 5e5))
        shape = [int(_log_between(rng, 300, max(1000, draws / 25))) for _ in range(nd)]
        ranks = [rng.choice([4, 5, 8, 10, 16]) if nd == 3 else rng.randint(3, 8) for _ in shape]
        return dict(kind="sparse", shape=_text(shape), ranks=_text(ranks), draws=draws,
                    sweeps=rng.randint(2, 8))
    if kind == "ops":
        side = _log_between(rng, 3e4, 1.2e7) ** (1.0 / 3)
        shape = [max(8, int(side * rng.uniform(0.6, 1.6))) for _ in range(3)]
        mode = rng.randrange(3)
        return dict(kind="ops", shape=_text(shape), mode=mode,
                    rows=rng.randint(4, min(32, shape[mode])), stream=stream)
    rank = rng.randint(6, 12)
    return dict(kind="warm", size=rng.randint(64, 256), rank=rank, latent=2 * rank,
                sketch_sweeps=rng.randint(0, 2), sweeps=rng.randint(2, 4), stream=stream)


# -- inputs -------------------------------------------------------------------
def _generator(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _f64(shape, g):
    return torch.randn(*shape, generator=g, dtype=torch.float64, device="cuda")


def _factors(shape, ranks, g):
    return [torch.linalg.qr(_f64((s, r), g))[0] for s, r in zip(shape, ranks)]


def _multiply(Xt, M, n):
    """Xt holds X with its modes reversed (C order = X column-major): X x_n M."""
    axis = Xt.dim() - 1 - n
    return torch.movedim(torch.tensordot(Xt, M, dims=([axis], [1])), -1, axis)


def _tucker(case, seed, dtype):
    """A Tucker product of an N(0, 1) core (scaled by decay ** (i + j + ...)) and
    orthonormal factors, plus noise; reversed modes, C-contiguous."""
    shape, ranks = _ints(case["shape"]), _ints(case["ranks"])
    g = _generator(seed)
    Xt = _f64(ranks[::-1], g)
    for axis, r in enumerate(ranks[::-1]):
        scale = case["decay"] ** torch.arange(r, dtype=torch.float64, device="cuda")
        Xt = Xt * scale.reshape([-1 if a == axis else 1 for a in range(len(ranks))])
    for n, U in enumerate(_factors(shape, ranks, g)):
        Xt = _multiply(Xt, U, n)
    Xt = Xt.contiguous()
    Xt += math.sqrt(case["noise"]) * _f64(shape[::-1], g)
    return Xt.to(dtype).contiguous()


def _reversed(Xt):
    return Xt.permute(*reversed(range(Xt.dim())))


def _coo(case, seed):
    """COO tensor: per mode a bounded Zipf(1.1) rank through a random
    permutation, duplicates merged by summing, lognormal values."""
    shape, draws = _ints(case["shape"]), case["draws"]
    g = _generator(seed)
    key = torch.zeros(draws, dtype=torch.int64, device="cuda")
    mult = 1
    for size in shape:
        w = torch.arange(1, size + 1, dtype=torch.float64, device="cuda") ** -1.1
        cdf = torch.cumsum(w, 0)
        u = torch.rand(draws, generator=g, dtype=torch.float64, device="cuda") * cdf[-1]
        rank = torch.searchsorted(cdf, u, right=True).clamp_(max=size - 1)
        key += torch.randperm(size, generator=g, device="cuda")[rank] * mult
        mult *= size
    vals = torch.exp(torch.randn(draws, generator=g, dtype=torch.float64, device="cuda"))
    key, order = torch.sort(key, stable=True)
    vals = vals[order]
    first = torch.ones_like(key, dtype=torch.bool)
    first[1:] = key[1:] != key[:-1]
    start = torch.nonzero(first).flatten()
    # Segment sums by differences would lose digits: sum each run in order.
    length = torch.diff(start, append=torch.tensor([draws], device="cuda"))
    merged = torch.segment_reduce(vals, "sum", lengths=length)
    key = key[start]
    idx = []
    for size in shape:
        idx.append(key % size)
        key = key // size
    return idx, merged, shape


def _sparse_start(case, seed):
    shape, ranks = _ints(case["shape"]), _ints(case["ranks"])
    g = _generator(seed + 77)
    return [U.contiguous() for U in _factors(shape, ranks, g)]


def _batch(case, seed):
    """One packed float32 buffer on the GPU, each tensor column-major, and
    packed orthonormal start factors.  The sizes and ranks belong to the case,
    the tensors to the seed."""
    count, lo, hi = case["count"], case["lo"], case["hi"]
    rng = np.random.default_rng([count, lo, hi, case["rlo"], case["rhi"]])
    shapes = rng.integers(lo, hi + 1, size=(count, 3))
    ranks = np.minimum(rng.integers(case["rlo"], case["rhi"] + 1, size=(count, 3)), shapes)
    for n in range(3):
        others = ranks[:, (n + 1) % 3] * ranks[:, (n + 2) % 3]
        ranks[:, n] = np.minimum(ranks[:, n], others)
    sizes = shapes.prod(axis=1)
    usz = (shapes * ranks).reshape(-1)
    gsz = ranks.prod(axis=1)
    first = lambda s: np.concatenate([[0], np.cumsum(s)[:-1]]).astype(np.int64)  # noqa: E731
    xoff, uoff, goff = first(sizes), first(usz), first(gsz)
    g = _generator(seed)

    # All factors at once, modes padded to the largest size and ranks to 8 by
    # zeros; orthonormal by the Cholesky factor of their Grams.
    rows = torch.as_tensor(shapes.reshape(-1), device="cuda")[:, None]
    cols = torch.as_tensor(ranks.reshape(-1), device="cuda")[:, None]

    def factors():
        some = torch.arange(8, device="cuda")[None, :] < cols
        A = _f64([3 * count, hi, 8], g) * some[:, None, :]
        A = A * (torch.arange(hi, device="cuda")[None, :] < rows)[:, :, None]
        L = torch.linalg.cholesky(A.mT @ A + torch.diag_embed((~some).double()))
        return torch.linalg.solve_triangular(L, A.mT, upper=False).mT

    Q, U0 = factors().reshape(count, 3, hi, 8), factors().reshape(count, 3, hi, 8)
    core = _f64((count, 8, 8, 8), g)
    keep = [torch.arange(8, device="cuda")[None, :] < torch.as_tensor(ranks[:, n], device="cuda")[:, None]
            for n in range(3)]
    core = core * (keep[0][:, :, None, None] & keep[1][:, None, :, None] & keep[2][:, None, None, :])
    X = torch.empty(int(sizes.sum()), dtype=torch.float32, device="cuda")
    noise = 1e-2 * _f64((int(sizes.sum()),), g)
    dims = [torch.as_tensor(shapes[:, n], device="cuda") for n in range(3)]
    at = torch.as_tensor(xoff, device="cuda")
    place = torch.arange(hi, device="cuda")
    for b in range(0, count, 128):
        e = min(count, b + 128)
        T = torch.einsum("tabc,tia->tibc", core[b:e], Q[b:e, 0])
        T = torch.einsum("tibc,tjb->tijc", T, Q[b:e, 1])
        T = torch.einsum("tijc,tkc->tkji", T, Q[b:e, 2])
        i0, i1, i2 = (d[b:e, None, None, None] for d in dims)
        k, j, i = place[None, :, None, None], place[None, None, :, None], place[None, None, None, :]
        inside = (k < i2) & (j < i1) & (i < i0)
        to = (at[b:e, None, None, None] + i + i0 * (j + i1 * k))[inside]
        X[to] = (T[inside] + noise[to]).to(torch.float32)
    U = torch.empty(int(usz.sum()), dtype=torch.float64, device="cuda")
    uat = torch.as_tensor(uoff, device="cuda")
    for b in range(0, 3 * count, 3072):
        e = min(3 * count, b + 3072)
        i, c = place[None, :, None], torch.arange(8, device="cuda")[None, None, :]
        inside = (i < rows[b:e, :, None]) & (c < cols[b:e, :, None])
        to = (uat[b:e, None, None] + i + rows[b:e, :, None] * c)[inside]
        U[to] = U0.reshape(3 * count, hi, 8)[b:e][inside]
    packed = {"count": count, "shapes": shapes.astype(np.int64).reshape(-1),
              "ranks": ranks.astype(np.int64).reshape(-1), "xoff": xoff, "uoff": uoff, "goff": goff,
              "X": X}
    return packed, U, int(gsz.sum())


def _decoder(case):
    """An orthonormal basis of the first Chebyshev polynomials: what training
    on this family arrives at."""
    x = np.linspace(-1.0, 1.0, case["size"])
    return np.asfortranarray(np.linalg.qr(np.polynomial.chebyshev.chebvander(x, case["latent"] - 1))[0])


def _family_member(case, seed):
    n, rank, latent = case["size"], case["rank"], case["latent"]
    g = _generator(seed)
    T = torch.as_tensor(np.polynomial.chebyshev.chebvander(np.linspace(-1.0, 1.0, n), latent - 1)).cuda()
    Xt = _f64((rank,) * 3, g)
    fade = torch.exp(-0.15 * torch.arange(rank, dtype=torch.float64, device="cuda"))
    Xt = Xt * fade[:, None, None] * fade[None, :, None] * fade[None, None, :]
    for m in range(3):
        Xt = _multiply(Xt, torch.linalg.qr(T @ _f64((latent, rank), g))[0], m)
    Xt = Xt.contiguous() + math.sqrt(1e-5) * _f64((n, n, n), g)
    return Xt.to(torch.float32).contiguous()


def prepare(case, seed):
    kind, ctx = case["kind"], _context()
    s = {"case": case, "ctx": ctx, "stream": _stream(case)}
    if kind in ("fp64", "mixed"):
        dtype = torch.float64 if case.get("dtype") == "f64" else torch.float32
        s["X"] = _reversed(_tucker(case, seed, dtype))
        s["ranks"] = _ints(case["ranks"])
    elif kind == "batched":
        s["packed"], s["U0"], gsize = _batch(case, seed)
        s["U"] = torch.empty_like(s["U0"])
        s["G"] = torch.empty(gsize, dtype=torch.float64, device="cuda")
        s["relerr"] = torch.empty(case["count"], dtype=torch.float64, device="cuda")
    elif kind == "sparse":
        idx, vals, shape = _coo(case, seed)
        s["sp"] = ctx.sptensor([i.cpu().numpy() for i in idx], vals.cpu().numpy(), shape)
        s["Ut"] = [U.cpu().numpy() for U in _sparse_start(case, seed)]
        s["ranks"] = _ints(case["ranks"])
    elif kind == "ops":
        shape, g = _ints(case["shape"]), _generator(seed)
        s["X"] = _reversed(_f64(shape[::-1], g))
        s["M"] = _reversed(_f64((shape[case["mode"]], case["rows"]), g))
    else:
        s["X"] = _reversed(_family_member(case, seed))
        s["D"] = _decoder(case)
    return s


# -- one pass -------------------------------------------------------------------
def run(s):
    case, ctx = s["case"], s["ctx"]
    if case["kind"] == "sparse":
        G, Ut, rep = s["sp"].hooi(s["ranks"], case["sweeps"], s["Ut"])
        return {"G": G, "U": Ut, "residual": rep["residual"]}
    with torch.cuda.stream(s["stream"]):
        if case["kind"] in ("fp64", "mixed"):
            more = dict(init=case["init"]) if case["kind"] == "fp64" else dict(
                inner_iters=2, precision=_PREC[case["prec"]])
            G, U, rep = ctx.hooi_dense(s["X"], s["ranks"], max_sweeps=case["sweeps"],
                                       tol=case["tol"], device_out=True, **more)
            return {"G": G, "U": U, "residual": rep["residual"], "sweeps": rep["sweeps"]}
        if case["kind"] == "batched":
            s["U"].copy_(s["U0"])
            ctx.hooi_batched_packed(s["packed"], s["U"], s["G"], s["relerr"],
                                    sweeps=case["sweeps"])
            return {"G": s["G"], "U": s["U"], "relerr": s["relerr"]}
        if case["kind"] == "ops":
            return {"Y": ctx.ttm(s["X"], s["M"], case["mode"]),
                    "S": ctx.gram(s["X"], case["mode"])}
        ranks = [case["rank"]] * 3
        U0, fit_sketch, fit_init = ctx.ws_init(s["X"], ranks, s["D"],
                                               sketch_sweeps=case["sketch_sweeps"])
        G, U, rep = ctx.hooi_dense(s["X"], ranks, U0=U0, max_sweeps=case["sweeps"],
                                   device_out=True)
        return {"G": G, "U": U, "U0": U0, "fit_init": fit_init, "residual": rep["residual"]}


# -- what a pass cannot do without ----------------------------------------------
def _dense_work(shape, ranks, sweeps, item):
    """X once and the results once; per sweep the two contractions of X that a
    dimension tree needs and, for each mode, the Gram of its unfolding."""
    size, core = math.prod(shape), math.prod(ranks)
    flops = 0.0
    for s, r in zip(shape, ranks):
        flops += float(s) * s * core / r
    flops += 2.0 * size * (ranks[0] + ranks[-1])
    return {"bytes": size * item + 8.0 * (core + sum(s * r for s, r in zip(shape, ranks))),
            "flops": sweeps * flops}


def work(case):
    kind = case["kind"]
    if kind in ("fp64", "mixed"):
        sweeps = case["sweeps"] if case["tol"] == 0.0 else 3
        return _dense_work(_ints(case["shape"]), _ints(case["ranks"]), sweeps,
                           8 if case.get("dtype") == "f64" else 4)
    if kind == "batched":
        side, r = 0.5 * (case["lo"] + case["hi"]), 0.5 * (case["rlo"] + case["rhi"])
        one = _dense_work([side] * 3, [r] * 3, case["sweeps"], 4)
        return {k: case["count"] * v for k, v in one.items()}
    if kind == "sparse":
        shape, ranks, nnz = _ints(case["shape"]), _ints(case["ranks"]), case["draws"]
        P = math.prod(ranks)
        rows = sum(s * r for s, r in zip(shape, ranks))
        flops = sum(2.0 * nnz * max(r for m, r in enumerate(ranks) if m != n) +
                    4.0 * min(s, nnz) * P for n, s in enumerate(shape))
        return {"bytes": nnz * (4.0 * len(shape) + 8) + 16.0 * rows, "flops": case["sweeps"] * flops}
    if kind == "ops":
        shape = _ints(case["shape"])
        size, n = math.prod(shape), shape[case["mode"]]
        out = size // n * case["rows"] + n * n
        return {"bytes": 8.0 * (size + out), "flops": 2.0 * size * case["rows"] + 1.0 * size * n}
    one = _dense_work([case["size"]] * 3, [case["rank"]] * 3, case["sweeps"], 4)
    one["flops"] += 2.0 * case["size"] ** 3 * (case["latent"] + case["rank"])
    return one


# -- the same results in 64 bits, by torch -----------------------------------------
def _orth(A):
    """The orthonormal basis of A's columns with a positive triangle."""
    Q, R = torch.linalg.qr(A)
    return Q * torch.where(torch.diagonal(R) < 0, -1.0, 1.0)


def _subspace(S, U, steps):
    for _ in range(steps):
        U = _orth(S @ U)
    return U


def _unfold(Xt, n):
    axis = Xt.dim() - 1 - n
    return torch.movedim(Xt, axis, 0).reshape(Xt.shape[axis], -1)


def _randn_start(shape, ranks, seed=1):
    """The default random start: Marsaglia's polar draws on the C library's
    rand(), mode by mode, orthonormalised."""
    libc = ctypes.CDLL(None)
    libc.srand(seed)
    top, U = 2147483647.0, []
    for s, r in zip(shape, ranks):
        v = np.empty(s * r)
        for k in range(s * r):
            while True:
                a, b = libc.rand() / top * 2 - 1, libc.rand() / top * 2 - 1
                q = a * a + b * b
                if 0 < q <= 1:
                    break
            v[k] = a * math.sqrt(-2 * math.log(q) / q)
        U.append(_orth(torch.as_tensor(v.reshape(r, s).T.copy()).cuda()))
    return U


def _splitmix_gaussian(n, seed):
    mask, out = (1 << 64) - 1, np.empty(n + 1)
    state = (seed * 0x9E3779B97F4A7C15 + 0x1234567) & mask

    def uniform():
        nonlocal state
        state = (state + 0x9E3779B97F4A7C15) & mask
        z = state
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        return (((z ^ (z >> 31)) >> 11) + 0.5) / 9007199254740992.0

    for i in range(0, n, 2):
        rad, turn = math.sqrt(-2 * math.log(uniform())), 2 * math.pi * uniform()
        out[i], out[i + 1] = rad * math.cos(turn), rad * math.sin(turn)
    return out[:n]


def _hosvd_start(Xt, shape, ranks):
    U = []
    for n, (s, r) in enumerate(zip(shape, ranks)):
        A = _unfold(Xt, n)
        start = torch.as_tensor(_splitmix_gaussian(s * r, 1000 + n).reshape(r, s).T.copy()).cuda()
        U.append(_subspace(A @ A.T, start, 30))
    return U


def _hooi(Xt, U, sweeps, tol, inner):
    nd, x2 = Xt.dim(), float((Xt * Xt).sum())
    done, last, residual = 0, -1.0, 0.0
    for _ in range(sweeps):
        for n in range(nd):
            Y = Xt
            for m in range(nd):
                if m != n:
                    Y = _multiply(Y, U[m].T, m)
            A = _unfold(Y, n)
            U[n] = _subspace(A @ A.T, U[n], inner)
        G = _multiply(Y, U[nd - 1].T, nd - 1)
        residual = math.sqrt(max(0.0, 1.0 - float((G * G).sum()) / x2))
        done += 1
        if tol > 0 and last >= 0 and abs(residual - last) < tol:
            break
        last = residual
    return G, U, residual, done


def _exact_sparse(case, seed):
    idx, vals, shape = _coo(case, seed)
    ranks, U = _ints(case["ranks"]), _sparse_start(case, seed)
    nd, rows = len(shape), 1 << 18

    def product(n):
        """Y_(n): row i_n, the other factors' Kronecker product, lowest mode fastest."""
        P = math.prod(r for m, r in enumerate(ranks) if m != n)
        Y = torch.zeros(shape[n], P, dtype=torch.float64, device="cuda")
        for b in range(0, vals.numel(), rows):
            K = vals[b:b + rows, None]
            for m in range(nd):
                if m != n:
                    K = (U[m][idx[m][b:b + rows]][:, :, None] * K[:, None, :]).flatten(1)
            Y.index_add_(0, idx[n][b:b + rows], K)
        return Y

    for _ in range(case["sweeps"]):
        for n in range(nd):
            Y = product(n)
            U[n] = _orth(Y @ (Y.T @ U[n]))
    L = product(nd - 1).T @ U[nd - 1]
    residual = math.sqrt(max(0.0, 1.0 - float((L * L).sum()) / float((vals * vals).sum())))
    return {"G": L.cpu().numpy(), "U": [u.cpu().numpy() for u in U], "residual": residual}


def _exact_batched(case, seed):
    if case["count"] > 128:
        return None
    packed, U0, gsize = _batch(case, seed)
    G, U, relerr = np.empty(gsize), np.empty(U0.numel()), np.empty(case["count"])
    X, U0 = packed["X"].cpu().double(), U0.cpu()
    for t in range(case["count"]):
        shape = [int(v) for v in packed["shapes"][3 * t:3 * t + 3]]
        ranks = [int(v) for v in packed["ranks"][3 * t:3 * t + 3]]
        o = int(packed["xoff"][t])
        Xt = X[o:o + math.prod(shape)].reshape(shape[::-1])
        start = []
        for n in range(3):
            o = int(packed["uoff"][3 * t + n])
            start.append(U0[o:o + shape[n] * ranks[n]].reshape(ranks[n], shape[n]).T)
        core, V, relerr[t], _ = _hooi(Xt, start, case["sweeps"], 0.0, 5)
        o = int(packed["goff"][t])
        G[o:o + core.numel()] = core.reshape(-1)
        for n in range(3):
            o = int(packed["uoff"][3 * t + n])
            U[o:o + V[n].numel()] = V[n].T.reshape(-1)
    return {"G": G, "U": U, "relerr": relerr}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("fp64", "mixed"):
        dtype = torch.float64 if case.get("dtype") == "f64" else torch.float32
        Xt = _tucker(case, seed, dtype).double()
        shape, ranks = _ints(case["shape"]), _ints(case["ranks"])
        start = (_hosvd_start(Xt, shape, ranks) if case.get("init") == "hosvd"
                 else _randn_start(shape, ranks))
        G, U, residual, done = _hooi(Xt, start, case["sweeps"], case["tol"],
                                     5 if kind == "fp64" else 2)
        return {"G": _reversed(G.contiguous()), "U": U, "residual": residual, "sweeps": done}
    if kind == "batched":
        return _exact_batched(case, seed)
    if kind == "sparse":
        return _exact_sparse(case, seed)
    if kind == "ops":
        shape, g = _ints(case["shape"]), _generator(seed)
        Xt = _f64(shape[::-1], g)
        M = _f64((shape[case["mode"]], case["rows"]), g).T
        A = _unfold(Xt, case["mode"])
        return {"Y": _reversed(_multiply(Xt, M, case["mode"])), "S": A @ A.T}
    # The warm start's own subspaces start from draws inside the library: only
    # what does not depend on their basis has a value here.
    return None
