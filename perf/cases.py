"""The work that programs using this package spend their time on, as measurable cases.

A case is a dict of plain values.  ``listed()`` gives the fixed ones, ``draw(rng)`` another
one of the same ranges, ``prepare`` what a program holds before the call, ``run`` one pass
through the public entry points, ``work`` the bytes and operations a pass cannot do without
and ``exact`` the values of the same outputs in 64 bits, from plain torch.

Families (``case["op"]``):

``apply``    mul!(C, S, A), mul!(C, A, S) and the adjoint forms, for the five compressors,
             with both element types.  ``rows`` x ``cols`` is the long (uncompressed) matrix: the
             input of a compression, the output of an expansion (``adjoint``).  Matrices are
             column-major, the package's native layout.
``randsvd``  rapproximate!(RandSVD): Gaussian sketch, power iterations, small SVD.
``batch``    one run of a grouped RandSVD plan over many uneven instances.
``ihs``      complete_solver + rsolve!(IHS) on a new least-squares problem, a fixed number of
             iterations, each with a fresh SparseSign sketch.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

NAME = "randlinearalgebra_b200"


def _package():
    """The package: its folder name is not a Python identifier, so it is loaded by path."""
    if NAME not in sys.modules:
        folder = os.path.join(os.getcwd(), "randlinearalgebra.jl_b200")
        spec = importlib.util.spec_from_file_location(NAME, os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[NAME] = mod
        spec.loader.exec_module(mod)
    return sys.modules[NAME]


rla = _package()


def _device():
    return torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")


# --------------------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------------------
def _apply(kind, side, rows, cols, s, f64=False, adjoint=False, nnz=1, **more):
    return {"op": "apply", "kind": kind, "side": side, "rows": rows, "cols": cols, "s": s, "nnz": nnz, "f64": f64,
            "adjoint": adjoint, **more}


def listed():
    return [
        # the smallest call: one dense Float64 block sketched for a small regression; launches
        # and host time count as much as the kernel
        _apply("sparse_sign", "left", 4096, 256, 512, f64=True, nnz=8, name="sparse_sign_left_f64_4096"),
        # the headline sketch applies: a tall Float32 matrix of 2 GiB to 4096 rows
        _apply("count_sketch", "left", 1 << 20, 512, 4096, name="count_sketch_left_f32_2p20"),
        _apply("srht", "left", 1 << 20, 512, 4096, name="srht_left_f32_2p20"),
        # the sketch of a sketch-and-solve least-squares request, ragged sizes, s = 4 cols
        _apply("sparse_sign", "left", 150001, 333, 1332, nnz=8, name="sparse_sign_left_f32_ragged"),
        # a Johnson-Lindenstrauss embedding of column vectors that are not a power of two long
        _apply("fjlt", "left", 100003, 96, 600, name="fjlt_left_f32_ragged"),
        # the default range-finder sketch A*S: SparseSign from the right, few columns
        _apply("sparse_sign", "right", 30011, 3000, 100, nnz=8, name="sparse_sign_right_f32"),
        # the dense sketch A*Omega of a range finder, Float32 accuracy
        _apply("gaussian", "right", 65536, 1024, 128, name="gaussian_right_f32"),
        # the way back, S'*Y: lifting sketched quantities to the long dimension (Float64)
        _apply("sparse_sign", "left", 1 << 17, 200, 1000, f64=True, adjoint=True, nnz=8, name="sparse_sign_lift_f64"),
        # whole calls: the mixed-precision RandSVD, and an ordinary Float64 one
        {"op": "randsvd", "m": 65536, "n": 8192, "l": 272, "rank": 512, "q": 2, "f64": False, "split": True,
         "name": "randsvd_split_f32_65536x8192"},
        {"op": "randsvd", "m": 3000, "n": 3000, "l": 30, "rank": 120, "q": 1, "f64": True, "split": False,
         "name": "randsvd_f64_3000"},
        # many uneven factorizations at once
        {"op": "batch", "count": 16, "m_lo": 4096, "m_hi": 65536, "n_lo": 64, "n_hi": 1024, "split": True,
         "name": "randsvd_batch_16"},
        # an iterative least-squares solve from scratch, one fresh sketch per iteration
        {"op": "ihs", "m": 1 << 17, "n": 256, "s": 1024, "its": 6, "name": "ihs_f32_2p17x256"},
    ]


def _log(rng, lo, hi):
    """Log-uniform whole number, odd ones among them."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """Sketch applies of every kind, side, type and direction; now and then a whole call."""
    what = rng.random()
    if what < 0.10:
        n = _log(rng, 300, 4000)
        m = _log(rng, n, 32768)
        split = rng.random() < 0.5
        l = rng.randint(10, min(200, n // 3))
        return {"op": "randsvd", "m": m, "n": n, "l": l, "rank": min(n, 2 * l), "q": rng.randint(0, 2),
                "f64": not split and rng.random() < 0.5, "split": split}
    if what < 0.15:
        return {"op": "batch", "count": rng.randint(4, 16), "m_lo": 4096, "m_hi": 65536, "n_lo": 64, "n_hi": 1024,
                "split": rng.random() < 0.5}
    if what < 0.22:
        n = _log(rng, 32, 512)
        return {"op": "ihs", "m": _log(rng, 1 << 14, 1 << 18), "n": n, "s": 4 * n, "its": rng.randint(2, 6)}
    kind = rng.choice(["sparse_sign", "sparse_sign", "count_sketch", "srht", "fjlt", "gaussian"])
    side = rng.choice(["left", "left", "right"])
    # elements of the long matrix: up to the headline shape for the streaming kinds, less where
    # a pass does more per element
    most = {"sparse_sign": 1 << 27, "count_sketch": 1 << 29, "srht": 1 << 29, "fjlt": 1 << 25, "gaussian": 1 << 27}[kind]
    long_dim = _log(rng, 1000, {"gaussian": 1 << 14, "fjlt": 1 << 17}.get(kind, 1 << 20 if side == "left" else 1 << 14))
    other = _log(rng, 16, min(most // long_dim, 512 if side == "left" else 1 << 16))
    rows, cols = (long_dim, other) if side == "left" else (other, long_dim)
    s = _log(rng, 32, min(4096 if side == "left" else 512, long_dim // 4))
    return _apply(kind, side, rows, cols, s, f64=rng.random() < 0.35, adjoint=rng.random() < 0.25,
                  nnz=rng.choice([2, 4, 8, 8]) if kind == "sparse_sign" else 1)


# --------------------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed))
    return g


def _normal(rows, cols, dtype, g):
    """Column-major rows x cols, N(0,1)."""
    return torch.randn(cols, rows, dtype=dtype, device=g.device, generator=g).t()


def _next_pow2(n):
    return 1 << max(0, (n - 1).bit_length())


def _sketch_draws(c, seed):
    """The random draws of an ``apply`` case in the recipes' own layout (0-based)."""
    rng = np.random.default_rng([int(seed), 11])
    L = c["rows"] if c["side"] == "left" else c["cols"]
    s, dt = c["s"], np.float64 if c["f64"] else np.float32
    kind = c["kind"]
    if kind in ("sparse_sign", "count_sketch"):
        nnz = c["nnz"]
        idx = np.sort(rng.integers(0, s, (L, nnz)), axis=1)
        bad = np.nonzero((np.diff(idx, axis=1) == 0).any(axis=1))[0]
        while bad.size:  # nnz distinct buckets per long index
            idx[bad] = np.sort(rng.integers(0, s, (bad.size, nnz)), axis=1)
            bad = bad[(np.diff(idx[bad], axis=1) == 0).any(axis=1)]
        scale = dt(1.0 / np.sqrt(float(nnz))) if kind == "sparse_sign" else dt(1.0)
        vals = np.where(rng.integers(0, 2, L * nnz) == 1, scale, -scale).astype(dt)
        return {"idx": idx.reshape(-1).astype(np.int64), "vals": vals}
    if kind == "gaussian":
        shape = (s, L) if c["side"] == "left" else (L, s)
        return {"vals": (rng.standard_normal(shape) / np.sqrt(float(s))).astype(dt)}
    N = _next_pow2(L)
    signs = rng.integers(0, 2, N).astype(np.uint8)
    if kind == "srht":
        return {"idx": rng.permutation(N)[:s].astype(np.int64), "signs": signs}
    q = min(1.0, 0.25 * math.log(L) ** 2 / L)
    # K (s x N): a Bernoulli(q) pattern with N(0,1) values, given by the columns of op
    n_major, n_minor = (N, s) if c["side"] == "left" else (s, N)
    pos = np.unique(rng.integers(0, n_major * n_minor, rng.binomial(s * N, q)))
    kptr = np.searchsorted(pos // n_minor, np.arange(n_major + 1)).astype(np.int64)
    return {"kptr": kptr, "idx": (pos % n_minor).astype(np.int64), "signs": signs,
            "vals": rng.standard_normal(pos.size).astype(dt)}


_KINDS = {"sparse_sign": "SparseSign", "count_sketch": "CountSketch", "srht": "SRHT", "fjlt": "FJLT",
          "gaussian": "Gaussian"}


def _sizes(c):
    """(input rows, input cols, output rows, output cols) of an ``apply`` case."""
    long_, short = (c["rows"], c["cols"]), ((c["s"], c["cols"]) if c["side"] == "left" else (c["rows"], c["s"]))
    return (*short, *long_) if c["adjoint"] else (*long_, *short)


def _apply_input(c, seed):
    r, k, _, _ = _sizes(c)
    return _normal(r, k, torch.float64 if c["f64"] else torch.float32, _gen(seed))


def _low_rank(m, n, rank, dtype, seed):
    """Column-major U diag(i^-1.5) V' + 1e-6 N(0,1)."""
    g = _gen(seed)
    U = torch.linalg.qr(torch.randn(m, rank, device=g.device, generator=g, dtype=dtype))[0]
    V = torch.linalg.qr(torch.randn(n, rank, device=g.device, generator=g, dtype=dtype))[0]
    sig = torch.arange(1, rank + 1, device=g.device, dtype=dtype) ** -1.5
    At = (V * sig) @ U.t()
    At.add_(torch.randn(n, m, device=g.device, generator=g, dtype=dtype), alpha=1e-6)
    return At.t()


def _omega(c, seed):
    rng = np.random.default_rng([int(seed), 13])
    dt = np.float64 if c["f64"] else np.float32
    return (rng.standard_normal((c["n"], c["l"])) / np.sqrt(float(c["l"]))).astype(dt)


def _batch_shapes(c):
    """The sizes of the instances depend on the case alone; their entries on the seed."""
    rng = np.random.default_rng(4)
    ms = rng.integers(c["m_lo"], c["m_hi"] + 1, size=c["count"])
    ns = rng.integers(c["n_lo"], c["n_hi"] + 1, size=c["count"])
    ks = rng.choice([16, 32, 64], size=c["count"])
    return [(int(m), int(n), int(min(k, n))) for m, n, k in zip(ms, ns, ks)]


def _decaying(m, n, g):
    """Column-major U diag(0.9^i) V' + 1e-6 N(0,1), Float32."""
    r = min(n, 160)
    U = torch.linalg.qr(torch.randn(m, r, device=g.device, generator=g))[0]
    V = torch.linalg.qr(torch.randn(n, r, device=g.device, generator=g))[0]
    At = (V * 0.9 ** torch.arange(r, device=g.device, dtype=torch.float32)) @ U.t()
    At.add_(torch.randn(n, m, device=g.device, generator=g), alpha=1e-6)
    return At.t()


def prepare(case, seed):
    c = case
    np_t = np.float64 if c.get("f64") else np.float32
    if c["op"] == "apply":
        A = _apply_input(c, seed)
        card = rla.Left() if c["side"] == "left" else rla.Right()
        more = {"nnz": c["nnz"]} if c["kind"] == "sparse_sign" else {}
        comp = getattr(rla, _KINDS[c["kind"]])(cardinality=card, compression_dim=c["s"], type=np_t, **more)
        # complete_compressor takes its long dimension from the matrix it will be applied to
        like = torch.empty(c["cols"], c["rows"], device="meta").t()
        S = rla.complete_compressor(comp, like, seed=int(seed))
        S.load_draws(**_sketch_draws(c, seed))
        _, _, r, k = _sizes(c)
        C = torch.zeros(k, r, dtype=A.dtype, device=A.device).t()
        return {"op": "apply", "A": A, "S": S.T if c["adjoint"] else S, "C": C, "left": c["side"] == "left"}
    if c["op"] == "randsvd":
        A = _low_rank(c["m"], c["n"], c["rank"], torch.float64 if c["f64"] else torch.float32, seed)
        comp = rla.Gaussian(cardinality=rla.Right(), compression_dim=c["l"], type=np_t)
        R = rla.complete_approximator(
            rla.RandSVD(compressor=comp, power_its=c["q"], orthogonalize=True, factor_type=np_t,
                        precision=rla.RLA_PREC_SPLIT_BF16 if c["split"] else rla.RLA_PREC_NATIVE), A, seed=int(seed))
        R.compressor.load_draws(vals=_omega(c, seed))
        return {"op": "randsvd", "A": A, "R": R}
    if c["op"] == "batch":
        g = _gen(seed)
        shapes = _batch_shapes(c)
        As = [_decaying(m, n, g) for m, n, _ in shapes]
        B = rla.RandSVDBatch(As, [k for _, _, k in shapes], [4000 + 7 * i for i in range(len(shapes))], autotune=False,
                             precision=rla.RLA_PREC_SPLIT_BF16 if c["split"] else rla.RLA_PREC_NATIVE)
        return {"op": "batch", "B": B}
    g = _gen(seed)
    A = _normal(c["m"], c["n"], torch.float32, g)
    b = A @ torch.randn(c["n"], device=A.device, generator=g) + 1e-3 * torch.randn(c["m"], device=A.device, generator=g)
    ihs = rla.IHS(compressor=rla.SparseSign(compression_dim=c["s"], nnz=8, type=np.float32),
                  log=rla.BasicLogger(max_it=c["its"]))
    return {"op": "ihs", "A": A, "b": b, "ihs": ihs, "seed": int(seed)}


def run(state):
    s = state
    if s["op"] == "apply":
        if s["left"]:
            rla.mul_(s["C"], s["S"], s["A"])
        else:
            rla.mul_(s["C"], s["A"], s["S"])
        return s["C"]
    if s["op"] == "randsvd":
        rla.rapproximate_(s["R"], s["A"])
        return {"U": s["R"].U, "S": s["R"].S, "V": s["R"].V}
    if s["op"] == "batch":
        s["B"].run()
        return {"U": s["B"].U, "S": s["B"].S, "V": s["B"].V}
    x = torch.zeros(s["A"].shape[1], device=s["A"].device)
    solver = rla.complete_solver(s["ihs"], x, s["A"], s["b"], seed=s["seed"])
    rla.rsolve_(solver, x, s["A"], s["b"])
    return x


def work(case):
    c = case
    es = 8 if c.get("f64") else 4
    if c["op"] == "apply":
        r, k, ro, ko = _sizes(c)
        L, nv = (c["rows"], c["cols"]) if c["side"] == "left" else (c["cols"], c["rows"])
        N = _next_pow2(L)
        per = {"sparse_sign": 2.0 * c["nnz"] * L, "count_sketch": 1.0 * L, "srht": N * math.log2(N),
               "fjlt": N * math.log2(N) + 0.5 * math.log(L) ** 2 * c["s"], "gaussian": 2.0 * L * c["s"]}[c["kind"]]
        dense = es * L * c["s"] if c["kind"] == "gaussian" else 0
        return {"bytes": es * (r * k + ro * ko) + dense, "flops": per * nv}
    if c["op"] == "randsvd":
        m, n, l = c["m"], c["n"], c["l"]
        return {"bytes": es * (m * n + (m + n) * l + n * l) + 8 * l, "flops": 2.0 * m * n * l * (2 * c["q"] + 2)}
    if c["op"] == "batch":
        sh = _batch_shapes(c)
        return {"bytes": sum(4 * (m * n + (m + n) * k) + 8 * k for m, n, k in sh),
                "flops": sum(4.0 * m * n * k for m, n, k in sh)}
    m, n, s = c["m"], c["n"], c["s"]
    return {"bytes": 4 * (m * n + m + n), "flops": c["its"] * (4.0 * m * n + 16.0 * m * n + 2.0 * s * n * n)}


# --------------------------------------------------------------------------------------
# the same outputs in 64 bits
# --------------------------------------------------------------------------------------
def _wht(X):
    """Natural-order Walsh-Hadamard transform of the columns."""
    N, nv = X.shape
    h = 1
    while h < N:
        Y = X.view(N // (2 * h), 2, h, nv)
        X = torch.stack((Y[:, 0] + Y[:, 1], Y[:, 0] - Y[:, 1]), dim=1).view(N, nv)
        h *= 2
    return X


def _operator(c, seed):
    """(compress, expand): the 64-bit maps R^L -> R^s and back on blocks of columns."""
    d = _sketch_draws(c, seed)
    dev = _device()
    L, s = (c["rows"] if c["side"] == "left" else c["cols"]), c["s"]
    dev_of = lambda a: torch.from_numpy(a).to(dev)  # noqa: E731
    if c["kind"] == "gaussian":
        G = dev_of(d["vals"]).double()
        G = G if c["side"] == "left" else G.t()
        return (lambda X: G @ X), (lambda Y: G.t() @ Y)
    if c["kind"] in ("sparse_sign", "count_sketch"):
        nnz = c["nnz"]
        idx, vals = dev_of(d["idx"]).view(L, nnz), dev_of(d["vals"]).double().view(L, nnz)

        def compress(X):
            Y = torch.zeros(s, X.shape[1], dtype=torch.float64, device=dev)
            for e in range(nnz):
                Y.index_add_(0, idx[:, e], vals[:, e:e + 1] * X)
            return Y

        return compress, (lambda Y: sum(vals[:, e:e + 1] * Y[idx[:, e]] for e in range(nnz)))
    N = _next_pow2(L)
    D = dev_of(d["signs"]).double().mul_(2).sub_(1).unsqueeze(1)
    if c["kind"] == "srht":
        rows, scale = dev_of(d["idx"]), math.sqrt(s) / math.sqrt(N)
        pick = lambda X: X[rows]  # noqa: E731
        put = lambda Y: torch.zeros(N, Y.shape[1], dtype=torch.float64, device=dev).index_copy_(0, rows, Y)  # noqa: E731
    else:
        q = min(1.0, 0.25 * math.log(L) ** 2 / L)
        scale = 1.0 / (math.sqrt(N) * math.sqrt(q) * math.sqrt(s))
        major = np.repeat(np.arange(d["kptr"].size - 1), np.diff(d["kptr"]))
        i, j = (d["idx"], major) if c["side"] == "left" else (major, d["idx"])
        i, j, v = dev_of(i), dev_of(j), dev_of(d["vals"]).double().unsqueeze(1)
        pick = lambda X: torch.zeros(s, X.shape[1], dtype=torch.float64, device=dev).index_add_(0, i, v * X[j])  # noqa: E731
        put = lambda Y: torch.zeros(N, Y.shape[1], dtype=torch.float64, device=dev).index_add_(0, j, v * Y[i])  # noqa: E731

    def compress(X):
        P = torch.zeros(N, X.shape[1], dtype=torch.float64, device=dev)
        P[:L] = X
        return pick(_wht(P.mul_(D))) * scale

    return compress, (lambda Y: (_wht(put(Y)) * D)[:L] * scale)


def _exact_apply(c, seed):
    A = _apply_input(c, seed)
    compress, expand = _operator(c, seed)
    f = expand if c["adjoint"] else compress
    X = A if c["side"] == "left" else A.t()
    L = c["rows"] if c["side"] == "left" else c["cols"]
    step = max(1, (1 << 25) // L)
    out = [f(X[:, k:k + step].double()).t() for k in range(0, X.shape[1], step)]
    out = torch.cat(out).t()
    return out if c["side"] == "left" else out.t()


def _exact_singular_values(c, seed):
    dt = torch.float64 if c["f64"] else torch.float32
    A = _low_rank(c["m"], c["n"], c["rank"], dt, seed).double()
    Q = torch.linalg.qr(A @ torch.from_numpy(_omega(c, seed)).to(A.device).double())[0]
    for _ in range(c["q"]):
        Q = torch.linalg.qr(A.t() @ Q)[0]
        Q = torch.linalg.qr(A @ Q)[0]
    return torch.linalg.svdvals(torch.linalg.qr(A.t() @ Q)[1])


def exact(case, seed):
    if case["op"] == "apply":
        return _exact_apply(case, seed)
    if case["op"] == "randsvd":
        # singular vectors are defined up to their signs
        return {"U": None, "S": _exact_singular_values(case, seed), "V": None}
    return None  # the draws are made inside the call
