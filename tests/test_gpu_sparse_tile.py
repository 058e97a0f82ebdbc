"""SparseSign / CountSketch compress on 32-vector tiles (csrc/rla_sparse_tile.cu): edges of
the chunks (640 long indices Float32, 320 Float64), of the bucket windows (1136 / 568 buckets,
up to eight), of the vector tiles and of the list lengths, all load paths (16-byte, any
alignment, strided), against the FP64 oracle on the same draws.

Tolerance: a bucket sums t = L * nnz / s terms (at most 20480 here) in Float32 in runs; the
random-walk error of such a sum is about sqrt(t) * 2^-24 / 2 of its own norm sqrt(t), times a few
levels of partial sums: below 1e-6 in the Frobenius norm; Float64 scales by 2^-29."""
import numpy as np
import pytest

from helpers import TOL, oracle_recipe, rel_err

pytestmark = pytest.mark.gpu

#       L, s, nnz, nv
SIZES = [(1, 1, 1, 1), (5, 2, 2, 3), (319, 3, 2, 31), (321, 16, 8, 32), (639, 31, 31, 33), (640, 32, 32, 1),
         (641, 100, 8, 65), (1281, 257, 8, 40), (3000, 568, 8, 33), (3000, 569, 4, 33), (2000, 1136, 8, 31),
         (2000, 1137, 3, 35), (1500, 4544, 2, 9), (1300, 9088, 8, 5), (20000, 20, 20, 64)]


def column_major(x, pad, dev):
    """x in a column-major device buffer whose leading dimension is rows + pad."""
    import torch
    r, c = x.shape
    buf = torch.zeros(c, r + pad, dtype=torch.from_numpy(x[:1, :1].copy()).dtype, device=dev)
    buf[:, :r] = torch.from_numpy(np.ascontiguousarray(x.T)).to(dev)
    return buf[:, :r].t()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("card", ["left", "right"])
@pytest.mark.parametrize("pad", [0, 1])
def test_tile_edges(rla, orc, dev, dtype, card, pad):
    for L, s, nnz, nv in SIZES:
        rng = np.random.default_rng([L, s, nnz, nv])
        cd = rla.Left() if card == "left" else rla.Right()
        comp = rla.SparseSign(cardinality=cd, compression_dim=s, nnz=nnz, type=dtype)
        shape = (L, nv) if card == "left" else (nv, L)
        A = rng.standard_normal(shape).astype(dtype)
        out = (s, nv) if card == "left" else (nv, s)
        C = rng.standard_normal(out).astype(dtype)
        S = rla.complete_compressor(comp, A, seed=5)
        R = oracle_recipe(orc, S)
        ref = C.astype(np.float64).copy(order="F")
        Ad, Cd = column_major(A, pad, dev), column_major(C, pad, dev)
        if card == "left":
            rla.mul_(Cd, S, Ad, 0.5, -2.0)
            orc.mul_SA(ref, R, A.astype(np.float64), 0.5, -2.0)
        else:
            rla.mul_(Cd, Ad, S, 0.5, -2.0)
            orc.mul_AS(ref, A.astype(np.float64), R, 0.5, -2.0)
        err = rel_err(Cd.cpu().numpy(), ref)
        assert err < TOL[dtype], (L, s, nnz, nv, err)


def test_count_sketch_strided_and_infinities(rla, orc, dev):
    """A row of A with an infinity reaches its own buckets only; the rest stays finite."""
    rng = np.random.default_rng(8)
    L, s, nv = 2000, 50, 70
    A = rng.standard_normal((nv, L)).astype(np.float32)
    A[3, 17] = np.inf
    S = rla.complete_compressor(rla.CountSketch(cardinality=rla.Right(), compression_dim=s, type=np.float32), A, seed=2)
    C = column_major(np.full((nv, s), np.nan, np.float32), 0, dev)
    rla.mul_(C, column_major(A, 0, dev), S)
    out = C.cpu().numpy()
    b, v = int(S.draws()["rowval"][17]), float(S.draws()["nzval"][17])
    assert out[3, b] == np.inf * v
    out[3, b] = 0.0
    assert np.isfinite(out).all()
    B = A.astype(np.float64)
    B[3, 17] = 0.0
    ref = np.zeros((nv, s), order="F")
    orc.mul_AS(ref, B, oracle_recipe(orc, S))
    ref[3, b] = 0.0
    assert rel_err(out, ref) < TOL[np.float32]


def test_loaded_draws_with_repeated_buckets(rla, orc, dev):
    """Loaded draws may repeat a bucket inside a long index; both entries count."""
    rng = np.random.default_rng(9)
    L, s, nnz, nv = 700, 12, 4, 34
    A = rng.standard_normal((L, nv))
    S = rla.complete_compressor(rla.SparseSign(compression_dim=s, nnz=nnz, type=np.float64), A, seed=2)
    idx = rng.integers(0, s, L * nnz)
    vals = np.where(rng.integers(0, 2, L * nnz) == 1, 0.5, -0.5)
    S.load_draws(idx=idx, vals=vals)
    dense = np.zeros((s, L))
    np.add.at(dense, (idx, np.repeat(np.arange(L), nnz)), vals)
    out = (S @ column_major(A, 0, dev)).cpu().numpy()
    assert rel_err(out, dense @ A) < TOL[np.float64]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_count_sketch_few_buckets(rla, orc, dev, dtype):
    """CountSketch up to 2080 buckets: groups of four entries (dense buckets) and single ones."""
    for L, s, nv, pad in [(1, 1, 1, 0), (639, 300, 33, 1), (5000, 319, 40, 0), (5000, 321, 40, 1), (20001, 1040, 31, 0),
                          (20001, 1041, 33, 1), (7000, 2080, 17, 0), (3000, 2, 5, 1)]:
        rng = np.random.default_rng([L, s])
        A = rng.standard_normal((L, nv)).astype(dtype)
        S = rla.complete_compressor(rla.CountSketch(compression_dim=s, type=dtype), A, seed=7)
        ref = np.zeros((s, nv), order="F")
        orc.mul_SA(ref, oracle_recipe(orc, S), A.astype(np.float64))
        C = column_major(np.zeros((s, nv), dtype), pad, dev)
        rla.mul_(C, S, column_major(A, pad, dev))
        assert rel_err(C.cpu().numpy(), ref) < TOL[dtype], (L, s, nv)


@pytest.mark.parametrize("nnz", [1, 8])
@pytest.mark.parametrize("s", [40, 900])
@pytest.mark.parametrize("used", [1, 3])
def test_all_entries_in_few_buckets(rla, dev, nnz, s, used):
    """Loaded draws that put every entry into one or three buckets: runs longer than an octet's
    share, which the octets of a warp add one after another."""
    rng = np.random.default_rng([nnz, s, used])
    L, nv = 1500, 34
    A = rng.standard_normal((L, nv))
    comp = (rla.CountSketch(compression_dim=s, type=np.float64) if nnz == 1
            else rla.SparseSign(compression_dim=s, nnz=nnz, type=np.float64))
    S = rla.complete_compressor(comp, A, seed=2)
    idx = 16 * rng.integers(0, used, L * nnz)
    vals = np.where(rng.integers(0, 2, L * nnz) == 1, 1.0, -1.0) * (1.0 if nnz == 1 else 1.0 / np.sqrt(nnz))
    S.load_draws(idx=idx, vals=vals)
    dense = np.zeros((s, L))
    np.add.at(dense, (idx, np.repeat(np.arange(L), nnz)), vals)
    out = (S @ column_major(A, 0, dev)).cpu().numpy()
    assert rel_err(out, dense @ A) < TOL[np.float64]
