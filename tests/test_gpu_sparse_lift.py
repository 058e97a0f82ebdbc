"""SparseSign / CountSketch expand on tiles of vectors (csrc/rla_sparse_lift.cu): edges of the
blocks of 32 long indices, of the vector tiles, odd and even nnz, aligned and odd leading
dimensions, both layouts, and the compression dimensions at which the staged row narrows from
128 to 64 to 32 bytes and the general kernel takes over, against the FP64 oracle.

Tolerance: at most nnz = 9 terms per output, so the error is below nnz * 2^-24 of the sum of
magnitudes, in the Frobenius norm below 9 * 2^-24 * sqrt(9) = 1.6e-6 at worst and about 1e-7
for random data; TOL is 1e-6 (Float32) and 1e-12 (Float64)."""
import numpy as np
import pytest

from helpers import TOL, oracle_recipe, rel_err
from test_gpu_sparse_tile import column_major

pytestmark = pytest.mark.gpu

#       L, s, nnz, nv
SIZES = [(1, 1, 1, 1), (31, 2, 2, 3), (32, 3, 3, 15), (33, 40, 8, 16), (513, 100, 9, 33), (1000, 1150, 4, 32),
         (700, 1170, 2, 17), (600, 2060, 8, 9), (600, 2100, 8, 8), (400, 3400, 1, 5), (400, 3600, 2, 4), (3000, 64, 8, 70)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("card", ["left", "right"])
@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("row_major", [False, True])
def test_lift_edges(rla, orc, dev, dtype, card, pad, row_major):
    import torch
    for L, s, nnz, nv in SIZES:
        rng = np.random.default_rng([L, s, nnz, nv])
        cd = rla.Left() if card == "left" else rla.Right()
        comp = rla.SparseSign(cardinality=cd, compression_dim=s, nnz=nnz, type=dtype)
        long_shape, short = ((L, nv), (s, nv)) if card == "left" else ((nv, L), (nv, s))
        Y = rng.standard_normal(short).astype(dtype)
        C = rng.standard_normal(long_shape).astype(dtype)
        S = rla.complete_compressor(comp, np.zeros(long_shape, dtype), seed=6)
        R = oracle_recipe(orc, S)
        Yd = column_major(Y, pad, dev)
        for alpha, beta in [(0.5, -2.0), (1.0, 0.0)]:
            ref = C.astype(np.float64).copy(order="F")
            Cd = torch.from_numpy(C.copy()).to(dev) if row_major else column_major(C, pad, dev)
            if card == "left":
                rla.mul_(Cd, S.T, Yd, alpha, beta)
                orc.mul_StA(ref, R, Y.astype(np.float64), alpha, beta)
            else:
                rla.mul_(Cd, Yd, S.T, alpha, beta)
                orc.mul_ASt(ref, Y.astype(np.float64), R, alpha, beta)
            err = rel_err(Cd.cpu().numpy(), ref)
            assert err < TOL[dtype], (L, s, nnz, nv, alpha, beta, err)
