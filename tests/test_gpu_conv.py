"""Gaussian applies in Float32 through the converting tensor-core kernel (csrc/rla_tc_conv.cu): edges
of the 128 x 64 tiles, of the k-blocks (32) and their chunks (128), one and several K splits, either
operand as the converted one, both layouts, aligned and odd leading dimensions, alpha and beta,
against the FP64 oracle on the same draws.

Tolerance: three BF16 terms hold all 24 bits of a Float32; the dropped term products are below
2^-24 of their factors and the FP32 accumulation of a chunk of 128 products adds at most a few
2^-24 relative to its partial sums: below 1e-6 in the Frobenius norm (4.6e-7 measured at K = 1024)."""
import numpy as np
import pytest

from helpers import TOL, oracle_recipe, rel_err
from test_gpu_sparse_tile import column_major

pytestmark = pytest.mark.gpu

#       L, s, nv
SIZES = [(1, 1, 1), (31, 3, 2), (32, 64, 128), (33, 65, 129), (127, 10, 300), (129, 200, 64), (700, 130, 127),
         (1000, 40, 3000), (4099, 33, 70), (5000, 300, 20), (257, 63, 5000)]


@pytest.mark.parametrize("card", ["left", "right"])
@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("row_major", [False, True])
def test_conv_edges(rla, orc, dev, card, adjoint, pad, row_major):
    import torch
    dtype = np.float32
    for L, s, nv in SIZES:
        rng = np.random.default_rng([L, s, nv])
        cd = rla.Left() if card == "left" else rla.Right()
        comp = rla.Gaussian(cardinality=cd, compression_dim=s, type=dtype)
        long_, short = ((L, nv), (s, nv)) if card == "left" else ((nv, L), (nv, s))
        A = rng.standard_normal(short if adjoint else long_).astype(dtype)
        C = rng.standard_normal(long_ if adjoint else short).astype(dtype)
        S = rla.complete_compressor(comp, np.zeros(long_, dtype), seed=4)
        R = oracle_recipe(orc, S)
        alpha, beta = (0.5, -2.0) if pad else (1.0, 0.0)
        ref = C.astype(np.float64).copy(order="F")
        Ad = torch.from_numpy(A.copy()).to(dev) if row_major else column_major(A, pad, dev)
        Cd = column_major(C, pad, dev)
        A64 = A.astype(np.float64)
        St = S.T if adjoint else S
        if card == "left":
            rla.mul_(Cd, St, Ad, alpha, beta)
            (orc.mul_StA if adjoint else orc.mul_SA)(ref, R, A64, alpha, beta)
        else:
            rla.mul_(Cd, Ad, St, alpha, beta)
            (orc.mul_ASt if adjoint else orc.mul_AS)(ref, A64, R, alpha, beta)
        err = rel_err(Cd.cpu().numpy(), ref)
        assert err < TOL[dtype], (L, s, nv, err)
