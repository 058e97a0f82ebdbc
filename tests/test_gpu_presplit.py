"""Gaussian applies in Float32 whose operands are both split into BF16 terms in memory
(gemm_f32_tc_presplit, csrc/rla_tc.cu): both result dimensions above 256 and K above 256, at that rule's
edges, one and several K splits, both sides, directions and layouts, odd leading dimensions, alpha and
beta, against the FP64 oracle on the same draws.  test_host_routes.py checks which kernel each runs.

Tolerance: three BF16 terms hold all 24 bits of a Float32, the dropped term products are below 2^-24 of
their factors, and a chunk of 128 products is accumulated in FP32: below TOL = 1e-6 in the Frobenius norm
as for the converting kernel (4.6e-7 at K = 1024)."""
import numpy as np
import pytest

from helpers import TOL, oracle_recipe, rel_err
from test_gpu_sparse_tile import column_major

pytestmark = pytest.mark.gpu

#        L, s, nv
SPLITS = [(257, 257, 257), (700, 300, 264), (3000, 260, 400), (513, 513, 1000), (300, 1100, 513)]


@pytest.mark.parametrize("card", ["left", "right"])
@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("row_major", [False, True])
def test_presplit_edges(rla, orc, dev, card, adjoint, pad, row_major):
    import torch
    dtype = np.float32
    for L, s, nv in SPLITS:
        rng = np.random.default_rng([L, s, nv])
        cd = rla.Left() if card == "left" else rla.Right()
        long_, short = ((L, nv), (s, nv)) if card == "left" else ((nv, L), (nv, s))
        A = rng.standard_normal(short if adjoint else long_).astype(dtype)
        C = rng.standard_normal(long_ if adjoint else short).astype(dtype)
        S = rla.complete_compressor(rla.Gaussian(cardinality=cd, compression_dim=s, type=dtype), np.zeros(long_, dtype), seed=4)
        R = oracle_recipe(orc, S)
        alpha, beta = (0.5, -2.0) if pad else (1.0, 0.0)
        ref = C.astype(np.float64).copy(order="F")
        Ad = torch.from_numpy(A.copy()).to(dev) if row_major else column_major(A, pad, dev)
        Cd = column_major(C, pad, dev)
        St = S.T if adjoint else S
        if card == "left":
            rla.mul_(Cd, St, Ad, alpha, beta)
            (orc.mul_StA if adjoint else orc.mul_SA)(ref, R, A.astype(np.float64), alpha, beta)
        else:
            rla.mul_(Cd, Ad, St, alpha, beta)
            (orc.mul_ASt if adjoint else orc.mul_AS)(ref, A.astype(np.float64), R, alpha, beta)
        err = rel_err(Cd.cpu().numpy(), ref)
        assert err < TOL[dtype], (L, s, nv, err)
