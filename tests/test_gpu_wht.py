"""Walsh-Hadamard sketches over the edges of the transform kernels (csrc/rla_wht.cu): the
shortest column of the chunked kernel (1024 Float32 / 512 Float64), several short columns in
one chunk, the chunk length itself (16384 / 8192), one, four and six bits above it (one and two
passes over the workspace), aligned and odd leading dimensions, both layouts of the operand
and of the result, against the FP64 oracle on the same draws.

Tolerance: a transform of N values adds in log2 N <= 20 levels, so its error is below
log2(N) * 2^-24 of the column norm (1.2e-6 at worst, about sqrt(20) * 2^-25 = 1.3e-7 for random
data); TOL is 1e-6 (Float32) and 1e-12 (Float64)."""
import numpy as np
import pytest

from helpers import TOL, oracle_recipe, rel_err
from test_gpu_sparse_tile import column_major

pytestmark = pytest.mark.gpu

#       L, s, nv
SIZES = [(511, 40, 3), (513, 60, 5), (1000, 100, 17), (1025, 33, 9), (3000, 200, 6), (8192, 300, 3), (8193, 300, 2),
         (16384, 500, 3), (16390, 300, 3), (100003, 200, 5), (262145, 300, 2), (600001, 400, 2)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["srht", "fjlt"])
@pytest.mark.parametrize("card", ["left", "right"])
@pytest.mark.parametrize("adjoint", [False, True])
def test_transform_edges(rla, orc, dev, dtype, kind, card, adjoint):
    for L, s, nv in SIZES:
        rng = np.random.default_rng([L, s, nv])
        cd = rla.Left() if card == "left" else rla.Right()
        comp = (rla.SRHT if kind == "srht" else rla.FJLT)(cardinality=cd, compression_dim=s, type=dtype)
        long_, short = ((L, nv), (s, nv)) if card == "left" else ((nv, L), (nv, s))
        A = rng.standard_normal(short if adjoint else long_).astype(dtype)
        C = rng.standard_normal(long_ if adjoint else short).astype(dtype)
        S = rla.complete_compressor(comp, np.zeros(long_, dtype), seed=4)
        R = oracle_recipe(orc, S)
        for pad, alpha, beta in [(0, 1.0, 0.0), (1, 0.5, -2.0)]:
            ref = C.astype(np.float64).copy(order="F")
            Ad, Cd = column_major(A, pad, dev), column_major(C, pad, dev)
            A64 = A.astype(np.float64)
            St = S.T if adjoint else S
            if card == "left":
                rla.mul_(Cd, St, Ad, alpha, beta)
                (orc.mul_StA if adjoint else orc.mul_SA)(ref, R, A64, alpha, beta)
            else:
                rla.mul_(Cd, Ad, St, alpha, beta)
                (orc.mul_ASt if adjoint else orc.mul_AS)(ref, A64, R, alpha, beta)
            err = rel_err(Cd.cpu().numpy(), ref)
            assert err < TOL[dtype], (L, s, nv, pad, err)


def test_workspace_batches(rla, orc, dev):
    """More columns than one 64 MB workspace batch holds (2^17 Float64 columns: 64 per batch)."""
    rng = np.random.default_rng(3)
    L, s, nv = 70001, 50, 70
    A = rng.standard_normal((L, nv))
    S = rla.complete_compressor(rla.FJLT(compression_dim=s, type=np.float64), A, seed=4)
    ref = np.zeros((s, nv), order="F")
    orc.mul_SA(ref, oracle_recipe(orc, S), A)
    assert rel_err((S @ column_major(A, 0, dev)).cpu().numpy(), ref) < TOL[np.float64]
    Y = rng.standard_normal((s, nv))
    back = np.zeros((L, nv), order="F")
    orc.mul_StA(back, oracle_recipe(orc, S), Y)
    assert rel_err((S.T @ column_major(Y, 0, dev)).cpu().numpy(), back) < TOL[np.float64]
