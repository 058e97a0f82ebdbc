"""SRHT of short columns (512 to 4096 padded) over both of its kernels, a CTA per column and several
columns per CTA (csrc/rla_wht.cu): few and many samples, up to every row of the padded column, sizes
below and above the rule between them, both directions and layouts, alpha and beta, against the FP64
oracle on the same draws.  test_host_routes.py checks which kernel each size runs.

Tolerance: a transform of N <= 4096 values adds in at most 12 levels after an expand's sum of the
samples of one position (one each here): an error of about sqrt(12) * 2^-25 = 1e-7 of the column norm
in Float32; TOL is 1e-6 (Float32) and 1e-12 (Float64)."""
import numpy as np
import pytest

from helpers import TOL, oracle_recipe, rel_err
from test_gpu_sparse_tile import column_major

pytestmark = pytest.mark.gpu

#        L, s, nv
SHORT = [(700, 1000, 3), (1000, 800, 40), (1024, 1024, 17), (1000, 100, 200), (2047, 2000, 40), (1500, 300, 30),
         (4000, 4000, 20), (4096, 4096, 5), (3000, 300, 9), (2500, 1, 2)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("card", ["left", "right"])
@pytest.mark.parametrize("adjoint", [False, True])
def test_short_columns(rla, orc, dev, dtype, card, adjoint):
    for L, s, nv in SHORT:
        rng = np.random.default_rng([L, s, nv])
        cd = rla.Left() if card == "left" else rla.Right()
        long_, short = ((L, nv), (s, nv)) if card == "left" else ((nv, L), (nv, s))
        A = rng.standard_normal(short if adjoint else long_).astype(dtype)
        C = rng.standard_normal(long_ if adjoint else short).astype(dtype)
        S = rla.complete_compressor(rla.SRHT(cardinality=cd, compression_dim=s, type=dtype), np.zeros(long_, dtype), seed=4)
        St = S.T if adjoint else S
        for pad, alpha, beta in [(0, 1.0, 0.0), (1, 0.5, -2.0)]:
            ref = C.astype(np.float64).copy(order="F")
            Ad, Cd = column_major(A, pad, dev), column_major(C, pad, dev)
            if card == "left":
                rla.mul_(Cd, St, Ad, alpha, beta)
                (orc.mul_StA if adjoint else orc.mul_SA)(ref, oracle_recipe(orc, S), A.astype(np.float64), alpha, beta)
            else:
                rla.mul_(Cd, Ad, St, alpha, beta)
                (orc.mul_ASt if adjoint else orc.mul_AS)(ref, A.astype(np.float64), oracle_recipe(orc, S), alpha, beta)
            err = rel_err(Cd.cpu().numpy(), ref)
            assert err < TOL[dtype], (L, s, nv, pad, err)
