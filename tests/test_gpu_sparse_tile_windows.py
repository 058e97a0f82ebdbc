"""SparseSign / CountSketch compress at the limits of the tile kernel and of its plan
(csrc/rla_sparse_tile.cu): one chunk of 640 long indices, its neighbours and two chunks; the last s
of one, two and eight bucket windows (1040 buckets each) and the first beyond, where other kernels
take over above 8320 buckets or 32 entries per long index; both types, sides and layouts, against the
FP64 oracle on the same draws.  test_host_routes.py checks which kernel each size runs.

Tolerance: a bucket sums L * nnz / s terms, at most 4000 here in one or two runs: an error of about
sqrt(4000) * 2^-25 of their norm in Float32, below TOL = 1e-6 in the Frobenius norm; Float64 scales by
2^-29 (TOL = 1e-12)."""
import numpy as np
import pytest

from helpers import TOL, oracle_recipe, rel_err
from test_gpu_sparse_tile import column_major

pytestmark = pytest.mark.gpu

#          L, s, nnz, nv
WINDOWS = [(639, 1040, 8, 33), (640, 1041, 2, 32), (641, 2080, 8, 17), (1279, 2081, 3, 31), (1280, 3120, 2, 16),
           (1281, 3121, 4, 5), (1500, 4160, 1, 40), (1500, 6240, 1, 33), (700, 6241, 2, 9), (2000, 8320, 1, 33), (1300, 8320, 2, 20),
           (1281, 8320, 8, 33), (660, 8320, 32, 7), (900, 8321, 2, 12), (900, 8321, 1, 12), (1000, 32, 32, 33), (1000, 40, 33, 33),
           (4000, 36, 32, 70)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("card", ["left", "right"])
@pytest.mark.parametrize("row_major", [False, True])
def test_windows(rla, orc, dev, dtype, card, row_major):
    import torch
    for L, s, nnz, nv in WINDOWS:
        rng = np.random.default_rng([L, s, nnz, nv])
        cd = rla.Left() if card == "left" else rla.Right()
        comp = (rla.CountSketch(cardinality=cd, compression_dim=s, type=dtype) if nnz == 1
                else rla.SparseSign(cardinality=cd, compression_dim=s, nnz=nnz, type=dtype))
        A = rng.standard_normal((L, nv) if card == "left" else (nv, L)).astype(dtype)
        C = rng.standard_normal((s, nv) if card == "left" else (nv, s)).astype(dtype)
        S = rla.complete_compressor(comp, A, seed=5)
        ref = C.astype(np.float64).copy(order="F")
        put = (lambda x: torch.from_numpy(x.copy()).to(dev)) if row_major else (lambda x: column_major(x, 1, dev))
        Ad, Cd = put(A), put(C)
        if card == "left":
            rla.mul_(Cd, S, Ad, 0.5, -2.0)
            orc.mul_SA(ref, oracle_recipe(orc, S), A.astype(np.float64), 0.5, -2.0)
        else:
            rla.mul_(Cd, Ad, S, 0.5, -2.0)
            orc.mul_AS(ref, A.astype(np.float64), oracle_recipe(orc, S), 0.5, -2.0)
        err = rel_err(Cd.cpu().numpy(), ref)
        assert err < TOL[dtype], (L, s, nnz, nv, err)
