"""SparseSign / CountSketch expand at sizes that run the staged kernel (csrc/rla_sparse_lift.cu): 8, 4 and 2
lanes per entry up to their last s, the unrolled entry counts and general ones up to 32, partial
blocks of 32 long indices and partial vector tiles, column-major results with vector stores, with odd
leading dimensions and with beta, row-major and mixed layouts, against the FP64 oracle on the same
draws.  test_host_routes.py checks, without a GPU, that every size here launches that kernel.

Tolerance: at most nnz = 32 terms per output added in sequence: the error is below 32 * 2^-24 of the
sum of magnitudes at worst, and for random data about sqrt(32) * 2^-24 / 2 = 1.7e-7 of the
result in the Frobenius norm; TOL is 1e-6 (Float32) and 1e-12 (Float64)."""
import numpy as np
import pytest

from helpers import TOL, oracle_recipe, rel_err
from test_gpu_sparse_tile import column_major

pytestmark = pytest.mark.gpu

#        L, s, nnz, nv, lanes per entry
SIZES = [(60011, 40, 8, 37, 8), (120011, 1095, 1, 33, 8), (60021, 300, 3, 50, 8), (40001, 64, 16, 21, 8),
         (30007, 64, 32, 19, 8), (120027, 1200, 2, 61, 4), (40009, 2380, 8, 131, 4), (120007, 3000, 4, 29, 2),
         (124003, 4309, 8, 40, 2), (126001, 3000, 3, 30, 2)]
#          row-major Y, row-major C, padding, alpha, beta
LAYOUTS = {"col": (False, False, 0, 1.0, 0.0), "col_odd": (False, False, 1, 0.5, 0.0), "col_beta": (False, False, 1, 0.5, -2.0), "row": (True, True, 0, 1.0, 0.0),
           "row_beta": (True, True, 0, 0.5, -2.0), "row_to_col": (True, False, 0, 1.0, 0.0),
           "col_to_row": (False, True, 0, 1.0, 0.0)}


def sizes(layout):
    """The sizes of a layout: staging a row-major Y for a column-major result pays later, with beta only for
    four entries and more."""
    return [z for z in SIZES if (layout != "row_to_col" or z[1] * z[4] <= 2400) and (layout != "col_beta" or z[2] >= 4)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("card", ["left", "right"])
def test_lift_sizes(rla, orc, dev, dtype, layout, card):
    import torch
    row_y, row_c, pad, alpha, beta = LAYOUTS[layout]
    for i, (L, s, nnz, nv, _) in enumerate(sizes(layout)):
        if (i % 2 == 0) != (card == "left"):  # half the sizes on each side
            continue
        rng = np.random.default_rng([L, s, nnz, nv])
        cd = rla.Left() if card == "left" else rla.Right()
        comp = rla.SparseSign(cardinality=cd, compression_dim=s, nnz=nnz, type=dtype)
        long_shape, short = ((L, nv), (s, nv)) if card == "left" else ((nv, L), (nv, s))
        Y = rng.standard_normal(short).astype(dtype)
        C = rng.standard_normal(long_shape).astype(dtype)
        S = rla.complete_compressor(comp, np.zeros(long_shape, dtype), seed=6)
        R = oracle_recipe(orc, S)
        put = lambda x, row: torch.from_numpy(x.copy()).to(dev) if row else column_major(x, pad, dev)
        # a column of a Right operand is a row-major vector: the layouts are those of the vectors
        Yd, Cd = (put(Y, row_y), put(C, row_c)) if card == "left" else (put(Y, not row_y), put(C, not row_c))
        ref = C.astype(np.float64).copy(order="F")
        if card == "left":
            rla.mul_(Cd, S.T, Yd, alpha, beta)
            orc.mul_StA(ref, R, Y.astype(np.float64), alpha, beta)
        else:
            rla.mul_(Cd, Yd, S.T, alpha, beta)
            orc.mul_ASt(ref, Y.astype(np.float64), R, alpha, beta)
        err = rel_err(Cd.cpu().numpy(), ref)
        assert err < TOL[dtype], (L, s, nnz, nv, err)
