"""Which kernels a call launches, on a fake CUDA runtime (fake_cuda.py; CPU only).  Each table holds
sizes on both sides of a rule; the times stand beside the rules in the sources."""
import re

import pytest

from fake_cuda import F32, F64, LEFT, RIGHT, fake  # noqa: F401 (fixture)


def grids(log, kernel):
    """(x, y, threads) of the kernel's launches."""
    out = []
    for line in log:
        m = re.match(r"launch \S*%s\S* grid=(\d+),(\d+),\d+ block=(\d+)" % kernel, line)
        if m:
            out.append(tuple(int(g) for g in m.groups()))
    return out


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("s", [100, 2048])
def test_partial_sums_of_one_tile_are_spread(fake, dtype, s):
    """A few vectors make one tile, whose partial sums come from every SM: a thread adds those of one
    element only."""
    ctx = fake.context()
    sk = fake.sketch(ctx, "sparse_sign", s, 1 << 17, dtype=dtype, nnz=2)
    fake.reset()
    assert fake.mul(ctx, sk, (s, 1 << 17, 1), LEFT) == 0
    (x, y, threads), = grids(fake.log(), "tile_reduce")
    windows = -(-s // 1040)
    assert x * y * threads >= s * (32 if dtype == F32 else 16) and x == windows
