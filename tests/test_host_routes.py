"""Which kernels a call launches, on a fake CUDA runtime (fake_cuda.py; CPU only).  Each table holds
sizes on both sides of a rule; the times stand beside the rules in the sources."""
import re

import pytest

import test_gpu_sparse_lift_sizes as lift
import test_gpu_sparse_tile_windows as windows
import test_gpu_presplit as presplit
import test_gpu_srht_short as srht_short
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


#        L, s, nnz, nv, dtype, row_major, kernel
EXPANDS = [
    # column-major results: few vectors, unrolled and general entry counts
    (1 << 20, 512, 8, 1, F32, False, "expand_kernel"), (1 << 20, 512, 8, 3, F32, False, "expand_kernel"),
    (1 << 20, 512, 8, 4, F32, False, "lift_kernelIfLi8ELi8E"), (1 << 20, 100, 1, 7, F32, False, "expand_kernel"),
    (1 << 20, 100, 1, 8, F32, False, "lift_kernelIfLi8ELi1E"), (1 << 20, 500, 3, 15, F64, False, "expand_kernel"),
    (1 << 20, 500, 3, 16, F64, False, "lift_kernelIdLi8ELi0E"),
    # not enough outputs for the staging
    (4096, 1000, 8, 64, F32, False, "expand_kernel"), (30000, 1000, 8, 16, F32, False, "expand_kernel"),
    (30000, 1000, 8, 64, F32, False, "lift_kernelIfLi8ELi8E"), (4096, 64, 1, 200, F32, False, "expand_kernel"),
    (4096, 64, 1, 1000, F32, False, "lift_kernelIfLi8ELi1E"),
    # narrower staged rows and the last one that fits
    (131072, 1095, 8, 200, F32, False, "lift_kernelIfLi8ELi8E"), (131072, 1096, 8, 200, F32, False, "lift_kernelIfLi4ELi8E"),
    (131072, 2380, 8, 200, F64, False, "lift_kernelIdLi4ELi8E"), (131072, 2381, 8, 200, F64, False, "lift_kernelIdLi2ELi8E"),
    (131072, 4309, 8, 200, F64, False, "lift_kernelIdLi2ELi8E"), (131072, 4310, 8, 200, F64, False, "expand_kernel"),
    (1 << 20, 4000, 3, 64, F64, False, "expand_kernel"), (131072, 4000, 3, 200, F64, False, "lift_kernelIdLi2ELi0E"),
    # row-major results
    (1 << 20, 64, 2, 1, F32, True, "expand_kernel"), (1 << 20, 64, 2, 2, F32, True, "lift_kernelIfLi8ELi2E"),
    (30000, 1000, 8, 32, F32, True, "expand_kernel"), (30000, 1000, 8, 1000, F32, True, "lift_kernelIfLi8ELi8E"),
    (4096, 64, 4, 64, F32, True, "expand_kernel"), (1 << 20, 4000, 1, 64, F64, True, "expand_kernel"),
    (1 << 20, 4000, 1, 32, F64, True, "lift_kernelIdLi2ELi1E"), (1 << 20, 4000, 8, 64, F64, True, "lift_kernelIdLi2ELi8E"),
]


@pytest.mark.parametrize("case", EXPANDS)
def test_expand_routes(fake, case):
    L, s, nnz, nv, dtype, row_major, kernel = case
    ctx = fake.context()
    sk = fake.sketch(ctx, "sparse_sign", s, L, dtype=dtype, nnz=nnz)
    fake.reset()
    assert fake.mul(ctx, sk, (s, L, nv), LEFT, adjoint=True, row_a=row_major, row_c=row_major) == 0
    launched = fake.launches()
    assert len(launched) == 1 and kernel in launched[0], launched


@pytest.mark.parametrize("card", [LEFT, RIGHT])
@pytest.mark.parametrize("dtype", [F32, F64])
def test_lift_sizes_reach_the_staged_kernel(fake, dtype, card):
    """Every size of test_gpu_sparse_lift_sizes.py, in each of its layouts."""
    ctx = fake.context()
    for layout, (row_y, row_c, pad, _, beta) in lift.LAYOUTS.items():
        for L, s, nnz, nv, lanes in lift.sizes(layout):
            sk = fake.sketch(ctx, "sparse_sign", s, L, card=card, dtype=dtype, nnz=nnz)
            fake.reset()
            rows = (row_y, row_c) if card == LEFT else (not row_y, not row_c)
            assert fake.mul(ctx, sk, (s, L, nv), card, True, *rows, beta=beta, pad=pad) == 0
            fixed = nnz if nnz in (1, 2, 4, 8) else 0
            name = "lift_kernelI%sLi%dELi%dE" % ("f" if dtype == F32 else "d", lanes, fixed)
            assert len(fake.launches()) == 1 and name in fake.launches()[0], (layout, L, s, nnz, nv, fake.launches())
            fake.lib.rla_sketch_destroy(sk)


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("L", [600, 1000, 5003, 16384, 100003])
def test_fjlt_expand_gathers_with_one_thread_per_element(fake, dtype, L):
    """The rows of the transposed sampling matrix differ in length and a short transform has few CTAs:
    S' * Y gathers into the workspace first, then transforms it."""
    ctx = fake.context()
    nv = 64
    sk = fake.sketch(ctx, "fjlt", 300, L, dtype=dtype)
    fake.reset()
    assert fake.mul(ctx, sk, (300, L, nv), LEFT, adjoint=True) == 0
    padded = 1 << (L - 1).bit_length()
    (x, _, threads), = grids(fake.log(), "csr_t_gather")
    assert x * threads >= min(padded * nv, 148 * 32 * 256)
    assert fake.launches()[0].find("csr_t_gather") > 0


@pytest.mark.parametrize("dtype,direct,staged", [(F32, 16, 17), (F64, 12, 13)])
def test_srht_expand_writes_few_row_major_vectors_directly(fake, dtype, direct, staged):
    """Tiles of 32 vectors that are mostly empty cost more than uncoalesced writes of a few vectors."""
    ctx = fake.context()
    L, s = 1 << 20, 100
    sk = fake.sketch(ctx, "srht", s, L, dtype=dtype)
    for nv in (2, direct, staged, 64):
        fake.reset()
        assert fake.mul(ctx, sk, (s, L, nv), LEFT, adjoint=True, row_c=True) == 0
        assert any("fjlt_expand_out" in k for k in fake.launches()) == (nv >= staged), nv


#       s, L, nv, tiles of 128 x 64, splits of K
GAUSS_SPLITS = [(64, 16384, 100, 1, 64), (200, 16384, 260, 10, 13), (250, 60000, 260, 10, 14), (100, 16384, 100, 2, 64),
                (64, 4096, 9600, 75, 3), (64, 4096, 9472, 74, 2), (64, 4096, 18944, 148, 1), (244, 11234, 2778, 88, 5),
                (130, 258299, 120, 3, 49), (64, 256, 9600, 75, 1), (256, 4096, 60000, 1876, 1)]


@pytest.mark.parametrize("case", GAUSS_SPLITS)
def test_gaussian_k_splits_fill_whole_rounds(fake, case):
    """The K splits of a Gaussian product leave no round of CTAs nearly empty."""
    s, L, nv, tiles, splits = case
    ctx = fake.context()
    sk = fake.sketch(ctx, "gaussian", s, L)
    fake.reset()
    assert fake.mul(ctx, sk, (s, L, nv), LEFT) == 0
    (x, y, _), = grids(fake.log(), "conv_gemm")
    assert (x, y) == (tiles, splits)
    rounds = lambda n: -(-tiles * n // 148) / n
    assert splits == 1 or rounds(splits) <= min(rounds(splits - 1), rounds(splits + 1)) * 1.1


@pytest.mark.parametrize("case", [(64, 4096, 9600, 1), (244, 11234, 2778, 1), (64, 4096, 9472, 2)])
def test_gaussian_takes_no_more_scratch_in_a_capture_than_one_round(fake, case):
    s, L, nv, splits = case
    ctx = fake.context()
    sk = fake.sketch(ctx, "gaussian", s, L)
    assert fake.mul(ctx, sk, (s, L, nv), LEFT) == 0
    fake.reset()
    fake.capturing(True)
    assert fake.mul(ctx, sk, (s, L, nv), LEFT, wait=False) == 0
    (_, y, _), = grids(fake.log(), "conv_gemm")
    assert y == splits


@pytest.mark.parametrize("s,nv", [(100, 100), (64, 100), (33, 7)])
def test_gaussian_split_sums_have_a_thread_per_element(fake, s, nv):
    ctx = fake.context()
    sk = fake.sketch(ctx, "gaussian", s, 16384)
    fake.reset()
    assert fake.mul(ctx, sk, (s, 16384, nv), LEFT) == 0
    (x, y, threads), = grids(fake.log(), "conv_reduce")
    assert x * y * threads >= s * nv


#       L, s, nnz, nv, dtype: calls whose (tile, window)s are cut between CTAs
CUTS = [(100000, 500, 8, 500, F32), (10000, 8320, 2, 3000, F32), (150001, 1332, 8, 333, F32),
        (100000, 6240, 3, 16, F64)]


@pytest.mark.parametrize("case", CUTS)
def test_tile_reduction_covers_the_cut_tiles_only(fake, case):
    """At most W - 1 (tile, window)s are cut by the borders of W workers, whatever their number is."""
    L, s, nnz, nv, dtype = case
    ctx = fake.context()
    sk = fake.sketch(ctx, "sparse_sign", s, L, dtype=dtype, nnz=nnz)
    fake.reset()
    assert fake.mul(ctx, sk, (s, L, nv), LEFT) == 0
    (w, _, _), = grids(fake.log(), "tile_compress")
    (x, y, threads), = grids(fake.log(), "tile_reduce")
    tiles = -(-nv // (32 if dtype == F32 else 16)) * -(-s // 1040)
    assert x == min(tiles, w - 1)


@pytest.mark.parametrize("case", [(1000, 1000, 2, 3000, F32), (640, 40, 8, 100000, F32), (1000, 1000, 3, 10000, F64)])
def test_short_tiles_are_not_cut(fake, case):
    """With a chunk or two per tile a CTA takes whole tiles: the partial sums would take longer."""
    L, s, nnz, nv, dtype = case
    ctx = fake.context()
    sk = fake.sketch(ctx, "sparse_sign", s, L, dtype=dtype, nnz=nnz)
    fake.reset()
    assert fake.mul(ctx, sk, (s, L, nv), LEFT) == 0
    assert len(fake.launches()) == 1 and "tile_compress" in fake.launches()[0]


#       L, s, nv, dtype, expand: a CTA per column, compress: a CTA per column
SRHT_SHORT = [(1000, 800, 40, F32, True, True), (1000, 300, 128, F32, True, False), (1000, 800, 4000, F32, False, False),
              (1000, 10, 128, F32, False, False), (2000, 2000, 64, F32, True, False), (2000, 300, 128, F32, False, False),
              (2000, 2000, 2000, F32, False, False), (4000, 4000, 64, F32, True, False), (4000, 4000, 2000, F32, False, False),
              (4000, 300, 8, F32, False, False), (8000, 4000, 8, F32, False, False), (500, 400, 5000, F32, True, True),
              (1000, 800, 128, F64, True, False), (2000, 2000, 128, F64, True, False), (4000, 2000, 128, F64, False, False)]


@pytest.mark.parametrize("case", SRHT_SHORT)
def test_srht_short_columns(fake, case):
    """A few short columns with many samples have a CTA each; otherwise several share one."""
    L, s, nv, dtype, expand, compress = case
    ctx = fake.context()
    sk = fake.sketch(ctx, "srht", s, L, dtype=dtype)
    for adjoint, column in ((True, expand), (False, compress)):
        fake.reset()
        assert fake.mul(ctx, sk, (s, L, nv), LEFT, adjoint=adjoint) == 0
        kernel = ("srht_expand_kernel" if adjoint else "srht_small_kernel") if column else "wht_near_kernel"
        assert len(fake.launches()) == 1 and kernel in fake.launches()[0], (adjoint, fake.launches())


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("adjoint", [False, True])
def test_srht_short_gpu_sizes_run_both_kernels(fake, dtype, adjoint):
    ctx = fake.context()
    seen = set()
    for L, s, nv in srht_short.SHORT:
        for card in (LEFT, RIGHT):
            sk = fake.sketch(ctx, "srht", s, L, dtype=dtype, card=card)
            fake.reset()
            assert fake.mul(ctx, sk, (s, L, nv), card, adjoint=adjoint) == 0
            seen.update(name for name in ("near", "srht_expand", "srht_small") for k in fake.launches() if name in k)
    assert seen == {"near", "srht_expand" if adjoint else "srht_small"}


@pytest.mark.parametrize("nnz,s,ctas", [(1, 1000, 8), (2, 1000, 7), (1, 4096, 4), (1, 8320, 4), (2, 8320, 4), (8, 8320, 2)])
def test_tile_plans_of_many_buckets_leave_room_for_several_ctas(fake, nnz, s, ctas):
    """The counters of the plan's ranking warps bound the CTAs per SM (228 KB of shared memory)."""
    ctx = fake.context()
    fake.reset()
    fake.sketch(ctx, "count_sketch" if nnz == 1 else "sparse_sign", s, 1 << 17, card=RIGHT, nnz=nnz)
    smem, = [int(re.search(r"smem=(\d+)", ln).group(1)) for ln in fake.log() if "bl_build" in ln]
    assert 228 * 1024 // (smem + 3072) >= ctas


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("card", [LEFT, RIGHT])
@pytest.mark.parametrize("row_major", [False, True])
def test_window_sizes_run_the_tile_kernel_up_to_its_limits(fake, dtype, card, row_major):
    ctx = fake.context()
    for L, s, nnz, nv in windows.WINDOWS:
        sk = fake.sketch(ctx, "count_sketch" if nnz == 1 else "sparse_sign", s, L, card=card, dtype=dtype, nnz=nnz)
        fake.reset()
        assert fake.mul(ctx, sk, (s, L, nv), card, row_a=row_major, row_c=row_major) == 0
        strided = (card == LEFT) == row_major
        tile = s <= 8320 and nnz <= 32 and (nnz > 1 or s <= 2080 or (card == RIGHT and strided))
        assert ("tile_compress" in fake.launches()[0]) == tile, (L, s, nnz, nv, fake.launches())
        fake.lib.rla_sketch_destroy(sk)


#      L, s, nnz, nv, dtype, row-major Y, row-major C, leading dimension + , beta, staged
EXPAND_COSTS = [
    # row-major results: a column-major operand is read across by the kernel with a thread per output
    (8000, 1000, 16, 500, F32, False, True, 0, 0.0, True), (1000, 1000, 8, 3000, F32, False, True, 0, 0.0, True),
    (1030, 840, 16, 3863, F32, False, True, 1, 0.0, True), (27284, 3088, 16, 346, F64, False, True, 0, 0.0, True),
    (8000, 1000, 3, 32, F32, False, True, 0, 0.0, False),
    # rows off 32-byte boundaries, results beyond L2
    (30000, 2000, 1, 1000, F64, True, True, 1, 0.0, False), (30000, 1000, 3, 1000, F64, True, True, 1, 0.0, False),
    (30000, 300, 8, 1000, F64, True, True, 1, 0.0, True), (30000, 1, 1, 1000, F64, False, True, 1, 0.0, False),
    (30000, 2000, 1, 1000, F64, True, True, 0, 0.0, True),
    # short columns
    (50, 50, 3, 100000, F64, False, False, 0, 0.0, False), (50, 10, 3, 100000, F32, False, False, 0, 0.0, False),
    (200, 50, 8, 40000, F64, False, False, 0, 0.0, True), (155, 12, 12, 49361, F64, True, False, 0, 0.0, True),
    # old values of the result
    (3683, 23, 2, 181, F32, True, True, 0, 0.5, False), (1599, 18, 1, 848, F32, True, True, 0, 0.5, False),
    (1000481, 3, 3, 22, F64, True, False, 1, 0.5, False), (4239, 90, 12, 179, F32, False, False, 0, 0.5, False),
    (131072, 1000, 8, 200, F64, False, False, 0, 0.5, True), (29150, 3884, 2, 1119, F64, False, True, 1, 0.5, False),
    (229508, 3223, 1, 198, F64, False, False, 0, 0.5, False), (229508, 3223, 1, 198, F64, False, False, 0, 0.0, True),
]


@pytest.mark.parametrize("case", EXPAND_COSTS)
def test_expand_cost_rules(fake, case):
    L, s, nnz, nv, dtype, row_y, row_c, pad, beta, staged = case
    ctx = fake.context()
    sk = fake.sketch(ctx, "sparse_sign", s, L, dtype=dtype, nnz=nnz)
    fake.reset()
    assert fake.mul(ctx, sk, (s, L, nv), LEFT, adjoint=True, row_a=row_y, row_c=row_c, pad=pad, beta=beta) == 0
    assert len(fake.launches()) == 1 and ("lift_kernel" in fake.launches()[0]) == staged, fake.launches()


@pytest.mark.parametrize("L,ahead", [(600, True), (10240, True), (10241, False), (150001, False)])
def test_tiles_of_few_chunks_read_old_values_ahead(fake, L, ahead):
    """With beta a short tile reads four old values per thread before it writes; the registers would slow
    down the sums of a long one, and there is nothing to read without beta."""
    ctx = fake.context()
    sk = fake.sketch(ctx, "sparse_sign", 300, L, nnz=4)
    for beta in (0.0, 0.5):
        fake.reset()
        assert fake.mul(ctx, sk, (300, L, 40), LEFT, beta=beta) == 0
        assert ("ELi4EEEvNS_10TileParams" in fake.launches()[0]) == (ahead and beta != 0), fake.launches()


@pytest.mark.parametrize("kind,s,L", [("srht", 5610, 22574), ("fjlt", 40, 5000), ("fjlt", 40, 60000)])
def test_transforms_with_beta_read_old_values_ahead(fake, kind, s, L):
    ctx = fake.context()
    sk = fake.sketch(ctx, kind, s, L)
    for beta in (0.0, 0.5):
        fake.reset()
        assert fake.mul(ctx, sk, (s, L, 6), LEFT, adjoint=True, beta=beta) == 0
        assert ("ELi2EEEvNS_9WhtParams" in fake.launches()[-1] or "ELi2EEEvNS_9WhtParamsIT_EEi" in fake.launches()[-1]) == (beta != 0)


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("card", [LEFT, RIGHT])
def test_presplit_sizes_are_split_beforehand(fake, card, adjoint):
    """Both result dimensions and the inner one above 256: the operands are split in memory."""
    ctx = fake.context()
    other = 0
    for L, s, nv in presplit.SPLITS + [(256, 300, 300), (300, 256, 300), (300, 300, 256)]:
        sk = fake.sketch(ctx, "gaussian", s, L, card=card)
        fake.reset()
        assert fake.mul(ctx, sk, (s, L, nv), card, adjoint=adjoint) == 0
        before = min(s, L, nv) > 256
        assert any("tc_gemm_f64acc" in k for k in fake.launches()) == before, (L, s, nv, fake.launches())
        other += any("conv_gemm" in k for k in fake.launches())
        fake.lib.rla_sketch_destroy(sk)
    assert other == 3


@pytest.mark.parametrize("dtype", [F32, F64])
def test_expand_of_one_strided_vector_has_threads_along_it(fake, dtype):
    ctx = fake.context()
    L, s = 551399, 6
    sk = fake.sketch(ctx, "sparse_sign", s, L, card=RIGHT, dtype=dtype, nnz=4)
    fake.reset()
    assert fake.mul(ctx, sk, (s, L, 1), RIGHT, adjoint=True, pad=1) == 0  # a row of a column-major result
    (x, y, threads), = grids(fake.log(), "expand_kernel")
    assert x * y * threads < 3 * L


#       L, s, nv, row-major Y, turned
SRHT_TURNED = [(44736, 6810, 820, True, True), (1 << 18, 4096, 100, True, True), (44736, 6810, 820, False, False),
               (16000, 4096, 820, True, False), (1 << 18, 40, 100, True, False), (44736, 6810, 1, True, False)]


@pytest.mark.parametrize("row_c", [False, True])
@pytest.mark.parametrize("case", SRHT_TURNED)
def test_srht_expand_turns_row_major_samples(fake, case, row_c):
    """Every chunk of a long column gathers all samples: rows are turned into columns once, but not in
    a graph capture, which would keep the scratch."""
    L, s, nv, row_y, turned = case
    ctx = fake.context()
    sk = fake.sketch(ctx, "srht", s, L)
    for capturing in (False, True):
        fake.reset()
        fake.capturing(capturing)
        assert fake.mul(ctx, sk, (s, L, nv), LEFT, adjoint=True, row_a=row_y, row_c=row_c, wait=False) == 0
        assert ("gather_columns" in fake.launches()[0]) == (turned and not capturing), fake.launches()
