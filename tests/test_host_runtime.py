"""Order of the library's host calls, on a fake CUDA runtime (fake_cuda.py; CPU only): device memory
that outlives a call comes from a pool shared by all contexts of a device, so it may be given back
only when no queued work can still touch it."""
import ctypes

import pytest

from fake_cuda import F32, F64, LEFT, RIGHT, fake, i64, vp  # noqa: F401 (fixture)

IHS, KACZMARZ, COLUMN = "ihs", 0, 1


def freed_while_queued(log):
    """Releases that are not ordered behind work queued before them: freed on the legacy stream (or
    with cudaFree, which does not wait for pool memory) with no wait for the stream since that work."""
    pending, bad = set(), []
    for line in log:
        call, *rest = line.split()
        stream = next((r[7:] for r in rest if r.startswith("stream=")), None)
        if call == "launch" or call in ("cudaMemsetAsync", "cudaMemcpyAsync"):
            pending.add(stream)
        elif call == "cudaStreamSynchronize":
            pending.discard(stream)
        elif call == "cudaDeviceSynchronize":
            pending.clear()
        elif call == "cudaFree" or (call == "cudaFreeAsync" and stream == "(nil)"):
            if pending:
                bad.append(line)
    return bad


def test_check_sees_a_planted_release():
    log = ["launch k grid=1 stream=0x10", "cudaFreeAsync 0x5 stream=(nil)"]
    assert freed_while_queued(log) == log[1:]
    assert freed_while_queued([log[0], "cudaStreamSynchronize stream=0x10", log[1]]) == []
    assert freed_while_queued([log[0], "cudaStreamSynchronize stream=0x20", log[1]]) == log[1:]
    assert freed_while_queued([log[0], "cudaFreeAsync 0x5 stream=0x10"]) == []


@pytest.mark.parametrize("kind,nnz", [("sparse_sign", 8), ("count_sketch", 1), ("srht", 1), ("fjlt", 1), ("gaussian", 1)])
@pytest.mark.parametrize("call", ["cudaMallocFromPoolAsync", "cudaMallocAsync", "launch"])
def test_failed_sketch_creation_waits_for_its_draws(fake, kind, nnz, call):
    """Whatever call of the creation fails, the buffers go back after the work queued on them."""
    ctx = fake.context()
    failed = 0
    for ok in range(12):
        fake.reset()
        fake.fail_after(call, ok)
        rc, sk = fake.create(ctx, kind, 40, 3000, nnz=nnz, card=RIGHT)
        if rc:
            failed += 1
            assert freed_while_queued(fake.log()) == [], (call, ok)
        else:
            fake.lib.rla_sketch_destroy(sk)
    assert failed or call == "cudaMallocAsync"
    fake.lib.rla_ctx_destroy(ctx)


@pytest.mark.parametrize("solver", [IHS, KACZMARZ, COLUMN])
@pytest.mark.parametrize("call", ["cudaMallocFromPoolAsync", "cudaMemsetAsync", "cudaEventCreateWithFlags",
                                  "cudaStreamCreateWithFlags"])
def test_failed_solver_creation_waits_for_its_memsets(fake, solver, call):
    ctx = fake.context()
    sk = fake.sketch(ctx, "sparse_sign", 64, 500 if solver != COLUMN else 20, nnz=4, card=LEFT if solver != COLUMN else RIGHT)
    failed = 0
    for ok in range(14):
        fake.reset()
        fake.fail_after(call, ok)
        h = vp()
        if solver == IHS:
            rc = fake.lib.rla_ihs_create(ctx, sk, F32, i64(500), i64(20), ctypes.c_double(1.0), ctypes.byref(h))
        else:
            rc = fake.lib.rla_proj_create(ctx, sk, solver, F32, i64(500), i64(20), ctypes.c_double(1.0),
                                          ctypes.byref(h))
        if rc:
            failed += 1
            assert freed_while_queued(fake.log()) == [], (call, ok)
        else:
            (fake.lib.rla_ihs_destroy if solver == IHS else fake.lib.rla_proj_destroy)(h)
    assert failed
    fake.lib.rla_sketch_destroy(sk)
    fake.lib.rla_ctx_destroy(ctx)


def pool_rule_violations(log):
    """Uses of pool memory that its order does not cover: filled by the legacy stream (cudaMemcpy) before
    the stream it was allocated on has been waited for, or released with cudaFree, which returns
    pool memory without waiting for the device."""
    fresh, pool, bad = {}, set(), []
    for line in log:
        call, *rest = line.split()
        stream = next((r[7:] for r in rest if r.startswith("stream=")), None)
        if call == "cudaMallocFromPoolAsync":
            fresh[rest[0]] = stream
            pool.add(rest[0])
        elif call == "cudaStreamSynchronize":
            fresh = {p: s for p, s in fresh.items() if s != stream}
        elif call == "cudaDeviceSynchronize":
            fresh = {}
        elif call == "cudaMemcpy" and rest[0] in fresh:
            bad.append(line)
        elif call == "cudaFree" and rest[0] in pool:
            bad.append(line)
    return bad


@pytest.mark.parametrize("card", [LEFT, RIGHT])
@pytest.mark.parametrize("dtype", [F32, F64])
def test_loaded_fjlt_draws_follow_the_pool_order(fake, card, dtype):
    """The matrix of loaded FJLT draws is allocated, filled and released in the order of the context's
    stream; loading twice replaces what the first load allocated."""
    ctx = fake.context()
    s, L, N = 5, 50, 64
    sk = fake.sketch(ctx, "fjlt", s, L, card=card, dtype=dtype)
    ncol, nrow = (N, s) if card == LEFT else (s, N)
    nnz = ncol
    kptr = (ctypes.c_int64 * (ncol + 1))(*range(ncol + 1))
    idx = (ctypes.c_int64 * nnz)(*[i % nrow for i in range(nnz)])
    vals = ((ctypes.c_float if dtype == F32 else ctypes.c_double) * nnz)(*[1.0] * nnz)
    signs = (ctypes.c_uint8 * N)()
    fake.reset()
    for _ in range(2):
        rc = fake.lib.rla_sketch_set_draws(ctx, sk, idx, vals, signs, kptr, i64(nnz))
        assert rc == 0, fake.lib.rla_ctx_last_error(ctx)
    assert any(ln.startswith("cudaMallocFromPoolAsync") for ln in fake.log())
    assert pool_rule_violations(fake.log()) == []
    fake.lib.rla_sketch_destroy(sk)
    fake.lib.rla_ctx_destroy(ctx)


def mismatched_releases(log):
    """Allocations that are released by the call of another allocator, or never."""
    open_, bad = {}, []
    for line in log:
        call, *rest = line.split()
        if call in ("cudaMalloc", "cudaMallocAsync", "cudaMallocFromPoolAsync"):
            open_[rest[0]] = call
        elif call in ("cudaFree", "cudaFreeAsync"):
            if open_.pop(rest[0]) == "cudaMalloc" and call == "cudaFreeAsync":
                bad.append(line)
    return bad + sorted(open_)


@pytest.mark.parametrize("pool", [True, False])
def test_buffers_are_released_by_their_own_allocator(fake, pool, tmp_path):
    """Also on a device whose pool cannot be made: the creation then fails, without a buffer that a
    release in stream order does not know."""
    fake = fake.fresh(tmp_path)
    ctx = fake.context()
    if not pool:
        fake.fail_after("cudaMemPoolCreate", 0)
    rc, sk = fake.create(ctx, "sparse_sign", 40, 3000, nnz=8)
    assert (rc == 0) == pool
    fake.lib.rla_sketch_destroy(sk)
    fake.lib.rla_ctx_destroy(ctx)
    assert mismatched_releases(fake.log()) == []


def test_nothing_is_allocated_into_a_capture(fake):
    """Memory that an object keeps must not become part of a graph that is being captured (it would
    be mapped only while the graph runs): the call is refused and leaves the object as it was."""
    ctx = fake.context()
    s, m, n = 40, 3000, 7
    sk = fake.sketch(ctx, "sparse_sign", s, m, nnz=4)
    # the scratch of the later call, so that the capture finds it large enough
    mul = fake.lib.rla_sketch_mul_sparse_t
    mul.argtypes = [vp, vp, i64, i64, vp, i64, i64, i64, i64, vp, vp, vp, ctypes.c_double, ctypes.c_double]
    call = lambda k: mul(ctx, k, s, n, 1 << 40, s, m, n, 5, 1 << 41, 1 << 42, 1 << 43, 1.0, 0.0)
    other = fake.sketch(ctx, "sparse_sign", s, m, nnz=4)
    assert call(other) == 0, fake.lib.rla_ctx_last_error(ctx)
    fake.reset()
    fake.capturing(True)
    assert call(sk) != 0
    assert not any("cudaMallocFromPoolAsync" in ln for ln in fake.log())
    fake.capturing(False)
    fake.reset()
    assert call(sk) == 0
    assert any("iota" in k for k in fake.launches())  # the plan is built by the call that runs


def test_srht_expand_keeps_no_scratch_in_a_capture(fake):
    """S' * Y into a row-major result goes through the context's scratch, but not in a graph capture:
    the graph would keep the buffer after a later call had grown (and released) it."""
    ctx = fake.context()
    s, L, nv = 40, 3000, 64
    sk = fake.sketch(ctx, "srht", s, L)
    staged = lambda: [k for k in fake.launches() if "fjlt_expand_out" in k]
    assert fake.mul(ctx, sk, (s, L, nv), LEFT, adjoint=True, row_c=True) == 0
    assert staged()  # and the scratch is now large enough
    fake.reset()
    fake.capturing(True)
    assert fake.mul(ctx, sk, (s, L, nv), LEFT, adjoint=True, row_c=True, wait=False) == 0
    assert fake.launches() and not staged()


def test_wide_strided_compress_keeps_no_scratch_in_a_capture(fake):
    """A * S with so many rows that their tiles fill the device many times over needs no partial sums:
    a graph capture takes none from the scratch, whose growth would release them."""
    ctx = fake.context()
    s, L, nv = 40, 3000, 19200  # 600 tiles of 5 chunks: 21 chunks per CTA, 25 with whole tiles
    sk = fake.sketch(ctx, "sparse_sign", s, L, card=RIGHT, nnz=4)
    wide = fake.sketch(ctx, "srht", 4000, 5000)
    assert fake.mul(ctx, wide, (4000, 5000, 5000), LEFT, row_a=True) == 0  # a large scratch
    for capturing in (False, True):
        fake.reset()
        fake.capturing(capturing)
        assert fake.mul(ctx, sk, (s, L, nv), RIGHT, wait=False) == 0
        k = fake.launches()
        assert any("tile_compress" in x for x in k) and any("tile_reduce" in x for x in k) == (not capturing)


@pytest.mark.parametrize("s,L,large", [(1000, 10000, False), (1000, 90000, False), (1000, 101000, True), (2100, 100000, True)])
def test_buffers_that_the_pool_cannot_keep_are_not_pool_memory(fake, s, L, large):
    """The pool unmaps what it holds above its threshold, and maps it again for the next allocation."""
    ctx = fake.context()
    fake.reset()
    sk = fake.sketch(ctx, "gaussian", s, L)
    log = fake.log()
    assert any(ln.startswith("cudaMalloc ") for ln in log) == large
    fake.lib.rla_sketch_destroy(sk)
    assert mismatched_releases(fake.log()) == [] and freed_while_queued(fake.log()) == []
    assert any(ln.startswith("cudaFree ") for ln in fake.log()) == large
    fake.lib.rla_ctx_destroy(ctx)


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("L,s", [(1 << 20, 40), (100003, 300), (5000, 40), (4096, 40), (700, 9)])
def test_srht_tables_are_as_short_as_the_samples(fake, dtype, L, s):
    """A draw copies tables of its samples to the device, and of a short column's positions."""
    ctx = fake.context()
    fake.reset()
    sk = fake.sketch(ctx, "srht", s, L, dtype=dtype)
    copied = sum(int(ln.split("bytes=")[1]) for ln in fake.log() if ln.startswith("cudaMemcpyAsync"))
    padded = 1 << (L - 1).bit_length()
    assert copied <= 4 * (3 * s + (padded + 1 if padded <= 4096 else 0))
    fake.lib.rla_sketch_destroy(sk)
    fake.lib.rla_ctx_destroy(ctx)
