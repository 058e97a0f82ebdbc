"""Sketches on several streams and threads at once, and in captured graphs: their buffers come from one
pool of the device, their plans from the context's stream, and shared-memory limits are remembered
per thread.  Results must be those of the same calls made alone, bit for bit (no kernel here adds
in an order that depends on timing)."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

#       kind, compression dimension, long dimension, vectors, nnz, side, adjoint
CALLS = [("SparseSign", 1041, 5000, 70, 4, "left", False), ("SparseSign", 100, 3001, 500, 8, "right", False),
         ("CountSketch", 3000, 20000, 33, 1, "right", False), ("SparseSign", 300, 60001, 40, 8, "left", True),
         ("SRHT", 300, 5003, 20, 1, "left", False), ("SRHT", 900, 1000, 20, 1, "left", True),
         ("FJLT", 60, 40000, 9, 1, "left", False), ("Gaussian", 70, 3000, 130, 1, "left", False)]


def operands(rla, dev, call, f64):
    """(recipe parameters, A, C, the arguments of the C call after the sketch)"""
    import torch
    kind, s, L, nv, nnz, side, adjoint = call
    left = side == "left"
    long_, short = ((L, nv), (s, nv)) if left else ((nv, L), (nv, s))
    a, c = (short, long_) if adjoint else (long_, short)
    dt = torch.float64 if f64 else torch.float32
    g = torch.Generator(device=dev)
    g.manual_seed(L + s)
    A = torch.randn(a[1], a[0], device=dev, dtype=dt, generator=g).t()
    C = torch.zeros(c[1], c[0], device=dev, dtype=dt).t()
    more = {"nnz": nnz} if kind == "SparseSign" else {}
    comp = getattr(rla, kind)(cardinality=rla.Left() if left else rla.Right(), compression_dim=s,
                              type=np.float64 if f64 else np.float32, **more)
    args = (0 if left else 1, int(adjoint), c[0], c[1], C.data_ptr(), c[0], 0, a[0], a[1], A.data_ptr(), a[0], 0, 1.0, 0.0)
    return comp, long_, A, C, args


def alone(rla, dev, call, f64, seed):
    comp, shape, A, C, _ = operands(rla, dev, call, f64)
    S = rla.complete_compressor(comp, np.empty(shape, np.float32), seed=seed)
    P = S.T if call[6] else S
    rla.mul_(C, P, A) if call[5] == "left" else rla.mul_(C, A, P)
    return C


def test_threads_with_their_own_streams(rla, dev):
    """Four threads, each with a context (and stream) of its own, create, apply, redraw and destroy
    sketches at the same time."""
    import torch
    from randlinearalgebra_b200 import _lib
    lib = _lib.lib()
    work = []
    for i, call in enumerate(CALLS):
        f64 = i % 2 == 1
        comp, shape, A, C, args = operands(rla, dev, call, f64)
        S = rla.complete_compressor(comp, np.empty(shape, np.float32), seed=40 + i)
        params = _lib.SketchParams(S.info.kind, S.info.card, S.info.dtype, call[1], call[2], call[4],
                                   getattr(comp, "block_size", 10), getattr(comp, "sparsity", 0.0), 40 + i)
        work.append((params, args, C, alone(rla, dev, call, f64, 40 + i), A, S))
    torch.cuda.synchronize()
    bad = []

    def run(t):
        try:
            torch.cuda.set_device(dev)
            ctx = ctypes.c_void_p()
            assert lib.rla_ctx_create(dev.index, None, ctypes.byref(ctx)) == 0
            for rep in range(6):
                for k in range(len(work)):
                    if k % 4 != t:  # a result buffer belongs to one thread
                        continue
                    params, args, C, ref, _, _ = work[k]
                    sk = ctypes.c_void_p()
                    _lib.check(lib.rla_sketch_create(ctx, ctypes.byref(params), ctypes.byref(sk)), ctx)
                    _lib.check(lib.rla_sketch_mul(ctx, sk, *args), ctx)
                    if not torch.equal(C, ref):
                        bad.append((k, rep))
                    torch.cuda.current_stream().synchronize()
                    _lib.check(lib.rla_sketch_update(ctx, sk), ctx)
                    _lib.check(lib.rla_sketch_destroy(sk), ctx)
            lib.rla_ctx_destroy(ctx)
        except Exception as e:  # noqa: BLE001
            bad.append((t, repr(e)))

    threads = [threading.Thread(target=run, args=(t,)) for t in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert bad == []


@pytest.mark.parametrize("call", CALLS[:7])
@pytest.mark.parametrize("f64", [False, True])
def test_captured_call(rla, dev, call, f64):
    """The same call recorded into a graph and replayed on new operands."""
    import torch
    from randlinearalgebra_b200 import _lib
    comp, shape, A, C, args = operands(rla, dev, call, f64)
    S = rla.complete_compressor(comp, np.empty(shape, np.float32), seed=9)
    P = S.T if call[6] else S
    mul = lambda: rla.mul_(C, P, A) if call[5] == "left" else rla.mul_(C, A, P)
    mul()  # the scratch that the capture will find
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        ctx = _lib.Context.get(dev.index)
        _lib.check(_lib.lib().rla_sketch_mul_async(ctx.handle, S.handle, *args), ctx.handle)
    A.copy_(torch.randn(A.shape[1], A.shape[0], device=dev, dtype=A.dtype).t())
    C.zero_()
    graph.replay()
    torch.cuda.synchronize()
    replayed = C.clone()
    C.zero_()
    mul()
    # a capture may give whole tiles to a CTA where a call cuts them: other partial sums
    tol = 1e-12 if f64 else 1e-6
    assert torch.linalg.norm(replayed - C) <= tol * torch.linalg.norm(C)
    del graph
