"""Folds captured into a CUDA graph.  Columns of up to 4096 16-byte groups take no scratch there,
so that a graph shares no partials or counters with what else runs; longer ones take no more of
it than one partial for every 4096 groups.  A captured result does not depend on what ran on the
stream before."""
import contextlib
import ctypes as C

import numpy as np
import pytest
import torch

import nt2_gb300.api as api

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def own_stream():
    """A stream that no earlier call has used: torch hands out pooled ones."""
    rt, raw = torch.cuda.cudart(), C.c_void_p()
    assert int(rt.cudaStreamCreate(C.addressof(raw))) == 0
    s = torch.cuda.ExternalStream(raw.value)
    s.wait_stream(torch.cuda.current_stream())
    try:
        yield s
    finally:
        torch.cuda.synchronize()


def allocations(cuda_lib):
    n = C.c_ulonglong()
    assert cuda_lib.nt2cuda_scratch_allocations(C.byref(n)) == 0
    return n.value


def table(n, dtype, seed, offset=0):
    x = torch.empty(n + 4, dtype=dtype, device="cuda")[offset:offset + n]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return x.copy_(torch.randn(n, generator=g, dtype=dtype, device="cuda") + 0.25)


def check(op, out, A, rows, cols, dim):
    a = A.double().view(cols, rows)
    axis = {0: (0, 1), 1: 1, 2: 0}[dim]
    n = {0: rows * cols, 1: rows, 2: cols}[dim]
    ref, mag = a.sum(axis).reshape(-1), a.abs().sum(axis).reshape(-1)
    u = 2.0 ** -24 if A.dtype == torch.float32 else 2.0 ** -53
    # plain sums: a rounding of the running sum for each of at most n terms
    if op == "sum":
        assert bool(((out.double() - ref).abs() <= u * n * mag).all())
    else:
        sd = a.std(axis, unbiased=True).reshape(-1)
        assert bool(((out.double() - sd).abs() <= 128 * u * (sd + ref.abs() / n) + 2.0 ** -45 * sd).all())


def capture(stream, op, A, rows, cols, dim, out):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        api.reduce(op, A, rows, cols, dim=dim, compensated=False, out=out)
    return g


def warm(stream, op, A, rows, cols, dim):
    with torch.cuda.stream(stream):
        api.reduce(op, A, rows, cols, dim=dim, compensated=False)
    stream.synchronize()


def m_of(rows, cols, dim):
    return {0: 1, 1: cols, 2: rows}[dim]


WHOLE = [("sum", 10001, 77, 1, torch.float32), ("sum", 16384, 5, 1, torch.float32), ("sum", 65536, 3, 1, torch.float32),
         ("sum", 1025, 7, 1, torch.float32), ("sum", 128, 128, 0, torch.float32), ("sum", 8192, 9, 1, torch.float64),
         ("stdev", 8191, 9, 1, torch.float64), ("stdev", 65536, 2, 1, torch.float32)]


@pytest.mark.parametrize("op,rows,cols,dim,dtype", WHOLE)
def test_captured_result_does_not_depend_on_earlier_calls(gpu, cuda_lib, op, rows, cols, dim, dtype):
    A = table(rows * cols, dtype, 7 * rows + cols)
    big = table(1 << 21, dtype, 1)
    out = [torch.zeros(m_of(rows, cols, dim), dtype=dtype, device="cuda") for _ in range(2)]
    api.reduce(op, A, rows, cols, dim=dim, compensated=False)         # loads the kernels
    torch.cuda.synchronize()
    with own_stream() as cold, own_stream() as used:
        warm(used, op, A, rows, cols, dim)
        warm(used, "sum", big, big.numel(), 1, 1)
        n = allocations(cuda_lib)
        g = [capture(s, op, A, rows, cols, dim, o) for s, o in zip((cold, used), out)]
        assert allocations(cuda_lib) == n
        for x in g:
            x.replay()
        torch.cuda.synchronize()
    check(op, out[0], A, rows, cols, dim)
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("op,rows,cols,dim,dtype", WHOLE)
def test_graph_outlives_the_scratch_of_its_stream(gpu, cuda_lib, op, rows, cols, dim, dtype):
    """A larger fold later on the stream grows its scratch; the graph does not use it."""
    A = table(rows * cols, dtype, 7 * rows + cols)
    big = table(1 << 21, dtype, 1)
    out = torch.zeros(m_of(rows, cols, dim), dtype=dtype, device="cuda")
    with own_stream() as s:
        warm(s, op, A, rows, cols, dim)
        g = capture(s, op, A, rows, cols, dim, out)
        n = allocations(cuda_lib)
        warm(s, "sum", big, 512, 4096, 2)                             # row sums in many chunks
        assert allocations(cuda_lib) > n
        g.replay()
        torch.cuda.synchronize()
    check(op, out, A, rows, cols, dim)


@pytest.mark.parametrize("dim", [1, 2])
def test_graph_keeps_the_scratch_it_holds(gpu, cuda_lib, dim):
    """A captured fold that does use scratch still writes its own after a larger fold on the
    stream has made that grow."""
    rows, cols = (200000, 3) if dim == 1 else (3, 200000)
    A, big = table(rows * cols, torch.float32, 5), table(1 << 21, torch.float32, 1)
    out = torch.zeros(m_of(rows, cols, dim), device="cuda")
    with own_stream() as s:
        warm(s, "sum", A, rows, cols, dim)
        g = capture(s, "sum", A, rows, cols, dim, out)
        n = allocations(cuda_lib)
        warm(s, "sum", big, 512, 4096, 2)
        assert allocations(cuda_lib) > n
        other = torch.full((1 << 20,), 3.0, device="cuda")            # what a freed buffer would be handed out as
        g.replay()
        torch.cuda.synchronize()
        assert bool((other == 3.0).all())
        check("sum", out, A, rows, cols, dim)
        with torch.cuda.stream(s):
            got = api.reduce("sum", big, 512, 4096, dim=2, compensated=False)
        s.synchronize()
    check("sum", got, big, 512, 4096, 2)


# the fold that warms the stream, and one whose partials (one for every 4096 16-byte groups of a
# column, or for every 64 to 128 columns of a strip of rows) fit what that allocated
FITS = [(("sum", 40000, 1, 1, 0), ("sum", 20000, 100, 1, 0), torch.float32),
        (("sum", 40000, 1, 1, 0), ("sum", 3333333, 1, 1, 1), torch.float32),
        (("sum", 40000, 1, 1, 0), ("sum", 20000, 60, 1, 1), torch.float64),
        (("sum", 40000, 1, 1, 0), ("stdev", 1 << 20, 2, 1, 0), torch.float64),
        (("sum", 128, 25000, 2, 0), ("sum", 128, 40000, 2, 0), torch.float32),
        (("sum", 20000, 3000, 1, 0), ("sum", 20000, 100, 1, 0), torch.float32)]


@pytest.mark.parametrize("first,then,dtype", FITS)
def test_capture_that_fits_the_scratch(gpu, cuda_lib, first, then, dtype):
    op0, rows0, cols0, dim0, off0 = first
    op, rows, cols, dim, off = then
    B, A = table(rows0 * cols0, dtype, 1, off0), table(rows * cols, dtype, 2, off)
    out = torch.zeros(m_of(rows, cols, dim), dtype=dtype, device="cuda")
    api.reduce(op, A, rows, cols, dim=dim, compensated=False)         # loads the kernels
    torch.cuda.synchronize()
    with own_stream() as s:
        warm(s, op0, B, rows0, cols0, dim0)
        n = allocations(cuda_lib)
        g = capture(s, op, A, rows, cols, dim, out)
        assert allocations(cuda_lib) == n
        g.replay()
        torch.cuda.synchronize()
    check(op, out, A, rows, cols, dim)
