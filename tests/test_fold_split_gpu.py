"""Folds of shapes whose columns or rows are cut into segments over warps, blocks and
bulk-copy units: edges of the cut, single elements against 16-byte loads, and folds
captured into a CUDA graph before their stream has scratch."""
import numpy as np
import pytest
import torch

import nt2_gb300.api as api

pytestmark = pytest.mark.gpu

# columns just below, at and above one cut, a remainder of one, long single columns with and
# without whole 16-byte groups, many short columns, and the first and last bulk-copy lengths
SHAPES = [(33, 5), (1023, 3), (1025, 7), (4097, 61), (8191, 129), (10001, 77), (65536, 3), (65540, 1), (70001, 11),
          (777, 1001), (262147, 1), (1048576, 2), (64, 5000), (31, 9000), (129, 700), (100, 20001)]


def table(rows, cols, dtype, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal(rows * cols) + 0.25).astype(dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("rows,cols", SHAPES)
@pytest.mark.parametrize("dim", [0, 1, 2])
def test_sum_max_stdev_against_fp64(gpu, cuda_lib, rows, cols, dim, dtype):
    a = table(rows, cols, dtype, 7 * rows + cols)
    A = torch.from_numpy(a).cuda()
    ref = a.astype(np.longdouble).reshape(cols, rows)
    axis = {0: None, 1: 1, 2: 0}[dim]
    n = {0: rows * cols, 1: rows, 2: cols}[dim]
    u = np.finfo(dtype).eps / 2
    # a sum of n terms: one rounding of the result and (FP32: compensated partials; FP64: plain
    # partial sums of at most n terms) n ulps of the sum of magnitudes in the worst case
    got = api.reduce("sum", A, rows, cols, dim=dim).cpu().numpy().astype(np.longdouble)
    exact, mag = np.atleast_1d(ref.sum(axis)), np.atleast_1d(np.abs(ref).sum(axis))
    per_term = 2.0 ** -44 if dtype == np.float32 else u
    assert np.all(np.abs(got - exact) <= u * np.abs(exact) + per_term * n * mag)
    got = api.reduce("max", A, rows, cols, dim=dim).cpu().numpy()
    assert np.array_equal(got, np.atleast_1d(a.reshape(cols, rows).max(axis)))
    if n > 1:
        got = api.reduce("stdev", A, rows, cols, dim=dim).cpu().numpy().astype(np.longdouble)
        sd = np.atleast_1d(ref.std(axis, ddof=1))
        mean = np.abs(np.atleast_1d(ref.mean(axis)))
        assert np.all(np.abs(got - sd) <= 64 * 2 * u * (sd + mean))


@pytest.mark.parametrize("rows,cols", [(10001, 77), (65536, 3), (1025, 7)])
def test_fold_captured_on_a_stream_without_scratch(gpu, cuda_lib, rows, cols):
    """These columns needed no scratch when one warp (or unit) folded each; a capture on a
    fresh stream still takes them."""
    a = table(rows, cols, np.float32, 3)
    A = torch.from_numpy(a).cuda()
    out = torch.zeros(cols, device="cuda")
    api.reduce("sum", A, rows, cols, dim=1, out=out)      # loads the kernels
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    out.zero_()
    with torch.cuda.graph(g, stream=s):
        api.reduce("sum", A, rows, cols, dim=1, out=out)
    g.replay()
    torch.cuda.synchronize()
    ref = a.astype(np.float64).reshape(cols, rows).sum(1)
    mag = np.abs(a.astype(np.float64)).reshape(cols, rows).sum(1)
    assert np.all(np.abs(out.cpu().numpy() - ref) <= 2.0 ** -24 * np.abs(ref) + 2.0 ** -44 * rows * mag)
