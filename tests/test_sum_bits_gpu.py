"""Plain sums of doubles drop no bits of a value: what huge terms of a lane's block cancel to keeps
what lies far below them, blocks that fit the lane's fixed point frame are summed exactly, and the
frame's edges (its lowest bit, its count of values, infinities, subnormals) hold."""
from fractions import Fraction

import numpy as np
import pytest
import torch

import nt2_gb300.api as api

pytestmark = pytest.mark.gpu

# (rows, cols, dim) and the offsets, along the folded dimension, of values that one lane takes one
# after the other: 16-byte loads and single elements down columns, bulk-copy tiles, along rows
LANES = [(2048, 40, 1, 64), (2049, 40, 1, 32), (131072, 3, 1, 512), (256, 640, 2, 8), (255, 640, 2, 8)]


def place(rows, cols, dim, step, values):
    """A table of zeros with `values` `step` apart in every column (dim 1) or row (dim 2)."""
    a = np.zeros((cols, rows))
    for i, v in enumerate(values):
        if dim == 1:
            a[:, i * step] = v
        else:
            a[i * step, :] = v
    return torch.from_numpy(a.reshape(-1)).cuda()


@pytest.mark.parametrize("rows,cols,dim,step", LANES)
@pytest.mark.parametrize("op", ["sum", "mean"])
@pytest.mark.parametrize("values", [(1e16, -1e16, 1e-3), (-1e16, 1e16, -1e-3), (1e200, -1e200, 3.0, 1e-9)])
def test_cancelled_block_keeps_its_small_values(gpu, cuda_lib, rows, cols, dim, step, op, values):
    got = api.reduce(op, place(rows, cols, dim, step, values), rows, cols, dim=dim).cpu().numpy()
    n = rows if dim == 1 else cols
    want = sum(values[2:])                       # one by one: the first two leave 0
    # NT2's mean is 1/n times the sum: two roundings more
    assert np.all(np.abs(got - (want if op == "sum" else want / n)) <= (0 if op == "sum" else 2.0 ** -52 * abs(want) / n))


@pytest.mark.parametrize("rows,cols,dim,step", LANES)
@pytest.mark.parametrize("below", [0, 27, 28, 29])
def test_blocks_within_a_frame_are_exact(gpu, cuda_lib, rows, cols, dim, step, below):
    """Every value of the table non-zero and within 29 binary orders of the largest: columns (or
    rows) of x, -x and one odd value per lane, whose sum is that of the odd values."""
    n = rows if dim == 1 else cols
    rng = np.random.default_rng(below + rows)
    small = np.ldexp(1.0 + 2.0 ** -52, -below)
    line = np.empty(n)
    period = 2 * step
    for i in range(n):                           # x and -x in turn, `step` apart: one lane's neighbours
        line[i] = 1.0 if (i // step) % 2 == 0 else -1.0
    line[n - n % period:] = small                # the rest, and one value of the first lane
    extra = n % period
    line[0] = small
    line[step] = small
    a = np.tile(line, (cols, 1)) if dim == 1 else np.tile(line[:, None], (1, rows))
    got = api.reduce("sum", torch.from_numpy(a.reshape(-1)).cuda(), rows, cols, dim=dim).cpu().numpy()
    exact = sum((Fraction(v) for v in line), Fraction(0))
    assert exact == (extra + 2) * Fraction(small)
    # partial sums of lanes and segments meet in plain additions of at most 2^12 terms of `small`
    assert np.all(np.abs(got - float(exact)) <= 2.0 ** -40 * float(exact))


def test_more_values_than_a_frame_holds(gpu, cuda_lib):
    """2^27 values of one sign with all bits set: a lane takes more than 1024 of them."""
    n, v = 1 << 27, 2.0 - 2.0 ** -52
    got = float(api.reduce("sum", torch.full((n,), v, dtype=torch.float64, device="cuda"), n, 1).cpu()[0])
    assert abs(Fraction(got) - n * Fraction(v)) <= Fraction(64, 2 ** 53) * n * Fraction(v)


@pytest.mark.parametrize("rows,cols,dim,step", LANES)
def test_values_no_frame_takes(gpu, cuda_lib, rows, cols, dim, step):
    inf, big, tiny = np.inf, 1.5e308, 5e-324
    for values, want in [((1.0, inf, 2.0), inf), ((inf, 1.0, -inf), np.nan), ((1.0, np.nan), np.nan), ((big, -big, big), big),
                         ((tiny, tiny, -3 * tiny), -tiny), ((1e-300, 1e-320, -1e-300), 1e-300 + 1e-320 - 1e-300),
                         ((-0.0, -0.0), 0.0), ((1e-30, 1.0, -1.0, 1e30, -1e30), 1e-30 + 1.0 - 1.0)]:
        got = api.reduce("sum", place(rows, cols, dim, step, values), rows, cols, dim=dim).cpu().numpy()
        assert np.array_equal(got, np.full(got.shape, want), equal_nan=True), (values, got[:4])
