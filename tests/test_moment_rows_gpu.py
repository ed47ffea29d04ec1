"""var and stdev of double rows keep a fixed-point frame in each lane: values above an open frame
close it, as 512 values do, and values no frame takes go their own way.  Held to the reductions'
bound, 64 eps (1 + |mean|/stdev) relative, and where a frame's pivot lies far from most of its
values to a few roundings in the mean."""
import numpy as np
import pytest
import torch

from nt2_gb300 import api

pytestmark = pytest.mark.gpu


def _rows(kind, rows, cols, rng):
    x = rng.standard_normal((rows, cols))
    k = np.arange(cols) / cols
    if kind == "rising":
        x *= np.exp2(200.0 * k)
    elif kind == "falling":
        x *= np.exp2(-200.0 * k)
    elif kind == "steps":
        x = np.abs(x) * np.exp2(40.0 * (np.arange(cols) // 90)) * np.where(np.arange(cols) % 2, -1.0, 1.0)
    elif kind == "late outlier":
        x[:, -1] = 1e9
    elif kind == "offset":
        x += 1e6
    return x


def _column_major(x):
    return torch.from_numpy(np.ascontiguousarray(x.T).reshape(-1)).cuda()


# rows take 16-byte loads (even) or single elements; columns in one chunk or several, with ends of
# blocks of 4, 8 and 16 trips
@pytest.mark.parametrize("rows", [2, 3, 64, 65])
@pytest.mark.parametrize("cols", [32, 33, 64, 127, 500, 1111])
@pytest.mark.parametrize("kind", ["normal", "rising", "falling", "steps", "late outlier", "offset"])
def test_frames_open_and_close(gpu, cuda_lib, rows, cols, kind):
    x = _rows(kind, rows, cols, np.random.default_rng(rows * cols))
    got = api.reduce("stdev", _column_major(x), rows, cols, dim=2).cpu().numpy()
    w = x.astype(np.longdouble)
    mean = w.mean(axis=1)
    want = np.sqrt(((w - mean[:, None]) ** 2).sum(axis=1) / (cols - 1))
    tol = 64 * 2.0 ** -52 * (1 + np.abs(mean) / want)
    assert np.all(np.abs(got - want) <= tol * want)


@pytest.mark.parametrize("rows", [2, 3])
@pytest.mark.parametrize("cols", [33, 1000, 20001])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 1e303])
@pytest.mark.parametrize("at", [0, 17, -1])
def test_values_no_frame_takes(gpu, cuda_lib, rows, cols, bad, at):
    x = np.random.default_rng(cols).standard_normal((rows, cols))
    x[1, at] = bad
    got = api.reduce("var", _column_major(x), rows, cols, dim=2).cpu().numpy()
    for i in {0, rows - 1} - {1}:
        assert abs(got[i] - x[i].var(ddof=1)) <= 64 * 2.0 ** -52 * got[i] * (1 + abs(x[i].mean()) / x[i].std())
    assert not np.isfinite(got[1])


@pytest.mark.parametrize("rows,cols", [(33, 70), (34, 70), (1000, 41), (10001, 7), (70, 1111), (65, 2000), (64, 2000)])
@pytest.mark.parametrize("dim", [0, 1, 2])
@pytest.mark.parametrize("value", [0.1, -1e16 / 3, 7e-200])
def test_equal_values_have_no_variance(gpu, cuda_lib, rows, cols, dim, value):
    """The frame's mean of equal values is that value, whatever pivot a ragged first trip gave."""
    x = torch.full((rows * cols,), value, dtype=torch.float64, device="cuda")
    assert float(api.reduce("stdev", x, rows, cols, dim=dim).abs().max()) == 0.0


@pytest.mark.parametrize("rows", [9761, 19522])
def test_pivot_far_from_the_values(gpu, cuda_lib, rows):
    """Rows long enough that a lane closes a frame at 512 values, whose first block (the first 64
    or 128 columns) is half as large as the rest: the squares about the pivot are 30 to 60 times
    M2, and no bit of M2 goes with them.  A variance takes some 30 roundings (closing the frames
    and merging 9 states), each at most u of M2 and u/sqrt(3) in the mean square, together 6 u."""
    cols, lead = 4300, 8 * (16 if rows % 2 else 8)
    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    x = torch.rand((cols, rows), generator=g, dtype=torch.float64, device="cuda") * 0.001 + 1.0
    x[:lead] -= 0.5
    got = api.reduce("var", x.reshape(-1), rows, cols, dim=2)
    pick = torch.arange(0, rows, rows // 400, device="cuda")
    w = x[:, pick].cpu().numpy().astype(np.longdouble)
    want = ((w - w.mean(axis=0)) ** 2).sum(axis=0) / (cols - 1)
    err = (got[pick].cpu().numpy() - want) / want
    assert float(np.sqrt((err ** 2).mean())) <= 6 * 2.0 ** -53
    assert float(np.abs(err).max()) <= 48 * 2.0 ** -53
