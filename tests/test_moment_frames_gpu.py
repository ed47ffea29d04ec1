"""var and stdev of double columns keep fixed-point frames per warp: values above an open
frame close it, ragged trips add zeros that are taken out again, and values no frame takes
go their own way.  Held to the reductions' bound, 64 eps (1 + |mean|/stdev) relative."""
import numpy as np
import pytest
import torch

from nt2_gb300 import api

pytestmark = pytest.mark.gpu


def _columns(kind, rows, cols, rng):
    x = rng.standard_normal((cols, rows))
    k = np.arange(rows) / rows
    if kind == "rising":
        x *= np.exp2(200.0 * k)
    elif kind == "falling":
        x *= np.exp2(-200.0 * k)
    elif kind == "steps":
        x = np.abs(x) * np.exp2(40.0 * (np.arange(rows) // 700)) * np.where(np.arange(rows) % 2, -1.0, 1.0)
    elif kind == "late outlier":
        x[:, -1] = 1e9
    elif kind == "offset":
        x += 1e6
    return x


@pytest.mark.parametrize("rows", [32, 33, 511, 513, 1024, 4099, 20001, 40000])
@pytest.mark.parametrize("kind", ["normal", "rising", "falling", "steps", "late outlier", "offset"])
def test_frames_open_and_close(gpu, cuda_lib, rows, kind):
    rng = np.random.default_rng(rows)
    cols = 3
    if kind == "steps" and rows > 4099:
        pytest.skip("its last steps would overflow")
    x = _columns(kind, rows, cols, rng)
    got = api.reduce("stdev", torch.from_numpy(x.reshape(-1)).cuda(), rows, cols, dim=1).cpu().numpy()
    w = x.astype(np.longdouble)
    mean = w.mean(axis=1)
    want = np.sqrt(((w - mean[:, None]) ** 2).sum(axis=1) / (rows - 1))
    tol = 64 * 2.0 ** -52 * (1 + np.abs(mean) / want)
    assert np.all(np.abs(got - want) <= tol * want)


@pytest.mark.parametrize("rows", [33, 1000, 20001])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("at", [0, 17, -1])
def test_values_no_frame_takes(gpu, cuda_lib, rows, bad, at):
    x = np.random.default_rng(rows).standard_normal((2, rows))
    x[1, at] = bad
    got = api.reduce("var", torch.from_numpy(x.reshape(-1)).cuda(), rows, 2, dim=1).cpu().numpy()
    assert abs(got[0] - x[0].var(ddof=1)) <= 64 * 2.0 ** -52 * got[0] * (1 + abs(x[0].mean()) / x[0].std())
    assert not np.isfinite(got[1])
