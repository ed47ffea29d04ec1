"""cumsum of long float columns, streamed through shared memory (k_scan_stream): lengths around
its tile (12288 elements) and 32-element rows, several columns, in place, plain and compensated,
non-finite values, and runs that must agree bit for bit."""
import numpy as np
import pytest
import torch

import nt2_gb300.api as api

pytestmark = pytest.mark.gpu

TILE = 12288
SHAPES = [(152 * TILE, 1), (152 * TILE + 1, 1), (153 * TILE - 1, 1), (193 * TILE + 8192 + 31, 1), (TILE, 152),
          (11 * TILE // 12, 304), (3 * TILE + 4, 203), (130 * TILE - 28, 5), (1000 * TILE + 8224, 1)]


def table(n, seed):
    return np.random.default_rng(seed).standard_normal(n).astype(np.float32)


@pytest.mark.parametrize("rows,cols", SHAPES)
@pytest.mark.parametrize("compensated", [True, False])
def test_against_fp64(gpu, cuda_lib, rows, cols, compensated):
    a = table(rows * cols, rows + cols)
    A = torch.from_numpy(a).cuda()
    out = api.cumulative("cumsum", A, rows, cols, dim=1, compensated=compensated)
    again = api.cumulative("cumsum", A, rows, cols, dim=1, compensated=compensated, out=A.clone())
    assert torch.equal(out, again)
    inplace = A.clone()
    api.cumulative("cumsum", inplace, rows, cols, dim=1, compensated=compensated, out=inplace)
    assert torch.equal(out, inplace)
    d = A.double().view(cols, rows)
    ref, mag = d.cumsum(1), d.abs().cumsum(1)
    # one rounding of the result; compensated partials to 2^-44 of the magnitudes, plain ones
    # a rounding for each element of a 32-element row, its warp, its block's warps and the prefix
    per = 2.0 ** -44 if compensated else 2.0 ** -24 * 64
    err = (out.double().view(cols, rows) - ref).abs()
    assert bool((err <= 2.0 ** -24 * ref.abs() + per * mag).all())


def test_nonfinite(gpu, cuda_lib):
    rows = 640 * TILE
    a = table(rows, 3)
    a[5 * TILE + 7] = np.inf
    a[200 * TILE] = np.nan
    out = api.cumulative("cumsum", torch.from_numpy(a).cuda(), rows, 1).cpu().numpy()
    assert np.isfinite(out[:5 * TILE + 7]).all()
    assert np.isposinf(out[5 * TILE + 7:200 * TILE]).all()
    assert np.isnan(out[200 * TILE:]).all()


def test_two_streams_at_once(gpu, cuda_lib):
    """Two scans whose blocks share the SMs: neither needs all its blocks resident."""
    rows = 600 * TILE
    tables = [torch.from_numpy(table(rows, 10 + i)).cuda() for i in range(2)]
    alone = [api.cumulative("cumsum", t, rows, 1) for t in tables]
    streams = [torch.cuda.Stream() for _ in tables]
    outs = [torch.empty_like(t) for t in tables]
    torch.cuda.synchronize()
    for _ in range(4):
        for s, t, o in zip(streams, tables, outs):
            with torch.cuda.stream(s):
                api.cumulative("cumsum", t, rows, 1, out=o)
    torch.cuda.synchronize()
    for o, r in zip(outs, alone):
        assert torch.equal(o, r)
