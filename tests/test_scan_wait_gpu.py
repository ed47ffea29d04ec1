"""Bounded waits of the streamed scan (k_scan_stream): where one runs out, its tiles are NaN,
never what the output held before; the wait is counted, and the next scan on the stream is
right.  (This module runs after the other scan tests, which assert that none of their own
waits ran out.)"""
import ctypes as C

import numpy as np
import pytest
import torch

import nt2_gb300.api as api

pytestmark = pytest.mark.gpu

TILE = 12288


def _count(cuda_lib):
    c = C.c_ulonglong()
    assert cuda_lib.nt2cuda_wait_timeouts(C.byref(c)) == 0
    return c.value


@pytest.mark.parametrize("rows,cols", [(60 * TILE + 8, 3), (160 * TILE + 13, 1), (1000 * TILE, 1)])
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("in_place", [False, True])
def test_tiles_of_waits_that_run_out(gpu, cuda_lib, rows, cols, kind, in_place):
    a = np.random.default_rng(rows + cols).standard_normal((cols, rows)).astype(np.float32)
    x = torch.from_numpy(a.reshape(-1)).cuda()
    ref = api.cumulative("cumsum", x, rows, cols, 1).cpu().numpy().reshape(cols, rows)
    y = x.clone() if in_place else torch.full_like(x, 7.0)
    before = y.cpu().numpy()[:TILE]
    count = _count(cuda_lib)
    st = cuda_lib.nt2cuda_selftest_stream_timeout(kind, (y if in_place else x).data_ptr(), rows, cols, y.data_ptr(),
                                                  torch.cuda.current_stream().cuda_stream)
    assert st == 5                                    # NT2CUDA_ERR_TIMEOUT
    assert _count(cuda_lib) > count
    got = y.cpu().numpy().reshape(cols, rows)
    if kind == 0:
        assert np.array_equal(got[0, :TILE], before)  # the tile that no block took
        assert np.isnan(got[0, TILE:]).all()
        assert np.array_equal(got[1:], ref[1:])
    else:
        assert np.isnan(got).all()
    count = _count(cuda_lib)
    assert np.array_equal(api.cumulative("cumsum", x, rows, cols, 1).cpu().numpy().reshape(cols, rows), ref)
    assert _count(cuda_lib) == count
