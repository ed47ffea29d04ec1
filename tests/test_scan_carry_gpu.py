"""Carries of cumsum between the tiles of long float columns: sums that cancel between
tiles, overflow and come back, subnormal and non-finite ones, on the streamed kernel (aligned
tables) and on the look-back (misaligned ones).  A prefix that floats can hold is finite, and
what huge terms of other tiles cancel to keeps its bits."""
import numpy as np
import pytest
import torch

import nt2_gb300.api as api

pytestmark = pytest.mark.gpu

TILES = 200
# streamed tiles, and the look-back's, which columns one element off a 16-byte boundary take
KERNELS = [("streamed", 12288, 0), ("look-back", 16384, 1)]


def cumsum(a, offset, compensated):
    x = torch.zeros(a.size + 4, device="cuda")[offset:offset + a.size]
    x.copy_(torch.from_numpy(a))
    out = torch.zeros(a.size + 4, device="cuda")[offset:offset + a.size]
    api.cumulative("cumsum", x, a.size, 1, 1, compensated=compensated, out=out)
    return out.cpu().numpy()


def bound(ref, mag, compensated):
    # one rounding of the result; compensated partials to 2^-44 of the magnitudes, plain ones a
    # rounding for each step of a tile's sum (at most 64 in a row)
    return 2.0 ** -24 * np.abs(ref) + (2.0 ** -44 if compensated else 2.0 ** -24 * 64) * mag


@pytest.mark.parametrize("compensated", [True, False])
@pytest.mark.parametrize("name,tile,offset", KERNELS)
def test_tiles_of_opposite_sign(gpu, cuda_lib, name, tile, offset, compensated):
    """Tiles that sum to +-2e37 in turn: every prefix lies in [0, 2.1e37], while the sums of
    all the positive or of all the negative tiles are beyond the largest float."""
    sign = np.where(np.arange(TILES) % 2 == 0, 1.0, -1.0)
    a = np.repeat(sign * 2e37 / tile, tile).astype(np.float32)
    got = cumsum(a, offset, compensated).astype(np.float64)
    ref = np.cumsum(a.astype(np.float64))
    mag = np.cumsum(np.abs(a.astype(np.float64)))
    assert np.isfinite(got).all()
    assert np.all(np.abs(got - ref) <= bound(ref, mag, compensated))


@pytest.mark.parametrize("compensated", [True, False])
@pytest.mark.parametrize("name,tile,offset", KERNELS)
def test_huge_terms_that_cancel_between_tiles(gpu, cuda_lib, name, tile, offset, compensated):
    """Two tiles whose only non-zero element is +-1e30: past them a prefix is the sum of the
    others, to the bits it has without them."""
    rng = np.random.default_rng(3)
    a = rng.standard_normal(TILES * tile).astype(np.float32)
    small = a.astype(np.float64)
    for t, v in ((3, 1e30), (7, -1e30), (40, -2e35), (180, 2e35)):
        a[t * tile:(t + 1) * tile] = 0
        small[t * tile:(t + 1) * tile] = 0
        a[t * tile + 1234] = v
    got = cumsum(a, offset, compensated).astype(np.float64)
    ref, mag = np.cumsum(small), np.cumsum(np.abs(small))
    t = np.arange(a.size) // tile
    keep = (t < 3) | ((t > 7) & (t < 40)) | (t > 180)
    assert np.all(np.abs(got - ref)[keep] <= bound(ref, mag, compensated)[keep])


@pytest.mark.parametrize("compensated", [True, False])
@pytest.mark.parametrize("name,tile,offset", KERNELS)
def test_prefixes_that_overflow_and_come_back(gpu, cuda_lib, name, tile, offset, compensated):
    """Prefixes beyond the largest float read inf; a tile that starts from one that floats can
    hold again is finite (the tile in which it comes back, 21, may read inf to its end)."""
    rng = np.random.default_rng(4)
    a = rng.standard_normal(TILES * tile).astype(np.float32)
    for k, v in ((10, 2e38), (11, 2e38), (12, 2e38), (20, -2e38), (21, -2e38), (22, -2e38)):
        a[k * tile:(k + 1) * tile] = 0
        a[k * tile + 77] = v
    got = cumsum(a, offset, compensated)
    exact = np.cumsum(a.astype(np.longdouble))
    t = np.arange(a.size) // tile
    over = exact > 3.4e38
    assert np.array_equal(np.isposinf(got)[t != 21], over[t != 21])
    assert np.isfinite(got[~over & (t != 21)]).all()
    small = np.where((t >= 10) & (t <= 22), 0, a.astype(np.float64))
    small[(t >= 13) & (t < 20)] = a[(t >= 13) & (t < 20)]
    ref, mag = np.cumsum(small), np.cumsum(np.abs(small))
    keep = (t < 10) | (t > 22)
    assert np.all(np.abs(got.astype(np.float64) - ref)[keep] <= bound(ref, mag, compensated)[keep])


@pytest.mark.parametrize("compensated", [True, False])
@pytest.mark.parametrize("name,tile,offset", KERNELS)
def test_subnormals_and_non_finite(gpu, cuda_lib, name, tile, offset, compensated):
    """Prefixes of the smallest subnormal are exact; -inf after inf is NaN from there on."""
    n = TILES * tile
    assert n < 1 << 24
    a = np.full(n, 2.0 ** -149, np.float32)
    got = cumsum(a, offset, compensated)
    assert np.array_equal(got, (np.arange(1, n + 1) * 2.0 ** -149).astype(np.float32))
    a[100 * tile + 5] = np.inf
    a[190 * tile + 9] = -np.inf
    got = cumsum(a, offset, compensated)
    assert np.isfinite(got[:100 * tile + 5]).all()
    assert np.isposinf(got[100 * tile + 5:190 * tile + 9]).all()
    assert np.isnan(got[190 * tile + 9:]).all()


@pytest.mark.parametrize("compensated", [True, False])
@pytest.mark.parametrize("offset", [0, 1])
def test_long_column_is_reproducible(gpu, cuda_lib, offset, compensated):
    """2^24 elements, streamed or chained through the look-back: the same bits each time."""
    a = np.random.default_rng(6).standard_normal(1 << 24).astype(np.float32)
    got = cumsum(a, offset, compensated)
    assert np.array_equal(got, cumsum(a, offset, compensated))
    ref, mag = np.cumsum(a.astype(np.float64)), np.cumsum(np.abs(a.astype(np.float64)))
    assert np.all(np.abs(got - ref) <= bound(ref, mag, compensated))
