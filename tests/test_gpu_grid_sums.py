"""The grid-wide FP64 sums (warps in integers, blocks into integer
accumulators): terms over the whole range of doubles, single terms, exact
sums, infinities and NaN, through the action of the momenta."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one block of a partial warp count to several sites a thread
DIMS = [(4, 4, 4, 4), (6, 4, 6, 10), (12, 12, 12, 24), (32, 32, 32, 40)]


def action(m, dims, mom):
    m.set_lattice(dims)
    m.mom_load(mom)
    return m.mom_action()


def want(mom):
    s = (mom[..., :6] ** 2).sum(-1) + 0.5 * (mom[..., 6:9] ** 2).sum(-1) - 4.0
    return math.fsum(s.sum(-1).tolist())


# all terms but the -4 are positive: a term takes under 50 roundings in its
# site, a thread adds at most 32 sites, a warp aligns 32 lanes, a block adds 8
# warps: 128 roundings of the sum
@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("lo,hi", [(0, 0), (-30, 30), (-140, 140), (100, 150), (-5, 8)])
def test_range(gpu, dims, lo, hi):
    m = gpu
    rng = np.random.default_rng(abs(lo) + hi + dims[0])
    V = int(np.prod(dims))
    mom = rng.standard_normal((V, 4, 10)) * 10.0 ** rng.uniform(lo, hi, (V, 1, 1))
    mom[..., 9] = 0
    ref = want(mom)
    got = action(m, dims, mom)
    assert abs(got - ref) <= 128 * 2.0 ** -53 * (abs(ref) + 32.0 * V)
    assert action(m, dims, mom) == got


@pytest.mark.parametrize("dims", DIMS)
def test_exact(gpu, dims):
    """Sums of small whole numbers have no rounding; a launch leaves nothing behind."""
    m = gpu
    V = int(np.prod(dims))
    mom = np.zeros((V, 4, 10))
    assert action(m, dims, mom) == -16.0 * V
    mom[..., 0] = np.arange(V)[:, None] % 5
    assert action(m, dims, mom) == 4.0 * float((np.arange(V) % 5 * (np.arange(V) % 5)).sum()) - 16.0 * V
    mom[:] = 0
    mom[V // 3, 2, 1] = 2.0 ** 20   # above every other term
    assert action(m, dims, mom) == 2.0 ** 40 - 16.0 * V
    assert action(m, dims, np.zeros((V, 4, 10))) == -16.0 * V


@pytest.mark.parametrize("dims", DIMS[:3])
@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e200])
def test_not_finite(gpu, dims, bad):
    m = gpu
    V = int(np.prod(dims))
    mom = np.ones((V, 4, 10))
    mom[V - 1, 3, 4] = bad
    got = action(m, dims, mom)
    assert math.isnan(got) if math.isnan(bad) else got == math.inf
    mom[V - 1, 3, 4] = 1.0
    assert math.isfinite(action(m, dims, mom))   # nothing is left behind
