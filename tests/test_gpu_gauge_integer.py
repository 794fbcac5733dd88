"""The FP64 gauge force and action with their paths in integer arithmetic:
links that are not unitary and of widely different size, links of zeros, an
infinity among the links, ragged lattices, one partial block."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

LATTICES = [(4, 4, 4, 4), (4, 4, 6, 8), (6, 10, 4, 6)]
BETA, U0, NF, EPS = 7.4, 0.89, 3, 0.017
# a product of six matrices: 5 x 8 roundings of the Frobenius norms' product,
# up to 3^2.5 of the product's norm, on either side
TOL = 1024 * 2.0 ** -53


def _both(m, oracle_cls, dims, U):
    from oracle.oracle import GaugeOracle
    G = GaugeOracle(oracle_cls(dims))
    zero = np.zeros((U.shape[0], 4, 10))
    m.set_lattice(dims)
    m.gauge_load(U)
    m.mom_load(zero)
    m.gauge_force(EPS, BETA, U0, NF)
    with np.errstate(all="ignore"):
        return m.mom_get(), G.force(U, EPS, BETA, U0, NF, zero), m.gauge_action(BETA, U0, NF), G.action(U, BETA, U0, NF)


@pytest.mark.parametrize("dims", LATTICES)
@pytest.mark.parametrize("kind", ["near_unit", "any", "scales", "small", "zeros"])
def test_force_and_action(gpu, oracle_cls, dims, kind):
    m = gpu
    rng = np.random.default_rng(7)
    U = m.gen_thin_links(dims, 43, 0.3)
    if kind != "near_unit":
        U = rng.standard_normal(U.shape)
    link = (U.shape[0], 4) + (1,) * (U.ndim - 2)
    if kind == "scales":
        U = U * 10.0 ** rng.uniform(-8, 8, link)
    if kind == "small":
        U = U * 1e-40          # products of six down to 1e-240
    if kind == "zeros":
        U = U * (rng.uniform(size=link) > 0.3)
    got, want, a, b = _both(m, oracle_cls, dims, np.ascontiguousarray(U))
    assert rel(got[..., :9], want[..., :9]) < TOL
    assert abs(a - b) < TOL * (abs(b) + U.shape[0] * 100)


def test_all_links_zero(gpu, oracle_cls):
    m = gpu
    dims = LATTICES[1]
    U = np.zeros_like(m.gen_thin_links(dims, 43, 0.3))
    got, want, a, b = _both(m, oracle_cls, dims, U)
    assert not got.any() and abs(a - b) < 1e-13 * abs(b)


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_not_finite(gpu, oracle_cls, bad):
    """A link that is not finite spoils the links whose paths meet it and no others."""
    m = gpu
    dims = LATTICES[2]
    U = m.gen_thin_links(dims, 44, 0.3)
    U.reshape(-1)[5 * 72 + 18 + 4] = bad
    got, want, a, b = _both(m, oracle_cls, dims, U)
    fine = np.isfinite(want[..., :9]).all(-1)
    assert np.array_equal(np.isfinite(got[..., :9]).all(-1), fine) and 0 < fine.sum() < fine.size
    assert rel(got[fine][:, :9], want[fine][:, :9]) < TOL
    assert not np.isfinite(a) and not np.isfinite(b)
