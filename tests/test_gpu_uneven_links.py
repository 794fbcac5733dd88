"""Links whose matrices have entries far below their largest one (free, weak
or diagonal fields): staples, the reverse of the staples and the gauge paths
keep the digits of the small entries, which one exponent per matrix does not
hold (csrc/mks_fixed.cuh: such fields are done in plain FP64)."""
import numpy as np
import pytest

from conftest import rel
from test_gpu_staples_integer import _fat, _reference

pytestmark = pytest.mark.gpu

DIMS = (6, 4, 6, 10)


def _matrices(links):
    return np.ascontiguousarray(links.reshape(links.shape[0], 4, 3, 3, 2)).view(np.complex128)[..., 0]


def _links(M):
    return np.ascontiguousarray(np.stack([M.real, M.imag], -1).reshape(M.shape[0], 4, 18))


def _weak(m, dims, eps):
    """exp(i eps H) to second order in eps, H traceless Hermitian"""
    rng = np.random.default_rng(5)
    V = int(np.prod(dims))
    H = rng.standard_normal((V, 4, 3, 3)) + 1j * rng.standard_normal((V, 4, 3, 3))
    H = (H + H.conj().swapaxes(-1, -2)) / 2
    H -= np.trace(H, axis1=-2, axis2=-1)[..., None, None] / 3 * np.eye(3)
    return _links(np.eye(3) + 1j * eps * H - 0.5 * eps ** 2 * H @ H)


def test_fat_links_of_diagonal_links(gpu):
    """Every path's diagonal entries have a size of their own, up to (1e-8, 1, 1e8)
    to the seventh power apart."""
    m = gpu
    m.set_lattice(DIMS)
    rng = np.random.default_rng(6)
    V = int(np.prod(DIMS))
    M = np.zeros((V, 4, 3, 3), complex)
    size = np.array([1e-8, 1.0, 1e8])
    M[..., range(3), range(3)] = size * np.exp(1j * rng.uniform(-3, 3, (V, 4, 3)))
    got = _matrices(_fat(m, _links(M)))
    for k in range(3):                     # each entry is the fat link of a field of phases
        one = np.zeros_like(M)
        one[..., 0, 0] = M[..., k, k]
        want, bound = _reference(DIMS, _links(one))
        assert np.all(np.abs(got[..., k, k] - _matrices(want)[..., 0, 0]) <= 128 * 2.0 ** -53 * bound)
    off = ~np.eye(3, dtype=bool)
    assert not got[..., off].any()


@pytest.mark.parametrize("eps", [1e-10, 1e-14])
def test_fat_links_of_a_weak_field(gpu, eps):
    """The fat links' part of order eps: 18 roundings of eps on three levels, on
    either side, of which the staples' coefficients add up to less than 8."""
    m = gpu
    m.set_lattice(DIMS)
    links = _weak(m, DIMS, eps)
    got, want = _matrices(_fat(m, links)), _matrices(_reference(DIMS, links)[0])
    off = ~np.eye(3, dtype=bool)
    for a, b in ((got[..., off], want[..., off]), (got[..., range(3), range(3)].imag, want[..., range(3), range(3)].imag)):
        assert np.abs(a - b).max() <= 8 * 128 * 2.0 ** -53 * 10 * eps


@pytest.mark.parametrize("dims", [(4, 4, 4, 4), DIMS])
@pytest.mark.parametrize("eps", [1e-10, 1e-13])
def test_gauge_force_of_a_weak_field(gpu, oracle_cls, dims, eps):
    """The force is of order eps: the real parts of the paths drop out."""
    from oracle.oracle import GaugeOracle
    m = gpu
    U = _weak(m, dims, eps)
    zero = np.zeros((U.shape[0], 4, 10))
    m.set_lattice(dims)
    m.gauge_load(U)
    m.mom_load(zero)
    m.gauge_force(0.02, 7.4, 0.89, 3)
    got, want = m.mom_get(), GaugeOracle(oracle_cls(dims)).force(U, 0.02, 7.4, 0.89, 3, zero)
    # 54 paths of up to five products; their sum cancels to about a tenth of its terms
    assert 0 < np.abs(want).max() < 100 * eps
    assert rel(got[..., :9], want[..., :9]) < 4096 * 2.0 ** -53


@pytest.mark.parametrize("action", ["hisq", "asqtad"])
def test_force_of_free_links(gpu, oracle_cls, action):
    m = gpu
    orc = oracle_cls(DIMS)
    V = int(np.prod(DIMS))
    U = np.zeros((V, 4, 18))
    U[..., [0, 8, 16]] = 1.0
    U = m.apply_phases(DIMS, U)
    m.set_lattice(DIMS)
    getattr(m, "load_%s_links" % action)(U)
    xs = [m.gen_vector(DIMS, 7 + k, m.EVENANDODD) for k in range(2)]
    mom = np.zeros((V, 4, 10))
    m.eo_fermion_force_multi(0.1, [1.0, -0.5], xs, mom, action=action)
    args = (U, 0.1, [1.0, -0.5], xs) if action == "hisq" else (U, 1.0, 0.1, [1.0, -0.5], xs)
    want = getattr(orc, "fermion_force_" + action)(*args)
    assert rel(mom[..., :9], want[..., :9]) < 1e-13


@pytest.mark.parametrize("dims", [(4, 4, 4, 4), DIMS])
def test_even_matrices_of_very_different_size(gpu, dims):
    """Matrices without small entries, of sizes 1e-20 to 1e20, with zeros among
    them: the integer staples' exponents."""
    m = gpu
    m.set_lattice(dims)
    rng = np.random.default_rng(8)
    V = int(np.prod(dims))
    links = rng.uniform(0.25, 1.0, (V, 4, 18)) * rng.choice([-1.0, 1.0], (V, 4, 18))
    links *= 10.0 ** rng.uniform(-20, 20, (V, 4, 1))
    links[rng.uniform(size=(V, 4)) < 0.2] = 0.0
    got = _fat(m, links)
    want, bound = _reference(dims, links)
    assert np.all(np.linalg.norm(got - want, axis=-1) <= 128 * 2.0 ** -53 * bound)
