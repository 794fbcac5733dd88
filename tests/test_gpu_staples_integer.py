"""The FP64 staples in integer arithmetic (csrc/mks_fixed_mat.cuh) and the
staple launches over directions: matrices of widely different size, zeros,
unit links, infinities and NaNs, and lattices on either side of the
four-directions-a-launch rule."""
import ctypes

import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

COEFFS = (1.0, -1 / 24, -1 / 16, 1 / 64, -1 / 384, -1 / 8)   # one_link, naik, 3, 5, 7, Lepage


def _fat(m, links):
    fat = np.zeros_like(links)
    c = (ctypes.c_double * 6)(*COEFFS)
    m.check(m.init().mks_fatlong_links(c, links.ctypes.data_as(m._lib.DP), fat.ctypes.data_as(m._lib.DP), None),
            "mks_fatlong_links")
    return fat


def _order(dims):
    nx, ny, nz, nt = dims
    t, z, y, x = np.meshgrid(np.arange(nt), np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    odd = ((x + y + z + t) & 1).reshape(-1)
    return np.concatenate([np.nonzero(odd == 0)[0], np.nonzero(odd == 1)[0]])


def _grid(dims, sites):
    """(V, ...) in MILC's order -> (t, z, y, x, ...)"""
    out = np.empty_like(sites)
    out[_order(dims)] = sites
    return out.reshape((dims[3], dims[2], dims[1], dims[0]) + sites.shape[1:])


def _sites(dims, grid):
    return np.ascontiguousarray(grid.reshape((-1,) + grid.shape[4:])[_order(dims)])


def _fatten(links, mm, adj, c):
    """load_fatlinks_cpu's recursion on grids: complex matrices, or their
    norms (mm = product, adj = identity, absolute coefficients)."""
    sh = lambda a, mu, k: np.roll(a, -k, 3 - mu)

    def staple(mu, nu, A):
        U = links[nu]
        up = mm(U, mm(sh(A, nu, 1), adj(sh(U, mu, 1))))
        return up + sh(mm(mm(adj(U), A), sh(U, mu, 1)), nu, -1)

    out = []
    for mu in range(4):
        f = c[0] * links[mu]
        for nu in range(4):
            if nu == mu:
                continue
            s = staple(mu, nu, links[mu])
            f = f + c[2] * s + c[5] * staple(mu, nu, s)
            for rho in range(4):
                if rho in (mu, nu):
                    continue
                q = staple(mu, rho, s)
                f = f + c[3] * q + c[4] * staple(mu, 6 - mu - nu - rho, q)
        out.append(f)
    return out


def _reference(dims, links):
    """(fat, sum over paths of |coefficient| times the links' norms) in MILC's layout."""
    g = _grid(dims, links.reshape(-1, 4, 3, 3, 2))
    U = [np.ascontiguousarray(g[..., mu, :, :, :]).view(np.complex128)[..., 0] for mu in range(4)]
    c = (COEFFS[0] - 6 * COEFFS[5],) + COEFFS[1:]
    with np.errstate(all="ignore"):
        F = _fatten(U, lambda a, b: a @ b, lambda a: a.conj().swapaxes(-1, -2), c)
        n = [np.linalg.norm(u, axis=(-1, -2)) for u in U]
        B = _fatten(n, lambda a, b: a * b, lambda a: a, [abs(x) for x in c])
    f = np.stack(F, 4)
    f = np.stack([f.real, f.imag], -1)
    return _sites(dims, f).reshape(-1, 4, 18), _sites(dims, np.stack(B, 4))


# 4^4: tiles of 32 sites exactly; 6x4x6x10: 720 sites of a parity, half a tile left
@pytest.mark.parametrize("dims", [(4, 4, 4, 4), (6, 4, 6, 10)])
def test_links_of_very_different_size(gpu, dims):
    m = gpu
    m.set_lattice(dims)
    rng = np.random.default_rng(2)
    V = int(np.prod(dims))
    links = rng.standard_normal((V, 4, 18)) * 10.0 ** rng.uniform(-20, 20, (V, 4, 1))
    links *= 10.0 ** rng.uniform(-6, 0, links.shape)
    links[rng.uniform(size=(V, 4)) < 0.2] = 0.0
    got = _fat(m, links)
    want, bound = _reference(dims, links)
    # three levels of products of 3x3 matrices, 18 roundings of 2^-53 each on either side
    assert np.all(np.linalg.norm(got - want, axis=-1) <= 128 * 2.0 ** -53 * bound)


def test_unit_links_are_exact(gpu):
    m = gpu
    dims = (6, 4, 6, 10)
    m.set_lattice(dims)
    links = np.zeros((int(np.prod(dims)), 4, 18))
    links[..., [0, 8, 16]] = 1.0
    got = _fat(m, links)
    one = got[0, 0, 0]
    assert np.array_equal(got, one * links) and abs(one - 2.0) < 4.0   # no rounding but the coefficients'


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_not_finite_links(gpu, bad):
    m = gpu
    dims = (6, 4, 6, 10)
    m.set_lattice(dims)
    links = m.gen_thin_links(dims, 3, 0.3)
    links[100, 2, 7] = bad
    got = _fat(m, links)
    want, _ = _reference(dims, links)
    ok = np.isfinite(want).all(-1)
    assert not ok.all() and np.array_equal(np.isfinite(got).all(-1), ok)
    assert rel(got[ok], want[ok]) < 1e-14


def test_force_of_a_vector_that_is_not_finite(gpu):
    """A NaN in one solution reaches the same momenta in FP64 (integer chains,
    plain FP64 where a matrix is not finite) as in FP32 arithmetic."""
    m = gpu
    dims = (12, 10, 12, 14)
    m.set_lattice(dims)
    U = m.apply_phases(dims, m.gen_thin_links(dims, 5, 0.3))
    x = m.gen_vector(dims, 6, m.EVENANDODD)
    x[77, 1] = np.nan
    masks = []
    try:
        for prec in (m.PREC_DOUBLE, m.PREC_SINGLE):
            m.md_precision(prec)
            m.load_hisq_links(U)
            mom = np.zeros((U.shape[0], 4, 10))
            m.eo_fermion_force_multi(0.1, [1.0], [x], mom)
            masks.append(np.isfinite(mom).all(-1))
    finally:
        m.md_precision(m.PREC_DOUBLE)
    assert np.array_equal(masks[0], masks[1]) and masks[0].any() and not masks[0].all()


# The two sides add the same staple terms in another order (no U(3) projection,
# whose derivative amplifies roundings, in the asqtad force): up to 60
# roundings of the sum of the terms' magnitudes, at most 3 times their sum with
# the asqtad coefficients; 256 roundings of the precision cover it.
@pytest.mark.parametrize("prec,eps", [("PREC_DOUBLE", 2.0 ** -53), ("PREC_SINGLE", 2.0 ** -24)])
def test_one_direction_a_launch(gpu, prec, eps):
    """Beyond 2^20 sites of a parity a launch takes one direction: a periodic
    tiling of a small lattice has the small one's asqtad force on every tile."""
    m = gpu
    small, times = (8, 8, 8, 22), (4, 4, 4, 3)
    big = tuple(a * b for a, b in zip(small, times))
    assert np.prod(big) // 2 > 2 ** 20
    reps = (times[3], times[2], times[1], times[0])
    U = m.gen_thin_links(small, 8, 0.3)
    x = m.gen_vector(small, 9, m.EVENANDODD)
    tile = lambda a: _sites(big, np.tile(_grid(small, a), reps + (1,) * (a.ndim - 1)))
    out = []
    try:
        m.md_precision(getattr(m, prec))
        for dims, links, v in ((small, U, x), (big, tile(U), tile(x))):
            m.set_lattice(dims)
            m.load_asqtad_links(links)
            mom = np.zeros((links.shape[0], 4, 10))
            m.eo_fermion_force_multi(0.1, [1.0], [v], mom, action="asqtad")
            out.append(mom)
    finally:
        m.md_precision(m.PREC_DOUBLE)
        m.set_lattice(small)
    assert rel(out[1], tile(out[0])) < 256 * eps
