"""The FP64 D_eo on links of widely different size (csrc/mks_fixed.cuh holds
the links of a slot to one exponent for the fat and one for the Naik links; a
slot whose links that does not suit is done in plain FP64): every site as
accurate as its own links and neighbours, whatever the rest of the lattice
holds."""
import numpy as np
import pytest

from conftest import hisq_setup


pytestmark = pytest.mark.gpu

# four threads per site in two waves and in one (2592 warps), and one thread per site
LATTICES = [(6, 4, 10, 12), (12, 12, 12, 24), (16, 16, 18, 36)]


def _order(dims):
    nx, ny, nz, nt = dims
    t, z, y, x = np.meshgrid(np.arange(nt), np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    odd = ((x + y + z + t) & 1).reshape(-1)
    return np.concatenate([np.nonzero(odd == 0)[0], np.nonzero(odd == 1)[0]])


def _site_bound(dims, fat, lng, src):
    """Sum over a site's 16 terms of |U| |v|, in MILC's site order."""
    order, grid = _order(dims), (dims[3], dims[2], dims[1], dims[0])

    def g(a):
        out = np.empty_like(a)
        out[order] = a
        return out.reshape(grid)

    v, s = g(np.linalg.norm(src, axis=1)), 0.0
    for mu in range(4):
        ax = 3 - mu
        for U, k in ((fat, 1), (lng, 3)):
            u = g(np.linalg.norm(U[:, mu].reshape(len(order), -1), axis=1))
            s = s + u * np.roll(v, -k, ax) + np.roll(u * v, k, ax)
    return s.reshape(-1)[order]


# on either side 192 products and sums per component, and the 16 terms' own
# roundings: 256 roundings of 2^-53 of the sum of the terms' norms
TOL = 256 * 2.0 ** -53


def _scaled(m, oracle_cls, dims, kind):
    U, orc, L = hisq_setup(m, oracle_cls, dims)
    fat, lng = L["fat"][0].copy(), L["lng"][0].copy()
    rng = np.random.default_rng(3)
    V = len(fat)
    if kind == "spread":
        fat *= 10.0 ** rng.uniform(-8, 8, (V, 4, 1))
        lng *= 10.0 ** rng.uniform(-8, 8, (V, 4, 1))
    elif kind == "mild":      # within the line where the integer form still serves
        fat *= 2.0 ** rng.uniform(-3.5, 0, (V, 4, 1))
    elif kind == "over":      # just beyond it
        fat *= 2.0 ** rng.uniform(-6, 0, (V, 4, 1))
    elif kind == "one_fat":
        fat[V // 3, 2] *= 2.0 ** 40
    elif kind == "one_lng":
        lng[V // 5, 1] *= 2.0 ** 60
    elif kind == "one_small":
        fat[V // 3, 3] *= 2.0 ** -40
    elif kind == "small_lng":
        lng *= 2.0 ** -45
    elif kind == "zeros":     # links that are switched off
        fat[rng.uniform(size=(V, 4)) < 0.3] = 0.0
        lng[:] = 0.0
    return orc, fat, lng


@pytest.mark.parametrize("dims", LATTICES)
@pytest.mark.parametrize("kind", ["spread", "mild", "over", "one_fat", "one_lng", "one_small", "small_lng", "zeros"])
def test_dslash(gpu, oracle_cls, dims, kind):
    m = gpu
    orc, fat, lng = _scaled(m, oracle_cls, dims, kind)
    m.set_lattice(dims)
    m.load_fn_links(fat, lng)
    dense = m.gen_vector(dims, 5, m.EVENANDODD)
    points = np.zeros_like(dense)
    points[:: 97] = dense[:: 97]
    for src in (dense, points):
        for par in (m.EVEN, m.ODD, m.EVENANDODD):
            got = np.zeros_like(src)
            m.dslash_fn_field(src, got, par)
            want = orc.dslash(fat, lng, src, par)
            b = _site_bound(dims, fat, lng, src)
            assert np.all(np.linalg.norm(got - want, axis=1) <= TOL * b)


@pytest.mark.parametrize("nsrc", [1, 2, 5, 12])
def test_cg_with_one_large_link(gpu, oracle_cls, nsrc):
    """One link of 2^20: the solution solves the system on every site the link
    does not touch (at its own even end the rounding of the large products
    shows).  The iterated residual stops at 1e-12 |b|; the products of the
    operator, whose norm is about 10 there, keep the true one within 1e-11."""
    m = gpu
    dims, mass = LATTICES[0], 0.1
    U, orc, L = hisq_setup(m, oracle_cls, dims)
    fat, lng = L["fat"][0].copy(), L["lng"][0]
    fat[17, 2] *= 2.0 ** 20
    m.set_lattice(dims)
    m.load_fn_links(fat, lng)
    srcs = [m.gen_vector(dims, 5 + k, m.EVEN) for k in range(nsrc)]
    xs = [np.zeros_like(s) for s in srcs]
    qic = m.QuarkInvertControl(resid=1e-12, max=900, nrestart=5, parity=m.EVEN, prec=m.PREC_DOUBLE)
    m.ks_congrad_block_parity(srcs, xs, qic, mass)
    V2 = len(fat) // 2
    for b, x in zip(srcs, xs):
        r = b - (4 * mass ** 2 * x - orc.dslash(fat, lng, orc.dslash(fat, lng, x, m.ODD), m.EVEN))
        site = np.linalg.norm(r[:V2], axis=1)
        site[17] = 0.0
        assert np.linalg.norm(site) <= 1e-11 * np.linalg.norm(b[:V2])


def test_slots_keep_their_own_form(gpu, oracle_cls):
    """Slots with links of either kind side by side, and a slot reloaded."""
    m = gpu
    dims = LATTICES[0]
    src = m.gen_vector(dims, 5, m.EVENANDODD)
    m.set_lattice(dims)
    for slot, kind in ((0, "plain"), (1, "one_fat"), (0, "spread"), (1, "plain"), (0, "plain")):
        orc, fat, lng = _scaled(m, oracle_cls, dims, kind)
        m.load_fn_links(fat, lng, slot=slot)
        got = np.zeros_like(src)
        m.dslash_fn_field(src, got, m.EVENANDODD, slot)
        want = orc.dslash(fat, lng, src, m.EVENANDODD)
        assert np.all(np.linalg.norm(got - want, axis=1) <= TOL * _site_bound(dims, fat, lng, src))

def _free(dims, kind):
    """Links with zero entries: free, diagonal, real, or an SU(2) block and a phase."""
    V = int(np.prod(dims))
    rng = np.random.default_rng(4)
    M = np.zeros((V, 4, 3, 3), complex)
    if kind == "free":
        M[..., range(3), range(3)] = 1.0
    elif kind == "diagonal":
        M[..., range(3), range(3)] = np.exp(1j * rng.uniform(-3, 3, (V, 4, 3)))
    elif kind == "real":
        M[:] = np.linalg.qr(rng.standard_normal((V, 4, 3, 3)))[0]
    else:
        q = rng.standard_normal((V, 4, 4))
        q /= np.linalg.norm(q, axis=-1, keepdims=True)
        a, b = q[..., 0] + 1j * q[..., 1], q[..., 2] + 1j * q[..., 3]
        M[..., 0, 0], M[..., 0, 1], M[..., 1, 0], M[..., 1, 1], M[..., 2, 2] = a, b, -b.conj(), a.conj(), 1.0
    return np.ascontiguousarray(np.stack([M.real, M.imag], -1).reshape(V, 4, 18))


@pytest.mark.parametrize("dims", LATTICES)
@pytest.mark.parametrize("kind", ["free", "diagonal", "real", "block"])
def test_small_components_beside_large_ones(gpu, oracle_cls, dims, kind):
    """Links that do not mix all components: a component of 1e-20 beside one
    of 1 keeps its digits."""
    m = gpu
    orc = oracle_cls(dims)
    links = _free(dims, kind)
    fat, lng = links, -links / 24
    m.set_lattice(dims)
    m.load_fn_links(fat, lng)
    src = m.gen_vector(dims, 5, m.EVENANDODD).reshape(-1, 3, 2)
    scale = np.ones((3, 2))
    if kind == "real":
        scale[:, 1] = 1e-20      # imaginary parts
    else:
        scale[2] = 1e-20         # the third colour
        if kind != "block":
            scale[1] = 1e-30
    for s in (scale, 1.0 / scale):
        v = np.ascontiguousarray((src * s).reshape(-1, 6))
        got = np.zeros_like(v)
        m.dslash_fn_field(v, got, m.EVENANDODD)
        want = orc.dslash(fat, lng, v, m.EVENANDODD)
        # per component: 256 roundings of the largest term of its own scale (|v| <= 6, |U| <= 1, 16 terms)
        err = np.abs(got - want).reshape(-1, 3, 2)
        assert np.all(err <= TOL * 16 * 6 * s)
