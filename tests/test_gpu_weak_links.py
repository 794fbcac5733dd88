"""Links close to ones that do not mix all components (weak and nearly real
fields): every real and imaginary part of D is as accurate as the terms that
make it up, and so is the gauge force of weak fields (csrc/mks_fixed.cuh:
FxUneven)."""
import numpy as np
import pytest

from conftest import hisq_setup, rel
from test_gpu_dslash_links import LATTICES, TOL, _order
from test_gpu_uneven_links import _links, _matrices, _weak

pytestmark = pytest.mark.gpu


def _part_bounds(dims, fat, lng, src):
    """Sums of |products| that make up each real and imaginary part of D."""
    order, grid = _order(dims), (dims[3], dims[2], dims[1], dims[0])

    def g(a):
        out = np.empty_like(a)
        out[order] = a
        return out.reshape(grid + a.shape[1:])

    v = g(np.abs(src.reshape(-1, 3, 2)))
    total = 0.0

    def mul(Ur, Ui, w):
        m = lambda U, x: np.einsum("...ij,...j->...i", U, x)
        return np.stack([m(Ur, w[..., 0]) + m(Ui, w[..., 1]), m(Ur, w[..., 1]) + m(Ui, w[..., 0])], -1)

    for mu in range(4):
        ax = 3 - mu
        for links, k in ((fat, 1), (lng, 3)):
            U = g(_matrices(links)[:, mu])
            r, i = np.abs(U.real), np.abs(U.imag)
            total = total + mul(r, i, np.roll(v, -k, ax))
            total = total + np.roll(mul(r.swapaxes(-1, -2), i.swapaxes(-1, -2), v), k, ax)
    return total.reshape((-1, 3, 2))[order]


def _field(m, dims, kind, eps):
    if kind == "weak":
        return _weak(m, dims, eps)
    rng = np.random.default_rng(9)
    V = int(np.prod(dims))
    R = np.linalg.qr(rng.standard_normal((V, 4, 3, 3)))[0]
    return _links(R + 1j * eps * rng.standard_normal(R.shape))


# 0.3 and 0.02 keep the integer form
@pytest.mark.parametrize("dims", LATTICES[:2])
@pytest.mark.parametrize("kind,eps", [("weak", 0.3), ("weak", 0.02), ("weak", 1e-3), ("weak", 1e-5), ("weak", 1e-7),
                                      ("real", 0.3), ("real", 1e-4), ("real", 1e-9)])
def test_parts_of_dslash(gpu, oracle_cls, dims, kind, eps):
    m = gpu
    orc = oracle_cls(dims)
    fat = _field(m, dims, kind, eps)
    lng = -fat / 24
    m.set_lattice(dims)
    m.load_fn_links(fat, lng)
    base = m.gen_vector(dims, 5, m.EVENANDODD).reshape(-1, 3, 2)
    scale = np.array([[1.0, 1.0], [1e-20, 1e-20], [1e-10, 1e-10]]) if kind == "weak" else \
        np.array([[1.0, 1e-20]] * 3)
    for s in (np.ones((3, 2)), scale):
        src = np.ascontiguousarray((base * s).reshape(-1, 6))
        got = np.zeros_like(src)
        m.dslash_fn_field(src, got, m.EVENANDODD)
        want = orc.dslash(fat, lng, src, m.EVENANDODD)
        assert np.all(np.abs(got - want).reshape(-1, 3, 2) <= TOL * _part_bounds(dims, fat, lng, src))


@pytest.mark.parametrize("eps", [1e-3, 1e-5, 1e-7])
def test_gauge_force(gpu, oracle_cls, eps):
    from oracle.oracle import GaugeOracle
    m = gpu
    dims = (6, 4, 6, 10)
    U = _weak(m, dims, eps)
    zero = np.zeros((U.shape[0], 4, 10))
    m.set_lattice(dims)
    m.gauge_load(U)
    m.mom_load(zero)
    m.gauge_force(0.02, 7.4, 0.89, 3)
    got, want = m.mom_get(), GaugeOracle(oracle_cls(dims)).force(U, 0.02, 7.4, 0.89, 3, zero)
    # 54 paths of up to five products; their sum cancels to about a tenth of its terms
    assert rel(got[..., :9], want[..., :9]) < 4096 * 2.0 ** -53


def test_smeared_fields_keep_their_form(gpu, oracle_cls):
    """The rules leave smeared fields of the tests' and the benchmark's kind in
    the integer form: a D of them takes four threads per site on small lattices."""
    import ctypes
    m = gpu
    dims = LATTICES[0]
    lib = m._lib.load()
    for a in (0.1, 0.2, 0.3, 1.0, 10.0):
        U, orc, L = hisq_setup(m, oracle_cls, dims, a=a)
        m.set_lattice(dims)
        m.load_fn_links(L["fat"][0], L["lng"][0])
        v = m.gen_vector(dims, 5, m.EVENANDODD)
        m.dslash_fn_field(v, np.zeros_like(v), m.EVENANDODD)
        G = ctypes.c_int()
        m.check(lib.mks_tuned_shape(m.PREC_DOUBLE, 1, ctypes.byref(G), None, None), "mks_tuned_shape")
        assert G.value == 4, a
