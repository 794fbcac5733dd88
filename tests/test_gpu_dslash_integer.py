"""The FP64 D_eo in integer arithmetic (csrc/mks_fixed.cuh) at the edges of its
format: values of widely different size, zeros, scales near the ends of the
FP64 range, infinities and NaNs in vectors and links, fields on an 8-byte
boundary, lattices on either side of the four-threads-per-site rule, and the
source counts of the FP64 block solver."""
import ctypes

import numpy as np
import pytest

from conftest import hisq_setup, rel

pytestmark = pytest.mark.gpu

# 4^4: one partial block; 6x4x10x12: ragged, four threads per site;
# 16x16x18x36: above the rule's line (82,944 sites of a parity)
LATTICES = [(4, 4, 4, 4), (6, 4, 10, 12), (16, 16, 18, 36)]


def _setup(m, oracle_cls, dims):
    U, orc, L = hisq_setup(m, oracle_cls, dims)
    m.set_lattice(dims)
    m.load_fn_links(L["fat"][0], L["lng"][0])
    return orc, L["fat"][0], L["lng"][0]


def _d(m, src, parity=None):
    out = np.zeros_like(src)
    m.dslash_fn_field(src, out, m.EVENANDODD if parity is None else parity)
    return out


def _neighbour_norms(dims, src):
    """Sum over a site's 16 neighbours of |v|, in MILC's site order."""
    nx, ny, nz, nt = dims
    t, z, y, x = np.meshgrid(np.arange(nt), np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    odd = ((x + y + z + t) & 1).reshape(-1)
    order = np.concatenate([np.nonzero(odd == 0)[0], np.nonzero(odd == 1)[0]])
    n = np.empty(len(order))
    n[order] = np.linalg.norm(src, axis=1)
    n = n.reshape(nt, nz, ny, nx)
    s = sum(np.roll(n, k, axis) for axis in range(4) for k in (1, -1, 3, -3))
    return s.reshape(-1)[order]


def _assert_close(dims, got, want, src):
    # FP64 sums of 192 products per component on either side, |U| <= 1.5: 256 roundings of 2^-53
    bound = 256 * 2.0 ** -53 * 1.5 * _neighbour_norms(dims, src)
    assert np.all(np.linalg.norm(got - want, axis=1) <= bound)


@pytest.mark.parametrize("dims", LATTICES)
def test_sites_of_very_different_size(gpu, oracle_cls, dims):
    m = gpu
    orc, fat, lng = _setup(m, oracle_cls, dims)
    src = m.gen_vector(dims, 5, m.EVENANDODD)
    rng = np.random.default_rng(1)
    src *= 10.0 ** rng.uniform(-30, 30, (src.shape[0], 1))        # per site
    src *= 10.0 ** rng.uniform(-8, 0, src.shape)                   # and per component
    src[rng.uniform(size=src.shape[0]) < 0.3] = 0.0
    _assert_close(dims, _d(m, src), orc.dslash(fat, lng, src, m.EVENANDODD), src)


@pytest.mark.parametrize("dims", LATTICES[:2])
def test_point_source_and_zero(gpu, oracle_cls, dims):
    m = gpu
    orc, fat, lng = _setup(m, oracle_cls, dims)
    src = np.zeros((int(np.prod(dims)), 6))
    assert not _d(m, src).any()
    src[3, 2] = 1.0
    got, want = _d(m, src), orc.dslash(fat, lng, src, m.EVENANDODD)
    assert np.array_equal(got == 0, want == 0)
    _assert_close(dims, got, want, src)


def test_power_of_two_scales(gpu, oracle_cls):
    """Blocks carry their exponent, so a power of two goes through exactly;
    down in the subnormals the result is rounded once."""
    m = gpu
    dims = LATTICES[1]
    _setup(m, oracle_cls, dims)
    src = m.gen_vector(dims, 6, m.EVENANDODD)
    ref = _d(m, src)
    for k in (-1000, -300, 300, 1000):
        assert np.array_equal(_d(m, np.ldexp(src, k)), np.ldexp(ref, k)), k
    tiny = np.ldexp(src, -1050)          # a few bits of each input are left
    got, want = _d(m, tiny), np.ldexp(_d(m, np.ldexp(tiny, 900)), -900)
    assert np.abs(got - want).max() <= 2 * 5e-324


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_not_finite_vectors(gpu, oracle_cls, bad):
    m = gpu
    dims = LATTICES[1]
    orc, fat, lng = _setup(m, oracle_cls, dims)
    src = m.gen_vector(dims, 7, m.EVENANDODD)
    src[17, 4] = bad
    src[-5, 1] = bad
    with np.errstate(all="ignore"):
        got, want = _d(m, src), orc.dslash(fat, lng, src, m.EVENANDODD)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    assert np.array_equal(got[inf], want[inf])
    ok = np.isfinite(want)
    assert np.all(np.isfinite(got[ok])) and rel(got[ok], want[ok]) < 1e-13


def test_not_finite_link(gpu, oracle_cls):
    m = gpu
    dims = LATTICES[1]
    orc, fat, lng = _setup(m, oracle_cls, dims)
    fat = fat.copy()
    fat[11, 2, 5] = np.nan
    m.load_fn_links(fat, lng)
    src = m.gen_vector(dims, 8, m.EVENANDODD)
    got, want = _d(m, src), orc.dslash(fat, lng, src, m.EVENANDODD)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.isnan(want).any()
    ok = ~np.isnan(want)
    assert rel(got[ok], want[ok]) < 1e-13


@pytest.mark.parametrize("parity", ["EVEN", "ODD", "EVENANDODD"])
def test_device_fields_on_an_8_byte_boundary(gpu, oracle_cls, parity):
    torch = pytest.importorskip("torch")
    m = gpu
    dims = LATTICES[1]
    _setup(m, oracle_cls, dims)
    src = m.gen_vector(dims, 9, m.EVENANDODD)
    par = getattr(m, parity)
    ref = _d(m, src, par)
    n = src.size
    a, b = torch.zeros(n + 1, dtype=torch.float64).cuda(), torch.zeros(n + 1, dtype=torch.float64).cuda()
    a[1:] = torch.from_numpy(src.reshape(-1))
    torch.cuda.synchronize()
    lib = m._lib.load()
    m.check(lib.mks_dslash_fn_field_dev(a[1:].data_ptr(), b[1:].data_ptr(), par, 0), "mks_dslash_fn_field_dev")
    assert np.array_equal(b[1:].cpu().numpy().reshape(src.shape), ref) and float(b[0]) == 0.0


@pytest.mark.parametrize("dims", LATTICES[1:])
@pytest.mark.parametrize("nsrc", [2, 5, 9, 16])
def test_fp64_block_solver_source_counts(gpu, oracle_cls, dims, nsrc):
    """Integer sums do not depend on the launch shape: each source of an FP64
    block solve takes the iterations of its own solve."""
    m = gpu
    _setup(m, oracle_cls, dims)
    srcs = [m.gen_vector(dims, 40 + k, m.EVEN) for k in range(nsrc)]
    qic = m.QuarkInvertControl(resid=1e-9, max=400, nrestart=5, parity=m.EVEN, prec=m.PREC_DOUBLE)
    xs = [np.zeros_like(s) for s in srcs]
    it, per = m.ks_congrad_block_parity(srcs, xs, qic, 0.1)
    for k in (0, nsrc // 2, nsrc - 1):
        x = np.zeros_like(srcs[k])
        n = m.ks_congrad_parity(srcs[k], x, qic, 0.1)
        assert per[k].converged == 1 and per[k].final_iters == n
        assert rel(xs[k], x) < 1e-12
