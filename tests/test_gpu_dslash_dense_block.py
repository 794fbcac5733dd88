"""The FP64 D of 16 < warps per SM <= 20 with several sources, whose warps go
by source: lattices that lie in that window on the device at hand; and sites
that are not finite within solves, with each shape of the D."""
import itertools

import numpy as np
import pytest

from conftest import hisq_setup, rel

pytestmark = pytest.mark.gpu


def _warps(vh, nsrc):
    """Warps of a launch of eight sites a warp, in blocks of a multiple of nsrc warps."""
    mult = 2 if nsrc <= 2 else 1
    return -(-vh // (8 * mult)) * mult * nsrc


def _dims_in_window(nsrc):
    torch = pytest.importorskip("torch")
    sm = torch.cuda.get_device_properties(0).multi_processor_count
    ext = range(4, 20, 2)
    for d in itertools.product(ext, ext, ext, range(4, 32, 2)):
        if d[0] <= d[1] <= d[2] <= d[3] and len(set(d)) > 2 and 16 * sm < _warps(int(np.prod(d)) // 2, nsrc) <= 20 * sm:
            return d
    raise AssertionError("no lattice in the window for %d SMs" % sm)


@pytest.mark.parametrize("nsrc", [1, 2, 3, 4])
def test_block_solve(gpu, oracle_cls, nsrc):
    m = gpu
    dims = _dims_in_window(nsrc)
    U, orc, L = hisq_setup(m, oracle_cls, dims)
    fat, lng = L["fat"][0], L["lng"][0]
    m.set_lattice(dims)
    m.load_fn_links(fat, lng)
    srcs = [m.gen_vector(dims, 60 + k, m.EVEN) for k in range(nsrc)]
    qic = m.QuarkInvertControl(resid=1e-9, max=400, nrestart=5, parity=m.EVEN, prec=m.PREC_DOUBLE)
    xs = [np.zeros_like(s) for s in srcs]
    it, per = m.ks_congrad_block_parity(srcs, xs, qic, 0.1)
    V2 = len(fat) // 2
    for k in range(nsrc):
        Dx = orc.dslash(fat, lng, orc.dslash(fat, lng, xs[k], m.ODD), m.EVEN)
        r = srcs[k] - (4 * 0.1 ** 2 * xs[k] - Dx)
        # the iterated residual stops the solve; the true one is within 1e-12 |b| of it in FP64
        assert per[k].converged == 1
        assert np.linalg.norm(r[:V2]) <= (1e-9 + 1e-12) * np.linalg.norm(srcs[k][:V2])


# four threads per site; the same in the window; one thread per site
@pytest.mark.parametrize("dims", [(6, 4, 10, 12), (12, 12, 12, 24), (16, 16, 18, 36)])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_not_finite_in_solves(gpu, oracle_cls, dims, bad):
    """A guess with one component that is not finite: the CG returns it as it
    is, with a residual that is not finite, and M^-1 carries it to the odd sites
    whose D reads it and to no others."""
    m = gpu
    mass = 0.1
    U, orc, L = hisq_setup(m, oracle_cls, dims)
    fat, lng = L["fat"][0], L["lng"][0]
    m.set_lattice(dims)
    m.load_fn_links(fat, lng)
    src = m.gen_vector(dims, 5, m.EVENANDODD)
    guess = m.gen_vector(dims, 6, m.EVEN)
    guess[7, 3] = bad
    qic = m.QuarkInvertControl(resid=1e-9, max=50, nrestart=2, parity=m.EVEN, prec=m.PREC_DOUBLE)
    x = guess.copy()
    m.ks_congrad_parity(src, x, qic, mass)
    assert np.array_equal(x, guess, equal_nan=True) and not np.isfinite(qic.final_rsq)
    x = guess.copy()
    m.mat_invert_uml_field(src, x, qic, mass)
    V2 = len(fat) // 2
    assert np.array_equal(x[:V2], guess[:V2], equal_nan=True)
    with np.errstate(all="ignore"):
        want = (src - orc.dslash(fat, lng, guess, m.ODD)) / (2 * mass)
    ok = np.isfinite(want[V2:])
    assert 0 < (~ok).sum() <= 16 * 6 and np.array_equal(np.isfinite(x[V2:]), ok)
    assert rel(x[V2:][ok], want[V2:][ok]) < 1e-13
