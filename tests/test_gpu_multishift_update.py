"""The multi-shift update kernel over its launch shapes: one, two or four
groups of shifts per tile of 32 sites (by lattice and shift count), a last
tile that is not full, up to the largest number of shifts, and the shadows of
the lowest search direction (FP16, integers).  Every shift's FP64 residual is
recomputed with the oracle's D."""
import numpy as np
import pytest

from conftest import hisq_setup

pytestmark = pytest.mark.gpu

# 6^4: 648 sites of a parity, 20 tiles and a quarter; four groups from 8 shifts on
# 14x12^2x28: two groups; 16^3x32: one group
SHAPES = [((6, 6, 6, 6), 1), ((6, 6, 6, 6), 5), ((6, 6, 6, 6), 32), ((14, 12, 12, 28), 9), ((16, 16, 16, 32), 4)]


@pytest.mark.parametrize("prec", ["PREC_DOUBLE", "PREC_SINGLE", "PREC_HALF"])
@pytest.mark.parametrize("dims,noff", SHAPES)
@pytest.mark.parametrize("resid", [1e-6, 1e-9])
def test_update_shapes(gpu, oracle_cls, dims, noff, prec, resid):
    m = gpu
    U, orc, L = hisq_setup(m, oracle_cls, dims)
    fat, lng = L["fat"][0], L["lng"][0]
    m.set_lattice(dims)
    m.load_fn_links(fat, lng)
    b = m.gen_vector(dims, 71, m.ODD)
    offs = np.logspace(-2, 1, noff)[::-1]     # the lowest shift comes last
    psim = [np.zeros_like(b) for _ in offs]
    qic = m.QuarkInvertControl(resid=resid, max=1000, nrestart=5, parity=m.ODD, prec=getattr(m, prec))
    it, per = m.ks_multicg_offset_field(b, psim, offs, qic)
    V2 = b.shape[0] // 2
    # FP64 stops on the iterated residual, as MILC does
    limit = resid * (1.5 if prec == "PREC_DOUBLE" else 1.01)
    for j in sorted({0, noff // 2, noff - 1}):
        Dx = orc.dslash(fat, lng, orc.dslash(fat, lng, psim[j], m.EVEN), m.ODD)
        r = b - (offs[j] * psim[j] - Dx)
        assert np.linalg.norm(r[V2:]) <= limit * np.linalg.norm(b[V2:]), j
        assert per[j].converged == 1 and not psim[j][:V2].any()
