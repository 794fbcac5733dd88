"""The FP64 D with four threads per site on either side of the line where its
warps no longer fit the chip at 16 per SM (the kernel of 96 registers, whose
FP64 tail takes one colour per thread)."""
import numpy as np
import pytest

from conftest import hisq_setup, rel

pytestmark = pytest.mark.gpu

# 18,816, 20,736 and 21,000 sites of a parity: 2352, 2592 and 2625 warps of
# eight sites against 2432; the last ends in an incomplete block
LATTICES = [(14, 12, 14, 16), (12, 12, 12, 24), (14, 10, 10, 30)]


@pytest.mark.parametrize("dims", LATTICES)
@pytest.mark.parametrize("nsrc", [1, 3, 4, 5])
def test_block_solve(gpu, oracle_cls, dims, nsrc):
    m = gpu
    U, orc, L = hisq_setup(m, oracle_cls, dims)
    fat, lng = L["fat"][0], L["lng"][0]
    m.set_lattice(dims)
    m.load_fn_links(fat, lng)
    srcs = [m.gen_vector(dims, 50 + k, m.EVEN) for k in range(nsrc)]
    qic = m.QuarkInvertControl(resid=1e-9, max=400, nrestart=5, parity=m.EVEN, prec=m.PREC_DOUBLE)
    xs = [np.zeros_like(s) for s in srcs]
    it, per = m.ks_congrad_block_parity(srcs, xs, qic, 0.1)
    for k in sorted({0, nsrc - 1}):
        V2 = srcs[k].shape[0] // 2
        Dx = orc.dslash(fat, lng, orc.dslash(fat, lng, xs[k], m.ODD), m.EVEN)
        r = srcs[k] - (4 * 0.1 ** 2 * xs[k] - Dx)
        # the iterated residual stops the solve; the true one is within
        # 1e-12 |b| of it in FP64
        assert np.linalg.norm(r[:V2]) <= (1e-9 + 1e-12) * np.linalg.norm(srcs[k][:V2])
        x = np.zeros_like(srcs[k])
        n = m.ks_congrad_parity(srcs[k], x, qic, 0.1)
        assert per[k].converged == 1 and per[k].final_iters == n
        assert rel(xs[k], x) < 1e-12
