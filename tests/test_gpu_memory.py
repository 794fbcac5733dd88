"""Calls under a limit on the library's device memory (MKS_MEM_LIMIT, in MiB):
what the library keeps for speed alone -- the links' integer copies -- is left
out or given back before a call is refused, and the results stay the same."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, rel

pytestmark = pytest.mark.gpu

# 16^3x32, 65,536 sites of a parity: a slot takes 252 MiB in FP64, FP32 and
# FP16, its integer copies 144 MiB, a load's staging 144 MiB (400 in all with
# small buffers), a field of one parity 3 MiB
CHILD = """
import sys, numpy as np
import milc_qcd_gb300 as m
what, out = sys.argv[1:3]
dims = (16, 16, 16, 32)
m.init(0)
m.set_lattice(dims)
U = m.apply_phases(dims, m.gen_thin_links(dims, 11, 0.3))
vec = lambda k, p: m.gen_vector(dims, k, p)
qic = lambda prec: m.QuarkInvertControl(resid=1e-9, max=400, nrestart=5, parity=m.EVEN, prec=prec)
res = []
def solve(n, prec):
    xs = [np.zeros((U.shape[0], 6)) for _ in range(n)]
    m.ks_congrad_block_parity([vec(k, m.EVEN) for k in range(n)], xs, qic(prec), 0.1)
    return xs
if what in ("hisq", "force", "gauge"):
    mom = np.zeros((U.shape[0], 4, 10))
    if what == "hisq":
        m.load_hisq_links(U, (0.0, -0.1))
        res += [a for slot in (0, 1) for a in m.get_fn_links(slot)]
    elif what == "force":
        for action in ("hisq", "asqtad"):
            getattr(m, "load_%s_links" % action)(U)
            mom[:] = 0
            m.eo_fermion_force_multi(0.1, [1.0, -0.5], [vec(k, m.EVENANDODD) for k in range(2)], mom, action=action)
            res.append(mom.copy())
    else:
        m.gauge_load(U)
        m.mom_load(mom)
        m.gauge_force(0.01, 7.4, 0.89, 3)
        res += [m.mom_get(), np.full_like(mom, m.gauge_action(7.4, 0.89, 3))]
else:
    m.load_fn_links(U, U / 24)
if what == "dslash":
    res.append(np.zeros((U.shape[0], 6)))
    m.dslash_fn_field(vec(1, m.EVENANDODD), res[0], m.EVENANDODD)
if what == "multishift":
    res = [np.zeros((U.shape[0], 6)) for _ in range(4)]
    m.ks_multicg_offset_field(vec(1, m.EVEN), res, [0.04, 0.1, 0.3, 1.0], qic(m.PREC_DOUBLE))
elif what == "uml":
    res = [np.zeros((U.shape[0], 6))]
    m.mat_invert_uml_field(vec(1, m.EVENANDODD), res[0], qic(m.PREC_SINGLE), 0.1)
elif what == "solve":
    res += solve(8, m.PREC_DOUBLE)
    res += solve(8, m.PREC_SINGLE)
np.save(out, np.stack(res))
"""


def _run(what, limit, path):
    env = dict(os.environ, MKS_MEM_LIMIT=str(limit), MKS_TUNE="0", PYTHONPATH=ROOT)
    p = subprocess.run([sys.executable, "-c", CHILD, what, str(path)], cwd=ROOT, env=env, capture_output=True,
                       text=True, timeout=300)
    return p.returncode, p.stderr, (np.load(path) if p.returncode == 0 else None)


# the least limits under which the calls passed before there were integer
# copies (to 16 MiB), and one where the copies fit beside the links but not
# beside a solve's fields as well.  D: 256 roundings; solutions: residuals of
# 1e-9 on either side, an operator between 0.04 and 16; links, force and paths:
# three levels of 18 roundings, which the projection's derivative multiplies
# by less than 16
@pytest.mark.parametrize("what,limits,tol", [
    ("dslash", [416], 256 * 2.0 ** -53), ("multishift", [416, 560], 1e-6), ("uml", [416, 560], 1e-6),
    ("solve", [576, 640], 1e-6),
    ("hisq", [992], 1024 * 2.0 ** -53), ("force", [976], 1024 * 2.0 ** -53), ("gauge", [304], 1024 * 2.0 ** -53)])
def test_limit(gpu, tmp_path, what, limits, tol):
    rc, err, want = _run(what, 0, tmp_path / "a.npy")
    assert rc == 0, err
    for limit in limits:
        rc, err, got = _run(what, limit, tmp_path / "b.npy")
        assert rc == 0, err
        assert all(rel(a, b) < tol for a, b in zip(got, want)), limit


def test_limit_holds(gpu, tmp_path):
    rc, err, _ = _run("dslash", 300, tmp_path / "a.npy")
    assert rc != 0 and "mks_load_fn_links" in err
