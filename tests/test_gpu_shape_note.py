"""MKS_SHAPE entries for the FP64 D, whose shape is a rule's: accepted, reported
once, without effect; entries for other precisions are not reported."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, numpy as np, milc_qcd_gb300 as m
dims = (6, 4, 10, 12)
m.init(0)
m.set_lattice(dims)
U = m.gen_thin_links(dims, 11, 0.3)
m.load_fn_links(U, U)
v = m.gen_vector(dims, 5, m.EVENANDODD)
out = np.zeros_like(v)
for _ in range(2):
    m.dslash_fn_field(v, out, m.EVENANDODD)
print(out.tobytes().hex()[:4096])
"""


def _run(shape):
    env = dict(os.environ, MKS_SHAPE=shape, PYTHONPATH=ROOT)
    p = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    return p.stdout, p.stderr


def test_note(gpu):
    want, err = _run("1:1:1:1:128,d0:1:1:1:256")
    assert "MKS_SHAPE" not in err
    for entry in ("2:1:1:1:128", "e2:2:1:2:256"):
        got, err = _run("1:1:1:1:128," + entry)
        assert got == want
        assert err.count("MKS_SHAPE") == 1 and '"%s"' % entry in err
