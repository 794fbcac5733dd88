"""Grid sums whose block totals cancel: what is left is good to 2^-63 of the
largest total (and to FP64 rounding), where FP64 sums keep 2^-53 of it."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (8, 8, 8, 8)   # 2048 sites of a parity: eight blocks of 256


def _plaquettes(m, values):
    """A field whose only plaquettes, 3 * value each, lie in the (x, y) planes
    of even sites in as many blocks."""
    nx, ny, nz, nt = DIMS

    def index(x, y, t):
        return ((x + nx * (y + ny * nz * t)) >> 1) + (x + y + t) % 2 * (nx * ny * nz * nt // 2)

    U = np.zeros((nx * ny * nz * nt, 4, 18))
    one = np.zeros(18)
    one[[0, 8, 16]] = 1.0
    for t, v in enumerate(values):           # z = 0; time slice t is block t of the even sites
        x = t % 2                            # an even corner
        U[index(x, 0, t), 0] = v * one
        U[index(x + 1, 0, t), 1] = one
        U[index(x, 1, t), 0] = one
        U[index(x, 0, t), 1] = one
    return U


@pytest.mark.parametrize("values", [
    [2.0 ** 14, -2.0 ** 13, -2.0 ** 13, 2.0 ** -60],
    [2.0 ** 14, -2.0 ** 13, -2.0 ** 13, -2.0 ** -60],
    [2.0 ** 32, -2.0 ** 31, -2.0 ** 31, 1.0 + 2.0 ** -52],
    [-2.0 ** 96, 2.0 ** 95, 2.0 ** 95, -2.0 ** -40, 2.0 ** -41],
    [2.0 ** 400, -2.0 ** 399, -2.0 ** 399, 2.0 ** -500],
    [2.0 ** 400, -2.0 ** 399, -2.0 ** 399],
    [1.0, 2.0 ** -53, 2.0 ** -100, 2.0 ** -160],
    [2.0 ** 200, -2.0 ** 200, 2.0 ** 100, -2.0 ** 100, 3.0, -2.0 ** -300],
])
def test_cancelling_blocks(gpu, values):
    m = gpu
    m.set_lattice(DIMS)
    for sign in (1.0, -1.0):
        v = [sign * x for x in values]
        m.gauge_load(_plaquettes(m, v))
        ss, st = m.plaquette()
        want = 3.0 * math.fsum(v)
        norm = 3.0 * np.prod(DIMS)
        assert st == 0.0
        assert abs(ss * norm - want) <= 3.0 * 2.0 ** -62 * max(map(abs, v)) + 4 * 2.0 ** -53 * abs(want)
