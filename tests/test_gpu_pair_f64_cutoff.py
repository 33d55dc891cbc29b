"""Pairs a relative 1e-8 inside the cut-off, where alpha^2 rc^2 is a power of
two and with it an end of the radial table of the FP64 pair sum: their Ewald
term, erfc(2) = 5e-3 of the Coulomb one at alpha rc = 2, counts in forces and
derivatives."""
import math

import numpy as np
import pytest

import tcp_allpair_gb300 as T

pytestmark = pytest.mark.gpu

L = 10.0
REL = 1e-12      # r from FP64 positions, 1e-15, times the slope of erfc, 2 (alpha r)^2 = 32 at most, and ten times that


@pytest.mark.parametrize("alpha_rc", [2.0, 4.0])
@pytest.mark.parametrize("k", [0, 2, 9, 16, 25, 35, 57, 63])
def test_pair_just_inside(alpha_rc, k):
    s = T.make_system(2, seed=1, alpha_rc=3.1)
    p = T.params_for(s, precision="fp64", ei="coulomb", recip="none")
    rc = 4.0 + k / 64.0 * 0.95
    a = alpha_rc / rc
    for d in range(3):
        p.box[d] = L
    p.rc, p.a = rc, a
    x = np.zeros((2, 3))
    x[1] = rc * (1.0 - 1e-8) * np.array([0.6, 0.48, 0.64])
    r = math.sqrt(float(np.sum(x[1] ** 2)))
    g = 2.0 * a / math.sqrt(math.pi) * math.exp(-(a * r) ** 2)
    u = math.erfc(a * r) / r                             # energy and -dU/dr of unit charges
    du = -(u + g) / r
    d2u = (2.0 * u + 2.0 * g) / r ** 2 + 2.0 * a * a * g
    qq = p.q[0] * p.q[1]
    w = np.zeros((2, 3))
    w[1] = x[1] / r
    with T.Context(p, 1, 1) as c:
        c.EWALD_SELF()
        c.upload(x=x)
        assert c.Force_direct_self() == pytest.approx(qq * u, rel=REL, abs=0.0)
        f = c.download(x=False, v=False)[2]
        hw = c.hvp(w)[0]
    assert f[1] == pytest.approx(-T.EPS * qq * du * w[1], rel=REL, abs=0.0)
    assert f[0] == pytest.approx(-f[1], rel=REL, abs=0.0)
    assert hw[1] == pytest.approx(T.EPS * qq * d2u * w[1], rel=REL, abs=0.0)
