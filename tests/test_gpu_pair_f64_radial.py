"""The radial functions of the FP64 pair sum and of its derivatives, one pair
at a time against 40-digit values: forces, energies, Hessian-vector products
and derivatives with respect to lambda over the whole range of each table and
past its ends.  Separations are multiples of 2^-20 in a box of 16 and the other
lengths powers of two (alpha: 0.5 or 0.75), so that the arguments alpha^2 r^2
and r^2/lambda^2 are exact and only the functions are looked at."""
import decimal
from decimal import Decimal as D

import numpy as np
import pytest

import tcp_allpair_gb300 as T

pytestmark = pytest.mark.gpu

decimal.getcontext().prec = 70
PI = D("3.14159265358979323846264338327950288419716939937510582097494459230781640629")
SPI = PI.sqrt()
ULP = 2.0 ** -52
EPS = D(T.EPS)


def erfc(z):
    """1 - 2/sqrt(pi) e^{-z^2} sum 2^n z^(2n+1)/(2n+1)!!: 40 digits are left for z < 8."""
    s = t = z
    n = 0
    while t > s * D(10) ** -69:
        n += 1
        t = t * 2 * z * z / (2 * n + 1)
        s += t
    return 1 - 2 / SPI * (-z * z).exp() * s


def context(ei, alpha, lam):
    s = T.make_system(2, seed=1, alpha_rc=3.1)
    p = T.params_for(s, precision="fp64", ei=ei, recip="none")
    for d in range(3):
        p.box[d] = 16.0
    p.rc, p.a, p.lambda_ei, p.rs = 7.9, alpha, lam, lam
    return T.Context(p, 1, 1)


def pair(c, r):
    """(energy, radial force on the second particle, radial and transverse H.w, dF/dlambda . w, dE/dlambda)"""
    x, w = np.zeros((2, 3)), np.zeros((2, 3))
    x[1, 0] = r
    w[1, :2] = 1.0
    c.upload(x=x)
    u = c.Force_direct_self()
    f = c.download(x=False, v=False)[2]
    hw, dfw = c.hvp(w)
    assert f[0, 0] == -f[1, 0] and np.all(hw[0] == -hw[1])
    return u, f[1, 0], hw[1, 0], hw[1, 1], dfw, c.adjoint_energy()[1]


def separations(lo, hi, seed):
    """log-uniform in r, r < 7.9, multiples of 2^-20"""
    r = np.exp(np.random.default_rng(seed).uniform(np.log(lo), np.log(min(hi, 7.89)), 60))
    return np.round(r * 2.0 ** 20) / 2.0 ** 20


def near(got, want, bound):
    assert abs(D(float(got)) - want) <= D(bound), (got, want, float(abs(D(float(got)) - want)) / bound)


def ewald(r, a):
    """U, -U'/r, U'' of erfc(ar)/r"""
    u = erfc(a * r) / r
    g = 2 * a / SPI * (-(a * r) ** 2).exp()
    return u, (u + g) / r ** 2, 2 * (u + g) / r ** 2 + 2 * a * a * g


# Of a function, 4 + x ulps: an argument rounded to FP64 makes e^{-x} uncertain
# by x/2, and the FP32 terms and the roundings of the sum weigh less than that.
# Of the constants and products around it, another 4.
def ulps(arg):
    return (8.0 + float(arg)) * ULP


@pytest.mark.parametrize("alpha", [0.5, 0.75])           # up to alpha^2 r^2 = 15.6 and 35
def test_ewald(alpha):
    a = D(alpha)
    with context("coulomb", alpha, 0.5) as c:
        c.EWALD_SELF()
        for r in separations(0.08 / alpha, 8.0, 3):
            e, f, hr, ht = pair(c, r)[:4]
            u, g1, d2 = ewald(D(r), a)
            tol = ulps((alpha * r) ** 2)
            near(e, -u, tol * float(u))
            near(f, -EPS * g1 * D(r), tol * T.EPS * float(g1) * r)
            near(ht, EPS * g1, tol * T.EPS * float(g1))
            near(hr, -EPS * d2, tol * T.EPS * float(d2 + 2 * g1))     # as the difference of two terms


def kelbg(r, lam):
    """U, -U'/r, U'' of the e-i term, d/dlambda of U and of -U'"""
    y = (r / lam) ** 2
    e, q = (-y).exp(), erfc(r / lam)
    u = SPI / lam * q - e / r                                        # U' = e^{-y}/r^2
    return u, -e / r ** 3, -2 * e * (1 / r ** 3 + 1 / (lam ** 2 * r)), -SPI * q / lam ** 2, -2 * e / lam ** 3


def deutsch(r, lam):
    s = r / lam
    e = (-s).exp()
    return (-e / r, -e * (1 + s) / r ** 3, -e * (2 + 2 * s + s * s) / r ** 3, -e / lam ** 2, -e / lam ** 3)


# The last octaves of the tables are coarser: from r^2/lambda^2 = 32 on (Kelbg,
# where the functions are below 1e-14 of the Coulomb term) and from r/rs = 22.6
# and 32 on (Deutsch, 1e-10 and 1e-14).
def far(ei, r, lam):
    if ei == "kelbg":
        return 5e-14 if (r / lam) ** 2 >= 32.0 else 0.0
    z = (r / lam) ** 2
    return 2.6e-11 if z >= 1024.0 else (2.4e-12 if z >= 512.0 else 0.0)


@pytest.mark.parametrize("ei,lam", [("kelbg", 0.5), ("kelbg", 1.0), ("deutsch", 0.25), ("deutsch", 0.5), ("deutsch", 1.0)])
def test_electron_ion(ei, lam):
    a = D(0.5)
    with context(ei, 0.5, lam) as c:
        c.EWALD_SELF()
        for r in separations(0.1 * lam, 7.9 * lam if ei == "kelbg" else 45.0 * lam, 4):
            e, f, hr, ht, dfw, dl = pair(c, r)
            x, arg = (0.5 * r) ** 2, (r / lam) ** (2 if ei == "kelbg" else 1)
            we, wi = ulps(x), ulps(arg) + far(ei, r, lam)
            u, g1, d2 = ewald(D(r), a)
            ui, gi, d2i, li, lf = (kelbg if ei == "kelbg" else deutsch)(D(r), D(lam))
            # qq = -1; the terms' errors relative to themselves
            near(e, -(u + ui), we * float(u) + wi * abs(float(ui)))
            near(f, -EPS * (g1 + gi) * D(r), T.EPS * r * (we * float(g1) + wi * abs(float(gi))))
            near(ht, EPS * (g1 + gi), T.EPS * (we * float(g1) + wi * abs(float(gi))))
            near(hr, -EPS * (d2 + d2i), T.EPS * (we * float(d2 + 2 * g1) + wi * abs(float(d2i + 2 * gi))))
            near(dl, -EPS * li, T.EPS * wi * abs(float(li)))
            near(dfw, -EPS * lf, T.EPS * wi * abs(float(lf)))
