"""The SPME chain on the meshes that spme_fft.cu transforms (32, 48, 64, 96,
128 a side) and, beside them, on meshes that go to cuFFT, against the FP64
oracle: every spline order, few particles (empty bins, fewer than a CTA),
particles on the box edges (supports that wrap), and crowded columns (a run of
the sorted list longer than one stage)."""
import numpy as np
import pytest

import oracle
import tcp_allpair_gb300 as T

pytestmark = pytest.mark.gpu

# FP32 transforms: the mesh is off by about 2^-24 sqrt(log2 K^3) = 3e-7 of its
# rms, and the spline derivatives multiply that by up to K/2 mesh lengths over
# the few that the potential varies on, so 64 x 3e-7 at most, twice that here.
FP32_FORCE = 4e-5


def recip(s, x, precision):
    with T.Context(T.params_for(s, precision=precision, recip="spme"), s.nel, s.nion) as c:
        c.EWALD_SELF()
        c.upload(x=x)
        um = c.Force_SPME4()
        return c.download(x=False, v=False, f=False, frec=True)[3], um


def check(s, x):
    fo, umo = oracle.Oracle.from_system(s, ei="kelbg").force_spme(x)
    f, um = recip(s, x, "fp64")
    assert um == pytest.approx(umo, rel=1e-11)
    assert oracle.rms_rel(f, fo) < 1e-10
    f, um = recip(s, x, "fp32c")
    assert um == pytest.approx(umo, rel=1e-5)
    assert oracle.rms_rel(f, fo) < FP32_FORCE


@pytest.mark.parametrize("K", [32, 48, 64, 96, 128, 40])
@pytest.mark.parametrize("order", [4, 5, 6, 7, 8])
def test_orders_and_meshes(K, order):
    s = T.make_system(777, seed=K + order, alpha_rc=3.1, K=K, order=order)
    x = s.x.copy()
    x[:6] = [[-0.5, -0.5, -0.5], [0.49999, 0.49999, 0.49999], [0.0, -0.5, 0.3], [0.5 - 1e-13, 0.1, 0.2], [0.2, 0.4999999, -0.5],
             [0.0, 0.0, 0.0]]
    x[:6] *= s.box
    check(s, x)


@pytest.mark.parametrize("K", [32, 40, 64])
@pytest.mark.parametrize("n", [2, 3, 65])
def test_few_particles(K, n):
    s = T.make_system(n, seed=n, alpha_rc=3.1, K=K, order=5)
    check(s, s.x)


@pytest.mark.parametrize("K,order", [(32, 4), (48, 6), (30, 5)])
def test_crowded_columns(K, order):
    """1,500 particles in four mesh columns: bins of hundreds, runs past one stage."""
    s = T.make_system(1500, seed=3, alpha_rc=3.1, K=K, order=order)
    x = s.x.copy()
    x[:, 1:] *= 2.0 / K
    check(s, x)
