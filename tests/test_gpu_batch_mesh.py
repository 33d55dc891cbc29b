"""Batch meshes with more than 1,024 points along one axis (single contexts
refuse them, batches take them): forces against the FP64 oracle on the same
mesh, beside a replica of an ordinary one, after a force call and after a step
of zero length (whose half kick bins the particles itself)."""
import numpy as np
import pytest

import oracle
import tcp_allpair_gb300 as T

pytestmark = pytest.mark.gpu

# FP32 transforms: the mesh is off by about 2^-24 sqrt(log2 K^3) = 3e-7 of its
# rms; the spline derivatives multiply that by up to K/2 mesh lengths, 540 here,
# over the few that the potential varies on.  The same again for other roundings.
RECIP = 2 * 540 * 3e-7
REAL = 2e-6          # the real-space sum's, as in the other batch tests


@pytest.mark.parametrize("order", [4, 7])
@pytest.mark.parametrize("axis,K", [(0, 1030), (1, 1030), (2, 1080)])
def test_long_axis(axis, K, order):
    n = 400
    ss = [T.make_system(n, lam=0.5, seed=k, alpha_rc=3.1, K=16, order=order) for k in range(2)]
    params = [T.params_for(s) for s in ss]
    params[1].K[axis] = K
    ss[1].K = tuple(params[1].K)
    # every mesh column of the long axis is reached, its ends among them
    ss[1].x[:, axis] = ((np.arange(n) + 0.5) / n - 0.5) * ss[1].box
    ss[1].x[:2, axis] = -0.5 * ss[1].box, 0.4999999 * ss[1].box
    with T.Batch(params, [s.nel for s in ss], [s.nion for s in ss]) as b:
        b.EWALD_SELF()
        for r, s in enumerate(ss):
            b.upload(r, x=s.x, v=np.zeros((n, 3)))
        b.force()
        f = [b.download(r, x=False, v=False)[2] for r in range(2)]
        b.md_steps(0.0, 1)
        g = [b.download(r, x=False, v=False)[2] for r in range(2)]
    for r, s in enumerate(ss):
        o = oracle.Oracle.from_system(s, ei="kelbg")
        fo = o.force_total(s.x)[0]
        bound = RECIP * np.sqrt(np.mean(o.force_spme(s.x)[0] ** 2)) + REAL * np.sqrt(np.mean(fo ** 2))
        for got in (f[r], g[r]):
            assert np.sqrt(np.mean((got - fo) ** 2)) < bound
