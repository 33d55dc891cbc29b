"""Contexts (and batches) that live side by side and need different amounts of
shared memory in the same kernels: the calls of the one that needs more have to
go on working, with the same results, after the other one is prepared.  The
limit of a kernel's dynamic shared memory belongs to the kernel, not to a
context."""
import numpy as np
import pytest

import oracle
import tcp_allpair_gb300 as T

pytestmark = pytest.mark.gpu

# The same kernels on the same inputs: only the order of the FP64 atomics (and,
# in FP32C, which CTA sums which pairs in two-float FP32) differs.
SAME = {"fp64": 1e-12, "fp32c": 1e-6}


def system(**kw):
    return T.make_system(300, lam=0.5, seed=4, **{"alpha_rc": 3.1, **kw})


def calls(c, w):
    c.force()
    f, frec = c.download(x=False, v=False, frec=True)[2:]
    return f, frec, c.hvp(w)[0]


@pytest.mark.parametrize("precision,recip,more,less", [
    # radial tables of the FP64 pair sum and of its derivatives, by alpha rc
    ("fp64", "none", dict(alpha_rc=3.1), dict(alpha_rc=2.8)),
    # one plane of the mesh and a stage of the spread, by the spline order
    ("fp64", "spme", dict(K=32, order=6), dict(K=32, order=4)),
    ("fp32c", "spme", dict(K=64, order=6), dict(K=64, order=4)),
    # rows of the spread on a mesh that cuFFT transforms, by the mesh length
    ("fp64", "spme", dict(K=80, order=5), dict(K=40, order=5)),
    ("fp32c", "spme", dict(K=80, order=5), dict(K=40, order=5)),
    # phase factors of the plain Ewald sum, by the largest index
    ("fp64", "ewald", dict(nmax2=64), dict(nmax2=9)),
    ("fp32c", "ewald", dict(nmax2=64), dict(nmax2=9)),
])
def test_larger_context_outlives_preparing_a_smaller(precision, recip, more, less):
    w = np.random.default_rng(4).normal(size=(300, 3))
    ctxs = []
    try:
        for kw in (more, less):
            kw = dict(kw)
            nmax2 = kw.pop("nmax2", 64)
            s = system(**kw)
            c = T.Context(T.params_for(s, precision=precision, recip=recip, nmax2=nmax2), s.nel, s.nion)
            ctxs.append(c)
            c.EWALD_SELF()
            c.upload(x=s.x)
            got = calls(c, w)
            if len(ctxs) == 1:
                want = got
        for f, fo in zip(calls(ctxs[0], w), want):
            if np.any(fo):                           # no reciprocal part: zeros on both sides
                assert oracle.rms_rel(f, fo) < SAME[precision]
    finally:
        for c in ctxs:
            c.close()


@pytest.mark.parametrize("more,less", [
    (dict(K=64, order=6), dict(K=64, order=4)),
    (dict(K=80, order=5), dict(K=40, order=5)),
])
def test_larger_batch_outlives_preparing_a_smaller(more, less):
    batches = []
    try:
        for kw in (more, less):
            s = system(**kw)
            b = T.Batch([T.params_for(s)], [s.nel], [s.nion])
            batches.append(b)
            b.EWALD_SELF()
            b.upload(0, x=s.x)
            b.force()
            if len(batches) == 1:
                want = b.download(0)[2]
        batches[0].force()
        assert oracle.rms_rel(batches[0].download(0)[2], want) < SAME["fp32c"]
    finally:
        for b in batches:
            b.close()
