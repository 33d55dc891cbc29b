"""The FP64 derivative kernel (tiles and radial tables) against the
ordered-pair kernel, whose radial functions come from exp, rsqrt and erfcx:
chunk edges, arguments past both ends of the tables, a Deutsch system whose
tables do not fit (alpha rc > 4), a non-cubic box."""
import numpy as np
import pytest

import oracle
import tcp_allpair_gb300 as T

pytestmark = pytest.mark.gpu

# pair terms within 1e-15 of the exact ones; close Kelbg pairs (r >= 0.2
# lambda) lose a factor 25 to cancellation, as much again over the sums
REL = 1e-12


def both(s, p):
    w = np.random.default_rng(s.n).normal(size=(s.n, 3))
    out = []
    for flags in (T.FLAG_ENERGY, T.FLAG_ENERGY | T.FLAG_DETERMINISTIC):
        with T.Context(p, s.nel, s.nion) as c:
            c.set_flags(flags)
            c.EWALD_SELF()
            c.upload(x=s.x)
            hw, dfw = c.hvp(w)
            out.append((hw, dfw, c.adjoint_energy()[1]))
    return out, w


def check(s, p):
    ((hw, dfw, dl), (ho, dfo, dlo)), w = both(s, p)
    assert oracle.rms_rel(hw, ho) < REL
    # sums of terms of one sign (dl) and of both signs (dF/dlambda . w): against n times the largest term's scale
    assert dl == pytest.approx(dlo, rel=1e-11, abs=1e-14)
    scale = np.sqrt(s.n) * abs(dlo) / (0.1 * T.EPS)
    assert abs(dfw - dfo) < 1e-11 * max(scale, 1e-3)


@pytest.mark.parametrize("ei", ["coulomb", "kelbg", "deutsch"])
@pytest.mark.parametrize("nel,nion", [(1, 1), (1, 32), (31, 33), (65, 64), (0, 97), (640, 603)])
def test_chunk_edges(ei, nel, nion):
    n = nel + nion
    s = T.make_system(n, lam=0.5, seed=n, alpha_rc=3.1, nel=nel)
    check(s, T.params_for(s, precision="fp64", ei=ei, recip="none"))


@pytest.mark.parametrize("ei", ["kelbg", "deutsch"])
@pytest.mark.parametrize("alpha_rc,lam", [(0.3, 0.5), (5.0, 0.3), (8.6, 3.0)])
def test_past_the_table_ends(ei, alpha_rc, lam):
    s = T.make_system(500, lam=lam, seed=5, alpha_rc=alpha_rc)
    check(s, T.params_for(s, precision="fp64", ei=ei, recip="none"))


def test_noncubic_box():
    s = T.make_system(600, lam=0.5, seed=6, alpha_rc=3.1)
    p = T.params_for(s, precision="fp64", ei="kelbg", recip="none")
    box = np.array([s.box, 1.1 * s.box, 0.9 * s.box])
    for d in range(3):
        p.box[d] = box[d]
    p.rc = 0.45 * s.box
    s.x = (np.random.default_rng(6).random((s.n, 3)) - 0.5) * box
    check(s, p)
