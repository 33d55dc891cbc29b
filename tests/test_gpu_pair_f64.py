"""The FP64 Newton-3 pair kernel (radial tables, warp tiles of 32 x 32) against
the ordered-pair FP64 kernel, which evaluates the same functions with exp,
rsqrt and erfcx: chunk edges, tiny systems, arguments past both ends of the
tables and lattice positions (separations with zero components)."""
import numpy as np
import pytest

import oracle
import tcp_allpair_gb300 as T

pytestmark = pytest.mark.gpu

# Each kernel's pair terms are within 4e-16 of the exact ones; close Kelbg
# pairs (r >= 0.2 lambda here) lose a factor 25 to cancellation, and a particle
# sums at most 2,000 of them: 1e-12 is ten times the sum of both.
REL = 1e-12


def both(s, p, flags=T.FLAG_ENERGY):
    out = []
    for extra in (0, T.FLAG_DETERMINISTIC):
        with T.Context(p, s.nel, s.nion) as c:
            c.set_flags(flags | extra)
            c.EWALD_SELF()
            c.upload(x=s.x)
            ur = c.Force_direct_self()
            out.append((c.download(x=False, v=False)[2], ur, c.histograms()[0]))
    return out


def check(s, p, flags=T.FLAG_ENERGY | T.FLAG_RDF):
    (f, ur, h), (fo, uo, ho) = both(s, p, flags)
    assert oracle.rms_rel(f, fo) < REL
    # Ur is a sum of n(n-1)/2 terms of both signs, none above 1/(0.1 a)
    assert abs(ur - uo) < REL * s.n * s.n * 10.0 / T.EPS
    assert np.array_equal(h, ho)


@pytest.mark.parametrize("ei", ["coulomb", "kelbg", "deutsch"])
@pytest.mark.parametrize("nel,nion", [(1, 1), (2, 0), (1, 32), (31, 33), (32, 32), (65, 64), (0, 97), (640, 603), (1000, 1001)])
def test_chunk_edges(ei, nel, nion):
    n = nel + nion
    s = T.make_system(n, lam=0.5, seed=n, alpha_rc=3.1, nel=nel)
    check(s, T.params_for(s, precision="fp64", ei=ei, recip="none"))


@pytest.mark.parametrize("ei", ["coulomb", "kelbg", "deutsch"])
@pytest.mark.parametrize("alpha_rc,lam", [(0.3, 0.5), (5.7, 0.1), (8.6, 3.0)])
def test_past_the_table_ends(ei, alpha_rc, lam):
    """alpha rc = 0.3: most pairs lie below the Ewald table (alpha r < 1/8); 8.6: pairs past its end."""
    s = T.make_system(700, lam=lam, seed=5, alpha_rc=alpha_rc)
    check(s, T.params_for(s, precision="fp64", ei=ei, recip="none"))


@pytest.mark.parametrize("ei", ["kelbg", "deutsch"])
def test_noncubic_box(ei):
    s = T.make_system(1100, lam=0.5, seed=6, alpha_rc=3.1)
    p = T.params_for(s, precision="fp64", ei=ei, recip="none")
    box = np.array([s.box, 1.1 * s.box, 0.9 * s.box])
    for d in range(3):
        p.box[d] = box[d]
    p.rc = 0.45 * s.box
    s.x = (np.random.default_rng(6).random((s.n, 3)) - 0.5) * box
    check(s, p)


def test_lattice_positions():
    """An 8^3 lattice: separations with zero components and with components of exactly half the box.  The
    cut-off lies between two lattice distances: a pair exactly on it may fall on either side by the rounding of
    the coordinates."""
    s = T.make_system(512, lam=0.5, seed=8, alpha_rc=3.1)
    g = (np.arange(8) - 4) * (s.box / 8)
    s.x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    p = T.params_for(s, precision="fp64", ei="coulomb", recip="none")
    p.rc = 0.47 * s.box
    (f, ur, _), (fo, uo, _) = both(s, p)
    # forces cancel by symmetry; a particle's largest pair force is eps/(L/8)^2
    assert np.max(np.abs(f - fo)) < 1e-12 * T.EPS / (s.box / 8) ** 2
    assert ur == pytest.approx(uo, rel=1e-11)
