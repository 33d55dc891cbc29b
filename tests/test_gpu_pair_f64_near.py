"""The near-pair masks and the ring of chunks of the FP64 Newton-3 kernels
(forces, and their derivatives) against the ordered-pair FP64 kernels: every split and group of the items, rings
of odd and even length, species that end inside a chunk, cut-offs that leave few
pairs or all of them, boxes that are not cubic."""
import numpy as np
import pytest

import oracle
import tcp_allpair_gb300 as T

pytestmark = pytest.mark.gpu

# A pair term is within 1e-14 of the exact one (close Kelbg pairs; 4e-16
# otherwise), and the terms of a particle add up to at most 100 times its force.
REL = 1e-12


@pytest.mark.parametrize("nel,nion,rc,shape,ei", [
    (97, 95, 0.5, (1, 1, 1), "kelbg"),           # eighths of a tile; 7 chunks
    (250, 260, 0.5, (1, 1, 1), "deutsch"),       # 17 chunks
    (700, 836, 0.5, (1, 1, 1), "kelbg"),         # quarters
    (33, 1500, 0.37, (1, 1.1, 0.9), "kelbg"),
    (1501, 1500, 0.5, (1, 1, 1), "kelbg"),       # halves; 94 chunks
    (2500, 2501, 0.5, (1, 1, 1), "kelbg"),       # whole tiles
    (2500, 2470, 0.03, (1, 1, 1), "kelbg"),      # a few pairs per particle
    (1500, 1470, 0.5, (0.25, 0.25, 0.25), "coulomb"),   # a droplet: every pair
    (4500, 4501, 0.5, (1, 1, 1), "kelbg"),       # two tiles
    (6001, 8010, 0.5, (1, 1, 1), "kelbg"),       # four tiles
    (0, 14016, 0.31, (1, 1, 1), "kelbg"),
])
def test_masks_and_ring(nel, nion, rc, shape, ei):
    n = nel + nion
    s = T.make_system(n, lam=0.5, seed=n, alpha_rc=3.1, nel=nel)
    p = T.params_for(s, precision="fp64", ei=ei, recip="none")
    x = np.array(s.x)
    droplet = max(shape) < 1
    for d in range(3):
        p.box[d] = s.box * (1 if droplet else shape[d])
        x[:, d] *= shape[d]
    p.rc = rc * s.box
    out = []
    for extra in (0, T.FLAG_DETERMINISTIC):
        with T.Context(p, nel, nion) as c:
            c.set_flags(T.FLAG_ENERGY | T.FLAG_RDF | extra)
            c.EWALD_SELF()
            c.upload(x=x)
            ur = c.Force_direct_self()
            out.append((c.download(x=False, v=False)[2], ur, c.histograms()[0]))
    (f, ur, h), (fo, uo, ho) = out
    assert oracle.rms_rel(f, fo) < REL
    assert abs(ur - uo) < REL * n * n * 10.0 / min(shape) / T.EPS   # n(n-1)/2 terms of both signs, none above 1/(0.1 a)
    assert np.array_equal(h, ho)


@pytest.mark.parametrize("nel,nion,rc,ei", [
    (150, 170, 0.5, "deutsch"),      # eighths of a tile
    (700, 836, 0.21, "kelbg"),       # quarters
    (1501, 1500, 0.5, "kelbg"),      # halves
    (2500, 2501, 0.5, "coulomb"),    # whole tiles
    (4500, 4501, 0.4, "kelbg"),      # two
    (6001, 8010, 0.5, "kelbg"),      # four
])
def test_derivatives(nel, nion, rc, ei):
    n = nel + nion
    s = T.make_system(n, lam=0.5, seed=n, alpha_rc=3.1, nel=nel)
    p = T.params_for(s, precision="fp64", ei=ei, recip="none")
    p.rc = rc * s.box
    w = np.random.default_rng(n).normal(size=(n, 3))
    out = []
    for flags in (T.FLAG_ENERGY, T.FLAG_ENERGY | T.FLAG_DETERMINISTIC):
        with T.Context(p, nel, nion) as c:
            c.set_flags(flags)
            c.EWALD_SELF()
            c.upload(x=s.x)
            hw, dfw = c.hvp(w)
            out.append((hw, dfw, c.adjoint_energy()[1]))
    (hw, dfw, dl), (ho, dfo, dlo) = out
    assert oracle.rms_rel(hw, ho) < REL
    # one sign; both signs, against sqrt(n) times the scale of its largest terms
    assert dl == pytest.approx(dlo, rel=1e-11, abs=1e-14)
    assert abs(dfw - dfo) < 1e-11 * max(np.sqrt(n) * abs(dlo) / (0.1 * T.EPS), 1e-3)
