"""RDF counts of the packed Newton-3 kernels against the ordered-pair kernel,
which bins every pair near an edge by the same exact integers: a cut-off inside
a bin, bins past the last one inside the cut-off, separations exactly on bin
edges and on the cut-off, one bin for everything, tiny systems.  Counts are
integers: they agree exactly."""
import numpy as np
import pytest

import tcp_allpair_gb300 as T

pytestmark = pytest.mark.gpu


def counts(s, p, extra=0):
    with T.Context(p, s.nel, s.nion) as c:
        c.set_flags(T.FLAG_RDF | extra)
        c.EWALD_SELF()
        c.upload(x=s.x)
        c.Force_direct_self()
        return c.histograms()[0]


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
@pytest.mark.parametrize("nel,nion,rc,bins,where", [
    (1, 1, 0.5, (500, 500, 500), "random"),
    (33, 0, 0.5, (500, 499.5, 480), "random"),
    (700, 645, 0.371, (371.3, 123.75, 77.01), "random"),       # rc inside a bin
    (700, 645, 0.5, (1400, 700, 501.5), "random"),             # rc past the last bin
    (700, 645, 0.5, (0.5, 1, 2), "random"),                    # bins wider than the box
    (256, 256, 0.5, (4, 40, 400), "lattice"),                  # on bin edges and on rc
    (256, 256, 0.47, (4.7, 47, 470), "lattice"),
    (700, 645, 0.5, (0, 500, 0), "random"),                    # no bin width
])
def test_counts_of_both_kernels(monkeypatch, variant, nel, nion, rc, bins, where):
    monkeypatch.setenv("TCP_PAIR_VARIANT", "10")
    monkeypatch.setenv("TCP_RDF_VARIANT", str(variant))
    s = T.make_system(nel + nion, lam=0.5, seed=7, alpha_rc=3.1, nel=nel)
    if where == "lattice":
        g = (np.arange(8) - 4) / 8.0 * s.box
        x = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
        s.x = np.ascontiguousarray(x[np.random.default_rng(1).permutation(len(x))])
    p = T.params_for(s, precision="fp32c", ei="coulomb", recip="none")
    p.rc = rc * s.box
    p.dx_ee, p.dx_ei, p.dx_ii = (p.rc / b if b else 0.0 for b in bins)
    assert np.array_equal(counts(s, p), counts(s, p, T.FLAG_DETERMINISTIC))
