"""A Hessian-vector product whose real-space part fails on the host (injected)
after its mesh work was queued on the second stream: the call reports it, and
the next calls, which sort particles into the same arrays on the main stream,
come after that work."""
import numpy as np
import pytest

import oracle
import tcp_allpair_gb300 as T
from tcp_allpair_gb300._abi import TCP_ERR_NOMEM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,K", [("fp64", 32), ("fp64", 40), ("fp32c", 32)])
def test_calls_after_a_failed_product(monkeypatch, precision, K):
    s = T.make_system(3000, lam=0.5, seed=9, alpha_rc=3.1, K=K, order=4)
    w = np.random.default_rng(9).normal(size=(s.n, 3))
    with T.Context(T.params_for(s, precision=precision), s.nel, s.nion) as c:
        c.EWALD_SELF()
        c.upload(x=s.x)
        um = c.Force_SPME4()
        frec = c.download(x=False, v=False, f=False, frec=True)[3]
        hw = c.hvp(w)[0]
        for _ in range(5):
            monkeypatch.setenv("TCP_INJECT_FAULT", "adj_pair")
            with pytest.raises(T.TcpError) as e:
                c.hvp(w)
            assert e.value.code == TCP_ERR_NOMEM
            monkeypatch.delenv("TCP_INJECT_FAULT")
            assert c.Force_SPME4() == um                 # sums in a fixed order
            assert np.array_equal(c.download(x=False, v=False, f=False, frec=True)[3], frec)
        # the pair sum's atomics: in FP32C it sums in FP32
        assert oracle.rms_rel(c.hvp(w)[0], hw) < (1e-12 if precision == "fp64" else 1e-5)
