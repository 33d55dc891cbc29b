"""Replica transfers: host arrays the device addresses in place, arrays at odd
addresses (copied on the host), the staged form (TCP_HOST_DIRECT=0), fields left
out, replicas of odd sizes beside each other."""
import numpy as np
import pytest

import tcp_allpair_gb300 as T

pytestmark = pytest.mark.gpu


def at(shape, offset):
    """A float64 array whose data start `offset` bytes past an 8-byte boundary."""
    raw = np.zeros(8 * int(np.prod(shape)) + 16, dtype=np.uint8)
    o = -raw.ctypes.data % 8 + offset
    return raw[o:o + 8 * int(np.prod(shape))].view(np.float64).reshape(shape)


@pytest.mark.parametrize("direct", ["1", "0"])
@pytest.mark.parametrize("offset", [0, 4])
def test_round_trip(monkeypatch, direct, offset):
    monkeypatch.setenv("TCP_HOST_DIRECT", direct)
    ss = [T.make_system(n, lam=0.5, seed=n, alpha_rc=3.1, K=16) for n in (33, 86, 513)]
    with T.Batch([T.params_for(s) for s in ss], [s.nel for s in ss], [s.nion for s in ss]) as b:
        b.EWALD_SELF()
        given = []
        for r, s in enumerate(ss):
            a = [at((s.n, 3), offset) for _ in range(3)]
            for k in range(3):
                a[k][:] = np.random.default_rng(10 * r + k).uniform(-0.5, 0.5, (s.n, 3)) * s.box
            given.append(a)
            b._chk(b.lib.tcp_batch_upload(b.h, r, *[q.ctypes.data for q in a]), "tcp_batch_upload")
        v = at((ss[1].n, 3), offset)
        v[:] = 7.0
        b._chk(b.lib.tcp_batch_upload(b.h, 1, None, v.ctypes.data, None), "tcp_batch_upload")
        given[1][1] = v
        for r, s in enumerate(ss):
            out = [at((s.n, 3), offset) for _ in range(3)]
            b._chk(b.lib.tcp_batch_download(b.h, r, *[q.ctypes.data for q in out]), "tcp_batch_download")
            for k in range(3):
                assert np.array_equal(out[k], given[r][k])
        f = at((ss[2].n, 3), offset)
        b._chk(b.lib.tcp_batch_download(b.h, 2, None, None, f.ctypes.data), "tcp_batch_download")
        assert np.array_equal(f, given[2][2])
