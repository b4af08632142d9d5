"""Substream skip-ahead around the edges of its blocks (256 streams each) and
far into the stream (the oracle's own jump reads 62 bits of the index, so the
reference here is the recurrence in Python's integers), and the calls that
report a rejection cap at once, from several threads: whole numbers equal,
outputs to the last bit those of a call made alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dm():
    import geantexascalepilot_b200 as g
    return g.ProxyDataManager()


M = (4294967087, 4294944443)
A = ([[0, 1, 0], [0, 0, 1], [-810728, 1403580, 0]], [[0, 1, 0], [0, 0, 1], [-1370589, 0, 527612]])


def _power(a, e, m):
    r = [[int(i == j) for j in range(3)] for i in range(3)]
    while e:
        if e & 1:
            r = _product(r, a, m)
        a, e = _product(a, a, m), e >> 1
    return r


def _product(a, b, m):
    return [[sum(a[i][k] * b[k][j] for k in range(3)) % m for j in range(3)] for i in range(3)]


def _substreams(seed, first, n):
    out = np.empty((n, 6))
    for c in range(2):
        one, j = _power(A[c], 1 << 76, M[c]), _power(A[c], first << 76, M[c])
        v = [sum(j[i][k] * int(seed[3 * c + k]) for k in range(3)) % M[c] for i in range(3)]
        for t in range(n):
            out[t, 3 * c:3 * c + 3] = v
            v = [sum(one[i][k] * v[k] for k in range(3)) % M[c] for i in range(3)]
    return out


@pytest.mark.parametrize("first", [0, 1, 255, 256, 2 ** 40 + 3, 2 ** 62 + 12345])
@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 1025])
def test_substreams_equal_the_recurrence(n, first):
    from geantexascalepilot_b200 import MRG32k3a
    for seed in ([12345.0] * 6, [4294967086.0, 0.0, 1.0, 4294944442.0, 7.0, 0.0]):
        got = MRG32k3a.to_states(MRG32k3a.substreams(seed, first, n)).numpy()
        assert np.array_equal(got, _substreams(seed, first, n))


def test_interactions_from_threads_equal_those_alone(dm):
    import torch
    from geantexascalepilot_b200 import MRG32k3a, ProxySeltzerBerger
    n, seed = 3001, [2024.0] * 6
    E = torch.logspace(-1, 4, n, dtype=torch.float64, device="cuda")
    d = torch.tensor([[0.0, 0.6, 0.8]], dtype=torch.float64, device="cuda").repeat(n, 1)
    model = ProxySeltzerBerger(dm, mode=1, Z=82, cut=0.0949, density_factor=1.4e-8, sb_table=2)

    def sample(first):
        st = MRG32k3a.substreams(seed, first, n)
        o = model.SampleSecondaries(E, d, st)
        return [st.cpu()] + [o[k].cpu() for k in sorted(o)]

    alone = [sample(k * n) for k in range(8)]
    got = [None] * 8

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(5):
                got[k] = sample(k * n)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, got):
        assert all(torch.equal(x, y) for x, y in zip(a, b))
