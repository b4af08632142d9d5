"""gx_post_step works on a batch of 16384 tracks or more in an order of its own (by
particle type and process within a block of 256): a batch gives each track what it
gets alone, at the edges of the blocks and of that rule, and slots without an
interaction are cleared."""
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("type", "status", "volume", "next_volume", "process", "boundary", "x", "y", "z", "dx", "dy", "dz", "ekin",
          "nil0", "nil1", "nil2", "pstep", "step", "snext", "safety")


@pytest.fixture(scope="module")
def dm():
    import geantexascalepilot_b200 as g
    return g.ProxyDataManager()


def _batch(g, cfg, index):
    """Tracks `index` of a fixed sequence: types, energies and places that mix the
    processes, on the streams of their places in the sequence."""
    import numpy as np
    k = np.asarray(index)
    rng = np.random.default_rng(11)
    d = rng.normal(size=(20000, 3))
    pos = rng.uniform(-190.0, 190.0, (20000, 3))
    E = 10.0 ** rng.uniform(-1.0, 4.0, 20000)
    d /= np.linalg.norm(d, axis=1)[:, None]
    t = g.TrackSoA.from_primaries(cfg, k % 3, E[k], pos[k], d[k])
    st = g.MRG32k3a.substreams(list(cfg.seed), 0, 20000)
    t.rng.view(6, t.capacity)[:, :len(k)] = st[:, k]
    return t


def _step(g, dm, cfg, t):
    import torch
    sec = g.TrackSoA(2 * t.n)
    edep = torch.zeros((1, 100), dtype=torch.float64, device="cuda")
    for _ in range(2):
        g.gpil(dm, cfg, t)
        g.propagate(dm, cfg, t)
        g.along_step(dm, cfg, t, edep)
        g.post_step(dm, cfg, t, sec, edep)
    n = t.n
    return ([getattr(t, f)[:n].cpu() for f in FIELDS] + [t.rng.view(6, t.capacity)[:, :n].cpu()],
            [getattr(sec, f).cpu() for f in FIELDS] + [sec.rng.view(6, sec.capacity).cpu()])


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 1025, 16383, 16384, 16641])
def test_a_batch_gives_each_track_what_it_gets_alone(dm, n):
    import numpy as np
    import torch
    import geantexascalepilot_b200 as g
    from geantexascalepilot_b200 import configs
    cfg, _, _ = configs.c2(1)
    cfg.Bz = 4.0
    whole, wsec = _step(g, dm, cfg, _batch(g, cfg, np.arange(n)))
    for i in sorted({0, n // 2, n - 1, min(n - 1, 255), min(n - 1, 256)}):
        alone, asec = _step(g, dm, cfg, _batch(g, cfg, [i]))
        for a, w in zip(alone, whole):
            assert torch.equal(a[..., 0], w[..., i])
        alive = [k for k in range(2) if asec[1][k] == 0]  # TRACK_ALIVE
        assert all(wsec[1][2 * i + k] == asec[1][k] for k in range(2))
        for a, w in zip(asec, wsec):
            assert all(torch.equal(a[..., k], w[..., 2 * i + k]) for k in alive)
