"""Tracks deferred to the overflow stacks are all transported.  With stores far
smaller than a shower and few tracks taken back at a time, the stores drain
completely while the last deferred tracks are on their way back, and the run has
to go on for them: the same steps, tracks and energies as with room for all, in
every loop that decides when a run is over (the plain loop, the repeating graph,
a graph of a given length, the profiling loop, the allocation-free one)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

KEYS = ("steps", "substeps", "tracks", "sec_gamma", "sec_electron", "sec_positron", "n_pair", "n_annih", "errors")


@pytest.fixture(scope="module")
def dm():
    import geantexascalepilot_b200 as g
    return g.ProxyDataManager()


def _run(dm, cfg, prims, nvol, **kw):
    import geantexascalepilot_b200 as g
    for k, v in kw.items():
        setattr(cfg, k, v)
    e, st, _ = g.transport(dm, cfg, *prims[:4], nvol=nvol)
    return e.cpu().numpy(), st


def _same(a, sa, b, sb):
    assert {k: sa[k] for k in KEYS} == {k: sb[k] for k in KEYS} and sa["errors"] == 0
    assert sb["peak_in_flight"] < sa["peak_in_flight"]  # the stores were too small
    np.testing.assert_allclose(b, a, rtol=1e-9, atol=1e-9 * a.max())
    assert abs(sa["escaped"] - sb["escaped"]) <= 1e-9 * max(1.0, sa["escaped"])


@pytest.mark.parametrize("refill_below", [1, 8])
@pytest.mark.parametrize("loop", [dict(engine=0), dict(engine=1), dict(engine=1, graph_iters=1),
                                  dict(engine=1, profile=1)], ids=["plain", "graph", "graph_of_1", "profile"])
def test_every_deferred_track_is_transported(dm, loop, refill_below):
    from geantexascalepilot_b200 import configs
    cfg, prims, nvol = configs.c2(2)
    a, sa = _run(dm, cfg, prims, nvol, precision=0, **loop)
    b, sb = _run(dm, cfg, prims, nvol, capacity=16, refill_below=refill_below)
    _same(a, sa, b, sb)


def test_every_deferred_track_is_transported_without_allocation(dm):
    """One shower that fills the static store (16384 tracks) and part of the stack."""
    import geantexascalepilot_b200 as g
    from geantexascalepilot_b200 import configs
    cfg, prims, nvol = configs.c2(1)
    prims = (prims[0], np.full(1, 5.0e5), prims[2], prims[3])
    a, sa = _run(dm, cfg, prims, nvol, precision=0, engine=0)
    cfg.refill_below = 1
    t, E, p, d = (torch.as_tensor(x, device="cuda") for x in prims)
    edep = torch.zeros((1, nvol), dtype=torch.float64, device="cuda")
    b, sb = g.transport_noalloc(dm, cfg, t, E, p, d, nvol=nvol, edep=edep)
    _same(a, sa, b.cpu().numpy(), sb)
