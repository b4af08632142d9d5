"""The iteration graph that repeats on the device ends whatever its body: one
compaction interval or several, whole multiples of it, with and without work, and
with the same tracks as a graph of a given length."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dm():
    import geantexascalepilot_b200 as g
    return g.ProxyDataManager()


@pytest.mark.parametrize("n", [0, 1, 3])
@pytest.mark.parametrize("interval", [1, 3, 8, 9, 64])
def test_repeating_graph_ends_and_equals_a_graph_of_a_given_length(dm, interval, n):
    import geantexascalepilot_b200 as g
    from geantexascalepilot_b200 import configs
    cfg, prims, nvol = configs.c2(n)
    cfg.interaction_interval = interval
    out = []
    for cfg.graph_iters in (5, 0):
        e, st, ps = g.transport(dm, cfg, *prims[:4], nvol=nvol, primary_steps=True)
        out.append((e.cpu().numpy(), st, ps.cpu().numpy()))
    (a, sa, pa), (b, sb, pb) = out
    body = -(-8 // interval) * interval  # the body holds at least 8 iterations, in whole intervals
    assert sb["iterations"] % body == 0 and sb["iterations"] >= body
    assert sb["errors"] == 0 and sa["steps"] == sb["steps"] and sa["tracks"] == sb["tracks"]
    assert np.array_equal(pa, pb)
    np.testing.assert_allclose(b, a, rtol=1e-9, atol=1e-9 * max(a.max(), 1.0))
