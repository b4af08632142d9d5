"""What gx_transport_tracks hands over after a number of iterations does not
depend on how many tracks there are: with one step per launch every track in
flight takes exactly one step in each iteration, and by default the turns are
those of steps_per_launch = 16."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dm():
    import geantexascalepilot_b200 as g
    return g.ProxyDataManager()


def _photons(n):
    """Low-energy photons in lead: most interact at once, most electrons stop where they start."""
    from geantexascalepilot_b200 import configs
    cfg, prims, nvol = configs.c1(n)
    rng = np.random.default_rng(11)
    pos = rng.uniform(-40.0, 40.0, (n, 3)) + np.array([0.0, 0.0, 50.0])
    cfg.charged_local = 0
    return cfg, (prims[0], rng.uniform(0.02, 0.5, n), pos, prims[3]), nvol


def _hand_over(dm, cfg, prims, nvol, iterations):
    import geantexascalepilot_b200 as g
    t = g.TrackSoA.from_primaries(cfg, *prims)
    out, _, st = g.transport_tracks(dm, cfg, t, max_iterations=iterations, nvol=nvol)
    assert st["errors"] == 0
    return out, st


def _sorted_state(out):
    a = out.numpy()
    rows = np.concatenate([a["rng"].astype(np.float64),
                           np.stack([a[f] for f in ("ekin", "x", "y", "z", "dx", "dy", "dz", "nil0", "nil1")], 1),
                           np.stack([a["type"], a["volume"]], 1).astype(np.float64)], 1)
    return rows[np.lexsort(rows.T[::-1])]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [500, 20000])  # both sides of 1024 interactions of a process in a launch
def test_one_step_per_launch_is_one_step_per_iteration(dm, n, precision):
    cfg, prims, nvol = _photons(n)
    cfg.precision, cfg.steps_per_launch = precision, 1
    steps = n
    for it in (1, 2, 3):
        out, st = _hand_over(dm, cfg, prims, nvol, it)
        assert st["steps"] == steps, it
        steps += out.n  # each of these takes one step in the next iteration


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [500, 20000])
def test_default_turns_are_sixteen_steps(dm, n, precision):
    cfg, prims, nvol = _photons(n)
    cfg.precision = precision
    cfg.geometry, cfg.axis, cfg.Bz = 1, 2, 4.0
    nvol = 100
    prims = (prims[0], prims[1] * 40.0) + prims[2:]
    for it in (1, 2):
        cfg.steps_per_launch = 0
        a, sa = _hand_over(dm, cfg, prims, nvol, it)
        cfg.steps_per_launch = 16
        b, sb = _hand_over(dm, cfg, prims, nvol, it)
        assert (sa["steps"], sa["substeps"], sa["tracks"], a.n) == (sb["steps"], sb["substeps"], sb["tracks"], b.n)
        assert a.n > 0 and np.array_equal(_sorted_state(a), _sorted_state(b))
