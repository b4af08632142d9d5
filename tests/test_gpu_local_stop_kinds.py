"""Electrons booked where they stop, against the same kernels that do not book them
(a run whose iterations are counted): each geometry, field and option that the rule
distinguishes, FP64 and FP32-mixed, with enough photons that it applies, and on both
sides of its 1024 interactions of a process in a launch.  The counts are whole
numbers, the deposits sums of the same terms in another order (1e-9)."""
import numpy as np
import pytest

from test_csg import mixed_geometry

pytestmark = pytest.mark.gpu

KEYS = ("steps", "substeps", "tracks", "sec_gamma", "sec_electron", "sec_positron", "n_pair", "n_annih", "errors")


@pytest.fixture(scope="module")
def dm():
    import geantexascalepilot_b200 as g
    m = g.ProxyDataManager()
    m.load_field_map()
    return m


def _photons(n, centre, half, energies):
    rng = np.random.default_rng(17)
    d = rng.normal(size=(n, 3))
    return (np.zeros(n, np.int32), rng.uniform(*energies, n), rng.uniform(-half, half, (n, 3)) + centre,
            d / np.linalg.norm(d, axis=1)[:, None])


def _booked_and_not(dm, cfg, prims, nvol):
    import geantexascalepilot_b200 as g
    a, sa, _ = g.transport(dm, cfg, *prims, nvol=nvol)
    t = g.TrackSoA.from_primaries(cfg, *prims)
    out, b, sb = g.transport_tracks(dm, cfg, t, max_iterations=100000, nvol=nvol)
    assert out.n == 0 and sb["booked_steps"] == 0
    assert {k: sa[k] for k in KEYS} == {k: sb[k] for k in KEYS} and sa["errors"] == 0
    a, b = a.cpu().numpy(), b.cpu().numpy()
    np.testing.assert_allclose(a, b, rtol=1e-9, atol=1e-9 * b.max())
    assert abs(sa["escaped"] - sb["escaped"]) <= 1e-9 * max(1.0, sb["escaped"])
    return sa


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("field", ["none", "uniform", "map"])
@pytest.mark.parametrize("geometry", ["layers", "box", "tree of boxes", "tree of solids"])
def test_booked_electrons_leave_what_transported_ones_leave(dm, geometry, field, precision):
    import geantexascalepilot_b200 as g
    from geantexascalepilot_b200 import configs
    cfg, _, nvol = configs.c1(1) if geometry == "box" else configs.c2(1)
    cfg.charged_local, cfg.precision = 0, precision
    centre = np.array([0.0, 0.0, 50.0 if geometry == "box" else 0.0])
    if geometry.startswith("tree"):
        tree = g.geometry.calorimeter(axis=cfg.axis) if geometry == "tree of boxes" else mixed_geometry()
        nvol, cfg.geometry = dm.load_geometry(tree), 2
        if geometry == "tree of solids":
            centre = np.array([100.0, -50.0, 20.0])
    cfg.Bz, cfg.field_map = (4.0 if field == "uniform" else 0.0), int(field == "map")
    st = _booked_and_not(dm, cfg, _photons(40000, centre, 40.0, (0.05, 0.5)), nvol)
    assert st["booked_steps"] > 1000


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("option", [dict(charged_local=1), dict(msc=1), dict(msc=2)])
def test_nothing_is_booked_where_the_rule_does_not_hold(dm, option, precision):
    from geantexascalepilot_b200 import configs
    cfg, _, nvol = configs.c2(1)
    cfg.precision = precision
    for k, v in option.items():
        setattr(cfg, k, v)
    st = _booked_and_not(dm, cfg, _photons(40000, 0.0, 40.0, (0.05, 0.5)), nvol)
    assert st["booked_steps"] == 0


@pytest.mark.parametrize("precision", [0, 1])
def test_from_1024_interactions_of_a_launch_on(dm, precision):
    """Photons that interact in their first launch, nearly all by the photo-electric
    effect; those still alive after it scattered."""
    import geantexascalepilot_b200 as g
    from geantexascalepilot_b200 import configs
    cfg, _, nvol = configs.c1(1)
    cfg.charged_local, cfg.precision = 0, precision
    prims = _photons(2000, np.array([0.0, 0.0, 50.0]), 20.0, (0.03, 0.08))
    out, _, _ = g.transport_tracks(dm, cfg, g.TrackSoA.from_primaries(cfg, *prims), max_iterations=1, nvol=nvol)
    t = out.numpy()
    absorbed = np.ones(2000, bool)
    absorbed[t["primary"][t["type"] == 0]] = False
    n = int(np.flatnonzero(np.cumsum(absorbed) == 1024)[0]) + 1
    for count, booked in ((n - 1, False), (n, True)):
        st = _booked_and_not(dm, cfg, tuple(p[:count] for p in prims), nvol)
        assert (st["booked_steps"] > 0) == booked, count
