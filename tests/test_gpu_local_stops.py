"""Electrons that come to rest where they are created are booked by the batched
engine's interaction kernels (from 1024 interactions of a launch on) and never
become tracks: the same steps, sub-steps, tracks and deposits as the plain loop,
which transports every one of them, in each geometry, field and option that the
rule distinguishes.  FP64: the counts are whole numbers, the deposits sums of the
same terms in another order (1e-9)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("steps", "substeps", "tracks", "sec_gamma", "sec_electron", "sec_positron", "n_pair", "n_annih", "errors")


@pytest.fixture(scope="module")
def dm():
    import geantexascalepilot_b200 as g
    return g.ProxyDataManager()


@pytest.mark.parametrize("Bz", [0.0, 4.0])
@pytest.mark.parametrize("geometry,charged_local", [("layers", 0), ("box", 0), ("box", 1), ("tree", 0)])
@pytest.mark.parametrize("n,energy", [(3, 50.0), (4000, 2.0)])
def test_batched_engine_equals_the_plain_loop(dm, n, energy, geometry, charged_local, Bz):
    import geantexascalepilot_b200 as g
    from geantexascalepilot_b200 import configs
    cfg, _, nvol = configs.c1(1)
    if geometry != "box":
        cfg, _, nvol = configs.c2(1)
    if geometry == "tree":
        nvol = dm.load_geometry(g.geometry.calorimeter(axis=cfg.axis))
        cfg.geometry = 2
    cfg.charged_local, cfg.Bz = charged_local, Bz
    rng = np.random.default_rng(5)
    pos = rng.uniform(-40.0, 40.0, (n, 3)) + (np.array([0.0, 0.0, 50.0]) if geometry == "box" else 0.0)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    prims = (np.zeros(n, np.int32), rng.uniform(0.02, 1.0, n) * energy, pos, d)
    out = []
    for engine in (0, 1):
        cfg.engine = engine
        e, st, ps = g.transport(dm, cfg, *prims, nvol=nvol, primary_steps=True)
        out.append((e.cpu().numpy(), st, ps.cpu().numpy()))
    (a, sa, pa), (b, sb, pb) = out
    assert {k: sa[k] for k in KEYS} == {k: sb[k] for k in KEYS} and sa["errors"] == 0
    assert sum(sb["transport_steps"]) == sb["steps"]
    assert np.array_equal(pa, pb)
    np.testing.assert_allclose(b, a, rtol=1e-9, atol=1e-9 * a.max())
    assert abs(sa["escaped"] - sb["escaped"]) <= 1e-9 * max(1.0, sa["escaped"])
