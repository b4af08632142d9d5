"""The batched engine against the plain loop in the FP64 parity variant, in the field
map and with multiple scattering: with no products fused the two run the same
operations on every track, so the counts are equal and the deposits are sums of the
same terms (1e-9).  (The product's FP64 kernels fuse products as the compiler
chooses in each, so theirs differ by a few steps in millions there.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("steps", "substeps", "tracks", "sec_gamma", "sec_electron", "sec_positron", "n_pair", "n_annih", "errors")


@pytest.fixture(scope="module")
def dm():
    import geantexascalepilot_b200 as g
    m = g.ProxyDataManager()
    m.load_field_map()
    return m


@pytest.mark.parametrize("field_map,msc", [(1, 0), (0, 1), (0, 2), (1, 2)])
def test_engines_agree_track_by_track(dm, field_map, msc):
    import geantexascalepilot_b200 as g
    from geantexascalepilot_b200 import configs
    cfg, prims, nvol = configs.c3(6, 6)
    cfg.precision, cfg.fp64_parity, cfg.field_map, cfg.msc = 0, 1, field_map, msc
    out = []
    for cfg.engine in (0, 1):
        e, st, ps = g.transport(dm, cfg, *prims[:4], nvol=nvol, primary_steps=True)
        out.append((e.cpu().numpy(), st, ps.cpu().numpy()))
    (a, sa, pa), (b, sb, pb) = out
    assert {k: sa[k] for k in KEYS} == {k: sb[k] for k in KEYS} and sa["errors"] == 0 and sa["steps"] > 100000
    assert np.array_equal(pa, pb)
    np.testing.assert_allclose(b, a, rtol=1e-9, atol=1e-9 * a.max())
    assert abs(sa["escaped"] - sb["escaped"]) <= 1e-9 * max(1.0, sa["escaped"])
