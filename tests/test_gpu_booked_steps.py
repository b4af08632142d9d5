"""The steps that the transport kernels make and those that the interaction kernels
book for electrons that stop where they are created are told apart: with one step
per launch a transport kernel makes one step for each record that it reads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,local", [(20000, True), (500, False)])  # 1024 interactions of a launch are the limit
def test_a_transport_kernel_makes_the_steps_that_are_not_booked(n, local, precision):
    import geantexascalepilot_b200 as g
    from geantexascalepilot_b200 import configs
    cfg, prims, nvol = configs.c1(n)
    rng = np.random.default_rng(11)
    pos = rng.uniform(-40.0, 40.0, (n, 3)) + np.array([0.0, 0.0, 50.0])
    cfg.charged_local, cfg.precision = 0, precision
    dm, E = g.ProxyDataManager(), rng.uniform(0.02, 0.5, n)
    for cfg.steps_per_launch in (1, 0):
        _, st, _ = g.transport(dm, cfg, prims[0], E, pos, prims[3], nvol=nvol)
        assert st["errors"] == 0 and (st["booked_steps"] > 0) == local
        made = np.array(st["transport_steps"]) - [0, st["booked_steps"], 0]
        assert sum(made) + st["booked_steps"] == st["steps"]
        if cfg.steps_per_launch == 1:
            assert list(made) == st["transport_read"]
        else:
            assert all(made >= st["transport_read"])
