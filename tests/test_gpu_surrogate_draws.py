"""The learned form's walk takes the random walk's normals from the same function as the FP32 step."""
import numpy as np
import pytest

from wacommplusplus_b200 import synthetic as syn
from wacommplusplus_b200.engine import Engine
from wacommplusplus_b200.types import default_config

pytestmark = pytest.mark.gpu

# Records whose first substep draws a normal on the edge between two floats: the Box-Muller transform
# by cos(2 pi u) and by cospi(2 u) round it to different ones (seed 5489, interval 1675900800).
ALONG_I = [129260329, 608104846, 1547727778, 1780776358, 1122334455, 7]
ALONG_J = [102851803, 157776535, 544102274, 1122334456, 8]


@pytest.mark.parametrize("axis,ids", [("i", ALONG_I), ("j", ALONG_J)])
def test_the_walk_draws_the_steps_normals(cuda_device, axis, ids):
    win = syn.config1_window(n_frames=2, eta=16, xi=17, s_rho=6, u=0.0, v=0.0)
    win.u[:], win.v[:], win.w[:] = 0.0, 0.0, 0.0
    win.times[1] = win.times[0] + 30.0  # one substep
    p = syn.uniform_particles(len(ids), win.eta, win.xi, seed=3, time=win.times[0])
    # on a node at the surface, where the position of both operators is exact
    p["id"], p["k"], p["j"], p["i"] = ids, 0.0, 7.0, 8.0
    got = []
    for learned in (0, 1):
        with Engine(0, surrogate=0) as engine:
            engine.set_config(default_config(random=True, randomSeed=5489, dti=30.0))
            engine.load_window(win)
            if learned:
                engine.set_surrogate()
                engine.set_options(surrogate=True)
            engine.set_particles(p)
            engine.move_interval(0)
            if learned:
                stats = engine.surrogate_stats()
                assert stats["run"] == len(ids) and stats["fallback"] == 0
            got.append(engine.get_particles()[axis])
    ahead = got[0] > (7.0 if axis == "j" else 8.0)  # backward from a node is not exact in FP32
    assert ahead[:3].all()
    assert np.array_equal(got[0][ahead], got[1][ahead])
