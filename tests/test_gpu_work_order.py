"""The order in which the particle step takes its records (the sort by cell and level, the records
that take no step last) changes no result: every record moves on its own."""
import numpy as np
import pytest

from wacommplusplus_b200 import synthetic as syn
from wacommplusplus_b200.engine import Engine
from wacommplusplus_b200.types import default_config

pytestmark = pytest.mark.gpu


def mixed_records(n, win, seed):
    """Records over every level, among them dead, off-grid, not yet released and barely alive ones."""
    rng = np.random.default_rng(seed)
    p = syn.uniform_particles(n, win.eta, win.xi, seed=seed, time=win.times[0])
    p["k"] = rng.uniform(-win.sRho + 0.5, 0.5, n)
    p["time"] += rng.choice([0.0, 1700.0, 3600.0, 9000.0], n)
    kind = rng.integers(0, 12, n)
    p["health"][kind == 0] = -1.0
    p["health"][kind == 1] = 1e-7
    p["j"][kind == 2] = win.eta + 3.0
    p["i"][kind == 3] = np.nan
    return p


# 16 x 17 cells of 6 levels: 1,633 bins, told apart from 1,633 records on
@pytest.mark.parametrize("n", [1, 31, 1632, 1633, 4099])
@pytest.mark.parametrize("arithmetic,direction", [("fp32", 1), ("fp32", -1), ("reference", 1)])
def test_records_do_not_depend_on_the_sort(cuda_device, n, arithmetic, direction):
    win = syn.config1_window(n_frames=3, eta=16, xi=17, s_rho=6)
    p = mixed_records(n, win, n)
    cfg = default_config(random=True, trackingDirection=direction, backwardDiffusion=1)
    got, counts = [], []
    for sort in (0, 1):
        with Engine(0, arithmetic=arithmetic, sort_by_cell=sort) as engine:
            engine.load_window(win)
            engine.set_config(cfg)
            engine.set_particles(p)
            engine.concentration_reset(win.T)
            for t in (1, 1 + direction):  # the second sort walks the first one's order
                engine.move_interval(t)
            got.append(engine.get_particles())
            counts.append(engine.concentration())
    assert got[0].tobytes() == got[1].tobytes()
    assert np.array_equal(counts[0], counts[1])


# around one, two and all lanes per warp (592 warps), and in and out of the partly filled launches
@pytest.mark.parametrize("n", [1, 592, 593, 1185, 18944, 18945])
@pytest.mark.parametrize("arithmetic", ["fp32", "reference"])
def test_records_do_not_depend_on_how_a_launch_is_spread(cuda_device, n, arithmetic):
    win = syn.config1_window(n_frames=2, eta=16, xi=17, s_rho=6)
    few, many = mixed_records(n, win, 5), mixed_records(40000, win, 6)
    many["id"] += 50000
    got = []
    for p in (few, np.concatenate([few, many])):  # the larger launch fills its warps
        with Engine(0, arithmetic=arithmetic, sort_by_cell=0) as engine:
            engine.load_window(win)
            engine.set_config(default_config(random=True))
            engine.set_particles(p)
            engine.move_interval(0)
            got.append(engine.get_particles()[:n])
    assert got[0].tobytes() == got[1].tobytes()


# 39,999 and 40,000 records have their normals drawn ahead of the step, 40,001 do not; with 601
# substeps the draws of 27,869 records fit their buffer and those of 27,893 do not
@pytest.mark.parametrize("n,dti", [(1, 30.0), (777, 0.1), (39999, 60.0), (40001, 60.0),
                                   (27869, 6.0), (27893, 6.0), (3001, 7.3)])
@pytest.mark.parametrize("chunk", [0, 7])
def test_normals_drawn_ahead_are_the_steps_own(cuda_device, n, dti, chunk):
    win = syn.config1_window(n_frames=2, eta=16, xi=17, s_rho=6)
    if dti < 1:
        win.times[1] = win.times[0] + 60.0  # 0.1 does not sum to whole substeps
    p = mixed_records(40001, win, 9)
    got = []
    for count in (n, 40001):
        with Engine(0, sort_by_cell=0, substeps_per_launch=chunk) as engine:
            engine.load_window(win)
            engine.set_config(default_config(random=True, dti=dti))
            engine.set_particles(p[:count])
            engine.move_interval(0)
            got.append(engine.get_particles()[:n])
    assert got[0].tobytes() == got[1].tobytes()
