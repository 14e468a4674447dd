"""The order in which the particle step takes its records (the sort by cell and level, the records
that take no step last) changes no result: every record moves on its own."""
import numpy as np
import pytest

from oracle import bindings as ob
from wacommplusplus_b200 import synthetic as syn
from wacommplusplus_b200.engine import Engine
from wacommplusplus_b200.types import default_config

pytestmark = pytest.mark.gpu


def mixed_records(n, win, seed):
    """Records over every level, among them dead, off-grid, not yet released and barely alive ones."""
    rng = np.random.default_rng(seed)
    p = syn.uniform_particles(n, win.eta, win.xi, seed=seed, time=win.times[0])
    p["k"] = rng.uniform(-win.sRho + 0.5, 0.5, n)
    p["time"] += rng.choice([0.0, 130.0, 1700.0, 3600.0, 4444.4, 9000.0, 10799.9], n)
    kind = rng.integers(0, 12, n)
    p["health"][kind == 0] = -1.0
    p["health"][kind == 1] = 1e-7
    p["j"][kind == 2] = win.eta + 3.0
    p["i"][kind == 3] = np.nan
    return p


# sorted from 37,889 records on; 64 x 65 cells of 10 levels: 41,601 bins, levels told apart from that
# many records on, release times in up to four parts; in up to sixteen on 16 x 17 cells
@pytest.mark.parametrize("n,eta,xi", [(1, 64, 65), (37888, 64, 65), (37889, 64, 65), (41600, 64, 65),
                                      (41601, 64, 65), (90000, 16, 17)])
@pytest.mark.parametrize("arithmetic,direction", [("fp32", 1), ("fp32", -1), ("reference", 1)])
def test_records_do_not_depend_on_the_sort(cuda_device, n, eta, xi, arithmetic, direction):
    win = syn.config1_window(n_frames=4, eta=eta, xi=xi, s_rho=10)
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


# the reference arithmetic keeps its velocity stencil up to 37,888 records
@pytest.mark.parametrize("drift", [0, 1])
def test_reference_arithmetic_with_and_without_the_kept_stencil(cuda_device, drift):
    win = syn.RealisticForcing(eta=40, xi=44, s_rho=6, n_frames=2, seed=4, dlon=0.002, dlat=0.002,
                               land_fraction=0.1, water_border=2).window()
    win.windU10, win.windV10 = syn.vector_series((40, 44), 2, 8.0, 3, 8.0)
    p = mixed_records(37889, win, 12)
    p["driftObjectType"], p["driftSide"] = np.arange(len(p)) % 23, 1
    cfg = default_config(random=True, driftModel=drift, hasWind=bool(drift))
    got = []
    for n in (37888, 37889):
        with Engine(0, arithmetic="reference") as engine:
            engine.load_window(win)
            engine.set_config(cfg)
            engine.set_particles(p[:n])
            engine.move_interval(0)
            got.append(engine.get_particles()[:37888])
    assert got[0].tobytes() == got[1].tobytes()


def test_reference_arithmetic_on_subnormal_and_fill_values(cuda_device):
    """Time blends round to float precision on the subnormal grid too: a vertical velocity of a few
    subnormal steps decides at the surface closure, and the fill value stays finite."""
    win = syn.config1_window(n_frames=2, eta=16, xi=17, s_rho=6)
    rng = np.random.default_rng(5)
    win.w[:] = (rng.integers(-3, 4, win.w.shape) * 1.401298464324817e-45).astype(np.float32)
    win.u[:, :, 12:, :] = 1e37
    p = mixed_records(3000, win, 14)
    p["k"][::2] = 0.0
    cfg = default_config(random=False, upperClosure=2)
    want = ob.oracle_move(cfg, p.copy(), win, 0, ob.SEMANTICS_HOST, threads=1)
    with Engine(0, arithmetic="reference") as engine:
        engine.load_window(win)
        engine.set_config(cfg)
        engine.set_particles(p)
        engine.move_interval(0)
        got = engine.get_particles()
    assert np.array_equal(got["health"] > 0, want["health"] > 0)
    for name in ("k", "j", "i"):
        assert np.array_equal(got[name], want[name], equal_nan=True), name


# one slab, five slabs and the ramp in the FP32 step; one and two slabs in the reference arithmetic
@pytest.mark.parametrize("n,arithmetic", [(393215, "fp32"), (393216, "fp32"), (2999999, "fp32"),
                                          (3000000, "fp32"), (393216, "reference"),
                                          (2097152, "reference")])
def test_host_buffer_slabs_at_the_edges_of_their_rule(cuda_device, n, arithmetic):
    win = syn.config1_window(n_frames=2, eta=16, xi=17, s_rho=6)
    win.times[1] = win.times[0] + 300.0
    p = mixed_records(n, win, 3)
    with Engine(0, arithmetic=arithmetic, rng="philox") as engine:
        engine.load_window(win)
        engine.set_config(default_config(random=True))
        engine.set_particles(p)
        engine.concentration_reset(2)
        engine.move_interval(0)
        resident, counts = engine.get_particles(), engine.concentration()
        engine.concentration_reset(2)
        engine.move_interval_host(0, p)
        assert p.tobytes() == resident.tobytes()
        assert np.array_equal(engine.concentration(), counts)
