"""Options of the plain step's launches: what is asked for is what is launched, with the same records."""
import numpy as np
import pytest

from test_gpu_dropin import same_records_packed_and_read
from test_gpu_work_order import mixed_records
from wacommplusplus_b200 import synthetic as syn
from wacommplusplus_b200.engine import Engine
from wacommplusplus_b200.types import default_config

pytestmark = pytest.mark.gpu


def walking_engine(n, intervals=1, **options):
    """An engine with n records in a random walk and its forcing loaded."""
    win = syn.config1_window(n_frames=intervals + 1, eta=16, xi=17, s_rho=6)
    engine = Engine(0, **options)
    engine.load_window(win)
    engine.set_config(default_config(random=True))
    engine.set_particles(syn.uniform_particles(n, win.eta, win.xi, seed=n, time=win.times[0]))
    return engine


def test_an_explicit_launch_shape_is_launched(cuda_device):
    """The automatic shape draws a small population's normals in a launch of their own."""
    records, launches = [], []
    for shape in (-1, 0, 1, 2, 3):
        with walking_engine(2000, 2, launch_shape=shape) as engine:
            for t in range(2):
                engine.move_interval(t)
            records.append(engine.get_particles().tobytes())
            launches.append(engine.stats()["launches"])
    assert all(r == records[0] for r in records)
    assert launches[1:] == [launches[0] - 1] * 4


def test_autotune_of_a_population_that_is_not_sorted_keeps_its_cadence(cuda_device):
    with walking_engine(2000, 6, sort_by_cell=3) as engine:
        before = engine.get_particles()
        shape, ms = engine.autotune(0)
        assert engine.options().launch_shape == shape and ms > 0
        assert engine.options().sort_by_cell == 3
        assert np.array_equal(before, engine.get_particles())


# five slabs of which the two at the ends are too small to be sorted, all five sorted from 530,446 on
@pytest.mark.parametrize("n", [393216, 530432, 530450])
def test_host_buffer_intervals_walk_the_sorted_slabs_orders_alone(cuda_device, n):
    with walking_engine(n, 3, rng="philox") as engine:
        p = engine.get_particles()
        for t in range(3):
            engine.move_interval(t)
        resident = engine.get_particles()
    with walking_engine(1, 3, rng="philox") as engine:
        for t in range(3):
            engine.move_interval_host(t, p)
    assert p.tobytes() == resident.tobytes()


# 96 MiB of node records and tables: packed from 1,048,576 records on
@pytest.mark.parametrize("n", [1048575, 1048576])
def test_the_drop_in_at_the_edge_of_its_packing_rule(cuda_device, n):
    win = syn.config1_window(n_frames=3, eta=512, xi=512, s_rho=4)
    win.times[:] = win.times[0] + 120.0 * np.arange(3)
    same_records_packed_and_read(win, n, False, 1)


# 27,915 records of 601 substeps fit the draws' buffer and 27,916 do not; 40,000 are drawn ahead and
# 40,001 are not; 0.1 and 7.3 do not sum to whole substeps. An engine's first interval draws in the step
# whatever the size.
@pytest.mark.parametrize("n,dti,ahead", [(1, 30.0, 1), (27915, 6.0, 1), (27916, 6.0, 0),
                                         (40000, 60.0, 1), (40001, 60.0, 0), (777, 0.1, 1),
                                         (3001, 7.3, 1)])
@pytest.mark.parametrize("chunk", [0, 7])
def test_normals_are_drawn_ahead_from_the_second_interval_on(cuda_device, n, dti, ahead, chunk):
    win = syn.config1_window(n_frames=3, eta=16, xi=17, s_rho=6)
    if dti < 1:
        win.times[:] = win.times[0] + 60.0 * np.arange(3)
    p = mixed_records(n, win, 9)
    got, launches = [], []
    for shape in (-1, 2):
        with Engine(0, sort_by_cell=0, launch_shape=shape, substeps_per_launch=chunk) as engine:
            engine.load_window(win)
            engine.set_config(default_config(random=True, dti=dti))
            engine.set_particles(p)
            for t in range(2):
                engine.move_interval(t)
                launches.append(engine.stats()["launches"])
            got.append(engine.get_particles())
    assert got[0].tobytes() == got[1].tobytes()
    assert launches == [launches[0], launches[0] + ahead, launches[0], launches[0]]


# 65 x 64 x 10: the stencil is kept up to 41,600 records
@pytest.mark.parametrize("drift", [0, 1])
def test_reference_arithmetic_at_the_edge_of_the_kept_stencil(cuda_device, drift):
    win = syn.RealisticForcing(eta=65, xi=64, s_rho=10, n_frames=2, seed=4, dlon=0.002, dlat=0.002,
                               land_fraction=0.1, water_border=2).window()
    win.windU10, win.windV10 = syn.vector_series((65, 64), 2, 8.0, 3, 8.0)
    p = mixed_records(41601, win, 12)
    p["driftObjectType"], p["driftSide"] = np.arange(len(p)) % 23, 1
    got = []
    for n in (41600, 41601):
        with Engine(0, arithmetic="reference") as engine:
            engine.load_window(win)
            engine.set_config(default_config(random=True, driftModel=drift, hasWind=bool(drift)))
            engine.set_particles(p[:n])
            engine.move_interval(0)
            got.append(engine.get_particles()[:41600])
    assert got[0].tobytes() == got[1].tobytes()


# 65 x 64 x 10: the drop-in keeps the stencil up to 41,600 records too
@pytest.mark.parametrize("n", [41600, 41601])
@pytest.mark.parametrize("environment", [False, True])
def test_the_drop_in_at_the_edge_of_the_kept_stencil(cuda_device, n, environment):
    win = syn.RealisticForcing(eta=65, xi=64, s_rho=10, n_frames=3, seed=8, land_fraction=0.1,
                               water_border=1).window()
    same_records_packed_and_read(win, n, environment, 1)


# intervals of three and four substeps, and launches of one
@pytest.mark.parametrize("seconds,chunk", [(90.0, 0), (120.0, 0), (120.0, 1)])
def test_records_of_short_launches_do_not_depend_on_the_sort(cuda_device, seconds, chunk):
    win = syn.config1_window(n_frames=3, eta=16, xi=17, s_rho=6)
    win.times[:] = win.times[0] + seconds * np.arange(3)
    p = mixed_records(40000, win, 4)
    p["time"] = win.times[0] + np.random.default_rng(4).choice([0.0, 31.0, 100.0, 150.0, 500.0], 40000)
    got = []
    for sort in (0, 1):
        with Engine(0, sort_by_cell=sort, substeps_per_launch=chunk) as engine:
            engine.load_window(win)
            engine.set_config(default_config(random=True))
            engine.set_particles(p)
            for t in range(2):
                engine.move_interval(t)
            got.append(engine.get_particles())
    assert got[0].tobytes() == got[1].tobytes()


# 255, 256 and 260 nodes: the records of a block of 256 leave it together
@pytest.mark.parametrize("eta,xi,s_rho", [(5, 17, 2), (8, 8, 3), (4, 13, 4)])
def test_node_records_at_the_edges_of_a_block(cuda_device, eta, xi, s_rho):
    win = syn.config1_window(n_frames=3, eta=eta, xi=xi, s_rho=s_rho)
    rng = np.random.default_rng(1)
    for name in ("u", "v", "w", "akt"):
        field = getattr(win, name)
        field[:] = rng.normal(0, 0.1, field.shape).astype(np.float32)
    same_records_packed_and_read(win, 600, False, 1)
