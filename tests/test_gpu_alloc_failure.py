"""A device allocation that fails leaves a handle that works once there is
memory: the call reports it, and what follows is as if it had not been made.

dem_test_fail_alloc (exported for these tests, not in the header) makes the
handle's n-th allocation from then on one that no device can serve, so the
error paths run without filling the device.
"""
import ctypes as C
import gc

import numpy as np
import pytest

from cases import coupled_case, make_system, settling_case
from gpu_util import compare_pairs, compare_state, pair_both

pytestmark = pytest.mark.gpu


def _gpu(p, n):
    from mfix_dem import GpuSystem
    return GpuSystem(p, n)


def _fail(g, nth=1):
    assert g._lib.dem_test_fail_alloc(g._h, C.c_int32(nth)) == 0


def _refused(call, *args, **kw):
    from mfix_dem import abi
    from mfix_dem.system import DemError
    with pytest.raises(DemError) as e:
        call(*args, **kw)
    assert e.value.code == abi.DEM_ERR_CUDA
    return str(e.value)


def _refused_at(make, what, call):
    """A system from make() whose call(system) has failed at the allocation
    that the message calls `what`."""
    for nth in range(1, 40):
        g = make()
        _fail(g, nth)
        if what in _refused(call, g):
            _fail(g, 0)
            return g
        g.close()
    raise AssertionError(what)


def test_next_call_is_not_blamed():
    """CUDA's pending error of a failed allocation is not taken for one of the
    launches of the next call."""
    from oracle_ffi import OracleSystem
    case, prm, arr, walls, info, grid, f = coupled_case()
    g, o = make_system(_gpu, prm, arr, walls), make_system(OracleSystem, prm, arr, walls)
    _fail(g)
    _refused(g.set_gas_fields, grid, f["ep_g"], f["u_g"], f["v_g"], f["w_g"])
    for s in (g, o):
        s.calc_force()
        s.cfnewvalues()
        s.nn = 1
        s.step(5)
    compare_state(g, o, exact=True)


@pytest.mark.parametrize("what", ["scan", "candidates"])
def test_first_build_repeated(what):
    """The particles counted into the search cells, and the pairs counted into
    the incoming lists, are counted once when the build is made again."""
    case, prm, arr, walls = settling_case(n_side=(14, 14, 14), box=(16e-3, 40e-3, 16e-3), spacing=0.99, nsn=5, seed=12)

    def make():
        s = _gpu(prm, arr["radius"].size)
        s.upload_state(arr["pos"], arr["vel"], arr["omega"], arr["radius"], arr["pmass"], arr["omoi"], arr["state"],
                       arr["phase"])
        return s

    from oracle_ffi import OracleSystem
    g = _refused_at(make, what, lambda s: s.init_neighbors())
    o = make_system(OracleSystem, prm, arr, walls)
    g.init_neighbors()
    compare_pairs(g, o)
    g.set_walls(*walls)
    for s in (g, o):
        s.step(23)
    compare_state(g, o, exact=True)
    compare_pairs(g, o)


def test_later_build_repeated():
    """A build inside a step that fails leaves the list before it whole, its
    length included: it can be made again and the run continued."""
    case, prm, sparse, walls = settling_case(n_side=(12, 12, 12), box=(40e-3, 40e-3, 40e-3), spacing=2.5, nsn=5,
                                             vmax=0.01, seed=13)
    dense = settling_case(n_side=(12, 12, 12), box=(40e-3, 40e-3, 40e-3), spacing=0.98, nsn=5, vmax=0.01, seed=13)[2]
    g, o = pair_both(prm, sparse, walls)
    n0 = g.pair_count()
    for s in (g, o):
        s.upload_state(dense["pos"], dense["vel"], dense["omega"], dense["radius"], dense["pmass"], dense["omoi"],
                       dense["state"], dense["phase"])
    _fail(g)
    assert "candidates" in _refused(g.step, 1)
    assert g.pair_count() == n0
    o.step(1)
    for s in (g, o):
        s.neighbour()
    assert g.pair_count() > 4 * n0
    compare_pairs(g, o)
    for s in (g, o):
        s.step(28, nn_first=2)
    compare_state(g, o, exact=True)
    compare_pairs(g, o)


@pytest.mark.parametrize("nth", [2, 6, 12])
def test_pair_arrays_given_back(nth):
    """Pair arrays that do not all fit leave the handle its old ones and the
    device its memory."""
    import torch
    prm, arr, walls = settling_case(n_side=(50, 40, 50), box=(52e-3, 42e-3, 52e-3), spacing=1.0, seed=15)[1:]
    n = arr["radius"].size
    g = make_system(_gpu, prm, arr, walls)
    ni, nb, pf = g.download_pairs()
    gc.collect()
    before, cap = torch.cuda.mem_get_info()[0], g.memory_info()["pair_capacity"]
    each = cap // n + 8
    many = np.minimum(np.arange(1, n + 1) * each, n * each) + 1
    _fail(g, nth)
    assert "pairs" in _refused(g.upload_pairs, many, np.ones(n * each, np.int32), np.zeros((n * each, 3)))
    # 12.8 MB and more were allocated before the one that failed; small blocks
    # of other handles may have gone back besides
    assert torch.cuda.mem_get_info()[0] >= before
    assert g.memory_info()["pair_capacity"] == cap
    for a, b in zip(g.download_pairs(), (ni, nb, pf)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("nth", [1, 2, 3, 4])
def test_walls_that_do_not_fit(nth):
    """Facets, or their bins, without room: no walls, until they are set again."""
    from oracle_ffi import OracleSystem
    prm, arr, walls = settling_case(n_side=(8, 6, 8), box=(9e-3, 40e-3, 9e-3), spacing=1.05, nsn=5, vmax=0.3, seed=18)[1:]
    none = (walls[0][:0], walls[1][:0])
    g, o = make_system(_gpu, prm, arr, walls), make_system(OracleSystem, prm, arr, none)
    _fail(g, nth)
    _refused(g.set_walls, *walls)
    for s in (g, o):
        s.step(12)
    compare_state(g, o, exact=True)
    for s in (g, o):
        s.set_walls(*walls)
        s.step(40)
    assert o.stats()["n_wall_contacts"] == g.stats()["n_wall_contacts"] > 0
    compare_state(g, o, exact=True)


def test_walls_past_the_limits_of_a_batch():
    """Facet bins that a batch has no room for: the system has no walls, the
    other keeps its own, and the room is free for smaller ones."""
    from mfix_dem import GpuBatch, abi, load_library
    from mfix_dem import params as P
    from mfix_dem.system import DemError
    from test_gpu_batch import _add, _compare, _entry
    a = settling_case(n_side=(8, 6, 8), box=(9e-3, 40e-3, 9e-3), spacing=1.05, nsn=5, vmax=0.3, seed=19)
    b = settling_case(n_side=(6, 6, 6), box=(9e-3, 40e-3, 9e-3), spacing=1.05, nsn=5, vmax=0.3, seed=20)
    lim = P.batch_limits(load_library(), [_entry(a), _entry(b)])
    many = tuple(np.concatenate([w] * 40) for w in b[3])
    lim.max_facets = 4000
    bt = GpuBatch(a[1], lim)
    ids = [_add(bt, a), _add(bt, (b[0], b[1], b[2], (b[3][0][:0], b[3][1][:0])))]
    with pytest.raises(DemError) as e:
        bt.set_walls(ids[1], *many)
    assert e.value.code == abi.DEM_ERR_CAPACITY and "bin" in str(e.value)
    bt.start(ids)
    bt.step(12)
    alone = [make_system(_gpu, *a[1:]), make_system(_gpu, b[1], b[2], (b[3][0][:0], b[3][1][:0]))]
    for sid, g in zip(ids, alone):
        g.step(12)
        _compare(bt, sid, g)
    bt.set_walls(ids[1], *b[3])
    alone[1].set_walls(*b[3])
    bt.step(40)
    for sid, g in zip(ids, alone):
        g.step(40)
        assert g.stats()["n_wall_contacts"] > 0
        _compare(bt, sid, g)
    bt.close()


@pytest.mark.parametrize("kind,nth", [("outflow", 1), ("inflow", 1), ("inflow", 2)])
def test_boundaries_that_do_not_fit(kind, nth):
    """The boundaries before stay (here none), until they are set again."""
    from inflow_cases import inflow_case
    from oracle_ffi import OracleSystem
    case, prm, arr, walls, bc, obc = inflow_case(outflow=True)
    g, o = make_system(_gpu, prm, arr, walls), make_system(OracleSystem, prm, arr, walls)
    _fail(g, nth)
    if kind == "outflow":
        _refused(g.set_outflow_bcs, [obc])
    else:
        _refused(g.set_inflow_bcs, [bc], seed=9)
    for s in (g, o):
        s.step(12)
    compare_state(g, o, exact=True)
    for s in (g, o):
        s.set_outflow_bcs([obc])
        s.set_inflow_bcs([bc], seed=9)
        s.step(100)
    compare_state(g, o, exact=True)
    assert g.stats()["n_inflow_added"] == o.stats()["n_inflow_added"] > 0


def test_tuning_that_fails_chooses_nothing():
    """The automatic launch shapes stay when the autotuner has no room for the
    histories it keeps (more of them than the upload staged)."""
    prm, arr, walls = settling_case(n_side=(12, 12, 12), spacing=0.75, jitter=0.01, seed=16)[1:]
    g = make_system(_gpu, prm, arr, walls)
    assert 26 * g.pair_count() > 100 * arr["radius"].size
    t = g.get_tuning()
    _fail(g)
    _refused(g.autotune)
    assert g.get_tuning() == t and t["gather_threads"] == 128


def _fine_gas(interp="GARG_2012"):
    """Spheres of 1 mm in fluid cells of 0.25 mm, several for each search cell."""
    prm, arr, walls = settling_case(n_side=(8, 10, 8), box=(10e-3, 15e-3, 10e-3), spacing=1.02, nsn=5, seed=14)[1:]
    grid, f = coupled_case(cells=(40, 60, 40), dx=0.25e-3, d=0.25e-3, n=600, interp=interp)[5:]
    return prm, arr, walls, (grid, f["ep_g"], f["u_g"], f["v_g"], f["w_g"])


@pytest.mark.parametrize("interp", ["GARG_2012", "NONE"])
def test_fluid_cells_counted_again(interp):
    """The particles of the fluid cells, on a grid of more cells than any scan
    before needed."""
    from oracle_ffi import OracleSystem
    prm, arr, walls, fields = _fine_gas(interp)
    g = _refused_at(lambda: make_system(_gpu, prm, arr, walls), "scan", lambda s: s.set_gas_fields(*fields))
    g._ncell = fields[1].shape[0]
    o = make_system(OracleSystem, prm, arr, walls)
    o.set_gas_fields(*fields)
    for steps in (0, 4):
        for s in (g, o):
            s.step(steps)
            s.comp_mean_fields()
        for a, b in zip(g.get_mean_fields(), o.get_mean_fields()):
            assert np.array_equal(a, b)
