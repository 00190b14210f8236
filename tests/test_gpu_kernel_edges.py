"""Sizes at which the kernels of a step change their way of working, against
the oracle.

- the pair kernels take windows of 128 pairs, a lane screening four of them:
  pair counts at and around multiples of both;
- the wall work takes one particle per thread up to two blocks per
  multiprocessor and four past that: bed sizes on both sides, with the counts
  not a multiple of four, alone and in a batch, in the launch of the pairs and
  in one of their own (split precision, timed parts);
- the scans take a second level past 4096 tiles of 2048 cells: a search grid
  just over it; their scratch grows between replays of captured steps;
- a pair list that outgrows its arrays inside a captured step, with empty rows
  behind the last one that fits;
- the contact counts of passes that integrate and passes that do not;
- gas fields set again, on the same grid (the arrays are kept) and on another;
- the FP64 pair kernel in small blocks, for lists that keep every resident warp
  busy for eight windows, against the larger ones;
- contact lists of more than 32 entries, and warps with more than 128;
- masses past the range in which quotients share a reciprocal;
- the deposition of more than one solids phase;
- coupled steps with either integrator, in split precision, and with periodic axes
  (where the cell search of the next step cannot ride on the integration).

FP64 results are the oracle's bit for bit (as everywhere in the parity tests);
the split path is held to the tolerances of its own tests (positions 1e-6,
velocities 1e-3 of the largest); coupled states to 1e-10 relative, since the
drag calls pow.
"""
import numpy as np
import pytest

from cases import coupled_case, make_coupled, make_system, settling_case, state_arrays
from gpu_util import compare_pairs, compare_state, pair_both, rel_err

pytestmark = pytest.mark.gpu


def _gpu(p, n):
    from mfix_dem import GpuSystem
    return GpuSystem(p, n)


def _chain(m, precision, nsn=10, rho=2500.0, kn=1000.0, intg="EULER"):
    """m + 1 spheres of 1 mm in a row along x, 0.98 d apart: m pairs, each in
    contact at the start, with small seeded velocities across the row."""
    from mfix_dem import params as P
    d, n = 1e-3, m + 1
    rng = np.random.default_rng(300 + m)
    pos = np.empty((3, n))
    pos[0] = (np.arange(n) + 2.0) * 0.98 * d
    pos[1] = pos[2] = 4.0 * d
    vel = rng.uniform(-0.02, 0.02, (3, n))
    arr = state_arrays(pos, vel, np.zeros((3, n)), np.full(n, 0.5 * d), np.full(n, rho))
    hi = ((n + 4.0) * d, 8.0 * d, 8.0 * d)
    case = P.DemCase(d_p0=(d,), ro_s0=(rho,), coll_model="LSD", kn=kn, kn_w=kn, des_en_input=0.9, intg_method=intg,
                     des_en_wall_input=[0.9], mew=0.2, mew_w=0.2, mew_r=0.01, mew_rw=0.01, domain_hi=hi,
                     neighbor_search_n=nsn, force_precision=precision)
    prm, _ = P.build_params(case, arr["radius"], arr["pmass"], arr["phase"], arr["state"])
    return prm, arr, P.default_walls((0.0, 0.0, 0.0), hi)


@pytest.mark.parametrize("m", [1, 2, 3, 4, 127, 128, 129, 255, 385])
@pytest.mark.parametrize("prec", ["fp64", "split"])
def test_pair_windows(m, prec):
    from mfix_dem import abi
    g, o = pair_both(*_chain(m, abi.DEM_PREC_SPLIT if prec == "split" else abi.DEM_PREC_FP64))
    assert g.pair_count() == m
    for steps in (1, 2, 30):
        g.step(steps)
        o.step(steps)
        if prec == "fp64":
            compare_state(g, o, exact=True)
            compare_pairs(g, o)
            assert g.stats()["n_contacts"] == o.stats()["n_contacts"]
    if prec == "split":
        sg, so = g.download_state(), o.download_state()
        assert rel_err(sg["pos"], so["pos"]) <= 1e-6
        assert rel_err(sg["vel"], so["vel"]) <= 1e-3


@pytest.mark.parametrize("n_side", [(43, 41, 42), (43, 41, 43), (45, 41, 43)])
def test_wall_work_by_size(n_side):
    """74,045, 75,808 and 79,334 spheres: one per thread up to 75,776 (148
    multiprocessors); the outer layers start at or in the walls."""
    box = tuple(0.999e-3 * k for k in n_side)
    case, prm, arr, walls = settling_case(n_side=n_side, box=box, spacing=0.999, jitter=0.01, vmax=0.2, nsn=5, seed=61)
    arr = {k: (v[..., :-1].copy() if v.ndim else v) for k, v in arr.items()}   # a count that is no multiple of four
    g, o = pair_both(prm, arr, walls)
    g.step(17)
    o.step(17)
    compare_state(g, o, exact=True)
    assert g.stats()["n_wall_contacts"] == o.stats()["n_wall_contacts"] > 1000
    fg, pg = g.download_wall_history()
    fo, po = o.download_wall_history()
    assert np.array_equal(fg, fo)
    assert np.array_equal(pg[fg >= 0], po[fo >= 0])


def _full_box(n_side, seed=61, **kw):
    """Spheres whose outer layers start at or in the walls, one less than the
    lattice holds."""
    box = tuple(0.999e-3 * k for k in n_side)
    case, prm, arr, walls = settling_case(n_side=n_side, box=box, spacing=0.999, jitter=0.01, vmax=0.2, nsn=5, seed=seed,
                                          **kw)
    return case, prm, {k: (v[..., :-1].copy() if v.ndim else v) for k, v in arr.items()}, walls


@pytest.mark.parametrize("coll", ["LSD", "HERTZ"])
@pytest.mark.parametrize("prec,timed", [("fp64", True), ("split", False), ("split", True)])
def test_walls_in_their_own_launch(coll, prec, timed):
    """79,334 spheres in split precision, or with the parts of the step timed."""
    from mfix_dem import abi
    case, prm, arr, walls = _full_box((45, 41, 43), coll=coll,
                                      precision=abi.DEM_PREC_SPLIT if prec == "split" else abi.DEM_PREC_FP64)
    g, o = pair_both(prm, arr, walls)
    if timed:
        g.set_profiling(2)
    g.step(17)
    o.step(17)
    assert o.stats()["n_wall_contacts"] > 1000
    if prec == "fp64":
        compare_state(g, o, exact=True)
        assert g.stats()["n_wall_contacts"] == o.stats()["n_wall_contacts"]
        assert all(np.array_equal(a, b) for a, b in zip(g.download_wall_history(), o.download_wall_history()))
    else:
        sg, so = g.download_state(), o.download_state()
        assert rel_err(sg["pos"], so["pos"]) <= 1e-6
        assert rel_err(sg["vel"], so["vel"]) <= 1e-3


@pytest.mark.parametrize("coll", ["LSD", "HERTZ"])
@pytest.mark.parametrize("prec", ["fp64", "split"])
def test_wall_work_of_a_batch(coll, prec):
    """Boxes of 41,327 and 39,311 spheres, together past 75,776, each against
    the oracle; the second box has other walls and another period."""
    from mfix_dem import abi
    from oracle_ffi import OracleSystem
    from test_gpu_batch import _add, _batch
    precision = abi.DEM_PREC_SPLIT if prec == "split" else abi.DEM_PREC_FP64
    cases = [_full_box((36, 28, 41), seed=62, coll=coll, precision=precision),
             _full_box((27, 52, 28), seed=63, coll=coll, mew=0.3, precision=precision)]
    bt = _batch(cases)
    ids = [_add(bt, c) for c in cases]
    bt.start(ids)
    bt.step(17)
    for sid, (case, prm, arr, walls) in zip(ids, cases):
        o = make_system(OracleSystem, prm, arr, walls)
        o.step(17)
        assert o.stats()["n_wall_contacts"] > 500
        sb, so = bt.download_state(sid), o.download_state()
        for k in ("pos", "vel", "omega"):
            if prec == "fp64":
                assert np.array_equal(sb[k], so[k]), k
            elif k != "omega":
                assert rel_err(sb[k], so[k]) <= (1e-6 if k == "pos" else 1e-3), k
    bt.close()


def test_scan_of_many_search_cells():
    """A DES grid of 205^3 cells (8.9 million with its ghost layers, past 4096
    tiles of 2048)."""
    from mfix_dem import params as P
    d, L = 1e-3, 0.65
    rng = np.random.default_rng(5)
    k = np.arange(12)
    cluster = np.stack(np.meshgrid(k, k, k, indexing="ij"), 0).reshape(3, -1) * 1.02 * d
    pos = np.concatenate([cluster + c for c in (0.004, 0.31, 0.632)], axis=1) + rng.uniform(-2e-5, 2e-5, (3, 3 * 1728))
    n = pos.shape[1]
    arr = state_arrays(pos, rng.uniform(-0.1, 0.1, (3, n)), np.zeros((3, n)), np.full(n, 0.5 * d), np.full(n, 2500.0))
    case = P.DemCase(d_p0=(d,), ro_s0=(2500.0,), coll_model="LSD", kn=1000.0, kn_w=1000.0, des_en_input=0.9,
                     des_en_wall_input=[0.9], mew=0.1, mew_w=0.1, domain_hi=(L, L, L), desgridsearch=(205, 205, 205),
                     neighbor_search_n=4)
    prm, _ = P.build_params(case, arr["radius"], arr["pmass"], arr["phase"], arr["state"])
    g, o = pair_both(prm, arr, P.default_walls((0.0, 0.0, 0.0), (L, L, L)))
    compare_pairs(g, o)
    g.step(9)
    o.step(9)
    compare_state(g, o, exact=True)
    compare_pairs(g, o)


def test_scan_scratch_grown_between_replays():
    """A fluid grid of more cells than any scan before it, set on a system whose
    steps have been captured: the next replays scan in the new scratch."""
    from test_gpu_alloc_failure import _fine_gas
    prm, arr, walls, fields = _fine_gas()
    g, o = pair_both(prm, arr, walls)
    for s in (g, o):
        s.step(1 + 4 + 4 * 5)   # one replay of each buffer parity that follows
    before = g.memory_info()["scratch_bytes"]
    for s in (g, o):
        s.set_gas_fields(*fields)
    assert g.memory_info()["scratch_bytes"] > before
    for s in (g, o):
        s.step(4 * 5)
    compare_state(g, o, exact=True)
    compare_pairs(g, o)


def test_captured_build_is_the_first():
    """A handle with uploaded pairs whose first build lies in a captured period,
    with many more search cells than particles."""
    from oracle_ffi import OracleSystem
    case, prm, arr, walls = settling_case(n_side=(8, 8, 8), box=(40e-3, 40e-3, 40e-3), spacing=1.0, nsn=5, seed=23)
    g, o = _gpu(prm, arr["radius"].size), make_system(OracleSystem, prm, arr, walls)
    g.upload_state(arr["pos"], arr["vel"], arr["omega"], arr["radius"], arr["pmass"], arr["omoi"], arr["state"],
                   arr["phase"])
    g.upload_pairs(*o.download_pairs())
    o.set_walls(walls[0][:0], walls[1][:0])
    for s in (g, o):
        s.step(1, nn_first=2)
        s.step(10, nn_first=6)
    compare_state(g, o, exact=True)
    compare_pairs(g, o)


def test_rows_of_an_overflowing_list():
    """1,000 spheres drawn together within one captured period, from no pair to
    several times the capacity of 16 n + 1024: the error is reported, every row
    ends inside the list that is left, steps over it run, and the list made
    again is the oracle's."""
    from mfix_dem import abi
    from mfix_dem import params as P
    from mfix_dem.system import DemError
    d, nsn, L = 1e-3, 5, 24e-3
    k = np.arange(10) - 4.5
    rng = np.random.default_rng(17)
    off = np.stack(np.meshgrid(k, k, k, indexing="ij")).reshape(3, -1) * 1.5 * d + rng.uniform(-1e-5, 1e-5, (3, 1000))
    n = off.shape[1]
    arr = state_arrays(0.5 * L + off, np.zeros((3, n)), np.zeros((3, n)), np.full(n, 0.5 * d), np.full(n, 2500.0))
    case = P.DemCase(d_p0=(d,), ro_s0=(2500.0,), coll_model="LSD", kn=1000.0, kn_w=1000.0, des_en_input=0.9,
                     des_en_wall_input=[0.9], mew=0.1, mew_w=0.1, grav=(0.0, 0.0, 0.0), domain_hi=(L, L, L),
                     neighbor_search_n=nsn)
    prm, _ = P.build_params(case, arr["radius"], arr["pmass"], arr["phase"], arr["state"])
    g, o = pair_both(prm, arr, P.default_walls((0.0, 0.0, 0.0), (L, L, L)))
    vel = -0.75 * off / (nsn * prm.dtsolid)
    for s in (g, o):
        s.step(nsn)
        s.upload_state(arr["pos"], vel, arr["omega"])
    assert g.pair_count() == 0
    cap = g.memory_info()["pair_capacity"]
    with pytest.raises(DemError) as e:
        g.step(nsn)
    assert e.value.code == abi.DEM_ERR_PAIR_OVERFLOW
    o.step(nsn)
    assert o.pair_count() > 2 * cap
    ni, nb, _ = g.download_pairs()
    assert nb.size == cap and ni[-1] == cap + 1
    assert (np.diff(ni) >= 0).all() and ni.max() <= cap + 1
    assert nb.min() >= 1 and nb.max() <= n
    whole = o.download_state()
    g.step(2, nn_first=2 * nsn + 1)
    assert np.isfinite(g.download_state()["vel"]).all()
    for s in (g, o):
        s.upload_state(whole["pos"], np.zeros((3, n)), whole["omega"])
        s.init_neighbors()
    compare_pairs(g, o)
    for s in (g, o):
        s.step(3, nn_first=2 * nsn + 1)
    compare_state(g, o, exact=True)


def test_contact_counts_of_mixed_passes():
    """Counts are those of the last force pass, whether it integrated or not."""
    case, prm, arr, walls = settling_case(n_side=(6, 10, 6), spacing=0.98, jitter=0.02, nsn=5)
    g, o = pair_both(prm, arr, walls)

    def same():
        a, b = g.stats(), o.stats()
        assert (a["n_contacts"], a["n_wall_contacts"]) == (b["n_contacts"], b["n_wall_contacts"])
        assert a["n_contacts"] > 0

    for s in (g, o):
        s.calc_force()
    same()
    for s in (g, o):
        s.cfnewvalues()
        s.nn = 1
        s.step(3)
    same()
    for s in (g, o):
        s.calc_force()
        s.calc_force()
        s.cfnewvalues()
    same()
    for s in (g, o):
        s.step(13, nn_first=6)
    same()
    compare_state(g, o, exact=True)


@pytest.mark.parametrize("prec", ["fp64", "split"])
def test_contact_counts_of_a_force_error(prec):
    """Behind dem_force_error, whose second pass is the last force evaluation,
    whether a step or a pass without integration came before."""
    from mfix_dem import abi
    case, prm, arr, walls = settling_case(n_side=(6, 10, 6), spacing=0.98, jitter=0.02, vmax=0.0, nsn=5,
                                          precision=abi.DEM_PREC_SPLIT if prec == "split" else abi.DEM_PREC_FP64)
    g, o = pair_both(prm, arr, walls)
    for again in range(2):
        for s in (g, o):
            s.calc_force()
        g.force_error()
        a, b = g.stats(), o.stats()
        assert (a["n_contacts"], a["n_wall_contacts"]) == (b["n_contacts"], b["n_wall_contacts"])
        assert a["n_contacts"] > 0 and a["n_wall_contacts"] > 0
        for s in (g, o):
            s.step(1)
        g.force_error()
        for s in (g, o):
            s.calc_force()
        assert g.stats()["n_contacts"] == o.stats()["n_contacts"]


@pytest.mark.parametrize("interp", ["GARG_2012", "NONE"])
def test_gas_fields_set_again(interp):
    from mfix_dem import configs
    from oracle_ffi import OracleSystem
    ct = coupled_case(interp=interp)
    g, o = make_coupled(_gpu, ct), make_coupled(OracleSystem, ct)
    grid, f = ct[5], ct[6]
    coarse = configs.coupled(n=1500, cells=(4, 12, 4), dx=2e-3, interp=interp)[5:7]
    for again in ((grid, f), (grid, {k: v * (1.0 if k == "ep_g" else 0.7) for k, v in f.items()}), coarse, (grid, f)):
        for s in (g, o):
            s.step_coupled(7)
            s.set_gas_fields(again[0], again[1]["ep_g"], again[1]["u_g"], again[1]["v_g"], again[1]["w_g"])
            s.step_coupled(6)
        compare_state(g, o)
        for a, b in zip(g.get_mean_fields(), o.get_mean_fields()):
            assert rel_err(a, b) <= 1e-10
        call = "drag_gs_gas1" if interp == "NONE" else "drag_gs_gas0"
        for a, b in zip(getattr(g, call)(), getattr(o, call)()):
            assert rel_err(a, b) <= 1e-10


def test_dense_list_in_small_blocks():
    """847,872 touching spheres: past eight windows of 128 pairs for each of
    the 16 warps that a multiprocessor (of 148) keeps."""
    n_side = (96, 92, 96)
    case, prm, arr, walls = settling_case(n_side=n_side, box=tuple(1.0e-3 * (k + 2) for k in n_side), spacing=0.98,
                                          jitter=0.01, vmax=0.1, nsn=5, seed=7)
    a, b = make_system(_gpu, prm, arr, walls), make_system(_gpu, prm, arr, walls)
    b.set_tuning({"pair_threads": 256, "pair_blocks_per_sm": 8, "gather_threads": 256, "neigh_threads": 128})
    for s in (a, b):
        s.step(7)
    assert a.pair_count() >= 8 * 128 * 16 * 148
    compare_state(a, b, exact=True)
    assert a.stats()["n_contacts"] == b.stats()["n_contacts"] > a.pair_count() // 2


@pytest.mark.parametrize("prec", ["fp64", "split"])
@pytest.mark.parametrize("big", [0, -1])
def test_long_contact_lists(big, prec):
    """A sphere of 10 mm with 80 of 1 mm touching it (numbered first: a row of
    80 pairs; last: 80 incoming ones) beside a block of 8^3 with up to six
    contacts each."""
    from mfix_dem import abi
    from mfix_dem import params as P
    R, r = 5e-3, 0.5e-3
    k = np.arange(80) + 0.5
    up, turn = 1.0 - 2.0 * k / 80, np.pi * (1.0 + 5.0 ** 0.5) * k
    ring = np.sqrt(1.0 - up * up)
    shell = 8e-3 + 0.999 * (R + r) * np.stack([ring * np.cos(turn), up, ring * np.sin(turn)])
    a = np.arange(8) * 0.98 * 2.0 * r
    block = np.stack(np.meshgrid(a, a, a, indexing="ij")).reshape(3, -1) + np.array([[20e-3], [4e-3], [4e-3]])
    small = np.concatenate([shell, block], axis=1)
    rng = np.random.default_rng(41)
    pos = np.concatenate([np.full((3, 1), 8e-3), small], axis=1)
    rad = np.concatenate([[R], np.full(small.shape[1], r)])
    if big == -1:
        pos, rad = np.roll(pos, -1, axis=1), np.roll(rad, -1)
    n = rad.size
    arr = state_arrays(pos, rng.uniform(-0.02, 0.02, (3, n)), np.zeros((3, n)), rad, np.full(n, 2500.0))
    hi = (32e-3, 16e-3, 16e-3)
    case = P.DemCase(d_p0=(2.0 * r,), ro_s0=(2500.0,), coll_model="LSD", kn=1000.0, kn_w=1000.0, des_en_input=0.9,
                     des_en_wall_input=[0.9], mew=0.2, mew_w=0.2, mew_r=0.01, mew_rw=0.01, domain_hi=hi,
                     neighbor_search_n=10, force_precision=abi.DEM_PREC_SPLIT if prec == "split" else abi.DEM_PREC_FP64)
    prm, _ = P.build_params(case, arr["radius"], arr["pmass"], arr["phase"], arr["state"])
    g, o = pair_both(prm, arr, P.default_walls((0.0, 0.0, 0.0), hi))
    for steps in (1, 2, 20):
        g.step(steps)
        o.step(steps)
        if prec == "fp64":
            compare_state(g, o, exact=True)
            compare_pairs(g, o)
    sg, so = g.download_state(), o.download_state()
    assert rel_err(sg["pos"], so["pos"]) <= 1e-6
    assert rel_err(sg["vel"], so["vel"]) <= 1e-3


@pytest.mark.parametrize("intg", ["EULER", "ADAMS_BASHFORTH"])
@pytest.mark.parametrize("scale", [1.0, 1e128])
def test_quotients_of_large_masses(scale, intg):
    """Density and stiffness times 1e128 (masses past 2^400): the same motion,
    with the accelerations divided plainly."""
    from mfix_dem import abi
    g, o = pair_both(*_chain(70, abi.DEM_PREC_FP64, rho=2500.0 * scale, kn=1000.0 * scale, intg=intg))
    for steps in (1, 2, 30):
        g.step(steps)
        o.step(steps)
        assert o.stats()["n_contacts"] > 0 or steps == 30
        compare_state(g, o, exact=True)
        compare_pairs(g, o)
    assert np.isfinite(g.download_state()["vel"]).all()


@pytest.mark.parametrize("interp", ["GARG_2012", "NONE"])
def test_deposition_of_two_phases(interp):
    """The coupled case with every third sphere of a lighter second phase: a
    node (or cell) sums its phases apart, four entries at a time, counts with
    every remainder."""
    import dataclasses
    from mfix_dem import params as P
    from oracle_ffi import OracleSystem
    case, prm, arr, walls, info, grid, f = coupled_case(interp=interp)
    d, rho = case.d_p0[0], case.ro_s0[0]
    case = dataclasses.replace(case, n_phases=2, d_p0=(d, d), ro_s0=(rho, 0.5 * rho), des_en_input=0.9,
                               des_en_wall_input=[0.9, 0.9])
    ph = 1 + (np.arange(arr["radius"].size) % 3 == 0)
    arr = state_arrays(arr["pos"], arr["vel"], arr["omega"], arr["radius"], np.where(ph == 1, rho, 0.5 * rho), phase=ph)
    prm, info = P.build_params(case, arr["radius"], arr["pmass"], arr["phase"], arr["state"])
    grid.ro_s[1] = 0.5 * rho
    ct = (case, prm, arr, walls, info, grid, f)
    g, o = make_coupled(_gpu, ct), make_coupled(OracleSystem, ct)
    for s in (g, o):
        s.step_coupled(8)
    compare_state(g, o)
    for a, b in zip(g.get_mean_fields(), o.get_mean_fields()):
        assert rel_err(a, b) <= 1e-10
    assert prm.n_phases == 2
    assert rel_err(g.calc_des_bedheight(), o.calc_des_bedheight()) <= 1e-10


@pytest.mark.parametrize("periodic", [(False, False, False), (True, False, True)])
@pytest.mark.parametrize("interp", ["GARG_2012", "NONE"])
@pytest.mark.parametrize("intg,prec", [("EULER", "fp64"), ("ADAMS_BASHFORTH", "fp64"), ("EULER", "split"),
                                       ("ADAMS_BASHFORTH", "split")])
def test_coupled_step_forms(intg, prec, interp, periodic):
    """The coupled case with its spheres in contact, 23 steps with three pair
    builds; with periodic x and z some cross a face."""
    import dataclasses
    from mfix_dem import abi
    from mfix_dem import params as P
    from oracle_ffi import OracleSystem
    case, prm, arr, walls, info, grid, f = coupled_case(spacing=0.99, nsn=10, interp=interp)
    case = dataclasses.replace(case, intg_method=intg, periodic=periodic,
                               force_precision=abi.DEM_PREC_SPLIT if prec == "split" else abi.DEM_PREC_FP64)
    prm, info = P.build_params(case, arr["radius"], arr["pmass"], arr["phase"], arr["state"])
    rng = np.random.default_rng(77)
    arr = dict(arr, vel=rng.uniform(-2.0, 2.0, arr["vel"].shape))
    if periodic[0]:   # the first layers about the faces
        arr["pos"] = arr["pos"] - np.array([[0.24e-3], [0.0], [0.24e-3]])
    walls = P.default_walls(case.domain_lo, case.domain_hi, periodic=periodic)
    ct = (case, prm, arr, walls, info, grid, f)
    g, o = make_coupled(_gpu, ct), make_coupled(OracleSystem, ct)
    x0 = o.download_state()["pos"][0]
    for steps in (1, 3, 19):
        for s in (g, o):
            s.step_coupled(steps)
        sg, so = g.download_state(), o.download_state()
        assert np.array_equal(sg["state"], so["state"])
        if prec == "fp64":
            compare_state(g, o)
            assert g.stats()["n_contacts"] == o.stats()["n_contacts"] > 100
        else:
            assert rel_err(sg["pos"], so["pos"]) <= 1e-6
            assert rel_err(sg["vel"], so["vel"]) <= 1e-3
        for a, b in zip(g.get_mean_fields(), o.get_mean_fields()):
            assert rel_err(a, b) <= (1e-10 if prec == "fp64" else 1e-4)
    if periodic[0]:
        assert (np.abs(so["pos"][0] - x0) > 4e-3).sum() > 3
