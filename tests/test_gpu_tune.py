"""The launch-shape autotuner changes no result.

A handle tuned partway (dem_autotune after 10 steps) must reach the same
state, bit for bit, as an untuned handle over the same steps; tuning a batch
likewise.  The chosen shapes are among the candidates, and those reported are
the ones that run."""
import numpy as np
import pytest

from mfix_dem import GpuSystem, abi
from cases import make_system, settling_case
from test_gpu_batch import _add, _batch, _cases, _compare

pytestmark = pytest.mark.gpu


def test_autotune_keeps_results():
    case, prm, arr, walls = settling_case(n_side=(8, 20, 8), spacing=0.98, jitter=0.03, coll="HERTZ",
                                          mew_r=0.01, seed=77)
    a = make_system(lambda p, n: GpuSystem(p, n), prm, arr, walls)
    b = make_system(lambda p, n: GpuSystem(p, n), prm, arr, walls)
    a.step(10)
    b.step(10)
    t = b.autotune(reps=3)
    assert t["pair_threads"] in (64, 128, 256) and t["pair_blocks_per_sm"] in (2, 4, 8, 16)
    assert t["gather_threads"] in (64, 128, 256) and t["neigh_threads"] in (32, 64, 128)
    assert t["pair_ms"] > 0 and t["gather_ms"] > 0 and t["neigh_ms"] > 0
    a.step(50)
    b.step(50)
    sa, sb = a.download_state(), b.download_state()
    for k in ("pos", "vel", "omega", "state"):
        assert np.array_equal(sa[k], sb[k]), k
    pa, pb = a.download_pairs(), b.download_pairs()
    for x, y in zip(pa, pb):
        assert np.array_equal(x, y)
    # set_tuning round trip
    b.set_tuning({"pair_threads": 128, "pair_blocks_per_sm": 4, "gather_threads": 64, "neigh_threads": 32})
    g = b.get_tuning()
    assert (g["pair_threads"], g["pair_blocks_per_sm"], g["gather_threads"], g["neigh_threads"]) == (128, 4, 64, 32)
    a.close()
    b.close()


def test_autotune_batch_keeps_results():
    cases = _cases(seeds=(51, 52, 53))
    bt = _batch(cases)
    ids = [_add(bt, c) for c in cases]
    bt.start(ids)
    bt.step(5)
    bt.autotune(reps=2)
    bt.step(45)
    from test_gpu_batch import _alone
    for sid, case in zip(ids, cases):
        g = _alone(case, 50)
        _compare(bt, sid, g)
        g.close()
    bt.close()


def _box(n_side, precision):
    _, prm, arr, walls = settling_case(n_side=n_side, box=tuple(1.0e-3 * (k + 2) for k in n_side), spacing=0.98,
                                       jitter=0.01, nsn=5, seed=7, precision=precision)
    return make_system(lambda p, n: GpuSystem(p, n), prm, arr, walls)


SHAPE = ("pair_threads", "pair_blocks_per_sm", "gather_threads", "neigh_threads")


# 1,728 spheres; 847,872, past eight windows of 128 pairs for each of the 16
# warps of a multiprocessor (of 148)
@pytest.mark.parametrize("n_side,precision,shape", [
    ((12, 12, 12), abi.DEM_PREC_FP64, (256, 8, 128, 128)),
    ((12, 12, 12), abi.DEM_PREC_SPLIT, (256, 8, 128, 128)),
    ((96, 92, 96), abi.DEM_PREC_FP64, (64, 8, 128, 128)),
    ((96, 92, 96), abi.DEM_PREC_SPLIT, (256, 8, 128, 128))])
def test_untuned_shapes(n_side, precision, shape):
    """An untuned handle reports the shapes its rules choose, and setting them
    changes none."""
    g = _box(n_side, precision)
    t = g.get_tuning()
    assert tuple(t[k] for k in SHAPE) == shape
    g.set_tuning(t)
    assert g.get_tuning() == t
    g.close()


def test_split_gather_shapes():
    """The split gather has blocks of 128 at most: a larger shape is taken as
    that, and the autotuner does not time it."""
    g = _box((12, 12, 12), abi.DEM_PREC_SPLIT)
    g.set_tuning({"pair_threads": 128, "pair_blocks_per_sm": 4, "gather_threads": 256, "neigh_threads": 64})
    assert g.get_tuning()["gather_threads"] == 128
    assert g.autotune(reps=3)["gather_threads"] in (64, 128)
    g.close()


def _on_a_floor():
    """400 spheres sliding on a floor of 12,800 facets of 0.25 mm, some five
    hundred in each DES cell; each starts inside a facet."""
    L, m, k = 20e-3, 80, 20
    case, prm, arr, _ = settling_case(n_side=(k, 1, k), box=(L, 12e-3, L), spacing=1.0, jitter=0.0, vmax=0.05, mew=0.3)
    arr["pos"] += np.array([[0.06e-3], [0.0], [0.09e-3]])
    arr["pos"][1], arr["vel"][1] = 0.499e-3, 0.0
    x, z = np.meshgrid(np.arange(m) * L / m, np.arange(m) * L / m, indexing="ij")
    p = np.stack([x, 0 * x, z], -1).reshape(-1, 3)
    ex, ez = np.array([L / m, 0, 0]), np.array([0, 0, L / m])
    tri = np.concatenate([np.stack([p, p + ez, p + ex], -1), np.stack([p + ex, p + ez, p + ex + ez], -1)])
    return prm, arr, (tri, np.tile([0.0, 1.0, 0.0], (tri.shape[0], 1)))


def test_autotune_times_the_walls():
    """The FP64 step does the walls in the pair launch, and so does the timed
    one: on a floor of many facets it takes several times the pairs alone.
    The wall histories are as they were."""
    prm, arr, floor = _on_a_floor()
    a, b, c = (make_system(lambda p, n: GpuSystem(p, n), prm, arr, w) for w in (floor, floor, (floor[0][:0], floor[1][:0])))
    for s in (a, b, c):
        s.step(10)
    t, bare = b.autotune(reps=20), c.autotune(reps=20)
    assert t["pair_ms"] > 3.0 * bare["pair_ms"]
    ha, hb = a.download_wall_history(), b.download_wall_history()
    assert (ha[0] > 0).sum() >= 400 and np.abs(ha[1]).max() > 0.0
    for x, y in zip(ha, hb):
        assert np.array_equal(x, y)
    for s in (a, b):
        s.step(40)
    sa, sb = a.download_state(), b.download_state()
    for k in ("pos", "vel", "omega", "state"):
        assert np.array_equal(sa[k], sb[k]), k
    for s in (a, b, c):
        s.close()
