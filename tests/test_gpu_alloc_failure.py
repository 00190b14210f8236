"""A device allocation that fails leaves a handle that works once there is
memory: the call reports it, and what follows is as if it had not been made.

dem_test_fail_alloc (exported for these tests, not in the header) makes the
handle's n-th allocation from then on one that no device can serve, so the
error paths run without filling the device.
"""
import ctypes as C

import numpy as np
import pytest

from cases import coupled_case, make_coupled, make_system
from gpu_util import compare_state, rel_err

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
