"""Dry cells whose depth is -0 (as -max(z, 0) gives) are dry cells: the second-order
reconstruction falls back to zero slopes there exactly as it does at +0."""
import ctypes

import numpy as np
import pytest

from adj_cases import _ptrs, copy_arrs, native_lib, scenario_case
from landslidehysea_gb300._abi import VARS

pyoracle = pytest.importorskip("pyoracle")


def coast(kind):
    p, arrs, _ = scenario_case(kind, 2)
    for k in (0, 3):
        arrs[k][arrs[k] == 0.0] = -0.0
    # a front that climbs the land: water moving toward the dry cells
    arrs[1] += 5.0 * arrs[0]
    arrs[2] -= 3.0 * arrs[0]
    return p, arrs


def by_oracle(p, arrs, n):
    a = copy_arrs(arrs)
    dt0 = pyoracle.initial_dt(p, a)
    _, dt, _ = pyoracle.run(p, a, n, dt=dt0)
    return dt0, dt, a


@pytest.mark.parametrize("kind", ["fjord", "shelf"])
def test_host_forward_equals_oracle(kind):
    p, arrs = coast(kind)
    n = 8
    dt0, dt, ref = by_oracle(p, arrs, n)
    assert all(np.isfinite(r).all() for r in ref)
    host = copy_arrs(arrs)
    dts = np.zeros(n + 1)
    assert native_lib("adj_host").adjh_forward(ctypes.byref(p), _ptrs(host), n, dts.ctypes.data) == 0
    assert dts[0] == dt0 and dts[n] == dt
    for k in range(6):
        assert np.array_equal(host[k], ref[k]), VARS[k]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["fjord", "shelf"])
def test_solver_equals_oracle(gpu_lib, kind):
    from landslidehysea_gb300.solver import Solver
    p, arrs = coast(kind)
    n = 8
    _, dt, ref = by_oracle(p, arrs, n)
    with Solver(p) as s:
        s.set_state({v: a.reshape(p.ny, p.nx) for v, a in zip(VARS, arrs)})
        s.step(n)
        s.synchronize()
        out = s.get_state()
        assert s.time()[1] == dt
    for k, v in enumerate(VARS[:6]):
        assert np.array_equal(out[v].reshape(-1), ref[k]), v
