"""The routes a step can take, against each other bit for bit: the flux pass
with a warp per block (small grids) and a tile per block (large ones), on
either side of the line; the colour passes, which peso other than 1 takes, on
one grid, in an ensemble and in a batch of adjoints beside a member that does
not need them."""
import numpy as np
import pytest

from adj_cases import copy_arrs, smooth_case
from landslidehysea_gb300 import scenarios
from landslidehysea_gb300._abi import VARS

pytestmark = pytest.mark.gpu
pyoracle = pytest.importorskip("pyoracle")


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("nx,ny", [(1000, 250), (1010, 252)])  # 3969 and 4096 tiles; the line lies at 4000
def test_small_and_large_grid_kernels(gpu_lib, oracle, nx, ny, order):
    from landslidehysea_gb300.solver import Solver
    sc = scenarios.shelf(nx=nx, ny=ny, dx=20.0, order=order, cfl=0.5 if order == 2 else 0.9)
    arrs = [np.ascontiguousarray(sc.state[v], dtype=np.float64).copy() for v in VARS]
    oracle.run(sc.params, arrs, 3, dt=oracle.initial_dt(sc.params, arrs))
    with Solver(sc.params) as s:
        s.set_state(sc.state)
        s.step(3)
        out = s.get_state()
    for k, v in enumerate(VARS[:6]):
        assert np.array_equal(out[v], arrs[k]), v


@pytest.mark.parametrize("order", [1, 2])
def test_ensemble_on_the_colour_passes(gpu_lib, oracle, order):
    from landslidehysea_gb300.solver import Batch
    scs = [scenarios.shelf(n=n, dx=25.0, seed=n, order=order, cfl=0.5) for n in (21, 40)]
    scs[1].params.peso = 0.9
    with Batch([sc.params for sc in scs]) as b:
        for k, sc in enumerate(scs):
            b.set_state(k, sc.state)
        b.step(9)
        b.synchronize()
        out = [b.get_state(k) for k in range(2)]
    for sc, o in zip(scs, out):
        arrs = [np.ascontiguousarray(sc.state[v], dtype=np.float64).copy() for v in VARS]
        oracle.run(sc.params, arrs, 9, dt=oracle.initial_dt(sc.params, arrs))
        for k, v in enumerate(VARS[:6]):
            assert np.array_equal(o[v], arrs[k]), v


@pytest.mark.parametrize("order", [1, 2])
def test_adjoints_on_the_colour_passes(gpu_lib, order):
    from landslidehysea_gb300.solver import Adjoint, AdjointBatch
    mem = [smooth_case(order=order), smooth_case(nx=23, ny=9, order=order), smooth_case(nx=2, ny=33, order=order)]
    mem[1][0].peso = 0.9
    n = 6
    state = lambda p, a: {v: a[i].reshape(p.ny, p.nx) for i, v in enumerate(VARS)}
    tg = []
    for p, a, g in mem:
        _, _, eta = pyoracle.misfit_run(p, copy_arrs(a), n, gauges=g)
        tg.append(eta + 0.01)
    with AdjointBatch([m[0] for m in mem], [m[2] for m in mem]) as B:
        J, _ = B.forward([state(p, a) for p, a, _ in mem], n, tg)
        grads, gps = B.gradient([1.0] * 3)
    for i, (p, a, g) in enumerate(mem):
        with Adjoint(p, g) as A:
            j, _ = A.forward(state(p, a), n, tg[i])
            grad, gp = A.gradient(1.0)
        assert j == J[i] and gp == gps[i]
        for v in VARS[:6]:
            assert np.array_equal(grad[v], grads[i][v]), (i, v)
