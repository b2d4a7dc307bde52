"""The colour passes, which parameters other than the reference's peso = 1 and beta >= 1 take (flux_fits), and
lsh_step_noalloc on a grid too wide for the flux pass: the single grid's overlapped and ordered steps, the
allocation-free step between calls of the flux pass on the same scratch, and the gradient, against the oracle."""
import ctypes

import numpy as np
import pytest

from adj_cases import copy_arrs, scenario_case, smooth_case, smooth_direction, wet_direction
from landslidehysea_gb300 import scenarios
from landslidehysea_gb300._abi import VARS

pytestmark = pytest.mark.gpu
pyoracle = pytest.importorskip("pyoracle")

OFF = pytest.mark.parametrize("name,value", [("peso", 0.9), ("beta", 0.9)])


def by_oracle(p, state, n):
    arrs = [np.ascontiguousarray(state[v], dtype=np.float64).copy() for v in VARS]
    t, dt, _ = pyoracle.run(p, arrs, n, dt=pyoracle.initial_dt(p, arrs))
    return t, dt, arrs


@pytest.mark.parametrize("order", [1, 2])
@OFF
def test_single_grid(gpu_lib, name, value, order):
    from landslidehysea_gb300.solver import Solver
    sc = scenarios.fjord(n=57, dcell_deg=0.007, order=order, cfl=0.5)
    setattr(sc.params, name, value)
    n = 40
    t, dt, ref = by_oracle(sc.params, sc.state, n)
    for ordered in (False, True):
        with Solver(sc.params) as s:
            s.set_state(sc.state)
            assert s.listed_tiles() == (0, 0)
            if ordered:
                for _ in range(n):
                    s.profile_step()
            else:
                s.step(n)
            s.synchronize()
            out = s.get_state()
            assert s.time()[:2] == (t, dt)
        for k, v in enumerate(VARS[:6]):
            assert np.array_equal(out[v], ref[k]), (v, ordered)


def test_noalloc_between_calls_of_the_flux_pass(gpu_lib):
    torch = pytest.importorskip("torch")
    mem = []
    for peso, kw in ((1.0, dict(n=40, dx=125.0)), (0.9, dict(n=57, dx=90.0)), (1.0, dict(nx=16000, ny=4, dx=2.0)),
                     (1.0, dict(nx=4, ny=4000, dx=2.0))):
        sc = scenarios.shelf(order=1, cfl=0.9, **kw)
        sc.params.peso = peso
        dev = [torch.tensor(np.ascontiguousarray(sc.state[v]), dtype=torch.float64, device="cuda") for v in VARS]
        mem.append((sc, dev, ctypes.c_double(0.0), ctypes.c_double(0.0)))
    calls, steps = 3, 4
    for _ in range(calls):  # each goes on from its own state, the scratch in other hands in between
        for sc, dev, t, dt in mem:
            ptrs = (ctypes.c_void_p * 7)(*[d.data_ptr() for d in dev])
            st = gpu_lib.lsh_step_noalloc(ctypes.byref(sc.params), ptrs, steps, ctypes.byref(t), ctypes.byref(dt), None)
            assert st == 0, gpu_lib.lsh_last_error().decode()
    torch.cuda.synchronize()
    for sc, dev, t, dt in mem:
        t_o, dt_o, ref = by_oracle(sc.params, sc.state, calls * steps)
        assert (t.value, dt.value) == (t_o, dt_o)
        for k, v in enumerate(VARS[:6]):
            assert np.array_equal(dev[k].cpu().numpy(), ref[k]), (sc.name, v)


@pytest.mark.parametrize("kind,order", [("smooth", 1), ("smooth", 2), ("fjord", 2)])
@OFF
def test_gradient_equals_tangent_linear(gpu_lib, name, value, kind, order):
    from landslidehysea_gb300.solver import Adjoint
    p, arrs, gauges = smooth_case(order=order) if kind == "smooth" else scenario_case(kind, order)
    setattr(p, name, value)
    n = 6
    _, _, eta = pyoracle.misfit_run(p, copy_arrs(arrs), n, gauges=gauges)
    tgt = eta + 0.01 * np.random.default_rng(5).standard_normal(eta.shape)
    with Adjoint(p, gauges) as A:
        J, _ = A.forward({v: a.reshape(p.ny, p.nx) for v, a in zip(VARS, arrs)}, n, tgt)
        g, gp = A.gradient(1.0)
    assert J == pyoracle.misfit_run(p, copy_arrs(arrs), n, gauges=gauges, target=tgt)[0]
    gpar = np.array([gp[k] for k in ("angle1", "mf0", "mfs", "r")])
    dirs = [(smooth_direction(p.nx, p.ny, 3, which=w) if kind == "smooth" else wet_direction(arrs, w, 3), [0, 0, 0, 0])
            for w in ((3,), (0,), (1, 2), (4, 5))]
    dirs += [([None] * 6, e) for e in ([1, 0, 0, 0], [0, 1, 0, 0], [0, 0, 1, 0], [0, 0, 0, 1])]
    for d, dpar in dirs:
        dd = [None if x is None else x.copy() for x in d]
        _, dJ, _, _ = pyoracle.tl_run(p, copy_arrs(arrs), dd, dpar, n, gauges=gauges, target=tgt)
        ad = sum(float(np.dot(g[v].reshape(-1), d[k])) for k, v in enumerate(VARS[:6]) if d[k] is not None)
        ad += float(np.dot(gpar, dpar))
        assert abs(ad - dJ) <= 1e-10 * max(abs(dJ), 1e-300), (dpar, dJ, ad)  # the flux pass's bound
