"""Tiles that nothing can reach are left out of a step (k_clock's lists): a
mostly dry grid, off the tile size both ways, with water and a granular layer
that run out over several tiles of dry land, against the oracle bit for bit at
both orders; then another state on the same context, whose water lies where the
first run left the tiles out."""
import numpy as np
import pytest

from landslidehysea_gb300._abi import VARS, default_params

pytestmark = pytest.mark.gpu

NX, NY, STEPS = 203, 121, 300


def columns(order, corner):
    """Land that falls away from `corner`, with a column of water and a granular pile inside it there."""
    p = default_params(NX, NY, order=order, dx=5.0, dy=5.0, cfl=0.5, r=0.5, angle_deg=4.0, mf0=0.02,
                       mfs=0.02, eps_h=1e-2, gravity=9.81, borde_sup=1.0, borde_inf=1.0, borde_izq=1.0, borde_der=1.0)
    p.track_eta_max = 1
    i, j = np.meshgrid(np.arange(NX), np.arange(NY))
    if corner:
        i, j = NX - 1 - i, NY - 1 - j
    wave = 0.3 * np.sin(0.2 * i) * np.cos(0.3 * j)
    st = {v: np.zeros((NY, NX)) for v in VARS}
    st["H"] = 5.0 + 0.04 * i + 0.02 * j + wave
    st["h2"] = np.where((i > 12) & (i < 30) & (j > 8) & (j < 25), 3.0, 0.0)
    st["h1"] = np.where((i < 44) & (j < 31), 7.0, 0.0) - st["h2"]
    return p, st


@pytest.mark.parametrize("order", [1, 2])
def test_a_front_over_dry_land(gpu_lib, oracle, order):
    from landslidehysea_gb300.solver import Solver
    oracle.set_threads(0)
    with Solver(columns(order, 0)[0]) as s:
        for corner in (0, 1):
            p, st = columns(order, corner)
            s.set_state(st)
            n, total = s.listed_tiles()
            assert n == total  # a new state lists every tile
            s.step(1)
            first = s.listed_tiles()[0]
            s.step(STEPS - 1)
            s.synchronize()
            last = s.listed_tiles()[0]
            assert 0 < first < last < total
            out, (t, dt, _), eta = s.get_state(), s.time(), s.eta_max()
            arrs = [np.ascontiguousarray(st[v]).copy() for v in VARS]
            em, et = arrs[0] + arrs[3] - arrs[6], np.zeros((NY, NX))
            t_o, dt_o, _ = oracle.run(p, arrs, STEPS, dt=oracle.initial_dt(p, arrs), eta=(em, et))
            assert (t, dt) == (t_o, dt_o)
            for k, v in enumerate(VARS[:6]):
                assert np.array_equal(out[v], arrs[k]), v
            assert np.array_equal(eta[0], em) and np.array_equal(eta[1], et)
            wet = (arrs[0] > 0) | (arrs[3] > 0)
            assert wet.sum() > 2 * ((st["h1"] > 0).sum())  # the front has crossed several tiles
