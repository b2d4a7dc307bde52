"""The flux pass and cell update (lsh_passes.cuh: flux_edge, update_cell) give
the colour passes' bits (do_edge, volume_cell), both compiled for the host:
the parity cases, and random films from 10 um to 1 m on odd and one-wide
grids, at the CFL step and at steps five times too long, where the positivity
limiter acts on chains of edges."""
import ctypes

import numpy as np
import pytest

from adj_cases import native_lib
from gpu_cases import PARITY_CASES, case
from landslidehysea_gb300._abi import VARS, default_params


def differing(oracle, p, state, nsteps, too_long):
    lib = native_lib("flux_host")
    lib.fluxc_compare.restype = ctypes.c_longlong
    lib.fluxc_compare.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_double, ctypes.c_double,
                                  ctypes.POINTER(ctypes.c_longlong)]
    arrs = [np.ascontiguousarray(state[v], dtype=np.float64).reshape(-1) for v in VARS]
    dt = oracle.initial_dt(p, arrs)
    marked = ctypes.c_longlong()
    bad = lib.fluxc_compare(ctypes.byref(p), (ctypes.c_void_p * 7)(*[a.ctypes.data for a in arrs]), nsteps,
                            dt * (5.0 if too_long else 1.0), 5.0 * dt if too_long else 0.0, ctypes.byref(marked))
    return bad, marked.value


@pytest.mark.parametrize("name", PARITY_CASES)
def test_flux_pass_equals_the_colour_passes(oracle, name):
    p, state, steps = case(name)
    p.track_eta_max = 1
    for too_long in (False, True):
        assert differing(oracle, p, state, min(steps, 25), too_long)[0] == 0


def films(nx, ny, order):
    rng = np.random.default_rng(5 + nx + 100 * ny)
    p = default_params(nx, ny, order=order, dx=3.0, dy=2.0, cfl=0.9, r=0.5, angle_deg=5.0, mf0=0.03, mfs=0.03, mfc=0.01,
                       eps_h=1e-3, borde_sup=1.0, borde_inf=0.0, borde_izq=-1.0, borde_der=1.0)
    sh = (ny, nx)
    h1 = np.where(rng.random(sh) < 0.3, 0.0, 10.0 ** rng.uniform(-5, 0, sh))
    h2 = np.where(rng.random(sh) < 0.5, 0.0, 10.0 ** rng.uniform(-5, 0, sh))
    st = {"h1": h1, "h2": h2, "H": rng.uniform(0, 2, sh)}
    for k, h in (("q1x", h1), ("q1y", h1), ("q2x", h2), ("q2y", h2)):
        st[k] = h * rng.normal(0, 3, sh)
    return p, st


FILMS = pytest.mark.parametrize("nx,ny", [(1, 1), (1, 7), (6, 1), (16, 17), (33, 5), (40, 40)])


@pytest.mark.parametrize("order", [1, 2])
@FILMS
def test_flux_pass_equals_the_colour_passes_on_films(oracle, nx, ny, order):
    p, st = films(nx, ny, order)
    for too_long in (False, True):
        bad, marked = differing(oracle, p, st, 10, too_long)
        assert bad == 0
        assert marked > 0 or nx * ny == 1  # the limiter's path was taken


@pytest.mark.parametrize("order", [1, 2])
@FILMS
def test_a_recomputed_stage_keeps_the_colour_passes_sums(oracle, nx, ny, order):
    """What the reverse sweep reads: accumulators, their partial sums, the reconstruction's branches."""
    p, st = films(nx, ny, order)
    lib = native_lib("flux_host")
    lib.fluxc_keep.restype = ctypes.c_longlong
    lib.fluxc_keep.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_double]
    arrs = [np.ascontiguousarray(st[v], dtype=np.float64).reshape(-1) for v in VARS]
    dt = oracle.initial_dt(p, arrs)
    for scale in (1.0, 5.0):
        assert lib.fluxc_keep(ctypes.byref(p), (ctypes.c_void_p * 7)(*[a.ctypes.data for a in arrs]), scale * dt) == 0
