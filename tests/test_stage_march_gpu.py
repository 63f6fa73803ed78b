"""The plane-marching stage kernel at the sizes where its tiling can go wrong:
grids smaller than a tile, partly filled last tiles in y and z, columns that are
no multiple of 16 (cp.async instead of TMA) or of 8 bytes (scalar RK accesses),
cut nodes next to a z-tile's edge, and both walls in one tile; with and without
the Sutherland laws, drag and convective exchange.  One step against the CPU
oracle: 1e-10 per field in FP64 and 1e-5 relative L2 in FP32, the tolerances of
the parity tests; every block form and both loaders give the same bits.
"""
import numpy as np
import pytest

import oracle_py as O
from conftest import field_errors

pytestmark = pytest.mark.gpu
FORMS = {"fp32": [(8, 16, 512), (8, 16, 384), (8, 8, 256)], "fp64": [(8, 8, 512), (8, 8, 256)]}
FULL = dict(alpha_s=0.002, sigma_s=5500.0, sutherland_viscosity=1, sutherland_conductivity=1)


@pytest.mark.parametrize("size,method,extra", [
    ((4, 4, 5), "RK4", {}), ((5, 7, 13), "RK4", FULL), ((9, 35, 33), "RK2", {}), ((17, 30, 45), "RK4", {}),
    ((12, 50, 97), "Euler", FULL), ((40, 14, 64), "RK4", {}), ((7, 26, 225), "RK4", {}),
])
def test_one_step_matches_oracle_in_every_form(size, method, extra, params_from_text, monkeypatch):
    from wildfires_b200 import Solver, configs
    Nx, Ny, Nz = size
    # a hill whose foot to top passes through several z-tiles where there are any
    case = configs.hill(Nx=Nx, Ny=Ny, Nz=Nz, Nt=1, L=60.0, H=0.5 * Nz, jitter=0.2, seed=Nz, method=method, **extra)
    P = params_from_text(configs.param_text(case.params))
    y0, p0 = case.fields(P)
    yo, po = O.steps(P, y0, p0, 1)
    for prec, tol in (("fp64", 1e-10), ("fp32", 1e-5)):
        first = None
        for flag in ("0", "1"):
            monkeypatch.setenv("WF_NO_TMA", flag)
            for form in FORMS[prec]:
                with Solver(P, prec) as s:
                    s.set_stage_tile(*form)
                    s.upload(y0, p0)
                    s.step(1)
                    y, p = s.download()
                if first is None:
                    first = (y, p)
                    for f, (linf, l2) in field_errors(P, y, yo).items():
                        assert l2 <= tol and (prec == "fp32" or linf <= tol), (prec, f, linf, l2)
                assert np.array_equal(y, first[0]) and np.array_equal(p, first[1]), (prec, flag, form)


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_long_walks_refill_the_planes_whose_walls_were_written(prec, params_from_text, monkeypatch):
    """Walks of more planes than the ring holds (260 x 130 x 24: ten and more), both walls in each tile:
    the values written beyond the walls of a plane, then the TMA box that takes its place, against
    copies that know no other way of writing.  Same bits."""
    from wildfires_b200 import Solver, configs
    case = configs.hill(Nx=260, Ny=130, Nz=24, Nt=1, L=200.0, H=12.0, jitter=0.2, seed=3)
    P = params_from_text(configs.param_text(case.params))
    y0, p0 = case.fields(P)
    out = []
    for flag in ("0", "1"):
        monkeypatch.setenv("WF_NO_TMA", flag)
        with Solver(P, prec) as s:
            s.upload(y0, p0)
            s.step(2)
            out.append(s.download())
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("size,extra", [((13, 30, 20), {}), ((9, 25, 33), FULL)])
def test_fuel_that_jumps_across_the_periodic_seam(size, extra, params_from_text):
    """The planes i = Nx-1 and j = Ny-1 repeat planes 0 in u, v, w and T, but their fuel is
    their own (an uneven bed need not close on itself): drag, reaction and convective
    exchange there take it, the SGS inputs that the neighbours read take plane 0's.  Phi
    against the CPU oracle with burning cells on the seam, in every form; tolerances as above.
    The oracle's SGS inputs of the seam take the seam's fuel for its neighbours on the seam: a
    difference of at most nu / T dS / 3d in a velocity's rate (dS what the fuel changes in T's
    rate, d the least spacing, 1/3 the divergence source's weight)."""
    from wildfires_b200 import Solver, configs
    Nx, Ny, Nz = size
    case = configs.hill(Nx=Nx, Ny=Ny, Nz=Nz, Nt=1, L=60.0, H=0.5 * Nz, jitter=0.2, seed=Nz, Y_h=3.0, **extra)
    P = params_from_text(configs.param_text(case.params))
    y0, _ = case.fields(P)
    r, N, rng = P.rec, Nx * Ny * Nz, np.random.default_rng(5)
    T, Y = y0[3 * N:4 * N].reshape(size), y0[4 * N:].reshape(Nx, Ny, r.Nz_Y_max)
    live = (np.arange(Nz) > P.cut_nodes()[..., None]) & (np.arange(Nz) < P.nz_y()[..., None])
    T[live] = 700.0 + 0.5 * (T[live] - 300.0)
    T[-1], T[:, -1] = T[0], T[:, 0]
    Y[:] = np.where(live[:, :, :Y.shape[2]], rng.uniform(0.0, 1.0, Y.shape) * (rng.uniform(size=Y.shape) < 0.8), 0.0)
    assert live[-1].any() and live[:, -1].any()
    want = O.phi(P, y0)
    closed = y0.copy()
    Yc = closed[4 * N:].reshape(Y.shape)
    Yc[-1], Yc[:, -1] = Yc[0], Yc[:, 0]
    dS = np.max(np.abs(O.phi(P, closed) - want)[3 * N:4 * N])
    sgs = r.mu * (T.max() / r.T_inf) / (r.T_inf * r.rho_inf) * dS / (3 * min(r.dx, r.dy, np.diff(P.z()).min()))
    for prec, tol in (("fp64", 1e-10), ("fp32", 1e-5)):
        for form in FORMS[prec]:
            with Solver(P, prec) as s:
                s.set_stage_tile(*form)
                got = s.phi(y0)
            for q, (f, (linf, l2)) in enumerate(field_errors(P, got, want).items()):
                k = want[q * N:(q + 1) * N]
                more = sgs / np.max(np.abs(k)) if f in "uvw" else 0.0
                assert l2 <= tol + more * np.sqrt(N) * np.max(np.abs(k)) / np.linalg.norm(k), (prec, form, f, linf, l2)
                assert prec == "fp32" or linf <= tol + more, (prec, form, f, linf, l2)
