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
