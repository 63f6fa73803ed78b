"""The pressure solve at the edges of its vertical solvers: for the Thomas kernel the
fewest planes, plane counts around the eight that are loaded ahead, systems that
do not fill a block's 32, and its largest number of planes (256); past that the
checkpointed kernel with a partial last segment, systems that do not fill a
block's 128 (Ny = 258), and y transforms of 8 and 16 points, whose blocks hold
the z weights of more slices than they have threads.  The FP64 solve against the
CPU oracle's within 1e-11 of the largest pressure: both round each elimination
step once or twice (1e-16), and the long waves amplify that by at most the square
of the number of planes (260^2, so 7e-12).
"""
import numpy as np
import pytest

import oracle_py as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(4, 4, 5), (5, 6, 9), (6, 63, 10), (9, 66, 17), (7, 130, 18),
                                  (6, 9, 257), (6, 9, 258), (5, 17, 259), (6, 9, 260), (4, 258, 258)])
def test_pressure_matches_oracle(size, params_from_text):
    from wildfires_b200 import Solver, configs
    Nx, Ny, Nz = size
    case = configs.hill(Nx=Nx, Ny=Ny, Nz=Nz, Nt=1, L=60.0, H=30.0, jitter=0.2, seed=Nz)
    P = params_from_text(configs.param_text(case.params))
    y0, p0 = case.fields(P)
    want, _ = O.pressure(P, y0, y0, p0)
    with Solver(P, "fp64") as s:
        got, _ = s.pressure(y0, y0, p0)
    assert np.max(np.abs(got - want)) <= 1e-11 * np.max(np.abs(want))
