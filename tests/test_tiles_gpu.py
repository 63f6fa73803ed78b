"""Block forms of the fused stage pass: every compiled form gives bit-identical
states (a cell's arithmetic does not depend on the tiling, and the Van Driest
shortcut only skips factors that are exactly 1), and a context has its form, by
precision and grid size or by WF_STAGE_TILE, from its creation on."""
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu
SHAPES32 = [(8, 16, 512), (8, 16, 384), (8, 8, 256)]


def _run(P, g, prec, shape, n):
    from wildfires_b200 import Solver
    with Solver(P, prec) as s:
        if shape is not None:
            s.set_stage_tile(*shape)
        s.upload(g["y0"], g["p0"])
        s.step(n)
        return s.download(), s.stage_tile()


@pytest.mark.parametrize("name", ["hill_rk4", "flat_33x33x16_10", "stretched_rk2"])
def test_tile_shapes_give_identical_states(name, params_from_text):
    g = load_golden(name)
    P = params_from_text(g["params"])
    n = int(g["nsteps"])
    (y0, p0), _ = _run(P, g, "fp32", SHAPES32[0], n)
    for shape in SHAPES32[1:]:
        (y, p), used = _run(P, g, "fp32", shape, n)
        assert used == shape
        assert np.array_equal(y, y0) and np.array_equal(p, p0), shape


def _grid(size, params_from_text):
    from wildfires_b200 import configs
    case = configs.hill(Nx=size[0], Ny=size[1], Nz=size[2], Nt=1, L=60.0, H=0.5 * size[2], jitter=0.2, seed=2)
    P = params_from_text(configs.param_text(case.params))
    return P, {"y0": case.fields(P)[0], "p0": case.fields(P)[1]}


@pytest.mark.parametrize("size,form64", [((33, 33, 16), (8, 8, 256)), ((50, 50, 39), (8, 8, 256)),
                                         ((50, 50, 40), (8, 8, 512))])
def test_form_by_precision_and_grid_from_creation_on(size, form64, params_from_text):
    """FP64 below 100,000 cells takes the smaller blocks; operators and steps use the same form."""
    from wildfires_b200 import Solver
    P, g = _grid(size, params_from_text)
    for prec, form in (("fp32", (8, 8, 256)), ("fp64", form64)):
        with Solver(P, prec) as s:
            assert s.stage_tile() == form
            s.phi(g["y0"])
            assert s.stage_tile() == form
            s.upload(g["y0"], g["p0"])
            s.step(1)
            assert s.stage_tile() == form


def test_form_named_in_the_environment(params_from_text, monkeypatch):
    from wildfires_b200 import Ensemble, Solver, WfError
    P, g = _grid((20, 30, 24), params_from_text)
    with Solver(P, "fp32") as s:
        want = s.phi(g["y0"])
    for form in SHAPES32:
        monkeypatch.setenv("WF_STAGE_TILE", "%dx%d/%d" % form)
        with Solver(P, "fp32") as s:
            assert s.stage_tile() == form
            assert np.array_equal(s.phi(g["y0"]), want)
    for bad in ("16x16", "8x16/256", "x", ""):
        monkeypatch.setenv("WF_STAGE_TILE", bad)
        with Solver(P, "fp32") as s:
            assert s.stage_tile() == (8, 8, 256)
            assert np.array_equal(s.phi(g["y0"]), want)
            s.upload(g["y0"], g["p0"])
            for _ in range(2):
                with pytest.raises(WfError, match="WF_STAGE_TILE"):
                    s.step(1)
            s.set_stage_tile(8, 16)
            s.step(1)
        with Ensemble([P], "fp32") as e:
            for _ in range(2):
                with pytest.raises(WfError, match="WF_STAGE_TILE"):
                    e.step(1)


def test_unknown_shape_is_rejected(params_from_text):
    from wildfires_b200 import Solver, WfError
    g = load_golden("hill_rk4")
    P = params_from_text(g["params"])
    with Solver(P, "fp32") as s:
        with pytest.raises(WfError):
            s.set_stage_tile(16, 16)
        with pytest.raises(WfError):
            s.set_stage_tile(8, 16, 256)


@pytest.mark.parametrize("name", ["hill_rk4", "vardens_rk4"])
def test_fp64_block_forms_give_identical_states(name, params_from_text):
    g = load_golden(name)
    P = params_from_text(g["params"])
    n = int(g["nsteps"])
    (y0, p0), _ = _run(P, g, "fp64", (8, 8, 256), n)
    for shape in [(8, 8, 512)]:
        (y, p), used = _run(P, g, "fp64", shape, n)
        assert used == shape
        assert np.array_equal(y, y0) and np.array_equal(p, p0), shape


@pytest.mark.parametrize("name", ["hill_rk4", "flat_33x33x16_10"])
def test_tma_and_cp_async_tile_loads_give_identical_states(name, params_from_text, monkeypatch):
    """State planes arrive by TMA; WF_NO_TMA=1 copies them by cp.async.  Same
    bits either way, for every compiled form."""
    g = load_golden(name)
    P = params_from_text(g["params"])
    n = int(g["nsteps"])
    for shape in SHAPES32:
        monkeypatch.setenv("WF_NO_TMA", "0")
        (y0, p0), _ = _run(P, g, "fp32", shape, n)
        monkeypatch.setenv("WF_NO_TMA", "1")
        (y, p), _ = _run(P, g, "fp32", shape, n)
        assert np.array_equal(y, y0) and np.array_equal(p, p0), shape


def test_tma_tile_loads_on_a_grid_with_interior_tiles(params_from_text, monkeypatch):
    """A grid with tiles that wrap around in y and tiles that do not (64 x 80 x 32, hill case):
    TMA and cp.async loads give bit-identical states after two steps, and all
    forms agree."""
    from wildfires_b200 import configs
    case = configs.hill(Nx=64, Ny=80, Nz=32, Nt=2, L=120.0, H=24.0, jitter=0.3, seed=6)
    P = params_from_text(configs.param_text(case.params))
    y0, p0 = case.fields(P)
    g = {"y0": y0, "p0": p0}
    out = []
    for flag in ("0", "1"):
        monkeypatch.setenv("WF_NO_TMA", flag)
        for shape in SHAPES32:
            (y, p), _ = _run(P, g, "fp32", shape, 2)
            out.append((y, p))
    for y, p in out[1:]:
        assert np.array_equal(y, out[0][0]) and np.array_equal(p, out[0][1])
