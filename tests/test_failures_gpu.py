"""Error paths, driven from the host (no GPU fault): every device allocation
wf_create makes is refused in turn by the library's failure injection; each time
wf_create returns WF_ERR_OOM with a message, hands back no context, and frees
what it had allocated (device memory in use returns to where it was), and a
context created afterwards works.  And a bounded wait that runs out."""
import ctypes as C

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


def test_every_refused_allocation_in_create_is_reported_and_cleaned_up(params_from_text):
    import torch
    from wildfires_b200 import Solver, _abi
    torch.cuda.set_device(0)
    L = _abi.lib()
    g = load_golden("hill_rk4")
    P = params_from_text(g["params"])
    for prec in (_abi.WF_FP64, _abi.WF_FP32_STENCIL):
        with Solver(P, "fp64" if prec == _abi.WF_FP64 else "fp32"):
            pass                                      # one-time set-up of the device
        torch.cuda.synchronize()
        free0 = torch.cuda.mem_get_info()[0]
        refused = 0
        for k in range(200):
            L.wf_inject_allocation_failure(k)
            h = C.c_void_p()
            st = L.wf_create(C.byref(P.rec), prec, C.byref(h))
            L.wf_inject_allocation_failure(-1)
            if st == 0:
                L.wf_destroy(h)
                break
            assert st == _abi.WF_ERR_OOM, (k, st)
            assert b"failure injection" in L.wf_last_error()
            assert not h.value
            refused += 1
        assert refused >= 10, refused                 # the context makes that many allocations
        torch.cuda.synchronize()
        assert abs(torch.cuda.mem_get_info()[0] - free0) <= 4 << 20
    with Solver(P, "fp32") as s:
        s.upload(g["y0"], g["p0"])
        s.step(2)
        y, _ = s.download()
    assert np.isfinite(y).all()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_a_plane_given_up_is_reported_by_the_next_call_that_waits(prec, params_from_text, monkeypatch):
    """With a wait limit of 0 (WF_STAGE_WAIT) the stage kernel gives up the first plane of every block: the call that next
    waits for the context reports it, once.  The grid's columns (16 planes) are copied by TMA."""
    from wildfires_b200 import Ensemble, Solver, _abi
    L, dp = _abi.lib(), C.POINTER(C.c_double)
    g = load_golden("flat_33x33x16_10")
    P = params_from_text(g["params"])
    x, y, p = np.array(g["y0"], dtype=np.float64), np.empty(P.state_size), np.empty(33 * 33 * 16)
    xp, yp, pp = (a.ctypes.data_as(dp) for a in (x, y, p))
    diag, rep = _abi.WfDiag(), _abi.WfReport()

    def reported(call):
        assert call() == _abi.WF_ERR_CUDA and b"state plane timed out" in L.wf_last_error()

    monkeypatch.setenv("WF_STAGE_WAIT", "0")
    with Solver(P, prec) as s:
        for wait in (lambda: L.wf_synchronize(s._h), lambda: L.wf_download_state(s._h, yp, pp),
                     lambda: L.wf_diagnostics(s._h, C.byref(diag)), lambda: L.wf_timestep_reports(s._h, C.byref(rep))):
            s.upload(g["y0"], g["p0"])
            s.step(1)
            reported(wait)
            s.synchronize()
        for op in (L.wf_phi, L.wf_rk):
            reported(lambda: op(s._h, xp, yp))
    with Ensemble([P, P], prec) as e:
        for m in e.members:
            m.upload(g["y0"], g["p0"])
        e.step(1)
        reported(lambda: L.wf_ensemble_synchronize(e._h))
        e.synchronize()
    monkeypatch.delenv("WF_STAGE_WAIT")
    with Solver(P, prec) as s:
        s.upload(g["y0"], g["p0"])
        s.step(1)
        s.download()
