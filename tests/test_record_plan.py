"""Switching the task records on or off between two factorizations."""
import numpy as np
import pytest

from pastix_b200 import analysis
from pastix_b200 import matrices as M


@pytest.mark.gpu
@pytest.mark.parametrize("fact,mixed", [("potrf", 1), ("getrf", 1), ("potrf", 0)])
def test_recording_gets_a_plan_of_its_own(fact, mixed):
    """The recorded factorization runs kernels of one tile per CTA, which read no fan-in segments and no tile
    pairs: with the panel TRSM by rows both plans otherwise look alike."""
    from pastix_b200 import autotune as AT
    from pastix_b200 import costmodel as CM
    from pastix_b200 import gpu as G
    rng = np.random.default_rng(2)
    A = M.convdiff_upwind(30, 29, 31, 10.0) if fact == "getrf" else M.diffusion_lognormal(30, 29, 31, 1.0, rng)
    s = G.Solver()
    s.set_iparm(G.IPARM_FACTORIZATION, G.FACT[fact])
    s.set_iparm(G.IPARM_MIXED, mixed)
    s.set_structure(analysis.analyze(A))
    s.set_spm(A)
    AT.set_knob(s, "trsm_gemm", 0)
    x, b = M.rhs_from_xtrue(A, 1, rng)
    err = []
    for on in (False, True, False):
        CM.record_tasks(s, on)
        if on:
            with pytest.raises(G.PastixGpuError):     # (the factor at hand was not recorded)
                CM.task_records(s)
        s.numfact(A.values)
        if on:
            info, ns = CM.task_records(s)
            assert ns.min() >= 0 and 0 < ns.max() < 1e9
        err.append(np.linalg.norm(s.solve(b) - x) / np.linalg.norm(x))
    s.close()
    assert max(err) <= 4 * min(err)     # (three orders of summation of one factor)


@pytest.mark.gpu
def test_recorded_panels_are_those_that_run():
    """The widest block runs one CTA per block row, recorded or not: far faster than on one CTA."""
    from pastix_b200 import autotune as AT
    from pastix_b200 import costmodel as CM
    from pastix_b200 import gpu as G
    rng = np.random.default_rng(2)
    A = M.diffusion_lognormal(30, 29, 31, 1.0, rng)
    s = G.Solver()
    s.set_iparm(G.IPARM_FACTORIZATION, G.FACT["potrf"])
    s.set_structure(analysis.analyze(A))
    s.set_spm(A)
    x, b = M.rhs_from_xtrue(A, 1, rng)
    CM.record_tasks(s)
    widest = []
    for wide in (128, 0):
        AT.set_knob(s, "wide_panel", wide)
        for _ in range(3):
            s.numfact(A.values)
        info, ns = CM.task_records(s)
        panel = info[:, 0] == 0
        assert ns[panel].min() >= 0 and ns[panel].max() < 1e8
        widest.append(ns[panel][np.argmax(info[panel, 2])])
        assert np.linalg.norm(s.solve(b) - x) <= 1e-10 * np.linalg.norm(x)
    s.close()
    assert 0 < widest[0] < 0.7 * widest[1]
