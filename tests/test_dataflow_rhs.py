"""The dataflow solve for any number of right-hand sides."""
import numpy as np
import pytest

from pastix_b200 import analysis
from pastix_b200 import matrices as M

RNG = np.random.default_rng
CASES = [
    ("potrf", lambda: M.diffusion_lognormal(20, 17, 19, 1.0, RNG(2)), True),
    ("getrf", lambda: M.convdiff_upwind(20, 17, 19, 10.0), False),
    ("hetrf", lambda: M.magnetic_laplacian(15, 14, 16, 0.5, RNG(3)), True),
    ("hetrf", lambda: M.magnetic_laplacian(15, 14, 16, 0.5, RNG(3)), False),
]


@pytest.mark.gpu
@pytest.mark.parametrize("nrhs", [3, 5, 7, 8, 9, 16, 17])
@pytest.mark.parametrize("fact,make,mixed", CASES, ids=["potrf_s", "getrf_d", "hetrf_c", "hetrf_z"])
def test_dataflow_solve_any_number_of_right_hand_sides(fact, make, mixed, nrhs):
    """Passes of 8 / 4 / 2 right-hand sides, partly filled last ones: every column as the per-level kernels'."""
    from pastix_b200 import autotune as AT
    from pastix_b200 import gpu as G
    A = make()
    s = G.Solver()
    s.set_iparm(G.IPARM_FACTORIZATION, G.FACT[fact])
    s.set_iparm(G.IPARM_MIXED, int(mixed))
    s.set_structure(analysis.analyze(A))
    s.set_spm(A)
    s.numfact(A.values)
    x, b = M.rhs_from_xtrue(A, nrhs, RNG(nrhs))
    b[:, nrhs // 2] *= 1e6      # (a column of another scale: no mixing between columns)
    x[:, nrhs // 2] *= 1e6
    got = s.solve(b)
    launches = s.stats()["solve_launches"]
    AT.set_knob(s, "solve_flow", 0)
    s.numfact(A.values)
    ref = s.solve(b)
    # the runs of levels went through the dataflow: a launch a pass each way instead of four a level
    assert launches < s.stats()["solve_launches"]
    err, base = (np.linalg.norm(v - x, axis=0) / np.linalg.norm(x, axis=0) for v in (got, ref))
    # both are the same factor's solves: rounding of another order of the same sums
    u = 2.0 ** (-24 if mixed else -53)
    assert np.all(err <= 2 * base.max() + 4 * u)
    s.close()
