"""A factorization that is refused while its graph is captured."""
import numpy as np
import pytest

from pastix_b200 import analysis
from pastix_b200 import matrices as M


@pytest.mark.gpu
def test_the_next_handle_is_none_the_wiser():
    """Complex128 LU blocks this wide are not provided: the refusal leaves no error behind for the next call."""
    from pastix_b200 import gpu as G
    rng = np.random.default_rng(1)
    A = M.convdiff_upwind(24, 25, 26, 10.0)
    A.values = A.values * np.exp(0.3j * rng.standard_normal(A.values.size))
    B = M.diffusion_lognormal(10, 10, 10, 1.0, rng)
    st, st2 = analysis.analyze(A), analysis.analyze(B)
    for _ in range(2):
        s = G.Solver()
        s.set_iparm(G.IPARM_FACTORIZATION, G.FACT["getrf"])
        s.set_structure(st)
        s.set_spm(A)
        with pytest.raises(G.PastixGpuError) as e:
            s.numfact(A.values)
        assert e.value.code == 3
        s.close()
        t = G.Solver()
        t.set_iparm(G.IPARM_FACTORIZATION, G.FACT["potrf"])
        t.set_structure(st2)
        t.set_spm(B)
        t.numfact(B.values)
        x, b = M.rhs_from_xtrue(B, 1, rng)
        assert np.linalg.norm(t.solve(b) - x) <= 1e-10 * np.linalg.norm(x)
        t.close()
