"""Tensor-core updates of the LDL and complex forms,
against the numpy restatement."""
import numpy as np
import pytest

from oracle.restate import sopalin_np as NP
from pastix_b200 import analysis
from pastix_b200 import matrices as M


def _phased(A, seed):
    """Complex general matrix with A's pattern and magnitudes."""
    A.values = A.values * np.exp(0.3j * np.random.default_rng(seed).standard_normal(A.values.size))
    return A


def _csym(A, seed):
    """Complex symmetric matrix, diagonally dominant as A is."""
    A.values = A.values * (1 + 0.05j * np.random.default_rng(seed).standard_normal(A.values.size))
    return A


RNG = np.random.default_rng
CASES = [
    ("potrf", lambda: M.diffusion_lognormal(20, 17, 19, 1.0, RNG(2))),
    ("sytrf", lambda: M.diffusion_lognormal(20, 17, 19, 1.0, RNG(2))),
    ("getrf", lambda: M.convdiff_upwind(20, 17, 19, 10.0)),
    ("potrf", lambda: M.magnetic_laplacian(15, 14, 16, -0.5, RNG(3))),
    ("hetrf", lambda: M.magnetic_laplacian(15, 14, 16, 0.5, RNG(3))),
    ("sytrf", lambda: _csym(M.diffusion_lognormal(15, 14, 16, 1.0, RNG(4)), 5)),
    ("getrf", lambda: _phased(M.convdiff_upwind(15, 14, 16, 10.0), 6)),
    ("sytrf", lambda: M.diffusion_lognormal(63, 50, 1, 0.5, RNG(7))),
]
IDS = ["potrf", "sytrf", "getrf", "potrf_z", "hetrf_z", "sytrf_z", "getrf_z", "sytrf_2d"]


def _error(A, st, fact, L, U):
    lay = NP.Layout(st["cblktab"], st["bloktab"])
    L0, U0 = NP.fillin(lay, A, st["permtab"], lu=fact == "getrf")
    NP.factorize(lay, L0, U0, fact, 0.0)
    mask = np.ones(lay.off[-1], bool)
    if fact != "getrf":
        for c in range(lay.cblknbr):
            k = int(lay.width[c])
            lay.panel(mask, c)[:k, :] &= np.tril(np.ones((k, k), bool))
    err = np.linalg.norm((L - L0)[mask]) / np.linalg.norm(L0[mask])
    if fact == "getrf":
        for c in range(lay.cblknbr):
            lay.panel(mask, c)[:int(lay.width[c]), :] = False
        err = max(err, np.linalg.norm((U - U0)[mask]) / np.linalg.norm(U0[mask]))
    return err


@pytest.mark.gpu
@pytest.mark.parametrize("mixed", [True, False], ids=["mixed", "fp64"])
@pytest.mark.parametrize("fact,make", CASES, ids=IDS)
def test_tensor_core_forms_match_restatement(fact, make, mixed):
    """Factors as close to the 64-bit restatement as the FMA tiles' (the tensor-core sums round less
    often), and the tensor cores carry the updates."""
    from pastix_b200 import autotune as AT
    from pastix_b200 import gpu as G
    A = make()
    st = analysis.analyze(A)
    errs = []
    for tc in (True, False):
        s = G.Solver()
        s.set_iparm(G.IPARM_FACTORIZATION, G.FACT[fact])
        s.set_iparm(G.IPARM_MIXED, int(mixed))
        s.set_structure(st)
        s.set_spm(A)
        if not tc:
            AT.set_knob(s, "mixed_gemm", 0)
            AT.set_knob(s, "dmma", 0)
        try:
            s.numfact(A.values)
        except G.PastixGpuError as e:
            s.close()
            if e.code == 3:
                pytest.skip("complex128 LU blocks this wide are not provided")
            raise
        stats = s.stats()
        if tc and A.grid[2] > 1:
            assert stats["tc_flops"] > 0.3 * stats["gemm_flops"] and stats["tc_timeouts"] == 0
        L, U = s.coeftab()
        errs.append(_error(A, st, fact, L, U))
        s.close()
    # unit roundoff times a few: diagonally dominant or of bounded growth; no worse than the FMA tiles
    # beyond the spread between two summation orders
    u = 2.0 ** (-24 if mixed else -53)
    assert errs[0] <= 32 * u
    assert errs[0] <= 1.5 * errs[1] + u / 4


@pytest.mark.gpu
@pytest.mark.parametrize("fact,make,mode", [
    ("potrf", lambda: M.diffusion_lognormal(40, 37, 39, 1.0, RNG(8)), 3),
    ("sytrf", lambda: M.diffusion_lognormal(40, 37, 39, 1.0, RNG(8)), 3),
    ("getrf", lambda: M.convdiff_upwind(36, 35, 37, 10.0), 3),
    ("hetrf", lambda: M.magnetic_laplacian(33, 34, 32, 0.5, RNG(9)), 3),
    ("potrf", lambda: M.diffusion_lognormal(40, 37, 39, 1.0, RNG(8)), 2),
    ("getrf", lambda: M.convdiff_upwind(36, 35, 37, 10.0), 2),
], ids=["potrf", "sytrf", "getrf", "hetrf", "potrf_3xtf32", "getrf_3xtf32"])
def test_fan_in_over_separator_chains(fact, make, mode):
    """Separators wide enough for chains of several cblks, whose deferred updates are summed before they
    are scattered, in single tiles and in pairs (mode 3: 3xFP16, 2: 3xTF32, without row scales): the factor
    agrees with the FMA tiles', which scatter every source on its own."""
    from pastix_b200 import autotune as AT
    from pastix_b200 import gpu as G
    A = make()
    st = analysis.analyze(A)
    s = G.Solver()
    s.set_iparm(G.IPARM_FACTORIZATION, G.FACT[fact])
    s.set_iparm(G.IPARM_MIXED, 1)
    s.set_structure(st)
    s.set_spm(A)
    AT.set_knob(s, "mixed_gemm", mode)
    AT.set_knob(s, "tc_pair_min", 0)
    s.numfact(A.values)
    assert s.stats()["tc_flops"] > 0.8 * s.stats()["gemm_flops"]
    tiles, several, pairs = s.plan_counts()
    assert tiles > several > pairs > 0
    L, U = s.coeftab()
    AT.set_knob(s, "mixed_gemm", 0)
    s.numfact(A.values)
    L0, U0 = s.coeftab()
    s.close()
    lay = NP.Layout(st["cblktab"], st["bloktab"])
    mask = np.ones(lay.off[-1], bool)
    if fact != "getrf":
        for c in range(lay.cblknbr):
            k = int(lay.width[c])
            lay.panel(mask, c)[:k, :] &= np.tril(np.ones((k, k), bool))
    # two single-precision factors of bounded growth, each within a few tens of roundoffs of the exact one
    for P, Q, m in ((L, L0, mask), (U, U0, None)) if U is not None else ((L, L0, mask),):
        d, q = (P - Q, Q) if m is None else ((P - Q)[m], Q[m])
        assert np.linalg.norm(d) <= 64 * 2.0 ** -24 * np.linalg.norm(q)


# --- sums of the LDL and complex forms -----------------------------------------
def _lower(st):
    lay = NP.Layout(st["cblktab"], st["bloktab"])
    mask = np.ones(lay.off[-1], bool)
    for c in range(lay.cblknbr):
        k = int(lay.width[c])
        lay.panel(mask, c)[:k, :] &= np.tril(np.ones((k, k), bool))
    return mask


def _mixed_factors(A, st, fact):
    """Single-precision factor on the tensor cores and on the FMA tiles."""
    from pastix_b200 import autotune as AT
    from pastix_b200 import gpu as G
    s = G.Solver()
    s.set_iparm(G.IPARM_FACTORIZATION, G.FACT[fact])
    s.set_iparm(G.IPARM_MIXED, 1)
    s.set_structure(st)
    s.set_spm(A)
    s.numfact(A.values)
    stats = s.stats()
    assert stats["tc_flops"] > 0.7 * stats["gemm_flops"]
    out = [s.coeftab()]
    AT.set_knob(s, "mixed_gemm", 0)
    s.numfact(A.values)
    out.append(s.coeftab())
    s.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("fact,make,spread", [
    ("sytrf", lambda: M.diffusion_lognormal(44, 43, 45, 1.0, RNG(8)), 1.08),
    ("sytrf", lambda: _csym(M.diffusion_lognormal(30, 29, 31, 1.0, RNG(4)), 5), 1.04),
], ids=["sytrf", "sytrf_z"])
def test_ldl_sums_are_as_close_as_the_fma_tiles(fact, make, spread):
    """Terms of one sign, over sources of up to some 200 columns: the tensor core's additions cut off, the FMA
    tiles' round to nearest, everything else is the same.  Errors against the 64-bit factor.  `spread`: the real
    form keeps its operands' 22 bits and the twelve cut-off additions of 64 columns, of 6 units 2^-25 of a sum
    beside the FMA chain's 4 to 5 (sums cut off over the whole depth: 1.18 of the FMA tiles' error, complex 1.06)."""
    from pastix_b200 import gpu as G
    A = make()
    st = analysis.analyze(A)
    s = G.Solver()
    s.set_iparm(G.IPARM_FACTORIZATION, G.FACT[fact])
    s.set_structure(st)
    s.set_spm(A)
    s.numfact(A.values)
    L0, _ = s.coeftab()
    s.close()
    m = _lower(st)
    e_tc, e_fma = (np.linalg.norm((L - L0)[m]) for L, _ in _mixed_factors(A, st, fact))
    assert e_tc <= spread * e_fma


def _times(A, f):
    A.values = A.values * f
    return A


@pytest.mark.gpu
@pytest.mark.parametrize("fact,make", [
    ("sytrf", lambda: _times(M.diffusion_lognormal(20, 17, 19, 0.3, RNG(2)), 1e36)),
    ("hetrf", lambda: _times(M.magnetic_laplacian(20, 19, 18, -0.5, RNG(3)), 1e35)),
    ("getrf", lambda: _times(_phased(M.convdiff_upwind(15, 14, 16, 10.0), 6), 1e35)),
    ("sytrf", lambda: _times(M.diffusion_lognormal(20, 17, 19, 0.3, RNG(2)), 1e-30)),
], ids=["sytrf_1e36", "hetrf_1e35", "getrf_z_1e35", "sytrf_1e-30"])
def test_matrices_of_extreme_scale(fact, make):
    """Rows near the largest float: an accumulator times one of its two scales leaves the range, the result
    does not.  The FMA tiles take these matrices, so the tensor cores have to."""
    A = make()
    st = analysis.analyze(A)
    (L, U), (L0, U0) = _mixed_factors(A, st, fact)
    m = _lower(st) if fact != "getrf" else np.ones(L.size, bool)
    for P, Q, k in ((L, L0, m),) + (((U, U0, m),) if U is not None else ()):
        q = Q[k].astype(np.complex128)
        d = P[k].astype(np.complex128) - q
        t = np.abs(q).max()
        # (as between the two in test_fan_in_over_separator_chains)
        assert np.linalg.norm(d / t) <= 64 * 2.0 ** -24 * np.linalg.norm(q / t)
