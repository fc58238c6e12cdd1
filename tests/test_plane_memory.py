"""Plans when device memory is short."""
import contextlib

import numpy as np
import pytest

from pastix_b200 import analysis
from pastix_b200 import matrices as M

RNG = np.random.default_rng


def _solver(A, st, fact, mixed=1, **knobs):
    from pastix_b200 import autotune as AT
    from pastix_b200 import gpu as G
    s = G.Solver()
    s.set_iparm(G.IPARM_FACTORIZATION, G.FACT[fact])
    s.set_iparm(G.IPARM_MIXED, mixed)
    s.set_structure(st)
    s.set_spm(A)
    for k, v in knobs.items():
        AT.set_knob(s, k, v)
    return s


def _free():
    import torch
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _takes(A, st, fact, **knobs):
    """Device memory a first factorization and solve take (the second of two handles: kernels are loaded)."""
    x, b = M.rhs_from_xtrue(A, 1, RNG(1))
    for _ in range(2):
        s = _solver(A, st, fact, **knobs)
        f0 = _free()
        s.numfact(A.values)
        s.solve(b)
        used = f0 - _free()
        s.close()
    return used


@contextlib.contextmanager
def _only(room):
    """All of the device's memory but `room` bytes taken."""
    import torch
    hog = torch.empty(_free() - room, dtype=torch.uint8, device="cuda")
    yield
    del hog
    _free()


def _check(s, A):
    x, b = M.rhs_from_xtrue(A, 1, RNG(1))
    assert np.linalg.norm(s.solve(b) - x) <= 1e-4 * np.linalg.norm(x)
    return s.stats()["tc_flops"]


@pytest.mark.gpu
def test_a_failed_allocation_is_made_good():
    """A factorization without room is refused, and the next one, with room, allocates what it lacks."""
    from pastix_b200 import gpu as G
    A = M.diffusion_lognormal(30, 29, 31, 1.0, RNG(2))
    st = analysis.analyze(A)
    _takes(A, st, "potrf")                                   # (kernels loaded)
    s = _solver(A, st, "potrf", mixed=0)
    with _only(16 * 2 ** 20):
        with pytest.raises(G.PastixGpuError) as e:
            s.numfact(A.values)
        assert e.value.code == 4
    s.numfact(A.values)
    _check(s, A)
    s.close()


@pytest.mark.gpu
def test_a_plan_that_fails_leaves_no_factor():
    """Its solve lists and inverses belong half to the plan that was not finished."""
    from pastix_b200 import gpu as G
    A = M.diffusion_lognormal(30, 29, 31, 1.0, RNG(2))
    st = analysis.analyze(A)
    room = _takes(A, st, "potrf") // 4
    s = _solver(A, st, "potrf")
    s.numfact(A.values)
    s.set_iparm(G.IPARM_MIXED, 0)
    with _only(room):
        with pytest.raises(G.PastixGpuError):
            s.numfact(A.values)
        with pytest.raises(G.PastixGpuError):
            s.solve(np.ones(A.n))
    s.set_iparm(G.IPARM_MIXED, 1)
    s.numfact(A.values)
    assert _check(s, A) > 0
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("fact,make", [
    ("sytrf", lambda: M.diffusion_lognormal(40, 39, 41, 1.0, RNG(2))),
    ("hetrf", lambda: M.magnetic_laplacian(30, 29, 31, 0.5, RNG(3))),
], ids=["sytrf", "hetrf"])
def test_no_room_for_the_planes_lasts_one_plan(fact, make):
    """LDL and complex planes that do not fit send their updates to the FMA tiles; the next plan, with room
    again, has them on the tensor cores."""
    from pastix_b200 import autotune as AT
    A = make()
    st = analysis.analyze(A)
    room = (_takes(A, st, fact) + _takes(A, st, fact, mixed_gemm=0)) // 2
    s = _solver(A, st, fact)
    with _only(room):
        s.numfact(A.values)
        assert _check(s, A) == 0
        s.numfact(A.values)
    AT.set_knob(s, "tc_min_mn", 8192)      # (the default: any knob asks for a new plan)
    s.numfact(A.values)
    assert _check(s, A) > 0
    s.close()


def _copies(nb, w, m, rng):
    """nb independent Hermitian systems, each a cblk of w columns with m rows that face a second cblk."""
    k = w + m
    v = np.tril(rng.uniform(-1, 1, (nb, k, k)) + 1j * rng.uniform(-1, 1, (nb, k, k)), -1)
    v[:, np.arange(k), np.arange(k)] = 2.0 * k
    o = np.arange(nb) * k
    cblk = [r for i, f in enumerate(o) for r in ([f, f + w - 1, 3 * i, 0], [f + w, f + k - 1, 3 * i + 2, 0])]
    blok = [r for i, f in enumerate(o) for r in ([f, f + w - 1, 2 * i, 2 * i], [f + w, f + k - 1, 2 * i, 2 * i + 1],
                                                 [f + w, f + k - 1, 2 * i + 1, 2 * i + 1])]
    n = nb * k
    st = dict(n=n, cblktab=np.array(cblk + [[n, n, 3 * nb, 0]], np.int64), bloktab=np.array(blok, np.int64),
              browtab=np.zeros(nb, np.int64), permtab=np.arange(n), peritab=np.arange(n))
    r, c = np.tril_indices(k)
    order = np.lexsort((r, c))
    r, c = r[order], c[order]
    colptr = np.concatenate([[0], np.cumsum(np.tile(k - np.arange(k), nb))]).astype(np.int64)
    A = M.SparseSystem(n, colptr, (o[:, None] + r[None, :]).ravel().astype(np.int64), v[:, r, c].ravel(),
                       M.PastixHermitian, (n, 1, 1))
    return A, st


@pytest.mark.gpu
def test_complex_ldl_keeps_no_plane_of_bare_rows():
    """Its updates read the rows times D and the B rows (two per row); the bare rows are an operand of the tall
    panels' TRSM only, and these panels are short: three planes of rows, not four."""
    nb, w, m = 64, 100, 150
    A, st = _copies(nb, w, m, RNG(5))
    plane = nb * (w + m) * ((2 * w + 63) // 64 * 64) * 4      # hi and lo halves of every row
    more = _takes(A, st, "hetrf") - _takes(A, st, "hetrf", mixed_gemm=0)
    assert 2.5 * plane < more < 3.5 * plane


@pytest.mark.gpu
@pytest.mark.parametrize("fact,make", [
    ("potrf", lambda: M.diffusion_lognormal(50, 49, 51, 1.0, RNG(2))),
    ("getrf", lambda: M.convdiff_upwind(50, 49, 51, 10.0)),
], ids=["potrf", "getrf"])
def test_planes_are_packed_where_whole_lines_do_not_fit(fact, make):
    """What fitted with rows padded to 8 halves still does."""
    A = make()
    st = analysis.analyze(A)
    w = st["cblktab"][:-1, 1] - st["cblktab"][:-1, 0] + 1
    rows = np.concatenate([[0], np.cumsum(st["bloktab"][:, 1] - st["bloktab"][:, 0] + 1)])
    h = rows[st["cblktab"][1:, 2]] - rows[st["cblktab"][:-1, 2]]
    src = (w >= 64) & (h >= w + 128)                         # (a lower bound: sources of tensor-core updates)
    pad = 4 * int((h * ((w + 63) // 64 * 64 - (w + 7) // 8 * 8))[src].sum()) * (2 if fact == "getrf" else 1)
    assert pad > 24 * 2 ** 20
    s = _solver(A, st, fact)
    with _only(_takes(A, st, fact) - pad // 2):
        s.numfact(A.values)
        assert _check(s, A) > 0
    s.close()
