"""Block-row factorization of the diagonal blocks (k_panel_rows) and of their
inverses, on two-cblk matrices whose widths sit at the edges of its 32-row
tiles, against the numpy restatement."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle.restate import sopalin_np as NP
from pastix_b200 import matrices as M

# first cblk's width, rows below it: the one-warp panels (at most 32 columns), one and two tiles, ragged last tiles, a panel solved in the
# kernel (height at most 256) and one that goes through the inverse, the widest block accepted
SHAPES = [(1, 5), (7, 40), (31, 33), (32, 64), (33, 1), (64, 40), (65, 31), (96, 33), (127, 200), (160, 129),
          (320, 64), (400, 7)]
FORMS = [("potrf", False), ("sytrf", False), ("getrf", False), ("potrf", True), ("hetrf", True), ("sytrf", True),
         ("getrf", True)]


def _matrix(fact, cplx, n, rng, neg=None):
    """Dense, diagonally dominant; general for LU, Hermitian (or complex symmetric) otherwise."""
    v = rng.uniform(-1, 1, (n, n)) + (1j * rng.uniform(-1, 1, (n, n)) if cplx else 0)
    if fact != "getrf":
        v = np.tril(v, -1)
        v = v + (v.T if fact == "sytrf" else v.conj().T)
    sign = -1.0 if fact in ("sytrf", "hetrf") else 1.0
    d = 2.0 * n * np.where(np.arange(n) % 3 == 1, sign, 1.0)
    if neg is not None:
        d[neg] = -d[neg]
    v[np.arange(n), np.arange(n)] = d
    low = v if fact == "getrf" else np.tril(v)
    A = sp.csc_matrix(low)
    mtx = M.PastixGeneral if fact == "getrf" else M.PastixSymmetric if fact == "sytrf" or not cplx else M.PastixHermitian
    return M.SparseSystem(n, A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data, mtx, (n, 1, 1))


def _structure(w, m):
    """A cblk of w columns with one block of m rows facing a second cblk."""
    n = w + m
    cblk = np.array([[0, w - 1, 0, 0], [w, n - 1, 2, 1], [n, n, 3, 2]], np.int64)
    blok = np.array([[0, w - 1, 0, 0], [w, n - 1, 0, 1], [w, n - 1, 1, 1]], np.int64)
    return dict(n=n, cblktab=cblk, bloktab=blok, browtab=np.array([1, 0], np.int64), permtab=np.arange(n),
                peritab=np.arange(n))


def _solver(A, st, fact, mixed):
    from pastix_b200 import gpu as G
    s = G.Solver()
    s.set_iparm(G.IPARM_FACTORIZATION, G.FACT[fact])
    s.set_iparm(G.IPARM_MIXED, int(mixed))
    s.set_structure(st)
    s.set_spm(A)
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("fact,cplx", FORMS)
@pytest.mark.parametrize("w,m", SHAPES)
def test_block_rows_match_restatement(fact, cplx, w, m, mixed):
    from pastix_b200 import gpu as G
    if fact == "getrf" and cplx and not mixed and w > 200:
        pytest.skip("complex128 LU blocks this wide are not provided (shared memory of the panel kernel)")
    rng = np.random.default_rng(100 * w + m)
    st = _structure(w, m)
    A = _matrix(fact, cplx, w + m, rng)
    s = _solver(A, st, fact, mixed)
    s.numfact(A.values)
    L, U = s.coeftab()
    lay = NP.Layout(st["cblktab"], st["bloktab"])
    L0, U0 = NP.fillin(lay, A, st["permtab"], lu=fact == "getrf")
    NP.factorize(lay, L0, U0, fact, 0.0)
    mask = np.ones(lay.off[-1], bool)
    if fact != "getrf":
        for c in range(lay.cblknbr):
            k = int(lay.width[c])
            lay.panel(mask, c)[:k, :] &= np.tril(np.ones((k, k), bool))
    # diagonally dominant: no growth, so the factor is within n u of the exact one (and of the restatement's)
    tol = (w + m) * 2.0 ** (-24 if mixed else -53) * (4 if cplx else 2)
    assert np.abs(L - L0)[mask].max() <= tol * np.abs(L0).max()
    if fact == "getrf":
        off = mask.copy()
        for c in range(lay.cblknbr):
            lay.panel(off, c)[:int(lay.width[c]), :] = False    # (U's diagonal block lives in L)
        assert np.abs(U - U0)[off].max() <= tol * np.abs(U0).max()
    # the solve reads the inverse where the panel is tall
    x, b = M.rhs_from_xtrue(A, 3, rng)
    assert np.abs(s.solve(b) - x).max() <= 8 * tol
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("w,col", [(20, 0), (20, 19), (96, 0), (96, 37), (96, 95)])
def test_negative_pivot_is_refused(w, col):
    """A negative pivot makes the Cholesky factor non-finite, as its square root would: the numfact fails."""
    from pastix_b200 import gpu as G
    st = _structure(w, 30)
    A = _matrix("potrf", False, w + 30, np.random.default_rng(3), neg=col)
    s = _solver(A, st, "potrf", False)
    with pytest.raises(G.PastixGpuError):
        s.numfact(A.values)
    s.close()


def _growing(fact, w, m, g, rng):
    """A = L L^t (LU: L U) whose first 32-column diagonal tile, -g below its diagonal, has an inverse of
    some (1 + g)^31."""
    n = w + m

    def lower():
        v = np.tril(rng.uniform(-1, 1, (n, n)) / 32, -1)
        v[:32, :32] = np.tril(-g * np.ones((32, 32)), -1)
        v[:, w:] = 0
        v[np.arange(n), np.arange(n)] = 1
        return v
    L = lower()
    R = lower().T if fact == "getrf" else L.T
    v = L @ R
    v[np.arange(w, n), np.arange(w, n)] += 2.0 * n
    A = sp.csc_matrix(v if fact == "getrf" else np.tril(v))
    mtx = M.PastixGeneral if fact == "getrf" else M.PastixSymmetric
    return v, M.SparseSystem(n, A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data, mtx, (n, 1, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("fact,mixed,w,m", [
    (f, x, w, m) for f in ("potrf", "sytrf", "getrf") for x in (False, True)
    for w, m in ([(50, 40), (64, 30)] if f == "getrf" and not x else [(64, 40), (96, 100), (130, 70)])])
def test_block_rows_solve_as_a_substitution_does(fact, mixed, w, m):
    """The rows X of the panel leave the residual of a substitution, |A - X U| <= k u |X| |U| (k terms a sum, and
    a few for the tile's factor), also where the tile's inverse is large: a product with the inverse alone leaves
    one larger by up to its condition (in single
    precision a smaller one, the matrix has to stay definite).  Panels that the kernel solves itself: at most 256
    rows, FP64 LU 96."""
    v, A = _growing(fact, w, m, 0.2 if mixed else 0.4, np.random.default_rng(w))
    v = v.astype(np.float32) if mixed else v
    st = _structure(w, m)
    s = _solver(A, st, fact, mixed)
    s.numfact(A.values)
    L, U = s.coeftab()
    s.close()
    lay = NP.Layout(st["cblktab"], st["bloktab"])
    P = lay.panel(L, 0).astype(np.float64)
    D, X = P[:w], P[w:]
    if fact == "getrf":
        sides = [(v[w:, :w], X, np.triu(D)), (v[:w, w:].T, lay.panel(U, 0).astype(np.float64)[w:],
                                              (np.tril(D, -1) + np.eye(w)).T)]
    elif fact == "sytrf":
        sides = [(v[w:, :w], X, np.diag(np.diag(D)) @ (np.tril(D, -1) + np.eye(w)).T)]
    else:
        sides = [(v[w:, :w], X, np.tril(D).T)]
    u = 2.0 ** (-24 if mixed else -53)
    for B, X, T in sides:
        assert np.abs(B - X @ T).max() <= 4 * w * u * (np.abs(X) @ np.abs(T)).max()
