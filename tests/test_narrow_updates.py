"""Narrow updates (facing blocks of at most 32 rows, one warp per 32-row slab)
and the panels of at most 32 columns they come from, at every offset of the
block in the facing cblk, against the numpy restatement."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle.restate import sopalin_np as NP
from pastix_b200 import matrices as M

W1, W2 = 41, 35     # the facing cblks


def _case(fact, cplx, w, off, n, rng):
    """Cblk 0 (w columns) faces cblk 1 with n rows from its column `off` and cblk 2 with 9; 1 faces all of 2."""
    N = w + W1 + W2
    r1, r2 = w + off, w + W1 + 3
    cblk = np.array([[0, w - 1, 0, 0], [w, w + W1 - 1, 3, 1], [w + W1, N - 1, 5, 2], [N, N, 6, 4]], np.int64)
    blok = np.array([[0, w - 1, 0, 0], [r1, r1 + n - 1, 0, 1], [r2, r2 + 8, 0, 2], [w, w + W1 - 1, 1, 1],
                     [w + W1, N - 1, 1, 2], [w + W1, N - 1, 2, 2]], np.int64)
    st = dict(n=N, cblktab=cblk, bloktab=blok, browtab=np.array([1, 2, 4], np.int64), permtab=np.arange(N),
              peritab=np.arange(N))
    v = rng.uniform(-1, 1, (N, N)) + (1j * rng.uniform(-1, 1, (N, N)) if cplx else 0)
    mask = np.ones((N, N), bool)
    below = np.zeros(N, bool)
    below[:w] = below[r1:r1 + n] = below[r2:r2 + 9] = True
    mask[~below, :w] = False
    mask[:w, ~below] = False
    v = v * mask
    if fact != "getrf":
        v = np.tril(v, -1)
        v = v + (v.T if fact == "sytrf" else v.conj().T)
    v[np.arange(N), np.arange(N)] = 2.0 * N
    A = sp.csc_matrix(v if fact == "getrf" else np.tril(v))
    mtx = M.PastixGeneral if fact == "getrf" else M.PastixSymmetric if fact == "sytrf" or not cplx else M.PastixHermitian
    return st, M.SparseSystem(N, A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data, mtx, (N, 1, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("fact,cplx", [("potrf", False), ("sytrf", False), ("getrf", False), ("hetrf", True)])
@pytest.mark.parametrize("w,off,n", [(1, 0, 1), (7, 1, 4), (12, 2, 5), (31, 3, 29), (32, 9, 32), (33, 6, 31), (70, 5, 8)])
def test_narrow_updates_match_restatement(fact, cplx, w, off, n, mixed):
    from pastix_b200 import gpu as G
    st, A = _case(fact, cplx, w, off, n, np.random.default_rng(w + 100 * off + n))
    s = G.Solver()
    s.set_iparm(G.IPARM_FACTORIZATION, G.FACT[fact])
    s.set_iparm(G.IPARM_MIXED, int(mixed))
    s.set_structure(st)
    s.set_spm(A)
    s.numfact(A.values)
    L, U = s.coeftab()
    s.close()
    lay = NP.Layout(st["cblktab"], st["bloktab"])
    L0, U0 = NP.fillin(lay, A, st["permtab"], lu=fact == "getrf")
    NP.factorize(lay, L0, U0, fact, 0.0)
    mask = np.ones(lay.off[-1], bool)
    for c in range(lay.cblknbr):
        k = int(lay.width[c])
        lay.panel(mask, c)[:k, :] &= np.tril(np.ones((k, k), bool)) if fact != "getrf" else True
    # diagonally dominant: within n u of the exact factor
    tol = st["n"] * 2.0 ** (-24 if mixed else -53) * (4 if cplx else 2)
    assert np.abs(L - L0)[mask].max() <= tol * np.abs(L0).max()
    if fact == "getrf":
        for c in range(lay.cblknbr):
            lay.panel(mask, c)[:int(lay.width[c]), :] = False
        assert np.abs(U - U0)[mask].max() <= tol * np.abs(U0).max()
