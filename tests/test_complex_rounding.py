"""Complex multiply-adds of the panel kernels round each part once."""
import numpy as np
import pytest

from pastix_b200 import matrices as M


def _blocks(nb, w, rng):
    """nb independent dense Hermitian blocks, values representable in single precision: a diagonal in
    (1.5, 1.9) that 31 updates of about 2^-10 each leave within (1, 2)."""
    v = (rng.uniform(-1, 1, (nb, w, w)) + 1j * rng.uniform(-1, 1, (nb, w, w))) * 2.0 ** -5
    v = np.tril(v, -1)
    v = v + v.conj().transpose(0, 2, 1)
    v[:, np.arange(w), np.arange(w)] = rng.uniform(1.5, 1.9, (nb, w))
    return v.astype(np.complex64).astype(np.complex128)


def _pivots(v, k):
    """d_k of the LDL^h factors."""
    a = v.copy()
    for j in range(k):
        l = a[:, j + 1:, j] / a[:, j, j].real[:, None]
        a[:, j + 1:, j + 1:] -= l[:, :, None] * a[:, None, j + 1:, j].conj()
    return a[:, k, k].real


@pytest.mark.gpu
@pytest.mark.parametrize("w", [32, 64])
def test_elimination_rounds_each_part_once(w):
    """The 31 updates of pivot 31 are added to a value of (1, 2): one rounding each is sqrt(31 / 12) units in
    the last place in the mean square, two are sqrt(2) times that; the line lies at the mean of the squares."""
    from pastix_b200 import gpu as G
    nb, rng = 256, np.random.default_rng(5)
    v = _blocks(nb, w, rng)
    n = nb * w
    first = np.arange(nb) * w
    cblk = np.array([[f, f + w - 1, i, 0] for i, f in enumerate(first)] + [[n, n, nb, 0]], np.int64)
    blok = np.array([[f, f + w - 1, i, i] for i, f in enumerate(first)], np.int64)
    st = dict(n=n, cblktab=cblk, bloktab=blok, browtab=np.zeros(0, np.int64), permtab=np.arange(n), peritab=np.arange(n))
    r, c = np.tril_indices(w)
    order = np.lexsort((r, c))
    r, c = r[order], c[order]
    colptr = np.concatenate([[0], np.cumsum(np.tile(w - np.arange(w), nb))]).astype(np.int64)
    rows = (first[:, None] + r[None, :]).ravel().astype(np.int64)
    A = M.SparseSystem(n, colptr, rows, v[:, r, c].ravel(), M.PastixHermitian, (n, 1, 1))
    s = G.Solver()
    s.set_iparm(G.IPARM_FACTORIZATION, G.FACT["hetrf"])
    s.set_iparm(G.IPARM_MIXED, 1)
    s.set_structure(st)
    s.set_spm(A)
    s.numfact(A.values)
    L, _ = s.coeftab()
    s.close()
    d = L.reshape(nb, w, w)[:, 31, 31].real
    assert np.all((d > 1) & (d < 2))
    rms = np.sqrt(np.mean((d - _pivots(v, 31)) ** 2)) * 2.0 ** 23
    assert rms <= np.sqrt(1.5 * 31 / 12)
