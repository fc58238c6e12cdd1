"""The calls a user of the solver makes, at the sizes they make them.

A case is one pass of a program that holds a `Solver` whose analysis and plan
are done (a new matrix on a known pattern in every time step, Newton step or
parameter sample, or new right-hand sides on kept factors):

  op "step"    numfact(values), then solve and refine to a 1e-13 residual
  op "direct"  numfact(values), then the plain solve, no refinement
  op "solve"   factors kept: the plain solve of FP64 factors, solve and
               refinement on single-precision ("mixed") ones

`fact` / `kind` name the factorization and the matrix: LL^t and LDL^t on
variable-coefficient diffusion, LU on upwind convection-diffusion, LDL^h on
the (complex, indefinite) magnetic Laplacian, on nx x ny x nz grids (nz 1: 2D);
`batch` > 0 is that many independent 2D systems of uneven side, as one forest.
Values and right-hand sides are drawn from the seed; b = A x_true.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from pastix_b200 import analysis, batch
from pastix_b200 import gpu as G
from pastix_b200 import matrices as M

REFINE_EPS = 1e-13


def _case(name, kind, fact, nx, ny, nz, mixed, op, nrhs, host=False, nsys=0):
    c = dict(kind=kind, fact=fact, nx=nx, ny=ny, nz=nz, mixed=mixed, op=op, nrhs=nrhs, host=host, batch=nsys)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest 3D problem a user has it do, through host arrays as the CPU library is called
        _case("lap20_step_host", "laplacian", "potrf", 20, 20, 20, False, "step", 1, host=True),
        # the smallest call of all: one right-hand side on kept factors
        _case("lap20_solve", "laplacian", "potrf", 20, 20, 20, False, "solve", 1),
        # a 2D problem of ordinary size and odd sides, one right-hand side
        _case("diff2d_step", "diffusion", "potrf", 501, 389, 1, True, "step", 1),
        # the headline problem: a million unknowns, single-precision factor and CG
        _case("diff100_step", "diffusion", "potrf", 100, 100, 100, True, "step", 1),
        # the same problem for a user who wants FP64 factors
        _case("diff100_direct_f64", "diffusion", "potrf", 100, 100, 100, False, "direct", 1),
        # many right-hand sides on kept factors
        _case("diff100_solve16", "diffusion", "potrf", 100, 100, 100, True, "solve", 16),
        # nonsymmetric: LU and GMRES, four right-hand sides
        _case("conv80_step", "convdiff", "getrf", 80, 80, 80, True, "step", 4),
        # nonsymmetric in FP64, odd sides and an odd number of right-hand sides
        _case("conv_odd_direct_f64", "convdiff", "getrf", 37, 45, 51, False, "direct", 3),
        # symmetric indefinite form, single precision without refinement, odd sides
        _case("ldlt_odd_direct", "diffusion", "sytrf", 53, 49, 61, True, "direct", 2),
        # complex Hermitian indefinite: complex64 factor and GMRES
        _case("mag60_step", "magnetic", "hetrf", 60, 60, 60, True, "step", 4),
        # complex128 factors, odd sides
        _case("mag_odd_direct_c128", "magnetic", "hetrf", 41, 33, 47, False, "direct", 2),
        # many small independent 2D systems at once, eight right-hand sides each
        _case("batch128_step", "diffusion", "potrf", 32, 256, 1, True, "step", 8, nsys=128),
    ]


def draw(rng):
    kind, fact, dim = rng.choice([("laplacian", "potrf", 3), ("diffusion", "potrf", 3), ("diffusion", "potrf", 2),
                                  ("diffusion", "sytrf", 3), ("convdiff", "getrf", 3), ("convdiff", "getrf", 2),
                                  ("magnetic", "hetrf", 3), ("diffusion", "potrf", 0)])
    mixed = rng.random() < 0.6
    op = rng.choice(["step", "step", "direct", "solve"])
    nrhs = rng.choice([1, 1, 2, 3, 4, 5, 8, 11, 16])

    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if dim == 0:
        lo = rng.randint(16, 48)
        return _case(None, kind, fact, lo, rng.randint(lo + 16, 256), 1, mixed, op, min(nrhs, 8), nsys=side(8, 96))
    if dim == 2:
        return _case(None, kind, fact, side(40, 700), side(40, 700), 1, mixed, op, nrhs, host=rng.random() < 0.2)
    top = {"magnetic": 52, "convdiff": 66}.get(kind, 80)
    m = side(12, top)
    nx, ny, nz = (max(8, min(top, int(round(m * rng.uniform(0.8, 1.2))))) for _ in range(3))
    return _case(None, kind, fact, nx, ny, nz, mixed, op, nrhs, host=nx * ny * nz < 60000 and rng.random() < 0.3)


# --- matrices -------------------------------------------------------------
def _sides(case):
    """Sides of the independent systems (the same for every seed: they are the pattern)."""
    if not case["batch"]:
        return [(case["nx"], case["ny"], case["nz"])]
    q = np.random.default_rng(7).integers(case["nx"], case["ny"] + 1, case["batch"])
    return [(int(s), int(s), 1) for s in q]


def _general(case):
    return case["kind"] == "convdiff"


@functools.lru_cache(maxsize=64)
def _pattern(nx, ny, nz, general):
    """CSC pattern of the grid matrix (0-based; lower triangle, or both for general ones) and, per
    column, which of the candidate rows (neighbours behind, itself, neighbours ahead) exist."""
    n = nx * ny * nz
    v = np.arange(n)
    x, y, z = v % nx, (v // nx) % ny, v // (nx * ny)
    ahead = [x < nx - 1, y < ny - 1, z < nz - 1]
    behind = [x > 0, y > 0, z > 0]
    off = [1, nx, nx * ny]
    cols = ([(behind[d], -off[d]) for d in (2, 1, 0)] if general else []) + [(np.ones(n, bool), 0)]
    cols += [(ahead[d], off[d]) for d in (0, 1, 2)]
    mask = np.stack([c[0] for c in cols], 1)
    rows = np.stack([v + c[1] for c in cols], 1)
    colptr = np.concatenate([[0], np.cumsum(mask.sum(1))]).astype(np.int64)
    return colptr, rows[mask].astype(np.int64), torch.from_numpy(mask)


@functools.lru_cache(maxsize=64)
def _analysis(nx, ny, nz, general):
    return analysis.analyze(_system(nx, ny, nz, "convdiff" if general else "diffusion"))


def _system(nx, ny, nz, kind):
    colptr, rowptr, _ = _pattern(nx, ny, nz, kind == "convdiff")
    mtx = {"convdiff": M.PastixGeneral, "magnetic": M.PastixHermitian}.get(kind, M.PastixSymmetric)
    values = np.zeros(1, np.complex128 if kind == "magnetic" else np.float64)   # (only its type is looked at)
    return M.SparseSystem(n=nx * ny * nz, colptr=colptr, rowptr=rowptr, values=values, mtxtype=mtx, grid=(nx, ny, nz))


@functools.lru_cache(maxsize=4)
def _forest(key):
    """Structure, pattern and first unknowns of the independent systems `key` as one block-diagonal one."""
    sides, kind = key
    systems = [_system(*s, kind) for s in sides]
    st, offs = batch.merge_structures([_analysis(*s, kind == "convdiff") for s in sides])
    nnz = np.concatenate([[0], np.cumsum([s.nnz for s in systems])])
    colptr = np.concatenate([[0]] + [s.colptr[1:] + k for s, k in zip(systems, nnz)]).astype(np.int64)
    rowptr = np.concatenate([s.rowptr + k for s, k in zip(systems, offs)]).astype(np.int64)
    merged = M.SparseSystem(n=int(offs[-1]), colptr=colptr, rowptr=rowptr, values=systems[0].values,
                            mtxtype=systems[0].mtxtype, grid=(int(offs[-1]), 1, 1))
    return st, merged, offs


def _structure(case):
    sides = _sides(case)
    if case["batch"]:
        return _forest((tuple(sides), case["kind"]))
    return _analysis(*sides[0], _general(case)), _system(*sides[0], case["kind"]), None


def _coefficients(nx, ny, nz, kind, gen, dev):
    """Per unknown: the diagonal, the entries ahead in its column (A[v + off_d, v]) and those behind
    (A[v - off_d, v], general matrices), as n-vectors, zero where there is no neighbour."""
    n, dim = nx * ny * nz, 3 if nz > 1 else 2
    v = torch.arange(n, device=dev)
    pos, ext, off = [v % nx, (v // nx) % ny, v // (nx * ny)], [nx, ny, nz], [1, nx, nx * ny]
    f64 = dict(dtype=torch.float64, device=dev)
    ahead = []
    if kind == "diffusion":      # face coefficients lognormal(0, 1), in 2D lognormal(0, 1/2); Dirichlet faces
        sigma = 1.0 if dim == 3 else 0.5
        diag = torch.zeros(n, **f64)
        for d in range(dim):
            inside = pos[d] < ext[d] - 1
            c = torch.exp(sigma * torch.randn(n, generator=gen, **f64))
            diag += c                                   # the face ahead (a neighbour or the boundary)
            lo = torch.exp(sigma * torch.randn(n, generator=gen, **f64))
            diag += torch.where(pos[d] > 0, torch.roll(c, off[d]), lo)
            ahead.append(torch.where(inside, -c, torch.zeros_like(c)))
        return diag, ahead, []
    if kind == "magnetic":       # Peierls phases, shifted to be indefinite
        for d in range(dim):
            th = 2 * math.pi * torch.rand(n, generator=gen, **f64)
            e = -torch.polar(torch.ones_like(th), -th)
            ahead.append(torch.where(pos[d] < ext[d] - 1, e, torch.zeros_like(e)))
        return torch.full((n,), 2.0 * dim - 0.5, dtype=torch.complex128, device=dev), ahead, []
    scale = torch.exp(0.05 * torch.randn(1, generator=gen, **f64))   # (a seed's own multiple of the matrix)
    if kind == "laplacian":
        one = torch.ones(n, **f64) * scale
        return 2.0 * dim * one, [torch.where(pos[d] < ext[d] - 1, -one, 0 * one) for d in range(dim)], []
    ph = 10.0 / (max(nx, ny, nz) + 1)                   # convection-diffusion, first-order upwind, Pe 10
    one = torch.ones(n, **f64) * scale
    ahead = [torch.where(pos[d] < ext[d] - 1, -(1 + ph) * one, 0 * one) for d in range(dim)]
    behind = [torch.where(pos[d] > 0, -one, 0 * one) for d in range(dim)]
    return dim * (2.0 + ph) * one, ahead, behind


def _values(nx, ny, nz, kind, co, dev):
    """The matrix values in the pattern's order."""
    diag, ahead, behind = co
    _, _, mask = _pattern(nx, ny, nz, kind == "convdiff")
    zero = torch.zeros_like(diag)
    pad = [zero] * (3 - len(ahead))
    cols = ((pad + behind[::-1]) if kind == "convdiff" else []) + [diag] + ahead + pad
    return torch.stack(cols, 1)[mask.to(dev)]


def _apply(nx, ny, nz, kind, co, x):
    """A x (x: nrhs x n) from the coefficients: A[v+o, v] = ahead[v], and the other triangle."""
    diag, ahead, behind = co
    b = diag * x
    for d, o in zip(range(len(ahead)), (1, nx, nx * ny)):
        a = ahead[d]
        b[:, o:] += (a * x)[:, :-o]
        if kind == "convdiff":
            b[:, :-o] += (behind[d] * x)[:, o:]
        else:
            b[:, :-o] += a.conj()[:-o] * x[:, o:]
    return b


def _inputs(case, seed, dev="cuda"):
    """(values, x_true, b) on the device; x_true and b as nrhs rows of n (a column-major n x nrhs block)."""
    gen = torch.Generator(device=dev).manual_seed(1000003 * seed + 17)
    vals, xs, bs = [], [], []
    for s in _sides(case):
        co = _coefficients(*s, case["kind"], gen, dev)
        n = s[0] * s[1] * s[2]
        comp = 2 if case["kind"] == "magnetic" else 1
        x = 2 * torch.rand(case["nrhs"], n, comp, generator=gen, dtype=torch.float64, device=dev) - 1
        x = torch.view_as_complex(x.contiguous()) if comp == 2 else x[:, :, 0]
        vals.append(_values(*s, case["kind"], co, dev))
        xs.append(x)
        bs.append(_apply(*s, case["kind"], co, x))
    cat = (lambda v, d: v[0].contiguous()) if len(vals) == 1 else (lambda v, d: torch.cat(v, d).contiguous())
    return cat(vals, 0), cat(xs, 1), cat(bs, 1)


# --- a pass ---------------------------------------------------------------
def prepare(case, seed):
    st, system, offs = _structure(case)
    values, _, b = _inputs(case, seed)
    s = G.Solver(device=torch.cuda.current_device())
    s.set_iparm(G.IPARM_FACTORIZATION, G.FACT[case["fact"]])
    s.set_iparm(G.IPARM_MIXED, 1 if case["mixed"] else 0)
    s.set_iparm(G.IPARM_REFINEMENT, G.REFINE["cg" if case["fact"] == "potrf" else "gmres"])
    s.set_dparm(G.DPARM_EPSILON_REFINEMENT, REFINE_EPS)
    s.set_structure(st)
    s.set_spm(system)
    if offs is not None:
        s.set_segments(offs)
    torch.cuda.synchronize()
    s.numfact(values)               # the plan, and for op "solve" the factors
    if case["host"]:
        values, b = values.cpu().numpy(), np.asfortranarray(b.cpu().numpy().T)
        x = None
    else:
        x = torch.empty_like(b)
    return dict(case=case, solver=s, values=values, b=b, x=x)


def run(state):
    case, s, b, x = state["case"], state["solver"], state["b"], state["x"]
    refined = case["op"] == "step" or (case["op"] == "solve" and case["mixed"])
    if case["op"] != "solve":
        s.numfact(state["values"])
    if case["host"]:
        return s.solve_and_refine(b) if refined else s.solve(b)
    nrhs, n = b.shape
    if refined:
        # (the C entry: the Python method of the name takes host arrays)
        rc = G.load().pastix_gpu_solve_and_refine(s._h, nrhs, ctypes.c_void_p(b.data_ptr()), n,
                                                  ctypes.c_void_p(x.data_ptr()), n)
        if rc:
            raise G.PastixGpuError("pastix_gpu_solve_and_refine", rc)
    else:
        x.copy_(b)
        torch.cuda.current_stream().synchronize()   # the solver works on a stream of its own
        s.solve_inplace(x, nrhs, n)
    return x


def exact(case, seed):
    """x_true: the solution of A x = b up to the rounding of b = A x_true, formed in 64 bits."""
    x = _inputs(case, seed)[1]
    return np.asfortranarray(x.cpu().numpy().T) if case["host"] else x


def work(case):
    """Flops of the factorization and one solve; the values, b and x once each, and for kept factors
    the factors once per sweep (they do not stay on the chip between the two)."""
    st, system, offs = _structure(case)
    cplx = case["kind"] == "magnetic"
    ct, bt = st["cblktab"], st["bloktab"]
    w = (ct[:-1, 1] - ct[:-1, 0] + 1).astype(np.float64)
    rows = np.concatenate([[0], np.cumsum(bt[:, 1] - bt[:, 0] + 1)])
    h = rows[ct[1:, 2]] - rows[ct[:-1, 2]]
    nnzl = float((h * w).sum() - (w * (w - 1) / 2).sum())
    mul = 4 if cplx else 1
    el = 16 if cplx else 8
    flops = 4.0 * mul * nnzl * case["nrhs"]
    size = 2.0 * el * system.n * case["nrhs"]
    if case["op"] == "solve":
        size += 2 * nnzl * (el / 2 if case["mixed"] else el)
    else:
        flops += mul * batch.system_flops(st, "getrf" if case["fact"] == "getrf" else "potrf")
        size += el * system.nnz
    return {"bytes": size, "flops": flops}


def tolerance(case):
    """Seen between two runs (the scatter-adds are atomic: their order differs): refined 1e-16 to 4e-13,
    plain FP64 solves 1e-16 to 5e-16, plain single-precision ones 2e-7 at 53 x 49 x 61 (1e-6 off the
    solution).  Stated for the worst conditioned of the range: a refined solution may differ by the 1e-13
    residual of its last iteration times a condition number of some 1e3 in the norm, the plain ones by
    the rounding of the type times the same, with the 2D grids of 700 x 700 the largest."""
    if case["op"] == "direct" and case["mixed"]:
        return {"rel": 3e-5, "max": 1e-3}
    if case["op"] == "step" or case["mixed"]:
        return {"rel": 1e-10, "max": 1e-8}
    return {"rel": 1e-13, "max": 1e-11}
