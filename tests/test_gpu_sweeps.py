"""The sweeps by packed 16-column pieces at the sizes where they can go wrong: the dense chain in one launch per sweep (a last
block of one pivot, partial 16-blocks, 8-, 32- and 64-pivot fronts, one and several blocks per worker) and by a launch per
front (more rows than one CTA takes), and the level-scheduled sweeps of the other fronts (narrow and wide fronts, the widest
on the 64-row substitution), for one right-hand side, the edges of a pass of eight, and every trans; diagonal blocks that are
too ill-conditioned for their inverses.  The bar is the parity tests': backward error at most 1e-14."""
import numpy as np
import pytest
import scipy.sparse as sp

import fplus_b200 as F
from fplus_b200 import workloads as W
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import torch
    assert torch.cuda.is_available(), "the GPU tests need a CUDA device"
    torch.cuda.init()
    return torch.device("cuda:0")


def _band(n, cplx, seed, hbw=5, ntau=3):
    """A band with ntau dense last rows and columns: the tail of it is one dense chain."""
    rng = np.random.default_rng(seed)
    k = np.arange(n, dtype=np.int64)
    rows = np.concatenate([k[(k + d >= 0) & (k + d < n)] for d in range(-hbw, hbw + 1)])
    cols = np.concatenate([k[(k + d >= 0) & (k + d < n)] + d for d in range(-hbw, hbw + 1)])
    t = n - 1 - np.arange(ntau, dtype=np.int64)
    rows = np.concatenate([rows, np.repeat(t, n), np.tile(k, ntau)])
    cols = np.concatenate([cols, np.tile(k, ntau), np.repeat(t, n)])
    _, first = np.unique(cols * n + rows, return_index=True)
    rows, cols = rows[first], cols[first]
    v = rng.standard_normal(len(rows)) + (1j * rng.standard_normal(len(rows)) if cplx else 0)
    Ap = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))]).astype(np.int64)
    return n, Ap, rows, v


def _check(m, S, N, nrhs, trans):
    n, Ap, Ai, Ax = m
    rng = np.random.default_rng(3 + nrhs)
    b = rng.standard_normal((n, nrhs)) + (1j * rng.standard_normal((n, nrhs)) if np.iscomplexobj(Ax) else 0)
    x = N.solve(b, trans)
    for r in range(nrhs):
        assert O.backward_error(n, Ap, Ai, Ax, x[:, r], b[:, r], trans) <= 1e-14, (nrhs, trans, r)


@pytest.mark.parametrize("nb", [32, 64])
@pytest.mark.parametrize("n", [129, 193, 257, 300, 611])
@pytest.mark.parametrize("cplx", [False, True])
def test_chain(gpu, cplx, n, nb):
    m = _band(n, cplx, n)
    S = F.analyze(*m[:3])
    S.set_front_shape(256, nb, 2)
    N = S.factor(m[3])
    assert N.info["f_dense"] < n
    for trans in ((0, 1, 2) if cplx else (0, 1)):
        for nrhs in (1, 2, 8, 9):
            _check(m, S, N, nrhs, trans)


@pytest.mark.parametrize("n,nb", [(2100, 32), (9300, 64)])
def test_chain_of_many_blocks(gpu, n, nb):
    """Chains of 66 and 146 blocks, a worker CTA per block."""
    m = _band(n, False, n)
    S = F.analyze(*m[:3])
    S.set_front_shape(256, nb, 2)
    N = S.factor(m[3])
    for trans in (0, 1):
        for nrhs in (1, 11):
            _check(m, S, N, nrhs, trans)


@pytest.mark.parametrize("cplx,nrhs", [(False, 1), (False, 9), (True, 1), (True, 5)])
def test_chain_of_several_blocks_per_worker(gpu, cplx, nrhs):
    """A chain of about 1,100 blocks of 8 pivots: seven or eight blocks per worker, their sums in shared memory (one
    right-hand side; real values) or in global memory (complex, several right-hand sides).  The solution equals, bit for bit,
    that of the launch per step that a captured graph takes, which has a CTA per block."""
    m = _band(9000, cplx, 6)
    n = m[0]
    S = F.analyze(*m[:3])
    S.set_front_shape(256, 8, 2)
    N = S.factor(m[3])
    assert (n - N.info["f_dense"]) // 8 > 7 * 147
    b = np.asfortranarray(np.random.default_rng(2).standard_normal((n, nrhs)) + (0j if cplx else 0))
    for trans in ((0, 1, 2) if cplx else (0, 1)):
        x = N.solve(b, trans)
        G = F.BatchGraph([N], nrhs, trans)
        G.upload(0, m[3], b)
        G.launch()
        assert G.status() == [0]
        assert np.array_equal(G.download(0).reshape(n, nrhs), x.reshape(n, nrhs)), trans
        for r in range(nrhs):
            assert O.backward_error(*m, x[:, r], b[:, r], trans) <= 1e-14


@pytest.mark.parametrize("ntau", [140, 230])
@pytest.mark.parametrize("cplx", [False, True])
def test_wide_chain(gpu, cplx, ntau):
    """Chain fronts of more than 197 rows, and of more than 256: a launch per front."""
    m = _band(900, cplx, 5, ntau=ntau)
    S = F.analyze(*m[:3])
    N = S.factor(m[3])
    P = S.plan(N.info["f_dense"])
    assert N.info["f_dense"] < m[0] and P["nrows"][P["col_front"][N.info["f_dense"]]:].max() > (256 if ntau == 230 else 197)
    for trans in ((0, 1, 2) if cplx else (0, 1)):
        for nrhs in (1, 2, 9):
            _check(m, S, N, nrhs, trans)


@pytest.mark.parametrize("cplx,width", [(False, 16), (False, 256), (False, 512), (False, 768), (True, 256), (True, 512)])
def test_levels(gpu, cplx, width):
    m = W.convdiff3d(12 if cplx else 16, 3)
    if cplx:
        m = (*m[:3], m[3] + 0.25j * np.random.default_rng(2).uniform(-1, 1, m[3].size))
    S = F.analyze(*m[:3])
    S.set_front_shape(width, 64, 2)
    N = S.factor(m[3])
    for trans in (0, 1):
        for nrhs in (1, 3, 8, 9, 33 if width < 512 else 17):     # (the widest fronts' vectors must fit one CTA: fewer at once)
            _check(m, S, N, nrhs, trans)


def _hard(kind, n, cplx, seed):
    """A dense matrix whose triangles hold 16 x 16 diagonal blocks with large inverses; what else it needs."""
    rng = np.random.default_rng(seed)
    i, j = np.indices((n, n))
    if kind.startswith("dependent"):           # columns within delta of a combination of the ones before them
        delta = float(kind.split(":")[1])
        A = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if cplx else 0)
        for c in (5, 15, 20, 37):
            A[:, c] = A[:, :c] @ rng.uniform(-1, 1, c) + delta * A[:, c]
    elif kind == "vandermonde":
        A = np.linspace(0.0, 1.0, n)[:, None] ** np.arange(n)
    elif kind == "kernel":
        t = np.linspace(0.0, 1.0, n)
        A = np.exp(-4.0 * (t[:, None] - t) ** 2)
    elif kind == "upper":                       # U = A
        A = np.where(i == j, 0.1, np.where((j > i) & (j // 16 == i // 16), -1.0, 0.0))
    else:                                       # "lower": L = A, multipliers of one
        A = np.where(i == j, 1.0, np.where((j < i) & (j // 16 == i // 16), -1.0, 0.0))
    if cplx:
        A = A * np.exp(0.7j)
    return n, np.arange(n + 1, dtype=np.int64) * n, np.tile(np.arange(n, dtype=np.int64), n), np.ascontiguousarray(A.T).ravel()


def _check_from_x(m, N, nrhs, trans):
    """b = op(A) x with a moderate x (a random b lets x grow along the small directions, which hides a large residual)."""
    n, Ap, Ai, Ax = m
    rng = np.random.default_rng(11 + nrhs)
    A = sp.csc_matrix((Ax, Ai, Ap), shape=(n, n))
    x = rng.uniform(-1, 1, (n, nrhs)) + (1j * rng.uniform(-1, 1, (n, nrhs)) if np.iscomplexobj(Ax) else 0)
    b = np.asarray({0: A, 1: A.T, 2: A.conj().T}[trans] @ x)
    y = N.solve(b, trans)
    worst = max(O.backward_error(n, Ap, Ai, Ax, y[:, r], b[:, r], trans) for r in range(nrhs))
    assert worst <= 1e-14, (nrhs, trans, worst)


@pytest.mark.parametrize("kind,n", [("dependent:1e-4", 64), ("dependent:1e-7", 64), ("dependent:1e-7", 180), ("vandermonde", 16),
                                    ("kernel", 32), ("upper", 16), ("upper", 180), ("lower", 48), ("lower", 180)])
@pytest.mark.parametrize("where", ["tree", "chain"])
@pytest.mark.parametrize("cplx", [False, True])
def test_ill_conditioned_diagonal_blocks(gpu, cplx, where, kind, n):
    """The backward error of a solve does not depend on the conditioning of the triangles' diagonal blocks: fronts of the
    tree (np <= 64 and wider), and the dense chain (every row taken as dense)."""
    m = _hard(kind, n, cplx, 4)
    eye = np.arange(n, dtype=np.int64)
    S = F.Symbolic.from_orders(*m[:3], eye, eye) if where == "chain" else F.analyze(*m[:3], pin_dense=0)
    assert np.array_equal(S.col_perm, eye) and np.array_equal(S.row_perm, eye)
    N = S.factor(m[3], F.default_options(equilibrate=0, pivot_rel=0.0, pin_dense=0))
    assert N.info["f_dense"] == (0 if where == "chain" else n)
    for trans in ((0, 1, 2) if cplx else (0, 1)):
        for nrhs in (1, 3, 9):
            _check_from_x(m, N, nrhs, trans)


def _row_error(m, x, b, trans):
    A = sp.csc_matrix((m[3], m[2], m[1]), shape=(m[0], m[0]))
    A = {0: A, 1: A.T, 2: A.conj().T}[trans]
    return float((abs(A @ x - b) / (abs(A) @ abs(x) + abs(b))).max())


@pytest.mark.parametrize("where", ["tree", "chain"])
@pytest.mark.parametrize("cplx", [False, True])
def test_graded_rows(gpu, cplx, where):
    """Every row's residual is small beside that row (or column, transposed) of an upper triangular matrix: 16 x 16 blocks of
    0.1 and -1 whose rows grow a hundredfold each (a large inverse that norms of the unscaled block do not show)."""
    n = 112
    m = _hard("upper", n, cplx, 1)
    A = m[3].reshape(n, n).T * 100.0 ** (np.arange(n) % 16)[:, None]
    eye = np.arange(n, dtype=np.int64)
    for trans in ((0, 1, 2) if cplx else (0, 1)):
        # (transposed: the columns grow, towards the first)
        B = A if trans == 0 else m[3].reshape(n, n).T * 100.0 ** (15 - np.arange(n) % 16)[None, :]
        mm = (*m[:3], np.ascontiguousarray(B.T).ravel())
        S = F.Symbolic.from_orders(*mm[:3], eye, eye) if where == "chain" else F.analyze(*mm[:3], pin_dense=0)
        N = S.factor(mm[3], F.default_options(equilibrate=0, pivot_rel=0.0, pin_dense=0))
        assert np.array_equal(N.p, eye)
        for nrhs in (1, 9):
            x = np.random.default_rng(nrhs).uniform(-1, 1, (n, nrhs))
            C = {0: B, 1: B.T, 2: B.conj().T}[trans]
            y = N.solve(C @ x, trans)
            assert max(_row_error(mm, y[:, r], (C @ x)[:, r], trans) for r in range(nrhs)) <= 1e-14


@pytest.mark.parametrize("delta", [1e-4, 1e-7])
@pytest.mark.parametrize("nb", [32, 64])
@pytest.mark.parametrize("cplx", [False, True])
def test_ill_conditioned_chain(gpu, cplx, nb, delta):
    """The same on the dense chain: columns all along it that depend on the two before them to delta."""
    n, Ap, Ai, Ax = _band(500, cplx, 8, hbw=5, ntau=3)
    A = sp.csc_matrix((Ax, Ai, Ap), shape=(n, n)).tolil()
    for c in range(40, n - 3, 23):
        A[:, c] = 0.7 * A[:, c - 1] - 0.4 * A[:, c - 2] + delta * A[:, c]
    A = A.tocsc()
    A.sort_indices()
    m = n, A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data.copy()
    eye = np.arange(n, dtype=np.int64)
    S = F.Symbolic.from_orders(*m[:3], eye, eye)
    S.set_front_shape(256, nb, 2)
    N = S.factor(m[3])
    assert N.info["f_dense"] < 200
    for trans in ((0, 1, 2) if cplx else (0, 1)):
        for nrhs in (1, 9):
            _check_from_x(m, N, nrhs, trans)


def test_device_bytes_count_the_packed_triangles(gpu):
    """info's device_bytes hold the factors and the triangles packed for the sweeps (16 x 16 blocks and panels)."""
    n = 100000
    k = np.arange(n)
    A = sp.csc_matrix((np.concatenate([np.full(n, 4.0), np.ones(2 * n - 2)]),
                       (np.concatenate([k, k[1:], k[:-1]]), np.concatenate([k, k[:-1], k[1:]]))), shape=(n, n))
    S = F.analyze(n, A.indptr.astype(np.int64), A.indices.astype(np.int64))
    N = S.factor(A.data)
    P = S.plan()
    npiv, nc = np.bincount(P["col_front"]), np.diff(P["col_ptr"])
    entries = int((P["nrows"] * npiv + npiv * (nc - npiv)).sum())
    packed = 512 * int((npiv >= 16).sum())          # fronts of one block: its upper and its lower triangle
    assert N.info["device_bytes"] >= 8 * (entries + packed) + 2 * 8 * A.nnz


def test_small_fronts_pack_small(gpu):
    """Fronts of a few pivots (here mostly one) take a few packed entries each, not whole 16 x 16 blocks."""
    n = 60000
    rng = np.random.default_rng(0)
    A = (sp.identity(n) * 4.0 + sp.coo_matrix((rng.standard_normal(n // 4), (rng.integers(0, n, n // 4), rng.integers(0, n, n // 4))),
                                              shape=(n, n))).tocsc()
    m = n, A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data
    S = F.analyze(*m[:3])
    N = S.factor(A.data)
    assert np.bincount(S.plan()["col_front"]).mean() < 1.5
    assert N.info["device_bytes"] < 24e6            # (over 180 MB with a block each)
    for nrhs in (1, 9):
        _check(m, S, N, nrhs, 0)


@pytest.mark.parametrize("cplx", [False, True])
def test_one_block_fronts(gpu, cplx):
    """Independent dense blocks of 1 to 20 pivots: every side of a packed block, in product and in substitution form."""
    rng = np.random.default_rng(5)
    blocks = []
    for k in range(1, 21):
        B = rng.standard_normal((k, k)) + (1j * rng.standard_normal((k, k)) if cplx else 0)
        blocks.append(B)
        if k > 2:
            B = B.copy()
            B[:, k - 2] = B[:, :k - 2] @ rng.uniform(-1, 1, k - 2) + 1e-6 * B[:, k - 2]
            blocks.append(B)
    A = sp.block_diag([sp.coo_matrix(B) for B in blocks], format="csc")
    A.sort_indices()
    m = A.shape[0], A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data.copy()
    S = F.analyze(*m[:3])
    N = S.factor(m[3])
    for trans in ((0, 1, 2) if cplx else (0, 1)):
        for nrhs in (1, 2, 8, 9):
            _check_from_x(m, N, nrhs, trans)
