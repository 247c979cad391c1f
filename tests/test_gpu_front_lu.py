"""The panel pivot-block LU (k_front_lu6) at the sizes where it can go wrong: dense matrices in the identity orders, so that
one front (or a few) holds the whole matrix: fewer pivots than a panel, the last panel partial, full and alone, rows at the
edges of a warp and of the 128-row form, blocks over 128 rows; equal moduli in a column, moduli whose squares leave the
range, a singular column, and the shared-memory form (variant 1) on the same blocks.  Then the cluster form (k_block_lu_cl)
on larger ones: rows and panels that do not divide, the shortest and longest shares of a CTA, the same special values, a
tie between rows of different CTAs; and the grid form (k_block_lu_mc) on the blocks beyond it.  The bar is that of the parity
tests: the oracle's pivots, L and U within 1e-12; the largest blocks against the panel-by-panel form."""
import numpy as np
import pytest
import scipy.sparse as sp

import fplus_b200 as F
import oracle as O

pytestmark = pytest.mark.gpu

FACTOR_TOL = 1e-12


@pytest.fixture(scope="module")
def gpu():
    import torch
    assert torch.cuda.is_available(), "the GPU tests need a CUDA device"
    torch.cuda.init()
    return torch.device("cuda:0")


def _rel(A, B):
    s = 1.0 / abs(B).max()                     # (the squares of the tiny case's entries underflow)
    return sp.linalg.norm((A - B) * s) / sp.linalg.norm(B * s)


def _dense(n, cplx, seed, kind="plain"):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if cplx else 0)
    if kind == "ties":          # the first column's moduli all equal: the smallest row wins
        A[:, 0] = np.where(rng.random(n) < 0.5, -1.0, 1.0)
    elif kind == "tiny":
        A = A * 1e-170
    elif kind == "zeros":
        A[rng.random((n, n)) < 0.6] = 0.0
        A[np.arange(n), np.arange(n)] += 1.0
    Ap = np.arange(n + 1, dtype=np.int64) * n
    Ai = np.tile(np.arange(n, dtype=np.int64), n)
    return n, Ap, Ai, np.ascontiguousarray(A.T).ravel()


def _check(m, equilibrate=1, variant=2, width=256):
    n, Ap, Ai, Ax = m
    S = F.analyze(n, Ap, Ai, pin_dense=0, equilibrate=equilibrate)
    S.set_front_shape(width, 64, variant)
    N = S.factor(Ax, F.default_options(equilibrate=equilibrate, pin_dense=0))
    orc = O.OracleLU(n, Ap, Ai, Ax, S.row_perm, S.col_perm, equilibrate=equilibrate)
    assert np.array_equal(N.p, orc.p), "pivot order differs from the oracle"
    L, U, _ = N.factors()
    assert _rel(L, orc.L) <= FACTOR_TOL and _rel(U, orc.U) <= FACTOR_TOL


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 63, 65, 96, 109, 116, 127, 128, 129, 145])
@pytest.mark.parametrize("cplx", [False, True])
def test_sizes(gpu, cplx, n):
    _check(_dense(n, cplx, n))


@pytest.mark.parametrize("cplx,n,width", [(True, 129, 32), (True, 161, 64), (True, 193, 32), (True, 224, 32), (True, 225, 16),
                                          (False, 257, 64), (False, 301, 64), (False, 512, 32), (False, 513, 32)])
def test_tall_sizes(gpu, cplx, n, width):
    """Fronts of more than 128 rows and `width` pivots, to the most rows of the panel form and one more."""
    _check(_dense(n, cplx, n), width=width)


@pytest.mark.parametrize("kind", ["ties", "tiny", "zeros"])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("variant", [1, 2])
def test_values(gpu, cplx, kind, variant):
    _check(_dense(90, cplx, 5, kind), equilibrate=0 if kind != "zeros" else 1, variant=variant)


@pytest.mark.parametrize("cplx", [False, True])
def test_singular_column(gpu, cplx):
    """A column that becomes zero (to rounding) in the elimination is reported at its step."""
    n, Ap, Ai, Ax = _dense(40, cplx, 3)
    A = Ax.reshape(n, n)                       # row j: column j
    A[20] = A[3]                               # column 20 equals column 3
    S = F.analyze(n, Ap, Ai, pin_dense=0, equilibrate=0)
    with pytest.raises(F.FplusError) as e:
        S.factor(Ax, F.default_options(equilibrate=0, pin_dense=0))
    assert e.value.code == F.FPLUS_ERR_SINGULAR


# (pivot blocks of n rows and up to 256 columns; per CTA n / 16 rows: 10 to 63, a share that ends in a partial warp; widths
# that leave panels of 1, 15, 16, 17 and 31 columns)
@pytest.mark.parametrize("n", [161, 175, 193, 224, 239, 255, 257, 272, 303, 513, 1000])
@pytest.mark.parametrize("cplx", [False, True])
def test_cluster_sizes(gpu, cplx, n):
    _check(_dense(n, cplx, n))


@pytest.mark.parametrize("kind", ["ties", "tiny", "zeros"])
@pytest.mark.parametrize("cplx", [False, True])
def test_cluster_values(gpu, cplx, kind):
    _check(_dense(300, cplx, 7, kind), equilibrate=0 if kind != "zeros" else 1)


@pytest.mark.parametrize("col", [1, 37, 250])
@pytest.mark.parametrize("cplx", [False, True])
def test_cluster_singular_column(gpu, cplx, col):
    """As above in a block of the cluster form: reported, at any step of a panel, by a kernel that ends."""
    n, Ap, Ai, Ax = _dense(300, cplx, 3)
    A = Ax.reshape(n, n)
    A[col] = A[0]
    S = F.analyze(n, Ap, Ai, pin_dense=0, equilibrate=0)
    with pytest.raises(F.FplusError) as e:
        S.factor(Ax, F.default_options(equilibrate=0, pin_dense=0))
    assert e.value.code == F.FPLUS_ERR_SINGULAR


def _tall(n, cplx, seed, w=40):
    """w dense columns and a diagonal, in the identity orders: fronts of n, n - 256, .. rows.  Column 0's moduli are all equal."""
    rng = np.random.default_rng(seed)
    rows = np.arange(n, dtype=np.int64)
    Ai = np.concatenate([np.tile(rows, w), rows[w:]])
    Ap = np.concatenate([np.arange(w + 1) * n, w * n + 1 + np.arange(n - w)]).astype(np.int64)
    Ax = rng.standard_normal(Ai.size) + (1j * rng.standard_normal(Ai.size) if cplx else 0)
    Ax[:n] = np.where(rng.random(n) < 0.5, -1.0, 1.0)
    return n, Ap, Ai, Ax


# (512 real, 256 complex rows per CTA of a 16-CTA cluster, and a few more than it holds)
@pytest.mark.parametrize("cplx,n", [(False, 8192), (False, 8201), (True, 4096), (True, 4105)])
def test_tallest_blocks(gpu, cplx, n):
    """The cluster form at its most rows, and the grid form above: the pivots of the panel-by-panel form (variant 6)."""
    m = _tall(n, cplx, n)
    eye = np.arange(n, dtype=np.int64)
    opts = F.default_options(equilibrate=0)
    p = []
    for variant in (2, 6):
        S = F.Symbolic.from_orders(*m[:3], eye, eye)
        S.set_front_shape(256, 64, variant)
        N = S.factor(m[3], opts)
        p.append(N.p)
        x = np.random.default_rng(1).uniform(-1, 1, n)
        b = sp.csc_matrix((m[3], m[2], m[1]), shape=(n, n)) @ x
        assert O.backward_error(*m, N.solve(b), b) <= 1e-14
        del N
    assert np.array_equal(p[0], p[1]) and p[0][0] == 0


@pytest.mark.parametrize("cplx", [False, True])
def test_grid_singular_column(gpu, cplx):
    """The grid form reports a dependent column, and ends."""
    n, Ap, Ai, Ax = _tall(4105 if cplx else 8201, cplx, 2)
    Ax[37 * n:38 * n] = Ax[n:2 * n]
    eye = np.arange(n, dtype=np.int64)
    S = F.Symbolic.from_orders(n, Ap, Ai, eye, eye)
    with pytest.raises(F.FplusError) as e:
        S.factor(Ax, F.default_options(equilibrate=0))
    assert e.value.code == F.FPLUS_ERR_SINGULAR
