"""The panel pivot-block LU (k_front_lu6) at the sizes where it can go wrong: dense matrices in the identity orders, so that
one front (or a few) holds the whole matrix: fewer pivots than a panel, the last panel partial, full and alone, rows at the
edges of a warp and of the 128-row form, blocks over 128 rows; equal moduli in a column, moduli whose squares leave the
range, a singular column, and the shared-memory form (variant 1) on the same blocks.  Then the cluster form (k_block_lu_cl)
on larger ones: rows and panels that do not divide, the shortest and longest shares of a CTA, the same special values, a
tie between rows of different CTAs.  The bar is that of the parity tests: the oracle's pivots, L and U within 1e-12."""
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


def _check(m, equilibrate=1, variant=2):
    n, Ap, Ai, Ax = m
    S = F.analyze(n, Ap, Ai, pin_dense=0, equilibrate=equilibrate)
    S.set_front_shape(256, 64, variant)
    N = S.factor(Ax, F.default_options(equilibrate=equilibrate, pin_dense=0))
    orc = O.OracleLU(n, Ap, Ai, Ax, S.row_perm, S.col_perm, equilibrate=equilibrate)
    assert np.array_equal(N.p, orc.p), "pivot order differs from the oracle"
    L, U, _ = N.factors()
    assert _rel(L, orc.L) <= FACTOR_TOL and _rel(U, orc.U) <= FACTOR_TOL


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 63, 65, 96, 109, 116, 127, 128, 129, 145])
@pytest.mark.parametrize("cplx", [False, True])
def test_sizes(gpu, cplx, n):
    _check(_dense(n, cplx, n))


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
