"""The sweeps by inverted 16 x 16 diagonal blocks at the sizes where they can go wrong: the dense chain in one launch (a last
block of one pivot, partial 16-blocks, 32- and 64-pivot fronts, one and several blocks per worker, the cluster and the
cooperative form) and the level-scheduled sweeps of the other fronts (narrow and wide fronts, the widest on the 64-row
substitution), for one right-hand side, the edges of a pass of eight, and every trans.  The bar is the parity tests': backward
error at most 1e-14."""
import numpy as np
import pytest

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
    """More than four blocks per worker in one cluster; a cooperative launch."""
    m = _band(n, False, n)
    S = F.analyze(*m[:3])
    S.set_front_shape(256, nb, 2)
    N = S.factor(m[3])
    for trans in (0, 1):
        for nrhs in (1, 11):
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
