"""Cholesky solves held to a bound in every entry, for right-hand sides, solutions and matrices whose entries lie many
binades apart.

A solve by a Cholesky factor in binary64 has x = x' + dx with |dx| <= g |A^-1| |L| |L^T| |x| entry by entry, g about
3 n u (u = EPS / 2) from the factor and the two substitutions. From n = 17 on an entry of the factor may be off by
10 n EPS of (|L| |L^T|)_ij more, so g = 12 n EPS. The exact solution and the bound are taken in extended precision.
"""
import functools

import numpy as np
import pytest

from helpers import EPS, spd, to_dev

pytestmark = pytest.mark.gpu
LD = np.longdouble


def chol(A):
    """The Cholesky factor in extended precision."""
    S, n = A.astype(LD), len(A)
    L = np.zeros((n, n), LD)
    for k in range(n):
        L[k:, k] = S[k:, k] / np.sqrt(S[k, k])
        S[k + 1:, k + 1:] -= np.outer(L[k + 1:, k], L[k + 1:, k])
    return L


def solve(L, B):
    """(L L^T)^-1 B in extended precision."""
    X = B.astype(LD)
    for k in range(len(L)):
        X[k] /= L[k, k]
        X[k + 1:] -= np.outer(L[k + 1:, k], X[k])
    for k in reversed(range(len(L))):
        X[k] = (X[k] - L[k + 1:, k] @ X[k + 1:]) / L[k, k]
    return X


@functools.lru_cache(maxsize=None)
def exact(n, data):
    """The factor R of a matrix given by its bytes, |R| |R^T|, and |A^-1| |R| |R^T|."""
    R = chol(np.frombuffer(data).reshape(n, n))
    M = np.abs(R) @ np.abs(R.T)
    return R, M, np.abs(solve(R, np.eye(n))) @ M


def check(A, B, X, L=None):
    """X (and the factor L) against the bounds above; B and X are n x r."""
    n = len(A)
    R, M, G = exact(n, np.ascontiguousarray(A).tobytes())
    want = solve(R, B)
    assert np.all(np.abs(X - want) <= 12 * n * EPS * (G @ np.abs(want)))
    if L is not None:
        L = np.tril(L).astype(LD)
        assert np.all(np.abs(np.tril(L @ L.T - A)) <= np.tril(11 * n * EPS * M))


def run(gpu, As, Bs):
    """posv of matrices of one size: (info, L, X)."""
    import torch

    A, B = np.stack(As), np.stack(Bs)
    L, X = gpu.col_major((len(A),), A.shape[1], A.shape[1], "cuda").zero_(), gpu.col_major((len(A),), *B.shape[1:], "cuda")
    info = gpu.posv(to_dev(A), L, to_dev(B), X)
    torch.cuda.synchronize()
    return info.cpu().numpy(), L.cpu().numpy(), X.cpu().numpy()


def apart(rng, n):
    """Systems whose solutions' entries lie far apart, with entries of the matrix that do not: (A, b)."""
    e = np.eye(n)
    first = np.ones(n)
    first[0] = 1e20
    yield e, first
    first[0] = 1e6
    yield 3 * e, first / 3
    for far in (1e6, 1e12, 1e100):  # independent blocks
        A = np.zeros((n, n))
        h = n // 2
        A[:h, :h], A[h:, h:] = spd(rng, h), spd(rng, n - h)
        b = rng.standard_normal(n)
        b[:h] *= far
        yield A, b
    yield 4 * e - np.eye(n, k=1) - np.eye(n, k=-1), e[0]  # a Green's function
    yield 4 * e - np.eye(n, k=1) - np.eye(n, k=-1), e[n - 1]
    for d in (1e-6, 1e-12, 1e-40):
        diag = np.where(np.arange(n) % 2, d, 1.0)
        yield np.diag(diag), diag
    yield spd(rng, n), 10.0 ** rng.uniform(-60, 60, n)


@pytest.mark.parametrize("n", [17, 31, 48, 64, 65, 130])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 8, 11])
def test_entries_of_the_solution(gpu, n, nrhs):
    """Every entry of X, one right-hand side beside others of another kind."""
    rng = np.random.default_rng(n)
    As, bs = zip(*apart(rng, n))
    Bs = [rng.standard_normal((n, nrhs)) for _ in bs]
    for k, b in enumerate(bs):
        Bs[k][:, k % nrhs] = b
    info, L, X = run(gpu, As, Bs)
    assert not info.any()
    for k in range(len(As)):
        check(As[k], Bs[k], X[k], L[k])


@pytest.mark.parametrize("n", [32, 48, 64])
def test_equal_correlations(gpu, n):
    """Columns of the factor whose norm grows with n (all correlations 0.999), constant right-hand sides of 2,000
    magnitudes: the sums of a substitution are bounded by no norm of a row."""
    A = np.full((n, n), 0.99)
    np.fill_diagonal(A, 0.991)
    beta = 1 + np.arange(2000) / 2000.0
    info, _, X = run(gpu, [A] * 250, [np.outer(np.ones(n), beta[8 * k:8 * k + 8]) for k in range(250)])
    assert not info.any()
    x = np.concatenate(list(X), axis=1)
    R, _, G = exact(n, A.tobytes())
    want = solve(R, np.ones((n, 1))) * beta.astype(LD)
    assert np.all(np.abs(x - want) <= 12 * n * EPS * (G @ np.abs(want)))


@pytest.mark.parametrize("n", [17, 48, 64, 65])
def test_non_finite_right_hand_sides(gpu, oracle_lib, n):
    """Infinities and NaN in a right-hand side go where binary64 substitutions take them; other columns stay."""
    rng = np.random.default_rng(n)
    A, B = spd(rng, n), rng.standard_normal((n, 4))
    B[3, 1], B[n - 1, 2], B[0, 3] = np.nan, np.inf, -np.inf
    _, _, X = run(gpu, [A] * 3, [B] * 3)
    want = oracle_lib.posv_batch(A[None], B[None])[1][0]
    assert np.array_equal(np.isfinite(X[0]), np.isfinite(want)) and X[0][n - 1, 2] == np.inf
    check(A, B[:, :1], X[0][:, :1])
