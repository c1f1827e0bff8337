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


def coupled(n):
    """Matrices whose unknowns are coupled weakly, directly or by way of many others: entries of the matrix, of its
    factor and of the solution fall far below their rows' largest."""
    rng = np.random.default_rng(n)
    i, h = np.arange(n), n // 2
    d = np.abs(i[:, None] - i[None, :])
    blocks = np.zeros((n, n))
    blocks[:h, :h], blocks[h:, h:] = spd(rng, h), spd(rng, n - h)
    for entry in (1e-20, 1e-9):
        A = blocks.copy()
        A[n - 2, 3] = A[3, n - 2] = entry
        yield A
    A = blocks.copy()
    A[h:, :h] = 1e-7 * rng.standard_normal((n - h, h))
    A[:h, h:] = A[h:, :h].T
    yield A
    yield np.exp(-(0.9 * d) ** 2 / 2) + 0.1 * np.eye(n)  # a Gaussian kernel
    yield np.exp(-3.0 * d)
    A = 4.0 * np.eye(n) - (d == 1) - (d == n - 1)  # a ring
    yield A
    yield A * np.outer(2.0 ** (i % 5 * 20), 2.0 ** (i % 5 * 20))


@pytest.mark.parametrize("n", [17, 33, 48, 64, 65, 129, 200])
def test_weakly_coupled_unknowns(gpu, n):
    import torch

    As = list(coupled(n))
    B = np.stack([np.eye(n)[0], np.eye(n)[n - 1], np.eye(n)[n // 2], np.random.default_rng(n).standard_normal(n)], 1)
    info, L, X = run(gpu, As, [B] * len(As))
    assert not info.any()
    for A, l, x in zip(As, L, X):
        check(A, B, x, l)
    P = to_dev(np.stack(As))  # in place
    info2 = gpu.potrf(P, P)
    torch.cuda.synchronize()
    assert not info2.any() and np.array_equal(np.tril(P.cpu().numpy()), np.tril(L))


@pytest.mark.parametrize("ns", [[17, 40, 64, 33], [20, 128, 65, 48], [300, 129, 18, 100]])
def test_weakly_coupled_ragged(gpu, ns):
    """The same through the ragged plan, and with the factor taken again in the adjoint."""
    import torch

    from blast_gb300.autograd import spd_solve_packed
    from blast_gb300.ragged import Packed, PosvPlan

    which = [(n, k) for n in ns if n <= 129 for k in range(7)] + [(n, 5) for n in ns if n > 129]
    As = [list(coupled(n))[k] for n, k in which]
    n = [a for a, _ in which]
    Bs = [np.eye(a)[:, :1] + (np.arange(a) == a - 1)[:, None] for a in n]
    A, B, X, L = (Packed(n, c, "cuda") for c in (n, [1] * len(n), [1] * len(n), n))
    A.fill_from(As)
    B.fill_from(Bs)
    plan = PosvPlan(A, B, X, L)
    plan.run()
    a, b = A.buf.clone().requires_grad_(), B.buf.clone().requires_grad_()
    spd_solve_packed(a, b, np.array(n), np.ones(len(n), dtype=np.int64), keep_factor=False).backward(B.buf)
    torch.cuda.synchronize()
    assert not plan.results()[0].any()
    at = 0
    for m, Ah, Bh, Lg, Xg in zip(n, As, Bs, L.to_list(), X.to_list()):
        check(Ah, Bh, Xg, Lg)
        check(Ah, Bh, b.grad[at:at + m].cpu().numpy()[:, None])
        at += m


@pytest.mark.parametrize("n", [65, 80, 150])
def test_weakly_coupled_mirror(gpu, n):
    """The entry for host memory: the device call's factor, with workspaces of its own."""
    import torch

    from blast_gb300 import _lib

    As = np.stack(list(coupled(n)))
    m = len(As)
    dA, dB = to_dev(As), to_dev(np.tile(np.eye(n)[:, :1], (m, 1, 1)))
    L, X = gpu.col_major((m,), n, n, "cuda").zero_(), gpu.col_major((m,), n, 1, "cuda")
    gpu.posv(dA, L, dB, X)
    hL, hX = torch.zeros(m * n * n).double().pin_memory(), torch.zeros(m * n).double().pin_memory()
    wL, wX = torch.empty(m * n * n, device="cuda").double(), torch.empty(m * n, device="cuda").double()
    info = torch.full((m,), -1, dtype=torch.int32, device="cuda")
    _lib.call("blastgpu_dposv_mirror_strided", n, 1, dA.data_ptr(), n, n * n, dB.data_ptr(), n, n, hL.data_ptr(), n, n * n,
              hX.data_ptr(), n, n, wL.data_ptr(), wX.data_ptr(), info.data_ptr(), m, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert not info.any()
    assert np.array_equal(np.tril(hL.numpy().reshape(m, n, n).transpose(0, 2, 1)), np.tril(L.cpu().numpy()))
    for k in range(m):
        check(As[k], np.eye(n)[:, :1], hX.numpy()[k * n:(k + 1) * n, None])


@pytest.mark.parametrize("n", [17, 33, 64, 65, 128, 300, 512])
def test_info_is_binary64s(gpu, oracle_lib, n):
    """Pivots down to nothing, and rows far too long for their diagonal: info as binary64 finds it."""
    import torch

    As = []
    for x in (2.0 ** -26 * np.sqrt(1 - 2.0 ** -10), 2.0 ** -26 * np.sqrt(1 - 2.0 ** -25), 2.0 ** -26):  # pivot 2^-62, 2^-77, 0
        A = np.eye(n)
        A[n - 1, n - 1] += 2.0 ** -52
        A[n - 1, 0] = A[0, n - 1] = 1.0
        A[n - 1, 1] = A[1, n - 1] = x
        As.append(A)
    for x in np.concatenate([np.linspace(0.1, 1.9999, 40), [1.99999]]):
        A = np.eye(n)
        A[n - 1, :n - 1] = A[:n - 1, n - 1] = x
        As.append(A)
    As = np.stack(As)
    P = to_dev(As)
    info = gpu.potrf(P, P)
    torch.cuda.synchronize()
    got = P.cpu().numpy()
    for k, A in enumerate(As):
        ref = np.zeros((n, n), order="F")
        want = oracle_lib.potrf(np.asfortranarray(A), ref)
        assert info[k] == want, (k, int(info[k]), want)
        if want == 0:
            assert np.allclose(np.tril(got[k]), np.tril(ref), rtol=10 * n * EPS, atol=0)


def structured(rng, n):
    """A sparse graph with weights over 12 decades, a Gram matrix with entries over 8, blocks with a weak dense coupling, a
    kernel in random order, and a matrix with one tiny entry among others that are not."""
    M = np.triu(rng.random((n, n)) < 0.2, 1) * 10.0 ** rng.uniform(-12, 0, (n, n)) * rng.choice([-1, 1], (n, n))
    M = M + M.T
    yield M + np.diag(np.abs(M).sum(1) * rng.uniform(1, 2) + 10.0 ** rng.uniform(-3, 0, n))
    G = rng.standard_normal((n, n)) * 10.0 ** rng.uniform(-8, 0, (n, n)) * (rng.random((n, n)) < 0.5)
    yield G @ G.T + 10.0 ** rng.uniform(-4, 0) * np.eye(n)
    A, h = np.zeros((n, n)), n // 3
    A[:h, :h], A[h:, h:] = spd(rng, h), spd(rng, n - h)
    C = rng.standard_normal((n, n)) * 10.0 ** rng.uniform(-14, -1)
    yield A + 0.05 * (C + C.T)
    x = rng.uniform(0, rng.choice([3, 10, 30]), n)
    yield np.exp(-np.abs(x[:, None] - x) ** 1.5) + 10.0 ** rng.uniform(-3, 0) * np.eye(n)
    A = spd(rng, n)
    A[n - 1, 1] = A[1, n - 1] = 10.0 ** rng.uniform(-20, -3)
    yield A


@pytest.mark.parametrize("n", [17, 48, 64, 100])
def test_structured_matrices(gpu, n):
    """Every entry of the solution, whatever becomes of single small entries of the factor."""
    rng = np.random.default_rng(n)
    As = [A for _ in range(12) for A in structured(rng, n)]
    Bs = [np.stack([np.eye(n)[rng.integers(n)], rng.standard_normal(n)], 1) for _ in As]
    info, _, X = run(gpu, As, Bs)
    assert not info.any()
    for A, B, x in zip(As, Bs, X):
        check(A, B, x)
