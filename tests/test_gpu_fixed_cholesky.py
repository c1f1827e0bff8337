"""The fixed-point Cholesky kernels (16 < n <= 512) at the edges of their tiles: blocks of 16, chunks of 32,
64 and 128 rows, one matrix or an odd number of them, and inputs that are not positive definite.

Tolerances: a factor entry is held to 2^-60 of its row's norm, below binary64's 2^-53, so the factor is
held to the library's bar against the oracle, 10 n eps normwise, and the solutions to 100 n eps.
"""
import numpy as np
import pytest

from helpers import EPS, normwise, spd, spd_batch, to_dev

pytestmark = pytest.mark.gpu

EDGES = [17, 31, 32, 33, 48, 49, 63, 64, 65, 79, 96, 127, 128, 129, 145, 257, 511, 512]


@pytest.mark.parametrize("n", EDGES)
def test_posv_against_oracle(gpu, oracle_lib, n):
    import torch

    rng = np.random.default_rng(n)
    batch, nrhs = 3, 1 + n % 9
    A, B = spd_batch(rng, batch, n), rng.standard_normal((batch, n, nrhs))
    # leading dimensions other than n: rows past n are not touched
    dA, dB = to_dev(A, ld=n + 1), to_dev(B, ld=n + 3)
    L = gpu.col_major((batch,), n, n, "cuda", ld=n + 2).zero_()
    X = gpu.col_major((batch,), n, nrhs, "cuda")
    info = gpu.posv(dA, L, dB, X)
    P = to_dev(A)
    info2 = gpu.potrf(P, P)
    torch.cuda.synchronize()
    assert not info.any() and not info2.any()
    Lr, Xr, _ = oracle_lib.posv_batch(A, B)
    for b in range(batch):
        assert normwise(np.tril(L.cpu().numpy()[b]), np.tril(Lr[b])) <= 10 * n * EPS
        assert normwise(X.cpu().numpy()[b], Xr[b]) <= 100 * n * EPS
    assert torch.equal(torch.tril(P), torch.tril(L))  # in place
    assert np.all(np.triu(L.cpu().numpy(), 1) == 0)


@pytest.mark.parametrize("n", [17, 33, 64, 65, 130, 300])
def test_units_of_the_unknowns(gpu, n):
    """A diagonal scaling by powers of two scales the factor and the solution, exactly."""
    import torch

    rng = np.random.default_rng(1000 + n)
    A, B = spd_batch(rng, 2, n), rng.standard_normal((2, n, 3))
    d = 2.0 ** rng.integers(-120, 121, (2, n))
    L0, L1 = (gpu.col_major((2,), n, n, "cuda").zero_() for _ in range(2))
    X0, X1 = (gpu.col_major((2,), n, 3, "cuda") for _ in range(2))
    gpu.posv(to_dev(A), L0, to_dev(B), X0)
    gpu.posv(to_dev(A * d[:, :, None] * d[:, None, :]), L1, to_dev(B * d[:, :, None]), X1)
    torch.cuda.synchronize()
    assert np.array_equal(L1.cpu().numpy(), L0.cpu().numpy() * d[:, :, None])
    assert np.array_equal(X1.cpu().numpy(), X0.cpu().numpy() / d[:, :, None])


@pytest.mark.parametrize("n", [20, 48, 64, 70, 150, 300])
def test_not_positive_definite(gpu, oracle_lib, n):
    """info is the first pivot that is not positive, for a negative pivot, an off-diagonal entry too large
    for its diagonal, NaN and infinity; the other matrices of the batch are solved."""
    import torch

    rng = np.random.default_rng(2000 + n)
    A, B = spd_batch(rng, 7, n), rng.standard_normal((7, n, 2))
    A[1, n // 2, n // 2] = -1.0
    A[2, n - 1, 3] = A[2, 3, n - 1] = 1e6 * n
    A[3, 18, 5] = np.nan
    A[4, 17, 17] = 0.0
    A[5, n - 2, 16] = np.inf
    dA, L, X = to_dev(A), gpu.col_major((7,), n, n, "cuda").zero_(), gpu.col_major((7,), n, 2, "cuda")
    info = gpu.posv(dA, L, to_dev(B), X).cpu().numpy()
    want = []
    for b in range(7):
        want.append(oracle_lib.potrf(np.asfortranarray(A[b]), np.zeros((n, n), order="F")))
    assert list(info) == want and want[0] == 0 and want[6] == 0
    Lr, Xr, _ = oracle_lib.posv_batch(A[[0, 6]], B[[0, 6]])
    for k, b in enumerate((0, 6)):
        assert normwise(np.tril(L.cpu().numpy()[b]), np.tril(Lr[k])) <= 10 * n * EPS
        assert normwise(X.cpu().numpy()[b], Xr[k]) <= 100 * n * EPS
    # columns before the failed pivot are the factor's, the later ones NaN
    c = want[1] - 1
    Lb = L.cpu().numpy()[1]
    ref = np.zeros((n, n), order="F")
    oracle_lib.potrf(np.asfortranarray(A[1]), ref)
    assert normwise(np.tril(Lb)[:, :c], np.tril(ref)[:, :c]) <= 10 * n * EPS
    assert np.isnan(np.tril(Lb)[c:, c:][np.tril_indices(n - c)]).all()
    assert np.isnan(X.cpu().numpy()[1]).all()


@pytest.mark.parametrize("n,cond", [(40, 1e10), (64, 1e6), (100, 1e12), (300, 1e8)])
def test_ill_conditioned_backward_error(gpu, n, cond):
    """Backward error of solutions that grow within a block: at most binary64's n eps (LAPACK's bound
    for a Cholesky solve has 3 n)."""
    import torch

    rng = np.random.default_rng(3000 + n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = (Q * np.logspace(0, -np.log10(cond), n)) @ Q.T
    A, b = (A + A.T) / 2, rng.standard_normal((n, 2))
    L, X = gpu.col_major((1,), n, n, "cuda").zero_(), gpu.col_major((1,), n, 2, "cuda")
    info = gpu.posv(to_dev(A[None]), L, to_dev(b[None]), X)
    torch.cuda.synchronize()
    assert not info.any()
    x = X.cpu().numpy()[0].astype(np.longdouble)
    for k in range(2):
        r = b[:, k] - A.astype(np.longdouble) @ x[:, k]
        be = np.abs(r).max() / (np.abs(A).sum(1).max() * np.abs(x[:, k]).max() + np.abs(b[:, k]).max())
        assert be <= n * EPS, be


def test_solution_scales_apart(gpu):
    """Right-hand sides of any magnitude, zero and non-finite ones among them."""
    import torch

    rng = np.random.default_rng(4000)
    n = 50
    A = spd(rng, n)[None]
    B = rng.standard_normal((1, n, 12)) * 10.0 ** np.linspace(-280, 280, 12)
    B[0, :, 4] = 0.0
    B[0, 7, 5] = np.nan
    L, X = gpu.col_major((1,), n, n, "cuda").zero_(), gpu.col_major((1,), n, 12, "cuda")
    gpu.posv(to_dev(A), L, to_dev(B), X)
    torch.cuda.synchronize()
    x = X.cpu().numpy()[0]
    assert np.all(x[:, 4] == 0) and np.isnan(x[:, 5]).all()
    for k in set(range(12)) - {4, 5}:
        s = 2.0 ** -np.floor(np.log2(np.abs(B[0, :, k]).max()))
        assert normwise(x[:, k] * s, np.linalg.solve(A[0], B[0, :, k] * s)) <= 100 * n * EPS


@pytest.mark.parametrize("ns", [[17, 64, 33, 48, 20], [65, 128, 40, 100], [200, 17, 512, 300, 64]])
def test_ragged_factor_is_the_uniform_one(gpu, ns):
    """The ragged solves factor with the same steps as the uniform calls: L is the same bits, whichever
    kernel a size goes to, an odd batch among them."""
    import torch

    from blast_gb300.ragged import Packed, PosvPlan

    rng = np.random.default_rng(sum(ns))
    As = [spd(rng, n) for n in ns]
    A, B, X, L = Packed(ns, ns, "cuda"), Packed(ns, [2] * len(ns), "cuda"), Packed(ns, [2] * len(ns), "cuda"), Packed(
        ns, ns, "cuda")
    A.fill_from(As)
    B.fill_from([rng.standard_normal((n, 2)) for n in ns])
    plan = PosvPlan(A, B, X, L)
    plan.run()
    torch.cuda.synchronize()
    assert not plan.results()[0].any()
    for n, Ah, Lg, Bh, Xg in zip(ns, As, L.to_list(), B.to_list(), X.to_list()):
        P = to_dev(Ah[None])
        gpu.potrf(P, P)
        torch.cuda.synchronize()
        assert np.array_equal(np.tril(Lg), np.tril(P.cpu().numpy()[0])), n
        assert normwise(Xg, np.linalg.solve(Ah, Bh)) <= 100 * n * EPS, n


@pytest.mark.parametrize("ns", [[3], [128, 1, 97, 0, 5, 66, 33], [65, 64, 63, 32, 31, 4, 2, 1], [127, 126, 125, 8, 100, 7, 0, 0, 16]])
def test_ragged_solves_share_a_warp(gpu, ns):
    """The backward substitutions of up to eight instances run in one warp: full and partial groups, sizes
    of all remainders by 4, instances without rows, and instances with no or several right-hand sides."""
    import torch

    from blast_gb300.autograd import spd_solve_packed
    from blast_gb300.ragged import Packed, PosvPlan

    rng = np.random.default_rng(sum(ns) + len(ns))
    rs = [(3 * i + 1) % 5 for i in range(len(ns))]
    As = [spd(rng, n) for n in ns]
    Bs = [rng.standard_normal((n, r)) for n, r in zip(ns, rs)]
    A, B, X, L = Packed(ns, ns, "cuda"), Packed(ns, rs, "cuda"), Packed(ns, rs, "cuda"), Packed(ns, ns, "cuda")
    A.fill_from(As)
    B.fill_from(Bs)
    plan = PosvPlan(A, B, X, L)
    plan.run()
    torch.cuda.synchronize()
    assert not plan.results()[0].any()
    a = A.buf.clone().requires_grad_()
    b = B.buf.clone().requires_grad_()
    x = spd_solve_packed(a, b, np.array(ns), np.array(rs))
    x.sum().backward()
    ga, gb, oa, ob = a.grad.cpu().numpy(), b.grad.cpu().numpy(), 0, 0
    for n, r, Ah, Bh, Xg in zip(ns, rs, As, Bs, X.to_list()):
        if n * r:
            want, g = np.linalg.solve(Ah, Bh), np.linalg.solve(Ah, np.ones((n, r)))
            assert normwise(Xg, want) <= 100 * n * EPS, n
            assert normwise(gb[ob:ob + n * r].reshape((n, r), order="F"), g) <= 100 * n * EPS, n
            assert normwise(ga[oa:oa + n * n].reshape((n, n), order="F"), -0.5 * (g @ want.T + want @ g.T)) <= 200 * n * EPS, n
        oa, ob = oa + n * n, ob + n * r


@pytest.mark.parametrize("n", [17, 24, 40, 48, 60, 61, 64])
@pytest.mark.parametrize("nrhs", [0, 3])
def test_host_order_is_the_device_order(gpu, n, nrhs):
    """The entry for operands in host memory reads and writes in another order: same bits, at leading
    dimensions that put the columns off the lines, with a pivot that is not positive, NaN and infinity."""
    import torch

    from blast_gb300 import _lib

    rng = np.random.default_rng(n + nrhs)
    A = spd_batch(rng, 5, n)
    A[1, n // 2, n // 2] = -1.0
    A[2, n - 1, 3] = np.nan
    A[3, n - 2, 1] = np.inf
    ld = n + 3
    dA, dB = to_dev(A, ld=ld), to_dev(rng.standard_normal((5, n, max(nrhs, 1))), ld=ld)
    L, X = gpu.col_major((5,), n, n, "cuda").zero_(), gpu.col_major((5,), n, max(nrhs, 1), "cuda").zero_()
    info = gpu.posv(dA, L, dB, X) if nrhs else gpu.potrf(dA, L)
    hL, hX = torch.zeros(5 * ld * n).double().pin_memory(), torch.zeros(5 * ld * n).double().pin_memory()
    wL, wX = torch.empty(5 * n * n, device="cuda").double(), torch.empty(5 * n * n, device="cuda").double()
    hinfo = torch.zeros(5, dtype=torch.int32, device="cuda")
    _lib.call("blastgpu_dposv_mirror_strided", n, nrhs, dA.data_ptr(), ld, dA.stride(0), dB.data_ptr(), ld,
              dB.stride(0), hL.data_ptr(), ld, ld * n, hX.data_ptr(), ld, ld * n, wL.data_ptr(), wX.data_ptr(),
              hinfo.data_ptr(), 5, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(hinfo, info.to(hinfo.dtype))
    gotL = np.tril(hL.numpy().reshape(5, n, ld).transpose(0, 2, 1)[:, :n])
    assert np.array_equal(gotL, np.tril(L.cpu().numpy()), equal_nan=True)
    assert not hL.numpy().reshape(5, n, ld)[:, :, n:].any()
    if nrhs:
        gotX = hX.numpy().reshape(5, n, ld)[:, :nrhs].transpose(0, 2, 1)[:, :n]
        assert np.array_equal(gotX, X.cpu().numpy(), equal_nan=True)
