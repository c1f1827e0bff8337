"""Both sides of every rule by which a uniform Cholesky call chooses its kernels (size, batch, right-hand sides): results
against the oracle, and the calls that are defined as a sequence of others against that sequence.

Tolerances are the library's: 10 n eps normwise for a factor, 100 n eps for a solution.
"""
import numpy as np
import pytest

from helpers import EPS, normwise, spd, spd_batch, to_dev

pytestmark = pytest.mark.gpu


def tiled(gpu, small, batch):
    """`batch` instances that repeat the ones in `small`, on the GPU."""
    import torch

    t = to_dev(small)
    out = gpu.col_major((batch,), small.shape[1], small.shape[2], "cuda")
    out.copy_(t.repeat(-(-batch // len(small)), 1, 1)[:batch])
    return out, [int(b) for b in np.unique(np.linspace(0, batch - 1, 5).astype(int))]


CASES = [(16, 3, 5), (17, 8, 3000), (17, 8, 9000), (20, 0, 9000), (21, 0, 9000), (21, 2, 31000), (25, 4, 9000), (27, 0, 31000),
         (28, 8, 9000), (30, 8, 31000), (28, 8, 31000), (45, 9, 9000), (48, 8, 31000), (65, 1, 4000), (65, 1, 5000), (71, 3, 6500),
         (71, 0, 7000), (72, 1, 7000), (100, 2, 300)]


@pytest.mark.parametrize("n,nrhs,batch", CASES)
def test_posv_either_side(gpu, oracle_lib, n, nrhs, batch):
    import torch

    rng = np.random.default_rng(n * 7 + nrhs)
    m = 7
    A, B = spd_batch(rng, m, n), rng.standard_normal((m, n, max(nrhs, 1)))
    A[3, 2, 2] = -1.0
    dA, some = tiled(gpu, A, batch)
    dB, _ = tiled(gpu, B, batch)
    L, X = gpu.col_major((batch,), n, n, "cuda").zero_(), gpu.col_major((batch,), n, max(nrhs, 1), "cuda")
    info = gpu.posv(dA, L, dB, X) if nrhs else gpu.potrf(dA, L)
    torch.cuda.synchronize()
    want = torch.zeros(batch, dtype=info.dtype)
    want[3::m] = 3
    assert torch.equal(info.cpu(), want)
    Lr, Xr, _ = oracle_lib.posv_batch(A, B)
    for b in some:
        if b % m != 3:
            assert normwise(np.tril(L[b].cpu().numpy()), np.tril(Lr[b % m])) <= 10 * n * EPS
            assert not nrhs or normwise(X[b].cpu().numpy(), Xr[b % m]) <= 100 * n * EPS


@pytest.mark.parametrize("n,nrhs,batch", [(64, 1, 50), (65, 1, 3900), (65, 1, 4100), (65, 8, 490), (65, 8, 510), (65, 16, 490), (128, 9, 2200),
                                          (128, 9, 2400), (160, 2, 5), (512, 1, 2), (513, 1, 2)])
def test_potrs_either_side(gpu, oracle_lib, n, nrhs, batch):
    import torch

    rng = np.random.default_rng(n + nrhs)
    A, B = spd_batch(rng, 2, n), rng.standard_normal((2, n, nrhs))
    Lr, Xr, _ = oracle_lib.posv_batch(A, B)
    dL, some = tiled(gpu, np.tril(Lr), batch)
    dB, _ = tiled(gpu, B, batch)
    X = gpu.col_major((batch,), n, nrhs, "cuda")
    gpu.potrs(dL, dB, X)
    torch.cuda.synchronize()
    for b in some:
        assert normwise(X[b].cpu().numpy(), Xr[b % 2]) <= 100 * n * EPS


@pytest.mark.parametrize("n,batch", [(16, 3), (17, 3), (18, 9000), (24, 9000), (33, 31000), (64, 40), (66, 9000), (70, 10)])
def test_syrk_potrf_is_syrk_then_potrf(gpu, oracle_lib, n, batch):
    """chol(0.5 C + 0.75 A A^T) on the sizes and batches that potrf sends different ways: the same bits as the two calls."""
    import torch

    rng = np.random.default_rng(n)
    A, C = rng.uniform(-1, 1, (5, n, 9)), np.stack([spd(rng, n) for _ in range(5)])
    dA, some = tiled(gpu, A, batch)
    dC, _ = tiled(gpu, C, batch)
    D, S = gpu.col_major((batch,), n, n, "cuda").zero_(), gpu.col_major((batch,), n, n, "cuda").zero_()
    info = gpu.syrk_potrf(0.75, dA, 0.5, dC, D)
    gpu.syrk_lower(0.75, dA, 0.5, dC, S)
    info2 = gpu.potrf(S, S)
    torch.cuda.synchronize()
    assert not info.any() and not info2.any() and torch.equal(D, S)
    for b in some:
        ref = np.zeros((n, n), order="F")
        oracle_lib.potrf(np.asfortranarray(0.5 * C[b % 5] + 0.75 * A[b % 5] @ A[b % 5].T), ref)
        assert normwise(np.tril(D[b].cpu().numpy()), np.tril(ref)) <= 10 * n * EPS


@pytest.mark.parametrize("n,nrhs,batch", [(24, 8, 300), (24, 8, 20000), (31, 3, 20000), (65, 2, 40), (96, 8, 33), (130, 1, 64)])
def test_host_batches_either_side(gpu, oracle_lib, n, nrhs, batch):
    """The entry for host memory, which chooses by other rules than the device call and solves on threads above n = 64:
    the same to rounding."""
    import torch

    from blast_gb300.host import PosvHostPipeline, pinned_col_major

    rng = np.random.default_rng(n)
    A, B = spd_batch(rng, 6, n), rng.standard_normal((6, n, nrhs))
    hA, hB, hL, hX = (pinned_col_major(batch, n, c) for c in (n, nrhs, n, nrhs))
    hA.copy_(torch.from_numpy(A).repeat(-(-batch // 6), 1, 1)[:batch])
    hB.copy_(torch.from_numpy(B).repeat(-(-batch // 6), 1, 1)[:batch])
    hL.zero_()
    info = torch.full((batch,), -1, dtype=torch.int32).pin_memory()
    PosvHostPipeline(n, nrhs, batch, "cuda", transport="mirror").run(hA, hB, hL, hX, info)
    torch.cuda.synchronize()
    assert not info.any()
    Lr, Xr, _ = oracle_lib.posv_batch(A, B)
    for b in np.unique(np.linspace(0, batch - 1, 5).astype(int)):
        assert normwise(np.tril(hL[b].numpy()), np.tril(Lr[b % 6])) <= 10 * n * EPS
        assert normwise(hX[b].numpy(), Xr[b % 6]) <= 100 * n * EPS
