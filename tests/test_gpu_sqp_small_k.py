"""GPU checks of the per-K gradient/Hessian kernels and the register SQP solves (K <= 16):
every K, row tiles of 64 and chunks of 32 that end early, several splits, packed rows at any
address, against the float64 restatement. Bars: those of the other tests of these passes
(1e-9; sums of up to a few hundred terms, each rounded at 2^-53, stay far below)."""
import numpy as np
import pytest
import torch

from oracle import em_oracle as orc
from oracle import solvers as osv

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(cuda):
    from adamixture_b200 import ops as _ops

    return _ops


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def placed(packed, offset):
    n = packed.size
    buf = torch.randint(0, 256, (n + 64,), dtype=torch.uint8, device="cuda")
    buf[offset:offset + n] = torch.from_numpy(packed.reshape(-1)).cuda()
    return buf[offset:offset + n].view(packed.shape)


@pytest.mark.parametrize("K", range(1, 18))
def test_gradients_and_hessians(ops, K):
    rng = np.random.default_rng(K)
    for N, M in ((1, 3), (33, 65), (64, 32), (129, 203)):
        G = rng.choice(4, size=(M, N), p=[0.3, 0.35, 0.3, 0.05]).astype(np.uint8)
        P = np.clip(rng.beta(0.8, 0.8, size=(M, K)), 1e-5, 1 - 1e-5)
        Q = np.clip(rng.dirichlet(np.full(K, 0.5), size=N), 1e-5, 1 - 1e-5)
        Q /= Q.sum(1, keepdims=True)
        packed = orc.pack(G)
        want = osv.grad_hess_q(G, P, Q), osv.grad_hess_p(G, P, Q)
        for off in (0, 5):
            Gp = placed(packed, off)
            got = ops.grad_hess_q(Gp, dev(P), dev(Q), M), ops.grad_hess_p(Gp, dev(P), dev(Q), M)
            for side in (0, 1):
                for x, ref in zip(got[side], want[side]):
                    np.testing.assert_allclose(x.cpu().numpy(), ref, rtol=1e-9, atol=1e-9 * np.abs(ref).max())


@pytest.mark.parametrize("K", [1, 2, 4, 5, 8, 9, 12, 13, 16])
def test_register_solves(ops, K):
    # both sides of every register-tableau width. Rows whose solution the oracle itself changes
    # under a relative change of 1e-13 in the Hessian (active sets that cycle to the iteration
    # limit) say nothing; the others are stable, and most rows are
    rng = np.random.default_rng(100 + K)
    n = 70
    A = rng.normal(size=(n, K, 2 * K + 2))
    H = A @ A.transpose(0, 2, 1) + np.eye(K)
    X = np.clip(rng.dirichlet(np.full(K, 0.7), size=n), 1e-5, 1 - 1e-5)
    X /= X.sum(1, keepdims=True)
    r = rng.normal(size=(n, K)) * 3.0 * K
    v = np.linalg.svd(np.ones((1, K)), full_matrices=True)[2].T.copy()
    H2 = H * (1.0 + 1e-13 * rng.choice([-1.0, 1.0], size=H.shape))
    H2 = 0.5 * (H2 + H2.transpose(0, 2, 1))
    for got, ref, ref2 in (
            (ops.sqp_solve_q(dev(H), dev(r), dev(X), dev(v), n, K), osv.sqp_solve_q(H, r, X, v), osv.sqp_solve_q(H2, r, X, v)),
            (ops.sqp_solve_p(dev(H), dev(r), dev(X), n, K), osv.sqp_solve_p(H, r, X), osv.sqp_solve_p(H2, r, X))):
        stable = np.abs(ref - ref2).max(1) < 1e-10
        assert stable.mean() > 0.5
        np.testing.assert_allclose(got.cpu().numpy()[stable], ref[stable], atol=1e-9)
