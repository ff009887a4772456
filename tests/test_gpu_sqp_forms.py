"""GPU check that the register form of the QP solves (K <= 16) gives the shared-memory form's
(larger K) results to the last bit, in the box: a problem of K parameters beside others that
are free and at their optimum is the same problem, and with 17 parameters in all the other form
solves it. Half of the problems are nearly singular, where every step's rounding shows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 2, 4, 5, 8, 9, 12, 13, 16])
def test_register_form_equals_shared_form(cuda, K):
    from adamixture_b200 import ops

    rng = np.random.default_rng(K)
    n, W = 400, 17
    A = rng.normal(size=(n, K, K + 2))
    A[::2, :, 2:] = 0.0
    H = np.zeros((n, W, W))
    H[:, :K, :K] = A @ A.transpose(0, 2, 1) + 1e-7 * np.eye(K)
    H[:, range(K, W), range(K, W)] = 1.0
    X = np.full((n, W), 0.5)
    X[:, :K] = np.clip(rng.dirichlet(np.full(K, 0.5), size=n), 1e-5, 1 - 1e-5)
    r = np.zeros((n, W))
    r[:, :K] = rng.normal(size=(n, K)) * np.where(np.arange(n) % 2, 3.0 * K, 1.0)[:, None]

    def dev(x):
        return torch.from_numpy(np.ascontiguousarray(x)).cuda()

    small = ops.sqp_solve_p(dev(H[:, :K, :K]), dev(r[:, :K]), dev(X[:, :K]), n, K)
    large = ops.sqp_solve_p(dev(H), dev(r), dev(X), n, W)
    assert torch.equal(small, large[:, :K]) and torch.equal(large[:, K:], torch.full_like(large[:, K:], 0.5))
