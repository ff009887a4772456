"""GPU check of the EM targets and the Adam move over the update kernels' ways to split the
rows: small launches with a thread per P element (blocks of 128 / K rows) and a thread or a warp per
Q row, larger ones and larger K with a thread or a warp per row."""
import numpy as np
import pytest
import torch

from oracle import em_oracle as orc

pytestmark = pytest.mark.gpu

LR, B1, B2, EPS, STEP = 0.005, 0.80, 0.88, 1e-8, 3


def adam(x, target, m, v):
    d = target - x
    m, v = B1 * m + (1 - B1) * d, B2 * v + (1 - B2) * d * d
    x = x + LR * (m / (1 - B1 ** STEP)) / (np.sqrt(v / (1 - B2 ** STEP)) + EPS)
    return np.clip(x, 1e-5, 1 - 1e-5), m, v


# few partials (a thread per row), many partials of few samples or few SNPs (a warp per row; the
# last block partly empty), K = 1, a K that leaves threads of a block idle, past 32, and 64
@pytest.mark.parametrize("N,M,K", [(1, 1, 1), (105, 91, 7), (33, 2049, 1), (33, 2049, 7), (65, 4097, 16),
                                   (9000, 130, 7), (9000, 129, 33), (41, 2049, 33), (41, 2049, 64)])
def test_update_matches_the_oracle(cuda, N, M, K):
    from adamixture_b200 import ops

    rng = np.random.default_rng(N + M + K)
    G = rng.choice(4, size=(M, N), p=[0.3, 0.35, 0.3, 0.05]).astype(np.uint8)
    P = rng.uniform(0.05, 0.95, size=(M, K))
    Q = rng.dirichlet(np.ones(K), size=N)
    # moments away from zero: the move then depends on a statistic's error by LR (1 - B1) / sqrt(v) at
    # most. Statistics agree to 1e-10 relative, so targets in [0, 1] to 2e-10 and the moments to
    # 1e-10, and P and Q to 0.005 x 0.41 x 2e-10 / sqrt(1.1) < 1e-12.
    mom = [rng.uniform(-0.1, 0.1, (M, K)), rng.uniform(0.5, 1, (M, K)),
           rng.uniform(-0.1, 0.1, (N, K)), rng.uniform(0.5, 1, (N, K))]
    A, B, T, _ = orc.em_stats(G, P, Q)
    tp = P * A / np.maximum((A - B) * P + B, 1e-5)
    q_bat = 2.0 * (G != 3).sum(0).astype(np.float64)
    e = Q * T / np.maximum(q_bat, 1e-5)[:, None]
    P1, mP, vP = adam(P, tp, mom[0], mom[1])
    Q1, mQ, vQ = adam(Q, e / np.maximum(e.sum(1, keepdims=True), 1e-5), mom[2], mom[3])
    Q1 /= Q1.sum(1, keepdims=True)

    def dev(x):
        return torch.from_numpy(np.ascontiguousarray(x)).cuda()

    Pd, Qd, (dmP, dvP, dmQ, dvQ) = dev(P), dev(Q), [dev(x) for x in mom]
    P32, Q32 = Pd.float(), Qd.float()
    ops.em_adam_iteration(dev(orc.pack(G)), Pd, Qd, P32, Q32, dmP, dvP, dmQ, dvQ, dev(q_bat), M, float(STEP), LR, B1,
                          B2, EPS, "f64")
    for got, ref, bar in ((Pd, P1, 1e-12), (Qd, Q1, 1e-12), (dmP, mP, 1e-10), (dvP, vP, 1e-10), (dmQ, mQ, 1e-10),
                          (dvQ, vQ, 1e-10)):
        assert np.abs(got.cpu().numpy() - ref).max() <= bar
    assert torch.equal(P32, Pd.float()) and torch.equal(Q32, Qd.float())


# at the line between the two forms, 592 blocks and one more: 8 rows of K = 15 a block, 32 blocks of Q
@pytest.mark.parametrize("M", [560 * 8, 560 * 8 + 1])
def test_both_forms_at_their_line(cuda, M):
    test_update_matches_the_oracle(cuda, 128, M, 15)
