"""GPU check of the float64 sweep's clamp of h on values that are not finite: it is
fmin(fmax(h, 1e-5), 1 - 1e-5), so a NaN goes to the lower bound, as -infinity does, and
+infinity to the upper. The SNPs' A and B stay finite then and are compared with the oracle's."""
import numpy as np
import pytest
import torch

from oracle import em_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [3, 7, 10, 16])   # both shared-memory layouts' widths
@pytest.mark.parametrize("N", [64, 77])         # whole rows of 8 samples, and not
def test_clamp_of_nan_and_infinities(cuda, K, N):
    from adamixture_b200 import ops

    rng = np.random.default_rng(K + N)
    M = 70
    G = rng.choice(4, size=(M, N), p=[0.3, 0.35, 0.3, 0.05]).astype(np.uint8)
    P = rng.uniform(0.05, 0.95, size=(M, K))
    Q = rng.dirichlet(np.ones(K), size=N).clip(1e-3)
    odd = {5: np.nan, 18: np.inf, 33: -np.inf}
    A, B, T, _ = orc.em_stats(G, P, Q)
    for j, v in odd.items():
        h = 1.0 - 1e-5 if v == np.inf else 1e-5
        seen = G[j] != 3
        A[j] = (np.where(seen, G[j], 0) / h) @ Q
        B[j] = (np.where(seen, 2.0 - G[j], 0) / (1.0 - h)) @ Q
        P[j, K // 2] = v

    def dev(x):
        return torch.from_numpy(np.ascontiguousarray(x)).cuda()

    gotA, gotB, _ = ops.em_stats(dev(orc.pack(G)), dev(P), dev(Q), M, "f64")
    np.testing.assert_allclose(gotA.cpu().numpy(), A, rtol=1e-10)
    np.testing.assert_allclose(gotB.cpu().numpy(), B, rtol=1e-10)
