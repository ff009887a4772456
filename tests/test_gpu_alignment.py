"""GPU checks that the alignment of the packed matrix (the sample count modulo 16 and the
address it starts at) does not change a result: every alignment reads the same genotypes."""
import numpy as np
import pytest
import torch

from oracle import em_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(cuda):
    from adamixture_b200 import ops as _ops

    return _ops


def placed(packed, offset):
    """The packed matrix `offset` bytes into a buffer whose other bytes are arbitrary codes."""
    n = packed.size
    buf = torch.randint(0, 256, (n + 64,), dtype=torch.uint8, device="cuda")
    buf[offset:offset + n] = torch.from_numpy(packed.reshape(-1)).cuda()
    return buf[offset:offset + n].view(packed.shape)


def cohort(N, M, K, seed):
    rng = np.random.default_rng(seed)
    G = rng.choice(4, size=(M, N), p=[0.3, 0.35, 0.3, 0.05]).astype(np.uint8)
    P = np.clip(rng.beta(0.8, 0.8, size=(M, K)), 1e-5, 1 - 1e-5)
    Q = rng.dirichlet(np.full(K, 0.5), size=N)
    return G, P, Q


@pytest.mark.parametrize("prec", ["f16", "bf16"])
@pytest.mark.parametrize("N,M", [(16, 40), (272, 1100), (17, 900), (131, 1799), (255, 130)])
def test_tensor_core_stats_do_not_depend_on_alignment(ops, prec, N, M):
    # N = 16, 272: the aligned kernel at offset 0 against the unaligned one; tiles that end
    # at, before and past the 128-sample and 896-SNP edges
    G, P, Q = cohort(N, M, 9, N + M)
    packed = orc.pack(G)
    P32, Q32 = torch.from_numpy(P).float().cuda(), torch.from_numpy(Q).float().cuda()
    ref = ops.em_stats(placed(packed, 0), P32, Q32, M, prec)
    for off in (1, 6, 8, 15):
        got = ops.em_stats(placed(packed, off), P32, Q32, M, prec)
        for g, r in zip(got, ref):
            assert torch.equal(g, r), off
