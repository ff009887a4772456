"""GPU checks of the tensor-core sweep where a CTA walks several sample tiles: both operand
formats, packed rows that start 16-byte aligned and not, 7 SNP tiles a CTA (the last CTA
fewer) and one, whose T buffers change every step. Bars: relative Frobenius error of each
statistic, 1e-3 (FP16) and 4e-3 (BF16), those of the other tests of this sweep; a lost or doubled
tile of T would show as at least 1/sqrt(tiles) > 2e-2."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def stats(g, P, Q):
    A, B, T = torch.empty_like(P), torch.empty_like(P), torch.zeros_like(Q)
    for j in range(0, g.shape[0], 2048):
        e = slice(j, j + 2048)
        h = (P[e] @ Q.T).clamp_(1e-5, 1 - 1e-5)
        seen = g[e] != 3
        a, b = g[e].double() * seen / h, (2.0 - g[e].double()) * seen / (1 - h)
        A[e], B[e] = a @ Q, b @ Q
        T += a.T @ P[e] + b.T @ (1 - P[e])
    return A, B, T


# 2 to 5 tiles a CTA: sample tiles over the splits that the plan may take (592 to 1,184 for
# one SNP block; 20 to 88 for 30)
@pytest.mark.parametrize("N,M,K", [(307_200, 100, 8), (307_203, 128, 11), (11_520, 26_000, 10), (11_531, 26_003, 16)])
@pytest.mark.parametrize("prec,bar", [("f16", 1e-3), ("bf16", 4e-3)])
def test_several_sample_tiles(cuda, N, M, K, prec, bar):
    from adamixture_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(N + M)
    g = torch.randint(0, 4, ((M + 3) // 4 * 4, N), generator=gen, device="cuda", dtype=torch.uint8)
    g[M:] = 0
    q = g.view(-1, 4, N)
    packed = (q[:, 0] | q[:, 1] << 2 | q[:, 2] << 4 | q[:, 3] << 6).contiguous()
    P = (0.05 + 0.9 * torch.rand((M, K), generator=gen, device="cuda")).contiguous()
    Q = torch.softmax(2 * torch.randn((N, K), generator=gen, device="cuda"), 1).contiguous()
    want = stats(g[:M], P.double(), Q.double())
    for got, ref in zip(ops.em_stats(packed, P, Q, M, prec), want):
        assert float((got - ref).norm() / ref.norm()) <= bar
