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


@pytest.mark.parametrize("N,M", [(1, 1), (3, 9), (15, 4), (16, 61), (17, 30), (511, 258), (528, 33), (4097, 70),
                                 (9001, 1003)])
def test_bed_and_statistics_do_not_depend_on_alignment(ops, N, M):
    # BED decode (unit and segment edges, a flipped and an unflipped matrix), frequencies (warp
    # and block per row) and per-sample counts (nibble, byte and 32-bit sums) at every kind
    # of start address
    for p in ([0.5, 0.25, 0.15, 0.1], [0.1, 0.2, 0.6, 0.1]):
        G = np.random.default_rng(N * M).choice(4, size=(M, N), p=p).astype(np.uint8)
        code = np.array([3, 2, 0, 1], dtype=np.uint8)[G]
        pad = np.full((M, -N % 4), 1, dtype=np.uint8)      # what the padding holds must not matter
        c = np.concatenate([code, pad], axis=1).reshape(M, -1, 4)
        bed = c[..., 0] | c[..., 1] << 2 | c[..., 2] << 4 | c[..., 3] << 6
        seen = G != 3
        if seen.any() and (G * seen).sum() / (2.0 * seen.sum()) >= 0.5:
            G = np.where(G == 0, 2, np.where(G == 2, 0, G)).astype(np.uint8)
        packed = orc.pack(G)
        cnt, tot = seen.sum(1), (G * seen).sum(1)
        f = np.where(cnt > 0, tot.astype(np.float32) / np.float32(2) / np.maximum(cnt, 1).astype(np.float32), 0)
        for off in (0, 1, 2, 7, 13):
            assert torch.equal(ops.bed_to_packed(placed(bed, off), N, M).cpu(), torch.from_numpy(packed)), off
            P = placed(packed, off)
            np.testing.assert_allclose(ops.allele_frequency(P, M).cpu().numpy(), f, rtol=2.0 ** -22, atol=0)
            assert np.array_equal(ops.sample_counts(P, M).cpu().numpy(), 2.0 * seen.sum(0))
            assert np.array_equal(ops.sample_het_counts(P, M).cpu().numpy(), (G == 1).sum(0))


def float32_bounds(G, P, Q):
    """Per-element error bounds of float32 statistics, u = 2^-24: h has K roundings (its terms
    are positive), 1 - rec inherits h's absolute error, the ratios and weights add a few more
    roundings, and a sum of n positive terms at most n; T's two parts are bounded by the sum
    of their magnitudes."""
    u, K, (M, N) = 2.0 ** -24, P.shape[1], G.shape
    h = np.clip(P @ Q.T, 1e-5, 1 - 1e-5)
    seen = G != 3
    a, b = np.where(seen, G / h, 0.0), np.where(seen, (2.0 - G) / (1 - h), 0.0)
    ea, eb = a * u * (K + 8), b * u * (K * h / (1 - h) + 8)
    A = ea @ Q + a @ Q * N * u
    B = eb @ Q + b @ Q * N * u
    T = (ea + eb).T @ P + eb.sum(0)[:, None] + ((a + b).T @ P + b.sum(0)[:, None]) * M * u
    return A, B, T


@pytest.mark.parametrize("K", range(1, 9))
def test_float32_sweep_of_small_k(ops, K):
    # every K with the packed-pair kernel: samples and SNPs that end inside a thread's 8, a
    # packed quad and a chunk, several sub-tiles and blocks, any start address
    for N, M in ((5, 3), (1024, 33), (1025, 64), (2051, 517)):
        G, P, Q = cohort(N, M, K, K * N + M)
        packed = orc.pack(G)
        P32, Q32 = torch.from_numpy(P).float().cuda(), torch.from_numpy(Q).float().cuda()
        Pd, Qd = P32.double().cpu().numpy(), Q32.double().cpu().numpy()
        want = orc.em_stats(G, Pd, Qd)[:3]
        ref = ops.em_stats(placed(packed, 0), P32, Q32, M, "f32")
        for g, w, tol in zip(ref, want, float32_bounds(G, Pd, Qd)):
            assert (np.abs(g.cpu().numpy() - w) <= tol).all()
        for off in (1, 6, 11):
            got = ops.em_stats(placed(packed, off), P32, Q32, M, "f32")
            assert all(torch.equal(g, r) for g, r in zip(got, ref)), off


@pytest.mark.parametrize("N,M,K", [(20_000, 48, 5), (30_001, 130, 16), (105, 8451, 7), (2048, 1300, 3), (1, 900, 2)])
def test_partials_of_few_rows(ops, N, M, K):
    # many partials for few P rows (wide, short matrices) or few Q rows: 32 threads a row, and the
    # small cohorts' partition. Float64 statistics: a sum of n positive terms is within n 2^-53
    # of the exact one, its terms within a few roundings and h's K 2^-53 over 1 - h
    G, P, Q = cohort(N, M, K, N + M)
    P, Q = np.clip(P, 0.01, 0.99), Q / Q.sum(1, keepdims=True)
    want = orc.em_stats(G, P, Q)[:3]
    got = ops.em_stats(placed(orc.pack(G), 0), torch.from_numpy(P).cuda(), torch.from_numpy(Q).cuda(), M, "f64")
    for g, w, n in zip(got, want, (N, N, 2 * M)):
        tol = (n + 100 * (K + 8)) * 2.0 ** -53
        np.testing.assert_allclose(g.cpu().numpy(), w, rtol=tol, atol=100 * tol)


@pytest.mark.parametrize("K", [1, 2, 5, 8, 10, 11, 16])
def test_float32_loglik_of_small_k(ops, K):
    # the packed-pair form: ragged samples, quads and chunks, exponents moved every 4 quads, any
    # start address. h has K roundings of 2^-24 and 1 - h inherits them; a pair of factors
    # rounds three times more
    for N, M in ((1, 1), (9, 35), (1025, 70), (2050, 517)):
        G, P, Q = cohort(N, M, K, K + N * M)
        packed = orc.pack(G)
        P32, Q32 = torch.from_numpy(P).float().cuda(), torch.from_numpy(Q).float().cuda()
        Pd, Qd = P32.double().cpu().numpy(), Q32.double().cpu().numpy()
        h = np.clip(Pd @ Qd.T, 1e-10, 1 - 1e-10)
        seen = G != 3
        g = np.where(seen, G, 0).astype(float)
        L = np.where(seen, g * np.log(h) + (2 - g) * np.log1p(-h), 0.0).sum()
        tol = 2.0 ** -24 * np.where(seen, g * K + (2 - g) * (K * h / (1 - h) + 1) + 2, 0.0).sum() + 1e-12 * abs(L)
        ref = ops.loglik_device(placed(packed, 0), P32, Q32, M, "f32")
        assert abs(float(ref) - L) <= tol
        for off in (1, 6, 15):
            assert torch.equal(ops.loglik_device(placed(packed, off), P32, Q32, M, "f32"), ref), off


@pytest.mark.parametrize("K", [1, 4, 7, 8, 10, 16])
def test_float64_sweep_and_loglik_do_not_depend_on_alignment(ops, K):
    # the aligned kernels (N % 8 = 0 at offset 0) against the word loads at every other address,
    # and ragged cohorts at all of them; the folded check too
    for N, M in ((256, 40), (264, 130), (105, 70), (515, 517)):
        G, P, Q = cohort(N, M, K, K + N + M)
        packed = orc.pack(G)
        Pd, Qd = torch.from_numpy(P).cuda(), torch.from_numpy(Q).cuda()
        ref = ll = None
        for off in (0, 1, 6, 8, 13):
            X = placed(packed, off)
            got = ops.em_stats(X, Pd, Qd, M, "f64")
            L = ops.loglik_device(X, Pd, Qd, M, "f64")
            ws = ops.em_workspace(M, N, K, "f64", X.device)
            ops.em_sweep_loglik(X, Pd, Qd, M, ws)
            assert torch.equal(ops.em_loglik_from_sweep(ws, M, N, K), L)
            if ref is None:
                ref, ll = got, L
                want = orc.em_stats(G, P, Q)[:3]
                assert all(np.abs(g.cpu().numpy() - w).max() <= 1e-11 * np.abs(w).max() for g, w in zip(got, want))
                assert abs(float(L) - orc.loglik(G, P, Q)) <= 1e-12 * abs(float(L))
            assert all(torch.equal(g, r) for g, r in zip(got, ref)) and torch.equal(L, ll), off
