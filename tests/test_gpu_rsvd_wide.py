"""GPU checks of the randomized-SVD products on columns of widely spread entries: one entry is 1,
the others are at a scale s below it, and the outputs looked at are those that do not meet the
large one (it is missing there), which float32 sums hold to the scale of the small ones.

Tolerance, against float64: down to s = 2^-34 the second level rounds an entry by at most 2^-61
of the largest (half a quantum of 2^-60 2^e, the largest in [2^e, 2^(e+1))), times an entry of the
centred matrix of at most 2 (cols: codes, flags and constant, 8); then the rounding of the
result to float32 and of the float64 sums that end it: cols adds three terms of up to 3 times
the large entry that cancel, 2^-50 with room. Below that an entry is summed in float32: n
roundings of 2^-24 of a partial sum. Float32 sums of entries at 2^-34 are bound to 2^-58 n^2 only."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(cuda):
    from adamixture_b200 import ops as _ops

    return _ops


def cohort(N, M, seed, spike, cols):
    """Genotypes whose sample `spike` (cols: SNP `spike`) is missing in every other SNP (sample)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    g = torch.randint(0, 4, ((M + 3) // 4 * 4, N), generator=gen, device="cuda", dtype=torch.uint8)
    if cols:
        g[spike, ::2] = 3
    else:
        g[::2, spike] = 3
    g[M:] = 0
    q = g.view(-1, 4, N)
    packed = (q[:, 0] | q[:, 1] << 2 | q[:, 2] << 4 | q[:, 3] << 6).contiguous()
    f = 0.05 + 0.45 * torch.rand(M, generator=gen, device="cuda")
    X = (g[:M].double() - 2.0 * f.double()[:, None]).masked_fill_(g[:M] == 3, 0.0)
    return packed, f, X, gen


# several CTAs a row tile; one CTA a row tile and several blocks; two passes
@pytest.mark.parametrize("N,M,L", [(2000, 301, 4), (1003, 40011, 20), (700, 900, 30)])
@pytest.mark.parametrize("side", ["rows", "cols"])
def test_outputs_that_meet_small_entries_only(ops, N, M, L, side):
    cols = side == "cols"
    n, spike = (M, 5) if cols else (N, 7)
    G, f, X, gen = cohort(N, M, N + L, spike, cols)
    product, A = (ops.rsvd_cols, X.T) if cols else (ops.rsvd_rows, X)
    scales = [1.0, 2.0 ** -10, 2.0 ** -20, 2.0 ** -34, 2.0 ** -60]
    F = torch.randn((n, L), generator=gen, device="cuda")
    F *= torch.tensor([scales[c % 5] for c in range(L)], device="cuda")
    F[spike] = 1.0
    got, F64 = product(G, f, F, M), F.double()
    ref, mag = A @ F64, A.abs() @ F64.abs()
    for c in range(L):
        s = scales[c % 5]
        tol = 2.0 ** -23 * ref[:, c].abs() + (2.0 ** -50 * float(F64[:, c].abs().max()) if cols else 0.0)
        tol = tol + (n * 2.0 ** -24 * mag[:, c] if s < 2.0 ** -34 else (8 if cols else 2) * n * 2.0 ** -61 * float(F64[:, c].abs().max()))
        if s == 1.0:   # not wide: the first level alone
            tol = tol + 8 * n * 2.0 ** -30 * float(F64[:, c].abs().max())
        err = (got[:, c].double() - ref[:, c]).abs()
        assert bool((err <= tol).all()), (c, s, float((err / tol).max()))
    # a column's values do not depend on its neighbours, nor on how they are split into passes
    alone = torch.cat([product(G, f, F[:, c:c + 1].contiguous(), M) for c in range(L)], 1)
    assert torch.equal(alone, got)


@pytest.mark.parametrize("n", [1, 2, 16, 255, 257])
def test_short_contractions(ops, n):
    # few entries: k = 4 to 8; entries at the line on both sides
    N, M = n, 64
    G, f, X, gen = cohort(N, M, n, 0, False)
    F = torch.randn((n, 8), generator=gen, device="cuda") * 2.0 ** -torch.arange(0, 32, 4, device="cuda")
    F[n // 2] = 1.0
    got, ref = ops.rsvd_rows(G, f, F, M).double(), X @ F.double()
    mag = X.abs() @ F.double().abs()
    # no further off than float32 sums are bound to be
    assert bool(((got - ref).abs() <= 2.0 ** -24 * ((n + 1) * mag + ref.abs())).all())


@pytest.mark.parametrize("bad", [1, 3, 70])
@pytest.mark.parametrize("side", ["rows", "cols"])
def test_entries_that_are_not_finite(ops, bad, side):
    # few: added one by one; more than the list holds: every output in turn. In f (cols) a missing
    # genotype keeps the SNP out of the sample's sum; in f (rows) the SNP's own outputs change
    cols = side == "cols"
    N, M, L = 257, 301, 5
    n = M if cols else N
    G, f, X, gen = cohort(N, M, bad, 2, cols)
    product = ops.rsvd_cols if cols else ops.rsvd_rows
    F = torch.randn((n, L), generator=gen, device="cuda")
    at = torch.randperm(n, generator=gen, device="cuda")[:bad]
    F[at, 1] = float("inf")
    F[at[:1], 2] = float("nan")
    F[at, 3] = torch.where(torch.arange(bad, device="cuda") % 2 == 0, float("inf"), -float("inf"))
    got = product(G, f, F, M)
    A = X.T if cols else X
    ref = (A[:, :, None] * F.double()[None]).sum(1)
    clean = ref.isfinite()
    assert torch.equal(got[~clean], ref[~clean].float()) or torch.equal(got.isnan(), ref.isnan())
    assert torch.equal(got.isposinf(), ref.isposinf()) and torch.equal(got.isneginf(), ref.isneginf())
    assert bool(((got - ref).abs()[clean] <= 2.0 ** -22 * (A.abs() @ F.double().abs().nan_to_num(0, 0, 0))[clean]).all())

    f[at] = float("nan")   # rows: `at` as SNPs
    F = torch.randn((n, L), generator=gen, device="cuda")
    got = product(G, f, F, M)
    miss = (X == 0) & torch.from_numpy(unpack(G, M) == 3).cuda()
    Xn = torch.where(miss, 0.0, (X + 0.0 * f.double()[:, None]))
    A = Xn.T if cols else Xn
    ref = (A[:, :, None] * F.double()[None]).sum(1)
    assert torch.equal(got.isnan(), ref.isnan())
    fine = ~ref.isnan()
    assert bool(((got - ref).abs()[fine] <= 2.0 ** -22 * (A.abs() @ F.double().abs())[fine]).all())


def unpack(G, M):
    g = G.cpu().numpy()
    return np.stack([g >> (2 * s) & 3 for s in range(4)], 1).reshape(-1, g.shape[1])[:M]


def test_a_column_of_nans_leaves_the_others_alone(ops):
    N, M, L = 300, 400, 4
    G, f, X, gen = cohort(N, M, 8, 2, False)
    B = torch.randn((N, L), generator=gen, device="cuda")
    Y = torch.randn((M, L), generator=gen, device="cuda")
    plain = ops.rsvd_rows(G, f, B, M), ops.rsvd_cols(G, f, Y, M)
    B[:, 2] = Y[:, 2] = float("nan")
    for got, ref in zip((ops.rsvd_rows(G, f, B, M), ops.rsvd_cols(G, f, Y, M)), plain):
        assert bool(got[:, 2].isnan().all())
        assert torch.equal(got[:, [0, 1, 3]], ref[:, [0, 1, 3]])
