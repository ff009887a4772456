"""GPU checks of the integer tensor-core products of the centred genotypes: edges of the
256-row tiles and 256-entry blocks, the factor widths where passes and tensor-memory stages
change, every start address of the packed matrix, columns of very different scales, and
columns that are not finite.

Tolerance: the factor is rounded to 2^-31 of its column's largest magnitude (half a quantum
of 2^-30 2^e, the magnitude in [2^(e-1), 2^e)), an entry of the centred matrix is at most 2
in magnitude, and the result is rounded to float32 once; the reference is float64."""
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
    n = packed.size
    buf = torch.randint(0, 256, (n + 64,), dtype=torch.uint8, device="cuda")
    buf[offset:offset + n] = torch.from_numpy(packed.reshape(-1)).cuda()
    return buf[offset:offset + n].view(packed.shape)


def case(N, M, L, seed):
    rng = np.random.default_rng(seed)
    G = rng.choice(4, size=(M, N), p=[0.35, 0.3, 0.2, 0.15]).astype(np.uint8)
    f = rng.uniform(0.0, 1.0, M).astype(np.float32)
    X = np.where(G == 3, 0.0, G - 2.0 * f[:, None].astype(np.float64))
    scale = 10.0 ** rng.uniform(-30, 30, L)
    B = (rng.standard_t(2, size=(N, L)) * scale).astype(np.float32)
    Y = (rng.standard_t(2, size=(M, L)) * scale).astype(np.float32)
    if L > 2:
        B[:, 1] = Y[:, 1] = 0.0
    return orc.pack(G), f, X, B, Y


def close(got, ref, n_red, F, terms):
    tol = terms * n_red * 2.0 ** -30 * np.abs(F).max(0) + 2.0 ** -23 * np.abs(ref)
    err = np.abs(got.cpu().numpy().astype(np.float64) - ref)
    assert (err <= tol).all(), (err / np.maximum(tol, 1e-300)).max()


@pytest.mark.parametrize("N,M,L", [(1, 1, 1), (255, 4, 4), (256, 256, 5), (257, 259, 20), (512, 1000, 24), (100, 513, 25),
                                   (1000, 255, 33), (16, 5000, 48), (3000, 70, 49), (770, 1030, 80)])
def test_products(ops, N, M, L):
    packed, f, X, B, Y = case(N, M, L, N * M + L)
    fd, Bd, Yd = (torch.from_numpy(x).cuda() for x in (f, B, Y))
    refY, refZ = X @ B.astype(np.float64), X.T @ Y.astype(np.float64)
    first = None
    for off in (0, 3, 8, 15):
        G = placed(packed, off)
        gotY, gotZ = ops.rsvd_rows(G, fd, Bd, M), ops.rsvd_cols(G, fd, Yd, M)
        if first is None:
            first = gotY, gotZ
            close(gotY, refY, N, B, 2)
            # codes (at most 3) and flags (at most 1, factor up to 3 times as large), the constant
            close(gotZ, refZ, M, Y, 8)
            acc = ops.rsvd_cols(G, fd, Yd, M, out=gotZ.clone(), accumulate=True)
            assert torch.equal(acc, gotZ + gotZ)
        assert torch.equal(gotY, first[0]) and torch.equal(gotZ, first[1]), off


def test_columns_that_are_not_finite(ops):
    N, M, L = 300, 270, 6
    packed, f, X, B, Y = case(N, M, L, 5)
    for F, bad, red in ((B, 7, "rows"), (Y, 9, "cols")):
        F[bad, 2], F[bad, 4] = np.inf, np.nan
        G, fd, Fd = placed(packed, 0), torch.from_numpy(f).cuda(), torch.from_numpy(F).cuda()
        got = (ops.rsvd_rows if red == "rows" else ops.rsvd_cols)(G, fd, Fd, M).cpu().numpy()
        A = X if red == "rows" else X.T
        with np.errstate(invalid="ignore"):
            ref = (A[:, :, None] * F.astype(np.float64)[None]).sum(1)
        assert np.array_equal(np.isnan(got), np.isnan(ref))
        assert np.array_equal(np.isposinf(got), np.isposinf(ref)) and np.array_equal(np.isneginf(got), np.isneginf(ref))
        fine = [c for c in range(L) if c not in (2, 4)]
        close(torch.from_numpy(got[:, fine]), ref[:, fine], A.shape[1], F[:, fine], 8)


def test_workspace_at_any_address_and_the_form_without_one(ops):
    from adamixture_b200._lib import AdxError, call, query_size

    N, M, L = 300, 900, 20
    packed, f, X, B, Y = case(N, M, L, 11)
    B /= np.abs(B).max(0).clip(1e-30)
    G, fd, Bd = placed(packed, 0), torch.from_numpy(f).cuda(), torch.from_numpy(B).cuda()
    nb = query_size("adx_rsvd_workspace_bytes", M, N, L)
    buf = torch.empty(nb + 8, dtype=torch.uint8, device="cuda")
    ref = ops.rsvd_rows(G, fd, Bd, M)
    st = torch.cuda.current_stream().cuda_stream
    for off in (1, 4):
        out = torch.empty((M, L), device="cuda")
        call("adx_rsvd_rows_ws", G.data_ptr(), M, N, fd.data_ptr(), Bd.data_ptr(), L, out.data_ptr(),
             buf.data_ptr() + off, nb, st)
        assert torch.equal(out, ref)
    with pytest.raises(AdxError, match="workspace too small"):
        call("adx_rsvd_rows_ws", G.data_ptr(), M, N, fd.data_ptr(), Bd.data_ptr(), L, ref.data_ptr(), buf.data_ptr(),
             1024, st)
    out = torch.empty((M, L), device="cuda")
    call("adx_rsvd_rows", G.data_ptr(), M, N, fd.data_ptr(), Bd.data_ptr(), L, out.data_ptr(), st)
    # float32 sums of N terms: each addition rounds by 2^-24 of the partial sum
    tol = N * 2.0 ** -24 * 2 * np.abs(B).sum(0)
    assert (np.abs(out.cpu().numpy() - X @ B.astype(np.float64)) <= tol).all()
