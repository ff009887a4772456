"""GPU checks of the pipeline of the integer tensor-core products: shapes whose CTAs walk many
blocks, so that the three load slots wrap and every A stage is filled several times at each
stage count (2, 3 and 4, set by the factor's width), and what a product does when a wait runs
out.

Tolerance: as in test_gpu_rsvd_tc.py; the reference is float64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(cuda):
    from adamixture_b200 import ops as _ops

    return _ops


def cohort(N, M, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    g = torch.randint(0, 4, ((M + 3) // 4 * 4, N), generator=gen, device="cuda", dtype=torch.uint8)
    g[M:] = 0
    q = g.view(-1, 4, N)
    packed = (q[:, 0] | q[:, 1] << 2 | q[:, 2] << 4 | q[:, 3] << 6).contiguous()
    f = torch.rand(M, generator=gen, device="cuda")
    X = (g[:M].double() - 2.0 * f.double()[:, None]).masked_fill_(g[:M] == 3, 0.0)
    return packed, f, X, gen


# rows: a CTA per 256 SNPs walks every block of samples (9 and 4); cols: 4 to 9 of the SNPs'
@pytest.mark.parametrize("N,M,L", [(2051, 38003, 16), (2048, 38000, 20), (2051, 38003, 24), (1003, 40011, 26)])
def test_many_blocks_a_cta(ops, N, M, L):
    G, f, X, gen = cohort(N, M, N + L)
    B = torch.randn((N, L), generator=gen, device="cuda")
    Y = torch.randn((M, L), generator=gen, device="cuda")
    for got, ref, n, F, terms in ((ops.rsvd_rows(G, f, B, M), X @ B.double(), N, B, 2),
                                  (ops.rsvd_cols(G, f, Y, M), X.T @ Y.double(), M, Y, 8)):
        tol = terms * n * 2.0 ** -30 * F.abs().amax(0).double() + 2.0 ** -23 * ref.abs()
        assert bool(((got.double() - ref).abs() <= tol).all())


@pytest.mark.parametrize("cols", [0, 1])
def test_a_wait_that_runs_out(ops, cols):
    # no wait gets a poll: every warp leaves its loop, the kernel ends by itself and says so in
    # every entry; the next product is not affected
    from adamixture_b200._lib import call, query_size

    N, M, L = 1003, 40011, 20
    G, f, X, gen = cohort(N, M, 3)
    F = torch.randn((M if cols else N, L), generator=gen, device="cuda")
    product = ops.rsvd_cols if cols else ops.rsvd_rows
    before = product(G, f, F, M)
    ws = torch.empty(query_size("adx_rsvd_workspace_bytes", M, N, L), dtype=torch.uint8, device="cuda")
    out = torch.zeros_like(before)
    call("adx_rsvd_wait_selftest", G.data_ptr(), M, N, f.data_ptr(), F.data_ptr(), L, cols, 0, out.data_ptr(),
         ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    assert bool(torch.isnan(out).all())
    assert torch.equal(product(G, f, F, M), before)
    assert np.isfinite(before.cpu().numpy()).all()


def test_status_of_the_workspace(ops):
    from adamixture_b200._lib import call

    N, M, L = 300, 900, 4
    G, f, X, gen = cohort(N, M, 5)
    B = torch.randn((N, L), generator=gen, device="cuda")
    ws = ops.rsvd_workspace(G.device, M, N, L)
    out = ops.rsvd_rows(G, f, B, M, ws=ws)
    ops.rsvd_check(ws)
    call("adx_rsvd_wait_selftest", G.data_ptr(), M, N, f.data_ptr(), B.data_ptr(), L, 0, 0, torch.empty_like(out).data_ptr(),
         ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    assert torch.equal(ops.rsvd_rows(G, f, B, M, ws=ws), out)   # a product of its own; the status stays
    with pytest.raises(RuntimeError, match="status 5"):
        ops.rsvd_check(ws)
    ops.rsvd_check(ws)   # read once


@pytest.mark.parametrize("caller", ["svd", "sharded", "frequencies", "supervised"])
def test_callers_raise_on_a_timeout(ops, monkeypatch, caller):
    # the word is set by hand in the workspaces that the callers make
    from adamixture_b200.model.init_dist import CudaInitBackend
    from adamixture_b200.model.svd_gpu import SVD_gpu
    from adamixture_b200.model.warm_start import m_step_P
    from adamixture_b200.src.supervised import init_p_supervised_gpu

    N, M, K = 60, 200, 3
    G, f, X, gen = cohort(N, M, 6)
    Q = torch.rand((N, K), generator=gen, device="cuda")
    run = {"svd": lambda: SVD_gpu(G, N, M, f, K, 1, 2, 1e-1, 256, G.device, 256),
           "sharded": lambda: CudaInitBackend().rsvd_rows(G, f, Q, M),
           "frequencies": lambda: m_step_P(G, Q, M),
           "supervised": lambda: init_p_supervised_gpu(G, np.arange(N) % (K + 1), K, M)}[caller]
    run()
    plain = ops.rsvd_workspace

    def timed_out(*args):
        ws = plain(*args)
        ws[:4].copy_(torch.tensor([5, 0, 0, 0], dtype=torch.uint8))
        return ws

    monkeypatch.setattr(ops, "rsvd_workspace", timed_out)
    with pytest.raises(RuntimeError, match="status 5"):
        run()


# more rows and more contracted entries than one launch takes (606,208 and 524,288), with a last
# launch that is nearly empty; one column wide, one with an infinity
@pytest.mark.parametrize("N,M", [(9, 1_212_421), (524_300, 9), (606_209, 6)])
def test_several_launches(ops, N, M):
    L = 6
    G, f, X, gen = cohort(N, M, N)
    B = torch.randn((N, L), generator=gen, device="cuda")
    Y = torch.randn((M, L), generator=gen, device="cuda")
    for product, A, F in ((ops.rsvd_rows, X, B), (ops.rsvd_cols, X.T, Y)):
        n = F.shape[0]
        F[:, 1] *= 2.0 ** -20
        F[n // 2, 1] = 1.0
        F[n - 1, 2] = float("inf")
        got, fine = product(G, f, F, M), [c for c in range(L) if c != 2]
        ref = A @ F[:, fine].double()
        tol = 8 * n * 2.0 ** -30 * F[:, fine].abs().amax(0).double() + 2.0 ** -23 * ref.abs()
        assert bool(((got[:, fine].double() - ref).abs() <= tol).all())
        assert bool((~got[:, 2].isfinite()).all())
        once = product(G, f, F, M, out=torch.zeros_like(got)) if product is ops.rsvd_rows else \
            product(G, f, F, M, out=torch.zeros_like(got), accumulate=True)
        assert torch.equal(once[:, fine], got[:, fine])


def test_products_in_a_row(ops):
    # a product's kernels overlap at their ends: products that read what the one before wrote, over
    # one workspace, without a pause and replayed from a graph, equal those run one at a time
    N, M, L = 700, 5003, 20
    G, f, X, gen = cohort(N, M, 9)
    ws = ops.rsvd_workspace(G.device, M, N, L)
    B0 = torch.randn((N, L), generator=gen, device="cuda")
    B0[:, 3] *= 2.0 ** -24   # wide: the second level too
    B0[5, 3] = 1.0
    want, B = [], B0
    for _ in range(6):
        Y = ops.rsvd_rows(G, f, B, M)
        torch.cuda.synchronize()
        B = ops.rsvd_cols(G, f, Y, M) * 2.0 ** -12
        torch.cuda.synchronize()
        want.append(B)
    Y, B = torch.empty((M, L), device="cuda"), B0.clone()

    def chain():
        out = []
        for _ in range(6):
            ops.rsvd_rows(G, f, B, M, out=Y, ws=ws)
            ops.rsvd_cols(G, f, Y, M, out=B, ws=ws)
            B.mul_(2.0 ** -12)
            out.append(B.clone())
        return out

    assert all(torch.equal(a, b) for a, b in zip(chain(), want))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    B.copy_(B0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        got = chain()
    for _ in range(3):
        B.copy_(B0)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    ops.rsvd_check(ws)


def test_frequencies_can_be_captured(ops):
    # the status is not read while a graph is being captured
    from adamixture_b200.model.warm_start import m_step_P

    N, M, K = 200, 900, 5
    G, f, X, gen = cohort(N, M, 10)
    Q = torch.softmax(torch.randn((N, K), generator=gen, device="cuda"), 1).double()
    want = m_step_P(G, Q, M)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        got = m_step_P(G, Q, M)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
