"""The randomized-SVD products' workspace is bounded: it does not grow with the SNPs past a
launch's share, at any width."""
import pytest

from adamixture_b200._lib import query_size


@pytest.mark.parametrize("L,most", [(20, 4e8), (26, 6e8), (80, 2e9)])
def test_bytes_stay_bounded(L, most):
    def nbytes(M, N):
        return query_size("adx_rsvd_workspace_bytes", M, N, L)

    assert nbytes(1_000_000, 1000) == nbytes(10_000_000, 1000) == nbytes(100_000_000, 1000) <= most
    assert nbytes(1000, 1_000_000) == nbytes(1000, 10_000_000) <= most
    assert nbytes(100, 100) < nbytes(10_000, 1000) < nbytes(300_000, 100_000) < nbytes(10_000_000, 1000)
