"""The float32 GEMM of large matrices (gemm_f32_tc.cu) where its launches and its three-term operands have their edges."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def k():
    from velox_b200.ops import kernels

    kernels._require_cuda()
    return kernels


@pytest.mark.parametrize("N,K", [(24600, 512), (1541, 8204)])
def test_more_rows_than_a_launch_takes(k, N, K):
    """8,000 rows a launch: the rows on both sides of the line, with a last launch of one tile and of one that splits its
    rows itself, as each alone."""
    gen = torch.Generator().manual_seed(N)
    w, b = torch.randn(N, K, generator=gen).cuda(), torch.randn(N, generator=gen).cuda()
    a = torch.randn(8040, K, generator=gen).cuda()
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    for M in (8016, 8040):
        out = torch.full((M + 1, N), 5.0, device="cuda")
        k.gemm_f32(a, w, b, out, M, status=status)
        assert torch.all(out[M] == 5.0)
        for first in (0, 7995, 8000, M - 9):
            alone = torch.empty(9, N, device="cuda")
            k.gemm_f32(a[first : first + 9].contiguous(), w, b, alone, 9, status=status)
            assert torch.equal(out[first : first + 9], alone), (M, first)
    assert int(status[0]) == 0
