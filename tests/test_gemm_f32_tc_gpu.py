"""The float32 GEMM of large matrices (gemm_f32_tc.cu) where its launches and its three-term operands have their edges."""
import math

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


@pytest.mark.parametrize("N,K", [(24600, 512), (1541, 8204)])
def test_sums_that_few_products_carry(k, N, K):
    """Rows of one, two and four numbers, and operands whose left-out terms are as large as they get and all of one sign:
    nothing averages out.  A product loses up to 2^-24 by what is left out, and its accumulator cuts off less than
    2^-23 of what has come together at each of the three products of full size."""
    gen = torch.Generator().manual_seed(K)
    w = torch.randn(N, K, generator=gen).cuda()
    a = torch.zeros(40, K)
    for row in range(36):
        at = torch.randperm(K, generator=gen)[: 1 << row % 3]
        a[row, at] = torch.randn(len(at), generator=gen)
    a = a.cuda()
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    for weights in (w, torch.full_like(w, 1.0038986), torch.full_like(w, -0.75 * 1.0038986)):
        a[36:] = 1.0038986
        for M in (40, 9):
            out = torch.empty(M, N, device="cuda")
            k.gemm_f32(a[40 - M :].contiguous(), weights, None, out, M, status=status)
            rows = a[40 - M :].double()
            size = rows.abs() @ weights.double().abs().T
            error = (out.double() - rows @ weights.double().T).abs()
            bound = torch.full((M, 1), 2.0 ** -24 + 3 * 2.0 ** -23, dtype=torch.float64, device="cuda")
            bound[M - 4 :] += 2.0 ** -24 * (K / 32)  # (chunks of 32 one after the other)
            assert bool((error <= bound * size + 1e-44).all()), (M, (error / size.clamp_min(1e-30)).max())
    assert int(status[0]) == 0


@pytest.mark.parametrize("N,K", [(24600, 512), (1541, 8204)])
def test_tiny_operands(k, N, K):
    """Operands whose third terms bfloat16 has no numbers for, in rows beside ordinary ones: as near as an FMA chain, and
    the same bits in every batch."""
    gen = torch.Generator().manual_seed(N + K)
    w = (torch.randn(N, K, generator=gen) * 0.02).cuda()
    a = torch.randn(33, K, generator=gen).cuda()
    exponents = [0, 60, 95, 100, 105, 109, 110, 111, 112, 115, 118, 120, 122]
    for row, e in enumerate(exponents):
        a[row] *= 2.0 ** -e
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out = torch.empty(33, N, device="cuda")
    k.gemm_f32(a, w, None, out, 33, status=status)
    want = a.double() @ w.double().T
    # (And half of the smallest float32 number, which a sum and 32 partial sums may lose.)
    error = (out.double() - want).abs().amax(1)
    assert bool((error <= 2 * 2.0 ** -24 * math.sqrt(K) * want.abs().amax(1) + 33 * 2.0 ** -150).all()), error / want.abs().amax(1)
    few = torch.empty(13, N, device="cuda")
    k.gemm_f32(a[:13].contiguous(), w, None, few, 13, status=status)
    assert torch.equal(few, out[:13])
    w[5] *= 2.0 ** -116
    k.gemm_f32(a, w, None, out, 33, status=status)
    want = a[13:].double() @ w[5].double()
    assert (out[13:, 5].double() - want).abs().max().item() <= 2 * 2.0 ** -24 * math.sqrt(K) * want.abs().max().item() + 33 * 2.0 ** -150
    assert int(status[0]) == 0


@pytest.mark.parametrize("N,K", [(17920, 1536), (1541, 8204)])
def test_rows_of_nan(k, N, K):
    """A batch of NaN does not hold the kernel up (one thread an element took 131 ms over the first of these, a plain batch 0.3)."""
    gen = torch.Generator().manual_seed(N)
    w, b = torch.randn(N, K, generator=gen).cuda(), torch.randn(N, generator=gen).cuda()
    a = torch.randn(1024, K, generator=gen).cuda()
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out = torch.empty(1024, N, device="cuda")
    clean, dirty = a.clone(), a.clone()
    a[:, 5] = float("nan")
    w_dirty = w.clone()
    w_dirty[:, 7] = float("nan")
    dirty[3, 9], dirty[900, K - 1] = float("inf"), float("nan")
    for rows, weights in ((a, w), (clean, w_dirty)):
        k.gemm_f32(rows, weights, b, out, 1024, status=status)
        assert bool(torch.isnan(out).all())
        start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        k.gemm_f32(rows, weights, b, out, 1024, status=status)
        stop.record()
        torch.cuda.synchronize()
        assert start.elapsed_time(stop) < 13.0
    w[2, 1], w[40, 3], b[8] = float("nan"), float("-inf"), float("nan")
    k.gemm_f32(dirty, w, b, out, 1024, status=status)
    want = dirty.double() @ w.double().T + b.double()
    assert torch.equal(torch.isnan(out), torch.isnan(want))
    assert torch.equal(torch.isposinf(out), torch.isposinf(want)) and torch.equal(torch.isneginf(out), torch.isneginf(want))
    assert int(status[0]) == 0
