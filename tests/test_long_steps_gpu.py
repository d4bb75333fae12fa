"""Projections of long steps (gemm_bf16_wide.cu): every epilogue against float64, at the edges of its tiles."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def k():
    from velox_b200.ops import kernels

    kernels._require_cuda()
    return kernels


@pytest.fixture()
def status():
    return torch.zeros(4, dtype=torch.int32, device="cuda")


def _operands(T, N, K, scale=1.0):
    gen = torch.Generator().manual_seed(T + N + K)
    x = torch.randn(T + 3, K, generator=gen).to(torch.bfloat16).cuda()
    w = (torch.randn(N, K, generator=gen) * scale / math.sqrt(K)).to(torch.bfloat16).cuda()
    return gen, x, w


# Rows that are no multiple of a tile, features short of a tile and one past it, inner sizes below a block and
# past one, more tiles than pairs of SMs; 0: the tile that the launcher takes.
SIZES = [(257, 200, 72), (300, 264, 1000), (513, 520, 64), (1030, 2056, 136), (700, 20000, 200)]


@pytest.mark.parametrize("T,N,K", SIZES)
@pytest.mark.parametrize("tokens", [0, 16, 144, 256])
def test_sums(k, status, T, N, K, tokens):
    gen, x, w = _operands(T, N, K)
    bias = torch.randn(N, generator=gen).cuda()
    want = x[:T].double() @ w.double().T + bias.double()
    scale = want.abs().max().item()
    start = torch.randn(T + 2, N, generator=gen).cuda()
    stream = start.clone()
    assert k.gemm_bf16_wide(x, w, bias, stream, k.GEMM_ADD_F32, T, status, tokens, 1)
    want += start[:T].double()
    # The accumulator cuts off what is below a unit in its last place, K / 16 times, and two additions round.
    assert (stream[:T].double() - want).abs().max().item() <= 2.0 ** -23 * (K / 16 + 2) * max(scale, want.abs().max().item())
    assert torch.equal(stream[T:], start[T:])
    again = start.clone()
    k.gemm_bf16_wide(x, w, bias, again, k.GEMM_ADD_F32, T, status, tokens, 1)
    assert torch.equal(again, stream)
    for chunks in (0, 3, 100):  # (the last: a block of the inner size each)
        again = start.clone()
        assert k.gemm_bf16_wide(x, w, bias, again, k.GEMM_ADD_F32, T, status, tokens, chunks)
        assert (again[:T].double() - want).abs().max().item() <= 2.0 ** -23 * (K / 16 + 4) * max(scale, want.abs().max().item())
        assert torch.equal(again[T:], start[T:])
    assert int(status[0]) == 0


@pytest.mark.parametrize("T,N,K", SIZES)
@pytest.mark.parametrize("tokens", [0, 32, 208])
def test_gated_activation(k, status, T, N, K, tokens):
    _, x, w = _operands(T, 2 * N, K, 2.0)
    out = torch.full((T + 2, N), 7.0, dtype=torch.bfloat16, device="cuda")
    assert k.gemm_bf16_wide(x, w, None, out, k.GEMM_SWIGLU, T, status, tokens)
    # (One rounding of the output, 2^-9 of it.)
    both = x[:T].double() @ w.double().T
    want = torch.nn.functional.silu(both[:, :N]) * both[:, N:]
    assert (out[:T].double() - want).abs().max().item() <= 2.0 ** -8 * want.abs().max().item()
    assert torch.all(out[T:] == 7.0)
    assert int(status[0]) == 0


@pytest.mark.parametrize("limit,alpha,shift,cubic", [(0.0, 1.5957691216, 0.0, 0.044715), (3.0, 1.702, 1.0, 0.0)])
@pytest.mark.parametrize("T,N,K", SIZES[:4])
def test_gated_activation_with_its_options(k, status, T, N, K, limit, alpha, shift, cubic):
    gen, x, w = _operands(T, 2 * N, K, 2.0)
    bias = torch.randn(2 * N, generator=gen).cuda()
    out = torch.full((T + 2, N), 7.0, dtype=torch.bfloat16, device="cuda")
    assert k.gemm_bf16_wide_glu(x, w, bias, out, T, limit, alpha, shift, status, cubic=cubic)
    gate, up = (x[:T].double() @ w.double().T + bias.double()).split(N, dim=1)
    if limit:
        gate, up = gate.clamp(max=limit), up.clamp(-limit, limit)
    want = gate * torch.sigmoid(alpha * (gate + cubic * gate ** 3)) * (up + shift)
    assert (out[:T].double() - want).abs().max().item() <= 2.0 ** -8 * want.abs().max().item()
    assert torch.all(out[T:] == 7.0)
    assert int(status[0]) == 0


@pytest.mark.parametrize("T,N,K", SIZES[:4])
@pytest.mark.parametrize("side", [0, 24, 136])
def test_activated_columns_beside_plain_ones(k, status, T, N, K, side):
    gen, x, w = _operands(T, N, K, 2.0)
    bias = torch.randn(N, generator=gen).cuda()
    out = torch.full((T + 2, N), 7.0, dtype=torch.bfloat16, device="cuda")
    act = torch.full((T + 2, N - side), 7.0, dtype=torch.bfloat16, device="cuda")
    assert k.gemm_bf16_wide_xielu(x, w, bias, out, act, side, 0.7, 0.9, T, status)
    z = x[:T].double() @ w.double().T + bias.double()
    want = torch.where(z > 0, 0.7 * z * z + z / 2, 0.9 * (torch.expm1(z.clamp(max=0)) - z) + z / 2)
    scale = max(z.abs().max().item(), want.abs().max().item())
    assert (act[:T].double() - want[:, side:]).abs().max().item() <= 2.0 ** -8 * scale
    if side:
        assert (out[:T, :side].double() - z[:, :side]).abs().max().item() <= 2.0 ** -8 * scale
    assert torch.all(out[:, side:] == 7.0) and torch.all(out[T:] == 7.0) and torch.all(act[T:] == 7.0)
    assert int(status[0]) == 0


def test_refuses_what_its_copies_cannot_take(k, status):
    x = torch.zeros(300, 60, dtype=torch.bfloat16, device="cuda")
    w = torch.zeros(256, 60, dtype=torch.bfloat16, device="cuda")
    out = torch.zeros(300, 256, device="cuda")
    assert not k.gemm_bf16_wide(x, w, None, out, k.GEMM_ADD_F32, 300, status)


# (tokens, N, K, mode): both sides of the lines as they were measured, and of what they are drawn between.
@pytest.mark.parametrize("T,N,K,mode,chunked,pays", [
    (300, 1536, 8960, 2, True, True), (300, 1536, 8960, 2, False, False), (768, 1536, 8960, 2, True, True),
    (769, 1536, 8960, 2, True, False), (300, 1536, 1536, 2, True, True), (300, 1536, 1536, 2, False, True),
    (768, 2048, 2048, 2, True, True), (769, 2048, 2048, 2, True, False), (536, 3584, 3584, 2, True, False),
    (2048, 3584, 3584, 2, True, True), (2048, 3584, 3584, 2, False, True), (1400, 3584, 18944, 2, True, False),
    (2048, 8960, 1536, 3, True, True), (300, 8960, 1536, 3, True, True), (1755, 4864, 896, 3, True, True),
    (1756, 4864, 896, 3, True, False), (536, 18944, 3584, 3, True, True), (300, 18944, 3584, 3, True, False),
    (2048, 18944, 3584, 6, True, True), (700, 8960, 1536, 6, True, False), (2048, 20736, 5120, 5, True, True),
    (700, 12544, 2048, 5, True, False)])
def test_which_products_pay(k, T, N, K, mode, chunked, pays):
    assert k.gemm_bf16_wide_pays(mode, T, N, K, chunked) is pays


def test_sums_beyond_768_tokens_repeat(k, status):
    """One chunk of the inner size: an element has one addition, whatever ran before."""
    _, x, w = _operands(1030, 1536, 8960)
    first = None
    for _ in range(6):
        stream = torch.ones(1030, 1536, device="cuda")
        assert k.gemm_bf16_wide(x, w, None, stream, k.GEMM_ADD_F32, 1030, status)
        first = stream if first is None else first
        assert torch.equal(stream, first)
    assert int(status[0]) == 0


# One product after the other on pairs of SMs and in the library, in all four ways.
@pytest.mark.parametrize("T,E,I,gate,down", [(300, 896, 4864, True, True), (1000, 1536, 8960, True, False),
                                             (300, 3584, 9000, False, True), (1800, 896, 4864, False, False)])
def test_feed_forward_on_both_sides_of_the_lines(k, status, T, E, I, gate, down):
    from types import SimpleNamespace

    from velox_b200.engine.runner import Workspace
    from velox_b200.parts.mlp import SwiGLU

    assert k.gemm_bf16_wide_pays(k.GEMM_SWIGLU, T, I, E, True) is gate and k.gemm_bf16_wide_pays(k.GEMM_ADD_F32, T, E, I, True) is down
    gen, x, w = _operands(T, 2 * I, E)
    w_down = (torch.randn(E, I, generator=gen) / math.sqrt(I)).to(torch.bfloat16).cuda()
    part = SwiGLU({"hidden_size": E, "intermediate_size": I}, {"gate_up.weight": w, "down.weight": w_down}, torch.bfloat16,
                  torch.device("cuda"))
    start = torch.randn(T + 3, E, generator=gen).cuda()
    stream = start.clone()
    ctx = SimpleNamespace(num_tokens=T, workspace=Workspace(T + 3, 8, torch.device("cuda")), residual=stream, status=status)
    out = part.forward(x, ctx)
    assert (out is None) is down
    both = x[:T].double() @ w.double().T
    want = (torch.nn.functional.silu(both[:, :I]) * both[:, I:]) @ w_down.double().T
    # The activation and, from the library, the product are rounded to bfloat16 (2^-9 of them); sums of I like errors.
    bound = 2.0 ** -7 * want.abs().max().item()
    got = stream - start if down else out
    assert (got[:T].double() - want).abs().max().item() <= bound
    assert torch.equal(stream[T:], start[T:]) and (down or torch.equal(stream, start))
    assert int(status[0]) == 0


def test_long_steps_repeat_with_the_switch():
    """VELOX_B200_DETERMINISTIC=1 (read at import, hence a process of its own): no sum of a long step is cut, also where
    the default cuts it (down projections of up to 768 tokens)."""
    import os
    import pathlib
    import subprocess
    import sys

    program = """
from types import SimpleNamespace
import torch
from velox_b200.engine.runner import Workspace
from velox_b200.ops.linear import adds_to_stream, linear
from velox_b200.parts.mlp import SwiGLU
dev = torch.device("cuda")
E, I = 1536, 8960
gen = torch.Generator(device=dev).manual_seed(1)
def matrix(rows, cols):
    return (torch.randn(rows, cols, generator=gen, device=dev) / cols ** 0.5).to(torch.bfloat16)
part = SwiGLU({"hidden_size": E, "intermediate_size": I}, {"gate_up.weight": matrix(2 * I, E), "down.weight": matrix(E, I)},
              torch.bfloat16, dev)
w_out = matrix(E, E)
status = torch.zeros(4, dtype=torch.int32, device=dev)
for T in (257, 700, 1030):
    x, act = matrix(T, E), matrix(T, I)
    assert not (T < 768 and adds_to_stream(act, part.w_down, T, status))
    first = None
    for _ in range(6):
        stream = torch.ones(T, E, device=dev)
        linear(x, w_out, None, stream, T, status=status, accumulate=True)
        linear(act, part.w_down, None, stream, T, status=status, accumulate=True)
        out = part.forward(x, SimpleNamespace(num_tokens=T, workspace=Workspace(T, 8, dev), residual=stream, status=status))
        both = [stream] + ([] if out is None else [out[:T].clone()])
        first = both if first is None else first
        assert all(torch.equal(a, b) for a, b in zip(both, first)), T
assert int(status[0]) == 0
"""
    root = str(pathlib.Path(__file__).resolve().parent.parent)
    env = dict(os.environ, VELOX_B200_DETERMINISTIC="1", PYTHONPATH=root + os.pathsep + os.environ.get("PYTHONPATH", ""))
    done = subprocess.run([sys.executable, "-c", program], env=env, cwd=root, capture_output=True, text=True, timeout=240)
    assert done.returncode == 0, done.stderr[-2000:]
