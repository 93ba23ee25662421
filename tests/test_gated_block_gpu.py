"""The parallel gated block's kernels where they change between one and four elements a thread: widths and strides that are
and are not multiples of four, the last element of a block of threads, few and many tokens, all output types.  Against
float64; the bounds are a few roundings of the float32 arithmetic and one of the output type."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
ROUND = {torch.float32: 0.0, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def close(got, want, dtype, scale=1.0):
    """Within 24 roundings of float32 of the larger of the value and `scale`, and one rounding of the output type."""
    want = want.double()
    size = torch.maximum(want.abs(), torch.full_like(want, scale))
    assert ((got.double() - want).abs() <= size * (24 * 2.0 ** -24 + ROUND[dtype])).all()


def rand(g, *shape):
    return torch.randn(*shape, device="cuda", generator=g)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,F,pad", [(1, 4, 0), (3, 508, 4), (3, 512, 0), (3, 516, 8), (3, 516, 1), (2, 513, 0), (70, 5632, 2048), (8, 512, 0), (9, 4, 0), (9, 508, 4),
                                     (9, 512, 0), (9, 516, 8), (9, 516, 1), (9, 513, 0)])
def test_bias_glu_widths(cuda, dtype, T, F, pad):
    from ferrum_b200.ops import lib as ops
    g = torch.Generator(device="cuda").manual_seed(F + pad)
    gu, bg, bu = rand(g, T, 2 * F + pad), rand(g, F), rand(g, F)
    act = torch.zeros(T + 1, F, device="cuda", dtype=dtype)
    for gate, up in ((bg, bu), (None, bu), (None, None)):
        ops.bias_glu(gu, gate, up, act[:T], T, F, "silu")
        if T > 8:          # fewer tokens run one feature a thread: the same bits
            first = torch.empty(8, F, device="cuda", dtype=dtype)
            ops.bias_glu(gu, gate, up, first, 8, F, "silu")
            assert torch.equal(first, act[:8])
        z = gu[:, :F].double() + (gate.double() if gate is not None else 0)
        u = gu[:, F:2 * F].double() + (up.double() if up is not None else 0)
        close(act[:T], torch.nn.functional.silu(z) * u, dtype)
    assert not act[T].any()


@pytest.mark.parametrize("T,E,pad", [(64, 256, 0), (65, 4, 0), (65, 1020, 4), (65, 1024, 0), (65, 1028, 0), (65, 1028, 1), (66, 1030, 2), (70, 2048, 0)])
@pytest.mark.parametrize("second", [True, False])
def test_gated_residual_widths(cuda, T, E, pad, second):
    from ferrum_b200.ops import lib as ops
    g = torch.Generator(device="cuda").manual_seed(E + pad)
    x, y1, y2 = rand(g, T + 1, E), rand(g, T, E), rand(g, T, E)
    g1, g2 = rand(g, T, E + pad)[:, :E], rand(g, T, E + pad)[:, pad:]
    c1, c2, c3 = rand(g, E), rand(g, E), rand(g, E)
    stage, state = rand(g, 4, E), torch.zeros(5, E, device="cuda")
    q_start = torch.tensor([0, T - 2, T], dtype=torch.int32, device="cuda")
    ctx = SimpleNamespace(q_start=q_start, slots=torch.tensor([3, 1], dtype=torch.int32, device="cuda"),
                          req_of_token=torch.tensor([0] * (T - 2) + [1] * 2, dtype=torch.int32, device="cuda"))
    want = x[:T].double() + y1.double() * torch.sigmoid(g1.double() + c1.double())
    if second:
        want += (y2.double() + c2.double()) * torch.sigmoid(g2.double() + c3.double())
    rest = x[T].clone()
    ops.gated_residual(x, T, y1, g1, c1, *((y2, c2, g2, c3) if second else ()), ctx=ctx, stage=stage, state=state)
    close(x[:T], want, torch.float32, 4.0)
    assert torch.equal(x[T], rest) and torch.equal(state[3], stage[0]) and torch.equal(state[1], stage[1])
    assert not state[[0, 2, 4]].any()


@pytest.mark.parametrize("E", [20, 1028, 2048])
@pytest.mark.parametrize("second", [True, False])
@pytest.mark.parametrize("biased", [True, False])
def test_gated_residual_of_64_and_65_tokens(cuda, E, second, biased):
    """A token's bits do not depend on how many others are in the step, and are those of sums whose only fused product is
    the second one."""
    from ferrum_b200.ops import lib as ops
    g = torch.Generator(device="cuda").manual_seed(E)
    x, y1, y2, g1, g2 = (rand(g, 65, E) for _ in range(5))
    c1, c2, c3 = (rand(g, E) if biased else None for _ in range(3))

    def run(n, rows, v1=y1, v2=y2):
        out = rows[:n].clone()
        ops.gated_residual(out, n, v1, g1, c1, *((v2, c2, g2, c3) if second else ()))
        return out

    few, many = run(64, x), run(65, x)
    assert torch.equal(few, many[:64])
    zero, one = torch.zeros_like(x), torch.ones_like(x)
    s1 = zero.clone()
    ops.gated_residual(s1, 65, one, g1, c1)         # 0 + 1 * sigmoid: the sigmoid's own bits
    add = y1 * s1
    if second:
        s2 = zero.clone()
        ops.gated_residual(s2, 65, one, g2, c3)
        # the exact product of two float32, rounded once with the sum (in float64: a second rounding shows in one of 2^28)
        add = ((y2 + c2 if biased else y2).double() * s2.double() + add.double()).float()
    assert (many != x + add).float().mean() < 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("E,groups", [(24, 8), (32, 8), (36, 9), (1020, 1), (1024, 2), (1032, 2), (2048, 8), (4112, 1)])
def test_norm_pair_shift_widths(cuda, dtype, E, groups):
    from ferrum_b200.ops import lib as ops
    g = torch.Generator(device="cuda").manual_seed(E)
    T = 7      # a request of five tokens from position 0 and one of two that goes on from its state
    x, w1, w2, s, state = rand(g, T, E), rand(g, E), rand(g, E), rand(g, E), rand(g, 4, E)
    stage = torch.zeros(2, E, device="cuda")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    ctx = SimpleNamespace(positions=i32([0, 1, 2, 3, 4, 9, 10]), req_of_token=i32([0] * 5 + [1] * 2), q_start=i32([0, 5, 7]),
                          slots=i32([2, 3]), n_reqs=2)
    a, m, b = (torch.empty(T, E, device="cuda", dtype=dtype) for _ in range(3))
    ops.norm_pair_shift(x, w1, w2, s, a, m, b, T, ctx, state, stage, groups, 1e-5)
    v = x.double().view(T, groups, -1)
    n = (v * torch.rsqrt((v * v).mean(-1, keepdim=True) + 1e-5)).view(T, E)
    want = n * w1.double()
    before = torch.cat([torch.zeros_like(want[:1]), want[:4], state[3:4].double(), want[5:6]])
    close(a, want, dtype, 4.0)
    close(m, want + (before - want) * s.double(), dtype, 16.0)
    close(b, n * w2.double(), dtype, 4.0)
    close(stage, want[[4, 6]], torch.float32, 4.0)
