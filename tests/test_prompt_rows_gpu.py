"""Row kernels whose grid or whose accesses depend on the number of tokens, the width and the alignment: the same bits as a
few tokens at a time, or float64 within a few roundings."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,F,pad", [(1, 4, 0), (2, 508, 4), (2, 512, 0), (3, 516, 8), (3, 516, 1), (2, 513, 0), (300, 8192, 0)])
def test_float32_swiglu_widths(cuda, T, F, pad):
    from ferrum_b200.ops import lib as ops
    g = torch.Generator(device="cuda").manual_seed(F + pad)
    gu = torch.randn(T, 2 * F + pad, device="cuda", generator=g) * 3
    act = torch.zeros(T + 1, F + pad, device="cuda")
    ops.swiglu(gu, act, T, F)
    want = torch.nn.functional.silu(gu[:, :F].double()) * gu[:, F:2 * F].double()
    # expf, a sum, a division and a product: within 8 roundings
    assert ((act[:T, :F].double() - want).abs() <= want.abs() * 8 * 2.0 ** -24 + 1e-30).all()
    assert not act[T].any() and not act[:, F:].any()


@pytest.mark.parametrize("T", [65, 300, 591, 592, 593, 800, 1183, 1184, 1185])
@pytest.mark.parametrize("Hq,Hkv,D,R,pairing", [(24, 8, 128, 128, 1), (3, 1, 20, 12, 0), (5, 5, 64, 64, 0)])
def test_float32_rotary_rows_do_not_depend_on_the_grid(cuda, T, Hq, Hkv, D, R, pairing):
    from ferrum_b200.ops import lib as ops
    g = torch.Generator(device="cuda").manual_seed(T + D)
    page, pages = 16, -(-T // 16)
    first = torch.randn(T, (Hq + 2 * Hkv) * D, device="cuda", generator=g)
    angles = torch.rand(T, R // 2, device="cuda", generator=g) * 6
    cos_sin = torch.stack([angles.cos(), angles.sin()], -1).contiguous()
    positions = torch.arange(T, dtype=torch.int32, device="cuda")
    req = torch.zeros(T, dtype=torch.int32, device="cuda")
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(1)).to(torch.int32).cuda()[None]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(step):
        qkv, plane = first.clone(), torch.zeros(pages, 2, Hkv, page, D, device="cuda")
        for t in range(0, T, step):
            n = min(step, T - t)
            ops.rope_cache_write(qkv[t:], n, positions[t:], req[t:], table, cos_sin, plane, plane.stride(0), page, Hq, Hkv, D, R,
                                 pairing, True, err)
        return qkv, plane

    (a, b), (c, d) = run(T), run(64)
    assert torch.equal(a, c) and torch.equal(b, d) and err.item() == 0


def test_float32_rotary_rows_take_no_longer_for_a_token_less(cuda):
    """The grid shrinks as the tokens grow, not all at once (with six blocks a token up to a line 800 tokens took longer than 1,184)."""
    from ferrum_b200.ops import lib as ops
    Hq, Hkv, D, page, T = 32, 8, 128, 16, 1184
    qkv, plane = torch.zeros(T, (Hq + 2 * Hkv) * D, device="cuda"), torch.zeros(T // page, 2, Hkv, page, D, device="cuda")
    cos_sin, positions = torch.ones(T, D // 2, 2, device="cuda"), torch.arange(T, dtype=torch.int32, device="cuda")
    req, table = torch.zeros(T, dtype=torch.int32, device="cuda"), torch.arange(T // page, dtype=torch.int32, device="cuda")[None]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def time(n):
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda._sleep(4_000_000)           # some 2 ms: all launches are queued before the first runs
        begin.record()
        for _ in range(40):
            ops.rope_cache_write(qkv, n, positions, req, table, cos_sin, plane, plane.stride(0), page, Hq, Hkv, D, D, 1, True, err)
        end.record()
        torch.cuda.synchronize()
        return begin.elapsed_time(end)

    time(T)
    few, many = (min(time(n) for _ in range(7)) for n in (800, T))
    assert few < 0.87 * many           # (1.04 with the line, 0.72 without)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("E", [512, 2044, 2048, 4096, 4100, 5120, 6144, 8188, 8192, 8196])
def test_norm_of_many_rows_covers_the_width(cuda, dtype, E):
    """Widths on both sides of every change of the block's size: all of a row is normed, nothing beside it."""
    from ferrum_b200.ops import lib as ops
    g = torch.Generator(device="cuda").manual_seed(E)
    x, w = torch.randn(70, E, device="cuda", generator=g), torch.randn(E, device="cuda", generator=g)
    out = torch.full((71, E), 7.0, device="cuda", dtype=dtype)
    ops.rmsnorm(x, w, out, 1e-5, n_rows=70)
    v = x.double()
    want = v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5) * w.double()
    # a sum of squares in a tree of some 20 levels, a root, a division and two products; one rounding of the output type
    bound = want.abs() * (24 * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0))
    assert ((out[:70].double() - want).abs() <= bound).all() and (out[70] == 7).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,E", [(1, 4), (3, 1028), (64, 2048), (65, 2048), (592, 2048), (593, 2048), (64, 4096), (296, 4096), (297, 4096), (8, 4100), (64, 8192),
                                 (65, 8200), (2, 16384), (70, 16384), (1200, 2052)])
def test_norm_scaled_add_on_both_sides_of_its_lines(cuda, dtype, T, E):
    """Token counts and widths where the kernel changes pieces a thread, threads a block and the place its weights are read."""
    from ferrum_b200.ops import lib as ops
    g = torch.Generator(device="cuda").manual_seed(T + E)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, y, w, w2, out = r(T + 1, E), r(T, E), r(E), r(E), torch.full((T + 1, E), 7.0, device="cuda", dtype=dtype)
    norm = lambda v, eps: v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)
    add = 0.7 * norm(y.double(), 1e-5) * w.double()
    want = x[:T].double() + add
    alone, both = x.clone(), x.clone()
    ops.norm_scaled_add(alone, y, w, 0.7, 1e-5, T)
    ops.norm_scaled_add(both, y, w, 0.7, 1e-5, T, norm=(w2, 1e-6, out))
    assert torch.equal(alone, both) and torch.equal(alone[T], x[T]) and (out[T] == 7).all()
    # a sum of squares in some 20 levels, a root, a division and three products; then the same of the new rows
    assert ((alone[:T].double() - want).abs() <= (x[:T].abs().double() + add.abs()) * 24 * 2.0 ** -24).all()
    want = norm(alone[:T].double(), 1e-6) * w2.double()
    rounding = {torch.float32: 0.0, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype]
    assert ((out[:T].double() - want).abs() <= want.abs() * (24 * 2.0 ** -24 + rounding) + 1e-7).all()


@pytest.mark.parametrize("T,E,K,ctas", [(1, 1028, 256, 0), (8, 4096, 4096, 0), (40, 2048, 2048, 32), (64, 4096, 2048, 0), (100, 2048, 1024, 40), (100, 3588, 2048, 0), (8, 8192, 4096, 0),
                                        (128, 8192, 1024, 0)])
def test_norm_scaled_add_of_partials(cuda, T, E, K, ctas):
    """A product left in several partials a tile (widths that end inside a tile too) gives the bits of the same sums stored."""
    from ferrum_b200.ops import lib as ops
    g = torch.Generator(device="cuda").manual_seed(E + K)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    a, b = r(T, K).bfloat16(), (r(E, K) * 0.05).bfloat16()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    floats, _ = ops.gemm_tc_workspace(T, E, K, False)
    part = ops.gemm_tc_deferred(a, b, err, torch.empty(floats, device="cuda"), n_ctas=ctas)
    y = torch.zeros(T, E, device="cuda")
    ops.residual_reduce(y, T, part)
    assert ((y - a.float() @ b.float().T).abs() <= 1e-2 * y.std()).all() and err.item() == 0
    x, w, w2 = r(T, E), r(E), r(E)
    one, two, three = x.clone(), x.clone(), x.clone()
    out, out2 = (torch.empty(T, E, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    ops.norm_scaled_add(one, y, w, 0.7, 1e-5, T, norm=(w2, 1e-6, out))
    ops.norm_scaled_add(two, None, w, 0.7, 1e-5, T, partials=part)
    ops.norm_scaled_add(three, None, w, 0.7, 1e-5, T, partials=part, norm=(w2, 1e-6, out2))
    assert torch.equal(one, two) and torch.equal(one, three) and torch.equal(out, out2)
