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


@pytest.mark.parametrize("T", [65, 300, 1183, 1184])
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
