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
