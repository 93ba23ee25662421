"""The tcgen05 attention of prompt portions with score scales that are not positive: masked keys stay masked, and the maximum
that the weights are taken against is that of the scaled scores."""
import numpy as np
import pytest
import torch

from test_kernels_gpu import ATT16, err_flag, ops, paged_setup  # noqa: F401  (ops is a fixture)

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(torch.int32).cuda()


@pytest.mark.parametrize("h16", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("scale", [-0.125, -1e-30, -0.0, 0.0, 1e-45])
@pytest.mark.parametrize("Hq,Hkv,D,window,kernel", [(4, 2, 64, 0, "single"), (8, 2, 128, 70, "single"), (8, 2, 128, 0, "wide"), (8, 2, 128, 0, "pair"),
                                                    (3, 3, 128, 90, "pair")])
def test_scales(ops, Hq, Hkv, D, window, kernel, scale, h16):
    from ferrum_b200.parts.attention_plan import build_host
    lens, qlens, ps = [137, 2600, 450], [137, 130, 450], 16      # whole prompts and a late portion, whose keys are split
    plane, table, ks, vs = paged_setup(lens, Hkv, D, ps, h16, 27)
    g = torch.Generator(device="cuda").manual_seed(28)
    q = torch.randn(sum(qlens), Hq * D, device="cuda", generator=g).to(h16)
    out = torch.full_like(q, float("nan"))
    pos0 = [n - ql for n, ql in zip(lens, qlens)]
    qs = np.concatenate([[0], np.cumsum(qlens)])
    req, e = np.repeat(np.arange(len(lens)), qlens), err_flag()
    ops.set_attention_pair_kernel(kernel == "pair")
    try:
        for h in build_host(qlens, pos0, Hq // Hkv, window, Hkv, ops.attention_tc_tokens(D, Hq // Hkv, ps, plane, plane.stride(0))):
            if h is None:
                continue
            assert h["kind"] == "tc"
            part_o, part_ml = torch.empty(max(1, h["n_slots"] * h["bm"] * D), device="cuda"), torch.empty(max(1, h["n_slots"] * h["bm"] * 2), device="cuda")
            ops.attention_tc(q, out, plane, plane.stride(0), ps, table, dev(qs), dev(pos0), dev(h["work"]), h["n_work"], part_o,
                             part_ml, Hq, Hkv, D, scale, window, e, wide_weights=kernel == "wide")
            if h["comb"].size:
                ops.attention_combine(out, part_o, part_ml, dev(qs), dev(req), dev(h["req_tile0"]), dev(h["tile_info"]),
                                      dev(h["comb"]), int(h["comb"].size), Hq, Hkv, D, h["bm"], 1)
    finally:
        ops.set_attention_pair_kernel(False)
    assert e.item() == 0
    for r, (n, ql) in enumerate(zip(lens, qlens)):
        qr = q[qs[r]:qs[r + 1]].double().view(ql, Hkv, Hq // Hkv, D)
        s = torch.einsum("thgd,shd->hgts", qr, ks[r].double()) * scale
        far = torch.arange(n - ql, n, device="cuda")[:, None] - torch.arange(n, device="cuda")[None]
        s = s.masked_fill((far < 0) | ((far >= window) if window else False), -torch.inf)
        ref = torch.einsum("hgts,shd->thgd", s.softmax(-1), vs[r].double()).reshape(ql, Hq * D)
        # as at positive scales: the weights and the result are rounded to 16 bits once each
        assert (out[qs[r]:qs[r + 1]].double() - ref).abs().max().item() <= ATT16[h16], r
