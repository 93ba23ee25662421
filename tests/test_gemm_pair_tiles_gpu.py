"""The CTA-pair product at every width of its token tiles, whole and cut, against float64."""
import ctypes
import math

import pytest
import torch


def plan(ops, M, rows, K, pairs):
    out = (ctypes.c_int * 3)()
    ops.lib().ferrum_gemm_pair_plan(ctypes.c_int(M), ctypes.c_longlong(rows), ctypes.c_int(K), ctypes.c_int(pairs), out)
    return tuple(out)


# (M, N, K, CTAs, gate and up, tokens per tile, cut): tiles that end one token past and one short of a border of 32,
# features that end inside a tile, a K of one block and of many
CASES = [(321, 256, 8192, 12, False, 64, False), (161, 256, 8192, 12, True, 64, False), (257, 256, 8192, 38, False, 64, True), (193,
         256, 8192, 34, True, 64, True), (257, 256, 64, 32, False, 96, False), (129, 256, 64, 26, True, 96, False), (257,
         256, 8192, 22, False, 96, True), (129, 256, 8192, 36, True, 96, True), (321, 1280, 8192, 16, False, 128, False),
         (321, 256, 8192, 16, False, 128, True), (257, 320, 64, 8, False, 160, False), (129, 320, 64, 8, True, 160, False),
         (289, 256, 8192, 16, False, 160, True), (129, 256, 8192, 14, True, 160, True), (321, 320, 64, 8, False, 192, False),
         (513, 320, 8192, 10, False, 192, True), (385, 320, 64, 8, False, 224, False), (193, 320, 64, 10, True, 224, False),
         (193, 640, 8192, 8, True, 224, True), (449, 320, 64, 10, False, 256, False),
         (65, 320, 64, 8, False, 96, False), (65, 300, 200, 6, True, 96, False), (97, 640, 8192, 10, False, 160, False),
         (128, 500, 8192, 14, True, 160, False), (128, 256, 64, 4, False, 96, False)]


def test_plan_widths():
    """The cases below are cut as their comment says, and the tiles of every plan cover the tokens."""
    from ferrum_b200.ops import lib as ops
    for M, N, K, ctas, dual, bt, cut in CASES:
        got = plan(ops, M, 2 * N if dual else N, K, ctas // 2)
        assert got == (bt, -(-M // bt), int(cut)), (M, N, K, ctas, dual, got)
    for M in (65, 129, 257, 300, 512, 2048, 20000):
        for rows in (128, 3072, 28672):
            for pairs in (1, 5, 74):
                bt, tiles, _ = plan(ops, M, rows, 4096, pairs)
                assert 64 <= bt <= 256 and bt % 32 == 0 and (tiles - 1) * bt < M <= tiles * bt


@pytest.mark.gpu
@pytest.mark.parametrize("h16", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,ctas,dual,bt,cut", CASES)
def test_pair_tiles(M, N, K, ctas, dual, bt, cut, h16):
    from ferrum_b200.ops import lib as ops
    ops.require_cuda()
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, device="cuda", generator=g).to(h16)
    w = (torch.randn(2 * N if dual else N, K, device="cuda", generator=g) / math.sqrt(K)).to(h16)
    floats, tiles = ops.gemm_tc_workspace(M, N, K, dual, ctas)
    ws, cnt, err = torch.empty(floats, device="cuda"), torch.zeros(tiles, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ref = x.double() @ w.double().T
    # Float32 sums of exact products, 16 at a time: each of K / 16 additions cuts off at most 2^-23 of the partial sum, and
    # no partial sum of these independent terms passes eight standard deviations.
    absref = (K / 16 + 2) * 2.0 ** -23 * 8 * (x.double().square() @ w.double().square().T).sqrt()
    half = 2.0 ** (-8 if h16 == torch.bfloat16 else -11)                # rounding of a result to the type
    if dual:
        out = torch.full((M, N), float("nan"), device="cuda", dtype=h16)
        ops.gemm_tc(x, w, out, ops.TC_SWIGLU, err, ws, cnt, n_ctas=ctas, M=M, N=N, dual_offset=N)
        gate, up = ref[:, :N], ref[:, N:]
        want = torch.nn.functional.silu(gate) * up
        # |d silu| <= 1.1; the activation's own float32 rounding is within 2^-20 of its factors
        bound = 1.1 * absref[:, :N] * up.abs() + absref[:, N:] * gate.abs() + 2.0 ** -20 * gate.abs() * up.abs() + half * want.abs() + 2.0 ** -24
        assert ((out.double() - want).abs() <= bound).all()
    else:
        out = torch.full((M, N + 8), float("nan"), device="cuda", dtype=h16)
        ops.gemm_tc(x, w, out, ops.TC_STORE_BF16, err, ws, cnt, n_ctas=ctas)
        assert ((out[:, :N].double() - ref).abs() <= absref + half * ref.abs() + 2.0 ** -24).all()
        assert out[:, N:].isnan().all()
        res = torch.randn(M, N, device="cuda", generator=g)
        acc = res.clone()
        ops.gemm_tc(x, w, acc, ops.TC_RESIDUAL, err, ws, cnt, n_ctas=ctas)
        assert ((acc.double() - res.double() - ref).abs() <= absref + 2.0 ** -23 * acc.double().abs()).all()
        # float32 results, through the tensor map where rows are 16-byte multiples and by the threads where not: the same bits
        plain = [torch.full((M, N + pad), float("nan"), device="cuda") for pad in (4, 1)]
        for out in plain:
            ops.gemm_tc(x, w, out, ops.TC_STORE_F32, err, ws, cnt, n_ctas=ctas)
            assert out[:, N:].isnan().all()
        assert ((plain[0][:, :N].double() - ref).abs() <= absref).all() and torch.equal(plain[0][:, :N], plain[1][:, :N])
    assert err.item() == 0 and cnt.abs().sum().item() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("h16", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M", [64, 65, 128, 129])
@pytest.mark.parametrize("N,K", [(4096, 4096), (5000, 520), (3072, 8192)])
def test_residual_left_or_added(M, N, K, h16):
    """A residual sum that the layers leave in partials for the next kernel is the same bits where the product adds it itself."""
    from ferrum_b200.ops import lib as ops
    ops.require_cuda()
    assert ops.gemm_tc_should_defer(M, N, K, False) == (M <= 128)
    if M > 128:
        return
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w, h = torch.randn(M, K, device="cuda", generator=g).to(h16), torch.randn(N, K, device="cuda", generator=g).to(h16), torch.randn(M, N, device="cuda", generator=g)
    floats, tiles = ops.gemm_tc_workspace(M, N, K, False)
    ws, cnt, err = torch.empty(floats, device="cuda"), torch.zeros(tiles, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    left, added = h.clone(), h.clone()
    ops.residual_reduce(left, M, ops.gemm_tc_deferred(x, w, err, ws))
    ops.gemm_tc(x, w, added, ops.TC_RESIDUAL, err, ws, cnt)
    assert err.item() == 0 and torch.equal(left, added)
