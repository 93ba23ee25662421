"""The float32 product on the tensor cores (csrc/kernels/gemm_split.cu) against float64 and against the CUDA cores' kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from ferrum_b200.ops import lib
    lib.require_cuda()
    return lib


def run(ops, x, w, M=None, add=None):
    M = x.shape[0] if M is None else M
    N, K = w.shape
    parts, partials = ops.gemm_split_workspace(M, N, K)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = add.clone() if add is not None else torch.full((M, N), float("nan"), device="cuda")
    ops.gemm_split(x, w, out, err, torch.empty(parts, device="cuda"), torch.empty(partials, device="cuda"), M=M, add=add is not None)
    assert err.item() == 0
    return out


# Edges: one token and the largest tile, a tile more; features and K that end inside a tile, a piece and 16 elements;
# one range of K and several (their number follows from N and K), also where rows are no multiples of 16 bytes apart.
@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (9, 2048, 2048), (16, 130, 1024), (65, 200, 520), (112, 127, 1032), (113, 1001, 512),
                                   (128, 129, 8), (129, 256, 4104), (300, 384, 3072), (257, 19000, 512), (2048, 128, 128)])
def test_gemm_split(ops, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randn(N, K, device="cuda", generator=g)
    ref = x.double() @ w.double().T
    # Of |x| |w|: 2^-24 for the products left out, 2^-22 for the matrix unit's cut-offs within a piece, half an ulp for
    # every piece and range that is added.
    bound = (x.double().abs() @ w.double().abs().T) * (2.0 ** -24 + 2.0 ** -22 + (K // 64 + 9) * 2.0 ** -24)
    out = run(ops, x, w)
    assert ((out.double() - ref).abs() <= bound).all()
    res = torch.randn(M, N, device="cuda", generator=g)
    total = run(ops, x, w, add=res)
    assert ((total.double() - res.double() - ref).abs() <= bound + 2.0 ** -24 * total.double().abs()).all()
    if ops.gemm_split_supported(x, w, M):       # where it stands in for the tiled kernel it is the closer of the two
        plain = torch.empty(M, N, device="cuda")
        ops.gemm_generic(x, w, plain, ops.EPI_STORE_F32)
        assert (out.double() - ref).norm() <= (plain.double() - ref).norm()
    # a token's result does not depend on the tokens beside it, nor on the row stride
    pick = [M - 1] + [i for i in (0, 3, 7) if i < M - 1]
    wide = torch.randn(len(pick), K + 12, device="cuda", generator=g)
    wide[:, :K] = x[pick]
    assert torch.equal(run(ops, wide[:, :K], w), out[pick])


@pytest.mark.parametrize("K", [512, 3072])
@pytest.mark.parametrize("kind", ["any", "long"])
def test_gemm_split_one_sign(ops, K, kind):
    """Where all products are positive nothing that is left out or cut off cancels: the error stays near half an ulp (2^-24) of the
    result and as much for the matrix unit's cut-offs.  "long": all lower bits of a significand set but for the last few, which makes
    the parts that are left out as large as they get."""
    g = torch.Generator(device="cuda").manual_seed(K)
    x, w = (torch.randn(n, K, device="cuda", generator=g).abs() for n in (300, 1024))
    if kind == "long":
        draw = lambda t, n: torch.randint(0, n, t.shape, device="cuda", generator=g)
        x, w = ((0x3F80FF00 + draw(t, 256) + (draw(t, 128) << 16)).to(torch.int32).view(torch.float32) for t in (x, w))
    ref = x.double() @ w.double().T
    assert ((run(ops, x, w).double() - ref).norm() / ref.norm()).item() <= 2.0 ** -23


def test_gemm_split_values(ops):
    """Large and small magnitudes keep their relative error."""
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(70, 1024, device="cuda", generator=g) * 1e18
    w = torch.randn(256, 1024, device="cuda", generator=g) * 1e-22
    ref = x.double() @ w.double().T
    assert ((run(ops, x, w).double() - ref).abs() <= (x.double().abs() @ w.double().abs().T) * 2.0 ** -20).all()
    # at the lower end of float32, subnormal operands among them, the three parts are still exact (an output may be subnormal itself:
    # half of its last place, 2^-150, comes on top); at the upper end the outputs are summed again plainly
    for up, down in ((1.0, 1e-36), (1e-33, 1e2), (1.0, 1e-38), (3e-39, 1e3), (1e30, 1e-37), (1e32, 1.0), (1e-3, 1e33), (1e13, 1e13)):
        a, b = (x.double() * (up * 1e-18)).float(), (w.double() * (down * 1e22)).float()
        ref = a.double() @ b.double().T
        assert ((run(ops, a, b).double() - ref).abs() <= (a.double().abs() @ b.double().abs().T) * 2.0 ** -18 + 2.0 ** -150).all(), (up, down)


# One range of K and several; features that end inside a quad, a warp's eight and a tile; more tokens than a tile.
@pytest.mark.parametrize("M,N,K", [(70, 256, 1024), (70, 250, 1032), (70, 1001, 512), (140, 9500, 1024), (65, 128, 8)])
@pytest.mark.parametrize("add", [False, True])
def test_gemm_split_not_finite(ops, M, N, K, add):
    """What is not finite comes out as the CUDA cores' kernel gives it: single elements, whole rows of tokens and of weights, sums that
    overflow."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x, w = torch.randn(M, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g)
    inf, nan = float("inf"), float("nan")
    x[3, K // 3], x[9, K - 1], x[20, 5], x[20, 6] = inf, -inf, nan, 2.0
    w[100, K // 2], w[7, K - 4], w[N - 1, 0] = inf, torch.tensor(0x7F800001, dtype=torch.int32).view(torch.float32).item(), -inf
    w[50, 3] = 3.4e38
    x[30] = 0.0
    x[31, 3] = 3.4e38
    w[60] = 0.0
    x[40], x[41], x[42], w[70], w[71] = nan, inf, -inf, nan, inf
    x[43, ::2], x[43, 1::2] = inf, 1.0
    x[44] = x[44].abs() * 1e36      # (overflows with w[72] only, in whatever order the terms are added)
    w[72] = w[72].abs() * 1e4
    x[M - 1, 0] = nan
    start = torch.randn(M, N, device="cuda", generator=g) if add else None
    got, want = run(ops, x, w, add=start), start.clone() if add else torch.empty(M, N, device="cuda")
    ops.gemm_generic(x, w, want, ops.EPI_RESIDUAL if add else ops.EPI_STORE_F32)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    inf = want.isinf()
    assert torch.equal(got[inf], want[inf])
    fine = want.isfinite()
    scale = x.nan_to_num(0, 0, 0).double().abs() @ w.nan_to_num(0, 0, 0).double().abs().T
    assert ((got - want).abs()[fine].double() <= 2.0 ** -14 * scale[fine] + 2.0 ** -22).all()


def test_gemm_split_linear(ops):
    """The layers' entry point takes this kernel where its rule says so, and both lanes' scratch is their own."""
    from ferrum_b200.engine.batch import StepContext
    from ferrum_b200.parts.linear import RESIDUAL, STORE, linear
    ctx = StepContext("cuda", 128, 4, [])
    g = torch.Generator(device="cuda").manual_seed(6)
    for M, N, K, split in ((64, 2048, 2048, False), (65, 2048, 2048, True), (65, 128, 512, True), (65, 127, 512, False), (65, 128, 508, False)):
        x = torch.randn(M, K, device="cuda", generator=g)
        w = torch.randn(N, K, device="cuda", generator=g)
        assert ops.gemm_split_supported(x, w, M) == split
        out = torch.zeros(M, N, device="cuda")
        linear(x, w, out, STORE, ctx, M=M)
        linear(x, w, out, RESIDUAL, ctx, M=M)
        assert ((out.double() - 2 * (x.double() @ w.double().T)).abs() <= 2.5e-7 * K * out.abs().max()).all()
    assert ctx.err.item() == 0
    a = ctx.gemm_split_scratch(65, 2048, 2048)
    ctx.lane = 1
    b = ctx.gemm_split_scratch(65, 2048, 2048)
    assert {t.data_ptr() for t in a}.isdisjoint({t.data_ptr() for t in b})
