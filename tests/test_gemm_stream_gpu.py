"""The float32 product of up to four tokens: edges of its groups of features, slices of K and tokens, rows with a stride, all
epilogues; against float64, and bit for bit against the kernel that takes more tokens."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 3, 8, 9, 131, 1187, 2370])
@pytest.mark.parametrize("K", [4, 508, 512, 516, 3076])
def test_float32_product_of_a_few_tokens(cuda, N, K):
    from ferrum_b200.ops import lib as ops
    g = torch.Generator(device="cuda").manual_seed(N * 5 + K)
    xw, ww = torch.randn(8, K + 8, device="cuda", generator=g), torch.randn(N + 1, K + 4, device="cuda", generator=g)
    x, w = xw[:, 4:4 + K], ww[:N, :K]
    many = torch.zeros(8, N, device="cuda")
    ops.gemm_generic(x, w, many, ops.EPI_STORE)
    exact = x.double() @ w.double().T
    # a sum's error: one rounding a term of a thread's chain (four elements a slice), five of the lanes', three of the warps'
    bound = (4 * -(-K // 512) + 8) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    for M in (1, 2, 3, 4):
        out = torch.full((M + 1, N + 3), 7.0, device="cuda")
        ops.gemm_generic(x, w, out[:, 1:], ops.EPI_STORE, M=M)
        assert ((out[:M, 1:N + 1].double() - exact[:M]).abs() <= bound[:M]).all()
        assert torch.equal(out[:M, 1:N + 1], many[:M])
        assert (out[M] == 7).all() and (out[:, 0] == 7).all() and (out[:, N + 1:] == 7).all()
        acc = torch.full((M, N), 3.0, device="cuda")
        ops.gemm_generic(x, w, acc, ops.EPI_RESIDUAL, M=M)
        assert torch.equal(acc, many[:M] + 3.0)
        ops.gemm_generic(x, w, acc, ops.EPI_STORE_F32, M=M)
        assert torch.equal(acc, many[:M])


@pytest.mark.parametrize("N,K", [(9, 4), (131, 516), (1187, 3076)])
def test_float32_product_of_a_few_tokens_with_values_that_are_not_finite(cuda, N, K):
    """An infinity or NaN reaches the outputs of its own token and feature and no others: those are the bits of the finite operands."""
    from ferrum_b200.ops import lib as ops
    g = torch.Generator(device="cuda").manual_seed(N + K)
    x, w = torch.randn(4, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g)
    clean = torch.empty(4, N, device="cuda")
    ops.gemm_generic(x, w, clean, ops.EPI_STORE)
    bad_x, bad_w = x.clone(), w.clone()
    bad_x[1, K // 2], bad_x[3, 0], bad_x[3, K - 1] = float("inf"), float("inf"), float("-inf")
    bad_w[N // 3, K - 1], bad_w[N - 1, 0] = float("nan"), float("-inf")
    for M in (1, 2, 3, 4):
        out = torch.empty(M, N, device="cuda")
        ops.gemm_generic(bad_x, bad_w, out, ops.EPI_STORE, M=M)
        with_one = bad_x[:M].double() @ bad_w.double().T
        assert torch.equal(out.isnan(), with_one.isnan()) and torch.equal(out.isinf(), with_one.isinf())
        assert torch.equal(out[out.isinf()].double(), with_one[out.isinf()])
        fine = torch.isfinite(with_one)
        assert torch.equal(out[fine], clean[:M][fine])
