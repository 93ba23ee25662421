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
