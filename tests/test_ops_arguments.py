"""Sizes that are integers but no Python ints (numpy scalars, as plans and tables hand them out) are taken by the wrappers and the
library's entry points."""
import ctypes

import numpy as np
import pytest
import torch


def test_entry_point_sizes():
    from ferrum_b200.ops import lib as ops
    can = ops.lib().ferrum_gemm_tc_can_defer
    for M, N, K in ((8, 4096, 4096), (300, 4096, 4096)):
        assert can(np.int64(M), np.int32(N), K, np.int8(0), np.uint16(148)) == can(M, N, K, 0, 148) == int(M == 8)
    assert ops.gemm_tc_workspace(np.int64(8), np.int64(4096), 4096, False) == ops.gemm_tc_workspace(8, 4096, 4096, False)
    with pytest.raises(TypeError):
        can(8.0, 4096, 4096, 0, 148)
    n = ctypes.c_int()
    ops.lib().ferrum_gemm_tc_workspace(np.int64(8), 4096, 4096, 0, 148, ctypes.byref(n))
    assert n.value == 32


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [np.int64, np.int32, lambda n: torch.tensor(n)])
def test_wrapper_sizes(kind):
    from ferrum_b200.ops import lib as ops
    ops.require_cuda()
    g = torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    x, w, gu = rand(5, 256), rand(64, 256), rand(5, 512).bfloat16()
    xb, wb, scale = x.bfloat16(), w.bfloat16(), rand(256)
    floats, tiles = ops.gemm_tc_workspace(5, 64, 256, False)
    ws, cnt = torch.empty(floats, device="cuda"), torch.zeros(tiles, dtype=torch.int32, device="cuda")
    logits, ids = rand(5, 64), torch.zeros(6, dtype=torch.int32, device="cuda")

    def results(n):
        a, b, c, d = (torch.zeros(5, n_cols, device="cuda", dtype=dt) for n_cols, dt in ((64, torch.float32), (64, torch.bfloat16), (256, torch.bfloat16), (256, torch.bfloat16)))
        ops.gemm_generic(x, w, a, ops.EPI_STORE_F32, M=n(5))
        ops.gemm_tc(xb, wb, b, ops.TC_STORE_BF16, err, ws, cnt, M=n(5), N=n(64))
        ops.rmsnorm(x, scale, c, 1e-5, n_rows=n(5))
        ops.swiglu(gu, d, n(5), n(256))
        ops.sample(logits, n(5), ids, err)
        assert err.item() == 0
        return a, b, c, d, ids.clone()
    for got, want in zip(results(kind), results(int)):
        assert torch.equal(got, want)
