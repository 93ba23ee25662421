"""Scratch buffers whose size follows a prompt portion by portion."""
import torch


def test_growth():
    """With a limit a buffer doubles up to it, so that a long prompt's portions move it a few times only; what no captured step reads
    leaves the generation alone."""
    from ferrum_b200.engine.batch import Scratch
    s = Scratch("cpu", guard=0)
    moves, at = 0, None
    for n in range(100, 16001, 100):
        v = s.get("rows", (n, 3), torch.int32, limit=12000 * 3, captured=False)
        assert v.shape == (n, 3) and v.is_contiguous()
        moves, at = moves + (v.data_ptr() != at), v.data_ptr()
        assert s.bytes() <= max(n, 12000) * 3 * 4
        if n == 12000:
            assert moves <= 8
    assert s.generation == 0
    s.get("rows", (16000, 3), torch.float32, limit=12000 * 3, captured=False)        # (another type begins anew)
    assert s.bytes() == 16000 * 3 * 4
    a = s.get("captured", (5,), torch.float32)
    assert s.generation == 1 and s.get("captured", (5,), torch.float32) is a
    s.get("captured", (6,), torch.float32)
    assert s.generation == 2 and s.bytes() == 16000 * 3 * 4 + 6 * 4                   # without a limit: what is asked for
    guarded = Scratch("cpu", guard=4)
    for n in (10, 20):
        guarded.get("rows", (n,), torch.int32, limit=100, captured=False)
        assert guarded.bytes() == n * 4 and guarded.check() == []


def test_split_scratch_follows_the_step():
    """The float32 product's scratch stops growing at the step's token limit."""
    from ferrum_b200.engine.batch import StepContext
    from ferrum_b200.ops import lib as ops
    ctx = StepContext("cpu", 2048, 4, [])
    moves = []
    for M in range(65, 2049, 31):
        before = ctx.scratch.generation
        parts, partials = ctx.gemm_split_scratch(M, 3072, 3072)
        assert (parts.numel(), partials.numel()) == ops.gemm_split_workspace(M, 3072, 3072)
        moves.append(ctx.scratch.generation - before)
    assert sum(moves) <= 2 * 6
    assert ctx.scratch.bytes() <= 4 * sum(ops.gemm_split_workspace(2048, 3072, 3072))
