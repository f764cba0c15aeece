"""The scratch pool's views, the buffers that only portions of prompts ask for, and the rules that choose chunks (CPU)."""
import pytest
import torch

from ccinfer_b200 import kernels
from ccinfer_b200.engine.runtime import Runtime, ScratchPool
from ccinfer_b200.errors import ScratchMoved


def test_scratch_views_follow_their_buffer():
    pool = ScratchPool("cpu")
    a = pool.get("x", (4, 8), torch.float32)
    assert pool.get("x", (4, 8), torch.float32) is a            # looked up, not made again
    b = pool.get("x", (2, 8), torch.float32)
    assert b.shape == (2, 8) and b.data_ptr() == a.data_ptr()
    assert pool.get("x", (4, 8), torch.float32).data_ptr() == a.data_ptr()
    c = pool.get("x", (16, 8), torch.float32)                   # larger: storage of its own, also for the old shape
    assert c.data_ptr() != a.data_ptr() and pool.get("x", (4, 8), torch.float32).data_ptr() == c.data_ptr()
    assert pool.get("x", (4, 8), torch.bfloat16).dtype == torch.bfloat16
    pool.freeze()
    assert pool.get("x", (16, 8), torch.float32).data_ptr() == c.data_ptr()
    with pytest.raises(ScratchMoved):
        pool.get("x", (17, 8), torch.float32)


def test_portions_run_in_chunks_where_the_layer_gains():
    """Few tokens of few heads wait for the launches of their layer: token by token, which launches less."""
    bf = torch.bfloat16

    def linear(portions, tokens, heads, dtype=bf, dk=128, dv=128):
        return kernels.chunk_recurrence_fits(dtype, dk, dv, tokens, portions * tokens * heads, False)

    def delta(portions, tokens, heads):
        return kernels.chunk_recurrence_fits(bf, 128, 128, tokens, portions * tokens * heads, True)

    def space(portions, tokens, heads):
        return kernels.ssm_chunks_fits(bf, 128, 64, tokens, portions * tokens * heads)

    assert not linear(2, 24, 16) and not linear(1, 128, 16) and not linear(16, 8, 32) and not linear(16, 11, 32)
    assert linear(2, 128, 16) and linear(1, 160, 1) and linear(16, 12, 32)
    assert not linear(4, 512, 16, torch.float32) and not linear(4, 512, 16, dk=96) and not linear(4, 512, 16, dv=48)
    assert not delta(1, 64, 32) and not delta(16, 31, 32) and delta(4, 64, 32) and delta(16, 32, 32) and delta(1, 160, 4)
    assert not space(1, 40, 64) and not space(16, 19, 128) and space(16, 20, 128) and space(2, 64, 64)
    assert not kernels.ssm_chunks_fits(bf, 96, 64, 512, 1 << 20) and not kernels.ssm_chunks_fits(bf, 64, 24, 512, 1 << 20)
