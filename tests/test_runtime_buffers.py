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


@pytest.mark.parametrize("moved,taps", [(None, 4), ("conv_bias", 4), ("conv", 1), ("state", 4)])
def test_state_space_rows_for_chunks_start_on_16_bytes(moved, taps):
    """The kernel that makes them takes nothing else; weights and states from elsewhere in a buffer go token by token."""
    from types import SimpleNamespace

    from ccinfer_b200.parts import SelectiveStateSpace
    part = SelectiveStateSpace(64, 4, 32, 64, 2, taps, 2, 1e-5,
                               {k: k for k in ("in", "conv", "conv_bias", "dt_bias", "A_log", "D", "norm", "o")})
    shapes = {s.name: s.shape for s in part.tensor_specs()}

    def place(name, shape, dtype):
        n = torch.Size(shape).numel()
        return torch.zeros(n + 1, dtype=dtype)[1:].view(shape) if name == moved else torch.zeros(shape, dtype=dtype)

    bf = torch.bfloat16
    part.bind(SimpleNamespace(dtype=bf, device="cpu"), lambda n: place(n, shapes[n], bf if n in ("in", "o") else torch.float32))
    conv = place("state", (3, max(taps - 1, 1), part.conv_width), bf)
    assert kernels.ssm_chunks_fits(bf, 64, 32, 200, 4 * 200)
    assert part.runs_in_chunks(conv, 200, 4 * 200) == (moved is None)
    assert not part.runs_in_chunks(conv, 20, 4 * 20)


def test_latent_portions_run_over_made_keys_where_that_is_shorter():
    """(rows seen, tokens brought by each portion, heads of 192 columns)"""
    def pays(rows, tokens, heads):
        return kernels.latent_dense_pays(rows, tokens, heads, 192)

    assert not pays([128], [32], 32) and not pays([640] * 4, [24] * 4, 16)   # short walks: the layer waits for its launches
    assert pays([768], [2], 16) and pays([128, 768], [64, 2], 16) and pays([6016], [2], 32)
    assert pays([512] * 4, [100] * 4, 32) and pays([256], [192], 1)          # many tokens, or one portion of many
    assert not pays([128] + [2048] * 15, [32] + [2] * 15, 32)                # many portions that see much
    assert not pays([4224] * 15, [2] * 15, 32)                               # ... its heads in groups
    assert pays([128] + [4224] * 4, [32] + [2] * 4, 32) and pays([128] + [16128] * 4, [32] + [2] * 4, 32)
    assert not pays([32768, 32768, 128], [400] * 3, 32)                      # more rows than the buffers hold


def test_experts_of_few_tokens_keep_the_tiles_that_suit_them():
    """(hidden, F, experts, chosen, tokens): 16 rows a tile until the chosen weights fill the pairs of SMs."""
    from ccinfer_b200.parts import MixtureOfExperts

    def rows(D, F, E, top, T, dtype=torch.bfloat16):
        return MixtureOfExperts(D, E, top, F, {"router": "r", "gate": "g{e}", "up": "u{e}", "down": "d{e}"},
                                activation="swiglu").tile_rows(T, dtype)

    for D, F, E, top, T in ((2048, 1024, 32, 4, 4), (2048, 768, 64, 8, 2), (4096, 1024, 8, 2, 4), (4096, 512, 16, 2, 6),
                            (2048, 2048, 32, 4, 1), (1024, 512, 32, 4, 32)):
        assert rows(D, F, E, top, T) == 16
    for D, F, E, top, T in ((4096, 3072, 32, 4, 1), (2048, 2048, 32, 4, 2), (2048, 1024, 32, 4, 5), (4096, 1024, 8, 2, 6), (2048, 768, 64, 8, 3), (4096, 512, 16, 2, 8),
                            (2048, 256, 64, 6, 8), (1024, 512, 32, 4, 64)):
        assert rows(D, F, E, top, T) == 64
        assert rows(D, F, E, top, T, torch.float32) == 16
    assert rows(4096, 3072, 32, 4, 192) == 320


def test_pages_leave_room_for_what_comes_late(monkeypatch):
    """With kv_memory_fraction the pools share what is free beside the buffers that a long prompt will ask for."""
    from types import SimpleNamespace

    from ccinfer_b200.engine.engine import Engine, EngineOptions
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device: (1 << 30, 2 << 30))
    opt = EngineOptions(page_size=16, kv_memory_fraction=0.5)
    me = SimpleNamespace(rt=SimpleNamespace(device="cuda:0"))
    for late in (0, 1 << 28, 1 << 31):
        pages, = Engine._pages_per_group(me, opt, [("all",)], [None], [1024], late)
        assert pages == max(1, max(0, (1 << 30) - late) // 2 // (16 * 1024))


@pytest.mark.gpu
def test_one_buffer_for_portions_of_any_length():
    rt = Runtime("cuda:0", torch.bfloat16, 64, 4)
    small = rt.late("seen", 1 << 16, torch.bfloat16)
    assert rt.late("seen", 1 << 10, torch.bfloat16).data_ptr() == small.data_ptr()
    before = rt.scratch_bytes()
    assert rt.late("seen", 1 << 20, torch.bfloat16).numel() >= 1 << 20
    assert rt.scratch_bytes() - before == (1 << 21) - (1 << 17)   # the larger one alone
