"""What the prefill attention's overlapped launch relies on, read from the source."""
import pytest
import torch

from sonicboom_b200 import ops
from sonicboom_b200.cache import Cache, KVNeed
from sonicboom_b200.engine.step import StepEntry, StepPlan
from test_launch_order import body


def test_the_next_kernel_starts_after_the_block_has_its_tensor_memory():
    """A product's block takes tensor memory before it waits for the kernel ahead of it: on the same SM it must not come first."""
    text = body("attn_tc5.cuh", "attn_prefill_tc5_kernel")
    assert 0 <= text.index("tmem_alloc(") < text.index("sb_pdl_launch()") < text.rindex("sb_pdl_wait()")
    assert text.count("sb_pdl_launch()") == 1


def test_the_plan_is_read_after_the_wait():
    """A caller may write the plan with the kernel right before, one that triggers at its first instruction."""
    text = body("attn_tc5.cuh", "attn_prefill_tc5_kernel")
    for name in ("p.seq_row0", "p.seq_pos0", "p.page_off", "p.page_ids"):
        assert text.rindex("sb_pdl_wait()") < text.index(name), name


@pytest.mark.gpu
@pytest.mark.parametrize("hq,hkv,hd", [(28, 4, 128), (8, 2, 64)])
def test_positions_moved_by_the_kernel_right_before(hq, hkv, hd):
    torch.manual_seed(hd)
    lens, ahead = [300, 1, 129], [64, 700, 62]
    cache = Cache([KVNeed(hkv, hd, 0)], [None], 2048, torch.bfloat16, "cuda:0")
    storage = cache.groups[0].entry_storage(0)
    storage.normal_()
    entries = []
    for n, at in zip(lens, ahead):
        slot = cache.open()
        cache.reserve(slot, at + n + 1)
        cache.advance(slot, at)
        entries.append(StepEntry(slot, [0] * n, []))
    plan = StepPlan(cache, entries, "cuda:0")
    plan.max_len += 1
    rows = sum(lens)
    q = torch.randn(rows, hq, hd, device="cuda:0").bfloat16()
    a = torch.randn(2048, 4096, device="cuda:0").bfloat16()
    busy = torch.empty(2048, 2048, device="cuda:0")

    def run(move):
        start = torch.tensor(ahead, dtype=torch.int32, device="cuda:0")
        last, out = start + 1, torch.empty(rows, hq * hd, device="cuda:0", dtype=torch.bfloat16)
        plan.seq_pos0.copy_(start if move else last)
        torch.cuda.synchronize()
        for _ in range(4):                                  # the attention is launched while these still run
            ops.linear(a, a, busy)
        if move:
            ops.advance_rows(plan.seq_pos0, last)
        return ops.attention(q, out, plan, 0, storage, hq, hkv, hd, 0, hd ** -0.5)
    assert torch.equal(run(False), run(True))
