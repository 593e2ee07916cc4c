"""What the prefill attention's overlapped launch relies on, read from the source."""
from test_launch_order import body


def test_the_next_kernel_starts_after_the_block_has_its_tensor_memory():
    """A product's block takes tensor memory before it waits for the kernel ahead of it: on the same SM it must not come first."""
    text = body("attn_tc5.cuh", "attn_prefill_tc5_kernel")
    assert 0 <= text.index("tmem_alloc(") < text.index("sb_pdl_launch()") < text.rindex("sb_pdl_wait()")
    assert text.count("sb_pdl_launch()") == 1
