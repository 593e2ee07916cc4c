"""What the kernels' overlapped launches rely on, read from the sources: kernels read a step's plan ahead of their waits,
so the kernels that start a step let their successors start only after a wait of their own."""
import re

import pytest

from sonicboom_b200.csrc.build import SRC_DIR


def body(source, name):
    """The text of one kernel's body."""
    text = (SRC_DIR / source).read_text()
    at = text.index("{", re.search(rf"\b{name}\(", text).end())
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i]
    raise AssertionError(f"{name}: no end")


@pytest.mark.parametrize("source,name", [("elementwise.cu", "embed_kernel"), ("elementwise.cu", "embed_norm_kernel"),
                                         ("seq_rows.cu", "embed_pair_kernel")])
def test_the_first_kernel_of_a_step_waits_before_it_triggers(source, name):
    text = body(source, name)
    assert 0 <= text.index("sb_pdl_wait()") < text.index("sb_pdl_launch()")


def test_rotation_behind_the_pair_kernel_reads_positions_after_its_wait():
    """The pair kernel (bn 0) triggers at its first instruction."""
    text = body("gemm_tc5.cu", "tc5_reduce_rope_kernel")
    assert 0 <= text.index("if (bn == 0) sb_pdl_wait()") < text.index("row_pos")
