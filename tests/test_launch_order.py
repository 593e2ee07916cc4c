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
    """The pair kernel (bn 0) triggers ahead of its own wait."""
    text = body("gemm_tc5.cu", "tc5_reduce_rope_kernel")
    assert 0 <= text.index("if (bn == 0) sb_pdl_wait()") < text.index("row_pos")


def with_tensor_memory():
    """(source, kernel) of every kernel that allocates tensor memory."""
    found = []
    for path in sorted(SRC_DIR.glob("*.cu*")):
        text = path.read_text()
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\(", text):
            if "tmem_alloc" in body(path.name, m.group(1)):
                found.append((path.name, m.group(1)))
    return found


def test_the_kernels_with_tensor_memory_are_found():
    assert {name for _, name in with_tensor_memory()} >= {
        "attn_prefill_tc5_kernel", "gemm_f32_tc5_kernel", "gemm_tc5_kernel", "gemm_tc5_persistent_kernel", "gemm_tc5_pair_kernel"}


@pytest.mark.parametrize("source,name", with_tensor_memory())
def test_successors_start_when_the_tensor_memory_is_taken(source, name):
    """A successor may take tensor memory ahead of its wait: on an SM where it came first, both would wait for good."""
    text = body(source, name)
    taken = text.index("__syncthreads()", text.index("tmem_alloc"))
    assert taken < text.index("sb_pdl_launch()")
