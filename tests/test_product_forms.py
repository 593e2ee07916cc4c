"""Which form a bfloat16 product takes: a rule on sizes that needs no device."""
import pytest

from sonicboom_b200 import ops

SMS = 148


@pytest.mark.parametrize("M", [65, 97, 128])
@pytest.mark.parametrize("N,K,epilogue,swapped", [
    (3584, 3584, ops.EPI_RESIDUAL, True), (4608, 3584, ops.EPI_BIAS, True), (1536, 8960, ops.EPI_NONE, True),      # K split
    (37888, 3584, ops.EPI_SWIGLU, True), (4096, 520, ops.EPI_SWIGLU, True),                     # gated, one wave of tiles
    (55296, 5120, ops.EPI_SWIGLU, False),                                                       # gated, more
    (152064, 3584, ops.EPI_NONE, False), (32768, 2048, ops.EPI_NONE, False), (4096, 520, ops.EPI_RESIDUAL, False),
    (192, 512, ops.EPI_NONE, False)])
def test_products_of_65_to_128_rows_stream_the_weights_only_where_that_is_faster(M, N, K, epilogue, swapped):
    l = ops.lib()
    assert bool(l.sb_gemm_tc5_swapped(M, N, K, SMS, epilogue)) == swapped
    assert (l.sb_gemm_tc5_scratch_bytes(M, N, K, SMS) > 0) == bool(swapped and epilogue != ops.EPI_SWIGLU)


def test_few_rows_always_and_many_never():
    for N, K in ((152064, 3584), (192, 512), (3584, 3584)):
        for epilogue in (ops.EPI_NONE, ops.EPI_SWIGLU):
            assert [ops.lib().sb_gemm_tc5_swapped(M, N, K, SMS, epilogue) for M in (1, 64, 129, 2048)] == [1, 1, 0, 0]
