"""Products of up to 8 rows whose blocks stay for several groups of weight rows: the bits of the same product in pieces of less
than a wave, which a block per group computes."""
import pytest
import torch

from sonicboom_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# a warp's share of K of less than one K block, of five to seven in flight, of eight (a block a group), and of several parts; N with a ragged last group
@pytest.mark.parametrize("K", [8, 72, 200, 1280, 1536, 1800, 2048, 3584])
@pytest.mark.parametrize("N", [9488, 12008, 17920])
@pytest.mark.parametrize("M", [1, 5, 8])
def test_pieces_give_the_same_bits(M, N, K):
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(N, K, device=DEV, dtype=torch.bfloat16) * K ** -0.5
    bias, res = torch.randn(N, device=DEV, dtype=torch.bfloat16), torch.randn(M, N, device=DEV)
    pieces = [slice(i, min(i + 4096, N)) for i in range(0, N, 4096)]
    for epi in (ops.EPI_NONE, ops.EPI_BIAS, ops.EPI_RESIDUAL, ops.EPI_RELU2, ops.EPI_SWIGLU):
        gated = epi == ops.EPI_SWIGLU
        if gated and N % 16:
            continue
        for dt in (torch.float32, torch.bfloat16):
            if epi == ops.EPI_RESIDUAL and dt != torch.float32:      # refused: the residual sum is kept in float32
                continue

            def product(s):
                out = torch.empty(M, (s.stop - s.start) // (2 if gated else 1), device=DEV, dtype=dt)
                return ops.linear(a, w[s], out, epi, bias=bias[s].contiguous() if epi == ops.EPI_BIAS else None,
                                  residual=res[:, s].contiguous() if epi == ops.EPI_RESIDUAL else None, kernel="skinny")
            assert torch.equal(product(slice(0, N)), torch.cat([product(s) for s in pieces], dim=1)), (epi, dt)
    if N % 16 == 0:
        for kw in (dict(gate=(2.0, 1.5)), dict(gate_kind=ops.GATE_GELU_TANH)):
            def gated_product(s):
                out = torch.empty(M, (s.stop - s.start) // 2, device=DEV, dtype=torch.bfloat16)
                return ops.linear(a, w[s], out, ops.EPI_SWIGLU, kernel="skinny", **kw)
            assert torch.equal(gated_product(slice(0, N)), torch.cat([gated_product(s) for s in pieces], dim=1))
