"""The gated delta scan on the tensor cores against the plain rule in float64 and the FFMA form."""
import pytest
import torch

from sonicboom_b200 import ops
from test_gpu_sipilorn import delta_cache, delta_case, run_delta

pytestmark = pytest.mark.gpu


def forced(case, columns, cuts):
    """The mixer's rows and the memory they leave behind, with the scan that `columns` names."""
    ops.force_gated_delta_columns(columns)
    try:
        H, G, d, dv = case["sizes"]
        cache = delta_cache(H, G, d, dv, case["taps"], 2)
        slot, outs, at = cache.open(), [], 0
        for n in cuts:
            outs += run_delta(case, cache, [(slot, case["proj"][at:at + n])], "chunks")
            at += n
        return torch.cat(outs).double(), {k: t[slot].clone() for k, t in cache.state.items()}
    finally:
        ops.force_gated_delta_columns(0)


# one and several groups of 32 columns, shared and own keys, no convolution; whole chunks, a ragged last one, steps of less than one
@pytest.mark.parametrize("H,G,d,dv,taps", [(2, 1, 128, 32, 4), (3, 3, 64, 32, 1), (4, 2, 64, 96, 3), (2, 1, 128, 128, 4)])
@pytest.mark.parametrize("keys,decays", [("random", "mixed"), ("repeated", "slow"), ("random", "fast")])
def test_scan_on_the_tensor_cores(H, G, d, dv, taps, keys, decays):
    case, ref = delta_case(H, G, d, dv, taps, 301, 5, keys, decays)
    for cuts in ([301], [160, 1, 15, 17, 108]):
        want, ring = forced(case, 2, cuts)
        got, ring2 = forced(case, 1, cuts)
        err, err_ffma = float((got - ref).norm() / ref.norm()), float((want - ref).norm() / ref.norm())
        # operands of 22 bits and more, sums of 128 terms: both are float32 rounding of the same recurrence
        assert err < 1.5 * err_ffma + 1e-7, (err, err_ffma)
        for k in ring:
            if k != (0, "memory"):
                assert torch.equal(ring[k], ring2[k])
        a, b = ring[(0, "memory")].double(), ring2[(0, "memory")].double()
        assert float((a - b).norm() / a.norm()) < 1e-5


def test_blocks_choose_the_scan():
    """More blocks of 32 columns than SMs run on the tensor cores, no more do not."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for H, which in ((sms // 4 + 1, 1), (sms // 4, 2)):
        case, _ = delta_case(H, H, 64, 128, 2, 40, 1, "random", "slow")
        auto, forms = forced(case, 0, [40])[0], [forced(case, c, [40])[0] for c in (1, 2)]
        assert torch.equal(auto, forms[which - 1]) and not torch.equal(forms[0], forms[1])
