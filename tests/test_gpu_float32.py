"""The float32 path's own kernels at the edges of their forms, against float64 and against the plain kernels."""
import pytest
import torch

import plain_model as pm
from sonicboom_b200 import ops
from sonicboom_b200.cache.kv import Cache, KVNeed
from sonicboom_b200.engine.step import StepEntry, StepPlan

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=0, scale=1.0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).mul_(scale).to(DEV)


# rows: one to 32 stream the weights (1, 2, 4 and groups of 8), 33 on are tiled at a K below 256 and run on the tensor
# cores from there on; K: one lane's 16 bytes, less and more than a warp's 128 values, odd numbers of K tiles; N: less than a
# block's rows or columns
@pytest.mark.parametrize("M", [1, 2, 3, 5, 8, 9, 32, 33, 48, 81, 112, 129, 201])
@pytest.mark.parametrize("N,K", [(16, 4), (48, 132), (1536, 1540), (272, 8960), (130, 100)])
def test_products(M, N, K):
    a, w, bias, res = rnd(M, K), rnd(N, K, seed=1, scale=K ** -0.5), rnd(N, seed=2), rnd(M, N, seed=3)
    y = a.double() @ w.double().T
    for epi, dtype in [(ops.EPI_NONE, torch.float32), (ops.EPI_BIAS, torch.float32), (ops.EPI_RESIDUAL, torch.float32),
                       (ops.EPI_RELU2, torch.float32), (ops.EPI_SWIGLU, torch.float32), (ops.EPI_NONE, torch.bfloat16)]:
        if epi == ops.EPI_SWIGLU and N % 16:
            continue
        want = {ops.EPI_BIAS: y + bias.double(), ops.EPI_RESIDUAL: y + res.double(), ops.EPI_RELU2: y.clamp(min=0) ** 2}.get(epi, y)
        if epi == ops.EPI_SWIGLU:
            z = y.view(M, -1, 2, 8)
            want = (torch.nn.functional.silu(z[:, :, 0]) * z[:, :, 1]).reshape(M, N // 2)
        errs = []
        for kernel in ("auto", "plain"):
            out = res.clone() if epi == ops.EPI_RESIDUAL else torch.full(want.shape, float("nan"), device=DEV, dtype=dtype)
            ops.linear(a, w, out, epi, bias=bias if epi == ops.EPI_BIAS else None,
                       residual=out if epi == ops.EPI_RESIDUAL else None, kernel=kernel)
            errs.append(float((out.double() - want).norm() / want.norm()))
        # sums of K terms that are rounded one after the other are off by about sqrt(K) / 2 * 2^-24 of their terms'
        # root mean square sum, squared or multiplied by about twice that
        assert errs[0] < (2 ** -8 if dtype == torch.bfloat16 else (K ** 0.5 + 8) * 2 ** -24 * 2), (epi, errs)
        assert errs[0] <= 1.3 * errs[1] + 2 ** -24, (epi, errs)     # and no more than the plain kernel's


@pytest.mark.parametrize("M,N,K", [(3, 40, 64), (33, 40, 64), (40, 272, 512), (201, 1536, 1540)])
def test_plain_is_the_plain_kernel(M, N, K):
    """Every output one chain over K, to the bit, in float32 as in the sums of bfloat16 operands of the same values; and at an
    address off 16 bytes, where "auto" takes it too."""
    a, w = rnd(M, K).bfloat16(), rnd(N, K, seed=1).bfloat16()
    got = [torch.empty(M, N, device=DEV) for _ in range(3)]
    ops.linear(a, w, got[0], kernel="plain")
    ops.linear(a.float(), w.float(), got[1], kernel="plain")
    off = torch.empty(M * K + 1, device=DEV)[1:].view(M, K)
    ops.linear(off.copy_(a), w.float(), got[2])
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("N,K", [(1536, 1536), (8960, 1536), (640, 8960), (512, 192)])
def test_products_of_a_row_in_batches_of_any_size(N, K):
    """The first rows alone and among more, over every change of form and of the number of blocks that share K: the same to
    rounding (each is off by the bound of `test_products`), and to the bit among up to 16 rows."""
    a, w = rnd(1000, K), rnd(N, K, seed=1)
    want = a.double() @ w.double().T
    outs = {}
    for M in (1, 3, 8, 16, 17, 32, 33, 64, 224, 225, 449, 1000):
        outs[M] = torch.empty(M, N, device=DEV)
        ops.linear(a[:M].contiguous(), w, outs[M])
    for M, out in outs.items():
        n = min(M, 3)
        diff = float((out[:n] - outs[1000][:n]).norm() / want[:n].norm())
        assert diff < (K ** 0.5 + 8) * 2 ** -24 * 4, (M, diff)
        if M <= 16:
            assert torch.equal(out, outs[16][:M])


# tiles of 128, 64 and 32 rows (the largest that gives each of 148 SMs a block), rows and columns that end inside a tile, K of
# one 16-byte column, of whole and of ragged tiles of 16
@pytest.mark.parametrize("M,N,tile", [(1000, 2400, 128), (897, 2450, 128), (500, 2400, 64), (1000, 1160, 64), (33, 130, 32), (97, 1536, 32)])
@pytest.mark.parametrize("K", [4, 48, 132, 252])
def test_tiled_products(M, N, tile, K):
    """Every output one chain over K, as the plain kernel adds it: the same bits."""
    blocks = lambda t: -(-M // t) * -(-N // 128)                               # noqa: E731
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms == 148:
        assert tile == next((t for t in (128, 64) if blocks(t) >= sms), 32)
    a, w, bias, res = rnd(M, K), rnd(N, K, seed=1), rnd(N, seed=2), rnd(M, N, seed=3)
    for epi, dtype in [(ops.EPI_NONE, torch.float32), (ops.EPI_BIAS, torch.float32), (ops.EPI_RESIDUAL, torch.float32),
                       (ops.EPI_RELU2, torch.float32), (ops.EPI_SWIGLU, torch.float32), (ops.EPI_BIAS, torch.bfloat16)]:
        if epi == ops.EPI_SWIGLU and N % 16:
            continue
        got = []
        for kernel in ("auto", "plain"):
            out = res.clone() if epi == ops.EPI_RESIDUAL else \
                torch.full((M, N // 2 if epi == ops.EPI_SWIGLU else N), float("nan"), device=DEV, dtype=dtype)
            ops.linear(a, w, out, epi, bias=bias if epi == ops.EPI_BIAS else None, residual=out if epi == ops.EPI_RESIDUAL else None,
                       kernel=kernel)
            got.append(out)
        assert torch.equal(got[0], got[1]) and bool(got[0].isfinite().all()), epi


# the tensor-core form: token tiles of 32 to 224, one more than a tile, three tiles; K of its least, with a ragged last stage, shared by
# a cluster; weight rows that end inside a tile; 17 rows of a wide product
@pytest.mark.parametrize("M,N,K", [(17, 8208, 256), (33, 8, 256), (64, 130, 260), (97, 1536, 1540), (128, 272, 8960), (193, 2048, 1536),
                                   (224, 400, 1024), (225, 136, 516), (449, 1000, 300), (672, 16, 4100)])
@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e12])
def test_products_of_split_operands(M, N, K, scale):
    a, w, bias, res = rnd(M, K, scale=scale), rnd(N, K, seed=1, scale=K ** -0.5), rnd(N, seed=2, scale=scale), rnd(M, N, seed=3, scale=scale)
    y = a.double() @ w.double().T
    for epi in (ops.EPI_NONE, ops.EPI_BIAS, ops.EPI_RESIDUAL, ops.EPI_RELU2, ops.EPI_SWIGLU):
        if epi == ops.EPI_SWIGLU and N % 16:
            continue
        want = {ops.EPI_BIAS: y + bias.double(), ops.EPI_RESIDUAL: y + res.double(), ops.EPI_RELU2: y.clamp(min=0) ** 2}.get(epi, y)
        if epi == ops.EPI_SWIGLU:
            z = y.view(M, -1, 2, 8)
            want = (torch.nn.functional.silu(z[:, :, 0]) * z[:, :, 1]).reshape(M, N // 2)
        out = res.clone() if epi == ops.EPI_RESIDUAL else torch.full(want.shape, float("nan"), device=DEV)
        ops.linear(a, w, out, epi, bias=bias if epi == ops.EPI_BIAS else None, residual=out if epi == ops.EPI_RESIDUAL else None)
        # an operand is off by up to 2^-22, a sum's roundings by a few 2^-24; squares and products of two sums by twice that; a
        # gate's exponential by 2^-24 of the gate's size, which at 1e12 matters for the gates that are within 100 of 0, next to none
        err = float((out.double() - want).norm() / want.norm())
        assert bool(out.isfinite().all()) and err < 2 ** -20, (epi, err)
    assert ops.tc5_status() == 0


# operands scaled by powers of two down to the subnormal range: rows, weights; rows of ordinary size, of zeros and of tiny values side
# by side (None)
@pytest.mark.parametrize("ea,ew", [(-60, 0), (-72, 0), (-100, 0), (-110, 0), (-116, 0), (-126, 0), (-130, 0), (-70, -70), (-110, 20), (0, -120),
                                   (20, -126), (None, 0), (None, -60)])
@pytest.mark.parametrize("M,N,K", [(40, 144, 512), (225, 136, 1028)])
def test_split_operands_of_any_size(M, N, K, ea, ew):
    """As close to 64 bits as the plain kernel, row by row."""
    a, w = rnd(M, K), rnd(N, K, seed=1).mul_(2.0 ** ew)
    if ea is None:
        sizes = torch.tensor([0.0, 2.0 ** -120, 1.0, 2.0 ** -50, 0.0, 2.0 ** -90, 2.0 ** 30], device=DEV)
        a *= sizes[torch.arange(M, device=DEV) % len(sizes)][:, None]
    else:
        a *= 2.0 ** (ea / 2)
        a *= 2.0 ** (ea - ea / 2)
    want = a.double() @ w.double().T
    err = []
    for kernel in ("auto", "plain"):
        out = torch.full((M, N), float("nan"), device=DEV)
        ops.linear(a, w, out, kernel=kernel)
        err.append((out.double() - want).norm(dim=1))
    # 2^-22 of an operand, a few 2^-24 of the sums, half a unit of the subnormal range for each
    assert bool((err[0] <= 1.3 * err[1] + 2 ** -22 * want.norm(dim=1) + N ** 0.5 * 2.0 ** -149).all())
    assert ops.tc5_status() == 0


def test_split_operands_let_what_is_not_finite_through():
    """Infinities, NaN of every pattern, values that round to infinity as TF32 and sums that overflow: as term by term."""
    M, N, K = 96, 144, 512
    a, w = rnd(M, K), rnd(N, K, seed=1)
    a[3, 7], a[40, 200], a[60, 0], a[61, 5] = float("inf"), float("-inf"), float("nan"), torch.finfo(torch.float32).max
    a[62, 9] = torch.tensor(0x7fffffff, dtype=torch.int32).view(torch.float32)
    a[63, 9] = torch.tensor(0x7f800001, dtype=torch.int32).view(torch.float32)
    w[:, 5].mul_(0.25).clamp_(-0.5, 0.5)
    out = torch.empty(M, N, device=DEV)
    ops.linear(a, w, out)
    want = a.double() @ w.double().T
    clean = [i for i in range(M) if i not in (3, 40, 60, 62, 63)]
    assert bool(out[clean].isfinite().all()) and bool(out[[60, 62, 63]].isnan().all())
    assert torch.equal(out[[3, 40]], want[[3, 40]].float())
    assert float((out[61].double() - want[61]).norm() / want[61].norm()) < 2 ** -20
    assert ops.tc5_status() == 0


@pytest.mark.parametrize("rows,K", [(4, 256), (40, 252), (40, 256)])           # streamed, tiled, on the tensor cores
def test_products_let_infinities_through(rows, K):
    a, w = rnd(40, K), rnd(64, K, seed=1).abs()
    a[3, 7], a[35, 200], a[39, 0] = float("inf"), float("-inf"), float("nan")
    out = torch.empty(rows, 64, device=DEV)
    ops.linear(a[:rows].contiguous(), w, out)
    assert bool((out[3] == float("inf")).all()) and bool(out[:3].isfinite().all())
    if rows == 40:
        assert bool((out[35] == float("-inf")).all()) and bool(out[39].isnan().all()) and bool(out[36:39].isfinite().all())


def attention_both(hq, hkv, hd, held, new, window=0, chunk=0, sink=None, softcap=0.0, bias=None, edit=None, seed=0):
    cache = Cache([KVNeed(hkv, hd, window, 0, chunk)], [None], 64 * sum((h + n + 63) // 64 for h, n in zip(held, new)),
                  torch.float32, DEV)
    storage = cache.groups[0].entry_storage(0)
    storage.copy_(rnd(*storage.shape, seed=seed))
    slots = [cache.open() for _ in held]
    for s, h, n in zip(slots, held, new):
        cache.reserve(s, h + n)
        cache.advance(s, h)
    if edit is not None:
        edit(cache, storage, slots)
    plan = StepPlan(cache, [StepEntry(s, [0] * n, []) for s, n in zip(slots, new)], DEV)
    q = rnd(sum(new), hq, hd, seed=seed + 1)
    outs = []
    for kernel in ("auto", "plain"):
        out = torch.full((sum(new), hq * hd), float("nan"), device=DEV)
        ops.attention(q, out, plan, 0, storage, hq, hkv, hd, window, hd ** -0.5, kernel=kernel, sink=sink, softcap=softcap,
                      chunk=chunk, bias=bias)
        outs.append(out)
    return outs


# one token's heads in the 16-row form (and one head more than fits), stretches in the 64- and 32-row forms; head sizes below,
# at and over each width; lengths around a tile of 64 keys and around all of a cluster's tiles, and longest lengths that make clusters
# of one, two and four blocks
@pytest.mark.parametrize("hq,hkv,hd", [(4, 2, 16), (12, 2, 128), (17, 1, 36), (16, 1, 64), (3, 3, 100), (2, 1, 256)])
@pytest.mark.parametrize("held,new", [([0, 63, 64, 511, 513, 1100], [1] * 6), ([0, 5, 200], [63, 130, 17]), ([0], [201]),
                                      ([0, 20, 63], [1] * 3), ([0, 64, 127], [1] * 3), ([3, 190, 255], [1] * 3), ([0, 10], [64, 30]),
                                      ([40, 0], [60, 128]), ([0] * 40, [200] * 40)])
def test_attention(hq, hkv, hd, held, new):
    sink = rnd(hq, seed=5)
    bias = ops.DistanceBias(rnd(hq, 33, seed=6))
    for kw in (dict(), dict(window=70), dict(chunk=96, sink=sink), dict(softcap=3.0, bias=bias), dict(window=1, sink=sink, bias=bias)):
        got, want = attention_both(hq, hkv, hd, held, new, **kw)
        # two orders of a softmax's sums in float32: 2^-24 of the largest value for each of about 16 roundings
        assert pm.rel_err(got.cpu(), want.cpu()) < 16 * 2 ** -24 * 2, kw


def test_attention_of_values_that_are_not_finite():
    """A later token's infinite value stays out of the rows that do not see it; the rows that do get what they get."""
    def edit(cache, storage, slots):
        page = cache.page_list(slots[0], 0)[1]
        storage[page, 1, :, 20] = float("inf")         # position 84
        storage[page, 0, :, 25] = float("nan")         # the key at 89
    got, want = attention_both(4, 2, 32, [10], [120], edit=edit)
    assert torch.equal(got.isfinite(), want.isfinite()) and bool(got[:74].isfinite().all())
    assert pm.rel_err(got[:74].cpu(), want[:74].cpu()) < 16 * 2 ** -24 * 2


def test_attention_of_a_plans_first_rows():
    """Queries for fewer rows than the plan has, as the plain kernel takes them: the others are neither read nor written."""
    cache = Cache([KVNeed(2, 32, 0, 0, 0)], [None], 64 * 4, torch.float32, DEV)
    storage = cache.groups[0].entry_storage(0)
    storage.copy_(rnd(*storage.shape))
    slots = [cache.open() for _ in range(2)]
    for s, h in zip(slots, (5, 40)):
        cache.reserve(s, h + 9)
        cache.advance(s, h)
    plan = StepPlan(cache, [StepEntry(s, [0] * 9, []) for s in slots], DEV)
    for n in (4, 9, 13):
        q = rnd(n, 4, 32, seed=1)
        out = torch.full((2, 18, 128), float("nan"), device=DEV)
        for o, kernel in zip(out, ("auto", "plain")):
            ops.attention(q, o[:n], plan, 0, storage, 4, 2, 32, 0, 32 ** -0.5, kernel=kernel)
        assert pm.rel_err(out[0, :n].cpu(), out[1, :n].cpu()) < 16 * 2 ** -24 * 2 and bool(out[0, n:].isnan().all())


@pytest.mark.parametrize("hq,hkv,hd", [(12, 2, 128), (3, 1, 64), (2, 1, 256), (16, 16, 32)])
@pytest.mark.parametrize("kw", [dict(), dict(window=150), dict(chunk=320, softcap=3.0)])
def test_attention_of_a_row_does_not_depend_on_the_launch(hq, hkv, hd, kw):
    """One sequence of 1,300 tokens whole (tiles of 64 rows), its rows in portions of one (16 rows) and of 20 (32 rows), and a portion
    beside other sequences: the same bits."""
    n, others = 1300, 30
    cache = Cache([KVNeed(hkv, hd, 0, 0, 0)], [None], 64 * (21 + others * 4), torch.float32, DEV)
    storage = cache.groups[0].entry_storage(0)
    storage.copy_(rnd(*storage.shape))
    seq, slots = cache.open(), [cache.open() for _ in range(others)]
    cache.reserve(seq, n)
    for s in slots:
        cache.reserve(s, 200)
    q = rnd(n, hq, hd, seed=1)

    def run(entries):
        plan = StepPlan(cache, [StepEntry(s, [0] * (hi - lo), []) for s, lo, hi in entries], DEV)
        rows = torch.cat([q[lo:hi] for _, lo, hi in entries]).contiguous()
        out = torch.empty(len(rows), hq * hd, device=DEV)
        ops.attention(rows, out, plan, 0, storage, hq, hkv, hd, kw.get("window", 0), hd ** -0.5, softcap=kw.get("softcap", 0.0),
                      chunk=kw.get("chunk", 0))
        return out

    whole = run([(seq, 0, n)])
    for lo, hi in [(0, 1), (63, 83), (511, 512), (512, 532), (777, 1100), (1280, 1300)]:
        cache.advance(seq, lo)
        alone, beside = run([(seq, lo, hi)]), run([(slots[0], 0, 7), (seq, lo, hi)] + [(s, 0, 200) for s in slots[1:]])
        assert torch.equal(alone, whole[lo:hi]) and torch.equal(beside[7:7 + hi - lo], whole[lo:hi]), (lo, hi)
