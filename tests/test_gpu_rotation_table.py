"""The q|k|v product of many rows that rotates as it ends, against the product and the rotation kernel: the same bits."""
import pytest
import torch

from sonicboom_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


@pytest.fixture
def widest_tiles():
    """256 columns for every product of many rows, as most sizes of a prompt have them: no K split, no narrower tile."""
    ops.force_tc5_tile_width(256)
    yield
    ops.force_tc5_tile_width(0)


# rows that end inside a tile and inside a warp; column tiles that are full, and last ones with 64, 128 and 192 columns
@pytest.mark.parametrize("rows", [129, 1025, 2048, 3007])
@pytest.mark.parametrize("hq,hkv,hd,K", [(28, 4, 128, 512), (12, 2, 128, 1536), (16, 4, 64, 200), (5, 5, 128, 72), (40, 8, 64, 264),
                                         (9, 2, 64, 136), (11, 2, 64, 200)])
@pytest.mark.parametrize("bias", [None, torch.float32, torch.bfloat16])
@pytest.mark.parametrize("has_kv", [True, False])
def test_table_gives_the_rotation_kernels_bits(widest_tiles, rows, hq, hkv, hd, K, bias, has_kv):
    torch.manual_seed(rows + K)
    N = (hq + (2 * hkv if has_kv else 0)) * hd
    w = torch.randn(N, K, device=DEV, dtype=torch.bfloat16) * K ** -0.5
    assert ops.takes_rotation_table(rows, w, hq, hkv, hd, hd, has_kv)
    h = torch.randn(rows, K, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(N, device=DEV).to(bias) if bias is not None else None
    inv = torch.rand(hd // 2, device=DEV)
    # three sequences, their pages in no order; the last one's last rows lie past its pages, one row before position 0
    cut = [0, rows // 3, rows // 2, rows]
    seq = [s for s in range(3) for _ in range(cut[s + 1] - cut[s])]
    pos = [r - cut[s] + (100 if s == 1 else 0) for r, s in enumerate(seq)]
    pos[5] = -1
    need = [(cut[s + 1] - cut[s] + 100 + 63) // 64 for s in range(3)]
    need[2] = max(1, need[2] - 3)
    off = [0, need[0], need[0] + need[1], sum(need)]
    pages = torch.randperm(sum(need)).tolist()
    where = (inv, i32(seq), i32(pos), i32(off), i32(pages), 64)
    angles = ops.rotation_table(where[2], inv, hd)
    theta = (where[2].float()[:, None] * inv).double()
    assert (angles.double() - torch.cat([theta.cos(), theta.sin()], 1)).abs().max() < 2.0 ** -22   # cosf, sinf: 2 ulp
    outs = []
    for table in (None, angles):
        cache = torch.full((sum(need), 2, hkv, 64, hd), 7.0, device=DEV, dtype=torch.bfloat16) if has_kv else None
        q = torch.full((rows, hq, hd), 9.0, device=DEV, dtype=torch.bfloat16)
        before = ops.LAUNCHES
        ops.qkv_rope_store(h, w, b, hq, hkv, hd, hd, *where, cache, q, table)
        assert ops.LAUNCHES - before == (2 if table is None else 1)
        outs.append((q, cache))
    assert torch.equal(outs[0][0], outs[1][0]) and not bool((outs[1][0] == 9.0).all(-1).any())
    assert not has_kv or torch.equal(outs[0][1], outs[1][1])
    assert ops.tc5_status() == 0


def test_a_table_is_left_alone_where_the_product_does_not_take_it():
    """Few rows, rows whose K is split, and operands off 16 bytes go the way they go without a table."""
    hq, hkv, hd, K = 12, 2, 128, 1536
    w = torch.randn(2048, K, device=DEV, dtype=torch.bfloat16) * 0.02
    inv = torch.rand(hd // 2, device=DEV)
    for rows, shift in ((1, 0), (40, 0), (200, 0), (2560, 4)):
        h = torch.randn(rows, K, device=DEV, dtype=torch.bfloat16)
        n_pages = (rows + 63) // 64
        where = (inv, i32([0] * rows), i32(list(range(rows))), i32([0, n_pages]), i32(list(range(n_pages))), 64)
        outs = []
        for table in (None, ops.rotation_table(where[2], inv, hd)):
            cache = torch.zeros(n_pages, 2, hkv, 64, hd, device=DEV, dtype=torch.bfloat16)
            q = torch.zeros(rows * hq * hd + shift, device=DEV, dtype=torch.bfloat16)[shift:].view(rows, hq, hd)
            ops.qkv_rope_store(h, w, None, hq, hkv, hd, hd, *where, cache, q, table)
            outs.append((q.clone(), cache))
        assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("rows,hq,hkv,hd,K,takes", [
    (128, 28, 4, 128, 3584, False), (512, 28, 4, 128, 3584, False),                                   # few rows, K split
    (768, 28, 4, 128, 3584, False), (769, 28, 4, 128, 3584, True), (2048, 28, 4, 128, 3584, True),    # one wave of narrower tiles; more
    (1024, 12, 2, 128, 1536, False), (2048, 12, 2, 128, 1536, False), (2049, 12, 2, 128, 1536, True),
    (3007, 5, 5, 128, 72, False)])                                                                     # a narrower tile wastes less
def test_which_products_take_a_table(rows, hq, hkv, hd, K, takes):
    if torch.cuda.get_device_properties(DEV).multi_processor_count != 148:
        pytest.skip("the sizes are those of 148 SMs")
    w = torch.empty((hq + 2 * hkv) * hd, K, device=DEV, dtype=torch.bfloat16)
    assert ops.takes_rotation_table(rows, w, hq, hkv, hd, hd) == takes
    assert not ops.takes_rotation_table(rows, w, hq, hkv, hd, hd // 2)
