"""Columns of 16 query rows of the decode kernels over packed rows.

They run from 9 query rows per kv head on, where they halve the columns and every worker has enough tiles; the same call with a
workspace that only the columns of eight rows fit takes those. Both forms are held to one another (same f16 weights up to the
reference maximum of a split, f32 sums: 1e-3 + 1e-3 |x|) and to the oracle for one batch entry."""
import importlib.util
from pathlib import Path

import numpy as np
import pytest
import torch

from gpu_util import assert_close, fmt, pkg, words

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
spec = importlib.util.spec_from_file_location("make_golden", ROOT / "tests" / "golden" / "make_golden.py")
MG = importlib.util.module_from_spec(spec)
spec.loader.exec_module(MG)


@pytest.fixture(scope="module")
def P():
    return pkg()


def case(P, f, b, hq, hkv, lq, lk, d, seed, rotation="none", pad=0):
    g = torch.Generator(device="cuda:0").manual_seed(seed)
    kq, vq = P.TurboQuantizer(fmt(P, *f), d, rotation, 42), P.TurboQuantizer(fmt(P, *f), d, rotation, 44)
    rows = []
    for q in (kq, vq):
        x = torch.randn((b * hkv * lk, d), generator=g, device="cuda:0")
        r = torch.zeros((b, hkv, lk + 3, q.row_words() + pad), dtype=torch.int32, device="cuda:0")
        r[:, :, :lk, : q.row_words()] = q.quantize_rows(x).view(b, hkv, lk, -1)
        rows.append(r)
    return torch.randn((b, hq, lq, d), generator=g, device="cuda:0"), rows[0], rows[1], kq, vq


# format, b, hq, hkv, lq, lk, d, padding of the rows in words, window on the left
WIDE = [
    ((2, 4), 8, 32, 8, 3, 3601, 128, 0, -1),   # 12 rows of 16, rows back to back
    ((4, 4), 8, 64, 8, 2, 3553, 128, 0, -1),   # 16 rows
    ((3, 4), 2, 16, 2, 4, 28900, 128, 0, -1),  # 32 rows: two columns per kv head; many segments per column (combine grid)
    ((5, 4), 8, 36, 4, 1, 7200, 128, 1, 700),  # a group of 9, padded rows, a window
    ((2, 4), 16, 16, 4, 4, 3590, 64, 0, -1),   # head dim 64
    ((4, 4), 16, 16, 4, 3, 3590, 64, 2, 33),
]


@pytest.mark.parametrize("f,b,hq,hkv,lq,lk,d,pad,wl", WIDE, ids=lambda x: str(x))
def test_wide_columns_against_narrow_ones_and_the_oracle(P, oracle, f, b, hq, hkv, lq, lk, d, pad, wl):
    q, k, v, kq, vq = case(P, f, b, hq, hkv, lq, lk, d, 5, pad=pad)
    c = P.FlashAttnConfig(d ** -0.5).window(None if wl < 0 else wl, 0)
    lens = torch.tensor([lk - 37 * (i % 5) for i in range(b)], dtype=torch.int32, device="cuda:0")
    wide = P.PackedAttention(q, k, v, lens, kq, vq, c)
    got = wide.run().clone()
    if hq // hkv * lq >= 16:  # (the partial rows of fewer take less workspace than two columns of eight)
        narrow = P.PackedAttention(q, k, v, lens, kq, vq, c)
        narrow.args.workspace_bytes = P._abi.lib().b200_tq_attention_workspace_bytes(narrow._ref) - 16  # too small for the wide columns
        small = narrow.run().clone()
        assert_close(got.cpu().numpy(), small.cpu().numpy(), 1e-3, 1e-3, "wide against narrow columns")
    i, n, w = b - 1, int(lens[b - 1]), kq.row_words()
    tab = np.zeros(64, np.float32)
    kd, vd = (words(x[i:i + 1, :, :n, :w].contiguous()) for x in (k, v))
    want = oracle.tq_attention(q[i:i + 1].cpu().numpy(), kd, vd, n, f, f, d ** -0.5, tab, wl=wl, wr=0)
    assert_close(got[i:i + 1].cpu().numpy(), want, what="wide columns")
    assert torch.equal(got, wide.run())  # whoever merges a column, the result is the same


@pytest.mark.parametrize("rows_of_a_block", [64, 96])
def test_wide_columns_over_blocks(P, rows_of_a_block):
    f, b, hq, hkv, lq, d, n = (2, 4), 8, 32, 8, 4, 128, 60
    g = torch.Generator(device="cuda:0").manual_seed(3)
    kq, vq = P.TurboQuantizer(fmt(P, *f), d, "hadamard", 42), P.TurboQuantizer(fmt(P, *f), d, "hadamard", 44)
    blocks, ks, vs = [], [], []
    for i in range(n):
        kb, vb = (x.quantize_rows(torch.randn((b * hkv * 96, d), generator=g, device="cuda:0")).view(b, hkv, 96, -1).contiguous() for x in (kq, vq))
        m = rows_of_a_block - (i % 3) * 5
        blocks.append(P.KvBlockRef(kb, vb, m))
        ks.append(kb[:, :, :m])
        vs.append(vb[:, :, :m])
    lk = sum(x.rows for x in blocks)
    q = torch.randn((b, hq, lq, d), generator=g, device="cuda:0")
    lens = torch.tensor([lk - 101 * i for i in range(b)], dtype=torch.int32, device="cuda:0")
    c = P.FlashAttnConfig(d ** -0.5).causal()
    got = P.attention_packed_blocks(q, blocks, kq, vq, c, kv_len=lens)
    want = P.attention_packed(q, torch.cat(ks, 2).contiguous(), torch.cat(vs, 2).contiguous(), lens, kq, vq, c)
    assert_close(got.cpu().numpy(), want.cpu().numpy(), 1e-3, 1e-3, "blocks against dense rows")


@pytest.mark.parametrize("pages", [1, 31, 32, 127, 128, 300])
def test_prefix_sums_of_the_block_table(P, pages):
    """Up to 127 blocks the attention's own blocks work the sums out, each for itself, above a kernel in front does; odd fill levels, empty
    blocks. Either way one copy in global memory, at the start of the workspace, is the combine grid's."""
    b, hq, hkv, d, f = 2, 8, 2, 128, (2, 4)
    g = torch.Generator(device="cuda:0").manual_seed(pages)
    kq, vq = P.TurboQuantizer(fmt(P, *f), d, "none", 42), P.TurboQuantizer(fmt(P, *f), d, "none", 44)
    fills = [(7 * i + 5) % 41 for i in range(pages)]
    blocks, ks, vs = [], [], []
    for n in fills:
        kb, vb = (q.quantize_rows(torch.randn((b * hkv * 40, d), generator=g, device="cuda:0")).view(b, hkv, 40, -1).contiguous() for q in (kq, vq))
        blocks.append(P.KvBlockRef(kb, vb, n))
        ks.append(kb[:, :, :n])
        vs.append(vb[:, :, :n])
    lk = sum(fills)
    c = P.FlashAttnConfig(d ** -0.5).causal()
    for lq in (1, 4):
        q = torch.randn((b, hq, lq, d), generator=g, device="cuda:0")
        lens = torch.tensor([lk, max(1, lk - 9)], dtype=torch.int32, device="cuda:0")
        call = P.PackedBlocksAttention(q, blocks, kq, vq, c, kv_len=lens)
        got = call.run()
        tiles = [(n + 31) // 32 for n in fills]
        sums = [sum(fills[:i]) for i in range(pages + 1)] + [sum(tiles[:i]) for i in range(pages + 1)]
        assert words(call._keep[-1][: 8 * (pages + 1)]).tolist() == sums
        want = P.attention_packed(q, torch.cat(ks, 2).contiguous(), torch.cat(vs, 2).contiguous(), lens, kq, vq, c)
        assert_close(got.cpu().numpy(), want.cpu().numpy(), 1e-3, 1e-3, f"{pages} blocks, {lq} query tokens")


@pytest.mark.parametrize("rotation", ["none", "hadamard"])
@pytest.mark.parametrize("b,lk", [(24, 9000), (1, 70000), (200, 700)])
def test_shares_and_merges_of_large_calls(P, rotation, b, lk):
    """Many tiles per worker, columns of few and of many segments, rows that leave L2 first."""
    f, hq, hkv, d = (2, 4), 16, 8, 128
    q, k, v, kq, vq = case(P, f, b, hq, hkv, 1, lk, d, 7, rotation)
    lens = torch.tensor([max(1, lk - (lk // 3) * (i % 3)) for i in range(b)], dtype=torch.int32, device="cuda:0")
    c = P.FlashAttnConfig(d ** -0.5).causal()
    got = P.attention_packed(q, k, v, lens, kq, vq, c)
    one = P.attention_packed(q, k, v, lens, kq, vq, P.FlashAttnConfig(d ** -0.5, splits=1).causal())  # one share per column
    assert_close(got.cpu().numpy(), one.cpu().numpy(), 1e-3, 1e-3, "shares of the work against one share per column")


# ---- where the columns of 16 rows begin. A call of 16 and more rows asks for the workspace of its widest form; with 16 bytes less it takes
# columns of eight, whose splits of the keys, and with them the last bits, are others.
def tiles_per_worker(tiles):
    return tiles * 8 * torch.cuda.get_device_properties(0).multi_processor_count  # two blocks of four workers per SM


def both_forms(P, call):
    got = call.run().clone()
    call.args.workspace_bytes = P._abi.lib().b200_tq_attention_workspace_bytes(call._ref) - 16
    return got, call.run().clone()


RULE = [
    # format, b, hq, hkv, lq, d, tiles per worker, window on the left, lengths in device memory, columns of 16 rows
    ((2, 4), 8, 32, 8, 4, 128, 12.0, -1, False, True),
    ((2, 4), 8, 32, 8, 4, 128, 8.0, -1, False, False),
    ((5, 4), 8, 32, 8, 4, 128, 8.0, -1, False, True),
    ((5, 4), 8, 32, 8, 4, 128, 5.0, -1, False, False),
    ((2, 4), 8, 32, 8, 4, 64, 11.0, -1, False, False),
    ((2, 4), 8, 32, 8, 4, 64, 15.0, -1, False, True),
    ((5, 4), 1, 32, 8, 4, 128, 9.0, -1, False, False),  # eight columns that 148 workers share each
    ((5, 4), 1, 32, 8, 4, 128, 13.0, -1, False, True),
    ((5, 4), 1, 32, 8, 4, 128, 13.0, -1, True, False),  # ... of which the lengths may be a small part
    ((5, 4), 1, 32, 8, 4, 128, 13.0, 300, False, False),  # a window: the tiles that it shows
    ((4, 4), 64, 32, 8, 8, 128, 18.0, -1, False, False),  # two short columns per kv head
    ((4, 4), 64, 32, 8, 8, 128, 26.0, -1, False, True),
]


@pytest.mark.parametrize("f,b,hq,hkv,lq,d,tiles,wl,dev,wide", RULE, ids=lambda x: str(x))
def test_where_columns_of_16_rows_begin(P, f, b, hq, hkv, lq, d, tiles, wl, dev, wide):
    lk = int(tiles_per_worker(tiles)) * 32 // (b * hkv * ((hq // hkv * lq + 15) // 16))
    q, k, v, kq, vq = case(P, f, b, hq, hkv, lq, lk, d, 11)
    c = P.FlashAttnConfig(d ** -0.5).window(None if wl < 0 else wl, 0)
    lens = torch.full((b,), lk, dtype=torch.int32, device="cuda:0") if dev else lk
    got, small = both_forms(P, P.PackedAttention(q, k, v, lens, kq, vq, c))
    assert_close(got.cpu().numpy(), small.cpu().numpy(), 1e-3, 1e-3, "the two forms")
    assert torch.equal(got, small) != wide
