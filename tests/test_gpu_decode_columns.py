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


def tiles_per_worker(tiles):
    return tiles * 8 * torch.cuda.get_device_properties(0).multi_processor_count  # two blocks of four workers per SM


def keys_for(tiles, b, hkv, rows):
    """Keys per sequence that give every worker of the grid of wide columns so many tiles."""
    return int(tiles_per_worker(tiles)) * 32 // (b * hkv * ((rows + 15) // 16))


def both_forms(P, call):
    """A call of 16 and more rows asks for the workspace of its widest form; with 16 bytes less it takes columns of eight."""
    got = call.run().clone()
    call.args.workspace_bytes = P._abi.lib().b200_tq_attention_workspace_bytes(call._ref) - 16
    return got, call.run().clone()


def oracle_entry(oracle, q, k, v, i, n, f, rotation, **kw):
    """The oracle's attention of batch entry i over its first n rows: in the rotated space, then rotated back."""
    d = q.shape[3]
    tab = np.concatenate([MG.tab_for(f[0], f[1], d)] * 2).astype(np.float32)
    qn = q[i:i + 1].float().cpu().numpy()
    if rotation == "hadamard":
        qn = oracle.rotate_rows(qn.reshape(-1, d), oracle.rotation_matrix(d, 1, 42)).reshape(qn.shape)
    want = oracle.tq_attention(qn, *(words(x[i:i + 1, :, :n].contiguous()) for x in (k, v)), n, f, f, d ** -0.5, tab, **kw)
    if rotation == "hadamard":
        want = oracle.rotate_rows(want.reshape(-1, d), oracle.rotation_matrix(d, 1, 44), transpose=True).reshape(want.shape)
    return want


# format, b, hq, hkv, lq, d, rotation, padding of the rows in words, window on the left, soft-capping, ALiBi, tiles per worker
WIDE = [(f, 8, 32, 8, 4, d, rot, 0, -1, 0.0, False, 18) for f in ((2, 4), (3, 4), (4, 4), (5, 4)) for d in (128, 64) for rot in ("none", "hadamard")] + [
    ((4, 4), 8, 64, 8, 2, 128, "none", 0, -1, 0.0, False, 18),
    ((2, 4), 8, 32, 8, 3, 128, "none", 0, -1, 0.0, False, 18),  # 12 rows
    ((5, 4), 8, 36, 4, 1, 128, "none", 1, -1, 0.0, False, 18),  # a group of 9, padded rows
    ((3, 4), 2, 16, 2, 4, 128, "none", 0, -1, 0.0, False, 52),  # 32 rows: two columns per kv head, many workers per column (combine grid)
    ((2, 4), 16, 16, 4, 4, 64, "none", 2, 10000, 0.0, False, 22),  # a window
    ((2, 4), 8, 32, 8, 4, 128, "hadamard", 0, -1, 20.0, False, 18),
    ((5, 4), 8, 32, 8, 4, 128, "none", 0, -1, 0.0, True, 18),
    ((3, 4), 8, 32, 8, 4, 64, "none", 0, 9000, 15.0, True, 18),
]


@pytest.mark.parametrize("f,b,hq,hkv,lq,d,rotation,pad,wl,softcap,alibi,tiles", WIDE, ids=lambda x: str(x))
def test_wide_columns_against_narrow_ones_and_the_oracle(P, oracle, f, b, hq, hkv, lq, d, rotation, pad, wl, softcap, alibi, tiles):
    rows = hq // hkv * lq
    lk = keys_for(tiles, b, hkv, rows)
    q, k, v, kq, vq = case(P, f, b, hq, hkv, lq, lk, d, 5, rotation, pad=pad)
    c = P.FlashAttnConfig(d ** -0.5).window(None if wl < 0 else wl, 0)
    c.softcap = softcap or None
    slopes = np.exp2(-np.arange(1, hq + 1) * 4.0 / hq).astype(np.float32) if alibi else None
    c.alibi_slopes = torch.from_numpy(slopes).to("cuda:0") if alibi else None
    lens = torch.tensor([lk - 37 * (i % 5) for i in range(b)], dtype=torch.int32, device="cuda:0")
    call = P.PackedAttention(q, k, v, lens, kq, vq, c)
    got = call.run().clone()
    assert torch.equal(got, call.run())  # whoever merges a column, the result is the same
    if rows >= 16:  # (the partial rows of fewer take less workspace than two columns of eight)
        got, small = both_forms(P, call)
        assert not torch.equal(got, small), "the call took columns of eight"
        assert_close(got.cpu().numpy(), small.cpu().numpy(), 1e-3, 1e-3, "wide against narrow columns")
    i, w = b - 1, kq.row_words()
    want = oracle_entry(oracle, q, k[..., :w], v[..., :w], i, int(lens[i]), f, rotation, wl=wl, wr=0, softcap=softcap, alibi=slopes)
    assert_close(got[i:i + 1].cpu().numpy(), want, what="wide columns")


@pytest.mark.parametrize("rotation", ["none", "hadamard"])
@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("f", [(0, 4), (2, 4), (3, 4), (4, 4), (5, 4)], ids=str)
def test_wide_columns_over_blocks(P, oracle, f, d, rotation):
    """Against columns of eight over the same blocks and over dense rows (TurboQuant-4: the kernel whose workers are pairs of warps), and
    the oracle; part-filled blocks whose last tiles are short."""
    b, hq, hkv, lq, page = 8, 32, 8, 4, 96
    g = torch.Generator(device="cuda:0").manual_seed(3)
    kq, vq = P.TurboQuantizer(fmt(P, *f), d, rotation, 42), P.TurboQuantizer(fmt(P, *f), d, rotation, 44)
    blocks, ks, vs, left = [], [], [], keys_for(20, b, hkv, hq // hkv * lq)
    while left > 0:
        kb, vb = (x.quantize_rows(torch.randn((b * hkv * page, d), generator=g, device="cuda:0")).view(b, hkv, page, -1).contiguous() for x in (kq, vq))
        m = min(left, page - (len(blocks) % 3) * 5)
        blocks.append(P.KvBlockRef(kb, vb, m))
        ks.append(kb[:, :, :m])
        vs.append(vb[:, :, :m])
        left -= m
    k, v, lk = torch.cat(ks, 2).contiguous(), torch.cat(vs, 2).contiguous(), sum(x.rows for x in blocks)
    q = torch.randn((b, hq, lq, d), generator=g, device="cuda:0")
    lens = torch.tensor([lk - 101 * i for i in range(b)], dtype=torch.int32, device="cuda:0")
    c = P.FlashAttnConfig(d ** -0.5).causal()
    got, small = both_forms(P, P.PackedBlocksAttention(q, blocks, kq, vq, c, kv_len=lens))
    assert not torch.equal(got, small), "the call took columns of eight"
    assert_close(got.cpu().numpy(), small.cpu().numpy(), 1e-3, 1e-3, "wide against narrow columns over blocks")
    dense = P.PackedAttention(q, k, v, lens, kq, vq, c)
    if f[0] != 0:
        dense.args.workspace_bytes = P._abi.lib().b200_tq_attention_workspace_bytes(dense._ref) - 16
    assert_close(got.cpu().numpy(), dense.run().cpu().numpy(), 1e-3, 1e-3, "blocks against dense rows")
    want = oracle_entry(oracle, q, k, v, b - 1, int(lens[b - 1]), f, rotation, wl=-1, wr=0)
    assert_close(got[b - 1:].cpu().numpy(), want, what="wide columns over blocks")


def test_wide_columns_gathered(P):
    """The rows of wide columns in the gathered buffer (a world of one), among them those of sequences without keys."""
    b, hq, hkv, lq, d, f = 8, 32, 8, 4, 128, (4, 4)
    lk = keys_for(18, b, hkv, 16)
    q, k, v, kq, vq = case(P, f, b, hq, hkv, lq, lk, d, 8)
    q = q.to(torch.bfloat16)
    lens = torch.tensor([lk, 0, lk - 5, lk, 40, lk, lk - 1, 0], dtype=torch.int32, device="cuda:0")
    c = P.FlashAttnConfig(d ** -0.5).causal()
    plain = P.PackedAttention(q, k, v, lens, kq, vq, c)
    got, small = both_forms(P, plain)
    assert not torch.equal(got, small), "the call took columns of eight"

    class Gather:  # what OutputGather provides, without symmetric memory
        pass
    gt = Gather()
    gt.buf = torch.full((2, 1, b * hq * lq, d), 7.0, dtype=torch.bfloat16, device="cuda:0")
    flags, state = torch.zeros(4, dtype=torch.int32, device="cuda:0"), torch.zeros(2, dtype=torch.int32, device="cuda:0")
    ptrs = torch.tensor([gt.buf.data_ptr(), flags.data_ptr()], dtype=torch.int64, device="cuda:0")
    gt.args = P._abi.PeerGather(ptrs.data_ptr(), ptrs.data_ptr() + 8, 1, 0, state.data_ptr(), state.data_ptr() + 4)
    out = P.PackedAttention(q, k, v, lens, kq, vq, c, gather=gt).run()
    torch.cuda.synchronize()
    assert torch.equal(out, got) and torch.equal(gt.buf[1, 0].view(b, hq, lq, d), got)


def test_static_call_takes_columns_of_eight(P):
    """The wide form's partial rows do not fit the built-in scratch, those of columns of eight do."""
    A, lib = P._abi, P._abi.lib()
    b, hq, hkv, lq, d, f = 8, 32, 8, 4, 128, (2, 4)
    lk = keys_for(18, b, hkv, 16)
    q, k, v, kq, vq = case(P, f, b, hq, hkv, lq, lk, d, 9)
    call = P.PackedAttention(q, k, v, lk, kq, vq, P.FlashAttnConfig(d ** -0.5).causal())
    assert lib.b200_tq_attention_workspace_bytes(call._ref) > A.STATIC_SCRATCH_BYTES
    got, small = both_forms(P, call)
    assert not torch.equal(got, small), "the call took columns of eight"
    call.out.fill_(float("nan"))
    A.check(lib.b200_tq_attention_static(call._ref, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(call.out, small)


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


# where the columns of 16 rows begin
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
    lk = keys_for(tiles, b, hkv, hq // hkv * lq)
    q, k, v, kq, vq = case(P, f, b, hq, hkv, lq, lk, d, 11)
    c = P.FlashAttnConfig(d ** -0.5).window(None if wl < 0 else wl, 0)
    lens = torch.full((b,), lk, dtype=torch.int32, device="cuda:0") if dev else lk
    got, small = both_forms(P, P.PackedAttention(q, k, v, lens, kq, vq, c))
    assert_close(got.cpu().numpy(), small.cpu().numpy(), 1e-3, 1e-3, "the two forms")
    assert torch.equal(got, small) != wide
