"""The decode kernel that splits by KV head (short contexts, head sizes 64 / 256): every way its plan can cut a batch, against the
oracle, several times over the same workspace."""
import math

import numpy as np
import pytest
import torch

from turboquant_b200 import TurboQuantPagedAttention, _cabi, synthetic
from turboquant_b200.paged_attention import kv_cache_shape

from tests.gpu_util import assert_attention_close

pytestmark = pytest.mark.gpu
DEV = "cuda"

# (query heads, KV heads, head size, lengths)
CASES = {
    "one_page": (32, 8, 128, [1]),
    "one_head_many_parts": (8, 1, 128, [2000]),                        # more parts than one merge warp takes
    "cut_heads": (32, 8, 128, [1024, 1000]),
    "whole_heads_and_empty_rows": (16, 8, 128, [256, 17, 0, 16, 15] * 3),
    "one_piece_each": (32, 8, 128, [500] * 30),
    "long_pieces": (40, 8, 128, [500] * 60),
    "long_pieces_cut": (56, 8, 128, [300] * 33),
    "ragged_even_cut": (8, 4, 128, [3000, 1, 40, 2500, 700, 16, 33, 129]),
    "odd_heads": (12, 6, 128, [700, 80, 5]),                            # head sets of two (padded head size 128 of another slot is below)
    "three_heads": (6, 3, 64, [700, 80, 5]),
    "many_heads": (32, 32, 128, [333, 90]),
    "many_sequences": (8, 4, 128, [20] * 300),                          # always cut evenly
    "head_96": (32, 8, 96, [100, 777]),
    "head_64": (16, 8, 64, [1500, 31, 0, 640]),
    "head_64_even": (16, 8, 64, [4000, 100, 100, 2000] * 8),
    "head_80": (8, 2, 80, [400, 65]),
    "head_256": (16, 8, 256, [900, 31, 0, 200]),
    "head_256_eight_columns": (32, 4, 256, [300, 47]),
}


@pytest.mark.parametrize("name", [n for n in CASES if n != "odd_heads"] + ["odd_heads"])
def test_every_cut_matches_the_oracle(oracle, name):
    hq, hkv, d, lens = CASES[name]
    if name == "odd_heads":
        d = 80                                                          # 128-wide heads come in 1, 2, 4, 8, 16 or multiples of 4
    attn = TurboQuantPagedAttention(hq, d, 1.0 / math.sqrt(d), hkv)
    case = synthetic.decode_case(seed=len(name), seq_lens=lens, dtype=torch.float16, heads=(hq, hkv), head_dim=d)
    cache = torch.zeros(kv_cache_shape(max(case.num_blocks, 1), 16, hkv, d), dtype=torch.uint8, device=DEV)
    attn.write(case.k.to(DEV), case.v.to(DEV), cache, case.slot_mapping.to(DEV))
    want = oracle.decode_paged(case.q.float().numpy(), cache.cpu().numpy(), case.block_table.numpy(), case.seq_lens.numpy(),
                               attn.signs(DEV).cpu().numpy(), attn.scale)
    q, bt, sl = case.q.to(DEV), case.block_table.to(DEV), case.seq_lens.to(DEV)
    for _ in range(3):
        out = torch.full_like(q, float("nan"))
        lse = torch.full(q.shape[:2], float("nan"), dtype=torch.float32, device=DEV)
        attn.decode(q, cache, bt, sl, out, lse)
        assert attn.status(len(lens), DEV) == 0
        assert_attention_close(out.float().cpu().numpy(), want, name)
        empty = np.array(lens) == 0
        assert (out.cpu().numpy()[empty] == 0).all() and np.isneginf(lse.cpu().numpy()[empty]).all()
        assert torch.isfinite(lse[torch.from_numpy(~empty)]).all()


# (query heads, KV heads, head size, queries a row): one to eight columns and the wide tiles
FEW_LIVE = [(32, 8, 128, 1), (8, 1, 128, 1), (8, 2, 128, 1), (16, 8, 64, 1), (4, 1, 64, 1), (16, 8, 256, 1), (2, 2, 256, 1), (8, 2, 128, 5), (8, 4, 128, 8)]


@pytest.mark.parametrize("hq,hkv,d,nq", FEW_LIVE)
@pytest.mark.parametrize("rows,live,tokens", [(257, 1, 320), (300, 2, 160), (512, 5, 400), (290, 3, 1)])
def test_many_rows_of_which_few_hold_tokens(oracle, hq, hkv, d, nq, rows, live, tokens):
    """A mixed step or a padded batch: the plan's list is shorter than the number of workers, on a fresh workspace and on one that a
    call with more work has filled."""
    lens = [0] * rows
    for i in range(live):
        lens[(7 + 61 * i) % rows] = tokens
    attn = TurboQuantPagedAttention(hq, d, 1.0 / math.sqrt(d), hkv)
    case = synthetic.decode_case(seed=rows + live, seq_lens=lens, dtype=torch.float16, heads=(hq, hkv), head_dim=d)
    cache = torch.zeros(kv_cache_shape(max(case.num_blocks, 1), 16, hkv, d), dtype=torch.uint8, device=DEV)
    attn.write(case.k.to(DEV), case.v.to(DEV), cache, case.slot_mapping.to(DEV))
    q = torch.randn(rows, nq, hq, d, generator=torch.Generator().manual_seed(3)).to(torch.float16)
    at = np.array(lens) > 0
    want = oracle.decode_paged(q[at].float().numpy().reshape(-1, hq, d), cache.cpu().numpy(), np.repeat(case.block_table.numpy()[at], nq, axis=0),
                               np.full(live * nq, tokens, np.int32), attn.signs(DEV).cpu().numpy(), attn.scale)
    q, bt, sl = q.to(DEV), case.block_table.to(DEV), case.seq_lens.to(DEV)
    full = torch.full_like(sl, tokens)                                  # every row, over the pages of the first (all ids are in range)
    for turn in range(2):
        out = torch.full_like(q, float("nan"))
        attn.decode_shared(q, cache, bt, sl, out)
        assert attn.status(rows, DEV, nq) == 0
        got = out.float().cpu().numpy()
        assert (got[~at] == 0).all()
        assert_attention_close(got[at].reshape(-1, hq, d), want, f"turn {turn}")
        if turn == 0:
            attn.decode_shared(q, cache, bt, full, out)


@pytest.mark.parametrize("hq,hkv,d,nq", [(8, 4, 128, 1), (4, 1, 64, 1), (4, 2, 256, 1), (8, 2, 128, 5)])
@pytest.mark.parametrize("rows", [33, 64, 255, 256, 257, 1023, 1025, 2100])
def test_batches_around_the_plans_groups(oracle, hq, hkv, d, nq, rows):
    """Groups of 32 sequences, eight of them loaded at a time, 32 of them remembered; empty groups among them and a long sequence at each end."""
    rng = np.random.default_rng(rows)
    lens = rng.integers(0, 60, rows)
    lens[32 * (rows // 64): 32 * (rows // 64) + 32] = 0
    lens[0], lens[-1] = 600, 777
    attn = TurboQuantPagedAttention(hq, d, 1.0 / math.sqrt(d), hkv)
    case = synthetic.decode_case(seed=rows, seq_lens=lens.tolist(), dtype=torch.float16, heads=(hq, hkv), head_dim=d)
    cache = torch.zeros(kv_cache_shape(case.num_blocks, 16, hkv, d), dtype=torch.uint8, device=DEV)
    attn.write(case.k.to(DEV), case.v.to(DEV), cache, case.slot_mapping.to(DEV))
    q = torch.randn(rows, nq, hq, d, generator=torch.Generator().manual_seed(1)).to(torch.float16)
    want = oracle.decode_paged(q.float().numpy().reshape(-1, hq, d), cache.cpu().numpy(), np.repeat(case.block_table.numpy(), nq, axis=0),
                               np.repeat(case.seq_lens.numpy(), nq), attn.signs(DEV).cpu().numpy(), attn.scale)
    out = torch.full_like(q, float("nan"), device=DEV)
    attn.decode_shared(q.to(DEV), cache, case.block_table.to(DEV), case.seq_lens.to(DEV), out)
    assert attn.status(rows, DEV, nq) == 0
    got = out.float().cpu().numpy()
    assert (got[lens == 0] == 0).all()
    assert_attention_close(got.reshape(-1, hq, d), want, f"{rows} rows")


def _exact(attn, cache, table, lens, q, causal=False, fp16_operands=False):
    """Attention over the cache's own bytes in 64 bits, in the rotated domain; q [rows, queries, heads, size].  ``fp16_operands``: with
    the queries and centroids rounded as the kernel's, which leaves the rounding of P times the V norm."""
    H, D, pd = attn.num_kv_heads, attn.head_size, attn.padded_dim
    rot = torch.ones(1, 1, dtype=torch.float64, device=DEV)
    while rot.shape[0] < pd:
        rot = torch.cat([torch.cat([rot, rot], 1), torch.cat([rot, -rot], 1)], 0)
    rot = rot / math.sqrt(pd) * attn.signs(DEV).double()
    centroids = _cabi.codebook(pd, 4)[0].double().to(DEV)
    q = torch.nn.functional.pad(q.double(), (0, pd - D)) @ rot.T
    if fp16_operands:
        unit = math.sqrt(pd) if D in (128, 96) else 1.0                 # those share the N(0, 1) table
        q, centroids = q.half().double(), (centroids * unit).half().double() / unit
    out = torch.zeros(q.shape, dtype=torch.float64, device=DEV)
    for b, n in enumerate(lens):
        slots = cache[:, table[b, : (n + 15) // 16].long()].flatten(1, 2)[:, :n]
        codes, norms = slots[..., : pd // 2], slots[..., pd // 2: pd // 2 + 2].contiguous().view(torch.float16).double()
        kv = torch.stack([centroids[(codes >> 4).long()], centroids[(codes & 15).long()]], -1).flatten(-2) * norms
        s = torch.einsum("nhgd,thd->nhgt", q[b].unflatten(1, (H, -1)), kv[0]) * attn.scale
        if causal:
            hidden = torch.arange(n, device=DEV)[None, :] >= n - torch.arange(q.shape[1] - 1, -1, -1, device=DEV)[:, None]
            s.masked_fill_(hidden[:, None, None], -math.inf)
        out[b] = torch.einsum("nhgt,thd->nhgd", s.softmax(-1), kv[1]).flatten(1, 2)
    return (out @ rot)[..., :D]


def _error(attn, nq, lens, v_scale, q_scale=1.0, causal=False, fp16_operands=False):
    """Relative error (2-norm) of a decode call in fp32 against 64 bits, N(0, 1) keys, values and queries times a scale."""
    H, D = attn.num_kv_heads, attn.head_size
    g = torch.Generator(DEV).manual_seed(11)
    case = synthetic.decode_case(seed=4, seq_lens=lens, heads=(H, H), head_dim=D)
    cache = torch.zeros(kv_cache_shape(case.num_blocks, 16, H, D), dtype=torch.uint8, device=DEV)
    k, v = (torch.randn(sum(lens), H, D, generator=g, device=DEV) for _ in range(2))
    attn.write(k, v * v_scale, cache, case.slot_mapping.to(DEV))
    q = torch.randn(len(lens), nq, attn.num_heads, D, generator=g, device=DEV) * q_scale
    table = case.block_table.to(DEV)
    out = (attn.decode_causal if causal else attn.decode_shared)(q, cache, table, case.seq_lens.to(DEV))
    want = _exact(attn, cache, table, lens, q, causal, fp16_operands)
    return float((out.double() - want).norm() / want.norm())


# Bounds: 1.15 times what these sizes show with the head's own fp16 centroids and the V norm as it is (3.6e-4 and 4.7e-4 at every scale; with
# the N(0, 1) centroids and 1 / sqrt(d) ahead of the rounding 4.7 ... 5.6e-4 at 80 and, at a scale of 1e-4, 6.8e-4 at 64 and 7.0e-4 at 256).
@pytest.mark.parametrize("hq,hkv,d,bound", [(16, 2, 80, 4.15e-4), (16, 8, 64, 5.4e-4), (16, 8, 256, 5.4e-4)])
@pytest.mark.parametrize("v_scale", [1e-4, 1e-3, 1.0, 50.0])
def test_error_of_other_head_sizes_at_any_size_of_v(hq, hkv, d, bound, v_scale):
    assert _error(TurboQuantPagedAttention(hq, d, 1.0 / math.sqrt(d), hkv), 1, [2000, 700, 4096], v_scale) <= bound


# Bound: 1.15 times the largest error of these calls at V scale 1 with the tcgen05 kernel (5.7e-4), whose operands are P and V^ apart; with 1 / sqrt(128) in
# front of the rounding they showed up to 8.7e-4 at a scale of 1e-4, and infinities from norms of 16000 on.
@pytest.mark.parametrize("hq,hkv,d,nq", [(8, 8, 128, 4), (32, 8, 128, 2), (16, 8, 128, 8), (24, 8, 128, 8), (32, 8, 128, 8), (32, 8, 96, 5)])
@pytest.mark.parametrize("v_scale", [1e-4, 1.0, 3000.0])
def test_error_of_causal_queries_at_any_size_of_v(hq, hkv, d, nq, v_scale):
    assert _error(TurboQuantPagedAttention(hq, d, 1.0 / math.sqrt(d), hkv), nq, [2000, 700, 4096], v_scale, causal=True) <= 6.6e-4


@pytest.mark.parametrize("hq,hkv,d,nq", [(16, 8, 64, 1), (16, 8, 256, 1), (16, 4, 128, 1), (16, 8, 128, 8), (24, 8, 128, 8), (32, 8, 128, 8)])
@pytest.mark.parametrize("order", ["up", "down", "spikes"])
def test_v_norms_of_many_sizes_in_a_sequence(hq, hkv, d, nq, order):
    """The warps' scale is lowered again and again, or once, by the first page or by a few tokens.  Bound: what is left after the operands'
    rounding is that of P times the norm, 2^-11 of each term at most."""
    lens = [2000, 700, 4096]
    size = {"up": lambda t: 10.0 ** (-3 + 6 * t), "down": lambda t: 10.0 ** (3 - 6 * t), "spikes": lambda t: 1.0 + 2500.0 * (torch.frac(t * 37.0) < 0.01)}[order]
    v_scale = torch.cat([size(torch.arange(n, device=DEV) / n) for n in lens])[:, None, None]
    attn = TurboQuantPagedAttention(hq, d, 1.0 / math.sqrt(d), hkv)
    assert _error(attn, nq, lens, v_scale, q_scale=3.0, fp16_operands=True) <= 2.0 ** -11


@pytest.mark.parametrize("heads,rows", [(16, 47), (16, 48), (32, 511), (32, 512), (48, 512)])
def test_one_column_on_either_side_of_its_route(oracle, heads, rows):
    """One query head per KV head on 16 KV heads or launches of 16: many rows go to the streaming kernel.  Bounds: 1.15 times the error of fp16
    operands and products (4.9e-4, see above) and of the fp16 output (2^-11 / sqrt(3)) over all rows; five times that for the worst head of a row."""
    lens = (np.arange(rows) * 7 % 40).tolist()
    attn = TurboQuantPagedAttention(heads, 128, 1.0 / math.sqrt(128), heads)
    case = synthetic.decode_case(seed=rows, seq_lens=lens, dtype=torch.float16, heads=(heads, heads), head_dim=128)
    cache = torch.zeros(kv_cache_shape(case.num_blocks, 16, heads, 128), dtype=torch.uint8, device=DEV)
    attn.write(case.k.to(DEV), case.v.to(DEV), cache, case.slot_mapping.to(DEV))
    want = oracle.decode_paged(case.q.float().numpy(), cache.cpu().numpy(), case.block_table.numpy(), case.seq_lens.numpy(), attn.signs(DEV).cpu().numpy(),
                               attn.scale)
    out = attn.decode(case.q.to(DEV), cache, case.block_table.to(DEV), case.seq_lens.to(DEV))
    assert attn.status(rows, DEV) == 0
    err = np.linalg.norm(out.float().cpu().numpy() - want, axis=-1)
    size = np.linalg.norm(want, axis=-1)
    assert np.linalg.norm(err) <= 6.5e-4 * np.linalg.norm(size)
    assert (err <= 5 * 6.5e-4 * size).all()
    assert (out.cpu().numpy()[np.array(lens) == 0] == 0).all()
