"""The split decode kernel with more than one tile of query columns (shared and causal queries): both sides of every tile edge, every
way the plan cuts a batch, a causal mask that crosses a page edge and hides whole pages, against the oracle."""
import math

import numpy as np
import pytest
import torch

from turboquant_b200 import TurboQuantPagedAttention, _cabi, synthetic
from turboquant_b200.paged_attention import kv_cache_shape

from tests.gpu_util import assert_attention_close

pytestmark = pytest.mark.gpu
DEV = "cuda"

LENS = {
    "one_token": [1],
    "cut_heads": [1030, 1000],
    "ragged": [700, 0, 17, 33, 5, 16, 129],
    "page_edges": [16, 17, 31, 32, 33, 48, 2, 19],
    "even_cut": [3000, 40, 2500, 333, 700, 16] * 3,
    "many": [20] * 40,
}


@pytest.mark.parametrize("heads,nq", [((4, 4), 7), ((8, 8), 8), ((8, 4), 5), ((16, 8), 8), ((20, 4), 3), ((12, 4), 6), ((24, 8), 8), ((28, 4), 4), ((8, 2), 8)])
@pytest.mark.parametrize("name", LENS)
def test_columns_and_cuts(oracle, heads, nq, name):
    (hq, hkv), lens, D = heads, LENS[name], 96 if heads == (8, 4) else 128
    attn = TurboQuantPagedAttention(hq, D, 1.0 / math.sqrt(D), hkv)
    case = synthetic.decode_case(seed=nq + len(name), seq_lens=lens, dtype=torch.float16, heads=(hq, hkv), head_dim=D)
    cache = torch.zeros(kv_cache_shape(max(case.num_blocks, 1), 16, hkv, D), dtype=torch.uint8, device=DEV)
    attn.write(case.k.to(DEV), case.v.to(DEV), cache, case.slot_mapping.to(DEV))
    B = len(lens)
    q = torch.randn(B, nq, hq, D, generator=torch.Generator().manual_seed(9)).to(torch.float16)
    table, signs = case.block_table.numpy(), attn.signs(DEV).cpu().numpy()
    for causal in (False, True):
        seen = np.array(lens)[:, None] - (np.arange(nq - 1, -1, -1)[None, :] if causal else np.zeros((1, nq), int))
        seen = np.maximum(seen, 0).astype(np.int32)
        want = oracle.decode_paged(q.float().numpy().reshape(B * nq, hq, D), cache.cpu().numpy(), np.repeat(table, nq, axis=0), seen.reshape(-1), signs, attn.scale)
        for _ in range(2):
            out = torch.full_like(q, float("nan"), device=DEV)
            lse = torch.full((B, nq, hq), float("nan"), dtype=torch.float32, device=DEV)
            call = attn.decode_causal if causal else attn.decode_shared
            call(q.to(DEV), cache, case.block_table.to(DEV), case.seq_lens.to(DEV), out, lse)
            assert attn.status(B, DEV, nq) == 0
            got = out.float().cpu().numpy()
            assert_attention_close(got.reshape(B * nq, hq, D), want, f"{name} {heads} x {nq} causal={causal}")
            assert (got[seen == 0] == 0).all() and np.isneginf(lse.cpu().numpy()[seen == 0]).all()
            assert np.isfinite(lse.cpu().numpy()[seen > 0]).all()


@pytest.mark.parametrize("heads,nq,D", [((4, 4), 7, 128), ((32, 8), 8, 128), ((32, 8), 5, 96), ((24, 8), 8, 96), ((8, 2), 8, 128), ((16, 16), 9, 128)])
@pytest.mark.parametrize("name", ["one_token", "ragged", "even_cut"])
def test_calls_that_set_their_grid(oracle, heads, nq, D, name):
    """These keep the tcgen05 kernel (causal queries and more than eight columns), head size 96 among them; and windows of the tokens as
    rotated partials, merged."""
    (hq, hkv), lens = heads, LENS[name]
    attn = TurboQuantPagedAttention(hq, D, 1.0 / math.sqrt(D), hkv, num_ctas=148)
    case = synthetic.decode_case(seed=nq + len(name), seq_lens=lens, dtype=torch.float16, heads=(hq, hkv), head_dim=D)
    cache = torch.zeros(kv_cache_shape(max(case.num_blocks, 1), 16, hkv, D), dtype=torch.uint8, device=DEV)
    attn.write(case.k.to(DEV), case.v.to(DEV), cache, case.slot_mapping.to(DEV))
    B = len(lens)
    q = torch.randn(B, nq, hq, D, generator=torch.Generator().manual_seed(9)).to(torch.float16)
    signs, bt, sl = attn.signs(DEV), case.block_table.to(DEV), case.seq_lens.to(DEV)
    for causal in (False, True):
        seen = np.maximum(np.array(lens)[:, None] - (np.arange(nq - 1, -1, -1)[None, :] if causal else np.zeros((1, nq), int)), 0).astype(np.int32)
        want = oracle.decode_paged(q.float().numpy().reshape(B * nq, hq, D), cache.cpu().numpy(), np.repeat(case.block_table.numpy(), nq, axis=0),
                                   seen.reshape(-1), signs.cpu().numpy(), attn.scale)
        out = (attn.decode_causal if causal else attn.decode_shared)(q.to(DEV), cache, bt, sl)
        assert attn.status(B, DEV, nq) == 0
        assert_attention_close(out.float().cpu().numpy().reshape(B * nq, hq, D), want, f"{name} {heads} x {nq} causal={causal}")
        if not causal:
            ws = attn.workspace(B, DEV, nq)
            windows = [(0, 512), (512, -1)]
            o = torch.empty(2, B, nq, hq, 128, dtype=torch.float32, device=DEV)
            lse = torch.empty(2, B, nq, hq, dtype=torch.float32, device=DEV)
            for i, (a, b) in enumerate(windows):
                _cabi.decode_paged_multi(q.to(DEV), cache, bt, sl, signs, attn.scale, ws, o[i], out_lse=lse[i], kv_begin=a, kv_end=b,
                                         rotated_partial=True, num_ctas=148)
            merged = torch.empty(B * nq, hq, D, dtype=torch.float32, device=DEV)
            _cabi.merge_rotated(o.view(2, B * nq, hq, 128), lse.view(2, B * nq, hq), signs, merged)
            assert attn.status(B, DEV, nq) == 0
            assert_attention_close(merged.cpu().numpy(), want, f"{name} {heads} x {nq}, windows")
