"""The split decode kernel with more than one tile of query columns (shared and causal queries): both sides of every tile edge, every
way the plan cuts a batch, a causal mask that crosses a page edge and hides whole pages, against the oracle."""
import math

import numpy as np
import pytest
import torch

from turboquant_b200 import TurboQuantPagedAttention, synthetic
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
