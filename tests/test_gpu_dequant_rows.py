"""Bulk dequantization at the edges of its units of work: 16 or 32 rows of a page, K rows before V rows, in the kernel of small jobs and (behind a
wide page table) in that of large ones.  fp32 output equals the oracle bit for bit, 16-bit output is its rounding."""
import numpy as np
import pytest
import torch

from turboquant_b200 import _cabi, synthetic

pytestmark = pytest.mark.gpu
DEV = "cuda"
LENS = [0, 1, 15, 16, 17, 33, 160, 0, 97]
SLOT = {64: 48, 96: 80, 128: 80, 256: 144}


def _cache(rng, pages, block, heads, dim, slot):
    """Random codes, finite fp16 norms."""
    cache = rng.integers(0, 256, (2, pages, block, heads, slot), dtype=np.uint8)
    padded = 1 << (dim - 1).bit_length()
    norms = rng.uniform(0.0, 20.0, cache.shape[:-1]).astype(np.float16)
    cache[..., padded // 2:padded // 2 + 2] = norms[..., None].view(np.uint8)
    return cache


def _want(oracle, cache, table, lens, signs, dim):
    block = cache.shape[2]
    slot = SLOT[dim]
    rows = []
    for which in range(2):
        parts = []
        for b, n in enumerate(lens):
            t = np.arange(n)
            got = np.ascontiguousarray(cache[which, table[b, t // block], t % block][..., :slot])
            parts.append(oracle.dequant_cache_rows(got, signs, dim).reshape(n, cache.shape[3], dim))
        rows.append(np.concatenate(parts))
    return rows


def _check(oracle, dim, heads, *, wide, block=16, slot=None, strided=False, listed=False, lens=LENS):
    rng = np.random.default_rng(dim + heads + block)
    slot = slot or SLOT[dim]
    signs = synthetic.make_signs(1 << (dim - 1).bit_length(), 42)
    need = max((n + block - 1) // block for n in lens)
    pages = sum((n + block - 1) // block for n in lens) + 2
    cache = _cache(rng, pages, block, heads, dim, slot)
    order, at = rng.permutation(pages), 0
    units = 2 * heads * block // 32 + 1
    width = need if not wide else max(need, 24 * 160 // (len(lens) * units) * units + 4000 // units)      # beyond the small jobs' bound
    table = np.zeros((len(lens), width), np.int32)
    for b, n in enumerate(lens):
        k = (n + block - 1) // block
        table[b, :k] = order[at:at + k]
        at += k
    want = _want(oracle, cache, table, lens, signs.numpy(), dim)
    total = sum(lens)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device=DEV)
    extra = {}
    pages_arg = torch.from_numpy(table).to(DEV)
    if listed:
        per = [(n + block - 1) // block for n in lens]
        pages_arg = torch.from_numpy(np.concatenate([table[b, :k] for b, k in enumerate(per)])).to(DEV)
        extra = dict(page_indptr=torch.tensor(np.concatenate([[0], np.cumsum(per)]), dtype=torch.int32, device=DEV), max_pages=width)
    for dtype in (torch.float32, torch.bfloat16, torch.float16):
        if strided:
            both = torch.full((total + 1, 2, heads, dim), 7.0, dtype=dtype, device=DEV)
            k, v = both[:total, 0], both[:total, 1]
        else:
            both = torch.full((2, total + 1, heads, dim), 7.0, dtype=dtype, device=DEV)
            k, v = both[0, :total], both[1, :total]
        _cabi.dequant_paged(torch.from_numpy(cache).to(DEV), pages_arg, torch.tensor(lens, dtype=torch.int32, device=DEV), cu, signs.to(DEV), k, v, **extra)
        for got, ref in ((k, want[0]), (v, want[1])):
            assert torch.equal(got.cpu(), torch.from_numpy(ref).to(dtype)), (dtype, dim, heads)
        rest = both[total] if strided else both[:, total]
        assert bool((rest == 7.0).all())      # nothing past the last row


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("dim,heads", [(128, 1), (128, 3), (128, 8), (96, 2), (96, 5), (64, 1), (64, 8), (64, 5), (256, 1), (256, 4), (256, 3)])
def test_edges_of_units(oracle, dim, heads, wide):
    _check(oracle, dim, heads, wide=wide)
    _check(oracle, dim, heads, wide=wide, strided=True)


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("dim,heads,block,slot,listed", [(128, 3, 5, None, False), (96, 4, 1, None, True), (128, 8, 16, 96, True), (64, 2, 16, 64, False),
                                                         (256, 2, 16, 160, True)])
def test_other_pages_and_slots(oracle, dim, heads, block, slot, listed, wide):
    """Page sizes that leave part units, slots with bytes behind them (copied row by row), lists of pages."""
    _check(oracle, dim, heads, wide=wide, block=block, slot=slot, listed=listed)


@pytest.mark.parametrize("dim", [64, 128])
def test_many_sequences(oracle, dim):
    """More sequences than a warp has lanes, most of them short or empty; a job of many units a warp against the oracle."""
    rng = np.random.default_rng(dim)
    _check(oracle, dim, 1, wide=False, lens=[int(n) for n in rng.integers(0, 40, 100)])
    _check(oracle, dim, 8, wide=True, lens=[int(n) for n in rng.integers(0, 70, 70)])
    _check(oracle, dim, 16, wide=False, lens=[3, 0, 60000 if dim == 64 else 66000, 20])


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("dim,heads", [(64, 3), (96, 2), (128, 3), (256, 2)])
def test_zeros_keep_their_sign(oracle, dim, heads, wide):
    """Rows of repeated codes, whose sums cancel: the outputs' bits, which tell -0 from +0, with norms of zero among them."""
    rng = np.random.default_rng(dim)
    padded, tokens = 1 << (dim - 1).bit_length(), 96
    cache = _cache(rng, tokens // 16, 16, heads, dim, SLOT[dim])
    rows = cache.reshape(-1, SLOT[dim])
    rows[:, :padded // 2] = np.repeat(rng.integers(0, 256, (len(rows), padded // 16), dtype=np.uint8), 8, axis=1)
    rows[::3, :padded // 2] = rows[::3, :1]
    rows[::5, :padded // 4], rows[::5, padded // 4:padded // 2] = rows[::5, :1], ~rows[::5, :1]
    rows[::7, padded // 2:padded // 2 + 2] = 0
    signs = synthetic.make_signs(padded, 42)
    table = np.zeros((1, 60000 if wide else tokens // 16), np.int32)      # a wide table: beyond the small jobs' bound
    table[0, :tokens // 16] = rng.permutation(tokens // 16)
    want = _want(oracle, cache, table, [tokens], signs.numpy(), dim)
    assert any((w == 0).any() for w in want)
    for dtype in (torch.float32, torch.bfloat16):
        k, v = (torch.empty(tokens, heads, dim, dtype=dtype, device=DEV) for _ in range(2))
        _cabi.dequant_paged(torch.from_numpy(cache).to(DEV), torch.from_numpy(table).to(DEV), torch.tensor([tokens], dtype=torch.int32, device=DEV),
                            torch.tensor([0, tokens], dtype=torch.int32, device=DEV), signs.to(DEV), k, v)
        for got, ref in ((k, want[0]), (v, want[1])):
            as_int = torch.int32 if dtype == torch.float32 else torch.int16
            assert torch.equal(got.cpu().view(as_int), torch.from_numpy(ref).to(dtype).view(as_int)), (dtype, dim)


@pytest.mark.parametrize("dim,heads", [(128, 1), (64, 1), (256, 1)])
def test_every_bad_page_is_counted_once(dim, heads):
    """A job of more units a warp than are looked up at a time, all of its pages outside the cache: as many faults as pages, and nothing written."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = 16 if dim == 256 else 32                                    # of a unit: a page of one head has 32
    pages = 33 * sms * (20 if dim == 64 else 12) * rows // 32 + 7       # warps of a block
    table = torch.full((1, pages), 5, dtype=torch.int32, device=DEV)
    table[0, ::3] = -1
    cache = torch.zeros((2, 5, 16, heads, SLOT[dim]), dtype=torch.uint8, device=DEV)
    k, v = (torch.full((pages * 16, heads, dim), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    before = _cabi.fault_counts()
    _cabi.dequant_paged(cache, table, torch.tensor([pages * 16], dtype=torch.int32, device=DEV), torch.tensor([0, pages * 16], dtype=torch.int32, device=DEV),
                        synthetic.make_signs(dim, 42).to(DEV), k, v)
    assert _cabi.fault_counts()[1] - before[1] == pages
    assert bool((k == 7.0).all()) and bool((v == 7.0).all())


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("dim,heads,batch,listed", [(128, 8, 257, False), (128, 3, 1000, True), (96, 1, 600, False), (64, 5, 511, True), (256, 2, 513, False)])
def test_more_sequences_than_parts_of_the_work_list(oracle, dim, heads, batch, listed, wide):
    """A block's list of work has 256 parts: one and more sequences each, the last ones without any, empty sequences alone and in runs; sequences of one
    token, whose pages hold units of nothing but free slots."""
    rng = np.random.default_rng(batch)
    lens = rng.choice([0, 1, 1, 3, 16, 17, 40], batch)
    lens[:9], lens[100:180], lens[-5:] = 0, 0, 0
    lens[200:230] = 1
    _check(oracle, dim, heads, wide=wide, lens=[int(n) for n in lens], listed=listed)


@pytest.mark.parametrize("dim,dtype", [(64, torch.bfloat16), (96, torch.float16), (128, torch.bfloat16), (128, torch.float32), (256, torch.bfloat16)])
def test_more_units_a_warp_than_are_looked_up_at_a_time(dim, dtype):
    """Over sixty units a warp (32 are looked up at a time, twice over), three sequences with part pages: one call of the large blocks against calls of the small ones."""
    heads, padded = 16, 1 << (dim - 1).bit_length()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = 62 * sms * (20 if dim == 64 else 12) * (16 if dim == 256 else 32)
    pages = rows // (2 * 16 * heads) + 1
    lens = [pages * 10 - 3, 37, pages * 6 + 40]
    per = [(n + 15) // 16 for n in lens]
    g = torch.Generator(device=DEV)
    g.manual_seed(dim)
    cache = torch.randint(0, 256, (2, sum(per), 16, heads, SLOT[dim]), dtype=torch.uint8, device=DEV, generator=g)
    norms = torch.rand(cache.shape[:-1] + (1,), device=DEV, generator=g).to(torch.float16) * 20
    cache[..., padded // 2:padded // 2 + 2] = norms.view(torch.uint8)
    order = torch.randperm(sum(per), generator=torch.Generator().manual_seed(dim)).to(torch.int32).to(DEV)
    signs = synthetic.make_signs(padded, 42).to(DEV)
    table = torch.zeros(3, max(per), dtype=torch.int32, device=DEV)
    for b, at in enumerate((0, per[0], per[0] + per[1])):
        table[b, :per[b]] = order[at:at + per[b]]
    cu = [0, lens[0], lens[0] + lens[1], sum(lens)]
    k, v = (torch.full((sum(lens) + 1, heads, dim), 7.0, dtype=dtype, device=DEV) for _ in range(2))
    _cabi.dequant_paged(cache, table, torch.tensor(lens, dtype=torch.int32, device=DEV), torch.tensor(cu, dtype=torch.int32, device=DEV), signs, k, v)
    assert bool((k[-1] == 7.0).all()) and bool((v[-1] == 7.0).all())
    step = 100                                                         # pages of a small call
    for b in range(3):
        for first in range(0, per[b], step):
            n = min(lens[b] - first * 16, step * 16)
            few_k, few_v = (torch.empty(n, heads, dim, dtype=dtype, device=DEV) for _ in range(2))
            _cabi.dequant_paged(cache, table[b:b + 1, first:first + step].contiguous(), torch.tensor([n], dtype=torch.int32, device=DEV),
                                torch.tensor([0, n], dtype=torch.int32, device=DEV), signs, few_k, few_v)
            at = cu[b] + first * 16
            assert torch.equal(k[at:at + n], few_k) and torch.equal(v[at:at + n], few_v), (b, first)
