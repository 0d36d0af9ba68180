"""TurboQuantPagedAttention as a plain Python object: it can be copied and pickled, also after calls, and an attribute
that is set between calls counts from the next one on."""
import copy
import pickle

import pytest
import torch

from turboquant_b200 import TurboQuantPagedAttention
from turboquant_b200.paged_attention import kv_cache_shape


@pytest.mark.parametrize("used", [False, True])
def test_copies(used):
    a = TurboQuantPagedAttention(32, 128, 0.25, 8)
    if used:
        pytest.importorskip("turboquant_b200._native")
        a.signs("cpu")
        assert a._calls is a._calls
    for b in (copy.copy(a), copy.deepcopy(a), pickle.loads(pickle.dumps(a))):
        assert (b.num_heads, b.head_size, b.scale, b.num_kv_heads, b.num_ctas) == (32, 128, 0.25, 8, 0)
        assert b._layer is None
        assert torch.equal(b.signs("cpu"), a.signs("cpu"))


def test_geometry_set_later_drops_the_native_layer():
    pytest.importorskip("turboquant_b200._native")
    a = TurboQuantPagedAttention(32, 128, 0.25, 8)
    first = a._calls
    a.scale = 0.5
    assert a._calls is not first


@pytest.mark.gpu
@pytest.mark.parametrize("head_size", [64, 128])
def test_scale_set_between_calls_and_copy_give_the_same_output(head_size):
    a = TurboQuantPagedAttention(8, head_size, 0.05, 4)
    gen = torch.Generator("cuda").manual_seed(5)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda", dtype=torch.float16)
    cache = torch.zeros(kv_cache_shape(4, 16, 4, head_size), dtype=torch.uint8, device="cuda")
    a.write(rand(64, 4, head_size), rand(64, 4, head_size), cache, torch.arange(64, device="cuda"))
    table = torch.arange(4, dtype=torch.int32, device="cuda").view(1, 4)
    lens = torch.tensor([61], dtype=torch.int32, device="cuda")
    q = 4 * rand(1, 8, head_size)

    def twice(x):
        outs = [x.decode(q, cache, table, lens) for _ in range(2)]
        assert torch.equal(*outs)
        return outs[0]

    before = twice(a)
    a.scale = 0.5
    want = twice(TurboQuantPagedAttention(8, head_size, 0.5, 4))
    assert not torch.equal(before, want)
    assert torch.equal(twice(a), want)
    assert torch.equal(twice(copy.deepcopy(a)), want)
