"""The cache write of many 16-bit rows of 96, or padded to 64 or 256, a lane (two lanes) a row.  Every byte equals the oracle's, and over many random
rows that of the kernel that divides and searches for every element."""
import numpy as np
import pytest
import torch

from turboquant_b200 import _cabi, synthetic

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _slot(d):
    padded = 1 << (d - 1).bit_length()
    return (padded // 2 + 2 * (padded // 64) + 15) // 16 * 16


def _write(k, v, slots, nb, heads, d, signs, path="auto", fill=0xEE, slot=None, zero_pad=False):
    cache = torch.full((2, nb, 16, heads, slot or _slot(d)), fill, dtype=torch.uint8, device=DEV)
    _cabi.write_kv_cache(cache, k, v, signs.to(DEV), slots, d, path=path, zero_pad=zero_pad)
    return cache.cpu().numpy()


def _special(x, dtype):
    """Rows off the common path and next to it: zeros, some zeros, tiny, subnormal, huge, infinite, NaN, one- and two-hot (ties)."""
    rows = x.view(-1, x.shape[-1])
    d = rows.shape[-1]
    rows[0] = 0.0
    rows[1, ::3] = 0.0
    rows[2] *= 1e-30
    rows[3] = 0.0
    rows[3, 5] = 1e-38 if dtype == torch.bfloat16 else 6e-8
    rows[4, 7] = 1e-25 if dtype == torch.bfloat16 else 6e-8       # one tiny value among ordinary ones
    rows[5] *= 1e30 if dtype == torch.bfloat16 else 1e4
    rows[6, d - 1] = float("inf")
    rows[7, 0] = float("nan")
    rows[8] = 0.0
    rows[8, d // 2] = -3.0
    rows[9] = 0.0
    rows[9, 1], rows[9, d - 2] = 1.0, -1.0
    rows[10] = 1.0
    rows[11, 3], rows[11, 4] = float("inf"), float("-inf")
    rows[12] = 3e38 if dtype == torch.bfloat16 else 6e4           # the sum of squares overflows (bf16)
    return x


def _same(got, want):
    """Codes everywhere, norms where they are numbers; a NaN's pattern is the canonical one here and its input's in the oracle."""
    np.testing.assert_array_equal(got[..., :_codes(got)], want[..., :_codes(want)])
    n = _codes(got)
    a, b = got[..., n:n + 2].copy().view(np.float16), want[..., n:n + 2].copy().view(np.float16)
    nan = np.isnan(b)
    assert np.isnan(a[nan]).all()
    np.testing.assert_array_equal(a[~nan].view(np.uint16), b[~nan].view(np.uint16))


def _codes(cache):
    return {48: 32, 64: 32, 80: 64, 144: 128, 160: 128}[cache.shape[-1]]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d,heads,tokens", [(64, 8, 523), (64, 1, 4129), (64, 20, 211), (64, 3, 1400), (56, 6, 701), (256, 8, 521), (256, 1, 4111), (256, 5, 833),
                                            (192, 16, 259), (136, 2, 2051), (96, 8, 1030), (96, 40, 207), (96, 3, 2735)])
def test_large_writes_vs_oracle(oracle, d, heads, tokens, dtype):
    gen = torch.Generator().manual_seed(d + heads)
    k = _special(torch.randn(tokens, heads, d, generator=gen), dtype).to(dtype)
    v = (torch.randn(tokens, heads, d, generator=gen) * 3.0).to(dtype)
    k[..., 3] *= 20.0
    padded = 1 << (d - 1).bit_length()
    signs = synthetic.make_signs(padded, 42)
    nb = (tokens + 15) // 16 + 2
    slots = torch.randperm(nb * 16, generator=gen)[:tokens]
    slots[torch.randperm(tokens, generator=gen)[:17]] = -1
    slots[40], slots[41] = nb * 16, 1 << 40                        # outside the cache: dropped and counted
    mapped = slots.clone()
    mapped[40] = mapped[41] = -1
    want = np.full((2, nb, 16, heads, _slot(d)), 0xEE, np.uint8)
    oracle.write_kv_cache(want, k.float().numpy(), v.float().numpy(), signs.numpy(), mapped.numpy(), d)
    before = _cabi.fault_counts()[0]
    got = _write(k.to(DEV), v.to(DEV), slots.to(DEV), nb, heads, d, signs)
    assert _cabi.fault_counts()[0] - before == 2
    _same(got, want)
    used = padded // 2 + 2 * (padded // 64)
    assert (got[..., used:] == 0xEE).all()                         # pad and skipped slots untouched
    np.testing.assert_array_equal((got == 0xEE).all(-1), (want == 0xEE).all(-1))
    # tokens apart (slices of a fused projection), 32-bit slots, zeroed pads, the second tensor first
    both = torch.zeros(tokens, 3 * heads + 1, d, dtype=dtype, device=DEV)
    both[:, heads:2 * heads], both[:, 2 * heads:3 * heads] = k.to(DEV), v.to(DEV)
    got = _write(both[:, heads:2 * heads], both[:, 2 * heads:3 * heads], mapped.to(torch.int32).to(DEV), nb, heads, d, signs, zero_pad=True)
    _same(got, want)
    live = ~(want == 0xEE).all(-1)
    assert (got[live][:, used:] == 0).all() and (got[~live] == 0xEE).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d,slot", [(64, None), (64, 64), (256, None), (256, 160), (96, None)])
def test_volume_vs_the_dividing_kernel(d, slot, dtype):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(d)
    tokens, heads = 1 << 15, 8
    k = torch.randn(tokens, heads, d, generator=gen, device=DEV)
    k[..., 17] *= 20.0
    v = torch.randn(tokens, heads, d, generator=gen, device=DEV)
    v[::5] *= 1e-3
    v[::7] *= 300.0
    v[::11, :, 2:] = 0.0                                           # two-hot: ties and values next to boundaries
    k, v = k.to(dtype), v.to(dtype)
    signs = synthetic.make_signs(1 << (d - 1).bit_length(), 42)
    slots = torch.randperm(tokens, generator=torch.Generator().manual_seed(1)).to(DEV)
    got = _write(k, v, slots, tokens // 16, heads, d, signs, slot=slot)
    want = _write(k, v, slots, tokens // 16, heads, d, signs, path="exact", slot=slot)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("d", [64, 96, 256])
def test_norms_whose_significand_is_all_ones(oracle, d):
    """There the refined reciprocal may miss the IEEE quotient."""
    gen = torch.Generator().manual_seed(5)
    left, four = 4.0 - 2.0 ** -21, []                              # the square of 2 - 2^-23, as squares of bf16 values
    for _ in range(4):
        a = torch.tensor(left ** 0.5, dtype=torch.float64).to(torch.bfloat16).double().item()
        if a * a > left:
            a = (torch.tensor(a, dtype=torch.bfloat16).view(torch.int16) - 1).view(torch.bfloat16).double().item()
        four.append(a)
        left -= a * a
    four = torch.tensor(four)
    total = torch.tensor(0.0)
    for a in four:
        total = total + a * a
    assert int(torch.sqrt(total).view(torch.int32)) & 0x7FFFFF == 0x7FFFFF
    x = torch.zeros(1200, 8, d)
    flips = torch.randint(0, 2, (9600, 4), generator=gen) * 2.0 - 1.0
    x.view(-1, d)[:, :4] = four * flips * torch.exp2(torch.randint(-10, 11, (9600, 1), generator=gen).float())
    x = x.to(torch.bfloat16)
    signs = synthetic.make_signs(1 << (d - 1).bit_length(), 42)
    slots = torch.arange(1200)
    want = np.full((2, 75, 16, 8, _slot(d)), 0xEE, np.uint8)
    oracle.write_kv_cache(want, x.float().numpy(), x.float().numpy(), signs.numpy(), slots.numpy(), d)
    _same(_write(x.to(DEV), x.to(DEV), slots.to(DEV), 75, 8, d, signs), want)


@pytest.mark.parametrize("d", [64, 256])
def test_signs_other_than_one_are_factors(oracle, d):
    gen = torch.Generator().manual_seed(9)
    x = torch.randn(700, 8, d, generator=gen).to(torch.float16)
    slots = torch.arange(700)
    for signs in (0.5 * synthetic.make_signs(d, 42), torch.randn(d, generator=gen) * 0.9):
        want = np.full((2, 44, 16, 8, _slot(d)), 0xEE, np.uint8)
        oracle.write_kv_cache(want, x.float().numpy(), x.float().numpy(), signs.numpy(), slots.numpy(), d)
        _same(_write(x.to(DEV), x.to(DEV), slots.to(DEV), 44, 8, d, signs), want)


@pytest.mark.parametrize("d,heads,tokens", [(64, 8, 600), (256, 3, 1500), (96, 5, 1700)])
def test_token_strides_that_are_no_multiple_of_a_row(d, heads, tokens):
    """K and V side by side with eight elements behind them, against the same rows dense."""
    gen = torch.Generator().manual_seed(d)
    both = torch.randn(tokens, 2 * heads * d + 8, generator=gen).to(torch.bfloat16).to(DEV)
    k, v = (t.unflatten(1, (heads, d)) for t in (both[:, :heads * d], both[:, heads * d:2 * heads * d]))
    signs = synthetic.make_signs(1 << (d - 1).bit_length(), 42)
    nb = (tokens + 15) // 16
    slots = torch.randperm(nb * 16, generator=gen)[:tokens].to(DEV)
    np.testing.assert_array_equal(_write(k, v, slots, nb, heads, d, signs), _write(k.contiguous(), v.contiguous(), slots, nb, heads, d, signs, path="exact"))


@pytest.mark.parametrize("d,heads", [(64, 8), (64, 3), (96, 8), (256, 5)])
def test_several_units_a_warp(d, heads):
    """Three units of every warp and a part of one, against the kernel that divides and searches for every element."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = 3 * sms * (20 if d == 64 else 12) * (16 if d == 256 else 32)
    tokens = rows // (2 * heads) + 37
    gen = torch.Generator(device=DEV)
    gen.manual_seed(d + heads)
    k, v = ((torch.randn(tokens, heads, d, generator=gen, device=DEV) * 2.0).to(torch.float16) for _ in range(2))
    signs = synthetic.make_signs(1 << (d - 1).bit_length(), 42)
    nb = (tokens + 15) // 16
    slots = torch.randperm(nb * 16, generator=torch.Generator().manual_seed(2))[:tokens].to(DEV)
    np.testing.assert_array_equal(_write(k, v, slots, nb, heads, d, signs), _write(k, v, slots, nb, heads, d, signs, path="exact"))
