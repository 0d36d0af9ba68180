"""The four-lane row kernels of the flat quantizer: every padded size, bit width, element type and pack order, row counts around
the eight rows of a warp pass, rows on the exceptional paths.  Codes, norms and dequantized values equal the oracle's bit for bit."""
import numpy as np
import pytest
import torch

from turboquant_b200 import _cabi, synthetic

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rows(n, dim, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(n, dim, generator=g)
    x[:, 1 % dim] *= 20.0                                  # an outlier channel
    for i, v in enumerate((0.0, 1e-30, 3e-5, 6e4)):        # zero, tiny and large rows
        if n > 8 + i:
            x[8 + i] = v
    if n > 16:
        x[13, 3], x[14, 5], x[15] = float("inf"), float("nan"), 0.0
        x[15, 7] = 1.0                                     # one-hot: ties of the transform's outputs
    return x.to(dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("dim,n", [(128, 1), (128, 7), (128, 65), (64, 8), (64, 1000), (96, 66), (72, 9), (256, 33), (192, 300)])
def test_rows_match_the_oracle(oracle, dim, n, dtype):
    signs = synthetic.make_signs(1 << (dim - 1).bit_length(), 42)
    x = _rows(n, dim, dtype, 3 + dim + n)
    for bits in (1, 2, 3, 4):
        per = 8 // bits
        want_p, want_n = oracle.quantize_flat(x.float().numpy(), signs.numpy(), bits)
        codes = (want_p[:, :, None] >> (bits * np.arange(per, dtype=np.uint8))) & ((1 << bits) - 1)
        want_c = (codes << (bits * np.arange(per - 1, -1, -1, dtype=np.uint8))).sum(axis=2).astype(np.uint8)
        for cache_order, want in ((False, want_p), (True, want_c)):
            p, norms = _cabi.quantize_flat(x.to(DEV), signs.to(DEV), bits, cache_order=cache_order)
            np.testing.assert_array_equal(p.cpu().numpy(), want, err_msg=f"bits {bits} cache order {cache_order}")
            # bit for bit, except that a NaN is the canonical one here and carries its input's payload in the oracle
            np.testing.assert_array_equal(norms.cpu().numpy(), want_n)
            out = _cabi.dequantize_flat(p, norms, signs.to(DEV), dim, bits, cache_order=cache_order)
            np.testing.assert_array_equal(out.cpu().numpy(), oracle.dequantize_flat(want_p, want_n, signs.numpy(), dim, bits))


@pytest.mark.parametrize("dim", [128, 100])                 # the row kernels and the plain ones
def test_pack_order_takes_any_truth_value(dim):
    x, signs = _rows(20, dim, torch.float16, 5).to(DEV), synthetic.make_signs(128, 42).to(DEV)
    want, norms = _cabi.quantize_flat(x, signs, 4, cache_order=True)
    low_first, _ = _cabi.quantize_flat(x, signs, 4, cache_order=False)
    assert not torch.equal(want, low_first)
    back = _cabi.dequantize_flat(want, norms, signs, dim, 4, cache_order=True)
    for yes, no in ((1, 0), (np.bool_(True), np.bool_(False)), ("cache", None)):
        assert torch.equal(_cabi.quantize_flat(x, signs, 4, cache_order=yes)[0], want)
        assert torch.equal(_cabi.quantize_flat(x, signs, 4, cache_order=no)[0], low_first)
        assert torch.equal(_cabi.dequantize_flat(want, norms, signs, dim, 4, cache_order=yes).nan_to_num(), back.nan_to_num())
        assert torch.equal(_cabi.dequantize_flat(low_first, norms, signs, dim, 4, cache_order=no).nan_to_num(), back.nan_to_num())
    with pytest.raises(ValueError):
        _cabi.quantize_flat(x, signs, 4, cache_order=np.array([True, False]))      # no truth value


@pytest.mark.parametrize("dim", [64, 128, 256])
def test_signs_beyond_one(oracle, dim):
    """Any sign vector is taken: the row kernels agree with the plain ones (which rows that start off their alignment take) and, where all
    values are finite, with the oracle."""
    g = torch.Generator().manual_seed(dim)
    x = _rows(50, dim, torch.float16, 4)
    odd = torch.empty(50 * dim + 1, dtype=torch.float16, device=DEV)[1:].view(50, dim)
    odd.copy_(x)
    ones = synthetic.make_signs(dim, 42)
    for name, signs in (("threes", 3.0 * ones), ("wide", torch.randn(dim, generator=g) * 1e6), ("fractions", 0.5 * ones), ("zeros", 0.0 * ones),
                        ("infinite", torch.where(torch.arange(dim) % 17 == 3, ones * float("inf"), ones)),
                        ("nan", torch.where(torch.arange(dim) == 5, ones * float("nan"), ones)), ("largest", ones * 3.4e38)):
        for bits in (1, 2, 3, 4):
            p, norms = _cabi.quantize_flat(x.to(DEV), signs.to(DEV), bits)
            plain, plain_norms = _cabi.quantize_flat(odd, signs.to(DEV), bits)
            assert torch.equal(p, plain), (name, bits)
            np.testing.assert_array_equal(norms.cpu().numpy(), plain_norms.cpu().numpy())
            if bool((signs.abs() < 1e30).all()):
                np.testing.assert_array_equal(p.cpu().numpy(), oracle.quantize_flat(x.float().numpy(), signs.numpy(), bits)[0], err_msg=f"{name} {bits}")


@pytest.mark.parametrize("dim,n", [(128, 8192), (128, 8200 + 17), (96, 8192 + 31), (72, 8195), (64, 49152), (64, 49152 + 33), (256, 2048), (256, 2048 + 15), (192, 2051),
                                   (128, 14300), (96, 9600 + 31), (72, 9603), (192, 4803)])
def test_dequantization_of_many_rows(oracle, dim, n):
    """Many rows, around the counts from which a lane (two lanes) takes a row: part units, short rows, both pack orders, any sign vector."""
    padded = 1 << (dim - 1).bit_length()
    rng = np.random.default_rng(dim + n)
    norms = rng.uniform(0.0, 30.0, n).astype(np.float32)
    norms[:3] = np.inf, np.nan, 0.0
    signs = synthetic.make_signs(padded, 42)
    for bits in (2, 3, 4):
        per = 8 // bits
        codes = rng.integers(0, 1 << bits, (n, padded // per, per), dtype=np.uint8)
        low = (codes << (bits * np.arange(per, dtype=np.uint8))).sum(axis=2).astype(np.uint8)
        high = (codes << (bits * np.arange(per - 1, -1, -1, dtype=np.uint8))).sum(axis=2).astype(np.uint8)
        want = oracle.dequantize_flat(low, norms, signs.numpy(), dim, bits)
        for packed, order in ((low, False), (high, True)):
            out = _cabi.dequantize_flat(torch.from_numpy(packed).to(DEV), torch.from_numpy(norms).to(DEV), signs.to(DEV), dim, bits, cache_order=order)
            np.testing.assert_array_equal(out.cpu().numpy(), want, err_msg=f"bits {bits} cache order {order}")
    # factors other than +-1, against the four-lane kernel (the same rows in short calls)
    signs = torch.from_numpy(rng.normal(size=padded).astype(np.float32)).to(DEV)
    packed, norms = torch.from_numpy(low).to(DEV), torch.from_numpy(norms).to(DEV)
    parts = [_cabi.dequantize_flat(packed[i:i + 2000], norms[i:i + 2000], signs, dim, 4) for i in range(0, n, 2000)]
    assert torch.equal(_cabi.dequantize_flat(packed, norms, signs, dim, 4).nan_to_num(), torch.cat(parts).nan_to_num())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("dim,n", [(128, 8192), (128, 8192 + 17), (96, 8192 + 31), (72, 8195), (64, 16384), (64, 16384 + 33), (256, 4096), (256, 4096 + 15), (192, 4099),
                                   (128, 9600 + 17), (96, 9600 + 31), (72, 9603)])
def test_quantization_of_many_rows(oracle, dim, n, dtype):
    """Many rows, around the counts from which a lane (two lanes) takes a row: part units, short rows, special rows, every width and both pack orders."""
    signs = synthetic.make_signs(1 << (dim - 1).bit_length(), 42)
    x = _rows(n, dim, dtype, 7 + dim + n)
    if dtype == torch.bfloat16:
        x[20, 5], x[21] = 1e-30, 0.0                       # a tiny value among ordinary ones; a zero row
        x[22] *= 1e-35
    for bits in (1, 2, 3, 4):
        per = 8 // bits
        want_p, want_n = oracle.quantize_flat(x.float().numpy(), signs.numpy(), bits)
        codes = (want_p[:, :, None] >> (bits * np.arange(per, dtype=np.uint8))) & ((1 << bits) - 1)
        want_c = (codes << (bits * np.arange(per - 1, -1, -1, dtype=np.uint8))).sum(axis=2).astype(np.uint8)
        for cache_order, want in ((False, want_p), (True, want_c)):
            p, norms = _cabi.quantize_flat(x.to(DEV), signs.to(DEV), bits, cache_order=cache_order)
            np.testing.assert_array_equal(p.cpu().numpy(), want, err_msg=f"bits {bits} cache order {cache_order}")
            np.testing.assert_array_equal(norms.cpu().numpy(), want_n)
    # factors other than +-1, against the four-lane kernel (the same rows in short calls)
    g = torch.Generator().manual_seed(n)
    for factors in (torch.randn(signs.numel(), generator=g), 3e30 * signs, torch.where(torch.arange(signs.numel()) == 5, float("nan"), signs)):
        factors = factors.to(DEV)
        for bits in (2, 4):
            p, norms = _cabi.quantize_flat(x.to(DEV), factors, bits)
            parts = [_cabi.quantize_flat(x[i:i + 2000].to(DEV), factors, bits) for i in range(0, n, 2000)]
            assert torch.equal(p, torch.cat([a for a, _ in parts]))
            np.testing.assert_array_equal(norms.cpu().numpy(), torch.cat([b for _, b in parts]).cpu().numpy())


@pytest.mark.parametrize("dim,n", [(64, 49152), (128, 14300), (256, 2048), (192, 4803)])
def test_zeros_keep_their_sign_in_many_rows(oracle, dim, n):
    """Rows of repeated codes, whose sums cancel: the outputs' bits, which tell -0 from +0, with norms of zero among them."""
    padded = 1 << (dim - 1).bit_length()
    rng = np.random.default_rng(dim)
    signs = synthetic.make_signs(padded, 42)
    norms = rng.uniform(0.5, 30.0, n).astype(np.float32)
    norms[::7] = 0.0
    for bits in (2, 3, 4):
        per = 8 // bits
        codes = np.repeat(rng.integers(0, 1 << bits, (n, padded // 8), dtype=np.uint8), 8, axis=1)
        codes[::3] = codes[::3, :1]
        codes[::5, :padded // 2], codes[::5, padded // 2:] = codes[::5, :1], (1 << bits) - 1 - codes[::5, :1]
        packed = (codes.reshape(n, padded // per, per) << (bits * np.arange(per, dtype=np.uint8))).sum(axis=2).astype(np.uint8)
        want = oracle.dequantize_flat(packed, norms, signs.numpy(), dim, bits)
        assert (want == 0).any()
        got = _cabi.dequantize_flat(torch.from_numpy(packed).to(DEV), torch.from_numpy(norms).to(DEV), signs.to(DEV), dim, bits)
        np.testing.assert_array_equal(got.cpu().numpy().view(np.int32), want.view(np.int32), err_msg=f"bits {bits}")


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def _same_as_short_calls(oracle, dim, n, dtype, widths=(1, 2, 3, 4)):
    """One call of n rows, there and back, against the same rows in calls short enough for the four-lane kernels, and the first and last against the oracle."""
    padded = 1 << (dim - 1).bit_length()
    short = {64: 16000, 128: 9000, 256: 1900}[padded]
    signs = synthetic.make_signs(padded, 42)
    x, on_gpu = _rows(n, dim, dtype, dim + n).to(DEV), signs.to(DEV)
    for bits in widths:
        for cache_order in (False, True):
            p, norms = _cabi.quantize_flat(x, on_gpu, bits, cache_order=cache_order)
            out = _cabi.dequantize_flat(p, norms, on_gpu, dim, bits, cache_order=cache_order)
            for i in range(0, n, short):
                few_p, few_norms = _cabi.quantize_flat(x[i:i + short], on_gpu, bits, cache_order=cache_order)
                assert torch.equal(p[i:i + short], few_p), (bits, cache_order, i)
                assert torch.equal(norms[i:i + short].nan_to_num(7.0), few_norms.nan_to_num(7.0))
                few = _cabi.dequantize_flat(few_p, few_norms, on_gpu, dim, bits, cache_order=cache_order)
                nan = few.isnan()
                assert torch.equal(out[i:i + short].isnan(), nan)
                assert torch.equal(out[i:i + short].masked_fill(nan, 0).view(torch.int32), few.masked_fill(nan, 0).view(torch.int32)), (bits, cache_order, i)
            if not cache_order:
                for part in (slice(0, 40), slice(n - 40, n)):
                    want_p, want_n = oracle.quantize_flat(x[part].float().cpu().numpy(), signs.numpy(), bits)
                    np.testing.assert_array_equal(p[part].cpu().numpy(), want_p)
                    np.testing.assert_array_equal(norms[part].cpu().numpy(), want_n)
                    np.testing.assert_array_equal(out[part].cpu().numpy(), oracle.dequantize_flat(want_p, want_n, signs.numpy(), dim, bits))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("dim,per_sm", [(64, 110), (64, 332), (128, 64), (128, 96), (96, 64), (72, 64), (256, 13), (256, 27), (136, 13), (136, 32)])
def test_rows_an_sm_where_the_kernels_change(oracle, dim, per_sm, dtype):
    for n in (per_sm * _sms(), per_sm * _sms() + 1):
        _same_as_short_calls(oracle, dim, n, dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("dim", [40, 64, 72, 96, 128, 136, 256])
def test_several_units_a_warp(oracle, dim, dtype):
    """Three units of every warp and a part of one: each stage of a warp's ring is filled again after it has been read out."""
    padded = 1 << (dim - 1).bit_length()
    a_round = _sms() * (20 if padded == 64 else 12) * (16 if padded == 256 else 32)
    _same_as_short_calls(oracle, dim, 3 * a_round + 5, dtype)
