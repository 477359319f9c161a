"""The rotation of qk_norm_rope rounds the double-precision result once, also where the fp32 arithmetic that serves nearly
all pairs cannot decide: next to the middle between two 16-bit values, at magnitudes where products over- or underflow,
on both sides of the type's largest value, at zeros and infinities.  All bits are compared, signs of zero included, except
that any NaN equals any other."""
import pytest
import torch

from oracle import vecattn_oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("what", ["ordinary", "boundaries", "extremes", "overflow", "zeros"])
def test_rotation_rounds_once(built_library, dtype, what):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    from vecattention_b200.preattn import qk_norm_rope
    g = torch.Generator().manual_seed(11)
    s, h = 700, 3
    x = torch.randn(1, s, h * 128, generator=g)
    cos, sin = torch.randn(s, 64, generator=g), torch.randn(s, 64, generator=g)
    if what == "boundaries":
        # results e + o * 2^-m exactly in the middle of two 16-bit values, or a last fp32 place beside it
        bits = 8 if dtype == torch.bfloat16 else 11
        x = 1 + torch.randint(0, 1 << (bits - 1), x.shape, generator=g) / float(1 << (bits - 1))
        x[..., 1::2] = 1.0
        cos[:] = 1.0
        sin[:] = -(2.0 ** -bits) * (1 + torch.randint(-2, 3, sin.shape, generator=g) * 2.0 ** -23)
    elif what == "extremes":
        # every product is 0 or above 2^-149 (2^-50 of each factor, times normal draws, none under 2^-26 and 2^-18): the
        # oracle's rounding goes through float32 and does not tell what underflows there to zero
        low, high = (-50, 120) if dtype == torch.bfloat16 else (-14, 14)
        x = x * 2.0 ** torch.randint(low, high + 1, x.shape, generator=g)
        x[:, ::7, ::5] = 0.0
        x[:, 3, 8:16] = float("inf")
        cos = cos * 2.0 ** torch.randint(-50, 30, cos.shape, generator=g)
        sin[::3] = 0.0
        sin[1::5] *= 2.0 ** -50
    elif what == "overflow":
        # results within two fp32 places of the middle between the largest value and what would be the next one
        bits, top = (8, 127) if dtype == torch.bfloat16 else (11, 15)
        x = (2 - 2.0 ** (1 - bits)) * 2.0 ** top * torch.where(x < 0, -1.0, 1.0)
        middle = (2 - 2.0 ** -bits) / (2 - 2.0 ** (1 - bits))
        cos = middle * (1 + torch.randint(-2, 3, cos.shape, generator=g) * 2.0 ** -23)
        sin[:] = 0.0
    elif what == "zeros":
        x = torch.where(x < 0, -0.0, 0.0)
        x[..., 7::64] = 1.0
        cos[5::50], sin[7::50] = float("inf"), float("nan")
    x, cos, sin = x.to(dtype), cos.contiguous(), sin.contiguous()
    q, k = qk_norm_rope(x.cuda(), x.cuda(), None, None, 1e-6, cos.cuda(), sin.cuda(), 0, heads=h)
    ref = O.rope_interleaved(x.view(1, s, h, 128).transpose(1, 2), cos, sin)
    for got in (q.cpu(), k.cpu()):
        number = ~ref.isnan()
        assert torch.equal(~got.isnan(), number)
        assert torch.equal(got.contiguous().view(torch.int16)[number], ref.contiguous().view(torch.int16)[number])


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_rows_of_zeros_take_no_longer(built_library, dtype):
    """Padding is as fast as anything else (measured: 1.05 times the time, 1.4 before; 1.25 leaves
    room for the clock)."""
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    from vecattention_b200.preattn import qk_norm_rope
    s, h = 30000, 24
    angle = torch.rand(s, 64, device="cuda")
    cos, sin = angle.cos(), angle.sin()
    w = torch.ones(h * 128, dtype=dtype, device="cuda")

    def fastest(x):
        times = []
        for _ in range(8):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            qk_norm_rope(x, x, w, w, 1e-6, cos, sin, 0, heads=h)
            e[1].record()
            torch.cuda.synchronize()
            times.append(e[0].elapsed_time(e[1]))
        return min(times)

    x = torch.randn(1, s, h * 128, device="cuda").to(dtype)
    assert fastest(torch.zeros_like(x)) <= 1.25 * fastest(x)
