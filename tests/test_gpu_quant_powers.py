"""act_quant with power-of-two scales: quotients formed with the scale's reciprocal are the exact ones, for every such scale that a bf16
block can have and every bf16 value below its maximum; blocks that hold NaN or infinities; every place in a CTA's share of the work."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _e4m3(x):
    return x.clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)      # (round to nearest even, as the oracle)


@pytest.mark.parametrize("first", [-14, 20, 60, 100])
def test_every_power_of_two_scale(first):
    import kernel
    every = torch.arange(0, 0x7F80, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.bfloat16)      # finite, not negative
    for e in range(first, min(first + 40, 128)):
        for frac in (1.0, 1.5, 1.75, 1.9921875):                             # 448 = 1.75 * 2^8: either side of a step of the scale
            top = torch.tensor(frac * 2.0 ** e, device="cuda").bfloat16()
            v = every[every <= top]
            v = torch.cat([v, v.new_zeros(-v.numel() % 127)]).view(-1, 127)
            x = torch.cat([v, top.expand(v.size(0), 1)], dim=1).contiguous()
            x[::2] *= -1
            q, s = kernel.act_quant(x, 128, "ue8m0")
            assert bool((torch.frexp(s)[0] == 0.5).all())
            assert torch.equal(q.view(torch.uint8), _e4m3((x.double() / s.double()).float()))


@pytest.mark.parametrize("fmt", [None, "ue8m0"])
@pytest.mark.parametrize("blocks", [1, 17, 24000])       # one block to a half-warp; four, the last CTA partly empty
def test_blocks_with_nan_and_infinities(fmt, blocks):
    import kernel
    g = torch.Generator(device="cuda").manual_seed(blocks)
    x = torch.randn(blocks, 128, generator=g, device="cuda", dtype=torch.float32).bfloat16()
    x[::3, 5] = float("nan")
    x[::5] = float("nan")                                 # nothing else: the scale of an empty block
    x[1::7, 127] = float("-inf")
    q, s = kernel.act_quant(x, 128, fmt)
    f = x.float()
    amax = torch.where(f.isnan(), 0.0, f.abs()).amax(dim=1).clamp(min=1e-4)
    want = amax / 448
    if fmt:
        want = torch.exp2(torch.ceil(torch.log2(want)))
    assert bool((((s[:, 0] - want).abs() <= 4e-7 * want) | (s[:, 0] == want)).all())          # div.full: within 2 ulp of the quotient
    nan = f.isnan() | (f.isinf() & s.isinf())
    assert bool(((q.view(torch.uint8) & 0x7F) == 0x7F)[nan].all()) and bool(((q.view(torch.uint8) & 0x7F) != 0x7F)[~nan].all())
    ok = (f / s)[~nan]
    err = (q.float()[~nan] - ok.clamp(-448, 448)).abs()
    assert bool((err <= ok.abs() / 16 + 2.0 ** -10 + 1e-5).all())             # half a step of e4m3 and the quotient's own rounding
